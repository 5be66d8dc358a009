"""GPU layer-transfer S matrix (smat_scalc) against the reference S-matrix
program (Smat/Scalc.c).

* the elimination behind it (smat_zsweep) and the LU solve (smat_zgesv) against
  numpy on random, pivoting-heavy and singular systems (block sizes straddling
  the 32-column panels, every cluster size, all exponents);
* the S matrix against the stock Scalc's own output on its fixtures
  (tests/golden/scalc_*.npz) and against the oracle restatement on larger
  seeded structures (lossy inner layers, every BoundC);
* the tensor-core product (smat_zgemm mode 1: FP64-accurate complex products
  from bf16 slices, Ozaki scheme) against an extended-precision product, per
  entry within its error bound, on ragged sizes, wide dynamic ranges, zero
  rows and columns; the stock-Scalc comparisons in both dense modes;
* the argument checks.
Tolerance: 1e-10 absolute on S entries (|S| <= 1); the reference's own
unitarity residual is 2e-14 on these cases.
"""
import glob
import os

import numpy as np
import pytest

from oracle import scalc_oracle as SO
from smatranem_gb300 import fdtd, scalc, workloads as W

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
FIXTURES = sorted(glob.glob(os.path.join(HERE, "golden", "scalc_*.npz")))


@pytest.mark.parametrize("n,nrhs", [(1, 1), (5, 3), (31, 7), (32, 32), (33, 40), (100, 64), (257, 300)])
def test_zgesv_matches_numpy(dense, n, nrhs):
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    A[np.arange(n), np.arange(n)] *= 1e-3  # small diagonal: every column pivots
    B = rng.standard_normal((n, nrhs)) + 1j * rng.standard_normal((n, nrhs))
    X, info = scalc.zgesv(A, B)
    assert info == 0
    ref = np.linalg.solve(A, B)
    assert np.abs(X - ref).max() <= 1e-10 * np.abs(ref).max()
    assert np.abs(A @ X - B).max() <= 1e-11 * np.abs(A).max() * np.abs(X).max() * n


def test_zgesv_reports_a_zero_pivot(built):
    A = np.eye(6, dtype=complex)
    A[3, 3] = 0.0
    _, info = scalc.zgesv(A, np.ones(6))
    assert info == 4  # 1-based, as LAPACK's INFO


def _zgemm_case(rng, m, n, k, spread):
    A = (rng.standard_normal((m, k)) + 1j * rng.standard_normal((m, k))) * 10.0 ** rng.uniform(-spread, spread, (m, 1))
    B = (rng.standard_normal((k, n)) + 1j * rng.standard_normal((k, n))) * 10.0 ** rng.uniform(-spread, spread, (1, n))
    if spread:  # entries far below their row's / column's largest, zero rows and columns
        A *= 10.0 ** rng.uniform(-6, 0, (m, k))
        A[m // 3, :] = 0
        B[:, n // 2] = 0
    return A, B


@pytest.mark.parametrize("m,n,k,spread", [(1, 1, 1, 0), (128, 32, 32, 0), (129, 33, 31, 0), (300, 70, 17, 3),
                                          (500, 260, 100, 0), (77, 500, 64, 8), (300, 40, 2048, 0)])
def test_zgemm_tensor_cores_within_bound(built, m, n, k, spread):
    """Per entry: |C - exact| <= 2e-15 k max|A row| max|B col| + 4 ulp of |C0| + |C|
    (the slices keep 55 bits of each scaled entry; the dropped slice pairs and
    the FP64 sums stay below that), the FP64 kernel on the same inputs."""
    rng = np.random.default_rng(m + 7 * n + 13 * k)
    A, B = _zgemm_case(rng, m, n, k, spread)
    C0 = rng.standard_normal((m, n)) + 1j * rng.standard_normal((m, n))
    alpha = 0.3 - 0.7j
    exact = C0.astype(np.clongdouble) + alpha * (A.astype(np.clongdouble) @ B.astype(np.clongdouble))
    rm = np.abs(np.concatenate([A.real, A.imag], axis=1)).max(axis=1, keepdims=True)
    cm = np.abs(np.concatenate([B.real, B.imag], axis=0)).max(axis=0, keepdims=True)
    for mode in (1, 0):
        got = scalc.zgemm(A, B, C0, alpha, mode=mode)
        err = np.abs(got - exact).astype(np.float64)
        bound = 2e-15 * k * abs(alpha) * rm * cm + 9e-16 * (np.abs(C0) + np.abs(got))
        assert np.all(err <= bound), (mode, float((err / bound).max()))


def test_zgemm_bounded_wait_gives_up(built):
    """A tensor-core product whose slice pair never arrives: its waits run out,
    it records error 1 and returns (no hang, no fault), and the next product
    on the device is right."""
    assert scalc.zgemm_wait_test() == 1
    rng = np.random.default_rng(5)
    A = rng.standard_normal((130, 20)) + 1j * rng.standard_normal((130, 20))
    B = rng.standard_normal((20, 40)) + 1j * rng.standard_normal((20, 40))
    got = scalc.zgemm(A, B, mode=1)
    assert np.abs(got - A @ B).max() <= 1e-13 * np.abs(A).max() * np.abs(B).max() * 20


def test_zgemm_argument_checks(built):
    with pytest.raises(ValueError):
        scalc.zgemm(np.ones((3, 2)), np.ones((3, 2)))  # inner sizes differ
    with pytest.raises(fdtd.FdtdError):
        scalc.zgemm(np.ones((3, 2)), np.ones((2, 2)), mode=2)
    with pytest.raises(fdtd.FdtdError):
        scalc.dense_mode(5)


@pytest.fixture(params=[1, 0], ids=["tensor_cores", "fp64_kernel"])
def dense(request, built):
    scalc.dense_mode(request.param)
    yield request.param
    scalc.dense_mode(1)


@pytest.mark.parametrize("path", FIXTURES, ids=[os.path.basename(p)[:-4] for p in FIXTURES])
def test_smatrix_matches_stock_scalc(dense, path):
    g = np.load(path)
    L = g["L"]
    nB, nT = (int(x) for x in g["nreal"])
    S, info = scalc.smatrix(g["meds"], float(g["omega"]), int(L[0]), int(L[1]), tuple(int(x) for x in g["bc"]),
                            g["XiB"], nB, g["XiT"], nT)
    assert np.abs(S - g["S"]).max() < 1e-10
    assert abs(info["unitarity"] - float(g["unitarity"])) < 1e-11
    nl = len(g["meds"])
    assert info["solves"] == 2 * (2 + 2 * (nl - 2) + 2)  # per direction: set_iniMat, 2 per layer... as Scalc


def _case(L0, L1, nl, bc, seed, lossy):
    from oracle import mode_oracle as MO
    om = 0.405
    med = W.port_layer(L0, L1, core=(3, 2), eps_core=12.11, eps_clad=2.085, seed=seed, jitter=0.2)
    port = MO.calc_Xi(med, om, L0, L1, bc)
    rng = np.random.default_rng(seed)
    meds = [med]
    for _ in range(nl - 2):
        m = med.copy()
        k = rng.integers(0, L0 * L1, size=max(1, L0 * L1 // 6))
        for r in (2, 3, 4):
            m[r, k] = rng.uniform(2.0, 12.0, size=k.size) + (1j * rng.uniform(0.0, 0.3, size=k.size) if lossy else 0)
        meds.append(m)
    meds.append(med)
    return om, np.array(meds), port["Xi"], port["num_real"]


@pytest.mark.parametrize("L0,L1,nl,bc,lossy", [(8, 6, 6, (0, 0), False), (7, 7, 5, (1, -1), True),
                                               (9, 5, 4, (-1, 1), False), (6, 6, 2, (1, 1), False)])
def test_smatrix_matches_oracle(dense, L0, L1, nl, bc, lossy):
    om, meds, Xi, nr = _case(L0, L1, nl, bc, L0 + 10 * L1, lossy)
    ref = SO.smatrix(list(meds), om, L0, L1, bc, Xi, nr, Xi, nr)
    S, info = scalc.smatrix(meds, om, L0, L1, bc, Xi, nr, Xi, nr)
    assert np.abs(S - ref).max() < 1e-10
    if not lossy:
        assert info["unitarity"] < 1e-10
    one, _ = scalc.smatrix(meds, om, L0, L1, bc, Xi, nr, Xi, nr, both_ways=False)
    assert np.abs(one[:, :nr] - ref[:, :nr]).max() < 1e-10


def test_smatrix_argument_checks(built):
    g = np.load(FIXTURES[0])
    L = g["L"]
    nB, nT = (int(x) for x in g["nreal"])
    meds = g["meds"].copy()
    meds[0, 2, 0] += 0.1j  # a lossy port layer: "V is not real in initial_calc"
    with pytest.raises(fdtd.FdtdError) as e:
        scalc.smatrix(meds, float(g["omega"]), int(L[0]), int(L[1]), (0, 0), g["XiB"], nB, g["XiT"], nT)
    assert e.value.code == -1
    with pytest.raises(fdtd.FdtdError):
        scalc.smatrix(g["meds"][:1], float(g["omega"]), int(L[0]), int(L[1]), (0, 0), g["XiB"], nB, g["XiT"], nT)


def test_grating_with_plane_wave_ports(built):
    """The bench's workload form at a small size: closed-form port basis, seeded grating."""
    L0, L1, om = 10, 8, 0.405
    th, Xi, nr = W.plane_wave_basis(L0, L1, omega=om)
    meds = W.grating_layers(L0, L1, 6, seed=7)
    ref = SO.smatrix(list(meds), om, L0, L1, (1, 1), Xi, nr, Xi, nr)
    S, info = scalc.smatrix(meds, om, L0, L1, (1, 1), Xi, nr, Xi, nr)
    assert np.abs(S - ref).max() < 1e-10
    assert info["unitarity"] < 1e-10


@pytest.mark.parametrize("L0,L1,bc,layers,n", [(1, 1, (0, 0), 2, 1), (3, 5, (1, 0), 3, 4), (4, 4, (1, 1), 2, 32),
                                               (3, 11, (0, 1), 3, 7), (8, 9, (1, -1), 4, 3)])
@pytest.mark.parametrize("mode", [1, 0])
def test_sweep_sizes_match_oracle(built, L0, L1, bc, layers, n, mode):
    """The Gauss-Jordan sweeps at orders around their blocks of 32 columns and
    their cluster sizes (NA = 2, 30, 32, 66, 144) and from one port mode to all
    of them, on lossy random layers between dense random port matrices: the
    restatement's S within 1e-9 of its largest entry, an LU form's own
    spread on such ports being under 1e-10; twice the same bits."""
    rng = np.random.default_rng(L0 * 31 + L1)
    NA = 2 * L0 * L1
    n = min(n, NA)
    meds = rng.uniform(1, 4, (layers, 6, L0 * L1)) + 0j
    meds[1:-1] += 0.1j * rng.uniform(0, 1, meds[1:-1].shape)
    Xi = [rng.standard_normal((2 * NA, 2 * NA)) + 1j * rng.standard_normal((2 * NA, 2 * NA)) for _ in range(2)]
    want = SO.smatrix(list(meds), 0.4, L0, L1, bc, Xi[0], n, Xi[1], n)
    try:
        scalc.dense_mode(mode)
        got, info = scalc.smatrix(meds, 0.4, L0, L1, bc, Xi[0], n, Xi[1], n)
        again, _ = scalc.smatrix(meds, 0.4, L0, L1, bc, Xi[0], n, Xi[1], n)
    finally:
        scalc.dense_mode(1)
    assert info["solves"] == 4 * layers and np.array_equal(got, again)
    assert np.abs(got - want).max() <= 1e-9 * np.abs(want).max()


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (130, 17, 5), (128, 16, 32), (257, 33, 40)])
def test_zgemm_results_round_to_nearest(built, m, n, k):
    """B of 8-bit entries (one digit: -128 would take two) meets every digit of A, so the product's integers are
    exact and each result is the exact sum rounded once to the nearest double:
    zeros, both signs, sums of a few bits beside a row's large entry, ties
    (entries a half unit above and below), and results outside the normal range
    (there within a unit of 2^-1074).  k > 32 adds the passes in turn."""
    from fractions import Fraction
    rng = np.random.default_rng(m * n + k)
    ints = rng.integers(-2 ** 53, 2 ** 53, (m, k, 2))
    ints[rng.random(ints.shape) < 0.3] = 0
    ints >>= rng.integers(0, 53, ints.shape)  # entries of every size beside the largest
    ints[:, 0, 0] = 2 ** 53  # the row's largest entry, which column 0 of B does not meet
    bints = rng.integers(-127, 128, (k, n, 2))
    bints[0, :, :] = 0
    if k > 1:
        bints[1:, 0, :] = 0
        bints[1, 0, 0] = 1  # sums of a single entry
    ea = rng.integers(-40, 40, m)
    ea[m // 2] = -600
    eb = rng.integers(-40, 40, n)
    eb[n // 2] = -440
    A = np.ldexp(ints[..., 0].astype(float), ea[:, None] - 53) + 1j * np.ldexp(ints[..., 1].astype(float), ea[:, None] - 53)
    B = np.ldexp(bints[..., 0].astype(float), eb - 7) + 1j * np.ldexp(bints[..., 1].astype(float), eb - 7)
    C = scalc.zgemm(A, B, mode=1)
    a, b = ints.astype(object), bints.astype(object)
    for r in range(0, m, max(1, m // 24)):
        for c in range(n):
            want = np.zeros(2)
            for k0 in range(0, k, 32):
                s = slice(k0, min(k, k0 + 32))
                re = sum(a[r, s, 0] * b[s, c, 0] - a[r, s, 1] * b[s, c, 1])
                im = sum(a[r, s, 0] * b[s, c, 1] + a[r, s, 1] * b[s, c, 0])
                want += [float(Fraction(int(v)) * Fraction(2) ** int(ea[r] + eb[c] - 60)) for v in (re, im)]
            got = np.array([C[r, c].real, C[r, c].imag])
            if np.abs(want).max() < 2.0 ** -1000:
                assert np.abs(got - want).max() <= 2.0 ** -1074, (r, c)
            else:
                assert np.array_equal(got, want), (r, c)


@pytest.mark.parametrize("m,n,k", [(128, 16, 32), (130, 17, 31), (257, 33, 64)])
def test_zgemm_is_within_half_a_unit_and_the_dropped_digits(built, m, n, k):
    """Entries of 53 bits, which the cut into digits keeps whole: what is left out
    are the digit pairs i + l >= 8 of 7 x 7, at most 64 2^14 (5 2^-78 + 4 2^-86
    + 3 2^-94 + ...) of row max times column max a pass, a half unit 2^-63 of it for
    the last level that is kept, and the rounding to a double, of the result and of
    each pass into it."""
    rng = np.random.default_rng(m + n + k)
    a, b = rng.integers(-2 ** 53, 2 ** 53, (m, k, 2)), rng.integers(-2 ** 53, 2 ** 53, (k, n, 2))
    A, B = (np.ldexp(x[..., 0].astype(float), -53) + 1j * np.ldexp(x[..., 1].astype(float), -53) for x in (a, b))
    a[:, 0, 0] = b[0, :, 0] = 2 ** 53 - 1
    A[:, 0], B[0, :] = 1 - 2.0 ** -53 + 1j * A[:, 0].imag, 1 - 2.0 ** -53 + 1j * B[0, :].imag
    C = scalc.zgemm(A, B, mode=1)
    a, b = a.astype(object), b.astype(object)
    passes = (k + 31) // 32
    left = passes * 2.0 ** 106 * (64 * (5 * 2.0 ** -64 + 5 * 2.0 ** -72) + 2.0 ** -63)  # in units of 2^-106
    for r in range(m):
        for v, want in ((C[r].real, a[r, :, 0] @ b[:, :, 0] - a[r, :, 1] @ b[:, :, 1]),
                        (C[r].imag, a[r, :, 0] @ b[:, :, 1] + a[r, :, 1] @ b[:, :, 0])):
            for got, w in zip(v, want):
                unit = 2.0 ** 106 * np.spacing(max(abs(got), 2.0 ** -53))
                err = abs(int(got * 2.0 ** 106) - w)
                # one pass: half a unit of the result; more: of the largest sum on the way too (below 2 k)
                assert err <= left + unit / 2 + (2.0 ** 106 * np.spacing(2.0 * k) if passes > 1 else 0), (r, err, left)


@pytest.mark.parametrize("L0,L1,layers", [(6, 5, 6), (10, 8, 10), (13, 11, 6)])
def test_gratings_to_the_last_digits(dense, L0, L1, layers):
    """S of gratings between plane-wave ports against the restatement (LAPACK):
    2 * layers eliminations of order NA a direction, each of relative error NA
    2^-53 at most on either side, at entries of S up to 1."""
    om = 0.405
    _, Xi, nr = W.plane_wave_basis(L0, L1, omega=om)
    meds = W.grating_layers(L0, L1, layers, seed=3)
    ref = SO.smatrix(list(meds), om, L0, L1, (1, 1), Xi, nr, Xi, nr)
    S, _ = scalc.smatrix(meds, om, L0, L1, (1, 1), Xi, nr, Xi, nr)
    assert np.abs(S - ref).max() <= 2 * 2 * layers * 2 * L0 * L1 * 2.0 ** -53


@pytest.mark.parametrize("L0,L1,bc,layers,n", [(1, 1, (0, 0), 2, 1), (3, 5, (1, 0), 3, 4), (4, 4, (1, 1), 2, 32),
                                               (3, 11, (0, 1), 3, 7), (8, 9, (1, -1), 4, 3)])
def test_random_ports_as_close_as_an_lu(dense, L0, L1, bc, layers, n):
    """Dense random port matrices, at the bound that an LU form keeps: 1e-10 of
    the largest entry."""
    rng = np.random.default_rng(L0 * 31 + L1)
    NA = 2 * L0 * L1
    n = min(n, NA)
    meds = rng.uniform(1, 4, (layers, 6, L0 * L1)) + 0j
    meds[1:-1] += 0.1j * rng.uniform(0, 1, meds[1:-1].shape)
    Xi = [rng.standard_normal((2 * NA, 2 * NA)) + 1j * rng.standard_normal((2 * NA, 2 * NA)) for _ in range(2)]
    want = SO.smatrix(list(meds), 0.4, L0, L1, bc, Xi[0], n, Xi[1], n)
    got, _ = scalc.smatrix(meds, 0.4, L0, L1, bc, Xi[0], n, Xi[1], n)
    assert np.abs(got - want).max() <= 1e-10 * np.abs(want).max()


# ---- the elimination (smat_zsweep) ----------------------------------------------


def _sweep_blocks(A, F, B, G, max_cluster=0):
    """A^-1, A^-1 F, B A^-1, G - B A^-1 F, perm and info by the sweep."""
    n = len(A)
    M, perm, info = scalc.zsweep(np.block([[A, F], [B, G]]), n, max_cluster)
    back = np.empty(n, int)
    back[perm] = np.arange(n)
    return M[:n, :n][:, back], M[:n, n:], -M[n:, :n][:, back], M[n:, n:], perm, info


def _pivots(A):
    """Rows that partial pivoting by |re| + |im| takes, column by column."""
    A, left, out = A.copy(), np.arange(len(A)), []
    for c in range(len(A)):
        p = int(np.argmax(np.abs(A[left, c].real) + np.abs(A[left, c].imag)))
        out.append(left[p])
        left = np.delete(left, p)
        A[left] -= np.outer(A[left, c] / A[out[-1], c], A[out[-1]])
    return np.array(out)


@pytest.mark.parametrize("n,extra", [(1, 0), (5, 3), (31, 1), (33, 40), (64, 0), (130, 9), (257, 300)])
def test_sweep_matches_numpy(dense, n, extra):
    """Small diagonals (every column pivots), orders around the panels of 32 and
    the cluster sizes: every block against numpy, the pivots in the order of
    partial pivoting."""
    rng = np.random.default_rng(n)
    z = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)
    A, F, B, G = z(n, n), z(n, extra), z(extra, n), z(extra, extra)
    A[np.arange(n), np.arange(n)] *= 1e-3
    X, XF, BX, S, perm, info = _sweep_blocks(A, F, B, G)
    assert info == 0 and np.array_equal(perm, _pivots(A))
    ref = np.linalg.inv(A)
    tol = 1e-10 * np.abs(ref).max()
    assert np.abs(X - ref).max() <= tol
    assert np.abs(A @ X - np.eye(n)).max() <= 1e-11 * np.abs(A).max() * np.abs(X).max() * n
    if extra:
        assert np.abs(XF - ref @ F).max() <= tol * n and np.abs(BX - B @ ref).max() <= tol * n
        assert np.abs(S - (G - B @ ref @ F)).max() <= tol * n * n


@pytest.mark.parametrize("n,max_cluster", [(300, 1), (356, 1), (357, 1), (700, 1), (1424, 4), (1425, 4), (600, 8),
                                           (5750, 0)])
def test_sweep_cluster_sizes(built, n, max_cluster):
    """Panels on smaller clusters, of more rows than a CTA has threads, and of rows
    that no longer fit shared memory (order 357 on one CTA, 1425 on four, 5697 on
    sixteen), against the inverse's definition."""
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    A[np.arange(n), np.arange(n)] *= 1e-3
    X, _, _, _, perm, info = _sweep_blocks(A, *(np.zeros(s) for s in ((n, 0), (0, n), (0, 0))), max_cluster)
    assert info == 0 and np.array_equal(np.sort(perm), np.arange(n))
    if n < 1000:
        assert np.array_equal(perm, _pivots(A))
    v = rng.standard_normal((n, 8))
    assert np.abs(A @ (X @ v) - v).max() <= 1e-11 * np.abs(A).max() * np.abs(X).max() * n * np.abs(v).max()


@pytest.mark.parametrize("scale", [2.0 ** 900, 2.0 ** -900])
def test_sweep_of_huge_and_tiny_entries(dense, scale):
    """Pivots whose square leaves the exponent range are no zero pivots."""
    rng = np.random.default_rng(3)
    A = rng.standard_normal((70, 70)) + 1j * rng.standard_normal((70, 70))
    X, _, _, _, perm, info = _sweep_blocks(A * scale, *(np.zeros(s) for s in ((70, 0), (0, 70), (0, 0))))
    assert info == 0 and np.array_equal(perm, _pivots(A))
    ref = np.linalg.inv(A)
    assert np.abs(X * scale - ref).max() <= 1e-11 * np.abs(ref).max()


def test_sweep_pivot_reciprocals(built):
    """The inverse of a diagonal matrix is its pivots' reciprocals: conj(d) / |d|^2
    with |d|^2 (two roundings), its reciprocal (one and 2^-57) and a product
    (one), a relative error of at most 4.5 2^-53 a part, over all exponents at
    which the result is a normal number."""
    from fractions import Fraction
    rng = np.random.default_rng(9)
    n = 1500
    d = np.ldexp(rng.uniform(0.5, 1, n), rng.integers(-1021, 1020, n)) * rng.choice([-1, 1], n) \
        + 1j * np.ldexp(rng.uniform(0.5, 1, n), rng.integers(-1021, 1020, n)) * rng.choice([-1, 1], n)
    near = np.abs(d.real) * np.ldexp(rng.uniform(0.5, 1, n), rng.integers(-20, 1, n))
    d = np.where(rng.random(n) < 0.7, d.real + 1j * near, d)  # parts of like size
    d[:4] = 2.0 ** -812, 2.0 ** 850, 2.0 ** -1021, 2.0 ** 1021
    X, _, _, _, perm, info = _sweep_blocks(np.diag(d), np.zeros((n, 0)), np.zeros((0, n)), np.zeros((0, 0)))
    assert info == 0 and np.array_equal(perm, np.arange(n))
    assert np.array_equal(X, np.diag(np.diag(X)))
    for v, x in zip(d, np.diag(X)):
        a, b = Fraction(v.real), Fraction(v.imag)
        s = a * a + b * b
        for got, want in ((x.real, a / s), (x.imag, -b / s)):
            if want == 0 or not Fraction(2) ** -1020 < abs(want) < Fraction(2) ** 1023:
                continue
            assert abs(Fraction(float(got)) - want) <= abs(want) * Fraction(9, 2) * Fraction(2) ** -53, v


@pytest.mark.parametrize("step", [2.0 ** -30, 2.0 ** -51])
def test_sweep_pivots_by_all_bits(built, step):
    """Of two candidates that differ in their last bits the larger is taken: within
    a warp, in two warps and on two CTAs."""
    n = 200
    for r, q in ((3, 9), (9, 3), (1, 190), (190, 1), (100, 101)):
        A = np.eye(n) * 0.5 + 0j
        A[r, 0], A[q, 0] = 1.0, 1.0 + step
        *_, perm, info = _sweep_blocks(A, np.zeros((n, 0)), np.zeros((0, n)), np.zeros((0, 0)))
        assert info == 0 and perm[0] == q


def test_sweep_reports_a_zero_pivot(dense):
    """A column without a pivot, in the first panel and in a later one."""
    rng = np.random.default_rng(4)
    for n, c in ((6, 3), (80, 50), (200, 140)):
        A = np.triu(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) + 4 * np.eye(n)
        A[c, c:] = 0
        *_, info = _sweep_blocks(A, np.zeros((n, 0)), np.zeros((0, n)), np.zeros((0, 0)))
        assert info == c + 1
    A = np.eye(40)
    A[:, 7] = 0
    *_, info = _sweep_blocks(A, np.zeros((40, 0)), np.zeros((0, 40)), np.zeros((0, 0)))
    assert info == 8  # 1-based, as LAPACK's INFO


def test_smatrix_of_a_singular_port_is_refused(dense):
    L0, L1, n = 4, 3, 2
    NA = 2 * L0 * L1
    meds = np.random.default_rng(1).uniform(1, 4, (3, 6, L0 * L1)) + 0j
    with pytest.raises(fdtd.FdtdError) as e:
        scalc.smatrix(meds, 0.4, L0, L1, (1, 1), np.zeros((2 * NA, 2 * NA)), n, np.eye(2 * NA), n)
    assert e.value.code == -6


def test_port_matrices_in_either_order(built):
    """Row-major, column-major and strided port matrices, alike or mixed, give
    the same bits."""
    rng = np.random.default_rng(5)
    L0, L1, n = 4, 3, 5
    NA = 2 * L0 * L1
    meds = rng.uniform(1, 4, (3, 6, L0 * L1)) + 0j
    X = [rng.standard_normal((2 * NA, 2 * NA)) + 1j * rng.standard_normal((2 * NA, 2 * NA)) for _ in range(2)]
    wide = np.zeros((2 * NA, 4 * NA), np.complex128)
    wide[:, ::2] = X[0]
    ref, _ = scalc.smatrix(meds, 0.4, L0, L1, (1, 1), np.asfortranarray(X[0]), n, np.asfortranarray(X[1]), n)
    for b in (X[0], np.asfortranarray(X[0]), wide[:, ::2]):
        for t in (X[1], np.asfortranarray(X[1])):
            got, _ = scalc.smatrix(meds, 0.4, L0, L1, (1, 1), b, n, t, n)
            assert np.array_equal(got, ref)
    ref, _ = scalc.smatrix(meds, 0.4, L0, L1, (1, 1), np.asfortranarray(X[0]), n, np.asfortranarray(X[0]), n)
    got, _ = scalc.smatrix(meds, 0.4, L0, L1, (1, 1), X[0], n, X[0], n)
    assert np.array_equal(got, ref)
