"""Performance cases: the work that users of this package have it do.

A case is a dict of plain values; ``kind`` says which entry points it goes
through:

* ``fdtd``: ``Plan.run`` over a stretch of a pulse run with the running DFT,
  then the S extraction (``Plan.overlap``) of one monitor plane.  ``source``
  names the structure: ``bend`` (curvilinear strip bend, a metric factor per
  cell), ``slab`` (uniform mesh, seeded inclusions), ``cube`` (block over a PEC
  plate), ``patches`` (PEC patch array on a slab, curved substrate), ``guide``
  (straight guide, PML on the z faces only).  ``tuned`` plans are autotuned
  first, as the integration guide advises for FP32; FP64 plans have one form.
* ``group``: ``Group.run`` over plans of uneven size in one launch per step.
* ``adjoint``: ``Plan.adjoint_grad``, forward with checkpoints and backward.
* ``scalc``: ``scalc.smatrix``, both directions, plane-wave ports.
* ``modes``: ``modes.solve`` of one port layer.

The structures depend on the case alone (a user keeps one and varies the
excitation), the excitations, objectives, gratings and port media on the seed.
"""
from __future__ import annotations

import ctypes
import functools
import math

import numpy as np
import torch

from smatranem_gb300 import fdtd as F
from smatranem_gb300 import modes as M
from smatranem_gb300 import scalc as S

OMEGA = 2 * math.pi * 0.1 / 1.55  # 1.55 um light, lengths in 0.1 um
PML = 12                          # cells of split PML, 6 on short axes
EPS_SI, EPS_OX = 12.11, 2.085


def listed():
    return [
        # the batched S matrix of the bend (2 ports x 4 modes), 21 wavelengths: the package's headline use
        dict(name="fdtd_bend_256x192x160_x8_fp32", kind="fdtd", source="bend", L0=256, L1=192, L2=160, batch=8,
             fp64=False, tuned=True, steps=64, nfreq=21),
        # one excitation of a device of ordinary size, as the drop-in program runs it with precision = FP32
        dict(name="fdtd_bend_160x160x120_fp32", kind="fdtd", source="bend", L0=160, L1=160, L2=120, batch=1,
             fp64=False, tuned=True, steps=96, nfreq=1),
        # a mesh of odd size straight from the mesher, two ports; a run of a ragged number of steps
        dict(name="fdtd_slab_131x117x103_x2_fp32", kind="fdtd", source="slab", L0=131, L1=117, L2=103, batch=2,
             fp64=False, tuned=True, steps=80, nfreq=11),
        # a wide domain with metal patches: half the large-domain configuration along each axis
        dict(name="fdtd_patches_320x320x256_fp32", kind="fdtd", source="patches", L0=320, L1=320, L2=256, batch=1,
             fp64=False, tuned=True, steps=32, nfreq=5),
        # the plain FP64 cube: the drop-in program's default precision, with a PEC plate, 11 wavelengths
        dict(name="fdtd_cube_96_fp64", kind="fdtd", source="cube", L0=96, L1=96, L2=96, batch=1, fp64=True,
             tuned=False, steps=64, nfreq=11),
        # a curvilinear FP64 run with two ports (the reference answer for an FP32 one)
        dict(name="fdtd_bend_130x98x81_x2_fp64", kind="fdtd", source="bend", L0=130, L1=98, L2=81, batch=2, fp64=True,
             tuned=False, steps=48, nfreq=3),
        # the smallest decks: a short guide in FP64, where launches and latency count
        dict(name="fdtd_guide_24x20x40_fp64", kind="fdtd", source="guide", L0=24, L1=20, L2=40, batch=1, fp64=True,
             tuned=False, steps=100, nfreq=1),
        # many structures of uneven size in one launch per step
        dict(name="group_6_slabs_bend_x4_fp32", kind="group", members=6, lo=104, hi=168, batch=4, steps=32, nfreq=3),
        # an inverse-design iteration: objective and gradient of every design cell
        dict(name="adjoint_design_160x160x120_fp32", kind="adjoint", L0=160, L1=160, L2=120, nx=60, ny=60, nz=20,
             fp64=False, steps=128, K=64),
        # the frequency-domain S matrix of a small and of an ordinary cross-section
        dict(name="scalc_grating_10x10", kind="scalc", L0=10, L1=10, layers=10),
        dict(name="scalc_grating_24x24", kind="scalc", L0=24, L1=24, layers=10),
        # the port modes of the bend's port layer
        dict(name="modes_port_256x192", kind="modes", L0=256, L1=192, nmodes=4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fdtd32", "fdtd32", "fdtd64", "fdtd64", "group", "adjoint", "scalc", "modes"])
    if kind in ("fdtd32", "fdtd64"):
        fp64 = kind == "fdtd64"
        source = rng.choice(["bend", "slab", "patches"] if not fp64 else ["bend", "slab", "cube", "guide"])
        side = [_log(rng, 48, 224 if not fp64 else 128) for _ in range(3)]
        if source == "cube":
            side = [side[0]] * 3
        elif source == "guide":
            side = [_log(rng, 16, 40), _log(rng, 16, 40), _log(rng, 32, 64)]
        if not fp64 and rng.random() < 0.6:
            side[0] -= side[0] % 4  # most meshes are made even along x, not all
        cells = side[0] * side[1] * side[2]
        batch = rng.choice([1, 1, 2, 4, 8])
        while batch > 1 and cells * batch > (4e7 if not fp64 else 4e6):
            batch //= 2
        return dict(kind="fdtd", source=source, L0=side[0], L1=side[1], L2=side[2], batch=batch, fp64=fp64,
                    tuned=not fp64 and rng.random() < 0.75, steps=rng.randrange(32, 129, 2),
                    nfreq=rng.choice([1, 3, 5, 11, 21]))
    if kind == "group":
        lo = _log(rng, 64, 128)
        return dict(kind="group", members=rng.randrange(2, 9), lo=lo, hi=rng.randrange(lo, 180),
                    batch=rng.choice([1, 2, 4, 8]), steps=rng.randrange(32, 65, 2), nfreq=rng.choice([1, 3, 5]))
    if kind == "adjoint":
        side = [_log(rng, 64, 160) for _ in range(3)]
        return dict(kind="adjoint", L0=side[0] - (side[0] % 4 if rng.random() < 0.7 else 0), L1=side[1],
                    L2=max(72, side[2] // 4 * 3), nx=rng.randrange(8, 24), ny=rng.randrange(8, 24),
                    nz=rng.randrange(4, 20), fp64=rng.random() < 0.25, steps=rng.randrange(64, 129),
                    K=rng.choice([16, 32, 64]))
    if kind == "scalc":
        return dict(kind="scalc", L0=_log(rng, 6, 24), L1=_log(rng, 6, 24), layers=rng.randrange(4, 11))
    return dict(kind="modes", L0=_log(rng, 24, 256), L1=_log(rng, 20, 192), nmodes=rng.randrange(1, 5))


# ---- structures ----------------------------------------------------------------------------------------------------


class Structure:
    """Real media with their metric factors ((L2, L1, L0, 3)), PML profiles per axis ((2, n): H and E sub-points),
    time step constants, monitor and source planes."""

    def __init__(self, L, mu, eps, sig, planes, iI, pec=None, bc=(0, 0, 0)):
        self.L, self.mu, self.eps, self.sig, self.planes, self.iI, self.pec, self.bc = L, mu, eps, sig, planes, iI, pec, bc
        e, m = eps[..., 0] + eps[..., 1] + eps[..., 2], mu[..., 0] + mu[..., 1] + mu[..., 2]
        r = (eps[..., 0] * eps[..., 1] * eps[..., 2]) / e * ((mu[..., 0] * mu[..., 1] * mu[..., 2]) / m)
        min_dt = 0.99 * float(r.min()) ** 0.25
        n = math.floor(2 * math.pi / (OMEGA * min_dt)) + 1
        dphi = 2 * math.pi / n
        self.dt = dphi / OMEGA
        self.tR = 0.5 * dphi / (self.dt * math.sin(0.5 * dphi))
        self.tI = 0.5 * OMEGA / math.cos(0.5 * dphi)

    @property
    def sigma(self):
        return np.concatenate([np.stack([s[0], s[1]], 1).reshape(-1) for s in self.sig])

    @property
    def split(self):
        """Cells in a PML, (L2, L1, L0)."""
        x, y, z = ((np.abs(s) > 2.3e-15).any(0) for s in self.sig)
        return x[None, None, :] | y[None, :, None] | z[:, None, None]


def _pml(n, cells, d):
    out = np.zeros((2, n))
    if cells:
        smax = 4 * 27.6 / (4 * OMEGA * cells * d)
        for h, shift in ((0, 0.5), (1, 1.0)):
            x = np.arange(n) + shift
            out[h] = smax * (np.clip((cells - x) / cells, 0, None) ** 3 + np.clip((x - (n - cells)) / cells, 0, None) ** 3)
    return out


def _uniform(eps, d, pec=None, planes=None, sides=True):
    L2, L1, L0 = eps.shape
    w = [PML if n >= 64 else 6 for n in (L0, L1, L2)]
    sig = [_pml(n, w[a] if sides or a == 2 else 0, d) for a, n in enumerate((L0, L1, L2))]
    e = np.repeat(eps[..., None] * d, 3, axis=3)
    p = planes or (w[2] + 1, L2 - w[2] - 2)
    return Structure((L0, L1, L2), np.full(e.shape, d), e, sig, p, (p[0] + 2, p[1] - 2), pec)


@functools.lru_cache(maxsize=32)
def structure(source, L0, L1, L2):
    x, y = np.arange(L0) - L0 / 2 + 0.5, np.arange(L1) - L1 / 2 + 0.5
    core = (np.abs(x)[None, None, :] <= max(3.0, L0 / 20)) & (np.abs(y)[None, :, None] <= max(2.0, L1 / 30)) & \
        np.ones((L2, 1, 1), bool)
    if source == "bend":  # cells of 15-25 nm, radius 2 um around the inner side: a metric factor per cell
        w = [PML if n >= 64 else 6 for n in (L0, L1, L2)]
        d0 = 0.15 + 0.10 * (1 - np.exp(-((np.arange(L0) - 0.2 * L0) / 40) ** 2))
        d1 = 0.15 + 0.10 * (1 - np.exp(-((np.arange(L1) - 0.5 * L1) / 30) ** 2))
        u0 = np.cumsum(d0) - d0.sum() * 0.2
        h2 = 0.2 * (1 + u0 / 20.0 * min(1.0, 10.0 / abs(u0[0])))
        H = [d0[None, None, :], d1[None, :, None], np.broadcast_to(h2, (L2, 1, L0))]
        full = np.ones((L2, L1, L0))
        mu = np.stack([H[(c + 1) % 3] * H[(c + 2) % 3] / H[c] * full for c in range(3)], 3)
        eps = np.where(core, EPS_SI, EPS_OX)[..., None] * mu
        sig = [_pml(n, w[a], d) for a, (n, d) in enumerate(((L0, d0.mean()), (L1, d1.mean()), (L2, 0.2)))]
        p = (w[2] + 1, L2 - w[2] - 2)
        return Structure((L0, L1, L2), mu, eps, sig, p, (p[0] + 2, p[1] - 2))
    if source == "slab":
        eps = np.where(np.abs(y)[None, :, None] <= 5.5, EPS_SI, EPS_OX) * np.ones((L2, 1, L0))
        r = np.random.RandomState(L0 * 7 + L1 * 3 + L2)
        for _ in range(r.randint(1, 7)):
            a = [r.randint(n // 5, n // 2) for n in (L2, L1, L0)]
            b = [v + r.randint(4, n // 3) for v, n in zip(a, (L2, L1, L0))]
            eps[a[0]:b[0], a[1]:b[1], a[2]:b[2]] = r.uniform(EPS_OX, EPS_SI)
        return _uniform(eps, 0.2)
    if source == "guide":
        return _uniform(np.where(core, EPS_SI, EPS_OX), 0.2, sides=False)
    z = np.arange(L2)
    if source == "cube":
        n = L0 * 5 // 16
        c = (np.abs(x) < n / 2)
        eps = np.where(c[None, None, :] & c[None, :, None] & (np.abs(z - L2 / 2 + 0.5) < n / 2)[:, None, None],
                       EPS_SI, 1.0)
        pl, zp = np.abs(x) < L0 * 5 / 24, L2 // 2 - n // 2 - L2 // 8
        pec = (z == zp)[:, None, None] & pl[None, :, None] & pl[None, None, :]
        return _uniform(eps, 0.2, pec.astype(np.uint8), planes=(zp + 3, L2 - PML - 8))
    # patches: a slab with a PEC patch array on its top face, the x arc on a radius of 50 um
    z0, z1 = int(0.3 * L2), int(0.5 * L2)
    eps = np.where((z >= z0) & (z < z1), EPS_OX, 1.0)[:, None, None, None]
    h0 = 1 + (z - L2 / 2 + 0.5) * 0.02 / 50.0
    mu = np.stack([0.2 / h0, 0.2 * h0, 0.2 * h0], 1)[:, None, None, :] * np.ones((1, L1, L0, 1))
    w = [PML if n >= 64 else 6 for n in (L0, L1, L2)]
    px = [((np.arange(n) % 40) >= 10) & ((np.arange(n) % 40) < 30) & (np.arange(n) > w[a]) & (np.arange(n) < n - w[a] - 1)
          for a, n in enumerate((L0, L1))]
    pec = ((z >= z1) & (z < z1 + 2))[:, None, None] & px[1][None, :, None] & px[0][None, None, :]
    p = (z1 - 4, z1 + 6)
    return Structure((L0, L1, L2), mu, eps * mu, [_pml(n, w[a], 0.2) for a, n in enumerate((L0, L1, L2))], p,
                     (z1 - 8, z1 + 10), pec.astype(np.uint8))


@functools.lru_cache(maxsize=32)
def media(source, L0, L1, L2):
    """What a plan is created from: flat complex media, sigma, PEC mask."""
    s = structure(source, L0, L1, L2)
    return (s.mu.reshape(-1).astype(np.complex128), s.eps.reshape(-1).astype(np.complex128), s.sigma,
            None if s.pec is None else s.pec.reshape(-1))


def sheets(L0, L1, batch, seed):
    """Mode-like source sheets (Gaussian spots, TE and TM in turn) and their overlap columns, one per excitation."""
    r = np.random.RandomState(seed % (1 << 31))
    out = []
    for b in range(batch):
        cx, cy = L0 / 2 + r.uniform(-2, 2), L1 / 2 + r.uniform(-2, 2)
        wx, wy = r.uniform(4, 9), r.uniform(3, 7)
        g = np.exp(-((np.arange(L0) - cx) / wx)[None, :] ** 2 - ((np.arange(L1) - cy) / wy)[:, None] ** 2).reshape(-1)
        g = g / math.sqrt(4.8 * float(np.sum(g * g)))
        H, E = np.zeros((L0 * L1, 2), np.complex128), np.zeros((L0 * L1, 2), np.complex128)
        if b % 2 == 0:
            E[:, 0], H[:, 1] = g, 2.4 * g
        else:
            E[:, 1], H[:, 0] = g, -2.4 * g
        out.append((H.reshape(-1), E.reshape(-1), np.concatenate([H[:, 0], H[:, 1], -E[:, 1], E[:, 0]])))
    return out


def pulse(s, steps, nfreq, seed):
    """The source waveform around a pulse's peak and the DFT phases of nfreq wavelengths (1.50-1.60 um)."""
    t = np.arange(steps) * s.dt + (seed % 97) * 0.1
    src, ph = np.zeros((steps, 6)), np.zeros((steps, nfreq, 4))
    for i, off in ((0, 0.5), (3, 1.0)):
        src[:, i] = np.exp(-0.5 * ((np.arange(steps) - steps / 2) / (0.6 * steps)) ** 2)
        src[:, i + 1] = np.sin(OMEGA * (t + off * s.dt))
    om = OMEGA * 1.55 / np.linspace(1.5, 1.6, nfreq) if nfreq > 1 else np.array([OMEGA])
    for i, off in ((0, 1.0), (2, 1.5)):
        ph[..., i], ph[..., i + 1] = np.cos(om * (t[:, None] + off * s.dt)), np.sin(om * (t[:, None] + off * s.dt))
    return src, ph


class _Accumulators:
    """A plan's DFT accumulators where they are, on the GPU."""

    def __init__(self, plan, b, f, q, shape):
        self.plan = plan  # a tensor on the buffer keeps its plan
        ptr, stride = ctypes.c_void_p(), ctypes.c_longlong()
        F._check(F.lib().smat_fdtd_dft_device(plan._h, b, f, q, ctypes.byref(ptr), ctypes.byref(stride)))
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<f8", data=(ptr.value, False), version=3)


def dft(plan):
    nf, nq = plan.dft_count()
    return torch.as_tensor(_Accumulators(plan, 0, 0, 0, (plan.batch, nf, nq, 4, plan.pl, 2)), device="cuda")


def make_plan(source, L0, L1, L2, batch, fp64, steps, nfreq, seed, tuned=False):
    s, (mu, eps, sigma, pec) = structure(source, L0, L1, L2), media(source, L0, L1, L2)
    p = F.Plan.create((L0, L1, L2, 0), s.bc, (*s.planes, s.iI[0], 1), s.tR, s.tI, mu, eps, sigma,
                      precision=F.FP64 if fp64 else F.FP32, batch=batch, pec=pec)
    if tuned:
        p.autotune(4)
    ex = sheets(L0, L1, batch, seed)
    for b, (H, E, _) in enumerate(ex):
        p.set_incident(b, H, E)
        top = b >= (batch + 1) // 2  # the second half of the excitations enter at the other port
        p.set_source_plane(b, s.iI[top], -1 if top else 1)
    src, ph = pulse(s, steps, nfreq, seed)
    p.set_schedule(src, planes=s.planes, phase=ph)
    return p, np.stack([e[2] for e in ex])


# ---- the cases -----------------------------------------------------------------------------------------------------


def _members(c):
    """(source, sizes, batch) of a group's plans: slabs from lo to hi, then a bend with a batch."""
    out = []
    for i in range(c["members"]):
        n = c["lo"] + (c["hi"] - c["lo"]) * i // max(1, c["members"] - 1)
        out.append(("slab", n - n % 8, n - (5 * i) % 13, max(40, n - (7 * i) % 17), 1))
    n = (c["lo"] + c["hi"]) // 2
    return out + [("bend", n - n % 4, n, n - 10, c["batch"])]


def _design(c):
    """The design box, centred, and its permittivity factors are part of the structure."""
    a = [(n - m) // 2 for n, m in ((c["L0"], c["nx"]), (c["L1"], c["ny"]), (c["L2"], c["nz"]))]
    return (a[0], a[0] + c["nx"], a[1], a[1] + c["ny"], a[2], a[2] + c["nz"])


@functools.lru_cache(maxsize=4)
def _design_structure(L0, L1, L2, box, seed):
    """A straight guide through a box of random permittivity."""
    x0, x1, y0, y1, z0, z1 = box
    eps = structure("guide", L0, L1, L2).eps[..., 0] / 0.2
    eps = eps.copy()
    eps[z0:z1, y0:y1, x0:x1] = np.random.RandomState(seed % (1 << 31)).uniform(EPS_OX, EPS_SI, (z1 - z0, y1 - y0, x1 - x0))
    s = _uniform(eps, 0.2)
    s.planes = (s.planes[0], min(z1 + 4, s.planes[1]))
    s.iI = (max(z0 - 4, s.planes[0] + 1), s.iI[1])
    return s


def _grating(c, seed):
    """Layers of media (6, L0*L1) between uniform ports, a rectangle of silicon somewhere on each inner one."""
    r = np.random.RandomState(seed % (1 << 31))
    L0, L1 = c["L0"], c["L1"]
    i0, i1 = np.tile(np.arange(L0), L1), np.repeat(np.arange(L1), L0)
    out = []
    for z in range(c["layers"]):
        eps = np.full(L0 * L1, EPS_OX)
        if 0 < z < c["layers"] - 1:
            a0, a1, w0, w1 = r.randint(L0), r.randint(L1), r.randint(1, L0), r.randint(1, L1)
            eps = np.where((((i0 - a0) % L0) < w0) & (((i1 - a1) % L1) < w1), r.uniform(4, EPS_SI), eps)
        one = np.ones(L0 * L1)
        out.append(np.stack([one, one, eps, eps, eps, one]).astype(np.complex128))
    return np.array(out)


@functools.lru_cache(maxsize=8)
def _ports(L0, L1):
    """The modes of a uniform periodic port layer in closed form (plane waves), propagating ones first: (Xi, number
    of propagating modes)."""
    n, w = L0 * L1, OMEGA
    i0, i1 = np.tile(np.arange(L0), L1), np.repeat(np.arange(L1), L0)
    modes = []
    for q in range(L1):
        for p in range(L0):
            k0, k1 = 2 * math.pi * p / L0, 2 * math.pi * q / L1
            d = np.array([np.exp(1j * k0) - 1, np.exp(1j * k1) - 1])
            c = np.array([d[1], -d[0]])
            Mk = w * np.eye(2) - np.outer(c.conj(), c) / (w * EPS_OX)
            nd = np.linalg.norm(d)
            ph = np.exp(1j * (k0 * i0 + k1 * i1)) / math.sqrt(n)
            for u in ([1, 0], [0, 1]) if nd == 0 else (c.conj() / nd, d / nd):
                u = np.asarray(u, np.complex128)
                modes.append((w * w * EPS_OX - nd * nd, np.kron(u, ph), np.kron(Mk @ u, ph)))
    modes.sort(key=lambda m: -m[0])
    N = 2 * n
    Xi, real = np.zeros((2 * N, 2 * N), np.complex128), sum(m[0] > 0 for m in modes)
    for j, (lam, h, e) in enumerate(modes):
        s = np.sqrt(complex(lam))
        t = 2 * np.arcsin(s / 2)
        f, b = np.concatenate([np.exp(-0.5j * t) * h, e / s]), np.concatenate([np.exp(0.5j * t) * h, -e / s])
        if j < real:
            f, b = (v / math.sqrt(abs(2 * np.vdot(v[:N], v[N:]).real)) for v in (f, b))
        else:
            z = np.sqrt(np.vdot(b[:N], f[N:]) + np.vdot(b[N:], f[:N]))
            f, b = f / z, b / z.conj()
        Xi[:, j], Xi[:, j + N] = f, b
    return Xi, real


def _port_layer(c, seed):
    """A silicon core in oxide on a graded mesh; the core's place and index vary a little."""
    r = np.random.RandomState(seed % (1 << 31))
    L0, L1 = c["L0"], c["L1"]
    d0 = 0.15 + 0.10 * (1 - np.exp(-((np.arange(L0) - 0.45 * L0) / (0.16 * L0)) ** 2))
    d1 = 0.15 + 0.10 * (1 - np.exp(-((np.arange(L1) - 0.5 * L1) / (0.16 * L1)) ** 2))
    x, y = np.cumsum(d0) - d0.sum() * 0.45 + r.uniform(-0.2, 0.2), np.cumsum(d1) - d1.sum() * 0.5 + r.uniform(-0.2, 0.2)
    d0, d1 = np.broadcast_to(d0[None, :], (L1, L0)), np.broadcast_to(d1[:, None], (L1, L0))
    core = (np.abs(x)[None, :] <= 2.6) & (np.abs(y)[:, None] <= 1.7)
    eps = np.where(core, EPS_SI + r.uniform(-0.3, 0.3), EPS_OX)
    f = [d1 * 0.2 / d0, 0.2 * d0 / d1, d0 * d1 / 0.2]
    return np.stack([f[0], f[1], eps * f[2], eps * f[1], eps * f[0], f[2]]).reshape(6, -1).astype(np.complex128)


def prepare(case, seed):
    c = case
    if c["kind"] == "fdtd":
        p, cols = make_plan(c["source"], c["L0"], c["L1"], c["L2"], c["batch"], c["fp64"], c["steps"], c["nfreq"], seed,
                            c["tuned"])
        return dict(case=c, plan=p, cols=cols)
    if c["kind"] == "group":
        ps = [make_plan(src, a, b, d, n, False, c["steps"], c["nfreq"], seed + i)[0]
              for i, (src, a, b, d, n) in enumerate(_members(c))]
        g = F.Group(ps)
        g.set_tuning(3, 1)
        return dict(case=c, group=g, plans=ps)
    if c["kind"] == "adjoint":
        L, box = (c["L0"], c["L1"], c["L2"]), _design(c)
        s = _design_structure(*L, box, seed)
        p = F.Plan.create((*L, 0), s.bc, (*s.planes, s.iI[0], 1), s.tR, s.tI, s.mu.reshape(-1), s.eps.reshape(-1),
                          s.sigma, precision=F.FP64 if c["fp64"] else F.FP32)
        if not c["fp64"]:
            p.autotune(4)
        (H, E, col), = sheets(L[0], L[1], 1, seed)
        p.set_incident(0, H, E)
        src, ph = pulse(s, c["steps"], 1, seed)
        p.set_schedule(src, planes=s.planes, phase=ph)
        return dict(case=c, plan=p, col=col, box=box)
    if c["kind"] == "scalc":
        Xi, n = _ports(c["L0"], c["L1"])
        return dict(case=c, meds=_grating(c, seed), Xi=Xi, n=n)
    return dict(case=c, med=_port_layer(c, seed))


def run(state):
    c = state["case"]
    if c["kind"] == "fdtd":
        p = state["plan"]
        p.run(0, c["steps"])
        return dict(dft=dft(p), S=p.overlap(0, 0, state["cols"]))
    if c["kind"] == "group":
        state["group"].run(0, c["steps"])
        return [dft(p) for p in state["plans"]]
    if c["kind"] == "adjoint":
        J, g, gc = state["plan"].adjoint_grad(c["steps"], c["K"], 0, 1, state["col"], state["box"])
        return dict(J=J, grad=g, grad_c=gc)
    if c["kind"] == "scalc":
        m, _ = S.smatrix(state["meds"], OMEGA, c["L0"], c["L1"], (1, 1), state["Xi"], state["n"], state["Xi"], state["n"])
        return m
    m = M.solve(state["med"], OMEGA, c["L0"], c["L1"], (0, 0), c["nmodes"])
    return dict(theta=m.theta, Xi=m.Xi)


def _step_work(L0, L1, L2, batch, fp64, nfreq, split):
    """One time step: the six components (and a PML cell's second half) of every cell read and written, the
    coefficients read; the DFT sums' share of their read and write each 32 steps (FP64: each step)."""
    n, w = L0 * L1 * L2, 8 if fp64 else 4
    acc = batch * nfreq * 2 * 4 * L0 * L1 * 16
    return (n * (12 * w * batch + 6 * w) + split * 12 * w * batch + 2 * acc / (1 if fp64 else 32),
            36 * n * batch + 4 * acc / 16)


def work(case):
    c = case
    if c["kind"] == "fdtd":
        split = int(structure(c["source"], c["L0"], c["L1"], c["L2"]).split.sum())
        b, f = _step_work(c["L0"], c["L1"], c["L2"], c["batch"], c["fp64"], c["nfreq"], split)
        return dict(bytes=b * c["steps"], flops=f * c["steps"])
    if c["kind"] == "group":
        t = [_step_work(a, b, d, n, False, c["nfreq"], int(structure(src, a, b, d).split.sum()))
             for src, a, b, d, n in _members(c)]
        return dict(bytes=sum(x[0] for x in t) * c["steps"], flops=sum(x[1] for x in t) * c["steps"])
    if c["kind"] == "adjoint":  # forward, recomputation and backward step: each moves a state
        n, w = c["L0"] * c["L1"] * c["L2"], 8 if c["fp64"] else 4
        inner = (c["L0"] - 2 * PML) * (c["L1"] - 2 * PML) * (c["L2"] - 2 * PML)
        b, f = _step_work(c["L0"], c["L1"], c["L2"], 1, c["fp64"], 1, n - inner)
        return dict(bytes=3 * b * c["steps"], flops=3 * f * c["steps"])
    n = 2 * c["L0"] * c["L1"]
    if c["kind"] == "scalc":  # per half layer an LU, a solve with n right-hand sides; two directions
        return dict(bytes=16 * (3 * c["layers"] * n + 8 * n * n), flops=4 * c["layers"] * (8 / 3 + 8) * n ** 3)
    # modes: the layer read, the mode columns written; a few thousand applications of the two stencils to a block
    return dict(bytes=16 * (3 * n + 4 * n * c["nmodes"]), flops=2000 * 12 * 14 * n)


# ---- the same in 64 bits, with torch and numpy alone ---------------------------------------------------------------


class _Exact:
    """The split-field step on float64 tensors (B, L2, L1, L0) per component and half."""

    def __init__(self, s, excitations, src, sides, scale=None):
        self.s, self.src, self.dev = s, src, "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=self.dev)  # noqa: E731
        L0, L1, L2 = s.L
        ax = [(1, 1, L0), (1, L1, 1), (L2, 1, 1)]
        self.A, self.B = [], []
        pec = None if s.pec is None else t(s.pec == 0)
        for h, m in ((0, s.mu), (1, s.eps)):
            A = [t(((s.tR - s.tI * s.sig[a][h]) / (s.tR + s.tI * s.sig[a][h])).reshape(ax[a])) for a in range(3)]
            G = [t((1 / (s.tR + s.tI * s.sig[a][h])).reshape(ax[a])) for a in range(3)]
            keep = pec if h and pec is not None else 1.0
            inv = [keep / t(m[..., c]) for c in range(3)]
            if h and scale is not None:
                inv = [v / scale for v in inv]
            self.A.append([[A[(c + k) % 3] * keep for c in range(3)] for k in (1, 2)])
            self.B.append([[inv[c] * G[(c + k) % 3] for c in range(3)] for k in (1, 2)])
        ok = t(~s.split)
        self.src_cells, n = [], len(excitations)
        for b, (H, E, _) in enumerate(excitations):
            z = s.iI[sides[b]]
            sheet = [t(v.real.reshape(L1, L0, 2)) for v in (E, H)]
            g = -1.0 if sides[b] else 1.0
            self.src_cells.append((z, [[g * ok[z] * x[..., 1], -g * ok[z] * x[..., 0]] for x in sheet]))
        zero = torch.zeros((n, L2, L1, L0), dtype=torch.float64, device=self.dev)
        self.F = [[[zero.clone() for _ in range(3)] for _ in range(2)] for _ in range(2)]  # [H, E][half][component]

    def curl(self, T, c, k, fwd):
        """The half curl along axis c+k of component c+3-k, its wrapped neighbours times the boundary factor (0)."""
        a, f = (c + k) % 3, T[(c + 3 - k) % 3]
        d, n = 3 - a, T[0].shape[3 - a]
        body = torch.diff(f, dim=d)
        edge = f.narrow(d, n - 1, 1) if fwd else f.narrow(d, 0, 1)
        out = torch.cat([body, -edge], d) if fwd else torch.cat([edge, body], d)
        return out if k == 1 else -out

    def half(self, F, T, h, row):
        new = [[], []]
        sg = 1.0 if h else -1.0
        for k in (1, 2):
            for c in range(3):
                w = self.curl(T, c, k, h == 1)
                if k == 1 and c < 2:
                    w = w.clone()
                    for b, (z, sh) in enumerate(self.src_cells):
                        w[b, z] = w[b, z] + row[h] * sh[h][c]
                new[k - 1].append(self.A[h][k - 1][c] * F[k - 1][c] + sg * self.B[h][k - 1][c] * w)
        return new

    def step(self, F, k):
        """F = [H, E] after step k."""
        row = (float(self.src[k, 0] * self.src[k, 1]), float(self.src[k, 3] * self.src[k, 4]))
        H = self.half(F[0], [F[1][0][c] + F[1][1][c] for c in range(3)], 0, row)
        E = self.half(F[1], [H[0][c] + H[1][c] for c in range(3)], 1, row)
        return [H, E]

    def samples(self, F):
        """(B, planes, 4, L0*L1): Hx, Hy, Ex, Ey."""
        out = [F[x][0][c][:, list(self.s.planes)] + F[x][1][c][:, list(self.s.planes)] for x in (0, 1) for c in (0, 1)]
        return torch.stack(out, 2).flatten(3)


def _exact_run(s, ex, batch, steps, nfreq, seed):
    src, ph = pulse(s, steps, nfreq, seed)
    e = _Exact(s, ex, src, [b >= (batch + 1) // 2 for b in range(batch)])
    n = s.L[0] * s.L[1]
    acc = torch.zeros((batch, nfreq, 2, 4, n, 2), dtype=torch.float64, device=e.dev)
    w = torch.as_tensor(ph, device=e.dev).reshape(steps, nfreq, 2, 2)
    for k in range(steps):
        e.F = e.step(e.F, k)
        x = e.samples(e.F)
        for f in range(nfreq):
            for v in range(4):
                for r in range(2):
                    acc[:, f, :, v, :, r] += w[k, f, v // 2, r] * x[:, :, v]
    return acc


def _exact_fdtd(c, seed):
    s, ex = structure(c["source"], c["L0"], c["L1"], c["L2"]), sheets(c["L0"], c["L1"], c["batch"], seed)
    acc = _exact_run(s, ex, c["batch"], c["steps"], c["nfreq"], seed)
    x = torch.view_as_complex(acc[0, :, 0].contiguous())  # (nfreq, 4, n)
    rows = torch.cat([x[:, 0], x[:, 1], -x[:, 3], x[:, 2]], 1).cpu().numpy()
    return dict(dft=acc, S=rows @ np.stack([e[2] for e in ex]).conj().T)


def _exact_adjoint(c, seed):
    L, box = (c["L0"], c["L1"], c["L2"]), _design(c)
    s = _design_structure(*L, box, seed)
    ex = sheets(L[0], L[1], 1, seed)
    src, ph = pulse(s, c["steps"], 1, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x0, x1, y0, y1, z0, z1 = box
    scale = torch.ones((3, z1 - z0, y1 - y0, x1 - x0), dtype=torch.float64, device=dev, requires_grad=True)
    e = _Exact(s, ex, src, [False])
    full = torch.ones((3, L[2], L[1], L[0]), dtype=torch.float64, device=dev)
    full[:, z0:z1, y0:y1, x0:x1] = scale
    for k in range(2):
        e.B[1][k] = [e.B[1][k][comp] / full[comp] for comp in range(3)]
    w = torch.view_as_complex(torch.as_tensor(ph, device=dev).reshape(c["steps"], 2, 2).contiguous())
    t = torch.as_tensor(ex[0][2], device=dev).reshape(4, -1)
    t = torch.stack([t[0], t[1], t[3], -t[2]])  # per sample Hx, Hy, Ex, Ey

    def segment(lo, hi, *flat):
        F = [[list(flat[6 * h + 3 * k:6 * h + 3 * k + 3]) for k in range(2)] for h in range(2)]
        acc = torch.zeros((), dtype=torch.complex128, device=dev)
        for k in range(lo, hi):
            F = e.step(F, k)
            x = e.samples(F)[0, 1]
            acc = acc + w[k, 0] * (t[:2].conj() * x[:2]).sum() + w[k, 1] * (t[2:].conj() * x[2:]).sum()
        return (acc, *[v for h in F for half in h for v in half])

    from torch.utils.checkpoint import checkpoint
    flat, total = [v for h in e.F for half in h for v in half], 0.0
    for lo in range(0, c["steps"], 16):
        acc, *flat = checkpoint(segment, lo, min(c["steps"], lo + 16), *flat, use_reentrant=False)
        total = total + acc
    J = total.real ** 2 + total.imag ** 2
    J.backward()
    g = scale.grad.cpu().numpy()
    return dict(J=float(J.detach()), grad=g.sum(0), grad_c=g)


def _operators(med, L0, L1, bc):
    """The two half-layer operators of a layer as dense matrices, from the forward differences with their wrap."""
    def diff(n, f):
        d = np.diag(np.full(n, -1.0)) + np.diag(np.ones(n - 1), 1)
        d[n - 1, 0] += f
        return d
    D0, D1 = np.kron(np.eye(L1), diff(L0, bc[0])), np.kron(diff(L1, bc[1]), np.eye(L0))
    v = OMEGA * np.real(med)
    maa = np.diag(np.concatenate([v[0], v[1]])) - np.vstack([D1.T, -D0.T]) @ (np.hstack([D1, -D0]) / v[2][:, None])
    mbb = np.diag(np.concatenate([v[3], v[4]])) - np.vstack([D0, D1]) @ (np.hstack([D0.T, D1.T]) / v[5][:, None])
    return maa, mbb


def _exact_scalc(c, seed):
    """The fields x_0 .. x_m of the half layers obey x_{j+1} = x_{j-1} + i iway M_j x_j; eliminated from the
    starting port, whose modes are a (given, forward) and b (unknown, backward), to the ending one."""
    Xi, n = _ports(c["L0"], c["L1"])
    N = Xi.shape[0] // 2
    ops = [_operators(m, c["L0"], c["L1"], (1, 1)) for m in _grating(c, seed)]
    order = [ops[0][1]] + [o[k] for o in ops[1:-1] for k in (0, 1)] + [ops[-1][0]]
    rot = np.roll(Xi, N, axis=0)

    def one_way(iway):
        P = Xi if iway == 1 else np.hstack([rot[:, N:], rot[:, :N]])
        if iway == 1:
            T = np.hstack([np.hstack([rot[:, :n], rot[:, N + n:]]), np.hstack([-rot[:, N:N + n], rot[:, n:N]])])
        else:
            T = np.hstack([np.hstack([-Xi[:, N:N + n], Xi[:, n:N]]), np.hstack([Xi[:, :n], Xi[:, N + n:]])])
        F1, F2, top = P[:N, :n], P[N:, :n], np.eye(n, N)
        B1, B2, F0 = P[:N, N:], P[N:, N:], np.zeros((n, n))

        def eliminate(F0, F1, F2, B0, B1, B2):
            B = np.linalg.solve(B2.T, np.vstack([B0, B1]).T).T
            F = np.vstack([F0, F1]) - B @ F2
            return F[:n], F[n:], B[:n], B[n:]

        F0, F1, B0, B1 = eliminate(F0, F1, F2, top, B1, B2)
        for Mj in order if iway == 1 else order[::-1]:
            F0, F1, B0, B1 = eliminate(F0, np.zeros_like(F1), F1, B0, np.eye(N), B1 + 1j * iway * Mj)
        C = T.conj().T @ np.vstack([np.hstack([F1, B1]), np.hstack([np.zeros((N, n)), np.eye(N)])])
        F0, F1, B0, B1 = eliminate(F0, C[:N, :n], C[N:, :n], B0, C[:N, n:], C[N:, n:])
        return np.vstack([F0, F1[:n]]), np.vstack([B0, B1[:n]])

    (F, B), (G, _) = one_way(1), one_way(-1)
    out = np.zeros((2 * n, 2 * n), np.complex128)
    out[:, :n], out[n:, n:], out[:n, n:] = F, G[:n], G[n:2 * n]
    return out


def _exact_modes(c, seed):
    """The leading eigenpairs of the dense operator, each polished by inverse iteration."""
    K, N = c["nmodes"], 2 * c["L0"] * c["L1"]
    maa, mbb = _operators(_port_layer(c, seed), c["L0"], c["L1"], (0, 0))
    A = mbb @ maa
    lam, X = np.linalg.eig(A)
    order = np.argsort(-lam.real)[:K]
    lam, X = lam[order].real, X[:, order].real
    theta, Xi = np.zeros(2 * K, np.complex128), np.zeros((2 * N, 2 * K), np.complex128)
    for j in range(K):
        h = np.linalg.solve(A - (lam[j] + 1e-12) * np.eye(N), X[:, j])
        h *= np.sign(h[np.abs(h).argmax()]) / np.linalg.norm(h)
        s = math.sqrt(h @ (A @ h))
        t = 2 * math.asin(s / 2)
        theta[j], theta[j + K] = t, -t
        for k, g in ((j, -1), (j + K, 1)):
            v = np.concatenate([np.exp(0.5j * g * t) * h, -g * (maa @ h) / s])
            Xi[:, k] = v / math.sqrt(abs(2 * np.vdot(v[:N], v[N:]).real))
    return dict(theta=theta, Xi=Xi)


def exact(case, seed):
    c = case
    if c["kind"] == "fdtd":
        return _exact_fdtd(c, seed)
    if c["kind"] == "group":
        out = []
        for i, (src, a, b, d, n) in enumerate(_members(c)):
            out.append(_exact_run(structure(src, a, b, d), sheets(a, b, n, seed + i), n, c["steps"], c["nfreq"], seed + i))
        return out
    if c["kind"] == "adjoint":
        return _exact_adjoint(c, seed)
    if c["kind"] == "scalc":
        return _exact_scalc(c, seed) if c["L0"] * c["L1"] <= 600 else None
    # a dense matrix of order 2 L0 L1
    return _exact_modes(c, seed) if c["L0"] * c["L1"] <= 900 else None
