/*
 * Frequency-domain S matrix by layer transfer on the GPU: the reference's
 * Smat/Scalc.c (main :74-96) with its dense steps on the device.
 *
 * Per direction (iway = +1 bottom -> top, -1 top -> bottom; NA = 2*L0*L1, No
 * modes of the starting port) the reference keeps F01 ((No+NA) x No), B01
 * ((No+NA) x NA), F2 (NA x No) and B2 (NA x NA):
 *   set_iniMat (:407-458): the starting port's full mode matrix Phi;
 *   per half layer (initial_calc :192-221, scattering_calc :227-261,
 *   final_calc :269-306): F2 <- field rows of F01, B2 <- field rows of B01
 *   + i*iway*(maa or mbb of the layer), field rows of B01 <- 1, inv_process;
 *   set_finMat (:461-517): project on the ending port's dual modes;
 *   inv_process (:316-400): B01 <- B01 B2^{-1}, F01 <- F01 - B01 F2, F2 = 0,
 *   B2 = 1.
 * Here a direction's state is one matrix, complex FP64 in HBM,
 *     M = [B2, F2; B, F]
 * with the rows of B01 and F01 below, and inv_process one Gauss-Jordan sweep
 * of B2 out of it (dense_z.cuh): every block that it needs comes out of the
 * same updates of rank 32.  Where the field rows of B01 are 1, as in every
 * half layer, the sweep's own block is that product and they are not kept:
 * after it [X, X F2; -B X, F - B X F2] is, up to signs and the order of the
 * columns, the next half layer's M but for the operator, which k_add_op adds
 * (maa and mbb are never formed: each row's stencil coefficients, those of
 * set_M :716-790).
 */
#include <cuda_runtime.h>

#include <chrono>
#include <cmath>
#include <complex>
#include <cstring>
#include <string>
#include <thread>
#include <vector>

#include "dense_z.cuh"
#include "host_internal.h"
#include "smatran_fdtd.h"
#include "trace.cuh"

namespace {

using smat::dense::sweep;
using smat::dense::zgemm_acc;

struct Geo {
    int L0, L1, NA1;
    double s0, s1, e0, e1;  // set_D's diagonal and wrap coefficients (as in the mode solver)
};

__device__ __forceinline__ double cw(int i, int La, double e) { return i < La - 1 ? 1.0 : e; }

/* B2[r, col] += i*sgn * M[r, col] over the stencil of row r; which = 0: maa,
 * 1: mbb; V = 6*NA1 complex set_V values.  One thread per row. */
__global__ void k_add_op(double2 *B2, int ld, Geo g, const double2 *__restrict__ V, int which, double sgn)
{
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    const int NA1 = g.NA1;
    if (r >= 2 * NA1) return;
    const int comp = r / NA1, p = r % NA1;
    const int i0 = p % g.L0, i1 = p / g.L0;
    double2 *row = B2 + r;
    auto pt = [&](int j0, int j1) {
        j0 = ((j0 % g.L0) + g.L0) % g.L0;
        j1 = ((j1 % g.L1) + g.L1) % g.L1;
        return j0 + g.L0 * j1;
    };
    auto emit = [&](int c, int q, double2 v) {  // += i*sgn*v
        double2 *e = row + (long long)ld * (c * NA1 + q);
        e->x -= sgn * v.y;
        e->y += sgn * v.x;
    };
    auto sc = [](double2 v, double f) { return make_double2(v.x * f, v.y * f); };
    auto c0 = [&](int j0) { return cw(((j0 % g.L0) + g.L0) % g.L0, g.L0, g.e0); };
    auto c1 = [&](int j1) { return cw(((j1 % g.L1) + g.L1) % g.L1, g.L1, g.e1); };
    if (which == 0) {
        /* curl terms w(q) = V2(q) (s1 x0(q) + c1 x0(q+e1) - s0 x1(q) - c0 x1(q+e0)), times f */
        auto wt = [&](int j0, int j1, double2 f) {
            const int q = pt(j0, j1);
            emit(0, q, sc(f, g.s1));
            emit(0, pt(j0, j1 + 1), sc(f, c1(j1)));
            emit(1, q, sc(f, -g.s0));
            emit(1, pt(j0 + 1, j1), sc(f, -c0(j0)));
        };
        const double2 *V2 = V + 2 * NA1;
        if (comp == 0) {  // V0 x0 + Ddown1 w
            emit(0, p, V[p]);
            wt(i0, i1, sc(V2[p], -g.s1));
            const int q = pt(i0, i1 - 1);
            wt(i0, i1 - 1, sc(V2[q], -c1(i1 - 1)));
        } else {  // V1 x1 - Ddown0 w
            emit(1, p, V[NA1 + p]);
            wt(i0, i1, sc(V2[p], g.s0));
            const int q = pt(i0 - 1, i1);
            wt(i0 - 1, i1, sc(V2[q], c0(i0 - 1)));
        }
    } else {
        /* u(q) = V5(q) (-s0 y0(q) - c0(q-e0) y0(q-e0) - s1 y1(q) - c1(q-e1) y1(q-e1)), times f */
        auto ut = [&](int j0, int j1, double2 f) {
            emit(0, pt(j0, j1), sc(f, -g.s0));
            emit(0, pt(j0 - 1, j1), sc(f, -c0(j0 - 1)));
            emit(1, pt(j0, j1), sc(f, -g.s1));
            emit(1, pt(j0, j1 - 1), sc(f, -c1(j1 - 1)));
        };
        const double2 *V5 = V + 5 * NA1;
        if (comp == 0) {  // V3 y0 + Dup0 u
            emit(0, p, V[3 * NA1 + p]);
            ut(i0, i1, sc(V5[p], g.s0));
            ut(i0 + 1, i1, sc(V5[pt(i0 + 1, i1)], c0(i0)));
        } else {  // V4 y1 + Dup1 u
            emit(1, p, V[4 * NA1 + p]);
            ut(i0, i1, sc(V5[p], g.s1));
            ut(i0, i1 + 1, sc(V5[pt(i0, i1 + 1)], c1(i1)));
        }
    }
}

/* A port's modes on the device, as the caller holds them: entry (r, c) at
 * r sr + c sc.  The kernels that read them take either order (each reads them
 * once; turning 85 MB of a 24 x 24 lattice round on the host took 28 of 172
 * ms). */
struct Port {
    const double2 *X;
    long long sr, sc;
    __device__ __forceinline__ double2 at(int r, int c) const { return X[r * sr + c * sc]; }
};

/* entry (r, c) of the full mode matrix of set_Phi (:521-551) from Xi (2NA x
 * 2NA, Mcalc's column order) */
__device__ __forceinline__ double2 phi(const Port &Xi, int NA, int iway, int r, int c)
{
    return iway == 1 ? Xi.at(r, c) : Xi.at(r < NA ? r + NA : r - NA, c < NA ? c + NA : c - NA);
}

/* conj of entry (r, c) of the dual mode matrix of set_tilPhi (:555-595) */
__device__ __forceinline__ double2 dual(const Port &Xi, int NA, int iway, int nimag, int r, int c)
{
    const int j = c < NA ? c : c - NA;
    const bool hi = c >= NA, real = j < nimag;
    if (iway == 1) r = r < NA ? r + NA : r - NA;
    /* the second half of Xi's columns: iway = 1, hi == real; -1, hi != real */
    const bool second = (iway == 1) == (hi == real);
    const bool neg = real && second;
    double2 v = Xi.at(r, second ? j + NA : j);
    if (neg) v.x = -v.x;
    else v.y = -v.y;
    return v;
}

/* set_iniMat (:407-458): M = [B2, F2; B0, F0; B1, F1] of the starting port,
 * (2 NA + No) x (NA + No) */
__global__ void k_start(double2 *__restrict__ M, const Port Xi, int NA, int No, int iway)
{
    const int rows = 2 * NA + No;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)rows * (NA + No)) return;
    const int r = (int)(t % rows), c = (int)(t / rows);
    const int pc = c < NA ? NA + c : c - NA; /* B: backward modes, F: forward ones */
    double2 v;
    if (r < NA) v = phi(Xi, NA, iway, NA + r, pc);
    else if (r < NA + No) v = make_double2(r - NA == c ? 1.0 : 0.0, 0.0);
    else v = phi(Xi, NA, iway, r - NA - No, pc);
    M[t] = v;
}

/* The next half layer's M = [B1, F1; B0, F0] ((NA + No) x (NA + No)) from a
 * swept matrix: rows r < NA of it are src rows r0 + r, the No others src rows
 * r1 + r.  Columns c < NA go to perm[c].  own: the first rows are the swept
 * block itself (X, X F2: sign + -), else extra rows (-B X, F - B X F2: - +),
 * as the last No are. */
__global__ void k_next(double2 *__restrict__ M, const double2 *__restrict__ X, int lds, int NA, int No, int r0, int r1,
                       int own, const int *__restrict__ perm)
{
    const int n = NA + No;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)n * n) return;
    const int r = (int)(t % n), c = (int)(t / n);
    double2 v = X[(r < NA ? r0 + r : r1 + r - NA) + (long long)lds * c];
    if ((c < NA) != (r < NA && own)) v = make_double2(-v.x, -v.y);
    M[r + (long long)n * (c < NA ? perm[c] : c)] = v;
}

/* set_finMat (:461-517) before the product: with S = [B1, F1; B0, F0] the last
 * half layer's state and T the dual modes, M = [lower rows of T^H [S1; 1], then
 * its first nimag rows, then B0, F0]: the part of the unit block here (zero in
 * the columns of F), B0 and F0 copied; LP ((NA + nimag) x NA): the factor of
 * S1 = [B1, F1] */
__global__ void k_final(double2 *__restrict__ M, double2 *__restrict__ LP, const double2 *__restrict__ S,
                        const Port Xi, int NA, int No, int nimag, int iway)
{
    const int rows = NA + nimag + No, n = NA + No;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)rows * n) return;
    const int r = (int)(t % rows), c = (int)(t / rows);
    const int tc = r < NA ? NA + r : r - NA; /* the dual mode of a projected row */
    double2 v = make_double2(0.0, 0.0);
    if (r < NA + nimag) {
        if (c < NA) {
            v = dual(Xi, NA, iway, nimag, NA + c, tc);
            LP[r + (long long)(NA + nimag) * c] = dual(Xi, NA, iway, nimag, c, tc);
        }
    } else {
        v = S[NA + (r - NA - nimag) + (long long)n * c];
    }
    M[t] = v;
}

/* the rows Smat_calc reads: out = [F01, the first nimag columns of B01], rows
 * [No of F0, B0; nimag of F1, B1], from the last swept matrix */
__global__ void k_result(double2 *__restrict__ out, const double2 *__restrict__ X, int NA, int No, int nimag,
                         const int *__restrict__ perm)
{
    const int N = No + nimag, lds = NA + N;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)N * (NA + No)) return;
    const int r = (int)(t % N), c = (int)(t / N);
    const double2 v = X[NA + (r < No ? nimag + r : r - No) + (long long)lds * c];
    if (c >= NA) out[r + (long long)N * (c - NA)] = v;
    else if (perm[c] < nimag) out[r + (long long)N * (No + perm[c])] = make_double2(-v.x, -v.y);
}

#define SCK(call)                                                                                                      \
    do {                                                                                                               \
        cudaError_t e_ = (call);                                                                                       \
        if (e_ != cudaSuccess) return smat_fail(SMAT_ECUDA, "%s: %s", #call, cudaGetErrorString(e_));                \
    } while (0)
#define RC(call)                                                                                                       \
    do {                                                                                                               \
        int r_ = (call);                                                                                               \
        if (r_) return r_;                                                                                             \
    } while (0)

struct Transfer {
    Geo g{};
    int NA = 0, No = 0;
    cudaStream_t st = nullptr;
    void *slab = nullptr; /* the one allocation that holds the matrices */
    double2 *M[2] = {nullptr, nullptr}, *LP = nullptr, *out = nullptr;
    smat::dense::SweepWs w{};
    int *dinfo = nullptr;
    int solves = 0;
    smat::dense::GemmCtx gm{0, nullptr, 0, nullptr}; /* how the products run */

    ~Transfer()
    {
        if (st) cudaStreamSynchronize(st);
        smat::dense::gemm_ctx_release(gm);
        cudaFree(slab);
        if (st) cudaStreamDestroy(st);
    }
    static unsigned blocks(long long n, int t) { return (unsigned)((n + t - 1) / t); }
    /* one inv_process on X = M[which] (rows x (NA + No)) */
    int solve(int which, int rows)
    {
        solves++;
        return sweep(NA, rows, NA + No, M[which], rows, w, gm, dinfo, st);
    }
    /* M[0] (k_next's arguments) <- M[1] */
    int next(int lds, int r0, int r1, int own)
    {
        const long long n = NA + No;
        k_next<<<blocks(n * n, 256), 256, 0, st>>>(M[0], M[1], lds, NA, No, r0, r1, own, w.perm);
        SCK(cudaPeekAtLastError());
        return SMAT_OK;
    }
    /* a half layer: the operator into B2, eliminate */
    int step(const double2 *V, int which, int iway)
    {
        const int n = NA + No;
        k_add_op<<<blocks(NA, 128), 128, 0, st>>>(M[0], n, g, V, which, (double)iway);
        SCK(cudaPeekAtLastError());
        std::swap(M[0], M[1]);
        RC(solve(1, n));
        return next(n, 0, NA, 1);
    }
};

/* Scalc's set_V (:838-880): omega * value, rows 2 and 5 inverted as conj(z)/|z|^2;
 * returns the count of entries with a nonzero imaginary part */
int scalc_V(const double *med, long long NA1, double omega, std::vector<std::complex<double>> &v)
{
    v.resize(6 * NA1);
    int comp = 0;
    for (long long k = 0; k < 6 * NA1; k++) {
        std::complex<double> z(med[2 * k] * omega, med[2 * k + 1] * omega);
        const int row = (int)(k / NA1);
        if (row == 2 || row == 5) z = std::conj(z) / (z.real() * z.real() + z.imag() * z.imag());
        v[k] = z;
        if (z.imag() != 0.0) comp++;
    }
    return comp;
}

/* one direction (main :74-94) of nlayers layers whose set_V values are at V
 * (6*NA1 each), the first at istart, in the direction of travel; Xs / Xe:
 * start / end port Xi (device) */
int one_way(Transfer &T, int iway, int nlayers, const double2 *V, const Port &Xs, const Port &Xe, int No, int Nimag,
            std::vector<std::complex<double>> &F01h, std::vector<std::complex<double>> &B01h)
{
    const int NA = T.NA, n = NA + No, N = No + Nimag;
    const long long lv = 6LL * T.g.NA1;
    T.No = No;
    auto layer = [&](int l) { return V + lv * (iway > 0 ? l : nlayers - 1 - l); };
    /* set_iniMat :407-458 */
    const int rows0 = 2 * NA + No;
    k_start<<<Transfer::blocks((long long)rows0 * n, 256), 256, 0, T.st>>>(T.M[1], Xs, NA, No, iway);
    SCK(cudaPeekAtLastError());
    RC(T.solve(1, rows0));
    RC(T.next(rows0, NA + No, NA, 0));
    /* initial_calc :192-221 */
    RC(T.step(layer(0), iway > 0 ? 1 : 0, iway));
    /* scattering_calc :227-261 */
    for (int l = 1; l + 1 < nlayers; l++)
        for (int sub = 0; sub < 2; sub++) RC(T.step(layer(l), ((1 - iway) / 2 + sub) % 2, iway));
    /* final_calc :269-306 */
    RC(T.step(layer(nlayers - 1), iway > 0 ? 0 : 1, iway));
    /* set_finMat :461-517 */
    const int rows1 = NA + N;
    k_final<<<Transfer::blocks((long long)rows1 * n, 256), 256, 0, T.st>>>(T.M[1], T.LP, T.M[0], Xe, NA, No, Nimag, iway);
    SCK(cudaPeekAtLastError());
    RC(zgemm_acc(NA + Nimag, n, NA, make_double2(1.0, 0.0), T.LP, NA + Nimag, T.M[0], n, T.M[1], rows1, &T.gm, T.st));
    RC(T.solve(1, rows1));
    k_result<<<Transfer::blocks((long long)N * n, 256), 256, 0, T.st>>>(T.out, T.M[1], NA, No, Nimag, T.w.perm);
    SCK(cudaPeekAtLastError());
    std::vector<std::complex<double>> h((size_t)N * N);
    SCK(cudaMemcpyAsync(h.data(), T.out, sizeof(double2) * h.size(), cudaMemcpyDeviceToHost, T.st));
    SCK(cudaStreamSynchronize(T.st));
    F01h.assign(h.begin(), h.begin() + (size_t)N * No);
    B01h.assign(h.begin() + (size_t)N * No, h.end());
    return SMAT_OK;
}

} // namespace

extern "C" int smat_scalc(int L0, int L1, const int BoundC[2], double omega, int nlayers, const double *meds,
                          const double *XiB, int nB, const double *XiT, int nT, int both_ways, double *S,
                          smat_scalc_info *info)
{
    return smat_scalc_ordered(L0, L1, BoundC, omega, nlayers, meds, XiB, nB, 0, XiT, nT, 0, both_ways, S, info);
}

extern "C" int smat_scalc_ordered(int L0, int L1, const int BoundC[2], double omega, int nlayers, const double *meds,
                                  const double *XiB, int nB, int rowsB, const double *XiT, int nT, int rowsT,
                                  int both_ways, double *S, smat_scalc_info *info)
{
    smat::TraceRange trace_("smat_scalc");
    const auto t0 = std::chrono::steady_clock::now();
    if (L0 <= 0 || L1 <= 0 || (long long)L0 * L1 > 8192)
        return smat_fail(SMAT_EINVAL, "smat_scalc: lattice %d x %d (dense transfer: 2*L0*L1 <= 16384)", L0, L1);
    if (!BoundC || BoundC[0] < -1 || BoundC[0] > 1 || BoundC[1] < -1 || BoundC[1] > 1)
        return smat_fail(SMAT_EINVAL, "smat_scalc: BoundC");
    if (nlayers < 2 || !meds || !XiB || !XiT || !S) return smat_fail(SMAT_EINVAL, "smat_scalc: nlayers = %d", nlayers);
    const int NA1 = L0 * L1, NA = 2 * NA1, N2 = 2 * NA;
    if (nB < 1 || nT < 1 || nB > NA || nT > NA) return smat_fail(SMAT_EINVAL, "smat_scalc: modes %d, %d", nB, nT);
    if (!(omega > 0) || !std::isfinite(omega)) return smat_fail(SMAT_EINVAL, "smat_scalc: omega = %g", omega);
    const int Nmax = std::max(nB, nT);
    const size_t cols = (size_t)Nmax + NA, rows = cols + NA;
    smat::dense::SweepWs form{};
    RC(smat::dense::sweep_setup(form, NA, 0));
    /* one transfer state per direction: device matrices, stream, product workspace */
    auto setup = [&](Transfer &T) {
        T.NA = NA;
        T.g.L0 = L0;
        T.g.L1 = L1;
        T.g.NA1 = NA1;
        T.g.s0 = L0 > 1 ? -1.0 : (double)BoundC[0];
        T.g.s1 = L1 > 1 ? -1.0 : (double)BoundC[1];
        T.g.e0 = L0 > 1 ? (double)BoundC[0] : 0.0;
        T.g.e1 = L1 > 1 ? (double)BoundC[1] : 0.0;
        SCK(cudaStreamCreateWithFlags(&T.st, cudaStreamNonBlocking));
        /* products up to (2 NA + No) x (NA + No) (the first sweep) */
        RC(smat::dense::gemm_ctx_alloc(T.gm, (int)rows, (int)cols, T.st));
        size_t used = 0;
        std::vector<std::pair<void **, size_t>> want;
        auto buf = [&](auto *&p, size_t n) {
            want.push_back({(void **)&p, used});
            used += (n * sizeof(*p) + 255) / 256 * 256;
        };
        buf(T.M[0], rows * cols);
        buf(T.M[1], rows * cols);
        buf(T.LP, cols * NA);
        buf(T.out, (size_t)(nB + nT) * (nB + nT));
        T.w = form;
        buf(T.w.lud, 32 * 32);
        buf(T.w.prow, T.gm.tc ? 0 : rows * 32);
        buf(T.w.bcol, T.gm.tc ? 0 : cols * 32);
        buf(T.w.mv, 64);
        buf(T.w.perm, NA);
        buf(T.w.rows, T.w.row_bytes);
        buf(T.dinfo, 1);
        if (cudaMalloc(&T.slab, used) != cudaSuccess) {
            cudaGetLastError();
            return smat_fail(SMAT_ENOMEM, "smat_scalc: %zu bytes of device memory", used);
        }
        for (auto &w : want) *w.first = (char *)T.slab + w.second;
        SCK(cudaMemsetAsync(T.dinfo, 0, sizeof(int), T.st));
        return (int)SMAT_OK;
    };
    /* both directions read the ports' modes and the layers' set_V values */
    struct Inputs {
        void *slab = nullptr;
        double2 *XB = nullptr, *XT = nullptr, *V = nullptr;
        ~Inputs() { cudaFree(slab); }
    } in;
    Transfer T;
    RC(setup(T));
    {
        const size_t nx = (size_t)N2 * N2, nv = 6 * (size_t)NA1;
        const bool same = XiB == XiT; /* in whatever order */
        if (cudaMalloc(&in.slab, sizeof(double2) * (nx * (same ? 1 : 2) + nv * nlayers)) != cudaSuccess) {
            cudaGetLastError();
            return smat_fail(SMAT_ENOMEM, "smat_scalc: device memory for the port modes");
        }
        in.XB = static_cast<double2 *>(in.slab);
        in.XT = same ? in.XB : in.XB + nx;
        in.V = in.XT + nx;
        std::vector<std::complex<double>> v, all;
        for (int l = 0; l < nlayers; l++) {
            /* a lossy inner layer is allowed (a warning in the reference) */
            const int comp = scalc_V(meds + (size_t)2 * 6 * NA1 * l, NA1, omega, v);
            if (comp && l == 0) return smat_fail(SMAT_EINVAL, "V is not real in initial_calc");
            if (comp && l == nlayers - 1) return smat_fail(SMAT_EINVAL, "V is not real in final_calc");
            all.insert(all.end(), v.begin(), v.end());
        }
        SCK(cudaMemcpyAsync(in.V, all.data(), sizeof(double2) * all.size(), cudaMemcpyHostToDevice, T.st));
        SCK(cudaMemcpyAsync(in.XB, XiB, sizeof(double2) * nx, cudaMemcpyHostToDevice, T.st));
        if (!same) SCK(cudaMemcpyAsync(in.XT, XiT, sizeof(double2) * nx, cudaMemcpyHostToDevice, T.st));
        SCK(cudaStreamSynchronize(T.st));
    }
    /* the backward pass on a state, stream and host thread of its own, so
     * that the two directions' latency-bound panel factorisations (a cluster
     * of 16 SMs) run beside each other's products; if the second state does
     * not fit the device, the passes run one after the other on the first */
    Transfer T2;
    const bool concurrent = both_ways && setup(T2) == SMAT_OK;
    if (both_ways && !concurrent) smat_clear_error();
    auto port = [N2](const double2 *X, int by_rows) { return by_rows ? Port{X, N2, 1} : Port{X, 1, N2}; };
    const Port PB = port(in.XB, rowsB), PT = port(in.XT, rowsT);
    const int N = nB + nT;
    std::vector<std::complex<double>> Sm((size_t)N * N, 0.0), F01h, B01h, F01b, B01b;
    int rc_back = SMAT_OK;
    std::string msg_back;
    std::thread back;
    if (concurrent) {
        int dev = 0;
        SCK(cudaGetDevice(&dev));
        back = std::thread([&, dev] {
            cudaSetDevice(dev);
            rc_back = one_way(T2, -1, nlayers, in.V, PT, PB, nT, nB, F01b, B01b);
            if (rc_back) msg_back = smat_last_error();
        });
    }
    /* forward: Smat_calc :148-158 */
    const int rc_fwd = one_way(T, 1, nlayers, in.V, PB, PT, nB, nT, F01h, B01h);
    if (back.joinable()) back.join();
    RC(rc_fwd);
    if (rc_back) return smat_fail(rc_back, "%s", msg_back.c_str());
    for (int c = 0; c < N; c++)
        for (int r = 0; r < N; r++)
            Sm[r + (size_t)N * c] = c < nB ? F01h[r + (size_t)N * c] : B01h[r + (size_t)N * (c - nB)];
    if (both_ways) { /* backward: Smat_calc :159-168 */
        if (!concurrent) RC(one_way(T, -1, nlayers, in.V, PT, PB, nT, nB, F01b, B01b));
        for (int c = nB; c < N; c++) {
            for (int r = nB; r < N; r++) Sm[r + (size_t)N * c] = F01b[(r - nB) + (size_t)N * (c - nB)];
            for (int r = 0; r < nB; r++) Sm[r + (size_t)N * c] = F01b[(r + nT) + (size_t)N * (c - nB)];
        }
    }
    if (concurrent) {
        int hinfo2 = 0;
        SCK(cudaMemcpyAsync(&hinfo2, T2.dinfo, sizeof(int), cudaMemcpyDeviceToHost, T2.st));
        SCK(cudaStreamSynchronize(T2.st));
        RC(smat::dense::gemm_ctx_check(T2.gm));
        if (hinfo2 != 0) return smat_fail(SMAT_ENUMERIC, "smat_scalc: singular matrix in the layer transfer (zgesv info)");
        T.solves += T2.solves;
    }
    int hinfo = 0;
    SCK(cudaMemcpyAsync(&hinfo, T.dinfo, sizeof(int), cudaMemcpyDeviceToHost, T.st));
    SCK(cudaStreamSynchronize(T.st));
    RC(smat::dense::gemm_ctx_check(T.gm));
    if (hinfo != 0) return smat_fail(SMAT_ENUMERIC, "smat_scalc: singular matrix in the layer transfer (zgesv info)");
    std::memcpy(S, Sm.data(), sizeof(double2) * Sm.size());
    if (info) {
        /* check_Smat :885-912 */
        double u = 0.0, t = 0.0;
        for (int c = 0; c < N; c++)
            for (int r = 0; r < N; r++) {
                std::complex<double> acc = 0.0;
                for (int k = 0; k < N; k++) acc += std::conj(Sm[k + (size_t)N * r]) * Sm[k + (size_t)N * c];
                if (r == c) acc -= 1.0;
                u += std::norm(acc);
                t += std::norm(Sm[r + (size_t)N * c] - Sm[c + (size_t)N * r]);
            }
        info->unitarity = std::sqrt(u);
        info->transpose = std::sqrt(t);
        info->solves = T.solves;
        info->ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    }
    return SMAT_OK;
}
