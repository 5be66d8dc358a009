/*
 * FP64 split-field FDTD step, bit-identical to the reference main_calc
 * (FDTDcalc/FDTDsplitfieldMetal.c:242-329).
 *
 * One thread per cell and component.  Every floating-point expression keeps
 * the reference's operands and order, and the file is compiled with
 * -fmad=false so that no multiply-add is fused: each result is the same IEEE
 * double the reference computes.  The two sweeps have no intra-sweep
 * dependence (the H sweep reads only E, the E sweep only H), so the
 * reference's sequential cell order does not matter.
 *
 * Deliberate differences that change no value: the boundary factor iBc in
 * {-1, 0, 1} multiplies by sign manipulation instead of a DMUL (bp*x for
 * finite x); products by the coefficients A and B are rounded on the integer
 * pipes (the same bits); an ordinary cell with no special neighbour skips the
 * curl of the aux arrays, which the reference evaluates as a sum of zeros; the 0.0 the
 * reference starts each curl sum from is dropped.  These can only flip the
 * sign of a zero.
 */
#include <cuda_runtime.h>

#include "fdtd_internal.cuh"
#include "imul64.cuh"

namespace smat {

/* bp*x for bp in {-1, 0, 1}: keep/flip masks on the bit pattern */
struct Sel {
    unsigned long long keep, flip;
};

__device__ __forceinline__ Sel make_sel(int bc, bool at_edge)
{
    Sel s{~0ull, 0ull};
    if (at_edge) {
        if (bc == 0) s.keep = 0x8000000000000000ull; /* 0*x = zero with the sign of x */
        else if (bc < 0) s.flip = 0x8000000000000000ull;
    }
    return s;
}

__device__ __forceinline__ double bmul(double x, Sel s)
{
    return __longlong_as_double((long long)((((unsigned long long)__double_as_longlong(x)) & s.keep) ^ s.flip));
}

/* What the curl of component c of a field [3][n3] reads at cell l, a1 = c+1,
 * a2 = c+2: components a1 and a2 of the cell, a2 of its neighbour along a1,
 * a1 of its neighbour along a2 (offsets o1, o2).  A component array holds
 * under 2^31 / 3 entries, so indexes are 32-bit. */
struct Near {
    double h1, h2, n2, n1;
};

/* a load that does not count on the data standing still for the whole kernel */
__device__ __forceinline__ double ld_coherent(const double *p)
{
    double v;
    asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ Near load_near(const double *__restrict__ F, int i1, int i2, int o1, int o2)
{
    return Near{ld_coherent(F + i1), ld_coherent(F + i2), ld_coherent(F + i2 + o1), ld_coherent(F + i1 + o2)};
}

/* The half curls from them.  pl: the term differentiated along axis a1 ("+"
 * half), mi: along a2; wrap: a neighbour lies across a face, with its
 * boundary factor s1, s2. */
template <bool FWD>
__device__ __forceinline__ void curl_near(Near v, bool wrap, Sel s1, Sel s2, double &pl, double &mi)
{
    if (__any_sync(__activemask(), wrap)) {
        v.n2 = bmul(v.n2, s1);
        v.n1 = bmul(v.n1, s2);
    }
    if (!FWD) {
        pl = v.h2 - v.n2;  /* +E - Bp*E(j-1)   (:407) */
        mi = -v.h1 + v.n1; /* -E + Bp*E(j-1)   (:410) */
    } else {
        pl = v.n2 - v.h2;  /* +Bp*H(j+1) - H   (:386) */
        mi = -v.n1 + v.h1; /* -Bp*H(j+1) + H   (:389) */
    }
}

/* Sheet source value of component v at pixel p (main :155-157 or explicit). */
__device__ __forceinline__ double sheet(const Src &s, int pl, int b, int k, bool efield, int v, int p)
{
    if (s.xsrc) return s.xsrc[(efield ? 2 * pl : 0) + v + 2 * p];
    const double *sc = s.sched + 6 * (long long)k + (efield ? 0 : 3);
    const double *w = s.inc + (long long)b * 8 * pl + (efield ? 4 * pl : 0) + 2 * (v + 2 * p);
    const double t = sc[1] * w[0] - (-sc[2]) * w[1]; /* creal(conj(ExpN)*inc) */
    return sc[0] * t;                                /* (2*env) * ... */
}

/* A x for an update factor A = (a)(1/b) of main :118-127.  Where a == b (no
 * loss, no stretch) that is x' * fl(1/x'), which rounds to 1 or to its
 * predecessor 1 - 2^-53, by the division's last bit; and (1 - 2^-53) x rounds
 * to the double next below |x| for every x above the smallest normal number
 * (x - x 2^-53 lies more than half a unit of the last place below x, or at
 * the next number itself where x is a power of two), to x for x at or below
 * it, for zeros, infinities and NaNs.  So for those two factors the product
 * is a subtraction on the bits, off the FP64 pipe. */
__device__ __forceinline__ double amul(double A, double x)
{
    const unsigned long long near1 = (unsigned long long)__double_as_longlong(A) - 0x3fefffffffffffffull;
    if (__any_sync(__activemask(), near1 > 1ull)) return A * x; /* a branch of the whole warp: no DMUL issued for it */
    const unsigned long long u = (unsigned long long)__double_as_longlong(x), lo = 0x0010000000000001ull;
    const bool dec = near1 == 0ull && (u & 0x7fffffffffffffffull) - lo < 0x7ff0000000000000ull - lo;
    return __longlong_as_double((long long)(u - (dec ? 1ull : 0ull)));
}

__device__ __forceinline__ int monitor_index64(const Dft &d, int j2)
{
    int q = -1;
#pragma unroll
    for (int i = 0; i < MAX_PLANES; i++)
        if (i < d.nq && d.planes[i] == j2) q = i;
    return q;
}

__device__ __forceinline__ double *ring64_at(const Dft &d, int pl, int b, int k, int q, int v)
{
    return d.ring64 + ((((long long)b * d.ringK + k % d.ringK) * d.nq + q) * 4 + v) * (long long)pl;
}

/* Component c of a cell of class 'h', 'e' or 'b' in a sweep: frozen (the H of
 * an 'e' cell, the E of an 'h' cell), else the stable form, which reads the
 * main array only and takes the backward difference also of H (:277-283,
 * :308-314).  f: its main slot; returns the new one.  Out of line: such cells
 * are rare. */
template <bool EF>
__device__ __noinline__ double metal_cell(const P64 &p, int cls, int b, int c, int j2, int px, double f)
{
    if (cls == (EF ? CLS_H : CLS_E)) return f;
    const Geo &g = p.g;
    const int n3 = (int)g.n3, l = px + g.pl * j2, a = p.addr[l];
    const int j[3] = {px % g.L0, px / g.L0, j2}, L[3] = {g.L0, g.L1, g.L2}, step[3] = {1, g.L0, g.pl};
    int o[3];
    Sel s[3];
    bool wrap = false;
    for (int x = 0; x < 3; x++) {
        const bool e = j[x] == 0;
        o[x] = (e ? L[x] - 1 : -1) * step[x];
        s[x] = make_sel(g.bc[x], e);
        wrap |= e;
    }
    const int a1 = (c + 1) % 3, a2 = (c + 2) % 3;
    double pl, mi;
    curl_near<false>(load_near((EF ? p.H : p.E) + (long long)b * 3 * n3, a1 * n3 + l, a2 * n3 + l, o[a1], o[a2]), wrap,
                     s[a1], s[a2], pl, mi);
    const double W = pl + mi;
    double *x = (EF ? p.Ea : p.Ha) + ((long long)b * 3 + c) * (p.lnotn + 1) + a;
    const double *ca = p.ca + (long long)(EF ? 6 + c : c) * p.lnotn + a;
    double v = *x;
    f += 0.5 * v;
    v = ca[0] * v + ca[3LL * p.lnotn] * (EF ? W : -W);
    f += 0.5 * v;
    *x = v;
    return f;
}

/* One sweep: EF = false H from E (main_calc :255-286), EF = true E from H
 * (:287-317).
 *
 * Two things bound it.  The FP64 pipe runs 1.7 operations a clock and SM
 * (measured), a warp's instruction holding it for 19 clocks however few of
 * its lanes take part: an ordinary cell costs 12 additions, a split cell 26,
 * an ordinary cell next to a split one 21 (products by B and A are taken off
 * it, imul and amul).  So what counts is warps whose cells take one path: with
 * 32 consecutive x in a warp every warp at an x face ran two or three paths;
 * here the cells of a plane are taken in the order p.ord of the host: the
 * columns x that lie in a PML, row by row, then the columns next to one in
 * the direction of this sweep's differences, column by column, then the
 * others, row by row.  And latency, of the loads and of the FP64 pipe (67
 * clocks): a thread takes one component of a cell, a block's three warps the
 * three components of 32 cells, which share the loaded lines in L1, so that
 * 39 warps fit an SM where 16 of whole cells did; a sweep is launched beside the
 * one before (launch_after) and has its coefficients and the addresses of its
 * aux slots by the time that one ends; and the aux slots, which fewer cells
 * have, are asked for before the main ones (after them: the same on large
 * grids, but 24 x 24 x 40 8.0 us a step instead of 6.0, the dependents falling
 * into step with one another).  Dense aux slots, which need no addresses, took
 * 48 bytes a cell and excitation more and gained nothing (119 us a step at
 * 96^3, now 111).  Excitations are fastest in the grid: the coefficients are
 * shared through L2.
 *
 * us a step of two sweeps, run after run: 96^3 cube (12-cell PML) 111, 130 x 98
 * x 81 bend of two excitations 243, 24 x 20 x 40 guide 5.2, where one thread per
 * cell with 32 consecutive x a warp and every operation on the FP64 pipe took
 * 170, 422 and 10.  Blocks of 32 cells rather than 64 or 128: 3 % and 10 % on the
 * cube, 10 % and 30 % on the guide, whose plane fills 15 of them.  13 resident
 * blocks (48 registers): 10 and 15 are within 7 %. */
template <bool EF>
__global__ void __launch_bounds__(96, 13) k_sweep64(const P64 p, const int rel)
{
    const Geo &g = p.g;
    const int b = blockIdx.x % p.batch, i = blockIdx.x / p.batch * 32 + threadIdx.x;
    const int j2 = blockIdx.y, c = threadIdx.y;
    if (i >= g.pl) return;
    const int2 od = p.ord[(EF ? g.pl : 0) + i]; /* pixel; 1: wraps along x, 2: along y */
    const int px = od.x, n3 = (int)g.n3, l = px + g.pl * j2;
    const bool ex = od.y & 1, ey = od.y & 2, ez = j2 == (EF ? g.L2 - 1 : 0);
    const int sd = EF ? 1 : -1;
    const int ox = ex ? -sd * (g.L0 - 1) : sd, oy = (ey ? -sd * (g.L1 - 1) : sd) * g.L0;
    const int oz = (ez ? -sd * (g.L2 - 1) : sd) * g.pl;
    /* axes a1 = c+1, a2 = c+2 */
    const int o1 = c == 0 ? oy : c == 1 ? oz : ox, o2 = c == 0 ? oz : c == 1 ? ox : oy;
    const bool w1 = c == 0 ? ey : c == 1 ? ez : ex, w2 = c == 0 ? ez : c == 1 ? ex : ey;
    const Sel s1 = make_sel(g.bc[c == 2 ? 0 : c + 1], w1), s2 = make_sel(g.bc[c == 0 ? 2 : c - 1], w2);
    const int i0 = c * n3 + l, i1 = (c == 2 ? 0 : c + 1) * n3 + l, i2 = (c == 0 ? 2 : c - 1) * n3 + l;
    const long long bo = (long long)b * 3 * n3;
    const int as = p.lnotn + 1;
    const long long ao = (long long)b * 3 * as;
    double *__restrict__ F = (EF ? p.E : p.H) + bo, *__restrict__ Fa = (EF ? p.Ea : p.Ha) + ao + (long long)c * as;
    const double *__restrict__ G = (EF ? p.H : p.E) + bo;
    const double *__restrict__ Ga1 = (EF ? p.Ha : p.Ea) + ao + (long long)(c == 2 ? 0 : c + 1) * as;
    const double *__restrict__ Ga2 = (EF ? p.Ha : p.Ea) + ao + (long long)(c == 0 ? 2 : c - 1) * as;
    const double *__restrict__ cm = p.cm + (EF ? 6 : 0) * g.n3, *__restrict__ ca = p.ca + (EF ? 6 + c : c) * (long long)p.lnotn;
    const int fl = p.flags[l], cls = fl & 7;
    const bool aux = cls == CLS_A || (fl & (EF ? FL_FWD : FL_BWD)); /* the curl takes aux slots in */
    const double A = cm[i0], B = cm[3 * g.n3 + i0];
    double Aa, Ba;
    int a = 0, n1 = 0, n2 = 0; /* aux slots of the cell and of its neighbours along a1, a2 */
    if (aux) {
        a = p.addr[l];
        n1 = p.addr[l + o1];
        n2 = p.addr[l + o2];
    }
    if (cls == CLS_A) {
        Aa = ca[a];
        Ba = ca[3LL * p.lnotn + a];
    }
    prior_done();
    next_may_start();
    double f = F[i0];
    double fa = 0.0;
    Near va;
    if (aux) {
        fa = Fa[a];
        va = Near{ld_coherent(Ga1 + a), ld_coherent(Ga2 + a), ld_coherent(Ga2 + n1), ld_coherent(Ga1 + n2)};
    }
    const Near v = load_near(G, i1, i2, o1, o2);
    double pl, mi, pa, ma;
    if (cls == CLS_N) {
        curl_near<EF>(v, w1 | w2, s1, s2, pl, mi);
        double W = pl + mi;
        if (j2 == p.s.iI[b] && c < 2) {
            const double t = p.s.sgn[b] * sheet(p.s, g.pl, b, *p.s.base + rel, !EF, 1 - c, px);
            W = c == 0 ? W + t : W - t;
        }
        f = amul(A, f) + imul<!EF>(B, W);
        if (aux) {
            curl_near<EF>(va, w1 | w2, s1, s2, pa, ma);
            f += imul<!EF>(B, pa + ma);
        }
    } else if (cls == CLS_A) {
        curl_near<EF>(v, w1 | w2, s1, s2, pl, mi);
        curl_near<EF>(va, w1 | w2, s1, s2, pa, ma);
        const double h = amul(A, f) + imul<!EF>(B, pl);
        f = h + imul<!EF>(B, pa);
        const double x = amul(Aa, fa) + imul<!EF>(Ba, mi);
        fa = x + imul<!EF>(Ba, ma);
        Fa[a] = fa;
    } else {
        f = metal_cell<EF>(p, cls, b, c, j2, px, f);
    }
    F[i0] = f;
    const int q = monitor_index64(p.d, j2);
    if (q >= 0 && c < 2 && p.d.ring64) {
        /* a plane through the PML (allowed for general schedules only; the
         * reference exits, :320) samples the total field main + aux */
        ring64_at(p.d, g.pl, b, *p.s.base + rel, q, (EF ? 2 : 0) + c)[px] = cls == CLS_A ? f + fa : f;
    }
}

/* running DFT on the monitor planes (main_calc :318-328), FP64 accumulators:
 * the samples of `count` steps ending at *base + rel_end, from the ring the
 * sweeps fill, folded in step by step.  acc += phase * x computed as (re +=
 * pr*x, im += pi*x), the value of the reference's complex product with a real
 * factor, in the reference's order: the same bits as one pass over the
 * accumulators every step, at 1/32 of their traffic and launches.  A thread
 * takes one pixel and component of one plane and excitation and every
 * gridDim.z / batch-th frequency.  96^3 cube, 11 wavelengths, 2 planes: 6.6 us
 * a step (half of it the FP64 pipe's additions), from 32 us.  RING false: a plan
 * without the ring (no room for it), one step. */
template <bool RING>
__global__ void __launch_bounds__(128) k_flush64(const P64 p, const int rel_end, const int count)
{
    const int px = blockIdx.x * 128 + threadIdx.x, q = blockIdx.y >> 2, v = blockIdx.y & 3;
    const int b = blockIdx.z % p.batch, f0 = blockIdx.z / p.batch, nf = gridDim.z / p.batch;
    const Geo &g = p.g;
    const Dft &d = p.d;
    if (px >= g.pl) return;
    const int k0 = *p.s.base + rel_end - count;
    const int qs = monitor_index64(d, d.planes[q]); /* the slot the sweeps fill, where a plane is listed twice */
    double now = 0.0;
    if (!RING) { /* count is 1: from the fields, as the sweeps sample them */
        const long long l = px + (long long)g.pl * d.planes[q], a = p.addr[l], as = p.lnotn + 1;
        now = (v < 2 ? p.H : p.E)[(3LL * b + v % 2) * g.n3 + l];
        if ((p.flags[l] & 7) == CLS_A) now += (v < 2 ? p.Ha : p.Ea)[(3LL * b + v % 2) * as + a];
    }
    for (int f = f0; f < d.nfreq; f += nf) {
        double *acc = d.acc + 2 * (((((long long)b * d.nfreq + f) * d.nq + q) * 4 + v) * g.pl + px);
        double re = acc[0], im = acc[1];
#pragma unroll 4
        for (int s = 0; s < count; s++) {
            const double x = RING ? ring64_at(d, g.pl, b, k0 + s, qs, v)[px] : now;
            const double *ph = (d.xphase ? d.xphase : d.phase + 4 * ((long long)(k0 + s) * d.nfreq + f)) + (v < 2 ? 0 : 2);
            re += imul(ph[0], x);
            im += imul(ph[1], x);
        }
        acc[0] = re;
        acc[1] = im;
    }
}

__global__ void k_bump(int *base, int by)
{
    *base += by;
}

__global__ void k_set(int *base, int value)
{
    *base = value;
}

/* max |x| as the bit pattern of a non-negative double (NaN sorts above Inf) */
__global__ void k_maxabs(const void *x, long long n, int is_double, unsigned long long *out)
{
    unsigned long long m = 0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const double v = is_double ? ((const double *)x)[i] : (double)((const float *)x)[i];
        const unsigned long long bits = (unsigned long long)__double_as_longlong(fabs(v));
        m = bits > m ? bits : m;
    }
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long t = __shfl_down_sync(0xffffffffu, m, o);
        m = t > m ? t : m;
    }
    if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

template <bool EF> static void launch_sweep64(const P64 &p, int rel, cudaStream_t st)
{
    const dim3 grid((p.g.pl + 31) / 32 * p.batch, p.g.L2), block(32, 3);
    launch_after(k_sweep64<EF>, grid, block, 0, st, p, rel);
}

void launch_h64(const P64 &p, int rel, cudaStream_t st) { launch_sweep64<false>(p, rel, st); }

void launch_e64(const P64 &p, int rel, cudaStream_t st) { launch_sweep64<true>(p, rel, st); }

/* the frequencies are spread over as many threads as fill the GPU's warps
 * (a chain of two operations a step and frequency, 67 clocks each) */
void launch_flush64(const P64 &p, int rel_end, int count, cudaStream_t st)
{
    if (p.d.nfreq <= 0 || p.d.nq <= 0 || count <= 0) return;
    const int nb = (p.g.pl + 127) / 128, used = nb * p.d.nq * 4 * p.batch;
    const int fill = 12 * plan::sm_count(); /* 12 blocks an SM */
    int nf = used >= fill ? 1 : (fill + used - 1) / used;
    if (nf > p.d.nfreq) nf = p.d.nfreq;
    (p.d.ring64 ? k_flush64<true> : k_flush64<false>)<<<dim3(nb, p.d.nq * 4, p.batch * nf), 128, 0, st>>>(p, rel_end, count);
}

void launch_bump(int *base, int by, cudaStream_t st) { k_bump<<<1, 1, 0, st>>>(base, by); }

void launch_set(int *base, int value, cudaStream_t st) { k_set<<<1, 1, 0, st>>>(base, value); }

void launch_maxabs(const void *x, long long n, int is_double, double *out, cudaStream_t st)
{
    k_maxabs<<<608, 256, 0, st>>>(x, n, is_double, (unsigned long long *)out);
}

} // namespace smat
