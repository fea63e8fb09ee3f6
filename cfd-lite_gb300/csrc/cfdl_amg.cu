// cfdl_amg.cu -- aggregation-AMG preconditioned CG for the pressure
// correction (FP64), and the mixed-precision form (FP32 AMG-PCG inner solve,
// FP64 residual and refinement).
//
// The reference solves the pressure correction with 4-block Jacobi / SSOR
// sweeps (multi_subdomain_solver, src/modules/mod_solver.f90:124-189), whose
// convergence degrades with the mesh size.  Here CG on the same singular
// Neumann system (right-hand side projected to zero mean) is preconditioned
// by one V-cycle of aggregation multigrid:
//   level l -> l+1   two damped-Jacobi sweeps, residual restricted by summing
//                    over each aggregate (P^T, P piecewise constant);
//   coarsest level   dense inverse of (A_L + c 11^T), which is A_L's
//                    pseudo-inverse on zero-sum right-hand sides;
//   level l+1 -> l   prolongation (injection, scaled by kOverCorrect) added
//                    in place, then two damped-Jacobi sweeps;
//   small levels     a case's levels of at most kTailRows rows and its
//                    coarsest solve run on one cluster of CTAs (k_v_tail).
// Pre- and post-smoothing match, so the preconditioner is symmetric and
// positive semi-definite, as CG requires.  The coarse operators are rebuilt
// at every pressure solve from the current coefficients (A_c = P^T A P).
#include "cfdl_amg.h"
#include "cfdl_device.cuh"
#include "cfdl_par.h"
#include <algorithm>
#include <cooperative_groups.h>
#include <new>

namespace cfdl {
namespace {

// Damped-Jacobi weights of a level's two smoothing sweeps.  Pre-smoothing
// runs the kOmega sweep from zero (k_v_jac0) and then the kOmega2 sweep;
// post-smoothing runs the kOmega sweep from the prolongated value and then
// the kOmega2 sweep.  Either way the error propagator is
// (I - kOmega2 D^-1 A)(I - kOmega D^-1 A), the same polynomial in D^-1 A
// before and after the coarse correction, so the V-cycle stays symmetric.
// rd = kOmega / D is stored per level; the second sweep scales it by
// kOmega2 / kOmega.  The two weights are the reciprocals of the roots of the
// degree-2 Chebyshev polynomial on [0.6, 2] (D^-1 A of these zero-row-sum
// M-matrices has its spectrum in [0, 2]): the pair damps the upper part of
// the spectrum more than two sweeps of one weight.  Measured on the 128^3
// cavity against 0.8 / 0.8: 2% less time per outer iteration, FP64 and
// mixed alike (Chebyshev on [0.5, 2] 1%, [0.4, 2] 1% more; a coarse
// over-correction of 2 instead of 3: 22% more).
constexpr double kOverCorrect = 3.0;   // scaling of the prolongated coarse correction
constexpr int kG = 8;                  // lanes per row on the small coarse levels
constexpr int kGroupedRows = 65536;    // levels below this many rows (per case) run grouped
constexpr int kTailRows = 2048;        // a case's levels at or below this many rows run in its V-cycle tail
enum { CNT_A0 = 9, CNT_A1, CNT_A2, CNT_A3, CNT_A4, CNT_A5 };

template <class T> struct LP {
    int n, W;
    const int *nb;
    const T *a, *dg, *rd;   // rd = omega / diagonal (the damped Jacobi scaling)
    T *r, *z, *t;
    const int *len;         // coarse levels: valid slots of each row, packed first (null on the mesh level)
    const short *nb16;      // mesh level: the neighbours as 16-bit offsets (CaseDev::nb16), or null
    int ld;                 // stride of a's and nb16's planes on the FP32 mesh level (n elsewhere)
};

template <class T> __device__ __forceinline__ LP<T> level(const CaseDev &C, int l);
template <> __device__ __forceinline__ LP<double> level<double>(const CaseDev &C, int l) {
    if (l == 0) return {C.ne, C.W, C.hf_nb, C.anb_p, C.ap_p, C.rap_p, C.kr, C.ks, C.ksh, nullptr, nullptr, C.ne};
    const AmgLevelDev &L = C.lev[l - 1];
    return {L.n, L.W, L.nb, L.a, L.dg, L.rd, L.r, L.z, L.t, L.len, nullptr, L.n};
}
template <> __device__ __forceinline__ LP<float> level<float>(const CaseDev &C, int l) {
    if (l == 0) return {C.ne, C.W, C.hf_nb, C.fanb_p, C.fdiag_p, C.frap_p, C.fr, C.fz, C.ft, nullptr, C.nb16, C.ld32};
    const AmgLevelDev &L = C.lev[l - 1];
    return {L.n, L.W, L.nb, L.a32, L.dg32, L.rd32, L.r32, L.z32, L.t32, L.len, nullptr, L.n};
}

// (A x)_i at a level; neighbours outside [0, n) (halos, padding) are skipped
template <class T> __device__ __forceinline__ T amul(const LP<T> &P, const T *x, int i) {
    T y[1];
    ell_row<1, T>(P.nb, P.a, P.dg[i], x, 0, P.n, P.W, i, y);
    return y[0];
}
// A thread's rows of a wide tile, two per step: rows i0 and i1, with ok0 and
// ok1 false past the tile's end.  The CG kernels issue both rows' loads
// before either row's stores: a store holds back every load after it (the
// compiler cannot tell that they do not alias), so one row per step made
// each row its own trip to memory.  Sums still run in row order.
#define FOR_ROW_PAIRS(t)                                                                            \
    for (int j_ = 0, i0 = (t).first + (int)threadIdx.x; j_ < (t).pad; j_ += 2, i0 += 2 * kTile)     \
        if (const int i1 = i0 + kTile, ok0 = i0 < (t).last, ok1 = j_ + 1 < (t).pad && i1 < (t).last; \
            true)

// CG's q = A p (FP64) over a thread's rows of a wide tile, returning its share
// of (p, q), two rows per step
__device__ __forceinline__ double cg_aq_rows(const LP<double> &P, const double *p, double *q, const Tile &t) {
    double v = 0;
    FOR_ROW_PAIRS(t) {
        double q0 = 0, q1 = 0, p0 = 0, p1 = 0;
        // amul's guarded coefficient loads measured faster in these multi-row
        // tiles than the mesh sweeps' eager ones
        if (ok0) { q0 = amul<double>(P, p, i0); p0 = p[i0]; }
        if (ok1) { q1 = amul<double>(P, p, i1); p1 = p[i1]; }
        if (ok0) { q[i0] = q0; v += p0 * q0; }
        if (ok1) { q[i1] = q1; v += p1 * q1; }
    }
    return v;
}
// CG's (r, z), two rows per step; its roundings spelled out (the split form
// has to have them)
__device__ __forceinline__ float cg_rz_rows(const float *r, const float *z, const Tile &t) {
    float v = 0;
    FOR_ROW_PAIRS(t) {
        float r0 = 0, z0 = 0, r1 = 0, z1 = 0;
        if (ok0) { r0 = r[i0]; z0 = z[i0]; }
        if (ok1) { r1 = r[i1]; z1 = z[i1]; }
        if (ok0) v = __fmaf_rn(r0, z0, v);
        if (ok1) v = __fadd_rn(v, __fmul_rn(r1, z1));
    }
    return v;
}
// CG's p = z (first iteration) or z + beta p, two rows per step
template <class T>
__device__ __forceinline__ void cg_p_rows(const T *z, T *p, bool first, T beta, const Tile &t) {
    FOR_ROW_PAIRS(t) {
        T z0 = 0, p0 = 0, z1 = 0, p1 = 0;
        if (ok0) { z0 = z[i0]; if (!first) p0 = p[i0]; }
        if (ok1) { z1 = z[i1]; if (!first) p1 = p[i1]; }
        if (ok0) p[i0] = first ? z0 : z0 + beta * p0;
        if (ok1) p[i1] = first ? z1 : z1 + beta * p1;
    }
}
// CG's x += alpha p; r -= alpha q, returning the share of (r, r), two rows
// per step
template <class T>
__device__ __forceinline__ T cg_x_rows(T *x, const T *p, T *r, const T *q, T a, const Tile &t) {
    T v = 0;
    FOR_ROW_PAIRS(t) {
        T x0 = 0, p0 = 0, r0 = 0, q0 = 0, x1 = 0, p1 = 0, r1 = 0, q1 = 0;
        if (ok0) { x0 = x[i0]; p0 = p[i0]; r0 = r[i0]; q0 = q[i0]; }
        if (ok1) { x1 = x[i1]; p1 = p[i1]; r1 = r[i1]; q1 = q[i1]; }
        if (ok0) { x[i0] = x0 + a * p0; const T rr = r0 - a * q0; r[i0] = rr; v = fma_rn(rr, rr, v); }
        if (ok1) { x[i1] = x1 + a * p1; const T rr = r1 - a * q1; r[i1] = rr; v = fma_rn(rr, rr, v); }
    }
    return v;
}
// Slots of a wide coarse row taken per step, their index, coefficient and
// vector loads issued together (sums stay in slot order): 8 for the FP32
// levels, 4 for FP64, where 8 took the sweeps from 48 to 64 registers and
// measured slower (the FP32 sweeps and tail measured 5-15% faster at 8)
template <class T> __host__ __device__ constexpr int coarse_chunk() { return sizeof(T) == 4 ? 8 : 4; }
// the same on a coarse level, over the row's valid slots only (the padding
// slots would subtract zero terms): kCh slots per step
template <class T> __device__ __forceinline__ T amul_coarse(const LP<T> &P, const T *x, int i) {
    if (P.W == 6 || P.W == 4 || !P.len) return amul<T>(P, x, i);
    constexpr int kCh = coarse_chunk<T>();
    const int len = P.len[i];
    T y = P.dg[i] * x[i];
    for (int k0 = 0; k0 < len; k0 += kCh) {
        int jj[kCh];
        T ak[kCh], xv[kCh];
#pragma unroll
        for (int u = 0; u < kCh; u++) jj[u] = k0 + u < len ? P.nb[(k0 + u) * P.n + i] : -1;
#pragma unroll
        for (int u = 0; u < kCh; u++) {
            const bool ok = (unsigned)jj[u] < (unsigned)P.n;
            ak[u] = ok ? P.a[(k0 + u) * P.n + i] : (T)0;
            if (!ok) jj[u] = i;
        }
#pragma unroll
        for (int u = 0; u < kCh; u++) xv[u] = x[jj[u]];
#pragma unroll
        for (int u = 0; u < kCh; u++) y -= ak[u] * xv[u];
    }
    return y;
}

// The first W slots of row i: neighbour j[k] (i itself for a slot outside
// [0, n)) and coefficient c[k] (0 there).  The coefficient's address does not
// depend on the index, so both loads are issued together: a load guarded by
// the index would wait for it, a second memory latency in the row's chain.
// kGuard: the row has P.W <= W slots (the mesh level, W = kMaxW); slots past
// P.W are not read.  kEager false: the coefficient load waits for the index
// (the coarse levels' kernels, where that form measured faster).
template <int W, class T, bool kGuard, bool kEager = true>
__device__ __forceinline__ void row_slots(const LP<T> &P, int i, int (&j)[W], T (&c)[W]) {
#pragma unroll
    for (int k = 0; k < W; k++) {
        const bool in = !kGuard || k < P.W;
        const int jj = in ? P.nb[k * P.n + i] : -1;
        const bool ok = (unsigned)jj < (unsigned)P.n;
        j[k] = ok ? jj : i;
        if (kEager) {
            const T ak = in ? P.a[k * P.n + i] : (T)0;
            c[k] = ok ? ak : (T)0;
        } else {
            c[k] = ok ? P.a[k * P.n + i] : (T)0;
        }
    }
}

// s + sum_j a_ij x_j over the row's couplings inside the level (the ELL values
// are the off-diagonal magnitudes: A = D - offdiag)
template <int W, class T, bool kGuard = false, bool kEager = true>
__device__ __forceinline__ T offsum_w(const LP<T> &P, const T *x, int i, T s = 0) {
    int j[W];
    T c[W];
    row_slots<W, T, kGuard, kEager>(P, i, j, c);
    T xj[W];
#pragma unroll
    for (int k = 0; k < W; k++) xj[k] = x[j[k]];
#pragma unroll
    for (int k = 0; k < W; k++) s += c[k] * xj[k];
    return s;
}

// The FP64 mesh level (level 0): at most kMaxW slots a row, every width on the
// short fixed-width paths (no wide-row code in the kernels that use these)
__device__ __forceinline__ double offsum_mesh(const LP<double> &P, const double *x, int i, double s) {
    if (P.W == 6) return offsum_w<6, double, false>(P, x, i, s);
    if (P.W == 4) return offsum_w<4, double, false>(P, x, i, s);
    return offsum_w<kMaxW, double, true>(P, x, i, s);
}

// The FP32 mesh level takes its rows two at a time, i (even) and i + 1, with
// 8-byte coefficient and 4-byte offset (k16; else 8-byte index) loads.  One row
// per thread was bound by the load instructions, not by the bytes: at 128^3
// two rows per thread move the same bytes in 18.7 instead of 24.7 us, and with
// int32 indices in 23.1 instead of 27.1; the FP64 sweep is bound by its FP64
// instructions and gains nothing.  Planes and vectors have an even length
// (CaseDev::ld32); the padding row of an odd level has no couplings.
template <int W, bool k16, bool kGuard>
__device__ __forceinline__ void pair_slots(const LP<float> &P, int i, int (&j)[2][W], float (&c)[2][W]) {
    const int n = P.n;
#pragma unroll
    for (int k = 0; k < W; k++) {
        const bool in = !kGuard || k < P.W;
        int j0 = -1, j1 = -1;
        float2 a = make_float2(0.f, 0.f);
        if (in) {
            if (k16) {
                const short2 d = *(const short2 *)&P.nb16[k * P.ld + i];
                j0 = d.x == kNb16None ? -1 : i + d.x;
                j1 = d.y == kNb16None ? -1 : i + 1 + d.y;
            } else if ((n & 1) == 0) {
                const int2 d = *(const int2 *)&P.nb[k * n + i];
                j0 = d.x;
                j1 = d.y;
            } else {                                       // odd rows: the planes are not aligned to pairs
                j0 = P.nb[k * n + i];
                j1 = i + 1 < n ? P.nb[k * n + i + 1] : -1;
            }
            a = *(const float2 *)&P.a[k * P.ld + i];
        }
        const bool ok0 = (unsigned)j0 < (unsigned)n, ok1 = (unsigned)j1 < (unsigned)n;
        j[0][k] = ok0 ? j0 : i;
        j[1][k] = ok1 ? j1 : i + 1;
        c[0][k] = ok0 ? a.x : 0.f;
        c[1][k] = ok1 ? a.y : 0.f;
    }
}
// the rows' off-diagonal sums of x (kRd: of rd[j] x[j], the product k_v_jac0
// would store: the same multiplication, so the same values)
template <int W, bool k16, bool kGuard, bool kRd>
__device__ __forceinline__ float2 pair_offsum(const LP<float> &P, const float *x, int i) {
    int j[2][W];
    float c[2][W], v[2][W];
    pair_slots<W, k16, kGuard>(P, i, j, c);
#pragma unroll
    for (int k = 0; k < W; k++)
#pragma unroll
        for (int u = 0; u < 2; u++) v[u][k] = kRd ? P.rd[j[u][k]] * x[j[u][k]] : x[j[u][k]];
    float2 s = make_float2(0.f, 0.f);
#pragma unroll
    for (int k = 0; k < W; k++) { s.x += c[0][k] * v[0][k]; s.y += c[1][k] * v[1][k]; }
    return s;
}
// the rows of A x
template <int W, bool k16, bool kGuard>
__device__ __forceinline__ float2 pair_amul(const LP<float> &P, const float *x, int i) {
    int j[2][W];
    float c[2][W], v[2][W];
    pair_slots<W, k16, kGuard>(P, i, j, c);
#pragma unroll
    for (int k = 0; k < W; k++)
#pragma unroll
        for (int u = 0; u < 2; u++) v[u][k] = x[j[u][k]];
    const float2 xi = *(const float2 *)&x[i], d = *(const float2 *)&P.dg[i];
    // d x_i - c_0 x_0 - c_1 x_1 - ...; its roundings are spelled out, so they do
    // not depend on which product the compiler would contract
    float2 s = make_float2(__fmaf_rn(d.x, xi.x, -__fmul_rn(c[0][0], v[0][0])), __fmaf_rn(d.y, xi.y, -__fmul_rn(c[1][0], v[1][0])));
#pragma unroll
    for (int k = 1; k < W; k++) { s.x = __fmaf_rn(-c[0][k], v[0][k], s.x); s.y = __fmaf_rn(-c[1][k], v[1][k], s.y); }
    return s;
}
// one row of A x, with pair_amul's roundings
template <int W, bool k16, bool kGuard>
__device__ __forceinline__ float row_amul(const LP<float> &P, const float *x, int i) {
    int j[W];
    float c[W], v[W];
#pragma unroll
    for (int k = 0; k < W; k++) {
        int jj = -1;
        float a = 0.f;
        if (!kGuard || k < P.W) {
            if (k16) { const int d = P.nb16[k * P.ld + i]; jj = d == (int)kNb16None ? -1 : i + d; }
            else jj = P.nb[k * P.n + i];
            a = P.a[k * P.ld + i];
        }
        const bool ok = (unsigned)jj < (unsigned)P.n;
        j[k] = ok ? jj : i;
        c[k] = ok ? a : 0.f;
    }
#pragma unroll
    for (int k = 0; k < W; k++) v[k] = x[j[k]];
    float s = __fmaf_rn(P.dg[i], x[i], -__fmul_rn(c[0], v[0]));
#pragma unroll
    for (int k = 1; k < W; k++) s = __fmaf_rn(-c[k], v[k], s);
    return s;
}
template <bool k16> __device__ __forceinline__ float row_amul_mesh(const LP<float> &P, const float *x, int i) {
    if (P.W == 6) return row_amul<6, k16, false>(P, x, i);
    if (P.W == 4) return row_amul<4, k16, false>(P, x, i);
    return row_amul<kMaxW, k16, true>(P, x, i);
}
template <bool k16, bool kRd = false> __device__ __forceinline__ float2 pair_offsum_mesh(const LP<float> &P, const float *x, int i) {
    if (P.W == 6) return pair_offsum<6, k16, false, kRd>(P, x, i);
    if (P.W == 4) return pair_offsum<4, k16, false, kRd>(P, x, i);
    return pair_offsum<kMaxW, k16, true, kRd>(P, x, i);
}
template <bool k16> __device__ __forceinline__ float2 pair_amul_mesh(const LP<float> &P, const float *x, int i) {
    if (P.W == 6) return pair_amul<6, k16, false>(P, x, i);
    if (P.W == 4) return pair_amul<4, k16, false>(P, x, i);
    return pair_amul<kMaxW, k16, true>(P, x, i);
}
// Valid slots of row i: a coarse row's couplings are packed in its first
// len[i] slots (the rest is padding up to the level's widest row, W).
template <class T> __device__ __forceinline__ int row_len(const LP<T> &P, int i) {
    return P.len ? P.len[i] : P.W;
}

template <class T> __device__ __forceinline__ T offsum(const LP<T> &P, const T *x, int i) {
    if (P.W == 6) return offsum_w<6, T, false, false>(P, x, i);
    if (P.W == 4) return offsum_w<4, T, false, false>(P, x, i);
    constexpr int kCh = coarse_chunk<T>();
    // wide coarse rows: kCh slots per step, loads issued together,
    // up to the row's own length (the padding would add zero terms)
    T s = 0;
    const int len = row_len(P, i);
    for (int k0 = 0; k0 < len; k0 += kCh) {
        int jj[kCh];
        T c[kCh], xv[kCh];
#pragma unroll
        for (int u = 0; u < kCh; u++) jj[u] = k0 + u < len ? P.nb[(k0 + u) * P.n + i] : -1;
#pragma unroll
        for (int u = 0; u < kCh; u++) {
            const bool ok = (unsigned)jj[u] < (unsigned)P.n;
            c[u] = ok ? P.a[(k0 + u) * P.n + i] : (T)0;
            xv[u] = x[ok ? jj[u] : i];
        }
#pragma unroll
        for (int u = 0; u < kCh; u++) s += c[u] * xv[u];
    }
    return s;
}
// damped Jacobi sweep from x: x + w D^-1 (r - A x) = (1 - w) x + (w/D)(r + offsum);
// kSweep 1 with w = kOmega (wrd = rd as stored), 2 with w = kOmega2
template <class T, int kSweep = 2> __device__ __forceinline__ T jacobi_step(T x, T r, T wrd, T off) {
    if (kSweep == 1) return (T)(1.0 - kOmega) * x + wrd * (r + off);
    return (T)(1.0 - kOmega2) * x + (wrd * (T)(kOmega2 / kOmega)) * (r + off);
}

// the same on the FP32 mesh level, its roundings spelled out (as pair_amul's)
template <int kSweep> __device__ __forceinline__ float pair_jacobi(float x, float r, float wrd, float off) {
    const float b = __fadd_rn(r, off);
    if (kSweep == 1) return __fmaf_rn((float)(1.0 - kOmega), x, __fmul_rn(wrd, b));
    return __fmaf_rn(__fmul_rn(wrd, (float)(kOmega2 / kOmega)), b, __fmul_rn((float)(1.0 - kOmega2), x));
}

__device__ __forceinline__ bool pactive(const CaseDev &C) { return C.sc->active_p != 0; }
__device__ __forceinline__ bool mactive(const CaseDev &C) { return C.sc->active32 != 0; }

// ------------------------------------------------------------ Galerkin
// Coarse row I of A_c = P^T A P for unsmoothed aggregation (k_amg_galg below):
// each off-diagonal slot is the sum of the fine couplings between aggregate I
// and its neighbour, in a fixed order.  The pressure-correction matrix has
// zero row sums (calc_coef_p: ap = sum of anb), and so has A_c, whose
// diagonal is therefore the sum of its row's off-diagonal couplings -- no
// pass over the aggregate's members or its internal couplings.

// prep_row of every row of a matrix that came from elsewhere (k_coef_p_mat does
// it for its own)
__global__ void __launch_bounds__(kTile) k_amg_prep0(const CaseDev *__restrict__ cases, const Tile *__restrict__ tiles) {
    CFDL_PDL_WAIT();
    const Tile t = tiles[blockIdx.x];
    const CaseDev &C = cases[t.c];
    const int i = t.first + (int)threadIdx.x;
    if (i >= t.last || C.sc->halted) return;
    // the row's loads before its stores (a store holds back the loads after it)
    const double ap = C.ap_p[i];
    double a[kMaxW];
#pragma unroll
    for (int k = 0; k < kMaxW; k++) a[k] = C.precision >= 1 && k < C.W ? C.anb_p[k * C.ne + i] : 0.0;
    prep_row(C, i, ap, a);
}

// Dense inverse of A_L + c 11^T at each case's coarsest level (one CTA per
// case, Gauss-Jordan; the matrix is SPD, no pivoting).  Each thread holds its
// entries in registers; per pivot k their owners publish the pivot row and
// column, the first n threads scale the row (R[k] = 1/p, one division per
// column), and every thread updates its own entries from Q and R.  The FP64
// pipe sets the pace: n^2/32 warp instructions of 16 clocks per pivot, behind
// two barriers and a quotient; 256, 512 and 1024 threads measure the same.
// With the matrix in shared memory the 37-row inverse of the 128^3 cavity
// took 77 us and the 8-row one of the 24^3 cavity 17; this takes 55 and 11.7.
constexpr int kInvThreads = 256;
__global__ void __launch_bounds__(kInvThreads) k_amg_coarse_inv(const CaseDev *__restrict__ cases, int ncases) {
    CFDL_PDL_WAIT();
    const int c = blockIdx.x;
    if (c >= ncases) return;
    const CaseDev &C = cases[c];
    if (C.precond != 1 || C.sc->halted) return;
    __shared__ double M[kAmgCoarsest * kAmgCoarsest];      // the matrix as it is assembled
    __shared__ double R[kAmgCoarsest], row[2][kAmgCoarsest], col[2][kAmgCoarsest], dg[kAmgCoarsest];
    const LP<double> P = level<double>(C, C.nlev);
    const int n = P.n, tid = (int)threadIdx.x;
    if (n > kAmgCoarsest) return;   // cannot happen: the builder coarsens to <= kAmgCoarsest
    if (tid < n) dg[tid] = P.dg[tid];
    __syncthreads();
    double dmax = 0.0;
    for (int i = 0; i < n; i++) dmax = fmax(dmax, fabs(dg[i]));
    const double cc = dmax > 0.0 ? dmax / n : 1.0;
    constexpr int kPer = kAmgCoarsest * kAmgCoarsest / kInvThreads;
    for (int e = tid; e < n * n; e += kInvThreads) M[e] = cc + (e / n == e % n ? dg[e / n] : 0.0);
    __syncthreads();
    if (C.nlev > 0) {
        for (int s = tid; s < P.W * n; s += kInvThreads) { // a coarse row has one slot per neighbour
            const int e = s % n, j = P.nb[s];
            const double a = P.a[s];
            if (j >= 0 && j < n) M[e * n + j] -= a;
        }
    } else if (tid < n) {                                  // cells of a mesh may share several faces: a thread to a row
        for (int k = 0; k < P.W; k++) {
            const int j = P.nb[k * n + tid];
            if (j >= 0 && j < n) M[tid * n + j] -= P.a[k * n + tid];
        }
    }
    __syncthreads();
    double m[kPer];
    short ei[kPer], ej[kPer];
    const int used = (n * n + kInvThreads - 1) / kInvThreads;
#pragma unroll
    for (int q = 0; q < kPer; q++) {
        const int e = tid + q * kInvThreads;
        ei[q] = e < n * n ? (short)(e / n) : (short)-1;
        ej[q] = e < n * n ? (short)(e % n) : (short)-1;
        m[q] = e < n * n ? M[e] : 0.0;
    }
    for (int k = 0; k < n; k++) {
        double *P0 = row[k & 1], *Q = col[k & 1];          // two of each: the next pivot's are written during this one's update
#pragma unroll
        for (int q = 0; q < kPer; q++) {
            if (q >= used) break;
            if (ei[q] == k) P0[ej[q]] = m[q];              // the pivot row
            if (ej[q] == k && ei[q] >= 0) Q[ei[q]] = m[q]; // the pivot column, before the update
        }
        __syncthreads();
        if (tid < n) R[tid] = div_rn(tid == k ? 1.0 : P0[tid], P0[k]);
        __syncthreads();
#pragma unroll
        for (int q = 0; q < kPer; q++) {
            if (q >= used) break;
            const int i = ei[q], j = ej[q];
            if (i < 0) continue;
            // one FP64 instruction whichever case an entry is: the pivot row,
            // the pivot column (-Q R) or the rest (m - Q R)
            const double rj = R[j], x = __fma_rn(-Q[i], rj, j == k ? 0.0 : m[q]);
            m[q] = i == k ? rj : x;
        }
    }
#pragma unroll
    for (int q = 0; q < kPer; q++) {
        if (ei[q] < 0) continue;
        const int e = ei[q] * n + ej[q];
        C.cinv[e] = m[q];
        if (C.precision >= 1) C.cinv32[e] = (float)m[q];
    }
}

// ------------------------------------------------------------ V-cycle
// t = w D^-1 r
template <class T>
__global__ void __launch_bounds__(kTile) k_v_jac0(const CaseDev *__restrict__ cases, const Tile *__restrict__ tiles, int l) {
    CFDL_PDL_WAIT();
    const Tile tl = tiles[blockIdx.x];
    const CaseDev &C = cases[tl.c];
    if (sizeof(T) == 8 ? !pactive(C) : !mactive(C)) return;
    const int i = tl.first + (int)threadIdx.x;
    if (i >= tl.last) return;
    const LP<T> P = level<T>(C, l);
    P.t[i] = P.rd[i] * P.r[i];
}

// z = t + w D^-1 (r - A t).  kToT: the sweep from z into t instead (the first
// post-smoothing sweep, after k_v_lift has added the prolongated coarse
// correction to z).
template <class T, bool kToT = false>
__global__ void __launch_bounds__(kTile) k_v_jac(const CaseDev *__restrict__ cases, const Tile *__restrict__ tiles, int l) {
    CFDL_PDL_WAIT();
    const Tile tl = tiles[blockIdx.x];
    const CaseDev &C = cases[tl.c];
    if (sizeof(T) == 8 ? !pactive(C) : !mactive(C)) return;
    const int i = tl.first + (int)threadIdx.x;
    if (i >= tl.last || (sizeof(T) == 8 && l == 0 && flow_fp64(C))) return;
    const LP<T> P = level<T>(C, l);
    const T *x = kToT ? P.z : P.t;
    T *y = kToT ? P.t : P.z;
    // the row's own values first: measured faster on the coarse levels
    y[i] = jacobi_step<T, kToT ? 1 : 2>(x[i], P.r[i], P.rd[i], offsum<T>(P, x, i));
}
// The FP64 mesh-level sweeps wait for two things at once: the FP64 pipe is 65%
// busy (eight instructions a row of six slots take 26.7 of 40.3 us at 128^3) and
// the algorithmic bytes move at 0.8 of the copy bandwidth.  Neither the launch
// shape nor the index width changed their time; two instructions a row fewer
// did (45.7 -> 43.1 us): the sum starts from r, and the second sweep's w2/D is a
// plane of its own (rap2_p) instead of w/D times w2/w.
// 32 registers, 8 CTAs per SM: the coarse levels' sweeps would spill 100+
// bytes under that cap, so these are kernels of their own.
// The roundings of both launch shapes are spelled out, so a case's result does
// not depend on the shape its launch takes.
__device__ __forceinline__ double sweep64(double om, double x, double w, double s) { return __fma_rn(w, s, __dmul_rn(om, x)); }
__device__ __forceinline__ double resid64(double r, double d, double z) { return __fma_rn(-d, z, r); }
template <bool kToT>
__global__ void __launch_bounds__(kTile, 8) k_v_jac_mesh(const CaseDev *__restrict__ cases, const Tile *__restrict__ tiles) {
    CFDL_PDL_WAIT();
    const Tile tl = tiles[blockIdx.x];
    const CaseDev &C = cases[tl.c];
    if (!pactive(C) || !flow_fp64(C)) return;
    const int i = tl.first + (int)threadIdx.x;
    if (i >= tl.last) return;
    const LP<double> P = level<double>(C, 0);
    const double *x = kToT ? P.z : P.t, *rd = kToT ? P.rd : C.rap2_p;
    double *y = kToT ? P.t : P.z;
    constexpr double om = kToT ? 1.0 - kOmega : 1.0 - kOmega2;
    y[i] = sweep64(om, x[i], rd[i], offsum_mesh(P, x, i, P.r[i]));
}
// The same two rows per thread, i (even) and i + 1, with 8-byte index and
// 16-byte coefficient and vector loads where the case's row count is even (an
// odd one's planes are not aligned to pairs: its rows go one after the other).
// Used where the mesh fills the SMs more than once: 43.1 -> 40 us at 128^3; on
// small meshes the longer thread is the latency (32^3: an outer iteration 3%
// slower).
template <int W, bool kGuard>
__device__ __forceinline__ double2 pair_sum64(const LP<double> &P, const double *x, int i, double2 s) {
    const int n = P.n;
    int j[2][W];
    double c[2][W], v[2][W];
#pragma unroll
    for (int k = 0; k < W; k++) {
        const bool in = !kGuard || k < P.W;
        int2 d = make_int2(-1, -1);
        double2 a = make_double2(0.0, 0.0);
        if (in) { d = *(const int2 *)&P.nb[k * n + i]; a = *(const double2 *)&P.a[k * n + i]; }
        const bool ok0 = (unsigned)d.x < (unsigned)n, ok1 = (unsigned)d.y < (unsigned)n;
        j[0][k] = ok0 ? d.x : i; j[1][k] = ok1 ? d.y : i + 1;
        c[0][k] = ok0 ? a.x : 0.0; c[1][k] = ok1 ? a.y : 0.0;
    }
#pragma unroll
    for (int k = 0; k < W; k++) { v[0][k] = x[j[0][k]]; v[1][k] = x[j[1][k]]; }
#pragma unroll
    for (int k = 0; k < W; k++) { s.x = __fma_rn(c[0][k], v[0][k], s.x); s.y = __fma_rn(c[1][k], v[1][k], s.y); }
    return s;
}
// s + the off-diagonal sums of rows i and i + 1 (both inside the level)
__device__ __forceinline__ double2 pair_sum64_mesh(const LP<double> &P, const double *x, int i, double2 s) {
    if (P.n & 1) return make_double2(offsum_mesh(P, x, i, s.x), offsum_mesh(P, x, i + 1, s.y));
    if (P.W == 6) return pair_sum64<6, false>(P, x, i, s);
    if (P.W == 4) return pair_sum64<4, false>(P, x, i, s);
    return pair_sum64<kMaxW, true>(P, x, i, s);
}
template <bool kToT>
__global__ void __launch_bounds__(kTile / 2, 16) k_v_jac_pair64(const CaseDev *__restrict__ cases, const Tile *__restrict__ tiles) {
    CFDL_PDL_WAIT();
    const Tile tl = tiles[blockIdx.x];
    const CaseDev &C = cases[tl.c];
    if (!pactive(C) || !flow_fp64(C)) return;
    const int i = tl.first + 2 * (int)threadIdx.x;
    if (i >= tl.last) return;
    const LP<double> P = level<double>(C, 0);
    const double *x = kToT ? P.z : P.t, *rd = kToT ? P.rd : C.rap2_p;
    double *y = kToT ? P.t : P.z;
    constexpr double om = kToT ? 1.0 - kOmega : 1.0 - kOmega2;
    if (i + 1 < P.n) {
        const double2 s = pair_sum64_mesh(P, x, i, *(const double2 *)&P.r[i]);
        const double2 xi = *(const double2 *)&x[i], w = *(const double2 *)&rd[i];
        *(double2 *)&y[i] = make_double2(sweep64(om, xi.x, w.x, s.x), sweep64(om, xi.y, w.y, s.y));
    } else {
        y[i] = sweep64(om, x[i], rd[i], offsum_mesh(P, x, i, P.r[i]));
    }
}
// The FP32 mesh-level sweeps, two rows per thread (pair_slots).  kFromR: the
// first pre-smoothing sweep, from t = w D^-1 r formed on the fly for the rows
// and their neighbours instead of read from k_v_jac0's pass (the same
// products, so the same z; one pass over the level fewer)
template <bool k16, bool kToT, bool kFromR>
__global__ void __launch_bounds__(kTile / 2, 16) k_v_jac_pair(const CaseDev *__restrict__ cases, const Tile *__restrict__ tiles) {
    CFDL_PDL_WAIT();
    const Tile tl = tiles[blockIdx.x];
    const CaseDev &C = cases[tl.c];
    if (!mactive(C)) return;
    const int i = tl.first + 2 * (int)threadIdx.x;
    if (i >= tl.last) return;
    const LP<float> P = level<float>(C, 0);
    const float *x = kFromR ? P.r : kToT ? P.z : P.t;
    float *y = kToT ? P.t : P.z;
    const float2 off = pair_offsum_mesh<k16, kFromR>(P, x, i);
    const float2 r = *(const float2 *)&P.r[i], rd = *(const float2 *)&P.rd[i];
    const float2 xi = kFromR ? make_float2(rd.x * r.x, rd.y * r.y) : *(const float2 *)&x[i];
    *(float2 *)&y[i] = make_float2(pair_jacobi<kToT ? 1 : 2>(xi.x, r.x, rd.x, off.x),
                                   pair_jacobi<kToT ? 1 : 2>(xi.y, r.y, rd.y, off.y));
}

// z = z + s P z_{l+1}: the prolongated coarse correction, added in place.
// With it as its own streaming pass, the sweep after it gathers each
// neighbour's corrected value once instead of the neighbour's aggregate and
// then the coarse value: the same values, a shorter load chain.
template <class T>
__global__ void __launch_bounds__(kTile) k_v_lift(const CaseDev *__restrict__ cases, const Tile *__restrict__ tiles, int l) {
    CFDL_PDL_WAIT();
    const Tile tl = tiles[blockIdx.x];
    const CaseDev &C = cases[tl.c];
    if (sizeof(T) == 8 ? !pactive(C) : !mactive(C)) return;
    const int i = tl.first + (int)threadIdx.x;
    if (i >= tl.last) return;
    const LP<T> P = level<T>(C, l);
    const AmgLevelDev &L = C.lev[l];
    const T *zc = sizeof(T) == 8 ? (const T *)L.z : (const T *)L.z32;
    P.z[i] = P.z[i] + (T)kOverCorrect * zc[L.agg[i]];
}

// t = r - A z (the smoothed residual)
template <class T>
__global__ void __launch_bounds__(kTile) k_v_resid(const CaseDev *__restrict__ cases, const Tile *__restrict__ tiles, int l) {
    CFDL_PDL_WAIT();
    const Tile tl = tiles[blockIdx.x];
    const CaseDev &C = cases[tl.c];
    if (sizeof(T) == 8 ? !pactive(C) : !mactive(C)) return;
    const int i = tl.first + (int)threadIdx.x;
    if (i >= tl.last) return;
    const LP<T> P = level<T>(C, l);
    P.t[i] = P.r[i] - amul_coarse<T>(P, P.z, i);
}
// the mesh level's residual, as its sweeps: FP64 with their register cap, FP32
// two rows per thread
__global__ void __launch_bounds__(kTile, 8) k_v_resid_mesh(const CaseDev *__restrict__ cases, const Tile *__restrict__ tiles) {
    CFDL_PDL_WAIT();
    const Tile tl = tiles[blockIdx.x];
    const CaseDev &C = cases[tl.c];
    if (!pactive(C) || !flow_fp64(C)) return;
    const int i = tl.first + (int)threadIdx.x;
    if (i >= tl.last) return;
    const LP<double> P = level<double>(C, 0);
    P.t[i] = offsum_mesh(P, P.z, i, resid64(P.r[i], P.dg[i], P.z[i]));
}
// The mesh level's residual in precision 1's order of sums (flow_fp64): r - A z
// with A z formed first, its roundings spelled out.
template <int W, bool kGuard> __device__ __forceinline__ double amul_order(const LP<double> &P, const double *x, int i) {
    int j[W];
    double c[W];
    row_slots<W, double, kGuard>(P, i, j, c);
    double s = __fma_rn(P.dg[i], x[i], -__dmul_rn(c[0], x[j[0]]));
#pragma unroll
    for (int k = 1; k < W; k++) s = __fma_rn(-c[k], x[j[k]], s);
    return s;
}
__global__ void __launch_bounds__(kTile) k_v_resid_order(const CaseDev *__restrict__ cases, const Tile *__restrict__ tiles) {
    CFDL_PDL_WAIT();
    const Tile tl = tiles[blockIdx.x];
    const CaseDev &C = cases[tl.c];
    if (!pactive(C) || flow_fp64(C)) return;
    const int i = tl.first + (int)threadIdx.x;
    if (i >= tl.last) return;
    const LP<double> P = level<double>(C, 0);
    const double y = P.W == 6 ? amul_order<6, false>(P, P.z, i) : P.W == 4 ? amul_order<4, false>(P, P.z, i) : amul_order<kMaxW, true>(P, P.z, i);
    P.t[i] = P.r[i] - y;
}
__global__ void __launch_bounds__(kTile / 2, 16) k_v_resid_pair64(const CaseDev *__restrict__ cases, const Tile *__restrict__ tiles) {
    CFDL_PDL_WAIT();
    const Tile tl = tiles[blockIdx.x];
    const CaseDev &C = cases[tl.c];
    if (!pactive(C) || !flow_fp64(C)) return;
    const int i = tl.first + 2 * (int)threadIdx.x;
    if (i >= tl.last) return;
    const LP<double> P = level<double>(C, 0);
    if (i + 1 < P.n) {
        const double2 r = *(const double2 *)&P.r[i], d = *(const double2 *)&P.dg[i], z = *(const double2 *)&P.z[i];
        *(double2 *)&P.t[i] = pair_sum64_mesh(P, P.z, i, make_double2(resid64(r.x, d.x, z.x), resid64(r.y, d.y, z.y)));
    } else {
        P.t[i] = offsum_mesh(P, P.z, i, resid64(P.r[i], P.dg[i], P.z[i]));
    }
}
template <bool k16>
__global__ void __launch_bounds__(kTile / 2, 16) k_v_resid_pair(const CaseDev *__restrict__ cases, const Tile *__restrict__ tiles) {
    CFDL_PDL_WAIT();
    const Tile tl = tiles[blockIdx.x];
    const CaseDev &C = cases[tl.c];
    if (!mactive(C)) return;
    const int i = tl.first + 2 * (int)threadIdx.x;
    if (i >= tl.last) return;
    const LP<float> P = level<float>(C, 0);
    const float2 y = pair_amul_mesh<k16>(P, P.z, i), r = *(const float2 *)&P.r[i];
    *(float2 *)&P.t[i] = make_float2(r.x - y.x, r.y - y.y);
}

// sum of t over the members of aggregate I of the level below L: four
// members per step, their indices and then their values loaded side by side,
// summed in member order (one member per step made every member two
// dependent trips to memory)
template <class T>
__device__ __forceinline__ T restrict_row(const AmgLevelDev &L, const T *t, int I) {
    const int m0 = L.mem_ptr[I], m1 = L.mem_ptr[I + 1];
    T s = 0;
    for (int m = m0; m < m1; m += 4) {
        int j[4];
        T x[4];
#pragma unroll
        for (int u = 0; u < 4; u++) j[u] = m + u < m1 ? L.mem[m + u] : -1;
#pragma unroll
        for (int u = 0; u < 4; u++) x[u] = j[u] >= 0 ? t[j[u]] : (T)0;
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (j[u] >= 0) s += x[u];
    }
    return s;
}

// r_{l1}[I] = sum of the residual t over the members of aggregate I (one
// thread per coarse row: the large levels, where rows outnumber lanes)
template <class T>
__global__ void __launch_bounds__(kTile) k_v_restrict(const CaseDev *__restrict__ cases, const Tile *__restrict__ tiles, int l1) {
    CFDL_PDL_WAIT();
    const Tile tl = tiles[blockIdx.x];
    const CaseDev &C = cases[tl.c];
    if (sizeof(T) == 8 ? !pactive(C) : !mactive(C)) return;
    const int I = tl.first + (int)threadIdx.x;
    if (I >= tl.last) return;
    const AmgLevelDev &L = C.lev[l1 - 1];
    const LP<T> F = level<T>(C, l1 - 1);
    T *rc = sizeof(T) == 8 ? (T *)L.r : (T *)L.r32;
    rc[I] = restrict_row<T>(L, F.t, I);
}

// Sum of a coarse slot's fine couplings af[src[q0..q1)), in list order: kCh
// indices and then kCh values loaded side by side (one by one, each entry was
// two trips to L2: at 128^3 the large levels took 79 us on average and now
// take 71 with kCh = 2, the small ones 35 and now 26 with 8; at 24^3 13.2 and
// 9.8).
template <int kCh>
__device__ __forceinline__ double gather_sum(const double *__restrict__ af, const int *__restrict__ src, int q0, int q1) {
    double v = 0.0;
    for (int q = q0; q < q1; q += kCh) {
        int j[kCh];
        double x[kCh];
#pragma unroll
        for (int u = 0; u < kCh; u++) j[u] = q + u < q1 ? src[q + u] : -1;
#pragma unroll
        for (int u = 0; u < kCh; u++) x[u] = j[u] >= 0 ? af[j[u]] : 0.0;
#pragma unroll
        for (int u = 0; u < kCh; u++)
            if (j[u] >= 0) v += x[u];
    }
    return v;
}

// Galerkin row I, one thread per row (large levels)
__global__ void __launch_bounds__(kTile) k_amg_gal(const CaseDev *__restrict__ cases, const Tile *__restrict__ tiles, int l) {
    CFDL_PDL_WAIT();
    const Tile t = tiles[blockIdx.x];
    const CaseDev &C = cases[t.c];
    const int I = t.first + (int)threadIdx.x;
    if (I >= t.last || C.sc->halted) return;
    const AmgLevelDev &L = C.lev[l - 1];
    const double *af = l == 1 ? C.anb_p : C.lev[l - 2].a;
    const bool mixed = C.precision >= 1;
    const int n = L.n;
    double dsum = 0.0;
    // padding slots (k >= len) keep the zeros they were created with
    const int len = L.len[I];
    const int *__restrict__ gp = L.g_ptr, *__restrict__ gs = L.g_src;
    int q0 = gp[I], q1 = gp[I + 1];
    for (int k = 0; k < len; k++) {
        const int s = k * n + I;
        int p0 = 0, p1 = 0;                  // the next slot's list, ahead of this one's gathers
        if (k + 1 < len) { p0 = gp[s + n]; p1 = gp[s + n + 1]; }
        const double v = gather_sum<2>(af, gs, q0, q1);
        q0 = p0; q1 = p1;
        L.a[s] = v;
        if (mixed) L.a32[s] = narrow_f32(v);
        dsum += v;
    }
    L.dg[I] = dsum;
    const double rd = div_rn(kOmega, dsum);
    L.rd[I] = rd;
    if (mixed) { L.dg32[I] = narrow_f32(dsum); L.rd32[I] = narrow_f32(rd); }
}

// ------------------------------------------------- the V-cycle's tail
// The small coarse levels of a case, from its tail level (the first level of
// at most kTailRows rows) down to the coarsest and back, on one cluster of
// kTailCtas CTAs: the steps of k_v_jac0 / k_v_jac / k_v_resid / k_v_restrict,
// the coarsest solve and k_v_lift / k_v_jac, one row per thread, each row's
// sum in its slot order.  A step is a fraction of a microsecond of arithmetic
// behind a chain of dependent loads of about 0.35 us each from L2, so the
// chain is what is cut: everything a step needs is staged in shared memory
// first, all of it in flight together (cp.async), and every CTA keeps a whole
// copy of the vectors that the next step gathers from, written by a row's
// owner into all CTAs' shared memory before the cluster barrier (0.6 us).
// Levels small enough are done whole by every CTA for itself, behind block
// barriers; more rows would cost more than the barrier, FP64 ones sooner (16
// clocks of the SM's FP64 pipe per warp and slot).
// Measured per V-cycle (events around the launch) against one CTA of 1024
// threads reading everything from L2 at every step: 128^3 cavity (levels of
// 662 and 37 rows) 43.5 -> 22.0 us FP64, 25.7 -> 15.0 FP32; 24^3 (1685, 105,
// 8 rows) 36.9 -> 20.0 FP32; 41^3 prisms (1263, 70, 6) 69 -> 30 FP64; twelve
// uneven cases 79 -> 30 FP64.
constexpr int kTailCtas = 8;                               // portable cluster size
constexpr int kTailBlock = kTailRows / kTailCtas;          // one row of the largest level per thread
constexpr int kTailMaxSmem = 200 * 1024;
static_assert(kTailBlock == 256, "a level done whole has at most this many rows");
template <class T> constexpr int tail_whole() { return sizeof(T) == 8 ? 128 : 256; }

// 4 or 8 bytes from global to shared memory, asynchronously
__device__ __forceinline__ void stage(float *s, const float *g) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(s)), "l"(g));
}
__device__ __forceinline__ void stage(int *s, const int *g) { stage((float *)s, (const float *)g); }
__device__ __forceinline__ void stage(double *s, const double *g) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(s)), "l"(g));
}

template <class T>
__global__ void __launch_bounds__(kTailBlock) k_v_tail(const CaseDev *__restrict__ cases, int ncases) {
    CFDL_PDL_WAIT();
    namespace cg = cooperative_groups;
    extern __shared__ __align__(16) unsigned char tail_mem[];
    __shared__ TailPlan Q;
    const int c = (int)blockIdx.x / kTailCtas, rank = (int)blockIdx.x % kTailCtas, tid = (int)threadIdx.x;
    if (c >= ncases) return;                               // the whole cluster
    const CaseDev &C = cases[c];
    const long long *plan = (const long long *)(sizeof(T) == 8 ? C.tail64 : C.tail32);
    if (C.precond != 1 || (sizeof(T) == 8 ? !pactive(C) : !mactive(C))) return;   // the whole cluster
    cg::cluster_group cluster = cg::this_cluster();
    auto started = cluster.barrier_arrive();               // waited for before the first write to another CTA
    static_assert(sizeof(TailPlan) % 8 == 0, "copied by 8-byte words");
    for (int j = tid; j < (int)(sizeof(TailPlan) / 8); j += kTailBlock) ((long long *)&Q)[j] = plan[j];
    __syncthreads();
    auto vec = [&](int off) { return (T *)(tail_mem + off); };
    auto idx = [&](int off) { return (int *)(tail_mem + off); };
    const int nl = Q.nl, nc = Q.nc;
    for (int l = 0; l < nl; l++) {
        const TailLevel &v = Q.lv[l];
        const int i = (v.whole ? 0 : rank * v.R) + tid;
        if (tid < v.R && i < v.n) {
            const T *a = (const T *)v.a + i;
            const int *nb = v.nb + i;
            for (int k = 0; k < v.S; k++) {
                stage(vec(v.sa) + k * v.R + tid, a + (size_t)k * v.n);
                stage(idx(v.snb) + k * v.R + tid, nb + (size_t)k * v.n);
            }
            stage(vec(v.srd) + tid, (const T *)v.rd + i);
            stage(vec(v.sdg) + tid, (const T *)v.dg + i);
            stage(idx(v.slen) + tid, v.len + i);
            if (l == 0) stage(vec(v.sr) + tid, (const T *)Q.r + i);
        }
        for (int j = tid; j < v.n; j += kTailBlock) {
            stage(idx(v.sagg) + j, v.agg + j);
            stage(idx(v.smem_) + j, v.mem + j);
        }
        const int n1 = l + 1 < nl ? Q.lv[l + 1].n : nc;
        for (int j = tid; j <= n1; j += kTailBlock) stage(idx(v.smptr) + j, v.mptr + j);
    }
    for (int e = tid; e < nc * nc; e += kTailBlock)        // transposed: a thread sums a row of it
        stage(vec(Q.sminv) + (e % nc) * nc + e / nc, (const T *)Q.minv + e);
    if (nl == 0)
        for (int e = tid; e < nc; e += kTailBlock) stage(vec(Q.sr) + e, (const T *)Q.r + e);
    // t = w D^-1 r of the whole tail level, by every CTA for itself
    auto t_down = [&](int l) { return Q.lv[l].whole ? Q.w[l & 1] : Q.t[l & 1]; };
    auto t_up = [&](int l) { return Q.lv[l].whole ? Q.w[(l + 1) & 1] : Q.t[(l + 1) & 1]; };
    if (nl > 0) {
        T *t = vec(t_down(0));
        const T *r = (const T *)Q.r, *rd = (const T *)Q.lv[0].rd;
        constexpr int kPer = kTailRows / kTailBlock;
        T rv[kPer], dv[kPer];
#pragma unroll
        for (int u = 0; u < kPer; u++) {
            const int j = tid + u * kTailBlock;
            rv[u] = j < Q.lv[0].n ? r[j] : (T)0;
            dv[u] = j < Q.lv[0].n ? rd[j] : (T)0;
        }
#pragma unroll
        for (int u = 0; u < kPer; u++) {
            const int j = tid + u * kTailBlock;
            if (j < Q.lv[0].n) t[j] = dv[u] * rv[u];
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    // one value of a level's vector, into every CTA's copy (a level done whole: into this one's)
    auto put = [&](const TailLevel &v, int off, int i, T x) {
        T *p = vec(off) + i;
        if (v.whole) { *p = x; return; }
#pragma unroll
        for (int k = 0; k < kTailCtas; k++) *cluster.map_shared_rank(p, k) = x;
    };
    auto sync = [&](const TailLevel &v) {
        if (v.whole) __syncthreads();
        else cluster.sync();
    };
    // s +- the sum of a_ij x(j) over the couplings of this thread's row i of a level, slots in order
    auto row_sum = [&](const TailLevel &v, int i, int len, T s, auto x, bool minus) {
        const int R = v.R, m = min(len, v.S);
        const T *sa = vec(v.sa) + tid;
        const int *sn = idx(v.snb) + tid;
        if (minus) {
#pragma unroll 4
            for (int k = 0; k < m; k++) s -= sa[k * R] * x(sn[k * R]);
        } else {
#pragma unroll 4
            for (int k = 0; k < m; k++) s += sa[k * R] * x(sn[k * R]);
        }
        for (int k = m; k < len; k++) {                    // slots that were not staged
            const T ak = ((const T *)v.a)[(size_t)k * v.n + i], xk = x(v.nb[(size_t)k * v.n + i]);
            if (minus) s -= ak * xk;
            else s += ak * xk;
        }
        return s;
    };
    // the residual of a level summed over the members of aggregate i, in member order
    auto restrict_to = [&](int l, int i) {
        const TailLevel &v = Q.lv[l];
        const T *tf = vec(t_down(l));
        const int *mm = idx(v.smem_), m0 = idx(v.smptr)[i], m1 = idx(v.smptr)[i + 1];
        T r = 0;
#pragma unroll 4
        for (int m = m0; m < m1; m++) r += tf[mm[m]];
        return r;
    };
    cluster.barrier_wait(std::move(started));
    for (int l = 0; l < nl; l++) {
        const TailLevel &v = Q.lv[l];
        const int i = (v.whole ? 0 : rank * v.R) + tid, tb = t_down(l);
        const bool mine = tid < v.R && i < v.n;
        const T rd = mine ? vec(v.srd)[tid] : (T)0;
        const int len = mine ? idx(v.slen)[tid] : 0;
        T r = 0;
        if (l == 0) {
            if (mine) r = vec(v.sr)[tid];
        } else {
            if (mine) {
                r = restrict_to(l - 1, i);
                vec(v.sr)[tid] = r;
                put(v, tb, i, rd * r);
            }
            sync(v);
        }
        const T *tc = vec(tb), *zc = vec(v.sz);
        T z = 0;
        if (mine) {
            z = jacobi_step<T>(tc[i], r, rd, row_sum(v, i, len, (T)0, [&](int j) { return tc[j]; }, false));
            put(v, v.sz, i, z);
        }
        sync(v);
        if (mine) put(v, tb, i, r - row_sum(v, i, len, vec(v.sdg)[tid] * z, [&](int j) { return zc[j]; }, true));
        sync(v);
    }
    // coarsest, by every CTA for itself: z_L = Minv r_L
    if (nl > 0) {
        for (int i = tid; i < nc; i += kTailBlock) vec(Q.sr)[i] = restrict_to(nl - 1, i);
        __syncthreads();
    }
    for (int i = tid; i < nc; i += kTailBlock) {
        const T *Mi = vec(Q.sminv) + i, *r = vec(Q.sr);
        T sum = 0;
#pragma unroll 8
        for (int j = 0; j < nc; j++) sum += Mi[j * nc] * r[j];
        vec(Q.sz)[i] = sum;
        if (nl == 0 && rank == 0) ((T *)Q.z)[i] = sum;
    }
    __syncthreads();
    const T sc = (T)kOverCorrect;
    for (int l = nl - 1; l >= 0; l--) {
        // t goes to the other buffer than on the way down: a slower CTA may
        // still be summing the last residual of that
        const TailLevel &v = Q.lv[l];
        const int i = (v.whole ? 0 : rank * v.R) + tid, tb = t_up(l);
        const bool mine = tid < v.R && i < v.n;
        const int len = mine ? idx(v.slen)[tid] : 0;
        const T *zl = vec(v.sz), *zc = vec(l + 1 < nl ? Q.lv[l + 1].sz : Q.sz), *tc = vec(tb);
        const int *ag = idx(v.sagg);
        const T r = mine ? vec(v.sr)[tid] : (T)0, rd = mine ? vec(v.srd)[tid] : (T)0;
        T tv = 0;
        if (mine) {
            const T xi = zl[i] + sc * zc[ag[i]];
            tv = jacobi_step<T, 1>(xi, r, rd, row_sum(v, i, len, (T)0, [&](int j) { return zl[j] + sc * zc[ag[j]]; }, false));
            put(v, tb, i, tv);
        }
        sync(v);
        if (mine) {
            const T z = jacobi_step<T>(tv, r, rd, row_sum(v, i, len, (T)0, [&](int j) { return tc[j]; }, false));
            if (l > 0) put(v, v.sz, i, z);
            else if (!v.whole || rank == 0) ((T *)Q.z)[i] = z;
        }
        if (l > 0) sync(v);
    }
}

// ------------------------------------------------- coarse levels, grouped
// Coarse rows are wide (up to ~30 couplings) and a thread that walked one
// alone would issue its index -> value -> vector loads one slot after the
// other: a chain of dependent loads that left the small levels latency-bound.
// On small levels each row is handled by G lanes that split its slots (and
// the Galerkin and restriction gather lists) and combine their partial sums
// with shuffles, in a fixed order.  Tiles hold kTile / G rows.
#define GROUP_HEAD                                                   \
    const Tile tl = tiles[blockIdx.x];                               \
    const CaseDev &C = cases[tl.c];                                  \
    const int g = (int)threadIdx.x & (G - 1);                        \
    const int i = tl.first + (int)threadIdx.x / G;                   \
    const bool ok = i < tl.last;

template <int G, class T> __device__ __forceinline__ T group_sum(T v) {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// sum_k a_ik x_j over the row's couplings inside the level, split over the group
template <int G, class T> __device__ __forceinline__ T group_offdiag(const LP<T> &P, const T *x, int i, bool ok, int g) {
    T s = 0;
    if (ok) {
        const int len = row_len(P, i);
        for (int k = g; k < len; k += G) {
            const int j = P.nb[k * P.n + i];
            if ((unsigned)j < (unsigned)P.n) s += P.a[k * P.n + i] * x[j];
        }
    }
    return group_sum<G>(s);
}

// z = t + w D^-1 (r - A t)
template <class T, int G>
__global__ void __launch_bounds__(kTile) k_vg_jac(const CaseDev *__restrict__ cases, const Tile *__restrict__ tiles, int l) {
    CFDL_PDL_WAIT();
    GROUP_HEAD
    if (sizeof(T) == 8 ? !pactive(C) : !mactive(C)) return;
    const LP<T> P = level<T>(C, l);
    const T off = group_offdiag<G, T>(P, P.t, i, ok, g);
    if (ok && g == 0) P.z[i] = jacobi_step<T>(P.t[i], P.r[i], P.rd[i], off);
}

// t = r - A z
template <class T, int G>
__global__ void __launch_bounds__(kTile) k_vg_resid(const CaseDev *__restrict__ cases, const Tile *__restrict__ tiles, int l) {
    CFDL_PDL_WAIT();
    GROUP_HEAD
    if (sizeof(T) == 8 ? !pactive(C) : !mactive(C)) return;
    const LP<T> P = level<T>(C, l);
    const T off = group_offdiag<G, T>(P, P.z, i, ok, g);
    if (ok && g == 0) P.t[i] = P.r[i] - (P.dg[i] * P.z[i] - off);
}

// r_{l1}[I] = sum of the residual t_{l1-1} over the members of aggregate I
template <class T, int G>
__global__ void __launch_bounds__(kTile) k_vg_restrict(const CaseDev *__restrict__ cases, const Tile *__restrict__ tiles, int l1) {
    CFDL_PDL_WAIT();
    GROUP_HEAD
    if (sizeof(T) == 8 ? !pactive(C) : !mactive(C)) return;
    const AmgLevelDev &L = C.lev[l1 - 1];
    const LP<T> F = level<T>(C, l1 - 1);
    T s = 0;
    if (ok)
        for (int m = L.mem_ptr[i] + g; m < L.mem_ptr[i + 1]; m += G) s += F.t[L.mem[m]];
    s = group_sum<G>(s);
    T *rc = sizeof(T) == 8 ? (T *)L.r : (T *)L.r32;
    if (ok && g == 0) rc[i] = s;
}

// t = x + w D^-1 (r - A x) with x = z + s P z_{l+1}
template <class T, int G>
__global__ void __launch_bounds__(kTile) k_vg_prolong(const CaseDev *__restrict__ cases, const Tile *__restrict__ tiles, int l) {
    CFDL_PDL_WAIT();
    GROUP_HEAD
    if (sizeof(T) == 8 ? !pactive(C) : !mactive(C)) return;
    const LP<T> P = level<T>(C, l);
    const AmgLevelDev &L = C.lev[l];
    const T *zc = sizeof(T) == 8 ? (const T *)L.z : (const T *)L.z32;
    const T sc = (T)kOverCorrect;
    T off = 0;
    if (ok) {
        const int len = row_len(P, i);
        for (int k = g; k < len; k += G) {
            const int j = P.nb[k * P.n + i];
            if ((unsigned)j < (unsigned)P.n) off += P.a[k * P.n + i] * (P.z[j] + sc * zc[L.agg[j]]);
        }
    }
    off = group_sum<G>(off);
    if (ok && g == 0) {
        const T xi = P.z[i] + sc * zc[L.agg[i]];
        P.t[i] = jacobi_step<T, 1>(xi, P.r[i], P.rd[i], off);
    }
}

// Galerkin row I of level l: each lane sums the gather lists of its slots
template <int G>
__global__ void __launch_bounds__(kTile) k_amg_galg(const CaseDev *__restrict__ cases, const Tile *__restrict__ tiles, int l) {
    CFDL_PDL_WAIT();
    GROUP_HEAD
    if (C.sc->halted) return;
    const AmgLevelDev &L = C.lev[l - 1];
    const double *af = l == 1 ? C.anb_p : C.lev[l - 2].a;
    const bool mixed = C.precision >= 1;
    const int n = L.n;
    double dsum = 0.0;
    const int *__restrict__ gp = L.g_ptr, *__restrict__ gs = L.g_src;
    if (ok)
        for (int k = g, len = L.len[i]; k < len; k += G) {
            const int sl = k * n + i;
            const double v = gather_sum<8>(af, gs, gp[sl], gp[sl + 1]);
            L.a[sl] = v;
            if (mixed) L.a32[sl] = narrow_f32(v);
            dsum += v;
        }
    dsum = group_sum<G>(dsum);
    if (ok && g == 0) {
        L.dg[i] = dsum;
        const double rd = div_rn(kOmega, dsum);
        L.rd[i] = rd;
        if (mixed) { L.dg32[i] = narrow_f32(dsum); L.rd32[i] = narrow_f32(rd); }
    }
}

// ------------------------------------------------------------ CG (FP64)
// r = b - mean, x = 0; ||r0||
__global__ void __launch_bounds__(kTile) k_apc_init(const CaseDev *__restrict__ cases, const Tile *__restrict__ tiles,
                                                    const int *__restrict__ cfirst, const int *__restrict__ cnt, double *partials) {
    CFDL_PDL_WAIT();
    const Tile t = tiles[blockIdx.x];
    const CaseDev &C = cases[t.c];
    SolveScalars *S = C.sc;
    const int tile0 = cfirst[t.c], ntiles = cnt[t.c];
    if (S->halted) return;
    double v[2] = {0, 0};
    FOR_CELLS(t) {
        const double r = C.b[i] - S->mean_b;
        C.kr[i] = r; C.phic[i] = 0.0;
        v[0] += r * r; v[1] += C.b[i] * C.b[i];
    }
    __shared__ double s[2];
    if (case_sums<2>(v, &C.counters[CNT_A0], partials, tile0, ntiles, s)) {
        if (threadIdx.x == 0) {
            const int cap = C.solve_mode == 0 ? C.nit : C.tight_maxit;
            S->r0norm_p = S->rnorm_p = sqrt(s[0]);
            S->mass_imbalance = sqrt(s[1]);
            S->iters_p = 0; S->status_p = 0; S->rz = 0.0;
            S->tol_p = (C.solve_mode == 0 ? C.rtol_p : C.tight_rtol) * S->r0norm_p;
            S->active_p = S->r0norm_p > S->tol_p && cap > 0;
            if (!isfinite(S->r0norm_p)) { S->active_p = 0; S->status_p = CFDL_ERR_NONFINITE; }
        }
    }
}

// beta = (r,z)/(r,z)_old (0 on the first iteration)
template <bool kSpl>
__global__ void __launch_bounds__(kTile) k_apc_rz(const CaseDev *__restrict__ cases, const Tile *__restrict__ tiles,
                                                  const int *__restrict__ cfirst, const int *__restrict__ cnt, double *partials) {
    CFDL_PDL_WAIT();
    const Tile t = tiles[blockIdx.x];
    const CaseDev &C = cases[t.c];
    SolveScalars *S = C.sc;
    const int tile0 = cfirst[t.c], ntiles = cnt[t.c];
    if (!S->active_p) return;
    __shared__ double s[1];
    bool last;
    if constexpr (kSpl) {
        double a[1] = {0}, b[1] = {0};
        const int i = split_row(t);
        if (i < t.last) {
            a[0] = C.kr[i];
            b[0] = C.ks[i];
        }
        last = split_sums<1>(a, b, &C.counters[CNT_A1], partials, tile0, ntiles, s);
    } else {
        // one row per step in FP64: the paired form (cg_rz_rows) measured slower
        // here (21.4 against 18.8 us a launch at 128^3)
        double v[1] = {0.0};
        FOR_CELLS(t) v[0] += C.kr[i] * C.ks[i];
        last = case_sums<1>(v, &C.counters[CNT_A1], partials, tile0, ntiles, s);
    }
    if (last) {
        if (threadIdx.x == 0) {
            S->beta_p = S->iters_p == 0 || S->rz == 0.0 ? 0.0 : s[0] / S->rz;
            S->rz = s[0];
            if (!isfinite(s[0])) { S->active_p = 0; S->status_p = CFDL_ERR_NONFINITE; }
        }
    }
}

// p = z + beta p; q = A p needs every p, so it is the next kernel
__global__ void __launch_bounds__(kTile) k_apc_p(const CaseDev *__restrict__ cases, const Tile *__restrict__ tiles) {
    CFDL_PDL_WAIT();
    const Tile t = tiles[blockIdx.x];
    const CaseDev &C = cases[t.c];
    const SolveScalars *S = C.sc;
    if (!S->active_p) return;
    cg_p_rows<double>(C.ks, C.kp, S->iters_p == 0, S->beta_p, t);
}

// q = A p; alpha = rz / (p, q)
template <bool kSpl>
__global__ void __launch_bounds__(kTile) k_apc_q(const CaseDev *__restrict__ cases, const Tile *__restrict__ tiles,
                                                 const int *__restrict__ cfirst, const int *__restrict__ cnt, double *partials) {
    CFDL_PDL_WAIT();
    const Tile t = tiles[blockIdx.x];
    const CaseDev &C = cases[t.c];
    SolveScalars *S = C.sc;
    const int tile0 = cfirst[t.c], ntiles = cnt[t.c];
    if (!S->active_p) return;
    __shared__ double s[1];
    bool last;
    if constexpr (kSpl) {
        double a[1] = {0}, b[1] = {0};
        const int i = split_row(t);
        if (i < t.last) {
            b[0] = amul<double>(level<double>(C, 0), C.kp, i);
            a[0] = C.kp[i];
            C.kv[i] = b[0];
        }
        last = split_sums<1>(a, b, &C.counters[CNT_A2], partials, tile0, ntiles, s);
    } else {
        double v[1] = {cg_aq_rows(level<double>(C, 0), C.kp, C.kv, t)};
        last = case_sums<1>(v, &C.counters[CNT_A2], partials, tile0, ntiles, s);
    }
    if (last) {
        if (threadIdx.x == 0) {
            if (!(s[0] > 0.0) || !isfinite(s[0])) {
                // runs only while ||r|| is above the tolerance, where p.Ap > 0 for the SPD system
                S->active_p = 0;
                S->status_p = isfinite(s[0]) ? CFDL_ERR_BREAKDOWN : CFDL_ERR_NONFINITE;
            }
            else S->alpha_p = S->rz / s[0];
        }
    }
}

// x += alpha p; r -= alpha q; ||r||
template <bool kSpl>
__global__ void __launch_bounds__(kTile) k_apc_x(const CaseDev *__restrict__ cases, const Tile *__restrict__ tiles,
                                                 const int *__restrict__ cfirst, const int *__restrict__ cnt, double *partials) {
    CFDL_PDL_WAIT();
    const Tile t = tiles[blockIdx.x];
    const CaseDev &C = cases[t.c];
    SolveScalars *S = C.sc;
    const int tile0 = cfirst[t.c], ntiles = cnt[t.c];
    if (!S->active_p) return;
    __shared__ double s[1];
    bool last;
    if constexpr (kSpl) {
        double a[1] = {0}, b[1] = {0};
        const int i = split_row(t);
        if (i < t.last) {
            const double al = S->alpha_p, x = C.phic[i], p = C.kp[i], r = C.kr[i] - al * C.kv[i];
            C.phic[i] = x + al * p;
            C.kr[i] = a[0] = b[0] = r;
        }
        last = split_sums<1>(a, b, &C.counters[CNT_A3], partials, tile0, ntiles, s);
    } else {
        // one row per step in FP64: the paired form (cg_x_rows, 48 registers
        // against 32) measured slower here (31.9 against 28.5 us a launch)
        double v[1] = {0};
        FOR_CELLS(t) {
            const double a = S->alpha_p;
            C.phic[i] = C.phic[i] + a * C.kp[i];
            const double r = C.kr[i] - a * C.kv[i];
            C.kr[i] = r;
            v[0] += r * r;
        }
        last = case_sums<1>(v, &C.counters[CNT_A3], partials, tile0, ntiles, s);
    }
    if (last) {
        if (threadIdx.x == 0) {
            const int cap = C.solve_mode == 0 ? C.nit : C.tight_maxit;
            const double rn = sqrt(s[0]);
            S->rnorm_p = rn;
            S->iters_p += 1;
            int act = rn > S->tol_p;
            if (!isfinite(rn)) { act = 0; S->status_p = CFDL_ERR_NONFINITE; }
            else if (act && S->iters_p >= cap) { act = 0; if (C.solve_mode == 1) S->status_p = CFDL_ERR_ITER_CAP; }
            S->active_p = act;
        }
    }
}

// the mesh level's neighbour offsets for CaseDev::nb16; overflow is set when
// an offset does not fit in 16 bits
__global__ void k_nb16(const int *__restrict__ nb, short *__restrict__ out, int ne, int ld, int W, unsigned *overflow) {
    const size_t s = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (s >= (size_t)W * ld) return;
    const int i = (int)(s % (size_t)ld), k = (int)(s / (size_t)ld);
    const int j = i < ne ? nb[(size_t)k * ne + i] : -1;       // the padding row has no neighbours
    short v = kNb16None;
    if (j >= 0 && j < ne) {
        const int d = j - i;
        if (d < -32767 || d > 32767) atomicOr(overflow, 1u);
        else v = (short)d;
    }
    out[s] = v;
}

}  // namespace

// ------------------------------------------------------------------ host
namespace {

template <class T, class A> int dupload(HostCase *hc, T **d, const std::vector<T, A> &h) {
    size_t bytes = std::max<size_t>(1, h.size()) * sizeof(T);
    if (int st = dev_alloc((void **)d, bytes)) return st;
    hc->amg_allocs.push_back(*d);
    hc->bytes += bytes;
    if (h.empty()) return CFDL_OK;
    return cuda_status(cudaMemcpy(*d, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice));
}
template <class T> int dzeros(HostCase *hc, T **d, size_t n) {
    if (int st = dev_alloc((void **)d, std::max<size_t>(1, n) * sizeof(T))) return st;
    hc->amg_allocs.push_back(*d);
    hc->bytes += std::max<size_t>(1, n) * sizeof(T);
    return cuda_status(cudaMemset(*d, 0, std::max<size_t>(1, n) * sizeof(T)));
}

// strength of each ELL slot = |area/(dr.n)| of its face; -1 marks the slots
// that are not interior couplings
void amg_strength(int ne, int W, const int *nb_in, const int *fc, const double *adn, FillVec<int> &nb,
                  FillVec<double> &strength) {
    nb.resize((size_t)W * ne);          // every slot written below (first touch in parallel)
    strength.resize((size_t)W * ne);
    parallel_for((long)nb.size(), [&](long b, long e) {
        for (long s = b; s < e; s++) {
            const int j = nb_in[s];
            if (j < 0 || j >= ne) { nb[s] = -1; strength[s] = 0.0; continue; }
            const int f = fc[s] >= 0 ? fc[s] : ~fc[s];
            nb[s] = j;
            strength[s] = std::fabs(adn[f]);
        }
    });
}

// Build and upload the hierarchy of one case (mesh-only, once).
int build_case_amg(HostCase *hc) {
    if (hc->amg) return CFDL_OK;
    CaseDev &d = hc->dev;
    const int ne = hc->ne, W = hc->W, nf = hc->nf;
    // the slot tables and face planes, read back from the device
    std::vector<int> nb0((size_t)W * ne), fc((size_t)W * ne);
    std::vector<double> adn(nf);
    int st;
    if ((st = cuda_status(cudaMemcpy(nb0.data(), d.hf_nb, nb0.size() * sizeof(int), cudaMemcpyDeviceToHost)))) return st;
    if ((st = cuda_status(cudaMemcpy(fc.data(), d.hf_fc, fc.size() * sizeof(int), cudaMemcpyDeviceToHost)))) return st;
    if ((st = cuda_status(cudaMemcpy(adn.data(), d.fgeo + (size_t)FG_ADN * nf, nf * sizeof(double), cudaMemcpyDeviceToHost)))) return st;
    FillVec<int> nb;
    FillVec<double> strength;
    amg_strength(ne, W, nb0.data(), fc.data(), adn.data(), nb, strength);
    AmgHierarchy *H = new AmgHierarchy;
    AmgFineView fv{ne, W, nb.data(), strength.data()};
    if ((st = build_amg_hierarchy(fv, *H))) { delete H; return st; }
    return upload_case_amg(hc, H);
}

}  // namespace

int prepare_case_amg(CasePrep *p) {
    if (!p || p->amg) return p ? CFDL_OK : CFDL_ERR_INVALID;
    FillVec<int> nb;
    FillVec<double> strength;
    amg_strength(p->ne, p->W, p->hf_nb.data(), p->hf_fc.data(), p->fgeo.data() + (size_t)FG_ADN * p->nf, nb, strength);
    AmgHierarchy *H = new (std::nothrow) AmgHierarchy;
    if (!H) return CFDL_ERR_OOM;
    AmgFineView fv{p->ne, p->W, nb.data(), strength.data()};
    int st = build_amg_hierarchy(fv, *H);
    if (st) { delete H; return st; }
    p->amg = H;
    return CFDL_OK;
}

// The plan of a case's tail for one precision.
// limit: the shared memory it may take.
template <class T> static int build_tail_plan(const HostCase *hc, const AmgLevelDev *lev, TailPlan &plan, int *smem,
                                              int limit = kTailMaxSmem) {
    const CaseDev &d = hc->dev;
    const int lt = d.amg_tail, nl = d.nlev - lt;
    constexpr int sz = (int)sizeof(T);
    TailPlan *P = &plan;
    int at = 0;
    auto take = [&](long bytes) { const int o = at; at += (int)((bytes + 15) & ~15L); return o; };
    auto rows = [&](int l) { return l == 0 ? hc->ne : lev[l - 1].n; };
    P->nl = nl;
    P->nc = d.ncoarse;
    P->sz = take((long)P->nc * sz);
    P->sr = take((long)P->nc * sz);
    P->sminv = take((long)P->nc * P->nc * sz);
    P->minv = sz == 8 ? (const void *)d.cinv : (const void *)d.cinv32;
    if (lt == 0) {                                         // no coarse level: the mesh level is solved directly
        P->r = sz == 8 ? (const void *)d.kr : (const void *)d.fr;
        P->z = sz == 8 ? (void *)d.ks : (void *)d.fz;
    } else {
        P->r = sz == 8 ? (const void *)lev[lt - 1].r : (const void *)lev[lt - 1].r32;
        P->z = sz == 8 ? (void *)lev[lt - 1].z : (void *)lev[lt - 1].z32;
    }
    for (int b = 0; b < 2; b++) {
        P->t[b] = take(nl > 0 ? (long)rows(lt) * sz : 0);
        P->w[b] = take((long)tail_whole<T>() * sz);
    }
    for (int l = 0; l < nl; l++) {
        const AmgLevelDev &A = lev[lt + l - 1], &B = lev[lt + l];   // level lt + l and the one below
        TailLevel &v = P->lv[l];
        v.n = A.n;
        v.whole = v.n <= tail_whole<T>();
        v.R = v.whole ? v.n : (v.n + kTailCtas - 1) / kTailCtas;
        v.a = sz == 8 ? (const void *)A.a : (const void *)A.a32;
        v.rd = sz == 8 ? (const void *)A.rd : (const void *)A.rd32;
        v.dg = sz == 8 ? (const void *)A.dg : (const void *)A.dg32;
        v.nb = A.nb; v.len = A.len;
        v.agg = B.agg; v.mem = B.mem; v.mptr = B.mem_ptr;
        v.srd = take((long)v.R * sz); v.sdg = take((long)v.R * sz); v.sr = take((long)v.R * sz);
        v.slen = take(4L * v.R);
        v.sz = take((long)v.n * sz);
        v.sagg = take(4L * v.n); v.smem_ = take(4L * v.n); v.smptr = take(4L * (B.n + 1));
    }
    for (int l = nl - 1; l >= 0; l--) {                    // the small levels first: the tail level takes what is left
        TailLevel &v = P->lv[l];
        const int room = limit - at - 32, per = v.R * (sz + 4);
        v.S = std::min(lev[lt + l - 1].W, room > 0 ? room / per : 0);
        v.sa = take((long)v.R * v.S * sz);
        v.snb = take(4L * v.R * v.S);
    }
    P->total = at;
    if (at > limit) return CFDL_ERR_MESH;                  // cannot happen with kTailMaxSmem (see TailPlan)
    *smem = at;
    return CFDL_OK;
}

static int upload_hierarchy(HostCase *hc, const AmgHierarchy *H) {
    CaseDev &d = hc->dev;
    const int ne = hc->ne;
    int st;
    const int nlev = (int)H->levels.size();
    std::vector<AmgLevelDev> devl(nlev);
    for (int l = 0; l < nlev; l++) {
        const AmgHostLevel &L = H->levels[l];
        AmgLevelDev &D = devl[l];
        D.n = L.n; D.W = L.W; D.n_fine = L.n_fine; D.W_fine = L.W_fine;
        if ((st = dupload(hc, (int **)&D.nb, L.nb))) return st;
        if ((st = dupload(hc, (int **)&D.agg, L.agg))) return st;
        if ((st = dupload(hc, (int **)&D.mem_ptr, L.mem_ptr))) return st;
        if ((st = dupload(hc, (int **)&D.mem, L.mem))) return st;
        if ((st = dupload(hc, (int **)&D.g_ptr, L.g_ptr))) return st;
        if ((st = dupload(hc, (int **)&D.g_src, L.g_src))) return st;
        {
            // valid slots of each row: the builder packs a row's couplings first
            std::vector<int> len((size_t)L.n, 0);
            for (int k = 0; k < L.W; k++)
                for (int c = 0; c < L.n; c++)
                    if (L.nb[(size_t)k * L.n + c] >= 0) len[c] = k + 1;
            if ((st = dupload(hc, (int **)&D.len, len))) return st;
        }
        if ((st = dzeros(hc, &D.a, (size_t)L.W * L.n))) return st;
        if ((st = dzeros(hc, &D.a32, (size_t)L.W * L.n))) return st;
        double **v64[] = {&D.dg, &D.rd, &D.r, &D.z, &D.t};
        for (double **p : v64) if ((st = dzeros(hc, p, (size_t)L.n))) return st;
        float **v32[] = {&D.dg32, &D.rd32, &D.r32, &D.z32, &D.t32};
        for (float **p : v32) if ((st = dzeros(hc, p, (size_t)L.n))) return st;
    }
    AmgLevelDev *dlev = nullptr;
    if ((st = dupload(hc, &dlev, devl))) return st;
    const int ncoarse = nlev ? H->levels.back().n : ne;
    if (ncoarse > kAmgCoarsest) return CFDL_ERR_MESH;
    if ((st = dzeros(hc, &d.cinv, (size_t)ncoarse * ncoarse))) return st;
    if ((st = dzeros(hc, &d.cinv32, (size_t)ncoarse * ncoarse))) return st;
    if (hc->cfg.precision >= 1) {   // the FP32 mesh kernels' 16-bit neighbour offsets, used when every one fits
        const size_t nslot = (size_t)hc->W * d.ld32;
        short *nb16 = nullptr;
        unsigned *flag = nullptr, over = 0;
        if ((st = dzeros(hc, &nb16, nslot)) || (st = dzeros(hc, &flag, 1))) return st;
        k_nb16<<<(unsigned)((nslot + kTile - 1) / kTile), kTile>>>(d.hf_nb, nb16, ne, d.ld32, hc->W, flag);
        if ((st = cuda_status(cudaGetLastError()))) return st;
        if ((st = cuda_status(cudaMemcpy(&over, flag, sizeof(unsigned), cudaMemcpyDeviceToHost)))) return st;
        d.nb16 = over ? nullptr : nb16;
    }
    d.nlev = nlev;
    d.ncoarse = ncoarse;
    d.lev = dlev;
    // the tail level: the first coarse level of at most kTailRows rows (the
    // coarsest always qualifies); a case without coarse levels solves its mesh
    // level directly (tail level 0)
    d.amg_tail = 0;
    for (int l = 1; l <= nlev; l++)
        if (H->levels[l - 1].n <= kTailRows) { d.amg_tail = l; break; }
    // both plans, uploaded once: the hierarchy does not change
    std::vector<TailPlan> plans(2);
    if ((st = build_tail_plan<double>(hc, devl.data(), plans[0], &hc->tail_smem64))) return st;
    if ((st = build_tail_plan<float>(hc, devl.data(), plans[1], &hc->tail_smem32))) return st;
    TailPlan *dp = nullptr;
    if ((st = dupload(hc, &dp, plans))) return st;
    d.tail64 = dp;
    d.tail32 = dp + 1;
    return CFDL_OK;
}

// Upload a host-built hierarchy into the case, which takes ownership of it.
// After a failure the case has none and the next solve builds it again.
int upload_case_amg(HostCase *hc, AmgHierarchy *H) {
    const size_t before = hc->bytes;
    hc->amg = H;
    const int st = upload_hierarchy(hc, H);
    if (!st) return CFDL_OK;
    for (void *p : hc->amg_allocs) cudaFree(p);
    hc->amg_allocs.clear();
    hc->bytes = before;
    delete hc->amg;
    hc->amg = nullptr;
    CaseDev &d = hc->dev;
    d.nlev = d.ncoarse = d.amg_tail = 0;
    d.lev = nullptr; d.cinv = nullptr; d.cinv32 = nullptr; d.nb16 = nullptr;
    d.tail64 = d.tail32 = nullptr;
    return st;
}


int ensure_amg(cfdl_ctx *ctx) {
    bool changed = false;
    for (HostCase *hc : ctx->cases) {
        if (!hc->amg) {
            int st = build_case_amg(hc);
            if (st) return st;
            changed = true;
        }
    }
    bool all16 = ctx->index16;
    for (HostCase *hc : ctx->cases) all16 = all16 && hc->dev.nb16 != nullptr;
    if (all16 != ctx->amg_nb16) { ctx->amg_nb16 = all16; destroy_graph(ctx); }
    if (!changed && ctx->amg_lmax >= 0) return CFDL_OK;
    ctx->amg_lmax = -1;                  // until the lists below are there
    int lmax = 0;
    for (HostCase *hc : ctx->cases) lmax = std::max(lmax, hc->dev.nlev);
    ctx->amg_cells.assign(lmax + 1, WorkList());
    ctx->amg_smooth.assign(lmax + 1, WorkList());
    ctx->amg_gcells.assign(lmax + 1, WorkList());
    ctx->amg_gsmooth.assign(lmax + 1, WorkList());
    ctx->amg_restr.assign(lmax + 1, WorkList());
    ctx->amg_grestr.assign(lmax + 1, WorkList());
    ctx->amg_grouped.assign(lmax + 1, 0);
    for (int l = 0; l <= lmax; l++) {
        std::vector<int> cells, smooth, restr;
        for (HostCase *hc : ctx->cases) {
            int n = l == 0 ? hc->ne : (l <= hc->dev.nlev ? hc->amg->levels[l - 1].n : 0);
            cells.push_back(l <= hc->dev.nlev ? n : 0);
            smooth.push_back(l < hc->dev.amg_tail ? n : 0);
            restr.push_back(l >= 1 && l <= hc->dev.amg_tail ? n : 0);
        }
        plan_worklist(ctx->amg_cells[l], cells);
        plan_worklist(ctx->amg_smooth[l], smooth);
        plan_worklist(ctx->amg_restr[l], restr);
        // lanes per row: 8 when every case's level is small, else the tuned
        // cgroup (1 = one thread per row); the mesh level is always 1.  The
        // lanes order a row's sum, and they go by the context's largest case: a
        // small case beside one whose level has kGroupedRows rows or more does
        // not have the bits it has alone
        const int nmax = *std::max_element(cells.begin(), cells.end());
        const int G = l == 0 ? 1 : nmax < kGroupedRows ? kG : ctx->cgroup;
        ctx->amg_grouped[l] = G;
        if (G > 1) {
            plan_worklist(ctx->amg_gcells[l], cells, kTile / G);
            plan_worklist(ctx->amg_gsmooth[l], smooth, kTile / G);
            plan_worklist(ctx->amg_grestr[l], restr, kTile / G);
        }
    }
    std::vector<WorkList *> lists;
    for (auto *v : {&ctx->amg_cells, &ctx->amg_smooth, &ctx->amg_restr, &ctx->amg_gcells, &ctx->amg_gsmooth, &ctx->amg_grestr})
        for (WorkList &wl : *v) lists.push_back(&wl);
    int st = upload_worklists(ctx, ctx->amg_list_buf, lists);
    // the tail's shared memory, once for the launches over these lists
    if (!st) st = cuda_status(cudaFuncSetAttribute(k_v_tail<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTailMaxSmem));
    if (!st) st = cuda_status(cudaFuncSetAttribute(k_v_tail<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTailMaxSmem));
    if (!st) st = upload_case_table(ctx);
    if (!st) ctx->amg_lmax = lmax;
    return st;
}

#define ALAUNCH(name, kern, WL, ...) ALAUNCH_N(name, kern, WL, kTile, ##__VA_ARGS__)
#define ALAUNCH_N(name, kern, WL, threads, ...)                                                      \
    do {                                                                                             \
        if ((WL).ntiles > 0) {                                                                       \
            const bool p_ = ctx->prof && prof_wants(ctx, name);                                      \
            if (p_) prof_begin(ctx, name);                                                           \
            launch_k(ctx->pdl, kern, (unsigned)(WL).ntiles, (unsigned)(threads), ctx->stream,             \
                     (const CaseDev *)ctx->d_cases, (const Tile *)(WL).d_tiles, ##__VA_ARGS__);          \
            if (p_) prof_end(ctx);                                                                   \
            ctx->launches++;                                                                         \
        }                                                                                            \
    } while (0)
#define CLAUNCH(name, kern, threads)                                                                 \
    do {                                                                                             \
        const int nc_ = (int)ctx->cases.size();                                                      \
        const bool p_ = ctx->prof && prof_wants(ctx, name);                                          \
        if (p_) prof_begin(ctx, name);                                                               \
        launch_k(ctx->pdl, kern, (unsigned)nc_, (unsigned)(threads), ctx->stream,                    \
                 (const CaseDev *)ctx->d_cases, nc_);                                                \
        if (p_) prof_end(ctx);                                                                       \
        ctx->launches++;                                                                             \
    } while (0)

// The V-cycle's tail: one cluster of kTailCtas CTAs per case
template <class T> static void launch_tail(cfdl_ctx *ctx) {
    const int nc = (int)ctx->cases.size();
    if (nc == 0) return;
    int smem = 0;                       // the largest plan of the cases
    for (const HostCase *hc : ctx->cases) smem = std::max(smem, sizeof(T) == 8 ? hc->tail_smem64 : hc->tail_smem32);
    const bool p_ = ctx->prof && prof_wants(ctx, "k_v_tail");
    if (p_) prof_begin(ctx, "k_v_tail");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(nc * kTailCtas));
    cfg.blockDim = dim3((unsigned)kTailBlock);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = kTailCtas;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = ctx->pdl ? 2 : 1;
    cudaLaunchKernelEx(&cfg, k_v_tail<T>, (const CaseDev *)ctx->d_cases, nc);
    if (p_) prof_end(ctx);
    ctx->launches++;
}

// Coarse operators of every level and the coarsest inverse.
static void amg_setup_operators(cfdl_ctx *ctx, bool prepped) {
    if (!prepped) ALAUNCH("k_amg_prep0", k_amg_prep0, ctx->cells);
    for (int l = 1; l <= ctx->amg_lmax; l++) {
        switch (ctx->amg_grouped[l]) {
        case 8: ALAUNCH("k_amg_gal", k_amg_galg<8>, ctx->amg_gcells[l], l); break;
        case 4: ALAUNCH("k_amg_gal", k_amg_galg<4>, ctx->amg_gcells[l], l); break;
        case 2: ALAUNCH("k_amg_gal", k_amg_galg<2>, ctx->amg_gcells[l], l); break;
        default: ALAUNCH("k_amg_gal", k_amg_gal, ctx->amg_cells[l], l);
        }
    }
    CLAUNCH("k_amg_coarse_inv", k_amg_coarse_inv, kInvThreads);
}

// One V-cycle z_0 = M^-1 r_0 on every active case.
// The kernels of one coarse-level step at a group size (1: one thread per row)
#define GROUPED(NAME, K, WLG, WL1, ...)                                          \
    switch (G) {                                                                \
    case 8: { auto kf_ = K<T, 8>; ALAUNCH(NAME, kf_, WLG, ##__VA_ARGS__); } break; \
    case 4: { auto kf_ = K<T, 4>; ALAUNCH(NAME, kf_, WLG, ##__VA_ARGS__); } break; \
    case 2: { auto kf_ = K<T, 2>; ALAUNCH(NAME, kf_, WLG, ##__VA_ARGS__); } break; \
    default: break;                                                             \
    }

// An FP32 mesh-level kernel, two rows per thread: with 16-bit neighbour offsets
// when every case has them, else with the int32 indices
#define MESH32(NAME, K, ...)                                                                              \
    if (n16) ALAUNCH_N(NAME, (K<true, ##__VA_ARGS__>), ctx->amg_smooth[0], kTile / 2);                    \
    else ALAUNCH_N(NAME, (K<false, ##__VA_ARGS__>), ctx->amg_smooth[0], kTile / 2);

// An FP64 mesh-level kernel: two rows per thread where one row per thread would
// fill the SMs (8 CTAs of kTile threads each) more than once.  Each row's
// arithmetic is the same either way.  KE: the form of the cases with the energy
// equation (flow_fp64), in precision 1's order of sums.
#define MESH64(NAME, K1, K2, KE, ...)                                                                     \
    if (any_flow_fp64(ctx)) {                                                                             \
        if (ctx->amg_smooth[0].ntiles > 8 * 152) ALAUNCH_N(NAME, K2, ctx->amg_smooth[0], kTile / 2);      \
        else ALAUNCH(NAME, K1, ctx->amg_smooth[0]);                                                       \
    }                                                                                                     \
    if (any_ordered(ctx)) ALAUNCH(NAME, KE, ctx->amg_smooth[0], ##__VA_ARGS__);

template <class T> static void vcycle(cfdl_ctx *ctx) {
    // Large levels run one thread per row (G = 1) or a few lanes per row
    // (the autotuned cgroup); small levels run 8 lanes per row, which
    // shortens each thread's chain of loads (amg_grouped[l] = G).
    const int L = ctx->amg_lmax;
    // the FP32 mesh-level kernels read 16-bit neighbour offsets when every
    // case has them: 52 B a row instead of 64, 19% faster at 128^3; the FP64
    // sweeps did not gain by them and keep int32
    const bool n16 = ctx->amg_nb16;
    for (int l = 0; l < L; l++) {
        int G = ctx->amg_grouped[l];
        if (G > 1) {
            ALAUNCH(l ? "k_v_jac0_c" : "k_v_jac0_f", k_v_jac0<T>, ctx->amg_smooth[l], l);
            GROUPED("k_v_jac_c", k_vg_jac, ctx->amg_gsmooth[l], 0, l)
            GROUPED("k_v_resid_c", k_vg_resid, ctx->amg_gsmooth[l], 0, l)
        } else if (l == 0 && sizeof(T) == 4) {
            // FP32 mesh level: t = w D^-1 r and the first sweep from it in one
            // pass (46.6 -> 33.2 us at 128^3).  The FP64 form keeps the two
            // passes: there the fused sweep measured slower (65.0 -> 74.7 us),
            // and so did the coarse levels' in both forms.
            MESH32("k_v_jacr_f", k_v_jac_pair, false, true)
            MESH32("k_v_resid_f", k_v_resid_pair)
        } else {
            ALAUNCH(l ? "k_v_jac0_c" : "k_v_jac0_f", k_v_jac0<T>, ctx->amg_smooth[l], l);
            if (l == 0) {
                MESH64("k_v_jac_f", k_v_jac_mesh<false>, k_v_jac_pair64<false>, k_v_jac<double>, 0)
                MESH64("k_v_resid_f", k_v_resid_mesh, k_v_resid_pair64, k_v_resid_order)
            } else {
                ALAUNCH("k_v_jac_c", (k_v_jac<T>), ctx->amg_smooth[l], l);
                ALAUNCH("k_v_resid_c", (k_v_resid<T>), ctx->amg_smooth[l], l);
            }
        }
        G = ctx->amg_grouped[l + 1];
        if (G > 1) { GROUPED(l ? "k_v_restrict_c" : "k_v_restrict_f", k_vg_restrict, ctx->amg_grestr[l + 1], 0, l + 1) }
        else ALAUNCH(l ? "k_v_restrict_c" : "k_v_restrict_f", k_v_restrict<T>, ctx->amg_restr[l + 1], l + 1);
    }
    // each case's small levels and its coarsest solve, one cluster per case
    launch_tail<T>(ctx);
    for (int l = L - 1; l >= 0; l--) {
        const int G = ctx->amg_grouped[l];
        if (G > 1) {
            GROUPED("k_v_prolong_c", k_vg_prolong, ctx->amg_gsmooth[l], 0, l)
            GROUPED("k_v_jac_c", k_vg_jac, ctx->amg_gsmooth[l], 0, l)
        } else {
            // z += s P z_{l+1}; t = J(z); z = J(t)
            ALAUNCH(l ? "k_v_lift_c" : "k_v_lift_f", k_v_lift<T>, ctx->amg_smooth[l], l);
            if (l == 0 && sizeof(T) == 4) {
                MESH32("k_v_jac_f", k_v_jac_pair, true, false)
                MESH32("k_v_jac_f", k_v_jac_pair, false, false)
            } else if (l == 0) {
                MESH64("k_v_jac_f", k_v_jac_mesh<true>, k_v_jac_pair64<true>, (k_v_jac<double, true>), 0)
                MESH64("k_v_jac_f", k_v_jac_mesh<false>, k_v_jac_pair64<false>, k_v_jac<double>, 0)
            } else {
                ALAUNCH("k_v_jac_c", (k_v_jac<T, true>), ctx->amg_smooth[l], l);
                ALAUNCH("k_v_jac_c", (k_v_jac<T>), ctx->amg_smooth[l], l);
            }
        }
    }
}

void launch_pc_mean(cfdl_ctx *ctx);

#define RED ctx->cellsv.d_case_first, ctx->cellsv.d_case_ntiles, ctx->d_partials
// the mixed form's FP64 norms only end its loops: their tiles need not keep the
// order of the FP32 sums (an outer iteration of precision 3 at 128^3: 2915 us with
// cellsv's tiles, 2897 so)
#define REDW ctx->cellsw.d_case_first, ctx->cellsw.d_case_ntiles, ctx->d_partials
#define REDS ctx->cellss.d_case_first, ctx->cellss.d_case_ntiles, ctx->d_partials
#define REDS32 ctx->cellss.d_case_first, ctx->cellss.d_case_ntiles, (float *)ctx->d_partials
#define RED32 ctx->cellsv.d_case_first, ctx->cellsv.d_case_ntiles, (float *)ctx->d_partials

// What the pressure solve needs of its matrix, once the matrix exists: the
// multigrid operators (AMG), or the level-0 FP32 copies and 1/ap (mixed
// Jacobi); the FP64 Jacobi form needs nothing.  In solve_uvwp this runs
// beside the momentum solve (cfdl_graph.cu): it depends on dc only.
void pressure_operators(cfdl_ctx *ctx, bool prepped) {
    const cfdl_config &c = ctx->cases[0]->cfg;
    prepped = prepped && c.precision >= 1;       // as launch_coef_p_matrix
    if (c.precond == 1) amg_setup_operators(ctx, prepped);
    else if (c.precision >= 1 && !prepped) ALAUNCH("k_amg_prep0", k_amg_prep0, ctx->cells);
}

// FP64 AMG-PCG: zero-mean right-hand side, x = 0 (operators already built)
void apc_init(cfdl_ctx *ctx) {
    launch_pc_mean(ctx);
    ALAUNCH("k_apc_init", k_apc_init, ctx->cellsv, RED);
}

// one preconditioned CG iteration
void apc_iter(cfdl_ctx *ctx) {
    vcycle<double>(ctx);
    if (ctx->cellss.ntiles) {
        ALAUNCH("k_apc_rz", k_apc_rz<true>, ctx->cellss, REDS);
        ALAUNCH("k_apc_p", k_apc_p, ctx->cells);
        ALAUNCH("k_apc_q", k_apc_q<true>, ctx->cellss, REDS);
        ALAUNCH("k_apc_x", k_apc_x<true>, ctx->cellss, REDS);
        return;
    }
    ALAUNCH("k_apc_rz", k_apc_rz<false>, ctx->cellsv, RED);
    ALAUNCH("k_apc_p", k_apc_p, ctx->cellsv);
    ALAUNCH("k_apc_q", k_apc_q<false>, ctx->cellsv, RED);
    ALAUNCH("k_apc_x", k_apc_x<false>, ctx->cellsv, RED);
}

int solve_pressure_amg(cfdl_ctx *ctx) {
    int st = ensure_amg(ctx);
    if (st) return st;
    apc_init(ctx);
    int cap = 0;
    for (auto *hc : ctx->cases) cap = std::max(cap, hc->cfg.solve_mode == 0 ? hc->cfg.nit : hc->cfg.tight_maxit);
    int it = 0, maxit = 0;
    while (it < cap) {
        const int chunk = poll_chunk(it, ctx->last_iters_p);
        for (int k = 0; k < chunk && it < cap; k++, it++) apc_iter(ctx);
        int a = poll_kind(ctx, 1, &maxit);
        if (a < 0) return CFDL_ERR_CUDA;
        if (a == 0) break;
    }
    ctx->last_iters_p = maxit;
    return cuda_status(cudaGetLastError());
}


// ------------------------------------------------------------------------
// Mixed precision: FP64 outer residual and refinement around an FP32 inner
// PCG (FP32 SpMV, preconditioner, vectors and dot-product accumulation).
// ------------------------------------------------------------------------
namespace {

enum { CNT_M0 = 15 };   // shares the last counter slot only with itself

// outer start: r64 = b - mean, x = 0
__global__ void __launch_bounds__(kTile) k_mx_init(const CaseDev *__restrict__ cases, const Tile *__restrict__ tiles,
                                                   const int *__restrict__ cfirst, const int *__restrict__ cnt, double *partials) {
    CFDL_PDL_WAIT();
    const Tile t = tiles[blockIdx.x];
    const CaseDev &C = cases[t.c];
    SolveScalars *S = C.sc;
    const int tile0 = cfirst[t.c], ntiles = cnt[t.c];
    if (S->halted) return;
    double v[2] = {0, 0};
    FOR_CELLS(t) {
        const double r = C.b[i] - S->mean_b;
        C.kr[i] = r; C.phic[i] = 0.0;
        v[0] += r * r; v[1] += C.b[i] * C.b[i];
    }
    __shared__ double s[2];
    if (case_sums<2>(v, &C.counters[CNT_A0], partials, tile0, ntiles, s)) {
        if (threadIdx.x == 0) {
            S->r0norm_p = S->rnorm_p = sqrt(s[0]);
            S->mass_imbalance = sqrt(s[1]);
            S->iters_p = 0; S->status_p = 0; S->outer_p = 0;
            S->tol_p = (C.solve_mode == 0 ? C.rtol_p : C.tight_rtol) * S->r0norm_p;
            S->active_p = S->r0norm_p > S->tol_p && (C.solve_mode == 0 ? C.nit : C.tight_maxit) > 0;
            if (!isfinite(S->r0norm_p)) { S->active_p = 0; S->status_p = CFDL_ERR_NONFINITE; }
        }
    }
}

// inner start: fr = (float) r64, fx = 0; ||fr|| in FP32
__global__ void __launch_bounds__(kTile) k_mx_start(const CaseDev *__restrict__ cases, const Tile *__restrict__ tiles,
                                                    const int *__restrict__ cfirst, const int *__restrict__ cnt, float *partials) {
    CFDL_PDL_WAIT();
    const Tile t = tiles[blockIdx.x];
    const CaseDev &C = cases[t.c];
    SolveScalars *S = C.sc;
    const int tile0 = cfirst[t.c], ntiles = cnt[t.c];
    if (!S->active_p) return;
    float v[1] = {0.f};
    FOR_CELLS(t) {
        const float r = narrow_f32(C.kr[i]);
        C.fr[i] = r; C.fx[i] = 0.f;
        v[0] += r * r;
    }
    __shared__ float s[1];
    if (case_sums<1>(v, &C.counters[CNT_A1], partials, tile0, ntiles, s)) {
        if (threadIdx.x == 0) {
            const float rn = sqrtf(s[0]);
            // inner tolerance: the reference's drop in mode 0; when tight, half the
            // drop still needed to reach the FP64 target, but no finer than FP32
            // iterates track the true residual (1e-5) and no coarser than 0.5
            const float need = rn > 0.f ? (float)(S->tol_p / (double)rn) : 1.f;
            const float eps = C.solve_mode == 0 ? (float)C.rtol_p : fminf(0.5f, fmaxf(1e-5f, 0.5f * need));
            S->rnorm32 = rn;
            S->tol32 = eps * rn;
            S->rz32 = 0.f;
            S->iters32 = 0;
            S->active32 = rn > 0.f && isfinite(rn);
        }
    }
}

// z = M^-1 r for the Jacobi preconditioner (the AMG form uses the V-cycle)
__global__ void __launch_bounds__(kTile) k_mx_jacobi(const CaseDev *__restrict__ cases, const Tile *__restrict__ tiles) {
    CFDL_PDL_WAIT();
    const Tile t = tiles[blockIdx.x];
    const CaseDev &C = cases[t.c];
    if (!C.sc->active32) return;
    FOR_CELLS(t) C.fz[i] = C.fr[i] * C.frap_p[i];
}

template <bool kSpl>
__global__ void __launch_bounds__(kTile) k_mx_rz(const CaseDev *__restrict__ cases, const Tile *__restrict__ tiles,
                                                 const int *__restrict__ cfirst, const int *__restrict__ cnt, float *partials) {
    CFDL_PDL_WAIT();
    const Tile t = tiles[blockIdx.x];
    const CaseDev &C = cases[t.c];
    SolveScalars *S = C.sc;
    const int tile0 = cfirst[t.c], ntiles = cnt[t.c];
    if (!S->active32) return;
    __shared__ float s[1];
    bool last;
    if constexpr (kSpl) {
        float a[1] = {0}, b[1] = {0};
        const int i = split_row(t);
        if (i < t.last) {
            // cg_rz_rows' roundings: a pair's second product is rounded by itself
            const float r = C.fr[i], z = C.fz[i];
            const bool second = threadIdx.x / (kTile / kSplit) % 2;
            a[0] = second ? __fmul_rn(r, z) : r;
            b[0] = second ? 1.f : z;
        }
        last = split_sums<1>(a, b, &C.counters[CNT_A2], partials, tile0, ntiles, s);
    } else {
        float v[1] = {cg_rz_rows(C.fr, C.fz, t)};
        last = case_sums<1>(v, &C.counters[CNT_A2], partials, tile0, ntiles, s);
    }
    if (last) {
        if (threadIdx.x == 0) {
            S->beta32 = S->iters32 == 0 || S->rz32 == 0.f ? 0.f : s[0] / S->rz32;
            S->rz32 = s[0];
            if (!isfinite(s[0])) S->active32 = 0;
        }
    }
}

__global__ void __launch_bounds__(kTile) k_mx_p(const CaseDev *__restrict__ cases, const Tile *__restrict__ tiles) {
    CFDL_PDL_WAIT();
    const Tile t = tiles[blockIdx.x];
    const CaseDev &C = cases[t.c];
    const SolveScalars *S = C.sc;
    if (!S->active32) return;
    cg_p_rows<float>(C.fz, C.fp, S->iters32 == 0, S->beta32, t);
}

// q = A p; alpha = rz / (p, q).  Bound by the latency of its gathers: six CTAs
// per SM (40 registers) instead of the four of the compiler's 62 took a mixed
// pressure solve on 176^3 cells from 12560 to 12285 us; seven and eight
// 12390.  With int32 indices 40 registers would spill.
template <bool k16, bool kSpl>
__global__ void __launch_bounds__(kTile, k16 ? 6 : 4) k_mx_q(const CaseDev *__restrict__ cases, const Tile *__restrict__ tiles,
                                                const int *__restrict__ cfirst, const int *__restrict__ cnt, float *partials) {
    CFDL_PDL_WAIT();
    const Tile t = tiles[blockIdx.x];
    const CaseDev &C = cases[t.c];
    SolveScalars *S = C.sc;
    const int tile0 = cfirst[t.c], ntiles = cnt[t.c];
    if (!S->active32) return;
    const LP<float> P = level<float>(C, 0);
    const float *p = C.fp;
    __shared__ float s[1];
    bool last;
    if constexpr (kSpl) {
        float a[1] = {0.f}, b[1] = {0.f};
        const int i = split_row(t);
        if (i < t.last) {
            b[0] = row_amul_mesh<k16>(P, p, i);
            a[0] = p[i];
            C.fq[i] = b[0];
        }
        last = split_sums<1>(a, b, &C.counters[CNT_A3], partials, tile0, ntiles, s);
    } else {
        // rows in pairs (pair_slots); then (p, q), each thread its rows 256 apart in
        // row order, which is the order of the FP32 sums
        __shared__ __align__(8) float qs[kMixedRows * kTile];   // solve_pressure_prepared and append_uvwp refuse wider tiles
        const int tid = (int)threadIdx.x;
        for (int i = t.first + 2 * tid; i < t.last; i += 2 * kTile) {
            const float2 y = pair_amul_mesh<k16>(P, p, i);
            *(float2 *)&C.fq[i] = y;
            *(float2 *)&qs[i - t.first] = y;
        }
        __syncthreads();
        float v[1] = {0.f};
        FOR_CELLS(t) v[0] += p[i] * qs[i - t.first];
        last = case_sums<1>(v, &C.counters[CNT_A3], partials, tile0, ntiles, s);
    }
    if (last) {
        if (threadIdx.x == 0) {
            if (!(s[0] > 0.f) || !isfinite(s[0])) S->active32 = 0;
            else S->alpha32 = S->rz32 / s[0];
        }
    }
}

template <bool kSpl>
__global__ void __launch_bounds__(kTile) k_mx_x(const CaseDev *__restrict__ cases, const Tile *__restrict__ tiles,
                                                const int *__restrict__ cfirst, const int *__restrict__ cnt, float *partials) {
    CFDL_PDL_WAIT();
    const Tile t = tiles[blockIdx.x];
    const CaseDev &C = cases[t.c];
    SolveScalars *S = C.sc;
    const int tile0 = cfirst[t.c], ntiles = cnt[t.c];
    if (!S->active32) return;
    __shared__ float s[1];
    bool last;
    if constexpr (kSpl) {
        float a[1] = {0}, b[1] = {0};
        const int i = split_row(t);
        if (i < t.last) {
            const float al = S->alpha32, x = C.fx[i], p = C.fp[i], r = C.fr[i] - al * C.fq[i];
            C.fx[i] = x + al * p;
            C.fr[i] = a[0] = b[0] = r;
        }
        last = split_sums<1>(a, b, &C.counters[CNT_A4], partials, tile0, ntiles, s);
    } else {
        float v[1] = {cg_x_rows<float>(C.fx, C.fp, C.fr, C.fq, S->alpha32, t)};
        last = case_sums<1>(v, &C.counters[CNT_A4], partials, tile0, ntiles, s);
    }
    if (last) {
        if (threadIdx.x == 0) {
            const float rn = sqrtf(s[0]);
            S->rnorm32 = rn;
            S->iters32 += 1;
            const int cap = C.solve_mode == 0 ? C.nit : C.tight_maxit;
            S->active32 = rn > S->tol32 && isfinite(rn) && S->iters32 < cap;
        }
    }
}

// x += (double) fx
__global__ void __launch_bounds__(kTile) k_mx_apply(const CaseDev *__restrict__ cases, const Tile *__restrict__ tiles) {
    CFDL_PDL_WAIT();
    const Tile t = tiles[blockIdx.x];
    const CaseDev &C = cases[t.c];
    if (!C.sc->active_p) return;
    FOR_CELLS(t) C.phic[i] = C.phic[i] + widen_f64(C.fx[i]);
}

// FP64 true residual r = (b - mean) - A x and the outer stopping test
template <bool kSpl>
__global__ void __launch_bounds__(kTile) k_mx_res(const CaseDev *__restrict__ cases, const Tile *__restrict__ tiles,
                                                  const int *__restrict__ cfirst, const int *__restrict__ cnt, double *partials) {
    CFDL_PDL_WAIT();
    const Tile t = tiles[blockIdx.x];
    const CaseDev &C = cases[t.c];
    SolveScalars *S = C.sc;
    const int tile0 = cfirst[t.c], ntiles = cnt[t.c];
    if (!S->active_p) return;
    __shared__ double s[1];
    bool last;
    if constexpr (kSpl) {
        double a[1] = {0}, b[1] = {0};
        const int i = split_row(t);
        if (i < t.last) {
            const LP<double> P = level<double>(C, 0);
            const double y = P.W == 6 ? amul_order<6, false>(P, C.phic, i) : P.W == 4 ? amul_order<4, false>(P, C.phic, i) : amul<double>(P, C.phic, i);
            a[0] = b[0] = (C.b[i] - S->mean_b) - y;
            C.kr[i] = a[0];
        }
        last = split_sums<1>(a, b, &C.counters[CNT_M0], partials, tile0, ntiles, s);
    } else {
        // two rows per step, both rows' loads before either store
        double v[1] = {0};
        const LP<double> P = level<double>(C, 0);
        const double mb = S->mean_b;
        FOR_ROW_PAIRS(t) {
            double r0 = 0.0, r1 = 0.0;
            if (ok0) r0 = (C.b[i0] - mb) - amul<double>(P, C.phic, i0);
            if (ok1) r1 = (C.b[i1] - mb) - amul<double>(P, C.phic, i1);
            if (ok0) { C.kr[i0] = r0; v[0] += r0 * r0; }
            if (ok1) { C.kr[i1] = r1; v[0] += r1 * r1; }
        }
        last = case_sums<1>(v, &C.counters[CNT_M0], partials, tile0, ntiles, s);
    }
    if (last) {
        if (threadIdx.x == 0) {
            const double rn = sqrt(s[0]);
            S->rnorm_p = rn;
            S->outer_p += 1;
            S->iters_p += S->iters32;
            int act = rn > S->tol_p;
            if (!isfinite(rn)) { act = 0; S->status_p = CFDL_ERR_NONFINITE; }
            else if (act && S->outer_p >= kMixedMaxOuter) { act = 0; if (C.solve_mode == 1) S->status_p = CFDL_ERR_ITER_CAP; }
            S->active_p = act;
        }
    }
}

}  // namespace

// mixed form: FP32 operator copies (+ coarse operators), FP64 start
void mx_init(cfdl_ctx *ctx) {
    launch_pc_mean(ctx);
    ALAUNCH("k_mx_init", k_mx_init, ctx->cellsw, REDW);
}
void mx_start(cfdl_ctx *ctx) { ALAUNCH("k_mx_start", k_mx_start, ctx->cellsv, RED32); }
void mx_inner_iter(cfdl_ctx *ctx) {
    if (ctx->cases[0]->cfg.precond == 1) vcycle<float>(ctx);
    else ALAUNCH("k_mx_jacobi", k_mx_jacobi, ctx->cellsv);
    const bool n16 = ctx->amg_nb16;
    if (ctx->cellss.ntiles) {
        ALAUNCH("k_mx_rz", k_mx_rz<true>, ctx->cellss, REDS32);
        ALAUNCH("k_mx_p", k_mx_p, ctx->cells);
        if (n16) ALAUNCH("k_mx_q", (k_mx_q<true, true>), ctx->cellss, REDS32);
        else ALAUNCH("k_mx_q", (k_mx_q<false, true>), ctx->cellss, REDS32);
        ALAUNCH("k_mx_x", k_mx_x<true>, ctx->cellss, REDS32);
        return;
    }
    ALAUNCH("k_mx_rz", k_mx_rz<false>, ctx->cellsv, RED32);
    ALAUNCH("k_mx_p", k_mx_p, ctx->cellsv);
    if (n16) ALAUNCH("k_mx_q", (k_mx_q<true, false>), ctx->cellsv, RED32);
    else ALAUNCH("k_mx_q", (k_mx_q<false, false>), ctx->cellsv, RED32);
    ALAUNCH("k_mx_x", k_mx_x<false>, ctx->cellsv, RED32);
}
void mx_finish(cfdl_ctx *ctx) {
    ALAUNCH("k_mx_apply", k_mx_apply, ctx->cellsv);
    if (ctx->cellss.ntiles) ALAUNCH("k_mx_res", k_mx_res<true>, ctx->cellss, REDS);
    else ALAUNCH("k_mx_res", k_mx_res<false>, ctx->cellsw, REDW);
}

int solve_pressure_mixed(cfdl_ctx *ctx) {
    int st;
    if (ctx->cases[0]->cfg.precond == 1 && (st = ensure_amg(ctx))) return st;
    mx_init(ctx);
    int cap = 0;
    for (auto *hc : ctx->cases) cap = std::max(cap, hc->cfg.solve_mode == 0 ? hc->cfg.nit : hc->cfg.tight_maxit);
    for (int outer = 0; outer < kMixedMaxOuter; outer++) {
        mx_start(ctx);
        int it = 0, maxit = 0;
        while (it < cap) {
            const int chunk = poll_chunk(it, ctx->last_iters_p);
            for (int k = 0; k < chunk && it < cap; k++, it++) mx_inner_iter(ctx);
            int a = poll_kind(ctx, 2, &maxit);
            if (a < 0) return CFDL_ERR_CUDA;
            if (a == 0) break;
        }
        ctx->last_iters_p = maxit;
        mx_finish(ctx);
        int a = poll_kind(ctx, 3, nullptr);
        if (a < 0) return CFDL_ERR_CUDA;
        if (a == 0) break;
    }
    return cuda_status(cudaGetLastError());
}
#undef RED
#undef RED32

}  // namespace cfdl

extern "C" int cfdl_amg_index_bytes(const cfdl_ctx *ctx) {
    return ctx ? (ctx->amg_nb16 && !ctx->cases.empty() && ctx->cases[0]->cfg.precision >= 1 ? 2 : 4) : -1;
}

extern "C" int cfdl_amg_info(cfdl_ctx *ctx, int maxlev, int *nlev, int *n, int *W) {
    using namespace cfdl;
    if (!ctx || ctx->cases.empty() || !nlev || maxlev < 0) return CFDL_ERR_INVALID;
    const HostCase *hc = ctx->cases[0];
    const int L = hc->amg ? (int)hc->amg->levels.size() : 0;
    *nlev = L;
    for (int l = 0; l <= L && l <= maxlev; l++) {
        if (n) n[l] = l == 0 ? hc->ne : hc->amg->levels[l - 1].n;
        if (W) W[l] = l == 0 ? hc->W : hc->amg->levels[l - 1].W;
    }
    return CFDL_OK;
}

extern "C" int cfdl_set_tail_smem(cfdl_ctx *ctx, int bytes) {
    using namespace cfdl;
    int st = check_ctx(ctx);
    if (st) return st;
    if (bytes < 0 || ctx->cases[0]->cfg.precond != 1) return CFDL_ERR_INVALID;
    if ((st = ensure_amg(ctx))) return st;
    const int limit = bytes == 0 || bytes > kTailMaxSmem ? kTailMaxSmem : bytes;
    std::vector<TailPlan> plans(2 * ctx->cases.size());
    std::vector<int> smem(2 * ctx->cases.size());
    for (size_t c = 0; c < ctx->cases.size(); c++) {
        const HostCase *hc = ctx->cases[c];
        std::vector<AmgLevelDev> lev(hc->dev.nlev);
        if (!lev.empty() && (st = cuda_status(cudaMemcpy(lev.data(), hc->dev.lev, lev.size() * sizeof(AmgLevelDev), cudaMemcpyDeviceToHost))))
            return st;
        if (build_tail_plan<double>(hc, lev.data(), plans[2 * c], &smem[2 * c], limit) ||
            build_tail_plan<float>(hc, lev.data(), plans[2 * c + 1], &smem[2 * c + 1], limit))
            return CFDL_ERR_INVALID;                       // less than the plans need beside the slots
    }
    if ((st = cuda_status(cudaStreamSynchronize(ctx->stream)))) return st;
    destroy_graph(ctx);                                    // captured launches carry the size
    for (size_t c = 0; c < ctx->cases.size(); c++) {
        HostCase *hc = ctx->cases[c];
        if ((st = cuda_status(cudaMemcpyAsync((void *)hc->dev.tail64, &plans[2 * c], 2 * sizeof(TailPlan), cudaMemcpyHostToDevice, ctx->stream))))
            return st;
        hc->tail_smem64 = smem[2 * c];
        hc->tail_smem32 = smem[2 * c + 1];
    }
    return cuda_status(cudaStreamSynchronize(ctx->stream));
}
