// cfdl_noalloc.cu -- pressure-correction solve that allocates nothing.
//
// Some hosts cannot call cudaMalloc: a Fortran code whose device memory is
// owned by another runtime or pool, a process that runs under a fixed memory
// budget, or a caller inside a loop where allocation is not allowed.  For
// them cfdl_solve_pc_noalloc solves the pressure-correction system with
// arrays the caller already holds on the device, in the reference's CSR
// layout, and keeps all of its own working storage (Krylov vectors, reduction
// partials, scalars) in one file-scope __device__ array of fixed size.
//
// Algorithm: the Jacobi-preconditioned CG of the context path (set_a_0 then
// CG from zero on the zero-mean right-hand side), the whole solve in one
// cooperative launch.  At up to 131072 rows an iteration's arithmetic is
// 1-4 us and the rest of it latency.  As three launches (A p with its dot
// product; x, r, z with theirs; p) with a host poll every few iterations it
// took 24 us an iteration at 729 rows, 28 at 64000 and 33 at 125000.  Here a
// thread owns a row: its coefficients, x, r, z and p stay in registers, and an
// iteration is two all-reduces with one exchange of z and p through L2 between
// them: 7.0, 12.3 to 13.7 and 15.0 to 15.8 us by the board.  About one CTA per
// SM, so that every SM's FP64 pipe (2 instructions per clock) takes an equal
// share.
//
// An all-reduce is barrier and sum in one: each CTA publishes its partials as
// 8-byte words that carry 32 bits of the value and the step's number, and
// every CTA polls all of them and sums them in CTA order (deterministic, the
// same in all CTAs).  The polls are bounded: a CTA that gives up sets its
// failure and leaves, and so do the others after it.
#include "cfdl_internal.h"
#include "cfdl_device.cuh"
#include <algorithm>
#include <climits>
#include <cstddef>

namespace cfdl {
namespace {

constexpr int kNaMaxCells = 131072;                 // CFDL_NOALLOC_MAX_CELLS
constexpr int kNaMaxCtas = 512;                     // CTAs of a solve (their partials' slots)
constexpr int kNaMinBlock = 128, kNaMaxBlock = 1024;
constexpr int kNaW = 6;                             // couplings of a row kept in registers
constexpr int kNaVals = 3;                          // values of the widest all-reduce
constexpr int kNaPolls = 1 << 22;                   // polls of a wait, about a second; and four for every half-face,
                                                    // all of which may lie in the row that the others wait for
constexpr int kNaRows = 8;                          // rows per thread where the SMs are too few for one

struct NoAllocScratch {
    double z[kNaMaxCells], p[kNaMaxCells];          // what neighbouring rows read
    ulonglong2 slot[2][kNaVals][kNaMaxCtas];        // partials of two consecutive all-reduces
    // how CG ended
    double rnorm, tol;
    int iters, bad;
    int fail;           // why CG stopped early: 0 it did not, 1 a non-finite value, 2 p.Ap <= 0, 3 a wait ran out
};

// Shared by every call on a device and kept between calls.
static __device__ __align__(256) NoAllocScratch g_na_scratch;

// The scalars of CG, one copy per CTA (every CTA forms the same ones).
struct NaScalars {
    double mean, rz, alpha, beta, rr, tol2;    // rr = ||r||^2, stopped at tol2 = (rtol ||r0||)^2
    int iters, bad, fail, active;
};
// The preconditioner is z = r (1 / d): a correctly rounded r / d took up to 0.6 us
// more of 13 an iteration at 64000 rows, and the solution's error against 64
// bits is the same to four digits with either (9^3 to 50^3 rows, tolerances of
// 1e-11 to 1e-13).  1 / d of a subnormal d is no number, so a matrix near the
// ends of the range (by its first diagonal entry) has its diagonal taken times
// this power of two: z and p are then scaled by it and x is not.
__device__ __forceinline__ double na_scale(double d) {
    const unsigned e = (unsigned)(__double2hiint(d) >> 20) & 0x7ffu;
    const int k = e < 1023u - 900u ? 200 : e > 1023u + 900u ? -200 : 0;
    return __hiloint2double((1023 + k) << 20, 0);
}
template <int NT> struct NaShared {
    double sm[kNaVals][NT], res[kNaVals];
    NaScalars c;
};

// Sums v over all CTAs; thread 0 of each then runs fin(sums), which updates
// the block's scalars: one thread, because an FP64 division or square root is
// 600 clocks of latency for one warp but 2500 when sixteen warps repeat it.
// False when a wait ran out.  step counts the all-reduces from 1.  With
// exchange, what the block wrote to global memory before is visible to every
// CTA after.
template <int K, int NT, class F>
__device__ __forceinline__ bool na_all_sum(NoAllocScratch *S, NaShared<NT> &B, const double (&v)[K], unsigned step,
                                           int polls, bool exchange, F fin) {
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nt = blockDim.x, n = gridDim.x;
    ulonglong2(*slot)[kNaMaxCtas] = S->slot[step & 1];
#pragma unroll
    for (int k = 0; k < K; k++) B.sm[k][tid] = v[k];
    __syncthreads();
    const unsigned long long tag = (unsigned long long)step << 32;
    if (wid < K) {                                  // a warp per value (blocks have at least four)
        constexpr int kPer = NT / 32;
        double a[kPer];
#pragma unroll
        for (int u = 0; u < kPer; u++) a[u] = u * 32 < nt ? B.sm[wid][u * 32 + lane] : 0.0;
#pragma unroll
        for (int o = kPer / 2; o > 0; o >>= 1)
#pragma unroll
            for (int u = 0; u < o; u++) a[u] += a[u + o];
        double s = a[0];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (lane == 0) {
            if (exchange) __threadfence();          // the block's writes, ordered before by the barrier
            const unsigned long long b = (unsigned long long)__double_as_longlong(s);
            ulonglong2 *w = &slot[wid][blockIdx.x];
            asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(&w->x), "l"(tag | (b >> 32)) : "memory");
            asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(&w->y), "l"(tag | (b & 0xffffffffull)) : "memory");
        }
    }
    __syncthreads();                                // sm is read; it takes the CTAs' partials next
    bool ok = true;
#pragma unroll
    for (int k = 0; k < K; k++)
        for (int cta = tid; cta < n; cta += nt) {
            const ulonglong2 *w = &slot[k][cta];
            unsigned long long x = 0, y = 0;
            int it = 0;
            do {
                asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(x) : "l"(&w->x) : "memory");
                asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(y) : "l"(&w->y) : "memory");
            } while (((x >> 32) != step || (y >> 32) != step) && ++it < polls);
            ok = ok && it < polls;
            if (cta < NT) B.sm[k][cta] = __longlong_as_double((long long)(x << 32 | (y & 0xffffffffull)));
        }
    if (exchange) __threadfence();
    ok = __syncthreads_and(ok);
    if (!ok) return false;
    if (wid < K) {
        double s0 = 0.0, s1 = 0.0;
        for (int i = lane; i < n; i += 64) {
            s0 += B.sm[wid][i];
            if (i + 32 < n) s1 += B.sm[wid][i + 32];
        }
        s0 += s1;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s0 += __shfl_xor_sync(0xffffffffu, s0, o);
        if (lane == 0) B.res[wid] = s0;
    }
    if (K > 1) __syncthreads();
    if (tid == 0) fin(B.res);
    __syncthreads();
    return true;
}

// The solve.  Thread t of the grid owns rows t, t + T, ... (T threads; R rows
// at most).  Indices are checked against ne and nh; a bad one is recorded and
// its access skipped.  NT: the largest block (1024 threads have 64 registers
// each, and spill; 512 have 128).
template <int R, int NT>
__global__ void __launch_bounds__(NT) k_na_solve(NoAllocScratch *S, int ne, int nh, const int *ef1, const int *idx,
                                                 const double *ap, const double *anb, const double *b, double *phic,
                                                 double rtol, int maxit, int polls) {
    const int T = (int)(gridDim.x * blockDim.x), t0 = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    __shared__ NaShared<NT> B;
    NaScalars &c = B.c;
    unsigned step = 0;
    double x[R], r[R], z[R], p[R], q[R], d[R], rd[R], a[R][kNaW];
    int j[R][kNaW], h0[R], h1[R];
    double s1[1] = {0.0}, s2[2], s3[3] = {0.0, 0.0, 0.0};
    const double scale = na_scale(ap[0]);
#pragma unroll
    for (int u = 0; u < R; u++) {
        const int i = t0 + u * T;
        x[u] = r[u] = z[u] = p[u] = q[u] = 0.0;
        d[u] = rd[u] = 1.0;
        h0[u] = h1[u] = 0;
#pragma unroll
        for (int k = 0; k < kNaW; k++) { a[u][k] = 0.0; j[u][k] = -1; }
        if (i >= ne) continue;
        r[u] = b[i];
        s1[0] += r[u];
        d[u] = ap[i];
        rd[u] = 1.0 / (d[u] * scale);
        h0[u] = idx[i] - 1;
        h1[u] = idx[i + 1] - 1;
        if (h0[u] < 0 || h1[u] > nh || h0[u] > h1[u]) { s3[2] = 1.0; h0[u] = h1[u] = 0; }
        for (int h = h0[u]; h < h1[u]; h++) {
            const int enb = (int)((unsigned)ef1[h] >> 5), lf = ef1[h] & 31;
            if (lf && (enb < 1 || enb > ne)) s3[2] = 1.0;
        }
#pragma unroll
        for (int k = 0; k < kNaW; k++) {
            const int h = h0[u] + k;
            if (h >= h1[u]) continue;
            const int enb = (int)((unsigned)ef1[h] >> 5), lf = ef1[h] & 31;
            if (lf && enb >= 1 && enb <= ne) { j[u][k] = enb - 1; a[u][k] = anb[h]; }
        }
    }
    auto give_up = [&]() { S->fail = 3; };
    if (!na_all_sum<1>(S, B, s1, ++step, polls, false, [&](const double *s) { c.mean = s[0] / ne; })) { give_up(); return; }
#pragma unroll
    for (int u = 0; u < R; u++) {
        const int i = t0 + u * T;
        if (i >= ne) continue;
        r[u] -= c.mean;
        z[u] = r[u] * rd[u];
        __stcg(&S->z[i], z[u]);
        s3[0] += r[u] * r[u];
        s3[1] += r[u] * z[u];
    }
    if (!na_all_sum<3>(S, B, s3, ++step, polls, true, [&](const double *s) {
            c.rz = s[1];
            c.rr = s[0];
            c.tol2 = rtol * rtol * s[0];
            c.beta = 0.0;
            c.iters = c.bad = 0;
            // a zero or non-finite diagonal entry makes z = r/ap, and so (r, z), non-finite
            c.fail = isfinite(c.rr) && isfinite(c.rz) ? 0 : 1;
            c.active = c.rr > c.tol2 && maxit > 0 && !c.fail;
            if (c.active && s[2] > 0.0) { c.bad = 1; c.active = 0; }
        })) { give_up(); return; }
    bool first = true;
    while (c.active) {
        // p = z + beta p, formed for the row and its neighbours (their p is not
        // written yet); q = A p
        const double beta = c.beta;
        s1[0] = 0.0;
#pragma unroll
        for (int u = 0; u < R; u++) {
            const int i = t0 + u * T;
            if (i >= ne) continue;
            double zn[kNaW], pn[kNaW];
#pragma unroll
            for (int k = 0; k < kNaW; k++) {
                const bool in = j[u][k] >= 0;
                zn[k] = in ? __ldcg(&S->z[j[u][k]]) : 0.0;
                pn[k] = in && !first ? __ldcg(&S->p[j[u][k]]) : 0.0;
            }
            p[u] = z[u] + beta * p[u];
            // two sums of three slots: half the dependent chain
            double s = d[u] * p[u], s4 = 0.0;
#pragma unroll
            for (int k = 0; k < kNaW; k += 2) {
                s -= a[u][k] * (zn[k] + beta * pn[k]);
                s4 += a[u][k + 1] * (zn[k + 1] + beta * pn[k + 1]);
            }
            s -= s4;
            for (int h = h0[u] + kNaW; h < h1[u]; h++) {    // rows of more couplings
                const int enb = (int)((unsigned)ef1[h] >> 5), lf = ef1[h] & 31;
                if (lf) s -= anb[h] * (__ldcg(&S->z[enb - 1]) + (first ? 0.0 : beta * __ldcg(&S->p[enb - 1])));
            }
            q[u] = s;
            s1[0] += p[u] * s;
        }
        first = false;
        if (!na_all_sum<1>(S, B, s1, ++step, polls, false, [&](const double *s) {
                // only runs while ||r|| is above the tolerance, where an SPD system has p.Ap > 0
                if (!isfinite(s[0])) { c.fail = 1; c.active = 0; }
                else if (!(s[0] > 0.0)) { c.fail = 2; c.active = 0; }
                else c.alpha = c.rz / s[0];
            })) { give_up(); return; }
        if (!c.active) break;
        const double alpha = c.alpha;
        s2[0] = s2[1] = 0.0;
#pragma unroll
        for (int u = 0; u < R; u++) {
            const int i = t0 + u * T;
            if (i >= ne) continue;
            x[u] += alpha * p[u];
            r[u] -= alpha * q[u];
            z[u] = r[u] * rd[u];
            __stcg(&S->z[i], z[u]);
            __stcg(&S->p[i], p[u]);
            s2[0] += r[u] * r[u];
            s2[1] += r[u] * z[u];
        }
        if (!na_all_sum<2>(S, B, s2, ++step, polls, true, [&](const double *s) {
                c.rr = s[0];
                c.iters += 1;
                c.beta = c.rz != 0.0 ? s[1] / c.rz : 0.0;
                c.rz = s[1];
                if (!isfinite(c.rr) || !isfinite(c.rz)) c.fail = 1;
                c.active = c.rr > c.tol2 && c.iters < maxit && !c.fail;
            })) { give_up(); return; }
    }
#pragma unroll
    for (int u = 0; u < R; u++)
        if (t0 + u * T < ne) phic[t0 + u * T] = x[u];
    if (t0 == 0) {
        S->rnorm = sqrt(c.rr); S->tol = sqrt(c.tol2);
        S->iters = c.iters; S->bad = c.bad;
        if (c.fail) S->fail = c.fail;
    }
}

// Device address of the scratch array on the current device.  The host-side
// symbol is only a stand-in, not a device address, so the address is asked
// of the runtime with the device current.  The first call on a device loads
// the library's device code there (make it before any stream capture); later
// calls only read the runtime's table.  Asking on every call, rather than
// keeping the first answer, keeps the address right after a cudaDeviceReset,
// which gives the device a new context and may place the array elsewhere.
int na_scratch(NoAllocScratch **out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_status(e);
    void *ptr = nullptr;
    e = cudaGetSymbolAddress(&ptr, g_na_scratch);
    if (e != cudaSuccess) return cuda_status(e);
    *out = static_cast<NoAllocScratch *>(ptr);
    return CFDL_OK;
}

}  // namespace
}  // namespace cfdl

using namespace cfdl;

// On at most max_sms SMs (0: all of the device's)
static int na_solve(int ne, int nh, const int *ef2nb1, const int *ef2nb_idx, const double *ap, const double *anb,
                    const double *b, double *phic, double rtol, int maxit, int max_sms, int *iters, double *rnorm) {
    if (ne <= 0 || nh <= 0 || !ef2nb1 || !ef2nb_idx || !ap || !anb || !b || !phic || !(rtol > 0) || maxit < 0)
        return CFDL_ERR_INVALID;
    if (ne > kNaMaxCells) return CFDL_ERR_TOO_LARGE;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) { cudaGetLastError(); return CFDL_ERR_NO_DEVICE; }
    NoAllocScratch *S = nullptr;
    int st = na_scratch(&S);
    if (st) return st;
    const cudaStream_t s0 = 0;
    // about one CTA per SM; where the SMs are fewer than the rows need at one row
    // a thread, a thread takes eight (its rows spill: an iteration on 10 SMs has
    // eight rows' loads in a chain anyway)
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return cuda_status(e);
    if (max_sms > 0 && sms > max_sms) sms = max_sms;
    if (sms > kNaMaxCtas) sms = kNaMaxCtas;
    const int rows = (long long)sms * kNaMaxBlock >= ne ? 1 : kNaRows;
    const int threads = (ne + rows - 1) / rows;
    int block = ((threads + sms - 1) / sms + 31) & ~31;
    if (block < kNaMinBlock) block = kNaMinBlock;
    if (block > kNaMaxBlock) return CFDL_ERR_TOO_LARGE;
    const int grid = (threads + block - 1) / block;
    const int polls = (int)std::min<long long>(kNaPolls + 4LL * nh, INT_MAX);
    // step numbers start over with every call: no slot may hold one
    e = cudaMemsetAsync(S->slot, 0, sizeof(NoAllocScratch) - offsetof(NoAllocScratch, slot), s0);
    if (e != cudaSuccess) return cuda_status(e);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.stream = s0;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;       // every CTA resident: they wait for one another
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    e = cudaLaunchKernelEx(&cfg, rows > 1 ? k_na_solve<kNaRows, 1024> : block > 512 ? k_na_solve<1, 1024> : k_na_solve<1, 512>, S, ne, nh, ef2nb1,
                           ef2nb_idx, ap, anb, b, phic, rtol, maxit, polls);
    struct { double rnorm, tol; int iters, bad, fail; } end = {};
    static_assert(offsetof(NoAllocScratch, fail) == offsetof(NoAllocScratch, rnorm) + 24, "the end record is copied whole");
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(&end, &S->rnorm, 28, cudaMemcpyDeviceToHost, s0);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s0);
    if (e != cudaSuccess) return cuda_status(e);
    if (end.fail == 3) return CFDL_ERR_CUDA;
    if (iters) *iters = end.iters;
    if (rnorm) *rnorm = end.rnorm;
    if (end.bad) return CFDL_ERR_INVALID;
    if (end.fail == 1 || !isfinite(end.rnorm)) return CFDL_ERR_NONFINITE;
    if (end.fail == 2) return CFDL_ERR_BREAKDOWN;
    if (end.rnorm > end.tol) return CFDL_ERR_ITER_CAP;       // stopped at maxit above the tolerance
    return CFDL_OK;
}

extern "C" int cfdl_solve_pc_noalloc(int ne, int nh, const int *ef2nb1, const int *ef2nb_idx, const double *ap,
                                     const double *anb, const double *b, double *phic, double rtol, int maxit,
                                     int *iters, double *rnorm) {
    return na_solve(ne, nh, ef2nb1, ef2nb_idx, ap, anb, b, phic, rtol, maxit, 0, iters, rnorm);
}

extern "C" int cfdl_solve_pc_noalloc_sms(int ne, int nh, const int *ef2nb1, const int *ef2nb_idx, const double *ap,
                                         const double *anb, const double *b, double *phic, double rtol, int maxit,
                                         int sms, int *iters, double *rnorm) {
    if (sms < 1) return CFDL_ERR_INVALID;
    return na_solve(ne, nh, ef2nb1, ef2nb_idx, ap, anb, b, phic, rtol, maxit, sms, iters, rnorm);
}
