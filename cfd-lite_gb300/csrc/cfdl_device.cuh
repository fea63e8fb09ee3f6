// cfdl_device.cuh -- device helpers shared by the kernels of libcfdgpu.
#pragma once
#include "cfdl_internal.h"

namespace cfdl {

// First statement of every kernel the launch macros start with programmatic
// dependent launch: the grid may be scheduled while its predecessor in the
// stream is finishing, and waits here until that predecessor has completed
// and its writes are visible (a no-op when launched the ordinary way).
#define CFDL_PDL_WAIT() asm volatile("griddepcontrol.wait;" ::: "memory")

// Deterministic sums over the kTile threads of a block: K sums of v land in
// shared out[0..K-1] (written by the first warp; the others read it after a barrier).  The order is a
// fixed tree over each warp's 32 values (lane l with l+16, then l+8, ...),
// then the warps' sums in warp order.
//
// FP64: through shared memory.  GB300 issues 2 FP64 thread-instructions per SM
// per clock, so a warp's FP64 add costs 16 clocks whatever its lanes hold: a
// shuffle tree in every warp spends 48 warp-adds per value (8 warps x 5
// steps, then the warps), more than the rows' own arithmetic when a thread has
// few rows.  Here each thread stores its K values and warp k alone forms the
// eight warps' trees of value k with every lane busy -- 4 adds for the first
// step of all eight trees, 2, 1, 1 and 1 for the next -- and the eight sums of
// all K values are added in order by one warp, a lane to a value: 9 K + 8
// warp-adds, the same sums in the same order.  (With each warp adding its own
// value's eight, 17 K, an FP64 outer iteration took 0.5% longer at 128^3, 0.8%
// in a batch, 2.7% with the energy solve on 77^3 cells.)
// One warp's part of the sum of v[0..kTile-1] (shared): the shuffle trees of the
// block's kTile / 32 warps, packed so that they take 9 warp adds; the sum of
// warp w's tree is left in dst[w].
__device__ __forceinline__ void warp_trees(const double *v, double *dst) {
    static_assert(kTile / 32 == 8, "the packing below is for eight warps");
    const int lane = threadIdx.x & 31;
    const bool b8 = (lane & 8) != 0, b4 = (lane & 4) != 0;
    // x[j]: lane l & 15 of tree w = 2 j + (lane >> 4) after its first step
    double x[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int at = (2 * j + (lane >> 4)) * 32 + (lane & 15);
        x[j] = v[at] + v[at + 16];
    }
    // second step: lanes with bit 8 clear take trees j, the others j + 1
    double y[2];
#pragma unroll
    for (int j = 0; j < 2; j++) {
        const double own = b8 ? x[2 * j + 1] : x[2 * j], other = b8 ? x[2 * j] : x[2 * j + 1];
        y[j] = own + __shfl_xor_sync(0xffffffffu, other, 8);
    }
    double z = (b4 ? y[1] : y[0]) + __shfl_xor_sync(0xffffffffu, b4 ? y[0] : y[1], 4);
    z += __shfl_xor_sync(0xffffffffu, z, 2);
    z += __shfl_xor_sync(0xffffffffu, z, 1);
    // the sum of warp w = 2 j + h, j = (bit 8) + 2 (bit 4), is in lane 16 h + 8 (j & 1) + 4 (j >> 1)
    if ((lane & 3) == 0) dst[2 * ((lane >> 3 & 1) + 2 * (lane >> 2 & 1)) + (lane >> 4)] = z;
}
// out[k] is written by thread k of the first warp
template <int K>
__device__ __forceinline__ void block_sums(double (&v)[K], double *out) {
    constexpr int kWarps = kTile / 32;
    __shared__ double sm[K][kTile], ws[K][kWarps];
#pragma unroll
    for (int k = 0; k < K; k++) sm[k][threadIdx.x] = v[k];
    __syncthreads();
    for (int k = threadIdx.x >> 5; k < K; k += kWarps) warp_trees(sm[k], ws[k]);
    __syncthreads();
    // the trees' sums in warp order, all values in one warp's lanes: 8 adds for
    // the K of them, not 8 for each
    if (threadIdx.x < K) {
        double s = 0.0;
#pragma unroll
        for (int w = 0; w < kWarps; w++) s += ws[threadIdx.x][w];
        out[threadIdx.x] = s;
    }
}
// FP32: a shuffle tree per warp, then the warps' sums in warp order (the order is
// part of the FP32 forms' results).  The trees of N values fold together: at
// each step a lane keeps half of the values and hands the other half over, so
// six values take 8 shuffles and adds instead of 30 (0.2% of an FP32 outer
// iteration).  Returns the sum of value k if `mine`: one lane per value.
template <int N, int O = 16, class T>
__device__ __forceinline__ T warp_sums(const T (&v)[N], int lane, int &k, bool &mine) {
    if constexpr (N == 1) {
        T z = v[0];
#pragma unroll
        for (int o = O; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
        k = 0;
        mine = (lane & (2 * O - 1)) == 0;
        return z;
    } else {
        constexpr int H = (N + 1) / 2;
        const bool up = (lane & O) != 0;
        T y[H];
#pragma unroll
        for (int j = 0; j < H; j++) {
            const T hi = j + H < N ? v[j + H < N ? j + H : 0] : v[j];
            y[j] = (up ? hi : v[j]) + __shfl_xor_sync(0xffffffffu, up ? v[j] : hi, O);
        }
        const T z = warp_sums<H, O / 2>(y, lane, k, mine);
        if (up) k += H;
        mine = mine && k < N;
        return z;
    }
}
template <int K>
__device__ __forceinline__ void block_sums(float (&v)[K], float *out) {
    __shared__ float sm[K][kTile / 32];
    int k;
    bool mine;
    const float z = warp_sums<K>(v, threadIdx.x & 31, k, mine);
    if (mine) sm[k][threadIdx.x >> 5] = z;
    __syncthreads();
    if (threadIdx.x < K) {
        float s = 0;
        for (int w = 0; w < kTile / 32; w++) s += sm[threadIdx.x][w];
        out[threadIdx.x] = s;
    }
}

// The second half of case_sums: the sums of a case's `ntiles` partials per value,
// thread-strided in a fixed order with four independent accumulators (so the
// loads overlap instead of forming one dependent chain), then the block sum.
template <int K, class T>
__device__ __forceinline__ void partial_sums(T (&v)[K], const T *part, int ntiles, T *s) {
    T a1[K], a2[K], a3[K];
#pragma unroll
    for (int k = 0; k < K; k++) v[k] = a1[k] = a2[k] = a3[k] = 0;
    int i = threadIdx.x;
    for (; i + 3 * kTile < ntiles; i += 4 * kTile)
#pragma unroll
        for (int k = 0; k < K; k++) {
            const T *p = part + (size_t)k * ntiles + i;
            v[k] += __ldcg(p);
            a1[k] += __ldcg(p + kTile);
            a2[k] += __ldcg(p + 2 * kTile);
            a3[k] += __ldcg(p + 3 * kTile);
        }
    for (; i < ntiles; i += kTile)
#pragma unroll
        for (int k = 0; k < K; k++) v[k] += __ldcg(&part[(size_t)k * ntiles + i]);
#pragma unroll
    for (int k = 0; k < K; k++) v[k] = (v[k] + a1[k]) + (a2[k] + a3[k]);
    block_sums<K>(v, s);
    __syncthreads();
}

// The K sums of v over all tiles of a case, in shared s[0..K-1] of the case's
// last tile to finish; returns true (to the whole block) in that tile only.
// tile0, ntiles: the case's tiles in the launch's work list; the case's
// partials are K planes of ntiles values from partials[tile0 * kNPart].
// Every tile publishes its partials and then raises the case's counter; the
// tile that brings it to ntiles sums all partials in tile order, so the
// result does not depend on which tile came last, and clears the counter.
// One thread writes the partials, fences and raises the counter: the fence
// then waits for those few stores only, not for the block's vector stores,
// which are read by later kernels alone.
template <int K, class T>
__device__ __forceinline__ bool case_sums(T (&v)[K], int *counter, T *partials, int tile0, int ntiles, T *s) {
    __shared__ int is_last;
    T *part = partials + (size_t)tile0 * kNPart;
    const int tile = (int)blockIdx.x - tile0;
    block_sums<K>(v, s);
    if (threadIdx.x < 32) __syncwarp();      // s is the first warp's
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < K; k++) __stcg(&part[(size_t)k * ntiles + tile], s[k]);
        __threadfence();
        const bool last = atomicAdd(counter, 1) == ntiles - 1;
        if (last) { *counter = 0; __threadfence(); }
        is_last = last;
    }
    __syncthreads();
    if (!is_last) return false;
    partial_sums<K>(v, part, ntiles, s);
    return true;
}

// Sums of a launch whose blocks each take up to M of a case's tiles in turn (a
// merged list), tile by tile in the order of case_sums: the same bits.  A block
// pays its start (tile, case, scalars: three dependent trips to L2), its two
// barriers, its fence and its count once for M tiles: an outer iteration with
// the energy solve (256 cells a tile) at 77^3 took 3530 us and takes 3200.  The
// FP32 flow solves (1024 cells a tile) did not gain by it.  After each tile
// put_sums files its values; merged_sums ends the block as case_sums does, over
// the partials of all `nsub` tiles of the case.  kSub: the most tiles a block
// may take.
template <class T> constexpr int kSumWidth = sizeof(T) == 4 ? kTile / 32 : kTile;
template <int K, class T, int kSub> __device__ __forceinline__ T *sum_buf() {
    __shared__ T buf[kSub * K * kSumWidth<T>];
    return buf;
}
template <int K, int kSub> __device__ __forceinline__ void put_sums(float (&v)[K], int m) {
    int k;
    bool mine;
    const float z = warp_sums<K>(v, threadIdx.x & 31, k, mine);
    if (mine) sum_buf<K, float, kSub>()[(m * K + k) * kSumWidth<float> + (threadIdx.x >> 5)] = z;
}
template <int K, int kSub> __device__ __forceinline__ void put_sums(double (&v)[K], int m) {
    double *buf = sum_buf<K, double, kSub>() + m * K * kSumWidth<double>;
#pragma unroll
    for (int k = 0; k < K; k++) buf[k * kSumWidth<double> + threadIdx.x] = v[k];
}
template <int K, class T, int kSub>
__device__ __forceinline__ bool merged_sums(int nm, int *counter, T *partials, int tile0, int ntiles, int M, int nsub, T *s) {
    __shared__ int is_last;
    T *part = partials + (size_t)tile0 * M * kNPart;
    const int at = ((int)blockIdx.x - tile0) * M, lane = threadIdx.x & 31;
    T *buf = sum_buf<K, T, kSub>();
    __syncthreads();
    if constexpr (sizeof(T) == 8) {
        for (int q = threadIdx.x >> 5; q < nm * K; q += kTile / 32)
            warp_trees(buf + q * kSumWidth<T>, buf + q * kSumWidth<T>);   // read before it is written
        __syncthreads();
    }
    if (threadIdx.x < 32) {
        for (int q = lane; q < nm * K; q += 32) {
            T x = 0;
#pragma unroll
            for (int w = 0; w < kTile / 32; w++) x += buf[q * kSumWidth<T> + w];
            __stcg(&part[(size_t)(q % K) * nsub + at + q / K], x);
        }
        __syncwarp();
        if (lane == 0) {
            __threadfence();
            const bool last = atomicAdd(counter, 1) == ntiles - 1;
            if (last) { *counter = 0; __threadfence(); }
            is_last = last;
        }
    }
    __syncthreads();
    if (!is_last) return false;
    T v[K];
    partial_sums<K>(v, part, nsub, s);
    return true;
}

// the tiles u of a block's tile t in a merged list, counted in nm, at most kSub
#define FOR_SUBTILES(u, t, mg, nm, kSub)                                                               \
    int nm = 0;                                                                                        \
    for (Tile u{(t).c, (t).first, (kSub) == 1 ? (t).last : min((t).last, (t).first + (mg).rows), (t).pad}; nm < (kSub) && u.first < (t).last; \
         u.first += (mg).rows, u.last = min((t).last, u.last + (mg).rows), nm++)
// case_sums of a plain list (kSub 1) or merged_sums of a merged one
template <int K, int kSub, class T>
__device__ __forceinline__ bool tile_sums(T (&v)[K], int nm, int *counter, T *partials, int tile0, int ntiles, const Merge &mg, int ne, T *s) {
    if constexpr (kSub == 1) return case_sums<K>(v, counter, partials, tile0, ntiles, s);
    else return merged_sums<K, T, kSub>(nm, counter, partials, tile0, ntiles, mg.M, (ne + mg.rows - 1) / mg.rows, s);
}

// A small context leaves most SMs idle with 1024 cells to a block, and each
// thread there goes through its four rows one after the other.  In a split list
// kSplit blocks share a tile: block j takes the columns of threads 64 j to
// 64 j + 63, one row per thread (split_row), and split_sums chains each column's
// products in row order, forms the two warps' trees and files them, so the sums
// have the bits of case_sums.  a, b: the factors of the row's share of each sum.
// At 32^3 cells a launch of the FP64 A ph went from 17 to 10 us, at 24^3 the
// FP32 one from 10 to 6.6.
__device__ __forceinline__ int split_row(const Tile &t) {
    constexpr int cols = kTile / kSplit;
    return t.first + (int)threadIdx.x / cols * kTile + t.pad * cols + (int)threadIdx.x % cols;
}
template <class T> __device__ __forceinline__ T fma_rn(T a, T b, T c) {
    if constexpr (sizeof(T) == 4) return __fmaf_rn(a, b, c);
    else return __fma_rn(a, b, c);
}
template <int K, class T>
__device__ __forceinline__ bool split_sums(const T (&a)[K], const T (&b)[K], int *counter, T *partials, int tile0, int nblocks, T *s) {
    constexpr int cols = kTile / kSplit, kWarps = kTile / 32;
    __shared__ T sa[K][kTile], sb[K][kTile];
    __shared__ int is_last;
    const int tid = (int)threadIdx.x, ntiles = nblocks / kSplit, at = (int)blockIdx.x - tile0;
#pragma unroll
    for (int k = 0; k < K; k++) { sa[k][tid] = a[k]; sb[k][tid] = b[k]; }
    __syncthreads();
    T *part = partials + (size_t)tile0 * kNPart;           // [K][ntiles][kWarps]
    if (tid < cols) {
        T v[K];
#pragma unroll
        for (int k = 0; k < K; k++) v[k] = 0;
#pragma unroll
        for (int g = 0; g < kSplit; g++)
#pragma unroll
            for (int k = 0; k < K; k++) v[k] = fma_rn(sa[k][g * cols + tid], sb[k][g * cols + tid], v[k]);
        int k;
        bool mine;
        const T z = warp_sums<K>(v, tid & 31, k, mine);
        if (mine) __stcg(&part[((size_t)k * ntiles + at / kSplit) * kWarps + at % kSplit * (cols / 32) + (tid >> 5)], z);
    }
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        const bool last = atomicAdd(counter, 1) == nblocks - 1;
        if (last) { *counter = 0; __threadfence(); }
        is_last = last;
    }
    __syncthreads();
    if (!is_last) return false;
    T v[K];
#pragma unroll
    for (int k = 0; k < K; k++) v[k] = 0;
    for (int i = tid; i < ntiles; i += kTile)
#pragma unroll
        for (int k = 0; k < K; k++) {
            const T *q = part + ((size_t)k * ntiles + i) * kWarps;
            T w[kWarps], x = 0;
#pragma unroll
            for (int u = 0; u < kWarps; u++) w[u] = __ldcg(q + u);
#pragma unroll
            for (int u = 0; u < kWarps; u++) x += w[u];
            v[k] += x;
        }
    block_sums<K>(v, s);
    __syncthreads();
    return true;
}

// Start of a case's momentum solve from s[0..2] = sum b'^2 and s[3..5] =
// sum r^2 per component (the whole block calls it; one thread per component).
constexpr int kCntMomInit = 0;           // its last-tile counter
__device__ __forceinline__ void mom_start(const CaseDev &C, const double *s) {
    const int q = threadIdx.x;
    if (q >= 3) return;
    SolveScalars *S = C.sc;
    const int cap = C.solve_mode == 0 ? C.nit : C.tight_maxit;
    S->bnorm[q] = sqrt(s[q]);
    S->r0norm[q] = S->rnorm[q] = sqrt(s[3 + q]);
    S->rho[q] = s[3 + q];
    S->alpha[q] = 1.0; S->omega[q] = 1.0; S->beta[q] = 0.0; S->half[q] = 0;
    S->iters[q] = 0; S->status[q] = 0;
    S->tol[q] = C.solve_mode == 0 ? C.rtol_u * S->r0norm[q] : C.tight_rtol * S->bnorm[q];
    S->active[q] = (S->r0norm[q] > S->tol[q]) && cap > 0;
    if (!isfinite(S->r0norm[q]) || !isfinite(S->bnorm[q])) { S->active[q] = 0; S->status[q] = CFDL_ERR_NONFINITE; }
}

__device__ __forceinline__ int face_of(int fc) { return fc >= 0 ? fc : ~fc; }

// Row i of an ELL operator, y_c = diag*x_c[i] - sum_k a[k][i]*x_c[nb[k][i]]
// for NC vectors x_c = x + c*stride.  Neighbours outside [0, n) (halos,
// padding) contribute nothing.  W is a compile-time width so the index and
// coefficient loads of all slots are issued before any arithmetic; invalid
// slots read x[i] with a zero coefficient instead of branching.
template <int W, int NC, class T>
__device__ __forceinline__ void ell_row_w(const int *__restrict__ nb, const T *__restrict__ a, T diag,
                                          const T *x, int stride, int n, int i, T (&y)[NC]) {
    int j[W];
    T c[W];
#pragma unroll
    for (int k = 0; k < W; k++) {
        const int jj = __ldg(&nb[k * n + i]);
        const bool ok = (unsigned)jj < (unsigned)n;
        j[k] = ok ? jj : i;
        c[k] = ok ? a[k * n + i] : (T)0;
    }
#pragma unroll
    for (int q = 0; q < NC; q++) {
        const T *xq = x + q * stride;
        T s = diag * xq[i];
#pragma unroll
        for (int k = 0; k < W; k++) s -= c[k] * xq[j[k]];
        y[q] = s;
    }
}

template <int NC, class T>
__device__ __forceinline__ void ell_row(const int *__restrict__ nb, const T *__restrict__ a, T diag, const T *x,
                                        int stride, int n, int W, int i, T (&y)[NC]) {
    if (W == 6) { ell_row_w<6, NC, T>(nb, a, diag, x, stride, n, i, y); return; }
    if (W == 4) { ell_row_w<4, NC, T>(nb, a, diag, x, stride, n, i, y); return; }
#pragma unroll
    for (int q = 0; q < NC; q++) y[q] = diag * x[q * stride + i];
    // wide rows (coarse levels): four slots per step, their index, coefficient
    // and vector loads issued together instead of one dependent chain per slot
    for (int k0 = 0; k0 < W; k0 += 4) {
        int jj[4];
        T ak[4];
#pragma unroll
        for (int u = 0; u < 4; u++) jj[u] = k0 + u < W ? nb[(k0 + u) * n + i] : -1;
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const bool ok = (unsigned)jj[u] < (unsigned)n;
            ak[u] = ok ? a[(k0 + u) * n + i] : (T)0;
            if (!ok) jj[u] = i;
        }
#pragma unroll
        for (int q = 0; q < NC; q++) {
            T xv[4];
#pragma unroll
            for (int u = 0; u < 4; u++) xv[u] = x[q * stride + jj[u]];
#pragma unroll
            for (int u = 0; u < 4; u++) y[q] -= ak[u] * xv[u];
        }
    }
}

// -x when neg, else x: a sign-bit flip in the integer pipe (no FP64 op)
__device__ __forceinline__ double flip_sign(double x, bool neg) {
    return __longlong_as_double(__double_as_longlong(x) ^ ((long long)neg << 63));
}
// max(x, 0) for non-NaN x, decided on the bit pattern (no FP64 op); -0 -> 0
__device__ __forceinline__ double positive_part(double x) {
    return __double_as_longlong(x) > 0 ? x : 0.0;
}
// -x when neg, else x, for FP32
__device__ __forceinline__ float flip_sign_f(float x, bool neg) {
    return __uint_as_float(__float_as_uint(x) ^ ((unsigned)neg << 31));
}

// FP64 <-> FP32 from the IEEE 754 binary64 / binary32 bit layouts, in the
// integer pipe: GB300 executes the hardware conversion instructions at its
// FP64 rate (2 per SM per clock), so a kernel that is meant to spend no FP64
// work converts this way.
//
// binary64 -> binary32, rounded to nearest (ties to even) on the 29 dropped
// mantissa bits; results below the binary32 normal range become a signed
// zero, overflow gives infinity, NaN stays NaN.
__device__ __forceinline__ float narrow_f32(double x) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const unsigned sign = (unsigned)(b >> 32) & 0x80000000u;
    const int e = (int)((b >> 52) & 0x7ffu);
    const unsigned long long m = b & 0xfffffffffffffull;
    if (e == 0x7ff) return __uint_as_float(sign | 0x7f800000u | (m ? 0x400000u : 0u));
    const int fe = e - 1023 + 127;
    if (fe <= 0) return __uint_as_float(sign);
    if (fe >= 255) return __uint_as_float(sign | 0x7f800000u);
    unsigned r = ((unsigned)fe << 23) | (unsigned)(m >> 29);
    const unsigned rem = (unsigned)(m & 0x1fffffffu);
    if (rem > 0x10000000u || (rem == 0x10000000u && (r & 1u))) r += 1u;   // a carry moves into the exponent
    return __uint_as_float(sign | r);
}
// binary32 -> binary64: exact for normal values; a binary32 subnormal gives a
// signed zero
__device__ __forceinline__ double widen_f64(float f) {
    const unsigned u = __float_as_uint(f);
    const unsigned long long sign = (unsigned long long)(u & 0x80000000u) << 32;
    const unsigned e = (u >> 23) & 0xffu, m = u & 0x7fffffu;
    if (e == 0) return __longlong_as_double((long long)sign);
    const unsigned long long de = e == 0xffu ? 0x7ffull : (unsigned long long)(e - 127 + 1023);
    return __longlong_as_double((long long)(sign | (de << 52) | ((unsigned long long)m << 29)));
}

// b / a, correctly rounded, for a row's quotients.  The built-in FP64 division
// is about 18 FP64 instructions; this is 7.  The reciprocal of a starts from
// the FP32 one (22 bits; FP32 and integer instructions only) and takes two
// Newton steps, y += y (1 - a y); the quotient q = b y is then corrected by its
// remainder, q += y (b - a q) (Markstein, IBM J. Res. Dev. 34, 1990).
//
// Why it rounds correctly, with significands 1 <= a, b < 2: the second step's y
// is within half an ulp of 1/a times 1 + 2^-32 (its exact value within 2^-86),
// so |a y - 1| <= 2^-54 a (1 + 2^-32), and b y is off b/a by less than one ulp.
// Where b/a is next to the middle of two numbers, q is therefore one of these
// two, half an ulp away; its remainder is exact, and the corrected value is off
// by less than half an ulp times 2^-54 a (1 + 2^-32).  The middle itself is at
// least 1/(2^54 A) from b/a with A = 2^52 a the integer significand (both over
// A, two integers that differ): 2/a against a/2 in the same unit, so the
// rounding falls on the right side for every a below 2 (1 - 2^-33).  A
// significand nearer to 2 can fail (1 / (2 - 2^-52) would come out 0.5), so all
// whose upper 20 bits are ones take the division, and so do numbers near the
// ends of either format's range, zeros and non-finite values.
__device__ __forceinline__ bool rcp_in_range(double a) {      // 2^-100 <= |a| < 2^101, significand below 2 - 2^-20
    const unsigned h = (unsigned)__double2hiint(a), e = h >> 20 & 0x7ffu;
    return e - (1023u - 100u) <= 200u && (h & 0xfffffu) != 0xfffffu;
}
// 1 / a within half an ulp times 1 + 2^-32, for a in range
__device__ __forceinline__ double rcp_near(double a) {
    const double y0 = widen_f64(__fdividef(1.0f, narrow_f32(a)));
    const double y1 = __fma_rn(y0, __fma_rn(-a, y0, 1.0), y0);
    return __fma_rn(y1, __fma_rn(-a, y1, 1.0), y1);
}
__device__ __forceinline__ double div_rn(double b, double a) {
    const unsigned e = (unsigned)(__double2hiint(b) >> 20) & 0x7ffu;
    if (!rcp_in_range(a) || e - (1023u - 500u) > 1000u) return b / a;
    const double y = rcp_near(a), q = __dmul_rn(b, y);
    return __fma_rn(__fma_rn(-a, q, b), y, q);
}

// the mesh level of the pressure multigrid: weights of the two sweeps
constexpr double kOmega = 0.557;   // first sweep
constexpr double kOmega2 = 1.242;  // second sweep

// What the pressure solve needs of row i of its matrix (diagonal ap, couplings
// a): the diagonal's inverse under the sweep weights and, in the mixed forms,
// the FP32 copies, converted in the integer pipe (GB300 runs the hardware
// conversions at its FP64 rate).
__device__ __forceinline__ void prep_row(const CaseDev &C, int i, double ap, const double (&a)[kMaxW]) {
    const bool mixed = C.precision >= 1;
    const double rd = div_rn(kOmega, ap);
    C.rap_p[i] = rd;
    if (!mixed) C.rap2_p[i] = rd * (kOmega2 / kOmega);
    if (mixed) {
        C.fdiag_p[i] = narrow_f32(ap);
        C.frap_p[i] = narrow_f32(rd);
#pragma unroll
        for (int k = 0; k < kMaxW; k++)
            if (k < C.W) C.fanb_p[k * C.ld32 + i] = narrow_f32(a[k]);
    }
}

}  // namespace cfdl
