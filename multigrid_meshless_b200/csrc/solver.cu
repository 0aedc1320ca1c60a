// solver.cu -- convergent Poisson solve for the pinned system
//     A p = b,  A = lap_Poison with row 0 replaced by p[0] = 0,
// the system whose solution the reference's multigrid_Poisson_solver
// (fractional_step_solver.h:150-196, p -= p[0] after each sweep) aims at.
//
// Preconditioner: one V-cycle in precision T (double or float)
//   smoother   Chebyshev polynomial in D^-1 A on interior rows, every step
//              followed by an exact solve of the boundary rows (a boundary
//              row couples only to itself and interior nodes, kdtree_functions.h:141-149);
//   transfer   interior residuals restricted with the RBF interpolation
//              weights of create_restriction_matrix (mesh_functions.h:533-600)
//              built for every non-boundary coarse row; corrections prolongated
//              with create_prolongation_matrix weights (mesh_functions.h:602-670)
//              built for every fine row, shifted so the pinned node gets none;
//   coarsest   dense inverse of the pinned coarsest operator.
// Outer: flexible GMRES in FP64 (residuals, Krylov basis, solution updates).
#include <cmath>

#include <type_traits>

#include "krylov.cuh"
#include "coop.cuh"
#include "rows.cuh"
#include "stencil.cuh"

namespace mgm {

template <int BS>
__device__ __forceinline__ double block_sum_d(double v, double *sm)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x < 32) {
        v = threadIdx.x < BS / 32 ? sm[threadIdx.x] : 0.0;
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    }
    __syncthreads();
    return v;
}

// ---------------------------------------------------------------------------
// smoother
// ---------------------------------------------------------------------------
// Row work of the V-cycle kernels, shared by the one-operation kernels and
// the fused coarse-level V-cycle (k_coarse_vcycle), which therefore give the
// same bits.

// A boundary row by the lanes of a warp: its stencil (fetch: the first 64
// slots), then its exact solve from the current e (value: lane 0).  A
// boundary row couples only to itself and interior nodes, so rows can be
// updated in place; the rows are stored row-major [nbl][k].
template <class T>
struct BndRow {
    static constexpr int Q = 2;
    int i = 0, w = 0, c[Q];
    T a[Q], di;
    __device__ __forceinline__ void fetch(int row, int lane, int nbl, const int *__restrict__ list, int k,
                                          const int *__restrict__ bidx, const T *__restrict__ bA,
                                          const T *__restrict__ dinv)
    {
        w = min(row, nbl - 1);
        i = ldk(list + w);
#pragma unroll
        for (int q = 0; q < Q; q++) {
            const long o = (long)w * k + min(lane + 32 * q, k - 1);
            c[q] = ldk(bidx + o);
            a[q] = ldk(bA + o);
        }
        di = ldk(dinv + i);
    }
    __device__ __forceinline__ T value(int lane, int k, const int *__restrict__ bidx, const T *__restrict__ bA,
                                       const T *r, const T *e) const
    {
        T v[Q], s = T(0);
        const T ri = __ldcg(r + i), ei = __ldcg(e + i);
#pragma unroll
        for (int q = 0; q < Q; q++) v[q] = __ldcg(e + c[q]);
#pragma unroll
        for (int q = 0; q < Q; q++)
            if (lane + 32 * q < k) s = fma_rn(a[q], v[q], s);
        for (int j = lane + 32 * Q; j < k; j += 32)
            s = fma_rn(__ldg(bA + (long)w * k + j), __ldcg(e + __ldg(bidx + (long)w * k + j)), s);
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        return fma_rn(ri - s, di, ei);
    }
};

// The same by 8 lanes, g = lane & 7, for the levels of kVecMinRows rows and
// more, where a warp per row is several waves of CTAs: 23k boundary rows of the
// 64^3 cube take 7.1 us a launch, 9.3 with a warp per row; on the small levels
// it is the longer chain (5.4k rows: 5.0 us against 4.2).  Lane g stands for
// lanes g, g + 8, g + 16 and g + 24 of the warp, so the sum has the same bits.
template <class T>
struct BndRow8 {
    int i = 0, w = 0, c[2][4];
    T a[2][4], di;
    __device__ __forceinline__ void fetch(int row, int g, int nbl, const int *__restrict__ list, int k,
                                          const int *__restrict__ bidx, const T *__restrict__ bA,
                                          const T *__restrict__ dinv)
    {
        w = min(row, nbl - 1);
        i = ldk(list + w);
#pragma unroll
        for (int q = 0; q < 2; q++)
            if (32 * q < k) {
#pragma unroll
                for (int v = 0; v < 4; v++) {
                    const long o = (long)w * k + min(g + 8 * v + 32 * q, k - 1);
                    c[q][v] = ldk(bidx + o);
                    a[q][v] = ldk(bA + o);
                }
            }
        di = ldk(dinv + i);
    }
    __device__ __forceinline__ T value(int g, int k, const int *__restrict__ bidx, const T *__restrict__ bA,
                                       const T *r, const T *e) const
    {
        T x[2][4], s[4] = {T(0), T(0), T(0), T(0)};
        const T ri = __ldcg(r + i), ei = __ldcg(e + i);
#pragma unroll
        for (int q = 0; q < 2; q++)
            if (32 * q < k) {
#pragma unroll
                for (int v = 0; v < 4; v++) x[q][v] = __ldcg(e + c[q][v]);
            }
#pragma unroll
        for (int q = 0; q < 2; q++)
#pragma unroll
            for (int v = 0; v < 4; v++)
                if (g + 8 * v + 32 * q < k) s[v] = fma_rn(a[q][v], x[q][v], s[v]);
        for (int j0 = 64; j0 < k; j0 += 32)
#pragma unroll
            for (int v = 0; v < 4; v++) {
                const int j = j0 + g + 8 * v;
                if (j < k) s[v] = fma_rn(__ldg(bA + (long)w * k + j), __ldcg(e + __ldg(bidx + (long)w * k + j)), s[v]);
            }
        T t = (s[0] + s[2]) + (s[1] + s[3]);
        for (int o = 4; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o, 8);
        return fma_rn(ri - t, di, ei);
    }
};
inline int bnd_blocks(int nbl, bool big) { return blocks_for((long)nbl * (big ? 8 : 32), 256); }

// Exact solve of the boundary rows: a warp per row (EARLY, the small levels) or
// 8 lanes per row.
template <class T, bool EARLY>
__global__ void __launch_bounds__(256) k_bnd_exact(int nbl, const int *__restrict__ list, int k,
                                                   const int *__restrict__ bidx, const T *__restrict__ bA,
                                                   const T *__restrict__ dinv, const T *r, T *e)
{
    constexpr int LANES = EARLY ? 32 : 8;
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) / LANES, g = threadIdx.x % LANES;
    std::conditional_t<EARLY, BndRow<T>, BndRow8<T>> B;
    B.fetch(w, g, nbl, list, k, bidx, bA, dinv);
    pdl_wait<EARLY>();
    const T v = B.value(g, k, bidx, bA, r, e);
    if (g == 0 && w < nbl) e[B.i] = v;
}

// The first step of a smoothing pass from e = 0.  There e is zero but on the
// boundary rows (their exact solve r_b / a_bb), so A e vanishes exactly on
// the rows without boundary neighbours and the step needs no operator:
// d = c2 D^-1 r, e' = d.  The rows with boundary neighbours (the near list)
// subtract those neighbours' terms, stored compactly in slot order (ELL
// [kb][ldn]: neighbour, weight, the neighbour's 1 / diagonal); the zero terms
// that are left out change no bit of the sum.  16 bytes per row instead of
// the operator's 6 k: 41.7 -> 6 us on level 0 of the 1M cavity.
// FROMV: r is converted here from the FP64 Krylov vector V_j (j = st->j_next)
// and stored for the later steps.
template <class T>
struct FirstArgs {
    int n, nn, kb, ldn, nrow;   // nrow: CTAs of the row part (the near rows' CTAs follow)
    const uint8_t *tag;         // 0 far, 1 boundary, 2 near
    const T *dinv;
    T *r, *out, *d;
    T c2;
    const int *near_list, *kb_idx;
    const T *kb_a, *kb_d;
    const double *V;
    long ldv;
    const FgState *st;
};

template <class T, bool FROMV>
__device__ __forceinline__ void first_row(const FirstArgs<T> &a, int i, int tg, T di)
{
    T ri;
    if constexpr (FROMV) {
        ri = (T)__ldcg(a.V + (long)__ldcg(&a.st->j_next) * a.ldv + i);
        a.r[i] = ri;
    } else {
        ri = __ldcg(a.r + i);
    }
    if (tg == 1) {
        a.out[i] = ri * di;
    } else if (tg == 0) {
        const T dv = a.c2 * di * ri;
        a.d[i] = dv;
        a.out[i] = T(0) + dv;
    }
}

constexpr int kFirstKB = 12;  // boundary slots of a near row fetched together
template <class T>
struct FirstNear {
    int i, c[kFirstKB];
    T w[kFirstKB], dn[kFirstKB], di;
    __device__ __forceinline__ void slots(const FirstArgs<T> &a, int t, int q0)
    {
#pragma unroll
        for (int q = 0; q < kFirstKB; q++) {
            const bool in = q0 + q < a.kb;
            const long o = (long)(in ? q0 + q : 0) * a.ldn + t;
            c[q] = ldk(a.kb_idx + o);
            w[q] = ldk(a.kb_a + o);
            dn[q] = ldk(a.kb_d + o);
            if (!in) w[q] = T(0);
        }
    }
    __device__ __forceinline__ void fetch(const FirstArgs<T> &a, int t)
    {
        i = ldk(a.near_list + t);
        di = ldk(a.dinv + i);
        slots(a, t, 0);
    }
    template <bool FROMV>
    __device__ __forceinline__ void finish(const FirstArgs<T> &a, int t)
    {
        const double *Vj = nullptr;
        if constexpr (FROMV) Vj = a.V + (long)__ldcg(&a.st->j_next) * a.ldv;
        auto rhs = [&](int x) -> T {
            if constexpr (FROMV) return (T)__ldcg(Vj + x);
            else return __ldcg(a.r + x);
        };
        const T ri = rhs(i);
        T s = T(0);
        for (int q0 = 0; q0 < a.kb; q0 += kFirstKB) {
            if (q0 > 0) slots(a, t, q0);
            T v[kFirstKB];
#pragma unroll
            for (int q = 0; q < kFirstKB; q++) v[q] = rhs(c[q]) * dn[q];
#pragma unroll
            for (int q = 0; q < kFirstKB; q++) s = fma_rn(w[q], v[q], s);
        }
        const T q = ri - s;
        const T dv = a.c2 * di * q;
        a.d[i] = dv;
        a.out[i] = T(0) + dv;
    }
};

template <class T, bool FROMV>
__device__ __forceinline__ void first_near(const FirstArgs<T> &a, int t)
{
    FirstNear<T> F;
    F.fetch(a, t);
    F.template finish<FROMV>(a, t);
}

template <class T, bool FROMV, bool EARLY>
__global__ void __launch_bounds__(256) k_first_step(const __grid_constant__ FirstArgs<T> a)
{
    if ((int)blockIdx.x < a.nrow) {
        const int i0 = blockIdx.x * blockDim.x + threadIdx.x, i = min(i0, a.n - 1);
        const int tg = ldk(a.tag + i);
        const T di = ldk(a.dinv + i);
        pdl_wait<EARLY>();
        if (i0 < a.n) first_row<T, FROMV>(a, i, tg, di);
        return;
    }
    const int t0 = ((int)blockIdx.x - a.nrow) * blockDim.x + threadIdx.x, t = min(t0, a.nn - 1);
    FirstNear<T> F;
    F.fetch(a, t);
    pdl_wait<EARLY>();
    if (t0 < a.nn) F.template finish<FROMV>(a, t);
}

// (P e_c)[0], the prolongated correction at the pinned node, by the 32 lanes
// of warp 0: the lanes fetch the operands of 32 slots at once (operand(j, a,
// x): weight and gathered value of slot j), then every lane sums the
// products in slot order, one fused multiply-add per slot -- the rounding of
// the row dots (ell_row_dot, ell_row_dot_o), so the shift has the bits a
// serial row-0 dot would give.
template <class T, class Op>
__device__ __forceinline__ T row0_dot_warp(int k, Op operand)
{
    const int lane = threadIdx.x & 31;
    T s = T(0);
    for (int j0 = 0; j0 < k; j0 += 32) {
        T a = T(0), x = T(0);
        if (j0 + lane < k) operand(j0 + lane, a, x);
        const int m = min(32, k - j0);
        for (int q = 0; q < m; q++) s = fma_rn(__shfl_sync(0xffffffffu, a, q), __shfl_sync(0xffffffffu, x, q), s);
    }
    return s;
}

// ---------------------------------------------------------------------------
// compact FP32 path: FP32 weights, neighbours stored as int16 offsets c - base
// (6 bytes per stencil slot instead of 8)
// ---------------------------------------------------------------------------
// A row of the fused coarse V-cycle: the vectors are loaded from L2, past the
// SM's L1 and the read-only path, because other CTAs rewrite them between passes.
template <class T>
__device__ __forceinline__ T ell_row_dot_o(const short *__restrict__ off, const T *__restrict__ A, const T *x, long n,
                                           int k, long i, int base)
{
    T s = T(0);
    int j = 0;
    for (; j + 8 <= k; j += 8) {
        int c[8];
        T a[8];
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const long o = (long)(j + q) * n + i;
            c[q] = base + (int)__ldg(off + o);
            a[q] = __ldg(A + o);
        }
#pragma unroll
        for (int q = 0; q < 8; q++) s = fma_rn(a[q], __ldcg(x + c[q]), s);
    }
    for (; j < k; j++) {
        const long o = (long)j * n + i;
        s = fma_rn(A[o], __ldcg(x + base + (int)off[o]), s);
    }
    return s;
}

// Compact level kernels (FP32 or FP64 weights, int16 offsets, ELL [k][ld],
// each row's slots sorted by neighbour index).
//
// k_level_v4: four consecutive rows per thread; the weights and offsets of
// rows i0..i0+3 come in as one 16-byte (FP32; two for FP64) and one 8-byte
// load per stencil slot (ld a multiple of 4; streamed past L1 with
// evict-first loads), so a thread has 8 operator loads and 16 gathers in
// flight per 4 slots.  For the large levels, which are bandwidth-bound.
// k_level_c1: one row per thread, for the small levels, which are latency-
// bound and need the threads more than the wide loads.
// Each row's sum runs in slot order in both, as in every other level kernel
// of the same precision, so all of them give the same bits.  MODE 0:
// Chebyshev step q = r - A e, d = c1 d + c2 D^-1 q, e' = e + d on interior
// rows (boundary rows copy e); MODE 1: residual q = r - A e on interior rows,
// 0 on boundary rows.
// ---------------------------------------------------------------------------
// One step on a level: the boundary rows' exact solve from the current e,
// then the Chebyshev step (MODE 0) or the residual (MODE 1) of the interior
// rows.  Only the near rows (interior rows with boundary neighbours) see the
// boundary rows' new values.
//
// Levels below kVecMinRows rows: two chained launches (k_bnd_exact,
// k_level_c1), each with its operands in registers before its wait.
// The larger levels (k_level_v4): one launch in three parts --
//   boundary  8 lanes per boundary row: e[b] (and out[b]); then one release
//             increment of sync[0] per CTA;
//   far       the interior rows without boundary neighbours;
//   near      a thread per near row, after a bounded wait for the boundary
//             part's increments; rows as their own ELL copy [k][ldn],
//             gathers from L2.
// The boundary part is dispatched before the near part (block order) and
// waits for nothing, so the near part's wait ends; it is bounded all the
// same: when it runs out the CTA sets *err (MGM_ERR_TIMEOUT on the host).
// The last near CTA to pass resets the two counters for the next launch.
// Same operands in the same order as separate launches: the same bits.
// ---------------------------------------------------------------------------
template <class T>
struct StepArgsL {
    int n, ld, k, kp, nbl, nn, ldn;
    int nbc, nfar, nnc, fb;  // CTAs of the three parts; far CTAs dispatched before the boundary part
    const void *gi;          // int16 offsets [k][ld] or 32-bit indices
    const T *A, *dinv;
    const uint8_t *tag;      // 0 far, 1 boundary, 2 near
    const T *r;
    T *e, *out, *d;
    T c1, c2;
    int first;
    const int *bnd_list, *bnd_idx;
    const T *bnd_A;
    const int *near_list, *near_idx;
    const T *near_A;
    unsigned *sync;          // {boundary CTAs done, near CTAs passed}
    int *err;
};

// the level's output of row i from its sum s
template <int MODE, class T>
__device__ __forceinline__ void step_out(const StepArgsL<T> &a, int i, T ri, T ei, T dprev, T di, T s)
{
    const T q = ri - s;
    if (MODE == 0) {
        const T dv = a.first ? a.c2 * di * q : a.c1 * dprev + a.c2 * di * q;
        a.d[i] = dv;
        a.out[i] = ei + dv;
    } else {
        a.out[i] = q;
    }
}

template <int MODE, class T>
__device__ __forceinline__ void step_bnd_part(const StepArgsL<T> &a, int blk)
{
    const int w = (blk * blockDim.x + threadIdx.x) >> 3, g = threadIdx.x & 7;
    BndRow8<T> B;
    B.fetch(w, g, a.nbl, a.bnd_list, a.k, a.bnd_idx, a.bnd_A, a.dinv);
    pdl_wait<false>();
    const T v = B.value(g, a.k, a.bnd_idx, a.bnd_A, a.r, a.e);
    if (g == 0 && w < a.nbl) {
        a.e[B.i] = v;
        a.out[B.i] = MODE == 0 ? v : T(0);
    }
    if (a.nnc == 0) return;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.sync) : "memory");
    }
}

template <int MODE, class T>
__device__ __forceinline__ void step_near_part(const StepArgsL<T> &a, int blk)
{
    __shared__ int go;
    const int t = blk * blockDim.x + threadIdx.x;
    const bool live = t < a.nn;
    const int tc = live ? t : 0;
    const int i = ldk(a.near_list + tc);
    const T di = ldk(a.dinv + i);
    pdl_wait<false>();
    if (threadIdx.x == 0) {
        int ok = 1;
        if (a.nbc > 0) {
            unsigned seen;
            long spins = 0;
            do {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(a.sync) : "memory");
                if (++spins > (1L << 20)) {
                    atomicExch(a.err, 1);
                    ok = 0;
                    break;
                }
            } while (seen < (unsigned)a.nbc);
        }
        go = ok;
    }
    __syncthreads();
    if (live && go) {
        const T ri = __ldcg(a.r + i);
        T ei = T(0), dprev = T(0), s = T(0);
        if (MODE == 0) {
            ei = __ldcg(a.e + i);
            if (!a.first) dprev = __ldcg(a.d + i);
        }
        int j = 0;
        for (; j + 8 <= a.k; j += 8) {
            RowChunk<T, 8, true> R;
            R.fetch(a.near_idx, a.near_A, a.ldn, t, 0, j);
            s = R.template dot<true>(a.e, s);
        }
        for (; j < a.k; j++) {
            const long o = (long)j * a.ldn + t;
            s = fma_rn(__ldg(a.near_A + o), __ldcg(a.e + __ldg(a.near_idx + o)), s);
        }
        step_out<MODE>(a, i, ri, ei, dprev, di, s);
    }
    if (threadIdx.x == 0 && go && a.nbc > 0 && atomicAdd(a.sync + 1, 1u) + 1u == (unsigned)a.nnc) {
        atomicExch(a.sync + 1, 0u);
        atomicExch(a.sync, 0u);
    }
}

// The step of the levels below kVecMinRows rows (and of any level whose
// neighbours do not fit int16 offsets, IDX), after k_bnd_exact: a thread per
// row, the whole row of up to KC slots in registers before the wait,
// 128-thread CTAs (twice the CTAs to spread over the SMs).
template <int MODE, class T, int KC, bool IDX>
__global__ void __launch_bounds__(128) k_level_c1(const __grid_constant__ StepArgsL<T> a)
{
    const int i0 = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = min(i0, a.n - 1);
    RowChunk<T, KC, IDX> R;
    R.fetch(a.gi, a.A, a.ld, i, i, 0);
    const T di = ldk(a.dinv + i);
    const int tg = ldk(a.tag + i);
    pdl_wait<true>();
    const T ri = __ldcg(a.r + i), ei = __ldcg(a.e + i);
    T dprev = T(0);
    if (MODE == 0 && !a.first) dprev = __ldcg(a.d + i);
    T s = R.template dot<true>(a.e, T(0));
    s = row_rest<true, T, KC, IDX>(a.gi, a.A, a.e, a.ld, a.kp, i, i, s);
    if (i0 >= a.n) return;
    if (tg == 1) {
        a.out[i] = MODE == 0 ? ei : T(0);
        return;
    }
    step_out<MODE>(a, i, ri, ei, dprev, di, s);
}

// the four weights of rows i0..i0+3 in slot o (evict-first)
__device__ __forceinline__ void load4(const float *A, long o, float (&a)[4])
{
    const float4 v = __ldcs(reinterpret_cast<const float4 *>(A + o));
    a[0] = v.x; a[1] = v.y; a[2] = v.z; a[3] = v.w;
}
__device__ __forceinline__ void load4(const double *A, long o, double (&a)[4])
{
    const double2 v0 = __ldcs(reinterpret_cast<const double2 *>(A + o));
    const double2 v1 = __ldcs(reinterpret_cast<const double2 *>(A + o + 2));
    a[0] = v0.x; a[1] = v0.y; a[2] = v1.x; a[3] = v1.y;
}

// FP32: 4 CTAs of 256 per SM (64 registers); FP64: 3 (twice the weight
// registers).  The first slots' operator loads are issued before the wait for
// the predecessor, so that they fill its tail.
template <int MODE, class T>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 4 : 3) k_level_v4(const __grid_constant__ StepArgsL<T> g)
{
    const int b = blockIdx.x;
    if (b >= g.fb && b < g.fb + g.nbc) {
        step_bnd_part<MODE, T>(g, b - g.fb);
        return;
    }
    if (b >= g.nfar + g.nbc) {
        step_near_part<MODE, T>(g, b - g.nfar - g.nbc);
        return;
    }
    const int n = g.n, ld = g.ld, k = g.k;
    const T *__restrict__ A = g.A;
    const short *__restrict__ off = static_cast<const short *>(g.gi);
    const T *__restrict__ e = g.e;
    const int i0 = ((b < g.fb ? b : b - g.nbc) * blockDim.x + threadIdx.x) * 4;
    const bool live = i0 < n;
    T s[4] = {T(0), T(0), T(0), T(0)};
    T a[4][4];
    int c[4][4];
    auto fetch = [&](int j) {
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const long o = (long)(j + q) * ld + i0;
            load4(A, o, a[q]);
            const uint2 ov = __ldcs(reinterpret_cast<const uint2 *>(off + o));
            c[q][0] = i0 + (int)(short)(ov.x & 0xffffu);
            c[q][1] = i0 + 1 + (int)(short)(ov.x >> 16);
            c[q][2] = i0 + 2 + (int)(short)(ov.y & 0xffffu);
            c[q][3] = i0 + 3 + (int)(short)(ov.y >> 16);
        }
    };
    auto use = [&] {
        // padding rows (i >= n) carry weight 0 and offset 0: clamp their gathers into the vector
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
            for (int v = 0; v < 4; v++) s[v] = fma_rn(a[q][v], __ldg(e + min(c[q][v], n - 1)), s[v]);
    };
    if (live && k >= 4) fetch(0);
    pdl_wait<false>();
    if (!live) return;
    int j = 0;
    if (k >= 4) {
        use();
        for (j = 4; j + 4 <= k; j += 4) {
            fetch(j);
            use();
        }
    }
    for (; j < k; j++) {
#pragma unroll
        for (int v = 0; v < 4; v++) {
            const long o = (long)j * ld + i0 + v;
            s[v] = fma_rn(__ldcs(A + o), __ldg(e + min(i0 + v + (int)__ldcs(off + o), n - 1)), s[v]);
        }
    }
#pragma unroll
    for (int v = 0; v < 4; v++) {
        const int i = i0 + v;
        if (i >= n) continue;
        const int tg = __ldg(g.tag + i);
        if (g.nbc == 0 && tg == 1) g.out[i] = MODE == 0 ? e[i] : T(0);
        if (tg == 1 || (tg == 2 && g.nbc)) continue;
        step_out<MODE>(g, i, g.r[i], MODE == 0 ? e[i] : T(0), MODE == 0 && !g.first ? g.d[i] : T(0), g.dinv[i], s[v]);
    }
}

// k_level_h4: k_level_v4 on the FP16 operator W ~ D^-1 A, four rows per
// thread interleaved: lane t of warp g holds rows 128 g + t + 32 v (v =
// 0..3), so that a warp's gathers for one slot and row set v come from 32
// consecutive rows and its per-row loads and stores are coalesced (measured
// 8% faster than consecutive rows here; k_level_v4 measured 4% slower with
// it).  One 16-byte load per stencil slot brings the four rows' weights
// (FP16) and offsets (int16):
// 4 bytes per slot instead of 6.  The off-diagonal weights enter in
// difference form, s = sum_{j != i} w_ij (e_j - e_i) + rho_i e_i, where the
// diagonal slot (offset 0) holds rho_i, the row sum of D^-1 A: the rows then
// keep their sums (a Laplacian row maps constants to ~0) whatever the FP16
// rounding of the single weights, which would otherwise perturb the smooth
// modes by (rounding error) x (condition number).  Sums in FP32, in slot
// order.  MODE 0: d = c1 d + c2 (D^-1 r - s), e' = e + d on interior rows;
// MODE 1: q = r - s / D^-1 on interior rows, 0 on boundary rows.
template <int MODE>
__device__ __forceinline__ void level_row_out_h(int i, float s, const float *__restrict__ dinv,
                                                const uint8_t *__restrict__ btag, const float *__restrict__ r,
                                                float ei, float *__restrict__ out, float *__restrict__ d, float c1,
                                                float c2, int first)
{
    if (MODE == 0) {
        if (btag[i]) { out[i] = ei; return; }
        const float q = dinv[i] * r[i] - s;
        const float di = first ? c2 * q : c1 * d[i] + c2 * q;
        d[i] = di;
        out[i] = ei + di;
    } else {
        out[i] = btag[i] ? 0.f : r[i] - s / dinv[i];
    }
}

__device__ __forceinline__ float h16(unsigned bits) { return __half2float(__ushort_as_half((unsigned short)bits)); }

template <int MODE>
__global__ void __launch_bounds__(256, 4) k_level_h4(int n, int ld, int k, const uint4 *__restrict__ W,
                                                  const float *__restrict__ dinv, const uint8_t *__restrict__ btag,
                                                  const float *__restrict__ r, const float *__restrict__ e,
                                                  float *__restrict__ out, float *__restrict__ d, float c1, float c2,
                                                  int first)
{
    pdl_enter();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int ib = (t >> 5) * 128 + (t & 31);   // rows ib + 32 v, v = 0..3
    if (ib >= n) return;
    const long q4 = ld >> 2;
    float s[4] = {0.f, 0.f, 0.f, 0.f}, ws[4] = {0.f, 0.f, 0.f, 0.f};
    int j = 0;
    for (; j + 4 <= k; j += 4) {
        uint4 w[4];
#pragma unroll
        for (int q = 0; q < 4; q++) w[q] = __ldcs(W + (long)(j + q) * q4 + t);
        float a[4][4];
        int o[4][4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            a[q][0] = h16(w[q].x & 0xffffu); a[q][1] = h16(w[q].x >> 16);
            a[q][2] = h16(w[q].y & 0xffffu); a[q][3] = h16(w[q].y >> 16);
            o[q][0] = (int)(short)(w[q].z & 0xffffu); o[q][1] = (int)(short)(w[q].z >> 16);
            o[q][2] = (int)(short)(w[q].w & 0xffffu); o[q][3] = (int)(short)(w[q].w >> 16);
        }
        // padding rows (i >= n) carry weight 0 and offset 0: clamp their gathers into the vector
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
            for (int v = 0; v < 4; v++) {
                s[v] += a[q][v] * __ldg(e + min(ib + 32 * v + o[q][v], n - 1));
                ws[v] += o[q][v] != 0 ? a[q][v] : 0.f;
            }
    }
    for (; j < k; j++) {
        const uint4 w = __ldcs(W + (long)j * q4 + t);
#pragma unroll
        for (int v = 0; v < 4; v++) {
            const unsigned hw = (v < 2 ? w.x : w.y) >> (16 * (v & 1)), ow = (v < 2 ? w.z : w.w) >> (16 * (v & 1));
            const float a = h16(hw & 0xffffu);
            const int o = (int)(short)(ow & 0xffffu);
            s[v] += a * __ldg(e + min(ib + 32 * v + o, n - 1));
            ws[v] += o != 0 ? a : 0.f;
        }
    }
#pragma unroll
    for (int v = 0; v < 4; v++) {
        const int i = ib + 32 * v;
        if (i < n) {
            const float ei = e[i];
            level_row_out_h<MODE>(i, s[v] - ws[v] * ei, dinv, btag, r, ei, out, d, c1, c2, first);
        }
    }
}

template <class T>
static StepArgsL<T> step_args_of(const SolveLevel<T> &L, T *e, T *out, T c1, T c2, int first)
{
    StepArgsL<T> a{};
    a.n = L.n; a.ld = L.ld; a.k = L.k; a.kp = (L.k + 7) & ~7; a.nbl = L.nb_list; a.nn = L.nn; a.ldn = L.ldn;
    a.gi = L.off ? (const void *)L.off : (const void *)L.idx;
    a.A = L.A; a.dinv = L.dinv; a.tag = L.tag;
    a.r = L.r; a.e = e; a.out = out; a.d = L.d;
    a.c1 = c1; a.c2 = c2; a.first = first;
    a.bnd_list = L.bnd_list; a.bnd_idx = L.bnd_idx; a.bnd_A = L.bnd_A;
    a.near_list = L.near_list; a.near_idx = L.near_idx; a.near_A = L.near_A;
    a.sync = L.sync; a.err = L.tma_err;
    return a;
}

template <class T>
static void launch_bnd(const SolveLevel<T> &L, T *e, cudaStream_t s, Chain &launch)
{
    const int nbb = bnd_blocks(L.nb_list, L.n >= kVecMinRows);
    if (nbb == 0) return;
    if (L.n < kVecMinRows)
        launch(k_bnd_exact<T, true>, nbb, 256, 0, s, L.nb_list, L.bnd_list, L.k, L.bnd_idx, L.bnd_A, L.dinv, L.r, e);
    else
        launch(k_bnd_exact<T, false>, nbb, 256, 0, s, L.nb_list, L.bnd_list, L.k, L.bnd_idx, L.bnd_A, L.dinv, L.r, e);
}

// the one-row-per-thread step: the smallest chunk that holds the row, so that
// the whole row is fetched before the wait (the rest of a wider row after it)
template <int MODE, class T, bool IDX>
static void launch_c1(const SolveLevel<T> &L, T *e, T *out, T c1, T c2, int first, cudaStream_t s, Chain &launch)
{
    const StepArgsL<T> a = step_args_of(L, e, out, c1, c2, first);
    const int grid = blocks_for(L.n, 128);
    if (a.kp <= 16) launch(k_level_c1<MODE, T, 8, IDX>, grid, 128, 0, s, a);
    else if (a.kp <= 24) launch(k_level_c1<MODE, T, 24, IDX>, grid, 128, 0, s, a);
    else if (a.kp <= 32 || sizeof(T) == 8) launch(k_level_c1<MODE, T, 32, IDX>, grid, 128, 0, s, a);
    else launch(k_level_c1<MODE, T, 40, IDX>, grid, 128, 0, s, a);
}

// the fused coarse V-cycle's transfers and dense solve (vectors from L2)
template <class T>
__device__ __forceinline__ void restrict_row(int i, int n, int k, const short *__restrict__ off,
                                             const int *__restrict__ base, const T *__restrict__ rw,
                                             const uint8_t *__restrict__ btag, const T *qf, T *rc)
{
    if (btag[i] || i == 0) { rc[i] = T(0); return; }
    rc[i] = ell_row_dot_o(off, rw, qf, n, k, i, base[i]);
}
// (P e_c)[0] of the compact prolongation, by warp 0 of a CTA (row0_dot_warp)
template <class T>
__device__ __forceinline__ T prolong_shift_warp(int n, int k, const short *__restrict__ off,
                                                const int *__restrict__ base, const T *__restrict__ pw, const T *ec)
{
    const int b0 = base[0];
    return row0_dot_warp<T>(k, [&](int j, T &a, T &x) {
        a = pw[(long)j * n];
        x = __ldcg(ec + b0 + (int)off[(long)j * n]);
    });
}
template <class T>
__device__ __forceinline__ void prolong_row(int i, int n, int k, const short *__restrict__ off,
                                            const int *__restrict__ base, const T *__restrict__ pw, const T *ec, T *ef,
                                            T shift)
{
    ef[i] = __ldcg(ef + i) + (ell_row_dot_o(off, pw, ec, n, k, i, base[i]) - shift);
}

// Restriction into a level: r_c[i] = sum_j Rw[j][i] q_f[...] on interior rows
// but row 0, 0 elsewhere.  FIRST (every level but the coarsest): the first
// smoothing step of the pass from e = 0 with it (k_first_step): the boundary
// rows' right-hand side is 0 there, so their e is 0 and d = c2 D^-1 r_c,
// e = d on every interior row.  EARLY: rows padded to a multiple of 8 slots,
// KC of them fetched before the wait.
template <class T>
struct TransferArgs {
    int n, k, kp;
    const void *gi;        // int16 offsets from base[i], or 32-bit indices, [k][n]
    const int *base;
    const T *w;
    const uint8_t *btag;
    const T *in;
    T *out;                // restriction: r_c; prolongation: e_f
    const T *dinv;
    T *d, *e;
    T c2;
};

template <class T, int KC, bool IDX, bool EARLY>
struct TransferRow {
    RowChunk<T, KC, IDX> R;
    int base = 0;
    __device__ __forceinline__ void fetch(const TransferArgs<T> &a, int i)
    {
        if constexpr (!IDX) base = ldk(a.base + i);
        if constexpr (EARLY) R.fetch(a.gi, a.w, a.n, i, base, 0);
        else R.fetch_to(a.gi, a.w, a.n, i, base, 0, a.k);
    }
    __device__ __forceinline__ T dot(const TransferArgs<T> &a, int i)
    {
        if constexpr (EARLY) {
            const T s = R.template dot<true>(a.in, T(0));
            return row_rest<true, T, KC, IDX>(a.gi, a.w, a.in, a.n, a.kp, i, base, s);
        } else {
            static_assert(KC == 8, "row_big takes chunks of 8");
            return row_big<T, IDX, false>(R, a.gi, a.w, a.in, a.n, a.k, i, base);
        }
    }
};

template <class T, int KC, bool IDX, bool EARLY, bool FIRST>
__global__ void __launch_bounds__(128) k_restrict(const __grid_constant__ TransferArgs<T> a)
{
    const int i0 = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = min(i0, a.n - 1);
    const bool inner = !ldk(a.btag + i);
    TransferRow<T, KC, IDX, EARLY> R;
    R.fetch(a, i);
    T di = T(0);
    if (FIRST) di = ldk(a.dinv + i);
    pdl_wait<EARLY>();
    T s = R.dot(a, i);
    if (i0 >= a.n) return;
    if (!inner || i == 0) s = T(0);
    a.out[i] = s;
    if (FIRST) {
        if (!inner) {
            a.e[i] = s * di;
        } else {
            const T dv = a.c2 * di * s;
            a.d[i] = dv;
            a.e[i] = T(0) + dv;
        }
    }
}

// Prolongation: e_f[i] += (P e_c)[i] - (P e_c)[0] (the shift keeps the pinned
// node uncorrected).  Warp 0 sums row 0 while the other warps sum their rows.
template <class T, int KC, bool IDX, bool EARLY, int BS>
__global__ void __launch_bounds__(BS) k_prolong(const __grid_constant__ TransferArgs<T> a)
{
    __shared__ T shift;
    const int i0 = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = min(i0, a.n - 1);
    TransferRow<T, KC, IDX, EARLY> R;
    R.fetch(a, i);
    // row 0's slots, one per lane of warp 0 (the first 32 before the wait)
    RowChunk<T, 1, IDX> R0;
    int b0 = 0;
    const int lane0 = min((int)threadIdx.x, a.k - 1);
    if (threadIdx.x < 32) {
        if constexpr (!IDX) b0 = ldk(a.base);
        R0.fetch(a.gi, a.w, a.n, 0, b0, lane0);
    }
    pdl_wait<EARLY>();
    if (threadIdx.x < 32) {
        const T s0 = row0_dot_warp<T>(a.k, [&](int j, T &w, T &x) {
            if (j >= 32) R0.fetch(a.gi, a.w, a.n, 0, b0, j);
            w = R0.a[0];
            x = __ldcg(a.in + R0.c[0]);
        });
        if (threadIdx.x == 0) shift = s0;
    }
    const T ei = __ldcg(a.out + i);
    const T s = R.dot(a, i);
    __syncthreads();
    if (i0 < a.n) a.out[i] = ei + (s - shift);
}

template <class T, bool IDX, bool FIRST>
static void launch_restrict_k(const TransferArgs<T> &a, cudaStream_t s, Chain &launch)
{
    const int grid = blocks_for(a.n, 128);
    if (a.n >= kVecMinRows) launch(k_restrict<T, 8, IDX, false, FIRST>, grid, 128, 0, s, a);
    else if (a.kp <= 16) launch(k_restrict<T, 8, IDX, true, FIRST>, grid, 128, 0, s, a);
    else if (a.kp <= 24) launch(k_restrict<T, 24, IDX, true, FIRST>, grid, 128, 0, s, a);
    else launch(k_restrict<T, 32, IDX, true, FIRST>, grid, 128, 0, s, a);
}

template <class T, bool FIRST>
static void launch_restrict(const SolveLevel<T> &C, const T *qf, T c2, cudaStream_t s, Chain &launch)
{
    TransferArgs<T> a{};
    a.n = C.n; a.k = C.kr; a.kp = (C.kr + 7) & ~7; a.base = C.r_base; a.w = C.r_w; a.btag = C.btag; a.in = qf;
    a.out = C.r; a.dinv = C.dinv; a.d = C.d; a.e = C.e; a.c2 = c2;
    a.gi = C.r_off ? (const void *)C.r_off : (const void *)C.r_idx;
    if (C.r_off) launch_restrict_k<T, false, FIRST>(a, s, launch);
    else launch_restrict_k<T, true, FIRST>(a, s, launch);
}

template <class T, bool IDX>
static void launch_prolong_k(const TransferArgs<T> &a, cudaStream_t s, Chain &launch)
{
    if (a.n >= kVecMinRows) launch(k_prolong<T, 8, IDX, false, 256>, blocks_for(a.n, 256), 256, 0, s, a);
    else if (a.kp <= 16) launch(k_prolong<T, 8, IDX, true, 128>, blocks_for(a.n, 128), 128, 0, s, a);
    else if (a.kp <= 24) launch(k_prolong<T, 24, IDX, true, 128>, blocks_for(a.n, 128), 128, 0, s, a);
    else launch(k_prolong<T, 32, IDX, true, 128>, blocks_for(a.n, 128), 128, 0, s, a);
}

template <class T>
static void launch_prolong(const SolveLevel<T> &L, const T *ec, cudaStream_t s, Chain &launch)
{
    TransferArgs<T> a{};
    a.n = L.n; a.k = L.kp; a.kp = (L.kp + 7) & ~7; a.base = L.p_base; a.w = L.p_w; a.in = ec; a.out = L.e;
    a.gi = L.p_off ? (const void *)L.p_off : (const void *)L.p_idx;
    if (L.p_off) launch_prolong_k<T, false>(a, s, launch);
    else launch_prolong_k<T, true>(a, s, launch);
}

// ---------------------------------------------------------------------------
// tile-streamed level kernels (FP32 compact operator)
//
// The operator is stored tile-major ([tile][k][kTileRows]: a tile's weights,
// and separately its int16 offsets, are contiguous).  A persistent CTA walks
// tiles of kTileRows rows; for each tile one thread issues two bulk
// asynchronous copies (cp.async.bulk, the TMA engine's 1-D form) into shared
// memory, completing on an mbarrier; two stages alternate, so the next tile's
// operator streams in while this tile's rows gather their neighbours.  A
// thread then reads its row's stencil from shared memory and issues its
// neighbour gathers back to back.  The products are summed in slot order, as
// in k_level_v4, so the results are the same bits.
//
// Every mbarrier wait is bounded: on time-out the CTA sets *err, waits (again
// bounded) for the copies it still has in flight, and stops.
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t *bar, unsigned count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, unsigned parity)
{
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, unsigned parity)
{
    for (int it = 0; it < (1 << 20); it++)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}
// global -> shared bulk copy; addresses 16-byte aligned, bytes a multiple of 16
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, unsigned bytes, uint64_t *bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

// One pipeline stage in shared memory: the tile's weights [k][kTileRows] f32
// and offsets [k][kTileRows] i16.
struct TileStage {
    int k;
    __device__ size_t a_off() const { return 0; }
    __device__ size_t o_off() const { return (size_t)k * kTileRows * sizeof(float); }
    __device__ size_t bytes() const { return (size_t)k * kTileRows * (sizeof(float) + sizeof(short)); }
};
__host__ inline size_t tile_stage_bytes(int k) { return (size_t)k * kTileRows * (sizeof(float) + sizeof(short)); }

// One thread issues the two bulk copies of tile `tile` (weights, offsets; the
// operator is stored tile-major) into stage memory `st`; the mbarrier expects
// exactly the bytes issued.
__device__ __forceinline__ void tile_issue(unsigned char *st, uint64_t *bar, int tile, int k, const float *At,
                                           const short *offt)
{
    const TileStage L{k};
    // the stage may have been read by the CTA's threads (generic proxy) before
    // the barrier that precedes this call: order those reads before the
    // copies' writes (async proxy)
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    mbar_expect_tx(bar, (unsigned)L.bytes());
    const long t0 = (long)tile * k * kTileRows;
    bulk_g2s(st + L.a_off(), At + t0, (unsigned)(k * kTileRows * sizeof(float)), bar);
    bulk_g2s(st + L.o_off(), offt + t0, (unsigned)(k * kTileRows * sizeof(short)), bar);
}

// MODE 0: Chebyshev step (as k_level_v4<0>); MODE 1: residual (as k_level_v4<1>).
// Chunked variant for any k <= kTileMaxK: the row's stencil is read from the
// stage while its gathers run, 8 at a time.
template <int MODE>
__global__ void __launch_bounds__(kTileRows) k_level_tiled(int n, int k, const short *__restrict__ offt,
                                                           const float *__restrict__ At, const float *__restrict__ dinv,
                                                           const uint8_t *__restrict__ btag,
                                                           const float *__restrict__ r, const float *__restrict__ e,
                                                           float *__restrict__ out, float *__restrict__ d, float c1,
                                                           float c2, int first, int *err)
{
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) uint64_t bar[2];
    __shared__ int ok_flag;
    const int tid = threadIdx.x;
    const int ntiles = (n + kTileRows - 1) / kTileRows;
    const TileStage L{k};
    const size_t stage = L.bytes();
    unsigned pending = 0;  // bit st: stage st has copies in flight (tracked by thread 0)
    if (tid == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    auto issue = [&](int tile, int st) {
        if (tid == 0) tile_issue(smem + st * stage, &bar[st], tile, k, At, offt);
        pending |= 1u << st;
    };
    int it = 0;
    if (blockIdx.x < ntiles) issue(blockIdx.x, 0);
    if (blockIdx.x + gridDim.x < ntiles) issue(blockIdx.x + gridDim.x, 1);
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x, it++) {
        const int st = it & 1;
        const unsigned parity = (unsigned)((it >> 1) & 1);
        if (tid == 0) ok_flag = mbar_wait_bounded(&bar[st], parity) ? 1 : 0;
        __syncthreads();
        if (!ok_flag) {
            if (tid == 0) {
                atomicOr(err, 1);
                // Best effort before the CTA exits: give the timed-out stage's
                // copies one more bounded spell, then wait (bounded) for the
                // other stage's, so that normally no bulk copy still writes
                // into this CTA's shared memory after it has returned.  The
                // host turns the error flag into MGM_ERR_TIMEOUT.
                mbar_wait_bounded(&bar[st], parity);
                const int o = st ^ 1;
                if (pending & (1u << o)) mbar_wait_bounded(&bar[o], (unsigned)(((it + 1) >> 1) & 1));
            }
            return;
        }
        mbar_try_wait(&bar[st], parity);  // completed: acquires the copied data for this thread
        pending &= ~(1u << st);
        unsigned char *sb = smem + st * stage;
        const int i = tile * kTileRows + tid;
        if (i < n) {
            const float ei = e[i];
            if (btag[i]) {
                out[i] = MODE == 0 ? ei : 0.f;
            } else {
                const float *a = (const float *)(sb + L.a_off()) + tid;
                const short *o = (const short *)(sb + L.o_off()) + tid;
                float s = 0.f;
                int j = 0;
                for (; j + 8 <= k; j += 8) {
                    float av[8], xv[8];
#pragma unroll
                    for (int q = 0; q < 8; q++) {
                        av[q] = a[(j + q) * kTileRows];
                        xv[q] = __ldg(e + i + (int)o[(j + q) * kTileRows]);
                    }
#pragma unroll
                    for (int q = 0; q < 8; q++) s += av[q] * xv[q];
                }
                for (; j < k; j++) s += a[j * kTileRows] * e[i + (int)o[j * kTileRows]];
                if (MODE == 0) {
                    const float q = r[i] - s;
                    const float di = first ? c2 * dinv[i] * q : c1 * d[i] + c2 * dinv[i] * q;
                    d[i] = di;
                    out[i] = ei + di;
                } else {
                    out[i] = r[i] - s;
                }
            }
        }
        __syncthreads();  // every thread is done with stage st
        if (tile + 2 * gridDim.x < ntiles) issue(tile + 2 * gridDim.x, st);
    }
}

// Register variant for k <= 32: a thread copies its row's whole stencil from
// the stage into registers, the CTA syncs, the freed stage starts the copies
// of the tile after next, and the threads issue all k neighbour gathers at
// once (k gathers in flight per row instead of 8).
template <int MODE>
__global__ void __launch_bounds__(kTileRows, 2) k_level_tiled_r(int n, int k, const short *__restrict__ offt,
                                                              const float *__restrict__ At,
                                                              const float *__restrict__ dinv,
                                                              const uint8_t *__restrict__ btag,
                                                              const float *__restrict__ r,
                                                              const float *__restrict__ e, float *__restrict__ out,
                                                              float *__restrict__ d, float c1, float c2, int first,
                                                              int *err)
{
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) uint64_t bar[2];
    __shared__ int ok_flag;
    const int tid = threadIdx.x;
    const int ntiles = (n + kTileRows - 1) / kTileRows;
    const TileStage L{k};
    const size_t stage = L.bytes();
    unsigned pending = 0;  // bit st: stage st has copies in flight (tracked by thread 0)
    if (tid == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    auto issue = [&](int tile, int st) {
        if (tid == 0) tile_issue(smem + st * stage, &bar[st], tile, k, At, offt);
        pending |= 1u << st;
    };
    if (blockIdx.x < ntiles) issue(blockIdx.x, 0);
    if (blockIdx.x + gridDim.x < ntiles) issue(blockIdx.x + gridDim.x, 1);
    int it = 0;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x, it++) {
        const int st = it & 1;
        const unsigned parity = (unsigned)((it >> 1) & 1);
        if (tid == 0) ok_flag = mbar_wait_bounded(&bar[st], parity) ? 1 : 0;
        __syncthreads();
        if (!ok_flag) {
            if (tid == 0) {
                atomicOr(err, 1);
                // Best effort before the CTA exits: give the timed-out stage's
                // copies one more bounded spell, then wait (bounded) for the
                // other stage's, so that normally no bulk copy still writes
                // into this CTA's shared memory after it has returned.  The
                // host turns the error flag into MGM_ERR_TIMEOUT.
                mbar_wait_bounded(&bar[st], parity);
                const int o = st ^ 1;
                if (pending & (1u << o)) mbar_wait_bounded(&bar[o], (unsigned)(((it + 1) >> 1) & 1));
            }
            return;
        }
        mbar_try_wait(&bar[st], parity);
        pending &= ~(1u << st);
        const unsigned char *sb = smem + st * stage;
        const float *as = (const float *)(sb + L.a_off());
        const short *os = (const short *)(sb + L.o_off());
        float a[32];
        int o[32];
#pragma unroll
        for (int j = 0; j < 32; j++) {
            a[j] = j < k ? as[j * kTileRows + tid] : 0.f;
            o[j] = j < k ? (int)os[j * kTileRows + tid] : 0;
        }
        __syncthreads();  // stage st is free again
        if (tile + 2 * (int)gridDim.x < ntiles) issue(tile + 2 * gridDim.x, st);
        const int i = tile * kTileRows + tid;
        if (i < n) {
            const float ei = e[i];
            if (btag[i]) {
                out[i] = MODE == 0 ? ei : 0.f;
            } else {
                float x[32];
#pragma unroll
                for (int j = 0; j < 32; j++) x[j] = j < k ? __ldg(e + i + o[j]) : 0.f;
                float s = 0.f;
#pragma unroll
                for (int j = 0; j < 32; j++)
                    if (j < k) s += a[j] * x[j];
                if (MODE == 0) {
                    const float q = r[i] - s;
                    const float di = first ? c2 * dinv[i] * q : c1 * d[i] + c2 * dinv[i] * q;
                    d[i] = di;
                    out[i] = ei + di;
                } else {
                    out[i] = r[i] - s;
                }
            }
        }
    }
}

template <class K>
static int tiled_grid(K kernel, int n, size_t smem)
{
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        MGM_CUDA(cudaGetDevice(&dev));
        MGM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    }
    int per_sm = 0;
    MGM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kTileRows, smem));
    const int tiles = (n + kTileRows - 1) / kTileRows;
    return std::max(1, std::min(tiles, sms * std::max(1, per_sm)));
}

template <int MODE>
static void launch_tiled(const SolveLevel<float> &L, const float *e, float *out, float c1, float c2, int first,
                         cudaStream_t s, Chain &launch)
{
    const size_t smem = 2 * tile_stage_bytes(L.k);
    if (L.k <= 32) {
        MGM_CUDA(cudaFuncSetAttribute(k_level_tiled_r<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)(2 * tile_stage_bytes(32))));
        launch.plain(k_level_tiled_r<MODE>, tiled_grid(k_level_tiled_r<MODE>, L.n, smem), kTileRows, smem, s, L.n,
                     L.k, L.offt, L.At, L.dinv, L.btag, L.r, e, out, L.d, c1, c2, first, L.tma_err);
    } else {
        MGM_CUDA(cudaFuncSetAttribute(k_level_tiled<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)(2 * tile_stage_bytes(kTileMaxK))));
        launch.plain(k_level_tiled<MODE>, tiled_grid(k_level_tiled<MODE>, L.n, smem), kTileRows, smem, s, L.n, L.k,
                     L.offt, L.At, L.dinv, L.btag, L.r, e, out, L.d, c1, c2, first, L.tma_err);
    }
}

// e = inv * r, one warp per row of the dense coarsest inverse
template <class T>
__device__ __forceinline__ void dense_row_warp(int w, int lane, int n, const T *__restrict__ inv, const T *r, T *e)
{
    const T *row = inv + (long)w * n;
    T s = T(0);
    for (int j = lane; j < n; j += 32) s += row[j] * __ldcg(r + j);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) e[w] = s;
}

// The first 1024 columns' operands are fetched before the wait.
template <class T>
__global__ void __launch_bounds__(256) k_dense_solve(int n, const T *__restrict__ inv, const T *r, T *e)
{
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    const T *row = inv + (long)w * n;
    constexpr int Q = 32;
    T a[Q];
    if (w < n) {
#pragma unroll
        for (int q = 0; q < Q; q++)
            if (lane + 32 * q < n) a[q] = ldk(row + lane + 32 * q);
    }
    pdl_wait<true>();
    if (w >= n) return;
    T s = T(0);
#pragma unroll
    for (int q = 0; q < Q; q++)
        if (lane + 32 * q < n) s = fma_rn(a[q], __ldcg(r + lane + 32 * q), s);
    for (int j = lane + 32 * Q; j < n; j += 32) s = fma_rn(__ldg(row + j), __ldcg(r + j), s);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) e[w] = s;
}

// ---------------------------------------------------------------------------
// fused coarse-level V-cycle
//
// The levels below kVecMinRows rows are latency-bound: each operation of the
// V-cycle on them (about 17 per level) is a short kernel whose launch and
// ramp cost as much as its work.  k_coarse_vcycle runs the whole V-cycle from
// level `first` down to the coarsest and back as ONE cooperative launch: one
// CTA per SM, every operation a grid-stride pass over the level's rows with
// the row work of the one-operation kernels (so the same bits), and a grid
// barrier between dependent passes.
// ---------------------------------------------------------------------------
constexpr int kFusedMaxLevels = 8, kFusedMaxCheb = 8, kFusedThreads = 512;

template <class T>
struct FusedLevel {
    int n, ld, k, nb_list, kr, kp;
    const short *off;
    const T *A, *dinv;
    const uint8_t *btag;
    const int *bnd_list, *bnd_idx;
    const T *bnd_A;
    const uint8_t *tag;   // near rows and their boundary slots (SolveLevel)
    int nn, ldn, kb;
    const int *near_list, *kb_idx;
    const T *kb_a, *kb_d;
    T *r, *e, *e2, *d, *q;
    const short *r_off;   // restriction into this level (compact)
    const int *r_base;
    const T *r_w;
    const short *p_off;   // prolongation from the next coarser level into this one (compact)
    const int *p_base;
    const T *p_w;
    T c1[kFusedMaxCheb], c2[kFusedMaxCheb];  // Chebyshev coefficients of each step
};

template <class T>
struct FusedArgs {
    int first, nl, deg;
    int cn;        // coarsest rows
    const T *cinv; // its dense inverse
    unsigned *bar; // grid barrier: {arrivals, generation}
    int *err;      // set when a barrier wait runs out
    FusedLevel<T> L[kFusedMaxLevels];
};

template <class T>
__global__ void __launch_bounds__(kFusedThreads) k_coarse_vcycle(const __grid_constant__ FusedArgs<T> a)
{
    const int nth = gridDim.x * blockDim.x, tid = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31, nwarp = nth >> 5, wid = tid >> 5;
    __shared__ T shift;
    unsigned gen = 0;
    if (threadIdx.x == 0) gen = *(volatile unsigned *)&a.bar[1];
#define MGM_SYNC() \
    if (!grid_barrier(a.bar, a.err, gen)) return
    T *cur[kFusedMaxLevels], *nxt[kFusedMaxLevels];
    auto bnd = [&](int l) -> bool {
        const FusedLevel<T> &L = a.L[l];
        for (int w = wid; w < L.nb_list; w += nwarp) {
            BndRow<T> B;
            B.fetch(w, lane, L.nb_list, L.bnd_list, L.k, L.bnd_idx, L.bnd_A, L.dinv);
            const T v = B.value(lane, L.k, L.bnd_idx, L.bnd_A, L.r, cur[l]);
            if (lane == 0) cur[l][B.i] = v;
        }
        return grid_barrier(a.bar, a.err, gen);
    };
    auto pass = [&](int l, int mode, T c1, T c2, int first, T *out) -> bool {
        const FusedLevel<T> &L = a.L[l];
        StepArgsL<T> g{};
        g.out = out; g.d = L.d; g.c1 = c1; g.c2 = c2; g.first = first;
        const T *e = cur[l];
        for (int i = tid; i < L.n; i += nth) {
            const T ei = __ldcg(e + i);
            if (L.btag[i]) {
                out[i] = mode == 0 ? ei : T(0);
                continue;
            }
            const T s = ell_row_dot_o(L.off, L.A, e, L.ld, L.k, i, i);
            const T ri = __ldcg(L.r + i), dprev = mode == 0 && !first ? __ldcg(L.d + i) : T(0);
            if (mode == 0) step_out<0>(g, i, ri, ei, dprev, L.dinv[i], s);
            else step_out<1>(g, i, ri, ei, dprev, L.dinv[i], s);
        }
        return grid_barrier(a.bar, a.err, gen);
    };
    // one smoothing pass on level l: deg Chebyshev steps, each followed by
    // the boundary rows' exact solve; from e = 0 (the first step by first_row
    // and first_near) or from the current e
    auto smooth = [&](int l, bool zero_start) -> bool {
        const FusedLevel<T> &L = a.L[l];
        if (!zero_start && !bnd(l)) return false;
        for (int st = 0; st < a.deg; st++) {
            if (st == 0 && zero_start) {
                FirstArgs<T> f{};
                f.n = L.n; f.nn = L.nn; f.kb = L.kb; f.ldn = L.ldn; f.tag = L.tag; f.dinv = L.dinv;
                f.r = L.r; f.out = nxt[l]; f.d = L.d; f.c2 = L.c2[0]; f.near_list = L.near_list;
                f.kb_idx = L.kb_idx; f.kb_a = L.kb_a; f.kb_d = L.kb_d;
                for (int i = tid; i < L.n; i += nth) first_row<T, false>(f, i, L.tag[i], L.dinv[i]);
                for (int t = tid; t < L.nn; t += nth) first_near<T, false>(f, t);
                if (!grid_barrier(a.bar, a.err, gen)) return false;
            } else if (!pass(l, 0, L.c1[st], L.c2[st], st == 0 ? 1 : 0, nxt[l])) {
                return false;
            }
            T *t = cur[l]; cur[l] = nxt[l]; nxt[l] = t;
            if (!bnd(l)) return false;
        }
        return true;
    };
    for (int l = a.first; l < a.nl; l++) { cur[l] = a.L[l].e; nxt[l] = a.L[l].e2; }
    for (int l = a.first; l < a.nl - 1; l++) {
        const FusedLevel<T> &L = a.L[l], &C = a.L[l + 1];
        if (!smooth(l, true)) return;
        if (!pass(l, 1, T(0), T(0), 0, L.q)) return;
        for (int i = tid; i < C.n; i += nth)
            restrict_row<T>(i, C.n, C.kr, C.r_off, C.r_base, C.r_w, C.btag, L.q, C.r);
        MGM_SYNC();
    }
    {
        const FusedLevel<T> &L = a.L[a.nl - 1];
        for (int w = wid; w < a.cn; w += nwarp) dense_row_warp<T>(w, lane, a.cn, a.cinv, L.r, cur[a.nl - 1]);
        MGM_SYNC();
    }
    for (int l = a.nl - 2; l >= a.first; l--) {
        const FusedLevel<T> &L = a.L[l];
        if (threadIdx.x < 32) {
            const T s = prolong_shift_warp<T>(L.n, L.kp, L.p_off, L.p_base, L.p_w, (const T *)cur[l + 1]);
            if (threadIdx.x == 0) shift = s;
        }
        __syncthreads();
        for (int i = tid; i < L.n; i += nth)
            prolong_row<T>(i, L.n, L.kp, L.p_off, L.p_base, L.p_w, (const T *)cur[l + 1], cur[l], shift);
        MGM_SYNC();
        if (!smooth(l, false)) return;
    }
#undef MGM_SYNC
}

// Whether levels first..nl-1 can run fused: small (one-row-per-thread)
// compact levels without the tile-streamed or FP16 operator.
template <class T>
static bool fusable(const std::vector<SolveLevel<T>> &Ls, int first, int deg)
{
    const int nl = (int)Ls.size();
    if (first >= nl - 1 || nl > kFusedMaxLevels || deg > kFusedMaxCheb || deg < 1) return false;
    for (int l = first; l < nl; l++) {
        const SolveLevel<T> &L = Ls[l];
        if (l < nl - 1) {
            if (L.n >= kVecMinRows || !L.off || L.At || L.W16 || !L.p_off) return false;
        }
        if (l > first && !L.r_off) return false;
    }
    return true;
}

template <class T>
static void launch_fused(std::vector<SolveLevel<T>> &Ls, const CoarseSolve<T> &cs, int first, int deg, double ratio,
                         cudaStream_t s, const FusedCtl &fc)
{
    FusedArgs<T> a{};
    a.first = first;
    a.nl = (int)Ls.size();
    a.deg = deg;
    a.cn = cs.n;
    a.cinv = cs.inv;
    a.bar = fc.bar;
    a.err = fc.err;
    for (int l = first; l < a.nl; l++) {
        const SolveLevel<T> &S = Ls[l];
        FusedLevel<T> &F = a.L[l];
        F.n = S.n; F.ld = S.ld; F.k = S.k; F.nb_list = S.nb_list; F.kr = S.kr; F.kp = S.kp;
        F.off = S.off; F.A = S.A; F.dinv = S.dinv; F.btag = S.btag;
        F.bnd_list = S.bnd_list; F.bnd_idx = S.bnd_idx; F.bnd_A = S.bnd_A;
        F.tag = S.tag; F.nn = S.nn; F.ldn = S.ldn; F.kb = S.kb; F.near_list = S.near_list;
        F.kb_idx = S.kb_idx; F.kb_a = S.kb_a; F.kb_d = S.kb_d;
        F.r = S.r; F.e = S.e; F.e2 = S.e2; F.d = S.d; F.q = S.q;
        F.r_off = S.r_off; F.r_base = S.r_base; F.r_w = S.r_w;
        F.p_off = S.p_off; F.p_base = S.p_base; F.p_w = S.p_w;
        // the coefficients smooth() passes to the level kernels, step by step
        const double lM = 1.05 * S.lmax, lm = S.lmax / ratio;
        const double th = 0.5 * (lM + lm), de = 0.5 * (lM - lm), sig = th / de;
        double rho = 1.0 / sig;
        for (int st = 0; st < deg; st++) {
            double c1 = 0, c2;
            if (st == 0) c2 = 1.0 / th;
            else {
                const double rn = 1.0 / (2.0 * sig - rho);
                c1 = rn * rho;
                c2 = 2.0 * rn / de;
                rho = rn;
            }
            F.c1[st] = (T)c1;
            F.c2[st] = (T)c2;
        }
    }
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(fc.blocks);
    cfg.blockDim = dim3(kFusedThreads);
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, k_coarse_vcycle<T>, a);
    if (e != cudaSuccess) throw Error{1, std::string("kernel launch (cooperative): ") + cudaGetErrorString(e)};
    MGM_LAUNCHED();
}

// Self-test of the grid barrier's bounded wait: CTA 1 returns without
// arriving, so CTA 0's wait runs out, sets *err and returns.
__global__ void k_barrier_selftest(unsigned *bar, int *err)
{
    unsigned gen = 0;
    if (threadIdx.x == 0) gen = *(volatile unsigned *)&bar[1];
    if (blockIdx.x == 1) return;
    grid_barrier(bar, err, gen);
}
cudaError_t launch_barrier_selftest(cudaStream_t s, unsigned *bar, int *err)
{
    return launch_cooperative(k_barrier_selftest, 2, 32, 0, s, bar, err);
}

// a cooperative launch of one CTA that does nothing (capture probe)
__global__ void k_coop_probe(int) {}
cudaError_t launch_coop_probe(cudaStream_t s)
{
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1);
    cfg.blockDim = dim3(32);
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_coop_probe, 0);
}

int fused_vcycle_blocks()
{
    int dev = 0, sms = 0, per32 = 0, per64 = 0;
    MGM_CUDA(cudaGetDevice(&dev));
    MGM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    MGM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per32, k_coarse_vcycle<float>, kFusedThreads, 0));
    MGM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per64, k_coarse_vcycle<double>, kFusedThreads, 0));
    MGM_REQUIRE(per32 >= 1 && per64 >= 1, "fused coarse V-cycle: a CTA does not fit on an SM");
    return sms;  // one CTA per SM
}

void SmootherProfile::mark(cudaStream_t s)
{
    if (used >= ev.size()) {
        size_t old = ev.size();
        ev.resize(std::max<size_t>(256, old * 2));
        for (size_t i = old; i < ev.size(); i++) MGM_CUDA(cudaEventCreate(&ev[i]));
    }
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    MGM_CUDA(cudaStreamIsCapturing(s, &st));
    // inside a capture the record must become an event-record node of the graph
    if (st == cudaStreamCaptureStatusActive) MGM_CUDA(cudaEventRecordWithFlags(ev[used++], s, cudaEventRecordExternal));
    else MGM_CUDA(cudaEventRecord(ev[used++], s));
}

void SmootherProfile::harvest()
{
    for (size_t i = 0; i + 1 < used; i += 2) {
        float t = 0;
        MGM_CUDA(cudaEventElapsedTime(&t, ev[i], ev[i + 1]));
        ms += t;
        launches++;
    }
    used = 0;
}

void SmootherProfile::harvest_graph(size_t first, size_t pairs)
{
    for (size_t q = 0; q < pairs; q++) {
        float t = 0;
        MGM_CUDA(cudaEventElapsedTime(&t, ev[first + 2 * q], ev[first + 2 * q + 1]));
        ms += t;
        launches++;
    }
}

SmootherProfile::~SmootherProfile()
{
    for (cudaEvent_t e : ev) cudaEventDestroy(e);
}

// step coefficients of the Chebyshev polynomial on [lmax / ratio, 1.05 lmax]
struct ChebCoef {
    double th, de, sig, rho;
    ChebCoef(double lmax, double ratio)
    {
        const double lM = 1.05 * lmax, lm = lmax / ratio;
        th = 0.5 * (lM + lm);
        de = 0.5 * (lM - lm);
        sig = th / de;
        rho = 1.0 / sig;
    }
    void next(int step, double &c1, double &c2)
    {
        c1 = 0;
        if (step == 0) {
            c2 = 1.0 / th;
        } else {
            const double rn = 1.0 / (2.0 * sig - rho);
            c1 = rn * rho;
            c2 = 2.0 * rn / de;
            rho = rn;
        }
    }
};

// One step on a level (MODE 0 Chebyshev, MODE 1 residual) with the boundary
// rows' exact solve before it, by the level's variant: the tile-streamed and
// FP16 kernels take the boundary rows as a launch of their own.
template <int MODE, class T>
static void launch_step(const SolveLevel<T> &L, T *e, T *out, T c1, T c2, int first, cudaStream_t s, Chain &launch,
                        SmootherProfile *prof)
{
    auto mark = [&] {
        if (prof) {
            prof->mark(s);
            launch.broken();
        }
    };
    if constexpr (sizeof(T) == 4) {
        if (L.At || L.W16) {
            launch_bnd(L, e, s, launch);
            mark();
            if (L.At)
                launch_tiled<MODE>(L, e, out, (float)c1, (float)c2, first, s, launch);
            else
                launch(k_level_h4<MODE>, blocks_for(L.ldi / 4, 256), 256, 0, s, L.n, L.ldi, L.k, L.W16, L.dinv,
                       L.btag, L.r, (const float *)e, out, L.d, c1, c2, first);
            mark();
            return;
        }
    }
    const bool big = L.off && L.n >= kVecMinRows;
    // One launch with the boundary part pays while that part is small beside
    // the far part (the 500^2 cavity, 63 CTAs beside 245: 17 us against
    // 16.0 + 4.2); in 3D it is not (the 64^3 cube, 721 beside 256; with four
    // times as many 44 us against 19.6 + 6.3, the far part waits for slots).
    const int nbc = bnd_blocks(L.nb_list, true), nfar = blocks_for(L.n, 1024);
    const bool one = big && nbc <= 2 * nfar;
    if (!one) launch_bnd(L, e, s, launch);
    mark();
    if (big) {
        StepArgsL<T> a = step_args_of(L, e, out, c1, c2, first);
        a.nfar = nfar;
        a.fb = nfar;
        if (one) {
            a.nbc = nbc;
            a.nnc = blocks_for(L.nn, 256);
            // more far CTAs than the chip holds at once: the boundary part
            // goes in the middle, where it fills freed slots; else after them
            if (nfar > 148 * 4) a.fb = nfar / 2;
        }
        launch(k_level_v4<MODE, T>, a.nbc + a.nfar + a.nnc, 256, 0, s, a);
    } else if (L.off) {
        launch_c1<MODE, T, false>(L, e, out, c1, c2, first, s, launch);
    } else {
        launch_c1<MODE, T, true>(L, e, out, c1, c2, first, s, launch);
    }
    mark();
}

// where the first smoothing step of level 0 takes its right-hand side from:
// the FP64 Krylov vector V_j (V non-null), else the level's r
struct FirstSrc {
    const double *V = nullptr;
    long ld = 0;
    const FgState *st = nullptr;
};

// the first step of a pass from e = 0, into L.e2; then the buffers swap
template <class T>
static void first_step(SolveLevel<T> &L, double ratio, const FirstSrc &src, cudaStream_t s, Chain &launch)
{
    double c1, c2;
    ChebCoef(L.lmax, ratio).next(0, c1, c2);
    FirstArgs<T> a{};
    a.n = L.n; a.nn = L.nn; a.kb = L.kb; a.ldn = L.ldn;
    a.nrow = blocks_for(L.n, 256);
    a.tag = L.tag; a.dinv = L.dinv; a.r = L.r; a.out = L.e2; a.d = L.d; a.c2 = (T)c2;
    a.near_list = L.near_list; a.kb_idx = L.kb_idx; a.kb_a = L.kb_a; a.kb_d = L.kb_d;
    a.V = src.V; a.ldv = src.ld; a.st = src.st;
    const int grid = a.nrow + blocks_for(L.nn, 256);
    const bool early = L.n < kVecMinRows;
    if (src.V) {
        if (early) launch(k_first_step<T, true, true>, grid, 256, 0, s, a);
        else launch(k_first_step<T, true, false>, grid, 256, 0, s, a);
    } else {
        if (early) launch(k_first_step<T, false, true>, grid, 256, 0, s, a);
        else launch(k_first_step<T, false, false>, grid, 256, 0, s, a);
    }
    std::swap(L.e, L.e2);
}

// Chebyshev steps from .. degree - 1 of a pass, each after the boundary rows'
// exact solve from the current e; the pass's last boundary solve is the
// caller's (the residual step does its own)
template <class T>
static void smooth_steps(SolveLevel<T> &L, int from, int degree, double ratio, cudaStream_t s, SmootherProfile *prof,
                         Chain &launch)
{
    ChebCoef cc(L.lmax, ratio);
    for (int step = 0; step < degree; step++) {
        double c1, c2;
        cc.next(step, c1, c2);
        if (step < from) continue;
        launch_step<0, T>(L, L.e, L.e2, (T)c1, (T)c2, step == 0 ? 1 : 0, s, launch, prof);
        std::swap(L.e, L.e2);
    }
}

template <class T>
static void vcycle_rec(std::vector<SolveLevel<T>> &Ls, const CoarseSolve<T> &cs, int l, int deg, double ratio,
                       cudaStream_t s, SmootherProfile *prof, Chain &launch, const FusedCtl *fused,
                       const FirstSrc &src)
{
    SmootherProfile *lp = (l == 0 && prof && prof->on) ? prof : nullptr;
    SolveLevel<T> &L = Ls[l];
    const int nl = (int)Ls.size();
    if (l == 0 && (nl == 1 || (fused && fused->on && fusable(Ls, 0, deg))) && src.V) {
        // level 0 itself is the fused or the dense level: r on its own
        fg_load<T>(L.n, src.V, src.ld, src.st, L.r, s);
        launch.broken();
    }
    if (fused && fused->on && fusable(Ls, l, deg)) {
        // levels l..nl-1 in one cooperative launch; each level's correction
        // ends in its e buffer, as after the 2 deg swaps of the per-level path
        launch_fused(Ls, cs, l, deg, ratio, s, *fused);
        launch.after_kernel = true;
        return;
    }
    if (l == nl - 1) {
        launch(k_dense_solve<T>, blocks_for((long)L.n * 32, 256), 256, 0, s, cs.n, cs.inv, L.r, L.e);
        return;
    }
    // from e = 0; below level 0 the restriction into the level did the first step (into e2)
    if (l == 0) first_step(L, ratio, src, s, launch);
    smooth_steps(L, 1, deg, ratio, s, lp, launch);
    launch_step<1, T>(L, L.e, L.q, T(0), T(0), 0, s, launch, nullptr);
    SolveLevel<T> &C = Ls[l + 1];
    if (l + 1 == nl - 1 || (fused && fused->on && fusable(Ls, l + 1, deg))) {
        launch_restrict<T, false>(C, L.q, T(0), s, launch);
    } else {
        double c1, c2;
        ChebCoef(C.lmax, ratio).next(0, c1, c2);
        std::swap(C.e, C.e2);
        launch_restrict<T, true>(C, L.q, (T)c2, s, launch);
    }
    vcycle_rec(Ls, cs, l + 1, deg, ratio, s, prof, launch, fused, src);
    launch_prolong<T>(L, C.e, s, launch);
    smooth_steps(L, 0, deg, ratio, s, lp, launch);
    launch_bnd(L, L.e, s, launch);
}

template <class T>
void vcycle(std::vector<SolveLevel<T>> &Ls, const CoarseSolve<T> &cs, int cheb_degree, double cheb_ratio,
            cudaStream_t s, SmootherProfile *prof, bool chain, const FusedCtl *fused, const double *V, long ldv,
            const FgState *st)
{
    Chain launch;
    launch.enabled = chain;
    FirstSrc src;
    src.V = V;
    src.ld = ldv;
    src.st = st;
    vcycle_rec(Ls, cs, 0, cheb_degree, cheb_ratio, s, prof, launch, fused, src);
}

// Chebyshev smoothing of A e = r on one level from e = 0 (r already in L.r);
// returns the buffer holding e.
template <class T>
const T *smooth_from_zero(SolveLevel<T> &L, int degree, double ratio, cudaStream_t s, bool chain)
{
    Chain launch;
    launch.enabled = chain;
    first_step(L, ratio, FirstSrc(), s, launch);
    smooth_steps(L, 1, degree, ratio, s, (SmootherProfile *)nullptr, launch);
    launch_bnd(L, L.e, s, launch);
    return L.e;
}
template const double *smooth_from_zero<double>(SolveLevel<double> &, int, double, cudaStream_t, bool);
template const float *smooth_from_zero<float>(SolveLevel<float> &, int, double, cudaStream_t, bool);

template void vcycle<double>(std::vector<SolveLevel<double>> &, const CoarseSolve<double> &, int, double, cudaStream_t,
                             SmootherProfile *, bool, const FusedCtl *, const double *, long, const FgState *);
template void vcycle<float>(std::vector<SolveLevel<float>> &, const CoarseSolve<float> &, int, double, cudaStream_t,
                            SmootherProfile *, bool, const FusedCtl *, const double *, long, const FgState *);

// ---------------------------------------------------------------------------
// spectral radius of D^-1 A restricted to interior rows (power iteration)
// ---------------------------------------------------------------------------
// w = D^-1 A (v scale) with scale the previous step's 1 / |w| (null: 1)
template <class T>
__global__ void __launch_bounds__(256) k_power_step(int n, int k, const int *__restrict__ idx, const T *__restrict__ A,
                                                    const T *__restrict__ dinv, const uint8_t *__restrict__ btag,
                                                    const double *__restrict__ v, const double *__restrict__ scale,
                                                    double *__restrict__ w, double *__restrict__ partial)
{
    __shared__ double sm[32];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const double f = scale ? *scale : 1.0;
    double val = 0.0;
    if (i < n && !btag[i]) {
        double s = 0.0;
        int j = 0;
        for (; j + 8 <= k; j += 8) {  // 8 slots' loads in flight, summed in slot order
            int c[8];
            double a[8], x[8];
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const long o = (long)(j + q) * n + i;
                c[q] = __ldg(idx + o);
                a[q] = (double)__ldg(A + o);
            }
#pragma unroll
            for (int q = 0; q < 8; q++) x[q] = __ldg(v + c[q]);
#pragma unroll
            for (int q = 0; q < 8; q++) s = fma(a[q], __dmul_rn(x[q], f), s);
        }
        for (; j < k; j++) {
            const long o = (long)j * n + i;
            s = fma((double)A[o], __dmul_rn(v[idx[o]], f), s);
        }
        val = (double)dinv[i] * s;
    }
    if (i < n) w[i] = val;
    double sq = block_sum_d<256>(val * val, sm);
    if (threadIdx.x == 0) partial[blockIdx.x] = sq;
}

__global__ void k_seed_vector(int n, const uint8_t *btag, double *v)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    // deterministic pseudo-random start vector (integer hash of the index)
    unsigned h = (unsigned)i * 2654435761u;
    h ^= h >> 16; h *= 2246822519u; h ^= h >> 13;
    v[i] = btag[i] ? 0.0 : ((double)(h & 0xffffff) / 16777216.0 - 0.5);
}

// The partials' sum in block order (through shared memory, added by one
// thread): out[0] = 1 / sqrt(sum), out[1] = sqrt(sum)
__global__ void __launch_bounds__(256) k_power_norm(const double *__restrict__ partial, int nparts, double *out)
{
    __shared__ double sm[2048];
    double s = 0;
    for (int t0 = 0; t0 < nparts; t0 += 2048) {
        const int m = min(2048, nparts - t0);
        __syncthreads();
        for (int t = threadIdx.x; t < m; t += 256) sm[t] = partial[t0 + t];
        __syncthreads();
        if (threadIdx.x == 0)
            for (int t = 0; t < m; t++) s += sm[t];
    }
    if (threadIdx.x == 0) {
        out[0] = s > 0 ? 1.0 / sqrt(s) : 0.0;
        out[1] = sqrt(s);
    }
}

// 40 steps without the host: the norm stays on the device and the next step
// applies it (with a read of each step's partials 160 steps of four levels of up
// to 250k rows took 10 ms, now 2.1)
template <class T>
void estimate_lmax(SolveLevel<T> &L, cudaStream_t s)
{
    const int nb = blocks_for(L.n, 256);
    DBuf<double> v(L.n), w(L.n), part(nb), norm(2);
    k_seed_vector<<<nb, 256, 0, s>>>(L.n, L.btag, v.p);
    MGM_LAUNCHED();
    constexpr int kSteps = 40;
    for (int it = 0; it < kSteps; it++) {
        k_power_step<T><<<nb, 256, 0, s>>>(L.n, L.k, L.idx, L.A, L.dinv, L.btag, v.p, it > 0 ? norm.p : nullptr, w.p,
                                           part.p);
        MGM_LAUNCHED();
        k_power_norm<<<1, 256, 0, s>>>(part.p, nb, norm.p);
        MGM_LAUNCHED();
        std::swap(v.p, w.p);
    }
    double h[2];
    norm.download(h, 2, s);
    MGM_CUDA(cudaStreamSynchronize(s));
    const double lam = h[1];  // |v| was 1 before the last step
    L.lmax = lam > 0 && std::isfinite(lam) ? lam : 2.0;
}

template void estimate_lmax<double>(SolveLevel<double> &, cudaStream_t);

}  // namespace mgm
