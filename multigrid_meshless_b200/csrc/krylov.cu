// krylov.cu -- FP64 vector kernels of the flexible GMRES outer iteration and
// the dense Gauss-Jordan (partial pivoting) used once at set-up for the
// coarsest-level inverse.
#include "coop.cuh"
#include "krylov.cuh"
#include "rows.cuh"

namespace mgm {

template <int BS>
__device__ __forceinline__ double bsum(double v, double *sm)
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

// r = b - A x  (A: pinned FP64 operator, ELL), and per-block |r|^2, |b|^2 partials
__global__ void __launch_bounds__(256) k_resid64(int n, int k, const int *__restrict__ idx, const double *__restrict__ A,
                                                 const double *__restrict__ b, const double *__restrict__ x,
                                                 double *__restrict__ r, double *__restrict__ part)
{
    __shared__ double sm[32];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double rr = 0, bb = 0;
    if (i < n) {
        const double ri = b[i] - ell_row_dot(idx, A, x, n, k, i);
        r[i] = ri;
        rr = ri * ri;
        bb = b[i] * b[i];
    }
    rr = bsum<256>(rr, sm);
    bb = bsum<256>(bb, sm);
    if (threadIdx.x == 0) { part[2 * blockIdx.x] = rr; part[2 * blockIdx.x + 1] = bb; }
}

// w = A z  (z in precision T)
template <class T>
__global__ void __launch_bounds__(256) k_apply64(int n, int k, const int *__restrict__ idx, const double *__restrict__ A,
                                                 const T *__restrict__ z, double *__restrict__ w)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    w[i] = ell_row_dot(idx, A, z, n, k, i);
}

// partial dot products h_c = V_c . w for c < cnt; part[c * nblk + blk]
__global__ void __launch_bounds__(256) k_multidot(int n, int cnt, const double *__restrict__ V, long ldv,
                                                  const double *__restrict__ w, double *__restrict__ part)
{
    __shared__ double sm[32];
    for (int c = 0; c < cnt; c++) {
        double s = 0.0;
        const double *vc = V + c * ldv;
        for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
            s = fma(vc[i], w[i], s);
        s = bsum<256>(s, sm);
        if (threadIdx.x == 0) part[(long)c * gridDim.x + blockIdx.x] = s;
    }
}

// out[c] = sum_t part[c * nblk + t]; one block per c
__global__ void k_reduce_parts(const double *__restrict__ part, int nblk, int cnt, double *__restrict__ out)
{
    __shared__ double sm[32];
    const int c = blockIdx.x;
    if (c >= cnt) return;
    double s = 0.0;
    for (int t = threadIdx.x; t < nblk; t += blockDim.x) s += part[(long)c * nblk + t];
    s = bsum<256>(s, sm);
    if (threadIdx.x == 0) out[c] = s;
}

// x += sum_c y[c] Z_c  (Z in precision T)
template <class T>
__global__ void __launch_bounds__(256) k_combine(int n, int cnt, const T *__restrict__ Z, long ldz,
                                                 const double *__restrict__ y, double *__restrict__ x)
{
    __shared__ double ys[kMaxKrylov + 1];
    for (int c = threadIdx.x; c < cnt; c += blockDim.x) ys[c] = y[c];
    __syncthreads();
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double s = x[i];
    for (int c = 0; c < cnt; c++) s = fma(ys[c], (double)Z[c * ldz + i], s);
    x[i] = s;
}

template <class T>
__global__ void k_copy_convert(long n, const double *__restrict__ in, T *__restrict__ out)
{
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = (T)in[i];
}

template <class T>
__global__ void k_copy_out(long n, const T *__restrict__ in, T *__restrict__ out)
{
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = in[i];
}

void resid64(int n, int k, const int *idx, const double *A, const double *b, const double *x, double *r, double *part,
             cudaStream_t s)
{
    k_resid64<<<blocks_for(n, 256), 256, 0, s>>>(n, k, idx, A, b, x, r, part);
    MGM_LAUNCHED();
}
template <class T>
void apply64(int n, int k, const int *idx, const double *A, const T *z, double *w, cudaStream_t s)
{
    k_apply64<T><<<blocks_for(n, 256), 256, 0, s>>>(n, k, idx, A, z, w);
    MGM_LAUNCHED();
}
template void apply64<double>(int, int, const int *, const double *, const double *, double *, cudaStream_t);
template void apply64<float>(int, int, const int *, const double *, const float *, double *, cudaStream_t);

int dot_blocks(int n) { return std::max(1, std::min(blocks_for(n, 256), 148 * 4)); }

void multidot(int n, int cnt, const double *V, long ldv, const double *w, double *part, double *out, cudaStream_t s)
{
    const int nb = dot_blocks(n);
    k_multidot<<<nb, 256, 0, s>>>(n, cnt, V, ldv, w, part);
    MGM_LAUNCHED();
    k_reduce_parts<<<cnt, 256, 0, s>>>(part, nb, cnt, out);
    MGM_LAUNCHED();
}
template <class T>
void combine(int n, int cnt, const T *Z, long ldz, const double *y, double *x, cudaStream_t s)
{
    k_combine<T><<<blocks_for(n, 256), 256, 0, s>>>(n, cnt, Z, ldz, y, x);
    MGM_LAUNCHED();
}
template void combine<double>(int, int, const double *, long, const double *, double *, cudaStream_t);
template void combine<float>(int, int, const float *, long, const double *, double *, cudaStream_t);
template <class T>
void copy_convert(long n, const double *in, T *out, cudaStream_t s)
{
    k_copy_convert<T><<<blocks_for(n, 256), 256, 0, s>>>(n, in, out);
    MGM_LAUNCHED();
}
template void copy_convert<double>(long, const double *, double *, cudaStream_t);
template void copy_convert<float>(long, const double *, float *, cudaStream_t);
template <class T>
void copy_out(long n, const T *in, T *out, cudaStream_t s)
{
    k_copy_out<T><<<blocks_for(n, 256), 256, 0, s>>>(n, in, out);
    MGM_LAUNCHED();
}
template void copy_out<double>(long, const double *, double *, cudaStream_t);
template void copy_out<float>(long, const float *, float *, cudaStream_t);

// ---------------------------------------------------------------------------
// device-resident FGMRES control (FgState, krylov.cuh)
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void set_cond(cudaGraphConditionalHandle h, int use, int v)
{
    if (use) cudaGraphSetConditional(h, v ? 1u : 0u);
}

__global__ void k_fg_init(FgState *st, int m, int max_total, int max_restarts, double tol)
{
    st->m = m;
    st->max_total = max_total;
    st->max_restarts = max_restarts;
    st->tol = tol;
    st->j = st->j_next = st->j_done = st->total_it = st->restarts = st->vcycles = 0;
    st->reorth = 0;
    st->go_outer = 1;
    st->go_inner = 0;
    st->status = FG_OK;
    st->beta = st->bnorm = 0.0;
    st->relres = 1.0;
    st->alpha = 0.0;
    st->solves_total++;
}

__global__ void k_fg_clear_totals(FgState *st)
{
    st->err_any = 0;
    st->vcycles_total = 0;
    st->cycles_total = 0;
    st->solves_total = 0;
    st->t_ns = 0;
    st->start_log_relres = 0.0;
}

__global__ void k_fg_time_mark(FgState *st, int end)
{
    const unsigned long long t = global_ns();
    if (end) st->t_ns += t - st->t_mark;
    else st->t_mark = t;
}

// Start of a restart cycle: |r|^2, |b|^2 from the residual kernel's per-block
// partials (fixed-order block reduction), the convergence test, and the
// Krylov right-hand side g = beta e_0.
__global__ void __launch_bounds__(256) k_fg_begin(FgState *st, const double *__restrict__ part, int nbres,
                                                  FgHandles hd)
{
    __shared__ double sm[32];
    double rr = 0.0, bb = 0.0;
    for (int t = threadIdx.x; t < nbres; t += blockDim.x) {
        rr += part[2 * t];
        bb += part[2 * t + 1];
    }
    rr = bsum<256>(rr, sm);
    bb = bsum<256>(bb, sm);
    if (threadIdx.x != 0) return;
    const double bnorm = sqrt(bb), beta = sqrt(rr);
    const double relres = bnorm > 0 ? beta / bnorm : 0.0;
    st->bnorm = bnorm;
    st->beta = beta;
    st->relres = relres;
    // the solve's first cycle: the residual its initial guess left
    if (st->restarts == 0 && st->total_it == 0 && relres > 0 && isfinite(relres))
        st->start_log_relres += log10(relres);
    st->j = 0;
    st->j_next = 0;
    st->j_done = 0;
    int go = 0;
    if (!isfinite(relres)) {
        st->status = FG_NONFINITE;
        st->err_any |= 1;
    } else if (!(bnorm == 0 || relres < st->tol || st->total_it >= st->max_total)) {
        go = 1;
        st->g[0] = beta;
        for (int i = 1; i <= st->m; i++) st->g[i] = 0.0;
    }
    st->go_inner = go;
    // the cycle begun here is the last one when the restart budget is spent
    st->go_outer = go && (st->restarts + 1 <= st->max_restarts);
    if (go) st->restarts++;
    st->cycles_total++;
    set_cond(hd.inner, hd.use, st->go_inner);
    set_cond(hd.outer, hd.use, st->go_outer);
}

// V_0 = r / beta
__global__ void k_fg_scale0(int n, double *__restrict__ V, const FgState *__restrict__ st)
{
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double d = st->beta;
    V[i] = d > 0 ? V[i] / d : 0.0;
}

template <class T>
__global__ void k_fg_load(int n, const double *__restrict__ V, long ld, const FgState *__restrict__ st,
                          T *__restrict__ out)
{
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = (T)V[st->j_next * ld + i];
}

// ---------------------------------------------------------------------------
// The Arnoldi step after the V-cycle, chained launches.
//
//   k_fg_apply   w = A z into V_{j+1}, Z_j = z; on levels below kVecMinRows
//                rows also the per-CTA partial sums of V_c . w (c <= j) and w . w
//   k_fg_dots    those partial sums on the larger levels
//   k_fg_orth1   h = the summed projections; w -= sum h_c V_c; partial sums of
//                V_c . w and w . w of the result
//   k_fg_orth2   when the first pass cancelled more than 1 - 1/sqrt(2) of |w|
//                (the Daniel-Gragg-Kaufman-Stewart test): w -= sum h2_c V_c,
//                partial sums of w . w
//   k_fg_end     w /= |w|; CTA 0: Hessenberg column, Givens rotations, the
//                residual estimate and the inner loop's condition
//
// A V-cycle reduces the error by about three, so w = A M v_j is close to v_j
// and the second pass runs nearly every time: orth1 reads each V_c once for
// the update and for the second pass's projections (a separate dot pass read
// them again).  Below kFgSmall rows every CTA sums the partial sums it needs
// itself; above, where they are up to 592 per vector, k_fg_reduce does.  The
// small levels' step is 4 launches where it was 13 (36 us of the 128 us a
// whole step took on 16k rows).
//
// Every sum keeps one order whatever kernel takes it: a thread's rows, the
// lanes of a warp and the warps of a CTA by halving, the CTAs' partial sums
// the same way from 256 threads.  The FP32 V-cycle inside the iteration
// amplifies the last bit of an FP64 sum to 1e-8 of the solution, so the order
// is part of the result.
// ---------------------------------------------------------------------------
constexpr int kFgThreads = 256, kFgWarps = kFgThreads / 32;
constexpr int kFgSmall = 65536;     // rows from which dot products and their reductions are launches of their own
constexpr int kFgChunk = 16;        // Krylov vectors whose values a thread keeps in registers

// part: [0] projections and |w|^2 of the first pass, [1] of the second, [2] the last |w|^2
static __host__ __device__ size_t fg_part_stride(int nb) { return (size_t)(kMaxKrylov + 2) * nb; }
size_t fg_part_doubles(int n) { return 2 * fg_part_stride(dot_blocks(n)) + dot_blocks(n); }

// the lanes' values by halving (lane 0)
__device__ __forceinline__ double warp_halve(double v)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}
// eight warps' values by halving
__device__ __forceinline__ double warps_halve(const double *s)
{
    return ((s[0] + s[4]) + (s[2] + s[6])) + ((s[1] + s[5]) + (s[3] + s[7]));
}

// out[c] = sum of partial row c (nb values) over the CTA, c < cnt
__device__ __forceinline__ void block_sum_parts(const double *part, int nb, int cnt, double *out,
                                                double (*sm)[kFgWarps])
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int c0 = 0; c0 < cnt; c0 += kFgChunk) {
        double v[kFgChunk];
#pragma unroll
        for (int q = 0; q < kFgChunk; q++) {
            v[q] = 0.0;
            if (c0 + q < cnt)
                for (int t = threadIdx.x; t < nb; t += kFgThreads) v[q] += __ldcg(part + (size_t)(c0 + q) * nb + t);
        }
#pragma unroll
        for (int q = 0; q < kFgChunk; q++) {
            if (c0 + q >= cnt) break;
            const double s = warp_halve(v[q]);
            if (lane == 0) sm[q][warp] = s;
        }
        __syncthreads();
        if (threadIdx.x < kFgChunk && c0 + threadIdx.x < cnt) out[c0 + threadIdx.x] = warps_halve(sm[threadIdx.x]);
        __syncthreads();
    }
}

// the CTA's sums of m per-thread values acc into part[(c0 + q) * nb + blk], q < m
__device__ __forceinline__ void block_store_parts(const double (&acc)[kFgChunk], int m, int c0, double *part, int nb,
                                                  double (*sm)[kFgWarps])
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int q = 0; q < kFgChunk; q++) {
        if (q >= m) break;
        const double v = warp_halve(acc[q]);
        if (lane == 0) sm[q][warp] = v;
    }
    __syncthreads();
    if (threadIdx.x < m) part[(size_t)(c0 + threadIdx.x) * nb + blockIdx.x] = warps_halve(sm[threadIdx.x]);
    __syncthreads();
}

// sums of the partial rows c < cnt (SECOND: of the second pass, the last row
// |w|^2 into st->nrm; third: one row, into st->nrm), one CTA per row
enum FgReduce { FG_RED_FIRST = 0, FG_RED_SECOND = 1, FG_RED_LAST = 2 };
template <int WHICH>
__global__ void __launch_bounds__(kFgThreads) k_fg_reduce(const double *part, int nb, FgState *st)
{
    __shared__ double sm[kFgChunk][kFgWarps];
    __shared__ double out[1];
    pdl_wait<true>();
    const int j = __ldcg(WHICH == FG_RED_FIRST ? &st->j_next : &st->j);
    const int c = blockIdx.x, cnt = WHICH == FG_RED_LAST ? 1 : j + 2;
    if (c >= cnt || (WHICH == FG_RED_LAST && !__ldcg(&st->reorth))) return;
    block_sum_parts(part + (size_t)c * nb, nb, 1, out, sm);
    if (threadIdx.x != 0) return;
    if (WHICH == FG_RED_FIRST) {
        st->h[c] = out[0];
        if (c == 0) st->j = j;
    } else if (WHICH == FG_RED_SECOND && c <= j) {
        st->h2[c] = out[0];
    } else {
        st->nrm = out[0];
    }
}

// a row of the operator in the level's own slot order: KC > 0 int16 offsets in
// padded rows, the first KC slots before the wait; KC = 0 by chunks of 8
// (IDX: 32-bit indices).  SMALL: in a kernel that releases its successor before
// its own wait, which gathers from L2.
template <int KC, bool IDX, bool SMALL>
struct FgRow {
    RowChunk<double, KC ? KC : 8, IDX> R;
    __device__ __forceinline__ void fetch(const FgOperator &op, int i)
    {
        if constexpr (KC > 0) R.fetch(op.gi, op.A, op.n, i, i, 0);
        else R.fetch_to(op.gi, op.A, op.n, i, i, 0, op.k);
    }
    template <class X>
    __device__ __forceinline__ double dot(const FgOperator &op, const X *x, int i)
    {
        if constexpr (KC > 0) {
            const double s = R.template dot<true>(x, 0.0);
            return row_rest<true, double, KC, IDX>(op.gi, op.A, x, op.n, op.kp, i, i, s);
        } else {
            return row_big<double, IDX, SMALL>(R, op.gi, op.A, x, op.n, op.k, i, i);
        }
    }
};

template <class T, int KC, bool IDX, bool SMALL>
__global__ void __launch_bounds__(kFgThreads) k_fg_apply(FgOperator op, const T *z, T *Z, double *V, long ld,
                                                         const FgState *st, double *part)
{
    __shared__ double sm[kFgChunk][kFgWarps];
    const int i0 = blockIdx.x * kFgThreads + threadIdx.x, i = min(i0, op.n - 1);
    FgRow<KC, IDX, SMALL> R;
    R.fetch(op, i);
    pdl_wait<SMALL>();
    const int j = __ldcg(&st->j_next);
    double w = R.dot(op, z, i);
    const bool live = i0 < op.n;
    if (live) {
        Z[(long)j * ld + i] = __ldcg(z + i);
        V[(long)(j + 1) * ld + i] = w;
    }
    if constexpr (SMALL) {
        // dot_blocks(n) CTAs, one row per thread
        for (int c0 = 0; c0 <= j + 1; c0 += kFgChunk) {
            const int m = min(kFgChunk, j + 2 - c0);
            double acc[kFgChunk];
#pragma unroll
            for (int q = 0; q < kFgChunk; q++) acc[q] = q < m && c0 + q <= j ? __ldcg(V + (long)(c0 + q) * ld + i) : w;
#pragma unroll
            for (int q = 0; q < kFgChunk; q++) acc[q] = live ? acc[q] * w : 0.0;
            block_store_parts(acc, m, c0, part, gridDim.x, sm);
        }
    }
}

__global__ void __launch_bounds__(kFgThreads, 2) k_fg_dots(int n, const double *V, long ld, const FgState *st,
                                                        double *part)
{
    __shared__ double sm[kFgChunk][kFgWarps];
    pdl_wait<true>();
    const int j = __ldcg(&st->j_next);
    const double *w = V + (long)(j + 1) * ld;
    for (int c0 = 0; c0 <= j + 1; c0 += kFgChunk) {
        const int m = min(kFgChunk, j + 2 - c0);
        double acc[kFgChunk];
#pragma unroll
        for (int q = 0; q < kFgChunk; q++) acc[q] = 0.0;
        const long step = (long)gridDim.x * kFgThreads;
        for (long i = (long)blockIdx.x * kFgThreads + threadIdx.x; i < n; i += step) {
            const double wi = __ldcg(w + i);
            double v[kFgChunk];
#pragma unroll
            for (int q = 0; q < kFgChunk; q++)
                if (q < m) v[q] = __ldcg(V + (long)(c0 + q) * ld + i);
#pragma unroll
            for (int q = 0; q < kFgChunk; q++)
                if (q < m) acc[q] = fma(v[q], wi, acc[q]);
        }
        block_store_parts(acc, m, c0, part, gridDim.x, sm);
    }
}

template <bool SMALL>
__global__ void __launch_bounds__(kFgThreads, 2) k_fg_orth1(int n, double *V, long ld, FgState *st,
                                                            const double *part, double *part2)
{
    __shared__ double hs[kMaxKrylov + 2];
    __shared__ double sm[kFgChunk][kFgWarps];
    pdl_wait<true>();
    const int j = __ldcg(&st->j_next), nb = gridDim.x;
    if constexpr (SMALL) {
        block_sum_parts(part, nb, j + 2, hs, sm);
        if (blockIdx.x == 0) {
            for (int c = threadIdx.x; c < j + 2; c += kFgThreads) st->h[c] = hs[c];
            if (threadIdx.x == 0) st->j = j;
        }
    } else {
        for (int c = threadIdx.x; c <= j; c += kFgThreads) hs[c] = __ldcg(&st->h[c]);
        __syncthreads();
    }
    double *w = V + (long)(j + 1) * ld;
    const long step = (long)nb * kFgThreads, first = (long)blockIdx.x * kFgThreads + threadIdx.x;
    if (j + 2 <= kFgChunk) {
        // the vectors' values stay in registers between the update and the products
        double acc[kFgChunk];
#pragma unroll
        for (int q = 0; q < kFgChunk; q++) acc[q] = 0.0;
        for (long i = first; i < n; i += step) {
            double v[kFgChunk], s = __ldcg(w + i);
#pragma unroll
            for (int q = 0; q < kFgChunk; q++)
                if (q <= j) v[q] = __ldcg(V + (long)q * ld + i);
#pragma unroll
            for (int q = 0; q < kFgChunk; q++)
                if (q <= j) s = fma(-hs[q], v[q], s);
            w[i] = s;
#pragma unroll
            for (int q = 0; q < kFgChunk; q++) {
                if (q <= j) acc[q] = fma(v[q], s, acc[q]);
                if (q == j + 1) acc[q] = fma(s, s, acc[q]);
            }
        }
        block_store_parts(acc, j + 2, 0, part2, nb, sm);
        return;
    }
    for (long i = first; i < n; i += step) {
        double s = __ldcg(w + i);
        for (int c = 0; c <= j; c++) s = fma(-hs[c], __ldcg(V + (long)c * ld + i), s);
        w[i] = s;
    }
    for (int c0 = 0; c0 <= j + 1; c0 += kFgChunk) {
        const int m = min(kFgChunk, j + 2 - c0);
        double acc[kFgChunk];
#pragma unroll
        for (int q = 0; q < kFgChunk; q++) acc[q] = 0.0;
        for (long i = first; i < n; i += step) {
            const double wi = w[i];
#pragma unroll
            for (int q = 0; q < kFgChunk; q++)
                if (q < m) acc[q] = fma(c0 + q <= j ? __ldcg(V + (long)(c0 + q) * ld + i) : wi, wi, acc[q]);
        }
        block_store_parts(acc, m, c0, part2, nb, sm);
    }
}

template <bool SMALL>
__global__ void __launch_bounds__(kFgThreads, 2) k_fg_orth2(int n, double *V, long ld, FgState *st,
                                                            const double *part2, double *part3)
{
    __shared__ double hs[kMaxKrylov + 2];
    __shared__ double sm[kFgChunk][kFgWarps];
    pdl_wait<true>();
    const int j = __ldcg(&st->j), nb = gridDim.x;
    const double ww = __ldcg(&st->h[j + 1]);
    bool again;
    if constexpr (SMALL) {
        block_sum_parts(part2, nb, j + 2, hs, sm);
        const double nrm = hs[j + 1];
        again = nrm < 0.5 * ww;
        if (blockIdx.x == 0) {
            for (int c = threadIdx.x; c <= j; c += kFgThreads) st->h2[c] = hs[c];
            if (threadIdx.x == 0) st->nrm = nrm;
        }
    } else {
        again = __ldcg(&st->nrm) < 0.5 * ww;
        for (int c = threadIdx.x; c <= j; c += kFgThreads) hs[c] = __ldcg(&st->h2[c]);
        __syncthreads();
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) st->reorth = again;
    if (!again) return;
    double *w = V + (long)(j + 1) * ld;
    const long step = (long)nb * kFgThreads;
    double acc[kFgChunk];
    acc[0] = 0.0;
    for (long i = (long)blockIdx.x * kFgThreads + threadIdx.x; i < n; i += step) {
        double s = __ldcg(w + i);
        for (int c0 = 0; c0 <= j; c0 += kFgChunk) {
            double v[kFgChunk];
#pragma unroll
            for (int q = 0; q < kFgChunk; q++)
                if (c0 + q <= j) v[q] = __ldcg(V + (long)(c0 + q) * ld + i);
#pragma unroll
            for (int q = 0; q < kFgChunk; q++)
                if (c0 + q <= j) s = fma(-hs[c0 + q], v[q], s);
        }
        w[i] = s;
        acc[0] = fma(s, s, acc[0]);
    }
    block_store_parts(acc, 1, 0, part3, nb, sm);
}

// V_{j+1} /= |w|.  CTA 0 ends the step: Hessenberg column j, the previous
// Givens rotations applied to it, a new rotation, the updated residual
// estimate |g_{j+1}| / |b|, and the inner loop's condition.  (The other CTAs
// read st->j, which the next step's first orthogonalisation rewrites;
// st->j_next is written here.)
template <bool SMALL>
__global__ void __launch_bounds__(kFgThreads) k_fg_end(int n, double *V, long ld, FgState *st, const double *part3,
                                                       int nb, FgHandles hd)
{
    __shared__ double s_nrm[1];
    __shared__ double sm[kFgChunk][kFgWarps];
    __shared__ double col[kMaxKrylov + 1], cs[kMaxKrylov], sn[kMaxKrylov];
    pdl_wait<true>();
    const int j = __ldcg(&st->j);
    const bool again = __ldcg(&st->reorth) != 0;
    if (SMALL && again) block_sum_parts(part3, nb, 1, s_nrm, sm);
    else if (threadIdx.x == 0) s_nrm[0] = __ldcg(&st->nrm);
    if (blockIdx.x == 0)
        for (int i = threadIdx.x; i <= j; i += kFgThreads) {
            col[i] = st->h[i] + (again ? st->h2[i] : 0.0);
            if (i < j) { cs[i] = st->cs[i]; sn[i] = st->sn[i]; }
        }
    __syncthreads();
    const double nrm = s_nrm[0], d = sqrt(nrm);
    double *w = V + (long)(j + 1) * ld;
    for (long i = (long)blockIdx.x * kFgThreads + threadIdx.x; i < n; i += (long)gridDim.x * kFgThreads)
        w[i] = d > 0 ? __ldcg(w + i) / d : 0.0;
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    const int m = st->m;
    col[j + 1] = sqrt(fmax(nrm, 0.0));
    for (int i = 0; i < j; i++) {
        const double t0 = cs[i] * col[i] + sn[i] * col[i + 1];
        col[i + 1] = -sn[i] * col[i] + cs[i] * col[i + 1];
        col[i] = t0;
    }
    const double a = col[j], b = col[j + 1];
    const double rden = hypot(a, b);
    const double csj = rden > 0 ? a / rden : 1.0, snj = rden > 0 ? b / rden : 0.0;
    st->cs[j] = csj;
    st->sn[j] = snj;
    double *H = st->H + (long)j * (m + 1);
    for (int i = 0; i < j; i++) H[i] = col[i];
    H[j] = rden;
    H[j + 1] = 0.0;
    const double gj = st->g[j], gn = -snj * gj;
    st->g[j + 1] = gn;
    st->g[j] = csj * gj;
    st->total_it++;
    st->vcycles++;
    st->vcycles_total++;
    st->j_done = j + 1;
    const double est = fabs(gn) / st->bnorm;
    int go = 0;
    if (!isfinite(est)) {
        // no update from this cycle; the outer loop stops (its condition is
        // set by k_fg_solve_y, a kernel of the outer loop's own body)
        st->status = FG_NONFINITE;
        st->err_any |= 1;
        st->go_outer = 0;
        st->j_done = 0;
    } else if (!(est < st->tol) && j + 1 < m) {
        go = 1;
        st->j_next = j + 1;
    }
    st->go_inner = go;
    set_cond(hd.inner, hd.use, go);
}

// r = b - A x, per-CTA {|r|^2, |b|^2}
template <int KC, bool IDX>
__global__ void __launch_bounds__(256) k_fg_resid(FgOperator op, const double *__restrict__ b, const double *x,
                                                  double *__restrict__ r, double *__restrict__ part)
{
    __shared__ double sm[32];
    const int i0 = blockIdx.x * blockDim.x + threadIdx.x, i = min(i0, op.n - 1);
    FgRow<KC, IDX, false> R;
    R.fetch(op, i);
    const double bi = b[i];
    asm volatile("" ::: "memory");  // the operator loads above stay ahead of the gathers
    const double ri = bi - R.dot(op, x, i);
    double rr = 0, bb = 0;
    if (i0 < op.n) {
        r[i] = ri;
        rr = ri * ri;
        bb = bi * bi;
    }
    rr = bsum<256>(rr, sm);
    bb = bsum<256>(bb, sm);
    if (threadIdx.x == 0) { part[2 * blockIdx.x] = rr; part[2 * blockIdx.x + 1] = bb; }
}

// y = H^-1 g (upper triangular, j_done columns); re-asserts the outer loop's
// condition, which an Arnoldi step may have cleared.  One warp brings the
// first kSolveCols columns into shared memory, one lane then solves by rows
// (each row's sum in column order): from global memory that chain of loads
// took 11 us for 15 columns.
constexpr int kSolveCols = 48;
__global__ void __launch_bounds__(32) k_fg_solve_y(FgState *st, FgHandles hd)
{
    __shared__ double H[kSolveCols][kSolveCols + 1], y[kMaxKrylov];
    const int jd = st->j_done, m = st->m, lane = threadIdx.x;
    if (lane == 0) set_cond(hd.outer, hd.use, st->go_outer);
    for (int q = 0; q < min(jd, kSolveCols); q++)
        for (int i = lane; i <= q; i += 32) H[i][q] = st->H[(long)q * (m + 1) + i];
    for (int i = lane; i < jd; i += 32) y[i] = st->g[i];
    __syncwarp();
    if (lane != 0) return;
    for (int i = jd - 1; i >= 0; i--) {
        double s = y[i];
        if (jd <= kSolveCols) {
#pragma unroll 8
            for (int q = i + 1; q < jd; q++) s -= H[i][q] * y[q];
            y[i] = s / H[i][i];
        } else {
            for (int q = i + 1; q < jd; q++) s -= st->H[(long)q * (m + 1) + i] * y[q];
            y[i] = s / st->H[(long)i * (m + 1) + i];
        }
        st->y[i] = y[i];
    }
}

// x += sum_{c < j_done} y[c] Z_c
template <class T>
__global__ void __launch_bounds__(256) k_fg_combine(int n, const T *__restrict__ Z, long ld,
                                                    const FgState *__restrict__ st, double *__restrict__ x)
{
    __shared__ double ys[kMaxKrylov + 1];
    const int cnt = st->j_done;
    if (cnt == 0) return;
    for (int c = threadIdx.x; c < cnt; c += blockDim.x) ys[c] = st->y[c];
    __syncthreads();
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double s = x[i];
    for (int c = 0; c < cnt; c++) s = fma(ys[c], (double)Z[c * ld + i], s);
    x[i] = s;
}

__global__ void k_fg_final(FgState *st)
{
    if (st->status == FG_OK && !(st->relres < st->tol) && st->bnorm > 0) {
        st->status = FG_NOT_CONVERGED;
        st->err_any |= 2;
    }
}

__global__ void k_fg_guess(FgState *st, double *ks, int nd)
{
    const double g0 = ks[0], G00 = ks[2];
    double c0 = 0.0, c1 = 0.0;
    auto one = [](double g, double G) {
        const double q = g / G;
        return G > 0 && isfinite(q) ? q : 0.0;
    };
    if (nd == 1) {
        c0 = one(g0, G00);
    } else {
        const double g1 = ks[1], G01 = ks[4], G11 = ks[5];
        const double det = G00 * G11 - G01 * G01;
        if (!(G00 > 0)) {
            c1 = one(g1, G11);
        } else if (!(G11 > 0) || !(det > 1e-12 * G00 * G11)) {
            c0 = one(g0, G00);
        } else {
            c0 = (G11 * g0 - G01 * g1) / det;
            c1 = (G00 * g1 - G01 * g0) / det;
            if (!isfinite(c0) || !isfinite(c1)) { c0 = one(g0, G00); c1 = 0.0; }
        }
    }
    ks[6] = c0;
    ks[7] = c1;
    st->alpha = nd == 1 ? c0 : c1;
}

__global__ void k_set_scalar(double *dst, double v) { *dst = v; }

void fg_init(FgState *st, int m, int max_total, int max_restarts, double tol, cudaStream_t s)
{
    k_fg_init<<<1, 1, 0, s>>>(st, m, max_total, max_restarts, tol);
    MGM_LAUNCHED();
}
void fg_clear_totals(FgState *st, cudaStream_t s)
{
    k_fg_clear_totals<<<1, 1, 0, s>>>(st);
    MGM_LAUNCHED();
}
void fg_time_mark(FgState *st, int end, cudaStream_t s)
{
    k_fg_time_mark<<<1, 1, 0, s>>>(st, end);
    MGM_LAUNCHED();
}
void fg_begin(FgState *st, const double *part, int nbres, FgHandles hd, cudaStream_t s)
{
    k_fg_begin<<<1, 256, 0, s>>>(st, part, nbres, hd);
    MGM_LAUNCHED();
}
void fg_scale0(int n, double *V, const FgState *st, cudaStream_t s)
{
    k_fg_scale0<<<blocks_for(n, 256), 256, 0, s>>>(n, V, st);
    MGM_LAUNCHED();
}
template <class T>
void fg_load(int n, const double *V, long ld, const FgState *st, T *out, cudaStream_t s)
{
    k_fg_load<T><<<blocks_for(n, 256), 256, 0, s>>>(n, V, ld, st, out);
    MGM_LAUNCHED();
}
template void fg_load<double>(int, const double *, long, const FgState *, double *, cudaStream_t);
template void fg_load<float>(int, const double *, long, const FgState *, float *, cudaStream_t);
template <class T>
void fg_arnoldi(const FgOperator &op, const T *z, T *Z, double *V, long ld, FgState *st, double *part, FgHandles hd,
                cudaStream_t s, Chain &launch)
{
    const int n = op.n, nb = dot_blocks(n), rows = blocks_for(n, kFgThreads), b = kFgThreads;
    double *part2 = part + fg_part_stride(nb), *part3 = part2 + fg_part_stride(nb);
    if (n < kFgSmall) {
        if (!op.idx16) launch(k_fg_apply<T, 0, true, true>, rows, b, 0, s, op, z, Z, V, ld, st, part);
        else if (op.kp <= 16) launch(k_fg_apply<T, 8, false, true>, rows, b, 0, s, op, z, Z, V, ld, st, part);
        else if (op.kp <= 24) launch(k_fg_apply<T, 24, false, true>, rows, b, 0, s, op, z, Z, V, ld, st, part);
        else launch(k_fg_apply<T, 32, false, true>, rows, b, 0, s, op, z, Z, V, ld, st, part);
        launch(k_fg_orth1<true>, nb, b, 0, s, n, V, ld, st, part, part2);
        launch(k_fg_orth2<true>, nb, b, 0, s, n, V, ld, st, part2, part3);
        launch(k_fg_end<true>, rows, b, 0, s, n, V, ld, st, part3, nb, hd);
        return;
    }
    if (op.idx16) launch(k_fg_apply<T, 0, false, false>, rows, b, 0, s, op, z, Z, V, ld, st, part);
    else launch(k_fg_apply<T, 0, true, false>, rows, b, 0, s, op, z, Z, V, ld, st, part);
    launch(k_fg_dots, nb, b, 0, s, n, V, ld, st, part);
    launch(k_fg_reduce<FG_RED_FIRST>, kMaxKrylov + 2, b, 0, s, part, nb, st);
    launch(k_fg_orth1<false>, nb, b, 0, s, n, V, ld, st, part, part2);
    launch(k_fg_reduce<FG_RED_SECOND>, kMaxKrylov + 2, b, 0, s, part2, nb, st);
    launch(k_fg_orth2<false>, nb, b, 0, s, n, V, ld, st, part2, part3);
    launch(k_fg_reduce<FG_RED_LAST>, 1, b, 0, s, part3, nb, st);
    launch(k_fg_end<false>, 148 * 8, b, 0, s, n, V, ld, st, part3, nb, hd);
}
template void fg_arnoldi<double>(const FgOperator &, const double *, double *, double *, long, FgState *, double *,
                                 FgHandles, cudaStream_t, Chain &);
template void fg_arnoldi<float>(const FgOperator &, const float *, float *, double *, long, FgState *, double *,
                                FgHandles, cudaStream_t, Chain &);

void fg_resid(const FgOperator &op, const double *b, const double *x, double *r, double *part, cudaStream_t s)
{
    const int nb = blocks_for(op.n, 256);
    if (!op.idx16) launch_k(k_fg_resid<0, true>, nb, 256, 0, s, op, b, x, r, part);
    else if (op.n >= kFgSmall) launch_k(k_fg_resid<0, false>, nb, 256, 0, s, op, b, x, r, part);
    else if (op.kp <= 16) launch_k(k_fg_resid<8, false>, nb, 256, 0, s, op, b, x, r, part);
    else if (op.kp <= 24) launch_k(k_fg_resid<24, false>, nb, 256, 0, s, op, b, x, r, part);
    else launch_k(k_fg_resid<32, false>, nb, 256, 0, s, op, b, x, r, part);
}
void fg_solve_y(FgState *st, FgHandles hd, cudaStream_t s)
{
    k_fg_solve_y<<<1, 32, 0, s>>>(st, hd);
    MGM_LAUNCHED();
}
template <class T>
void fg_combine(int n, const T *Z, long ld, const FgState *st, double *x, cudaStream_t s)
{
    k_fg_combine<T><<<blocks_for(n, 256), 256, 0, s>>>(n, Z, ld, st, x);
    MGM_LAUNCHED();
}
template void fg_combine<double>(int, const double *, long, const FgState *, double *, cudaStream_t);
template void fg_combine<float>(int, const float *, long, const FgState *, double *, cudaStream_t);
void fg_final(FgState *st, cudaStream_t s)
{
    k_fg_final<<<1, 1, 0, s>>>(st);
    MGM_LAUNCHED();
}
void fg_guess_coefficients(FgState *st, double *ks, int nd, cudaStream_t s)
{
    k_fg_guess<<<1, 1, 0, s>>>(st, ks, nd);
    MGM_LAUNCHED();
}
void set_scalar(double *dst, double v, cudaStream_t s)
{
    k_set_scalar<<<1, 1, 0, s>>>(dst, v);
    MGM_LAUNCHED();
}

// ---------------------------------------------------------------------------
// dense Gauss-Jordan with partial pivoting, one matrix, set-up only
// ---------------------------------------------------------------------------
// In place and in one cooperative launch.  CTA b owns rows b, b + grid, ... (in
// shared memory where they fit) and never moves one: a row carries its logical
// position, and column slot c holds the inverse's column for the row that was
// pivot c.  At step c every CTA offers its largest |entry| of column c among the
// rows not yet used (ties: lowest position) with that row's values; after one
// grid barrier all take the same winner, scale its row and update their own
// rows.  The operations on an entry, and their order, are those of elimination
// on [M | I] with row swaps, whose other entries are zeros and ones.  A step is
// the barrier and two dependent L2 reads: 6.9 us at 896 rows (7.4 with the
// candidates read by one warp), against 15 us as four launches over the matrix
// of twice the width (1024 threads 8.2; 74 CTAs 9.2).
constexpr int kInvThreads = 512;

struct alignas(16) InvCand {  // read and written as one int4
    double v;
    int pos, row;
};

__global__ void __launch_bounds__(kInvThreads, 1) k_dense_inverse(int n, int k, const int *__restrict__ idx,
                                                                  const double *__restrict__ A, double *gM,
                                                                  double *cand_row, InvCand *cand, int *state,
                                                                  double *__restrict__ inv64,
                                                                  float *__restrict__ inv32)
{
    extern __shared__ __align__(16) unsigned char inv_smem[];
    __shared__ InvCand win;
    __shared__ InvCand wcand[kInvThreads / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, G = gridDim.x, b = blockIdx.x;
    const int mine = (n - b + G - 1) / G;  // own rows b + q G
    const int maxr = (n + G - 1) / G;
    double *const sc = reinterpret_cast<double *>(inv_smem);  // the scaled pivot row
    double *const fs = sc + n;                                // own rows' entries of the step's column
    int *const piv = reinterpret_cast<int *>(fs + maxr);      // pivot row of each step
    int *const pos = piv + n + (n & 1);                       // own rows' logical positions
    double *const rows = gM ? gM + (long)b * maxr * n : reinterpret_cast<double *>(pos + ((maxr + 1) & ~1));
    unsigned *const bar = reinterpret_cast<unsigned *>(state);
    int *const err = state + 2;
    unsigned gen = 0;
    if (tid == 0) gen = *(volatile unsigned *)&bar[1];
    for (int q = 0; q < mine; q++)
        for (int c = tid; c < n; c += kInvThreads) rows[(long)q * n + c] = 0.0;
    __syncthreads();
    for (int q = tid; q < mine; q += kInvThreads) {  // duplicates in a row accumulate, in slot order
        pos[q] = b + q * G;
        for (int j = 0; j < k; j++) {
            const long o = (long)j * n + b + q * G;
            rows[(long)q * n + idx[o]] += A[o];
        }
    }
    __syncthreads();
    auto better = [](const InvCand &x, const InvCand &y) {  // x before y
        return x.v > y.v || (x.v == y.v && x.pos < y.pos);
    };
    auto warp_best = [&](InvCand x) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            InvCand y;
            y.v = __shfl_xor_sync(0xffffffffu, x.v, o);
            y.pos = __shfl_xor_sync(0xffffffffu, x.pos, o);
            y.row = __shfl_xor_sync(0xffffffffu, x.row, o);
            if (better(y, x)) x = y;
        }
        return x;
    };
    // offers this CTA's candidate for column c
    auto offer = [&](int c) {
        InvCand best{-2.0, n, -1};
        for (int q = tid; q < mine; q += kInvThreads)
            if (pos[q] >= c) {
                const double v = fabs(rows[(long)q * n + c]);
                const InvCand x{v >= 0.0 ? v : -1.0, pos[q], b + q * G};  // a NaN after every number
                if (better(x, best)) best = x;
            }
        if (mine > 32) {  // else warp 0 has them all
            best = warp_best(best);
            if (lane == 0) wcand[warp] = best;
            __syncthreads();
            if (warp == 0) best = lane < kInvThreads / 32 ? wcand[lane] : InvCand{-2.0, n, -1};
        }
        if (warp == 0) {
            best = warp_best(best);
            if (lane == 0) {
                win = best;
                __stcg(reinterpret_cast<int4 *>(cand + (c & 1) * G + b), *reinterpret_cast<const int4 *>(&best));
            }
        }
        __syncthreads();
        if (win.row >= 0) {
            const double *r = rows + (long)((win.row - b) / G) * n;
            double *o = cand_row + (long)((c & 1) * G + b) * n;
            for (int t = tid; t < n; t += kInvThreads) __stcg(o + t, r[t]);
        }
    };
    offer(0);
    for (int c = 0; c < n; c++) {
        if (!grid_barrier(bar, err, gen)) return;
        // the winner: a candidate per thread, then every warp over the warps' best
        InvCand best{-2.0, n, -1};
        if (tid < G) {
            const int4 raw = __ldcg(reinterpret_cast<const int4 *>(cand + (c & 1) * G + tid));
            best = *reinterpret_cast<const InvCand *>(&raw);
        }
        if (warp < (G + 31) / 32) {
            best = warp_best(best);
            if (lane == 0) wcand[warp] = best;
        }
        __syncthreads();
        best = warp_best(lane < (G + 31) / 32 ? wcand[lane] : InvCand{-2.0, n, -1});
        if (tid == 0) piv[c] = best.row;
        const int P = best.row, pp = best.pos, owner = P % G;
        const double *src = cand_row + (long)((c & 1) * G + owner) * n;
        const double p = __ldcg(src + c);
        for (int t = tid; t < n; t += kInvThreads) sc[t] = (t == c ? 1.0 : __ldcg(src + t)) / p;
        // the row at position c and the pivot row change places
        for (int q = tid; q < mine; q += kInvThreads) {
            if (b + q * G == P) pos[q] = c;
            else if (pos[q] == c) pos[q] = pp;
            fs[q] = rows[(long)q * n + c];
        }
        __syncthreads();
        for (int q = 0; q < mine; q++) {
            double *r = rows + (long)q * n;
            const double f = fs[q];
            const bool pivot = b + q * G == P;
            for (int t = tid; t < n; t += kInvThreads) {
                if (pivot) r[t] = sc[t];
                else if (f != 0.0) r[t] = fma(-f, sc[t], t == c ? 0.0 : r[t]);
            }
        }
        __syncthreads();
        if (c + 1 < n) offer(c + 1);
    }
    for (int q = 0; q < mine; q++)
        for (int t = tid; t < n; t += kInvThreads) {
            const double v = rows[(long)q * n + t];
            const long o = (long)pos[q] * n + piv[t];
            inv64[o] = v;
            inv32[o] = (float)v;
        }
}

void dense_inverse(int n, int k, const int *idx, const double *A, double *inv64, float *inv32, cudaStream_t s,
                   int most_ctas)
{
    constexpr size_t kMostSmem = 220 * 1024;
    MGM_CUDA(cudaFuncSetAttribute(k_dense_inverse, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMostSmem));
    // a candidate per thread: no more CTAs than threads
    const int grid = std::min({n, most_ctas, kInvThreads, cooperative_ctas(k_dense_inverse, kInvThreads, kMostSmem)});
    const int maxr = (n + grid - 1) / grid;
    // scaled pivot row, column entries, pivots, positions, and the rows where they fit
    const size_t head = sizeof(double) * (n + maxr) + sizeof(int) * ((size_t)n + (n & 1) + ((maxr + 1) & ~1));
    const size_t own = sizeof(double) * (size_t)maxr * n;
    const bool fits = head + own <= 200 * 1024;
    DBuf<double> M, cand_row((size_t)2 * grid * n);
    if (!fits) M.alloc((size_t)grid * maxr * n);
    DBuf<InvCand> cand((size_t)2 * grid);
    DBuf<int> state(4);
    state.zero(s);
    const size_t smem = head + (fits ? own : 0);
    MGM_CUDA(launch_cooperative(k_dense_inverse, grid, kInvThreads, smem, s, n, k, idx, A, fits ? nullptr : M.p,
                                cand_row.p, cand.p, state.p, inv64, inv32));
    MGM_LAUNCHED();
    int h[4];
    state.download(h, 4, s);
    MGM_CUDA(cudaStreamSynchronize(s));
    check_barrier(h[2], "dense inverse");
}

}  // namespace mgm
