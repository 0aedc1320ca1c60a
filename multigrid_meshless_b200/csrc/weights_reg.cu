// weights_reg.cu -- the per-node saddle-point weight solves with the system in
// registers (orders up to kRegMaxOrder; the shared-memory kernels of setup.cu
// take the larger ones and give the same bits).
//
// A CTA solves one system at a time, two lanes of a warp per column of [A | I]:
// lane c holds the column's even rows in registers, lane c + 16 the odd rows
// (NT rows in all, the order rounded up to a multiple of 4, padding rows
// zero).  Step i subtracts pc t_j from row j, pc the column's entry in the
// pivot row (one shuffle brings it to the other lane) and t_j = A_ji / A_ii
// with t_i = 0, so both lanes run the same instructions.  After every second
// step the registers rotate by one (row l's result goes to register l - 1), so
// the two pivot rows of a pair of steps are always register 0 and the loop
// over the steps is not unrolled.  t is a reciprocal of the pivot and five
// operations per row, longer than the update itself: above order 32 (reg_ahead)
// a warp of its own takes column i + 1 as it was before step i, applies step i
// to it and divides while the other warps are still in step i; below, the warp
// that holds the column divides after its own update.  Either way all read t
// after the step's one barrier.
//
// Work left out without changing a bit: the identity columns beyond the
// stencil (never read), an identity column before its own row becomes the
// pivot row (its entry in the pivot row is zero), the duplicate halves of the
// symmetric RBF block, the scaling of the left half.
//
// Bound: latency at 24 warps per SM, then the shared-memory words of t (12
// broadcast 16-byte loads per 48 FP64 instructions of a warp).  Measured on 20k
// systems, 30 nodes with 15 monomials: 76.9 ns per system against 212 in shared
// memory (20 nodes with 10: 33.4 against 92.9; 47 with 15: 173 against 682),
// 86.1 with the division after the update.  Before the operators' rows were one
// pass, with the division after the update: 94, a whole column per thread (12
// warps per SM) 101, two warps per 32 columns with t computed by every warp 113.
#include <algorithm>

#include "mgm_internal.cuh"
#include "weights.cuh"

namespace mgm {

constexpr int kRegMaxOrder = 64;
constexpr int kRegPow = 8;  // coordinate powers kept per node (degrees above take the shared-memory kernels)

struct RegArgs {
    int n, m, dim, phs;
    int degree;                  // largest exponent of the monomials
    MonoDev mono;
    const double *x, *y, *z;     // source nodes
    const int *cloud;            // [..][m]
    // derivative rows
    const double *nx, *ny, *nz;
    const uint8_t *btag;         // tags of the rows
    double *Dx, *Dy, *Dz, *lap, *lapP;
    // transfer rows
    const double *tx, *ty, *tz;
    const int *src_pt;
    int rows_from, only_interior;
    double *W;
};

// a / b, correctly rounded, from y = 1 / b correctly rounded: two corrections by
// the exact remainder (Markstein 1990: the first makes the quotient faithful,
// the second correct).  The theorem wants no underflow or overflow on the way
// and a divisor whose significand is not all ones; other operands take the
// division itself.
__device__ __forceinline__ bool rcp_usable(double b)
{
    const unsigned hi = (unsigned)__double2hiint(b), lo = (unsigned)__double2loint(b);
    const unsigned e = (hi >> 20) & 0x7ff;
    return e - 523u < 1000u && !((hi & 0xfffffu) == 0xfffffu && lo == 0xffffffffu);
}
__device__ __forceinline__ double div_by(double a, double b, double y, bool usable)
{
    const unsigned ea = ((unsigned)__double2hiint(a) >> 20) & 0x7ff;
    if (a == 0.0 && usable) return a * y;
    if (!usable || ea - 523u >= 1000u) return MGM_DIV(a, b);
    double q = __dmul_rn(a, y);
    q = __fma_rn(__fma_rn(-b, q, a), y, q);
    return __fma_rn(__fma_rn(-b, q, a), y, q);
}

// Orders above 32 give the division its own warp, which works a step ahead: 8
// CTAs per SM hide the division's chain at order 30 (33.4 ns per system, 37.0
// with the warp), 4 or fewer do not (order 35 60.4 -> 52.9, 45 86.1 -> 76.9, 53
// 179 -> 150, 62 219 -> 173).
constexpr bool reg_ahead(int NT) { return NT > 32; }
// a warp per 16 columns, and the warp that divides
constexpr int reg_threads(int NT, int cols) { return (cols + 15) / 16 * 32 + (reg_ahead(NT) ? 32 : 0); }

// bytes of shared memory: L[4][NT] | col[2][NT] | t[2][NT] | diag, rdiag[NT] | A[N][N] | sx,sy,sz[m] |
// res[4][m] | pw[3][kRegPow][m], then perm[NT], pos[NT], use[NT] ints (NT a multiple of 4)
inline size_t reg_smem_bytes(int N, int m, int NT)
{
    return sizeof(double) * (4 * NT + 2 * NT + 2 * NT + 2 * NT + (size_t)N * N + (3 + 4 + 3 * kRegPow) * m) +
           sizeof(int) * 3 * NT;
}

// CTAs per SM the register budget is set for
constexpr int reg_min_blocks(int NT) { return NT <= 32 ? 8 : (NT <= 48 ? 3 : 2); }

template <int NT, bool TRANSFER>
__global__ void __launch_bounds__(reg_threads(NT, 2 * NT), reg_min_blocks(NT)) k_weights_reg(const __grid_constant__ RegArgs g)
{
    constexpr int RH = NT / 2;
    extern __shared__ __align__(16) double sm[];
    const int m = g.m, np = g.mono.np, N = m + np;
    double *L = sm;                     // [4][NT]
    double *cb = L + 4 * NT;            // [2][2][RH]
    double *tb = cb + 2 * NT;           // [2][2][RH]
    double *diag = tb + 2 * NT, *rdiag = diag + NT;
    double *A = rdiag + NT;             // [N][N]
    double *sx = A + (size_t)N * N, *sy = sx + m, *sz = sy + m;
    double *res = sz + m;               // [4][m]
    double *pw = res + 4 * m;           // [3][kRegPow][m]
    int *perm = (int *)(pw + 3 * kRegPow * m), *pos = perm + NT, *use = pos + NT;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int h = lane >> 4, ci = warp * 16 + (lane & 15);  // the lane's half of the rows, its column
    const int nops = TRANSFER ? 1 : (g.dim == 3 ? 4 : 3);
    const Team tm = Team::block();
    // the next system's nodes, fetched while the current one is solved
    double nx_ = 0, ny_ = 0, nz_ = 0;
    auto fetch_nodes = [&](long nd) {
        if (nd >= g.n || tid >= m) return;
        const long sd = TRANSFER ? g.src_pt[nd] : nd;
        const int c = g.cloud[sd * m + tid];
        nx_ = g.x[c]; ny_ = g.y[c]; nz_ = g.z[c];
    };
    fetch_nodes(blockIdx.x);
    for (long node = blockIdx.x; node < g.n; node += gridDim.x) {
        if (TRANSFER) {
            const bool skip = g.only_interior ? (g.btag[node] != 0) : (node < g.rows_from);
            if (skip) {
                for (int j = tid; j < m; j += blockDim.x) g.W[node * m + j] = 0.0;
                fetch_nodes(node + gridDim.x);
                continue;
            }
        }
        const long seed = TRANSFER ? g.src_pt[node] : node;
        __syncthreads();  // the previous system's shared data has been read
        if (tid < m) { sx[tid] = nx_; sy[tid] = ny_; sz[tid] = nz_; }
        const bool tagged = g.btag[node] != 0;
        __syncthreads();
        fetch_nodes(node + gridDim.x);
        // RBF block: pairs (i, i + d mod m), d = 1 .. m / 2, both halves from one evaluation
        const int half = (m - 1) / 2, pairs = m * half + (m % 2 == 0 ? m / 2 : 0);
        for (int e = tid; e < pairs; e += blockDim.x) {
            const int d = e / m + 1, i = e - (d - 1) * m;
            const int j = i + d < m ? i + d : i + d - m;
            const int lo = min(i, j), hi = max(i, j);  // the reference evaluates (cloud[lo], cloud[hi])
            const double p1[3] = {sx[lo], sy[lo], sz[lo]}, p2[3] = {sx[hi], sy[hi], sz[hi]};
            const double v = mgm_phs_rbf(p1, p2, g.phs, g.dim);
            A[lo * N + hi] = v;
            A[hi * N + lo] = v;
        }
        // coordinate powers (x_j - x_0)^e, e = 1 .. degree, one evaluation each
        const int deg = g.degree;
        for (int e = tid; e < 3 * deg * m; e += blockDim.x) {
            const int nd = e % m, r = e / m, ax = r / deg, ex = r - ax * deg + 1;
            const double *c = ax == 0 ? sx : (ax == 1 ? sy : sz);
            if (ax < g.dim) pw[(ax * kRegPow + ex - 1) * m + nd] = mgm_pow_int(MGM_SUB(c[nd], c[0]), ex);
        }
        __syncthreads();
        for (int e = tid; e < m * np; e += blockDim.x) {
            const int t = e / m, nd = e - t * m;
            const int ex = g.mono.px[t], ey = g.mono.py[t], ez = g.mono.pz[t];
            double v = 1;
            if (ex != 0) v = MGM_MUL(v, pw[(ex - 1) * m + nd]);
            if (ey != 0) v = MGM_MUL(v, pw[(kRegPow + ey - 1) * m + nd]);
            if (ez != 0) v = MGM_MUL(v, pw[(2 * kRegPow + ez - 1) * m + nd]);
            A[nd * N + m + t] = v;
            A[(m + t) * N + nd] = v;
        }
        for (int e = tid; e < np * np; e += blockDim.x) A[(m + e / np) * N + m + e % np] = 0.0;
        for (int e = tid; e < m; e += blockDim.x) A[e * N + e] = 0.0;
        if (TRANSFER) {
            const double p1[3] = {g.tx[node], g.ty[node], g.tz[node]};
            const double s0[3] = {g.x[seed], g.y[seed], g.z[seed]};
            transfer_row(tm, m, np, g.dim, g.phs, g.mono, sx, sy, sz, p1, s0, L);
        } else {
            // all operators' rows in one pass, a thread per entry
            for (int e = tid; e < nops * N; e += blockDim.x) {
                const int o = e / N, c = e - o * N;
                L[o * NT + c] = operator_row0_entry(o == nops - 1 ? 3 : o, c, m, g.dim, g.phs, g.mono, sx, sy, sz);
            }
        }
        __syncthreads();
        // the bubble pass on column 0 from the last row up: the carried row
        // rises while the row above it is smaller
        if (tid == 0) {
            int carried = N - 1;
            double cv = A[(N - 1) * N];
#pragma unroll 8
            for (int i = N - 1; i > 0; i--) {
                const double up = A[(i - 1) * N];
                const bool rise = up < cv;
                perm[i] = rise ? i - 1 : carried;
                if (!rise) { carried = i - 1; cv = up; }
            }
            perm[0] = carried;
        }
        __syncthreads();
        for (int p = tid; p < N; p += blockDim.x) pos[perm[p]] = p;
        __syncthreads();
        double a[RH];
        const bool left = ci < N;
        const int q = ci - N;  // identity column of row q
        const int mypos = left ? -1 : (q < m ? pos[q] : 2 * NT);
        // the warp's first step, even: 0 with a left column, else when the
        // first of its identity columns' rows is the pivot
        int start = left ? 0 : mypos & ~1;
        for (int o = 16; o > 0; o >>= 1) start = min(start, __shfl_xor_sync(0xffffffffu, start, o));
        if (left) {
#pragma unroll
            for (int l = 0; l < RH; l++) {
                const int p = 2 * l + h;
                a[l] = p < N ? A[perm[p] * N + ci] : 0.0;
            }
        } else {
            // rows in the order they have at step `start`
            int at = (mypos - start) >> 1;
            if (at < 0) at += RH;
#pragma unroll
            for (int l = 0; l < RH; l++) a[l] = (mypos & 1) == h && l == at ? 1.0 : 0.0;
        }
        // column c as it stands, for the dividing warp
        auto post = [&](int c) {
            if (warp != (c >> 4) || (lane & 15) != (c & 15)) return;
            double *o = cb + (c & 1) * NT + h * RH;
#pragma unroll
            for (int l = 0; l < RH; l += 2) *reinterpret_cast<double2 *>(o + l) = make_double2(a[l], a[l + 1]);
        };
        // the entry in the pivot row, from the lane of its half
        auto pivot_entry = [&](int half) {
            return __shfl_sync(0xffffffffu, a[0], (lane & 15) + 16 * half);
        };
        constexpr bool AHEAD = reg_ahead(NT);
        const bool divider = AHEAD && warp == (int)(blockDim.x >> 5) - 1;
        constexpr int U = (NT + 31) / 32;
        // t of step i + 1, by the dividing warp: column i + 1 through step i,
        // divided by its pivot (update false: column 0, for step 0).  Positions
        // e = half * RH + register, as they are before step i; after an odd step
        // the registers have turned by one.
        auto divide = [&](int i, bool update) {
            const double *col = cb + ((i + 1) & 1) * NT, *t = tb + (i & 1) * NT;
            const int odd = i & 1;                                // step i's half (position odd * RH)
            const int at = !update ? 0 : odd ? 1 : RH;            // the row of step i + 1
            double u[U];
            const double pc = update ? col[odd * RH] : 0.0;
#pragma unroll
            for (int q = 0; q < U; q++) {
                const int e = lane + 32 * q;
                u[q] = e < NT ? col[e] : 0.0;
                if (update && e < NT) u[q] = MGM_SUB(u[q], MGM_MUL(pc, t[e]));
            }
            double piv = u[0];
#pragma unroll
            for (int q = 1; q < U; q++)
                if (at >= 32 * q) piv = u[q];
            piv = __shfl_sync(0xffffffffu, piv, at & 31);
            const bool ok = rcp_usable(piv);
            const double y = ok ? __drcp_rn(piv) : 0.0;
            double *o = tb + ((i + 1) & 1) * NT;
#pragma unroll
            for (int q = 0; q < U; q++) {
                const int e = lane + 32 * q;
                if (e >= NT) continue;
                int to = e;
                if (update && odd) to = e == 0 ? RH - 1 : e == RH ? NT - 1 : e - 1;
                o[to] = e == at ? 0.0 : div_by(u[q], piv, y, ok);
            }
        };
        // without it: t of step i + 1 from its column, by the column's own warp
        auto divide_own = [&](int i) {
            if (warp != (i >> 4)) return;
            post(i);
            __syncwarp();
            const double *col = cb + (i & 1) * NT;
            double *t = tb + (i & 1) * NT;
            const int at = (i & 1) * RH;  // the pivot row: register 0 of its half
            const double piv = col[at];
            const bool ok = rcp_usable(piv);
            const double y = ok ? __drcp_rn(piv) : 0.0;
#pragma unroll
            for (int j0 = 0; j0 < NT; j0 += 32) {
                const int j = j0 + lane;
                if (j < NT) t[j] = j == at ? 0.0 : div_by(col[j], piv, y, ok);
            }
        };
        if constexpr (AHEAD) {
            post(0);
            if (N > 1) post(1);
            __syncthreads();
            if (divider) divide(-1, false);
        } else {
            divide_own(0);
        }
        __syncthreads();
        if (divider) {
#pragma unroll 1
            for (int i = 0; i < N; i++) {
                if (i + 1 < N) divide(i, true);
                __syncthreads();
            }
        } else {
            int i = 0;
#pragma unroll 1
            for (; i < N; i += 2) {
                if (i >= start) {
                    const double pc = pivot_entry(0);
                    const double *t = tb + h * RH;
#pragma unroll
                    for (int l = 0; l < RH; l += 2) {
                        if (l % 8 == 0) __syncwarp();  // keeps the loads of t from all moving up (registers)
                        const double2 tj = *reinterpret_cast<const double2 *>(t + l);
                        a[l] = MGM_SUB(a[l], MGM_MUL(pc, tj.x));
                        a[l + 1] = MGM_SUB(a[l + 1], MGM_MUL(pc, tj.y));
                    }
                }
                if constexpr (!AHEAD) {
                    if (i + 1 >= N) break;
                    divide_own(i + 1);
                } else if (i + 2 < N) post(i + 2);
                __syncthreads();
                if (i + 1 >= N) break;
                if (i >= start) {
                    const double pc = pivot_entry(1);
                    const double *t = tb + NT + h * RH;
                    double first = 0.0;
#pragma unroll
                    for (int l = 0; l < RH; l += 2) {
                        if (l % 8 == 0) __syncwarp();
                        const double2 tj = *reinterpret_cast<const double2 *>(t + l);
                        const double u = MGM_SUB(a[l], MGM_MUL(pc, tj.x));
                        if (l > 0) a[l - 1] = u;
                        else first = u;
                        a[l] = MGM_SUB(a[l + 1], MGM_MUL(pc, tj.y));
                    }
                    a[RH - 1] = first;
                }
                if constexpr (!AHEAD) {
                    if (i + 2 < N) divide_own(i + 2);
                } else if (i + 3 < N) post(i + 3);
                __syncthreads();
            }
        }
        // register l now holds row 2 (l + N / 2 mod RH) + h; the identity
        // columns go through shared memory (the matrix has been read), where
        // all threads divide them by the diagonal
        __syncthreads();
        const int turned = N >> 1;
        double *mine = A + (!left && q < m ? q : 0);
#pragma unroll
        for (int l = 0; l < RH; l++) {
            const int lr = l + turned < RH ? l + turned : l + turned - RH, p = 2 * lr + h;
            if (left) {
                if (p == ci) {
                    diag[p] = a[l];
                    use[p] = rcp_usable(a[l]);
                    rdiag[p] = use[p] ? __drcp_rn(a[l]) : 0.0;
                }
            } else if (q < m && p < N) {
                mine[(size_t)p * m] = a[l];
            }
        }
        __syncthreads();
        for (int e = tid; e < N * m; e += blockDim.x) {
            const int p = e / m;
            A[e] = div_by(A[e], diag[p], rdiag[p], use[p]);
        }
        __syncthreads();
        // row o of the result: sum_c L_o[c] inverse[c][q], c ascending
        // (mat_lib.h:214-228, 720-726), a thread per o and q
        for (int e = tid; e < nops * m; e += blockDim.x) {
            const int o = e / m, q1 = e - o * m;
            double s = 0.0;
#pragma unroll 4
            for (int c = 0; c < N; c++) s = MGM_ADD(s, MGM_MUL(L[o * NT + c], A[(size_t)c * m + q1]));
            if (TRANSFER) g.W[node * m + q1] = s;
            else res[e] = s;
        }
        if (!TRANSFER) {
            __syncthreads();
            const bool bnd = tagged;
            for (int j = tid; j < m; j += blockDim.x) {
                const long o = node * m + j;
                const bool d3 = g.dim == 3;
                const double dx = res[j], dy = res[m + j], dl = res[(nops - 1) * m + j];
                const double dz = d3 ? res[2 * m + j] : 0.0;
                g.Dx[o] = dx;
                g.Dy[o] = dy;
                if (d3) g.Dz[o] = dz;
                g.lap[o] = dl;
                double v = dl;
                if (bnd) {
                    v = MGM_ADD(MGM_MUL(dx, g.nx[node]), MGM_MUL(dy, g.ny[node]));
                    if (d3) v = MGM_ADD(v, MGM_MUL(dz, g.nz[node]));
                }
                g.lapP[o] = v;
            }
        }
    }
}
template <int NT, bool TRANSFER>
static void launch_reg(const RegArgs &g, cudaStream_t s)
{
    const int N = g.m + g.mono.np;
    const int threads = reg_threads(NT, N + g.m);
    const size_t smem = reg_smem_bytes(N, g.m, NT);
    auto kern = k_weights_reg<NT, TRANSFER>;
    // the kernel's limit holds for all threads of the process: one value for all the orders it takes
    MGM_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)reg_smem_bytes(NT, NT, NT)));
    int per_sm = 0;
    MGM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem));
    const int grid = (int)std::min<long>(g.n, 148L * std::max(1, per_sm));
    launch_k(kern, grid, threads, smem, s, g);
}

template <bool TRANSFER>
static bool weights_reg(RegArgs &g, cudaStream_t s)
{
    for (int t = 0; t < g.mono.np; t++)
        g.degree = std::max({g.degree, (int)g.mono.px[t], (int)g.mono.py[t], (int)g.mono.pz[t]});
    const int N = g.m + g.mono.np;
    if (N > kRegMaxOrder || g.degree > kRegPow) return false;
    switch ((N + 3) / 4) {
    case 0: case 1: case 2: case 3: case 4: launch_reg<16, TRANSFER>(g, s); break;
    case 5: launch_reg<20, TRANSFER>(g, s); break;
    case 6: launch_reg<24, TRANSFER>(g, s); break;
    case 7: launch_reg<28, TRANSFER>(g, s); break;
    case 8: launch_reg<32, TRANSFER>(g, s); break;
    case 9: launch_reg<36, TRANSFER>(g, s); break;
    case 10: launch_reg<40, TRANSFER>(g, s); break;
    case 11: launch_reg<44, TRANSFER>(g, s); break;
    case 12: launch_reg<48, TRANSFER>(g, s); break;
    case 13: launch_reg<52, TRANSFER>(g, s); break;
    case 14: launch_reg<56, TRANSFER>(g, s); break;
    case 15: launch_reg<60, TRANSFER>(g, s); break;
    default: launch_reg<64, TRANSFER>(g, s); break;
    }
    return true;
}

bool derivative_weights_reg(int n, int k, int dim, int phs, const Monomials &mono, const double *x, const double *y,
                            const double *z, const double *nx, const double *ny, const double *nz,
                            const uint8_t *btag, const int *cloud, double *Dx, double *Dy, double *Dz, double *lap,
                            double *lapP, cudaStream_t s)
{
    RegArgs g{};
    g.n = n; g.m = k; g.dim = dim; g.phs = phs; g.mono = to_dev(mono);
    g.x = x; g.y = y; g.z = z; g.cloud = cloud;
    g.nx = nx; g.ny = ny; g.nz = nz; g.btag = btag;
    g.Dx = Dx; g.Dy = Dy; g.Dz = Dz; g.lap = lap; g.lapP = lapP;
    return weights_reg<false>(g, s);
}

bool transfer_weights_reg(int nt, const double *tx, const double *ty, const double *tz, const uint8_t *tbtag,
                          const int *src_pt, int rows_from, int only_interior, int ks, int dim, int phs,
                          const Monomials &mono, const double *sx, const double *sy, const double *sz,
                          const int *scloud, double *W, cudaStream_t s)
{
    RegArgs g{};
    g.n = nt; g.m = ks; g.dim = dim; g.phs = phs; g.mono = to_dev(mono);
    g.x = sx; g.y = sy; g.z = sz; g.cloud = scloud;
    g.btag = tbtag; g.tx = tx; g.ty = ty; g.tz = tz; g.src_pt = src_pt;
    g.rows_from = rows_from; g.only_interior = only_interior; g.W = W;
    return weights_reg<true>(g, s);
}

}  // namespace mgm
