// rows.cuh -- a thread's row of an ELL operator for the latency-bound kernel
// chains of the solver (V-cycle, Arnoldi step).
#pragma once
#include "mgm_internal.cuh"

namespace mgm {

// ---------------------------------------------------------------------------
// Programmatic dependent launch in the V-cycle's and the Arnoldi step's kernels.  A level's
// operators, lists and diagonals do not change between set-ups, so a kernel
// fetches its rows' share of them into registers before it waits for its
// predecessor (ldk: a volatile load, which the compiler does not move past
// the wait), and only the vectors (r, e, d, q) after.  A chain of 30-slot steps
// over 16k rows runs at 1.4 us per launch that way, against 2.9 us with the
// loads after the wait.  EARLY: the kernels of levels below kVecMinRows rows, which
// gather vectors from L2 (__ldcg); the large levels gather through L1.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float ldk(const float *p)
{
    float v;
    asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ double ldk(const double *p)
{
    double v;
    asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ int ldk(const int *p)
{
    int v;
    asm volatile("ld.global.nc.s32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ int ldk(const short *p)
{
    short v;
    asm volatile("ld.global.nc.s16 %0, [%1];" : "=h"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ int ldk(const uint8_t *p)
{
    unsigned short v;
    asm volatile("ld.global.nc.u8 %0, [%1];" : "=h"(v) : "l"(p));
    return v;
}

// EARLY: the successor is allowed before the wait, after the operator loads
// (1.4 us per step of the chain above, against 2.0 us after the wait and
// 2.9 us before the loads).  Several small kernels may then be resident at
// once, which is why they gather from L2.
template <bool EARLY>
__device__ __forceinline__ void pdl_wait()
{
    if constexpr (EARLY) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if constexpr (!EARLY) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <bool EARLY, class T>
__device__ __forceinline__ T gather(const T *p)
{
    if constexpr (EARLY) return __ldcg(p);
    else return __ldg(p);
}

// A thread's row of an ELL operator, KC slots at a time: weights and gather
// indices (int16 offsets from `base`, or 32-bit indices) by fetch, then the
// gathers together and the products summed in slot order, one fused
// multiply-add per slot as in ell_row_dot and ell_row_dot_o.  The small
// levels' operators are padded to a multiple of 8 slots (weight 0, offset 0,
// which change no bit of a sum), so a full chunk needs no test per slot: with
// one, the compiler spent 250 registers and ~10 us on a 30-slot row.
template <class T, int KC, bool IDX>
struct RowChunk {
    T a[KC];
    int c[KC];
    __device__ __forceinline__ void fetch(const void *__restrict__ gi, const T *__restrict__ A, long ld, long i,
                                          int base, int j0)
    {
        const T *pa = A + (long)j0 * ld + i;
        const int *pi = static_cast<const int *>(gi) + (long)j0 * ld + i;
        const short *po = static_cast<const short *>(gi) + (long)j0 * ld + i;
#pragma unroll
        for (int q = 0; q < KC; q++) {
            if constexpr (IDX) c[q] = ldk(pi + q * ld);
            else c[q] = base + ldk(po + q * ld);
            a[q] = ldk(pa + q * ld);
        }
    }
    // the same of a row of k slots; past its end the last slot again (not summed)
    __device__ __forceinline__ void fetch_to(const void *__restrict__ gi, const T *__restrict__ A, long ld, long i,
                                             int base, int j0, int k)
    {
        const T *pa = A + (long)j0 * ld + i;
        const int *pi = static_cast<const int *>(gi) + (long)j0 * ld + i;
        const short *po = static_cast<const short *>(gi) + (long)j0 * ld + i;
#pragma unroll
        for (int q = 0; q < KC; q++) {
            if constexpr (IDX) c[q] = ldk(pi);
            else c[q] = base + ldk(po);
            a[q] = ldk(pa);
            const long st = j0 + q + 1 < k ? ld : 0;
            pa += st;
            if constexpr (IDX) pi += st;
            else po += st;
        }
    }
    template <bool EARLY, class X>
    __device__ __forceinline__ T dot(const X *x, T s) const
    {
        X v[KC];
#pragma unroll
        for (int q = 0; q < KC; q++) v[q] = gather<EARLY>(x + c[q]);
#pragma unroll
        for (int q = 0; q < KC; q++) s = fma_rn(a[q], (T)v[q], s);
        return s;
    }
};

// the slots of a padded row (kp, a multiple of 8) beyond the chunk fetched first
template <bool EARLY, class T, int KC, bool IDX, class X>
__device__ __forceinline__ T row_rest(const void *gi, const T *A, const X *x, long ld, int kp, long i, int base, T s)
{
    for (int j0 = KC; j0 < kp; j0 += 8) {
        RowChunk<T, 8, IDX> R;
        R.fetch(gi, A, ld, i, base, j0);
        s = R.template dot<EARLY>(x, s);
    }
    return s;
}

// a whole row of k slots, 8 at a time, none beyond k read (the large levels, and
// level 0 with 32-bit indices at any size, where EARLY says how to gather),
// the next 8 slots' operator in flight during the current gathers; R: the first
// chunk, by fetch_to (prolongation to 1M rows of 30 slots: 63 us with each
// chunk's loads after the last one's gathers and the last k mod 8 slots one by
// one, now 45)
template <class T, bool IDX, bool EARLY, class X>
__device__ __forceinline__ T row_big(RowChunk<T, 8, IDX> &R, const void *gi, const T *A, const X *x, long ld, int k,
                                     long i, int base)
{
    T s = T(0);
    for (int j = 0; j < k; j += 8) {
        RowChunk<T, 8, IDX> N;
        X v[8];
        if (j + 8 < k) N.fetch_to(gi, A, ld, i, base, j + 8, k);
        else N = R;
#pragma unroll
        for (int q = 0; q < 8; q++) v[q] = gather<EARLY>(x + R.c[q]);
#pragma unroll
        for (int q = 0; q < 8; q++)
            if (j + q < k) s = fma_rn(R.a[q], (T)v[q], s);
        R = N;
    }
    return s;
}

}  // namespace mgm
