// timple.cu -- the time-implicit (TIMPLE) step of the reference,
// time_implicit_solver (header_files/timple_solver.h:40-410), on the GPU.
//
// Every product, quotient and sum is rounded separately (MGM_*), in the
// reference's order, so that the kernels are bit-identical to the reference's
// C loops run in the same (data-parallel) sweep order.  Operators are ELL
// [k][n]; the level-0 fields are the context's.
#include "ctx.cuh"

namespace mgm {

void poisson_solve(mgm_ctx *c, int mode, bool timple);

namespace {

struct TimpleArgs {
    int n, k;
    const int *idx;
    const double *Dx, *Dy, *Dz, *lap;
    const uint8_t *btag;
    const double *nx, *ny, *nz;
    double *u, *v, *w, *u_new, *v_new, *w_new, *u_old, *v_old, *w_old;
    double *p_old, *pprime, *dpdx, *dpdy, *dpdz, *dpdn, *source;
    double dt, rho, mu, nu, facRe, facdt;
};

// time_implicit_solver's set-up loop (:44-49): u_old = u = u_new, p' = 0
__global__ void k_t_begin(TimpleArgs a)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    a.u_old[i] = a.u_new[i]; a.u[i] = a.u_new[i];
    a.v_old[i] = a.v_new[i]; a.v[i] = a.v_new[i];
    a.w_old[i] = a.w_new[i]; a.w[i] = a.w_new[i];
    a.pprime[i] = 0;
}

// the start of each TIMPLE iteration (:51-56): u = u_new, p' = 0
__global__ void k_t_iter(TimpleArgs a)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    a.u[i] = a.u_new[i]; a.v[i] = a.v_new[i]; a.w[i] = a.w_new[i];
    a.pprime[i] = 0;
}

// A thread's row, slots j0.. in order, of NW operators over the shared gather
// index: 4 slots at a time, the next 4 slots' indices and weights in flight
// while the current gathers are.  A level has a few such rows per scheduler
// and one slot at a time is a chain of two memory latencies.
template <int NW>
struct TimpleRow {
    static constexpr int C = 4;
    int c[C];
    double w[NW][C];
    const double *W[NW];
    __device__ __forceinline__ void fetch(const TimpleArgs &a, int i, int j)
    {
#pragma unroll
        for (int q = 0; q < C; q++) {
            const long o = (long)min(j + q, a.k - 1) * a.n + i;
            c[q] = __ldg(a.idx + o);
#pragma unroll
            for (int m = 0; m < NW; m++) w[m][q] = __ldg(W[m] + o);
        }
    }
    // op(weights, values) with the values of the NX fields x at the slot's index
    template <int NX, class Op>
    __device__ __forceinline__ void run(const TimpleArgs &a, int i, int j0, const double *const (&x)[NX], Op op)
    {
        fetch(a, i, j0);
        for (int j = j0; j < a.k; j += C) {
            double v[C][NX], wc[C][NW];
#pragma unroll
            for (int q = 0; q < C; q++) {
#pragma unroll
                for (int m = 0; m < NX; m++) v[q][m] = x[m][c[q]];
#pragma unroll
                for (int m = 0; m < NW; m++) wc[q][m] = w[m][q];
            }
            if (j + C < a.k) fetch(a, i, j + C);
#pragma unroll
            for (int q = 0; q < C; q++)
                if (j + q < a.k) op(wc[q], v[q]);
        }
    }
};

// One momentum sweep of calculate_intermediate_velocity_implicit (:88-173) in
// data-parallel order: interior rows from the previous sweep's values (in*),
// boundary rows copied.  The operators are read once for all components (once
// per component and slot by slot a sweep of the 250k-row annulus took 115 us,
// now 50).
template <int DIM>
__global__ void __launch_bounds__(128) k_t_momentum(TimpleArgs a, const double *__restrict__ iu,
                                                    const double *__restrict__ iv, const double *__restrict__ iw,
                                                    double *__restrict__ ou, double *__restrict__ ov,
                                                    double *__restrict__ ow)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    if (a.btag[i]) {
        ou[i] = iu[i]; ov[i] = iv[i];
        if (DIM == 3) ow[i] = iw[i];
        return;
    }
    double *comp_out[3] = {ou, ov, ow};
    const double *comp_old[3] = {a.u_old, a.v_old, a.w_old};
    const double *grad[3] = {a.dpdx, a.dpdy, a.dpdz};
    const double lap0 = a.lap[i], dx0 = a.Dx[i], dy0 = a.Dy[i];
    const double dz0 = DIM == 3 ? a.Dz[i] : 0.0;
    const double ui = a.u[i], vi = a.v[i], wi = a.w[i];
    double t1[DIM] = {}, t2[DIM] = {}, t3[DIM] = {}, t4[DIM] = {}, own[DIM], old[DIM], gr[DIM];
    const double *xs[DIM];
    xs[0] = iu;
    xs[1] = iv;
    if constexpr (DIM == 3) xs[2] = iw;
#pragma unroll
    for (int q = 0; q < DIM; q++) { own[q] = xs[q][i]; old[q] = comp_old[q][i]; gr[q] = grad[q][i]; }
    TimpleRow<DIM + 1> R;
    R.W[0] = a.Dx;
    R.W[1] = a.Dy;
    R.W[2] = a.lap;
    if constexpr (DIM == 3) R.W[3] = a.Dz;
    R.template run<DIM>(a, i, 1, xs, [&](const double (&w)[DIM + 1], const double (&x)[DIM]) {
#pragma unroll
        for (int q = 0; q < DIM; q++) {
            t1[q] = MGM_ADD(t1[q], MGM_MUL(w[0], x[q]));
            t2[q] = MGM_ADD(t2[q], MGM_MUL(w[1], x[q]));
            t4[q] = MGM_ADD(t4[q], MGM_MUL(w[2], x[q]));
            if constexpr (DIM == 3) t3[q] = MGM_ADD(t3[q], MGM_MUL(w[3], x[q]));
        }
    });
    const double advection_x = MGM_MUL(ui, dx0), advection_y = MGM_MUL(vi, dy0);
    const double diffusion = MGM_MUL(MGM_MUL(-a.facRe, a.mu), lap0);
    const double unsteady0 = MGM_DIV(1., MGM_MUL(a.dt, a.facdt));
#pragma unroll
    for (int q = 0; q < DIM; q++) {
        double denom;
        if (q < 2) {
            denom = MGM_ADD(MGM_MUL(a.rho, MGM_ADD(MGM_ADD(advection_x, advection_y), unsteady0)), diffusion);
            if (DIM == 3) denom = MGM_ADD(denom, MGM_MUL(MGM_MUL(a.rho, wi), dz0));
        } else {
            const double advection_z = MGM_MUL(wi, dz0);
            denom = MGM_ADD(MGM_MUL(a.rho, MGM_ADD(MGM_ADD(MGM_ADD(advection_x, advection_y), advection_z), unsteady0)),
                            diffusion);
        }
        const double advection = MGM_ADD(MGM_ADD(MGM_MUL(ui, t1[q]), MGM_MUL(vi, t2[q])), MGM_MUL(wi, t3[q]));
        const double unsteady = MGM_DIV(old[q], MGM_MUL(a.dt, a.facdt));
        double num = MGM_MUL(a.rho, MGM_SUB(unsteady, advection));
        num = MGM_SUB(num, MGM_MUL(MGM_MUL(MGM_MUL(MGM_SUB(a.facRe, 1.0), a.mu), lap0), own[q]));
        num = MGM_ADD(num, MGM_MUL(a.mu, t4[q]));
        num = MGM_SUB(num, gr[q]);
        comp_out[q][i] = MGM_DIV(num, denom);
    }
}

// dpdx, dpdy(, dpdz) = the gradient of one field.  UPDATE: of p', followed by
// update_velocity_implicit (:351-363): interior velocities and pressure; pref
// gets the new p_old[0].
template <int DIM, bool UPDATE>
__global__ void __launch_bounds__(128) k_t_gradient(TimpleArgs a, const double *__restrict__ f,
                                                    double *__restrict__ pref)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    double g[DIM] = {};
    TimpleRow<DIM> R;
    R.W[0] = a.Dx;
    R.W[1] = a.Dy;
    if constexpr (DIM == 3) R.W[2] = a.Dz;
    const double *const xs[1] = {f};
    R.template run<1>(a, i, 0, xs, [&](const double (&w)[DIM], const double (&x)[1]) {
#pragma unroll
        for (int q = 0; q < DIM; q++) g[q] = MGM_ADD(g[q], MGM_MUL(w[q], x[0]));
    });
    a.dpdx[i] = g[0];
    a.dpdy[i] = g[1];
    if constexpr (DIM == 3) a.dpdz[i] = g[2];
    if constexpr (UPDATE) {
        double p = a.p_old[i];
        if (!a.btag[i]) {
            a.u_new[i] = MGM_SUB(a.u_new[i], MGM_DIV(MGM_MUL(a.dt, g[0]), a.rho));
            a.v_new[i] = MGM_SUB(a.v_new[i], MGM_DIV(MGM_MUL(a.dt, g[1]), a.rho));
            if constexpr (DIM == 3) a.w_new[i] = MGM_SUB(a.w_new[i], MGM_DIV(MGM_MUL(a.dt, g[2]), a.rho));
            p = MGM_ADD(p, MGM_MUL(1.0, f[i]));
            a.p_old[i] = p;
        }
        if (i == 0) *pref = p;
    }
}

// calculate_mass_residual_implicit (:177-201): the components' own derivatives,
// then the source from the divergence (dpdz is 0 in 2D: never written there, as
// in the reference)
template <int DIM>
__global__ void __launch_bounds__(128) k_t_mass(TimpleArgs a)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    double g[DIM] = {};
    TimpleRow<DIM> R;
    R.W[0] = a.Dx;
    R.W[1] = a.Dy;
    const double *xs[DIM];
    xs[0] = a.u_new;
    xs[1] = a.v_new;
    if constexpr (DIM == 3) { R.W[2] = a.Dz; xs[2] = a.w_new; }
    R.template run<DIM>(a, i, 0, xs, [&](const double (&w)[DIM], const double (&x)[DIM]) {
#pragma unroll
        for (int q = 0; q < DIM; q++) g[q] = MGM_ADD(g[q], MGM_MUL(w[q], x[q]));
    });
    a.dpdx[i] = g[0];
    a.dpdy[i] = g[1];
    double gz;
    if constexpr (DIM == 3) a.dpdz[i] = gz = g[2];
    else gz = a.dpdz[i];
    a.source[i] = a.btag[i] ? 0.0 : MGM_DIV(MGM_MUL(a.rho, MGM_ADD(MGM_ADD(g[0], g[1]), gz)), a.dt);
}

// p_old -= p_old[0] (:364-368), the reference value as k_t_gradient left it
__global__ void k_t_shift(int n, double *p, const double *pref)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) p[i] = MGM_SUB(p[i], *pref);
}

// update_boundary_pressure (:371-410).  The velocity terms are assigned, not
// accumulated, inside the stencil loop (:378-392), so only the last stencil
// slot contributes; the pressure of a boundary row reads interior nodes only.
template <int DIM>
__global__ void k_t_bnd_pressure(TimpleArgs a)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int n = a.n, k = a.k;
    if (i >= n || !a.btag[i]) return;
    const double ui = a.u[i], vi = a.v[i], wi = a.w[i];
    double temp1 = 0, temp2 = 0, temp3 = 0;
    {
        const long o = (long)(k - 1) * n + i;
        const int c = a.idx[o];
        const double L = a.lap[o], dx = a.Dx[o], dy = a.Dy[o];
        const double dz = DIM == 3 ? a.Dz[o] : 0.0;
        const double un = a.u_new[c], vn = a.v_new[c];
        temp1 = MGM_MUL(MGM_MUL(a.nu, L), un);
        temp1 = MGM_SUB(temp1, MGM_MUL(MGM_MUL(ui, un), dx));
        temp1 = MGM_SUB(temp1, MGM_MUL(MGM_MUL(vi, un), dy));
        if (DIM == 3) temp1 = MGM_SUB(temp1, MGM_MUL(MGM_MUL(wi, un), dz));
        temp2 = MGM_MUL(MGM_MUL(a.nu, L), vn);
        temp2 = MGM_SUB(temp2, MGM_MUL(MGM_MUL(ui, vn), dx));
        temp2 = MGM_SUB(temp2, MGM_MUL(MGM_MUL(vi, vn), dy));
        if (DIM == 3) temp2 = MGM_SUB(temp2, MGM_MUL(MGM_MUL(wi, vn), dz));
        if (DIM == 3) {
            const double wn = a.w_new[c];
            temp3 = MGM_MUL(MGM_MUL(a.nu, L), wn);
            temp3 = MGM_SUB(temp3, MGM_MUL(MGM_MUL(ui, wn), dx));
            temp3 = MGM_SUB(temp3, MGM_MUL(MGM_MUL(vi, wn), dy));
            temp3 = MGM_SUB(temp3, MGM_MUL(MGM_MUL(wi, wn), dz));
        }
    }
    const double nxi = a.nx[i], nyi = a.ny[i], nzi = a.nz[i];
    const double dpdn =
        MGM_MUL(a.rho, MGM_ADD(MGM_ADD(MGM_MUL(temp1, nxi), MGM_MUL(temp2, nyi)), MGM_MUL(temp3, nzi)));
    a.dpdn[i] = dpdn;
    double sumx = 0, sumy = 0, sumz = 0, Ap = 0.0;
    TimpleRow<DIM> R;
    R.W[0] = a.Dx;
    R.W[1] = a.Dy;
    if constexpr (DIM == 3) R.W[2] = a.Dz;
    const double *const xs[1] = {a.p_old};
    R.template run<1>(a, i, 1, xs, [&](const double (&w)[DIM], const double (&x)[1]) {
        sumx = MGM_ADD(sumx, MGM_MUL(w[0], x[0]));
        sumy = MGM_ADD(sumy, MGM_MUL(w[1], x[0]));
        if constexpr (DIM == 3) sumz = MGM_ADD(sumz, MGM_MUL(w[2], x[0]));
    });
    Ap = MGM_ADD(Ap, MGM_MUL(a.Dx[i], nxi));
    Ap = MGM_ADD(Ap, MGM_MUL(a.Dy[i], nyi));
    if (DIM == 3) Ap = MGM_ADD(Ap, MGM_MUL(a.Dz[i], nzi));
    a.p_old[i] =
        MGM_DIV(MGM_SUB(MGM_SUB(MGM_SUB(dpdn, MGM_MUL(sumx, nxi)), MGM_MUL(sumy, nyi)), MGM_MUL(sumz, nzi)), Ap);
}

// steady-state error partials (:62-67): e += (du^2 + dv^2) [+ dw^2]
template <int DIM>
__global__ void k_t_steady(TimpleArgs a, double *partial)
{
    __shared__ double sm[256];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double e = 0.0;
    if (i < a.n) {
        const double du = MGM_SUB(a.u_new[i], a.u_old[i]), dv = MGM_SUB(a.v_new[i], a.v_old[i]);
        e = MGM_ADD(MGM_MUL(du, du), MGM_MUL(dv, dv));
        if (DIM == 3) {
            const double dw = MGM_SUB(a.w_new[i], a.w_old[i]);
            e = MGM_ADD(e, MGM_MUL(dw, dw));
        }
    }
    sm[threadIdx.x] = e;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) sm[threadIdx.x] += sm[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[blockIdx.x] = sm[0];
}

// the partials through shared memory, added in order by one thread (straight
// from global memory 1000 of them took 38 us)
__global__ void __launch_bounds__(256) k_t_steady_finish(const double *partial, int nparts, int n, double *out)
{
    __shared__ double sm[2048];
    double s = 0.0;
    for (int t0 = 0; t0 < nparts; t0 += 2048) {
        const int m = min(2048, nparts - t0);
        __syncthreads();
        for (int t = threadIdx.x; t < m; t += 256) sm[t] = partial[t0 + t];
        __syncthreads();
        if (threadIdx.x == 0)
            for (int t = 0; t < m; t++) s += sm[t];
    }
    if (threadIdx.x == 0) *out = sqrt(s / n);
}

TimpleArgs timple_args(mgm_ctx *c)
{
    Level &L = c->L[0];
    TimpleArgs a{};
    a.n = L.n; a.k = L.k; a.idx = L.idx.p;
    a.Dx = L.Dx.p; a.Dy = L.Dy.p; a.Dz = L.Dz.p; a.lap = L.lap.p;
    a.btag = L.btag.p; a.nx = L.nx.p; a.ny = L.ny.p; a.nz = L.nz.p;
    a.u = c->u.p; a.v = c->v.p; a.w = c->w.p;
    a.u_new = c->u_new.p; a.v_new = c->v_new.p; a.w_new = c->w_new.p;
    a.u_old = c->u_old.p; a.v_old = c->v_old.p; a.w_old = c->w_old.p;
    a.p_old = c->p_old.p; a.pprime = L.p.p; a.dpdx = c->dpdx.p; a.dpdy = c->dpdy.p; a.dpdz = c->dpdz.p;
    a.dpdn = c->dpdn.p; a.source = L.src.p;
    a.dt = c->dt; a.rho = c->rho; a.mu = c->rho / c->Re; a.nu = c->nu; a.facRe = c->facRe; a.facdt = c->facdt;
    return a;
}

}  // namespace

// calculate_intermediate_velocity_implicit (:72-175)
static void timple_momentum(mgm_ctx *c)
{
    cudaStream_t s = c->s;
    const int n = c->L[0].n, dim = c->dim, nb = blocks_for(n, 128);
    TimpleArgs a = timple_args(c);
    if (dim == 3) k_t_gradient<3, false><<<nb, 128, 0, s>>>(a, c->p_old.p, nullptr);
    else k_t_gradient<2, false><<<nb, 128, 0, s>>>(a, c->p_old.p, nullptr);
    MGM_LAUNCHED();
    double *in[3] = {c->u_new.p, c->v_new.p, c->w_new.p}, *out[3] = {c->tu.p, c->tv.p, c->tw.p};
    for (int sw = 0; sw < c->iter_momentum; sw++) {
        if (dim == 3) k_t_momentum<3><<<nb, 128, 0, s>>>(a, in[0], in[1], in[2], out[0], out[1], out[2]);
        else k_t_momentum<2><<<nb, 128, 0, s>>>(a, in[0], in[1], in[2], out[0], out[1], out[2]);
        MGM_LAUNCHED();
        for (int q = 0; q < 3; q++) std::swap(in[q], out[q]);
    }
    if (in[0] != c->u_new.p) {
        double *dst[3] = {c->u_new.p, c->v_new.p, c->w_new.p};
        for (int q = 0; q < dim; q++)
            MGM_CUDA(cudaMemcpyAsync(dst[q], in[q], sizeof(double) * n, cudaMemcpyDeviceToDevice, s));
    }
}

// calculate_mass_residual_implicit (:177-201)
static void timple_mass(mgm_ctx *c)
{
    const int nb = blocks_for(c->L[0].n, 128);
    if (c->dim == 3) k_t_mass<3><<<nb, 128, 0, c->s>>>(timple_args(c));
    else k_t_mass<2><<<nb, 128, 0, c->s>>>(timple_args(c));
    MGM_LAUNCHED();
}

// update_velocity_implicit (:341-369)
static void timple_update(mgm_ctx *c)
{
    cudaStream_t s = c->s;
    Level &L = c->L[0];
    const int n = L.n, nb = blocks_for(n, 256), nr = blocks_for(n, 128);
    if (c->dim == 3) k_t_gradient<3, true><<<nr, 128, 0, s>>>(timple_args(c), L.p.p, c->scal.p);
    else k_t_gradient<2, true><<<nr, 128, 0, s>>>(timple_args(c), L.p.p, c->scal.p);
    MGM_LAUNCHED();
    k_t_shift<<<nb, 256, 0, s>>>(n, c->p_old.p, c->scal.p);
    MGM_LAUNCHED();
}

// update_boundary_pressure (:371-410)
static void timple_boundary_pressure(mgm_ctx *c)
{
    const int nb = blocks_for(c->L[0].n, 256);
    if (c->dim == 3) k_t_bnd_pressure<3><<<nb, 256, 0, c->s>>>(timple_args(c));
    else k_t_bnd_pressure<2><<<nb, 256, 0, c->s>>>(timple_args(c));
    MGM_LAUNCHED();
}

// time_implicit_solver (timple_solver.h:40-70)
double timple_step(mgm_ctx *c, int mode)
{
    cudaStream_t s = c->s;
    const int n = c->L[0].n, nb = blocks_for(n, 256);
    TimpleArgs a = timple_args(c);
    k_t_begin<<<nb, 256, 0, s>>>(a);
    MGM_LAUNCHED();
    for (int it = 0; it < c->iter_timple; it++) {
        if (it > 0) {  // the first iteration's state is k_t_begin's
            k_t_iter<<<nb, 256, 0, s>>>(a);
            MGM_LAUNCHED();
        }
        timple_momentum(c);
        timple_mass(c);
        poisson_solve(c, mode, true);  // the pressure-correction equation, on p' (L.p)
        c->vcycles_acc += mode == MGM_MODE_REFERENCE ? c->num_vcycles : c->last_iters;
        timple_update(c);
        timple_boundary_pressure(c);
    }
    if (c->dim == 3) k_t_steady<3><<<nb, 256, 0, s>>>(a, c->partial.p);
    else k_t_steady<2><<<nb, 256, 0, s>>>(a, c->partial.p);
    MGM_LAUNCHED();
    k_t_steady_finish<<<1, 256, 0, s>>>(c->partial.p, nb, n, c->scal.p + 1);
    MGM_LAUNCHED();
    double e = 0;
    MGM_CUDA(cudaMemcpyAsync(&e, c->scal.p + 1, sizeof(double), cudaMemcpyDeviceToHost, s));
    MGM_CUDA(cudaStreamSynchronize(s));
    return e;
}

void timple_part(mgm_ctx *c, int part, int mode)
{
    switch (part) {
    case MGM_TIMPLE_MOMENTUM: timple_momentum(c); break;
    case MGM_TIMPLE_MASS: timple_mass(c); break;
    case MGM_TIMPLE_PRESSURE: poisson_solve(c, mode, true); break;
    case MGM_TIMPLE_UPDATE: timple_update(c); break;
    case MGM_TIMPLE_BOUNDARY_PRESSURE: timple_boundary_pressure(c); break;
    default: throw Error{MGM_ERR_ARG, "mgm_timple_part: unknown part"};
    }
    MGM_CUDA(cudaStreamSynchronize(c->s));
}

}  // namespace mgm

using namespace mgm;

namespace {
template <class F>
int tguard(F &&f)
{
    const TrimScope trim;
    try {
        f();
        return MGM_OK;
    } catch (const Error &e) {
        set_error(e.code, e.msg);
        return e.code;
    } catch (const std::exception &e) {
        set_error(MGM_ERR_ARG, e.what());
        return MGM_ERR_ARG;
    }
}
}  // namespace

extern "C" {

int mgm_set_timple(mgm_ctx *c, int iter_timple, int iter_momentum, double facRe, double facdt)
{
    return tguard([&] {
        MGM_REQUIRE(c != nullptr, "null context");
        MGM_CUDA(cudaSetDevice(c->device));
        alloc_stream(c->s);
        MGM_REQUIRE(iter_timple >= 1 && iter_momentum >= 1 && facdt > 0, "mgm_set_timple: bad parameters");
        c->iter_timple = iter_timple;
        c->iter_momentum = iter_momentum;
        c->facRe = facRe;
        c->facdt = facdt;
    });
}

int mgm_timple_part(mgm_ctx *c, int part, int mode)
{
    return tguard([&] {
        MGM_REQUIRE(c != nullptr, "null context");
        MGM_CUDA(cudaSetDevice(c->device));
        alloc_stream(c->s);
        MGM_REQUIRE(c->setup_done && c->dt > 0, "mgm_timple_part: call mgm_setup and mgm_set_flow first");
        timple_part(c, part, mode);
    });
}

int mgm_timple_run(mgm_ctx *c, int mode, int nsteps, double *step_ms, long long *vcycles, double *steady_err)
{
    return tguard([&] {
        MGM_REQUIRE(c != nullptr, "null context");
        MGM_CUDA(cudaSetDevice(c->device));
        alloc_stream(c->s);
        MGM_REQUIRE(c->setup_done && c->dt > 0, "mgm_timple_run: call mgm_setup and mgm_set_flow first");
        MGM_REQUIRE(nsteps >= 0, "mgm_timple_run: nsteps < 0");
        cudaEvent_t ev[2] = {nullptr, nullptr};
        MGM_CUDA(cudaEventCreate(&ev[0]));
        MGM_CUDA(cudaEventCreate(&ev[1]));
        try {
            c->vcycles_acc = 0;
            double e = 0;
            MGM_CUDA(cudaEventRecord(ev[0], c->s));
            for (int t = 0; t < nsteps; t++) e = timple_step(c, mode);
            MGM_CUDA(cudaEventRecord(ev[1], c->s));
            MGM_CUDA(cudaEventSynchronize(ev[1]));
            float ms = 0;
            MGM_CUDA(cudaEventElapsedTime(&ms, ev[0], ev[1]));
            if (step_ms) *step_ms = ms;
            if (vcycles) *vcycles = c->vcycles_acc;
            if (steady_err) *steady_err = e;
        } catch (...) {
            cudaEventDestroy(ev[0]);
            cudaEventDestroy(ev[1]);
            throw;
        }
        cudaEventDestroy(ev[0]);
        cudaEventDestroy(ev[1]);
    });
}

int mgm_timple_step(mgm_ctx *c, int mode, double *steady_err)
{
    return tguard([&] {
        MGM_REQUIRE(c != nullptr, "null context");
        MGM_CUDA(cudaSetDevice(c->device));
        alloc_stream(c->s);
        MGM_REQUIRE(c->setup_done && c->dt > 0, "mgm_timple_step: call mgm_setup and mgm_set_flow first");
        const double e = timple_step(c, mode);
        if (steady_err) *steady_err = e;
    });
}

}  // extern "C"
