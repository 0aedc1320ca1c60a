// Set-up kernels called from the tests without the C ABI (built by probe.py).
#include "../multigrid_meshless_b200/csrc/krylov.cu"
#include "../multigrid_meshless_b200/csrc/mem.cu"
#include "../multigrid_meshless_b200/csrc/setup.cu"

namespace mgm {
// what the included files want of the others, not called here
long long g_launches = 0;
bool derivative_weights_reg(int, int, int, int, const Monomials &, const double *, const double *, const double *,
                            const double *, const double *, const double *, const uint8_t *, const int *, double *,
                            double *, double *, double *, double *, cudaStream_t)
{
    return false;
}
bool transfer_weights_reg(int, const double *, const double *, const double *, const uint8_t *, const int *, int, int,
                          int, int, int, const Monomials &, const double *, const double *, const double *,
                          const int *, double *, cudaStream_t)
{
    return false;
}
}  // namespace mgm

extern "C" int probe_inv_cand_align() { return (int)alignof(mgm::InvCand); }

namespace {
template <class F>
int code_of(F &&f)
{
    try {
        const mgm::CallStream call;
        f(call.s);
        return 0;
    } catch (const mgm::Error &e) {
        return e.code;
    }
}
}  // namespace

// the inverse of an ELL operator [k][n] and the breadth-first order of row-major
// clouds [n][k] on at most `most` CTAs; 0 or the error's code
extern "C" int probe_dense_inverse(int n, int k, const int *idx, const double *A, double *inv64, float *inv32, int most)
{
    return code_of([&](cudaStream_t s) {
        const size_t nn = (size_t)n * n;
        mgm::DBuf<int> di((size_t)n * k);
        mgm::DBuf<double> dA((size_t)n * k), d64(nn);
        mgm::DBuf<float> d32(nn);
        di.upload(idx, (size_t)n * k, s);
        dA.upload(A, (size_t)n * k, s);
        mgm::dense_inverse(n, k, di.p, dA.p, d64.p, d32.p, s, most);
        d64.download(inv64, nn, s);
        d32.download(inv32, nn, s);
        MGM_CUDA(cudaStreamSynchronize(s));
    });
}

extern "C" int probe_bfs_order(int n, int k, const int *cloud, int *queue, int *reached, int most)
{
    return code_of([&](cudaStream_t s) {
        mgm::DBuf<int> dc((size_t)n * k), dq(n);
        dc.upload(cloud, (size_t)n * k, s);
        *reached = mgm::bfs_order(n, k, dc.p, dq.p, s, most);
        dq.download(queue, n, s);
        MGM_CUDA(cudaStreamSynchronize(s));
    });
}
