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
