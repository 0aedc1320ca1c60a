// The network's backward kernels called from the tests on given arrays (built by
// probe.py), launched as loss_and_grad launches them.
#include "../include/mgm.h"
#include "../multigrid_meshless_b200/csrc/mem.cu"
#include "../multigrid_meshless_b200/csrc/mpnn.cu"

namespace mgm {
// what the included files want of the others, not called here
long long g_launches = 0;
void set_error(int, const std::string &) {}
void scan_exclusive(const int *, int *, int, int *, cudaStream_t) {}
}  // namespace mgm
extern "C" int mgm_step(mgm_ctx *, int, double *) { return 0; }

namespace {
template <class F>
int code_of(F &&f)
{
    try {
        const mgm::CallStream call;
        f(call.s);
        return 0;
    } catch (const mgm::Error &e) {
        fprintf(stderr, "%s\n", e.msg.c_str());
        return e.code;
    }
}
}  // namespace

// dz = dH [z > 0], gbias = its column sums, gW = cat^T dz (cat: BF16 bits [n][192])
extern "C" int probe_dW(int n, const float *dH, const float *z, const uint16_t *cat, float *dz, float *gbias, float *gW)
{
    using namespace mgm;
    return code_of([&](cudaStream_t s) {
        const size_t nh = (size_t)n * kH, nc = (size_t)n * kCat;
        DBuf<float> d_h(nh), d_z(nh), d_dz(nh), d_b(kH), d_w((size_t)kCat * kH);
        DBuf<uint16_t> d_c(nc);
        d_h.upload(dH, nh, s);
        d_z.upload(z, nh, s);
        d_c.upload(cat, nc, s);
        d_b.zero(s);
        d_w.zero(s);
        MGM_CUDA(cudaFuncSetAttribute(k_dW, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDwSmem));
        k_dW<<<std::min(blocks_for(n, kTile), 148), kDwThreads, kDwSmem, s>>>(
            n, d_h.p, d_z.p, reinterpret_cast<const bf16 *>(d_c.p), d_dz.p, d_b.p, d_w.p);
        MGM_LAUNCHED();
        d_dz.download(dz, nh, s);
        d_b.download(gbias, kH, s);
        d_w.download(gW, (size_t)kCat * kH, s);
        MGM_CUDA(cudaStreamSynchronize(s));
    });
}

// dH += dz W_self^T + mean of the in-edges' dz W_mean^T + their lap-weighted sum W_lap^T (WT: BF16 bits [64][192])
extern "C" int probe_back(int n, int k, int edges, const int *tptr, const int *tpos, const float *lapS, const float *dz,
                          const uint16_t *WT, float *dH)
{
    using namespace mgm;
    return code_of([&](cudaStream_t s) {
        const size_t nh = (size_t)n * kH, nk = (size_t)n * k;
        DBuf<int> d_p(n + 1), d_e(edges);
        DBuf<float> d_l(nk), d_dz(nh), d_h(nh);
        DBuf<uint16_t> d_w((size_t)kH * kCat);
        d_p.upload(tptr, n + 1, s);
        d_e.upload(tpos, edges, s);
        d_l.upload(lapS, nk, s);
        d_dz.upload(dz, nh, s);
        d_h.upload(dH, nh, s);
        d_w.upload(WT, (size_t)kH * kCat, s);
        MGM_CUDA(cudaFuncSetAttribute(k_back, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBackSmem));
        k_back<<<blocks_for(n, kTile), 256, kBackSmem, s>>>(n, k, 1.f / k, d_p.p, d_e.p, d_l.p, d_dz.p,
                                                            reinterpret_cast<const bf16 *>(d_w.p), d_h.p);
        MGM_LAUNCHED();
        d_h.download(dH, nh, s);
        MGM_CUDA(cudaStreamSynchronize(s));
    });
}
