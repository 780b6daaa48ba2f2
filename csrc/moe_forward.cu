// The sparse mixture after its router in ONE call: rows sorted by expert, gate / up product with the activation, down product,
// weighted combination -- six launches that read the routing on the device.  One host call and one workspace instead of
// four calls with an allocation each: at 64 tokens (width 1024, 16 experts) the launches take 36 us of GPU time and the four
// calls from Python 80 us of host time.
#include "common.cuh"
#include "gemm_tcgen05.cuh"

NXD_API int nxd_moe_sort_rows(const void* h, const int* idx, int* counts, int* slot, const float* in_scale, void* x, long long P,
                              int top, int W, int E, void* stream);
NXD_API int nxd_experts_gemm_bf16(const void* a, const void* b, void* d, const int* counts, int E, int rows, int pairs, int N,
                                  int K, int mode, float limit, float alpha, float up_shift, void* stream);
NXD_API int nxd_moe_gather_combine(int dtype, const void* ys, const int* slot, const int* idx, const float* wts, const void* h,
                                   const void* shared_out, const float* sgate, float* y, long long N, int top, int W, int E,
                                   void* stream);

namespace {

struct Layout {      // byte offsets into the workspace
    long long rows, counts, slot, x, act, ys, bytes;
};

Layout layout(long long N, int top, int W, int F, int E) {
    auto up = [](long long v) { return (v + 255) / 256 * 256; };
    Layout l;
    l.rows = N * top + (long long)E * nxd_gemm::kSegAlign;
    l.counts = 0;
    l.slot = up(l.counts + 4ll * E);
    l.x = up(l.slot + 4 * N * top);
    l.act = up(l.x + 2 * l.rows * W);
    l.ys = up(l.act + 2 * l.rows * F);
    l.bytes = up(l.ys + 2 * l.rows * W);
    return l;
}

}  // namespace

NXD_API long long nxd_moe_sorted_workspace(long long N, int top, int W, int F, int E) { return layout(N, top, W, F, E).bytes; }

// h [N, W] bf16, idx / wts [N, top] (index >= E: identity expert), in_scale [N, top] fp32 or NULL (the pair's input row is
// multiplied by it), w_in [E, W, 2 F] (gated: gate | up) or [E, W, F] (max(., 0)^2), w_down [E, F, W], shared_out [N, W] bf16
// or NULL, sgate [N] fp32 or NULL -> y [N, W] fp32.  work: nxd_moe_sorted_workspace bytes, 256-byte aligned.  W and F
// multiples of 8, E <= 128, all operands 16-byte aligned.
NXD_API int nxd_moe_sorted_forward(const void* h, const int* idx, const float* wts, const float* in_scale, const void* w_in,
                                   const void* w_down, const void* shared_out, const float* sgate, float* y, void* work,
                                   long long N, int top, int W, int F, int E, int gated, float limit, float alpha,
                                   float up_shift, void* stream) {
    if (N == 0) return 0;
    const Layout l = layout(N, top, W, F, E);
    NXD_REQUIRE(l.rows < (1ll << 31), "sorted experts: %lld rows", l.rows);
    char* base = static_cast<char*>(work);
    int* counts = reinterpret_cast<int*>(base + l.counts);
    int* slot = reinterpret_cast<int*>(base + l.slot);
    void *x = base + l.x, *act = base + l.act, *ys = base + l.ys;
    const int rows = (int)l.rows, pairs = (int)(N * top);
    NXD_CHECK_CUDA(cudaMemsetAsync(counts, 0, 4ll * E, (cudaStream_t)stream));
    int rc = nxd_moe_sort_rows(h, idx, counts, slot, in_scale, x, N * top, top, W, E, stream);
    if (rc) return rc;
    rc = nxd_experts_gemm_bf16(x, w_in, act, counts, E, rows, pairs, F, W, gated ? nxd_gemm::kSegGlu : nxd_gemm::kSegRelu2, limit,
                               alpha, up_shift, stream);
    if (rc) return rc;
    rc = nxd_experts_gemm_bf16(act, w_down, ys, counts, E, rows, pairs, W, F, nxd_gemm::kSegPlain, limit, alpha, up_shift, stream);
    if (rc) return rc;
    return nxd_moe_gather_combine(0, ys, slot, idx, wts, h, shared_out, sgate, y, N, top, W, E, stream);
}
