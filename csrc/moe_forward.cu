// The sparse mixture in ONE call, after its router or with it: rows sorted by expert, gate / up product with the activation, down
// product, weighted combination, and a shared expert's two products -- launches that read the routing on the device.  One host call and
// one workspace instead of five calls with allocations: 64 tokens (width 1024, 4 of 16 experts) are five launches, 37 us of GPU time
// and 43 eagerly; with the router in a call of its own, a memset and separate counting 41 and 62, in calls of their own 80.
#include "common.cuh"
#include "gemm_tcgen05.cuh"

NXD_API int nxd_moe_router(int dtype, const void* h, const float* wr, const float* corr, const float* wsg, int* idx, float* wts,
                           float* sgate, long long N, int W, int R, int top, float out_scale, const float* zbias, int mode,
                           void* stream);
NXD_API int nxd_moe_sort_counts_itself(long long P);
NXD_API int nxd_moe_sort_rows(const void* h, const int* idx, int* counts, int* slot, const float* in_scale, float* row_scale,
                              void* x, long long P, int top, int W, int E, void* stream);
NXD_API int nxd_experts_gemm_bf16(const void* a, const void* b, void* d, const int* counts, const float* row_scale, int E,
                                  int rows, int pairs, int N, int K, int mode, float limit, float alpha, float up_shift,
                                  void* stream);
NXD_API int nxd_moe_gather_combine(int dtype, const void* ys, const int* slot, const int* idx, const float* wts, const void* h,
                                   const void* shared_out, const float* sgate, float* y, long long N, int top, int W, int E,
                                   void* stream);

namespace {

struct Layout {      // byte offsets into the workspace
    long long rows, counts, slot, scale, x, act, ys, s_act, s_out, idx, wts, sgate, bytes;
};

// The experts' outputs are kept in fp32 up to the weighted sum, as the per-pair GEMVs keep them, at every size: a captured step
// had no other path before, and a batch must not lose bits by growing.  Rounded to bf16 they would be half the traffic: 8190 tokens
// x 2048, top 2: 97 + 26 us for the down product and the combination instead of 104 + 35, and an error of 0.0023 instead of 0.0017.
Layout layout(long long N, int top, int W, int F, int E, int Fs) {
    auto up = [](long long v) { return (v + 255) / 256 * 256; };
    Layout l;
    l.rows = N * top + (long long)E * nxd_gemm::kSegAlign;
    l.counts = 0;
    l.slot = up(l.counts + 4ll * (E + 1));
    l.scale = up(l.slot + 4 * N * top);
    l.x = up(l.scale + 4 * l.rows);
    l.act = up(l.x + 2 * l.rows * W);
    l.ys = up(l.act + 2 * l.rows * F);
    l.s_act = up(l.ys + 4 * l.rows * W);
    l.s_out = up(l.s_act + 2 * N * Fs);
    l.idx = up(l.s_out + (Fs > 0 ? 4 * N * W : 0));      // nxd_moe_routed_forward
    l.wts = up(l.idx + 4 * N * top);
    l.sgate = up(l.wts + 4 * N * top);
    l.bytes = up(l.sgate + (Fs > 0 ? 4 * N : 0));
    return l;
}

}  // namespace

NXD_API long long nxd_moe_sorted_workspace(long long N, int top, int W, int F, int E, int Fs) {
    return layout(N, top, W, F, E, Fs).bytes;
}

// h [N, W] bf16, idx / wts [N, top] (index >= E: identity expert), in_scale [N, top] fp32 or NULL (the pair's input row is
// multiplied by it), w_in [E, W, 2 F] (gated: gate | up) or [E, W, F] (max(., 0)^2), w_down [E, F, W], a shared expert s_in
// [W, 2 Fs] or [W, Fs], s_down [Fs, W] (Fs 0: none) with its clamp s_limit and gate sgate [N] fp32 or NULL -> y [N, W] fp32.
// work: nxd_moe_sorted_workspace bytes, 256-byte aligned.  W, F and Fs multiples of 8, E <= 128, operands 16-byte aligned.
NXD_API int nxd_moe_sorted_forward(const void* h, const int* idx, const float* wts, const float* in_scale, const void* w_in,
                                   const void* w_down, const void* s_in, const void* s_down, const float* sgate, float* y,
                                   void* work, long long N, int top, int W, int F, int E, int Fs, int gated, float limit,
                                   float s_limit, float alpha, float up_shift, void* stream) {
    if (N == 0) return 0;
    const Layout l = layout(N, top, W, F, E, Fs);
    NXD_REQUIRE(l.rows < (1ll << 31), "sorted experts: %lld rows", l.rows);
    char* base = static_cast<char*>(work);
    int* counts = reinterpret_cast<int*>(base + l.counts);
    int* slot = reinterpret_cast<int*>(base + l.slot);
    void *x = base + l.x, *act = base + l.act, *ys = base + l.ys;
    const int rows = (int)l.rows, pairs = (int)(N * top);
    if (!nxd_moe_sort_counts_itself(N * top)) NXD_CHECK_CUDA(cudaMemsetAsync(counts, 0, 4ll * (E + 1), (cudaStream_t)stream));
    NXD_REQUIRE(in_scale == nullptr || gated, "sorted experts: %s", "a weight on the input needs gated experts");
    float* scale = in_scale != nullptr ? reinterpret_cast<float*>(base + l.scale) : nullptr;
    int rc = nxd_moe_sort_rows(h, idx, counts, slot, in_scale, scale, x, N * top, top, W, E, stream);
    if (rc) return rc;
    rc = nxd_experts_gemm_bf16(x, w_in, act, counts, scale, E, rows, pairs, F, W, gated ? nxd_gemm::kSegGlu : nxd_gemm::kSegRelu2,
                               limit, alpha, up_shift, stream);
    if (rc) return rc;
    rc = nxd_experts_gemm_bf16(act, w_down, ys, counts, nullptr, E, rows, pairs, W, F, nxd_gemm::kSegPlain, limit, alpha, up_shift,
                               stream);
    if (rc) return rc;
    void* s_out = nullptr;
    if (Fs > 0) {
        s_out = base + l.s_out;
        rc = nxd_experts_gemm_bf16(h, s_in, base + l.s_act, counts + E, nullptr, 1, (int)N, (int)N, Fs, W,
                                   gated ? nxd_gemm::kSegGlu : nxd_gemm::kSegRelu2, s_limit, alpha, up_shift, stream);
        if (rc) return rc;
        rc = nxd_experts_gemm_bf16(base + l.s_act, s_down, s_out, counts + E, nullptr, 1, (int)N, (int)N, W, Fs,
                                   nxd_gemm::kSegPlain, s_limit, alpha, up_shift, stream);
        if (rc) return rc;
    }
    return nxd_moe_gather_combine(2, ys, slot, idx, wts, h, s_out, sgate, y, N, top, W, E, stream);
}

// The same with its router in front (see nxd_moe_router: R outputs, wr [R, W], corr / zbias [R] or NULL, wsg [W] or NULL), the weight on
// the expert's output.  The routing stays in the workspace.
NXD_API int nxd_moe_routed_forward(const void* h, const float* wr, const float* corr, const float* wsg, const float* zbias, int R,
                                   float out_scale, int mode, const void* w_in, const void* w_down, const void* s_in,
                                   const void* s_down, float* y, void* work, long long N, int top, int W, int F, int E, int Fs,
                                   int gated, float limit, float s_limit, float alpha, float up_shift, void* stream) {
    if (N == 0) return 0;
    const Layout l = layout(N, top, W, F, E, Fs);
    char* base = static_cast<char*>(work);
    int* idx = reinterpret_cast<int*>(base + l.idx);
    float *wts = reinterpret_cast<float*>(base + l.wts), *sgate = wsg != nullptr && Fs > 0 ? reinterpret_cast<float*>(base + l.sgate) : nullptr;
    const int rc = nxd_moe_router(0, h, wr, corr, wsg, idx, wts, sgate, N, W, R, top, out_scale, zbias, mode, stream);
    if (rc) return rc;
    return nxd_moe_sorted_forward(h, idx, wts, nullptr, w_in, w_down, s_in, s_down, sgate, y, work, N, top, W, F, E, Fs, gated, limit,
                                  s_limit, alpha, up_shift, stream);
}
