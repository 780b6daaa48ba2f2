// Sparse mixture-of-experts feed-forward without host synchronisation: router, expert GEMVs that follow the expert
// index on the device ("selective loading": only the chosen experts' weights are touched), clamped gated activation,
// and the weighted combination in fp32.  bf16 or fp32 activations / expert weights; router in fp32.
//
//   router        z = Wr h (+ logit bias);  s = softmax(z);  choice = s + correction;  the `top` largest choices are taken,
//                 weight = s * out_scale (not renormalised);  optional second output sigmoid(<w_sg, h>) per token.
//                 renormalise: the `top` largest LOGITS are taken and the weights are the softmax over the chosen
//                 logits only (times out_scale)
//                 sigmoid scores (mode 2): s = sigmoid(z) per expert instead of the softmax, otherwise as the first form
//                 normalised scores (mode 3): the first form with the chosen s divided by their sum (+ 1e-20)
//   activation    g = min(gate, limit), u = clamp(up, -limit, limit);  a = g * sigmoid(alpha * g) * (u + up_shift)
//                 (limit = +inf, alpha = 1, up_shift = 0: plain silu(gate) * up)
//                 experts without a gate: a = max(up, 0)^2
//   expert index >= E means an identity expert: its output is the token's input itself
// Expert weights are stored [E, in, out] (the layout of the grouped expert layers), gate | up fused on the out dim.
#include "common.cuh"
#include "gemm_tcgen05.cuh"

namespace {

__device__ __forceinline__ float ldf(const float* p) { return *p; }
__device__ __forceinline__ float ldf(const bf16* p) { return __bfloat162float(*p); }
__device__ __forceinline__ void stf(float* p, float v) { *p = v; }
__device__ __forceinline__ void stf(bf16* p, float v) { *p = __float2bfloat16_rn(v); }
__device__ __forceinline__ void ld2(const float* p, float& a, float& b) {
    const float2 v = *reinterpret_cast<const float2*>(p);
    a = v.x;
    b = v.y;
}
__device__ __forceinline__ void ld2(const bf16* p, float& a, float& b) {
    const float2 v = __bfloat1622float2(*reinterpret_cast<const bf162*>(p));
    a = v.x;
    b = v.y;
}

// kind 0: g * sigmoid(alpha g); kind 1: the tanh form of gelu, 0.5 g (1 + tanh(c (g + 0.044715 g^3))) with c = sqrt(2 / pi),
// written through 0.5 (1 + tanh(a)) = sigmoid(2 a)
__device__ __forceinline__ float glu_act(float g, float u, float limit, float alpha, float up_shift, int kind = 0) {
    g = fminf(g, limit);
    u = fminf(fmaxf(u, -limit), limit);
    const float a = kind == 1 ? 1.5957691216057308f * (g + 0.044715f * g * g * g) : alpha * g;
    return g / (1.f + expf(-a)) * (u + up_shift);
}

// ---- router ---------------------------------------------------------------------------------------------------------
constexpr int RT_WARPS = 4, RT_SHARE_WARPS = 8;

// parts of the width that the warps of one token's CTA take: all warps busy also with few outputs
__host__ __device__ inline int router_parts(int R, int warps) {
    const int groups = (R + 3) / 4;
    return groups < warps ? warps / groups : 1;
}

// 8 consecutive values of a row
__device__ __forceinline__ void ld8(const float* p, float* f) {
    *reinterpret_cast<float4*>(f) = *reinterpret_cast<const float4*>(p);
    *reinterpret_cast<float4*>(f + 4) = *reinterpret_cast<const float4*>(p + 4);
}
__device__ __forceinline__ void ld8(const bf16* p, float* f) { unpack8(*reinterpret_cast<const bf16x8*>(p), f); }

// acc[t][i] += <h row t, wr row i> over the columns of this lane in every `parts`-th piece of 32 V from piece `part` on.  V = 8: 16- /
// 32-byte loads (W a multiple of 8, aligned rows); V = 1: any W.  Rows past nt / nr repeat the last one (their sums are not used).
template <typename T, int V, int TOK, int G>
__device__ __forceinline__ void router_dots(const T* h, const float* wr, int W, int nt, int nr, float (&acc)[TOK][G], int part = 0,
                                            int parts = 1) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int t = 0; t < TOK; ++t)
#pragma unroll
        for (int i = 0; i < G; ++i) acc[t][i] = 0.f;
#pragma unroll (TOK == 1 ? 2 : 1)
    for (int c = (part * 32 + lane) * V; c < W; c += parts * 32 * V) {
        float hv[TOK][V];
#pragma unroll
        for (int t = 0; t < TOK; ++t) {
            const T* p = h + (long long)min(t, nt - 1) * W + c;
            if constexpr (V == 8) ld8(p, hv[t]);
            else hv[t][0] = ldf(p);
        }
#pragma unroll
        for (int i = 0; i < G; ++i) {
            const float* p = wr + (long long)min(i, nr - 1) * W + c;
            float wv[V];
            if constexpr (V == 8) ld8(p, wv);
            else wv[0] = *p;
#pragma unroll
            for (int t = 0; t < TOK; ++t)
#pragma unroll
                for (int j = 0; j < V; ++j) acc[t][i] = fmaf(hv[t][j], wv[j], acc[t][i]);
        }
    }
}

// One warp: scores and choice of token n from its logits ps [R]; cs [R]: scratch (choice scores).
__device__ __forceinline__ void router_select(float* ps, float* cs, const float* corr, int* idx, float* wts, long long n, int R,
                                              int top, float out_scale, int mode) {
    const bool renorm = mode == 1;
    const int lane = threadIdx.x & 31;
    if (renorm) {                // the choice is made on the logits themselves
        for (int r = lane; r < R; r += 32) cs[r] = ps[r];
    } else if (mode == 2) {      // independent sigmoid scores
        for (int r = lane; r < R; r += 32) {
            const float p = 1.f / (1.f + expf(-ps[r]));
            ps[r] = p;
            cs[r] = p + (corr != nullptr ? corr[r] : 0.f);
        }
    } else {
        float mx = -INFINITY;
        for (int r = lane; r < R; r += 32) mx = fmaxf(mx, ps[r]);
        mx = warp_max(mx);
        float sum = 0.f;
        for (int r = lane; r < R; r += 32) sum += expf(ps[r] - mx);
        sum = warp_sum(sum);
        const float inv = 1.f / sum;
        __syncwarp();
        for (int r = lane; r < R; r += 32) {
            const float p = expf(ps[r] - mx) * inv;
            ps[r] = p;
            cs[r] = p + (corr != nullptr ? corr[r] : 0.f);
        }
    }
    __syncwarp();
    for (int k = 0; k < top; ++k) {
        float best = -INFINITY;
        int bi = 0x7fffffff;
        for (int r = lane; r < R; r += 32) {
            const float c = cs[r];
            if (c > best) {       // lanes scan upwards: the lowest index wins a tie inside a lane
                best = c;
                bi = r;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ob > best || (ob == best && oi < bi)) {
                best = ob;
                bi = oi;
            }
        }
        if (bi >= R) bi = 0;      // every score NaN: keep the index in range
        if (lane == 0) {
            idx[n * top + k] = bi;
            wts[n * top + k] = (renorm || mode == 3) ? ps[bi] : ps[bi] * out_scale;
            cs[bi] = -INFINITY;
        }
        __syncwarp();
    }
    if (mode == 3 && lane == 0) {
        float sum = 1e-20f;
        for (int k = 0; k < top; ++k) sum += wts[n * top + k];
        const float inv = out_scale / sum;
        for (int k = 0; k < top; ++k) wts[n * top + k] *= inv;
    }
    if (renorm && lane == 0) {   // softmax over the chosen logits only; the first pick is the largest
        const float mx = wts[n * top];
        float sum = 0.f;
        for (int k = 0; k < top; ++k) {
            const float e = expf(wts[n * top + k] - mx);
            wts[n * top + k] = e;
            sum += e;
        }
        const float inv = out_scale / sum;
        for (int k = 0; k < top; ++k) wts[n * top + k] *= inv;
    }
}

// A CTA of RT_WARPS warps.  SHARE: one token and up to RT_SHARE_WARPS warps, they share its experts and the width (few tokens: the latency of
// one token counts, a chain of loads along the width; 64 tokens against four warps that share the outputs only, 1024 x 16 5.6 -> 4.9 us,
// 1024 x 64 14.1 -> 9.1, 2048 x 8 6.9 -> 4.3, 4096 x 8 11.3 -> 5.2).  Else every warp takes TOK tokens and all experts, so a row of wr that is
// loaded serves TOK tokens (many tokens: the fp32 rows of wr come from L1 / L2 and are the larger operand).
template <typename T, int V, int TOK, bool SHARE>
__global__ void __launch_bounds__((SHARE ? RT_SHARE_WARPS : RT_WARPS) * 32)
moe_router_kernel(const T* __restrict__ h, const float* __restrict__ wr, const float* __restrict__ corr,
                  const float* __restrict__ wsg, int* __restrict__ idx, float* __restrict__ wts,
                  float* __restrict__ sgate, long long N, int W, int R, int top, float out_scale,
                  const float* __restrict__ zbias, int mode) {
    extern __shared__ float smem[];
    pdl_wait();
    constexpr int G = SHARE ? 4 : 8;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long n0 = SHARE ? blockIdx.x : ((long long)blockIdx.x * RT_WARPS + warp) * TOK;
    if (n0 >= N) return;                            // SHARE: never; else whole warps, which share nothing
    const int nt = (int)min((long long)TOK, N - n0);
    const T* hr = h + n0 * W;
    if constexpr (SHARE) {
        const int warps = blockDim.x >> 5, groups = (R + G - 1) / G, parts = router_parts(R, warps), part = parts > 1 ? warp / groups : 0;
        float* ps = smem + R;                                       // scratch [R], sums [parts][R], the gate's [warps]
        float* gate = ps + parts * R;
        for (int r0 = (parts > 1 ? warp % groups : warp) * G; r0 < R && part < parts; r0 += warps * G) {
            float acc[1][G];
            router_dots<T, V, 1, G>(hr, wr + (long long)r0 * W, W, 1, R - r0, acc, part, parts);
#pragma unroll
            for (int i = 0; i < G; ++i) {
                const float z = warp_sum(acc[0][i]);
                if (lane == 0 && r0 + i < R) ps[part * R + r0 + i] = z;
            }
        }
        const bool gated = wsg != nullptr && sgate != nullptr;
        if (gated) {
            float acc[1][1];
            router_dots<T, V, 1, 1>(hr, wsg, W, 1, 1, acc, warp, warps);
            const float z = warp_sum(acc[0][0]);
            if (lane == 0) gate[warp] = z;
        }
        pdl_trigger();
        __syncthreads();
        if (warp != 0) return;
        for (int r = lane; r < R; r += 32) {
            float z = ps[r];
            for (int i = 1; i < parts; ++i) z += ps[i * R + r];
            ps[r] = z + (zbias != nullptr ? zbias[r] : 0.f);
        }
        if (gated && lane == 0) {
            float z = gate[0];
            for (int i = 1; i < warps; ++i) z += gate[i];
            sgate[n0] = 1.f / (1.f + expf(-z));
        }
        __syncwarp();
        router_select(ps, smem, corr, idx, wts, n0, R, top, out_scale, mode);
    } else {
        float* ps = smem + warp * (TOK + 1) * R;                    // logits [TOK][R], then scratch [R]
        for (int r0 = 0; r0 < R; r0 += G) {
            float acc[TOK][G];
            router_dots<T, V, TOK, G>(hr, wr + (long long)r0 * W, W, nt, R - r0, acc);
#pragma unroll
            for (int t = 0; t < TOK; ++t)
#pragma unroll
                for (int i = 0; i < G; ++i) {
                    const float z = warp_sum(acc[t][i]);
                    if (lane == 0 && r0 + i < R) ps[t * R + r0 + i] = z + (zbias != nullptr ? zbias[r0 + i] : 0.f);
                }
        }
        if (wsg != nullptr && sgate != nullptr) {
            float acc[TOK][1];
            router_dots<T, V, TOK, 1>(hr, wsg, W, nt, 1, acc);
#pragma unroll
            for (int t = 0; t < TOK; ++t) {
                const float z = warp_sum(acc[t][0]);
                if (lane == 0 && t < nt) sgate[n0 + t] = 1.f / (1.f + expf(-z));
            }
        }
        pdl_trigger();
        __syncwarp();
        for (int t = 0; t < nt; ++t) {
            router_select(ps + t * R, ps + TOK * R, corr, idx, wts, n0 + t, R, top, out_scale, mode);
            __syncwarp();
        }
    }
}

// ---- gate/up GEMV + activation for (token, expert) pairs ----------------------------------------------------------------
constexpr int GV_WARPS = 8;

template <typename T, bool VEC>
__global__ void __launch_bounds__(GV_WARPS * 32)
moe_gate_up_act_kernel(const T* __restrict__ h, const T* __restrict__ wgu, const int* __restrict__ idx,
                       T* __restrict__ act, int pairs_per_token, int W, int F, int E, float limit, float alpha,
                       float up_shift, const float* __restrict__ in_scale) {
    extern __shared__ float smem[];
    constexpr int PER = VEC ? 2 : 1, COLS = 32 * PER;
    float* hs = smem;                                  // [W]
    float* red = smem + W;                             // [GV_WARPS][COLS][2]
    const long long p = blockIdx.x;
    const int e = idx != nullptr ? idx[p] : 0;
    if (e < 0 || e >= E) return;                       // identity expert: no intermediate
    const long long t = p / pairs_per_token;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float xs = in_scale != nullptr ? in_scale[p] : 1.f;       // the pair's weight applied to the expert's INPUT
    for (int c = threadIdx.x; c < W; c += GV_WARPS * 32) hs[c] = ldf(h + t * W + c) * xs;
    __syncthreads();
    const int f0 = blockIdx.y * COLS + lane * PER;
    const int per = (W + GV_WARPS - 1) / GV_WARPS;
    const int k_lo = warp * per, k_hi = min(W, k_lo + per);
    float g0 = 0.f, g1 = 0.f, u0 = 0.f, u1 = 0.f;
    if (f0 < F) {
        const T* base = wgu + (long long)e * W * 2 * F;
#pragma unroll 4
        for (int k = k_lo; k < k_hi; ++k) {
            const T* row = base + (long long)k * 2 * F;
            const float hv = hs[k];
            if (VEC) {
                float a, b, c, d;
                ld2(row + f0, a, b);
                ld2(row + F + f0, c, d);
                g0 = fmaf(hv, a, g0);
                g1 = fmaf(hv, b, g1);
                u0 = fmaf(hv, c, u0);
                u1 = fmaf(hv, d, u1);
            } else {
                g0 = fmaf(hv, ldf(row + f0), g0);
                u0 = fmaf(hv, ldf(row + F + f0), u0);
            }
        }
    }
    float* mine = red + ((long long)warp * COLS + lane * PER) * 2;
    mine[0] = g0;
    mine[1] = u0;
    if (VEC) {
        mine[2] = g1;
        mine[3] = u1;
    }
    __syncthreads();
    if (threadIdx.x < COLS) {
        const int f = blockIdx.y * COLS + threadIdx.x;
        if (f < F) {
            float g = 0.f, u = 0.f;
#pragma unroll
            for (int w = 0; w < GV_WARPS; ++w) {
                g += red[((long long)w * COLS + threadIdx.x) * 2];
                u += red[((long long)w * COLS + threadIdx.x) * 2 + 1];
            }
            stf(act + p * F + f, glu_act(g, u, limit, alpha, up_shift));
        }
    }
}

// the same for experts without a gate: act = max(h @ wu, 0)^2, wu [E, W, F]
template <typename T, bool VEC>
__global__ void __launch_bounds__(GV_WARPS * 32)
moe_up_relu2_kernel(const T* __restrict__ h, const T* __restrict__ wu, const int* __restrict__ idx, T* __restrict__ act,
                    int pairs_per_token, int W, int F, int E) {
    extern __shared__ float smem[];
    constexpr int PER = VEC ? 2 : 1, COLS = 32 * PER;
    float* hs = smem;                                  // [W]
    float* red = smem + W;                             // [GV_WARPS][COLS]
    const long long p = blockIdx.x;
    const int e = idx != nullptr ? idx[p] : 0;
    if (e < 0 || e >= E) return;                       // identity expert: no intermediate
    const long long t = p / pairs_per_token;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int c = threadIdx.x; c < W; c += GV_WARPS * 32) hs[c] = ldf(h + t * W + c);
    __syncthreads();
    const int f0 = blockIdx.y * COLS + lane * PER;
    const int per = (W + GV_WARPS - 1) / GV_WARPS;
    const int k_lo = warp * per, k_hi = min(W, k_lo + per);
    float u0 = 0.f, u1 = 0.f;
    if (f0 < F) {
        const T* base = wu + (long long)e * W * F + f0;
#pragma unroll 8
        for (int k = k_lo; k < k_hi; ++k) {
            const float hv = hs[k];
            if (VEC) {
                float a, b;
                ld2(base + (long long)k * F, a, b);
                u0 = fmaf(hv, a, u0);
                u1 = fmaf(hv, b, u1);
            } else {
                u0 = fmaf(hv, ldf(base + (long long)k * F), u0);
            }
        }
    }
    red[warp * COLS + lane * PER] = u0;
    if (VEC) red[warp * COLS + lane * PER + 1] = u1;
    __syncthreads();
    if (threadIdx.x < COLS) {
        const int f = blockIdx.y * COLS + threadIdx.x;
        if (f < F) {
            float u = 0.f;
#pragma unroll
            for (int w = 0; w < GV_WARPS; ++w) u += red[w * COLS + threadIdx.x];
            u = fmaxf(u, 0.f);
            stf(act + p * F + f, u * u);
        }
    }
}

// ---- down GEMV + weighted combination (+ identity experts, + gated shared expert) -> fp32 ---------------------------
template <typename T, bool VEC>
__global__ void __launch_bounds__(GV_WARPS * 32)
moe_down_combine_kernel(const T* __restrict__ act, const T* __restrict__ wd, const int* __restrict__ idx,
                        const float* __restrict__ wts, const T* __restrict__ h, const T* __restrict__ act_s,
                        const T* __restrict__ wds, const float* __restrict__ sgate, float* __restrict__ y, int top, int W,
                        int F, int Fs, int E) {
    constexpr int PER = VEC ? 2 : 1, COLS = 32 * PER;
    __shared__ float red[GV_WARPS][COLS];
    const long long t = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int c0 = blockIdx.y * COLS + lane * PER;
    float a0 = 0.f, a1 = 0.f;
    if (c0 < W) {
        for (int j = 0; j < top; ++j) {
            const int e = idx[t * top + j];
            const float wgt = wts[t * top + j];
            if (e < 0 || e >= E) {
                if (warp == 0) {
                    a0 = fmaf(wgt, ldf(h + t * W + c0), a0);
                    if (VEC) a1 = fmaf(wgt, ldf(h + t * W + c0 + 1), a1);
                }
                continue;
            }
            const T* arow = act + (t * top + j) * F;
            const T* base = wd + (long long)e * F * W;
            const int per = (F + GV_WARPS - 1) / GV_WARPS;
            const int f_lo = warp * per, f_hi = min(F, f_lo + per);
            float s0 = 0.f, s1 = 0.f;
#pragma unroll 4
            for (int f = f_lo; f < f_hi; ++f) {
                const float av = ldf(arow + f);
                if (VEC) {
                    float p, q;
                    ld2(base + (long long)f * W + c0, p, q);
                    s0 = fmaf(av, p, s0);
                    s1 = fmaf(av, q, s1);
                } else {
                    s0 = fmaf(av, ldf(base + (long long)f * W + c0), s0);
                }
            }
            a0 = fmaf(wgt, s0, a0);
            a1 = fmaf(wgt, s1, a1);
        }
        if (act_s != nullptr) {
            const float wgt = sgate != nullptr ? sgate[t] : 1.f;
            const T* arow = act_s + t * Fs;
            const int per = (Fs + GV_WARPS - 1) / GV_WARPS;
            const int f_lo = warp * per, f_hi = min(Fs, f_lo + per);
            float s0 = 0.f, s1 = 0.f;
#pragma unroll 4
            for (int f = f_lo; f < f_hi; ++f) {
                const float av = ldf(arow + f);
                if (VEC) {
                    float p, q;
                    ld2(wds + (long long)f * W + c0, p, q);
                    s0 = fmaf(av, p, s0);
                    s1 = fmaf(av, q, s1);
                } else {
                    s0 = fmaf(av, ldf(wds + (long long)f * W + c0), s0);
                }
            }
            a0 = fmaf(wgt, s0, a0);
            a1 = fmaf(wgt, s1, a1);
        }
    }
    red[warp][lane * PER] = a0;
    if (VEC) red[warp][lane * PER + 1] = a1;
    __syncthreads();
    if (threadIdx.x < COLS) {
        const int c = blockIdx.y * COLS + threadIdx.x;
        if (c < W) {
            float s = 0.f;
#pragma unroll
            for (int w = 0; w < GV_WARPS; ++w) s += red[w][threadIdx.x];
            y[t * W + c] = s;
        }
    }
}

// ---- pieces of the sorted (GEMM) path: activation over [M, 2F], gather-combine -------------------------------------------
template <typename T>
__global__ void clamped_glu_kernel(const T* __restrict__ gu, T* __restrict__ out, long long M, int F, float limit,
                                   float alpha, float up_shift) {
    const long long total = M * F;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const long long m = i / F;
        const int f = (int)(i - m * F);
        stf(out + i, glu_act(ldf(gu + m * 2 * F + f), ldf(gu + m * 2 * F + F + f), limit, alpha, up_shift));
    }
}

// gate and up are column ranges of a wider row (a fused projection output), each with an optional fp32 bias
template <typename T>
__global__ void glu_bias_kernel(const T* __restrict__ src, long long ld, int gate_off, int up_off,
                                const float* __restrict__ gb, const float* __restrict__ ub, T* __restrict__ out, long long M,
                                int F, float limit, float alpha, float up_shift, int kind) {
    const long long total = M * F;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const long long m = i / F;
        const int f = (int)(i - m * F);
        const float g = ldf(src + m * ld + gate_off + f) + (gb != nullptr ? gb[f] : 0.f);
        const float u = ldf(src + m * ld + up_off + f) + (ub != nullptr ? ub[f] : 0.f);
        stf(out + i, glu_act(g, u, limit, alpha, up_shift, kind));
    }
}

// the same with eight consecutive bf16 columns per thread (16-byte accesses, biases as two float4 each)
__global__ void glu_bias_vec_kernel(const bf16* __restrict__ src, long long ld, int gate_off, int up_off,
                                    const float* __restrict__ gb, const float* __restrict__ ub, bf16* __restrict__ out,
                                    long long M, int F8, float limit, float alpha, float up_shift, int kind) {
    const int f = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
    if (f >= F8 * 8) return;
    float bg[8], bu[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) bg[j] = bu[j] = 0.f;
    if (gb != nullptr) {
        *reinterpret_cast<float4*>(bg) = *reinterpret_cast<const float4*>(gb + f);
        *reinterpret_cast<float4*>(bg + 4) = *reinterpret_cast<const float4*>(gb + f + 4);
    }
    if (ub != nullptr) {
        *reinterpret_cast<float4*>(bu) = *reinterpret_cast<const float4*>(ub + f);
        *reinterpret_cast<float4*>(bu + 4) = *reinterpret_cast<const float4*>(ub + f + 4);
    }
    for (long long m = blockIdx.y; m < M; m += gridDim.y) {
        float g[8], u[8], o[8];
        unpack8(*reinterpret_cast<const bf16x8*>(src + m * ld + gate_off + f), g);
        unpack8(*reinterpret_cast<const bf16x8*>(src + m * ld + up_off + f), u);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = glu_act(g[j] + bg[j], u[j] + bu[j], limit, alpha, up_shift, kind);
        *reinterpret_cast<bf16x8*>(out + m * F8 * 8 + f) = pack8(o);
    }
}

// Programmatic dependents beside the end of the kernel before go to the few SMs that have room by then and stay there.  For the sorting
// kernel and the combination that is worth it while they have few blocks themselves and the router, a block per token, leaves SMs free:
// 2048 x 8 experts, the step as a graph, dependents or not, 64 tokens 66.5 / 66.7 us, 400 84.3 / 71.2, 800 87.3 / 75.5; 1024 x 16 64 tokens
// 31.9 / 32.1, 300 41.3 / 35.3, 6000 156.3 / 153.1.  (The line lies above 100 and below 150 tokens.)  For the same reason every kernel
// of the step triggers behind its work: beside the router, the products' shared memory took its L1 away (24 -> 35 us at width 4096).
template <typename... KArgs, typename... Args>
cudaError_t launch_beside(long long tokens, void (*kernel)(KArgs...), dim3 grid, dim3 block, cudaStream_t stream, Args... args) {
    if (tokens <= 128) return nxd_launch_pdl(kernel, grid, block, 0, stream, args...);
    kernel<<<grid, block, 0, stream>>>(args...);
    return cudaGetLastError();
}

// Bound by memory.  V = 8: a thread takes 8 consecutive columns (16-byte loads of bf16 rows, W a multiple of 8, aligned
// rows); V = 1: any W.  8190 tokens x 2048, top 2: 61 us with one column per thread, 24 us on bf16 outputs (134 MB), 35 us on fp32
// outputs (201 MB, 5.8 TB/s).
// TY: type of the experts' outputs (bf16 or fp32)
template <typename T, int V, typename TY = T>
__global__ void moe_gather_combine_kernel(const TY* __restrict__ ys, const int* __restrict__ slot,
                                          const int* __restrict__ idx, const float* __restrict__ wts,
                                          const T* __restrict__ h, const TY* __restrict__ shared_out,
                                          const float* __restrict__ sgate, float* __restrict__ y, int top, int W, int E) {
    pdl_wait();
    const long long t = blockIdx.x;
    for (int c = threadIdx.x * V; c < W; c += blockDim.x * V) {
        float a[V];
#pragma unroll
        for (int i = 0; i < V; ++i) a[i] = 0.f;
        auto add = [&](const auto* row, float wgt) {
            float v[V];
            if constexpr (V == 8) ld8(row + c, v);
            else v[0] = ldf(row + c);
#pragma unroll
            for (int i = 0; i < V; ++i) a[i] = fmaf(wgt, v[i], a[i]);
        };
        for (int j = 0; j < top; ++j) {
            const int e = idx[t * top + j];
            const float wgt = wts[t * top + j];
            if (e < 0 || e >= E) add(h + t * W, wgt);
            else add(ys + (long long)slot[t * top + j] * W, wgt);
        }
        if (shared_out != nullptr) add(shared_out + t * W, sgate != nullptr ? sgate[t] : 1.f);
        if constexpr (V == 8) {
            float4* dst = reinterpret_cast<float4*>(y + t * W + c);
            dst[0] = make_float4(a[0], a[1], a[2], a[3]);
            dst[1] = make_float4(a[4], a[5], a[6], a[7]);
        } else {
            y[t * W + c] = a[0];
        }
    }
    pdl_trigger();
}

// ---- rows sorted by expert, without a host read ---------------------------------------------------------------------------
// count: how many pairs chose every expert, and every pair's place among its expert's pairs (in no particular order: a row's
// result does not depend on its place).  gather: expert e's rows start where segment_starts (gemm_tcgen05.cuh) says, which the
// grouped product works out the same way; a warp copies one pair's input row there (8190 tokens x 2048, top 2: 24 us for
// 134 MB; a host-side argsort, bincount and index before: 50 us of GPU time and two waits for the device).
constexpr int CNT_THREADS = 256, CNT_PAIRS = 2048;      // pairs per block

__global__ void __launch_bounds__(CNT_THREADS)
moe_count_kernel(const int* __restrict__ idx, int* __restrict__ counts, int* __restrict__ place, long long P, int top, int E) {
    extern __shared__ int hist[];                       // [E] pairs of this block, then [E] the block's first place
    int* first = hist + E;
    pdl_wait();
    for (int e = threadIdx.x; e < E; e += CNT_THREADS) hist[e] = 0;
    __syncthreads();
    if (blockIdx.x == 0 && threadIdx.x == 0) counts[E] = (int)(P / top);      // the tokens: rows of a shared expert
    const long long p0 = (long long)blockIdx.x * CNT_PAIRS;
    int mine[CNT_PAIRS / CNT_THREADS];
#pragma unroll
    for (int i = 0; i < CNT_PAIRS / CNT_THREADS; ++i) {
        const long long p = p0 + i * CNT_THREADS + threadIdx.x;
        const int e = p < P ? idx[p] : -1;
        mine[i] = e >= 0 && e < E ? atomicAdd(hist + e, 1) : 0;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < E; e += CNT_THREADS) first[e] = hist[e] > 0 ? atomicAdd(counts + e, hist[e]) : 0;
    __syncthreads();
    pdl_trigger();
#pragma unroll
    for (int i = 0; i < CNT_PAIRS / CNT_THREADS; ++i) {
        const long long p = p0 + i * CNT_THREADS + threadIdx.x;
        const int e = p < P ? idx[p] : -1;
        if (e >= 0 && e < E) place[p] = first[e] + mine[i];
    }
}

constexpr int GA_WARPS = 8;

// slot [P] (in: place, out: row of the pair); x [rows, W] <- h[p / top]; row_scale [rows] <- in_scale[p] (both NULL: none)
__global__ void __launch_bounds__(GA_WARPS * 32)
moe_gather_rows_kernel(const bf16* __restrict__ h, const int* __restrict__ idx, const int* __restrict__ counts,
                       int* __restrict__ slot, const float* __restrict__ in_scale, float* __restrict__ row_scale,
                       bf16* __restrict__ x, long long P, int top, int W8, int E) {
    __shared__ int row0[nxd_gemm::kSegMaxExperts + 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    pdl_wait();
    if (warp == 0) nxd_gemm::segment_starts(counts, E, 0, row0, nullptr);
    __syncthreads();
    const long long p = (long long)blockIdx.x * GA_WARPS + warp;
    if (p >= P) return;
    const int e = idx[p];
    if (e < 0 || e >= E) return;                        // identity expert: the combination reads h itself
    const int row = row0[e] + slot[p];
    __syncwarp();                                       // every lane has read the place
    if (lane == 0) {
        slot[p] = row;
        if (in_scale != nullptr) row_scale[row] = in_scale[p];
    }
    const bf16x8* src = reinterpret_cast<const bf16x8*>(h) + p / top * W8;
    bf16x8* dst = reinterpret_cast<bf16x8*>(x) + (long long)row * W8;
#pragma unroll 4
    for (int c = lane; c < W8; c += 32) dst[c] = src[c];
    pdl_trigger();
}

// Both of the above for few pairs, in one launch and without zeroed counts: every block counts all pairs itself, a warp finds its
// pair's place by counting the earlier ones of its expert.  A captured step, width 1024, 4 of 16 experts: 64 tokens 41.0 -> 36.9 us, 512
// (2048 pairs) 49.2 -> 41.1.
constexpr int FEW_PAIRS = 2048;

__global__ void __launch_bounds__(GA_WARPS * 32)
moe_sort_few_kernel(const bf16* __restrict__ h, const int* __restrict__ idx, int* __restrict__ counts, int* __restrict__ slot,
                    const float* __restrict__ in_scale, float* __restrict__ row_scale, bf16* __restrict__ x, int P, int top, int W8,
                    int E) {
    __shared__ int expert[FEW_PAIRS], cnt[nxd_gemm::kSegMaxExperts], row0[nxd_gemm::kSegMaxExperts + 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int e = threadIdx.x; e < E; e += GA_WARPS * 32) cnt[e] = 0;
    __syncthreads();
    pdl_wait();
    for (int p = threadIdx.x; p < P; p += GA_WARPS * 32) {
        const int e = idx[p];
        expert[p] = e;
        if (e >= 0 && e < E) atomicAdd(cnt + e, 1);
    }
    __syncthreads();
    if (blockIdx.x == 0) {
        for (int e = threadIdx.x; e < E; e += GA_WARPS * 32) counts[e] = cnt[e];
        if (threadIdx.x == 0) counts[E] = P / top;      // the tokens: rows of a shared expert
    }
    if (warp == 0) nxd_gemm::segment_starts(cnt, E, 0, row0, nullptr);
    __syncthreads();
    const int p = blockIdx.x * GA_WARPS + warp;
    if (p >= P) return;
    const int e = expert[p];
    if (e < 0 || e >= E) return;                        // identity expert: the combination reads h itself
    int before = 0;
    for (int q = lane; q < p; q += 32) before += expert[q] == e;
    const int row = row0[e] + __reduce_add_sync(0xffffffffu, before);
    if (lane == 0) {
        slot[p] = row;
        if (in_scale != nullptr) row_scale[row] = in_scale[p];
    }
    const bf16x8* src = reinterpret_cast<const bf16x8*>(h) + (long long)(p / top) * W8;
    bf16x8* dst = reinterpret_cast<bf16x8*>(x) + (long long)row * W8;
#pragma unroll 4
    for (int c = lane; c < W8; c += 32) dst[c] = src[c];
    pdl_trigger();
}

}  // namespace

// dtype: 0 bf16, 1 fp32 (activations and expert weights).  R = router outputs (experts + identity experts).
// zbias [R] fp32 or NULL: added to the logits; mode 0: softmax scores; 1: choice on the logits, weights = softmax over the
// chosen ones; 2: sigmoid scores; 3: softmax scores, the chosen ones divided by their sum.
NXD_API int nxd_moe_router(int dtype, const void* h, const float* wr, const float* corr, const float* wsg, int* idx,
                           float* wts, float* sgate, long long N, int W, int R, int top, float out_scale,
                           const float* zbias, int mode, void* stream) {
    if (N == 0) return 0;
    NXD_REQUIRE(top >= 1 && top <= R, "router: top %d of %d", top, R);
    NXD_REQUIRE((size_t)8 * R * sizeof(float) <= 48 * 1024, "router: %d outputs", R);
    const bool vec = W % 8 == 0 && ((uintptr_t)h % 16) == 0 && ((uintptr_t)wr % 16) == 0 && ((uintptr_t)wsg % 16) == 0;
    // A CTA per token (tok 0), a warp per token (1) or a warp per 4 tokens (4).  us at 1000 / 2400 / 4000 / 8000 tokens: 256 x 16 7 / 11 /
    // 17 / 30, 7 / 10 / 12 / 21 and 16 / 17 / 17 / 21; 1024 x 64 26 / 56 / 94 / 178, 37 / 59 / 80 / 155 and 52 / 58 / 60 / 79; scalar
    // loads (50 x 64) 10 / 20 / 25 / 42, 14 / 17 / 22 / 38 and 33 / 35 / 36 / 40.  The logits of 16 tokens must fit shared memory.
    const long long sms = nxd_num_sms(), load = (long long)W * R;
    const bool quad = (N >= (vec ? 24 : 64) * sms && N * load >= 1ll << 25) || (vec && N >= 16 * sms && load >= 1 << 16);
    const int tok = N < 8 * sms ? 0 : quad && (size_t)RT_WARPS * 5 * R * sizeof(float) <= 48 * 1024 ? 4 : 1;
    // a token's CTA has eight warps while all tokens together leave room for them (with eight / four, 1000 tokens of 1024 x 16 11.9 / 9.6 us,
    // 400 6.3 / 6.4) and each has a piece to work on (256 x 16: 3.4 / 3.1)
    const int pieces = (R + 3) / 4 * ((W + (vec ? 255 : 31)) / (vec ? 256 : 32));
    const int warps = tok == 0 && N <= 3 * sms && pieces > RT_WARPS ? RT_SHARE_WARPS : RT_WARPS;
    const size_t smem = ((size_t)(tok == 0 ? 1 + router_parts(R, warps) : RT_WARPS * (tok + 1)) * R + (tok == 0 ? warps : 0)) * sizeof(float);
    const unsigned blocks = (unsigned)(tok == 0 ? N : (N + RT_WARPS * tok - 1) / (RT_WARPS * tok));
#define NXD_RT(T, V, TOK, SHARE)                                                                                        \
    NXD_CHECK_CUDA(nxd_launch_pdl(moe_router_kernel<T, V, TOK, SHARE>, dim3(blocks), dim3(warps * 32), smem, (cudaStream_t)stream, \
                                  (const T*)h, wr, corr, wsg, idx, wts, sgate, N, W, R, top, out_scale, zbias, mode))
#define NXD_RT_V(T, V)                                                                                                  \
    do {                                                                                                                \
        if (tok == 0) NXD_RT(T, V, 1, true);                                                                            \
        else if (tok == 1) NXD_RT(T, V, 1, false);                                                                      \
        else NXD_RT(T, V, 4, false);                                                                                    \
    } while (0)
    if (dtype == 0) {
        if (vec) NXD_RT_V(bf16, 8); else NXD_RT_V(bf16, 1);
    } else {
        if (vec) NXD_RT_V(float, 8); else NXD_RT_V(float, 1);
    }
#undef NXD_RT_V
#undef NXD_RT
    NXD_LAUNCH_CHECK();
    return 0;
}

// Rows of the pairs sorted by expert.  counts [E + 1] int32: ZEROED by the caller (unless nxd_moe_sort_counts_itself(P)), out: pairs
// of every expert, then P / top;
// slot [P] int32 out: the pair's row in x (not written for identity experts); x [rows, W] bf16 with rows >= P + 32 E, W a
// multiple of 8; row_scale [rows] <- in_scale [P] of the row's pair (both fp32, or both NULL).
NXD_API int nxd_moe_sort_counts_itself(long long P) { return P <= FEW_PAIRS; }

NXD_API int nxd_moe_sort_rows(const void* h, const int* idx, int* counts, int* slot, const float* in_scale, float* row_scale,
                              void* x, long long P, int top, int W, int E, void* stream) {
    if (P == 0) return 0;
    NXD_REQUIRE(E > 0 && E <= nxd_gemm::kSegMaxExperts && W % 8 == 0, "sort rows: %d experts, width %d", E, W);
    NXD_REQUIRE(((uintptr_t)h % 16) == 0 && ((uintptr_t)x % 16) == 0, "sort rows: rows must be 16-byte aligned");
    cudaStream_t st = (cudaStream_t)stream;
    if (nxd_moe_sort_counts_itself(P)) {
        NXD_CHECK_CUDA(launch_beside(P / top, moe_sort_few_kernel, dim3((unsigned)((P + GA_WARPS - 1) / GA_WARPS)), dim3(GA_WARPS * 32), st,
                                     (const bf16*)h, idx, counts, slot, in_scale, row_scale, (bf16*)x, (int)P, top, W / 8, E));
        NXD_LAUNCH_CHECK();
        return 0;
    }
    NXD_CHECK_CUDA(nxd_launch_pdl(moe_count_kernel, dim3((unsigned)((P + CNT_PAIRS - 1) / CNT_PAIRS)), dim3(CNT_THREADS),
                                  2 * E * sizeof(int), st, idx, counts, slot, P, top, E));
    NXD_LAUNCH_CHECK();
    NXD_CHECK_CUDA(nxd_launch_pdl(moe_gather_rows_kernel, dim3((unsigned)((P + GA_WARPS - 1) / GA_WARPS)), dim3(GA_WARPS * 32), 0, st,
                                  (const bf16*)h, idx, (const int*)counts, slot, in_scale, row_scale, (bf16*)x, P, top, W / 8, E));
    NXD_LAUNCH_CHECK();
    return 0;
}

// act[p, :] = activation(h[p / pairs_per_token] @ wgu[idx[p]]) for P pairs; idx NULL = expert 0 for every pair (a dense
// gated MLP); pairs whose index is outside [0, E) are identity experts and are skipped.  in_scale [P] fp32 or NULL: the
// pair's input row is multiplied by it (routing weight on the expert's input).
NXD_API int nxd_moe_gate_up_act(int dtype, const void* h, const void* wgu, const int* idx, void* act, long long P,
                                int pairs_per_token, int W, int F, int E, float limit, float alpha, float up_shift,
                                const float* in_scale, void* stream) {
    if (P == 0) return 0;
    NXD_REQUIRE(P < (1ll << 31), "gate/up: %lld pairs", P);
    const bool vec = (F % 2) == 0;
    const int cols = vec ? 64 : 32;
    const size_t smem = (size_t)(W + GV_WARPS * cols * 2) * sizeof(float);
    NXD_REQUIRE(smem <= 200 * 1024, "gate/up: input width %d", W);
    dim3 grid((unsigned)P, (F + cols - 1) / cols);
    cudaStream_t st = (cudaStream_t)stream;
#define NXD_GU(T, V)                                                                                                  \
    do {                                                                                                              \
        auto kern = moe_gate_up_act_kernel<T, V>;                                                                     \
        if (smem > 48 * 1024)                                                                                         \
            NXD_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));       \
        kern<<<grid, GV_WARPS * 32, smem, st>>>((const T*)h, (const T*)wgu, idx, (T*)act, pairs_per_token, W, F, E,   \
                                                limit, alpha, up_shift, in_scale);                                    \
    } while (0)
    if (dtype == 0) {
        if (vec) NXD_GU(bf16, true); else NXD_GU(bf16, false);
    } else {
        if (vec) NXD_GU(float, true); else NXD_GU(float, false);
    }
#undef NXD_GU
    NXD_LAUNCH_CHECK();
    return 0;
}

// act[p, :] = max(h[p / pairs_per_token] @ wu[idx[p]], 0)^2; wu [E, W, F]; idx as in nxd_moe_gate_up_act.
NXD_API int nxd_moe_up_relu2(int dtype, const void* h, const void* wu, const int* idx, void* act, long long P,
                             int pairs_per_token, int W, int F, int E, void* stream) {
    if (P == 0) return 0;
    NXD_REQUIRE(P < (1ll << 31), "up: %lld pairs", P);
    const bool vec = (F % 2) == 0;
    const int cols = vec ? 64 : 32;
    const size_t smem = (size_t)(W + GV_WARPS * cols) * sizeof(float);
    NXD_REQUIRE(smem <= 200 * 1024, "up: input width %d", W);
    dim3 grid((unsigned)P, (F + cols - 1) / cols);
    cudaStream_t st = (cudaStream_t)stream;
#define NXD_UP(T, V)                                                                                                  \
    do {                                                                                                              \
        auto kern = moe_up_relu2_kernel<T, V>;                                                                        \
        if (smem > 48 * 1024)                                                                                         \
            NXD_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));       \
        kern<<<grid, GV_WARPS * 32, smem, st>>>((const T*)h, (const T*)wu, idx, (T*)act, pairs_per_token, W, F, E);   \
    } while (0)
    if (dtype == 0) {
        if (vec) NXD_UP(bf16, true); else NXD_UP(bf16, false);
    } else {
        if (vec) NXD_UP(float, true); else NXD_UP(float, false);
    }
#undef NXD_UP
    NXD_LAUNCH_CHECK();
    return 0;
}

// y[t] = sum_j wts[t, j] * (idx[t, j] in [0, E) ? act[t * top + j] @ wd[idx[t, j]] : h[t])
//        + (act_s ? (sgate ? sgate[t] : 1) * act_s[t] @ wds : 0)                                  -> fp32 [N, W]
NXD_API int nxd_moe_down_combine(int dtype, const void* act, const void* wd, const int* idx, const float* wts,
                                 const void* h, const void* act_s, const void* wds, const float* sgate, float* y,
                                 long long N, int top, int W, int F, int Fs, int E, void* stream) {
    if (N == 0) return 0;
    NXD_REQUIRE(N < (1ll << 31), "down/combine: %lld tokens", N);
    const bool vec = (W % 2) == 0;
    const int cols = vec ? 64 : 32;
    dim3 grid((unsigned)N, (W + cols - 1) / cols);
    cudaStream_t st = (cudaStream_t)stream;
#define NXD_DC(T, V)                                                                                                  \
    moe_down_combine_kernel<T, V><<<grid, GV_WARPS * 32, 0, st>>>((const T*)act, (const T*)wd, idx, wts, (const T*)h, \
                                                                  (const T*)act_s, (const T*)wds, sgate, y, top, W, F,  \
                                                                  Fs, E)
    if (dtype == 0) {
        if (vec) NXD_DC(bf16, true); else NXD_DC(bf16, false);
    } else {
        if (vec) NXD_DC(float, true); else NXD_DC(float, false);
    }
#undef NXD_DC
    NXD_LAUNCH_CHECK();
    return 0;
}

NXD_API int nxd_clamped_glu(int dtype, const void* gate_up, void* out, long long M, int F, float limit, float alpha,
                            float up_shift, void* stream) {
    if (M == 0) return 0;
    long long blocks = (M * F + 255) / 256;
    const long long cap = (long long)nxd_num_sms() * 16;
    if (blocks > cap) blocks = cap;
    if (dtype == 0)
        clamped_glu_kernel<bf16><<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>((const bf16*)gate_up, (bf16*)out, M, F,
                                                                                    limit, alpha, up_shift);
    else
        clamped_glu_kernel<float><<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>((const float*)gate_up, (float*)out, M,
                                                                                     F, limit, alpha, up_shift);
    NXD_LAUNCH_CHECK();
    return 0;
}

// ys [pairs, W]: expert outputs in sorted order, slot [N, top]: row of ys of every (token, choice); identity experts read h.
// dtype 0 bf16, 1 fp32, 2: bf16 h with fp32 ys and shared_out.
NXD_API int nxd_moe_gather_combine(int dtype, const void* ys, const int* slot, const int* idx, const float* wts,
                                   const void* h, const void* shared_out, const float* sgate, float* y, long long N,
                                   int top, int W, int E, void* stream) {
    if (N == 0) return 0;
    NXD_REQUIRE(N < (1ll << 31), "combine: %lld tokens", N);
    auto al = [](const void* p) { return ((uintptr_t)p % 16) == 0; };
    const bool vec = W % 8 == 0 && al(ys) && al(h) && al(shared_out) && al(y);
#define NXD_GC(T, V)                                                                                     \
    NXD_CHECK_CUDA(launch_beside(N, moe_gather_combine_kernel<T, V>, dim3((unsigned)N), dim3(128), (cudaStream_t)stream, \
                                 (const T*)ys, slot, idx, wts, (const T*)h, (const T*)shared_out, sgate, y, top, W, E))
    if (dtype == 2) {
#define NXD_GC_WIDE(V)                                                                                   \
    NXD_CHECK_CUDA(launch_beside(N, moe_gather_combine_kernel<bf16, V, float>, dim3((unsigned)N), dim3(128), (cudaStream_t)stream, \
                                 (const float*)ys, slot, idx, wts, (const bf16*)h, (const float*)shared_out, sgate, y, top, W, E))
        if (vec) NXD_GC_WIDE(8); else NXD_GC_WIDE(1);
#undef NXD_GC_WIDE
    } else if (dtype == 0) {
        if (vec) NXD_GC(bf16, 8); else NXD_GC(bf16, 1);
    } else {
        if (vec) NXD_GC(float, 8); else NXD_GC(float, 1);
    }
#undef NXD_GC
    NXD_LAUNCH_CHECK();
    return 0;
}

NXD_API int nxd_glu_bias(int dtype, const void* src, long long ld, int gate_off, int up_off, const float* gate_bias,
                         const float* up_bias, void* out, long long M, int F, float limit, float alpha, float up_shift,
                         int act_kind, void* stream) {
    if (M * F == 0) return 0;
    long long blocks = (M * F + 255) / 256;
    const long long cap = (long long)nxd_num_sms() * 16;
    if (blocks > cap) blocks = cap;
    if (dtype == 0 && F % 8 == 0 && ld % 8 == 0 && gate_off % 8 == 0 && up_off % 8 == 0 && ((uintptr_t)src % 16) == 0 &&
        ((uintptr_t)out % 16) == 0 && ((uintptr_t)gate_bias % 16) == 0 && ((uintptr_t)up_bias % 16) == 0) {
        const int F8 = F / 8, threads = F8 >= 256 ? 256 : ((F8 + 31) / 32) * 32;
        const long long rows_cap = (long long)nxd_num_sms() * 32;         // rows beyond that are walked by the same CTAs
        dim3 grid((F8 + threads - 1) / threads, (unsigned)(M < rows_cap ? M : rows_cap));
        glu_bias_vec_kernel<<<grid, threads, 0, (cudaStream_t)stream>>>((const bf16*)src, ld, gate_off, up_off, gate_bias,
                                                                        up_bias, (bf16*)out, M, F8, limit, alpha, up_shift,
                                                                        act_kind);
        NXD_LAUNCH_CHECK();
        return 0;
    }
    if (dtype == 0)
        glu_bias_kernel<bf16><<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>((const bf16*)src, ld, gate_off, up_off,
                                                                                 gate_bias, up_bias, (bf16*)out, M, F, limit,
                                                                                 alpha, up_shift, act_kind);
    else
        glu_bias_kernel<float><<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>((const float*)src, ld, gate_off, up_off,
                                                                                  gate_bias, up_bias, (float*)out, M, F,
                                                                                  limit, alpha, up_shift, act_kind);
    NXD_LAUNCH_CHECK();
    return 0;
}
