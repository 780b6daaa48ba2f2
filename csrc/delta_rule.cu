// Gated delta rule: a recurrent mixer whose per-head state S [D, Dv] (fp32, one per cache line) is decayed, corrected by
// the error of its own prediction and read out, token by token:
//
//     S <- g_t * S;   u = beta_t (v_t - S^T k_t);   S <- S + k_t u^T;   o_t = S^T q_t
//
// g_t is one number per head, or one per head and key channel (it then scales the rows of S).  Queries, keys and values
// come out of a short causal convolution over time (per channel, no bias) followed by silu; queries and keys are then
// unit vectors per head (the queries also scaled).  Four kernels:
//
//   delta_prep         convolution + silu (+ unit norm) of the step's q | k | v channels -> fp32; tokens before the step
//                      come from the line's convolution state (the last taps - 1 raw projections), zeros before the
//                      start of the sequence
//   delta_conv_state   moves the convolution state to the end of the step
//   delta_gates        decays exp(-exp(A) softplus(a + bias)) and beta = sigmoid(b) from the fp32 pre-activations, in
//                      place, one thread per value
//   delta_scan         the recurrence.  The columns of S are independent, so a thread owns a slice of one column in
//                      registers (R lanes share a column and split its rows); the step's tokens stream through shared
//                      memory in blocks of 16.  Per token both dot products are taken against the decayed
//                      state in one pass, o = (gS)^T q + u (k . q), then the rank-one update.  A row that starts at
//                      position 0 starts from the zero state, any other row continues from its line's state; padding
//                      tokens (t >= n_new[b]) change nothing and come out as zeros.
// This file is compiled without fast-math: the state lives for thousands of steps.
#include "common.cuh"
#include "delta_chunks.cuh"
#include "mma_sync.cuh"

namespace {

using nxd_delta::CH;
using nxd_delta::CHUNK_FLOATS;
using nxd_delta::CW_COLS;

__device__ __forceinline__ float ldf(const float* p) { return *p; }
__device__ __forceinline__ float ldf(const bf16* p) { return __bfloat162float(*p); }

__device__ __forceinline__ float silu_f(float z) { return z / (1.f + expf(-z)); }
__device__ __forceinline__ float softplus_f(float z) { return z > 20.f ? z : log1pf(expf(z)); }

constexpr int MAX_TAPS = 32;

// raw projection of channel `c` (column `col` of the row) at step index s (may be negative: before the step)
template <typename T>
__device__ __forceinline__ float conv_input(const T* __restrict__ proj, long long ld, const float* __restrict__ state,
                                            long long row0, int s, int p0, int K, int C, int c, long long col) {
    if (s >= 0) return ldf(proj + (row0 + s) * ld + col);
    if (p0 + s < 0) return 0.f;                                  // before the start of the sequence
    return state[(long long)(K + s) * C + c];                    // slot K + s holds position p0 + s
}

template <typename T>
__global__ void delta_prep_kernel(const T* __restrict__ proj, long long ld, int off_q, int off_k, int off_v,
                                  const float* __restrict__ conv_w, const float* __restrict__ conv_state,
                                  float* __restrict__ qn, float* __restrict__ kn, float* __restrict__ vn,
                                  const int* __restrict__ q_start, const int* __restrict__ n_new,
                                  const int* __restrict__ seq_ids, long long units, int Tn, int H, int G, int D, int Dv,
                                  int taps, float qscale, float unit_eps) {
    const int lane = threadIdx.x & 31;
    const long long unit = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (unit >= units) return;
    const int per_row = 2 * G + H;
    const long long n = unit / per_row;
    const int u = (int)(unit % per_row);
    const int b = (int)(n / Tn), t = (int)(n % Tn);
    if (n_new != nullptr && t >= n_new[b]) return;
    const int C = 2 * G * D + H * Dv, K = taps - 1;
    int cbase, dim;
    long long col;
    float* dst;
    bool unitnorm;
    float mul = 1.f;
    if (u < G) {
        cbase = u * D, col = off_q + (long long)u * D, dim = D, dst = qn + (n * G + u) * D, unitnorm = true, mul = qscale;
    } else if (u < 2 * G) {
        cbase = G * D + (u - G) * D, col = off_k + (long long)(u - G) * D, dim = D, dst = kn + (n * G + (u - G)) * D;
        unitnorm = true;
    } else {
        cbase = 2 * G * D + (u - 2 * G) * Dv, col = off_v + (long long)(u - 2 * G) * Dv, dim = Dv;
        dst = vn + (n * H + (u - 2 * G)) * Dv, unitnorm = false;
    }
    const int line = seq_ids != nullptr ? seq_ids[b] : b;
    const int p0 = q_start[b];
    const float* st = conv_state + (long long)line * K * C;
    const long long row0 = (long long)b * Tn;
    float ss = 0.f;
    for (int i = lane; i < dim; i += 32) {
        const float* w = conv_w + (long long)(cbase + i) * taps;
        float acc = 0.f;
        for (int j = 0; j < taps; ++j)
            acc = fmaf(w[j], conv_input(proj, ld, st, row0, t - (K - j), p0, K, C, cbase + i, col + i), acc);
        const float v = silu_f(acc);
        dst[i] = v;
        ss = fmaf(v, v, ss);
    }
    if (!unitnorm) return;
    ss = warp_sum(ss);
    const float r = mul / sqrtf(ss + unit_eps);
    for (int i = lane; i < dim; i += 32) dst[i] *= r;            // every lane rescales what it wrote itself
}

// The same for 4 taps and sizes of 32 V channels (D = 32 V, Dv a multiple): a lane owns V neighbouring channels of one query,
// key or value piece and walks a strip of tokens with the last three inputs in registers, so every projection value is
// read once (the general kernel reads it once per tap, 2 bytes at a time).  Bound by memory: 4 x 2048 tokens, 4 + 4 heads of
// 128 and 4 of 256 (100 MB with the fp32 results): 44 us, 177 us with the general kernel.
constexpr int PREP_STRIP = 16, PREP_SHORT = 4, PREP_AHEAD = 4;

template <int V>
__device__ __forceinline__ void ld_v(const float* p, float* f) {
    if constexpr (V == 2) {
        const float2 a = *reinterpret_cast<const float2*>(p);
        f[0] = a.x, f[1] = a.y;
    } else {
#pragma unroll
        for (int i = 0; i < V; i += 4) *reinterpret_cast<float4*>(f + i) = *reinterpret_cast<const float4*>(p + i);
    }
}
template <int V>
__device__ __forceinline__ void ld_v(const bf16* p, float* f) {
    uint32_t w[V / 2];
    if constexpr (V == 2) w[0] = *reinterpret_cast<const uint32_t*>(p);
    if constexpr (V == 4) *reinterpret_cast<uint2*>(w) = *reinterpret_cast<const uint2*>(p);
    if constexpr (V == 8) *reinterpret_cast<uint4*>(w) = *reinterpret_cast<const uint4*>(p);
#pragma unroll
    for (int i = 0; i < V / 2; ++i) {
        const float2 a = __bfloat1622float2(*reinterpret_cast<const bf162*>(w + i));
        f[2 * i] = a.x, f[2 * i + 1] = a.y;
    }
}
template <int V>
__device__ __forceinline__ void st_v(float* p, const float* f) {
    if constexpr (V == 2) *reinterpret_cast<float2*>(p) = make_float2(f[0], f[1]);
    else
#pragma unroll
        for (int i = 0; i < V; i += 4) *reinterpret_cast<float4*>(p + i) = make_float4(f[i], f[i + 1], f[i + 2], f[i + 3]);
}

template <typename T, int V>
__global__ void __launch_bounds__(256)
delta_prep_strip_kernel(const T* __restrict__ proj, long long ld, int off_q, int off_k, int off_v,
                        const float* __restrict__ conv_w, const float* __restrict__ conv_state, float* __restrict__ qn,
                        float* __restrict__ kn, float* __restrict__ vn, const int* __restrict__ q_start,
                        const int* __restrict__ n_new, const int* __restrict__ seq_ids, int units, int Tn, int H, int G, int Dv,
                        float qscale, float unit_eps, int strip) {
    pdl_wait();
    constexpr int D = 32 * V, TAPS = 4, K = TAPS - 1;
    const int lane = threadIdx.x & 31, u = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (u >= units) return;
    const int b = blockIdx.z, s0 = blockIdx.y * strip;
    const int n = n_new != nullptr ? min(n_new[b], Tn) : Tn;
    const int s_end = min(n, s0 + strip);
    if (s0 >= s_end) return;
    const int C = 2 * G * D + H * Dv;
    const int c = u * D + lane * V;                              // channel in q | k | v order
    long long col;
    float* dst;                                                  // of the batch row's first token
    long long pitch;
    if (u < G) {
        col = off_q + c, dst = qn + (long long)b * Tn * G * D + c, pitch = (long long)G * D;
    } else if (u < 2 * G) {
        col = off_k + c - G * D, dst = kn + (long long)b * Tn * G * D + c - G * D, pitch = (long long)G * D;
    } else {
        col = off_v + c - 2 * G * D, dst = vn + (long long)b * Tn * H * Dv + c - 2 * G * D, pitch = (long long)H * Dv;
    }
    const int line = seq_ids != nullptr ? seq_ids[b] : b, p0 = q_start[b];
    const float* st = conv_state + (long long)line * K * C;
    const T* src = proj + (long long)b * Tn * ld + col;
    float w[V * TAPS], x[TAPS + PREP_AHEAD - 1][V];              // x[i]: inputs of step s - K + i
#pragma unroll
    for (int i = 0; i < V * TAPS; i += 4)
        *reinterpret_cast<float4*>(w + i) = *reinterpret_cast<const float4*>(conv_w + (long long)c * TAPS + i);
#pragma unroll
    for (int i = 0; i < K; ++i) {
        const int s = s0 - K + i;
        if (s >= 0) {
            ld_v<V>(src + s * ld, x[i]);
        } else {
#pragma unroll
            for (int e = 0; e < V; ++e) x[i][e] = p0 + s < 0 ? 0.f : st[(long long)(K + s) * C + c + e];
        }
    }
    const float mul = u < G ? qscale : 1.f;
    for (int s = s0; s < s_end; s += PREP_AHEAD) {
#pragma unroll
        for (int a = 0; a < PREP_AHEAD; ++a)
            ld_v<V>(src + min(s + a, s_end - 1) * ld, x[K + a]);
#pragma unroll
        for (int a = 0; a < PREP_AHEAD; ++a) {
            if (s + a >= s_end) break;
            float v[V], ss = 0.f;
#pragma unroll
            for (int e = 0; e < V; ++e) {
                float acc = 0.f;
#pragma unroll
                for (int j = 0; j < TAPS; ++j) acc = fmaf(w[e * TAPS + j], x[a + j][e], acc);
                v[e] = silu_f(acc);
                ss = fmaf(v[e], v[e], ss);
            }
            if (u < 2 * G) {
                const float r = mul / sqrtf(warp_sum(ss) + unit_eps);
#pragma unroll
                for (int e = 0; e < V; ++e) v[e] *= r;
            }
            st_v<V>(dst + (s + a) * pitch, v);
        }
#pragma unroll
        for (int i = 0; i < K; ++i)
#pragma unroll
            for (int e = 0; e < V; ++e) x[i][e] = x[PREP_AHEAD + i][e];
    }
    pdl_trigger();      // behind the work, as in all kernels of a prompt: at their start, 4 x 1500 tokens of 8 heads of 256 x 512 took 839 us,
                        // 826 so, 831 without programmatic dependents (blocks that start early crowd the SMs that have room)
}

template <typename T, int V>
int launch_prep_strip(const void* proj, long long ld, int off_q, int off_k, int off_v, const float* conv_w,
                      const float* conv_state, float* qn, float* kn, float* vn, const int* q_start, const int* n_new,
                      const int* seq_ids, int B, int Tn, int H, int G, int Dv, float qscale, float unit_eps, cudaStream_t st) {
    const int units = 2 * G + H * (Dv / (32 * V));
    // short strips (every input read 1.75 times) while long ones would be too few warps: 1 x 64 tokens, 4 + 4 heads of 128 and 4 of
    // 256: 13.1 us in strips of 16, 7.6 in strips of 4 (13.8 in the general kernel); 8 x 128 tokens, 3 x 16 heads of 128: 19.2 / 20.2
    const int strip = (long long)units * ((Tn + PREP_STRIP - 1) / PREP_STRIP) * B < 1536 ? PREP_SHORT : PREP_STRIP;
    dim3 grid((units + 7) / 8, (Tn + strip - 1) / strip, B);
    NXD_CHECK_CUDA((nxd_launch_pdl(delta_prep_strip_kernel<T, V>, grid, dim3(256), 0, st, (const T*)proj, ld, off_q, off_k, off_v,
        conv_w, conv_state, qn, kn, vn, q_start, n_new, seq_ids, units, Tn, H, G, Dv, qscale, unit_eps, strip)));
    NXD_LAUNCH_CHECK();
    return 0;
}

template <typename T>
__global__ void delta_conv_state_kernel(const T* __restrict__ proj, long long ld, int off_q, int off_k, int off_v,
                                        float* __restrict__ conv_state, const int* __restrict__ q_start,
                                        const int* __restrict__ n_new, const int* __restrict__ seq_ids, int B, int Tn,
                                        int GD, int C, int taps) {
    pdl_wait();
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)B * C) return;
    const int b = (int)(idx / C), c = (int)(idx % C);
    const int n = n_new != nullptr ? min(n_new[b], Tn) : Tn;
    if (n <= 0) return;
    const int K = taps - 1;
    const int line = seq_ids != nullptr ? seq_ids[b] : b;
    const int p0 = q_start[b];
    const long long col = c < GD ? off_q + c : (c < 2 * GD ? off_k + (c - GD) : off_v + (c - 2 * GD));
    float* st = conv_state + (long long)line * K * C;
    float vals[MAX_TAPS];
    for (int s = 0; s < K; ++s)                                  // slot s <- position (p0 + n) - K + s
        vals[s] = conv_input(proj, ld, st, (long long)b * Tn, n - K + s, p0, K, C, c, col);
    for (int s = 0; s < K; ++s) st[(long long)s * C + c] = vals[s];
    pdl_trigger();
}

constexpr int SCAN_THREADS = 128, SCAN_TS = 16;

// In place: a <- exp(-exp(a_log[h]) softplus(a + dt_bias)) for the decay pre-activations (per head: one column, per
// channel: D columns per head), b <- sigmoid(b) for the beta pre-activations.  One thread per value.
__global__ void delta_gates_kernel(float* __restrict__ apre, long long ld_a, int a_off, float* __restrict__ bpre,
                                   long long ld_b, int b_off, const float* __restrict__ a_log,
                                   const float* __restrict__ dt_bias, long long N, int H, int per_head) {
    pdl_wait();
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int cols = H * per_head + H;                 // decay columns, then beta columns
    if (idx >= N * cols) return;
    const long long n = idx / cols;
    const int c = (int)(idx - n * cols);
    if (c < H * per_head) {
        float* p = apre + n * ld_a + a_off + c;
        *p = expf(-expf(a_log[c / per_head]) * softplus_f(*p + dt_bias[c]));
    } else {
        float* p = bpre + n * ld_b + b_off + (c - H * per_head);
        *p = 1.f / (1.f + expf(-*p));
    }
    pdl_trigger();
}

__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}

// A thread keeps NPT rows of one state column in registers; the R lanes that share a column sit cpw = 32 / R lanes apart.
// In shared memory the NPT values that a lane reads per token are padded to NPT + 4 floats, so that the R simultaneous
// 16-byte reads of a warp fall into different banks.  Blocks of TS tokens are double-buffered: with ASYNC the next block
// is fetched by cp.async (16 bytes a copy; key / value sizes and pitches that are multiples of 4) while the current one
// is consumed; otherwise by plain loads.
template <int NPT, bool ASYNC>
__global__ void __launch_bounds__(SCAN_THREADS)
delta_scan_kernel(const float* __restrict__ qn, const float* __restrict__ kn, const float* __restrict__ vn,
                  const float* __restrict__ gate, long long ld_a, int a_off, const float* __restrict__ beta,
                  long long ld_b, int b_off, float* __restrict__ S, float* __restrict__ out,
                  const int* __restrict__ q_start, const int* __restrict__ n_new, const int* __restrict__ seq_ids, int Tn,
                  int H, int G, int D, int Dv, int per_channel, int R, int TS) {
    extern __shared__ __align__(16) float smem[];
    constexpr int PITCH = NPT + 4;
    const int DS = R * PITCH, CT = SCAN_THREADS / R, cpw = 32 / R;      // floats per token; columns per block / per warp
    const int per_buf = TS * DS * (per_channel ? 3 : 2) + TS * CT + 2 * TS;
    float* kq = smem + 2 * per_buf;                    // [TS] k . q of the block being consumed
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int r = lane / cpw, cl = lane % cpw;
    const int col0 = blockIdx.x * CT, col = col0 + warp * cpw + cl;
    const int h = blockIdx.y, b = blockIdx.z, kvh = h / (H / G);
    const int n = n_new != nullptr ? min(n_new[b], Tn) : Tn;
    const long long row0 = (long long)b * Tn;
    float* orow = out + (row0 * H + h) * Dv;           // + t * H * Dv + col
    if (r == 0 && col < Dv)
        for (int t = max(n, 0); t < Tn; ++t) orow[(long long)t * H * Dv + col] = 0.f;
    if (n <= 0) return;
    const int line = seq_ids != nullptr ? seq_ids[b] : b;
    float* Sb = S + ((long long)line * H + h) * D * Dv;
    float s[NPT];
    const bool fresh = q_start[b] == 0;
#pragma unroll
    for (int ii = 0; ii < NPT; ++ii) {
        const int i = r * NPT + ii;
        s[ii] = (!fresh && i < D && col < Dv) ? Sb[(long long)i * Dv + col] : 0.f;
    }
    const int Dpad = R * NPT;
    // buffer layout: k [TS][DS] | q [TS][DS] | (g [TS][DS]) | v [TS][CT] | g per head [TS] | beta [TS]
    auto fetch = [&](int t0, int buf) {
        float* ks = smem + buf * per_buf;
        float* qs = ks + TS * DS;
        float* gs = qs + TS * DS;
        float* vs = gs + (per_channel ? TS * DS : 0);
        float* gh = vs + TS * CT;
        float* bs = gh + TS;
        const int cnt = min(TS, n - t0);
        if (ASYNC) {
            const int c4 = Dpad / 4;                   // 16-byte pieces per token
            for (int idx = tid; idx < cnt * c4; idx += SCAN_THREADS) {
                const int tt = idx / c4, i = (idx - tt * c4) * 4;
                const long long row = row0 + t0 + tt;
                const int at = tt * DS + (i / NPT) * PITCH + (i % NPT);
                const bool ok = i < D;
                const long long src = (row * G + kvh) * D + (ok ? i : 0);
                mma::cp_async16((uint32_t)__cvta_generic_to_shared(ks + at), kn + src, ok);
                mma::cp_async16((uint32_t)__cvta_generic_to_shared(qs + at), qn + src, ok);
                if (per_channel)
                    mma::cp_async16((uint32_t)__cvta_generic_to_shared(gs + at),
                                    gate + row * ld_a + a_off + (long long)h * D + (ok ? i : 0), ok);
            }
            const int v4 = CT / 4;
            for (int idx = tid; idx < cnt * v4; idx += SCAN_THREADS) {
                const int tt = idx / v4, c = (idx - tt * v4) * 4;
                const bool ok = col0 + c < Dv;
                mma::cp_async16((uint32_t)__cvta_generic_to_shared(vs + tt * CT + c),
                                vn + ((row0 + t0 + tt) * H + h) * Dv + (ok ? col0 + c : 0), ok);
            }
            if (tid < cnt) {
                const long long row = row0 + t0 + tid;
                cp_async4((uint32_t)__cvta_generic_to_shared(bs + tid), beta + row * ld_b + b_off + h);
                if (!per_channel) cp_async4((uint32_t)__cvta_generic_to_shared(gh + tid), gate + row * ld_a + a_off + h);
            }
        } else {
            for (int idx = tid; idx < cnt * Dpad; idx += SCAN_THREADS) {
                const int tt = idx / Dpad, i = idx - tt * Dpad;
                const long long row = row0 + t0 + tt;
                float kv = 0.f, qv = 0.f, gv = 1.f;
                if (i < D) {
                    kv = kn[(row * G + kvh) * D + i];
                    qv = qn[(row * G + kvh) * D + i];
                    if (per_channel) gv = gate[row * ld_a + a_off + (long long)h * D + i];
                }
                const int at = tt * DS + (i / NPT) * PITCH + (i % NPT);
                ks[at] = kv;
                qs[at] = qv;
                if (per_channel) gs[at] = gv;
            }
            for (int idx = tid; idx < cnt * CT; idx += SCAN_THREADS) {
                const int tt = idx / CT, c = idx - tt * CT;
                vs[idx] = col0 + c < Dv ? vn[((row0 + t0 + tt) * H + h) * Dv + col0 + c] : 0.f;
            }
            if (tid < cnt) {
                const long long row = row0 + t0 + tid;
                bs[tid] = beta[row * ld_b + b_off + h];
                if (!per_channel) gh[tid] = gate[row * ld_a + a_off + h];
            }
        }
        mma::cp_async_commit();
    };
    fetch(0, 0);
    int buf = 0;
    for (int t0 = 0; t0 < n; t0 += TS, buf ^= 1) {
        const int cnt = min(TS, n - t0);
        if (t0 + TS < n) {
            fetch(t0 + TS, buf ^ 1);                   // the other buffer was released by the barrier that ended the last round
            mma::cp_async_wait<1>();
        } else {
            mma::cp_async_wait<0>();
        }
        __syncthreads();
        const float* ks = smem + buf * per_buf;
        const float* qs = ks + TS * DS;
        const float* gs = qs + TS * DS;
        const float* vs = gs + (per_channel ? TS * DS : 0);
        const float* gh = vs + TS * CT;
        const float* bs = gh + TS;
        for (int tt = warp; tt < cnt; tt += SCAN_THREADS / 32) {
            float d = 0.f;
            for (int i = lane; i < Dpad; i += 32) {
                const int at = tt * DS + (i / NPT) * PITCH + (i % NPT);
                d = fmaf(ks[at], qs[at], d);
            }
            d = warp_sum(d);
            if (lane == 0) kq[tt] = d;
        }
        __syncthreads();
        for (int tt = 0; tt < cnt; ++tt) {
            const float4* k4 = reinterpret_cast<const float4*>(ks + tt * DS + r * PITCH);
            const float4* q4 = reinterpret_cast<const float4*>(qs + tt * DS + r * PITCH);
            float kreg[NPT];
            float d1[4] = {0.f, 0.f, 0.f, 0.f}, d2[4] = {0.f, 0.f, 0.f, 0.f};      // four independent chains each
            if (per_channel) {
                const float4* g4 = reinterpret_cast<const float4*>(gs + tt * DS + r * PITCH);
#pragma unroll
                for (int v = 0; v < NPT / 4; ++v) {
                    const float4 kv = k4[v], qv = q4[v], gv = g4[v];
                    kreg[4 * v] = kv.x, kreg[4 * v + 1] = kv.y, kreg[4 * v + 2] = kv.z, kreg[4 * v + 3] = kv.w;
                    s[4 * v] *= gv.x, s[4 * v + 1] *= gv.y, s[4 * v + 2] *= gv.z, s[4 * v + 3] *= gv.w;
                    d1[0] = fmaf(s[4 * v], kv.x, d1[0]), d1[1] = fmaf(s[4 * v + 1], kv.y, d1[1]);
                    d1[2] = fmaf(s[4 * v + 2], kv.z, d1[2]), d1[3] = fmaf(s[4 * v + 3], kv.w, d1[3]);
                    d2[0] = fmaf(s[4 * v], qv.x, d2[0]), d2[1] = fmaf(s[4 * v + 1], qv.y, d2[1]);
                    d2[2] = fmaf(s[4 * v + 2], qv.z, d2[2]), d2[3] = fmaf(s[4 * v + 3], qv.w, d2[3]);
                }
            } else {
                const float g = gh[tt];
#pragma unroll
                for (int v = 0; v < NPT / 4; ++v) {
                    const float4 kv = k4[v], qv = q4[v];
                    kreg[4 * v] = kv.x, kreg[4 * v + 1] = kv.y, kreg[4 * v + 2] = kv.z, kreg[4 * v + 3] = kv.w;
                    s[4 * v] *= g, s[4 * v + 1] *= g, s[4 * v + 2] *= g, s[4 * v + 3] *= g;
                    d1[0] = fmaf(s[4 * v], kv.x, d1[0]), d1[1] = fmaf(s[4 * v + 1], kv.y, d1[1]);
                    d1[2] = fmaf(s[4 * v + 2], kv.z, d1[2]), d1[3] = fmaf(s[4 * v + 3], kv.w, d1[3]);
                    d2[0] = fmaf(s[4 * v], qv.x, d2[0]), d2[1] = fmaf(s[4 * v + 1], qv.y, d2[1]);
                    d2[2] = fmaf(s[4 * v + 2], qv.z, d2[2]), d2[3] = fmaf(s[4 * v + 3], qv.w, d2[3]);
                }
            }
            float e1 = (d1[0] + d1[1]) + (d1[2] + d1[3]), e2 = (d2[0] + d2[1]) + (d2[2] + d2[3]);
            for (int off = cpw; off < 32; off <<= 1) {
                e1 += __shfl_xor_sync(0xffffffffu, e1, off);
                e2 += __shfl_xor_sync(0xffffffffu, e2, off);
            }
            const float u = bs[tt] * (vs[tt * CT + warp * cpw + cl] - e1);
#pragma unroll
            for (int ii = 0; ii < NPT; ++ii) s[ii] = fmaf(kreg[ii], u, s[ii]);
            if (r == 0 && col < Dv) orow[(long long)(t0 + tt) * H * Dv + col] = fmaf(u, kq[tt], e2);
        }
        __syncthreads();                               // everyone is done with this buffer and with kq
    }
    if (col < Dv) {
#pragma unroll
        for (int ii = 0; ii < NPT; ++ii) {
            const int i = r * NPT + ii;
            if (i < D) Sb[(long long)i * Dv + col] = s[ii];
        }
    }
}

template <int NPT>
int launch_scan(const float* qn, const float* kn, const float* vn, const float* gate, long long ld_a, int a_off,
                const float* beta, long long ld_b, int b_off, float* S, float* out, const int* q_start, const int* n_new,
                const int* seq_ids, int B, int Tn, int H, int G, int D, int Dv, int per_channel, int R, cudaStream_t st) {
    const int DS = R * (NPT + 4), CT = SCAN_THREADS / R;
    int TS = SCAN_TS;                                  // tokens per block: fewer for very wide keys (shared memory)
    auto bytes = [&](int ts) {
        return (size_t)(2 * (ts * DS * (per_channel ? 3 : 2) + ts * CT + 2 * ts) + ts) * sizeof(float);
    };
    while (TS > 1 && bytes(TS) > 100 * 1024) TS >>= 1;
    const size_t smem = bytes(TS);
    auto al = [](const void* p) { return ((uintptr_t)p % 16) == 0; };
    const bool async = D % 4 == 0 && Dv % 4 == 0 && CT % 4 == 0 && al(qn) && al(kn) && al(vn) &&
                       (!per_channel || (ld_a % 4 == 0 && a_off % 4 == 0 && al(gate)));
    dim3 grid((Dv + CT - 1) / CT, H, B);
#define NXD_LAUNCH_SCAN(A)                                                                                               \
    do {                                                                                                                 \
        auto kern = delta_scan_kernel<NPT, A>;                                                                           \
        if (smem > 32 * 1024)                                                                                            \
            NXD_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));          \
        kern<<<grid, SCAN_THREADS, smem, st>>>(qn, kn, vn, gate, ld_a, a_off, beta, ld_b, b_off, S, out, q_start, n_new,  \
                                               seq_ids, Tn, H, G, D, Dv, per_channel, R, TS);                            \
    } while (0)
    if (async) NXD_LAUNCH_SCAN(true); else NXD_LAUNCH_SCAN(false);
#undef NXD_LAUNCH_SCAN
    NXD_LAUNCH_CHECK();
    return 0;
}

// ---- chunk-wise form (one decay per head) --------------------------------------------------------------------------------
// For a chunk of CH tokens with start state S, Gamma_t the product of the chunk's decays up to t and L[t][s] their product
// over (s, t], the errors u of all tokens solve one triangular system:
//
//   A[t][s] = beta_t L[t][s] (k_t . k_s), s < t;    (I + A) U = diag(beta) (V - diag(Gamma) K S)
//   O = diag(Gamma) Q S + P U,  P[t][s] = L[t][s] (q_t . k_s), s <= t;    S <- Gamma_CH S + (diag(L[CH-1][.]) K)^T U
//
// With M = (I + A)^-1 diag(beta) and R = V - diag(Gamma) K S:  U = M R,  P U = (P M) R.
// (the WY form of Householder products; Yang, Wang, Zhang, Shen, Kim, "Parallelizing Linear Transformers with the Delta Rule
// over Sequence Length").  Decay ratios are products, never quotients or exponentials of sums, so a decay of any size is
// exact to rounding and underflows to the right limit.  delta_chunk_system makes M, P M, Gamma and L[CH-1][.] of every (chunk, head,
// row) in parallel, in fp64; delta_chunks.cu has the rest, on the tensor cores; delta_chunk_scan_fp32 serves where its operand tiles cost
// more than they save (tensor_core_scan).
constexpr int CW_THREADS = 256, DPITCH = CH + 4, CP = CH + 4;

// c [8 x 8] += a [8 x 4] b [4 x 8]: a is row lane / 4, column lane % 4; b row lane % 4, column lane / 4; c row lane / 4, columns
// 2 (lane % 4) and the next
__device__ __forceinline__ void mma_f64(double (&c)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(c[0]), "+d"(c[1])
        : "d"(a), "d"(b));
}

// All in fp64, rounded once at the end.  With neighbouring keys that are nearly parallel and decays near one, P sums errors u that
// cancel: fp32 dot products, an fp32 inverse and P U as two products put 7e-7 into the output where token by token is off by 1.1e-7.
// The entries of P M are small again where that happens, and the output is 1.0e-7 off.  (The state sums rounded u as well and
// can be 1.7 times as far off as token by token: 3.4e-7 against 2.0e-7.)
template <int D>
__global__ void __launch_bounds__(CW_THREADS, 2)
delta_chunk_system_kernel(const float* __restrict__ qn, const float* __restrict__ kn, const float* __restrict__ gate,
                          long long ld_a, int a_off, const float* __restrict__ beta, long long ld_b, int b_off,
                          float* __restrict__ scratch, const int* __restrict__ n_new, int Tn, int chunk0, int H, int G) {
    pdl_wait();
    extern __shared__ __align__(16) float smem[];
    double* Kd = reinterpret_cast<double*>(smem);      // [CH][DPITCH] 64 key channels at a time; then X = (I + A)^-1
    double* Qd = Kd + CH * DPITCH;                     // [CH][DPITCH] the same of the queries; then P
    double* Ad = Qd + CH * DPITCH;                     // [CH][DPITCH] L; then A
    __shared__ float gs[CH], bs[CH];
    const int c = chunk0 + blockIdx.x, h = blockIdx.y, b = blockIdx.z, kvh = h / (H / G), tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5, lr = lane >> 2, lc = lane & 3;
    const int n = n_new != nullptr ? min(n_new[b], Tn) : Tn;
    const int nt = min(CH, n - c * CH);  // real tokens; the others change nothing (k = q = 0, beta = 0, g = 1)
    if (nt <= 0) return;                 // the scan does not look at this chunk
    const long long row0 = (long long)b * Tn + c * CH;
    float* out = scratch + (((long long)b * H + h) * gridDim.x + blockIdx.x) * CHUNK_FLOATS;
    // keys and queries of 64 channels on their way: the first ones while the decays are multiplied up, the others behind the products
    float4 kv[4], qv[4];
    auto fetch = [&](int d0) {
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            const int i = tid + x * CW_THREADS, t = i >> 4, d = (i & 15) * 4;
            const long long src = ((row0 + min(t, nt - 1)) * G + kvh) * D + d0 + d;
            kv[x] = *reinterpret_cast<const float4*>(kn + src), qv[x] = *reinterpret_cast<const float4*>(qn + src);
            if (t >= nt) kv[x] = qv[x] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    fetch(0);
    if (tid < CH) {
        gs[tid] = tid < nt ? gate[(row0 + tid) * ld_a + a_off + h] : 1.f;
        bs[tid] = tid < nt ? beta[(row0 + tid) * ld_b + b_off + h] : 0.f;
    }
    __syncthreads();
    if (tid <= CH) {                     // column s = tid of L: running products of the decays behind s; the last thread: Gamma
        const int s = tid < CH ? tid : -1;
        double l = 1.;
        for (int t = s + 1; t < CH; ++t) {
            l *= gs[t];
            if (s < 0) out[2 * CH * CH + t] = (float)l;
            else Ad[t * DPITCH + s] = l;
        }
        if (s >= 0) {
            Ad[s * DPITCH + s] = 1.;
            out[2 * CH * CH + CH + s] = (float)l;
        }
    }
    // eight rows of K and of Q per warp against the keys up to them (the sub-partitions' two warps: 2 x 9 tiles each)
    const int rt = warp < 4 ? warp : 11 - warp;
    double kk[8][2] = {}, qk[8][2] = {};
    for (int d0 = 0; d0 < D; d0 += 64) {
        __syncthreads();
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            const int i = tid + x * CW_THREADS, t = i >> 4, d = (i & 15) * 4;
            double2* kd = reinterpret_cast<double2*>(Kd + t * DPITCH + d);
            double2* qd = reinterpret_cast<double2*>(Qd + t * DPITCH + d);
            kd[0] = make_double2(kv[x].x, kv[x].y), kd[1] = make_double2(kv[x].z, kv[x].w);
            qd[0] = make_double2(qv[x].x, qv[x].y), qd[1] = make_double2(qv[x].z, qv[x].w);
        }
        if (d0 + 64 < D) fetch(d0 + 64);
        __syncthreads();
#pragma unroll 1
        for (int d = 0; d < 64; d += 4) {
            const double ka = Kd[(rt * 8 + lr) * DPITCH + d + lc], qa = Qd[(rt * 8 + lr) * DPITCH + d + lc];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (j > rt) break;
                const double kb = Kd[(j * 8 + lr) * DPITCH + d + lc];
                mma_f64(kk[j], ka, kb);
                mma_f64(qk[j], qa, kb);
            }
        }
    }
    __syncthreads();                     // keys and queries have been read: their places take X and P
    {
        const int t = rt * 8 + lr;
        const double bt = bs[t];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (j > rt) break;
#pragma unroll
            for (int x = 0; x < 2; ++x) {              // entries above the diagonal are never read
                const int at = t * DPITCH + j * 8 + 2 * lc + x;
                const double l = Ad[at];
                Qd[at] = l * qk[j][x];
                Ad[at] = bt * l * kk[j][x];
            }
        }
    }
    __syncthreads();
    // Eight columns of X and of P M per warp, eight rows at a time: matrix instructions for the blocks left of the diagonal one,
    // single steps inside it that leave out what lies above the diagonal instead of multiplying it by zero (a token that is not a
    // number does not reach the tokens before it).
    const int c0 = warp * 8 + 2 * lc;
    const double b0 = bs[c0], b1 = bs[c0 + 1];
    auto put = [&](float* dst, int i, double v0, double v1) {
        const int t = i * 8 + lr;
        *reinterpret_cast<float2*>(dst + t * CH + c0) = make_float2(c0 <= t ? (float)(v0 * b0) : 0.f, c0 < t ? (float)(v1 * b1) : 0.f);
    };
    for (int i = 0; i < warp; ++i) {
        put(out, i, 0., 0.);
        put(out + CH * CH, i, 0., 0.);
    }
    for (int i = warp; i < 8; ++i) {
        double v[2] = {}, y[2] = {};
        for (int s = warp * 8; s < i * 8; s += 4) {
            const double xb = Kd[(s + lc) * DPITCH + warp * 8 + lr];
            mma_f64(v, Ad[(i * 8 + lr) * DPITCH + s + lc], xb);
            mma_f64(y, Qd[(i * 8 + lr) * DPITCH + s + lc], xb);
        }
        v[0] = (i == warp && lr == 2 * lc ? 1. : 0.) - v[0];
        v[1] = (i == warp && lr == 2 * lc + 1 ? 1. : 0.) - v[1];
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const double x0 = __shfl_sync(0xffffffffu, v[0], r * 4 + lc), x1 = __shfl_sync(0xffffffffu, v[1], r * 4 + lc);
            const int at = (i * 8 + lr) * DPITCH + i * 8 + r;
            if (lr > r) {
                const double a = Ad[at];
                v[0] -= a * x0;
                v[1] -= a * x1;
            }
            if (lr >= r) {
                const double p = Qd[at];
                y[0] += p * x0;
                y[1] += p * x1;
            }
        }
        *reinterpret_cast<double2*>(Kd + (i * 8 + lr) * DPITCH + c0) = make_double2(v[0], v[1]);
        __syncwarp();
        put(out, i, v[0], v[1]);
        put(out + CH * CH, i, y[0], y[1]);
    }
    pdl_trigger();
}

// The rest in fp32, per (32 value columns, head, row), sequential over chunks with the state slice in shared memory: four products per
// chunk, register-tiled, on packed pairs of fp32 multiply-adds (pairs run along the contraction, so both operands are read as 16-byte
// pieces and nothing is shuffled).  Bound by the fp32 pipes and the chain of a chunk's phases (11 us of 128 x 256 alone on an SM).
__device__ __forceinline__ ulonglong2 ld_pairs(const float* p) { return *reinterpret_cast<const ulonglong2*>(p); }

// acc[i][j] += <a row i, b row j> over 4 values
template <int R, int C>
__device__ __forceinline__ void dot_step(uint64_t (&acc)[R][C], const ulonglong2 (&a)[R], const ulonglong2 (&b)[C]) {
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j < C; ++j) acc[i][j] = f2_fma(a[i].y, b[j].y, f2_fma(a[i].x, b[j].x, acc[i][j]));
}

template <int R, int C>
__device__ __forceinline__ void add_pairs(uint64_t (&acc)[R][C], const uint64_t (&part)[R][C]) {
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j < C; ++j) asm("add.rn.f32x2 %0, %0, %1;" : "+l"(acc[i][j]) : "l"(part[i][j]));
}

// grid (Dv / 32, H, B).  Rows of a thread in the 64-row products: 4 w + rg and 60 - 4 w + rg (w the warp, rg = lane / 8), so
// that the triangular products cost every warp the same; columns cg + 8 i (cg = lane % 8).
template <int D>
__global__ void __launch_bounds__(CW_THREADS, D == 64 ? 2 : 1)
delta_chunk_scan_fp32_kernel(const float* __restrict__ qn, const float* __restrict__ kn, const float* __restrict__ vn,
                             const float* __restrict__ scratch, float* __restrict__ S, float* __restrict__ out,
                             const int* __restrict__ q_start, const int* __restrict__ n_new, const int* __restrict__ seq_ids, int Tn,
                             int NC, int H, int G, int Dv) {
    extern __shared__ __align__(16) float smem[];
    constexpr int DP = D + 4, DT = D / 32, KB = D <= 128 ? 2 : 1;     // KB: buffers of K
    float* Kb = smem;                          // [KB][CH][DP]
    float* Qs = Kb + KB * CH * DP;             // [CH][DP]
    float* Ss = Qs + CH * DP;                  // [32][DP] the state slice, a value column per row
    float* Ms = Ss + CW_COLS * DP;             // [CH][CP]
    float* Ps = Ms + CH * CP;                  // [CH][CP] P M
    float* Rs = Ps + CH * CP;                  // [32][CP] V - diag(Gamma) K S, a value column per row
    float* Us = Rs + CW_COLS * CP;             // [32][CP] U
    float* gam2 = Us + CW_COLS * CP;           // [2][2 CH] Gamma and L[CH-1][.] of this chunk and the next
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int col0 = blockIdx.x * CW_COLS, h = blockIdx.y, b = blockIdx.z, kvh = h / (H / G);
    const int n = n_new != nullptr ? min(n_new[b], Tn) : Tn;
    const long long row0 = (long long)b * Tn;
    float* orow = out + (row0 * H + h) * Dv + col0;              // + t * H * Dv
    for (int i = tid; i < (Tn - max(n, 0)) * CW_COLS; i += CW_THREADS)       // padding rows
        orow[(long long)(max(n, 0) + i / CW_COLS) * H * Dv + i % CW_COLS] = 0.f;
    if (n <= 0) return;
    const int line = seq_ids != nullptr ? seq_ids[b] : b;
    float* Sb = S + ((long long)line * H + h) * D * Dv + col0;
    const bool fresh = q_start[b] == 0;
    for (int i = tid; i < D * CW_COLS; i += CW_THREADS) {
        const int d = i / CW_COLS, j = i % CW_COLS;
        Ss[j * DP + d] = fresh ? 0.f : Sb[(long long)d * Dv + j];
    }
    const float* chunk0 = scratch + ((long long)b * H + h) * NC * CHUNK_FLOATS;
    const int chunks = (n + CH - 1) / CH;
    auto rows = [&](const float* src, float* dst, int c) {       // K or Q rows of chunk c
        if (c < chunks)
            for (int i = tid; i < CH * (D / 4); i += CW_THREADS) {
                const int t = i / (D / 4), d = (i % (D / 4)) * 4;
                const bool ok = c * CH + t < n;
                mma::cp_async16((uint32_t)__cvta_generic_to_shared(dst + t * DP + d),
                                src + ((row0 + (ok ? c * CH + t : 0)) * G + kvh) * D + d, ok);
            }
    };
    auto square = [&](int off, float* dst, int c) {              // M or P of chunk c
        if (c < chunks)
            for (int i = tid; i < CH * (CH / 4); i += CW_THREADS) {
                const int t = i / (CH / 4), x = (i % (CH / 4)) * 4;
                mma::cp_async16((uint32_t)__cvta_generic_to_shared(dst + t * CP + x),
                                chunk0 + (long long)c * CHUNK_FLOATS + off + t * CH + x, true);
            }
    };
    auto factors = [&](int c) {                                  // Gamma and L[CH-1][.] of chunk c
        if (c < chunks && tid < 2 * CH / 4)
            mma::cp_async16((uint32_t)__cvta_generic_to_shared(gam2 + (c & 1) * 2 * CH + tid * 4),
                            chunk0 + (long long)c * CHUNK_FLOATS + 2 * CH * CH + tid * 4, true);
    };
    rows(kn, Kb, 0);
    rows(qn, Qs, 0);
    square(0, Ms, 0);
    factors(0);
    mma::cp_async_commit();
    square(CH * CH, Ps, 0);
    mma::cp_async_commit();
    const int rg = lane >> 3, cg = lane & 7, ra = 4 * warp + rg, rb = 60 - 4 * warp + rg;
    for (int c = 0; c < chunks; ++c) {
        const float* Ks = Kb + (KB == 2 ? (c & 1) * CH * DP : 0);
        const int t0 = c * CH;
        const float *gam = gam2 + (c & 1) * 2 * CH, *last = gam + CH;
        float v[2][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            v[0][i] = t0 + ra < n ? vn[((row0 + t0 + ra) * H + h) * Dv + col0 + cg + 8 * i] : 0.f;
            v[1][i] = t0 + rb < n ? vn[((row0 + t0 + rb) * H + h) * Dv + col0 + cg + 8 * i] : 0.f;
        }
        mma::cp_async_wait<1>();               // everything but P
        __syncthreads();
        if (KB == 2) {
            rows(kn, Kb + ((c + 1) & 1) * CH * DP, c + 1);
            mma::cp_async_commit();
        }
        uint64_t acc[4][4] = {};               // K S of rows ra, rb; Q S of rows ra, rb
#pragma unroll 1
        for (int d0 = 0; d0 < D; d0 += 16) {   // sums of 16 first: half the rounding error of one long chain
            uint64_t part[4][4] = {};
#pragma unroll
            for (int d = d0; d < d0 + 16; d += 4) {
                const ulonglong2 a[4] = {ld_pairs(Ks + ra * DP + d), ld_pairs(Ks + rb * DP + d), ld_pairs(Qs + ra * DP + d),
                                         ld_pairs(Qs + rb * DP + d)};
                ulonglong2 sb[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) sb[j] = ld_pairs(Ss + (cg + 8 * j) * DP + d);
                dot_step(part, a, sb);
            }
            add_pairs(acc, part);
        }
        const float ga = gam[ra], gb = gam[rb];
        float o[2][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            Rs[(cg + 8 * i) * CP + ra] = fmaf(-ga, f2_lo(acc[0][i]) + f2_hi(acc[0][i]), v[0][i]);
            Rs[(cg + 8 * i) * CP + rb] = fmaf(-gb, f2_lo(acc[1][i]) + f2_hi(acc[1][i]), v[1][i]);
            o[0][i] = ga * (f2_lo(acc[2][i]) + f2_hi(acc[2][i]));
            o[1][i] = gb * (f2_lo(acc[3][i]) + f2_hi(acc[3][i]));
        }
        __syncthreads();
        rows(qn, Qs, c + 1);                   // the queries of this chunk have been used
        mma::cp_async_commit();
        // rows ra and rb of a lower triangular 64 x 64 matrix times the columns of X [32][CP]
        auto triangular = [&](const float* M, const float* X, uint64_t (&y)[2][4]) {
            const int e = 4 * warp, f = 60 - 4 * warp;           // the blocks of the diagonal: [e, e + 4) and [f, f + 4)
#pragma unroll 1
            for (int s0 = 0; s0 < f; s0 += 16) {                 // sums of 16 first, as above
                uint64_t part[2][4] = {};
#pragma unroll
                for (int s = s0; s < s0 + 16; s += 4) {
                    if (s >= f) break;
                    const ulonglong2 a = ld_pairs(M + rb * CP + s);
                    ulonglong2 xb[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        xb[j] = ld_pairs(X + (cg + 8 * j) * CP + s);
                        part[1][j] = f2_fma(a.y, xb[j].y, f2_fma(a.x, xb[j].x, part[1][j]));
                    }
                    if (s >= e) continue;
                    const ulonglong2 c = ld_pairs(M + ra * CP + s);
#pragma unroll
                    for (int j = 0; j < 4; ++j) part[0][j] = f2_fma(c.y, xb[j].y, f2_fma(c.x, xb[j].x, part[0][j]));
                }
                add_pairs(y, part);
            }
            // on the diagonal the entries behind the row's own are left out, not multiplied by zero: a token that is not a
            // number does not reach the tokens before it
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int row = half ? rb : ra, s = half ? f : e;
                const float4 m = *reinterpret_cast<const float4*>(M + row * CP + s);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float4 x = *reinterpret_cast<const float4*>(X + (cg + 8 * j) * CP + s);
                    float d = m.x * x.x;
                    if (rg >= 1) d = fmaf(m.y, x.y, d);
                    if (rg >= 2) d = fmaf(m.z, x.z, d);
                    if (rg >= 3) d = fmaf(m.w, x.w, d);
                    y[half][j] = f2_pack(f2_lo(y[half][j]) + d, f2_hi(y[half][j]));
                }
            }
        };
        uint64_t y[2][4] = {};
        triangular(Ms, Rs, y);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            Us[(cg + 8 * i) * CP + ra] = f2_lo(y[0][i]) + f2_hi(y[0][i]);
            Us[(cg + 8 * i) * CP + rb] = f2_lo(y[1][i]) + f2_hi(y[1][i]);
        }
        mma::cp_async_wait<KB>();              // P of this chunk (the groups behind it: Q and, with two buffers, K)
        __syncthreads();
        square(0, Ms, c + 1);
        factors(c + 1);
        mma::cp_async_commit();
#pragma unroll
        for (int i = 0; i < 4; ++i) y[0][i] = y[1][i] = 0ull;
        triangular(Ps, Rs, y);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (t0 + ra < n) orow[(long long)(t0 + ra) * H * Dv + cg + 8 * i] = o[0][i] + (f2_lo(y[0][i]) + f2_hi(y[0][i]));
            if (t0 + rb < n) orow[(long long)(t0 + rb) * H * Dv + cg + 8 * i] = o[1][i] + (f2_lo(y[1][i]) + f2_hi(y[1][i]));
        }
        // S[.][j] <- Gamma S + sum_s last_s U[s][j] K[s][.]: DT key channels x 4 value columns per thread
        {
            const int d0 = ((warp & 3) * 8 + cg) * DT, j0 = (warp >> 2) * 16 + rg;       // columns j0 + 4 i
            const uint64_t gl = f2_pack(gam[CH - 1], gam[CH - 1]);
            uint64_t st[4][DT / 2] = {};       // the chunk's own part; the decayed state joins it once
#pragma unroll 1
            for (int s0 = 0; s0 < CH; s0 += 16) {
                uint64_t part[4][DT / 2] = {};
#pragma unroll 2
                for (int s = s0; s < s0 + 16; s += 4) {
                    float u[4][4], lw[4];
                    *reinterpret_cast<float4*>(lw) = *reinterpret_cast<const float4*>(last + s);
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        *reinterpret_cast<float4*>(u[i]) = *reinterpret_cast<const float4*>(Us + (j0 + 4 * i) * CP + s);
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        uint64_t kv[DT / 2];
#pragma unroll
                        for (int x = 0; x < DT / 2; ++x)
                            kv[x] = *reinterpret_cast<const uint64_t*>(Ks + (s + q) * DP + d0 + 2 * x);
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const float w = u[i][q] * lw[q];
                            const uint64_t ww = f2_pack(w, w);
#pragma unroll
                            for (int x = 0; x < DT / 2; ++x) part[i][x] = f2_fma(kv[x], ww, part[i][x]);
                        }
                    }
                }
                add_pairs(st, part);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int x = 0; x < DT / 2; ++x) {
                    uint64_t* at = reinterpret_cast<uint64_t*>(Ss + (j0 + 4 * i) * DP + d0 + 2 * x);
                    *at = f2_fma(*at, gl, st[i][x]);
                }
        }
        __syncthreads();                       // K, P, U and the old state are free
        if (KB == 1) rows(kn, Kb, c + 1);
        mma::cp_async_commit();
        square(CH * CH, Ps, c + 1);
        mma::cp_async_commit();
    }
    for (int i = tid; i < D * CW_COLS; i += CW_THREADS) {
        const int d = i / CW_COLS, j = i % CW_COLS;
        Sb[(long long)d * Dv + j] = Ss[j * DP + d];
    }
}

// The tensor-core scan reads operand tiles (147 to 344 KB) that another kernel writes per (row, head, chunk); with one or two slices of 32
// value columns and enough (row, head) pairs to fill the chip they cost more than its short chain saves.  Tensor cores / fp32, us, 1024
// tokens:  one slice, 64 and 128 channels, 64 pairs 181 / 207 and 235 / 279, 96 247 / 246 and 330 / 332, 256 612 / 484 and 852 / 732;
// two slices of 64 channels, 256 pairs 683 / 692, 512 1340 / 1266, and 192 tokens, 96 pairs 64 / 69, 128 88 / 80, 384 213 / 207 (320
// tokens 333 / 335).  Two slices of 128 channels, 512 pairs 1826 / 1959.  One slice of 256 channels crosses at 96 too (128 pairs 764 /
// 613, 512 1515 / 1214 at 512 tokens), but up to 256 pairs a row is to come out the same alone and among others.
bool tensor_core_scan(int B, int Tn, int H, int D, int Dv) {
    const long long pairs = (long long)B * H;
    if (Dv == CW_COLS) return pairs < (D == 256 ? 257 : 96);
    if (Dv == 2 * CW_COLS && D == 64) return pairs < (Tn <= 5 * CH ? 128 : 512);
    return true;
}

// What is worked on at once: rows of the batch and chunks of them, whose operand tiles (147 to 344 KB per row, head and chunk; the systems
// take 33 KB more) are half a gigabyte at most, or one chunk of one row.  Longer steps and larger batches run in several launches.  A
// launch takes six chunks if it can and fewer rows for it: a block of the scan sets up and moves its state for one chunk as for many (64
// rows of 1024 tokens, 32 heads of 256 x 256, chunk by chunk 27.1 ms, by four 20.4, by six to eight 19.5; 8 rows of 421 tokens, 32 heads
// of 256 x 128, four rows with all chunks 898 us, all rows with six 868).
struct Segment {
    int rows, chunks;
};

Segment segment(int B, int Tn, int H, int D) {
    const int NC = (Tn + CH - 1) / CH;
    const long long fit = max(1ll, (512ll << 20) / ((long long)H * nxd_delta::chunk_tiles(D) * nxd_delta::TILE_BYTES));
    const int parts = (int)min((long long)B, ((long long)B * min(NC, 6) + fit - 1) / fit), rows = (B + parts - 1) / parts;
    return {rows, (int)max(1ll, min((long long)NC, fit / rows))};
}

template <int D>
int launch_chunks(const nxd_delta::Step& p, const float* gate, long long ld_a, int a_off, const float* beta, long long ld_b, int b_off,
                  float* scratch, bool tensor_cores, long long wait_clocks, cudaStream_t st) {
    const int NC = (p.Tn + CH - 1) / CH;
    const size_t smem = (size_t)3 * CH * DPITCH * sizeof(double);
    NXD_CHECK_CUDA(nxd_allow_smem<delta_chunk_system_kernel<D>>((int)smem));
    if (!tensor_cores) {
        constexpr int DP = D + 4;
        constexpr int scan = ((D <= 128 ? 3 : 2) * CH * DP + CW_COLS * DP + 2 * CH * CP + 2 * CW_COLS * CP + 4 * CH) * (int)sizeof(float);
        static_assert(scan <= 232448, "shared memory");
        NXD_CHECK_CUDA(nxd_allow_smem<delta_chunk_scan_fp32_kernel<D>>(scan));
        NXD_CHECK_CUDA((nxd_launch_pdl(delta_chunk_system_kernel<D>, dim3(NC, p.H, p.B), dim3(CW_THREADS), smem, st, p.qn, p.kn,
            gate, ld_a, a_off, beta, ld_b, b_off, scratch, p.n_new, p.Tn, 0, p.H, p.G)));
        NXD_LAUNCH_CHECK();
        delta_chunk_scan_fp32_kernel<D><<<dim3(p.Dv / CW_COLS, p.H, p.B), CW_THREADS, scan, st>>>(
            p.qn, p.kn, p.vn, scratch, p.S, p.out, p.q_start, p.n_new, p.seq_ids, p.Tn, NC, p.H, p.G, p.Dv);
        NXD_LAUNCH_CHECK();
        return 0;
    }
    const Segment seg = segment(p.B, p.Tn, p.H, D);
    uint8_t* tiles = reinterpret_cast<uint8_t*>(scratch);
    float* systems = scratch + (long long)seg.rows * p.H * seg.chunks * (nxd_delta::chunk_tiles(D) * nxd_delta::TILE_BYTES / 4);
    for (int b0 = 0; b0 < p.B; b0 += seg.rows) {
        nxd_delta::Step r = p;
        const long long t0 = (long long)b0 * p.Tn;
        r.B = min(seg.rows, p.B - b0);
        r.qn += t0 * p.G * D, r.kn += t0 * p.G * D, r.vn += t0 * p.H * p.Dv, r.out += t0 * p.H * p.Dv, r.q_start += b0;
        if (p.n_new != nullptr) r.n_new += b0;
        if (p.seq_ids != nullptr) r.seq_ids += b0;
        else r.S += (long long)b0 * p.H * D * p.Dv;
        for (int c0 = 0; c0 < NC; c0 += seg.chunks) {
            const int count = min(seg.chunks, NC - c0);
            NXD_CHECK_CUDA((nxd_launch_pdl(delta_chunk_system_kernel<D>, dim3(count, p.H, r.B), dim3(CW_THREADS), smem, st, r.qn,
                r.kn, gate + t0 * ld_a, ld_a, a_off, beta + t0 * ld_b, ld_b, b_off, systems, r.n_new, p.Tn, c0, p.H, p.G)));
            NXD_LAUNCH_CHECK();
            if (int rc = nxd_delta::launch_chunks_tc(r, systems, tiles, c0, count, wait_clocks, st)) return rc;
        }
    }
    return 0;
}

}  // namespace

// dtype of proj: 0 bf16, 1 fp32.  proj [B * Tn, ld]: raw q (G * D channels) at column off_q, k (G * D) at off_k, v
// (H * Dv) at off_v.  conv_w fp32 [2 G D + H Dv, taps] in q | k | v order, last column = the current token.  conv_state fp32
// [lines, taps - 1, C]: the last raw projections of every line (read here, moved on by nxd_delta_conv_state).
// qn, kn [B * Tn, G, D], vn [B * Tn, H, Dv] fp32: silu(conv), queries and keys divided by sqrt(sum x^2 + unit_eps), queries
// times qscale.  q_start [B], n_new [B] or NULL, seq_ids [B] or NULL as in the attention entry points.
NXD_API int nxd_delta_prep(int dtype, const void* proj, long long ld, int off_q, int off_k, int off_v, const float* conv_w,
                           const float* conv_state, float* qn, float* kn, float* vn, const int* q_start, const int* n_new,
                           const int* seq_ids, int B, int Tn, int H, int G, int D, int Dv, int taps, float qscale,
                           float unit_eps, void* stream) {
    const long long units = (long long)B * Tn * (2 * G + H);
    if (units == 0) return 0;
    NXD_REQUIRE(taps >= 1 && taps <= MAX_TAPS, "short convolution with %d taps", taps);
    const int wpb = 8;
    const unsigned blocks = (unsigned)((units + wpb - 1) / wpb);
    cudaStream_t st = (cudaStream_t)stream;
    {   // strips: V channels per lane, all rows and offsets multiples of V values, results and taps aligned
        const int V = D / 32;
        auto al = [](const void* p, size_t n) { return ((uintptr_t)p % n) == 0; };
        if (taps == 4 && (D == 64 || D == 128 || D == 256) && Dv % D == 0 && ld % V == 0 && off_q % V == 0 && off_k % V == 0 &&
            off_v % V == 0 && al(proj, 16) && al(conv_w, 16) && al(qn, 16) && al(kn, 16) && al(vn, 16) && B < 65536 &&
            (Tn + PREP_SHORT - 1) / PREP_SHORT < 65536) {
#define NXD_STRIP(T, V_)                                                                                                   \
    return launch_prep_strip<T, V_>(proj, ld, off_q, off_k, off_v, conv_w, conv_state, qn, kn, vn, q_start, n_new, seq_ids, B, \
                                    Tn, H, G, Dv, qscale, unit_eps, st)
            if (dtype == 0) {
                if (V == 2) NXD_STRIP(bf16, 2);
                if (V == 4) NXD_STRIP(bf16, 4);
                NXD_STRIP(bf16, 8);
            }
            if (V == 2) NXD_STRIP(float, 2);
            if (V == 4) NXD_STRIP(float, 4);
            NXD_STRIP(float, 8);
#undef NXD_STRIP
        }
    }
    if (dtype == 0)
        delta_prep_kernel<bf16><<<blocks, wpb * 32, 0, st>>>((const bf16*)proj, ld, off_q, off_k, off_v, conv_w, conv_state, qn,
                                                            kn, vn, q_start, n_new, seq_ids, units, Tn, H, G, D, Dv, taps,
                                                            qscale, unit_eps);
    else
        delta_prep_kernel<float><<<blocks, wpb * 32, 0, st>>>((const float*)proj, ld, off_q, off_k, off_v, conv_w, conv_state,
                                                             qn, kn, vn, q_start, n_new, seq_ids, units, Tn, H, G, D, Dv,
                                                             taps, qscale, unit_eps);
    NXD_LAUNCH_CHECK();
    return 0;
}

// After nxd_delta_prep of the same step: slot s of the line's state <- raw projection of position end - (taps - 1) + s,
// end = q_start + n_new (zeros before the start of the sequence).  Rows without real tokens keep their state.
NXD_API int nxd_delta_conv_state(int dtype, const void* proj, long long ld, int off_q, int off_k, int off_v,
                                 float* conv_state, const int* q_start, const int* n_new, const int* seq_ids, int B, int Tn,
                                 int H, int G, int D, int Dv, int taps, void* stream) {
    const int C = 2 * G * D + H * Dv;
    if ((long long)B * C == 0 || taps <= 1) return 0;
    NXD_REQUIRE(taps <= MAX_TAPS, "short convolution with %d taps", taps);
    const unsigned blocks = (unsigned)(((long long)B * C + 255) / 256);
    cudaStream_t st = (cudaStream_t)stream;
    if (dtype == 0)
        NXD_CHECK_CUDA((nxd_launch_pdl(delta_conv_state_kernel<bf16>, dim3(blocks), dim3(256), 0, st, (const bf16*)proj, ld, off_q,
            off_k, off_v, conv_state, q_start, n_new, seq_ids, B, Tn, G * D, C, taps)));
    else
        NXD_CHECK_CUDA((nxd_launch_pdl(delta_conv_state_kernel<float>, dim3(blocks), dim3(256), 0, st, (const float*)proj, ld,
            off_q, off_k, off_v, conv_state, q_start, n_new, seq_ids, B, Tn, G * D, C, taps)));
    NXD_LAUNCH_CHECK();
    return 0;
}

// Floats of scratch with which nxd_delta_scan runs the chunk-wise form, 0 where it does not apply: one decay per head, key
// sizes of 64 / 128 / 256, value sizes in whole slices of 32 columns, steps of at least three chunks.
NXD_API long long nxd_delta_scan_scratch(int B, int Tn, int H, int D, int Dv, int per_channel) {
    if (per_channel || (D != 64 && D != 128 && D != 256) || Dv % CW_COLS != 0 || Tn < 3 * CH || B > 65535 || H > 65535) return 0;
    if (!tensor_core_scan(B, Tn, H, D, Dv)) return (long long)B * H * ((Tn + CH - 1) / CH) * CHUNK_FLOATS;
    const Segment seg = segment(B, Tn, H, D);
    return (long long)seg.rows * H * seg.chunks * (CHUNK_FLOATS + nxd_delta::chunk_tiles(D) * nxd_delta::TILE_BYTES / 4);
}

// qn, kn, vn as written by nxd_delta_prep.  apre fp32 [B * Tn, ld_a]: decay pre-activation of head h at column a_off + h
// (per_channel == 0) or of (h, key channel i) at a_off + h * D + i; dt_bias [H] or [H * D], a_log [H]:
// g = exp(-exp(a_log) softplus(apre + dt_bias)).  bpre fp32 [B * Tn, ld_b]: beta = sigmoid(bpre[b_off + h]).  Both are
// OVERWRITTEN with g and beta (a first kernel, one thread per value; the recurrence then reads them).
// S fp32 [lines, H, D, Dv], updated in place.  out fp32 [B * Tn, H, Dv].  scratch: nxd_delta_scan_scratch floats, or NULL
// (token by token).
// wait_clocks: the clocks after which a wait inside the chunk-wise form gives up (nxd_delta_scan_status), -1: two seconds.
NXD_API int nxd_delta_scan_limited(const float* qn, const float* kn, const float* vn, float* apre, long long ld_a, int a_off,
                                   float* bpre, long long ld_b, int b_off, const float* a_log, const float* dt_bias, float* S,
                                   float* out, const int* q_start, const int* n_new, const int* seq_ids, int B, int Tn, int H, int G,
                                   int D, int Dv, int per_channel, float* scratch, long long wait_clocks, void* stream) {
    if ((long long)B * Tn * H * Dv == 0) return 0;
    NXD_REQUIRE(G > 0 && H % G == 0, "delta rule: %d heads over %d query/key heads", H, G);
    NXD_REQUIRE(D >= 1 && D <= 1024, "delta rule: key size %d", D);
    cudaStream_t st = (cudaStream_t)stream;
    const long long N = (long long)B * Tn;
    const int per_head = per_channel ? D : 1;
    const long long vals = N * ((long long)H * per_head + H);
    NXD_CHECK_CUDA((nxd_launch_pdl(delta_gates_kernel, dim3((unsigned)((vals + 255) / 256)), dim3(256), 0, st, apre, ld_a, a_off,
        bpre, ld_b, b_off, a_log, dt_bias, N, H, per_head)));
    NXD_LAUNCH_CHECK();
    auto al = [](const void* p) { return ((uintptr_t)p % 16) == 0; };
    const long long floats = nxd_delta_scan_scratch(B, Tn, H, D, Dv, per_channel);
    // values, state and outputs at any address run on the fp32 scan, where the scratch holds its systems of all chunks
    const bool tc = tensor_core_scan(B, Tn, H, D, Dv) && al(vn) && al(S) && al(out);
    if (scratch != nullptr && floats > 0 && al(qn) && al(kn) && al(scratch) &&
        (tc || (long long)B * H * ((Tn + CH - 1) / CH) * CHUNK_FLOATS <= floats)) {
        const nxd_delta::Step step{qn, kn, vn, S, out, q_start, n_new, seq_ids, B, Tn, H, G, D, Dv};
        if (D == 64) return launch_chunks<64>(step, apre, ld_a, a_off, bpre, ld_b, b_off, scratch, tc, wait_clocks, st);
        if (D == 128) return launch_chunks<128>(step, apre, ld_a, a_off, bpre, ld_b, b_off, scratch, tc, wait_clocks, st);
        return launch_chunks<256>(step, apre, ld_a, a_off, bpre, ld_b, b_off, scratch, tc, wait_clocks, st);
    }
    // rows of a column per thread (NPT) and lanes per column (R, a power of two): the smallest slice that keeps R <= 4,
    // wider keys spread over more lanes (measured at 8 heads of 256 x 512, 2 x 4096 tokens: slices of 32 / 16 / 8 rows take
    // 4.5 / 7.8 / 13.8 ms -- fewer columns per CTA re-read the keys and queries more often)
    const int npt = D <= 32 ? 8 : (D <= 64 ? 16 : 32);
    int R = 1;
    while (R * npt < D) R <<= 1;
#define NXD_SCAN(N_)                                                                                                     \
    return launch_scan<N_>(qn, kn, vn, apre, ld_a, a_off, bpre, ld_b, b_off, S, out, q_start, n_new, seq_ids, B, Tn, H, G, \
                           D, Dv, per_channel, R, st)
    if (npt == 8) NXD_SCAN(8);
    if (npt == 16) NXD_SCAN(16);
    NXD_SCAN(32);
#undef NXD_SCAN
}

NXD_API int nxd_delta_scan(const float* qn, const float* kn, const float* vn, float* apre, long long ld_a, int a_off,
                           float* bpre, long long ld_b, int b_off, const float* a_log, const float* dt_bias, float* S,
                           float* out, const int* q_start, const int* n_new, const int* seq_ids, int B, int Tn, int H, int G,
                           int D, int Dv, int per_channel, float* scratch, void* stream) {
    return nxd_delta_scan_limited(qn, kn, vn, apre, ld_a, a_off, bpre, ld_b, b_off, a_log, dt_bias, S, out, q_start, n_new, seq_ids, B,
                                  Tn, H, G, D, Dv, per_channel, scratch, -1, stream);
}
