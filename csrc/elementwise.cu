// SwiGLU and RoPE for sm_100a.
//
// SwiGLU: reference examples/training/llama/modeling_llama_nxd.py:197-208 -- the fused
// gate_up projection (ColumnParallel, stride=2) yields [T, 2*I] with the local gate
// chunk first and the local up chunk second; out = silu(gate) * up.
//
// RoPE: reference modeling_llama_nxd.py:398-399 (HF rotate-half) and the inference
// variant examples/inference/modules/attention/utils.py:27-41.  Applied IN PLACE
// on the fused QKV GEMM output viewed as [T, heads_total, D]: the first
// `n_rot_heads` heads (q heads then k heads) are rotated, v heads are untouched.
// Backward is the same kernel with the sine negated (inverse rotation).
#include "common.cuh"

namespace {

__global__ void swiglu_fwd_kernel(const bf16* __restrict__ gu, bf16* __restrict__ out, size_t rows, int I) {
    pdl_trigger();
    pdl_wait();
    const int nvec = I >> 3;
    const size_t total = rows * (size_t)nvec;
    for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (size_t)gridDim.x * blockDim.x) {
        const size_t r = idx / nvec;
        const int c = (int)(idx % nvec);
        const bf16x8* g = reinterpret_cast<const bf16x8*>(gu + r * 2 * (size_t)I);
        const bf16x8* u = reinterpret_cast<const bf16x8*>(gu + r * 2 * (size_t)I + I);
        float gv[8], uv[8], o[8];
        bf16x8 pg = g[c], pu = u[c];
        unpack8(pg, gv);
        unpack8(pu, uv);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const float sg = 1.f / (1.f + __expf(-gv[k]));
            o[k] = gv[k] * sg * uv[k];
        }
        reinterpret_cast<bf16x8*>(out + r * (size_t)I)[c] = pack8(o);
    }
}

__global__ void swiglu_bwd_kernel(const bf16* __restrict__ gu, const bf16* __restrict__ dy,
                                  bf16* __restrict__ dgu, size_t rows, int I) {
    pdl_trigger();
    pdl_wait();
    const int nvec = I >> 3;
    const size_t total = rows * (size_t)nvec;
    for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (size_t)gridDim.x * blockDim.x) {
        const size_t r = idx / nvec;
        const int c = (int)(idx % nvec);
        const bf16x8* g = reinterpret_cast<const bf16x8*>(gu + r * 2 * (size_t)I);
        const bf16x8* u = reinterpret_cast<const bf16x8*>(gu + r * 2 * (size_t)I + I);
        const bf16x8* d = reinterpret_cast<const bf16x8*>(dy + r * (size_t)I);
        float gv[8], uv[8], dv[8], dg[8], du[8];
        bf16x8 pg = g[c], pu = u[c], pd = d[c];
        unpack8(pg, gv);
        unpack8(pu, uv);
        unpack8(pd, dv);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const float sg = 1.f / (1.f + __expf(-gv[k]));
            const float silu = gv[k] * sg;
            dg[k] = dv[k] * uv[k] * sg * (1.f + gv[k] * (1.f - sg));
            du[k] = dv[k] * silu;
        }
        reinterpret_cast<bf16x8*>(dgu + r * 2 * (size_t)I)[c] = pack8(dg);
        reinterpret_cast<bf16x8*>(dgu + r * 2 * (size_t)I + I)[c] = pack8(du);
    }
}

// One thread takes 8 (x1, x2) pairs, columns [8c, 8c+8) and [D/2 + 8c, ...), of kHeads heads of a token: the table entries
// and the position are read once for them and 2 kHeads 16-byte loads are in flight.  Heads from n_rot on are copied
// (n_heads = heads_total, x != y) or left alone (n_heads = n_rot, x == y).  Bound by memory: 8192 tokens x 40 heads of 128, 32 of
// them rotated, 30 us on average for one launch out of place (168 MB) and one in place (134 MB), against 23 us of copy and 31 us of
// rotation each with one head per thread.
template <int kHeads>
__global__ void rope_kernel(const bf16* x, bf16* y, const float* __restrict__ cos_t, const float* __restrict__ sin_t,
                            const int* __restrict__ positions, size_t T, int heads_total, int n_heads, int n_rot, int D,
                            int pos_div, int pos_mod, float sin_sign) {
    pdl_trigger();
    pdl_wait();
    const int half_vec = D >> 4;  // 16-byte vectors in half a head
    const int groups = (n_heads + kHeads - 1) / kHeads;
    const size_t total = T * (size_t)groups * half_vec;
    for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (size_t)gridDim.x * blockDim.x) {
        const int c = (int)(idx % half_vec);
        const size_t tg = idx / half_vec;
        const int h0 = (int)(tg % groups) * kHeads;
        const size_t t = tg / groups;
        const size_t at = (t * heads_total + h0) * (size_t)D + c * 8;
        bf16x8 va[kHeads], vb[kHeads];
#pragma unroll
        for (int j = 0; j < kHeads; ++j) {
            if (h0 + j < n_heads) {
                va[j] = *reinterpret_cast<const bf16x8*>(x + at + (size_t)j * D);
                vb[j] = *reinterpret_cast<const bf16x8*>(x + at + (size_t)j * D + (D >> 1));
            }
        }
        float cs[8], sn[8];
        if (h0 < n_rot) {
            const int pos = positions ? positions[t] : (int)((t / pos_div) % pos_mod);
            const float4* cp = reinterpret_cast<const float4*>(cos_t + (size_t)pos * (D >> 1) + c * 8);
            const float4* sp = reinterpret_cast<const float4*>(sin_t + (size_t)pos * (D >> 1) + c * 8);
            const float4 c0 = cp[0], c1 = cp[1], s0 = sp[0], s1 = sp[1];
            cs[0] = c0.x, cs[1] = c0.y, cs[2] = c0.z, cs[3] = c0.w, cs[4] = c1.x, cs[5] = c1.y, cs[6] = c1.z, cs[7] = c1.w;
            sn[0] = s0.x, sn[1] = s0.y, sn[2] = s0.z, sn[3] = s0.w, sn[4] = s1.x, sn[5] = s1.y, sn[6] = s1.z, sn[7] = s1.w;
        }
#pragma unroll
        for (int j = 0; j < kHeads; ++j) {
            if (h0 + j >= n_heads) break;
            if (h0 + j < n_rot) {
                float a[8], b[8], oa[8], ob[8];
                unpack8(va[j], a);
                unpack8(vb[j], b);
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const float s = sn[k] * sin_sign;
                    oa[k] = a[k] * cs[k] - b[k] * s;
                    ob[k] = b[k] * cs[k] + a[k] * s;
                }
                va[j] = pack8(oa);
                vb[j] = pack8(ob);
            }
            *reinterpret_cast<bf16x8*>(y + at + (size_t)j * D) = va[j];
            *reinterpret_cast<bf16x8*>(y + at + (size_t)j * D + (D >> 1)) = vb[j];
        }
    }
}

// Prompt step: queries and keys rotated in place, and the step's rotated keys and values written to the cache, in one pass over the
// projection.  Item = 8 columns of each half of a head.  Bound by memory; on 2048 tokens x 48 heads of 64 it replaces the rotation
// (9.4 us), two transposing copies (8.8), the cache write (3.6) and four index conversions (8).
__global__ void rope_cache_kernel(bf16* __restrict__ x, const float* __restrict__ cos_t, const float* __restrict__ sin_t,
                                  const int* __restrict__ positions, bf16* __restrict__ cache_k, bf16* __restrict__ cache_v,
                                  const int* __restrict__ seq_ids, const int* __restrict__ block_table, long long stride_b,
                                  long long stride_h, int page_size, int max_pages, int Tn, size_t rows, int n_q, int n_kv, int D) {
    pdl_trigger();
    pdl_wait();
    const int half_vec = D >> 4, heads = n_q + 2 * n_kv;
    const size_t total = rows * (size_t)heads * half_vec;
    for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (size_t)gridDim.x * blockDim.x) {
        const int c = (int)(idx % half_vec);
        const size_t th = idx / half_vec;
        const int h = (int)(th % heads);
        const size_t row = th / heads;
        bf16* base = x + (row * heads + h) * (size_t)D;
        bf16x8 va = reinterpret_cast<bf16x8*>(base)[c], vb = reinterpret_cast<bf16x8*>(base + (D >> 1))[c];
        if (h < n_q + n_kv) {
            const int pos = positions[row];
            float a[8], b[8], oa[8], ob[8];
            unpack8(va, a);
            unpack8(vb, b);
            const float4* cp = reinterpret_cast<const float4*>(cos_t + (size_t)pos * (D >> 1) + c * 8);
            const float4* sp = reinterpret_cast<const float4*>(sin_t + (size_t)pos * (D >> 1) + c * 8);
            const float4 c0 = cp[0], c1 = cp[1], s0 = sp[0], s1 = sp[1];
            const float cs[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
            const float sn[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                oa[k] = a[k] * cs[k] - b[k] * sn[k];
                ob[k] = b[k] * cs[k] + a[k] * sn[k];
            }
            va = pack8(oa);
            vb = pack8(ob);
            reinterpret_cast<bf16x8*>(base)[c] = va;
            reinterpret_cast<bf16x8*>(base + (D >> 1))[c] = vb;
        }
        if (h >= n_q) {
            const int b = (int)(row / Tn), t = (int)(row % Tn);
            const int line = seq_ids ? seq_ids[b] : b, at = positions[(size_t)b * Tn] + t;     // rows follow the first position
            const int kv = h < n_q + n_kv ? h - n_q : h - n_q - n_kv;
            size_t off;
            if (block_table)
                off = (size_t)block_table[(size_t)line * max_pages + at / page_size] * stride_b + (size_t)kv * stride_h +
                      (size_t)(at % page_size) * D;
            else
                off = (size_t)line * stride_b + (size_t)kv * stride_h + (size_t)at * D;
            bf16* dst = (h < n_q + n_kv ? cache_k : cache_v) + off;
            reinterpret_cast<bf16x8*>(dst)[c] = va;
            reinterpret_cast<bf16x8*>(dst + (D >> 1))[c] = vb;
        }
    }
}

inline int grid_for(size_t work_items, int threads) {
    size_t blocks = (work_items + threads - 1) / threads;
    const size_t cap = (size_t)nxd_num_sms() * 16;
    if (blocks > cap) blocks = cap;
    if (blocks < 1) blocks = 1;
    return (int)blocks;
}

}  // namespace

NXD_API int nxd_swiglu_fwd(const void* gate_up, void* out, long long rows, int I, void* stream) {
    NXD_REQUIRE(I % 8 == 0, "swiglu: I=%d must be a multiple of 8", I);
    if (rows == 0) return 0;
    const size_t work = (size_t)rows * (I / 8);
    NXD_CHECK_CUDA((nxd_launch_pdl(swiglu_fwd_kernel, dim3(grid_for(work, 256)), dim3(256), 0, (cudaStream_t)stream,
        (const bf16*)gate_up, (bf16*)out, (size_t)rows, I)));
    NXD_LAUNCH_CHECK();
    return 0;
}

NXD_API int nxd_swiglu_bwd(const void* gate_up, const void* dy, void* dgate_up, long long rows, int I,
                           void* stream) {
    NXD_REQUIRE(I % 8 == 0, "swiglu_bwd: I=%d must be a multiple of 8", I);
    if (rows == 0) return 0;
    const size_t work = (size_t)rows * (I / 8);
    NXD_CHECK_CUDA((nxd_launch_pdl(swiglu_bwd_kernel, dim3(grid_for(work, 256)), dim3(256), 0, (cudaStream_t)stream,
        (const bf16*)gate_up, (const bf16*)dy, (bf16*)dgate_up, (size_t)rows, I)));
    NXD_LAUNCH_CHECK();
    return 0;
}

// x [T, heads_total, D] bf16 -> y (x itself, or another buffer): the first n_rot_heads heads rotated at positions[t] (int32; NULL:
// (t / pos_div) % pos_mod), the others copied.  cos / sin [max_pos, D / 2] fp32; inverse != 0: the transpose rotation (backward).
// D a multiple of 16, x and y 16-byte aligned.
NXD_API int nxd_rope(const void* x, void* y, const float* cos_t, const float* sin_t, const int* positions, long long T,
                     int heads_total, int n_rot_heads, int D, int pos_div, int pos_mod, int inverse, void* stream) {
    NXD_REQUIRE(D % 16 == 0, "rope: head dim %d must be a multiple of 16", D);
    NXD_REQUIRE(n_rot_heads <= heads_total, "rope: n_rot_heads > heads_total");
    const int n_heads = x == y ? n_rot_heads : heads_total;
    if (T == 0 || n_heads == 0) return 0;
    // four heads per thread where that leaves 2^16 threads and a warp reads 64 bytes or more of each half head: heads of 128, 40 of
    // them: 1000 tokens in place 5.4 us with one head per thread, 4.6 with four, 8192 tokens 28.9 / 21.9, but 64 tokens 2.3 / 3.1;
    // 48 heads of 64: 2048 tokens 8.4 / 11.0, 8192 tokens out of place 30.1 / 35.9
    const size_t quads = (size_t)T * ((n_heads + 3) / 4) * (D / 16);
    const bool four = D >= 128 && quads >= 1 << 16;
    const size_t work = four ? quads : (size_t)T * n_heads * (D / 16);
    auto kern = four ? rope_kernel<4> : rope_kernel<1>;
    NXD_CHECK_CUDA((nxd_launch_pdl(kern, dim3(grid_for(work, 256)), dim3(256), 0, (cudaStream_t)stream, (const bf16*)x, (bf16*)y,
        cos_t, sin_t, positions, (size_t)T, heads_total, n_heads, n_rot_heads, D, pos_div < 1 ? 1 : pos_div, pos_mod < 1 ? 1 :
        pos_mod, inverse ? -1.f : 1.f)));
    NXD_LAUNCH_CHECK();
    return 0;
}

NXD_API int nxd_rope_inplace(void* x, const float* cos_t, const float* sin_t, const int* positions, long long T,
                             int heads_total, int n_rot_heads, int D, int pos_div, int pos_mod, int inverse,
                             void* stream) {
    return nxd_rope(x, x, cos_t, sin_t, positions, T, heads_total, n_rot_heads, D, pos_div, pos_mod, inverse, stream);
}

// qkv [B * Tn, n_q + 2 n_kv, D] bf16 (q | k | v heads): q and k rotated in place at positions [B * Tn] int32; row t of sequence b
// goes to cache row positions[b * Tn] + t of line seq_ids[b] (NULL: b).  Cache as in nxd_kv_cache_update.  D a multiple of 16.
NXD_API int nxd_rope_cache_write(void* qkv, const float* cos_t, const float* sin_t, const int* positions, void* cache_k,
                                 void* cache_v, const int* seq_ids, const int* block_table, long long stride_b, long long stride_h,
                                 int page_size, int max_pages, int B, int Tn, int n_q, int n_kv, int D, void* stream) {
    NXD_REQUIRE(D % 16 == 0, "rope_cache: head dim %d must be a multiple of 16", D);
    const size_t rows = (size_t)B * Tn;
    if (rows == 0) return 0;
    NXD_CHECK_CUDA(nxd_launch_pdl(rope_cache_kernel, dim3(grid_for(rows * (n_q + 2 * n_kv) * (D / 16), 256)), dim3(256), 0,
                                  (cudaStream_t)stream, (bf16*)qkv, cos_t, sin_t, positions, (bf16*)cache_k, (bf16*)cache_v, seq_ids,
                                  block_table, stride_b, stride_h, page_size > 0 ? page_size : 1, max_pages, Tn, rows, n_q, n_kv, D));
    NXD_LAUNCH_CHECK();
    return 0;
}
