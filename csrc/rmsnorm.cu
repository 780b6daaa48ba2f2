// RMSNorm forward / backward for sm_100a.
//
// Replaces the reference's fp64-upcast torch ops
// (examples/training/llama/modeling_llama_nxd.py:142-149) and the inference
// `RmsNorm` custom call (examples/inference/modules/custom_calls.py:5-16).
//
// Layout: x [rows, H] bf16 row-major, H % 8 == 0.  One CTA per row keeps the row
// in registers as fp32 between the sum-of-squares pass and the scale pass, so HBM
// traffic is exactly one read + one write of the activation (HBM-bound op).
// Optional fused residual add:  s = x + r;  y = rmsnorm(s);  s is also written.
//
// Backward: dx = rstd * (g - xhat * mean(g * xhat)),  g = dy * w,  xhat = x * rstd
//           dw = sum_rows(dy * xhat)   -> persistent CTAs accumulate per-thread
//           partials in registers, write [P, H] fp32 partials to scratch, and a
//           second kernel reduces the P partial rows.
#include <cuda_pipeline.h>

#include "common.cuh"

namespace {

template <int VPT>  // 16-byte vectors per thread
__global__ void rmsnorm_fwd_kernel(const bf16* __restrict__ x, const bf16* __restrict__ res,
                                   const bf16* __restrict__ w, bf16* __restrict__ y,
                                   bf16* __restrict__ res_out, float* __restrict__ rstd_out, int H,
                                   float eps) {
    __shared__ float red[32];
    pdl_trigger();
    pdl_wait();
    const int row = blockIdx.x;
    const int nvec = H >> 3;
    const bf16x8* xr = reinterpret_cast<const bf16x8*>(x + (size_t)row * H);
    const bf16x8* rr = res ? reinterpret_cast<const bf16x8*>(res + (size_t)row * H) : nullptr;
    float v[VPT][8];
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
        const int c = threadIdx.x + i * blockDim.x;
        if (c < nvec) {
            bf16x8 p = xr[c];
            unpack8(p, v[i]);
            if (rr) {
                float r[8];
                bf16x8 q = rr[c];
                unpack8(q, r);
#pragma unroll
                for (int k = 0; k < 8; ++k) v[i][k] += r[k];
                if (res_out) {
                    // round the residual stream to bf16 once, and normalise the rounded value
                    bf16x8 s = pack8(v[i]);
                    reinterpret_cast<bf16x8*>(res_out + (size_t)row * H)[c] = s;
                    unpack8(s, v[i]);
                }
            }
#pragma unroll
            for (int k = 0; k < 8; ++k) ss += v[i][k] * v[i][k];
        }
    }
    ss = block_sum(ss, red);
    const float rstd = rsqrtf(ss / (float)H + eps);
    if (threadIdx.x == 0 && rstd_out) rstd_out[row] = rstd;
    const bf16x8* wr = reinterpret_cast<const bf16x8*>(w);
    bf16x8* yr = reinterpret_cast<bf16x8*>(y + (size_t)row * H);
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
        const int c = threadIdx.x + i * blockDim.x;
        if (c < nvec) {
            float wv[8], o[8];
            bf16x8 p = wr[c];
            unpack8(p, wv);
#pragma unroll
            for (int k = 0; k < 8; ++k) o[k] = v[i][k] * rstd * wv[k];
            yr[c] = pack8(o);
        }
    }
}

// Bound by memory (3 reads and a write per element with a residual gradient).  A thread copies its own columns of the CTA's next
// rows into shared memory with cp.async, kRing - 1 rows ahead, and reads only what it copied itself: no barrier for the data, one
// for the row's sum.  The grid is what is resident at once: up to 4 CTAs per SM, each with rings of 6 kRing H bytes (3072 columns:
// 221 KB per SM, two thirds of it without a residual gradient).  8192 x 3072 (201 MB): 71 us with the next row prefetched into
// registers (113 of them: 3 CTAs per SM for a grid of 4), 44 us.
// 8 VPT columns per thread and at most 512 threads: 2048, 8192 and kRingMaxH columns with 1, 2 and 4 vectors.  Three rows of more
// than 12842 columns do not fit shared memory, so the widest instance keeps two.
constexpr int kRingMaxH = 16384;

template <int VPT>
struct RingCfg {
    static constexpr int kRows = VPT == 4 ? 2 : 3;
    static constexpr int kMaxH = VPT == 1 ? 2048 : VPT == 2 ? 8192 : kRingMaxH;
    static constexpr int kCtas = VPT == 4 ? 2 : 4;           // per SM that the registers (48, 58 and 109 a thread) let run
    static constexpr int smem(int H) { return kRows * 3 * H * 2; }
};

template <int VPT>
__global__ void __launch_bounds__(VPT == 1 ? 256 : 512)
rmsnorm_bwd_ring_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ x, const bf16* __restrict__ w,
                        const float* __restrict__ rstd, const bf16* __restrict__ dres, bf16* __restrict__ dx,
                        float* __restrict__ dw_partial, int rows, int H) {
    pdl_trigger();
    pdl_wait();
    constexpr int kRing = RingCfg<VPT>::kRows;
    extern __shared__ __align__(16) bf16x8 ring[];       // [kRing][dy | x | dres][nvec]
    __shared__ float red[2][32];
    const int nvec = H >> 3, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = (blockDim.x + 31) >> 5;
    float dwacc[VPT][8];
    bf16x8 wv[VPT];
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
        const int c = threadIdx.x + i * blockDim.x;
#pragma unroll
        for (int k = 0; k < 8; ++k) dwacc[i][k] = 0.f;
        if (c < nvec) wv[i] = reinterpret_cast<const bf16x8*>(w)[c];
    }
    auto fetch = [&](int row, int slot) {
        if (row < rows) {
            bf16x8* dst = ring + (size_t)slot * 3 * nvec;
            const size_t at = (size_t)row * H;
#pragma unroll
            for (int i = 0; i < VPT; ++i) {
                const int c = threadIdx.x + i * blockDim.x;
                if (c < nvec) {
                    __pipeline_memcpy_async(dst + c, dy + at + c * 8, 16);
                    __pipeline_memcpy_async(dst + nvec + c, x + at + c * 8, 16);
                    if (dres != nullptr) __pipeline_memcpy_async(dst + 2 * nvec + c, dres + at + c * 8, 16);
                }
            }
        }
        __pipeline_commit();
    };
#pragma unroll
    for (int j = 0; j < kRing - 1; ++j) fetch(blockIdx.x + j * gridDim.x, j);
    int slot = 0, par = 0;
    for (int row = blockIdx.x; row < rows; row += gridDim.x) {
        const float rs = rstd[row];
        {   // the slot read in the last round is free: this thread alone uses its columns
            const int ahead = slot == 0 ? kRing - 1 : slot - 1;
            const long long next = row + (long long)(kRing - 1) * gridDim.x;
            fetch(next < rows ? (int)next : rows, ahead);
        }
        __pipeline_wait_prior(kRing - 1);
        const bf16x8* src = ring + (size_t)slot * 3 * nvec;
        float dot = 0.f;
#pragma unroll
        for (int i = 0; i < VPT; ++i) {
            const int c = threadIdx.x + i * blockDim.x;
            if (c < nvec) {
                float d[8], xv[8], wf[8];
                unpack8(src[c], d);
                unpack8(src[nvec + c], xv);
                unpack8(wv[i], wf);
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const float xh = xv[k] * rs;
                    dot += d[k] * wf[k] * xh;
                    dwacc[i][k] += d[k] * xh;
                }
            }
        }
        dot = warp_sum(dot);
        if (lane == 0) red[par][warp] = dot;
        __syncthreads();                                 // red[par] is written again two rows on, behind the next row's barrier
        dot = warp_sum(lane < nwarps ? red[par][lane] : 0.f) / (float)H;
        bf16x8* dxr = reinterpret_cast<bf16x8*>(dx + (size_t)row * H);
#pragma unroll
        for (int i = 0; i < VPT; ++i) {
            const int c = threadIdx.x + i * blockDim.x;
            if (c < nvec) {
                float d[8], xv[8], wf[8], o[8];
                unpack8(src[c], d);
                unpack8(src[nvec + c], xv);
                unpack8(wv[i], wf);
#pragma unroll
                for (int k = 0; k < 8; ++k) o[k] = rs * (d[k] * wf[k] - xv[k] * rs * dot);
                if (dres != nullptr) {                   // fused add of the gradient flowing through the residual branch
                    float r[8];
                    unpack8(src[2 * nvec + c], r);
#pragma unroll
                    for (int k = 0; k < 8; ++k) o[k] += r[k];
                }
                dxr[c] = pack8(o);
            }
        }
        par ^= 1;
        slot = slot + 1 == kRing ? 0 : slot + 1;
    }
    float* out = dw_partial + (size_t)blockIdx.x * H;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
        const int c = threadIdx.x + i * blockDim.x;
        if (c < nvec) {
            float4* o4 = reinterpret_cast<float4*>(out + (size_t)c * 8);
            o4[0] = make_float4(dwacc[i][0], dwacc[i][1], dwacc[i][2], dwacc[i][3]);
            o4[1] = make_float4(dwacc[i][4], dwacc[i][5], dwacc[i][6], dwacc[i][7]);
        }
    }
}

// dw[h] = sum_p partial[p, h]; optionally accumulates into an fp32 buffer.  32 columns per block (one 128-byte line of a
// partial row per warp), kSumWarps warps take every kSumWarps-th row, 8 loads in flight each.  592 rows x 3072: 29 us with one
// thread per column, 5 us.
constexpr int kSumWarps = 16;

__global__ void __launch_bounds__(32 * kSumWarps)
colsum_partials_kernel(const float* __restrict__ partial, int P, int H, bf16* __restrict__ dw_bf16,
                       float* __restrict__ dw_f32, int accumulate) {
    pdl_trigger();
    pdl_wait();
    __shared__ float part[kSumWarps][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, h = blockIdx.x * 32 + lane;
    float s = 0.f;
    if (h < H) {
#pragma unroll 8
        for (int p = warp; p < P; p += kSumWarps) s += partial[(size_t)p * H + h];
    }
    part[warp][lane] = s;
    __syncthreads();
    if (warp != 0 || h >= H) return;
#pragma unroll
    for (int i = 1; i < kSumWarps; ++i) s += part[i][lane];
    if (dw_f32) dw_f32[h] = accumulate ? dw_f32[h] + s : s;
    if (dw_bf16) dw_bf16[h] = __float2bfloat16(s);
}

struct NormCfg {
    int threads;
    int vpt;
};

NormCfg pick_cfg(int H) {
    const int nvec = H / 8;
    NormCfg c;
    if (nvec <= 128) {
        c.vpt = 1;
    } else if (nvec <= 512) {
        c.vpt = 2;
    } else if (nvec <= 2048) {
        c.vpt = 4;
    } else {
        c.vpt = 8;
    }
    int t = (nvec + c.vpt - 1) / c.vpt;
    t = ((t + 31) / 32) * 32;
    if (t > 1024) t = 1024;
    if (t < 32) t = 32;
    c.threads = t;
    return c;
}

}  // namespace

// Number of partial rows (persistent CTAs) the backward kernel uses; the scratch
// buffer passed to nxd_rmsnorm_bwd must hold nxd_rmsnorm_bwd_num_partials * H floats.
NXD_API int nxd_rmsnorm_bwd_num_partials(int rows) {
    int p = nxd_num_sms() * 4;
    if (p > rows) p = rows;
    if (p < 1) p = 1;
    return p;
}

NXD_API int nxd_rmsnorm_fwd(const void* x, const void* residual, const void* w, void* y, void* residual_out,
                            float* rstd, int rows, int H, float eps, void* stream) {
    NXD_REQUIRE(H % 8 == 0 && H <= 65536, "rmsnorm: H=%d must be a multiple of 8 and <= 65536", H);
    if (rows == 0) return 0;
    NormCfg c = pick_cfg(H);
    cudaStream_t s = (cudaStream_t)stream;
#define LAUNCH(V)                                                                                          \
    NXD_CHECK_CUDA(nxd_launch_pdl(rmsnorm_fwd_kernel<V>, dim3(rows), dim3(c.threads), 0, s, (const bf16*)x,   \
                                  (const bf16*)residual, (const bf16*)w, (bf16*)y, (bf16*)residual_out, rstd, H, eps))
    switch (c.vpt) {
        case 1: LAUNCH(1); break;
        case 2: LAUNCH(2); break;
        case 4: LAUNCH(4); break;
        default: LAUNCH(8); break;
    }
#undef LAUNCH
    NXD_LAUNCH_CHECK();
    return 0;
}

template <int VPT>
static int rmsnorm_bwd_ring(const void* dy, const void* x, const void* w, const float* rstd, const void* dresidual, void* dx,
                            float* scratch, int& P, int rows, int H, cudaStream_t s) {
    using C = RingCfg<VPT>;
    const int smem = C::smem(H), threads = ((H / 8 + VPT - 1) / VPT + 31) / 32 * 32;
    NXD_CHECK_CUDA(nxd_allow_smem<rmsnorm_bwd_ring_kernel<VPT>>(C::smem(C::kMaxH)));
    // resident CTAs per SM: 227 KB of shared memory (1 KB of it reserved per CTA); the registers let C::kCtas run
    int per_sm = 232448 / (smem + 1024 + 256);
    if (per_sm > C::kCtas) per_sm = C::kCtas;
    if (P > per_sm * nxd_num_sms()) P = per_sm * nxd_num_sms();
    NXD_CHECK_CUDA((nxd_launch_pdl(rmsnorm_bwd_ring_kernel<VPT>, dim3(P), dim3(threads), smem, s, (const bf16*)dy, (const bf16*)x,
        (const bf16*)w, rstd, (const bf16*)dresidual, (bf16*)dx, scratch, rows, H)));
    NXD_LAUNCH_CHECK();
    return 0;
}

// scratch: P * H floats
static int rmsnorm_bwd_impl(const void* dy, const void* x, const void* w, const float* rstd, const void* dresidual,
                            void* dx, void* dw_bf16, float* dw_f32, int accumulate, float* scratch, int P, int rows,
                            int H, cudaStream_t s) {
    const int rc = H <= RingCfg<1>::kMaxH   ? rmsnorm_bwd_ring<1>(dy, x, w, rstd, dresidual, dx, scratch, P, rows, H, s)
                   : H <= RingCfg<2>::kMaxH ? rmsnorm_bwd_ring<2>(dy, x, w, rstd, dresidual, dx, scratch, P, rows, H, s)
                                            : rmsnorm_bwd_ring<4>(dy, x, w, rstd, dresidual, dx, scratch, P, rows, H, s);
    if (rc) return rc;
    NXD_CHECK_CUDA((nxd_launch_pdl(colsum_partials_kernel, dim3((H + 31) / 32), dim3(32 * kSumWarps), 0, s, scratch, P, H,
        (bf16*)dw_bf16, dw_f32, accumulate)));
    NXD_LAUNCH_CHECK();
    return 0;
}

// rows == 0: nothing to differentiate, but a caller that asked for a fresh dW (accumulate == 0) still gets zeros
// (the column-sum kernel with no partial rows reads nothing and stores 0).
static int rmsnorm_bwd_empty(void* dw_bf16, float* dw_f32, int accumulate, int H, cudaStream_t s) {
    if (accumulate || (dw_bf16 == nullptr && dw_f32 == nullptr)) return 0;
    NXD_CHECK_CUDA((nxd_launch_pdl(colsum_partials_kernel, dim3((H + 31) / 32), dim3(32 * kSumWarps), 0, s, nullptr, 0, H,
        (bf16*)dw_bf16, dw_f32, 0)));
    NXD_LAUNCH_CHECK();
    return 0;
}

// scratch: caller-provided device buffer of nxd_rmsnorm_bwd_num_partials(rows) * H floats.
NXD_API int nxd_rmsnorm_bwd(const void* dy, const void* x, const void* w, const float* rstd,
                            const void* dresidual, void* dx, void* dw_bf16, float* dw_f32, int accumulate,
                            float* scratch, int rows, int H, void* stream) {
    NXD_REQUIRE(H % 8 == 0 && H <= 65536, "rmsnorm_bwd: H=%d must be a multiple of 8 and <= 65536", H);
    NXD_REQUIRE(scratch != nullptr, "rmsnorm_bwd: scratch buffer is required");
    if (rows == 0) return rmsnorm_bwd_empty(dw_bf16, dw_f32, accumulate, H, (cudaStream_t)stream);
    NXD_REQUIRE(H <= kRingMaxH, "rmsnorm_bwd: H=%d, at most %d columns", H, kRingMaxH);
    return rmsnorm_bwd_impl(dy, x, w, rstd, dresidual, dx, dw_bf16, dw_f32, accumulate, scratch,
                            nxd_rmsnorm_bwd_num_partials(rows), rows, H, (cudaStream_t)stream);
}

// ---------------------------------------------------------------------------------------------------------
// Allocation-free variant of the backward pass.
//
// nxd_rmsnorm_bwd() asks its caller for a scratch buffer (the per-CTA partial sums of dW).  Some callers have no
// way to provide one: a host program that handed the whole HBM pool to another allocator at start-up (so a later
// cudaMalloc fails or fragments the pool), a latency-critical loop that cannot tolerate the device-wide
// synchronisation cudaMalloc / cudaFree imply, or a plug-in running inside someone else's operator callback where
// device memory may only come from that host's allocator.  For them the partial sums live in the library image
// itself: a file-scope __device__ array of kStaticScratchFloats floats (4 MiB) that every GPU which loads the
// library keeps until the process exits.
//
//   * Limit: H <= kStaticMaxH (8192).  The number of partial rows is reduced to fit (at least 128 rows of partials
//     remain at the largest H), which changes the summation order of dW slightly but not the result beyond fp32
//     rounding.  Larger H is rejected with an error; use nxd_rmsnorm_bwd() (up to 16384 columns) with your own buffer instead.
//   * The first call on each device resolves the array's device address (cudaGetSymbolAddress with that device
//     current).  Make that first call before you start capturing a stream into a graph.
//   * All calls share the one array.  Nothing in it has to start at zero -- every partial row that is read is
//     written earlier in the same call -- and its contents after a call are meaningless.  Two calls whose kernels
//     can overlap on the GPU (different streams) race on it; serialise them.
//   * The call itself performs no cudaMalloc / cudaFree and calls no allocating library routine.
// ---------------------------------------------------------------------------------------------------------
namespace {

constexpr int kStaticScratchFloats = 1 << 20;
constexpr int kStaticMaxH = 8192;
constexpr int kStaticMaxDevices = 64;

static __device__ __align__(256) float g_rmsnorm_bwd_static_scratch[kStaticScratchFloats];

// In host code the name above is only a handle for the symbol, not an address the GPU can use: resolve it per device.
int static_scratch_for_current_device(float** out) {
    static float* ptrs[kStaticMaxDevices] = {nullptr};
    int dev = 0;
    NXD_CHECK_CUDA(cudaGetDevice(&dev));
    NXD_REQUIRE(dev >= 0 && dev < kStaticMaxDevices, "rmsnorm_bwd_static: device index %d out of range", dev);
    float* p = __atomic_load_n(&ptrs[dev], __ATOMIC_ACQUIRE);
    if (p == nullptr) {
        void* addr = nullptr;
        NXD_CHECK_CUDA(cudaGetSymbolAddress(&addr, g_rmsnorm_bwd_static_scratch));
        NXD_REQUIRE(addr != nullptr, "rmsnorm_bwd_static: could not resolve the scratch symbol on device %d", dev);
        p = static_cast<float*>(addr);
        __atomic_store_n(&ptrs[dev], p, __ATOMIC_RELEASE);
    }
    *out = p;
    return 0;
}

}  // namespace

NXD_API int nxd_rmsnorm_bwd_static_max_h(void) { return kStaticMaxH; }

NXD_API int nxd_rmsnorm_bwd_static(const void* dy, const void* x, const void* w, const float* rstd,
                                   const void* dresidual, void* dx, void* dw_bf16, float* dw_f32, int accumulate,
                                   int rows, int H, void* stream) {
    NXD_REQUIRE(H % 8 == 0 && H > 0, "rmsnorm_bwd_static: H=%d must be a positive multiple of 8", H);
    NXD_REQUIRE(H <= kStaticMaxH,
                "rmsnorm_bwd_static: H=%d exceeds the built-in scratch limit of %d columns; call nxd_rmsnorm_bwd with a "
                "caller-provided scratch buffer instead",
                H, kStaticMaxH);
    NXD_REQUIRE(rows >= 0, "rmsnorm_bwd_static: negative row count");
    if (rows == 0) return rmsnorm_bwd_empty(dw_bf16, dw_f32, accumulate, H, (cudaStream_t)stream);
    float* scratch = nullptr;
    if (int rc = static_scratch_for_current_device(&scratch)) return rc;
    int P = nxd_rmsnorm_bwd_num_partials(rows);
    const int fit = kStaticScratchFloats / H;
    if (P > fit) P = fit;
    return rmsnorm_bwd_impl(dy, x, w, rstd, dresidual, dx, dw_bf16, dw_f32, accumulate, scratch, P, rows, H,
                            (cudaStream_t)stream);
}
