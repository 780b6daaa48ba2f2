// Retention of long steps on the 5th-gen tensor cores (tcgen05), chunk-wise, with fp32 accuracy:
//
//   S_{c+1} = decay^n S_c + U_c,  U_c = sum_s decay^(n-1-s) k_s v_s^T;     o_t = decay^(t+1) S_c^T q_t + sum_{s<=t} P[t][s] v_s,
//   P[t][s] = decay^(t-s) (q_t . k_s)                                       (t, s counted inside the chunk of kC tokens)
//
// Rotation, decays and state are fp32.  Every matrix operand is handed to the tensor cores as three bf16 pieces
// x = x0 + x1 + x2 (each the rounded remainder of the ones before: 24 bits), and a product of two takes the six piece
// products that reach 2^-24, the smallest first.  The tensor cores accumulate in fp32 but cut instead of rounding
// (measured: 6.6e-8 over 64 terms, 2.3e-7 over 256, 1e-6 over 1024), so an accumulator takes 64 terms and is then added to
// the epilogue's registers.  Against float64 the result is closer than the fp32 kernels of retention.cu, which these replace for
// long steps of key sizes up to 256.  Kernels:
//   prep     rotated queries and keys, keys times decay^(n-1-s), values -> pieces; chunk-major, padding tokens as zeros
//   <kU>     U_c of all chunks, one product of K = kC per chunk
//   states   sequential over chunks, one thread per four state elements: state at every chunk's start -> pieces, line's state
//   <kP>     P of all chunks; decay and causal mask in the epilogue, result split into pieces
//   <kO>     both output products of a tile in one pass, [P | q] over [V ; S_c]
// The three products run the persistent CTA-pair pipeline of gemm_tcgen05.cu with 256 x 128 tiles; 64 terms are 24 MMAs over the three
// pieces of both operands, each piece (24 KB) in a slot of its own that is free again behind its last product: the smallest pieces are
// used first, so their slots load again while the others are multiplied (all pieces as one stage, two stages: every stage waited for its
// loads).  The chunk is as long as the tile is high: a shorter one would leave half the rows of the CTA pair empty, and the state traffic
// falls with the chunk's length.
// 2 x 4096 tokens, 8 heads of 256 x 512, fp32 (stages and rows through shared memory before): prep 158 -> 150 us, products 166 + 95 + 64 ->
// 145 + 82 + 57, states 52; 633 -> 560 us through the entry point, 3482 us on the fp32 kernels (error against float64 1.6e-7 against
// 3.4e-7).  2.6 GB of pieces and intermediates at 5.2 TB/s: memory bounds it now.
#include "attn_tc_common.cuh"
#include "common.cuh"
#include "gemm_tcgen05.cuh"
#include "ptx.cuh"

namespace {

using namespace nxd_attn;
using nxd_gemm::make_tmap_3d;

constexpr int kC = 256;              // tokens of a chunk
constexpr int kBN = 128, kBK = 64;
constexpr int kSlots = 8, kAcc = 4;
constexpr int kThreads = 256;
constexpr int kABytes = 128 * kBK * 2, kBBytes = (kBN / 2) * kBK * 2;       // one piece: this CTA's rows of A, its half of B
constexpr int kSlotBytes = kABytes + kBBytes;                               // one piece of both
constexpr int kStagingOff = kSlots * kSlotBytes;
constexpr int kStagingPerWarp = 2 * 32 * 128;
constexpr int kTableOff = kStagingOff + 4 * kStagingPerWarp;                // kP: decay^j, j < kC
constexpr int kBarOff = kTableOff + kC * 4;
constexpr int kSmem = kBarOff + (2 * kSlots + 2 * kAcc) * 8 + 16 + 1024;
static_assert(kSmem <= 232448, "shared memory budget exceeded");

enum { kU = 0, kP = 1, kO = 2 };

// Slots of the ring: a block of 64 terms takes three, its pieces 2, 1 and 0
struct Slot {
    int i = 0;
    uint32_t phase = 0;
    __device__ __forceinline__ void next() {
        if (++i == kSlots) i = 0, phase ^= 1;
    }
};

__device__ __forceinline__ float ldf(const float* p) { return *p; }
__device__ __forceinline__ float ldf(const bf16* p) { return __bfloat162float(*p); }

// x -> three bf16 pieces, 16 bytes of eight values each
__device__ __forceinline__ void split8(const float* x, bf16x8 (&p)[3]) {
    float r[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) r[i] = x[i];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        p[k] = pack8(r);
        float f[8];
        unpack8(p[k], f);
#pragma unroll
        for (int i = 0; i < 8; ++i) r[i] -= f[i];
    }
}

struct Args {
    const float* decay;
    const int *n_new, *flag, *bad;     // flag [E], bad [E][Dv]: see prep
    int E, NC, H, Tn, D, Dv, n_tiles, k_blocks1, k_blocks2;
    int pos_o[3];
};

// MODE kU: A = decayed keys [kC, D] (MN-major), B = values [kC, Dv] (MN-major), D = U [D, Dv] fp32
// MODE kP: A = queries [kC, D] (K-major), B = keys [kC, D] (K-major), D = P [kC, kC] as pieces
// MODE kO: A = P, then queries (K-major), B = values, then states [D, Dv] (MN-major), D = out [B, T, H, Dv] fp32
// NB: pieces of the values (1: bf16 values are one piece)
template <int MODE, int NB>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
retention_tc_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                    const __grid_constant__ CUtensorMap tmap_a2, const __grid_constant__ CUtensorMap tmap_b2,
                    const __grid_constant__ CUtensorMap tmap_d, const Args p) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = ptx::align_smem_1024(smem_raw);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + kBarOff);
    uint64_t* empty = full + kSlots;
    uint64_t* acc_full = empty + kSlots;
    uint64_t* acc_empty = acc_full + kAcc;
    uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(acc_empty + kAcc);
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const uint32_t rank = ptx::cluster_ctarank();
    const bool leader = rank == 0;
    const int num_tiles = p.E * p.n_tiles, k_blocks = p.k_blocks1 + p.k_blocks2;
    constexpr bool A_MN = MODE == kU, B_MN = MODE != kP;
    constexpr int NB1 = MODE == kP ? 3 : NB;               // pieces of the first B operand

    if (warp == 0 && lane == 0) {
        ptx::prefetch_tensormap(&tmap_a);
        ptx::prefetch_tensormap(&tmap_b);
        ptx::prefetch_tensormap(&tmap_d);
    }
    if (warp == 1 && lane == 0) {
        for (int i = 0; i < kSlots; ++i) {
            ptx::mbar_init(&full[i], 1);
            ptx::mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < kAcc; ++i) {
            ptx::mbar_init(&acc_full[i], 1);
            ptx::mbar_init(&acc_empty[i], 8);              // both CTAs' epilogue warps
        }
        ptx::fence_barrier_init();
    }
    if (warp == 2) ptx::tmem_alloc<2>(tmem_ptr, kAcc * kBN);        // ahead of the wait, as in gemm_tcgen05.cu
    ptx::tcgen05_fence_before();
    ptx::cluster_sync();
    ptx::tcgen05_fence_after();
    const uint32_t tmem = *tmem_ptr;
    pdl_wait();

    if (warp == 0) {
        if (lane == 0) {
            Slot st;
            for (int tile = blockIdx.x >> 1; tile < num_tiles; tile += gridDim.x >> 1) {
                const int e = tile / p.n_tiles, tn = tile % p.n_tiles;
                const int m0 = (int)rank * 128, n0 = tn * kBN + (int)rank * (kBN / 2);
                for (int kb = 0; kb < k_blocks; ++kb) {
                    const bool second = kb >= p.k_blocks1;
                    const int k0 = (second ? kb - p.k_blocks1 : kb) * kBK;
                    const int nb = second ? 3 : NB1;
                    const CUtensorMap* ma = second ? &tmap_a2 : &tmap_a;
                    const CUtensorMap* mb = second ? &tmap_b2 : &tmap_b;
#pragma unroll
                    for (int x = 2; x >= 0; --x) {
                        uint8_t* sa = smem + st.i * kSlotBytes;
                        uint8_t* sb = sa + kABytes;
                        ptx::mbar_wait(&empty[st.i], st.phase ^ 1);
                        if (leader) ptx::mbar_arrive_expect_tx(&full[st.i], 2 * (kABytes + (x < nb ? kBBytes : 0)));
                        if constexpr (A_MN) {
                            ptx::tma_load_3d_pair(ma, &full[st.i], sa, m0, k0, e * 3 + x);
                            ptx::tma_load_3d_pair(ma, &full[st.i], sa + kBK * 128, m0 + 64, k0, e * 3 + x);
                        } else {
                            ptx::tma_load_3d_pair(ma, &full[st.i], sa, k0, m0, e * 3 + x);
                        }
                        if (x < nb) {
                            if constexpr (B_MN) ptx::tma_load_3d_pair(mb, &full[st.i], sb, n0, k0, e * nb + x);
                            else ptx::tma_load_3d_pair(mb, &full[st.i], sb, k0, n0, e * nb + x);
                        }
                        st.next();
                    }
                }
            }
        }
    } else if (warp == 1) {
        if (leader && ptx::elect_one()) {
            constexpr uint32_t idesc = ptx::make_idesc_bf16(256, kBN, A_MN ? 1 : 0, B_MN ? 1 : 0);
            constexpr uint32_t a_lbo = A_MN ? kBK * 128 : 16, b_lbo = B_MN ? kBK * 128 : 16;
            constexpr uint32_t a_step = A_MN ? 2048 : 32, b_step = B_MN ? 2048 : 32;
            Slot st;
            int acc = 0;
            uint32_t acc_ph = 0;
            for (int tile = blockIdx.x >> 1; tile < num_tiles; tile += gridDim.x >> 1) {
                for (int kb = 0; kb < k_blocks; ++kb) {
                    const int nb = kb >= p.k_blocks1 ? 3 : NB1;
                    ptx::mbar_wait(&acc_empty[acc], acc_ph ^ 1);
                    uint32_t sa[3];
                    uint64_t* freed[3];
#pragma unroll
                    for (int x = 2; x >= 0; --x) {
                        ptx::mbar_wait(&full[st.i], st.phase);
                        sa[x] = ptx::smem_u32(smem + st.i * kSlotBytes);
                        freed[x] = &empty[st.i];
                        st.next();
                    }
                    ptx::tcgen05_fence_after();
                    uint32_t add = 0;
                    auto product = [&](int x, int y) {
#pragma unroll
                        for (int k = 0; k < kBK / 16; ++k) {
                            const uint64_t da = ptx::make_smem_desc(sa[x] + k * a_step, a_lbo, 1024);
                            const uint64_t db = ptx::make_smem_desc(sa[y] + kABytes + k * b_step, b_lbo, 1024);
                            ptx::umma_bf16<2>(tmem + acc * kBN, da, db, idesc, add);
                            add = 1;
                        }
                    };
                    product(2, 0);                          // the smallest first
                    if (nb == 3) product(0, 2);
                    ptx::umma_commit_pair(freed[2], 0b11);
                    if (nb == 3) {
                        product(1, 1);
                        product(0, 1);
                    }
                    product(1, 0);
                    ptx::umma_commit_pair(freed[1], 0b11);
                    product(0, 0);
                    ptx::umma_commit_pair(freed[0], 0b11);
                    ptx::umma_commit_pair(&acc_full[acc], 0b11);
                    if (++acc == kAcc) acc = 0, acc_ph ^= 1;
                }
            }
        }
    } else if (warp >= 4) {
        const int q = warp & 3;
        uint8_t* stg = smem + kStagingOff + q * kStagingPerWarp;
        float* table = reinterpret_cast<float*>(smem + kTableOff);
        int buf = 0, acc = 0;
        uint32_t acc_ph = 0;
        for (int tile = blockIdx.x >> 1; tile < num_tiles; tile += gridDim.x >> 1) {
            const int e = tile / p.n_tiles, n0 = (tile % p.n_tiles) * kBN;
            const int c = e % p.NC, bh = e / p.NC, h = bh % p.H, b = bh / p.H;
            const int row0 = (int)rank * 128 + q * 32, row = row0 + lane;       // row of the tile: key channel or token
            float weight = 1.f;
            if (MODE == kO) weight = powf(p.decay[h], (float)(row + 1));
            if (MODE == kP) {
                const float a = p.decay[h];
                named_bar_sync(1, 128);                     // every warp is done with the last tile's table
                for (int i = threadIdx.x - 128; i < kC; i += 128) table[i] = powf(a, (float)i);
                named_bar_sync(1, 128);
            }
            float r[kBN];
#pragma unroll
            for (int i = 0; i < kBN; ++i) r[i] = 0.f;
            for (int kb = 0; kb < k_blocks; ++kb) {
                ptx::mbar_wait(&acc_full[acc], acc_ph);
                ptx::tcgen05_fence_after();
                const uint32_t at = tmem + ((uint32_t)(q * 32) << 16) + acc * kBN;
                const float w = MODE == kO && kb >= p.k_blocks1 ? weight : 1.f;
#pragma unroll
                for (int x = 0; x < kBN; x += 32) {
                    uint32_t v[32];
                    ptx::tmem_ld_32x32b_x32(at + x, v);
                    ptx::tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 32; ++i) r[x + i] = fmaf(w, __uint_as_float(v[i]), r[x + i]);
                }
                ptx::tcgen05_fence_before();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive_cluster(&acc_empty[acc], 0);
                if (++acc == kAcc) acc = 0, acc_ph ^= 1;
            }
            if (MODE == kP) {
#pragma unroll
                for (int i = 0; i < kBN; ++i) {
                    const int s = n0 + i;
                    r[i] = s <= row ? r[i] * table[max(row - s, 0)] : 0.f;
                }
#pragma unroll
                for (int g = 0; g < kBN / 64; ++g) {
#pragma unroll
                    for (int x = 0; x < 3; ++x) {           // piece x of 64 columns; r keeps the remainder
                        if (lane == 0) ptx::bulk_wait_read<1>();
                        __syncwarp();
                        uint8_t* dst = stg + buf * (32 * 128) + lane * 128;
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const bf16x8 v = pack8(r + g * 64 + j * 8);
                            float f[8];
                            unpack8(v, f);
#pragma unroll
                            for (int i = 0; i < 8; ++i) r[g * 64 + j * 8 + i] -= f[i];
                            *reinterpret_cast<bf16x8*>(dst + ((j ^ (lane & 7)) << 4)) = v;
                        }
                        ptx::fence_proxy_async();
                        __syncwarp();
                        if (lane == 0) {
                            ptx::tma_store_3d(&tmap_d, stg + buf * (32 * 128), n0 + g * 64, row0, e * 3 + x);
                            ptx::bulk_commit();
                        }
                        buf ^= 1;
                    }
                }
            } else {
                if (MODE == kO) {
                    const int t = c * kC + row, n = p.n_new != nullptr ? min(p.n_new[b], p.Tn) : p.Tn;
                    if (t >= n) {                           // padding tokens come out as zeros
#pragma unroll
                        for (int i = 0; i < kBN; ++i) r[i] = 0.f;
                    } else if (p.flag[e] != 0) {            // a value that is not finite: see prep
                        const int* bad = p.bad + (long long)e * p.Dv + n0;
#pragma unroll
                        for (int i = 0; i < kBN; ++i)
                            if (n0 + i < p.Dv && bad[i] != 0 && row >= kC - bad[i]) r[i] = __int_as_float(0x7fffffff);
                    }
                }
#pragma unroll
                for (int g = 0; g < kBN / 32; ++g) {
                    if (lane == 0) ptx::bulk_wait_read<1>();
                    __syncwarp();
                    uint8_t* dst = stg + buf * (32 * 128) + lane * 128;
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        *reinterpret_cast<float4*>(dst + ((j ^ (lane & 7)) << 4)) =
                            make_float4(r[g * 32 + 4 * j], r[g * 32 + 4 * j + 1], r[g * 32 + 4 * j + 2], r[g * 32 + 4 * j + 3]);
                    ptx::fence_proxy_async();
                    __syncwarp();
                    if (lane == 0) {
                        const int col = n0 + g * 32;
                        if (MODE == kU) {
                            if (col < p.Dv && row0 < p.D) ptx::tma_store_3d(&tmap_d, stg + buf * (32 * 128), col, row0, e);
                        } else if (col < p.Dv && c * kC + row0 < p.Tn) {
                            int x[4];
                            x[0] = col;
                            coords(p.pos_o, c * kC + row0, h, b, x);
                            tma_store_4d(&tmap_d, stg + buf * (32 * 128), x[0], x[1], x[2], x[3]);
                        }
                        ptx::bulk_commit();
                    }
                    buf ^= 1;
                }
            }
        }
        if (lane == 0) ptx::bulk_wait<0>();
    }
    ptx::tcgen05_fence_before();
    ptx::cluster_sync();
    if (warp == 2) ptx::tmem_dealloc<2>(tmem, kAcc * kBN);
}

constexpr int PT = 32, PREP_THREADS = 256;

// eight consecutive values of a row
template <typename T>
__device__ __forceinline__ void load8(const T* src, int vec, float (&f)[8]) {
    if (!vec) {
#pragma unroll
        for (int x = 0; x < 8; ++x) f[x] = ldf(src + x);
    } else if constexpr (sizeof(T) == 2) {
        unpack8(*reinterpret_cast<const bf16x8*>(src), f);
    } else {
        *reinterpret_cast<float4*>(f) = *reinterpret_cast<const float4*>(src);
        *reinterpret_cast<float4*>(f + 4) = *reinterpret_cast<const float4*>(src + 4);
    }
}

// grid (3 * chunks * kC / PT, H, B): the queries, the keys or the values of PT tokens of a head.  q3 / k3 / kd3 [E][3][kC][D], v3
// [E][NB][kC][Dv].  Bound by memory: no shared memory and no barrier between a thread's loads and its stores, so that enough loads are in
// flight (rows laid out in shared memory for the rotation, two CTAs a SM: 159 us at the sizes above).  A thread rotates eight pairs of
// `halves`, which lie half a rotation apart, at a time.
// A value that is not finite would reach the tokens before it through 0 * value: it goes over as zero, the first such token s
// of a column is kept as bad[e][j] = kC - s, and the consumers put NaN where it would have arrived.
// vec: bit 0 the rows of proj in 16-byte loads, bit 1 the rotation in whole vectors
template <typename T, int NB>
__global__ void __launch_bounds__(PREP_THREADS)
retention_tc_prep_kernel(const T* __restrict__ proj, long long ld, int q_off, int k_off, int v_off,
                         const float* __restrict__ decay, bf16* __restrict__ q3, bf16* __restrict__ k3, bf16* __restrict__ kd3,
                         bf16* __restrict__ v3, int* __restrict__ flag, int* __restrict__ bad, const int* __restrict__ q_start,
                         const int* __restrict__ n_new, int Tn, int NC, int H, int D, int Dv, float kscale,
                         const float* __restrict__ rope_cos, const float* __restrict__ rope_sin, int rot, int halves,
                         int max_pos, int vec) {
    pdl_trigger();
    pdl_wait();
    __shared__ float fade[PT];               // decay^(n - 1 - s) of the chunk's tokens
    const int hd = blockIdx.y, role = blockIdx.x % 3, b = blockIdx.z, tid = threadIdx.x;
    const int t0 = (int)(blockIdx.x / 3) * PT, c = t0 / kC, s0 = t0 % kC;
    const int n = n_new != nullptr ? min(n_new[b], Tn) : Tn;
    const int nt = max(0, min(PT, n - t0)), chunk_n = min(kC, n - c * kC);
    const long long e = ((long long)b * H + hd) * NC + c, row0 = (long long)b * Tn + t0;
    auto put = [&](bf16* base, int pieces, int width, int t, int d, const float (&f)[8]) {
        bf16x8 w[3];
        split8(f, w);
#pragma unroll
        for (int x = 0; x < 3; ++x)
            if (x < pieces)
                *reinterpret_cast<bf16x8*>(base + ((e * pieces + x) * kC + s0 + t) * width + d) = w[x];
    };
    if (role == 2) {
        const int W8 = Dv / 8;
#pragma unroll 4
        for (int i = tid; i < PT * W8; i += PREP_THREADS) {
            const int t = i / W8, d = (i - t * W8) * 8;
            float f[8] = {};
            if (t < nt) {
                load8(proj + (row0 + t) * ld + v_off + (long long)hd * Dv + d, vec & 1, f);
#pragma unroll
                for (int x = 0; x < 8; ++x)
                    if (!isfinite(f[x])) {
                        f[x] = 0.f;
                        atomicMax(bad + e * Dv + d + x, kC - (s0 + t));
                        atomicMax(flag + e, 1);
                    }
            }
            put(v3, NB, Dv, t, d, f);
        }
        return;
    }
    if (role == 1) {
        if (tid < PT) fade[tid] = tid < nt ? powf(decay[hd], (float)(chunk_n - 1 - (s0 + tid))) : 0.f;
        __syncthreads();
    }
    bf16* out = role == 0 ? q3 : k3;
    const T* src = proj + row0 * ld + (role == 0 ? q_off : k_off) + hd * D;
    const float scale = role == 0 ? 1.f : kscale;
    const int half = rope_cos != nullptr ? rot / 2 : 0, p0 = half > 0 ? q_start[b] + t0 : 0;
    auto finish = [&](int t, int d, float (&f)[8]) {
        put(out, 3, D, t, d, f);
        if (role == 1) {
            const float a = fade[t];
#pragma unroll
            for (int x = 0; x < 8; ++x) f[x] *= a;
            put(kd3, 3, D, t, d, f);
        }
    };
    auto load = [&](int t, int d, float (&f)[8]) {
        load8(src + t * ld + d, vec & 1, f);
#pragma unroll
        for (int x = 0; x < 8; ++x) f[x] *= scale;
    };
    const bool pairs = half > 0 && halves && (vec & 2);           // an item is two vectors half a rotation apart, or one behind it
    const int items = pairs ? half / 8 + (D - rot) / 8 : D / 8;
#pragma unroll 2
    for (int i = tid; i < PT * items; i += PREP_THREADS) {
        const int t = i / items, x = i - t * items;
        const long long at = half > 0 ? (long long)min(p0 + t, max_pos - 1) * half : 0;
        if (pairs && x < half / 8) {
            const int d = x * 8;
            float u[8] = {}, v[8] = {};
            if (t < nt) {
                float cs[8], sn[8];
                load(t, d, u);
                load(t, d + half, v);
                load8(rope_cos + at + d, 1, cs);
                load8(rope_sin + at + d, 1, sn);
#pragma unroll
                for (int y = 0; y < 8; ++y) {
                    const float a = u[y], g = v[y];
                    u[y] = a * cs[y] - g * sn[y];
                    v[y] = g * cs[y] + a * sn[y];
                }
            }
            finish(t, d, u);
            finish(t, d + half, v);
            continue;
        }
        const int d = pairs ? rot + (x - half / 8) * 8 : x * 8;
        float f[8] = {};
        if (t < nt) {
            load(t, d, f);
            if (!pairs && d < 2 * half) {
                float g[8];
#pragma unroll
                for (int y = 0; y < 8; ++y) {
                    const int dd = d + y;
                    g[y] = f[y];
                    if (dd >= 2 * half) continue;
                    const bool first = halves ? dd < half : (dd & 1) == 0;
                    const int j = halves ? (first ? dd : dd - half) : dd / 2;
                    const float cs = rope_cos[at + j], sn = rope_sin[at + j];
                    const float o = halves ? ldf(src + t * ld + (first ? dd + half : dd - half)) * scale : f[y ^ 1];
                    g[y] = first ? f[y] * cs - o * sn : f[y] * cs + o * sn;
                }
#pragma unroll
                for (int y = 0; y < 8; ++y) f[y] = g[y];
            }
        }
        finish(t, d, f);
    }
}

// grid (ceil(D * Dv / 4 / 256), H, B): a thread walks the chunks of four state elements, four chunks' loads in flight.
// s3 [E][3][D][Dv] <- pieces of the state at the start of every chunk; the line's state <- state after the step.
__global__ void __launch_bounds__(256)
retention_tc_states_kernel(const float* __restrict__ U, bf16* __restrict__ s3, float* __restrict__ state,
                           const float* __restrict__ decay, const int* __restrict__ flag, const int* __restrict__ bad,
                           const int* __restrict__ q_start, const int* __restrict__ n_new, const int* __restrict__ seq_ids, int Tn,
                           int NC, int H, int Dv, long long E4) {
    pdl_trigger();
    pdl_wait();
    const long long at = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (at >= E4) return;
    const int hd = blockIdx.y, b = blockIdx.z, j = (int)(at * 4 % Dv);
    const int n = n_new != nullptr ? min(n_new[b], Tn) : Tn;
    const int line = seq_ids != nullptr ? seq_ids[b] : b;
    float4* home = reinterpret_cast<float4*>(state) + ((long long)line * H + hd) * E4 + at;
    float4 s = q_start[b] == 0 ? make_float4(0.f, 0.f, 0.f, 0.f) : *home;
    const float a = decay[hd], whole = powf(a, (float)kC);
    const long long e0 = ((long long)b * H + hd) * NC;
    constexpr int AHEAD = 4;
    for (int c0 = 0; c0 < NC; c0 += AHEAD) {
        float4 u[AHEAD];
#pragma unroll
        for (int i = 0; i < AHEAD; ++i)
            u[i] = c0 + i < NC ? reinterpret_cast<const float4*>(U)[(e0 + c0 + i) * E4 + at] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) {
            const int c = c0 + i;
            if (c >= NC) break;
            float r[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
            for (int x = 0; x < 3; ++x) {
                bf162 lo = __floats2bfloat162_rn(r[0], r[1]), hi = __floats2bfloat162_rn(r[2], r[3]);
                const float2 l = __bfloat1622float2(lo), g = __bfloat1622float2(hi);
                r[0] -= l.x, r[1] -= l.y, r[2] -= g.x, r[3] -= g.y;
                reinterpret_cast<uint2*>(s3)[((e0 + c) * 3 + x) * E4 + at] =
                    make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
            }
            const int nt = min(kC, n - c * kC);
            if (nt <= 0) continue;
            const float f = nt == kC ? whole : powf(a, (float)nt);
            s = make_float4(fmaf(f, s.x, u[i].x), fmaf(f, s.y, u[i].y), fmaf(f, s.z, u[i].z), fmaf(f, s.w, u[i].w));
            if (flag[e0 + c] != 0) {
                const int* d = bad + (e0 + c) * Dv + j;
                const float nan = __int_as_float(0x7fffffff);
                if (d[0]) s.x = nan;
                if (d[1]) s.y = nan;
                if (d[2]) s.z = nan;
                if (d[3]) s.w = nan;
            }
        }
    }
    if (n > 0) *home = s;
}

struct Layout {      // byte offsets into the workspace
    long long q3, k3, kd3, v3, u, s3, flag, bad, bytes;
};

Layout layout(long long E, int D, int Dv, int NB) {
    auto up = [](long long v) { return (v + 255) / 256 * 256; };
    Layout l;
    const long long qk = up(E * 3 * kC * D * 2), pp = up(E * 3 * kC * kC * 2);
    l.q3 = 0;
    l.k3 = l.q3 + qk;
    l.kd3 = l.k3 + qk;                                   // P's pieces take the decayed keys' place once U is done
    l.v3 = l.kd3 + (qk > pp ? qk : pp);
    l.u = l.v3 + up(E * NB * kC * Dv * 2);
    l.s3 = l.u + up(E * D * Dv * 4);
    l.flag = l.s3 + up(E * 3 * D * Dv * 2);
    l.bad = l.flag + E * 4;
    l.bytes = up(l.bad + E * Dv * 4);
    return l;
}

template <int MODE, int NB>
int launch(const CUtensorMap& a, const CUtensorMap& b, const CUtensorMap& a2, const CUtensorMap& b2, const CUtensorMap& d,
           const Args& p, cudaStream_t st) {
    auto kern = retention_tc_kernel<MODE, NB>;
    NXD_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
    const int clusters = min(nxd_num_sms() / 2, p.E * p.n_tiles);
    NXD_CHECK_CUDA((nxd_launch_pdl(kern, dim3(clusters * 2), dim3(kThreads), kSmem, st, a, b, a2, b2, d, p)));
    NXD_LAUNCH_CHECK();
    return 0;
}

template <typename T, int NB>
int run(const T* proj, long long ld, int q_off, int k_off, int v_off, const float* decay, float* state, float* out, char* work,
        const int* q_start, const int* n_new, const int* seq_ids, int B, int Tn, int H, int D, int Dv, float kscale,
        const float* rope_cos, const float* rope_sin, int rot, int halves, int max_pos, cudaStream_t st) {
    const int NC = (Tn + kC - 1) / kC, E = B * H * NC;
    const Layout l = layout(E, D, Dv, NB);
    bf16 *q3 = (bf16*)(work + l.q3), *k3 = (bf16*)(work + l.k3), *kd3 = (bf16*)(work + l.kd3), *v3 = (bf16*)(work + l.v3);
    bf16 *s3 = (bf16*)(work + l.s3), *p3 = kd3;
    float* u = (float*)(work + l.u);
    int *flag = (int*)(work + l.flag), *bad = (int*)(work + l.bad);
    NXD_CHECK_CUDA(cudaMemsetAsync(flag, 0, l.bytes - l.flag, st));
    const int per = 16 / (int)sizeof(T);
    const int vec = (ld % per == 0 && q_off % per == 0 && k_off % per == 0 && v_off % per == 0 && ((uintptr_t)proj % 16) == 0) |
                    (rot % 16 == 0 && (((uintptr_t)rope_cos | (uintptr_t)rope_sin) % 16) == 0 ? 2 : 0);
    NXD_CHECK_CUDA((nxd_launch_pdl(retention_tc_prep_kernel<T, NB>, dim3(3 * NC * (kC / PT), H, B), dim3(PREP_THREADS), 0, st,
        proj, ld, q_off, k_off, v_off, decay, q3, k3, kd3, v3, flag, bad, q_start, n_new, Tn, NC, H, D, Dv, kscale, rope_cos,
        rope_sin, rot, halves, max_pos, vec)));
    NXD_LAUNCH_CHECK();
    Args p{};
    p.decay = decay; p.n_new = n_new; p.flag = flag; p.bad = bad;
    p.E = E; p.NC = NC; p.H = H; p.Tn = Tn; p.D = D; p.Dv = Dv;
    CUtensorMap mq, mk, mkd, mv, ms, mp_in, mp_out, mu, mo;
    int rc;
    const long long e3 = 3ll * E, cd = (long long)kC * D, cv = (long long)kC * Dv, dv = (long long)D * Dv;
    if ((rc = make_tmap_3d(&mq, q3, D, kC, e3, D, cd, kBK, 128))) return rc;
    if ((rc = make_tmap_3d(&mk, k3, D, kC, e3, D, cd, kBK, kBN / 2))) return rc;
    if ((rc = make_tmap_3d(&mkd, kd3, D, kC, e3, D, cd, 64, kBK))) return rc;
    if ((rc = make_tmap_3d(&mv, v3, Dv, kC, (long long)NB * E, Dv, cv, 64, kBK))) return rc;
    if ((rc = make_tmap_3d(&ms, s3, Dv, D, e3, Dv, dv, 64, kBK))) return rc;
    if ((rc = make_tmap_3d(&mp_in, p3, kC, kC, e3, kC, (long long)kC * kC, kBK, 128))) return rc;
    if ((rc = make_tmap_3d(&mp_out, p3, kC, kC, e3, kC, (long long)kC * kC, 64, 32))) return rc;
    if ((rc = make_tmap_3d(&mu, u, Dv, D, E, Dv, dv, 32, 32, 4))) return rc;
    if ((rc = make_tmap_bhsd(&mo, out, Dv, Tn, H, B, (long long)H * Dv, Dv, (long long)Tn * H * Dv, 32, p.pos_o, 4))) return rc;
    p.n_tiles = (Dv + kBN - 1) / kBN;
    p.k_blocks1 = kC / kBK, p.k_blocks2 = 0;
    if ((rc = launch<kU, NB>(mkd, mv, mkd, mv, mu, p, st))) return rc;
    const long long E4 = dv / 4;
    NXD_CHECK_CUDA((nxd_launch_pdl(retention_tc_states_kernel, dim3((unsigned)((E4 + 255) / 256), H, B), dim3(256), 0, st, u, s3,
        state, decay, flag, bad, q_start, n_new, seq_ids, Tn, NC, H, Dv, E4)));
    NXD_LAUNCH_CHECK();
    p.n_tiles = kC / kBN;
    p.k_blocks1 = D / kBK;
    if ((rc = launch<kP, 3>(mq, mk, mq, mk, mp_out, p, st))) return rc;
    p.n_tiles = (Dv + kBN - 1) / kBN;
    p.k_blocks1 = kC / kBK, p.k_blocks2 = D / kBK;
    return launch<kO, NB>(mp_in, mv, mq, ms, mo, p, st);
}

}  // namespace

// Bytes of workspace of nxd_retention_tc, 0 where it does not apply (key sizes of 64 / 128 / 192 / 256, value sizes in 64s).
NXD_API long long nxd_retention_tc_workspace(int dtype, int B, int Tn, int H, int D, int Dv) {
    if (D % 64 != 0 || D > 256 || Dv % 64 != 0 || D <= 0 || Dv <= 0 || B >= 65536 || H >= 65536) return 0;
    const long long E = (long long)B * H * ((Tn + kC - 1) / kC);
    if (E <= 0 || 3 * E >= (1ll << 30) / 8) return 0;
    return layout(E, D, Dv, dtype == 0 ? 1 : 3).bytes;
}

// As nxd_retention_chunkwise, with `work` of nxd_retention_tc_workspace bytes (256-byte aligned); out and state 16-byte aligned.
NXD_API int nxd_retention_tc(int dtype, const void* proj, long long ld, int q_off, int k_off, int v_off, const float* decay,
                             float* state, float* out, void* work, const int* q_start, const int* n_new, const int* seq_ids,
                             int B, int Tn, int H, int D, int Dv, float kscale, const float* rope_cos, const float* rope_sin,
                             int rot, int halves, int max_pos, void* stream) {
    if (B * Tn == 0) return 0;
    NXD_REQUIRE(rope_cos == nullptr || (rot % 2 == 0 && rot <= D && max_pos > 0), "retention: rotation over %d of %d", rot, D);
    NXD_REQUIRE(nxd_retention_tc_workspace(dtype, B, Tn, H, D, Dv) > 0, "retention: no tensor-core form for %d x %d", D, Dv);
    NXD_REQUIRE((((uintptr_t)out | (uintptr_t)state) & 15) == 0 && ((uintptr_t)work & 255) == 0, "retention: %s", "alignment");
    cudaStream_t st = (cudaStream_t)stream;
    if (dtype == 0)
        return run<bf16, 1>((const bf16*)proj, ld, q_off, k_off, v_off, decay, state, out, (char*)work, q_start, n_new, seq_ids, B,
                            Tn, H, D, Dv, kscale, rope_cos, rope_sin, rot, halves, max_pos, st);
    return run<float, 3>((const float*)proj, ld, q_off, k_off, v_off, decay, state, out, (char*)work, q_start, n_new, seq_ids, B, Tn,
                         H, D, Dv, kscale, rope_cos, rope_sin, rot, halves, max_pos, st);
}
