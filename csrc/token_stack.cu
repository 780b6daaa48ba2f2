// All decoder layers of a token-generation step in one cooperative launch, for one sequence of the plain Llama layer (RMSNorm, fused
// q | k | v projection, rotation, attention over the cache, SwiGLU; bf16 weights, fp32 sums, activations rounded to bf16 where the
// kernels of gemm_smallm.cu and decode_attention.cu round them).
//
// Such a step reads every weight once, and a chain of kernels cannot keep that stream going: each kernel's first weights arrive
// after its launch, and its last sums, its results' way through memory and the next launch leave the memory idle.  Here the weights
// have one ring per CTA: a producer warp walks the CTA's share of all weights of all layers in the order in which they are used, up to
// 192 KB ahead of the eight warps that multiply -- as much as memory delivers in 4 us.  A layer is six steps:
//   q|k|v    norm inside; pairs of rows (d, d + D/2), rotated, to the CTAs that attend; k and v into the cache as well
//   attention  CTA per KV head and part of the keys, which come through the ring like weights; the parts of a head are merged by its CTAs
//   o        adds the stream
//   gate|up  norm inside; pairs of rows (gate j, up j) -> silu(gate) up
//   down     adds the stream
// A CTA has whole rows, and warp w the w-th eighth of every row, so that its share of the activations stays in registers for the whole
// step (fp32 multiply-adds keep up with the stream; tensor cores would want 16 sequences) and no warp waits for another before the
// step's sums.
//
// A token through 16 layers of 2048, 2048 tokens in the cache, and the head: 675 us as a chain of kernels, 578 here.  Four layers and no head,
// 200 / 2048 / 16384 / 131072 tokens: 2048 wide 160 / 164 / 194 / 336 as a chain, 133 / 139 / 164 / 316 here; 3072 wide 223 / 229 / 273 /
// 553 and 196 / 200 / 239 / 521.  A layer takes some 56 thousand clocks, its weights 36 of them.  What is left are the six times that every
// CTA waits for the slowest one (4000 clocks each under load), and instructions: every step's code is fetched once a layer, so it is kept
// short (loops unrolled further and a copy of the products per step: 623 us against 600 at that time).  Copies in flight: 64 KB a CTA; with 32 the stream is slower (649 against 584 at that time),
// with 192 everything else waits behind them (743 against 702).
//
// Waits end: one that has taken `limit` clocks gives up, the CTA sends nothing more and leaves NaN in its part of the result, so all
// others give up too; the caller's word, which may be pinned host memory, and nxd_token_stack_status say so.
#include <cudaTypedefs.h>

#include <type_traits>

#include "attn_tc_common.cuh"
#include "decode_common.cuh"
#include "mma_sync.cuh"
#include "ptx.cuh"

namespace {

using nxd_decode::CacheDst;
using nxd_decode::cache_row;

constexpr int kWarps = 8, kThreads = (kWarps + 1) * 32;
constexpr int kRingBytes = 196608, kPartBytes = 28672;   // the weights; the phase's sums or the warps' attention states
constexpr int kSmem = kRingBytes + kPartBytes;
constexpr int kFlightBytes = 65536;                      // of a CTA's copies in flight
constexpr int kMaxLayers = 64, kPartKeys = 256;
// Parts of a head's keys.  With 18 nearly all CTAs attend, with 16 the others' weights keep the stream going: 4 layers of 2048 / 3072, 8000
// tokens 154 us with 16 and 161 with 18 / 219 and 226, 32768 190 and 192 / 281 and 285, 65536 235 and 233 / 364 and 366, 131072 330 and 316 /
// 526 and 521.
constexpr int kFewParts = 16, kMaxParts = 18, kManyKeys = 65536;
constexpr long long kWaitClocks = 4000000000ll;          // two seconds

struct Layer {
    const bf16 *norm1, *qkv, *o, *norm2, *gate_up, *down;
    bf16 *k, *v;
    float eps1, eps2;
};

// What one CTA hands to others goes through memory as words of four bytes and the number of the layer (from 1 on) that they belong to, so
// that neither side needs a fence or a barrier: who reads a word polls it until the number is there.  (A barrier over the grid instead:
// 1000 to 2700 clocks of fence behind the weights in flight, two or more polls of 600, and then the loads: 637 us a token.)
// A buffer is written again a layer later, when every CTA has read it: each vector needs all rows of the one before, from all CTAs.
typedef unsigned long long word;

struct Args {
    Layer layer[kMaxLayers];
    int layers, H, I, n_q, n_kv;
    const bf16* hidden;                  // [H]
    bf16* out;                           // [H]
    // words of two bf16 values: the stream inside a layer and behind it [H / 2], queries [n_q, D / 2] (d and d + D / 2), the step's
    // keys and values [n_kv, 2, D / 2], attention [H / 2], activations [I / 2]; words of one fp32 value: parts of the attention
    // [n_kv, parts, G D], their maxima and sums [n_kv, parts, G, 2]
    word *mid, *x, *q, *kv, *attn, *act, *part_o, *part_ml;
    const float *cos_t, *sin_t;
    const int *positions, *lengths;
    CacheDst cache;                      // k, v: per layer
    float scale_log2;
    long long limit;
    int* gave_up;                        // the caller's, or null
};

__device__ int stack_gave_up;

__device__ __forceinline__ void consumers() { nxd_attn::named_bar_sync(1, kWarps * 32); }

__device__ __forceinline__ bool wait(uint64_t* bar, uint32_t parity, long long limit, volatile int* dead) {
    long long start = 0;
    for (int i = 1;; ++i) {
        if (limit > 0 && ptx::mbar_try_wait(bar, parity)) return true;
        if (limit > 0 && (i & 63) != 0) continue;
        if (*dead) return false;
        const long long now = clock64();
        if (start == 0) start = now;
        if (now - start < limit) continue;
        *dead = 1;
        return false;
    }
}

__device__ __forceinline__ void send(word* dst, uint32_t value, int number) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(dst), "l"((word)(uint32_t)number << 32 | value) : "memory");
}
__device__ __forceinline__ ulonglong2 look(const word* src) {        // two neighbouring words
    ulonglong2 v;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(src) : "memory");
    return v;
}
// N pairs of words, once all of them have that number
template <int N, typename At>
__device__ __forceinline__ bool receive(At at, int number, uint2 (&out)[N], long long limit, volatile int* dead) {
    long long start = 0;
    for (int i = 1;; ++i) {
        bool all = limit > 0;
#pragma unroll
        for (int j = 0; j < N; ++j) {
            const ulonglong2 v = look(at(j));
            all = all && (int)(v.x >> 32) == number && (int)(v.y >> 32) == number;
            out[j] = make_uint2((uint32_t)v.x, (uint32_t)v.y);
        }
        if (all) return true;
        if (limit > 0 && (i & 15) != 0) continue;
        if (*dead) return false;
        const long long now = clock64();
        if (start == 0) start = now;
        if (now - start < limit) continue;
        *dead = 1;
        return false;
    }
}
__device__ __forceinline__ uint32_t two(float lo, float hi) {
    const bf162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}

// four bf16 values of two registers -> two pairs of fp32
__device__ __forceinline__ void widen(uint2 w, uint64_t (&f)[2]) {
    f[0] = f2_pack(__uint_as_float(w.x << 16), __uint_as_float(w.x & 0xffff0000u));
    f[1] = f2_pack(__uint_as_float(w.y << 16), __uint_as_float(w.y & 0xffff0000u));
}
__device__ __forceinline__ float rounded(float v) { return __bfloat162float(__float2bfloat16(v)); }

__device__ __forceinline__ float largest(float v) {      // of a warp; sm_100a
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// R sums over the lanes at once: the lanes with the same lane / (32 / R) end with that sum
template <int R>
__device__ __forceinline__ float sum_rows(float (&a)[R]) {
    const int lane = threadIdx.x & 31;
    int off = 16;
#pragma unroll
    for (int n = R; n > 1; n /= 2, off /= 2) {
        const bool upper = lane & off;
#pragma unroll
        for (int i = 0; i < n / 2; ++i) {
            const float keep = upper ? a[i + n / 2] : a[i], send = upper ? a[i] : a[i + n / 2];
            a[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
        }
    }
#pragma unroll
    for (; off > 0; off /= 2) a[0] += __shfl_xor_sync(0xffffffffu, a[0], off);
    return a[0];
}

// Rows of NV * 1024 values: as many as a slot takes, in powers of two
constexpr int rows_per_slot(int NV, int slot) {
    int r = 8;
    while (r > 1 && r * NV * 2048 > slot) r /= 2;
    return r;
}

// This warp's eighth of R rows times its share of the activations -> sums over the lane's values
template <int NV, int R, int BATCH>
__device__ __forceinline__ void multiply(const uint8_t* mine, const uint64_t (&x)[NV][2], float (&acc)[BATCH], int first) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
        uint64_t a = 0;
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            uint64_t w[2];
            widen(*reinterpret_cast<const uint2*>(mine + r * (NV * 2048) + v * 256), w);
            a = f2_fma(w[0], x[v][0], a);
            a = f2_fma(w[1], x[v][1], a);
        }
        acc[first + r] = f2_lo(a) + f2_hi(a);
    }
}

// grid: one CTA per SM, all resident (cooperative launch).  H = n_q D = NVH * 1024, I = NVI * 1024, G query heads per KV head.
template <int NVH, int NVI, int D, int G>
__global__ void __launch_bounds__(kThreads, 1) token_stack_kernel(const __grid_constant__ Args p) {
    constexpr int kSlotBytes = 32768, kSlots = kRingBytes / kSlotBytes, kFlight = kFlightBytes / kSlotBytes;
    constexpr int RH = rows_per_slot(NVH, kSlotBytes), RI = rows_per_slot(NVI, kSlotBytes), KH = NVH * 1024, KI = NVI * 1024;
    constexpr int kKeys = kSlotBytes / (4 * D);              // of a slot: rows of keys, then of values
    static_assert(RH >= 2 && RH * NVH * 2048 <= kSlotBytes && RI * NVI * 2048 <= kSlotBytes && 128 % kKeys == 0, "a slot holds whole pairs of rows");
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ uint64_t full[kSlots], empty[kSlots];
    __shared__ float red[kWarps];
    __shared__ volatile int dead;
    __shared__ int verdict;
    float* part = reinterpret_cast<float*>(smem + kSlots * kSlotBytes);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int cta = blockIdx.x, ctas = gridDim.x;
    if (tid == 0) {
        for (int i = 0; i < kSlots; ++i) {
            ptx::mbar_init(&full[i], 1);
            ptx::mbar_init(&empty[i], kWarps);
        }
        dead = 0;
        ptx::fence_barrier_init();
    }
    __syncthreads();

    // this CTA's units: pairs of rows of q | k | v and of gate | up, rows of o and down
    auto first_of = [&](int n, int c) { return (int)((long long)n * c / ctas); };
    const int n_qkv = (p.n_q + 2 * p.n_kv) * (D / 2);
    const int qkv0 = first_of(n_qkv, cta), qkvs = first_of(n_qkv, cta + 1) - qkv0;
    const int h0 = 2 * first_of(KH / 2, cta), hs = 2 * first_of(KH / 2, cta + 1) - h0;
    const int i0 = 2 * first_of(KI / 2, cta), is = 2 * first_of(KI / 2, cta + 1) - i0;

    // attention: parts of kPartKeys keys, one for a CTA at most
    const int length = p.lengths[0], position = p.positions[0];
    const int parts = max(1, min(min((length + kPartKeys - 1) / kPartKeys, length > kManyKeys ? kMaxParts : kFewParts), ctas / p.n_kv));
    const bool attends = cta < p.n_kv * parts;
    const int kv_head = cta / parts, my_part = cta % parts;
    const int keys_per = ((length + parts - 1) / parts + 127) / 128 * 128, key0 = my_part * keys_per;
    const int keys = attends ? max(0, min(length, key0 + keys_per) - key0) : 0;

    if (warp == kWarps) {
        if (lane != 0) return;
        int st = 0, issued = 0;
        uint32_t ph = 1;
        bool live = true;
        // the next slot, once it is free and enough of the copies before it have landed
        auto claim = [&](uint32_t bytes) {
            const int i = issued - kFlight;
            live = live && wait(&empty[st], ph, p.limit, &dead) && (i < 0 || wait(&full[i % kSlots], (uint32_t)(i / kSlots) & 1, p.limit, &dead));
            if (live) ptx::mbar_arrive_expect_tx(&full[st], bytes);
            return live;
        };
        auto put = [&](int at, const void* src, int bytes) { nxd_attn::bulk_load_1d(smem + st * kSlotBytes + at, src, (uint32_t)bytes, &full[st]); };
        auto next = [&] {
            ++issued;
            if (++st == kSlots) st = 0, ph ^= 1;
        };
        auto fill = [&](const bf16* w, int K, int R, int rows, bool in_a_row, auto row_of) {
            for (int r0 = 0; r0 < rows; r0 += R) {
                const int n = min(R, rows - r0);
                if (!claim(n * K * 2)) return;
                if (in_a_row) put(0, w + (long long)row_of(r0) * K, n * K * 2);
                else
                    for (int i = 0; i < n; ++i) put(i * K * 2, w + (long long)row_of(r0 + i) * K, K * 2);
                next();
            }
        };
        for (int l = 0; live && l < p.layers; ++l) {
            const Layer& w = p.layer[l];
            fill(w.qkv, KH, RH, 2 * qkvs, false, [&](int r) {
                const int u = qkv0 + r / 2;
                return u / (D / 2) * D + u % (D / 2) + (r & 1) * (D / 2);
            });
            for (int k0 = 0; k0 < keys; k0 += kKeys) {   // rows that lie in a row: all of them, or up to a page's end
                const int n = min(kKeys, keys - k0);
                if (!claim(n * D * 4)) break;
                for (int i = 0; i < n;) {
                    const int pos = key0 + k0 + i, run = p.cache.block_table ? min(n - i, p.cache.page_size - pos % p.cache.page_size) : n;
                    const size_t row = cache_row(p.cache, 0, kv_head, pos, D);
                    put(i * D * 2, w.k + row, run * D * 2);
                    put((kKeys + i) * D * 2, w.v + row, run * D * 2);
                    i += run;
                }
                next();
            }
            fill(w.o, KH, RH, hs, true, [&](int r) { return h0 + r; });
            fill(w.gate_up, KH, RH, 2 * is, false, [&](int r) { return i0 + r / 2 + (r & 1) * KI; });
            fill(w.down, KI, RI, hs, true, [&](int r) { return h0 + r; });
        }
        if (!live) {                     // copies in flight still land in this CTA's memory
            int none = 0;
            for (int j = max(0, issued - kSlots); j < issued; ++j)
                wait(&full[j % kSlots], (uint32_t)(j / kSlots) & 1, kWaitClocks, &none);
        }
        return;
    }

    int st = 0;
    uint32_t ph = 0;
    // the sums over the lanes of BATCH rows at once: a chain of shuffles per slot would take longer than its loads
    constexpr int BATCH = 8;
    auto rows_times = [&](auto nv, const auto& x, int rows) {
        constexpr int NV = decltype(nv)::value, R = rows_per_slot(NV, kSlotBytes), N = R < BATCH ? BATCH : R;
        bool live = true;
        for (int r0 = 0; live && r0 < rows; r0 += N) {
            float acc[N];
#pragma unroll
            for (int r = 0; r < N; r += R) {
                if (!live || r0 + r >= rows) {
#pragma unroll
                    for (int i = 0; i < R; ++i) acc[r + i] = 0.f;
                    continue;
                }
                live = __all_sync(0xffffffffu, wait(&full[st], ph, p.limit, &dead));
                multiply<NV, R, N>(smem + st * kSlotBytes + warp * (NV * 256) + lane * 8, x, acc, r);
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(&empty[st]);
                if (++st == kSlots) st = 0, ph ^= 1;
            }
            const float sum = sum_rows<N>(acc);
            const int row = r0 + lane / (32 / N);
            if (lane % (32 / N) == 0 && row < rows) part[row * kWarps + warp] = sum;
        }
        consumers();
    };
    auto sum_of = [&](int row) {
        const float4* s = reinterpret_cast<const float4*>(part + row * kWarps);
        const float4 a = s[0], c = s[1];
        return ((a.x + a.y) + (a.z + a.w)) + ((c.x + c.y) + (c.z + c.w));
    };
    // this warp's share of a vector
    const int base_h = warp * (NVH * 128) + lane * 4, base_i = warp * (NVI * 128) + lane * 4;
    auto h_words = [&](const word* src) {
        return [=](int v) { return src + (base_h + v * 128) / 2; };
    };
    // norm weights come from memory, behind the weights in flight: they are asked for a phase ahead
    auto norm_weights = [&](const bf16* weight, uint2 (&w)[NVH]) {
#pragma unroll
        for (int v = 0; v < NVH; ++v) w[v] = *reinterpret_cast<const uint2*>(weight + base_h + v * 128);
    };
    auto normalised = [&](const word* src, int number, const uint2 (&w)[NVH], float eps, uint64_t (&x)[NVH][2]) {
        uint2 raw[NVH];
        if (number == 0) {
#pragma unroll
            for (int v = 0; v < NVH; ++v) raw[v] = *reinterpret_cast<const uint2*>(p.hidden + base_h + v * 128);
        } else {
            receive(h_words(src), number, raw, p.limit, &dead);
        }
        uint64_t ss = 0;
#pragma unroll
        for (int v = 0; v < NVH; ++v) {
            widen(raw[v], x[v]);
            ss = f2_fma(x[v][0], x[v][0], ss);
            ss = f2_fma(x[v][1], x[v][1], ss);
        }
        const float mine = warp_sum(f2_lo(ss) + f2_hi(ss));
        if (lane == 0) red[warp] = mine;
        consumers();
        float all = 0.f;
#pragma unroll
        for (int i = 0; i < kWarps; ++i) all += red[i];
        const float rstd = rsqrtf(all / (float)KH + eps);
#pragma unroll
        for (int v = 0; v < NVH; ++v) {
            uint64_t f[2];
            widen(w[v], f);
#pragma unroll
            for (int i = 0; i < 2; ++i)
                x[v][i] = f2_pack(rounded(f2_lo(x[v][i]) * rstd * f2_lo(f[i])), rounded(f2_hi(x[v][i]) * rstd * f2_hi(f[i])));
        }
    };
    using NVh = std::integral_constant<int, NVH>;
    using NVi = std::integral_constant<int, NVI>;

    // the stream's values of this thread's pair of rows, inside a layer and behind it
    const int pair_r = 2 * tid;
    const bool has_pair = pair_r < hs;
    float2 stream = make_float2(0.f, 0.f), mid = stream;
    if (has_pair) stream = __bfloat1622float2(*reinterpret_cast<const bf162*>(p.hidden + h0 + pair_r));
    uint2 norm_w[NVH];
    norm_weights(p.layer[0].norm1, norm_w);
    // this thread's pair of q | k | v: its angle does not change from layer to layer
    const int rot_head = (qkv0 + tid) / (D / 2), rot_d = (qkv0 + tid) % (D / 2);
    const bool has_rot = tid < qkvs;
    float rot_cos = 1.f, rot_sin = 0.f;
    if (has_rot && rot_head < p.n_q + p.n_kv)
        rot_cos = p.cos_t[(size_t)position * (D / 2) + rot_d], rot_sin = p.sin_t[(size_t)position * (D / 2) + rot_d];
    for (int l = 0; l < p.layers; ++l) {
        const Layer& w = p.layer[l];
        const int number = l + 1;
        CacheDst cache = p.cache;
        cache.k = w.k, cache.v = w.v;
        // q | k | v, o, gate | up: one copy of the code that multiplies, which would be fetched anew for every step
#pragma unroll 1
        for (int step = 0; step < 3; ++step) {
            uint64_t x[NVH][2];
            if (step == 1) {
                // attention.  Keys and values come through the ring, ahead of the activations; only the step's own row had not been written
                // then, and goes into its slot here.  Four warps take 128 keys and the other four the next 128, a warp a quarter of a slot at
                // a time: the tiles, and so the weights that are rounded to bf16 beside their tiles' largest ones, are those of
                // decode_attn_mma_kernel.  Scores on mma.sync, keys as its 16 rows and the group's query heads as its 8 columns; its 16 terms
                // are taken from the row in an order in which every lane loads 16 bytes at once.  Values by multiply-adds of pairs, eight
                // lanes a row (as mma.sync operands they would have to be transposed, eight rows of one bank at a time).  A slot then takes
                // less than the memory does: with the scores by multiply-adds and shuffles too, 2600 clocks against 1200, and beyond 20000
                // tokens the chain of kernels was faster (figures above; 131072 tokens 498 and 731 us).
                if (attends) {
                    constexpr int kE = D / 8, kV = kE / 8, kTile = kKeys / 4, kHalf = D / 2, kWords = 4 * kV;
                    static_assert(G <= 4 && kTile % 16 == 0 && kTile <= 32, "a lane for every key of a tile, columns for its heads");
                    const int sub = lane >> 3, l8 = lane & 7, row = lane >> 2, t4 = lane & 3, own = position - key0;
                    float m[G], sum[G];
                    uint64_t o[G][kE / 2];
                    uint4 qb[D / 32];                            // of query head lane / 4: values 32 i + 8 (lane % 4) and the next seven
                    uint4 own_k[kV], own_v[kV];
                    {
                        // a word holds the values d and d + D / 2
                        const int head = kv_head * G + min(row, G - 1), d0 = D == 64 ? (l8 & 3) * 8 : l8 * 8;
                        uint2 raw[kWords + 8];
                        receive(
                            [&](int j) {
                                return j < kWords ? p.q + head * kHalf + t4 * 8 + j / 4 * 32 + j % 4 * 2
                                                  : p.kv + (kv_head * 2 + (j - kWords) / 4) * kHalf + d0 + j % 4 * 2;
                            },
                            number, raw, p.limit, &dead);
                        auto eight = [&](int first, bool upper) {
                            uint32_t r[4];
#pragma unroll
                            for (int i = 0; i < 4; ++i) r[i] = __byte_perm(raw[first + i].x, raw[first + i].y, upper ? 0x7632 : 0x5410);
                            return make_uint4(r[0], r[1], r[2], r[3]);
                        };
#pragma unroll
                        for (int i = 0; i < D / 32; ++i) {
                            qb[i] = eight(i % kV * 4, i >= kV);
                            if (row >= G) qb[i] = make_uint4(0, 0, 0, 0);
                        }
#pragma unroll
                        for (int v = 0; v < kV; ++v) {
                            const bool upper = D == 64 ? l8 >= 4 : v == 1;
                            own_k[v] = eight(kWords, upper);
                            own_v[v] = eight(kWords + 4, upper);
                        }
                    }
#pragma unroll
                    for (int g = 0; g < G; ++g) {
                        m[g] = -INFINITY, sum[g] = 0.f;
#pragma unroll
                        for (int e = 0; e < kE / 2; ++e) o[g][e] = 0;
                    }
                    // the tile's scores, then its weights, each twice: what a multiply-add of a pair takes
                    float* const scores = part + 4096 + warp * 256;
                    ulonglong2* const weights = reinterpret_cast<ulonglong2*>(scores);
                    for (int kb = 0; kb < keys; kb += kKeys) {
                        const bool ours = kb / 128 % 2 == warp / 4;
                        // the warps that skip a slot wait for it as well: `empty` counts arrivals, not warps, and one that is ahead by a round of
                        // the ring would arrive a second time in the place of one that still reads
                        if (!__all_sync(0xffffffffu, wait(&full[st], ph, p.limit, &dead))) break;
                        const int first = warp % 4 * kTile;                  // of the slot's keys
                        uint8_t* const kt = smem + st * kSlotBytes + first * D * 2;
                        const uint8_t* const vt = kt + kKeys * D * 2;
                        if (ours) {
                            if (own >= kb + first && own < kb + first + kTile) {
                                if (sub == 0) {
#pragma unroll
                                    for (int v = 0; v < kV; ++v) {
                                        const int at = (own - kb - first) * D * 2 + (l8 + v * 8) * 16;
                                        *reinterpret_cast<uint4*>(kt + at) = own_k[v];
                                        *reinterpret_cast<uint4*>(kt + kKeys * D * 2 + at) = own_v[v];
                                    }
                                }
                                ptx::fence_proxy_async();                    // the slot's next copy comes behind these stores
                                __syncwarp();
                            }
#pragma unroll
                            for (int r0 = 0; r0 < kTile; r0 += 16) {
                                float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                                for (int i = 0; i < D / 32; ++i) {
                                    const uint4 a = *reinterpret_cast<const uint4*>(kt + (r0 + row) * D * 2 + (t4 + 4 * i) * 16);
                                    const uint4 b = *reinterpret_cast<const uint4*>(kt + (r0 + row + 8) * D * 2 + (t4 + 4 * i) * 16);
                                    const uint32_t lo[4] = {a.x, b.x, a.y, b.y}, hi[4] = {a.z, b.z, a.w, b.w};
                                    mma::mma16816(c, lo, qb[i].x, qb[i].y);
                                    mma::mma16816(c, hi, qb[i].z, qb[i].w);
                                }
                                if (t4 < 2) {
                                    *reinterpret_cast<float2*>(scores + (r0 + row) * 4 + 2 * t4) = make_float2(c[0], c[1]);
                                    *reinterpret_cast<float2*>(scores + (r0 + row + 8) * 4 + 2 * t4) = make_float2(c[2], c[3]);
                                }
                            }
                            __syncwarp();
                            float sc[4];                                     // the scores of the lane's key
                            *reinterpret_cast<float4*>(sc) = *reinterpret_cast<const float4*>(scores + lane % kTile * 4);
                            __syncwarp();
                            const bool mine = lane < kTile && kb + first + lane < keys;
#pragma unroll
                            for (int g = 0; g < G; ++g) {
                                const float t = mine ? sc[g] * p.scale_log2 : -INFINITY;
                                const float top = fmaxf(m[g], largest(t)), use = top == -INFINITY ? 0.f : top, fade = exp2f(m[g] - use);
                                m[g] = top;
                                const float exact = exp2f(t - use);
                                sum[g] = fmaf(sum[g], fade, exact);
                                sc[g] = rounded(exact);
                                const uint64_t fades = f2_pack(fade, fade);
#pragma unroll
                                for (int e = 0; e < kE / 2; ++e) o[g][e] = f2_mul(o[g][e], fades);
                            }
                            if (lane < kTile) {
                                weights[lane * 2] = make_ulonglong2(f2_pack(sc[0], sc[0]), f2_pack(sc[1], sc[1]));
                                weights[lane * 2 + 1] = make_ulonglong2(f2_pack(sc[2], sc[2]), f2_pack(sc[3], sc[3]));
                            }
                            __syncwarp();
                            const bool whole = kb + first + kTile <= keys;
#pragma unroll(D == 64 ? 4 : 1)
                            for (int u = 0; u < kTile; u += 4) {
                                uint64_t v[kE / 2];
#pragma unroll
                                for (int i = 0; i < kV; ++i) {
                                    const uint4 raw = *reinterpret_cast<const uint4*>(vt + (u + sub) * D * 2 + (l8 + i * 8) * 16);
                                    uint64_t f[2];
                                    widen(make_uint2(raw.x, raw.y), f);
                                    v[i * 4] = f[0], v[i * 4 + 1] = f[1];
                                    widen(make_uint2(raw.z, raw.w), f);
                                    v[i * 4 + 2] = f[0], v[i * 4 + 3] = f[1];
                                }
                                if (!whole && kb + first + u + sub >= keys) {                // what lies behind the last key may be anything
#pragma unroll
                                    for (int e = 0; e < kE / 2; ++e) v[e] = 0;
                                }
                                const ulonglong2 w01 = weights[(u + sub) * 2], w23 = weights[(u + sub) * 2 + 1];
                                const uint64_t w[4] = {w01.x, w01.y, w23.x, w23.y};
#pragma unroll
                                for (int g = 0; g < G; ++g)
#pragma unroll
                                    for (int e = 0; e < kE / 2; ++e) o[g][e] = f2_fma(w[g], v[e], o[g][e]);
                            }
                        }
                        __syncwarp();
                        if (lane == 0) ptx::mbar_arrive(&empty[st]);
                        if (++st == kSlots) st = 0, ph ^= 1;
                    }
                    constexpr int kRow = D + 4;                  // values, maximum, sum
#pragma unroll
                    for (int g = 0; g < G; ++g) {
                        const float t = warp_sum(sum[g]);
                        float* dst = part + (warp * G + g) * kRow;
#pragma unroll
                        for (int e = 0; e < kE; ++e) {
                            float y = e % 2 == 0 ? f2_lo(o[g][e / 2]) : f2_hi(o[g][e / 2]);
                            y += __shfl_xor_sync(0xffffffffu, y, 8);
                            y += __shfl_xor_sync(0xffffffffu, y, 16);
                            if (sub == 0) dst[(e / 8) * 64 + l8 * 8 + e % 8] = y;
                        }
                        if (lane == 0) dst[D] = m[g], dst[D + 1] = t;
                    }
                    consumers();
                    word* const mine = p.part_o + (size_t)cta * (G * D);             // [kv_head, part] is this CTA's number
                    for (int i = tid; i < G * D && !dead; i += kWarps * 32) {
                        const int g = i / D, d = i - g * D;
                        float top = -INFINITY, t = 0.f, y = 0.f;
#pragma unroll
                        for (int x = 0; x < kWarps; ++x) top = fmaxf(top, part[(x * G + g) * kRow + D]);
#pragma unroll
                        for (int x = 0; x < kWarps; ++x) {
                            const float* src = part + (x * G + g) * kRow;
                            const float f = src[D] == -INFINITY ? 0.f : exp2f(src[D] - top);
                            t = fmaf(src[D + 1], f, t);
                            y = fmaf(src[d], f, y);
                        }
                        send(mine + i, __float_as_uint(y), number);
                        if (d == 0) {
                            send(p.part_ml + ((size_t)cta * G + g) * 2, __float_as_uint(top), number);
                            send(p.part_ml + ((size_t)cta * G + g) * 2 + 1, __float_as_uint(t), number);
                        }
                    }
                    // this CTA's share of the values of all parts, a pair of them a thread
                    const int v0 = G * D / 2 * my_part / parts, v1 = G * D / 2 * (my_part + 1) / parts, first = cta - my_part;
                    for (int i = v0 + tid; i < v1; i += kWarps * 32) {
                        const int g = 2 * i / D;
                        float top = -INFINITY, t = 0.f, y0 = 0.f, y1 = 0.f;
                        for (int s0 = 0; s0 < parts; s0 += 4) {
                            uint2 raw[8];                                            // of four parts: the pair of values, maximum and sum
                            receive(
                                [&](int j) {
                                    const size_t c = first + min(s0 + j / 2, parts - 1);
                                    return j % 2 == 0 ? p.part_o + c * (G * D) + 2 * i : p.part_ml + (c * G + g) * 2;
                                },
                                number, raw, p.limit, &dead);
                            float now = top;
#pragma unroll
                            for (int j = 0; j < 4; ++j) now = fmaxf(now, __uint_as_float(raw[2 * j + 1].x));
                            const float use = now == -INFINITY ? 0.f : now, fade = exp2f(top - use);
                            top = now, t *= fade, y0 *= fade, y1 *= fade;
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                const float f = s0 + j < parts ? exp2f(__uint_as_float(raw[2 * j + 1].x) - use) : 0.f;
                                t = fmaf(__uint_as_float(raw[2 * j + 1].y), f, t);
                                y0 = fmaf(__uint_as_float(raw[2 * j].x), f, y0);
                                y1 = fmaf(__uint_as_float(raw[2 * j].y), f, y1);
                            }
                        }
                        const float inv = t > 0.f ? 1.f / t : 0.f;
                        if (!dead) send(p.attn + kv_head * (G * D / 2) + i, two(y0 * inv, y1 * inv), number);
                    }
                }
                uint2 raw[NVH];
                receive(h_words(p.attn), number, raw, p.limit, &dead);
#pragma unroll
                for (int v = 0; v < NVH; ++v) widen(raw[v], x[v]);
                consumers();                 // the warps' states or sums have been read
            } else {
                normalised(step == 0 ? p.x : p.mid, step == 0 ? l : number, norm_w, step == 0 ? w.eps1 : w.eps2, x);
            }
            rows_times(NVh(), x, step == 0 ? 2 * qkvs : step == 1 ? hs : 2 * is);
            if (step == 0) {
                if (has_rot && !dead) {
                    const float y = rounded(sum_of(2 * tid)), z = rounded(sum_of(2 * tid + 1));
                    // values go over as they are: turned by nothing, one that is not finite would reach its partner as inf * 0
                    const bool turned = rot_head < p.n_q + p.n_kv;
                    const float lo = turned ? y * rot_cos - z * rot_sin : y, hi = turned ? z * rot_cos + y * rot_sin : z;
                    if (rot_head < p.n_q) {
                        send(p.q + rot_head * (D / 2) + rot_d, two(lo, hi), number);
                    } else {
                        const bool value = !turned;
                        const int kvh = rot_head - p.n_q - (value ? p.n_kv : 0);
                        send(p.kv + (kvh * 2 + value) * (D / 2) + rot_d, two(lo, hi), number);
                        bf16* dst = (value ? cache.v : cache.k) + cache_row(cache, 0, kvh, position, D);
                        dst[rot_d] = __float2bfloat16(lo);
                        dst[rot_d + D / 2] = __float2bfloat16(hi);
                    }
                }
                norm_weights(w.norm2, norm_w);
                if (attends) consumers();    // the sums have been read
            } else if (step == 1) {
                if (has_pair && !dead) {
                    const uint32_t v = two(sum_of(pair_r) + stream.x, sum_of(pair_r + 1) + stream.y);
                    mid = __bfloat1622float2(*reinterpret_cast<const bf162*>(&v));
                    send(p.mid + (h0 + pair_r) / 2, v, number);
                }
            } else {
                if (2 * tid < is && !dead) {
                    float y[2];
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const float g = rounded(sum_of(4 * tid + 2 * j)), up = rounded(sum_of(4 * tid + 2 * j + 1));
                        y[j] = g / (1.f + __expf(-g)) * up;
                    }
                    send(p.act + i0 / 2 + tid, two(y[0], y[1]), number);
                }
            }
        }

        if (number < p.layers) norm_weights(p.layer[number].norm1, norm_w);
        {
            uint64_t x[NVI][2];
            uint2 raw[NVI];
            receive([&](int v) { return p.act + (base_i + v * 128) / 2; }, number, raw, p.limit, &dead);
#pragma unroll
            for (int v = 0; v < NVI; ++v) widen(raw[v], x[v]);
            consumers();                     // the sums have been read
            rows_times(NVi(), x, hs);
        }
        if (has_pair && !dead) {
            const uint32_t v = two(sum_of(pair_r) + mid.x, sum_of(pair_r + 1) + mid.y);
            stream = __bfloat1622float2(*reinterpret_cast<const bf162*>(&v));
            if (number < p.layers) send(p.x + (h0 + pair_r) / 2, v, number);
            else *reinterpret_cast<uint32_t*>(p.out + h0 + pair_r) = v;
        }
        consumers();
        if (tid == 0) verdict = dead;        // one answer for all warps: some may give up while others have not asked yet
        consumers();
        if (verdict != 0) break;
    }
    if (verdict != 0) {
        if (tid == 0) {
            stack_gave_up = 1;
            if (p.gave_up != nullptr) *reinterpret_cast<volatile int*>(p.gave_up) = 1;
        }
        if (has_pair) *reinterpret_cast<uint32_t*>(p.out + h0 + pair_r) = 0x7fff7fffu;
    }
}

struct Scratch {             // words, all zero before the launch
    long long mid, x, q, kv, attn, act, part_o, part_ml, words;
};

Scratch scratch_of(int H, int I, int n_q, int n_kv, int D) {
    Scratch s;
    long long at = 0;
    auto take = [&](long long words) {
        const long long here = at;
        at += (words + 31) / 32 * 32;
        return here;
    };
    s.mid = take(H / 2), s.x = take(H / 2), s.q = take(H / 2), s.kv = take(n_kv * D), s.attn = take(H / 2), s.act = take(I / 2);
    s.part_o = take((long long)n_q * kMaxParts * D), s.part_ml = take(2ll * n_q * kMaxParts);
    s.words = at;
    return s;
}

template <int NVH, int NVI, int D, int G>
int launch(const Args& a, long long words, cudaStream_t st) {
    constexpr auto kernel = token_stack_kernel<NVH, NVI, D, G>;
    NXD_CHECK_CUDA(nxd_allow_smem<kernel>(kSmem));
    NXD_CHECK_CUDA(cudaMemsetAsync(a.mid, 0, (size_t)words * sizeof(word), st));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)nxd_num_sms());
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    NXD_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kernel, a));
    NXD_LAUNCH_CHECK();
    return 0;
}

// The layers that are compiled: hidden size / 1024 (query heads x head size as well), feed-forward / 1024, head size, group.  words 0: asks
int dispatch(const Args& a, int D, long long words, cudaStream_t st) {
    const int g = a.n_q / a.n_kv;
    if (a.H == 2048 && a.I == 8192 && D == 64 && g == 4) return words ? launch<2, 8, 64, 4>(a, words, st) : 0;
    if (a.H == 3072 && a.I == 8192 && D == 128 && g == 3) return words ? launch<3, 8, 128, 3>(a, words, st) : 0;
    return -1;
}

}  // namespace

// Bytes of scratch (256-byte aligned) with which nxd_token_stack runs a step of B sequences through such layers, 0 where it does not:
// one sequence (of several, every phase waits longer for its activations, and the tensor cores' kernels take no longer than for one).
NXD_API long long nxd_token_stack_scratch(int layers, int B, int H, int I, int n_q, int n_kv, int D) {
    if (layers < 1 || layers > kMaxLayers || B != 1 || n_kv < 1 || n_q % n_kv != 0 || n_q * D != H) return 0;
    Args a;
    a.H = H, a.I = I, a.n_q = n_q, a.n_kv = n_kv;
    const int sms = nxd_num_sms();
    // a CTA's rows: sums in shared memory, and a thread for every pair of them
    const int most = 2 * ((max(I, (n_q + 2 * n_kv) * (D / 2)) / 2 + sms - 1) / sms);
    if (dispatch(a, D, 0, nullptr) != 0 || 2 * most * kWarps * 4 > kPartBytes || most > kWarps * 32 || n_kv > sms ||
        kWarps * (n_q / n_kv) * (D + 4) * 4 > kPartBytes)
        return 0;
    return scratch_of(H, I, n_q, n_kv, D).words * (long long)sizeof(word);
}

// Whether a CTA on every SM of the device can be resident on that stream: not if it belongs to a green context of fewer SMs, where such a
// cooperative launch fails (and a chain of kernels runs).
NXD_API int nxd_token_stack_runs_on(void* stream) {
    static PFN_cuStreamGetCtx_v12050 get_ctx = nullptr;
    static PFN_cuGreenCtxGetDevResource_v12040 get_resource = nullptr;
    if (get_ctx == nullptr || get_resource == nullptr) {
        void *a = nullptr, *b = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuStreamGetCtx", &a, 12050, cudaEnableDefault, &q) != cudaSuccess || a == nullptr ||
            cudaGetDriverEntryPointByVersion("cuGreenCtxGetDevResource", &b, 12040, cudaEnableDefault, &q) != cudaSuccess || b == nullptr) {
            cudaGetLastError();
            return 1;                    // a driver without green contexts
        }
        get_ctx = reinterpret_cast<PFN_cuStreamGetCtx_v12050>(a);
        get_resource = reinterpret_cast<PFN_cuGreenCtxGetDevResource_v12040>(b);
    }
    const int sms = nxd_num_sms();       // a runtime call: the driver's need a context
    CUcontext ctx = nullptr;
    CUgreenCtx green = nullptr;
    CUdevResource r;
    if (get_ctx((CUstream)stream, &ctx, &green) != CUDA_SUCCESS || green == nullptr) return 1;
    return get_resource(green, &r, CU_DEV_RESOURCE_TYPE_SM) == CUDA_SUCCESS && (int)r.sm.smCount >= sms;
}

// hidden, out [H] bf16; pointers: per layer the weights input norm [H], q | k | v [(n_q + 2 n_kv) D, H], o [H, H], norm behind the
// attention [H], gate | up [2 I, H], down [H, I], all contiguous and 16-byte aligned, and the caches of keys and values; eps: the two
// norms' per layer.  positions, lengths: the sequence's, int32, the step's token the last of its length; cache as for
// nxd_smallm_qkv_rope_cache.  wait_clocks: -1, or the limit of a wait.  gave_up: a word of device or pinned host memory that a step which
// gave up a wait sets to 1, or NULL.
NXD_API int nxd_token_stack_telling(const void* hidden, void* out, const void* const* pointers, const float* eps, int layers,
                                    const float* cos_t, const float* sin_t, const int* positions, const int* lengths, const int* seq_ids,
                                    const int* block_table, long long stride_b, long long stride_h, int page_size, int max_pages,
                                    void* scratch, int H, int I, int n_q, int n_kv, int D, float scale, long long wait_clocks,
                                    int* gave_up, void* stream) {
    NXD_REQUIRE(nxd_token_stack_scratch(layers, 1, H, I, n_q, n_kv, D) > 0, "token_stack: no kernel for %d layers of %d", layers, H);
    Args a = {};
    for (int l = 0; l < layers; ++l) {
        const void* const* w = pointers + 8 * l;
        for (int i = 0; i < 8; ++i) NXD_REQUIRE(w[i] != nullptr && ((uintptr_t)w[i] & 15) == 0, "token_stack: layer %d: alignment", l);
        a.layer[l] = Layer{(const bf16*)w[0], (const bf16*)w[1], (const bf16*)w[2], (const bf16*)w[3], (const bf16*)w[4],
                           (const bf16*)w[5], (bf16*)w[6], (bf16*)w[7], eps[2 * l], eps[2 * l + 1]};
    }
    NXD_REQUIRE((((uintptr_t)hidden | (uintptr_t)out) & 15) == 0 && ((uintptr_t)scratch & 255) == 0 && stride_b % 8 == 0 && stride_h % 8 == 0,
                "token_stack: %s", "alignment");
    const Scratch s = scratch_of(H, I, n_q, n_kv, D);
    word* base = (word*)scratch;
    a.layers = layers, a.H = H, a.I = I, a.n_q = n_q, a.n_kv = n_kv;
    a.hidden = (const bf16*)hidden, a.out = (bf16*)out;
    a.mid = base + s.mid, a.x = base + s.x, a.q = base + s.q, a.kv = base + s.kv, a.attn = base + s.attn, a.act = base + s.act;
    a.part_o = base + s.part_o, a.part_ml = base + s.part_ml;
    a.cos_t = cos_t, a.sin_t = sin_t, a.positions = positions, a.lengths = lengths;
    a.cache = CacheDst{nullptr, nullptr, block_table, seq_ids, stride_b, stride_h, page_size > 0 ? page_size : 1, max_pages};
    a.scale_log2 = scale * 1.4426950408889634f;
    a.limit = wait_clocks < 0 ? kWaitClocks : wait_clocks;
    a.gave_up = gave_up;
    return dispatch(a, D, s.words, (cudaStream_t)stream);
}

NXD_API int nxd_token_stack(const void* hidden, void* out, const void* const* pointers, const float* eps, int layers, const float* cos_t,
                            const float* sin_t, const int* positions, const int* lengths, const int* seq_ids, const int* block_table,
                            long long stride_b, long long stride_h, int page_size, int max_pages, void* scratch, int H, int I,
                            int n_q, int n_kv, int D, float scale, long long wait_clocks, void* stream) {
    return nxd_token_stack_telling(hidden, out, pointers, eps, layers, cos_t, sin_t, positions, lengths, seq_ids, block_table, stride_b,
                                   stride_h, page_size, max_pages, scratch, H, I, n_q, n_kv, D, scale, wait_clocks, nullptr, stream);
}

// *gave_up <- whether a step on this device gave up a wait since the last call (its results are NaN).  Waits for the stream.
NXD_API int nxd_token_stack_status(int* gave_up, void* stream) {
    const cudaStream_t st = (cudaStream_t)stream;
    const int none = 0;
    NXD_CHECK_CUDA(cudaMemcpyFromSymbolAsync(gave_up, stack_gave_up, sizeof(int), 0, cudaMemcpyDeviceToHost, st));
    NXD_CHECK_CUDA(cudaStreamSynchronize(st));
    if (*gave_up == 0) return 0;
    NXD_CHECK_CUDA(cudaMemcpyToSymbolAsync(stack_gave_up, &none, sizeof(int), 0, cudaMemcpyHostToDevice, st));
    NXD_CHECK_CUDA(cudaStreamSynchronize(st));
    return 0;
}
