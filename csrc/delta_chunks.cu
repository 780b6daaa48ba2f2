// Gated delta rule in chunks of 64 tokens on the 5th-gen tensor cores, with fp32 accuracy (the systems of the chunks: delta_rule.cu).
// With W = M diag(Gamma) K and Q' = diag(Gamma) Q - P M diag(Gamma) K, which do not depend on the state,
//
//   U = M V - W S;     O = P M V + Q' S;     S <- Gamma_CH S + (diag(L[CH-1][.]) K)^T U
//
//   delta_chunk_factors  per (chunk, head, row), in parallel: W and Q' in fp32; every left operand as three bf16 pieces
//                        x = x0 + x1 + x2 (24 bits), laid out as the scan's shared memory wants it
//   delta_chunk_scan     per (32 value columns, head, row), sequential over chunks: two products of 128 rows per chunk,
//                        [M ; P M] V + [-W ; Q'] S (rows: 64 errors U, 64 outputs) and decayed keys^T U
//
// The chain over chunks is what takes the time, so everything that does not wait for the state is out of it.  The state is fp32 in
// registers (a thread owns one key channel's 32 columns) and goes over as pieces in shared memory, as do V and U.  One MMA takes a
// piece of the left operand against all pieces of the right one that matter side by side: x0 [y0 | y1 | y2], x1 [y0 | y1], x2 y0 --
// the left operand, which bounds an MMA of so few columns, is read 3 times per 16 terms and not 6, and products of different size
// have accumulators of their own.  The tensor cores cut where fp32 rounds: an accumulator takes 64 terms (32 where tensor memory has
// room), x0 y0 shares its accumulator with nothing, the rest is added in fp32.  (With x1 y0 and x2 y0 in it the output was 1.5e-7
// off instead of 0.8e-7.)
//
// 4 x 2048 tokens, 4 heads of 128 x 256: factors 39 us, scan 100 us, against 350 us for the whole in fp32 on the multiply-add pipes.  A
// chunk takes the scan 3.1 us: 48 MMAs of 41 to 57 clocks (41 with 32 columns, 57 with 96), the rest latencies of its four hand-overs.
#include <type_traits>

#include "delta_chunks.cuh"
#include "ptx.cuh"

namespace {

using namespace nxd_delta;

constexpr int kThreads = 384;
constexpr int kRow = CW_COLS * 2;                        // bytes of a row of the right operands: one SWIZZLE_64B row
constexpr int kSmall = CH * kRow;                        // one piece of U or V

__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// x -> three bf16 pieces (each the rounded remainder of the ones before), N pairs of values
template <int N>
__device__ __forceinline__ void split(const uint64_t* x, uint32_t (&p)[3][N]) {
    const uint64_t minus = f2_pack(-1.f, -1.f);
#pragma unroll
    for (int i = 0; i < N; ++i) {
        uint64_t r = x[i];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p[k][i]) : "f"(f2_hi(r)), "f"(f2_lo(r)));
            if (k < 2) r = f2_fma(f2_pack(__uint_as_float(p[k][i] << 16), __uint_as_float(p[k][i] & 0xffff0000u)), minus, r);
        }
    }
}

// Left operands: pieces on the grid of their row.  x0 is the multiple of g next to x, where 256 g is just above the row's largest value,
// x1 that of g / 512.  Small values then leave x0 to the large ones: sums of products of multiples of one g that are near one another
// hold in an accumulator, where with pieces of every value's own exponent (eight bits of a small one too) the tensor cores cut the low
// ends of all products but the largest.  Against the scan in float64, 128 x 256 (pieces of own exponents, these, fp32 multiply-adds):
// decays of 0.2 a token, state 0.93, 0.45, 0.50e-7 and output 0.60, 0.41, 0.54e-7; 0.5 a token, 0.97, 0.55, 0.60 and 0.64, 0.47, 0.63;
// 0.85 a token, 1.03, 0.90, 0.92 and 0.74, 0.57, 0.84; 0.998 a token, 1.18, 1.01, 1.36 and 1.25, 0.93, 1.38.
__device__ __forceinline__ float grid_shift(float largest) {     // x + shift - shift: x on the grid g
    const uint32_t e = min(__float_as_uint(largest) & 0x7f800000u, (127u + 100u) << 23);         // beyond: pieces of own exponents
    return __uint_as_float(e) * (1.5f * 65536.f);                // 2^e / 128 * 1.5 * 2^23
}

// V = 2, 4 or 8 values, shift[i] that of value i's row, to memory with the pieces PIECE_BYTES apart
template <int V>
__device__ __forceinline__ void split_store(const float* x, const uint64_t (&shift)[V / 2], uint8_t* dst) {
    const uint64_t minus = f2_pack(-1.f, -1.f), down = f2_pack(1.f / 512.f, 1.f / 512.f);
    uint32_t w[3][V / 2];
#pragma unroll
    for (int i = 0; i < V / 2; ++i) {
        uint64_t r = f2_pack(x[2 * i], x[2 * i + 1]), c = shift[i];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const uint64_t y = k < 2 ? f2_fma(c, minus, f2_add(r, c)) : r;
            asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(w[k][i]) : "f"(f2_hi(y)), "f"(f2_lo(y)));
            if (k < 2) r = f2_fma(f2_pack(__uint_as_float(w[k][i] << 16), __uint_as_float(w[k][i] & 0xffff0000u)), minus, r);
            c = f2_mul(c, down);
        }
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        uint8_t* at = dst + k * PIECE_BYTES;
        if constexpr (V == 2) *reinterpret_cast<uint32_t*>(at) = w[k][0];
        if constexpr (V == 4) *reinterpret_cast<uint2*>(at) = make_uint2(w[k][0], w[k][1]);
        if constexpr (V == 8) *reinterpret_cast<uint4*>(at) = make_uint4(w[k][0], w[k][1], w[k][2], w[k][3]);
    }
}

constexpr int FT = 256, MTP = 132;

// grid (chunks, H, B).  A warp takes 8 of the 128 rows [M ; P M] twice (w and 15 - w, so that the triangles cost every warp the same),
// a lane D / 32 key channels; sums of 8 terms first.  What lies above the diagonal is left out, not multiplied by zero: a token
// that is not a number does not reach the tokens before it.
template <int D>
__global__ void __launch_bounds__(FT, D == 256 ? 1 : 2)
delta_chunk_factors_kernel(const float* __restrict__ qn, const float* __restrict__ kn, const float* __restrict__ systems,
                           uint8_t* __restrict__ tiles, const int* __restrict__ n_new, int Tn, int c0, int H, int G) {
    pdl_wait();
    constexpr int V = D / 32, A1 = D / 64;
    extern __shared__ __align__(16) float smem[];
    float* Ks = smem;                                    // [CH][D]
    float* MT = Ks + CH * D;                             // [CH][MTP] column s of [M ; P M] times Gamma_s
    __shared__ float gam[CH], last[CH], row_max[2][2 * CH];
    __shared__ unsigned channel_max[D];                  // bits of non-negative values, which are in order
    const int c = c0 + blockIdx.x, h = blockIdx.y, b = blockIdx.z, kvh = h / (H / G), tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    const int n = n_new != nullptr ? min(n_new[b], Tn) : Tn;
    const int nt = min(CH, n - c * CH);
    if (nt <= 0) return;
    const long long row0 = (long long)b * Tn + c * CH, e = ((long long)b * H + h) * gridDim.x + blockIdx.x;
    const float* sys = systems + e * CHUNK_FLOATS;
    uint8_t* img = tiles + e * chunk_tiles(D) * TILE_BYTES;
    if (tid < CH) gam[tid] = sys[2 * CH * CH + tid];
    else if (tid < 2 * CH) last[tid - CH] = sys[2 * CH * CH + tid];
    if (tid < D) channel_max[tid] = 0u;
    float4 kv[D / 16], m[2][4];                          // every load of the block is in flight at once
#pragma unroll
    for (int x = 0; x < D / 16; ++x) {
        const int i = tid + x * FT, t = i / (D / 4), d = (i % (D / 4)) * 4;
        kv[x] = t < nt ? *reinterpret_cast<const float4*>(kn + ((row0 + t) * G + kvh) * D + d) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const int mr = tid & 127, ms = (tid >> 7) * 16;      // row and first term of [M ; P M]; the second piece is 32 terms on
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int x = 0; x < 4; ++x) m[i][x] = *reinterpret_cast<const float4*>(sys + mr * CH + ms + 32 * i + 4 * x);
#pragma unroll
    for (int x = 0; x < D / 16; ++x) *reinterpret_cast<float4*>(Ks + (tid + x * FT) * 4) = kv[x];
    {
        float mx = 0.f;
#pragma unroll
        for (int i = 0; i < 32; ++i) mx = fmaxf(mx, fabsf(reinterpret_cast<const float*>(m)[i]));
        row_max[tid >> 7][mr] = mx;
    }
    __syncthreads();
    {
        float mx = 0.f;                                  // decayed keys: a thread takes a channel's share of the tokens
#pragma unroll 16
        for (int t = tid / D; t < CH; t += FT / D) mx = fmaxf(mx, fabsf(Ks[t * D + tid % D] * last[t]));
        atomicMax(&channel_max[tid % D], __float_as_uint(mx));
    }
    const float m_shift = grid_shift(fmaxf(row_max[0][mr], row_max[1][mr]));
    const uint64_t m_shift2[4] = {f2_pack(m_shift, m_shift), f2_pack(m_shift, m_shift), f2_pack(m_shift, m_shift), f2_pack(m_shift, m_shift)};
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int s = ms + 32 * i;
        const float* f = reinterpret_cast<const float*>(m[i]);
#pragma unroll
        for (int x = 0; x < 16; ++x) MT[(s + x) * MTP + mr] = f[x] * gam[s + x];
#pragma unroll
        for (int x = 0; x < 2; ++x) split_store<8>(f + 8 * x, m_shift2, img + mr * 128 + (((s / 8 + x) ^ (mr & 7)) << 4));
    }
    __syncthreads();
    const int d0 = lane * V;
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
        const int r0 = (half ? 15 - warp : warp) * 8, t0 = r0 & (CH - 1);        // half 0: rows of M, half 1: rows of P M
        float q[8][V];
        if (half) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float* src = qn + ((row0 + min(t0 + i, nt - 1)) * G + kvh) * D + d0;
                if constexpr (V == 2) *reinterpret_cast<float2*>(q[i]) = *reinterpret_cast<const float2*>(src);
                else
#pragma unroll
                    for (int x = 0; x < V; x += 4) *reinterpret_cast<float4*>(q[i] + x) = *reinterpret_cast<const float4*>(src + x);
            }
        }
        uint64_t acc[4][V] = {};                         // pairs of rows
#pragma unroll 1
        for (int s0 = 0; s0 <= t0; s0 += 8) {
            uint64_t part[4][V] = {};
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const ulonglong2 m0 = *reinterpret_cast<const ulonglong2*>(MT + (s0 + j) * MTP + r0);
                const ulonglong2 m1 = *reinterpret_cast<const ulonglong2*>(MT + (s0 + j) * MTP + r0 + 4);
                const uint64_t m[4] = {m0.x, m0.y, m1.x, m1.y};
                float k[V];
                if constexpr (V == 2) *reinterpret_cast<float2*>(k) = *reinterpret_cast<const float2*>(Ks + (s0 + j) * D + d0);
                else
#pragma unroll
                    for (int x = 0; x < V; x += 4)
                        *reinterpret_cast<float4*>(k + x) = *reinterpret_cast<const float4*>(Ks + (s0 + j) * D + d0 + x);
                if (s0 < t0) {
#pragma unroll
                    for (int x = 0; x < V; ++x)
#pragma unroll
                        for (int i = 0; i < 4; ++i) part[i][x] = f2_fma(m[i], f2_pack(k[x], k[x]), part[i][x]);
                } else {                                 // the diagonal block: rows j and on
#pragma unroll
                    for (int x = 0; x < V; ++x)
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            float lo = f2_lo(part[i][x]), hi = f2_hi(part[i][x]);
                            if (2 * i >= j) lo = fmaf(f2_lo(m[i]), k[x], lo);
                            if (2 * i + 1 >= j) hi = fmaf(f2_hi(m[i]), k[x], hi);
                            part[i][x] = f2_pack(lo, hi);
                        }
                }
            }
#pragma unroll
            for (int x = 0; x < V; ++x)
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[i][x] = f2_add(acc[i][x], part[i][x]);
        }
        uint8_t* dst = img + (1 + d0 / 64) * TILE_BYTES + (d0 & 7) * 2;
        const int piece16 = (d0 & 63) >> 3;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int r = r0 + i, t = t0 + i;
            float w[V];
#pragma unroll
            for (int x = 0; x < V; ++x) w[x] = (i & 1) ? f2_hi(acc[i / 2][x]) : f2_lo(acc[i / 2][x]);
#pragma unroll
            for (int x = 0; x < V; ++x) w[x] = half ? fmaf(gam[t], t < nt ? q[i][x] : 0.f, -w[x]) : -w[x];
            float mx = 0.f;
#pragma unroll
            for (int x = 0; x < V; ++x) mx = fmaxf(mx, fabsf(w[x]));
            const float shift = grid_shift(__uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(mx))));
            uint64_t shift2[V / 2];
#pragma unroll
            for (int x = 0; x < V / 2; ++x) shift2[x] = f2_pack(shift, shift);
            split_store<V>(w, shift2, dst + r * 128 + ((piece16 ^ (r & 7)) << 4));
        }
    }
    for (int i = tid; i < CH * (D / 8); i += FT) {       // decayed keys, channels along the rows of 128 bytes
        const int t = i / (D / 8), d = (i % (D / 8)) * 8;
        float k[8];
#pragma unroll
        for (int x = 0; x < 8; ++x) k[x] = Ks[t * D + d + x] * last[t];
        uint64_t shift[4];
#pragma unroll
        for (int x = 0; x < 4; ++x)
            shift[x] = f2_pack(grid_shift(__uint_as_float(channel_max[d + 2 * x])), grid_shift(__uint_as_float(channel_max[d + 2 * x + 1])));
        split_store<8>(k, shift, img + (1 + A1 + d / 128) * TILE_BYTES + ((d >> 6) & 1) * 8192 + t * 128 + ((((d & 63) >> 3) ^ (t & 7)) << 4));
    }
    pdl_trigger();
}

template <int D>
struct Cfg {
    static constexpr int kA1 = D / 64, kA3 = D == 256 ? 2 : 1, kTiles = chunk_tiles(D);
    static constexpr int kSPiece = D * kRow;
    static constexpr int kSlots = D == 256 ? 9 : 11;      // pieces of tiles in flight
    static constexpr int kOffS = kSlots * PIECE_BYTES, kOffU = kOffS + 3 * kSPiece, kOffV = kOffU + 3 * kSmall;
    static constexpr int kOffBar = kOffV + 3 * kSmall;
    static constexpr int kSmem = kOffBar + 512 + 1024;
    static constexpr int kBlocks = D == 256 ? 2 : 1;     // key channels of an epilogue thread
    static constexpr int kAccCols = 3 * CW_COLS;         // x0 y0 | x0 y1 + x1 y0 | x0 y2 + x1 y1 + x2 y0
    // accumulators per product: of 32 terms where tensor memory has room (the state's update takes those of [-W ; Q'] S again)
    static constexpr int kHalves1 = D == 64 ? 2 : 1, kHalvesV = D == 256 ? 1 : 2;
    static constexpr int kAccV = kA1 * kHalves1 * kAccCols;
    static_assert(kAccV + kHalvesV * kAccCols <= 512 && 2 * kA3 <= kA1 * kHalves1, "tensor memory");
    static_assert(kSmem <= 232448, "shared memory");
};

// SWIZZLE_64B, MN-major: rows (terms) of 32 columns, groups of 8 rows 512 bytes apart, groups of 32 columns (the pieces) `piece`
// bytes apart
__device__ __forceinline__ uint64_t desc_b(uint32_t addr, uint32_t piece) {
    return (uint64_t)((addr & 0x3FFFF) >> 4) | (uint64_t)(piece >> 4) << 16 | (uint64_t)(512 >> 4) << 32 | (uint64_t)1 << 46 |
           (uint64_t)4 << 61;
}

// Waits end.  One that has taken `limit` clocks (kWaitClocks is two seconds; the longest ones take some microseconds) gives up: `dead`
// ends the other waits of the block, nxd_delta_scan_status tells the host, and NaN goes where results are missing.  A limit of zero
// gives up without asking.
constexpr long long kWaitClocks = 4000000000ll;

__device__ int scan_gave_up;

__device__ __forceinline__ bool wait(uint64_t* bar, uint32_t parity, long long limit, volatile int* dead) {
    long long start = 0;
    for (int i = 1;; ++i) {
        if (limit > 0 && ptx::mbar_try_wait(bar, parity)) return true;
        if (limit > 0 && (i & 63) != 0) continue;        // the rest asked after every try: 227 us instead of 216 (4 heads of 64 x 128, 2 x 3497)
        if (*dead) return false;
        const long long now = clock64();
        if (start == 0) start = now;
        if (now - start < limit) continue;
        *dead = 1;
        scan_gave_up = 1;
        return false;
    }
}

// the same for whole warps: the lanes leave it together and with one answer, as barriers and tensor-memory loads behind it want them
__device__ __forceinline__ bool wait_warp(uint64_t* bar, uint32_t parity, long long limit, volatile int* dead) {
    return __all_sync(0xffffffffu, wait(bar, parity, limit, dead));
}

constexpr int kPairs = CW_COLS / 4;                      // pairs of columns of an epilogue thread (half of the columns)

// an accumulator's columns of this thread: the sum of its three parts
__device__ __forceinline__ void add_acc(uint32_t tmem, uint64_t (&big)[kPairs], uint64_t (&small)[kPairs]) {
    uint32_t v[3][2 * kPairs];
#pragma unroll
    for (int x = 0; x < 3; ++x) ptx::tmem_ld_32x32b_x16(tmem + x * CW_COLS, v[x]);
    ptx::tmem_ld_wait();
    auto pair = [&](int x, int j) { return f2_pack(__uint_as_float(v[x][2 * j]), __uint_as_float(v[x][2 * j + 1])); };
#pragma unroll
    for (int j = 0; j < kPairs; ++j) {
        big[j] = f2_add(big[j], pair(0, j));
        small[j] = f2_add(small[j], f2_add(pair(2, j), pair(1, j)));
    }
}

// N pairs of values of a right operand's row, from group g0 of eight values on -> pieces
template <int N>
__device__ __forceinline__ void put_row(uint8_t* base, int piece, int row, int g0, const uint64_t* x) {
    uint32_t p[3][N];
    split<N>(x, p);
#pragma unroll
    for (int i = 0; i < N / 4; ++i)
#pragma unroll
        for (int k = 0; k < 3; ++k)
            *reinterpret_cast<uint4*>(base + k * piece + row * kRow + (((g0 + i) ^ ((row >> 1) & 3)) << 4)) =
                make_uint4(p[k][4 * i], p[k][4 * i + 1], p[k][4 * i + 2], p[k][4 * i + 3]);
}

// Warps: 0 copies tiles, 1 issues the MMAs, 2-3 split V (a thread per token), 4-11 own the state and the epilogues (a thread per row
// of the products and half of the columns)
template <int D>
__global__ void __launch_bounds__(kThreads, 1)
delta_chunk_scan_kernel(const Step p, const float* __restrict__ systems, const uint8_t* __restrict__ tiles, int c0, int count,
                        long long limit) {
    using C = Cfg<D>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = ptx::align_smem_1024(smem_raw);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + C::kOffBar);
    uint64_t *empty = full + C::kSlots, *s_full = empty + C::kSlots, *u_full = s_full + 1, *v_full = u_full + 1, *accv = v_full + 1;
    uint64_t *acc1 = accv + 1, *acc3 = acc1 + C::kA1;    // accumulators: V, each 64 terms of the state, the state's update
    uint64_t* drained = acc3 + 1;                        // every MMA has run
    uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(drained + 1);
    __shared__ int bad[2][CW_COLS], any_bad[2];          // first token of a column whose value is not finite
    __shared__ int dead;
    // the warp's number as a value that the compiler knows to be the warp's: an MMA issued under a branch on threadIdx takes 60 clocks,
    // one by the elected thread of such a warp 35
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int col0 = blockIdx.x * CW_COLS, h = blockIdx.y, b = blockIdx.z;
    pdl_wait();                                          // and no tensor memory before
    const int n = p.n_new != nullptr ? min(p.n_new[b], p.Tn) : p.Tn;
    const long long row0 = (long long)b * p.Tn;
    float* orow = p.out + (row0 * p.H + h) * p.Dv + col0;                        // + t * H * Dv
    const long long pitch = (long long)p.H * p.Dv;
    if (c0 == 0)                                         // padding rows
        for (int i = tid; i < (p.Tn - max(n, 0)) * CW_COLS; i += kThreads)
            orow[(max(n, 0) + i / CW_COLS) * pitch + i % CW_COLS] = 0.f;
    const int chunks = min(count, (n + CH - 1) / CH - c0);
    if (chunks <= 0) return;
    const int line = p.seq_ids != nullptr ? p.seq_ids[b] : b;
    const long long e0 = ((long long)b * p.H + h) * count;
    if (tid == 0) {
        for (int i = 0; i < C::kSlots; ++i) {
            ptx::mbar_init(&full[i], 1);
            ptx::mbar_init(&empty[i], 1);
        }
        ptx::mbar_init(s_full, kThreads - 128);
        ptx::mbar_init(u_full, kThreads - 128);
        ptx::mbar_init(v_full, CH);
        ptx::mbar_init(accv, 1);
        for (int i = 0; i < C::kA1; ++i) ptx::mbar_init(&acc1[i], 1);
        ptx::mbar_init(acc3, 1);
        ptx::mbar_init(drained, 1);
        dead = 0;
        ptx::fence_barrier_init();
    }
    if (warp == 1) ptx::tmem_alloc<1>(tmem_ptr, 512);
    ptx::tcgen05_fence_before();
    __syncthreads();
    ptx::tcgen05_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_ptr, 0);

    if (warp == 0) {
        if (lane == 0) {
            const uint8_t* src = tiles + e0 * C::kTiles * TILE_BYTES;             // piece by piece
            const int total = chunks * C::kTiles * 3;
            int i = 0;
            for (; i < total; ++i) {
                const int st = i % C::kSlots;
                if (!wait(&empty[st], (uint32_t)(i / C::kSlots + 1) & 1, limit, &dead)) break;
                // D = 64: the decayed keys are the first half of their tile (what the other rows multiply is not read)
                const uint32_t bytes = D == 64 && i % (C::kTiles * 3) >= (C::kTiles - 1) * 3 ? PIECE_BYTES / 2 : PIECE_BYTES;
                ptx::mbar_arrive_expect_tx(&full[st], bytes);
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                                 ptx::smem_u32(smem + st * PIECE_BYTES)),
                             "l"(src + (long long)i * PIECE_BYTES), "r"(bytes), "r"(ptx::smem_u32(&full[st]))
                             : "memory");
            }
            int none = 0;                                // copies that no MMA has waited for still land in this block's memory
            for (int j = max(0, i - C::kSlots); j < i; ++j)
                wait(&full[j % C::kSlots], (uint32_t)(j / C::kSlots) & 1, kWaitClocks, &none);
        }
    } else if (warp == 1) {
        if (ptx::elect_one()) {
            int st = 0;                                  // slot of the next piece
            uint32_t st_ph = 0;
            // D[tmem columns] = one tile x 64 rows of a right operand, `halves` accumulators of 64 / halves terms.  One thread issues
            // some fifty MMAs per chunk on the chain's critical path: a descriptor costs it one addition.
            auto product = [&](auto keys, auto halves, uint32_t col, uint64_t db0) {
                constexpr bool kKeys = decltype(keys)::value;
                constexpr int kPer = 4 / decltype(halves)::value, kStep = (kKeys ? 2048 : 32) >> 4;
#pragma unroll
                for (int x = 0; x < 3; ++x) {
                    if (!wait(&full[st], st_ph, limit, &dead)) return false;
                    ptx::tcgen05_fence_after();
                    const uint64_t da0 = ptx::make_smem_desc(ptx::smem_u32(smem + st * PIECE_BYTES), kKeys ? 8192 : 16, 1024);
                    constexpr uint32_t major = kKeys ? 1u << 15 : 0u;
                    const uint32_t idesc = ptx::make_idesc_bf16(128, (3 - x) * CW_COLS, 0, 1) | major;
#pragma unroll
                    for (int k = 0; k < CH / 16; ++k)
                        ptx::umma_bf16<1>(tmem + col + (k / kPer) * C::kAccCols + x * CW_COLS, da0 + k * kStep,
                                          db0 + k * (16 * kRow >> 4), idesc, k % kPer > 0 || x > 0);
                    ptx::umma_commit(&empty[st]);
                    if (++st == C::kSlots) st = 0, st_ph ^= 1;
                }
                return true;
            };
            using Two = std::integral_constant<int, 2>;
            using HV = std::integral_constant<int, C::kHalvesV>;
            using H1 = std::integral_constant<int, C::kHalves1>;
            const uint64_t ds = desc_b(ptx::smem_u32(smem + C::kOffS), C::kSPiece), du = desc_b(ptx::smem_u32(smem + C::kOffU), kSmall);
            const uint64_t dv = desc_b(ptx::smem_u32(smem + C::kOffV), kSmall);
            for (int c = 0; c < chunks; ++c) {
                const uint32_t ph = c & 1;
                if (!wait(v_full, ph, limit, &dead) || !product(std::false_type(), HV(), C::kAccV, dv)) break;
                ptx::umma_commit(accv);
                if (!wait(s_full, ph, limit, &dead)) break;
                bool ok = true;
                for (int kb = 0; kb < C::kA1 && ok; ++kb) {
                    ok = product(std::false_type(), H1(), kb * C::kHalves1 * C::kAccCols, ds + kb * (64 * kRow >> 4));
                    if (ok) ptx::umma_commit(&acc1[kb]);
                }
                if (!ok) break;
                if (!wait(u_full, ph, limit, &dead)) break;
                // the state's update takes the accumulators that the epilogue has just read
                for (int db = 0; db < C::kA3 && ok; ++db) ok = product(std::true_type(), Two(), 2 * db * C::kAccCols, du);
                if (!ok) break;
                ptx::umma_commit(acc3);
            }
            int none = 0;                                // tensor memory is given back behind the last MMA
            ptx::umma_commit(drained);
            wait(drained, 0, kWaitClocks, &none);
        }
    } else if (warp < 4) {
        const int t = tid - 64;
        const float* src = p.vn + ((row0 + t) * p.H + h) * p.Dv + col0;          // + chunk * CH * H * Dv
        float v[CW_COLS];
        auto fetch = [&](int c) {
            const bool ok = (c0 + c) * CH + t < n;
#pragma unroll
            for (int j = 0; j < CW_COLS; j += 4)
                *reinterpret_cast<float4*>(v + j) = ok ? *reinterpret_cast<const float4*>(src + (long long)(c0 + c) * CH * pitch + j)
                                                       : make_float4(0.f, 0.f, 0.f, 0.f);
        };
        fetch(0);
        bool live = true;
        for (int c = 0; c < chunks; ++c) {
            // the last V has been used.  What gives up runs on to the end: the barrier below wants both warps
            if (c > 0 && live) live = wait_warp(accv, (uint32_t)(c - 1) & 1, limit, &dead);
            // A value that is not finite would reach the tokens before it through 0 * value: it goes over as zero, and the epilogue puts
            // NaN where it would have arrived
            if (t < CW_COLS) bad[c & 1][t] = CH;
            if (t == 0) any_bad[c & 1] = 0;
            asm volatile("bar.sync 2, 64;" ::: "memory");
#pragma unroll
            for (int j = 0; j < CW_COLS; ++j)
                if (!isfinite(v[j])) {
                    v[j] = 0.f;
                    atomicMin(&bad[c & 1][j], t);
                    any_bad[c & 1] = 1;
                }
            uint64_t v2[CW_COLS / 2];
#pragma unroll
            for (int j = 0; j < CW_COLS / 2; ++j) v2[j] = f2_pack(v[2 * j], v[2 * j + 1]);
            put_row<CW_COLS / 2>(smem + C::kOffV, kSmall, t, 0, v2);
            ptx::fence_proxy_async();
            ptx::mbar_arrive(v_full);
            if (c + 1 < chunks) fetch(c + 1);
        }
    } else {
        const int row = (warp & 3) * 32 + lane, half = warp >= 8, j0 = half * 2 * kPairs;       // tensor-memory lane, first column
        const uint32_t at = tmem + ((uint32_t)((warp & 3) * 32) << 16) + j0;
        const bool mine = row < D;                                               // key channels row (and row + 128)
        float* Sb = p.S + (((long long)line * p.H + h) * D + (mine ? row : 0)) * p.Dv + col0 + j0;
        const bool fresh = c0 == 0 && p.q_start[b] == 0;
        uint64_t s[C::kBlocks][kPairs];
        auto put_state = [&](int i) {
            if (mine) put_row<kPairs>(smem + C::kOffS, C::kSPiece, row + 128 * i, 2 * half, s[i]);
        };
#pragma unroll
        for (int i = 0; i < C::kBlocks; ++i) {
#pragma unroll
            for (int j = 0; j < kPairs; j += 2) {
                const ulonglong2 v = !fresh && mine ? *reinterpret_cast<const ulonglong2*>(Sb + 128ll * i * p.Dv + 2 * j) : make_ulonglong2(0, 0);
                s[i][j] = v.x, s[i][j + 1] = v.y;
            }
            put_state(i);
        }
        ptx::fence_proxy_async();
        ptx::mbar_arrive(s_full);
        const uint64_t nan = f2_pack(__int_as_float(0x7fffffff), __int_as_float(0x7fffffff));
        const volatile int* gone = &dead;
        int c = 0;
        for (; c < chunks; ++c) {
            const uint32_t ph = c & 1;
            const float gamma = systems[(e0 + c) * CHUNK_FLOATS + 2 * CH * CH + CH - 1];
            uint64_t r[kPairs] = {}, small[kPairs] = {}, rv[kPairs] = {};        // sums of their own for V and for the state
            if (!wait_warp(accv, ph, limit, &dead)) break;
            ptx::tcgen05_fence_after();
#pragma unroll
            for (int a = 0; a < C::kHalvesV; ++a) add_acc(at + C::kAccV + a * C::kAccCols, rv, small);
            bool ok = true;
#pragma unroll
            for (int kb = 0; kb < C::kA1; ++kb) {
                ok = ok && wait_warp(&acc1[kb], ph, limit, &dead);
                ptx::tcgen05_fence_after();
                if (!ok) continue;
#pragma unroll
                for (int a = 0; a < C::kHalves1; ++a) add_acc(at + (kb * C::kHalves1 + a) * C::kAccCols, r, small);
            }
            if (!ok) break;
            ptx::tcgen05_fence_before();
            const int t = row & (CH - 1);
#pragma unroll
            for (int j = 0; j < kPairs; ++j) r[j] = f2_add(rv[j], f2_add(r[j], small[j]));
            if (any_bad[ph] != 0) {
#pragma unroll
                for (int j = 0; j < kPairs; ++j)
                    r[j] = f2_pack(t >= bad[ph][j0 + 2 * j] ? f2_lo(nan) : f2_lo(r[j]), t >= bad[ph][j0 + 2 * j + 1] ? f2_hi(nan) : f2_hi(r[j]));
            }
            if (row < CH) put_row<kPairs>(smem + C::kOffU, kSmall, row, 2 * half, r);
            ptx::fence_proxy_async();
            ptx::mbar_arrive(u_full);
            const int tok = (c0 + c) * CH + t;
            if (__any_sync(0xffffffffu, *gone != 0)) break;     // another role gave up: the products may be of anything
            if (row >= CH && tok < n) {
#pragma unroll
                for (int j = 0; j < kPairs; j += 2)
                    *reinterpret_cast<ulonglong2*>(orow + tok * pitch + j0 + 2 * j) = make_ulonglong2(r[j], r[j + 1]);
            }
            if (!wait_warp(acc3, ph, limit, &dead)) break;
            ptx::tcgen05_fence_after();
            const uint64_t gamma2 = f2_pack(gamma, gamma);
#pragma unroll
            for (int i = 0; i < C::kBlocks; ++i) {
#pragma unroll
                for (int j = 0; j < kPairs; ++j) r[j] = small[j] = 0ull;
#pragma unroll
                for (int a = 0; a < 2; ++a) add_acc(at + (2 * i + a) * C::kAccCols, r, small);
#pragma unroll
                for (int j = 0; j < kPairs; ++j) s[i][j] = f2_fma(gamma2, s[i][j], f2_add(r[j], small[j]));
                if (c + 1 < chunks) put_state(i);
            }
            ptx::tcgen05_fence_before();
            if (c + 1 < chunks) {
                ptx::fence_proxy_async();
                ptx::mbar_arrive(s_full);
            }
        }
        if (c < chunks || *gone != 0) {                  // given up
#pragma unroll
            for (int i = 0; i < C::kBlocks; ++i)
#pragma unroll
                for (int j = 0; j < kPairs; ++j) s[i][j] = nan;
            if (row >= CH)
                for (int tok = (c0 + c) * CH + row - CH; tok < n; tok += CH)
                    for (int j = 0; j < 2 * kPairs; ++j) orow[tok * pitch + j0 + j] = f2_lo(nan);
        }
        if (mine) {
#pragma unroll
            for (int i = 0; i < C::kBlocks; ++i)
#pragma unroll
                for (int j = 0; j < kPairs; j += 2)
                    *reinterpret_cast<ulonglong2*>(Sb + 128ll * i * p.Dv + 2 * j) = make_ulonglong2(s[i][j], s[i][j + 1]);
        }
    }
    __syncwarp();
    ptx::tcgen05_fence_before();
    __syncthreads();
    if (warp == 1) ptx::tmem_dealloc<1>(tmem, 512);
}

template <int D>
int launch(const Step& s, const float* systems, uint8_t* tiles, int c0, int count, long long limit, cudaStream_t st) {
    constexpr int factors = (CH * D + CH * MTP) * 4;
    NXD_CHECK_CUDA(nxd_allow_smem<delta_chunk_factors_kernel<D>>(factors));
    NXD_CHECK_CUDA(nxd_allow_smem<delta_chunk_scan_kernel<D>>(Cfg<D>::kSmem));
    NXD_CHECK_CUDA((nxd_launch_pdl(delta_chunk_factors_kernel<D>, dim3(count, s.H, s.B), dim3(FT), factors, st, s.qn, s.kn,
        systems, tiles, s.n_new, s.Tn, c0, s.H, s.G)));
    NXD_LAUNCH_CHECK();
    NXD_CHECK_CUDA((nxd_launch_pdl(delta_chunk_scan_kernel<D>, dim3(s.Dv / CW_COLS, s.H, s.B), dim3(kThreads), Cfg<D>::kSmem, st,
        s, systems, tiles, c0, count, limit)));
    NXD_LAUNCH_CHECK();
    return 0;
}

}  // namespace

int nxd_delta::launch_chunks_tc(const Step& s, const float* systems, uint8_t* tiles, int c0, int count, long long wait_clocks,
                                cudaStream_t st) {
    const long long limit = wait_clocks < 0 ? kWaitClocks : wait_clocks;
    if (s.D == 64) return launch<64>(s, systems, tiles, c0, count, limit, st);
    if (s.D == 128) return launch<128>(s, systems, tiles, c0, count, limit, st);
    return launch<256>(s, systems, tiles, c0, count, limit, st);
}

// *gave_up <- whether a scan on this device gave up a wait since the last call (its outputs and states are NaN from there on).  Waits
// for the stream.
NXD_API int nxd_delta_scan_status(int* gave_up, void* stream) {
    const cudaStream_t st = (cudaStream_t)stream;
    const int none = 0;
    NXD_CHECK_CUDA(cudaMemcpyFromSymbolAsync(gave_up, scan_gave_up, sizeof(int), 0, cudaMemcpyDeviceToHost, st));
    NXD_CHECK_CUDA(cudaStreamSynchronize(st));
    if (*gave_up == 0) return 0;
    NXD_CHECK_CUDA(cudaMemcpyToSymbolAsync(scan_gave_up, &none, sizeof(int), 0, cudaMemcpyHostToDevice, st));
    NXD_CHECK_CUDA(cudaStreamSynchronize(st));
    return 0;
}
