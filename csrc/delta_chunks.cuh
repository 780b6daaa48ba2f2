// Chunk-wise gated delta rule: what the kernels of delta_rule.cu (the chunk's triangular systems) and delta_chunks.cu (everything
// behind them) share.
#pragma once
#include "common.cuh"

namespace nxd_delta {

constexpr int CH = 64;                                   // tokens of a chunk
constexpr int CW_COLS = 32;                              // value columns of a CTA of the scan
// per (row, head, chunk): M [CH][CH] = (I + A)^-1 diag(beta), P M [CH][CH], Gamma [CH], L[CH-1][.] [CH]
constexpr int CHUNK_FLOATS = 2 * CH * CH + 2 * CH;
// one operand tile of the scan: 128 rows x 64 terms in three bf16 pieces, as it lies in shared memory
constexpr int PIECE_BYTES = 128 * 64 * 2, TILE_BYTES = 3 * PIECE_BYTES;

// tiles of a chunk: [M ; P M], D / 64 of [-W ; Q'], one per 128 key channels of the decayed keys
constexpr int chunk_tiles(int D) { return 1 + D / 64 + (D == 256 ? 2 : 1); }

struct Step {
    const float *qn, *kn, *vn;
    float *S, *out;
    const int *q_start, *n_new, *seq_ids;
    int B, Tn, H, G, D, Dv;
};

// factors and scan of the chunks [c0, c0 + count), whose systems are in `systems`; wait_clocks: the clocks after which a wait inside
// the scan gives up, -1: two seconds
int launch_chunks_tc(const Step& s, const float* systems, uint8_t* tiles, int c0, int count, long long wait_clocks, cudaStream_t st);

}  // namespace nxd_delta
