// The decode GEMM of the prefill rows (t3_gemm.cu): arguments and launch, shared with the call chains in t3_prefill.cu.
#pragma once

#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace t3 {

// The most activation rows one tile holds: its accumulator is 128 outputs (tensor-memory lanes) x rows (columns)
constexpr uint32_t kGemmTileRows = 256;

// The operands as TMA sees them
struct GemmMaps {
    CUtensorMap rows[4];   // the prepared rows, f16 [rows, K]: boxes of 64 inputs x 256, 128, 64 and 32 rows (tiled_rows)
    CUtensorMap out[5];    // with DecodeGemmArgs::bulk_out: the 16-bit outputs [rows, N], boxes of 64 outputs x 128, 64, 32, 16 and 8 rows
    CUtensorMap codes[2];  // a weight's (or bank's) codes as 64-bit words [expert, K / 16, N n / 64]: boxes of 4 tile rows x 8 tiles
};

// What a tile of `cols` rows loads: at most two boxes, since a TMA instruction costs the loading thread more than the rows past
// the tile cost the copy (four boxes a slot left the tensor cores waiting for rows a third of the time)
__host__ __device__ constexpr uint32_t tiled_rows(uint32_t cols) {
    return cols > 192u ? 256u : cols > 128u ? 192u : cols > 96u ? 128u : cols > 64u ? 96u : cols > 32u ? 64u : 32u;
}

struct DecodeGemmArgs {
    uint32_t K, N;              // one op's inner and outer widths
    uint32_t n, mask, ops;
    uint32_t op_rows;           // rows between op 0's and op 1's activations
    // Tiles of rows: (expert, first row, rows, 0), entries range[0] .. range[1] (routed); null: one matrix cut every `tile_rows` rows
    const int4* tiles;
    const uint32_t* range;
    uint32_t dense_rows, tile_rows, dense_tiles;
    uint32_t pair;              // 128-output blocks a unit of work takes: 1 or 2
    // The output rotation in the epilogue: svh[op] + expert * svh_stride is the op's scale vector; the finished values go to y
    // (dtype y_dt, one op), or to z [ops][rows][N] as f16 when y is null
    const __half* svh[2];       // null svh[0] (a kept weight only): no rotation, the inner products rounded once into y
    size_t svh_stride;
    __half* z;
    size_t z_op_stride;
    void* y;
    int y_dt;
    uint32_t bulk_out;          // 16-bit results leave by TMA (maps.out); y or z then starts on 16 bytes
    const void* scores;         // y only, or null: each row's f16 value times its score, as the final sum of one slot a row has it
    int score_dt;
    // K slices (dense, at least two, eight at most): a cluster of `ksplit` CTAs a unit, slice z running inputs 128 floor(K / 128 *
    // z / ksplit) .. and leaving its f32 accumulators in part [N / 128][ksplit][rows][128]; after the cluster's barrier each CTA
    // adds the slices of its share of the rows in slice order and finishes them. 0 or 1: one CTA runs all of K.
    uint32_t ksplit;
    float* part;
    uint32_t kept;              // codes[0] is a kept weight: f16 (or bf16) [N, K], boxes of 64 inputs x 128 outputs; nothing is decoded
    uint32_t bf16;              // kept weight and rows are bf16
    uint32_t* err;
    int overlap;                // launch with the programmatic-dependent-launch attribute: the rows (and nothing else that is read
                                // here but weights and, routed, the tiles) are the stream's previous kernel's output, and that
                                // kernel lets this one start only after its own wait
    uint32_t beside;            // with overlap: the rows were complete before the stream's previous kernel (a GEMM of another bank on the
                                // same rows) started, so they are not waited for; this kernel still ends after that one
};

// max_units: an upper bound of the launch's units of work (the kernel is persistent; a smaller grid serves a small call)
cudaError_t launch_decode_gemm(const GemmMaps& maps, const DecodeGemmArgs& a, uint32_t max_units, int codebook, cudaStream_t stream);

}  // namespace t3
