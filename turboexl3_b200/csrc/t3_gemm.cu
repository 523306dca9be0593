// The decode GEMM of the prefill rows: z = f16(xp W_hat) and the output rotation, with the trellis decoded into TENSOR MEMORY.
//
// The product is taken transposed: D [128 outputs x rows] = W_hat^T x xp^T. The weight tile is the MMA's A operand, read from
// tensor memory, and the prepared rows are its B operand, K-major in shared memory as they lie in global memory. A lane's
// decoded words of a 16x16 tile are the A fragment of the transposed tile (the pack's tensor-core order), which is the register
// layout of tcgen05.st.16x128b: a tile goes to tensor memory in one instruction, with no swizzled shared-memory stores and no
// proxy fence, and shared memory carries only the rows. The accumulator's columns are rows, so a tile is any multiple of 16
// rows up to 256 and an expert of 80 rows costs five sixteenths of the MMA time of a 256-row one: nothing is padded to 128.
//
// What bounds it: a decoded 16x16 tile costs about 55 issued warp instructions, epilogue and waits included (55.3 of a routed gate|up at K3, 55.2
// of 2048 -> 6144 at K4; 67 of a routed down, whose units are 512 inputs), an MMA of 64 inputs x 128 outputs x R rows takes 2 R cycles,
// so up to about 200 rows a tile the decode's issue slots bound the kernel and past that the tensor cores do. Calls of thousands of rows run at the board's power limit (980 W, 1.4 to 1.8 GHz), where what a pass costs is its
// energy: with the decode skipped 2048 -> 6144 at 4096 rows took 88 us of 117, with the rows' copies skipped 103. (An MMA that
// reads its A operand from tensor memory ran at the full rate from 128 columns on: 64 cycles at 128, 128 at 256; with both operands in shared memory a 256-column one took 171.)
//
// One persistent CTA a multiprocessor, 28 warps by role (the rings run on across tiles, so nothing is set up per tile):
//   warps 0-7    epilogue     warps 8-23  decode     24  codes: TMA into the code ring
//   25  rows: TMA into the row ring     26  tcgen05.mma     27  the output rotation's tcgen05.mma, finished tiles out by TMA
// A ring stage is 64 weight tiles (64 tensor-memory columns), one of two shapes chosen per tile of rows:
//   wide   two 128-output blocks x 64 inputs, up to 128 rows: both blocks read one copy of the rows
//   deep   one block x 128 inputs, up to 256 rows
// A decode warp takes eight tiles of every other stage: waits, fences and arrivals are paid once for the eight.
//
// Epilogue: the 128-point output rotation is a tensor-core product as well, D2 = H128 x z^T with H128 (+-1, f16) resident in
// tensor memory: accumulators -> f16 z, transposed to shared memory by stmatrix -> MMA over the same columns, or free ones (Sub::early) ->
// scaled by svh, rounded, transposed again and sent out by TMA or stored in 256-byte runs. (On the warps' mma.sync with butterflies a row
// cost four times the instructions, and issue slots are what the decode needs.) From a 256-row tile's last MMA to the next tile's first took
// 5900 cycles of 23300 and takes 4400 of 20400; of a routed pair of 80-row tiles (512 inputs) 6500 of 13400, now 3000 to 4000 of 10400.
//
// Every wait is bounded: one that runs out sets a bit of the device error word and a flag that ends every other role's waits,
// and the CTA walks to its exit, freeing its tensor memory on the way.
#include <atomic>
#include <type_traits>

#include "t3_common.cuh"
#include "t3_gemm.h"
#include "t3_internal.h"
#include "t3_tcgen05.cuh"

#ifndef T3_CB
#error "T3_CB: the codebook this unit is compiled for"
#endif

namespace t3 {
namespace {

constexpr uint32_t kEpiWarps = 8, kDecWarps = 16;
constexpr uint32_t kCodeWarp = kEpiWarps + kDecWarps, kRowWarp = kCodeWarp + 1, kMmaWarp = kCodeWarp + 2, kRotWarp = kCodeWarp + 3;
constexpr uint32_t kThreads = 32u * (kRotWarp + 1u);
constexpr uint32_t kCodeStages = 4;        // stages of the code ring: even, so that a slot is always the same decode group's
constexpr uint32_t kStages = 3;            // operand stages in tensor memory
static_assert(kCodeStages % 2u == 0u, "see decode_stages");
// The decode warps work as two groups of eight on alternate stages, a warp on both of a stage's 64 x 128 blocks: eight tiles a
// visit, so that a visit's waits, arrivals and ring arithmetic are paid half as often as with sixteen warps on every stage (five
// issued instructions a tile fewer), and sixteen warps to issue from (eight alone left a third of the issue slots empty).
constexpr uint32_t kGroupWarps = 8;
constexpr uint32_t kStageTiles = 64;       // weight tiles a stage
constexpr uint32_t kStageCols = 64;        // tensor-memory columns a stage (32 a 64 x 128 block)
// tensor memory: accumulators in columns 0-255, operand stages in 256-447, H128 (128 x 128 f16) in 448-511
constexpr uint32_t kTmemCols = 512, kTmemA = 256, kTmemH = 448;
// Units whose accumulators leave room for one part's rotation beside them in columns 256 - rows .. 255: their accumulators are
// given back as soon as z is in shared memory, and the next unit's MMAs run under the rotation, the finish and the stores. (A launch
// has either blocks in pairs or one at a time, so no early unit's accumulators reach another's rotation columns.)
constexpr uint32_t kEarlyWide = 80, kEarlyDeep = 128;
static_assert(3u * kEarlyWide <= kTmemA && 2u * kEarlyDeep <= kTmemA, "accumulators and one part's rotation");
constexpr uint32_t kRowBytes = kGemmTileRows * 128u;   // a row slot: 64 inputs of up to 256 rows
constexpr uint32_t kKeptBytes = 128u * 128u;           // 64 inputs of a kept weight's 128 outputs, behind the slot's rows
constexpr uint32_t kZBytes = 2u * 128u * 128u;         // 128 rows x 128 outputs, f16, as two K-major halves; two of them

constexpr uint32_t row_slots(uint32_t n) { return n != 0u && n <= 64u ? 4u : 3u; }  // what fits beside the code ring
constexpr uint32_t smem_bytes(uint32_t n, uint32_t slots) {
    return slots * kRowBytes + 2u * kZBytes + kCodeStages * kStageTiles * 2u * n + 512u + 1024u;
}
static_assert(smem_bytes(128, 3) <= 227u * 1024u && smem_bytes(64, 4) <= 227u * 1024u, "shared memory of a CTA");

// one accumulator's worth of work: `blocks` 128-output blocks (2 in wide form) from block `blk` on, of one tile of rows
struct Sub {
    uint32_t e, first, rows, cols, op, blk, blocks;
    uint32_t k0, k1;  // its range of 64-input steps
    bool wide;
    bool early;       // the accumulators are free once their sums are in z: the rotation has columns of its own
    __device__ __forceinline__ uint32_t parts() const { return wide ? blocks : (cols > 128u ? 2u : 1u); }  // of up to 128 columns
    __device__ __forceinline__ uint32_t part_cols(uint32_t c) const { return wide ? cols : min(128u, cols - 128u * c); }
    __device__ __forceinline__ uint32_t rot_col(uint32_t c) const { return early ? 256u - cols : part_col(c); }  // its rotation's
    __device__ __forceinline__ uint32_t part_col(uint32_t c) const { return wide && early ? c * cols : 128u * c; }  // part c's columns
};

// the CTA's units in order; f(sub) returns false to stop
template <typename F>
__device__ __forceinline__ void for_each_sub(const DecodeGemmArgs& a, F&& f) {
    const uint32_t ncol = a.N / 128u, per_op = (ncol + a.pair - 1u) / a.pair, per_tile = per_op * a.ops;
    const uint32_t tile0 = a.tiles ? a.range[0] : 0u, tiles = a.tiles ? a.range[1] - tile0 : a.dense_tiles;
    const uint32_t total = tiles * per_tile;
    const bool sliced = a.ksplit > 1u;
    for (uint32_t u = sliced ? blockIdx.y : blockIdx.x; u < total; u += sliced ? total : gridDim.x) {
        const uint32_t t = u / per_tile, r = u - t * per_tile;
        Sub s;
        s.op = r / per_op;
        const uint32_t b0 = (r - s.op * per_op) * a.pair, nb = min(a.pair, ncol - b0);
        if (a.tiles) {
            const int4 d = a.tiles[tile0 + t];
            s.e = (uint32_t)d.x, s.first = (uint32_t)d.y, s.rows = (uint32_t)d.z;
        } else {
            s.e = 0, s.first = t * a.tile_rows, s.rows = min(a.tile_rows, a.dense_rows - s.first);
        }
        s.cols = (s.rows + 15u) & ~15u;
        s.wide = a.pair == 2u && s.cols <= 128u;
        s.blocks = s.wide ? nb : 1u;
        s.early = !sliced && a.svh[0] != nullptr && s.cols <= (a.pair == 2u ? kEarlyWide : kEarlyDeep);
        s.k0 = 0, s.k1 = a.K / 64u;
        if (sliced) s.k0 = 2u * (a.K / 128u * blockIdx.x / a.ksplit), s.k1 = 2u * (a.K / 128u * (blockIdx.x + 1u) / a.ksplit);
        for (uint32_t b = 0; b < nb; b += s.blocks) {
            s.blk = b0 + b;
            if (!f(s)) return;
        }
    }
}

// Waits for a barrier phase; false when the wait ran out, or once any wait of the CTA has (`dead` says so to all of them: from
// then on no wait takes time, so every role still walks to the end of its work, on values nobody will use). NAP: nanoseconds
// a warp sleeps between polls, for the roles whose waits are long and not urgent.
constexpr uint32_t kTries = 1u << 22;
template <uint32_t NAP = 0>
__device__ __forceinline__ bool wait_phase(uint32_t bar, uint32_t parity, volatile uint32_t* dead, uint32_t* err, uint32_t bit) {
    if (mbar_try(bar, parity)) return true;
#pragma unroll 1
    for (uint32_t i = 0; i < kTries; ++i) {
        if (NAP) __nanosleep(NAP);
        if (mbar_try(bar, parity)) return true;
        if (*dead) return false;
    }
    *dead = 1u;
    if (err) atomicOr(err, bit);
    return false;
}

// a ring position and the parity of its round (a wait for the parity before a fresh barrier's first phase returns at once, so a
// first round needs no case of its own)
template <uint32_t SLOTS>
struct Ring {
    uint32_t slot = 0, parity = 0;
    __device__ __forceinline__ void next(uint32_t by = 1) {
        slot += by;
        if (slot >= SLOTS) slot -= SLOTS, parity ^= 1u;
    }
};

// A decode group's pass over its stages of one sub-tile (every other one, `visits` of them from the ring's position on). A warp's
// tiles lie a row of 8 tiles apart in the code stage: four along K of the stage's first block, four of its second (PARTS 2).
// FULL: the codeword is the whole 16-bit window (no mask).
//
// A wait by parity can only tell a barrier's current phase from the one before, so whoever waits for a phase must know that the
// phase before it is over. A group that came back to a code slot which the OTHER group used last would not (its codes may not
// even have landed: the wait would return at once, on the round before); with an even ring a slot stays with one group. On the
// operand ring of three stages the group has always seen a later stage's MMAs complete than the ones before those it waits for.
template <int NN, int CB, bool FULL, uint32_t PARTS>
__device__ __forceinline__ void decode_stages(uint32_t visits, Ring<kCodeStages>& cring, Ring<kStages>& ring, uint32_t codes, uint32_t stage_bytes, uint32_t n,
                                              uint32_t first_tile, const LanePlan<(NN > 0 ? NN : 16)>& plan, uint32_t mask,
                                              uint32_t lane, uint32_t tmem_dst, uint32_t full_c, uint32_t full_a, volatile uint32_t* dead,
                                              uint32_t* err) {
    constexpr int NP = NN > 0 ? NN : 16;
    constexpr uint32_t kRaw = raw_words(NP);
    const uint32_t tile_bytes = 2u * (NN > 0 ? (uint32_t)NN : n);
    uint32_t at[kRaw];
#pragma unroll
    for (uint32_t j = 0; j < kRaw; ++j) at[j] = codes + first_tile * tile_bytes + plan.idx[j] * 4u;
#pragma unroll 1
    for (uint32_t k = 0; k < visits; ++k) {
        const uint32_t cbar = full_c + 16u * cring.slot, abar = full_a + 16u * ring.slot, off = cring.slot * stage_bytes;
        const uint32_t col = tmem_dst + ring.slot * kStageCols;
        wait_phase<20>(cbar, cring.parity, dead, err, kErrFullWait);
#pragma unroll
        for (uint32_t p = 0; p < PARTS; ++p) {
            uint32_t raw[4][kRaw];
            if (NN > 0) {
#pragma unroll
                for (uint32_t i = 0; i < 4u; ++i)
#pragma unroll
                    for (uint32_t j = 0; j < kRaw; ++j)
                        asm volatile("ld.shared.b32 %0, [%1];" : "=r"(raw[i][j]) : "r"(at[j] + off + (p * 4u + i) * 16u * (uint32_t)NP));
            }
            if (p == 0) {
                wait_phase<20>(abar + 8u, ring.parity ^ 1u, dead, err, kErrEmptyWait);
                tc_fence_after();
            }
#pragma unroll
            for (uint32_t i = 0; i < 4u; ++i) {
                uint32_t w[4];
                if (NN > 0)
                    decode_raw<NP, CB, FULL>(raw[i], plan, mask, w);
                else
                    decode_lane_any<CB>(static_cast<const uint32_t*>(__cvta_shared_to_generic(
                                            codes + off + (first_tile + (p * 4u + i) * 8u) * tile_bytes)), n, lane, mask, w);
                tmem_st_tile(col + 32u * p + 8u * i, w);
                // the last tile's words are in registers by now: the code slot may be refilled while this stage is finished
                if (p + 1u == PARTS && i == 2u && NN > 0) {
                    __syncwarp();
                    if (lane == 0) mbar_arrive_addr(cbar + 8u);
                }
            }
        }
        tmem_st_wait();
        tc_fence_before();
        if (lane == 0) {
            if (NN == 0) mbar_arrive_addr(cbar + 8u);
            mbar_arrive_addr(abar);
        }
        cring.next(2), ring.next(2);
    }
}

// A warp's 16 outputs of up to 128 accumulator columns: f(r, v) gets columns r .. r + 31. Two loads are on their way at once and one
// wait is for both (tcgen05.wait::ld knows no single load; a load's latency for every 32 columns was half of what the epilogue took); the second
// wait only keeps its registers' use behind it.
template <typename F>
__device__ __forceinline__ void for_columns(uint32_t taddr, uint32_t cols, F&& f) {
    uint32_t v[2][16];
#pragma unroll
    for (uint32_t r = 0; r < 128u; r += 64u) {
        if (r >= cols) break;
        tmem_ld_16x32(taddr + r, v[0]);
        tmem_ld_16x32(taddr + r + 32u, v[1]);
        tmem_ld_wait(v[0]);
        f(r, v[0]);
        tmem_ld_wait(v[1]);
        if (r + 32u < cols) f(r + 32u, v[1]);
    }
}

// The sums of an accumulator part as f16 z^T, K-major in the part's buffer (st_at: where this lane's stmatrix row goes): the output
// rotation's B operand
__device__ __forceinline__ void z_part(uint32_t taddr, uint32_t cols, uint32_t st_at) {
    for_columns(taddr, cols, [&](uint32_t r, const uint32_t (&v)[16]) {
#pragma unroll
        for (uint32_t p = 0; p < 2u; ++p) {
            auto pk = [&](uint32_t j) { return pack_half2(__uint_as_float(v[8u * p + j]), __uint_as_float(v[8u * p + j + 1u])); };
            if (r + 16u * p < cols) stmatrix4_trans(st_at + (r + 16u * p) * 128u, pk(0), pk(2), pk(4), pk(6));
        }
    });
}

// (a, b) x s
__device__ __forceinline__ float2 mul2(uint32_t a, uint32_t b, float s) {
    float2 r;
    asm("{\n\t.reg .b64 u, v, w;\n\tmov.b64 u, {%2, %3};\n\tmov.b64 v, {%4, %4};\n\tmul.rn.f32x2 w, u, v;\n\tmov.b64 {%0, %1}, w;\n\t}"
        : "=f"(r.x), "=f"(r.y)
        : "r"(a), "r"(b), "f"(s));
    return r;
}

// One part of up to 128 columns of a finished accumulator, warp (q, h)'s 16 outputs of it: rotated sums x scale, rounded to f16, then in
// the output's dtype (PLAIN: rounded once). 16-bit results are transposed into the part's buffer (st_at: where this lane's
// stmatrix row goes), f32 ones go to y, rows below `live`, at once (y at the part's first row and this lane's output g). A body a
// dtype: with the three in one the code was long enough to be fetched anew for every tile, 1700 cycles a part against 500.
template <bool PLAIN, int DT>
__device__ __forceinline__ void finish_part_as(uint32_t taddr, uint32_t cols, float s0, float s1, uint32_t st_at, float* y, size_t N,
                                               uint32_t live, uint32_t t) {
    for_columns(taddr, cols, [&](uint32_t r, const uint32_t (&v)[16]) {
#pragma unroll
        for (uint32_t p = 0; p < 2u; ++p) {
            uint32_t w[4];
#pragma unroll
            for (uint32_t j = 0; j < 4u; ++j) {  // rows 8 (j >> 1) + 2t and the next of 16, output g or g + 8 (j odd)
                const uint32_t a = v[8u * p + 2u * j], b = v[8u * p + 2u * j + 1u];
                float2 u = PLAIN ? make_float2(__uint_as_float(a), __uint_as_float(b)) : mul2(a, b, (j & 1u) ? s1 : s0);
                if (DT == (int)kF32) {
                    const uint32_t row = r + 16u * p + (j >> 1) * 8u + 2u * t;
                    float* at = y + row * N + ((j & 1u) ? 8u : 0u);
                    if (row < live) at[0] = round_half(u.x);
                    if (row + 1u < live) at[N] = round_half(u.y);
                    continue;
                }
                w[j] = pack_half2(u.x, u.y);
                if (DT == (int)kBf16) {
                    if (!PLAIN) u = __half22float2(*reinterpret_cast<const __half2*>(&w[j]));
                    const __nv_bfloat162 o = __floats2bfloat162_rn(u.x, u.y);
                    w[j] = *reinterpret_cast<const uint32_t*>(&o);
                }
            }
            if (DT != (int)kF32 && r + 16u * p < cols) stmatrix4_trans(st_at + (r + 16u * p) * 128u, w[0], w[1], w[2], w[3]);
        }
    });
}
template <bool PLAIN>
__device__ __forceinline__ void finish_part(uint32_t taddr, uint32_t cols, float s0, float s1, int dt, uint32_t st_at, float* y,
                                            size_t N, uint32_t live, uint32_t t) {
    if (dt == (int)kF16) finish_part_as<PLAIN, kF16>(taddr, cols, s0, s1, st_at, y, N, live, t);
    else if (dt == (int)kBf16) finish_part_as<PLAIN, kBf16>(taddr, cols, s0, s1, st_at, y, N, live, t);
    else finish_part_as<PLAIN, kF32>(taddr, cols, s0, s1, st_at, y, N, live, t);
}

// A part's 16-bit rows from its buffer to y, 256 bytes a row (`warp` of the epilogue's eight); a caller's y may be aligned to 8
// bytes only
__device__ __forceinline__ void store_part(uint32_t buffer, uint16_t* y, size_t N, uint32_t rows, uint32_t warp, uint32_t lane) {
    const uint32_t j = lane & 15u;
    const bool wide = aligned16(y);
#pragma unroll 4
    for (uint32_t r = 2u * warp + (lane >> 4); r < rows; r += 2u * kEpiWarps) {
        uint4 w;
        asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(w.x), "=r"(w.y), "=r"(w.z), "=r"(w.w)
                     : "r"(buffer + (j >> 3) * 16384u + r * 128u + (((j & 7u) ^ (r & 7u)) << 4)));
        uint16_t* at = y + r * N + 8u * j;
        if (wide) *reinterpret_cast<uint4*>(at) = w;
        else reinterpret_cast<uint2*>(at)[0] = make_uint2(w.x, w.y), reinterpret_cast<uint2*>(at)[1] = make_uint2(w.z, w.w);
    }
}

// A part's rows by TMA, boxes of at least eight rows (a box starts where the 128-byte swizzle does), and what is left of it by the warp
// (x: the part's first output, y: its first row in maps.out, at: that value's place in memory). Lane 0 keeps the copies as a bulk group.
__device__ __forceinline__ void send_part(const GemmMaps& maps, uint32_t buffer, int x, int y, uint16_t* at, size_t N, uint32_t rows, uint32_t lane) {
    const uint32_t whole = rows & ~7u;
    if (lane == 0) {
        uint32_t r = 0;
#pragma unroll
        for (uint32_t i = 0; i < 5u; ++i) {
            const uint32_t h = 128u >> i;
            if (whole - r < h) continue;
            tma_store_2d(&maps.out[i], x, y + (int)r, buffer + r * 128u);
            tma_store_2d(&maps.out[i], x + 64, y + (int)r, buffer + 16384u + r * 128u);
            r += h;
        }
        bulk_commit();
    }
    for (uint32_t i = lane; i < (rows - whole) * 16u; i += 32u) {
        const uint32_t r = whole + (i >> 4), j = i & 15u;
        uint4 w;
        asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(w.x), "=r"(w.y), "=r"(w.z), "=r"(w.w)
                     : "r"(buffer + (j >> 3) * 16384u + r * 128u + (((j & 7u) ^ (r & 7u)) << 4)));
        *reinterpret_cast<uint4*>(at + r * N + 8u * j) = w;
    }
    __syncwarp();
}

// store_part with each row's f16 values times its score (of the part's first row on), stored as the final sum of one slot a row stores
// them: 0 + w v in f32, rounded once to y's dtype (y at the part's first value, element `at` of a.y)
__device__ __forceinline__ void store_scored(uint32_t buffer, const DecodeGemmArgs& a, size_t first, size_t at, uint32_t rows, uint32_t warp, uint32_t lane) {
    const uint32_t j = lane & 15u;
#pragma unroll 2
    for (uint32_t r = 2u * warp + (lane >> 4); r < rows; r += 2u * kEpiWarps) {
        uint32_t w[4];
        asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3])
                     : "r"(buffer + (j >> 3) * 16384u + r * 128u + (((j & 7u) ^ (r & 7u)) << 4)));
        const float score = load_act(a.scores, a.score_dt, first + r);
#pragma unroll
        for (uint32_t half = 0; half < 2u; ++half) {
            const float2 u = unpack_half2(w[2u * half]), v = unpack_half2(w[2u * half + 1u]);
            float f[4] = {u.x, u.y, v.x, v.y};
#pragma unroll
            for (uint32_t i = 0; i < 4u; ++i) f[i] = __fadd_rn(0.0f, __fmul_rn(score, f[i]));
            store_act4(a.y, a.y_dt, at + r * (size_t)a.N + 8u * j + 4u * half, f);
        }
    }
}

// The output rotation of a part on the tensor cores (one thread): D2 = H128 x z^T into the columns at tmem_d
__device__ __forceinline__ void rotate_part(uint32_t tmem, uint32_t tmem_d, uint32_t z, uint32_t idesc, uint32_t rot_full) {
    const uint32_t hi = (uint32_t)(umma_desc(0) >> 32), lo = (uint32_t)umma_desc(z);
#pragma unroll
    for (uint32_t kk = 0; kk < 8u; ++kk)
        umma_f16_ts(tmem_d, tmem + kTmemH + 8u * kk, lo + (((kk >> 2) * 16384u + (kk & 3u) * 32u) >> 4), hi, kk != 0u, idesc);
    umma_commit(rot_full);
}

__device__ __forceinline__ void add_to(float2& a, float2 b) { a.x += b.x, a.y += b.y; }
__device__ __forceinline__ void add_to(float4& a, float4 b) { a.x += b.x, a.y += b.y, a.z += b.z, a.w += b.w; }
// Sums over `slices` (at most MOST) of `count` values `next` apart, in slice order; f(at, sums) gets those of values `at` ..
template <uint32_t MOST, typename V, typename F>
__device__ __forceinline__ void sum_slices(const float* slab, size_t next, uint32_t slices, uint32_t count, uint32_t tid, F&& f) {
    constexpr uint32_t kAtOnce = 3, kWide = sizeof(V) / 4u;
    for (uint32_t i0 = tid * kWide; i0 < count; i0 += kAtOnce * kThreads * kWide) {
        V p[kAtOnce][MOST];
#pragma unroll
        for (uint32_t k = 0; k < kAtOnce; ++k)
#pragma unroll
            for (uint32_t z = 0; z < MOST; ++z)
                if (z < slices && i0 + k * kThreads * kWide < count) p[k][z] = __ldcg(reinterpret_cast<const V*>(slab + z * next + i0 + k * kThreads * kWide));
#pragma unroll
        for (uint32_t k = 0; k < kAtOnce; ++k) {
            if (i0 + k * kThreads * kWide >= count) break;
            V sum = p[k][0];
#pragma unroll
            for (uint32_t z = 1; z < MOST; ++z)
                if (z < slices) add_to(sum, p[k][z]);
            f(i0 + k * kThreads * kWide, sum);
        }
    }
}

// KEPT: the weight is a kept W_hat (or W_std), [N, K] 16-bit, loaded by TMA beside the rows as a shared-memory operand: the
// same products in the same order, nothing decoded.
template <int NN, int CB, bool KEPT = false>
__global__ void __launch_bounds__(kThreads, 1) decode_gemm_kernel(const __grid_constant__ GemmMaps maps, const DecodeGemmArgs a) {
    constexpr uint32_t kSlots = KEPT ? 3u : row_slots(NN), kSlotBytes = KEPT ? kRowBytes + kKeptBytes : kRowBytes;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem = (smem_addr(smem_raw) + 1023u) & ~1023u;
    const uint32_t n = NN > 0 ? (uint32_t)NN : (KEPT ? 0u : a.n), tile_bytes = 2u * n, stage_bytes = kStageTiles * tile_bytes;
    const uint32_t z_s = smem + kSlots * kSlotBytes, codes = z_s + 2u * kZBytes;
    // barriers, a full / empty pair a ring slot: codes, operands in tensor memory, rows
    const uint32_t full_c = codes + kCodeStages * stage_bytes, full_a = full_c + 16u * kCodeStages;
    const uint32_t full_b = full_a + 16u * kStages, empty_b = full_b + 8u * 4u;
    // acc_free: the accumulators may be written again; all_free: the rotation's columns too (the same moment unless Sub::early)
    const uint32_t acc_full = empty_b + 8u * 4u, acc_free = acc_full + 8u, all_free = acc_full + 16u;
    // z_full, rot_full: a pair each, one barrier a part of up to 128 columns
    const uint32_t z_full = acc_full + 24u, rot_full = acc_full + 40u;
    // and with outputs by TMA: a part's values are in its buffer, its buffer is read
    const uint32_t fin_full = acc_full + 56u, z_free = acc_full + 72u;
    uint8_t* generic = smem_raw + (smem - smem_addr(smem_raw));
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(generic + (acc_full + 88u - smem));
    volatile uint32_t* dead = tmem_slot + 1;

    const uint32_t tid = threadIdx.x, lane = tid & 31u;
    // the warp's number as a value the compiler knows to be the same in every lane: the roles' loops then run on uniform registers
    const uint32_t warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0);
    if (tid == 0) {
        auto init = [&](uint32_t bar, uint32_t count) { mbar_init(reinterpret_cast<uint64_t*>(generic + (bar - smem)), count); };
        for (uint32_t s = 0; s < kCodeStages; ++s) init(full_c + 16u * s, 1u), init(full_c + 16u * s + 8u, kGroupWarps);
        for (uint32_t s = 0; s < kStages; ++s) init(full_a + 16u * s, kGroupWarps), init(full_a + 16u * s + 8u, 1u);
        for (uint32_t s = 0; s < kSlots; ++s) init(full_b + 8u * s, 1u), init(empty_b + 8u * s, 1u);
        init(acc_full, 1u), init(acc_free, kEpiWarps), init(all_free, kEpiWarps);
        for (uint32_t c = 0; c < 2u; ++c) init(z_full + 8u * c, kEpiWarps), init(rot_full + 8u * c, 1u), init(fin_full + 8u * c, kEpiWarps), init(z_free + 8u * c, 1u);
        *dead = 0u;
        mbar_init_fence();
    }
    if (warp == kMmaWarp) tmem_alloc(tmem_slot, kTmemCols);
    if (warp == kRowWarp && lane < 6u) prefetch_map(lane < 4u ? &maps.rows[lane] : &maps.codes[lane == 5u && a.ops > 1u]);
    if (tid == 32u) pdl_trigger();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xFFFFFFFFu, *tmem_slot, 0);
    const bool sliced = a.ksplit > 1u;
    // H128 as an A operand in tensor memory: element (i, j) has the sign of popcount(i & j)
    if (warp < 8u) {
        const uint32_t i = 32u * (warp & 3u) + 16u * ((warp >> 2) & 1u) + (lane >> 2), j0 = 2u * (lane & 3u);
        auto pair = [](uint32_t r, uint32_t c) {
            return ((__popc(r & c) & 1) ? 0xBC00u : 0x3C00u) | ((__popc(r & (c + 1u)) & 1) ? 0xBC000000u : 0x3C000000u);
        };
        for (uint32_t kk = 0; kk < 8u; ++kk) {
            const uint32_t j = 16u * kk + j0;
            const uint32_t w[4] = {pair(i, j), pair(i, j + 8u), pair(i + 8u, j), pair(i + 8u, j + 8u)};
            tmem_st_tile(tmem + kTmemH + 8u * kk + ((i & ~7u) << 16), w);
        }
        tmem_st_wait();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();

    if (warp >= kEpiWarps && warp < kCodeWarp) {
        // ---- decode: quarter q of the lanes (32 outputs a block), tile column 2q + half of a block, stages of the group's parity
        const uint32_t q = warp & 3u, half = ((warp - kEpiWarps) >> 2) & 1u, group = (warp - kEpiWarps) / kGroupWarps;
        LanePlan<(NN > 0 ? NN : 16)> plan;
        plan.init(lane);
        const uint32_t dst = tmem + kTmemA + ((32u * q + 16u * half) << 16), col = 2u * q + half;
        Ring<kCodeStages> cring;
        Ring<kStages> ring;
        if (group) cring.next(), ring.next();
        uint32_t ahead = group;  // stages from a sub-tile's first to the group's next one: 0 or 1
        const bool full = a.mask == 0xFFFFu;
        if (!KEPT) for_each_sub(a, [&](const Sub& s) {
            const uint32_t stages = s.wide ? s.k1 - s.k0 : (s.k1 - s.k0) / 2u, visits = (stages + 1u - ahead) / 2u;
            auto run = [&](auto fullw, auto parts) {
                decode_stages<NN, CB, decltype(fullw)::value, decltype(parts)::value>(visits, cring, ring, codes, stage_bytes, n, col, plan,
                                                                                      a.mask, lane, dst, full_c, full_a, dead, a.err);
            };
            using One = std::integral_constant<uint32_t, 1>;
            using Two = std::integral_constant<uint32_t, 2>;
            if (s.wide && s.blocks == 1u) full ? run(std::true_type(), One()) : run(std::false_type(), One());  // no second block
            else full ? run(std::true_type(), Two()) : run(std::false_type(), Two());
            ahead = (ahead + stages) & 1u;  // an odd number of stages hands the next sub-tile's first one to the other group
            return true;
        });
    } else if (warp == kCodeWarp) {
        // ---- code ring: a stage is two boxes of 4 tile rows x 8 tiles, the unit's two blocks (wide) or two runs of 64 inputs
        // (deep). A slot is free again when every decode warp has its words in registers.
        Ring<kCodeStages> ring;
        if (!KEPT) for_each_sub(a, [&](const Sub& s) {
            const CUtensorMap* map = &maps.codes[s.op];
            const uint32_t words = n * 2u, box = 4u * 8u * tile_bytes;  // 64-bit words of a row of 8 tiles
            const bool two = !s.wide || s.blocks == 2u;
            const int x0 = (int)(s.blk * words), x1 = x0 + (s.wide ? (int)words : 0), e = (int)s.e, dy = s.wide ? 0 : 4;
            for (uint32_t k = 4u * s.k0; k < 4u * s.k1; k += s.wide ? 4u : 8u, ring.next()) {
                const uint32_t bar = full_c + 16u * ring.slot, dst = codes + ring.slot * stage_bytes;
                if (!wait_phase<64>(bar + 8u, ring.parity ^ 1u, dead, a.err, kErrEmptyWait)) return false;
                __syncwarp();
                if (elect_one()) {
                    mbar_arrive_expect_tx_addr(bar, two ? 2u * box : box);
                    tma_load_3d(dst, map, x0, (int)k, e, bar);
                    if (two) tma_load_3d(dst + box, map, x1, (int)k + dy, e, bar);
                }
            }
            return true;
        });
    } else if (warp == kRowWarp) {
        // ---- row ring: 64 inputs of the tile's rows a slot. The rows are the previous kernel's output; the other roles' inputs
        // are not, so the codes stream in and the first stages decode while that kernel finishes.
        if (!a.beside) pdl_wait();
        Ring<kSlots> ring;
        for_each_sub(a, [&](const Sub& s) {
            const int row0 = (int)(s.op * a.op_rows + s.first);
            // one box, or one and a half-sized one
            const uint32_t load = tiled_rows(s.cols), big = load == 192u ? 128u : load == 96u ? 64u : load;
            const CUtensorMap* map = &maps.rows[big == 256u ? 0 : big == 128u ? 1 : big == 64u ? 2 : 3];
            for (uint32_t k = s.k0; k < s.k1; ++k, ring.next()) {
                const uint32_t bar = full_b + 8u * ring.slot, dst = smem + ring.slot * kSlotBytes;
                if (!wait_phase<32>(empty_b + 8u * ring.slot, ring.parity ^ 1u, dead, a.err, kErrEmptyWait)) return false;
                __syncwarp();
                if (elect_one()) {
                    mbar_arrive_expect_tx_addr(bar, load * 128u + (KEPT ? kKeptBytes : 0u));
                    if (KEPT) tma_load_2d(dst + kRowBytes, &maps.codes[0], (int)(k * 64u), (int)(s.blk * 128u), bar);
                    tma_load_2d(dst, map, (int)(k * 64u), row0, bar);
                    if (load != big) tma_load_2d(dst + big * 128u, map + 1, (int)(k * 64u), row0 + (int)big, bar);
                }
            }
            return true;
        });
        if (a.beside) pdl_wait();
    } else if (warp == kMmaWarp) {
        // ---- MMA: the whole warp walks the rings, one elected lane issues (see elect_one)
        uint32_t subs = 0;
        Ring<kStages> ring_a;
        Ring<kSlots> ring_b;
        auto wait = [&](uint32_t bar, uint32_t parity, uint32_t bit) {
            wait_phase(bar, parity, dead, a.err, bit);
            tc_fence_after();
            __syncwarp();
        };
        const uint32_t desc_hi = (uint32_t)(umma_desc(0) >> 32), desc0 = (uint32_t)umma_desc(smem);
        for_each_sub(a, [&](const Sub& s) {
            if (subs > 0u) {
                wait(acc_free, (subs - 1u) & 1u, kErrMmaWait);
                // accumulators wide enough to reach the last unit's rotation (which finished the one before: a phase's parity is enough)
                if (!s.early) wait(all_free, (subs - 1u) & 1u, kErrMmaWait);
            }
            ++subs;
            const uint32_t second = tmem + s.part_col(1);
            const uint32_t idesc = idesc_m128(s.cols) | (KEPT && a.bf16 ? kIdescBf16 : 0u), k64 = s.k1 - s.k0;
            uint32_t acc = 0;
            // four steps of 16 inputs on one row slot against one 64-input operand block (a second block's into its accumulator)
            auto steps = [&](uint32_t a_col, bool both) {
                const uint32_t lo = desc0 + ring_b.slot * (kSlotBytes >> 4);
#pragma unroll
                for (uint32_t kk = 0; kk < 4u; ++kk) {
                    if (KEPT) {
                        const uint64_t hi = (uint64_t)desc_hi << 32;
                        umma_f16(tmem, hi | (lo + (kRowBytes >> 4) + kk * 2u), hi | (lo + kk * 2u), kk ? 1u : acc, idesc);
                        continue;
                    }
                    umma_f16_ts(tmem, a_col + kk * 8u, lo + kk * 2u, desc_hi, kk ? 1u : acc, idesc);
                    if (both) umma_f16_ts(second, a_col + 32u + kk * 8u, lo + kk * 2u, desc_hi, kk ? 1u : acc, idesc);
                }
                umma_commit(empty_b + 8u * ring_b.slot);
            };
            const uint32_t stages = s.wide ? k64 : k64 / 2u;
#pragma unroll 1
            for (uint32_t k = 0; k < stages; ++k, ring_a.next()) {
                const uint32_t a_col = tmem + kTmemA + ring_a.slot * kStageCols;
                wait(full_b + 8u * ring_b.slot, ring_b.parity, kErrFullWait);
                if (!KEPT) wait(full_a + 16u * ring_a.slot, ring_a.parity, kErrFullWait);
                if (s.wide) {
                    if (elect_one()) {
                        if (s.blocks == 2u) steps(a_col, true);
                        else steps(a_col, false);
                        umma_commit(full_a + 16u * ring_a.slot + 8u);
                    }
                } else {
                    if (elect_one()) steps(a_col, false);
                    acc = 1u;
                    ring_b.next();
                    wait(full_b + 8u * ring_b.slot, ring_b.parity, kErrFullWait);
                    if (elect_one()) {
                        steps(a_col + 32u, false);
                        if (!KEPT) umma_commit(full_a + 16u * ring_a.slot + 8u);
                    }
                }
                acc = 1u;
                ring_b.next();
            }
            if (elect_one()) umma_commit(acc_full);
            return true;
        });
    } else if (warp == kRotWarp) {
        // ---- output rotation, a part at a time, once every epilogue warp's z is in the part's buffer (a warp of its own: the MMA warp
        // is on the next unit by then); then the finished parts' way out, where that is by TMA: the epilogue warps, which have a sixth of
        // the issue slots beside the decode, are on to the next unit meanwhile
        uint32_t turns[2] = {0, 0};
        uint16_t* const y16 = a.y ? static_cast<uint16_t*>(a.y) : reinterpret_cast<uint16_t*>(a.z);
        if (!sliced && a.svh[0] != nullptr) for_each_sub(a, [&](const Sub& s) {
            const uint32_t parts = s.parts();
#pragma unroll
            for (uint32_t c = 0; c < 2u; ++c) {
                if (c >= parts) break;
                wait_phase<32>(z_full + 8u * c, turns[c]++ & 1u, dead, a.err, kErrMmaWait);
                tc_fence_after();
                __syncwarp();
                const uint32_t to = tmem + s.rot_col(c), idesc = idesc_m128(s.part_cols(c));
                if (elect_one()) rotate_part(tmem, to, z_s + c * kZBytes, idesc, rot_full + 8u * c);
            }
            if (!a.bulk_out) return true;
#pragma unroll
            for (uint32_t c = 0; c < 2u; ++c) {
                if (c >= parts) break;
                wait_phase<32>(fin_full + 8u * c, (turns[c] - 1u) & 1u, dead, a.err, kErrMmaWait);
                __syncwarp();
                const uint32_t row = s.first + (s.wide ? 0u : 128u * c), x = (s.blk + (s.wide ? c : 0u)) * 128u;
                send_part(maps, z_s + c * kZBytes, (int)x, (int)(s.op * a.op_rows + row), y16 + s.op * a.z_op_stride + (size_t)row * a.N + x, a.N,
                          min(s.part_cols(c), s.rows - (s.wide ? 0u : 128u * c)), lane);
            }
            if (lane == 0) {
                if (parts == 2u) bulk_wait_read<1>(), mbar_arrive_addr(z_free);
                bulk_wait_read<0>();
                mbar_arrive_addr(z_free + 8u * (parts - 1u));
            }
            __syncwarp();
            return true;
        });
    } else {
        // ---- epilogue, warp (q, h): tensor-memory lanes (outputs) 32 q + 16 h .. + 15
        const uint32_t q = warp & 3u, h = warp >> 2, g = lane >> 2, t = lane & 3u;
        // where this lane's stmatrix row goes: row 8 (m >> 1) + i of 16, outputs 32 q + 16 h + 8 (m & 1) ..
        const uint32_t m = lane >> 3, i8 = lane & 7u;
        const uint32_t st_at = z_s + (q >> 1) * 16384u + ((m >> 1) * 8u + i8) * 128u + ((((q & 1u) * 4u + h * 2u + (m & 1u)) ^ i8) << 4);
        const uint32_t my_lanes = tmem + ((32u * q + 16u * h) << 16);
        const int dt = a.y && !a.scores ? a.y_dt : (int)kF16;
        const bool plain = KEPT && a.svh[0] == nullptr;
        uint16_t* const y16 = a.y ? static_cast<uint16_t*>(a.y) : reinterpret_cast<uint16_t*>(a.z);
        uint32_t subs = 0, rots = 0;  // rots: the next rotation's parity, a bit a part
        const bool bulk = a.bulk_out != 0u && !plain;
        auto arrive = [&](uint32_t bar) {
            __syncwarp();
            if (lane == 0) mbar_arrive_addr(bar);
        };
        // one warp polls, the others wait at the named barrier, where they issue nothing (every wait ends, so all eight get there)
        auto meet = [&]() { named_sync(1, 32u * kEpiWarps); };
        auto await = [&](uint32_t bar, uint32_t parity) {
            if (warp == 0) wait_phase<32>(bar, parity, dead, a.err, kErrMmaWait);
            meet();
            tc_fence_after();
        };
        for_each_sub(a, [&](const Sub& s) {
            float sc[2][2] = {};  // the scales of outputs g and g + 8 of this warp's 16, per block
            if (!plain) {
                const __half* svh = (s.op ? a.svh[1] : a.svh[0]) + (size_t)s.e * a.svh_stride + s.blk * 128u + 32u * q + 16u * h + g;
#pragma unroll
                for (uint32_t b = 0; b < 2u; ++b)
#pragma unroll
                    for (uint32_t j = 0; j < 2u; ++j)
                        if (b < s.blocks) sc[b][j] = kHadScale * __half2float(svh[b * 128u + 8u * j]);
            }
            await(acc_full, subs++ & 1u);
            const uint32_t parts = s.parts();
            if (sliced) {
                // This slice's sums to its place in the slab, a lane an output: a row's 128 are four 128-byte stores. (In the finish's
                // fragment layout a store went to four rows, 32 bytes each, and 200 rows took 2.7 us.)
                float* slab = a.part + (((size_t)s.blk * a.ksplit + blockIdx.x) * a.dense_rows + s.first) * 128u + 32u * q + lane;
#pragma unroll 1
                for (uint32_t r = 32u * h; r < s.cols; r += 64u) {
                    uint32_t v[32];
                    tmem_ld_32x32(tmem + ((32u * q) << 16) + r, v);
#pragma unroll
                    for (uint32_t j = 0; j < 32u; ++j)
                        if (r + j < s.rows) __stcg(slab + (size_t)(r + j) * 128u, __uint_as_float(v[j]));
                }
                return true;
            }
            // this warp's z of a part is in its buffer and the columns its rotation goes to are read
            auto z_done = [&](uint32_t c) {
                proxy_fence();
                tc_fence_before();
                arrive(z_full + 8u * c);
            };
            if (!plain) {
#pragma unroll 1
                for (uint32_t c = 0; c < parts; ++c) {
                    if (bulk) {  // the buffer's last part has left
                        wait_phase<32>(z_free + 8u * c, ((rots >> c) & 1u) ^ 1u, dead, a.err, kErrMmaWait);
                        __syncwarp();
                    }
                    z_part(my_lanes + s.part_col(c), s.part_cols(c), st_at + c * kZBytes);
                    if (c == 0u || !s.early) z_done(c);
                }
                if (s.early) {
                    tc_fence_before();
                    arrive(acc_free);
                }
            }
#pragma unroll 1
            for (uint32_t c = 0; c < parts; ++c) {
                if (!plain) {
                    if (s.early && c == 1u) z_done(c);  // the first part's rotation is read
                    await(rot_full + 8u * c, (rots >> c) & 1u);
                    rots ^= 1u << c;
                }
                const uint32_t cols = s.part_cols(c), blk = s.blk + (s.wide ? c : 0u), row0 = s.wide ? 0u : 128u * c;
                const bool second = s.wide && c == 1u;
                const float s0 = second ? sc[1][0] : sc[0][0], s1 = second ? sc[1][1] : sc[0][1];
                float* y32 = static_cast<float*>(a.y) + (size_t)(s.first + row0) * a.N + blk * 128u + 32u * q + 16u * h + g;
                const uint32_t from = my_lanes + s.rot_col(c);
                if (plain)
                    finish_part<true>(from, cols, s0, s1, dt, st_at + c * kZBytes, y32, a.N, s.rows - row0, t);
                else
                    finish_part<false>(from, cols, s0, s1, dt, st_at + c * kZBytes, y32, a.N, s.rows - row0, t);
                if (bulk) {
                    proxy_fence();
                    arrive(fin_full + 8u * c);
                }
            }
            // everything is read
            tc_fence_before();
            if (!s.early) arrive(acc_free);
            arrive(all_free);
            if (dt == (int)kF32 || bulk) return true;
            meet();
            for (uint32_t c = 0; c < parts; ++c) {
                const uint32_t row0 = s.wide ? 0u : 128u * c;
                if (a.scores) {
                    store_scored(z_s + c * kZBytes, a, s.first + row0, (size_t)(s.first + row0) * a.N + (s.blk + (s.wide ? c : 0u)) * 128u,
                                 min(s.part_cols(c), s.rows - row0), warp, lane);
                    continue;
                }
                store_part(z_s + c * kZBytes, y16 + s.op * a.z_op_stride + (size_t)(s.first + row0) * a.N + (s.blk + (s.wide ? c : 0u)) * 128u,
                           a.N, min(s.part_cols(c), s.rows - row0), warp, lane);
            }
            meet();  // the buffers are read: the next tile's values may overwrite them
            return true;
        });
    }
    if (sliced) {
        // The slices of a unit meet: every CTA of the cluster has left its sums in the slab once the cluster's barrier is passed;
        // CTA z then adds the slices, in slice order, of its share of the rows and finishes those.
        tc_fence_before();
        asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
        __syncthreads();
        tc_fence_after();
        Sub s = {};
        for_each_sub(a, [&](const Sub& mine) { s = mine; return true; });
        const uint32_t per = (s.rows + a.ksplit - 1u) / a.ksplit, lo = min(per * blockIdx.x, s.rows), live = min(per, s.rows - lo);
        const float* slab = a.part + ((size_t)s.blk * a.ksplit * a.dense_rows + s.first + lo) * 128u;
        const size_t next = (size_t)a.dense_rows * 128u;
        auto put = [&](uint32_t at, uint32_t w) {  // two rounded sums, values `at` and at + 1 of the share
            const uint32_t r = at >> 7, o = at & 127u;
            asm volatile("st.shared.b32 [%0], %1;" ::"r"(z_s + (o >> 6) * 16384u + r * 128u + ((((o & 63u) >> 3) ^ (r & 7u)) << 4) + (o & 7u) * 2u), "r"(w)
                         : "memory");
        };
        // three loads a slice and thread at once: of two values of up to eight slices, or of four of up to four
        if (a.ksplit > 4u)
            sum_slices<8, float2>(slab, next, a.ksplit, live * 128u, tid, [&](uint32_t at, float2 v) { put(at, pack_half2(v.x, v.y)); });
        else
            sum_slices<4, float4>(slab, next, a.ksplit, live * 128u, tid, [&](uint32_t at, float4 v) {
                put(at, pack_half2(v.x, v.y));
                put(at + 2u, pack_half2(v.z, v.w));
            });
        proxy_fence();
        __syncthreads();
        const uint32_t cols = (live + 15u) & ~15u;
        if (live > 0u) {
            if (warp == kMmaWarp) {
                if (elect_one()) rotate_part(tmem, tmem, z_s, idesc_m128(cols), rot_full);
            } else if (warp < kEpiWarps) {
                const uint32_t q = warp & 3u, h = warp >> 2, g = lane >> 2, t = lane & 3u, m = lane >> 3, i8 = lane & 7u;
                const uint32_t st_at = z_s + (q >> 1) * 16384u + ((m >> 1) * 8u + i8) * 128u + ((((q & 1u) * 4u + h * 2u + (m & 1u)) ^ i8) << 4);
                const uint32_t o = 32u * q + 16u * h + g;
                const size_t out0 = (size_t)(s.first + lo) * a.N + s.blk * 128u;
                const __half* svh = a.svh[0] + s.blk * 128u + o;
                const float s0 = kHadScale * __half2float(svh[0]), s1 = kHadScale * __half2float(svh[8]);
                wait_phase(rot_full, 0u, dead, a.err, kErrMmaWait);
                __syncwarp();
                tc_fence_after();
                finish_part<false>(tmem + ((32u * q + 16u * h) << 16), cols, s0, s1, a.y_dt, st_at, static_cast<float*>(a.y) + out0 + o, a.N,
                                   live, t);
                if (a.y_dt != (int)kF32) {
                    named_sync(1, 32u * kEpiWarps);
                    store_part(z_s, static_cast<uint16_t*>(a.y) + out0, a.N, live, warp, lane);
                }
            }
        }
    }
    // a CTA that gave up lets the copies in flight land before its shared memory goes away
    if (*dead)
        for (uint32_t i = 0; i < 1000u; ++i) __nanosleep(1000);
    tc_fence_before();
    __syncthreads();
    if (warp == kMmaWarp) {
        tc_fence_after();
        tmem_dealloc(tmem, kTmemCols);
    }
}

template <int NN, int CB, bool KEPT = false>
cudaError_t launch_one(const GemmMaps& maps, const DecodeGemmArgs& a, uint32_t units, uint32_t sms, cudaStream_t stream) {
    void (*const fn)(const GemmMaps, const DecodeGemmArgs) = decode_gemm_kernel<NN, CB, KEPT>;
    auto bytes = [](uint32_t n) { return KEPT ? smem_bytes(0, 3) + 3u * kKeptBytes : smem_bytes(n, row_slots(NN)); };
    static std::atomic<uint64_t> ready{0};  // devices (by ordinal) on which the kernel may use its shared memory
    const cudaError_t rc = allow_smem_once(ready, reinterpret_cast<const void*>(fn), bytes(NN > 0 ? NN : 128));
    if (rc != cudaSuccess) return rc;
    if (a.ksplit <= 1u) return launch_overlapped(fn, dim3(units < sms ? units : sms), kThreads, bytes(a.n), stream, a.overlap != 0, 1u, maps, a);
    return launch_overlapped(fn, dim3(a.ksplit, units), kThreads, bytes(a.n), stream, a.overlap != 0, a.ksplit, maps, a);
}

}  // namespace

#define T3_GEMM_NAME2(cb) launch_decode_gemm_cb##cb
#define T3_GEMM_NAME(cb) T3_GEMM_NAME2(cb)
cudaError_t T3_GEMM_NAME(T3_CB)(const GemmMaps& maps, const DecodeGemmArgs& a, uint32_t units, uint32_t sms, cudaStream_t stream) {
#if T3_CB == 0
    if (a.kept) return launch_one<0, 0, true>(maps, a, units, sms, stream);
#endif
    switch (a.n) {
#define T3_CASE(NN) \
    case NN: return launch_one<NN, T3_CB>(maps, a, units, sms, stream);
        T3_CASE(16) T3_CASE(32) T3_CASE(48) T3_CASE(64) T3_CASE(80) T3_CASE(96) T3_CASE(112) T3_CASE(128)
#undef T3_CASE
        default: return launch_one<0, T3_CB>(maps, a, units, sms, stream);
    }
}

}  // namespace t3
