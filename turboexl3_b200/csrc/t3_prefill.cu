// Prefill-row kernels (more than 32 activation rows): the trellis is decoded inside the weight loader of a tcgen05 GEMM.
//
//   route   : counting sort of the row-slots by expert + a table of row tiles (the reference's route:
//             src/core/kernels/prefill/froute_count.metal, table_2.metal; src/kernels/hip/prefill/prefill.hip:22-71)
//   prep    : input rotation of every sorted row, f16, natural order (format.prepareInput, src/core/format.zig:334-345)
//   gemm    : z = f16(xp W_hat) and the output rotation (t3_gemm.cu; the reference's GEMM with the decode in the loader:
//             src/core/kernels/prefill/gemm_4.metal, src/kernels/hip/prefill/prefill.hip:125-216, on Apple / gfx11 matrix units)
//   mid     : gate and up finish, SwiGLU, the down projection's prepare (src/kernels/hip/routed.hpp:64-112)
//   fin     : per row, every slot's down finish and the score-weighted sum in slot order
//             (src/kernels/hip/prefill/prefill.hip:243-264); a dense linear's finish runs in its GEMM's epilogue.
// Every wait is bounded: a wait that runs out sets a bit of the device error word and the kernel walks to its exit,
// freeing its tensor memory on the way.
#include "t3_common.cuh"
#include "t3_gemm.h"
#include "t3_internal.h"

namespace t3 {
namespace {

// ---- route ---------------------------------------------------------------------------------------------------------

__global__ void route_count_kernel(const uint32_t* inds, uint32_t slots, uint32_t experts, uint32_t* counts) {
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < slots) atomicAdd(&counts[min(inds[s], experts - 1u)], 1u);
}

// How an expert's c rows are cut into tiles: as few as hold them (a tile decodes its expert's weights once whatever its rows,
// and the decode is most of what a routed GEMM costs), of equal height in multiples of 16.
__device__ __forceinline__ uint32_t tile_height(uint32_t c) {
    const uint32_t cuts = (c + kGemmTileRows - 1u) / kGemmTileRows;
    return cuts ? ((c + cuts - 1u) / cuts + 15u) & ~15u : 16u;
}

// the most tiles any routing of `slots` row-slots gives
size_t routed_tiles_max(size_t slots, uint32_t experts) {
    const size_t cut = slots / kGemmTileRows + experts;
    return cut < slots ? cut : slots;
}

// one CTA: each expert's first sorted position (exclusive scan of the counts) into `cursor`, the tiles (expert, first
// position, rows, 0) in expert order and their number
__global__ void __launch_bounds__(1024) route_plan_kernel(const uint32_t* counts, uint32_t experts, uint32_t* cursor, int4* tiles,
                                                          uint32_t* n_tiles) {
    __shared__ uint32_t s_scan[2][1024];
    __shared__ uint32_t base[2];
    const uint32_t tid = threadIdx.x;
    if (tid < 2u) base[tid] = 0;
    __syncthreads();
    // experts are walked in chunks of 1024 with running bases
    for (uint32_t e0 = 0; e0 < experts; e0 += 1024u) {
        const uint32_t e = e0 + tid;
        const uint32_t c = e < experts ? counts[e] : 0u, h = tile_height(c), cuts = (c + h - 1u) / h;
        s_scan[0][tid] = c, s_scan[1][tid] = cuts;
        __syncthreads();
        for (uint32_t off = 1; off < 1024u; off <<= 1) {  // inclusive Hillis-Steele scans
            const uint32_t add0 = tid >= off ? s_scan[0][tid - off] : 0u, add1 = tid >= off ? s_scan[1][tid - off] : 0u;
            __syncthreads();
            s_scan[0][tid] += add0, s_scan[1][tid] += add1;
            __syncthreads();
        }
        if (e < experts) {
            const uint32_t first = base[0] + s_scan[0][tid] - c, at = base[1] + s_scan[1][tid] - cuts;
            cursor[e] = first;
            for (uint32_t i = 0; i < cuts; ++i) {
                const uint32_t lo = i * h, r = c - lo < h ? c - lo : h;
                tiles[at + i] = make_int4((int)e, (int)(first + lo), (int)r, 0);
            }
        }
        __syncthreads();
        if (tid < 2u) base[tid] += s_scan[tid][1023];
        __syncthreads();
    }
    if (tid == 0) *n_tiles = base[1];
}

__global__ void route_scatter_kernel(const uint32_t* inds, uint32_t slots, uint32_t experts, uint32_t* cursor,
                                     uint32_t* order, uint32_t* inv) {
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= slots) return;
    const uint32_t p = atomicAdd(&cursor[min(inds[s], experts - 1u)], 1u);
    order[p] = s;
    inv[s] = p;
}

// ---- prepare / mid / finish ------------------------------------------------------------------------------------------

constexpr uint32_t kRowsPerCta = 64;  // 8 warps x 8 positions

// how many CTAs share a position group's 128-blocks, so that small calls still fill the GPU
uint32_t spread(uint32_t positions, uint32_t nblk) {
    const uint32_t groups = (positions + kRowsPerCta - 1u) / kRowsPerCta;
    const uint32_t want = (1184u + groups - 1u) / groups;
    return want < 1u ? 1u : (want > nblk ? nblk : want);
}

// this lane's position in a warp's group of eight; returns false when the whole warp is past the end
__device__ __forceinline__ bool my_position(uint32_t count, uint32_t lane, uint32_t& p, bool& live) {
    const uint32_t first = (blockIdx.y * 8u + (threadIdx.x >> 5)) * 8u;
    if (first >= count) return false;
    const uint32_t mine = first + (lane >> 2);
    live = mine < count;
    p = live ? mine : count - 1u;
    return true;
}

// grid (spread, ceil(P / 64)), 256 threads. Dense: position = row, suh shared. Routed: position p -> slot order[p] -> row
// slot / topk, suh of the slot's expert; the second op (up) reuses the row with its own suh.
struct PrepArgs {
    const void* x;
    int x_dt;
    const __half* suh[2];
    uint32_t K, positions, topk, experts, ops;
    const uint32_t *order, *inds;  // null for a dense linear
    const uint32_t* row_map;       // routed: the x row of each row-slot when the call gathers rows, else slot / topk
    __half* xp;                    // [ops][positions][K]
};
__global__ void __launch_bounds__(256, 3) prep_rows_kernel(const PrepArgs a) {
    const uint32_t lane = threadIdx.x & 31u, q = lane & 3u;
    uint32_t p;
    bool live;
    if (!my_position(a.positions, lane, p, live)) return;
    uint32_t row = p, e = 0;
    if (a.order) {
        const uint32_t slot = a.order[p];
        row = a.row_map ? a.row_map[slot] : slot / a.topk;
        e = min(a.inds[slot], a.experts - 1u);
    }
    const HadB hb = had_b(lane);
    for (uint32_t blk = blockIdx.x; blk < (a.K >> 7); blk += gridDim.x) {
        const uint32_t col = blk * 128u + 4u * q;
        float xv[8][4];
#pragma unroll
        for (int i = 0; i < 8; ++i) load_act4(a.x, a.x_dt, (size_t)row * a.K + col + 16u * i, xv[i]);
        for (uint32_t op = 0; op < a.ops; ++op) {
            const __half* suh = (op ? a.suh[1] : a.suh[0]) + (size_t)e * a.K + col;
            float v[8][4], out[8][4];
            bool unit = true;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                float sc[4];
                load_half4(suh + 16 * i, sc);
                unit = unit && all_unit(sc);
#pragma unroll
                for (int j = 0; j < 4; ++j) v[i][j] = round_half(xv[i][j]) * sc[j];
            }
            h128_split(v, __all_sync(0xFFFFFFFFu, unit) != 0, hb, out);
            if (live) {
                const size_t o = ((size_t)op * a.positions + p) * a.K + col;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) out[i][j] *= kHadScale;
                    store_act4(a.xp, kF16, o + 16u * i, out[i]);
                }
            }
        }
    }
}

__device__ __forceinline__ float swiglu_f32(float g, float u, float limit, int clamp_at) {
    if (limit > 0.0f) {
        u = u > limit ? limit : (u < -limit ? -limit : u);
        if (clamp_at == 0) g = g > limit ? limit : g;
    }
    float s = g / (1.0f + expf(-g));
    if (limit > 0.0f && clamp_at != 0) s = s > limit ? limit : s;
    return s * u;
}

// grid (spread, ceil(P / 64)): SwiGLU of the finished gate and up values (the GEMM's epilogue finished them) and the
// down projection's prepare, per sorted position
struct MidArgs {
    const __half* z;  // [2][P][inter]: finished gate, finished up
    const __half* down_suh;
    const uint32_t *order, *inds;
    uint32_t positions, inter, experts;
    float limit;
    int clamp_at;
    __half* hd;  // [P][inter]
};
__global__ void __launch_bounds__(256, 3) mid_kernel(const MidArgs a) {
    const uint32_t lane = threadIdx.x & 31u, q = lane & 3u;
    uint32_t p;
    bool live;
    if (!my_position(a.positions, lane, p, live)) return;
    const uint32_t e = min(a.inds[a.order[p]], a.experts - 1u);
    const HadB hb = had_b(lane);
    for (uint32_t blk = blockIdx.x; blk < (a.inter >> 7); blk += gridDim.x) {
        const size_t eo = (size_t)e * a.inter + blk * 128u + 4u * q, zo = (size_t)p * a.inter + blk * 128u + 4u * q;
        float g[8][4], u[8][4];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            load_half4(a.z + zo + 16 * i, g[i]);
            load_half4(a.z + (size_t)a.positions * a.inter + zo + 16 * i, u[i]);
        }
        bool unit = true;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            float sd[4];
            load_half4(a.down_suh + eo + 16 * i, sd);
            unit = unit && all_unit(sd);
#pragma unroll
            for (int j = 0; j < 4; ++j) g[i][j] = round_half(swiglu_f32(g[i][j], u[i][j], a.limit, a.clamp_at)) * sd[j];
        }
        h128_split(g, __all_sync(0xFFFFFFFFu, unit) != 0, hb, u);
        if (live)
#pragma unroll
            for (int i = 0; i < 8; ++i) {
#pragma unroll
                for (int j = 0; j < 4; ++j) u[i][j] *= kHadScale;
                store_act4(a.hd, kF16, zo + 16u * i, u[i]);
            }
    }
}

// grid (spread, ceil(rows / 64)): per row, the score-weighted sum of its slots' finished down outputs (through inv) in
// slot order, then the optional shared-expert add in the output dtype
struct FinArgs {
    const __half* zd;  // [P][hidden]: each sorted position's finished down output (the per-slot v)
    const uint32_t* inv;
    const void* scores;
    int score_dt;
    const void* shared;
    void* y;
    int y_dt;
    uint32_t rows, hidden, topk;
};
__global__ void __launch_bounds__(256) moe_fin_kernel(const FinArgs a) {
    // a warp a row, a lane four consecutive elements of a 128-block: every slot's 256 bytes are one coalesced read
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t row = blockIdx.y * 8u + warp;
    if (row >= a.rows) return;
    for (uint32_t blk = blockIdx.x; blk < (a.hidden >> 7); blk += gridDim.x) {
        const uint32_t col = blk * 128u + 4u * lane;
        float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        for (uint32_t k0 = 0; k0 < a.topk; k0 += 4u) {  // four slots' loads in flight, the sum still in slot order
            float w[4], v[4][4];
#pragma unroll
            for (uint32_t i = 0; i < 4u; ++i) {
                const uint32_t k = k0 + i < a.topk ? k0 + i : a.topk - 1u;
                const size_t slot = (size_t)row * a.topk + k;
                w[i] = load_act(a.scores, a.score_dt, slot);
                load_half4(a.zd + (size_t)a.inv[slot] * a.hidden + col, v[i]);
            }
#pragma unroll
            for (uint32_t i = 0; i < 4u; ++i)
                if (k0 + i < a.topk)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[j] = __fadd_rn(acc[j], __fmul_rn(w[i], v[i][j]));
        }
        const size_t o = (size_t)row * a.hidden + col;
        if (a.shared) {
            float t[4], sh[4];
            store_act4(a.y, a.y_dt, o, acc);  // the routed output's rounding point
            load_act4(a.y, a.y_dt, o, t);
            load_act4(a.shared, a.y_dt, o, sh);
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[j] = __fadd_rn(t[j], sh[j]);
        }
        store_act4(a.y, a.y_dt, o, acc);
    }
}

// ---- host side -----------------------------------------------------------------------------------------------------

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled() {
    static EncodeTiledFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            p = nullptr;
        return reinterpret_cast<EncodeTiledFn>(p);
    }();
    return fn;
}

// 16-bit [rows, K] row-major, boxes of 64 x bm, 128-byte swizzle, rows past the end read as zero
bool make_a_map(CUtensorMap* map, const void* base, uint64_t rows, uint64_t K, uint32_t bm) {
    EncodeTiledFn fn = encode_tiled();
    if (!fn) return false;
    const cuuint64_t dims[2] = {K, rows};
    const cuuint64_t strides[1] = {K * 2u};
    const cuuint32_t box[2] = {64, bm};
    const cuuint32_t estr[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool make_row_maps(GemmMaps* maps, const void* rows_base, uint64_t rows, uint32_t K) {
    for (int i = 0; i < 4; ++i)
        if (!make_a_map(&maps->rows[i], rows_base, rows, K, 256u >> i)) return false;
    return true;
}

// the decode GEMM's maps: the prepared rows [rows, K] and the codes of one weight (experts 1) or bank, for up to two ops
bool make_gemm_maps(GemmMaps* maps, const void* rows_base, uint64_t rows, uint32_t K, const void* op0, const void* op1, uint32_t N,
                    uint32_t n, uint32_t experts) {
    EncodeTiledFn fn = encode_tiled();
    if (!fn || !make_row_maps(maps, rows_base, rows, K)) return false;
    const cuuint64_t dims[3] = {(cuuint64_t)N * n / 64u, K / 16u, experts};
    const cuuint64_t strides[2] = {dims[0] * 8u, dims[0] * 8u * dims[1]};
    const cuuint32_t box[3] = {2u * n, 4, 1}, estr[3] = {1, 1, 1};
    for (int op = 0; op < (op1 ? 2 : 1); ++op)
        if (fn(&maps->codes[op], CU_TENSOR_MAP_DATA_TYPE_INT64, 3, const_cast<void*>(op ? op1 : op0), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return false;
    return true;
}

size_t up256(size_t v) { return (v + 255u) & ~(size_t)255u; }

// multiprocessors of the device (a decode GEMM CTA fits each)
uint32_t one_wave_ctas() {
    static int sms = [] {
        int dev = 0, n = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
            n = 148;
        return n;
    }();
    return (uint32_t)sms;
}

}  // namespace

cudaError_t launch_decode_gemm_cb0(const GemmMaps&, const DecodeGemmArgs&, uint32_t units, uint32_t sms, cudaStream_t);
cudaError_t launch_decode_gemm_cb1(const GemmMaps&, const DecodeGemmArgs&, uint32_t units, uint32_t sms, cudaStream_t);
cudaError_t launch_decode_gemm(const GemmMaps& maps, const DecodeGemmArgs& a, uint32_t max_units, int codebook, cudaStream_t stream) {
    const uint32_t sms = one_wave_ctas();
    return codebook == kMcg ? launch_decode_gemm_cb1(maps, a, max_units, sms, stream) : launch_decode_gemm_cb0(maps, a, max_units, sms, stream);
}

// ---- dense linear, more than 32 rows ---------------------------------------------------------------------------------

// K slices of a dense linear of few rows: a call of up to 512 rows is one or two tiles of rows, out / 128 CTAs each, every one
// decoding all of its 128 columns' weights (a 6144 -> 2048 linear would run on 16 CTAs). Such calls cut K into slices, a CTA a
// slice, that meet in global memory (see DecodeGemmArgs::ksplit). Two arms, 33..256 rows and 257..512, each with a slice count
// that follows the geometry alone, so a row's bytes do not depend on the call's row count within an arm. The count: what fills two CTAs a multiprocessor at the arm's most
// tiles, eight at most (the tile's last arriver reads every slice), four K stages a slice at least — eight where K is short
// (under 64 stages), and there only while every CTA has a multiprocessor to itself and only in the first arm: with short K
// the slab's traffic and two CTAs sharing a multiprocessor cost what the slices save (measured: 2048 -> 6144 at 256 rows
// 35 us in three slices against 29, 2048 -> 2048 at 512 rows 32 us in four against 28).
uint32_t prefill_ksplit(size_t rows, uint32_t in, uint32_t out) {
    if (rows > 512u) return 1u;
    const uint32_t ncol = out / 128u, ksteps = in / 64u, sms = one_wave_ctas();
    const bool long_k = ksteps >= 64u;
    const uint32_t mtiles = rows <= 256u ? 2u : 4u;
    if (mtiles == 4u && !long_k) return 1u;
    uint32_t s = (2u * sms) / (mtiles * ncol);
    s = s < 8u ? s : 8u;
    const uint32_t by_k = long_k ? ksteps / 4u : ksteps / 8u;
    s = s < by_k ? s : by_k;
    if (s < 2u) return 1u;
    if (!long_k && mtiles * ncol * s > sms) return 1u;
    return s;
}

// the prepared rows (the GEMM's epilogue finishes into y, so the inner products of an unsliced call never reach memory);
// for a sliced call the slices' partial sums and the tiles' arrival counters as well
size_t prefill_linear_workspace(size_t rows, uint32_t in, uint32_t out) {
    size_t bytes = up256(rows * in * 2u);
    const uint32_t s = prefill_ksplit(rows, in, out);
    if (s > 1u) {
        const size_t mtiles = (rows + 127u) / 128u, ncol = out / 128u;
        bytes += up256(mtiles * ncol * s * 128u * 128u * 4u) + up256(mtiles * ncol * 4u);
    }
    return bytes;
}

// Rows a tile of the dense decode GEMM holds: of the ways to cut the rows into equal tiles, the one whose rounds of tiles over
// the multiprocessors take the least time. A tile's time, in cycles: per 64 inputs the decode of a 64 x 128 block (about 480
// at the issue rate the decode warps reach) or its MMAs (2 a row), whichever is more, then the epilogue.
uint32_t dense_tile_rows(uint32_t rows, uint32_t in, uint32_t ncol) {
    const uint32_t sms = one_wave_ctas(), fewest = (rows + kGemmTileRows - 1u) / kGemmTileRows;
    uint32_t best_h = kGemmTileRows;
    uint64_t best = ~0ull;
    for (uint32_t cuts = fewest; cuts <= 2u * fewest + 1u; ++cuts) {
        const uint32_t h = ((rows + cuts - 1u) / cuts + 15u) & ~15u, tiles = (rows + h - 1u) / h;
        const uint32_t step = 2u * h > 480u ? 2u * h : 480u;
        const uint64_t cost = (((uint64_t)tiles * ncol + sms - 1u) / sms) * ((in / 64u) * step + 1500u + 10u * h);
        if (cost < best) best = cost, best_h = h;
    }
    return best_h;
}

cudaError_t launch_prefill_linear(const PrefillLinearArgs& p, int codebook, cudaStream_t stream, int* launches) {
    uint8_t* ws = static_cast<uint8_t*>(p.workspace);
    __half* xp = reinterpret_cast<__half*>(ws);
    PrepArgs pa = {};
    pa.x = p.x;
    pa.x_dt = p.x_dt;
    pa.suh[0] = pa.suh[1] = static_cast<const __half*>(p.suh);
    pa.K = p.in;
    pa.positions = p.rows;
    pa.topk = 1;
    pa.experts = 1;
    pa.xp = xp;
    pa.ops = 1;
    prep_rows_kernel<<<dim3(spread(p.rows, p.in / 128u), (p.rows + kRowsPerCta - 1u) / kRowsPerCta), 256, 0, stream>>>(pa);
    const uint32_t ncol = p.out / 128u, ksplit = prefill_ksplit(p.rows, p.in, p.out);
    GemmMaps maps;
    const bool mapped = p.resident ? make_row_maps(&maps, xp, p.rows, p.in) && make_a_map(&maps.codes[0], p.resident, p.out, p.in, 128u)
                                   : make_gemm_maps(&maps, xp, p.rows, p.in, p.trellis, nullptr, p.out, p.n, 1);
    if (!mapped) return cudaErrorNotSupported;
    DecodeGemmArgs d = {};
    d.K = p.in;
    d.N = p.out;
    d.n = p.n;
    d.mask = p.mask;
    d.ops = 1;
    d.dense_rows = p.rows;
    d.tile_rows = dense_tile_rows(p.rows, p.in, ncol * ksplit);
    d.dense_tiles = (p.rows + d.tile_rows - 1u) / d.tile_rows;
    d.pair = 1;
    d.svh[0] = d.svh[1] = static_cast<const __half*>(p.svh);
    d.y = p.y;
    d.y_dt = p.x_dt;
    d.ksplit = ksplit;
    d.part = reinterpret_cast<float*>(ws + up256((size_t)p.rows * p.in * 2u));  // a sliced call's slab, behind the prepared rows
    d.kept = p.resident != nullptr;
    d.err = p.err;
    const cudaError_t rc = launch_decode_gemm(maps, d, d.dense_tiles * ncol, codebook, stream);
    if (rc == cudaSuccess) *launches += 2;  // the output rotation runs in the GEMM's epilogue
    return rc;
}

// ---- the un-rotated trunk, more than 32 rows ----------------------------------------------------------------------------

// One launch: both operands by TMA as they lie in memory (x [rows, in] and W_std transposed [out, in], the same 16-bit
// dtype), the epilogue rounds the f32 accumulators once into y (dense.residentPlain, src/core/dense.zig:1261-1263: "one
// matmul of x against its resident W_std in x's dtype").
cudaError_t launch_plain_linear(const void* x, int dt, uint32_t rows, const void* w_std_t, uint32_t in, uint32_t out, void* y,
                                uint32_t* err, cudaStream_t stream) {
    GemmMaps maps;
    if (!make_row_maps(&maps, x, rows, in) || !make_a_map(&maps.codes[0], w_std_t, out, in, 128u)) return cudaErrorNotSupported;
    DecodeGemmArgs d = {};
    d.K = in;
    d.N = out;
    d.ops = 1;
    d.dense_rows = rows;
    d.tile_rows = dense_tile_rows(rows, in, out / 128u);
    d.dense_tiles = (rows + d.tile_rows - 1u) / d.tile_rows;
    d.pair = 1;
    d.y = y;
    d.y_dt = dt;
    d.kept = 1;
    d.bf16 = dt == (int)kBf16;
    d.err = err;
    return launch_decode_gemm(maps, d, d.dense_tiles * (out / 128u), kMul1, stream);
}

// ---- routed experts, more than 32 rows --------------------------------------------------------------------------------

namespace {
struct MoeWs {
    uint32_t *counts, *cursor, *order, *inv;
    int4* tiles;
    uint32_t* n_tiles;
    __half *xp, *zgu, *hd, *zd;
    size_t total;
};
MoeWs carve_moe(uint8_t* base, size_t slots, uint32_t experts, uint32_t hidden, uint32_t inter) {
    MoeWs w;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        uint8_t* p = base ? base + off : nullptr;
        off += up256(bytes);
        return p;
    };
    w.counts = reinterpret_cast<uint32_t*>(take((size_t)experts * 4u));
    w.cursor = reinterpret_cast<uint32_t*>(take((size_t)experts * 4u));
    w.order = reinterpret_cast<uint32_t*>(take(slots * 4u));
    w.inv = reinterpret_cast<uint32_t*>(take(slots * 4u));
    w.tiles = reinterpret_cast<int4*>(take(routed_tiles_max(slots, experts) * 16u));
    w.n_tiles = reinterpret_cast<uint32_t*>(take(4u));
    w.xp = reinterpret_cast<__half*>(take(2u * slots * hidden * 2u));
    w.zgu = reinterpret_cast<__half*>(take(2u * slots * inter * 2u));
    w.hd = reinterpret_cast<__half*>(take(slots * inter * 2u));
    w.zd = reinterpret_cast<__half*>(take(slots * hidden * 2u));
    w.total = off;
    return w;
}

}  // namespace

size_t prefill_moe_workspace(size_t rows, uint32_t topk, uint32_t experts, uint32_t hidden, uint32_t inter) {
    return carve_moe(nullptr, rows * topk, experts, hidden, inter).total;
}

cudaError_t launch_prefill_moe(const MoeArgs& a, void* workspace, int codebook, cudaStream_t stream, int* launches) {
    const size_t slots = (size_t)a.rows * a.topk;
    const uint32_t S = (uint32_t)slots, H = a.hidden, I = a.inter;
    MoeWs w = carve_moe(static_cast<uint8_t*>(workspace), slots, a.experts, H, I);
    const uint32_t* inds = static_cast<const uint32_t*>(a.inds);
    cudaError_t rc = cudaMemsetAsync(w.counts, 0, (size_t)a.experts * 4u, stream);
    if (rc != cudaSuccess) return rc;
    route_count_kernel<<<(S + 255u) / 256u, 256, 0, stream>>>(inds, S, a.experts, w.counts);
    route_plan_kernel<<<1, 1024, 0, stream>>>(w.counts, a.experts, w.cursor, w.tiles, w.n_tiles);
    route_scatter_kernel<<<(S + 255u) / 256u, 256, 0, stream>>>(inds, S, a.experts, w.cursor, w.order, w.inv);

    PrepArgs pa = {};
    pa.x = a.x;
    pa.x_dt = a.x_dt;
    pa.suh[0] = static_cast<const __half*>(a.gate_suh);
    pa.suh[1] = static_cast<const __half*>(a.up_suh);
    pa.K = H;
    pa.positions = S;
    pa.topk = a.topk;
    pa.experts = a.experts;
    pa.order = w.order;
    pa.inds = inds;
    pa.row_map = a.row_map;
    pa.xp = w.xp;
    pa.ops = 2;
    prep_rows_kernel<<<dim3(spread(S, H / 128u), (S + kRowsPerCta - 1u) / kRowsPerCta), 256, 0, stream>>>(pa);

    // two 128-output blocks a unit of work: a tile of up to 128 rows runs both on one copy of its rows
    const size_t max_tiles = routed_tiles_max(slots, a.experts);
    auto units = [&](uint32_t outs, uint32_t ops) {
        const size_t u = max_tiles * ops * ((outs / 128u + 1u) / 2u);
        return (uint32_t)(u < (1u << 20) ? u : 1u << 20);
    };
    GemmMaps maps;
    if (!make_gemm_maps(&maps, w.xp, 2u * slots, H, a.gate_t, a.up_t, I, a.n, a.experts)) return cudaErrorNotSupported;
    DecodeGemmArgs g = {};
    g.K = H;
    g.N = I;
    g.n = a.n;
    g.mask = a.mask;
    g.ops = 2;
    g.op_rows = S;
    g.tiles = w.tiles;
    g.n_tiles = w.n_tiles;
    g.pair = 2;
    g.z = w.zgu;
    g.z_op_stride = slots * I;
    g.svh[0] = static_cast<const __half*>(a.gate_svh);  // the epilogue finishes gate and up with the tile's expert's scales
    g.svh[1] = static_cast<const __half*>(a.up_svh);
    g.svh_stride = I;
    g.err = a.err;
    rc = launch_decode_gemm(maps, g, units(I, 2u), codebook, stream);
    if (rc != cudaSuccess) return rc;

    MidArgs m = {w.zgu, static_cast<const __half*>(a.down_suh), w.order, inds, S, I, a.experts, a.limit, a.clamp_at, w.hd};
    mid_kernel<<<dim3(spread(S, I / 128u), (S + kRowsPerCta - 1u) / kRowsPerCta), 256, 0, stream>>>(m);

    if (!make_gemm_maps(&maps, w.hd, slots, I, a.down_t, nullptr, H, a.n, a.experts)) return cudaErrorNotSupported;
    DecodeGemmArgs d = g;
    d.K = I;
    d.N = H;
    d.ops = 1;
    d.z = w.zd;
    d.z_op_stride = 0;
    d.svh[0] = d.svh[1] = static_cast<const __half*>(a.down_svh);  // each slot's finished down output, the per-slot v
    d.svh_stride = H;
    rc = launch_decode_gemm(maps, d, units(H, 1u), codebook, stream);
    if (rc != cudaSuccess) return rc;

    FinArgs f = {w.zd, w.inv, a.scores, a.score_dt, a.shared, a.y, a.y_dt, a.rows, H, a.topk};
    if (a.shared_ready) {  // only this launch reads `shared`
        rc = cudaStreamWaitEvent(stream, static_cast<cudaEvent_t>(a.shared_ready), 0);
        if (rc != cudaSuccess) return rc;
    }
    const uint32_t fin_groups = (a.rows + 7u) / 8u, fin_want = (1184u + fin_groups - 1u) / fin_groups;
    moe_fin_kernel<<<dim3(fin_want < H / 128u ? fin_want : H / 128u, fin_groups), 256, 0, stream>>>(f);
    *launches += 8;
    return cudaGetLastError();
}

}  // namespace t3
