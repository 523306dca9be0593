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
#include "t3_slot.cuh"

namespace t3 {
namespace {

// ---- route ---------------------------------------------------------------------------------------------------------

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

// Where the router's expert ids lie: one bank (bank_of null: the id is the expert), or several banks of one geometry at rates
// of their own (layer expert g is expert local_of[g] of bank bank_of[g]). Experts are numbered bank by bank: bank b's from
// base[b] on. The ids and both arrays are the caller's: each is clamped into its range, since a number indexes the counters here
// and the bank's arrays later.
struct ExpertMap {
    const int64_t *bank_of, *local_of;
    uint32_t base[kMixedBanksMax + 1];
    uint32_t banks, ids;  // banks (none empty); router ids
    static __device__ uint32_t clamped(int64_t v, uint32_t count) { return (uint32_t)min(max(v, (int64_t)0), (int64_t)count - 1); }
    __device__ uint32_t number(uint32_t id) const {
        id = min(id, ids - 1u);
        if (!bank_of) return id;
        const uint32_t b = clamped(bank_of[id], banks);
        return base[b] + clamped(local_of[id], base[b + 1u] - base[b]);
    }
    // the bank of an expert number, and the number inside it
    __device__ uint32_t bank(uint32_t e) const {
        uint32_t b = 0;
        while (b + 1u < banks && e >= base[b + 1u]) ++b;
        return b;
    }
};

// One launch counts the row-slots of every expert and remembers each slot's rank among its expert's (a block counts in shared
// memory and reserves its ranks with one atomic an expert); the last block to finish lays out the experts: first[e] the
// expert's first sorted position, tiles (expert inside its bank, first position, rows, 0) in expert order, range[b] .. range[b +
// 1] bank b's tiles. counts and `ticket` are zero before the launch. (Counting, laying out and a second pass of atomics to
// scatter were three launches and 20 us.) A call of one block (`whole`: `where` and `inv` are given) keeps its counts in shared memory and
// scatters its slots itself: no clearing and no second launch, 33 rows of 512 experts of 2048 x 512 237.5 -> 231.3 us.
struct Scatter {
    const uint32_t* row_map;
    uint32_t topk;
    SlotId ids;
    uint2* where;
    uint32_t* inv;
    // slot s of expert number e at sorted position p: the x row it reads, its bank and expert
    __device__ void put(const ExpertMap& map, uint32_t s, uint32_t e, uint32_t p) const {
        const uint32_t b = map.bank(e);
        where[p] = make_uint2(row_map ? row_map[s] : s / topk, ids.pack(b, e - map.base[b]));
        inv[s] = p;
    }
};
constexpr uint32_t kRouteThreads = 1024, kRouteSlots = 4096, kRouteExperts = 8192;
__global__ void __launch_bounds__(kRouteThreads) route_plan_kernel(const uint32_t* inds, uint32_t slots, const __grid_constant__ ExpertMap map,
                                                                   uint32_t* counts, uint32_t* ticket, uint32_t* rank, uint32_t* first,
                                                                   int4* tiles, uint32_t* range, const Scatter whole) {
    extern __shared__ uint32_t hist[];  // one counter an expert, then its base in this block's ranks; empty past kRouteExperts
    __shared__ uint32_t s_sum[2][32], s_base[2], s_last;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, experts = map.base[map.banks];
    const bool shared_hist = experts <= kRouteExperts;
    const uint32_t lo = blockIdx.x * kRouteSlots;
    const bool single = whole.where != nullptr;
    pdl_wait();  // the routing may be the previous kernel's output, and the workspace its own
    pdl_trigger();
    uint32_t mine_e[kRouteSlots / kRouteThreads], mine_r[kRouteSlots / kRouteThreads];
    if (shared_hist) {
        for (uint32_t e = tid; e < experts; e += kRouteThreads) hist[e] = 0u;
        __syncthreads();
    }
#pragma unroll
    for (uint32_t i = 0; i < kRouteSlots / kRouteThreads; ++i) {
        const uint32_t s = lo + i * kRouteThreads + tid;
        if (s >= slots) break;
        mine_e[i] = map.number(inds[s]);
        mine_r[i] = atomicAdd(shared_hist ? &hist[mine_e[i]] : &counts[mine_e[i]], 1u);
    }
    if (tid < 2u) s_base[tid] = 0u;
    if (!single) {
        if (shared_hist) {
            __syncthreads();
            for (uint32_t e = tid; e < experts; e += kRouteThreads)
                if (hist[e]) hist[e] = atomicAdd(&counts[e], hist[e]);
            __syncthreads();
        }
#pragma unroll
        for (uint32_t i = 0; i < kRouteSlots / kRouteThreads; ++i) {
            const uint32_t s = lo + i * kRouteThreads + tid;
            if (s >= slots) break;
            rank[s] = mine_r[i] + (shared_hist ? hist[mine_e[i]] : 0u);
        }
        __threadfence();
        __syncthreads();
        if (tid == 0) s_last = atomicAdd(ticket, 1u) == gridDim.x - 1u;
        __syncthreads();
        if (!s_last) return;
        __threadfence();
    } else {
        __syncthreads();
    }
    for (uint32_t e0 = 0; e0 < experts; e0 += kRouteThreads) {  // experts in runs of a thread each, with running bases
        const uint32_t e = e0 + tid, c = e < experts ? (single ? hist[e] : __ldcg(&counts[e])) : 0u, h = tile_height(c), cuts = (c + h - 1u) / h;
        uint32_t in0 = c, in1 = cuts;  // inclusive scans: inside a warp, then over the warps' sums
#pragma unroll
        for (uint32_t off = 1; off < 32u; off <<= 1) {
            const uint32_t a0 = __shfl_up_sync(0xFFFFFFFFu, in0, off), a1 = __shfl_up_sync(0xFFFFFFFFu, in1, off);
            if (lane >= off) in0 += a0, in1 += a1;
        }
        if (lane == 31u) s_sum[0][warp] = in0, s_sum[1][warp] = in1;
        __syncthreads();
        if (warp == 0) {
            uint32_t t0 = s_sum[0][lane], t1 = s_sum[1][lane];
#pragma unroll
            for (uint32_t off = 1; off < 32u; off <<= 1) {
                const uint32_t a0 = __shfl_up_sync(0xFFFFFFFFu, t0, off), a1 = __shfl_up_sync(0xFFFFFFFFu, t1, off);
                if (lane >= off) t0 += a0, t1 += a1;
            }
            s_sum[0][lane] = t0, s_sum[1][lane] = t1;
        }
        __syncthreads();
        const uint32_t pos = s_base[0] + in0 - c + (warp ? s_sum[0][warp - 1u] : 0u);
        const uint32_t at = s_base[1] + in1 - cuts + (warp ? s_sum[1][warp - 1u] : 0u);
        if (e < experts) {
            if (single) hist[e] = pos;
            else first[e] = pos;
            const uint32_t b = map.bank(e);
            for (uint32_t i = 0; i < cuts; ++i) {
                const uint32_t r0 = i * h, r = c - r0 < h ? c - r0 : h;
                tiles[at + i] = make_int4((int)(e - map.base[b]), (int)(pos + r0), (int)r, 0);
            }
            for (uint32_t k = 0; k < map.banks; ++k)
                if (map.base[k] == e) range[k] = at;
        }
        __syncthreads();
        if (tid < 2u) s_base[tid] += s_sum[tid][31];
        __syncthreads();
    }
    if (tid <= map.banks && map.base[tid] >= experts) range[tid] = s_base[1];
    if (!single) return;
#pragma unroll
    for (uint32_t i = 0; i < kRouteSlots / kRouteThreads; ++i) {  // (the loop above ended on a barrier: every expert's position is in place)
        const uint32_t s = i * kRouteThreads + tid;
        if (s >= slots) break;
        whole.put(map, s, mine_e[i], hist[mine_e[i]] + mine_r[i]);
    }
}

// every slot's sorted position (inv), and per position the x row it reads and its bank and expert (SlotId)
__global__ void route_scatter_kernel(const uint32_t* inds, uint32_t slots, const __grid_constant__ ExpertMap map, const uint32_t* rank,
                                     const uint32_t* first, const Scatter to) {
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    pdl_wait();
    pdl_trigger();
    if (s >= slots) return;
    const uint32_t e = map.number(inds[s]);
    to.put(map, s, e, first[e] + rank[s]);
}

// ---- prepare / mid / finish ------------------------------------------------------------------------------------------

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

// The prepares work on (position, 128-block) pairs, eight consecutive pairs a warp: a position's blocks lie side by side in
// memory, so a warp reads and writes runs of up to 2 KB (with eight positions' same block a warp, 256 bytes a row, the
// prepare of 65536 slots of 7168 x 2 wrote at 2.5 TB/s). A few CTAs a multiprocessor walk the pairs.
constexpr uint32_t kPairsPerCta = 64;  // 8 warps x 8 pairs
uint32_t pair_ctas(size_t positions, uint32_t nblk) {
    const size_t want = (positions * nblk + kPairsPerCta - 1u) / kPairsPerCta, most = (size_t)one_wave_ctas() * 12u;
    return (uint32_t)(want < most ? want : most);
}

// 256 threads. Dense and one-expert calls (where null): positions are the call's rows. Routed: position p reads row
// where[p].x with the scales of its expert (where[p].y); the second op (up) reuses the row with its own suh.
//
// RUNS: a quad keeps one 128-block and walks `chunk` consecutive positions: sorted positions share their expert in runs, so the block's
// scales are read once a run and kept as two words of signs. What bounds the kernel is L1: a 16-byte access of eight quads touches
// eight lines, and of 24 accesses for a pair of ops eight were scales and four the row read twice. 40960 slots of 2048 x 2: 95 us (87 %
// of L1's rate), 81 with the signs kept, 72 with the row kept in registers too (three CTAs a multiprocessor; with four it spilled). Scales
// that are not signs are read again for every position, which takes what it took without the runs: 114 us either way.
// Else (one op, calls of a round or two of warps) a quad takes one (position, block) and nothing stands between its loads of the row and of
// the scales. Linears, us, in the other form / this: 2048 -> 6144 at 520 rows 20.5 / 20.2, 3072 -> 3072 at 300 21.6 / 21.4, 6144 -> 2048 at
// 400 22.9 / 22.4. (With registers for four CTAs a multiprocessor 20.5, 20.8 and 22.9, but 2048 -> 6144 at 128 17.4 -> 17.8. Two ops, which
// would read the row twice, lose: 64 experts of 4096 x 1024 at 300 rows 233.0 / 234.2.)
struct PrepArgs {
    const void* x;
    int x_dt;
    const __half* suh[2][kMixedBanksMax];  // per op and bank, expert-major
    uint32_t K, positions, ops, chunk;
    const uint2* where;
    SlotId ids;               // how where[p].y is packed
    const uint32_t* row_map;  // where null: position p reads row row_map[p], or row p / topk
    uint32_t topk;
    __half* xp;  // [ops][positions][K]
};
template <bool RUNS>
__global__ void __launch_bounds__(256, 3) prep_rows_kernel(const __grid_constant__ PrepArgs a) {
    const uint32_t lane = threadIdx.x & 31u, q = lane & 3u, nblk = a.K >> 7;
    const uint32_t chunk = RUNS ? a.chunk : 1u, units = (a.positions + chunk - 1u) / chunk * nblk;  // (the callers keep positions x width under 2^31)
    pdl_wait();
    pdl_trigger();  // after the wait: the GEMM that follows reads the tiles ahead of its own
    const bool wide_x = aligned16(a.x);
    const HadB hb = had_b(lane);
    auto put = [&](const uint32_t (&w)[4][4], uint32_t op, uint32_t p, uint32_t col) {
        uint4* o = reinterpret_cast<uint4*>(a.xp + ((size_t)op * a.positions + p) * a.K + col);
#pragma unroll
        for (int s = 0; s < 4; ++s) o[4 * s] = make_uint4(w[s][0], w[s][1], w[s][2], w[s][3]);
    };
    for (uint32_t u0 = (blockIdx.x * 8u + (threadIdx.x >> 5)) * 8u; u0 < units; u0 += gridDim.x * kPairsPerCta) {
        const uint32_t u = min(u0 + (lane >> 2), units - 1u), c = u / nblk, col = (u - c * nblk) * 128u + 8u * q;
        const bool mine = u0 + (lane >> 2) < units;
        uint32_t held = 0, signs[2] = {0u, 0u};  // the expert whose signs are held
        bool fresh = a.chunk > 1u, plain = fresh;  // (with one position a quad there is nothing to keep)
#pragma unroll 1
        for (uint32_t i = 0; i < chunk; ++i) {
            const uint32_t at = c * chunk + i, p = min(at, a.positions - 1u);
            uint32_t row, id = 0;
            if (a.where) {
                const uint2 w = a.where[p];
                row = w.x, id = w.y;
            } else {
                row = a.row_map ? a.row_map[p] : p / a.topk;
            }
            const size_t scale_at = (size_t)a.ids.expert(id) * a.K + col;
            const uint32_t bank = a.ids.bank(id);
            if (!RUNS) {
                const __half* sp = a.suh[0][bank] + scale_at;
                uint32_t w[4][4];
#pragma unroll
                for (int s = 0; s < 4; ++s) load_half8(a.x, a.x_dt, wide_x, (size_t)row * a.K + col + 32u * s, w[s]);
                rotate_block(w, sp, aligned16(sp), hb);
                if (mine) put(w, 0u, p, col);
                continue;
            }
            if (a.chunk > 1u && __any_sync(0xFFFFFFFFu, fresh || id != held)) {
                uint32_t odd = 0;
                for (uint32_t op = 0; op < a.ops; ++op) {
                    const __half* sp = (op ? a.suh[1][bank] : a.suh[0][bank]) + scale_at;
                    const uint32_t m = sign_mask(sp, aligned16(sp), odd);
                    if (op) signs[1] = m;
                    else signs[0] = m;
                }
                plain = __any_sync(0xFFFFFFFFu, odd != 0u) == 0;
                held = id, fresh = false;
            }
            uint32_t x[4][4];
#pragma unroll
            for (int s = 0; s < 4; ++s) load_half8(a.x, a.x_dt, wide_x, (size_t)row * a.K + col + 32u * s, x[s]);
#pragma unroll 1
            for (uint32_t op = 0; op < a.ops; ++op) {
                uint32_t w[4][4];
#pragma unroll
                for (int s = 0; s < 4; ++s)
#pragma unroll
                    for (int p = 0; p < 4; ++p) w[s][p] = x[s][p];
                if (plain) {
                    apply_signs(w, op ? signs[1] : signs[0]);
                    rotate_signed(w, hb);
                } else {
                    const __half* sp = (op ? a.suh[1][bank] : a.suh[0][bank]) + scale_at;
                    rotate_block(w, sp, aligned16(sp), hb);
                }
                if (mine && at < a.positions) put(w, op, p, col);
            }
        }
    }
}
// The positions a quad walks: up to eight, while two rounds of warps are left
cudaError_t launch_prep(PrepArgs& pa, bool overlap, cudaStream_t stream) {
    const size_t pairs = (size_t)pa.positions * (pa.K / 128u), chunk = pairs / ((size_t)one_wave_ctas() * 32u * 8u * 2u);
    pa.chunk = (uint32_t)(chunk < 1u ? 1u : chunk > 8u ? 8u : chunk);
    return launch_overlapped(pa.chunk > 1u || pa.ops > 1u ? prep_rows_kernel<true> : prep_rows_kernel<false>, dim3(pair_ctas((pa.positions + pa.chunk - 1u) / pa.chunk, pa.K / 128u)), 256, 0, stream, overlap, 1, pa);
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

// SwiGLU of the finished gate and up values (the GEMM's epilogue finished them) and the
// down projection's prepare, per sorted position
struct MidArgs {
    const __half* z;  // [2][P][inter]: finished gate, finished up
    const __half* down_suh[kMixedBanksMax];
    const uint2* where;  // or null: one expert
    SlotId ids;
    uint32_t positions, inter;
    float limit;
    int clamp_at;
    __half* hd;  // [P][inter]
};
__global__ void __launch_bounds__(256, 4) mid_kernel(const __grid_constant__ MidArgs a) {
    const uint32_t lane = threadIdx.x & 31u, q = lane & 3u, nblk = a.inter >> 7;
    const uint32_t pairs = a.positions * nblk;
    pdl_wait();
    pdl_trigger();  // after the wait: the GEMM that follows reads the tiles ahead of its own
    const HadB hb = had_b(lane);
    for (uint32_t f0 = (blockIdx.x * 8u + (threadIdx.x >> 5)) * 8u; f0 < pairs; f0 += gridDim.x * kPairsPerCta) {
        const bool live = f0 + (lane >> 2) < pairs;
        const uint32_t f = live ? f0 + (lane >> 2) : pairs - 1u;
        const uint32_t p = f / nblk, col = (f - p * nblk) * 128u + 8u * q;
        const uint32_t id = a.where ? a.where[p].y : 0u;
        const __half* suh = a.down_suh[a.ids.bank(id)] + (size_t)a.ids.expert(id) * a.inter + col;
        const bool wide_s = aligned16(suh);
        const size_t zo = (size_t)p * a.inter + col;
        uint32_t g[4][4], u[4][4];
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            load_16b(a.z + zo + 32 * s, true, g[s]);
            load_16b(a.z + (size_t)a.positions * a.inter + zo + 32 * s, true, u[s]);
        }
#pragma unroll
        for (int s = 0; s < 4; ++s)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 gv = unpack_half2(g[s][j]), uv = unpack_half2(u[s][j]);
                g[s][j] = pack_half2(swiglu_f32(gv.x, uv.x, a.limit, a.clamp_at), swiglu_f32(gv.y, uv.y, a.limit, a.clamp_at));
            }
        rotate_block(g, suh, wide_s, hb);
        if (live) {
            uint4* o = reinterpret_cast<uint4*>(a.hd + zo);
#pragma unroll
            for (int s = 0; s < 4; ++s) o[4 * s] = make_uint4(g[s][0], g[s][1], g[s][2], g[s][3]);
        }
    }
}

// grid (column runs, ceil(rows / 8)): per row, the score-weighted sum of its slots' finished down outputs (through inv) in
// slot order, then the optional shared-expert add in the output dtype
struct FinArgs {
    const __half* zd;  // [P][hidden]: each sorted position's finished down output (the per-slot v)
    const uint32_t* inv;  // or null: slot s's is row s
    const void* scores;
    int score_dt;
    const void* shared;
    void* y;
    int y_dt;
    uint32_t rows, hidden, topk;
};
__global__ void __launch_bounds__(256) moe_fin_kernel(const FinArgs a) {
    // A warp a row, a lane eight consecutive elements of two 128-blocks: a slot's 512 bytes are one coalesced read, eight slots'
    // in flight at once (four 8-byte reads a lane left the kernel waiting on memory: 49 us where its bytes take 28). Lane k holds
    // slot k's weight and place for the whole row (top-k is 32 at most).
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t row = blockIdx.y * 8u + warp;
    pdl_wait();
    pdl_trigger();
    if (row >= a.rows) return;
    const size_t slot = (size_t)row * a.topk + min(lane, a.topk - 1u);
    const float my_w = load_act(a.scores, a.score_dt, slot);
    const uint32_t my_at = a.inv ? a.inv[slot] : (uint32_t)slot;
    for (uint32_t c0 = blockIdx.x * 256u; c0 < a.hidden; c0 += gridDim.x * 256u) {
        const uint32_t col = c0 + lane * 8u;
        const bool in = col < a.hidden;  // the last run may be one 128-block
        float acc[8] = {};
        for (uint32_t k0 = 0; k0 < a.topk; k0 += 8u) {
            uint4 v[8];
#pragma unroll
            for (uint32_t i = 0; i < 8u; ++i) {
                const uint32_t at = __shfl_sync(0xFFFFFFFFu, my_at, (k0 + i) & 31u);
                v[i] = make_uint4(0u, 0u, 0u, 0u);
                if (in && k0 + i < a.topk) v[i] = __ldcs(reinterpret_cast<const uint4*>(a.zd + (size_t)at * a.hidden + col));
            }
#pragma unroll
            for (uint32_t i = 0; i < 8u; ++i) {
                if (k0 + i >= a.topk) break;
                const float w = __shfl_sync(0xFFFFFFFFu, my_w, (k0 + i) & 31u);
                const uint32_t u[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 f = unpack_half2(u[j]);
                    acc[2 * j] = __fadd_rn(acc[2 * j], __fmul_rn(w, f.x));
                    acc[2 * j + 1] = __fadd_rn(acc[2 * j + 1], __fmul_rn(w, f.y));
                }
            }
        }
        if (!in) continue;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            float f[4] = {acc[4 * half], acc[4 * half + 1], acc[4 * half + 2], acc[4 * half + 3]};
            const size_t o = (size_t)row * a.hidden + col + 4u * half;
            if (a.shared) {
                float sh[4];
                load_act4(a.shared, a.y_dt, o, sh);
#pragma unroll
                for (int j = 0; j < 4; ++j) {  // the routed output's rounding point, then the add in f32
                    const float t = a.y_dt == kF32 ? f[j] : a.y_dt == kF16 ? round_half(f[j]) : __bfloat162float(__float2bfloat16_rn(f[j]));
                    f[j] = __fadd_rn(t, sh[j]);
                }
            }
            store_act4(a.y, a.y_dt, o, f);
        }
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

// the outputs' maps (see GemmMaps::out), 16-bit [rows, N]
bool make_out_maps(GemmMaps* maps, const void* base, uint64_t rows, uint32_t N) {
    for (int i = 0; i < 5; ++i)
        if (!make_a_map(&maps->out[i], base, rows, N, 128u >> i)) return false;
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

}  // namespace

cudaError_t launch_decode_gemm_cb0(const GemmMaps&, const DecodeGemmArgs&, uint32_t units, uint32_t sms, cudaStream_t);
cudaError_t launch_decode_gemm_cb1(const GemmMaps&, const DecodeGemmArgs&, uint32_t units, uint32_t sms, cudaStream_t);
cudaError_t launch_decode_gemm(const GemmMaps& maps, const DecodeGemmArgs& a, uint32_t max_units, int codebook, cudaStream_t stream) {
    const uint32_t sms = one_wave_ctas();
    return codebook == kMcg ? launch_decode_gemm_cb1(maps, a, max_units, sms, stream) : launch_decode_gemm_cb0(maps, a, max_units, sms, stream);
}

// ---- dense linear, more than 32 rows ---------------------------------------------------------------------------------

// Clusters of `s` decode GEMM CTAs (one a multiprocessor) that are resident at once. Of B200's 148 multiprocessors, by cluster size:
// what cudaOccupancyMaxActiveClusters gives for the kernel at every rate tried (n 16, 64, 128). Written down because a call's slice
// count, hence its bytes and its workspace, follows from it and must be the same without a device.
uint32_t resident_clusters(uint32_t s) {
    static const uint32_t resident[9] = {0, 148, 74, 45, 33, 26, 22, 15, 15};
    return resident[s] * one_wave_ctas() / 148u;
}

// K slices of a dense linear of few rows: a call of up to 512 rows is one or two tiles of rows, out / 128 CTAs each, every one
// decoding all of its 128 columns' weights (a 6144 -> 2048 linear would run on 16 CTAs). Such calls cut K into slices, a CTA a
// slice, that meet in global memory (see DecodeGemmArgs::ksplit). Two arms, 33..256 rows and 257..512, each with a slice count
// that follows the geometry alone, so a row's bytes do not depend on the call's row count within an arm. The count: the most
// (eight at most) whose clusters are all resident at once — a second wave doubles the call: 6144 -> 2048 at 200 rows took 33 us
// in eight slices, of which fifteen clusters fit and sixteen are needed, against 18 in six — four 64-input steps a slice at
// least, eight where K is short (under 64 steps), and there only in the first arm and while the slab's traffic is small.
uint32_t prefill_ksplit(size_t rows, uint32_t in, uint32_t out) {
    if (rows > 512u) return 1u;
    const uint32_t ncol = out / 128u, ksteps = in / 64u, sms = one_wave_ctas();
    const bool long_k = ksteps >= 64u;
    const uint32_t mtiles = rows <= 256u ? 2u : 4u, units = ncol * mtiles / 2u;
    if (mtiles == 4u && !long_k) return 1u;
    const uint32_t by_slab = (2u * sms) / (mtiles * ncol), by_k = long_k ? ksteps / 4u : ksteps / 8u;
    uint32_t s = 8;
    while (s > 1u && (s > by_slab || s > by_k || units > resident_clusters(s))) --s;
    if (s < 2u) return 1u;
    if (!long_k && mtiles * ncol * s > sms) return 1u;
    return s;
}

// the prepared rows (the GEMM's epilogue finishes into y, so the inner products of an unsliced call never reach memory); for a
// sliced call the slices' partial sums as well (sized in whole 128-row tiles and a word a tile, as callers of this size expect)
size_t prefill_linear_workspace(size_t rows, uint32_t in, uint32_t out) {
    size_t bytes = up256(rows * in * 2u);
    const uint32_t s = prefill_ksplit(rows, in, out);
    if (s > 1u) {
        const size_t mtiles = (rows + 127u) / 128u, ncol = out / 128u;
        bytes += up256(mtiles * ncol * s * 128u * 128u * 4u) + up256(mtiles * ncol * 4u);
    }
    return bytes;
}

// Rows a tile of the dense decode GEMM holds: of the ways to cut the rows into equal tiles, the one whose rounds of units (`units` a
// tile, `at_once` of them resident: a CTA each, or a cluster of a sliced call) take the least time. A unit's time, in cycles: per 64
// of its inputs the decode of a 64 x 128 block (about 480 at the issue rate the decode warps reach) or its MMAs (2 a row), whichever
// is more, then the epilogue. (A sliced call's CTAs counted one by one, as if they needed no cluster, cut 4096 -> 1024 in eight
// slices into two tiles, of whose sixteen clusters fifteen fit: 22.0 us at 200 rows, 20.4 at 100 and 27.7 at 512, against 14.9,
// 12.6 and 19.2 in one round.)
uint32_t dense_tile_rows(uint32_t rows, uint32_t inputs, uint32_t units, uint32_t at_once) {
    const uint32_t fewest = (rows + kGemmTileRows - 1u) / kGemmTileRows;
    uint32_t best_h = kGemmTileRows;
    uint64_t best = ~0ull;
    for (uint32_t cuts = fewest; cuts <= 2u * fewest + 1u; ++cuts) {
        const uint32_t h = ((rows + cuts - 1u) / cuts + 15u) & ~15u, tiles = (rows + h - 1u) / h;
        const uint32_t step = 2u * h > 480u ? 2u * h : 480u;
        const uint64_t cost = (((uint64_t)tiles * units + at_once - 1u) / at_once) * ((inputs / 64u) * step + 1500u + 10u * h);
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
    pa.suh[0][0] = pa.suh[1][0] = static_cast<const __half*>(p.suh);
    pa.K = p.in;
    pa.positions = p.rows;
    pa.topk = 1;
    pa.xp = xp;
    pa.ops = 1;
    cudaError_t rc = launch_prep(pa, p.overlap != 0, stream);
    if (rc != cudaSuccess) return rc;
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
    d.tile_rows = dense_tile_rows(p.rows, p.in / ksplit, ncol, resident_clusters(ksplit));
    d.dense_tiles = (p.rows + d.tile_rows - 1u) / d.tile_rows;
    d.pair = 1;
    d.svh[0] = d.svh[1] = static_cast<const __half*>(p.svh);
    d.y = p.y;
    d.y_dt = p.x_dt;
    d.ksplit = ksplit;
    d.part = reinterpret_cast<float*>(ws + up256((size_t)p.rows * p.in * 2u));  // a sliced call's slab, behind the prepared rows
    d.kept = p.resident != nullptr;
    d.bulk_out = ksplit == 1u && p.x_dt != (int)kF32 && aligned16(p.y);
    if (d.bulk_out && !make_out_maps(&maps, p.y, p.rows, p.out)) return cudaErrorNotSupported;
    d.err = p.err;
    // Overlapped, the GEMM's set-up and first codes run beside the prepare, which counts in a short call; in a long one the GEMM's
    // CTAs take the prepare's slots. Overlapped against not, 2048 -> 6144: 21.4 / 23.2 us at 520 rows, 51.5 / 52.8 at 2048, 71.1 / 71.3
    // at 3072, 99.1 / 98.3 at 4096; 2048 -> 2048 17.8 / 20.4 .. 24.7 / 26.3 at 2048, 41.9 / 43.4 at 4096; 4096 -> 4096 K2 level at
    // 2048, 1.5 % slower from 3072 on; 7168 -> 1536 and 6144 -> 2048 faster throughout (1-5 %).
    d.overlap = p.rows <= 2048u && p.overlap;
    rc = launch_decode_gemm(maps, d, d.dense_tiles * ncol, codebook, stream);
    if (rc == cudaSuccess) *launches += 2;  // the output rotation runs in the GEMM's epilogue
    return rc;
}

// ---- the un-rotated trunk, more than 32 rows ----------------------------------------------------------------------------

// One launch: both operands by TMA as they lie in memory (x [rows, in] and W_std transposed [out, in], the same 16-bit
// dtype), the epilogue rounds the f32 accumulators once into y (dense.residentPlain, src/core/dense.zig:1261-1263: "one
// matmul of x against its resident W_std in x's dtype").
cudaError_t launch_plain_linear(const void* x, int dt, uint32_t rows, const void* w_std_t, uint32_t in, uint32_t out, void* y,
                                uint32_t* err, bool overlap, cudaStream_t stream) {
    GemmMaps maps;
    if (!make_row_maps(&maps, x, rows, in) || !make_a_map(&maps.codes[0], w_std_t, out, in, 128u)) return cudaErrorNotSupported;
    DecodeGemmArgs d = {};
    d.K = in;
    d.N = out;
    d.ops = 1;
    d.dense_rows = rows;
    d.tile_rows = dense_tile_rows(rows, in, out / 128u, one_wave_ctas());
    d.dense_tiles = (rows + d.tile_rows - 1u) / d.tile_rows;
    d.pair = 1;
    d.y = y;
    d.y_dt = dt;
    d.kept = 1;
    d.bf16 = dt == (int)kBf16;
    d.err = err;
    d.overlap = overlap;
    return launch_decode_gemm(maps, d, d.dense_tiles * (out / 128u), kMul1, stream);
}

// ---- routed experts, more than 32 rows --------------------------------------------------------------------------------

namespace {
struct MoeWs {
    uint32_t *counts, *first, *rank, *inv, *range;
    uint2* where;
    int4* tiles;
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
    w.counts = reinterpret_cast<uint32_t*>(take(((size_t)experts + 1u) * 4u));  // and the ticket
    w.first = reinterpret_cast<uint32_t*>(take((size_t)experts * 4u));
    w.rank = reinterpret_cast<uint32_t*>(take(slots * 4u));
    w.inv = reinterpret_cast<uint32_t*>(take(slots * 4u));
    w.where = reinterpret_cast<uint2*>(take(slots * 8u));
    w.tiles = reinterpret_cast<int4*>(take(routed_tiles_max(slots, experts) * 16u));
    w.range = reinterpret_cast<uint32_t*>(take((kMixedBanksMax + 1u) * 4u));
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

cudaError_t launch_prefill_moe(const MoeArgs& a, const MixedBanks* mixed, void* workspace, int codebook, cudaStream_t stream,
                               int* launches) {
    const size_t slots = (size_t)a.rows * a.topk;
    const uint32_t S = (uint32_t)slots, H = a.hidden, I = a.inter;
    const MoeWs w = carve_moe(static_cast<uint8_t*>(workspace), slots, a.experts, H, I);
    const uint32_t* inds = static_cast<const uint32_t*>(a.inds);
    MixedBanks one;
    if (!mixed) {
        one.count = 1;
        one.n[0] = a.n;
        one.bank[0] = {a.gate_t, a.up_t, a.down_t, a.gate_suh, a.gate_svh, a.up_suh, a.up_svh, a.down_suh, a.down_svh, a.experts};
    }
    const MixedBanks& banks = mixed ? *mixed : one;
    // one expert (a shared expert's chain): the slots are in order as they stand, the chain is a dense one
    const bool routed = a.experts > 1u, overlap = a.overlap != 0;
    const SlotId ids = {SlotId::bits_for(banks.count)};
    cudaError_t rc;
    if (routed) {
        ExpertMap map = {};
        map.banks = banks.count;
        map.ids = mixed ? mixed->ids : a.experts;
        map.bank_of = mixed ? mixed->bank_of : nullptr;
        map.local_of = mixed ? mixed->local_of : nullptr;
        for (uint32_t b = 0; b < banks.count; ++b) map.base[b + 1u] = map.base[b] + banks.bank[b].experts;
        const Scatter scatter = {a.row_map, a.topk, ids, w.where, w.inv};
        const uint32_t blocks = (S + kRouteSlots - 1u) / kRouteSlots, hist_bytes = a.experts <= kRouteExperts ? a.experts * 4u : 0u;
        const bool whole = blocks == 1u && hist_bytes != 0u;
        if (!whole) rc = cudaMemsetAsync(w.counts, 0, ((size_t)a.experts + 1u) * 4u, stream);
        else rc = cudaSuccess;
        if (rc != cudaSuccess) return rc;
        rc = launch_overlapped(route_plan_kernel, dim3(blocks), kRouteThreads, hist_bytes, stream, overlap && whole, 1, inds, S, map, w.counts,
                               w.counts + a.experts, w.rank, w.first, w.tiles, w.range, whole ? scatter : Scatter{});
        if (rc == cudaSuccess && !whole)
            rc = launch_overlapped(route_scatter_kernel, dim3((S + 255u) / 256u), 256, 0, stream, overlap, 1, inds, S, map,
                                   static_cast<const uint32_t*>(w.rank), static_cast<const uint32_t*>(w.first), scatter);
        if (rc != cudaSuccess) return rc;
        *launches += whole ? 1 : 2;
    }
    PrepArgs pa = {};
    pa.x = a.x;
    pa.x_dt = a.x_dt;
    MidArgs m = {};
    for (uint32_t b = 0; b < banks.count; ++b) {
        pa.suh[0][b] = static_cast<const __half*>(banks.bank[b].gate_suh);
        pa.suh[1][b] = static_cast<const __half*>(banks.bank[b].up_suh);
        m.down_suh[b] = static_cast<const __half*>(banks.bank[b].down_suh);
    }
    pa.K = H;
    pa.positions = S;
    pa.where = m.where = routed ? w.where : nullptr;
    pa.ids = m.ids = ids;
    pa.row_map = a.row_map;
    pa.topk = a.topk;
    pa.xp = w.xp;
    pa.ops = 2;
    rc = launch_prep(pa, overlap, stream);
    if (rc != cudaSuccess) return rc;
    *launches += 2;  // and the SwiGLU's

    // A unit of work is two 128-output blocks where tiles of up to 128 rows are the rule (both run on one copy of the rows) and
    // there are units enough for every multiprocessor; else one. Two blocks against one, us a layer: 512 experts of 2048 x 512 K3
    // 674 / 751 at 80 slots an expert, 780 / 856 at 112, 903 / 944 at 128, 1070 / 1082 at 160, 1395 / 1334 at 224; 128 of 2048 x 768 K4
    // 262 / 287 at 80, 323 / 325 at 128, 370 / 368 at 160, 461 / 447 at 224; 64 of 4096 x 1024 K4 294 / 304 at 80, 336 / 335 at 112,
    // 417 / 401 at 160. Past 160 nothing is quicker with two; between 112 and 160 it goes by the geometry.
    auto gemm = [&](DecodeGemmArgs& g, const __half* rows, uint64_t rows_total) -> cudaError_t {
        const uint32_t ncol = g.N / 128u;
        g.mask = a.mask;
        g.op_rows = S;
        g.err = a.err;
        g.overlap = routed ? 0 : a.overlap;
        const bool down = g.ops == 1u;
        for (uint32_t b = 0; b < banks.count; ++b) {
            const BankTab& t = banks.bank[b];
            g.n = banks.n[b];
            g.svh[0] = static_cast<const __half*>(down ? t.down_svh : t.gate_svh);  // the epilogue finishes with the tile's expert's scales
            g.svh[1] = static_cast<const __half*>(t.up_svh);
            g.svh_stride = g.N;
            size_t units;
            if (routed) {
                const size_t tiles = routed_tiles_max(slots, t.experts);
                g.pair = slots <= (size_t)160u * a.experts && tiles * g.ops * ((ncol + 1u) / 2u) >= 2u * one_wave_ctas() ? 2u : 1u;
                g.tiles = w.tiles;
                g.range = w.range + b;
                units = tiles * g.ops * ((ncol + g.pair - 1u) / g.pair);
            } else {
                g.pair = 1;
                g.dense_rows = S;
                g.tile_rows = dense_tile_rows(S, g.K, ncol * g.ops, one_wave_ctas());
                g.dense_tiles = (S + g.tile_rows - 1u) / g.tile_rows;
                units = (size_t)g.dense_tiles * g.ops * ncol;
            }
            GemmMaps maps;
            if (!make_gemm_maps(&maps, rows, rows_total, g.K, down ? t.down_t : t.gate_t, down ? nullptr : t.up_t, g.N, g.n, t.experts))
                return cudaErrorNotSupported;
            g.bulk_out = g.scores == nullptr;
            if (g.bulk_out && !make_out_maps(&maps, g.z, (uint64_t)g.ops * S, g.N)) return cudaErrorNotSupported;
            // A bank's CTAs start as the one's before it run out of units (the first bank's start after the rows are complete): three banks
            // of 170 experts are five rounds each with the last half empty, 4096 rows of 512 experts at 2, 3 and 4 bits 728 -> 703 us
            if (b > 0u) g.overlap = a.overlap, g.beside = a.overlap != 0;
            const cudaError_t e = launch_decode_gemm(maps, g, (uint32_t)(units < (1u << 20) ? units : 1u << 20), codebook, stream);
            if (e != cudaSuccess) return e;
            *launches += 1;
        }
        return cudaSuccess;
    };
    DecodeGemmArgs gu = {};
    gu.K = H;
    gu.N = I;
    gu.ops = 2;
    gu.z = w.zgu;
    gu.z_op_stride = slots * I;
    rc = gemm(gu, w.xp, 2u * slots);
    if (rc != cudaSuccess) return rc;

    m.z = w.zgu;
    m.positions = S;
    m.inter = I;
    m.limit = a.limit;
    m.clamp_at = a.clamp_at;
    m.hd = w.hd;
    rc = launch_overlapped(mid_kernel, dim3(pair_ctas(S, I / 128u)), 256, 0, stream, overlap, 1, m);
    if (rc != cudaSuccess) return rc;

    // One slot a row of a one-expert bank: nothing to gather, so the GEMM's epilogue weights each row and stores it as y (the final
    // sum's launch and its pass over v fall away: 12 of 88 us at 4096 rows of 2048 x 512)
    const bool direct = !routed && a.topk == 1u && !a.shared;
    DecodeGemmArgs d = {};
    d.K = I;
    d.N = H;
    d.ops = 1;
    d.z = w.zd;  // each slot's finished down output, the per-slot v
    if (direct) d.y = a.y, d.y_dt = a.y_dt, d.scores = a.scores, d.score_dt = a.score_dt;
    rc = gemm(d, w.hd, slots);
    if (rc != cudaSuccess) return rc;

    if (direct) return cudaGetLastError();
    FinArgs f = {w.zd, routed ? w.inv : nullptr, a.scores, a.score_dt, a.shared, a.y, a.y_dt, a.rows, H, a.topk};
    if (a.shared_ready) {  // only this launch reads `shared`
        rc = cudaStreamWaitEvent(stream, static_cast<cudaEvent_t>(a.shared_ready), 0);
        if (rc != cudaSuccess) return rc;
    }
    const uint32_t fin_groups = (a.rows + 7u) / 8u, fin_want = (1184u + fin_groups - 1u) / fin_groups, fin_cols = (H + 255u) / 256u;
    rc = launch_overlapped(moe_fin_kernel, dim3(fin_want < fin_cols ? fin_want : fin_cols, fin_groups), 256, 0, stream,
                           overlap && !a.shared_ready, 1, f);
    if (rc != cudaSuccess) return rc;
    *launches += 1;
    return cudaGetLastError();
}

}  // namespace t3
