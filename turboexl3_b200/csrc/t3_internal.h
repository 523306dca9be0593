// Host-side declarations shared by the library's translation units (not part of the public C ABI).
#pragma once

#include <atomic>

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "../../include/t3.h"

namespace t3 {

struct RingPlan {
    uint32_t stage_rows, stages;
};

// One dense linear at decode rows (rows <= 32)
struct DenseArgs {
    const void* x;            // [rows, in], dtype x_dt
    const void* xp_g;         // or null: the rows already prepared (f16 [rows, in], lane order inside every 16) by t3_dense_prep,
                              // which the CTAs copy in instead of rotating x themselves (calls of more than 8 rows)
    void* y;                  // [rows, out], dtype x_dt
    const uint8_t* trellis;   // [in/16, out/16, n] u16
    const void* suh;          // f16 [in]
    const void* svh;          // f16 [out]
    uint32_t rows, in, out, n, mask;
    int x_dt;
    float* part;              // or null. Set: the K slices' partial sums meet in global memory, [out/128][split][rows][128] f32, not
                              // in a cluster's shared memory (any slice count, CTAs placed one by one: large linears whose
                              // CTA count then fills the multiprocessors evenly)
    uint32_t* counters;       // with part: [out/128] arrivals a block, zero before the launch; the last arriver finishes the block
    uint32_t split;           // K slices (the cluster size unless `part` is set)
    uint32_t slice_max;       // inputs of the largest K slice
    uint16_t alone;           // a CTA takes more than half a multiprocessor's shared memory (see kSmemAlone); 2: a large linear's
    uint16_t tile_over;       // row capacity 32: the K groups' partial-sum tile lies over the prepared rows (see gemv_smem)
    RingPlan ring;
    int overlap;              // launch with the programmatic-dependent-launch attribute
    uint32_t* err;
    unsigned long long* trace;  // optional: SM cycle counts at the phases of CTA (0, 0) (see t3_set_trace)
};
// (136 bytes of arguments, us a launch: 2048 -> 6144 K3 at one row 7.66 -> 7.72, 9216 -> 2688 10.52 -> 10.61)
static_assert(sizeof(DenseArgs) <= 128, "two lines of the constant cache");

// One more bank of a banked call (an expert streamer's slot banks: the same geometry and rate, its own slot count)
struct BankTab {
    const uint8_t *gate_t, *up_t, *down_t;
    const void *gate_suh, *gate_svh, *up_suh, *up_svh, *down_suh, *down_svh;
    uint32_t experts;
};
constexpr uint32_t kSkipId = 0xFFFFFFFFu;  // a banked call's id for a row-slot that runs no expert

// The routed chain at decode rows (rows <= 32): row-slot s = row * topk + k runs expert inds[s]
struct MoeArgs {
    const void* x;            // [rows, hidden], dtype x_dt
    int x_dt;
    const void* inds;         // [rows * topk] i32/u32
    const void* scores;       // [rows * topk], dtype score_dt
    int score_dt;
    const uint8_t *gate_t, *up_t, *down_t;
    const void *gate_suh, *gate_svh, *up_suh, *up_svh, *down_suh, *down_svh;  // f16, expert-major
    uint32_t experts, hidden, inter, topk, rows, n, mask;
    float limit;              // SwiGLU clamp, 0 = none
    int clamp_at;             // 0 gate_in, 1 silu_out
    void* hd;                 // scratch f16 [rows * topk, inter]: the down projection's prepared inputs
    void* v;                  // scratch f16 [rows * topk, hidden]: each row-slot's finished down output
    void* y;                  // [rows, hidden], dtype x_dt
    const void* shared;       // optional [rows, hidden] dtype x_dt added at y's rounding point, or null
    const uint32_t* row_map;  // prefill rows only: row-slot p reads x's row row_map[p] (top-1 over gathered rows), or null
    int y_dt;                 // y's dtype: x_dt, except for the gathered-rows and banked entries
    uint32_t banked;          // decode rows, top-1: inds holds packed ids (bank << 24 | slot); banks 1 and 2 in ext; scores null = 1
    BankTab ext[2];
    void* shared_ready;       // host side only: an event the last launch (the one that reads `shared`) waits for, or null
    uint32_t row_cap;                  // rows a CTA's decode of an expert's weights serves (8 or 16): an expert with more members takes more CTAs
    uint32_t split_gu, slice_max_gu;   // K slices of gate|up (cluster = 2 * split_gu), largest slice
    uint32_t split_d, slice_max_d;     // K slices of down
    uint32_t per_d;                    // output blocks of down a CTA takes (1 unless split_d is)
    uint32_t alone_gu;                 // gate|up's CTAs take more than half a multiprocessor's shared memory each (see kSmemAlone)
    RingPlan ring_gu, ring_d;
    uint32_t down_early;               // gate|up lets the down launch start as soon as it has the routing (see plan_moe_decode)
    int overlap;
    uint32_t* err;
};

// Raises a kernel's dynamic shared-memory limit on the current device, once a device (`ready`: a bit an ordinal, one word a
// kernel): the driver call costs more than the check.
inline cudaError_t allow_smem_once(std::atomic<uint64_t>& ready, const void* kernel, uint32_t bytes) {
    int dev = 0;
    cudaError_t rc = cudaGetDevice(&dev);
    if (rc != cudaSuccess) return rc;
    const uint64_t bit = dev < 64 ? 1ull << dev : 0ull;
    if (ready.load(std::memory_order_acquire) & bit) return cudaSuccess;
    rc = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (rc == cudaSuccess) ready.fetch_or(bit, std::memory_order_release);
    return rc;
}

// A launch that may start while the stream's previous kernel is still running (`overlap`; the kernel orders itself with pdl_wait,
// see t3_common.cuh), of one CTA or a cluster of `cluster` along grid x.
template <typename... Params>
cudaError_t launch_overlapped(void (*fn)(Params...), dim3 grid, uint32_t block, uint32_t smem, cudaStream_t stream, bool overlap,
                              uint32_t cluster, const Params&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    unsigned n = 0;
    if (overlap) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster > 1u) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = cluster;
        attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
        ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, fn, args...);
}

// remembers, per host thread, the kernel a decode-row launch is about to run (t3_last_kernel_symbol names it)
void note_symbol(const void* kernel);

cudaError_t launch_dense_gemv(const DenseArgs& a, int codebook, cudaStream_t stream);
// the input rotation of every row once, into a.xp_g (ahead of launch_dense_gemv on the same stream)
cudaError_t launch_dense_prep(const DenseArgs& a, cudaStream_t stream);
constexpr uint32_t kFusedRows = 8;  // up to this many rows a dense decode-row CTA rotates x itself
cudaError_t launch_moe_gate_up(const MoeArgs& a, int codebook, cudaStream_t stream);
cudaError_t launch_moe_down(const MoeArgs& a, int codebook, cudaStream_t stream);
cudaError_t launch_moe_merge(const MoeArgs& a, cudaStream_t stream);

// shared-memory bytes the GEMV CTAs of a plan need (for admission before launch)
uint32_t gemv_smem_bytes(uint32_t row_cap, uint32_t xrows, uint32_t slice_max, uint32_t cluster, uint32_t n, RingPlan ring, bool alone = false,
                         uint32_t buffers = 1, bool over = false);
// the most dynamic shared memory a GEMV CTA may be launched with
constexpr uint32_t kGemvSmemLimit = 200u * 1024u;
uint32_t row_cap_for(uint32_t rows);

// Row limits of the prefill calls. The routed chain's last launch has its rows, eight a group, in a grid dimension (65535 at most);
// the dense and the row-slot limits are what these entry points have always admitted.
constexpr size_t kPrefillDenseRowsMax = (size_t)65535 * 64;
constexpr size_t kPrefillMoeRowsMax = (size_t)65535 * 8;
constexpr size_t kPrefillSlotsMax = (size_t)65535 * 64;

// One dense linear at prefill rows (rows > 32): prepare -> tcgen05 GEMM with the decode in its weight loader -> finish
struct PrefillLinearArgs {
    const void* x;
    void* y;
    const uint8_t* trellis;
    const void* resident;  // W_hat transposed, f16 [out, in], kept by the caller: the GEMM loads it instead of decoding; or null
    const void* suh;
    const void* svh;
    uint32_t rows, in, out, n, mask;
    int x_dt;
    void* workspace;  // prefill_linear_workspace bytes
    uint32_t* err;
    int overlap;      // launch with the programmatic-dependent-launch attribute
};
size_t prefill_linear_workspace(size_t rows, uint32_t in, uint32_t out);
cudaError_t launch_prefill_linear(const PrefillLinearArgs& p, int codebook, cudaStream_t stream, int* launches);
// Several banks of one geometry, each at a rate of its own (a layer whose experts were quantised at different bit widths): the
// router's expert g is expert local_of[g] of bank bank_of[g] (device arrays of `ids` entries).
constexpr uint32_t kMixedBanksMax = 8;
struct MixedBanks {
    uint32_t count, ids;
    const int64_t *bank_of, *local_of;
    BankTab bank[kMixedBanksMax];
    uint32_t n[kMixedBanksMax];
};
// t3_linear and its workspace; far_x: x lies across the bus (a host array the kernels read in place), so at decode rows it is
// rotated once by a launch of its own: read by every 128-output block instead, a row of 1536 crossed the bus 192 times for 24576
// outputs
size_t linear_workspace(size_t rows, int in_dim, int out_dim, int n, bool far_x);
int linear_call(const void* x, int x_dtype, size_t rows, const void* trellis, const void* suh, const void* svh, int in_dim, int out_dim,
                int n, t3_decode dec, void* y, void* workspace, size_t workspace_bytes, void* stream, bool far_x);
// The routed chain at prefill rows: route -> prepare -> GEMM(gate|up) -> mid -> GEMM(down) -> finish
size_t prefill_moe_workspace(size_t rows, uint32_t topk, uint32_t experts, uint32_t hidden, uint32_t inter);
// mixed: the banks in the place of a's own (whose geometry, rows and clamp count; a.experts is the sum of the banks'), or null
cudaError_t launch_prefill_moe(const MoeArgs& a, const MixedBanks* mixed, void* workspace, int codebook, cudaStream_t stream, int* launches);

// W_hat f16 from the trellis: [in, out], or transposed [out, in]
cudaError_t launch_dequant(const uint8_t* trellis, uint32_t in, uint32_t out, uint32_t n, uint32_t mask, int codebook,
                           int transposed, void* what, cudaStream_t stream);
// W_hat transposed [out, in] f16 -> W_std transposed in dtype dt (f16 / bf16), in place: diag(suh) H W_hat H diag(svh)
cudaError_t launch_unrot(void* w_t, const void* suh, const void* svh, uint32_t in, uint32_t out, int dt, cudaStream_t stream);
// y = x W_std (x and the weight in the same 16-bit dtype, f32 accumulation, one rounding): the plain tensor-core GEMM
cudaError_t launch_plain_linear(const void* x, int dt, uint32_t rows, const void* w_std_t, uint32_t in, uint32_t out, void* y,
                                uint32_t* err, bool overlap, cudaStream_t stream);
// the expert-parallel dispatch plan of one rank's routing (see ep_plan_kernel); world 1..8, experts a multiple of world
cudaError_t launch_ep_plan(const uint32_t* inds, uint32_t rows, uint32_t topk, uint32_t experts, uint32_t world, uint32_t* order,
                           uint32_t* where, uint32_t* send_rows, void* meta, int* counts, cudaStream_t stream);
// test hook: a one-warp kernel whose bounded wait runs out (about a second) and sets the full-wait bit of `err`
cudaError_t launch_wait_runs_out(uint32_t* err, cudaStream_t stream);
// all 65,536 codewords through the kernels' decoders: out[cw] = f16 bits (test hook)
cudaError_t launch_codebook_table(int codebook, uint32_t mask, uint16_t* out, cudaStream_t stream);

}  // namespace t3
