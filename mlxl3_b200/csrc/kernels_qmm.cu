// Tensor-core product for many activation rows (prefill, verify batches, grouped experts): trellis tiles are decoded into
// tensor memory, where tcgen05.mma reads them as its A operand; the accumulator is in tensor memory too.
//
// Reference behaviour replaced: native/shaders/_qmm_tensor_shared_kernel.metal (decode a weight tile
// once, share it across row groups, matrix-unit product with fp32 accumulation) driven by
// native/src/linear.rs:1874-2081, with the output rotation of native/src/linear.rs:1940-1963.
//
// Mapping.  The product is computed transposed, D[out, token] = W^T[out, in] . Xhat^T[in, token]:
//  * an item is 128 output columns (the 128 lanes of tensor memory) x one tile of up to NT tokens (the MMA's N); its
//    inputs are walked in stages of 128.  The stages of all items, item after item, are dealt out to the CTAs of ONE wave
//    in equal runs (one CTA per SM), so no SM idles whatever the shape; a CTA that holds a whole item rotates and stores
//    it, CTAs that share one leave fp32 pieces and the last to arrive adds them in input order;
//  * A operand: sixteen decoder warps in two groups that take alternate stages; a warp owns the 32 lanes of its quarter of
//    tensor memory = two 16-column tiles, of four of the stage's eight tile rows.  A lane's eight weights of a tile are the
//    fragment of the 16x128b store shape, so a decoded tile goes from registers to tensor memory in one instruction;
//  * B operand: rotated activations, two TMA tensor copies of [tile tokens, 64 in] fp16 per stage, 128-byte swizzle;
//  * packed words: one bulk copy per stage (8 tile rows x 8 tiles are contiguous in the quad layout);
//  * one thread issues the stage's eight products and one commit, which frees the A stage and the activation slot.
//  * tiles of up to 64 tokens, several of them on a CTA: two accumulators, so that four more warps finish an item while the next one
//    is multiplied.
//
// What bounds it: up to 64 rows the decode, and of it the issue slots: the decode loop alone (words resident in shared memory,
// tensor-memory stores and nothing else) executes 43 warp instructions per 16x16 tile at 4 bits and 48 at 3, in 47 to 49 and 51 to 53
// cycles per tile and scheduler; in the kernel all roles together execute 51 (4 bits), at 0.80 per cycle (instruction cache
// misses, the single-thread roles), 64 cycles per tile from the first stage to the last.  The clock is 1845 MHz by the cycle counter
// while tensor-core instructions run (nvidia-smi reports 1965).  A stage takes the same time however many SMs work and wherever the
// weights come from (measured with 37, 74 and 148 SMs, and with all stages reading the same ones).  At NT = 256 a stage takes 1320 cycles, 1024 of them products, and back to back the power cap holds the clock at 1560.
// Stages of 128 inputs and a single barrier per stage are there because the single-thread roles share the schedulers with
// decoders that keep the integer pipes full: an instruction of theirs takes about eight cycles, a stage of any of them 400 to
// 600.  For the same reason the issuing loop is unrolled over the ring and its thread picked by elect.sync; the producers'
// loops stay rolled (all three unrolled: 714 ns per 64 inputs against 523).  Us per call with the input rotation: 64 rows
// 4096->14336, 4 bits, 21.4; 16 rows 5120->2x25600, 3 bits, 72.0.
// Every wait is bounded in time; a wait that gives up sets the status word and the kernel still releases its tensor memory.
#include <cuda.h>

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "kernels.h"
#include "hadamard.cuh"
#include "tile_decode.cuh"

namespace b200exl3 {

// What a CTA is built for: tiles of up to 64 tokens, where every item has CTAs of its own or where a CTA holds several; large tiles.
enum class QmmForm { kSmall, kSmallItems, kLarge };

namespace {

// The single-thread roles take the lowest warp numbers: the scheduler favours older warps.
constexpr int kMmaWarp = 0, kWeightWarp = 1, kActWarp = 2, kFirstDecoder = 4;
constexpr int kStageCols = 64;                         // tensor-memory columns of an A stage: two fp16 inputs each
constexpr int kChunk = 16;                             // tokens four warps finish at a time

template <int K, int NT, bool FIN>
struct QmmShape {
    static constexpr int kGroups = 2;                  // groups of eight decoder warps that take alternate stages
    static constexpr int kDecoders = 8 * kGroups;
    // Small tiles: two accumulators, and with FIN four warps that finish an item while the next one is decoded and multiplied; the
    // decoders finish only the CTA's last item.  Before, the pipeline drained at every item (5000 cycles, 2000 of them waiting for the last
    // products): 16 rows 5120->2x25600, 3 bits, 84.8 -> 80.1 us; expert block 37 / 256 tokens 176 -> 165 / 250 -> 230.  Without FIN a
    // CTA has one item, and the warps would have nothing to do but to start with it.  Us with / without them, 4 bits: 24 rows 2048->2048
    // 9.3 / 9.05, 4096->4096 12.4 / 11.9, 64 rows 14336->4096 25.8 / 25.4, 4096->14336 21.7 / 21.55.  (The loop over several items that
    // large tiles take instead spills here: 24 rows 4096->14336 22.7.)
    // Large tiles leave no tensor memory for a second accumulator: their decoders finish every item.
    static constexpr uint32_t kAccums = NT == 64 ? 2 : 1;
    static constexpr int kFinishers = NT == 64 ? 4 : kDecoders;
    static constexpr int kThreads = 32 * (kFirstDecoder + kDecoders + (FIN ? kFinishers : 0));
    // Small tiles get the registers of 768 threads, 80 each, also when 640 start: that leaves room on the SM for a CTA of the kernel after
    // this one, whose 256 threads rotate the next call's input and may lie there until this kernel is done.  With 89 registers they
    // waited for SMs that a full wave does not leave: us with 89 / 80, 4 bits, 64 rows 4096->4096 14.9 / 12.8, 24 rows 8192->2048 14.5 / 12.8,
    // 16 rows 14336->4096 22.5 / 20.4, 48 rows 10240->1280 15.5 / 13.6; level where the grid leaves 20 SMs or more.
    static constexpr int kBoundThreads = NT == 64 ? 768 : kThreads;
    static constexpr int kSlots = NT == 64 ? 6 : 4;    // A stages in tensor memory beside the accumulators
    // Packed stages (2048 * K bytes) in flight.  A multiple of the decoder groups, so that a slot always belongs to one group:
    // parity alone does not tell a phase from the one after the next, and a group that met a slot only every other time could
    // take a copy that has not landed for its own.  With two slots above 4 bits the decoders waited for the copies: 1969 rows
    // 7936->1408, 6 bits, 98 -> 83 us; 128 rows 4096->14336, 8 bits, 37.9 -> 31.
    static constexpr int kRaw = NT == 64 && K <= 4 ? 6 : 4;
    static_assert(kRaw % kGroups == 0, "a slot belongs to one group");
    static constexpr int kBSlots = NT == 64 ? kSlots : 2;   // activation stages in shared memory; divides kSlots
    static constexpr uint32_t kBHalfBytes = NT * 128;  // NT tokens x 64 fp16
    static constexpr uint32_t kBSlotBytes = 2 * kBHalfBytes;
    static constexpr uint32_t kEpilogueBytes = (kDecoders / 4 + (NT == 64 && FIN ? 1 : 0)) * 2 * kChunk * 128 * sizeof(__half);
    static_assert(kAccums * NT + kSlots * kStageCols <= 512 && kSlots % kGroups == 0 && kSlots % kBSlots == 0, "tensor memory");
};
template <int K, int NT, bool FIN>
constexpr size_t qmm_smem_bytes() {
    using S = QmmShape<K, NT, FIN>;
    return 1024 + S::kBSlots * S::kBSlotBytes + static_cast<size_t>(S::kRaw) * 2048 * K + S::kEpilogueBytes;
}

__device__ __forceinline__ uint64_t umma_desc(uint32_t smem_byte_addr) {
    // K-major operand, 128-byte swizzle: 8-row groups 1024 bytes apart, descriptor version 1
    uint64_t d = 0;
    d |= static_cast<uint64_t>((smem_byte_addr & 0x3ffffu) >> 4);
    d |= static_cast<uint64_t>(1) << 16;                 // leading byte offset (unused for swizzled K-major)
    d |= static_cast<uint64_t>(1024 >> 4) << 32;         // stride byte offset
    d |= static_cast<uint64_t>(1) << 46;                 // version
    d |= static_cast<uint64_t>(2) << 61;                 // SWIZZLE_128B
    return d;
}

__device__ __forceinline__ void tmem_alloc(uint32_t* smem_dst, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(smem_dst)), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
// D[tmem] (+)= A[tmem] . B[smem]
__device__ __forceinline__ void umma_f16_ts(uint32_t d, uint32_t a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}"
        ::"r"(d), "r"(a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// One lane of a converged warp.  Products issued under `if (elect_one())` take 30 cycles each, under `if (lane == 0)` 68
// (128 x 16..64 tile, back to back): the first branch is known to be uniform, as the descriptors' registers want it.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}
// The same by the lanes for which `arrive` holds, without a branch; bar is a shared-memory address.
__device__ __forceinline__ void mbar_arrive(bool arrive, uint32_t bar) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %1, 0;\n@p mbarrier.arrive.shared::cta.b64 _, [%0];\n}"
                 ::"r"(bar), "r"(static_cast<uint32_t>(arrive)) : "memory");
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int c0, int c1, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(smem_addr(dst)), "l"(map), "r"(smem_addr(bar)), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// 16 lanes x 8 columns: the weights of one decoded tile, row g and g + 8, inputs 2q, 2q+1 and 2q+8, 2q+9 of the lane
template <int OFFSET>
__device__ __forceinline__ void tmem_st_tile(uint32_t taddr, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3) {
    asm volatile("tcgen05.st.sync.aligned.16x128b.x2.b32 [%0+%5], {%1,%2,%3,%4};" ::"r"(taddr), "r"(a0), "r"(a1), "r"(a2), "r"(a3), "n"(OFFSET));
}

// Wait that gives up after about a quarter of a second, or at once when another role of the CTA has
// already given up, so that a lost copy or a miscounted barrier ends the kernel instead of hanging it.
__device__ __noinline__ bool qmm_wait_slow(uint64_t* bar, uint32_t parity, volatile int* cta_failed) {
    for (int i = 0; i < 64; ++i)
        if (mbar_try_wait(bar, parity)) return true;
    constexpr uint32_t kNap = 20000;                             // the hardware wakes the thread when the phase completes
    const unsigned long long t0 = global_ns();
    while (true) {
        if (mbar_try_wait_for(bar, parity, kNap)) return true;
        if (*cta_failed || global_ns() - t0 > 250000000ull) { *cta_failed = 1; return false; }
    }
}
__device__ __forceinline__ bool qmm_wait(uint64_t* bar, uint32_t parity, volatile int* cta_failed) {
    return mbar_try_wait(bar, parity) || qmm_wait_slow(bar, parity, cta_failed);
}
// Barrier of some warps.  Not the aligned form (`bar.sync`), which all lanes of a warp have to execute as one: lanes come here
// from branches of their own (lane 0 from an atomic or an arrival), where nothing but a warp barrier brings them together again.
// The same holds for the instructions marked .sync.aligned -- allocation and release of tensor memory, its loads and stores and
// the waits for them: each has a warp barrier before it with no branch on the lane, no elected lane and no polling loop in
// between, and the branches around it are on values that all lanes share (warp, item, token counts).
__device__ __forceinline__ void group_sync(int id, int threads) {
    __syncwarp();
    asm volatile("barrier.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
    __syncwarp();
}

// What an item is: where its weights, its activation rows and its outputs are.
struct QmmItem {
    int wblock;      // column block of the weight array
    int cblock;      // column block of the output space (dense) or of the projection's columns (experts)
    int brow;        // first activation row
    int n;           // tokens
    int tok0;        // first token of the batch (dense) / first output row (experts)
};
template <int NT>
__device__ __forceinline__ QmmItem qmm_item(const QmmArgs& p, uint32_t item) {
    QmmItem it;
    if (p.map_expert != nullptr) {
        const int sp = static_cast<int>(item) / p.map_blocks, j = static_cast<int>(item) - sp * p.map_blocks;
        const int seg = sp / p.map_proj, proj = sp - seg * p.map_proj;
        const int expert = static_cast<int>(min(p.map_expert[seg], static_cast<uint32_t>(p.map_experts - 1)));
        it.wblock = proj * p.map_stride_blocks + expert * p.map_blocks + j;
        it.cblock = j;
        it.brow = it.tok0 = proj * p.map_slots + p.map_row0[seg];
        it.n = p.map_rows[seg];
    } else {
        const int cb = static_cast<int>(item) / p.tiles, t = static_cast<int>(item) - cb * p.tiles;
        int grp = 0;
        while (grp + 1 < p.groups && cb * 128 >= p.gcol0[grp + 1]) ++grp;
        it.wblock = it.cblock = cb;
        it.tok0 = t * p.tile_tokens;
        it.brow = grp * p.rows + it.tok0;
        it.n = min(p.rows - it.tok0, p.tile_tokens);
    }
    return it;
}

// Where the outputs of an item go: base of its columns in the member's rows, this lane's four output scales.
struct QmmStore {
    void* y;
    int64_t ld, col;
    const __half* bias;
    __half sv[4];
};
__device__ __forceinline__ QmmStore qmm_store_of(const QmmArgs& p, const QmmItem& it, int lane) {
    QmmStore st;
    int grp = 0;
    while (grp + 1 < p.groups && it.cblock * 128 >= p.gcol0[grp + 1]) ++grp;
    const int col = it.cblock * 128 + lane * 4;
    st.y = p.gy[grp];
    st.ld = p.gout[grp];
    st.col = col - p.gcol0[grp];
    st.bias = p.bias ? p.bias + col : nullptr;
    *reinterpret_cast<uint2*>(st.sv) = *reinterpret_cast<const uint2*>(p.svh + col);
    return st;
}
// four columns of one rotated row: scaled and stored
__device__ __forceinline__ void qmm_store4(const QmmArgs& p, const QmmStore& st, int64_t t, __half (&h)[4]) {
#pragma unroll
    for (int e = 0; e < 4; ++e) h[e] = __hmul_rn(h[e], st.sv[e]);
    store4_from_half(st.y, p.y_dtype, t * st.ld + st.col, h, st.bias);
}

// Staging rows are 128 fp16 with the 16-byte chunks 8..15 swapped in pairs, so that eight lanes that read 32 neighbouring
// bytes each use all banks.
__device__ __forceinline__ int stage_col(int col) { return col ^ ((col & 64) >> 3); }

// Four staged rows (one warp's own): rotated, scaled and stored.  Eight lanes share a row, sixteen columns each: four of the
// seven butterfly stages stay in registers and a lane has sixteen independent chains, against four columns a lane, five
// shuffle stages and four chains for one row at a time.  512 rows 4096->14336, 4 bits: 78.2 -> 71.6 us with the sums below.
__device__ __forceinline__ void qmm_finish4(__half* rows, const QmmArgs& p, const QmmStore& st, int64_t t0, int n, int lane) {
    __align__(16) __half2 h[8];
    const int l8 = lane & 7, flip = l8 >> 2;
    uint4* const mine = reinterpret_cast<uint4*>(rows + (lane >> 3) * 128 + l8 * 16);
    reinterpret_cast<uint4*>(h)[0] = mine[flip];
    reinterpret_cast<uint4*>(h)[1] = mine[flip ^ 1];
    float v[16];
#pragma unroll
    for (int i = 0; i < 8; ++i) { const float2 f = __half22float2(h[i]); v[2 * i] = f.x; v[2 * i + 1] = f.y; }
#pragma unroll
    for (int s = 1; s <= 8; s <<= 1)
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if (!(i & s)) { const float x = v[i], y = v[i | s]; v[i] = __fadd_rn(x, y); v[i | s] = __fsub_rn(x, y); }
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = round_half(v[i]);
#pragma unroll
    for (int bit = 1; bit <= 4; bit <<= 1) {
        const float sign = (lane & bit) ? -1.0f : 1.0f;               // upper half: peer - own, exact in one fma
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = __fmaf_rn(sign, v[i], __shfl_xor_sync(0xffffffffu, v[i], bit));
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
        h[i] = __halves2half2(__float2half_rn(__fmul_rn(round_half(v[2 * i]), had_scale())), __float2half_rn(__fmul_rn(round_half(v[2 * i + 1]), had_scale())));
    mine[flip] = reinterpret_cast<const uint4*>(h)[0];
    mine[flip ^ 1] = reinterpret_cast<const uint4*>(h)[1];
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 4; ++j)
        if (j < n) {
            __align__(8) __half o[4];
            *reinterpret_cast<uint2*>(o) = *reinterpret_cast<const uint2*>(rows + j * 128 + stage_col(lane * 4));
            qmm_store4(p, st, t0 + j, o);
        }
    __syncwarp();
}

template <int K, int CB, int NT, bool FIN>
__global__ void __launch_bounds__(QmmShape<K, NT, FIN>::kBoundThreads, 1)
qmm_kernel(const __grid_constant__ CUtensorMap xmap, const QmmArgs p) {
    using S = QmmShape<K, NT, FIN>;
    // Dependent launch: this kernel may be scheduled under the tail of the kernel before it (the input rotation, the
    // glue of the expert block).  The packed weights are nobody's output, so the barriers, the tensor memory and the
    // first weight copies do not wait; what that kernel wrote -- the rotated rows, the segment table -- is read only
    // after griddepcontrol.wait (expert-mapped mode: at once, the table is read first; otherwise by the activation
    // producer before its first copy), and nothing is stored to global memory before it either (the decoders wait
    // before the epilogue).
    pdl_launch_dependents();
    if (p.map_expert != nullptr) pdl_wait();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int kRawWords = 512 * K;                       // a packed stage: 8 tile rows x 2 quads x 32K words
    constexpr uint32_t kRawBytes = kRawWords * 4;
    __shared__ __align__(8) uint64_t full[S::kSlots], done[S::kSlots], full2[S::kSlots], half[S::kSlots], raw_full[S::kRaw], raw_empty[S::kRaw];
    __shared__ __align__(8) uint64_t accum_full[S::kAccums], accum_free[S::kAccums], last_full;
    __shared__ uint32_t tmem_base_slot, s_last[2];
    __shared__ volatile int s_failed;

    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;   // warp: uniform
    const uint32_t spi = static_cast<uint32_t>(p.in) / kQmmStageIn;                       // stages of an item
    const uint32_t items = p.map_expert != nullptr ? static_cast<uint32_t>(*p.map_count * p.map_proj * p.map_blocks) : static_cast<uint32_t>(p.items);
    // one run per CTA, at least one stage each; the launch keeps total * CTAs below 2^32
    const uint32_t total = items * spi, G = min(gridDim.x, total);
    if (blockIdx.x >= G) return;
    const uint32_t s0 = total * blockIdx.x / G, s1 = total * (blockIdx.x + 1) / G;
    if (s0 == s1) return;                                                        // uniform for the CTA; nothing is allocated yet
    const int count = static_cast<int>(s1 - s0);
    unsigned long long* tr = p.trace ? p.trace + blockIdx.x * 8 : nullptr;
    if (tr && threadIdx.x == 0) tr[0] = global_ns();

    // shared memory: activation ring | packed ring | epilogue staging; the swizzled operand needs 1024-byte alignment
    unsigned char* b_base = smem_raw + ((1024u - (smem_addr(smem_raw) & 1023u)) & 1023u);
    uint32_t* raw_base = reinterpret_cast<uint32_t*>(b_base + S::kBSlots * S::kBSlotBytes);
    __half* stage_base = reinterpret_cast<__half*>(raw_base + S::kRaw * kRawWords);

    if (threadIdx.x == 0) {
        // a stage is full when its eight decoder warps and its activation copies have arrived (of a large tile the first half;
        // the second has a barrier of its own, and so has the end of the first half's products)
        for (int s = 0; s < S::kSlots; ++s) { mbar_init(&full[s], 9); mbar_init(&done[s], 1); mbar_init(&full2[s], 1); mbar_init(&half[s], 1); }
        for (int s = 0; s < S::kRaw; ++s) { mbar_init(&raw_full[s], 1); mbar_init(&raw_empty[s], 8); }
        mbar_init(&last_full, 1);
        for (uint32_t s = 0; s < S::kAccums; ++s) { mbar_init(&accum_full[s], 1); mbar_init(&accum_free[s], S::kFinishers); }
        s_failed = 0;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncwarp();                                                // thread 0 comes from a branch of its own
    if (warp == kMmaWarp) tmem_alloc(&tmem_base_slot, 512);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base_slot;
    const uint32_t first_item = s0 / spi, k0 = s0 - first_item * spi;            // first item and its first stage here
    const uint32_t last_item = (s1 - 1) / spi;
    const int last_stages = static_cast<int>(s1 - max(s0, last_item * spi));     // stages of the last item here
    if (tr && threadIdx.x == 0) tr[1] = global_ns();

    int buf = 0;                                                 // half of the staging rows that the next sixteen tokens go through
    // Epilogue of an item (or of this CTA's part of it) by W warps, of which this is the one numbered w: the sixteen decoders, or
    // the four warps that finish items while the next one is decoded.
    auto finish_item = [&](auto warps, const int w, const uint32_t item, const uint32_t seg, const int stages, const uint32_t quarter_lanes,
                           __half* staging, uint32_t* last, const int quad_bar, const int all_bar) {
        constexpr int W = decltype(warps)::value;
        const int quad = w >> 2, quarter = w & 3;
        const uint32_t acc = quarter_lanes + (seg % S::kAccums) * NT;
        const QmmItem info = qmm_item<NT>(p, item);
        QmmStore store{};
        if (p.yhat == nullptr) store = qmm_store_of(p, info, lane);
        // The decoders that take only the last item have a barrier of their own for it: they may come several items early, when the
        // parity of a barrier that completes once every two items does not tell their phase from an older one.
        const bool single = W > S::kFinishers;
        qmm_wait(single ? &last_full : &accum_full[seg % S::kAccums], single ? 0u : (seg / S::kAccums) & 1u, &s_failed);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        __syncwarp();
        const bool complete = stages == static_cast<int>(spi);
        // parts of shared items in order of (CTA, item): CTA + item numbers them; with more items than CTAs, two per CTA
        const size_t piece_floats = static_cast<size_t>(p.tile_tokens) * 128;
        float* piece = p.pieces + (items < G ? blockIdx.x + item : 2 * blockIdx.x + (seg > 0 ? 1 : 0)) * piece_floats;
        // chunks of 16 tokens: four warps hold 32 columns each of the same tokens
        for (int c = quad * kChunk; c < info.n; c += W / 4 * kChunk) {
            uint32_t r[16];
            __syncwarp();
            tmem_ld16(acc + c, r);
            if (!complete || p.yhat != nullptr) {
                float* dst = complete ? p.yhat + static_cast<int64_t>(info.tok0 + c) * p.yhat_ld + info.cblock * 128 + quarter * 32 + lane
                                      : piece + c * 128 + quarter * 32 + lane;
                const int64_t ld = complete ? p.yhat_ld : 128;
#pragma unroll
                for (int i = 0; i < kChunk; ++i)
                    if (c + i < info.n) dst[i * ld] = __uint_as_float(r[i]);
            } else {
                // the output rotation runs over the 128 columns of a token: transposed through shared memory, then
                // every warp rotates four tokens
                __half* stage = staging + (quad * 2 + buf) * (kChunk * 128);
#pragma unroll
                for (int i = 0; i < kChunk; ++i) stage[i * 128 + stage_col(quarter * 32 + lane)] = __float2half_rn(__uint_as_float(r[i]));
                group_sync(quad_bar, 128);
                if (c + quarter * 4 < info.n)
                    qmm_finish4(stage + quarter * 512, p, store, info.tok0 + c + quarter * 4, info.n - c - quarter * 4, lane);
                buf ^= 1;
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0 && W == S::kFinishers) mbar_arrive(&accum_free[seg % S::kAccums]);   // the accumulator may be overwritten
        __syncwarp();
        if (!complete) {
            // CTAs share the item: this one's part is a piece; the last to arrive adds the pieces in input order
            const uint32_t x0 = item * spi;
            const uint32_t c_first = ((x0 + 1) * G - 1) / total, c_last = ((x0 + spi) * G - 1) / total;
            __threadfence();
            group_sync(all_bar, W * 32);
            if (w == 0 && lane == 0) {
                const unsigned int before = atomicAdd(p.counters + item, 1u);
                *last = before == c_last - c_first;
                if (*last) p.counters[item] = 0;            // leave the scratch ready for the next call
            }
            group_sync(all_bar, W * 32);
            if (*last) {
                __threadfence();
                // the first CTA's part is its last one if it starts before the item, the others' their first
                const size_t stride = items < G ? piece_floats : 2 * piece_floats;
                const float* base = p.pieces + (items < G ? c_first + item : 2 * c_first) * piece_floats + lane * 4;
                const float* base0 = base + (items >= G && total * c_first / G < x0 ? piece_floats : 0);
                const int pieces = static_cast<int>(c_last - c_first) + 1;
                auto store_sum = [&](int t, const float4& a) {
                    *reinterpret_cast<float4*>(p.yhat + static_cast<int64_t>(info.tok0 + t) * p.yhat_ld + info.cblock * 128 + lane * 4) = a;
                };
                if (info.n <= W) {
                    // few rows: one per warp, up to four parts in flight
                    if (w < info.n) {
                        float4 a = __ldcg(reinterpret_cast<const float4*>(base0 + w * 128));
                        const float* src = base + stride + w * 128;
#pragma unroll 4
                        for (int q = 1; q < pieces; ++q, src += stride) {
                            const float4 part = __ldcg(reinterpret_cast<const float4*>(src));
                            a.x = __fadd_rn(a.x, part.x); a.y = __fadd_rn(a.y, part.y); a.z = __fadd_rn(a.z, part.z); a.w = __fadd_rn(a.w, part.w);
                        }
                        if (p.yhat != nullptr) {
                            store_sum(w, a);
                        } else {
                            __half h[4] = {__float2half_rn(a.x), __float2half_rn(a.y), __float2half_rn(a.z), __float2half_rn(a.w)};
                            warp_hadamard128_f16(h, lane);
                            qmm_store4(p, store, info.tok0 + w, h);
                        }
                    }
                } else {
                    __half* mine = staging + w * 512;
                    for (int t0 = w * 4; t0 < info.n; t0 += 4 * W) {
                        int row[4];
                        float4 a[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            row[i] = min(t0 + i, info.n - 1) * 128;
                            a[i] = __ldcg(reinterpret_cast<const float4*>(base0 + row[i]));
                        }
                        const float* src = base + stride;
#pragma unroll 1
                        for (int q = 1; q < pieces; ++q, src += stride) {
                            float4 part[4];
#pragma unroll
                            for (int i = 0; i < 4; ++i) part[i] = __ldcg(reinterpret_cast<const float4*>(src + row[i]));
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                a[i].x = __fadd_rn(a[i].x, part[i].x); a[i].y = __fadd_rn(a[i].y, part[i].y);
                                a[i].z = __fadd_rn(a[i].z, part[i].z); a[i].w = __fadd_rn(a[i].w, part[i].w);
                            }
                        }
                        if (p.yhat != nullptr) {
#pragma unroll
                            for (int i = 0; i < 4; ++i)
                                if (t0 + i < info.n) store_sum(t0 + i, a[i]);
                        } else {
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                __align__(8) const __half2 h[2] = {__floats2half2_rn(a[i].x, a[i].y), __floats2half2_rn(a[i].z, a[i].w)};
                                *reinterpret_cast<uint2*>(mine + i * 128 + stage_col(lane * 4)) = *reinterpret_cast<const uint2*>(h);
                            }
                            __syncwarp();
                            qmm_finish4(mine, p, store, info.tok0 + t0, info.n - t0, lane);
                        }
                    }
                    group_sync(all_bar, W * 32);        // the next item stages in other warps' rows
                }
            }
        }
    };

    if (FIN && warp >= kFirstDecoder + S::kDecoders) {
        // ================= finishing warps: every item of the CTA but its last, while the next one is decoded =================
        pdl_wait();
        const int w = warp - kFirstDecoder - S::kDecoders;
        const uint32_t quarter_lanes = tmem + (static_cast<uint32_t>((w & 3) * 32) << 16);
        for (uint32_t item = first_item; item < last_item; ++item)
            finish_item(std::integral_constant<int, 4>{}, w, item, item - first_item, static_cast<int>(item == first_item ? spi - k0 : spi), quarter_lanes,
                        stage_base + S::kDecoders / 4 * 2 * kChunk * 128, &s_last[1], 5, 6);
    } else if (warp >= kFirstDecoder) {
        // ================= decoders: packed words -> A stages in tensor memory; then the epilogue of each item =================
        const int dec = warp - kFirstDecoder, group = dec >> 3, rows4 = (dec >> 2) & 1, quarter = dec & 3;   // quarter == warp & 3: the lanes it may access
        const LaneGeom<K> geom(lane);
        // this warp's two tiles of each row: half of a quad of four interleaved tiles
        const uint32_t* words = raw_base + rows4 * (256 * K) + (quarter >> 1) * (32 * K) + (quarter & 1) * 2;
        const int j2 = geom.i2 * 4, j1 = geom.i1 * 4, j0 = geom.i0 * 4;
        const uint32_t lanes = tmem + (static_cast<uint32_t>(quarter * 32) << 16);
        // What a stage costs a warp beside its eight tiles is kept to few instructions, since the integer pipe is what bounds the
        // loop: lane 0 waits for the packed words and the others for the A stage in ONE instruction, lanes 0 and 1 arrive at two
        // barriers in one, and what depends on the slot is stepped instead of computed.  Instructions per tile in all roles, 4 bits:
        // 54.9 -> 51.2 (43.1 are the decode); 16 rows 5120->2x25600, 3 bits, 80.1 -> 72.0 us; 64 rows 4096->14336, 4 bits,
        // 24.1 -> 21.7; expert block 37 / 256 tokens 165 -> 143 / 230 -> 213.  The loop unrolled over the ring of slots executes 49.6
        // but misses the instruction cache twice as often (78.8 us); two rows at a time, rolled: 53.0 and 74.9 us.
        const uint32_t wait_bar = smem_addr(lane == 0 ? raw_full : done), arrive_bar = smem_addr(lane == 0 ? raw_empty : full);
        const bool arrives = lane < 2;
        const uint32_t a_stages = lanes + S::kAccums * NT + rows4 * 32;
        // byte offsets of the slots' barriers (A stage, packed stage, the one this lane waits and arrives for); parity it waits for
        uint32_t at = group * 8, raw_at = group * 8, my_at = group * 8, par = lane == 0 ? 0u : 1u;
        const uint32_t my_end = lane == 0 ? S::kRaw * 8 : S::kSlots * 8;
        int it = group;
        auto decode_until = [&](const int end) {
#pragma unroll 1
            for (; it < end; it += S::kGroups) {
                // the packed stage has landed, and the MMAs that read this A stage last time are done
                if (!__all_sync(0xffffffffu, mbar_try_wait(wait_bar + my_at, par))) {
                    const bool ready = qmm_wait(lane == 0 ? &raw_full[my_at / 8] : &done[my_at / 8], par, &s_failed);
                    if (!__all_sync(0xffffffffu, ready)) break;
                }
                __syncwarp();
                // the stores below come after the products that read this A stage last
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t* rw = words + (S::kRaw == S::kSlots ? at : raw_at) * (kRawWords / 8);
                const uint32_t dst = a_stages + at * (kStageCols / 8);
                uint2 w2[4], w1[4], w0[4];
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const uint32_t* row = rw + r * (64 * K);
                    w2[r] = *reinterpret_cast<const uint2*>(row + j2);
                    w1[r] = *reinterpret_cast<const uint2*>(row + j1);
                    w0[r] = make_uint2(0, 0);
                    if constexpr (K >= 5) w0[r] = *reinterpret_cast<const uint2*>(row + j0);
                }
                auto tile_pair = [&](auto row) {
                    constexpr int r = decltype(row)::value;
                    uint32_t a0, a1, a2, a3;
                    lane_weights_exact<K, CB>(w2[r].x, w1[r].x, w0[r].x, geom.slack, a0, a1, a2, a3);
                    tmem_st_tile<r * 8>(dst, a0, a1, a2, a3);
                    lane_weights_exact<K, CB>(w2[r].y, w1[r].y, w0[r].y, geom.slack, a0, a1, a2, a3);
                    tmem_st_tile<r * 8 + (16 << 16)>(dst, a0, a1, a2, a3);
                };
                tile_pair(std::integral_constant<int, 0>{});
                tile_pair(std::integral_constant<int, 1>{});
                tile_pair(std::integral_constant<int, 2>{});
                tile_pair(std::integral_constant<int, 3>{});
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                mbar_arrive(arrives, arrive_bar + (S::kRaw == S::kSlots ? at : my_at));   // decoded; the packed words were consumed
                at += S::kGroups * 8;
                if constexpr (S::kRaw == S::kSlots) {
                    if (at >= S::kSlots * 8) { at -= S::kSlots * 8; par ^= 1u; }
                    my_at = at;
                } else {
                    if (at >= S::kSlots * 8) at -= S::kSlots * 8;
                    raw_at += S::kGroups * 8;
                    if (raw_at >= S::kRaw * 8) raw_at -= S::kRaw * 8;
                    my_at += S::kGroups * 8;
                    if (my_at >= my_end) { my_at -= my_end; par ^= 1u; }
                }
            }
        };
        auto finish = [&](uint32_t item, uint32_t seg, int stages) {
            if (seg == 0 || S::kFinishers < S::kDecoders) {
                pdl_wait();                                      // returns at once: the kernel before ended long ago
                if (tr && dec == 0 && lane == 0) tr[2] = global_ns();
            }
            finish_item(std::integral_constant<int, S::kDecoders>{}, dec, item, seg, stages, lanes, stage_base, &s_last[0], 1 + (dec >> 2), 8);
        };
        if constexpr (S::kFinishers < S::kDecoders) {
            // the finishing warps take every item but the last, which nothing is decoded behind
            decode_until(count);
            finish(last_item, last_item - first_item, last_stages);
        } else {
            int seg_begin = 0;
            for (uint32_t item = first_item, k_first = k0; seg_begin < count; ++item, k_first = 0) {
                const int seg_end = min(count, seg_begin + static_cast<int>(spi - k_first));
                decode_until(seg_end);
                finish(item, item - first_item, seg_end - seg_begin);
                seg_begin = seg_end;
            }
        }
        if (tr && dec == 0 && lane == 0) tr[5] = global_ns();
    } else if (warp == kWeightWarp) {
        // ================= weight producer: one bulk copy (8 tile rows x 8 tiles, contiguous) per stage =================
        if (elect_one()) {
            uint32_t item = first_item, par = 0;
            int done_before = 0, rem = min(count, static_cast<int>(spi - k0)), run = rem;
            const uint32_t* src = p.wq + quad_row_offset(8 * static_cast<int>(k0), qmm_item<NT>(p, item).wblock, p.in / 16, K);
            bool running = true;
            while (running) {
#pragma unroll 1
                for (int s = 0; s < S::kRaw; ++s) {
                    if (!qmm_wait(&raw_empty[s], par ^ 1u, &s_failed)) { running = false; break; }
                    mbar_expect_tx(&raw_full[s], kRawBytes);
                    bulk_copy_g2s(raw_base + s * kRawWords, src, kRawBytes, &raw_full[s]);
                    src += kRawWords;
                    if (--rem == 0) {
                        done_before += run;
                        if (done_before == count) { running = false; break; }
                        run = rem = min(count - done_before, static_cast<int>(spi));
                        src = p.wq + quad_row_offset(0, qmm_item<NT>(p, ++item).wblock, p.in / 16, K);
                    }
                }
                par ^= 1u;
            }
        }
    } else if (warp == kActWarp) {
        // ================= activation producer: tensor copies of [tokens, 64 inputs] =================
        if (elect_one()) {
            pdl_wait();
            uint32_t item = first_item, par = 0;
            int done_before = 0, rem = min(count, static_cast<int>(spi - k0)), x = static_cast<int>(k0) * kQmmStageIn;
            int run = rem;                                                       // stages of the current item here
            QmmItem info = qmm_item<NT>(p, item);
            int boxes = p.map_expert != nullptr ? (info.n + 15) >> 4 : 1;        // expert segments come in boxes of 16 rows
            uint32_t box_bytes = static_cast<uint32_t>(boxes * p.box_rows) * 256u;
            bool running = true;
            while (running) {
#pragma unroll 1
                for (int s = 0; s < S::kSlots; ++s) {
                    // the slot is free once the MMAs of the stage that used it last (kBSlots stages ago) are done
                    constexpr int kB = S::kBSlots;
                    const int before = (s + S::kSlots - kB) % S::kSlots;
                    unsigned char* dst = b_base + (s % kB) * S::kBSlotBytes;
                    const uint32_t before_par = s >= kB ? par : par ^ 1u;
                    if constexpr (NT > 64) {
                        // Only two slots fit beside 256 tokens, and a stage of products is shorter than a copy takes: each
                        // half of a slot is asked for as soon as its own products are done, and multiplied as soon as it
                        // lands (2000 rows 14336->4096, 3 bits: 283 -> 269 us).
                        if (!qmm_wait(&half[before], before_par, &s_failed)) { running = false; break; }
                        mbar_expect_tx(&full[s], box_bytes / 2);
                        tma_load_2d(dst, &xmap, x, info.brow, &full[s]);
                        if (!qmm_wait(&done[before], before_par, &s_failed)) { running = false; break; }
                        mbar_expect_tx(&full2[s], box_bytes / 2);
                        tma_load_2d(dst + S::kBHalfBytes, &xmap, x + 64, info.brow, &full2[s]);
                    } else {
                        if (!qmm_wait(&done[before], before_par, &s_failed)) { running = false; break; }
                        mbar_expect_tx(&full[s], box_bytes);
                        tma_load_2d(dst, &xmap, x, info.brow, &full[s]);
                        tma_load_2d(dst + S::kBHalfBytes, &xmap, x + 64, info.brow, &full[s]);
                        for (int b = 1; b < boxes; ++b) {
                            tma_load_2d(dst + b * 2048, &xmap, x, info.brow + b * 16, &full[s]);
                            tma_load_2d(dst + S::kBHalfBytes + b * 2048, &xmap, x + 64, info.brow + b * 16, &full[s]);
                        }
                    }
                    x += kQmmStageIn;
                    if (--rem == 0) {
                        done_before += run;
                        if (done_before == count) { running = false; break; }
                        run = rem = min(count - done_before, static_cast<int>(spi));
                        x = 0;
                        info = qmm_item<NT>(p, ++item);
                        if (p.map_expert != nullptr) { boxes = (info.n + 15) >> 4; box_bytes = static_cast<uint32_t>(boxes) * 4096u; }
                    }
                }
                par ^= 1u;
            }
            if (tr) tr[7] = global_ns();
        }
    } else if (warp == kMmaWarp) {
        // ================= MMA issuer =================
        if (elect_one()) {
            uint32_t item = first_item, par = 0, seg = 0, accumulate = 0, d = tmem;
            int left = count, rem = min(count, static_cast<int>(spi - k0));
            auto instr_desc = [&](uint32_t i) -> uint32_t {
                const int n16 = (qmm_item<NT>(p, i).n + 15) >> 4;
                return (1u << 4) /* D = fp32; A, B = fp16, K-major */ | (static_cast<uint32_t>(n16 * 2) << 17) /* N */ | ((128u >> 4) << 24) /* M */;
            };
            uint32_t idesc = instr_desc(item);
            const uint64_t b_desc0 = umma_desc(smem_addr(b_base));
            bool running = true;
            while (running) {
#pragma unroll
                for (int s = 0; s < S::kSlots; ++s) {
                    if (rem == 0) {
                        umma_commit(S::kFinishers < S::kDecoders && left == 0 ? &last_full : &accum_full[seg % S::kAccums]);   // accumulator of this item complete
                        if (left == 0) { running = false; break; }
                        ++seg;
                        // the accumulator of kAccums items ago has been read
                        if (seg >= S::kAccums && !qmm_wait(&accum_free[seg % S::kAccums], (seg / S::kAccums - 1) & 1u, &s_failed)) { running = false; break; }
                        d = tmem + (seg % S::kAccums) * NT;
                        idesc = instr_desc(++item);
                        rem = min(left, static_cast<int>(spi));
                        accumulate = 0;
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    }
                    if (!qmm_wait(&full[s], par, &s_failed)) { running = false; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t bd = b_desc0 + (s % S::kBSlots) * (S::kBSlotBytes >> 4);
#pragma unroll
                    for (int kk = 0; kk < 8; ++kk) {                             // 8 x 16 inputs: two halves of 64
                        if (NT > 64 && kk == 4) {
                            umma_commit(&half[s]);
                            if (!qmm_wait(&full2[s], par, &s_failed)) { running = false; break; }
                            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        }
                        umma_f16_ts(d, tmem + S::kAccums * NT + s * kStageCols + kk * 8, bd + (kk >> 2) * (S::kBHalfBytes >> 4) + (kk & 3) * 2, idesc,
                                    kk > 0 ? 1u : accumulate);
                    }
                    if (NT > 64 && !running) break;
                    accumulate = 1;
                    umma_commit(&done[s]);                                       // A stage and activation slot free once these MMAs have read them
                    --rem;
                    --left;
                }
                par ^= 1u;
            }
            if (s_failed) {
                umma_commit(&last_full);
                for (uint32_t a = 0; a < S::kAccums; ++a) umma_commit(&accum_full[a]);
            }
            if (tr) tr[3] = global_ns();
        }
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");   // every warp's last access before the memory is given back
    if (tr && threadIdx.x == 0) tr[6] = global_ns();
    if (s_failed) {
        // copies that were still in flight when a wait gave up must land before the CTA's shared memory is released
        const unsigned long long t0 = global_ns();
        while (global_ns() - t0 < 2000000ull) __nanosleep(1000);
    }
    __syncwarp();
    if (warp == kMmaWarp) tmem_dealloc(tmem, 512);
    if (threadIdx.x == 0 && s_failed) {
        pdl_wait();
        atomicExch(p.error, 3u);
    }
}

template <int K, int CB, int NT, bool FIN>
cudaError_t qmm_launch_shape(const CUtensorMap& map, const QmmArgs& p, int grid, cudaStream_t stream) {
    constexpr size_t smem = qmm_smem_bytes<K, NT, FIN>();
    auto kernel = qmm_kernel<K, CB, NT, FIN>;
    static PerDeviceOnce attribute;                         // once per kernel and device
    if (attribute.needed()) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        if (e != cudaSuccess) return e;
        attribute.mark();
    }
    return launch_dependent(kernel, dim3(static_cast<unsigned>(grid)), dim3(QmmShape<K, NT, FIN>::kThreads), smem, stream, map, p);
}

template <int K, int CB>
cudaError_t qmm_launch_form(const CUtensorMap& map, const QmmArgs& p, int grid, QmmForm form, cudaStream_t stream) {
    if (form == QmmForm::kSmall) return qmm_launch_shape<K, CB, 64, false>(map, p, grid, stream);
    if (form == QmmForm::kSmallItems) return qmm_launch_shape<K, CB, 64, true>(map, p, grid, stream);
    return qmm_launch_shape<K, CB, 256, false>(map, p, grid, stream);
}

}  // namespace

#ifdef B200_QMM_K

// One width per translation unit (kernels_qmm_k1.cu and its neighbours): they compile side by side, and the first call of a program
// loads the kernels of its width alone: 2.6 ms, 41 with all widths in one module.
template <int K>
cudaError_t qmm_launch_k(int cb, const CUtensorMap& map, const QmmArgs& p, int grid, QmmForm form, cudaStream_t stream) {
    if (cb == 0) return qmm_launch_form<K, 0>(map, p, grid, form, stream);
    if (cb == 1) return qmm_launch_form<K, 1>(map, p, grid, form, stream);
    return qmm_launch_form<K, 2>(map, p, grid, form, stream);
}
template cudaError_t qmm_launch_k<B200_QMM_K>(int, const CUtensorMap&, const QmmArgs&, int, QmmForm, cudaStream_t);

#else

namespace {

using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                              const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                              CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeFn encode_fn() {
    static EncodeFn fn = [] {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) != cudaSuccess || qres != cudaDriverEntryPointSuccess)
            return static_cast<EncodeFn>(nullptr);
        return reinterpret_cast<EncodeFn>(ptr);
    }();
    return fn;
}

// rotated activations [rows, in] fp16 as a 2-D tensor: boxes of 64 inputs x box_rows tokens, 128-byte swizzle
bool encode_rows(CUtensorMap* map, const __half* xhat, int in, int64_t rows, int box_rows) {
    EncodeFn encode = encode_fn();
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(in), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(in) * sizeof(__half)};
    const cuuint32_t box[2] = {64, static_cast<cuuint32_t>(box_rows)};
    const cuuint32_t elem[2] = {1, 1};
    return encode && encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<__half*>(xhat), dims, strides, box, elem,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

template <int K>
cudaError_t qmm_launch_k(int cb, const CUtensorMap& map, const QmmArgs& p, int grid, QmmForm form, cudaStream_t stream);

static cudaError_t qmm_dispatch(int k, int cb, const CUtensorMap& map, const QmmArgs& p, int grid, QmmForm form, cudaStream_t stream) {
    switch (k) {
        case 1: return qmm_launch_k<1>(cb, map, p, grid, form, stream);
        case 2: return qmm_launch_k<2>(cb, map, p, grid, form, stream);
        case 3: return qmm_launch_k<3>(cb, map, p, grid, form, stream);
        case 4: return qmm_launch_k<4>(cb, map, p, grid, form, stream);
        case 5: return qmm_launch_k<5>(cb, map, p, grid, form, stream);
        case 6: return qmm_launch_k<6>(cb, map, p, grid, form, stream);
        case 7: return qmm_launch_k<7>(cb, map, p, grid, form, stream);
        case 8: return qmm_launch_k<8>(cb, map, p, grid, form, stream);
        default: return cudaErrorInvalidValue;
    }
}

std::atomic<unsigned long long*> g_qmm_trace{nullptr};
static std::atomic<int> g_qmm_splits{0};                              // 0 = one wave of CTAs with equal runs of stages
void qmm_set_tuning(int splits) { g_qmm_splits = splits > 0 ? splits : 0; }

// CTAs of a launch over `items` items of `stages` stages: the same number for every item, or one wave of equal runs.
int64_t qmm_grid(const QmmPlan& plan, int64_t items, int64_t stages) {
    return plan.splits > 0 ? items * plan.splits : std::min<int64_t>(sm_count(), items * stages);
}
static size_t qmm_piece_count(int64_t items, int64_t grid) { return static_cast<size_t>(items < grid ? grid + items : 2 * grid); }

// at most one wave of CTAs shares items, so there are two parts per CTA or fewer, of at most 256 tokens (a forced split: any number)
size_t qmm_most_piece_bytes(int64_t rows) {
    if (g_qmm_splits.load() > 0) return size_t{1} << 60;
    return static_cast<size_t>(sm_count()) * 2 * static_cast<size_t>(std::min<int64_t>(256, (rows + 15) / 16 * 16)) * 128 * sizeof(float);
}

// How a batch is cut up: tokens per item and CTAs per item (or one wave of equal runs).  Microseconds fitted to 40000 measured launches
// (76 layers of 512 to 14336 inputs and 512 to 25600 outputs, 9 to 2000 rows, 1 to 6 and 8 bits, calls back to back with dependent
// launch), small and large tiles, items with CTAs of their own and equal runs each for themselves: a launch; a stage, mostly decode, with
// a share that grows with the tokens and one that grows with the SMs at work; an end of an item or of a part of one; parts that
// are written, counted and read again by the last CTA; and the next call's input rotation, whose CTAs lie on the SMs that the last
// wave leaves (eight each) and, beside a small tile's CTA of the form without finishing warps, one on the others: where they do not all
// find a place the next call starts later (100 rows 4096->1024: 96 CTAs 12.2 us, 144 CTAs 14.4).
// Over those 2311 batches the choice is 0.8 % above the best one measured on average (1.0 % over layers left out of the fit).  The
// estimate before it, fitted to an older form of the kernel and without the bits, was at 2.3 %: of 1014 batches of 26 layers that neither
// was fitted to, 217 are cut in another way now, 7 % faster on average; 12 lost more than 3 %, at most 10 % (24 rows 5888->4736, 4 bits,
// 13.4 -> 14.8 us).  Us, 4 bits: 90 rows 2304->8704 17.8 -> 14.4, 400 rows 640->10752 28.7 -> 23.7, 64 rows 4096->14336 21.55 ->
// 21.4, 512 rows 4096<->14336 (MLP block, 3 bits) 227 -> 224, 1999 rows 4096->6144 (group, 6 bits) 152 -> 143.5.
struct QmmCost { double launch, load, rotate, late, late_cta, stage_tile, stage, stage_load, end, end_tile, shared, shared_tile, part, part_tile; };
static constexpr QmmCost kQmmCost[2][2] = {                                  // [tiles above 64 tokens][equal runs]
    {{1.38, 0.967, 1.21, 1.03, 0.14, 0.056, 0.351, 0.118, 2.8, 0.717, 1.43, 0.521, 0.104, 0.248},
     {7.08, 0.138, 0.807, 0.047, 0.326, 0.0, 0.469, 0.0, 0.038, 1.45, 0.4, 1.72, 0.043, 0.306}},
    {{1.29, 2.21, 0.771, 0.732, 0.005, 0.029, 0.521, 0.036, 2.03, 1.86, 1.77, 0.249, 0.245, 0.18},
     {0.0, 0.0, 0.663, 5.88, 0.0, 0.08, 0.477, 0.0, 1.67, 1.1, 1.02, 0.093, 0.403, 0.11}}};

static double qmm_cost_us(int64_t sms, int64_t rows, int in, int k, int64_t items, int64_t stages, int tile, int64_t splits) {
    const QmmCost& c = kQmmCost[tile > 64][splits == 0];
    const int64_t grid = splits > 0 ? items * splits : std::min(sms, items * stages);
    const int64_t waves = (grid + sms - 1) / sms, run = splits > 0 ? (stages + splits - 1) / splits : (items * stages + grid - 1) / grid;
    const bool whole = splits == 0 && items % grid == 0;                     // equal runs of whole items
    const double parts = splits > 0 ? static_cast<double>(splits) : whole ? 1.0 : static_cast<double>(items < grid ? (grid + items - 1) / items + 1 : 2);
    const double ends = splits > 0 ? 1.0 : static_cast<double>(whole ? items / grid : (run + stages - 1) / stages + 1);
    const double bits = k == 4 || k == 8 ? 1.0 : k == 3 ? 1.09 : k < 3 ? 1.06 : 1.15;         // of a tile's decode
    const double t = tile / 64.0, load = static_cast<double>(std::min(grid, sms)) / static_cast<double>(sms);
    const int64_t busy = grid - (waves - 1) * sms, late = std::max<int64_t>(0, prepare_ctas(rows, in) - (sms - busy) * 8 - (tile <= 64 && splits > 0 ? busy : 0));
    return c.launch + c.load * load + c.rotate * 1e-6 * static_cast<double>(rows * in) + (late > 0 ? c.late : 0.0) + c.late_cta * late / sms +
           waves * (run * (c.stage_tile * t + bits * (c.stage + c.stage_load * load)) + ends * (c.end + c.end_tile * t)) +
           (parts > 1 ? c.shared + c.shared_tile * t + parts * (c.part + c.part_tile * t) : 0.0);
}

static QmmPlan make_qmm_plan(int in, int out, int k, int64_t rows, bool whole_items, int forced, int64_t sms) {
    QmmPlan plan{};
    const int64_t col_blocks = out / 128, stages = in / kQmmStageIn;
    // the items of one launch need an arrival counter each, and stages x CTAs must fit 32 bits: more rows go in passes
    const int64_t max_items = std::min<int64_t>(4000, (int64_t{1} << 31) / (stages * 1024));
    const int64_t max_tiles = std::max<int64_t>(1, max_items / col_blocks);
    plan.pass_rows = std::min(rows, max_tiles * 256);
    double best = 0;
    for (const int target : {16, 32, 48, 64, 96, 128, 192, 256}) {
        const int64_t tiles = (plan.pass_rows + target - 1) / target;
        if (tiles > max_tiles) continue;
        // equal tiles of whole sixteens: N of the MMA is a multiple of 16
        const int tile = static_cast<int>(((plan.pass_rows + tiles - 1) / tiles + 15) / 16 * 16);
        const int64_t items = tiles * col_blocks;
        auto consider = [&](int64_t splits) {
            // of whole sixteens, so that all rows with as many are cut alike: workspace sizes step by them
            const double t = qmm_cost_us(sms, (plan.pass_rows + 15) / 16 * 16, in, k, items, stages, tile, splits);
            if (best == 0 || t < best) { best = t; plan.tile_tokens = tile; plan.splits = static_cast<int>(splits); }
        };
        if (whole_items) consider(1);
        else if (forced) consider(std::max<int64_t>(1, std::min<int64_t>(forced, stages)));
        else {
            // whole items also in up to three waves: their stages are not cut, and nothing waits for parts
            for (int64_t splits = 1; splits <= stages && items * splits <= (splits == 1 ? 3 * sms : sms); ++splits) consider(splits);
            if (items * stages > sms) consider(0);
        }
    }
    const int64_t items = (plan.pass_rows + plan.tile_tokens - 1) / plan.tile_tokens * col_blocks;
    plan.piece_bytes = plan.splits == 1 ? 256 : qmm_piece_count(items, qmm_grid(plan, items, stages)) * plan.tile_tokens * 128 * sizeof(float);
    return plan;
}

// Weighing the choices takes a few microseconds of the host and a call asks twice: a thread remembers its last plans.
QmmPlan plan_qmm(int in, int out, int k, int64_t rows, bool whole_items) {
    struct Entry { int in, out, k, forced, sms; int64_t rows; bool whole; QmmPlan plan; };
    thread_local Entry cache[64] = {};
    const int forced = g_qmm_splits.load(), sms = sm_count();
    Entry& e = cache[(static_cast<unsigned>(in) / 128 * 7 + static_cast<unsigned>(out) / 128 * 3 + static_cast<unsigned>(rows)) % 64];
    if (e.in != in || e.out != out || e.k != k || e.rows != rows || e.whole != whole_items || e.forced != forced || e.sms != sms)
        e = {in, out, k, forced, sms, rows, whole_items, make_qmm_plan(in, out, k, rows, whole_items, forced, sms)};
    return e.plan;
}

cudaError_t launch_qmm(QmmArgs p, const __half* xhat, int k, int cb, const QmmPlan& plan, cudaStream_t stream) {
    if (p.in % 128 || p.out % 128 || p.rows <= 0 || p.rows > plan.pass_rows || p.groups < 1) return cudaErrorInvalidValue;
    CUtensorMap map;
    if (!encode_rows(&map, xhat, p.in, static_cast<int64_t>(p.groups) * p.rows, plan.tile_tokens)) return cudaErrorInvalidValue;
    p.tile_tokens = p.box_rows = plan.tile_tokens;
    p.tiles = (p.rows + plan.tile_tokens - 1) / plan.tile_tokens;
    p.items = p.tiles * (p.out / 128);
    p.trace = g_qmm_trace.load();
    const int64_t stages = p.in / kQmmStageIn, grid = qmm_grid(plan, p.items, stages);
    if (p.items * stages * grid >= (int64_t{1} << 32)) return cudaErrorInvalidValue;
    const QmmForm form = plan.tile_tokens > 64 ? QmmForm::kLarge : plan.splits > 0 ? QmmForm::kSmall : QmmForm::kSmallItems;
    return qmm_dispatch(k, cb, map, p, static_cast<int>(grid), form, stream);
}

size_t qmm_mapped_piece_bytes() { return static_cast<size_t>(sm_count()) * 2 * kQmmSegRows * 128 * sizeof(float); }

cudaError_t launch_qmm_mapped(QmmArgs p, const __half* xhat, int max_segments, int k, int cb, cudaStream_t stream) {
    if (p.in % 128 || p.map_blocks <= 0 || max_segments <= 0 || p.map_proj <= 0 || p.map_slots <= 0 || p.yhat == nullptr) return cudaErrorInvalidValue;
    const int64_t stages = static_cast<int64_t>(max_segments) * p.map_proj * p.map_blocks * (p.in / kQmmStageIn);
    if (stages * sm_count() >= (int64_t{1} << 32)) return cudaErrorInvalidValue;
    CUtensorMap map;
    constexpr int box = 16;      // segments are short: only the boxes that hold rows are fetched (the last may reach into the next segment's)
    if (!encode_rows(&map, xhat, p.in, static_cast<int64_t>(p.map_proj) * p.map_slots, box)) return cudaErrorInvalidValue;
    p.groups = 1; p.gcol0[0] = 0;
    p.tile_tokens = kQmmSegRows; p.box_rows = box;
    p.trace = nullptr;
    return qmm_dispatch(k, cb, map, p, sm_count(), QmmForm::kSmallItems, stream);
}

#endif

}  // namespace b200exl3
