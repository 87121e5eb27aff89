// Launch policy and K dispatch of the fused linear-layer kernels.
//
// The reference picks a split-K factor and tile width per shape for Apple GPUs
// (native/src/contracts.rs:1995-2012, native/src/linear.rs:899-919); only the meaning is kept
// (partials are summed in fp32 before the output rotation), the numbers are chosen for 148 SMs.
#include "common.cuh"
#include "kernels.h"

#include <algorithm>
#include <atomic>

namespace b200exl3 {

cudaError_t qmv_dispatch_k1(const QmvArgs&, int, bool, const QmvPlan&, cudaStream_t);
cudaError_t qmv_dispatch_k2(const QmvArgs&, int, bool, const QmvPlan&, cudaStream_t);
cudaError_t qmv_dispatch_k3(const QmvArgs&, int, bool, const QmvPlan&, cudaStream_t);
cudaError_t qmv_dispatch_k4(const QmvArgs&, int, bool, const QmvPlan&, cudaStream_t);
cudaError_t qmv_dispatch_k5(const QmvArgs&, int, bool, const QmvPlan&, cudaStream_t);
cudaError_t qmv_dispatch_k6(const QmvArgs&, int, bool, const QmvPlan&, cudaStream_t);
cudaError_t qmv_dispatch_k7(const QmvArgs&, int, bool, const QmvPlan&, cudaStream_t);
cudaError_t qmv_dispatch_k8(const QmvArgs&, int, bool, const QmvPlan&, cudaStream_t);

// Process-wide knobs; atomics because handles may be used from several threads while another thread sets an option.
static std::atomic<int> g_ctas_per_sm{2};   // CTAs per SM the grid is sized for (one wave)
static std::atomic<int> g_force_grid{0};    // > 0 overrides the grid size (tuning and tests)
static std::atomic<int> g_pdl{0};           // programmatic dependent launch between consecutive layers: 0 off, 1 late trigger, 2 early

bool pdl_enabled() { return g_pdl.load() != 0; }

int sm_count() {
    static std::atomic<int> cached[64];
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) {
        (void)cudaGetLastError();
        return kDefaultSmCount;
    }
    int n = cached[device].load(std::memory_order_relaxed);
    if (n > 0) return n;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || n <= 0) {
        (void)cudaGetLastError();
        return kDefaultSmCount;
    }
    cached[device].store(n, std::memory_order_relaxed);
    return n;
}

void qmv_set_tuning(int ctas_per_sm, int force_grid, int pdl) {
    if (ctas_per_sm > 0) g_ctas_per_sm = ctas_per_sm;
    g_force_grid = force_grid > 0 ? force_grid : 0;
    g_pdl = pdl > 0 ? pdl : 0;
}

static std::atomic<unsigned long long*> g_trace{nullptr};
void qmv_set_trace(unsigned long long* device_buffer) { g_trace = device_buffer; }

QmvPlan plan_qmv(int in, int out, int k, int64_t rows, bool full_grid) {
    QmvPlan plan{};
    plan.col_blocks = out / 128;
    const int tiles_k = in / 16;
    const int r = static_cast<int>(std::min<int64_t>(rows, kQmvMaxRows));
    const int forced = g_force_grid.load();
    const int64_t rb = tiles_k, rt = rb * plan.col_blocks;
    // CTAs of a layer, for `resident` of them per SM
    auto grid_for = [&](int resident) {
        const int64_t sms = sm_count();
        int64_t grid = forced > 0 ? forced : sms * resident;
        // the layer is dealt out in whole rows of 8 tiles: no more warps than rows
        grid = std::max<int64_t>(1, std::min(grid, rt / kQmvWarps));
        // a warp's range must not exceed one column block (it then touches at most two blocks)
        const int64_t min_warps = (rt + rb - 2) / (rb - 1) + 1;
        grid = std::max(grid, (min_warps + kQmvWarps - 1) / kQmvWarps);
        if (forced > 0 || full_grid) return static_cast<int>(grid);
        // Against that full grid: m whole CTAs for every column block.  Fewer CTAs share a block, none works on two, and a
        // warp that holds more rows rotates fewer 128-input blocks twice -- worth more than the last few idle SMs while a
        // layer is small.  Nanoseconds fitted to 168 sweeps (512..14336 inputs, 512..14336 outputs, 1, 2, 4 and 8 rows, 3, 4
        // and 6 bits; the choice is 1.5 % above the best grid measured, never more than 1.2 % above the full one): a
        // row of a warp, a row of an SM, a part of a block, a second CTA on an SM, a 128-input block a warp rotates.  The
        // row count is left out so that a row's sums are added in the same order in every batch of up to 8.
        // 4096->4096, 4 bits, 1 row: 12.4 -> 11.4 us; 4096->1024, 2 rows: 15.5 -> 12.5.
        // `full_grid`: the layers of a decode step and the expert block, whose prologues and neighbours fill the SMs that
        // this would leave idle (one token of the expert block 31.1 us with the full grid, 31.9 without).
        auto cost = [&](int64_t ctas, int64_t warp_rows, int64_t sm_rows, int64_t parts, int64_t spans) {
            return 181 * warp_rows + 42 * sm_rows + 149 * parts + (ctas > sms ? 407 : 0) + 628 * spans;
        };
        const int64_t full = grid, rows_w = (rt + full * kQmvWarps - 1) / (full * kQmvWarps);
        int64_t best = 59 + cost(full, rows_w, (full + sms - 1) / sms * rt / full, (full + plan.col_blocks - 1) / plan.col_blocks + 1, (rows_w + 6) / 8 + 1);
        for (int64_t m = 1; m <= 64 && m * plan.col_blocks <= sms * resident && m * kQmvWarps <= rb; ++m) {
            const int64_t ctas = m * plan.col_blocks, warps = m * kQmvWarps, n = (rb + warps - 1) / warps;
            // a warp's rows start at a 128-input block (8 rows) or divide one, or lie anywhere
            const int64_t spans = rb % warps == 0 && n % 8 == 0 ? n / 8 : rb % warps == 0 && 8 % n == 0 ? 1 : (n + 6) / 8 + 1;
            const int64_t t = cost(ctas, n, (ctas + sms - 1) / sms * rb / m, m, spans);
            if (t < best) { best = t; grid = ctas; }
        }
        return static_cast<int>(grid);
    };
    // Per warp: [ring of packed rows | rotated activations | staged result tile of its first block | of its second].  The
    // second tile is staged when the activations are no longer read, so with rows that come rotated it shares their place.
    auto layout = [&](int x_blocks, int tile_stride) {
        const int ring = qmv_chunk_rows(k) * qmv_slots(k) * 64 * k * static_cast<int>(sizeof(uint32_t));
        const int tile = r * tile_stride * static_cast<int>(sizeof(float));
        plan.tile_stride = tile_stride;
        plan.x_blocks = x_blocks;
        // rows eight words apart modulo 32 banks: the eight rows of a fragment load hit different banks
        plan.xs_stride = x_blocks * 128 + (plan.fused_rotation ? 0 : 8);
        const int xs = r * plan.xs_stride * static_cast<int>(sizeof(__half));
        plan.xs_offset = ring;
        plan.stage_offset = (ring + (plan.fused_rotation ? xs : std::max(xs, tile)) + 15) / 16 * 16;
        plan.stage2_offset = plan.fused_rotation ? plan.stage_offset + tile : plan.xs_offset;
        plan.warp_smem = (plan.stage_offset + (plan.fused_rotation ? 2 : 1) * tile + 15) / 16 * 16;
        plan.smem_bytes = static_cast<size_t>(plan.warp_smem) * kQmvWarps;
    };
    plan.fused_rotation = r <= kQmvFusedRows;
    // Two 8-row blocks need about twice the registers: one CTA per SM.  Up to 8 rows two CTAs share an SM where their shared
    // memory allows it (all widths up to 6 bits), because twice the warps decode; where it does not, the grid is one wave of
    // single CTAs (4096 -> 4096, 4 bits, 8 rows: 116 KB per CTA ran a grid for two per SM in two waves, 51 us).
    int resident = r <= 8 ? g_ctas_per_sm.load() : 1;
    if (plan.fused_rotation) layout(kQmvXBlocks, kQmvRedStride);
    else {
        layout(2, kQmvRedStride);
        // a tile without the padding costs a few bank conflicts once per warp, the second CTA is worth more
        if (resident > 1 && plan.smem_bytes > kQmvSharedSmemBytes) layout(1, 128);
        if (resident > 1 && plan.smem_bytes > kQmvSharedSmemBytes) { resident = 1; layout(2, kQmvRedStride); }
    }
    plan.grid = grid_for(resident);
    plan.max_pieces = static_cast<int>((plan.grid + plan.col_blocks - 1) / plan.col_blocks + 1);
    const int pdl = g_pdl.load();
    plan.pdl = pdl != 0;
    plan.pdl_early = pdl == 2;
    return plan;
}

size_t qmv_partial_bytes(const QmvPlan& plan, int out, int64_t rows) {
    const int64_t r = std::min<int64_t>(rows, kQmvMaxRows);
    return (static_cast<size_t>(plan.col_blocks) * plan.max_pieces * r * 128 * sizeof(float) + 255) / 256 * 256;
}

cudaError_t block_dispatch_k1(const QmvArgs&, int, bool, const BlockPlan&, cudaStream_t);
cudaError_t block_dispatch_k2(const QmvArgs&, int, bool, const BlockPlan&, cudaStream_t);
cudaError_t block_dispatch_k3(const QmvArgs&, int, bool, const BlockPlan&, cudaStream_t);
cudaError_t block_dispatch_k4(const QmvArgs&, int, bool, const BlockPlan&, cudaStream_t);
cudaError_t block_dispatch_k5(const QmvArgs&, int, bool, const BlockPlan&, cudaStream_t);
cudaError_t block_dispatch_k6(const QmvArgs&, int, bool, const BlockPlan&, cudaStream_t);
cudaError_t block_dispatch_k7(const QmvArgs&, int, bool, const BlockPlan&, cudaStream_t);
cudaError_t block_dispatch_k8(const QmvArgs&, int, bool, const BlockPlan&, cudaStream_t);

static std::atomic<int> g_block_cluster{0};
void block_set_tuning(int cluster) { g_block_cluster = cluster < -1 ? 0 : std::min(cluster, kBlockCluster); }

// Clusters of 1..8 CTAs that a B200 holds at one CTA per SM (a cluster lies inside one processing cluster of SMs); a constant, so
// that a layer's sums are added in the same order on every GPU.  A board whose SMs lie otherwise may hold fewer, and a layer then runs in
// two waves; a GPU test compares (b200exl3_plan_query, "clusters").
static constexpr int kResident[kBlockCluster] = {148, 74, 45, 33, 26, 22, 15, 15};

// Microseconds fitted to sweeps of 1..8 CTAs over 22 shapes (512..14336 inputs, 128..28672 outputs, 2, 3, 4 and 6 bits, one
// row; the choice is 1 % above the best measured on average): `rb` rows of 16 inputs over `parts` CTAs, a row of 16 inputs per
// warp, the sum over a cluster, a second wave of single CTAs.
static double block_us(int64_t rb, int parts, int cluster, int64_t waves, int k) {
    const bool even = k == 4 || k == 8;                      // the cheapest widths to decode
    const double warp_rows = 0.5 * (static_cast<double>(((rb + parts - 1) / parts + kBlockWarps - 1) / kBlockWarps) + static_cast<double>(rb) / (parts * kBlockWarps));
    return 0.7 + waves * (2.7 + (even ? 0.89 : 1.04) * warp_rows) + (cluster > 1 ? 1.0 + 0.04 * cluster : 0.0);
}

// Fitted to 159 measured calls (8 to 128 experts of 512 <-> 256 to 4096 <-> 14336, top 1 to 8, 1 to 300 slots, 1 to 8 bits; 2 %
// off on average): products that a wave of clusters holds, products that are dealt out over the grid by rows of 16 inputs per warp
// (a warp holds one column block's rows at most, so many slots of a large expert take more than a wave of CTAs), glue launches.
// Independent of the options that change how a product is cut, as the form decides what a workspace holds.
double moe_slots_us(int in, int hidden, int top_k, int k, int64_t slots) {
    const double row = k == 3 ? 1.12 : k == 5 || k == 6 ? 1.23 : k == 8 ? 1.07 : 1.01;
    const int64_t sms = sm_count();
    auto dealt = [&](int64_t rb, int64_t blocks) {
        const int64_t rt = rb * blocks, warps = (rt + rb - 2) / (rb - 1) + 1;
        const int64_t grid = std::max(std::max<int64_t>(1, std::min(2 * sms, rt / kQmvWarps)), (warps + kQmvWarps - 1) / kQmvWarps);
        const int64_t waves = (grid + 2 * sms - 1) / (2 * sms), rows = (rt + grid * kQmvWarps - 1) / (grid * kQmvWarps);
        return 6.9 + row * static_cast<double>(waves * rows) * (grid > sms ? 1.0 : 0.7);
    };
    const int64_t gu_rows = in / 16, gu_blocks = slots * 2 * hidden / 128, down_rows = hidden / 16, down_blocks = slots * in / 128;
    double us = 0.0, fused = 0.0;
    for (int n = 1; 2 * n <= kBlockCluster; ++n)
        if (gu_blocks / 2 <= kResident[2 * n - 1]) {
            const double t = block_us(gu_rows, n, 2 * n, 1, k);
            if (fused == 0.0 || t < fused) fused = t;
        }
    if (fused > 0.0) us += 1.06 * fused;
    else us += 3.3 + (gu_blocks <= kResident[0] ? 1.06 * block_us(gu_rows, 1, 1, 1, k) : dealt(gu_rows, gu_blocks));
    us += down_blocks <= kResident[0] ? 1.06 * block_us(down_rows, 1, 1, 1, k) : dealt(down_rows, down_blocks);
    if (top_k > kBlockCluster || down_blocks / top_k > kResident[top_k - 1]) us += 3.3;
    return us;
}

BlockPlan plan_block(int in, int out, int k, int64_t rows, BlockUse use, int top_k) {
    BlockPlan plan{};
    const int forced = g_block_cluster.load();
    const int64_t rb = in / 16, blocks = out / 128;
    if (rows > kBlockRows || forced < 0 || g_force_grid.load() > 0) return plan;
    const int ring = qmv_chunk_rows(k) * qmv_slots(k) * 64 * k * static_cast<int>(sizeof(uint32_t));
    auto lay_out = [&](int cluster, int parts, int64_t r) {
        // a part's rows may begin and end inside a block of 128 inputs
        const int nblk = static_cast<int>(std::min<int64_t>(in / 128, (rb + parts - 1) / parts / 8 + 2));
        plan.cluster = cluster;
        plan.parts = parts;
        plan.warp_smem = (std::max(ring, static_cast<int>(r) * kQmvRedStride * static_cast<int>(sizeof(float))) + 15) / 16 * 16;
        plan.xs_offset = plan.warp_smem * kBlockWarps;
        plan.xs_stride = nblk * 128 + 8;                     // rows four words apart modulo 32 banks
        plan.stage_offset = plan.xs_offset + (static_cast<int>(r) * plan.xs_stride * static_cast<int>(sizeof(__half)) + 15) / 16 * 16;
        // the parts of the rows that a CTA finishes (down product: its own sum, and the slots')
        plan.smem_bytes = static_cast<size_t>(plan.stage_offset) + ((r + cluster - 1) / cluster * cluster + 1) * 128 * sizeof(float);
        // One CTA per SM: where two fit, the hardware puts the CTAs of the next launch in pairs on the SMs that are free first, and the
        // launch takes as long as such a pair (4096->4096, 4 bits, clusters of 4: 9.5 us instead of 8.2).
        plan.smem_bytes = std::max(plan.smem_bytes, kQmvSharedSmemBytes + 4096);
        return plan.smem_bytes <= static_cast<size_t>(kQmvMaxSmemBytes);
    };
    int cluster = 1, parts = 1;
    int64_t clusters = blocks;
    if (use == BlockUse::kMapped) {
        plan.use = top_k > 0 || blocks <= kResident[0];
        cluster = parts = std::max(1, top_k);
    } else if (use == BlockUse::kDown) {
        if (top_k < 1 || top_k > kBlockCluster) return plan;
        cluster = top_k;
        clusters = blocks / top_k;
        plan.use = lay_out(cluster, 1, rows) && clusters <= kResident[top_k - 1];
    } else {
        // The cluster's cost against the other kernel's launch, its decode over all SMs and the parts of its blocks.  The row
        // count is left out, so that a row's sums are added in the same order in every batch of up to 8 (with 8 rows the other
        // kernel is further behind where the inputs are few, because its input rotation is a launch of its own).
        const int projections = use == BlockUse::kGateUp ? 2 : 1;
        const bool even = k == 4 || k == 8;                  // the cheapest widths to decode
        double best = forced > 0 || projections > 1 ? 1e30 : 7.0 + (even ? 0.00042 : 0.00048) * static_cast<double>(rb * blocks) + 0.004 * rb;
        for (int n = 1; n * projections <= kBlockCluster && n <= rb; ++n) {
            const int m = n * projections;
            const int64_t waves = m == 1 && blocks > kResident[0] ? 2 : 1;
            if (forced > 0 && projections == 1 ? m != forced : blocks / projections > waves * kResident[m - 1]) continue;
            if (!lay_out(m, n, projections > 1 ? 1 : kBlockRows)) continue;
            const double t = block_us(rb, n, m, waves, k);
            if (t < best) { best = t; cluster = m; parts = n; plan.use = true; }
        }
        clusters = blocks / projections;
    }
    plan.use = plan.use && lay_out(cluster, parts, rows);
    plan.grid = static_cast<int>(clusters) * cluster;
    const int pdl = g_pdl.load();
    plan.pdl = pdl != 0;
    plan.pdl_early = pdl == 2;
    return plan;
}

cudaError_t launch_block(QmvArgs args, int k, int cb, bool exact, const BlockPlan& plan, cudaStream_t stream) {
    if (!plan.use || args.rows <= 0 || args.rows > kBlockRows || (args.map_count != nullptr && args.map_early)) return cudaErrorInvalidValue;
    args.tiles_k = args.in / 16;
    args.trace = g_trace.load();
    args.cluster = plan.cluster;
    args.warp_smem = plan.warp_smem;
    args.xs_offset = plan.xs_offset;
    args.xs_stride = plan.xs_stride;
    args.stage_offset = plan.stage_offset;
    args.x_wide = args.x != nullptr && four_at_once(args.x, args.x_dtype) ? 1 : 0;
    args.pdl_early = plan.pdl_early ? 1 : 0;
    switch (k) {
        case 1: return block_dispatch_k1(args, cb, exact, plan, stream);
        case 2: return block_dispatch_k2(args, cb, exact, plan, stream);
        case 3: return block_dispatch_k3(args, cb, exact, plan, stream);
        case 4: return block_dispatch_k4(args, cb, exact, plan, stream);
        case 5: return block_dispatch_k5(args, cb, exact, plan, stream);
        case 6: return block_dispatch_k6(args, cb, exact, plan, stream);
        case 7: return block_dispatch_k7(args, cb, exact, plan, stream);
        case 8: return block_dispatch_k8(args, cb, exact, plan, stream);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_qmv(QmvArgs args, int k, int cb, bool exact, const QmvPlan& plan, cudaStream_t stream) {
    if (args.rows <= 0 || args.rows > kQmvMaxRows) return cudaErrorInvalidValue;
    args.tiles_k = args.in / 16;
    if (args.map_selected == nullptr) args.tiles_n = args.out / 16;   // the expert-mapped caller gives the bank's width
    args.max_pieces = plan.max_pieces;
    args.trace = g_trace.load();
    args.warp_smem = plan.warp_smem;
    args.xs_offset = plan.xs_offset;
    args.stage_offset = plan.stage_offset;
    args.stage2_offset = plan.stage2_offset;
    args.tile_stride = plan.tile_stride;
    args.x_blocks = plan.x_blocks;
    args.xs_stride = plan.xs_stride;
    args.pdl_early = plan.pdl_early ? 1 : 0;
    switch (k) {
        case 1: return qmv_dispatch_k1(args, cb, exact, plan, stream);
        case 2: return qmv_dispatch_k2(args, cb, exact, plan, stream);
        case 3: return qmv_dispatch_k3(args, cb, exact, plan, stream);
        case 4: return qmv_dispatch_k4(args, cb, exact, plan, stream);
        case 5: return qmv_dispatch_k5(args, cb, exact, plan, stream);
        case 6: return qmv_dispatch_k6(args, cb, exact, plan, stream);
        case 7: return qmv_dispatch_k7(args, cb, exact, plan, stream);
        case 8: return qmv_dispatch_k8(args, cb, exact, plan, stream);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace b200exl3
