// Fused EXL3 linear layer for up to 8 activation rows with a cluster of CTAs per 128-column block, in ONE launch: input rotation
// (with the operator fused in front) -> trellis decode x activation product -> sum over the cluster -> output rotation.
//
// Reference behaviour replaced: the same as kernels_qmv_impl.cuh (native/shaders/_qmv_tile_kernel.metal with its prologue and
// epilogue kernels, native/src/linear.rs:847-996), whose tile decode, product and row epilogues are used here.
//
// Why beside that kernel, which deals ANY layer out evenly over the SMs: while a layer is small its time is a chain, not decode.
// Stamps of that kernel, 4096 -> 4096, 4 bits, one row, us after the layer before is done: rotated 0.8, tiles done 5.4 (eight
// warps per SM, two per scheduler: 66 cycles per tile, 45 with four), geometry of the block worked out 6.7, and 3.6 more for the
// parts that CTAs exchange through global memory (store, fence, count, fence, read); from 3 rows on a launch of its own rotates
// the input.  Here a column block belongs to a cluster and nothing else, so:
//  * the CTAs of a cluster split the block's inputs, the sixteen warps of a CTA split its rows; there is no geometry to work out;
//  * the CTA's inputs are rotated once, by all warps together, for any of the 1..8 rows (the other kernel: by every warp for
//    itself, or in a launch of its own);
//  * partial sums go to the CTA that finishes the row through distributed shared memory: one barrier instead of the five steps;
//  * output scales are asked for before the product.
// What bounds it: the chain (3.4 us of launch, rotation and output, 1.0 to 1.3 more for a cluster's sum), then the decode: 0.89 us for
// a row of 16 inputs per warp at 4 bits (16 warps per SM, 50 cycles per tile and scheduler), 1.04 at 2, 3, 5 and 6.
// Us per call back to back, 4 bits, other kernel -> this: one row 4096->4096 11.5 -> 7.8, 14336->4096 21.2 -> 16.9, 4096->14336
// 21.1 -> 17.9, 1024->1024 7.9 -> 4.5; 8 rows 15.9 -> 10.1, 26.4 -> 24.1, 28.1 -> 25.6, 11.4 -> 5.6; 3 rows 2176->1408, 5 bits,
// 11.9 -> 6.0.  One CTA per SM: with two, the next launch's CTAs pair up on the SMs that are free first (9.5 us instead of 8.2 for
// the first).  The next launch is let in once this one's inputs are there: it takes the SMs as they become free.
#pragma once

#include "kernels_qmv_impl.cuh"

namespace b200exl3 {

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// the address of a shared-memory word of this CTA in CTA `rank` of the cluster, and a store to such an address
__device__ __forceinline__ uint32_t cluster_addr(const void* p, int rank) {
    uint32_t d;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(smem_addr(p)), "r"(rank));
    return d;
}
__device__ __forceinline__ void cluster_store(uint32_t addr, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}

// Four columns of one input row after the operator fused in front of the layer, as the separate kernels compute them.
template <int kFused>
__device__ __forceinline__ void block_input(const QmvArgs& p, const void* x, int row, int col, float inv_rms, bool store_sum, __half (&v)[4]) {
    const int64_t at = static_cast<int64_t>(row) * p.in + col;
    const int pro = QMV_PRO(p);
    if (pro == 0) {
        if (p.x_wide) load4_as_half<true>(x, p.x_dtype, at, v);
        else load4_as_half<false>(x, p.x_dtype, at, v);
        return;
    }
    const uint2 xv = __ldcg(reinterpret_cast<const uint2*>(static_cast<const __half*>(x) + at));
    const __half2* xh = reinterpret_cast<const __half2*>(&xv);
    __half2 r[2];
    if (pro == 2) {
        const uint2 uv = __ldcg(reinterpret_cast<const uint2*>(p.pro_aux + at));
        const __half2* uh = reinterpret_cast<const __half2*>(&uv);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const float2 f = __half22float2(xh[j]);
            const __half2 sg = __floats2half2_rn(1.0f / (1.0f + expf(-f.x)), 1.0f / (1.0f + expf(-f.y)));
            r[j] = __hmul2_rn(__hmul2_rn(xh[j], sg), uh[j]);
        }
    } else {
        const uint2 wv = *reinterpret_cast<const uint2*>(p.pro_weight + col);
        const __half2* wh = reinterpret_cast<const __half2*>(&wv);
        __half2 s[2] = {xh[0], xh[1]};
        if (pro == 1 && p.pro_aux != nullptr) {
            const uint2 av = __ldcg(reinterpret_cast<const uint2*>(p.pro_aux + at));
            const __half2* ah = reinterpret_cast<const __half2*>(&av);
            s[0] = __hadd2_rn(s[0], ah[0]);
            s[1] = __hadd2_rn(s[1], ah[1]);
        }
        if (pro == 1 && store_sum && p.pro_sum != nullptr) {
            __align__(8) __half2 keep[2] = {s[0], s[1]};
            *reinterpret_cast<uint2*>(p.pro_sum + at) = *reinterpret_cast<const uint2*>(keep);
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const float2 f = __half22float2(s[j]);
            r[j] = __hmul2_rn(wh[j], __floats2half2_rn(f.x * inv_rms, f.y * inv_rms));
        }
    }
    v[0] = __low2half(r[0]); v[1] = __high2half(r[0]); v[2] = __low2half(r[1]); v[3] = __high2half(r[1]);
}

// Epilogue 4: the SwiGLU glue of the expert block (native/src/moe.rs:438-533; SiLU path, both rotations without intermediate
// rounding) on columns [col, col + 4) of a slot's gate and up products: they are rotated and scaled, multiplied, and rotated again
// as the input of the down product.  The arithmetic of glu_down_input_kernel, statement by statement.
__device__ __forceinline__ void block_glu(const QmvArgs& p, int64_t slot, int64_t expert, int col, const float4& graw, const float4& uraw, int lane) {
    const int hidden = p.map_blocks << 7;
    const float scale = had_scale();
    __align__(8) __half sg[4], su[4], sd[4];
    *reinterpret_cast<uint2*>(sg) = __ldg(reinterpret_cast<const uint2*>(p.glu_svh + (expert * 2) * hidden + col));
    *reinterpret_cast<uint2*>(su) = __ldg(reinterpret_cast<const uint2*>(p.glu_svh + (expert * 2 + 1) * hidden + col));
    *reinterpret_cast<uint2*>(sd) = __ldg(reinterpret_cast<const uint2*>(p.glu_down_suh + expert * hidden + col));
    float gv[4] = {round_half(graw.x), round_half(graw.y), round_half(graw.z), round_half(graw.w)};
    float uv[4] = {round_half(uraw.x), round_half(uraw.y), round_half(uraw.z), round_half(uraw.w)};
    warp_hadamard128<false, false>(gv, lane);
    warp_hadamard128<false, false>(uv, lane);
    float d[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float gate = round_half(__fmul_rn(__fmul_rn(gv[j], scale), __half2float(sg[j])));
        const float up = round_half(__fmul_rn(__fmul_rn(uv[j], scale), __half2float(su[j])));
        const float act = round_half(__fmul_rn(glu_silu(gate), up));
        d[j] = round_half(__fmul_rn(act, __half2float(sd[j])));
    }
    warp_hadamard128<false, false>(d, lane);
    __align__(8) __half h[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) h[j] = __float2half_rn(__fmul_rn(d[j], scale));
    *reinterpret_cast<uint2*>(p.glu_out + slot * hidden + col) = *reinterpret_cast<uint2*>(h);
}

// Epilogue 3, first half: a slot's columns [col, col + 4) of the down product rotated and scaled by the expert's output scales and
// the slot's routing weight (native/src/moe.rs:586-609, as finish_and_reduce_kernel computes it).
__device__ __forceinline__ void block_scale_slot(const QmvArgs& p, int slot, const __half* svh, const float4& a, int lane, float (&v)[4]) {
    __half h[4] = {__float2half_rn(a.x), __float2half_rn(a.y), __float2half_rn(a.z), __float2half_rn(a.w)};
    warp_hadamard128_f16(h, lane);
    const uint2 svw = *reinterpret_cast<const uint2*>(svh);
    const __half* sv = reinterpret_cast<const __half*>(&svw);
    if (p.epi_score_f32) {
        const float score = reinterpret_cast<const float*>(p.epi_scores)[slot];
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = __fmul_rn(__half2float(__hmul_rn(h[e], sv[e])), score);
    } else {
        const __half score = reinterpret_cast<const __half*>(p.epi_scores)[slot];
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = __half2float(__hmul_rn(__hmul_rn(h[e], sv[e]), score));
    }
}
// ... second half: added over the token's slots, in slot order, in the routing weights' type; `parked` [slots][128]
__device__ __forceinline__ void block_add_slots(const QmvArgs& p, int64_t at, int top_k, const float* parked) {
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
    for (int t = 0; t < top_k; ++t) {
        const float4 r = *reinterpret_cast<const float4*>(parked + t * 128);
        const float f[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            if (t == 0) acc[e] = f[e];
            else if (p.epi_score_f32) acc[e] = __fadd_rn(acc[e], f[e]);
            else acc[e] = __half2float(__hadd_rn(__float2half_rn(acc[e]), __float2half_rn(f[e])));
        }
    }
    if (p.epi_score_f32) {
        *reinterpret_cast<float4*>(reinterpret_cast<float*>(p.gy[0]) + at) = make_float4(acc[0], acc[1], acc[2], acc[3]);
    } else {
        __align__(8) __half o16[4] = {__float2half_rn(acc[0]), __float2half_rn(acc[1]), __float2half_rn(acc[2]), __float2half_rn(acc[3])};
        *reinterpret_cast<uint2*>(reinterpret_cast<__half*>(p.gy[0]) + at) = *reinterpret_cast<const uint2*>(o16);
    }
}

// kFused: 0 = no operator fused around the layer, 1 = those of a dense decoder (prologues 1..3, epilogues 1..2), 2 = the gate and up
// products of the expert block with the SwiGLU glue behind them (epilogue 4), 3 = its down product with the weighted sum over a
// token's slots behind it (epilogue 3).
template <int K, int CB, int MODE, int kFused>
__global__ void __launch_bounds__(kBlockWarps * 32, 1)
block_kernel(const __grid_constant__ QmvArgs p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int WARPS = kBlockWarps;
    constexpr int R = qmv_chunk_rows(K);                    // rows per bulk copy
    constexpr int SLOTS = qmv_slots(K);                     // chunks in flight per warp
    constexpr int kRowWords = 64 * K;
    constexpr uint32_t kRowBytes = kRowWords * 4;
    __shared__ __align__(8) uint64_t s_bar[WARPS][SLOTS];
    __shared__ float s_sq[2][WARPS];

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, q = lane & 3;
    const int rows = p.rows;
    const int m = p.cluster;
    const int rank = static_cast<int>(blockIdx.x) % m, unit = static_cast<int>(blockIdx.x) / m;
    // The cluster's CTAs share the inputs of one column block; of the expert block's gate and up products, of the same block of
    // both (first half: gate); of its down product they are the slots of one token, each with all inputs of its own expert.
    int cblock = unit, part = rank, parts = m;
    if (kFused == 2) {
        const int slot = unit / p.map_blocks;
        parts = m >> 1;
        cblock = (slot * 2 + rank / parts) * p.map_blocks + (unit - slot * p.map_blocks);
        part = rank % parts;
    }
    if (kFused == 3) {
        const int token = unit / p.map_blocks;
        cblock = (token * m + rank) * p.map_blocks + (unit - token * p.map_blocks);
        part = 0;
        parts = 1;
    }
    const int r0 = p.tiles_k * part / parts, n_rows = p.tiles_k * (part + 1) / parts - r0;
    const int w0 = r0 + n_rows * warp / WARPS, w1 = r0 + n_rows * (warp + 1) / WARPS;     // rows of 16 inputs of this warp
    const int kb0 = r0 >> 3, nblk = ((r0 + n_rows - 1) >> 3) - kb0 + 1;                    // 128-input blocks of this CTA

    unsigned char* mine = smem_raw + static_cast<size_t>(warp) * p.warp_smem;
    uint32_t* ring = reinterpret_cast<uint32_t*>(mine);                                   // SLOTS chunks; afterwards the warp's result tile
    __half* xs = reinterpret_cast<__half*>(smem_raw + p.xs_offset);                       // [rows][xs_stride] rotated inputs of this CTA
    float* sums = reinterpret_cast<float*>(smem_raw + p.stage_offset);                    // [rows this CTA finishes][cluster][128]
    uint64_t* bars = s_bar[warp];
    if (m > 1) cluster_arrive();                            // ... is running: its shared memory may be written once all have arrived
    if (lane == 0) {
#pragma unroll
        for (int i = 0; i < SLOTS; ++i) mbar_init(bars + i, 1);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncwarp();
    const bool tracing = p.trace != nullptr && threadIdx.x == 0;
    if (tracing) p.trace[blockIdx.x * 8 + 0] = global_ns();
    if (p.pdl_early) pdl_launch_dependents();

    // ---- which columns, activations and scales -------------------------------------------------------------------------
    int wblock = cblock, slot = 0, expert = 0;
    const void* x = p.x;
    const __half* xhat = p.xhat;
    const __half* suh = p.suh;
    if (p.map_selected != nullptr) {
        // The routes are another kernel's output.  They are read before the wait only where this library has launched a kernel in
        // between that was itself released by them (map_early).
        if (!p.map_early) pdl_wait();
        const int sp = cblock / p.map_blocks;
        slot = sp / p.map_proj;
        const int proj = sp - slot * p.map_proj;
        if (kFused == 0 && p.map_count != nullptr && slot >= *p.map_count) {      // no such slot: the whole cluster is done
            if (m > 1) cluster_wait();
            return;
        }
        expert = static_cast<int>(min(p.map_selected[slot], static_cast<uint32_t>(p.map_experts - 1)));   // unsigned: an id of 2^31 or more is clamped too
        wblock = proj * p.map_stride_blocks + expert * p.map_blocks + (cblock - sp * p.map_blocks);
        suh += (static_cast<int64_t>(expert) * p.map_proj + proj) * p.in;
        if (xhat != nullptr) xhat += static_cast<int64_t>(sp) * p.xhat_group_stride;
        else x = static_cast<const char*>(x) + static_cast<int64_t>(slot / p.map_top_k) * p.in * dtype_size(p.x_dtype);
    } else {
        const int grp = qmv_group_of(p, cblock);
        suh += static_cast<int64_t>(grp) * p.in;
        if (xhat != nullptr) xhat += grp * p.xhat_group_stride;
    }

    // ---- start streaming weights: they depend on nothing ----------------------------------------------------------------
    const char* src = reinterpret_cast<const char*>(p.wq + quad_row_offset(w0, wblock, p.tiles_k, K));
    int left = w1 - w0;                                     // rows not asked for yet
    auto refill = [&](int s) {
        const int n = min(R, left);
        if (lane == 0) {
            mbar_expect_tx(bars + s, n * kRowBytes);
            bulk_copy_g2s(ring + s * (R * kRowWords), src, n * kRowBytes, bars + s);
        }
        src += R * kRowBytes;
        left -= n;
    };
#pragma unroll
    for (int i = 0; i < SLOTS; ++i)
        if (left > 0) refill(i);
    // the output scales are read last: on their way into the caches by then
    const int block_col = kFused >= 2 ? (cblock % p.map_blocks) * 128 + lane * 4 : cblock * 128 + lane * 4;
    const __half* svh = p.svh + (kFused == 3 ? static_cast<int64_t>(expert) * (p.map_blocks << 7) : 0) + block_col;
    if (p.svh != nullptr && warp == 0 && (kFused == 3 || rank < rows)) asm volatile("prefetch.global.L1 [%0];" ::"l"(svh));
    if (p.map_selected == nullptr || p.map_early) pdl_wait();
    if (!p.pdl_early) pdl_launch_dependents();
    if (tracing) p.trace[blockIdx.x * 8 + 1] = global_ns();

    // ---- rotate the CTA's inputs into shared memory, a (row, 128-block) per warp at a time -------------------------------
    float inv_rms[2] = {0.0f, 0.0f};                        // fused RMSNorm (at most two rows)
    if (QMV_PRO(p) == 3) {
        // the layer before left the sum of squares of every 128-block: added in a fixed order
#pragma unroll
        for (int row = 0; row < 2; ++row)
            if (row < rows) {
                float acc = 0.0f;
                for (int b = lane; b < (p.in >> 7); b += 32) acc += __ldcg(p.pro_sumsq + row * (p.in >> 7) + b);
#pragma unroll
                for (int d = 16; d >= 1; d >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, d);
                inv_rms[row] = rsqrtf(acc / static_cast<float>(p.in) + p.pro_eps);
            }
    } else if (QMV_PRO(p) == 1) {
        // the CTA's warps share the whole row; every CTA adds it in the same order
        const __half* xr = static_cast<const __half*>(x);
#pragma unroll 1
        for (int row = 0; row < rows; ++row) {
            float acc = 0.0f;
            for (int i = static_cast<int>(threadIdx.x) * 8; i < p.in; i += WARPS * 256) {
                const int64_t at = static_cast<int64_t>(row) * p.in + i;
                const uint4 xv = __ldcg(reinterpret_cast<const uint4*>(xr + at));
                const __half2* xh = reinterpret_cast<const __half2*>(&xv);
                uint4 rv = make_uint4(0, 0, 0, 0);
                if (p.pro_aux != nullptr) rv = __ldcg(reinterpret_cast<const uint4*>(p.pro_aux + at));
                const __half2* rh = reinterpret_cast<const __half2*>(&rv);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 f = __half22float2(p.pro_aux != nullptr ? __hadd2_rn(xh[j], rh[j]) : xh[j]);
                    acc = fmaf(f.x, f.x, acc);
                    acc = fmaf(f.y, f.y, acc);
                }
            }
#pragma unroll
            for (int d = 16; d >= 1; d >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, d);
            if (lane == 0) s_sq[row][warp] = acc;
        }
        __syncthreads();
#pragma unroll
        for (int row = 0; row < 2; ++row)
            if (row < rows) {
                float acc = 0.0f;
                for (int w = 0; w < WARPS; ++w) acc += s_sq[row][w];
                inv_rms[row] = rsqrtf(acc / static_cast<float>(p.in) + p.pro_eps);
            }
    }
    if (xhat != nullptr) {
        for (int u = warp; u < rows * nblk; u += WARPS) {
            const int row = u / nblk, b = u - row * nblk;
            *reinterpret_cast<uint2*>(xs + row * p.xs_stride + b * 128 + lane * 4) =
                __ldcg(reinterpret_cast<const uint2*>(xhat + static_cast<int64_t>(row) * p.in + (kb0 + b) * 128 + lane * 4));
        }
    } else {
        // four units at a time: their loads are on their way together
        constexpr int kUnits = 4;
        const int units = rows * nblk;
#pragma unroll 1
        for (int u0 = warp; u0 < units; u0 += kUnits * WARPS) {
            __half v[kUnits][4];
            uint2 scale[kUnits];
#pragma unroll
            for (int i = 0; i < kUnits; ++i) {
                const int u = u0 + i * WARPS, row = u / nblk, col = (kb0 + u - row * nblk) * 128 + lane * 4;
                if (u < units) {
                    scale[i] = __ldg(reinterpret_cast<const uint2*>(suh + col));
                    block_input<kFused>(p, x, row, col, row == 0 ? inv_rms[0] : inv_rms[1], cblock == 0, v[i]);
                }
            }
#pragma unroll
            for (int i = 0; i < kUnits; ++i) {
                const int u = u0 + i * WARPS, row = u / nblk, b = u - row * nblk;
                if (u < units) {
                    const __half* sc = reinterpret_cast<const __half*>(&scale[i]);
                    __align__(8) __half h[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) h[j] = __hmul_rn(v[i][j], sc[j]);
                    warp_hadamard128_f16(h, lane);
                    *reinterpret_cast<uint2*>(xs + row * p.xs_stride + b * 128 + lane * 4) = *reinterpret_cast<const uint2*>(h);
                }
            }
        }
    }
    __syncthreads();
    if (tracing) p.trace[blockIdx.x * 8 + 2] = global_ns();

    // ---- decode x activations --------------------------------------------------------------------------------------------
    float acc[8][1][4];
#pragma unroll
    for (int t = 0; t < 8; ++t)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[t][0][i] = 0.0f;
    bool copy_lost = false;
    {
        const LaneGeom<K> geom(lane);
        // lanes whose activation row does not exist multiply the last row again: those columns of the product are never stored
        const uint32_t* xfrag = reinterpret_cast<const uint32_t*>(xs + min(g, rows - 1) * p.xs_stride + (w0 * 16 - kb0 * 128)) + q;
        int s = 0;
        uint32_t parity = 0;
#pragma unroll 1
        for (int r = w0; r < w1; r += R) {
            if (!copy_lost && !mbar_wait(bars + s, parity)) copy_lost = true;            // after a lost copy: no more waits
            const uint32_t* row_words = ring + s * (R * kRowWords);
            const int run = min(R, w1 - r);
#pragma unroll 1
            for (int j = 0; j < run; ++j) {
                const uint32_t p0 = xfrag[0], p1 = xfrag[4];
                uint32_t bx[1][4];
                if constexpr (MODE == 0) {
                    bx[0][0] = prmt(p0, p0, 0x1010); bx[0][1] = prmt(p0, p0, 0x3232);
                    bx[0][2] = prmt(p1, p1, 0x1010); bx[0][3] = prmt(p1, p1, 0x3232);
                } else {
                    bx[0][0] = p0; bx[0][1] = p1; bx[0][2] = 0; bx[0][3] = 0;
                }
                qmv_row<K, CB, 1, MODE, true>(row_words, geom, 0, 8, bx, acc);
                xfrag += 8;
                row_words += kRowWords;
            }
            __syncwarp();                                                                // every lane has read the slot
            if (left > 0) refill(s);
            if (++s == SLOTS) { s = 0; parity ^= 1u; }
        }
    }
    if (copy_lost && lane == 0) atomicExch(p.error, 1u);

    // ---- the warps' tiles go where their weights were; the CTA's sum over its warps, in warp order, to the CTA that finishes the row
    float* const tile = reinterpret_cast<float*>(mine);
#pragma unroll
    for (int t = 0; t < 8; ++t)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = 2 * q + (i & 1), col = t * 16 + g + ((i & 2) ? 8 : 0);
            if (row < rows) tile[row * kQmvRedStride + col] = acc[t][0][i];
        }
    __syncthreads();
    if (tracing) p.trace[blockIdx.x * 8 + 3] = global_ns();
    if (m > 1) cluster_wait();                              // all CTAs of the cluster run
    for (int i = threadIdx.x; i < rows * 128; i += WARPS * 32) {
        const float* t = reinterpret_cast<const float*>(smem_raw) + (i >> 7) * kQmvRedStride + (i & 127);
        const int stride = p.warp_smem / 4;
        float v[WARPS];
#pragma unroll
        for (int w = 0; w < WARPS; ++w) v[w] = t[w * stride];
#pragma unroll
        for (int w = 1; w < WARPS; ++w) v[0] = __fadd_rn(v[0], v[w]);
        if (kFused == 3 || m == 1) {
            sums[i] = v[0];
        } else if (kFused == 2) {
            cluster_store(cluster_addr(sums + rank * 128 + i, 0), v[0]);
        } else {
            // row r is finished by CTA r % m, which keeps the parts of its rows [r / m][part][128]
            const int row = i >> 7, to = row % m;
            cluster_store(cluster_addr(sums + ((row / m) * m + rank) * 128 + (i & 127), to), v[0]);
        }
    }
    if (kFused == 3) {
        // rotated, scaled by the expert's output scales and the slot's routing weight, then added over the token's slots in slot
        // order: the arithmetic and the order of finish_and_reduce_kernel
        __syncthreads();
        if (warp == 0) {
            const float4 a = *reinterpret_cast<const float4*>(sums + lane * 4);
            float v[4];
            block_scale_slot(p, slot, svh, a, lane, v);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float* to = sums + 128 + rank * 128 + lane * 4 + e;
                if (rank == 0) *to = v[e];
                else cluster_store(cluster_addr(to, 0), v[e]);
            }
        }
        __syncwarp();
        if (m > 1) { cluster_arrive(); cluster_wait(); }
        if (rank == 0 && warp == 0) {
            __syncwarp();
            block_add_slots(p, static_cast<int64_t>(unit / p.map_blocks) * (p.map_blocks << 7) + block_col, m, sums + 128 + lane * 4);
        }
    } else {
        if (m > 1) { __syncwarp(); cluster_arrive(); cluster_wait(); }
        else __syncthreads();
        if (kFused == 2) {
            if (rank == 0 && warp == 0) {
                float4 gu[2];
#pragma unroll
                for (int proj = 0; proj < 2; ++proj) {
                    const float* src4 = sums + proj * parts * 128 + lane * 4;
                    gu[proj] = *reinterpret_cast<const float4*>(src4);
                    for (int r = 1; r < parts; ++r) {
                        const float4 b = *reinterpret_cast<const float4*>(src4 + r * 128);
                        gu[proj].x = __fadd_rn(gu[proj].x, b.x); gu[proj].y = __fadd_rn(gu[proj].y, b.y);
                        gu[proj].z = __fadd_rn(gu[proj].z, b.z); gu[proj].w = __fadd_rn(gu[proj].w, b.w);
                    }
                }
                block_glu(p, slot, expert, block_col, gu[0], gu[1], lane);
            }
        } else if (rank + warp * m < rows) {
            const float* src4 = sums + warp * m * 128 + lane * 4;
            float4 a = *reinterpret_cast<const float4*>(src4);
#pragma unroll 1
            for (int r = 1; r < m; ++r) {
                const float4 b = *reinterpret_cast<const float4*>(src4 + r * 128);
                a.x = __fadd_rn(a.x, b.x); a.y = __fadd_rn(a.y, b.y); a.z = __fadd_rn(a.z, b.z); a.w = __fadd_rn(a.w, b.w);
            }
            qmv_finish_row<kFused>(p, cblock, rank + warp * m, a, lane);
        }
    }
    if (tracing) p.trace[blockIdx.x * 8 + 5] = global_ns();
}

template <int K, int CB, int MODE, int FUSED>
cudaError_t block_launch_one(const QmvArgs& p, const BlockPlan& plan, cudaStream_t stream) {
    auto kernel = block_kernel<K, CB, MODE, FUSED>;
    static PerDeviceOnce attribute;                         // once per kernel and device: allow the largest carve-out
    if (attribute.needed()) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kQmvMaxSmemBytes);
        if (e != cudaSuccess) return e;
        attribute.mark();
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>(plan.grid));
    cfg.blockDim = dim3(kBlockWarps * 32);
    cfg.dynamicSmemBytes = plan.smem_bytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(plan.cluster);
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = plan.pdl ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, p);
}

// Clusters of `cluster` CTAs that the current device holds at once, with as much shared memory as one CTA per SM may take.
template <int K, int CB, int MODE, int FUSED>
cudaError_t block_resident(int cluster, int* clusters) {
    auto kernel = block_kernel<K, CB, MODE, FUSED>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kQmvMaxSmemBytes);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>(cluster));
    cfg.blockDim = dim3(kBlockWarps * 32);
    cfg.dynamicSmemBytes = kQmvMaxSmemBytes;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(cluster);
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaOccupancyMaxActiveClusters(clusters, kernel, &cfg);
}

template <int K, int CB, int MODE>
cudaError_t block_launch_fused(const QmvArgs& p, const BlockPlan& plan, cudaStream_t stream) {
    if (p.epilogue == 4) return block_launch_one<K, CB, MODE, 2>(p, plan, stream);
    if (p.epilogue == 3) return block_launch_one<K, CB, MODE, 3>(p, plan, stream);
    return p.prologue != 0 || p.epilogue != 0 ? block_launch_one<K, CB, MODE, 1>(p, plan, stream) : block_launch_one<K, CB, MODE, 0>(p, plan, stream);
}

template <int K>
cudaError_t block_launch_k(const QmvArgs& p, int cb, bool exact, const BlockPlan& plan, cudaStream_t stream) {
    if (cb == 2) return block_launch_fused<K, 2, 1>(p, plan, stream);
    if (cb == 0) return exact ? block_launch_fused<K, 0, 1>(p, plan, stream) : block_launch_fused<K, 0, 0>(p, plan, stream);
    return exact ? block_launch_fused<K, 1, 1>(p, plan, stream) : block_launch_fused<K, 1, 0>(p, plan, stream);
}

}  // namespace b200exl3
