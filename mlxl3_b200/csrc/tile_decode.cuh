// Register-level decode of one 16x16 EXL3 tile by one warp, shared by the fused small-batch kernel
// and the tensor-core prefill kernel.
//
// Lane L owns states 8L..8L+7 of the tile = elements (rows 2q+{0,1,8,9}, columns g and g+8) of the
// weight tile W[16 inputs, 16 outputs] (q = L%4, g = L/4), which is the A-fragment of mma.m16n8k16
// for W^T (reference: native/src/codec.rs:126-138).
#pragma once

#include "codec.cuh"

namespace b200exl3 {

// ---- hash of the eight states of a lane -------------------------------------------------------------

template <int CB>
__device__ __forceinline__ constexpr uint32_t hash_mul() { return CB == 0 ? 89226354u : (CB == 1 ? 0xcbac1fedu : 0x83dcd12du); }
template <int CB>
__device__ __forceinline__ constexpr uint32_t hash_add() { return CB == 0 ? 64248484u : 0u; }

// bits [O, O + 16) of v, O at most 16.  The left shift is spelled in PTX: written in C++, the pair of shifts takes as long as a
// shift and a mask (cycles per tile at 3 bits: the few-row loop 56.6 both, 49.8 like this; the many-row decoder's 58.7 and 51.0).
template <int O>
__device__ __forceinline__ uint32_t window(uint32_t v) {
    if constexpr (O == 0) return v & 0xffffu;
    else if constexpr (O == 16) return v >> 16;
    else {
        uint32_t d;
        asm("shl.b32 %0, %1, %2;" : "=r"(d) : "r"(v), "n"(16 - O));
        return d >> 16;
    }
}

// b[j] = state_j * M + C for the lane's states j = 0..7 (32-bit wrap-around).  (w0:w1:w2) are the
// stream words that end at the word holding the lane's last bit; `slack` bits of w2 lie past it.
template <int K, int CB>
__device__ __forceinline__ void lane_hashes(uint32_t w2, uint32_t w1, uint32_t w0, int slack, uint32_t (&b)[8]) {
    constexpr uint32_t M = hash_mul<CB>(), C = hash_add<CB>();
    if constexpr (K == 4 || K == 8) {
        uint32_t P[4];
        if constexpr (K == 4) {
            // states at bit offsets 0,4,...,28: P[p] = {offset 4p (state 7-p), offset 4p+16 (state 3-p)}
            P[0] = w2; P[1] = __funnelshift_r(w2, w1, 4); P[2] = __funnelshift_r(w2, w1, 8); P[3] = __funnelshift_r(w2, w1, 12);
        } else {
            // states at bit offsets 0,8,...,56: {0,16} {8,24} {32,48} {40,56} = states {7,5} {6,4} {3,1} {2,0}
            P[0] = w2; P[1] = __funnelshift_r(w2, w1, 8);
            P[2] = w1; P[3] = __funnelshift_r(w1, w0, 8);
        }
        constexpr uint32_t C2 = C + (C << 16);
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            const uint32_t hi = P[p] >> 16;
            const uint32_t bh = hi * M + C;
            const uint32_t t = P[p] * M + C2;
            uint32_t bl;                                   // t - (bh << 16) as one multiply-add
            asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(bl) : "r"(bh), "r"(0xffff0000u), "r"(t));
            if constexpr (K == 4) {
                b[7 - p] = bl; b[3 - p] = bh;
            } else {
                const int jl = p == 0 ? 7 : (p == 1 ? 6 : (p == 2 ? 3 : 2));
                b[jl] = bl; b[jl - 2] = bh;
            }
        }
    } else {
        // The states are 16-bit windows at bit offsets 0, K, .., 7K from the lane's end.  A few registers are funnelled out
        // of the stream words so that every window lies at an offset 0..16 of one of them; there it costs ONE instruction of
        // the logic pipe, the one that bounds the decode: nothing but a shift at offset 16, a mask at 0, and in between a left
        // shift, which the integer multiply-add pipe can take, followed by the right shift that drops what lies below.
        // Cycles per tile and scheduler against a shift and a mask per state, 16 warps, words in shared memory: the few-row
        // loop (two mma.sync a tile) 54.8 -> 47.5 at 2 bits, 56.6 -> 49.8 at 3, 59.9 -> 50.9 at 5, 59.1 -> 50.9 at 6; the
        // many-row decoder's loop (stores to tensor memory) 59.0 -> 52.1, 58.7 -> 51.0, 61.5 -> 54.1, 62.1 -> 53.6.
        uint32_t v[8];
        const uint32_t n = __funnelshift_r(w2, w1, slack);                       // offsets 0..31
        if constexpr (K <= 2) {
            v[7] = window<0>(n); v[6] = window<K>(n); v[5] = window<2 * K>(n); v[4] = window<3 * K>(n);
            v[3] = window<4 * K>(n); v[2] = window<5 * K>(n); v[1] = window<6 * K>(n); v[0] = window<7 * K>(n);
        } else if constexpr (K == 3) {
            const uint32_t m = __funnelshift_r(w2, w1, slack + 5);                  // offsets 5..36 (slack is at most 24)
            v[7] = window<0>(n); v[6] = window<3>(n);
            v[5] = window<1>(m); v[4] = window<4>(m); v[3] = window<7>(m); v[2] = window<10>(m); v[1] = window<13>(m); v[0] = window<16>(m);
        } else {
            const uint32_t n1 = __funnelshift_r(w1, w0, slack);                     // offsets 32..63
            if constexpr (K == 5) {
                const uint32_t m = __funnelshift_r(n, n1, 19);                      // offsets 19..50
                v[7] = window<0>(n); v[6] = window<5>(n); v[5] = window<10>(n); v[4] = window<15>(n);
                v[3] = window<1>(m); v[2] = window<6>(m); v[1] = window<11>(m); v[0] = window<16>(m);
            } else if constexpr (K == 6) {
                const uint32_t m = __funnelshift_r(n, n1, 14);                      // offsets 14..45
                v[7] = window<0>(n); v[6] = window<6>(n); v[5] = window<12>(n);
                v[4] = window<4>(m); v[3] = window<10>(m); v[2] = window<16>(m);
                v[1] = window<4>(n1); v[0] = window<10>(n1);
            } else {
                const uint32_t m = __funnelshift_r(n, n1, 19);                      // offsets 19..50
                const uint32_t l = __funnelshift_r(n1, w0 >> slack, 1);             // offsets 33..64
                v[7] = window<0>(n); v[6] = window<7>(n); v[5] = window<14>(n);
                v[4] = window<2>(m); v[3] = window<9>(m); v[2] = window<16>(m);
                v[1] = window<9>(l); v[0] = window<16>(l);
            }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) b[j] = v[j] * M + C;
    }
}

// Per-lane geometry of the stream words, constant for the whole kernel.
template <int K>
struct LaneGeom {
    int i2, i1, i0, slack;     // word indices inside a tile; bits of word i2 that lie past the lane's last bit
    __device__ __forceinline__ explicit LaneGeom(int lane) {
        constexpr int NW = 8 * K;
        const int end = 8 * K * (lane + 1);
        i2 = (end - 1) >> 5;
        slack = ((i2 + 1) << 5) - end;
        i1 = i2 >= 1 ? i2 - 1 : i2 - 1 + NW;
        i0 = i2 >= 2 ? i2 - 2 : i2 - 2 + NW;
    }
};

// The lane's eight weights as the reference's bit-exact fp16 values, packed as the four A-fragment
// registers of W^T: a0 = (out g; in 2q,2q+1), a1 = (out g+8; in 2q,2q+1), a2 = (out g; in 2q+8,2q+9),
// a3 = (out g+8; in 2q+8,2q+9).
template <int K, int CB>
__device__ __forceinline__ void lane_weights_exact(uint32_t w2, uint32_t w1, uint32_t w0, int slack, uint32_t& a0,
                                                   uint32_t& a1, uint32_t& a2, uint32_t& a3) {
    uint32_t b[8];
    lane_hashes<K, CB>(w2, w1, w0, slack, b);
    if constexpr (CB == 2) {
        const __half2 inv = __half2half2(__ushort_as_half(0x1eee));
        const __half2 bias = __half2half2(__ushort_as_half(0xc931));
        auto pair = [&](uint32_t x, uint32_t y) {
            uint32_t v = prmt(__dp4a(x, 0x01010101u, 0x6400u), __dp4a(y, 0x01010101u, 0x6400u), 0x5410);
            __half2 w = __hfma2(*reinterpret_cast<__half2*>(&v), inv, bias);
            return *reinterpret_cast<uint32_t*>(&w);
        };
        a0 = pair(b[0], b[1]); a1 = pair(b[4], b[5]); a2 = pair(b[2], b[3]); a3 = pair(b[6], b[7]);
    } else {
        // a weight is the fp16 sum of the two halves of its masked hash: two scalar adds that select their halves
        // (no repacking before them) and one merge -- one logic-pipe instruction less per pair than packing
        // (lo, lo) and (hi, hi) first
        auto pair = [&](uint32_t x, uint32_t y) {
            x = lop3_and_xor(x, 0x8fff8fffu, 0x3b603b60u);
            y = lop3_and_xor(y, 0x8fff8fffu, 0x3b603b60u);
            const __half2 hx = *reinterpret_cast<__half2*>(&x), hy = *reinterpret_cast<__half2*>(&y);
            const __half2 w = __halves2half2(__hadd_rn(__low2half(hx), __high2half(hx)), __hadd_rn(__low2half(hy), __high2half(hy)));
            return *reinterpret_cast<const uint32_t*>(&w);
        };
        a0 = pair(b[0], b[1]); a1 = pair(b[4], b[5]); a2 = pair(b[2], b[3]); a3 = pair(b[6], b[7]);
    }
}

}  // namespace b200exl3
