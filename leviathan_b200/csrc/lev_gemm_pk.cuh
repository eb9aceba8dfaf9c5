// Weight decode of the tensor-core GEMMs (lev_gemm_pk.cu): one 16-row tile x 64-column chunk of the fragment-major
// repack (layout: lev_stream.cu) to bf16 in the K-major 128-byte-swizzled tile that tcgen05.mma reads.
//
// A warp owns the tile: lane (g, t) holds bytes of rows g and g + 8 and writes 16 values of each.  Every value is
// formed exactly in f32 as the block decoders form it and rounded once to bf16.  What bounds the decode is issue
// slots, so a nibble becomes a value in a byte permute (it lands in the mantissa of 128.0 or 2^23) and one packed
// floating-point instruction for two values, scales are formed once per quad and handed round by shuffles, and odd
// rows write the other half of their values first: the eight lanes of a shared-memory wavefront (two rows x four
// 16-byte pieces, or four rows x two) then cover all 32 banks.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "lev_stream_math.cuh"

namespace {

__device__ __forceinline__ unsigned bf16_pair(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const unsigned*>(&v);
}
// two f32 operations in one instruction (each rounded as on its own)
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 v;
    asm("mov.b64 %0, {%1, %2};\n" : "=l"(v) : "f"(lo), "f"(hi));
    return v;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 v;
    asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(v) : "l"(a), "l"(b), "l"(c));
    return v;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 v;
    asm("add.rn.f32x2 %0, %1, %2;\n" : "=l"(v) : "l"(a), "l"(b));
    return v;
}
__device__ __forceinline__ unsigned bf16_pair2(f32x2 a) {
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;\n" : "=f"(lo), "=f"(hi) : "l"(a));
    return bf16_pair(lo, hi);
}
__device__ __forceinline__ void sts128(unsigned a, uint4 v) {
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};\n" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ void sts64(unsigned a, unsigned x, unsigned y) {
    asm volatile("st.shared.v2.u32 [%0], {%1, %2};\n" ::"r"(a), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ uint4 lds_v4(unsigned a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ uint2 lds_v2(unsigned a) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];\n" : "=r"(v.x), "=r"(v.y) : "r"(a));
    return v;
}
__device__ __forceinline__ unsigned lds_u16(unsigned a) {
    unsigned short v;
    asm volatile("ld.shared.u16 %0, [%1];\n" : "=h"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ int lds_s8(unsigned a) {
    int v;
    asm volatile("ld.shared.s8 %0, [%1];\n" : "=r"(v) : "r"(a));
    return v;
}
// byte I of w in the mantissa of 128.0 (128 + byte, for bytes below 128), or of 2^23
template <int I>
__device__ __forceinline__ float in128(unsigned w) { return __uint_as_float(__byte_perm(w, 0x43000000u, 0x7044u + (I << 8))); }
template <int I>
__device__ __forceinline__ float in2p23(unsigned w) { return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7650u + I)); }

// what a lane needs of itself, computed once
struct DecodeLane {
    unsigned q_off;   // its 16 bytes of a chunk
    unsigned g, t, odd;
    unsigned o0;      // byte offset (row g) of the piece it writes first; the others by exclusive or
    unsigned sh0;     // Q4_K: shift of the nibbles it writes first
    int src;          // first lane of its quad
};
template <int TYPE>
__device__ __forceinline__ DecodeLane decode_lane(int lane) {
    DecodeLane L;
    L.q_off = 16u * (unsigned)lane;
    L.g = (unsigned)lane >> 2;
    L.t = (unsigned)lane & 3u;
    L.odd = L.g & 1u;
    L.sh0 = 4u * L.odd;
    L.src = lane & ~3;
    if (TYPE == LEV_GGML_Q4_K) L.o0 = L.g * 128u + (((L.t + 4u * L.odd) ^ L.g) << 4);
    else L.o0 = L.g * 128u + (((4u * L.odd + (L.t >> 1)) ^ L.g) << 4) + 8u * (L.t & 1u);   // block 1 / sub-blocks 2, 3 first
    return L;
}

// Scales of the two chunks p and p + 2 of a K-step (one warp's share of it).  The four lanes of a quad work on the same
// two rows, so each forms a quarter of the products (Q4_K: one of the four sub-blocks; Q6_K: two of the eight) and
// hands them round by shuffles.
struct DecodeScales {
    float a[2][2];   // Q4_K: [row half] d * sc, -dmin * m of sub-block 4 (t >> 1) + 2 p + (t & 1);
                     // Q6_K: [chunk p / p + 2][row half] d * scale of sub-block t
};
template <int TYPE>
__device__ __forceinline__ void decode_scales(unsigned raw, int p, const DecodeLane& L, DecodeScales& S) {
    if (TYPE == LEV_GGML_Q4_K) {
        // 6-bit scales and mins (rust/crates/lev-cpu/src/lib.rs:64-74)
        const unsigned sel = 0x7650u + 2u * (unsigned)p + (L.t & 1u);
        auto byte = [sel](unsigned w) { return __uint_as_float(__byte_perm(w, 0x4B000000u, sel)) - 8388608.0f; };
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const uint4 h = lds_v4(raw + r * 128 + 16 * L.g);
            const unsigned sc = L.t < 2 ? (h.y & 0x3F3F3F3Fu) : ((h.w & 0x0F0F0F0Fu) | ((h.y >> 2) & 0x30303030u));
            const unsigned mn = L.t < 2 ? (h.z & 0x3F3F3F3Fu) : (((h.w >> 4) & 0x0F0F0F0Fu) | ((h.z >> 2) & 0x30303030u));
            S.a[r][0] = __fmul_rn(h2f_bits(h.x & 0xffffu), byte(sc));
            S.a[r][1] = __fmul_rn(-h2f_bits(h.x >> 16), byte(mn));
        }
    } else if (TYPE == LEV_GGML_Q6_K) {
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const float d = h2f_bits(lds_u16(raw + 256 + r * 16 + 2 * L.g));
#pragma unroll
            for (int cc = 0; cc < 2; cc++)
                S.a[cc][r] = __fmul_rn(d, (float)lds_s8(raw + r * 128 + 16 * L.g + 4 * (p + 2 * cc) + L.t));
        }
    }
}

// Q4_K: the chunk is sub-blocks 2c (low nibbles, 16-byte pieces 0..3 of the row) and 2c + 1 (high, pieces 4..7).
// value = d1 * q - m1 with d1 = d * sc, m1 = dmin * m; d1 * q is exact in f32 (11 + 6 + 4 bits), so the fused
// multiply-add rounds once like the reference's multiply-then-subtract (rust/crates/lev-cpu/src/lib.rs:110-130).
__device__ __forceinline__ uint4 q4k_piece(unsigned wa, unsigned wb, unsigned sh, float d1, float nm1) {
    const unsigned a = (wa >> sh) & 0x0F0F0F0Fu, b = (wb >> sh) & 0x0F0F0F0Fu;
    const f32x2 d2 = pack2(d1, d1), m2 = pack2(nm1, nm1), off = pack2(-8388608.0f, -8388608.0f);
    auto f = [&](float lo, float hi) { return bf16_pair2(fma2(d2, add2(pack2(lo, hi), off), m2)); };
    return make_uint4(f(in2p23<0>(a), in2p23<1>(a)), f(in2p23<2>(a), in2p23<3>(a)), f(in2p23<0>(b), in2p23<1>(b)),
                      f(in2p23<2>(b), in2p23<3>(b)));
}
template <int CC>
__device__ __forceinline__ void q4k_chunk(unsigned raw, int c, unsigned wt, const DecodeLane& L, const DecodeScales& S) {
    const uint4 q = lds_v4(raw + 256 + c * 512 + L.q_off);
    const int s0 = L.src + 2 * CC + (int)L.odd, s1 = s0 ^ 1;   // lanes with the scales of the piece written first / second
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const float d0 = __shfl_sync(0xffffffffu, S.a[r][0], s0), m0 = __shfl_sync(0xffffffffu, S.a[r][1], s0);
        const float d1 = __shfl_sync(0xffffffffu, S.a[r][0], s1), m1 = __shfl_sync(0xffffffffu, S.a[r][1], s1);
        const unsigned wa = r ? q.z : q.x, wb = r ? q.w : q.y;
        sts128(wt + r * 1024 + L.o0, q4k_piece(wa, wb, L.sh0, d0, m0));
        sts128(wt + r * 1024 + (L.o0 ^ 64u), q4k_piece(wa, wb, 4u - L.sh0, d1, m1));
    }
}

// Q4_0: two blocks of 32; lane t has bytes 4t..4t+3 of both: columns 4t.. (low) and 16 + 4t.. (high) of each.
// d * (128 + q) - 136 d = d * (q - 8): every step is exact (Sources/LeviathanCore/Q4.swift:54-69).
__device__ __forceinline__ void q40_piece(unsigned a, unsigned n4, f32x2 d2, f32x2 c2) {
    sts64(a, bf16_pair2(fma2(d2, pack2(in128<0>(n4), in128<1>(n4)), c2)), bf16_pair2(fma2(d2, pack2(in128<2>(n4), in128<3>(n4)), c2)));
}
__device__ __forceinline__ void q40_chunk(unsigned raw, int c, unsigned wt, const DecodeLane& L) {
    const uint4 q = lds_v4(raw + c * 576 + 64 + L.q_off);
    const uint2 sc = lds_v2(raw + c * 576 + 8 * L.g);
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const unsigned s = r ? sc.y : sc.x, w0 = r ? q.z : q.x, w1 = r ? q.w : q.y;
        const float da = h2f_bits(L.odd ? s >> 16 : s & 0xffffu), db = h2f_bits(L.odd ? s & 0xffffu : s >> 16);
        const unsigned a = L.odd ? w1 : w0, b = L.odd ? w0 : w1;
        const float ca = __fmul_rn(da, -136.0f), cb = __fmul_rn(db, -136.0f);
        const f32x2 da2 = pack2(da, da), db2 = pack2(db, db), ca2 = pack2(ca, ca), cb2 = pack2(cb, cb);
        const unsigned at = wt + r * 1024;
        q40_piece(at + L.o0, a & 0x0F0F0F0Fu, da2, ca2);
        q40_piece(at + (L.o0 ^ 32u), (a >> 4) & 0x0F0F0F0Fu, da2, ca2);
        q40_piece(at + (L.o0 ^ 64u), b & 0x0F0F0F0Fu, db2, cb2);
        q40_piece(at + (L.o0 ^ 96u), (b >> 4) & 0x0F0F0F0Fu, db2, cb2);
    }
}

// Q6_K: four sub-blocks of 16; lane t has elements 4t..4t+3 of each.  Level = 4 low bits (word m & 1, nibble m >> 1,
// byte {0, 2, 1, 3}[j]) | 2 high bits << 4 (at bit {4, 6, 2, 0, 8, 10, 12, 14}[2m + (j >> 1)] + 16 (j & 1)).
// value = (d * scale) * (level - 32) = ds * (128 + level) - 160 ds, exact (18 + 6 bits; Sources/LeviathanCore/Q6.swift:24-62).
template <int M>
__device__ __forceinline__ unsigned q6k_levels(unsigned w0, unsigned w1, unsigned h) {
    constexpr int kPos[8] = {4, 6, 2, 0, 8, 10, 12, 14};
    constexpr int p0 = kPos[2 * M], p1 = kPos[2 * M + 1];
    const unsigned w = M & 1 ? w1 : w0, n = M >= 2 ? (w >> 4) : w;
    const unsigned h0 = p0 >= 4 ? (h >> (p0 >= 4 ? p0 - 4 : 0)) : (h << (p0 >= 4 ? 0 : 4 - p0));
    const unsigned h1 = p1 >= 12 ? (h >> (p1 >= 12 ? p1 - 12 : 0)) : (h << (p1 >= 12 ? 0 : 12 - p1));
    return (n & 0x0F0F0F0Fu) | (h0 & 0x00300030u) | (h1 & 0x30003000u);
}
__device__ __forceinline__ void q6k_piece(unsigned a, unsigned lv, float ds, float c160) {
    const f32x2 d2 = pack2(ds, ds), c2 = pack2(c160, c160);
    sts64(a, bf16_pair2(fma2(d2, pack2(in128<0>(lv), in128<2>(lv)), c2)), bf16_pair2(fma2(d2, pack2(in128<1>(lv), in128<3>(lv)), c2)));
}
template <int CC>
__device__ __forceinline__ void q6k_chunk(unsigned raw, int c, unsigned wt, const DecodeLane& L, const DecodeScales& S) {
    const uint4 q = lds_v4(raw + 288 + c * 512 + L.q_off);
    const uint2 hq = lds_v2(raw + 2336 + c * 256 + (L.q_off >> 1));
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const unsigned w0 = r ? q.z : q.x, w1 = r ? q.w : q.y, h = r ? hq.y : hq.x;
        const unsigned lv[4] = {q6k_levels<0>(w0, w1, h), q6k_levels<1>(w0, w1, h), q6k_levels<2>(w0, w1, h), q6k_levels<3>(w0, w1, h)};
        const unsigned at = wt + r * 1024;
#pragma unroll
        for (int m = 0; m < 4; m++) {
            const float s = __shfl_sync(0xffffffffu, S.a[CC][r], L.src + (int)((unsigned)m ^ (2u * L.odd)));
            q6k_piece(at + (L.o0 ^ (32u * m)), L.odd ? lv[m ^ 2] : lv[m], s, __fmul_rn(s, -160.0f));
        }
    }
}

// chunk c = p + 2 CC of the K-step whose scales S holds
template <int TYPE, int CC>
__device__ __forceinline__ void decode_chunk(unsigned raw, int p, unsigned wt, const DecodeLane& L, const DecodeScales& S) {
    if (TYPE == LEV_GGML_Q4_K) q4k_chunk<CC>(raw, p + 2 * CC, wt, L, S);
    else if (TYPE == LEV_GGML_Q6_K) q6k_chunk<CC>(raw, p + 2 * CC, wt, L, S);
    else q40_chunk(raw, p + 2 * CC, wt, L);
}

}  // namespace
