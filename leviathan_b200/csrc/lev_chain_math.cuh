// One K-step of the one-column decode matvec in column-group arithmetic, shared by the persistent kernel
// (lev_chain.cu; 4-bit formats in the integer form at the end) and the one-launch kernel's single-column form (lev_dense.cu).
//
// The eight columns of an mma.m16n8k16 are four sub-block groups x two activation terms: the B fragments of
// 64-column chunk c are non-zero only in column group c, so one accumulator per lane collects four sub-blocks at
// once and the block scales are applied once per K-step by the lane that owns the sub-block.  Operands are
// shared-memory addresses: the step's packed bytes (see lev_stream.cu for the layout), the fragments of its four
// chunks ([term][quad lane][32 B] per chunk, 1 KB per K-step) and the sums that go with them.
#pragma once
#include "lev_stream_math.cuh"

namespace {

constexpr float kTerm1 = 4.8828125e-4f;  // 2^-11: weight of the second activation term

// Shared-memory loads and the tensor-core product as plain (non-volatile) asm: the compiler may
// interleave them freely inside a K-step.  What orders them against the waits is a data dependency: the
// caller passes every base address through order_after() once the wait that guards the bytes is over.
__device__ __forceinline__ void order_after(unsigned& addr) { asm volatile("" : "+r"(addr)::"memory"); }
__device__ __forceinline__ uint4 lds128(unsigned a) {
    uint4 v;
    asm("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ uint2 lds64(unsigned a) {
    uint2 v;
    asm("ld.shared.v2.u32 {%0, %1}, [%2];\n" : "=r"(v.x), "=r"(v.y) : "r"(a));
    return v;
}
__device__ __forceinline__ unsigned lds32(unsigned a) {
    unsigned v;
    asm("ld.shared.u32 %0, [%1];\n" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ unsigned lds16(unsigned a) {
    unsigned short v;
    asm("ld.shared.u16 %0, [%1];\n" : "=h"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ void mma(float* d, unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// first product of a chain: the accumulator input is the zero register
__device__ __forceinline__ void mma0(float* d, unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}

// products of 32 columns with s8 digits, exact in 32-bit integers: weights u8 or s8; the forms with a 0 start from zero
__device__ __forceinline__ void imma(int* d, unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void imma0(int* d, unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}
__device__ __forceinline__ void imma_s8(int* d, unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void imma0_s8(int* d, unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}
// 16 (q - 8) of the high / low nibbles q of four bytes, as signed bytes
__device__ __forceinline__ unsigned high_s8(unsigned w) { return (w & 0xF0F0F0F0u) ^ 0x80808080u; }
__device__ __forceinline__ unsigned low_s8(unsigned w) { return ((w << 4) & 0xF0F0F0F0u) ^ 0x80808080u; }
// byte k of w divided by 16, as a float: 2^19 + byte / 16, minus 2^19
__device__ __forceinline__ float byte_to_float_16th(unsigned w, unsigned k) {
    return __uint_as_float(__byte_perm(w, 0x49000000u, 0x7650u + k)) - 524288.0f;
}

// ---------------------------------------------------------------------------
// One column of the 4-bit formats runs in integers.  The activations of a K-step (256 columns) are one power of two
// times 31-bit integers, x = 2^(e - 30) * n with |x| < 2^e, and n is four signed bytes, n = sum d_i 256^i with d_i in
// [-128, 127]: the eight columns of an mma.m16n8k32 (u8 nibbles as they sit in the bytes, times s8 digits) are two
// chunk parities x four digits.  A nibble mask yields four weights where the f16 form's yields two, half as many
// products and fragment loads are issued, the sums are exact integers, and n keeps an activation to 2^-31 of its K-step's
// largest (the f16 form's two terms: 2^-22 of its own size, and nothing beyond the f16 range): error against f64 on normal
// activations 1e-7 (Q4_0) and 2e-7 (Q4_K) of the result where the f16 form shows 9e-7.  FFN set of the persistent kernel
// 32.3 -> 30.2 us, [12288 x 6144] Q4_K 14.7 -> 13.4 us.  lev_dense.cu stays with the f16 form: job lists of one column gained
// nothing (28.2 against 27.7 us for a MoE layer of one token, where two processes of one build differ by 1.5 %: the tables
// cost what a short share wins back), and plain products agree with their wider calls there.
// Table of a K-step: fragments [chunk][digit][quad lane][four mma registers] (1 KB); after all fragments kOneColAux bytes
// per K-step: Q4_K: activation sums of the eight sub-blocks (f32); then, both, the power of two (f32; NaN where an
// activation is not finite, so that the results are).  Q4_0 needs no sums: its products take q - 8 as it is.
// ---------------------------------------------------------------------------
template <int TYPE>
constexpr unsigned kOneColAux = TYPE == LEV_GGML_Q4_K ? 40u : TYPE == LEV_GGML_Q6_K ? 128u : 8u;
constexpr unsigned kZeroBytes = 528;   // zeros that stand in for the fragments of the other parity

// Builds the entries of one (chunk, quad lane): v[m] are the four activations of mma register m (chunk_col order).
// Sixteen neighbouring lanes hold one K-step; the whole warp takes part, `live` is uniform over a K-step.
// Returns true where an activation lies outside the f16 range or is not finite (what the f16 forms report).
template <int TYPE>
__device__ __forceinline__ bool int_tables(const float4* v, int chunk, int tt, bool live, uint4* frags, unsigned char* aux) {
    unsigned most = 0;
    bool bad = false;
#pragma unroll
    for (int m = 0; m < 4; m++) {
        const float f[4] = {v[m].x, v[m].y, v[m].z, v[m].w};
        unsigned mm = 0;
#pragma unroll
        for (int j = 0; j < 4; j++) mm = max(mm, __float_as_uint(f[j]) & 0x7fffffffu);
        // 65520 and above round to an f16 infinity; the high-nibble slots hold a sixteenth there
        bad |= mm >= __float_as_uint(chunk_hi<TYPE>(m) ? 65520.0f * 16.0f : 65520.0f);
        most = max(most, mm);
    }
#pragma unroll
    for (int d = 1; d < 16; d <<= 1) most = max(most, __shfl_xor_sync(0xffffffffu, most, d));
    int e = (int)(most >> 23) - 126;   // every |x| < 2^e
    if (e < -96) e = -96;
    const float f = __uint_as_float((unsigned)(157 - e) << 23);
    unsigned T[4][4];   // [mma register][digit]: four elements' bytes
    float plain[2] = {0.f, 0.f};
#pragma unroll
    for (int m = 0; m < 4; m++) {
        auto digits = [f](float x) { return ((unsigned)__float2int_rn(x * f) + 0x00808080u) ^ 0x00808080u; };
        const unsigned a = digits(v[m].x), b = digits(v[m].y), c = digits(v[m].z), d = digits(v[m].w);
        const unsigned ab0 = __byte_perm(a, b, 0x5140), ab2 = __byte_perm(a, b, 0x7362), cd0 = __byte_perm(c, d, 0x5140),
                       cd2 = __byte_perm(c, d, 0x7362);
        T[m][0] = __byte_perm(ab0, cd0, 0x5410);
        T[m][1] = __byte_perm(ab0, cd0, 0x7632);
        T[m][2] = __byte_perm(ab2, cd2, 0x5410);
        T[m][3] = __byte_perm(ab2, cd2, 0x7632);
        plain[m >> 1] += (v[m].x + v[m].z) + (v[m].y + v[m].w);
    }
    if (live) {
#pragma unroll
        for (int i = 0; i < 4; i++) frags[chunk * 16 + i * 4 + tt] = make_uint4(T[0][i], T[1][i], T[2][i], T[3][i]);
    }
    unsigned char* mine = aux + (size_t)(chunk >> 2) * kOneColAux<TYPE>;
    const int c = chunk & 3;
    if (TYPE == LEV_GGML_Q4_K) {
#pragma unroll
        for (int hf = 0; hf < 2; hf++) {
            float s = plain[hf];
            s += __shfl_xor_sync(0xffffffffu, s, 1);
            s += __shfl_xor_sync(0xffffffffu, s, 2);
            if (live && tt == 0) reinterpret_cast<float*>(mine)[c * 2 + hf] = s;
        }
    }
    if (live && c == 0 && tt == 0)
        *reinterpret_cast<float*>(mine + kOneColAux<TYPE> - 8) = most >= 0x7f800000u ? __uint_as_float(0x7fc00000u) : __uint_as_float((unsigned)(97 + e) << 23);
    return bad && live;
}

// what a lane needs of itself in every K-step, computed once
struct LaneConst {
    unsigned q_off;      // 16 * lane: this lane's 16 bytes of a chunk's weights
    unsigned hdr_off;    // 16 * g: header / scale row of row g
    unsigned x_off;      // Q6_K: fragments (term, t) inside a chunk's 256 bytes
    unsigned i_off;      // 4-bit formats: fragments (digit, t)
    unsigned grp;        // Q6_K: the chunk whose fragments this lane supplies (column group g / 2)
    unsigned t, g;
    unsigned sh16, shp;  // 16 * (t & 1); 16 * (t / 2)
    float place;         // what the digits of this lane's accumulator columns are worth: 1 or 65536
    unsigned zero_s;     // kZeroBytes zero bytes in shared memory

    __device__ __forceinline__ void init(int lane, unsigned zeros) {
        g = (unsigned)lane >> 2;
        t = (unsigned)lane & 3u;
        q_off = 16u * (unsigned)lane;
        hdr_off = 16u * g;
        x_off = ((g & 1u) * 4u + t) * 32u;
        i_off = ((g & 3u) * 4u + t) * 16u;
        grp = g >> 1;
        sh16 = 16u * (t & 1u);
        shp = 16u * (t >> 1);
        place = t & 1u ? 65536.0f : 1.0f;
        zero_s = zeros;
    }
};

// ---------------------------------------------------------------------------
// one K-step, one activation column.  The eight mma columns are (sub-block group s = 0..3) x (term):
// the B fragments of chunk c are non-zero in group c only, so after the K-step lane (g, t) holds, in
// accumulator columns 2t and 2t+1, the two terms of what chunk t contributed to rows g and g + 8.
// st / xk / ak: shared-memory addresses of the step's bytes, of the fragments and of the sums of its
// four chunks.  Lanes outside group c read the zero block instead of chunk c's fragments.
// ---------------------------------------------------------------------------
template <int TYPE>
__device__ __forceinline__ void chain_step(unsigned st, unsigned xk, unsigned ak, const LaneConst& L, float& ya, float& yb) {
    const unsigned t = L.t;
    const unsigned mine = xk + L.x_off;
    if (TYPE == LEV_GGML_Q4_K) {
        const uint4 h0 = lds128(st + L.hdr_off), h1 = lds128(st + 128 + L.hdr_off);
        // four accumulator chains (low / high nibbles x even / odd chunks): chunks write disjoint columns,
        // so the pairs are simply added afterwards
        float lo[4], hi[4], lo2[4], hi2[4];
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const uint4 q = lds128(st + 256 + c * 512 + L.q_off);
            const unsigned xa = L.grp == (unsigned)c ? mine + c * 256 : L.zero_s;
            const uint4 x0 = lds128(xa), x1 = lds128(xa + 16);
            const unsigned w0 = q.x, w1 = q.y, w2 = q.z, w3 = q.w;
            const unsigned w0s = w0 >> 8, w1s = w1 >> 8, w2s = w2 >> 8, w3s = w3 >> 8;
            float* Lo = c & 1 ? lo2 : lo;
            float* Hi = c & 1 ? hi2 : hi;
            if (c < 2) {
                mma0(Lo, w0 & 0x000F000Fu, w2 & 0x000F000Fu, w0s & 0x000F000Fu, w2s & 0x000F000Fu, x0.x, x0.y);
                mma0(Hi, w0 & 0x00F000F0u, w2 & 0x00F000F0u, w0s & 0x00F000F0u, w2s & 0x00F000F0u, x1.x, x1.y);
            } else {
                mma(Lo, w0 & 0x000F000Fu, w2 & 0x000F000Fu, w0s & 0x000F000Fu, w2s & 0x000F000Fu, x0.x, x0.y);
                mma(Hi, w0 & 0x00F000F0u, w2 & 0x00F000F0u, w0s & 0x00F000F0u, w2s & 0x00F000F0u, x1.x, x1.y);
            }
            mma(Lo, w1 & 0x000F000Fu, w3 & 0x000F000Fu, w1s & 0x000F000Fu, w3s & 0x000F000Fu, x0.z, x0.w);
            mma(Hi, w1 & 0x00F000F0u, w3 & 0x00F000F0u, w1s & 0x00F000F0u, w3s & 0x00F000F0u, x1.z, x1.w);
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
            lo[j] += lo2[j];
            hi[j] += hi2[j];
        }
        // this lane owns sub-blocks 2t (low nibbles of chunk t) and 2t+1 (high nibbles) of its two rows:
        // 6-bit scales and mins (rust/crates/lev-cpu/src/lib.rs:64-74)
        const unsigned sa = t < 2 ? (h0.y & 0x3F3F3F3Fu) : ((h0.w & 0x0F0F0F0Fu) | ((h0.y >> 2) & 0x30303030u));
        const unsigned sb = t < 2 ? (h1.y & 0x3F3F3F3Fu) : ((h1.w & 0x0F0F0F0Fu) | ((h1.y >> 2) & 0x30303030u));
        const unsigned ma = t < 2 ? (h0.z & 0x3F3F3F3Fu) : (((h0.w >> 4) & 0x0F0F0F0Fu) | ((h0.z >> 2) & 0x30303030u));
        const unsigned mb = t < 2 ? (h1.z & 0x3F3F3F3Fu) : (((h1.w >> 4) & 0x0F0F0F0Fu) | ((h1.z >> 2) & 0x30303030u));
        const unsigned sab = sa >> L.sh16, sbb = sb >> L.sh16, mab = ma >> L.sh16, mbb = mb >> L.sh16;
        const float dA = h2f_bits(h0.x & 0xffffu) * 16777216.0f, dB = h2f_bits(h1.x & 0xffffu) * 16777216.0f;  // d * 2^24
        const float dminA = h2f_bits(h0.x >> 16), dminB = h2f_bits(h1.x >> 16);
        const uint2 sxb = lds64(ak + 8 * t);  // activation sums of sub-blocks 2t, 2t+1
        const float sx0 = __uint_as_float(sxb.x), sx1 = __uint_as_float(sxb.y);
        const float pa = fmaf(byte_to_float(sab, 0), fmaf(lo[1], kTerm1, lo[0]), byte_to_float(sab, 1) * fmaf(hi[1], kTerm1, hi[0]));
        const float pb = fmaf(byte_to_float(sbb, 0), fmaf(lo[3], kTerm1, lo[2]), byte_to_float(sbb, 1) * fmaf(hi[3], kTerm1, hi[2]));
        const float qa = fmaf(byte_to_float(mab, 0), sx0, byte_to_float(mab, 1) * sx1);
        const float qb = fmaf(byte_to_float(mbb, 0), sx0, byte_to_float(mbb, 1) * sx1);
        ya = fmaf(dA, pa, fmaf(-dminA, qa, ya));
        yb = fmaf(dB, pb, fmaf(-dminB, qb, yb));
    } else if (TYPE == LEV_GGML_Q6_K) {
        // accumulator m: 16-value sub-block m of every chunk, starting at -32 * 2^-24 * (sum the tensor core sees)
        const uint4 k01 = lds128(ak + 32 * t), k23 = lds128(ak + 32 * t + 16);
        float acc[4][4] = {{__uint_as_float(k01.x), __uint_as_float(k01.y), __uint_as_float(k01.x), __uint_as_float(k01.y)},
                           {__uint_as_float(k01.z), __uint_as_float(k01.w), __uint_as_float(k01.z), __uint_as_float(k01.w)},
                           {__uint_as_float(k23.x), __uint_as_float(k23.y), __uint_as_float(k23.x), __uint_as_float(k23.y)},
                           {__uint_as_float(k23.z), __uint_as_float(k23.w), __uint_as_float(k23.z), __uint_as_float(k23.w)}};
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const uint4 q = lds128(st + 288 + c * 512 + L.q_off);
            const uint2 hq = lds64(st + 2336 + c * 256 + (L.q_off >> 1));
            const unsigned xa = L.grp == (unsigned)c ? mine + c * 256 : L.zero_s;
            const uint4 x0 = lds128(xa), x1 = lds128(xa + 16);
            const unsigned w0 = q.x, w1 = q.y, w2 = q.z, w3 = q.w;
            const unsigned w0s = w0 >> 8, w1s = w1 >> 8, w2s = w2 >> 8, w3s = w3 >> 8;
            const unsigned ha = hq.x, hb = hq.y;
            const unsigned ha_r2 = ha >> 2, ha_l2 = ha << 2, ha_l4 = ha << 4, ha_r4 = ha >> 4, ha_r6 = ha >> 6;
            const unsigned hb_r2 = hb >> 2, hb_l2 = hb << 2, hb_l4 = hb << 4, hb_r4 = hb >> 4, hb_r6 = hb >> 6;
            mma(acc[0], (w0 & 0x000F000Fu) | (ha & 0x00300030u), (w2 & 0x000F000Fu) | (hb & 0x00300030u),
                (w0s & 0x000F000Fu) | (ha_r2 & 0x00300030u), (w2s & 0x000F000Fu) | (hb_r2 & 0x00300030u), x0.x, x0.y);
            mma(acc[1], (w1 & 0x000F000Fu) | (ha_l2 & 0x00300030u), (w3 & 0x000F000Fu) | (hb_l2 & 0x00300030u),
                (w1s & 0x000F000Fu) | (ha_l4 & 0x00300030u), (w3s & 0x000F000Fu) | (hb_l4 & 0x00300030u), x0.z, x0.w);
            mma(acc[2], (w0 & 0x00F000F0u) | (ha & 0x03000300u), (w2 & 0x00F000F0u) | (hb & 0x03000300u),
                (w0s & 0x00F000F0u) | (ha_r2 & 0x03000300u), (w2s & 0x00F000F0u) | (hb_r2 & 0x03000300u), x1.x, x1.y);
            mma(acc[3], (w1 & 0x00F000F0u) | (ha_r4 & 0x03000300u), (w3 & 0x00F000F0u) | (hb_r4 & 0x03000300u),
                (w1s & 0x00F000F0u) | (ha_r6 & 0x03000300u), (w3s & 0x00F000F0u) | (hb_r6 & 0x03000300u), x1.z, x1.w);
        }
        // this lane owns sub-blocks 4t .. 4t+3 (chunk t) of its two rows: int8 scales = word t of the row's 16
        const unsigned scA = lds32(st + L.hdr_off + 4 * t) ^ 0x80808080u;
        const unsigned scB = lds32(st + 128 + L.hdr_off + 4 * t) ^ 0x80808080u;
        const float dA = h2f_bits(lds16(st + 256 + 2 * L.g)) * 16777216.0f, dB = h2f_bits(lds16(st + 272 + 2 * L.g)) * 16777216.0f;
        float pa = 0.f, pb = 0.f;
#pragma unroll
        for (int m = 0; m < 4; m++) {
            // float(byte + 128) - 128 without the conversion unit
            const float sA = __uint_as_float(__byte_perm(scA, 0x4B000000u, 0x7650u + m)) - 8388736.0f;
            const float sB = __uint_as_float(__byte_perm(scB, 0x4B000000u, 0x7650u + m)) - 8388736.0f;
            pa = fmaf(sA, fmaf(acc[m][1], kTerm1, acc[m][0]), pa);
            pb = fmaf(sB, fmaf(acc[m][3], kTerm1, acc[m][2]), pb);
        }
        ya = fmaf(dA, pa, ya);
        yb = fmaf(dB, pb, yb);
    } else {
        // Q4_0: accumulator b = 32-value block b of every chunk, starting at -8 * 2^-24 * (sum seen)
        const uint4 kk = lds128(ak + 16 * t);
        float a0[4] = {__uint_as_float(kk.x), __uint_as_float(kk.y), __uint_as_float(kk.x), __uint_as_float(kk.y)};
        float a1[4] = {__uint_as_float(kk.z), __uint_as_float(kk.w), __uint_as_float(kk.z), __uint_as_float(kk.w)};
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const uint4 q = lds128(st + c * 576 + 64 + L.q_off);
            const unsigned xa = L.grp == (unsigned)c ? mine + c * 256 : L.zero_s;
            const uint4 x0 = lds128(xa), x1 = lds128(xa + 16);
            const unsigned w0 = q.x, w1 = q.y, w2 = q.z, w3 = q.w;
            const unsigned w0s = w0 >> 8, w1s = w1 >> 8, w2s = w2 >> 8, w3s = w3 >> 8;
            mma(a0, w0 & 0x000F000Fu, w2 & 0x000F000Fu, w0s & 0x000F000Fu, w2s & 0x000F000Fu, x0.x, x0.y);
            mma(a1, w1 & 0x000F000Fu, w3 & 0x000F000Fu, w1s & 0x000F000Fu, w3s & 0x000F000Fu, x1.x, x1.y);
            mma(a0, w0 & 0x00F000F0u, w2 & 0x00F000F0u, w0s & 0x00F000F0u, w2s & 0x00F000F0u, x0.z, x0.w);
            mma(a1, w1 & 0x00F000F0u, w3 & 0x00F000F0u, w1s & 0x00F000F0u, w3s & 0x00F000F0u, x1.z, x1.w);
        }
        // this lane owns the two blocks of chunk t: fp16 d of (row g, blk 0 | blk 1), (row g+8, ...)
        const uint2 sc = lds64(st + t * 576 + 8 * L.g);
        const float dA0 = h2f_bits(sc.x & 0xffffu) * 16777216.0f, dA1 = h2f_bits(sc.x >> 16) * 16777216.0f;
        const float dB0 = h2f_bits(sc.y & 0xffffu) * 16777216.0f, dB1 = h2f_bits(sc.y >> 16) * 16777216.0f;
        ya = fmaf(dA0, fmaf(a0[1], kTerm1, a0[0]), fmaf(dA1, fmaf(a1[1], kTerm1, a1[0]), ya));
        yb = fmaf(dB0, fmaf(a0[3], kTerm1, a0[2]), fmaf(dB1, fmaf(a1[3], kTerm1, a1[2]), yb));
    }
}

// The same K-step in integers (tables of int_tables): 4-bit formats.
template <int TYPE>
__device__ __forceinline__ void int_step(unsigned st, unsigned xk, unsigned ak, const LaneConst& L, float& ya, float& yb) {
    static_assert(TYPE != LEV_GGML_Q6_K, "4-bit formats");
    const unsigned t = L.t;
    // fragments of the even / odd chunks, zeros for the lanes of the other parity
    const unsigned even = L.g < 4u ? xk + L.i_off : L.zero_s, odd = L.g < 4u ? L.zero_s : xk + 256u + L.i_off;
    if (TYPE == LEV_GGML_Q4_K) {
        const uint4 h0 = lds128(st + L.hdr_off), h1 = lds128(st + 128 + L.hdr_off);
        int lo[2][4], hi[2][4];   // [chunk pair]: low / high nibbles (these 16x)
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const uint4 q = lds128(st + 256 + c * 512 + L.q_off);
            const uint4 x = lds128((c & 1 ? odd : even) + (c >> 1) * 512);
            if (c & 1) {
                imma(lo[c >> 1], q.x & 0x0F0F0F0Fu, q.z & 0x0F0F0F0Fu, q.y & 0x0F0F0F0Fu, q.w & 0x0F0F0F0Fu, x.x, x.y);
                imma(hi[c >> 1], q.x & 0xF0F0F0F0u, q.z & 0xF0F0F0F0u, q.y & 0xF0F0F0F0u, q.w & 0xF0F0F0F0u, x.z, x.w);
            } else {
                imma0(lo[c >> 1], q.x & 0x0F0F0F0Fu, q.z & 0x0F0F0F0Fu, q.y & 0x0F0F0F0Fu, q.w & 0x0F0F0F0Fu, x.x, x.y);
                imma0(hi[c >> 1], q.x & 0xF0F0F0F0u, q.z & 0xF0F0F0F0u, q.y & 0xF0F0F0F0u, q.w & 0xF0F0F0F0u, x.z, x.w);
            }
        }
        // this lane holds two digits of chunk t / 2 (pair 0) and chunk 2 + t / 2 (pair 1): sub-blocks 2c (low nibbles)
        // and 2c + 1; their 6-bit scales (rust/crates/lev-cpu/src/lib.rs:64-74)
        const unsigned sa0 = (h0.y & 0x3F3F3F3Fu) >> L.shp, sa1 = ((h0.w & 0x0F0F0F0Fu) | ((h0.y >> 2) & 0x30303030u)) >> L.shp;
        const unsigned sb0 = (h1.y & 0x3F3F3F3Fu) >> L.shp, sb1 = ((h1.w & 0x0F0F0F0Fu) | ((h1.y >> 2) & 0x30303030u)) >> L.shp;
        // |digit sum| <= 32 * 240 * 128, 257 times that stays below 2^28
        auto val = [](int a, int b) { return (float)(a + 256 * b); };
        float pa = byte_to_float(sa0, 0) * val(lo[0][0], lo[0][1]), pb = byte_to_float(sb0, 0) * val(lo[0][2], lo[0][3]);
        pa = fmaf(byte_to_float_16th(sa0, 1), val(hi[0][0], hi[0][1]), pa);
        pb = fmaf(byte_to_float_16th(sb0, 1), val(hi[0][2], hi[0][3]), pb);
        pa = fmaf(byte_to_float(sa1, 0), val(lo[1][0], lo[1][1]), pa);
        pb = fmaf(byte_to_float(sb1, 0), val(lo[1][2], lo[1][3]), pb);
        pa = fmaf(byte_to_float_16th(sa1, 1), val(hi[1][0], hi[1][1]), pa);
        pb = fmaf(byte_to_float_16th(sb1, 1), val(hi[1][2], hi[1][3]), pb);
        // min term: this lane's share is sub-blocks 2t, 2t + 1
        const unsigned ma = t < 2 ? (h0.z & 0x3F3F3F3Fu) : (((h0.w >> 4) & 0x0F0F0F0Fu) | ((h0.z >> 2) & 0x30303030u));
        const unsigned mb = t < 2 ? (h1.z & 0x3F3F3F3Fu) : (((h1.w >> 4) & 0x0F0F0F0Fu) | ((h1.z >> 2) & 0x30303030u));
        const unsigned mab = ma >> L.sh16, mbb = mb >> L.sh16;
        const float dminA = h2f_bits(h0.x >> 16), dminB = h2f_bits(h1.x >> 16);
        const uint2 sxb = lds64(ak + 8 * t);
        const float sx0 = __uint_as_float(sxb.x), sx1 = __uint_as_float(sxb.y);
        const float qa = fmaf(byte_to_float(mab, 0), sx0, byte_to_float(mab, 1) * sx1);
        const float qb = fmaf(byte_to_float(mbb, 0), sx0, byte_to_float(mbb, 1) * sx1);
        const float scale = __uint_as_float(lds32(ak + 32)) * L.place;
        ya = fmaf(scale * h2f_bits(h0.x & 0xffffu), pa, fmaf(-dminA, qa, ya));
        yb = fmaf(scale * h2f_bits(h1.x & 0xffffu), pb, fmaf(-dminB, qb, yb));
    } else {
        // Q4_0: accumulators [chunk pair][block], 16 times the sums
        const float scale = __uint_as_float(lds32(ak)) * (0.0625f * L.place);
        const unsigned own = L.t >> 1;   // this lane holds two digits of chunk own (pair 0) and 2 + own (pair 1)
#pragma unroll
        for (int p = 0; p < 2; p++) {
            int acc[2][4];
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const uint4 q = lds128(st + (2 * p + j) * 576 + 64 + L.q_off);
                const uint4 x = lds128((j ? odd : even) + p * 512);
                if (j) {
                    imma_s8(acc[0], low_s8(q.x), low_s8(q.z), high_s8(q.x), high_s8(q.z), x.x, x.y);
                    imma_s8(acc[1], low_s8(q.y), low_s8(q.w), high_s8(q.y), high_s8(q.w), x.z, x.w);
                } else {
                    imma0_s8(acc[0], low_s8(q.x), low_s8(q.z), high_s8(q.x), high_s8(q.z), x.x, x.y);
                    imma0_s8(acc[1], low_s8(q.y), low_s8(q.w), high_s8(q.y), high_s8(q.w), x.z, x.w);
                }
            }
            // fp16 d of (row g, blk 0 | blk 1), (row g+8, ...) of the chunk
            const uint2 sc = lds64(st + (2 * p + own) * 576 + 8 * L.g);
            auto val = [](int a, int b) { return (float)(a + 256 * b); };
            const float pa = fmaf(h2f_bits(sc.x & 0xffffu), val(acc[0][0], acc[0][1]), h2f_bits(sc.x >> 16) * val(acc[1][0], acc[1][1]));
            const float pb = fmaf(h2f_bits(sc.y & 0xffffu), val(acc[0][2], acc[0][3]), h2f_bits(sc.y >> 16) * val(acc[1][2], acc[1][3]));
            ya = fmaf(scale, pa, ya);
            yb = fmaf(scale, pb, yb);
        }
    }
}

}  // namespace
