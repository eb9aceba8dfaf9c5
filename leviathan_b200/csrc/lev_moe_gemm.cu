// Grouped dequant-GEMM of the routed MoE at prefill-sized token counts (tcgen05 + TMEM), sm_100a: the Q4_0 weight rows of
// an expert are the MMA's M (128 per CTA), the tokens routed to it its N (up to 64 or 256 per job).
//
// An expert's weights are decoded for a few dozen tokens only, so the decode bounds the kernel (512 tokens of 128
// experts, top-8: issue slots 68 %, ALU 61 % used, tensor cores active 18 % of the time), and it is cut to the bone
// here: operands are f16.  A nibble masked in place under the exponent of 1024 is the f16 number 1024 + q (or 1024 +
// 16 q), one packed f16 operation makes it q - 8 exactly and one multiplies by the block's f16 scale, so two weights
// cost three instructions where bf16 through f32 (lev_gemm_pk.cuh) costs five, and the one rounding is to 11 bits
// instead of 8.  Activation rows are scaled by a power of two so that their largest element lies in [2^14, 2^15):
// they keep 11 bits wherever they matter (bf16 kept 8), nothing overflows, and the epilogue multiplies the power
// back.  Experts whose scales could overflow f16 in d * (q - 8) do not take this form.
//
// The pairs a mask yields are columns (4t, 4t + 2), (16 + 4t, ...), (4t + 1, 4t + 3), ...: the activation rows are
// stored in that order (k_rows_f16), which leaves the dot product as it is.
//
// Roles of the 31 warps as in lev_gemm_pk.cu, with three teams of eight decode warps; tiles come from the device-side
// job list.  A stage holds one 64-column chunk, or two where jobs are small (then a decode warp fills two chunks per
// handshake and the MMA warp waits once per eight MMAs).  gate_up tiles interleave 16 gate rows with the 16 up rows
// that go with them, so gelu(gate) * up is formed in the epilogue by one exchange between half-warps.
#include "lev_gemm_pk.cuh"
#include "lev_umma.cuh"
#include "lev_stream.h"

#include <type_traits>

namespace {

constexpr int MG_CHUNK_BYTES = 128 * 64 * 2;   // decoded weights of a 64-column chunk
constexpr int MG_RAW_SLOTS = 3;
constexpr int MG_TEAMS = 3;                    // teams of eight decode warps, one per 16-row tile
constexpr int MG_STAGES = 3;                   // 48 KB each in both forms (KC = 1: 256 tokens, KC = 2: 64)
// A team steps MG_TEAMS stages at a time and may pass over a K-step of the raw ring (a tile whose number of stages is odd
// ends in a K-step of one stage), where a wait by parity alone could be satisfied by the phase before.  With as many
// stages as teams the release of a stage says that all stages before it have been decoded: see the decode loop.
static_assert(MG_STAGES == MG_TEAMS && MG_RAW_SLOTS == 3, "the decode loop's waits rely on it");
static_assert(MG_STAGES * (MG_CHUNK_BYTES + 256 * 128) + MG_RAW_SLOTS * 8 * (int)kStepBytesQ4 + 1024 <= 225 * 1024, "shared memory of a CTA");
constexpr int MG_DECODE_WARPS = 8 * MG_TEAMS;
constexpr int MG_MMA_WARP = MG_DECODE_WARPS + 4, MG_RAW_WARP = MG_MMA_WARP + 1, MG_X_WARP = MG_MMA_WARP + 2;
constexpr int MG_THREADS = (MG_X_WARP + 1) * 32;
constexpr int MG_BOX_ROWS = 64;                // tokens of one TMA box

struct MgArgs {
    const unsigned char* packed;
    int spt, kt;            // 256-column K-steps per tile, 64-column chunks of the whole K
    int rows;               // gate_up: inter (gate rows, as many up rows); down: hidden
    int row_tiles;          // CTA tiles per job
    const int* njobs;
    const int4* jobs;       // {local expert, first grouped position, tokens, -}
    const float* scale;     // [position] power of two the activations were divided by
    const int* out_row;     // down: [position] row of out
    float* out;             // gate_up: [position][inter] gelu(gate) * up; down: [out_row][hidden]
    int job_tokens;
    int* status;
};

// 64-column chunk c of a 16-row tile to f16, columns in the order above.  Odd rows write block 1 first: see lev_gemm_pk.cuh.
__device__ __forceinline__ unsigned h2_add(unsigned a, unsigned b) {
    unsigned v;
    asm("add.rn.f16x2 %0, %1, %2;\n" : "=r"(v) : "r"(a), "r"(b));
    return v;
}
__device__ __forceinline__ unsigned h2_fma(unsigned a, unsigned b, unsigned c) {
    unsigned v;
    asm("fma.rn.f16x2 %0, %1, %2, %3;\n" : "=r"(v) : "r"(a), "r"(b), "r"(c));
    return v;
}
__device__ __forceinline__ unsigned h2_mul(unsigned a, unsigned b) {
    unsigned v;
    asm("mul.rn.f16x2 %0, %1, %2;\n" : "=r"(v) : "r"(a), "r"(b));
    return v;
}
__device__ __forceinline__ uint4 q40_word_f16(unsigned w, unsigned d2) {
    const unsigned ws = w >> 8;
    // 1024 + q - 1032; (1024 + 16 q) / 16 - 72
    auto lo = [d2](unsigned x) { return h2_mul(h2_add((x & 0x000F000Fu) | 0x64006400u, 0xE408E408u), d2); };
    auto hi = [d2](unsigned x) { return h2_mul(h2_fma((x & 0x00F000F0u) | 0x64006400u, 0x2C002C00u, 0xD480D480u), d2); };
    return make_uint4(lo(w), hi(w), lo(ws), hi(ws));
}
__device__ __forceinline__ void q40_chunk_f16(unsigned raw, int c, unsigned wt, const DecodeLane& L, unsigned o0) {
    const uint4 q = lds_v4(raw + c * 576 + 64 + L.q_off);
    const uint2 sc = lds_v2(raw + c * 576 + 8 * L.g);
    const unsigned sel0 = L.odd ? 0x3232u : 0x1010u, sel1 = L.odd ? 0x1010u : 0x3232u;   // the block's d, twice
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const unsigned s = r ? sc.y : sc.x, w0 = r ? q.z : q.x, w1 = r ? q.w : q.y;
        sts128(wt + r * 1024 + o0, q40_word_f16(L.odd ? w1 : w0, __byte_perm(s, 0u, sel0)));
        sts128(wt + r * 1024 + (o0 ^ 64u), q40_word_f16(L.odd ? w0 : w1, __byte_perm(s, 0u, sel1)));
    }
}

__device__ __forceinline__ void mbar_arrive_n(unsigned bar, unsigned n) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(n) : "memory");
}

// GATE_UP: the expert's gate_up tensor and the fused activation; else the down tensor.  KC: chunks per stage.
template <bool GATE_UP, int KC>
__global__ void __launch_bounds__(MG_THREADS, 1) k_moe_gemm(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ MgArgs A) {
    extern __shared__ unsigned char smem_dyn[];
    __shared__ __align__(8) unsigned long long full[MG_STAGES], empty[MG_STAGES];
    __shared__ __align__(8) unsigned long long full_raw[MG_RAW_SLOTS], empty_raw[MG_RAW_SLOTS], acc_full[2], acc_empty[2];
    __shared__ unsigned tmem_base_s;
    __shared__ int abort_s;
    constexpr unsigned kStep = kStepBytesQ4;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned smem = (smem_u32(smem_dyn) + 1023u) & ~1023u;
    const unsigned x_chunk = (unsigned)A.job_tokens * 128u;             // tokens of one chunk
    const unsigned stage_bytes = KC * (MG_CHUNK_BYTES + x_chunk);       // [KC] weights, [KC] tokens
    const unsigned raw_ring = smem + MG_STAGES * stage_bytes;

    if (threadIdx.x == 0) {
        abort_s = 0;
        for (int s = 0; s < MG_STAGES; s++) {
            mbar_init(smem_u32(&full[s]), 1 + 8);
            mbar_init(smem_u32(&empty[s]), 1);
        }
        for (int s = 0; s < MG_RAW_SLOTS; s++) {
            mbar_init(smem_u32(&full_raw[s]), 1);
            mbar_init(smem_u32(&empty_raw[s]), 8 * (4 / KC));
        }
        for (int s = 0; s < 2; s++) {
            mbar_init(smem_u32(&acc_full[s]), 1);
            mbar_init(smem_u32(&acc_empty[s]), 4);
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    }
    if (warp == MG_MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_base_s)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    pdl_launch_dependents();
    pdl_wait();   // the job list belongs to the launches before
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const unsigned tmem_base = tmem_base_s;
    volatile int* abort_flag = &abort_s;
    const int total = *A.njobs * A.row_tiles, first = (int)blockIdx.x, units = (int)gridDim.x;
    const int nu = (A.kt + KC - 1) / KC;   // stages of a tile
    const int tiles16 = A.rows >> 4;       // 16-row tiles of the gate rows / of the expert

    if (warp < MG_DECODE_WARPS) {
        // ---- decode: 16-row tile w & 7 of the CTA tile, every third stage from w >> 3 on ----
        const int tl = warp & 7;
        const DecodeLane L = decode_lane<LEV_GGML_Q4_0>(lane);
        const unsigned o0 = L.g * 128u + (((L.t + 4u * L.odd) ^ L.g) << 4);
        Ring st(MG_STAGES), raw(MG_RAW_SLOTS);
        int u = warp >> 3;                     // stage inside the tile
        st.step(u);
        const unsigned wt0 = smem + (unsigned)tl * 2048u, raw0 = raw_ring + (unsigned)tl * kStep;
        bool ok = true;
        constexpr int UPG = 4 / KC;            // stages of a 256-column K-step
        int at = 0;                            // K-step (of the tile) the raw ring stands at
        for (int tile = first; tile < total && ok; tile += units) {
            const int rt = tile % A.row_tiles;
            const bool live = (GATE_UP ? rt * 4 + (tl >> 1) : rt * 8 + tl) < tiles16;
            for (; u < nu; u += MG_TEAMS) {
                raw.step(u / UPG - at);
                at = u / UPG;
                // The stage first: its release means that every stage up to the one MG_STAGES before has been decoded, so
                // the K-step that held this raw slot before has landed, and the parity below can only mean this one.
                ok &= pk_wait(smem_u32(&empty[st.s]), st.ph ^ 1u, abort_flag);
                ok = __all_sync(0xffffffffu, pk_wait(smem_u32(&full_raw[raw.s]), raw.ph, abort_flag) & ok);
                if (!ok) break;
                const unsigned src = raw0 + (unsigned)raw.s * (8u * kStep);
                const int c = (u % UPG) * KC;
                const unsigned wt = wt0 + (unsigned)st.s * stage_bytes;
                if (live) {
                    q40_chunk_f16(src, c, wt, L, o0);
                    if (KC == 2) q40_chunk_f16(src, c + 1, wt + MG_CHUNK_BYTES, L, o0);
                }
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(smem_u32(&full[st.s]));
                    // one release per stage of the K-step; the tile's last stage also gives those that do not exist
                    mbar_arrive_n(smem_u32(&empty_raw[raw.s]), u == nu - 1 ? UPG - u % UPG : 1);
                }
                st.step(MG_TEAMS);
            }
            ok = __all_sync(0xffffffffu, ok);
            u -= nu;
            at -= A.spt;
        }
    } else if (warp < MG_MMA_WARP) {
        // ---- epilogue: lane = weight row, columns = tokens ----
        const int quarter = warp & 3;
        Ring ac(2);
        for (int tile = first; tile < total; tile += units) {
            const int rt = tile % A.row_tiles;
            const int4 job = __ldcg(A.jobs + tile / A.row_tiles);
            const int row = GATE_UP ? (rt * 4 + quarter) * 16 + (lane & 15) : rt * 128 + quarter * 32 + lane;
            const bool live = row < A.rows;
            if (!__all_sync(0xffffffffu, pk_wait(smem_u32(&acc_full[ac.s]), ac.ph, abort_flag))) break;
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const unsigned src = tmem_base + ((unsigned)(quarter * 32) << 16) + (unsigned)ac.s * 256u;
#pragma unroll 1
            for (int c = 0; c < job.z; c += 16) {
                const int mine = c + (lane & 15) < job.z ? job.y + c + (lane & 15) : job.y;   // this lane's column: its position,
                const float sc = __ldcg(A.scale + mine);                                     // scale and output row
                const int orow = GATE_UP ? mine : __ldcg(A.out_row + mine);
                unsigned v[16];
                tmem_ld16(src + (unsigned)c, v);
                asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
                if (GATE_UP) {
                    // lanes 0..15 hold gate rows, 16..31 the up rows that go with them: the lower half takes columns
                    // c .. c + 7, the upper half c + 8 .. c + 15
                    const bool up = lane >= 16;
#pragma unroll
                    for (int q = 0; q < 8; q++) {
                        const float got = __shfl_xor_sync(0xffffffffu, __uint_as_float(up ? v[q] : v[8 + q]), 16);
                        const float g0 = up ? got : __uint_as_float(v[q]), u0 = up ? __uint_as_float(v[8 + q]) : got;
                        const int col = q + (up ? 8 : 0);
                        const float s = __shfl_sync(0xffffffffu, sc, col);
                        if (live && c + col < job.z) A.out[(int64_t)(job.y + c + col) * A.rows + row] = gelu_tanh_up(g0 * s, u0 * s);
                    }
                } else {
#pragma unroll
                    for (int q = 0; q < 16; q++) {
                        const float s = __shfl_sync(0xffffffffu, sc, q);
                        const int o = __shfl_sync(0xffffffffu, orow, q);
                        if (live && c + q < job.z) A.out[(int64_t)o * A.rows + row] = __uint_as_float(v[q]) * s;
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&acc_empty[ac.s]));
            ac.step(1);
        }
    } else if (warp == MG_MMA_WARP) {
        // ---- MMA issue (see lev_gemm_pk.cu) ----
        const unsigned elected = elect_lane();
        Ring st(MG_STAGES), ac(2);
        int cnt = first < total ? __ldcg(A.jobs + first / A.row_tiles).z : 0;
        for (int tile = first; tile < total; tile += units) {
            const int next = tile + units < total ? __ldcg(A.jobs + (tile + units) / A.row_tiles).z : 0;   // a tile ahead
            const unsigned n = ((unsigned)__shfl_sync(0xffffffffu, cnt, 0) + 15u) & ~15u;
            // D f32, A and B f16, both K-major, M = 128
            const unsigned idesc = (1u << 4) | ((n >> 3) << 17) | ((128u >> 4) << 24);
            pk_wait(smem_u32(&acc_empty[ac.s]), ac.ph ^ 1u, abort_flag);
            const unsigned d = tmem_base + (unsigned)ac.s * 256u;
            for (int u = 0; u < nu; u++) {
                pk_wait(smem_u32(&full[st.s]), st.ph, abort_flag);
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const unsigned ws = smem + (unsigned)st.s * stage_bytes, xs = ws + KC * MG_CHUNK_BYTES;
                pk_mma4<1>(d, pk_desc_lo(ws), pk_desc_lo(xs), idesc, u ? 1u : 0u, elected);
                if (KC == 2) pk_mma4<1>(d, pk_desc_lo(ws + MG_CHUNK_BYTES), pk_desc_lo(xs + x_chunk), idesc, 1u, elected);
                pk_commit<1>(smem_u32(&empty[st.s]), elected);
                st.step(1);
            }
            pk_commit<1>(smem_u32(&acc_full[ac.s]), elected);
            ac.step(1);
            cnt = next;
        }
    } else if (warp == MG_RAW_WARP) {
        // ---- raw weights ----
        Ring raw(MG_RAW_SLOTS);
        bool ok = true;
        int e = first < total ? __ldcg(A.jobs + first / A.row_tiles).x : 0;
        for (int tile = first; tile < total && ok; tile += units) {
            const int next = tile + units < total ? __ldcg(A.jobs + (tile + units) / A.row_tiles).x : 0;
            const int rt = tile % A.row_tiles;
            const int t16 = GATE_UP ? rt * 4 + (lane >> 1) : rt * 8 + lane;
            const bool has = lane < 8 && t16 < tiles16;
            const int n = __popc(__ballot_sync(0xffffffffu, has));
            const int64_t at = GATE_UP ? ((int64_t)e * 2 + (lane & 1)) * tiles16 + t16 : (int64_t)e * tiles16 + t16;
            const unsigned char* src = A.packed + at * A.spt * (int64_t)kStep;
            for (int g = 0; g < A.spt; g++) {
                ok = __all_sync(0xffffffffu, pk_wait(smem_u32(&empty_raw[raw.s]), raw.ph ^ 1u, abort_flag));
                if (!ok) break;
                const unsigned bar = smem_u32(&full_raw[raw.s]);
                if (lane == 0) mbar_expect(bar, (unsigned)n * kStep);
                __syncwarp();
                if (has) bulk_copy(raw_ring + ((unsigned)raw.s * 8u + (unsigned)lane) * kStep, src + (int64_t)g * kStep, kStep, bar);
                raw.step(1);
            }
            e = next;
        }
    } else {
        // ---- token tiles: boxes of 64 positions, as many as the job needs ----
        const unsigned elected = elect_lane();
        Ring st(MG_STAGES);
        int4 job = first < total ? __ldcg(A.jobs + first / A.row_tiles) : make_int4(0, 0, 0, 0);
        for (int tile = first; tile < total; tile += units) {
            const int4 next = tile + units < total ? __ldcg(A.jobs + (tile + units) / A.row_tiles) : job;
            const int pos0 = __shfl_sync(0xffffffffu, job.y, 0), boxes = (__shfl_sync(0xffffffffu, job.z, 0) + MG_BOX_ROWS - 1) / MG_BOX_ROWS;
            for (int u = 0; u < nu; u++) {
                pk_wait(smem_u32(&empty[st.s]), st.ph ^ 1u, abort_flag);
                const unsigned bar = smem_u32(&full[st.s]), dst = smem + (unsigned)st.s * stage_bytes + KC * MG_CHUNK_BYTES;
                pk_expect(bar, (unsigned)(boxes * KC) * (MG_BOX_ROWS * 128u), elected);
                if (KC == 2) {   // jobs of up to 64 tokens
                    pk_tma<1>(dst, &xmap, u * 128, pos0, bar, elected);
                    pk_tma<1>(dst + x_chunk, &xmap, u * 128 + 64, pos0, bar, elected);
                } else {
                    for (int b = 0; b < boxes; b++)
                        pk_tma<1>(dst + (unsigned)b * (MG_BOX_ROWS * 128u), &xmap, u * 64, pos0 + b * MG_BOX_ROWS, bar, elected);
                }
                st.step(1);
            }
            job = next;
        }
        for (int s = 0; s < MG_STAGES; s++) {   // the tensor core's last releases
            pk_wait(smem_u32(&empty[st.s]), st.ph ^ 1u, abort_flag);
            st.step(1);
        }
    }
    pk_finish(abort_flag, A.status, LEV_DEV_TIMEOUT);
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    if (warp == MG_MMA_WARP) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(512) : "memory");
}

// Activation rows for k_moe_gemm: f32 row (of the token of pair perm[pos], or row pos itself) -> f16, scaled by the
// power of two that brings its largest magnitude into [2^14, 2^15), 64-column chunks in the column order of
// q40_word_f16.  One block of 128 threads per position; a thread makes 16-byte pieces from two 16-byte loads, or from
// eight single ones where the caller's rows do not start on 16 bytes.
template <bool VEC>
__global__ void __launch_bounds__(128) k_rows_f16(const float* __restrict__ x, const int* __restrict__ perm, const int* __restrict__ total_pos,
                                                  int top_k, int cols, uint4* __restrict__ out, float* __restrict__ scale) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ unsigned wmax[4];
    const int pos = blockIdx.x;
    if (pos >= *total_pos) return;
    const float* row = x + (int64_t)(perm ? perm[pos] / top_k : pos) * cols;
    const int pieces = cols >> 3, tid = threadIdx.x;
    constexpr int kMost = 8;   // 8192 columns
    float4 a[kMost], b[kMost];
    unsigned m = 0;
#pragma unroll
    for (int i = 0; i < kMost; i++) {
        const int d = tid + 128 * i;
        if (128 * i < pieces && d < pieces) {
            const float* src = row + (d >> 3) * 64 + ((d >> 2) & 1) * 32 + (d & 3) * 4;
            if (VEC) {
                a[i] = __ldcg(reinterpret_cast<const float4*>(src));
                b[i] = __ldcg(reinterpret_cast<const float4*>(src) + 4);
            } else {
                a[i] = make_float4(__ldcg(src), __ldcg(src + 1), __ldcg(src + 2), __ldcg(src + 3));
                b[i] = make_float4(__ldcg(src + 16), __ldcg(src + 17), __ldcg(src + 18), __ldcg(src + 19));
            }
        }
    }
#pragma unroll
    for (int i = 0; i < kMost; i++) {
        if (128 * i < pieces && tid + 128 * i < pieces) {
            const float v[8] = {a[i].x, a[i].y, a[i].z, a[i].w, b[i].x, b[i].y, b[i].z, b[i].w};
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const unsigned u = __float_as_uint(v[j]) & 0x7fffffffu;   // magnitudes order like integers
                if (u < 0x7f800000u) m = max(m, u);
            }
        }
    }
    m = __reduce_max_sync(0xffffffffu, m);
    if ((tid & 31) == 0) wmax[tid >> 5] = m;
    __syncthreads();
    m = max(max(wmax[0], wmax[1]), max(wmax[2], wmax[3]));
    // exponent of the largest finite magnitude e: factor 2^(14 - e), its inverse 2^(e - 14); infinities and NaN stay what
    // they are.  Both stay in the normal range: e is held to [-111, 127].
    int e = (int)(m >> 23) - 127;
    if (m == 0u) e = 14;
    if (e < -111) e = -111;
    const float f = __uint_as_float((unsigned)(127 + 14 - e) << 23), inv = __uint_as_float((unsigned)(127 - 14 + e) << 23);
    if (tid == 0) scale[pos] = inv;
    uint4* dst = out + (int64_t)pos * pieces;
#pragma unroll
    for (int i = 0; i < kMost; i++) {
        const int d = tid + 128 * i;
        if (128 * i < pieces && d < pieces) {
            auto h2 = [f](float lo, float hi) {
                const __half2 h = __floats2half2_rn(lo * f, hi * f);
                return *reinterpret_cast<const unsigned*>(&h);
            };
            dst[d] = make_uint4(h2(a[i].x, a[i].z), h2(b[i].x, b[i].z), h2(a[i].y, a[i].w), h2(b[i].y, b[i].w));
        }
    }
}

// act[pair id] = the activation row of its position (diagnostic output)
__global__ void k_act_by_pair(const float* __restrict__ act, const int* __restrict__ perm, const int* __restrict__ total_pos, int inter,
                              float* __restrict__ out) {
    pdl_launch_dependents();
    pdl_wait();
    const int64_t n = (int64_t)(*total_pos) * inter;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t pos = i / inter;
        out[(int64_t)perm[pos] * inter + (i - pos * inter)] = act[i];
    }
}

template <bool GATE_UP, int KC>
int launch_mg(lev_ctx* ctx, const CUtensorMap& map, const MgArgs& A, int grid, size_t smem) {
    static bool configured[16] = {};   // the most a launch may ask for: see lev_gemm_pk.cu
    if (!configured[ctx->device & 15]) {
        LEV_CUDA(ctx, cudaFuncSetAttribute(k_moe_gemm<GATE_UP, KC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)ctx->prop.sharedMemPerBlockOptin - 1024));
        configured[ctx->device & 15] = true;
    }
    LEV_CUDA(ctx, launch_pdl(k_moe_gemm<GATE_UP, KC>, dim3((unsigned)grid), dim3(MG_THREADS), smem, ctx->stream, map, A));
    ctx->launches++;
    return lev_cuda_check(ctx, cudaGetLastError(), "k_moe_gemm");
}

}  // namespace

// Tokens of a job: 64 with two chunks per stage while an expert's share mostly fits that (a Poisson share of 40 exceeds
// 64 once in ten thousand), else 256 (one accumulator of two).  The pairs are those of all experts, resident or not.
int lev_moe_gemm_job_tokens(int64_t pairs, int experts) { return pairs <= 40 * (int64_t)experts ? 64 : 256; }

bool lev_moe_gemm_supported(const lev_moe_weights* w) {
    const lev_weights *gu = w->gate_up, *dn = w->down;
    // the GGUF-order copy released: the caller has asked for the f32-activation kernels
    return gu && dn && gu->packed && dn->packed && gu->raw && dn->raw && !gu->large_scale && !dn->large_scale && w->hidden % 16 == 0 &&
           w->inter % 16 == 0 && encode_tiled() != nullptr;
}

// bytes of lev_moe_gemm_run's work buffer
size_t lev_moe_gemm_bytes(const lev_moe_weights* w, int64_t pairs) {
    auto up = [](size_t v) { return (v + 255) & ~(size_t)255; };
    return up((size_t)pairs * w->inter * 4) + up((size_t)pairs * w->hidden * 2) + up((size_t)pairs * w->inter * 2) + 2 * up((size_t)pairs * 4);
}

// y[pair id][hidden] of every grouped pair: rows to f16, gate_up with the activation, rows to f16, down
int lev_moe_gemm_run(lev_ctx* ctx, const lev_moe_weights* w, const float* x, int64_t pairs, int top_k, const int* perm, const int* total_pos,
                     const int* njobs, const int4* jobs, int job_tokens, int max_jobs, void* work, float* y, float* act_out) {
    EncodeTiledFn enc = encode_tiled();
    if (!enc) return lev_fail(ctx, LEV_UNSUPPORTED, "cuTensorMapEncodeTiled is not available");
    auto up = [](size_t v) { return (v + 255) & ~(size_t)255; };
    char* p = (char*)work;
    float* act = (float*)p;
    p += up((size_t)pairs * w->inter * 4);
    uint4* xh = (uint4*)p;
    p += up((size_t)pairs * w->hidden * 2);
    uint4* ah = (uint4*)p;
    p += up((size_t)pairs * w->inter * 2);
    float* xs = (float*)p;
    p += up((size_t)pairs * 4);
    float* as = (float*)p;
    const int kc = job_tokens <= 64 ? 2 : 1, sms = ctx->prop.multiProcessorCount;
    for (int half = 0; half < 2; half++) {
        const lev_weights* t = half ? w->down : w->gate_up;
        const bool vec = half || ((uintptr_t)x & 15) == 0;   // columns are a multiple of 32: every row is aligned like the first
        LEV_CUDA(ctx, launch_pdl(vec ? k_rows_f16<true> : k_rows_f16<false>, dim3((unsigned)pairs), dim3(128), (size_t)0, ctx->stream,
                                 half ? (const float*)act : x, half ? (const int*)nullptr : perm, total_pos, top_k, (int)t->cols, half ? ah : xh,
                                 half ? as : xs));
        ctx->launches++;
        LEV_TRY(lev_cuda_check(ctx, cudaGetLastError(), "k_rows_f16"));
        CUtensorMap map;
        const cuuint64_t gdim[2] = {(cuuint64_t)t->cols, (cuuint64_t)pairs};
        const cuuint64_t gstride[1] = {(cuuint64_t)t->cols * 2};
        const cuuint32_t box[2] = {64, MG_BOX_ROWS};
        const cuuint32_t estr[2] = {1, 1};
        CUresult cr = enc(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, half ? (void*)ah : (void*)xh, gdim, gstride, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (cr != CUDA_SUCCESS) return lev_fail(ctx, LEV_KERNEL_FAILED, "cuTensorMapEncodeTiled failed (%d)", (int)cr);
        MgArgs A;
        A.packed = t->packed;
        A.spt = (int)(lev_stream_chunks(t) / 4);
        A.kt = (int)((t->cols + 63) / 64);
        A.rows = half ? w->hidden : w->inter;
        A.row_tiles = half ? (w->hidden + 127) / 128 : (w->inter + 63) / 64;
        A.njobs = njobs;
        A.jobs = jobs;
        A.scale = half ? as : xs;
        A.out_row = perm;
        A.out = half ? y : act;
        A.job_tokens = job_tokens;
        A.status = ctx->d_status;
        const size_t stage = (size_t)kc * (MG_CHUNK_BYTES + job_tokens * 128), raw = (size_t)MG_RAW_SLOTS * 8 * kStepBytesQ4;
        const size_t smem = MG_STAGES * stage + raw + 1024;
        const int64_t most = (int64_t)max_jobs * A.row_tiles;
        const int grid = (int)(most < sms ? most : sms);
        LEV_TRY(half ? (kc == 2 ? launch_mg<false, 2>(ctx, map, A, grid, smem) : launch_mg<false, 1>(ctx, map, A, grid, smem))
                     : (kc == 2 ? launch_mg<true, 2>(ctx, map, A, grid, smem) : launch_mg<true, 1>(ctx, map, A, grid, smem)));
    }
    if (act_out) {
        const int64_t n = pairs * w->inter, blocks = (n + 255) / 256, cap = (int64_t)sms * 8;
        LEV_CUDA(ctx, launch_pdl(k_act_by_pair, dim3((unsigned)(blocks < cap ? blocks : cap)), dim3(256), (size_t)0, ctx->stream, (const float*)act,
                                 perm, total_pos, w->inter, act_out));
        ctx->launches++;
        return lev_cuda_check(ctx, cudaGetLastError(), "k_act_by_pair");
    }
    return LEV_OK;
}
