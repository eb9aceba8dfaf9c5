// Prefill dequant-GEMM on the fifth-generation tensor cores (tcgen05 + TMEM), sm_100a.
//
//   Y[t][r] = sum_k bf16(W[r][k]) * X[t][k],  f32 accumulate in tensor memory
//
// Weights are decoded bit-exactly as the block decoders form them and rounded once to bf16; activations are bf16
// already (rust/crates/lev-forge/src/coopmat.rs:236-425, oracle rust/crates/lev-cli/src/main.rs:1201-1217).
//
// The weight rows are the MMA's M (128 per CTA) and the tokens its N (up to 512 columns of tensor memory), so a
// decoded weight tile is used for up to 512 tokens.  More than 128 tokens run as CTA pairs (cta_group::2, M = 256):
// each CTA decodes its own 128 rows and loads half of the tokens, and the pair's tensor cores read both halves, which
// halves the token traffic from L2 and the shared-memory reads per product.  Roles of a CTA's 23 warps:
//   * warp 21: raw weight bytes by bulk copies, one 256-column K-step of the eight 16-row tiles (lev_stream.cu's
//     repack: every format comes in aligned contiguous runs there, which GGUF rows of 210-byte blocks do not);
//   * warp 22: token tiles by TMA (64 k per stage, 128-byte swizzle);
//   * warps 0..15: decode (lev_gemm_pk.cuh); warp w takes tile w & 7 and the 64-column chunks of parity w >> 3;
//   * warp 20: MMA issue (the pair's leader only); tcgen05.commit hands stages back to both CTAs;
//   * warps 16..19: epilogue, overlapping the next tile when two accumulators fit (up to 256 tokens).
// CTAs (pairs) are persistent and take every gridDim-th (row tile, K split, token tile).
//
// Measured against the form with tokens as M (256 tokens x 176 rows, GGUF rows decoded straight from global memory)
// on [12288 x 4096] Q4_K: 512 tokens 74 -> 52 us (995 TFLOP/s), 2048 tokens 293 -> 157 us (1313), 64 tokens 34 -> 28;
// [4096 x 12288] Q6_K at 301 tokens 280 -> 37 us; [262144 x 2816] Q6_K at 32 tokens 753 -> 232 us.  What bounds it:
// at 512 tokens the tensor cores (active in 75 % of the cycles of the SMs that have a tile, issue slots 38 % used), at 64
// the decode (issue slots 61 %, ALU 58 %, tensor cores 17 %), in between both (301 tokens of Q6_K: 50, 47, 57 %).
//
// Every wait is bounded by about a second of SM clocks; a CTA that gives up sets LEV_DEV_TIMEOUT, lets its copies
// land, frees its tensor memory and returns.
#include <cuda.h>

#include <type_traits>

#include "lev_gemm_pk.cuh"
#include "lev_umma.cuh"
#include "lev_stream.h"

namespace {

constexpr int PK_KS = 64;                    // k per stage: one 128-byte swizzle row of bf16
constexpr int PK_W_BYTES = 128 * PK_KS * 2;  // decoded weights of a stage
constexpr int PK_MAX_STAGES = 8;
constexpr int PK_RAW_SLOTS = 3;
constexpr int PK_DECODE_WARPS = 16;
// 16 decode warps, four epilogue warps, then:
constexpr int PK_MMA_WARP = 20, PK_RAW_WARP = 21, PK_X_WARP = 22;
constexpr int PK_THREADS = (PK_X_WARP + 1) * 32;
constexpr int PK_TMEM_COLS = 512;

struct PkArgs {
    const unsigned char* packed;
    int spt;               // 256-column K-steps per 16-row tile
    int kt;                // 64-column K-steps of the whole K
    int tiles16;           // 16-row tiles of the tensor
    int64_t rows;
    int tokens;
    int row_tiles, tok_tiles, splits, groups_per_split;
    int n_part;            // tokens of one MMA (its N); parts MMAs side by side make a tile
    int parts;
    int stages, acc_stages;
    float* y;              // [split][tokens][rows]
    int* status;
};

// tile k of this CTA (pair): row tile, K range in 64-column steps, first token
struct PkTile {
    int rt, z, t0, k0, kt;
};
__device__ __forceinline__ PkTile pk_tile(const PkArgs& A, int tile) {
    PkTile T;
    const int tt = tile % A.tok_tiles, r = tile / A.tok_tiles;
    T.z = r % A.splits;
    T.rt = r / A.splits;
    T.t0 = tt * A.n_part * A.parts;
    T.k0 = T.z * A.groups_per_split * 4;
    const int left = A.kt - T.k0;
    T.kt = left < A.groups_per_split * 4 ? left : A.groups_per_split * 4;
    return T;
}

template <int TYPE, int CG>
__global__ void __launch_bounds__(PK_THREADS, 1) k_gemm_pk(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ PkArgs A) {
    extern __shared__ unsigned char smem_dyn[];
    __shared__ __align__(8) unsigned long long full[PK_MAX_STAGES], empty[PK_MAX_STAGES];
    __shared__ __align__(8) unsigned long long full_raw[PK_RAW_SLOTS], empty_raw[PK_RAW_SLOTS], acc_full[2], acc_empty[2];
    __shared__ unsigned tmem_base_s;
    __shared__ int abort_s;
    constexpr unsigned kStep = (unsigned)step_bytes(TYPE);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned rank = CG == 2 ? cluster_rank() : 0u;
    const int unit = (int)blockIdx.x / CG, units = (int)gridDim.x / CG;
    const int total = A.row_tiles * A.splits * A.tok_tiles;
    // stages (1024-byte aligned: decoded weights, then this CTA's tokens), then the ring of raw K-steps
    const unsigned smem = (smem_u32(smem_dyn) + 1023u) & ~1023u;
    const unsigned part_bytes = (unsigned)(A.n_part / CG) * 128u;   // this CTA's tokens of one MMA, one stage
    const unsigned stage_bytes = PK_W_BYTES + (unsigned)A.parts * part_bytes;
    const unsigned raw_ring = smem + (unsigned)A.stages * stage_bytes;

    if (threadIdx.x == 0) {
        abort_s = 0;
        for (int s = 0; s < PK_MAX_STAGES; s++) {
            mbar_init(smem_u32(&full[s]), 1 + 8 * CG);   // the token boxes' bytes and the decode warps
            mbar_init(smem_u32(&empty[s]), 1);
        }
        for (int s = 0; s < PK_RAW_SLOTS; s++) {
            mbar_init(smem_u32(&full_raw[s]), 1);
            mbar_init(smem_u32(&empty_raw[s]), PK_DECODE_WARPS);
        }
        for (int s = 0; s < 2; s++) {
            mbar_init(smem_u32(&acc_full[s]), 1);
            mbar_init(smem_u32(&acc_empty[s]), 4 * CG);
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    }
    if (warp == PK_MMA_WARP) {
        if (CG == 2) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_base_s)), "r"(PK_TMEM_COLS)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_base_s)), "r"(PK_TMEM_COLS)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
        }
    }
    pdl_launch_dependents();
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (CG == 2) cluster_sync_all();   // the pair's barriers are initialised before either CTA arrives at the other's
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const unsigned tmem_base = tmem_base_s;
    volatile int* abort_flag = &abort_s;

    if (warp < PK_DECODE_WARPS) {
        // ---- decode: tile w & 7, chunks of parity w >> 3 ----
        const int tl = warp & 7, p = warp >> 3;
        const DecodeLane L = decode_lane<TYPE>(lane);
        Ring st(A.stages), raw(PK_RAW_SLOTS);
        st.step(p);
        const unsigned wt0 = smem + (unsigned)tl * 2048u, raw0 = raw_ring + (unsigned)tl * kStep;
        const unsigned full_c = CG == 2 ? map_to_rank(smem_u32(&full[0]), 0) : smem_u32(&full[0]);
        bool ok = true;
        auto chunk = [&](auto cc_tag, unsigned src, bool live, const DecodeScales& S) {
            constexpr int CC = decltype(cc_tag)::value;
            ok &= pk_wait(smem_u32(&empty[st.s]), st.ph ^ 1u, abort_flag);   // not branched on here: the warp stays together
            if (live) decode_chunk<TYPE, CC>(src, p, wt0 + (unsigned)st.s * stage_bytes, L, S);
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");  // the tensor core reads through the async proxy
            __syncwarp();
            if (lane == 0) {
                if (CG == 2) mbar_arrive_cluster(full_c + 8u * (unsigned)st.s);
                else mbar_arrive(full_c + 8u * (unsigned)st.s);
            }
            st.step(2);
        };
        for (int tile = unit; tile < total && ok; tile += units) {
            const PkTile T = pk_tile(A, tile);
            const bool live = (T.rt * CG + (int)rank) * 8 + tl < A.tiles16;
            for (int left = T.kt - p; left + p > 0 && ok; left -= 4) {   // K-steps from this warp's first of the group on
                ok = __all_sync(0xffffffffu, pk_wait(smem_u32(&full_raw[raw.s]), raw.ph, abort_flag) & ok);
                const unsigned src = raw0 + (unsigned)raw.s * (8u * kStep);
                DecodeScales S;
                if (live) decode_scales<TYPE>(src, p, L, S);
                if (left > 0) chunk(std::integral_constant<int, 0>(), src, live, S);
                if (left > 2) chunk(std::integral_constant<int, 1>(), src, live, S);
                if (lane == 0) mbar_arrive(smem_u32(&empty_raw[raw.s]));
                raw.step(1);
            }
            ok = __all_sync(0xffffffffu, ok);
            // an odd number of K-steps: the parities change places
            if (T.kt & 1) {
                if (p) st.step(1);
                else st.back();
            }
        }
    } else if (warp < PK_MMA_WARP) {
        // ---- epilogue: lane = weight row, columns = tokens ----
        pdl_wait();
        const int quarter = warp & 3;
        Ring ac(A.acc_stages);
        const int n_tile = A.n_part * A.parts;
        for (int tile = unit; tile < total; tile += units) {
            const PkTile T = pk_tile(A, tile);
            if (!__all_sync(0xffffffffu, pk_wait(smem_u32(&acc_full[ac.s]), ac.ph, abort_flag))) break;
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const int64_t row = ((int64_t)T.rt * CG + rank) * 128 + quarter * 32 + lane;
            const int n = A.tokens - T.t0 < n_tile ? A.tokens - T.t0 : n_tile;
            float* dst = A.y + ((int64_t)T.z * A.tokens + T.t0) * A.rows + row;
            const unsigned src = tmem_base + ((unsigned)(quarter * 32) << 16) + (unsigned)ac.s * 256u;
#pragma unroll 1
            for (int c = 0; c < n; c += 32) {
                unsigned v[32];
                if (c + 32 <= n_tile) tmem_ld32(src + (unsigned)c, v);
                else tmem_ld16(src + (unsigned)c, v);   // n_tile is a multiple of 16
                asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
                if (row < A.rows) {
#pragma unroll
                    for (int q = 0; q < 32; q++)
                        if (c + q < n) dst[(int64_t)(c + q) * A.rows] = __uint_as_float(v[q]);
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                const unsigned bar = smem_u32(&acc_empty[ac.s]);
                if (CG == 2) mbar_arrive_cluster(map_to_rank(bar, 0));
                else mbar_arrive(bar);
            }
            ac.step(1);
        }
    } else if (warp == PK_MMA_WARP) {
        // ---- MMA issue: the pair's leader.  The whole warp walks the loop and one elected lane issues, so that
        // descriptors and addresses stay in uniform registers (a single-lane loop took 180 cycles per MMA to issue
        // beside the decode warps, and was what bounded the kernel); a wait that ran out is not branched on: what
        // follows stays in bounds. ----
        if (rank == 0) {
            const unsigned elected = elect_lane();
            // D f32, A and B bf16, both K-major
            const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(A.n_part >> 3) << 17) | ((unsigned)((128 * CG) >> 4) << 24);
            Ring st(A.stages), ac(A.acc_stages);
            for (int tile = unit; tile < total; tile += units) {
                const int kt = pk_tile(A, tile).kt;
                pk_wait(smem_u32(&acc_empty[ac.s]), ac.ph ^ 1u, abort_flag);
                const unsigned d = tmem_base + (unsigned)ac.s * 256u;
                for (int it = 0; it < kt; it++) {
                    pk_wait(smem_u32(&full[st.s]), st.ph, abort_flag);
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    const unsigned ws = smem + (unsigned)st.s * stage_bytes;
                    const unsigned a_lo = pk_desc_lo(ws), b_lo = pk_desc_lo(ws + PK_W_BYTES);
                    pk_mma4<CG>(d, a_lo, b_lo, idesc, it ? 1u : 0u, elected);
                    if (A.parts == 2) pk_mma4<CG>(d + (unsigned)A.n_part, a_lo, b_lo + (part_bytes >> 4), idesc, it ? 1u : 0u, elected);
                    pk_commit<CG>(smem_u32(&empty[st.s]), elected);
                    st.step(1);
                }
                pk_commit<CG>(smem_u32(&acc_full[ac.s]), elected);
                ac.step(1);
            }
        }
    } else if (warp == PK_RAW_WARP) {
        // ---- raw weights: constants, requested before the launch this one depends on has finished ----
        Ring raw(PK_RAW_SLOTS);
        bool ok = true;
        for (int tile = unit; tile < total && ok; tile += units) {
            const PkTile T = pk_tile(A, tile);
            const int first = (T.rt * CG + (int)rank) * 8;
            int n = A.tiles16 - first;
            n = n < 0 ? 0 : (n > 8 ? 8 : n);
            const unsigned char* src = A.packed + ((int64_t)(first + lane) * A.spt + (T.k0 >> 2)) * kStep;
            for (int g = 0; 4 * g < T.kt && ok; g++) {
                ok = __all_sync(0xffffffffu, pk_wait(smem_u32(&empty_raw[raw.s]), raw.ph ^ 1u, abort_flag));
                if (!ok) break;
                const unsigned bar = smem_u32(&full_raw[raw.s]);
                if (lane == 0) mbar_expect(bar, (unsigned)n * kStep);
                __syncwarp();
                if (lane < n) bulk_copy(raw_ring + ((unsigned)raw.s * 8u + (unsigned)lane) * kStep, src + (int64_t)g * kStep, kStep, bar);
                raw.step(1);
            }
        }
    } else {
        // ---- token tiles (a wait that ran out is not branched on, as above) ----
        pdl_wait();
        const unsigned elected = elect_lane();
        const unsigned full_c = CG == 2 ? map_to_rank(smem_u32(&full[0]), 0) : smem_u32(&full[0]);
        Ring st(A.stages);
        for (int tile = unit; tile < total; tile += units) {
            const PkTile T = pk_tile(A, tile);
            const int y0 = T.t0 + (int)rank * (A.n_part / CG);
            for (int it = 0; it < T.kt; it++) {
                pk_wait(smem_u32(&empty[st.s]), st.ph ^ 1u, abort_flag);
                const unsigned bar = full_c + 8u * (unsigned)st.s, dst = smem + (unsigned)st.s * stage_bytes + PK_W_BYTES;
                if (rank == 0) pk_expect(smem_u32(&full[st.s]), (unsigned)(A.parts * CG) * part_bytes, elected);
                pk_tma<CG>(dst, &xmap, (T.k0 + it) * PK_KS, y0, bar, elected);
                if (A.parts == 2) pk_tma<CG>(dst + part_bytes, &xmap, (T.k0 + it) * PK_KS, y0 + A.n_part, bar, elected);
                st.step(1);
            }
        }
        // the tensor core's last releases have arrived before the CTA goes (they may come from the pair's leader)
        for (int s = 0; s < A.stages; s++) {
            pk_wait(smem_u32(&empty[st.s]), st.ph ^ 1u, abort_flag);
            st.step(1);
        }
    }
    pk_finish(abort_flag, A.status, LEV_DEV_TIMEOUT);
    if (CG == 2) cluster_sync_all();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    if (warp == PK_MMA_WARP) {
        if (CG == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(PK_TMEM_COLS) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(PK_TMEM_COLS) : "memory");
    }
}

// y = sum over the K splits' partial products, in split order (the same bits on every run)
__global__ void __launch_bounds__(256) k_gemm_split_sum(const float4* __restrict__ part, int splits, int64_t n4, float4* __restrict__ y) {
    pdl_launch_dependents();
    pdl_wait();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (int64_t)gridDim.x * blockDim.x) {
        float4 a = __ldcs(part + i);
        for (int z = 1; z < splits; z++) {
            const float4 b = __ldcs(part + (int64_t)z * n4 + i);
            a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
        }
        y[i] = a;
    }
}

// How a call is cut: token tiles of at most 512 columns of tensor memory (two MMAs of at most 256), and a K split
// where the row tiles leave SMs idle.  The candidate with the smallest estimated time wins: waves of tiles, each
// K-step of a tile costing what its MMAs take (2 clocks per token: 256 x N x 64 at the dense bf16 rate, half of that
// per CTA of a pair) or what the decode of 128 x 64 weights takes (measured), whichever is longer; a fixed cost per
// tile (pipeline fill, epilogue); and for a split the partial sums' trip through L2 and the launch that adds them.
struct PkPlan {
    int cg, tok_tiles, parts, n_part, splits, groups_per_split, stages, units;
    size_t smem;
};
PkPlan pk_plan(lev_ctx* ctx, int type, int64_t rows, int64_t kt, int64_t tokens, bool can_split) {
    PkPlan best = {};
    double best_t = 0;
    const int cg = tokens > 128 ? 2 : 1;
    const int64_t units = ctx->prop.multiProcessorCount / cg, row_tiles = (rows + 128 * cg - 1) / (128 * cg), groups = (kt + 3) / 4;
    const double decode = type == LEV_GGML_Q4_0 ? 550 : 650;
    const int64_t least = (tokens + 511) / 512;
    for (int64_t tt = least; tt <= 2 * least; tt++) {
        const int64_t per = (tokens + tt - 1) / tt, parts = per > 256 ? 2 : 1, q = cg == 2 ? 32 : 16;
        const int64_t n_part = ((per + parts - 1) / parts + q - 1) / q * q, n = n_part * parts;
        for (int64_t z0 = 1; z0 <= (can_split ? 16 : 1) && z0 <= groups; z0++) {
            const int64_t gps = (groups + z0 - 1) / z0, z = (groups + gps - 1) / gps;
            const int64_t waves = (row_tiles * tt * z + units - 1) / units;
            const double step = 2.0 * n > decode ? 2.0 * n : decode;
            double t = waves * (4.0 * gps * step + (n > 256 ? 14.0 * n : 1000.0)) + 2500 + 14.0 * n;
            if (z > 1) t += (2.0 * z + 1.0) * tokens * rows * 4 / 4000.0 + 4000;
            if (best_t == 0 || t < best_t) {
                best_t = t;
                best = {cg, (int)tt, (int)parts, (int)n_part, (int)z, (int)gps, 0, (int)units, 0};
            }
        }
    }
    const size_t raw = (size_t)PK_RAW_SLOTS * 8 * step_bytes(type), stage = PK_W_BYTES + (size_t)best.parts * (best.n_part / cg) * 128;
    const size_t cap = ctx->prop.sharedMemPerBlockOptin - 1024 - 1024;   // static barriers, alignment of the stages
    int64_t s = (int64_t)((cap - raw) / stage);
    best.stages = (int)(s > PK_MAX_STAGES ? PK_MAX_STAGES : s);
    best.smem = best.stages * stage + raw + 1024;
    return best;
}

template <int TYPE, int CG>
int launch_pk(lev_ctx* ctx, const CUtensorMap& map, const PkArgs& A, int grid, size_t smem) {
    static bool configured[16] = {};   // the most a launch may ask for, so that two threads' first calls cannot undercut each other
    if (!configured[ctx->device & 15]) {
        LEV_CUDA(ctx, cudaFuncSetAttribute(k_gemm_pk<TYPE, CG>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)ctx->prop.sharedMemPerBlockOptin - 1024));
        configured[ctx->device & 15] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(PK_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = CG;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = CG == 2 ? 2 : 1;
    LEV_CUDA(ctx, cudaLaunchKernelEx(&cfg, k_gemm_pk<TYPE, CG>, map, A));
    return LEV_OK;
}

// Allocations that may happen beside a stream capture (of this call or of another thread): cudaMalloc is no stream
// operation and legal there, but a capture in global mode has it refused unless the thread says that it knows.
struct CaptureRelaxed {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    CaptureRelaxed() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~CaptureRelaxed() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

bool split_alloc(lev_split_buffer* b, unsigned long long stream, unsigned long long capture, size_t bytes) {
    *b = {stream, capture, nullptr, 0};
    const CaptureRelaxed relaxed;
    if (cudaMalloc(&b->p, bytes) != cudaSuccess) return false;
    b->bytes = bytes;
    return true;
}

// The buffer of a call's partial products, or NULL: the call is then planned without a split.
float* split_buffer(lev_ctx* ctx, size_t bytes, bool prompt) {
    lev_split_buffers& B = ctx->split;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    unsigned long long stream = (unsigned long long)(uintptr_t)ctx->stream, capture = 0;
    if (cudaStreamGetCaptureInfo(ctx->stream, &cs, &capture) != cudaSuccess) return nullptr;
    if (cs == cudaStreamCaptureStatusNone) {
        {
            const CaptureRelaxed relaxed;   // the id is not to be had from a stream that is being captured
            if (cudaStreamGetId(ctx->stream, &stream) != cudaSuccess) return nullptr;
        }
        lev_split_buffer* b = B.eager;
        while (b < B.eager + B.eagers && b->stream != stream) b++;
        if (b == B.eager + LEV_SPLIT_EAGER) return nullptr;
        if (b == B.eager + B.eagers) {
            if (!split_alloc(b, stream, 0, bytes + bytes / 4)) return nullptr;
            B.eagers++;
        } else if (b->bytes < bytes) {   // grows; only this stream's calls use it
            const CaptureRelaxed relaxed;
            if (cudaStreamSynchronize(ctx->stream) != cudaSuccess) return nullptr;
            cudaFree(b->p);
            if (!split_alloc(b, stream, 0, bytes + bytes / 4)) return nullptr;
        }
        return (float*)b->p;
    }
    lev_split_buffer* list = prompt ? B.prompt : B.batch;
    int& n = prompt ? B.prompts : B.batches;
    size_t most = 0;
    for (int i = n - 1; i >= 0; i--)
        if (!prompt || (list[i].stream == stream && list[i].capture == capture)) {
            if (list[i].bytes >= bytes) return (float*)list[i].p;
            most = list[i].bytes > most ? list[i].bytes : most;
        }
    if (n == (prompt ? LEV_SPLIT_PROMPT : LEV_SPLIT_BATCH) || !split_alloc(&list[n], stream, capture, bytes > 2 * most ? bytes : 2 * most))
        return nullptr;
    return (float*)list[n++].p;
}

}  // namespace

// shapes the tensor-memory kernel serves: repacked tensors, activations on a 16-byte boundary
bool lev_gemm_tc_supported(const lev_weights* w, const void* x_bf16, int64_t tokens) {
    if (!w->packed || w->cols % 8 != 0 || ((uintptr_t)x_bf16 & 15) != 0 || tokens < 1) return false;
    return encode_tiled() != nullptr;
}

int lev_gemm_tc_run(lev_ctx* ctx, const lev_weights* w, const void* x_bf16, int64_t tokens, float* y) {
    EncodeTiledFn enc = encode_tiled();
    if (!enc) return lev_fail(ctx, LEV_UNSUPPORTED, "cuTensorMapEncodeTiled is not available");
    const int64_t kt = (w->cols + PK_KS - 1) / PK_KS;
    const bool can_split = ((uintptr_t)y & 15) == 0 && (tokens * w->rows) % 4 == 0;
    PkPlan P = pk_plan(ctx, w->type, w->rows, kt, tokens, can_split);
    // Captured calls split like eager ones (the same bits): the buffer is one that graphs may hold.
    float* part = nullptr;
    if (P.splits > 1 && !(part = split_buffer(ctx, (size_t)P.splits * tokens * w->rows * sizeof(float), tokens > 128 || w->type == LEV_GGML_Q6_K))) {
        cudaGetLastError();   // out of memory is no error of this call
        P = pk_plan(ctx, w->type, w->rows, kt, tokens, false);
    }
    CUtensorMap map;
    const cuuint64_t gdim[2] = {(cuuint64_t)w->cols, (cuuint64_t)tokens};
    const cuuint64_t gstride[1] = {(cuuint64_t)w->cols * 2};
    const cuuint32_t box[2] = {PK_KS, (cuuint32_t)(P.n_part / P.cg)};
    const cuuint32_t estr[2] = {1, 1};
    CUresult cr = enc(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(x_bf16), gdim, gstride, box, estr,
                      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (cr != CUDA_SUCCESS) return lev_fail(ctx, LEV_KERNEL_FAILED, "cuTensorMapEncodeTiled failed (%d)", (int)cr);
    PkArgs A;
    A.packed = w->packed;
    A.spt = (int)(lev_stream_chunks(w) / 4);
    A.kt = (int)kt;
    A.tiles16 = (int)((w->rows + 15) / 16);
    A.rows = w->rows;
    A.tokens = (int)tokens;
    A.row_tiles = (int)((w->rows + 128 * P.cg - 1) / (128 * P.cg));
    A.tok_tiles = P.tok_tiles;
    A.splits = P.splits;
    A.groups_per_split = P.groups_per_split;
    A.n_part = P.n_part;
    A.parts = P.parts;
    A.stages = P.stages;
    A.acc_stages = P.n_part * P.parts <= 256 ? 2 : 1;
    A.y = part ? part : y;
    A.status = ctx->d_status;
    const int64_t tiles = (int64_t)A.row_tiles * A.splits * A.tok_tiles;
    const int grid = (int)(tiles < P.units ? tiles : P.units) * P.cg;
    int st;
    if (P.cg == 2)
        st = w->type == LEV_GGML_Q6_K   ? launch_pk<LEV_GGML_Q6_K, 2>(ctx, map, A, grid, P.smem)
             : w->type == LEV_GGML_Q4_K ? launch_pk<LEV_GGML_Q4_K, 2>(ctx, map, A, grid, P.smem)
                                        : launch_pk<LEV_GGML_Q4_0, 2>(ctx, map, A, grid, P.smem);
    else
        st = w->type == LEV_GGML_Q6_K   ? launch_pk<LEV_GGML_Q6_K, 1>(ctx, map, A, grid, P.smem)
             : w->type == LEV_GGML_Q4_K ? launch_pk<LEV_GGML_Q4_K, 1>(ctx, map, A, grid, P.smem)
                                        : launch_pk<LEV_GGML_Q4_0, 1>(ctx, map, A, grid, P.smem);
    if (st) return st;
    ctx->launches++;
    LEV_TRY(lev_cuda_check(ctx, cudaGetLastError(), "k_gemm_pk"));
    if (part) {
        const int64_t n4 = tokens * w->rows / 4;
        const int64_t blocks = (n4 + 255) / 256, cap = (int64_t)ctx->prop.multiProcessorCount * 8;
        LEV_CUDA(ctx, launch_pdl(k_gemm_split_sum, dim3((unsigned)(blocks < cap ? blocks : cap)), dim3(256), (size_t)0, ctx->stream,
                                 (const float4*)part, P.splits, n4, (float4*)y));
        ctx->launches++;
        return lev_cuda_check(ctx, cudaGetLastError(), "k_gemm_split_sum");
    }
    return LEV_OK;
}
