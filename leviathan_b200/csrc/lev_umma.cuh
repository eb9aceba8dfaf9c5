// What the tcgen05 kernels share (lev_gemm_pk.cu, lev_moe_gemm.cu): bounded waits, ring positions, MMA issue from a
// converged warp, TMA boxes, tensor-memory reads, CTA pairs.
#pragma once
#include <cuda.h>

#include "lev_stream_math.cuh"

namespace {

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
__device__ __forceinline__ unsigned map_to_rank(unsigned a, unsigned rank) {
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(unsigned cluster_bar) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];\n" ::"r"(cluster_bar) : "memory");
}
__device__ __forceinline__ unsigned pk_try(unsigned bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok;
}
// the same with the thread suspended for up to 20 us meanwhile: the polls of idle warps take issue slots otherwise
__device__ __forceinline__ unsigned pk_try_suspended(unsigned bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(20000u)
        : "memory");
    return ok;
}
// bounded wait (about a second); false on timeout or when another thread of the CTA has already given up
__device__ __noinline__ bool pk_wait_slow(unsigned bar, unsigned parity, volatile int* abort_flag) {
    long long t_start = 0;
    for (unsigned i = 1;; i++) {
        if (pk_try_suspended(bar, parity)) return true;
        if ((i & 15u) == 0) {
            if (*abort_flag) return false;
            const long long now = clock64();
            if (t_start == 0) t_start = now;
            else if (now - t_start > kWaitCycles) {
                *abort_flag = 1;
                return false;
            }
        }
    }
}
__device__ __forceinline__ bool pk_wait(unsigned bar, unsigned parity, volatile int* abort_flag) {
    return pk_try(bar, parity) || pk_wait_slow(bar, parity, abort_flag);
}
// A CTA's last steps after its roles.  A thread that knows of a wait that ran out lets copies in flight land; the status
// is set behind the barrier, because the warp that gave up may be the last to get here.
__device__ __forceinline__ void pk_finish(volatile int* abort_flag, int* status, int bit) {
    __syncwarp();
    if (*abort_flag)
        for (const long long t0 = clock64(); clock64() - t0 < 4000000LL;) {}
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (threadIdx.x == 0 && *abort_flag) atomicOr(status, bit);
}
// ring position: stage and phase parity
struct Ring {
    int s, n;
    unsigned ph;
    __device__ __forceinline__ Ring(int stages) : s(0), n(stages), ph(0) {}
    __device__ __forceinline__ void step(int k) {   // k at most n
        s += k;
        if (s >= n) {
            s -= n;
            ph ^= 1u;
        }
    }
    __device__ __forceinline__ void back() {
        if (--s < 0) {
            s += n;
            ph ^= 1u;
        }
    }
};

// low word of a shared-memory matrix descriptor (K-major); the high word is the same for every operand
__device__ __forceinline__ unsigned pk_desc_lo(unsigned a) { return ((a >> 4) & 0x3FFFu) | (1u << 16); }
// one K-step (four MMAs of K = 16: descriptors step by 32 bytes) of one part of the tile, issued by the elected lane
// of a converged warp
template <int CG>
__device__ __forceinline__ void pk_mma4(unsigned d, unsigned a_lo, unsigned b_lo, unsigned idesc, unsigned acc, unsigned elected) {
    constexpr unsigned kDescHi = (unsigned)((1024 >> 4) | (1u << 14) | (2u << 29));   // 8-row stride, version, 128-byte swizzle
#define LEV_MMA4(GROUP)                                                                                        \
    asm volatile(                                                                                              \
        "{\n .reg .pred p, q, t;\n .reg .b32 a, b;\n .reg .b64 da, db;\n"                                      \
        " setp.ne.b32 p, %5, 0;\n setp.ne.b32 q, %6, 0;\n setp.eq.b32 t, %4, %4;\n"                            \
        " mov.b64 da, {%1, %4};\n mov.b64 db, {%2, %4};\n"                                                     \
        " @q tcgen05.mma.cta_group::" GROUP ".kind::f16 [%0], da, db, %3, p;\n"                                \
        " add.u32 a, %1, 2;\n add.u32 b, %2, 2;\n mov.b64 da, {a, %4};\n mov.b64 db, {b, %4};\n"               \
        " @q tcgen05.mma.cta_group::" GROUP ".kind::f16 [%0], da, db, %3, t;\n"                                \
        " add.u32 a, %1, 4;\n add.u32 b, %2, 4;\n mov.b64 da, {a, %4};\n mov.b64 db, {b, %4};\n"               \
        " @q tcgen05.mma.cta_group::" GROUP ".kind::f16 [%0], da, db, %3, t;\n"                                \
        " add.u32 a, %1, 6;\n add.u32 b, %2, 6;\n mov.b64 da, {a, %4};\n mov.b64 db, {b, %4};\n"               \
        " @q tcgen05.mma.cta_group::" GROUP ".kind::f16 [%0], da, db, %3, t;\n}\n" ::"r"(d),                   \
        "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(kDescHi), "r"(acc), "r"(elected)                                 \
        : "memory")
    if (CG == 2) LEV_MMA4("2");
    else LEV_MMA4("1");
#undef LEV_MMA4
}
template <int CG>
__device__ __forceinline__ void pk_commit(unsigned bar, unsigned elected) {
    if (CG == 2)
        asm volatile(
            "{\n .reg .pred q;\n setp.ne.b32 q, %2, 0;\n"
            " @q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n}\n" ::"r"(bar),
            "h"((unsigned short)3), "r"(elected)
            : "memory");
    else
        asm volatile(
            "{\n .reg .pred q;\n setp.ne.b32 q, %1, 0;\n @q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(bar),
            "r"(elected)
            : "memory");
}
// One box of the token tile; bar is a cluster address (the leader's barrier for a CTA pair).  Like the MMAs, issued by
// the elected lane of a converged warp: from a single-lane branch one box took 250 cycles to issue.
template <int CG>
__device__ __forceinline__ void pk_tma(unsigned dst, const CUtensorMap* map, int x, int y, unsigned bar, unsigned elected) {
    if (CG == 2)
        asm volatile(
            "{\n .reg .pred q;\n setp.ne.b32 q, %5, 0;\n"
            " @q cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n}\n" ::"r"(dst),
            "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar), "r"(elected)
            : "memory");
    else
        asm volatile(
            "{\n .reg .pred q;\n setp.ne.b32 q, %5, 0;\n"
            " @q cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n}\n" ::"r"(dst),
            "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar), "r"(elected)
            : "memory");
}
__device__ __forceinline__ void pk_expect(unsigned bar, unsigned bytes, unsigned elected) {
    asm volatile(
        "{\n .reg .pred q;\n setp.ne.b32 q, %2, 0;\n @q mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n}\n" ::"r"(bar), "r"(bytes), "r"(elected)
        : "memory");
}
__device__ __forceinline__ unsigned elect_lane() {
    unsigned e;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(e));
    return e;
}

__device__ __forceinline__ void tmem_ld32(unsigned a, unsigned* v) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
          "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]),
          "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]),
          "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(a)
        : "memory");
}
__device__ __forceinline__ void tmem_ld16(unsigned a, unsigned* v) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
          "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(a)
        : "memory");
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled() {
    static const EncodeTiledFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        return cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess
                   ? (EncodeTiledFn)p
                   : (EncodeTiledFn) nullptr;
    }();
    return fn;
}

}  // namespace
