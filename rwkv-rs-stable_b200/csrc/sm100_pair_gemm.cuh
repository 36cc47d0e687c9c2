// Main loop of a bf16 matrix product on pairs of CTAs: D[256 x width] = A[256 x K] B[width x K]^T, both operands row-major in
// global memory, fp32 accumulators in TMEM.  The kernel around it has the epilogue.
//
// A cluster of two CTAs on neighbouring SMs works on one tile (tcgen05 with cta_group::2): each holds 128 rows of A, half of the
// tile's columns of B, and the accumulators of its 128 rows and all columns.  Per product an SM then reads half of B from its own
// shared memory and TMA writes half of it, where one CTA on a 128 x 256 tile reads and writes all of it.  A CTA's share of a
// K slice of 64 is 16 KB of A and up to 16 KB of B, 128-byte swizzle, in a ring of six.  Bound by the tensor cores, at large sizes by
// the power they draw; what moves through shared memory and L2 costs power too.  Measured: the channel mixer of 4096 rows, C = 2048,
// F = 8192 (275 GFLOP), 250 us on single CTAs, 226 on pairs.
//
// Barriers: `full` in the first CTA alone (its own bytes and its peer's), `empty` and `tmem_full` in both (one commit arrives at
// both), `tmem_empty` in the first alone (four epilogue warps of each CTA).  Every wait is bounded.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "sm100_umma.cuh"

namespace rwkv7 {
namespace sm100 {

constexpr int kPairM = 256, kPairN = 256, kPairK = 64, kPairStages = 6;
constexpr int kPairThreads = 192;   // TMA warp, MMA warp, four epilogue warps
constexpr uint32_t kPairHalf = 128 * kPairK * 2;   // one CTA's share of a K slice of A, or (at most) of B
constexpr uint32_t kPairSmem = kPairStages * 2 * kPairHalf + 1024 /*barriers*/;

// Loads into this CTA's shared memory; the bytes are counted on a barrier of the pair's first CTA.  (No multicast.)
__device__ __forceinline__ void tma_load_2d_pair(void *smem_dst, const CUtensorMap *map, int x, int y, uint32_t first_bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(smem_u32(smem_dst)), "l"(map), "r"(first_bar), "r"(x), "r"(y)
        : "memory");
}
__device__ __forceinline__ void umma_f16_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, bool accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"((uint32_t)accumulate)
        : "memory");
}
// One arrival at this barrier of both CTAs when all products issued so far are done.
__device__ __forceinline__ void umma_commit_pair(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
                 "h"((uint16_t)3)
                 : "memory");
}
// Warp-wide, by one warp of each CTA.
__device__ __forceinline__ void tmem_alloc_pair(uint32_t *smem_dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

struct PairMaps {
    CUtensorMap a;   // [M, K] bf16, box 128 x 64
    CUtensorMap b;   // [N, K] bf16, box width / 2 x 64
};
// One tile of a pair: first row and column, K slices k0 .. k0 + slices - 1.
struct PairItem {
    int m0, n0, k0, slices;
};

// `Items`: bool operator()(int i, PairItem &) gives the pair's i-th tile, false behind the last.
struct PairGemm {
    unsigned char *smem;
    uint64_t *full, *empty, *tmem_full, *tmem_empty;
    uint32_t *tmem_slot;
    uint32_t rank, tmem;

    // All threads.  1024-byte aligned shared memory.
    __device__ __forceinline__ void begin(unsigned char *room, const PairMaps &maps, int warp) {
        smem = room;
        full = reinterpret_cast<uint64_t *>(smem + kPairStages * 2 * kPairHalf);
        empty = full + kPairStages;
        tmem_full = empty + kPairStages;
        tmem_empty = tmem_full + 2;
        tmem_slot = reinterpret_cast<uint32_t *>(tmem_empty + 2);
        rank = cluster_ctarank();
        if (threadIdx.x == 0) {
            for (int s = 0; s < kPairStages; ++s) {
                mbar_init(&full[s], 1);
                mbar_init(&empty[s], 1);
            }
            for (int b = 0; b < 2; ++b) {
                mbar_init(&tmem_full[b], 1);
                mbar_init(&tmem_empty[b], 8);
            }
            mbar_fence_init();
            tma_prefetch_desc(&maps.a);
            tma_prefetch_desc(&maps.b);
        }
        if (warp == 1) tmem_alloc_pair(tmem_slot, 512);
        tc_fence_before();
        __syncthreads();
        cluster_sync_all();   // (the peer's barriers are set up)
        tc_fence_after();
        tmem = *tmem_slot;
    }
    // All threads, last.  (Neither CTA leaves while the other's products or arrivals can still reach it.)
    __device__ __forceinline__ void end(int warp) {
        tc_fence_before();
        __syncthreads();
        cluster_sync_all();
        if (warp == 1) tmem_dealloc_pair(tmem, 512);
    }
    // One thread of either CTA.  False when a wait expired.  The first stages' slices of B are requested before `a_is_there` returns,
    // nothing of A is.
    template <typename Items, typename F>
    __device__ __forceinline__ bool produce(const PairMaps &maps, int width, const Items &items, const F &a_is_there) {
        uint32_t it = 0;
        bool ok = true;
        PairItem w;
        auto bar = [&](uint32_t s) { return map_to_cta(smem_u32(&full[s]), 0); };
        auto load_a = [&](uint32_t s, int k) {
            tma_load_2d_pair(smem + s * 2 * kPairHalf, &maps.a, k * kPairK, w.m0 + (int)rank * 128, bar(s));
        };
        auto load_b = [&](uint32_t s, int k) {
            if (rank == 0) mbar_expect_tx(&full[s], 2 * kPairHalf + (uint32_t)width * kPairK * 2);
            tma_load_2d_pair(smem + s * 2 * kPairHalf + kPairHalf, &maps.b, k * kPairK, w.n0 + (int)rank * (width / 2), bar(s));
        };
        const int ahead = items(0, w) ? min(kPairStages, w.slices) : 0;
        for (int j = 0; j < ahead; ++j) load_b(j, w.k0 + j);
        a_is_there();
        for (int j = 0; j < ahead; ++j) load_a(j, w.k0 + j);
        for (int i = 0; ok && items(i, w); ++i) {
            for (int k = w.k0; k < w.k0 + w.slices; ++k, ++it) {
                if (it < (uint32_t)ahead) continue;
                const uint32_t s = it % kPairStages, ph = (it / kPairStages) & 1;
                if (!mbar_wait(&empty[s], ph ^ 1)) { ok = false; break; }
                load_b(s, k);
                load_a(s, k);
            }
        }
        // What is in flight lands, and the products' arrivals come, before the CTA leaves.
        for (uint32_t j = it > kPairStages ? it - kPairStages : 0; j < it; ++j) {
            const uint32_t s = j % kPairStages, ph = (j / kPairStages) & 1;
            if (ok) ok = mbar_wait(&empty[s], ph);
            else if (rank == 0) mbar_wait(&full[s], ph, 100000u);
        }
        return ok;
    }
    // One thread of the first CTA.
    template <typename Items>
    __device__ __forceinline__ bool multiply(int width, const Items &items) {
        const uint32_t idesc = make_idesc(kFmtBF16, kPairM, width, false, false);
        uint32_t it = 0;
        PairItem w;
        for (int i = 0; items(i, w); ++i) {
            const uint32_t buf = i & 1;
            if (!mbar_wait_cluster(&tmem_empty[buf], ((i >> 1) & 1) ^ 1)) return false;
            tc_fence_after();
            for (int k = 0; k < w.slices; ++k, ++it) {
                const uint32_t s = it % kPairStages, ph = (it / kPairStages) & 1;
                if (!mbar_wait_cluster(&full[s], ph)) return false;
                tc_fence_after();
                const uint32_t a = smem_u32(smem + s * 2 * kPairHalf), b = a + kPairHalf;
#pragma unroll
                for (int e = 0; e < kPairK / 16; ++e)
                    umma_f16_pair(tmem + buf * kPairN, make_smem_desc(a + e * 32, 16, 1024), make_smem_desc(b + e * 32, 16, 1024), idesc, k > 0 || e > 0);
                umma_commit_pair(&empty[s]);
            }
            umma_commit_pair(&tmem_full[buf]);
        }
        return true;
    }
    // Epilogue warps: the accumulators of tile i are complete, and have been read.
    __device__ __forceinline__ bool complete(int i) {
        if (!mbar_wait_cluster(&tmem_full[i & 1], (i >> 1) & 1)) return false;
        tc_fence_after();
        return true;
    }
    __device__ __forceinline__ void release(int i) {
        tc_fence_before();
        __syncwarp();
        if ((threadIdx.x & 31) == 0) mbar_arrive_cluster(map_to_cta(smem_u32(&tmem_empty[i & 1]), 0));
    }
};

}  // namespace sm100
}  // namespace rwkv7
