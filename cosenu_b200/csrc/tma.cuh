// Shared pieces of the TMA-pipelined stage kernels (stage_tma.cu: FD,
// stage_fv.cuh: FV): bounded mbarrier waits, tensor-map copies, ensemble table
// helpers and the launch interface.
#pragma once

#include <cuda.h>

#include <type_traits>

#include "chain.cuh"
#include "common.cuh"

namespace cosenu {

namespace tma {

constexpr int TZ = 32;           // cells per tile (one warp lane each)
constexpr int HALO = 4;          // cells each side in the input box
// tensor maps per ensemble member (MapIdx lists them)
constexpr int NMAP = 8;
#define TMA_MAX_NVZ 1024

__device__ __forceinline__ uint32_t smem_u32(const void *p)
{
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ unsigned long long gtimer()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ bool mbar_try(uint64_t *bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait; returns false (and records `code`) when `limit_ns` passes.
// Once any wait in the grid has expired (*err != 0) later waits give up
// at once, so a broken pipeline ends within one time limit.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, int *err, int code,
                                          unsigned long long limit_ns)
{
    if (mbar_try(bar, parity)) return true;
    volatile int *verr = err;
    unsigned long long t0 = 0;
    for (uint32_t n = 1;; ++n) {
        if (mbar_try(bar, parity)) return true;
        // (rarely: the error word and the timer are long-latency reads)
        if ((n & 15) == 0) {
            const unsigned long long now = gtimer();
            if (t0 == 0) t0 = now;
            if (*verr != 0 || now - t0 > limit_ns) {
                atomicCAS(err, 0, code);
                return false;
            }
        }
    }
}

// Wait for the completion of copies already issued, whatever *err says
// (bounded by `limit_ns`, code 3 on expiry): the producer's last act.
__device__ __forceinline__ void mbar_drain(uint64_t *bar, uint32_t parity, int *err,
                                           unsigned long long limit_ns)
{
    if (mbar_try(bar, parity)) return;
    const unsigned long long t0 = gtimer();
    for (uint32_t n = 1;; ++n) {
        if (mbar_try(bar, parity)) return;
        if ((n & 63) == 0 && gtimer() - t0 > limit_ns) {
            atomicCAS(err, 0, 3);
            return;
        }
    }
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar)
{
    asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(
                     smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, int x, int y, int z,
                                            uint64_t *bar)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(dst)),
        "l"((uint64_t)map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
        : "memory");
}

// Brings a tensor map held in global memory into the TMA unit's cache.
__device__ __forceinline__ void prefetch_map(const CUtensorMap *map)
{
    asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)map) : "memory");
}

template <int NCONS> __device__ __forceinline__ void consumer_sync()
{
    asm volatile("bar.sync 1, %0;" ::"n"(NCONS) : "memory");
}

// Arrival counter of a ring buffer without a producer warp: acquire-release
// add, so the last warp's refill is ordered after every warp's reads.
__device__ __forceinline__ uint32_t ring_release_count(uint32_t *cnt)
{
    uint32_t old;
    asm volatile("atom.acq_rel.cta.shared::cta.add.u32 %0, [%1], 1;"
                 : "=r"(old)
                 : "r"(smem_u32(cnt))
                 : "memory");
    return old;
}

// Orders this thread's generic-proxy view of shared memory before the bulk
// copies it issues next.
__device__ __forceinline__ void fence_proxy_async_smem()
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// Index of each operand's tensor map among a member's NMAP maps (ensembles).
// FP64:      0 Y (halo box), 1 U0 (halo), 2 U1 (halo), 3 Y (tile), 4 A (tile), 5 U0 (tile)
// FP32-bulk: 0 current Y (halo), 1 D1 (halo), 2 D2 (halo), 3 D2 (tile), 5 D1 (tile), 6 D3 (halo),
//            7 current Y (halo) in the row count of stage 4
// (FV launches copy U0 at FP64 stage 3 and D1, D2 at FP32-bulk stage 4 row by row,
// without a map.)
template <bool INC, int STAGE> struct MapIdx {
    static constexpr int X = STAGE == 1 ? 0 : (STAGE == 3 ? 2 : (INC && STAGE == 4 ? 6 : 1));
    static constexpr int Y = INC ? (STAGE == 4 ? 7 : 0) : 3;
    static constexpr int A = INC ? 5 : (STAGE == 3 ? 5 : 4);
    static constexpr int B = 3;
};

// The operand maps of one launch: X (stage input with halo), Y, A and B (see
// the kernels' Layout; unused ones are ignored).
// chained: the launch follows another stage launch of the same call (launch_after).
struct StageMaps {
    const CUtensorMap *x, *y, *a, *b;
    bool chained;
};

}  // namespace tma

static_assert(sizeof(StageArgs) % 8 == 0, "StageArgs is copied to shared memory in 8-byte words");

// Ghost cells that hold output cell z of a tile under the periodic boundary
// (updateBufferZone, src/nuosc.hpp:212-278), written by the cell's own lane; `row`
// points at cell 0 of its row and component.
template <class TOUT>
__device__ __forceinline__ void periodic_ghosts(TOUT *row, const StageArgs &a, int z, TOUT u)
{
    if (z < a.H) row[z + a.nz] = u;
    if (z >= a.nz - a.H) row[z - a.nz] = u;
}

// Ghost cells of rows [v0, v1) that follow from a tile (at z0) at a row's end:
// periodic copies, or the open boundary's first cell on the left and running
// linear extrapolation on the right.  One thread per row and component, after a
// barrier behind the stores of the tile's cells: under the open boundary, written
// inside the chunk loop, one lane stored 4 cells of 8 components in turn while
// the stage waited (FD, 4000 x 100 cells: 139 us a step against 69 under the
// periodic one).  PERIODIC: the periodic copies too.
template <bool PERIODIC, class TOUT>
__device__ __forceinline__ void fill_ghosts(TOUT *U, const StageArgs &a, int v0, int v1, int z0,
                                            int tid, int nthr)
{
    // cells [s, s + n) copied to [d, d + n), four loads in flight
    auto copy = [](TOUT *row, int d, int s, int n) {
        for (int g = 0; g < n; g += 4) {
            TOUT x[4];
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (g + k < n) x[k] = row[s + g + k];
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (g + k < n) row[d + g + k] = x[k];
        }
    };
    const int zr = max(z0, a.nz - a.H);  // the tile's cells that wrap to the left
#pragma unroll 2
    for (int i = tid; i < (v1 - v0) * NCOMP; i += nthr) {
        TOUT *row = U + (i % NCOMP) * a.cs + (long long)(v0 + i / NCOMP) * a.ld + HP;
        if (PERIODIC && a.bc == 0) {
            if (z0 == 0) copy(row, a.nz, 0, a.H);
            copy(row, zr - a.nz, zr, min(z0 + tma::TZ, a.nz) - zr);
        } else {
            if (z0 == 0) {
                const TOUT x = row[0];
                for (int g = 1; g <= a.H; ++g) row[-g] = x;
            }
            if (z0 + tma::TZ >= a.nz) {
                TOUT p0 = row[a.nz - 2], p1 = row[a.nz - 1];
                for (int g = 0; g < a.H; ++g) {
                    const TOUT x = p1 * TOUT(2) - p0;
                    row[a.nz + g] = x;
                    p0 = p1;
                    p1 = x;
                }
            }
        }
    }
}

constexpr int TMA_SMEM_MAX = 232448;  // opt-in shared memory per block on sm_100
constexpr int TMA_SMEM_SM = 233472;   // shared memory per SM (1 KB reserved per block)

inline int tma_smem_limit(int minb)
{
    return minb == 1 ? TMA_SMEM_MAX : TMA_SMEM_SM / minb - 1024;
}

// FV launches (stage_fv.cu, FP32-bulk's in stage_fv32.cu); nblocks <= 0: sets the
// kernels' attributes.
cudaError_t launch_fv_tma(const tma::StageMaps &m, const StageArgs &a, int stage, int fp32, int *err,
                          int nblocks, cudaStream_t s, const BatchDev *bd);
cudaError_t launch_fv_bulk(const tma::StageMaps &m, const StageArgs &a, int stage, int *err,
                           int nblocks, cudaStream_t s, const BatchDev *bd);
int fv_blocks_per_sm();
int fv_box_x(int elem_bytes);

}  // namespace cosenu
