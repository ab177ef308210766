// TMA-pipelined RK4 stage kernel of the FV scheme (WENO7, src/rhs_fv.hpp:115-236),
// for single simulations of any size and for ensembles.
//
// Same arithmetic and epilogue as rk4_stage_kernel (stage.cu); what changes is
// how the work reaches the SM.  A block is persistent over work items, each a
// run of 8-row chunks of a 32-cell z tile (Seg; the last tile of a row may be
// partial).  Chunks of 8 rows x (32 + 2*4)
// cells of all 8 components of the stage input, and the matching cells of the operands the
// combine reads, stream into a ring of NBUF shared-memory buffers with
// cp.async.bulk.tensor (one 3-D tensor-map copy per operand and chunk); eight
// warps take one row each.  There is no producer warp: the last warp to
// release a buffer issues its next copies, so a block is 8 warps and two
// blocks per SM get 128 registers per thread.
//
// FP64 issue bounds this kernel (WENO7 on 8 components: about 500 of the 600
// FP64 operations per cell and stage), so a row is done in two phases.
//   Faces: a lane reconstructs four consecutive faces of one component from
//   twelve cells (six 16-byte shared loads), which share their second to
//   fourth differences and one division (weno.cuh), and leaves them in a 1 KB
//   slot of its warp; two passes of four components.
//   Cells: a lane takes one cell, its two faces per component, the source
//   terms, the stage combine, the stores and the moments.
// One face per lane and cell (shuffling for the neighbour's) cost 75 + 5
// operations a face instead of 55 + 5, and left each warp one dependent chain
// at a time: FP64 pipe 63 % busy.
//
// The upwind face at a tile's edge belongs to the neighbouring tile's cells:
// each chunk, two warps (in turn) compute all 64 of them (8 rows x 8
// components) at full lane occupancy and publish them in shared memory
// (s_edge, one mbarrier per ring buffer).
//
// The operands that only the combine reads and that would leave no room for
// two blocks per SM in the ring (U at FP64 stage 3, D1 and D2 at FP32-bulk
// stage 4) are copied by each warp for its own row into a single slot
// (cp.async at the start of the row, waited for after the face phase, which
// hides the copy; loads into registers stalled the face phase's own loads).
//
// A single simulation's tiles are cut along v into pieces of equal height
// (fv_piece_rows) where whole tiles would leave block slots empty; each item
// writes the moments of its piece, and the next stage sums a tile's pieces in
// order.  Items are dealt out along z within a v band, so that the blocks
// running together read neighbouring cells of the same rows: an even split into
// contiguous runs of chunks kept the slots fuller but read 256-byte fragments
// all over the state (nz 65536 x nvz 512: stage 1 1.62 -> 1.75 ms, stage 3
// 2.23 -> 2.80 ms).
//
// Every wait is bounded in time (globaltimer, limit StageArgs::wait_ns): on
// expiry the kernel records a code in *err and carries on along the same
// control path, so no barrier is left waiting and the host reports the error.
// After a failed wait a warp does not release its buffer, so the buffer's
// release count never completes and no warp refills it; before the block
// exits one thread waits (bounded again) for the copies in flight, so no block
// ends while a bulk copy still writes into its shared memory.
#pragma once

#include "tma.cuh"
#include "weno.cuh"

namespace cosenu {

namespace fv {

constexpr int R = 8;              // rows per chunk = warps per block
constexpr int NTHR = R * 32;
constexpr int NE = R * NCOMP / 32;  // edge warps per chunk
constexpr int FW = tma::TZ;       // doubles per component in a warp's face slot
constexpr int OWN = 2048;         // bytes per warp of an own-cell operand row
static_assert(R * NCOMP % 32 == 0 && (R & (R - 1)) == 0,
              "edge warps: whole warps, rows a power of two");

// Width of an input box row: the tile plus HALO cells each side, rounded up
// so that the row is a multiple of 16 bytes (TMA) and the 16-byte loads of a
// quarter-warp (4 quads of cells x 2 components, see quad_of) hit distinct
// banks: components 84 words (42 doubles) or 48 words (48 floats) apart.
template <class T> constexpr int xw() { return sizeof(T) == 8 ? 42 : 48; }

template <class TIN, class TOUT, int STAGE> struct Layout {
    static constexpr bool INC = inc_form<TIN, TOUT>();
    static constexpr int XW = xw<TIN>();
    static constexpr int XB = NCOMP * R * XW * (int)sizeof(TIN);
    // Y: FP64 stages 2-3 read it at their own cells; FP32-bulk stages 2-4 read
    // it with the halo (their input is Y + D)
    static constexpr int YW = INC ? (STAGE >= 2 ? xw<double>() : 0)
                                  : ((STAGE == 2 || STAGE == 3) ? tma::TZ : 0);
    static constexpr int YB = NCOMP * R * YW * 8;
    // FP64 stage 4: A at its own cells
    static constexpr int AB = (!INC && STAGE == 4) ? NCOMP * R * tma::TZ * 8 : 0;
    static constexpr int BUF = ((XB + YB + AB) + 127) / 128 * 128;
    // operands that each warp copies for its own row (single-buffered)
    static constexpr bool OWNED = INC ? STAGE == 4 : STAGE == 3;
    static_assert(XB % 128 == 0 && YB % 128 == 0, "TMA destinations 128-byte aligned");
    // shared memory after the ring (offsets in bytes)
    static constexpr int fixed(int nbuf)
    {
        return 2 * nbuf * 8                           // full, ebar
               + (1 + R) * NMOM * tma::TZ * 8         // s_mom, s_red
               + (int)sizeof(StageArgs)               // batched: current member
               + nbuf * R * NCOMP * 8                 // s_edge
               + R * 4 * FW * 8                       // s_face
               + (OWNED ? R * OWN : 0)                // s_own
               + nbuf * 8;                            // release counts, last chunks
    }
    static constexpr int smem(int nbuf) { return nbuf * BUF + fixed(nbuf); }
};

// The copies of one ring buffer, all completing on `bar`.
template <class L>
__device__ __forceinline__ void issue_chunk(unsigned char *buf, uint64_t *bar,
                                            const CUtensorMap *px, const CUtensorMap *py,
                                            const CUtensorMap *pa, int z0, int row0)
{
    tma::mbar_expect_tx(bar, L::XB + L::YB + L::AB);
    tma::tma_load_3d(buf, px, HP + z0 - tma::HALO, 0, row0, bar);
    if (L::YB)
        tma::tma_load_3d(buf + L::XB, py, HP + z0 - (L::INC ? tma::HALO : 0), 0, row0, bar);
    if (L::AB) tma::tma_load_3d(buf + L::XB + L::YB, pa, HP + z0, 0, row0, bar);
}

__device__ __forceinline__ void cp16(void *dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(tma::smem_u32(dst)), "l"(src)
                 : "memory");
}

// Position of face z of component k (of four) in a warp's face slot: the 16-byte
// pairs of odd components are swapped, so that the pairs a quarter-warp stores
// (every second pair of two components) fall in distinct banks.
__device__ __forceinline__ int face_at(int k, int z) { return k * FW + (z ^ ((k & 1) << 1)); }

__device__ __forceinline__ void load12(const double *p, double *x)
{
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        const double2 v = reinterpret_cast<const double2 *>(p)[i];
        x[2 * i] = v.x;
        x[2 * i + 1] = v.y;
    }
}

__device__ __forceinline__ void load12(const float *p, float *x)
{
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const float4 v = reinterpret_cast<const float4 *>(p)[i];
        x[4 * i] = v.x;
        x[4 * i + 1] = v.y;
        x[4 * i + 2] = v.z;
        x[4 * i + 3] = v.w;
    }
}

// One run of chunks of a tile: chunks [c0, c1) of z tile zt of member inst, the
// tile's moments in np pieces, this run the piece-th.
struct Seg {
    int inst, zt, c0, c1, piece, np;
};

// Item i of a single simulation: z tile i % nzt of v band i / nzt.
__device__ __forceinline__ Seg seg_of(int i, const StageArgs &a, int nzt)
{
    Seg s;
    s.inst = 0;
    s.piece = i / nzt;
    s.zt = i - s.piece * nzt;
    s.np = a.nvt;
    const int pc = (a.tv + R - 1) / R;
    s.c0 = s.piece * pc;
    s.c1 = min(s.c0 + pc, (a.nvz + R - 1) / R);
    return s;
}

// Ensemble table entry (batch.cu): member, z tile, c0 | c1 << 16, piece | np << 16.
__device__ __forceinline__ Seg seg_of(const int4 e)
{
    return Seg{e.x, e.y, e.z & 0xffff, e.z >> 16, e.w & 0xffff, e.w >> 16};
}

}  // namespace fv

// TIN: type of the streamed stage input (FP64: the stage value U or Y;
// FP32-bulk: Y at stage 1, the increment D after).  TOUT: type of the output
// (FP64: U', U'' or Y; FP32-bulk: D1, D2, D3, then the new Y).  The
// right-hand side is evaluated in FP64 in both forms, except the FP32-bulk
// WENO7 weights and candidates (FP32 on FP64 stencil differences).
// LARGE: the order of FP32-bulk's candidate sum (weno.cuh; FP64: true).
template <int STAGE, class TIN, class TOUT, int NBUF, bool BATCHED, int MINB, bool LARGE>
__global__ void __launch_bounds__(fv::NTHR, MINB)
    rk4_stage_fv_kernel(const __grid_constant__ CUtensorMap mX,
                        const __grid_constant__ CUtensorMap mY,
                        const __grid_constant__ CUtensorMap mA,
                        const __grid_constant__ StageArgs a0, int *err, const BatchDev bd)
{
    using namespace tma;
    using fv::R;
    using fv::NE;
    using fv::FW;
    using L = fv::Layout<TIN, TOUT, STAGE>;
    using MI = MapIdx<L::INC, STAGE>;
    constexpr bool INC = L::INC;
    constexpr bool YPLUS = INC && STAGE >= 2;  // the input is Y + D
    constexpr int XW = L::XW, YW = L::YW;
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char *s_own = smem + NBUF * L::BUF;  // [R][OWN]
    double(*s_face)[4 * FW] =
        reinterpret_cast<double(*)[4 * FW]>(s_own + (L::OWNED ? R * fv::OWN : 0));  // [R]
    double(*s_mom)[TZ] = reinterpret_cast<double(*)[TZ]>(s_face + R);                // [6][TZ]
    double(*s_red)[NMOM][TZ] = reinterpret_cast<double(*)[NMOM][TZ]>(s_mom + NMOM);       // [R]
    double(*s_edge)[R][NCOMP] = reinterpret_cast<double(*)[R][NCOMP]>(s_red + R);         // [NBUF]
    uint64_t *full = reinterpret_cast<uint64_t *>(s_edge + NBUF);
    uint64_t *ebar = full + NBUF;  // edge faces of buffer b published
    StageArgs *s_args = reinterpret_cast<StageArgs *>(ebar + NBUF);
    // per ring buffer, the warps' release count and the last chunk whose
    // copies went into it
    uint32_t *s_cnt = reinterpret_cast<uint32_t *>(s_args + 1);
    int *s_last = reinterpret_cast<int *>(s_cnt + NBUF);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // this block's items: every gridDim.x-th of a single simulation, or a run of
    // the ensemble table; chunk ch of the item at position p is the block's n-th
    // chunk, and its copies go into buffer n % NBUF
    const int nzt = (a0.nz + TZ - 1) / TZ;
    int p_first = blockIdx.x, p_end = BATCHED ? 0 : nzt * a0.nvt;
    const int p_step = BATCHED ? 1 : gridDim.x;
    auto seg_at = [&](int p) {
        if constexpr (BATCHED) return fv::seg_of(bd.table[p]);
        else return fv::seg_of(p, a0, nzt);
    };
    auto issue_at = [&](const fv::Seg &s, int ch, uint32_t n) {
        if (a0.stall) return;
        const int b = n % NBUF;
        if constexpr (BATCHED) {
            const CUtensorMap *m = &bd.maps[s.inst * NMAP];
            fv::issue_chunk<L>(smem + b * L::BUF, &full[b], &m[MI::X], &m[MI::Y], &m[MI::A],
                               s.zt * TZ, ch * R);
        } else {
            fv::issue_chunk<L>(smem + b * L::BUF, &full[b], &mX, &mY, &mA, s.zt * TZ, ch * R);
        }
        s_last[b] = (int)n;
    };
    // (p, s, ch) moved k chunks on; false past the block's last segment
    auto advance = [&](int &p, fv::Seg &s, int &ch, int k) -> bool {
        for (; k > 0; --k) {
            if (++ch == s.c1) {
                p += p_step;
                if (p >= p_end) return false;
                s = seg_at(p);
                ch = s.c0;
            }
        }
        return true;
    };
    // moment m of cell zz of a segment's tile: its pieces in order
    auto moment_in = [&](const fv::Seg &s, int m, int zz) {
        const StageArgs &a = BATCHED ? bd.args[s.inst * 4 + STAGE - 1] : a0;
        double x = 0.0;
        if ((a.flags & F_COLL) && s.zt * TZ + zz < a.nz) {
            const double *q = a.Min + (long long)m * a.nz + s.zt * TZ + zz;
            const long long st = (long long)NMOM * a.nz;
            x = q[0];
            for (int k = 1; k < s.np; k += 8) {  // eight loads in flight
                double y[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) y[j] = k + j < s.np ? q[(k + j) * st] : 0.0;
#pragma unroll
                for (int j = 0; j < 8; ++j) x += y[j];
            }
        }
        return x;
    };

    if (tid == 0) {
        if constexpr (!BATCHED) {
            prefetch_map(&mX);
            if (L::YB) prefetch_map(&mY);
            if (L::AB) prefetch_map(&mA);
        }
        for (int b = 0; b < NBUF; ++b) {
            mbar_init(&full[b], 1);
            mbar_init(&ebar[b], NE * 32);
            s_cnt[b] = 0;
            s_last[b] = -1;
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if constexpr (BATCHED) {
        p_first = bd.range[blockIdx.x];
        p_end = bd.range[blockIdx.x + 1];
    }
    fv::Seg cur{0, 0, 0, 0, 0, 0};
    if (p_first < p_end) cur = seg_at(p_first);
    double vz_l = 0.0, fac_l = 0.0;  // row values, see the chunk loop
    auto load_rows = [&](const StageArgs &a, int ch) {
        const int vl = min((ch + lane) * R + warp, a.nvz - 1);
        vz_l = __ldg(&a.vz[vl]);
        fac_l = __ldg(&a.rowfac[vl]);
    };
    if (!BATCHED) load_rows(a0, cur.c0);
    previous_launch();  // (what is read above, no stage writes)
    if (tid == 0 && p_first < p_end) {
        int p = p_first;
        fv::Seg s = cur;
        int ch = s.c0;
        for (uint32_t n = 0; n < (uint32_t)NBUF; ++n) {
            issue_at(s, ch, n);
            if (!advance(p, s, ch, 1)) break;
        }
    }
    // moments of the stage input for the first tile (not by the issuing warp)
    static_assert(NMOM < R, "one warp per moment, after warp 0");
    if (p_first < p_end && warp >= 1 && warp <= NMOM)
        s_mom[warp - 1][lane] = moment_in(cur, warp - 1, lane);
    __syncthreads();

    // face phase: this lane's quad of cells and its component (of four per
    // pass).  A quarter-warp covers quads 0-3 or 4-7 of two components, which
    // keeps its 16-byte loads and stores free of bank conflicts.
    const int qz = 4 * ((lane & 3) | ((lane >> 1) & 4));   // first cell of the quad
    const int qc = ((lane >> 2) & 1) | ((lane >> 3) & 2);  // component within the pass

    uint32_t it = 0;
    int s_inst = -1;  // member whose arguments s_args holds
    for (int p = p_first; p < p_end;) {
        const int inst = cur.inst;
        const int pn = p + p_step;
        const fv::Seg nxt = pn < p_end ? seg_at(pn) : cur;
        if (BATCHED && inst != s_inst) {
            // a new member: its arguments into shared memory.  Read from there
            // (like a0 from parameter space) they cost no registers across the
            // chunk loop and cannot alias the stores to U and A.  The previous
            // segment's epilogue ended with a barrier.
            if (tid < (int)(sizeof(StageArgs) / 8))
                reinterpret_cast<long long *>(s_args)[tid] =
                    reinterpret_cast<const long long *>(&bd.args[inst * 4 + STAGE - 1])[tid];
            __syncthreads();
            s_inst = inst;
        }
        const StageArgs &a = BATCHED ? *s_args : a0;
        const bool coll = (a.flags & F_COLL) != 0;
        const bool advec = (a.flags & F_ADVEC_OFF) == 0;
        const bool open_bc = a.bc != 0;
        const int z0 = cur.zt * TZ;
        const int z = z0 + lane;
        const bool inz = z < a.nz;  // (the last tile of a row may be partial)
        // the next segment's input moments, in a register until the epilogue
        const bool new_tile = nxt.inst != inst || nxt.zt != cur.zt;
        double mnext = 0.0;
        if (tid < NMOM * TZ && new_tile) mnext = moment_in(nxt, tid / TZ, tid % TZ);
        // this warp's moment slots (the previous segment's epilogue has read them)
#pragma unroll
        for (int m = 0; m < NMOM; ++m) s_red[warp][m][lane] = 0.0;

        if (BATCHED || p != p_first) load_rows(a, cur.c0);  // (the first: above)
        for (int ch = cur.c0; ch < cur.c1; ++ch, ++it) {
            const int b = it % NBUF;
            const int v = ch * R + warp;
            const bool valid = v < a.nvz;
            const int vr = valid ? v : a.nvz - 1;
            const long long ro = (long long)vr * a.ld + HP;
            // this row's velocity and advection factor from the host tables:
            // lane l holds those of the warp's row l chunks after chunk c0 + 32 k
            const int cl = (ch - cur.c0) % 32;
            if (cl == 0 && ch != cur.c0) load_rows(a, ch);
            const double vzv = __shfl_sync(0xffffffffu, vz_l, cl);
            const double factor = __shfl_sync(0xffffffffu, fac_l, cl);
            if constexpr (L::OWNED) {
                // the combine's own operands, for after the face phase
                unsigned char *own = s_own + warp * fv::OWN;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int n = lane + 32 * i;  // 16-byte piece of the row
                    if constexpr (INC) {
                        const float *T = (i < 2 ? a.T1 : a.T2) + ((n >> 3) & 7) * a.cs + ro + z0;
                        fv::cp16(own + 16 * n, T + 4 * (n & 7));
                    } else {
                        const double *U0 = static_cast<const double *>(a.U) + (n >> 4) * a.cs;
                        fv::cp16(own + 16 * n, U0 + ro + z0 + 2 * (n & 15));
                    }
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
            }
            const bool landed = mbar_wait(&full[b], (it / NBUF) & 1, err, 2, a0.wait_ns);
            const unsigned char *buf = smem + b * L::BUF;
            // cell 0 of component 0 of row r in the input boxes (HALO cells each
            // side); a row's components are XW (YW) cells apart
            auto xrow_of = [&](int r) {
                return reinterpret_cast<const TIN *>(buf) + r * (NCOMP * XW) + HALO;
            };
            auto yrow_of = [&](int r) {
                return reinterpret_cast<const double *>(buf + L::XB) + r * (NCOMP * YW) +
                       (INC ? HALO : 0);
            };
            const TIN *xrow = xrow_of(warp);
            const double *yrow = yrow_of(warp);
            const int dir = (vzv >= 0.0) ? 1 : -1;
            const double sfac = dir > 0 ? factor : -factor;

            double o[NCOMP];
            if (advec) {
                // edge faces of this chunk: warps 2ch, 2ch + 1 (mod R) in turn,
                // lane -> (row 4h + lane / 8, component lane % 8)
                const int h = (warp - NE * ch) & (R - 1);
                if (h < NE) {
                    const int r = h * (32 / NCOMP) + (lane >> 3), q = lane & (NCOMP - 1);
                    // the row's velocity as in the host table (same operations)
                    const double ve = __dadd_rn(
                        a.v0, __dmul_rn(__dadd_rn((double)min(ch * R + r, a.nvz - 1), 0.5), a.dv));
                    const int s = ve >= 0.0 ? 1 : -1;
                    const int je = s > 0 ? -1 : TZ;
                    const TIN *x = xrow_of(r) + q * XW + je;
                    const double *y = yrow_of(r) + q * YW + je;
                    if constexpr (INC) {
                        auto dif = [&](int n) {  // u(je + n s) - u(je)
                            return YPLUS ? (float)(y[n * s] - y[0]) + ((float)x[n * s] - (float)x[0])
                                         : (float)((double)x[n * s] - (double)x[0]);
                        };
                        const float f = weno7_inc<LARGE>(dif(-3), dif(-2), dif(-1), dif(1), dif(2),
                                                         dif(3), YPLUS ? (float)x[0] : 0.f);
                        s_edge[b][r][q] = (YPLUS ? y[0] : (double)x[0]) + (double)f;
                    } else {
                        double dl[6];
#pragma unroll
                        for (int k = 0; k < 6; ++k)
                            dl[k] = (double)x[(k - 2) * s] - (double)x[(k - 3) * s];
                        s_edge[b][r][q] = __fma_rn(weno7_corr12(dl), 1.0 / 12.0, (double)x[0]);
                    }
                    mbar_arrive(&ebar[b]);
                }
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    // four faces of component 4p + qc
                    const int q = 4 * p + qc;
                    double f[4];
                    if constexpr (INC) {
                        float xs[12] = {0.f}, c[4];
                        double ys[12];
                        if constexpr (YPLUS) {
                            fv::load12(yrow + q * YW + qz - HALO, ys);
                            fv::load12(xrow + q * XW + qz - HALO, xs);
                        } else {
                            fv::load12(xrow + q * XW + qz - HALO, ys);
                        }
                        auto dif = [&](int i, int j) {
                            const float e = (float)(ys[j] - ys[i]);
                            return YPLUS ? e + (xs[j] - xs[i]) : e;
                        };
                        weno7_inc_quad<LARGE>(dif, dir, xs + 4, c);
#pragma unroll
                        for (int k = 0; k < 4; ++k) f[k] = ys[k + 4] + (double)c[k];
                    } else {
                        double xs[12], dl[9], c[4];
                        fv::load12(xrow + q * XW + qz - HALO, xs);
                        if (dir > 0) {
#pragma unroll
                            for (int k = 0; k < 9; ++k) dl[k] = xs[k + 2] - xs[k + 1];
                            weno7_quad(dl, c);
                        } else {
                            double cr[4];
#pragma unroll
                            for (int k = 0; k < 9; ++k) dl[k] = xs[9 - k] - xs[10 - k];
                            weno7_quad(dl, cr);
#pragma unroll
                            for (int k = 0; k < 4; ++k) c[k] = cr[3 - k];
                        }
#pragma unroll
                        for (int k = 0; k < 4; ++k) f[k] = __fma_rn(c[k], 1.0 / 12.0, (double)xs[k + 4]);
                    }
                    double *w = s_face[warp];
                    *reinterpret_cast<double2 *>(w + fv::face_at(qc, qz)) = make_double2(f[0], f[1]);
                    *reinterpret_cast<double2 *>(w + fv::face_at(qc, qz + 2)) =
                        make_double2(f[2], f[3]);
                    __syncwarp();
                    if (p == 0) mbar_wait(&ebar[b], (it / NBUF) & 1, err, 2, a0.wait_ns);
                    // upwind flux difference (rhs_fv.hpp:143-162) of this lane's
                    // cell; the face at the tile's upwind edge comes from s_edge
                    const int nb = lane - dir;
                    const bool edge = nb < 0 || nb >= TZ;
                    const double *eb = s_edge[b][warp] + 4 * p;
                    const double *p0 = edge ? eb : w + fv::face_at(0, nb);
                    const double *p1 = edge ? eb + 1 : w + fv::face_at(1, nb);
                    const int step = edge ? 2 : 2 * FW;
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const double fown = w[fv::face_at(k, lane)];
                        double fnb = (k & 1 ? p1 : p0)[(k >> 1) * step];
                        if (open_bc) {
                            // flux ghosts under OPEN_BC (updateBufferZone on rflux/lflux,
                            // rhs_fv.hpp:118-119): rflux[-1] = rflux[0],
                            // lflux[nz] = 2 lflux[nz-1] - lflux[nz-2]
                            if (dir > 0 && z == 0) fnb = fown;
                            if (dir < 0 && z == a.nz - 1)
                                fnb = fown * 2.0 - w[fv::face_at(k, lane - 1)];
                        }
                        o[4 * p + k] = sfac * (fown - fnb);
                    }
                    __syncwarp();
                }
            } else {
                // the edge warps arrive all the same, so that the barrier's phases
                // follow the ring: an ensemble's block may go on to a member that
                // advects
                if (((warp - NE * ch) & (R - 1)) < NE) mbar_arrive(&ebar[b]);
#pragma unroll
                for (int q = 0; q < NCOMP; ++q) o[q] = 0.0;
            }

            double c[NCOMP];
#pragma unroll
            for (int q = 0; q < NCOMP; ++q)
                c[q] = YPLUS ? yrow[q * YW + lane] + (double)xrow[q * XW + lane]
                             : (double)xrow[q * XW + lane];
            if (a.flags & F_VAC) {
                // read where used: batched, a is in shared memory and a
                // per-tile copy would hold registers across the chunk loop
                const double pmo = a.pmo, ct = a.ct, st = a.st;
                o[EE] += -2.0 * st * c[EXI] * pmo;
                o[XX] += 2.0 * st * c[EXI] * pmo;
                o[EXR] += -2.0 * ct * c[EXI] * pmo;
                o[EXI] += (2.0 * ct * c[EXR] + st * (c[EE] - c[XX])) * pmo;
                o[BEE] += -2.0 * st * c[BEXI] * pmo;
                o[BXX] += 2.0 * st * c[BEXI] * pmo;
                o[BEXR] += -2.0 * ct * c[BEXI] * pmo;
                o[BEXI] += (2.0 * ct * c[BEXR] + st * (c[BEE] - c[BXX])) * pmo;
            }
            if (a.flags & F_MAT) {
                const double hm = a.Hm[min(z, a.nz - 1)];
                o[EXR] += hm * c[EXI];
                o[EXI] += -hm * c[EXR];
                o[BEXR] += -hm * c[BEXI];
                o[BEXI] += hm * c[BEXR];
            }
            if (coll) {
                // this tile's input moments, read where used (they stay in
                // shared memory until the tile epilogue replaces them)
                const double mudv = a.mu * a.dv;
                const double SA = s_mom[0][lane] - vzv * s_mom[3][lane],
                             SB = s_mom[1][lane] - vzv * s_mom[4][lane],
                             SC = s_mom[2][lane] - vzv * s_mom[5][lane];
                const double Iee = 2.0 * (c[EXR] * SA - c[EXI] * SB);
                const double Ibee = 2.0 * (c[BEXR] * SA + c[BEXI] * SB);
                o[EE] += mudv * Iee;
                o[XX] += mudv * (-Iee);
                o[EXR] += mudv * ((c[XX] - c[EE]) * SA + c[EXI] * SC);
                o[EXI] += mudv * (-(c[XX] - c[EE]) * SB - c[EXR] * SC);
                o[BEE] += mudv * Ibee;
                o[BXX] += mudv * (-Ibee);
                o[BEXR] += mudv * ((c[BXX] - c[BEE]) * SA - c[BEXI] * SC);
                o[BEXI] += mudv * ((c[BXX] - c[BEE]) * SB + c[BEXR] * SC);
            }

            if constexpr (L::OWNED) {
                asm volatile("cp.async.wait_group 0;" ::: "memory");
                __syncwarp();
            }
            // stage combine.  FP64 (stage values, A written once by stage 3 from
            // U, U' and Y) or FP32-bulk (increments, common.cuh).
            const double dt = a.dt;
            // own-cell tiles: [row][component][TZ cells]
            const double *ys =
                reinterpret_cast<const double *>(buf + L::XB) + warp * (NCOMP * TZ) + lane;
            const double *as =
                reinterpret_cast<const double *>(buf + L::XB + L::YB) + warp * (NCOMP * TZ) + lane;
            const double *u0 =  // FP64 stage 3: U, about to be overwritten by U''
                reinterpret_cast<const double *>(s_own + warp * fv::OWN) + lane;
            const float *d12 =  // FP32-bulk stage 4: D1, then D2
                reinterpret_cast<const float *>(s_own + warp * fv::OWN) + lane;
            TOUT u[NCOMP];
            double anew[NCOMP];  // FP64 stage 3: the accumulator
            double um[NCOMP];    // the output as a stage value (for the moments)
#pragma unroll
            for (int q = 0; q < NCOMP; ++q) {
                const double kk = o[q];
                if constexpr (INC) {
                    // the base state at this cell: stage 1 reads Y itself
                    const double y = STAGE == 1 ? c[q] : yrow[q * YW + lane];
                    if (STAGE <= 3) {
                        u[q] = (TOUT)((STAGE == 3 ? dt : 0.5 * dt) * kk);
                        um[q] = y + (double)u[q];
                    } else {
                        const double d3 = (double)xrow[q * XW + lane];
                        const double d1 = (double)d12[q * TZ], d2 = (double)d12[(NCOMP + q) * TZ];
                        const double yn = y + (d1 + 2.0 * d2 + d3) * (1.0 / 3.0) + (dt / 6.0) * kk;
                        u[q] = (TOUT)yn;
                        um[q] = yn;
                    }
                } else {
                    if (STAGE == 1) {
                        u[q] = (TOUT)(c[q] + (0.5 * dt) * kk);
                    } else if (STAGE == 2 || STAGE == 3) {
                        const double y = ys[q * TZ];
                        u[q] = (TOUT)(y + (STAGE == 2 ? 0.5 * dt : dt) * kk);
                        if (STAGE == 3)
                            anew[q] = y + (u0[q * TZ] - y) * (1.0 / 3.0) + (c[q] - y) * (2.0 / 3.0) +
                                      (dt / 3.0) * kk;
                    } else {
                        u[q] = (TOUT)(as[q * TZ] + (dt / 6.0) * kk);
                    }
                    um[q] = (double)u[q];
                }
            }
            // this warp is done with the buffer (after a failed wait it keeps it:
            // the count never completes and no warp refills the buffer)
            __syncwarp();
            if (lane == 0 && landed &&
                ring_release_count(&s_cnt[b]) == (it / NBUF) * R + (R - 1)) {
                // the last of the R warps to release buffer b: its next chunk
                fence_proxy_async_smem();
                int p2 = p;
                fv::Seg s2 = cur;
                int ch2 = ch;
                if (advance(p2, s2, ch2, NBUF)) issue_at(s2, ch2, it + NBUF);
            }

            if (valid) {  // (uniform over the warp)
                TOUT *row = static_cast<TOUT *>(a.U) + ro;
#pragma unroll
                for (int q = 0; q < NCOMP; ++q) {
                    if (inz) {
                        row[q * a.cs + z] = u[q];
                        if (!INC && STAGE == 3) a.A[q * a.cs + ro + z] = anew[q];
                    }
                }
                if (coll && inz) {
                    const double Am = um[EXI] + um[BEXI];
                    const double Bm = um[EXR] - um[BEXR];
                    const double Cm = um[EE] - um[XX] - um[BEE] + um[BXX];
                    s_red[warp][0][lane] += Am;
                    s_red[warp][1][lane] += Bm;
                    s_red[warp][2][lane] += Cm;
                    s_red[warp][3][lane] += vzv * Am;
                    s_red[warp][4][lane] += vzv * Bm;
                    s_red[warp][5][lane] += vzv * Cm;
                }
            }
        }
        // ghost cells (written by the cells' own lanes in the chunk loop, periodic
        // ones too cost every tile: nz 65536 x nvz 512 7.33 -> 7.70 ms a step)
        if (z0 == 0 || z0 + TZ > a.nz - a.H) {
            __syncthreads();
            fill_ghosts<true>(static_cast<TOUT *>(a.U), a, cur.c0 * R, min(cur.c1 * R, a.nvz), z0, tid,
                        fv::NTHR);
        }
        if (pn >= p_end) next_launch();  // (chain.cuh)
        // segment epilogue: its output moments (fixed-order sum over warps) and
        // the next segment's input moments
        if (coll || BATCHED) {
            __syncthreads();
            if (tid < NMOM * TZ) {
                const int m = tid / TZ, zz = tid % TZ;
                double s = 0.0;
#pragma unroll
                for (int w = 0; w < R; ++w) s += s_red[w][m][zz];
                if (coll && z0 + zz < a.nz)
                    a.Mout[(long long)(cur.piece * NMOM + m) * a.nz + z0 + zz] = s;
                if (new_tile) s_mom[m][zz] = mnext;  // every warp read this tile's values above
            }
            __syncthreads();
        }
        p = pn;
        cur = nxt;
    }
    // the last copies issued into each buffer have landed before the block
    // exits (in normal operation the warps have waited for them)
    __syncthreads();
    if (tid == 0)
        for (int b = 0; b < NBUF; ++b)
            if (s_last[b] >= 0)
                mbar_drain(&full[b], ((uint32_t)s_last[b] / NBUF) & 1, err, a0.wait_ns);
}

// ---------------------------------------------------------------------------
// host side

template <int STAGE, class TIN, class TOUT, int NB, int MINB>
inline cudaError_t launch_nb(const tma::StageMaps &m, const StageArgs &a, int *err, int nblocks,
                             cudaStream_t s, const BatchDev *bd)
{
    constexpr bool INC = inc_form<TIN, TOUT>();
    auto kern = rk4_stage_fv_kernel<STAGE, TIN, TOUT, NB, false, MINB, true>;
    auto kernb = rk4_stage_fv_kernel<STAGE, TIN, TOUT, NB, true, MINB, true>;
    if (INC && (a.flags & F_SMALL)) kern = rk4_stage_fv_kernel<STAGE, TIN, TOUT, NB, false, MINB, !INC>;
    if (nblocks <= 0) {  // preparation call: shared-memory limit and carveout (bd: both kernels)
        for (auto k : {kern, kernb}) {
            if (k == kernb && !bd) continue;
            cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 TMA_SMEM_MAX);
            if (e == cudaSuccess)
                e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout,
                                         (int)cudaSharedmemCarveoutMaxShared);
            if (e != cudaSuccess) return e;
        }
        return cudaSuccess;
    }
    constexpr int shmem = fv::Layout<TIN, TOUT, STAGE>::smem(NB);
    return launch_after(m.chained, bd ? kernb : kern, nblocks, fv::NTHR, shmem, s, *m.x, *m.y, *m.a,
                        a, err, bd ? *bd : BatchDev{});
}

template <int STAGE, class TIN, class TOUT>
inline cudaError_t launch_one(const tma::StageMaps &m, const StageArgs &a, int *err, int nblocks,
                              cudaStream_t s, const BatchDev *bd)
{
    using L = fv::Layout<TIN, TOUT, STAGE>;
    constexpr int lim = TMA_SMEM_SM / 2 - 1024;
    constexpr int NB2 = L::smem(4) <= lim ? 4 : (L::smem(3) <= lim ? 3 : 2);
    static_assert(L::smem(2) <= lim, "two blocks per SM");
    constexpr int NB1 = L::smem(4) <= TMA_SMEM_MAX ? 4 : 3;
    if (fv_blocks_per_sm() == 1) return launch_nb<STAGE, TIN, TOUT, NB1, 1>(m, a, err, nblocks, s, bd);
    return launch_nb<STAGE, TIN, TOUT, NB2, 2>(m, a, err, nblocks, s, bd);
}

}  // namespace cosenu
