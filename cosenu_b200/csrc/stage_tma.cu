// TMA-pipelined RK4 stage kernel of the FD scheme (src/rhs_fd.hpp:6-148); the
// FV scheme's is stage_fv.cuh.
//
// Same arithmetic and epilogue as rk4_stage_kernel (stage.cu); what changes
// is how the operands reach the SM.  Each block is persistent over work items:
// z tiles of 32 cells (the last of a row may be partial) that span all nvz
// rows, or v bands of them where whole tiles would leave SMs idle
// (fd_piece_rows; an item then writes the moments of its band, and the next
// stage sums a tile's bands in order).  One producer warp streams chunks of 8 (or
// 12) rows x (32 + 2*4) cells of all 8 components of the stage input, and the
// matching cells of Y and A, into a ring of NBUF shared-memory buffers with
// cp.async.bulk.tensor (one 3-D tensor-map copy per operand and chunk, box
// {cells, components, rows}); the consumer warps take one row each, read
// their stencil from shared memory and write the results with coalesced
// stores.  Full/empty mbarriers order the ring.  With up to NBUF-1 chunks in
// flight (~100 KB per SM) the kernel keeps HBM busy without depending on
// occupancy, which the register-heavy FP64 right-hand side limits.  One block
// per SM.  Per-row velocities and advection factors equal the host's tables
// (src/nuosc.hpp:88-92, rhs_fd.hpp:57) and are recomputed in registers.
//
// The common variant of manage.py (central FD4 + KO3) is a compile-time fast
// path; the upwind / lopsided / KO5 variants take the generic path.
//
// Every wait is bounded in time (globaltimer, limit StageArgs::wait_ns): on
// expiry the kernel records a code in *err and carries on along the same
// control path, so no barrier is left waiting and the host reports the error.
// After a failed wait a consumer warp does not release its buffer, so the
// producer's next wait on that buffer fails too and it stops issuing copies;
// before the block exits it waits (bounded again) for the copies in flight, so
// no block ends while a bulk copy still writes into its shared memory.
#include <algorithm>
#include <cstdlib>

#include "tma.cuh"

namespace cosenu {

namespace tma {

// Width of an input box row: the tile plus HALO cells each side, rounded up so
// that the row is a multiple of 16 bytes (TMA).
template <class T> constexpr int xw() { return sizeof(T) == 8 ? 42 : 44; }
// v rows per chunk = consumer warps.  The stages that move few bytes per cell
// (FP64 stage 1, FP32-bulk stages 1-3) are bound by latency and run 12 (13
// warps, ~126 registers, no spills: 0.230 -> 0.205 ms for FP64 stage 1 at nz
// 32768 x nvz 256); the HBM-bound stages keep 8, whose smaller chunks keep
// fewer bytes in flight (12 rows: FP64 stage 3 0.436 -> 0.490 ms).
template <int STAGE, bool INC> constexpr int rows()
{
    return ((!INC && STAGE == 1) || (INC && STAGE <= 3)) ? 12 : 8;
}

// One ring buffer holds, for R rows, boxes laid out [row][component][cell]
// (the tensor maps put components before rows): the input box X, then Y, then
// the own-cell tiles A (and B).
template <class TIN, class TOUT, int STAGE> struct Layout {
    static constexpr bool INC = inc_form<TIN, TOUT>();
    static constexpr int R = rows<STAGE, INC>();
    static constexpr int NTHR = R * 32 + 32;  // consumer warps + producer warp
    // FP64 stage 3 streams the most bytes per chunk: its 40-cell rows keep a
    // two-buffer ring within half an SM's shared memory (two blocks per SM)
    static constexpr int XW = (!INC && STAGE == 3) ? TZ + 2 * HALO : xw<TIN>();
    static constexpr int XB = NCOMP * R * XW * (int)sizeof(TIN);
    // Y: FP64 stages 2-3 read it at their own cells; FP32-bulk stages 2-4 read
    // it with the halo (their input is Y + D)
    static constexpr int YW =
        INC ? (STAGE >= 2 ? xw<double>() : 0) : ((STAGE == 2 || STAGE == 3) ? TZ : 0);
    static constexpr int YB = NCOMP * R * YW * 8;
    // FP64 stage 3: U at its own cells (about to be overwritten by U''); stage
    // 4: A.  FP32-bulk stage 4: D1 then D2 at its own cells.
    static constexpr int AB = INC ? (STAGE == 4 ? 2 * NCOMP * R * TZ * 4 : 0)
                                  : (STAGE >= 3 ? NCOMP * R * TZ * 8 : 0);
    static constexpr int BUF = ((XB + YB + AB) + 127) / 128 * 128;
    // output moments: registers per warp, paired at the tile's end
    static constexpr int NRED = R / 2;  // moment slots in shared memory
};

// The copies of one ring buffer: the stage input box (X) and, where the
// stage reads them, Y and the own-cell tiles A (and B), all completing on
// `bar`.  Coordinates: (cell, component 0, first row of the chunk).
template <class L>
__device__ __forceinline__ void issue_chunk(unsigned char *buf, uint64_t *bar, const CUtensorMap *px,
                                            const CUtensorMap *py, const CUtensorMap *pa,
                                            const CUtensorMap *pb, int z0, int row0)
{
    mbar_expect_tx(bar, L::XB + L::YB + L::AB);
    tma_load_3d(buf, px, HP + z0 - HALO, 0, row0, bar);
    if (L::YB) tma_load_3d(buf + L::XB, py, HP + z0 - (L::INC ? HALO : 0), 0, row0, bar);
    if (L::AB && !L::INC) tma_load_3d(buf + L::XB + L::YB, pa, HP + z0, 0, row0, bar);
    if (L::AB && L::INC) {
        tma_load_3d(buf + L::XB + L::YB, pa, HP + z0, 0, row0, bar);
        tma_load_3d(buf + L::XB + L::YB + L::AB / 2, pb, HP + z0, 0, row0, bar);
    }
}

}  // namespace tma

// Work item: z tile zt of member inst, rows [v0, v1), v band vt of nvt.
struct FdItem {
    int inst, zt, v0, v1, vt, nvt;
};

// FD: velocity and advection factor of row i, recomputed with round-to-nearest
// operations so the bits equal the host tables (capi.cu, src/nuosc.hpp:88-92,
// rhs_fd.hpp:57).  The FD stages are bound by memory latency, and a table load
// per chunk slowed them (FP64 stages 1, 2, 4 at nz 32768 x nvz 256 by 8 %).
__device__ __forceinline__ void fd_row_values(double v0, double dv, double dz, int fd_advec, int i,
                                              double &v, double &f)
{
    v = __dadd_rn(v0, __dmul_rn(__dadd_rn((double)i, 0.5), dv));
    const double sv = (double)((0.0 < v) - (v < 0.0));
    const double d12 = __dmul_rn(12.0, dz);
    if (fd_advec == 0) f = __ddiv_rn(-v, d12);                      // centre
    else if (fd_advec == 1) f = __ddiv_rn(__dmul_rn(-sv, v), d12);  // upwind
    else f = __ddiv_rn(__dmul_rn(sv, v), d12);                       // lopsided
}

// Weights of one row's combined advection (src/rhs_fd.hpp:53-73) and
// Kreiss-Oliger (:128-145) stencil for the neighbours -1 .. -T, then +1 .. +T
// (T = 2: central FD4 + KO3; T = 3: any).  One difference and one multiply-add
// per neighbour; the separate stencils, with the upwind side indexed by sign(v)
// and a branch per component and variant, took 96-99 us a step on 4000 x 100
// cells where the central one took 69.
template <bool GEN>
__device__ __forceinline__ void fd_weights(const StageArgs &a, double v, double f, double *w)
{
    const double e = a.ko_eps;
    if constexpr (!GEN) {
        w[0] = -8.0 * f - 4.0 * e;
        w[1] = f + e;
        w[2] = 8.0 * f - 4.0 * e;
        w[3] = e - f;
    } else {
        const bool k5 = a.ko_order == 5;
        const double e1 = k5 ? 15.0 * e : -4.0 * e, e2 = k5 ? -6.0 * e : e, e3 = k5 ? e : 0.0;
        if (a.fd_advec == 0) {
            w[0] = e1 - 8.0 * f;
            w[1] = e2 + f;
            w[2] = e3;
            w[3] = e1 + 8.0 * f;
            w[4] = e2 - f;
            w[5] = e3;
        } else {
            // weights of the upwind neighbours 1 .. 3 and the downwind one
            const bool up = a.fd_advec == 1;
            const double u1 = e1 + (up ? -36.0 : 18.0) * f, u2 = e2 + (up ? 18.0 : -6.0) * f,
                         u3 = e3 + (up ? -4.0 : 1.0) * f, d1 = e1 + (up ? 0.0 : -3.0) * f;
            const bool left = v > 0.0;  // (v = 0: f = 0, both sides alike)
            w[0] = left ? u1 : d1;
            w[1] = left ? u2 : e2;
            w[2] = left ? u3 : e3;
            w[3] = left ? d1 : u1;
            w[4] = left ? e2 : u2;
            w[5] = left ? e3 : u3;
        }
    }
}

// TIN: type of the streamed stage input (FP64: the stage value U or Y;
// FP32-bulk: Y at stage 1, the increment D after).  TOUT: type of the output
// (FP64: U', U'' or Y; FP32-bulk: D1, D2, D3, then the new Y).  The
// right-hand side is evaluated in FP64 in both forms.
template <bool GEN, int STAGE, class TIN, class TOUT, int NBUF, bool BATCHED, int MINB>
__global__ void __launch_bounds__(tma::Layout<TIN, TOUT, STAGE>::NTHR, MINB)
    rk4_stage_tma_kernel(const __grid_constant__ CUtensorMap mX,
                         const __grid_constant__ CUtensorMap mY,
                         const __grid_constant__ CUtensorMap mA,
                         const __grid_constant__ CUtensorMap mB,
                         const __grid_constant__ StageArgs a0, int *err, const BatchDev bd)
{
    using namespace tma;
    using L = Layout<TIN, TOUT, STAGE>;
    constexpr int R = L::R;
    auto consumer_sync = tma::consumer_sync<R * 32>;
    using MI = MapIdx<L::INC, STAGE>;
    constexpr bool INC = L::INC;
    extern __shared__ __align__(1024) unsigned char smem[];
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + NBUF * L::BUF);
    uint64_t *empty = full + NBUF;
    double(*s_mom)[TZ] = reinterpret_cast<double(*)[TZ]>(empty + NBUF);  // [6][TZ]
    double(*s_red)[NMOM][TZ] = reinterpret_cast<double(*)[NMOM][TZ]>(s_mom + NMOM);  // [NRED]
    StageArgs *s_args = reinterpret_cast<StageArgs *>(s_red + L::NRED);  // batched: current member
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // a single simulation's items: all z tiles of a v band, then the next band's
    const int nzt = BATCHED ? 1 : (a0.nz + TZ - 1) / TZ;
    const int nitems = BATCHED ? bd.ntiles : nzt * a0.nvt;
    auto item_at = [&](int t) {
        FdItem i;
        if constexpr (BATCHED) {
            const int4 e = bd.table[t];  // (member, z tile, -, rows)
            i = FdItem{e.x, e.y, 0, e.w, 0, 1};
        } else {
            i.inst = 0;
            i.vt = t / nzt;
            i.zt = t - i.vt * nzt;
            i.nvt = a0.nvt;
            i.v0 = i.vt * a0.tv;
            i.v1 = min(i.v0 + a0.tv, a0.nvz);
        }
        return i;
    };

    if (tid == 0) {
        if constexpr (!BATCHED) {
            tma::prefetch_map(&mX);
            if (L::YB) tma::prefetch_map(&mY);
            if (L::AB) tma::prefetch_map(&mA);
            if (INC && L::AB) tma::prefetch_map(&mB);
        }
        for (int b = 0; b < NBUF; ++b) {
            tma::mbar_init(&full[b], 1);
            tma::mbar_init(&empty[b], R);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    previous_launch();  // (all threads: the producer's copies, the consumers' loads and stores)

    if (warp == R) {
        // ------------------------------------------------------------ producer
        if (lane == 0 && !a0.stall) {
            uint32_t it = 0;
            bool issuing = true;  // false once a wait has failed: no further copies
            const bool rr = !BATCHED || bd.range == nullptr;  // interleaved tiles
            const int t_first = rr ? blockIdx.x : bd.range[blockIdx.x];
            const int t_end = rr ? nitems : bd.range[blockIdx.x + 1];
            const int t_step = rr ? gridDim.x : 1;
            // items are read one ahead, and (batched) a new member's tensor maps
            // (global memory) are prefetched while the previous tile streams
            FdItem cur{};
            if (t_first < t_end) cur = item_at(t_first);
            for (int t = t_first; t < t_end && issuing; t += t_step) {
                const bool has_next = t + t_step < t_end;
                FdItem nxt = cur;
                if (has_next) nxt = item_at(t + t_step);
                const int inst = cur.inst;
                const CUtensorMap *px = BATCHED ? &bd.maps[inst * NMAP + MI::X] : &mX;
                const CUtensorMap *py = BATCHED ? &bd.maps[inst * NMAP + MI::Y] : &mY;
                const CUtensorMap *pa = BATCHED ? &bd.maps[inst * NMAP + MI::A] : &mA;
                const CUtensorMap *pb = BATCHED ? &bd.maps[inst * NMAP + MI::B] : &mB;
                const int z0 = cur.zt * TZ;
                const int nch = (cur.v1 - cur.v0 + R - 1) / R;
                for (int ch = 0; ch < nch; ++ch, ++it) {
                    if (BATCHED && ch == 0 && has_next && nxt.inst != inst) {
                        const CUtensorMap *m = &bd.maps[nxt.inst * NMAP];
                        tma::prefetch_map(&m[MI::X]);
                        if (L::YB) tma::prefetch_map(&m[MI::Y]);
                        if (L::AB) tma::prefetch_map(&m[MI::A]);
                        if (INC && L::AB) tma::prefetch_map(&m[MI::B]);
                    }
                    const int b = it % NBUF;
                    if (it >= (uint32_t)NBUF &&
                        !tma::mbar_wait(&empty[b], ((it / NBUF) - 1) & 1, err, 1, a0.wait_ns)) {
                        issuing = false;  // a consumer gave up: buffer b may still be in use
                        break;
                    }
                    issue_chunk<L>(smem + b * L::BUF, &full[b], px, py, pa, pb, z0,
                                   cur.v0 + ch * R);
                }
                cur = nxt;
            }
            // the last copy issued into each buffer has landed before the block
            // may exit (in normal operation the consumers have waited for it)
            for (uint32_t j = it > (uint32_t)NBUF ? it - NBUF : 0; j < it; ++j)
                tma::mbar_drain(&full[j % NBUF], (j / NBUF) & 1, err, a0.wait_ns);
        }
        return;
    }

    // ---------------------------------------------------------------- consumers
    // this block's items: a contiguous range of the ensemble table, or every
    // gridDim.x-th one of a single simulation
    const bool rr = !BATCHED || bd.range == nullptr;
    const int t_first = rr ? blockIdx.x : bd.range[blockIdx.x];
    const int t_end = rr ? nitems : bd.range[blockIdx.x + 1];
    const int t_step = rr ? gridDim.x : 1;
    // moment m of cell zz of an item's tile: its bands in order
    auto moment_in = [&](const FdItem &i, int m, int zz) {
        const StageArgs &a = BATCHED ? bd.args[i.inst * 4 + STAGE - 1] : a0;
        double x = 0.0;
        if ((a.flags & F_COLL) && i.zt * TZ + zz < a.nz) {
            const double *q = a.Min + (long long)m * a.nz + i.zt * TZ + zz;
            const long long st = (long long)NMOM * a.nz;
            x = q[0];
            for (int k = 1; k < i.nvt; k += 8) {  // eight loads in flight
                double y[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) y[j] = k + j < i.nvt ? q[(k + j) * st] : 0.0;
#pragma unroll
                for (int j = 0; j < 8; ++j) x += y[j];
            }
        }
        return x;
    };
    FdItem ahead{};  // batched: the next table entry, read one item ahead
    if (t_first < t_end) ahead = item_at(t_first);
    // moments of the stage input for the first tile
    if (t_first < t_end && tid < NMOM * TZ)
        s_mom[tid / TZ][tid % TZ] = moment_in(ahead, tid / TZ, tid % TZ);
    consumer_sync();

    uint32_t it = 0;
    int s_inst = -1;  // member whose arguments s_args holds
    for (int t = t_first; t < t_end; t += t_step) {
        // (a single simulation's items are cheap to work out again, and their
        // fields would hold registers across the chunk loop)
        const FdItem cur = BATCHED ? ahead : item_at(t);
        const int inst = cur.inst, v0 = cur.v0, v1 = cur.v1;
        const int tn = t + t_step;
        if (BATCHED && tn < t_end) ahead = item_at(tn);
        if (BATCHED && inst != s_inst) {
            // a new member: its arguments into shared memory.  Read from there
            // (like a0 from parameter space) they cost no registers across the
            // chunk loop and cannot alias the stores to U and A.  The previous
            // tile's epilogue ended with a consumer barrier.
            if (tid < (int)(sizeof(StageArgs) / 8))
                reinterpret_cast<long long *>(s_args)[tid] =
                    reinterpret_cast<const long long *>(&bd.args[inst * 4 + STAGE - 1])[tid];
            consumer_sync();
            s_inst = inst;
        }
        const StageArgs &a = BATCHED ? *s_args : a0;
        const int nch = (v1 - v0 + R - 1) / R;
        const bool coll = (a.flags & F_COLL) != 0;
        const bool advec = (a.flags & F_ADVEC_OFF) == 0;
        const int z0 = cur.zt * TZ;
        const int z = z0 + lane;
        // the next item's input moments, in a register until the epilogue
        double mnext = 0.0;
        if (tid < NMOM * TZ && tn < t_end) mnext = moment_in(BATCHED ? ahead : item_at(tn), tid / TZ, tid % TZ);
        double macc[NMOM] = {0, 0, 0, 0, 0, 0};
        // only tiles at a row's ends hold cells that ghosts copy
        const bool wrap = a.bc == 0 && (z0 == 0 || z0 + TZ > a.nz - a.H);
        for (int ch = 0; ch < nch; ++ch, ++it) {
            const int b = it % NBUF;
            const int v = v0 + ch * R + warp;
            const int vr = min(v, a.nvz - 1);
            double vzv, factor;
            fd_row_values(a.v0, a.dv, a.dz, a.fd_advec, vr, vzv, factor);
            const bool landed = tma::mbar_wait(&full[b], (it / NBUF) & 1, err, 2, a0.wait_ns);
            const unsigned char *buf = smem + b * L::BUF;
            // this warp's row in the input boxes (HALO cells each side); a row's
            // components are XW (YW) cells apart
            constexpr int XW = L::XW, YW = L::YW;
            const TIN *xrow = reinterpret_cast<const TIN *>(buf) + warp * (NCOMP * XW) + HALO;
            const double *yrow = reinterpret_cast<const double *>(buf + L::XB) +
                                 warp * (NCOMP * YW) + (INC ? HALO : 0);
            // the stage input at cell j of this row (j in [-HALO, TZ + HALO))
            auto in = [&](int q, int j) -> double {
                if constexpr (INC && STAGE >= 2)
                    return yrow[q * YW + j] + (double)xrow[q * XW + j];
                else
                    return (double)xrow[q * XW + j];
            };

            double c[NCOMP], o[NCOMP];
#pragma unroll
            for (int q = 0; q < NCOMP; ++q) c[q] = in(q, lane);
            // vacuum, matter, advection and dissipation, (collective below)
#pragma unroll
            for (int q = 0; q < NCOMP; ++q) o[q] = 0.0;
            if (a.flags & F_VAC) {
                // read where used: batched, a is in shared memory and a
                // per-tile copy would hold registers across the chunk loop
                const double pmo = a.pmo, ct = a.ct, st = a.st;
                o[EE] = -pmo * 2.0 * st * c[EXI];
                o[XX] = pmo * 2.0 * st * c[EXI];
                o[EXR] = -pmo * 2.0 * ct * c[EXI];
                o[EXI] = pmo * (2.0 * ct * c[EXR] + st * (c[EE] - c[XX]));
                o[BEE] = -pmo * 2.0 * st * c[BEXI];
                o[BXX] = pmo * 2.0 * st * c[BEXI];
                o[BEXR] = -pmo * 2.0 * ct * c[BEXI];
                o[BEXI] = pmo * (2.0 * ct * c[BEXR] + st * (c[BEE] - c[BXX]));
            }
            if (a.flags & F_MAT) {
                const double hm = a.Hm[min(z, a.nz - 1)];
                o[EXR] += hm * c[EXI];
                o[EXI] += -hm * c[EXR];
                o[BEXR] += -hm * c[BEXI];
                o[BEXI] += hm * c[BEXR];
            }
            double ko[NCOMP];
            if constexpr (!GEN && !INC) {
                // FP64's central variant is bound by HBM and keeps the separate
                // sums: advection now, dissipation after the collective term
                const double ko_eps = a.ko_eps, fa = advec ? factor : 0.0;
#pragma unroll
                for (int q = 0; q < NCOMP; ++q) {
                    const double m2 = in(q, lane - 2), m1 = in(q, lane - 1), p1 = in(q, lane + 1),
                                 p2 = in(q, lane + 2);
                    o[q] += fa * ((m2 - p2) - 8.0 * (m1 - p1));
                    ko[q] = ko_eps * (m2 + p2 - 4.0 * (m1 + p1) + 6.0 * c[q]);
                }
            } else {
                // advection and dissipation as one stencil of differences from
                // the centre (the weights of either sum to zero); FP32-bulk,
                // latency bound at 128 registers: nz 32768 x nvz 256, stages 2
                // and 3 0.276 -> 0.245 ms each
                constexpr int TAPS = GEN ? 3 : 2;
                double w[2 * TAPS];
                fd_weights<GEN>(a, vzv, advec ? factor : 0.0, w);
#pragma unroll
                for (int q = 0; q < NCOMP; ++q) {
                    double x = 0.0;
#pragma unroll
                    for (int k = 1; k <= TAPS; ++k) {
                        x += w[k - 1] * (in(q, lane - k) - c[q]);
                        x += w[TAPS + k - 1] * (in(q, lane + k) - c[q]);
                    }
                    o[q] += x;
                    ko[q] = 0.0;
                }
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
            if constexpr (!GEN && !INC) {
#pragma unroll
                for (int q = 0; q < NCOMP; ++q) o[q] += ko[q];
            }
            // stage combine.  FP64 (stage values, A written once by stage 3 from
            // U in the A slot, U' and Y) or FP32-bulk (increments, common.cuh).
            const double dt = a.dt;
            // own-cell tiles: [row][component][TZ cells]
            const double *ys =
                reinterpret_cast<const double *>(buf + L::XB) + warp * (NCOMP * TZ) + lane;
            const double *as =
                reinterpret_cast<const double *>(buf + L::XB + L::YB) + warp * (NCOMP * TZ) + lane;
            const float *d1s =
                reinterpret_cast<const float *>(buf + L::XB + L::YB) + warp * (NCOMP * TZ) + lane;
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
                        const double d1 = (double)d1s[q * TZ];
                        const double d2 = (double)d1s[NCOMP * R * TZ + q * TZ];
                        const double d3 = (double)xrow[q * XW + lane];
                        const double yn = y + (d1 + 2.0 * d2 + d3) * (1.0 / 3.0) + (dt / 6.0) * kk;
                        u[q] = (TOUT)yn;
                        um[q] = yn;
                    }
                    anew[q] = 0.0;
                } else {
                    if (STAGE == 1) {
                        u[q] = (TOUT)(c[q] + (0.5 * dt) * kk);
                        anew[q] = 0.0;
                    } else if (STAGE == 2 || STAGE == 3) {
                        const double y = ys[q * TZ];
                        u[q] = (TOUT)(y + (STAGE == 2 ? 0.5 * dt : dt) * kk);
                        anew[q] = STAGE == 3 ? y + (as[q * TZ] - y) * (1.0 / 3.0) +
                                                   (c[q] - y) * (2.0 / 3.0) + (dt / 3.0) * kk
                                             : 0.0;  // stage 2 leaves A alone
                    } else {
                        u[q] = (TOUT)(as[q * TZ] + (dt / 6.0) * kk);
                        anew[q] = 0.0;
                    }
                    um[q] = (double)u[q];
                }
            }
            // this warp is done with the buffer (after a failed wait it keeps
            // the buffer: the producer's wait on it fails and it stops issuing)
            __syncwarp();
            if (lane == 0 && landed) tma::mbar_arrive(&empty[b]);

            if (v < v1 && z < a.nz) {  // (the last tile may be partial)
                TOUT *U = static_cast<TOUT *>(a.U);
                const long long ro = (long long)v * a.ld + HP;
#pragma unroll
                for (int q = 0; q < NCOMP; ++q) {
                    TOUT *row = U + q * a.cs + ro;
                    row[z] = u[q];
                    if (!INC && STAGE == 3) a.A[q * a.cs + ro + z] = anew[q];
                    if (wrap) periodic_ghosts(row, a, z, u[q]);
                }
                if (coll) {
                    const double Am = um[EXI] + um[BEXI];
                    const double Bm = um[EXR] - um[BEXR];
                    const double Cm = um[EE] - um[XX] - um[BEE] + um[BXX];
                    macc[0] += Am;
                    macc[1] += Bm;
                    macc[2] += Cm;
                    macc[3] += vzv * Am;
                    macc[4] += vzv * Bm;
                    macc[5] += vzv * Cm;
                }
            }
        }
        if (a.bc != 0 && (z0 == 0 || z0 + TZ >= a.nz)) {
            consumer_sync();
            fill_ghosts<false>(static_cast<TOUT *>(a.U), a, v0, v1, z0, tid, R * 32);
        }
        if (tn >= t_end) next_launch();  // (chain.cuh)
        // item epilogue: output moments (fixed-order sum over warps) and the
        // next item's input moments
        if (coll || BATCHED) {
            // warps w and w + R/2 pair up, then the R/2 pair sums are added
            // in a fixed order
            if (warp >= R / 2) {
#pragma unroll
                for (int m = 0; m < NMOM; ++m) s_red[warp - R / 2][m][lane] = macc[m];
            }
            consumer_sync();
            if (warp < R / 2) {
#pragma unroll
                for (int m = 0; m < NMOM; ++m) s_red[warp][m][lane] += macc[m];
            }
            consumer_sync();
            if (tid < NMOM * TZ) {
                const int m = tid / TZ, zz = tid % TZ;
                double s = 0.0;
#pragma unroll
                for (int w = 0; w < R / 2; ++w) s += s_red[w][m][zz];
                const int vt = BATCHED ? 0 : t / nzt;
                if (coll && z0 + zz < a.nz)
                    a.Mout[(long long)(vt * NMOM + m) * a.nz + z0 + zz] = s;
                s_mom[m][zz] = mnext;  // every consumer read this tile's values above
            }
            consumer_sync();
        }
    }
}

// ---------------------------------------------------------------------------
// host side

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                                  const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                  const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn()
{
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
    }
    return fn;
}

// 3-D map over one 8-component buffer: (cells of a padded row, components,
// rows), so that a box lands in shared memory as [row][component][cell]
int make_state_map(CUtensorMap *map, const void *base, int elem_bytes, int ld, int nvz,
                   long long cs, int box_cells, int box_rows)
{
    EncodeTiledFn fn = encode_fn();
    if (!fn) return -1;
    cuuint64_t dims[3] = {(cuuint64_t)ld, (cuuint64_t)NCOMP, (cuuint64_t)nvz};
    cuuint64_t strides[2] = {(cuuint64_t)cs * elem_bytes, (cuuint64_t)ld * elem_bytes};
    cuuint32_t box[3] = {(cuuint32_t)box_cells, (cuuint32_t)NCOMP, (cuuint32_t)box_rows};
    cuuint32_t es[3] = {1, 1, 1};
    CUresult r = fn(map, elem_bytes == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64
                                         : CU_TENSOR_MAP_DATA_TYPE_FLOAT32,
                    3, const_cast<void *>(base), dims, strides, box, es,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : (int)r;
}

// Width of the input box of a halo operand; FP64 stage 3 of FD (`narrow`)
// reads its stage input in 40-cell rows (Layout).
int tma_box_x(int scheme, int elem_bytes, bool narrow)
{
    if (scheme == FV) return fv_box_x(elem_bytes);
    if (narrow) return tma::TZ + 2 * tma::HALO;
    return elem_bytes == 8 ? tma::xw<double>() : tma::xw<float>();
}
int tma_box_tile() { return tma::TZ; }
// Rows of a map's box: `wide` for the operands of the 12-row FD stages.
int tma_box_rows(int scheme, bool wide) { return scheme == FD && wide ? 12 : 8; }
// largest nvz the TMA layout is offered for (the range its tests cover; the
// kernels themselves keep no per-row state in shared memory)
int tma_max_nvz() { return TMA_MAX_NVZ; }

// Shared memory of one block with an NB-deep ring.
template <class TIN, class TOUT, int STAGE>
static int tma_smem(int NB)
{
    using L = tma::Layout<TIN, TOUT, STAGE>;
    return NB * L::BUF + 2 * NB * 8 + (1 + L::NRED) * NMOM * tma::TZ * 8 + (int)sizeof(StageArgs);
}

template <bool GEN, int STAGE, class TIN, class TOUT, int NB, int MINB>
static cudaError_t launch_nb(const tma::StageMaps &m, const StageArgs &a, int *err, int nblocks,
                             cudaStream_t s, const BatchDev *bd)
{
    auto kern = rk4_stage_tma_kernel<GEN, STAGE, TIN, TOUT, NB, false, MINB>;
    auto kernb = rk4_stage_tma_kernel<GEN, STAGE, TIN, TOUT, NB, true, MINB>;
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
    const int shmem = tma_smem<TIN, TOUT, STAGE>(NB);
    constexpr int NT = tma::Layout<TIN, TOUT, STAGE>::NTHR;
    return launch_after(m.chained, bd ? kernb : kern, nblocks, NT, shmem, s, *m.x, *m.y, *m.a, *m.b,
                        a, err, bd ? *bd : BatchDev{});
}

// Rows of a v band of a single simulation's tiles: the height for which the
// rounds of items over the SMs take the fewest chunk times, summed over the four
// stages, at one chunk of overhead per item.  us a step by height, [chosen]: 1000 x
// 37 8 20.1, [12] 17.1, 16 19.1, 32 27.1; 2000 x 64 16 30.0, [32] 27.1, 64 43.5;
// 4000 x 100 16 78, 32 72, 64 66.4, [100] 67.0; 8192 x 128 32 174, 64 176, [128]
// 168; 16384 x 64 16 202, [32] 175, 64 172.
int fd_piece_rows(int nz, int nvz, int fp32, int nsm)
{
    const int nzt = (nz + tma::TZ - 1) / tma::TZ;
    const int r[4] = {12, fp32 ? 12 : 8, fp32 ? 12 : 8, 8};  // rows()
    int best = nvz;
    double cost = 1e300;
    for (int nvt = 1; nvt <= (nvz + 3) / 4; ++nvt) {
        const int tv = ((nvz + nvt - 1) / nvt + 3) / 4 * 4;
        const long long items = (long long)nzt * ((nvz + tv - 1) / tv);
        double c = 0.0;
        for (int s = 0; s < 4; ++s) c += (tv + r[s] - 1) / r[s] + 1.0;
        c *= (double)((items + nsm - 1) / nsm);
        if (c < cost) {
            cost = c;
            best = std::min(tv, nvz);
        }
    }
    return best;
}

// Ring depth of the FD kernel (one block per SM): the deepest ring of at most
// 4 buffers that total at most 144 KB.  Measured at nz 32768 x nvz 256:
// stages of 53-54 KB chunks (FP64 stage 3) are fastest with 2 buffers
// (0.441 / 0.534 / 0.545 ms with 2 / 3 / 4), FP64 stages 2 and 4 (38 KB) with
// 3, the FP32-bulk stages (48 KB chunks) with 3 (stage 4: 0.358 ms with 2,
// 0.320 ms with 3).
// COSENU_TMA_RING=n (2..4) overrides the depth where it fits.
static int tma_ring_env()
{
    static int v = -1;
    if (v < 0) {
        const char *e = getenv("COSENU_TMA_RING");
        v = (e && e[0] >= '2' && e[0] <= '4' && e[1] == 0) ? e[0] - '0' : 0;
    }
    return v;
}

template <class TIN, class TOUT, int STAGE>
static int tma_fd_ring()
{
    using L = tma::Layout<TIN, TOUT, STAGE>;
    int nb = 2;
    while (nb < 4 && (nb + 1) * L::BUF <= 144 * 1024) ++nb;
    const int e = tma_ring_env();
    if (e) nb = e;
    while (nb > 2 && tma_smem<TIN, TOUT, STAGE>(nb) > tma_smem_limit(1)) --nb;
    return nb;
}

// Blocks per SM.  FD (memory bound): one, with the deepest ring that fits;
// COSENU_TMA_MINB_FD=2 runs two blocks per SM (<= 112 registers each, half the
// shared memory) instead.
static int tma_minb_fd_env()
{
    static int v = -1;
    if (v < 0) {
        const char *e = getenv("COSENU_TMA_MINB_FD");
        v = (e && e[0] == '2') ? 2 : 1;
    }
    return v;
}

int tma_blocks_per_sm(int scheme) { return scheme == FV ? fv_blocks_per_sm() : tma_minb_fd_env(); }

// Blocks of a single simulation: every block slot, or one item each.
int tma_blocks(int scheme, int nz, int nvt, int nsm)
{
    return (int)std::min<long long>((long long)((nz + tma::TZ - 1) / tma::TZ) * nvt,
                                    (long long)tma_blocks_per_sm(scheme) * nsm);
}

template <bool GEN, int STAGE, class TIN, class TOUT>
static cudaError_t launch_one(const tma::StageMaps &m, const StageArgs &a, int *err, int nblocks,
                              cudaStream_t s, const BatchDev *bd)
{
#define LNB(NB, MINB) launch_nb<GEN, STAGE, TIN, TOUT, NB, MINB>(m, a, err, nblocks, s, bd)
    if (tma_minb_fd_env() == 2) {
        const int lim = tma_smem_limit(2);
        if (tma_smem<TIN, TOUT, STAGE>(4) <= lim) return LNB(4, 2);
        if (tma_smem<TIN, TOUT, STAGE>(3) <= lim) return LNB(3, 2);
        return LNB(2, 2);
    }
    switch (tma_fd_ring<TIN, TOUT, STAGE>()) {
    case 2: return LNB(2, 1);
    case 3: return LNB(3, 1);
    default: return LNB(4, 1);
    }
#undef LNB
}

template <bool GEN>
static cudaError_t launch_p(const tma::StageMaps &m, const StageArgs &a, int stage, int fp32,
                            int *err, int nblocks, cudaStream_t s, const BatchDev *bd)
{
    if (fp32) {
        // FP32-bulk: Y in, D1 out; Y + D1 in, D2 out; Y + D2 in, D3 out; Y + D3 in, Y' out
        switch (stage) {
        case 1: return launch_one<GEN, 1, double, float>(m, a, err, nblocks, s, bd);
        case 2: return launch_one<GEN, 2, float, float>(m, a, err, nblocks, s, bd);
        case 3: return launch_one<GEN, 3, float, float>(m, a, err, nblocks, s, bd);
        case 4: return launch_one<GEN, 4, float, double>(m, a, err, nblocks, s, bd);
        }
    } else {
        switch (stage) {
        case 1: return launch_one<GEN, 1, double, double>(m, a, err, nblocks, s, bd);
        case 2: return launch_one<GEN, 2, double, double>(m, a, err, nblocks, s, bd);
        case 3: return launch_one<GEN, 3, double, double>(m, a, err, nblocks, s, bd);
        case 4: return launch_one<GEN, 4, double, double>(m, a, err, nblocks, s, bd);
        }
    }
    return cudaErrorInvalidValue;
}

static cudaError_t launch_any(const tma::StageMaps &m, const StageArgs &a, int scheme, int stage,
                              int fp32, int *err, int nblocks, cudaStream_t s, const BatchDev *bd)
{
    if (scheme == FV) return launch_fv_tma(m, a, stage, fp32, err, nblocks, s, bd);
    const bool gen = a.fd_advec != 0 || a.ko_order == 5;
    return gen ? launch_p<true>(m, a, stage, fp32, err, nblocks, s, bd)
               : launch_p<false>(m, a, stage, fp32, err, nblocks, s, bd);
}

cudaError_t launch_rk4_stage_tma(const CUtensorMap &mX, const CUtensorMap &mY,
                                 const CUtensorMap &mA, const CUtensorMap &mB, const StageArgs &a,
                                 int scheme, int stage, int fp32, int *err, int nblocks,
                                 cudaStream_t s, bool chained)
{
    const tma::StageMaps m{&mX, &mY, &mA, &mB, chained};
    return launch_any(m, a, scheme, stage, fp32, err, nblocks, s, nullptr);
}

// Ensemble launch: `a` carries the variant switches shared by every instance
// (scheme variant, precision); per-instance values come from bd.
cudaError_t launch_rk4_stage_tma_batch(const BatchDev &bd, const StageArgs &a, int scheme,
                                       int stage, int fp32, int *err, int nblocks,
                                       cudaStream_t s, bool chained)
{
    CUtensorMap z{};
    const tma::StageMaps m{&z, &z, &z, &z, chained};
    return launch_any(m, a, scheme, stage, fp32, err, nblocks, s, &bd);
}

// Sets the shared-memory attribute of the kernels a simulation (batched: or an
// ensemble) of this variant launches, on the current device.  The first call
// loads them, 0.4 ms each.
cudaError_t tma_prepare(int scheme, int fp32, bool gen, bool batched, bool small)
{
    CUtensorMap m{};
    const BatchDev bd{};
    const tma::StageMaps maps{&m, &m, &m, &m, false};
    StageArgs a{};
    a.fd_advec = gen;
    a.ko_order = 3;
    a.flags = small ? F_SMALL : 0;
    for (int st = 1; st <= 4; ++st) {
        cudaError_t e = launch_any(maps, a, scheme, st, fp32, nullptr, 0, nullptr,
                                   batched ? &bd : nullptr);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace cosenu
