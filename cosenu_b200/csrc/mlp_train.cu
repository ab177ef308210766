// Fused minibatch kernels of the surrogate network's training (mlp.cu drives
// them): tcgen05 GEMMs whose epilogues do what separate launches did.
//
// A training step is latency bound: batches of 64 rows through 512-wide layers
// are 0.1 GFLOP, and the step was 29 launches of about 7 us (11 GEMMs on 8 to
// 32 CTAs with a four-stage ring, 18 elementwise ones).  Here it is eight:
//   forward, layers 0 .. L-1: C = X W^T + b; hidden layers write Z (FP32) and
//       GELU(Z) (BF16); the last one writes the loss gradient dZ (BF16), the
//       loss partials, and updates its own bias;
//   backward, one launch per layer l = L-1 .. 0: the tiles of dX_l (dZ_{l-1} =
//       dZ_l W_l x GELU'(Z_{l-1}), with the bias update of layer l-1) together
//       with the tiles of dW_{l+1} = dZ_{l+1}^T X_{l+1} and their AdamW update.
//       The weight update runs one launch behind dX, so W_l still holds the
//       forward's weights when dX_l reads it; the last launch has dW_1 and dW_0.
// Tiles are 128 x 16: 16 columns put 32 CTAs on a 512-wide layer and 128 on a
// 512 x 512 weight gradient (64 columns: 8 and 32), and an operand's whole K is
// staged at once (up to 128 x 576 x 2 B), so a GEMM is one round trip to L2, 4 MMAs
// per 64 k behind it, and one commit.  2000 rows in batches of 64 (an epoch and the
// read-back of the parameters): 6.85 -> 2.88 ms, 2.29 with overlapping launches
// (chain.cuh): the next one's blocks start when every tile has its accumulator,
// and allocate and wait behind the epilogues.
//
// Every sum runs in the order of the separate kernels (k in steps of 16 within
// one accumulator; bias gradients row by row), so the parameters a training
// run ends with are bit for bit the same.
//
// Shared-memory operand layout as in mlp_gemm.cu (canonical K-major UMMA, no
// swizzle): 8-wide k chunk c at c * LBO, row r of a chunk at r * 16 bytes, LBO
// = rows * 16 + 16.  With at most 64 rows the A tile holds 64; the MMA still
// reads 128, the upper 64 from whatever follows, and those accumulator rows are
// never read back.  Waits are bounded (one second) and recorded in *err.
#include <cuda_bf16.h>

#include <cstdint>
#include <initializer_list>

#include "chain.cuh"
#include "mlp_math.cuh"
#include "mlp_train.h"

namespace mlptrain {

using namespace mlpmath;

constexpr int NTHR = 256;
constexpr int TM = 128;  // accumulator rows (TMEM lanes)
constexpr int TN = 16;   // accumulator columns
constexpr int TMEM_COLS = 32;  // smallest allocation
constexpr uint32_t LBO_B = TN * 16 + 16;
constexpr unsigned long long WAIT_NS = 1000000000ull;
constexpr int SRED = TM * (TN + 1) * 4;  // the accumulator tile in FP32
constexpr int TILE = TM * TN * 4;        // an FP32 operand tile of the epilogue
constexpr int TAIL = 64;                 // mbarrier, TMEM slot

// kind::f16, FP32 accumulator, BF16 K-major operands (see mlp_gemm.cu)
constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TN >> 3) << 17) |
                           ((uint32_t)(TM >> 4) << 24);

__host__ __device__ constexpr int lbo_a(int rt) { return rt * 16 + 16; }

// Shared memory for a K-deep GEMM with rt A rows.  The MMA reads 128 rows of
// the last chunk whatever rt is: the B tile and the tail that follow cover it.
// ntile: epilogue tiles.
__host__ __device__ constexpr int smem_bytes(int rt, int k64, int ntile)
{
    const int a = k64 * 8 * lbo_a(rt), b = k64 * 8 * (int)LBO_B;
    return a + (b > 2048 ? b : 2048) + SRED + ntile * TILE + TAIL;
}

__device__ __forceinline__ uint32_t su32(const void *p)
{
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ unsigned long long gtime()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void bar_wait(uint32_t bar, uint32_t parity, int *err)
{
    unsigned long long t0 = 0;
    for (uint32_t n = 1;; ++n) {
        uint32_t ok;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            " selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return;
        if ((n & 63) == 0) {
            const unsigned long long t = gtime();
            if (t0 == 0) t0 = t;
            if (t - t0 > WAIT_NS) {
                atomicCAS(err, 0, 1);
                return;
            }
        }
    }
}

__device__ __forceinline__ uint64_t sdesc(uint32_t saddr, uint32_t lbo)
{
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) |
           ((uint64_t)(128u >> 4) << 32) | (1ull << 46);
}

// ROWS (16 or a multiple of 32) x K of a K-major operand straight to their
// place; rows and k past the end are zero-filled without a read.  Thread -> k
// chunk tid & 7 of row tid / 8 + 32 i, all k groups: the addresses only step.
__device__ __forceinline__ void copy_rows(unsigned char *s, uint32_t lbo, int rows,
                                          const __nv_bfloat16 *X, int ld, int rtot, int ktot,
                                          int r0)
{
    const int kc = threadIdx.x & 7, r = threadIdx.x >> 3, nk = (ktot + 63) / 64;
#pragma unroll 1
    for (int rr = r; rr < rows; rr += NTHR / 8) {
        const bool inr = r0 + rr < rtot;
        const __nv_bfloat16 *src = X + (inr ? (long long)(r0 + rr) * ld : 0) + kc * 8;
        uint32_t dst = su32(s + kc * lbo + rr * 16);
#pragma unroll 4
        for (int g = 0; g < nk; ++g) {
            const bool in = inr && g * 64 + kc * 8 < ktot;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst),
                         "l"(in ? src + g * 64 : X), "r"(in ? 16 : 0)
                         : "memory");
            dst += 8 * lbo;
        }
    }
}

// this thread's copies have landed
__device__ __forceinline__ void wait_copies()
{
    asm volatile("cp.async.wait_all;" ::: "memory");
}

__device__ __forceinline__ uint32_t word(const uint4 &v, int w)
{
    return w == 0 ? v.x : w == 1 ? v.y : w == 2 ? v.z : v.w;
}

// An 8 (k) x 8 (rows) block of a row-contiguous operand: row j of X holds k =
// kg + j; transposed in registers and written as 8 rows of 16 bytes.
struct Block8 {
    uint4 v[8];
    __device__ __forceinline__ void load(const __nv_bfloat16 *X, int ld, int ktot, int kg, int rg,
                                         bool in)
    {
#pragma unroll
        for (int j = 0; j < 8; ++j)
            v[j] = (in && kg + j < ktot)
                       ? __ldcg(reinterpret_cast<const uint4 *>(X + (long long)(kg + j) * ld + rg))
                       : make_uint4(0, 0, 0, 0);
    }
    __device__ __forceinline__ void store(unsigned char *dst) const
    {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t sel = (i & 1) ? 0x7632u : 0x5410u;
            uint4 o;
            o.x = __byte_perm(word(v[0], i >> 1), word(v[1], i >> 1), sel);
            o.y = __byte_perm(word(v[2], i >> 1), word(v[3], i >> 1), sel);
            o.z = __byte_perm(word(v[4], i >> 1), word(v[5], i >> 1), sel);
            o.w = __byte_perm(word(v[6], i >> 1), word(v[7], i >> 1), sel);
            *reinterpret_cast<uint4 *>(dst + i * 16) = o;
        }
    }
};

// Warp 0: n MMAs of K 16 over consecutive k, issued by one elected lane, and
// their commit; `fresh`: the first one overwrites the accumulator.  The whole
// warp runs the loop so that the descriptors live in uniform registers (one
// thread in a divergent branch took 80 cycles an MMA to move them there).
__device__ __forceinline__ void mma_steps(uint32_t tmem, uint32_t sa, uint32_t la, uint32_t sb,
                                          int n, bool fresh, uint32_t bar)
{
    uint64_t da = sdesc(sa, la), db = sdesc(sb, LBO_B);
    uint32_t acc = fresh ? 0u : 1u;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 4
    for (int k = 0; k < n; ++k) {
        asm volatile(
            "{\n .reg .pred p, q;\n elect.sync _|q, 0xffffffff;\n setp.ne.b32 p, %4, 0;\n"
            " @q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
            "l"(da), "l"(db), "r"(IDESC), "r"(acc)
            : "memory");
        acc = 1;
        da += 2 * la >> 4;
        db += 2 * LBO_B >> 4;
    }
    asm volatile(
        "{\n .reg .pred q;\n elect.sync _|q, 0xffffffff;\n"
        " @q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(
            bar)
        : "memory");
}

// This thread's warp, uniform over it.
__device__ __forceinline__ int warp_id() { return __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0); }

// 16 columns (n0 ..) of rows r0 .. r0 + rows of a row-major FP32 matrix, to
// tile[row][16]; zeros past the end.
__device__ __forceinline__ void copy_tile(float *tile, const float *X, int ld, int rtot, int ntot,
                                          int r0, int n0, int rows)
{
#pragma unroll 1
    for (int q = threadIdx.x; q < rows * 4; q += NTHR) {
        const int r = q >> 2, c = (q & 3) * 4;
        const bool in = r0 + r < rtot && n0 + c < ntot;
        const float *src = in ? X + (long long)(r0 + r) * ld + n0 + c : X;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(su32(tile + r * TN + c)),
                     "l"(src), "r"(in ? 16 : 0)
                     : "memory");
    }
}

// The CTA's fixed pieces: TMEM, one mbarrier, the FP32 tiles.
struct Cta {
    unsigned char *a, *b;
    float *tile;          // epilogue operands
    float (*red)[TN + 1]; // accumulator, then the epilogue's results
    uint64_t *bar;
    uint32_t tmem, phase;
    __device__ __forceinline__ Cta(unsigned char *smem, int rt, int k64, int ntile)
    {
        a = smem;
        b = smem + k64 * 8 * lbo_a(rt);
        unsigned char *end = smem + smem_bytes(rt, k64, ntile);
        bar = reinterpret_cast<uint64_t *>(end - TAIL);
        red = reinterpret_cast<float(*)[TN + 1]>(end - TAIL - SRED);
        tile = reinterpret_cast<float *>(end - TAIL - SRED - ntile * TILE);
        uint32_t *slot = reinterpret_cast<uint32_t *>(bar + 1);
        phase = 0;
        if (threadIdx.x < 32) {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                             su32(slot)),
                         "r"(TMEM_COLS));
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
        }
        if (threadIdx.x == 0) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(su32(bar)));
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        tmem = *slot;
    }
    // all threads: the accumulator (row = TMEM lane) to red, visible to all; the
    // accumulator and the operand tiles are then free for the next MMAs
    __device__ __forceinline__ void spill()
    {
        if (threadIdx.x < TM) {
            uint32_t r[TN];
            const uint32_t taddr = tmem + ((threadIdx.x >> 5) << 21);  // lanes 32 warp .. + 31
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,"
                "%13,%14,%15}, [%16];\n"
                : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
                  "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
                  "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                : "r"(taddr));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int j = 0; j < TN; ++j) red[threadIdx.x][j] = __uint_as_float(r[j]);
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    }
    // all threads: shared memory staged so far is visible to the tensor core
    __device__ __forceinline__ void staged()
    {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
    }
    // all threads: the committed MMAs are done, the accumulator readable
    __device__ __forceinline__ void done(int *err)
    {
        bar_wait(su32(bar), phase, err);
        phase ^= 1;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    }
    __device__ __forceinline__ void release()
    {
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        if (threadIdx.x < 32) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                         "r"(TMEM_COLS));
        }
    }
};

// acc = A(rows m0 .. m0 + rt) x B over all K: A K-major from global; B either
// K-major rows n0 .. n0 + 16 of W, or (TB) row-contiguous, W[k][n0 ..].
template <bool TB>
__device__ __forceinline__ void gemm_rows(Cta &c, const __nv_bfloat16 *A, int lda, int M, int K,
                                          const __nv_bfloat16 *W, int ldw, int N, int m0, int n0,
                                          int rt, bool load_b, int *err)
{
    const int nk = (K + 63) / 64;
    const uint32_t la = lbo_a(rt);
    Block8 blk;  // (at most 256 8 x 8 blocks of B: K <= 1024)
    const int ng = threadIdx.x & 1, kc = threadIdx.x >> 1;
    const bool mine = TB && load_b && kc < nk * 8;
    if (mine) blk.load(W, ldw, K, kc * 8, n0 + ng * 8, n0 + ng * 8 < N);
    copy_rows(c.a, la, rt, A, lda, M, K, m0);
    if (!TB && load_b) copy_rows(c.b, LBO_B, TN, W, ldw, N, K, n0);
    if (mine) blk.store(c.b + kc * LBO_B + ng * 128);
    wait_copies();
    c.staged();
    if (warp_id() == 0)
        mma_steps(c.tmem, su32(c.a), la, su32(c.b), nk * 4, true, su32(c.bar));
    c.done(err);
}

// Column sums of the FP32 tile (rows in order, continuing s), then the bias
// update of this CTA's 16 columns.
__device__ __forceinline__ float column_sum(const float (*red)[TN + 1], int rows, float s)
{
    #pragma unroll 8
    for (int m = 0; m < rows; ++m) s += red[m][threadIdx.x];
    return s;
}

__device__ __forceinline__ void bias_update(const Args &p, int l, int n, float db)
{
    const size_t i = p.boff[l] + n;
    adamw(p.w[i], p.m1[i], p.m2[i], db, p.opt, 0.f);
    p.wb[i] = __float2bfloat16(p.w[i]);
}

// The epilogues run element by element in rolled loops, thread -> column tid &
// 15 of row tid / 16 + 16 i: a launch runs each instruction once or twice, so
// unrolled epilogues (16 erf or AdamW updates per thread, 10-20 KB of code) were
// bound by instruction fetch (10-20 us a launch).  Their operands are copied to
// shared memory ahead of the MMAs.

// Forward of layer l over all rows, 16 columns per CTA.
__global__ void __launch_bounds__(NTHR) fwd_kernel(const __grid_constant__ Args p, int l, int rt)
{
    extern __shared__ __align__(1024) unsigned char smem[];
    const int K = p.din[l], N = p.dout[l], n0 = blockIdx.x * TN, tid = threadIdx.x;
    const bool last = l == p.nl - 1;
    const int col = tid & (TN - 1), n = n0 + col;
    Cta c(smem, rt, (K + 63) / 64, 1);
    previous_launch();
    const float bias = n < N ? p.w[p.boff[l] + n] : 0.f;
    const __nv_bfloat16 *X = l == 0 ? p.x : p.h[l - 1];
    float db = 0.f, loss = 0.f;
#pragma unroll 1
    for (int m0 = 0; m0 < p.rows; m0 += rt) {
        if (last) copy_tile(c.tile, p.t, N, p.rows, N, m0, n0, rt);
        gemm_rows<false>(c, X, K, p.rows, K, p.wb + p.woff[l], K, N, m0, n0, rt, m0 == 0, p.err);
        next_launch();
        c.spill();
#pragma unroll 1
        for (int r = tid / TN; r < rt && m0 + r < p.rows; r += NTHR / TN) {
            const float v = c.red[r][col] + bias;
            if (n >= N) break;
            const long long i = (long long)(m0 + r) * N + n;
            if (!last) {
                p.z[l][i] = v;
                p.h[l][i] = __float2bfloat16(gelu(v));
            } else {
                // loss 1/(rows N) sum (y - t)^2 and its gradient
                const float d = v - c.tile[r * TN + col];
                loss += d * d;
                const float g = 2.f * d * p.scale;
                p.dz[l][i] = __float2bfloat16(g);
                c.red[r][col] = g;
            }
        }
        __syncthreads();
        if (last && tid < TN) db = column_sum(c.red, min(rt, p.rows - m0), db);
        __syncthreads();
    }
    if (last) {
        if (tid < TN && n < N) bias_update(p, l, n, db);
        for (int off = 16; off > 0; off >>= 1) loss += __shfl_down_sync(0xffffffffu, loss, off);
        if ((tid & 31) == 0) c.red[0][tid >> 5] = loss;
        __syncthreads();
        if (tid == 0) {
            float x = 0.f;
            for (int w = 0; w < NTHR / 32; ++w) x += c.red[0][w];
            p.loss[blockIdx.x] = x;
        }
    }
    c.release();
}

// dZ_{l-1} = (dZ_l W_l) x GELU'(Z_{l-1}), 16 columns (of din) per CTA, and the
// bias of layer l-1.
__device__ __forceinline__ void dx_tile(const Args &p, int l, int rt, int tile, unsigned char *smem)
{
    const int K = p.dout[l], N = p.din[l], n0 = tile * TN, tid = threadIdx.x;
    const int col = tid & (TN - 1);
    Cta c(smem, rt, (K + 63) / 64, 1);
    previous_launch();
    float db = 0.f;
#pragma unroll 1
    for (int m0 = 0; m0 < p.rows; m0 += rt) {
        copy_tile(c.tile, p.z[l - 1], N, p.rows, N, m0, n0, rt);
        gemm_rows<true>(c, p.dz[l], K, p.rows, K, p.wb + p.woff[l], N, N, m0, n0, rt, m0 == 0,
                        p.err);
        next_launch();
        c.spill();
#pragma unroll 1
        for (int r = tid / TN; r < rt && m0 + r < p.rows; r += NTHR / TN) {
            const float g = c.red[r][col] * gelu_grad(c.tile[r * TN + col]);
            p.dz[l - 1][(long long)(m0 + r) * N + n0 + col] = __float2bfloat16(g);
            c.red[r][col] = g;
        }
        __syncthreads();
        if (tid < TN) db = column_sum(c.red, min(rt, p.rows - m0), db);
        __syncthreads();
    }
    if (tid < TN) bias_update(p, l - 1, n0 + tid, db);
    c.release();
}

// dW_l = dZ_l^T X_l over the rows, a 128 x 16 tile, then AdamW on it.
__device__ __forceinline__ void dw_tile(const Args &p, int l, int tile, unsigned char *smem)
{
    const int N = p.din[l], M = p.dout[l], nt = N / TN;
    const int m0 = tile / nt * TM, n0 = tile % nt * TN, tid = threadIdx.x, col = tid & (TN - 1);
    const __nv_bfloat16 *X = l == 0 ? p.x : p.h[l - 1];
    Cta c(smem, TM, 1, 3);
    previous_launch();
    const uint32_t la = lbo_a(TM);
    const size_t wo = p.woff[l];
    copy_tile(c.tile, p.w + wo, N, M, N, m0, n0, TM);
    copy_tile(c.tile + TM * TN, p.m1 + wo, N, M, N, m0, n0, TM);
    copy_tile(c.tile + 2 * TM * TN, p.m2 + wo, N, M, N, m0, n0, TM);
#pragma unroll 1
    for (int k0 = 0; k0 < p.rows; k0 += 64) {
        // threads 0-127: one 8 x 8 block of A each; 128-143: of B
        Block8 blk;
        const int kc = tid & 7, rg = (tid >> 3) & 15;
        if (tid < 128)
            blk.load(p.dz[l], M, p.rows, k0 + kc * 8, m0 + rg * 8, m0 + rg * 8 < M);
        else if (rg < 2)
            blk.load(X, N, p.rows, k0 + kc * 8, n0 + rg * 8, true);
        if (k0 > 0) c.done(p.err);  // the previous MMAs have read the tiles
        if (tid < 128)
            blk.store(c.a + kc * la + rg * 128);
        else if (rg < 2)
            blk.store(c.b + kc * LBO_B + rg * 128);
        c.staged();
        if (warp_id() == 0)
            mma_steps(c.tmem, su32(c.a), la, su32(c.b), 4, k0 == 0, su32(c.bar));
    }
    wait_copies();
    next_launch();
    c.done(p.err);
    c.spill();
#pragma unroll 2
    for (int r = tid / TN; r < TM && m0 + r < M; r += NTHR / TN) {
        const int q = r * TN + col;
        float w = c.tile[q], a = c.tile[TM * TN + q], b = c.tile[2 * TM * TN + q];
        adamw(w, a, b, c.red[r][col], p.opt, p.opt.wd);
        const size_t i = wo + (size_t)(m0 + r) * N + n0 + col;
        p.w[i] = w;
        p.m1[i] = a;
        p.m2[i] = b;
        p.wb[i] = __float2bfloat16(w);
    }
    c.release();
}

// One backward launch: ndx tiles of dX_lx, then the nw0 tiles of dW_lw0, then
// those of dW_lw1.
__global__ void __launch_bounds__(NTHR) bwd_kernel(const __grid_constant__ Args p, int lx, int ndx,
                                                   int lw0, int nw0, int lw1, int rt)
{
    extern __shared__ __align__(1024) unsigned char smem[];
    const int b = blockIdx.x;
    if (b < ndx)
        dx_tile(p, lx, rt, b, smem);
    else if (b < ndx + nw0)
        dw_tile(p, lw0, b - ndx, smem);
    else
        dw_tile(p, lw1, b - ndx - nw0, smem);
}

constexpr int SMEM_MAX = 232448;  // opt-in shared memory per block on sm_100

static int tile_rows(int rows) { return rows <= 64 ? 64 : TM; }
static int k64(int k) { return (k + 63) / 64; }

int loss_tiles(int n_out) { return (n_out + TN - 1) / TN; }

bool fits(int nl, const int *din, const int *dout, int rows)
{
    // The column tiles loop over the rows; the general kernels have row tiles.  An
    // epoch of 8192 rows, us, separate / fused by batch: 64 25177 / 6944, 256 8014 /
    // 3888, 512 4936 / 3483, 1024 3452 / 3285, 2048 2708 / 3195.  An operand's whole
    // K has to fit in shared memory.
    if (nl < 2 || nl > MAXL || rows > 512) return false;
    for (int l = 0; l < nl; ++l) {
        const int k = din[l] > dout[l] ? din[l] : dout[l];
        if (k > 1024 || smem_bytes(tile_rows(rows), k64(k), 1) > SMEM_MAX) return false;
        if (din[l] % TN || dout[l] % 8 || (l < nl - 1 && dout[l] % TN)) return false;
    }
    return true;
}

cudaError_t prepare()
{
    for (auto k : {(const void *)fwd_kernel, (const void *)bwd_kernel}) {
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MAX);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t step(const Args &a, cudaStream_t s, bool chained)
{
    cudaError_t e = cudaSuccess;
    const int rt = tile_rows(a.rows), L = a.nl;
    for (int l = 0; l < L && e == cudaSuccess; ++l)
        e = launch_after(chained || l > 0, fwd_kernel, (a.dout[l] + TN - 1) / TN, NTHR,
                         smem_bytes(rt, k64(a.din[l]), 1), s, a, l, rt);
    auto dw_tiles = [&](int l) { return (a.dout[l] + TM - 1) / TM * (a.din[l] / TN); };
    const int dw_smem = smem_bytes(TM, 1, 3);
    for (int l = L - 1; l >= 1 && e == cudaSuccess; --l) {
        const int ndx = a.din[l] / TN, nw = l + 1 < L ? dw_tiles(l + 1) : 0;
        const int dx_smem = smem_bytes(rt, k64(a.dout[l]), 1);
        e = launch_after(true, bwd_kernel, ndx + nw, NTHR, dx_smem > dw_smem ? dx_smem : dw_smem, s,
                         a, l, ndx, l + 1, nw, 0, rt);
    }
    const int n1 = dw_tiles(1), n0 = dw_tiles(0);
    if (e == cudaSuccess)
        e = launch_after(true, bwd_kernel, n1 + n0, NTHR, dw_smem, s, a, 0, 0, 1, n1, 0, rt);
    return e;
}

}  // namespace mlptrain
