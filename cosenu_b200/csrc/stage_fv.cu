// FV stage launches, FP64 (FP32-bulk: stage_fv32.cu), and the choice of pieces.
// The precisions are two modules: a process loads the one it uses, and one module
// of both is large enough that it is stored compressed (a process' first FV
// simulation, 600 x 32 cells: 18 ms to create).
#include <algorithm>
#include <cstdlib>

#include "stage_fv.cuh"

namespace cosenu {

// Two blocks per SM, each with the deepest ring that fits in half the SM
// (COSENU_TMA_MINB=1 selects one block per SM with a 4-deep ring).
static int minb_env()
{
    static int v = -1;
    if (v < 0) {
        const char *e = getenv("COSENU_TMA_MINB");
        v = (e && e[0] == '1') ? 1 : 2;
    }
    return v;
}

int fv_blocks_per_sm() { return minb_env(); }
int fv_box_x(int elem_bytes) { return elem_bytes == 8 ? fv::xw<double>() : fv::xw<float>(); }

// Rows of a v piece of a single simulation's tiles: the height (a multiple of
// 8) for which the rounds of items over the block slots take the fewest
// chunk times, at half a chunk of overhead per item.  us a step by height in chunks,
// [chosen]: 600 x 32 [1] 21.9, 2 31.6, 4 54.1; 1024 x 64 [1] 28.1, 2 33.1, 4 53.9;
// 2400 x 100 1 79.8, [2] 77.5, 4 81.6; 9600 x 64 1 183, [2] 165, 4 171; 4000 x 100 2
// 114, 5 113, [7] 116, 13 149; 16384 x 64 1 308, 2 267, [8] 274.  It misses 2400 x 32
// (1 37.3, [2] 42.4: 300 chunks on 296 slots) and 8192 x 128 (3 260, [16] 284).
int fv_piece_rows(int nz, int nvz, int nsm)
{
    const int nzt = (nz + tma::TZ - 1) / tma::TZ, nch = (nvz + fv::R - 1) / fv::R;
    const int slots = minb_env() * nsm;
    int best = nch;
    double cost = 1e300;
    for (int nvt = 1; nvt <= nch; ++nvt) {
        const int pc = (nch + nvt - 1) / nvt;
        const long long items = (long long)nzt * ((nch + pc - 1) / pc);
        const double c = (double)((items + slots - 1) / slots) * (pc + 0.5);
        if (c < cost) {
            cost = c;
            best = pc;
        }
    }
    return best * fv::R;
}

cudaError_t launch_fv_tma(const tma::StageMaps &m, const StageArgs &a, int stage, int fp32, int *err,
                          int nblocks, cudaStream_t s, const BatchDev *bd)
{
    if (fp32) return launch_fv_bulk(m, a, stage, err, nblocks, s, bd);
    switch (stage) {
    case 1: return launch_one<1, double, double>(m, a, err, nblocks, s, bd);
    case 2: return launch_one<2, double, double>(m, a, err, nblocks, s, bd);
    case 3: return launch_one<3, double, double>(m, a, err, nblocks, s, bd);
    case 4: return launch_one<4, double, double>(m, a, err, nblocks, s, bd);
    }
    return cudaErrorInvalidValue;
}

}  // namespace cosenu
