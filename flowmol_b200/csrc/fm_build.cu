// fm_build.cu -- the list build of one system by warp (fm_build.cuh): one warp
// per cell, or per 2x2x2 cells of a sparse system.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <type_traits>

#include "fm_common.cuh"
#include "fm_device.cuh"
#include "fm_force.cuh"
#include "fm_build.cuh"

namespace fm {

namespace {

// Neighbour rows of every extended cell, one warp per cell or, for sparse
// systems (BLOCKS), per block of 2x2x2 cells (grid-stride); the routines and
// their pair-set argument are in fm_build.cuh.  Both give the same rows.
template <bool BLOCKS, bool TILE>
__global__ void __launch_bounds__(NB_THREADS, 8) k_build_nlist(FmDev d, int gated, int iter)
{
    pdl_enter();
    if (!gate(d, gated)) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    using Shared = typename std::conditional<BLOCKS, BlockShared<TILE>, BuildShared<TILE>>::type;
    // per-warp staging in dynamic shared memory (the largest variants pass 48 KB)
    extern __shared__ __align__(16) unsigned char build_smem[];
    Shared *sh = reinterpret_cast<Shared *>(build_smem);
    CellSys y;
    y.P = cur_pos(d, d.sc->pset);
    y.cell_start = d.cell_start;
    y.mol_off = 0;
    for (int k = 0; k < 3; k++) { y.ne[k] = d.ne[k]; y.cs[k] = d.cs[k]; y.hd[k] = d.hd[k]; y.L[k] = d.L[k]; }
    y.rn2 = d.rn2;
    y.nbr = d.nbr;
    y.nnbr = d.nnbr;
    y.maxn = d.maxn;
    y.max_nbr = &d.sc->max_nbr;
    y.nbr16 = d.nbr16; y.maxn16 = d.maxn16; y.tT = d.tile_T; y.tR = d.tile_R; y.blk_off = d.blk_off;
    y.tdummy = d.tile ? tile_boff(d.tile_ucap, d.tile_R) : 0;
    for (int k = 0; k < 3; k++) y.tnb[k] = d.tile_nb[k];
    y.dd = d.dd;
    for (int k = 0; k < 3; k++) y.org[k] = d.dd ? d.org[k] : 0;
    uint32_t over = 0u;
    const int nwork = BLOCKS ? ((d.ne[0] + 1) / 2) * ((d.ne[1] + 1) / 2) * ((d.ne[2] + 1) / 2) : d.ncell;
    // work units handed out NB_CHUNK at a time, so warps that meet empty or
    // halo cells take more: no tail of a few warps with dense cells left
    for (;;) {
        int u0 = 0;
        if (lane == 0) u0 = atomicAdd(&d.sc->build_next, NB_CHUNK);
        u0 = __shfl_sync(0xffffffffu, u0, 0);
        if (u0 >= nwork) break;
        const int u1 = min(u0 + NB_CHUNK, nwork);
        for (int u = u0; u < u1; u++) {
            if constexpr (BLOCKS) over |= build_block<TILE>(y, u, sh[warp], lane);
            else over |= build_cell<TILE>(y, u, sh[warp], lane);
        }
    }
    if (lane == 0 && (over & BUILD_OVER_LIST)) raise_status(d, ST_NLIST, iter);
}

constexpr int kSMs = 148;
inline int nblk(long long n, int t) { return (int)((n + t - 1) / t); }

// The list build walks the cells grid-stride with every block resident (one
// wave: a second partial wave would double the kernel's time).
template <bool BLOCKS, bool TILE>
static size_t build_smem_bytes()
{
    using Shared = typename std::conditional<BLOCKS, BlockShared<TILE>, BuildShared<TILE>>::type;
    return sizeof(Shared) * NB_WARPS;
}

template <bool BLOCKS, bool TILE>
static int build_grid(int nwork)
{
    static int resident = 0;
    if (resident == 0) {
        int dev = 0, nsm = kSMs, per_sm = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
        cudaFuncSetAttribute(k_build_nlist<BLOCKS, TILE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)build_smem_bytes<BLOCKS, TILE>());
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_build_nlist<BLOCKS, TILE>, NB_THREADS,
                                                      build_smem_bytes<BLOCKS, TILE>());
        resident = std::max(nsm, 1) * std::max(per_sm, 1);
    }
    return std::min(nblk(nwork, NB_WARPS), resident);
}

template <bool BLOCKS, bool TILE>
static void launch_build_t(const FmDev &d, int nwork, int gated, int iter, cudaStream_t st)
{
    const int g = build_grid<BLOCKS, TILE>(nwork);  // (sets the kernel's shared-memory attribute once)
    pdl_launch_smem(k_build_nlist<BLOCKS, TILE>, g, NB_THREADS, build_smem_bytes<BLOCKS, TILE>(), st, d,
                    gated, iter);
}

}  // namespace

void launch_build_nlist(const FmDev &d, int gated, int iter, cudaStream_t st)
{
    if (d.build_rows) {
        launch_rows(d, gated, iter, st);
        return;
    }
    cudaMemsetAsync(&d.sc->build_next, 0, sizeof(int32_t), st);
    const int nb = ((d.ne[0] + 1) / 2) * ((d.ne[1] + 1) / 2) * ((d.ne[2] + 1) / 2);
    const int nw = d.build_blocks ? nb : d.ncell;
    switch ((d.build_blocks ? 2 : 0) + (d.tile ? 1 : 0)) {
    case 0: launch_build_t<false, false>(d, nw, gated, iter, st); break;
    case 1: launch_build_t<false, true>(d, nw, gated, iter, st); break;
    case 2: launch_build_t<true, false>(d, nw, gated, iter, st); break;
    default: launch_build_t<true, true>(d, nw, gated, iter, st); break;
    }
}

}  // namespace fm
