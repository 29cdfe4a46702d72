// fm_rows.cu -- the list build of one system by molecule (fm_rows.cuh).
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "fm_common.cuh"
#include "fm_device.cuh"
#include "fm_force.cuh"
#include "fm_rows.cuh"

namespace fm {

namespace {

// Whether the build runs. Its grid has more blocks than fit at once, and one
// whose row overflows raises ST_NLIST while others have yet to start: they go
// on, so that max_nbr covers every row and one growth fits them all. (After an
// overflow of an earlier step positions and cells stand still, and the build
// only repeats its rows.)
__device__ __forceinline__ bool rows_gate(const FmDev &d, int gated)
{
    if (*(volatile uint32_t *)&d.sc->status & (ST_FATAL & ~ST_NLIST)) return false;
    return !gated || d.sc->rebuild;
}

template <int G>
__global__ void __launch_bounds__(ROWS_THREADS) k_rows(FmDev d, int gated, int iter)
{
    pdl_enter();
    if (!rows_gate(d, gated)) return;
    __shared__ RowsShared<G> sh[ROWS_THREADS / 32];
    CellSys y;
    y.P = cur_pos(d, d.sc->pset);
    y.cell_start = d.cell_start;
    y.mol_off = 0;
    for (int k = 0; k < 3; k++) { y.ne[k] = d.ne[k]; y.L[k] = d.L[k]; }
    y.rn2 = d.rn2;
    y.nbr = d.nbr;
    y.maxn = d.maxn;
    y.dd = d.dd;
    const bool strays = d.sc->strays != 0;
    const int i = (int)(((long long)blockIdx.x * ROWS_THREADS + threadIdx.x) / G), g = threadIdx.x % G;
    int cnt = 0;
    if (i < d.n) {
        const int c = d.cell_of[i];
        const int cx = c % d.ne[0], cy = (c / d.ne[0]) % d.ne[1], cz = c / (d.ne[0] * d.ne[1]);
        // a subdomain's halo copies are partners only: no rows
        if (!(d.dd && (is_halo(cx, d.ne[0]) || is_halo(cy, d.ne[1]) || is_halo(cz, d.ne[2]))))
            cnt = rows_build<G>(y, i, c, strays, g, sh[threadIdx.x >> 5]);
        if (g == 0) d.nnbr[i] = min(cnt, d.maxn);
    }
    const int most = __reduce_max_sync(0xffffffffu, cnt);
    if ((threadIdx.x & 31) == 0) {
        // one address for all warps: look before the atomic
        if (most > *(volatile int32_t *)&d.sc->max_nbr) atomicMax(&d.sc->max_nbr, most);
        if (most > d.maxn) raise_status(d, ST_NLIST, iter);
    }
}

// The same by fours, for dense systems.
__global__ void __launch_bounds__(ROWS_THREADS) k_rows_four(FmDev d, int gated, int iter)
{
    pdl_enter();
    if (!rows_gate(d, gated)) return;
    __shared__ RowsShared<32> sh[ROWS_THREADS / 32];
    CellSys y;
    y.P = cur_pos(d, d.sc->pset);
    y.cell_start = d.cell_start;
    y.mol_off = 0;
    for (int k = 0; k < 3; k++) { y.ne[k] = d.ne[k]; y.L[k] = d.L[k]; }
    y.rn2 = d.rn2;
    y.nbr = d.nbr;
    y.nnbr = d.nnbr;
    y.maxn = d.maxn;
    y.dd = d.dd;
    const int warp = threadIdx.x >> 5, u = blockIdx.x * (ROWS_THREADS / 32) + warp;
    if (u >= rows_four_units(d.ne)) return;
    const int most = rows_four_unit(y, u, d.sc->strays != 0, threadIdx.x & 31, sh[warp]);
    if ((threadIdx.x & 31) == 0) {
        if (most > *(volatile int32_t *)&d.sc->max_nbr) atomicMax(&d.sc->max_nbr, most);
        if (most > d.maxn) raise_status(d, ST_NLIST, iter);
    }
}

template <int G>
void launch_rows_g(const FmDev &d, int gated, int iter, cudaStream_t st)
{
    const int blocks = std::max(1, (int)(((long long)d.n * G + ROWS_THREADS - 1) / ROWS_THREADS));
    pdl_launch(k_rows<G>, blocks, ROWS_THREADS, st, d, gated, iter);
}

}  // namespace

void launch_rows(const FmDev &d, int gated, int iter, cudaStream_t st)
{
    const int lanes = rows_lanes(d.density * d.cs[0] * d.cs[1] * d.cs[2]);
    if (lanes == 32 && d.n >= ROWS_FOUR_MOLECULES) {
        pdl_launch(k_rows_four, (rows_four_units(d.ne) + ROWS_THREADS / 32 - 1) / (ROWS_THREADS / 32), ROWS_THREADS, st, d,
                   gated, iter);
        return;
    }
    switch (lanes) {
    case 8: launch_rows_g<8>(d, gated, iter, st); break;
    case 16: launch_rows_g<16>(d, gated, iter, st); break;
    default: launch_rows_g<32>(d, gated, iter, st); break;
    }
}

}  // namespace fm
