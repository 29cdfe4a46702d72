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

template <int G, bool POLY>
__global__ void __launch_bounds__(ROWS_THREADS) k_rows(FmDev d, int gated, int iter)
{
    pdl_enter();
    if (frozen(d) || (gated && !d.sc->rebuild)) return;
    __shared__ RowsShared<G> sh;
    CellSys y;
    y.P = cur_pos(d, d.sc->pset);
    y.cell_start = d.cell_start;
    y.mol_off = 0;
    for (int k = 0; k < 3; k++) { y.ne[k] = d.ne[k]; y.L[k] = d.L[k]; }
    y.rn2 = d.rn2;
    y.nbr = d.nbr;
    y.maxn = d.maxn;
    y.chain = d.chain; y.subchain = d.subchain; y.bflag = d.bflag;
    y.bnd = d.bnd;
    y.dd = d.dd;
    const bool strays = d.sc->strays != 0;
    const int i = (int)(((long long)blockIdx.x * ROWS_THREADS + threadIdx.x) / G), g = threadIdx.x % G;
    int cnt = 0, nb = 0;
    if (i < d.n) {
        const int c = d.cell_of[i];
        const int cx = c % d.ne[0], cy = (c / d.ne[0]) % d.ne[1], cz = c / (d.ne[0] * d.ne[1]);
        // a subdomain's halo copies are partners only: no rows
        if (!(d.dd && (is_halo(cx, d.ne[0]) || is_halo(cy, d.ne[1]) || is_halo(cz, d.ne[2]))))
            cnt = rows_build<G, POLY>(y, i, c, strays, g, sh, nb);
        if (g == 0) {
            d.nnbr[i] = min(cnt, d.maxn);
            if (POLY) d.nbond[i] = min(nb, 4);
        }
    }
    const int most = __reduce_max_sync(0xffffffffu, cnt), mostb = POLY ? __reduce_max_sync(0xffffffffu, nb) : 0;
    if ((threadIdx.x & 31) == 0) {
        // one address for all warps: look before the atomic
        if (most > *(volatile int32_t *)&d.sc->max_nbr) atomicMax(&d.sc->max_nbr, most);
        const uint32_t bit = (most > d.maxn ? ST_NLIST : 0u) | (mostb > 4 ? ST_BOND : 0u);  // too_many_bonds_error
        if (bit) raise_status(d, bit, iter);
    }
}

template <int G>
void launch_rows_g(const FmDev &d, int gated, int iter, cudaStream_t st)
{
    const int blocks = std::max(1, (int)(((long long)d.n * G + ROWS_THREADS - 1) / ROWS_THREADS));
    if (d.potential_flag == 1) pdl_launch(k_rows<G, true>, blocks, ROWS_THREADS, st, d, gated, iter);
    else pdl_launch(k_rows<G, false>, blocks, ROWS_THREADS, st, d, gated, iter);
}

}  // namespace

void launch_rows(const FmDev &d, int gated, int iter, cudaStream_t st)
{
    switch (rows_lanes(d.density * d.cs[0] * d.cs[1] * d.cs[2])) {
    case 8: launch_rows_g<8>(d, gated, iter, st); break;
    case 16: launch_rows_g<16>(d, gated, iter, st); break;
    default: launch_rows_g<32>(d, gated, iter, st); break;
    }
}

}  // namespace fm
