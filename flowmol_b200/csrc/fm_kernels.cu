// fm_kernels.cu -- sm_100a kernels of the per-timestep MD hot path.
//
// Data layout (device): positions as double4 {x, y, z, 0} so a neighbour
// gather is one 32-byte sector; velocities and accelerations as FP64 SoA for
// coalesced streaming; molecules re-ordered by cell at every rebuild so a
// warp's neighbours share L1 lines.  Distance tests are FP64 without FMA
// contraction (__dmul_rn/__dadd_rn) and periodic images are formed as
// x_src + (+/-)domain, the same two roundings the reference performs when it
// copies a halo molecule (messenger.serial.f90:401, 509) and subtracts
// (linklist.f90:749-750) -- so pair sets match the reference bit for bit.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <type_traits>

#include "fm_common.cuh"
#include "fm_device.cuh"
#include "fm_force_list.cuh"
#include "fm_tile.cuh"

namespace fm {

thread_local bool pdl_capture = false;

namespace {


// ---------------------------------------------------------------------------
// integrator (simulation_move_particles_vv.f90:64-69, 132-135)
// ---------------------------------------------------------------------------

__global__ void k_reset_scalars(FmDev d)
{
    FmScalars *s = d.sc;
    s->rmax = 0.0;
    s->vmax2 = 0ull;
    s->rebuild = 0;
    s->status = 0u;
    s->fail_iter = -1;
    s->max_nbr = 0;
    s->escape_slot = -1;
    s->rebuilds = 0;
    s->digest = 0ull;
    s->digest_n = 0;
    s->nrec_pending = 0;
    s->disp_reset = 1;  // rdisp is allocated as zeros at the first check
    s->dmax = 0ull;
    for (int q = 0; q < 6; q++) s->pacc[q] = 0.0;
    s->pcount = 0;
    s->tile_next = 0;
    s->umax = 0;
}

// r = (r + dt v) + (0.5 dt^2) a ; v = v + (0.5 dt) a   -- pass 1, in place.
__global__ void k_move1(FmDev d)
{
    pdl_enter();
    if (frozen(d)) return;
    double4 *P = cur_pos(d, d.sc->pset);
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    double m2 = 0.0;
    if (i < d.n) {
        double4 p = P[i];
        double vx = d.vx[i], vy = d.vy[i], vz = d.vz[i];
        double ax = d.ax[i], ay = d.ay[i], az = d.az[i];
        p.x = __dadd_rn(__dadd_rn(p.x, __dmul_rn(d.dt, vx)), __dmul_rn(d.half_dt2, ax));
        p.y = __dadd_rn(__dadd_rn(p.y, __dmul_rn(d.dt, vy)), __dmul_rn(d.half_dt2, ay));
        p.z = __dadd_rn(__dadd_rn(p.z, __dmul_rn(d.dt, vz)), __dmul_rn(d.half_dt2, az));
        vx = __dadd_rn(vx, __dmul_rn(d.half_dt, ax));
        vy = __dadd_rn(vy, __dmul_rn(d.half_dt, ay));
        vz = __dadd_rn(vz, __dmul_rn(d.half_dt, az));
        P[i] = p;
        d.vx[i] = vx; d.vy[i] = vy; d.vz[i] = vz;
        m2 = norm2_rn(vx, vy, vz);
    }
    block_vmax2(d, m2);
}

__global__ void k_move2(FmDev d)
{
    pdl_enter();
    if (frozen(d)) return;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < d.n) {
        d.vx[i] = __dadd_rn(d.vx[i], __dmul_rn(d.half_dt, d.ax[i]));
        d.vy[i] = __dadd_rn(d.vy[i], __dmul_rn(d.half_dt, d.ay[i]));
        d.vz[i] = __dadd_rn(d.vz[i], __dmul_rn(d.half_dt, d.az[i]));
    }
}

// simulation_move_particles_lfv NVE (simulation_move_particles_lfv.f90:81-92), in place.
__global__ void k_move_lfv(FmDev d)
{
    pdl_enter();
    if (frozen(d)) return;
    double4 *P = cur_pos(d, d.sc->pset);
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    double m2 = 0.0;
    if (i < d.n) {
        double4 p = P[i];
        double vx = __dadd_rn(d.vx[i], __dmul_rn(d.dt, d.ax[i]));
        double vy = __dadd_rn(d.vy[i], __dmul_rn(d.dt, d.ay[i]));
        double vz = __dadd_rn(d.vz[i], __dmul_rn(d.dt, d.az[i]));
        p.x = __dadd_rn(p.x, __dmul_rn(d.dt, vx));
        p.y = __dadd_rn(p.y, __dmul_rn(d.dt, vy));
        p.z = __dadd_rn(p.z, __dmul_rn(d.dt, vz));
        P[i] = p;
        d.vx[i] = vx; d.vy[i] = vy; d.vz[i] = vz;
        m2 = norm2_rn(vx, vy, vz);
    }
    block_vmax2(d, m2);
}

__global__ void k_vmax(FmDev d)
{
    pdl_enter();
    if (frozen(d)) return;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    double m2 = 0.0;
    if (i < d.n) m2 = norm2_rn(d.vx[i], d.vy[i], d.vz[i]);
    block_vmax2(d, m2);
}

// Rebuild criterion 2 (simulation_checkrebuild.f90:106-121): rdisp += v dt
// for every molecule (v as the check sees it), and the largest |component|
// into sc->dmax.  After a rebuild the reference deallocates rdisp (:150-152),
// so the next check starts it from zero.
__global__ void k_disp(FmDev d)
{
    pdl_enter();
    if (frozen(d)) return;
    const bool restart = d.sc->disp_reset != 0;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    double m = 0.0;
    if (i < d.n) {
        const double x = __dadd_rn(restart ? 0.0 : d.rdx[i], __dmul_rn(d.vx[i], d.dt));
        const double y = __dadd_rn(restart ? 0.0 : d.rdy[i], __dmul_rn(d.vy[i], d.dt));
        const double z = __dadd_rn(restart ? 0.0 : d.rdz[i], __dmul_rn(d.vz[i], d.dt));
        d.rdx[i] = x; d.rdy[i] = y; d.rdz[i] = z;
        m = fmax(fabs(x), fmax(fabs(y), fabs(z)));
    }
    m = warp_max(m);
    __shared__ double wmax[32];
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) wmax[w] = m;
    __syncthreads();
    if (w == 0) {
        const int nw = (blockDim.x + 31) >> 5;
        double v = l < nw ? wmax[l] : 0.0;
        v = warp_max(v);
        if (l == 0 && v > 0.0) atomicMax(&d.sc->dmax, (unsigned long long)__double_as_longlong(v));
    }
}

// ---------------------------------------------------------------------------
// rebuild decision (simulation_checkrebuild.f90:34, 83-99, 101-103, 106-121, 148-155)
// ---------------------------------------------------------------------------

__device__ __forceinline__ int decide(const FmDev &d, int iter, int flip, int crit, int fixed_rebuild,
                                      double half_min_delta)
{
    FmScalars *s = d.sc;
    if (flip) s->pset ^= 1;
    int rebuild = ((iter + 1) % d.tplot) == 0 ? 1 : 0;
    if (crit == 0) {
        double vmax = sqrt(__longlong_as_double((long long)s->vmax2));
        s->rmax = __dadd_rn(s->rmax, __dmul_rn(vmax, d.dt));
        if (s->rmax > half_min_delta) rebuild = 1;
    } else if (crit == 1) {
        if ((iter % fixed_rebuild) == 0) rebuild = 1;
    } else if (crit == 2) {
        // any(abs(rdisp(:,n)) > 0.5 minval(delta_rneighbr))
        if (__longlong_as_double((long long)s->dmax) > half_min_delta) rebuild = 1;
        s->dmax = 0ull;
        s->disp_reset = rebuild;
    }
    s->vmax2 = 0ull;
    if (rebuild) {
        s->rmax = 0.0;
        s->rebuilds += 1;
    }
    s->rebuild = rebuild;
    return rebuild;
}

__global__ void k_decide(FmDev d, int iter, int flip, int crit, int fixed_rebuild, double half_min_delta)
{
    pdl_enter();
    if (d.sc->status & ST_FATAL) return;
    decide(d, iter, flip, crit, fixed_rebuild, half_min_delta);
}

// The decision as the first node of the rebuild graph (fm_api.cu): the
// iteration comes from the device (g_iter, set by the host at the start of a
// range and advanced here), and the outcome opens the graph's conditional
// body -- the rebuild kernels -- or skips it without launching anything.  A
// frozen state skips it (the handle's default, 0).
__global__ void k_decide_graph(FmDev d, int flip, int crit, int fixed_rebuild, double half_min_delta,
                               cudaGraphConditionalHandle cond, int body_kernels)
{
    FmScalars *s = d.sc;
    const int iter = s->g_iter;
    s->g_iter = iter + 1;
    s->cur_iter = iter;
    if (s->status & ST_FATAL) return;
    const int rebuild = decide(d, iter, flip, crit, fixed_rebuild, half_min_delta);
    if (rebuild) s->graph_kernels += body_kernels;
    cudaGraphSetConditional(cond, rebuild ? 1u : 0u);
}

__global__ void k_set_graph_iter(FmDev d, int iter) { d.sc->g_iter = iter; }

// ---------------------------------------------------------------------------
// cell binning by counting sort (linklist.f90:2645-2679; sendmols wrap
// messenger.serial.f90:961-1028)
// ---------------------------------------------------------------------------



__global__ void k_wrap_bin(FmDev d, int wrap, int bin, int gated, int iter)
{
    pdl_enter();
    if (!gate(d, gated)) return;
    double4 *P = cur_pos(d, d.sc->pset);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < d.n; i += gridDim.x * blockDim.x) {
        double4 p = P[i];
        if (wrap) {
            double4 q = p;
            if (q.x >= d.hd[0]) q.x = __dsub_rn(q.x, d.L[0]);
            if (q.x < -d.hd[0]) q.x = __dadd_rn(q.x, d.L[0]);
            if (q.y >= d.hd[1]) q.y = __dsub_rn(q.y, d.L[1]);
            if (q.y < -d.hd[1]) q.y = __dadd_rn(q.y, d.L[1]);
            if (q.z >= d.hd[2]) q.z = __dsub_rn(q.z, d.L[2]);
            if (q.z < -d.hd[2]) q.z = __dadd_rn(q.z, d.L[2]);
            if (q.x != p.x || q.y != p.y || q.z != p.z) P[i] = q;
            p = q;
        }
        if (!bin) continue;
        bool bad = false;
        int cx = bin_axis(p.x, d.hd[0], d.cs[0], d.ne[0], bad);
        int cy = bin_axis(p.y, d.hd[1], d.cs[1], d.ne[1], bad);
        int cz = bin_axis(p.z, d.hd[2], d.cs[2], d.ne[2], bad);
        if (bad) {
            raise_status(d, ST_ESCAPE, iter);
            d.sc->escape_slot = i;
        }
        int c = cx + d.ne[0] * (cy + d.ne[1] * cz);
        d.cell_of[i] = c;
        atomicAdd(&d.cell_count[c], 1);
    }
}

// Exclusive scan of the per-cell counts in two parallel passes over tiles of
// SCAN_TILE cells: tile sums, then each tile adds the sum of the tiles before
// it and scans itself.  The counts are zeroed so the scatter can reuse them
// as cursors.
constexpr int SCAN_THREADS = 1024;
constexpr int SCAN_PER = 4;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_PER;

__device__ __forceinline__ int block_excl_scan(int v, int *total)
{
    __shared__ int ws[SCAN_THREADS / 32];
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) ws[w] = incl;
    __syncthreads();
    if (w == 0) {
        int x = lane < SCAN_THREADS / 32 ? ws[lane] : 0, xi = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int t = __shfl_up_sync(0xffffffffu, xi, o);
            if (lane >= o) xi += t;
        }
        if (lane < SCAN_THREADS / 32) ws[lane] = xi - x;
        if (lane == SCAN_THREADS / 32 - 1) ws[SCAN_THREADS / 32 - 1] = xi - x, *total = xi;
    }
    __syncthreads();
    return ws[w] + incl - v;
}

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_tiles(FmDev d, int gated)
{
    pdl_enter();
    if (!gate(d, gated)) return;
    __shared__ int tot;
    const int base = blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_PER;
    int local = 0;
#pragma unroll
    for (int k = 0; k < SCAN_PER; k++)
        if (base + k < d.ncell) local += d.cell_count[base + k];
    block_excl_scan(local, &tot);
    if (threadIdx.x == 0) d.tile_sum[blockIdx.x] = tot;
    if (threadIdx.x == 0 && blockIdx.x == 0) d.sc->strays = 0;  // for k_sort_cells
}

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_apply(FmDev d, int gated)
{
    pdl_enter();
    if (!gate(d, gated)) return;
    __shared__ int tot, prefix;
    if (threadIdx.x < 32) {
        int acc = 0;
        for (int b = threadIdx.x; b < (int)blockIdx.x; b += 32) acc += d.tile_sum[b];
        acc = warp_sum(acc);
        if (threadIdx.x == 0) prefix = acc;
    }
    const int base = blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_PER;
    int cnt[SCAN_PER];
    int local = 0;
#pragma unroll
    for (int k = 0; k < SCAN_PER; k++) {
        cnt[k] = base + k < d.ncell ? d.cell_count[base + k] : 0;
        local += cnt[k];
    }
    int run = block_excl_scan(local, &tot) + prefix;
#pragma unroll
    for (int k = 0; k < SCAN_PER; k++) {
        if (base + k < d.ncell) {
            d.cell_start[base + k] = run;
            d.cell_count[base + k] = 0;
        }
        run += cnt[k];
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) d.cell_start[d.ncell] = prefix + tot;
}

__global__ void k_scatter(FmDev d, int gated)
{
    pdl_enter();
    if (!gate(d, gated)) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < d.n; i += gridDim.x * blockDim.x) {
        int c = d.cell_of[i];
        if (c < 0) continue;  // a subdomain's departed molecule or stale halo copy
        int slot = d.cell_start[c] + atomicAdd(&d.cell_count[c], 1);
        d.perm[slot] = i;
    }
}

// Atomics make the in-cell order arbitrary; sorting each cell by the
// molecules' identity (slot_of: upload index, or global number in a
// subdomain) makes the whole rebuild deterministic and independent of the
// previous order, so that a subdomain lays out a cell's molecules exactly as
// the undivided system does.  Ahead of the identity goes the octant of the
// cell (sub_cell), so that the four molecules of a line are near each other
// and the partners that neighbouring list entries name share lines.  One
// warp per cell.
constexpr int SORT_WARPS = 8;
__device__ __forceinline__ unsigned long long sort_key(const FmDev &d, const double4 *P, int o, int c)
{
    const int ne0 = d.ne[0], ne1 = d.ne[1];
    const int g0 = c % ne0 + (d.dd ? d.org[0] : 0), g1 = (c / ne0) % ne1 + (d.dd ? d.org[1] : 0);
    const int g2 = c / (ne0 * ne1) + (d.dd ? d.org[2] : 0);
    const int oct = sub_cell(P[o], g0, g1, g2, d.hd, d.cs);
    return (unsigned long long)oct << 32 | (unsigned)d.slot_of[o];
}
// What is left to do for cell c, slots [b, b + m), once it is sorted.
__device__ __forceinline__ void sorted_cell(const FmDev &d, int c, int m)
{
    d.cell_count[c] = 0;  // leave counts zeroed for the next histogram
    if (m > 0 && !d.dd) {
        const int cx = c % d.ne[0], cy = (c / d.ne[0]) % d.ne[1], cz = c / (d.ne[0] * d.ne[1]);
        if (is_halo(cx, d.ne[0]) || is_halo(cy, d.ne[1]) || is_halo(cz, d.ne[2])) d.sc->strays = 1;
    }
}
__global__ void __launch_bounds__(32 * SORT_WARPS) k_sort_cells(FmDev d, int gated)
{
    pdl_enter();
    if (!gate(d, gated)) return;
    const int lane = threadIdx.x & 31;
    const double4 *P = cur_pos(d, d.sc->pset);
    for (int c = blockIdx.x * SORT_WARPS + (threadIdx.x >> 5); c < d.ncell; c += gridDim.x * SORT_WARPS) {
        const int b = d.cell_start[c], e = d.cell_start[c + 1];
        warp_sort_cell(d.perm, b, e - b, lane, [&](int o) { return sort_key(d, P, o, c); });
        for (int k = b + lane; k < e; k += 32) d.cell_of[k] = c;  // by new slot from here on
        if (lane == 0) sorted_cell(d, c, e - b);
    }
}

// The same for sparse systems (two or three molecules a cell): eight lanes sort
// a cell of up to eight, four cells a warp, and the warp then takes the larger
// ones in turn.  262,144 FENE beads in 110,592 cells: 57 us with a warp a cell.
__global__ void __launch_bounds__(32 * SORT_WARPS) k_sort_cells_sparse(FmDev d, int gated)
{
    pdl_enter();
    if (!gate(d, gated)) return;
    const int lane = threadIdx.x & 31, l8 = lane & 7;
    const double4 *P = cur_pos(d, d.sc->pset);
    for (int c0 = 4 * (blockIdx.x * SORT_WARPS + (threadIdx.x >> 5)); c0 < d.ncell; c0 += 4 * gridDim.x * SORT_WARPS) {
        const int c = c0 + (lane >> 3);
        const bool in = c < d.ncell;
        const int b = in ? d.cell_start[c] : 0, m = in ? d.cell_start[c + 1] - b : 0;
        warp_sort_four_cells(d.perm, b, m, lane, [&](int o) { return sort_key(d, P, o, c); });
        if (m <= 8 && l8 < m) d.cell_of[b + l8] = c;  // by new slot from here on
        if (in && l8 == 0) sorted_cell(d, c, m);
        for (unsigned large = __ballot_sync(0xffffffffu, l8 == 0 && m > 8); large != 0u; large &= large - 1u) {
            const int from = __ffs(large) - 1;
            const int lc = c0 + (from >> 3), lb = __shfl_sync(0xffffffffu, b, from), lm = __shfl_sync(0xffffffffu, m, from);
            warp_sort_cell(d.perm, lb, lm, lane, [&](int p) { return sort_key(d, P, p, lc); });
            for (int k = lane; k < lm; k += 32) d.cell_of[lb + k] = lc;
        }
    }
}

// Gather into scratch in cell order, then copy back, so every array keeps
// its address (the step loop never needs to know whether a rebuild ran).
__global__ void k_reorder_gather(FmDev d, int gated, double4 *tpos, int32_t *tuidx)
{
    pdl_enter();
    if (!gate(d, gated)) return;
    const double4 *P = cur_pos(d, d.sc->pset);
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < d.n; s += gridDim.x * blockDim.x) {
        int o = d.perm[s];
        tpos[s] = P[o];
        d.tvx[s] = d.vx[o]; d.tvy[s] = d.vy[o]; d.tvz[s] = d.vz[o];
        d.tax[s] = d.ax[o]; d.tay[s] = d.ay[o]; d.taz[s] = d.az[o];
        tuidx[s] = d.slot_of[o];
        if (d.potential_flag == 1) {
            d.tchain[s] = d.chain[o]; d.tsubchain[s] = d.subchain[o]; d.tbflag[s] = d.bflag[o];
            if (d.funcy) d.tfuncy[s] = d.funcy[o];
        }
    }
}

__global__ void k_reorder_copy(FmDev d, int gated, const double4 *tpos, const int32_t *tuidx)
{
    pdl_enter();
    if (!gate(d, gated)) return;
    double4 *P = cur_pos(d, d.sc->pset);
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < d.n; s += gridDim.x * blockDim.x) {
        P[s] = tpos[s];
        d.vx[s] = d.tvx[s]; d.vy[s] = d.tvy[s]; d.vz[s] = d.tvz[s];
        d.ax[s] = d.tax[s]; d.ay[s] = d.tay[s]; d.az[s] = d.taz[s];
        d.slot_of[s] = tuidx[s];
        if (d.potential_flag == 1) {
            d.slot_by_upload[tuidx[s]] = s;
            d.chain[s] = d.tchain[s]; d.subchain[s] = d.tsubchain[s]; d.bflag[s] = d.tbflag[s];
            if (d.funcy) d.funcy[s] = d.tfuncy[s];
        }
    }
}

// ---------------------------------------------------------------------------
// neighbour list from shared-memory cell tiles
// (pair set of assign_to_neighbourlist_halfint_opt, linklist.f90:660-804,
//  1118-1180, stored in both directions)
// ---------------------------------------------------------------------------

// Staging segment table of the tiled force path, one warp per block: the
// exclusive prefix of the block's 128 segment sizes (fm_tile.cuh) and their
// total.  A block whose total exceeds the force kernel's capacity raises
// ST_TILE; the host grows the capacity and builds again.
constexpr int BS_THREADS = 256;
__global__ void __launch_bounds__(BS_THREADS) k_blk_seg(FmDev d, int gated, int iter)
{
    pdl_enter();
    if (!gate(d, gated)) return;
    const int lane = threadIdx.x & 31;
    constexpr int WPB = BS_THREADS / 32;
    int umax = 0;
    for (int blk = blockIdx.x * WPB + (threadIdx.x >> 5); blk < d.tile_nblk; blk += gridDim.x * WPB) {
        const int bx = blk % d.tile_nb[0], by = (blk / d.tile_nb[0]) % d.tile_nb[1];
        const int bz = blk / (d.tile_nb[0] * d.tile_nb[1]);
        int32_t *out = d.blk_off + (size_t)blk * TILE_NSEGP;
        int carry = 0;
#pragma unroll
        for (int h = 0; h < TILE_NSEG / 32; h++) {
            int st, cnt, code;
            tile_segment(d.ne, d.cell_start, 2 * bx, 2 * by, 2 * bz, h * 32 + lane, st, cnt, code);
            int incl = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
            out[h * 32 + lane] = carry + incl - cnt;
            carry += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (lane == 0) out[TILE_NSEG] = carry;
        umax = max(umax, carry);
    }
    umax = __reduce_max_sync(0xffffffffu, umax);
    if (lane == 0 && umax > 0) {
        atomicMax(&d.sc->umax, umax);
        if (umax > d.tile_ucap) raise_status(d, ST_TILE, iter);
    }
}

// ---------------------------------------------------------------------------
// forces (simulation_compute_forces_LJ_neigbr*, simulation_compute_forces.f90
// :551-726) fused with move(2) and the next move(1)
// ---------------------------------------------------------------------------

// Discovery key of the bond (j, entry) in the reference's list build
// (assign_to_neighbourlist_halfint_opt, linklist.f90:660-804, where
// check_update_adjacentbeadinfo appends each bonded pair to both rows as it is
// met): interior cells in (x, y, z) loop order with z fastest; in each cell
// first the in-cell pairs (list order, the later member after the earlier),
// then the 13 forward shifts (shift, owner, partner); the cells' lists are in
// decreasing molecule number (head insertion, assign_to_cell loops 1..np).
// A pair across the periodic boundary is met only in the halo sweeps that
// follow (:778-802): after every interior pair, ordered here by the partner's
// molecule number.
__device__ int ang_cell_of(const FmDev &d, int s)
{
    int lo = 0, hi = d.ncell - 1;  // largest c with cell_start[c] <= s
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (d.cell_start[mid] <= s) lo = mid; else hi = mid - 1;
    }
    return lo;
}
__device__ int ang_list_pos(const FmDev &d, int c, int s)
{
    const int me = d.slot_of[s];
    int pos = 0;
    for (int t = d.cell_start[c]; t < d.cell_start[c + 1]; t++) pos += d.slot_of[t] > me ? 1 : 0;
    return pos;
}
__device__ unsigned long long ang_key(const FmDev &d, int j, int e)
{
    const int p = e & NB_INDEX_MASK, code = e >> NB_SHIFT_BITS;
    if (code != NB_NOSHIFT) return (1ull << 62) | (unsigned long long)d.slot_of[p];
    const int SX[13] = {1, 1, 0, -1, 0, 1, 1, 0, -1, -1, -1, 0, 1};  // the 13 forward shifts (:686-688)
    const int SY[13] = {0, 1, 1, 1, 0, 0, 1, 1, 1, 0, -1, -1, -1};
    const int SZ[13] = {0, 0, 0, 0, 1, 1, 1, 1, 1, 1, 1, 1, 1};
    const int cj = ang_cell_of(d, j), cp = ang_cell_of(d, p);
    const int ne0 = d.ne[0], ne1 = d.ne[1];
    const int jx = cj % ne0, jy = (cj / ne0) % ne1, jz = cj / (ne0 * ne1);
    const int px = cp % ne0, py = (cp / ne0) % ne1, pz = cp / (ne0 * ne1);
    const int pj = ang_list_pos(d, cj, j), pp = ang_list_pos(d, cp, p);
    int oc = cj, sub = 0, pa = min(pj, pp), pb = max(pj, pp);
    if (cj != cp) {
        const int dx = px - jx, dy = py - jy, dz = pz - jz;
        for (int k = 0; k < 13; k++) {
            if (SX[k] == dx && SY[k] == dy && SZ[k] == dz) { oc = cj; sub = 1 + k; pa = pj; pb = pp; }
            if (SX[k] == -dx && SY[k] == -dy && SZ[k] == -dz) { oc = cp; sub = 1 + k; pa = pp; pb = pj; }
        }
    }
    const int ox = oc % ne0, oy = (oc / ne0) % ne1, oz = oc / (ne0 * ne1);
    const unsigned long long rank = ((unsigned long long)(ox - 1) * (unsigned)(d.nc[1]) + (unsigned)(oy - 1)) *
                                        (unsigned)(d.nc[2]) + (unsigned)(oz - 1);
    return (rank << 34) | ((unsigned long long)sub << 30) | ((unsigned long long)pa << 15) | (unsigned long long)pb;
}

__global__ void k_angular_order(FmDev d, int gated, int iter)
{
    pdl_enter();
    if (!gate(d, gated)) return;
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < d.n; j += gridDim.x * blockDim.x) {
        if (d.funcy[j] != 2) continue;
        if (d.nbond[j] != 2) { raise_status(d, ST_ANGLE, iter); continue; }
        const int e0 = d.bnd[(size_t)j * 4], e1 = d.bnd[(size_t)j * 4 + 1];
        if (ang_key(d, j, e1) < ang_key(d, j, e0)) {
            d.bnd[(size_t)j * 4] = e1;
            d.bnd[(size_t)j * 4 + 1] = e0;
        }
    }
}

__global__ void k_set_funcy(FmDev d, const int32_t *funcy_up)
{
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u < d.n) d.funcy[u] = funcy_up[u];  // slots still equal upload indices
}

// ---------------------------------------------------------------------------
// tiled forces: the same pair sums, partners read from a shared-memory
// staging of the block's neighbourhood (fm_tile.cuh) instead of gathered
// from global memory one list entry at a time
// ---------------------------------------------------------------------------

// One CTA takes a block of 2x2x2 cells at a time (handed out from an atomic
// counter): it stages the positions of the block's 4x4x4-cell neighbourhood,
// periodic images applied with the same single FP64 add as every other path
// (image(): x_src +/- L), as FP64 rows of 32 candidates; then T lanes per
// owner walk the owner's row of 16-bit staging offsets, T consecutive entries
// at a time, and evaluate each pair exactly as k_force does (FP64 cutoff test
// without contraction, the same pair_acc and epilogue).  Record partials are
// written per block (a fixed row whatever CTA took it), so the record sums do
// not depend on the hand-out order.
constexpr int FT_THREADS = FORCE_THREADS;
constexpr int FT_WARPS = FT_THREADS / 32;

// FP32 LJ pair of the precision form on the tiled path: the pair magnitude
// 48 s^7 - 24 s^4 = s^4 (48 s^3 - 24) in FP32 from an approximate reciprocal
// (rcp.approx, relative error ~2^-23 -- far inside the form's 1e-5
// tolerance), scaled by the FP64 rij; LJ_energy 4 (s^6 - s^3) - potshift on
// record steps.
template <bool REC>
__device__ __forceinline__ double lj32_pair(double r2, double dx, double dy, double dz, double potshift,
                                            double &fx, double &fy, double &fz, double &pe, double &vir)
{
    const float r2f = __double2float_rn(r2);
    float s;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(s) : "f"(r2f));
    const float s2 = s * s, s3 = s2 * s, s4 = s2 * s2;
    const double acc = (double)(s4 * fmaf(48.0f, s3, -24.0f));
    fx = fma(acc, dx, fx); fy = fma(acc, dy, fy); fz = fma(acc, dz, fz);
    if (REC) {
        pe += (double)(4.0f * (s3 * s3 - s3)) - potshift;
        vir += acc * r2;
    }
    return acc;
}

__device__ __forceinline__ uint2 ld_stream_uint2(const uint2 *p)
{
    uint2 r;
    asm("ld.global.nc.L1::no_allocate.v2.u32 {%0, %1}, [%2];" : "=r"(r.x), "=r"(r.y) : "l"(p));
    return r;
}

template <int T, bool REC, int MODE, int PREC>
__global__ void __launch_bounds__(FT_THREADS, REC ? 2 : 4) k_force_tile(FmDev d)
{
    constexpr bool NEEDW = (PREC & 6) != 0;  // Mie types / Soddemann bead flags ride in w
    constexpr bool LJ32 = PREC == 1;         // plain LJ, FP32 pair magnitude
    constexpr int R = NEEDW ? 4 : 3;
    constexpr int G = 32 / T;                // owners per warp per pass
    extern __shared__ double stg[];
    __shared__ int s_off[TILE_NSEGP];
    __shared__ int s_start[TILE_NSEG];
    __shared__ int s_code[TILE_NSEG];
    __shared__ int s_opre[9], s_ostart[8];
    __shared__ int s_blk, s_frozen, s_onext;
    pdl_enter();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) s_frozen = frozen(d) ? 1 : 0;
    // the dummy candidate after the capacity: far from every owner (the
    // staging below never writes index ucap)
    if (tid < R) stg[tile_woff(d.tile_ucap, R) + 32 * tid] = tid < 3 ? 1e30 : 1.0;
    __syncthreads();
    if (s_frozen) return;
    const int pset = d.sc->pset;
    const double4 *__restrict__ P = cur_pos(d, pset);
    const int sub = lane % T, og = lane / T;
    const unsigned dummy = (unsigned)tile_boff(d.tile_ucap, R);
    const unsigned lim2 = dummy | (dummy << 16);  // no byte offset beyond the dummy's
    const char *sbase = reinterpret_cast<const char *>(stg);
    const double Lx = d.L[0], Ly = d.L[1], Lz = d.L[2];
    const double rc2 = d.rc2;
    double m2max = 0.0;
    for (;;) {
        if (tid == 0) {
            const int b = atomicAdd(&d.sc->tile_next, 1);
            // every CTA takes exactly one number past the last block; the CTA
            // that takes the very last one resets the counter for the next launch
            if (b == d.tile_nblk + (int)gridDim.x - 1) d.sc->tile_next = 0;
            s_blk = b;
            s_onext = 0;
        }
        __syncthreads();
        const int blk = s_blk;
        if (blk >= d.tile_nblk) break;
        const int bx = blk % d.tile_nb[0], by = (blk / d.tile_nb[0]) % d.tile_nb[1];
        const int bz = blk / (d.tile_nb[0] * d.tile_nb[1]);
        const int x0 = 2 * bx, y0 = 2 * by, z0 = 2 * bz;
        if (tid < TILE_NSEG) {
            int st, cnt, code;
            tile_segment(d.ne, d.cell_start, x0, y0, z0, tid, st, cnt, code);
            s_start[tid] = st;
            s_code[tid] = code;
        }
        if (tid < TILE_NSEGP) s_off[tid] = d.blk_off[(size_t)blk * TILE_NSEGP + tid];
        if (warp == FT_WARPS - 1) {  // the block's owner cells a + 2b + 4c and their prefix
            int cnt = 0, st = 0;
            if (lane < 8) {
                const int x = x0 + (lane & 1), yy = y0 + ((lane >> 1) & 1), z = z0 + (lane >> 2);
                if (x < d.ne[0] && yy < d.ne[1] && z < d.ne[2]) {
                    const int c = x + d.ne[0] * (yy + d.ne[1] * z);
                    st = d.cell_start[c];
                    cnt = d.cell_start[c + 1] - st;
                }
            }
            int incl = cnt;
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
            if (lane < 8) { s_opre[lane + 1] = incl; s_ostart[lane] = st; }
            if (lane == 0) s_opre[0] = 0;
        }
        __syncthreads();
        // stage, two candidates per thread per pass (both loads in flight); a
        // block above the capacity was refused by k_blk_seg before the build
        const int U = min(s_off[TILE_NSEG], d.tile_ucap);
        for (int c0 = tid; c0 < U; c0 += 2 * FT_THREADS) {
            double4 p[2];
            int code[2], cc[2];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int c = min(c0 + h * FT_THREADS, U - 1);  // a repeat of the last is harmless
                int k = 0;  // segment containing c: largest k with s_off[k] <= c
#pragma unroll
                for (int step = 64; step > 0; step >>= 1)
                    if (k + step < TILE_NSEG && s_off[k + step] <= c) k += step;
                p[h] = ldg_pos(P + s_start[k] + (c - s_off[k]));
                code[h] = s_code[k];
                cc[h] = c;
            }
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int w = tile_woff(cc[h], R);
                stg[w] = image(p[h].x, (code[h] & 3) - 1, Lx);
                stg[w + 32] = image(p[h].y, ((code[h] >> 2) & 3) - 1, Ly);
                stg[w + 64] = image(p[h].z, ((code[h] >> 4) & 3) - 1, Lz);
                if (NEEDW) stg[w + 96] = p[h].w;
            }
        }
        __syncthreads();
        const int nown = s_opre[8];
        double pacc[RS_N];
#pragma unroll
        for (int q = 0; q < RS_N; q++) pacc[q] = 0.0;
        // owner groups: handed out from a shared counter (the warps of a block
        // finish together), or in a fixed order on record steps so that the
        // block's record partial is summed in the same order every time
        for (int pass = 0;; pass++) {
            int base;
            if (REC) {
                base = (warp + pass * FT_WARPS) * G;
            } else {
                if (lane == 0) base = atomicAdd(&s_onext, G);
                base = __shfl_sync(0xffffffffu, base, 0);
            }
            if (base >= nown) break;
            const int k = base + og;
            const bool act = k < nown;
            int i = 0;
            if (act) {
                int oc = 0;
#pragma unroll
                for (int q = 1; q < 8; q++) oc += k >= s_opre[q] ? 1 : 0;
                i = s_ostart[oc] + (k - s_opre[oc]);
            }
            double fx = 0.0, fy = 0.0, fz = 0.0, pe = 0.0, vir = 0.0;
            double rf[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
            double4 pi = make_double4(0.0, 0.0, 0.0, 0.0);
            if (act) {
                pi = ldg_pos(P + i);
                const int nch = (d.nnbr[i] + 4 * T - 1) / (4 * T);  // rows are padded to whole chunks
                const uint2 *row = reinterpret_cast<const uint2 *>(d.nbr16 + tile_row16(i, d.maxn16)) + sub;
                for (int c = 0; c < nch; c++) {
                    uint2 e = ld_stream_uint2(row + c * T);
                    e.x = __vminu2(e.x, lim2);
                    e.y = __vminu2(e.y, lim2);
                    const unsigned off[4] = {e.x & 0xffffu, e.x >> 16, e.y & 0xffffu, e.y >> 16};
                    double xj[4], yj[4], zj[4], wj[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const double *pj = reinterpret_cast<const double *>(sbase + off[q]);
                        xj[q] = pj[0];
                        yj[q] = pj[32];
                        zj[q] = pj[64];
                        wj[q] = NEEDW ? pj[96] : 0.0;
                    }
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const double dx = __dsub_rn(pi.x, xj[q]);
                        const double dy = __dsub_rn(pi.y, yj[q]);
                        const double dz = __dsub_rn(pi.z, zj[q]);
                        const double r2 = norm2_rn(dx, dy, dz);
                        if (r2 < rc2) {
                            double acc;
                            if (LJ32) acc = lj32_pair<REC>(r2, dx, dy, dz, d.potshift, fx, fy, fz, pe, vir);
                            else acc = pair_acc<PREC, REC>(d, r2, dx, dy, dz, pi.w, wj[q], fx, fy, fz, pe, vir);
                            if (REC && d.pressure) add_rf(rf, acc, dx, dy, dz);
                        }
                    }
                }
            }
            if (T > 1) {
#pragma unroll
                for (int o = T / 2; o > 0; o >>= 1) {
                    fx += __shfl_xor_sync(0xffffffffu, fx, o);
                    fy += __shfl_xor_sync(0xffffffffu, fy, o);
                    fz += __shfl_xor_sync(0xffffffffu, fz, o);
                    if (REC) {
                        pe += __shfl_xor_sync(0xffffffffu, pe, o);
                        vir += __shfl_xor_sync(0xffffffffu, vir, o);
                        if (d.pressure) {
#pragma unroll
                            for (int q = 0; q < 6; q++) rf[q] += __shfl_xor_sync(0xffffffffu, rf[q], o);
                        }
                    }
                }
            }
            if (act && sub == 0) {
                double part[RS_N];
#pragma unroll
                for (int q = 0; q < RS_N; q++) part[q] = 0.0;
                const double m2 = owner_finish<REC, MODE, PREC>(d, pset, P, i, fx, fy, fz, pe, vir, part, rf);
                m2max = fmax(m2max, m2);
                if (REC) {
#pragma unroll
                    for (int q = 0; q < RS_N; q++)
                        pacc[q] = q == RS_PEMAX ? fmax(pacc[q], part[q]) : pacc[q] + part[q];
                }
            }
        }
        if (REC) block_partials(d, pacc, blk);
        __syncthreads();  // the next block overwrites the staging
    }
    if (MODE >= 2) block_vmax2(d, m2max);
}

// Decodes tiled rows into the generic int32 layout (rows of maxn at out),
// owner by owner: its block from its cell (cell_start), each offset back to
// a staging position, its segment by the block's prefix, and the segment's
// slot and image code (test hooks only).
__global__ void k_tile_to_generic(FmDev d, int32_t *out, int maxn)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.n) return;
    int lo = 0, hi = d.ncell - 1;  // largest c with cell_start[c] <= i
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (d.cell_start[mid] <= i) lo = mid; else hi = mid - 1;
    }
    const int c = lo;
    const int cx = c % d.ne[0], cy = (c / d.ne[0]) % d.ne[1], cz = c / (d.ne[0] * d.ne[1]);
    const int blk = tile_block_of(d.tile_nb, cx, cy, cz);
    const int32_t *off = d.blk_off + (size_t)blk * TILE_NSEGP;
    const int cnt = min(d.nnbr[i], maxn);
    const uint16_t *row = d.nbr16 + tile_row16(i, d.maxn16);
    for (int k = 0; k < cnt; k++) {
        const int cand = tile_cand(row[tile_pos16(k, d.tile_T)], d.tile_R);
        int s = 0;
        for (int step = 64; step > 0; step >>= 1)
            if (s + step < TILE_NSEG && off[s + step] <= cand) s += step;
        int st, n, code;
        tile_segment(d.ne, d.cell_start, cx & ~1, cy & ~1, cz & ~1, s, st, n, code);
        out[nb_row(i, maxn) + nb_col(k)] = (st + (cand - off[s])) | (code << NB_SHIFT_BITS);
    }
}

// Neumaier-compensated reduction of the per-block partials into one record
// (evaluate_macroscopic_properties, simulation_record.f90:1205-1314).
// One block: every thread sums a share of the rows, the warps merge by a fixed
// xor tree and one thread per quantity merges the warps, so that nothing
// longer than a few dozen merges is ever waited for (one thread merging all
// 256 took 47-72 us a record step, whatever the system's size).
constexpr int REC_THREADS = 512;
__global__ void __launch_bounds__(REC_THREADS) k_record(FmDev d, int iter, double simtime)
{
    pdl_enter();
    if (frozen(d)) return;
    __shared__ double ws[RS_N][REC_THREADS / 32], wc[RS_N][REC_THREADS / 32], tot[RS_N];
    const int nq = d.pressure ? (int)RS_N : (int)RS_PXX;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double sum[RS_N], cmp[RS_N];
#pragma unroll
    for (int k = 0; k < RS_N; k++) { sum[k] = 0.0; cmp[k] = 0.0; }
    for (int b = threadIdx.x; b < d.nblocks_force; b += REC_THREADS) {
#pragma unroll
        for (int k = 0; k < RS_N; k++) {
            if (k >= nq) break;
            const double x = d.partial[(size_t)b * RS_N + k];
            if (k == RS_PEMAX) sum[k] = fmax(sum[k], x);
            else neumaier(sum[k], cmp[k], x);
        }
    }
#pragma unroll
    for (int k = 0; k < RS_N; k++) {
        if (k >= nq) break;
        if (k == RS_PEMAX) {
            sum[k] = warp_max(sum[k]);
        } else {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const double s2 = __shfl_xor_sync(0xffffffffu, sum[k], o), c2 = __shfl_xor_sync(0xffffffffu, cmp[k], o);
                nmerge(sum[k], cmp[k], s2, c2);
            }
        }
        if (lane == 0) { ws[k][w] = sum[k]; wc[k][w] = cmp[k]; }
    }
    __syncthreads();
    if (threadIdx.x < nq) {
        const int k = threadIdx.x;
        double s = ws[k][0], c = wc[k][0];
        for (int q = 1; q < REC_THREADS / 32; q++) {
            if (k == RS_PEMAX) s = fmax(s, ws[k][q]);
            else nmerge(s, c, ws[k][q], wc[k][q]);
        }
        tot[k] = s + c;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const double gnp = (double)d.n;
        FmRecord r;
        r.iter = iter;
        r.pad_ = 0;
        r.simtime = simtime;
        r.vsum = tot[RS_VSUM];
        r.mv2sum = tot[RS_MV2];
        r.virial = tot[RS_VIR];
        r.kinenergy = (0.5 * r.mv2sum) / gnp;
        r.potenergy = (0.5 * tot[RS_PE]) / gnp + d.pot_slrc;
        r.totenergy = r.kinenergy + r.potenergy;
        r.temperature = r.mv2sum / (3.0 * gnp);
        r.pressure = (d.density / (gnp * 3.0)) * (r.mv2sum + r.virial / 2.0) + d.p_slrc;
        int slot = d.sc->nrec_pending % d.rec_cap;
        d.rec[slot] = r;
        d.sc->nrec_pending += 1;
        if (d.pressure) {  // Pxy = Pxy + Pxytemp / volume (simulation_record.f90:3213-3217)
            const double volume = d.L[0] * d.L[1] * d.L[2];
            for (int q = 0; q < 6; q++) d.sc->pacc[q] += tot[RS_PXX + q] / volume;
            d.sc->pcount += 1;
        }
        if (tot[RS_PEMAX] > 10000.0) raise_status(d, ST_PE, iter);
    }
}

// Record partials from per-molecule arrays and current velocities
// (evaluate_macroscopic_properties reads potenergymol, virialmol and v).
constexpr int MACRO_THREADS = 256;
__global__ void __launch_bounds__(MACRO_THREADS) k_macro_partials(FmDev d)
{
    pdl_enter();
    if (frozen(d)) return;
    int i = blockIdx.x * MACRO_THREADS + threadIdx.x;
    double part[RS_N] = {};
    if (i < d.n) {
        double vx = d.vx[i], vy = d.vy[i], vz = d.vz[i];
        if (d.integrator == 0) {  // leap-frog records v + a dt/2
            vx = __dadd_rn(vx, __dmul_rn(__dmul_rn(0.5, d.ax[i]), d.dt));
            vy = __dadd_rn(vy, __dmul_rn(__dmul_rn(0.5, d.ay[i]), d.dt));
            vz = __dadd_rn(vz, __dmul_rn(__dmul_rn(0.5, d.az[i]), d.dt));
        }
        const double mass = d.mie ? d.mie_mass[mie_type(cur_pos(d, d.sc->pset)[i].w) - 1] : 1.0;
        part[RS_PE] = d.pe[i];
        part[RS_VIR] = d.vir[i];
        part[RS_MV2] = mass * norm2_rn(vx, vy, vz);
        part[RS_VSUM] = mass * __dadd_rn(__dadd_rn(vx, vy), vz);
        part[RS_PEMAX] = d.pe[i];
        if (d.pressure) {
            const double *q = d.rf6 + 6 * (size_t)i;
            const double rf[6] = {q[0], q[1], q[2], q[3], q[4], q[5]};
            pressure_part(part, vx, vy, vz, rf);
        }
    }
    block_partials<MACRO_THREADS>(d, part, blockIdx.x);
}

// ---------------------------------------------------------------------------
// all pairs with per-axis minimum image (simulation_compute_forces_LJ_AP,
// simulation_compute_forces.f90:280-341), both sides evaluated per molecule
// ---------------------------------------------------------------------------

constexpr int AP_THREADS = 128;
template <bool REC, int MODE, int PREC>
__global__ void __launch_bounds__(AP_THREADS) k_all_pairs(FmDev d, int lanes)
{
    pdl_enter();
    if (frozen(d)) return;
    const int pset = d.sc->pset;
    const double4 *P = cur_pos(d, pset);
    const int i = (blockIdx.x * AP_THREADS + threadIdx.x) / lanes, lane = threadIdx.x % lanes;
    const bool active = i < d.n;
    __shared__ double4 tile[AP_THREADS];
    double4 pi = active ? P[i] : make_double4(0, 0, 0, 0);
    double fx = 0.0, fy = 0.0, fz = 0.0, pe = 0.0, vir = 0.0;
    for (int t0 = 0; t0 < d.n; t0 += AP_THREADS) {
        int j0 = t0 + threadIdx.x;
        if (j0 < d.n) tile[threadIdx.x] = P[j0];
        __syncthreads();
        int m = min(AP_THREADS, d.n - t0);
        if (active) {
            for (int q = lane; q < m; q += lanes) {
                if (t0 + q == i) continue;
                double4 pj = tile[q];
                double r[3] = {__dsub_rn(pi.x, pj.x), __dsub_rn(pi.y, pj.y), __dsub_rn(pi.z, pj.z)};
                double r2 = 0.0;
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    if (fabs(r[k]) > d.hd[k]) r[k] = __dsub_rn(r[k], copysign(d.L[k], r[k]));
                    r2 = __dadd_rn(r2, __dmul_rn(r[k], r[k]));
                }
                if (r2 < d.rc2) pair_acc<PREC, REC>(d, r2, r[0], r[1], r[2], pi.w, pj.w, fx, fy, fz, pe, vir);
            }
        }
        __syncthreads();
    }
    for (int o = lanes >> 1; o > 0; o >>= 1) {
        fx += __shfl_xor_sync(0xffffffffu, fx, o);
        fy += __shfl_xor_sync(0xffffffffu, fy, o);
        fz += __shfl_xor_sync(0xffffffffu, fz, o);
        if (REC) {
            pe += __shfl_xor_sync(0xffffffffu, pe, o);
            vir += __shfl_xor_sync(0xffffffffu, vir, o);
        }
    }
    double part[RS_N] = {};
    double m2 = 0.0;
    const double rf[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};  // simulation_compute_forces_LJ_AP records no rf
    if (active && lane == 0) m2 = epilogue<REC, MODE, (PREC & 2) != 0>(d, pset, i, pi, fx, fy, fz, pe, vir, part, rf);
    if (REC) block_partials<AP_THREADS>(d, part, blockIdx.x);
    if (MODE >= 2) block_vmax2(d, m2);
}

// ---------------------------------------------------------------------------
// test hooks and layout conversion
// ---------------------------------------------------------------------------

__device__ __forceinline__ uint64_t mix64(uint64_t x)
{
    x ^= x >> 30; x *= 0xbf58476d1ce4e5b9ull;
    x ^= x >> 27; x *= 0x94d049bb133111ebull;
    x ^= x >> 31;
    return x;
}

__global__ void k_pair_digest(FmDev d, const int32_t *glob_of_upload)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    uint64_t h = 0ull;
    long long cnt = 0;
    if (i < d.n) {
        int gi = glob_of_upload[d.slot_of[i]];
        const int32_t *L = d.nbr + nb_row(i, d.maxn);
        for (int k = 0; k < d.nnbr[i]; k++) {
            int e = L[nb_col(k)];
            int j = e & NB_INDEX_MASK;
            int code6 = e >> NB_SHIFT_BITS;
            int sx = (code6 & 3) - 1, sy = ((code6 >> 2) & 3) - 1, sz = ((code6 >> 4) & 3) - 1;
            int code = (sx + 1) + 3 * (sy + 1) + 9 * (sz + 1);
            int gj = glob_of_upload[d.slot_of[j]];
            if (code == 13) {
                if (gi < gj) {  // both directions are stored; count the unordered pair once
                    h += mix64(((uint64_t)(uint32_t)gi << 32) ^ (uint64_t)(uint32_t)gj);
                    cnt++;
                }
            } else {
                h += mix64((((uint64_t)(uint32_t)gi << 32) ^ (uint64_t)(uint32_t)gj) * 31ull + (uint64_t)code + 0x9e3779b97f4a7c15ull);
                cnt++;
            }
        }
    }
    h = warp_sum<unsigned long long>(h);
    cnt = warp_sum<long long>(cnt);
    if ((threadIdx.x & 31) == 0 && (h || cnt)) {
        atomicAdd((unsigned long long *)&d.sc->digest, (unsigned long long)h);
        atomicAdd((unsigned long long *)&d.sc->digest_n, (unsigned long long)cnt);
    }
}

// Types of an uploaded state (slots still equal upload indices).
// w of each position from the Mie type (moltype) and the Soddemann bead flag
// (solvent_flag 1: 1 for a chain bead, 0 for a solvent molecule, chainID 0):
// the type, the flag, or the type + 32 x the flag with both.  Run after either
// is uploaded, while slots still equal upload indices; a part not uploaded
// yet reads as 0 (type) or the zeroed chain ids.
__global__ void k_set_w(FmDev d)
{
    int u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= d.n) return;
    const int type = d.mie && d.mie_type_up ? d.mie_type_up[u] : 0;
    const int flag = d.solvent ? (d.chain[u] != 0 ? 1 : 0) : 0;
    cur_pos(d, d.sc->pset)[u].w = (double)(type + (d.mie ? 32 : 1) * flag);
}

// upload order u -> slot u (uploads start in upload order)
__global__ void k_scatter_state(FmDev d, const double *r3, const double *v3, const double *a3)
{
    int u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= d.n) return;
    double4 *P = cur_pos(d, d.sc->pset);
    P[u] = make_double4(r3[3 * (size_t)u], r3[3 * (size_t)u + 1], r3[3 * (size_t)u + 2],
                        d.mie ? (double)d.mie_type_up[u] : 0.0);
    d.vx[u] = v3[3 * (size_t)u]; d.vy[u] = v3[3 * (size_t)u + 1]; d.vz[u] = v3[3 * (size_t)u + 2];
    if (a3) { d.ax[u] = a3[3 * (size_t)u]; d.ay[u] = a3[3 * (size_t)u + 1]; d.az[u] = a3[3 * (size_t)u + 2]; }
    else { d.ax[u] = 0.0; d.ay[u] = 0.0; d.az[u] = 0.0; }
    d.slot_of[u] = u;
}

__global__ void k_gather_state(FmDev d, double *r3, double *v3, double *a3, int32_t *uidx_out, double *pe,
                               double *vir)
{
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= d.n) return;
    int u = d.slot_of[s];
    const double4 *P = cur_pos(d, d.sc->pset);
    if (r3) { double4 p = P[s]; r3[3 * (size_t)u] = p.x; r3[3 * (size_t)u + 1] = p.y; r3[3 * (size_t)u + 2] = p.z; }
    if (v3) { v3[3 * (size_t)u] = d.vx[s]; v3[3 * (size_t)u + 1] = d.vy[s]; v3[3 * (size_t)u + 2] = d.vz[s]; }
    if (a3) { a3[3 * (size_t)u] = d.ax[s]; a3[3 * (size_t)u + 1] = d.ay[s]; a3[3 * (size_t)u + 2] = d.az[s]; }
    if (uidx_out) uidx_out[s] = u;
    if (pe) pe[u] = d.pe[s];
    if (vir) vir[u] = d.vir[s];
}

inline int nblk(int n, int t) { return (n + t - 1) / t; }

}  // namespace

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------


void launch_reset_scalars(const FmDev &d, cudaStream_t st) { k_reset_scalars<<<1, 1, 0, st>>>(d); }
void launch_move1(const FmDev &d, cudaStream_t st) { pdl_launch(k_move1, nblk(d.n, 256), 256, st, d); }
void launch_move2(const FmDev &d, cudaStream_t st) { pdl_launch(k_move2, nblk(d.n, 256), 256, st, d); }
void launch_vmax(const FmDev &d, cudaStream_t st) { pdl_launch(k_vmax, nblk(d.n, 256), 256, st, d); }
void launch_move_lfv(const FmDev &d, cudaStream_t st) { pdl_launch(k_move_lfv, nblk(d.n, 256), 256, st, d); }
void launch_disp(const FmDev &d, cudaStream_t st) { pdl_launch(k_disp, nblk(d.n, 256), 256, st, d); }

void launch_decide_graph(const FmDev &d, int flip, int crit, int fixed_rebuild, double half_min_delta,
                         cudaGraphConditionalHandle cond, int body_kernels, cudaStream_t st)
{
    k_decide_graph<<<1, 1, 0, st>>>(d, flip, crit, fixed_rebuild > 0 ? fixed_rebuild : 1, half_min_delta, cond,
                                    body_kernels);
}

void launch_set_graph_iter(const FmDev &d, int iter, cudaStream_t st) { k_set_graph_iter<<<1, 1, 0, st>>>(d, iter); }

void launch_decide(const FmDev &d, int iter, int flip, int crit, int fixed_rebuild, double half_min_delta,
                   cudaStream_t st)
{
    pdl_launch(k_decide, 1, 1, st, d, iter, flip, crit, fixed_rebuild > 0 ? fixed_rebuild : 1, half_min_delta);
}
// Gated kernels run grid-stride loops on a bounded grid, so that a launch the
// device decision turns into a no-op costs a few microseconds at most.
constexpr int kSMs = 148;
inline int sgrid(int n, int t, int per_sm) { return std::min(nblk(n, t), kSMs * per_sm); }

void launch_wrap_bin(const FmDev &d, int wrap, int bin, int gated, int iter, cudaStream_t st)
{
    pdl_launch(k_wrap_bin, sgrid(d.n, 256, 8), 256, st, d, wrap, bin, gated, iter);
}
int scan_tiles(int ncell) { return nblk(ncell, SCAN_TILE); }
void launch_scan_cells(const FmDev &d, int gated, cudaStream_t st)
{
    pdl_launch(k_scan_tiles, scan_tiles(d.ncell), SCAN_THREADS, st, d, gated);
    pdl_launch(k_scan_apply, scan_tiles(d.ncell), SCAN_THREADS, st, d, gated);
}
void launch_scatter(const FmDev &d, int gated, cudaStream_t st)
{
    pdl_launch(k_scatter, sgrid(d.n, 256, 8), 256, st, d, gated);
    if (d.density * d.cs[0] * d.cs[1] * d.cs[2] < 5.0)
        pdl_launch(k_sort_cells_sparse, sgrid((d.ncell + 3) / 4, SORT_WARPS, 8), 32 * SORT_WARPS, st, d, gated);
    else
        pdl_launch(k_sort_cells, sgrid(d.ncell, SORT_WARPS, 8), 32 * SORT_WARPS, st, d, gated);
}
void launch_reorder(const FmDev &d, int gated, double4 *tpos, int32_t *tuidx, cudaStream_t st)
{
    pdl_launch(k_reorder_gather, sgrid(d.n, 256, 8), 256, st, d, gated, tpos, tuidx);
    pdl_launch(k_reorder_copy, sgrid(d.n, 256, 8), 256, st, d, gated, tpos, tuidx);
}
void launch_angular_order(const FmDev &d, int gated, int iter, cudaStream_t st)
{
    pdl_launch(k_angular_order, sgrid(d.n, 256, 8), 256, st, d, gated, iter);
}

void launch_set_funcy(const FmDev &d, const int32_t *funcy_up, cudaStream_t st)
{
    k_set_funcy<<<nblk(d.n, 256), 256, 0, st>>>(d, funcy_up);
}

void launch_blk_seg(const FmDev &d, int gated, int iter, cudaStream_t st)
{
    pdl_launch(k_blk_seg, sgrid(d.tile_nblk, BS_THREADS / 32, 8), BS_THREADS, st, d, gated, iter);
}

// Staging capacity of the tiled force kernel: list entries are 16-bit byte
// offsets into the staging, so it holds at most tile_ucap_max(R) candidates
// (2720 for x y z, 2016 with w) plus the dummy -- at most ~64 KB.
constexpr int TILE_SMEM_MAX = 232448 - 4096;
int tile_ucap_limit(int R) { return tile_ucap_max(R); }
size_t tile_smem_bytes(const FmDev &d) { return (size_t)tile_stage_doubles(d.tile_ucap, d.tile_R) * 8; }

template <int T, bool REC, int MODE, int PREC>
static void launch_force_tile_k(const FmDev &d, cudaStream_t st)
{
    auto k = k_force_tile<T, REC, MODE, PREC>;
    static size_t smem_set = 0;
    static int grid_for = -1, grid = 0;
    const size_t smem = tile_smem_bytes(d);
    if (smem_set == 0) {
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, TILE_SMEM_MAX);
        smem_set = 1;
    }
    if (grid_for != (int)smem) {  // resident CTAs at this staging size
        int dev = 0, nsm = kSMs, per_sm = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, FT_THREADS, smem);
        grid = std::max(nsm, 1) * std::max(per_sm, 1);
        grid_for = (int)smem;
    }
    pdl_launch_smem(k, std::min(grid, d.tile_nblk), FT_THREADS, smem, st, d);
}

template <int T>
static void launch_force_tile(const FmDev &d, int record, int mode, cudaStream_t st)
{
#define FM_TILE_CASE(R, M)                                                          \
    if (record == R && mode == M) {                                                 \
        switch (d.precision + 2 * d.mie + 4 * d.solvent) {                          \
        case 0: launch_force_tile_k<T, R, M, 0>(d, st); break;                      \
        case 1: launch_force_tile_k<T, R, M, 1>(d, st); break;                      \
        case 2: launch_force_tile_k<T, R, M, 2>(d, st); break;                      \
        case 3: launch_force_tile_k<T, R, M, 3>(d, st); break;                      \
        case 4: launch_force_tile_k<T, R, M, 4>(d, st); break;                      \
        case 5: launch_force_tile_k<T, R, M, 5>(d, st); break;                      \
        case 6: launch_force_tile_k<T, R, M, 6>(d, st); break;                      \
        default: launch_force_tile_k<T, R, M, 7>(d, st); break;                     \
        }                                                                           \
        return;                                                                     \
    }
    FM_TILE_CASE(0, 0) FM_TILE_CASE(0, 1) FM_TILE_CASE(0, 2) FM_TILE_CASE(0, 3)
    FM_TILE_CASE(1, 0) FM_TILE_CASE(1, 1) FM_TILE_CASE(1, 2) FM_TILE_CASE(1, 3)
#undef FM_TILE_CASE
}

void launch_tile_to_generic(const FmDev &d, int32_t *out, int maxn, cudaStream_t st)
{
    k_tile_to_generic<<<nblk(d.n, 128), 128, 0, st>>>(d, out, maxn);
}

int force_blocks(int n, int tpm) { return nblk(n * tpm, FORCE_THREADS); }
// Lanes per molecule: one lane's walk over all the others is what a small
// system waits for, a larger one for its blocks to fill the GPU evenly. FP64, us
// a step with 1 / 8 / 16 / 32 lanes: 500 molecules 98 / 17 / 12 / 10, 4,000: 598
// / 90 / 61 / 60, 6,912: 989 / 166 / 139 / 146, 8,788: 1,244 / 223 / 220 / 305, 16,384:
// 2,314 / 649 / 875 / 884, 37,044: 5,729 / 2,456 / 3,219 / 4,036; with 1 / 8 lanes
// 62,500: 9,806 / 6,696, 131,072: 29,232 / 27,924, 256,000: 105,890 / 104,400.
static int all_pairs_lanes(int n) { return n <= 8192 ? 32 : 8; }
int all_pairs_blocks(int n) { return nblk((long long)n * all_pairs_lanes(n), AP_THREADS); }

void launch_force(const FmDev &d, int record, int mode, int tpm, cudaStream_t st)
{
    if (d.tile) {
        if (d.tile_T == 4) launch_force_tile<4>(d, record, mode, st);
        else launch_force_tile<8>(d, record, mode, st);
        return;
    }
    if (d.mie || d.solvent) launch_force_types(d, record, mode, tpm, st);
    else launch_force_lj(d, record, mode, tpm, st);
}

void launch_all_pairs(const FmDev &d, int record, int mode, cudaStream_t st)
{
    const int g = all_pairs_blocks(d.n), lanes = all_pairs_lanes(d.n);
#define FM_AP_CASE(R, M)                                                            \
    if (record == R && mode == M) {                                                 \
        switch (d.precision + 2 * d.mie) {                                          \
        case 0: pdl_launch(k_all_pairs<R, M, 0>, g, AP_THREADS, st, d, lanes); break;           \
        case 1: pdl_launch(k_all_pairs<R, M, 1>, g, AP_THREADS, st, d, lanes); break;           \
        case 2: pdl_launch(k_all_pairs<R, M, 2>, g, AP_THREADS, st, d, lanes); break;           \
        default: pdl_launch(k_all_pairs<R, M, 3>, g, AP_THREADS, st, d, lanes); break;          \
        }                                                                           \
        return;                                                                     \
    }
    FM_AP_CASE(0, 0) FM_AP_CASE(0, 1) FM_AP_CASE(0, 2) FM_AP_CASE(0, 3)
    FM_AP_CASE(1, 0) FM_AP_CASE(1, 1) FM_AP_CASE(1, 2) FM_AP_CASE(1, 3)
#undef FM_AP_CASE
}

int macro_blocks(int n) { return nblk(n, MACRO_THREADS); }
void launch_macro_partials(const FmDev &d, cudaStream_t st)
{
    pdl_launch(k_macro_partials, macro_blocks(d.n), MACRO_THREADS, st, d);
}

void launch_record(const FmDev &d, int iter, double simtime, cudaStream_t st)
{
    pdl_launch(k_record, 1, REC_THREADS, st, d, iter, simtime);
}

void launch_pair_digest(const FmDev &d, const int32_t *glob_of_upload, cudaStream_t st)
{
    k_pair_digest<<<nblk(d.n, 256), 256, 0, st>>>(d, glob_of_upload);
}

void launch_set_types(const FmDev &d, cudaStream_t st) { k_set_w<<<nblk(d.n, 256), 256, 0, st>>>(d); }

void launch_set_bead_flags(const FmDev &d, cudaStream_t st) { k_set_w<<<nblk(d.n, 256), 256, 0, st>>>(d); }

__global__ static void k_count_up(int32_t *out, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = i + 1;
}
void launch_count_up(int32_t *out, int n, cudaStream_t st) { k_count_up<<<nblk(n, 256), 256, 0, st>>>(out, n); }

void launch_scatter_state(const FmDev &d, const double *r3, const double *v3, const double *a3, cudaStream_t st)
{
    k_scatter_state<<<nblk(d.n, 256), 256, 0, st>>>(d, r3, v3, a3);
}

void launch_gather_state(const FmDev &d, double *r3, double *v3, double *a3, int32_t *uidx, double *pe,
                         double *vir, cudaStream_t st)
{
    k_gather_state<<<nblk(d.n, 256), 256, 0, st>>>(d, r3, v3, a3, uidx, pe, vir);
}

}  // namespace fm
