// fm_rows.cuh -- neighbour rows by molecule: the list build of the gather
// force path, shared by the single-system kernel (fm_rows.cu) and the slot
// engine (fm_engine_kernels.cu).
//
// The pair set and the row order are those of build_cell (fm_build.cuh; pair
// set of assign_to_neighbourlist_halfint_opt, linklist.f90:660-804,
// 1118-1180): the candidates of the 27 cells around the owner's, cell by cell
// (x fastest), a cell's real molecules before the images a halo cell holds,
// each accepted when the exact FP64 test (dx^2+dy^2)+dz^2 < rneighbr2 says so.
//
// Shape: G consecutive lanes take a molecule. Cells are x fastest, so the
// neighbours of a cell in one (y, z) row of cells are one contiguous slot
// range and a molecule away from the x faces walks nine ranges (worked out one
// per lane and left in shared memory), G candidates a step: each lane loads one
// position and makes the exact test, the step's hits are one ballot, and a
// hit's place in the row is the count so far plus its rank in the ballot, so
// rows are in visiting order without any buffer. G is 32 for ranges of more than
// 20 candidates, 16 above 10, else 8 (rows_lanes).
//
// It is for systems that do not fill the GPU: the chain of steps of one
// molecule is short, where the build by warp (fm_build.cuh: a cell, or 2x2x2 of
// them, per warp) waits for the serial work of one warp, ~90 us however small
// the system is: a whole rebuild (cells, sort, reorder, rows) of 2,048 LJ
// molecules takes 34 us instead of 132, one of 32,000 90 instead of 152 (by
// fours, below). Bound by issue at larger sizes (some 80 instructions a step, 8
// of them FP64): the kernel alone takes 170 us by fours and 264 by molecule at
// 108,000 molecules against 155 by warp, whose staging in shared memory tests
// four owners per candidate loaded.
#pragma once
#include "fm_build.cuh"

namespace fm {

constexpr int ROWS_THREADS = 128;

// Lanes per molecule for per_cell molecules a cell: a range is three cells.
inline int rows_lanes(double per_cell) { return 3.0 * per_cell > 20.0 ? 32 : 3.0 * per_cell > 10.0 ? 16 : 8; }

// Candidate ranges of a molecule in cell c, in row order: range number r of
// rows_count(y, c) is slots [b, e) as entry bits `code` show them.  Cells x0 ..
// x1 of a row of cells are one range; the images that a halo cell at the low
// (high) x face holds come before (after) it.
__device__ __forceinline__ int rows_count(const CellSys &y, int cx) { return !y.dd && (cx == 1 || cx == y.ne[0] - 2) ? 18 : 9; }
__device__ __forceinline__ void rows_range(const CellSys &y, int cx, int cy, int cz, int n, int r, int &b, int &e,
                                           int &code)
{
    const int ne0 = y.ne[0], ne1 = y.ne[1], ne2 = y.ne[2];
    const int q = n == 18 ? r >> 1 : r;
    const bool image_x = n == 18 && ((r & 1) == (cx == 1 ? 0 : 1));
    const int y2 = cy + q % 3 - 1, z2 = cz + q / 3 - 1;
    int sx = 0, sy = 0, sz = 0, x0 = cx - 1, x1 = cx + 1;
    if (!y.dd) {  // (a subdomain's halo cells hold copies, met like any other cell's members)
        sy = y2 == 0 ? -1 : (y2 == ne1 - 1 ? 1 : 0);
        sz = z2 == 0 ? -1 : (z2 == ne2 - 1 ? 1 : 0);
        if (cx == 1) x0 = 1;
        if (cx == ne0 - 2) x1 = ne0 - 2;
        if (image_x) {
            sx = cx == 1 ? -1 : 1;
            x0 = x1 = cx == 1 ? ne0 - 2 : 1;
        }
    }
    const int32_t *row = y.cell_start + ne0 * ((y2 - sy * (ne1 - 2)) + ne1 * (z2 - sz * (ne2 - 2)));
    b = row[x0] - y.mol_off;
    e = row[x1 + 1] - y.mol_off;
    code = ((sx + 1) | ((sy + 1) << 2) | ((sz + 1) << 4)) << NB_SHIFT_BITS;
}

// The same with real molecules binned in halo cells (a coordinate exactly on a
// lower face): cell by cell, a halo cell's real members before its images, and
// no range between two halo cells.  Calls range(b, e, code).
template <typename F>
__device__ __forceinline__ void rows_strays(const CellSys &y, int cx, int cy, int cz, F &&range)
{
    const int ne0 = y.ne[0], ne1 = y.ne[1], ne2 = y.ne[2];
    const bool chalo = is_halo(cx, ne0) || is_halo(cy, ne1) || is_halo(cz, ne2);
#pragma unroll 1
    for (int q = 0; q < 54; q++) {
        const int k = q >> 1;
        const int x2 = cx + k % 3 - 1, y2 = cy + (k / 3) % 3 - 1, z2 = cz + k / 9 - 1;
        if (x2 < 0 || y2 < 0 || z2 < 0 || x2 >= ne0 || y2 >= ne1 || z2 >= ne2) continue;
        const bool h2 = is_halo(x2, ne0) || is_halo(y2, ne1) || is_halo(z2, ne2);
        if ((chalo && h2) || ((q & 1) && !h2)) continue;
        int sx = 0, sy = 0, sz = 0;
        if (q & 1) {
            sx = x2 == 0 ? -1 : (x2 == ne0 - 1 ? 1 : 0);
            sy = y2 == 0 ? -1 : (y2 == ne1 - 1 ? 1 : 0);
            sz = z2 == 0 ? -1 : (z2 == ne2 - 1 ? 1 : 0);
        }
        const int c = (x2 - sx * (ne0 - 2)) + ne0 * ((y2 - sy * (ne1 - 2)) + ne1 * (z2 - sz * (ne2 - 2)));
        range(y.cell_start[c] - y.mol_off, y.cell_start[c + 1] - y.mol_off,
              ((sx + 1) | ((sy + 1) << 2) | ((sz + 1) << 4)) << NB_SHIFT_BITS);
    }
}

// The ranges of a warp's groups, worked out one per lane.
template <int G>
struct RowsShared {
    int2 be[32 / G][18];
    int code[32 / G][18];
};

// Row of molecule i (cell c) of system y by the G consecutive lanes of a warp
// that are given it (lane g of them). Returns the row's length to every lane of
// the group.
template <int G>
__device__ __forceinline__ int rows_build(const CellSys &y, int i, int c, bool strays, int g, RowsShared<G> &sh)
{
    const unsigned shift = (threadIdx.x & 31u) & ~(unsigned)(G - 1);
    const unsigned ones = G == 32 ? 0xffffffffu : (1u << (G & 31)) - 1u;
    const unsigned group = ones << shift, lt = (1u << g) - 1u;
    const double4 pi = ldg_pos(y.P + i);
    const int maxn = y.maxn;
    int32_t *const row = y.nbr + nb_row(i, maxn);
    int cnt = 0;
    const int cx = c % y.ne[0], cy = (c / y.ne[0]) % y.ne[1], cz = c / (y.ne[0] * y.ne[1]);
    const int self_e = i | (NB_NOSHIFT << NB_SHIFT_BITS);
    auto scan = [&](int b, int e, int code) {
        for (int k = b; k < e; k += G) {
            const int j = k + g;
            const bool in = j < e;
            const double4 p = ldg_pos(y.P + (in ? j : b));
            double xj = p.x, yj = p.y, zj = p.z;
            if (code != NB_NOSHIFT << NB_SHIFT_BITS) {
                const int im = code >> NB_SHIFT_BITS;
                xj = image(xj, (im & 3) - 1, y.L[0]);
                yj = image(yj, ((im >> 2) & 3) - 1, y.L[1]);
                zj = image(zj, ((im >> 4) & 3) - 1, y.L[2]);
            }
            const double r2 = norm2_rn(__dsub_rn(pi.x, xj), __dsub_rn(pi.y, yj), __dsub_rn(pi.z, zj));
            const bool hit = in && r2 < y.rn2 && (j | code) != self_e;
            const unsigned m = (__ballot_sync(group, hit) >> shift) & ones;
            const int at = cnt + __popc(m & lt);
            if (hit && at < maxn) row[nb_col(at)] = j | code;
            cnt += __popc(m);
        }
    };
    if (strays) {
        rows_strays(y, cx, cy, cz, scan);
        return cnt;
    }
    const int n = rows_count(y, cx), gi = (threadIdx.x & 31) / G;
    __syncwarp(group);
    for (int r = g; r < n; r += G) {
        int b, e, code;
        rows_range(y, cx, cy, cz, n, r, b, e, code);
        sh.be[gi][r] = make_int2(b, e);
        sh.code[gi][r] = code;
    }
    __syncwarp(group);
#pragma unroll 1
    for (int r = 0; r < n; r++) {
        const int2 be = sh.be[gi][r];
        scan(be.x, be.y, sh.code[gi][r]);
    }
    return cnt;
}

// Rows of up to four molecules i0 .. i0 + own - 1 of cell c by a warp: as
// rows_build with 32 lanes, the four tests of a candidate sharing its load and
// the walk over the ranges (80 -> 45 instructions a test). Returns the longest
// row.
__device__ __forceinline__ int rows_four(const CellSys &y, int i0, int own, int n, bool strays, int cx, int cy, int cz,
                                         int lane, RowsShared<32> &sh)
{
    const unsigned lt = (1u << lane) - 1u;
    const int maxn = y.maxn;
    double ox[4], oy[4], oz[4];
    int cnt[4];
    unsigned row[4];
    int32_t *const base = y.nbr + nb_row(i0, maxn);  // the four rows are within one group's width of it
#pragma unroll
    for (int w = 0; w < 4; w++) {
        const int i = i0 + min(w, own - 1);
        const double4 p = ldg_pos(y.P + i);
        ox[w] = w < own ? p.x : 1e30; oy[w] = p.y; oz[w] = p.z;  // no molecule: r^2 is huge
        row[w] = (unsigned)(nb_row(i, maxn) - nb_row(i0, maxn));
        cnt[w] = 0;
    }
    auto scan = [&](int b, int e, int code) {
        const bool shifted = code != NB_NOSHIFT << NB_SHIFT_BITS;
        for (int k = b; k < e; k += 32) {
            const int j = k + lane;
            const double4 p = ldg_pos(y.P + min(j, e - 1));
            double xj = p.x, yj = p.y, zj = p.z;
            if (shifted) {
                const int im = code >> NB_SHIFT_BITS;
                xj = image(xj, (im & 3) - 1, y.L[0]);
                yj = image(yj, ((im >> 2) & 3) - 1, y.L[1]);
                zj = image(zj, ((im >> 4) & 3) - 1, y.L[2]);
            }
            if (j >= e) xj = -1e30;
            const int self = shifted ? -1 : j - i0;  // 0 .. 3: the candidate is that molecule
#pragma unroll
            for (int w = 0; w < 4; w++) {
                const double r2 = norm2_rn(__dsub_rn(ox[w], xj), __dsub_rn(oy[w], yj), __dsub_rn(oz[w], zj));
                const bool hit = r2 < y.rn2 && self != w;
                const unsigned m = __ballot_sync(0xffffffffu, hit);
                const int at = cnt[w] + __popc(m & lt);
                if (hit && at < maxn) base[row[w] + (unsigned)nb_col(at)] = j | code;
                cnt[w] += __popc(m);
            }
        }
    };
    if (strays) {
        rows_strays(y, cx, cy, cz, scan);
    } else {
#pragma unroll 1
        for (int r = 0; r < n; r++) scan(sh.be[0][r].x, sh.be[0][r].y, sh.code[0][r]);
    }
    int most = 0;
#pragma unroll
    for (int w = 0; w < 4; w++) {
        if (lane == w && w < own) y.nnbr[i0 + w] = min(cnt[w], maxn);
        most = max(most, cnt[w]);
    }
    return most;
}

// Unit u of the build by fours: ROWS_SPLIT warps share an interior cell. Where
// halo cells have molecules (strays, or a subdomain's copies, which get no
// rows), the first of a cell's warps looks after an equal share of them.
constexpr int ROWS_SPLIT = 5;
constexpr int ROWS_FOUR_MOLECULES = 16384;  // a warp's chain is longer: a whole rebuild of 2,048 molecules 50 us against 34
__host__ __device__ inline int rows_four_units(const int (&ne)[3])
{
    return (ne[0] - 2) * (ne[1] - 2) * (ne[2] - 2) * ROWS_SPLIT;
}
__device__ __forceinline__ int rows_four_unit(const CellSys &y, int u, bool strays, int lane, RowsShared<32> &sh)
{
    const int ne0 = y.ne[0], ne1 = y.ne[1], ne2 = y.ne[2];
    const int q = u / ROWS_SPLIT, part = u % ROWS_SPLIT;
    const int cx = 1 + q % (ne0 - 2), cy = 1 + (q / (ne0 - 2)) % (ne1 - 2), cz = 1 + q / ((ne0 - 2) * (ne1 - 2));
    const int c = cx + ne0 * (cy + ne1 * cz);
    int most = 0;
    const int b = y.cell_start[c] - y.mol_off, m = y.cell_start[c + 1] - y.mol_off - b;
    if (4 * part < m) {
        const int n = rows_count(y, cx);
        __syncwarp();
        if (!strays && lane < n) {
            int rb, re, code;
            rows_range(y, cx, cy, cz, n, lane, rb, re, code);
            sh.be[0][lane] = make_int2(rb, re);
            sh.code[0][lane] = code;
        }
        __syncwarp();
        for (int g = 4 * part; g < m; g += 4 * ROWS_SPLIT)
            most = max(most, rows_four(y, b + g, min(4, m - g), n, strays, cx, cy, cz, lane, sh));
    }
    if ((strays || y.dd) && part == 0) {
        const int nint = (ne0 - 2) * (ne1 - 2) * (ne2 - 2);
        for (int h = q; h < ne0 * ne1 * ne2; h += nint) {
            const int hx = h % ne0, hy = (h / ne0) % ne1, hz = h / (ne0 * ne1);
            if (!(is_halo(hx, ne0) || is_halo(hy, ne1) || is_halo(hz, ne2))) continue;
            const int hb = y.cell_start[h] - y.mol_off, hm = y.cell_start[h + 1] - y.mol_off - hb;
            if (y.dd) {
                for (int k = lane; k < hm; k += 32) y.nnbr[hb + k] = 0;
                continue;
            }
            for (int g = 0; g < hm; g += 4)
                most = max(most, rows_four(y, hb + g, min(4, hm - g), 0, true, hx, hy, hz, lane, sh));
        }
    }
    return most;
}

}  // namespace fm
