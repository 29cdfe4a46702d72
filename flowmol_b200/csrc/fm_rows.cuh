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
// rows are in visiting order without any buffer. G is the power of two nearest
// the length of a range.
//
// It is for systems that do not fill the GPU: the chain of steps of one
// molecule is short, where the build by warp (fm_build.cuh: a cell, or 2x2x2 of
// them, per warp) waits for the serial work of one warp, ~100 us however small
// the system is: a rebuild of 2,048 LJ molecules costs 34 us instead of 132,
// one of 32,000 104 instead of 152, a Soddemann solution of 25,092 beads (bonds
// looked up as well) 58 us for the rows instead of 290. Bound by issue at
// larger sizes (~45 instructions a step beside the 8 FP64 ones): at 108,000
// molecules 264 us against 160 by warp, whose shared staging tests four owners
// per candidate loaded.
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

// A group's ranges, worked out one per lane.
template <int G>
struct RowsShared {
    int2 be[ROWS_THREADS / G][18];
    int code[ROWS_THREADS / G][18];
};

// Row of molecule i (cell c) of system y by the G consecutive lanes of a warp
// that are given it (lane g of them). Returns the row's length and, through
// nb, its number of bonds, to every lane of the group.
template <int G, bool POLY>
__device__ __forceinline__ int rows_build(const CellSys &y, int i, int c, bool strays, int g, RowsShared<G> &sh, int &nb)
{
    const unsigned shift = (threadIdx.x & 31u) & ~(unsigned)(G - 1);
    const unsigned ones = G == 32 ? 0xffffffffu : (1u << (G & 31)) - 1u;
    const unsigned group = ones << shift, lt = (1u << g) - 1u;
    const double4 pi = ldg_pos(y.P + i);
    const int maxn = y.maxn;
    int32_t *const row = y.nbr + nb_row(i, maxn);
    int cnt = 0;
    nb = 0;
    int4 bf = make_int4(0, 0, 0, 0);
    int ochain = 0;
    if (POLY) { ochain = y.chain[i]; bf = y.bflag[i]; }
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
            if (POLY) {  // a candidate of the owner's chain whose subchain bit is set is bonded
                bool bond = in && y.chain[in ? j : b] == ochain && (j | code) != self_e;
                if (__any_sync(group, bond)) {
                    const int pos = bond ? y.subchain[j] - 1 : -1, grp = pos / 31;
                    const int word = grp == 0 ? bf.x : grp == 1 ? bf.y : grp == 2 ? bf.z : bf.w;
                    bond = pos >= 0 && grp < 4 && ((word >> (pos % 31)) & 1);
                    const unsigned mb = (__ballot_sync(group, bond) >> shift) & ones;
                    const int bat = nb + __popc(mb & lt);
                    if (bond && bat < 4) y.bnd[(size_t)i * 4 + bat] = j | code;
                    nb += __popc(mb);
                }
            }
        }
    };
    if (strays) {
        rows_strays(y, cx, cy, cz, scan);
        return cnt;
    }
    const int n = rows_count(y, cx), gi = threadIdx.x / G;
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

}  // namespace fm
