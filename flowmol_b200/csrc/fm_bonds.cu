// fm_bonds.cu -- bonds of polymers, found after every list build.
//
// The reference's check_update_adjacentbeadinfo (linklist.f90:2542-2584) bonds
// an owner with every candidate of the cells scanned for its list -- at any
// distance -- that has its chain and whose subchain bit is set in its bin_bflag
// words (get_bondflag, modules.f90:602-610, 31 bits per word). Instead of
// comparing chains for every candidate of the list build, a molecule looks up
// the few beads its flags name in a table of (chain, subchain) made when the
// monomers are uploaded, and keeps those whose cell is next to its own, in the
// order the list build would have met them. The comparisons were half of the
// build's time: 212 us per build of the 262,144-bead FENE melt with them.
// Where a named bead is not unique, or real molecules are binned in halo cells,
// a molecule scans its candidates instead.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "fm_common.cuh"
#include "fm_device.cuh"
#include "fm_force.cuh"
#include "fm_rows.cuh"

namespace fm {

namespace {

constexpr unsigned long long BT_EMPTY = ~0ull;
constexpr int BT_NONE = -1, BT_MANY = -2;
constexpr int BOND_SUBS = 4 * 31;  // subchain numbers the flag words can name

__device__ __forceinline__ unsigned long long bead_key(int chain, int sub)
{
    return (unsigned long long)(unsigned)chain << 32 | (unsigned)sub;
}
// The finaliser of splitmix64 (Steele, Lea and Flood, OOPSLA 2014) with other
// shifts and without its last one: the upper half of the product is taken.
__device__ __forceinline__ unsigned bead_hash(unsigned long long x)
{
    x ^= x >> 29; x *= 0xbf58476d1ce4e5b9ull;
    x ^= x >> 32; x *= 0x94d049bb133111ebull;
    return (unsigned)(x >> 32);
}
__device__ __forceinline__ bool names(const int4 &bf, int sub)
{
    const int pos = sub - 1, grp = pos / 31;
    const int word = grp == 0 ? bf.x : grp == 1 ? bf.y : grp == 2 ? bf.z : bf.w;
    return pos >= 0 && grp < 4 && ((word >> (pos % 31)) & 1);
}

// Slots still equal upload indices.
__global__ void k_bond_table(FmDev d)
{
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= d.n) return;
    const int sub = d.subchain[u];
    if (sub < 1 || sub > BOND_SUBS) return;  // no flag can name it
    const unsigned long long key = bead_key(d.chain[u], sub);
    for (unsigned h = bead_hash(key) & d.bt_mask;; h = (h + 1) & d.bt_mask) {  // the table is at most half full
        unsigned long long was = *(volatile unsigned long long *)&d.bt_key[h];
        if (was == BT_EMPTY) was = atomicCAS(&d.bt_key[h], BT_EMPTY, key);
        if (was != BT_EMPTY && was != key) continue;  // another bead's place
        if (*(volatile int *)&d.bt_val[h] != BT_MANY && atomicCAS(&d.bt_val[h], BT_NONE, u) != BT_NONE)
            d.bt_val[h] = BT_MANY;
        return;
    }
}

// Bonds of molecule i by scanning its candidates, in row order; returns how many.
__device__ int scan_bonds(const FmDev &d, int i, int cx, int cy, int cz, int chain, const int4 &bf, bool strays)
{
    CellSys y;
    y.cell_start = d.cell_start;
    y.mol_off = 0;
    y.dd = 0;
    for (int k = 0; k < 3; k++) y.ne[k] = d.ne[k];
    int nb = 0;
    auto range = [&](int b, int e, int code) {
        for (int j = b; j < e; j++) {
            if (d.chain[j] != chain || !names(bf, d.subchain[j]) || (j | code) == (i | (NB_NOSHIFT << NB_SHIFT_BITS))) continue;
            if (nb < 4) d.bnd[(size_t)i * 4 + nb] = j | code;
            nb++;
        }
    };
    if (strays) {
        rows_strays(y, cx, cy, cz, range);
    } else {
        const int n = rows_count(y, cx);
        for (int r = 0; r < n; r++) {
            int b, e, code;
            rows_range(y, cx, cy, cz, n, r, b, e, code);
            range(b, e, code);
        }
    }
    return nb;
}

// Offset of cell p from cell c along an axis of ne extended cells (two of them
// halo), and the image it is seen as: nearest across the boundary.
__device__ __forceinline__ int cell_offset(int p, int c, int ne, int &image_of)
{
    int o = p - c;
    image_of = 0;
    if (o == ne - 3) { o = -1; image_of = -1; }       // last interior cell, seen below the first
    else if (o == 3 - ne) { o = 1; image_of = 1; }
    return o;
}

__global__ void k_bonds(FmDev d, int gated, int iter)
{
    pdl_enter();
    if (!gate(d, gated)) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.n) return;
    const int4 bf = d.bflag[i];
    int nb = 0;
    if ((bf.x | bf.y | bf.z | bf.w) != 0) {
        const int chain = d.chain[i], c = d.cell_of[i], ne0 = d.ne[0], ne1 = d.ne[1];
        const int cx = c % ne0, cy = (c / ne0) % ne1, cz = c / (ne0 * ne1);
        bool scan = d.sc->strays != 0;
        unsigned long long key[4];  // (cell order, slot): the order in which the build meets them
        int ent[4];
        for (int w = 0; w < 4 && !scan; w++) {
            unsigned bits = (unsigned)(w == 0 ? bf.x : w == 1 ? bf.y : w == 2 ? bf.z : bf.w) & 0x7fffffffu;
            for (; bits != 0u && !scan; bits &= bits - 1u) {
                const unsigned long long want = bead_key(chain, 31 * w + __ffs(bits));
                int u = BT_NONE;
                for (unsigned h = bead_hash(want) & d.bt_mask;; h = (h + 1) & d.bt_mask) {
                    const unsigned long long k = d.bt_key[h];
                    if (k == want) u = d.bt_val[h];
                    if (k == want || k == BT_EMPTY) break;
                }
                if (u == BT_NONE) continue;
                if (u == BT_MANY) { scan = true; continue; }
                const int p = d.slot_by_upload[u];
                if (p == i) continue;
                const int pc = d.cell_of[p];
                int ix, iy, iz;
                const int ox = cell_offset(pc % ne0, cx, ne0, ix), oy = cell_offset((pc / ne0) % ne1, cy, ne1, iy);
                const int oz = cell_offset(pc / (ne0 * ne1), cz, d.ne[2], iz);
                if (abs(ox) > 1 || abs(oy) > 1 || abs(oz) > 1) continue;  // not scanned from here
                const unsigned long long at = (unsigned long long)((ox + 1) + 3 * (oy + 1) + 9 * (oz + 1)) << 32 | (unsigned)p;
                int e = p | ((ix + 1) | ((iy + 1) << 2) | ((iz + 1) << 4)) << NB_SHIFT_BITS;
                unsigned long long k = at;
#pragma unroll
                for (int q = 0; q < 4; q++) {  // insertion
                    if (q < nb && key[q] > k) {
                        const unsigned long long tk = key[q]; key[q] = k; k = tk;
                        const int te = ent[q]; ent[q] = e; e = te;
                    } else if (q == nb) {
                        key[q] = k; ent[q] = e;
                    }
                }
                nb++;
            }
        }
        if (scan) {
            nb = scan_bonds(d, i, cx, cy, cz, chain, bf, d.sc->strays != 0);
        } else {
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (q < nb) d.bnd[(size_t)i * 4 + q] = ent[q];
        }
    }
    d.nbond[i] = min(nb, 4);
    if (nb > 4) raise_status(d, ST_BOND, iter);  // too_many_bonds_error
}

}  // namespace

// Places of the table for n molecules: a power of two, at most half of it used.
size_t bond_table_size(int n)
{
    size_t s = 64;
    while (s < 2 * (size_t)n) s *= 2;
    return s;
}

void launch_bond_table(const FmDev &d, cudaStream_t st)
{
    cudaMemsetAsync(d.bt_key, 0xff, ((size_t)d.bt_mask + 1) * sizeof(unsigned long long), st);
    cudaMemsetAsync(d.bt_val, 0xff, ((size_t)d.bt_mask + 1) * sizeof(int32_t), st);
    k_bond_table<<<(d.n + 255) / 256, 256, 0, st>>>(d);
}

void launch_bonds(const FmDev &d, int gated, int iter, cudaStream_t st)
{
    pdl_launch(k_bonds, (d.n + 127) / 128, 128, st, d, gated, iter);
}

}  // namespace fm
