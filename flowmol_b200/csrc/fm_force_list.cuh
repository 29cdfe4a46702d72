// fm_force_list.cuh -- the force kernel of the neighbour-list modes: pair sums
// over list rows, bonds and angles, and the integrator epilogue.  Its
// instantiations are spread over fm_force_lj.cu (LJ / WCA) and
// fm_force_types.cu (Mie types, Soddemann solvent).
#pragma once
#include "fm_force.cuh"

namespace fm {

// FENE springs of molecule i (simulation_compute_forces_poly,
// simulation_compute_forces.f90:731-789): accijmag = -k/(1 - r^2/R0^2)
// (FENE_accijmag, setup_set_parameters.f90:348-358), energy
// 0.5 k R0^2 log(1 - r^2/R0^2) (:371-380), in FP64 for every precision form.
// A bond at or beyond R0 is the reference's polymer_bond_error.
template <bool REC, bool MIE>
__device__ __forceinline__ void fene_bonds(const FmDev &d, const double4 *P, int i, double &fx, double &fy,
                                           double &fz, double &pe, double &vir, double (&rf)[6])
{
    const double4 pi = P[i];
    const int nb = d.nbond[i];
    for (int b = 0; b < nb; b++) {
        const int e = d.bnd[(size_t)i * 4 + b];
        const int code = e >> NB_SHIFT_BITS;
        const double4 pj = P[e & NB_INDEX_MASK];
        const double xj = (code & 3) != 1 ? __dadd_rn(pj.x, (code & 3) == 2 ? d.L[0] : -d.L[0]) : pj.x;
        const double yj = ((code >> 2) & 3) != 1 ? __dadd_rn(pj.y, ((code >> 2) & 3) == 2 ? d.L[1] : -d.L[1]) : pj.y;
        const double zj = ((code >> 4) & 3) != 1 ? __dadd_rn(pj.z, ((code >> 4) & 3) == 2 ? d.L[2] : -d.L[2]) : pj.z;
        const double dx = __dsub_rn(pi.x, xj), dy = __dsub_rn(pi.y, yj), dz = __dsub_rn(pi.z, zj);
        const double r2 = norm2_rn(dx, dy, dz);
        if (MIE) {
            // harmonic_accijmag / harmonic_energy (setup_set_parameters.f90:384-437):
            // -k (|r| - r0)/|r| and k/2 (|r| - r0)^2, constants by type pair
            const FmMiePair &m = d.mie_pair[(mie_type(pi.w) - 1) + MIE_MAXT * (mie_type(pj.w) - 1)];
            const double rm = sqrt(r2), dr = rm - m.r0;
            const double acc = -m.k * dr / rm;
            fx += acc * dx; fy += acc * dy; fz += acc * dz;
            if (REC) {
                pe += 0.5 * m.k * (dr * dr);
                vir += acc * r2;
                if (d.pressure) add_rf(rf, acc, dx, dy, dz);  // :768-770
            }
            continue;
        }
        if (r2 >= d.R0_2) {
            uint32_t old = atomicOr(&d.sc->status, ST_BOND);
            if ((old & ST_FATAL) == 0u) d.sc->fail_iter = -2;
            continue;
        }
        const double q = r2 / d.R0_2;
        const double acc = -d.k_c / (1.0 - q);
        fx += acc * dx; fy += acc * dy; fz += acc * dz;
        if (REC) {
            pe += 0.5 * d.k_c * d.R0 * d.R0 * log(1.0 - q);
            vir += acc * r2;
            if (d.pressure) add_rf(rf, acc, dx, dy, dz);  // :768-770
        }
    }
}

// ---------------------------------------------------------------------------
// angular_potential (simulation_compute_forces_angular,
// simulation_compute_forces.f90:981-1048; angular_harmonic_force,
// setup_set_parameters.f90:441-489)
// ---------------------------------------------------------------------------

// The reference's triple of middle bead j: i = its first bond, k = its second
// (in discovery order), rij = r_i - r_j, rjk = r_j - r_k with the partners'
// periodic images (x_src +/- L, one rounding), theta = acos(rij.rjk /
// (|rij| |rjk|)) and
//   aForce(1) = -(k (theta - theta_0) / (|rij| sin theta)) (rjk/|rjk| - rij/|rij| cos theta)
//   aForce(3) = -(k (theta - theta_0) / (|rjk| sin theta)) (rij/|rij| - rjk/|rjk| cos theta)
//   aForce(2) = -aForce(1) - aForce(3)   (all zero when theta < 1e-5);
// the reference then subtracts aForce(1), (2), (3) from the forces on i, j,
// k.  Every molecule evaluates the triples it belongs to in the middle
// bead's frame, so the three see the same numbers.  k_ijk < 1e-5 leaves the
// reference's result unset: ST_ANGLE.
__device__ __forceinline__ bool angular_triple(const FmDev &d, const double4 *P, int j, double (&f1)[3],
                                               double (&f3)[3])
{
    const int e0 = d.bnd[(size_t)j * 4], e1 = d.bnd[(size_t)j * 4 + 1];
    const double4 pj = P[j], pi = P[e0 & NB_INDEX_MASK], pk = P[e1 & NB_INDEX_MASK];
    const int c0 = e0 >> NB_SHIFT_BITS, c1 = e1 >> NB_SHIFT_BITS;
    const double ri[3] = {image(pi.x, (c0 & 3) - 1, d.L[0]), image(pi.y, ((c0 >> 2) & 3) - 1, d.L[1]),
                          image(pi.z, ((c0 >> 4) & 3) - 1, d.L[2])};
    const double rk[3] = {image(pk.x, (c1 & 3) - 1, d.L[0]), image(pk.y, ((c1 >> 2) & 3) - 1, d.L[1]),
                          image(pk.z, ((c1 >> 4) & 3) - 1, d.L[2])};
    const double rj[3] = {pj.x, pj.y, pj.z};
    const int nt = d.ang_nt;
    const int q = (mie_type(pi.w) - 1) + nt * ((mie_type(pj.w) - 1) + nt * (mie_type(pk.w) - 1));
    const double kk = d.ang_k[q], t0 = d.ang_t0[q];
    f1[0] = f1[1] = f1[2] = 0.0;
    f3[0] = f3[1] = f3[2] = 0.0;
    if (kk < 1e-5) return false;
    double rij[3], rjk[3];
#pragma unroll
    for (int c = 0; c < 3; c++) { rij[c] = __dsub_rn(ri[c], rj[c]); rjk[c] = __dsub_rn(rj[c], rk[c]); }
    const double mij = sqrt(norm2_rn(rij[0], rij[1], rij[2]));
    const double mjk = sqrt(norm2_rn(rjk[0], rjk[1], rjk[2]));
    const double dot = __dadd_rn(__dadd_rn(__dmul_rn(rij[0], rjk[0]), __dmul_rn(rij[1], rjk[1])),
                                 __dmul_rn(rij[2], rjk[2]));
    const double th = acos(dot / (mij * mjk));
    if (th < 1e-5) return true;
    const double ct = cos(th), stt = sin(th);
    const double a1 = kk * (th - t0) / (mij * stt), a3 = kk * (th - t0) / (mjk * stt);
#pragma unroll
    for (int c = 0; c < 3; c++) {
        f1[c] = -a1 * (rjk[c] / mjk - rij[c] / mij * ct);
        f3[c] = -a3 * (rij[c] / mij - rjk[c] / mjk * ct);
    }
    return true;
}

// The angular forces on molecule m (added to its force sum before the
// division by its mass): -aForce(2) of its own triple when it is a middle
// bead, and -aForce(1) or -aForce(3) of each bonded middle bead's triple in
// which it is the bead i or k.
__device__ __forceinline__ void angular_forces(const FmDev &d, const double4 *P, int m, double &fx, double &fy,
                                               double &fz)
{
    double f1[3], f3[3];
    bool ok = true;
    if (d.funcy[m] == 2) {
        ok &= angular_triple(d, P, m, f1, f3);
        fx += f1[0] + f3[0]; fy += f1[1] + f3[1]; fz += f1[2] + f3[2];  // -aForce(2)
    }
    const int nb = d.nbond[m];
    for (int b = 0; b < nb; b++) {
        const int e = d.bnd[(size_t)m * 4 + b];
        const int p = e & NB_INDEX_MASK;
        if (d.funcy[p] != 2) continue;
        const int c = e >> NB_SHIFT_BITS;  // m as p sees it: the opposite image
        const int back = m | (((2 - (c & 3)) | ((2 - ((c >> 2) & 3)) << 2) | ((2 - ((c >> 4) & 3)) << 4))
                              << NB_SHIFT_BITS);
        ok &= angular_triple(d, P, p, f1, f3);
        if (d.bnd[(size_t)p * 4] == back) { fx -= f1[0]; fy -= f1[1]; fz -= f1[2]; }
        else if (d.bnd[(size_t)p * 4 + 1] == back) { fx -= f3[0]; fy -= f3[1]; fz -= f3[2]; }
        else ok = false;
    }
    if (!ok) {
        uint32_t old = atomicOr(&d.sc->status, ST_ANGLE);
        if ((old & ST_FATAL) == 0u) d.sc->fail_iter = -3;
    }
}

// Pair sum of molecule i over its list row: a lane of the molecule's TPM
// takes 4 entries per step (row_entries) and issues their 4 gathers before any
// arithmetic.  The gathers are unconditional (past the row's end the molecule
// reads itself): under a condition the compiler splits the 256-bit loads into
// three, 102M L1 wavefronts instead of 63M and 0.40 ms instead of 0.27 at 1M.  Entries without an image
// shift (all but the rows of boundary cells) skip the shift decoding.
template <int TPM, bool REC, int PREC>
__device__ __forceinline__ void list_pairs(const FmDev &d, const double4 *__restrict__ P, int i, int lane,
                                           const double4 &pi, double &fx, double &fy, double &fz, double &pe,
                                           double &vir, double (&rf)[6])
{
    const int cnt = d.nnbr[i];
    const int32_t *__restrict__ L = d.nbr + nb_row(i, d.maxn);
    const double Lx = d.L[0], Ly = d.L[1], Lz = d.L[2];
    const double rc2 = d.rc2;
    for (int s = 0; row_first<TPM>(s) < cnt; s++) {
        const int left = row_left<TPM>(s, lane, cnt);
        const int4 e4 = row_entries<TPM>(L, s, lane, left);
        // past the row's end the molecule itself, which the cutoff test leaves out
        const int self = i | (NB_NOSHIFT << NB_SHIFT_BITS);
        const int ev[4] = {left > row_off<TPM>(0) ? e4.x : self, left > row_off<TPM>(1) ? e4.y : self,
                           left > row_off<TPM>(2) ? e4.z : self, left > row_off<TPM>(3) ? e4.w : self};
        double4 pj[4];
#pragma unroll
        for (int q = 0; q < 4; q++) pj[q] = ldg_pos(P + (ev[q] & NB_INDEX_MASK));
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int code = ev[q] >> NB_SHIFT_BITS;
            double xj = pj[q].x, yj = pj[q].y, zj = pj[q].z;
            if (code != NB_NOSHIFT) {
                const int ssx = (code & 3) - 1, ssy = ((code >> 2) & 3) - 1, ssz = ((code >> 4) & 3) - 1;
                xj = ssx ? __dadd_rn(xj, ssx > 0 ? Lx : -Lx) : xj;
                yj = ssy ? __dadd_rn(yj, ssy > 0 ? Ly : -Ly) : yj;
                zj = ssz ? __dadd_rn(zj, ssz > 0 ? Lz : -Lz) : zj;
            }
            const double dx = __dsub_rn(pi.x, xj);
            const double dy = __dsub_rn(pi.y, yj);
            const double dz = __dsub_rn(pi.z, zj);
            const double r2 = norm2_rn(dx, dy, dz);
            if (left > row_off<TPM>(q) && r2 < rc2) {
                const double acc = pair_acc<PREC, REC>(d, r2, dx, dy, dz, pi.w, pj[q].w, fx, fy, fz, pe, vir);
                // every partner of i in the full list: the half list's i and j sides
                if (REC && d.pressure) add_rf(rf, acc, dx, dy, dz);
            }
        }
    }
}

// Bonded terms and the integrator epilogue of molecule i once its pair sum is
// complete; returns |v|^2 after a position update (epilogue()).
template <bool REC, int MODE, int PREC>
__device__ __forceinline__ double owner_finish(const FmDev &d, int pset, const double4 *__restrict__ P, int i,
                                               double fx, double fy, double fz, double pe, double vir,
                                               double (&part)[RS_N], double (&rf)[6])
{
    if constexpr ((PREC & 6) == 6) {
        // Mie + Soddemann: the Soddemann pairs are not divided by a mass
        // (:852-860), the bonds of simulation_compute_forces_poly are
        // (:752-754)
        const double4 pi = P[i];
        double bx = 0.0, by = 0.0, bz = 0.0;
        if (d.potential_flag == 1) fene_bonds<REC, true>(d, P, i, bx, by, bz, pe, vir, rf);
        const double mass = d.mie_mass[mie_type(pi.w) - 1];
        fx += bx / mass; fy += by / mass; fz += bz / mass;
        return epilogue<REC, MODE, true, false>(d, pset, i, pi, fx, fy, fz, pe, vir, part, rf);
    } else {
        if (d.potential_flag == 1) fene_bonds<REC, (PREC & 2) != 0>(d, P, i, fx, fy, fz, pe, vir, rf);
        if constexpr ((PREC & 2) != 0) {  // angular_potential needs the Mie types
            if (d.angular) angular_forces(d, P, i, fx, fy, fz);
        }
        // a(:,i) = sum acc rij / mass (LJ_mass = 1; Mie_mass by type)
        return epilogue<REC, MODE, (PREC & 2) != 0>(d, pset, i, P[i], fx, fy, fz, pe, vir, part, rf);
    }
}

// Four resident blocks hide the gathers' latency (three, at 66 registers,
// take 0.31 ms instead of 0.27 at 1M), on record steps too, although their sums
// spill a little: 0.48 -> 0.40 ms at 1M in FP64, 77 -> 63 us at 108,000 with the
// pressure tensor, against two blocks.  Lanes on
// neighbouring entries against lanes on four entries each: 338 -> 308 us with
// four lanes at 1M, 42.4 -> 36.7 at 108,000, 19.6 -> 17.7 at 32,000.
template <int TPM, bool REC, int MODE, int PREC>
__global__ void __launch_bounds__(FORCE_THREADS, (PREC & 6) != 0 ? 2 : 4) k_force(FmDev d)
{
    pdl_enter();
    if (frozen(d)) return;
    const int pset = d.sc->pset;
    const double4 *__restrict__ P = cur_pos(d, pset);
    const int gt = blockIdx.x * FORCE_THREADS + threadIdx.x;
    const int i = gt / TPM;
    const int lane = gt % TPM;
    const bool active = i < d.n;
    double fx = 0.0, fy = 0.0, fz = 0.0, pe = 0.0, vir = 0.0;
    double rf[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    if (active) list_pairs<TPM, REC, PREC>(d, P, i, lane, P[i], fx, fy, fz, pe, vir, rf);
    if (TPM > 1) {
#pragma unroll
        for (int o = TPM / 2; o > 0; o >>= 1) {
            fx += __shfl_xor_sync(0xffffffffu, fx, o);
            fy += __shfl_xor_sync(0xffffffffu, fy, o);
            fz += __shfl_xor_sync(0xffffffffu, fz, o);
            if (REC) {
                pe += __shfl_xor_sync(0xffffffffu, pe, o);
                vir += __shfl_xor_sync(0xffffffffu, vir, o);
                if (d.pressure) {
#pragma unroll
                    for (int k = 0; k < 6; k++) rf[k] += __shfl_xor_sync(0xffffffffu, rf[k], o);
                }
            }
        }
    }
    double part[RS_N] = {};
    double m2 = 0.0;
    if (active && lane == 0) m2 = owner_finish<REC, MODE, PREC>(d, pset, P, i, fx, fy, fz, pe, vir, part, rf);
    if (REC) block_partials(d, part, blockIdx.x);
    if (MODE >= 2) block_vmax2(d, m2);
}

}  // namespace fm
