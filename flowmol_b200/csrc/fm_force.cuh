// fm_force.cuh -- what the kernels of one system share (fm_kernels.cu,
// fm_rows.cu): the status word, the pair expressions, the integrator epilogue,
// the record partials and the |v|^2 maximum.
#pragma once
#include "fm_common.cuh"
#include "fm_device.cuh"

namespace fm {

constexpr int FORCE_THREADS = 256;

__device__ __forceinline__ bool frozen(const FmDev &d) { return (d.sc->status & ST_FATAL) != 0u; }

// Whether a rebuild kernel runs: `gated` kernels only on the steps that rebuild.
__device__ __forceinline__ bool gate(const FmDev &d, int gated)
{
    if (frozen(d)) return false;
    if (gated && !d.sc->rebuild) return false;
    return true;
}

// w of a position: the Mie type (1-based), the Soddemann bead flag (1 for a
// chain bead), or with both the type plus 32 times the flag.
__device__ __forceinline__ int mie_type(double w) { return ((int)w) & 31; }
template <bool MIE>
__device__ __forceinline__ int bead_flag(double w) { return MIE ? ((int)w) >> 5 : (int)w; }

__device__ __forceinline__ void raise_status(const FmDev &d, uint32_t bit, int iter)
{
    if (iter == ITER_DEVICE) iter = d.sc->cur_iter;
    uint32_t old = atomicOr(&d.sc->status, bit);
    if ((old & ST_FATAL) == 0u) d.sc->fail_iter = iter;
}

// Block max of a non-negative double folded into sc->vmax2 (u64 order of
// non-negative doubles equals their numeric order).
__device__ __forceinline__ void block_vmax2(const FmDev &d, double m2)
{
    __shared__ double wmax[32];
    m2 = warp_max(m2);
    int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) wmax[w] = m2;
    __syncthreads();
    if (w == 0) {
        int nw = (blockDim.x + 31) >> 5;
        double v = l < nw ? wmax[l] : 0.0;
        v = warp_max(v);
        if (l == 0 && v > 0.0) atomicMax(&d.sc->vmax2, (unsigned long long)__double_as_longlong(v));
    }
}

// One pair inside the cutoff: acc (the pair force over rij) accumulated as
// acc * rij, and on record steps the energy and acc * r^2.  PREC bit 0: FP32
// pair magnitude (FP64 rij scales it); bit 1: Mie_potential 1, constants by
// the molecules' types (w of the positions): Mie_accijmag and Mie_energy
// (setup_set_parameters.f90:149-204) with real powers, as s**(lr/2+1).
// Otherwise LJ_accijmag = 48 (s^7 - s^4/2), s = 1/r^2, and LJ_energy
// (:105-135).
template <int PREC, bool REC>
__device__ __forceinline__ double pair_acc(const FmDev &d, double r2, double dx, double dy, double dz, double wi,
                                           double wj, double &fx, double &fy, double &fz, double &pe, double &vir)
{
    constexpr bool F32 = (PREC & 1) != 0, MIE = (PREC & 2) != 0, SOD = (PREC & 4) != 0;
    if (SOD) {
        // simulation_compute_forces_Soddemann_neigbr_halfint (:793-888): WCA
        // inside wca_cut2, the cosine well eps a s^2 sin(a s + b) beyond it
        // (the reference's expression, s = 1/r^2); no potshift.  The WCA force
        // is get_accijmag: Mie_accijmag of the pair's types with
        // Mie_potential 1, its energy the LJ-WCA expression either way.
        const double eps = d.sod_eps[bead_flag<MIE>(wi) + bead_flag<MIE>(wj)];
        const bool wca = r2 < SOD_WCA_CUT2;
        if (!F32) {
            const double s = __drcp_rn(r2);
            const double s2 = s * s;
            double acc;
            if (wca && MIE) {
                const FmMiePair &m = d.mie_pair[(mie_type(wi) - 1) + MIE_MAXT * (mie_type(wj) - 1)];
                acc = m.ceps * (m.lr * pow(s, m.er1) - m.ala * pow(s, m.ea1));
            } else if (wca) {
                const double s4 = s2 * s2;
                acc = 48.0 * (s4 * s2 * s - 0.5 * s4);  // get_accijmag = LJ_accijmag
            } else {
                acc = (eps * SOD_A * s2) * sin(s * SOD_A + SOD_B);
            }
            fx += acc * dx; fy += acc * dy; fz += acc * dz;
            if (REC) {
                if (wca) {
                    const double s3 = s2 * s, s6 = s3 * s3;
                    pe += 4.0 * (s6 - s3 + 0.25) - eps;
                } else {
                    pe += 0.5 * eps * (cos(SOD_A * r2 + SOD_B) - 1.0);
                }
                vir += acc * r2;
            }
        } else {
            const float s = rcp_f32((float)r2);
            const float s2 = s * s;
            float accf;
            if (wca && MIE) {
                const FmMiePair &m = d.mie_pair[(mie_type(wi) - 1) + MIE_MAXT * (mie_type(wj) - 1)];
                accf = (float)m.ceps * ((float)m.lr * powf(s, (float)m.er1) - (float)m.ala * powf(s, (float)m.ea1));
            } else if (wca) {
                const float s4 = s2 * s2;
                accf = 48.0f * (s4 * s2 * s - 0.5f * s4);
            } else {
                accf = ((float)eps * (float)SOD_A * s2) * sinf(s * (float)SOD_A + (float)SOD_B);
            }
            const double acc = (double)accf;
            fx = fma(acc, dx, fx); fy = fma(acc, dy, fy); fz = fma(acc, dz, fz);
            if (REC) {
                if (wca) {
                    const float s3 = s2 * s, s6 = s3 * s3;
                    pe += (double)(4.0f * (s6 - s3 + 0.25f)) - eps;
                } else {
                    pe += (double)(0.5f * (float)eps * (cosf((float)SOD_A * (float)r2 + (float)SOD_B) - 1.0f));
                }
                vir += acc * r2;
            }
        }
        return 0.0;  // the Soddemann routine records no pressure-tensor term
    }
    if (MIE) {
        const FmMiePair &m = d.mie_pair[(mie_type(wi) - 1) + MIE_MAXT * (mie_type(wj) - 1)];
        if (!F32) {
            const double s = __drcp_rn(r2);  // == 1.0 / r2
            const double acc = m.ceps * (m.lr * pow(s, m.er1) - m.ala * pow(s, m.ea1));
            fx += acc * dx; fy += acc * dy; fz += acc * dz;
            if (REC) {
                pe += m.ceps * (pow(s, m.er) - m.alpha * pow(s, m.ea)) - m.shift;
                vir += acc * r2;
            }
            return acc;
        } else {
            const float s = rcp_f32((float)r2);
            const double acc = (double)((float)m.ceps * ((float)m.lr * powf(s, (float)m.er1) -
                                                         (float)m.ala * powf(s, (float)m.ea1)));
            fx = fma(acc, dx, fx); fy = fma(acc, dy, fy); fz = fma(acc, dz, fz);
            if (REC) {
                pe += (double)((float)m.ceps * (powf(s, (float)m.er) - (float)m.alpha * powf(s, (float)m.ea))) - m.shift;
                vir += acc * r2;
            }
            return acc;
        }
    } else if (!F32) {
        const double s = __drcp_rn(r2);  // == 1.0 / r2 (both correctly rounded)
        const double s2 = s * s, s4 = s2 * s2;
        const double acc = 48.0 * (s4 * s2 * s - 0.5 * s4);
        fx += acc * dx; fy += acc * dy; fz += acc * dz;
        if (REC) {
            const double s3 = s2 * s, s6 = s3 * s3;
            pe += 4.0 * (s6 - s3) - d.potshift;  // LJ_energy (:126-135)
            vir += acc * r2;
        }
        return acc;
    } else {
        // FP32 pair magnitude; the FP64 rij scales it (one conversion)
        const float s = rcp_f32((float)r2);
        const float s2 = s * s, s4 = s2 * s2;
        const double acc = (double)(48.0f * (s4 * s2 * s - 0.5f * s4));
        fx = fma(acc, dx, fx); fy = fma(acc, dy, fy); fz = fma(acc, dz, fz);
        if (REC) {
            const float s3 = s2 * s, s6 = s3 * s3;
            pe += (double)(4.0f * (s6 - s3)) - d.potshift;
            vir += acc * r2;
        }
        return acc;
    }
}

// pressure_tensor_forces (simulation_record.f90:6239-6256): rf += acc rij rij,
// the six distinct components xx yy zz xy xz yz.
__device__ __forceinline__ void add_rf(double (&rf)[6], double acc, double dx, double dy, double dz)
{
    const double ax = acc * dx, ay = acc * dy, az = acc * dz;
    rf[0] += ax * dx; rf[1] += ay * dy; rf[2] += az * dz;
    rf[3] += ax * dy; rf[4] += ax * dz; rf[5] += ay * dz;
}

// Record-step pressure terms of one molecule: v v + rf/2 (cumulative_pressure
// case 1, simulation_record.f90:3170-3199; no mass factor there).
__device__ __forceinline__ void pressure_part(double (&part)[RS_N], double wx, double wy, double wz,
                                              const double (&rf)[6])
{
    part[RS_PXX] = wx * wx + rf[0] / 2.0; part[RS_PYY] = wy * wy + rf[1] / 2.0;
    part[RS_PZZ] = wz * wz + rf[2] / 2.0; part[RS_PXY] = wx * wy + rf[3] / 2.0;
    part[RS_PXZ] = wx * wz + rf[4] / 2.0; part[RS_PYZ] = wy * wz + rf[5] / 2.0;
}

// Integrator epilogue of molecule i with its summed LJ force: stores a (and PE
// and virial on record steps) and, by MODE,
//   1  move(2)                               (simulation_move_particles_vv.f90:132-135)
//   2  move(2) + move(1) of the next step    (:64-69), new positions into pset^1
//   3  leap-frog v += dt a, r += dt v        (simulation_move_particles_lfv.f90:81-92)
// The record partials use v after move(2) for velocity Verlet and v + a dt/2
// for leap-frog (simulation_record.f90:1236-1252).  Returns |v|^2 after a
// position update (modes 2, 3), else 0.
// DIV false: the forces are accelerations already (the Soddemann pairs and
// the mass-divided bonds of a Mie + Soddemann system); the kinetic terms are
// still mass-weighted.
template <bool REC, int MODE, bool MIE = false, bool DIV = true>
__device__ __forceinline__ double epilogue(const FmDev &d, int pset, int i, double4 p, double fx, double fy,
                                           double fz, double pe, double vir, double (&part)[RS_N],
                                           const double (&rf)[6])
{
    if (REC && d.pressure) {  // kept for a record taken after the move (fm_evaluate_macroscopic_properties)
        double *q = d.rf6 + 6 * (size_t)i;
#pragma unroll
        for (int k = 0; k < 6; k++) q[k] = rf[k];
    }
    double mass = 1.0;  // LJ_mass; Mie_mass = mass_lookup(moltype)
    if (MIE) {
        mass = d.mie_mass[mie_type(p.w) - 1];
        if (DIV) { fx = fx / mass; fy = fy / mass; fz = fz / mass; }
    }
    d.ax[i] = fx; d.ay[i] = fy; d.az[i] = fz;
    if (REC) { d.pe[i] = pe; d.vir[i] = vir; }
    double vx = d.vx[i], vy = d.vy[i], vz = d.vz[i];
    double m2 = 0.0;
    if (MODE == 3) {
        if (REC) {
            const double wx = __dadd_rn(vx, __dmul_rn(__dmul_rn(0.5, fx), d.dt));
            const double wy = __dadd_rn(vy, __dmul_rn(__dmul_rn(0.5, fy), d.dt));
            const double wz = __dadd_rn(vz, __dmul_rn(__dmul_rn(0.5, fz), d.dt));
            part[RS_PE] = pe; part[RS_VIR] = vir; part[RS_PEMAX] = pe;
            part[RS_MV2] = MIE ? mass * norm2_rn(wx, wy, wz) : norm2_rn(wx, wy, wz);
            part[RS_VSUM] = MIE ? mass * __dadd_rn(__dadd_rn(wx, wy), wz) : __dadd_rn(__dadd_rn(wx, wy), wz);
            if (d.pressure) pressure_part(part, wx, wy, wz, rf);
        }
        vx = __dadd_rn(vx, __dmul_rn(d.dt, fx));
        vy = __dadd_rn(vy, __dmul_rn(d.dt, fy));
        vz = __dadd_rn(vz, __dmul_rn(d.dt, fz));
        p.x = __dadd_rn(p.x, __dmul_rn(d.dt, vx));
        p.y = __dadd_rn(p.y, __dmul_rn(d.dt, vy));
        p.z = __dadd_rn(p.z, __dmul_rn(d.dt, vz));
        cur_pos(d, pset ^ 1)[i] = p;
        d.vx[i] = vx; d.vy[i] = vy; d.vz[i] = vz;
        return norm2_rn(vx, vy, vz);
    }
    if (MODE >= 1) {
        vx = __dadd_rn(vx, __dmul_rn(d.half_dt, fx));
        vy = __dadd_rn(vy, __dmul_rn(d.half_dt, fy));
        vz = __dadd_rn(vz, __dmul_rn(d.half_dt, fz));
    }
    if (REC) {
        double wx = vx, wy = vy, wz = vz;
        if (MODE == 0 && d.integrator == 0) {  // forces only, leap-frog record velocity
            wx = __dadd_rn(vx, __dmul_rn(__dmul_rn(0.5, fx), d.dt));
            wy = __dadd_rn(vy, __dmul_rn(__dmul_rn(0.5, fy), d.dt));
            wz = __dadd_rn(vz, __dmul_rn(__dmul_rn(0.5, fz), d.dt));
        }
        part[RS_PE] = pe; part[RS_VIR] = vir; part[RS_PEMAX] = pe;
        part[RS_MV2] = MIE ? mass * norm2_rn(wx, wy, wz) : norm2_rn(wx, wy, wz);
        part[RS_VSUM] = MIE ? mass * __dadd_rn(__dadd_rn(wx, wy), wz) : __dadd_rn(__dadd_rn(wx, wy), wz);
        if (d.pressure) pressure_part(part, wx, wy, wz, rf);
    }
    if (MODE == 2) {
        p.x = __dadd_rn(__dadd_rn(p.x, __dmul_rn(d.dt, vx)), __dmul_rn(d.half_dt2, fx));
        p.y = __dadd_rn(__dadd_rn(p.y, __dmul_rn(d.dt, vy)), __dmul_rn(d.half_dt2, fy));
        p.z = __dadd_rn(__dadd_rn(p.z, __dmul_rn(d.dt, vz)), __dmul_rn(d.half_dt2, fz));
        vx = __dadd_rn(vx, __dmul_rn(d.half_dt, fx));
        vy = __dadd_rn(vy, __dmul_rn(d.half_dt, fy));
        vz = __dadd_rn(vz, __dmul_rn(d.half_dt, fz));
        cur_pos(d, pset ^ 1)[i] = p;
        m2 = norm2_rn(vx, vy, vz);
    }
    if (MODE >= 1) { d.vx[i] = vx; d.vy[i] = vy; d.vz[i] = vz; }
    return m2;
}

// (s, c) += (s2, c2): Neumaier merge of two compensated partial sums.
__device__ __forceinline__ void nmerge(double &s, double &c, double s2, double c2)
{
    neumaier(s, c, s2);
    c += c2;
}

// Block reduction of the record partials into row `row` of d.partial:
// Neumaier-compensated sums in a fixed tree order (warp xor tree, then the
// warps in index order), the row holding the compensated value rounded once;
// PE max for the PE check.
template <int NT = FORCE_THREADS>
__device__ __forceinline__ void block_partials(const FmDev &d, double v[RS_N], int row)
{
    __shared__ double ws[RS_N][NT / 32], wc[RS_N][NT / 32];
    int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    const int nq = d.pressure ? (int)RS_N : (int)RS_PXX;  // the pressure terms only where they are summed
#pragma unroll
    for (int k = 0; k < RS_N; k++) {
        if (k >= nq) break;
        double x = v[k], c = 0.0;
        if (k == RS_PEMAX) {
            x = warp_max(x);
        } else {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const double x2 = __shfl_xor_sync(0xffffffffu, x, o), c2 = __shfl_xor_sync(0xffffffffu, c, o);
                nmerge(x, c, x2, c2);
            }
        }
        if (l == 0) { ws[k][w] = x; wc[k][w] = c; }
    }
    __syncthreads();
    if (threadIdx.x < nq) {
        int k = threadIdx.x;
        double acc = ws[k][0], cmp = wc[k][0];
        for (int q = 1; q < NT / 32; q++) {
            if (k == RS_PEMAX) acc = fmax(acc, ws[k][q]);
            else nmerge(acc, cmp, ws[k][q], wc[k][q]);
        }
        d.partial[(size_t)row * RS_N + k] = k == RS_PEMAX ? acc : acc + cmp;
    }
}

}  // namespace fm
