// FP64 CUDA kernels of one Eucclhyd Lagrange + remap cycle on GB300.
//
// Cycle structure (reference: Eucclhyd::executeTimeLoopN,
// eucclhyd_remap/EucclhydRemap.cc:84-195):
//   ke_begin     cycle start, reset of the dt reduction
//   ke_cell_pre  computeEOS, computePressionMoyenne, computeGradients,
//                computeMass, computem_cell_deltat (+ block min of dt)
//   ke_nodes     extrapolateValue, computeG, computeNodeDissipationMatrixAndG,
//                computeBoundaryNodeVelocities, computeNodeVelocity, the
//                Lagrange node positions
//   ke_cells     computeLagrangeVolumeAndCenterOfGravity, computeSubCellForce
//                (recomputed per cell from the corner extrapolations),
//                updateCellCenteredLagrangeVariables, the Lagrangian face
//                lengths of the remap
//   sweep x2     the shared directional remap (vnr.cu launch_sweep)
//   ke_final     remapCellcenteredVariable (PhaseRemapFinal.cc:17-232)
//   ke_end       computedeltat, updateTime, loop condition and time swap
//
// Corner quantities live per (cell, corner k); the reference keeps them per
// (node, slot of the cell).  The sub-cell forces are not stored: the cell
// kernel recomputes them from the corner extrapolations and the new node
// velocities, and keeps only their per-material sums for the next cycle's
// pressure gradients (computeGradients, PhaseLagrange.cc:225-244).  All
// arithmetic keeps the reference's operation order (--fmad=false).
#include <cuda_runtime.h>

#include "../internal.h"
#include "items.cuh"
#include "scheme_math.cuh"

namespace hydro {

int launch_sweep(const RunView& v, int sweep, cudaStream_t s, const LaunchHook* hook,
                 const std::function<void(int)>& before);

namespace {

constexpr int kBX = 32, kBY = 4;

#define DV __device__ __forceinline__

DV double ldg(const double* p, long long i) { return __ldg(p + i); }
DV double gam(const RunView& v, int m) {
  return m == 0 ? v.gamma[0] : (m == 1 ? v.gamma[1] : v.gamma[2]);
}
DV double gm1m(const RunView& v, int m) {
  return m == 0 ? v.gm1[0] : (m == 1 ? v.gm1[1] : v.gm1[2]);
}
// store of a value read from the same address: left out when the bits are
// the ones already there
DV void st_new(double* a, double old_v, double new_v) {
  if (ubits(new_v) != ubits(old_v)) *a = new_v;
}
DV int eosm(const RunView& v, int m) {
  return m == 0 ? v.eos[0] : (m == 1 ? v.eos[1] : v.eos[2]);
}
// dot product accumulated from 0.0 (includes/Freefunctions.h:15-20); the
// first addition 0.0 + a0 b0 is plus_zero (integer pipe)
DV double dot2(double a0, double a1, double b0, double b1) {
  double r = plus_zero(a0 * b0);
  r += a1 * b1;
  return r;
}
// dot2 is exactly +0 when one vector is two zeros and the other finite
// (plus_zero of a signed zero, plus a signed zero)
DV bool dot2_zero(double a0, double a1, double b0, double b1) {
  return (iszero(a0) && iszero(a1) && is_finite(b0) && is_finite(b1)) ||
         (iszero(b0) && iszero(b1) && is_finite(a0) && is_finite(a1));
}
// x + dot2(a, b), with x + (+0) = plus_zero(x) where the product is +0
DV double add_dot2(double x, double a0, double a1, double b0, double b1) {
  return dot2_zero(a0, a1, b0, b1) ? plus_zero(x) : x + dot2(a0, a1, b0, b1);
}

// block-wide min of ordered encodings, one atomic per block
DV void block_min(unsigned long long dtv, Ctrl* C) {
  __shared__ unsigned long long smin_s[32];
  const int tid = threadIdx.y * blockDim.x + threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const int nw = (blockDim.x * blockDim.y + 31) >> 5;
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long a = __shfl_xor_sync(0xffffffffu, dtv, o);
    dtv = a < dtv ? a : dtv;
  }
  if (lane == 0) smin_s[warp] = dtv;
  __syncthreads();
  if (warp == 0) {
    dtv = lane < nw ? smin_s[lane] : ~0ull;
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long a = __shfl_xor_sync(0xffffffffu, dtv, o);
      dtv = a < dtv ? a : dtv;
    }
    if (lane == 0 && dtv != ~0ull) atomicMin(&C->dt_min_bits, dtv);
  }
  __syncthreads();
}

// ------------------------------------------------------------- control
DV void euc_begin_at(const RunView& v) {
  Ctrl& C = *v.ctrl;
  if (C.done || (C.err & ~HYDRO_ERR_NEGATIVE)) {
    C.active = 0;
    C.done = 1;
    return;
  }
  if (output_pause_here(C)) {
    C.active = 0;
    return;
  }
  C.active = 1;
  C.n += 1;
  C.dt_min_bits = ord_bits(1.7976931348623157e308);
}
__global__ void ke_begin(RunView v) { euc_begin_at(v); }

// computedeltat (EucclhydRemap.cc:203-221): the cycle's cell dt minimum
// gives dt_{n+1}; updateTime; the loop condition and the swap of t, dt.
// The Lagrange positions and the remap of this cycle used dt_n.
DV void euc_end_at(const RunView& v) {
  Ctrl& C = *v.ctrl;
  if (!C.active) return;
  const double red = from_ord(C.dt_min_bits);
  C.dt_np1 = smin(v.euc_cfl * red, C.dt_n * 1.05);
  if (dlt(C.dt_np1, v.dt_min)) C.err |= HYDRO_ERR_DT_MIN;
  C.t_np1 = C.t_n + C.dt_np1;
  const bool cont = (C.n + 1 < v.max_iter) && dlt(C.t_np1, v.final_time);
  C.t_n = C.t_np1;
  C.dt_n = C.dt_np1;
  if (cont)
    C.x_then_y = !C.x_then_y;
  else
    C.done = 1;
  if (C.err & ~HYDRO_ERR_NEGATIVE) C.done = 1;
}
__global__ void ke_end(RunView v) { euc_end_at(v); }

// The pressure of material m of cell c by computeEOSGP / computeEOSVoid
// (PhaseLagrange.cc:70-109); the other EOS ids keep the stored value (their
// reference routines only print).  A perfect gas's zero density and finite
// factors give the product's signed zero.
DV double cell_pressure(const RunView& v, int m, double rm, double em, long long c) {
  const int eos = eosm(v, m);
  if (eos == HYDRO_EOS_PERFECT_GAS) return mulz(mulz(gm1m(v, m), rm), em);
  return (eos == HYDRO_EOS_VOID) ? 0. : v.pm[m * v.pitch + c];
}
// its sound speed (read only where the cell's density is not positive)
DV double material_sound(const RunView& v, int m, double rm, double pm, long long c) {
  const int eos = eosm(v, m);
  if (eos == HYDRO_EOS_PERFECT_GAS) return pos(rm) ? sqrt_ip(div_ip(gam(v, m) * pm, rm)) : 1.e-20;
  return (eos == HYDRO_EOS_VOID) ? 1.e-20 : v.cm[m * v.pitch + c];
}

// ------------------------------------------------- cell state of step n
// computeEOS + computeEOSGP / computeEOSVoid (PhaseLagrange.cc:70-109),
// computePressionMoyenne (:139-155), computeGradients (:160-246; the
// fracvol-gradient part only feeds the particle scheme), computeMass
// (:251-261), computem_cell_deltat (:302-316).
// The mean-pressure step replaces the sound speed by the mixture's wherever
// the density is positive, and nothing else reads a material's sound speed:
// those are formed (and the stored one read) only in the other cells.
template <int NB = 0>
struct EucCellPre {
  __device__ __forceinline__ void operator()(const RunView& v, int i, int j) const {
    unsigned long long dtb = ~0ull;
    if (i < v.ny && j < v.nx) {
      const long long P = v.pitch, NP = v.npitch;
      const long long c = (long long)i * v.nx + j;
      const int nb = NB ? NB : v.nbmat;
      // the inputs, ahead of the stores (which would order later loads
      // behind them)
      double rm[3], em[3], fm[3], mfm[3];
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        if (m >= nb) break;
        rm[m] = v.rhom[m * P + c];
        em[m] = v.em[m * P + c];
        fm[m] = v.fm[m * P + c];
        mfm[m] = v.mfm[m * P + c];
      }
      const double rho = v.rho[c], V = ldg(v.evol, c);
      const double u0 = v.uc[c], u1 = v.uc[P + c], per = ldg(v.perim, c);
      double p = 0., pm[3];
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        if (m >= nb) break;
        pm[m] = cell_pressure(v, m, rm[m], em[m], c);
        p = addz(p, mul_frac(fm[m], pm[m]));  // 0.0 + t first
      }
      double snd;
      if (pos(rho)) {
        snd = sqrt_ip(div_ip(v.gamma[0] * p, rho));
      } else {
        snd = v.c[c];
        for (int m = 0; m < nb; ++m) {
          const double r = v.rhom[m * P + c];
          snd = smax(snd, material_sound(v, m, r, cell_pressure(v, m, r, v.em[m * P + c], c), c));
        }
      }
      if (v.space_order == 2) {
        const long long n0 = (long long)i * (v.nx + 1) + j;
        const long long nd[4] = {n0, n0 + 1, n0 + v.nx + 2, n0 + v.nx + 1};
        double r14[4] = {0.0, 0.0, 0.0, 0.0};
        double cu[4][2], cl[4][2];
        bool still = true;  // every corner velocity a zero, every l finite
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          cu[k][0] = v.u[nd[k]];
          cu[k][1] = v.u[NP + nd[k]];
          cl[k][0] = ldg(v.lpc, (2 * k) * P + c);
          cl[k][1] = ldg(v.lpc, (2 * k + 1) * P + c);
          still = still && iszero(cu[k][0]) && iszero(cu[k][1]) && is_finite(cl[k][0]) &&
                  is_finite(cl[k][1]);
        }
        double fs[6];
#pragma unroll
        for (int q = 0; q < 6; ++q)
          if (q < 2 * nb) fs[q] = v.Fs[q * P + c];
        // then every product is a signed zero and each sum from 0.0 is +0
        if (!still) {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const double a0 = cu[k][0], a1 = cu[k][1], l0 = cl[k][0], l1 = cl[k][1];
            const double t[4] = {a0 * l0, a0 * l1, a1 * l0, a1 * l1};
#pragma unroll
            for (int q = 0; q < 4; ++q) r14[q] = (k == 0) ? plus_zero(t[q]) : r14[q] + t[q];
          }
        }
        // one denominator, 4 + 2 nbmat quotients
        const SharedDiv SV = shared_div(V);
#pragma unroll
        for (int q = 0; q < 4; ++q) v.vg[q * P + c] = qdiv_shared(SV, r14[q]);
        // per-material pressure gradients from last cycle's corner-force
        // sums, in place
#pragma unroll
        for (int q = 0; q < 6; ++q)
          if (q < 2 * nb) st_new(v.Fs + q * P + c, fs[q], qdiv_shared(SV, fs[q]));
      }
#pragma unroll
      for (int m = 0; m < 3; ++m)
        if (m < nb) v.pm[m * P + c] = pm[m];
      v.p[c] = p;
      v.c[c] = snd;
      const double cmass = rho * V;
      v.cell_mass[c] = cmass;
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        if (m >= nb) break;
        v.cmassm[m * P + c] = mul_frac(mfm[m], cmass);
      }
      const double un = face_len(u0, u1);  // sqrt(dot(u, u))
      const double cdt = (v.projection == 1) ? div_ip(V, per * addz(un, snd)) : div_ip(V, per * snd);
      if (!is_nan(cdt)) dtb = ord_bits(cdt);
    }
    block_min(dtb, v.ctrl);
  }
};

// Eucclhyd::nodeVelocityBoundaryCondition (ConditionsLimites.cc:109-123)
DV void bc_velocity(int bc, double V0, double V1, const double* Mp, const double* G,
                    double& o0, double& o1) {
  if (bc == kBcSym) {
    const double mv0 = dot2(Mp[0], Mp[1], V0, V1), mv1 = dot2(Mp[2], Mp[3], V0, V1);
    const double s = div_ip(dot2(G[0], G[1], V0, V1), dot2(mv0, mv1, V0, V1));
    o0 = V0 * s;
    o1 = V1 * s;
  } else if (bc == kBcImposed) {
    o0 = V0;
    o1 = V1;
  } else if (bc == 202) {  // free: inverse(Mp) . G
    const double alpha = div_ip(1.0, Mp[0] * Mp[3] - Mp[1] * Mp[2]);
    const double i0 = Mp[3] * alpha, i1 = -Mp[1] * alpha, i2 = -Mp[2] * alpha,
                 i3 = Mp[0] * alpha;
    o0 = dot2(i0, i1, G[0], G[1]);
    o1 = dot2(i2, i3, G[0], G[1]);
  } else {
    o0 = 0.0;
    o1 = 0.0;
  }
}

// ----------------------------------------------------------- node solve
// extrapolateValue (:322-479), computeG (:484-505),
// computeNodeDissipationMatrixAndG (:511-527), computeBoundaryNodeVelocities
// (ConditionsLimites.cc:19-107), computeNodeVelocity (:532-543),
// computeLagrangePosition nodes (:573-580).
//
// INNER: the node has four cells, in fixed corners (no indexed arrays, which
// would live in local memory).  Two shortcuts, each one branch for a block of
// work and exact:
//  - a material absent around the node (pressures and force sums of all its
//    cells zeros): its extrapolated pressures are +0 (the sum from p = +-0
//    and a +0 product, between a minimum +-0 and a maximum of at least the
//    smallest normal number), their shares of the cells' pressures zeros;
//  - corner matrices without off-diagonal entries (every Cartesian mesh; the
//    set-up's cmat_diag flag): m01 = +-0, so a dot product with it is the
//    other term made non-negative zero (x + (+-0) = x), its sums are +0, the
//    determinant is Mp00 Mp11 - (+0), the inverse is diagonal up to zeros.
// 1792 x 768 cells, 3 materials: 472 -> 322 us (five blocks per SM; four to
// ten within 10 %); with the boundary's nodes in warps of their own and the
// material count compiled in 296 us, and 70 x 30 cells 33 -> 22 us.
template <int NB = 0>
struct EucNodes {
  template <bool INNER>
  DV void node(const RunView& v, int i, int j) const {
    const Ctrl& C = *v.ctrl;
    const long long P = v.pitch, NP = v.npitch;
    const long long p = (long long)i * (v.nx + 1) + j;
    const int nb = NB ? NB : v.nbmat;
    // cells of the node in getCellsOfNode order (CartesianMesh2D.cc:97-108)
    // and the node's position in each
    long long cells[4];
    int loc[4], kc = 0;
    const long long c00 = (long long)i * v.nx + j;
    if (INNER) {
      kc = 4;
      cells[0] = c00; loc[0] = 0;
      cells[1] = c00 - 1; loc[1] = 1;
      cells[2] = c00 - v.nx; loc[2] = 3;
      cells[3] = c00 - v.nx - 1; loc[3] = 2;
    } else {
      if (i < v.ny && j < v.nx) { cells[kc] = c00; loc[kc++] = 0; }
      if (i < v.ny && j > 0) { cells[kc] = c00 - 1; loc[kc++] = 1; }
      if (i > 0 && j < v.nx) { cells[kc] = c00 - v.nx; loc[kc++] = 3; }
      if (i > 0 && j > 0) { cells[kc] = c00 - v.nx - 1; loc[kc++] = 2; }
    }
#define NODE_CELLS(t) _Pragma("unroll") for (int t = 0; t < 4; ++t) if (INNER || t < kc)
    const double X0 = ldg(v.xs, j), X1 = ldg(v.ys, i);
    double pe_tot[4], ue0[4], ue1[4];
    if (v.space_order == 2) {
      double d0[4], d1[4];
      bool dfin = true;
      NODE_CELLS(t) {
        d0[t] = X0 - ldg(v.xcc, cells[t]);
        d1[t] = X1 - ldg(v.xcc, P + cells[t]);
        dfin = dfin && is_finite(d0[t]) && is_finite(d1[t]);
        pe_tot[t] = 0.;
      }
      for (int m = 0; m < nb; ++m) {
        double pm[4], g0[4], g1[4], fm[4];
        unsigned long long any = 0;
        NODE_CELLS(t) {
          pm[t] = v.pm[m * P + cells[t]];
          g0[t] = v.Fs[(2 * m) * P + cells[t]];
          g1[t] = v.Fs[(2 * m + 1) * P + cells[t]];
          fm[t] = v.fm[m * P + cells[t]];
          any |= ubits(pm[t]) | ubits(g0[t]) | ubits(g1[t]);
          if (!is_finite(fm[t]) || neg(fm[t])) any = kMag;
        }
        if (dfin && (any & kMag) == 0) {
          NODE_CELLS(t) v.peex[(loc[t] * nb + m) * P + cells[t]] = 0.;
          continue;
        }
        double minP = 1.7976931348623157e308;
        double maxP = 2.2250738585072014e-308;  // numeric_limits<double>::min()
        NODE_CELLS(t) minP = smin(minP, pm[t]);
        NODE_CELLS(t) maxP = smax(maxP, pm[t]);
        NODE_CELLS(t) {
          const double pr = add_dot2(pm[t], g0[t], g1[t], d0[t], d1[t]);
          const double pe = smax(smin(maxP, pr), minP);
          v.peex[(loc[t] * nb + m) * P + cells[t]] = pe;
          pe_tot[t] = addz(pe_tot[t], mul_frac(fm[t], pe));  // 0.0 + t first
        }
      }
      NODE_CELLS(t) v.pex[loc[t] * P + cells[t]] = pe_tot[t];
      double vc0[4], vc1[4];
      NODE_CELLS(t) {
        vc0[t] = v.uc[cells[t]];
        vc1[t] = v.uc[P + cells[t]];
      }
      double minVx = 1.7976931348623157e308, maxVx = 2.2250738585072014e-308;
      double minVy = 1.7976931348623157e308, maxVy = 2.2250738585072014e-308;
      NODE_CELLS(t) minVx = smin(minVx, vc0[t]);
      NODE_CELLS(t) maxVx = smax(maxVx, vc0[t]);
      NODE_CELLS(t) minVy = smin(minVy, vc1[t]);
      NODE_CELLS(t) maxVy = smax(maxVy, vc1[t]);
      NODE_CELLS(t) {
        const long long c = cells[t];
        const double vt0 = add_dot2(vc0[t], v.vg[c], v.vg[P + c], d0[t], d1[t]);
        const double vt1 = add_dot2(vc1[t], v.vg[2 * P + c], v.vg[3 * P + c], d0[t], d1[t]);
        ue0[t] = smax(smin(maxVx, vt0), minVx);
        ue1[t] = smax(smin(maxVy, vt1), minVy);
        v.uex[(2 * loc[t]) * P + c] = ue0[t];
        v.uex[(2 * loc[t] + 1) * P + c] = ue1[t];
      }
    } else {
      NODE_CELLS(t) {
        const long long c = cells[t];
        const int k = loc[t];
        pe_tot[t] = v.p[c];
        ue0[t] = v.uc[c];
        ue1[t] = v.uc[P + c];
        v.pex[k * P + c] = pe_tot[t];
        v.uex[(2 * k) * P + c] = ue0[t];
        v.uex[(2 * k + 1) * P + c] = ue1[t];
#pragma unroll
        for (int m = 0; m < 3; ++m) {
          if (m >= nb) break;
          v.peex[(k * nb + m) * P + c] = v.pm[m * P + c];
        }
      }
    }
    // G and the node dissipation matrix: sums from 0.0, 0.0 + x as plus_zero
    double G[2] = {0.0, 0.0};
    double Mp[4] = {0.0, 0.0, 0.0, 0.0};
    bool diag = C.cmat_diag != 0;  // m01 = (+-0) * s: a zero for a finite s
    double sc[4];
    NODE_CELLS(t) {
      sc[t] = v.rho[cells[t]] * v.c[cells[t]];
      diag = diag && is_finite(sc[t]) && is_finite(ue0[t]) && is_finite(ue1[t]);
    }
    if (diag) {
      NODE_CELLS(t) {
        const long long c = cells[t];
        const int k = loc[t];
        const double m00 = ldg(v.cmat, (3 * k) * P + c) * sc[t];
        const double m11 = ldg(v.cmat, (3 * k + 2) * P + c) * sc[t];
        const double l0 = ldg(v.lpc, (2 * k) * P + c), l1 = ldg(v.lpc, (2 * k + 1) * P + c);
        // a zero velocity with finite entries: (+0) + l pe
        const double q0 = l0 * pe_tot[t], q1 = l1 * pe_tot[t];
        const double g0 = (iszero(ue0[t]) && is_finite(m00)) ? plus_zero(q0)
                                                             : plus_zero(m00 * ue0[t]) + q0;
        const double g1 = (iszero(ue1[t]) && is_finite(m11)) ? plus_zero(q1)
                                                             : plus_zero(m11 * ue1[t]) + q1;
        G[0] = (t == 0) ? plus_zero(g0) : G[0] + g0;
        G[1] = (t == 0) ? plus_zero(g1) : G[1] + g1;
        Mp[0] = (t == 0) ? plus_zero(m00) : Mp[0] + m00;
        Mp[3] = (t == 0) ? plus_zero(m11) : Mp[3] + m11;
      }
    } else {
      NODE_CELLS(t) {
        const long long c = cells[t];
        const int k = loc[t];
        const double s = sc[t];
        const double m00 = ldg(v.cmat, (3 * k) * P + c) * s;
        const double m01 = ldg(v.cmat, (3 * k + 1) * P + c) * s;
        const double m11 = ldg(v.cmat, (3 * k + 2) * P + c) * s;
        const double l0 = ldg(v.lpc, (2 * k) * P + c), l1 = ldg(v.lpc, (2 * k + 1) * P + c);
        // mv + l * pe, with (+0) + y = plus_zero(y) where mv = dot2(m, ue) is +0
        const double g0 = dot2_zero(m00, m01, ue0[t], ue1[t])
                              ? plus_zero(l0 * pe_tot[t])
                              : dot2(m00, m01, ue0[t], ue1[t]) + l0 * pe_tot[t];
        const double g1 = dot2_zero(m01, m11, ue0[t], ue1[t])
                              ? plus_zero(l1 * pe_tot[t])
                              : dot2(m01, m11, ue0[t], ue1[t]) + l1 * pe_tot[t];
        G[0] = (t == 0) ? plus_zero(g0) : G[0] + g0;
        G[1] = (t == 0) ? plus_zero(g1) : G[1] + g1;
        Mp[0] = (t == 0) ? plus_zero(m00) : Mp[0] + m00;
        Mp[1] = (t == 0) ? plus_zero(m01) : Mp[1] + m01;
        Mp[3] = (t == 0) ? plus_zero(m11) : Mp[3] + m11;
      }
      Mp[2] = Mp[1];  // the same sums
    }
#undef NODE_CELLS
    // node velocity: the boundary rule of the last list holding the node
    // (sides, then corners), inverse(Mp) . G inside
    double u0, u1;
    if (!INNER) {
      boundary(v, i, j, Mp, G, u0, u1);
    } else {
      // inverse(Mp) . G: with G two zeros the result is dot2(i, G) = +0 as
      // long as the inverse is finite: |Mp| < 2^500 and |det| >= 2^-500
      // bound it by 2^1000, so the reciprocal and the products are not
      // formed
      constexpr unsigned long long kLo = 523ull << 52, kHi = 1523ull << 52;
      const bool mod = (ubits(Mp[0]) & kMag) < kHi && (ubits(Mp[1]) & kMag) < kHi &&
                       (ubits(Mp[2]) & kMag) < kHi && (ubits(Mp[3]) & kMag) < kHi;
      const double det = diag ? Mp[0] * Mp[3] : Mp[0] * Mp[3] - Mp[1] * Mp[2];
      const bool inv = mod && (ubits(det) & kMag) >= kLo;  // finite: |Mp| < 2^500
      if (inv && iszero(G[0]) && iszero(G[1])) {
        u0 = 0.0;
        u1 = 0.0;
      } else if (inv && diag && is_finite(G[0]) && is_finite(G[1])) {
        const double alpha = div_ip(1.0, det);
        u0 = plus_zero(Mp[3] * alpha * G[0]);
        u1 = plus_zero(Mp[0] * alpha * G[1]);
      } else {
        bc_velocity(202, 0.0, 0.0, Mp, G, u0, u1);
      }
    }
    v.u[p] = u0;
    v.u[NP + p] = u1;
    v.XL[p] = addz(X0, mulz(u0, C.dt_n));
    v.XL[NP + p] = addz(X1, mulz(u1, C.dt_n));
  }
  static __device__ __noinline__ void boundary(const RunView& v, int i, int j, const double* Mp,
                                               const double* G, double& u0, double& u1) {
    const bool top = (i == v.ny), bot = (i == 0), lft = (j == 0), rgt = (j == v.nx);
    if ((top || bot) && (lft || rgt)) {
      const int b1 = top ? v.bc_top : v.bc_bottom;
      const double* V1 = top ? v.v_top : v.v_bottom;
      const int b2 = lft ? v.bc_left : v.bc_right;
      const double* V2 = lft ? v.v_left : v.v_right;
      const double A0 = V1[0], A1 = V1[1], B0 = V2[0], B1 = V2[1];
      u0 = 0.0;
      u1 = 0.0;
      if (b1 == kBcSym && b2 == kBcSym) {
        const double na = sqrt_ip(dot2(A0, A1, A0, A1)), nbb = sqrt_ip(dot2(B0, B1, B0, B1));
        if (fabs(fabs(dot2(A0, A1, B0, B1)) - na * nbb) < 1.0E-8)
          bc_velocity(kBcSym, A0, A1, Mp, G, u0, u1);
      } else if (b1 == kBcImposed && b2 == kBcImposed) {
        u0 = half(A0 + B0);
        u1 = half(A1 + B1);
      } else if (b1 == 202 && b2 == 202) {
        bc_velocity(202, A0, A1, Mp, G, u0, u1);
      }
    } else if (lft) {
      bc_velocity(v.bc_left, v.v_left[0], v.v_left[1], Mp, G, u0, u1);
    } else if (rgt) {
      bc_velocity(v.bc_right, v.v_right[0], v.v_right[1], Mp, G, u0, u1);
    } else if (top) {
      bc_velocity(v.bc_top, v.v_top[0], v.v_top[1], Mp, G, u0, u1);
    } else {
      bc_velocity(v.bc_bottom, v.v_bottom[0], v.v_bottom[1], Mp, G, u0, u1);
    }
  }
  __device__ __forceinline__ void operator()(const RunView& v, int i, int j) const {
    if (i > v.ny || j > v.nx) return;
    if (i > 0 && i < v.ny && j > 0 && j < v.nx) node<true>(v, i, j);
    else edge_node(v, i, j);
  }
  // out of line: the inner nodes' registers are not spent on it
  static __device__ __noinline__ void edge_node(const RunView& v, int i, int j) {
    EucNodes<NB>{}.template node<false>(v, i, j);
  }
};

// ----------------------------------------------------- cell Lagrange step
// computeLagrangeVolumeAndCenterOfGravity (:671-716), computeSubCellForce
// (:625-666), updateCellCenteredLagrangeVariables (:746-1010), and the
// Lagrangian face lengths that give HvLagrange (remap/PhaseRemap1.cc:57-71).
//
// The kernel is bound by the FP64 pipe (191 instructions per cell with all
// materials and the full corner matrices in every cell: 734 us at 1792 x 768
// cells and 3 materials, 427 us now; eight blocks per SM timed fastest of 3
// to 8 there).  Three whole-cell reductions, each exact and one branch:
//  - one material p (its fractions exactly 1, the others' fractions +0, their
//    densities and corner pressures zeros): the others' forces are +0 (l * (a
//    zero) + a zero), so their force sums are +0 and their conserved values
//    signed zeros; where p's corner pressures and rho_p c are the cell's bit
//    for bit, its forces are the cell's and are formed once;
//  - corner matrices without off-diagonal entries (cmat_diag, see EucNodes);
//  - every velocity difference at the corners a zero: no matrix product.
template <int NB = 0>
struct EucCells {
  // The sub-cell force l (-pe) + M s (u - u_ex) of one corner.
  struct Corner {
    double l0, l1, c00, c01, c11, du0, du1;
    bool still, diag;  // du zeros and small entries; c01 a zero, du finite
  };
  static DV bool small(double x) { return (ubits(x) & kMag) < 0x5fe0000000000000ull; }  // 2^511
  static DV void force(const Corner& q, double pe, double s, double& f0, double& f1) {
    const double mp = -pe;
    if (q.still && small(s)) {
      f0 = plus_zero(q.l0 * mp);
      f1 = plus_zero(q.l1 * mp);
    } else if (q.diag && is_finite(s)) {
      f0 = q.l0 * mp + plus_zero(q.c00 * s * q.du0);
      f1 = q.l1 * mp + plus_zero(q.c11 * s * q.du1);
    } else {
      const double m00 = q.c00 * s, m01 = q.c01 * s, m11 = q.c11 * s;
      f0 = q.l0 * mp + dot2(m00, m01, q.du0, q.du1);
      f1 = q.l1 * mp + dot2(m01, m11, q.du0, q.du1);
    }
  }
  // NS material slots: 1 (the material p) or 3 (all of the run's).
  template <int NS>
  static DV void body(const RunView& v, long long c, const long long* nd, const CellGeom& G,
                      int p) {
    const Ctrl& C = *v.ctrl;
    const long long P = v.pitch, NP = v.npitch;
    const int nb = NB ? NB : v.nbmat, nbl = NS == 1 ? 1 : nb;
    auto mat = [&](int m) { return NS == 1 ? p : m; };
    const double vol = G.vol;
    const double rho = v.rho[c], snd = v.c[c];
    const double s = rho * snd;
    double se[NS];
#pragma unroll
    for (int m = 0; m < NS; ++m) {
      se[m] = 0.0;
      if (m < nbl) {
        const double rm = v.rhom[mat(m) * P + c];
        se[m] = (NS == 1 && ubits(rm) == ubits(rho)) ? s : rm * snd;
      }
    }
    const bool diag = C.cmat_diag != 0;
    double r2 = 0.0, r3a = 0.0, r3b = 0.0;
    double un0[4], un1[4], Fe0[4][NS], Fe1[4][NS];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const double u0 = v.u[nd[k]], u1 = v.u[NP + nd[k]];
      un0[k] = u0;
      un1[k] = u1;
      Corner q;
      q.l0 = ldg(v.lpc, (2 * k) * P + c);
      q.l1 = ldg(v.lpc, (2 * k + 1) * P + c);
      const bool uz = iszero(u0) && iszero(u1);
      const bool t2z = uz && is_finite(q.l0) && is_finite(q.l1);  // dot2(l, u) = +0
      const double t2 = t2z ? 0.0 : dot2(q.l0, q.l1, u0, u1);
      r2 = (k == 0) ? plus_zero(t2) : (t2z ? plus_zero(r2) : r2 + t2);
      const double ux0 = v.uex[(2 * k) * P + c], ux1 = v.uex[(2 * k + 1) * P + c];
      // velocity differences; any zero difference gives the same dot2, so
      // two zeros minus two zeros need not be formed
      q.du0 = q.du1 = 0.0;
      bool duz = uz && iszero(ux0) && iszero(ux1);
      if (!duz) {
        q.du0 = u0 - ux0;
        q.du1 = u1 - ux1;
        duz = iszero(q.du0) && iszero(q.du1);
      }
      q.c00 = ldg(v.cmat, (3 * k) * P + c);
      q.c11 = ldg(v.cmat, (3 * k + 2) * P + c);
      q.c01 = diag ? 0.0 : ldg(v.cmat, (3 * k + 1) * P + c);
      q.diag = diag && is_finite(q.du0) && is_finite(q.du1);
      q.still = duz && small(q.c00) && small(q.c01) && small(q.c11);
      const double pex = v.pex[k * P + c];
      double f0, f1;
      force(q, pex, s, f0, f1);
      r3a = (k == 0) ? plus_zero(f0) : r3a + f0;
      r3b = (k == 0) ? plus_zero(f1) : r3b + f1;
#pragma unroll
      for (int m = 0; m < NS; ++m) {
        if (m >= nbl) break;
        const double pe = v.peex[(k * nb + mat(m)) * P + c];
        if (NS == 1 && ubits(pe) == ubits(pex) && ubits(se[m]) == ubits(s)) {
          Fe0[k][m] = f0;
          Fe1[k][m] = f1;
        } else {
          force(q, pe, se[m], Fe0[k][m], Fe1[k][m]);
        }
      }
    }
    const double dt = C.dt_n;
    const double cmass = v.cell_mass[c];
    // (dt / cmass) * r2: a zero r2 times a finite quotient (|dt| < 2^500,
    // |cmass| >= 2^-500) is the zero of the xor of the three signs
    constexpr unsigned long long kLo = 523ull << 52, kHi = 1523ull << 52;  // 2^-500, 2^500
    const bool qfin = (ubits(dt) & kMag) < kHi && (ubits(cmass) & kMag) >= kLo &&
                      is_finite(cmass);
    double rhoL;
    if (iszero(r2) && qfin) {
      const double dr2 = from_bits((ubits(dt) ^ ubits(cmass) ^ ubits(r2)) & ~kMag);
      rhoL = div_ip(1.0, addz(div_ip(1.0, rho), dr2));
    } else {
      rhoL = div_ip(1.0, addz(div_ip(1.0, rho), div_ip(dt, cmass) * r2));
    }
    const double uc0 = v.uc[c], uc1 = v.uc[P + c];
    const double uL0 = addz(uc0, qdiv(mulz(r3a, dt), cmass));
    const double uL1 = addz(uc1, qdiv(mulz(r3b, dt), cmass));
    const double mid0 = half(addz(uc0, uL0)), mid1 = half(addz(uc1, uL1));
    double pr4[NS], fsa[NS], fsb[NS];
#pragma unroll
    for (int m = 0; m < NS; ++m) pr4[m] = fsa[m] = fsb[m] = 0.0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const double d0 = subz(un0[k], mid0), d1 = subz(un1[k], mid1);
      const bool dz = iszero(d0) && iszero(d1);
#pragma unroll
      for (int m = 0; m < NS; ++m) {
        if (m >= nbl) break;
        const bool t4z = dz && is_finite(Fe0[k][m]) && is_finite(Fe1[k][m]);  // dot2 = +0
        const double t4 = t4z ? 0.0 : dot2(Fe0[k][m], Fe1[k][m], d0, d1);
        pr4[m] = (k == 0) ? plus_zero(t4) : (t4z ? plus_zero(pr4[m]) : pr4[m] + t4);
        // (p's sums are the cell's where its forces are)
        fsa[m] = (k == 0) ? plus_zero(Fe0[k][m]) : fsa[m] + Fe0[k][m];
        fsb[m] = (k == 0) ? plus_zero(Fe1[k][m]) : fsb[m] + Fe1[k][m];
      }
    }
    double peL[NS];
    const double thr = v.threshold;
#pragma unroll
    for (int m = 0; m < NS; ++m) {
      if (m >= nbl) break;
      peL[m] = 0.;
      const double f = v.fm[mat(m) * P + c], cmm = v.cmassm[mat(m) * P + c];
      if (dgt(f, thr) && nz(cmm)) {
        // ((f * dt) / cmm) * pr4: a zero pr4 times a finite quotient (|f| and
        // |dt| below 2^250, |cmm| >= 2^-500: under 2^1000) is a signed zero
        constexpr unsigned long long kMid = 1273ull << 52;  // 2^250
        const double em = v.em[mat(m) * P + c];
        const bool pz = iszero(pr4[m]) && (ubits(f) & kMag) < kMid && (ubits(dt) & kMag) < kMid &&
                        (ubits(cmm) & kMag) >= kLo && is_finite(cmm);
        if (pz)
          peL[m] = addz(em, from_bits((ubits(f) ^ ubits(dt) ^ ubits(cmm) ^ ubits(pr4[m])) & ~kMag));
        else
          peL[m] = addz(em, div_ip(mul_frac(f, dt), cmm) * pr4[m]);
      }
    }
    // ULagrange and Phi
    const int ncomp = v.ncomp;
    double uv[NS], um[NS], ue[NS];
#pragma unroll
    for (int m = 0; m < NS; ++m) {
      if (m >= nbl) break;
      const double mv = mul_frac(v.mfm[mat(m) * P + c], vol);  // ((mf * vol) * rho) * e
      uv[m] = mul_frac(v.fm[mat(m) * P + c], vol);
      um[m] = mulz(mv, rhoL);
      ue[m] = mulz(um[m], peL[m]);
    }
    const double vr = (NS == 1) ? um[0] : vol * rhoL;  // 1 * vol * rhoL
    const double px = mulz(vr, uL0), py = mulz(vr, uL1);
    const double ke = (v.conservative == 1) ? 0.5 * vol * rhoL * (uL0 * uL0 + uL1 * uL1) : 0.0;
#pragma unroll
    for (int m = 0; m < NS; ++m) {
      if (m >= nbl) break;
      v.UL[mat(m) * P + c] = uv[m];
      v.UL[(nb + mat(m)) * P + c] = um[m];
      v.UL[(2 * nb + mat(m)) * P + c] = ue[m];
    }
    v.UL[3 * nb * P + c] = px;
    v.UL[(3 * nb + 1) * P + c] = py;
    if (ncomp > 3 * nb + 2) v.UL[(3 * nb + 2) * P + c] = ke;
    // the other materials of a single-material cell (vol > 0): U = (+0, (+0)
    // rhoL, ((+0) rhoL) (+0)) and what Phi makes of them
    const double zr = mulz(0.0, rhoL), ze = mulz(zr, 0.0);
    if (v.pb == 1) {
      double sv = 0., sm = 0.;
#pragma unroll
      for (int m = 0; m < NS; ++m)
        if (m < nbl) {
          sv = addz(sv, uv[m]);
          sm = addz(sm, um[m]);
        }
#pragma unroll
      for (int m = 0; m < NS; ++m) {
        if (m >= nbl) break;
        v.Phi[mat(m) * P + c] = qdiv(uv[m], sv);
        v.Phi[(nb + mat(m)) * P + c] = nz(uv[m]) ? qdiv(um[m], uv[m]) : 0.;
        v.Phi[(2 * nb + mat(m)) * P + c] = nz(um[m]) ? qdiv(ue[m], um[m]) : 0.;
      }
      const SharedDiv Sm = shared_div(sm);
      v.Phi[3 * nb * P + c] = qdiv_shared(Sm, px);
      v.Phi[(3 * nb + 1) * P + c] = qdiv_shared(Sm, py);
      if (v.conservative == 1) v.Phi[(3 * nb + 2) * P + c] = qdiv_shared(Sm, ke);
    } else {
      const SharedDiv Sv = shared_div(vol);  // one denominator, ncomp quotients
#pragma unroll
      for (int m = 0; m < NS; ++m) {
        if (m >= nbl) break;
        v.Phi[mat(m) * P + c] = qdiv_shared(Sv, uv[m]);
        v.Phi[(nb + mat(m)) * P + c] = qdiv_shared(Sv, um[m]);
        v.Phi[(2 * nb + mat(m)) * P + c] = qdiv_shared(Sv, ue[m]);
      }
      v.Phi[3 * nb * P + c] = qdiv_shared(Sv, px);
      v.Phi[(3 * nb + 1) * P + c] = qdiv_shared(Sv, py);
      if (v.conservative == 1) v.Phi[(3 * nb + 2) * P + c] = qdiv_shared(Sv, ke);
    }
    if (NS == 1)
      for (int m = 0; m < nb; ++m) {
        if (m == p) continue;
        v.UL[m * P + c] = 0.0;
        v.UL[(nb + m) * P + c] = zr;
        v.UL[(2 * nb + m) * P + c] = ze;
        v.Phi[m * P + c] = 0.0;
        v.Phi[(nb + m) * P + c] = (v.pb == 1) ? 0.0 : zr;  // (+-0) / vol
        v.Phi[(2 * nb + m) * P + c] = (v.pb == 1 && !nz(zr)) ? 0.0 : ze;
        v.Fs[(2 * m) * P + c] = 0.0;
        v.Fs[(2 * m + 1) * P + c] = 0.0;
      }
    // per-material corner-force sums for the next cycle's gradients, and
    // the Lagrangian geometry (volume, centroid, HvLagrange widths)
#pragma unroll
    for (int m = 0; m < NS; ++m) {
      if (m >= nbl) break;
      v.Fs[(2 * mat(m)) * P + c] = fsa[m];
      v.Fs[(2 * mat(m) + 1) * P + c] = fsb[m];
    }
    v.vL[c] = vol;
    v.XcL[c] = G.xc0;
    v.XcL[P + c] = G.xc1;
    if (v.order > 1) {
      v.Hx[c] = G.hx;
      v.Hy[c] = G.hy;
    }
  }
  __device__ __forceinline__ void operator()(const RunView& v, int i, int j) const {
    const unsigned lanes = lanes_inside(i < v.ny && j < v.nx);
    if (i >= v.ny || j >= v.nx) return;
    const long long P = v.pitch, NP = v.npitch;
    const long long c = (long long)i * v.nx + j;
    const int nb = NB ? NB : v.nbmat;
    const long long n0 = (long long)i * (v.nx + 1) + j;
    const long long nd[4] = {n0, n0 + 1, n0 + v.nx + 2, n0 + v.nx + 1};
    double X[4][2];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      X[k][0] = v.XL[nd[k]];
      X[k][1] = v.XL[NP + nd[k]];
    }
    // one material: fractions exactly 1 / +0, zero densities and corner
    // pressures of the others, a finite cell density and sound speed
    int p = -1;
    bool single = true;
    for (int m = 0; m < nb; ++m) {
      constexpr unsigned long long kOne = 0x3ff0000000000000ull;
      const unsigned long long f = ubits(v.fm[m * P + c]), mf = ubits(v.mfm[m * P + c]);
      if (f == kOne && mf == kOne) {
        single = single && p < 0;
        p = m;
      } else {
        unsigned long long z = ubits(v.rhom[m * P + c]);
#pragma unroll
        for (int k = 0; k < 4; ++k) z |= ubits(v.peex[(k * nb + m) * P + c]);
        single = single && (f | mf) == 0 && (z & kMag) == 0;
      }
    }
    single = single && p >= 0 && is_finite(v.rho[c]) && is_finite(v.c[c]);
    // Lagrangian geometry; a cell whose four nodes kept their Euler
    // positions (bit for bit) has the geometry the set-up formed with the
    // same function from the same numbers (loaded with the positions).
    // The geometry is stored at the end: a store here would order every
    // later load behind it.
    double g0v[5];
#pragma unroll
    for (int q = 0; q < 5; ++q) g0v[q] = ldg(v.geo0, q * P + c);
    const unsigned long long x0 = ubits(ldg(v.xs, j)), x1 = ubits(ldg(v.xs, j + 1));
    const unsigned long long y0 = ubits(ldg(v.ys, i)), y1 = ubits(ldg(v.ys, i + 1));
    const bool rest = ubits(X[0][0]) == x0 && ubits(X[0][1]) == y0 && ubits(X[1][0]) == x1 &&
                      ubits(X[1][1]) == y0 && ubits(X[2][0]) == x1 && ubits(X[2][1]) == y1 &&
                      ubits(X[3][0]) == x0 && ubits(X[3][1]) == y1;
    CellGeom G;
    if (rest) {
      G.vol = g0v[0];
      G.xc0 = g0v[1];
      G.xc1 = g0v[2];
      G.hx = g0v[3];
      G.hy = g0v[4];
    } else {
      G = euc_cell_geometry(X, v.order > 1);
    }
    single = single && pos(G.vol) && is_finite(G.vol) && nonneg(v.threshold);
    // the warp takes one of the two bodies: with both, its lanes would wait
    // for each other's (triple point 70 x 30: 45 us with one, 61 us with two)
    if (__all_sync(lanes, single)) body<1>(v, c, nd, G, p);
    else body<3>(v, c, nd, G, 0);
  }
};

// --------------------------------------------------------- remap final
// Eucclhyd::remapCellcenteredVariable (PhaseRemapFinal.cc:17-200)
//
// single: a cell that holds one material p (the others' volume, mass and
// energy +0.0, p's volume and mass positive and finite, the threshold in
// [0, 1)).  The general path then reduces exactly to volt = vn_p (x + +0 =
// x), masset = Um_p, vn_p' = vn_p (vol / vn_p) with the others +0, f = mf = 1
// and +0 (x / x, +0 / x, neither moved by the threshold), rho = 0.0 + Um_p /
// vn_p', e_p = Ue_p / Um_p + dec, e = 0.0 + e_p, and the others' density +0
// and energy 0.0 + dec.  A value that leaves these ranges (a negative or NaN
// density or energy) returns false before any store.  One branch for the
// cell: 35 -> 8 FP64 instructions, 119 -> 64 us at 1792 x 768 cells and 3
// materials.
template <int NB = 0>
struct EucFinal {
  static DV void store_velocity(const RunView& v, long long c, double un0, double un1) {
    // velocities for the outputs (PhaseRemapFinal.cc:200-213): kept where
    // the velocity is zero, else pushed away from zero to the threshold
    const double thr = v.threshold;
    const long long P = v.pitch;
    v.uc[c] = un0;
    v.uc[P + c] = un1;
    if (pos(un0)) v.uco[c] = smax(un0, thr);
    else if (neg(un0)) v.uco[c] = smin(un0, -thr);
    if (pos(un1)) v.uco[P + c] = smax(un1, thr);
    else if (neg(un1)) v.uco[P + c] = smin(un1, -thr);
  }
  // lanes: those of the warp that are inside the mesh, which all call this
  static DV bool single(const RunView& v, long long c, unsigned lanes) {
    const long long P = v.pitch;
    const int nb = NB ? NB : v.nbmat;
    const double* U = v.UL + c;
    const double thr = v.threshold;
    if (!(nonneg(thr) && dlt(thr, 1.0))) return false;
    int p = -1, nonzero = 0;
    double vn = 0., um = 0., ue = 0.;
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      if (m >= nb) break;
      const double a = U[m * P], b = U[(nb + m) * P], e = U[(2 * nb + m) * P];
      if ((ubits(a) | ubits(b) | ubits(e)) != 0ull) {
        p = m;
        ++nonzero;
        vn = a;
        um = b;
        ue = e;
      }
    }
    // (a warp with a mixed cell takes the general path whole, not both)
    if (!__all_sync(lanes, nonzero == 1)) return false;
    if (!(pos(vn) && is_finite(vn) && pos(um) && is_finite(um))) return false;
    const double q0 = U[3 * nb * P], q1 = U[(3 * nb + 1) * P];
    const double vol = ldg(v.evol, c);
    const double r = qdiv(vol, vn);
    if (!(pos(r) && is_finite(r))) return false;
    const double vnp = mul1z(vn, r);
    if (!(pos(vnp) && is_finite(vnp))) return false;
    const double dm = qdiv(um, vnp), pe = qdiv(ue, um);
    if (neg(dm) || neg(pe) || is_nan(dm) || is_nan(pe)) return false;
    const double dens = plus_zero(dm);
    const SharedDiv Smv = shared_div(dens * vol);
    const double un0 = qdiv_shared(Smv, q0), un1 = qdiv_shared(Smv, q1);
    double dec = 0.;
    if (v.conservative == 1)
      dec = qdiv(U[(3 * nb + 2) * P], um) - 0.5 * (un0 * un0 + un1 * un1);
    if (!is_finite(dec)) return false;
    const double em = addz(pe, dec), eo = addz(0.0, dec);
    const double e = plus_zero(em);
    if (is_nan(e)) return false;
    v.mixte[c] = 0;
    v.pure[c] = p;
    v.rho[c] = dens;
    v.e[c] = e;
    store_velocity(v, c, un0, un1);
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      if (m >= nb) break;
      const bool here = m == p;
      v.fm[m * P + c] = here ? 1.0 : 0.0;
      v.mfm[m * P + c] = here ? 1.0 : 0.0;
      v.rhom[m * P + c] = here ? dm : 0.0;
      v.em[m * P + c] = here ? em : eo;
    }
    return true;
  }
  __device__ __forceinline__ void operator()(const RunView& v, int i, int j) const {
    const unsigned lanes = lanes_inside(i < v.ny && j < v.nx);
    if (i >= v.ny || j >= v.nx) return;
    Ctrl& C = *v.ctrl;
    const long long P = v.pitch;
    const long long c = (long long)i * v.nx + j;
    if (single(v, c, lanes)) return;
    const int nb = NB ? NB : v.nbmat;
    const double thr = v.threshold;
    const double* U = v.UL + c;  // second sweep output
    const double vol = ldg(v.evol, c);
    double volt = 0., masset = 0., vn[3];
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      if (m >= nb) break;
      vn[m] = U[m * P];
      volt = (m == 0) ? plus_zero(vn[m]) : volt + vn[m];  // 0.0 + x first
      masset = (m == 0) ? plus_zero(U[(nb + m) * P]) : masset + U[(nb + m) * P];
    }
    double vnorm = 0.;
    const double r = qdiv(vol, volt);
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      if (m >= nb) break;
      vn[m] *= r;
      vnorm = (m == 0) ? plus_zero(vn[m]) : vnorm + vn[m];
    }
    double f[3], mf[3], sf = 0.;
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      if (m >= nb) break;
      f[m] = qdiv(vn[m], vnorm);
      if (dlt(f[m], thr)) f[m] = 0.;
      sf = (m == 0) ? plus_zero(f[m]) : sf + f[m];
    }
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      if (m >= nb) break;
      f[m] = qdiv(f[m], sf);
    }
    int matcell = 0, imatpure = -1;
    for (int m = 0; m < nb; ++m)
      if (pos(f[m])) {
        matcell++;
        imatpure = m;
      }
    v.mixte[c] = (matcell > 1) ? 1 : 0;
    v.pure[c] = (matcell > 1) ? -1 : imatpure;
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      if (m >= nb) break;
      mf[m] = qdiv(U[(nb + m) * P], masset);
    }
    double fmt = 0.;
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      if (m >= nb) break;
      if (dlt(f[m], thr)) mf[m] = 0.;
      fmt = (m == 0) ? plus_zero(mf[m]) : fmt + mf[m];
    }
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      if (m >= nb) break;
      mf[m] = qdiv(mf[m], fmt);
    }
    double dm[3] = {0., 0., 0.}, dens = 0.;
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      if (m >= nb) break;
      if (dgt(f[m], thr)) dm[m] = qdiv(U[(nb + m) * P], vn[m]);
      const double fd = mul_frac(f[m], dm[m]);
      dens = (m == 0) ? plus_zero(fd) : dens + fd;
    }
    const double mv = dens * vol;
    const double un0 = qdiv(U[3 * nb * P], mv), un1 = qdiv(U[(3 * nb + 1) * P], mv);
    double pe[3] = {0., 0., 0.};
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      if (m >= nb) break;
      if (dgt(f[m], thr) && nz(U[(nb + m) * P]))
        pe[m] = qdiv(U[(2 * nb + m) * P], U[(nb + m) * P]);
    }
    double dec = 0.;
    if (v.conservative == 1)
      dec = qdiv(U[(3 * nb + 2) * P], masset) - 0.5 * (un0 * un0 + un1 * un1);
    double e = 0.;
    double rhom[3], em[3];
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      if (m >= nb) break;
      rhom[m] = dm[m];
      em[m] = pe[m];
      em[m] += dec;
      const double te = mul_frac(mf[m], em[m]);
      e = (m == 0) ? plus_zero(te) : e + te;
    }
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      if (m >= nb) break;
      if (neg(pe[m]) || neg(dm[m])) {
        rhom[m] = 0.;
        em[m] = 0.;
        mf[m] = 0.;
        f[m] = 0.;
        atomicOr(&C.err, HYDRO_ERR_NEGATIVE);
      }
    }
    if (is_nan(e) || is_nan(dens)) {
      atomicOr(&C.err, HYDRO_ERR_NAN);
      atomicMin((unsigned long long*)&C.err_cell, (unsigned long long)c);
    }
    v.rho[c] = dens;
    v.e[c] = e;
    store_velocity(v, c, un0, un1);
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      if (m >= nb) break;
      v.fm[m * P + c] = f[m];
      v.mfm[m * P + c] = mf[m];
      v.rhom[m * P + c] = rhom[m];
      v.em[m * P + c] = em[m];
    }
  }
};

// The mean pressure that Eucclhyd::dumpVariables writes: computeEOS +
// computePressionMoyenne (PhaseLagrange.cc:70-155) on the current state,
// i.e. what the next cycle's first kernel computes, into out[c].
__global__ void __launch_bounds__(kBX* kBY) ke_out_pressure(RunView v, double* out) {
  const int i = blockIdx.y * kBY + threadIdx.y, j = blockIdx.x * kBX + threadIdx.x;
  if (i >= v.ny || j >= v.nx) return;
  const long long c = (long long)i * v.nx + j;
  double p = 0.;
  for (int m = 0; m < v.nbmat; ++m) {
    const double pm =
        cell_pressure(v, m, v.rhom[m * v.pitch + c], v.em[m * v.pitch + c], c);
    p += v.fm[m * v.pitch + c] * pm;
  }
  out[c] = p;
}

template <class F>
__device__ __forceinline__ void plain_items(const RunView& v, const F& f) {
  if (!v.ctrl->active) return;
  f(v, blockIdx.y * kBY + threadIdx.y, blockIdx.x * kBX + threadIdx.x);
}

template <int NB>
__global__ void __launch_bounds__(kBX* kBY, 8) ke_cell_pre(RunView v) { plain_items(v, EucCellPre<NB>{}); }
template <int NB>
__global__ void __launch_bounds__(kBX* kBY, 5) ke_nodes(RunView v, SplitGrid g) { split_node_items(v, g, EucNodes<NB>{}); }
template <int NB>
__global__ void __launch_bounds__(kBX* kBY, 8) ke_cells(RunView v) { plain_items(v, EucCells<NB>{}); }
template <int NB>
__global__ void __launch_bounds__(kBX* kBY, 10) ke_final(RunView v) { plain_items(v, EucFinal<NB>{}); }

// Batched launches of the Eucclhyd phases (the batch's VNR runs are skipped;
// the remap sweeps are the shared batched kernels of vnr.cu).
constexpr int kE = HYDRO_SCHEME_EUCCLHYD;
__global__ void __launch_bounds__(kBatchThreads, 8) kbe_cell_pre(BatchArgs b) { batch_items(b, EucCellPre<>{}, kE); }
__global__ void __launch_bounds__(kBatchThreads, 8) kbe_nodes(BatchArgs b) { batch_items(b, EucNodes<>{}, kE); }
__global__ void __launch_bounds__(kBatchThreads, 8) kbe_cells(BatchArgs b) { batch_items(b, EucCells<>{}, kE); }
__global__ void __launch_bounds__(kBatchThreads, 10) kbe_final(BatchArgs b) { batch_items(b, EucFinal<>{}, kE); }
// one thread per Eucclhyd run: cycle start and end
__global__ void kbe_begin(const RunView* views, const int* ninst) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= *ninst) return;
  const RunView v = views[r];
  if (v.scheme == kE) euc_begin_at(v);
}
__global__ void kbe_end(const RunView* views, const int* ninst, int* done) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= *ninst) return;
  const RunView v = views[r];
  if (v.scheme != kE) return;
  euc_end_at(v);
  done[r] = v.ctrl->done;
}

}  // namespace

int launch_euc_out_pressure(const RunView& v, double* out, cudaStream_t s) {
  const dim3 cg((v.nx + kBX - 1) / kBX, (v.ny + kBY - 1) / kBY);
  ke_out_pressure<<<cg, dim3(kBX, kBY), 0, s>>>(v, out);
  return 1;
}

// One Eucclhyd phase of a batched cycle: kPhEucCellPre, kPhEucNodes,
// kPhEucCells, kPhEucFinal on the tile arguments a, or (ph < 0) the
// per-run cycle start (-1) / end (-2).
void launch_batch_euc(int ph, const BatchLaunch& L, const BatchArgs& a, int grid,
                      cudaStream_t s) {
  const int T = kBatchThreads, rg = (L.max_inst + T - 1) / T;
  switch (ph) {
    case -1: kbe_begin<<<rg, T, 0, s>>>(L.views, L.ninst); break;
    case -2: kbe_end<<<rg, T, 0, s>>>(L.views, L.ninst, L.done); break;
    case kPhEucCellPre: kbe_cell_pre<<<grid, T, 0, s>>>(a); break;
    case kPhEucNodes: kbe_nodes<<<grid, T, 0, s>>>(a); break;
    case kPhEucCells: kbe_cells<<<grid, T, 0, s>>>(a); break;
    case kPhEucFinal: kbe_final<<<grid, T, 0, s>>>(a); break;
    default: break;
  }
}
// resident blocks per SM of the Eucclhyd phase kernels
int batch_occupancy_euc(int* blocks_per_sm) {
  const int ph[4] = {kPhEucCellPre, kPhEucNodes, kPhEucCells, kPhEucFinal};
  const void* fns[4] = {(const void*)kbe_cell_pre, (const void*)kbe_nodes,
                        (const void*)kbe_cells, (const void*)kbe_final};
  for (int k = 0; k < 4; ++k) {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fns[k], kBatchThreads, 0) !=
        cudaSuccess)
      return -1;
    blocks_per_sm[ph[k]] = n;
  }
  return 0;
}

// One Eucclhyd cycle on stream s (kind ids: 0 begin, 12 cell_pre, 13 nodes,
// 14 cells, sweeps, 15 final, 10 end).  Returns the number of kernels.
template <int NB>
static int launch_cycle_n(const RunView& v, cudaStream_t s, const LaunchHook* hook) {
  const dim3 blk(kBX, kBY);
  const dim3 cg((v.nx + kBX - 1) / kBX, (v.ny + kBY - 1) / kBY);
  int nk = 0;
  auto H = [&](int kind) {
    if (hook) (*hook)(kind);
  };
  H(0); ke_begin<<<1, 1, 0, s>>>(v); ++nk;
  H(12); ke_cell_pre<NB><<<cg, blk, 0, s>>>(v); ++nk;
  SplitGrid sg;
  const dim3 sng = split_node_grid(v.nx, v.ny, &sg);
  H(13); ke_nodes<NB><<<sng, blk, 0, s>>>(v, sg); ++nk;
  H(14); ke_cells<NB><<<cg, blk, 0, s>>>(v); ++nk;
  for (int sweep = 1; sweep <= 2; ++sweep) nk += launch_sweep(v, sweep, s, hook, nullptr);
  H(15); ke_final<NB><<<cg, blk, 0, s>>>(v); ++nk;
  H(10); ke_end<<<1, 1, 0, s>>>(v); ++nk;
  H(-1);
  return nk;
}

int launch_cycle_euc(const RunView& v, cudaStream_t s, const LaunchHook* hook) {
  if (v.nbmat == 1) return launch_cycle_n<1>(v, s, hook);
  if (v.nbmat == 2) return launch_cycle_n<2>(v, s, hook);
  return launch_cycle_n<3>(v, s, hook);
}

}  // namespace hydro
