// Richards residual, analytic Jacobian assembly and stencil matvec.
//
// Two launch forms, bitwise equal.  Gather: every cell computes the fluxes (or
// flux derivatives) of its own six faces; a face shared by two cells is
// evaluated by both with the same operands in the same order.  March: a warp
// walks a strip of rows up through the planes and evaluates (almost) every
// face once.  Neither needs atomics.  Per-cell relative permeabilities are produced by a first pass
// (k_vg_all) so that each cell's van Genuchten state is evaluated once per
// iterate and shared by the residual and the Jacobian.
#include "march_rule.h"
#include "pfgpu_device.cuh"
#include "pdl.cuh"
#include "pfgpu_kernels.h"

namespace pfgpu {

// (i, j, k) of a thread in a 3-D launch (x across the block's threads,
// rows in y, one plane per blockIdx.z): no integer division
__device__ __forceinline__ bool launch_ijk(int nx, int ny, int nz, int &i, int &j, int &k) {
  i = blockIdx.x * blockDim.x + threadIdx.x;
  j = blockIdx.y * blockDim.y + threadIdx.y;
  k = blockIdx.z;
  return i < nx && j < ny && k < nz;
}

// Van Genuchten state of every cell at one pressure iterate: kr, dkr/dp, S,
// dS/dp (problem_phase_rel_perm.c:1312-1361, problem_saturation.c:342-412).
// The residual uses kr and S; the Jacobian at the same iterate reuses all four.
// STEP: the iterate is formed here, pn = u + lam pp (lam from lam_p when
// given), and written too.  Bound by instruction issue and FP64 arithmetic (84 %
// of the slots, the FP64 pipe active 55 %): two logarithms, two exponentials and
// a square root per unsaturated cell (k_saturation, with the same ones and half
// the bytes, takes four fifths of the time).  512x512x50 after a timestep: 181
// us (memory floor 97 us, 48 B per cell with a field of alpha), with the step 185;
// the reference's logarithms and powers one by one, a division per reciprocal
// and per n, took 191 us there, and the trial step 43 us of its own.
// q: 1/(rho g), and m = 1 - 1/n of a uniform n
struct VGUniform {
  double inv_rg, m;
};
__device__ __forceinline__ VGAll vg_cell(const DevProblem &P, const VGUniform &q, const VG &vg,
                                         double pc) {
  const double m = P.vgn ? 1.0 - fast_rcp(vg.n) : q.m;
  VGAll v = vg_all(P, pc, vg, q.inv_rg, m);
  if (P.krt) {  // relative permeability from the lookup table
    if (pc >= 0.0) {
      v.kr = 1.0;
      v.dkr = 0.0;
    } else {
      const double head = fabs(pc) / (P.density * P.gravity);
      v.kr = krt_lookup(P, head, 0);
      v.dkr = krt_lookup(P, head, 1);
    }
  }
  return v;
}
// Six blocks per SM against five: residual with this pass at 256x256x50 107.3 us
// against 108.3, 512x512x50 380 against 385; two cells per thread in 16-byte
// accesses 109.9 and 389 (times after a timestep: at zero pressure, where
// nothing is evaluated, the wider accesses looked better).
template <bool STEP>
__global__ void __launch_bounds__(256, 6) k_vg_all(DevProblem P, VGUniform q,
                         const double *__restrict__ p, double *__restrict__ kr,
                         double *__restrict__ dkr, double *__restrict__ sat,
                         double *__restrict__ dsat, const double *__restrict__ pp,
                         const double *lam_p, double lam, double *__restrict__ pn) {
  const long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (c >= P.n) return;
  const VG vg = vg_at(P, c);  // (fields: older than the kernel before this one)
  pdl_enter();
  double pc = p[c];
  if (STEP) {
    const double a = lam_p ? *lam_p : lam;
    if (a != 0.0) pc = fma(a, pp[c], pc);
    pn[c] = pc;
  }
  const VGAll v = vg_cell(P, q, vg, pc);
  kr[c] = v.kr;
  dkr[c] = v.dkr;
  sat[c] = v.s;
  dsat[c] = v.ds;
}

__global__ void k_saturation(DevProblem P, VGUniform q, const double *__restrict__ p,
                             double *__restrict__ s) {
  const long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (c >= P.n) return;
  const VG vg = vg_at(P, c);
  const double m = P.vgn ? 1.0 - fast_rcp(vg.n) : q.m;
  pdl_enter();
  s[c] = vg_all(P, p[c], vg, q.inv_rg, m).s;
}

// Residual (nl_function_eval.c:167-2323).  Accumulation order per cell
// follows the reference: accumulation, storage, sources, then the face
// fluxes scattered from the k-1, j-1, i-1 neighbours, the cell's own three
// upper faces, and finally the boundary patches in patch order.
// SURF: slopes and/or overland flow present (false: flat box, the lean path)
// VEL: also write the face velocities and overland fluxes (VelOut): interior
// faces as flux / area (nl_function_eval.c:845-848), boundary faces as the
// patch loops store them (vel_vec[vel_idx], :1227-1230, :1432, :1681-1687,
// :1775-1781), q_overlnd_x / y = ke, kn of the column (:1648-1656)
//
// residual_cell is everything of one cell's F but the interior face fluxes,
// which the caller supplies: the lower z / y / x faces (fl_z, fl_y, fl_x,
// used where k, j, i > 0) and the cell's own right / front / upper faces
// (0 on the domain's upper faces).  Both launch forms below pass the values
// of the same flux functions with the same operands, so their F is equal
// bit for bit.
// ponding and routing term of an overland top cell: the change of the ponded
// depth and the divergence of the routed flux
__device__ __forceinline__ double ponding(const DevProblem &P, double dt, double vol, double pc,
                                          double po, double dqx, double dqy) {
  const double div = __dadd_rn(dqx / P.dx, dqy / P.dy);
  return __dadd_rn(__dmul_rn(vol, pmax0(pc) - pmax0(po)) / P.dz,
                   __dmul_rn(__dmul_rn(dt, vol), div) / P.dz);
}

template <bool SURF, bool VEL>
__device__ __forceinline__ void residual_cell(const DevProblem &P, int i, int j, int k,
                                              long long c, const double *__restrict__ p,
                                              const double *__restrict__ p_old, double dt,
                                              double *__restrict__ f, const VelOut &V,
                                              double pc, double krc, double sat, double so,
                                              double po, double zm, double fl_z, double fl_y, double fl_x,
                                              double u_right, double u_front, double u_upper) {
  const long long sz = (long long)P.nx * P.ny;
  const double rho = P.density, g = P.gravity;
  const double vol = P.dx * P.dy * P.dz;
  // (multiply-adds written out here and in the fluxes, so that every launch
  // form rounds alike)
  const double vz = vol * zm;
  double fc = __dmul_rn(__dmul_rn(__dmul_rn(sat, rho) - __dmul_rn(so, rho), P.porosity), vz);
  fc = fma(__dmul_rn(P.sstorage, vz),
           __dmul_rn(__dmul_rn(pc, sat), rho) - __dmul_rn(__dmul_rn(po, so), rho), fc);
  if (P.et) fc = fma(-__dmul_rn(vz, dt), __ldg(P.et + c), fc);
  // neighbours' scatter (reference loop order: plane k-1, row j-1, cell i-1)
  fc = fma(-dt, fl_z, fc);
  fc = fma(-dt, fl_y, fc);
  fc = fma(-dt, fl_x, fc);
  fc = fma(dt, u_right + u_front + u_upper, fc);
  if (VEL) {
    const long long fx1 = (long long)(P.nx + 1), cyz = (long long)P.nx * (P.ny + 1);
    if (V.vx && i + 1 < P.nx)
      V.vx[(i + 1) + fx1 * (j + (long long)P.ny * k)] = u_right / (P.dy * P.dz * zm * 1.0);
    if (V.vy && j + 1 < P.ny)
      V.vy[i + (long long)P.nx * (j + 1) + cyz * k] = u_front / (P.dx * P.dz * zm * 1.0);
    if (V.vz && k + 1 < P.nz) V.vz[c + sz] = u_upper / (P.dx * P.dy * 1.0 * 1.0);
  }

  // boundary patches (nl_function_eval.c:979-1435)
  if (i > 0 && i < P.nx - 1 && j > 0 && j < P.ny - 1 && k > 0 && k < P.nz - 1) {
    f[c] = fc;
    return;
  }
  const double ffx = P.dy * P.dz, ffy = P.dx * P.dz, ffz = P.dx * P.dy;
  const bool onf[6] = {i == 0, i == P.nx - 1, j == 0, j == P.ny - 1, k == 0, k == P.nz - 1};
#pragma unroll
  for (int face = 0; face < 6; face++) {
    if (!onf[face]) continue;
    const double value = __ldg(P.bc_val[face] + face_slot(P, face, i, j, k));
    const double dir = (face & 1) ? 1.0 : -1.0;
    double u_new;
    double vel = 0.0;  // this face's velocity (VEL)
    if (P.bc_type[face] == 0 || P.bc_type[face] == 5) {
      // FluxConst, or SeepageFace (nl_function_eval.c:1692-1784): a flux
      // face whose top face also drains the ponded water
      double q_ov = 0.0;
      if (P.bc_type[face] == 5 && face == 5) {
        q_ov = (vol / P.dz) * dt * (pmax0(pc) - 0.0);
        fc += q_ov;
      }
      double h = (face < 2) ? ffx * zm : (face < 4) ? ffy * zm : ffz;
      u_new = h * value;
      if (VEL) vel = (P.bc_type[face] == 0) ? value : (u_new + q_ov / dt) / h;
    } else if (SURF && P.bc_type[face] == 2) {
      // OverlandKinematic top face (nl_function_eval.c:1786-2000): ponding and
      // routing term, then the rain flux like FluxConst
      const OvCell o = ov_cell(P, i, j);
      double ke = -(o.sfx / (o.sq * o.n)) * pow(ov_press_x(P, p, i, j, o), (5.0 / 3.0));
      double kn = -(o.sfy / (o.sq * o.n)) * pow(ov_press_y(P, p, i, j, o), (5.0 / 3.0));
      double kw = 0.0, ks = 0.0;
      if (i > 0) {
        const OvCell ow = ov_cell(P, i - 1, j);
        kw = -(ow.sfx / (ow.sq * ow.n)) * pow(ov_press_x(P, p, i - 1, j, ow), (5.0 / 3.0));
      } else if (o.sfx > 0.0) {  // outflow through the lower x edge
        kw = -(o.sfx / (o.sq * o.n)) * pow(pmax0(pc), (5.0 / 3.0));
      }
      if (j > 0) {
        const OvCell os = ov_cell(P, i, j - 1);
        ks = -(os.sfy / (os.sq * os.n)) * pow(ov_press_y(P, p, i, j - 1, os), (5.0 / 3.0));
      } else if (o.sfy > 0.0) {  // outflow through the lower y edge
        ks = -(o.sfy / (o.sq * o.n)) * pow(pmax0(pc), (5.0 / 3.0));
      }
      const double q_ov = ponding(P, dt, vol, pc, po, ke - kw, kn - ks);
      fc += q_ov;
      u_new = ffz * value;
      if (VEL) {
        vel = (u_new + q_ov / dt) / ffz;
        if (V.qx) V.qx[i + (long long)P.nx * j] = ke;
        if (V.qy) V.qy[i + (long long)P.nx * j] = kn;
      }
    } else if (SURF && P.bc_type[face] == 4) {
      // OverlandFlow top face (nl_function_eval.c:1437-1690): each face flux
      // is the upwind part of the two columns' own fluxes, plus the spin-up
      // damping term; with OverlandFlowSpinUp the ponded head drains in
      // place of the ponding and routing term (:1659-1673)
      const double qw = ovf_q<true>(P, p, i - 1, j), qc = ovf_q<true>(P, p, i, j),
                   qe = ovf_q<true>(P, p, i + 1, j);
      const double kw = pmax0(qw) - pmax0(-qc), ke = pmax0(qc) - pmax0(-qe);
      const double qs = ovf_q<false>(P, p, i, j - 1), qm = ovf_q<false>(P, p, i, j),
                   qn = ovf_q<false>(P, p, i, j + 1);
      const double ks = pmax0(qs) - pmax0(-qm), kn = pmax0(qm) - pmax0(-qn);
      double q_ov = ponding(P, dt, vol, pc, po, ke - kw, kn - ks);
      if (P.ov_p2 != 0.0 || P.ov_spinup == 1) {
        const double damp = exp(fmin(pc, 0.0) * P.ov_p1) * P.ov_p2;
        q_ov = fma(vol * dt / P.dz, damp, q_ov);
        if (P.ov_spinup == 1) q_ov = (vol / P.dz) * dt * ((pmax0(pc) - 0.0) + damp);
      }
      fc += q_ov;
      u_new = ffz * value;
      if (VEL) {
        vel = (u_new + q_ov / dt) / ffz;
        if (V.qx) V.qx[i + (long long)P.nx * j] = ke;
        if (V.qy) V.qy[i + (long long)P.nx * j] = kn;
      }
    } else if (SURF && P.bc_type[face] == 3) {
      // OverlandDiffusive top face (nl_function_eval.c:2028-2259): the same
      // ponding and routing term with the diffusive-wave face fluxes
      const OvdCol o = ovd_col(P, p, i, j);
      double qxw, qys;
      ovd_q_edges(P, o, i, j, qxw, qys);
      const double ke = ovd_qx(o), kn = ovd_qy(o);
      const double kw = i > 0 ? ovd_qx(ovd_col(P, p, i - 1, j)) : qxw;
      const double ks = j > 0 ? ovd_qy(ovd_col(P, p, i, j - 1)) : qys;
      const double q_ov = ponding(P, dt, vol, pc, po, ke - kw, kn - ks);
      fc += q_ov;
      u_new = ffz * value;
      if (VEL) {
        vel = (u_new + q_ov / dt) / ffz;
        if (V.qx) V.qx[i + (long long)P.nx * j] = ke;
        if (V.qy) V.qy[i + (long long)P.nx * j] = kn;
      }
    } else {
      const VG v = vg_at(P, c);
      double krg = vg_kr(P, value, v.alpha, v.n);
      if (face < 4) {
        double h = (face < 2) ? ffx * zm : ffy * zm;
        double kk = __ldg((face < 2 ? P.kx : P.ky) + c);
        double dd = (face < 2) ? P.dx : P.dy;
        if (dir < 0) {
          double diff = value - pc;
          u_new = upstream(value, pc, krg * rho, krc * rho);
          u_new = u_new * h * (kk * P.inv_visc) * 2.0 * (diff / dd);
        } else {
          double diff = pc - value;
          u_new = upstream(pc, value, krc * rho, krg * rho);
          u_new = u_new * h * (kk * P.inv_visc) * 2.0 * (diff / dd);
        }
      } else {
        double sep = P.dz * zm;
        double lower, upper;
        if (dir < 0) {
          lower = value / sep - 0.25 * rho * g;
          upper = pc / sep + 0.25 * rho * g;
          u_new = upstream(lower, upper, krg * rho, krc * rho);
        } else {
          lower = (pc / sep) - 0.25 * rho * g * 1.0;
          upper = (value / sep) + 0.25 * rho * g * 1.0;
          u_new = upstream(lower, upper, krc * rho, krg * rho);
        }
        u_new = u_new * ffz * (__ldg(P.kz + c) * P.inv_visc) * 2.0 * (lower - upper);
      }
      // DirichletBC: u_new / h (nl_function_eval.c:1227-1230)
      if (VEL) vel = u_new / ((face < 2) ? ffx * zm : (face < 4) ? ffy * zm : ffz);
    }
    fc = fma(dt * dir, u_new, fc);
    if (VEL) {
      const int up = face & 1;
      if (face < 2 && V.vx)
        V.vx[(i + up) + (long long)(P.nx + 1) * (j + (long long)P.ny * k)] = vel;
      else if (face >= 2 && face < 4 && V.vy)
        V.vy[i + (long long)P.nx * (j + up) + (long long)P.nx * (P.ny + 1) * k] = vel;
      else if (face >= 4 && V.vz)
        V.vz[c + up * sz] = vel;
    }
  }
  f[c] = fc;
}

// Gather form: every cell evaluates all six of its face fluxes (a face shared
// by two cells is evaluated by both, with the same operands in the same
// order).
template <bool SURF, bool VEL = false>
__global__ void __launch_bounds__(256, 5) k_residual(DevProblem P, const double *__restrict__ p,
                           const double *__restrict__ p_old, const double *__restrict__ s_old,
                           const double *__restrict__ kr, const double *__restrict__ satv,
                           double dt, double *__restrict__ f, VelOut V = VelOut{}) {
  pdl_enter();
  if (P.dtp) dt = *P.dtp;
  int i, j, k;
  if (!launch_ijk(P.nx, P.ny, P.nz, i, j, k)) return;
  const long long c = i + (long long)P.nx * (j + (long long)P.ny * k);
  const long long sy = P.nx, sz = (long long)P.nx * P.ny;
  const double g = P.gravity;
  const FluxConst A = flux_const(P);
  const double zm = __ldg(P.zmult + k);
  const double pc = p[c];
  const double kxc = __ldg(P.kx + c), kyc = __ldg(P.ky + c), kzc = __ldg(P.kz + c);
  const double krc = kr[c];
  double fl_z = 0.0, fl_y = 0.0, fl_x = 0.0;
  if (k > 0) {
    long long l = c - sz;
    double zl = __ldg(P.zmult + k - 1);
    fl_z = flux_z(P, A.cz, p[l], pc, __ldg(P.kz + l), kzc, kr[l], krc, zl, zm, k - 1);
    if (P.fbz) fl_z = fl_z * fb_z(P, l);
  }
  double gs = 0.0, gc = g;
  if (j > 0) {
    long long s = c - sy;
    if (SURF) tfg_face_y(P, i, j - 1, gs, gc);
    fl_y = flux_xy(P.inv_dy, A.cy, p[s], pc, __ldg(P.ky + s), kyc, kr[s], krc, zm, gs, gc);
    if (P.fby) fl_y = fl_y * fb_y(P, s);
  }
  if (i > 0) {
    long long w = c - 1;
    if (SURF) tfg_face_x(P, i - 1, j, gs, gc);
    fl_x = flux_xy(P.inv_dx, A.cx, p[w], pc, __ldg(P.kx + w), kxc, kr[w], krc, zm, gs, gc);
    if (P.fbx) fl_x = fl_x * fb_x(P, w);
  }
  double u_right = 0.0, u_front = 0.0, u_upper = 0.0;
  if (i + 1 < P.nx) {
    long long e = c + 1;
    if (SURF) tfg_face_x(P, i, j, gs, gc);
    u_right = flux_xy(P.inv_dx, A.cx, pc, p[e], kxc, __ldg(P.kx + e), krc, kr[e], zm, gs, gc);
    if (P.fbx) u_right = u_right * fb_x(P, c);
  }
  if (j + 1 < P.ny) {
    long long nn = c + sy;
    if (SURF) tfg_face_y(P, i, j, gs, gc);
    u_front = flux_xy(P.inv_dy, A.cy, pc, p[nn], kyc, __ldg(P.ky + nn), krc, kr[nn], zm, gs, gc);
    if (P.fby) u_front = u_front * fb_y(P, c);
  }
  if (k + 1 < P.nz) {
    long long u = c + sz;
    u_upper = flux_z(P, A.cz, pc, p[u], kzc, __ldg(P.kz + u), krc, kr[u], zm,
                     __ldg(P.zmult + k + 1), k);
    if (P.fbz) u_upper = u_upper * fb_z(P, c);
  }
  residual_cell<SURF, VEL>(P, i, j, k, c, p, p_old, dt, f, V, pc, krc, satv[c], s_old[c],
                           p_old[c], zm, fl_z, fl_y, fl_x, u_right, u_front, u_upper);
}

// March form (one permeability field for the three directions, no face
// velocities): a warp owns 32 columns of a row and walks up through planes
// k0 .. k0 + kchunk - 1.  Lane l holds column i = 31 w + l - 1; it evaluates the
// east face of its column, which the next lane takes by a shuffle as its west
// face (lane 0 only provides), both y faces, and the upper z face, which stays
// in a register as the lower one of the next plane: four faces per cell instead
// of six and half the loads, with no barrier and no shared memory.  Every flux
// is the same function of the same operands as in the gather form.
// Bound by instruction issue (62 % of the slots, 368 instructions per cell) and
// the latency its occupancy leaves: the four faces are evaluated without a branch
// between them and an inner cell meets one test for the boundary patches.
// 512x512x50: 211 us, gather form 295 (memory floor 114 us, 56 B per cell).
// Four blocks of 64 registers per SM: with the van Genuchten pass, 197x123x37
// 33.9 us; three 36.8, five 41.4.  With the slopes of a terrain-following grid,
// which need more registers, three give 52.5 us at 256x256x20, four 57.2, gather
// 67.2.  Two rows per warp (3.6 faces per cell, 96 registers) were slower than
// gather: 20 warps per SM hide too little.

// a column's value of one plane
struct MCell {
  double p, k, kr;
};
__device__ __forceinline__ MCell mcell(const DevProblem &P, const double *__restrict__ p,
                                       const double *__restrict__ kr, int c) {
  return MCell{p[c], __ldg(P.kx + c), kr[c]};
}

template <bool SURF>
__global__ void __launch_bounds__(32 * MARCH_WARPS, SURF ? 3 : 4) k_residual_march(
    DevProblem P, const double *__restrict__ p, const double *__restrict__ p_old,
    const double *__restrict__ s_old, const double *__restrict__ kr,
    const double *__restrict__ satv, double dt, double *__restrict__ f, int kchunk) {
  pdl_enter();
  if (P.dtp) dt = *P.dtp;
  const int lane = threadIdx.x, nx = P.nx, ny = P.ny, nz = P.nz;
  const int j = blockIdx.y * MARCH_WARPS + threadIdx.y;
  if (j >= ny) return;
  const int i = blockIdx.x * MARCH_COLS + lane - 1;
  const int k0 = blockIdx.z * kchunk, k1 = min(nz, k0 + kchunk);
  const bool in = i >= 0 && i < nx, out = in && lane > 0, east = in && i + 1 < nx;
  const bool south = j > 0, north = j + 1 < ny;
  const int ii = in ? i : (i < 0 ? 0 : nx - 1), sz = nx * ny;
  const FluxConst A = flux_const(P);
  const VelOut V{};
  const bool barriers = P.fbx || P.fby || P.fbz;
  // gravity terms of the column's faces (constant through the planes)
  double gse = 0.0, gce = P.gravity, gss = 0.0, gcs = P.gravity, gsn = 0.0, gcn = P.gravity;
  if (SURF) {
    if (east) tfg_face_x(P, ii, j, gse, gce);
    if (south) tfg_face_y(P, ii, j - 1, gss, gcs);
    if (north) tfg_face_y(P, ii, j, gsn, gcn);
  }
  int c = ii + nx * (j + ny * k0);
  MCell q = mcell(P, p, kr, c);
  double lz = 0.0, zm = __ldg(P.zmult + k0);
  if (k0 > 0) {
    const MCell a = mcell(P, p, kr, c - sz);
    lz = flux_z(P, A.cz, a.p, q.p, a.k, q.k, a.kr, q.kr, __ldg(P.zmult + k0 - 1), zm, k0 - 1);
    if (P.fbz) lz = lz * fb_z(P, c - sz);
  }
  for (int k = k0; k < k1; k++, c += sz) {
    const bool up = k + 1 < nz;
    const double zu = up ? __ldg(P.zmult + k + 1) : zm;
    // every operand first
    const MCell n = mcell(P, p, kr, up ? c + sz : c);
    const MCell e = mcell(P, p, kr, east ? c + 1 : c);
    const MCell s = mcell(P, p, kr, south ? c - nx : c);
    const MCell t = mcell(P, p, kr, north ? c + nx : c);
    const double sat = satv[c], so = s_old[c], po = p_old[c];
    // the four faces side by side, without a branch: one that does not exist
    // is evaluated against the cell itself and dropped
    const Mean mx = mean_xy(q.k, e.k), ms = mean_xy(s.k, q.k), mn = mean_xy(q.k, t.k),
               mz = mean_z(q.k, n.k, zm, zu);
    double kx = mx.near(), ks = ms.near(), kn = mn.near(), kz = mz.near();
    if (mx.far() | ms.far() | mn.far() | mz.far()) {
      kx = mx.value();
      ks = ms.value();
      kn = mn.value();
      kz = mz.value();
    }
    double ux = flux_xy_km(P.inv_dx, A.cx, kx, q.p, e.p, q.kr, e.kr, zm, gse, gce);
    double us = flux_xy_km(P.inv_dy, A.cy, ks, s.p, q.p, s.kr, q.kr, zm, gss, gcs);
    double un = flux_xy_km(P.inv_dy, A.cy, kn, q.p, t.p, q.kr, t.kr, zm, gsn, gcn);
    double uz = flux_z_km(P, A.cz, kz, q.p, n.p, q.kr, n.kr, k);
    if (barriers) {
      if (P.fbx) ux = ux * fb_x(P, c);
      if (P.fby) {
        if (south) us = us * fb_y(P, c - nx);
        un = un * fb_y(P, c);
      }
      if (P.fbz) uz = uz * fb_z(P, c);
    }
    ux = east ? ux : 0.0;
    us = south ? us : 0.0;
    un = north ? un : 0.0;
    uz = up ? uz : 0.0;
    const double wx = __shfl_up_sync(0xffffffffu, ux, 1);
    if (out)
      residual_cell<SURF, false>(P, i, j, k, c, p, p_old, dt, f, V, q.p, q.kr, sat, so, po, zm, lz,
                                 us, i > 0 ? wx : 0.0, ux, un, uz);
    lz = uz;
    q = n;
    zm = zu;
  }
}

// Flux derivatives of one x (or y) face between a (left) and b (right)
// (richards_jacobian_eval.c:618-660): returns west/east and symmetric parts.
// TA is the arithmetic of the face terms: double for the FP64 Jacobian; for
// a Jacobian stored in FP32 the face terms are formed in FP32 too (their
// products round no worse than the storage), while the upwind decisions, the
// pressure differences they come from and the row sums stay FP64.
template <typename TA>
struct FaceDer {
  TA lo, hi, sym;  // d/dp of the face flux w.r.t. lower cell (negated), upper cell; sym part
};

__device__ __forceinline__ float mul_rn_t(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn_t(double a, double b) { return __dmul_rn(a, b); }
// Mean in the face arithmetic
template <typename TA>
struct MeanT {
  TA num, den;
  __device__ __forceinline__ TA near() const { return quotient_near(num, den); }
  __device__ __forceinline__ bool far() const { return rcp_far(den); }
  __device__ __forceinline__ TA value() const {
    return far() ? (den ? num / den : TA(0)) : near();
  }
};
template <typename TA>
__device__ __forceinline__ MeanT<TA> mean_xy_t(TA a, TA b) {
  return MeanT<TA>{mul_rn_t(mul_rn_t(TA(2), a), b), a + b};
}
template <typename TA>
__device__ __forceinline__ MeanT<TA> mean_z_t(TA a, TA b, TA c, TA d) {
  return MeanT<TA>{mul_rn_t(mul_rn_t(c + d, a), b), fma(b, c, mul_rn_t(a, d))};
}
template <typename TA>
__device__ __forceinline__ TA harmonic_t(TA a, TA b) {
  return mean_xy_t(a, b).value();
}
template <typename TA>
__device__ __forceinline__ TA harmonic_dz_t(TA a, TA b, TA c, TA d) {
  return mean_z_t(a, b, c, d).value();
}

// What a face term needs of a cell: the pressure in FP64 (its differences take
// the upwind decision), K, kr rho and dkr rho in the face arithmetic,
// converted once per cell
template <typename TA>
struct JCell {
  double p;
  TA k, prod, prod_der;
};
template <typename TA>
__device__ __forceinline__ JCell<TA> jcell(const double *__restrict__ p, const double *kk,
                                           const double *__restrict__ kr,
                                           const double *__restrict__ dkr, double rho,
                                           long long c) {
  return JCell<TA>{p[c], (TA)__ldg(kk + c), (TA)(kr[c] * rho), (TA)(dkr[c] * rho)};
}
// constants of the x / y faces: area dt / (spacing viscosity), and the
// spacing and its reciprocal
template <typename TA>
struct JFace {
  TA c, d;
  double inv_d;
};

// x_coeff / y_coeff (richards_jacobian_eval.c:662, 692): FB * dt * ...; the
// upwinded terms of the reference's macros with their common factors formed once
template <typename TA>
__device__ __forceinline__ FaceDer<TA> face_der_xy(const JFace<TA> &F, double fb, TA km,
                                                   const JCell<TA> &a, const JCell<TA> &b,
                                                   TA zm, double dir_g, double dir_g_c) {
  const double diff64 = a.p - b.p;
  const bool lower = ((diff64 * F.inv_d) * dir_g_c - dir_g) >= 0.0;  // flow from a to b
  const TA diff = (TA)diff64, dgc = (TA)dir_g_c, dg = (TA)dir_g;
  const TA coeff = mul_rn_t(mul_rn_t(mul_rn_t((TA)fb, F.c), zm), km);
  // derivative of the upwind cell's mobility times the driving difference
  const TA drive = mul_rn_t(coeff, fma(diff, dgc, -mul_rn_t(F.d, dg)));
  const TA sym = mul_rn_t(mul_rn_t(-coeff, lower ? a.prod : b.prod), dgc);
  FaceDer<TA> r;
  r.sym = sym;
  r.lo = lower ? fma(-drive, a.prod_der, sym) : sym;
  r.hi = lower ? sym : fma(drive, b.prod_der, sym);
  return r;
}

// z face between a (lower) and b (upper) (richards_jacobian_eval.c:697-745);
// the terms with the density's derivative are zero (constant density)
template <typename TA>
__device__ __forceinline__ FaceDer<TA> face_der_z(const DevProblem &P, TA cz, double fb, TA km,
                                                  const JCell<TA> &a, const JCell<TA> &b,
                                                  int k) {
  const double rg = P.density * P.gravity;
  const double inv_sep = __ldg(P.zface + 3 * k);
  const double lower_cond = fma(a.p, inv_sep, -__dmul_rn(__ldg(P.zface + 3 * k + 1), rg));
  const double upper_cond = fma(b.p, inv_sep, __dmul_rn(__ldg(P.zface + 3 * k + 2), rg));
  const double diff64 = lower_cond - upper_cond;
  const bool lower = diff64 >= 0.0;
  const TA coeff = mul_rn_t(mul_rn_t((TA)fb, cz), km);
  const TA drive = mul_rn_t(coeff, (TA)diff64);
  const TA sym = mul_rn_t(mul_rn_t(-coeff, (TA)inv_sep), lower ? a.prod : b.prod);
  FaceDer<TA> r;
  r.sym = sym;
  r.lo = lower ? fma(-drive, a.prod_der, sym) : sym;
  r.hi = lower ? sym : fma(drive, b.prod_der, sym);
  return r;
}

// Jacobian assembly (richards_jacobian_eval.c:217-1420).  Writes the full
// 7-point J (C W E S N L U, FP64 or FP32) and the symmetric preconditioner
// matrix (C E N U: full diagonal, symmetric off-diagonal parts; PCMatrixType
// PFSymmetric), in the preconditioner's precision.
//
// jacobian_cell is everything of one cell's row but the interior face
// derivatives, which the caller supplies: the lower z / y / x faces' (lo, hi)
// parts (used where k, j, i > 0) and the cell's own upper faces (zero on the
// domain's upper faces).  Both launch forms below pass the values of the
// same face functions with the same operands, so their J and PC matrix are
// equal bit for bit.
template <typename TA>
struct FaceLH {
  TA lo, hi;
};

template <typename TJ, typename TP, bool SURF>
__device__ __forceinline__ void jacobian_cell(const DevProblem &P, int i, int j, int k,
                                              long long c, const double *__restrict__ p,
                                              const double *__restrict__ kr,
                                              const double *__restrict__ dkr, double dt,
                                              const JacOut<TJ> &J, const PCOut<TP> &M,
                                              double pc, double sat, double dsat, double zm,
                                              FaceLH<TJ> dl_z, FaceLH<TJ> dl_y, FaceLH<TJ> dl_x,
                                              const FaceDer<TJ> &de, const FaceDer<TJ> &dn,
                                              const FaceDer<TJ> &du) {
  const long long sy = P.nx;
  const double rho = P.density, g = P.gravity, drho = 0.0;
  const double vol = P.dx * P.dy * P.dz;
  const double ffx = P.dy * P.dz, ffy = P.dx * P.dz, ffz = P.dx * P.dy;

  double vol2 = vol * zm;
  double cp = 0.0;
  cp += (dsat * rho + sat * drho) * P.porosity * vol2 +
        P.sstorage * vol2 * (dsat * rho * pc + sat * drho * pc + sat * rho);

  double w = 0.0, s = 0.0, l = 0.0, e = 0.0, nn = 0.0, u = 0.0;
  double es = 0.0, ns = 0.0, us = 0.0;
  if (k > 0) {
    cp += -dl_z.hi;
    l = dl_z.lo;
  }
  if (j > 0) {
    cp += -dl_y.hi;
    s = dl_y.lo;
  }
  if (i > 0) {
    cp += -dl_x.hi;
    w = dl_x.lo;
  }
  double west_t = 0.0, south_t = 0.0, lower_t = 0.0;
  if (i + 1 < P.nx) {
    west_t = de.lo;
    e = de.hi;
    es = de.sym;
  }
  if (j + 1 < P.ny) {
    south_t = dn.lo;
    nn = dn.hi;
    ns = dn.sym;
  }
  if (k + 1 < P.nz) {
    lower_t = du.lo;
    u = du.hi;
    us = du.sym;
  }
  cp += -(west_t + south_t + lower_t);

  // Dirichlet patches (richards_jacobian_eval.c:1049-1200); flux patches
  // leave the row as is (their boundary entries are zero)
  const bool onf[6] = {i == 0, i == P.nx - 1, j == 0, j == P.ny - 1, k == 0, k == P.nz - 1};
  if (onf[0] || onf[1] || onf[2] || onf[3] || onf[4] || onf[5])
#pragma unroll
  for (int face = 0; face < 6; face++) {
    if (!onf[face] || P.bc_type[face] != 1) continue;
    const double value = __ldg(P.bc_val[face] + face_slot(P, face, i, j, k));
    const double den_d = rho;
    const double prod = kr[c] * rho, prod_der = dkr[c] * rho + kr[c] * drho;
    const double kxc = __ldg(P.kx + c), kyc = __ldg(P.ky + c), kzc = __ldg(P.kz + c);
    const VG v = vg_at(P, c);
    const double prod_val = vg_kr(P, value, v.alpha, v.n) * den_d;
    // above the top layer the z_mult ghost keeps the 1 it was initialised
    // with (problem_dz_scale.c:92)
    const double zu = (k + 1 < P.nz) ? __ldg(P.zmult + k + 1) : 1.0;
    double coeff, diff, o_temp;
    switch (face) {
      case 0:
        coeff = dt * ffx * zm * (2.0 / P.dx) * kxc * P.inv_visc;
        diff = value - pc;
        o_temp = coeff * (diff * upstream(value, pc, 0.0, prod_der) -
                          upstream(value, pc, prod_val, prod));
        break;
      case 1:
        coeff = dt * ffx * zm * (2.0 / P.dx) * kxc * P.inv_visc;
        diff = pc - value;
        o_temp = -coeff * (diff * upstream(pc, value, prod_der, 0.0) +
                           upstream(pc, value, prod, prod_val));
        break;
      case 2:
        coeff = dt * ffy * zm * (2.0 / P.dy) * kyc * P.inv_visc;
        diff = value - pc;
        o_temp = coeff * (diff * upstream(value, pc, 0.0, prod_der) -
                          upstream(value, pc, prod_val, prod));
        break;
      case 3:
        coeff = dt * ffy * zm * (2.0 / P.dy) * kyc * P.inv_visc;
        diff = pc - value;
        o_temp = -coeff * (diff * upstream(pc, value, prod_der, 0.0) +
                           upstream(pc, value, prod, prod_val));
        break;
      case 4: {
        coeff = dt * ffz * (2.0 / (P.dz * amean(zm, zu))) * kzc * P.inv_visc;
        double lc = (value)-0.5 * P.dz * zm * den_d * g;
        double uc = (pc) + 0.5 * P.dz * zm * rho * g;
        diff = lc - uc;
        o_temp = coeff * (diff * upstream(lc, uc, 0.0, prod_der) +
                          ((-1.0 - g * 0.5 * P.dz * zm * drho) * upstream(lc, uc, prod_val, prod)));
        break;
      }
      default: {
        coeff = dt * ffz * (2.0 / (P.dz * amean(zm, zu))) * kzc * P.inv_visc;
        double lc = (pc)-0.5 * P.dz * zm * rho * g;
        double uc = (value) + 0.5 * P.dz * zm * den_d * g;
        diff = lc - uc;
        o_temp = -coeff * (diff * upstream(lc, uc, prod_der, 0.0) +
                           ((1.0 - g * 0.5 * P.dz * zm * drho) * upstream(lc, uc, prod, prod_val)));
        break;
      }
    }
    cp -= o_temp;
  }

  // SeepageFace on the top face (richards_jacobian_eval.c:1319-1345), in
  // patch order after the Dirichlet corrections
  if (k == P.nz - 1 && P.bc_type[5] == 5 && pc >= 0.0) cp += (vol / P.dz) * dt * (1.0 + 0.0);

  // kinematic overland terms of a top cell, MGSemi form
  // (richards_jacobian_eval.c:1863-1990, CALCDER of overlandflow_eval_Kin.c),
  // added after every other term.  In the symmetric storage the west / south
  // terms belong to the neighbour's E / N entry (lower coefficient aliasing,
  // matrix.c:484-490): E(i) gets this cell's east term, then the east
  // neighbour's west term, in the reference's loop order.
  // difference-quotient mode: an OverlandFlow top cell with p > 0 gets
  // vol zm / (dz mean(zm, 1)) (dt + 1), the z_mult ghost above the top layer
  // keeping its initial 1 (problem_dz_scale.c:92), and no surface terms
  if (M.fd && k == P.nz - 1 && P.bc_type[5] == 4 && pc > 0.0)
    cp += (vol * zm) / (P.dz * (0.5 * (zm + 1.0))) * (dt + 1);
  if (SURF && !M.fd && k == P.nz - 1 && P.bc_type[5] == 2) {
    const double cx = (vol / ffy) * dt, cy = (vol / ffx) * dt;
    const double two3 = 2.0 / 3.0;
    const OvCell o = ov_cell(P, i, j);
    const double qxt = -(5.0 / 3.0) * (o.sfx / (o.sq * o.n)) * pow(ov_press_x(P, p, i, j, o), two3);
    const double qyt = -(5.0 / 3.0) * (o.sfy / (o.sq * o.n)) * pow(ov_press_y(P, p, i, j, o), two3);
    const double ke_d = pmax0(qxt), kn_d = pmax0(qyt);
    double kw_d = 0.0, ks_d = 0.0, ke_w = 0.0, kn_s = 0.0;
    if (i > 0) {
      const OvCell ow = ov_cell(P, i - 1, j);
      const double q = -(5.0 / 3.0) * (ow.sfx / (ow.sq * ow.n)) *
                       pow(ov_press_x(P, p, i - 1, j, ow), two3);
      kw_d = -pmax0(-q);
      ke_w = pmax0(q);
    } else if (o.sfx > 0.0) {
      const double q = -(5.0 / 3.0) * (o.sfx / (o.sq * o.n)) * pow(pmax0(pc), two3);
      kw_d = -pmax0(-q);
      ke_w = pmax0(q);
    }
    if (j > 0) {
      const OvCell os = ov_cell(P, i, j - 1);
      const double q = -(5.0 / 3.0) * (os.sfy / (os.sq * os.n)) *
                       pow(ov_press_y(P, p, i, j - 1, os), two3);
      ks_d = -pmax0(-q);
      kn_s = pmax0(q);
    } else if (o.sfy > 0.0) {
      const double q = -(5.0 / 3.0) * (o.sfy / (o.sq * o.n)) * pow(pmax0(pc), two3);
      ks_d = -pmax0(-q);
      kn_s = pmax0(q);
    }
    if (pc > 0.0)
      cp += (vol / P.dz) + cx * (ke_d - kw_d) + cy * (kn_d - ks_d);
    const double tw = cx * (ke_w), te = cx * (-pmax0(-qxt));
    const double ts = cy * (kn_s), tn = cy * (-pmax0(-qyt));
    w -= tw;
    e += te;
    s -= ts;
    nn += tn;
    es += te;
    if (i + 1 < P.nx) es -= cx * (ke_d);  // the east neighbour's west term
    ns += tn;
    if (j + 1 < P.ny) ns -= cy * (kn_d);  // the north neighbour's south term
  }
  // OverlandFlow terms of a top cell, MGSemi form
  // (richards_jacobian_eval.c:2028-2090, CALCDER of overlandflow_eval.c):
  // the derivative parts of each column's own flux; neighbours' parts give
  // the off-diagonals, and the east neighbour's west term lands in E(i)
  // With OverlandFlowSpinUp the patch's own diagonal term of a cell with
  // p >= 0 comes first (richards_jacobian_eval.c:1258-1268) and the
  // derivative parts are zero (their evaluation is skipped, :1287); a
  // non-ponded cell gets the derivative of the spin-up damping term.
  if (SURF && !M.fd && k == P.nz - 1 && P.bc_type[5] == 4) {
    const bool spin = P.ov_spinup == 1;
    if (spin && pc >= 0.0) cp += (vol / P.dz) * dt * (1.0 + 0.0);
    const double cx = (vol / ffy) * dt, cy = (vol / ffx) * dt;
    const double qx = spin ? 0.0 : ovf_qder<true>(P, pc, i, j);
    const double qy = spin ? 0.0 : ovf_qder<false>(P, pc, i, j);
    const double ke_d = pmax0(qx), kw_d = -pmax0(-qx);
    const double kn_d = pmax0(qy), ks_d = -pmax0(-qy);
    // the neighbours' derivative parts: ke of i-1, kw of i+1, kn of j-1, ks of j+1
    const double ke_w = i > 0 && !spin ? pmax0(ovf_qder<true>(P, p[c - 1], i - 1, j)) : 0.0;
    const double kw_e =
        i + 1 < P.nx && !spin ? -pmax0(-ovf_qder<true>(P, p[c + 1], i + 1, j)) : 0.0;
    const double kn_s = j > 0 && !spin ? pmax0(ovf_qder<false>(P, p[c - sy], i, j - 1)) : 0.0;
    const double ks_n =
        j + 1 < P.ny && !spin ? -pmax0(-ovf_qder<false>(P, p[c + sy], i, j + 1)) : 0.0;
    if (pc > 0.0)
      cp += (vol / P.dz) + cx * (ke_d - kw_d) + cy * (kn_d - ks_d);
    else
      cp += 0.0 + dt * (vol / P.dz) * (P.ov_p1 * exp(fmin(pc, 0.0) * P.ov_p1) * P.ov_p2);
    const double tw = cx * (ke_w), te = cx * (kw_e);
    const double ts = cy * (kn_s), tn = cy * (ks_n);
    w -= tw;
    e += te;
    s -= ts;
    nn += tn;
    es += te;
    if (i + 1 < P.nx) es -= cx * (ke_d);  // the east neighbour's west term
    ns += tn;
    if (j + 1 < P.ny) ns -= cy * (kn_d);  // the north neighbour's south term
  }
  // diffusive overland terms of a top cell, MGSemi form
  // (richards_jacobian_eval.c:1989-2026, CALCDER of
  // overlandflow_eval_diffusive.c): off-diagonals from the non-symmetric
  // derivative parts.  In the symmetric storage the west term of an i = 0
  // cell lands in the x_lower ghost column of E, which MGSemi's setup reads:
  // it is returned in wgv for the multigrid's ghost plane.
  double wgv = 0.0;
  if (SURF && !M.fd && k == P.nz - 1 && P.bc_type[5] == 3) {
    const double cx = (vol / ffy) * dt, cy = (vol / ffx) * dt;
    const OvdCol o = ovd_col(P, p, i, j);
    double ke_d, kens, kn_d, knns;
    ovd_der_x(P, o, ke_d, kens);
    ovd_der_y(P, o, kn_d, knns);
    double kw_d = 0.0, kwns = 0.0, ks_d = 0.0, ksns = 0.0;
    ovd_der_edges(P, o, i, j, kw_d, kwns, ks_d, ksns);
    if (i > 0) ovd_der_x(P, ovd_col(P, p, i - 1, j), kwns, kw_d);
    if (j > 0) ovd_der_y(P, ovd_col(P, p, i, j - 1), ksns, ks_d);
    if (pc > 0.0)
      cp += (vol / P.dz) + cx * (ke_d - kw_d) + cy * (kn_d - ks_d);
    const double tw = cx * (kwns), te = cx * (kens);
    const double ts = cy * (ksns), tn = cy * (knns);
    w -= tw;
    e += te;
    s -= ts;
    nn += tn;
    if (i == 0) wgv -= tw;
    es += te;
    if (i + 1 < P.nx) es -= cx * (ke_d);  // the east neighbour's west term
    ns += tn;
    if (j + 1 < P.ny) ns -= cy * (kn_d);  // the north neighbour's south term
  }
  if (J.c) {
    J.c[c] = (TJ)cp;
    J.w[c] = (TJ)w;
    J.e[c] = (TJ)e;
    J.s[c] = (TJ)s;
    J.n[c] = (TJ)nn;
    J.l[c] = (TJ)l;
    J.u[c] = (TJ)u;
  }
  if (M.c) {
    M.c[c] = (TP)cp;
    M.e[c] = (TP)es;
    M.n[c] = (TP)ns;
    M.u[c] = (TP)us;
    if (M.wg && i == 0) M.wg[j + (long long)P.ny * k] = (TP)wgv;
  }
}

template <typename TA>
struct JConst {
  JFace<TA> x, y;
  TA cz;
  __device__ __forceinline__ JConst(const DevProblem &P, double dt) {
    const TA q = (TA)dt * (TA)P.inv_visc;
    x = JFace<TA>{q * (TA)(P.dy * P.dz) * (TA)P.inv_dx, (TA)P.dx, P.inv_dx};
    y = JFace<TA>{q * (TA)(P.dx * P.dz) * (TA)P.inv_dy, (TA)P.dy, P.inv_dy};
    cz = q * ((TA)P.dx * (TA)P.dy);
  }
};

// Gather form: every cell evaluates the derivative parts of all six of its
// faces.
template <typename TJ, typename TP, bool SURF>
__global__ void __launch_bounds__(128, 8) k_jacobian(DevProblem P, const double *__restrict__ p,
                           const double *__restrict__ kr, const double *__restrict__ dkr,
                           const double *__restrict__ satv, const double *__restrict__ dsatv,
                           double dt, JacOut<TJ> J, PCOut<TP> M) {
  pdl_enter();
  if (P.dtp) dt = *P.dtp;
  using TA = TJ;  // arithmetic of the face terms (see face_der_xy)
  int i, j, k;
  if (!launch_ijk(P.nx, P.ny, P.nz, i, j, k)) return;
  const long long c = i + (long long)P.nx * (j + (long long)P.ny * k);
  const long long sy = P.nx, sz = (long long)P.nx * P.ny;
  const double rho = P.density, g = P.gravity;
  const JConst<TA> A(P, dt);
  const double zm = __ldg(P.zmult + k);
  const JCell<TA> q = jcell<TA>(p, P.kx, kr, dkr, rho, c);
  const TA kyc = P.ky == P.kx ? q.k : (TA)__ldg(P.ky + c);
  const TA kzc = P.kz == P.kx ? q.k : (TA)__ldg(P.kz + c);
  const JCell<TA> qy{q.p, kyc, q.prod, q.prod_der}, qz{q.p, kzc, q.prod, q.prod_der};
  FaceLH<TA> dl_z{}, dl_y{}, dl_x{};
  FaceDer<TA> de{}, dn{}, du{};
  if (k > 0) {
    const JCell<TA> o = jcell<TA>(p, P.kz, kr, dkr, rho, c - sz);
    const double zl = __ldg(P.zmult + k - 1);
    const FaceDer<TA> d = face_der_z<TA>(P, A.cz, fb_z(P, c - sz),
                                         harmonic_dz_t<TA>(o.k, qz.k, (TA)zl, (TA)zm), o, qz,
                                         k - 1);
    dl_z = {d.lo, d.hi};
  }
  double gs = 0.0, gc = g;
  if (j > 0) {
    if (SURF) tfg_face_y(P, i, j - 1, gs, gc);
    const JCell<TA> o = jcell<TA>(p, P.ky, kr, dkr, rho, c - sy);
    const FaceDer<TA> d = face_der_xy<TA>(A.y, fb_y(P, c - sy), harmonic_t<TA>(o.k, qy.k), o, qy,
                                          (TA)zm, gs, gc);
    dl_y = {d.lo, d.hi};
  }
  if (i > 0) {
    if (SURF) tfg_face_x(P, i - 1, j, gs, gc);
    const JCell<TA> o = jcell<TA>(p, P.kx, kr, dkr, rho, c - 1);
    const FaceDer<TA> d = face_der_xy<TA>(A.x, fb_x(P, c - 1), harmonic_t<TA>(o.k, q.k), o, q,
                                          (TA)zm, gs, gc);
    dl_x = {d.lo, d.hi};
  }
  if (i + 1 < P.nx) {
    if (SURF) tfg_face_x(P, i, j, gs, gc);
    const JCell<TA> o = jcell<TA>(p, P.kx, kr, dkr, rho, c + 1);
    de = face_der_xy<TA>(A.x, fb_x(P, c), harmonic_t<TA>(q.k, o.k), q, o, (TA)zm, gs, gc);
  }
  if (j + 1 < P.ny) {
    if (SURF) tfg_face_y(P, i, j, gs, gc);
    const JCell<TA> o = jcell<TA>(p, P.ky, kr, dkr, rho, c + sy);
    dn = face_der_xy<TA>(A.y, fb_y(P, c), harmonic_t<TA>(qy.k, o.k), qy, o, (TA)zm, gs, gc);
  }
  if (k + 1 < P.nz) {
    const JCell<TA> o = jcell<TA>(p, P.kz, kr, dkr, rho, c + sz);
    const double zu = __ldg(P.zmult + k + 1);
    du = face_der_z<TA>(P, A.cz, fb_z(P, c), harmonic_dz_t<TA>(qz.k, o.k, (TA)zm, (TA)zu), qz, o,
                        k);
  }
  jacobian_cell<TJ, TP, SURF>(P, i, j, k, c, p, kr, dkr, dt, J, M, q.p, satv[c], dsatv[c], zm,
                              dl_z, dl_y, dl_x, de, dn, du);
}

// March form (as k_residual_march): a face's (lo, hi) parts go to the lane of
// the next column by shuffles and to the next plane in registers.
// The gather form converts every operand of every face to the face arithmetic
// (103 conversions and reciprocals per cell on a pipe of 16 lanes), this one a
// cell's values once per thread that needs them, and evaluates the four faces
// without a branch between them.  512x512x50, FP32: 293 us against 439, FP64 474
// against 519.  Blocks per SM in FP64, with the van Genuchten pass: three (80
// registers) 512x512x50 640 us and 24x500x50 34.2; two (128) 622 and 41.1, whose
// smaller waves leave more of the last one empty (2 % slower over 122 shapes).
template <typename TJ, typename TP, bool SURF>
__global__ void __launch_bounds__(32 * MARCH_WARPS, sizeof(TJ) == 8 || SURF ? 3 : 4)
    k_jacobian_march(
    DevProblem P, const double *__restrict__ p, const double *__restrict__ kr,
    const double *__restrict__ dkr, const double *__restrict__ satv,
    const double *__restrict__ dsatv, double dt, JacOut<TJ> J, PCOut<TP> M, int kchunk) {
  using TA = TJ;
  pdl_enter();
  if (P.dtp) dt = *P.dtp;
  const int lane = threadIdx.x, nx = P.nx, ny = P.ny, nz = P.nz;
  const int j = blockIdx.y * MARCH_WARPS + threadIdx.y;
  if (j >= ny) return;
  const int i = blockIdx.x * MARCH_COLS + lane - 1;
  const int k0 = blockIdx.z * kchunk, k1 = min(nz, k0 + kchunk);
  const bool in = i >= 0 && i < nx, out = in && lane > 0, east = in && i + 1 < nx;
  const bool south = j > 0, north = j + 1 < ny;
  const int ii = in ? i : (i < 0 ? 0 : nx - 1), sz = nx * ny;
  const double rho = P.density;
  const JConst<TA> A(P, dt);
  double gse = 0.0, gce = P.gravity, gss = 0.0, gcs = P.gravity, gsn = 0.0, gcn = P.gravity;
  if (SURF) {
    if (east) tfg_face_x(P, ii, j, gse, gce);
    if (south) tfg_face_y(P, ii, j - 1, gss, gcs);
    if (north) tfg_face_y(P, ii, j, gsn, gcn);
  }
  int c = ii + nx * (j + ny * k0);
  const bool barriers = P.fbx || P.fby || P.fbz;
  auto cell = [&](int q) { return jcell<TA>(p, P.kx, kr, dkr, rho, q); };
  JCell<TA> q = cell(c);
  FaceLH<TA> lz = {};
  double zm = __ldg(P.zmult + k0);
  if (k0 > 0) {
    const JCell<TA> o = cell(c - sz);
    const double zl = __ldg(P.zmult + k0 - 1);
    const FaceDer<TA> d = face_der_z<TA>(P, A.cz, fb_z(P, c - sz),
                                         harmonic_dz_t<TA>(o.k, q.k, (TA)zl, (TA)zm), o, q, k0 - 1);
    lz = {d.lo, d.hi};
  }
  for (int k = k0; k < k1; k++, c += sz) {
    const bool up = k + 1 < nz;
    const double zu = up ? __ldg(P.zmult + k + 1) : zm;
    const JCell<TA> n = cell(up ? c + sz : c), e = cell(east ? c + 1 : c);
    const JCell<TA> s = cell(south ? c - nx : c), t = cell(north ? c + nx : c);
    const double sat = satv[c], dsat = dsatv[c];
    // the four faces side by side (as in k_residual_march)
    const MeanT<TA> mx = mean_xy_t<TA>(q.k, e.k), ms = mean_xy_t<TA>(s.k, q.k),
                    mn = mean_xy_t<TA>(q.k, t.k), mz = mean_z_t<TA>(q.k, n.k, (TA)zm, (TA)zu);
    TA kx = mx.near(), ks = ms.near(), kn = mn.near(), kz = mz.near();
    if (mx.far() | ms.far() | mn.far() | mz.far()) {
      kx = mx.value();
      ks = ms.value();
      kn = mn.value();
      kz = mz.value();
    }
    double bx = 1.0, bs = 1.0, bn = 1.0, bz = 1.0;
    if (barriers) {
      bx = fb_x(P, c);
      if (south) bs = fb_y(P, c - nx);
      bn = fb_y(P, c);
      bz = fb_z(P, c);
    }
    FaceDer<TA> dx = face_der_xy<TA>(A.x, bx, kx, q, e, (TA)zm, gse, gce);
    const FaceDer<TA> ds = face_der_xy<TA>(A.y, bs, ks, s, q, (TA)zm, gss, gcs);
    FaceDer<TA> dn = face_der_xy<TA>(A.y, bn, kn, q, t, (TA)zm, gsn, gcn);
    FaceDer<TA> dz = face_der_z<TA>(P, A.cz, bz, kz, q, n, k);
    if (!east) dx = FaceDer<TA>{};
    if (!north) dn = FaceDer<TA>{};
    if (!up) dz = FaceDer<TA>{};
    const FaceLH<TA> dsl = south ? FaceLH<TA>{ds.lo, ds.hi} : FaceLH<TA>{};
    FaceLH<TA> wx;
    wx.lo = __shfl_up_sync(0xffffffffu, dx.lo, 1);
    wx.hi = __shfl_up_sync(0xffffffffu, dx.hi, 1);
    if (out)
      jacobian_cell<TJ, TP, SURF>(P, i, j, k, c, p, kr, dkr, dt, J, M, q.p, sat, dsat, zm, lz, dsl,
                                  wx, dx, dn, dz);
    lz = {dz.lo, dz.hi};
    q = n;
    zm = zu;
  }
}

// y = J x (matvec.c:35-330 order: y = 0, then C W E S N L U), FP64 accumulate
template <typename TJ>
__global__ void k_matvec7(int nx, int ny, int nz, JacIn<TJ> J, const double *__restrict__ x,
                          double *__restrict__ y) {
  pdl_enter();
  int i, j, k;
  if (!launch_ijk(nx, ny, nz, i, j, k)) return;
  const long long c = i + (long long)nx * (j + (long long)ny * k);
  const long long sy = nx, sz = (long long)nx * ny;
  double acc = 0.0;
  acc += (double)J.c[c] * x[c];
  acc += (double)J.w[c] * (i > 0 ? x[c - 1] : 0.0);
  acc += (double)J.e[c] * (i + 1 < nx ? x[c + 1] : 0.0);
  acc += (double)J.s[c] * (j > 0 ? x[c - sy] : 0.0);
  acc += (double)J.n[c] * (j + 1 < ny ? x[c + sy] : 0.0);
  acc += (double)J.l[c] * (k > 0 ? x[c - sz] : 0.0);
  acc += (double)J.u[c] * (k + 1 < nz ? x[c + sz] : 0.0);
  y[c] = acc;
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
static inline unsigned blocks_for(long long n, int bs) { return (unsigned)((n + bs - 1) / bs); }

// 3-D launch covering (nx, ny, nz) with `threads` threads per block
static inline void shape(int nx, int ny, int nz, int threads, dim3 &grid, dim3 &block) {
  const int bx = gather_columns(nx, threads);
  int by = threads / bx;
  if (by > ny) by = ny;
  block = dim3(bx, by, 1);
  grid = dim3((nx + bx - 1) / bx, (ny + by - 1) / by, nz);
}
// the tuned shape (bx, by) when one is set, else the heuristic
static inline void shape_tuned(int nx, int ny, int nz, int threads, const int tile[2],
                               dim3 &grid, dim3 &block) {
  if (!tile || tile[0] <= 0 || tile[1] <= 0) {
    shape(nx, ny, nz, threads, grid, block);
    return;
  }
  block = dim3(tile[0], tile[1], 1);
  grid = dim3((nx + tile[0] - 1) / tile[0], (ny + tile[1] - 1) / tile[1], nz);
}

static VGUniform vg_uniform(const DevProblem &P) {
  return VGUniform{1.0 / (P.density * P.gravity), 1.0 - 1.0 / P.vgn0};
}
template <bool STEP>
static void vg_launch(const DevProblem &P, const double *p, double *kr, double *dkr, double *sat,
                      double *dsat, const double *pp, const double *lam_p, double lam, double *pn,
                      cudaStream_t st) {
  launch_pdl(k_vg_all<STEP>, dim3(blocks_for(P.n, 256)), dim3(256), st, P, vg_uniform(P), p, kr,
             dkr, sat, dsat, pp, lam_p, lam, pn);
}
void launch_vg_all(const DevProblem &P, const double *p, double *kr, double *dkr, double *sat,
                   double *dsat, cudaStream_t st) {
  vg_launch<false>(P, p, kr, dkr, sat, dsat, nullptr, nullptr, 0.0, nullptr, st);
}
void launch_vg_step(const DevProblem &P, const double *u, const double *pp, const double *lam_p,
                    double lam, double *unew, double *kr, double *dkr, double *sat, double *dsat,
                    cudaStream_t st) {
  vg_launch<true>(P, u, kr, dkr, sat, dsat, pp, lam_p, lam, unew, st);
}

void launch_saturation(const DevProblem &P, const double *p, double *s, cudaStream_t st) {
  launch_pdl(k_saturation, dim3(blocks_for(P.n, 256)), dim3(256), st, P, vg_uniform(P), p, s);
}

// March (planes per chunk) or gather (0): the march form reads one permeability
// field; march_pays knows the rest.  PFGPU_RESIDUAL_FACE_ONCE=1 / 0 forces
// march / gather (bitwise the same results).
static int march_chunk(const DevProblem &P, MarchKernel kernel, bool slopes) {
  static const int forced = [] {
    const char *e = getenv("PFGPU_RESIDUAL_FACE_ONCE");
    return e && *e ? (*e == '1' ? 1 : 0) : -1;
  }();
  if (forced == 0 || P.ky != P.kx || P.kz != P.kx) return 0;
  if (forced < 0 && !march_pays(kernel, slopes, P.nx, P.ny, P.nz)) return 0;
  return march_planes(P.nx, P.ny, P.nz);
}
static dim3 march_grid(const DevProblem &P, int kchunk) {
  return dim3((P.nx + MARCH_COLS - 1) / MARCH_COLS,
              (P.ny + MARCH_WARPS - 1) / MARCH_WARPS,
              (P.nz + kchunk - 1) / kchunk);
}

template <bool SURF, bool VEL>
static void launch_residual_t(const DevProblem &P, const double *p, const double *p_old,
                              const double *s_old, const double *kr, const double *sat,
                              double dt, double *f, cudaStream_t st, const VelOut &vel) {
  if constexpr (!VEL) {
    if (const int kchunk = march_chunk(P, MARCH_RESIDUAL, SURF)) {
      launch_pdl(k_residual_march<SURF>, march_grid(P, kchunk), dim3(32, MARCH_WARPS), st, P, p,
                 p_old, s_old, kr, sat, dt, f, kchunk);
      return;
    }
  }
  dim3 g, b;
  shape_tuned(P.nx, P.ny, P.nz, 256, P.tile[0], g, b);
  launch_pdl(k_residual<SURF, VEL>, dim3(g), dim3(b), st, P, p, p_old, s_old, kr, sat, dt, f, vel);
}

void launch_residual(const DevProblem &P, const double *p, const double *p_old,
                     const double *s_old, const double *kr, const double *sat, double dt,
                     double *f, cudaStream_t st, const VelOut *vel) {
  const bool surf = P.tfg_xs || P.bc_type[5] == 2 || P.bc_type[5] == 3 || P.bc_type[5] == 4;
  if (vel) {
    if (surf)
      launch_residual_t<true, true>(P, p, p_old, s_old, kr, sat, dt, f, st, *vel);
    else
      launch_residual_t<false, true>(P, p, p_old, s_old, kr, sat, dt, f, st, *vel);
    return;
  }
  if (surf)
    launch_residual_t<true, false>(P, p, p_old, s_old, kr, sat, dt, f, st, VelOut{});
  else
    launch_residual_t<false, false>(P, p, p_old, s_old, kr, sat, dt, f, st, VelOut{});
}

template <typename TJ, typename TP>
void launch_jacobian(const DevProblem &P, const double *p, const double *kr,
                     const double *dkr, const double *sat, const double *dsat, double dt,
                     JacOut<TJ> J, PCOut<TP> M, cudaStream_t st) {
  const bool surf = P.tfg_xs || P.bc_type[5] == 2 || P.bc_type[5] == 3 || P.bc_type[5] == 4;
  const int kchunk =
      march_chunk(P, sizeof(TJ) == 8 ? MARCH_JACOBIAN_F64 : MARCH_JACOBIAN_F32, surf);
  if (kchunk) {
    if (surf)
      launch_pdl(k_jacobian_march<TJ, TP, true>, march_grid(P, kchunk), dim3(32, MARCH_WARPS), st,
                 P, p, kr, dkr, sat, dsat, dt, J, M, kchunk);
    else
      launch_pdl(k_jacobian_march<TJ, TP, false>, march_grid(P, kchunk), dim3(32, MARCH_WARPS), st,
                 P, p, kr, dkr, sat, dsat, dt, J, M, kchunk);
    return;
  }
  dim3 g, b;
  shape_tuned(P.nx, P.ny, P.nz, 128, P.tile[1], g, b);
  if (surf)
    launch_pdl(k_jacobian<TJ, TP, true>, dim3(g), dim3(b), st, P, p, kr, dkr, sat, dsat, dt, J, M);
  else
    launch_pdl(k_jacobian<TJ, TP, false>, dim3(g), dim3(b), st, P, p, kr, dkr, sat, dsat, dt, J,
               M);
}

template <typename TJ>
void launch_matvec7(int nx, int ny, int nz, JacIn<TJ> J, const double *x, double *y,
                    cudaStream_t st, const int *tile) {
  dim3 g, b;
  shape_tuned(nx, ny, nz, 256, tile, g, b);
  launch_pdl(k_matvec7<TJ>, dim3(g), dim3(b), st, nx, ny, nz, J, x, y);
}

template void launch_jacobian<double, double>(const DevProblem &, const double *,
                                              const double *, const double *, const double *,
                                              const double *, double, JacOut<double>,
                                              PCOut<double>, cudaStream_t);
template void launch_jacobian<float, float>(const DevProblem &, const double *, const double *,
                                            const double *, const double *, const double *,
                                            double, JacOut<float>, PCOut<float>, cudaStream_t);
template void launch_matvec7<double>(int, int, int, JacIn<double>, const double *, double *,
                                     cudaStream_t, const int *);
template void launch_matvec7<float>(int, int, int, JacIn<float>, const double *, double *,
                                    cudaStream_t, const int *);

}  // namespace pfgpu
