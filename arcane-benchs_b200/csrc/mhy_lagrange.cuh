// mhy_lagrange.cuh -- the Lagrange-phase cell kernel (geometry, corner
// vectors, density, pseudo-viscosity, energy, remap variables and the face
// data of the remap), templated on the number of environments K.
#pragma once

#include "mhy_kernels.cuh"

namespace mhy {

// ------------------------------------------------------------------------
// Lagrange phase, cells: UpdatePosition (cell centre), ComputeGeometricValues,
// UpdateDensity, ComputeArtificialViscosity, UpdateEnergyAndPressure (GP),
// computeVariablesForRemap_PBorn0 and computeFaceQuantitesForRemap for the
// cell's low faces, with the face-only terms of computeGradPhiFace and the
// upwind reconstruction precomputed (dx_f, (x_f - x_c).n0 for both cells).
// (MahycoModule.cc:913-928, 1054-1262, 1331-1370, 517-528, 1715-1726;
// PrepareRemap.cc:33-55, 93-117, 311-332; RemapADIService.cc:171-172, 710.)
__device__ __forceinline__ D3 load_xl(const Dims& dm, const double* __restrict__ x0, const double* __restrict__ vh,
                                      double dt, long long n) {
  return d3(x0[n], x0[dm.N + n], x0[2 * dm.N + n]) + dt * d3(vh[n], vh[dm.N + n], vh[2 * dm.N + n]);
}

// Half cross product 0.5 * (a - c) x (b - c) (MahycoModule.cc:2206-2239).
template <typename T>
__device__ __forceinline__ Vec3<T> half_cross(Vec3<T> a, Vec3<T> b, Vec3<T> c) { return T(0.5) * cross(a - c, b - c); }

// Corner vectors accumulated face by face.  Each corner's two six-term sums
// of MahycoModule.cc:2242-2257 take two consecutive terms from each of its
// three faces, in increasing face order, so adding them as the faces are
// visited keeps the reference's order; a corner is finished as soon as its
// third face is done.
template <typename T> struct CornerAcc { Vec3<T> s1, s2; };
template <typename T>
__device__ __forceinline__ void acc_start(CornerAcc<T>& a, Vec3<T> t1, Vec3<T> t2, Vec3<T> u1, Vec3<T> u2) {
  a.s1 = t1 + t2; a.s2 = u1 + u2;
}
template <typename T>
__device__ __forceinline__ void acc_add(CornerAcc<T>& a, Vec3<T> t1, Vec3<T> t2, Vec3<T> u1, Vec3<T> u2) {
  a.s1 = a.s1 + t1; a.s1 = a.s1 + t2; a.s2 = a.s2 + u1; a.s2 = a.s2 + u2;
}

// The 8 corner vectors of a hexahedron with nodes x (SN_trigo order),
// streamed: finish(a, cqs_a) is called as soon as corner a is complete
// (MahycoModule.cc:2195-2258, face centres as in :1080-1087).  T = double is
// the reference's arithmetic; T = float (mixed form) takes x relative to the
// cell centre, where every term has the size of the cell and nothing cancels.
template <typename T, typename Finish>
__device__ __forceinline__ void corner_vectors(const Vec3<T> x[8], Finish&& finish) {
  const T t12 = T(1.) / T(12.), q = T(0.25);
  auto fin = [&](int a, const CornerAcc<T>& ac) { finish(a, t12 * (T(5.) * ac.s1 + ac.s2)); };
  CornerAcc<T> k0, k1, k2, k3, k4, k5, k6, k7;
  {
    const Vec3<T> c0 = q * (x[0] + x[3] + x[2] + x[1]);
    const Vec3<T> n04 = half_cross(x[0], x[3], c0), n03 = half_cross(x[3], x[2], c0);
    const Vec3<T> n02 = half_cross(x[2], x[1], c0), n01 = half_cross(x[1], x[0], c0);
    acc_start(k0, n01, n04, n02, n03);
    acc_start(k1, n01, n02, n04, n03);
    acc_start(k2, n02, n03, n01, n04);
    acc_start(k3, n03, n04, n01, n02);
  }
  {
    const Vec3<T> c1 = q * (x[0] + x[4] + x[7] + x[3]);
    const Vec3<T> n05 = half_cross(x[0], x[4], c1), n12 = half_cross(x[4], x[7], c1);
    const Vec3<T> n08 = half_cross(x[7], x[3], c1), n04 = half_cross(x[3], x[0], c1);
    acc_add(k0, n04, n05, n08, n12);
    acc_add(k3, n08, n04, n05, n12);
    acc_start(k4, n05, n12, n08, n04);
    acc_start(k7, n08, n12, n04, n05);
  }
  {
    const Vec3<T> c2 = q * (x[0] + x[1] + x[5] + x[4]);
    const Vec3<T> n01 = half_cross(x[0], x[1], c2), n06 = half_cross(x[1], x[5], c2);
    const Vec3<T> n09 = half_cross(x[5], x[4], c2), n05 = half_cross(x[4], x[0], c2);
    acc_add(k0, n05, n01, n06, n09);
    fin(0, k0);
    acc_add(k1, n01, n06, n09, n05);
    acc_add(k4, n05, n09, n01, n06);
    acc_start(k5, n06, n09, n01, n05);
  }
  {
    const Vec3<T> c3 = q * (x[4] + x[5] + x[6] + x[7]);
    const Vec3<T> n09 = half_cross(x[4], x[5], c3), n10 = half_cross(x[5], x[6], c3);
    const Vec3<T> n11 = half_cross(x[6], x[7], c3), n12 = half_cross(x[7], x[4], c3);
    acc_add(k4, n09, n12, n10, n11);
    fin(4, k4);
    acc_add(k5, n09, n10, n12, n11);
    acc_start(k6, n11, n10, n12, n09);
    acc_add(k7, n12, n11, n09, n10);
  }
  {
    const Vec3<T> c4 = q * (x[1] + x[2] + x[6] + x[5]);
    const Vec3<T> n02 = half_cross(x[1], x[2], c4), n07 = half_cross(x[2], x[6], c4);
    const Vec3<T> n10 = half_cross(x[6], x[5], c4), n06 = half_cross(x[5], x[1], c4);
    acc_add(k1, n06, n02, n10, n07);
    fin(1, k1);
    acc_add(k2, n07, n02, n06, n10);
    acc_add(k5, n10, n06, n07, n02);
    fin(5, k5);
    acc_add(k6, n10, n07, n06, n02);
  }
  {
    const Vec3<T> c5 = q * (x[2] + x[3] + x[7] + x[6]);
    const Vec3<T> n03 = half_cross(x[2], x[3], c5), n08 = half_cross(x[3], x[7], c5);
    const Vec3<T> n11 = half_cross(x[7], x[6], c5), n07 = half_cross(x[6], x[2], c5);
    acc_add(k2, n07, n03, n11, n08);
    fin(2, k2);
    acc_add(k3, n08, n03, n07, n11);
    fin(3, k3);
    acc_add(k6, n07, n11, n03, n08);
    fin(6, k6);
    acc_add(k7, n11, n08, n07, n03);
    fin(7, k7);
  }
}

// Remap face data from a cell's nodes (PrepareRemap.cc:41-55, 105-117;
// RemapADIService.cc:710): for the low face of each direction |A| along d, u_f and
// (x_f - x_c).n0 with this cell as the next cell; for the high face (x_f - x_c).n0
// with this cell as the previous one.  Face node order: X (0,3,7,4), Y (0,1,5,4), Z (0,1,2,3) low;
// X (1,2,6,5), Y (3,2,6,7), Z (4,5,6,7) high, in SN_trigo cell-node numbers.
// In FP64 the values of boundary faces are written too and read by nobody:
// without a branch the faces' arithmetic overlaps the chain of the thermodynamics.
// T = float takes x relative to the cell centre (xc = 0).  HC: also the cell
// widths along each direction into fd.h (order 3 and the generalised limiters).
// nlo(d), nhi(d): the normals of the low and high face of direction d; vn(a):
// the Lagrange velocity of cell node a.
template <typename T, bool HC, typename Nlo, typename Nhi, typename Vn>
__device__ __forceinline__ void face_data(const Dims& dm, int i, int j, int k, const Vec3<T> x[8], Vec3<T> xc,
                                          const FaceData& fd, Nlo&& nlo, Nhi&& nhi, Vn&& vn) {
  const T q = T(.25);
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const int id = d == 0 ? i : (d == 1 ? j : k);
    double hsum = 0;            // order 3: cell width along d (RemapADIService.cc:240-257)
    const int lo[3][4] = {{0, 3, 7, 4}, {0, 1, 5, 4}, {0, 1, 2, 3}};
    const int hi[3][4] = {{1, 2, 6, 5}, {3, 2, 6, 7}, {4, 5, 6, 7}};
    const long long off = d == 0 ? 0 : (d == 1 ? dm.Fx : dm.Fx + dm.Fy);
    if (sizeof(T) == 8 || id > 0) {
      const long long f = dm.fid(d, i, j, k);
      const D3 nrm = nlo(d);
      const Vec3<T> nr = Vec3<T>{(T)nrm.x, (T)nrm.y, (T)nrm.z};
      const Vec3<T> a0 = x[lo[d][0]], a1 = x[lo[d][1]], a2 = x[lo[d][2]], a3 = x[lo[d][3]];
      Vec3<T> xf = Vec3<T>{0, 0, 0};
      xf = xf + q * a0; xf = xf + q * a1; xf = xf + q * a2; xf = xf + q * a3;
      D3 vs = d3(0., 0., 0.);
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        vs = vs + vn(lo[d][b]);
      }
      const Vec3<T> cr = T(0.5) * cross(a2 - a0, a3 - a1);
      double A = fabs((double)comp(cr, d));
      if (!(fabs(comp(nrm, d)) >= 1.0E-10)) A = 0.;   // RemapADIService.cc:925 filter: no flux
      const long long t = f - off;
      fd.A[d][t] = A;
      fd.u[d][t] = dot(.25 * vs, nrm);
      fd.df[d][t] = (double)dot(xf - xc, nr);
      if constexpr (HC) { if (id > 0) hsum += norm2(xf - xc); }
    }
    if (sizeof(T) == 8 || id + 1 < dm.ncd(d)) {
      const long long f = dm.fid(d, i + (d == 0), j + (d == 1), k + (d == 2));
      const D3 nrm = nhi(d);
      const Vec3<T> nr = Vec3<T>{(T)nrm.x, (T)nrm.y, (T)nrm.z};
      Vec3<T> xf = Vec3<T>{0, 0, 0};
      xf = xf + q * x[hi[d][0]]; xf = xf + q * x[hi[d][1]]; xf = xf + q * x[hi[d][2]]; xf = xf + q * x[hi[d][3]];
      fd.db[d][f - off] = (double)dot(xf - xc, nr);
      if constexpr (HC) { if (id + 1 < dm.ncd(d)) hsum += norm2(xf - xc); }
    }
    if constexpr (HC) fd.h[d * dm.C + dm.cid(i, j, k)] = hsum;
  }
}

// schema-csts energy of one environment of a cell (MahycoModule.cc:1776-1810,
// updateEnergyAndPressureforGP; or by Newton on f, :1552-1613 with
// MahycoModule.h:433-445, the first iteration always run as in newton_eint).
// cn1, cn, cdn, con: the corner-vector sums v.cqs dt, v.cqs_n dt,
// (v - v_n).cqs_n (dt - dt_old), v_n.cqs_n dt_old.  The n-1 pseudo-viscosity
// is zero: the remap resets the n-level fields (PrepareRemap.cc:485-550)
// before saveValuesAtN copies them into it.  pf gets the pressure that
// updateVelocityForward reads: p_n, or the last Newton EOS value; the
// kernel stores it plus this cycle's pseudo-viscosity.  g, eos, pinf: the
// environment's adiabatic constant, EOS and limit tension.
__device__ __forceinline__ double csts_eint(const Phys& ph, double g, int eos, double pinf, double cn1, double cn,
                                            double cdn, double con, double e0, double r, double m, double pn,
                                            double qn, double q, double& pf) {
  const double qnm1 = 0.;
  if (!ph.with_newton) {
    const double denom = 1 + 0.5 * (g - 1.0) * r * cn1 / m;
    const double numer = e0 - (0.5 * (pn + qn) * cn / m) - (0.5 * q * cn1 / m) + (0.25 * (pn + qn) * cdn / m) -
                         (0.5 * (qn - qnm1) * con / m);
    pf = pn;
    return numer / denom;
  }
  const double cdon = 0., epsilon = ph.threshold, itermax = 50;
  const double en = e0;
  double e = en, pp, dpde;
  int i = 0;
  do {
    if (eos == 1) pp = ((g - 1.) * r * e) - (g * pinf);
    else pp = (g - 1.) * r * e;
    dpde = (g - 1.) * r;
    const double fe = e - en + 0.5 * (pp + q) * cn1 / m + 0.5 * (pn + qn) * cn / m - 0.25 * (pn + qn) * cdn / m +
                      0.5 * (q - qnm1) * cdon / m;
    const double enew = e - fe / (1. + 0.5 * dpde * cn1 / m);
    e = enew;
    i++;
  } while (i < itermax && fabs(e - en + 0.5 * (pp + q) * cn1 / m + 0.5 * (pn + qn) * cn / m -
                                0.25 * (pn + qn) * cdn / m + 0.5 * (q - qnm1) * cdon / m) >= epsilon);
  pf = pp;
  return e;
}

// Lagrange thermodynamics of a cell of one environment (MahycoModule.cc:1331-1426
// updateDensity, :454-578 computeArtificialViscosity, :1659-1770
// updateEnergyAndPressureforGP): the characteristic length, density,
// pseudo-viscosity and energy.  SP: the quotients of mhy_quot.h, without a
// branch, so that this chain of a dozen dependent quotients overlaps the face
// data; *oor is raised where they may differ and the cell is done again by
// thermo_one_exact.  Measured on B200 with plain quotients -> with these: cell
// kernel of Sedov 128^3 377 -> 323 us in FP64, 230 -> 219 us in the mixed form.
struct ThermoIn { double V, inv_dt, rn, m, cs, p, q, e; };
struct ThermoOut { double L, nd, qn, en, pf; };
template <bool CSTS, bool F32, bool SP, bool NEWTON>
__device__ __forceinline__ ThermoOut thermo_one(const Phys& ph, const ThermoIn& in, double Lface, double cn1, double cn,
                                                double cdn, double con, unsigned* oor) {
  ThermoOut o;
  o.pf = 0.;
  // racine-cubique-volume: the project cube root (the reference's bits) in
  // FP64; the mixed form takes CUDA's FP32 cube root of the FP64 volume (L
  // feeds the viscosity and the CFL bound only)
  if (ph.lc_mode == 0) {
    if constexpr (F32) o.L = (double)cbrtf((float)in.V);
    else o.L = pow_third_of<SP>(in.V, oor);
  } else {
    o.L = Lface;
  }
  const double nd = qu<double, SP>(in.m, in.V, oor);
  const double irn = rc<double, SP>(in.rn, oor), ind = rc<double, SP>(nd, oor);
  const double tau = 0.5 * (irn + ind);
  const double itau = rc<double, SP>(tau, oor);
  const double du = dv<double, SP>(in.inv_dt * (ind - irn), tau, itau, oor);
  double qn = 0.;
  const double g = ph.gamma;
  if (du < 0.0) qn = itau * (-0.5 * o.L * in.cs * du + (g + 1) / 2.0 * o.L * o.L * du * du);
  o.nd = nd;
  o.qn = qn;
  if constexpr (CSTS)
    o.en = csts_eint(ph, g, ph.eos, ph.pinf, cn1, cn, cdn, con, in.e, nd, in.m, in.p, in.q, qn, o.pf);
  else
    o.en = energy_update<SP, NEWTON>(ph.with_newton != 0, ph.pseudo_centree != 0, ph.eos, g, ph.pinf, ph.threshold,
                                     in.q, qn, ind, irn, nd, in.p, in.e, oor);
  return o;
}
template <bool CSTS, bool F32>
__device__ __noinline__ ThermoOut thermo_one_exact(Phys ph, ThermoIn in, double Lface, double cn1, double cn, double cdn,
                                                   double con) {
  return thermo_one<CSTS, F32, false, true>(ph, in, Lface, cn1, cn, cdn, con, nullptr);
}

// Lagrange thermodynamics of a mesh with K > 1 environments, then the remap
// variables (MahycoModule.cc:1331-1426 updateDensity, :454-578
// computeArtificialViscosity, :1659-1770 updateEnergyAndPressureforGP,
// PrepareRemap.cc:258-437 computeVariablesForRemap_PBorn0).  Pure cells take
// the single-environment formulas with their environment's gamma; a mixed
// cell works environment by environment on V_k = f_k V (MahycoModule.cc:1274-1295).
// U holds the 3K+1 non-zero remap variables [V_k | V_k rho_k | V_k rho_k e_k |
// V q] as planes; V is kept in Vlag, the divisor of Phi on the first sweep.
// The global density m/V is stored for every cell: the remap keeps it in a
// mixed cell whose fractions leave one environment only (RemapADIFinal.cc:561-562).
// pbphi (pente-borne): Phi of the first sweep for the cell's environments,
// volume fraction, density and internal energy after this step, and q of
// the last of them (PrepareRemap.cc:201-212); the other environments' planes
// are left as they are.  CSTS: each environment's energy by csts_eint from
// the cell's corner-vector sums cssum (cn1, cn, cdn, con), and pf = the
// global p + q the forward step reads (MahycoModule.cc:792-831): a pure
// cell's p_n or Newton pressure plus its q, a mixed cell's mean p_n plus
// sum_k f_k q_k (MahycoModule.cc:454-578).
// rn: the density before the step.  SP: the quotients of mhy_quot.h (see
// thermo_one); where *oor is raised the cell is done again by
// lagrange_thermo_env_exact, which writes all of it anew.
template <int K, bool CSTS, bool SP, bool NEWTON>
__device__ __forceinline__ void lagrange_thermo_env(const Phys& ph, const EnvState& env, int c, int C,
                                                    const ThermoIn& in, double Lc, double* __restrict__ rho,
                                                    double* __restrict__ U,
                                                    double* __restrict__ Vlag, double* __restrict__ pbphi,
                                                    const double* cssum, double* __restrict__ pf, unsigned* oor) {
  constexpr int NV = 3 * K + 1;
  const double V = in.V;
  const double nd = qu<double, SP>(in.m, V, oor);
  const double irn = rc<double, SP>(in.rn, oor), ind = rc<double, SP>(nd, oor);
  const double tau = 0.5 * (irn + ind);
  const double itau = rc<double, SP>(tau, oor);
  const double du = dv<double, SP>(in.inv_dt * (ind - irn), tau, itau, oor);
  const uint32_t mk = env.mask[c];
  const bool pc = ph.pseudo_centree != 0;
  double u[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) u[v] = 0.;
  if (__popc(mk) == 1) {
    const int ke = __ffs(mk) - 1;
    const double g = env.gamma[ke];
    double qn = 0.;
    if (du < 0.0) qn = itau * (-0.5 * Lc * in.cs * du + (g + 1) / 2.0 * Lc * Lc * du * du);
    double en;
    if constexpr (CSTS) {
      double pforward;
      en = csts_eint(ph, g, env.eos[ke], env.pinf[ke], cssum[0], cssum[1], cssum[2], cssum[3], in.e, nd, in.m,
                     in.p, in.q, qn, pforward);
      pf[c] = pforward + qn;
    } else {
      en = energy_update<SP, NEWTON>(ph.with_newton != 0, pc, env.eos[ke], g, env.pinf[ke], ph.threshold, in.q, qn, ind,
                                     irn, nd, in.p, in.e, oor);
    }
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (k == ke) { u[k] = V; u[K + k] = V * nd; u[2 * K + k] = V * nd * en; }
    u[3 * K] = V * qn;
    if (pbphi) {
      pbphi[ke * C + c] = env.fg[c]; pbphi[(K + ke) * C + c] = nd; pbphi[(2 * K + ke) * C + c] = en;
      pbphi[3 * K * C + c] = qn;
    }
  } else {
    const double csc = in.cs;
    double qg = 0.;                                              // the mixed cell's pseudo-viscosity sum_k f_k q_k
#pragma unroll
    for (int k = 0; k < K; ++k) {
      if (!(mk >> k & 1)) continue;
      const int o = k * C + c;
      const double vk = env.f[o] * V;
      const double rk = qu<double, SP>(env.m[o], vk, oor);
      const double irnk = rc<double, SP>(env.rho[o], oor), irk = rc<double, SP>(rk, oor);
      const double tauk = 0.5 * (irnk + irk);
      const double g = env.gamma[k];
      double qk = 0.;
      if (du < 0.0) qk = rc<double, SP>(tauk, oor) * (-0.5 * Lc * csc * du + (g + 1) / 2.0 * Lc * Lc * du * du);
      double ek;
      if constexpr (CSTS) {
        double pk_unused;
        ek = csts_eint(ph, g, env.eos[k], env.pinf[k], cssum[0], cssum[1], cssum[2], cssum[3], env.e[o], rk, env.m[o],
                       env.p[o], env.q[o], qk, pk_unused);
        qg += qk * env.f[o];
      } else {
        ek = energy_update<SP, NEWTON>(ph.with_newton != 0, pc, env.eos[k], g, env.pinf[k], ph.threshold, env.q[o], qk,
                                       irk, irnk, rk, env.p[o], env.e[o], oor);
      }
      u[k] = vk;
      u[K + k] = vk * rk;
      u[2 * K + k] = vk * rk * ek;
      u[3 * K] = vk * qk;                                        // the last environment wins (P:318-330)
      if (pbphi) {
        pbphi[o] = env.f[o]; pbphi[K * C + o] = rk; pbphi[2 * K * C + o] = ek; pbphi[3 * K * C + c] = qk;
      }
    }
    if constexpr (CSTS) pf[c] = in.p + qg;                      // the mean p_n: no EOS runs before the forward step
  }
#pragma unroll
  for (int v = 0; v < NV; ++v) U[v * C + c] = u[v];
  Vlag[c] = V;
  rho[c] = nd;
}
template <int K, bool CSTS>
__device__ __noinline__ void lagrange_thermo_env_exact(Phys ph, EnvState env, int c, int C, ThermoIn in, double Lc,
    double* rho, double* U, double* Vlag, double* pbphi, double cn1, double cn, double cdn, double con, double* pf) {
  const double cssum[4] = {cn1, cn, cdn, con};
  lagrange_thermo_env<K, CSTS, false, true>(ph, env, c, C, in, Lc, rho, U, Vlag, pbphi, cssum, pf, nullptr);
}

// The characteristic length and the thermodynamics of a cell, then its remap
// variables, whichever number of environments.  Lface: the length of
// faces-opposees (used when lc_mode is 1).  NEWTON: the kernels of contexts with
// with-newton, and of batches with an instance that has it.  Measured on B200:
// one kernel for both spills (two gases 256x128x128 without Newton 2.74 -> 2.81 ms
// a cycle); Newton by way of the exact form costs a copy of its arguments and plain
// quotients in every cell (a cycle with Newton 3.14 ms there and 460 us with three
// gases on 90x60x60, 2.89 ms and 405 us in these kernels).
template <int K, bool CSTS, bool F32, bool NEWTON>
__device__ __forceinline__ void cell_thermo(const Phys& ph, const EnvState& env, const FaceData& fd, int c, int C,
                                            const ThermoIn& in, double Lface, double* __restrict__ rho,
                                            double* __restrict__ L, double* __restrict__ U, double* __restrict__ Vlag,
                                            double cn1, double cn, double cdn, double con, double* __restrict__ pf) {
  unsigned oor = 0u;
  if constexpr (K == 1) {
    ThermoOut t = thermo_one<CSTS, F32, true, NEWTON>(ph, in, Lface, cn1, cn, cdn, con, &oor);
    if (oor) t = thermo_one_exact<CSTS, F32>(ph, in, Lface, cn1, cn, cdn, con);
    L[c] = t.L;
    if constexpr (CSTS) pf[c] = t.pf + t.qn;                      // the forward force's p + q (q: this cycle's)
    U[c] = in.V;
    U[C + c] = in.V * t.nd;
    U[2 * C + c] = in.V * t.nd * t.en;
    U[3 * C + c] = in.V * t.qn;
    if (fd.pbphi) { fd.pbphi[c] = t.nd; fd.pbphi[C + c] = t.en; fd.pbphi[2 * C + c] = t.qn; }
  } else {
    double Lc = Lface;
    if (ph.lc_mode == 0) {
      if constexpr (F32) Lc = (double)cbrtf((float)in.V);
      else {
        unsigned lo = 0u;
        Lc = pow_third_of<true>(in.V, &lo);
        if (lo) Lc = pow_third(in.V);
      }
    }
    L[c] = Lc;
    const double cssum[4] = {cn1, cn, cdn, con};
    lagrange_thermo_env<K, CSTS, true, NEWTON>(ph, env, c, C, in, Lc, rho, U, Vlag, fd.pbphi, cssum, pf, &oor);
    if (oor)
      lagrange_thermo_env_exact<K, CSTS>(ph, env, c, C, in, Lc, rho, U, Vlag, fd.pbphi, cn1, cn, cdn, con, pf);
  }
}

// faces-opposees: the length from the distances of opposite face centres.
__device__ __forceinline__ double face_length(const D3 x[8]) {
  D3 fc[6];
  face_centres(x, fc);
  const double d1 = norm2(fc[0] - fc[3]), d2 = norm2(fc[2] - fc[5]), d3_ = norm2(fc[1] - fc[4]);
  return (d1 * d2 * d3_) / (d1 * d2 + d1 * d3_ + d2 * d3_);
}

// CSTS (schema-csts, FP64 only): vnb = the backward node velocity of this
// cycle, pf = the pressure plus pseudo-viscosity of the forward step.
template <int K, typename R, bool CSTS, bool HC, bool NEWTON>
__device__ __forceinline__ void k_cyc_lagrange_cells_body(Dims dm, const Scalars* __restrict__ S, Phys ph,
    const double* __restrict__ x0, const double* __restrict__ vh, const double* __restrict__ n0,
    double* __restrict__ rho, const double* __restrict__ e, const double* __restrict__ q,
    const double* __restrict__ p, const double* __restrict__ cs, const double* __restrict__ mass,
    double* __restrict__ cqs, float* __restrict__ cqs32, double* __restrict__ L, double* __restrict__ U,
    double* __restrict__ xcs, FaceData fd, EnvState env, double* __restrict__ Vlag,
    int bx_, int by_, int bz_, const double* __restrict__ vnb = nullptr, double* __restrict__ pf = nullptr) {
  static_assert(!CSTS || sizeof(R) == 8, "schema-csts: FP64");
  int i, j, k;
  if (!block_item(dm.nx, dm.ny, dm.nz, bx_, by_, bz_, i, j, k)) return;
  const long long c = dm.cid(i, j, k);
  const long long C = dm.C;
  const double dt = S->dt;
  D3 x[8];
#pragma unroll
  for (int a = 0; a < 8; ++a)
    x[a] = load_xl(dm, x0, vh, dt, dm.nid(i + kCellNodeOff[a][0], j + kCellNodeOff[a][1], k + kCellNodeOff[a][2]));
  D3 sm = d3(0., 0., 0.);
#pragma unroll
  for (int a = 0; a < 8; ++a) sm = sm + x[a];
  const D3 xc = .125 * sm;
  xcs[c] = xc.x; xcs[C + c] = xc.y; xcs[2 * C + c] = xc.z;

  // corner vectors and volume V = 1/3 sum x_a . cqs_a (MahycoModule.cc:1224-1262)
  constexpr bool F32 = sizeof(R) == 4;
  double cs_cn1 = 0., cs_cn = 0., cs_cdn = 0., cs_con = 0.;   // schema-csts sums
  double V = 0;
  F3 xr[8];
  if constexpr (F32) {
    // mixed form: FP32 corner vectors from coordinates relative to the
    // centre (kept in FP32 for the force), volume summed in FP64
#pragma unroll
    for (int a = 0; a < 8; ++a)
      xr[a] = F3{(float)(x[a].x - xc.x), (float)(x[a].y - xc.y), (float)(x[a].z - xc.z)};
    float dv[8];
    corner_vectors<float>(xr, [&](int a, F3 o) {
      cqs32[(a * 3 + 0) * C + c] = o.x; cqs32[(a * 3 + 1) * C + c] = o.y; cqs32[(a * 3 + 2) * C + c] = o.z;
      dv[a] = dot(xr[a], o);
    });
#pragma unroll
    for (int a = 0; a < 8; ++a) V += (double)dv[a];
  } else {
    double dv[8], dv1[8];
    if constexpr (CSTS) {
      // the sums over the previous corner vectors, before they are overwritten
#pragma unroll
      for (int a = 0; a < 8; ++a) {
        const long long nn = dm.nid(i + kCellNodeOff[a][0], j + kCellNodeOff[a][1], k + kCellNodeOff[a][2]);
        const D3 va = d3(vh[nn], vh[dm.N + nn], vh[2 * dm.N + nn]);
        const D3 vb = d3(vnb[nn], vnb[dm.N + nn], vnb[2 * dm.N + nn]);
        const D3 cq = d3(cqs[(a * 3 + 0) * C + c], cqs[(a * 3 + 1) * C + c], cqs[(a * 3 + 2) * C + c]);
        cs_cn += dot(va, cq) * dt;
        cs_cdn += dot(va - vb, cq) * (dt - S->old_dt);
        cs_con += dot(vb, cq) * S->old_dt;
      }
    }
    corner_vectors<double>(x, [&](int a, D3 o) {
      cqs[(a * 3 + 0) * C + c] = o.x; cqs[(a * 3 + 1) * C + c] = o.y; cqs[(a * 3 + 2) * C + c] = o.z;
      dv[a] = dot(x[a], o);
      if constexpr (CSTS) {
        const long long nn = dm.nid(i + kCellNodeOff[a][0], j + kCellNodeOff[a][1], k + kCellNodeOff[a][2]);
        dv1[a] = dot(d3(vh[nn], vh[dm.N + nn], vh[2 * dm.N + nn]), o) * dt;
      }
    });
#pragma unroll
    for (int a = 0; a < 8; ++a) V += dv[a];
    if constexpr (CSTS) {
#pragma unroll
      for (int a = 0; a < 8; ++a) cs_cn1 += dv1[a];
    }
  }
  V *= 1. / 3;
  double Lc = 0.;
  if (ph.lc_mode != 0) {
    if constexpr (F32) {
      D3 xx[8];
#pragma unroll
      for (int a = 0; a < 8; ++a) xx[a] = d3(xr[a].x, xr[a].y, xr[a].z);
      Lc = face_length(xx);
    } else {
      Lc = face_length(x);
    }
  }
  const ThermoIn in{V, S->inv_dt, rho[c], mass[c], cs[c], p[c], q[c], e[c]};
  cell_thermo<K, CSTS, F32, NEWTON>(ph, env, fd, (int)c, (int)C, in, Lc, rho, L, U, Vlag, cs_cn1, cs_cn, cs_cdn, cs_con, pf);
  auto normal = [&](long long f) { return d3(n0[f], n0[dm.F + f], n0[2 * dm.F + f]); };
  auto nlo = [&](int d) { return normal(dm.fid(d, i, j, k)); };
  auto nhi = [&](int d) { return normal(dm.fid(d, i + (d == 0), j + (d == 1), k + (d == 2))); };
  auto vn = [&](int a) {
    const long long nn = dm.nid(i + kCellNodeOff[a][0], j + kCellNodeOff[a][1], k + kCellNodeOff[a][2]);
    return d3(vh[nn], vh[dm.N + nn], vh[2 * dm.N + nn]);
  };
  if constexpr (F32) face_data<float, false>(dm, i, j, k, xr, F3{0.f, 0.f, 0.f}, fd, nlo, nhi, vn);
  else face_data<double, HC>(dm, i, j, k, x, xc, fd, nlo, nhi, vn);
}

template <int K, typename R, bool HC, bool NEWTON>
__global__ void __launch_bounds__(128, sizeof(R) == 4 ? 5 : 3) k_cyc_lagrange_cells(Dims dm,
    const Scalars* __restrict__ S, Phys ph,
    const double* __restrict__ x0, const double* __restrict__ vh, const double* __restrict__ n0,
    double* __restrict__ rho, const double* __restrict__ e, const double* __restrict__ q,
    const double* __restrict__ p, const double* __restrict__ cs, const double* __restrict__ mass,
    double* __restrict__ cqs, float* __restrict__ cqs32, double* __restrict__ L, double* __restrict__ U,
    double* __restrict__ xcs, FaceData fd, EnvState env, double* __restrict__ Vlag, int linear) {
  k_cyc_lagrange_cells_body<K, R, false, HC, NEWTON>(dm, S, ph, x0, vh, n0, rho, e, q, p, cs, mass, cqs, cqs32, L, U,
                                                     xcs, fd, env, Vlag, blockIdx.x, linear ? -1 : (int)blockIdx.y, blockIdx.z);
}

// ------------------------------------------------------------------------
// The cell kernel over columns of cells (all but schema-csts).  A block takes
// kColThreads consecutive cells of one z layer (x fastest) and marches up a
// segment of layers.  The node planes it needs are copied to shared memory one
// layer ahead (cp.async), so that their latency passes under the arithmetic of
// the layer before, and each node's Lagrangian coordinates are formed once a
// block instead of once for each of its 8 cells.  The cell's own state and the
// normals of its faces are copied at the start of its layer and used at its end.
// Bound: FP64 latency with 12 warps an SM (168 registers hold the corner
// vectors' sums; the FP64 work alone takes 150 us and the bytes 165 us on Sedov
// 128^3).  Measured on B200 against one thread a cell with the nodes gathered
// from memory: 323 -> 249 us there (315 us with strips of a length known at run
// time only), 1372 -> 1100 us on a batch of 24 meshes 32^3..96^3, 868 -> 665 us
// with two gases on 256x128x128.
constexpr int kColPriv = 24;         // doubles a cell: 18 normals (low and high faces), 6 state values

// Nodes of a strip: a plane of nodes comes as two strips, from the low row of
// the block's first cell onwards and from one row up; a strip holds the block's
// cells, one node more a row that it touches and one for its last cell.  Two
// lengths, known at compile time so that a cell's nodes lie at fixed offsets:
// one for rows of 22 cells and more, one for any row of two cells and more.
constexpr int kColStrip = 136, kColStripWide = 200;
__host__ __device__ __forceinline__ int col_strip(int nx) {
  return kColThreads + (kColThreads + nx - 2) / nx + 2 <= kColStrip ? kColStrip : kColStripWide;
}
__host__ __device__ __forceinline__ size_t col_smem(int strip) {
  return (size_t)(3 * 12 * strip + kColPriv * kColThreads) * sizeof(double);
}

__device__ __forceinline__ void cp_async8(double* s, const double* g) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(s)), "l"(g));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;"); }
template <int Left> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(Left) : "memory"); }

template <int K, bool HC, int strip, bool NEWTON>
__device__ __forceinline__ void lagrange_columns(const CycleArgs& A, int bx, int seg) {
  extern __shared__ double col_mem[];
  const Dims& dm = A.dm;
  const int nx = dm.nx, ny = dm.ny, nz = dm.nz, nnx = nx + 1, np = nnx * (ny + 1);
  const int tid = threadIdx.x;
  const int N = (int)dm.N, C = (int)dm.C, F = (int)dm.F;
  double* const priv = col_mem + 36 * strip;                      // [kColPriv][kColThreads]
  int k0, k1;
  col_layers(nx, ny, nz, seg, k0, k1);
  const int p0 = bx * kColThreads, p = p0 + tid;
  const bool cell = p < nx * ny;
  const int i = p % nx, j = p / nx;
  const int b0 = p0 + p0 / nx;                                    // plane index of the first cell's node
  const int off = p + j - b0;                                     // this cell's node (i, j) in the low strip
  const double dt = A.S->dt, inv_dt = A.S->inv_dt;

  // node plane k -> buffer k % 3: x0 (planes 0..2) and vh (3..5) of both strips
  auto fetch = [&](int k) {
    double* buf = col_mem + (k % 3) * 12 * strip;
#pragma unroll
    for (int s = 0; s < 2; ++s)
      for (int t = tid; t < strip; t += kColThreads) {
        const int n = b0 + s * nnx + t;
        if (n < np) {
          const int g = n + np * k;
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            cp_async8(buf + (s * 6 + c) * strip + t, A.x0 + c * N + g);
            cp_async8(buf + (s * 6 + 3 + c) * strip + t, A.vh + c * N + g);
          }
        }
      }
  };
  // the elements this thread copied: coordinates x0 -> x0 + vh dt
  auto advance = [&](int k) {
    double* buf = col_mem + (k % 3) * 12 * strip;
#pragma unroll
    for (int s = 0; s < 2; ++s)
      for (int t = tid; t < strip; t += kColThreads)
        if (b0 + s * nnx + t < np) {
#pragma unroll
          for (int c = 0; c < 3; ++c)
            buf[(s * 6 + c) * strip + t] = buf[(s * 6 + c) * strip + t] + buf[(s * 6 + 3 + c) * strip + t] * dt;
        }
  };
  fetch(k0);
  fetch(k0 + 1);
  cp_commit();
  cp_wait<0>();
  advance(k0);
#pragma unroll 1
  for (int k = k0; k < k1; ++k) {
    cp_wait<0>();
    advance(k + 1);
    __syncthreads();                       // plane k + 1 is whole; plane k - 1 is read by nobody any more
    const int c = p + nx * ny * k;
    if (cell) {
      // normals: low face of x, y, z, then high; rho, mass, cs, p, q, e
      const int fx = i + nnx * (j + ny * k), fy = (int)dm.Fx + i + nx * (j + (ny + 1) * k), fz = (int)(dm.Fx + dm.Fy) + c;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const double* na = A.n0 + (long long)a * F;
        cp_async8(priv + (0 + a) * kColThreads + tid, na + fx);
        cp_async8(priv + (3 + a) * kColThreads + tid, na + fy);
        cp_async8(priv + (6 + a) * kColThreads + tid, na + fz);
        cp_async8(priv + (9 + a) * kColThreads + tid, na + fx + 1);
        cp_async8(priv + (12 + a) * kColThreads + tid, na + fy + nx);
        cp_async8(priv + (15 + a) * kColThreads + tid, na + fz + nx * ny);
      }
      cp_async8(priv + 18 * kColThreads + tid, A.st.rho + c);
      cp_async8(priv + 19 * kColThreads + tid, A.st.mass + c);
      cp_async8(priv + 20 * kColThreads + tid, A.st.cs + c);
      cp_async8(priv + 21 * kColThreads + tid, A.st.p + c);
      cp_async8(priv + 22 * kColThreads + tid, A.st.q + c);
      cp_async8(priv + 23 * kColThreads + tid, A.st.e + c);
    }
    cp_commit();
    if (k + 1 < k1) fetch(k + 2);
    cp_commit();
    const double* const lo = col_mem + (k % 3) * 12 * strip + off;
    const double* const hi = col_mem + ((k + 1) % 3) * 12 * strip + off;
    // component a of the vector at node n of the cell (first = 0: coordinates, 3: velocities)
    auto node = [&](int n, int first) {
      const double* b = (n < 4 ? lo : hi) + (kCellNodeOff[n][1] * 6 + first) * strip + kCellNodeOff[n][0];
      return d3(b[0], b[strip], b[2 * strip]);
    };
    if (cell) {
      double V = 0;
      {
        D3 x[8];
#pragma unroll
        for (int a = 0; a < 8; ++a) x[a] = node(a, 0);
        // corner vectors and volume V = 1/3 sum x_a . cqs_a (MahycoModule.cc:1224-1262)
        double dvv[8];
        corner_vectors<double>(x, [&](int a, D3 o) {
          A.cqs[(a * 3 + 0) * C + c] = o.x; A.cqs[(a * 3 + 1) * C + c] = o.y; A.cqs[(a * 3 + 2) * C + c] = o.z;
          dvv[a] = dot(x[a], o);
        });
#pragma unroll
        for (int a = 0; a < 8; ++a) V += dvv[a];
        V *= 1. / 3;
      }
      cp_wait<1>();                        // the cell's own state and normals; the next plane may still be on its way
      // the nodes again from shared memory: holding them through the corner vectors would spill
      D3 x[8];
      D3 sm = d3(0., 0., 0.);
#pragma unroll
      for (int a = 0; a < 8; ++a) { x[a] = node(a, 0); sm = sm + x[a]; }
      const D3 xc = .125 * sm;
      const double* const pv = priv + tid;
      const ThermoIn in{V, inv_dt, pv[18 * kColThreads], pv[19 * kColThreads], pv[20 * kColThreads],
                        pv[21 * kColThreads], pv[22 * kColThreads], pv[23 * kColThreads]};
      auto nlo = [&](int d) { const double* b = pv + 3 * d * kColThreads; return d3(b[0], b[kColThreads], b[2 * kColThreads]); };
      auto nhi = [&](int d) { const double* b = pv + (9 + 3 * d) * kColThreads; return d3(b[0], b[kColThreads], b[2 * kColThreads]); };
      auto vn = [&](int a) { return node(a, 3); };
      double Lc = 0.;
      A.xc[c] = xc.x; A.xc[C + c] = xc.y; A.xc[2 * C + c] = xc.z;
      if (A.ph.lc_mode != 0) Lc = face_length(x);
      cell_thermo<K, false, false, NEWTON>(A.ph, A.env, A.fd, c, C, in, Lc, A.st.rho, A.L, A.U[0], A.Vlag, 0., 0., 0.,
                                           0., nullptr);
      face_data<double, HC>(dm, i, j, k, x, xc, A.fd, nlo, nhi, vn);
    }
  }
}

template <int K, bool HC, int STRIP, bool NEWTON>
__global__ void __launch_bounds__(kColThreads, STRIP == kColStrip ? 3 : 2) k_cyc_lagrange_columns(const __grid_constant__ CycleArgs a) {
  lagrange_columns<K, HC, STRIP, NEWTON>(a, blockIdx.x, blockIdx.y);
}

// The same over a batch's column table (instance, chunk, segment).  The
// instance's arguments are read from shared memory where they are used:
// fifty pointers in registers would spill.
template <int K, bool HC, int STRIP, bool NEWTON>
__global__ void __launch_bounds__(kColThreads, STRIP == kColStrip ? 3 : 2) k_bat_lagrange_columns(const CycleArgs* __restrict__ D,
                                                                         const int4* __restrict__ W, int nw) {
  __shared__ CycleArgs a;
  for (int w = blockIdx.x; w < nw; w += gridDim.x) {
    const int4 t = W[w];
    __syncthreads();                       // the previous item's reads are done
    static_assert(sizeof(CycleArgs) % sizeof(double) == 0, "copied as doubles");
    for (int x = threadIdx.x; x < (int)(sizeof(CycleArgs) / sizeof(double)); x += kColThreads)
      reinterpret_cast<double*>(&a)[x] = reinterpret_cast<const double*>(D + t.x)[x];
    __syncthreads();
    lagrange_columns<K, HC, STRIP, NEWTON>(a, t.y, t.z);
  }
}

// Whether a context's FP64 cell kernel takes columns: not on small meshes, whose
// few blocks do not hide the copy of the first planes (100x5x5: 13.9 us against
// 9.9 us for one thread a cell; 37^3, 50,653 cells: 14.8 against 13.1), and not
// where the layers leave threads idle (col_filled).  The mixed form keeps one
// thread a cell: in columns it took 236 to 294 us on Sedov 128^3 against 219 to 230.
constexpr long long kColMinCells = 65536;
inline bool takes_columns(const CycleArgs& a) {
  return !a.ph.precision && a.dm.C >= kColMinCells &&
         col_filled(a.dm.C, (long long)kColThreads * col_blocks(a.dm.nx, a.dm.ny) * a.dm.nz);
}

template <int K, bool HC, bool NEWTON>
static void launch_columns(const CycleArgs& a, cudaStream_t s) {
  const Dims& dm = a.dm;
  const int strip = col_strip(dm.nx);
  const size_t smem = col_smem(strip);
  auto kern = strip == kColStrip ? k_cyc_lagrange_columns<K, HC, kColStrip, NEWTON>
                                 : k_cyc_lagrange_columns<K, HC, kColStripWide, NEWTON>;
  smem_opt_in((const void*)kern, smem);
  kern<<<dim3(col_blocks(dm.nx, dm.ny), col_segments(dm.nx, dm.ny, dm.nz)), kColThreads, smem, s>>>(a);
}

// The cell kernel of a context, all but schema-csts.
template <int K, bool NEWTON>
static void launch_cells(const CycleArgs& a, cudaStream_t s) {
  const bool hc = a.fd.h != nullptr;               // cell widths: order 3 or the generalised limiters
  if (takes_columns(a)) {
    if (hc) launch_columns<K, true, NEWTON>(a, s);
    else launch_columns<K, false, NEWTON>(a, s);
    return;
  }
  int linear;
  const dim3 nbc = cell_grid(a.dm, linear);
  auto kern = a.ph.precision ? k_cyc_lagrange_cells<K, float, false, NEWTON>
                             : (hc ? k_cyc_lagrange_cells<K, double, true, NEWTON> : k_cyc_lagrange_cells<K, double, false, NEWTON>);
  kern<<<nbc, 128, 0, s>>>(a.dm, a.S, a.ph, a.x0, a.vh, a.n0, a.st.rho, a.st.e, a.st.q, a.st.p, a.st.cs, a.st.mass,
                           a.cqs, a.cqs32, a.L, a.U[0], a.xc, a.fd, a.env, a.Vlag, linear);
}
template <int K>
static void launch_cells(const CycleArgs& a, cudaStream_t s) {
  if (a.ph.with_newton) launch_cells<K, true>(a, s);
  else launch_cells<K, false>(a, s);
}

template <int K, bool HC, bool NEWTON>
static void launch_bat_columns(const BatchPlan& P, cudaStream_t s, KernelMarks* m) {
  const size_t smem = col_smem(P.col_strip);
  auto kern = P.col_strip == kColStrip ? k_bat_lagrange_columns<K, HC, kColStrip, NEWTON>
                                       : k_bat_lagrange_columns<K, HC, kColStripWide, NEWTON>;
  smem_opt_in((const void*)kern, smem);
  if (P.ncwork > 0)
    kern<<<persistent_grid((const void*)kern, kColThreads, smem, P.ncwork, P.occ_pct[BK_LCELLS]), kColThreads, smem, s>>>(
        P.descs, P.cwork, P.ncwork);
  mark(m, BK_LCELLS, s);
}
// What of a batch takes no columns: the cell tiles of BK_LCELLS.
template <int K, typename R, bool HC, bool CSTS, bool NEWTON>
__global__ void __launch_bounds__(128, sizeof(R) == 4 ? 5 : 3) k_bat_lagrange_cells(const CycleArgs* __restrict__ D,
                                                                                   const int4* __restrict__ W, int nw) {
  for (int w = blockIdx.x; w < nw; w += gridDim.x) {
    const int4 t = W[w];
    const CycleArgs& a = D[t.x];
    k_cyc_lagrange_cells_body<K, R, CSTS, HC, NEWTON>(a.dm, a.S, a.ph, a.x0, a.vh, a.n0, a.st.rho, a.st.e, a.st.q, a.st.p,
                                              a.st.cs, a.st.mass, a.cqs, CSTS ? nullptr : a.cqs32, a.L, a.U[0], a.xc,
                                              a.fd, a.env, a.Vlag, t.y, t.z, t.w, a.vnb, a.pf);
  }
}

template <int K, typename R, bool HC, bool CSTS, bool NEWTON>
static void launch_bat_tiles(const BatchPlan& P, cudaStream_t s, KernelMarks* m) {
  auto kern = k_bat_lagrange_cells<K, R, HC, CSTS, NEWTON>;
  if (P.nwork[BK_LCELLS] > 0)
    kern<<<persistent_grid((const void*)kern, 128, 0, P.nwork[BK_LCELLS], P.occ_pct[BK_LCELLS]), 128, 0, s>>>(
        P.descs, P.work[BK_LCELLS], P.nwork[BK_LCELLS]);
  mark(m, BK_LCELLS, s);
}

// The cell kernel of a batch, all but schema-csts.
template <int K, typename R, bool HC, bool NEWTON>
static void launch_bat_cells(const BatchPlan& P, cudaStream_t s, KernelMarks* m) {
  if constexpr (sizeof(R) == 8) {
    if (P.columns) { launch_bat_columns<K, HC, NEWTON>(P, s, m); return; }
  }
  launch_bat_tiles<K, R, HC, false, NEWTON>(P, s, m);
}
template <int K, typename R, bool HC>
static void launch_bat_cells(const BatchPlan& P, cudaStream_t s, KernelMarks* m) {
  if (P.newton) launch_bat_cells<K, R, HC, true>(P, s, m);
  else launch_bat_cells<K, R, HC, false>(P, s, m);
}

}  // namespace mhy
