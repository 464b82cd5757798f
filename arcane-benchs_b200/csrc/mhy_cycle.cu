// mhy_cycle.cu -- fused sm_100a kernels of one Lagrange + ADI-remap cycle
// (single environment, plain FP64).
//
// Ten launches per cycle:
//   k_cyc_lagrange_nodes      nodes: force from the previous corner vectors, velocity, BCs
//   k_cyc_lagrange_cells      cells: corner vectors, volume, length, density, viscosity, energy,
//                             remap variables U, and the geometry of each cell's low faces
//   3 x sweep, cells         face gradients, limited cell gradients, upwind face values,
//                             fluxes and U update (1D stencil along d); the last one also
//                             finalises the cell state (remapVariables + EOS)
//   3 x sweep, nodes         dual mass fluxes, limited nodal gradients, upwind momentum and
//                             kinetic-energy update; the last one also gives the node
//                             velocity and mass
//   k_dt_min, k_dt_finish     CFL reduction and the new dt
//
// Every expression keeps the operation order of the reference (see the
// citations), so with --fmad=false the results equal the CPU oracle bit for bit.
#include <map>
#include <mutex>

#include "mhy_lagrange.cuh"
#include "mhy_line.cuh"
#include "mhy_march.cuh"

namespace mhy {

// ------------------------------------------------------------------------
// Lagrange phase, nodes: SaveValuesAtN (v_n = v, x = x0), UpdateVelocity,
// ApplyBoundaryCondition (MahycoModule.cc:308-450, 589-665, 936-1004).

// Nodal force sum_c (p_c + q_c) cqs_c[node] over the up to 8 cells of node
// (i, j, k) in increasing cell id (updateForceAndVelocity, MahycoModule.cc:638-651).
// SUMMED: p already holds p + q (q unused).
template <typename CQ, bool SUMMED = false>
__device__ __forceinline__ D3 node_force(const Dims& dm, int i, int j, int k, const double* __restrict__ p,
                                         const double* __restrict__ q, const CQ* __restrict__ cqs) {
  const int loc[2][2][2] = {{{0, 4}, {3, 7}}, {{1, 5}, {2, 6}}};
  D3 F = d3(0, 0, 0);
#pragma unroll
  for (int dk = 1; dk >= 0; --dk)
#pragma unroll
    for (int dj = 1; dj >= 0; --dj)
#pragma unroll
      for (int di = 1; di >= 0; --di) {
        const int ci = i - di, cj = j - dj, ck = k - dk;
        if (ci < 0 || cj < 0 || ck < 0 || ci >= dm.nx || cj >= dm.ny || ck >= dm.nz) continue;
        const long long c = dm.cid(ci, cj, ck);
        const int l = loc[di][dj][dk];
        const double pq = SUMMED ? p[c] : p[c] + q[c];
        F = F + pq * d3((double)cqs[(l * 3 + 0) * dm.C + c], (double)cqs[(l * 3 + 1) * dm.C + c],
                        (double)cqs[(l * 3 + 2) * dm.C + c]);
      }
  return F;
}

// The same sum with every load issued before the first addition: the loads of
// the form above follow one another in groups, cell by cell, which costs little
// where many warps are in flight and eight round trips where few are.
template <typename CQ>
__device__ __forceinline__ D3 node_force_gathered(const Dims& dm, int i, int j, int k, const double* __restrict__ p,
                                                  const double* __restrict__ q, const CQ* __restrict__ cqs) {
  const int loc[2][2][2] = {{{0, 4}, {3, 7}}, {{1, 5}, {2, 6}}};
  double pc[8], qc[8];
  CQ w[8][3];
  bool in[8];
#pragma unroll
  for (int a = 0; a < 8; ++a) {
    const int di = ~a & 1, dj = ~(a >> 1) & 1, dk = ~(a >> 2) & 1, ci = i - di, cj = j - dj, ck = k - dk;
    in[a] = !(ci < 0 || cj < 0 || ck < 0 || ci >= dm.nx || cj >= dm.ny || ck >= dm.nz);
    const long long c = in[a] ? dm.cid(ci, cj, ck) : 0;
    const int l = loc[di][dj][dk];
    pc[a] = p[c];
    qc[a] = q[c];
#pragma unroll
    for (int e = 0; e < 3; ++e) w[a][e] = cqs[(l * 3 + e) * dm.C + c];
  }
  D3 F = d3(0, 0, 0);
#pragma unroll
  for (int a = 0; a < 8; ++a)
    if (in[a]) F = F + (pc[a] + qc[a]) * d3((double)w[a][0], (double)w[a][1], (double)w[a][2]);
  return F;
}

// vnb (schema-csts only, else null): v_n taken back from n to n-1/2 with
// the same force first, updateVelocityBackward (MahycoModule.cc:693, 743-781),
// and kept for the energy and the remap face velocities.
template <typename CQ, bool GATHERED = false>
__device__ __forceinline__ void k_cyc_lagrange_nodes_body(Dims dm, const Scalars* __restrict__ S,
    const double* __restrict__ p, const double* __restrict__ q, const CQ* __restrict__ cqs,
    const double* __restrict__ nm, const double* __restrict__ v, const uint16_t* __restrict__ bcmask, BCTable bct,
    double* __restrict__ vh, double* __restrict__ vnb,
    int bx_, int by_, int bz_) {
  int i, j, k;
  if (!block_item(dm.nx + 1, dm.ny + 1, dm.nz + 1, bx_, by_, bz_, i, j, k)) return;
  const long long n = dm.nid(i, j, k);
  const double dtv = 0.5 * (S->old_dt + S->dt);
  D3 F;
  if constexpr (GATHERED) F = node_force_gathered<CQ>(dm, i, j, k, p, q, cqs);
  else F = node_force<CQ>(dm, i, j, k, p, q, cqs);
  const double s = dtv / nm[n];
  D3 vb = d3(v[n], v[dm.N + n], v[2 * dm.N + n]);
  if (vnb) {
    const double sb = (-0.5 * S->old_dt) / nm[n];
    vb = vb + sb * F;
    vnb[n] = vb.x; vnb[dm.N + n] = vb.y; vnb[2 * dm.N + n] = vb.z;
  }
  D3 u = vb + s * F;
  const unsigned mask = bcmask[n];
  if (mask)
    for (int b = 0; b < bct.nb; ++b)
      if (mask >> b & 1u) {
        if (bct.type[b] == 0) u.x = bct.value[b];
        else if (bct.type[b] == 1) u.y = bct.value[b];
        else u.z = bct.value[b];
      }
  vh[n] = u.x; vh[dm.N + n] = u.y; vh[2 * dm.N + n] = u.z;
}

template <typename CQ, bool GATHERED>
__global__ void __launch_bounds__(128) k_cyc_lagrange_nodes(Dims dm, const Scalars* __restrict__ S,
    const double* __restrict__ p, const double* __restrict__ q, const CQ* __restrict__ cqs,
    const double* __restrict__ nm, const double* __restrict__ v, const uint16_t* __restrict__ bcmask, BCTable bct,
    double* __restrict__ vh, double* __restrict__ vnb) {
  k_cyc_lagrange_nodes_body<CQ, GATHERED>(dm, S, p, q, cqs, nm, v, bcmask, bct, vh, vnb, blockIdx.x, -1, 0);
}

// schema-csts, updateVelocityForward (PrepareRemap.cc:456, MahycoModule.cc:
// 792-831): vf = v_h + (0.5 dt / m) F with this cycle's corner vectors and the
// current pressure plus this cycle's pseudo-viscosity (pq, summed by the cell
// kernel; no boundary condition); xl = the Lagrangian node coordinates
// x0 + v_h dt, which the remap keeps.
__device__ __forceinline__ void csts_forward_item(const Dims& dm, const Scalars* __restrict__ S,
    const double* __restrict__ pq, const double* __restrict__ cqs,
    const double* __restrict__ nm, const double* __restrict__ x0, const double* __restrict__ vh,
    double* __restrict__ vf, double* __restrict__ xl, int bx_, int by_, int bz_) {
  int i, j, k;
  if (!block_item(dm.nx + 1, dm.ny + 1, dm.nz + 1, bx_, by_, bz_, i, j, k)) return;
  const long long n = dm.nid(i, j, k), N = dm.N;
  const double dt = S->dt;
  const D3 F = node_force<double, true>(dm, i, j, k, pq, nullptr, cqs);
  const double s = (0.5 * dt) / nm[n];
  const D3 u = d3(vh[n], vh[N + n], vh[2 * N + n]);
  const D3 w = u + s * F;
  vf[n] = w.x; vf[N + n] = w.y; vf[2 * N + n] = w.z;
#pragma unroll
  for (int a = 0; a < 3; ++a) xl[a * N + n] = x0[a * N + n] + vh[a * N + n] * dt;
}

__global__ void __launch_bounds__(128) k_csts_forward(Dims dm, const Scalars* __restrict__ S,
    const double* __restrict__ pq, const double* __restrict__ cqs,
    const double* __restrict__ nm, const double* __restrict__ x0, const double* __restrict__ vh,
    double* __restrict__ vf, double* __restrict__ xl) {
  csts_forward_item(dm, S, pq, cqs, nm, x0, vh, vf, xl, blockIdx.x, -1, 0);
}

// schema-csts remap face velocities (PrepareRemap.cc:69-79): u_f =
// (0.25 sum over the face nodes of 0.5 (v + v_n)) . n0, with v the forward
// velocity and v_n the backward one, for every face of every direction.
__device__ __forceinline__ void csts_face_u_item(const Dims& dm, const double* __restrict__ vf,
    const double* __restrict__ vnb, const double* __restrict__ n0, const FaceData& fd, long long f) {
  if (f >= dm.F) return;
  int d; long long t;
  if (f < dm.Fx) { d = 0; t = f; } else if (f < dm.Fx + dm.Fy) { d = 1; t = f - dm.Fx; } else { d = 2; t = f - dm.Fx - dm.Fy; }
  int i, j, k; dm.fdijk(d, t, i, j, k);
  long long fn[4]; face_node_ids(dm, d, i, j, k, fn);
  const long long N = dm.N;
  D3 vm = d3(0., 0., 0.);
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const long long m = fn[a];
    vm = vm + 0.5 * (d3(vf[m], vf[N + m], vf[2 * N + m]) + d3(vnb[m], vnb[N + m], vnb[2 * N + m]));
  }
  fd.u[d][t] = dot(.25 * vm, d3(n0[f], n0[dm.F + f], n0[2 * dm.F + f]));
}

__global__ void __launch_bounds__(128) k_csts_face_u(Dims dm, const double* __restrict__ vf,
    const double* __restrict__ vnb, const double* __restrict__ n0, FaceData fd) {
  csts_face_u_item(dm, vf, vnb, n0, fd, blockIdx.x * (long long)blockDim.x + threadIdx.x);
}


// Cell sweep along x: lanes run along the rows, loads and stores as they are.
// cells_x_line is one lane's loads and line step.  The body runs it with
// speculative FP64 quotients (not in the pente-borne form, whose quotients
// stay exact); in a warp where any lane's were out of range it recomputes
// the segment exactly out of line (cells_x_line_exact reloads the inputs, so
// that none of them stays live across the common path), then stores.
template <bool LAST, typename R, bool O3, bool GL, bool PB, bool SP>
__device__ __forceinline__ void cells_x_line(const Dims& dm, const Scalars* __restrict__ S, const Phys& ph,
    const FaceData& fd, const double* __restrict__ n0, const double* __restrict__ xcs, const double* __restrict__ ofn,
    const double* __restrict__ Uin, const double* __restrict__ Ve, int bx_, double* out,
    unsigned* oor) {
  const int lane = threadIdx.x & 31;
  const int nd = dm.nx, C = (int)dm.C, F = (int)dm.F;
  const RowPos rp = row_pos(bx_, nd, dm.ny, C);
  const int s = rp.s, c = rp.id;                // s: position of this lane's cell along x
  const bool valid = rp.valid;
  const bool inner = valid && s >= 1;                  // this lane's low face is an inner face
  const bool infr = valid && s + 1 <= nd - 1;
  const bool upd = valid && lane >= 2 && lane < 2 + kLineUpd;
  const int t = inner ? c + rp.j + dm.ny * rp.k : 0;   // a row of faces is one longer; x faces come first
  CellIn in;
  in.U[0] = in.U[1] = in.U[2] = in.U[3] = 0.; in.xc[0] = in.xc[1] = in.xc[2] = 0.;
  in.db = in.df = in.u = in.A = 0.; in.n[0] = in.n[1] = in.n[2] = 0.; in.ob = in.of = in.vol = 0.; in.h = 0.;
  if (valid) {
    in.U[0] = Uin[c]; in.U[1] = Uin[C + c]; in.U[2] = Uin[2 * C + c]; in.U[3] = Uin[3 * C + c];
    in.xc[0] = xcs[c]; in.xc[1] = xcs[C + c]; in.xc[2] = xcs[2 * C + c];
    if constexpr (GL || PB) in.h = fd.h[c];
    if constexpr (PB) {
      in.pb[0] = ph.pb_first ? fd.pbphi[c] : 0.; in.pb[1] = ph.pb_first ? fd.pbphi[C + c] : 0.;
      in.pb[2] = fd.pbphi[2 * C + c];
      in.ob = ofn[1 * C + c]; in.of = ofn[4 * C + c];      // every lane's two faces take part
    }
  }
  if (inner) {
    in.db = fd.db[0][t]; in.df = fd.df[0][t]; in.u = fd.u[0][t]; in.A = fd.A[0][t];
    in.n[0] = n0[t]; in.n[1] = n0[F + t]; in.n[2] = n0[2 * F + t];
    if constexpr (O3) {
      const int Fd = (int)dm.Fx;
#pragma unroll
      for (int v = 0; v < 4; ++v) in.pf3[v] = fd.phi3[v * Fd + t];
    }
  }
  if (upd) {
    in.ob = ofn[1 * C + c]; in.of = ofn[4 * C + c];
    if (LAST) in.vol = Ve[c];
  }
  cell_line<LAST, R, O3, GL, PB, SP>(ph, S->dt, S, valid, inner, infr, upd, in, out, oor);
}

template <bool LAST, typename R, bool O3, bool GL, bool PB>
__device__ __noinline__ LineOut<LAST ? kCellOutLast : kCellOutMid> cells_x_line_exact(Dims dm, const Scalars* S,
    Phys ph, FaceData fd, const double* n0, const double* xcs, const double* ofn, const double* Uin, const double* Ve,
    int bx_) {
  LineOut<LAST ? kCellOutLast : kCellOutMid> o;
  cells_x_line<LAST, R, O3, GL, PB, false>(dm, S, ph, fd, n0, xcs, ofn, Uin, Ve, bx_, o.v, nullptr);
  return o;
}

template <bool LAST, typename R, bool O3 = false, bool GL = false, bool PB = false>
__device__ __forceinline__ void k_cyc_sweep_cells_x_body(Dims dm, const Scalars* __restrict__ S,
    Phys ph, FaceData fd, const double* __restrict__ n0, const double* __restrict__ xcs,
    const double* __restrict__ ofn, const double* __restrict__ Uin, double* __restrict__ Uout,
    double* __restrict__ dpf, CellState st,
    int bx_) {
  constexpr int NO = LAST ? kCellOutLast : kCellOutMid;
  const int lane = threadIdx.x & 31;
  if (row_first(bx_) >= (int)dm.C) return;             // whole warp leaves together
  double out[NO];
  if constexpr (sizeof(R) == 8 && !PB) {
    unsigned oor = 0u;
    cells_x_line<LAST, R, O3, GL, PB, true>(dm, S, ph, fd, n0, xcs, ofn, Uin, st.Ve, bx_, out, &oor);
    if (__any_sync(0xffffffffu, oor != 0u)) {
      const auto o = cells_x_line_exact<LAST, R, O3, GL, PB>(dm, S, ph, fd, n0, xcs, ofn, Uin, st.Ve, bx_);
#pragma unroll
      for (int a = 0; a < NO; ++a) out[a] = o.v[a];
    }
  } else {
    cells_x_line<LAST, R, O3, GL, PB, false>(dm, S, ph, fd, n0, xcs, ofn, Uin, st.Ve, bx_, out, nullptr);
  }
  const int C = (int)dm.C, c = row_first(bx_) - 2 + lane;
  if (c >= C || lane < 2 || lane >= 2 + kLineUpd) return;
  if (!LAST) {
#pragma unroll
    for (int v = 0; v < 4; ++v) Uout[v * C + c] = out[v];
    dpf[c] = out[4];
  } else {
    st.rho[c] = out[0]; st.e[c] = out[1]; st.q[c] = out[2]; st.mass[c] = out[3]; st.p[c] = out[4]; st.cs[c] = out[5];
    dpf[c] = out[6];
    if (st.mf) st.mf[c] = out[7];
  }
}

template <bool LAST, typename R, bool O3 = false, bool GL = false, bool PB = false>
__global__ void __launch_bounds__(32 * kLineWarps, kLineMinBlocks) k_cyc_sweep_cells_x(Dims dm, const Scalars* __restrict__ S,
    Phys ph, FaceData fd, const double* __restrict__ n0, const double* __restrict__ xcs,
    const double* __restrict__ ofn, const double* __restrict__ Uin, double* __restrict__ Uout,
    double* __restrict__ dpf, CellState st) {
  k_cyc_sweep_cells_x_body<LAST, R, O3, GL, PB>(dm, S, ph, fd, n0, xcs, ofn, Uin, Uout, dpf, st, blockIdx.x);
}

// Cell sweep along y (D = 1) or z (D = 2), staged through shared memory.
// Block (bx, by, bz): x = 8 bx .. 8 bx + 7, positions 28 by - 2 .. 28 by + 29
// along D, and bz = the remaining coordinate (z for D = 1, y for D = 2).
template <bool LAST, int W, bool O3 = false>
struct CellTileSize {
  static constexpr int NB = LAST ? 17 : 16;           // staged input arrays
  static constexpr int NA = NB + (O3 ? 4 : 0);        // + the order-3 face values
  static constexpr size_t bytes = (size_t)NA * TileGeom<W>::arr * sizeof(double);
};

// One lane's line step of a cell y/z sweep, from the staged tile (each warp
// reads only its own tile row, which no other warp writes).
template <int D, bool LAST, typename R, int W, bool O3, bool GL, bool PB, bool SP>
__device__ __forceinline__ void cells_t_line(const Dims& dm, const Scalars* __restrict__ S, const Phys& ph,
    const FaceData& fd, int bx_, int by_, int bz_, double* out, unsigned* oor) {
  constexpr int NB = CellTileSize<LAST, W, O3>::NB;
  constexpr int kTileArr = TileGeom<W>::arr, kTileLd = TileGeom<W>::ld;
  extern __shared__ double smem_dyn[];
  const double* tile = smem_dyn;                      // [NA][W][ld]
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int i0 = bx_ * W, seg0 = by_ * kLineUpd - 2, o = bz_;
  const int nd = dm.ncd(D), C = (int)dm.C;
  // line w, position lane
  const int s = seg0 + lane;
  const bool line_ok = i0 + w < dm.nx;
  const bool valid = line_ok && s >= 0 && s < nd;
  const bool inner = line_ok && s >= 1 && s <= nd - 1;
  const bool infr = s + 1 <= nd - 1;
  const bool upd = valid && lane >= 2 && lane < 2 + kLineUpd;
  const double* row = tile + w * kTileLd + lane;
  CellIn in;
  in.U[0] = row[0]; in.U[1] = row[kTileArr]; in.U[2] = row[2 * kTileArr]; in.U[3] = row[3 * kTileArr];
  in.xc[0] = row[4 * kTileArr]; in.xc[1] = row[5 * kTileArr]; in.xc[2] = row[6 * kTileArr];
  in.db = row[7 * kTileArr]; in.df = row[8 * kTileArr]; in.u = row[9 * kTileArr]; in.A = row[10 * kTileArr];
  in.n[0] = row[11 * kTileArr]; in.n[1] = row[12 * kTileArr]; in.n[2] = row[13 * kTileArr];
  in.ob = row[14 * kTileArr]; in.of = row[15 * kTileArr];
  in.vol = LAST ? row[(NB - 1) * kTileArr] : 0.;
  in.h = 0.;
  in.pb[0] = in.pb[1] = in.pb[2] = 0.;
  if ((GL || PB) && valid) {
    const int i = i0 + w;
    const int c = D == 1 ? i + dm.nx * (s + dm.ny * o) : i + dm.nx * (o + dm.ny * s);
    in.h = fd.h[D * C + c];
    if constexpr (PB) {
      if (ph.pb_first) { in.pb[0] = fd.pbphi[c]; in.pb[1] = fd.pbphi[C + c]; }
      in.pb[2] = fd.pbphi[2 * C + c];
    }
  }
  if constexpr (O3) {
#pragma unroll
    for (int a = 0; a < 4; ++a) in.pf3[a] = row[(NB + a) * kTileArr];
  }
  cell_line<LAST, R, O3, GL, PB, SP>(ph, S->dt, S, valid, inner, infr, upd, in, out, oor);
}

template <int D, bool LAST, typename R, int W, bool O3, bool GL, bool PB>
__device__ __noinline__ LineOut<LAST ? kCellOutLast : kCellOutMid> cells_t_line_exact(Dims dm, const Scalars* S,
    Phys ph, FaceData fd, int bx_, int by_, int bz_) {
  LineOut<LAST ? kCellOutLast : kCellOutMid> o;
  cells_t_line<D, LAST, R, W, O3, GL, PB, false>(dm, S, ph, fd, bx_, by_, bz_, o.v, nullptr);
  return o;
}

template <int D, bool LAST, typename R, int W, bool O3 = false, bool GL = false, bool PB = false>
__device__ __forceinline__ void k_cyc_sweep_cells_t_body(Dims dm, const Scalars* __restrict__ S,
    Phys ph, FaceData fd, const double* __restrict__ n0, const double* __restrict__ xcs,
    const double* __restrict__ ofn, const double* __restrict__ Uin, double* __restrict__ Uout,
    double* __restrict__ dpf, CellState st,
    int bx_, int by_, int bz_) {
  constexpr int NA = CellTileSize<LAST, W, O3>::NA, NB = CellTileSize<LAST, W, O3>::NB;
  constexpr int kTileArr = TileGeom<W>::arr, kTileLd = TileGeom<W>::ld;
  extern __shared__ double smem_dyn[];
  double* tile = smem_dyn;                            // [NA][W][ld]
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int i0 = bx_ * W, seg0 = by_ * kLineUpd - 2, o = bz_;
  const int nd = dm.ncd(D), C = (int)dm.C, F = (int)dm.F;
  const int foff = D == 1 ? (int)dm.Fx : (int)(dm.Fx + dm.Fy);
  const int lb = D == 1 ? 2 : 0, lf = D == 1 ? 5 : 3;   // back / front faces of d in cell-face order
  // thread (x, p) of the staging layout; also used for the stores at the end
  const int sx = tid % W, sp = tid / W;
  const int si = i0 + sx, ss = seg0 + sp;
  const bool s_valid = si < dm.nx && ss >= 0 && ss < nd;
  const int sc = D == 1 ? si + dm.nx * (ss + dm.ny * o) : si + dm.nx * (o + dm.ny * ss);
  {
    const bool s_inner = si < dm.nx && ss >= 1 && ss <= nd - 1;
    const int st_ = D == 1 ? si + dm.nx * (ss + (dm.ny + 1) * o) : sc;   // face index within direction D
    double v[NA];
#pragma unroll
    for (int a = 0; a < NA; ++a) v[a] = 0.;
    if (s_valid) {
      v[0] = Uin[sc]; v[1] = Uin[C + sc]; v[2] = Uin[2 * C + sc]; v[3] = Uin[3 * C + sc];
      v[4] = xcs[sc]; v[5] = xcs[C + sc]; v[6] = xcs[2 * C + sc];
      v[14] = ofn[lb * C + sc]; v[15] = ofn[lf * C + sc];
      if (LAST) v[NB - 1] = st.Ve[sc];
    }
    if (s_inner) {
      v[7] = fd.db[D][st_]; v[8] = fd.df[D][st_]; v[9] = fd.u[D][st_]; v[10] = fd.A[D][st_];
      const int f = foff + st_;
      v[11] = n0[f]; v[12] = n0[F + f]; v[13] = n0[2 * F + f];
      if constexpr (O3) {
        const int Fd = (int)(D == 1 ? dm.Fy : dm.F - dm.Fx - dm.Fy);
#pragma unroll
        for (int a = 0; a < 4; ++a) v[NB + a] = fd.phi3[a * Fd + st_];
      }
    }
#pragma unroll
    for (int a = 0; a < NA; ++a) tile[a * kTileArr + sx * kTileLd + sp] = v[a];
  }
  __syncthreads();
  constexpr int NO = LAST ? kCellOutLast : kCellOutMid;
  double out[NO];
  if constexpr (sizeof(R) == 8 && !PB) {
    unsigned oor = 0u;
    cells_t_line<D, LAST, R, W, O3, GL, PB, true>(dm, S, ph, fd, bx_, by_, bz_, out, &oor);
    if (__any_sync(0xffffffffu, oor != 0u)) {
      const auto o2 = cells_t_line_exact<D, LAST, R, W, O3, GL, PB>(dm, S, ph, fd, bx_, by_, bz_);
#pragma unroll
      for (int a = 0; a < NO; ++a) out[a] = o2.v[a];
    }
  } else {
    cells_t_line<D, LAST, R, W, O3, GL, PB, false>(dm, S, ph, fd, bx_, by_, bz_, out, nullptr);
  }
  const int s = seg0 + lane;
  const bool upd = i0 + w < dm.nx && s >= 0 && s < nd && lane >= 2 && lane < 2 + kLineUpd;
  double* row = tile + w * kTileLd + lane;
  // each lane overwrites only the tile column it read itself
  if (upd) {
#pragma unroll
    for (int a = 0; a < NO; ++a) row[a * kTileArr] = out[a];
  }
  __syncthreads();
  if (!(s_valid && sp >= 2 && sp < 2 + kLineUpd)) return;
  const double* r = tile + sx * kTileLd + sp;
  if (!LAST) {
#pragma unroll
    for (int v = 0; v < 4; ++v) Uout[v * C + sc] = r[v * kTileArr];
    dpf[sc] = r[4 * kTileArr];
  } else {
    st.rho[sc] = r[0]; st.e[sc] = r[kTileArr]; st.q[sc] = r[2 * kTileArr]; st.mass[sc] = r[3 * kTileArr];
    st.p[sc] = r[4 * kTileArr]; st.cs[sc] = r[5 * kTileArr]; dpf[sc] = r[6 * kTileArr];
    if (st.mf) st.mf[sc] = r[7 * kTileArr];
  }
}

template <int D, bool LAST, typename R, int W, bool O3 = false, bool GL = false, bool PB = false>
__global__ void __launch_bounds__(32 * W, TileGeom<W>::minb) k_cyc_sweep_cells_t(Dims dm, const Scalars* __restrict__ S,
    Phys ph, FaceData fd, const double* __restrict__ n0, const double* __restrict__ xcs,
    const double* __restrict__ ofn, const double* __restrict__ Uin, double* __restrict__ Uout,
    double* __restrict__ dpf, CellState st) {
  k_cyc_sweep_cells_t_body<D, LAST, R, W, O3, GL, PB>(dm, S, ph, fd, n0, xcs, ofn, Uin, Uout, dpf, st, blockIdx.x, blockIdx.y,
                                              blockIdx.z);
}

void smem_opt_in(const void* kernel, size_t bytes) {
  if (bytes <= 48 * 1024) return;
  static std::mutex mu;
  static std::map<std::pair<const void*, int>, size_t> done;
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lk(mu);
  size_t& have = done[std::make_pair(kernel, dev)];
  if (have >= bytes) return;
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  have = bytes;
}


// ------------------------------------------------------------------------
// Host-side launchers.
template <int D, bool LAST, typename R, int W, bool O3 = false, bool GL = false, bool PB = false>
static void sweep_cells_t_w(const CycleArgs& a, const double* Uin, double* Uout, cudaStream_t s) {
  const Dims& dm = a.dm;
  const int nseg = (dm.ncd(D) + kLineUpd - 1) / kLineUpd;
  const dim3 g((dm.nx + W - 1) / W, nseg, D == 1 ? dm.nz : dm.ny);
  const size_t smem = CellTileSize<LAST, W, O3>::bytes;
  auto kern = k_cyc_sweep_cells_t<D, LAST, R, W, O3, GL, PB>;
  smem_opt_in((const void*)kern, smem);
  kern<<<g, 32 * W, smem, s>>>(dm, a.S, a.ph, a.fd, a.n0, a.xc, a.ofn, Uin, Uout, a.dpf, a.st);
}

template <int D, bool LAST, typename R>
static void sweep_cells_t(const CycleArgs& a, const double* Uin, double* Uout, cudaStream_t s) {
  if constexpr (sizeof(R) == 8) {
    const bool o3 = a.ph.ordre_projection == 3, gl = a.ph.ordre_projection > 1 && a.ph.lim_cell >= 3;
    if (a.ph.pb) { sweep_cells_t_w<D, LAST, R, kLineWarps, false, false, true>(a, Uin, Uout, s); return; }
    if (o3 && gl) { sweep_cells_t_w<D, LAST, R, kLineWarps, true, true>(a, Uin, Uout, s); return; }
    if (o3) { sweep_cells_t_w<D, LAST, R, kLineWarps, true, false>(a, Uin, Uout, s); return; }
    if (gl) { sweep_cells_t_w<D, LAST, R, kLineWarps, false, true>(a, Uin, Uout, s); return; }
  }
  if constexpr (sizeof(R) == 4) {
    if (march_cells(a.dm.N, 1)) { sweep_cells_launch_m<D, LAST>(a, LAST ? 2 : (Uin == a.U[0] ? 0 : 1), s); return; }
  }
  const int w = a.lines[BK_CELLS_X + D];
  if (w == 32) sweep_cells_t_w<D, LAST, R, 32>(a, Uin, Uout, s);
  else if (w == 16) sweep_cells_t_w<D, LAST, R, 16>(a, Uin, Uout, s);
  else sweep_cells_t_w<D, LAST, R, 8>(a, Uin, Uout, s);
}

template <int D, typename R>
static void sweep_cells_d(const CycleArgs& a, bool last, const double* Uin, double* Uout, cudaStream_t s) {
  const Dims& dm = a.dm;
  const int T = 32 * kLineWarps;
  if constexpr (D == 0) {
    const int g = row_chunks(dm.C);
    const bool o3 = sizeof(R) == 8 && a.ph.ordre_projection == 3;
    const bool gl = sizeof(R) == 8 && a.ph.ordre_projection > 1 && a.ph.lim_cell >= 3;
    if constexpr (sizeof(R) == 8) {
      if (a.ph.pb) {
        auto kern = last ? k_cyc_sweep_cells_x<true, R, false, false, true> : k_cyc_sweep_cells_x<false, R, false, false, true>;
        kern<<<g, T, 0, s>>>(dm, a.S, a.ph, a.fd, a.n0, a.xc, a.ofn, Uin, Uout, a.dpf, a.st);
        return;
      }
    }
    if (o3 || gl) {
      auto kern = o3 ? (gl ? (last ? k_cyc_sweep_cells_x<true, R, true, true> : k_cyc_sweep_cells_x<false, R, true, true>)
                           : (last ? k_cyc_sweep_cells_x<true, R, true, false> : k_cyc_sweep_cells_x<false, R, true, false>))
                     : (last ? k_cyc_sweep_cells_x<true, R, false, true> : k_cyc_sweep_cells_x<false, R, false, true>);
      kern<<<g, T, 0, s>>>(dm, a.S, a.ph, a.fd, a.n0, a.xc, a.ofn, Uin, Uout, a.dpf, a.st);
    } else if (last) {
      k_cyc_sweep_cells_x<true, R><<<g, T, 0, s>>>(dm, a.S, a.ph, a.fd, a.n0, a.xc, a.ofn, Uin, Uout, a.dpf, a.st);
    } else {
      k_cyc_sweep_cells_x<false, R><<<g, T, 0, s>>>(dm, a.S, a.ph, a.fd, a.n0, a.xc, a.ofn, Uin, Uout, a.dpf, a.st);
    }
  } else {
    if (last) sweep_cells_t<D, true, R>(a, Uin, Uout, s);
    else sweep_cells_t<D, false, R>(a, Uin, Uout, s);
  }
}

// Node kernel: 128 consecutive nodes per block (rows of nx+1 nodes would leave
// most of a second block idle).
void launch_lagrange_nodes(const CycleArgs& a, cudaStream_t s) {
  const unsigned nbn = (unsigned)((a.dm.N + 127) / 128);
  const bool few = a.dm.C < kSmallMesh;
  if (a.ph.precision) {
    auto kern = few ? k_cyc_lagrange_nodes<float, true> : k_cyc_lagrange_nodes<float, false>;
    kern<<<nbn, 128, 0, s>>>(a.dm, a.S, a.st.p, a.st.q, a.cqs32, a.nm, a.v, a.bcmask, a.bct, a.vh, nullptr);
  } else {
    auto kern = few ? k_cyc_lagrange_nodes<double, true> : k_cyc_lagrange_nodes<double, false>;
    kern<<<nbn, 128, 0, s>>>(a.dm, a.S, a.st.p, a.st.q, a.cqs, a.nm, a.v, a.bcmask, a.bct, a.vh,
                             a.ph.csts ? a.vnb : nullptr);
  }
}

void launch_csts_forward(const CycleArgs& a, cudaStream_t s) {
  const unsigned nbn = (unsigned)((a.dm.N + 127) / 128);
  k_csts_forward<<<nbn, 128, 0, s>>>(a.dm, a.S, a.pf, a.cqs, a.nm, a.x0, a.vh, a.vf, a.xl);
  k_csts_face_u<<<(unsigned)((a.dm.F + 127) / 128), 128, 0, s>>>(a.dm, a.vf, a.vnb, a.n0, a.fd);
}

// The schema-csts form of the FP64 cell kernel (K environments).
template <int K, bool HC>
__global__ void __launch_bounds__(128, 3) k_cyc_lagrange_cells_csts(Dims dm,
    const Scalars* __restrict__ S, Phys ph,
    const double* __restrict__ x0, const double* __restrict__ vh, const double* __restrict__ n0,
    double* __restrict__ rho, const double* __restrict__ e, const double* __restrict__ q,
    const double* __restrict__ p, const double* __restrict__ cs, const double* __restrict__ mass,
    double* __restrict__ cqs, double* __restrict__ L, double* __restrict__ U,
    double* __restrict__ xcs, FaceData fd, EnvState env, double* __restrict__ Vlag, int linear,
    const double* __restrict__ vnb, double* __restrict__ pf) {
  k_cyc_lagrange_cells_body<K, double, true, HC, false>(dm, S, ph, x0, vh, n0, rho, e, q, p, cs, mass, cqs, nullptr, L, U, xcs, fd,
                                             env, Vlag, blockIdx.x, linear ? -1 : (int)blockIdx.y, blockIdx.z, vnb, pf);
}

void launch_lagrange_cells_csts_env(const CycleArgs& a, cudaStream_t s) {
  int linear;
  const dim3 nbc = cell_grid(a.dm, linear);
  const bool hc = a.fd.h != nullptr;
  auto kern = a.K == 2 ? (hc ? k_cyc_lagrange_cells_csts<2, true> : k_cyc_lagrange_cells_csts<2, false>)
            : a.K == 3 ? (hc ? k_cyc_lagrange_cells_csts<3, true> : k_cyc_lagrange_cells_csts<3, false>)
                       : (hc ? k_cyc_lagrange_cells_csts<4, true> : k_cyc_lagrange_cells_csts<4, false>);
  kern<<<nbc, 128, 0, s>>>(a.dm, a.S, a.ph, a.x0, a.vh, a.n0, a.st.rho, a.st.e, a.st.q, a.st.p, a.st.cs, a.st.mass,
                           a.cqs, a.L, a.U[0], a.xc, a.fd, a.env, a.Vlag, linear, a.vnb, a.pf);
}

// Cell kernels: rows of 128 cells when nx is a multiple of 128, else 128
// consecutive cells per block.
dim3 cell_grid(const Dims& dm, int& linear) {
  linear = dm.nx % 128 != 0;
  if (linear) return dim3((unsigned)((dm.C + 127) / 128), 1, 1);
  return dim3(dm.nx / 128, dm.ny, dm.nz);
}

void launch_lagrange_cells(const CycleArgs& a, cudaStream_t s) {
  int linear;
  const dim3 nbc = cell_grid(a.dm, linear);
  const bool hc = a.fd.h != nullptr;               // cell widths: order 3 or the generalised limiters
  if (a.ph.csts) {
    auto kern = hc ? k_cyc_lagrange_cells_csts<1, true> : k_cyc_lagrange_cells_csts<1, false>;
    kern<<<nbc, 128, 0, s>>>(a.dm, a.S, a.ph, a.x0, a.vh, a.n0, a.st.rho, a.st.e, a.st.q, a.st.p, a.st.cs, a.st.mass,
                             a.cqs, a.L, a.U[0], a.xc, a.fd, a.env, a.Vlag, linear, a.vnb, a.pf);
    return;
  }
  launch_cells<1>(a, s);
}

// Three sweeps d = (i + sens) % 3 (RemapADIService.cc:28-30).  U: Lagrange
// writes U[0]; sweeps read U[0] -> U[1] -> U[0] and the last one finalises.
// U_dual: the first sweep builds it from the Lagrange velocity and writes
// ud[0]; then ud[0] -> ud[1]; the last one writes the node velocity and mass.
// Order-3 face values of direction D (RemapADIService.cc:583-641,
// Remap-ordre-3.cc:7-131) for one environment: Phi of the six cells around
// each inner face (clamped at the ends of the line) from the sweep's input U,
// the cell widths h along D and u_f dt; written to fd.phi3 [4][F_D].
template <int D, bool SP>
__device__ __forceinline__ void o3_faces_item(const Dims& dm, const Scalars* __restrict__ S,
    const double* __restrict__ Uin, const FaceData& fd, long long t, unsigned* oor) {
  const long long Fd = D == 0 ? dm.Fx : (D == 1 ? dm.Fy : dm.F - dm.Fx - dm.Fy);
  if (t >= Fd) return;
  int i, j, k; dm.fdijk(D, t, i, j, k);
  const int id = D == 0 ? i : (D == 1 ? j : k), n = dm.ncd(D);
  if (id <= 0 || id >= n) return;                     // boundary faces carry no flux
  // cells bbb, bb, b | f, ff, fff along D, clamped at the ends of the line
  int pos[6];
  pos[2] = id - 1; pos[1] = pos[2] > 0 ? pos[2] - 1 : pos[2]; pos[0] = pos[1] > 0 ? pos[1] - 1 : pos[1];
  pos[3] = id; pos[4] = pos[3] + 1 < n ? pos[3] + 1 : pos[3]; pos[5] = pos[4] + 1 < n ? pos[4] + 1 : pos[4];
  const long long C = dm.C;
  double y[4][6], h[6];
#pragma unroll
  for (int a = 0; a < 6; ++a) {
    const long long c = D == 0 ? dm.cid(pos[a], j, k) : (D == 1 ? dm.cid(i, pos[a], k) : dm.cid(i, j, pos[a]));
    const double U[4] = {Uin[c], Uin[C + c], Uin[2 * C + c], Uin[3 * C + c]};
    double P[4];
    phi_of<double, SP>(U, P, oor);
#pragma unroll
    for (int v = 0; v < 4; ++v) y[v][a] = P[v];
    h[a] = fd.h[D * C + c];
  }
  const O3Coef k3 = o3_coef<SP>(h, fd.u[D][t] * S->dt, oor);
#pragma unroll
  for (int v = 0; v < 4; ++v) fd.phi3[v * Fd + t] = o3_value(k3, y[v]);
}

// The face with speculative quotients, and with plain ones where those raised
// the flag (it reads nothing that it writes).  Bound by its sixty quotients a
// face; measured on B200, 90x75x66: 78 -> 54 us a direction.
template <int D>
__device__ __noinline__ void o3_face_exact(Dims dm, const Scalars* S, const double* Uin, FaceData fd, long long t) {
  o3_faces_item<D, false>(dm, S, Uin, fd, t, nullptr);
}
template <int D>
__device__ __forceinline__ void o3_face(const Dims& dm, const Scalars* __restrict__ S, const double* __restrict__ Uin,
                                        const FaceData& fd, long long t) {
  unsigned oor = 0u;
  o3_faces_item<D, true>(dm, S, Uin, fd, t, &oor);
  if (oor) o3_face_exact<D>(dm, S, Uin, fd, t);
}

template <int D>
__global__ void __launch_bounds__(128) k_o3_faces(Dims dm, const Scalars* __restrict__ S,
    const double* __restrict__ Uin, FaceData fd) {
  o3_face<D>(dm, S, Uin, fd, blockIdx.x * (long long)blockDim.x + threadIdx.x);
}

template <typename R>
static void remap_impl(const CycleArgs& a0, int sens, cudaStream_t s, KernelMarks* m, SweepFork* fork) {
  int prev = 0;
  CycleArgs a = a0;
  for (int it = 0; it < 3; ++it) {
    if (fork) fork->begin_cells(a, it, s);
    const int d = (it + sens) % 3;
    const bool first = it == 0, last = it == 2;
    a.ph.pb_first = first;
    const double* uin = a.U[it & 1];
    double* uout = a.U[(it + 1) & 1];
    const double* udin = a.ud[(it + 1) & 1];
    double* udout = a.ud[it & 1];
    if (sizeof(R) == 8 && a.ph.ordre_projection == 3) {
      const long long Fd = d == 0 ? a.dm.Fx : (d == 1 ? a.dm.Fy : a.dm.F - a.dm.Fx - a.dm.Fy);
      const unsigned nb = (unsigned)((Fd + 127) / 128);
      if (d == 0) k_o3_faces<0><<<nb, 128, 0, s>>>(a.dm, a.S, uin, a.fd);
      else if (d == 1) k_o3_faces<1><<<nb, 128, 0, s>>>(a.dm, a.S, uin, a.fd);
      else k_o3_faces<2><<<nb, 128, 0, s>>>(a.dm, a.S, uin, a.fd);
    }
    if (d == 0) sweep_cells_d<0, R>(a, last, uin, uout, s);
    else if (d == 1) sweep_cells_d<1, R>(a, last, uin, uout, s);
    else sweep_cells_d<2, R>(a, last, uin, uout, s);
    mark(m, BK_CELLS_X + d, s);
    sweep_nodes<1, R>(a, d, first, last, prev, udin, udout, fork ? fork->nodes_stream(it, s) : s);
    mark(m, BK_NODES_X + d, s);
    prev |= 1 << d;
  }
}

// conservation-energie-totale for one environment (RemapADIFinal.cc:751-773,
// then the EOS that follows the remap, PrepareRemap.cc:553-558): the
// 0.25 (ec_proj - ec_reconst) terms of the cell's 8 nodes (written by the
// last node sweep) summed in cell-node order from 0, floored at 0 as
// std::max(0., delta) does, times the cell's mass fraction, added to e; p and
// c again from the new e.
__device__ __forceinline__ void cons_ec_cell(const Dims& dm, const Phys& ph, const double* __restrict__ ecn,
    const double* __restrict__ mf, const double* __restrict__ rho, double* __restrict__ e, double* __restrict__ p,
    double* __restrict__ cs, int i, int j, int k) {
  const long long c = dm.cid(i, j, k);
  double delta_ec = 0.;
#pragma unroll
  for (int a = 0; a < 8; ++a)
    delta_ec += ecn[dm.nid(i + kCellNodeOff[a][0], j + kCellNodeOff[a][1], k + kCellNodeOff[a][2])];
  delta_ec = smax(0., delta_ec);
  const double en = e[c] + mf[c] * delta_ec;
  double pr, cc;
  eos_pc(ph.eos, ph.gamma, ph.pinf, rho[c], en, pr, cc);
  e[c] = en;
  p[c] = pr;
  cs[c] = cc;
}

__global__ void __launch_bounds__(128) k_cons_ec(Dims dm, Phys ph, const double* __restrict__ ecn,
    const double* __restrict__ mf, const double* __restrict__ rho, double* __restrict__ e, double* __restrict__ p,
    double* __restrict__ cs, int linear) {
  int i, j, k;
  if (!block_item(dm.nx, dm.ny, dm.nz, blockIdx.x, linear ? -1 : (int)blockIdx.y, blockIdx.z, i, j, k)) return;
  cons_ec_cell(dm, ph, ecn, mf, rho, e, p, cs, i, j, k);
}

void launch_cons_ec(const CycleArgs& a, cudaStream_t s) {
  int linear;
  const dim3 nbc = cell_grid(a.dm, linear);
  k_cons_ec<<<nbc, 128, 0, s>>>(a.dm, a.ph, a.ecn, a.st.mf, a.st.rho, a.st.e, a.st.p, a.st.cs, linear);
}

void launch_remap(const CycleArgs& a, int sens, cudaStream_t s, KernelMarks* m, SweepFork* fork) {
  if (a.ph.precision) { remap_impl<float>(a, sens, s, m, fork); return; }
  if (a.ph.csts) {
    // schema-csts: the remap starts from the forward velocity (U_dual,
    // Phi_dual, PrepareRemap.cc:411-433) on the Lagrangian coordinates
    CycleArgs b = a;
    b.vh = a.vf;
    remap_impl<double>(b, sens, s, m, fork);
    return;
  }
  remap_impl<double>(a, sens, s, m, fork);
}

void launch_delta_t(const CycleArgs& a, cudaStream_t s) {
  int linear;
  const dim3 nbc = cell_grid(a.dm, linear);
  k_dt_min<<<nbc, 128, 0, s>>>(a.dm, a.S, a.L, a.st.cs, a.vnorm, linear);
  if (!a.ph.ext_dt) k_dt_finish<<<1, 1, 0, s>>>(a.S, a.ph);
}

// ------------------------------------------------------------------------
// Batched cycle: the same kernel bodies, driven by per-kernel work tables over
// many instances (persistent grids).  Kernels with shared memory start each
// work item with a barrier, since the previous item's last reads of the tile
// may still be in flight in other warps.

void batch_work_shape(const Dims& dm, int K, int kind, int lines, bool march, int& gx, int& gy, int& gz) {
  const int nx = dm.nx, ny = dm.ny, nz = dm.nz;
  auto cdiv = [](int a, int b) { return (a + b - 1) / b; };
  const int W = lines;                            // lines per block of the y/z sweeps
  if (march) {                                    // y/z sweep: chunks of the plane x segments of the lines
    const bool nodes = kind >= BK_NODES_X;
    const int D = kind - (nodes ? BK_NODES_X : BK_CELLS_X), e = nodes ? 1 : 0;
    const int points = (nx + e) * ((D == 1 ? nz : ny) + e);
    gx = cdiv(points, kMarchThreads); gy = march_segments(dm.ncd(D) + e, points, march_len(lines)); gz = 1;
    return;
  }
  switch (kind) {
    case BK_LNODES: gx = (int)cdiv((int)dm.N, 128); gy = -1; gz = 1; break;      // linear chunks
    case BK_LCELLS:
      if (nx % 128) { gx = (int)cdiv((int)dm.C, 128); gy = -1; gz = 1; }        // linear chunks
      else { gx = nx / 128; gy = ny; gz = nz; }
      break;
    case BK_CELLS_X:
      if (K == 1) { gx = row_chunks(dm.C); gy = gz = 1; }                      // chunks of the rows' sequence
      else { gx = cdiv(nx, kLineUpd); gy = cdiv(ny, kLineWarps); gz = nz; }
      break;
    case BK_CELLS_Y: gx = cdiv(nx, W); gy = cdiv(ny, kLineUpd); gz = nz; break;
    case BK_CELLS_Z: gx = cdiv(nx, W); gy = cdiv(nz, kLineUpd); gz = ny; break;
    case BK_NODES_X: gx = row_chunks(dm.N); gy = gz = 1; break;
    case BK_NODES_Y: gx = cdiv(nx + 1, W); gy = cdiv(ny + 1, kLineUpd); gz = nz + 1; break;
    default: gx = cdiv(nx + 1, W); gy = cdiv(nz + 1, kLineUpd); gz = ny + 1; break;
  }
}

template <typename R>
__global__ void __launch_bounds__(128) k_bat_lagrange_nodes(const CycleArgs* __restrict__ D,
                                                            const int4* __restrict__ W, int nw) {
  for (int w = blockIdx.x; w < nw; w += gridDim.x) {
    const int4 t = W[w];
    const CycleArgs& a = D[t.x];
    if constexpr (sizeof(R) == 4)
      k_cyc_lagrange_nodes_body<float>(a.dm, a.S, a.st.p, a.st.q, a.cqs32, a.nm, a.v, a.bcmask, a.bct, a.vh, nullptr,
                                       t.y, t.z, t.w);
    else   // vnb: schema-csts (null otherwise)
      k_cyc_lagrange_nodes_body<double>(a.dm, a.S, a.st.p, a.st.q, a.cqs, a.nm, a.v, a.bcmask, a.bct, a.vh, a.vnb,
                                        t.y, t.z, t.w);
  }
}

// schema-csts of every instance: the forward velocity and the Lagrangian
// coordinates over the node tiles, then the face velocities over the face
// work table (instance, chunk of 128 faces of all directions)
__global__ void __launch_bounds__(128) k_bat_csts_forward(const CycleArgs* __restrict__ D, const int4* __restrict__ W,
                                                          int nw) {
  for (int w = blockIdx.x; w < nw; w += gridDim.x) {
    const int4 t = W[w];
    const CycleArgs& a = D[t.x];
    csts_forward_item(a.dm, a.S, a.pf, a.cqs, a.nm, a.x0, a.vh, a.vf, a.xl, t.y, t.z, t.w);
  }
}

__global__ void __launch_bounds__(128) k_bat_csts_face_u(const CycleArgs* __restrict__ D, const int4* __restrict__ W,
                                                         int nw) {
  for (int w = blockIdx.x; w < nw; w += gridDim.x) {
    const int4 t = W[w];
    const CycleArgs& a = D[t.x];
    csts_face_u_item(a.dm, a.vf, a.vnb, a.n0, a.fd, (long long)t.y * 128 + threadIdx.x);
  }
}

template <bool LAST, typename R, bool GL = false, bool PB = false, bool O3 = false>
__global__ void __launch_bounds__(32 * kLineWarps, kLineMinBlocks) k_bat_sweep_cells_x(
    const CycleArgs* __restrict__ D, const int4* __restrict__ W, int nw, int it) {
  for (int w = blockIdx.x; w < nw; w += gridDim.x) {
    const int4 t = W[w];
    const CycleArgs& a = D[t.x];
    if constexpr (PB) {   // the first sweep of a remap takes Phi from the Lagrange phase
      Phys ph = a.ph;
      ph.pb_first = it == 0;
      k_cyc_sweep_cells_x_body<LAST, R, O3, GL, PB>(a.dm, a.S, ph, a.fd, a.n0, a.xc, a.ofn, a.U[it & 1],
                                                a.U[(it + 1) & 1], a.dpf, a.st, t.y);
    } else {
      k_cyc_sweep_cells_x_body<LAST, R, O3, GL, PB>(a.dm, a.S, a.ph, a.fd, a.n0, a.xc, a.ofn, a.U[it & 1],
                                                a.U[(it + 1) & 1], a.dpf, a.st, t.y);
    }
  }
}

template <int DD, bool LAST, typename R, int LW, bool GL = false, bool PB = false, bool O3 = false>
__global__ void __launch_bounds__(32 * LW, TileGeom<LW>::minb) k_bat_sweep_cells_t(
    const CycleArgs* __restrict__ D, const int4* __restrict__ W, int nw, int it) {
  for (int w = blockIdx.x; w < nw; w += gridDim.x) {
    const int4 t = W[w];
    const CycleArgs& a = D[t.x];
    __syncthreads();
    if constexpr (PB) {
      Phys ph = a.ph;
      ph.pb_first = it == 0;
      k_cyc_sweep_cells_t_body<DD, LAST, R, LW, O3, GL, PB>(a.dm, a.S, ph, a.fd, a.n0, a.xc, a.ofn, a.U[it & 1],
                                                        a.U[(it + 1) & 1], a.dpf, a.st, t.y, t.z, t.w);
    } else {
      k_cyc_sweep_cells_t_body<DD, LAST, R, LW, O3, GL, PB>(a.dm, a.S, a.ph, a.fd, a.n0, a.xc, a.ofn, a.U[it & 1],
                                                        a.U[(it + 1) & 1], a.dpf, a.st, t.y, t.z, t.w);
    }
  }
}

// Order-3 face values of direction D over the face work table of D: items
// (instance, chunk of 128 consecutive faces), the sweep's input U[it & 1].
template <int D>
__global__ void __launch_bounds__(128) k_bat_o3_faces(const CycleArgs* __restrict__ A, const int4* __restrict__ W,
                                                      int nw, int it) {
  for (int w = blockIdx.x; w < nw; w += gridDim.x) {
    const int4 t = W[w];
    const CycleArgs& a = A[t.x];
    o3_face<D>(a.dm, a.S, a.U[it & 1], a.fd, (long long)t.y * 128 + threadIdx.x);
  }
}

template <bool FIRST, bool LAST, typename R, bool GL = false>
__global__ void __launch_bounds__(32 * kLineWarps, kLineMinBlocks) k_bat_sweep_nodes_x(
    const CycleArgs* __restrict__ D, const int4* __restrict__ W, int nw, int it, int prev) {
  for (int w = blockIdx.x; w < nw; w += gridDim.x) {
    const int4 t = W[w];
    const CycleArgs& a = D[t.x];
    // schema-csts: the forward velocity on the Lagrangian coordinates (xl is null otherwise)
    k_cyc_sweep_nodes_x_body<FIRST, LAST, 1, R, GL>(a.dm, a.S, a.ph, prev, a.x0, a.xl, a.ph.csts ? a.vf : a.vh, a.nm,
                                                 a.ud[(it + 1) & 1], a.ud[it & 1], a.dpf, a.Gd, a.st.mass, a.v, a.nm,
                                                 a.vnorm, t.y, a.ecn);
  }
}

template <int DD, bool FIRST, bool LAST, typename R, int LW, bool GL = false>
__global__ void __launch_bounds__(32 * LW, TileGeom<LW>::minb) k_bat_sweep_nodes_t(
    const CycleArgs* __restrict__ D, const int4* __restrict__ W, int nw, int it, int prev) {
  for (int w = blockIdx.x; w < nw; w += gridDim.x) {
    const int4 t = W[w];
    const CycleArgs& a = D[t.x];
    __syncthreads();
    k_cyc_sweep_nodes_t_body<DD, FIRST, LAST, 1, R, LW, GL>(a.dm, a.S, a.ph, prev, a.x0, a.xl,
                                                         a.ph.csts ? a.vf : a.vh, a.nm, a.ud[(it + 1) & 1],
                                                         a.ud[it & 1], a.dpf, a.Gd, a.st.mass, a.v, a.nm, a.vnorm,
                                                         t.y, t.z, t.w, a.ecn);
  }
}

__global__ void __launch_bounds__(128) k_bat_dt_min(const CycleArgs* __restrict__ D, const int4* __restrict__ W,
                                                    int nw) {
  for (int w = blockIdx.x; w < nw; w += gridDim.x) {
    const int4 t = W[w];
    const CycleArgs& a = D[t.x];
    __syncthreads();
    dt_min_body(a.dm, a.S, a.L, a.st.cs, a.vnorm, t.y, t.z, t.w);
  }
}

// conservation-energie-totale over the Lagrange cell kernel's tiles, for the
// instances that have it
__global__ void __launch_bounds__(128) k_bat_cons_ec(const CycleArgs* __restrict__ D, const int4* __restrict__ W,
                                                     int nw) {
  for (int w = blockIdx.x; w < nw; w += gridDim.x) {
    const int4 t = W[w];
    const CycleArgs& a = D[t.x];
    if (!a.ph.cons_ec) continue;
    int i, j, k;
    if (block_item(a.dm.nx, a.dm.ny, a.dm.nz, t.y, t.z, t.w, i, j, k))
      cons_ec_cell(a.dm, a.ph, a.ecn, a.st.mf, a.st.rho, a.st.e, a.st.p, a.st.cs, i, j, k);
  }
}

// one thread per instance: each instance's own dt (per-instance options)
__global__ void k_bat_dt_finish(const CycleArgs* __restrict__ D, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dt_finish_body(D[i].S, D[i].ph);
}

// Resident blocks of a persistent grid for `kernel`: SMs x blocks per SM
// (queried once per kernel and device), scaled by pct percent.
template <class Kern>
static int persistent_blocks(Kern kernel, int threads, size_t smem, int nwork, int pct) {
  static std::mutex mu;
  static std::map<std::pair<const void*, int>, int> cache;
  int dev = 0;
  cudaGetDevice(&dev);
  int g = 0;
  {
    std::lock_guard<std::mutex> lk(mu);
    const auto key = std::make_pair(reinterpret_cast<const void*>(kernel), dev);
    auto itc = cache.find(key);
    if (itc == cache.end()) {
      int sms = 0, per = 0;
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, smem);
      itc = cache.emplace(key, (per > 0 ? per : 1) * (sms > 0 ? sms : 1)).first;
    }
    g = itc->second;
  }
  if (pct > 0 && pct < 100) g = (int)(((long long)g * pct + 99) / 100);
  if (g < 1) g = 1;
  return nwork < g ? (nwork > 0 ? nwork : 1) : g;
}

int persistent_grid(const void* kernel, int threads, size_t smem, int nwork, int pct) {
  return persistent_blocks(kernel, threads, smem, nwork, pct);
}

void batch_column_shape(const Dims& dm, int& blocks, int& segments, int& strip) {
  blocks = col_blocks(dm.nx, dm.ny);
  segments = col_segments(dm.nx, dm.ny, dm.nz);
  strip = col_strip(dm.nx);
}

// The y/z sweeps of a batch with a table of marching work (FP64 node sweeps
// march on the first sweep of a remap only).
bool batch_marches(const CycleArgs& a, int kind, long long nodes) {
  if (kind == BK_NODES_Y || kind == BK_NODES_Z) return march_nodes(nodes, a.ph.precision, true);
  if (kind == BK_CELLS_Y || kind == BK_CELLS_Z) return a.K == 1 && march_cells(nodes, a.ph.precision);
  return false;
}

void mark(KernelMarks* m, int kind, cudaStream_t s) {
  if (!m || m->n >= KernelMarks::kMax) return;
  cudaEventRecord(m->ev[m->n], s);
  m->kind[m->n++] = kind;
}

// One persistent launch over the work table of `kind`; tk is the tuning slot
// (grid percentage and timing mark): the kind itself, or BK_DT_MIN.
template <class Kern, class... Args>
static void launch_persistent(Kern kernel, int threads, size_t smem, const BatchPlan& P, int kind, int tk,
                              cudaStream_t s, KernelMarks* marks, Args... args) {
  const int nwork = P.nwork[kind];
  smem_opt_in((const void*)kernel, smem);
  if (nwork > 0) kernel<<<persistent_blocks(kernel, threads, smem, nwork, P.occ_pct[tk]), threads, smem, s>>>(args...);
  mark(marks, tk, s);
}

template <int DD, bool LAST, typename R, int LW, bool GL, bool PB = false, bool O3 = false>
static void bat_cells_t(const BatchPlan& P, int it, cudaStream_t s, KernelMarks* m) {
  const int kind = BK_CELLS_X + DD;
  launch_persistent(k_bat_sweep_cells_t<DD, LAST, R, LW, GL, PB, O3>, 32 * LW, CellTileSize<LAST, LW, O3>::bytes, P,
                    kind, kind, s, m, P.descs, P.work[kind], P.nwork[kind], it);
}

// Order 3: the face values of direction DD from the sweep's input (no mark of
// their own: their time counts towards the cell sweep's slot).
template <int DD>
static void launch_bat_o3_faces(const BatchPlan& P, int it, cudaStream_t s) {
  auto kern = k_bat_o3_faces<DD>;
  if (P.o3nwork[DD] > 0)
    kern<<<persistent_blocks(kern, 128, 0, P.o3nwork[DD], 100), 128, 0, s>>>(P.descs, P.o3work[DD], P.o3nwork[DD], it);
}

template <int DD, bool LAST, typename R, bool GL>
static void bat_cells_d(const BatchPlan& P, int it, cudaStream_t s, KernelMarks* m) {
  const int kind = BK_CELLS_X + DD;
  if constexpr (sizeof(R) == 8) {
    if (P.o3) {   // order 3: the face values first, then the O3 cell sweeps, 8 lines
      launch_bat_o3_faces<DD>(P, it, s);
      if constexpr (DD == 0)
        launch_persistent(k_bat_sweep_cells_x<LAST, R, GL, false, true>, 32 * kLineWarps, 0, P, kind, kind, s, m,
                          P.descs, P.work[kind], P.nwork[kind], it);
      else
        bat_cells_t<DD, LAST, R, 8, GL, false, true>(P, it, s, m);
      return;
    }
    if (P.pb) {   // pente-borne: its own cell sweeps (the widths too), 8 lines
      if constexpr (DD == 0)
        launch_persistent(k_bat_sweep_cells_x<LAST, R, false, true>, 32 * kLineWarps, 0, P, kind, kind, s, m, P.descs,
                          P.work[kind], P.nwork[kind], it);
      else
        bat_cells_t<DD, LAST, R, 8, false, true>(P, it, s, m);
      return;
    }
  }
  if constexpr (DD == 0) {
    launch_persistent(k_bat_sweep_cells_x<LAST, R, GL>, 32 * kLineWarps, 0, P, kind, kind, s, m, P.descs, P.work[kind],
                      P.nwork[kind], it);
  } else {
    if constexpr (sizeof(R) == 4) {
      if (P.march[kind]) {
        launch_march(k_bat_sweep_cells_m<DD, LAST>, P, kind, s, m, P.descs, P.mwork[kind], P.nmwork[kind], it,
                     march_len(P.lines[kind]));
        return;
      }
    }
    const int w = P.lines[kind];
    if (GL || w == 8) bat_cells_t<DD, LAST, R, 8, GL>(P, it, s, m);   // the G limiters keep 8 lines
    else if (w == 32) bat_cells_t<DD, LAST, R, 32, false>(P, it, s, m);
    else bat_cells_t<DD, LAST, R, 16, false>(P, it, s, m);
  }
}

template <int DD, bool FIRST, bool LAST, typename R, int LW, bool GL>
static void bat_nodes_t(const BatchPlan& P, int it, int prev, cudaStream_t s, KernelMarks* m) {
  const int kind = BK_NODES_X + DD;
  launch_persistent(k_bat_sweep_nodes_t<DD, FIRST, LAST, R, LW, GL>, 32 * LW, NodeTileSize<DD, FIRST, LAST, 1, LW>::bytes,
                    P, kind, kind, s, m, P.descs, P.work[kind], P.nwork[kind], it, prev);
}

template <int DD, bool FIRST, bool LAST, typename R, bool GL>
static void bat_nodes_d(const BatchPlan& P, int it, int prev, cudaStream_t s, KernelMarks* m) {
  const int kind = BK_NODES_X + DD;
  if constexpr (DD == 0) {
    launch_persistent(k_bat_sweep_nodes_x<FIRST, LAST, R, GL>, 32 * kLineWarps, 0, P, kind, kind, s, m, P.descs,
                      P.work[kind], P.nwork[kind], it, prev);
  } else {
    if constexpr (sizeof(R) == 4 || FIRST) {
      if (P.march[kind]) {
        launch_march(k_bat_sweep_nodes_m<DD, FIRST, LAST, 1, R, GL>, P, kind, s, m, P.descs, P.mwork[kind],
                     P.nmwork[kind], prev, march_len(P.lines[kind]));
        return;
      }
    }
    const int w = P.lines[kind];
    if (GL || w == 8) bat_nodes_t<DD, FIRST, LAST, R, 8, GL>(P, it, prev, s, m);
    else if (w == 32) bat_nodes_t<DD, FIRST, LAST, R, 32, false>(P, it, prev, s, m);
    else bat_nodes_t<DD, FIRST, LAST, R, 16, false>(P, it, prev, s, m);
  }
}

template <int DD, typename R, bool GL>
static void bat_sweep(const BatchPlan& P, int it, int prev, cudaStream_t s, KernelMarks* m) {
  const bool first = it == 0, last = it == 2;
  if (last) bat_cells_d<DD, true, R, GL>(P, it, s, m);
  else bat_cells_d<DD, false, R, GL>(P, it, s, m);
  if (first) bat_nodes_d<DD, true, false, R, GL>(P, it, prev, s, m);
  else if (last) bat_nodes_d<DD, false, true, R, GL>(P, it, prev, s, m);
  else bat_nodes_d<DD, false, false, R, GL>(P, it, prev, s, m);
}

template <typename R, bool GL>
static void bat_sweeps(const BatchPlan& P, int sens, cudaStream_t s, KernelMarks* m) {
  int prev = 0;
  for (int it = 0; it < 3; ++it) {
    const int d = (it + sens) % 3;
    if (d == 0) bat_sweep<0, R, GL>(P, it, prev, s, m);
    else if (d == 1) bat_sweep<1, R, GL>(P, it, prev, s, m);
    else bat_sweep<2, R, GL>(P, it, prev, s, m);
    prev |= 1 << d;
  }
}

void launch_bat_cons_ec(const BatchPlan& P, cudaStream_t s) {
  if (P.cons_ec)
    launch_persistent(k_bat_cons_ec, 128, 0, P, BK_LCELLS, BK_LCELLS, s, nullptr, P.descs, P.work[BK_LCELLS],
                      P.nwork[BK_LCELLS]);
}

void launch_bat_lagrange_nodes(const BatchPlan& P, cudaStream_t s, KernelMarks* m) {
  if (P.precision)
    launch_persistent(k_bat_lagrange_nodes<float>, 128, 0, P, BK_LNODES, BK_LNODES, s, m, P.descs, P.work[BK_LNODES], P.nwork[BK_LNODES]);
  else
    launch_persistent(k_bat_lagrange_nodes<double>, 128, 0, P, BK_LNODES, BK_LNODES, s, m, P.descs, P.work[BK_LNODES], P.nwork[BK_LNODES]);
}

void launch_bat_dt(const BatchPlan& P, cudaStream_t s, KernelMarks* m) {
  // the dt reduction walks the cell tiles of the Lagrange cell kernel
  launch_persistent(k_bat_dt_min, 128, 0, P, BK_LCELLS, BK_DT_MIN, s, m, P.descs, P.work[BK_LCELLS], P.nwork[BK_LCELLS]);
  k_bat_dt_finish<<<(P.ninst + 127) / 128, 128, 0, s>>>(P.descs, P.ninst);
  mark(m, BK_DT_FINISH, s);
}

void launch_bat_csts_forward(const BatchPlan& P, cudaStream_t s) {
  if (!P.csts) return;
  launch_persistent(k_bat_csts_forward, 128, 0, P, BK_LNODES, BK_LNODES, s, nullptr, P.descs, P.work[BK_LNODES],
                    P.nwork[BK_LNODES]);
  if (P.nfwork > 0)
    k_bat_csts_face_u<<<persistent_blocks(k_bat_csts_face_u, 128, 0, P.nfwork, 100), 128, 0, s>>>(P.descs, P.fwork,
                                                                                                 P.nfwork);
}

void launch_batch_cycle(const BatchPlan& P, int sens, cudaStream_t s, KernelMarks* m) {
  if (P.K > 1) { launch_batch_cycle_env(P, sens, s, m); return; }
  launch_bat_lagrange_nodes(P, s, m);
  const bool hc = P.gl || P.pb || P.o3;   // the G limiters, pente-borne, order 3: the cell widths too
  if (P.precision) launch_bat_cells<1, float, false>(P, s, m);
  else if (P.csts && hc) launch_bat_tiles<1, double, true, true, false>(P, s, m);
  else if (P.csts) launch_bat_tiles<1, double, false, true, false>(P, s, m);
  else if (hc) launch_bat_cells<1, double, true>(P, s, m);
  else launch_bat_cells<1, double, false>(P, s, m);
  launch_bat_csts_forward(P, s);   // PrepareRemap.cc:456, then the face velocities
  if (P.precision) bat_sweeps<float, false>(P, sens, s, m);
  else if (P.gl) bat_sweeps<double, true>(P, sens, s, m);
  else bat_sweeps<double, false>(P, sens, s, m);
  launch_bat_cons_ec(P, s);
  launch_bat_dt(P, s, m);
}

}  // namespace mhy
