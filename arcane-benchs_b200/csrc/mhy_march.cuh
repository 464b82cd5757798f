// mhy_march.cuh -- the y and z sweeps of the remap: one thread marches along a
// segment of one line, with the neighbouring lines' threads side by side in x.
//
// Every array is read and written in rows along x as it lies in memory, the
// stencil along the line is a window in registers (no shuffles, no shared
// memory, no barriers), and the next position is loaded while this one is
// worked on.  A segment re-reads two positions at each end.
#pragma once

#include "mhy_line.cuh"

namespace mhy {

// Threads of a block: consecutive points of the plane across the sweep
// direction (x fastest).
constexpr int kMarchThreads = 128;

// The part [a, b) of a line of n items that segment `seg` of nseg updates.
__host__ __device__ __forceinline__ void march_range(int n, int seg, int nseg, int& a, int& b) {
  a = (int)((long long)n * seg / nseg);
  b = (int)((long long)n * (seg + 1) / nseg);
}

// Segments of a line of n items over a plane of `points` lines: `len` items
// a segment, shorter where that many threads would not fill the chip
// (kMarchFill threads), down to (n + 3) / 4 segments: 4 or 3 items each (2 and 3
// on a line of 5).
constexpr int kMarchFill = 148 * 4 * kMarchThreads;
__host__ __device__ __forceinline__ int march_segments(int n, int points, int len) {
  const int by_len = (n + len - 1) / len, fill = (kMarchFill + points - 1) / points, most = (n + 3) / 4;
  const int want = fill < most ? fill : most;
  return by_len > want ? by_len : want;
}
// Items a segment, from the tuning's lines setting (8, 16 or 32).
__host__ __device__ __forceinline__ int march_len(int lines) { return 2 * lines; }

// Which y/z sweeps march; the others stage tiles.  A marching thread holds its
// window in 128 registers, so 16 warps an SM where the staged sweeps have 32:
// it gains where instructions or bandwidth bound a sweep, and loses where
// latency does, in FP64 with its long quotients and on meshes that are a wave
// or two of blocks.  Measured on B200, staged -> marching: Sedov 128^3 in the
// mixed form, cell sweeps 85-92 -> 67-70 us, node sweeps 89-115 -> 66-100 us, a
// cycle 864 -> 780 us; but 240 -> 259 us at 80^3 and 398 -> 410 us at 96^3.
// FP64 node sweeps of a remap's first direction (no U_dual to divide) 112 ->
// 78 us, the later ones 123 -> 105 us there but 86 -> 101 us on a dense flow
// with vanLeer (211x97x61).  `nodes`: of the mesh, or of all of a batch.
constexpr long long kMarchMinNodes = 1500000;
inline bool march_nodes(long long nodes, int precision, bool first) {
  return nodes >= kMarchMinNodes && (precision || first);
}
inline bool march_cells(long long nodes, int precision) { return nodes >= kMarchMinNodes && precision; }

// ---- nodes ------------------------------------------------------------------
// One step of a node sweep reads the node at position q, forms the front
// difference quotients and the limited gradient of q - 1, and updates q - 2
// (the expressions of node_line).
template <int D, bool FIRST, bool LAST, int K, typename R, bool GL, bool SP, bool BAT>
__device__ __forceinline__ void nodes_march(const CycleArgs& A, int prev_inner, int point, int seg, int nseg,
                                            unsigned* oor) {
  constexpr int it = FIRST ? 0 : (LAST ? 2 : 1);                 // the sweep of the remap
  const Dims& dm = A.dm;
  const Phys& ph = A.ph;
  const int nx = dm.nx, ny = dm.ny, nz = dm.nz;
  const int N = (int)dm.N, C = (int)dm.C;
  const int nn = dm.ncd(D) + 1;
  const int i = point % (nx + 1), o = point / (nx + 1);          // o: z for D = 1, y for D = 2
  int a, b;
  march_range(nn, seg, nseg, a, b);
  const int nb = D == 1 ? i + (nx + 1) * (ny + 1) * o : point;   // node at position 0
  const int ns = D == 1 ? nx + 1 : (nx + 1) * (ny + 1);          // and its stride along D
  // the four cell lines around the node line: (x - 1 | x) x (o - 1 | o)
  const int no = D == 1 ? nz : ny;
  const int cs = D == 1 ? nx : nx * ny;
  const bool cx0 = i > 0, cx1 = i < nx, co0 = o > 0, co1 = o < no;
  const int cO = D == 1 ? nx * ny : nx;                          // stride of o
  const int cb = i + cO * o;                             // cell (i, o) at position 0
  const bool grad_on = ph.ordre_projection > 1;
  const int lim = grad_on ? ph.limiteur_id : -1;
  const R order2 = (R)(ph.ordre_projection - 1);
  const double dt = A.S->dt;
  // the node is inner along an earlier direction of this cycle, or lies on a
  // boundary plane of another one: the same all along the line
  constexpr int kDo = D == 1 ? 2 : 1;                            // the direction of o
  const bool updated = ((prev_inner & 1) && i > 0 && i < nx) || ((prev_inner >> kDo & 1) && o > 0 && o < no);
  const bool on_plane = i == 0 || i == nx || o == 0 || o == no;
  // the arrays are named where they are used: in a batch they come from shared
  // memory (k_bat_sweep_nodes_m), and two dozen pointers in registers would spill.
  // schema-csts: the forward velocity on the Lagrangian coordinates
  auto vh = [&](int n) { return (A.ph.csts ? A.vf : A.vh)[n]; };
  auto xs = [&](int n) { return (A.xl ? A.xl : A.x0)[D * N + n]; };
  const bool xabs = A.xl != nullptr;
  auto coord = [&](double x, double v) { return xabs ? x : x + v * dt; };

  // what a node brings: the coordinate and velocity along D, and either the
  // Lagrange velocity (FIRST) or U_dual
  constexpr int NW = FIRST ? 3 : 5;
  double rx[2], rv[2], rw[2][NW];
  auto load = [&](int slot, int q) {
    const int n = nb + ns * q;
    rx[slot] = xs(n);
    if constexpr (FIRST) {
#pragma unroll
      for (int c = 0; c < 3; ++c) rw[slot][c] = vh(c * N + n);
      rv[slot] = rw[slot][D];
    } else {
      rv[slot] = vh(D * N + n);
#pragma unroll
      for (int c = 0; c < 5; ++c) rw[slot][c] = A.ud[(it + 1) & 1][c * N + n];
    }
  };

  // the window, indexed by slots
  R P[4][4], G[4][3], g[4][3];
  double xw[4], un[4], ff[4], mp[4][4];
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    xw[s] = un[s] = ff[s] = 0.;
#pragma unroll
    for (int c = 0; c < 4; ++c) { P[s][c] = 0; mp[s][c] = 0.; }
#pragma unroll
    for (int c = 0; c < 3; ++c) { G[s][c] = 0; g[s][c] = 0; }
  }
  const int q0 = a - 2 > 0 ? a - 2 : 0;
  load(0, q0);
  rx[1] = rv[1] = 0.;
#pragma unroll
  for (int c = 0; c < NW; ++c) rw[1][c] = 0.;
  constexpr int s0 = 0, s1 = 1, s2 = 2, s3 = 3, cur = 0;         // slots: q - 3, q - 2, q - 1, q
#pragma unroll 1
  for (int q = q0; q <= b + 1; ++q) {
    if constexpr (BAT) asm volatile("" ::: "memory");            // no pointer is kept over a step
    if (q + 1 < nn && q <= b) load(cur ^ 1, q + 1);
    const int m = q - 2;
    // loads of the position that this step updates
    double ud[5] = {0., 0., 0., 0., 0.}, dp[4 * K], mn = 0.;
    const bool own = m >= a, half = m >= a - 1 && m >= 0 && m < nn - 1;
    const int n = nb + ns * m;
#pragma unroll
    for (int e = 0; e < 4 * K; ++e) dp[e] = 0.;
    if constexpr (LAST) {
#pragma unroll
      for (int c = 0; c < 4; ++c) mp[s1][c] = 0.;
    }
    if (half) {
      const int c = cb + cs * m;
      // DualPhaseRemap.cc:299-340: s1 over (D + 1) % 3, s2 over (D + 2) % 3;
      // D = 1: s1 over z, s2 over x; D = 2: s1 over x, s2 over y
#pragma unroll
      for (int e = 0; e < K; ++e) {
        if (cx0 && co0) dp[e] = A.dpf[e * C + c - 1 - cO];
        if (D == 1 ? (cx1 && co0) : (cx0 && co1)) dp[K + e] = A.dpf[e * C + c - (D == 1 ? cO : 1)];
        if (D == 1 ? (cx0 && co1) : (cx1 && co0)) dp[2 * K + e] = A.dpf[e * C + c - (D == 1 ? 1 : cO)];
        if (cx1 && co1) dp[3 * K + e] = A.dpf[e * C + c];
      }
      if constexpr (LAST) {
        if (cx0 && co0) mp[s1][0] = A.st.mass[c - 1 - cO];
        if (cx1 && co0) mp[s1][1] = A.st.mass[c - cO];
        if (cx0 && co1) mp[s1][2] = A.st.mass[c - 1];
        if (cx1 && co1) mp[s1][3] = A.st.mass[c];
      }
    }
    if (own) {
      if constexpr (FIRST) mn = A.nm[n];
      else {
#pragma unroll
        for (int c = 0; c < 5; ++c) ud[c] = A.ud[(it + 1) & 1][c * N + n];
      }
    }
    // the new node
    if (q < nn) {
      if (FIRST || !updated) {
        D3 u;
        if constexpr (FIRST) u = d3(rw[cur][0], rw[cur][1], rw[cur][2]);
        else {
          const int nq = nb + ns * q;
          u = d3(vh(nq), vh(N + nq), vh(2 * N + nq));
        }
        un[s3] = norm2(u);
        P[s3][0] = (R)u.x; P[s3][1] = (R)u.y; P[s3][2] = (R)u.z; P[s3][3] = (R)(0.5 * un[s3]);
      } else if constexpr (!FIRST) {
        const R ms = (R)rw[cur][3], rm = rc<R, SP>(ms, oor);
        P[s3][0] = dv<R, SP>((R)rw[cur][0], ms, rm, oor); P[s3][1] = dv<R, SP>((R)rw[cur][1], ms, rm, oor);
        P[s3][2] = dv<R, SP>((R)rw[cur][2], ms, rm, oor); P[s3][3] = dv<R, SP>((R)rw[cur][4], ms, rm, oor);
      }
      xw[s3] = coord(rx[cur], rv[cur]);
      // front difference quotients of q - 1
      if (grad_on && q > q0) {
        const R hf = (R)(xw[s3] - xw[s2]), rf = rc<R, SP>(hf, oor);
#pragma unroll
        for (int c = 0; c < 3; ++c) g[s2][c] = dv<R, SP>(P[s3][c] - P[s2][c], hf, rf, oor);
      }
    }
    // limited gradient of q - 1
    if (q >= a && q >= 1 && q - 1 < nn) {
      if (grad_on && q >= 2 && q < nn) {
        if constexpr (GL) {
          // generalised limiters (DualPhaseRemap.cc:48-64, UtilesRemap.cc:15-80, 346-377): the dual widths
          const bool bb = q >= 3, fr = q + 1 < nn;
          const int nq = nb + ns * (q - 1);
          const double xp2 = fr ? coord(xs(nq + 2 * ns), vh(D * N + nq + 2 * ns)) : 0.;
          const double xb2 = bb ? (q - 3 >= q0 ? xw[s0] : coord(xs(nq - 2 * ns), vh(D * N + nq - 2 * ns))) : 0.;
          const R h0 = (R)(0.5 * (xw[s3] - xw[s1]));
          R hmo, hpl;
          if (!bb) { hmo = R(0); hpl = (R)(0.5 * (xp2 - xw[s2])); }
          else if (!fr) { hpl = R(0); hmo = (R)(0.5 * (xw[s2] - xb2)); }
          else { hmo = (R)(0.5 * (xw[s2] - xb2)); hpl = (R)(0.5 * (xp2 - xw[s2])); }
#pragma unroll
          for (int c = 0; c < 3; ++c)
            G[s2][c] = flux_limiter_g<R, SP>(lim, g[s2][c], g[s1][c], P[s2][c], P[s3][c], P[s1][c], h0, hpl, hmo, oor);
        } else {
          limited_slopes<3, R, true, SP, true>(lim, g[s1], g[s2], G[s2], oor);
        }
      } else {
        // not inner along D: the gradient an earlier sweep left, or zero with the generalised limiters
        const int nq = nb + ns * (q - 1);
#pragma unroll
        for (int c = 0; c < 3; ++c) G[s2][c] = (GL && grad_on) ? R(0) : (R)A.Gd[c * N + nq];
      }
    }
    // sum of 0.25 * dual mass flux of the 4 cells in front of m
    ff[s1] = 0.;
    if (half) {
      double f = 0.;
#pragma unroll
      for (int e = 0; e < 4 * K; ++e) f += 0.25 * dp[e];
      ff[s1] = f;
    }
    if (own) {
      const bool inner = m >= 1 && m <= nn - 2;
      if constexpr (FIRST) {
        D3 u1;
        if constexpr (sizeof(R) == 8) u1 = d3(P[s1][0], P[s1][1], P[s1][2]);
        else u1 = d3(vh(n), vh(N + n), vh(2 * N + n));
        ud[0] = mn * u1.x; ud[1] = mn * u1.y; ud[2] = mn * u1.z; ud[3] = mn; ud[4] = 0.5 * mn * un[s1];
      }
      if (inner) {
        dual_update<R>(D, order2, (R)dt, ff[s0], ff[s1], P[s0], P[s1], P[s2], G[s0], G[s1], G[s2],
                       (R)(xw[s1] - xw[s0]), (R)(xw[s2] - xw[s1]), ud);
        if (grad_on && on_plane) {
#pragma unroll
          for (int c = 0; c < 3; ++c) A.Gd[c * N + n] = (double)G[s1][c];
        }
      }
      if constexpr (!LAST) {
#pragma unroll
        for (int c = 0; c < 5; ++c) A.ud[it & 1][c * N + n] = ud[c];
      } else {
        const double ms = ud[3];
        D3 u;
        double rm = 0.;
        if (ms != 0.) {
          rm = rc<double, SP>(ms, oor);
          u = d3(dv<double, SP>(ud[0], ms, rm, oor), dv<double, SP>(ud[1], ms, rm, oor), dv<double, SP>(ud[2], ms, rm, oor));
        } else {
          u = d3(vh(n), vh(N + n), vh(2 * N + n));
        }
        // node mass: increasing cell id, z outer, y, x inner
        const double* b0 = mp[s0];
        const double* a0 = mp[s1];
        double sm = 0.;
        if (D == 1) {
          sm += b0[0]; sm += b0[1]; sm += a0[0]; sm += a0[1]; sm += b0[2]; sm += b0[3]; sm += a0[2]; sm += a0[3];
        } else {
          sm += b0[0]; sm += b0[1]; sm += b0[2]; sm += b0[3]; sm += a0[0]; sm += a0[1]; sm += a0[2]; sm += a0[3];
        }
        A.v[n] = u.x; A.v[N + n] = u.y; A.v[2 * N + n] = u.z;
        A.nm[n] = .125 * sm;
        A.vnorm[n] = norm2(u);
        // conservation-energie-totale (RemapADIFinal.cc:757-764), see node_line
        if (A.ecn)
          A.ecn[n] = ms != 0. ? 0.25 * (dv<double, SP>(ud[4], ms, rm, oor) - 0.5 * (u.x * u.x + u.y * u.y + u.z * u.z)) : 0.;
      }
    }
    // shift the window
#pragma unroll
    for (int s = 0; s < 3; ++s) {
      xw[s] = xw[s + 1]; un[s] = un[s + 1]; ff[s] = ff[s + 1];
#pragma unroll
      for (int c = 0; c < 4; ++c) { P[s][c] = P[s + 1][c]; mp[s][c] = mp[s + 1][c]; }
#pragma unroll
      for (int c = 0; c < 3; ++c) { G[s][c] = G[s + 1][c]; g[s][c] = g[s + 1][c]; }
    }
    rx[0] = rx[1]; rv[0] = rv[1];
#pragma unroll
    for (int c = 0; c < NW; ++c) rw[0][c] = rw[1][c];
  }
}

template <int D, bool FIRST, bool LAST, int K, typename R, bool GL>
__device__ __noinline__ void nodes_march_exact(const CycleArgs* A, int prev_inner, int point, int seg, int nseg) {
  nodes_march<D, FIRST, LAST, K, R, GL, false, false>(*A, prev_inner, point, seg, nseg, nullptr);
}

// Work item (bx, seg): kMarchThreads points of the plane, one segment.  A
// thread whose FP64 quotients left the guarded range does its segment again
// with exact ones: nothing that it wrote is read in the same sweep.
template <int D, bool FIRST, bool LAST, int K, typename R, bool GL, bool BAT>
__device__ __forceinline__ void sweep_nodes_march(const CycleArgs& A, int prev_inner, int len, int bx_, int seg) {
  const int points = (A.dm.nx + 1) * ((D == 1 ? A.dm.nz : A.dm.ny) + 1);
  const int point = bx_ * kMarchThreads + threadIdx.x;
  if (point >= points) return;
  const int nseg = march_segments(A.dm.ncd(D) + 1, points, len);
  unsigned oor = 0u;
  nodes_march<D, FIRST, LAST, K, R, GL, sizeof(R) == 8, BAT>(A, prev_inner, point, seg, nseg, &oor);
  if constexpr (sizeof(R) == 8) {
    if (oor) nodes_march_exact<D, FIRST, LAST, K, R, GL>(&A, prev_inner, point, seg, nseg);
  }
}

// 4 blocks of 128 threads: 128 registers hold the window with few spills.
template <int D, bool FIRST, bool LAST, int K, typename R, bool GL = false>
__global__ void __launch_bounds__(kMarchThreads, 4) k_cyc_sweep_nodes_m(const __grid_constant__ CycleArgs a, int prev_inner,
                                                                        int len) {
  sweep_nodes_march<D, FIRST, LAST, K, R, GL, false>(a, prev_inner, len, blockIdx.x, blockIdx.y);
}

// One instance's arguments into shared memory, by all threads of the block.
__device__ __forceinline__ void copy_args(CycleArgs& to, const CycleArgs* from) {
  static_assert(sizeof(CycleArgs) % sizeof(double) == 0, "copied as doubles");
  __syncthreads();                         // the previous item's reads are done
  for (int x = threadIdx.x; x < (int)(sizeof(CycleArgs) / sizeof(double)); x += blockDim.x)
    reinterpret_cast<double*>(&to)[x] = reinterpret_cast<const double*>(from)[x];
  __syncthreads();
}

// The same over a batch's work table (instance, plane chunk, segment).
template <int D, bool FIRST, bool LAST, int K, typename R, bool GL = false>
__global__ void __launch_bounds__(kMarchThreads, 4) k_bat_sweep_nodes_m(const CycleArgs* __restrict__ A,
    const int4* __restrict__ W, int nw, int prev, int len) {
  __shared__ CycleArgs a;
  for (int w = blockIdx.x; w < nw; w += gridDim.x) {
    const int4 t = W[w];
    copy_args(a, A + t.x);
    sweep_nodes_march<D, FIRST, LAST, K, R, GL, true>(a, prev, len, t.y, t.z);
  }
}

// ---- cells of one environment, mixed form ------------------------------------
// One step reads the cell at position q and its low face, forms that face's
// gradient, the limited gradient of q - 1, the upwind face value of the low
// face of q - 1, and updates the cell q - 2 (the expressions of cell_line).
template <int D, bool LAST, bool BAT>
__device__ __forceinline__ void cells_march(const CycleArgs& A, int it, int point, int seg, int nseg) {
  using R = float;
  const Dims& dm = A.dm;
  const Phys& ph = A.ph;
  const int nx = dm.nx;
  const int C = (int)dm.C, F = (int)dm.F;
  const int nd = dm.ncd(D);
  const int i = point % nx, o = point / nx;                       // o: z for D = 1, y for D = 2
  int a, b;
  march_range(nd, seg, nseg, a, b);
  const int cb0 = D == 1 ? i + nx * dm.ny * o : point;          // cell at position 0
  const int cs = D == 1 ? nx : nx * dm.ny;                      // and its stride along D
  const int fb0 = D == 1 ? i + nx * (dm.ny + 1) * o : point;    // low face within direction D
  const int foff = D == 1 ? (int)dm.Fx : (int)(dm.Fx + dm.Fy);
  constexpr int lb = D == 1 ? 2 : 0, lf = D == 1 ? 5 : 3;         // back / front faces of D in cell-face order
  const int lim = ph.ordre_projection > 1 ? ph.lim_cell : -1;
  const R order2 = (R)(ph.ordre_projection - 1);
  const double dt = A.S->dt;

  double rU[2][4], rx[2][3], rn[2][3], rdb[2], rdf[2], ru[2], rA[2];
  auto load = [&](int slot, int q) {
    const int c = cb0 + cs * q;
#pragma unroll
    for (int v = 0; v < 4; ++v) rU[slot][v] = A.U[it & 1][v * C + c];
#pragma unroll
    for (int v = 0; v < 3; ++v) rx[slot][v] = A.xc[v * C + c];
    if (q >= 1) {
      const int t = fb0 + cs * q;
      rdb[slot] = A.fd.db[D][t]; rdf[slot] = A.fd.df[D][t];
      ru[slot] = A.fd.u[D][t]; rA[slot] = A.fd.A[D][t];
#pragma unroll
      for (int v = 0; v < 3; ++v) rn[slot][v] = A.n0[v * F + foff + t];
    }
  };
  // the window, indexed by slots
  R P[4][4], G[4][4], g[4][4], Fv[4][4], fx[4];    // fx: (x_f - x_c).n0 of the upwind cell
  double xc[4][3], uf[4], Af[4];
  bool back[4];
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    uf[s] = Af[s] = 0.; fx[s] = 0; back[s] = false;
#pragma unroll
    for (int v = 0; v < 4; ++v) { P[s][v] = 0; G[s][v] = 0; g[s][v] = 0; Fv[s][v] = 0; }
#pragma unroll
    for (int v = 0; v < 3; ++v) xc[s][v] = 0.;
  }
  const int q0 = a - 2 > 0 ? a - 2 : 0;
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    rdb[s] = rdf[s] = ru[s] = rA[s] = 0.;
#pragma unroll
    for (int v = 0; v < 4; ++v) rU[s][v] = 0.;
#pragma unroll
    for (int v = 0; v < 3; ++v) { rx[s][v] = 0.; rn[s][v] = 0.; }
  }
  load(0, q0);
  constexpr int s1 = 1, s2 = 2, s3 = 3, cur = 0;                  // slots: q - 2, q - 1, q
#pragma unroll 1
  for (int q = q0; q <= b + 1; ++q) {
    if constexpr (BAT) asm volatile("" ::: "memory");             // no pointer is kept over a step
    if (q + 1 < nd && q <= b) load(cur ^ 1, q + 1);
    const int m = q - 2;
    const bool own = m >= a;
    const int c = cb0 + cs * m;
    double U[4] = {0., 0., 0., 0.}, ob = 0., of = 0., vol = 0.;
    if (own) {
#pragma unroll
      for (int v = 0; v < 4; ++v) U[v] = A.U[it & 1][v * C + c];
      ob = A.ofn[lb * C + c]; of = A.ofn[lf * C + c];
      if (LAST) vol = A.st.Ve[c];
    }
#pragma unroll
    for (int v = 0; v < 4; ++v) { g[s3][v] = 0; Fv[s2][v] = 0; }
    // the new cell and its low face
    if (q < nd) {
      phi_of<R, false>(rU[cur], P[s3], nullptr);
#pragma unroll
      for (int v = 0; v < 3; ++v) xc[s3][v] = rx[cur][v];
      if (q > q0) {                                     // both cells of the face are at hand, and q >= 1
        const double dx = dot(d3(xc[s3][0], xc[s3][1], xc[s3][2]) - d3(xc[s2][0], xc[s2][1], xc[s2][2]),
                              d3(rn[cur][0], rn[cur][1], rn[cur][2]));
        const R dxR = (R)dx, r = rc<R, false>(dxR, nullptr);
#pragma unroll
        for (int v = 1; v < 4; ++v) g[s3][v] = dv<R, false>(P[s3][v] - P[s2][v], dxR, r, nullptr);
        uf[s3] = ru[cur]; Af[s3] = rA[cur];
        back[s3] = ru[cur] * dx > 0.0;
        fx[s3] = (R)(back[s3] ? rdb[cur] : rdf[cur]);
      }
    }
    // limited gradient of q - 1, then the upwind value of its low face
    if (q >= a && q >= 1 && q - 1 < nd) {
      limited_grad<R>(lim, g[s2], g[s3], G[s2]);
      if (q >= 2 && q > a) face_value<R>(order2, back[s2], fx[s2], P[s1], G[s1], P[s2], G[s2], Fv[s2]);
    }
    if (own) {
      const bool in1 = m >= 1, fr1 = m + 1 <= nd - 1;
      const double cb = in1 ? ob * uf[s1] * Af[s1] * dt : 0.;
      const double cf = fr1 ? of * uf[s2] * Af[s2] * dt : 0.;
      double u[4], dpm = 0.;
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        double flux_face = 0., dp = 0.;
        if (in1) { const double fl = (double)((R)cb * Fv[s1][v]); flux_face += fl; dp += 0.5 * fl * ob; }
        if (fr1) { const double fl = (double)((R)cf * Fv[s2][v]); flux_face += fl; dp += 0.5 * fl * of; }
        u[v] = U[v] - flux_face;
        if (v == 1) dpm = dp;
      }
      if (u[1] < 0.) u[1] = 0.;
      if (u[2] < 0.) u[2] = 0.;
      if constexpr (!LAST) {
#pragma unroll
        for (int v = 0; v < 4; ++v) A.U[(it + 1) & 1][v * C + c] = u[v];
      } else {
        double out[8];
        finalize_cell_mixed(ph, A.S, vol, u, out);
        A.st.rho[c] = out[0]; A.st.e[c] = out[1]; A.st.q[c] = out[2]; A.st.mass[c] = out[3];
        A.st.p[c] = out[4]; A.st.cs[c] = out[5];
        if (A.st.mf) A.st.mf[c] = out[7];
      }
      A.dpf[c] = dpm;
    }
    // shift the window
#pragma unroll
    for (int s = 1; s < 3; ++s) {
      uf[s] = uf[s + 1]; Af[s] = Af[s + 1]; fx[s] = fx[s + 1]; back[s] = back[s + 1];
#pragma unroll
      for (int v = 0; v < 4; ++v) { P[s][v] = P[s + 1][v]; G[s][v] = G[s + 1][v]; g[s][v] = g[s + 1][v]; Fv[s][v] = Fv[s + 1][v]; }
#pragma unroll
      for (int v = 0; v < 3; ++v) xc[s][v] = xc[s + 1][v];
    }
    rdb[0] = rdb[1]; rdf[0] = rdf[1]; ru[0] = ru[1]; rA[0] = rA[1];
#pragma unroll
    for (int v = 0; v < 4; ++v) rU[0][v] = rU[1][v];
#pragma unroll
    for (int v = 0; v < 3; ++v) { rx[0][v] = rx[1][v]; rn[0][v] = rn[1][v]; }
  }
}

template <int D, bool LAST, bool BAT>
__device__ __forceinline__ void sweep_cells_march(const CycleArgs& A, int it, int len, int bx_, int seg) {
  const int points = A.dm.nx * (D == 1 ? A.dm.nz : A.dm.ny);
  const int point = bx_ * kMarchThreads + threadIdx.x;
  if (point >= points) return;
  cells_march<D, LAST, BAT>(A, it, point, seg, march_segments(A.dm.ncd(D), points, len));
}

template <int D, bool LAST>
__global__ void __launch_bounds__(kMarchThreads, 4) k_cyc_sweep_cells_m(const __grid_constant__ CycleArgs a, int it, int len) {
  sweep_cells_march<D, LAST, false>(a, it, len, blockIdx.x, blockIdx.y);
}

// The same over a batch's work table (instance, plane chunk, segment).
template <int D, bool LAST>
__global__ void __launch_bounds__(kMarchThreads, 4) k_bat_sweep_cells_m(const CycleArgs* __restrict__ A,
    const int4* __restrict__ W, int nw, int it, int len) {
  __shared__ CycleArgs a;
  for (int w = blockIdx.x; w < nw; w += gridDim.x) {
    const int4 t = W[w];
    copy_args(a, A + t.x);
    sweep_cells_march<D, LAST, true>(a, it, len, t.y, t.z);
  }
}

// ------------------------------------------------------------------------
// Host-side launchers.
template <int D, bool FIRST, bool LAST, int K, typename R, bool GL>
static void sweep_nodes_launch_m(const CycleArgs& a, int prev, cudaStream_t s) {
  const Dims& dm = a.dm;
  const int points = (dm.nx + 1) * ((D == 1 ? dm.nz : dm.ny) + 1), len = march_len(a.lines[BK_NODES_X + D]);
  const dim3 g((points + kMarchThreads - 1) / kMarchThreads, march_segments(dm.ncd(D) + 1, points, len));
  k_cyc_sweep_nodes_m<D, FIRST, LAST, K, R, GL><<<g, kMarchThreads, 0, s>>>(a, prev, len);
}

template <int D, bool LAST>
static void sweep_cells_launch_m(const CycleArgs& a, int it, cudaStream_t s) {
  const Dims& dm = a.dm;
  const int points = dm.nx * (D == 1 ? dm.nz : dm.ny), len = march_len(a.lines[BK_CELLS_X + D]);
  const dim3 g((points + kMarchThreads - 1) / kMarchThreads, march_segments(dm.ncd(D), points, len));
  k_cyc_sweep_cells_m<D, LAST><<<g, kMarchThreads, 0, s>>>(a, it, len);
}

template <class Kern, class... Args>
static void launch_march(Kern kern, const BatchPlan& P, int kind, cudaStream_t s, KernelMarks* m, Args... args) {
  if (P.nmwork[kind] > 0)
    kern<<<persistent_grid((const void*)kern, kMarchThreads, 0, P.nmwork[kind], P.occ_pct[kind]), kMarchThreads, 0, s>>>(args...);
  mark(m, kind, s);
}

// ------------------------------------------------------------------------
// Node sweeps of a context.


template <int D, bool FIRST, bool LAST, int K, typename R, int W, bool GL = false>
static void sweep_nodes_launch_w(const CycleArgs& a, int prev, const double* udin, double* udout, cudaStream_t s) {
  const Dims& dm = a.dm;
  const int nseg = (dm.ncd(D) + 1 + kLineUpd - 1) / kLineUpd;
  const dim3 g((dm.nx + 1 + W - 1) / W, nseg, (D == 1 ? dm.nz : dm.ny) + 1);
  const size_t smem = NodeTileSize<D, FIRST, LAST, K, W>::bytes;
  auto kern = k_cyc_sweep_nodes_t<D, FIRST, LAST, K, R, W, GL>;
  smem_opt_in((const void*)kern, smem);
  kern<<<g, 32 * W, smem, s>>>(dm, a.S, a.ph, prev, a.x0, a.xl, a.vh, a.nm, udin, udout, a.dpf, a.Gd, a.st.mass, a.v,
                               a.nm, a.vnorm, a.ecn);
}

template <int D, bool FIRST, bool LAST, int K, typename R>
static void sweep_nodes_launch(const CycleArgs& a, int prev, const double* udin, double* udout, cudaStream_t s) {
  const Dims& dm = a.dm;
  const int T = 32 * kLineWarps;
  // the generalised limiters (FP64) have their own kernels
  const bool gl = sizeof(R) == 8 && a.ph.ordre_projection > 1 && a.ph.limiteur_id >= 3;
  if constexpr (D == 0) {
    const int g = row_chunks(dm.N);
    if (gl)
      k_cyc_sweep_nodes_x<FIRST, LAST, K, R, true><<<g, T, 0, s>>>(dm, a.S, a.ph, prev, a.x0, a.xl, a.vh, a.nm, udin,
                                                                udout, a.dpf, a.Gd, a.st.mass, a.v, a.nm, a.vnorm, a.ecn);
    else
      k_cyc_sweep_nodes_x<FIRST, LAST, K, R><<<g, T, 0, s>>>(dm, a.S, a.ph, prev, a.x0, a.xl, a.vh, a.nm, udin, udout,
                                                       a.dpf, a.Gd, a.st.mass, a.v, a.nm, a.vnorm, a.ecn);
  } else {
    if constexpr (sizeof(R) == 4 || FIRST) {
      if (march_nodes(dm.N, a.ph.precision, FIRST)) {
        if constexpr (sizeof(R) == 8) {
          if (gl) { sweep_nodes_launch_m<D, FIRST, LAST, K, R, true>(a, prev, s); return; }
        }
        sweep_nodes_launch_m<D, FIRST, LAST, K, R, false>(a, prev, s);
        return;
      }
    }
    if constexpr (sizeof(R) == 8) {
      if (gl) { sweep_nodes_launch_w<D, FIRST, LAST, K, R, kLineWarps, true>(a, prev, udin, udout, s); return; }
    }
    // lines per block of this sweep (the tuning; K > 1 meshes keep 8)
    const int w = K == 1 ? a.lines[BK_NODES_X + D] : kLineWarps;
    if (w == 32) sweep_nodes_launch_w<D, FIRST, LAST, K, R, 32>(a, prev, udin, udout, s);
    else if (w == 16) sweep_nodes_launch_w<D, FIRST, LAST, K, R, 16>(a, prev, udin, udout, s);
    else sweep_nodes_launch_w<D, FIRST, LAST, K, R, 8>(a, prev, udin, udout, s);
  }
}

// One node sweep along D of a mesh with K environments (dual mass fluxes in K planes).
template <int D, int K, typename R>
static void sweep_nodes_d(const CycleArgs& a, bool first, bool last, int prev, const double* udin, double* udout,
                          cudaStream_t s) {
  if (first) sweep_nodes_launch<D, true, false, K, R>(a, prev, udin, udout, s);
  else if (last) sweep_nodes_launch<D, false, true, K, R>(a, prev, udin, udout, s);
  else sweep_nodes_launch<D, false, false, K, R>(a, prev, udin, udout, s);
}

// R: evaluation precision of the sweep (double, or float in the mixed form).
template <int K, typename R = double>
static void sweep_nodes(const CycleArgs& a, int d, bool first, bool last, int prev, const double* udin,
                        double* udout, cudaStream_t s) {
  if (d == 0) sweep_nodes_d<0, K, R>(a, first, last, prev, udin, udout, s);
  else if (d == 1) sweep_nodes_d<1, K, R>(a, first, last, prev, udin, udout, s);
  else sweep_nodes_d<2, K, R>(a, first, last, prev, udin, udout, s);
}


}  // namespace mhy
