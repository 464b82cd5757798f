// mhy_noalloc.cu -- the CFL time-step reduction for callers that cannot
// allocate device memory.
//
// Who needs it: a host framework that owns every device allocation (Arcane
// hands out its variables from its own allocator and unified memory; a plugin
// is not supposed to call cudaMalloc behind its back), and code that records
// its work into a stream capture, where cudaMalloc is not a legal call.  Such a
// caller already holds the mesh fields on the device and only needs the time
// step computed from them.
//
// The reduction needs scratch memory (one partial minimum per block of the
// first pass).  Here that scratch is a file-scope __device__ array, so the
// entry point allocates nothing: it issues one or two kernel launches on the
// caller's stream and returns.
//
// Limits and sharing, stated for users:
//  * the scratch holds kNoAllocBlocks partial minima (64 KiB per GPU, kept by
//    every GPU that loads this library until the process exits);
//  * the first pass uses at most kNoAllocBlocks blocks of 256 threads; meshes
//    are limited to kNoAllocMaxCells cells (64 a thread), larger ones are
//    rejected with MHY_ERR_ARG.  Small meshes take one launch, which leaves the
//    scratch alone;
//  * every call on a device shares the same scratch and leaves its partial
//    minima there; each call writes every slot it reads before reading it, so
//    nothing has to be cleared, but calls that overlap on the GPU (different
//    streams, or different host threads on one device) race on the scratch and
//    must be serialised by the caller;
//  * the first call on a device looks up the scratch's device address with
//    cudaGetSymbolAddress (with that device current); make that first call
//    before any stream capture.  The address is kept per device together with
//    the identity of the device's current CUDA context, and looked up again
//    when that context has changed (after cudaDeviceReset, for instance), so
//    the first call after such a reset must also come before any capture;
//  * a cell whose L / (c + max |v|) is NaN or negative (an inverted cell, a NaN
//    field) is not skipped: the call then writes out[0] = NaN and out[1] = 0,
//    a time step below any positive deltat-min, so a caller that checks the
//    new dt against deltat-min stops as the reference does (MahycoModule.cc:
//    2152-2159).  The context's own reduction raises MHY_STATUS_NAN_DT for the
//    same cells.
#include <cuda.h>
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <mutex>

#include "mhy_kernels.cuh"

namespace mhy {
namespace {

constexpr int kNoAllocBlocks = 8192;
constexpr int kNoAllocThreads = 256;
constexpr int kNoAllocCellsPerThread = 64;
constexpr long long kNoAllocMaxCells = (long long)kNoAllocBlocks * kNoAllocThreads * kNoAllocCellsPerThread;
constexpr int kNoAllocLayers = 4;                   // a segment's layers on meshes that do not fill the chip
constexpr int kNoAllocCluster = 8;                  // blocks of the portable cluster size
constexpr int kNoAllocClusterThreads = 1024;
constexpr unsigned long long kDblMaxBits = 0x7fefffffffffffffull;
// A block's partial minimum is the bit pattern of a non-negative double (bit
// 63 clear); bit 63 set records that the block met an invalid cell.
constexpr unsigned long long kInvalidBit = 0x8000000000000000ull;

static __device__ __align__(256) unsigned long long g_dt_scratch[kNoAllocBlocks];

constexpr int kMaxDevices = 64;
std::mutex g_mutex;
struct ScratchAddr {
  unsigned long long* addr = nullptr;
  unsigned long long ctx_id = 0;   // CUDA context the address belongs to (0: unknown)
};
ScratchAddr g_scratch[kMaxDevices];

// Identity of the calling thread's current CUDA context (cuCtxGetId through
// the runtime's driver entry points, so the library does not link libcuda);
// 0 when there is none or the driver cannot say.
unsigned long long current_ctx_id() {
  using GetCurrent = CUresult (*)(CUcontext*);
  using GetId = CUresult (*)(CUcontext, unsigned long long*);
  static GetCurrent get_current = nullptr;
  static GetId get_id = nullptr;
  static bool looked_up = false;
  if (!looked_up) {             // under g_mutex
    void* f1 = nullptr;
    void* f2 = nullptr;
    cudaDriverEntryPointQueryResult q1 = cudaDriverEntryPointSymbolNotFound, q2 = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f1, cudaEnableDefault, &q1) == cudaSuccess &&
        q1 == cudaDriverEntryPointSuccess)
      get_current = reinterpret_cast<GetCurrent>(f1);
    if (cudaGetDriverEntryPoint("cuCtxGetId", &f2, cudaEnableDefault, &q2) == cudaSuccess &&
        q2 == cudaDriverEntryPointSuccess)
      get_id = reinterpret_cast<GetId>(f2);
    cudaGetLastError();
    looked_up = true;
  }
  if (!get_current || !get_id) return 0;
  CUcontext ctx = nullptr;
  unsigned long long id = 0;
  if (get_current(&ctx) != CUDA_SUCCESS || !ctx) return 0;
  if (get_id(ctx, &id) != CUDA_SUCCESS) return 0;
  return id;
}

__device__ __forceinline__ unsigned long long block_min(unsigned long long best, unsigned long long* wmin) {
  for (int o = 16; o > 0; o >>= 1) {
    unsigned long long other = __shfl_down_sync(0xffffffffu, best, o);
    best = other < best ? other : best;
  }
  if ((threadIdx.x & 31) == 0) wmin[threadIdx.x >> 5] = best;
  __syncthreads();
  best = kDblMaxBits;
  if (threadIdx.x < 32) {
    best = threadIdx.x < (blockDim.x >> 5) ? wmin[threadIdx.x] : kDblMaxBits;
    for (int o = 16; o > 0; o >>= 1) {
      unsigned long long other = __shfl_down_sync(0xffffffffu, best, o);
      best = other < best ? other : best;
    }
  }
  return best;  // valid in thread 0
}

// computeHydroDeltaT (MahycoModule.cc:2047-2060) over the cells (p, k0..k1) of
// one column: min of L / (c + max over the cell's nodes of |v|) as the bit
// pattern of a non-negative double (they order like integers); invalid is set
// where a value is NaN or negative.  The maximum is taken over |v|^2, in the
// cell-node order, with one root a cell: the root is monotonic, so its result
// is the maximum of the roots.  The four nodes of a layer's top are the next
// layer's bottom.  Q (four) layers are loaded before the first root and division,
// whose branches would keep the loads apart.
template <int Q>
__device__ __forceinline__ unsigned long long column_dt_min(const Dims& dm, const double* __restrict__ L,
                                                            const double* __restrict__ cs,
                                                            const double* __restrict__ v, int p, int k0, int k1,
                                                            bool& invalid) {
  unsigned long long best = kDblMaxBits;
  const int nx = dm.nx, nnx = nx + 1, np = nnx * (dm.ny + 1), layer = nx * dm.ny;
  const int n0 = p + p / nx;                        // node (i, j) of the plane
  const long long N = dm.N;
  auto speed2 = [&](int n) {                         // the operations of |v| up to the root
    const double x = v[n], y = v[N + n], z = v[2 * N + n];
    return x * x + y * y + z * z;
  };
  auto plane = [&](int k, double* s) {
    const int n = n0 + np * k;
    s[0] = speed2(n); s[1] = speed2(n + 1); s[2] = speed2(n + nnx + 1); s[3] = speed2(n + nnx);
  };
  double b[4];
  plane(k0, b);
  for (int k = k0; k < k1; k += Q) {
    double vmax[Q], lc[Q], cc[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int kq = k + q < k1 ? k + q : k1 - 1;   // past the end the last cell again
      double t[4];
      plane(kq + 1, t);
      lc[q] = L[p + layer * kq];
      cc[q] = cs[p + layer * kq];
      vmax[q] = 0.;
#pragma unroll
      for (int a = 0; a < 4; ++a) vmax[q] = amax(b[a], vmax[q]);
#pragma unroll
      for (int a = 0; a < 4; ++a) vmax[q] = amax(t[a], vmax[q]);
      if (k + q + 1 < k1) {
#pragma unroll
        for (int a = 0; a < 4; ++a) b[a] = t[a];
      }
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const double dx_sound = lc[q] / (cc[q] + sqrt(vmax[q]));
      const unsigned long long bits = (unsigned long long)__double_as_longlong(dx_sound);
      if (dx_sound >= 0.) best = bits < best ? bits : best;
      else invalid = true;
    }
  }
  return best;
}

// The new dt of computeDeltaT (MahycoModule.cc:2144-2150) from the minimum:
// min(cfl * min, 1.05 * dt_old, deltat_max); NaN and 0 after an invalid cell.
__device__ __forceinline__ void write_dt(unsigned long long best, bool bad, double cfl, double dt_old,
                                         double deltat_max, double* __restrict__ out) {
  if (bad) {
    out[0] = __longlong_as_double(0x7ff8000000000000ll);     // quiet NaN: no valid minimum
    out[1] = 0.;
    return;
  }
  const double minimum_aux = __longlong_as_double((long long)best);
  double new_dt = cfl * minimum_aux;
  new_dt = amin(new_dt, 1.05 * dt_old);
  new_dt = amin(new_dt, deltat_max);
  out[0] = minimum_aux;
  out[1] = new_dt;
}

// The minimum over this block's part of the mesh (valid in thread 0), with
// kInvalidBit set when the block met a NaN or negative value.  A thread walks
// segments of `layers` layers of a column, a grid apart.
template <int Q>
__device__ __forceinline__ unsigned long long block_partial(const Dims& dm, const double* __restrict__ L,
                                                            const double* __restrict__ cs,
                                                            const double* __restrict__ v, int layers) {
  __shared__ unsigned long long wmin[32];
  __shared__ int bad;
  if (threadIdx.x == 0) bad = 0;
  __syncthreads();
  unsigned long long best = kDblMaxBits;
  bool invalid = false;
  // (column, segment), columns fastest; kNoAllocMaxCells keeps the counts in 32 bits
  const unsigned points = (unsigned)dm.nx * dm.ny, items = points * (unsigned)((dm.nz + layers - 1) / layers);
  for (unsigned w = blockIdx.x * blockDim.x + threadIdx.x; w < items; w += gridDim.x * blockDim.x) {
    const int seg = (int)(w / points), p = (int)(w - seg * points), k0 = seg * layers;
    const int k1 = k0 + layers < dm.nz ? k0 + layers : dm.nz;
    const unsigned long long b = column_dt_min<Q>(dm, L, cs, v, p, k0, k1, invalid);
    best = b < best ? b : best;
  }
  if (invalid) bad = 1;                             // benign race: every writer stores 1
  best = block_min(best, wmin);                     // its barrier also orders the writes to `bad`
  return bad ? best | kInvalidBit : best;
}

// First pass: one partial minimum per block.
template <int Q>
__global__ void __launch_bounds__(kNoAllocThreads) k_dt_partial_noalloc(Dims dm, const double* __restrict__ L,
    const double* __restrict__ cs, const double* __restrict__ v, int layers, unsigned long long* __restrict__ scratch) {
  const unsigned long long best = block_partial<Q>(dm, L, cs, v, layers);
  if (threadIdx.x == 0) scratch[blockIdx.x] = best;
}

// The whole call on one cluster: its first block gathers the partial minima in
// its shared memory.
template <int Q>
__global__ void __launch_bounds__(kNoAllocClusterThreads) k_dt_cluster_noalloc(Dims dm, const double* __restrict__ L,
    const double* __restrict__ cs, const double* __restrict__ v, double cfl, double dt_old, double deltat_max,
    double* __restrict__ out) {
  __shared__ unsigned long long part[kNoAllocCluster];
  auto cluster = cooperative_groups::this_cluster();
  cluster.barrier_arrive();                         // this block runs
  unsigned long long best = block_partial<Q>(dm, L, cs, v, Q);
  cluster.barrier_wait();                           // every block runs, so its shared memory is there
  if (threadIdx.x == 0) cluster.map_shared_rank(part, 0)[blockIdx.x] = best;
  cluster.sync();
  if (blockIdx.x || threadIdx.x) return;
  unsigned long long bad = 0ull;
  best = kDblMaxBits;
  for (unsigned b = 0; b < kNoAllocCluster; ++b) {
    const unsigned long long m = part[b] & ~kInvalidBit;
    bad |= part[b] & kInvalidBit;
    best = m < best ? m : best;
  }
  write_dt(best, bad != 0ull, cfl, dt_old, deltat_max, out);
}

// Second pass: minimum of the partial minima, then the new dt.
__global__ void k_dt_final_noalloc(const unsigned long long* __restrict__ scratch, int nparts, double cfl,
                                   double dt_old, double deltat_max, double* __restrict__ out) {
  __shared__ unsigned long long wmin[32];
  __shared__ int bad;
  if (threadIdx.x == 0) bad = 0;
  __syncthreads();
  unsigned long long best = kDblMaxBits;
  bool invalid = false;
  for (int t = threadIdx.x; t < nparts; t += blockDim.x) {
    const unsigned long long s = scratch[t];
    if (s & kInvalidBit) invalid = true;
    const unsigned long long b = s & ~kInvalidBit;
    best = b < best ? b : best;
  }
  if (invalid) bad = 1;
  best = block_min(best, wmin);
  if (threadIdx.x == 0) write_dt(best, bad, cfl, dt_old, deltat_max, out);
}

}  // namespace
}  // namespace mhy

extern "C" int mhy_compute_hydro_dt_noalloc(int32_t nx, int32_t ny, int32_t nz, const double* L, const double* cs,
                                            const double* v, double cfl, double dt_old, double deltat_max,
                                            double* out, void* stream) {
  using namespace mhy;
  if (nx < 1 || ny < 1 || nz < 1 || !L || !cs || !v || !out) return MHY_ERR_ARG;
  Dims dm{};
  dm.nx = nx; dm.ny = ny; dm.nz = nz;
  dm.C = (long long)nx * ny * nz;
  dm.N = (long long)(nx + 1) * (ny + 1) * (nz + 1);
  if (dm.C > kNoAllocMaxCells) return MHY_ERR_ARG;  // beyond the scratch's capacity
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return MHY_ERR_CUDA;
  unsigned long long* scratch = nullptr;
  {
    std::lock_guard<std::mutex> lock(g_mutex);
    ScratchAddr& sa = g_scratch[dev];
    const unsigned long long id = current_ctx_id();
    if (!sa.addr || id == 0 || id != sa.ctx_id) {
      // set-up of this device (or of its new context): the scratch's device address
      void* p = nullptr;
      if (cudaGetSymbolAddress(&p, g_dt_scratch) != cudaSuccess || !p) {
        cudaGetLastError();
        sa = ScratchAddr{};
        return MHY_ERR_CUDA;
      }
      sa.addr = static_cast<unsigned long long*>(p);
      sa.ctx_id = current_ctx_id();                 // the lookup has made the context current
    }
    scratch = sa.addr;
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // A thread walks segments of 4 layers, of 8 where those still fill the chip
  // (148 SMs x 8 blocks), and of one layer where longer ones do not pay:
  //  * one layer of cells: there is nothing to walk, and the other three of a chunk
  //    of four would be the same cell again (2048x1024x1 91 -> 51 us, 500x500x1 17
  //    -> 13);
  //  * layers of less than 4 cells: neighbouring threads would read lines that lie
  //    a segment apart (1x1x32000 38 -> 9 us, 1x1x2000000 138 -> 78, 1x2x1000000
  //    68 -> 57; from 4 cells on segments are ahead: 2x2x500000 50 us against 65);
  //  * layers of less than 128 cells on meshes of 8,193 to 65,536 cells, for the same
  //    reason while that many threads are resident at once (8x8x512 10.7 -> 8.5 us,
  //    1x8x4090 12.6 -> 8.5; nothing between the two at 8x8x1030).
  // One cluster of eight blocks where it has a thread for every segment: a second
  // launch costs more than eight SMs lose.  Measured on B200, the call, against
  // one thread a cell with its eight nodes and roots in two launches: 100x5x5 11.9
  // -> 9.0 us, 32^3 11.9 -> 8.9, 64^3 14.3 -> 11.9, 128^3 66 -> 37, 2048x1024x1 72
  // -> 51, 1x1x2000000 76 -> 78 (a cluster with two segments a thread, for 40^3,
  // took 13.6 us against 11.9 in two launches and was left out).
  const long long points = (long long)nx * ny;
  const bool narrow = points < 128 && dm.C > 8192 && dm.C <= 65536;
  const int q = nz == 1 || points < 4 || narrow ? 1 : kNoAllocLayers;
  const long long segments = points * ((nz + q - 1) / q);
  if (segments <= kNoAllocCluster * kNoAllocClusterThreads) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = kNoAllocCluster;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(kNoAllocCluster);
    cfg.blockDim = dim3((unsigned)((segments + 32 * kNoAllocCluster - 1) / (32 * kNoAllocCluster)) * 32);
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    auto kern = q == 1 ? k_dt_cluster_noalloc<1> : k_dt_cluster_noalloc<kNoAllocLayers>;
    cudaLaunchKernelEx(&cfg, kern, dm, L, cs, v, cfl, dt_old, deltat_max, out);
  } else {
    const int layers = q == 1 || points * ((nz + 7) / 8) < 148LL * 8 * kNoAllocThreads ? q : 8;
    const long long want = (points * ((nz + layers - 1) / layers) + kNoAllocThreads - 1) / kNoAllocThreads;
    const int nblocks = (int)(want < kNoAllocBlocks ? want : kNoAllocBlocks);
    auto first = q == 1 ? k_dt_partial_noalloc<1> : k_dt_partial_noalloc<kNoAllocLayers>;
    first<<<nblocks, kNoAllocThreads, 0, s>>>(dm, L, cs, v, layers, scratch);
    k_dt_final_noalloc<<<1, 1024, 0, s>>>(scratch, nblocks, cfl, dt_old, deltat_max, out);
  }
  if (cudaGetLastError() != cudaSuccess) return MHY_ERR_CUDA;
  return MHY_OK;
}
