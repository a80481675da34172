// sph_noalloc.cu — SPH density by direct summation for callers that cannot
// allocate device memory.
//
// Some callers of this library must not call cudaMalloc: a code that runs
// inside another application's fixed device-memory budget (an in-situ
// analysis hook handed particle arrays by a host simulation, or a process
// whose allocator is owned by a framework), or a caller that must not risk
// the implicit device synchronisation of cudaMalloc/cudaFree in a
// latency-critical loop.  sph_density_noalloc serves them: the caller passes
// device pointers to the inputs and the output, and every intermediate array
// (cell keys, sorted order, cell starts, sorted positions, scan workspace)
// lives in one file-scope __device__ array of fixed size.
//
// The array is SPH_NOALLOC_SCRATCH_BYTES per GPU and exists on every GPU that
// loads the library until the process exits.  Its device address is looked
// up once per device, with that device current, on the first call made on
// it (cudaGetSymbolAddress).  Every call uses the same array, so calls that
// overlap on the GPU (concurrent streams, several host threads) race and
// give wrong results; the function synchronises its stream before
// returning.  What must start at zero or at a sentinel is cleared by the
// call itself.
//
// The density is circuit1's direct summation (circuit1.f90:253-296):
//   rho_i = sum_{j != i, r_ij <= krad h_i} m_j W(r_ij, h_i) + m_i W(0, h_i)
// over the particles as given (no periodic images), with the neighbour
// test of the kd-tree search (kdtree2.f90:1673-1678) in FP64.
#include <cub/device/device_scan.cuh>

#include <cmath>
#include <cstddef>
#include <mutex>
#include <string>

#include "sph_internal.h"

namespace sph {
namespace {

constexpr size_t kScratchBytes = SPH_NOALLOC_SCRATCH_BYTES;
static __device__ __align__(256) unsigned char g_noalloc_scratch[kScratchBytes];

constexpr int kMaxDevices = 64;
void* g_scratch_ptr[kMaxDevices] = {nullptr};
std::mutex g_scratch_mu;

// Device address of the scratch array on the current device (looked up once).
int scratch_address(void** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return sph_fail(SPH_ERR_CUDA, std::string("cudaGetDevice: ") + cudaGetErrorString(e));
  if (dev < 0 || dev >= kMaxDevices) return sph_fail(SPH_ERR_CUDA, "device index out of range");
  std::lock_guard<std::mutex> lk(g_scratch_mu);
  if (!g_scratch_ptr[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess || !p)
      return sph_fail(SPH_ERR_CUDA, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
    g_scratch_ptr[dev] = p;
  }
  *out = g_scratch_ptr[dev];
  return SPH_OK;
}

constexpr int TPB = 256;
inline int nblocks(int64_t n) { return int((n + TPB - 1) / TPB > 0 ? (n + TPB - 1) / TPB : 1); }

__device__ __forceinline__ double pos_of(const double* a, int64_t i) { return a ? a[i] : 0.0; }

// What the host used to read back before it could size the grid, planned on
// the device instead: one wait for the GPU per call, at its end.
struct NaPlan {
  unsigned long long red[7];  // min x, y, z and h as ~key, max x, y, z as key (0 = nothing seen)
  unsigned int blocks_done;
  int err;     // 0, or why there is no grid (the later kernels then write nothing)
  int status;  // first error of the density sum
  Grid g;          // (nx counts the fine cells along x)
  double fx;       // how much shorter a cell is along x than L: 4, or 1
};

__device__ __forceinline__ unsigned long long umax64(unsigned long long a, unsigned long long b) {
  return a > b ? a : b;
}

// Bounding box and smallest h, then, in the last block to finish, the grid.
// The block's threads reduce through shuffles and shared memory and leave
// 7 atomics per block; one set per particle, all on the same 7 words, took
// 1.21 ms at 262,144 particles, this 6 us.
// Cell edge L: half of krad h_min, widened until the grid fits the scratch.
// Along x, where a row's candidates are one run, the cells are L / 4 if that
// fits: the run then ends closer to the sphere and no row is added
// (262,144 particles in 3D: 627 us with cells of L, 583 with L / 4).
__global__ void __launch_bounds__(TPB) k_na_reduce(const double* x, const double* y,
                                                   const double* z, const double* h, int64_t n,
                                                   double krad, int64_t max_cells, NaPlan* pl) {
  // (h starts at 1e308: infinite and NaN radii alone give one cell for all)
  unsigned long long v[7] = {0, 0, 0, ~dkey(1e308), 0, 0, 0};
  for (int64_t i = blockIdx.x * int64_t(TPB) + threadIdx.x; i < n; i += int64_t(gridDim.x) * TPB) {
    const unsigned long long k[4] = {dkey(pos_of(x, i)), dkey(pos_of(y, i)), dkey(pos_of(z, i)),
                                     dkey(h[i])};
    for (int d = 0; d < 3; ++d) {
      v[d] = umax64(v[d], ~k[d]);
      v[4 + d] = umax64(v[4 + d], k[d]);
    }
    v[3] = umax64(v[3], ~k[3]);
  }
  __shared__ unsigned long long part[TPB / 32][7];
  for (int k = 0; k < 7; ++k) {
    for (int o = 16; o > 0; o >>= 1) v[k] = umax64(v[k], __shfl_xor_sync(0xffffffffu, v[k], o));
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5][k] = v[k];
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  for (int k = 0; k < 7; ++k) {
    for (int w = 1; w < TPB / 32; ++w) v[k] = umax64(v[k], part[w][k]);
    atomicMax(&pl->red[k], v[k]);
  }
  __threadfence();
  if (atomicAdd(&pl->blocks_done, 1u) != gridDim.x - 1) return;
  double lo[3], hi[3];
  for (int k = 0; k < 3; ++k) {
    lo[k] = dkey_inv(~atomicMax(&pl->red[k], 0ull));
    hi[k] = dkey_inv(atomicMax(&pl->red[4 + k], 0ull));
  }
  const double hmin = dkey_inv(~atomicMax(&pl->red[3], 0ull));
  if (!(hmin > 0) || !isfinite(hmin)) {
    pl->err = SPH_ERR_IC_H;
    return;
  }
  for (int k = 0; k < 3; ++k)
    if (!isfinite(lo[k]) || !isfinite(hi[k])) {
      pl->err = SPH_ERR_Q_NAN;
      return;
    }
  double L = 0.5 * (krad * hmin);
  int64_t ncell = 0;
  int n3[3] = {1, 1, 1};
  double fx = 4.0;
  for (int guard = 0;; ++guard) {
    double ex[3];
    for (int k = 0; k < 3; ++k) ex[k] = (hi[k] - lo[k]) / L;
    fx = 4.0;
    ex[0] *= fx;
    if (grid_dims(ex, max_cells, n3, &ncell)) break;
    fx = 1.0;
    ex[0] = (hi[0] - lo[0]) / L;
    if (grid_dims(ex, max_cells, n3, &ncell)) break;
    if (guard > 401) {
      pl->err = SPH_ERR_GRID;
      return;
    }
    L *= guard < 401 ? 1.25 : 2.0;  // (the widest: 1.25^401 krad h_min, no half of it)
  }
  pl->g.ox = lo[0]; pl->g.oy = lo[1]; pl->g.oz = lo[2];
  pl->g.L = L; pl->g.invL = 1.0 / L;
  pl->fx = fx;
  pl->g.nx = n3[0]; pl->g.ny = n3[1]; pl->g.nz = n3[2];
}

// cell coordinate of a position in cell units, clamped to the grid (NaN -> 0)
__device__ __forceinline__ int na_clamp(double f, int nc) {
  f = floor(f);
  if (!(f >= 0.0)) return 0;
  if (f >= double(nc - 1)) return nc - 1;
  return int(f);
}

// Counting sort by cell: each particle takes a slot of its cell (in
// whatever order the atomics come), the cells' starts follow from a scan of
// the counts, and k_na_gather puts each cell's particles in increasing
// index, so that the sums below do not depend on the atomics' order.
__global__ void k_na_keys(const double* x, const double* y, const double* z, int64_t n,
                          const NaPlan* pl, uint32_t* keys, int32_t* slot, int32_t* count) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= n || pl->err) return;
  const Grid g = pl->g;
  const uint32_t cx = na_clamp((pos_of(x, i) - g.ox) * g.invL * pl->fx, g.nx);
  const uint32_t cy = na_clamp((pos_of(y, i) - g.oy) * g.invL, g.ny);
  const uint32_t cz = na_clamp((pos_of(z, i) - g.oz) * g.invL, g.nz);
  const uint32_t key = cx + uint32_t(g.nx) * (cy + uint32_t(g.ny) * cz);
  keys[i] = key;
  slot[i] = atomicAdd(&count[key], 1);
}
__global__ void k_na_scatter(int64_t n, const NaPlan* pl, const uint32_t* keys,
                             const int32_t* slot, const int32_t* cstart, int32_t* members) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= n || pl->err) return;
  members[cstart[keys[i]] + slot[i]] = int32_t(i);
}
__global__ void k_na_gather(const double* x, const double* y, const double* z, const double* m,
                            int64_t n, const NaPlan* pl, const uint32_t* keys,
                            const int32_t* cstart, const int32_t* members, int32_t* order,
                            double4* sorted) {
  const int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (pl->err) return;
  const int32_t i = k < n ? members[k] : 0;
  const uint32_t key = keys[i];
  const int32_t at = place_in_cell<TPB>(members, k < n, i, cstart[key], cstart[key + 1]);
  if (k >= n) return;
  order[at] = i;
  sorted[at] = make_double4(pos_of(x, i), pos_of(y, i), pos_of(z, i), m[i]);
}

// the neighbour predicate's squared distance (kdtree2.f90:1673-1678)
__device__ __forceinline__ double na_dist2(const double4& b, const double4& a) {
  const double d0 = __dadd_rn(b.x, -a.x), d1 = __dadd_rn(b.y, -a.y), d2 = __dadd_rn(b.z, -a.z);
  return __dadd_rn(__dadd_rn(__dmul_rn(d0, d0), __dmul_rn(d1, d1)), __dmul_rn(d2, d2));
}

// The rows of cells that a particle's sphere touches, each cut to the chord
// of the sphere, in cell units.  A particle's position in cell units is off
// by at most its own rounding (the grid has at most 4 n + 4096 cells, so
// well below 1e-6), which the margins cover.  NaN radius: the first cell.
template <int DIM>
struct NaRows {
  double u0, u1, u2, rc2, fx;
  int cy0, cz0, ny_r, rows;
  __device__ __forceinline__ NaRows(const Grid& g, double fx_, const double4& p, double R2) : fx(fx_) {
    u0 = (p.x - g.ox) * g.invL;
    u1 = (p.y - g.oy) * g.invL;
    u2 = (p.z - g.oz) * g.invL;
    const double rc = (sqrt(R2) * (1.0 + 1e-9) + 1e-300) * g.invL + 1e-6;
    rc2 = rc * rc;
    cy0 = DIM >= 2 ? na_clamp(u1 - rc, g.ny) : 0;
    cz0 = DIM == 3 ? na_clamp(u2 - rc, g.nz) : 0;
    ny_r = DIM >= 2 ? na_clamp(u1 + rc, g.ny) - cy0 + 1 : 1;
    rows = ny_r * (DIM == 3 ? na_clamp(u2 + rc, g.nz) - cz0 + 1 : 1);  // (at most all cells)
  }
  // the sorted particles first .. first + len - 1 of row r
  __device__ __forceinline__ void run(const Grid& g, const int32_t* cstart, int r, int32_t& first,
                                      int32_t& len) const {
    const int cy = cy0 + r % ny_r, cz = cz0 + r / ny_r;
    double rem = rc2;
    if (DIM >= 2) {
      const double d = fmax(0.0, fmax(double(cy) - u1, u1 - double(cy + 1)) - 1e-6);
      rem -= d * d;
    }
    if (DIM == 3) {
      const double d = fmax(0.0, fmax(double(cz) - u2, u2 - double(cz + 1)) - 1e-6);
      rem -= d * d;
    }
    if (rem < 0.0) return;
    const double w = sqrt(rem) + 1e-6;
    const int64_t row = int64_t(g.nx) * (cy + int64_t(g.ny) * cz);
    first = __ldg(cstart + row + na_clamp((u0 - w) * fx, g.nx));
    len = __ldg(cstart + row + na_clamp((u0 + w) * fx, g.nx) + 1) - first;
  }
};

// The sum over the neighbours, one warp per particle, particles in cell
// order (the warps of a block share their candidates' cache lines).  Lane r
// finds the run of sorted particles of the r-th row of cells that the sphere
// touches (the row cut to the chord of the sphere); the runs, end to end,
// are walked 32 candidates at a time, one per lane, and the candidates that
// are neighbours go, packed, to a queue in shared memory, from which 32 at a
// time get their kernel value: it costs several times a test and less than
// half the candidates are neighbours.  A NaN radius is reported from the
// radius itself: its run, the first cell's, may hold no particle.  (A lone
// particle is not refused: no other one would have met it.)
// Bound by instruction issue (65 % of the slots; FP64 pipe 28 %): 1,800
// instructions a particle, of them 385 FP64.  One thread per particle in the
// caller's order over whole cells of edge krad h_min (7 tests a neighbour,
// every load a cache line of its own) took 2.54 ms for 262,144 particles in
// 3D, M6, two threads per particle in cell order 0.75 ms, this 0.58 ms.
constexpr int DTPB = 128;
template <int K, int DIM>
__global__ void __launch_bounds__(DTPB)
k_na_density(const double* h, int64_t n, NaPlan* pl, double krad, double wcv,
             const int32_t* cstart, const int32_t* order, const double4* sorted, double* rho) {
  constexpr unsigned FULL = 0xffffffffu;
  __shared__ double2 queues[DTPB / 32][64];  // (r^2, m), a ring of 64
  __shared__ int2 run_lists[DTPB / 32][32];
  double2* const queue = queues[threadIdx.x / 32];
  int2* const runs = run_lists[threadIdx.x / 32];
  const int k = int(blockIdx.x * (DTPB / 32) + threadIdx.x / 32);  // the warp's particle
  const int lane = threadIdx.x & 31;
  if (k >= n || pl->err) return;
  const Grid g = pl->g;
  const double4 pi = sorted[k];
  const int32_t i = order[k];
  const double hi = h[i];
  const double kh = __dmul_rn(krad, hi);
  const double R2 = __dmul_rn(kh, kh);
  const double ih = 1.0 / hi;
  const NaRows<DIM> sphere(g, pl->fx, pi, R2);
  double sum = 0.0;
  bool bad = lane == 0 && n > 1 && !(R2 >= 0.0);
  unsigned head = 0;  // the queue's first entry
  int held = 0;       // and its length
  auto value = [&](bool on) {
    if (on) {
      const double2 v = queue[(head + lane) & 63u];
      const double q = sqrt(v.x) * ih;
      bad |= !(q >= 0.0);
      sum += v.y * kshape_f<K, double>(q);
    }
  };
  for (int r0 = 0; r0 < sphere.rows; r0 += 32) {
    int32_t first = 0, len = 0;
    const int r = r0 + lane;
    if (r < sphere.rows) sphere.run(g, cstart, r, first, len);
    // the non-empty runs to the first lanes, with their places end to end
    const unsigned some = __ballot_sync(FULL, len > 0);
    if (len > 0) runs[__popc(some & ((1u << lane) - 1u))] = make_int2(first, len);
    __syncwarp();
    const int2 mine = runs[lane];
    first = mine.x;
    len = lane < __popc(some) ? mine.y : 0;
    int end = len;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int t = __shfl_up_sync(FULL, end, d);
      if (lane >= d) end += t;
    }
    const int total = __shfl_sync(FULL, end, 31);
    const int begin = len > 0 ? end - len : total;  // (no run: never begins)
    const int32_t shift = first - begin;
    for (int p0 = 0; p0 < total; p0 += 32) {
      // this lane's run: the last one that begins at or before p0 + lane
      const unsigned here = begin >= p0 && begin < p0 + 32 ? 1u << (begin - p0) : 0u;
      const unsigned starts = __reduce_or_sync(FULL, here);
      const int before = __popc(__ballot_sync(FULL, begin < p0));
      const int run = before + __popc(starts & (0xffffffffu >> (31 - lane))) - 1;
      const int32_t q = p0 + lane + __shfl_sync(FULL, shift, run);
      bool hit = false;
      double sd = 0.0, mj = 0.0;
      if (p0 + lane < total) {
        const double4 pj = sorted[q];
        sd = na_dist2(pj, pi);
        mj = pj.w;
        hit = !(sd > R2) && q != k;  // the particle itself: neighboursearch.f90:190
      }
      const unsigned hits = __ballot_sync(FULL, hit);
      if (hit)
        queue[(head + held + __popc(hits & ((1u << lane) - 1u))) & 63u] = make_double2(sd, mj);
      held += __popc(hits);
      __syncwarp();
      if (held >= 32) {
        value(true);
        head += 32;
        held -= 32;
        __syncwarp();
      }
    }
    __syncwarp();  // (the next rows overwrite the runs)
  }
  value(lane < held);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(FULL, sum, o);
  if (lane == 0) {
    const double self = pi.w * kshape_f<K, double>(0.0);
    rho[i] = wcv * (sum + self) / ipow<DIM>(hi);
  }
  if (bad) atomicCAS(&pl->status, 0, SPH_ERR_Q_NAN);
}

// Two lanes per particle, for 1D and 2D sets that fill the GPU that way:
// their few short rows leave most of a warp's lanes without a candidate
// (262,144 particles, M6: 2D 194 us a call against 287 us with a warp per
// particle, 1D 92 against 182; at 5,000 particles, where the warps are
// needed to fill the SMs, 2D 85 against 68).
template <int K, int DIM>
__global__ void __launch_bounds__(DTPB)
k_na_density2(const double* h, int64_t n, NaPlan* pl, double krad, double wcv,
              const int32_t* cstart, const int32_t* order, const double4* sorted, double* rho) {
  const int k = int((blockIdx.x * int64_t(DTPB) + threadIdx.x) / 2);
  const int sub = threadIdx.x & 1;
  if (pl->err) return;
  double sum = 0.0, hi = 1.0, mi = 0.0;
  bool bad = false;
  if (k < n) {
    const Grid g = pl->g;
    const double4 pi = sorted[k];
    mi = pi.w;
    hi = h[order[k]];
    const double kh = __dmul_rn(krad, hi);
    const double R2 = __dmul_rn(kh, kh);
    const double ih = 1.0 / hi;
    bad = n > 1 && !(R2 >= 0.0);
    const NaRows<DIM> sphere(g, pl->fx, pi, R2);
    // the rows in turn; of the one row of 1D, and where far outliers have made
    // the cells so wide that a sphere meets 3 rows at most (5 otherwise), the
    // candidates (100,000 particles in one cell: 43 ms by rows, 24 so)
    const bool by_row = DIM == 2 && sphere.rows > 3;
    const int row_step = by_row ? 2 : 1, step = by_row ? 1 : 2;
    for (int r = by_row ? sub : 0; r < sphere.rows; r += row_step) {
      int32_t first = 0, len = 0;
      sphere.run(g, cstart, r, first, len);
      for (int t = by_row ? 0 : sub; t < len; t += step) {
        const int32_t q = first + t;
        const double4 pj = sorted[q];
        const double sd = na_dist2(pj, pi);
        if (sd > R2 || q == k) continue;  // the particle itself: neighboursearch.f90:190
        const double q_ = sqrt(sd) * ih;
        bad |= !(q_ >= 0.0);
        sum += pj.w * kshape_f<K, double>(q_);
      }
    }
  }
  sum += __shfl_xor_sync(0xffffffffu, sum, 1);
  if (k < n && sub == 0) {
    const double self = mi * kshape_f<K, double>(0.0);
    rho[order[k]] = wcv * (sum + self) / ipow<DIM>(hi);
  }
  if (bad) atomicCAS(&pl->status, 0, SPH_ERR_Q_NAN);
}

struct NaLaunch {
  const double* h;
  int64_t n;
  NaPlan* pl;
  double krad, wcv;
  const int32_t* cstart;
  const int32_t* order;
  const double4* sorted;
  double* rho;
  cudaStream_t s;
};
template <int K, int DIM>
void launch_density_d(const NaLaunch& a) {
  auto blocks = [&](int lanes) { return int((a.n * lanes + DTPB - 1) / DTPB); };
  // 30,000: two lanes each are then a fifth of the GPU's threads (148 x
  // 2048); measured crossing between 5,000 and 100,000
  if (DIM <= 2 && a.n >= 30000)
    k_na_density2<K, DIM><<<blocks(2), DTPB, 0, a.s>>>(a.h, a.n, a.pl, a.krad, a.wcv, a.cstart,
                                                      a.order, a.sorted, a.rho);
  else
    k_na_density<K, DIM><<<blocks(32), DTPB, 0, a.s>>>(a.h, a.n, a.pl, a.krad, a.wcv, a.cstart,
                                                      a.order, a.sorted, a.rho);
}
template <int K>
void launch_density(int dim, const NaLaunch& a) {
  if (dim == 3) launch_density_d<K, 3>(a);
  else if (dim == 2) launch_density_d<K, 2>(a);
  else launch_density_d<K, 1>(a);
}

// carve `bytes` (256-aligned) out of the scratch array
struct Carver {
  unsigned char* base;
  size_t used = 0;
  void* take(size_t bytes) {
    void* p = base + used;
    used += (bytes + 255) & ~size_t(255);
    return p;
  }
};

}  // namespace
}  // namespace sph

using namespace sph;

extern "C" int sph_density_noalloc(const double* x, const double* y, const double* z,
                                   const double* m, const double* h, int64_t n, int dim,
                                   int kernel_id, double* rho, void* stream) {
  if (n < 1 || n > SPH_NOALLOC_MAX_PARTICLES)
    return sph_fail(SPH_ERR_ARG, "sph_density_noalloc: n must be in 1.." +
                                     std::to_string(SPH_NOALLOC_MAX_PARTICLES) + ", got " +
                                     std::to_string(n));
  if (dim < 1 || dim > 3) return sph_fail(SPH_ERR_ARG, "sph_density_noalloc: dim must be 1, 2 or 3");
  if (kernel_id < 0 || kernel_id > 2) return sph_fail(SPH_ERR_ARG, "sph_density_noalloc: bad kernel id");
  if (!x || !m || !h || !rho || (dim >= 2 && !y) || (dim == 3 && !z))
    return sph_fail(SPH_ERR_ARG, "sph_density_noalloc: null device pointer");
  if (dim < 2) y = nullptr;
  if (dim < 3) z = nullptr;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // The scratch address is the current device's; a stream of another device
  // would run the kernels there with this device's address.
  if (s) {
    int cur = -1, sdev = -1;
    cudaError_t ge = cudaGetDevice(&cur);
    if (ge == cudaSuccess) ge = cudaStreamGetDevice(s, &sdev);
    if (ge != cudaSuccess)
      return sph_fail(SPH_ERR_CUDA, std::string("sph_density_noalloc: ") + cudaGetErrorString(ge));
    if (sdev != cur)
      return sph_fail(SPH_ERR_ARG, "sph_density_noalloc: the stream belongs to device " +
                                       std::to_string(sdev) + ", the current device is " +
                                       std::to_string(cur));
  }
  void* base = nullptr;
  int rc = scratch_address(&base);
  if (rc) return rc;
  // knorm / krad of the kernel bases (base_m4.f90:12,18; base_m6.f90:13,17; base_gauss.f90:15,19)
  const double pi = 4.0 * std::atan(1.0);
  const double norms[3][3] = {{2. / 3., 10. / (7. * pi), 1. / pi},
                              {1. / 120., 7. / (478. * pi), 1. / (120. * pi)},
                              {1. / std::sqrt(pi), 1. / pi, 1. / std::pow(pi, 1.5)}};
  const double krads[3] = {2.0, 3.0, 10.0};
  const double wcv = norms[kernel_id][dim - 1], krad = krads[kernel_id];

  Carver cv{static_cast<unsigned char*>(base)};
  // (the plan and the counts lie side by side: one clear serves both)
  const int64_t max_cells = 4 * n + 4096;
  auto* plan = static_cast<NaPlan*>(cv.take(sizeof(NaPlan)));
  auto* cstart = static_cast<int32_t*>(cv.take(sizeof(int32_t) * (max_cells + 1)));
  const size_t clear_bytes = cv.used;
  auto* keys = static_cast<uint32_t*>(cv.take(sizeof(uint32_t) * n));
  auto* slot = static_cast<int32_t*>(cv.take(sizeof(int32_t) * n));
  auto* members = static_cast<int32_t*>(cv.take(sizeof(int32_t) * n));
  auto* order = static_cast<int32_t*>(cv.take(sizeof(int32_t) * n));
  auto* sorted = static_cast<double4*>(cv.take(sizeof(double4) * n));
  size_t scan_bytes = 0;
  cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, cstart, cstart, int(max_cells + 1), s);
  void* scan_tmp = cv.take(scan_bytes);
  if (cv.used > kScratchBytes) return sph_fail(SPH_ERR_ARG, "sph_density_noalloc: scratch too small for n");

  cudaError_t e = cudaMemsetAsync(plan, 0, clear_bytes, s);
  if (e != cudaSuccess) return sph_fail(SPH_ERR_CUDA, cudaGetErrorString(e));
  // (4 particles per thread: fewer blocks, so fewer atomics, at no loss)
  k_na_reduce<<<nblocks((n + 3) / 4), TPB, 0, s>>>(x, y, z, h, n, krad, max_cells, plan);
  k_na_keys<<<nblocks(n), TPB, 0, s>>>(x, y, z, n, plan, keys, slot, cstart);
  cub::DeviceScan::ExclusiveSum(scan_tmp, scan_bytes, cstart, cstart, int(max_cells + 1), s);
  k_na_scatter<<<nblocks(n), TPB, 0, s>>>(n, plan, keys, slot, cstart, members);
  k_na_gather<<<nblocks(n), TPB, 0, s>>>(x, y, z, m, n, plan, keys, cstart, members, order, sorted);
  const NaLaunch a{h, n, plan, krad, wcv, cstart, order, sorted, rho, s};
  if (kernel_id == SPH_KERNEL_M6) launch_density<KM6>(dim, a);
  else if (kernel_id == SPH_KERNEL_M4) launch_density<KM4>(dim, a);
  else launch_density<KGAUSS>(dim, a);
  // this library's own kernels (reduce, keys, scatter, gather, density); the
  // scan's kernels are CUB's and are not counted, as in the engine's launch
  // counter
  note_launch(5);
  int code[2] = {0, 0};  // NaPlan::err, NaPlan::status
  static_assert(offsetof(NaPlan, status) == offsetof(NaPlan, err) + sizeof(int), "read as a pair");
  e = cudaMemcpyAsync(code, &plan->err, sizeof(code), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) return sph_fail(SPH_ERR_CUDA, std::string("sph_density_noalloc: ") + cudaGetErrorString(e));
  if (code[0] == SPH_ERR_IC_H) return sph_fail(SPH_ERR_IC_H, "smoothing length <= 0");
  if (code[0] == SPH_ERR_GRID) return sph_fail(SPH_ERR_GRID, "cell grid would not fit");
  const int rc_sum = code[0] ? code[0] : code[1];
  if (rc_sum) return sph_fail(rc_sum, "q is nan");
  return SPH_OK;
}
