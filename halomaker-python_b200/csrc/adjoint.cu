// Differentiable pieces: the SPH density with fixed neighbour lists and its
// adjoint, and the gradient of the direct-sum halo potential.
//
// Density (omp_compute_density, f90:2816-2838) for particle i with its list of
// nv neighbours n_0..n_{nv-1} sorted by distance at the list's reference
// configuration:
//   r = d_{nv-1} / 2,  u_k = d_k / r,
//   rho_i = C (sum_{k<nv-1} m_{n_k} W(u_k) + m_i) / r^3,  C = xyzlong / pi_f,
// with the reference's periodic distance.  The forward uses the same
// explicitly rounded arithmetic as the finder, so with the finder's own lists
// it reproduces the finder's densities bit for bit.
// Adjoint: with upstream g_i = dL/drho_i and e_k the unit separation
// (min-image, pointing from i to n_k),
//   drho_i/dd_k     = C m_{n_k} W'(u_k) / r^4                       (k < nv-1)
//   drho_i/dd_{nv-1} = (C/2) [ -sum_k m_{n_k} W'(u_k) d_k / r^5 - 3 S / r^4 ]
//   dL/dx_{n_k} += g_i drho_i/dd_k e_k,   dL/dx_i -= g_i drho_i/dd_k e_k.
// The weights are recomputed from positions (nothing is stored between the
// passes); contributions are scattered with FP64 atomics, neighbouring
// components together.
//
// Potential gradient (det_halo_energies_1b3 CHP:1413-1427 direct sum,
// E_h = -G sum_{i<j} m_i m_j / r_ij):
//   dE_h/dx_i = G m_i sum_{j != i} m_j (x_i - x_j) / r_ij^3  = -F_i,
// evaluated per halo over all member pairs, positions taken relative to the
// halo's densest member with the reference's strict min-image rule; scaled by
// an upstream weight per halo.
#include <cuda_runtime.h>
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdint>
#include <mutex>
#include <new>
#include <string>
#include <vector>

#include "engine.h"
#include "exact.cuh"
#include "pair64.cuh"
#include "row32.cuh"

namespace ahop {

__device__ __forceinline__ double spline_deriv(double x) {
  // d/dx of the cubic spline of f90:3270-3287
  if (x <= 1.0) return -3.0 * x + 2.25 * x * x;
  if (x <= 2.0) {
    const double y = 2.0 - x;
    return -0.75 * y * y;
  }
  return 0.0;
}

// signed min-image separation b - a along one axis (|.| as in the reference)
__device__ __forceinline__ double pdelta(double a, double b, double L) {
  double d = b - a;
  if (d > 0.5 * L) d -= L;
  else if (d < -0.5 * L) d += L;
  return d;
}

struct AdjArgs {
  const double* pos;   // [n][3]
  const double* mass;  // [n]
  const double4* p4;   // [n] (x, y, z, m), or null: read pos and mass
  const int32_t* nei;  // [n][nv], 0-based
  int64_t n;
  int nv;
  double Lx, Ly, Lz, xyzlong;
};

__global__ void __launch_bounds__(256) pack_kernel(const double* __restrict__ pos, const double* __restrict__ mass,
                                                   int64_t n, double4* __restrict__ p4) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) p4[i] = make_double4(pos[3 * i], pos[3 * i + 1], pos[3 * i + 2], mass[i]);
}

// Both density kernels take one particle per thread and are bound by gathering
// its neighbours from L2 in the caller's (random) order.  kPacked reads them
// from 32-byte rows written beforehand (one sector each instead of 2.75 of the
// (n, 3) positions and the masses); the lists of a warp's 32 particles are read
// as rows of 128 bytes and turned in shared memory.
// 2,097,152 particles with 32 neighbours, ms: forward 0.87 (L2 at 87 % of its
// rate) -> 0.44, backward 2.39 -> 1.13 (latency of the gathers, 28 warps per
// SM: 24 with four neighbours unrolled 1.19, 32 spill, 1.26; the atomics alone
// were 3 x 32 sectors per neighbour and warp).
constexpr int kAB = 128;                   // threads per block
constexpr int64_t kPackMin = 32768;        // below, the extra launch costs more than it saves

template <bool kPacked>
__device__ __forceinline__ double4 particle(const AdjArgs& A, int64_t j) {
  if (kPacked) return load_row(A.p4 + j);
  return make_double4(A.pos[3 * j], A.pos[3 * j + 1], A.pos[3 * j + 2], A.mass[j]);
}

// Entries [k0, k0 + 32) of the lists of a warp's 32 particles from i0 on.
__device__ __forceinline__ void stage_lists(const AdjArgs& A, int64_t i0, int k0, int lane, int32_t (*tile)[33]) {
  __syncwarp();
#pragma unroll 8
  for (int r = 0; r < 32; ++r)
    tile[r][lane] = (i0 + r < A.n && k0 + lane < A.nv) ? A.nei[(i0 + r) * A.nv + k0 + lane] : 0;
  __syncwarp();
}

template <bool kPacked>
__global__ void __launch_bounds__(kAB) density_fixed_kernel(AdjArgs A, double* __restrict__ dens) {
  __shared__ int32_t s_tile[kAB / 32][32][33];
  const int lane = threadIdx.x & 31;
  int32_t(*tile)[33] = s_tile[threadIdx.x >> 5];
  const int64_t i0 = blockIdx.x * (int64_t)kAB + (threadIdx.x & ~31), i = i0 + lane;
  if (i0 >= A.n) return;
  const bool live = i < A.n;
  const double4 me = particle<kPacked>(A, live ? i : A.n - 1);
  const int64_t jl = live ? A.nei[(size_t)A.nv * i + A.nv - 1] : 0;
  const double4 last = particle<kPacked>(A, jl);
  const double dl = pdist2(me.x, me.y, me.z, last.x, last.y, last.z, A.Lx, A.Ly, A.Lz);
  const double r = xmul(xsqrt(dl), 0.5);
  const double r3 = xmul(xmul(r, r), r);
  const double unsr = xdiv(1.0, r);
  double contrib = 0.0;
  for (int k0 = 0; k0 < A.nv - 1; k0 += 32) {
    stage_lists(A, i0, k0, lane, tile);
    const int m = min(32, A.nv - 1 - k0);
#pragma unroll 4
    for (int k = 0; k < m; ++k) {
      const double4 q = particle<kPacked>(A, tile[lane][k]);
      const double d2 = pdist2(me.x, me.y, me.z, q.x, q.y, q.z, A.Lx, A.Ly, A.Lz);
      contrib = xadd(contrib, xmul(q.w, spline(xmul(xsqrt(d2), unsr))));
    }
  }
  const double pi_f = (double)3.141592654f;
  if (live) dens[i] = xdiv(xmul(A.xyzlong, xadd(contrib, me.w)), xmul(pi_f, r3));
}

// The gradient's contributions of a warp's 32 particles to one neighbour each
// (zero: none) go to memory three neighbouring doubles at a time: through
// shared memory lane l takes element l, l + 32 and l + 64 of the 32 vectors, so
// that one instruction's atomics share sectors.
__device__ __forceinline__ void scatter_add(double* __restrict__ gpos, int64_t j, double vx, double vy, double vz,
                                            int lane, double* sv, int64_t* sj) {
  __syncwarp();
  sv[3 * lane] = vx; sv[3 * lane + 1] = vy; sv[3 * lane + 2] = vz;
  sj[lane] = 3 * j;
  __syncwarp();
#pragma unroll
  for (int t = 0; t < 3; ++t) {
    const int e = 32 * t + lane, s = e / 3;
    const double v = sv[e];
    if (v != 0.0) atomicAdd(&gpos[sj[s] + (e - 3 * s)], v);
  }
}

template <bool kPacked>
__global__ void __launch_bounds__(kAB, 7) density_adjoint_kernel(AdjArgs A, const double* __restrict__ gdens,
                                                                 double* __restrict__ gpos) {
  __shared__ int32_t s_tile[kAB / 32][32][33];
  __shared__ double s_v[kAB / 32][96];
  __shared__ int64_t s_j[kAB / 32][32];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  int32_t(*tile)[33] = s_tile[wib];
  const int64_t i0 = blockIdx.x * (int64_t)kAB + (threadIdx.x & ~31), i = i0 + lane;
  if (i0 >= A.n) return;
  const double g = i < A.n ? gdens[i] : 0.0;
  // a particle without an upstream gradient (and a lane past the end) adds
  // nothing and reads none of its neighbours, whatever its position and list hold
  const bool act = g != 0.0;  // (NaN: yes)
  if (!__any_sync(0xffffffffu, act)) return;
  const double C = A.xyzlong / (double)3.141592654f;
  const double4 me = particle<kPacked>(A, act ? i : 0);
  const int64_t jl = act ? A.nei[(size_t)A.nv * i + A.nv - 1] : 0;
  const double4 last = particle<kPacked>(A, jl);
  const double lx = pdelta(me.x, last.x, A.Lx), ly = pdelta(me.y, last.y, A.Ly), lz = pdelta(me.z, last.z, A.Lz);
  const double dlast = sqrt(lx * lx + ly * ly + lz * lz);
  const double r = 0.5 * dlast;
  double S = me.w, T = 0.0;  // T = sum m W'(u) d
  double gi0 = 0, gi1 = 0, gi2 = 0;
  const double r4 = r * r * r * r, w4 = g * C / r4;
  for (int k0 = 0; k0 < A.nv - 1; k0 += 32) {
    stage_lists(A, i0, k0, lane, tile);
    const int m = min(32, A.nv - 1 - k0);
#pragma unroll 1  // unrolled, the divisions' slow paths spill
    for (int k = 0; k < m; ++k) {
      const int64_t j = act ? tile[lane][k] : 0;
      const double4 q = particle<kPacked>(A, j);
      const double dx = pdelta(me.x, q.x, A.Lx), dy = pdelta(me.y, q.y, A.Ly), dz = pdelta(me.z, q.z, A.Lz);
      const double d2 = dx * dx + dy * dy + dz * dz;
      // one rounding each: through a reciprocal root and 1 / r a pair's term is
      // off by up to 8.5 half units in the last place instead of 3, and no faster
      const double d = sqrt(d2);
      const double u = d / r;
      S += q.w * spline(u);
      const double wm = q.w * spline_deriv(u);
      T += wm * d;
      const bool use = act && d2 > 0.0;  // selects the products: 0 times an infinite separation is no zero
      const double a = w4 * wm / d;      // times the separation vector = times e_k
      const double vx = use ? a * dx : 0.0, vy = use ? a * dy : 0.0, vz = use ? a * dz : 0.0;
      gi0 -= vx; gi1 -= vy; gi2 -= vz;
      scatter_add(gpos, j, vx, vy, vz, lane, s_v[wib], s_j[wib]);
    }
  }
  // through r = d_last / 2
  const double drho_dr = C * (-T / (r4 * r) - 3.0 * S / r4);  // d rho / d r = C [-T/r^5 - 3 S/r^4]
  const bool use = act && dlast > 0.0;
  const double a = g * 0.5 * drho_dr / dlast;
  const double vx = use ? a * lx : 0.0, vy = use ? a * ly : 0.0, vz = use ? a * lz : 0.0;
  scatter_add(gpos, jl, vx, vy, vz, lane, s_v[wib], s_j[wib]);
  scatter_add(gpos, i, gi0 - vx, gi1 - vy, gi2 - vz, lane, s_v[wib], s_j[wib]);
}

// dE/dx for every member: one block per item, 256 rows [i0, i0 + 256) of halo
// h against its members [j0, j1); two rows per thread, partner tiles of 256 in
// shared memory.  Positions relative to the member at centre[h] (the densest)
// with the strict min-image rule.  Bound by the FP64 pipe, 17 operations per
// ordered pair; the partners are split so that a few large halos still fill
// the device (500 halos, 217M pairs: backward pass 3.0 -> 0.75 ms).  A row tile
// with one item is added to gpos here, the others leave their sums in part for
// epot_grad_fold_kernel, which adds them in item order.
constexpr int kGT = 256;              // rows per item and partner tile
constexpr int kGB = 128;              // threads per block: two rows each
constexpr int64_t kGItems = 4736;     // items aimed at (four per resident block)
constexpr int kGMinJ = 512;           // partners per item, at least

struct GradItem {
  int32_t h, i0, j0, j1;
  int32_t part;  // slot of the item's sums in part, -1: the tile's only item
};
struct GradTile {
  int32_t h, i0, first, count;  // a row tile's part slots [first, first + count)
};

__global__ void __launch_bounds__(kGB) epot_grad_kernel(const int64_t* __restrict__ off,
                                                       const GradItem* __restrict__ items,
                                                       const double* __restrict__ pos, const double* __restrict__ mass,
                                                       const int32_t* __restrict__ centre, const double* __restrict__ gh,
                                                       double L, int periodic, double G, double* __restrict__ part,
                                                       double* __restrict__ gpos) {
  __shared__ __align__(16) double2 s_xy[kGT], s_zm[kGT];
  const int tid = threadIdx.x;
  const GradItem it = items[blockIdx.x];
  const int64_t base = off[it.h];
  const int32_t n = (int32_t)(off[it.h + 1] - base);
  const int64_t c = base + centre[it.h];
  const double cx = pos[3 * c], cy = pos[3 * c + 1], cz = pos[3 * c + 2];
  auto rel = [&](double v, double cc) {
    double d = v - cc;
    if (periodic) {
      if (d > 0.5 * L) d -= L;
      if (d < -0.5 * L) d += L;
    }
    return d;
  };
  double x[2], y[2], z[2], ax[2] = {0.0, 0.0}, ay[2] = {0.0, 0.0}, az[2] = {0.0, 0.0};
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int32_t i = it.i0 + r * kGB + tid;
    x[r] = y[r] = z[r] = -3.0e30;  // past the end: no use made of the sums
    if (i < n) {
      x[r] = rel(pos[3 * (base + i)], cx);
      y[r] = rel(pos[3 * (base + i) + 1], cy);
      z[r] = rel(pos[3 * (base + i) + 2], cz);
    }
  }
  const bool two = it.i0 + kGB + (tid & ~31) < n;  // uniform per warp: second rows exist
  for (int32_t j0 = it.j0; j0 < it.j1; j0 += kGT) {
    for (int t = tid; t < kGT; t += kGB) {
      const int32_t j = j0 + t;
      double px = 3.0e30, py = 3.0e30, pz = 3.0e30, m = 0.0;  // past the end: no mass, finite distance
      if (j < it.j1) {
        px = rel(pos[3 * (base + j)], cx);
        py = rel(pos[3 * (base + j) + 1], cy);
        pz = rel(pos[3 * (base + j) + 2], cz);
        m = mass[base + j];
      }
      s_xy[t] = make_double2(px, py);
      s_zm[t] = make_double2(pz, m);
    }
    __syncthreads();
    const int jend = min(kGT, it.j1 - j0);
    double tx[2] = {0.0, 0.0}, ty[2] = {0.0, 0.0}, tz[2] = {0.0, 0.0};  // this tile's sums
    auto pair = [&](int r, const double2& a, const double2& b) {
      const double dx = x[r] - a.x, dy = y[r] - a.y, dz = z[r] - b.x;
      const double v = rsqrt3(sep2(dx, dy, dz));
      const double f = b.y * v * (v * v);
      tx[r] += f * dx; ty[r] += f * dy; tz[r] += f * dz;
    };
    if (j0 != it.i0) {
      const int j4 = (jend + 3) & ~3;
      if (two) {
#pragma unroll 4
        for (int jj = 0; jj < j4; ++jj) {
          const double2 a = s_xy[jj], b = s_zm[jj];
          pair(0, a, b);
          pair(1, a, b);
        }
      } else {
#pragma unroll 4
        for (int jj = 0; jj < j4; ++jj) pair(0, s_xy[jj], s_zm[jj]);
      }
    }
    // the member itself (r2 = 0) and coincident members drop out, as in the
    // forward sum: the diagonal tile always, any other tile whose sums a
    // coincident member made NaN, goes pair by pair with the test
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      if (it.i0 + r * kGB + tid < n && (j0 == it.i0 || !(fabs(tx[r]) + fabs(ty[r]) + fabs(tz[r]) <= DBL_MAX))) {
        tx[r] = ty[r] = tz[r] = 0.0;
        for (int jj = 0; jj < jend; ++jj) {
          const double2 a = s_xy[jj], b = s_zm[jj];
          const double dx = x[r] - a.x, dy = y[r] - a.y, dz = z[r] - b.x;
          const double r2 = dx * dx + dy * dy + dz * dz;
          if (r2 > 0.0) {
            const double inv = rsqrt(r2);
            const double f = b.y * (inv * inv * inv);
            tx[r] += f * dx; ty[r] += f * dy; tz[r] += f * dz;
          }
        }
      }
      ax[r] += tx[r]; ay[r] += ty[r]; az[r] += tz[r];
    }
    __syncthreads();
  }
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int32_t i = it.i0 + r * kGB + tid;
    if (i >= n) continue;
    if (it.part >= 0) {
      double* o = part + (size_t)it.part * (3 * kGT) + r * kGB + tid;
      o[0] = ax[r]; o[kGT] = ay[r]; o[2 * kGT] = az[r];
    } else {
      const double s = gh[it.h] * G * mass[base + i];
      gpos[3 * (base + i)] += s * ax[r];
      gpos[3 * (base + i) + 1] += s * ay[r];
      gpos[3 * (base + i) + 2] += s * az[r];
    }
  }
}

__global__ void __launch_bounds__(kGT) epot_grad_fold_kernel(const int64_t* __restrict__ off,
                                                            const GradTile* __restrict__ tiles,
                                                            const double* __restrict__ mass,
                                                            const double* __restrict__ gh, double G,
                                                            const double* __restrict__ part,
                                                            double* __restrict__ gpos) {
  const GradTile t = tiles[blockIdx.x];
  const int64_t base = off[t.h];
  const int64_t i = t.i0 + threadIdx.x;
  if (i >= off[t.h + 1] - base) return;
  double a[3] = {0.0, 0.0, 0.0};
  for (int k = 0; k < t.count; ++k) {
    const double* o = part + (size_t)(t.first + k) * (3 * kGT) + threadIdx.x;
    a[0] += o[0]; a[1] += o[kGT]; a[2] += o[2 * kGT];
  }
  const double s = gh[t.h] * G * mass[base + i];
  for (int d = 0; d < 3; ++d) gpos[3 * (base + i) + d] += s * a[d];
}

// The packed particle rows of a density call: stream-ordered memory of a pool
// of this file (one per device, so calls on several streams and threads do not
// meet), which keeps up to kRowsKeep bytes between calls.
constexpr unsigned long long kRowsKeep = 256ull << 20;
struct RowPools {
  std::mutex m;
  cudaMemPool_t pool[64] = {};
};
static RowPools& row_pools() {
  static RowPools* p = new RowPools();
  return *p;
}

// The pool's calls wait for no stream, but count as unsafe beside a capture on
// another thread, and would end it: they are made in the relaxed mode.
struct RelaxedCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

struct Packed {
  void* p = nullptr;
  cudaStream_t st = nullptr;
  // sets A.p4 for large n, unless the stream is being captured (a graph would
  // own the memory)
  int make(AdjArgs& A, cudaStream_t s) {
    if (A.n < kPackMin) return AHOP_OK;
    RelaxedCapture relaxed;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    AHOP_CUDA_TRY(cudaStreamIsCapturing(s, &cs));
    if (cs != cudaStreamCaptureStatusNone) return AHOP_OK;
    int dev = 0;
    AHOP_CUDA_TRY(cudaGetDevice(&dev));
    if (dev >= 64) return AHOP_OK;
    RowPools& R = row_pools();
    cudaMemPool_t pool;
    {
      std::lock_guard<std::mutex> g(R.m);
      if (!R.pool[dev]) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t np = nullptr;
        AHOP_CUDA_TRY(cudaMemPoolCreate(&np, &props));
        unsigned long long keep = kRowsKeep;
        AHOP_CUDA_TRY(cudaMemPoolSetAttribute(np, cudaMemPoolAttrReleaseThreshold, &keep));
        R.pool[dev] = np;
      }
      pool = R.pool[dev];
    }
    if (cudaMallocFromPoolAsync(&p, (size_t)A.n * 32, pool, s) != cudaSuccess) {
      cudaGetLastError();  // no room: the kernels read the caller's arrays
      p = nullptr;
      return AHOP_OK;
    }
    st = s;
    pack_kernel<<<(unsigned)((A.n + 255) / 256), 256, 0, s>>>(A.pos, A.mass, A.n, static_cast<double4*>(p));
    AHOP_CUDA_TRY(cudaGetLastError());
    A.p4 = static_cast<const double4*>(p);
    return AHOP_OK;
  }
  int done() {
    if (!p) return AHOP_OK;
    RelaxedCapture relaxed;
    void* q = p;
    p = nullptr;
    AHOP_CUDA_TRY(cudaFreeAsync(q, st));
    return AHOP_OK;
  }
  ~Packed() { done(); }
};

// Items, tiles and partial sums of ahop_epot_grad, kept between calls.  A call
// takes an idle set of its device, or a new one while others are in use on
// other threads or streams, and gives it back when its kernels are done; up to
// kGradKeep bytes of idle sets stay.
constexpr size_t kGradKeep = (size_t)256 << 20;
struct GradWork {
  int device = -1;
  DevBuf items, tiles, part;
  GradWork* next = nullptr;
  size_t bytes() const { return items.bytes + tiles.bytes + part.bytes; }
  void release() { items.release(); tiles.release(); part.release(); }
};
struct GradPool {
  std::mutex m;
  GradWork* idle = nullptr;
  size_t bytes = 0;  // of the idle sets
};
static GradPool& grad_pool() {
  static GradPool* p = new GradPool();
  return *p;
}

struct GradLease {
  GradWork* w = nullptr;
  cudaStream_t st = nullptr;
  bool done = false;  // the kernels that use the set have ended
  bool take(int device, cudaStream_t s) {
    st = s;
    GradPool& P = grad_pool();
    std::lock_guard<std::mutex> g(P.m);
    for (GradWork** at = &P.idle; *at; at = &(*at)->next)
      if ((*at)->device == device) {
        w = *at;
        *at = w->next;
        P.bytes -= w->bytes();
        return true;
      }
    w = new (std::nothrow) GradWork();
    if (w) w->device = device;
    return w != nullptr;
  }
  ~GradLease() {
    if (!w) return;
    if (!done) cudaStreamSynchronize(st);
    GradPool& P = grad_pool();
    {
      std::lock_guard<std::mutex> g(P.m);
      if (P.bytes + w->bytes() <= kGradKeep) {
        P.bytes += w->bytes();
        w->next = P.idle;
        P.idle = w;
        return;
      }
    }
    w->release();
    delete w;
  }
};

void release_adjoint_memory() {
  {
    RowPools& R = row_pools();
    std::lock_guard<std::mutex> g(R.m);
    for (cudaMemPool_t p : R.pool)
      if (p) cudaMemPoolTrimTo(p, 0);
  }
  GradPool& P = grad_pool();
  std::lock_guard<std::mutex> g(P.m);
  int now = 0;
  cudaGetDevice(&now);
  while (GradWork* w = P.idle) {
    P.idle = w->next;
    cudaSetDevice(w->device);
    w->release();
    delete w;
  }
  P.bytes = 0;
  cudaSetDevice(now);
}

}  // namespace ahop

using namespace ahop;

extern "C" {

int ahop_density_fixed(const AhopAdjParams* p, const double* d_pos, const double* d_mass, const int32_t* d_nei,
                       int64_t n, double* d_dens, void* stream) {
  if (!p || p->nvoisins < 2 || n <= 0) { set_error("bad density_fixed arguments"); return AHOP_EINVAL; }
  AdjArgs A{d_pos, d_mass, nullptr, d_nei, n, p->nvoisins, p->xlong, p->ylong, p->zlong, p->xlong * p->ylong * p->zlong};
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  Packed rows;
  int rc;
  if ((rc = rows.make(A, st))) return rc;
  const unsigned grid = (unsigned)((n + kAB - 1) / kAB);
  if (A.p4) density_fixed_kernel<true><<<grid, kAB, 0, st>>>(A, d_dens);
  else density_fixed_kernel<false><<<grid, kAB, 0, st>>>(A, d_dens);
  AHOP_CUDA_TRY(cudaGetLastError());
  return rows.done();
}

int ahop_density_adjoint(const AhopAdjParams* p, const double* d_pos, const double* d_mass, const int32_t* d_nei,
                         int64_t n, const double* d_gdens, double* d_gpos, void* stream) {
  if (!p || p->nvoisins < 2 || n <= 0) { set_error("bad density_adjoint arguments"); return AHOP_EINVAL; }
  AdjArgs A{d_pos, d_mass, nullptr, d_nei, n, p->nvoisins, p->xlong, p->ylong, p->zlong, p->xlong * p->ylong * p->zlong};
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  Packed rows;
  int rc;
  if ((rc = rows.make(A, st))) return rc;
  const unsigned grid = (unsigned)((n + kAB - 1) / kAB);
  if (A.p4) density_adjoint_kernel<true><<<grid, kAB, 0, st>>>(A, d_gdens, d_gpos);
  else density_adjoint_kernel<false><<<grid, kAB, 0, st>>>(A, d_gdens, d_gpos);
  AHOP_CUDA_TRY(cudaGetLastError());
  return rows.done();
}

int ahop_epot_grad(const AhopHaloParams* p, const int64_t* d_off, const int64_t* h_off, int64_t nhalo,
                   const double* d_pos, const double* d_mass, const int32_t* d_centre, const double* d_gh,
                   double* d_gpos, void* stream) {
  if (!p || nhalo < 0 || !h_off) { set_error("bad epot_grad arguments"); return AHOP_EINVAL; }
  double pairs = 0.0;  // ordered
  for (int64_t h = 0; h < nhalo; ++h) {
    const double n = (double)(h_off[h + 1] - h_off[h]);
    pairs += n * n;
  }
  const int64_t fit = (int64_t)(pairs / ((double)kGItems * kGT));
  const int64_t chunk = std::max<int64_t>(kGMinJ, (fit + kGT - 1) / kGT * kGT);
  std::vector<GradItem> items;
  std::vector<GradTile> tiles;
  int32_t parts = 0;
  for (int64_t h = 0; h < nhalo; ++h) {
    const int64_t n = h_off[h + 1] - h_off[h];
    const int32_t per = (int32_t)((n + chunk - 1) / chunk);
    for (int64_t i0 = 0; i0 < n; i0 += kGT) {
      if (per > 1) tiles.push_back(GradTile{(int32_t)h, (int32_t)i0, parts, per});
      for (int64_t j0 = 0; j0 < n; j0 += chunk)
        items.push_back(GradItem{(int32_t)h, (int32_t)i0, (int32_t)j0, (int32_t)std::min(n, j0 + chunk),
                                 per > 1 ? parts++ : -1});
    }
  }
  if (items.empty()) return AHOP_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int dev = 0;
  AHOP_CUDA_TRY(cudaGetDevice(&dev));
  GradLease lease;
  if (!lease.take(dev, st)) { set_error("out of memory"); return AHOP_ENOMEM; }
  GradWork& W = *lease.w;
  AHOP_CUDA_TRY(W.items.ensure(items.size() * sizeof(GradItem)));
  AHOP_CUDA_TRY(W.tiles.ensure(tiles.size() * sizeof(GradTile)));
  AHOP_CUDA_TRY(W.part.ensure((size_t)parts * (3 * kGT) * 8));
  AHOP_CUDA_TRY(cudaMemcpyAsync(W.items.p, items.data(), items.size() * sizeof(GradItem), cudaMemcpyHostToDevice, st));
  if (!tiles.empty())
    AHOP_CUDA_TRY(cudaMemcpyAsync(W.tiles.p, tiles.data(), tiles.size() * sizeof(GradTile), cudaMemcpyHostToDevice, st));
  epot_grad_kernel<<<(unsigned)items.size(), kGB, 0, st>>>(d_off, W.items.as<GradItem>(), d_pos, d_mass, d_centre,
                                                           d_gh, p->Lbox, p->periodic, p->gravconst,
                                                           W.part.as<double>(), d_gpos);
  AHOP_CUDA_TRY(cudaGetLastError());
  if (!tiles.empty()) {
    epot_grad_fold_kernel<<<(unsigned)tiles.size(), kGT, 0, st>>>(d_off, W.tiles.as<GradTile>(), d_mass, d_gh,
                                                                  p->gravconst, W.part.as<double>(), d_gpos);
    AHOP_CUDA_TRY(cudaGetLastError());
  }
  AHOP_CUDA_TRY(cudaStreamSynchronize(st));
  lease.done = true;
  return AHOP_OK;
}

}  // extern "C"
