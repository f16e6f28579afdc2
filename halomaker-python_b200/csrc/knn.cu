// Morton-bucketed tree build and periodic kNN with the SPH cubic-spline
// density: one query per lane (a warp per query leaf), one warp per query for
// small sets.
//
// Replaces create_tree_structure/create_KDtree (f90:2967-3221),
// omp_find_nearest_parts/walk_tree2 (f90:2841-2962) and omp_compute_density
// (f90:2816-2838) of the reference.
//
// Layout: particles are radix-sorted by a 63-bit Morton key; leaf j holds the
// 32 consecutive sorted particles [32j, 32j+32); each internal level groups 32
// consecutive nodes of the level below.  Every node stores its padded
// axis-aligned box as centre + half-width (6 doubles).  The kNN result of a
// query is the set of its nvoisins nearest particles under the reference's
// periodic distance, ordered by (distance, particle index); distances and the
// density use the reference's exact expression order in explicitly rounded
// FP64 (no FMA), so the density matches the reference bit for bit whenever the
// neighbour order does.
#include <algorithm>
#include <cub/cub.cuh>
#include <cfloat>
#include <climits>
#include <cstring>
#include <math_constants.h>

#include "engine.h"
#include "exact.cuh"

namespace ahop {

// ---------------------------------------------------------------- Morton keys
__device__ __forceinline__ unsigned long long spread21(unsigned int v) {
  unsigned long long x = v & 0x1fffffULL;
  x = (x | (x << 32)) & 0x1f00000000ffffULL;
  x = (x | (x << 16)) & 0x1f0000ff0000ffULL;
  x = (x | (x << 8)) & 0x100f00f00f00f00fULL;
  x = (x | (x << 4)) & 0x10c30c30c30c30c3ULL;
  x = (x | (x << 2)) & 0x1249249249249249ULL;
  return x;
}

__device__ __forceinline__ unsigned int quant21(double v, double half, double L) {
  double u = (v + half) / L;  // [0,1) for v in [-L/2, L/2)
  double q = u * 2097152.0;
  if (!(q >= 0.0)) q = 0.0;
  if (q > 2097151.0) q = 2097151.0;
  return (unsigned int)q;
}

__global__ void morton_kernel(const double* __restrict__ pos, int64_t n, double Lx, double Ly, double Lz,
                              unsigned long long* __restrict__ key, int32_t* __restrict__ idx) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  double x = pos[3 * i + 0], y = pos[3 * i + 1], z = pos[3 * i + 2];
  unsigned int qx = quant21(x, 0.5 * Lx, Lx), qy = quant21(y, 0.5 * Ly, Ly), qz = quant21(z, 0.5 * Lz, Lz);
  key[i] = (spread21(qx) << 2) | (spread21(qy) << 1) | spread21(qz);
  idx[i] = (int32_t)i;
}

__global__ void gather_sorted_kernel(const double* __restrict__ pos, const double* __restrict__ mass,
                                     const int32_t* __restrict__ orig, int64_t n, double* __restrict__ x,
                                     double* __restrict__ y, double* __restrict__ z, double* __restrict__ m,
                                     double4* __restrict__ p4, int32_t* __restrict__ rank) {
  int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (s >= n) return;
  int32_t o = orig[s];
  const double px = pos[3 * (int64_t)o + 0], py = pos[3 * (int64_t)o + 1], pz = pos[3 * (int64_t)o + 2];
  const double pm = mass[o];
  x[s] = px;
  y[s] = py;
  z[s] = pz;
  m[s] = pm;
  p4[s] = make_double4(px, py, pz, pm);
  rank[o] = (int32_t)s;
}

// Box storage: 6 doubles per node: cx, cy, cz, wx, wy, wz (centre, padded half-width).
__device__ __forceinline__ void warp_minmax(double& lo, double& hi) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
}

// Leaf boxes: one warp per leaf.
__global__ void leaf_box_kernel(const double* __restrict__ x, const double* __restrict__ y,
                                const double* __restrict__ z, int64_t n, int64_t nleaf, double pad,
                                double* __restrict__ box) {
  int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  int lane = threadIdx.x & 31;
  if (w >= nleaf) return;
  int64_t p = w * kLeaf + lane;
  bool v = p < n;
  double lx = v ? x[p] : DBL_MAX, hx = v ? x[p] : -DBL_MAX;
  double ly = v ? y[p] : DBL_MAX, hy = v ? y[p] : -DBL_MAX;
  double lz = v ? z[p] : DBL_MAX, hz = v ? z[p] : -DBL_MAX;
  warp_minmax(lx, hx);
  warp_minmax(ly, hy);
  warp_minmax(lz, hz);
  if (lane == 0) {
    double* b = box + 6 * w;
    b[0] = 0.5 * (lx + hx); b[1] = 0.5 * (ly + hy); b[2] = 0.5 * (lz + hz);
    b[3] = 0.5 * (hx - lx) + pad; b[4] = 0.5 * (hy - ly) + pad; b[5] = 0.5 * (hz - lz) + pad;
  }
}

// Internal boxes: one warp per node over its (<= 32) child boxes.
__global__ void node_box_kernel(const double* __restrict__ child, int64_t nchild, int64_t nnode,
                                double* __restrict__ box) {
  int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  int lane = threadIdx.x & 31;
  if (w >= nnode) return;
  int64_t c = w * kFan + lane;
  bool v = c < nchild;
  double lo[3], hi[3];
  for (int k = 0; k < 3; ++k) {
    lo[k] = v ? child[6 * c + k] - child[6 * c + 3 + k] : DBL_MAX;
    hi[k] = v ? child[6 * c + k] + child[6 * c + 3 + k] : -DBL_MAX;
    warp_minmax(lo[k], hi[k]);
  }
  if (lane == 0) {
    double* b = box + 6 * w;
    for (int k = 0; k < 3; ++k) {
      b[k] = 0.5 * (lo[k] + hi[k]);
      b[3 + k] = 0.5 * (hi[k] - lo[k]) * (1.0 + 1e-12) + 1e-300;
    }
  }
}

int stage_sort_and_tree(Engine& E, const double* d_pos, const double* d_mass) {
  const int64_t n = E.n;
  const Params& P = E.prm;
  cudaStream_t st = E.stream;
  AHOP_CUDA_TRY(E.layout_sort());
  AHOP_CUDA_TRY(E.d_x.ensure(n * 8));
  AHOP_CUDA_TRY(E.d_y.ensure(n * 8));
  AHOP_CUDA_TRY(E.d_z.ensure(n * 8));
  AHOP_CUDA_TRY(E.d_m.ensure(n * 8));
  AHOP_CUDA_TRY(E.d_orig.ensure(n * 4));
  AHOP_CUDA_TRY(E.d_rank.ensure(n * 4));
  const int T = 256;
  unsigned grid = (unsigned)((n + T - 1) / T);
  E.launches++;
  morton_kernel<<<grid, T, 0, st>>>(d_pos, n, P.xlong, P.ylong, P.zlong, E.d_key.as<unsigned long long>(),
                                    E.d_idx.as<int32_t>());
  AHOP_CUDA_TRY(cudaGetLastError());
  // All 63 key bits: the low ones order the leaves of clumps far smaller than
  // the mean spacing (a clump 1e-5 of the box across, 200,000 particles: kNN
  // 144.8 ms with the bits below 2^-8 of the mean spacing left out, 1.2 with
  // all of them, for two radix passes of eight)
  size_t tmp = 0;
  cub::DeviceRadixSort::SortPairs(nullptr, tmp, E.d_key.as<unsigned long long>(),
                                  E.d_key2.as<unsigned long long>(), E.d_idx.as<int32_t>(),
                                  E.d_orig.as<int32_t>(), (int)n, 0, 63, st);
  AHOP_CUDA_TRY(E.d_cub.ensure(tmp));
  E.cub_calls++;
  AHOP_CUDA_TRY(cub::DeviceRadixSort::SortPairs(E.d_cub.p, tmp, E.d_key.as<unsigned long long>(),
                                                E.d_key2.as<unsigned long long>(), E.d_idx.as<int32_t>(),
                                                E.d_orig.as<int32_t>(), (int)n, 0, 63, st));
  E.launches++;
  if (E.mass_pending) {  // host path: the masses were uploaded on the copy stream
    AHOP_CUDA_TRY(cudaStreamWaitEvent(st, E.ev_mass, 0));
    E.mass_pending = false;
  }
  // the keys and the permutation's first copy give way to the rows
  gather_sorted_kernel<<<grid, T, 0, st>>>(d_pos, d_mass, E.d_orig.as<int32_t>(), n, E.d_x.as<double>(),
                                           E.d_y.as<double>(), E.d_z.as<double>(), E.d_m.as<double>(), E.rows(),
                                           E.d_rank.as<int32_t>());
  AHOP_CUDA_TRY(cudaGetLastError());
  // levels
  int64_t cnt = (n + kLeaf - 1) / kLeaf;
  int nlev = 0;
  int64_t off = 0;
  for (;;) {
    if (nlev >= kMaxLevels) { set_error("too many tree levels"); return AHOP_EINVAL; }
    E.lev_off[nlev] = off;
    E.lev_cnt[nlev] = cnt;
    off += cnt;
    nlev++;
    if (cnt == 1) break;
    cnt = (cnt + kFan - 1) / kFan;
  }
  E.lev_off[nlev] = off;
  E.nlev = nlev;
  AHOP_CUDA_TRY(E.d_box.ensure(off * 6 * 8));
  double* box = E.d_box.as<double>();
  double pad = 1e-12 * fmax(P.xlong, fmax(P.ylong, P.zlong));
  {
    int64_t threads = E.lev_cnt[0] * 32;
    E.launches++;
    leaf_box_kernel<<<(unsigned)((threads + T - 1) / T), T, 0, st>>>(E.d_x.as<double>(), E.d_y.as<double>(),
                                                                     E.d_z.as<double>(), n, E.lev_cnt[0], pad,
                                                                     box);
    AHOP_CUDA_TRY(cudaGetLastError());
  }
  for (int l = 1; l < nlev; ++l) {
    int64_t threads = E.lev_cnt[l] * 32;
    E.launches++;
    node_box_kernel<<<(unsigned)((threads + T - 1) / T), T, 0, st>>>(
        box + 6 * E.lev_off[l - 1], E.lev_cnt[l - 1], E.lev_cnt[l], box + 6 * E.lev_off[l]);
    AHOP_CUDA_TRY(cudaGetLastError());
  }
  return AHOP_OK;
}

// ------------------------------------------------------------------ kNN kernel
struct KnnArgs {
  const double4* p4;   // x, y, z, m per sorted slot
  const double* m;
  const int32_t* orig;
  const double* box;
  int64_t lev_off[kMaxLevels];
  int64_t lev_cnt[kMaxLevels];
  int nlev;
  int64_t n;
  int32_t n32;  // n as int32 (n < 2^31 is checked at the boundary)
  double Lx, Ly, Lz, xyzlong;
  int nv;       // nvoisins (<= 32)
  int nstore;   // neighbours written per particle
  int32_t* nei; // [n][nstore] sorted-slot ids
  double* dens; // [n]
  float eabs2;  // absolute margin of FP32 distances (twice 2^-46 of the largest box length)
  float gpad;   // padding of a box of queries rounded to float
  float near;   // 0.49 of the smallest box length
  int obase;    // float exponent of the lowest octave bin: the 31 octaves up to 4 (largest box length)^2
  int* err;     // error flag (stack overflow)
  int* next;    // next query leaf of the chunk to take
  int leaf0, nchunk;  // query leaves [leaf0, leaf0 + nchunk) of this pair of launches
  int32_t* coll;      // [nchunk][kCollect][32] collected slots of each query; the bound's bits for count 0
  uint8_t* ccnt;      // [nchunk][32] collected particles (0: per-query search)
  int32_t* lost;      // queries of the chunk left to the per-query search, and their number
  int* nlost;
  unsigned long long* kstats;   // profiled instances: counters (ahop_debug_tree_stats)
  const float4* box32;          // boxes of every level in FP32, widened (leaf_box32_kernel)
};

constexpr int kStack = 256;  // traversal stack entries per warp

__device__ __forceinline__ double box_dist2(const double* __restrict__ b, double qx, double qy, double qz,
                                            double Lx, double Ly, double Lz) {
  double dx = fabs(b[0] - qx); dx = fmin(dx, Lx - dx); dx = fmax(0.0, dx - b[3]);
  double dy = fabs(b[1] - qy); dy = fmin(dy, Ly - dy); dy = fmax(0.0, dy - b[4]);
  double dz = fabs(b[2] - qz); dz = fmin(dz, Lz - dz); dz = fmax(0.0, dz - b[5]);
  return dx * dx + dy * dy + dz * dz;
}

// The warp's running neighbour list of the per-query search: lane i holds the
// i-th nearest (ld, ls): squared distance, sorted slot; empty slots hold +inf.
struct WarpList {
  double ld;
  int32_t ls;
  double r2;   // acceptance bound: the smaller of the nv-th entry and cap
  double cap;  // an upper bound of the query's final nv-th distance known in advance (+inf: none)
};

// Insert the particles of one leaf that belong in the list.  Candidates at
// exactly the nv-th distance are taken in too: an exact distance tie is
// settled by particle index, so one that does not precede the last entry
// lands at position nv and drops out.  Particle indices are only read for
// such ties.
template <int C>
__device__ __forceinline__ void leaf_insert(const KnnArgs& A, WarpList& L, int32_t leaf, int64_t self, double qx,
                                            double qy, double qz, int lane) {
  const int nvv = C ? C : A.nv;
  const int32_t p = leaf * kLeaf + lane;
  const bool v = (p < A.n32) && (p != (int32_t)self);
  double d = CUDART_INF;
  if (v) {
    const double4 c = A.p4[p];
    d = pdist2(qx, qy, qz, c.x, c.y, c.z, A.Lx, A.Ly, A.Lz);
  }
  unsigned mask = __ballot_sync(0xffffffffu, v && d <= L.r2);
  if (!mask) return;
  const double last = __shfl_sync(0xffffffffu, L.ld, nvv - 1);
  const bool even = v && d == last && d < CUDART_INF;
  if (__any_sync(0xffffffffu, even)) {
    // ties with the last entry: only those before it by particle index go in
    // (a clump of many coincident particles is all ties)
    const int32_t lo = A.orig[__shfl_sync(0xffffffffu, L.ls, nvv - 1)];
    mask &= ~__ballot_sync(0xffffffffu, even && A.orig[p] > lo);
  }
  while (mask) {
    const int src = __ffs(mask) - 1;
    const double cd = __shfl_sync(0xffffffffu, d, src);
    const int32_t cs = leaf * kLeaf + src;
    bool prec = (lane < nvv) && (L.ld < cd);
    const bool tie = (lane < nvv) && (L.ld == cd);
    if (__any_sync(0xffffffffu, tie)) {
      const int32_t co = A.orig[cs];
      if (tie) prec = A.orig[L.ls] < co;
    }
    const int pos = __popc(__ballot_sync(0xffffffffu, prec));
    const double ud = __shfl_up_sync(0xffffffffu, L.ld, 1);
    const int32_t us = __shfl_up_sync(0xffffffffu, L.ls, 1);
    if (lane > pos) { L.ld = ud; L.ls = us; }
    if (lane == pos) { L.ld = cd; L.ls = cs; }
    if (lane >= nvv) { L.ld = CUDART_INF; L.ls = -1; }
    // the bound is refreshed once per leaf: a candidate that an earlier one
    // of this leaf pushed beyond the list finds every entry ahead of it
    // (pos = nv) and changes nothing
    mask &= ~(1u << src);
  }
  L.r2 = fmin(__shfl_sync(0xffffffffu, L.ld, nvv - 1), L.cap);
}

// Per-query depth-first traversal from the root, nearest child first (queries
// that the lane-per-query path hands over).  A box at exactly the bound is
// entered: the boxes are padded, so that happens only at distance 0, where
// coincident particles beyond the nv-th are settled by particle index.
template <int C>
__device__ void query_dfs(const KnnArgs& A, WarpList& L, int64_t s, double qx, double qy, double qz, int lane,
                          int32_t* s_node, double* s_bd) {
  const int top = A.nlev - 1;
  int sp = 0;
  if (lane == 0) { s_node[0] = (top << 27) | 0; s_bd[0] = 0.0; }
  sp = 1;
  __syncwarp();
  while (sp > 0) {
    --sp;
    const int32_t ent = s_node[sp];
    const double bd = s_bd[sp];
    __syncwarp();
    if (!(bd <= L.r2)) continue;
    const int lvl = ent >> 27;
    const int64_t j = ent & ((1 << 27) - 1);
    if (lvl == 0) {
      leaf_insert<C>(A, L, j, s, qx, qy, qz, lane);
      continue;
    }
    const int64_t c = j * kFan + lane;
    const bool valid = c < A.lev_cnt[lvl - 1];
    double bdc = CUDART_INF;
    if (valid) bdc = box_dist2(A.box + 6 * (A.lev_off[lvl - 1] + c), qx, qy, qz, A.Lx, A.Ly, A.Lz);
    const bool cand = valid && bdc <= L.r2;
    const unsigned mask = __ballot_sync(0xffffffffu, cand);
    if (!mask) continue;
    const int cnt = __popc(mask);
    if (sp + cnt > kStack) {  // cannot happen for <= 7 levels; guard anyway
      if (lane == 0) atomicExch(A.err, 1);
      break;
    }
    double best = cand ? bdc : CUDART_INF;
    int bl = lane;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      double ob = __shfl_xor_sync(0xffffffffu, best, o);
      int ol = __shfl_xor_sync(0xffffffffu, bl, o);
      if (ob < best || (ob == best && ol < bl)) { best = ob; bl = ol; }
    }
    if (cand) {
      // the nearest on top, the others below it in Morton order
      int r = __popc(mask & ((1u << lane) - 1));
      int slot;
      if (lane == bl) slot = sp + cnt - 1;
      else {
        int rb = __popc(mask & ((1u << bl) - 1));
        slot = sp + cnt - 2 - (r < rb ? r : r - 1);
      }
      s_node[slot] = ((lvl - 1) << 27) | (int32_t)c;
      s_bd[slot] = bdc;
    }
    sp += cnt;
    __syncwarp();
  }
}

// SPH density (f90:2816-2838) in the exact evaluation order, and the stored
// neighbour slots.  The nv - 1 terms are summed in list order by lane 0 from
// the warp's scratch st (32 doubles of shared memory), not with a shuffle per
// term.
template <int C>
__device__ __forceinline__ void finish_query(const KnnArgs& A, const WarpList& L, int64_t s, int lane, double* st) {
  const int nv = C ? C : A.nv;
  const double dlast = __shfl_sync(0xffffffffu, L.ld, nv - 1);
  const double r = xmul(xsqrt(dlast), 0.5);
  const double r3 = xmul(xmul(r, r), r);
  const double unsr = xdiv(1.0, r);
  double term = 0.0;
  if (lane < nv - 1) term = xmul(A.m[L.ls], spline(xmul(xsqrt(L.ld), unsr)));
  st[lane] = term;
  __syncwarp();
  if (lane == 0) {
    double contrib = 0.0;
    for (int i = 0; i < nv - 1; ++i) contrib = xadd(contrib, st[i]);
    const double pi_f = (double)3.141592654f;  // f90:58 single-precision literal
    A.dens[s] = xdiv(xmul(A.xyzlong, xadd(contrib, A.m[s])), xmul(pi_f, r3));
  }
  if (lane < A.nstore) A.nei[s * A.nstore + lane] = L.ls;
  __syncwarp();  // st is the fallback search stack of the next query
}

// Boxes in FP32 for the candidate tests: centre rounded to
// float, half width widened to cover that rounding plus every rounding of the
// FP32 test below (2^-21 L), so the FP32 distance is never above the exact
// point-to-box distance: a pruning bound, looser by a negligible margin.
// The centre's w: twice what the node's pairs can be apart beyond a box length
// on some axis (the boxes' padding, for one); the reference's distance is 0
// there, which only the per-query search takes, so beyond 1e-9 of the box it
// is +inf (a particle outside the box, and the leaves across the box from it),
// as where FP32 coordinates are too coarse (particles outside [-L, L]) or squares
// leave the range of floats (inbox = 0: L above 1e15, or below 1e-8, where the
// 2^-149 of a subnormal square, 6e-23 as a distance, exceeds eabs2 = 2^-45 L).
__global__ void leaf_box32_kernel(const double* __restrict__ box, int64_t nbox, double Lx, double Ly, double Lz,
                                  int inbox, float4* __restrict__ out) {
  const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (j >= nbox) return;
  const double* b = box + 6 * j;
  const double* root = box + 6 * (nbox - 1);
  const double L[3] = {Lx, Ly, Lz};
  const double pad = fmax(Lx, fmax(Ly, Lz)) * 0x1p-21;
  float c[3], w[3];
  double over = 0.0;
  bool in = inbox;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    c[k] = (float)b[k];
    w[k] = __double2float_ru(b[3 + k] + fabs(b[k] - (double)c[k]) + pad);
    in = in && fabs(root[k]) + root[3 + k] <= 1.001 * L[k];  // (the pad aside)
    over = fmax(over, fabs(b[k] - root[k]) + b[3 + k] + root[3 + k] - L[k]);
  }
  in = in && over <= 1e-9 * fmin(Lx, fmin(Ly, Lz));
  out[2 * j] = make_float4(c[0], c[1], c[2], in ? __double2float_ru(2.0 * over) : CUDART_INF_F);
  out[2 * j + 1] = make_float4(w[0], w[1], w[2], 0.f);
}

// ---- one query per lane -------------------------------------------------------
// Bound by instruction issue: 1,620 warp instructions per query (8M-particle
// clustered box; one warp per query with a list in registers took 3,751, most
// of them in visiting each query's own leaves and inserting one by one), 16.7M
// particles in 35.9 ms against 87.3, 2M in 4.65 against 13.1.
// The main path works on a query leaf's 32 particles at once, lane = query, so
// every per-query step costs 1/32 of a warp instruction per query and the
// particles of a candidate leaf are read from shared memory by all 32 queries.
// Distances in the two scans are FP32, relative to the query leaf's centre;
// they only select: a scan's bound is widened by the FP32 error, and what is
// within it is ranked by the exact FP64 (distance, particle index) afterwards.
constexpr int kKnnWarps = 4;       // warps per block
constexpr int kKnnBlocks = 6;      // collect: blocks per SM (80 registers, 8.5 KB of shared memory per warp)
constexpr int kFinWarps = 4;       // finish: warps per block
constexpr int kFinBlocks = 5;      // finish: blocks per SM
constexpr int kLostBlocks = 16;    // blocks per SM for the queries left over: usually few, at times whole chunks
constexpr int kBatch = 256;        // candidate leaves sorted and counted at a time
constexpr int kVisMax = 160;       // counted leaves per query leaf, three times the mean; beyond, a warp for each
                                   // of the 32 queries is as cheap and ends sooner (262,144 particles, three
                                   // boxes: 0.95-1.11 ms at 160, 0.94-1.24 at 352; 2M and 16.7M: the same)
// Nodes opened and candidate leaves listed per query leaf, far above the means
// (about 40 and 125): a leaf strung over distant clumps would otherwise keep
// one warp long after the others are done (three boxes each, without the limits
// and with: 262,144 particles 1.13-1.40 ms, 0.95-1.11; 2M 5.2-6.1, 4.65; 16.7M
// 41-51, 35.9).
constexpr int kNodeMax = 256, kCandMax = 768;
// Up to here every query gets a warp of its own: a set of fewer query leaves
// than resident warps (3,552) takes as long as its slowest leaf.  Measured
// (ms, per query | per lane, means of three boxes): 20,000 particles 0.20 |
// 0.50, 70,001 0.56 | 0.62, 98,304 0.76 | 0.76, 131,072 1.02 | 0.85, 262,144
// 2.01 | 1.05.
constexpr int kPerQueryMax = 98304;
constexpr int kTravStack = 192;    // traversal stack: at most 31 nodes waiting per level and 32 at the last
constexpr int kTile = 64;          // particles staged: up to 31 left over and one leaf
constexpr int kBins = 32;          // distance bins per query: 8 per octave of d^2, four octaves
constexpr int kBinShift = 20;      // float bits per bin
constexpr int kCollect = 48;       // particles collected per query (beyond: per-query search)
constexpr int kWindows = 6;        // times the bins of a query are laid lower or cut finer
constexpr int kChunkLeaves = 1 << 18;  // query leaves per pair of launches (1.6 GB of collected slots)
static_assert((kBatch & (kBatch - 1)) == 0, "the candidate sort pads to a power of two");
// leaves (level 0) are listed and the root (at most level kMaxLevels - 1) is popped alone
static_assert((kMaxLevels - 3) * (kFan - 1) + kFan <= kTravStack, "the traversal's nodes fit the stack");

// Shared memory of a warp of the collect kernel, 8.5 KB:
//   bins  [bin][lane]                        A to C
//   key   a batch of candidates, sorted      B, C; with cand: the three leaves of step A
//   cand  a batch of candidates, unsorted    B; then the boxes of a chunk of leaves, C and D
//   stack the traversal                      B, C
//   tile  staged particles x, y, z, slot     C, D
//   group four boxes of eight queries          B
//   vis   the counted leaves                 C, D
constexpr int kOffBins = 0;
constexpr int kOffKey = kBins * 32 * 4, kOffSeed = kOffKey;
constexpr int kOffCand = kOffKey + kBatch * 4, kOffBox = kOffCand;
constexpr int kOffStack = kOffCand + kBatch * 4;
constexpr int kOffTile = kOffStack + kTravStack * 4;
constexpr int kOffGroup = kOffTile + 4 * kTile * 4;
constexpr int kOffVis = kOffGroup + 4 * sizeof(float4) * 2;
constexpr int kWarpBytes = kOffVis + kVisMax * 4;
static_assert(kOffBox + 64 * 16 <= kOffStack, "a chunk's boxes end before the stack");
static_assert(kOffSeed + 3 * 96 * 4 <= kOffStack, "the leaves of step A end before the stack");
static_assert(kWarpBytes % 16 == 0 && kOffTile % 16 == 0 && kOffGroup % 16 == 0, "16-byte loads");
static_assert(kCollect < 63 && kCollect > 33, "entry numbers take 6 bits; room for nv + 1");

__device__ __forceinline__ unsigned long long pack2(float v) {
  const unsigned u = __float_as_uint(v);
  return ((unsigned long long)u << 32) | u;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// The reference's periodic squared distance (pdist2): |a - b| <= L/2 is its
// own minimum with L - |a - b| (also rounded), beyond that L - |a - b| is.
__device__ __forceinline__ double pdist_sel(double a, double b, double L, double h) {
  double d = fabs(xsub(a, b));
  if (d > h) d = fmax(0.0, xsub(L, d));
  return d;
}

struct Query {
  double x, y, z;                      // exact position
  unsigned long long nx, ny, nz;       // minus the position relative to the leaf's centre, twice (f32x2)
  float fx, fy, fz;                    // position rounded to float, for the box tests
};

__device__ __forceinline__ double exact_dist2(const KnnArgs& A, const Query& q, const double4& p) {
  const double dx = pdist_sel(q.x, p.x, A.Lx, 0.5 * A.Lx), dy = pdist_sel(q.y, p.y, A.Ly, 0.5 * A.Ly),
               dz = pdist_sel(q.z, p.z, A.Lz, 0.5 * A.Lz);
  return xadd(xadd(xmul(dx, dx), xmul(dy, dy)), xmul(dz, dz));
}

// Lower bound of the squared distance from this lane's query to a widened box.
__device__ __forceinline__ float query_box_lb(const Query& q, const float4& c, const float4& w, float Lx, float Ly,
                                              float Lz) {
  float dx = fabsf(c.x - q.fx); dx = fminf(dx, Lx - dx); dx = fmaxf(0.f, __fsub_rd(dx, w.x));
  float dy = fabsf(c.y - q.fy); dy = fminf(dy, Ly - dy); dy = fmaxf(0.f, __fsub_rd(dy, w.y));
  float dz = fabsf(c.z - q.fz); dz = fminf(dz, Lz - dz); dz = fmaxf(0.f, __fsub_rd(dz, w.z));
  return __fadd_rd(__fadd_rd(__fmul_rd(dx, dx), __fmul_rd(dy, dy)), __fmul_rd(dz, dz));
}

// Eight consecutive queries of a leaf as a box, with the largest bound of the eight.
struct Group {
  float4 c;   // centre, bound on exact distances^2
  float4 w;   // half widths, padded
};

// Lower bound of the squared periodic distance between a group's box and a
// widened box (c, w), rounded down.
__device__ __forceinline__ float group_box_lb(const Group& g, const float4& c, const float4& w, float Lx, float Ly,
                                              float Lz) {
  const float4 gc = g.c, gw = g.w;
  float dx = fabsf(gc.x - c.x); dx = fminf(dx, Lx - dx); dx = fmaxf(0.f, __fsub_rd(__fsub_rd(dx, gw.x), w.x));
  float dy = fabsf(gc.y - c.y); dy = fminf(dy, Ly - dy); dy = fmaxf(0.f, __fsub_rd(__fsub_rd(dy, gw.y), w.y));
  float dz = fabsf(gc.z - c.z); dz = fminf(dz, Lz - dz); dz = fmaxf(0.f, __fsub_rd(__fsub_rd(dz, gw.z), w.z));
  return __fadd_rd(__fadd_rd(__fmul_rd(dx, dx), __fmul_rd(dy, dy)), __fmul_rd(dz, dz));
}

struct GroupsLb {
  float lb;  // to the nearest group
  bool in;   // within some group's bound
};
__device__ __forceinline__ GroupsLb groups_lb(const Group* g, const float4& c, const float4& w, float Lx, float Ly,
                                              float Lz) {
  GroupsLb r{CUDART_INF_F, false};
#pragma unroll 1
  for (int i = 0; i < 4; ++i) {
    const float d = group_box_lb(g[i], c, w, Lx, Ly, Lz);
    r.in |= d <= g[i].c.w;
    r.lb = fminf(r.lb, d);
  }
  return r;
}

// Half extent and centre of v over each eight consecutive lanes.
__device__ __forceinline__ void group_extent(float v, float& c, float& h) {
  float lo = v, hi = v;
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) {
    lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  c = 0.5f * (lo + hi);
  h = fmaxf(__fsub_ru(hi, c), __fsub_ru(c, lo));
}

// One leaf's particle in this lane, from memory and then as a row of a tile:
// relative to (ox, oy, oz) (nearest image), as floats; a lane past the end
// holds a particle far outside every bound.
struct LeafPart {
  double x, y, z;
  bool v;
};
__device__ __forceinline__ LeafPart load_part(const KnnArgs& A, int32_t leaf, int lane) {
  const int32_t p = leaf * kLeaf + lane;
  LeafPart r;
  r.v = p < A.n32;
  const double4 c = A.p4[r.v ? p : A.n32 - 1];
  r.x = c.x; r.y = c.y; r.z = c.z;
  return r;
}
__device__ __forceinline__ float fold_rel(double v, double o, double L) {
  double d = v - o;
  if (d > 0.5 * L) d -= L;
  else if (d < -0.5 * L) d += L;
  return (float)d;
}
// Squared FP32 distances (as float bits) of this lane's query to n staged
// particles (a multiple of four), four at a time: f(j, k0, k1, k2, k3).
// fold: the periodic image is taken per pair (wide leaves and bounds near
// half the box); otherwise the staged image is every query's.
template <class F>
__device__ __forceinline__ void tile_dist(const KnnArgs& A, const Query& q, const float* tx, const float* ty,
                                          const float* tz, int n, bool fold, F f) {
  if (fold) {
    const float Lx = (float)A.Lx, Ly = (float)A.Ly, Lz = (float)A.Lz;
    auto key = [&](int j) {
      float dx = fabsf(tx[j] + __uint_as_float((unsigned)q.nx)); dx = fminf(dx, fabsf(Lx - dx));
      float dy = fabsf(ty[j] + __uint_as_float((unsigned)q.ny)); dy = fminf(dy, fabsf(Ly - dy));
      float dz = fabsf(tz[j] + __uint_as_float((unsigned)q.nz)); dz = fminf(dz, fabsf(Lz - dz));
      return __float_as_uint(dx * dx + dy * dy + dz * dz);
    };
#pragma unroll 1
    for (int j = 0; j < n; j += 4) f(j, key(j), key(j + 1), key(j + 2), key(j + 3));
    return;
  }
#pragma unroll 2
  for (int j = 0; j < n; j += 4) {
    const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(tx + j);
    const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(ty + j);
    const ulonglong2 z = *reinterpret_cast<const ulonglong2*>(tz + j);
    const unsigned long long xa = add2(x.x, q.nx), xb = add2(x.y, q.nx);
    const unsigned long long ya = add2(y.x, q.ny), yb = add2(y.y, q.ny);
    const unsigned long long za = add2(z.x, q.nz), zb = add2(z.y, q.nz);
    const unsigned long long da = fma2(za, za, fma2(ya, ya, mul2(xa, xa)));
    const unsigned long long db = fma2(zb, zb, fma2(yb, yb, mul2(xb, xb)));
    f(j, (unsigned)da, (unsigned)(da >> 32), (unsigned)db, (unsigned)(db >> 32));
  }
}

// Batcher's merge exchange on N keys in registers (N <= 64): the passes of
// step P, then P / 2 and so on; compare (i, i + D) where i & P equals R.
template <int N, int P, int D, bool kHigh>
__device__ __forceinline__ void exchange_pass(unsigned (&k)[N]) {
#pragma unroll
  for (int i = 0; i + D < N; ++i) {
    if ((i & P) == (kHigh ? P : 0)) {
      const unsigned a = min(k[i], k[i + D]), b = max(k[i], k[i + D]);
      k[i] = a;
      k[i + D] = b;
    }
  }
}
template <int N, int P, int R>
__device__ __forceinline__ void exchange_high(unsigned (&k)[N]) {
  if constexpr (R > P) {
    exchange_pass<N, P, R - P, true>(k);
    exchange_high<N, P, R / 2>(k);
  }
}
template <int N, int T, int P>
__device__ __forceinline__ void merge_exchange(unsigned (&k)[N]) {
  if constexpr (P > 0) {
    exchange_pass<N, P, P, false>(k);
    exchange_high<N, P, T>(k);
    merge_exchange<N, T, P / 2>(k);
  }
}

// This lane's collected particles: entry e's slot, and the sort keys.
struct Column {
  const int32_t* coll;     // [entry][lane]
  unsigned* key;           // [entry][lane]
  __device__ __forceinline__ int32_t slot(int e) const { return coll[e * 32]; }
  __device__ __forceinline__ int32_t sorted(int i) const { return slot((int)(key[i * 32] & 63u)); }
};

// Sort the column's cnt entries by exact (distance, particle index), the query
// itself last: key i's 6 lowest bits become the entry number of the i-th.
// Keys are the distance rounded up to float with the entry number in those
// bits, through Batcher's merge-exchange network in registers (32 queries per
// instruction, no shuffles); distances that share the upper 26 bits among the
// first nv + 1 entries (within 2^-17, or exact ties) are put in order by an
// insertion pass on the exact values.  most: the warp's largest cnt.
__device__ __forceinline__ void sort_column(const KnnArgs& A, const Query& q, int32_t self, const Column& L, int cnt,
                                            int most, int nvv) {
#pragma unroll 8
  for (int e = 0; e < most; ++e) {
    const int32_t t = e < cnt ? L.slot(e) : self;
    const double d = exact_dist2(A, q, A.p4[t]);
    L.key[e * 32] = t == self ? 0xffffffffu : ((__float_as_uint(__double2float_ru(d)) & ~63u) | (unsigned)e);
  }
  unsigned k[kCollect];
#pragma unroll
  for (int e = 0; e < kCollect; ++e) k[e] = e < most ? L.key[e * 32] : 0xffffffffu;
  merge_exchange<kCollect, 32, 32>(k);
  bool tie = false;
#pragma unroll
  for (int i = 0; i < 32; ++i)
    tie |= i < nvv && k[i + 1] != 0xffffffffu && ((k[i] ^ k[i + 1]) < 64u);
#pragma unroll
  for (int i = 0; i < kCollect; ++i)
    if (i < most) L.key[i * 32] = k[i];
  if (tie) {
    double dp = exact_dist2(A, q, A.p4[L.sorted(0)]);
    for (int i = 1; i < cnt - 1; ++i) {
      const unsigned ki = L.key[i * 32];
      const int32_t t = L.sorted(i);
      const double d = exact_dist2(A, q, A.p4[t]);
      int j = i;
      if (d <= dp) {
        const int32_t o = A.orig[t];
        while (j > 0) {
          const int32_t u = L.sorted(j - 1);
          const double du = exact_dist2(A, q, A.p4[u]);
          if (du < d || (du == d && A.orig[u] < o)) break;
          L.key[j * 32] = L.key[(j - 1) * 32];
          --j;
        }
      }
      if (j != i) L.key[j * 32] = ki;
      else dp = d;
    }
  }
}

// One warp per query leaf (its 32 Morton-consecutive particles), lane = query.
//  A. the distances to the leaf's own and its two adjacent leaves' particles
//     are counted in bins of the float bits (first whole octaves, then 8 bins
//     per octave below the octave that holds the (nv+1)-th, the query itself
//     included): the upper edge of the bin that holds it bounds the radius;
//  B. a traversal from the root collects the leaves that some query's bound
//     reaches, in batches sorted by box-to-box distance;
//  C. the candidates are counted nearest-first into the same bins, each lane
//     lowering its edge while nv + 1 particles stay below it; a leaf that no
//     query's bound reaches any more is skipped.  A lane left with too many
//     particles below its edge lays its bins lower or finer and counts again;
//  D. the counted leaves are read again and the slots of every particle below
//     its lane's final edge are collected (33 to 40 of them for nv = 32).
// Boxes are tested in B one per lane against four boxes of eight queries each
// with their own bounds, in C one by one against every query; in C and D the
// particles of a leaf are tested one per lane against the query leaf's box
// grown by the largest bound, and only those within are staged for the 32
// queries.
// knn_finish_kernel sorts and sums; apart from this one because the two bodies
// together do not fit the instruction cache.  Queries that collect more than
// kCollect particles (many equal distances), and whole leaves that count too
// many leaves or have too few particles around, are left to the per-query
// search there, below the bound they have (count 0).
// kProf: the counters and cycle stamps of the profiling API.
template <int C, bool kProf>
__global__ void __launch_bounds__(kKnnWarps * 32, kKnnBlocks) knn_collect_kernel(KnnArgs A) {
  extern __shared__ __align__(16) unsigned char s_raw[];
  unsigned char* const W = s_raw + (threadIdx.x >> 5) * kWarpBytes;
  const int lane = threadIdx.x & 31;
  const int nleaf = (int)A.lev_cnt[0];
  const int top = A.nlev - 1;
  const int nvv = C ? C : A.nv, need = nvv + 1;
  const float Lxf = (float)A.Lx, Lyf = (float)A.Ly, Lzf = (float)A.Lz;
  unsigned* const col = reinterpret_cast<unsigned*>(W + kOffBins) + lane;
  float* const tile = reinterpret_cast<float*>(W + kOffTile);
  int32_t* const tslot = reinterpret_cast<int32_t*>(W + kOffTile) + 3 * kTile;
  unsigned* const skey = reinterpret_cast<unsigned*>(W + kOffKey);
  int32_t* const scand = reinterpret_cast<int32_t*>(W + kOffCand);
  int32_t* const sstack = reinterpret_cast<int32_t*>(W + kOffStack);
  float4* const sbox = reinterpret_cast<float4*>(W + kOffBox);
  Group* const sgroup = reinterpret_cast<Group*>(W + kOffGroup);
  int32_t* const svis = reinterpret_cast<int32_t*>(W + kOffVis);
  for (;;) {
    int jl = 0;
    if (lane == 0) jl = atomicAdd(A.next, 1);
    jl = __shfl_sync(0xffffffffu, jl, 0);
    if (jl >= A.nchunk) break;
    const int row0 = jl;  // within the chunk
    jl += A.leaf0;
    const long long t_0 = kProf ? clock64() : 0;
    const int32_t s = jl * kLeaf + lane;
    const bool live = s < A.n32;
    const int32_t self = live ? s : A.n32 - 1;  // lanes past the end repeat the last query
    const double* ob = A.box + 6 * (int64_t)jl;
    const double ox = ob[0], oy = ob[1], oz = ob[2];
    Query q;
    {
      const double4 p = A.p4[self];
      q.x = p.x; q.y = p.y; q.z = p.z;
    }
    q.fx = (float)q.x; q.fy = (float)q.y; q.fz = (float)q.z;
    const float lx = (float)(q.x - ox), ly = (float)(q.y - oy), lz = (float)(q.z - oz);
    q.nx = pack2(-lx); q.ny = pack2(-ly); q.nz = pack2(-lz);
    // largest query coordinate: the FP32 coordinates of a pair within d of each
    // other are off by at most 2^-24 (2 amax + 2 d) per axis, far inside the
    // margins of widen()
    const float amax = __uint_as_float(__reduce_max_sync(
        0xffffffffu, __float_as_uint(fmaxf(fabsf(lx), fmaxf(fabsf(ly), fabsf(lz))))));
    const float beyond = A.box32[2 * (int64_t)jl].w;  // pairs more than a box length apart (leaf_box32_kernel)
    const float eabs2 = 0x1p-19f * amax + A.eabs2 + beyond;
    bool whole = !(beyond < CUDART_INF_F);  // the per-query search for the whole leaf
    // a bound on FP32 distances -> a bound on exact ones, and back: (sqrt(e)
    // (1 + 2^-19) + 2 eabs)^2 covers both steps
    auto widen = [&](float e2) {
      const float d = sqrtf(e2) * (1.f + 0x1p-19f) + eabs2;
      return d * d * (1.f + 0x1p-20f);
    };
    // ---- A: bound from the three leaves around.  The images of the tiles are
    // the nearest to the leaf's centre, perhaps not to every query: their
    // distances are never below the periodic ones, so the bound holds.
    float* const seed = reinterpret_cast<float*>(W + kOffSeed);
    int nt = 0;
    for (int k = 0; k < 3; ++k) {
      const int l = k == 0 ? jl : (k == 1 ? jl + 1 : jl - 1);
      if (l < 0 || l >= nleaf) continue;
      const LeafPart p = load_part(A, l, lane);
      seed[nt + lane] = p.v ? fold_rel(p.x, ox, A.Lx) : 1e18f;
      seed[96 + nt + lane] = p.v ? fold_rel(p.y, oy, A.Ly) : 1e18f;
      seed[192 + nt + lane] = p.v ? fold_rel(p.z, oz, A.Lz) : 1e18f;
      nt += 32;
    }
#pragma unroll 8
    for (int b = 0; b < kBins; ++b) col[b * 32] = 0u;
    __syncwarp();
    // whole octaves, the 31 up to 4 L^2 and one for "farther" (no particle
    // there); a lane with nv + 1 in the lowest looks 30 octaves lower, where
    // that one is the highest
    int oct = 0, obase = A.obase;
    for (bool lower = !whole; lower;) {
      tile_dist(A, q, seed, seed + 96, seed + 192, nt, false,
                [&](int, unsigned k0, unsigned k1, unsigned k2, unsigned k3) {
                  atomicAdd(&col[min(max((int)(k0 >> 23) - obase, 0), kBins - 1) * 32], 1u);
                  atomicAdd(&col[min(max((int)(k1 >> 23) - obase, 0), kBins - 1) * 32], 1u);
                  atomicAdd(&col[min(max((int)(k2 >> 23) - obase, 0), kBins - 1) * 32], 1u);
                  atomicAdd(&col[min(max((int)(k3 >> 23) - obase, 0), kBins - 1) * 32], 1u);
                });
      int cum = 0;
      oct = 0;
#pragma unroll 8
      for (int b = 0; b < kBins; ++b) {
        cum += (int)col[b * 32];
        col[b * 32] = 0u;
        if (cum < need) oct = b + 1;
      }
      const bool low = oct == 0 && obase > 0;
      if (low) obase -= kBins - 2;
      lower = __any_sync(0xffffffffu, low);
    }
    whole |= __any_sync(0xffffffffu, oct >= kBins - 1);
    unsigned lim = (unsigned)(obase + oct + 1) << 23;  // float bits: upper edge, exclusive
    int shift = kBinShift;
    int wbase = (int)(lim >> shift) - kBins;      // bin b: bits [(wbase + b) << shift, (wbase + b + 1) << shift)
    int binned = 0, ebin = kBins - 1;             // particles below the edge, the edge's bin
    auto count4 = [&](int, unsigned k0, unsigned k1, unsigned k2, unsigned k3) {
      if (min(min(k0, k1), min(k2, k3)) < lim) {
        if (k0 < lim) { atomicAdd(&col[max((int)(k0 >> shift) - wbase, 0) * 32], 1u); ++binned; }
        if (k1 < lim) { atomicAdd(&col[max((int)(k1 >> shift) - wbase, 0) * 32], 1u); ++binned; }
        if (k2 < lim) { atomicAdd(&col[max((int)(k2 >> shift) - wbase, 0) * 32], 1u); ++binned; }
        if (k3 < lim) { atomicAdd(&col[max((int)(k3 >> shift) - wbase, 0) * 32], 1u); ++binned; }
      }
    };
    float bnd = CUDART_INF_F;  // exact distances^2 beyond this cannot be among the nv nearest
    auto tighten = [&]() {  // whether any lane's bound moved
      bool moved = false;
      for (int h = (int)col[ebin * 32]; ebin > 0 && binned - h >= need; h = (int)col[ebin * 32]) {
        binned -= h;
        --ebin;
        moved = true;
      }
      if (moved) {
        lim = (unsigned)(wbase + ebin + 1) << shift;
        bnd = widen(__uint_as_float(lim));
      }
      return __any_sync(0xffffffffu, moved);
    };
    if (!whole) {
      tile_dist(A, q, seed, seed + 96, seed + 192, nt, false, count4);
      bnd = widen(__uint_as_float(lim));
      tighten();
    }
    // the staged images are those of the nearest image for every pair that
    // matters only while the bound and the leaf fit half the box
    const float maxb = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(bnd)));
    const bool fold = !(sqrtf(maxb) + amax < A.near);
    float grown;  // FP32 bound on a particle's distance from the query leaf's box
    const float hx = __double2float_ru(ob[3]), hy = __double2float_ru(ob[4]), hz = __double2float_ru(ob[5]);
    {
      float4 c, w;
      group_extent(q.fx, c.x, w.x); group_extent(q.fy, c.y, w.y); group_extent(q.fz, c.z, w.z);
      w.x += A.gpad; w.y += A.gpad; w.z += A.gpad;  // rounding of the queries to float
      c.w = w.w = 0.f;
      if ((lane & 7) == 0) sgroup[lane >> 3] = Group{c, w};
    }
    // the largest bounds of the groups and of all lanes (negative: this lane needs nothing)
    auto regrow = [&]() {
      float b = bnd;
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) b = fmaxf(b, __shfl_xor_sync(0xffffffffu, b, o));
      __syncwarp();
      if ((lane & 7) == 0) sgroup[lane >> 3].c.w = b;
      b = fmaxf(b, 0.f);
      b = fmaxf(b, __shfl_xor_sync(0xffffffffu, b, 8));
      b = fmaxf(b, __shfl_xor_sync(0xffffffffu, b, 16));
      grown = widen(b);
      __syncwarp();
    };
    __syncwarp();
    regrow();
    const long long t_a = kProf ? clock64() : 0;
    long long t_b = t_a, t_c = t_a, c_cand = 0;
    int cnt = 0;  // collected particles
    int nvis = 0, ncand_all = 0, npop = 0;
    int window = 0;  // 0: counting candidates, then the number of times bins were laid lower or finer
    unsigned ntest = 0, nread = 0;
    if (!whole) {
      // Walks a list of leaves in chunks of 32: tests each leaf's box against
      // every query (test), loads the next leaf's particles while the current
      // one is staged, and hands the staged ones on in groups of 32: take(leaf)
      // says whether to stage a leaf, use(n) works on the n staged particles.
      auto walk = [&](const int32_t* list, int nlist, bool test, auto&& take, auto&& use) {
        int fill = 0;
        for (int c0 = 0; c0 < nlist; c0 += 32) {
          bool in = c0 + lane < nlist;
          const int32_t mine = in ? list[c0 + lane] : 0;
          __syncwarp();
          if (test) {
            const float4 bc = A.box32[2 * (int64_t)mine], bw = A.box32[2 * (int64_t)mine + 1];
            sbox[2 * lane] = bc;
            sbox[2 * lane + 1] = bw;
            in = in && groups_lb(sgroup, bc, bw, Lxf, Lyf, Lzf).in;
            __syncwarp();
          }
          unsigned mask = __ballot_sync(0xffffffffu, in);
          if (!mask) continue;
          int src = __ffs(mask) - 1;
          int32_t cur = __shfl_sync(0xffffffffu, mine, src);
          LeafPart part = load_part(A, cur, lane);
          while (mask) {
            const int32_t leaf_now = cur;
            const LeafPart now = part;
            const int at = src;
            mask &= mask - 1;
            src = mask ? __ffs(mask) - 1 : at;
            cur = __shfl_sync(0xffffffffu, mine, src);
            part = load_part(A, cur, lane);
            if (kProf) ++ntest;
            if ((!test || __any_sync(0xffffffffu,
                                     query_box_lb(q, sbox[2 * at], sbox[2 * at + 1], Lxf, Lyf, Lzf) <= bnd)) &&
                take(leaf_now)) {
              const float fx = fold_rel(now.x, ox, A.Lx), fy = fold_rel(now.y, oy, A.Ly),
                          fz = fold_rel(now.z, oz, A.Lz);
              const float dx = fmaxf(fabsf(fx) - hx, 0.f), dy = fmaxf(fabsf(fy) - hy, 0.f),
                          dz = fmaxf(fabsf(fz) - hz, 0.f);
              const bool keep = now.v && (fold || fmaf(dz, dz, fmaf(dy, dy, dx * dx)) <= grown);
              const unsigned km = __ballot_sync(0xffffffffu, keep);
              if (keep) {
                const int to = fill + __popc(km & ((1u << lane) - 1));
                tile[to] = fx;
                tile[kTile + to] = fy;
                tile[2 * kTile + to] = fz;
                tslot[to] = leaf_now * kLeaf + lane;
              }
              fill += __popc(km);
              if (fill >= 32) {
                __syncwarp();
                use(32);
                fill -= 32;
                if (kProf) nread += 32;
                const float mx = tile[32 + lane], my = tile[kTile + 32 + lane], mz = tile[2 * kTile + 32 + lane];
                const int32_t ms = tslot[32 + lane];
                __syncwarp();
                if (lane < fill) {
                  tile[lane] = mx;
                  tile[kTile + lane] = my;
                  tile[2 * kTile + lane] = mz;
                  tslot[lane] = ms;
                }
              }
            }
          }
        }
        if (fill) {
          const int n4 = (fill + 3) & ~3;
          if (lane < n4 - fill) {
            tile[fill + lane] = 1e18f;
            tile[kTile + fill + lane] = 1e18f;
            tile[2 * kTile + fill + lane] = 1e18f;
          }
          __syncwarp();
          use(n4);
          if (kProf) nread += n4;
        }
        __syncwarp();
      };
      int sp = 1;
      if (lane == 0) sstack[0] = top << 27;
      __syncwarp();
      unsigned lim_kept = 0u;
      float bnd_kept = 0.f;
      bool again = false;   // this lane counts in the current lower window
      for (;;) {
        const int32_t* list = svis;
        int nlist = nvis;
        if (window == 0) {
          // ---- B: a batch of candidate leaves, sorted by box-to-box distance
          const long long t_t = kProf ? clock64() : 0;
          int ncand = 0;
          if (top == 0) {  // a single leaf
            if (lane == 0) { skey[0] = 0u; scand[0] = 0; }
            ncand = 1;
            sp = 0;
          }
          while (sp > 0) {
            if (++npop > kNodeMax) { whole = true; break; }
            --sp;
            const int32_t ent = sstack[sp];
            __syncwarp();
            const int lvl = ent >> 27;
            const int64_t c = (int64_t)(ent & ((1 << 27) - 1)) * kFan + lane;
            GroupsLb g{CUDART_INF_F, false};
            if (c < A.lev_cnt[lvl - 1]) {
              const float4* b = A.box32 + 2 * (A.lev_off[lvl - 1] + c);
              g = groups_lb(sgroup, b[0], b[1], Lxf, Lyf, Lzf);
            }
            const unsigned hit = __ballot_sync(0xffffffffu, g.in);
            const int cnt = __popc(hit);
            if (!cnt) continue;
            const int r = __popc(hit & ((1u << lane) - 1));
            const bool mine = (hit >> lane) & 1u;
            if (lvl == 1) {
              if (ncand + cnt > kBatch) { ++sp; break; }  // the batch is full: this node again, after it
              if (mine) {
                // sort key: the leaf-to-leaf distance rounded down to 20 bits, then the place
                skey[ncand + r] = ((__float_as_uint(g.lb) >> 11) << 12) | (unsigned)(ncand + r);
                scand[ncand + r] = (int32_t)c;
              }
              ncand += cnt;
            } else {
              if (sp + cnt > kTravStack) { whole = true; break; }
              if (mine) sstack[sp + r] = ((lvl - 1) << 27) | (int32_t)c;
              sp += cnt;
            }
            __syncwarp();
          }
          __syncwarp();
          ncand_all += ncand;
          if (whole || ncand_all > kCandMax) { whole = true; break; }
          int N = 32;
          while (N < ncand) N <<= 1;
          for (int i = ncand + lane; i < N; i += 32) skey[i] = 0xffffffffu;
          __syncwarp();
          for (int k = 2; k <= N; k <<= 1) {
            for (int j = k >> 1; j > 0; j >>= 1) {
              for (int t = lane; t < (N >> 1); t += 32) {
                const int i = ((t & ~(j - 1)) << 1) | (t & (j - 1));
                const unsigned u = skey[i], v = skey[i + j];
                if ((u > v) == ((i & k) == 0)) { skey[i] = v; skey[i + j] = u; }
              }
              __syncwarp();
            }
          }
          // the leaves in that order, in the keys' place
          for (int i = lane; i < ncand; i += 32) skey[i] = (unsigned)scand[skey[i] & (kBatch - 1)];
          __syncwarp();
          list = reinterpret_cast<const int32_t*>(skey);
          nlist = ncand;
          if (kProf) c_cand += clock64() - t_t;
        }
        // ---- C: count
        walk(
            list, nlist, true,
            [&](int32_t leaf_now) {
              if (window > 0) return true;
              if (nvis < kVisMax) {
                if (lane == 0) svis[nvis] = leaf_now;
                ++nvis;
              } else {
                whole = true;
              }
              return leaf_now < jl - 1 || leaf_now > jl + 1;  // those are counted in A
            },
            [&](int n) {
              tile_dist(A, q, tile, tile + kTile, tile + 2 * kTile, n, fold, count4);
              if (tighten()) regrow();
            });
        if (whole) break;
        if (window == 0 && sp > 0) continue;
        // lanes with too many particles below their edge count the listed leaves
        // again: where the edge is the lowest bin's, with the bins laid below it;
        // else (a far clump inside one bin) with the edge's bin cut in 32
        if (window > 0 && !again) { lim = lim_kept; bnd = bnd_kept; }
        again = binned > kCollect - 4 && shift > kBinShift - 15;
        if (window == kWindows || !__any_sync(0xffffffffu, again)) break;
        ++window;
        lim_kept = lim;
        bnd_kept = bnd;
        if (again) {
          if (ebin == 0 && shift == kBinShift) {
            wbase = (int)(lim >> shift) - kBins;
          } else {
            wbase = (wbase + ebin) << 5;
            shift -= 5;
          }
          ebin = kBins - 1;
          binned = 0;
#pragma unroll 8
          for (int b = 0; b < kBins; ++b) col[b * 32] = 0u;
        } else {
          lim = 0u;
          bnd = -1.f;
        }
        regrow();
      }
      t_c = kProf ? clock64() : 0;
      t_b = t_a + c_cand;
      if (!whole) {
        // ---- D: collect
        regrow();
        const unsigned lim2 = __float_as_uint(bnd);  // at most this: FP32 distance of any of the nv + 1 nearest
        int32_t* const out = A.coll + (size_t)row0 * (kCollect * 32) + lane;
        walk(
            svis, nvis, false, [&](int32_t) { return true; },
            [&](int n) {
              tile_dist(A, q, tile, tile + kTile, tile + 2 * kTile, n, fold,
                        [&](int j, unsigned k0, unsigned k1, unsigned k2, unsigned k3) {
                          if (min(min(k0, k1), min(k2, k3)) <= lim2) {
                            const int4 t = *reinterpret_cast<const int4*>(tslot + j);
                            if (k0 <= lim2) { if (cnt < kCollect) out[cnt * 32] = t.x; ++cnt; }
                            if (k1 <= lim2) { if (cnt < kCollect) out[cnt * 32] = t.y; ++cnt; }
                            if (k2 <= lim2) { if (cnt < kCollect) out[cnt * 32] = t.z; ++cnt; }
                            if (k3 <= lim2) { if (cnt < kCollect) out[cnt * 32] = t.w; ++cnt; }
                          }
                        });
            });
      }
    }
    if (cnt > kCollect || cnt < need) {
      cnt = 0;
      if (live) {
        A.coll[(size_t)row0 * (kCollect * 32) + lane] = (int32_t)__float_as_uint(bnd >= 0.f ? bnd : CUDART_INF_F);
        A.lost[atomicAdd(A.nlost, 1)] = row0 * 32 + lane;
      }
    }
    A.ccnt[(size_t)row0 * 32 + lane] = (uint8_t)cnt;
    if (kProf) {
      const unsigned c = __reduce_add_sync(0xffffffffu, live ? (unsigned)cnt : 0u);
      const unsigned lost = __popc(__ballot_sync(0xffffffffu, live && cnt == 0));
      if (lane == 0) {
        atomicAdd(&A.kstats[3], (unsigned long long)c);
        atomicAdd(&A.kstats[5], (unsigned long long)lost);
      }
    }
    __syncwarp();
    if (kProf && lane == 0) {
      const long long t_e = clock64();
      unsigned long long* ph = A.kstats + 24;
      atomicAdd(&A.kstats[0], 1ULL);
      atomicAdd(&A.kstats[1], (unsigned long long)ncand_all);
      atomicAdd(&A.kstats[2], (unsigned long long)nvis);
      atomicAdd(&A.kstats[8], (unsigned long long)ntest);
      atomicAdd(&A.kstats[9], (unsigned long long)nread);
      atomicAdd(&A.kstats[10], (unsigned long long)window);
      if (whole) atomicAdd(&A.kstats[4], 1ULL);
      atomicAdd(&A.kstats[whole ? 6 : 7], (unsigned long long)(t_e - t_0));
      if (!whole) {
        atomicAdd(&ph[0], (unsigned long long)(t_a - t_0));
        atomicAdd(&ph[1], (unsigned long long)(t_b - t_a));
        atomicAdd(&ph[2], (unsigned long long)(t_c - t_b));
        atomicAdd(&ph[3], (unsigned long long)(t_e - t_c));
      }
    }
  }
}

// The collected particles of each query (lane = query) in exact order, the SPH
// density in the reference's evaluation order (f90:2816-2838) and the stored
// neighbour slots.
template <int C, bool kProf>
__global__ void __launch_bounds__(kFinWarps * 32, kFinBlocks) knn_finish_kernel(KnnArgs A) {
  __shared__ __align__(16) unsigned s_sort[kFinWarps][kCollect * 32];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int row0 = blockIdx.x * kFinWarps + wib;
  if (row0 >= A.nchunk) return;
  const long long t_0 = kProf ? clock64() : 0;
  const int nvv = C ? C : A.nv;
  const int32_t s0 = (A.leaf0 + row0) * kLeaf, s = s0 + lane;
  const bool live = s < A.n32;
  const int32_t self = live ? s : A.n32 - 1;
  Query q;
  const double4 me = A.p4[self];
  q.x = me.x; q.y = me.y; q.z = me.z;
  const int cnt = live ? (int)A.ccnt[(size_t)row0 * 32 + lane] : 0;
  const int32_t* const coll = A.coll + (size_t)row0 * (kCollect * 32) + lane;
  const Column L{coll, s_sort[wib] + lane};
  sort_column(A, q, self, L, cnt, (int)__reduce_max_sync(0xffffffffu, (unsigned)cnt), nvv);
  if (cnt) {
    const double dlast = exact_dist2(A, q, A.p4[L.sorted(nvv - 1)]);
    const double r = xmul(xsqrt(dlast), 0.5);
    const double r3 = xmul(xmul(r, r), r);
    const double unsr = xdiv(1.0, r);
    double contrib = 0.0;
    int32_t* out = A.nei + (size_t)s * A.nstore;
#pragma unroll 4
    for (int i = 0; i < nvv; ++i) {
      const int32_t t = L.sorted(i);
      if (i < A.nstore) out[i] = t;
      const double4 p = A.p4[t];
      if (i < nvv - 1) contrib = xadd(contrib, xmul(p.w, spline(xmul(xsqrt(exact_dist2(A, q, p)), unsr))));
    }
    const double pi_f = (double)3.141592654f;  // f90:58 single-precision literal
    A.dens[s] = xdiv(xmul(A.xyzlong, xadd(contrib, me.w)), xmul(pi_f, r3));
  }
  if (kProf && lane == 0) atomicAdd(A.kstats + 28, (unsigned long long)(clock64() - t_0));
}

// One warp per query: the queries of a chunk that the lane-per-query kernels
// left over (kAll false), below the bound they have, or every query of a small
// set (kAll) and those left without a bound, below the (nv+1)-th distance (to 8
// bits) among the particles of its own and the two adjacent leaves.
template <int C, bool kAll>
__global__ void __launch_bounds__(kFinWarps * 32) knn_query_kernel(KnnArgs A) {
  __shared__ double s_bd[kFinWarps][kStack];
  __shared__ int32_t s_node[kFinWarps][kStack];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int nq = kAll ? A.n32 : *A.nlost;
  const int nvv = C ? C : A.nv;
  for (int i = blockIdx.x * kFinWarps + wib; i < nq; i += gridDim.x * kFinWarps) {
    int32_t s = i;
    double cap = CUDART_INF;
    if (!kAll) {
      const int at = A.lost[i];
      s = A.leaf0 * kLeaf + at;
      cap = (double)__uint_as_float((unsigned)A.coll[(size_t)(at >> 5) * (kCollect * 32) + (at & 31)]);
    }
    const double4 p = A.p4[s];
    if (kAll || !(cap < CUDART_INF)) {
      unsigned k[3];
#pragma unroll
      for (int t = 0; t < 3; ++t) {
        const int32_t c = ((s >> 5) + t - 1) * kLeaf + lane;
        k[t] = 0x7F800000u;
        if (c >= 0 && c < A.n32) {
          const double4 r = A.p4[c];
          k[t] = __float_as_uint(__double2float_ru(pdist2(p.x, p.y, p.z, r.x, r.y, r.z, A.Lx, A.Ly, A.Lz)));
        }
      }
      // smallest edge (multiple of 2^15 in the float bits) with nv + 1 at or below it
      unsigned lo = 0u;
      for (unsigned bit = 1u << 30; bit >= 1u << 15; bit >>= 1) {
        const unsigned e = lo | (bit - 1u);
        const int c = __popc(__ballot_sync(0xffffffffu, k[0] <= e)) + __popc(__ballot_sync(0xffffffffu, k[1] <= e)) +
                      __popc(__ballot_sync(0xffffffffu, k[2] <= e));
        if (c < nvv + 1) lo |= bit;
      }
      lo |= 0x7fffu;
      cap = lo < 0x7F800000u ? (double)__uint_as_float(lo) : CUDART_INF;
    }
    WarpList W{CUDART_INF, -1, cap, cap};
    query_dfs<C>(A, W, s, p.x, p.y, p.z, lane, s_node[wib], s_bd[wib]);
    finish_query<C>(A, W, s, lane, s_bd[wib]);
    __syncwarp();
  }
}

int stage_knn_density(Engine& E) {
  const int64_t n = E.n;
  const Params& P = E.prm;
  E.nstore = E.req_store > 0 ? E.req_store : P.nhop;
  if (E.nstore < P.nhop) E.nstore = P.nhop;
  if (E.nstore > P.nvoisins) E.nstore = P.nvoisins;
  AHOP_CUDA_TRY(E.d_nei.ensure((size_t)n * E.nstore * 4));
  AHOP_CUDA_TRY(E.d_dens.ensure(n * 8));
  KnnArgs A;
  A.p4 = E.rows();
  A.m = E.d_m.as<double>();
  A.orig = E.d_orig.as<int32_t>();
  A.box = E.d_box.as<double>();
  const int64_t nbox = E.lev_off[E.nlev];  // boxes of every level
  AHOP_CUDA_TRY(E.d_box32.ensure((size_t)nbox * 32 + 32));
  A.box32 = E.d_box32.as<float4>();
  const double Lmin = std::min(P.xlong, std::min(P.ylong, P.zlong)), Lmax = std::max(P.xlong, std::max(P.ylong, P.zlong));
  E.launches++;
  leaf_box32_kernel<<<(unsigned)((nbox + 255) / 256), 256, 0, E.stream>>>(
      A.box, nbox, P.xlong, P.ylong, P.zlong, Lmax < 1e15 && Lmin > 1e-8, E.d_box32.as<float4>());
  AHOP_CUDA_TRY(cudaGetLastError());
  for (int l = 0; l < kMaxLevels; ++l) { A.lev_off[l] = E.lev_off[l]; A.lev_cnt[l] = E.lev_cnt[l]; }
  A.nlev = E.nlev;
  A.n = n;
  A.n32 = (int32_t)n;
  A.Lx = P.xlong; A.Ly = P.ylong; A.Lz = P.zlong; A.xyzlong = P.xyzlong;
  A.eabs2 = (float)(0x1p-45 * Lmax);
  A.gpad = (float)(0x1p-22 * Lmax);
  A.near = (float)(0.49 * Lmin);
  {
    const float l2 = (float)(4.0 * Lmax * Lmax);
    uint32_t bits;
    std::memcpy(&bits, &l2, 4);
    A.obase = (int)(bits >> 23) - (kBins - 2);
  }
  A.nv = P.nvoisins;
  A.nstore = E.nstore;
  A.nei = E.d_nei.as<int32_t>();
  A.dens = E.d_dens.as<double>();
  AHOP_CUDA_TRY(E.d_flags.ensure(512));
  AHOP_CUDA_TRY(cudaMemsetAsync(E.d_flags.p, 0, 512, E.stream));
  A.err = E.d_flags.as<int>();
  A.next = E.d_flags.as<int>() + 1;
  A.kstats = reinterpret_cast<unsigned long long*>(E.d_flags.as<char>() + 64);
  int nsm = 148;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, E.device);
  // the default nvoisins = 32 has its own build with the count fixed at compile time
  const bool nv32 = P.nvoisins == 32;
  const bool prof = E.task_profile;
  auto kcol = nv32 ? (prof ? knn_collect_kernel<32, true> : knn_collect_kernel<32, false>)
                   : (prof ? knn_collect_kernel<0, true> : knn_collect_kernel<0, false>);
  auto kfin = nv32 ? (prof ? knn_finish_kernel<32, true> : knn_finish_kernel<32, false>)
                   : (prof ? knn_finish_kernel<0, true> : knn_finish_kernel<0, false>);
  const size_t smem = (size_t)kKnnWarps * kWarpBytes;
  AHOP_CUDA_TRY(cudaFuncSetAttribute(kcol, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int per_sm = 0;
  AHOP_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kcol, kKnnWarps * 32, smem));
  if (per_sm < 1) per_sm = 1;
  const int64_t nleaf = E.lev_cnt[0];
  const int64_t chunk = std::min<int64_t>(nleaf, kChunkLeaves);
  const bool all = n <= kPerQueryMax;
  if (!all) AHOP_CUDA_TRY(E.d_dens_orig.ensure((size_t)chunk * (kCollect * 32 * 4 + 32 * 4 + 32)));
  A.coll = E.d_dens_orig.as<int32_t>();
  A.lost = A.coll + (size_t)chunk * kCollect * 32;
  A.ccnt = reinterpret_cast<uint8_t*>(A.lost + (size_t)chunk * 32);
  A.nlost = A.next + 1;
  AHOP_CUDA_TRY(cudaEventRecord(E.ev[9], E.stream));
  if (all) {
    const unsigned g = (unsigned)((n + kFinWarps - 1) / kFinWarps);
    if (nv32) knn_query_kernel<32, true><<<g, kFinWarps * 32, 0, E.stream>>>(A);
    else knn_query_kernel<0, true><<<g, kFinWarps * 32, 0, E.stream>>>(A);
    AHOP_CUDA_TRY(cudaGetLastError());
    E.launches++;
  }
  for (int64_t l0 = all ? nleaf : 0; l0 < nleaf; l0 += chunk) {
    A.leaf0 = (int)l0;
    A.nchunk = (int)std::min(chunk, nleaf - l0);
    if (l0) AHOP_CUDA_TRY(cudaMemsetAsync(A.next, 0, 8, E.stream));
    // one resident wave; every warp takes the next query leaf when it is done with one
    const int64_t want = (A.nchunk + kKnnWarps - 1) / kKnnWarps;
    kcol<<<(unsigned)std::min((int64_t)nsm * per_sm, want), kKnnWarps * 32, smem, E.stream>>>(A);
    kfin<<<(unsigned)((A.nchunk + kFinWarps - 1) / kFinWarps), kFinWarps * 32, 0, E.stream>>>(A);
    const unsigned lgrid = (unsigned)std::min<int64_t>(nsm * kLostBlocks, (A.nchunk * 32 + kFinWarps - 1) / kFinWarps);
    if (nv32) knn_query_kernel<32, false><<<lgrid, kFinWarps * 32, 0, E.stream>>>(A);
    else knn_query_kernel<0, false><<<lgrid, kFinWarps * 32, 0, E.stream>>>(A);
    AHOP_CUDA_TRY(cudaGetLastError());
    E.launches += 3;
  }
  AHOP_CUDA_TRY(cudaEventRecord(E.ev[10], E.stream));
  // the error flag is looked at after the next stage's synchronisation
  AHOP_CUDA_TRY(cudaMemcpyAsync(E.h_scalars + Engine::kHostScalars - 1, E.d_flags.p, 4, cudaMemcpyDeviceToHost,
                                E.stream));
  if (prof) {
    AHOP_CUDA_TRY(cudaMemcpyAsync(E.knn_stats, E.d_flags.as<char>() + 64, 12 * 8, cudaMemcpyDeviceToHost, E.stream));
    AHOP_CUDA_TRY(cudaMemcpyAsync(E.knn_phase, E.d_flags.as<char>() + 64 + 24 * 8, 5 * 8, cudaMemcpyDeviceToHost,
                                  E.stream));
    AHOP_CUDA_TRY(cudaStreamSynchronize(E.stream));
  } else {
    std::memset(E.knn_stats, 0, sizeof E.knn_stats);
    std::memset(E.knn_phase, 0, sizeof E.knn_phase);
  }
  return AHOP_OK;
}

bool knn_failed(Engine& E) {
  int32_t e;
  std::memcpy(&e, E.h_scalars + Engine::kHostScalars - 1, 4);
  if (e) set_error("kNN traversal stack overflow");
  return e != 0;
}

}  // namespace ahop
