// Internal state of the AdaptaHOP engine (one per process, like the Fortran
// module neiKDtree).  All particle arrays live in HBM in Morton-sorted order
// ("s" index); orig[s] maps back to the caller's 0-based particle index.
#pragma once
#include <cstdint>
#include <string>
#include <vector>
#include <cuda_runtime.h>

#include "ahop_b200.h"

namespace ahop {

// Growable device buffer; never shrinks until close().
struct DevBuf {
  void* p = nullptr;
  size_t bytes = 0;
  cudaError_t ensure(size_t need) {
    if (need <= bytes) return cudaSuccess;
    if (p) cudaFree(p);
    p = nullptr;
    bytes = 0;
    cudaError_t e = cudaMalloc(&p, need ? need : 16);
    if (e == cudaSuccess) bytes = need ? need : 16;
    else p = nullptr;
    return e;
  }
  void release() {
    if (p) cudaFree(p);
    p = nullptr;
    bytes = 0;
  }
  template <class T> T* as() const { return static_cast<T*>(p); }
};

// A buffer whose size follows counts that differ a little from one snapshot to
// the next (groups, links, nodes): when it has to grow it takes an eighth more,
// 32 MB at most, since each growth is a cudaFree and a cudaMalloc (262,144
// particles: a call that grows them 10.5 ms instead of 5.3).  A call that runs
// out of memory gives everything back and runs again without (with_room in
// capi.cu), so that slack never takes the room of a later buffer.
inline thread_local bool exact_buffers = false;
struct CountBuf : DevBuf {
  cudaError_t ensure(size_t need) {
    if (p && need > bytes && !exact_buffers) {
      const size_t slack = need / 8 < ((size_t)32 << 20) ? need / 8 : (size_t)32 << 20;
      if (DevBuf::ensure(need + slack) == cudaSuccess) return cudaSuccess;
      cudaGetLastError();
    }
    return DevBuf::ensure(need);
  }
};

// A part of a buffer.
struct DevView {
  void* p = nullptr;
  template <class T> T* as() const { return static_cast<T*>(p); }
};

// Growable pinned host buffer (module outputs live here; fast D2H).
struct HostBuf {
  void* p = nullptr;
  size_t bytes = 0;
  cudaError_t ensure(size_t need) {
    if (need <= bytes) return cudaSuccess;
    if (p) cudaFreeHost(p);
    p = nullptr;
    bytes = 0;
    cudaError_t e = cudaMallocHost(&p, need ? need : 16);
    if (e == cudaSuccess) bytes = need ? need : 16;
    return e;
  }
  void release() {
    if (p) cudaFreeHost(p);
    p = nullptr;
    bytes = 0;
  }
  template <class T> T* as() const { return static_cast<T*>(p); }
};

struct Params {
  int64_t npart = 0;
  int32_t nusedpart = 0;
  int32_t nvoisins = 32, nhop = 16, nlevelmax = 30, nmembthresh = 20, nMembers = 20, nbPes = 1;
  double rho_threshold = 80.0, fudge = 4.0, alphap = 1.0, epsilon = 0.0, fudgepsilon = 1e-5;
  double massp = 0, boxsize = 1, boxsize2 = 1, Lf = 1;
  double xlong = 1, ylong = 1, zlong = 1, xlongs2 = 0.5, ylongs2 = 0.5, zlongs2 = 0.5, xyzlong = 1;
  bool verbose = false, megaverbose = false, optimize_nodes = false;
  std::string method = "MSM";
  AhopInit init{};
};

// Node record on the device; same fields as the Fortran `supernode`
// (f90:160-174).
struct NodeRec {
  double rho_saddle, density, densmax, radius, truemass, pos[3];
  int32_t mass, level, mother, firstchild, nsisters, sister;
};

constexpr int kLeaf = 32;         // particles per leaf bucket
constexpr int kFan = 32;          // children per internal node
constexpr int kMaxLevels = 8;
constexpr int kMaxProfiledWaves = 64;
// parts of the small flag block d_flags (512 bytes, cleared before the kNN)
constexpr int kFlagHop = 320;
constexpr int kProfRow = 32;  // int64 entries per structure-tree task-profile row

struct Engine {
  Params prm;
  int device = -1;
  cudaStream_t stream = nullptr;  // stream of the current call
  cudaStream_t stream2 = nullptr; // structure tree: large tasks run here beside the small ones
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
  int tree_cluster = 1;           // CTAs per wide structure-tree task in use (1: no clusters)
  int tree_cluster_req = 4;       // CTAs asked for (debug API: 4 or 1)
  int tree_cluster_for = 0;       // the request tree_cluster was chosen for (0: none yet)
  int tree_par_cap = 0;           // cap on the wide tasks' shared union-find array (0: none; debug API)
  cudaStream_t stream_copy = nullptr;   // host path: density copy-out during the later stages
  cudaEvent_t ev_dens = nullptr, ev_copied = nullptr;
  cudaEvent_t ev_mass = nullptr;        // host path: masses uploaded on the copy stream
  cudaEvent_t ev_posup = nullptr;       // host path: positions uploaded (the masses follow)
  bool mass_pending = false;            // ... and not yet waited for by the compute stream
  cudaEvent_t wave_ev[4] = {};          // per-wave timing (task profile only)
  float wave_prof[4 * 64] = {};         // per wave: small tasks, ms, large tasks, ms
  int32_t nwave_prof = 0;
  int32_t big_task = 512;               // structure-tree tasks above this many groups use wide blocks
  cudaEvent_t ev[16] = {};
  int32_t launches = 0, cub_calls = 0, waves = 0, hop_passes = 0;  // counters of the current compute
  int32_t forest_rounds = 0, forest_edges = 0;                        // saddle forest of the current compute
  unsigned long long tree_stats[11] = {};                             // structure-tree kernel counters
  unsigned long long knn_stats[12] = {};
  unsigned long long knn_phase[5] = {};                              // kNN kernel cycles by phase
  bool events_ready = false;
  AhopTimings timings{};

  int64_t n = 0;          // particles in the current run
  int32_t nstore = 16;    // neighbours stored per particle
  int32_t req_store = 0;  // requested via debug API (0 = nhop)
  bool task_profile = false;  // per-task structure-tree profile (debug API)
  bool have_result = false;
  bool have_groups = false;   // the call's hop targets and groups are there

  // inputs / sorted particle arrays
  DevBuf d_pos_in, d_mass_in;            // staging for host inputs
  // One buffer of 32 bytes per particle: sort keys and permutations, hop targets
  // and roots as sub-arrays (layout_sort); from the sorted gather to the end of
  // the kNN, when none of them is in use, it holds the particles as (x, y, z, m)
  // rows, one sector per gathered particle.
  DevBuf d_sort;
  DevView d_key, d_key2, d_idx, d_idx2;  // sort keys (key and key2 are adjacent), sort values and scratch
  DevView d_hop, d_root;                 // per sorted slot
  cudaError_t layout_sort() {
    const size_t N = ((size_t)n + 1 + 63) / 64 * 64;  // n + 1 entries each, 256-byte boundaries
    const cudaError_t e = d_sort.ensure(32 * N);
    if (e != cudaSuccess) return e;
    char* b = d_sort.as<char>();
    d_key.p = b;
    d_key2.p = b + 8 * N;
    d_idx.p = b + 16 * N;
    d_idx2.p = b + 20 * N;
    d_hop.p = b + 24 * N;
    d_root.p = b + 28 * N;
    return cudaSuccess;
  }
  double4* rows() const { return d_sort.as<double4>(); }
  DevBuf d_x, d_y, d_z, d_m;             // sorted SoA
  DevBuf d_orig;                         // orig index (0-based) per sorted slot
  DevBuf d_rank;                         // sorted slot per orig index
  DevBuf d_box;                          // AABBs of all levels (6 doubles each)
  DevBuf d_box32;                        // AABBs of all levels in FP32, widened (2 float4 each)
  int32_t nlev = 0;
  int64_t lev_off[kMaxLevels + 1] = {};
  int64_t lev_cnt[kMaxLevels] = {};
  CountBuf d_cub;                          // CUB scratch

  // kNN / density
  DevBuf d_nei;                          // [n][nstore] sorted-slot neighbour ids
  DevBuf d_dens;                         // density in sorted order
  // hop / groups
  DevBuf d_group;                        // per sorted slot
  DevBuf d_peakflag;                     // per orig index
  int32_t ngroups = 0;
  CountBuf d_densg;                        // [ngroups+1] peak density per group
  CountBuf d_gpeak;                        // [ngroups+1] sorted slot of peak
  CountBuf d_goff;                         // [ngroups+2] member CSR offsets (desc orig order)
  DevBuf d_gmem;                         // [nactive] sorted slots
  CountBuf d_gmem_rho;                     // [nactive] member density in desc-density order
  CountBuf d_gmem_rho_pref;                // [nactive] prefix sums of density (desc density order)
  int64_t nactive = 0;
  // saddles
  CountBuf d_sad_key, d_sad_key2, d_sad_val, d_sad_val2, d_sad_cnt, d_sad_keep, d_sad_kpos;
  DevBuf d_flags;                        // small device error/status flags
  CountBuf d_soff;                       // final CSR: row offsets,
  int32_t* sisad = nullptr;              // neighbour groups (inside d_sad_key2)
  double* srho = nullptr;                // and saddles (inside d_sad_key)
  int32_t nconn = 0;
  // nodes
  CountBuf d_nodes;                        // NodeRec[nnodesmax+1]
  CountBuf d_tree_scratch;
  CountBuf d_task_sort;                    // wave task ordering scratch
  DevBuf d_tprof;                        // per-task profile rows (debug)
  CountBuf d_forest;                       // saddle-forest scratch
  CountBuf d_moff, d_misad, d_mrho;        // saddle forest CSR (rows by decreasing saddle)
  int32_t* m_isad = nullptr;             // sorted forest rows inside d_misad / d_mrho
  double* m_rho = nullptr;
  CountBuf d_pairs;                        // (node, group) pair keys, sort double buffer
  CountBuf d_pair_sums;                    // [npairs][8] per-pair sums
  CountBuf d_node_aux;                     // per node: pair range, posref
  int32_t nnodes = 0;
  DevBuf d_liste;                        // [n] node id per ORIG particle (1-based), 0 none
  DevBuf d_dens_orig;                    // [n] density in ORIG order; before that the kNN's collected slots
  CountBuf d_rtab, d_itab;                 // exported tables

  // host copies (module outputs), pinned
  HostBuf h_liste, h_itab, h_dens, h_rtab;
  int64_t h_n = 0, h_nused = 0;

  // small pinned host scalars; the last is the kNN's error flag
  int64_t* h_scalars = nullptr;
  static constexpr int kHostScalars = 16;
};

Engine& engine();
void set_error(const std::string& s);

// Stage entry points (return AHOP_* codes).
int stage_sort_and_tree(Engine& E, const double* d_pos_aos, const double* d_mass);
int stage_knn_density(Engine& E);
bool knn_failed(Engine& E);  // after a synchronisation of the stream: the kNN kernels' error, with set_error
int stage_hop_groups(Engine& E);
int stage_saddles(Engine& E);
void saddles_counted(Engine& E);  // after a synchronisation of the stream: sets nconn
int stage_nodes(Engine& E);
void release_adjoint_memory();  // workspaces of the gradients (adjoint.cu)
void release_reader_memory();   // staging of the part-file reader (ramses.cu)
int build_saddle_forest(Engine& E);  // maximum spanning forest of the saddle rows (forest.cu)

}  // namespace ahop

#define AHOP_CUDA_TRY(expr)                                                                      \
  do {                                                                                            \
    cudaError_t _e = (expr);                                                                      \
    if (_e != cudaSuccess) {                                                                      \
      ::ahop::set_error(std::string(#expr) + ": " + cudaGetErrorString(_e) + " at " + __FILE__ + \
                        ":" + std::to_string(__LINE__));                                          \
      return (_e == cudaErrorMemoryAllocation) ? AHOP_ENOMEM : AHOP_ECUDA;                        \
    }                                                                                             \
  } while (0)
