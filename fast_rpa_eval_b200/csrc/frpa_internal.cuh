// Internal helpers shared by the frpa CUDA sources (not part of the C ABI).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "frpa.h"

namespace frpa {

// ---------------------------------------------------------------- errors --

// Records a failure for frpa_last_error()/frpa_last_error_message() and
// returns the status so callers can `return fail(...)`.
int fail(int status, const char *fmt, ...);
void clear_error();

#define FRPA_CUDA_TRY(call)                                                                      \
  do {                                                                                           \
    cudaError_t e_ = (call);                                                                     \
    if (e_ != cudaSuccess)                                                                       \
      return ::frpa::fail(FRPA_ERR_CUDA, "%s:%d: %s: %s", __FILE__, __LINE__, #call,             \
                          cudaGetErrorString(e_));                                               \
  } while (0)

#define FRPA_CHECK_ARG(cond, ...)                                                                \
  do {                                                                                           \
    if (!(cond)) return ::frpa::fail(FRPA_ERR_INVALID, __VA_ARGS__);                             \
  } while (0)

#define FRPA_TRY(call)                                                                           \
  do {                                                                                           \
    int s_ = (call);                                                                             \
    if (s_ != FRPA_OK) return s_;                                                                \
  } while (0)

// Launch-time check: configuration errors surface here, execution errors at
// the next synchronising call.
#define FRPA_LAUNCH_CHECK() FRPA_CUDA_TRY(cudaGetLastError())

// One-time setup per device (kernel attributes, constant-memory uploads) that
// several host threads may reach at the same time: `fn` runs under a lock and
// is retried by the next caller until it has succeeded once for `device`.
class PerDeviceOnce {
 public:
  template <class F>
  int run(int device, F &&fn) {
    std::lock_guard<std::mutex> lk(mu_);
    if (device >= 0 && device < 64 && done_[device]) return FRPA_OK;
    const int st = fn();
    if (st == FRPA_OK && device >= 0 && device < 64) done_[device] = true;
    return st;
  }

 private:
  std::mutex mu_;
  bool done_[64] = {};
};

// ------------------------------------------------------------ device math --

// Exactly rounded product and sum (no FMA contraction), used wherever the
// reference's x86-64 arithmetic decides a branch (dist^2 vs radii).
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub_rn(double a, double b) { return __dsub_rn(a, b); }

// 64-bit FP tensor-core MMA, m8n8k4 (A row-major 8x4, B col-major 4x8).
// Fragments: a = A[lane>>2][lane&3], b = B[lane&3][lane>>2],
// c/d = C[lane>>2][2*(lane&3) + {0,1}].
__device__ __forceinline__ void dmma_8x8x4(double &d0, double &d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// cp.async with zero fill: copies `src_bytes` (0 or the full size) and
// zero-fills the rest of the destination.
__device__ __forceinline__ void cp_async_8(void *smem_dst, const void *gmem_src, int src_bytes) {
  unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem_dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(gmem_src), "r"(src_bytes));
}
__device__ __forceinline__ void cp_async_16(void *smem_dst, const void *gmem_src, int src_bytes) {
  unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem_dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem_src), "r"(src_bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

inline int ceil_div(int a, int b) { return (a + b - 1) / b; }
inline long long ceil_div_ll(long long a, long long b) { return (a + b - 1) / b; }

// ---------------------------------------------------------- plan memory --

// A plan's device memory, one allocation: arrays up to 256 KiB go up in one
// copy, larger ones each from where they are (their sources have to live until
// commit), workspaces are left as they come.  (One allocation and copy per array
// made creating a small plan mostly driver calls.  Above about 1.2 MB the driver maps
// memory for an allocation, 0.6 ms with its release: a sum-up plan of 30 centres and
// 20,000 points, whose arrays one by one came from its pools, takes 2.2 ms for 1.8; of
// 64 points 0.06 for 0.29, of 50,000 points 4.8 for 5.0.)
struct PlanMemory {
  static constexpr size_t STAGED = 256 << 10;
  struct Part {
    void **dst;
    const void *src;  // nullptr: staged
    size_t off, bytes;
  };
  std::vector<Part> staged, tail;
  std::vector<unsigned char> host;
  size_t tail_bytes = 0;

  static size_t padded(size_t n) { return (std::max<size_t>(n, 8) + 255) / 256 * 256; }
  void array(void **dst, const void *src, size_t bytes) {
    if (bytes > STAGED) {
      tail.push_back({dst, src, tail_bytes, bytes});
      tail_bytes += padded(bytes);
      return;
    }
    staged.push_back({dst, nullptr, host.size(), bytes});
    host.resize(host.size() + padded(bytes));
    if (bytes) memcpy(host.data() + staged.back().off, src, bytes);
  }
  void space(void **dst, size_t bytes) {
    tail.push_back({dst, nullptr, tail_bytes, bytes});
    tail_bytes += padded(bytes);
  }
  size_t total() const { return padded(host.size() + tail_bytes); }
  // into *base, allocated here unless it is already there (with total() bytes)
  int commit(unsigned char **base, size_t *bytes) {
    *bytes = total();
    if (!*base && cudaMalloc((void **)base, *bytes) != cudaSuccess) {
      *base = nullptr;
      return fail(FRPA_ERR_OOM, "plan: allocation of %zu bytes failed", *bytes);
    }
    for (const Part &p : staged) *p.dst = *base + p.off;
    for (const Part &p : tail) *p.dst = *base + host.size() + p.off;
    if (!host.empty()) FRPA_CUDA_TRY(cudaMemcpy(*base, host.data(), host.size(), cudaMemcpyHostToDevice));
    for (const Part &p : tail)
      if (p.src) FRPA_CUDA_TRY(cudaMemcpy(*p.dst, p.src, p.bytes, cudaMemcpyHostToDevice));
    return FRPA_OK;
  }
};

// ------------------------------------------------------------ rho1 plan --

// One unit of rho1 work: a point tile of one non-empty grid batch
// (the reference's valid-batch list, device_data.cu:242-260, refined into
// point tiles and ordered by decreasing cost for the persistent scheduler).
struct Rho1WorkItem {
  int batch;         // index into the caller's batch arrays
  int nc;            // n_compute_c of the batch
  int np;            // points in the batch
  int p0;            // first point of this tile
  int pn;            // points in this tile
  int ib_off;        // offset of the batch's basis list in the compact list
  int prefix;        // n_point_batches_prefix_sum[batch]
  int key;           // locality key: MinHash of the batch's basis functions
  long long wave_off;  // i_batch_2_wave_offset[batch]
};
static_assert(sizeof(Rho1WorkItem) == 40, "work item layout");

// Split-int8 rho1 (rho1_split_i8.cu).  A work item is a point tile of one
// batch; its phi digits live in the A scratch, the batch's P1c digits (per
// perturbation) in the B scratch.  Offsets are relative to the scratch of
// the item's group: groups of consecutive batches are packed and contracted
// in turn, so the scratch holds one group at a time.
struct I8Item {
  int batch, nc, p0, pn;
  int prefix, rows8, n_nt, n_kc;  // rows8 = pn rounded up to 8; N tiles of 32 rows; K chunks of 32
  long long wave_off;
  long long a_off;       // bytes of the item's first A chunk
  long long b_off;       // bytes of the batch's first B chunk (t = 0)
  long long b_tstride;   // B bytes per perturbation
  int sa_off;            // first per-point scale of the item
  int sb_off;            // first per-row scale of the batch (t = 0)
  int sb_tstride;        // per-row scales per perturbation (n_nt * 32)
  int pad_;
};
static_assert(sizeof(I8Item) == 80, "I8Item layout");

// One N tile of one batch and perturbation, packed by one CTA.
struct I8BTile {
  int ib_off, nc, jn, t;
  int n_kc, sb_off;  // K chunks; first per-row scale of the tile
  long long b_off;                 // bytes of the tile's first chunk
};
static_assert(sizeof(I8BTile) == 32, "I8BTile layout");

struct I8Group {
  int item0, item1;   // items [item0, item1)
  int tile0, tile1;   // B tiles [tile0, tile1)
  long long a_bytes, b_bytes;
  int sa_len, sb_len;
};

// Adjoint / first-order H: ranges of the work lists for a group of batches: its
// batches, and its (i, j) tiles, the n_upper of them with j >= i first.
struct H1Group {
  int first, n_first, tiles, n_tiles, n_upper;
};

struct Rho1Plan {
  int device = 0;
  // one allocation holds the arrays made with the plan; a list replaced later
  // (a tuning) has its own
  unsigned char *arena = nullptr;
  size_t arena_bytes = 0;
  void release(void *p) const {
    const unsigned char *c = static_cast<const unsigned char *>(p);
    if (c && (c < arena || c >= arena + arena_bytes)) cudaFree(p);
  }
  int T = 1;
  int n_batches = 0;
  int n_full_points = 0;
  int n_basis = 0;
  int n_max_batch_size = 0;
  int n_max_compute = 0;
  long long wave_len = 0;
  int n_items = 0;
  int n_valid_batches = 0;
  long long n_valid_points = 0;  // points in batches with n_compute > 0
  int wave_aligned16 = 0;        // every batch offset even -> 16-byte loads
  // device copies
  Rho1WorkItem *d_items = nullptr;
  int *d_ib = nullptr;        // compact 1-based basis lists
  int *d_map = nullptr;       // i_valid_point_2_i_full_points_map
  int *d_counter = nullptr;   // persistent scheduler cursor
  int grid_fp64 = 0;
  // plans whose batches have at most SMALL_MAX_NC functions: the list of
  // rho1_fp64_small.cu (empty otherwise, and where the general kernel is taken)
  Rho1WorkItem *d_items_small = nullptr;
  int n_items_small = 0;
  // adjoint and first-order H: work list in groups (first_order_h.cu), built
  // with the plan, and the scratch that the first call allocates: fixed-point
  // accumulator (zero between calls while h1_clean) and A of one group
  void *d_h1_items = nullptr, *d_h1_tiles = nullptr;
  long long h1_budget = 512LL << 20;  // bytes of A per group
  std::vector<H1Group> h1_groups;
  long long h1_a_len = 0;
  int h1_at_once = 1;  // perturbations per launch (the scratch holds A of each)
  double *h1_a = nullptr;       // A: behind the accumulator, or a buffer lent by the caller
  double *h1_a_lent = nullptr;  // (the host-array entry, which makes a plan per call)
  size_t h1_a_lent_bytes = 0;
  bool h1_clean = false;
  unsigned long long *d_h1_acc = nullptr;
  // split-BF16 path: <= 128-point tiles, per-row P1 scales, device error flags
  Rho1WorkItem *d_items_split = nullptr;
  int n_items_split = 0;
  double *d_rowmax = nullptr;
  int *d_err = nullptr;
  // tunings (frpa_rho1_plan_set_tuning) and the host copy of the valid
  // batches the work lists are rebuilt from (one item per batch, p0 = 0)
  int fp64_tile_points = 64;   // 64 or 128 points per FP64 work item
  int fp64_ctas_per_sm = 0;    // 0: as many as fit
  int split_tile_points = 128; // <= 128 points per split-BF16 work item
  int fp64_small = 0;          // kernel for small batches: 0 by estimated time, 1 never, 2 always
  int order = 2;               // 0: largest items first, 1: batch order, 2: locality key
  // the FP64 work list in FP64_CHUNKS pieces of consecutive batches (6%, 44%,
  // 44%, 6% of the cost): chunk c holds items [fp64_chunk_items[c], fp64_chunk_items[c + 1])
  // of batches [fp64_chunk_batches[c], fp64_chunk_batches[c + 1]), so the
  // host-buffer entry point can overlap copies with compute chunk by chunk
  std::vector<int> fp64_chunk_items, fp64_chunk_batches;
  std::vector<Rho1WorkItem> h_batches;
  std::vector<int> h_ib;  // host copy of the compact basis lists
  // split-int8 path: work lists (built with the plan) and the scratch
  // (allocated by the first split-int8 execution, reused afterwards)
  I8Item *d_i8_items = nullptr;
  I8BTile *d_i8_tiles = nullptr;
  std::vector<I8Group> i8_groups;
  long long i8_budget = 4LL << 30;  // bytes of A + B scratch per group
  int i8_wave4 = 0;                  // every batch's phi offset a multiple of 4 doubles
  // two scratch sets: group g is packed into set g % 2 on a side stream while
  // group g - 1 is contracted on the caller's stream
  unsigned char *d_i8_a[2] = {nullptr, nullptr}, *d_i8_b[2] = {nullptr, nullptr};
  double *d_i8_sa[2] = {nullptr, nullptr}, *d_i8_sb[2] = {nullptr, nullptr};
  cudaStream_t i8_side = nullptr;
  cudaEvent_t i8_ev_start = nullptr, i8_ev_packed[2] = {nullptr, nullptr}, i8_ev_done[2] = {nullptr, nullptr};
};

// Work lists of a plan's valid batches (one entry per batch in `batches`).
// work-list order (0 largest first, 1 batch order, 2 locality key) and the key
void rho1_order_items(std::vector<Rho1WorkItem> *items, int order);
int rho1_locality_key(const int *ib, int nc);
constexpr int FP64_CHUNKS = 4;
// FP64 work items, chunk by chunk (FP64_CHUNKS ranges of consecutive batches
// holding 6%, 44%, 44% and 6% of the cost, n_batches = the caller's batch
// count), each chunk in the given order; the chunk boundaries go to
// chunk_items / chunk_batches
void rho1_fp64_build_items(const std::vector<Rho1WorkItem> &batches, int tile_points, int order, int n_batches,
                           std::vector<Rho1WorkItem> *out, std::vector<int> *chunk_items,
                           std::vector<int> *chunk_batches);

int rho1_fp64_launch(const Rho1Plan &plan, int n_active, const double *wave, const double *gwave,
                     const double *P1, const double *bias, const double *gbias, double *rho, double *grad,
                     cudaStream_t stream);
// The FP64 kernel over the items of one chunk only, without zeroing the
// outputs (the caller zeroes them once before the first chunk).
int rho1_fp64_launch_chunk(const Rho1Plan &plan, int chunk, int n_active, const double *wave, const double *gwave,
                           const double *P1, const double *bias, const double *gbias, double *rho, double *grad,
                           cudaStream_t stream);
int rho1_fp64_grid(int device);
constexpr int SMALL_MAX_NC = 120;  // P1c, two phi tiles and a work1 tile fit one SM's shared memory
void rho1_small_build_items(const std::vector<Rho1WorkItem> &batches, int T, int n_sm, int order, int use,
                            std::vector<Rho1WorkItem> *out);
int rho1_small_configure(int device);
int rho1_small_launch(const Rho1Plan &plan, int n_active, const double *wave, const double *gwave, const double *P1,
                      const double *bias, const double *gbias, double *rho, double *grad, cudaStream_t stream);
int rho1_fp64_fused_bias_launch(const Rho1Plan &plan, int n_active, int n_atoms, int j_atom_begin, int j_coord,
                                const int *atom_valid, const double *density_matrix, const double *wave,
                                const double *gwave, const double *P1, const double *bias, const double *gbias,
                                double *rho, double *grad, cudaStream_t stream);
int rho1_split_launch(const Rho1Plan &plan, int n_active, const double *wave, const double *gwave,
                      const double *P1, const double *bias, const double *gbias, double *rho, double *grad,
                      cudaStream_t stream);
void rho1_split_build_items(const std::vector<Rho1WorkItem> &batches, int tile_points, int order,
                            std::vector<Rho1WorkItem> *out);

int p1_rowmax_launch(const Rho1Plan &plan, const double *P1, cudaStream_t stream);
int rho1_i8_build(Rho1Plan *plan);  // work lists and groups from plan->h_batches
void rho1_i8_free(Rho1Plan *plan);
int rho1_i8_launch(Rho1Plan &plan, int n_active, const double *wave, const double *gwave, const double *P1,
                   const double *bias, const double *gbias, double *rho, double *grad, cudaStream_t stream);

int synth_p1_window(const int *gidx, int n, int T, double scale, unsigned long long seed, double *out,
                    cudaStream_t stream);
int rho1_bias_part2_launch(const Rho1Plan &plan, const int *h_atom_valid, const int *d_atom_valid, int n_atoms,
                           int j_atom_begin, int j_atom_end, int j_coord, int T, const double *wave,
                           const double *gwave, const double *dm, double *bias, cudaStream_t stream);
// First-order H and the rho1 adjoint (first_order_h.cu): deterministic
// fixed-point accumulation into an (n_basis, n_basis, T) output.
void rho1_h1_build_items(const std::vector<Rho1WorkItem> &batches, long long budget, std::vector<unsigned char> *items,
                         std::vector<unsigned char> *tile_list, std::vector<H1Group> *groups, long long *a_len);
int rho1_h1_rebuild(Rho1Plan *plan, long long budget);
size_t rho1_h1_a_bytes(Rho1Plan &plan);
int rho1_adjoint_run(Rho1Plan &plan, int n_active, const double *wave, const double *gwave, const double *g_rho,
                     const double *g_grad, double *dP1, cudaStream_t stream);
int rho1_first_order_h_run(Rho1Plan &plan, int n_active, int n_atoms, int j_atom_begin, int j_coord,
                           const int *atom_valid, const double *wave, const double *gwave, const double *hwave,
                           const double *vsigma, const double *gradient_rho, const double *H_prefactor1,
                           const double *fogr, const double *vhg, const double *rho1, const double *v2rho2,
                           const double *v2rhosigma, const double *v2sigma2, const double *partition_tab,
                           double *first_order_H, cudaStream_t stream);

// ----------------------------------------------------------- sum-up plan --

struct SumupPlan;  // defined in sumup.cu

// Launches a kernel that may start while its predecessor in the stream is still
// running: it calls grid_wait() before it touches anything the predecessor
// writes (or that its own outputs' readers may still use), and the predecessor
// calls grid_release() when its dependents may come in.  Arrays that another
// launch of the chain writes are not `__restrict__` here: the qualifier says that
// nothing else changes them while the kernel runs, which would let the compiler
// read them before grid_wait() or through the read-only path.  The start-up of small
// launches overlaps that way: the sum-up of 2,000 points, 20 atoms (three
// launches) 32.5 -> 26.6 us, rho1 of 64 batches of 40-120 functions (two) 32.6 ->
// 29.7 us.  The chain's first launch is an ordinary one, so everything queued
// before it is complete.
template <class... K, class... A>
cudaError_t launch_chained(void (*kernel)(K...), dim3 grid, int threads, size_t smem, cudaStream_t stream, A... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, K(args)...);
}
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

}  // namespace frpa
