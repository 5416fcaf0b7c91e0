// Plain FP64 first-order density (rho1) and its gradient for plans whose batches
// all have at most SMALL_MAX_NC compute functions and 16-byte aligned phi rows, where
// that is the faster way (rho1_small_build_items; rho1_fp64.cu has the semantics and
// the kernel for everything else; the sums are formed in the same order, so both give
// the same bits).
//
// Such batches are short: the general kernel takes a handful of 32-wide K chunks
// per row tile, each a memory latency behind a barrier, gathers P1c once per 64
// points and reads phi again for every row tile and in the epilogue.  Here a CTA
// (one per SM) gathers the whole P1c of a batch into shared memory once, and its
// two groups of 8 warps run over the batch's points 16 at a time, each with its own
// barrier: one group's epilogue overlaps the other's MMAs.  phi of a group's next
// pass is copied while this one is multiplied, the MMA loop goes through all of K
// without a barrier, the epilogue takes phi from shared memory, and grad phi (read
// once) is loaded into registers before the MMAs.
// Bound: latency (two barriers per pass, one P1c gather per batch), then the FP64
// tensor pipe.
#include <algorithm>
#include <vector>

#include "frpa_internal.cuh"

namespace frpa {
namespace {

constexpr int THREADS = 512, WARPS = THREADS / 32;
constexpr int GROUPS = 2, GW = WARPS / GROUPS;  // groups of 8 warps
constexpr int PTS = 16;                         // points per pass of a group: two 8-point blocks
constexpr int RG = GW;                          // a group's warps go along the 8-row blocks
constexpr int LDW = 2 * 64 + 2;  // W[point][row]: 2 (mod 8) doubles, conflict-free fragment stores
static_assert(SMALL_MAX_NC <= 2 * RG * 8 && PTS == 2 * GW, "two row blocks and two points per warp");

// Leading dimension of the P1c and phi tiles: 4 (mod 16) doubles (conflict-free
// fragment loads), at least nc rounded up to whole 8-row blocks.
__host__ __device__ __forceinline__ int small_ld(int nc) { return ((nc + 7) / 8 * 8 + 11) / 16 * 16 + 4; }
size_t small_smem(int nc_max) {
  const size_t ld = small_ld(nc_max), rows = (nc_max + 3) & ~3;
  return sizeof(double) * (rows * ld + GROUPS * (2 * PTS * ld + PTS * LDW));
}

struct SmallParams {
  const Rho1WorkItem *items;
  int n_items, T, n_active, n_basis, n_full_points, n_max_batch_size, n_batches, nc_max;
  int *counter;
  const int *ib_all, *map;
  const double *wave, *gwave, *P1, *bias, *gbias;
  double *rho, *grad;
};

// The fragments of step ks + 1 are loaded before the MMAs of step ks: with two
// warps per sub-partition nothing else covers a shared-memory load.
template <int CM, int CN>
__device__ __forceinline__ void small_mma(double (&acc)[2][2][2], const double *A, const double *B, int ld, int nks) {
  double a[CM], b[CN];
  auto load = [&](int ks, double (&x)[CM], double (&y)[CN]) {
#pragma unroll
    for (int mi = 0; mi < CM; ++mi) x[mi] = A[ks * 4 * ld + mi * RG * 8];
#pragma unroll
    for (int ni = 0; ni < CN; ++ni) y[ni] = B[ni * 8 * ld + ks * 4];
  };
  load(0, a, b);
#pragma unroll 4
  for (int ks = 0; ks < nks; ++ks) {
    double x[CM], y[CN];
    load(min(ks + 1, nks - 1), x, y);
#pragma unroll
    for (int mi = 0; mi < CM; ++mi)
#pragma unroll
      for (int ni = 0; ni < CN; ++ni) dmma_8x8x4(acc[mi][ni][0], acc[mi][ni][1], a[mi], b[ni]);
#pragma unroll
    for (int mi = 0; mi < CM; ++mi) a[mi] = x[mi];
#pragma unroll
    for (int ni = 0; ni < CN; ++ni) b[ni] = y[ni];
  }
}

// Halves 2 N values over lanes 4 N apart: lanes with that bit keep the upper ones.
template <int N>
__device__ __forceinline__ void fold(double (&v)[8], int lane) {
  const bool upper = (lane & (4 * N)) != 0;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const double keep = upper ? v[i + N] : v[i], give = upper ? v[i] : v[i + N];
    v[i] = keep + __shfl_xor_sync(0xffffffffu, give, 4 * N);
  }
}

__global__ void __launch_bounds__(THREADS, 1) rho1_small_kernel(const SmallParams P) {
  extern __shared__ __align__(16) double smem[];
  __shared__ int s_ib[SMALL_MAX_NC], s_next;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int group = warp / GW, gw = warp % GW;  // gw: this warp's pair of points in the epilogue
  // first of its row blocks: the second group starts two sub-partitions further, so
  // that the blocks left over by rounds of 8 fall on different tensor pipes
  const int rb = (gw + 2 * group) % RG;
  const int g = lane >> 2, q = lane & 3;
  const int ld = small_ld(P.nc_max);
  // As[k][m]; per group Bs[2][n][k] and Ws[n][m]
  double *As = smem, *Bs = As + ((P.nc_max + 3) & ~3) * ld + group * (2 * PTS * ld + PTS * LDW);
  double *Ws = Bs + 2 * PTS * ld;
  auto group_sync = [&] { asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(32 * GW) : "memory"); };
  const long long nb2 = (long long)P.n_basis * P.n_basis;

  grid_wait();  // the cleared outputs and cursor
  for (int it = blockIdx.x; it < P.n_items;) {
    const Rho1WorkItem W = P.items[it];
    const int nc = W.nc, ncp = (nc + 3) & ~3, nb = (nc + 7) / 8, nMt = (nc + 63) / 64;
    const int passes = (W.pn + PTS - 1) / PTS;
    const int cm = (nb - rb + RG - 1) / RG;  // this warp's row blocks (0..2)
    if (tid == 0) s_next = (int)gridDim.x + atomicAdd(P.counter, 1);
    if (tid < nc) s_ib[tid] = __ldg(P.ib_all + W.ib_off + tid) - 1;
    const double *phi = P.wave + W.wave_off + (long long)W.p0 * ncp;
    const double *gph = P.gwave + 3 * W.wave_off + 3LL * W.p0 * ncp;
    // phi of pass j into buffer `buf`: warp -> points, lanes -> 16-byte pieces of a row; zero past n_compute
    auto load_phi = [&](int j, int buf) {
      double *B = Bs + buf * PTS * ld;
      const int left = W.pn - j * PTS;
#pragma unroll
      for (int r = 0; r < PTS / GW; ++r) {
        const int n = gw + r * GW;
        if (n >= left) break;
        const double *row = phi + (long long)(j * PTS + n) * ncp;
        for (int k = 2 * lane; k < ncp; k += 64) {
          const int bytes = k + 1 < nc ? 16 : (k < nc ? 8 : 0);
          cp_async_16(B + n * ld + k, bytes ? row + k : row, bytes);
        }
      }
    };
    for (int t = 0; t < P.T; ++t) {
      __syncthreads();  // the list is there; the last perturbation's (or item's) tiles are consumed
      {
        // P1c(i, k) = P1(ib_i, ib_k): warp -> columns k, lanes -> rows; zero up to whole blocks
        const double *P1t = P.P1 + t * nb2;
        for (int k = warp; k < ncp; k += WARPS) {
          const double *col = P1t + (long long)s_ib[k < nc ? k : 0] * P.n_basis;
          for (int m = lane; m < nb * 8; m += 32) {
            const bool ok = m < nc && k < nc;
            cp_async_8(As + k * ld + m, ok ? col + s_ib[m] : P1t, ok ? 8 : 0);
          }
        }
      }
      if (group < passes) load_phi(group, 0);
      cp_async_commit();
      cp_async_wait<0>();
      __syncthreads();  // all of P1c is there
      for (int j = group, buf = 0; j < passes; j += GROUPS, buf ^= 1) {
        const int left = min(PTS, W.pn - j * PTS);
        // this warp's two points of the pass: grad phi rows, bias and map entries
        const int p_warp = 2 * gw;
        double2 gx[2][3];  // [point][component], of one 64-row tile
        auto load_grad = [&](int mt) {
          const int r0 = mt * 64 + 2 * lane;
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const double *src = gph + 3LL * (j * PTS + p_warp + i) * ncp + r0;
#pragma unroll
            for (int c = 0; c < 3; ++c)
              gx[i][c] = r0 < ncp && p_warp + i < left ? __ldg(reinterpret_cast<const double2 *>(src + c * ncp))
                                                       : make_double2(0.0, 0.0);
          }
        };
        load_grad(0);
        // after the sums lane 4 (2 c + i) holds component c of point i
        const int c_out = lane >> 3, p_out = p_warp + (lane >> 2 & 1);
        const bool out = (lane & 3) == 0 && p_out < left;
        const int pp = W.p0 + j * PTS + p_out;
        const long long bidx = pp + (long long)P.n_max_batch_size * (W.batch + (long long)P.n_batches * t);
        double offset = 0.0;
        int full = 0;
        if (out) {
          offset = c_out == 0 ? __ldg(P.bias + bidx) : __ldg(P.gbias + 3 * bidx + c_out - 1);
          if (c_out == 0) full = __ldg(P.map + W.prefix + pp);
        }
        cp_async_wait<0>();
        group_sync();  // phi of this pass is there; the group is done with its last pass
        if (j + GROUPS < passes) load_phi(j + GROUPS, buf ^ 1);
        cp_async_commit();
        const double *B = Bs + buf * PTS * ld;
        double acc[2][2][2] = {};
        const int cn = left > 8 ? 2 : 1;  // point blocks
        const double *a0 = As + q * ld + rb * 8 + g, *b0 = B + g * ld + q;
        if (cm == 2 && cn == 2)
          small_mma<2, 2>(acc, a0, b0, ld, ncp / 4);
        else if (cm == 2 && cn == 1)
          small_mma<2, 1>(acc, a0, b0, ld, ncp / 4);
        else if (cm == 1 && cn == 2)
          small_mma<1, 2>(acc, a0, b0, ld, ncp / 4);
        else if (cm == 1 && cn == 1)
          small_mma<1, 1>(acc, a0, b0, ld, ncp / 4);
#pragma unroll
        for (int mi = 0; mi < 2; ++mi)
          if (mi < cm) {
#pragma unroll
            for (int ni = 0; ni < 2; ++ni)
#pragma unroll
              for (int h = 0; h < 2; ++h)
                Ws[(ni * 8 + 2 * q + h) * LDW + (mi * RG + rb) * 8 + g] = acc[mi][ni][h];
          }
        group_sync();
        // Two points per warp: lane l takes rows 2 l, 2 l + 1 of each 64-row tile; the
        // eight sums (component, point) go over the lanes, the tiles in order.
        double tot = 0.0;
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) {
          if (mt >= nMt) break;
          const int r0 = mt * 64 + 2 * lane;
          const bool in_block = r0 < ncp, ok0 = r0 < nc, ok1 = r0 + 1 < nc;
          double v[8];
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int p = p_warp + i;
            const bool live = in_block && p < left;
            double2 w = make_double2(0.0, 0.0), f = w;
            if (live) {
              w = *reinterpret_cast<const double2 *>(Ws + p * LDW + r0);
              f = *reinterpret_cast<const double2 *>(B + p * ld + r0);
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const double2 x = c == 0 ? f : gx[i][c > 0 ? c - 1 : 0];
              v[2 * c + i] = live ? fma(ok1 ? x.y : 0.0, w.y, (ok0 ? x.x : 0.0) * w.x) : 0.0;
            }
          }
          if (mt == 0 && nMt > 1) load_grad(1);
          fold<4>(v, lane);
          fold<2>(v, lane);
          fold<1>(v, lane);
          v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
          v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
          tot += v[0];
        }
        if (out) {
          if (c_out > 0)
            P.grad[3 * bidx + c_out - 1] = tot * 2 - offset;
          else if (t < P.n_active)
            P.rho[full + (long long)P.n_full_points * t] = tot + offset;
        }
      }
    }
    it = s_next;      // written before the first barrier
    __syncthreads();  // read by everyone before the next item's first thread writes it
  }
}

}  // namespace

constexpr int STEP = GROUPS * PTS;  // points of a pass of both groups

namespace {

// The time of a persistent launch over items on `slots` SMs (or halves of one): with
// no more items than slots the longest, else the mean load of a slot and part of the
// longest item at the end.
struct LaunchTime {
  double sum = 0.0, longest = 0.0;
  long long n = 0;
  void add(long long count, double item) {
    n += count;
    sum += count * item;
    longest = std::max(longest, item);
  }
  double total(int slots, double tail) const {
    return n <= slots ? longest : std::max(longest, sum / slots + tail * longest);
  }
};

// Times in microseconds of an item's parts, fitted to both kernels' launches on 453
// plans (4 to 6,000 batches of 1 to 120 functions and 4 to 1,000 points, some with one
// batch of 2,000 or 20,000, one to four perturbations; rms error 9% each).  `cold` is
// 1 where the arrays are much larger than L2 and goes to 0 with their size.
//
// This kernel: the item's start, and per perturbation the P1c gather and `steps`
// passes of both groups (a batch of at most 16 points is one pass of one group).
double item_time(int nc, int np, int T, int steps, double cold) {
  const double nc2 = (double)nc * nc, pass = (1.39 * (1.0 + 0.34 * cold) + 4.2e-4 * nc2) * (np <= PTS ? 0.58 : 1.0);
  return 1.05 + T * (0.67 + 2.4e-4 * nc2 + steps * pass);
}
// The general kernel: an item of at most 64 points, two CTAs per SM.
double general_item_time(int nc, double points, int T, double cold) {
  const int row_tiles = ceil_div(nc, 64);
  return 0.46 + row_tiles * (4.75 * cold * (1.0 + 0.37 * (T - 1)) +
                             T * (3.04 + 0.6 * (nc / 32.0 + 0.33) + 0.0039 * points)) +
         T * 1.17e-5 * points * nc * nc;
}
// A batch as the search for the limit sees it: time of a part = start + step x its steps.
struct BatchTime {
  int steps;
  double start, step;
  BatchTime(const Rho1WorkItem &b, int T, double cold)
      : steps(ceil_div(b.np, STEP)),
        start(item_time(b.nc, b.np, T, 0, cold)),
        step(item_time(b.nc, b.np, T, 1, cold) - start) {}
  // the fewest parts whose time is at most `limit`
  int parts(double limit) const {
    if (start + step * steps <= limit) return 1;
    return ceil_div(steps, std::max(1, (int)((limit - start) / step)));
  }
};

}  // namespace

// Work items: every batch in equal parts of at most a time limit, the limit that makes
// the launch shortest (none, where the batches are many and alike).  Few items are
// taken largest first.
// use 0: no items, so that the general kernel is taken, where that one's launch is
// shorter; 1: none; 2: always.  Which one is depends on how often P1c is gathered (per
// item here, per 64 points there) and on what covers a gather (nothing here, the SM's
// other CTA there).  Measured, us, general kernel / this one: 64 batches of 40-120
// functions, 100-200 points 22 / 13 (148: 35 / 35 of 20-120; 2,000: 403 / 364);
// 2,000 batches of 110-120 functions, 60-64 points 256 / 304, 8-16 points 159 / 142;
// 600 batches of 16-24 functions, 250-400 points, four perturbations 309 / 385.  On the
// 453 plans the choice costs 0.2% of the better kernel's time in the mean, 15% at most.
void rho1_small_build_items(const std::vector<Rho1WorkItem> &batches, int T, int n_sm, int order, int use,
                            std::vector<Rho1WorkItem> *out) {
  out->clear();
  if (use == 1) return;
  double bytes = 0.0;  // phi and grad phi, biases and grad rho1
  int np_max = 0;
  for (const Rho1WorkItem &b : batches) {
    bytes += 32.0 * ((b.nc + 3) & ~3) * b.np;
    np_max = std::max(np_max, b.np);
  }
  bytes += 64.0 * T * np_max * batches.size();
  const double cold = std::min(1.0, bytes / 1e8);
  std::vector<BatchTime> times;
  times.reserve(batches.size());
  for (const Rho1WorkItem &b : batches)
    if (b.np > 0) times.emplace_back(b, T, cold);
  double limit = 1e30, best = 1e30;
  for (double l = 5.0; l < 1e9; l *= 1.4) {
    LaunchTime launch;
    bool cut = false;
    for (const BatchTime &b : times) {
      const int parts = b.parts(l);
      cut = cut || parts > 1;
      launch.add(parts, b.start + b.step * (parts == 1 ? b.steps : ceil_div(b.steps, parts)));
    }
    const double t = 2.2 + launch.total(n_sm, 0.44);
    if (t < best) {
      best = t;
      limit = l;
    }
    if (!cut) break;
  }
  if (use == 0) {
    LaunchTime general;
    for (const Rho1WorkItem &b : batches) {
      const int tiles = ceil_div(b.np, 64);
      if (tiles > 0) general.add(tiles, general_item_time(b.nc, (double)b.np / tiles, T, cold));
    }
    if (best > 1.03 * (3.6 + general.total(2 * n_sm, 0.68))) return;
  }
  size_t at = 0;
  for (const Rho1WorkItem &b : batches) {
    if (b.np == 0) continue;
    const int steps = ceil_div(b.np, STEP), parts = times[at++].parts(limit);
    for (int k = 0, p0 = 0; k < parts; ++k) {  // the 32-point steps dealt out evenly
      const int w = STEP * (steps / parts + (k < steps % parts ? 1 : 0));
      out->push_back(Rho1WorkItem{b.batch, b.nc, b.np, p0, std::min(w, b.np - p0), b.ib_off, b.prefix, b.key,
                                  b.wave_off});
      p0 += w;
    }
  }
  rho1_order_items(out, (long long)out->size() <= 4LL * n_sm ? 0 : order);
}

// Shared-memory attribute of the kernel, once per device (outside any capture).
int rho1_small_configure(int device) {
  static PerDeviceOnce configured;
  return configured.run(device, []() -> int {
    FRPA_CUDA_TRY(cudaFuncSetAttribute(rho1_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)small_smem(SMALL_MAX_NC)));
    return FRPA_OK;
  });
}

// The whole plan; the cursor must be zero.
int rho1_small_launch(const Rho1Plan &plan, int n_active, const double *wave, const double *gwave, const double *P1,
                      const double *bias, const double *gbias, double *rho, double *grad, cudaStream_t stream) {
  int n_sm = 148;
  FRPA_CUDA_TRY(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, plan.device));
  const SmallParams P{plan.d_items_small, plan.n_items_small, plan.T, n_active, plan.n_basis, plan.n_full_points,
                      plan.n_max_batch_size, plan.n_batches, plan.n_max_compute, plan.d_counter, plan.d_ib, plan.d_map,
                      wave, gwave, P1, bias, gbias, rho, grad};
  FRPA_CUDA_TRY(launch_chained(rho1_small_kernel, std::min(n_sm, plan.n_items_small), THREADS,
                               small_smem(plan.n_max_compute), stream, P));
  FRPA_LAUNCH_CHECK();
  return FRPA_OK;
}

}  // namespace frpa
