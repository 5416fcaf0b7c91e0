// The first-order H integration and the adjoint of rho1 with respect to P1,
// one engine for both: per batch and perturbation t, a contraction over the
// batch's points of a per-point combination A(i, p) of phi, grad phi and the
// Hessian of phi with phi itself, scattered into an (n_basis, n_basis, T)
// matrix through the batch's compute-function list.
//
// First-order H (fast_rap_src_dfpt_gpu_eval/evaluate_first_order_H.cpp:77-215):
//   A(i, p) = cs1(i, p) = c_phi(p) phi_i + sum_k c_grad_k(p) d_k phi_i
//             + [i in atom j's range] sum_k c_hess_k(p) hess_i(k, j_coord),
//   c_phi = (H_prefactor1 + pf3) / 2, c_grad = pf2, c_hess = -pf5 with the
//   reference's per-point prefactors (:144-168), and
//   H(ib_i, ib_j, t) += sum_p A(i, p) phi_j(p) + phi_i(p) A(j, p)
//   (its rank-2k update and symmetric scatter, :192-215).
// Adjoint of rho1 (evaluate_first_order_rho.cpp:149-207):
//   A(i, p) = g_rho(map p, t) phi_i + 2 sum_d g_grad(d, p, b, t) d_d phi_i,
//   dP1(ib_i, ib_j, t) += sum_p A(i, p) phi_j(p).
// With g_rho = w v and no g_grad the adjoint is the first-order H with every
// exchange-correlation term zero.
//
// Work, two passes, over all perturbations at once where their scratch allows.  The
// first is bound by memory: it reads phi, grad phi (and the Hessian rows of atom j)
// once, writes A in phi's layout to a scratch array and finds the bound of the
// contributions that fixes the accumulation's scale (below), which needs a pass over
// the inputs anyway.  The second is one CTA per (i, j) tile of at most 64 x 64 of one
// batch: a plain product of A and phi on the FP64 MMA (mma.sync m8n8k4, the only FP64
// tensor instruction of sm_100a), both streamed by asynchronous copies three or four
// stages of 16 points ahead, because batches are small (tens to some hundred
// functions) and what counts is latency.  A batch's rows are split evenly into
// tiles whose widths are multiples of 8, and the 8-row blocks of a tile go round
// the warps, so that a narrow tile loads all four tensor pipes.  The symmetric H
// computes the tiles with j >= i only, each from both products.  Where A would
// take more than the plan's budget (512 MiB, less where that cannot be allocated),
// the first pass only finds the bound, and groups of batches that fit are then
// combined and multiplied in turn.  Measured, 1,600 batches of 100-200 points,
// n_compute 40-120, n_basis 4,000 (one B200): first-order H 1.60 ms (A rebuilt in
// every tile from synchronous loads, 128-bit sums with a carry) -> 0.60 ms; adjoint
// 1.21 -> 0.43 ms, of it first pass 0.16 (60% of the HBM bandwidth), tiles 0.22,
// last pass 0.05.
//
// Determinism.  Batches overlap in the output, so tiles of different batches
// add into the same entries.  Every contribution is added as a 100-bit
// fixed-point integer held in two 64-bit words of one 16-byte entry (a high and
// a low part, both signed, each summed with its own no-return atomic: the low
// word has room for the sum over every batch, so no carry and no wait for
// another thread's sum; both parts come from the addition of 1.5 2^52, which
// leaves an integer in the mantissa), and integer addition does not depend
// on the order: two runs give bit-identical results.  The fixed-point scale 2^s
// is fixed per call before any addition from a bound of the inputs (a pass over
// phi, grad phi, Hessian and the per-point coefficients): every single
// contribution is below 2^emax, at most 2 n_batches contributions meet in one
// entry, so with s = 100 - emax - ceil(log2(2 n_batches)) every partial sum
// stays below 2^100 and each contribution is represented to 2^-s, about 2^-80
// of the largest one.  A last pass converts each entry to FP64 (one rounding),
// adds it to the output and leaves the accumulator zero for the next call.
#include <climits>
#include <cstring>
#include <vector>

#include "frpa_internal.cuh"

namespace frpa {
namespace {

constexpr int TILE = 64, KC = 16, THREADS = 256;
constexpr int LD = TILE + 4;  // [k = point][row]: stride = 4 (mod 16) doubles, conflict-free fragment loads
constexpr int EMAX_EMPTY = -2139062144;  // 0x80808080: no non-zero bound seen
constexpr int H1_FLAG_NONFINITE = 16;    // device flag: a non-finite input reached the accumulation

// One batch of a group; its (i, j) tiles are w rows wide (the last one less).
struct H1Item {
  int batch, nc, np, ib_off, prefix, w;
  long long wave_off;
  long long a_off;  // the batch's A in the scratch of its group
};
struct H1Tile {
  int item;               // the batch
  unsigned short m0, n0;  // first row along i and j (multiples of 8)
};

// Per-point inputs of the first-order H, reference layouts
// (evaluate_first_order_H.cpp:13-53); nullptr members mean "adjoint mode".
struct H1Inputs {
  const double *vsigma, *gradient_rho, *hessian, *H_prefactor1, *fogr, *vhg, *rho1, *v2rho2, *v2rhosigma,
      *v2sigma2, *partition_tab;
  const int *atom_valid;  // (n_atoms + 1, n_batches), 0-based compute ranges
  int n_atoms, j_atom_begin, j_coord;
};

struct H1Args {
  int mode;  // 0: adjoint, 1: first-order H
  int n_active, n_basis, n_full_points, n_max_batch_size, n_batches;
  const int *ib_all, *map;
  const double *wave, *gwave;
  const double *g_rho, *g_grad;  // adjoint mode
  H1Inputs h;                     // first-order H mode
  ulonglong2 *acc;                // (n_basis, n_basis, T): low part, high part
  double *A;                      // scratch: A(i, p) at a_off + p ncp + i, the
  long long a_stride;             // perturbations of one launch this far apart
  int *emax;                      // per perturbation
  int grad;       // grad phi enters A (always, except an adjoint without g_grad)
  int aligned16;  // phi, grad phi rows start on 16-byte boundaries
  int *err;
};

// Coefficients of A(i, p) for one point of batch b, perturbation t.
struct PointCoef {
  double c_phi, c_grad[3], c_hess[3];
};

__device__ __forceinline__ PointCoef point_coef(const H1Args &a, int b, int p, int prefix, int t) {
  PointCoef c;
  const long long f = a.map[prefix + p];
  const long long bp = p + (long long)a.n_max_batch_size * (b + (long long)a.n_batches * t);
  if (a.mode == 0) {
    c.c_phi = (a.g_rho != nullptr && t < a.n_active) ? a.g_rho[f + (long long)a.n_full_points * t] : 0.0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      c.c_grad[k] = a.g_grad ? 2.0 * a.g_grad[3 * bp + k] : 0.0;
      c.c_hess[k] = 0.0;
    }
    return c;
  }
  // evaluate_first_order_H.cpp:144-168, same operation order
  const H1Inputs &h = a.h;
  const long long nmb = a.n_max_batch_size;
  const double pf1 = h.H_prefactor1[bp];
  const double *fog = h.fogr + 3 * bp;
  const double *gr = h.gradient_rho + 3 * f;
  const double vsig = h.vsigma[3 * nmb * b + 3 * p];
  const double v2r2 = h.v2rho2[3 * nmb * b + 3 * p];
  const double v2rs = h.v2rhosigma[6 * nmb * b + 6 * p];
  const double v2s2 = h.v2sigma2[6 * nmb * b + 6 * p];
  const double w = h.partition_tab[f];
  const double r1 = h.rho1[f + (long long)a.n_full_points * t];
  double lfos = 0.0;
#pragma unroll
  for (int k = 0; k < 3; ++k) lfos = __dadd_rn(lfos, __dmul_rn(fog[k], gr[k]));
  lfos = __dmul_rn(lfos, 2.0);
  const double inner = __dadd_rn(__dmul_rn(v2rs, r1), __dmul_rn(v2s2, lfos));
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    c.c_grad[k] = __dadd_rn(__dmul_rn(__dmul_rn(__dmul_rn(2.0, w), gr[k]), inner),
                            __dmul_rn(__dmul_rn(__dmul_rn(2.0, w), vsig), fog[k]));
    c.c_hess[k] = -__dmul_rn(__dmul_rn(__dmul_rn(2.0, vsig), w), gr[k]);
  }
  const double pf3 = __dmul_rn(w, __dadd_rn(__dadd_rn(h.vhg[f + (long long)a.n_full_points * t], __dmul_rn(v2r2, r1)),
                                            __dmul_rn(v2rs, lfos)));
  c.c_phi = __dmul_rn(0.5, __dadd_rn(pf1, pf3));
  return c;
}

// Hessian component of hess_i(k, j_coord) (evaluate_first_order_H.cpp:6-10,185).
__device__ __forceinline__ int hess_component(int k, int j_coord) {
  const int r = j_coord - 1;
  return k == 0 ? r : (k == 1 ? (r == 0 ? 1 : (r == 1 ? 3 : 4)) : (r == 0 ? 2 : (r == 1 ? 4 : 5)));
}

// Compute-function range [vs, ve) of atom j_atom_begin + t in batch b
// (atom_valid_n_compute_c_batches, evaluate_first_order_H.cpp:131-133),
// clipped to the batch's compute functions; a range that leaves them sets
// device flag bit 3 (once, from the bound pass) and is clipped, never read
// outside the batch.
__device__ __forceinline__ void atom_range(const H1Args &a, int b, int t, int nc, int *vs, int *ve, bool flag) {
  const int atom = a.h.j_atom_begin + t;  // 1-based
  int s0 = 0, s1 = 0;
  if (atom >= 1 && atom <= a.h.n_atoms) {
    s0 = a.h.atom_valid[(atom - 1) + (long long)(a.h.n_atoms + 1) * b];
    s1 = a.h.atom_valid[atom + (long long)(a.h.n_atoms + 1) * b];
  }
  const int c0 = min(max(s0, 0), nc), c1 = min(max(s1, c0), nc);
  if (flag && (c0 != s0 || c1 != s1)) atomicOr(a.err, 8);
  *vs = c0;
  *ve = c1;
}

// ---------------------------------------------------------------- bound

// The largest |x| of a warp as an upper bound that is exact to 2^-20: the high
// words are reduced (one instruction), a non-zero value counts as at least 1.
__device__ __forceinline__ unsigned magnitude(double x) {
  const unsigned h = (unsigned)__double2hiint(x) & 0x7fffffffu;
  return h | (h == 0 && __double2loint(x) != 0 ? 1u : 0u);
}
__device__ __forceinline__ double upper_bound(unsigned h) {
  return h == 0 ? 0.0 : (h >= 0x7ff00000u ? __hiloint2double(0x7ff00000, 0) : __hiloint2double((int)h + 1, 0));
}

// One block per batch of the list, perturbation t = t0 + blockIdx.z: A(i, p) to the scratch (WRITE)
// and, unless the scale is already known (BOUND), bound_b = sum_p max_i |A(i, p)|
// max_j |phi_j(p)| (twice that for the symmetric H), of which the binary exponent
// goes to an atomicMax.  The points' coefficients come first, a thread each; then
// half a warp per point, 16-byte loads (a whole warp leaves most lanes idle in the
// last 64 rows of a small batch).  gridDim.y blocks share a batch's points; each
// bounds its own part and counts it gridDim.y times.
template <bool WRITE, bool BOUND>
__global__ void __launch_bounds__(THREADS) h1_combine_kernel(const H1Item *__restrict__ items, int t0, H1Args a) {
  __shared__ double red[THREADS / 16];
  __shared__ PointCoef s_c[THREADS];
  const H1Item W = items[blockIdx.x];
  const int t = t0 + blockIdx.z;
  const int nc = W.nc, ncp = (nc + 3) & ~3;
  const int part = (W.np + (int)gridDim.y - 1) / (int)gridDim.y;
  const int p_first = blockIdx.y * part, np = min(W.np, p_first + part);
  const int half = threadIdx.x >> 4, lane = threadIdx.x & 15;
  const unsigned members = 0xffffu << (threadIdx.x & 16);  // this half warp
  int vs = 0, ve = 0;
  if (a.mode == 1) atom_range(a, W.batch, t, nc, &vs, &ve, BOUND);
  double sum = 0.0;
  bool finite = true;
  for (int p0 = p_first; p0 < np; p0 += THREADS) {
    __syncthreads();
    if (p0 + (int)threadIdx.x < np) s_c[threadIdx.x] = point_coef(a, W.batch, p0 + threadIdx.x, W.prefix, t);
    __syncthreads();
    const int pe = min(np, p0 + THREADS);
    for (int p = p0 + half; p < pe; p += THREADS / 16) {
      const PointCoef c = s_c[p - p0];
      const double *phi = a.wave + W.wave_off + (long long)p * ncp;
      const double *gph = a.gwave + 3 * W.wave_off + 3LL * p * ncp;
      const double *hph = a.mode == 1 ? a.h.hessian + 6 * W.wave_off + 6LL * p * ncp : nullptr;
      double *A = a.A + a.a_stride * blockIdx.z + W.a_off + (long long)p * ncp;
      unsigned mp = 0, ma = 0;
      // two rows at a time (i even): a vector that starts below n_compute ends by ncp
#pragma unroll 2
      for (int i = 2 * lane; i < nc; i += 32) {
        double f[2], g[3][2] = {{0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}};
        if (a.aligned16) {
          const double2 x = __ldg(reinterpret_cast<const double2 *>(phi + i));
          f[0] = x.x;
          f[1] = x.y;
          if (a.grad) {
#pragma unroll
            for (int k = 0; k < 3; ++k) {
              const double2 y = __ldg(reinterpret_cast<const double2 *>(gph + i + k * ncp));
              g[k][0] = y.x;
              g[k][1] = y.y;
            }
          }
        } else {
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            f[e] = __ldg(phi + i + e);
            if (a.grad) {
#pragma unroll
              for (int k = 0; k < 3; ++k) g[k][e] = __ldg(gph + i + e + k * ncp);
            }
          }
        }
        double v[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          v[e] = c.c_phi * f[e];
          if (a.grad) {
#pragma unroll
            for (int k = 0; k < 3; ++k) v[e] = fma(c.c_grad[k], g[k][e], v[e]);
          }
          if (i + e >= vs && i + e < ve) {
#pragma unroll
            for (int k = 0; k < 3; ++k)
              v[e] = fma(c.c_hess[k], __ldg(hph + i + e + hess_component(k, a.h.j_coord) * ncp), v[e]);
          }
          if (i + e >= nc) v[e] = f[e] = 0.0;  // row padding
          mp = max(mp, magnitude(f[e]));
          ma = max(ma, magnitude(v[e]));
        }
        if (WRITE) *reinterpret_cast<double2 *>(A + i) = make_double2(v[0], v[1]);
      }
      if (BOUND) {
        const double term =
            upper_bound(__reduce_max_sync(members, ma)) * upper_bound(__reduce_max_sync(members, mp));
        if (!(term <= 1.0e300)) finite = false;  // NaN, Inf or beyond what the bound can carry
        if (lane == 0) sum += term;
      }
    }
  }
  if (!BOUND) return;
  if (lane == 0) red[half] = finite ? sum : -1.0;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    bool ok = true;
    for (int w = 0; w < THREADS / 16; ++w) {
      if (red[w] < 0.0) ok = false;
      s += red[w];
    }
    if (!ok || !(s <= 1.0e300)) {
      atomicOr(a.err, H1_FLAG_NONFINITE);
      return;
    }
    s *= (a.mode == 1 ? 2.0 : 1.0) * gridDim.y;
    if (s > 0.0) {
      int e = 0;
      frexp(s, &e);  // s < 2^e
      atomicMax(a.emax + t, e);
    }
  }
}

__host__ __device__ __forceinline__ int ceil_log2(long long n) {
  int k = 0;
  while ((1LL << k) < n) ++k;
  return k;
}

// The split of the fixed-point integer x = high 2^low + lowpart, |lowpart| <= 2^(low - 1):
// the sum of 2 n_batches low parts stays below 2^62 and the sum of the high parts
// below 2^62 (`bits` of the whole: 100 up to 2^24 batches); of a single
// contribution both parts are below 2^51.
struct FixedPoint {
  int low, bits;
};
__host__ __device__ __forceinline__ FixedPoint fixed_point(int n_batches) {
  const int c = ceil_log2(2LL * (n_batches > 0 ? n_batches : 1));
  const int low = c <= 13 ? 50 : 63 - c;
  return FixedPoint{low, low + 62 < 100 ? low + 62 : 100};
}
// The fixed-point exponent of this call (see the file comment).
__device__ __forceinline__ int fixed_scale(int emax, int n_batches) {
  return fixed_point(n_batches).bits - emax - ceil_log2(2LL * (n_batches > 0 ? n_batches : 1));
}

// Powers of two that take a value to its fixed-point parts.
struct FixedScale {
  double s1, s2;        // 2^s as a product (s can exceed the exponent range)
  double low, inv_low;  // 2^low, 2^-low
  double limit;         // 2^(bits - ceil(log2(2 n_batches))): above every contribution
};
__device__ __forceinline__ FixedScale make_scale(int emax, int n_batches) {
  const FixedPoint f = fixed_point(n_batches);
  const int s = fixed_scale(emax, n_batches);
  return FixedScale{ldexp(1.0, s / 2), ldexp(1.0, s - s / 2), ldexp(1.0, f.low), ldexp(1.0, -f.low),
                    ldexp(1.0, s + emax)};
}

// v 2^s rounded to an integer, in two parts; false for a value the scale cannot
// hold (a non-finite input, flagged by the bound).
__device__ __forceinline__ bool to_fixed(double v, const FixedScale &f, long long *lo, long long *hi) {
  const double V = v * f.s1 * f.s2, magic = 6755399441055744.0;  // 1.5 2^52
  const double th = fma(V, f.inv_low, magic);
  const double tl = fma(magic - th, f.low, V) + magic;  // the difference is exact, the sum rounds to an integer
  *hi = __double_as_longlong(th) - __double_as_longlong(magic);
  *lo = __double_as_longlong(tl) - __double_as_longlong(magic);
  return fabs(V) < f.limit;
}

__device__ __forceinline__ void add_fixed(ulonglong2 *entry, long long lo, long long hi) {
  if (lo) atomicAdd(&entry->x, (unsigned long long)lo);
  if (hi) atomicAdd(&entry->y, (unsigned long long)hi);
}

// ----------------------------------------------------------------- tiles

// One chunk's products of a warp: CM of the tile's 8-row blocks along i (stride 2
// blocks, the warps' round), CN along j (stride 4 blocks).
template <int CM, int CN>
__device__ __forceinline__ void tile_mma(double (&acc)[4][2][2], const double *X, const double *Y) {
#pragma unroll
  for (int ks = 0; ks < KC / 4; ++ks) {
    double fa[CM], fb[CN];
#pragma unroll
    for (int mi = 0; mi < CM; ++mi) fa[mi] = X[ks * 4 * LD + mi * 16];
#pragma unroll
    for (int ni = 0; ni < CN; ++ni) fb[ni] = Y[ks * 4 * LD + ni * 32];
#pragma unroll
    for (int mi = 0; mi < CM; ++mi)
#pragma unroll
      for (int ni = 0; ni < CN; ++ni) dmma_8x8x4(acc[mi][ni][0], acc[mi][ni][1], fa[mi], fb[ni]);
  }
}
__device__ __forceinline__ void tile_mma_any(int shape, double (&acc)[4][2][2], const double *X, const double *Y) {
  switch (shape) {  // 2 CM + CN, uniform over the warp
    case 2 * 4 + 2: tile_mma<4, 2>(acc, X, Y); break;
    case 2 * 3 + 2: tile_mma<3, 2>(acc, X, Y); break;
    case 2 * 2 + 2: tile_mma<2, 2>(acc, X, Y); break;
    case 2 * 1 + 2: tile_mma<1, 2>(acc, X, Y); break;
    case 2 * 4 + 1: tile_mma<4, 1>(acc, X, Y); break;
    case 2 * 3 + 1: tile_mma<3, 1>(acc, X, Y); break;
    case 2 * 2 + 1: tile_mma<2, 1>(acc, X, Y); break;
    case 2 * 1 + 1: tile_mma<1, 1>(acc, X, Y); break;
    default: break;
  }
}

template <bool SYM>
struct TileShape {
  static constexpr int STAGES = SYM ? 3 : 4, ARRAYS = SYM ? 4 : 2, CTAS = SYM ? 2 : 3;
  static constexpr int SMEM = (int)sizeof(double) * STAGES * ARRAYS * KC * LD;
};

template <bool SYM, bool MANY>
__global__ void __launch_bounds__(THREADS, TileShape<SYM>::CTAS)
    h1_tile_kernel(const H1Item *__restrict__ items, const H1Tile *__restrict__ tiles, int n_tiles, int t0, int n_t,
                   H1Args a) {
  // a stage: A of the tile's i rows and phi of its j rows; if SYM, phi of the i rows and A of the j rows
  constexpr int STAGES = TileShape<SYM>::STAGES, ARRAYS = TileShape<SYM>::ARRAYS, BUF = KC * LD;
  extern __shared__ __align__(16) double smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp >> 2, wn = warp & 3, g = lane >> 2, q = lane & 3;
  // MANY: the tiles of perturbation t0, then of t0 + 1, ... (n_t of them)
  int t = t0, emax = a.emax[t0];
  if (!MANY && emax == EMAX_EMPTY) return;  // every contribution is zero
  FixedScale scale = make_scale(emax, a.n_batches);
  const int n_all = MANY ? n_tiles * n_t : n_tiles;
  H1Tile tile = tiles[MANY ? blockIdx.x % n_tiles : blockIdx.x];
  for (int it = blockIdx.x; it < n_all; it += gridDim.x) {
    const int z = MANY ? it / n_tiles : 0;
    const H1Item W = items[tile.item];
    const int m0 = tile.m0, n0 = tile.n0, mw = min(W.w, W.nc - m0), nw = min(W.w, W.nc - n0);
    if (it + (int)gridDim.x < n_all) tile = tiles[MANY ? (it + gridDim.x) % n_tiles : it + gridDim.x];
    if (MANY) {
      if (t != t0 + z) {
        t = t0 + z;
        emax = a.emax[t];
        scale = make_scale(emax, a.n_batches);
      }
      if (emax == EMAX_EMPTY) continue;
    }
    ulonglong2 *entries = a.acc + (long long)a.n_basis * a.n_basis * t;
    const int nc = W.nc, np = W.np, ncp = (nc + 3) & ~3;
    const bool diag = m0 == n0;
    const double *phi = a.wave + W.wave_off, *amat = a.A + a.a_stride * z + W.a_off;
    double acc[4][2][2];
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
      for (int y = 0; y < 2; ++y) acc[x][y][0] = acc[x][y][1] = 0.0;

    const int nmi = (mw + 7) / 8, nni = (nw + 7) / 8;  // 8-row blocks of the tile
    // Copies: lane -> two rows of the tile, warp -> points warp and warp + 8 of a
    // chunk.  Rows past n_compute (up to whole blocks) and points past the batch
    // are zero.
    const int r = 2 * lane;
    auto copy = [&](double *dst, const double *src, int i0, int blocks, int k0, bool wide) {
      if (r >= blocks * 8) return;
      const int i = i0 + r, left = nc - i;
#pragma unroll
      for (int j = 0; j < KC / 8; ++j) {
        const int k = warp + 8 * j, p = k0 + k;
        const double *from = src + (long long)p * ncp + i;
        double *to = dst + k * LD + r;
        if (wide) {
          const int bytes = p < np ? (left > 1 ? 16 : (left > 0 ? 8 : 0)) : 0;
          cp_async_16(to, bytes ? from : src, bytes);
        } else {
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const bool ok = p < np && left > e;
            cp_async_8(to + e, ok ? from + e : src, ok ? 8 : 0);
          }
        }
      }
    };
    auto load = [&](int c) {
      double *S = smem + (c % STAGES) * ARRAYS * BUF;
      const int k0 = c * KC;
      copy(S, amat, m0, nmi, k0, true);
      copy(S + BUF, phi, n0, nni, k0, a.aligned16);
      if (SYM && !diag) {  // a diagonal tile has both on both sides
        copy(S + 2 * BUF, phi, m0, nmi, k0, a.aligned16);
        copy(S + 3 * BUF, amat, n0, nni, k0, true);
      }
    };
    const int nch = (np + KC - 1) / KC;
    __syncthreads();  // the last item's stages are consumed
#pragma unroll
    for (int c = 0; c < STAGES - 1; ++c) {
      if (c < nch) load(c);
      cp_async_commit();
    }
    const int cm = (nmi - wm + 1) / 2, cn = (nni - wn + 3) / 4;  // this warp's blocks
    const int shape = cm > 0 && cn > 0 ? 2 * cm + cn : 0;
    const int off_m = q * LD + g + wm * 8, off_n = q * LD + g + wn * 8;
    for (int c = 0; c < nch; ++c) {
      cp_async_wait<STAGES - 2>();
      __syncthreads();
      if (c + STAGES - 1 < nch) load(c + STAGES - 1);
      cp_async_commit();
      const double *S = smem + (c % STAGES) * ARRAYS * BUF;
      tile_mma_any(shape, acc, S + off_m, S + BUF + off_n);
      if (SYM) tile_mma_any(shape, acc, (diag ? S + BUF : S + 2 * BUF) + off_m, (diag ? S : S + 3 * BUF) + off_n);
    }
    cp_async_wait<0>();
    // add the tile (and, for an off-diagonal symmetric tile, its transpose)
    long long col[2][2];
#pragma unroll
    for (int ni = 0; ni < 2; ++ni)
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        const int j = (ni * 4 + wn) * 8 + 2 * q + hh;
        col[ni][hh] = j < nw && n0 + j < nc ? __ldg(a.ib_all + W.ib_off + n0 + j) - 1 : -1;
      }
#pragma unroll
    for (int mi = 0; mi < 4; ++mi) {
      const int i = (mi * 2 + wm) * 8 + g;
      if (i >= mw || m0 + i >= nc) continue;
      const long long row = __ldg(a.ib_all + W.ib_off + m0 + i) - 1;
#pragma unroll
      for (int ni = 0; ni < 2; ++ni)
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          const long long c = col[ni][hh];
          long long lo, hi;
          if (c < 0 || !to_fixed(acc[mi][ni][hh], scale, &lo, &hi)) continue;
          add_fixed(entries + row + c * a.n_basis, lo, hi);
          if (SYM && !diag) add_fixed(entries + c + row * a.n_basis, lo, hi);
        }
    }
  }
}

// out(e) += (the entry) 2^-s, one rounding; entries no tile touched add 0.  The
// entries are zeroed for the next call.
__global__ void h1_finalize_kernel(long long n, ulonglong2 *__restrict__ acc_all, const int *emax_p, int n_batches,
                                   double *__restrict__ out_all) {
  const int t = blockIdx.y, emax = emax_p[t];
  ulonglong2 *acc = acc_all + n * t;
  double *out = out_all + n * t;
  if (emax == EMAX_EMPTY) return;
  const int s = fixed_scale(emax, n_batches), low = fixed_point(n_batches).low;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
    const ulonglong2 w = acc[e];
    if ((w.x | w.y) == 0) continue;
    acc[e] = make_ulonglong2(0, 0);
    const __int128 x = (__int128)(long long)w.y * ((__int128)1 << low) + (__int128)(long long)w.x;
    if (x == 0) continue;
    // magnitude as two unsigned words of one sign: no cancellation, the
    // result within 2 ulp, and the same bits on every run
    const unsigned __int128 m = x < 0 ? (unsigned __int128)(-x) : (unsigned __int128)x;
    const double v = ldexp((double)(unsigned long long)(m >> 64), 64) + (double)(unsigned long long)m;
    out[e] += ldexp(x < 0 ? -v : v, -s);
  }
}

}  // namespace

// Groups of batches, in locality order (`key`, then cost, so that the entries
// neighbouring batches share are added to while they are in L2), whose A fits
// `budget` bytes (or one batch): one item per batch (for the first pass), and per
// group its tiles, those with j >= i first (the symmetric H takes only them).
void rho1_h1_build_items(const std::vector<Rho1WorkItem> &batches, long long budget, std::vector<unsigned char> *items,
                         std::vector<unsigned char> *tile_list, std::vector<H1Group> *groups, long long *a_len) {
  std::vector<Rho1WorkItem> order;
  order.reserve(batches.size());
  for (const Rho1WorkItem &b : batches)
    if (b.nc > 0 && b.np > 0) order.push_back(b);
  rho1_order_items(&order, 2);
  std::vector<H1Item> v;
  std::vector<H1Tile> tiles, lower;
  v.reserve(order.size());
  groups->clear();
  *a_len = 0;
  for (size_t b0 = 0; b0 < order.size();) {
    H1Group g{(int)v.size(), 0, (int)tiles.size(), 0, 0};
    lower.clear();
    long long len = 0;
    size_t b1 = b0;
    for (; b1 < order.size(); ++b1) {
      const Rho1WorkItem &b = order[b1];
      const long long need = (long long)((b.nc + 3) & ~3) * b.np;
      if (b1 > b0 && (len + need) * (long long)sizeof(double) > budget) break;
      const int w = (ceil_div(b.nc, ceil_div(b.nc, TILE)) + 7) / 8 * 8;
      for (int m0 = 0; m0 < b.nc; m0 += w)
        for (int n0 = 0; n0 < b.nc; n0 += w)
          (n0 >= m0 ? tiles : lower).push_back(H1Tile{(int)v.size(), (unsigned short)m0, (unsigned short)n0});
      v.push_back(H1Item{b.batch, b.nc, b.np, b.ib_off, b.prefix, w, b.wave_off, len});
      len += need;
    }
    g.n_first = (int)v.size() - g.first;
    g.n_upper = (int)tiles.size() - g.tiles;
    tiles.insert(tiles.end(), lower.begin(), lower.end());
    g.n_tiles = (int)tiles.size() - g.tiles;
    groups->push_back(g);
    *a_len = std::max(*a_len, len);
    b0 = b1;
  }
  items->resize(v.size() * sizeof(H1Item));
  if (!v.empty()) memcpy(items->data(), v.data(), items->size());
  tile_list->resize(tiles.size() * sizeof(H1Tile));
  if (!tiles.empty()) memcpy(tile_list->data(), tiles.data(), tile_list->size());
}

// Groups for another budget: the scratch goes, and the lists are made and uploaded
// again (synchronous; not inside a stream capture).
int rho1_h1_rebuild(Rho1Plan *plan, long long budget) {
  std::vector<unsigned char> items, tiles;
  std::vector<H1Group> groups;
  long long a_len = 0;
  rho1_h1_build_items(plan->h_batches, budget, &items, &tiles, &groups, &a_len);
  void *d_items = nullptr, *d_tiles = nullptr;
  if (cudaMalloc(&d_items, std::max<size_t>(items.size(), 16)) != cudaSuccess ||
      cudaMalloc(&d_tiles, std::max<size_t>(tiles.size(), 16)) != cudaSuccess) {
    cudaGetLastError();
    cudaFree(d_items);
    return fail(FRPA_ERR_OOM, "first-order H / adjoint: work list allocation failed");
  }
  if ((!items.empty() && cudaMemcpy(d_items, items.data(), items.size(), cudaMemcpyHostToDevice) != cudaSuccess) ||
      (!tiles.empty() && cudaMemcpy(d_tiles, tiles.data(), tiles.size(), cudaMemcpyHostToDevice) != cudaSuccess)) {
    cudaFree(d_items);
    cudaFree(d_tiles);
    return fail(FRPA_ERR_CUDA, "first-order H / adjoint: work list upload failed");
  }
  cudaFree(plan->d_h1_acc);
  plan->d_h1_acc = nullptr;
  plan->release(plan->d_h1_items);
  plan->release(plan->d_h1_tiles);
  plan->d_h1_items = d_items;
  plan->d_h1_tiles = d_tiles;
  plan->h1_groups = groups;
  plan->h1_a_len = a_len;
  return FRPA_OK;
}

// All perturbations in one launch each of the passes, while their A fits the budget:
// one at a time a small problem leaves most SMs idle and waits for a chain of launches
// per perturbation.  Measured, us, H / adjoint, four perturbations one at a time ->
// together: 20 batches of 20-120 functions 238 / 171 -> 75 / 61; 150: 473 / 268 ->
// 267 / 173; 1,600 batches of 40-120: 2,994 / 2,081 -> 2,796 / 1,990.
size_t rho1_h1_a_bytes(Rho1Plan &plan) {
  plan.h1_at_once = 1;
  if (plan.h1_groups.size() == 1)
    plan.h1_at_once = (int)std::max(
        1LL, std::min<long long>(plan.T, plan.h1_budget / std::max(1LL, 8 * plan.h1_a_len)));
  return sizeof(double) * (size_t)plan.h1_a_len * plan.h1_at_once;
}

// Scratch: the accumulator, two words per entry of (n_basis, n_basis, T), zero
// between calls (the finalize pass clears what the tiles touched), the exponent
// words, and A of one group (of as many perturbations as the call takes at once);
// allocated by the first call (outside stream capture).  Where it does not fit, with
// fewer perturbations, then with groups of half the size, down to single batches.
// A caller's own buffer for A (h1_a_lent) is used where it is large enough.
static int h1_scratch(Rho1Plan &plan, cudaStream_t stream) {
  if (plan.d_h1_acc) return FRPA_OK;
  static PerDeviceOnce configured;
  FRPA_TRY(configured.run(plan.device, []() -> int {
    for (auto kernel : {h1_tile_kernel<true, false>, h1_tile_kernel<true, true>})
      FRPA_CUDA_TRY(
          cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, TileShape<true>::SMEM));
    for (auto kernel : {h1_tile_kernel<false, false>, h1_tile_kernel<false, true>})
      FRPA_CUDA_TRY(
          cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, TileShape<false>::SMEM));
    return FRPA_OK;
  }));
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  FRPA_CUDA_TRY(cudaStreamIsCapturing(stream, &cap));
  if (cap != cudaStreamCaptureStatusNone)
    return fail(FRPA_ERR_INVALID,
                "first-order H / adjoint: the accumulator is allocated by the first call; call once before "
                "capturing a graph");
  const size_t n = (size_t)plan.n_basis * plan.n_basis * plan.T;
  const size_t words = 2 * sizeof(unsigned long long) * n, flags = (sizeof(int) * plan.T + 255) / 256 * 256;
  const bool lent = plan.h1_a_lent_bytes >= rho1_h1_a_bytes(plan) && plan.h1_a_lent_bytes > 0;
  for (;;) {
    const size_t a_bytes = lent ? 0 : sizeof(double) * (size_t)plan.h1_a_len;
    const size_t bytes = words + flags + a_bytes * plan.h1_at_once;
    if (cudaMalloc((void **)&plan.d_h1_acc, bytes) == cudaSuccess) {
      unsigned char *own = reinterpret_cast<unsigned char *>(plan.d_h1_acc) + words + flags;
      plan.h1_a = lent ? plan.h1_a_lent : reinterpret_cast<double *>(own);
      break;
    }
    cudaGetLastError();  // a refused allocation is no launch's error
    plan.d_h1_acc = nullptr;
    if (!lent && plan.h1_at_once > 1) {
      plan.h1_at_once /= 2;
      continue;
    }
    const long long a_len = plan.h1_a_len;
    if (a_bytes > 0) FRPA_TRY(rho1_h1_rebuild(&plan, (long long)a_bytes / 2));
    if (plan.h1_a_len == a_len)
      return fail(FRPA_ERR_OOM, "first-order H / adjoint: %zu bytes of scratch could not be allocated", bytes);
  }
  plan.h1_clean = false;
  return FRPA_OK;
}

template <bool SYM>
static int h1_tiles(const H1Item *items, const H1Tile *tiles, int n_tiles, int t, int n_t, const H1Args &a, int n_sm,
                    cudaStream_t stream) {
  const int grid = (int)std::min<long long>((long long)n_tiles * n_t, n_sm * TileShape<SYM>::CTAS);
  auto kernel = n_t > 1 ? h1_tile_kernel<SYM, true> : h1_tile_kernel<SYM, false>;
  kernel<<<grid, THREADS, TileShape<SYM>::SMEM, stream>>>(items, tiles, n_tiles, t, n_t, a);
  FRPA_LAUNCH_CHECK();
  return FRPA_OK;
}

// mode 0: the adjoint over all tiles; mode 1: the first-order H over the tiles
// with j >= i.  `out` (n_basis, n_basis, T) is accumulated into.
static int h1_run(Rho1Plan &plan, int mode, int n_active, const double *wave, const double *gwave,
                  const double *g_rho, const double *g_grad, const H1Inputs *h, double *out, cudaStream_t stream) {
  if (plan.h1_groups.empty()) return FRPA_OK;
  FRPA_TRY(h1_scratch(plan, stream));
  const size_t nb2 = (size_t)plan.n_basis * plan.n_basis, n = nb2 * plan.T;
  ulonglong2 *acc = reinterpret_cast<ulonglong2 *>(plan.d_h1_acc);
  int *emax = reinterpret_cast<int *>(acc + n);
  // zero already unless this is the first call or an earlier one failed half-way
  if (!plan.h1_clean) FRPA_CUDA_TRY(cudaMemsetAsync(acc, 0, n * sizeof(ulonglong2), stream));
  plan.h1_clean = false;
  FRPA_CUDA_TRY(cudaMemsetAsync(emax, 0x80, sizeof(int) * plan.T, stream));
  H1Args a{};
  a.mode = mode;
  a.n_active = n_active;
  a.n_basis = plan.n_basis;
  a.n_full_points = plan.n_full_points;
  a.n_max_batch_size = plan.n_max_batch_size;
  a.n_batches = plan.n_batches;
  a.ib_all = plan.d_ib;
  a.map = plan.d_map;
  a.wave = wave;
  a.gwave = gwave;
  a.g_rho = g_rho;
  a.g_grad = g_grad;
  if (h) a.h = *h;
  a.acc = acc;
  a.A = plan.h1_a;
  a.a_stride = plan.h1_a_len;
  a.emax = emax;
  a.err = plan.d_err;
  a.grad = mode == 1 || g_grad != nullptr;
  a.aligned16 = plan.wave_aligned16 && !(((uintptr_t)wave | (uintptr_t)gwave) & 15);
  const H1Item *items = static_cast<const H1Item *>(plan.d_h1_items);
  const H1Tile *tiles = static_cast<const H1Tile *>(plan.d_h1_tiles);
  int n_sm = 148;
  FRPA_CUDA_TRY(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, plan.device));
  const bool one_group = plan.h1_groups.size() == 1;
  // the adjoint's g_grad covers every perturbation, everything else the active ones
  const int n_t = mode == 0 && g_grad ? plan.T : std::max(0, n_active);
  for (int t = 0, n = 1; t < n_t; t += n) {
    n = std::min(plan.h1_at_once, n_t - t);  // more than 1 only with one group
    if (!one_group) {
      for (const H1Group &g : plan.h1_groups) {
        h1_combine_kernel<false, true><<<dim3(g.n_first, 2), THREADS, 0, stream>>>(items + g.first, t, a);
        FRPA_LAUNCH_CHECK();
      }
    }
    for (const H1Group &g : plan.h1_groups) {
      if (one_group)
        h1_combine_kernel<true, true><<<dim3(g.n_first, 2, n), THREADS, 0, stream>>>(items + g.first, t, a);
      else
        h1_combine_kernel<true, false><<<dim3(g.n_first, 2), THREADS, 0, stream>>>(items + g.first, t, a);
      FRPA_LAUNCH_CHECK();
      if (mode == 1)
        FRPA_TRY(h1_tiles<true>(items, tiles + g.tiles, g.n_upper, t, n, a, n_sm, stream));
      else
        FRPA_TRY(h1_tiles<false>(items, tiles + g.tiles, g.n_tiles, t, n, a, n_sm, stream));
    }
  }
  if (n_t > 0) {
    h1_finalize_kernel<<<dim3(n_sm * 8, n_t), 256, 0, stream>>>((long long)nb2, acc, emax, plan.n_batches, out);
    FRPA_LAUNCH_CHECK();
  }
  plan.h1_clean = true;
  return FRPA_OK;
}

int rho1_adjoint_run(Rho1Plan &plan, int n_active, const double *wave, const double *gwave, const double *g_rho,
                     const double *g_grad, double *dP1, cudaStream_t stream) {
  return h1_run(plan, 0, n_active, wave, gwave, g_rho, g_grad, nullptr, dP1, stream);
}

int rho1_first_order_h_run(Rho1Plan &plan, int n_active, int n_atoms, int j_atom_begin, int j_coord,
                           const int *atom_valid, const double *wave, const double *gwave, const double *hwave,
                           const double *vsigma, const double *gradient_rho, const double *H_prefactor1,
                           const double *fogr, const double *vhg, const double *rho1, const double *v2rho2,
                           const double *v2rhosigma, const double *v2sigma2, const double *partition_tab,
                           double *first_order_H, cudaStream_t stream) {
  H1Inputs h{vsigma, gradient_rho, hwave, H_prefactor1, fogr, vhg, rho1, v2rho2, v2rhosigma, v2sigma2,
             partition_tab, atom_valid, n_atoms, j_atom_begin, j_coord};
  return h1_run(plan, 1, n_active, wave, gwave, nullptr, nullptr, &h, first_order_H, stream);
}

}  // namespace frpa
