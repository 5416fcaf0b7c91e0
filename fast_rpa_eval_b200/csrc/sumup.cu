// Hartree potential sum-up from atomic multipoles (near-field spline + far-field
// analytic multipoles), FP64.
//
// Reference: fast_rap_src_dfpt_gpu_eval/sum_up_whole_potential.cpp:195-503 (CPU),
// .../sum_up_whole_potential.cu:548-769 (GPU: four launches, near and far field
// in separate kernels).  Per valid point p, perturbation t and centre slot ic
// (in the order of centers_hartree_potential):
//   d = p - R_centre, d2 = d.d               (rounded op by op, :395-402)
//   lam = l_hartree[species]; while (outer_potential_radius(lam) < d2 && lam > 0) lam--
//   d2 <  multipole_radius_sq:  near field  = sum_{lm <= lam} spline_lm(i_r_log) Y_lm(d_hat)
//   d2 <  1e8:                  far field   = sum_{n < n_cc(lam)} x^i y^j z^k Fp[nn] cc[n] Q[l,m]
//   delta_v(p, t) += contribution, in slot order.
//
// This file keeps every branch decision bit-identical to the reference (d2 and
// the comparisons use exactly rounded products and sums) and re-designs the
// arithmetic for the FP64 pipe:
//
// * Far field (fast path).  The caller's (index_cc, cc) table is converted once,
//   exactly, into a polynomial in the Kelvin-inverted coordinates u = d / r^2:
//   every table term x^i y^j z^k Fp[nn] is multiplied through by
//   (x^2+y^2+z^2)^(l-nn) / r^(2(l-nn)), which turns it into u^(a,b,c) / r with
//   a+b+c = l.  Per (centre, t) the multipole moments are folded in by a
//   prepare kernel, so one (point, centre) pair costs one Horner evaluation of
//   C(lam+3, 3) fused multiply-adds (84 at l = 6) instead of the 176-term table
//   loop.  The Horner degree is lam, specialised at compile time per warp-
//   uniform lam (the l_max-specialised AOT kernels of the reference's
//   task3_jit/version5, but derived from the runtime table rather than baked in).
// * Near field, in a launch of its own after the far field's except for dense
//   points around few centres.  Real Y_lm by the associated-Legendre recursion
//   fused with the Hermite spline dot, read straight from the caller's
//   (L^2, 2, n_hartree_grid, atom, t) table (the two grid nodes needed are one
//   contiguous 4 L^2 run), so the reference's per-call transpose is not needed.
// * Which pairs are near, far or skipped is decided for a warp's points at once
//   wherever the box around them allows it (the points are in spatial order).
// * Generic path.  When the fast path's preconditions do not hold (a
//   centers_hartree_potential list that is not the identity, whose far field
//   the reference evaluates with the loop slot as centre, :161-162/:183; or a
//   table whose rows are not homogeneous multipole terms), a kernel that mirrors
//   the reference table loop exactly is used instead.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <utility>
#include <vector>

#include "frpa_internal.cuh"
#include "kelvin_horner.cuh"

namespace frpa {

constexpr int SU_LMAX = FRPA_SUMUP_MAX_L;  // 8
constexpr int SU_THREADS = 128;
constexpr int SU_CHUNK = 8;      // centre records per shared-memory chunk (two buffers) at the highest l

// Near-field constants: Y_lm = K[l][m] Q_l^m(z) {C_m, S_m}; recursion
// Q_l^m = RA[l][m] z Q_{l-1}^m - RB[l][m] Q_{l-2}^m; DF[m] = (2m-1)!!.
__constant__ double c_K[SU_LMAX + 1][SU_LMAX + 1];
__constant__ double c_Kcos[SU_LMAX + 1][SU_LMAX + 1];
__constant__ double c_RA[SU_LMAX + 1][SU_LMAX + 1];
__constant__ double c_RB[SU_LMAX + 1][SU_LMAX + 1];
__constant__ double c_DF[SU_LMAX + 1];
// the near-field kernel's copy of K, RA, RB, for threads that each read another entry
__device__ double d_near_tables[3][SU_LMAX + 1][SU_LMAX + 1];
__host__ __device__ constexpr int n_kelvin(int L) { return kelvin_count(L); }

// record layout (doubles) for one (centre slot, t)
enum : int {
  R_X = 0, R_Y, R_Z, R_MRS, R_LAM0, R_ATOM, R_RGM, R_LINC, R_NGRID, R_SAFE, R_OPR  // R_OPR .. R_OPR+L
};
__host__ __device__ constexpr int rec_coef_off(int L) { return (R_OPR + L + 2) & ~1; }
// R_SAFE: no coefficient above SAFE_COEF and no far pair closer than
// sqrt(SAFE_MRS), so that every partial sum of the far-field polynomial is
// finite (165 terms of at most 1e100 x 1e20^8) and 0 x (partial sum) is 0
constexpr double SAFE_COEF = 1e100, SAFE_MRS = 1e-40;
__host__ __device__ constexpr int rec_stride(int L) { return rec_coef_off(L) + kelvin_slots(L); }

// Box around a warp's points (points that are not finite, and lanes without a
// point, left out: every pair of theirs is skipped; an empty box is infinitely
// far from everything).
struct Box {
  double lo[3], hi[3];
};

struct SumupPlan {
  int device = 0;
  unsigned char *arena = nullptr;  // the device allocation behind the pointers below
  size_t arena_bytes = 0;
  bool arena_lent = false;  // the caller's
  int T = 1, L = 0, L2 = 1, lma = 0, icc_dim0 = 0, mc_dim = 0, hfla = 0;
  int n_full_points = 0, n_valid_points = 0, n_centers = 0, n_chp = 0, n_atoms = 0, n_species = 0;
  int n_hartree_grid = 0;
  int fast = 0;
  int n_coef = 0, rs = 0;
  // device const arrays
  int *d_map = nullptr;
  // valid points in spatial (Morton) order, for warp-uniform branches: their valid-point
  // index, full index and coordinates (x, y, z rows of n_valid_points), so that the fast
  // kernels' loads coalesce and none waits for an index
  int *d_order = nullptr, *d_pfull = nullptr;
  double *d_pxyz = nullptr;
  Box *d_pbox = nullptr;  // of every 32 of them
  double *d_coord = nullptr;
  int *d_species = nullptr, *d_species_center = nullptr, *d_l_hartree = nullptr, *d_n_grid = nullptr;
  int *d_c2a = nullptr, *d_chp = nullptr, *d_icc = nullptr, *d_ncc = nullptr, *d_ijkmax = nullptr;
  int *d_icc_packed = nullptr;  // (i | j<<8 | k<<16 | nn<<24) per row
  double *d_cc = nullptr, *d_cc_xyz = nullptr, *d_rgm = nullptr, *d_linc = nullptr;
  int *d_slot = nullptr;                            // coefficient -> position in a record
  int *d_conv_ptr = nullptr, *d_conv_lm = nullptr;  // Kelvin conversion (CSR by coefficient): (l, m) slot,
  double2 *d_conv_fc = nullptr;                     // factor and cc of the table row
  // workspaces
  double *d_mc = nullptr;    // (mc_dim, n_atoms, T)
  double *d_recs = nullptr;  // (rs, n_chp, T)
  double4 *d_heads = nullptr;  // (n_chp, T): centre and near radius^2, for the near-field launch's search
  int *d_err = nullptr;      // device-side input error flags
  // adjoint: transpose of the Kelvin conversion (by table row; coefficients in
  // the dQ kernels' order), the table rows of each (l, m), per point-block partial
  // sums (n_coef, n_chp, T, adj_nz) and the slots of each atom (CSR, ascending)
  int *d_convT_ptr = nullptr, *d_convT_k = nullptr;
  double *d_convT_f = nullptr;
  int *d_lm_ptr = nullptr, *d_lm_row = nullptr;
  double *d_dcoef_part = nullptr;
  int adj_nz = 1, adj_pts = 4096;
  int *d_atom_slot_ptr = nullptr, *d_atom_slots = nullptr;
};

namespace {

// ------------------------------------------------------------ prepare ---

// multipole_c = cc * Q with the l cap and the 1e-10 threshold
// (sum_up_whole_potential.cpp:357-378); rows past n_cc(l_hartree_max_far_distance)
// are zero (the reference leaves them uninitialised).
__global__ void sumup_multipole_c_kernel(int n_atoms, int L, int L2, int mc_dim, int icc_dim0, int lma,
                                         const int *__restrict__ icc, const int *__restrict__ ncc,
                                         const double *__restrict__ cc, const int *__restrict__ lhmfd,
                                         const double *__restrict__ Q, double *__restrict__ mc,
                                         int *__restrict__ err) {
  const int a = blockIdx.x, t = blockIdx.y;
  int lh = lhmfd[a + n_atoms * t];
  if (lh < 0 || lh > L || lh > lma) {
    if (threadIdx.x == 0) atomicOr(err, 1);
    lh = lh < 0 ? 0 : (lh > L ? L : lh);
  }
  const int nmax = ncc[lh];
  for (int n = threadIdx.x; n < mc_dim; n += blockDim.x) {
    double v = 0.0;
    if (n < nmax) {
      const int l = icc[n], m = icc[n + icc_dim0];
      const double q = Q[(l * l + l + m) + (long long)L2 * (a + (long long)n_atoms * t)];
      v = (l <= lh && fabs(q) > 1e-10) ? cc[n] * q : 0.0;
    }
    mc[n + (long long)mc_dim * (a + (long long)n_atoms * t)] = v;
  }
}

// Per (slot, t) record for the fast kernels: centre, radii, l_hartree, near
// field parameters and the Kelvin coefficients (CSR contraction of
// multipole_c = cc Q with the l cap and the 1e-10 threshold of
// sum_up_whole_potential.cpp:357-378, formed on the way).  Also checks
// l_hartree_max_far_distance of every atom, as sumup_multipole_c_kernel does.
__global__ void __launch_bounds__(128)
    sumup_prep_kernel(int L, int lma, int n_atoms, int n_chp, int n_coef, int rs, const int *__restrict__ chp,
                      const int *__restrict__ c2a, const int *__restrict__ species,
                      const int *__restrict__ species_center, const int *__restrict__ l_hartree,
                      const int *__restrict__ n_grid, const double *__restrict__ rgm,
                      const double *__restrict__ linc, const double *__restrict__ cc_xyz,
                      const double *__restrict__ mrs, const double *__restrict__ opr,
                      const int *__restrict__ lhmfd, const double *__restrict__ Q, const int *__restrict__ slot_of,
                      const int *__restrict__ conv_ptr, const int *__restrict__ conv_lm,
                      const double2 *__restrict__ conv_fc, double *__restrict__ recs, double4 *__restrict__ heads,
                      int *__restrict__ err) {
  __shared__ double q_kept[(SU_LMAX + 1) * (SU_LMAX + 1)];
  const int slot = blockIdx.x, t = blockIdx.y, L2 = (L + 1) * (L + 1);
  grid_release();
  if (slot < n_atoms && threadIdx.x == 0) {
    const int lh = lhmfd[slot + n_atoms * t];
    if (lh < 0 || lh > L || lh > lma) atomicOr(err, 1);
  }
  if (slot >= n_chp) return;
  const int cur = chp[slot] - 1;
  const int atom = c2a[cur] - 1;
  const long long at = atom + (long long)n_atoms * t;
  const int lh = min(max(lhmfd[at], 0), L);
  for (int lm = threadIdx.x; lm < L2; lm += blockDim.x) {
    const double q = Q[lm + L2 * at];
    q_kept[lm] = (lm < (lh + 1) * (lh + 1) && fabs(q) > 1e-10) ? q : 0.0;
  }
  double *r = recs + (long long)rs * (slot + (long long)n_chp * t);
  for (int l = threadIdx.x; l <= L; l += blockDim.x) r[R_OPR + l] = opr[l + (L + 1) * at];
  __syncthreads();
  bool small = true;
  for (int k = threadIdx.x; k < n_coef; k += blockDim.x) {
    double s = 0.0;
    const int e1 = conv_ptr[k + 1];
#pragma unroll 4
    for (int e = conv_ptr[k]; e < e1; ++e) {
      const double q = q_kept[conv_lm[e]];
      const double2 fc = conv_fc[e];
      s += fc.x * (q != 0.0 ? fc.y * q : 0.0);
    }
    r[rec_coef_off(L) + slot_of[k]] = s;
    small = small && fabs(s) <= SAFE_COEF;
  }
  const bool safe = __syncthreads_and(small);
  if (threadIdx.x == 0) {
    const int sp = species_center[cur] - 1;
    const double m = mrs[at];
    r[R_X] = cc_xyz[3 * cur + 0];
    r[R_Y] = cc_xyz[3 * cur + 1];
    r[R_Z] = cc_xyz[3 * cur + 2];
    r[R_MRS] = m;
    r[R_LAM0] = (double)l_hartree[species[atom] - 1];
    r[R_ATOM] = (double)atom;
    r[R_RGM] = rgm[sp];
    r[R_LINC] = linc[sp];
    r[R_NGRID] = (double)n_grid[sp];
    r[R_SAFE] = safe && m >= SAFE_MRS ? 1.0 : 0.0;
    heads[slot + (long long)n_chp * t] = make_double4(cc_xyz[3 * cur], cc_xyz[3 * cur + 1], cc_xyz[3 * cur + 2], m);
  }
}

// ------------------------------------------------------- device pieces ---

// Near-field geometry of one pair (sum_up_whole_potential.cpp:411-477, spline
// :12-52): the trig values exactly as the reference forms them, the spline
// interval and its four Hermite weights.
struct NearGeom {
  double x, y, z;         // unit vector
  double ta, tb, tc, td;  // weights of (value, slope) at the interval's two nodes
  int i_spl;              // interval, 1-based
};

__device__ __forceinline__ NearGeom near_geometry(double dx, double dy, double dz, double d2, double rgm, double linc,
                                                  int ngrid) {
  NearGeom G;
  const double dist = sqrt(d2);
  const double din0 = dx / dist, din1 = dy / dist, din2 = dz / dist;
  const double r_log = 1.0 + log(dist / rgm) / linc;
  double cph, sph, ab;
  const double abmax = fmax(fabs(din0), fabs(din1));
  if (abmax > 1.0e-36) {
    ab = sqrt(add_rn(mul_rn(din0, din0), mul_rn(din1, din1)));
    cph = din0 / ab;
    sph = din1 / ab;
  } else {
    cph = 1.0;
    sph = 0.0;
    ab = 0.0;
  }
  double ct, st;
  const double abcmax = fmax(abmax, fabs(din2));
  if (abcmax > 1.0e-36) {
    const double abc = sqrt(add_rn(mul_rn(ab, ab), mul_rn(din2, din2)));
    ct = din2 / abc;
    st = ab / abc;
  } else {
    ct = 0.0;
    st = 1.0;
  }
  G.x = st * cph;
  G.y = st * sph;
  G.z = ct;
  int i_spl = (int)r_log;
  i_spl = i_spl < 1 ? 1 : i_spl;
  i_spl = i_spl > ngrid - 1 ? ngrid - 1 : i_spl;
  G.i_spl = i_spl;
  const double u = r_log - i_spl;
  G.ta = (u - 1) * (u - 1) * (1 + 2 * u);
  G.tb = (u - 1) * (u - 1) * u;
  G.tc = u * u * (3 - 2 * u);
  G.td = u * u * (u - 1);
  return G;
}

// Near field of one pair by one thread (generic path and dense points): Y_lm by
// recursion fused with the Hermite spline dot.
__device__ double near_field(int lam, int L2, double dx, double dy, double dz, double d2, double rgm, double linc,
                             int ngrid, const double *__restrict__ spl) {
  const NearGeom G = near_geometry(dx, dy, dz, d2, rgm, linc, ngrid);
  const double x = G.x, y = G.y, z = G.z;
  const double *g0 = spl + (long long)2 * L2 * (G.i_spl - 1);
  const double *g1 = g0 + 2 * L2;
  auto S = [&](int i) { return g0[i] * G.ta + g0[i + L2] * G.tb + g1[i] * G.tc + g1[i + L2] * G.td; };
  double acc = 0.0;
  double C = 1.0, Sm = 0.0;
  for (int m = 0; m <= lam; ++m) {
    if (m > 0) {
      const double c2 = x * C - y * Sm;
      Sm = x * Sm + y * C;
      C = c2;
    }
    double q_prev = 0.0, q_prev2 = 0.0;  // Q_{l-1}^m, Q_{l-2}^m
    for (int l = m; l <= lam; ++l) {
      const double ql = (l == m) ? c_DF[m] : c_RA[l][m] * z * q_prev - c_RB[l][m] * q_prev2;
      q_prev2 = q_prev;
      q_prev = ql;
      const int base = l * l + l;
      if (m == 0) {
        acc += c_K[l][0] * ql * S(base);
      } else {
        acc += c_Kcos[l][m] * ql * C * S(base + m);
        acc += c_K[l][m] * ql * Sm * S(base - m);
      }
    }
  }
  return acc;
}

// The same as a call, so that its registers do not count against the far field's.
__device__ __noinline__ double near_field_call(int lam, int L, const double *rec_near, double dx, double dy, double dz,
                                               double d2, const double *__restrict__ spl) {
  return near_field(lam, (L + 1) * (L + 1), dx, dy, dz, d2, rec_near[0], rec_near[1], (int)rec_near[2], spl);
}

// l_atom_max at squared distance d2 (sum_up_whole_potential.cpp:404-411).
__device__ __forceinline__ int lam_at(const double *opr, int lam0, double d2) {
  int l = lam0;
  while (opr[l] < d2 && l > 0) --l;
  return l;
}

// --------------------------------------------------- far-field kernel ---

__device__ __forceinline__ Box empty_box() {
  Box b;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    b.lo[c] = __longlong_as_double(0x7ff0000000000000LL);
    b.hi[c] = -b.lo[c];
  }
  return b;
}

__device__ __forceinline__ Box warp_box(const double (&p)[3], bool live) {
  Box b = empty_box();
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    if (live) b.lo[c] = b.hi[c] = p[c];
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      b.lo[c] = fmin(b.lo[c], __shfl_xor_sync(0xffffffffu, b.lo[c], o));
      b.hi[c] = fmax(b.hi[c], __shfl_xor_sync(0xffffffffu, b.hi[c], o));
    }
  }
  return b;
}

// At plan creation: the valid points' full indices and coordinates in the plan's
// spatial order, and the box of every 32 of them (60 shuffles a warp, in both point
// kernels of every call, before: 60,001 points, 150 atoms, four perturbations 0.71 ->
// 0.67 ms, 2 million points, 500 atoms 8.54 -> 8.50 ms).
__global__ void sumup_gather_points_kernel(int n_valid, const int *__restrict__ map, const int *__restrict__ order,
                                           const double *__restrict__ coord, int *__restrict__ pfull,
                                           double *__restrict__ pxyz, Box *__restrict__ pbox) {
  const int lane = threadIdx.x & 31;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i - lane < n_valid; i += gridDim.x * blockDim.x) {
    double p[3] = {0.0, 0.0, 0.0};
    if (i < n_valid) {
      const int f = map[order[i]];
      pfull[i] = f;
      for (int c = 0; c < 3; ++c) pxyz[i + (long long)c * n_valid] = p[c] = coord[3LL * f + c];
    }
    const bool live = i < n_valid && isfinite(p[0]) && isfinite(p[1]) && isfinite(p[2]);
    const Box b = warp_box(p, live);
    if (lane == 0) pbox[i / 32] = b;
  }
}

// The box of groups [g0, g0 + N) of 32 points (those that exist).
template <int N>
__device__ __forceinline__ Box group_box(const Box *__restrict__ pbox, int g0, int n_valid) {
  Box b = empty_box();
#pragma unroll
  for (int j = 0; j < N; ++j)
    if ((g0 + j) * 32 < n_valid) {
      const Box &o = pbox[g0 + j];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        b.lo[c] = fmin(b.lo[c], __ldg(&o.lo[c]));
        b.hi[c] = fmax(b.hi[c], __ldg(&o.hi[c]));
      }
    }
  return b;
}

// Bounds of the squared distance from (cx, cy, cz) to the box's points, widened
// by 1e-12 (the exactly rounded d2 of a pair is within 1e-15 of the true one).
__device__ __forceinline__ void box_distance(const Box &b, double cx, double cy, double cz, double *near2,
                                             double *far2) {
  const double c[3] = {cx, cy, cz};
  double n2 = 0.0, f2 = 0.0;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const double gap = fmax(fmax(b.lo[k] - c[k], c[k] - b.hi[k]), 0.0);
    const double span = fmax(fabs(b.lo[k] - c[k]), fabs(c[k] - b.hi[k]));
    n2 = fma(gap, gap, n2);
    f2 = fma(span, span, f2);
  }
  *near2 = n2 * (1.0 - 1e-12);
  *far2 = f2 * (1.0 + 1e-12);
}

constexpr int CLS_SKIP = -1, CLS_MIXED = SU_LMAX + 1;  // 0..SU_LMAX: every point far with that l_atom_max

// One record for one warp's box; near: this launch has the near field too.
__device__ __forceinline__ int classify(const Box &b, const double *rec, bool near) {
  double n2, f2;
  box_distance(b, rec[R_X], rec[R_Y], rec[R_Z], &n2, &f2);
  const double mrs = rec[R_MRS];
  if (n2 >= 1e8 || (!near && f2 < mrs)) return CLS_SKIP;  // beyond the far field, or the near-field launch's
  if (!(n2 >= mrs) || !(f2 < 1e8)) return CLS_MIXED;
  // l_atom_max does not grow with the distance
  const int l0 = (int)rec[R_LAM0], l = lam_at(rec + R_OPR, l0, n2);
  return l == lam_at(rec + R_OPR, l0, f2) ? l : CLS_MIXED;
}

// Far field of PPT points per thread, blockIdx.y = perturbation.  A warp owns
// 32 PPT neighbouring points of the plan's spatial order and one of `slices`
// interleaved parts of the records (1, 2 or 4; the parts' sums are added in
// order at the end), so a small point set still fills the chip.
//
// The bound is the FP64 pipe (83 multiply-adds of the polynomial at l = 6 and
// 16 operations of geometry per pair) and the registers' read ports, which hold
// a multiply-add of three distinct operands to two thirds of the pipe: see
// gen_kelvin.py for the order that gets round it, which is why a thread takes
// four points where there are enough.  Everything else is decided once per
// (warp, record): lane s classifies record s of a chunk against the box of the
// warp's points, and a record that is far with one l_atom_max for all of them
// runs without a comparison or a vote (the rule is exact: bounds widened by more
// than the rounding of d2).  A record whose radii the box straddles takes the
// exact per-pair decisions and, if it is safe, one pass per 32 points at the
// largest l_atom_max present in which a lane's higher degrees are multiplied by
// zero (kelvin_masked_eval); an unsafe one takes a pass per l_atom_max.  (A box
// per 32 points as well was slower: 7.9 ms below, and 6% on truncated radii.)
// NEAR: the near field too, each thread its own point's (near_inline says when).
// CODES: the decisions are written as well, each where it is taken: the far field's
// (and, if NEAR, the near field's) here, otherwise the near field's by its launch.
// The sums go to delta_v as additions without a returned value (one per point, so
// nothing depends on an order): a read before them was one latency more per CTA.
// The two record buffers hold as many records as fit (8 at l_max 8, 12 at 6, 32
// below 4): fewer barriers, at which the warps wait for the one with the most
// mixed records (8 for every l_max: 3% more on 2,000 to 100,000 points).
// Measured, 500 atoms, 2 million points, l_max 6: 9.4 ms (two points per thread,
// decisions per pair, near field inside) -> 7.7 ms, 70% of the FP64 peak (two
// points per thread 8.7 ms, in the compiler's order 9.0 ms); with rsqrt() for the
// inverse distances 2% more (l_max 4: 5%) than with a refinement written out here.
template <int PPT, bool CODES, bool NEAR>
__global__ void __launch_bounds__(SU_THREADS, PPT == 4 ? 4 : (PPT == 2 ? 5 : 6))
    sumup_far_kernel(int n_valid, int n_full, const int *__restrict__ order, const int *__restrict__ pfull,
                     const double *__restrict__ pxyz, const Box *__restrict__ pbox, int n_chp, int L,
                     const double *recs, int slices, double *dv, unsigned char *codes,
                     const double *__restrict__ spline, int n_atoms, int n_hartree_grid) {
  const int RS = rec_stride(L), CO = rec_coef_off(L);
  __shared__ __align__(16) double srec[2][SU_CHUNK * rec_stride(SU_LMAX)];
  const int CH = min(32, (SU_CHUNK * rec_stride(SU_LMAX) / RS) & ~3);  // records per chunk
  __shared__ double part[SU_THREADS / 32][32 * PPT];
  __shared__ Box boxes[SU_THREADS / 32];  // read by the classification only: not worth registers
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, t = blockIdx.y;
  const unsigned FULL = 0xffffffffu;
  const int slice = warp & (slices - 1);
  const int base = (blockIdx.x * (SU_THREADS / 32) / slices + warp / slices) * (32 * PPT);

  int vidx[PPT], full[PPT];
  double px[PPT], py[PPT], pz[PPT], v[PPT];
  bool valid[PPT], live[PPT];
#pragma unroll
  for (int j = 0; j < PPT; ++j) {
    const int slot = base + j * 32 + lane;
    valid[j] = slot < n_valid;
    vidx[j] = CODES && valid[j] ? order[slot] : 0;
    full[j] = valid[j] ? pfull[slot] : 0;
    px[j] = valid[j] ? pxyz[slot] : 0.0;
    py[j] = valid[j] ? pxyz[slot + (long long)n_valid] : 0.0;
    pz[j] = valid[j] ? pxyz[slot + 2LL * n_valid] : 0.0;
    live[j] = valid[j] && isfinite(px[j]) && isfinite(py[j]) && isfinite(pz[j]);
    v[j] = 0.0;
  }
  {
    const Box b = group_box<PPT>(pbox, base / 32, n_valid);
    if (lane == 0) boxes[warp] = b;
    __syncwarp();
  }
  bool any_live = false;
#pragma unroll
  for (int j = 0; j < PPT; ++j) any_live = any_live || live[j];
  const bool work = CODES || __any_sync(FULL, any_live);
  grid_wait();  // the records; only the plan's points are read before
  grid_release();

  const double *src = recs + (long long)RS * n_chp * t;
  auto load = [&](int c0, int buf) {  // records c0.. of this perturbation (RS is even: 16-byte copies)
    const int n = min(CH, n_chp - c0) * RS / 2;
    const double *from = src + (long long)RS * c0;
    for (int e = tid; e < n; e += SU_THREADS) cp_async_16(&srec[buf][2 * e], from + 2 * e, 16);
    cp_async_commit();
  };
  load(0, 0);
  for (int c0 = 0, buf = 0; c0 < n_chp; c0 += CH, buf ^= 1) {
    const int nch = min(CH, n_chp - c0);
    cp_async_wait<0>();
    __syncthreads();  // this chunk is there; every warp is done with the other buffer
    if (c0 + CH < n_chp) load(c0 + CH, buf ^ 1);
    if (!work) continue;
    const double *chunk = srec[buf];
    const int cls_mine = lane < nch ? classify(boxes[warp], chunk + lane * RS, NEAR) : CLS_SKIP;
    for (int s = slice; s < nch; s += slices) {
      const double *rec = chunk + s * RS;
      const int cls = __shfl_sync(FULL, cls_mine, s);
      if (CODES && cls != CLS_MIXED) {
#pragma unroll
        for (int j = 0; j < PPT; ++j)
          if (valid[j])
            codes[vidx[j] + (long long)n_valid * ((c0 + s) + (long long)n_chp * t)] =
                (unsigned char)(live[j] && cls != CLS_SKIP ? 16 + cls : 0);
      }
      if (cls == CLS_SKIP) continue;
      const double cx = rec[R_X], cy = rec[R_Y], cz = rec[R_Z];
      if (cls < CLS_MIXED) {
        double ux[PPT], uy[PPT], uz[PPT], P[PPT], rinv[PPT];
#pragma unroll
        for (int j = 0; j < PPT; ++j) {
          const double dx = px[j] - cx, dy = py[j] - cy, dz = pz[j] - cz;
          rinv[j] = rsqrt(fma(dz, dz, fma(dy, dy, dx * dx)));
          const double ir2 = rinv[j] * rinv[j];
          ux[j] = dx * ir2;
          uy[j] = dy * ir2;
          uz[j] = dz * ir2;
        }
        kelvin_eval<PPT>(cls, rec + CO, ux, uy, uz, P);
#pragma unroll
        for (int j = 0; j < PPT; ++j) v[j] = fma(P[j], rinv[j], v[j]);
        continue;
      }
      const double mrs = rec[R_MRS];
      const int lam0 = (int)rec[R_LAM0];
      const bool safe = rec[R_SAFE] != 0.0;
#pragma unroll 1
      for (int j = 0; j < PPT; ++j) {  // one body for all points: selects instead of indexed registers
        double x = px[0], y = py[0], z = pz[0];
        bool val = valid[0];
        int vi = vidx[0];
#pragma unroll
        for (int i = 1; i < PPT; ++i)
          if (j == i) {
            x = px[i];
            y = py[i];
            z = pz[i];
            val = valid[i];
            vi = vidx[i];
          }
        const double dx = sub_rn(x, cx), dy = sub_rn(y, cy), dz = sub_rn(z, cz);
        const double d2 = add_rn(add_rn(mul_rn(dx, dx), mul_rn(dy, dy)), mul_rn(dz, dz));
        const int lam = lam_at(rec + R_OPR, lam0, d2);
        const bool is_near = val && d2 < mrs, is_far = val && !is_near && d2 < 1e8;
        if (CODES && val)
          codes[vi + (long long)n_valid * ((c0 + s) + (long long)n_chp * t)] =
              (unsigned char)(is_far ? 16 + lam : (NEAR && is_near ? 1 + lam : 0));
        const double ri = is_far ? rsqrt(d2) : 0.0;
        const double ir2 = ri * ri;
        const double ux = is_far ? dx * ir2 : 0.0, uy = is_far ? dy * ir2 : 0.0, uz = is_far ? dz * ir2 : 0.0;
        double P = 0.0, sum = 0.0;
        bool pend = is_far;
        while (__any_sync(FULL, pend)) {
          const int top = __reduce_max_sync(FULL, pend ? lam : -1);
          kelvin_masked_eval(top, rec + CO, &ux, &uy, &uz, min(lam, top), &P);
          if (pend && (safe || lam == top)) {
            sum = P * ri;
            pend = false;
          }
        }
        if (NEAR && is_near)
          sum = near_field_call(lam, L, rec + R_RGM, dx, dy, dz, d2,
                                spline + 2LL * (L + 1) * (L + 1) * n_hartree_grid *
                                             ((long long)rec[R_ATOM] + (long long)n_atoms * t));
        if (is_far || (NEAR && is_near)) {
#pragma unroll
          for (int i = 0; i < PPT; ++i)
            if (j == i) v[i] += sum;
        }
      }
    }
  }
  if (slices > 1) {
#pragma unroll
    for (int j = 0; j < PPT; ++j) part[warp][j * 32 + lane] = v[j];
    __syncthreads();
    if (slice != 0) return;
#pragma unroll
    for (int j = 0; j < PPT; ++j)
      for (int k = 1; k < slices; ++k) v[j] += part[warp + k][j * 32 + lane];
  }
#pragma unroll
  for (int j = 0; j < PPT; ++j)
    if (live[j]) atomicAdd(dv + full[j] + (long long)n_full * t, v[j]);
}

// -------------------------------------------------- near-field kernel ---

constexpr int NF_THREADS = 128;
constexpr int NF_MAX_SLICES = 8;  // warps that may share 32 points
constexpr int NF_PAIRS = 32;      // pairs evaluated together, one per lane

struct NearWarp {
  double x[NF_PAIRS], y[NF_PAIRS], z[NF_PAIRS];  // unit vectors
  double h[NF_PAIRS][4];                         // Hermite weights
  const double *run[NF_PAIRS];                   // the 4 (L + 1)^2 spline values of the interval
  double val[NF_PAIRS];
  int lam[NF_PAIRS];
  int owner[2 * NF_PAIRS], slot[2 * NF_PAIRS];  // pairs found: lane of the point, centre slot
  unsigned touched;
};

// Near field of 32 neighbouring points per warp, blockIdx.y = perturbation.  The
// lanes test the centres against the box of the points, 32 at a time; only the
// few that can be near are looked at per point (exact d2), and the near pairs go
// to a queue that is evaluated 32 pairs at a time, so that sparse hits cost no
// more than dense ones.  The geometry (square roots, divisions, a logarithm)
// takes one lane per pair; the sum over (l, m) eight lanes, lane m the orders +-m
// (lane 0 also +-8): for every l their loads are one contiguous stretch of the
// pair's run of 4 (L + 1)^2 values and none waits for the recursion.
// What bounds it is L1 (85% busy): a pair reads 1.6 KB of spline (l_max 6).  Whole
// warps along a run, with the harmonics in shared memory, had fewer L1 lookups but
// were slower (1.57 ms against 0.94 ms on 2 million points, 500 atoms).  Where the
// points are few, 2 to 8 warps share 32 points and take the candidate centres in
// turn (2,000 points, 20 atoms: 76 us with one).  Every sum has a fixed order.
template <int L, bool CODES>
__global__ void __launch_bounds__(32 * NF_MAX_SLICES)
    sumup_near_kernel(int n_valid, int n_full, const int *__restrict__ pfull, const double *__restrict__ pxyz,
                      const Box *__restrict__ pbox, int n_chp, int n_atoms, int n_hartree_grid, int slices,
                      const double *recs, const double4 *heads, const double *__restrict__ spline, double *dv,
                      const int *__restrict__ order, unsigned char *codes) {
  constexpr int RS = rec_stride(L), L2 = (L + 1) * (L + 1);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double s_ra[L2], s_rb[L2], s_k[L2];  // (l, m) at l (L + 1) + m
  const unsigned FULL = 0xffffffffu;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, t = blockIdx.y;
  NearWarp &W = reinterpret_cast<NearWarp *>(smem_raw)[warp];
  for (int e = tid; e < L2; e += blockDim.x) {
    const int l = e / (L + 1), m = e % (L + 1);
    s_k[e] = d_near_tables[0][l][m];
    s_ra[e] = d_near_tables[1][l][m];
    s_rb[e] = d_near_tables[2][l][m];
  }
  __syncthreads();
  const int slice = warp & (slices - 1);
  const int pt = ((blockIdx.x * (blockDim.x >> 5) + warp) / slices) * 32 + lane;
  const bool valid = pt < n_valid;
  const double px = valid ? pxyz[pt] : 0.0, py = valid ? pxyz[pt + (long long)n_valid] : 0.0,
               pz = valid ? pxyz[pt + 2LL * n_valid] : 0.0;
  const Box box = group_box<1>(pbox, pt / 32, n_valid);
  grid_wait();  // the far field's sums (and, before them, the records); only plan data is read before
  const int m8 = lane & 7, grp = lane >> 3;
  double v = 0.0;
  bool touched = false;

  auto evaluate = [&](int n) {  // the first n (<= 32) pairs of the queue
    __syncwarp();
    {
      const bool has = lane < n;
      const int o = has ? W.owner[lane] : lane;
      const double x = __shfl_sync(FULL, px, o), y = __shfl_sync(FULL, py, o), z = __shfl_sync(FULL, pz, o);
      if (has) {
        const double *rec = recs + (long long)RS * (W.slot[lane] + (long long)n_chp * t);
        const double dx = sub_rn(x, rec[R_X]), dy = sub_rn(y, rec[R_Y]), dz = sub_rn(z, rec[R_Z]);
        const double d2 = add_rn(add_rn(mul_rn(dx, dx), mul_rn(dy, dy)), mul_rn(dz, dz));
        const NearGeom G = near_geometry(dx, dy, dz, d2, rec[R_RGM], rec[R_LINC], (int)rec[R_NGRID]);
        W.x[lane] = G.x;
        W.y[lane] = G.y;
        W.z[lane] = G.z;
        W.h[lane][0] = G.ta;
        W.h[lane][1] = G.tb;
        W.h[lane][2] = G.tc;
        W.h[lane][3] = G.td;
        const int lam = lam_at(rec + R_OPR, (int)rec[R_LAM0], d2);
        W.lam[lane] = lam;
        if (CODES)
          codes[order[pt - lane + o] + (long long)n_valid * (W.slot[lane] + (long long)n_chp * t)] =
              (unsigned char)(1 + lam);
        W.run[lane] = spline + (long long)2 * L2 *
                                   (n_hartree_grid * ((long long)rec[R_ATOM] + (long long)n_atoms * t) + G.i_spl - 1);
      }
    }
    __syncwarp();
    for (int k0 = 0; k0 < n; k0 += 4) {
      const int k = k0 + grp;
      double acc = 0.0;
      if (k < n) {
        const double *run = W.run[k];
        const double z = W.z[k], ta = W.h[k][0], tb = W.h[k][1], tc = W.h[k][2], td = W.h[k][3];
        const int lam = W.lam[k];
        auto S = [&](int i) {
          return __ldg(run + i) * ta + __ldg(run + i + L2) * tb + __ldg(run + i + 2 * L2) * tc +
                 __ldg(run + i + 3 * L2) * td;
        };
        // (x + i y)^m8 and ^8 by squaring
        double C = 1.0, Sn = 0.0, bc = W.x[k], bs = W.y[k];
#pragma unroll
        for (int bit = 1; bit < 8; bit <<= 1) {
          if (m8 & bit) {
            const double c2 = C * bc - Sn * bs;
            Sn = C * bs + Sn * bc;
            C = c2;
          }
          const double b2 = bc * bc - bs * bs;
          bs = 2.0 * bc * bs;
          bc = b2;
        }
        if (m8 & 1) C = -C;  // the cosine terms carry (-1)^m
        double q = 0.0, q1 = 0.0;
#pragma unroll
        for (int l = 0; l <= L; ++l) {
          if (m8 <= l && l <= lam) {
            const int e = l * (L + 1) + m8;
            const double qn = l == m8 ? c_DF[m8] : s_ra[e] * z * q - s_rb[e] * q1;
            q1 = q;
            q = qn;
            double term = C * S(l * l + l + m8);
            if (m8 > 0) term += Sn * S(l * l + l - m8);
            acc += s_k[e] * q * term;
          }
        }
        if (L >= 8 && m8 == 0 && lam >= 8) acc += c_K[8][8] * c_DF[8] * (bc * S(80) + bs * S(64));
      }
#pragma unroll
      for (int o = 4; o; o >>= 1) acc += __shfl_xor_sync(FULL, acc, o);
      if (m8 == 0 && k < n) W.val[k] = acc;
    }
    __syncwarp();
    for (int k = 0; k < n; ++k)
      if (W.owner[k] == lane) {
        v += W.val[k];
        touched = true;
      }
    __syncwarp();
  };

  int queued = 0, seen = 0;
  for (int c0 = 0; c0 < n_chp; c0 += 32) {
    bool cand = false;
    if (c0 + lane < n_chp) {
      const double4 h = heads[c0 + lane + (long long)n_chp * t];
      double n2, f2;
      box_distance(box, h.x, h.y, h.z, &n2, &f2);
      cand = n2 < h.w;
    }
    for (unsigned todo = __ballot_sync(FULL, cand); todo; todo &= todo - 1) {
      if ((seen++ & (slices - 1)) != slice) continue;
      const int s = c0 + __ffs(todo) - 1;
      const double4 h = heads[s + (long long)n_chp * t];
      const double dx = sub_rn(px, h.x), dy = sub_rn(py, h.y), dz = sub_rn(pz, h.z);
      const double d2 = add_rn(add_rn(mul_rn(dx, dx), mul_rn(dy, dy)), mul_rn(dz, dz));
      const bool is_near = valid && d2 < h.w;
      const unsigned nm = __ballot_sync(FULL, is_near);
      if (is_near) {
        const int at = queued + __popc(nm & ((1u << lane) - 1));
        W.owner[at] = lane;
        W.slot[at] = s;
      }
      queued += __popc(nm);
      if (queued >= NF_PAIRS) {
        evaluate(NF_PAIRS);
        queued -= NF_PAIRS;
        if (lane < queued) {  // the rest moves up
          W.owner[lane] = W.owner[NF_PAIRS + lane];
          W.slot[lane] = W.slot[NF_PAIRS + lane];
        }
      }
    }
  }
  if (queued > 0) evaluate(queued);
  if (slices > 1) {
    W.val[lane] = v;
    const unsigned any = __ballot_sync(FULL, touched);
    if (lane == 0) W.touched = any;
    __syncthreads();
    if (slice != 0) return;
    for (int k = 1; k < slices; ++k) {
      const NearWarp &O = reinterpret_cast<NearWarp *>(smem_raw)[warp + k];
      if (O.touched >> lane & 1) {
        v += O.val[lane];
        touched = true;
      }
    }
  }
  if (touched) atomicAdd(dv + pfull[pt] + (long long)n_full * t, v);
}

// ------------------------------------------------------ generic kernel ---

// Mirrors the reference loop exactly, including the far field's use of the
// loop slot as centre (sum_up_whole_potential.cpp:91-187 called with i_center + 1).
__global__ void __launch_bounds__(SU_THREADS)
    sumup_generic_kernel(int n_valid, int n_full, const int *__restrict__ map, const double *__restrict__ coord,
                         int n_active, int n_chp, int n_atoms, int L, int L2, int n_hartree_grid, int hfla,
                         const int *__restrict__ chp, const int *__restrict__ c2a, const int *__restrict__ species,
                         const int *__restrict__ species_center, const int *__restrict__ l_hartree,
                         const int *__restrict__ n_grid, const double *__restrict__ rgm,
                         const double *__restrict__ linc, const double *__restrict__ cc_xyz,
                         const double *__restrict__ mrs, const double *__restrict__ opr,
                         const int *__restrict__ ncc, const int *__restrict__ icc_packed,
                         const int *__restrict__ ijkmax, int mc_dim, const double *__restrict__ mc,
                         const double *__restrict__ spline, double *__restrict__ dv,
                         unsigned char *__restrict__ codes) {
  const int iv = blockIdx.x * SU_THREADS + threadIdx.x;
  if (iv >= n_valid) return;
  const int f = map[iv];
  const double px = coord[3LL * f], py = coord[3LL * f + 1], pz = coord[3LL * f + 2];
  for (int t = 0; t < n_active; ++t) {
    double v = dv[f + (long long)n_full * t];
    for (int ic = 0; ic < n_chp; ++ic) {
      const int cur = chp[ic] - 1;
      const int atom = c2a[cur] - 1;
      const double dx = sub_rn(px, cc_xyz[3 * cur]), dy = sub_rn(py, cc_xyz[3 * cur + 1]),
                   dz = sub_rn(pz, cc_xyz[3 * cur + 2]);
      const double d2 = add_rn(add_rn(mul_rn(dx, dx), mul_rn(dy, dy)), mul_rn(dz, dz));
      int lam = l_hartree[species[atom] - 1];
      const double *o = opr + (long long)(L + 1) * (atom + (long long)n_atoms * t);
      while (o[lam] < d2 && lam > 0) --lam;
      unsigned char code = 0;
      if (d2 < mrs[atom + (long long)n_atoms * t]) {
        const int sp = species_center[cur] - 1;
        const double *spl = spline + (long long)2 * L2 * n_hartree_grid * (atom + (long long)n_atoms * t);
        v += near_field(lam, L2, dx, dy, dz, d2, rgm[sp], linc[sp], n_grid[sp], spl);
        code = (unsigned char)(1 + lam);
      } else if (d2 < 1e8) {
        const double dist = sqrt(d2);
        double Fp[2 * SU_LMAX + 4];
        const double dsq = dist * dist;
        int k = 1;
        Fp[0] = 1.0 / dist;
        for (int l = 1; l <= lam + hfla; ++l) {
          k -= 2;
          Fp[l] = Fp[l - 1] * k / dsq;
        }
        const double ex = px - cc_xyz[3 * ic], ey = py - cc_xyz[3 * ic + 1], ez = pz - cc_xyz[3 * ic + 2];
        int maxp = ijkmax[3 * lam];
        maxp = max(maxp, ijkmax[3 * lam + 1]);
        maxp = max(maxp, ijkmax[3 * lam + 2]);
        double pw[3][2 * SU_LMAX + 2];
        pw[0][0] = pw[1][0] = pw[2][0] = 1.0;
        for (int i = 1; i <= maxp; ++i) {
          pw[0][i] = ex * pw[0][i - 1];
          pw[1][i] = ey * pw[1][i - 1];
          pw[2][i] = ez * pw[2][i - 1];
        }
        const double *m = mc + (long long)mc_dim * ((c2a[ic] - 1) + (long long)n_atoms * t);
        double dpot = 0.0;
        const int nend = ncc[lam];
        for (int n = 0; n < nend; ++n) {
          const int pk = icc_packed[n];
          const int ii = pk & 255, jj = (pk >> 8) & 255, kk = (pk >> 16) & 255, nn = (pk >> 24) & 255;
          dpot += pw[0][ii] * pw[1][jj] * pw[2][kk] * Fp[nn] * m[n];
        }
        v += dpot;
        code = (unsigned char)(16 + lam);
      }
      if (codes) codes[iv + (long long)n_valid * (ic + (long long)n_chp * t)] = code;
    }
    dv[f + (long long)n_full * t] = v;
  }
}

int launch_prep(const SumupPlan &P, int n_active, const int *lhmfd, const double *mrs, const double *opr,
                const double *Q, cudaStream_t stream) {
  sumup_prep_kernel<<<dim3(std::max(P.n_chp, P.n_atoms), n_active), 128, 0, stream>>>(
      P.L, P.lma, P.n_atoms, P.n_chp, P.n_coef, P.rs, P.d_chp, P.d_c2a, P.d_species, P.d_species_center,
      P.d_l_hartree, P.d_n_grid, P.d_rgm, P.d_linc, P.d_cc_xyz, mrs, opr, lhmfd, Q, P.d_slot, P.d_conv_ptr,
      P.d_conv_lm, P.d_conv_fc, P.d_recs, P.d_heads, P.d_err);
  FRPA_LAUNCH_CHECK();
  return FRPA_OK;
}

template <bool CODES>
int launch_near(const SumupPlan &P, int n_active, const double *spline, double *dv, unsigned char *codes,
                cudaStream_t stream) {
  int n_sm = 148;
  FRPA_CUDA_TRY(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, P.device));
  const int groups = ceil_div(P.n_valid_points, 32);
  // candidate centres split over up to 8 warps until the warps fill the chip (16 per SM)
  int slices = 1, threads = NF_THREADS;
  while ((long long)groups * n_active * slices < 16LL * n_sm && slices < NF_MAX_SLICES) slices *= 2;
  if (32 * slices > threads) threads = 32 * slices;
  const dim3 grid(ceil_div(groups, threads / 32 / slices), n_active);
  const size_t smem = (threads / 32) * sizeof(NearWarp);
  switch (P.L) {
#define FRPA_NEAR_CASE(LL)                                                                                        \
  case LL:                                                                                                        \
    FRPA_CUDA_TRY(launch_chained(sumup_near_kernel<LL, CODES>, grid, threads, smem, stream, P.n_valid_points,     \
                                 P.n_full_points, P.d_pfull, P.d_pxyz, P.d_pbox, P.n_chp, P.n_atoms,              \
                                 P.n_hartree_grid, slices, P.d_recs, P.d_heads, spline, dv, P.d_order, codes));   \
    break;
    FRPA_NEAR_CASE(0) FRPA_NEAR_CASE(1) FRPA_NEAR_CASE(2) FRPA_NEAR_CASE(3) FRPA_NEAR_CASE(4)
    FRPA_NEAR_CASE(5) FRPA_NEAR_CASE(6) FRPA_NEAR_CASE(7) FRPA_NEAR_CASE(8)
#undef FRPA_NEAR_CASE
    default:
      return fail(FRPA_ERR_UNSUPPORTED, "sum-up: l_pot_max %d above %d", P.L, SU_LMAX);
  }
  FRPA_LAUNCH_CHECK();
  return FRPA_OK;
}

template <int PPT, bool CODES, bool NEAR>
int launch_far(const SumupPlan &P, int n_active, int slices, const double *spline, double *dv, unsigned char *codes,
               cudaStream_t stream) {
  const int groups = SU_THREADS / 32 / slices;  // point groups per CTA
  const dim3 grid(ceil_div(ceil_div(P.n_valid_points, 32 * PPT), groups), n_active);
  FRPA_CUDA_TRY(launch_chained(sumup_far_kernel<PPT, CODES, NEAR>, grid, SU_THREADS, 0, stream, P.n_valid_points,
                               P.n_full_points, P.d_order, P.d_pfull, P.d_pxyz, P.d_pbox, P.n_chp, P.L, P.d_recs,
                               slices, dv, codes, spline, P.n_atoms, P.n_hartree_grid));
  FRPA_LAUNCH_CHECK();
  return FRPA_OK;
}

// Where a warp's 32 points mostly share a centre's near sphere, each thread adds its
// own near field in the far-field launch: the launch of its own (10 us and a chain of
// latencies per group of points) pays only where a warp's near pairs are few or their
// sums long.  Measured, us, own launch / inline:
//   points per centre        1 centre                     10 centres      50 centres      200 centres
//   l_max 4: 2,000, 16,000   21 / 12, 26 / 17 (2)         31 / 20, 72 / 51  106 / 91, 370 / 311  562 / 513 (2,000)
//   l_max 2: 2,000, 16,000   18 / 13, 20 / 13 (2)         24 / 15, 51 / 35  75 / 60, 213 / 201   350 / 369 (2,000)
//   l_max 5: 2,000, 64,000   - , 24 / 18                  43 / 32, 116 / 108 (8)  167 / 196 (2,000)
//   l_max 6: 8,000, 64,000   26 / 19, 28 / 20             72 / 61, 134 / 159 (8)  312 / 397 (8,000)
// (in brackets: at another number of centres, or the one size).  Above l_max 4 it also
// pays around 2 to 8 centres while the points are enough for one warp to have its own
// and few enough for about one round of warps, which the chain of latencies then sets:
// 3 centres, 33,000 points each, l_max 6 58 / 43, l_max 8 87 / 65 (8,000 each: 29 / 39,
// 43 / 60; 128,000 each: 72 / 80, 111 / 129); 8 centres, 16,000 each 92 / 70, 139 / 106
// (32,000 each: 111 / 104, 164 / 157; 64,000 each: 134 / 159).  Not at l_max 7, whose
// orders fill the own launch's eight lanes: 5 centres, 40,000 each 93 / 113.
bool near_inline(int L, int n_points, int n_active, int n_centres) {
  const int most = L <= 4 ? 128 : (L == 5 ? 16 : 1);
  if (n_centres <= most && n_points >= 2048LL * n_centres) return true;
  if (L <= 4 && n_centres == 1) return true;  // 64 points: 10.6 / 8.3
  const long long points = (long long)n_points * n_active;
  return L != 7 && n_centres <= 8 && n_points >= 8192LL * n_centres && points >= 40000 && points <= 262144;
}

template <bool CODES>
int launch_fast(const SumupPlan &P, int n_active, const double *spline, double *dv, unsigned char *codes,
                cudaStream_t stream) {
  int n_sm = 148;
  FRPA_CUDA_TRY(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, P.device));
  // four points per thread share every coefficient load; the fewer warps that
  // leaves, the more the records are split (over 2, then 4 warps), then the
  // fewer points a thread takes, until the warps fill the chip twice (16 per SM)
  const long long want = 2LL * 16 * n_sm;
  int ppt = 4, slices = 1;
  auto warps = [&] { return (long long)ceil_div(P.n_valid_points, 32 * ppt) * n_active * slices; };
  while (warps() < want && slices < 4 && P.n_chp >= 4 * slices) slices *= 2;
  while (warps() < want && ppt > 1) ppt /= 2;
  if (near_inline(P.L, P.n_valid_points, n_active, P.n_chp)) {
    if (ppt > 1) return launch_far<2, CODES, true>(P, n_active, slices, spline, dv, codes, stream);
    return launch_far<1, CODES, true>(P, n_active, slices, spline, dv, codes, stream);
  }
  if (ppt == 4)
    FRPA_TRY((launch_far<4, CODES, false>(P, n_active, slices, spline, dv, codes, stream)));
  else if (ppt == 2)
    FRPA_TRY((launch_far<2, CODES, false>(P, n_active, slices, spline, dv, codes, stream)));
  else
    FRPA_TRY((launch_far<1, CODES, false>(P, n_active, slices, spline, dv, codes, stream)));
  return launch_near<CODES>(P, n_active, spline, dv, codes, stream);
}

// -------------------------------------------------------- adjoint (dQ) ---

// The coefficients with x exponent in [A0, A1) for degrees <= L: how many, and
// the position of (a, b, c) among them.
template <int L, int A0, int A1>
struct CoefRange {
  static constexpr int before(int a) {  // coefficients with x exponent in [A0, a)
    int n = 0;
    for (int q = A0; q < a; ++q) n += (L - q + 1) * (L - q + 2) / 2;
    return n;
  }
  static constexpr int count = before(A1);
  static constexpr int index(int a, int b, int c) {
    int n = before(a);
    for (int q = 0; q < b; ++q) n += L - a - q + 1;
    return n + c;
  }
};

// acc(a, b, c) += w x^a y^b z^c for the range's coefficients of degree <= LAM
template <int L, int A0, int A1, int LAM>
__device__ __forceinline__ void dcoef_add(double *acc, double w, double x, double y, const double *zp) {
  using R = CoefRange<L, A0, A1>;
  double wa = w;
#pragma unroll
  for (int a = 0; a < A1 && a <= LAM; ++a) {
    if (a >= A0) {
      double wab = wa;
#pragma unroll
      for (int b = 0; a + b <= LAM; ++b) {
#pragma unroll
        for (int c = 0; a + b + c <= LAM; ++c) acc[R::index(a, b, c)] = fma(wab, zp[c], acc[R::index(a, b, c)]);
        wab *= y;
      }
    }
    wa *= x;
  }
}

template <int L, int A0, int A1, int... LAM>
__device__ __forceinline__ void dcoef_switch(std::integer_sequence<int, LAM...>, int lam, double *acc, double w,
                                             double x, double y, const double *zp) {
  ((lam == LAM ? dcoef_add<L, A0, A1, LAM>(acc, w, x, y, zp) : (void)0), ...);
}

// One pass over a block's points for the coefficients with x exponent in
// [A0, A1): each thread adds its points in registers, then the block's sums go
// to part[] (recursive halving over the lanes, the warps in order).
template <int L, int A0, int A1>
__device__ __forceinline__ void dcoef_pass(int n_valid, const int *__restrict__ pfull,
                                           const double *__restrict__ pxyz, const double *__restrict__ rec,
                                           const double *__restrict__ gt, int p_begin, int p_end, double *red,
                                           double *__restrict__ part) {
  using R = CoefRange<L, A0, A1>;
  constexpr int N = R::count, NP = (N + 31) / 32 * 32;
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double cx = rec[R_X], cy = rec[R_Y], cz = rec[R_Z], mrs = rec[R_MRS];
  const int lam0 = (int)rec[R_LAM0];
  double acc[NP];
#pragma unroll
  for (int k = 0; k < NP; ++k) acc[k] = 0.0;
  // a point's loads are issued one turn ahead, its full index two turns
  struct Point {
    double x, y, z, g;
  };
  const int first = p_begin + warp * 32 + lane;
  auto index = [&](int iv) { return iv < p_end ? __ldg(pfull + iv) : 0; };
  auto fetch = [&](int iv, int f) {
    Point P{0.0, 0.0, 0.0, 0.0};
    if (iv < p_end) {
      P.x = __ldg(pxyz + iv);
      P.y = __ldg(pxyz + iv + (long long)n_valid);
      P.z = __ldg(pxyz + iv + 2LL * n_valid);
      P.g = __ldg(gt + f);
    }
    return P;
  };
  Point next = fetch(first, index(first));
  int f_next = index(first + SU_THREADS);
  for (int iv = first; iv - lane < p_end; iv += SU_THREADS) {
    const bool in = iv < p_end;
    const Point P = next;
    next = fetch(iv + SU_THREADS, f_next);
    f_next = index(iv + 2 * SU_THREADS);
    const double dx = sub_rn(P.x, cx), dy = sub_rn(P.y, cy), dz = sub_rn(P.z, cz);
    const double d2 = add_rn(add_rn(mul_rn(dx, dx), mul_rn(dy, dy)), mul_rn(dz, dz));
    const bool is_far = in && !(d2 < mrs) && d2 < 1e8;
    unsigned todo = __ballot_sync(FULL, is_far);
    if (!todo) continue;
    const int lam = lam_at(rec + R_OPR, lam0, d2);
    const double ri = is_far ? rsqrt(d2) : 0.0, ir2 = ri * ri;
    const double gw = is_far ? P.g * ri : 0.0;
    const double ux = dx * ir2, uy = dy * ir2, uz = dz * ir2;
    // neighbouring points mostly share l_atom_max; each value present is one
    // pass, the other lanes adding zeros
    while (todo) {
      const int sel = __shfl_sync(FULL, lam, __ffs(todo) - 1);
      const bool mine = is_far && lam == sel;
      todo &= ~__ballot_sync(FULL, mine);
      const double z = mine ? uz : 0.0;
      double zp[L + 1];
      zp[0] = 1.0;
#pragma unroll
      for (int e = 1; e <= L; ++e) zp[e] = zp[e - 1] * z;
      dcoef_switch<L, A0, A1>(std::make_integer_sequence<int, L + 1>{}, sel, acc, mine ? gw : 0.0, mine ? ux : 0.0,
                              mine ? uy : 0.0, zp);
    }
  }
#pragma unroll
  for (int k0 = 0; k0 < NP; k0 += 32) {
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      const bool upper = (lane & o) != 0;
#pragma unroll
      for (int i = 0; i < o; ++i) {
        const double keep = upper ? acc[k0 + i + o] : acc[k0 + i], give = upper ? acc[k0 + i] : acc[k0 + i + o];
        acc[k0 + i] = keep + __shfl_xor_sync(FULL, give, o);
      }
    }
    red[warp * NP + k0 + lane] = acc[k0];  // lane holds coefficient k0 + lane
  }
  __syncthreads();
  for (int k = threadIdx.x; k < N; k += SU_THREADS) {
    double v = 0.0;
    for (int w = 0; w < SU_THREADS / 32; ++w) v += red[w * NP + k];
    part[CoefRange<L, 0, L + 1>::before(A0) + k] = v;
  }
  __syncthreads();
}

// x exponents of the second pass on: one pass up to l_max 6 (84 sums in
// registers), two above (64 + 56 and 81 + 84)
__host__ __device__ constexpr int dcoef_split(int L) { return L <= 6 ? L + 1 : 2; }

// part[z, t, slot, (a, b, c)] = sum over point block z of g(p, t) u^(a,b,c) / r
// over the far-field pairs whose l_atom_max reaches the degree (the derivative of
// the far field's polynomial with respect to its coefficients), in a fixed order.
// The bound is the FP64 pipe: a multiply-add per coefficient, a multiplication per
// (a, b) and the geometry, about 140 operations a pair at l_max 6 (the first form
// walked the points once per 32 coefficients, with two multiplications and a
// multiply-add each: 1.05 ms on 100 atoms and 200,000 points, now 0.37 ms).
template <int L>
__global__ void __launch_bounds__(SU_THREADS, 2)
    sumup_dcoef_kernel(int n_valid, int n_full, const int *__restrict__ pfull, const double *__restrict__ pxyz,
                       int n_chp, const double *__restrict__ recs, const double *__restrict__ g, int pts_per_block,
                       double *__restrict__ part) {
  constexpr int NK = kelvin_count(L), A1 = dcoef_split(L);
  __shared__ double red[SU_THREADS / 32 * 96];
  const int slot = blockIdx.x, t = blockIdx.y;
  const int p_begin = blockIdx.z * pts_per_block, p_end = min(n_valid, p_begin + pts_per_block);
  const double *rec = recs + (long long)rec_stride(L) * (slot + (long long)n_chp * t);
  double *out = part + (long long)NK * (slot + (long long)n_chp * (t + (long long)gridDim.y * blockIdx.z));
  const double *gt = g + (long long)n_full * t;
  dcoef_pass<L, 0, A1>(n_valid, pfull, pxyz, rec, gt, p_begin, p_end, red, out);
  if constexpr (A1 <= L)
    dcoef_pass<L, A1, L + 1>(n_valid, pfull, pxyz, rec, gt, p_begin, p_end, red, out);
}

constexpr int DQ_THREADS = 256;
static_assert(DQ_THREADS >= kelvin_count(SU_LMAX), "a thread per coefficient");

// dQ of one atom and perturbation: its slots' coefficient gradients (in a fixed
// order), back through the Kelvin conversion and cc to (l, m),
// where the forward kept the moment (l <= l_hartree_max_far_distance,
// |Q| > 1e-10).  A warp per (l, m), lanes over its table rows.  Perturbations
// past n_active get zeros.
__global__ void __launch_bounds__(DQ_THREADS)
    sumup_dq_kernel(int n_atoms, int L, int n_chp, int n_coef, int n_active, int nz, const int *__restrict__ slot_ptr,
                    const int *__restrict__ slots, const int *__restrict__ lm_ptr, const int *__restrict__ lm_row,
                    const int *__restrict__ convT_ptr, const int *__restrict__ convT_k,
                    const double *__restrict__ convT_f, const double *__restrict__ cc, const int *__restrict__ lhmfd,
                    const double *__restrict__ Q, const double *__restrict__ part, double *__restrict__ dQ) {
  __shared__ double dc[(SU_LMAX + 1) * (SU_LMAX + 2) * (SU_LMAX + 3) / 6], part_sum[DQ_THREADS];
  const int a = blockIdx.x, t = blockIdx.y, L2 = (L + 1) * (L + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double *out = dQ + (long long)L2 * (a + (long long)n_atoms * t);
  if (t >= n_active) {
    for (int lm = threadIdx.x; lm < L2; lm += blockDim.x) out[lm] = 0.0;
    return;
  }
  const long long stride = (long long)n_coef * n_chp * n_active;
  // up to 16 threads per coefficient, each a range of the point blocks
  const int shares = min(16, DQ_THREADS / n_coef), share = threadIdx.x / n_coef, k = threadIdx.x - share * n_coef;
  if (share < shares) {
    const int z0 = nz * share / shares, z1 = nz * (share + 1) / shares;
    double s = 0.0;
    for (int q = slot_ptr[a]; q < slot_ptr[a + 1]; ++q) {
      const double *p = part + k + (long long)n_coef * (slots[q] + (long long)n_chp * t);
#pragma unroll 8
      for (int z = z0; z < z1; ++z) s += p[stride * z];
    }
    part_sum[threadIdx.x] = s;
  }
  __syncthreads();
  if (threadIdx.x < n_coef) {
    double s = part_sum[threadIdx.x];
    for (int i = 1; i < shares; ++i) s += part_sum[threadIdx.x + i * n_coef];
    dc[threadIdx.x] = s;
  }
  __syncthreads();
  const int lh = min(max(lhmfd[a + n_atoms * t], 0), L);
  for (int lm = warp; lm < L2; lm += blockDim.x / 32) {
    double s = 0.0;
    if (lm < (lh + 1) * (lh + 1) && fabs(Q[lm + (long long)L2 * (a + (long long)n_atoms * t)]) > 1e-10) {
      for (int r = lm_ptr[lm] + lane; r < lm_ptr[lm + 1]; r += 32) {
        const int n = lm_row[r];
        double m = 0.0;
        for (int e = convT_ptr[n]; e < convT_ptr[n + 1]; ++e) m += convT_f[e] * dc[convT_k[e]];
        s += cc[n] * m;
      }
#pragma unroll
      for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    }
    if (lane == 0) out[lm] = s;
  }
}

int launch_dq(const SumupPlan &P, int n_active, const int *lhmfd, const double *Q, const double *g, double *dQ,
              cudaStream_t stream) {
  const dim3 grid(P.n_chp, n_active, P.adj_nz);
  switch (P.L) {
#define FRPA_DCOEF_CASE(LL)                                                                                       \
  case LL:                                                                                                        \
    sumup_dcoef_kernel<LL><<<grid, SU_THREADS, 0, stream>>>(P.n_valid_points, P.n_full_points, P.d_pfull,           \
                                                             P.d_pxyz, P.n_chp, P.d_recs, g, P.adj_pts,            \
                                                             P.d_dcoef_part);                                      \
    break;
    FRPA_DCOEF_CASE(0) FRPA_DCOEF_CASE(1) FRPA_DCOEF_CASE(2) FRPA_DCOEF_CASE(3) FRPA_DCOEF_CASE(4)
    FRPA_DCOEF_CASE(5) FRPA_DCOEF_CASE(6) FRPA_DCOEF_CASE(7) FRPA_DCOEF_CASE(8)
#undef FRPA_DCOEF_CASE
    default:
      return fail(FRPA_ERR_UNSUPPORTED, "sum-up adjoint: l_pot_max %d above %d", P.L, SU_LMAX);
  }
  FRPA_LAUNCH_CHECK();
  sumup_dq_kernel<<<dim3(P.n_atoms, P.T), DQ_THREADS, 0, stream>>>(
      P.n_atoms, P.L, P.n_chp, P.n_coef, n_active, P.adj_nz, P.d_atom_slot_ptr, P.d_atom_slots, P.d_lm_ptr, P.d_lm_row,
      P.d_convT_ptr, P.d_convT_k, P.d_convT_f, P.d_cc, lhmfd, Q, P.d_dcoef_part, dQ);
  FRPA_LAUNCH_CHECK();
  return FRPA_OK;
}

}  // namespace

// ------------------------------------------------------------ host side ---

static int sumup_upload_constants_once() {
  double K[SU_LMAX + 1][SU_LMAX + 1] = {}, Kc[SU_LMAX + 1][SU_LMAX + 1] = {};
  double RA[SU_LMAX + 1][SU_LMAX + 1] = {}, RB[SU_LMAX + 1][SU_LMAX + 1] = {}, DF[SU_LMAX + 1] = {};
  const double four_pi = 12.566370614359172953850573533118;
  for (int m = 0; m <= SU_LMAX; ++m) {
    double d = 1.0;
    for (int k = 1; k <= 2 * m - 1; k += 2) d *= k;
    DF[m] = d;
  }
  for (int l = 0; l <= SU_LMAX; ++l)
    for (int m = 0; m <= l; ++m) {
      double ratio = 1.0;
      for (int k = l - m + 1; k <= l + m; ++k) ratio /= k;
      double k0 = std::sqrt((2 * l + 1) / four_pi * ratio);
      if (m > 0) k0 *= std::sqrt(2.0);
      K[l][m] = k0;
      Kc[l][m] = (m & 1) ? -k0 : k0;
      if (l > m) {
        RA[l][m] = (double)(2 * l - 1) / (l - m);
        RB[l][m] = (double)(l + m - 1) / (l - m);
      }
    }
  FRPA_CUDA_TRY(cudaMemcpyToSymbol(c_K, K, sizeof(K)));
  FRPA_CUDA_TRY(cudaMemcpyToSymbol(c_Kcos, Kc, sizeof(Kc)));
  FRPA_CUDA_TRY(cudaMemcpyToSymbol(c_RA, RA, sizeof(RA)));
  FRPA_CUDA_TRY(cudaMemcpyToSymbol(c_RB, RB, sizeof(RB)));
  FRPA_CUDA_TRY(cudaMemcpyToSymbol(c_DF, DF, sizeof(DF)));
  FRPA_CUDA_TRY(cudaMemcpyToSymbol(d_near_tables, K, sizeof(K), 0));
  FRPA_CUDA_TRY(cudaMemcpyToSymbol(d_near_tables, RA, sizeof(RA), sizeof(K)));
  FRPA_CUDA_TRY(cudaMemcpyToSymbol(d_near_tables, RB, sizeof(RB), 2 * sizeof(K)));
  return FRPA_OK;
}

// The constant tables, uploaded once per device (plan creation and the
// allocation-free entry point may reach this from several host threads).
int sumup_upload_constants(int device) {
  static PerDeviceOnce uploaded;
  return uploaded.run(device, sumup_upload_constants_once);
}

void sumup_plan_free(SumupPlan *P) {
  if (!P) return;
  if (!P->arena_lent) cudaFree(P->arena);
  delete P;
}

// Validates the constant inputs (every device access stays in bounds for any
// per-call data once these hold) and uploads them.
// lend: where given, provides the plan's memory (kept by the caller).
int sumup_plan_create(SumupPlan **out, const frpa_sumup_desc *D, int (*lend)(size_t bytes, void **p)) {
  *out = nullptr;
  FRPA_CHECK_ARG(D != nullptr, "sumup: null descriptor");
  const int L = D->l_pot_max, lma = D->l_max_analytic_multipole, T = D->atom_tile_size;
  FRPA_CHECK_ARG(T >= 1 && T <= FRPA_MAX_ATOM_TILE, "sumup: atom tile size %d out of range", T);
  FRPA_CHECK_ARG(L >= 0 && L <= SU_LMAX, "sumup: l_pot_max %d unsupported (0..%d)", L, SU_LMAX);
  FRPA_CHECK_ARG(lma >= 0 && lma <= 2 * SU_LMAX, "sumup: l_max_analytic_multipole %d out of range", lma);
  FRPA_CHECK_ARG(D->hartree_force_l_add >= 0 && L + D->hartree_force_l_add <= 2 * SU_LMAX + 3,
                 "sumup: hartree_force_l_add %d out of range", D->hartree_force_l_add);
  FRPA_CHECK_ARG(D->n_full_points >= 0 && D->n_valid_points >= 0 && D->n_atoms > 0 && D->n_centers > 0 &&
                     D->n_centers_hartree_potential >= 0 && D->n_species > 0 && D->n_hartree_grid >= 2 &&
                     D->index_cc_dim_0 > 0,
                 "sumup: bad sizes");
  FRPA_CHECK_ARG(D->n_full_points < (1 << 30) && D->n_valid_points <= D->n_full_points,
                 "sumup: n_valid_points %d > n_full_points %d", D->n_valid_points, D->n_full_points);
  const int *ncc = D->n_cc_lm_ijk;
  FRPA_CHECK_ARG(lma >= L, "sumup: l_max_analytic_multipole %d < l_pot_max %d", lma, L);
  for (int l = 0; l <= lma; ++l)
    FRPA_CHECK_ARG(ncc[l] >= 0 && ncc[l] <= D->index_cc_dim_0 && (l == 0 || ncc[l] >= ncc[l - 1]),
                   "sumup: n_cc_lm_ijk not a cumulative count within index_cc_dim_0");
  const int icc_dim0 = D->index_cc_dim_0;
  const int mc_dim = ncc[L];
  for (int n = 0; n < ncc[L]; ++n) {
    const int l = D->index_cc[n], m = D->index_cc[n + icc_dim0];
    FRPA_CHECK_ARG(l >= 0 && l <= L && m >= -l && m <= l, "sumup: index_cc row %d has bad (l, m)", n);
    for (int c = 2; c <= 4; ++c)
      FRPA_CHECK_ARG(D->index_cc[n + c * icc_dim0] >= 0 && D->index_cc[n + c * icc_dim0] <= 2 * SU_LMAX + 1,
                     "sumup: index_cc row %d power out of range", n);
    const int nn = D->index_cc[n + 5 * icc_dim0];
    FRPA_CHECK_ARG(nn >= 0 && nn <= L + D->hartree_force_l_add, "sumup: index_cc row %d Fp index %d", n, nn);
  }
  for (int l = 0; l <= L; ++l)
    for (int c = 0; c < 3; ++c)
      FRPA_CHECK_ARG(D->index_ijk_max_cc[c + 3 * l] >= -1 && D->index_ijk_max_cc[c + 3 * l] <= 2 * SU_LMAX + 1,
                     "sumup: index_ijk_max_cc out of range");
  for (int i = 0; i < D->n_valid_points; ++i)
    FRPA_CHECK_ARG(D->i_valid_point_2_i_full_points_map[i] >= 0 &&
                       D->i_valid_point_2_i_full_points_map[i] < D->n_full_points,
                   "sumup: valid-point map entry %d out of range", i);
  for (int i = 0; i < D->n_centers_hartree_potential; ++i) {
    const int c = D->centers_hartree_potential[i];
    FRPA_CHECK_ARG(c >= 1 && c <= D->n_centers, "sumup: centers_hartree_potential[%d] = %d", i, c);
    FRPA_CHECK_ARG(i < D->n_centers, "sumup: more centre slots than centres");
  }
  for (int c = 0; c < D->n_centers; ++c) {
    FRPA_CHECK_ARG(D->center_to_atom[c] >= 1 && D->center_to_atom[c] <= D->n_atoms, "sumup: center_to_atom[%d]", c);
    FRPA_CHECK_ARG(D->species_center[c] >= 1 && D->species_center[c] <= D->n_species, "sumup: species_center[%d]", c);
  }
  for (int a = 0; a < D->n_atoms; ++a)
    FRPA_CHECK_ARG(D->species[a] >= 1 && D->species[a] <= D->n_species, "sumup: species[%d]", a);
  for (int s = 0; s < D->n_species; ++s) {
    FRPA_CHECK_ARG(D->l_hartree[s] >= 0 && D->l_hartree[s] <= L, "sumup: l_hartree[%d] = %d > l_pot_max", s,
                   D->l_hartree[s]);
    FRPA_CHECK_ARG(D->n_grid[s] >= 2 && D->n_grid[s] <= D->n_hartree_grid, "sumup: n_grid[%d]", s);
  }

  // fast-path eligibility and the exact Kelvin conversion of the table
  bool fast = true;
  for (int i = 0; i < D->n_centers_hartree_potential && fast; ++i)
    if (D->centers_hartree_potential[i] != i + 1) fast = false;
  std::vector<std::vector<std::pair<int, double>>> conv(n_kelvin(L));
  for (int n = 0; n < ncc[L] && fast; ++n) {
    const int l = D->index_cc[n];
    const int i = D->index_cc[n + 2 * icc_dim0], j = D->index_cc[n + 3 * icc_dim0], k = D->index_cc[n + 4 * icc_dim0];
    const int nn = D->index_cc[n + 5 * icc_dim0];
    int lrow = 0;  // rows must be grouped by l as n_cc_lm_ijk says
    while (lrow < L && n >= ncc[lrow]) ++lrow;
    if (lrow != l || 2 * nn != l + i + j + k || nn > l) {
      fast = false;
      break;
    }
    const int s = l - nn;
    double fnn = (nn & 1) ? -1.0 : 1.0;
    for (int q = 1; q <= 2 * nn - 1; q += 2) fnn *= q;
    for (int s1 = 0; s1 <= s; ++s1)
      for (int s2 = 0; s1 + s2 <= s; ++s2) {
        const int s3 = s - s1 - s2;
        double multi = 1.0;  // s! / (s1! s2! s3!)
        for (int q = 2; q <= s; ++q) multi *= q;
        for (int q = 2; q <= s1; ++q) multi /= q;
        for (int q = 2; q <= s2; ++q) multi /= q;
        for (int q = 2; q <= s3; ++q) multi /= q;
        conv[kelvin_index(i + 2 * s1, j + 2 * s2, k + 2 * s3)].push_back({n, fnn * multi});
      }
  }
  std::vector<int> conv_ptr(n_kelvin(L) + 1, 0), conv_lm;
  std::vector<double2> conv_fc;
  for (int q = 0; q < n_kelvin(L); ++q) {
    for (auto &e : conv[q]) {
      const int l = D->index_cc[e.first], m = D->index_cc[e.first + icc_dim0];
      conv_lm.push_back(l * l + l + m);
      conv_fc.push_back(make_double2(e.second, D->cc[e.first]));
    }
    conv_ptr[q + 1] = (int)conv_lm.size();
  }
  // transpose (by table row) for the adjoint, and the rows of each (l, m)
  std::vector<int> convT_ptr(std::max(1, mc_dim) + 1, 0), convT_k;
  std::vector<double> convT_f;
  std::vector<int> lm_ptr((L + 1) * (L + 1) + 1, 0), lm_row;
  {
    std::vector<std::vector<std::pair<int, double>>> byrow(std::max(1, mc_dim));
    int at = 0;  // the dQ kernels keep the coefficients by a, b, c
    for (int a = 0; a <= L; ++a)
      for (int b = 0; a + b <= L; ++b)
        for (int c = 0; a + b + c <= L; ++c, ++at)
          for (auto &e : conv[kelvin_index(a, b, c)]) byrow[e.first].push_back({at, e.second});
    for (size_t n = 0; n < byrow.size(); ++n) {
      for (auto &e : byrow[n]) {
        convT_k.push_back(e.first);
        convT_f.push_back(e.second);
      }
      convT_ptr[n + 1] = (int)convT_k.size();
    }
    for (int lm = 0; lm < (L + 1) * (L + 1); ++lm) {
      for (int n = 0; n < mc_dim; ++n) {
        const int l = D->index_cc[n], m = D->index_cc[n + icc_dim0];
        if (l * l + l + m == lm) lm_row.push_back(n);
      }
      lm_ptr[lm + 1] = (int)lm_row.size();
    }
  }
  std::vector<int> packed(std::max(1, icc_dim0), 0);
  for (int n = 0; n < ncc[L]; ++n)
    packed[n] = D->index_cc[n + 2 * icc_dim0] | (D->index_cc[n + 3 * icc_dim0] << 8) |
                (D->index_cc[n + 4 * icc_dim0] << 16) | (D->index_cc[n + 5 * icc_dim0] << 24);

  SumupPlan *P = new SumupPlan();
  FRPA_CUDA_TRY(cudaGetDevice(&P->device));
  P->T = T;
  P->L = L;
  P->L2 = (L + 1) * (L + 1);
  P->lma = lma;
  P->icc_dim0 = icc_dim0;
  P->mc_dim = mc_dim > 0 ? mc_dim : 1;
  P->hfla = D->hartree_force_l_add;
  P->n_full_points = D->n_full_points;
  P->n_valid_points = D->n_valid_points;
  P->n_centers = D->n_centers;
  P->n_chp = D->n_centers_hartree_potential;
  P->n_atoms = D->n_atoms;
  P->n_species = D->n_species;
  P->n_hartree_grid = D->n_hartree_grid;
  P->fast = fast ? 1 : 0;
  P->n_coef = n_kelvin(L);
  P->rs = rec_stride(L);
  int st = FRPA_OK;
  PlanMemory mem;
#define UP(field, src, bytes) mem.array((void **)&P->field, (src), (bytes));
  UP(d_map, D->i_valid_point_2_i_full_points_map, sizeof(int) * (size_t)D->n_valid_points);
  // Morton order of the valid points (21 bits per axis over their bounding box)
  const int nv = D->n_valid_points;
  std::vector<int> ord(nv);
  {
    if (nv > 0) {
      double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
      for (int i = 0; i < nv; ++i)
        for (int c = 0; c < 3; ++c) {
          const double x = D->coord_points[3LL * D->i_valid_point_2_i_full_points_map[i] + c];
          lo[c] = std::min(lo[c], x);
          hi[c] = std::max(hi[c], x);
        }
      auto spread = [](uint64_t v) {
        v &= 0x1fffff;
        v = (v | v << 32) & 0x1f00000000ffffull;
        v = (v | v << 16) & 0x1f0000ff0000ffull;
        v = (v | v << 8) & 0x100f00f00f00f00full;
        v = (v | v << 4) & 0x10c30c30c30c30c3ull;
        v = (v | v << 2) & 0x1249249249249249ull;
        return v;
      };
      std::vector<std::pair<uint64_t, int>> key(nv);
      for (int i = 0; i < nv; ++i) {
        uint64_t k = 0;
        for (int c = 0; c < 3; ++c) {
          const double x = D->coord_points[3LL * D->i_valid_point_2_i_full_points_map[i] + c];
          const double w = hi[c] > lo[c] ? (x - lo[c]) / (hi[c] - lo[c]) : 0.0;
          const uint64_t q = (uint64_t)std::min(2097151.0, std::max(0.0, w * 2097151.0));
          k |= spread(q) << c;
        }
        key[i] = {k, i};
      }
      std::sort(key.begin(), key.end());
      for (int i = 0; i < nv; ++i) ord[i] = key[i].second;
    }
    UP(d_order, ord.data(), sizeof(int) * (size_t)nv);
  }
  UP(d_coord, D->coord_points, sizeof(double) * 3 * (size_t)D->n_full_points);
  UP(d_species, D->species, sizeof(int) * D->n_atoms);
  UP(d_species_center, D->species_center, sizeof(int) * D->n_centers);
  UP(d_l_hartree, D->l_hartree, sizeof(int) * D->n_species);
  UP(d_n_grid, D->n_grid, sizeof(int) * D->n_species);
  UP(d_c2a, D->center_to_atom, sizeof(int) * D->n_centers);
  UP(d_chp, D->centers_hartree_potential, sizeof(int) * (size_t)P->n_chp);
  UP(d_icc, D->index_cc, sizeof(int) * 6 * (size_t)icc_dim0);
  UP(d_ncc, D->n_cc_lm_ijk, sizeof(int) * (lma + 1));
  UP(d_ijkmax, D->index_ijk_max_cc, sizeof(int) * 3 * (lma + 1));
  UP(d_icc_packed, packed.data(), sizeof(int) * packed.size());
  UP(d_cc, D->cc, sizeof(double) * icc_dim0);
  UP(d_cc_xyz, D->coords_center, sizeof(double) * 3 * (size_t)D->n_centers);
  UP(d_rgm, D->r_grid_min, sizeof(double) * D->n_species);
  UP(d_linc, D->log_r_grid_inc, sizeof(double) * D->n_species);
  std::vector<int> slot_of(n_kelvin(L));
  for (int a = 0; a <= L; ++a)
    for (int b = 0; a + b <= L; ++b)
      for (int c = 0; a + b + c <= L; ++c) slot_of[kelvin_index(a, b, c)] = kelvin_slot(a, b, c);
  UP(d_slot, slot_of.data(), sizeof(int) * slot_of.size());
  UP(d_conv_ptr, conv_ptr.data(), sizeof(int) * conv_ptr.size());
  UP(d_conv_lm, conv_lm.data(), sizeof(int) * conv_lm.size());
  UP(d_conv_fc, conv_fc.data(), sizeof(double2) * conv_fc.size());
  UP(d_lm_ptr, lm_ptr.data(), sizeof(int) * lm_ptr.size());
  UP(d_lm_row, lm_row.data(), sizeof(int) * lm_row.size());
  UP(d_convT_ptr, convT_ptr.data(), sizeof(int) * convT_ptr.size());
  UP(d_convT_k, convT_k.data(), sizeof(int) * convT_k.size());
  UP(d_convT_f, convT_f.data(), sizeof(double) * convT_f.size());
  // adjoint: point blocks of 512 to 4096 points (more past 262,144 points, at most
  // 64 blocks there), as small as still gives about 2,400 blocks, but no more per
  // centre than the chip takes at once (296: with few centres the last kernel's sum
  // over a thousand of them took longer than the points); partials added in order
  {
    const long long pairs = (long long)P->n_valid_points * P->n_chp * T;
    const long long most = std::max(4096, ceil_div(P->n_valid_points, 64));
    const long long least = std::max(512, ceil_div(P->n_valid_points, 296));
    P->adj_pts = (int)((std::min(most, std::max(least, pairs / 2400)) + 127) / 128 * 128);
    P->adj_nz = std::max(1, ceil_div(P->n_valid_points, P->adj_pts));
  }
  std::vector<int> cnt(P->n_atoms + 1, 0), slots(std::max(1, P->n_chp));
  {
    std::vector<int> atom_of(std::max(1, P->n_chp));
    for (int q = 0; q < P->n_chp; ++q) {
      atom_of[q] = D->center_to_atom[D->centers_hartree_potential[q] - 1] - 1;
      ++cnt[atom_of[q] + 1];
    }
    for (int a = 0; a < P->n_atoms; ++a) cnt[a + 1] += cnt[a];
    std::vector<int> fill(cnt.begin(), cnt.end() - 1);
    for (int q = 0; q < P->n_chp; ++q) slots[fill[atom_of[q]]++] = q;  // ascending within each atom
  }
  UP(d_atom_slot_ptr, cnt.data(), sizeof(int) * cnt.size());
  UP(d_atom_slots, slots.data(), sizeof(int) * slots.size());
  const int no_flags = 0;
  UP(d_err, &no_flags, sizeof(int));
#undef UP
  const size_t chp = std::max(1, P->n_chp);
  mem.space((void **)&P->d_pfull, sizeof(int) * (size_t)P->n_valid_points);
  mem.space((void **)&P->d_pxyz, sizeof(double) * 3 * (size_t)P->n_valid_points);
  mem.space((void **)&P->d_pbox, sizeof(Box) * (size_t)ceil_div(P->n_valid_points, 32));
  mem.space((void **)&P->d_mc, sizeof(double) * (size_t)P->mc_dim * P->n_atoms * T);
  mem.space((void **)&P->d_recs, sizeof(double) * (size_t)P->rs * chp * T);
  mem.space((void **)&P->d_heads, sizeof(double4) * chp * T);
  mem.space((void **)&P->d_dcoef_part, sizeof(double) * (size_t)n_kelvin(L) * chp * T * P->adj_nz);
  if (st == FRPA_OK && lend) {
    P->arena_lent = true;
    st = lend(mem.total(), (void **)&P->arena);
  }
  if (st == FRPA_OK) st = mem.commit(&P->arena, &P->arena_bytes);
  if (st == FRPA_OK && P->n_valid_points > 0) {
    sumup_gather_points_kernel<<<std::min(1184, ceil_div(P->n_valid_points, 256)), 256>>>(
        P->n_valid_points, P->d_map, P->d_order, P->d_coord, P->d_pfull, P->d_pxyz, P->d_pbox);
    if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(0) != cudaSuccess)
      st = fail(FRPA_ERR_CUDA, "sumup: point ordering failed");
  }
  if (st == FRPA_OK) st = sumup_upload_constants(P->device);
  if (st != FRPA_OK) {
    sumup_plan_free(P);
    return st;
  }
  *out = P;
  return FRPA_OK;
}

int sumup_plan_is_fast(const SumupPlan *P) { return P->fast; }

int sumup_execute(const SumupPlan *P, int n_active, int force_generic, const int *lhmfd, const double *mrs,
                  const double *opr, const double *Q, const double *spline, double *dv, unsigned char *codes,
                  cudaStream_t stream) {
  FRPA_CHECK_ARG(n_active >= 0 && n_active <= P->T, "sumup: %d active perturbations > tile %d", n_active, P->T);
  if (n_active == 0 || P->n_valid_points == 0 || P->n_chp == 0) return FRPA_OK;
  if (P->fast && !force_generic) {
    FRPA_TRY(launch_prep(*P, n_active, lhmfd, mrs, opr, Q, stream));
    if (codes) return launch_fast<true>(*P, n_active, spline, dv, codes, stream);
    return launch_fast<false>(*P, n_active, spline, dv, nullptr, stream);
  }
  sumup_multipole_c_kernel<<<dim3(P->n_atoms, n_active), 128, 0, stream>>>(
      P->n_atoms, P->L, P->L2, P->mc_dim, P->icc_dim0, P->lma, P->d_icc, P->d_ncc, P->d_cc, lhmfd, Q, P->d_mc,
      P->d_err);
  FRPA_LAUNCH_CHECK();
  const int grid = (P->n_valid_points + SU_THREADS - 1) / SU_THREADS;
  sumup_generic_kernel<<<grid, SU_THREADS, 0, stream>>>(
      P->n_valid_points, P->n_full_points, P->d_map, P->d_coord, n_active, P->n_chp, P->n_atoms, P->L, P->L2,
      P->n_hartree_grid, P->hfla, P->d_chp, P->d_c2a, P->d_species, P->d_species_center, P->d_l_hartree,
      P->d_n_grid, P->d_rgm, P->d_linc, P->d_cc_xyz, mrs, opr, P->d_ncc, P->d_icc_packed, P->d_ijkmax, P->mc_dim,
      P->d_mc, spline, dv, codes);
  FRPA_LAUNCH_CHECK();
  return FRPA_OK;
}

int sumup_read_error_flags(const SumupPlan *P, int *flags) {
  FRPA_CUDA_TRY(cudaMemcpy(flags, P->d_err, sizeof(int), cudaMemcpyDeviceToHost));
  FRPA_CUDA_TRY(cudaMemset(P->d_err, 0, sizeof(int)));
  return FRPA_OK;
}

int sumup_adjoint_q(const SumupPlan *P, int n_active, const int *lhmfd, const double *mrs, const double *opr,
                    const double *Q, const double *g, double *dQ, cudaStream_t stream) {
  if (!P->fast)
    return fail(FRPA_ERR_UNSUPPORTED,
                "sumup adjoint: dQ is implemented for the fast path only (identity centers_hartree_potential and a "
                "homogeneous multipole table); this plan uses the generic far-field kernel");
  FRPA_CHECK_ARG(n_active >= 0 && n_active <= P->T, "sumup adjoint: n_active %d", n_active);
  if (n_active == 0 || P->n_chp == 0 || P->n_valid_points == 0) {
    FRPA_CUDA_TRY(cudaMemsetAsync(dQ, 0, sizeof(double) * (size_t)P->L2 * P->n_atoms * P->T, stream));
    return FRPA_OK;
  }
  FRPA_TRY(launch_prep(*P, n_active, lhmfd, mrs, opr, Q, stream));
  return launch_dq(*P, n_active, lhmfd, Q, g, dQ, stream);
}

}  // namespace frpa

// ------------------------------------------------ allocation-free variant
//
// frpa_sumup_execute_noalloc: the sum-up for callers that cannot let a
// library call cudaMalloc / cudaFree, such as a host code that hands the GPU
// a fixed memory budget managed by its own pool, or one that keeps several
// streams busy and cannot afford cudaFree's implicit device-wide
// synchronisation.  The caller passes every input and the output as device
// pointers; the only scratch this path needs (the packed multipole table and
// the per-atom multipole coefficients) lives in the file-scope array below,
// which every GPU that loads the library holds until the process exits.
// It runs the reference-mirroring (generic) kernel.

namespace frpa {

constexpr size_t NOALLOC_SCRATCH_BYTES = 8u << 20;  // 8 MiB per device
static __device__ __align__(256) unsigned char g_noalloc_scratch[NOALLOC_SCRATCH_BYTES];

namespace {

__global__ void noalloc_pack_table_kernel(int n_rows, int icc_dim0, const int *__restrict__ icc,
                                          int *__restrict__ packed) {
  for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < n_rows; n += gridDim.x * blockDim.x)
    packed[n] = icc[n + 2 * icc_dim0] | (icc[n + 3 * icc_dim0] << 8) | (icc[n + 4 * icc_dim0] << 16) |
                (icc[n + 5 * icc_dim0] << 24);
}

std::mutex g_noalloc_mu;
void *g_noalloc_addr[64] = {nullptr};

// Device address of the scratch array for the current device, looked up once
// per device (host code may not use the array's name as an address).
int noalloc_scratch_address(int device, unsigned char **out) {
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  if (device < 0 || device >= 64) return fail(FRPA_ERR_UNSUPPORTED, "noalloc sum-up: device %d", device);
  if (!g_noalloc_addr[device]) {
    void *p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess)
      return fail(FRPA_ERR_CUDA, "noalloc sum-up: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
    FRPA_TRY(sumup_upload_constants(device));
    // the input-flag word at the start of the array collects the flags of
    // every call on this device until frpa_sumup_noalloc_flags reads it
    e = cudaMemset(p, 0, sizeof(int));
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e != cudaSuccess)
      return fail(FRPA_ERR_CUDA, "noalloc sum-up: clearing the flag word failed: %s", cudaGetErrorString(e));
    g_noalloc_addr[device] = p;
  }
  *out = static_cast<unsigned char *>(g_noalloc_addr[device]);
  return FRPA_OK;
}

}  // namespace
}  // namespace frpa

extern "C" int frpa_sumup_execute_noalloc(
    int atom_tile_size, int j_atom_begin, int j_atom_end, int n_full_points, int l_max_analytic_multipole,
    int index_cc_dim_0, int n_valid_points, int l_pot_max, int n_hartree_grid, int n_centers,
    int n_centers_hartree_potential, int n_atoms, int hartree_force_l_add, int n_species, const int *species,
    const int *species_center, const int *l_hartree_max_far_distance, const int *i_valid_point_2_i_full_points_map,
    const double *coord_points, const double *multipole_radius_sq, const double *outer_potential_radius,
    const double *multipole_moments, const double *spline, const int *l_hartree, const int *n_grid,
    const int *n_cc_lm_ijk, const int *centers_hartree_potential, const int *center_to_atom, const int *index_cc,
    const int *index_ijk_max_cc, const double *cc, const double *coords_center, const double *r_grid_min,
    const double *log_r_grid_inc, double *delta_v_hartree, void *stream_) {
  using namespace frpa;
  clear_error();
  const int T = atom_tile_size, L = l_pot_max, n_active = j_atom_end - j_atom_begin + 1;
  FRPA_CHECK_ARG(T >= 1 && T <= FRPA_MAX_ATOM_TILE, "noalloc sum-up: atom tile size %d out of range", T);
  FRPA_CHECK_ARG(L >= 0 && L <= SU_LMAX, "noalloc sum-up: l_pot_max %d unsupported (0..%d)", L, SU_LMAX);
  FRPA_CHECK_ARG(l_max_analytic_multipole >= L && index_cc_dim_0 > 0, "noalloc sum-up: bad multipole table sizes");
  FRPA_CHECK_ARG(hartree_force_l_add >= 0 && L + hartree_force_l_add <= 2 * SU_LMAX + 3,
                 "noalloc sum-up: hartree_force_l_add %d out of range", hartree_force_l_add);
  FRPA_CHECK_ARG(n_active <= T, "noalloc sum-up: j_atom_end - j_atom_begin + 1 = %d > ATOM_TILE_SIZE %d", n_active, T);
  FRPA_CHECK_ARG(n_full_points >= 0 && n_valid_points >= 0 && n_valid_points <= n_full_points && n_atoms > 0 &&
                     n_centers > 0 && n_centers_hartree_potential >= 0 &&
                     n_centers_hartree_potential <= n_centers && n_species > 0 && n_hartree_grid >= 2,
                 "noalloc sum-up: bad sizes");
  FRPA_CHECK_ARG(species && species_center && l_hartree_max_far_distance && i_valid_point_2_i_full_points_map &&
                     coord_points && multipole_radius_sq && outer_potential_radius && multipole_moments && spline &&
                     l_hartree && n_grid && n_cc_lm_ijk && centers_hartree_potential && center_to_atom && index_cc &&
                     index_ijk_max_cc && cc && coords_center && r_grid_min && log_r_grid_inc && delta_v_hartree,
                 "noalloc sum-up: null device pointer");
  // scratch layout: [error flag | packed table rows | multipole coefficients
  // (index_cc_dim_0, n_atoms, T)]; the coefficient block is sized by
  // index_cc_dim_0, an upper bound of n_cc_lm_ijk[l_pot_max] known on the host.
  const size_t flag_bytes = 256;
  const size_t table_bytes = ((size_t)index_cc_dim_0 * sizeof(int) + 255) / 256 * 256;
  const size_t mc_bytes = sizeof(double) * (size_t)index_cc_dim_0 * n_atoms * T;
  const size_t need = flag_bytes + table_bytes + mc_bytes;
  FRPA_CHECK_ARG(need <= NOALLOC_SCRATCH_BYTES,
                 "noalloc sum-up: needs %zu bytes of scratch (index_cc_dim_0 %d x n_atoms %d x tile %d), more than "
                 "the %zu bytes this entry point has; use frpa_sumup_plan_create / frpa_sumup_execute",
                 need, index_cc_dim_0, n_atoms, T, (size_t)NOALLOC_SCRATCH_BYTES);
  int device = 0;
  FRPA_CUDA_TRY(cudaGetDevice(&device));
  unsigned char *base = nullptr;
  FRPA_TRY(noalloc_scratch_address(device, &base));
  if (n_active <= 0 || n_valid_points == 0 || n_centers_hartree_potential == 0) return FRPA_OK;
  cudaStream_t stream = (cudaStream_t)stream_;
  int *err = reinterpret_cast<int *>(base);
  int *packed = reinterpret_cast<int *>(base + flag_bytes);
  double *mc = reinterpret_cast<double *>(base + flag_bytes + table_bytes);
  const int L2 = (L + 1) * (L + 1);
  // every scratch word read below is written first in this call, so nothing
  // left by an earlier call is used; the flag word (bit 0: an
  // l_hartree_max_far_distance entry outside 0..l_pot_max, clamped) keeps
  // collecting until frpa_sumup_noalloc_flags reads and clears it
  noalloc_pack_table_kernel<<<(index_cc_dim_0 + 255) / 256, 256, 0, stream>>>(index_cc_dim_0, index_cc_dim_0,
                                                                               index_cc, packed);
  FRPA_LAUNCH_CHECK();
  sumup_multipole_c_kernel<<<dim3(n_atoms, n_active), 128, 0, stream>>>(
      n_atoms, L, L2, index_cc_dim_0, index_cc_dim_0, l_max_analytic_multipole, index_cc, n_cc_lm_ijk, cc,
      l_hartree_max_far_distance, multipole_moments, mc, err);
  FRPA_LAUNCH_CHECK();
  const int grid = (n_valid_points + SU_THREADS - 1) / SU_THREADS;
  sumup_generic_kernel<<<grid, SU_THREADS, 0, stream>>>(
      n_valid_points, n_full_points, i_valid_point_2_i_full_points_map, coord_points, n_active,
      n_centers_hartree_potential, n_atoms, L, L2, n_hartree_grid, hartree_force_l_add, centers_hartree_potential,
      center_to_atom, species, species_center, l_hartree, n_grid, r_grid_min, log_r_grid_inc, coords_center,
      multipole_radius_sq, outer_potential_radius, n_cc_lm_ijk, packed, index_ijk_max_cc, index_cc_dim_0, mc, spline,
      delta_v_hartree, nullptr);
  FRPA_LAUNCH_CHECK();
  return FRPA_OK;
}

extern "C" int frpa_sumup_noalloc_flags(int *flags, void *stream_) {
  using namespace frpa;
  clear_error();
  FRPA_CHECK_ARG(flags != nullptr, "noalloc sum-up flags: null output");
  int device = 0;
  FRPA_CUDA_TRY(cudaGetDevice(&device));
  unsigned char *base = nullptr;
  FRPA_TRY(noalloc_scratch_address(device, &base));
  cudaStream_t stream = (cudaStream_t)stream_;
  int v = 0;
  FRPA_CUDA_TRY(cudaMemcpyAsync(&v, base, sizeof(int), cudaMemcpyDeviceToHost, stream));
  FRPA_CUDA_TRY(cudaMemsetAsync(base, 0, sizeof(int), stream));
  FRPA_CUDA_TRY(cudaStreamSynchronize(stream));
  *flags = v;
  return FRPA_OK;
}
