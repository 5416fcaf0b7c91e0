// First-order density bias, part 2: the density-matrix term of rho1 for the
// displacement of atom j along j_coord, the input `first_order_rho_bias_part2`
// of the rho1 step.  Per grid batch and atom j of the tile, with
// fw = -d phi / d x_{j_coord} and A_j the batch's compute functions of atom j
// (the range atom_valid_n_compute_c_batches(j-1 .. j, batch)):
//   bias(p, j) = sum_i phi_i(p) sum_{k in A_j} DM(ib_i, ib_k) fw_k(p)
//              + sum_{i in A_j} fw_i(p) sum_k DM(ib_i, ib_k) phi_k(p)
// Reference: fast_rap_src_dfpt_gpu_eval/generate_first_order_rho_bias_part2.cpp:11-168
// (two DGEMMs and two per-point dot products per (batch, atom), through the
// host).  Here the two terms are one contraction with the symmetrised slab
//   S(i, k) = DM(ib_i, ib_k) + DM(ib_k, ib_i),  k in A_j,
//   bias(p, j) = sum_k fw_k(p) M(k, p),  M(k, p) = sum_i S(i, k) phi_i(p):
// M is a (functions of the atoms) x (points) x (n_compute) product on the FP64
// MMA, 24 functions x 64 points at a time, and the sum over k its epilogue.
// Atoms with no compute function in a batch get bias 0, as in the reference
// (:152-156); batches without compute functions are left untouched.
//
// What bounds it: an atom is in few of the batches (a 1,000-atom problem: 3 to
// 4% of them), so most work items only write zeros, and the others stream phi
// once (the flops are small: 20 n_compute a point and atom).  So the functions
// of all the call's atoms in an item share one pass over phi (neighbouring
// atoms are in the same items, and an item that did them in turn was the last
// to finish); a CTA looks at two items, half the list apart because the list's
// neighbours tend to be active together; and a pass is a two-stage pipeline
// over 32-wide chunks of i: phi by 16-byte asynchronous copies, S by plain
// gathers (lanes along i, so that one of its two terms is contiguous) held in
// registers while the MMAs of the chunk before run.  Measured, 4,000 batches of
// 100-300 points, n_compute 100-600, four of 1,000 atoms (one B200): one thread
// per point walking its phi row 1.1 to 3.0 ms, by the atoms; this form 0.16 to
// 0.43 ms, at 2.4 TB/s of DRAM reads in the latter (L1 58% busy: the gathers).
#include <algorithm>

#include "frpa_internal.cuh"

namespace frpa {
namespace {

constexpr int BZ_THREADS = 128;
constexpr int BZ_PTS = 64;     // points per pass: 4 warps x 16
constexpr int BZ_IC = 32;      // contraction chunk
constexpr int BZ_KG = 24;      // functions per pass (three 8-row MMA tiles)
constexpr int BZ_MAXA = 64;    // compute functions of one atom in one batch
constexpr int BZ_ITEMS = 2;    // most items per CTA
constexpr int BZ_LDB = BZ_IC + 4;  // stride = 4 (mod 16) doubles: conflict-free fragment loads
constexpr int BZ_LDS = BZ_KG + 4;  // 12 (mod 16): likewise

struct BiasSmem {
  double B[2][BZ_PTS * BZ_LDB];  // phi(i, p) of a chunk: [p][i]; after a pass, its products [k][p]
  double S[2][BZ_IC * BZ_LDS];   // S(i, k) of a chunk: [i][k]
  Rho1WorkItem item[BZ_ITEMS];
  int vs[BZ_ITEMS][FRPA_MAX_ATOM_TILE];       // first compute function of each atom
  int off[BZ_ITEMS][FRPA_MAX_ATOM_TILE + 1];  // running count of the atoms' functions
  int fn[BZ_KG], ft[BZ_KG];                   // a pass's functions: position in the batch, atom
};
static_assert(BZ_KG * BZ_PTS <= BZ_PTS * BZ_LDB, "a pass's products fit a phi stage");

// The biases of item m for every atom with functions in it.
__device__ __forceinline__ void bias_item(BiasSmem &M, int m, int n_active, int jc, int n_basis, int nmb,
                                          int n_batches, const int *__restrict__ ib_all,
                                          const double *__restrict__ wave, const double *__restrict__ gwave,
                                          const double *__restrict__ dm, int aligned16, double *__restrict__ bias) {
  const Rho1WorkItem &W = M.item[m];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
  const int nc = W.nc, ncp = (nc + 3) & ~3, nch = (nc + BZ_IC - 1) / BZ_IC;
  const int *ibl = ib_all + W.ib_off;
  const int n_fn = M.off[m][n_active];
  for (int pp = 0; pp < W.pn; pp += BZ_PTS) {
    const int pn = min(BZ_PTS, W.pn - pp);
    const double *phi = wave + W.wave_off + (long long)(W.p0 + pp) * ncp;
    const double *gph = gwave + 3 * W.wave_off + 3LL * (W.p0 + pp) * ncp + (long long)jc * ncp;
    for (int kg = 0; kg < n_fn; kg += BZ_KG) {
      const int kn = min(BZ_KG, n_fn - kg), nkt = (kn + 7) >> 3;
      if (tid < kn) {
        int t = 0;
        while (M.off[m][t + 1] <= kg + tid) ++t;
        M.ft[tid] = t;
        M.fn[tid] = M.vs[m][t] + kg + tid - M.off[m][t];
      }
      __syncthreads();
      // this thread's columns k = warp + 4 j of the pass and row i = lane of each chunk
      long long col[BZ_KG / 4];
#pragma unroll
      for (int j = 0; j < BZ_KG / 4; ++j) {
        const int k = warp + 4 * j;
        col[j] = k < kn ? (long long)(__ldg(ibl + M.fn[k]) - 1) : -1;
      }
      auto load_phi = [&](int c) {
        double *Bs = M.B[c & 1];
        const int i0 = c * BZ_IC;
        if (aligned16) {
#pragma unroll
          for (int j = 0; j < (BZ_PTS * BZ_IC / 2) / BZ_THREADS; ++j) {
            const int e = tid + BZ_THREADS * j, ip = e & (BZ_IC / 2 - 1), n = e / (BZ_IC / 2), i = i0 + 2 * ip;
            const int bytes = n < pn ? (i + 1 < nc ? 16 : (i < nc ? 8 : 0)) : 0;
            cp_async_16(&Bs[n * BZ_LDB + 2 * ip], bytes ? phi + i + (long long)n * ncp : phi, bytes);
          }
        } else {
#pragma unroll
          for (int j = 0; j < (BZ_PTS * BZ_IC) / BZ_THREADS; ++j) {
            const int e = tid + BZ_THREADS * j, ii = e & (BZ_IC - 1), n = e / BZ_IC, i = i0 + ii;
            const bool ok = n < pn && i < nc;
            cp_async_8(&Bs[n * BZ_LDB + ii], ok ? phi + i + (long long)n * ncp : phi, ok ? 8 : 0);
          }
        }
        cp_async_commit();
      };
      double d0[BZ_KG / 4], d1[BZ_KG / 4];
      // the rows' basis indices are loaded a chunk before the gathers that need them
      auto row_of = [&](int c) { return c * BZ_IC + lane < nc ? __ldg(ibl + c * BZ_IC + lane) - 1 : -1; };
      int next_row = row_of(0);
      auto load_dm = [&](int c) {
        const long long row = next_row;
        next_row = row_of(c + 1);
#pragma unroll
        for (int j = 0; j < BZ_KG / 4; ++j) {
          const bool ok = row >= 0 && col[j] >= 0;
          d0[j] = ok ? __ldg(dm + row + col[j] * n_basis) : 0.0;
          d1[j] = ok ? __ldg(dm + col[j] + row * n_basis) : 0.0;
        }
      };
      auto store_dm = [&](int c) {
#pragma unroll
        for (int j = 0; j < BZ_KG / 4; ++j) M.S[c & 1][lane * BZ_LDS + warp + 4 * j] = d0[j] + d1[j];
      };
      double acc[BZ_KG / 8][2][2];
#pragma unroll
      for (int a = 0; a < BZ_KG / 8; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
      load_phi(0);
      load_dm(0);
      store_dm(0);
      cp_async_wait<0>();
      __syncthreads();
      for (int c = 0; c < nch; ++c) {
        if (c + 1 < nch) {
          load_phi(c + 1);
          load_dm(c + 1);
        }
        const double *Bs = M.B[c & 1], *Ss = M.S[c & 1];
        if (warp * 16 < pn) {
#pragma unroll
          for (int ks = 0; ks < BZ_IC / 4; ++ks) {
            double b[2];
#pragma unroll
            for (int n = 0; n < 2; ++n) b[n] = Bs[(warp * 16 + n * 8 + g) * BZ_LDB + ks * 4 + q];
#pragma unroll
            for (int kt = 0; kt < BZ_KG / 8; ++kt)
              if (kt < nkt) {
                const double a = Ss[(ks * 4 + q) * BZ_LDS + kt * 8 + g];
#pragma unroll
                for (int n = 0; n < 2; ++n) dmma_8x8x4(acc[kt][n][0], acc[kt][n][1], a, b[n]);
              }
          }
        }
        if (c + 1 < nch) store_dm(c + 1);
        cp_async_wait<0>();
        __syncthreads();
      }
      // lane (g, q) holds M(kt 8 + g, n 8 + 2 q + h): its products with fw, [k][p]
      double *Pr = M.B[0];
#pragma unroll
      for (int kt = 0; kt < BZ_KG / 8; ++kt) {
        const int k = kt * 8 + g;
        if (k >= kn) continue;
        const double *gk = gph + M.fn[k];
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int p = warp * 16 + n * 8 + 2 * q + h;
            if (p < pn) Pr[k * BZ_PTS + p] = -__ldg(gk + 3LL * p * ncp) * acc[kt][n][h];
          }
      }
      __syncthreads();
      // per point and atom, the functions in order; an atom whose functions go
      // over two passes continues from what the same thread wrote
      const int p = tid & (BZ_PTS - 1);
      if (p < pn) {
        for (int k = 0; k < kn;) {
          const int t = M.ft[k];
          int e = k;
          while (e < kn && M.ft[e] == t) ++e;
          if ((t & 1) == tid / BZ_PTS) {
            double *out = bias + (W.p0 + pp + p) + (long long)nmb * (W.batch + (long long)n_batches * t);
            double v = kg + k > M.off[m][t] ? *out : 0.0;
            for (int x = k; x < e; ++x) v += Pr[x * BZ_PTS + p];
            *out = v;
          }
          k = e;
        }
      }
      __syncthreads();
    }
  }
}

// CTA c takes items c and c + stride
__global__ void __launch_bounds__(BZ_THREADS, 4) bias_part2_kernel(
    const Rho1WorkItem *__restrict__ items, int n_items, int stride, const int *__restrict__ ib_all,
    const int *__restrict__ atom_valid, int n_atoms, int j_atom_begin, int n_active, int j_coord, int n_basis,
    int n_max_batch_size, int n_batches, const double *__restrict__ wave, const double *__restrict__ gwave,
    const double *__restrict__ dm, double *__restrict__ bias, int aligned16, int *__restrict__ err) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  BiasSmem &M = *reinterpret_cast<BiasSmem *>(smem_raw);
  const int tid = threadIdx.x;
  const int mine = min(BZ_ITEMS, (n_items - (int)blockIdx.x + stride - 1) / stride);
  static_assert(BZ_ITEMS * FRPA_MAX_ATOM_TILE <= BZ_THREADS, "one thread per (item, atom)");
  if (tid < mine * n_active) {
    const int m = tid / n_active, t = tid - m * n_active;
    const Rho1WorkItem W = items[blockIdx.x + m * stride];
    if (t == 0) M.item[m] = W;
    const int *av = atom_valid + (long long)(n_atoms + 1) * W.batch + j_atom_begin + t;
    const int vs = av[-1], cnt = av[0] - vs;
    const bool outside = cnt > 0 && (vs < 0 || cnt > BZ_MAXA || vs + cnt > W.nc);
    if (outside && W.p0 == 0) atomicOr(err, 8);  // outside the batch: flag, write nothing
    M.vs[m][t] = outside ? -1 : max(vs, 0);
    M.off[m][t + 1] = outside ? 0 : max(cnt, 0);
  }
  __syncthreads();
  const int warp = tid >> 5, lane = tid & 31;
  for (int e = warp; e < mine * n_active; e += BZ_THREADS / 32) {  // atoms without functions here: zeros
    const int m = e / n_active, t = e - m * n_active;
    if (M.off[m][t + 1] != 0 || M.vs[m][t] < 0) continue;
    const Rho1WorkItem &W = M.item[m];
    double *out = bias + W.p0 + (long long)n_max_batch_size * (W.batch + (long long)n_batches * t);
    for (int p = lane; p < W.pn; p += 32) out[p] = 0.0;
  }
  __syncthreads();
  if (tid < mine) {
    M.off[tid][0] = 0;
    for (int t = 0; t < n_active; ++t) M.off[tid][t + 1] += M.off[tid][t];
  }
  __syncthreads();
  for (int m = 0; m < mine; ++m)
    if (M.off[m][n_active] > 0)
      bias_item(M, m, n_active, j_coord - 1, n_basis, n_max_batch_size, n_batches, ib_all, wave, gwave, dm, aligned16,
                bias);
}

}  // namespace

// Host checks of the atom ranges, then one launch over the plan's work items.
int rho1_bias_part2_launch(const Rho1Plan &plan, const int *h_atom_valid, const int *d_atom_valid, int n_atoms,
                           int j_atom_begin, int j_atom_end, int j_coord, int T, const double *wave,
                           const double *gwave, const double *dm, double *bias, cudaStream_t stream) {
  const int n_active = j_atom_end - j_atom_begin + 1;
  FRPA_CHECK_ARG(j_coord >= 1 && j_coord <= 3, "bias part 2: j_coord %d not 1..3", j_coord);
  FRPA_CHECK_ARG(n_active >= 1 && n_active <= T, "bias part 2: atoms %d..%d do not fit the tile of %d", j_atom_begin,
                 j_atom_end, T);
  FRPA_CHECK_ARG(j_atom_begin >= 1 && j_atom_end <= n_atoms, "bias part 2: atoms %d..%d outside 1..%d", j_atom_begin,
                 j_atom_end, n_atoms);
  FRPA_CHECK_ARG(wave && gwave && dm && bias && d_atom_valid, "bias part 2: null device pointer");
  if (h_atom_valid) {
    for (const Rho1WorkItem &b : plan.h_batches)
      for (int j = j_atom_begin; j <= j_atom_end; ++j) {
        const int *av = h_atom_valid + (long long)(n_atoms + 1) * b.batch;
        const int vs = av[j - 1], ve = av[j];
        FRPA_CHECK_ARG(vs >= 0 && ve >= vs && ve <= b.nc && ve - vs <= BZ_MAXA,
                       "bias part 2: batch %d atom %d compute range [%d, %d) invalid (n_compute %d, at most %d per "
                       "atom)",
                       b.batch, j, vs, ve, b.nc, BZ_MAXA);
      }
  }
  if (plan.n_items == 0) return FRPA_OK;
  static PerDeviceOnce configured;
  FRPA_TRY(configured.run(plan.device, []() -> int {
    FRPA_CUDA_TRY(
        cudaFuncSetAttribute(bias_part2_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(BiasSmem)));
    return FRPA_OK;
  }));
  int n_sm = 148;
  FRPA_CUDA_TRY(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, plan.device));
  // one item per CTA until the CTAs fill the chip (four per SM), then two
  const int per_cta = std::max(1, std::min(BZ_ITEMS, plan.n_items / (4 * n_sm)));
  const int grid = ceil_div(plan.n_items, per_cta);
  const int aligned16 = plan.wave_aligned16 && !((uintptr_t)wave & 15);
  bias_part2_kernel<<<grid, BZ_THREADS, sizeof(BiasSmem), stream>>>(
      plan.d_items, plan.n_items, grid, plan.d_ib, d_atom_valid, n_atoms, j_atom_begin, n_active, j_coord,
      plan.n_basis, plan.n_max_batch_size, plan.n_batches, wave, gwave, dm, bias, aligned16, plan.d_err);
  FRPA_LAUNCH_CHECK();
  return FRPA_OK;
}

}  // namespace frpa
