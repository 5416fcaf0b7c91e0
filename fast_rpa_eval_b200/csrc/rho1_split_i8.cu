// Split-precision rho1 on the integer tensor cores (tcgen05 kind::i8):
// work1 = P1c * phi at FP64-grade accuracy from exact int32 sums of 8-bit
// digit products, with the per-point dot products in FP64.
//
// Same semantics as the plain FP64 path (rho1_fp64.cu,
// fast_rap_src_dfpt_gpu_eval/evaluate_first_order_rho.cpp:116-209).
//
// Numerics.  Each FP64 operand x of a row (one grid point's phi over the
// batch's compute functions, or one row of P1) with scale 2^e,
// max|x| < 0.9921875 2^e, is rounded to the integer X = rint(x 2^(39 - e))
// and written in balanced base 256, X = a0 2^32 + a1 2^24 + a2 2^16 +
// a3 2^8 + a4, every digit a signed byte (|a0| <= 127 since
// |X| < 2^39 - 2^31 - 2^23 - 2^15 - 2^7).  The product of two rows is the sum
// of the 19 digit products with s + u <= 5, accumulated per level L = s + u
// in six int32 TMEM accumulators; |a_s b_u| <= 2^14, so every level stays
// exact for K < 26,000 (at most five products per level).  Recombined in FP64:
//   work1(i, p) = 2^(eA + eB - 54) (L0 2^40 + L1 2^32 + L2 2^24 + L3 2^16 + L4 2^8 + L5).
// What remains is the rounding of the operands to 2^-40 of their row scale
// and the dropped levels 6..8 (2^-48 per product); keeping level 5 removes
// the error term that dominated with levels 0..4 only (3.5x larger than the
// operand rounding in a CPU emulation of these steps).
//
// Data flow, three launches per group of batches:
//   1. pack A: one CTA per eight points of a work item (<= 128 points of one
//      batch) finds the per-point scales and writes phi's five digit planes in
//      the tcgen05 shared-memory tile image (K-major, no swizzle, 8 x 16-byte
//      core matrices), one 32-wide K chunk after another;
//   2. pack B: one CTA per (batch, perturbation, N tile of 32 rows, the last
//      one zero-padded) gathers P1c = P1[ib, ib] (lanes along P1's contiguous
//      rows) and writes its digit planes the same way;
//   3. contract: one persistent CTA per SM.  A loader warp moves each stage's
//      (two K chunks') A and B planes into a 3-stage shared-memory ring with
//      two bulk copies; an MMA warp issues a chunk's 19 digit products as five
//      tcgen05.mma.kind::i8 (M = 128 points, K = 32; the digit levels run
//      along N: A plane s times B planes 0..min(4, 5-s), into the level
//      accumulators from level s on) in one of two sets (2 x 192 of 512 TMEM
//      columns); 8 epilogue warps read a finished set (tcgen05.ld), recombine
//      in FP64 and contract with phi and grad phi (FP64, 256-bit loads from
//      global memory issued four columns ahead) while the MMAs of the next
//      tile fill the other set.
// What bounds the contraction (8,000 batches of 100-600 functions, 7.1 ms): a
// chunk's MMAs take 304 cycles, but their operands are 40 KB and its copies
// 21 KB through the 128 bytes a cycle of shared memory (~480 cycles, measured
// with the epilogue's loads and sums left out), and with the 10 KB of phi and
// grad phi the SMs draw ~10 TB/s from L2 (620 cycles).  Issue used to bound
// it (660 cycles): six copies, two waits and two commits per 32-wide chunk from
// single threads, and waiting warps that polled a global timer.  Not kept,
// all slower or equal: 8 stages (26 KB of L1 left for the epilogue's loads),
// 4 chunks a stage, sixteen epilogue warps (spills), a second set of phi
// registers under setmaxnreg, smaller groups of batches.
// The packed operands cost a write and a read of ~5 bytes per P1c and phi
// element, in exchange the contraction has no gathers, no conversions and
// no register-staged loads on its critical path.  Every mbarrier wait is
// bounded in time; on a timeout the kernel records an error flag, waits
// (bounded) for its copies and MMAs in flight, frees TMEM and returns.
#include <algorithm>
#include <vector>

#include "frpa_internal.cuh"
#include "sm100_sync.cuh"

namespace frpa {
namespace {

using namespace sm100;

constexpr int I8_M = 128;      // points per work item (TMEM lanes)
constexpr int I8_N = 32;       // rows i per N tile (accumulator columns per level)
constexpr int I8_KC = 32;      // K per chunk: one kind::i8 instruction
constexpr int I8_LEVELS = 6;   // digit levels s + u = 0..5
constexpr int I8_SLICES = 5;   // digit planes per operand
constexpr int I8_SETS = 2;     // accumulator sets: a tile's epilogue overlaps the next tile's MMAs
constexpr int I8_CHUNKS = 2;   // chunks per stage
constexpr int I8_STAGES = 3;
constexpr int I8_EPI_WARPS = 8;  // warps 0..7: lane quarter w % 4, column half w / 4; warp 0 owns TMEM
constexpr int I8_COLS = I8_N / 2;  // 16 accumulator columns per epilogue warp
constexpr int EPI_BUFS = 2;        // four-column steps whose phi and grad phi are in registers
constexpr int I8_LOAD_WARP = 8;  // issues the bulk copies
constexpr int I8_MMA_WARP = 9;   // issues the MMAs
constexpr int I8_THREADS = 32 * 10;
constexpr int I8_ROWB = I8_KC;                         // bytes per tile row of one plane
constexpr int I8_A_PLANE = I8_M * I8_ROWB;             // 4096
constexpr int I8_B_CHUNK = I8_SLICES * I8_N * I8_ROWB;  // 5120: the five planes of a B chunk
constexpr uint32_t I8_LBO = 128;                       // K-adjacent core matrices
constexpr uint32_t I8_SBO = 256;                       // 8-row groups
constexpr int I8_TMEM_COLS = 512;
constexpr int I8_SET_COLS = I8_LEVELS * I8_N;          // 192

static_assert(I8_SETS * I8_SET_COLS <= I8_TMEM_COLS, "accumulators fit TMEM");

// Instruction descriptor: kind::i8, D = S32, A = B = signed 8-bit, both
// K-major, M = 128; N is or-ed in per tile.
constexpr uint32_t I8_IDESC = (2u << 4)                         // D format S32
                              | (1u << 7)                       // A signed 8-bit
                              | (1u << 10)                      // B signed 8-bit
                              | ((uint32_t)(I8_M >> 4) << 24);  // M
__device__ __forceinline__ uint32_t idesc_n(int n) { return I8_IDESC | ((uint32_t)(n >> 3) << 17); }

__device__ __forceinline__ void umma_i8(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate));
}

// Byte offset of (row r, K half kg) inside one plane of a tile.
__device__ __forceinline__ int plane_off(int r, int kg) { return (r >> 3) * (int)I8_SBO + kg * 128 + (r & 7) * 16; }

// Row scale: 2^e with max|x| < 0.9921875 2^e (e >= -960 so that 2^(39 - e)
// stays finite); sc39 = 2^(39 - e) for the digits, s23 = 2^(e - 23) for the
// recombination.
__device__ __forceinline__ void digit_scale(double m, double *sc39, double *s23) {
  int e = 0;
  if (m > 0.0) {
    const double f = frexp(m, &e);
    if (f >= 0.9921875) ++e;
  }
  e = max(e, -960);
  *sc39 = ldexp(1.0, 39 - e);
  *s23 = ldexp(1.0, e - 23);
}

// The digits of one value.
//   t = fma(x, sc39, 1.5 2^52) holds X = rint(x sc39) in its mantissa, so
//   bits(t) - 0x4338000000000000 = X exactly; X + 0x80808080 = a0 2^32 + sum
//   c_s 2^(8 (4 - s)) with bytes c_s in [0, 255], i.e. the balanced digits
//   a_s = c_s - 128 (= c_s ^ 0x80 as a signed byte) and a0 the high word.
__device__ __forceinline__ void digit_bits(double x, double sc39, int *hi, uint32_t *lo) {
  const double t = fma(x, sc39, 6755399441055744.0);
  const long long xp = __double_as_longlong(t) + (0x80808080LL - 0x4338000000000000LL);
  *hi = (int)(xp >> 32);
  *lo = (uint32_t)xp;
}

// Four values' digits as one word per plane.
__device__ __forceinline__ void digit_words(const int *hi, const uint32_t *lo, uint32_t (&plane)[I8_SLICES]) {
  plane[0] = __byte_perm(__byte_perm((uint32_t)hi[0], (uint32_t)hi[1], 0x40),
                         __byte_perm((uint32_t)hi[2], (uint32_t)hi[3], 0x40), 0x5410);
#pragma unroll
  for (int s = 1; s < I8_SLICES; ++s) {
    const uint32_t b = (uint32_t)(4 - s), sel = b | ((b + 4) << 4);
    plane[s] = __byte_perm(__byte_perm(lo[0], lo[1], sel), __byte_perm(lo[2], lo[3], sel), 0x5410) ^ 0x80808080u;
  }
}

// Sixteen consecutive values of one row as five 16-byte digit planes.
__device__ __forceinline__ void digits16(const double (&x)[16], double sc39, uint4 (&plane)[I8_SLICES]) {
  int hi[16];
  uint32_t lo[16], w[4][I8_SLICES];
#pragma unroll
  for (int j = 0; j < 16; ++j) digit_bits(x[j], sc39, &hi[j], &lo[j]);
#pragma unroll
  for (int q = 0; q < 4; ++q) digit_words(hi + 4 * q, lo + 4 * q, w[q]);
#pragma unroll
  for (int s = 0; s < I8_SLICES; ++s) plane[s] = make_uint4(w[0][s], w[1][s], w[2][s], w[3][s]);
}

// ------------------------------------------------------------ pack kernels

// Four doubles from a 32-byte aligned address, not kept in L1.
__device__ __forceinline__ void ld4(const double *p, double *v) {
  asm volatile("ld.global.nc.L1::no_allocate.v4.f64 {%0,%1,%2,%3}, [%4];"
               : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3])
               : "l"(p));
}

constexpr int PA_ROWS = 8;  // rows (points) per CTA: one 8-row group of the tile image
constexpr int PA_GROUPS = I8_M / PA_ROWS;
constexpr int PA_WARPS = 8;
constexpr int PA_THREADS = 32 * PA_WARPS;

// Four values of one row -> one 32-bit word of each digit plane (see digit_bits).
__device__ __forceinline__ void digits4(const double (&x)[4], double sc39, uint32_t (&plane)[I8_SLICES]) {
  int hi[4];
  uint32_t lo[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) digit_bits(x[j], sc39, &hi[j], &lo[j]);
  digit_words(hi, lo, plane);
}

// phi of eight points of one work item -> A scratch: chunk kc, plane s at
// a_off + (5 kc + s) rows8 32 bytes; rows pn..rows8-1 and k >= nc are zero.
// Memory bound: phi is read (for the digits a second time, from L2) and five
// bytes a value are written.  Lane (row r = lane / 4, quarter q = lane % 4) of
// warp w takes the values 16 kg + 4 q..+3 of row r for kg = w, w + 8, ...: a
// warp's load covers 128 contiguous bytes of each of its eight rows and its
// stores 128 contiguous bytes of a plane.  A CTA lives for one chain of
// latencies, so what counts is how many of them an SM holds: with all 2048
// threads and the second read 1.52 ms for 8,000 batches of 100-600 functions
// (7.3 GB in and out), with the values kept in registers between the maximum
// and the digits 2.31 ms (three CTAs an SM), and 1.86 ms for sixteen points at
// a time in a CTA per item.
__global__ void __launch_bounds__(PA_THREADS, 2048 / PA_THREADS) i8_pack_a_kernel(const I8Item *__restrict__ items,
                                                               const double *__restrict__ wave,
                                                               unsigned char *__restrict__ a_scr,
                                                               double *__restrict__ sa, int vec) {
  __shared__ double s_max[PA_WARPS][PA_ROWS];
  const I8Item &W = items[blockIdx.x / PA_GROUPS];
  const int row0 = (int)(blockIdx.x % PA_GROUPS) * PA_ROWS;
  if (row0 >= W.rows8) return;
  const int nc = W.nc, ncp = (nc + 3) & ~3, n_kg = 2 * W.n_kc;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = lane >> 2, q = lane & 3;
  const int p = row0 + r;
  const bool live = p < W.pn;
  const double *row = wave + W.wave_off + (long long)(W.p0 + (live ? p : 0)) * ncp + 4 * q;
  const int kend = live ? nc - 4 * q : 0;  // values of this lane's row from its quarter on
  auto load = [&](int kg, double (&x)[4]) {
    const int k = 16 * kg;
    if (vec) {  // rows start on 32-byte boundaries; a vector that starts below nc ends by ncp
      if (k < kend) {
        ld4(row + k, x);
#pragma unroll
        for (int j = 1; j < 4; ++j) x[j] = k + j < kend ? x[j] : 0.0;  // the row padding
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) x[j] = 0.0;
      }
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) x[j] = k + j < kend ? __ldg(row + k + j) : 0.0;
    }
  };
  double m = 0.0;
#pragma unroll 2
  for (int kg = warp; kg < n_kg; kg += PA_WARPS) {
    double x[4];
    load(kg, x);
#pragma unroll
    for (int j = 0; j < 4; ++j) m = fmax(m, fabs(x[j]));
  }
  m = fmax(m, __shfl_xor_sync(0xffffffffu, m, 1));
  m = fmax(m, __shfl_xor_sync(0xffffffffu, m, 2));
  if (q == 0) s_max[warp][r] = m;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < PA_WARPS; ++w) m = fmax(m, s_max[w][r]);
  double sc39, s23;
  digit_scale(m, &sc39, &s23);
  if (warp == 0 && q == 0) sa[W.sa_off + p] = s23;
  const long long plane_bytes = (long long)W.rows8 * I8_ROWB;
  unsigned char *dst = a_scr + W.a_off + plane_off(p, 0) + 4 * q;
#pragma unroll 2
  for (int kg = warp; kg < n_kg; kg += PA_WARPS) {
    double x[4];
    uint32_t w[I8_SLICES];
    load(kg, x);
    digits4(x, sc39, w);
    unsigned char *d = dst + (kg >> 1) * I8_SLICES * plane_bytes + (kg & 1) * I8_LBO;
#pragma unroll
    for (int s = 0; s < I8_SLICES; ++s) *reinterpret_cast<uint32_t *>(d + s * plane_bytes) = w[s];
  }
}

constexpr int PB_WARPS = 4;
constexpr int PB_THREADS = 32 * PB_WARPS;

// P1c rows of one N tile -> B scratch: chunk kc, plane s at
// b_off + (5 kc + s) 1024 bytes; rows >= nc and k >= nc are zero.  Lane = row
// (P1's contiguous index), warp w takes the 16-wide K groups w, w + 4, ...; a
// group's sixteen column indices come from shared memory as four 128-bit
// broadcasts, and its sixteen gathers are in flight together.
__global__ void __launch_bounds__(PB_THREADS) i8_pack_b_kernel(const I8BTile *__restrict__ tiles,
                                                               const int *__restrict__ ib_all,
                                                               const double *__restrict__ P1,
                                                               const double *__restrict__ rowmax, int n_basis,
                                                               unsigned char *__restrict__ b_scr,
                                                               double *__restrict__ sb) {
  __shared__ __align__(16) int s_ib[(FRPA_MAX_N_COMPUTE + 31) / 32 * 32];
  const I8BTile B = tiles[blockIdx.x];
  const int nc = B.nc;
  for (int i = threadIdx.x; i < B.n_kc * I8_KC; i += PB_THREADS)
    s_ib[i] = i < nc ? __ldg(ib_all + B.ib_off + i) - 1 : 0;
  __syncthreads();
  const int r = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i = B.jn * I8_N + r;
  const bool rok = i < nc;
  const int ibr = rok ? s_ib[i] : 0;
  const double *col = P1 + (long long)n_basis * n_basis * B.t + ibr;
  double sc39, s23;
  digit_scale(rok ? __ldg(rowmax + ibr + (long long)n_basis * B.t) : 0.0, &sc39, &s23);
  if (warp == 0) sb[B.sb_off + r] = rok ? s23 * 0.00390625 : 0.0;  // 2^(e - 31): the recombination sums 256 S
  unsigned char *dst = b_scr + B.b_off + plane_off(r, 0);
  for (int kg = warp; kg < 2 * B.n_kc; kg += PB_WARPS) {
    const int k0 = kg * 16, kn = rok ? nc - k0 : 0;
    double x[16];
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const int4 id = *reinterpret_cast<const int4 *>(s_ib + k0 + 4 * v);
      x[4 * v + 0] = 4 * v + 0 < kn ? __ldg(col + (long long)id.x * n_basis) : 0.0;
      x[4 * v + 1] = 4 * v + 1 < kn ? __ldg(col + (long long)id.y * n_basis) : 0.0;
      x[4 * v + 2] = 4 * v + 2 < kn ? __ldg(col + (long long)id.z * n_basis) : 0.0;
      x[4 * v + 3] = 4 * v + 3 < kn ? __ldg(col + (long long)id.w * n_basis) : 0.0;
    }
    uint4 plane[I8_SLICES];
    digits16(x, sc39, plane);
    unsigned char *d = dst + (kg >> 1) * I8_B_CHUNK + (kg & 1) * I8_LBO;
#pragma unroll
    for (int s = 0; s < I8_SLICES; ++s) *reinterpret_cast<uint4 *>(d + s * I8_N * I8_ROWB) = plane[s];
  }
}

// ------------------------------------------------------ contraction kernel

struct I8Smem {
  unsigned char A[I8_STAGES][I8_CHUNKS * I8_SLICES * I8_A_PLANE];  // chunks and planes at their packed distance
  unsigned char B[I8_STAGES][I8_CHUNKS * I8_B_CHUNK];
  double partial[2][4][I8_M];              // upper column half's per-point sums
  unsigned long long full[I8_STAGES];
  unsigned long long empty[I8_STAGES];
  unsigned long long acc_full[I8_SETS];
  unsigned long long acc_empty[I8_SETS];
  unsigned long long drain;
  unsigned long long ep_sum[2];   // partial sums published by the upper column half
  unsigned long long ep_free[2];  // partial-sum buffer released by the lower half
  uint32_t tmem_base;
  int abort_flag;
};

struct I8Params {
  const I8Item *items;
  int n_items;
  const int *map;
  int T, n_active, n_full_points, n_max_batch_size, n_batches;
  const double *wave, *gwave, *bias, *gbias;
  const unsigned char *a_scr, *b_scr;
  const double *sa, *sb;
  double *rho, *grad;
  int *err;
  int wave_vec;  // every phi / grad phi row starts on a 32-byte boundary: 256-bit loads
};

// A warp-uniform value as the compiler can see it (uniform registers feed the
// descriptors and loop bounds of the issuing warps).
__device__ __forceinline__ int uniform(int x) { return __shfl_sync(0xffffffffu, x, 0); }

// The loader warp (converged, one elected lane issues): every stage's A planes
// and B planes, one bulk copy each, into the ring.  The planes of an A chunk
// keep their packed distance of rows8 x 32 bytes, so that they are one copy:
// issuing a copy takes ~70 cycles, and one per plane kept the loader busy for
// 460 of a chunk's 660 cycles.
__device__ void loader_role(const I8Params &P, I8Smem &S) {
  volatile int *abort_flag = &S.abort_flag;
  uint32_t fill = 0;
  for (int it = blockIdx.x; it < P.n_items; it += gridDim.x) {
    const I8Item &W = P.items[it];
    const int n_kc = uniform(W.n_kc), n_nt = uniform(W.n_nt);
    const uint32_t a_bytes = (uint32_t)(uniform(W.rows8) * I8_SLICES * I8_ROWB);
    const unsigned char *asrc = P.a_scr + W.a_off;
    for (int t = 0; t < P.T; ++t) {
      const unsigned char *bsrc = P.b_scr + W.b_off + t * W.b_tstride;  // the tiles' chunks, back to back
      for (int jn = 0; jn < n_nt; ++jn)
        for (int kc = 0; kc < n_kc; kc += I8_CHUNKS, ++fill) {
          const int st = fill % I8_STAGES;
          const uint32_t n = (uint32_t)min(I8_CHUNKS, n_kc - kc);
          if (!warp_wait_all(&S.empty[st], ((fill / I8_STAGES) & 1) ^ 1, abort_flag, P.err)) goto out;
          if (elect_one()) {
            mbar_arrive_expect_tx(&S.full[st], n * (a_bytes + I8_B_CHUNK));
            bulk_g2s(S.A[st], asrc + (long long)kc * a_bytes, n * a_bytes, &S.full[st]);
            bulk_g2s(S.B[st], bsrc, n * I8_B_CHUNK, &S.full[st]);
          }
          __syncwarp();
          bsrc += n * I8_B_CHUNK;
        }
    }
  }
out:
  // the copies of the last (up to) I8_STAGES fills land before the CTA exits
  const uint32_t n = fill < (uint32_t)I8_STAGES ? fill : (uint32_t)I8_STAGES;
  for (uint32_t f = fill - n; f < fill; ++f)
    if (!mbar_wait_quiet(&S.full[f % I8_STAGES], (f / I8_STAGES) & 1)) atomicOr(P.err, 4);
}

// One K chunk's 19 digit products (five MMAs; six in a tile's first chunk).
// Digit levels run along N: B planes 0..m of a chunk are one contiguous matrix
// of 32 (m + 1) rows, so A plane s times planes 0..min(4, 5-s), written from
// accumulator column 32 s on, puts product (s, u) into the columns of level
// s + u.  In the first chunk A plane 1 starts levels 1..5 and plane 0 level 0.
template <bool FIRST>
__device__ __forceinline__ void chunk_mmas(uint32_t dcol, uint64_t adesc, uint32_t plane, uint64_t bdesc) {
  if (FIRST) {
    umma_i8(dcol + I8_N, adesc + plane, bdesc, idesc_n(5 * I8_N), 0u);
    umma_i8(dcol, adesc, bdesc, idesc_n(I8_N), 0u);
    umma_i8(dcol + I8_N, adesc, bdesc + (I8_N * I8_ROWB >> 4), idesc_n(4 * I8_N), 1u);
  } else {
    umma_i8(dcol, adesc, bdesc, idesc_n(5 * I8_N), 1u);
    umma_i8(dcol + I8_N, adesc + plane, bdesc, idesc_n(5 * I8_N), 1u);
  }
  umma_i8(dcol + 2 * I8_N, adesc + 2 * plane, bdesc, idesc_n(4 * I8_N), 1u);
  umma_i8(dcol + 3 * I8_N, adesc + 3 * plane, bdesc, idesc_n(3 * I8_N), 1u);
  umma_i8(dcol + 4 * I8_N, adesc + 4 * plane, bdesc, idesc_n(2 * I8_N), 1u);
}

// The MMA warp (converged, one elected lane issues): per N tile, all K chunks
// into the six level accumulators of the tile's set (sets alternate by tile).
// Rows rows8..127 of an A plane are the next plane's bytes: they only reach
// TMEM lanes that no epilogue thread uses.
__device__ void mma_role(const I8Params &P, I8Smem &S, uint32_t tmem) {
  volatile int *abort_flag = &S.abort_flag;
  uint32_t fill = 0, tile_ctr = 0;
  for (int it = blockIdx.x; it < P.n_items; it += gridDim.x) {
    const I8Item &W = P.items[it];
    const int n_kc = uniform(W.n_kc), n_tiles = uniform(W.n_nt) * P.T;
    const uint32_t plane = (uint32_t)(uniform(W.rows8) * I8_ROWB) >> 4;  // descriptor units
    for (int j = 0; j < n_tiles; ++j, ++tile_ctr) {
      const int set = tile_ctr & 1;
      const uint32_t dcol = tmem + (uint32_t)(set * I8_SET_COLS);
      if (!warp_wait_all(&S.acc_empty[set], ((tile_ctr >> 1) & 1) ^ 1, abort_flag, P.err)) goto out;
      for (int kc = 0; kc < n_kc; kc += I8_CHUNKS, ++fill) {
        const int st = fill % I8_STAGES;
        if (!warp_wait_all(&S.full[st], (fill / I8_STAGES) & 1, abort_flag, P.err)) goto out;
        tc_fence_after();
        if (elect_one()) {
          const uint64_t adesc = smem_desc<I8_LBO, I8_SBO>(smem_u32(S.A[st]));
          const uint64_t bdesc = smem_desc<I8_LBO, I8_SBO>(smem_u32(S.B[st]));
          if (kc == 0)
            chunk_mmas<true>(dcol, adesc, plane, bdesc);
          else
            chunk_mmas<false>(dcol, adesc, plane, bdesc);
#pragma unroll
          for (int q = 1; q < I8_CHUNKS; ++q)
            if (kc + q < n_kc)
              chunk_mmas<false>(dcol, adesc + q * I8_SLICES * plane, plane, bdesc + q * (I8_B_CHUNK >> 4));
          umma_commit(&S.empty[st]);
          if (kc + I8_CHUNKS >= n_kc) umma_commit(&S.acc_full[set]);
        }
        __syncwarp();
      }
    }
  }
out:
  // no MMA may be in flight when TMEM is released
  if (elect_one()) umma_commit(&S.drain);
  __syncwarp();
  if (!mbar_wait_quiet(&S.drain, 0)) atomicOr(P.err, 4);
}

// FP64 operands of one four-column step of an epilogue warp: phi and
// grad phi at rows i0..i0+3 of one point's column.  Values at rows >=
// n_compute (the row padding, possibly garbage) are masked where they are used.
struct EpiRegs {
  double f[4], gx[4], gy[4], gz[4];
};

__device__ __forceinline__ void epi_load(EpiRegs &E, const double *__restrict__ phi, const double *__restrict__ gph,
                                         int ncp, int nc, int i0, bool live, bool vec) {
  if (vec) {  // 32-byte loads: i0 and the row starts are multiples of 4, rows end at ncp >= i0 + 4
    if (live && i0 < nc) {
      ld4(phi + i0, E.f);
      ld4(gph + i0, E.gx);
      ld4(gph + ncp + i0, E.gy);
      ld4(gph + 2 * ncp + i0, E.gz);
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) E.f[e] = E.gx[e] = E.gy[e] = E.gz[e] = 0.0;
    }
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const bool ok = live && i0 + j < nc;
      E.f[j] = ok ? __ldg(phi + i0 + j) : 0.0;
      E.gx[j] = ok ? __ldg(gph + i0 + j) : 0.0;
      E.gy[j] = ok ? __ldg(gph + i0 + j + ncp) : 0.0;
      E.gz[j] = ok ? __ldg(gph + i0 + j + 2 * ncp) : 0.0;
    }
  }
}

// Four columns of a tile: recombine the six levels in FP64 and contract with
// phi and grad phi; rows at or past `lim` are outside n_compute.
__device__ __forceinline__ void epi_step(const EpiRegs &E, uint32_t acc, const double *__restrict__ sbv, int lim,
                                            double &r, double &gx, double &gy, double &gz) {
  uint32_t v[I8_LEVELS][4];
#pragma unroll
  for (int l = 0; l < I8_LEVELS; ++l) tmem_ld4(acc + (uint32_t)(l * I8_N), v[l]);
  tmem_wait_ld();
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    // 256 S = (L0 256 + L1) 2^32 + (L2 256 + L3) 2^16 + (L4 256 + L5), each pair exact in int64
    const long long hi = (long long)(int)v[0][e] * 256 + (int)v[1][e];
    const long long mid = (long long)(int)v[2][e] * 256 + (int)v[3][e];
    const long long lo = (long long)(int)v[4][e] * 256 + (int)v[5][e];
    const double w = fma((double)hi, 4294967296.0, fma((double)mid, 65536.0, (double)lo)) * __ldg(sbv + e);
    const bool ok = e < lim;
    r = fma(ok ? E.f[e] : 0.0, w, r);
    gx = fma(ok ? E.gx[e] : 0.0, w, gx);
    gy = fma(ok ? E.gy[e] : 0.0, w, gy);
    gz = fma(ok ? E.gz[e] : 0.0, w, gz);
  }
}

// Epilogue warp w reads TMEM lanes 32 (w % 4).. (its points) and columns
// 16 (w / 4)..+15 of each level accumulator of the tile's set, four at a time.
// The phi / grad phi registers of a four-column step are loaded again as soon
// as the step is done, two steps ahead of their use and across the tiles of an
// item.  The set is released after its last read; meanwhile the MMAs of the
// next tile fill the other set.  The two warps of a lane quarter add their
// partial sums through shared memory at each perturbation's end.
__device__ void epilogue_role(const I8Params &P, I8Smem &S, uint32_t tmem, int warp, int lane) {
  int *err = P.err;
  volatile int *abort_flag = &S.abort_flag;
  const int quarter = warp & 3, half = warp >> 2;
  const int p = quarter * 32 + lane;  // TMEM lane = point within the tile
  const uint32_t lane_base = tmem + ((uint32_t)(quarter * 32) << 16);
  const int cbase = half * I8_COLS;
  const bool vec = P.wave_vec != 0;
  uint32_t tile_ctr = 0, sum_ctr = 0;
  for (int it = blockIdx.x; it < P.n_items; it += gridDim.x) {
    const I8Item &W = P.items[it];
    const int nc = W.nc, ncp = (nc + 3) & ~3, n_nt = W.n_nt;
    const bool live = p < W.pn;
    const long long pt = W.p0 + (live ? p : 0);
    const double *phi = P.wave + W.wave_off + pt * ncp;
    const double *gph = P.gwave + 3 * W.wave_off + 3 * pt * ncp;
    EpiRegs E[EPI_BUFS];
#pragma unroll
    for (int q = 0; q < EPI_BUFS; ++q) epi_load(E[q], phi, gph, ncp, nc, cbase + 4 * q, live, vec);
    for (int t = 0; t < P.T; ++t) {
      double r = 0.0, gx = 0.0, gy = 0.0, gz = 0.0;
      const double *sbv = P.sb + W.sb_off + (long long)t * W.sb_tstride + cbase;
      for (int jn = 0; jn < n_nt; ++jn, ++tile_ctr, sbv += I8_N) {
        const int set = tile_ctr & 1;
        const uint32_t acc = lane_base + (uint32_t)(set * I8_SET_COLS + cbase);
        const int lim = live ? nc - (jn * I8_N + cbase) : 0;  // rows from this column on inside n_compute
        const int next = (jn + 1 < n_nt ? (jn + 1) * I8_N : (t + 1 < P.T ? 0 : nc)) + cbase;
        if (!warp_wait(&S.acc_full[set], (tile_ctr >> 1) & 1, abort_flag, err, lane)) return;
        tc_fence_after();
#pragma unroll
        for (int q = 0; q < I8_COLS / 4; ++q) {
          epi_step(E[q % EPI_BUFS], acc + 4 * q, sbv + 4 * q, lim - 4 * q, r, gx, gy, gz);
          if (q == I8_COLS / 4 - 1) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&S.acc_empty[set]);
          }
          const int ahead = 4 * (q + EPI_BUFS);
          epi_load(E[q % EPI_BUFS], phi, gph, ncp, nc,
                   ahead < I8_COLS ? jn * I8_N + cbase + ahead : next + ahead - I8_COLS, live, vec);
        }
      }
      // combine the two column halves of this point and write
      const int sp = sum_ctr & 1;
      if (half == 1) {
        if (!warp_wait(&S.ep_free[sp], ((sum_ctr >> 1) & 1) ^ 1, abort_flag, err, lane)) return;
        S.partial[sp][0][p] = r;
        S.partial[sp][1][p] = gx;
        S.partial[sp][2][p] = gy;
        S.partial[sp][3][p] = gz;
        mbar_arrive(&S.ep_sum[sp]);
      } else {
        if (!warp_wait(&S.ep_sum[sp], (sum_ctr >> 1) & 1, abort_flag, err, lane)) return;
        r += S.partial[sp][0][p];
        gx += S.partial[sp][1][p];
        gy += S.partial[sp][2][p];
        gz += S.partial[sp][3][p];
        mbar_arrive(&S.ep_free[sp]);
        if (live) {
          const double sA = P.sa[W.sa_off + p];
          const int pp = W.p0 + p;
          const long long bidx = pp + (long long)P.n_max_batch_size * (W.batch + (long long)P.n_batches * t);
          P.grad[3 * bidx + 0] = (gx * sA) * 2 - P.gbias[3 * bidx + 0];
          P.grad[3 * bidx + 1] = (gy * sA) * 2 - P.gbias[3 * bidx + 1];
          P.grad[3 * bidx + 2] = (gz * sA) * 2 - P.gbias[3 * bidx + 2];
          if (t < P.n_active) P.rho[P.map[W.prefix + pp] + (long long)P.n_full_points * t] = r * sA + P.bias[bidx];
        }
      }
      ++sum_ctr;
    }
  }
}

__global__ void __launch_bounds__(I8_THREADS, 1) rho1_i8_kernel(const I8Params P) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  I8Smem &S = *reinterpret_cast<I8Smem *>(smem_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int s = 0; s < I8_STAGES; ++s) {
      mbar_init(&S.full[s], 1);
      mbar_init(&S.empty[s], 1);
    }
    for (int s = 0; s < I8_SETS; ++s) {
      mbar_init(&S.acc_full[s], 1);
      mbar_init(&S.acc_empty[s], I8_EPI_WARPS);
    }
    mbar_init(&S.drain, 1);
    for (int h = 0; h < 2; ++h) {
      mbar_init(&S.ep_sum[h], I8_M);
      mbar_init(&S.ep_free[h], I8_M);
    }
    S.abort_flag = 0;
    mbar_init_fence();
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&S.tmem_base)),
                 "r"(I8_TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = S.tmem_base;

  if (warp < I8_EPI_WARPS) {
    epilogue_role(P, S, tmem, warp, lane);
    __syncwarp();
  } else if (warp == I8_LOAD_WARP) {
    loader_role(P, S);
    __syncwarp();
  } else if (warp == I8_MMA_WARP) {
    mma_role(P, S, tmem);
    __syncwarp();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(I8_TMEM_COLS));
  }
}

int i8_smem_bytes() { return (int)sizeof(I8Smem) + 128; }

}  // namespace

// Work lists and groups from the plan's valid batches: batches by decreasing
// cost (nc^2 np), each split into point tiles of <= 128 points (evenly), the
// tiles of a batch adjacent; consecutive batches form a group while its A + B
// scratch stays within plan->i8_budget (a batch larger than that is a group
// of its own).
int rho1_i8_build(Rho1Plan *plan) {
  // Groups follow the lexicographic order of the batches' (ascending) basis
  // lists, so that batches over the same atoms are packed together and
  // their P1c gathers meet in L2; inside a group the contraction takes the
  // batches by decreasing cost (nc^2 np), a batch's point tiles adjacent.
  std::vector<Rho1WorkItem> batches = plan->h_batches;
  const int *ibh = plan->h_ib.data();
  std::stable_sort(batches.begin(), batches.end(), [ibh](const Rho1WorkItem &a, const Rho1WorkItem &b) {
    return std::lexicographical_compare(ibh + a.ib_off, ibh + a.ib_off + a.nc, ibh + b.ib_off, ibh + b.ib_off + b.nc);
  });
  const int T = plan->T;
  std::vector<I8Item> items;
  std::vector<I8BTile> tiles;
  std::vector<I8Group> groups;
  I8Group g{0, 0, 0, 0, 0, 0, 0, 0};
  for (const Rho1WorkItem &bt : batches) {
    if (bt.np == 0) continue;
    const int nc = bt.nc, n_nt = ceil_div(nc, I8_N), n_kc = ceil_div(nc, I8_KC);
    const long long b_t = (long long)n_nt * n_kc * I8_B_CHUNK;  // the last N tile is padded with zero rows
    const int ntiles = ceil_div(bt.np, I8_M), width = ceil_div(bt.np, ntiles);
    long long a_need = 0;
    for (int p0 = 0; p0 < bt.np; p0 += width) {
      const int pn = std::min(width, bt.np - p0);
      a_need += (long long)n_kc * I8_SLICES * (((pn + 7) / 8) * 8) * I8_ROWB;
    }
    const long long need = a_need + b_t * T;
    if (g.item1 > g.item0 && g.a_bytes + g.b_bytes + need > plan->i8_budget) {
      groups.push_back(g);
      g = I8Group{(int)items.size(), (int)items.size(), (int)tiles.size(), (int)tiles.size(), 0, 0, 0, 0};
    }
    const long long b_off = g.b_bytes;
    const int sb_off = g.sb_len;
    for (int t = 0; t < T; ++t)
      for (int jn = 0; jn < n_nt; ++jn)
        tiles.push_back(I8BTile{bt.ib_off, nc, jn, t, n_kc, sb_off + t * n_nt * I8_N + jn * I8_N,
                                b_off + t * b_t + (long long)jn * n_kc * I8_B_CHUNK});
    for (int p0 = 0; p0 < bt.np; p0 += width) {
      const int pn = std::min(width, bt.np - p0), rows8 = ((pn + 7) / 8) * 8;
      I8Item it{};
      it.batch = bt.batch;
      it.nc = nc;
      it.p0 = p0;
      it.pn = pn;
      it.prefix = bt.prefix;
      it.rows8 = rows8;
      it.n_nt = n_nt;
      it.n_kc = n_kc;
      it.wave_off = bt.wave_off;
      it.a_off = g.a_bytes;
      it.b_off = b_off;
      it.b_tstride = b_t;
      it.sa_off = g.sa_len;
      it.sb_off = sb_off;
      it.sb_tstride = n_nt * I8_N;
      items.push_back(it);
      g.a_bytes += (long long)n_kc * I8_SLICES * rows8 * I8_ROWB;
      g.sa_len += I8_M;
    }
    g.b_bytes += b_t * T;
    g.sb_len += T * n_nt * I8_N;
    g.item1 = (int)items.size();
    g.tile1 = (int)tiles.size();
  }
  if (g.item1 > g.item0) groups.push_back(g);
  for (const I8Group &q : groups)  // cost order inside each group (siblings stay adjacent)
    std::stable_sort(items.begin() + q.item0, items.begin() + q.item1, [](const I8Item &a, const I8Item &b) {
      return a.nc != b.nc ? a.nc > b.nc : a.batch < b.batch;
    });
  plan->i8_wave4 = 1;
  for (const Rho1WorkItem &bt : batches)
    if (bt.wave_off & 3) plan->i8_wave4 = 0;
  cudaFree(plan->d_i8_items);
  cudaFree(plan->d_i8_tiles);
  plan->d_i8_items = nullptr;
  plan->d_i8_tiles = nullptr;
  plan->i8_groups = groups;
  if (items.empty()) return FRPA_OK;
  if (cudaMalloc((void **)&plan->d_i8_items, sizeof(I8Item) * items.size()) != cudaSuccess ||
      cudaMalloc((void **)&plan->d_i8_tiles, sizeof(I8BTile) * tiles.size()) != cudaSuccess)
    return fail(FRPA_ERR_OOM, "rho1 split-int8: work list allocation failed");
  FRPA_CUDA_TRY(cudaMemcpy(plan->d_i8_items, items.data(), sizeof(I8Item) * items.size(), cudaMemcpyHostToDevice));
  FRPA_CUDA_TRY(cudaMemcpy(plan->d_i8_tiles, tiles.data(), sizeof(I8BTile) * tiles.size(), cudaMemcpyHostToDevice));
  return FRPA_OK;
}

static void i8_free_scratch(Rho1Plan *plan) {
  for (int k = 0; k < 2; ++k) {
    cudaFree(plan->d_i8_a[k]);
    cudaFree(plan->d_i8_b[k]);
    cudaFree(plan->d_i8_sa[k]);
    cudaFree(plan->d_i8_sb[k]);
    plan->d_i8_a[k] = plan->d_i8_b[k] = nullptr;
    plan->d_i8_sa[k] = plan->d_i8_sb[k] = nullptr;
  }
}

void rho1_i8_free(Rho1Plan *plan) {
  cudaFree(plan->d_i8_items);
  cudaFree(plan->d_i8_tiles);
  plan->d_i8_items = nullptr;
  plan->d_i8_tiles = nullptr;
  i8_free_scratch(plan);
  if (plan->i8_side) cudaStreamDestroy(plan->i8_side);
  if (plan->i8_ev_start) cudaEventDestroy(plan->i8_ev_start);
  for (int k = 0; k < 2; ++k) {
    if (plan->i8_ev_packed[k]) cudaEventDestroy(plan->i8_ev_packed[k]);
    if (plan->i8_ev_done[k]) cudaEventDestroy(plan->i8_ev_done[k]);
    plan->i8_ev_packed[k] = plan->i8_ev_done[k] = nullptr;
  }
  plan->i8_side = nullptr;
  plan->i8_ev_start = nullptr;
}

// Scratch sets sized for the largest group (two when there are several
// groups) and the side stream, created on first use (not while the stream is
// being captured into a graph).
static int i8_scratch(Rho1Plan &plan, cudaStream_t stream) {
  if (plan.d_i8_a[0]) return FRPA_OK;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  FRPA_CUDA_TRY(cudaStreamIsCapturing(stream, &cap));
  if (cap != cudaStreamCaptureStatusNone)
    return fail(FRPA_ERR_INVALID,
                "rho1 split-int8: the packed-operand scratch is allocated by the first execution; execute once "
                "before capturing a graph");
  long long a = 16, b = 16;
  int sa = 1, sb = 1;
  for (const I8Group &g : plan.i8_groups) {
    a = std::max(a, g.a_bytes);
    b = std::max(b, g.b_bytes);
    sa = std::max(sa, g.sa_len);
    sb = std::max(sb, g.sb_len);
  }
  const int sets = plan.i8_groups.size() > 1 ? 2 : 1;
  for (int k = 0; k < sets; ++k)
    if (cudaMalloc((void **)&plan.d_i8_a[k], a) != cudaSuccess ||
        cudaMalloc((void **)&plan.d_i8_b[k], b) != cudaSuccess ||
        cudaMalloc((void **)&plan.d_i8_sa[k], sizeof(double) * sa) != cudaSuccess ||
        cudaMalloc((void **)&plan.d_i8_sb[k], sizeof(double) * sb) != cudaSuccess) {
      i8_free_scratch(&plan);
      return fail(FRPA_ERR_OOM, "rho1 split-int8: %d scratch sets of %lld + %lld bytes could not be allocated",
                  sets, a, b);
    }
  if (!plan.i8_side) {
    FRPA_CUDA_TRY(cudaStreamCreateWithFlags(&plan.i8_side, cudaStreamNonBlocking));
    FRPA_CUDA_TRY(cudaEventCreateWithFlags(&plan.i8_ev_start, cudaEventDisableTiming));
    for (int k = 0; k < 2; ++k) {
      FRPA_CUDA_TRY(cudaEventCreateWithFlags(&plan.i8_ev_packed[k], cudaEventDisableTiming));
      FRPA_CUDA_TRY(cudaEventCreateWithFlags(&plan.i8_ev_done[k], cudaEventDisableTiming));
    }
  }
  return FRPA_OK;
}

int rho1_i8_launch(Rho1Plan &plan, int n_active, const double *wave, const double *gwave, const double *P1,
                   const double *bias, const double *gbias, double *rho, double *grad, cudaStream_t stream) {
  FRPA_CUDA_TRY(cudaMemsetAsync(rho, 0, sizeof(double) * (size_t)plan.n_full_points * plan.T, stream));
  FRPA_CUDA_TRY(cudaMemsetAsync(
      grad, 0, sizeof(double) * 3 * (size_t)plan.n_max_batch_size * plan.n_batches * plan.T, stream));
  if (plan.i8_groups.empty()) return FRPA_OK;
  FRPA_TRY(i8_scratch(plan, stream));
  FRPA_TRY(p1_rowmax_launch(plan, P1, stream));
  static PerDeviceOnce configured;
  const int smem = i8_smem_bytes();
  FRPA_TRY(configured.run(plan.device, [smem]() -> int {
    FRPA_CUDA_TRY(cudaFuncSetAttribute(rho1_i8_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    return FRPA_OK;
  }));
  int n_sm = 148;
  FRPA_CUDA_TRY(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, plan.device));
  I8Params P;
  P.map = plan.d_map;
  P.T = plan.T;
  P.n_active = n_active;
  P.n_full_points = plan.n_full_points;
  P.n_max_batch_size = plan.n_max_batch_size;
  P.n_batches = plan.n_batches;
  P.wave = wave;
  P.gwave = gwave;
  P.bias = bias;
  P.gbias = gbias;
  P.rho = rho;
  P.grad = grad;
  P.err = plan.d_err;
  P.wave_vec = (plan.i8_wave4 && !(((uintptr_t)wave | (uintptr_t)gwave) & 31)) ? 1 : 0;
  // group g: packed on the side stream into scratch set g % 2 (after the
  // contraction of group g - 2 released it), contracted on the caller's
  // stream; the side stream joins back before the last contraction
  const int sets = plan.d_i8_a[1] ? 2 : 1;
  FRPA_CUDA_TRY(cudaEventRecord(plan.i8_ev_start, stream));
  FRPA_CUDA_TRY(cudaStreamWaitEvent(plan.i8_side, plan.i8_ev_start, 0));
  const int n_groups = (int)plan.i8_groups.size();
  for (int gi = 0; gi < n_groups; ++gi) {
    const I8Group &g = plan.i8_groups[gi];
    const int k = gi % sets, ni = g.item1 - g.item0, nt = g.tile1 - g.tile0;
    if (gi >= sets) FRPA_CUDA_TRY(cudaStreamWaitEvent(plan.i8_side, plan.i8_ev_done[k], 0));
    i8_pack_a_kernel<<<ni * PA_GROUPS, PA_THREADS, 0, plan.i8_side>>>(plan.d_i8_items + g.item0, wave, plan.d_i8_a[k],
                                                                      plan.d_i8_sa[k], P.wave_vec);
    FRPA_LAUNCH_CHECK();
    i8_pack_b_kernel<<<nt, PB_THREADS, 0, plan.i8_side>>>(plan.d_i8_tiles + g.tile0, plan.d_ib, P1, plan.d_rowmax,
                                                          plan.n_basis, plan.d_i8_b[k], plan.d_i8_sb[k]);
    FRPA_LAUNCH_CHECK();
    FRPA_CUDA_TRY(cudaEventRecord(plan.i8_ev_packed[k], plan.i8_side));
    FRPA_CUDA_TRY(cudaStreamWaitEvent(stream, plan.i8_ev_packed[k], 0));
    P.items = plan.d_i8_items + g.item0;
    P.n_items = ni;
    P.a_scr = plan.d_i8_a[k];
    P.b_scr = plan.d_i8_b[k];
    P.sa = plan.d_i8_sa[k];
    P.sb = plan.d_i8_sb[k];
    rho1_i8_kernel<<<std::min(n_sm, ni), I8_THREADS, smem, stream>>>(P);
    FRPA_LAUNCH_CHECK();
    if (gi + sets < n_groups) FRPA_CUDA_TRY(cudaEventRecord(plan.i8_ev_done[k], stream));
  }
  return FRPA_OK;
}

}  // namespace frpa
