// FP64 products over the grid on the 5th-generation tensor cores (tcgen05), by
// exact integer slices:
//   out[i][j] = scale * sum_k A[i][k] B[j][k]   (real K, or complex as real K)
//
// A row's values over one K split of 2048 share the power of two 2^e above twice their
// largest magnitude.  x 2^-e is rounded to a 64-bit fixed-point number and cut into
// eight signed base-256 digits d_1 .. d_8, x = 2^e sum_i d_i 2^(1 - 8 i), each a small
// integer that BF16 holds exactly (the error-free slicing of K. Ozaki et al.,
// Numer. Algorithms 59 (2012) 95).  Digit products of equal order i + j are summed in
// one FP32 accumulator: |d| <= 128 (64 for d_1), so 128 products of up to eight pairs
// stay within 2^24 and every sum is exact.  The 36 pairs with i + j <= 9 are formed.
// Every 128 values of K the accumulators are read out and added, weighted by their
// order, to two 64-bit integers per output, again exactly; a split ends with one
// conversion of each to FP64 and their sum, and the splits are added in order.
//
// Accuracy: the pairs left out and the rounding of the digits come to less than
// 9 x 2^-64 2^(e_a + e_b) a term, so a split is off by at most 9 u B, B = 2^(e_a + e_b),
// u = 2^-53 (by about 0.02 u B where the terms' errors are independent).  That is an
// error against the rows' largest values; where these do not meet (packets apart, rows
// of wide range) it could exceed what FP64 sums leave, which is relative to S =
// sum |a||b|.  So S is formed as well, a ninth product of magnitudes cut to BF16, and an
// output whose splits do not add up to 8 S >= B is summed in FP64 instead
// (k_ex_direct): every output is within 72 u S and the roundings of adding the splits,
// where a running FP64 sum over K terms is within K u S.  S of a complex output is that
// of its real and imaginary part together.  Rows with an infinity or a NaN give NaN
// (fbse_gram) or the FP64 sum (exciton kernels).
//
// Why: FP64 arithmetic runs at 2 lanes per clock and SM on this chip (1.25 TFLOP/s),
// 36 BF16 products at 1900 TFLOP/s are forty times that.  Measured: a complex 196 x
// 196 product over 85184 points 115 ms on the SIMT kernel, 2.5 ms here (digits and
// exponents 0.64, their products 1.77 or 0.91 PFLOP/s of padded tiles, 48% of the
// measured BF16 rate, magnitudes 0.12, sums 0.06): a 128 x 64 MMA reads 192 bytes of
// shared memory per clock, more than there are, the read-outs do not overlap the MMAs,
// and a CTA's start and end cost as much as eleven of its 64 stages.  fbse_gram of 128
// real states of 133380 points 57 -> 0.56 ms.  Error against extended precision, 2-norm,
// 216000 complex terms: 4e-16 (adding 211 splits; 6e-16 for rows of wide range, in FP64),
// the SIMT kernel's 4e-16 to 3.6e-15.
//
// Operands are images of whole tiles, written once per product and moved by bulk
// copies: 128 (A) or 64 (B) rows x 32 values x 8 slices and the magnitudes, each slice
// in the unswizzled K-major core-matrix layout (8 rows x 16 bytes contiguous, row groups
// next, 16-byte columns of K last).  CTA: 128 x 64 outputs; eight order sums of 64
// FP32 columns fill the 512 columns of tensor memory, and two stages of 96 KB the
// shared memory; the magnitudes' product is a launch of its own with one sum and eight
// stages of 12 KB, two CTAs per SM.  Warp 0 copies, warp 1 issues the MMAs, warps 2 to 9
// read the sums out.  Every wait is bounded: on a timeout the kernel records an error, waits
// (bounded) for what it issued, frees its tensor memory and returns.
#include <algorithm>
#include <cstdint>

#include "fbse_async.cuh"
#include "fbse_internal.cuh"

namespace fbse {
namespace ex {

using namespace fbse::async;

constexpr int kM = 128, kN = 64, kK = 32;  // CTA tile, values of K per stage
constexpr int kSlices = 8, kOrders = 8;
constexpr int kTileA = kM * kK * 2, kTileB = kN * kK * 2;  // bytes of one slice
constexpr int kBlockA = (kSlices + 1) * kTileA, kBlockB = (kSlices + 1) * kTileB;  // a k block of an image
constexpr int kDrain = 128 / kK;        // stages between read-outs
// stages per split.  Fixed, and chunks of K are whole splits added in order, so a
// result's bits depend on the rows' length alone: not on how many rows there are, nor
// on the room for the images.  64: a CTA's start and end cost six stages, and the 16
// tiles of 196 x 196 complex products of 85184 points fill 8.8 waves of 152 CTAs.
constexpr int kSplit = 64;
constexpr int kReadWarps = 8, kThreads = 32 * (2 + kReadWarps);
constexpr int kCols = kN / 2;           // columns of a reading thread
constexpr int kNonFinite = 1 << 20;     // exponent of a row that holds an infinity or NaN
constexpr int kZeroRow = -(1 << 20);    // and of one that is zero
constexpr int kExpMax = 900;            // |e_a + e_b| beyond this: the bounds could leave FP64's range

// the product of the digits (8 slices, 8 sums) or of the magnitudes (1 and 1)
template <bool MAG> struct Shape {
  static constexpr int slices = MAG ? 1 : kSlices, orders = MAG ? 1 : kOrders;
  static constexpr int stages = MAG ? 8 : 2, drain = MAG ? kSplit : kDrain;
  static constexpr int bytes_a = slices * kTileA, bytes_b = slices * kTileB, bytes = bytes_a + bytes_b;
  static constexpr size_t smem = (size_t)stages * bytes + 128;
};

// shared-memory matrix descriptor, K-major, no swizzle: lbo between the 16-byte
// columns of K, sbo between groups of 8 rows
__device__ __forceinline__ uint64_t desc(uint32_t saddr, uint32_t lbo, uint32_t sbo)
{
  return (uint64_t)((saddr & 0x3FFFF) >> 4) | (uint64_t)(lbo >> 4) << 16 | (uint64_t)(sbo >> 4) << 32 | (uint64_t)1 << 46;
}

// instruction descriptor: D = F32, A = B = BF16, both K-major
constexpr uint32_t kIdesc =
    (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kN >> 3) << 17) | ((uint32_t)(kM >> 4) << 24);

__device__ __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t acc)
{
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(kIdesc), "r"(acc));
}
__device__ __forceinline__ void commit(uint64_t *bar)
{
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

// A images [mp / 128][nkb], B images [np / 64][nkb]; the CTA (x, y, z) forms rows
// 128 x, columns 64 y over the k blocks of split z: part[z][row][col], MAG:
// mag[z][row][col], in units of 2^(ea + eb).
// ea [split][mp], eb [split][n1]: the rows' exponents (n1 = np, or np / 2 when B's
// second half of rows rearranges the first).
template <bool MAG>
__global__ void __launch_bounds__(kThreads, MAG ? 2 : 1)
    k_ex_gemm(const unsigned char *__restrict__ A, const unsigned char *__restrict__ B, long nkb,
              const int *__restrict__ ea, const int *__restrict__ eb, double *__restrict__ part, float *__restrict__ mag,
              long mp, long np, long n1, int *__restrict__ status)
{
  using Sh = Shape<MAG>;
  constexpr int ST = Sh::stages;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char *stage = smem_raw + ((128 - (smem_u32(smem_raw) & 127)) & 127);
  __shared__ __align__(8) uint64_t full_bar[ST], free_bar[ST], sums_bar, read_bar, last_bar;
  __shared__ uint32_t tmem_base;
  __shared__ int fail;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long kb0 = (long)blockIdx.z * kSplit;
  const int nk = (int)(min(nkb, kb0 + kSplit) - kb0);
  const int ndrain = (nk + Sh::drain - 1) / Sh::drain;
  if (threadIdx.x == 0) {
    for (int s = 0; s < ST; s++) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&free_bar[s], 1);
    }
    mbar_init(&sums_bar, 1);
    mbar_init(&last_bar, 1);
    mbar_init(&read_bar, kReadWarps);
    fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                 "n"(Sh::orders * kN));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = tmem_base;
  int issued = 0;  // stages copied (thread 0)
  if (threadIdx.x == 0) {
    const unsigned char *a = A + ((long)blockIdx.x * nkb + kb0) * kBlockA + (MAG ? kSlices * kTileA : 0);
    const unsigned char *b = B + ((long)blockIdx.y * nkb + kb0) * kBlockB + (MAG ? kSlices * kTileB : 0);
    bool ok = true;
    for (int it = 0; it < nk && ok; it++) {
      const int s = it % ST;
      if (it >= ST) ok = mbar_wait(&free_bar[s], (uint32_t)((it / ST - 1) & 1));
      if (!ok) break;
      unsigned char *buf = stage + s * Sh::bytes;
      mbar_expect_tx(&full_bar[s], Sh::bytes);
      bulk_copy(buf, a + (long)it * kBlockA, Sh::bytes_a, &full_bar[s]);
      bulk_copy(buf + Sh::bytes_a, b + (long)it * kBlockB, Sh::bytes_b, &full_bar[s]);
      issued = it + 1;
    }
    if (!ok) atomicExch(&fail, 1);
  } else if (threadIdx.x == 32) {
    bool ok = true;
    for (int it = 0; it < nk && ok; it++) {
      const int s = it % ST;
      if (it % Sh::drain == 0 && it > 0) ok = mbar_wait(&read_bar, (uint32_t)((it / Sh::drain - 1) & 1));
      if (ok) ok = mbar_wait(&full_bar[s], (uint32_t)((it / ST) & 1));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;");
      const uint32_t a0 = smem_u32(stage + s * Sh::bytes), b0 = a0 + Sh::bytes_a;
#pragma unroll 1
      for (int kk = 0; kk < kK / 16; kk++) {
        const uint32_t first = (it % Sh::drain == 0 && kk == 0) ? 0u : 1u;
        const uint64_t da = desc(a0 + kk * 2 * (kM * 16), kM * 16, 128), db = desc(b0 + kk * 2 * (kN * 16), kN * 16, 128);
#pragma unroll
        for (int g = 0; g < Sh::orders; g++)
#pragma unroll
          for (int i = 0; i <= g; i++)  // slices i and g - i, counted from 0
            mma(tmem + g * kN, da + (uint64_t)(i * (kTileA >> 4)), db + (uint64_t)((g - i) * (kTileB >> 4)),
                i == 0 ? first : 1u);
      }
      commit(&free_bar[s]);
      if (it % Sh::drain == Sh::drain - 1 || it == nk - 1) commit(&sums_bar);
    }
    commit(&last_bar);  // arrives once every MMA issued is done, whichever wait ended the loop
    if (!ok) atomicExch(&fail, 1);
  } else if (warp >= 2) {
    // lanes: rows 32 (warp % 4) ..; columns: half of the tile
    const int quad = warp & 3, half = (warp - 2) >> 2;
    const uint32_t at = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(half * kCols);
    const long row = (long)blockIdx.x * kM + quad * 32 + lane, col = (long)blockIdx.y * kN + half * kCols;
    auto dst = [&] { return ((long)blockIdx.z * mp + row) * np + col; };
    long long hi[MAG ? 1 : kCols], lo[MAG ? 1 : kCols];
    if constexpr (!MAG) {
#pragma unroll
      for (int j = 0; j < kCols; j++) hi[j] = lo[j] = 0;
    }
    bool ok = true;
    for (int d = 0; d < ndrain && ok; d++) {
      ok = mbar_wait(&sums_bar, (uint32_t)(d & 1));
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll
      for (int j0 = 0; j0 < kCols; j0 += 4) {
        uint32_t r[Sh::orders][4];
#pragma unroll
        for (int g = 0; g < Sh::orders; g++)
          asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                       : "=r"(r[g][0]), "=r"(r[g][1]), "=r"(r[g][2]), "=r"(r[g][3])
                       : "r"(at + (uint32_t)(g * kN + j0)));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if constexpr (MAG) {
          *reinterpret_cast<uint4 *>(mag + dst() + j0) = make_uint4(r[0][0], r[0][1], r[0][2], r[0][3]);
        } else {
#pragma unroll
          for (int j = 0; j < 4; j++) {
#pragma unroll
            for (int g = 0; g < 4; g++) {
              hi[j0 + j] += (long long)__float2int_rn(__uint_as_float(r[g][j])) * (1 << (8 * (3 - g)));
              lo[j0 + j] += (long long)__float2int_rn(__uint_as_float(r[g + 4][j])) * (1 << (8 * (3 - g)));
            }
          }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;");
      __syncwarp();
      if (lane == 0) mbar_arrive(&read_bar);
    }
    if (!ok) {
      if (lane == 0) atomicExch(&fail, 1);
    } else if constexpr (!MAG) {
      // order g (0 ..) weighs 2^(-14 - 8 g): hi counts 2^-38, lo 2^-70
      const int er = ea[(long)blockIdx.z * mp + row];
      const int *ec = eb + (long)blockIdx.z * n1 + col % n1;
      double *out = part + dst();
#pragma unroll
      for (int j = 0; j < kCols; j++) {
        const int c = ec[j];
        double v = scalbn((double)hi[j], er + c - 38) + scalbn((double)lo[j], er + c - 70);
        if (er == kNonFinite || c == kNonFinite) v = __longlong_as_double(0x7ff8000000000000LL);
        out[j] = v;
      }
    }
  }
  __syncthreads();
  if (fail) {
    // copies and MMAs still in flight finish before the CTA leaves (bounded)
    if (threadIdx.x == 0) {
      atomicExch(status, 1);
      for (int it = issued > ST ? issued - ST : 0; it < issued; it++)
        mbar_wait(&full_bar[it % ST], (uint32_t)((it / ST) & 1));
    }
    if (threadIdx.x == 32) mbar_wait(&last_bar, 0u);
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(Sh::orders * kN));
}

// exponent of each (row, split): 2^e above twice the largest magnitude, or kZeroRow / kNonFinite
__global__ void __launch_bounds__(256) k_ex_exp(const double *__restrict__ src, long ld, int nrows, long k_len, long k0,
                                                long rows_p, int *__restrict__ e)
{
  const long row = blockIdx.x;
  int ex = -1021;
  if (row < nrows) {
    const long b = k0 + (long)blockIdx.y * kSplit * kK, end = min(k_len, b + kSplit * kK);
    unsigned m = 0;  // biased exponents, 1 for denormal values
    for (long k = b + threadIdx.x; k < end; k += blockDim.x) {
      const unsigned long long x = (unsigned long long)__double_as_longlong(src[row * ld + k]) << 1;
      if (x) m = max(m, max(1u, (unsigned)(x >> 53)));
    }
    __shared__ unsigned w[8];
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int i = 1; i < 8; i++) m = max(m, w[i]);
      ex = m == 0x7ffu ? kNonFinite : m == 0 ? kZeroRow : (int)m - 1021;
    }
  }
  if (threadIdx.x == 0) e[(long)blockIdx.y * rows_p + row] = ex;
}

// digits and magnitudes of eight values of one row: how the value of K index k comes from the row
//   0: x[k]   1: odd k negated   2: pairs swapped   3: pairs swapped, odd k negated
template <int ROWS>
__global__ void __launch_bounds__(256)
    k_ex_slice(const double *__restrict__ src, long ld, int nrows, long k_len, long k0, int mode, long rows_p, long nkb,
               const int *__restrict__ e, unsigned char *__restrict__ img)
{
  constexpr int kTile = ROWS * kK * 2;
  const long total = rows_p * nkb * 4;
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < total; t += (long)gridDim.x * blockDim.x) {
    const long row = t % rows_p, kc = t / rows_p, kb = kc / 4;
    if (row >= nrows) continue;  // rows that fill the tile meet outputs that nobody reads
    const int c16 = (int)(kc % 4);
    const long k = k0 + kc * 8;
    const int ea = e[(kb / kSplit) * rows_p + row];
    uint32_t word[kSlices + 1][4];
    unsigned long long prev = 0;
    uint32_t prev_mag = 0;
#pragma unroll
    for (int u = 0; u < 8; u++) {
      const long ks = k + (mode >= 2 ? u ^ 1 : u);
      double x = 0.0;
      if (ks < k_len) x = src[row * ld + ks];
      if ((mode & 1) && (u & 1)) x = -x;
      // 64-bit fixed point of x 2^-ea, then a bias that makes every byte digit + 128
      const unsigned long long bits = (unsigned long long)__double_as_longlong(x);
      const int be = (int)(bits >> 52) & 0x7ff;
      unsigned long long v = (bits & 0xfffffffffffffULL) | (be ? 0x10000000000000ULL : 0ULL);
      const int sh = (be ? be : 1) - 1012 - ea;
      if (sh >= 0) v <<= min(sh, 9);
      else v = -sh > 62 ? 0ULL : (v + (1ULL << (-sh - 1))) >> -sh;
      if (bits >> 63) v = 0ULL - v;
      v += 0x8080808080808080ULL;
      // |x| 2^-ea cut to BF16, at least 2^-60 unless zero: a sum of products of magnitudes
      // is zero only when every product is, and is not above the true one otherwise (2^-60
      // is far below the digits' resolution)
      uint32_t mg = 0;
      if (bits << 1) mg = (uint32_t)max(67 << 7, be ? (be - 896 - ea) * 128 + (int)((bits >> 45) & 0x7f) : 0);
      if (u & 1) {
#pragma unroll
        for (int s = 0; s < kSlices; s++) {
          const float f0 = __uint_as_float(0x4b000000u | (uint32_t)((prev >> (56 - 8 * s)) & 0xff)) - 8388736.0f;
          const float f1 = __uint_as_float(0x4b000000u | (uint32_t)((v >> (56 - 8 * s)) & 0xff)) - 8388736.0f;
          word[s][u >> 1] = __byte_perm(__float_as_uint(f0), __float_as_uint(f1), 0x7632);
        }
        word[kSlices][u >> 1] = prev_mag | mg << 16;
      }
      prev = v;
      prev_mag = mg;
    }
    const int r = (int)(row % ROWS);
    unsigned char *dst = img + (((row / ROWS) * nkb + kb) * (kSlices + 1)) * kTile + (c16 * ROWS + r) * 16;
#pragma unroll
    for (int s = 0; s <= kSlices; s++)
      *reinterpret_cast<uint4 *>(dst + s * kTile) = make_uint4(word[s][0], word[s][1], word[s][2], word[s][3]);
  }
}

// out[i][j] = scale * (sum of the splits' real columns, imaginary columns), the splits
// of all chunks in order: a chunk adds to the sums of those before it, the last one
// scales.  bound[i][j]: 8 S - B of the splits so far; the last chunk lists the outputs
// where it is negative (nan: but for those of rows that are not finite).
__global__ void __launch_bounds__(256)
    k_ex_reduce(const double *__restrict__ part, const float *__restrict__ mag, const int *__restrict__ ea,
                const int *__restrict__ eb, int nsplit, long mp, long np, long n1, int m, int n, bool cplx, bool first,
                bool last, bool nan, double scale, double *__restrict__ bound, double2 *__restrict__ out,
                int *__restrict__ list, int *__restrict__ nlist)
{
  const long total = (long)m * n;
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < total; e += (long)gridDim.x * blockDim.x) {
    const long i = e / n, j = e % n;
    double2 o = first ? make_double2(0, 0) : out[e];
    double d = first ? 0.0 : bound[e];
#pragma unroll 12
    for (int s = 0; s < nsplit; s++) {
      const long at = ((long)s * mp + i) * np + j;
      o.x += part[at];
      float g = mag[at];
      if (cplx) {
        o.y += part[at + n1];
        g += mag[at + n1];
      }
      const int ex = ea[s * mp + i] + eb[s * n1 + j];
      // nothing where every product of the split is zero; beyond kExpMax (rows that are not
      // finite among them) the output is listed
      const double w = __longlong_as_double((long long)(ex + 1023) << 52);
      const double t = abs(ex) > kExpMax ? -INFINITY : fma((double)fmaf(8.0f, g, -1.0f), w, d);
      d = g == 0.0f ? d : t;
    }
    if (!last) {
      out[e] = o;
      bound[e] = d;
      continue;
    }
    out[e] = make_double2(o.x * scale, o.y * scale);
    if (!(d >= 0.0) && !(nan && isnan(o.x))) list[atomicAdd(nlist, 1)] = (int)e;
  }
}

// the listed outputs as FP64 sums, a CTA each: out = scale sum_l f(A_i[l]) B_j[l].  Rows
// that do not meet are rare and this is the slow way: 130 x 130 complex outputs of 47520
// points 6.7 ms where all are listed, 1.2 ms where none is.
template <ExactKind KIND>
__global__ void __launch_bounds__(256)
    k_ex_direct(const double *__restrict__ A, long lda, const double *__restrict__ B, long ldb, int n, long L, double scale,
                const int *__restrict__ list, const int *__restrict__ nlist, double2 *__restrict__ out)
{
  __shared__ double2 w[8];
  const int count = *nlist;
  for (int q = blockIdx.x; q < count; q += gridDim.x) {
    const int e = list[q];
    const double *a = A + (long)(e / n) * lda, *b = B + (long)(e % n) * ldb;
    constexpr int U = 4;  // sums of a thread, every 1024th term each
    double r[U] = {}, t[U] = {};
    for (long l0 = threadIdx.x; l0 < L; l0 += U * 256) {
#pragma unroll
      for (int u = 0; u < U; u++) {
        const long l = l0 + u * 256;
        if (l >= L) break;
        if constexpr (KIND == kExactReal) {
          r[u] = fma(a[l], b[l], r[u]);
        } else {
          const double2 x = reinterpret_cast<const double2 *>(a)[l], y = reinterpret_cast<const double2 *>(b)[l];
          const double s = KIND == kExactConj ? -x.y : x.y;
          r[u] = fma(-s, y.y, fma(x.x, y.x, r[u]));
          t[u] = fma(s, y.x, fma(x.x, y.y, t[u]));
        }
      }
    }
    double re = (r[0] + r[1]) + (r[2] + r[3]), im = (t[0] + t[1]) + (t[2] + t[3]);
    for (int o = 16; o > 0; o >>= 1) {
      re += __shfl_xor_sync(0xffffffffu, re, o);
      im += __shfl_xor_sync(0xffffffffu, im, o);
    }
    if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = make_double2(re, im);
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int v = 1; v < 8; v++) {
        re += w[v].x;
        im += w[v].y;
      }
      out[e] = make_double2(re * scale, im * scale);
    }
    __syncthreads();
  }
}

}  // namespace ex

int exact_nt(fbse_ctx *c, const double *A, long lda, int ma, const double *B, long ldb, int nb, long L, ExactKind kind,
             double scale, double2 *out)
{
  using namespace ex;
  if ((double)ma * nb > 2.0e9) return set_err(c, FBSE_ERR_OOM, "exact product: too many outputs");
  const bool cplx = kind != kExactReal;
  const long K = cplx ? 2 * L : L;
  const long mp = (ma + kM - 1) / kM * kM, n1 = (nb + kN - 1) / kN * kN, np = cplx ? 2 * n1 : n1;
  const long nkb_all = (K + kK - 1) / kK;
  // images of a K chunk within 4 GB (fbse_tuning.tc_image_bytes sets another size), its
  // partial sums within 2 GB, at least one split
  const long row_bytes = (long)(kSlices + 1) * kK * 2;
  const double budget = c->tune.tc_image_bytes > 0 ? c->tune.tc_image_bytes : 4.0e9;
  const long fit = std::min((long)(budget / (double)(row_bytes * (mp + np))) / kSplit, 2000000000L / (12 * mp * np));
  const long nsplit_all = (nkb_all + kSplit - 1) / kSplit, nchunk = (nsplit_all + std::max(1L, fit) - 1) / std::max(1L, fit);
  const long nsplit = (nsplit_all + nchunk - 1) / nchunk, nkb = std::min(nkb_all, nsplit * kSplit);
  const size_t img_a = (size_t)(mp * nkb * row_bytes), img_b = (size_t)(np * nkb * row_bytes);
  const size_t part_b = (size_t)nsplit * mp * np * sizeof(double), bound_b = ((size_t)ma * nb + 1) / 2 * sizeof(double2);
  const size_t mag_b = part_b / 2, exp_b = (size_t)nsplit * (mp + n1) * sizeof(int), list_b = (size_t)ma * nb * sizeof(int);
  void *scratch = nullptr;
  int rc = cached(c, kSlotTc, img_a + img_b + part_b + bound_b + mag_b + exp_b + list_b + 256, &scratch);
  if (rc) return rc;
  unsigned char *ia = static_cast<unsigned char *>(scratch), *ib = ia + img_a;
  double *part = reinterpret_cast<double *>(ib + img_b);
  double *bound = reinterpret_cast<double *>(reinterpret_cast<unsigned char *>(part) + part_b);
  float *mag = reinterpret_cast<float *>(reinterpret_cast<unsigned char *>(bound) + bound_b);
  int *ea = reinterpret_cast<int *>(reinterpret_cast<unsigned char *>(mag) + mag_b), *eb = ea + nsplit * mp;
  int *list = eb + nsplit * n1, *status = list + (size_t)ma * nb, *nlist = status + 1;
  FBSE_CUDA(c, cudaMemsetAsync(status, 0, 2 * sizeof(int), c->stream));
  FBSE_CUDA(c, cudaFuncSetAttribute(k_ex_gemm<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Shape<false>::smem));
  FBSE_CUDA(c, cudaFuncSetAttribute(k_ex_gemm<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Shape<true>::smem));
  const int mode_b[2] = {kind == kExactPlain ? 1 : 0, kind == kExactPlain ? 2 : 3};
  auto grid = [](long n) { return (unsigned)std::min<long>((n + 255) / 256, 152 * 32); };
  for (long ch = 0; ch < nchunk; ch++) {
    const long kb0 = ch * nsplit * kSplit, kb = std::min(nkb, nkb_all - kb0), k0 = kb0 * kK;
    const long ns = (kb + kSplit - 1) / kSplit;
    k_ex_exp<<<dim3((unsigned)mp, (unsigned)ns), 256, 0, c->stream>>>(A, lda, ma, K, k0, mp, ea);
    FBSE_CHECK_LAUNCH(c);
    k_ex_slice<kM><<<grid(mp * kb * 4), 256, 0, c->stream>>>(A, lda, ma, K, k0, 0, mp, kb, ea, ia);
    FBSE_CHECK_LAUNCH(c);
    k_ex_exp<<<dim3((unsigned)n1, (unsigned)ns), 256, 0, c->stream>>>(B, ldb, nb, K, k0, n1, eb);
    FBSE_CHECK_LAUNCH(c);
    for (int h = 0; h < (cplx ? 2 : 1); h++) {
      k_ex_slice<kN><<<grid(n1 * kb * 4), 256, 0, c->stream>>>(B, ldb, nb, K, k0, mode_b[h], n1, kb, eb,
                                                               ib + (size_t)h * n1 * kb * row_bytes);
      FBSE_CHECK_LAUNCH(c);
    }
    const dim3 g((unsigned)(mp / kM), (unsigned)(np / kN), (unsigned)ns);
    k_ex_gemm<false><<<g, kThreads, Shape<false>::smem, c->stream>>>(ia, ib, kb, ea, eb, part, nullptr, mp, np, n1, status);
    FBSE_CHECK_LAUNCH(c);
    k_ex_gemm<true><<<g, kThreads, Shape<true>::smem, c->stream>>>(ia, ib, kb, ea, eb, nullptr, mag, mp, np, n1, status);
    FBSE_CHECK_LAUNCH(c);
    k_ex_reduce<<<grid((long)ma * nb), 256, 0, c->stream>>>(part, mag, ea, eb, (int)ns, mp, np, n1, ma, nb, cplx, ch == 0,
                                                             ch == nchunk - 1, kind != kExactPlain, scale, bound, out, list,
                                                             nlist);
    FBSE_CHECK_LAUNCH(c);
  }
  const unsigned gd = (unsigned)std::min<long>((long)ma * nb, 152 * 8);
  if (kind == kExactReal) k_ex_direct<kExactReal><<<gd, 256, 0, c->stream>>>(A, lda, B, ldb, nb, L, scale, list, nlist, out);
  else if (kind == kExactConj) k_ex_direct<kExactConj><<<gd, 256, 0, c->stream>>>(A, lda, B, ldb, nb, L, scale, list, nlist, out);
  else k_ex_direct<kExactPlain><<<gd, 256, 0, c->stream>>>(A, lda, B, ldb, nb, L, scale, list, nlist, out);
  FBSE_CHECK_LAUNCH(c);
  int hs = 0;
  if (d2h(c->stream, &hs, status, sizeof(int)) != cudaSuccess) return set_err(c, FBSE_ERR_CUDA, "exact product");
  if (hs) {
    c->tc_poisoned = 1;
    return set_err(c, FBSE_ERR_NOCONV, "exact product: a tensor-core wait timed out");
  }
  return FBSE_OK;
}

}  // namespace fbse
