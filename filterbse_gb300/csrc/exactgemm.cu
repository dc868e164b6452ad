// FP64 products over the grid on the 5th-generation tensor cores (tcgen05), by
// exact integer slices:
//   out[i][j] = scale * sum_k A[i][k] B[j][k]   (real K, or complex as real K)
//
// A row's values over one K split (512 to 4096 of them) share the power of two 2^e above
// twice their largest magnitude.  x 2^-e is rounded to a 64-bit fixed-point number and cut into
// eight signed base-256 digits d_1 .. d_8, x = 2^e sum_i d_i 2^(1 - 8 i), each a small
// integer that BF16 holds exactly (the error-free slicing of K. Ozaki et al.,
// Numer. Algorithms 59 (2012) 95).  Digit products of equal order i + j are summed in
// one FP32 accumulator: |d| <= 128 (64 for d_1), so 128 products of up to eight pairs
// stay within 2^24 and every sum is exact.  The 36 pairs with i + j <= 9 are formed.
// Every 128 values of K the accumulators are read out and added, weighted by their
// order, to two 64-bit integers per output, again exactly; a split ends with one
// conversion of each to FP64 and their sum; the splits are added with compensation.
//
// Accuracy: the pairs left out and the rounding of the digits come to less than
// 9 x 2^-64 2^(e_a + e_b) a term, so a split is off by at most 18 u B, B = 2^(e_a + e_b),
// u = 2^-53 (by about 0.02 u B where the terms' errors are independent).  That is an
// error against the rows' largest values; where these do not meet (packets apart, rows
// of wide range) it could exceed what FP64 sums leave, which is relative to S =
// sum |a||b|.  So S is formed as well, a ninth product of magnitudes cut to BF16, and an
// output whose splits do not add up to 8 S >= B is summed in FP64 instead
// (k_ex_direct): every output is within 144 u S and a rounding or two,
// where a running FP64 sum over K terms is within K u S.  S of a complex output is that
// of its real and imaginary part together.  Rows with an infinity or a NaN give NaN
// (fbse_gram) or the FP64 sum (exciton kernels).
//
// Why: FP64 arithmetic runs at 2 lanes per clock and SM on this chip (1.25 TFLOP/s),
// 36 BF16 products at 1900 TFLOP/s are forty times that.  Measured: a complex 196 x
// 196 product over 85184 points 115 ms on the SIMT kernel, 2.3 ms here (digits and
// exponents 0.53, their products 1.64 or 0.98 PFLOP/s of padded tiles, 51% of the
// measured BF16 rate, magnitudes 0.10, sums 0.07): a 128 x 64 MMA reads 192 bytes of
// shared memory per clock, more than there are, and the read-outs do not overlap the
// MMAs.  fbse_gram of 128 real states of 133380 points 57 -> 0.55 ms.  Error against
// extended precision, 2-norm, 216000 complex terms: 4e-17 to 8e-17 (6e-16 for rows of wide
// range, in FP64), the SIMT kernel's 4e-16 to 3.6e-15.
//
// Operands are images of whole tiles, written once per product and moved by bulk
// copies: 128 (A) or 64 (B) rows x 32 values x 8 slices and the magnitudes, each slice
// in the unswizzled K-major core-matrix layout (8 rows x 16 bytes contiguous, row groups
// next, 16-byte columns of K last).  CTA: 128 x 64 outputs; eight order sums of 64
// FP32 columns fill the 512 columns of tensor memory, and two stages of 96 KB the
// shared memory; the magnitudes' product is a launch of its own with one sum and eight
// stages of 12 KB, two CTAs per SM.  Warp 0 copies, warp 1 issues the MMAs, warps 2 to 9
// read the sums out.  Every wait is bounded: on a timeout the kernel records an error,
// waits (bounded) for what it issued, frees its tensor memory and returns.
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
// Stages per split, of some 2048 values: from the rows' length alone, and chunks of K are
// whole splits added in order, so a result's bits depend neither on how many rows there
// are nor on the room for the images.  A multiple of 76 splits of up to 128 stages: with
// 1, 2, 4, .. tiles the 152 CTAs get the same number of items; 16 at least.  fbse_gram of
// 81 x 4 and 196 x 196 complex elements of 85184 points (75 splits of 71 stages) 528 and
// 2427 us, with 64 stages always 555 and 2600; of 1 x 1 of 133380 (76 of 110) 611, with up
// to 96 stages 700; of 2744 real points (16 stages) 167, with 32 at least 216; of 196 x 196
// complex elements of 13824 points 665, with 8 at least 717.
inline long split_stages(long nkb)
{
  const long k = (nkb + 76 * 128 - 1) / (76 * 128);
  return std::max(16L, (nkb + 76 * k - 1) / (76 * k));
}
constexpr int kReadWarps = 8, kThreads = 32 * (2 + kReadWarps);
constexpr int kCols = kN / 2;           // columns of a reading thread
constexpr int kNonFinite = 1 << 20;     // exponent of a row that holds an infinity or NaN
constexpr int kZeroRow = -(1 << 20);    // and of one that is zero
constexpr int kExpMax = 900;            // |e_a + e_b| beyond this: the bounds could leave FP64's range

// the product of the digits (8 slices, 8 sums) or of the magnitudes (1 and 1)
template <bool MAG> struct Shape {
  static constexpr int slices = MAG ? 1 : kSlices, orders = MAG ? 1 : kOrders;
  static constexpr int stages = MAG ? 8 : 2, drain = MAG ? 1 << 20 : kDrain;
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

// A images [mp / 128][nkb], B images [np / 64][nkb]; a CTA walks the items (tile x, y of
// outputs, split z), tiles fastest, and a tile's sums are part[z][row][col], MAG:
// mag[z][row][col], in units of 2^(ea + eb).  The copies run ahead into the next item, and
// its MMAs run while this item's sums are converted and stored: separate CTAs for the
// items paid for a start and an end of 28 us each.
// ea [split][mp], eb [split][n1]: the rows' exponents (n1 = np, or np / 2 when B's
// second half of rows rearranges the first).
template <bool MAG>
__global__ void __launch_bounds__(kThreads, MAG ? 2 : 1)
    k_ex_gemm(const unsigned char *__restrict__ A, const unsigned char *__restrict__ B, long nkb, long kb_split,
              int items, const int *__restrict__ ea, const int *__restrict__ eb, double *__restrict__ part, float *__restrict__ mag,
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
  const int gx = (int)(mp / kM), tiles = gx * (int)(np / kN);
  // item q: rows 128 x, columns 64 y over the nk k blocks from kb0 on of split z
  struct Item {
    int x, y, z, nk;
    long kb0;
  };
  auto item = [&](int q) {
    Item t;
    t.z = q / tiles;
    t.y = (q - t.z * tiles) / gx;
    t.x = q - t.z * tiles - t.y * gx;
    t.kb0 = t.z * kb_split;
    t.nk = (int)(min(nkb, t.kb0 + kb_split) - t.kb0);
    return t;
  };
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
    bool ok = true;
    for (int q = blockIdx.x; q < items && ok; q += gridDim.x) {
      const Item t = item(q);
      const unsigned char *a = A + (t.x * nkb + t.kb0) * kBlockA + (MAG ? kSlices * kTileA : 0);
      const unsigned char *b = B + (t.y * nkb + t.kb0) * kBlockB + (MAG ? kSlices * kTileB : 0);
      for (int it = 0; it < t.nk; it++, issued++) {
        const int s = issued % ST;
        if (issued >= ST) ok = mbar_wait(&free_bar[s], (uint32_t)((issued / ST - 1) & 1));
        if (!ok) break;
        unsigned char *buf = stage + s * Sh::bytes;
        mbar_expect_tx(&full_bar[s], Sh::bytes);
        bulk_copy(buf, a + (long)it * kBlockA, Sh::bytes_a, &full_bar[s]);
        bulk_copy(buf + Sh::bytes_a, b + (long)it * kBlockB, Sh::bytes_b, &full_bar[s]);
      }
    }
    if (!ok) atomicExch(&fail, 1);
  } else if (threadIdx.x == 32) {
    bool ok = true;
    int used = 0, drains = 0;  // stages, read-outs handed over
    for (int q = blockIdx.x; q < items && ok; q += gridDim.x) {
      const int nk = item(q).nk;
      for (int it = 0; it < nk; it++, used++) {
        const int s = used % ST;
        if (it % Sh::drain == 0 && drains > 0) ok = mbar_wait(&read_bar, (uint32_t)((drains - 1) & 1));
        if (ok) ok = mbar_wait(&full_bar[s], (uint32_t)((used / ST) & 1));
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
        if (it % Sh::drain == Sh::drain - 1 || it == nk - 1) {
          commit(&sums_bar);
          drains++;
        }
      }
    }
    commit(&last_bar);  // arrives once every MMA issued is done, whichever wait ended the loop
    if (!ok) atomicExch(&fail, 1);
  } else if (warp >= 2) {
    // lanes: rows 32 (warp % 4) ..; columns: half of the tile
    const int quad = warp & 3, half = (warp - 2) >> 2;
    const uint32_t at = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(half * kCols);
    bool ok = true;
    int drains = 0;
    for (int q = blockIdx.x; q < items && ok; q += gridDim.x) {
      long long hi[MAG ? 1 : kCols], lo[MAG ? 1 : kCols];
      if constexpr (!MAG) {
#pragma unroll
        for (int j = 0; j < kCols; j++) hi[j] = lo[j] = 0;
      }
      auto dst = [&] {
        const Item t = item(q);
        return (t.z * mp + (long)t.x * kM + quad * 32 + lane) * np + (long)t.y * kN + half * kCols;
      };
      const int ndrain = (item(q).nk + Sh::drain - 1) / Sh::drain;
      for (int d = 0; d < ndrain; d++, drains++) {
        ok = mbar_wait(&sums_bar, (uint32_t)(drains & 1));
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
      if (!ok) break;
      if constexpr (!MAG) {
        // order g (0 ..) weighs 2^(-14 - 8 g): hi counts 2^-38, lo 2^-70
        const Item t = item(q);
        const int er = ea[t.z * mp + (long)t.x * kM + quad * 32 + lane];
        const int *ec = eb + t.z * n1 + ((long)t.y * kN + half * kCols) % n1;
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
    if (!ok && lane == 0) atomicExch(&fail, 1);
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
                                                long k_split, long rows_p, int *__restrict__ e)
{
  const long row = blockIdx.x;
  int ex = -1021;
  if (row < nrows) {
    const long b = k0 + blockIdx.y * k_split, end = min(k_len, b + k_split);
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
// img2: a second image of the same rows, in mode2
template <int ROWS>
__global__ void __launch_bounds__(256)
    k_ex_slice(const double *__restrict__ src, long ld, int nrows, long k_len, long k0, long kb_split, int mode, int mode2,
               long rows_p, long nkb, const int *__restrict__ e, unsigned char *__restrict__ img,
               unsigned char *__restrict__ img2)
{
  constexpr int kTile = ROWS * kK * 2;
  const long total = rows_p * nkb * 4;
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < total; t += (long)gridDim.x * blockDim.x) {
    const long row = t % rows_p, kc = t / rows_p, kb = kc / 4;
    if (row >= nrows) continue;  // rows that fill the tile meet outputs that nobody reads
    const int c16 = (int)(kc % 4);
    const long k = k0 + kc * 8;
    const int ea = e[(kb / kb_split) * rows_p + row];
    unsigned long long x[8];
#pragma unroll
    for (int u = 0; u < 8; u++)
      x[u] = k + u < k_len ? (unsigned long long)__double_as_longlong(src[row * ld + k + u]) : 0ULL;
    auto write = [&](int md, unsigned char *image) {
      uint32_t word[kSlices + 1][4];
      unsigned long long prev = 0;
      uint32_t prev_mag = 0;
#pragma unroll
      for (int u = 0; u < 8; u++) {
        const unsigned long long bits = md >= 2 ? x[u ^ 1] : x[u];
        const bool neg = (bits >> 63) != ((md & 1) & (u & 1));
        // 64-bit fixed point of x 2^-ea, then a bias that makes every byte digit + 128
        const int be = (int)(bits >> 52) & 0x7ff;
        unsigned long long v = (bits & 0xfffffffffffffULL) | (be ? 0x10000000000000ULL : 0ULL);
        const int sh = (be ? be : 1) - 1012 - ea;
        if (sh >= 0) v <<= min(sh, 9);
        else v = -sh > 62 ? 0ULL : (v + (1ULL << (-sh - 1))) >> -sh;
        if (neg) v = 0ULL - v;
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
      unsigned char *dst = image + (((row / ROWS) * nkb + kb) * (kSlices + 1)) * kTile + (c16 * ROWS + r) * 16;
#pragma unroll
      for (int s = 0; s <= kSlices; s++)
        *reinterpret_cast<uint4 *>(dst + s * kTile) = make_uint4(word[s][0], word[s][1], word[s][2], word[s][3]);
    };
    write(mode, img);
    if (img2) write(mode2, img2);
  }
}

// out[i][j] = scale * (sum of the splits' real columns, imaginary columns), the splits
// of all chunks in order: a chunk adds to the sums of those before it, the last one
// scales.  Compensated (W. Kahan, Comm. ACM 8 (1965) 40), so that some 100 additions leave
// one rounding: rest[i][j] carries what o lacks.  bound[i][j]: 8 S - B of the splits so far; the last chunk lists the outputs
// where it is negative (nan: but for those of rows that are not finite).
__global__ void __launch_bounds__(256)
    k_ex_reduce(const double *__restrict__ part, const float *__restrict__ mag, const int *__restrict__ ea,
                const int *__restrict__ eb, int nsplit, long mp, long np, long n1, int m, int n, bool cplx, bool first,
                bool last, bool nan, double scale, double *__restrict__ bound, double2 *__restrict__ rest,
                double2 *__restrict__ out, int *__restrict__ list, int *__restrict__ nlist)
{
  const long total = (long)m * n;
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < total; e += (long)gridDim.x * blockDim.x) {
    const long i = e / n, j = e % n;
    double2 o = first ? make_double2(0, 0) : out[e], r = first ? make_double2(0, 0) : rest[e];
    auto add = [](double &sum, double &low, double p) {
      const double y = p - low, t = sum + y;
      low = (t - sum) - y;
      sum = t;
    };
    double d = first ? 0.0 : bound[e];
#pragma unroll 12
    for (int s = 0; s < nsplit; s++) {
      const long at = ((long)s * mp + i) * np + j;
      add(o.x, r.x, part[at]);
      float g = mag[at];
      if (cplx) {
        add(o.y, r.y, part[at + n1]);
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
      rest[e] = r;
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
             double scale, double2 *out, double *out_host)
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
  const long ks = split_stages(nkb_all);
  const long fit = std::min((long)(budget / (double)(row_bytes * (mp + np))) / ks, 2000000000L / (12 * mp * np));
  const long nsplit_all = (nkb_all + ks - 1) / ks, nchunk = (nsplit_all + std::max(1L, fit) - 1) / std::max(1L, fit);
  const long nsplit = (nsplit_all + nchunk - 1) / nchunk, nkb = std::min(nkb_all, nsplit * ks);
  const size_t img_a = (size_t)(mp * nkb * row_bytes), img_b = (size_t)(np * nkb * row_bytes);
  const size_t part_b = (size_t)nsplit * mp * np * sizeof(double), bound_b = ((size_t)ma * nb + 1) / 2 * sizeof(double2);
  const size_t mag_b = part_b / 2, exp_b = (size_t)nsplit * (mp + n1) * sizeof(int), list_b = (size_t)ma * nb * sizeof(int);
  const size_t out_b = out ? 0 : (size_t)ma * nb * sizeof(double2);
  const size_t rest_b = nchunk > 1 ? (size_t)ma * nb * sizeof(double2) : 0;
  void *scratch = nullptr;
  int rc = cached(c, kSlotTc, img_a + img_b + part_b + out_b + rest_b + bound_b + mag_b + exp_b + list_b + 256, &scratch);
  if (rc) return rc;
  unsigned char *ia = static_cast<unsigned char *>(scratch), *ib = ia + img_a;
  double *part = reinterpret_cast<double *>(ib + img_b);
  double2 *rest = reinterpret_cast<double2 *>(reinterpret_cast<unsigned char *>(part) + part_b + out_b);
  double *bound = reinterpret_cast<double *>(reinterpret_cast<unsigned char *>(rest) + rest_b);
  if (!out) out = reinterpret_cast<double2 *>(reinterpret_cast<unsigned char *>(part) + part_b);
  float *mag = reinterpret_cast<float *>(reinterpret_cast<unsigned char *>(bound) + bound_b);
  int *ea = reinterpret_cast<int *>(reinterpret_cast<unsigned char *>(mag) + mag_b), *eb = ea + nsplit * mp;
  int *list = eb + nsplit * n1, *status = list + (size_t)ma * nb, *nlist = status + 1;
  FBSE_CUDA(c, cudaMemsetAsync(status, 0, 2 * sizeof(int), c->stream));
  FBSE_CUDA(c, cudaFuncSetAttribute(k_ex_gemm<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Shape<false>::smem));
  FBSE_CUDA(c, cudaFuncSetAttribute(k_ex_gemm<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Shape<true>::smem));
  auto grid = [](long n) { return (unsigned)std::min<long>((n + 255) / 256, 152 * 32); };
  for (long ch = 0; ch < nchunk; ch++) {
    const long kb0 = ch * nsplit * ks, kb = std::min(nkb, nkb_all - kb0), k0 = kb0 * kK;
    const long ns = (kb + ks - 1) / ks;
    k_ex_exp<<<dim3((unsigned)mp, (unsigned)ns), 256, 0, c->stream>>>(A, lda, ma, K, k0, ks * kK, mp, ea);
    FBSE_CHECK_LAUNCH(c);
    k_ex_slice<kM><<<grid(mp * kb * 4), 256, 0, c->stream>>>(A, lda, ma, K, k0, ks, 0, 0, mp, kb, ea, ia, nullptr);
    FBSE_CHECK_LAUNCH(c);
    k_ex_exp<<<dim3((unsigned)n1, (unsigned)ns), 256, 0, c->stream>>>(B, ldb, nb, K, k0, ks * kK, n1, eb);
    FBSE_CHECK_LAUNCH(c);
    k_ex_slice<kN><<<grid(n1 * kb * 4), 256, 0, c->stream>>>(B, ldb, nb, K, k0, ks, kind == kExactPlain ? 1 : 0,
                                                             kind == kExactPlain ? 2 : 3, n1, kb, eb, ib,
                                                             cplx ? ib + (size_t)n1 * kb * row_bytes : nullptr);
    FBSE_CHECK_LAUNCH(c);
    const int items = (int)(mp / kM * (np / kN) * ns);
    k_ex_gemm<false><<<std::min(items, 152), kThreads, Shape<false>::smem, c->stream>>>(ia, ib, kb, ks, items, ea, eb, part,
                                                                                        nullptr, mp, np, n1, status);
    FBSE_CHECK_LAUNCH(c);
    k_ex_gemm<true><<<std::min(items, 304), kThreads, Shape<true>::smem, c->stream>>>(ia, ib, kb, ks, items, ea, eb, nullptr,
                                                                                      mag, mp, np, n1, status);
    FBSE_CHECK_LAUNCH(c);
    k_ex_reduce<<<grid((long)ma * nb), 256, 0, c->stream>>>(part, mag, ea, eb, (int)ns, mp, np, n1, ma, nb, cplx, ch == 0,
                                                             ch == nchunk - 1, kind != kExactPlain, scale, bound, rest, out,
                                                             list, nlist);
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
  if (out_host && d2h(c->stream, out_host, out, (size_t)ma * nb * sizeof(double2)) != cudaSuccess)
    return set_err(c, FBSE_ERR_CUDA, "exact product: download");
  return FBSE_OK;
}

}  // namespace fbse
