// FP64 products over the grid on the 5th-generation tensor cores (tcgen05), by
// exact integer slices:
//   out[i][j] = scale * sum_k A[i][k] B[j][k]   (real K, or complex as real K)
//
// A row's values over one K split share the power of two 2^e above twice their
// largest magnitude.  x 2^-e is rounded to a 64-bit fixed-point number and cut into
// eight signed base-256 digits d_1 .. d_8, x = 2^e sum_i d_i 2^(1 - 8 i), each a small
// integer that BF16 holds exactly (the error-free slicing of K. Ozaki et al.,
// Numer. Algorithms 59 (2012) 95).  Digit products of equal order i + j are summed in
// one FP32 accumulator: |d| <= 128 (64 for d_1), so 128 products of up to eight pairs
// stay below 2^24 and every sum is exact.  The 36 pairs with i + j <= 9 are formed;
// those left out are below 2^-61 of the rows' largest product.  Every 128 values of
// K the accumulators are read out and added, weighted by their order, to two 64-bit
// integers per output, again exactly; a split ends with one conversion to FP64, so
// its sum carries one rounding where a running FP64 sum carries one per term.
//
// Why: FP64 arithmetic runs at 2 lanes per clock and SM on this chip (1.25 TFLOP/s),
// 36 BF16 products at 1900 TFLOP/s are forty times that.  Measured: a complex 196 x
// 196 product over 85184 points 115 -> 1.5 ms on the SIMT kernel and here (plus 0.6 ms
// of slicing; the MMAs run at 1.07 PFLOP/s, 56% of the measured BF16 rate: A 128 x 64
// MMA reads 192 bytes of shared memory per clock, more than there are, and the
// read-outs do not overlap the MMAs), a real 128 x 128 one over 133380 points 10 ->
// 0.2 ms.  Its error against extended precision, 2-norm, 216000 complex terms:
// 2.5e-16 to 3.4e-16, the SIMT kernel's 3.9e-16 to 3.6e-15.
//
// Operands are images of whole tiles, written once per product and moved by bulk
// copies: 128 (A) or 64 (B) rows x 32 values x 8 slices, each slice in the
// unswizzled K-major core-matrix layout (8 rows x 16 bytes contiguous, row groups
// next, 16-byte columns of K last).  CTA: 128 x 64 outputs; eight order sums of 64
// FP32 columns fill the 512 columns of tensor memory, and two stages of 96 KB the
// shared memory.  Warp 0 copies, warp 1 issues the MMAs, warps 2 to 9 read the sums
// out.  Every wait is bounded: on a timeout the kernel records an error, waits
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
constexpr int kStageA = kSlices * kTileA, kStageB = kSlices * kTileB, kStage = kStageA + kStageB;
constexpr int kDrain = 128 / kK;        // stages between read-outs
// stages per split.  Fixed, and chunks of K are whole splits added in order, so a
// result's bits depend on the rows' length alone: not on how many rows there are, nor
// on the room for the images.  64: a CTA's start and end cost six stages, and the 16
// tiles of 196 x 196 complex products of 85184 points fill 8.8 waves of 152 CTAs.
constexpr int kSplit = 64;
constexpr int kReadWarps = 8, kThreads = 32 * (2 + kReadWarps);
constexpr int kCols = kN / 2;           // columns of a reading thread
constexpr int kNonFinite = 1 << 20;     // exponent of a row that holds an infinity or NaN
constexpr size_t kSmem = 2 * (size_t)kStage + 128;

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
__device__ __forceinline__ void arrive(uint64_t *bar)
{
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// A images [mp / 128][nkb], B images [np / 64][nkb]; the CTA (x, y, z) forms rows
// 128 x, columns 64 y over the k blocks of split z: part[z][row][col].
// ea [split][mp], eb [split][n1]: the rows' exponents (n1 = np, or np / 2 when B's
// second half of rows rearranges the first).
__global__ void __launch_bounds__(kThreads, 1)
    k_ex_gemm(const unsigned char *__restrict__ A, const unsigned char *__restrict__ B, long nkb,
              const int *__restrict__ ea, const int *__restrict__ eb, double *__restrict__ part, long mp, long np,
              long n1, int *__restrict__ status)
{
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char *stage = smem_raw + ((128 - (smem_u32(smem_raw) & 127)) & 127);
  __shared__ __align__(8) uint64_t full_bar[2], free_bar[2], sums_bar, read_bar, last_bar;
  __shared__ uint32_t tmem_base;
  __shared__ int fail;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long kb0 = (long)blockIdx.z * kSplit;
  const int nk = (int)(min(nkb, kb0 + kSplit) - kb0);
  const int ndrain = (nk + kDrain - 1) / kDrain;
  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; s++) {
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
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&tmem_base)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = tmem_base;
  int issued = 0;  // stages copied (thread 0)
  if (threadIdx.x == 0) {
    const unsigned char *a = A + ((long)blockIdx.x * nkb + kb0) * kStageA;
    const unsigned char *b = B + ((long)blockIdx.y * nkb + kb0) * kStageB;
    bool ok = true;
    for (int it = 0; it < nk && ok; it++) {
      const int s = it & 1;
      if (it >= 2) ok = mbar_wait(&free_bar[s], (uint32_t)(((it >> 1) - 1) & 1));
      if (!ok) break;
      unsigned char *buf = stage + s * kStage;
      mbar_expect_tx(&full_bar[s], kStage);
      bulk_copy(buf, a + (long)it * kStageA, kStageA, &full_bar[s]);
      bulk_copy(buf + kStageA, b + (long)it * kStageB, kStageB, &full_bar[s]);
      issued = it + 1;
    }
    if (!ok) atomicExch(&fail, 1);
  } else if (threadIdx.x == 32) {
    bool ok = true;
    for (int it = 0; it < nk && ok; it++) {
      const int s = it & 1;
      if (it % kDrain == 0 && it > 0) ok = mbar_wait(&read_bar, (uint32_t)((it / kDrain - 1) & 1));
      if (ok) ok = mbar_wait(&full_bar[s], (uint32_t)((it >> 1) & 1));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;");
      const uint32_t a0 = smem_u32(stage + s * kStage), b0 = a0 + kStageA;
#pragma unroll 1
      for (int kk = 0; kk < kK / 16; kk++) {
        const uint32_t first = (it % kDrain == 0 && kk == 0) ? 0u : 1u;
        const uint64_t da = desc(a0 + kk * 2 * (kM * 16), kM * 16, 128), db = desc(b0 + kk * 2 * (kN * 16), kN * 16, 128);
#pragma unroll
        for (int g = 0; g < kOrders; g++)
#pragma unroll
          for (int i = 0; i <= g; i++)  // slices i and g - i, counted from 0
            mma(tmem + g * kN, da + (uint64_t)(i * (kTileA >> 4)), db + (uint64_t)((g - i) * (kTileB >> 4)),
                i == 0 ? first : 1u);
      }
      commit(&free_bar[s]);
      if (it % kDrain == kDrain - 1 || it == nk - 1) commit(&sums_bar);
    }
    commit(&last_bar);  // arrives once every MMA issued is done, whichever wait ended the loop
    if (!ok) atomicExch(&fail, 1);
  } else if (warp >= 2) {
    // lanes: rows 32 (warp % 4) ..; columns: half of the tile
    const int quad = warp & 3, half = (warp - 2) >> 2;
    long long hi[kCols], lo[kCols];
#pragma unroll
    for (int j = 0; j < kCols; j++) hi[j] = lo[j] = 0;
    const uint32_t at = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(half * kCols);
    bool ok = true;
    for (int d = 0; d < ndrain && ok; d++) {
      ok = mbar_wait(&sums_bar, (uint32_t)(d & 1));
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll
      for (int j0 = 0; j0 < kCols; j0 += 4) {
        uint32_t r[kOrders][4];
#pragma unroll
        for (int g = 0; g < kOrders; g++)
          asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                       : "=r"(r[g][0]), "=r"(r[g][1]), "=r"(r[g][2]), "=r"(r[g][3])
                       : "r"(at + (uint32_t)(g * kN + j0)));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int j = 0; j < 4; j++) {
#pragma unroll
          for (int g = 0; g < 4; g++) {
            hi[j0 + j] += (long long)__float2int_rn(__uint_as_float(r[g][j])) * (1 << (8 * (3 - g)));
            lo[j0 + j] += (long long)__float2int_rn(__uint_as_float(r[g + 4][j])) * (1 << (8 * (3 - g)));
          }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;");
      __syncwarp();
      if (lane == 0) arrive(&read_bar);
    }
    if (!ok) {
      if (lane == 0) atomicExch(&fail, 1);
    } else {
      // order g (0 ..) weighs 2^(-14 - 8 g): hi counts 2^-38, lo 2^-70
      const long row = (long)blockIdx.x * kM + quad * 32 + lane, col = (long)blockIdx.y * kN + half * kCols;
      const int er = ea[(long)blockIdx.z * mp + row];
      const int *ec = eb + (long)blockIdx.z * n1 + col % n1;
      double *dst = part + ((long)blockIdx.z * mp + row) * np + col;
#pragma unroll
      for (int j = 0; j < kCols; j++) {
        const int c = ec[j];
        double v = scalbn((double)hi[j], er + c - 38) + scalbn((double)lo[j], er + c - 70);
        if (er == kNonFinite || c == kNonFinite) v = __longlong_as_double(0x7ff8000000000000LL);
        dst[j] = v;
      }
    }
  }
  __syncthreads();
  if (fail) {
    // copies and MMAs still in flight finish before the CTA leaves (bounded)
    if (threadIdx.x == 0) {
      atomicExch(status, 1);
      for (int it = issued > 2 ? issued - 2 : 0; it < issued; it++) mbar_wait(&full_bar[it & 1], (uint32_t)((it >> 1) & 1));
    }
    if (threadIdx.x == 32) mbar_wait(&last_bar, 0u);
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
}

// exponent of each (row, split): 2^e above twice the largest magnitude
__global__ void __launch_bounds__(256) k_ex_exp(const double *__restrict__ src, long ld, int nrows, long k_len, long k0,
                                                long rows_p, int *__restrict__ e)
{
  const long row = blockIdx.x;
  int ex = -1021;
  if (row < nrows) {
    const long b = k0 + (long)blockIdx.y * kSplit * kK, end = min(k_len, b + kSplit * kK);
    unsigned m = 0;  // biased exponents
    for (long k = b + threadIdx.x; k < end; k += blockDim.x)
      m = max(m, ((unsigned)__double2hiint(src[row * ld + k]) >> 20) & 0x7ffu);
    __shared__ unsigned w[8];
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int i = 1; i < 8; i++) m = max(m, w[i]);
      ex = m == 0x7ffu ? kNonFinite : (int)max(m, 1u) - 1021;
    }
  }
  if (threadIdx.x == 0) e[(long)blockIdx.y * rows_p + row] = ex;
}

// digits of eight values of one row: how the value of K index k comes from the row
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
    const int c16 = (int)(kc % 4);
    const long k = k0 + kc * 8;
    const int ea = e[(kb / kSplit) * rows_p + row];
    uint32_t word[kSlices][4];
    unsigned long long prev = 0;
#pragma unroll
    for (int u = 0; u < 8; u++) {
      const long ks = k + (mode >= 2 ? u ^ 1 : u);
      double x = 0.0;
      if (row < nrows && ks < k_len) x = src[row * ld + ks];
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
      if (u & 1) {
#pragma unroll
        for (int s = 0; s < kSlices; s++) {
          const float f0 = __uint_as_float(0x4b000000u | (uint32_t)((prev >> (56 - 8 * s)) & 0xff)) - 8388736.0f;
          const float f1 = __uint_as_float(0x4b000000u | (uint32_t)((v >> (56 - 8 * s)) & 0xff)) - 8388736.0f;
          word[s][u >> 1] = __byte_perm(__float_as_uint(f0), __float_as_uint(f1), 0x7632);
        }
      }
      prev = v;
    }
    const int r = (int)(row % ROWS);
    unsigned char *dst = img + (((row / ROWS) * nkb + kb) * kSlices) * kTile + (c16 * ROWS + r) * 16;
#pragma unroll
    for (int s = 0; s < kSlices; s++)
      *reinterpret_cast<uint4 *>(dst + s * kTile) = make_uint4(word[s][0], word[s][1], word[s][2], word[s][3]);
  }
}

// out[i][j] = scale * (sum of the splits' real columns, imaginary columns), the splits
// of all chunks in order: a chunk adds to the sums of those before it, the last one scales
__global__ void k_ex_reduce(const double *__restrict__ part, int nsplit, long mp, long np, int m, int n, long im_col,
                            bool first, bool last, double scale, double2 *__restrict__ out)
{
  const long total = (long)m * n;
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < total; e += (long)gridDim.x * blockDim.x) {
    const long i = e / n, j = e % n;
    double2 o = first ? make_double2(0, 0) : out[e];
#pragma unroll 4
    for (int s = 0; s < nsplit; s++) {
      const double *p = part + ((long)s * mp + i) * np;
      o.x += p[j];
      if (im_col) o.y += p[im_col + j];
    }
    out[e] = last ? make_double2(o.x * scale, o.y * scale) : o;
  }
}

}  // namespace ex

int exact_nt(fbse_ctx *c, const double *A, long lda, int ma, const double *B, long ldb, int nb, long L, ExactKind kind,
             double scale, double2 *out)
{
  using namespace ex;
  if (c->tc_poisoned)
    return set_err(c, FBSE_ERR_CUDA, "tensor-core path disabled: an earlier tensor-core wait timed out in this context");
  const bool cplx = kind != kExactReal;
  const long K = cplx ? 2 * L : L;
  const long mp = (ma + kM - 1) / kM * kM, n1 = (nb + kN - 1) / kN * kN, np = cplx ? 2 * n1 : n1;
  const long nkb_all = (K + kK - 1) / kK;
  // images of a K chunk within 4 GB (fbse_tuning.tc_image_bytes sets another size), its
  // partial sums within 2 GB, at least one split
  const long row_bytes = (long)kSlices * kK * 2;
  const double budget = c->tune.tc_image_bytes > 0 ? c->tune.tc_image_bytes : 4.0e9;
  const long fit = std::min((long)(budget / (double)(row_bytes * (mp + np))) / kSplit, 2000000000L / (8 * mp * np));
  const long nsplit_all = (nkb_all + kSplit - 1) / kSplit, nchunk = (nsplit_all + std::max(1L, fit) - 1) / std::max(1L, fit);
  const long nsplit = (nsplit_all + nchunk - 1) / nchunk, nkb = std::min(nkb_all, nsplit * kSplit);
  const size_t img_a = (size_t)(mp * nkb * row_bytes), img_b = (size_t)(np * nkb * row_bytes);
  const size_t part_b = (size_t)nsplit * mp * np * sizeof(double), exp_b = (size_t)nsplit * (mp + n1) * sizeof(int);
  void *scratch = nullptr;
  int rc = cached(c, kSlotTc, img_a + img_b + part_b + exp_b + 256, &scratch);
  if (rc) return rc;
  unsigned char *ia = static_cast<unsigned char *>(scratch), *ib = ia + img_a;
  double *part = reinterpret_cast<double *>(ib + img_b);
  int *ea = reinterpret_cast<int *>(reinterpret_cast<unsigned char *>(part) + part_b), *eb = ea + nsplit * mp;
  int *status = ea + nsplit * (mp + n1);
  FBSE_CUDA(c, cudaMemsetAsync(status, 0, sizeof(int), c->stream));
  FBSE_CUDA(c, cudaFuncSetAttribute(k_ex_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem));
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
    k_ex_gemm<<<dim3((unsigned)(mp / kM), (unsigned)(np / kN), (unsigned)ns), kThreads, kSmem, c->stream>>>(
        ia, ib, kb, ea, eb, part, mp, np, n1, status);
    FBSE_CHECK_LAUNCH(c);
    k_ex_reduce<<<grid((long)ma * nb), 256, 0, c->stream>>>(part, (int)ns, mp, np, ma, nb, cplx ? n1 : 0, ch == 0,
                                                             ch == nchunk - 1, scale, out);
    FBSE_CHECK_LAUNCH(c);
  }
  int hs = 0;
  if (d2h(c->stream, &hs, status, sizeof(int)) != cudaSuccess) return set_err(c, FBSE_ERR_CUDA, "exact product");
  if (hs) {
    c->tc_poisoned = 1;
    return set_err(c, FBSE_ERR_NOCONV, "exact product: a tensor-core wait timed out");
  }
  return FBSE_OK;
}

}  // namespace fbse
