// Complex "NT" product on the 5th-generation tensor cores (tcgen05, TMEM
// accumulators) with three-term split-TF32 products:
//   C[i][j] = sum_k A[i][k] B[j][k],  A = Ah + Al, B = Bh + Bl (TF32 parts),
//   C ~ Ah Bh^T + Ah Bl^T + Al Bh^T  (the Al Bl^T term is below FP32 rounding)
// accumulated in FP32 in tensor memory, split over K into FP32 partial
// tiles that are summed in FP64 afterwards.
//
// CTA: 128 x 256 outputs, 288 threads.  Eight warps load the complex rows (the next
// k block's while this one is multiplied), split them and write the tiles the MMA
// reads: 128 rows x 128 bytes (K-major, 128-byte swizzle: the 16-byte chunk c of
// row r sits at chunk c ^ (r % 8)) holding the real parts of 16 points, then their
// imaginary parts, one tile for the high and one for the low parts.  Two stages of A
// (128 rows) and B (256 rows): 96 KB each.  A thread of the ninth warp issues the
// MMAs (M = 128, N = 256, K = 8) of the real and of the imaginary accumulator, all of
// tensor memory, from the same tiles: Re = Ar Br - Ai Bi (A negated by the
// instruction), Im = Ar Bi + Ai Br.  Their commit frees the stage; at the end the
// eight warps read the accumulators out (lanes by warp % 4, Re or Im by warp / 4).
// Every wait is bounded: on a timeout the kernel records an error code, waits
// (bounded) for its MMAs, frees its tensor memory and returns.
//
// The tensor pipe bounds it: 24 MMAs a k block, 139 cycles each at the nominal TF32
// rate, against 48 KB read, of which the other row tile's CTA finds B's part in L2.
// With the split operands written to memory first, and B's twice for the two
// accumulators' two kernels, a product of 256 x 256 x 96^3 moved 30 GB and took 5.2 ms;
// 1.6 ms here (1.3 ms at the nominal rate).
#include <cstdint>
#include <cstdlib>

#include "fbse_internal.cuh"
#include "fbse_async.cuh"

namespace fbse {
namespace tc {

using namespace fbse::async;

constexpr int kBM = 128, kBN = 256, kBP = 16;   // CTA tile: M x N, points per k block
constexpr int kBK = 2 * kBP;                     // FP32 values per tile row: real parts, then imaginary parts
constexpr int kTileBytes = kBM * kBK * 4;        // one 128 x 32 tile: 16 KB
constexpr int kStageBytes = 6 * kTileBytes;      // Ah, Al (1 tile each), Bh, Bl (2 each)
constexpr int kStages = 2;
constexpr int kLoaders = 256;                     // loading threads (and the epilogue's)
constexpr int kItems = (kBM + kBN) * 4 / kLoaders;  // quarters of a row (4 points) a thread loads per k block
// shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row groups
// 1024 bytes apart (stride byte offset), leading byte offset unused (1)
__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr)
{
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFF) >> 4);       // start address
  d |= (uint64_t)1 << 16;                        // leading byte offset (unused for this layout)
  d |= (uint64_t)(1024 >> 4) << 32;              // stride byte offset
  d |= (uint64_t)1 << 46;                        // fixed 0b001
  d |= (uint64_t)2 << 61;                        // 128-byte swizzle
  return d;
}

// instruction descriptor: D = F32, A = B = TF32, both K-major, N = 256, M = 128;
// bit 13 negates A
__host__ __device__ constexpr uint32_t idesc_tf32(bool neg_a)
{
  return (1u << 4)                   // D format F32
         | (2u << 7)                 // A format TF32
         | (2u << 10)                // B format TF32
         | ((neg_a ? 1u : 0u) << 13)
         | ((uint32_t)(kBN >> 3) << 17)
         | ((uint32_t)(kBM >> 4) << 24);
}

template <bool NEG>
__device__ __forceinline__ void mma_tf32(uint32_t dtmem, uint64_t adesc, uint64_t bdesc, uint32_t acc)
{
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(dtmem),
      "l"(adesc), "l"(bdesc), "r"(idesc_tf32(NEG)), "r"(acc));
}

__device__ __forceinline__ void mma_commit(uint64_t *bar)
{
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

// round to the nearest TF32 value (10 mantissa bits, ties away from zero) and
// clear the 13 low bits, so that x - tf32(x) is exactly the part the tensor
// core does not see
__device__ __forceinline__ float tf32_round(float x)
{
  uint32_t u = __float_as_uint(x);
  if ((u & 0x7f800000u) != 0x7f800000u) u = (u + 0x1000u) & 0xffffe000u;
  return __uint_as_float(u);
}

// a thread's quarter rows of a k block: item i is 4 points (quarter t % 4) of row
// row_of(t, i) of the CTA's 128 rows of A and 256 of B.  Neighbouring groups of four
// lanes take rows 4 apart, whose swizzled chunks share no bank.
__device__ __forceinline__ int row_of(int t, int i)
{
  const int l = (t >> 2) & 7;
  return i * (kLoaders / 4) + (t >> 5) * 8 + ((l & 1) << 2 | l >> 1);
}

__device__ __forceinline__ void load_block(float2 (&v)[kItems][4], const float2 *const (&rows)[kItems], long p0, long L)
{
#pragma unroll
  for (int i = 0; i < kItems; i++)
#pragma unroll
    for (int e = 0; e < 4; e++)
      v[i][e] = rows[i] && p0 + e < L ? __ldg(rows[i] + p0 + e) : make_float2(0.0f, 0.0f);
}

// C partials: re, im[split][i][j] for i < mp (rows, multiple of 128), j < np
// (multiple of 256).  The CTA (bx, by, bz) covers rows 128 bx, columns 256 by and
// k blocks [kb0, kb1) of split bz, counted from the chunk's first one kbase; rows of A
// beyond ma, of B beyond nb and points beyond L are zero.
__global__ void __launch_bounds__(kLoaders + 32, 1)
    k_tc_gemm_nt(const float2 *__restrict__ A, int ma, const float2 *__restrict__ B, int nb, long L, long kbase, long nkb,
                 long kb_per_split, float *__restrict__ re, float *__restrict__ im, long mp, long np,
                 int *__restrict__ status)
{
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  // 1024-byte alignment of the stage buffers (the swizzle atom)
  unsigned char *stage = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
  __shared__ __align__(8) uint64_t full_bar[kStages], free_bar[kStages], done_bar;
  __shared__ uint32_t tmem_base;
  __shared__ int fail;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long kb0 = (long)blockIdx.z * kb_per_split;
  const long kb1 = min(nkb, kb0 + kb_per_split);
  const long nk = kb1 - kb0;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; s++) {
      mbar_init(&full_bar[s], kLoaders);
      mbar_init(&free_bar[s], 1);
    }
    mbar_init(&done_bar, 1);
    fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    // all 512 FP32 columns x 128 lanes of tensor memory: the two accumulators
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&tmem_base)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = tmem_base;
  int ok = 1;
  if (threadIdx.x < kLoaders) {
    const int t = threadIdx.x, q = t & 3;
    const float2 *rows[kItems];
    uint32_t dst[kItems];  // byte offset in a stage of the item's real parts, high
#pragma unroll
    for (int i = 0; i < kItems; i++) {
      const int r = row_of(t, i);
      const bool is_a = r < kBM;
      const long g = is_a ? (long)blockIdx.x * kBM + r : (long)blockIdx.y * kBN + (r - kBM);
      rows[i] = g < (is_a ? ma : nb) ? (is_a ? A : B) + g * L : nullptr;
      // tiles: Ah, Al, Bh (rows 0 - 127, 128 - 255), Bl
      const int tile = is_a ? 0 : 2 + (r - kBM) / kBM;
      dst[i] = (uint32_t)(tile * kTileBytes + (r % kBM) * 128 + ((q ^ (r & 7)) << 4));
    }
    float2 v[kItems][4];
    const long p0 = (kbase + kb0) * kBP + 4 * q;
    if (nk > 0) load_block(v, rows, p0, L);
    for (long it = 0; it < nk; it++) {
      const int s = (int)(it % kStages);
      if (it >= kStages) ok = mbar_wait(&free_bar[s], (uint32_t)(((it / kStages) - 1) & 1));
      if (!ok) break;
      unsigned char *buf = stage + (long)s * kStageBytes;
#pragma unroll
      for (int i = 0; i < kItems; i++) {
        const uint32_t lo = dst[i] < 2 * kTileBytes ? kTileBytes : 2 * kTileBytes;  // from the high to the low part
        float xr[4], xi[4], yr[4], yi[4];
#pragma unroll
        for (int e = 0; e < 4; e++) {
          xr[e] = tf32_round(v[i][e].x);
          xi[e] = tf32_round(v[i][e].y);
          yr[e] = tf32_round(v[i][e].x - xr[e]);
          yi[e] = tf32_round(v[i][e].y - xi[e]);
        }
        unsigned char *o = buf + dst[i], *oi = buf + (dst[i] ^ 64);  // the imaginary parts are chunk q + 4
        *reinterpret_cast<float4 *>(o) = make_float4(xr[0], xr[1], xr[2], xr[3]);
        *reinterpret_cast<float4 *>(oi) = make_float4(xi[0], xi[1], xi[2], xi[3]);
        *reinterpret_cast<float4 *>(o + lo) = make_float4(yr[0], yr[1], yr[2], yr[3]);
        *reinterpret_cast<float4 *>(oi + lo) = make_float4(yi[0], yi[1], yi[2], yi[3]);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      mbar_arrive(&full_bar[s]);
      if (it + 1 < nk) load_block(v, rows, p0 + (it + 1) * kBP, L);
    }
    if (!ok) atomicExch(&fail, 1);
  } else if (lane == 0) {
    // MMA issuer
    for (long it = 0; it < nk && ok; it++) {
      const int s = (int)(it % kStages);
      ok = mbar_wait(&full_bar[s], (uint32_t)((it / kStages) & 1));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;");
      const uint32_t b0 = smem_u32(stage + (long)s * kStageBytes);
      const uint32_t a_hi = b0, a_lo = b0 + kTileBytes, b_hi = b0 + 2 * kTileBytes, b_lo = b0 + 4 * kTileBytes;
      const uint32_t t_re = tmem, t_im = tmem + kBN;
#pragma unroll
      for (int kk = 0; kk < 2; kk++) {  // K = 8 TF32 (32 bytes) per instruction
        const uint32_t r = kk * 32, i = 64 + kk * 32;  // real and imaginary parts of 8 points
        const uint32_t first = (it == 0 && kk == 0) ? 0u : 1u;
        mma_tf32<false>(t_re, sw128_desc(a_hi + r), sw128_desc(b_hi + r), first);
        mma_tf32<false>(t_re, sw128_desc(a_hi + r), sw128_desc(b_lo + r), 1u);
        mma_tf32<false>(t_re, sw128_desc(a_lo + r), sw128_desc(b_hi + r), 1u);
        mma_tf32<true>(t_re, sw128_desc(a_hi + i), sw128_desc(b_hi + i), 1u);
        mma_tf32<true>(t_re, sw128_desc(a_hi + i), sw128_desc(b_lo + i), 1u);
        mma_tf32<true>(t_re, sw128_desc(a_lo + i), sw128_desc(b_hi + i), 1u);
        mma_tf32<false>(t_im, sw128_desc(a_hi + r), sw128_desc(b_hi + i), first);
        mma_tf32<false>(t_im, sw128_desc(a_hi + r), sw128_desc(b_lo + i), 1u);
        mma_tf32<false>(t_im, sw128_desc(a_lo + r), sw128_desc(b_hi + i), 1u);
        mma_tf32<false>(t_im, sw128_desc(a_hi + i), sw128_desc(b_hi + r), 1u);
        mma_tf32<false>(t_im, sw128_desc(a_hi + i), sw128_desc(b_lo + r), 1u);
        mma_tf32<false>(t_im, sw128_desc(a_lo + i), sw128_desc(b_hi + r), 1u);
      }
      mma_commit(&free_bar[s]);  // the stage is free once these MMAs have read it
    }
    mma_commit(&done_bar);  // and the accumulators are final once every MMA issued is done
    if (!ok) atomicExch(&fail, 1);
  }
  __syncwarp();
  // everyone waits for the accumulators (bounded)
  const bool done = nk > 0 ? mbar_wait(&done_bar, 0u) : true;
  asm volatile("tcgen05.fence::after_thread_sync;");
  __syncthreads();
  if (!done || fail) {
    if (threadIdx.x == 0) atomicExch(status, 1);
  } else if (warp < kLoaders / 32) {
    // epilogue: warps w and w + 4 read lanes 32 (w % 4) .. + 31 (rows) of Re and Im, 32 columns at a time
    const long row = (long)blockIdx.x * kBM + (warp & 3) * 32 + lane;
    float *dst = (warp < 4 ? re : im) + ((long)blockIdx.z * mp + row) * np + (long)blockIdx.y * kBN;
#pragma unroll 1
    for (int c0 = 0; c0 < kBN; c0 += 32) {
      uint32_t r[32];
      const uint32_t taddr = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)((warp >> 2) * kBN + c0);
      if (nk > 0) {
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
            "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
              "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
              "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]),
              "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]),
              "=r"(r[30]), "=r"(r[31])
            : "r"(taddr));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      } else {
#pragma unroll
        for (int j = 0; j < 32; j++) r[j] = 0;
      }
#pragma unroll
      for (int j = 0; j < 32; j += 4)
        *reinterpret_cast<float4 *>(dst + c0 + j) =
            make_float4(__uint_as_float(r[j]), __uint_as_float(r[j + 1]), __uint_as_float(r[j + 2]),
                        __uint_as_float(r[j + 3]));
    }
  }
  // after a timed-out wait, MMAs this CTA issued may still write the
  // accumulators: the issuing thread waits once more (bounded) before the
  // tensor memory is released; the host treats status = 1 as fatal for the
  // context's tensor-core path
  if (!done && nk > 0 && threadIdx.x == kLoaders) mbar_wait(&done_bar, 0u);
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
}

// out[i][j] = scale * (sum over splits of P0[i][j] (real part), P1 (imaginary)).
// Eight warps share 32 outputs: a warp sums every eighth split in order, the eight
// sums are added in order (864 splits of 256 x 256 by one thread an output: 0.80 ms,
// 0.45 ms here, the FP64 pipe with the conversions 82% busy).
__global__ void __launch_bounds__(256) k_tc_reduce(const float *__restrict__ P0, const float *__restrict__ P1, int nsplit,
                                                   long mp, long np, int m, int n, double scale, double2 *__restrict__ out)
{
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __shared__ double2 part[8][32];
  const long total = (long)m * n;
  for (long e0 = blockIdx.x * 32L; e0 < total; e0 += gridDim.x * 32L) {
    const long e = e0 + lane, i = e / n, j = e - i * n;
    double re = 0, im = 0;
    if (e < total) {
#pragma unroll 4
      for (int s = w; s < nsplit; s += 8) {
        re += (double)P0[((long)s * mp + i) * np + j];
        im += (double)P1[((long)s * mp + i) * np + j];
      }
    }
    part[w][lane] = make_double2(re, im);
    __syncthreads();
    if (w == 0 && e < total) {
      re = im = 0;
      for (int q = 0; q < 8; q++) {
        re += part[q][lane].x;
        im += part[q][lane].y;
      }
      out[e] = make_double2(re * scale, im * scale);
    }
    __syncthreads();
  }
}

}  // namespace tc

// ---------------------------------------------------------------------------
// complex products on the tensor cores (the BSE contraction):
//   out[i][j] = scale * sum_r A[i][r] B[j][r]
// A: ma rows, B: nb rows, L complex columns
// ---------------------------------------------------------------------------
static unsigned grid_of(long n)
{
  long g = (n + 255) / 256;
  if (g > 152L * 16) g = 152L * 16;
  return (unsigned)(g < 1 ? 1 : g);
}

int tc_complex_nt(fbse_ctx *c, const float2 *A, int ma, const float2 *B, int nb, long L, double scale, double2 *out)
{
  using namespace tc;
  if (c->tc_poisoned)
    return set_err(c, FBSE_ERR_CUDA, "tensor-core path disabled: an earlier tensor-core wait timed out in this context");
  const long mp = ((ma + kBM - 1) / kBM) * kBM;
  const long np = ((nb + kBN - 1) / kBN) * kBN;
  const long nkb_all = (L + kBP - 1) / kBP;
  // a launch covers a chunk of K whose split operands come to 24 GB
  // (fbse_tuning.tc_image_bytes sets another size)
  const double budget = c->tune.tc_image_bytes > 0 ? c->tune.tc_image_bytes : 24.0e9;
  long nkb_c = std::max<long>(1, (long)(budget / ((2.0 * mp + 4.0 * np) * kBK * 4.0)));
  if (nkb_c > nkb_all) nkb_c = nkb_all;
  const long nchunk = (nkb_all + nkb_c - 1) / nkb_c;
  // splits per chunk: at most 64 k blocks (768 accumulating MMAs) per split --
  // the tensor core's FP32 accumulation truncates, so its error grows with the
  // number of MMAs summed into one accumulator -- with the FP32 partials of
  // all chunks within 16 GB and at least two CTAs per SM
  const long tiles = (mp / kBM) * (np / kBN);
  long sps = std::max<long>(1, (nkb_c + 63) / 64);
  const long max_total = std::max<long>(nchunk, (long)(16.0e9 / (2.0 * 4.0 * mp * np)));
  if (sps * nchunk > max_total) sps = std::max<long>(1, max_total / nchunk);
  const long want = std::min<long>(nkb_c, (2 * 152 + tiles - 1) / tiles);
  if (sps < want) sps = want;
  const long kbs = (nkb_c + sps - 1) / sps;
  sps = (nkb_c + kbs - 1) / kbs;
  const long nsplit = sps * nchunk;
  const size_t part_n = (size_t)nsplit * mp * np;
  // partial tiles and the wait status, kept in the context between calls (grown on
  // demand, released by fbse_destroy)
  const size_t need = 2 * part_n * sizeof(float) + 256;
  void *scratch = nullptr;
  if (cached(c, kSlotTc, need, &scratch)) return set_err(c, FBSE_ERR_OOM, "tensor-core GEMM scratch");
  float *p0 = static_cast<float *>(scratch), *p1 = p0 + part_n;
  int *status = reinterpret_cast<int *>(static_cast<char *>(scratch) + need - 256);
  int rc = FBSE_OK;
  // launch errors end the call through the cleanup below (no early return)
  auto launched = [&](int nk) {
    FBSE_COUNT(nk);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) rc = set_err(c, FBSE_ERR_CUDA, std::string("tensor-core launch: ") + cudaGetErrorString(e));
    return e == cudaSuccess;
  };
  do {
    if (cudaMemsetAsync(status, 0, sizeof(int), c->stream) != cudaSuccess) { rc = set_err(c, FBSE_ERR_CUDA, "memset"); break; }
    const size_t smem = (size_t)kStages * kStageBytes + 1024;
    if (cudaFuncSetAttribute(tc::k_tc_gemm_nt, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
        cudaSuccess) { rc = set_err(c, FBSE_ERR_CUDA, "tensor-core GEMM attribute"); break; }
    for (long ch = 0; ch < nchunk && !rc; ch++) {
      const long nkb = std::min<long>(nkb_c, nkb_all - ch * nkb_c);
      const long nsp = (nkb + kbs - 1) / kbs;
      float *q0 = p0 + (size_t)ch * sps * mp * np, *q1 = p1 + (size_t)ch * sps * mp * np;
      if (nsp < sps) {  // a short last chunk: its unused partial slots must read as zero
        const size_t tail = (size_t)(sps - nsp) * mp * np * sizeof(float);
        if (cudaMemsetAsync(q0 + (size_t)nsp * mp * np, 0, tail, c->stream) != cudaSuccess ||
            cudaMemsetAsync(q1 + (size_t)nsp * mp * np, 0, tail, c->stream) != cudaSuccess) {
          rc = set_err(c, FBSE_ERR_CUDA, "tensor-core product: partial clear");
          break;
        }
      }
      dim3 g((unsigned)(mp / kBM), (unsigned)(np / kBN), (unsigned)nsp);
      tc::k_tc_gemm_nt<<<g, kLoaders + 32, smem, c->stream>>>(A, ma, B, nb, L, ch * nkb_c, nkb, kbs, q0, q1, mp, np, status);
      if (!launched(1)) break;
    }
    if (rc) break;
    tc::k_tc_reduce<<<grid_of(8 * (long)ma * nb), 256, 0, c->stream>>>(p0, p1, (int)nsplit, mp, np, ma, nb, scale, out);
    if (!launched(1)) break;
    int hs = 0;
    if (d2h(c->stream, &hs, status, sizeof(int)) != cudaSuccess) { rc = set_err(c, FBSE_ERR_CUDA, "tensor-core GEMM"); break; }
    if (hs) {
      c->tc_poisoned = 1;
      rc = set_err(c, FBSE_ERR_NOCONV, "tensor-core GEMM: a wait timed out");
    }
  } while (0);
  cudaStreamSynchronize(c->stream);
  return rc;
}

}  // namespace fbse
