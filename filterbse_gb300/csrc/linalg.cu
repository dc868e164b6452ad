// Orthogonalisation, subspace diagonalisation and sigma_E on the GPU.
//
// Replaces mod_ortho (thin SVD, filter_mpi/ortho.c:5-187), mod_diag
// (diag_H: n H psi, H_ij = dv <psi_i|H|psi_j>, dsyev/zheev, rotation,
// filter_mpi/Hmat.c:5-297) and mod_sigma (calc_sigma_E, two more H psi per
// state, filter_mpi/energy.c:383-539) with one Rayleigh-Ritz pass:
//
//   1. HPsi = H Psi                       (batched H psi, all n states)
//   2. G = dv Psi^H Psi, M = dv Psi^H HPsi (split-K GEMMs, FP64 partial sums)
//   3. G = V diag(l) V^H                  (FP64 Jacobi on the GPU)
//   4. keep l_i >= l_max * cut (the span of the left singular vectors with
//      s_i / s_0 above the cutoff), X = V_k diag(l_k)^{-1/2}
//   5. H' = X^H M X,  H' = U diag(E) U^H  (FP64 Jacobi on the GPU)
//   6. C = X U;  Psi_f = Psi C and HPsi_f = HPsi C in one pass, whose epilogue
//      forms the residual r_i = HPsi_f,i - E_i Psi_f,i and the norms
//   7. sigma_i = ||r_i|| / ||Psi_f,i||, states normalised (normalize_all).
// H is applied n times in total instead of the reference's 3n, and the Ritz
// vectors' residuals come from the same two GEMMs that build the vectors.
#include <algorithm>
#include <cmath>
#include <numeric>

#include <cstdlib>

#include <type_traits>

#include "fbse_internal.cuh"

namespace fbse {

int pack_states(fbse_ctx *c, const double *src, void *dst, long nsrc);
int unpack_states(fbse_ctx *c, const void *src, double *dst, long ndst);

// ---------------------------------------------------------------------------
// C[i][j] (+)= sum_l conj(A[i][l]) B[j][l]  over a K-chunk, i < n, j < n.
// A, B: n vectors of length L (complex: interleaved FP64 pairs; real: FP64).
// Tile 64 x 64 outputs per CTA (32 x 32 in FP64), 256 threads, K step 16.
// Compute type T (float for the mixed path, double for the FP64 path);
// partials are written in FP64: part[chunk][i][j].  Both products this file
// forms (Psi^H Psi and Psi^H H Psi) are Hermitian, so only tiles with
// ti <= tj are computed (blockIdx.x enumerates them) and an off-diagonal
// tile is also stored conjugate-transposed.  Shared tiles hold complex values
// as C<T> with one element of padding per K row, so the transposing stores
// (consecutive threads: consecutive k) and the float2 / double2 reads of the
// product loop are free of bank conflicts.
// ---------------------------------------------------------------------------
// (hi, lo) += x with TwoSum: hi + lo keeps the exact sum to about twice the
// working precision (Knuth, The Art of Computer Programming vol. 2, 4.2.2)
template <typename T> __device__ __forceinline__ void two_sum_acc(T &hi, T &lo, T x)
{
  const T s = hi + x;
  const T bb = s - hi;
  const T err = (hi - (s - bb)) + (x - bb);
  hi = s;
  lo += err;
}

template <typename T, bool CPLX, int MINB, int TM = 64>
__global__ void __launch_bounds__(256, MINB) k_gram(const double *__restrict__ A, const double *__restrict__ B, int n,
                                              long L, long kchunk, double2 *__restrict__ part)
{
  constexpr int TK = 16, R = TM / 16;
  using E = typename std::conditional<CPLX, C<T>, T>::type;
  __shared__ E As[TK][TM + 1];
  __shared__ E Bs[TK][TM + 1];
  // pair (ti, tj), ti <= tj, of 64 x 64 blocks from the linear index, and the tile's
  // corner in it.  Both halves of a diagonal block are formed (they differ in their
  // last bits), so the tile size changes no value
  constexpr int S = 64 / TM;
  const int nt = (n + 63) / 64;
  int ti = 0, rem = blockIdx.x / (S * S);
  while (rem >= nt - ti) { rem -= nt - ti; ti++; }
  const int tj = ti + rem, sub = blockIdx.x % (S * S);
  const int i0 = ti * 64 + sub / S * TM, j0 = tj * 64 + sub % S * TM;
  if (i0 >= n || j0 >= n) return;
  const long k0 = blockIdx.z * kchunk;
  const long k1 = min(L, k0 + kchunk);
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  // FP32: the sums of each K step of 16 products are added into a
  // float-float pair (hi, lo) with TwoSum (Knuth), so the long sums over the
  // grid keep about 48 bits; FP64: plain accumulation
  T accr[R][R], acci[R][R];
  T hir[R][R], hii[R][R], lor[R][R], loi[R][R];
#pragma unroll
  for (int a = 0; a < R; a++)
#pragma unroll
    for (int b = 0; b < R; b++) { accr[a][b] = 0; acci[a][b] = 0; hir[a][b] = hii[a][b] = lor[a][b] = loi[a][b] = 0; }
  for (long kb = k0; kb < k1; kb += TK) {
    // load: TM rows x 16 k for A and B; thread t loads rows (t / 16) + 16 q, k = t % 16
#pragma unroll
    for (int q = 0; q < R; q++) {
      const int r = ty + 16 * q, kk = tx;
      const long k = kb + kk;
      const bool okA = (i0 + r < n) && (k < k1);
      const bool okB = (j0 + r < n) && (k < k1);
      if constexpr (CPLX) {
        const double2 va = okA ? reinterpret_cast<const double2 *>(A)[(long)(i0 + r) * L + k] : make_double2(0, 0);
        const double2 vb = okB ? reinterpret_cast<const double2 *>(B)[(long)(j0 + r) * L + k] : make_double2(0, 0);
        As[kk][r] = mk<T>((T)va.x, (T)va.y);
        Bs[kk][r] = mk<T>((T)vb.x, (T)vb.y);
      } else {
        As[kk][r] = okA ? (T)A[(long)(i0 + r) * L + k] : T(0);
        Bs[kk][r] = okB ? (T)B[(long)(j0 + r) * L + k] : T(0);
      }
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < TK; kk++) {
      T ar[R], ai[R], br[R], bi[R];
#pragma unroll
      for (int a = 0; a < R; a++) {
        if constexpr (CPLX) {
          const C<T> u = As[kk][ty + 16 * a], v = Bs[kk][tx + 16 * a];
          ar[a] = u.x; ai[a] = u.y; br[a] = v.x; bi[a] = v.y;
        } else {
          ar[a] = As[kk][ty + 16 * a]; br[a] = Bs[kk][tx + 16 * a];
          ai[a] = bi[a] = T(0);
        }
      }
#pragma unroll
      for (int a = 0; a < R; a++)
#pragma unroll
        for (int b = 0; b < R; b++) {
          // conj(a) * b; FP64 spells its roundings out (they decide phases, see the caller)
          if constexpr (sizeof(T) == 8) {
            if constexpr (CPLX) {
              accr[a][b] = __dadd_rn(accr[a][b], __fma_rn(ar[a], br[b], __dmul_rn(ai[a], bi[b])));
              acci[a][b] = __dadd_rn(acci[a][b], __fma_rn(ar[a], bi[b], -__dmul_rn(ai[a], br[b])));
            } else {
              accr[a][b] = __dadd_rn(accr[a][b], __dmul_rn(ar[a], br[b]));
            }
          } else {
            accr[a][b] += ar[a] * br[b] + (CPLX ? ai[a] * bi[b] : T(0));
            if (CPLX) acci[a][b] += ar[a] * bi[b] - ai[a] * br[b];
          }
        }
    }
    if constexpr (sizeof(T) == 4) {
#pragma unroll
      for (int a = 0; a < R; a++)
#pragma unroll
        for (int b = 0; b < R; b++) {
          two_sum_acc(hir[a][b], lor[a][b], accr[a][b]);
          accr[a][b] = 0;
          if (CPLX) {
            two_sum_acc(hii[a][b], loi[a][b], acci[a][b]);
            acci[a][b] = 0;
          }
        }
    }
    __syncthreads();
  }
  double2 *P = part + (long)blockIdx.z * n * n;
#pragma unroll
  for (int a = 0; a < R; a++)
#pragma unroll
    for (int b = 0; b < R; b++) {
      const int i = i0 + ty + 16 * a, j = j0 + tx + 16 * b;
      double vr = (double)accr[a][b], vi = (double)acci[a][b];
      if constexpr (sizeof(T) == 4) {
        vr = (double)hir[a][b] + (double)lor[a][b];
        vi = (double)hii[a][b] + (double)loi[a][b];
      }
      if (i < n && j < n) {
        P[(long)i * n + j] = make_double2(vr, vi);
        if (ti != tj) P[(long)j * n + i] = make_double2(vr, -vi);
      }
    }
}

__global__ void k_sum_partials(const double2 *__restrict__ part, int nchunk, long nn, double scale,
                               double2 *__restrict__ out)
{
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < nn; e += (long)gridDim.x * blockDim.x) {
    double r = 0, im = 0;
    for (int c = 0; c < nchunk; c++) { r += part[(long)c * nn + e].x; im += part[(long)c * nn + e].y; }
    out[e] = make_double2(r * scale, im * scale);
  }
}

// ---------------------------------------------------------------------------
// small dense FP64 complex GEMM: C[m][p] = op(A) op(B), row-major,
// opA = 'N' (A is m x k) or 'H' (A is k x m, conjugate-transposed)
// ---------------------------------------------------------------------------
__global__ void k_zgemm(int m, int p, int k, const double2 *__restrict__ A, int lda, bool ah,
                        const double2 *__restrict__ B, int ldb, bool bh, double2 *__restrict__ Cm, int ldc)
{
  const int i = blockIdx.y * 16 + threadIdx.y, j = blockIdx.x * 16 + threadIdx.x;
  if (i >= m || j >= p) return;
  double r = 0, im = 0;
  for (int l = 0; l < k; l++) {
    double2 a = ah ? A[(long)l * lda + i] : A[(long)i * lda + l];
    if (ah) a.y = -a.y;
    double2 b = bh ? B[(long)j * ldb + l] : B[(long)l * ldb + j];
    if (bh) b.y = -b.y;
    r += a.x * b.x - a.y * b.y;
    im += a.x * b.y + a.y * b.x;
  }
  Cm[(long)i * ldc + j] = make_double2(r, im);
}

int zgemm_dev(fbse_ctx *c, int m, int p, int k, const double2 *A, int lda, bool ah, const double2 *B, int ldb, bool bh,
              double2 *C, int ldc)
{
  dim3 b(16, 16), g((p + 15) / 16, (m + 15) / 16);
  k_zgemm<<<g, b, 0, c->stream>>>(m, p, k, A, lda, ah, B, ldb, bh, C, ldc);
  FBSE_CHECK_LAUNCH(c);
  return FBSE_OK;
}

// ---------------------------------------------------------------------------
// Hermitian eigensolver: cyclic two-sided Jacobi with the round-robin pairing
// (n/2 disjoint rotations per round, n-1 rounds per sweep), one cooperative
// launch per sweep.  A (n x n, row-major, Hermitian) is diagonalised; V
// accumulates the unitary so that A_in = V diag(A_out) V^H.
//
// The pairs of a round cover every index once, so every element of A lies in one
// 2 x 2 block (row pair a, column pair b) and every element of V in one 1 x 2
// block (row i, column pair b).  A block is rotated from both sides at once,
// A_blk <- U_a^H A_blk U_b:
//   rows:    new p = cs a_p - sn e^{i phi} a_q,   new q = sn a_p + cs e^{i phi} a_q
//   columns: new p = cs a_p - sn e^{-i phi} a_q,  new q = sn a_p + cs e^{-i phi} a_q
// and the rotated pair's off-diagonal element, zero in exact arithmetic, is set to
// zero.  A dummy index (q = n for odd n) carries the identity.
//
// The arithmetic of every element and rotation is fixed: eigenvectors of a
// rank-deficient overlap carry phases that follow the last bits of this sum order
// (a filtered set's null directions are rounding noise, and every rotation passes
// a phase on), so a different but equally accurate formula turns whole Ritz sets.
//
// A round is a chain of latencies (the pair's elements from L2, the rotation's
// roots, the update, the grid barrier), so it has one barrier: a round reads A from
// one buffer and writes every element to another, and each tile of 8 x 8 blocks (or
// 8 pairs x 32 rows of V) computes the rotations of its own 16 pairs.  Tiles of 64
// threads spread the FP64 work (2 lanes per clock and SM) over every SM from n = 128
// on.  Larger matrices share the rotations behind a second barrier (jacobi_eig_dev).
// Measured per round against two barriers and a thread per block of the whole matrix:
// n = 128 12.5 -> 6.6 us, n = 196 12.7 -> 6.9 us, n = 115 real 12.4 -> 6.6 us.
// ---------------------------------------------------------------------------
struct __align__(16) Rot {
  double cs, sn, pr, pi;  // U = D J:  U_pp = cs, U_pq = sn, U_qp = -sn e^{-i phi}, U_qq = cs e^{-i phi}
};

__device__ __forceinline__ void rr_pair(int r, int slot, int m, int &p, int &q)
{  // round-robin tournament: player m-1 fixed, the others rotate
  int a, b;
  if (slot == 0) { a = m - 1; b = r % (m - 1); }
  else { a = (r + slot) % (m - 1); b = (r - slot + (m - 1)) % (m - 1); }
  p = min(a, b);
  q = max(a, b);
}

// the rotation that zeroes the pair's off-diagonal element
__device__ __forceinline__ Rot pair_rotation(const double2 *__restrict__ A, int n, int p, int q)
{
  Rot R{1.0, 0.0, 1.0, 0.0};
  if (q < n) {
    const double app = __ldcg(&A[(long)p * n + p]).x, aqq = __ldcg(&A[(long)q * n + q]).x;
    const double2 apq = __ldcg(&A[(long)p * n + q]);
    const double mag = hypot(apq.x, apq.y);
    if (mag > 1e-300 && mag > 1e-18 * sqrt(fabs(app * aqq))) {
      const double tau = (aqq - app) / (2.0 * mag);
      const double t = (tau >= 0 ? 1.0 : -1.0) / (fabs(tau) + sqrt(1.0 + tau * tau));
      R.cs = 1.0 / sqrt(1.0 + t * t);
      R.sn = t * R.cs;
      R.pr = apq.x / mag;  // e^{i phi}
      R.pi = apq.y / mag;
    }
  }
  return R;
}

// grid-wide barrier number `gen` (1, 2, ..) of a cooperative launch; bounded
__device__ __forceinline__ bool grid_barrier(unsigned *counter, unsigned target)
{
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(counter) : "memory");
    int done = 0;
    for (long i = 0; i < (1L << 26) && !done; i++) {
      unsigned v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(counter) : "memory");
      done = (int)(v - target) >= 0;
    }
    ok = done;
  }
  __syncthreads();
  return ok != 0;
}

constexpr int kJT = 8, kJRows = 32, kJThreads = 64;  // pairs per tile side, V rows per tile

// REAL: every imaginary part is zero and stays zero.  off[0..1]: off-diagonal and
// diagonal sums of squares, off[2]: nonzero when a barrier gave up, then the CTAs'
// partial sums.  count0: arrivals of earlier launches on this counter.  rots: room for
// the round's m / 2 rotations when they are formed once, behind a barrier of their own,
// else null.
template <bool REAL>
__global__ void __launch_bounds__(kJThreads) k_jacobi_sweep(double2 *__restrict__ A0, double2 *__restrict__ A1,
                                                            double2 *__restrict__ V, int n, int m,
                                                            Rot *__restrict__ rots, unsigned *__restrict__ counter,
                                                            unsigned count0, double *__restrict__ off)
{
  const int half = m / 2, T = (half + kJT - 1) / kJT, TV = (n + kJRows - 1) / kJRows;
  const int na = T * T, ntile = na + T * TV;
  const int tid = threadIdx.x;
  __shared__ Rot rot[2 * kJT];
  // (p, q) <- (cs p - sn w q, sn p + cs w q), w the (conjugated) phase; the roundings
  // are spelled out (row: of which product of w q's imaginary part)
  auto turn = [](const Rot &R, double2 w, double2 &ap, double2 &aq, bool row) {
    double2 x;
    x.x = REAL ? __dmul_rn(w.x, aq.x) : __fma_rn(w.x, aq.x, -__dmul_rn(w.y, aq.y));
    x.y = row ? __fma_rn(w.y, aq.x, __dmul_rn(w.x, aq.y)) : __fma_rn(w.x, aq.y, __dmul_rn(w.y, aq.x));
    const double2 y = ap;
    ap.x = __fma_rn(R.cs, y.x, -__dmul_rn(R.sn, x.x));
    aq.x = __fma_rn(R.sn, y.x, __dmul_rn(R.cs, x.x));
    if (REAL) return;
    ap.y = __fma_rn(R.cs, y.y, -__dmul_rn(R.sn, x.y));
    aq.y = __fma_rn(R.sn, y.y, __dmul_rn(R.cs, x.y));
  };
  unsigned gen = count0;
  for (int r = 0; r < m - 1; r++) {
    const double2 *src = (r & 1) ? A1 : A0;
    double2 *dst = (r & 1) ? A0 : A1;
    if (rots) {
      for (int s = blockIdx.x * kJThreads + tid; s < half; s += gridDim.x * kJThreads) {
        int p, q;
        rr_pair(r, s, m, p, q);
        rots[s] = pair_rotation(src, n, p, q);
      }
      gen += gridDim.x;
      if (!grid_barrier(counter, gen)) {
        if (tid == 0) off[2] = 1.0;
        return;
      }
    }
    for (int tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
      const bool on_a = tile < na;
      // tiles of pairs; V: pairs tb, rows ta
      const int ta = on_a ? tile / T : (tile - na) % TV, tb = on_a ? tile % T : (tile - na) / TV;
      // this thread's block(s) on their way while the rotations are formed
      const int la = tid / kJT, lb = tid % kJT, sa = ta * kJT + la, sb = tb * kJT + lb;
      int pa = 0, qa = n, pb = 0, qb = n;
      const bool live = sb < half && (!on_a || sa < half);
      if (live) {
        rr_pair(r, sb, m, pb, qb);
        if (on_a) rr_pair(r, sa, m, pa, qa);
      }
      double2 x[2][2];
      double2 v[kJRows / kJT][2];
      if (live && on_a) {
        x[0][0] = __ldcg(&src[(long)pa * n + pb]);
        x[0][1] = qb < n ? __ldcg(&src[(long)pa * n + qb]) : make_double2(0, 0);
        x[1][0] = qa < n ? __ldcg(&src[(long)qa * n + pb]) : make_double2(0, 0);
        x[1][1] = qa < n && qb < n ? __ldcg(&src[(long)qa * n + qb]) : make_double2(0, 0);
      } else if (live && qb < n) {
#pragma unroll
        for (int u = 0; u < kJRows / kJT; u++) {
          const int row = ta * kJRows + la + kJT * u;
          if (row >= n) continue;
          v[u][0] = __ldcg(&V[(long)row * n + pb]);
          v[u][1] = __ldcg(&V[(long)row * n + qb]);
        }
      }
      __syncthreads();  // the previous tile is done with rot
      if (tid < 2 * kJT) {
        const int s = (tid < kJT ? ta * kJT : tb * kJT - kJT) + tid;
        if (s < half && (on_a || tid >= kJT)) {
          if (rots) {
            const double2 *t = reinterpret_cast<const double2 *>(rots + s);
            const double2 j = __ldcg(t), phase = __ldcg(t + 1);
            rot[tid] = Rot{j.x, j.y, phase.x, phase.y};
          } else {
            int p, q;
            rr_pair(r, s, m, p, q);
            rot[tid] = pair_rotation(src, n, p, q);
          }
        }
      }
      __syncthreads();
      if (!live) continue;
      const Rot &Rb = rot[kJT + lb];
      const double2 wb = make_double2(Rb.pr, -Rb.pi);
      if (on_a) {
        const Rot &Ra = rot[la];
        const double2 wa = make_double2(Ra.pr, Ra.pi);
        turn(Ra, wa, x[0][0], x[1][0], true);
        turn(Ra, wa, x[0][1], x[1][1], true);
        turn(Rb, wb, x[0][0], x[0][1], false);
        turn(Rb, wb, x[1][0], x[1][1], false);
        if (sa == sb && !(Ra.cs == 1.0 && Ra.sn == 0.0)) x[0][1] = x[1][0] = make_double2(0, 0);
        __stcg(&dst[(long)pa * n + pb], x[0][0]);
        if (qb < n) __stcg(&dst[(long)pa * n + qb], x[0][1]);
        if (qa < n) __stcg(&dst[(long)qa * n + pb], x[1][0]);
        if (qa < n && qb < n) __stcg(&dst[(long)qa * n + qb], x[1][1]);
      } else if (qb < n) {
#pragma unroll
        for (int u = 0; u < kJRows / kJT; u++) {
          const int row = ta * kJRows + la + kJT * u;
          if (row >= n) continue;
          turn(Rb, wb, v[u][0], v[u][1], false);
          __stcg(&V[(long)row * n + pb], v[u][0]);
          __stcg(&V[(long)row * n + qb], v[u][1]);
        }
      }
    }
    gen += gridDim.x;
    if (!grid_barrier(counter, gen)) {
      if (tid == 0) off[2] = 1.0;
      return;
    }
  }
  // off-diagonal Frobenius norm and diagonal norm: per-CTA partials summed by
  // CTA 0 in a fixed order, so that the sweep count is the same on every run
  const double2 *A = ((m - 1) & 1) ? A1 : A0;
  double so = 0, sd = 0;
  for (long e = blockIdx.x * (long)kJThreads + tid; e < (long)n * n; e += (long)gridDim.x * kJThreads) {
    const double2 a = __ldcg(&A[e]);
    const double t = a.x * a.x + a.y * a.y;
    if (e / n == e % n) sd += t;
    else so += t;
  }
  __shared__ double ws[2][kJThreads / 32];
  auto warp_sums = [&](double &x, double &y) {
    for (int o = 16; o > 0; o >>= 1) {
      x += __shfl_xor_sync(0xffffffffu, x, o);
      y += __shfl_xor_sync(0xffffffffu, y, o);
    }
  };
  warp_sums(so, sd);
  if ((tid & 31) == 0) {
    ws[0][tid >> 5] = so;
    ws[1][tid >> 5] = sd;
  }
  __syncthreads();
  if (tid == 0) {
    __stcg(&off[3 + 2 * blockIdx.x], ws[0][0] + ws[0][1]);
    __stcg(&off[4 + 2 * blockIdx.x], ws[1][0] + ws[1][1]);
  }
  gen += gridDim.x;
  if (!grid_barrier(counter, gen)) {
    if (tid == 0) off[2] = 1.0;
    return;
  }
  if (blockIdx.x == 0 && tid < 32) {
    double to = 0, td = 0;
    for (int i = tid; i < (int)gridDim.x; i += 32) {
      to += __ldcg(&off[3 + 2 * i]);
      td += __ldcg(&off[4 + 2 * i]);
    }
    warp_sums(to, td);
    if (tid == 0) {
      off[0] = to;
      off[1] = td;
    }
  }
}

__global__ void k_identity(double2 *V, int n)
{
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < (long)n * n; e += (long)gridDim.x * blockDim.x)
    V[e] = make_double2(e / n == e % n ? 1.0 : 0.0, 0.0);
}

// eigen-decomposition of the Hermitian n x n matrix A (device, overwritten);
// V (device, n x n) receives the eigenvectors as columns, w (host) the
// eigenvalues in the order of V's columns.  real: A has no imaginary part
int jacobi_eig_dev(fbse_ctx *c, double2 *A, double2 *V, int n, std::vector<double> &w, bool real)
{
  const int m = n + (n & 1);
  const void *kernel = real ? (const void *)k_jacobi_sweep<true> : (const void *)k_jacobi_sweep<false>;
  int dev = 0, nsm = 0, per_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kJThreads, 0);
  const long T = (m / 2 + kJT - 1) / kJT, tiles = T * T + T * ((n + kJRows - 1) / kJRows);
  // a tile per CTA, up to four CTAs per SM (more only lengthen the barrier; eight gain 3%
  // at n = 1600 and lose 10% at 784)
  const int most = nsm * std::min(4, std::max(1, per_sm));
  const int blocks = (int)std::min<long>(std::max<long>(1, tiles), most);
  // A tile that forms its 16 rotations spends two thirds of its FP64 time on them, which
  // is hidden behind the barrier while every tile has a CTA and SM time to itself (n up to
  // 320).  With more tiles than CTAs the rotations are formed once, behind a second
  // barrier: eigensolve of n = 360 52 -> 46 ms, 784 394 -> 259, 1600 3.56 -> 2.03 s (0.33
  // and 2.43 s with a thread per block and two barriers), 3360 18 s (22).  The values are
  // the same.
  const bool table = tiles > most;
  // the second buffer of A, the norms and their partials, the barrier's counter,
  // kept in the context between calls
  const size_t a_bytes = (size_t)n * n * sizeof(double2), rot_bytes = table ? m / 2 * sizeof(Rot) : 0;
  const size_t off_bytes = (3 + 2 * (size_t)blocks) * sizeof(double);
  void *scratch = nullptr;
  int rc = cached(c, kSlotJacobi, a_bytes + rot_bytes + off_bytes + 16, &scratch);
  if (rc) return rc;
  double2 *A1 = static_cast<double2 *>(scratch), *cur = A, *other = A1;
  Rot *rots = table ? reinterpret_cast<Rot *>(A1 + (size_t)n * n) : nullptr;
  double *off = reinterpret_cast<double *>(static_cast<char *>(scratch) + a_bytes + rot_bytes);
  unsigned *counter = reinterpret_cast<unsigned *>(off + 3 + 2 * blocks), count = 0;
  FBSE_CUDA(c, cudaMemsetAsync(off, 0, off_bytes + 16, c->stream));
  FBSE_COUNT(1); k_identity<<<256, 256, 0, c->stream>>>(V, n);
  double h[3] = {0, 0, 0};
  bool conv = (n < 2);
  for (int sweep = 0; sweep < 60 && !conv; sweep++) {
    int mm = m;
    void *args[] = {&cur, &other, &V, &n, &mm, &rots, &counter, &count, &off};
    FBSE_COUNT(1); if (cudaLaunchCooperativeKernel(kernel, blocks, kJThreads, args, 0, c->stream) != cudaSuccess) {
      rc = set_err(c, FBSE_ERR_CUDA, std::string("jacobi launch: ") + cudaGetErrorString(cudaGetLastError()));
      break;
    }
    // m - 1 rounds, twice with the table, and the norms
    count += (unsigned)(table ? 2 * m - 1 : m) * (unsigned)blocks;
    if ((m - 1) & 1) std::swap(cur, other);
    if (cudaMemcpyAsync(h, off, 3 * sizeof(double), cudaMemcpyDeviceToHost, c->stream) != cudaSuccess ||
        cudaStreamSynchronize(c->stream) != cudaSuccess) {
      rc = set_err(c, FBSE_ERR_CUDA, "jacobi sweep");
      break;
    }
    if (h[2] != 0) { rc = set_err(c, FBSE_ERR_NOCONV, "jacobi: a grid barrier timed out"); break; }
    if (!(h[0] == h[0])) { rc = set_err(c, FBSE_ERR_NAN, "jacobi: NaN in matrix"); break; }
    if (h[0] <= 1e-30 * h[1] || h[0] < 1e-300) conv = true;
  }
  if (!rc && !conv) rc = set_err(c, FBSE_ERR_NOCONV, "jacobi eigensolver did not converge in 60 sweeps");
  if (!rc) {
    // only the diagonal is needed on the host: one strided copy (pitch n + 1)
    std::vector<double2> d((size_t)n);
    if (cudaMemcpy2DAsync(d.data(), sizeof(double2), cur, (size_t)(n + 1) * sizeof(double2), sizeof(double2), (size_t)n,
                          cudaMemcpyDeviceToHost, c->stream) != cudaSuccess ||
        cudaStreamSynchronize(c->stream) != cudaSuccess)
      rc = set_err(c, FBSE_ERR_CUDA, "jacobi download");
    w.resize(n);
    for (int i = 0; i < n && !rc; i++) w[i] = d[i].x;
  }
  return rc;
}

// ---------------------------------------------------------------------------
// rotation with residual epilogue
//   P[i][l] = sum_j Psi[j][l] C[j][i],  Q[i][l] = sum_j HPsi[j][l] C[j][i]
//   out[i][l] = P;  part[blk][i] += |Q - E_i P|^2, |P|^2, Re(conj(P) Q)
// tile: 128 grid elements x 32 output states per CTA, 256 threads; the state
// tiles of one grid tile are consecutive blocks (they share the grid tile's
// Psi / H Psi through L2, so the states stream from DRAM once), and the next
// j block is loaded into registers while the current one is multiplied
// ---------------------------------------------------------------------------
// PART 2: rotate Psi and H Psi together; PART 0: Psi only (writes out);
// PART 1: H Psi only, reading the rotated Psi back from out for the residual
// sums (two launches of half the accumulators each: two CTAs per SM instead
// of one for the FP32 path).
template <typename T, bool CPLX, int PART>
__global__ void __launch_bounds__(256, PART == 2 ? 1 : 2) k_rotate(const double *__restrict__ Psi, const double *__restrict__ HPsi, int n,
                                                long L, const double2 *__restrict__ Cm, int k,
                                                const double *__restrict__ E, double *__restrict__ out,
                                                double *__restrict__ part)
{
  constexpr int TL = 128, TS = 32, TJ = 8;
  constexpr int NU = TJ * TL / 256;  // Psi / H Psi tile values per thread
  static_assert(TJ * TS == 256, "one coefficient per thread and j block");
  const int nsb = (k + TS - 1) / TS;
  const long bx = blockIdx.x / nsb;
  const long l0 = bx * TL;
  const int s0 = (int)(blockIdx.x % nsb) * TS;
  // complex values as C<T>: one float2 / double2 access per value
  using Elt = typename std::conditional<CPLX, C<T>, T>::type;
  using Raw = typename std::conditional<CPLX, double2, double>::type;
  __shared__ Elt Ps[TJ][TL];
  __shared__ Elt Hs[TJ][TL];
  __shared__ C<T> Cs[TJ][TS];
  __shared__ double red[TS][3];
  const int tl = threadIdx.x % 32;  // 4 grid elements per thread: tl + 32 q
  const int ts = threadIdx.x / 32;  // 4 output states per thread: ts + 8 r
  T pr[4][4], pim[4][4], qr[4][4], qim[4][4];
#pragma unroll
  for (int a = 0; a < 4; a++)
#pragma unroll
    for (int b = 0; b < 4; b++) { pr[a][b] = pim[a][b] = qr[a][b] = qim[a][b] = 0; }
  if (threadIdx.x < TS * 3) red[threadIdx.x / 3][threadIdx.x % 3] = 0;
  Raw rp[NU], rh[NU];
  double2 rc;
  auto fetch = [&](int jb) {
#pragma unroll
    for (int u = 0; u < NU; u++) {
      const int t = threadIdx.x + 256 * u;
      const int j = jb + t / TL;
      const long l = l0 + t % TL;
      const bool ok = (j < n) && (l < L);
      if constexpr (CPLX) {
        if constexpr (PART != 1) rp[u] = ok ? reinterpret_cast<const double2 *>(Psi)[(long)j * L + l] : make_double2(0, 0);
        if constexpr (PART != 0) rh[u] = ok ? reinterpret_cast<const double2 *>(HPsi)[(long)j * L + l] : make_double2(0, 0);
      } else {
        if constexpr (PART != 1) rp[u] = ok ? Psi[(long)j * L + l] : 0.0;
        if constexpr (PART != 0) rh[u] = ok ? HPsi[(long)j * L + l] : 0.0;
      }
    }
    const int j = jb + threadIdx.x / TS, sc = s0 + threadIdx.x % TS;
    rc = (j < n && sc < k) ? Cm[(long)j * k + sc] : make_double2(0, 0);
  };
  fetch(0);
  for (int jb = 0; jb < n; jb += TJ) {
#pragma unroll
    for (int u = 0; u < NU; u++) {
      const int t = threadIdx.x + 256 * u;
      const int jj = t / TL, ll = t % TL;
      if constexpr (CPLX) {
        if constexpr (PART != 1) Ps[jj][ll] = mk<T>((T)rp[u].x, (T)rp[u].y);
        if constexpr (PART != 0) Hs[jj][ll] = mk<T>((T)rh[u].x, (T)rh[u].y);
      } else {
        if constexpr (PART != 1) Ps[jj][ll] = (T)rp[u];
        if constexpr (PART != 0) Hs[jj][ll] = (T)rh[u];
      }
    }
    Cs[threadIdx.x / TS][threadIdx.x % TS] = mk<T>((T)rc.x, (T)rc.y);
    __syncthreads();
    if (jb + TJ < n) fetch(jb + TJ);
#pragma unroll
    for (int jj = 0; jj < TJ; jj++) {
#pragma unroll
      for (int a = 0; a < 4; a++) {
        const int ll = tl + 32 * a;
        T xr = T(0), xi = T(0), yr = T(0), yi = T(0);
        if constexpr (CPLX) {
          if constexpr (PART != 1) { const C<T> x = Ps[jj][ll]; xr = x.x; xi = x.y; }
          if constexpr (PART != 0) { const C<T> y = Hs[jj][ll]; yr = y.x; yi = y.y; }
        } else {
          if constexpr (PART != 1) xr = Ps[jj][ll];
          if constexpr (PART != 0) yr = Hs[jj][ll];
        }
#pragma unroll
        for (int b = 0; b < 4; b++) {
          const int ss = ts + 8 * b;
          const C<T> cv = Cs[jj][ss];
          const T cr = cv.x, ci = cv.y;
          // two multiply-adds a value, one for real states, whose coefficients are real
          // (128 real FP64 states of 133380 points 17.2 -> 7.7 ms, 128 FP32 spinors of
          // 86^3 17.0 -> 14.8 ms)
          if constexpr (PART != 1) {
            pr[a][b] += xr * cr;
            if constexpr (CPLX) {
              pr[a][b] -= xi * ci;
              pim[a][b] += xr * ci;
              pim[a][b] += xi * cr;
            }
          }
          if constexpr (PART != 0) {
            qr[a][b] += yr * cr;
            if constexpr (CPLX) {
              qr[a][b] -= yi * ci;
              qim[a][b] += yr * ci;
              qim[a][b] += yi * cr;
            }
          }
        }
      }
    }
    __syncthreads();
  }
  // epilogue
#pragma unroll
  for (int b = 0; b < 4; b++) {
    const int s = s0 + ts + 8 * b;
    double rr = 0, pp = 0, pq = 0;
    if (s < k) {
      const double e = E[s];
#pragma unroll
      for (int a = 0; a < 4; a++) {
        const long l = l0 + tl + 32 * a;
        if (l < L) {
          double Pr, Pi;
          if constexpr (PART != 1) {
            Pr = pr[a][b];
            Pi = CPLX ? (double)pim[a][b] : 0.0;
            if (CPLX) {
              out[((long)s * L + l) * 2] = Pr;
              out[((long)s * L + l) * 2 + 1] = Pi;
            } else {
              out[(long)s * L + l] = Pr;
            }
            if constexpr (PART == 0) continue;
          } else {
            Pr = CPLX ? out[((long)s * L + l) * 2] : out[(long)s * L + l];
            Pi = CPLX ? out[((long)s * L + l) * 2 + 1] : 0.0;
          }
          const double Qr = qr[a][b], Qi = CPLX ? (double)qim[a][b] : 0.0;
          const double dr = Qr - e * Pr, di = Qi - e * Pi;
          rr += dr * dr + di * di;
          pp += Pr * Pr + Pi * Pi;
          pq += Pr * Qr + Pi * Qi;
        }
      }
    }
    for (int o = 16; o > 0; o >>= 1) {
      rr += __shfl_xor_sync(0xffffffffu, rr, o);
      pp += __shfl_xor_sync(0xffffffffu, pp, o);
      pq += __shfl_xor_sync(0xffffffffu, pq, o);
    }
    if (tl == 0) {
      red[ts + 8 * b][0] = rr;
      red[ts + 8 * b][1] = pp;
      red[ts + 8 * b][2] = pq;
    }
  }
  __syncthreads();
  if (PART != 0 && threadIdx.x < TS) {
    const int s = s0 + threadIdx.x;
    if (s < k) {
      double *P = part + (bx * k + s) * 3;
      P[0] = red[threadIdx.x][0];
      P[1] = red[threadIdx.x][1];
      P[2] = red[threadIdx.x][2];
    }
  }
}

// out[3 s + q] = the sum of the rotation's per-tile partials, one CTA per state
// (a thread's tiles in order, then a fixed tree); one thread per state walked the
// 10^4 partials of 86^3 in 3.0 ms
__global__ void __launch_bounds__(128) k_sum_rot(const double *__restrict__ part, int nblk, int k, double *__restrict__ out)
{
  const int s = blockIdx.x;
  double v[3] = {0, 0, 0};
  for (int t = threadIdx.x; t < nblk; t += blockDim.x) {
#pragma unroll
    for (int q = 0; q < 3; q++) v[q] += part[((long)t * k + s) * 3 + q];
  }
  __shared__ double w[4][3];
#pragma unroll
  for (int q = 0; q < 3; q++) {
    for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
    if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5][q] = v[q];
  }
  __syncthreads();
  if (threadIdx.x < 3) out[3 * s + threadIdx.x] = (w[0][threadIdx.x] + w[1][threadIdx.x]) + (w[2][threadIdx.x] + w[3][threadIdx.x]);
}

__global__ void k_scale_copy(const double *__restrict__ src, double *__restrict__ dst, long stlen, long k,
                             const double *__restrict__ f)
{
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < k * stlen; i += (long)gridDim.x * blockDim.x)
    dst[i] = src[i] * f[i / stlen];
}

// X[j][s] = V[j][keep[s]] / sqrt(l[keep[s]])
__global__ void k_build_x(const double2 *__restrict__ V, int n, const int *__restrict__ keep,
                          const double *__restrict__ lam, int k, double2 *__restrict__ X)
{
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < (long)n * k; e += (long)gridDim.x * blockDim.x) {
    const int j = (int)(e / k), s = (int)(e % k);
    const double f = 1.0 / sqrt(lam[s]);
    const double2 v = V[(long)j * n + keep[s]];
    X[e] = make_double2(v.x * f, v.y * f);
  }
}

__global__ void k_hermitize(double2 *A, int n)
{
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < (long)n * n; e += (long)gridDim.x * blockDim.x) {
    const int i = (int)(e / n), j = (int)(e % n);
    if (i > j) continue;
    const double2 a = A[(long)i * n + j], b = A[(long)j * n + i];
    const double2 h = make_double2(0.5 * (a.x + b.x), 0.5 * (a.y - b.y));
    A[(long)i * n + j] = h;
    A[(long)j * n + i] = make_double2(h.x, -h.y);
  }
}

// permute the columns of U (k x k): U2[:, s] = U[:, perm[s]]
__global__ void k_permute_cols(const double2 *__restrict__ U, const int *__restrict__ perm, int k,
                               double2 *__restrict__ U2)
{
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < (long)k * k; e += (long)gridDim.x * blockDim.x) {
    const int i = (int)(e / k), s = (int)(e % k);
    U2[e] = U[(long)i * k + perm[s]];
  }
}

// q[s] = sum_i conj(C[i][s]) T[i][s] (real part): the quadratic forms
// C_s^H A C_s from T = A C, for the k columns of the n x k matrix C
__global__ void k_quad_diag(const double2 *__restrict__ Cm, const double2 *__restrict__ Tm, int n, int k,
                            double *__restrict__ q)
{
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < k; s += gridDim.x * blockDim.x) {
    double v = 0;
    for (int i = 0; i < n; i++) {
      const double2 a = Cm[(long)i * k + s], b = Tm[(long)i * k + s];
      v += a.x * b.x + a.y * b.y;
    }
    q[s] = v;
  }
}

template <typename T>
static int gram_t(fbse_ctx *c, const double *A, const double *B, int n, long L, double2 *out, double scale,
                  double2 *part, int nchunk, long kchunk)
{
  auto sums = [&]() -> int {
    k_sum_partials<<<256, 256, 0, c->stream>>>(part, nchunk, (long)n * n, scale, out);
    FBSE_CHECK_LAUNCH(c);
    return FBSE_OK;
  };
  if constexpr (sizeof(T) == 8) {
    // FP64 sums run at the FP64 pipe's rate whatever the tile, so 32 x 32 tiles, which
    // give more CTAs (the same sums as 64 x 64): 10.0 -> 7.5 ms for 128 real states of 133380 points (5.4 ms of FP64 pipe).  The exact
    // products of exactgemm.cu take 0.2 ms, but their last bits differ (see the
    // caller).
    const int nt = (n + 63) / 64;
    const dim3 g(4 * nt * (nt + 1) / 2, 1, nchunk);
    if (c->is_complex) k_gram<T, true, 2, 32><<<g, 256, 0, c->stream>>>(A, B, n, L, kchunk, part);
    else k_gram<T, false, 2, 32><<<g, 256, 0, c->stream>>>(A, B, n, L, kchunk, part);
    FBSE_CHECK_LAUNCH(c);
    return sums();
  } else {
    const int nt = (n + 63) / 64;
    dim3 g(nt * (nt + 1) / 2, 1, nchunk);
    // resident CTAs per SM: one (no register cap) or two (a cap of 128
    // registers, which spills the FP32 path's float-float accumulators a
    // little); the same sums either way, so the autotuner picks by time
    auto launch = [&](long v) -> int {
      if (c->is_complex) {
        if (v == 2) k_gram<T, true, 2><<<g, 256, 0, c->stream>>>(A, B, n, L, kchunk, part);
        else k_gram<T, true, 1><<<g, 256, 0, c->stream>>>(A, B, n, L, kchunk, part);
      } else {
        if (v == 2) k_gram<T, false, 2><<<g, 256, 0, c->stream>>>(A, B, n, L, kchunk, part);
        else k_gram<T, false, 1><<<g, 256, 0, c->stream>>>(A, B, n, L, kchunk, part);
      }
      return launch_status(c);
    };
    long minb = 1;
    const std::string prob = std::string("fp32") + (c->is_complex ? " complex" : " real") +
                             " n=" + std::to_string(n) + " L=" + std::to_string(L);
    int rc = autotune(c, "gram CTAs per SM", prob, {1, 2}, launch, &minb);
    if (rc) return rc;
    if ((rc = launch(minb))) return rc;
    FBSE_COUNT(1);
    return sums();
  }
}

// default overlap cut of the mixed path, relative to the largest eigenvalue.
// Measured on the 3 nm CdSe spinor dot (256 filtered states): a cut of 1e-10
// keeps 250 pairs and matches 148 levels of the FP64 pipeline against 228 and
// 142 at 1e-6, but the extra directions are noise of the FP32 recursion and
// they leave the converged vectors less accurate (on the CsPbI3 cube the
// smallest singular value of the mixed / FP64 cluster overlaps drops from
// 1 - 4e-8 to 1 - 9e-6), so the default keeps 1e-6
constexpr double kMixedRitzCut = 1e-6;

template <typename T>
static int ortho_diag_sigma_t(fbse_ctx *c, double *psitot, long n_, long *n_kept, double *eval, double *sigma)
{
  const int n = (int)n_;
  const long len = (long)c->nspin * c->ngrid;     // points per state
  const long stlen = (long)(c->is_complex + 1) * len;
  const long L = len;                              // vector length in (complex or real) elements
  int rc = FBSE_OK;
  // scratch: HPsi (n states FP64), rotated states (n states FP64), working states
  double *hpsi = nullptr, *rot = nullptr;
  void *work = nullptr;
  double2 *G = nullptr, *M = nullptr, *V = nullptr, *X = nullptr, *Hp = nullptr, *Tm = nullptr, *U = nullptr,
          *Cm = nullptr, *part = nullptr, *G0 = nullptr;
  double *lam = nullptr, *Ed = nullptr, *rpart = nullptr, *rsum = nullptr, *fac = nullptr, *quad = nullptr;
  constexpr bool kMixed = sizeof(T) == 4;
  int *keepd = nullptr, *permd = nullptr;
  const long chunk_states = 16;
  const long nw_chunk = c->is_complex ? chunk_states : chunk_states / 2;
  const int nchunk = (int)std::min<long>(std::max<long>(1, L / 4096), 1024);
  const long kchunk = (L + nchunk - 1) / nchunk;
  const int nrb = (int)((L + 127) / 128);
  auto alloc = [&](void **p, size_t b) -> bool {
    if (dev_alloc(c, p, b) == cudaSuccess) return true;
    rc = set_err(c, FBSE_ERR_OOM, "ortho/diag scratch");
    return false;
  };
  // The Ritz vectors follow the last bits of this step's sums: close pairs by their
  // size (FP32: a change of 1e-7 in H psi moved vectors by up to 2e-3, 128 states of
  // 86^3), and every complex vector by its phase, which Jacobi takes from elements
  // that have almost vanished.  So this step keeps one set of H psi kernels and one
  // sum order whatever H psi itself uses, and with them the vectors of earlier runs.
  // It applies H once per state, the filter thousands of times.
  struct Steady {
    fbse_ctx *c;
    explicit Steady(fbse_ctx *c_) : c(c_) { c->steady = 1; }
    ~Steady() { c->steady = 0; }
  } steady(c);
  do {
    {
      void *a = nullptr, *b = nullptr;
      if (cached(c, kSlotHpsi, (size_t)n * stlen * sizeof(double), &a) ||
          cached(c, kSlotRot, (size_t)n * stlen * sizeof(double), &b)) { rc = FBSE_ERR_OOM; break; }
      hpsi = (double *)a;
      rot = (double *)b;
    }
    // the mixed path applies H in FP32 here unless told otherwise (FP64 H psi
    // measured no better on the 3 nm dot: the FP32 recursion's noise in the
    // filtered states, not the operator, limits the projected problem)
    const bool h64 = kMixed && c->tune.ritz_hpsi == 2;
    if (!alloc(&work, (size_t)2 * nw_chunk * len * (h64 ? sizeof(double2) : sizeof(C<T>)))) break;
    const size_t nn = (size_t)n * n;
    if (!alloc((void **)&G, nn * sizeof(double2)) || !alloc((void **)&M, nn * sizeof(double2)) ||
        !alloc((void **)&V, nn * sizeof(double2)) || !alloc((void **)&X, nn * sizeof(double2)) ||
        !alloc((void **)&Hp, nn * sizeof(double2)) || !alloc((void **)&Tm, nn * sizeof(double2)) ||
        !alloc((void **)&U, nn * sizeof(double2)) || !alloc((void **)&Cm, nn * sizeof(double2)) ||
        !alloc((void **)&part, (size_t)nchunk * nn * sizeof(double2)) || !alloc((void **)&lam, n * sizeof(double)) ||
        !alloc((void **)&Ed, n * sizeof(double)) || !alloc((void **)&rpart, (size_t)nrb * n * 3 * sizeof(double)) ||
        !alloc((void **)&rsum, (size_t)n * 3 * sizeof(double)) || !alloc((void **)&fac, n * sizeof(double)) ||
        !alloc((void **)&keepd, n * sizeof(int)) || !alloc((void **)&permd, n * sizeof(int)) ||
        !alloc((void **)&G0, nn * sizeof(double2)) || !alloc((void **)&quad, 2 * (size_t)n * sizeof(double)))
      break;
    // 1. HPsi in chunks of working states
    for (long s0 = 0; s0 < n && !rc; s0 += chunk_states) {
      const long ns = std::min<long>(chunk_states, n - s0);
      const long nw = c->is_complex ? ns : (ns + 1) / 2;
      if (h64) {
        double2 *w0 = reinterpret_cast<double2 *>(work), *w1 = w0 + nw_chunk * len;
        if ((rc = pack<double>(c, psitot + s0 * stlen, w0, ns))) break;
        if ((rc = hpsi_apply<double>(c, w0, w1, nw, 1.0, 0.0))) break;
        if ((rc = unpack<double>(c, w1, hpsi + s0 * stlen, ns))) break;
      } else {
        C<T> *w0 = reinterpret_cast<C<T> *>(work), *w1 = w0 + nw_chunk * len;
        if ((rc = pack<T>(c, psitot + s0 * stlen, w0, ns))) break;
        if ((rc = hpsi_apply<T>(c, w0, w1, nw, 1.0, 0.0))) break;
        if ((rc = unpack<T>(c, w1, hpsi + s0 * stlen, ns))) break;
      }
    }
    if (rc) break;
    // 2. Gram and projected H (dv-weighted)
    if ((rc = gram_t<T>(c, psitot, psitot, n, L, G, c->dv, part, nchunk, kchunk))) break;
    if ((rc = gram_t<T>(c, psitot, hpsi, n, L, M, c->dv, part, nchunk, kchunk))) break;
    FBSE_COUNT(2); k_hermitize<<<64, 256, 0, c->stream>>>(G, n);
    k_hermitize<<<64, 256, 0, c->stream>>>(M, n);
    if (cudaMemcpyAsync(G0, G, nn * sizeof(double2), cudaMemcpyDeviceToDevice, c->stream) != cudaSuccess) {
      rc = set_err(c, FBSE_ERR_CUDA, "overlap copy");
      break;
    }
    // 3. overlap eigen-decomposition
    std::vector<double> w;
    if ((rc = jacobi_eig_dev(c, G, V, n, w, !c->is_complex))) break;
    // 4. rank cutoff (ortho.c:68-75 keeps s_i/s_0 >= 1e-10); the overlap
    //    resolves l_i / l_max to the precision of its products and of the
    //    states (fbse_tuning.ritz_cut overrides the default)
    double lmax = 0;
    for (double v : w) lmax = std::max(lmax, v);
    const double cut = lmax * (c->tune.ritz_cut > 0 ? c->tune.ritz_cut : (kMixed ? kMixedRitzCut : 1e-12));
    std::vector<int> keep;
    std::vector<int> order(n);
    std::iota(order.begin(), order.end(), 0);
    std::sort(order.begin(), order.end(), [&](int a, int b) { return w[a] > w[b]; });
    for (int i : order)
      if (w[i] > cut && w[i] >= lmax * 1e-20) keep.push_back(i);
    const int k = (int)keep.size();
    *n_kept = k;
    if (k == 0) { rc = set_err(c, FBSE_ERR_NAN, "orthogonalisation kept no states"); break; }
    std::vector<double> lk(k);
    for (int s = 0; s < k; s++) lk[s] = w[keep[s]];
    if (h2d(c->stream, keepd, keep.data(), k * sizeof(int)) != cudaSuccess ||
        h2d(c->stream, lam, lk.data(), k * sizeof(double)) != cudaSuccess) {
      rc = set_err(c, FBSE_ERR_CUDA, "orthogonalisation: basis upload");
      break;
    }
    FBSE_COUNT(1); k_build_x<<<64, 256, 0, c->stream>>>(V, n, keepd, lam, k, X);
    // 5. H' = X^H M X  (k x k), Hermitian eigen-decomposition
    if ((rc = zgemm_dev(c, n, k, n, M, n, false, X, k, false, Tm, k))) break;   // Tm = M X   (n x k)
    if ((rc = zgemm_dev(c, k, k, n, X, k, true, Tm, k, false, Hp, k))) break;  // Hp = X^H Tm (k x k)
    FBSE_COUNT(1); k_hermitize<<<64, 256, 0, c->stream>>>(Hp, k);
    std::vector<double> e;
    if ((rc = jacobi_eig_dev(c, Hp, U, k, e, !c->is_complex))) break;
    std::vector<int> perm(k);
    std::iota(perm.begin(), perm.end(), 0);
    std::sort(perm.begin(), perm.end(), [&](int a, int b) { return e[a] < e[b]; });
    std::vector<double> es(k);
    for (int s = 0; s < k; s++) es[s] = e[perm[s]];
    if (h2d(c->stream, permd, perm.data(), k * sizeof(int)) != cudaSuccess ||
        h2d(c->stream, Ed, es.data(), k * sizeof(double)) != cudaSuccess) {
      rc = set_err(c, FBSE_ERR_CUDA, "diagonalisation: eigenvalue upload");
      break;
    }
    FBSE_COUNT(1); k_permute_cols<<<64, 256, 0, c->stream>>>(U, permd, k, Tm);
    // 6. C = X U  (n x k); rotate Psi and HPsi with the residual epilogue
    if ((rc = zgemm_dev(c, n, k, k, X, k, false, Tm, k, false, Cm, k))) break;
    if constexpr (kMixed) {
      // the Rayleigh quotients of the exact combinations Psi C from the FP64
      // small matrices: (C^H M C)_ss / (C^H G C)_ss (X and Hp are free now)
      if ((rc = zgemm_dev(c, n, k, n, M, n, false, Cm, k, false, X, k))) break;
      if ((rc = zgemm_dev(c, n, k, n, G0, n, false, Cm, k, false, Hp, k))) break;
      FBSE_COUNT(2);
      k_quad_diag<<<(k + 127) / 128, 128, 0, c->stream>>>(Cm, X, n, k, quad);
      k_quad_diag<<<(k + 127) / 128, 128, 0, c->stream>>>(Cm, Hp, n, k, quad + n);
    }
    const dim3 gr((unsigned)(nrb * ((k + 31) / 32)));
    if constexpr (sizeof(T) == 4) {  // FP32: two half-register launches (Psi, then H Psi + residuals)
      if (c->is_complex) {
        k_rotate<T, true, 0><<<gr, 256, 0, c->stream>>>(psitot, hpsi, n, L, Cm, k, Ed, rot, rpart);
        k_rotate<T, true, 1><<<gr, 256, 0, c->stream>>>(psitot, hpsi, n, L, Cm, k, Ed, rot, rpart);
      } else {
        k_rotate<T, false, 0><<<gr, 256, 0, c->stream>>>(psitot, hpsi, n, L, Cm, k, Ed, rot, rpart);
        k_rotate<T, false, 1><<<gr, 256, 0, c->stream>>>(psitot, hpsi, n, L, Cm, k, Ed, rot, rpart);
      }
      FBSE_COUNT(1);
    } else {
      if (c->is_complex) k_rotate<T, true, 2><<<gr, 256, 0, c->stream>>>(psitot, hpsi, n, L, Cm, k, Ed, rot, rpart);
      else k_rotate<T, false, 2><<<gr, 256, 0, c->stream>>>(psitot, hpsi, n, L, Cm, k, Ed, rot, rpart);
    }
    FBSE_LAUNCH_OR_BREAK(c, rc);
    FBSE_COUNT(1); k_sum_rot<<<k, 128, 0, c->stream>>>(rpart, nrb, k, rsum);
    std::vector<double> hs(3 * k), hq(2 * (size_t)n);
    if (cudaMemcpyAsync(hs.data(), rsum, 3 * k * sizeof(double), cudaMemcpyDeviceToHost, c->stream) != cudaSuccess ||
        (kMixed && cudaMemcpyAsync(hq.data(), quad, 2 * (size_t)n * sizeof(double), cudaMemcpyDeviceToHost,
                                   c->stream) != cudaSuccess) ||
        cudaStreamSynchronize(c->stream) != cudaSuccess) { rc = set_err(c, FBSE_ERR_CUDA, "rotation"); break; }
    // 7. normalise; report the Rayleigh quotient rho = <psi|H psi>/<psi|psi> of
    //    the returned state and sigma = ||(H - rho) psi|| / ||psi||.  rho differs
    //    from the Ritz value E by the basis' departure from orthonormality
    //    (X^H G X = I up to eps * cond(G)); for the reference's SVD basis the
    //    two agree, so rho is the closer match to its eig_vals and is what
    //    calc_sigma_E reports for the state.  With r = ||(H - E) psi||^2:
    //    ||(H - rho) psi||^2 = r - (rho - E)^2 ||psi||^2.  The mixed path
    //    takes rho from the FP64 small matrices (the FP32 rotation loses
    //    digits where C is large, on near-dependent filtered states) and
    //    sigma from the rotated states.
    std::vector<double> f(k);
    for (int s = 0; s < k; s++) {
      const double pp = hs[3 * s + 1];
      const double nrm = pp * c->dv;
      if (!(nrm > 0)) { rc = set_err(c, FBSE_ERR_NAN, "Norm is 0/NAN after diagonalisation"); break; }
      f[s] = 1.0 / std::sqrt(nrm);
      const double rho = kMixed ? hq[s] / hq[n + s] : hs[3 * s + 2] / pp;
      const double d = rho - es[s];
      eval[s] = rho;
      sigma[s] = std::sqrt(std::fabs(hs[3 * s] / pp - d * d));
    }
    if (rc) break;
    if (h2d(c->stream, fac, f.data(), k * sizeof(double)) != cudaSuccess) {
      rc = set_err(c, FBSE_ERR_CUDA, "normalisation: factor upload");
      break;
    }
    k_scale_copy<<<4096, 256, 0, c->stream>>>(rot, psitot, stlen, k, fac);
    FBSE_LAUNCH_OR_BREAK(c, rc);
    if (cudaStreamSynchronize(c->stream) != cudaSuccess) rc = set_err(c, FBSE_ERR_CUDA, "ortho/diag/sigma");
  } while (0);
  cudaStreamSynchronize(c->stream);
  void *bufs[] = {work, G, M, V, X, Hp, Tm, U, Cm, part, lam, Ed, rpart, rsum, fac, keepd, permd, G0, quad};
  for (void *b : bufs)
    if (b) cudaFree(b);
  return rc;
}

// ---------------------------------------------------------------------------
// general FP64 products over a slab of points [off, off + len) of each state:
//   gram:   out[i][j] = dv sum_l conj(A_i[l]) B_j[l]          (na x nb)
//   rotate: out_j[l] = sum_i C[i][j] A_i[l]                   (k states)
// A, B, out: psitot rows (stlen doubles; complex states are (re, im) pairs,
// l counts complex values then).  64 x 64 output tile per CTA for the Gram,
// FP64 split-K partials summed in order.
// ---------------------------------------------------------------------------
template <bool CPLX>
__global__ void __launch_bounds__(256) k_gram_slab(const double *__restrict__ A, long na, const double *__restrict__ B,
                                                   long nb, long stride, long off, long len, long kchunk,
                                                   double2 *__restrict__ part)
{
  constexpr int TM = 64, TK = 16;
  __shared__ double2 As[TK][TM + 1], Bs[TK][TM + 1];
  const long i0 = (long)blockIdx.x * TM, j0 = (long)blockIdx.y * TM;
  const long k0 = off + blockIdx.z * kchunk, k1 = min(off + len, k0 + kchunk);
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  double ar_[4][4] = {}, ai_[4][4] = {};
  for (long kb = k0; kb < k1; kb += TK) {
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int r = ty + 16 * q;
      const long k = kb + tx;
      double2 va = make_double2(0, 0), vb = make_double2(0, 0);
      if (i0 + r < na && k < k1) va = CPLX ? reinterpret_cast<const double2 *>(A + (i0 + r) * stride)[k]
                                           : make_double2(A[(i0 + r) * stride + k], 0.0);
      if (j0 + r < nb && k < k1) vb = CPLX ? reinterpret_cast<const double2 *>(B + (j0 + r) * stride)[k]
                                           : make_double2(B[(j0 + r) * stride + k], 0.0);
      As[tx][r] = va;
      Bs[tx][r] = vb;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < TK; kk++)
#pragma unroll
      for (int a = 0; a < 4; a++) {
        const double2 u = As[kk][ty + 16 * a];
#pragma unroll
        for (int b = 0; b < 4; b++) {
          const double2 v = Bs[kk][tx + 16 * b];
          ar_[a][b] += u.x * v.x + u.y * v.y;
          ai_[a][b] += u.x * v.y - u.y * v.x;
        }
      }
    __syncthreads();
  }
  double2 *P = part + (long)blockIdx.z * na * nb;
#pragma unroll
  for (int a = 0; a < 4; a++)
#pragma unroll
    for (int b = 0; b < 4; b++) {
      const long i = i0 + ty + 16 * a, j = j0 + tx + 16 * b;
      if (i < na && j < nb) P[i * nb + j] = make_double2(ar_[a][b], ai_[a][b]);
    }
}

template <bool CPLX>
__global__ void k_rotate_slab(const double *__restrict__ A, long na, const double2 *__restrict__ Cm, long k,
                              long stride, long off, long len, double *__restrict__ out)
{
  const long total = k * len;
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < total; e += (long)gridDim.x * blockDim.x) {
    const long j = e / len, l = off + e % len;
    double re = 0, im = 0;
    for (long i = 0; i < na; i++) {
      const double2 cc = Cm[i * k + j];
      if (CPLX) {
        const double2 a = reinterpret_cast<const double2 *>(A + i * stride)[l];
        re += cc.x * a.x - cc.y * a.y;
        im += cc.x * a.y + cc.y * a.x;
      } else {
        re += cc.x * A[i * stride + l];
      }
    }
    if (CPLX) reinterpret_cast<double2 *>(out + j * stride)[l] = make_double2(re, im);
    else out[j * stride + l] = re;
  }
}

int gram_slab(fbse_ctx *c, const double *A, long na, const double *B, long nb, long off, long len, double *out_host)
{
  const long L = (long)c->nspin * c->ngrid;
  const long stride = (long)(c->is_complex + 1) * L;
  if (na < 1 || nb < 1 || off < 0 || len < 1 || off + len > L || na > 65535 * 64L || nb > 65535 * 64L)
    return set_err(c, FBSE_ERR_ARG, "fbse_gram: sizes");
  if (len >= kExactMin && na <= 65535 && nb <= 65535 && !c->tc_poisoned) {
    const int w = c->is_complex + 1;
    // the result in the product's own scratch: a captured graph may hold the addresses of
    // the context's other buffers
    const int rx = exact_nt(c, A + off * w, stride, (int)na, B + off * w, stride, (int)nb, len,
                            c->is_complex ? kExactConj : kExactReal, c->dv, nullptr, out_host);
    if (rx != FBSE_ERR_OOM) return rx;
  }
  const int nchunk = (int)std::min<long>(std::max<long>(1, len / 8192), 256);
  const long kchunk = (len + nchunk - 1) / nchunk;
  double2 *part = nullptr, *sum = nullptr;
  if (dev_alloc(c, &part, (size_t)nchunk * na * nb * sizeof(double2)) != cudaSuccess ||
      dev_alloc(c, &sum, (size_t)na * nb * sizeof(double2)) != cudaSuccess) {
    cudaGetLastError();
    if (part) cudaFree(part);
    return set_err(c, FBSE_ERR_OOM, "fbse_gram: scratch");
  }
  int rc = FBSE_OK;
  do {
    dim3 g((unsigned)((na + 63) / 64), (unsigned)((nb + 63) / 64), (unsigned)nchunk);
    if (c->is_complex) k_gram_slab<true><<<g, 256, 0, c->stream>>>(A, na, B, nb, stride, off, len, kchunk, part);
    else k_gram_slab<false><<<g, 256, 0, c->stream>>>(A, na, B, nb, stride, off, len, kchunk, part);
    FBSE_LAUNCH_OR_BREAK(c, rc);
    k_sum_partials<<<256, 256, 0, c->stream>>>(part, nchunk, na * nb, c->dv, sum);
    FBSE_LAUNCH_OR_BREAK(c, rc);
    if (d2h(c->stream, out_host, sum, (size_t)na * nb * sizeof(double2)) != cudaSuccess)
      rc = set_err(c, FBSE_ERR_CUDA, "fbse_gram: download");
  } while (0);
  cudaStreamSynchronize(c->stream);
  cudaFree(part);
  cudaFree(sum);
  return rc;
}

int rotate_slab(fbse_ctx *c, const double *A, long na, const double *C_host, long k, long off, long len, double *out)
{
  const long L = (long)c->nspin * c->ngrid;
  const long stride = (long)(c->is_complex + 1) * L;
  if (na < 1 || k < 1 || off < 0 || len < 1 || off + len > L) return set_err(c, FBSE_ERR_ARG, "fbse_rotate: sizes");
  double2 *Cd = nullptr;
  if (dev_alloc(c, &Cd, (size_t)na * k * sizeof(double2)) != cudaSuccess) {
    cudaGetLastError();
    return set_err(c, FBSE_ERR_OOM, "fbse_rotate: coefficients");
  }
  int rc = FBSE_OK;
  do {
    if (h2d(c->stream, Cd, C_host, (size_t)na * k * sizeof(double2)) != cudaSuccess) {
      rc = set_err(c, FBSE_ERR_CUDA, "fbse_rotate: upload");
      break;
    }
    const long total = k * len;
    const unsigned g = (unsigned)std::min<long>((total + 255) / 256, 152L * 64);
    if (c->is_complex) k_rotate_slab<true><<<g, 256, 0, c->stream>>>(A, na, Cd, k, stride, off, len, out);
    else k_rotate_slab<false><<<g, 256, 0, c->stream>>>(A, na, Cd, k, stride, off, len, out);
    FBSE_LAUNCH_OR_BREAK(c, rc);
    if (cudaStreamSynchronize(c->stream) != cudaSuccess) rc = set_err(c, FBSE_ERR_CUDA, "fbse_rotate");
  } while (0);
  cudaFree(Cd);
  return rc;
}

int ortho_diag_sigma(fbse_ctx *c, double *psitot, long n, long *n_kept, double *eval, double *sigma)
{
  if (n > 8192) return set_err(c, FBSE_ERR_UNSUPPORTED, "more than 8192 states in one subspace");
  return c->precision == FBSE_MIXED ? ortho_diag_sigma_t<float>(c, psitot, n, n_kept, eval, sigma)
                                    : ortho_diag_sigma_t<double>(c, psitot, n, n_kept, eval, sigma);
}

}  // namespace fbse
