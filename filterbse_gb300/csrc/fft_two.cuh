// Two-factor FFT kernels for axis lengths n = P Q, P <= 16 a radix that a
// thread transforms in registers (fft_radix.cuh) and Q one such radix up to 31,
// or any odd number of 27 .. 255 (stage_sym): the reference's grid rule gives
// every even length, so factors 2 x 43 or 4 x 37 are as common as smooth ones.
//
// Decomposition (input n = t + P m, output k = k1 + Q k2):
//   X[k1 + Q k2] = sum_t w_P^{t k2} [ w_n^{t k1} sum_m x[t + P m] w_Q^{m k1} ]
// Stage A transforms the Q values at positions t + P m and leaves Y_t[k1],
// already times w_n^{t k1}, at positions t + P k1; stage B transforms the P
// values at positions P k1 .. P k1 + P - 1.  Both stages are in place, and the
// twiddle of position p is tw[p] in both directions.  The result for k = k1 + Q k2
// stays at position k2 + P k1: every pass between the forward and the inverse
// transform of an axis is pointwise in that axis, so x and y keep this order
// (AxisPlan::ord maps a position to its k, AxisPlan::k2o is the kinetic table in
// it) and no pass reorders.  The inverse runs the stages backwards (B with the
// twiddles, then A), as a forward transform of exchanged real and imaginary parts.
//
// A stage's work items are (butterfly, line) pairs with the line fastest, so the
// lanes of a warp take consecutive lines (one broadcast twiddle, coalesced or
// conflict-free accesses) and no lane idles when the line count is not a
// multiple of 32.
//
// Why: the one-radix-per-pass Stockham kernels (fft.cu) spend 3-4 shared-memory
// round trips and an integer division per element on such lengths, and lengths
// with a prime above 8 take a direct sum per output.  Measured, H psi through
// those kernels -> these:
//   116 x 117 x 120, 4 spinors, FP32 (memory and latency bound)  2101 -> 360 us
//   96^3, 4 spinors, FP32 (127 terms of a filter)                  742 -> 161 us
//   96^3, 6 spinors, FP64 (FP64 pipe bound; projectors 1.6 ms)     5131 -> 3794 us
//   57 x 52 x 45, 8 packed states, FP64 (radices 13, 19)           1911 -> 477 us
#pragma once

#include <algorithm>
#include <type_traits>

#include "fft_radix.cuh"

namespace fbse {
namespace two {

// x / d for x * d < 2^32
struct Div {
  unsigned d, m;
  __host__ __device__ explicit Div(unsigned d_ = 1) : d(d_), m((unsigned)(0xffffffffu / d_) + 1u) {}
  __device__ __forceinline__ unsigned operator()(unsigned x) const { return d == 1 ? x : __umulhi(x, m); }
};

template <typename T> struct Axis {
  int n, P, Q;
  const C<T> *tw;   // tw[t + P k1] = w_n^{t k1}
  const C<T> *sym;  // stage_sym's coefficients when Q is transformed there, else null
};

// calls f(integral_constant<R>) for the run-time radix r.  BIG: the set with the
// radices above 16 (kernels with BIG also hold stage_sym)
template <bool BIG, typename F> __device__ __forceinline__ void with_radix(int r, F f)
{
#define FBSE_R(R) \
  case R: f(std::integral_constant<int, R>{}); break;
  switch (r) {
    FBSE_R(1) FBSE_R(2) FBSE_R(3) FBSE_R(4) FBSE_R(5) FBSE_R(6) FBSE_R(7) FBSE_R(8) FBSE_R(9) FBSE_R(10) FBSE_R(11)
    FBSE_R(12) FBSE_R(13) FBSE_R(14) FBSE_R(15) FBSE_R(16)
    default:
      if constexpr (BIG) {
        switch (r) {
          FBSE_R(17) FBSE_R(18) FBSE_R(19) FBSE_R(20) FBSE_R(21) FBSE_R(23) FBSE_R(24) FBSE_R(25) FBSE_R(29)
          FBSE_R(31)
        }
      }
  }
#undef FBSE_R
}

template <typename T> __device__ __forceinline__ C<T> exch(C<T> v) { return mk<T>(v.y, v.x); }

// one stage over L lines: butterflies j < nb at positions first(j) + step i,
// i < R.  ld(line, position) and st(line, position, value); TW: multiply by
// tw[position] before the store
template <typename T, bool BIG, bool TW, typename Ld, typename St>
__device__ __forceinline__ void stage(int R, int nb, int mul, int step, const Div &lines, const C<T> *__restrict__ tw,
                                      Ld ld, St st)
{
  with_radix<BIG>(R, [&](auto rc) {
    constexpr int RR = decltype(rc)::value;
    const unsigned items = (unsigned)nb * lines.d;
    for (unsigned it = threadIdx.x; it < items; it += blockDim.x) {
      const unsigned j = lines(it);
      const int c = (int)(it - j * lines.d), p0 = (int)j * mul;
      C<T> v[RR];
#pragma unroll
      for (int i = 0; i < RR; i++) v[i] = ld(c, p0 + i * step);
      dft<T, RR>(v);
#pragma unroll
      for (int i = 0; i < RR; i++) {
        if (TW && i > 0) v[i] = cmul<T>(v[i], __ldg(tw + p0 + i * step));
        st(c, p0 + i * step, v[i]);
      }
    }
  });
}
// stage A for an odd Q too large for a thread's registers: P butterflies of Q
// values, each shared by the threads of its row blocks.  With a_r = x_r + x_{Q-r}
// and b_r = x_r - x_{Q-r} (formed in place first), row q of the block sums
// e_q = x_0 + sum_r cos a_r and o_q = sum_r sin b_r, which give X_q and X_{Q-q}:
// Q multiply-adds per value, the quarter of a direct sum.  kSymRows rows per
// thread share each a_r, b_r, and kSymLines lines share each coefficient (FP32,
// where the loads and not the FP32 pipe bound the sums); the lanes of a warp take
// consecutive lines, so the coefficients are broadcasts.  A group of lines keeps
// its sums in registers until every thread has read the group's values, so the
// stage is in place.
// H psi without projectors, FP32, 8 states: 86^3 307 us, 118^3 800 us (the loads of
// the coefficients bound it: two lines a thread measured 342 and 861 us with one,
// and 362 and 939 us with the next coefficients fetched ahead); FP64, 4 states of
// 86^3: 2212 us, 60% of the FP64 pipe.  The direct sums took 4 times as long.
template <typename T> constexpr int kSymLines = sizeof(T) == 4 ? 2 : 1;

// a row block's coefficients of one r, 16 bytes a load
__device__ __forceinline__ void ld_coef(const float2 *w, float2 (&cs)[kSymRows])
{
  const float4 *v = reinterpret_cast<const float4 *>(w);
#pragma unroll
  for (int i = 0; i < kSymRows / 2; i++) {
    const float4 q = __ldg(v + i);
    cs[2 * i] = make_float2(q.x, q.y);
    cs[2 * i + 1] = make_float2(q.z, q.w);
  }
}
__device__ __forceinline__ void ld_coef(const double2 *w, double2 (&cs)[kSymRows])
{
#pragma unroll
  for (int i = 0; i < kSymRows; i++) cs[i] = __ldg(w + i);
}

template <typename T, bool TW, typename Ld, typename At, typename St>
__device__ __forceinline__ void stage_sym(const Axis<T> &a, const Div &lines, Ld ld, At at, St st)
{
  const int P = a.P, Q = a.Q, H = Q >> 1, nqb = (H + kSymRows) / kSymRows, L = (int)lines.d;
  const Div dp((unsigned)P);
  for (unsigned it = threadIdx.x; it < (unsigned)((H + 1) * P * L); it += blockDim.x) {
    const unsigned j = lines(it), r = dp(j);
    const int c = (int)(it - j * L), t = (int)(j - r * P);
    const C<T> x = ld(c, t + P * (int)r);
    if (r == 0) {
      at(c, t) = x;
    } else {
      const C<T> y = ld(c, t + P * (Q - (int)r));
      at(c, t + P * (int)r) = cadd<T>(x, y);
      at(c, t + P * (Q - (int)r)) = csub<T>(x, y);
    }
  }
  __syncthreads();
  // a thread's lines: c and c + half of its group
  const int per = P * nqb, Lg = kSymLines<T> * ((int)blockDim.x / per);  // the launch gives at least per threads
  for (int l0 = 0; l0 < L; l0 += Lg) {
    const int nl = min(Lg, L - l0), half = (nl + kSymLines<T> - 1) / kSymLines<T>;
    const int j = (int)threadIdx.x / half, k = (int)threadIdx.x % half;
    const int qb = (int)dp((unsigned)j), t = j - qb * P;
    int c[kSymLines<T>];
    bool act[kSymLines<T>];
#pragma unroll
    for (int u = 0; u < kSymLines<T>; u++) {
      act[u] = j < per && k + u * half < nl;
      c[u] = l0 + (act[u] ? k + u * half : k);
    }
    C<T> e[kSymLines<T>][kSymRows], o[kSymLines<T>][kSymRows];
    if (act[0]) {
#pragma unroll
      for (int u = 0; u < kSymLines<T>; u++) {
        const C<T> x0 = at(c[u], t);
#pragma unroll
        for (int i = 0; i < kSymRows; i++) {
          e[u][i] = x0;
          o[u][i] = mk<T>(T(0), T(0));
        }
      }
      const C<T> *w = a.sym + (long)qb * kSymRows;
      for (int r = 1; r <= H; r++, w += (long)nqb * kSymRows) {
        C<T> cs[kSymRows];
        ld_coef(w, cs);
#pragma unroll
        for (int u = 0; u < kSymLines<T>; u++) {
          const C<T> s = at(c[u], t + P * r), d = at(c[u], t + P * (Q - r));
#pragma unroll
          for (int i = 0; i < kSymRows; i++) {
            e[u][i].x += cs[i].x * s.x;
            e[u][i].y += cs[i].x * s.y;
            o[u][i].x += cs[i].y * d.x;
            o[u][i].y += cs[i].y * d.y;
          }
        }
      }
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kSymLines<T>; u++) {
      if (!act[u]) continue;
#pragma unroll
      for (int i = 0; i < kSymRows; i++) {
        const int q = qb * kSymRows + i;
        if (q > H) break;
        if (q == 0) {
          st(c[u], t, e[u][i]);
          continue;
        }
        const int p0 = t + P * q, p1 = t + P * (Q - q);
        C<T> v0 = mk<T>(e[u][i].x + o[u][i].y, e[u][i].y - o[u][i].x);
        C<T> v1 = mk<T>(e[u][i].x - o[u][i].y, e[u][i].y + o[u][i].x);
        if (TW) {
          v0 = cmul<T>(v0, __ldg(a.tw + p0));
          v1 = cmul<T>(v1, __ldg(a.tw + p1));
        }
        st(c[u], p0, v0);
        st(c[u], p1, v1);
      }
    }
  }
}

// stage A: P butterflies of Q values; stage B: Q butterflies of P values.
// at(line, position): the values' place in shared memory
template <typename T, bool BIG, bool TW, typename Ld, typename At, typename St>
__device__ __forceinline__ void stage_a(const Axis<T> &a, const Div &lines, Ld ld, At at, St st)
{
  if constexpr (BIG) {
    if (a.sym) {
      stage_sym<T, TW>(a, lines, ld, at, st);
      return;
    }
  }
  stage<T, BIG, TW>(a.Q, a.P, 1, a.P, lines, a.tw, ld, st);
}
template <typename T, bool TW, typename Ld, typename St>
__device__ __forceinline__ void stage_b(const Axis<T> &a, const Div &lines, Ld ld, St st)
{
  stage<T, false, TW>(a.P, a.Q, a.P, 1, lines, a.tw, ld, st);
}

__device__ __forceinline__ void copy_async(float2 *dst, const float2 *src)
{
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ void copy_async(double2 *dst, const double2 *src)
{
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// out = ca (r + V phi) + cb phi
template <typename T>
__device__ __forceinline__ C<T> epilogue(C<T> r, C<T> ph, const T *__restrict__ pot, long g, T ca, T cb)
{
  if (pot) {
    const T V = pot[g];
    r.x += V * ph.x;
    r.y += V * ph.y;
  }
  return mk<T>(ca * r.x + cb * ph.x, ca * r.y + cb * ph.y);
}

// ---------------------------------------------------------------------------
// plane pass: one xy plane per CTA in shared memory (row stride nx | 1: lanes on
// consecutive x or consecutive y are free of bank conflicts).
//   INV false: y forward (its first stage reads the plane from global memory,
//   lanes along x), x forward, store
//   INV true: load, x inverse, y inverse; the last y stage holds final values
//   with lanes along x and writes out = ca (r + V phi) + cb phi itself
// Registers: 64 (FP32, up to 1024 threads a CTA) / 128 (FP64, up to 512) keep two
// or more CTAs of a 100 x 100 plane on an SM, whose phases then overlap.
// ---------------------------------------------------------------------------
template <typename T, bool BIG> struct PlaneShape {
  static constexpr int threads = (sizeof(T) == 4 ? 1024 : 512) / (BIG ? 2 : 1);
};

template <typename T, bool BIG, bool INV>
__global__ void __launch_bounds__(PlaneShape<T, BIG>::threads, 1)
    k_two_plane(const C<T> *__restrict__ in, C<T> *__restrict__ out, Axis<T> ax, Axis<T> ay, Div dx, Div dy,
                const C<T> *__restrict__ phi, const T *__restrict__ pot, long ngrid, T ca, T cb)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C<T> *S = reinterpret_cast<C<T> *>(smem_raw);
  const int nx = ax.n, pitch = nx | 1;
  const unsigned npl = (unsigned)nx * ay.n;
  const long base = (long)blockIdx.x * npl;
  auto ycol = [&](int x, int y) -> C<T> & { return S[y * pitch + x]; };
  auto xrow = [&](int y, int x) -> C<T> & { return S[y * pitch + x]; };
  auto ldy = [&](int x, int y) { return ycol(x, y); };
  auto sty = [&](int x, int y, C<T> v) { ycol(x, y) = v; };
  auto ldx = [&](int y, int x) { return xrow(y, x); };
  auto stx = [&](int y, int x, C<T> v) { xrow(y, x) = v; };
  if constexpr (!INV) {
    const C<T> *src = in + base;
    stage_a<T, BIG, true>(ay, dx, [&](int x, int y) { return src[y * nx + x]; }, ycol, sty);
    __syncthreads();
    stage_b<T, false>(ay, dx, ldy, sty);
    __syncthreads();
    stage_a<T, BIG, true>(ax, dy, ldx, xrow, stx);
    __syncthreads();
    stage_b<T, false>(ax, dy, ldx, stx);
    __syncthreads();
    C<T> *dst = out + base;
#pragma unroll 4
    for (unsigned i = threadIdx.x; i < npl; i += blockDim.x) {
      const unsigned y = dx(i);
      dst[i] = S[i + y * (pitch - nx)];
    }
  } else {
    const C<T> *src = in + base;
    for (unsigned i = threadIdx.x; i < npl; i += blockDim.x) {
      const unsigned y = dx(i);
      copy_async(S + i + y * (pitch - nx), src + i);
    }
    copy_wait();
    __syncthreads();
    stage_b<T, true>(ax, dy, [&](int y, int x) { return exch<T>(xrow(y, x)); }, stx);
    __syncthreads();
    stage_a<T, BIG, false>(ax, dy, ldx, xrow, stx);
    __syncthreads();
    stage_b<T, true>(ay, dx, ldy, sty);
    __syncthreads();
    const C<T> *ph = phi + base;
    const T *V = pot ? pot + base % ngrid : nullptr;
    C<T> *dst = out + base;
    stage_a<T, BIG, false>(ay, dx, ldy, ycol, [&](int x, int y, C<T> v) {
      const int o = y * nx + x;
      dst[o] = epilogue<T>(exch<T>(v), ph[o], V, o, ca, cb);
    });
  }
}

// ---------------------------------------------------------------------------
// line kernels: tiles of up to L lines in shared memory
// ---------------------------------------------------------------------------
template <typename T, bool BIG> struct LineShape {
  static constexpr int threads = BIG ? 256 : 512;
  static constexpr int ctas = sizeof(T) == 4 ? 2 : 1;
};

// z: forward, times the kinetic factor (or the k-space array ka.kq), inverse.
// A tile is L consecutive points of the flattened xy plane, whatever nx is.
template <typename T, bool BIG>
__global__ void __launch_bounds__(LineShape<T, BIG>::threads, LineShape<T, BIG>::ctas)
    k_two_z(C<T> *__restrict__ data, Axis<T> az, int L, int ntile, long ngrid, KinArgs ka)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C<T> *S = reinterpret_cast<C<T> *>(smem_raw);
  const long blk = blockIdx.x / ntile;
  const int c0 = (int)(blockIdx.x - blk * ntile) * L;
  const int nl = min(L, (int)ka.nxy - c0);
  const Div lines((unsigned)nl);
  const long es = ka.nxy;
  C<T> *d = data + blk * ngrid + c0;
  auto at = [&](int c, int z) -> C<T> & { return S[z * L + c]; };
  auto lds = [&](int c, int z) { return S[z * L + c]; };
  auto sts = [&](int c, int z, C<T> v) { S[z * L + c] = v; };
  stage_a<T, BIG, true>(az, lines, [&](int c, int z) { return d[z * es + c]; }, at, sts);
  __syncthreads();
  with_radix<false>(az.P, [&](auto rc) {
    constexpr int RR = decltype(rc)::value;
    const unsigned items = (unsigned)(az.Q * nl);
    for (unsigned it = threadIdx.x; it < items; it += blockDim.x) {
      const unsigned k1 = lines(it);
      const int c = (int)(it - k1 * nl);
      C<T> *s = S + (int)k1 * RR * L + c;
      C<T> v[RR];
#pragma unroll
      for (int i = 0; i < RR; i++) v[i] = s[i * L];
      dft<T, RR>(v);
      const int g = c0 + c, y = g / (int)ka.nx, x = g - y * (int)ka.nx;
      if (ka.kq) {
        const double2 *q = ka.kq + kin_xy(ka, x, y);
#pragma unroll
        for (int i = 0; i < RR; i++) {
          const double2 w = q[(long)((int)k1 + az.Q * i) * es];
          v[i] = cmul<T>(v[i], mk<T>((T)w.x, (T)w.y));
        }
      } else {
#pragma unroll
        for (int i = 0; i < RR; i++) v[i] = cscale<T>(v[i], kin_factor<T>(ka, x, y, (int)k1 + az.Q * i));
      }
#pragma unroll
      for (int i = 0; i < RR; i++) v[i] = exch<T>(v[i]);
      dft<T, RR>(v);
#pragma unroll
      for (int i = 0; i < RR; i++) {
        if (i > 0) v[i] = cmul<T>(v[i], __ldg(az.tw + (int)k1 * RR + i));
        s[i * L] = v[i];
      }
    }
  });
  __syncthreads();
  stage_a<T, BIG, false>(az, lines, lds, at, [&](int c, int z, C<T> v) { d[z * es + c] = exch<T>(v); });
}

// what a line pass does besides its transform
enum LineMode { kForward, kInverse, kFinal };  // kFinal: inverse, then out = ca (r + V phi) + cb phi

// y lines: L consecutive x of one plane, global memory to global memory, one exchange
template <typename T, bool BIG, LineMode MODE>
__global__ void __launch_bounds__(LineShape<T, BIG>::threads, LineShape<T, BIG>::ctas)
    k_two_y(const C<T> *in, C<T> *out, Axis<T> ay, int nx, int L, int ntile, const C<T> *__restrict__ phi,
            const T *__restrict__ pot, long ngrid, T ca, T cb)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C<T> *S = reinterpret_cast<C<T> *>(smem_raw);
  const long pl = blockIdx.x / ntile;
  const int x0 = (int)(blockIdx.x - pl * ntile) * L;
  const Div lines((unsigned)min(L, nx - x0));
  const long off = pl * nx * ay.n + x0;
  const C<T> *src = in + off;
  C<T> *dst = out + off;
  auto at = [&](int c, int y) -> C<T> & { return S[y * L + c]; };
  auto lds = [&](int c, int y) { return S[y * L + c]; };
  auto sts = [&](int c, int y, C<T> v) { S[y * L + c] = v; };
  if constexpr (MODE == kForward) {
    stage_a<T, BIG, true>(ay, lines, [&](int c, int y) { return src[y * nx + c]; }, at, sts);
    __syncthreads();
    stage_b<T, false>(ay, lines, lds, [&](int c, int y, C<T> v) { dst[y * nx + c] = v; });
  } else {
    stage_b<T, true>(ay, lines, [&](int c, int y) { return exch<T>(src[y * nx + c]); }, sts);
    __syncthreads();
    if constexpr (MODE == kInverse) {
      stage_a<T, BIG, false>(ay, lines, lds, at, [&](int c, int y, C<T> v) { dst[y * nx + c] = exch<T>(v); });
    } else {
      const C<T> *ph = phi + off;
      const T *V = pot ? pot + off % ngrid : nullptr;  // a plane lies inside one block
      stage_a<T, BIG, false>(ay, lines, lds, at, [&](int c, int y, C<T> v) {
        const int o = y * nx + c;
        dst[o] = epilogue<T>(exch<T>(v), ph[o], V, o, ca, cb);
      });
    }
  }
}

// x lines: L contiguous lines through shared memory with an odd line stride
// (coalesced copies, lanes on consecutive lines in the stages)
template <typename T, bool BIG, LineMode MODE>
__global__ void __launch_bounds__(LineShape<T, BIG>::threads, LineShape<T, BIG>::ctas)
    k_two_x(const C<T> *in, C<T> *out, Axis<T> ax, Div dn, long nlines, int L, const C<T> *__restrict__ phi,
            const T *__restrict__ pot, long ngrid, T ca, T cb)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C<T> *S = reinterpret_cast<C<T> *>(smem_raw);
  const int n = ax.n, pitch = n | 1;
  const long l0 = (long)blockIdx.x * L;
  const Div lines((unsigned)min((long)L, nlines - l0));
  const unsigned count = lines.d * n;
  const long off = l0 * n;
  const C<T> *src = in + off;
  for (unsigned i = threadIdx.x; i < count; i += blockDim.x) copy_async(S + i + dn(i) * (pitch - n), src + i);
  copy_wait();
  __syncthreads();
  auto at = [&](int y, int x) -> C<T> & { return S[y * pitch + x]; };
  auto ldx = [&](int y, int x) { return S[y * pitch + x]; };
  auto stx = [&](int y, int x, C<T> v) { S[y * pitch + x] = v; };
  if constexpr (MODE == kForward) {
    stage_a<T, BIG, true>(ax, lines, ldx, at, stx);
    __syncthreads();
    stage_b<T, false>(ax, lines, ldx, stx);
  } else {
    stage_b<T, true>(ax, lines, [&](int y, int x) { return exch<T>(S[y * pitch + x]); }, stx);
    __syncthreads();
    stage_a<T, BIG, false>(ax, lines, ldx, at, stx);
  }
  __syncthreads();
  C<T> *dst = out + off;
#pragma unroll 4
  for (unsigned i = threadIdx.x; i < count; i += blockDim.x) {
    C<T> r = S[i + dn(i) * (pitch - n)];
    if (MODE != kForward) r = exch<T>(r);
    if (MODE == kFinal) {
      const long g = off + i;  // the lines of a tile may lie in two blocks
      r = epilogue<T>(r, phi[g], pot, pot ? g % ngrid : 0, ca, cb);
    }
    dst[i] = r;
  }
}

}  // namespace two
}  // namespace fbse

// ---------------------------------------------------------------------------
// launches
// ---------------------------------------------------------------------------
namespace fbse {
namespace two {

template <typename T> static Axis<T> axis_of(const AxisPlan &p)
{
  if constexpr (sizeof(T) == 4) return {p.n, p.P, p.Q, p.two32, p.sym32};
  else return {p.n, p.P, p.Q, p.two64, p.sym64};
}

// threads that share one line in stage A: the butterflies, times the row blocks of stage_sym
inline long line_threads(const AxisPlan &p) { return p.sym64 ? (long)p.P * ((p.Q / 2 + kSymRows) / kSymRows) : p.P; }

template <typename K, typename... Args>
static int launch(fbse_ctx *c, K kernel, long grid, int threads, size_t smem, Args... args)
{
  if (grid > 2147483647L) return set_err(c, FBSE_ERR_UNSUPPORTED, "FFT batch too large for one launch");
  FBSE_CUDA(c, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kernel<<<(unsigned)grid, threads, smem, c->stream>>>(args...);
  FBSE_CHECK_LAUNCH(c);
  return FBSE_OK;
}

inline int round32(long v, long lo, long hi)
{
  const long r = (std::max(v, lo) + 31) / 32 * 32;
  return (int)std::min(r, hi);
}

// threads of a plane CTA: the register file's share when as many CTAs as fit
// (shared memory, or the planes there are) sit on each SM
template <typename T, bool BIG> static int plane_threads(fbse_ctx *c, size_t smem, long grid)
{
  const long fit = std::max<long>(1, std::min<long>((long)(228 * 1024 / (smem + 1024)), (grid + 151) / 152));
  const long px = line_threads(c->ax[0]), py = line_threads(c->ax[1]);
  const long work = std::max(px * c->ny, py * c->nx);
  return round32(std::min<long>(work, PlaneShape<T, BIG>::threads / fit / 32 * 32), std::max<long>(128, std::max(px, py)),
                 PlaneShape<T, BIG>::threads);
}

// lines per tile of n points: 256-byte segments, half of that when a launch
// would leave SMs idle, fewer when a long axis would take more than half an SM's
// shared memory
template <typename T> static int tile_lines(long lines, long groups, int n)
{
  const int full = std::max(2, std::min(256 / (int)sizeof(C<T>), (int)(112 * 1024 / ((n | 1) * sizeof(C<T>)))));
  int L = groups * ((lines + full - 1) / full) < 304 ? full / 2 : full;
  const long nt = (lines + L - 1) / L;
  return (int)((lines + nt - 1) / nt);  // even tiles
}

}  // namespace two

template <typename T> size_t two_plane_smem(const fbse_ctx *c) { return (size_t)(c->nx | 1) * c->ny * sizeof(C<T>); }

template <typename T>
int two_plane(fbse_ctx *c, const C<T> *in, C<T> *out, long nblk, bool inv, const C<T> *phi, const T *pot, T ca, T cb)
{
  using namespace two;
  const size_t smem = two_plane_smem<T>(c);
  const long grid = nblk * c->nz;
  const Axis<T> ax = axis_of<T>(c->ax[0]), ay = axis_of<T>(c->ax[1]);
  const Div dx((unsigned)c->nx), dy((unsigned)c->ny);
  const bool big = ax.Q > 16 || ay.Q > 16;
  const int th = big ? plane_threads<T, true>(c, smem, grid) : plane_threads<T, false>(c, smem, grid);
  auto go = [&](auto k) { return launch(c, k, grid, th, smem, in, out, ax, ay, dx, dy, phi, pot, c->ngrid, ca, cb); };
  if (big) return inv ? go(k_two_plane<T, true, true>) : go(k_two_plane<T, true, false>);
  return inv ? go(k_two_plane<T, false, true>) : go(k_two_plane<T, false, false>);
}

template <typename T> int two_z(fbse_ctx *c, C<T> *data, long nblk, const KinArgs &ka)
{
  using namespace two;
  const Axis<T> az = axis_of<T>(c->ax[2]);
  const int L = tile_lines<T>(ka.nxy, nblk, az.n);
  const int ntile = (int)((ka.nxy + L - 1) / L);
  const size_t smem = (size_t)az.n * L * sizeof(C<T>);
  if (az.Q > 16)
    return launch(c, k_two_z<T, true>, nblk * ntile, round32(line_threads(c->ax[2]) * L, 64, LineShape<T, true>::threads), smem,
                  data, az, L, ntile, c->ngrid, ka);
  return launch(c, k_two_z<T, false>, nblk * ntile, round32(line_threads(c->ax[2]) * L, 64, LineShape<T, false>::threads), smem,
                data, az, L, ntile, c->ngrid, ka);
}

template <typename T>
int two_y(fbse_ctx *c, const C<T> *in, C<T> *out, long nblk, int mode, const C<T> *phi, const T *pot, T ca, T cb)
{
  using namespace two;
  const Axis<T> ay = axis_of<T>(c->ax[1]);
  const int L = tile_lines<T>(c->nx, nblk * c->nz, ay.n);
  const int ntile = (int)((c->nx + L - 1) / L);
  const size_t smem = (size_t)ay.n * L * sizeof(C<T>);
  const bool big = ay.Q > 16;
  const int th = round32(line_threads(c->ax[1]) * L, 64, big ? LineShape<T, true>::threads : LineShape<T, false>::threads);
  auto go = [&](auto k) {
    return launch(c, k, nblk * c->nz * ntile, th, smem, in, out, ay, (int)c->nx, L, ntile, phi, pot, c->ngrid, ca, cb);
  };
  if (mode == kForward) return big ? go(k_two_y<T, true, kForward>) : go(k_two_y<T, false, kForward>);
  if (mode == kInverse) return big ? go(k_two_y<T, true, kInverse>) : go(k_two_y<T, false, kInverse>);
  return big ? go(k_two_y<T, true, kFinal>) : go(k_two_y<T, false, kFinal>);
}

template <typename T>
int two_x(fbse_ctx *c, const C<T> *in, C<T> *out, long nblk, int mode, const C<T> *phi, const T *pot, T ca, T cb)
{
  using namespace two;
  const Axis<T> ax = axis_of<T>(c->ax[0]);
  const long nlines = nblk * c->ny * c->nz;
  const int L = tile_lines<T>(nlines, 1, ax.n);
  const size_t smem = (size_t)(ax.n | 1) * L * sizeof(C<T>);
  const Div dn((unsigned)ax.n);
  const bool big = ax.Q > 16;
  const int th = round32(line_threads(c->ax[0]) * L, 64, big ? LineShape<T, true>::threads : LineShape<T, false>::threads);
  auto go = [&](auto k) {
    return launch(c, k, (nlines + L - 1) / L, th, smem, in, out, ax, dn, nlines, L, phi, pot, c->ngrid, ca, cb);
  };
  if (mode == kForward) return big ? go(k_two_x<T, true, kForward>) : go(k_two_x<T, false, kForward>);
  if (mode == kInverse) return big ? go(k_two_x<T, true, kInverse>) : go(k_two_x<T, false, kInverse>);
  return big ? go(k_two_x<T, true, kFinal>) : go(k_two_x<T, false, kFinal>);
}

}  // namespace fbse
