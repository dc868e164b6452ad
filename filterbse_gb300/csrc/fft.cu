// Batched mixed-radix 3D FFT for the kinetic term of H.
//
// Replaces kinetic() (filter_mpi/hamiltonian.c:62-99), i.e. FFTW's
// fftw_plan_dft_3d(nz, ny, nx) forward transform, the ksqr multiply and the
// unnormalised backward transform (plans made in filter_mpi/aux.c:259-270).
//
// Axes of 64, 128 and 256 points take the register-resident kernels
// (fft_fast.cuh), axes with two register radices the two-factor kernels
// (fft_two.cuh); every other length, and fbse_tuning.fft_kernels = 1, takes the
// kernels of this file:
// Each axis is a self-sorting mixed-radix Stockham FFT on lines held in shared
// memory.  The grid sizes the reference's auto-grid produces are arbitrary
// (e.g. 57 x 52 x 45 = 3*19 x 4*13 x 9*5), so an axis is factored into
// register radices: powers of two grouped into radix-16 / 8 / 4 / 2 passes
// (in-register DIF butterflies with compile-time roots) and the odd primes
// 3, 5, 7 (in-register direct DFTs with roots from the axis table); a larger
// prime takes a shared-memory pass with a scratch line.  Each pass is in place:
// every thread reads its butterflies' inputs into registers, the block
// synchronises, then the outputs are written -- so a pass costs one read and
// one write of shared memory and two barriers, and the butterfly radices keep
// the number of passes at 2-3 for typical axes (128 = 16 x 8).  Lanes of a
// warp always take consecutive lines at the same butterfly index, so index
// arithmetic and twiddles are warp-uniform; row-major lines use an odd row
// stride so the accesses are free of bank conflicts.  Twiddles come from one
// table of n roots e^{-2 pi i t/n} per axis, computed on the host in extended
// precision.
//
// Plane path (an xy plane fits in shared memory, the usual case in FP32):
//   pass 1  per (block, z): load the plane, x then y forward, store
//   pass 2  z lines in tiles of x-columns: forward, multiply by
//           min(kx^2 + ky^2 + kz^2 terms, KE_max)/N computed from the indices
//           exactly as filter_mpi/init.c:318-351 builds ksqr, inverse
//   pass 3  per (block, z): y then x inverse, fused epilogue
//           out = a (T psi + V psi) + b psi
// Line path (larger planes, FP64): x, y, z-fused, y, x passes.
// Blocks are processed in chunks sized so that a chunk's scratch stays in L2
// between the passes.
#include <cmath>

#include "fbse_internal.cuh"
#include "fft_common.cuh"

namespace fbse {

struct Stages {
  int n;
  int nst;
  int radix[kMaxStages];
  int big;  // 1 when a radix exceeds the register limit (needs a scratch line)
};
constexpr int kLineThreads = 256, kPlaneThreads = 1024;

constexpr int kRegMax = 8;  // odd radices above this take the scratch pass

static std::vector<int> factorize(int n)
{
  std::vector<int> r;
  int a = 0;
  while (n % 2 == 0) { a++; n /= 2; }
  while (a > 4) { r.push_back(16); a -= 4; }
  if (a > 0) r.push_back(1 << a);
  for (int p = 3; (long)p * p <= n; p += 2)
    while (n % p == 0) { r.push_back(p); n /= p; }
  if (n > 1) r.push_back(n);
  return r;
}

// n = P Q for the two-factor kernels: both radices at most 16 and as close as
// possible, else the largest P with a register radix up to 31, else with an
// odd Q up to kSymMax (stage_sym); false: none of them.
// Of two radices up to 16 the larger is P on the mixed path's short axes, where the
// stage that reads global memory has P butterflies a line and too few of them
// otherwise (2 blocks of 44^3: 23.5 us with 4 x 11, 20.0 with 11 x 4; 57 x 52 x 45:
// 26.2 and 25.5; 80^3: the same within 2%), and Q on long ones, where more loads in
// flight per thread pay (8 blocks of 96^3: 123.9 us with 8 x 12, 129.5 with 12 x 8;
// 116 x 117 x 120: 273 and 281).  FP64 gains from 60 points on with radices up to 10
// (4 blocks of 60^3 249 -> 244 us, 72^3 451 -> 443, one of 80^3 170 -> 166) and loses
// below and with larger ones (4 of 45^3 151 -> 159, 8 of 44^3 231 -> 262).
constexpr int kSymMin = 27, kSymMax = 255, kShortAxis = 80;
static bool larger_first(int n, int q, bool mixed) { return n <= kShortAxis && (mixed || (n >= 60 && q <= 10)); }
static bool two_factors(int n, bool mixed, int *P, int *Q)
{
  for (int set = 0; set < 3; set++)
    for (int p = 16; p >= 1; p--) {
      const int q = n / p;
      if (n % p || q < p) continue;
      const bool second = q == 17 || q == 18 || q == 19 || q == 20 || q == 21 || q == 23 || q == 24 || q == 25 ||
                          q == 29 || q == 31;
      const bool third = q % 2 == 1 && q >= kSymMin && q <= kSymMax;
      if (set == 0 ? q <= 16 : set == 1 ? second : third) {
        const bool swap = set == 0 && larger_first(n, q, mixed);
        *P = swap ? q : p;
        *Q = swap ? p : q;
        return true;
      }
    }
  return false;
}

int plan_axis(fbse_ctx *c, AxisPlan &p, int n)
{
  if (n < 1) return set_err(c, FBSE_ERR_ARG, "grid axis must have at least one point");
  std::vector<int> f = factorize(n);
  if ((int)f.size() > kMaxStages) return set_err(c, FBSE_ERR_UNSUPPORTED, "axis length has too many factors");
  p.n = n;
  p.nst = (int)f.size();
  for (int i = 0; i < p.nst; i++) p.radix[i] = f[i];
  std::vector<double2> h64(n);
  std::vector<float2> h32(n);
  for (int t = 0; t < n; t++) {
    // e^{-2 pi i t / n} in extended precision, then rounded
    long double a = 2.0L * 3.14159265358979323846264338327950288L * (long double)t / (long double)n;
    double cr = (double)cosl(a), ci = -(double)sinl(a);
    h64[t] = make_double2(cr, ci);
    h32[t] = make_float2((float)cr, (float)ci);
  }
  FBSE_CUDA(c, cudaMalloc(&p.tw64, n * sizeof(double2)));
  FBSE_CUDA(c, cudaMalloc(&p.tw32, n * sizeof(float2)));
  FBSE_CUDA(c, cudaMemcpy(p.tw64, h64.data(), n * sizeof(double2), cudaMemcpyHostToDevice));
  FBSE_CUDA(c, cudaMemcpy(p.tw32, h32.data(), n * sizeof(float2), cudaMemcpyHostToDevice));
  if (two_factors(n, c->precision == FBSE_MIXED, &p.P, &p.Q)) {
    std::vector<double2> t64(n);
    std::vector<float2> t32(n);
    for (int k1 = 0; k1 < p.Q; k1++)
      for (int t = 0; t < p.P; t++) {
        t64[t + p.P * k1] = h64[t * k1 % n];
        t32[t + p.P * k1] = h32[t * k1 % n];
      }
    FBSE_CUDA(c, cudaMalloc(&p.two64, n * sizeof(double2)));
    FBSE_CUDA(c, cudaMalloc(&p.two32, n * sizeof(float2)));
    FBSE_CUDA(c, cudaMemcpy(p.two64, t64.data(), n * sizeof(double2), cudaMemcpyHostToDevice));
    FBSE_CUDA(c, cudaMemcpy(p.two32, t32.data(), n * sizeof(float2), cudaMemcpyHostToDevice));
  }
  if (p.P > 0 && p.Q >= kSymMin && p.Q != 29 && p.Q != 31) {
    // stage_sym's coefficients [r - 1][row block][row], rows beyond Q / 2 zero
    const int h = p.Q / 2, rows = (h + kSymRows) / kSymRows * kSymRows;
    std::vector<double2> s64((size_t)h * rows, make_double2(0, 0));
    std::vector<float2> s32((size_t)h * rows, make_float2(0, 0));
    for (int r = 1; r <= h; r++)
      for (int q = 0; q <= h; q++) {
        const double2 w = h64[(long)q * r % p.Q * (n / p.Q)];
        s64[(size_t)(r - 1) * rows + q] = make_double2(w.x, -w.y);
        s32[(size_t)(r - 1) * rows + q] = make_float2((float)w.x, (float)-w.y);
      }
    FBSE_CUDA(c, cudaMalloc(&p.sym64, s64.size() * sizeof(double2)));
    FBSE_CUDA(c, cudaMalloc(&p.sym32, s32.size() * sizeof(float2)));
    FBSE_CUDA(c, cudaMemcpy(p.sym64, s64.data(), s64.size() * sizeof(double2), cudaMemcpyHostToDevice));
    FBSE_CUDA(c, cudaMemcpy(p.sym32, s32.data(), s32.size() * sizeof(float2), cudaMemcpyHostToDevice));
  }
  return FBSE_OK;
}

void free_axis(AxisPlan &p)
{
  void *bufs[] = {p.tw64, p.tw32, p.two64, p.two32, p.sym64, p.sym32, p.ord, p.k2o, p.k2of};
  for (void *b : bufs)
    if (b) cudaFree(b);
  p = AxisPlan();
}

static Stages stages_of(const AxisPlan &p)
{
  Stages s;
  s.n = p.n;
  s.nst = p.nst;
  s.big = 0;
  for (int i = 0; i < kMaxStages; i++) {
    s.radix[i] = p.radix[i];
    if (i < p.nst && p.radix[i] > kRegMax && p.radix[i] != 16) s.big = 1;
  }
  return s;
}

// butterflies of a line in the register pass that has most
static int most_butterflies(const AxisPlan &p)
{
  int most = 0;
  for (int i = 0; i < p.nst; i++)
    if (p.radix[i] <= kRegMax || p.radix[i] == 16) most = std::max(most, p.n / p.radix[i]);
  return most;
}

template <typename T> static const C<T> *roots(const AxisPlan &p);
template <> const C<float> *roots<float>(const AxisPlan &p) { return p.tw32; }
template <> const C<double> *roots<double>(const AxisPlan &p) { return p.tw64; }

// direct DFT for an odd radix with roots w[e] = e^{sg 2 pi i e / R}
template <typename T, int R>
__device__ __forceinline__ void dft_odd(C<T> *v, const C<T> *w)
{
  C<T> o[R];
#pragma unroll
  for (int q = 0; q < R; q++) {
    C<T> acc = v[0];
#pragma unroll
    for (int r = 1; r < R; r++) acc = cadd<T>(acc, cmul<T>(v[r], w[(q * r) % R]));
    o[q] = acc;
  }
#pragma unroll
  for (int q = 0; q < R; q++) v[q] = o[q];
}

template <typename T>
__device__ __forceinline__ void dft3(C<T> *v, T sg)
{
  const T h = T(0.86602540378443864676372317075293618);
  const C<T> s12 = cadd<T>(v[1], v[2]), d12 = csub<T>(v[1], v[2]);
  const C<T> t = mk<T>(v[0].x - T(0.5) * s12.x, v[0].y - T(0.5) * s12.y);
  const C<T> iu = mk<T>(-sg * h * d12.y, sg * h * d12.x);
  v[0] = cadd<T>(v[0], s12);
  v[1] = cadd<T>(t, iu);
  v[2] = csub<T>(t, iu);
}

template <typename T, int R> struct IsPow2 { static constexpr bool value = (R & (R - 1)) == 0; };

// a register pass whose lines have more butterflies than the CTA has threads (axes of
// 514 points and more on the line kernels): in place a thread would have to hold
// several, so the results go to a scratch of L lines (element i of line c at
// scr[i * L + c]) and are copied back.  The products of pass_reg.
template <typename T, int R>
__device__ __noinline__ void pass_wide(C<T> *buf, int es, int ls, int n, int L, int Ns, const C<T> *__restrict__ tw,
                                       bool inv, C<T> *scr)
{
  const int nb = n / R, twstep = n / (Ns * R);
  const T sg = inv ? T(1) : T(-1);
  for (int wi = threadIdx.x; wi < nb * L; wi += blockDim.x) {
    const int c = wi % L, j = wi / L, k = j % Ns;
    const C<T> *x = buf + c * ls;
    C<T> v[R];
    v[0] = x[j * es];
#pragma unroll
    for (int q = 1; q < R; q++) {
      C<T> t = tw[q * k * twstep];
      if (inv) t.y = -t.y;
      v[q] = cmul<T>(x[(j + q * nb) * es], t);
    }
    C<T> *o = scr + ((j / Ns) * Ns * R + k) * L + c;
    if constexpr (IsPow2<T, R>::value) {
      dif_pow2<T, R>(v, sg);
#pragma unroll
      for (int q = 0; q < R; q++) o[q * Ns * L] = v[bitrev(q, ilog2(R))];
    } else {
      if constexpr (R == 3) {
        dft3<T>(v, sg);
      } else {
        C<T> w[R];
#pragma unroll
        for (int e = 0; e < R; e++) {
          w[e] = tw[e * nb];
          if (inv) w[e].y = -w[e].y;
        }
        dft_odd<T, R>(v, w);
      }
#pragma unroll
      for (int q = 0; q < R; q++) o[q * Ns * L] = v[q];
    }
  }
  __syncthreads();
  for (int wi = threadIdx.x; wi < n * L; wi += blockDim.x) {
    const int c = wi % L, i = wi / L;
    buf[c * ls + i * es] = scr[i * L + c];
  }
  __syncthreads();
}

// ---------------------------------------------------------------------------
// one in-place Stockham pass of radix R over L lines (element i of line c at
// buf[c * ls + i * es]); lanes take consecutive lines at one butterfly index.
// WIDE: a line may have more butterflies than the CTA threads (pass_wide, with scr);
// kernels without it keep the registers that its calls would take
// ---------------------------------------------------------------------------
template <typename T, int R, bool WIDE>
__device__ __forceinline__ void pass_reg(C<T> *buf, int es, int ls, int n, int L, int Ns, const C<T> *__restrict__ tw,
                                      bool inv, C<T> *scr)
{
  if constexpr (WIDE) {
    if (n / R > (int)blockDim.x) {
      pass_wide<T, R>(buf, es, ls, n, L, Ns, tw, inv, scr);
      return;
    }
  }
  constexpr int kMaxE = R;                              // one butterfly per thread per round
  constexpr int BMAX = (kMaxE / R) > 0 ? kMaxE / R : 1;
  const int nb = n / R;
  const int twstep = n / (Ns * R);
  const T sg = inv ? T(1) : T(-1);
  C<T> w[IsPow2<T, R>::value ? 1 : R];
  if (!IsPow2<T, R>::value && R != 3) {
#pragma unroll
    for (int e = 0; e < (IsPow2<T, R>::value ? 1 : R); e++) {
      C<T> r = tw[e * nb];
      if (inv) r.y = -r.y;
      w[e] = r;
    }
  }
  const int lines_per_round = max(1, (int)(blockDim.x * BMAX) / nb);
  for (int l0 = 0; l0 < L; l0 += lines_per_round) {
    const int lr = min(lines_per_round, L - l0);
    const int tb = nb * lr;
    C<T> v[BMAX][R];
#pragma unroll
    for (int b = 0; b < BMAX; b++) {
      const int wi = threadIdx.x + b * blockDim.x;
      if (wi < tb) {
        const int c = l0 + wi % lr, j = wi / lr;
        const int k = j % Ns;
        const C<T> *x = buf + c * ls;
        v[b][0] = x[j * es];
#pragma unroll
        for (int q = 1; q < R; q++) {
          C<T> t = tw[q * k * twstep];
          if (inv) t.y = -t.y;
          v[b][q] = cmul<T>(x[(j + q * nb) * es], t);
        }
      }
    }
    __syncthreads();
#pragma unroll
    for (int b = 0; b < BMAX; b++) {
      const int wi = threadIdx.x + b * blockDim.x;
      if (wi < tb) {
        const int c = l0 + wi % lr, j = wi / lr;
        const int k = j % Ns;
        const int ob = (j / Ns) * Ns * R + k;
        C<T> *x = buf + c * ls;
        if (IsPow2<T, R>::value) {
          dif_pow2<T, R>(v[b], sg);
#pragma unroll
          for (int q = 0; q < R; q++) x[(ob + q * Ns) * es] = v[b][bitrev(q, ilog2(R))];
        } else {
          if (R == 3) dft3<T>(v[b], sg);
          else dft_odd<T, R>(v[b], w);
#pragma unroll
          for (int q = 0; q < R; q++) x[(ob + q * Ns) * es] = v[b][q];
        }
      }
    }
    __syncthreads();
  }
}

// a pass with a radix above the register limit: direct DFT from buf into a
// scratch of L lines (element i of line c at scr[i * L + c]), then copy back.  The
// inputs take their twiddles in place first; a thread then sums kBigQ outputs of
// kBigL lines, so that a value and a root each serve several products.  Each output
// is the same sum in the same order as one at a time.
// (The Rayleigh-Ritz step relies on that, so the roundings are spelled out.)  16 FP32
// spinors of 86^3, the five passes 3.1 -> 2.5 ms; the launch bounds that cap the
// kernels at 64 registers made every other pass spill.
template <typename T> constexpr int kBigL = sizeof(T) == 4 ? 4 : 2;
constexpr int kBigQ = 4;
__device__ __forceinline__ float2 cmul_rn(float2 a, float2 b)
{
  return make_float2(__fmaf_rn(a.x, b.x, -__fmul_rn(a.y, b.y)), __fmaf_rn(a.x, b.y, __fmul_rn(a.y, b.x)));
}
__device__ __forceinline__ double2 cmul_rn(double2 a, double2 b)
{
  return make_double2(__fma_rn(a.x, b.x, -__dmul_rn(a.y, b.y)), __fma_rn(a.x, b.y, __dmul_rn(a.y, b.x)));
}
template <typename T>
__device__ __noinline__ void pass_big(C<T> *buf, int es, int ls, int n, int L, int R, int Ns, const C<T> *__restrict__ tw,
                         bool inv, C<T> *scr)
{
  const int nb = n / R;
  const int twstep = n / (Ns * R);
  if (Ns > 1) {
    for (int wi = threadIdx.x; wi < (n - nb) * L; wi += blockDim.x) {
      const int c = wi % L, i = nb + wi / L;
      const int r = i / nb, k = (i - r * nb) % Ns;
      C<T> t = tw[r * k * twstep];
      if (inv) t.y = -t.y;
      C<T> *x = buf + c * ls + i * es;
      *x = cmul_rn(*x, t);
    }
    __syncthreads();
  }
  constexpr int NL = kBigL<T>, NQ = kBigQ;
  const int lg = (L + NL - 1) / NL, qg = (R + NQ - 1) / NQ;
  for (int wi = threadIdx.x; wi < lg * qg * nb; wi += blockDim.x) {
    const int c0 = wi % lg, rest = wi / lg;
    const int j = rest % nb, q0 = (rest / nb) * NQ;
    const C<T> *x[NL];
    C<T> acc[NL][NQ];
#pragma unroll
    for (int u = 0; u < NL; u++) {
      x[u] = buf + min(c0 + u * lg, L - 1) * ls + j * es;  // beyond the last line: not stored
#pragma unroll
      for (int v = 0; v < NQ; v++) acc[u][v] = *x[u];
    }
    int e[NQ];
#pragma unroll
    for (int v = 0; v < NQ; v++) e[v] = 0;
    for (int r = 1; r < R; r++) {
      C<T> t[NQ];
#pragma unroll
      for (int v = 0; v < NQ; v++) {
        e[v] += q0 + v;
        if (e[v] >= R) e[v] -= R;
        if (q0 + v >= R) e[v] = 0;  // beyond the last output: not stored
        t[v] = tw[e[v] * nb];
        if (inv) t[v].y = -t[v].y;
      }
#pragma unroll
      for (int u = 0; u < NL; u++) {
        const C<T> y = x[u][r * nb * es];
#pragma unroll
        for (int v = 0; v < NQ; v++) acc[u][v] = cadd<T>(acc[u][v], cmul_rn(y, t[v]));
      }
    }
    const int ob = (j / Ns) * Ns * R + j % Ns;
#pragma unroll
    for (int u = 0; u < NL; u++)
#pragma unroll
      for (int v = 0; v < NQ; v++)
        if (c0 + u * lg < L && q0 + v < R) scr[(ob + (q0 + v) * Ns) * L + c0 + u * lg] = acc[u][v];
  }
  __syncthreads();
  for (int wi = threadIdx.x; wi < n * L; wi += blockDim.x) {
    const int c = wi % L, i = wi / L;
    buf[c * ls + i * es] = scr[i * L + c];
  }
  __syncthreads();
}

// the passes a kernel holds: register radices in place; those and pass_big; every one.
// A call costs registers whether it is taken or not, so only the line kernels of such
// axes have them
enum Passes { kInPlace, kBig, kWide };
// CTAs per SM of a line kernel: 64 registers a thread do for the register radices (16 FP32
// states of 120 x 112 x 60 997 us, with 128 registers 1109) and make pass_big spill
template <Passes PASSES> constexpr int kLineCtas = PASSES == kInPlace ? 4 : 2;

template <typename T, Passes PASSES>
__device__ void fft_lines(C<T> *buf, int es, int ls, int L, const Stages &st, const C<T> *tw, bool inv, C<T> *scr)
{
  int Ns = 1;
  for (int s = 0; s < st.nst; s++) {
    const int R = st.radix[s];
    switch (R) {
      case 2: pass_reg<T, 2, PASSES == kWide>(buf, es, ls, st.n, L, Ns, tw, inv, scr); break;
      case 3: pass_reg<T, 3, PASSES == kWide>(buf, es, ls, st.n, L, Ns, tw, inv, scr); break;
      case 4: pass_reg<T, 4, PASSES == kWide>(buf, es, ls, st.n, L, Ns, tw, inv, scr); break;
      case 5: pass_reg<T, 5, PASSES == kWide>(buf, es, ls, st.n, L, Ns, tw, inv, scr); break;
      case 7: pass_reg<T, 7, PASSES == kWide>(buf, es, ls, st.n, L, Ns, tw, inv, scr); break;
      case 8: pass_reg<T, 8, PASSES == kWide>(buf, es, ls, st.n, L, Ns, tw, inv, scr); break;
      case 16: pass_reg<T, 16, PASSES == kWide>(buf, es, ls, st.n, L, Ns, tw, inv, scr); break;
      default:
        if constexpr (PASSES != kInPlace) pass_big<T>(buf, es, ls, st.n, L, R, Ns, tw, inv, scr);
        break;
    }
    Ns *= R;
  }
}

// ---------------------------------------------------------------------------
// plane pass: one (block, z) plane of ny x nx in shared memory, rows stored
// with an odd stride nxp.
//   MODE 0: forward x then y, store to out
//   MODE 1: inverse y then x, epilogue out = a (kin + V phi) + b phi
// ---------------------------------------------------------------------------
template <typename T, int MODE>
__global__ void __launch_bounds__(kPlaneThreads, 1) k_fft_plane(const C<T> *__restrict__ in, C<T> *__restrict__ out, Stages sx,
                                                   Stages sy, const C<T> *__restrict__ twxg,
                                                   const C<T> *__restrict__ twyg, const C<T> *__restrict__ phi,
                                                   const T *__restrict__ pot, long ngrid, T ca, T cb)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nx = sx.n, ny = sy.n;
  const int nxp = nx | 1;
  const int npl = nx * ny;
  C<T> *twx = reinterpret_cast<C<T> *>(smem_raw);
  C<T> *twy = twx + nx;
  C<T> *P = twy + ny;
  for (int t = threadIdx.x; t < nx; t += blockDim.x) twx[t] = twxg[t];
  for (int t = threadIdx.x; t < ny; t += blockDim.x) twy[t] = twyg[t];
  const long base = (long)blockIdx.x * npl;
#pragma unroll 8
  for (int t = threadIdx.x; t < npl; t += blockDim.x) P[(t / nx) * nxp + t % nx] = in[base + t];
  __syncthreads();
  if (MODE == 0) {
    fft_lines<T, kInPlace>(P, 1, nxp, ny, sx, twx, false, nullptr);  // rows
    fft_lines<T, kInPlace>(P, nxp, 1, nx, sy, twy, false, nullptr);  // columns
#pragma unroll 8
    for (int t = threadIdx.x; t < npl; t += blockDim.x) out[base + t] = P[(t / nx) * nxp + t % nx];
  } else {
    fft_lines<T, kInPlace>(P, nxp, 1, nx, sy, twy, true, nullptr);
    fft_lines<T, kInPlace>(P, 1, nxp, ny, sx, twx, true, nullptr);
#pragma unroll 8
    for (int t = threadIdx.x; t < npl; t += blockDim.x) {
      const long g = base + t;
      C<T> v = P[(t / nx) * nxp + t % nx];
      const C<T> ph = phi[g];
      if (pot) {
        const T V = pot[g % ngrid];
        v.x += V * ph.x;
        v.y += V * ph.y;
      }
      v.x = ca * v.x + cb * ph.x;
      v.y = ca * v.y + cb * ph.y;
      out[g] = v;
    }
  }
}

// ---------------------------------------------------------------------------
// x line pass (line path): L contiguous lines per CTA, line stride n|1.
// EPI = 1: fused out = a (kin + V phi) + b phi.
// ---------------------------------------------------------------------------
template <typename T, int EPI, Passes PASSES>
__global__ void __launch_bounds__(kLineThreads, kLineCtas<PASSES>) k_fft_x(const C<T> *__restrict__ in, C<T> *__restrict__ out, Stages st,
                                               const C<T> *__restrict__ twg, long nlines, int L, bool inv,
                                               const C<T> *__restrict__ phi, const T *__restrict__ pot, long ngrid,
                                               T ca, T cb)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int n = st.n, np = n | 1;
  C<T> *tw = reinterpret_cast<C<T> *>(smem_raw);
  C<T> *A = tw + n;
  C<T> *S = A + (long)L * np;  // scratch of passes that are not in place
  for (int t = threadIdx.x; t < n; t += blockDim.x) tw[t] = twg[t];
  const long line0 = (long)blockIdx.x * L;
  const int nl = (int)min((long)L, nlines - line0);
  const long off = line0 * n;
#pragma unroll 8
  for (int t = threadIdx.x; t < nl * n; t += blockDim.x) A[(t / n) * np + t % n] = in[off + t];
  __syncthreads();
  fft_lines<T, PASSES>(A, 1, np, nl, st, tw, inv, PASSES != kInPlace ? S : nullptr);
#pragma unroll 8
  for (int t = threadIdx.x; t < nl * n; t += blockDim.x) {
    C<T> v = A[(t / n) * np + t % n];
    if (EPI == 1) {
      const long g = off + t;
      const C<T> ph = phi[g];
      if (pot) {
        const T V = pot[g % ngrid];
        v.x += V * ph.x;
        v.y += V * ph.y;
      }
      v.x = ca * v.x + cb * ph.x;
      v.y = ca * v.y + cb * ph.y;
    }
    out[off + t] = v;
  }
}

// ---------------------------------------------------------------------------
// column pass (y or z lines): a tile of TX consecutive x columns of one
// (block, plane) with element stride es.  Tile o addresses
// base = (o / cnt) * s1 + (o % cnt) * s2 + xt * TX.
// KMUL: forward, multiply by the kinetic factor, inverse (z pass only).
// ---------------------------------------------------------------------------
template <typename T, bool KMUL, Passes PASSES>
__global__ void __launch_bounds__(kLineThreads, kLineCtas<PASSES>) k_fft_cols(C<T> *__restrict__ data, Stages st, const C<T> *__restrict__ twg,
                                                  long es, int nxc, int TX, int nxt, long cnt, long s1, long s2,
                                                  bool inv, KinArgs ka)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int n = st.n;
  C<T> *tw = reinterpret_cast<C<T> *>(smem_raw);
  C<T> *A = tw + n;
  C<T> *S = A + (long)TX * n;  // scratch of passes that are not in place
  for (int t = threadIdx.x; t < n; t += blockDim.x) tw[t] = twg[t];
  const long o = blockIdx.x / nxt;
  const int xt = blockIdx.x % nxt;
  const int x0 = xt * TX;
  const int L = min(TX, nxc - x0);
  const long base = (o / cnt) * s1 + (o % cnt) * s2 + x0;
#pragma unroll 8
  for (int t = threadIdx.x; t < n * L; t += blockDim.x) {
    const int cc = t % L, i = t / L;
    A[i * L + cc] = data[base + (long)i * es + cc];
  }
  __syncthreads();
  fft_lines<T, PASSES>(A, L, 1, L, st, tw, KMUL ? false : inv, PASSES != kInPlace ? S : nullptr);
  if (KMUL) {
    const int jy = (int)(o % cnt);
    if (ka.kq) {
      // convolution: multiply by the k-space array (hartree, bse_cplx/hartree.c:19-27)
      for (int t = threadIdx.x; t < n * L; t += blockDim.x) {
        const int cc = t % L, i = t / L;
        const double2 q = ka.kq[(long)i * ka.nxy + kin_xy(ka, x0 + cc, jy)];
        A[t] = cmul<T>(A[t], mk<T>((T)q.x, (T)q.y));
      }
    } else {
      for (int t = threadIdx.x; t < n * L; t += blockDim.x) {
        const int cc = t % L, i = t / L;
        A[t] = cscale<T>(A[t], kin_factor<T>(ka, x0 + cc, jy, i));
      }
    }
    __syncthreads();
    fft_lines<T, PASSES>(A, L, 1, L, st, tw, true, PASSES != kInPlace ? S : nullptr);
  }
#pragma unroll 8
  for (int t = threadIdx.x; t < n * L; t += blockDim.x) {
    const int cc = t % L, i = t / L;
    data[base + (long)i * es + cc] = A[i * L + cc];
  }
}

}  // namespace fbse

#include "fft_fast.cuh"

namespace fbse {

template <typename T> static const T *pot_of(fbse_ctx *c);
template <> const float *pot_of<float>(fbse_ctx *c) { return c->pot32; }
template <> const double *pot_of<double>(fbse_ctx *c) { return c->pot64; }

static int cols_tile(int nx, int elem)
{
  const int t = elem <= 8 ? 32 : 16;
  return nx < t ? nx : t;
}

static int max_smem()
{
  static int v = -1;
  if (v < 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) v = 48 * 1024;
  }
  return v;
}

// f with the kind of passes that an axis needs.  Tiles of which an SM holds two at most
// take the kernels with 128 registers as well (16 FP32 states of 512 x 40 x 64 1649 ->
// 1540 us)
template <typename F> static int with_passes(bool big, bool wide, size_t smem, F f)
{
  if (wide) return f(std::integral_constant<Passes, kWide>{});
  if (big || 3 * (smem + 1024) > 228 * 1024) return f(std::integral_constant<Passes, kBig>{});
  return f(std::integral_constant<Passes, kInPlace>{});
}

template <typename T>
static int launch_x(fbse_ctx *c, const C<T> *in, C<T> *out, long nblk, bool inv, int epi, const C<T> *phi,
                    const T *pot, T ca, T cb)
{
  const AxisPlan &p = c->ax[0];
  const int n = p.n;
  const long nlines = nblk * c->ny * c->nz;
  Stages st = stages_of(p);
  const bool wide = most_butterflies(p) > kLineThreads;
  int L = 32;
  while (L > 1 && (size_t)(n + (wide || st.big ? 2L : 1L) * L * (n | 1)) * sizeof(C<T>) > (size_t)max_smem()) L /= 2;
  const size_t smem = (size_t)(n + (wide || st.big ? 2L : 1L) * L * (n | 1)) * sizeof(C<T>);
  const long grid = (nlines + L - 1) / L;
  auto go = [&](auto kernel, const C<T> *ph, const T *v, T ea, T eb) -> int {
    FBSE_CUDA(c, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kernel<<<grid, kLineThreads, smem, c->stream>>>(in, out, st, roots<T>(p), nlines, L, inv, ph, v, c->ngrid, ea, eb);
    FBSE_CHECK_LAUNCH(c);
    return FBSE_OK;
  };
  auto pick = [&](auto passes) -> int {
    constexpr Passes P = decltype(passes)::value;
    return epi ? go(k_fft_x<T, 1, P>, phi, pot, ca, cb) : go(k_fft_x<T, 0, P>, nullptr, nullptr, T(1), T(0));
  };
  return with_passes(st.big, wide, smem, pick);
}

// the z pass's multiplier: the kinetic tables, or the k-space array kq, for x and
// y positions in k order or (xo, yo) in a two-factor transform's order
static KinArgs kin_args(fbse_ctx *c, const double2 *kq, bool xo, bool yo)
{
  const AxisPlan &x = c->ax[0], &y = c->ax[1];
  return {xo ? x.k2o : c->k2x,   yo ? y.k2o : c->k2y,   c->k2z, xo ? x.k2of : c->k2xf, yo ? y.k2of : c->k2yf, c->k2zf,
          c->kemax_scaled, kq, c->nx, c->nx * c->ny, xo ? x.ord : nullptr, yo ? y.ord : nullptr};
}

template <typename T>
static int launch_cols(fbse_ctx *c, C<T> *data, long nblk, int axis, bool inv, bool kmul, const KinArgs &ka)
{
  const AxisPlan &p = c->ax[axis];
  const int n = p.n;
  const Stages st = stages_of(p);
  int TX = cols_tile((int)c->nx, (int)sizeof(C<T>));
  const bool wide = most_butterflies(p) > kLineThreads;
  auto bytes = [&] { return (size_t)(n + (wide || st.big ? 2L : 1L) * TX * n) * sizeof(C<T>); };
  // narrower tiles where a long axis' register passes need the scratch
  while (!st.big && wide && TX > 1 && bytes() > (size_t)max_smem()) TX = (TX + 1) / 2;
  const int nxt = (int)((c->nx + TX - 1) / TX);
  long es, cnt, s1, s2, nouter;
  if (axis == 1) {  // y lines: outer = block*nz + z
    es = c->nx;
    cnt = 1;
    s1 = c->nx * c->ny;
    s2 = 0;
    nouter = nblk * c->nz;
  } else {  // z lines: outer = block*ny + y
    es = c->nx * c->ny;
    cnt = c->ny;
    s1 = c->ngrid;
    s2 = c->nx;
    nouter = nblk * c->ny;
  }
  const size_t smem = bytes();
  if (smem > (size_t)max_smem()) return set_err(c, FBSE_ERR_UNSUPPORTED, "FFT axis too long for shared memory");
  const long grid = nouter * nxt;
  auto go = [&](auto kernel) -> int {
    FBSE_CUDA(c, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kernel<<<grid, kLineThreads, smem, c->stream>>>(data, st, roots<T>(p), es, (int)c->nx, TX, nxt, cnt, s1, s2, inv, ka);
    FBSE_CHECK_LAUNCH(c);
    return FBSE_OK;
  };
  auto pick = [&](auto passes) -> int {
    constexpr Passes P = decltype(passes)::value;
    return kmul ? go(k_fft_cols<T, true, P>) : go(k_fft_cols<T, false, P>);
  };
  return with_passes(st.big, wide, smem, pick);
}

template <typename T> static size_t plane_smem(fbse_ctx *c)
{
  const long nx = c->nx, ny = c->ny;
  return (size_t)(nx + ny + (nx | 1) * ny) * sizeof(C<T>);
}

template <typename T>
static int launch_plane(fbse_ctx *c, const C<T> *in, C<T> *out, long nblk, int mode, const C<T> *phi, const T *pot,
                        T ca, T cb)
{
  const size_t smem = plane_smem<T>(c);
  const long grid = nblk * c->nz;
  Stages sx = stages_of(c->ax[0]), sy = stages_of(c->ax[1]);
  if (mode == 0) {
    FBSE_CUDA(c, cudaFuncSetAttribute(k_fft_plane<T, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    k_fft_plane<T, 0><<<grid, kPlaneThreads, smem, c->stream>>>(in, out, sx, sy, roots<T>(c->ax[0]), roots<T>(c->ax[1]),
                                                       nullptr, nullptr, c->ngrid, T(1), T(0));
  } else {
    FBSE_CUDA(c, cudaFuncSetAttribute(k_fft_plane<T, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    k_fft_plane<T, 1><<<grid, kPlaneThreads, smem, c->stream>>>(in, out, sx, sy, roots<T>(c->ax[0]), roots<T>(c->ax[1]), phi,
                                                       pot, c->ngrid, ca, cb);
  }
  FBSE_CHECK_LAUNCH(c);
  return FBSE_OK;
}

// ---------------------------------------------------------------------------
// register-resident kernels (fft_fast.cuh) for axes of 64, 128, 256 points;
// fbse_tuning.fft_kernels = 1 selects the mixed-radix kernels for every axis,
// = 2 the mixed-radix line passes
// ---------------------------------------------------------------------------
static bool fast_axis_ok(fbse_ctx *c, long n) { return c->tune.fft_kernels == 0 && (n == 64 || n == 128 || n == 256); }

template <typename T> static bool fast_plane_ok(fbse_ctx *c)
{
  if (c->tune.fft_kernels != 0 || c->nx != c->ny) return false;
  if (c->nx == 64) return fast::PlaneCfg<T, 64>::smem() <= (size_t)max_smem();
  if (c->nx == 128 && sizeof(C<T>) == 8) return fast::PlaneCfg<T, 128>::smem() <= (size_t)max_smem();
  return false;
}

template <typename T, int N>
static int launch_plane_fast_n(fbse_ctx *c, const C<T> *in, C<T> *out, long nblk, int mode, const C<T> *phi,
                               const T *pot, T ca, T cb)
{
  using Cfg = fast::PlaneCfg<T, N>;
  const size_t smem = Cfg::smem();
  const long grid = nblk * c->nz;
  const C<T> *rt = roots<T>(c->ax[0]);
  if (mode == 0) {
    FBSE_CUDA(c, cudaFuncSetAttribute(fast::k_plane_fast<T, N, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem));
    fast::k_plane_fast<T, N, 0><<<grid, Cfg::THREADS, smem, c->stream>>>(in, out, rt, nullptr, nullptr, c->ngrid,
                                                                          T(1), T(0));
  } else {
    FBSE_CUDA(c, cudaFuncSetAttribute(fast::k_plane_fast<T, N, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem));
    fast::k_plane_fast<T, N, 1><<<grid, Cfg::THREADS, smem, c->stream>>>(in, out, rt, phi, pot, c->ngrid, ca, cb);
  }
  FBSE_CHECK_LAUNCH(c);
  return FBSE_OK;
}

// the two-CTA cluster variant (fbse_tuning.fft_plane_cluster = 1) of the 128 x 128 FP32 plane
template <typename T, int N>
static int launch_plane_cl_n(fbse_ctx *c, const C<T> *in, C<T> *out, long nblk, int mode, const C<T> *phi,
                             const T *pot, T ca, T cb)
{
  using Cfg = fast::ClCfg<T, N>;
  const size_t smem = Cfg::smem();
  const long grid = 2 * nblk * c->nz;
  const C<T> *rt = roots<T>(c->ax[0]);
  if (mode == 0) {
    FBSE_CUDA(c, cudaFuncSetAttribute(fast::k_plane_cl<T, N, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    fast::k_plane_cl<T, N, 0><<<grid, Cfg::THREADS, smem, c->stream>>>(in, out, rt, nullptr, nullptr, c->ngrid, T(1),
                                                                        T(0));
  } else {
    FBSE_CUDA(c, cudaFuncSetAttribute(fast::k_plane_cl<T, N, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    fast::k_plane_cl<T, N, 1><<<grid, Cfg::THREADS, smem, c->stream>>>(in, out, rt, phi, pot, c->ngrid, ca, cb);
  }
  FBSE_CHECK_LAUNCH(c);
  return FBSE_OK;
}

template <typename T>
static int launch_plane_fast(fbse_ctx *c, const C<T> *in, C<T> *out, long nblk, int mode, const C<T> *phi,
                             const T *pot, T ca, T cb)
{
  if (c->nx == 64) return launch_plane_fast_n<T, 64>(c, in, out, nblk, mode, phi, pot, ca, cb);
  if constexpr (sizeof(C<T>) == 8) {
    if (c->nx == 128 && c->tune.fft_plane_cluster == 1) return launch_plane_cl_n<T, 128>(c, in, out, nblk, mode, phi, pot, ca, cb);
  }
  if constexpr (sizeof(C<T>) == 8) {
    if (c->nx == 128) return launch_plane_fast_n<T, 128>(c, in, out, nblk, mode, phi, pot, ca, cb);
  }
  return set_err(c, FBSE_ERR_UNSUPPORTED, "no register-resident plane kernel for this size");
}

template <typename T, int N>
static int launch_cols_fast_n(fbse_ctx *c, C<T> *data, long nblk, int axis, bool inv, bool kmul, const KinArgs &ka)
{
  using Cfg = fast::ColsCfg<T, N>;
  const int nxt = (int)((c->nx + 31) / 32);
  long es, cnt, s1, s2, nouter;
  if (axis == 1) {
    es = c->nx; cnt = 1; s1 = c->nx * c->ny; s2 = 0; nouter = nblk * c->nz;
  } else {
    es = c->nx * c->ny; cnt = c->ny; s1 = c->ngrid; s2 = c->nx; nouter = nblk * c->ny;
  }
  const size_t smem = Cfg::smem();
  const long grid = nouter * nxt;
  const C<T> *rt = roots<T>(c->ax[axis]);
  if (kmul) {
    FBSE_CUDA(c, cudaFuncSetAttribute(fast::k_cols_fast<T, N, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem));
    fast::k_cols_fast<T, N, true><<<grid, Cfg::THREADS, smem, c->stream>>>(data, rt, es, (int)c->nx, nxt, cnt, s1,
                                                                            s2, inv, ka);
  } else {
    FBSE_CUDA(c, cudaFuncSetAttribute(fast::k_cols_fast<T, N, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem));
    fast::k_cols_fast<T, N, false><<<grid, Cfg::THREADS, smem, c->stream>>>(data, rt, es, (int)c->nx, nxt, cnt, s1,
                                                                             s2, inv, ka);
  }
  FBSE_CHECK_LAUNCH(c);
  return FBSE_OK;
}

// two-factor kernels (fft_two.cuh): any other length that has the two factors
static bool two_axis_ok(fbse_ctx *c, int axis)
{
  return c->tune.fft_kernels == 0 && !c->steady && c->ax[axis].P > 0 && !fast_axis_ok(c, c->ax[axis].n);
}

// y or z lines; z (kmul): forward, multiply, inverse
template <typename T>
static int launch_cols_any(fbse_ctx *c, C<T> *data, long nblk, int axis, bool inv, bool kmul, const KinArgs &ka)
{
  if (two_axis_ok(c, axis))
    return kmul ? two_z<T>(c, data, nblk, ka) : two_y<T>(c, data, data, nblk, inv ? 1 : 0, nullptr, nullptr, T(1), T(0));
  switch (fast_axis_ok(c, c->ax[axis].n) ? c->ax[axis].n : 0) {
    case 64: return launch_cols_fast_n<T, 64>(c, data, nblk, axis, inv, kmul, ka);
    case 128: return launch_cols_fast_n<T, 128>(c, data, nblk, axis, inv, kmul, ka);
    case 256: return launch_cols_fast_n<T, 256>(c, data, nblk, axis, inv, kmul, ka);
    default: return launch_cols<T>(c, data, nblk, axis, inv, kmul, ka);
  }
}

int zpass_kinetic(fbse_ctx *c, float2 *data, long nblk)
{
  return launch_cols_any<float>(c, data, nblk, 2, false, true, kin_args(c, nullptr, false, false));
}

template <typename T, int N>
static int launch_x_fast_n(fbse_ctx *c, const C<T> *in, C<T> *out, long nblk, bool inv, int epi, const C<T> *phi,
                           const T *pot, T ca, T cb)
{
  using Cfg = fast::XCfg<T, N>;
  const long nlines = nblk * c->ny * c->nz;
  const size_t smem = Cfg::smem();
  const long grid = (nlines + Cfg::LINES - 1) / Cfg::LINES;
  const C<T> *rt = roots<T>(c->ax[0]);
  if (epi) {
    FBSE_CUDA(c, cudaFuncSetAttribute(fast::k_x_fast<T, N, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    fast::k_x_fast<T, N, 1><<<grid, Cfg::THREADS, smem, c->stream>>>(in, out, rt, nlines, inv, phi, pot, c->ngrid,
                                                                      ca, cb);
  } else {
    FBSE_CUDA(c, cudaFuncSetAttribute(fast::k_x_fast<T, N, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    fast::k_x_fast<T, N, 0><<<grid, Cfg::THREADS, smem, c->stream>>>(in, out, rt, nlines, inv, nullptr, nullptr,
                                                                      c->ngrid, T(1), T(0));
  }
  FBSE_CHECK_LAUNCH(c);
  return FBSE_OK;
}

template <typename T>
static int launch_x_any(fbse_ctx *c, const C<T> *in, C<T> *out, long nblk, bool inv, int epi, const C<T> *phi,
                        const T *pot, T ca, T cb)
{
  if (two_axis_ok(c, 0)) return two_x<T>(c, in, out, nblk, inv ? (epi ? 2 : 1) : 0, phi, pot, ca, cb);
  switch (fast_axis_ok(c, c->nx) ? c->nx : 0) {
    case 64: return launch_x_fast_n<T, 64>(c, in, out, nblk, inv, epi, phi, pot, ca, cb);
    case 128: return launch_x_fast_n<T, 128>(c, in, out, nblk, inv, epi, phi, pot, ca, cb);
    case 256: return launch_x_fast_n<T, 256>(c, in, out, nblk, inv, epi, phi, pot, ca, cb);
    default: return launch_x<T>(c, in, out, nblk, inv, epi, phi, pot, ca, cb);
  }
}

// whole planes in shared memory (three passes over memory) or y and x lines (five) for
// nblk blocks of the two-factor kernels.  FP32 passes are bound by memory and latency:
// planes when they fit (8 blocks of 96^3 124 us, lines 131; 1 of 57 x 52 x 45 25 us,
// lines 38).  FP64 passes are bound by the FP64 pipe, which a last wave of planes leaves
// half idle: lines unless the planes fill whole waves of the 152 SMs (2 blocks of 96^3
// 595 us, lines 455; 12 of 96^3 2598, lines 2458; 150 planes of 72 x 70 252, lines 292)
template <typename T> static bool two_planes(fbse_ctx *c, long nblk)
{
  const long n = nblk * c->nz, waves = (n + 151) / 152;
  return two_plane_smem<T>(c) <= (size_t)max_smem() && (sizeof(T) == 4 || n * 100 >= 97 * 152 * waves);
}

// out = a (F^-1 K F in + V in) + b in with K = the capped kinetic factor, or
// the complex k-space array kq when given (then V is not applied); cb blocks
// per launch sequence
template <typename T>
static int fft_op_chunked(fbse_ctx *c, const C<T> *in, C<T> *out, C<T> *work, long nblk, double a, double b,
                          int with_v, const double2 *kq, long cb)
{
  int rc;
  const Stages sx = stages_of(c->ax[0]), sy = stages_of(c->ax[1]);
  const T *pot = with_v ? pot_of<T>(c) : nullptr;
  const bool fplane = fast_plane_ok<T>(c);
  // x and y both of two factors (64, 128 and 256 points are): whole planes in shared
  // memory, or y and x lines with the same arithmetic in the same order
  const bool both = !fplane && c->tune.fft_kernels == 0 && !c->steady && c->ax[0].P > 0 && c->ax[1].P > 0;
  const bool lines = two_axis_ok(c, 0) || two_axis_ok(c, 1);
  // the mixed-radix planes also beside a two-factor y axis, in FP32, when x has no two
  // factors and y is short: 1 and 16 states of 512 x 10 x 64 97 and 475 us (lines 159, 475), of
  // 1024 x 10 x 64 132 and 788 (162, 895), 768 x 20 x 64 164 and 1103 (216, 1322);
  // 512 x 30 x 64 186 and 1237 (161, 1209).  A long y axis gains from lines at every width.
  const bool rod = sizeof(T) == 4 && c->ax[0].P == 0 && c->ny < 28;
  const bool plane = (!lines || rod) && !sx.big && !sy.big &&
                     std::max(most_butterflies(c->ax[0]), most_butterflies(c->ax[1])) <= kPlaneThreads &&
                     plane_smem<T>(c) <= (size_t)max_smem() && c->tune.fft_kernels != 2;
  // which of x and y the z pass meets in a two-factor transform's order
  const bool xo = both || (!fplane && !plane && two_axis_ok(c, 0));
  const bool yo = both || (!fplane && !plane && two_axis_ok(c, 1));
  const KinArgs ka = kin_args(c, kq, xo, yo);
  for (long b0 = 0; b0 < nblk; b0 += cb) {
    const long nb = (nblk - b0 < cb) ? nblk - b0 : cb;
    const C<T> *ci = in + b0 * c->ngrid;
    C<T> *co = out + b0 * c->ngrid;
    C<T> *wk = work;  // reused by every chunk: a chunk's intermediate passes can stay in L2
    if (fplane) {
      if ((rc = launch_plane_fast<T>(c, ci, wk, nb, 0, nullptr, nullptr, T(1), T(0)))) return rc;
      if ((rc = launch_cols_any<T>(c, wk, nb, 2, false, true, ka))) return rc;
      if ((rc = launch_plane_fast<T>(c, wk, co, nb, 1, ci, pot, (T)a, (T)b))) return rc;
    } else if (both && two_planes<T>(c, nb)) {
      if ((rc = two_plane<T>(c, ci, wk, nb, false, nullptr, nullptr, T(1), T(0)))) return rc;
      if ((rc = launch_cols_any<T>(c, wk, nb, 2, false, true, ka))) return rc;
      if ((rc = two_plane<T>(c, wk, co, nb, true, ci, pot, (T)a, (T)b))) return rc;
    } else if (both) {
      if ((rc = two_y<T>(c, ci, wk, nb, 0, nullptr, nullptr, T(1), T(0)))) return rc;
      if ((rc = two_x<T>(c, wk, wk, nb, 0, nullptr, nullptr, T(1), T(0)))) return rc;
      if ((rc = launch_cols_any<T>(c, wk, nb, 2, false, true, ka))) return rc;
      if ((rc = two_x<T>(c, wk, wk, nb, 1, nullptr, nullptr, T(1), T(0)))) return rc;
      if ((rc = two_y<T>(c, wk, co, nb, 2, ci, pot, (T)a, (T)b))) return rc;
    } else if (plane) {
      if ((rc = launch_plane<T>(c, ci, wk, nb, 0, nullptr, nullptr, T(1), T(0)))) return rc;
      if ((rc = launch_cols<T>(c, wk, nb, 2, false, true, ka))) return rc;
      if ((rc = launch_plane<T>(c, wk, co, nb, 1, ci, pot, (T)a, (T)b))) return rc;
    } else {
      if ((rc = launch_x_any<T>(c, ci, wk, nb, false, 0, nullptr, nullptr, T(1), T(0)))) return rc;
      if ((rc = launch_cols_any<T>(c, wk, nb, 1, false, false, ka))) return rc;
      if ((rc = launch_cols_any<T>(c, wk, nb, 2, false, true, ka))) return rc;
      if ((rc = launch_cols_any<T>(c, wk, nb, 1, true, false, ka))) return rc;
      if ((rc = launch_x_any<T>(c, wk, co, nb, true, 1, ci, pot, (T)a, (T)b))) return rc;
    }
  }
  return FBSE_OK;
}

// blocks per launch sequence: fixed by fbse_tuning.fft_chunk_blocks or
// autotuned (every block gets the same bits either way: the FP64 two-factor plane
// and line kernels, between which a launch's blocks decide, share their stages;
// a smaller chunk keeps its intermediate passes in L2, a larger one fills the GPU
// better)
template <typename T>
static int fft_op_apply(fbse_ctx *c, const C<T> *in, C<T> *out, C<T> *work, long nblk, double a, double b,
                        int with_v, const double2 *kq)
{
  long cb = c->tune.fft_chunk_blocks;
  if (cb == 0) {
    cb = nblk;
    if (nblk >= 4 && (const void *)in != (const void *)out) {
      std::vector<long> cands{nblk};
      for (long v : {16L, 8L, 4L, 2L})
        if (v < nblk) cands.push_back(v);
      // the Rayleigh-Ritz step runs other kernels on all but these grids
      const bool other = c->steady && !(fast_axis_ok(c, c->nx) && fast_axis_ok(c, c->ny) && fast_axis_ok(c, c->nz));
      const std::string prob = std::string(sizeof(T) == 4 ? "fp32" : "fp64") + " grid=" + std::to_string(c->nx) +
                               "x" + std::to_string(c->ny) + "x" + std::to_string(c->nz) +
                               " blocks=" + std::to_string(nblk) + (kq ? " convolution" : " kinetic") +
                               (other ? " Rayleigh-Ritz" : "");
      int rc = autotune(c, "fft blocks per launch", prob, cands,
                        [&](long v) { return fft_op_chunked<T>(c, in, out, work, nblk, a, b, with_v, kq, v); }, &cb);
      if (rc) return rc;
    }
  }
  return fft_op_chunked<T>(c, in, out, work, nblk, a, b, with_v, kq, cb < nblk ? cb : nblk);
}

template <typename T>
int kinetic_apply(fbse_ctx *c, const C<T> *in, C<T> *out, C<T> *work, long nblk, double a, double b, int with_v)
{
  return fft_op_apply<T>(c, in, out, work, nblk, a, b, with_v, nullptr);
}

template <typename T>
int conv_apply(fbse_ctx *c, const C<T> *in, C<T> *out, C<T> *work, long nblk, const double2 *kq)
{
  return fft_op_apply<T>(c, in, out, work, nblk, 1.0, 0.0, 0, kq);
}

// unnormalised forward 3D DFT of one FP64 block in place (FFTW_FORWARD of the
// reference's fftw_plan_dft_3d); work: one block of scratch
int forward_fft64(fbse_ctx *c, double2 *data, double2 *work)
{
  int rc;
  if ((rc = launch_x<double>(c, data, work, 1, false, 0, nullptr, nullptr, 1.0, 0.0))) return rc;
  const KinArgs ka = kin_args(c, nullptr, false, false);
  if ((rc = launch_cols<double>(c, work, 1, 1, false, false, ka))) return rc;
  if ((rc = launch_cols<double>(c, work, 1, 2, false, false, ka))) return rc;
  FBSE_CUDA(c, cudaMemcpyAsync(data, work, c->ngrid * sizeof(double2), cudaMemcpyDeviceToDevice, c->stream));
  return FBSE_OK;
}

template int conv_apply<float>(fbse_ctx *, const C<float> *, C<float> *, C<float> *, long, const double2 *);
template int conv_apply<double>(fbse_ctx *, const C<double> *, C<double> *, C<double> *, long, const double2 *);
template int kinetic_apply<float>(fbse_ctx *, const C<float> *, C<float> *, C<float> *, long, double, double, int);
template int kinetic_apply<double>(fbse_ctx *, const C<double> *, C<double> *, C<double> *, long, double, double, int);

}  // namespace fbse
