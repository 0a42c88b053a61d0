// kmhd_fft.cu -- longitudinal real FFTs fused with the grid-space products.
//
// Each (r, theta) line is handled by one CTA with every component of the line
// in shared memory, so inverse FFT -> products -> forward FFT never touch HBM.
// Convention (t_sph_single_FFTW.F90 normalisation with the FFTPACK slot order of
// PARALLEL_src/SPH_SHELL_src/t_sph_FFTPACK5.f90:183-331):
//   x_j = a_0 + sum_{k>=1} (a_k cos(2 pi jk/N) + b_k sin(2 pi jk/N)),
//   a_0 = (1/N) sum x_j, a_k = (2/N) sum x_j cos, b_k = (2/N) sum x_j sin.
// Two real components travel as one complex sequence z = x_a + i x_b.  The
// inverse transform is an in-place mixed-radix decimation in frequency
// (natural spectrum in, digit-reversed grid out); the products are pointwise,
// so they run on the digit-reversed grid; the forward transform is its exact
// transpose (decimation in time, digit-reversed in, natural out).  No
// reordering pass exists.  The first inverse pass reads the staged spectra
// directly and skips the band L < k < N-L, which is zero.
// Products: cal_cross_prod_w_coef_smp, cal_vec_scalar_prod_w_coef_smp,
// cal_dot_prod_w_coef_smp (CORE_src/BASE/cal_products_smp.f90) as called by
// nonlinear_terms_in_rtp (MHD_src/sph_MHD/cal_nonlinear_sph_MHD.f90:64-128).
#include <cuda.h>

#include <algorithm>
#include <cstring>
#include <type_traits>
#include <utility>

#include "kmhd_internal.cuh"

namespace kmhd {
namespace {

constexpr int kFftThreads = 256;
constexpr int kRtmOrders = 1 << kRtmShift;

// mbarrier + bulk copies (staging of a line's spectra)
constexpr long long kFftSpinCap = 1ll << 22;  // try_wait rounds (each may suspend for microseconds)
__device__ __forceinline__ unsigned ssa(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool fbar_wait(unsigned long long* b, unsigned parity, long long cap = kFftSpinCap) {
  for (long long it = 0; it < cap; ++it) {
    unsigned ok;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(ssa(b)), "r"(parity));
    if (ok) return true;
  }
  return false;
}

__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
template <int SIGN>
__device__ __forceinline__ double2 mul_si(double2 a) {  // a * (SIGN i)
  return SIGN > 0 ? make_double2(-a.y, a.x) : make_double2(a.y, -a.x);
}

// y_q = sum_r x_r e^{SIGN 2 pi i r q / R}, in place, compile-time R.
template <int R, int SIGN>
struct DFT;
template <int SIGN>
struct DFT<2, SIGN> {
  __device__ static void run(double2* x) {
    const double2 a = x[0], b = x[1];
    x[0] = cadd(a, b);
    x[1] = csub(a, b);
  }
};
template <int SIGN>
struct DFT<4, SIGN> {
  __device__ static void run(double2* x) {
    const double2 a = cadd(x[0], x[2]), b = csub(x[0], x[2]);
    const double2 c = cadd(x[1], x[3]), d = mul_si<SIGN>(csub(x[1], x[3]));
    x[0] = cadd(a, c);
    x[1] = cadd(b, d);
    x[2] = csub(a, c);
    x[3] = csub(b, d);
  }
};
template <int SIGN>
struct DFT<3, SIGN> {
  __device__ static void run(double2* x) {
    const double s3 = 0.86602540378443864676 * (double)SIGN;
    const double2 t = cadd(x[1], x[2]);
    const double2 d = csub(x[1], x[2]);
    const double2 u = make_double2(-d.y * s3, d.x * s3);
    const double2 v = make_double2(x[0].x - 0.5 * t.x, x[0].y - 0.5 * t.y);
    x[0] = cadd(x[0], t);
    x[1] = cadd(v, u);
    x[2] = csub(v, u);
  }
};
template <int SIGN>
struct DFT<5, SIGN> {
  __device__ static void run(double2* x) {
    const double c1 = 0.30901699437494742410, c2 = -0.80901699437494742410;
    const double s1 = 0.95105651629515357212 * (double)SIGN, s2 = 0.58778525229247312917 * (double)SIGN;
    const double2 a1 = cadd(x[1], x[4]), b1 = csub(x[1], x[4]);
    const double2 a2 = cadd(x[2], x[3]), b2 = csub(x[2], x[3]);
    const double2 x0 = x[0];
    const double2 t1 = make_double2(x0.x + c1 * a1.x + c2 * a2.x, x0.y + c1 * a1.y + c2 * a2.y);
    const double2 t2 = make_double2(x0.x + c2 * a1.x + c1 * a2.x, x0.y + c2 * a1.y + c1 * a2.y);
    const double2 u1 = make_double2(-(s1 * b1.y + s2 * b2.y), s1 * b1.x + s2 * b2.x);
    const double2 u2 = make_double2(-(s2 * b1.y - s1 * b2.y), s2 * b1.x - s1 * b2.x);
    x[0] = make_double2(x0.x + a1.x + a2.x, x0.y + a1.y + a2.y);
    x[1] = cadd(t1, u1);
    x[4] = csub(t1, u1);
    x[2] = cadd(t2, u2);
    x[3] = csub(t2, u2);
  }
};
template <int SIGN>
struct DFT<8, SIGN> {
  __device__ static void run(double2* x) {
    const double h = 0.70710678118654752440;
    double2 e[4] = {x[0], x[2], x[4], x[6]}, o[4] = {x[1], x[3], x[5], x[7]};
    DFT<4, SIGN>::run(e);
    DFT<4, SIGN>::run(o);
    o[1] = make_double2(h * (o[1].x - (double)SIGN * o[1].y), h * (o[1].y + (double)SIGN * o[1].x));
    o[2] = mul_si<SIGN>(o[2]);
    o[3] = make_double2(h * (-o[3].x - (double)SIGN * o[3].y), h * (-o[3].y + (double)SIGN * o[3].x));
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      x[k] = cadd(e[k], o[k]);
      x[k + 4] = csub(e[k], o[k]);
    }
  }
};

template <int SIGN>
__device__ __forceinline__ double2 twd(const double2* __restrict__ tw, int idx) {
  const double2 w = __ldg(tw + idx);
  return SIGN > 0 ? w : make_double2(w.x, -w.y);
}

// Twiddles w^(j q), q = 0, 1, ..., of one radix-R butterfly (w = e^{2 pi i / N})
// with a table load every K-th q only: a running product w^(j q) = w^(j (q - 1)) w^j,
// restarted from the table at q = K, 2 K, ..., so at most K - 1 products separate
// a twiddle from a table value (K = 8: within 2e-15 of e^{2 pi i j q / N} for
// N = 48 .. 3072, checked against exact values).
// K = 8 in the first and last passes of the specialised kernels, whose lanes
// read 32 different table entries per load (at L = 511 an FFT kernel of 20.6 ms
// took 21.7 ms restarting every fourth q, 23.5 ms loading every twiddle; that
// kernel has since been rebuilt).
// K = 4 in the run-time passes and at N = 3072.  One frequency alone (b_trans, rms in
// 2^-53 at N = 384, 450, 768): 0.76, 0.85, 0.76; with K = 8 1.05, 1.07, 1.01, with every
// twiddle from the table 0.64, 0.78, 0.65.  What T of the default set takes from its
// partner at L = 127: 5.2e-16, 8.5e-16, 4.6e-16; smooth spectra show no difference
// between K = 4 and the table.  The table alone costs 6 to 7% of a separable
// transform at L = 127 (0.78 -> 0.83 ms), K = 4 less than 1%.
constexpr int kTwSpecial = 8, kTwRun = 4;
template <int SIGN, int K>
struct TwiddleRun {
  const double2* tw;
  int j;
  double2 w1, cur;
  __device__ __forceinline__ TwiddleRun(const double2* __restrict__ t, int jj) : tw(t), j(jj) {
    w1 = twd<SIGN>(tw, j);
    cur = make_double2(1.0, 0.0);
  }
  // w^(j q) for the next q (called for q = 1, 2, ... in order)
  __device__ __forceinline__ double2 next(int q) {
    cur = q % K == 0 ? twd<SIGN>(tw, j * q) : (q == 1 ? w1 : cmul(cur, w1));
    return cur;
  }
};

// ---------------------------------------------------------------------------
// Passes of run-time N: the radices P.fac (composite, at most 16) over nseq
// sequences zs entries apart.  Entry i of a sequence sits at index i ^ ((i >> 3
// ^ i >> 6) & 7) where N is a multiple of eight (power-of-two strides would
// meet in few banks), at i otherwise.
struct Seqs {
  double2* z;
  int n, zs, N, msk;
  __device__ Seqs(double2* z_, int n_, int zs_, int N_) : z(z_), n(n_), zs(zs_), N(N_), msk(N_ % 8 == 0 ? 7 : 0) {}
  __device__ __forceinline__ int ix(int i) const { return i ^ (((i >> 3) ^ (i >> 6)) & msk); }
};

// Complex spectrum of pair pp at frequency k from a line's records.  z = x + i y,
// X[m] = (a - i b)/2 for m > 0, X[0] = a, X[N-m] = conj(X[m]).
// line: the line's block rows, bs doubles apart (staged: rtm_row; in place in
// rtm: rtm_row nr nth).
// src: where the pair's components are; two: it holds two.
__device__ __forceinline__ double2 spec_at(const Plan& P, const double* line, long long bs, const PairPos& src, bool two,
                                           int k) {
  // no branch around the loads: a butterfly's loads go out together (zero-band
  // frequencies load order 0)
  const int N = P.nph, L = P.L;
  const bool mirror = k >= N - L, zero = k > L && !mirror;
  const int m = mirror ? N - k : zero ? 0 : k;
  const double* s = line + (m >> P.mbs) * bs;
  const double2 c0 = *reinterpret_cast<const double2*>(s + src.x(m));
  const double2 c1 = *reinterpret_cast<const double2*>(s + (two ? src.y(m) : src.x(m)));
  const double h = zero ? 0.0 : m == 0 ? 1.0 : 0.5;
  const double h1 = two ? h : 0.0, hs = m == 0 ? 0.0 : mirror ? -h : h, hs1 = m == 0 ? 0.0 : mirror ? -h1 : h1;
  // m = 0: (a_x, a_y); else x / 2 -+ i y / 2 of the two components
  return m == 0 ? make_double2(h * c0.x, h1 * c1.x) : make_double2(h * c0.x + hs1 * c1.y, h1 * c1.x - hs * c0.y);
}

// ---------------------------------------------------------------------------
// Composite radices.  e^{2 pi i k / 48}: cos and sin of the first quadrant, k = 0..11
__host__ __device__ constexpr double c48q(int k) {
  constexpr double c[12] = {1.0, 0.9914448613738104, 0.9659258262890683, 0.9238795325112867,
                            0.8660254037844386, 0.7933533402912352, 0.7071067811865476, 0.6087614290087207,
                            0.5, 0.3826834323650898, 0.25881904510252074, 0.1305261922200516};
  return c[k];
}
// cos and sin of 2 pi k / R for the radices that do not divide 48
__host__ __device__ constexpr double cos9(int k) {
  constexpr double c[9] = {1.0, 0.76604444311897803520, 0.17364817766693034885, -0.5, -0.93969262078590838405,
                           -0.93969262078590838405, -0.5, 0.17364817766693034885, 0.76604444311897803520};
  return c[k];
}
__host__ __device__ constexpr double sin9(int k) {
  constexpr double c[9] = {0.0, 0.64278760968653932632, 0.98480775301220805936, 0.86602540378443864676,
                           0.34202014332566873304, -0.34202014332566873304, -0.86602540378443864676,
                           -0.98480775301220805936, -0.64278760968653932632};
  return c[k];
}
// multiples of 12 degrees, k = 0 .. 29 (R = 15: 2 e, R = 10: 3 e)
__host__ __device__ constexpr double cos30(int k) {
  constexpr double c[8] = {1.0, 0.97814760073380563793, 0.91354545764260089550, 0.80901699437494742410,
                           0.66913060635885821383, 0.5, 0.30901699437494742410, 0.10452846326765347140};
  k = k % 30;
  if (k > 15) k = 30 - k;
  return k <= 7 ? c[k] : -c[15 - k];
}
__host__ __device__ constexpr double sin30(int k) {
  constexpr double c[8] = {0.0, 0.20791169081775933710, 0.40673664307580020775, 0.58778525229247312917,
                           0.74314482547739423501, 0.86602540378443864676, 0.95105651629515357212,
                           0.99452189536827333692};
  k = k % 30;
  if (k > 15) return -sin30(30 - k);
  return k <= 7 ? c[k] : c[15 - k];
}
// x * e^{SIGN 2 pi i e / R}, e and R compile-time, R | 48 or R = 9, 10, 15
template <int R, int E, int SIGN>
__device__ __forceinline__ double2 rot(double2 x) {
  if constexpr (48 % R != 0) {
    if constexpr (E % R == 0) return x;
    constexpr double c = R == 9 ? cos9(E % 9) : cos30(E % R * (30 / (R == 9 ? 10 : R)));
    constexpr double sn = (R == 9 ? sin9(E % 9) : sin30(E % R * (30 / (R == 9 ? 10 : R)))) * (double)SIGN;
    return make_double2(x.x * c - x.y * sn, x.x * sn + x.y * c);
  } else {
  constexpr int k = (E * (48 / R)) % 48;
  constexpr int q = k / 12, k0 = k % 12;
  if constexpr (k0 == 0) {
    // multiples of 90 degrees
    if constexpr (q == 0) return x;
    else if constexpr (q == 2) return make_double2(-x.x, -x.y);
    else if constexpr ((q == 1) == (SIGN > 0)) return make_double2(-x.y, x.x);  // * i
    else return make_double2(x.y, -x.x);                                        // * -i
  } else {
    // (c, s) of angle k * 7.5 degrees
    constexpr double c0 = c48q(k0), s0 = c48q(12 - k0);
    constexpr double c = q == 0 ? c0 : q == 1 ? -s0 : q == 2 ? -c0 : s0;
    constexpr double sn = (q == 0 ? s0 : q == 1 ? c0 : q == 2 ? -s0 : -c0) * (double)SIGN;
    return make_double2(x.x * c - x.y * sn, x.x * sn + x.y * c);
  }
  }
}

// DFT of length A*B (Cooley-Tukey, n = B n1 + n2, k = k1 + A k2), in place.
template <int A, int B, int SIGN>
struct DFT2F {
  template <int N2, int K1>
  __device__ static void tw_one(double2* y) {
    y[N2 * A + K1] = rot<A * B, N2 * K1, SIGN>(y[N2 * A + K1]);
  }
  __device__ static void run(double2* x) {
    double2 y[A * B];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) {
      double2 t[A];
#pragma unroll
      for (int n1 = 0; n1 < A; ++n1) t[n1] = x[B * n1 + n2];
      DFT<A, SIGN>::run(t);
#pragma unroll
      for (int k1 = 0; k1 < A; ++k1) y[n2 * A + k1] = t[k1];
    }
    twiddle_all(y, std::make_integer_sequence<int, A * B>{});
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) {
      double2 t[B];
#pragma unroll
      for (int n2 = 0; n2 < B; ++n2) t[n2] = y[n2 * A + k1];
      DFT<B, SIGN>::run(t);
#pragma unroll
      for (int k2 = 0; k2 < B; ++k2) x[k1 + A * k2] = t[k2];
    }
  }
  template <int... I>
  __device__ static void twiddle_all(double2* y, std::integer_sequence<int, I...>) {
    (tw_one<I / A, I % A>(y), ...);
  }
};
template <int SIGN> struct DFT<6, SIGN> { __device__ static void run(double2* x) { DFT2F<3, 2, SIGN>::run(x); } };
template <int SIGN> struct DFT<9, SIGN> { __device__ static void run(double2* x) { DFT2F<3, 3, SIGN>::run(x); } };
template <int SIGN> struct DFT<10, SIGN> { __device__ static void run(double2* x) { DFT2F<5, 2, SIGN>::run(x); } };
template <int SIGN> struct DFT<15, SIGN> { __device__ static void run(double2* x) { DFT2F<5, 3, SIGN>::run(x); } };
template <int SIGN> struct DFT<12, SIGN> { __device__ static void run(double2* x) { DFT2F<3, 4, SIGN>::run(x); } };
template <int SIGN> struct DFT<16, SIGN> { __device__ static void run(double2* x) { DFT2F<4, 4, SIGN>::run(x); } };
template <int SIGN> struct DFT<24, SIGN> { __device__ static void run(double2* x) { DFT2F<3, 8, SIGN>::run(x); } };
template <int SIGN> struct DFT<1, SIGN> { __device__ static void run(double2*) {} };

#define KMHD_RADIX_SWITCH(R, CALL) \
  switch (R) {                     \
    case 2: CALL(2); break;        \
    case 3: CALL(3); break;        \
    case 4: CALL(4); break;        \
    case 5: CALL(5); break;        \
    case 6: CALL(6); break;        \
    case 8: CALL(8); break;        \
    case 9: CALL(9); break;        \
    case 10: CALL(10); break;      \
    case 12: CALL(12); break;      \
    case 15: CALL(15); break;      \
    default: CALL(16); break;      \
  }

// First inverse pass: sequence i is pair q0 + i dq of the line at line + i ls
// (block rows bs doubles apart, see spec_at).
template <int R>
__device__ __forceinline__ void dif_first(const Seqs Z, const Plan& P, const double* line, long long ls, long long bs,
                                          int nc, int q0, int dq) {
  const int N = Z.N, s = N / R;
  for (int it = threadIdx.x; it < Z.n * s; it += blockDim.x) {
    const int pp = it / s, j = it - pp * s;
    double2 x[R];
    const int q = q0 + pp * dq;
    const PairPos src(P, q, nc, P.nvb, P.mixb);
#pragma unroll
    for (int r = 0; r < R; ++r) x[r] = spec_at(P, line + pp * ls, bs, src, 2 * q + 1 < nc, j + r * s);
    DFT<R, +1>::run(x);
    double2* base = Z.z + pp * Z.zs;
    TwiddleRun<+1, kTwRun> tr(P.twid, j);
#pragma unroll
    for (int q = 0; q < R; ++q) base[Z.ix(j + q * s)] = q == 0 ? x[0] : cmul(x[q], tr.next(q));
  }
}
__device__ __noinline__ void dif_first_dispatch(const Seqs Z, const Plan& P, const double* line, long long ls,
                                                long long bs, int nc, int q0, int dq) {
#define KMHD_CALL(R) dif_first<R>(Z, P, line, ls, bs, nc, q0, dq)
  KMHD_RADIX_SWITCH(P.fac[0], KMHD_CALL)
#undef KMHD_CALL
}

// One in-place DIF (SIGN > 0: butterfly, then twiddle) or DIT (SIGN < 0, its
// transpose) pass of radix R over blocks of span entries.
template <int R, int SIGN>
__device__ __forceinline__ void mid_pass(const Seqs Z, int span, const double2* __restrict__ tw) {
  const int N = Z.N, s = span / R, nbf = N / R, stw = N / span;
  for (int it = threadIdx.x; it < Z.n * nbf; it += blockDim.x) {
    const int pp = it / nbf, rem = it - pp * nbf;
    const int b = rem / s, j = rem - b * s;
    double2* base = Z.z + pp * Z.zs;
    const int i0 = b * span + j;
    double2 x[R];
    if (s == 1) {  // one butterfly per block: every twiddle is 1
#pragma unroll
      for (int r = 0; r < R; ++r) x[r] = base[Z.ix(i0 + r)];
      DFT<R, SIGN>::run(x);
#pragma unroll
      for (int q = 0; q < R; ++q) base[Z.ix(i0 + q)] = x[q];
      continue;
    }
    TwiddleRun<SIGN, kTwRun> tr(tw, j * stw);
    if constexpr (SIGN > 0) {
#pragma unroll
      for (int r = 0; r < R; ++r) x[r] = base[Z.ix(i0 + r * s)];
      DFT<R, +1>::run(x);
#pragma unroll
      for (int q = 0; q < R; ++q) base[Z.ix(i0 + q * s)] = q == 0 ? x[0] : cmul(x[q], tr.next(q));
    } else {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const double2 v = base[Z.ix(i0 + r * s)];
        x[r] = r == 0 ? v : cmul(v, tr.next(r));
      }
      DFT<R, -1>::run(x);
#pragma unroll
      for (int q = 0; q < R; ++q) base[Z.ix(i0 + q * s)] = x[q];
    }
  }
}
__device__ __noinline__ void dif_dispatch(const Seqs Z, int R, int span, const double2* tw) {
#define KMHD_CALL(R) mid_pass<R, +1>(Z, span, tw)
  KMHD_RADIX_SWITCH(R, KMHD_CALL)
#undef KMHD_CALL
}
__device__ __noinline__ void dit_dispatch(const Seqs Z, int R, int span, const double2* tw) {
#define KMHD_CALL(R) mid_pass<R, -1>(Z, span, tw)
  KMHD_RADIX_SWITCH(R, KMHD_CALL)
#undef KMHD_CALL
}

// The inverse passes after the first, and every forward pass.
__device__ void dif_rest(const Seqs& Z, const Plan& P) {
  int span = Z.N / P.fac[0];
  for (int f = 1; f < P.nfac; ++f) {
    dif_dispatch(Z, P.fac[f], span, P.twid);
    __syncthreads();
    span /= P.fac[f];
  }
}
__device__ void dit_all(const Seqs& Z, const Plan& P) {
  int span = 1;
  for (int f = P.nfac - 1; f >= 0; --f) {
    span *= P.fac[f];
    dit_dispatch(Z, P.fac[f], span, P.twid);
    __syncthreads();
  }
}

// Stage the records of line (th, r) into st via cp.async (16 B each).
__device__ void prefetch_line(double* st, const double* rtm, int nc, const Plan& P, int th, int r) {
  const int row = rtm_row(P, nc);
  const long long bs = (long long)P.nth * P.nr * row;
  const double* base = rtm + rtm_off(P, 0, th, r, nc);
  const int per = row / 2, n = rtm_blocks(P) * per;
  for (int it = threadIdx.x; it < n; it += blockDim.x) {
    const int b = it / per, c = it - b * per;
    cp_async16(st + 2 * it, base + b * bs + 2 * c);
  }
  cp_async_commit();
}

// Forward records of one order of a pair: (a0, b0) of its first component at dx,
// (a1, b1) of its second at dy (two: it has one; split: not the same sector; al: sectors are aligned).
__device__ __forceinline__ void store_rec(double* dx, double* dy, bool two, bool split, bool al, double a0, double b0,
                                          double a1, double b1) {
  if (two && !split) {
    st_sector(dx, al, a0, b0, a1, b1);
  } else {
    *reinterpret_cast<double2*>(dx) = make_double2(a0, b0);
    if (two) *reinterpret_cast<double2*>(dy) = make_double2(a1, b1);
  }
}

// Records of order m from the natural-order forward spectrum of one pair:
// zm = z[m], wm = z[N - m].
__device__ __forceinline__ void store_pair(double* base, long long bs, const Plan& P, int m, int pp, int nc, bool al,
                                           double2 zm, double2 wm) {
  const double aN = 1.0 / (double)P.nph;
  double a0, b0, a1, b1;
  if (m == 0) {
    a0 = zm.x * aN; a1 = zm.y * aN; b0 = 0.0; b1 = 0.0;
  } else {
    a0 = (zm.x + wm.x) * aN;
    b0 = (wm.y - zm.y) * aN;
    a1 = (zm.y + wm.y) * aN;
    b1 = (zm.x - wm.x) * aN;
  }
  const PairPos dst(P, pp, nc, P.nvf, P.mixf);
  double* d = base + (m >> P.mbs) * bs;
  store_rec(d + dst.x(m), d + dst.y(m), 2 * pp + 1 < nc, dst.split, al, a0, b0, a1, b1);
}

// Natural-order forward spectra of the sequences -> records: sequence i is pair
// q0 + i dq of the line that starts at base + i ls.  Lanes take consecutive
// orders of one sequence: eight lanes write 256 contiguous bytes.
__device__ __forceinline__ void store_seqs(const Seqs& Z, const Plan& P, double* base, long long ls, int nc, int q0,
                                           int dq) {
  const int N = P.nph, L = P.L;
  const long long bs = (long long)P.nth * P.nr * rtm_row(P, nc);
  const bool al = rtm_aligned(P, nc);
  auto ix = [&](int i) { return Z.ix(i); };
  int m = threadIdx.x, pp = 0;
  for (int it = threadIdx.x; it < (L + 1) * Z.n; it += blockDim.x, m += blockDim.x) {
    while (m > L) { m -= L + 1; ++pp; }
    const double2* zp = Z.z + pp * Z.zs;
    store_pair(base + pp * ls, bs, P, m, q0 + pp * dq, nc, al, zp[ix(m)],
               m == 0 ? make_double2(0.0, 0.0) : zp[ix(N - m)]);
  }
}
// x[a], selected without dynamic register indexing.
template <int M>
__device__ __forceinline__ double selv(const double* x, int a) {
  double v = x[0];
#pragma unroll
  for (int q = 1; q < M; ++q)
    if (a == q) v = x[q];
  return v;
}

// Grid products of one point.  Backward vector v is (rr, th, ph)[v], scalar s
// is sc[s]; forward vector i goes to (orr, oth, oph)[i], scalar j to os[j].  MV*
// / MS* are compile-time maxima, the plan's counts (EX: equal to them) are <= them.
template <int MVB, int MSB, int MVF, int MSF, bool EX>
__device__ __forceinline__ void point_products(const double* rr, const double* th, const double* ph, const double* sc,
                                               const Plan& P, double* orr, double* oth, double* oph, double* os) {
  const int nvf = EX ? MVF : P.nvf, nsf = EX ? MSF : P.nsf;
#pragma unroll
  for (int i = 0; i < MVF; ++i) {
    if (i < nvf) {
      const double cf = P.pcoef[i];
      const int a = P.pa[i], b = P.pb[i];
      const double x0 = selv<MVB>(rr, a), x1 = selv<MVB>(th, a), x2 = selv<MVB>(ph, a);
      if (P.pkind[i] == KMHD_PROD_CROSS) {
        const double y0 = selv<MVB>(rr, b), y1 = selv<MVB>(th, b), y2 = selv<MVB>(ph, b);
        orr[i] = (x1 * y2 - x2 * y1) * cf;
        oth[i] = (x2 * y0 - x0 * y2) * cf;
        oph[i] = (x0 * y1 - x1 * y0) * cf;
      } else {
        const double s = selv<MSB>(sc, b);
        orr[i] = x0 * s * cf;
        oth[i] = x1 * s * cf;
        oph[i] = x2 * s * cf;
      }
    }
  }
#pragma unroll
  for (int j = 0; j < MSF; ++j) {
    if (j < nsf) {
      const int q = nvf + j;
      const double cf = P.pcoef[q];
      const int a = P.pa[q], b = P.pb[q];
      if (P.pkind[q] == KMHD_PROD_DOT) {
        os[j] = (selv<MVB>(rr, a) * selv<MVB>(rr, b) + selv<MVB>(th, a) * selv<MVB>(th, b) +
                 selv<MVB>(ph, a) * selv<MVB>(ph, b)) * cf;
      } else {
        os[j] = selv<MSB>(sc, a) * selv<MSB>(sc, b) * cf;
      }
    }
  }
}

// Product lists known at compile time (vector-valued products first): the
// field sets of the reference's MHD, convection and heat runs.  Where they have a
// mixed forward pair its scalar is a dot product (Plan::mixf = -1).  PK = 0: the
// plan's list, read at run time.
constexpr int kX = KMHD_PROD_CROSS, kVS = KMHD_PROD_VEC_SCALAR, kDot = KMHD_PROD_DOT;
struct ProdList {
  int nvb, nsb, nvf, nsf, n;
  int kind[6], a[6], b[6];
};
constexpr ProdList kProdLists[6] = {
    {},
    // u, omega, B + T -> omega x u, u x B, u T + u . omega
    {3, 1, 3, 1, 4, {kX, kX, kVS, kDot}, {1, 0, 0, 0}, {0, 2, 0, 1}},
    // u, omega, B, J + T -> omega x u, J x B, u x B, u T
    {4, 1, 4, 0, 4, {kX, kX, kX, kVS}, {1, 3, 0, 0}, {0, 2, 2, 0}},
    // u, omega, B, J + T, C -> omega x u, J x B, u x B, u T, u C + u . omega
    {4, 2, 5, 1, 6, {kX, kX, kX, kVS, kVS, kDot}, {1, 3, 0, 0, 0, 0}, {0, 2, 2, 0, 1, 1}},
    // u, omega + T -> omega x u, u T + u . omega
    {2, 1, 2, 1, 3, {kX, kVS, kDot}, {1, 0, 0}, {0, 0, 1}},
    // u + T -> u T
    {1, 1, 1, 0, 1, {kVS}, {0}, {0}}};

// the entry of kProdLists that is the plan's list, or 0
inline int prod_list(const Plan& p) {
  for (int k = 1; k < 6; ++k) {
    const ProdList& q = kProdLists[k];
    if (p.nvb != q.nvb || p.nsb != q.nsb || p.nvf != q.nvf || p.nsf != q.nsf || p.nprod != q.n) continue;
    bool same = true;
    for (int i = 0; i < q.n; ++i) same = same && p.pkind[i] == q.kind[i] && p.pa[i] == q.a[i] && p.pb[i] == q.b[i];
    if (same) return k;
  }
  return 0;
}

// point_products for list PK > 0.
template <int PK, int I = 0>
__device__ __forceinline__ void point_products_k(const double* rr, const double* th, const double* ph, const double* sc,
                                                 const Plan& P, double* orr, double* oth, double* oph, double* os) {
  constexpr ProdList q = kProdLists[PK];
  if constexpr (I < q.n) {
    constexpr int a = q.a[I], b = q.b[I];
    const double cf = P.pcoef[I];
    if constexpr (q.kind[I] == kX) {
      orr[I] = (th[a] * ph[b] - ph[a] * th[b]) * cf;
      oth[I] = (ph[a] * rr[b] - rr[a] * ph[b]) * cf;
      oph[I] = (rr[a] * th[b] - th[a] * rr[b]) * cf;
    } else if constexpr (q.kind[I] == kVS) {
      orr[I] = rr[a] * sc[b] * cf;
      oth[I] = th[a] * sc[b] * cf;
      oph[I] = ph[a] * sc[b] * cf;
    } else {
      os[I - q.nvf] = (rr[a] * rr[b] + th[a] * th[b] + ph[a] * ph[b]) * cf;
    }
    point_products_k<PK, I + 1>(rr, th, ph, sc, P, orr, oth, oph, os);
  }
}

// Pointwise products on the digit-reversed grid (sequence zs entries apart),
// backward pairs in, forward pairs out (pairs: see rtm_off, mixed_pair); PK: the
// product list (0: the plan's).
template <int PK>
__device__ __forceinline__ void products(double2* z, int zs, int N, const Plan& P) {
  constexpr ProdList q = kProdLists[PK];
  constexpr int MVB = PK ? q.nvb : kMaxVec, MSB = PK ? q.nsb : kMaxScl, MVF = PK ? q.nvf : kMaxVec,
                MSF = PK ? q.nsf : kMaxScl;
  const int nvb = PK ? MVB : P.nvb, nsb = PK ? MSB : P.nsb, nvf = PK ? MVF : P.nvf, nsf = PK ? MSF : P.nsf;
  const bool mixb = PK ? mixed_pair(MVB, MSB) >= 0 : P.mixb >= 0, mixf = PK ? false : P.mixf >= 0;
  for (int pos = threadIdx.x; pos < N; pos += blockDim.x) {
    constexpr int VB = MVB > 0 ? MVB : 1, SB = MSB > 0 ? MSB : 1, VF = MVF > 0 ? MVF : 1, SF = MSF > 0 ? MSF : 1;
    double rr[VB] = {}, th[VB] = {}, ph[VB] = {}, sc[SB] = {};
    double orr[VF] = {}, oth[VF] = {}, oph[VF] = {}, os[SF] = {};
    // list entry f of the pairs that start at pair nv
    auto entry = [&](int nv, int f) { return reinterpret_cast<double*>(z + (nv + (f >> 1)) * zs + pos) + (f & 1); };
#pragma unroll
    for (int v = 0; v < MVB; ++v)
      if (v < nvb) {
        const double2 w = z[v * zs + pos];
        const double e = *entry(nvb, v);
        const bool sp = mixb && v == nvb - 1;  // (r, phi), (theta, scalar)
        rr[v] = sp ? w.x : e;
        th[v] = sp ? e : w.x;
        ph[v] = w.y;
      }
#pragma unroll
    for (int k = 0; k < MSB; ++k)
      if (k < nsb) sc[k] = *entry(nvb, nvb + k);
    if constexpr (PK > 0) point_products_k<PK>(rr, th, ph, sc, P, orr, oth, oph, os);
    else point_products<MVB, MSB, MVF, MSF, false>(rr, th, ph, sc, P, orr, oth, oph, os);
#pragma unroll
    for (int v = 0; v < MVF; ++v)
      if (v < nvf) {
        const bool sp = mixf && v == nvf - 1;
        z[v * zs + pos] = make_double2(sp ? orr[v] : oth[v], oph[v]);
        *entry(nvf, v) = sp ? oth[v] : orr[v];
      }
#pragma unroll
    for (int k = 0; k < MSF; ++k)
      if (k < nsf) *entry(nvf, nvf + k) = os[k];
    if ((nvf + nsf) & 1) *entry(nvf, nvf + nsf) = 0.0;
  }
}

template <int PK>
__global__ void __launch_bounds__(kFftThreads) k_fft_cycle(const __grid_constant__ Plan P, int line0, int nlines) {
  extern __shared__ double4 smraw[];
  const int N = P.nph;
  const int npb = (P.ncb + 1) / 2, npf = (P.ncf + 1) / 2;
  const int npair = npb > npf ? npb : npf;
  double2* z = reinterpret_cast<double2*>(smraw);
  double* st = reinterpret_cast<double*>(z + npair * N);
  const Seqs ZB(z, npb, N, N), ZF(z, npf, N, N);
  int line = line0 + blockIdx.x;
  if (line >= nlines) return;
  prefetch_line(st, P.rtm_b, P.ncb, P, line % P.nth, line / P.nth);
  while (line < nlines) {
    const int th = line % P.nth, r = line / P.nth;
    cp_async_wait<0>();
    __syncthreads();
    dif_first_dispatch(ZB, P, st, 0, rtm_row(P, P.ncb), P.ncb, 0, 1);
    __syncthreads();
    const int next = line + gridDim.x;
    if (next < nlines) prefetch_line(st, P.rtm_b, P.ncb, P, next % P.nth, next / P.nth);
    dif_rest(ZB, P);
    products<PK>(z, N, N, P);
    __syncthreads();
    dit_all(ZF, P);
    store_seqs(ZF, P, P.rtm_f + rtm_off(P, 0, th, r, P.ncf), 0, P.ncf, 0, 1);
    __syncthreads();
    line = next;
  }
}

// Lines whose grid fits in shared memory but not together with the staged
// spectra of the next line (many fields, e.g. 14 + 16 components at
// Nphi = 1536: 197 KB of grid pairs): the first pass reads the line's spectra
// in place from the rtm records, everything else as k_fft_cycle.
template <int PK>
__global__ void __launch_bounds__(kFftThreads) k_fft_cycle_direct(const __grid_constant__ Plan P, int line0, int nlines) {
  extern __shared__ double4 smraw[];
  const int N = P.nph;
  double2* z = reinterpret_cast<double2*>(smraw);
  const Seqs ZB(z, (P.ncb + 1) / 2, N, N), ZF(z, (P.ncf + 1) / 2, N, N);
  const long long bs = (long long)P.nth * P.nr * rtm_row(P, P.ncb);
  for (int line = line0 + blockIdx.x; line < nlines; line += gridDim.x) {
    const int th = line % P.nth, r = line / P.nth;
    dif_first_dispatch(ZB, P, P.rtm_b + rtm_off(P, 0, th, r, P.ncb), 0, bs, P.ncb, 0, 1);
    __syncthreads();
    dif_rest(ZB, P);
    products<PK>(z, N, N, P);
    __syncthreads();
    dit_all(ZF, P);
    store_seqs(ZF, P, P.rtm_f + rtm_off(P, 0, th, r, P.ncf), 0, P.ncf, 0, 1);
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Wide lines (one line of every component does not fit in shared memory, e.g.
// Nphi = 3072 with 10 components): the pairs go through shared memory one at a
// time.  The cycle keeps the line's grid in a per-CTA global scratch
// (pairs x N x 16 bytes, L2-resident), forms the products there and runs the
// forward transforms pair by pair from it.
template <int PK>
__global__ void __launch_bounds__(kFftThreads) k_fft_cycle_wide(const __grid_constant__ Plan P, int line0, int nlines) {
  extern __shared__ double4 smraw[];
  const int N = P.nph;
  const int npb = (P.ncb + 1) / 2, npf = (P.ncf + 1) / 2;
  const int npm = npb > npf ? npb : npf;
  double2* z = reinterpret_cast<double2*>(smraw);
  double2* sc = P.fft_scratch + (long long)blockIdx.x * npm * N;
  const Seqs Z(z, 1, N, N);
  // the first pass reads the line's spectra in place (rtm records, block rows
  // bs apart): one line of a wide grid is too large to stage, and a small
  // CTA keeps several resident per SM
  const long long bs = (long long)P.nth * P.nr * rtm_row(P, P.ncb);
  for (int line = line0 + blockIdx.x; line < nlines; line += gridDim.x) {
    const int th = line % P.nth, r = line / P.nth;
    const double* st = P.rtm_b + rtm_off(P, 0, th, r, P.ncb);
    for (int pp = 0; pp < npb; ++pp) {
      dif_first_dispatch(Z, P, st, 0, bs, P.ncb, pp, 0);
      __syncthreads();
      dif_rest(Z, P);
      for (int i = threadIdx.x; i < N; i += blockDim.x) sc[(long long)pp * N + i] = z[i];
      __syncthreads();
    }
    products<PK>(sc, N, N, P);
    __syncthreads();
    for (int q = 0; q < npf; ++q) {
      for (int i = threadIdx.x; i < N; i += blockDim.x) z[i] = sc[(long long)q * N + i];
      __syncthreads();
      dit_all(Z, P);
      store_seqs(Z, P, P.rtm_f + rtm_off(P, 0, th, r, P.ncf), 0, P.ncf, q, 0);
      __syncthreads();
    }
  }
}

constexpr int kGridThreads = 256;  // separable kernels: at most, at 128 registers

// Component of part c (0, 1) of FFT pair pp (mixed: see mixed_pair).
__device__ __forceinline__ int pair_comp(int pp, int c, int nv, int mixed) {
  if (mixed >= 0 && pp == nv - 1) return 3 * pp + 2 * c;
  if (pp == mixed) return c ? 3 * nv : 3 * nv - 2;
  if (pp < nv) return 3 * pp + 1 + c;
  const int f = 2 * (pp - nv) + c;
  return f < nv ? 3 * f : 2 * nv + f;
}

// Separable transforms between the spectra and the grid field[node + nnod c],
// node = r + nr (th + nth phi).  No product couples the components, so one CTA
// takes one pair of rad neighbouring radii of one latitude: its grid accesses
// are rad contiguous doubles (with one radius per CTA every lane of a grid
// access was a sector of its own: at L = 127, Nr = 65 the inverse took 0.65 ms
// and the forward 0.52 ms, now 0.35 and 0.33).  Sequences lie
// N + 1 entries apart, so the radii of one point are in different banks.
// Block order: pair fastest, then radial block, then latitude.
__global__ void __launch_bounds__(kGridThreads, 2)
    k_fft_bwd_grid(const __grid_constant__ Plan P, double* __restrict__ fld, int lrad) {
  const int rad = 1 << lrad;
  extern __shared__ double4 smraw[];
  const int N = P.nph, npb = (P.ncb + 1) / 2, nrb = (P.nr + rad - 1) / rad;
  const int q = blockIdx.x % npb, rest = blockIdx.x / npb;
  const int r0 = (rest % nrb) * rad, th = rest / nrb;
  const int nrad = min(rad, P.nr - r0);
  const Seqs Z(reinterpret_cast<double2*>(smraw), nrad, N + 1, N);
  const long long ls = (long long)P.nth * rtm_row(P, P.ncb);
  dif_first_dispatch(Z, P, P.rtm_b + rtm_off(P, 0, th, r0, P.ncb), ls, ls * P.nr, P.ncb, q, 0);
  __syncthreads();
  dif_rest(Z, P);
  const long long nnod = (long long)P.nr * P.nth * N;
  const bool two = 2 * q + 1 < P.ncb;
  const int mixed = P.mixb;
  double* f0 = fld + nnod * pair_comp(q, 0, P.nvb, mixed) + r0 + (long long)P.nr * th;
  double* f1 = two ? fld + nnod * pair_comp(q, 1, P.nvb, mixed) + r0 + (long long)P.nr * th : nullptr;
  const long long ps = (long long)P.nr * P.nth;
#pragma unroll 4
  for (int it = threadIdx.x; it < N << lrad; it += blockDim.x) {
    const int r = it & (rad - 1), pos = it >> lrad;
    if (r >= nrad) continue;
    const long long o = ps * __ldg(P.digrev + pos) + r;
    const double2 v = Z.z[r * Z.zs + Z.ix(pos)];
    f0[o] = v.x;
    if (two) f1[o] = v.y;
  }
}
__global__ void __launch_bounds__(kGridThreads, 2)
    k_fft_fwd_grid(const __grid_constant__ Plan P, const double* __restrict__ frc, int lrad) {
  const int rad = 1 << lrad;
  extern __shared__ double4 smraw[];
  const int N = P.nph, npf = (P.ncf + 1) / 2, nrb = (P.nr + rad - 1) / rad;
  const int q = blockIdx.x % npf, rest = blockIdx.x / npf;
  const int r0 = (rest % nrb) * rad, th = rest / nrb;
  const int nrad = min(rad, P.nr - r0);
  const Seqs Z(reinterpret_cast<double2*>(smraw), nrad, N + 1, N);
  const long long nnod = (long long)P.nr * P.nth * N;
  const bool two = 2 * q + 1 < P.ncf;
  const int mixed = P.mixf;
  const double* __restrict__ f0 = frc + nnod * pair_comp(q, 0, P.nvf, mixed) + r0 + (long long)P.nr * th;
  const double* __restrict__ f1 = two ? frc + nnod * pair_comp(q, 1, P.nvf, mixed) + r0 + (long long)P.nr * th : nullptr;
  const long long ps = (long long)P.nr * P.nth;
  // eight grid loads of a thread in flight
  constexpr int U = 4;
  for (int it = threadIdx.x; it < N << lrad; it += U * blockDim.x) {
    double lo[U], hi[U];
    int ix[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int e = it + u * blockDim.x, r = e & (rad - 1), pos = e >> lrad;
      ix[u] = e < N << lrad && r < nrad ? r * Z.zs + Z.ix(pos) : -1;
      const long long o = ix[u] >= 0 ? ps * __ldg(P.digrev + pos) + r : 0;
      lo[u] = __ldg(f0 + o);
      hi[u] = two ? __ldg(f1 + o) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (ix[u] >= 0) Z.z[ix[u]] = make_double2(lo[u], hi[u]);
  }
  __syncthreads();
  dit_all(Z, P);
  store_seqs(Z, P, P.rtm_f + rtm_off(P, 0, th, r0, P.ncf), (long long)P.nth * rtm_row(P, P.ncf), P.ncf, q, 0);
}

// ---------------------------------------------------------------------------
// bytes of one staged line
size_t staged_bytes(const Plan& p) { return sizeof(double) * (size_t)rtm_blocks(p) * rtm_row(p, p.ncb); }

size_t smem_cycle_f(const Plan& p) {
  const int npair = ((p.ncb > p.ncf ? p.ncb : p.ncf) + 1) / 2;
  // grid pairs, alignment of the staging to 128 bytes, staged spectra, mbarrier
  return sizeof(double2) * ((size_t)npair * (p.nph + 1)) + 128 + staged_bytes(p) + 16;
}

// ---------------------------------------------------------------------------
// Fused-pass variant for N = F0 * M * 4 (F0 in {3, 6, 12, 24}, M in {4, 16}):
// inverse passes radix F0 (reading the staged spectra), radix M, radix 4; the
// last inverse radix-4 pass, the grid products and the first forward radix-4
// pass share one item (4 grid points of every component in registers), so a
// line takes five sweeps over shared memory instead of nine.  The radix-4
// passes of span 4 carry no twiddles.  Swizzle i -> i ^ (((i >> 3) ^ (i >> 6))
// & 7) inside each pair sequence (pairs N + 1 entries apart) keeps every
// quarter warp on 8 distinct 16-byte bank groups in all passes at N = 1536.
constexpr int kFftThreadsF = 384;

// Threads of one staged CTA.  Every variant fills the register file
// (168 registers x 384 threads per SM): at N = 1536 one line takes the whole
// shared memory, so one CTA has them all; the shorter lines leave room for
// several CTAs per SM, whose barriers and record stores then overlap, and a
// pass of theirs has fewer items than 384 threads could take (N / F0 or N / M
// per pair).  FFT ms at 384 threads -> here: L = 255, Nr = 129 (N = 768) 2.04 ->
// 1.75; L = 127, Nr = 65 (N = 384) 0.306 -> 0.234; L = 63, Nr = 65 (N = 192) 0.118 ->
// 0.071; L = 31, Nr = 33 (N = 96) 0.027 -> 0.015.  (160, 128, 96 and 64 threads were
// slower than these, before the passes were rebuilt.)
__host__ __device__ constexpr int ff_threads(int n) { return n == 768 ? 192 : n == 384 ? 96 : n == 192 ? 64 : n == 96 ? 32 : kFftThreadsF; }

__host__ __device__ constexpr int ff_mid(int n) { return (n % 64 == 0 && (n / 64 == 3 || n / 64 == 6 || n / 64 == 12 || n / 64 == 24)) ? 16 : 4; }
__host__ __device__ constexpr int ff_first(int n) { return n / (4 * ff_mid(n)); }
__device__ __forceinline__ int swf(int i) { return i ^ (((i >> 3) ^ (i >> 6)) & 7); }

// DFT of length 3B whose middle third of inputs (n = B .. 2B-1) is zero: the
// first-stage length-3 transforms see (x0, 0, x2).
template <int A, int B, int SIGN>
struct DFT2F_ZM;
template <int B, int SIGN>
struct DFT2F_ZM<3, B, SIGN> {
  template <int N2, int K1>
  __device__ static void tw_one(double2* y) {
    y[N2 * 3 + K1] = rot<3 * B, N2 * K1, SIGN>(y[N2 * 3 + K1]);
  }
  template <int... I>
  __device__ static void twiddle_all(double2* y, std::integer_sequence<int, I...>) {
    (tw_one<I / 3, I % 3>(y), ...);
  }
  __device__ static void run(double2* x) {
    const double s3 = 0.86602540378443864676 * (double)SIGN;
    double2 y[3 * B];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) {
      const double2 a = x[n2], c = x[2 * B + n2];
      const double2 v = make_double2(a.x - 0.5 * c.x, a.y - 0.5 * c.y);
      const double2 u = make_double2(c.y * s3, -c.x * s3);  // -(SIGN i sqrt3/2) c
      y[n2 * 3 + 0] = cadd(a, c);
      y[n2 * 3 + 1] = cadd(v, u);
      y[n2 * 3 + 2] = csub(v, u);
    }
    twiddle_all(y, std::make_integer_sequence<int, 3 * B>{});
#pragma unroll
    for (int k1 = 0; k1 < 3; ++k1) {
      double2 t[B];
#pragma unroll
      for (int n2 = 0; n2 < B; ++n2) t[n2] = y[n2 * 3 + k1];
      DFT<B, SIGN>::run(t);
#pragma unroll
      for (int k2 = 0; k2 < B; ++k2) x[k1 + 3 * k2] = t[k2];
    }
  }
};

// Shared-memory index of entry i of a pair sequence: swf(i).  The passes below
// compute it with the bits that are compile-time constants folded out.
//
// First inverse pass: radix F0 over the whole line (span N, stride S1 = N/F0),
// inputs from the staged spectra.  Twiddles w^(j q) are read straight from the
// table (j q < N here).  When N = 3 (L + 1) (PR), the middle third of the
// inputs (L < k < N - L) is zero and the outer thirds need no range checks.
// line / bs: the line's block rows, staged or in place (see spec_at).
template <int N, bool PR, bool INPLACE = false>
__device__ __forceinline__ void ff_dif_first(const Plan& P, const double* line, long long bs, int nc, int nv, int mixed,
                                             double2* z, int npair, const double2* __restrict__ tw) {
  constexpr int R = ff_first(N), S1 = N / R, NP = N + 1, T3 = R / 3;
  for (int it = threadIdx.x; it < npair * S1; it += blockDim.x) {
    const int pp = it / S1, j = it - pp * S1;
    double2 x[R];
    if constexpr (PR) {
      // N = 3 (L + 1), S1 = (L + 1) / T3: input r < T3 is order m = j + r S1
      // (m = 0 only at j = r = 0); input r >= 2 T3 is the mirror of order
      // m = N - j - r S1 (m = L + 1, a zero, only at j = 0, r = 2 T3).  S1 and
      // N are multiples of the block's orders, so the inputs of one thread are
      // whole block rows apart.
      static_assert(S1 % kRtmOrders == 0, "orders per rtm block");
      const bool two = 2 * pp + 1 < nc;  // the pair holds two components
      const PairPos src(P, pp, nc, nv, mixed);
      int ux = src.x(j), uy = src.y(j), dx = src.x(-j), dy = src.y(-j);
      const double* up = line + (j >> kRtmShift) * bs;
      const double* dn = line + ((-j) >> kRtmShift) * bs;
      // staged sectors lie 32 bytes apart: lanes 4..7 of each eight read the
      // second half first, so a quarter warp covers all banks (a split pair's
      // components are the two halves of two sectors)
      const bool hu = !INPLACE && two && (j & 4), hd = !INPLACE && two && ((-j) & 4);
      if (!two) uy = ux, dy = dx;
      const int u0 = hu ? uy : ux, u1 = hu ? ux : uy, d0 = hd ? dy : dx, d1 = hd ? dx : dy;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        if (r >= T3 && r < 2 * T3) {
          x[r] = make_double2(0.0, 0.0);
          continue;
        }
        const bool mir = r >= 2 * T3;
        if (mir && r == 2 * T3 && j == 0) {  // order L + 1
          x[r] = make_double2(0.0, 0.0);
          continue;
        }
        const double* s = mir ? dn + ((N - r * S1) / kRtmOrders) * bs : up + ((r * S1) / kRtmOrders) * bs;
        double2 c0 = *reinterpret_cast<const double2*>(s + (mir ? d0 : u0));
        double2 c1 = two ? *reinterpret_cast<const double2*>(s + (mir ? d1 : u1)) : make_double2(0.0, 0.0);
        if (!INPLACE && (mir ? hd : hu)) {
          const double2 t = c0;
          c0 = c1;
          c1 = t;
        }
        if (mir) {
          x[r] = make_double2(0.5 * c0.x - 0.5 * c1.y, 0.5 * c0.y + 0.5 * c1.x);
        } else {
          x[r] = (r == 0 && j == 0) ? make_double2(c0.x, c1.x)
                                    : make_double2(0.5 * c0.x + 0.5 * c1.y, 0.5 * c1.x - 0.5 * c0.y);
        }
      }
      DFT2F_ZM<3, T3, +1>::run(x);
    } else {
      const PairPos src(P, pp, nc, nv, mixed);
#pragma unroll
      for (int r = 0; r < R; ++r) x[r] = spec_at(P, line, bs, src, 2 * pp + 1 < nc, j + r * S1);
      DFT<R, +1>::run(x);
    }
    double2* zp = z + pp * NP;
    TwiddleRun<+1, kTwSpecial> tr(tw, j);
    if constexpr (S1 % 64 == 0) {
      const int jj = j ^ ((j >> 3) & 7);
#pragma unroll
      for (int q = 0; q < R; ++q) {
        const double2 v = q == 0 ? x[0] : cmul(x[q], tr.next(q));
        zp[(jj ^ (((q * S1) >> 6) & 7)) + q * S1] = v;
      }
    } else {
#pragma unroll
      for (int q = 0; q < R; ++q) zp[swf(j + q * S1)] = q == 0 ? x[0] : cmul(x[q], tr.next(q));
    }
  }
}

// Last forward pass (transpose of ff_dif_first, radix F0 over the whole line)
// and the record stores.  Butterfly j holds the frequencies j + q S1; order m =
// j + q S1 needs them and N - m = (S1 - j) + (F0 - 1 - q) S1, which butterfly
// S1 - j holds: the lanes are arranged so that j and S1 - j share a warp and
// the mirrors come by shuffles.  The outputs never return to shared memory
// (separate passes for the butterflies and the stores took 4.0k + 3.5k of a
// line's 28k cycles at N = 1536), and eight lanes store 256 contiguous bytes.
// With PR (N = 3 (L + 1)) only the outer thirds of the output are orders or
// mirrors.
template <int N, bool PR>
__device__ __forceinline__ void ff_dit_store(const double2* z, int npair, const Plan& P, double* base, long long bs,
                                             int nc, int nv, int mixed, const double2* __restrict__ tw) {
  constexpr int R = ff_first(N), S1 = N / R, NP = N + 1;
  constexpr int QM = PR ? R / 3 : (R + 1) / 2;  // orders j + q S1 <= L < N / 2 have q < QM
  static_assert(S1 == 64 || S1 == 16, "lane arrangement");
  const int lane = threadIdx.x & 31, L = P.L;
  for (int w0 = threadIdx.x - lane; w0 < npair * S1; w0 += blockDim.x) {
    int pp, j, mate;  // mate: the lane of butterfly S1 - j (itself for j = 0, S1 / 2)
    if constexpr (S1 == 64) {
      pp = w0 / S1;
      if ((w0 & 32) == 0) {  // 0 .. 15, 63 .. 49, 32
        j = lane < 16 ? lane : lane == 31 ? 32 : 79 - lane;
        mate = lane == 0 || lane == 31 ? lane : lane < 16 ? lane + 15 : lane - 15;
      } else {  // 16 .. 31, 48 .. 33
        j = lane < 16 ? 16 + lane : 64 - lane;
        mate = lane ^ 16;
      }
    } else {
      pp = (w0 + lane) / S1;
      j = lane & 15;
      mate = (lane & 16) | ((16 - j) & 15);
    }
    const bool ok = pp < npair;
    const double2* zp = z + (ok ? pp : 0) * NP;
    double2 x[R];
    TwiddleRun<-1, kTwSpecial> tr(tw, j);
    const int jj = j ^ ((j >> 3) & 7);
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const double2 v = S1 % 64 == 0 ? zp[(jj ^ (((q * S1) >> 6) & 7)) + q * S1] : zp[swf(j + q * S1)];
      x[q] = q == 0 ? v : cmul(v, tr.next(q));
    }
    DFT<R, -1>::run(x);
    const bool two = 2 * pp + 1 < nc;
    const PairPos dst(P, pp, nc, nv, mixed);
    double* dx = base + (j >> kRtmShift) * bs + dst.x(j);
    double* dy = base + (j >> kRtmShift) * bs + dst.y(j);
    const double aN = 1.0 / (double)N;
#pragma unroll
    for (int q = 0; q < QM; ++q) {
      double2 wm;
      wm.x = __shfl_sync(0xffffffffu, x[R - 1 - q].x, mate);
      wm.y = __shfl_sync(0xffffffffu, x[R - 1 - q].y, mate);
      if (q > 0 && j == 0) wm = x[R - q];
      const double2 zm = x[q];
      const bool m0 = q == 0 && j == 0;
      if (!ok || (!PR && j + q * S1 > L)) continue;
      const long long o = (q * S1 / kRtmOrders) * bs;
      const double a0 = m0 ? zm.x * aN : (zm.x + wm.x) * aN, b0 = m0 ? 0.0 : (wm.y - zm.y) * aN;
      const double a1 = m0 ? zm.y * aN : (zm.y + wm.y) * aN, b1 = m0 ? 0.0 : (zm.x - wm.x) * aN;
      store_rec(dx + o, dy + o, two, dst.split, true, a0, b0, a1, b1);
    }
  }
}

// Middle pass of radix M over span SP = N/F0 (stride SP/M = 4): butterfly
// block b fastest across threads.  For SP = 64 the swizzle of element r is
// ((j + 4r) ^ (r/2) ^ (b % 8)) within the block, j < 4.
template <int N, int SIGN, int TS = 1>
__device__ __forceinline__ void ff_mid_pass(double2* z, int npair, const double2* __restrict__ tw) {
  constexpr int R = ff_mid(N), SP = N / ff_first(N), s = SP / R, nbf = N / R, NB = N / SP, stw = TS * (N / SP);  // TS: entries of tw per w_N
  constexpr int NP = N + 1;
  for (int it = threadIdx.x; it < npair * nbf; it += blockDim.x) {
    const int pp = it / nbf, rem = it - pp * nbf;
    const int b = rem % NB, j = rem / NB;
    double2* zp = z + pp * NP + b * SP;
    double2 x[R];
    if constexpr (SP == 64 && s == 4) {
      // element e = 4r + j (j < 4): e >> 3 = r / 2, so swf gives
      // 8 (r / 2) + ((j ^ (b % 8)) ^ (r / 2) ^ 4 (r % 2))
      const int jb = j ^ (b & 7);
#define KMHD_MIDX(r) (8 * ((r) >> 1) + (jb ^ (((r) >> 1) ^ (4 * ((r) & 1)))))
      if constexpr (SIGN > 0) {
#pragma unroll
        for (int r = 0; r < R; ++r) x[r] = zp[KMHD_MIDX(r)];
        DFT<R, +1>::run(x);
#pragma unroll
        for (int q = 0; q < R; ++q) zp[KMHD_MIDX(q)] = q == 0 ? x[0] : cmul(x[q], twd<+1>(tw, j * q * stw));
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const double2 v = zp[KMHD_MIDX(r)];
          x[r] = r == 0 ? v : cmul(v, twd<-1>(tw, j * r * stw));
        }
        DFT<R, -1>::run(x);
#pragma unroll
        for (int q = 0; q < R; ++q) zp[KMHD_MIDX(q)] = x[q];
      }
#undef KMHD_MIDX
    } else {
      if constexpr (SIGN > 0) {
#pragma unroll
        for (int r = 0; r < R; ++r) x[r] = z[pp * NP + swf(b * SP + j + r * s)];
        DFT<R, +1>::run(x);
#pragma unroll
        for (int q = 0; q < R; ++q)
          z[pp * NP + swf(b * SP + j + q * s)] = q == 0 ? x[0] : cmul(x[q], twd<+1>(tw, j * q * stw));
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const double2 v = z[pp * NP + swf(b * SP + j + r * s)];
          x[r] = r == 0 ? v : cmul(v, twd<-1>(tw, j * r * stw));
        }
        DFT<R, -1>::run(x);
#pragma unroll
        for (int q = 0; q < R; ++q) z[pp * NP + swf(b * SP + j + q * s)] = x[q];
      }
    }
  }
}

// Last inverse radix-4 pass + products + first forward radix-4 pass, for the
// grid points 4b .. 4b+3 of every pair.  Register slots: pair v < MV is slot
// v, list pair k is slot MV + k (at pair nv + k of z).  EX: the plan's counts
// equal the template's.
template <int N, int MVB, int MSB, int MVF, int MSF, bool EX, int PK>
__device__ __forceinline__ void ff_fused(double2* z, const Plan& P) {
  constexpr int NP = N + 1;
  constexpr int VB = MVB > 0 ? MVB : 1, SB = MSB > 0 ? MSB : 1, VF = MVF > 0 ? MVF : 1, SF = MSF > 0 ? MSF : 1;
  constexpr int FB = MVB + MSB, FF = MVF + MSF;                     // list entries
  constexpr int NPB = MVB + (FB + 1) / 2, NPF = MVF + (FF + 1) / 2;  // register slots
  constexpr int NPM = NPB > NPF ? NPB : NPF;
  const int nvb = EX ? MVB : P.nvb, nvf = EX ? MVF : P.nvf;
  const int nlb = EX ? (FB + 1) / 2 : (P.nvb + P.nsb + 1) / 2, nlf = EX ? (FF + 1) / 2 : (P.nvf + P.nsf + 1) / 2;
  const int nff = EX ? FF : P.nvf + P.nsf;
  const bool mixb = (EX ? mixed_pair(MVB, MSB) : P.mixb) >= 0, mixf = PK > 0 ? false : P.mixf >= 0;
  for (int b = threadIdx.x; b < N / 4; b += blockDim.x) {
    const int e0 = (4 * b) ^ (((b >> 1) ^ (b >> 4)) & 7);  // swf(4b + r) = e0 ^ r
    double2 v[NPM][4];
#pragma unroll
    for (int s = 0; s < NPB; ++s) {
      if (s < MVB ? s < nvb : s - MVB < nlb) {
        const double2* zp = z + (s < MVB ? s : nvb + s - MVB) * NP;
#pragma unroll
        for (int r = 0; r < 4; ++r) v[s][r] = zp[e0 ^ r];
        DFT<4, +1>::run(v[s]);
      } else {
#pragma unroll
        for (int r = 0; r < 4; ++r) v[s][r] = make_double2(0.0, 0.0);
      }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      double rr[VB] = {}, th[VB] = {}, ph[VB] = {}, sc[SB] = {};
      double orr[VF] = {}, oth[VF] = {}, oph[VF] = {}, os[SF] = {};
      auto lst = [&](int f) { return (f & 1) ? v[MVB + f / 2][r].y : v[MVB + f / 2][r].x; };
#pragma unroll
      for (int q = 0; q < MVB; ++q) {
        const bool sp = mixb && q == nvb - 1;  // (r, phi), (theta, scalar)
        rr[q] = sp ? v[q][r].x : lst(q);
        th[q] = sp ? lst(q) : v[q][r].x;
        ph[q] = v[q][r].y;
      }
#pragma unroll
      for (int q = 0; q < MSB; ++q) {
        if constexpr (EX) {
          sc[q] = lst(MVB + q);
        } else {
#pragma unroll
          for (int f = 0; f < FB; ++f)
            if (f == nvb + q) sc[q] = lst(f);
        }
      }
      if constexpr (PK > 0) point_products_k<PK>(rr, th, ph, sc, P, orr, oth, oph, os);
      else point_products<MVB, MSB, MVF, MSF, EX>(rr, th, ph, sc, P, orr, oth, oph, os);
      // forward list entry f: r of a vector (theta in the mixed pair), scalar or (odd count) zero
      auto out = [&](int f) {
        const int c = f < MVF ? f : 0;
        const double ve = mixf && f == nvf - 1 ? oth[c] : orr[c];
        if (EX) return f < MVF ? ve : f < FF ? os[f < MVF ? 0 : (f < FF ? f - MVF : 0)] : 0.0;
        double x = f < nvf && f < MVF ? ve : 0.0;
#pragma unroll
        for (int q = 0; q < MSF; ++q)
          if (f == nvf + q && f < nff) x = os[q];
        return x;
      };
#pragma unroll
      for (int q = 0; q < MVF; ++q) v[q][r] = make_double2(mixf && q == nvf - 1 ? orr[q] : oth[q], oph[q]);
#pragma unroll
      for (int k = 0; k < (FF + 1) / 2; ++k) v[MVF + k][r] = make_double2(out(2 * k), out(2 * k + 1));
    }
#pragma unroll
    for (int s = 0; s < NPF; ++s) {
      if (s < MVF ? s < nvf : s - MVF < nlf) {
        DFT<4, -1>::run(v[s]);
        double2* zp = z + (s < MVF ? s : nvf + s - MVF) * NP;
#pragma unroll
        for (int r = 0; r < 4; ++r) zp[e0 ^ r] = v[s][r];
      }
    }
  }
}

// shared memory of half a line
size_t smem_half(const Plan& p) {
  const int npair = ((p.ncb > p.ncf ? p.ncb : p.ncf) + 1) / 2;
  return sizeof(double2) * (size_t)npair * (p.nph / 2 + 1);
}

// cuTensorMapEncodeTiled, resolved through the runtime (no link-time
// dependency on the driver library, so the library also loads on hosts
// without a GPU driver); null when unavailable.
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn encode_tiled() {
  static const EncodeTiledFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      return static_cast<EncodeTiledFn>(nullptr);
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  return fn;
}

// Boxes of a line: a box has at most 256 doubles along the block row (16
// components; 17, the most there are, take two).
__host__ __device__ constexpr int line_boxes(int row) { return row > 256 ? 2 : 1; }

// Tensor map of rtm_b for k_fft_cycle_f and _half: [block][r][theta][block row],
// box (block row or half of it, 1, 1, all blocks).  False when a line is not
// line_boxes() boxes (the caller then takes a kernel without the map).
bool make_rtm_map(const Plan& p, CUtensorMap* map) {
  const int row = rtm_row(p, p.ncb), nblk = rtm_blocks(p), nx = row / line_boxes(row);
  if (nx > 256 || nblk > 256 || !p.rtm_b) return false;
  const cuuint64_t dims[4] = {(cuuint64_t)row, (cuuint64_t)p.nth, (cuuint64_t)p.nr, (cuuint64_t)nblk};
  const cuuint64_t strides[3] = {8ull * row, 8ull * row * p.nth, 8ull * row * p.nth * p.nr};
  const cuuint32_t box[4] = {(cuuint32_t)nx, 1, 1, (cuuint32_t)nblk};
  const cuuint32_t es[4] = {1, 1, 1, 1};
  const EncodeTiledFn enc = encode_tiled();
  if (!enc) return false;
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 4, const_cast<double*>(p.rtm_b), dims, strides, box, es,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// L2 prefetch of a line's spectra (row: its block row); x of the second box is a
// multiple of 16 bytes
__device__ __forceinline__ void prefetch_l2(const CUtensorMap& tmap, int row, int th, int r) {
  const int nx = row / line_boxes(row);
  for (int x = 0; x < row; x += nx)
    asm volatile("cp.async.bulk.prefetch.tensor.4d.L2.global.tile [%0, {%1, %2, %3, %4}];\n" ::"l"(
                     reinterpret_cast<uint64_t>(&tmap)),
                 "r"(x), "r"(th), "r"(r), "r"(0)
                 : "memory");
}

// fn(integral_constant<int, I>) for every I of the sequence
template <typename F, int... I>
__device__ __forceinline__ void for_constants(F& fn, std::integer_sequence<int, I...>) {
  (fn(std::integral_constant<int, I>()), ...);
}

// One line per pass of the loop.  STG: the next line's spectra arrive during
// the current line by one TMA tensor load (thread 0; one bulk copy per block
// row, issued by the lanes of warp 0, held that warp up for 5.2k of a line's
// 28k cycles), completion on an mbarrier with a bounded wait.  Without STG
// only the grid fits in shared memory: the first pass reads the line's records
// in place, after an L2 prefetch issued one line ahead.
// NT threads: fewer threads leave more registers to each for the fused
// products of many fields (the unstaged variants).
template <int N, int MVB, int MSB, int MVF, int MSF, bool EX, bool PR, int PK, bool STG = true, int NT = kFftThreadsF>
__global__ void __launch_bounds__(NT, kFftThreadsF / NT)
    k_fft_cycle_f(const __grid_constant__ Plan P, int line0, int nlines, const __grid_constant__ CUtensorMap tmap) {
  extern __shared__ double4 smraw[];
  constexpr int NP = N + 1;
  // eight orders per rtm block
  const int ncb = EX ? 3 * MVB + MSB : P.ncb, ncf = EX ? 3 * MVF + MSF : P.ncf;
  const int npb = (ncb + 1) / 2, npf = (ncf + 1) / 2;
  const int npair = npb > npf ? npb : npf;
  const int nvb = EX ? MVB : P.nvb, nvf = EX ? MVF : P.nvf;
  const int mixb = EX ? mixed_pair(MVB, MSB) : P.mixb, mixf = PK > 0 ? -1 : P.mixf;
  double2* z = reinterpret_cast<double2*>(smraw);
  // staged spectra, 128-byte aligned, then the mbarrier
  double* st = reinterpret_cast<double*>((reinterpret_cast<uintptr_t>(z + npair * NP) + 127) & ~static_cast<uintptr_t>(127));
  const int row = 2 * kRtmOrders * ncb, nblk = (P.L + kRtmOrders) >> kRtmShift;
  unsigned long long* bar = reinterpret_cast<unsigned long long*>(st + nblk * row);
  int line = line0 + blockIdx.x;
  if (line >= nlines) return;
  auto rest = [&](int th, int r) {
    ff_mid_pass<N, +1>(z, npb, P.twid);
    __syncthreads();
    ff_fused<N, MVB, MSB, MVF, MSF, EX, PK>(z, P);
    __syncthreads();
    ff_mid_pass<N, -1>(z, npf, P.twid);
    __syncthreads();
    ff_dit_store<N, PR>(z, npf, P, P.rtm_f + rtm_off(P, 0, th, r, ncf),
                        (long long)P.nth * P.nr * (2 * kRtmOrders) * ncf, ncf, nvf, mixf, P.twid);
    __syncthreads();
  };
  if constexpr (!STG) {
    for (; line < nlines; line += gridDim.x) {
      const int th = line % P.nth, r = line / P.nth, next = line + gridDim.x;
      if (threadIdx.x == 0 && next < nlines) prefetch_l2(tmap, row, next % P.nth, next / P.nth);
      ff_dif_first<N, PR, true>(P, P.rtm_b + rtm_off(P, 0, th, r, ncb), (long long)P.nth * P.nr * row, ncb,
                                nvb, mixb, z, npb, P.twid);
      __syncthreads();
      rest(th, r);
    }
    return;
  }
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(ssa(bar)));
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  auto stage = [&](int ln) {
    if (threadIdx.x != 0) return;
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(ssa(bar)),
                 "r"((unsigned)(nblk * row * 8)) : "memory");
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");  // the first pass's reads of st
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
        "[%6];\n" ::"r"(ssa(st)),
        "l"(reinterpret_cast<uint64_t>(&tmap)), "r"(0), "r"(ln % P.nth), "r"(ln / P.nth), "r"(0), "r"(ssa(bar))
        : "memory");
  };
  __syncthreads();
  // lines theta fastest: concurrent CTAs touch neighbouring rows of one (m block, r)
  stage(line);
  unsigned phase = 0;
  while (line < nlines) {
    const int th = line % P.nth, r = line / P.nth;
    const bool late = !fbar_wait(bar, phase);
    phase ^= 1u;
    if (__syncthreads_or(late)) {
      // the staging did not complete in time: report it, let the copy land, stop
      if (threadIdx.x == 0) {
        if (P.err) atomicExch(P.err, KMHD_ERR_TIMEOUT);
        (void)fbar_wait(bar, phase ^ 1u);
      }
      return;
    }
    ff_dif_first<N, PR>(P, st, row, ncb, nvb, mixb, z, npb, P.twid);
    __syncthreads();
    const int next = line + gridDim.x;
    if (next < nlines) stage(next);
    rest(th, r);
    line = next;
  }
}

// ---------------------------------------------------------------------------
// Lines of N = 2 NH longitudes whose NH-point halves fit the specialised passes
// (N = 3072, NH = 1536).  A radix-2 step splits the line into the grid points of
// even and odd j: half h is the NH-point inverse transform of
//   x_h[k] = (X[k] + (-1)^h X[k + NH]) w_N^(h k),
// it goes through the products and back to its spectrum A_h on its own, and
//   X[k] = A_0[k] + w_N^-k A_1[k],  X[k + NH] = A_0[k] - w_N^-k A_1[k].
// So every component of half a line is in shared memory at once; only A_0 waits
// in the CTA's global scratch (L2), written and read back by the same thread.
// Going pair by pair with the whole line in the scratch instead took 17.1 ms at
// L = 1023, Nr = 17.  w_N^(h (j + r S1)) = w_N^(h j) w_48^r: the first factor is
// common to a butterfly and goes into the twiddles, the second is compile-time.
template <int NH, int H, bool PR>
__device__ __forceinline__ void ff_half_first(const Plan& P, const double* line, long long bs, int nc, int nv, int mixed,
                                              double2* z, int npair) {
  constexpr int R = ff_first(NH), S1 = NH / R, NP = NH + 1;
  static_assert(R == 24 && S1 == 64, "w_48 rotations, whole block rows");
  const int L = P.L;
  const double2* __restrict__ tw = P.twid;
  for (int it = threadIdx.x; it < npair * S1; it += blockDim.x) {
    const int pp = it / S1, j = it - pp * S1;
    const bool two = 2 * pp + 1 < nc;
    const PairPos src(P, pp, nc, nv, mixed);
    const int ux = src.x(j), uy = src.y(j), dx = src.x(-j), dy = src.y(-j);
    const double* up = line + (j >> kRtmShift) * bs;
    const double* dn = line + ((-j) >> kRtmShift) * bs;
    const double2 zero = make_double2(0.0, 0.0);
    double2 x[R];
    auto input = [&](auto rc) {
      constexpr int r = decltype(rc)::value;
      // k = j + r S1 is order k if k <= L; k + NH mirrors order NH - k if that is <= L
      const int k = j + r * S1;
      double2 u = zero, d = zero;
      if ((!PR || r < 2 * R / 3) && (PR || k <= L)) {
        const double* s = up + (r * S1 / kRtmOrders) * bs;
        const double2 c0 = *reinterpret_cast<const double2*>(s + ux);
        const double2 c1 = two ? *reinterpret_cast<const double2*>(s + uy) : zero;
        u = r == 0 && j == 0 ? make_double2(c0.x, c1.x)
                             : make_double2(0.5 * c0.x + 0.5 * c1.y, 0.5 * c1.x - 0.5 * c0.y);
      }
      if (PR ? r >= R / 3 && (r > R / 3 || j > 0) : NH - k <= L) {
        const double* s = dn + ((NH - r * S1) / kRtmOrders) * bs;
        const double2 c0 = *reinterpret_cast<const double2*>(s + dx);
        const double2 c1 = two ? *reinterpret_cast<const double2*>(s + dy) : zero;
        d = make_double2(0.5 * c0.x - 0.5 * c1.y, 0.5 * c0.y + 0.5 * c1.x);
      }
      x[r] = H == 0 ? cadd(u, d) : rot<48, r, +1>(csub(u, d));
    };
    for_constants(input, std::make_integer_sequence<int, R>{});
    DFT<R, +1>::run(x);
    double2* zp = z + pp * NP;
    // w_N^(j (2 q + H)): running product (see TwiddleRun)
    const double2 w1 = twd<+1>(tw, 2 * j);
    double2 cur = make_double2(1.0, 0.0);
    const int jj = j ^ ((j >> 3) & 7);
#pragma unroll
    for (int q = 0; q < R; ++q) {
      cur = q % kTwRun == 0 ? (H == 0 && q == 0 ? cur : twd<+1>(tw, j * (2 * q + H))) : cmul(cur, w1);
      zp[(jj ^ (((q * S1) >> 6) & 7)) + q * S1] = H == 0 && q == 0 ? x[0] : cmul(x[q], cur);
    }
  }
}

// Last forward pass of half H: H = 0 leaves A_0 in the scratch, H = 1 forms the
// line's spectrum and stores the records (lane arrangement of ff_dit_store:
// order m = j + q S1 takes X[N - m] from butterfly S1 - j, entry R - 1 - q).
template <int NH, int H, bool PR>
__device__ __forceinline__ void ff_half_store(const double2* z, int npair, const Plan& P, double2* __restrict__ sc,
                                              double* base, long long bs, int nc, int nv, int mixed) {
  constexpr int R = ff_first(NH), S1 = NH / R, NP = NH + 1;
  constexpr int QM = PR ? 2 * R / 3 : R;  // orders j + q S1 <= L < NH
  const double2* __restrict__ tw = P.twid;
  const int lane = threadIdx.x & 31, L = P.L;
  for (int w0 = threadIdx.x - lane; w0 < npair * S1; w0 += blockDim.x) {
    const int pp = w0 / S1, hi = w0 & 32;
    const int j = hi ? (lane < 16 ? 16 + lane : 64 - lane) : (lane < 16 ? lane : lane == 31 ? 32 : 79 - lane);
    const int mate = hi ? lane ^ 16 : (lane == 0 || lane == 31 ? lane : lane < 16 ? lane + 15 : lane - 15);
    const double2* zp = z + pp * NP;
    double2 x[R];
    const double2 w1 = twd<-1>(tw, 2 * j);
    double2 cur = make_double2(1.0, 0.0);
    const int jj = j ^ ((j >> 3) & 7);
#pragma unroll
    for (int q = 0; q < R; ++q) {
      cur = q == 0 ? cur : q % kTwRun == 0 ? twd<-1>(tw, 2 * j * q) : cmul(cur, w1);
      const double2 v = zp[(jj ^ (((q * S1) >> 6) & 7)) + q * S1];
      x[q] = q == 0 ? v : cmul(v, cur);
    }
    DFT<R, -1>::run(x);
    double2* a0 = sc + pp * NH + hi + lane;  // entry q at a0[q S1]
    if constexpr (H == 0) {
#pragma unroll
      for (int q = 0; q < R; ++q) a0[q * S1] = x[q];
    } else {
      const double2 wj = twd<-1>(tw, j);
      auto turn = [&](auto qc) {
        constexpr int q = decltype(qc)::value;
        x[q] = rot<48, q, -1>(cmul(x[q], wj));  // w_N^-k A_1[k]
      };
      for_constants(turn, std::make_integer_sequence<int, R>{});
      const bool two = 2 * pp + 1 < nc;
      const PairPos dst(P, pp, nc, nv, mixed);
      double* dx = base + (j >> kRtmShift) * bs + dst.x(j);
      double* dy = base + (j >> kRtmShift) * bs + dst.y(j);
      const double aN = 1.0 / (double)(2 * NH);
      auto put = [&](int q, double2 zm, double2 wm) {
        if (!PR && j + q * S1 > L) return;
        const bool m0 = q == 0 && j == 0;
        const long long o = (q * S1 / kRtmOrders) * bs;
        const double c0 = m0 ? zm.x * aN : (zm.x + wm.x) * aN, s0 = m0 ? 0.0 : (wm.y - zm.y) * aN;
        const double c1 = m0 ? zm.y * aN : (zm.y + wm.y) * aN, s1 = m0 ? 0.0 : (zm.x - wm.x) * aN;
        store_rec(dx + o, dy + o, two, dst.split, true, c0, s0, c1, s1);
      };
      auto from_mate = [&](double2 v) {
        return make_double2(__shfl_sync(0xffffffffu, v.x, mate), __shfl_sync(0xffffffffu, v.y, mate));
      };
#pragma unroll
      for (int q = 0; q < R / 2; ++q) {
        const int p = R - 1 - q;
        const double2 aq = a0[q * S1], ap = a0[p * S1];
        // entries q and p of the line: X[k] = a + x, X[k + NH] = a - x
        double2 wq = from_mate(csub(ap, x[p])), wp = from_mate(csub(aq, x[q]));
        if (j == 0) {  // mirrors of its own: entry R - q
          if (q > 0) wq = csub(a0[(R - q) * S1], x[R - q]);
          wp = csub(a0[(R - p) * S1], x[R - p]);
        }
        put(q, cadd(aq, x[q]), wq);
        if (p < QM) put(p, cadd(ap, x[p]), wp);
      }
    }
  }
}

template <int NH, int MVB, int MSB, int MVF, int MSF, bool EX, bool PR, int PK>
__global__ void __launch_bounds__(kFftThreadsF, 1)
    k_fft_cycle_half(const __grid_constant__ Plan P, int line0, int nlines, const __grid_constant__ CUtensorMap tmap) {
  extern __shared__ double4 smraw[];
  const int ncb = EX ? 3 * MVB + MSB : P.ncb, ncf = EX ? 3 * MVF + MSF : P.ncf;
  const int npb = (ncb + 1) / 2, npf = (ncf + 1) / 2;
  const int nvb = EX ? MVB : P.nvb, nvf = EX ? MVF : P.nvf;
  const int mixb = EX ? mixed_pair(MVB, MSB) : P.mixb, mixf = PK > 0 ? -1 : P.mixf;
  double2* z = reinterpret_cast<double2*>(smraw);
  double2* sc = P.fft_scratch + (long long)blockIdx.x * (npb > npf ? npb : npf) * P.nph;
  const long long bsb = (long long)P.nth * P.nr * (2 * kRtmOrders) * ncb, bsf = (long long)P.nth * P.nr * (2 * kRtmOrders) * ncf;
  for (int line = line0 + blockIdx.x; line < nlines; line += gridDim.x) {
    const int th = line % P.nth, r = line / P.nth, next = line + gridDim.x;
    if (threadIdx.x == 0 && next < nlines) prefetch_l2(tmap, 2 * kRtmOrders * ncb, next % P.nth, next / P.nth);
    const double* src = P.rtm_b + rtm_off(P, 0, th, r, ncb);
    double* dst = P.rtm_f + rtm_off(P, 0, th, r, ncf);
    auto half = [&](auto hc) {
      constexpr int H = decltype(hc)::value;
      ff_half_first<NH, H, PR>(P, src, bsb, ncb, nvb, mixb, z, npb);
      __syncthreads();
      ff_mid_pass<NH, +1, 2>(z, npb, P.twid);
      __syncthreads();
      ff_fused<NH, MVB, MSB, MVF, MSF, EX, PK>(z, P);
      __syncthreads();
      ff_mid_pass<NH, -1, 2>(z, npf, P.twid);
      __syncthreads();
      ff_half_store<NH, H, PR>(z, npf, P, sc, dst, bsf, ncf, nvf, mixf);
      __syncthreads();
    };
    half(std::integral_constant<int, 0>());
    half(std::integral_constant<int, 1>());
  }
}

// the specialised kernels' conditions besides shared memory
bool ff_usable(const Plan& p, CUtensorMap* map) {
  std::memset(map, 0, sizeof(*map));
  return p.mbs == kRtmShift && make_rtm_map(p, map);
}

template <int N, int MVB, int MSB, int MVF, int MSF, bool EX, bool PR, int PK, bool STG = true, int NT = ff_threads(N)>
cudaError_t run_cycle_fk(const Plan& p, const CUtensorMap& map, cudaStream_t s) {
  auto kern = k_fft_cycle_f<N, MVB, MSB, MVF, MSF, EX, PR, PK, STG, NT>;
  const int npair = ((p.ncb > p.ncf ? p.ncb : p.ncf) + 1) / 2;
  const size_t smem = STG ? smem_cycle_f(p) : sizeof(double2) * (size_t)npair * (N + 1);
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int dev = 0, nsm = 0, occ = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, NT, smem);
  if (occ < 1) occ = 1;
  // lines (r, theta) of the radial window, theta fastest
  const int line0 = p.r_lo * p.nth, nlines = p.r_hi * p.nth;
  int grid = nsm * occ;
  if (grid > nlines - line0) grid = nlines - line0;
  if (grid <= 0) return cudaSuccess;
  kern<<<grid, NT, smem, s>>>(p, line0, nlines, map);
  return cudaGetLastError();
}

// N = 3072 by halves; the standard set at compile time, any other at run time
template <int MVB, int MSB, int MVF, int MSF, bool EX, bool PR, int PK>
cudaError_t run_cycle_half(const Plan& p, const CUtensorMap& map, cudaStream_t s) {
  auto kern = k_fft_cycle_half<1536, MVB, MSB, MVF, MSF, EX, PR, PK>;
  const size_t smem = smem_half(p);
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const int line0 = p.r_lo * p.nth, nlines = p.r_hi * p.nth;
  const int grid = std::min(std::min(nsm, p.fft_scratch_ctas), nlines - line0);
  if (grid <= 0) return cudaSuccess;
  kern<<<grid, kFftThreadsF, smem, s>>>(p, line0, nlines, map);
  return cudaGetLastError();
}
cudaError_t run_cycle_half(const Plan& p, const CUtensorMap& map, cudaStream_t s) {
  const bool pr = p.nph == 3 * (p.L + 1);
  if (prod_list(p) == 1)
    return pr ? run_cycle_half<3, 1, 3, 1, true, true, 1>(p, map, s) : run_cycle_half<3, 1, 3, 1, true, false, 1>(p, map, s);
  return pr ? run_cycle_half<kMaxVec, kMaxScl, kMaxVec, kMaxScl, false, true, 0>(p, map, s)
            : run_cycle_half<kMaxVec, kMaxScl, kMaxVec, kMaxScl, false, false, 0>(p, map, s);
}

// by N = 3 (L + 1) and the product list
template <int N, int MVB, int MSB, int MVF, int MSF, bool EX, int PK, bool STG, int NT>
cudaError_t run_cycle_fp(const Plan& p, const CUtensorMap& map, cudaStream_t s) {
  const bool pr = p.nph == 3 * (p.L + 1);
  if (PK > 0 && prod_list(p) == PK)
    return pr ? run_cycle_fk<N, MVB, MSB, MVF, MSF, EX, true, PK, STG, NT>(p, map, s)
              : run_cycle_fk<N, MVB, MSB, MVF, MSF, EX, false, PK, STG, NT>(p, map, s);
  return pr ? run_cycle_fk<N, MVB, MSB, MVF, MSF, EX, true, 0, STG, NT>(p, map, s)
            : run_cycle_fk<N, MVB, MSB, MVF, MSF, EX, false, 0, STG, NT>(p, map, s);
}

// Staged specialised kernel of the plan's N at its own field counts.
template <int MVB, int MSB, int MVF, int MSF, int PK>
cudaError_t run_cycle_n(const Plan& p, cudaStream_t s, bool* handled) {
  *handled = true;
  CUtensorMap map;
  if (smem_cycle_f(p) <= 227 * 1024 && ff_usable(p, &map)) {
    switch (p.nph) {
      case 96: return run_cycle_fp<96, MVB, MSB, MVF, MSF, true, PK, true, ff_threads(96)>(p, map, s);
      case 192: return run_cycle_fp<192, MVB, MSB, MVF, MSF, true, PK, true, ff_threads(192)>(p, map, s);
      case 384: return run_cycle_fp<384, MVB, MSB, MVF, MSF, true, PK, true, ff_threads(384)>(p, map, s);
      case 768: return run_cycle_fp<768, MVB, MSB, MVF, MSF, true, PK, true, ff_threads(768)>(p, map, s);
      case 1536: return run_cycle_fp<1536, MVB, MSB, MVF, MSF, true, PK, true, ff_threads(1536)>(p, map, s);
      default: break;
    }
  }
  *handled = false;
  return cudaSuccess;
}

size_t smem_cycle(const Plan& p) {
  const int npair = ((p.ncb > p.ncf ? p.ncb : p.ncf) + 1) / 2;
  return sizeof(double2) * (size_t)npair * p.nph + staged_bytes(p);
}

// Threads of the run-time-radix cycle kernels: about two butterflies of a
// radix-12 pass per thread, so that short lines leave room for several CTAs
int generic_threads(const Plan& p, int npair) {
  const int want = (npair * p.nph / 24 + 31) / 32 * 32;
  return want < 64 ? 64 : want > kFftThreads ? kFftThreads : want;
}

template <typename K>
cudaError_t launch_generic(K kern, const Plan& p, size_t smem, int nt, int max_grid, cudaStream_t s) {
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int dev = 0, nsm = 0, occ = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, nt, smem);
  if (occ < 1) occ = 1;
  const int line0 = p.r_lo * p.nth, nlines = p.r_hi * p.nth;
  int grid = std::min(max_grid > 0 ? max_grid : nsm * occ, nlines - line0);
  if (grid <= 0) return cudaSuccess;
  kern<<<grid, nt, smem, s>>>(p, line0, nlines);
  return cudaGetLastError();
}

template <int PK>
cudaError_t run_generic(const Plan& p, cudaStream_t s, bool staged) {
  const int npair = ((p.ncb > p.ncf ? p.ncb : p.ncf) + 1) / 2;
  const int nt = generic_threads(p, npair);
  if (staged) return launch_generic(k_fft_cycle<PK>, p, smem_cycle(p), nt, 0, s);
  const size_t direct = sizeof(double2) * (size_t)npair * p.nph;
  if (direct <= 227 * 1024) return launch_generic(k_fft_cycle_direct<PK>, p, direct, nt, 0, s);
  if (!p.fft_scratch) return cudaErrorInvalidValue;
  return launch_generic(k_fft_cycle_wide<PK>, p, sizeof(double2) * (size_t)p.nph, kFftThreads, p.fft_scratch_ctas, s);
}
cudaError_t run_generic(const Plan& p, cudaStream_t s, bool staged) {
  switch (prod_list(p)) {
    case 1: return run_generic<1>(p, s, staged);
    case 2: return run_generic<2>(p, s, staged);
    case 3: return run_generic<3>(p, s, staged);
    case 4: return run_generic<4>(p, s, staged);
    case 5: return run_generic<5>(p, s, staged);
    default: return run_generic<0>(p, s, staged);
  }
}

// Failure-path self-test: the staging wait on an mbarrier that nothing
// completes runs out and records KMHD_ERR_TIMEOUT; the kernel returns.
__global__ void k_selftest_fft_wait(int* err) {
  __shared__ unsigned long long bar;
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(ssa(&bar)));
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0 && !fbar_wait(&bar, 0, kSelfTestSpinCap)) atomicExch(err, KMHD_ERR_TIMEOUT);
}

}  // namespace

cudaError_t launch_selftest_fft_wait(int* err, cudaStream_t s) {
  k_selftest_fft_wait<<<1, 32, 0, s>>>(err);
  return cudaGetLastError();
}

bool fft_line_fits(const Plan& p) {
  return smem_cycle(p) <= 227 * 1024 || smem_cycle_f(p) <= 227 * 1024;
}

size_t smem_direct(const Plan& p) {
  const int npair = ((p.ncb > p.ncf ? p.ncb : p.ncf) + 1) / 2;
  return sizeof(double2) * (size_t)npair * p.nph;
}

cudaError_t launch_fft_cycle(const Plan& p, cudaStream_t s) {
  if (smem_cycle(p) > 227 * 1024 && smem_cycle_f(p) > 227 * 1024) {
    // the specialised passes need (N + 1)-strided pairs: at most 16 pairs more
    CUtensorMap map;
    if (smem_direct(p) + 16 * 16 <= 227 * 1024 && ff_usable(p, &map)) {
      // the reference's full MHD set (u, omega, B, J + T, C -> five vectors + one scalar) at its own counts
      if (p.nph == 1536 && p.nvb == 4 && p.nsb == 2 && p.nvf == 5 && p.nsf == 1)
        return run_cycle_fp<1536, 4, 2, 5, 1, true, 3, false, kFftThreadsF>(p, map, s);
      // the dynamo benchmark set (u, omega, B, J + T -> omega x u, J x B, u x B, u T)
      if (p.nph == 1536 && p.nvb == 4 && p.nsb == 1 && p.nvf == 4 && p.nsf == 0)
        return run_cycle_fp<1536, 4, 1, 4, 0, true, 2, false, 256>(p, map, s);
      if (p.nph == 1536) return run_cycle_fp<1536, kMaxVec, kMaxScl, kMaxVec, kMaxScl, false, 0, false, kFftThreadsF>(p, map, s);
      if (p.nph == 768) return run_cycle_fp<768, kMaxVec, kMaxScl, kMaxVec, kMaxScl, false, 0, false, kFftThreadsF>(p, map, s);
    }
    if (p.nph == 3072 && p.fft_scratch && smem_half(p) <= 227 * 1024 && ff_usable(p, &map)) return run_cycle_half(p, map, s);
    return run_generic(p, s, false);
  }
  bool handled = false;
  cudaError_t e = cudaSuccess;
  if (p.nvb == 3 && p.nsb == 1 && p.nvf == 3 && p.nsf == 1) e = run_cycle_n<3, 1, 3, 1, 1>(p, s, &handled);
  else if (p.nvb == 2 && p.nsb == 1 && p.nvf == 2 && p.nsf == 1) e = run_cycle_n<2, 1, 2, 1, 4>(p, s, &handled);
  else if (p.nvb == 1 && p.nsb == 1 && p.nvf == 1 && p.nsf == 0) e = run_cycle_n<1, 1, 1, 0, 5>(p, s, &handled);
  if (handled) return e;
  return run_generic(p, s, smem_cycle(p) <= 227 * 1024);
}

// Radii per CTA (log2) of the separable transforms: eight (64-byte grid accesses)
// while two CTAs fit on an SM, four or fewer for longer lines; a shell of
// fewer radii takes what it has.
static int grid_lrad(const Plan& p) {
  int l = 3;
  while (l > 0 && ((sizeof(double2) * (size_t)(p.nph + 1) << l) > (l > 2 ? 110 : 227) * 1024 || (1 << (l - 1)) >= p.nr)) --l;
  return l;
}

template <typename K, typename T>
static cudaError_t launch_grid(K kern, const Plan& p, int npair, T field, cudaStream_t s) {
  const int l = grid_lrad(p);
  const size_t smem = sizeof(double2) * (size_t)(p.nph + 1) << l;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  // 16 warps per SM: four CTAs of 128 threads while their lines fit, else two of 256
  const int nt = 4 * smem <= 226 * 1024 ? kGridThreads / 2 : kGridThreads;
  kern<<<npair * ((p.nr + (1 << l) - 1) >> l) * p.nth, nt, smem, s>>>(p, field, l);
  return cudaGetLastError();
}

cudaError_t launch_fft_bwd_grid(const Plan& p, double* fld, cudaStream_t s) {
  return launch_grid(k_fft_bwd_grid, p, (p.ncb + 1) / 2, fld, s);
}

cudaError_t launch_fft_fwd_grid(const Plan& p, const double* frc, cudaStream_t s) {
  return launch_grid(k_fft_fwd_grid, p, (p.ncf + 1) / 2, frc, s);
}

}  // namespace kmhd
