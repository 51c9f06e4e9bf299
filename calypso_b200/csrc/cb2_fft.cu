// cb2_fft.cu -- longitudinal transform fused with the grid-space products.
//
// One thread block per (theta, r) row: the Fourier coefficients of the 13
// backward components (u, w, B, J vectors and T) are turned into grid values
// in shared memory, the nonlinear products are formed pointwise, and the 12
// product components are transformed back -- the grid never goes to HBM.
// This replaces back_MHD_FFT_sel_from_recv, s_cal_nonlinear_sph_MHD and
// fwd_MHD_FFT_sel_from_recv of the reference (MHD_src/sph_MHD/
// MHD_FFT_selector.F90:185-249, cal_nonlinear_sph_MHD.f90:35-84) and the
// rtm <-> rtp transposes around them.
//
// Normalisation (t_MHD_multi_FFTW.F90:220-355):
//   f(phi_p) = a_0 + sum_{m=1..L} (a_m cos m phi_p + b_m sin m phi_p),
//   a_0 = (1/N) sum f, a_m = (2/N) sum f cos, b_m = (2/N) sum f sin.
// Two real rows share one complex FFT (x + i y), N = 3^a 2^b: a four-step
// transform where N = 3 (L + 1), L + 1 = 32 .. 256, else a shared-memory
// Stockham autosort transform with radix 3, 4 and 2 stages.
#include <algorithm>
#include <cmath>
#include <vector>

#include "cb2_internal.cuh"

namespace cb2 {

template <typename T> struct C2;
template <> struct C2<double> { using t = double2; };
template <> struct C2<float> { using t = float2; };

template <typename T2>
__device__ inline T2 cmul(T2 a, T2 b) {
  T2 r;
  r.x = a.x * b.x - a.y * b.y;
  r.y = a.x * b.y + a.y * b.x;
  return r;
}

// Two real rows x, y share one complex transform z = x + i y.  The rounding
// error of a transform is relative to the larger row, so a row far below its
// partner would carry the partner's error.  Where the rows of a pair can be
// of any size -- the float64 step kernel (parity with the oracle for any
// field sizes), the generic float32 kernel and the standalone transforms of
// caller-given components -- the second row is multiplied by 2^(ex - ey),
// ex and ey the exponents of the two rows' largest magnitudes (passed as
// the bit patterns of non-negative floats), which puts both rows at the
// same size; the factor is exact and is undone after the transform (1 when
// either row is zero or subnormal).  The float32 four-step and Stockham step
// kernels pair rows of related size (components of one field, or a field
// and its curl) and do without: on the L255 bench state the scaling changed
// neither the per-term errors nor the energy drift and cost 14 % of the
// kernel's time.
__device__ __forceinline__ int pair_exp(unsigned mx_bits, unsigned my_bits) {
  const int ex = (int)(mx_bits >> 23), ey = (int)(my_bits >> 23);
  if (ex == 0 || ey == 0) return 0;
  return max(-120, min(120, ex - ey));
}
__device__ __forceinline__ float pow2i(int e) { return __int_as_float((127 + e) << 23); }
__device__ __forceinline__ unsigned abs_bits(float x) { return __float_as_uint(x) & 0x7FFFFFFFu; }

// the same for either precision: magnitudes as ordered bit patterns and the
// power-of-two factor of the second row (inverse when `inv`)
template <typename T> struct PairBits;
template <> struct PairBits<float> {
  using U = unsigned;
  __device__ static U abs_bits(float x) { return __float_as_uint(x) & 0x7FFFFFFFu; }
  __device__ static float factor(U mx, U my, bool inv) {
    const int e = pair_exp(mx, my);
    return pow2i(inv ? -e : e);
  }
};
// (float64: the high words, which order the exponents; 32-bit maxima reduce
// over a warp in one instruction)
template <> struct PairBits<double> {
  using U = unsigned;
  __device__ static U abs_bits(double x) { return (U)__double2hiint(x) & 0x7FFFFFFFu; }
  __device__ static double factor(U mx, U my, bool inv) {
    const int ex = (int)(mx >> 20), ey = (int)(my >> 20);
    if (ex == 0 || ey == 0) return 1.0;
    const int e = max(-1000, min(1000, ex - ey));
    return __hiloint2double((1023 + (inv ? -e : e)) << 20, 0);
  }
};

struct FFTPlan {
  int n, nst;
  int rad[24];
};

// one Stockham stage set; returns the buffer that holds the result
template <typename T, typename T2>
__device__ T2 *block_fft(T2 *x, T2 *y, const FFTPlan &pl, const T2 *tw, int sign) {
  const int N = pl.n;
  int Ns = 1;
  const T s32 = (T)(0.5 * sqrt(3.0));
  for (int st = 0; st < pl.nst; st++) {
    const int R = pl.rad[st];
    const int nb = N / R;
    for (int j = threadIdx.x; j < nb; j += blockDim.x) {
      int k = j % Ns;
      T2 v[4];
      for (int r = 0; r < R; r++) {
        T2 a = x[j + r * nb];
        if (r > 0 && k > 0) {
          int e = (r * k * (N / (Ns * R))) % N;
          T2 w = tw[e];
          if (sign > 0) w.y = -w.y;
          a = cmul(a, w);
        }
        v[r] = a;
      }
      T2 o[4];
      if (R == 2) {
        o[0].x = v[0].x + v[1].x; o[0].y = v[0].y + v[1].y;
        o[1].x = v[0].x - v[1].x; o[1].y = v[0].y - v[1].y;
      } else if (R == 4) {
        T2 a0, a1, a2, a3;
        a0.x = v[0].x + v[2].x; a0.y = v[0].y + v[2].y;
        a1.x = v[0].x - v[2].x; a1.y = v[0].y - v[2].y;
        a2.x = v[1].x + v[3].x; a2.y = v[1].y + v[3].y;
        T dx = v[1].x - v[3].x, dy = v[1].y - v[3].y;
        // forward (sign < 0): (v1 - v3) * (-i); inverse: * (+i)
        if (sign < 0) { a3.x = dy; a3.y = -dx; } else { a3.x = -dy; a3.y = dx; }
        o[0].x = a0.x + a2.x; o[0].y = a0.y + a2.y;
        o[1].x = a1.x + a3.x; o[1].y = a1.y + a3.y;
        o[2].x = a0.x - a2.x; o[2].y = a0.y - a2.y;
        o[3].x = a1.x - a3.x; o[3].y = a1.y - a3.y;
      } else {  // R == 3
        T2 t1, t2, t3;
        t1.x = v[1].x + v[2].x; t1.y = v[1].y + v[2].y;
        t2.x = v[0].x - (T)0.5 * t1.x; t2.y = v[0].y - (T)0.5 * t1.y;
        T dx = v[1].x - v[2].x, dy = v[1].y - v[2].y;
        // forward: (v1 - v2) * (-i sqrt3/2); inverse: * (+i sqrt3/2)
        if (sign < 0) { t3.x = s32 * dy; t3.y = -s32 * dx; } else { t3.x = -s32 * dy; t3.y = s32 * dx; }
        o[0].x = v[0].x + t1.x; o[0].y = v[0].y + t1.y;
        o[1].x = t2.x + t3.x; o[1].y = t2.y + t3.y;
        o[2].x = t2.x - t3.x; o[2].y = t2.y - t3.y;
      }
      int d = (j / Ns) * Ns * R + k;
      for (int r = 0; r < R; r++) y[d + r * Ns] = o[r];
    }
    __syncthreads();
    T2 *t = x; x = y; y = t;
    Ns *= R;
  }
  return x;
}

struct ProdCoef {
  double cv, cl, ci, ct;
};

// ---------------------------------------------------------------------------
// The fused products kernels over the order-major Fourier layout (MLayoutT).
// Input 4 vectors (u, w, B, J) + 1 scalar (T), output 4 vectors (w x u, J x B,
// u x B, u T).  At one (theta, k) the 26 input values of an order m are one run
// of 10 (P block) and one of 16 (D block), the 24 output values one of 8 and
// one of 16; element j of a run:
__device__ inline void m_comp_of_in(int j, int &c, int &s) {
  // P block (k, field, s): fields 0..3 = r of u, w, B, J; 4 = T
  if (j < 10) { const int f = j >> 1; s = j & 1; c = (f < 4) ? 3 * f : 12; return; }
  // D block (k, vector, {theta s0, theta s1, phi s0, phi s1})
  const int jd = j - 10, v = jd >> 2, q = jd & 3;
  c = 3 * v + 1 + (q >> 1); s = q & 1;
}

__device__ inline void m_comp_of_out(int j, int &c, int &s) {
  if (j < 8) { s = j & 1; c = 3 * (j >> 1); return; }
  const int jd = j - 8, v = jd >> 2, q = jd & 3;
  c = 3 * v + 1 + (q >> 1); s = q & 1;
}

// ---------------------------------------------------------------------------
// Compile-time FFT passes for N = 3 * 2^b (the zonal grids 96 .. 768 that
// the shells use): radix 3 first, then radix 16 while it divides, then the
// remaining 8, 4 or 2 (768 = 3 16 16: three passes).  Every butterfly is a
// register DFT; with N and the radices known at compile time every index
// division is by a constant.  The twiddles of stage st are one table
// w^(r k), r = 1..R-1, k = 0..NS-1, contiguous in k.  Rows in shared memory
// carry one pad element per 16 (index i -> i + i/16), which keeps the
// stride-NS writes of the radix-16 stages free of bank conflicts.
template <int N>
struct Plan3x2 {
  static constexpr int radix(int st) {
    if (st == 0) return 3;
    int n = N / 3;
    for (int q = 1; q < st; q++) n /= (n % 16 == 0) ? 16 : n;
    return (n % 16 == 0) ? 16 : n;
  }
  static constexpr int nst() {
    int n = N / 3, s = 1;
    while (n > 1) { n /= (n % 16 == 0) ? 16 : n; s++; }
    return s;
  }
  static constexpr int ns(int st) {   // product of the radices before stage st
    int p = 1;
    for (int q = 0; q < st; q++) p *= radix(q);
    return p;
  }
  static constexpr int off(int st) {
    int o = 0;
    for (int q = 0; q < st; q++) o += (radix(q) - 1) * ns(q);
    return o;
  }
  static constexpr int ntw() { return off(nst()); }
  static constexpr int NP = N + N / 16;   // padded row length
};

__host__ __device__ __forceinline__ int fpad(int i) { return i + (i >> 4); }

template <typename T2> struct ScalarOf;
template <> struct ScalarOf<float2> { using t = float; };
template <> struct ScalarOf<double2> { using t = double; };

template <typename T2>
__host__ __device__ __forceinline__ T2 cadd(T2 a, T2 b) { return T2{a.x + b.x, a.y + b.y}; }
template <typename T2>
__host__ __device__ __forceinline__ T2 csub(T2 a, T2 b) { return T2{a.x - b.x, a.y - b.y}; }
// float32 pairs on sm_100: one packed float32x2 instruction for both lanes,
// each lane rounded as the scalar add (b (-1) + a is a - b exactly), so the
// results are those of the scalar forms
__host__ __device__ __forceinline__ float2 cadd(float2 a, float2 b) {
#if defined(__CUDA_ARCH__) && __CUDA_ARCH__ >= 1000
  return __fadd2_rn(a, b);
#else
  return float2{a.x + b.x, a.y + b.y};
#endif
}
__host__ __device__ __forceinline__ float2 csub(float2 a, float2 b) {
#if defined(__CUDA_ARCH__) && __CUDA_ARCH__ >= 1000
  return __ffma2_rn(b, float2{-1.0f, -1.0f}, a);
#else
  return float2{a.x - b.x, a.y - b.y};
#endif
}
template <typename T2>
__host__ __device__ __forceinline__ T2 cmulf(T2 a, T2 b) {
  return T2{a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x};
}
// multiply by -i (forward) or +i (inverse)
template <int SIGN, typename T2>
__host__ __device__ __forceinline__ T2 rot90(T2 a) {
  return (SIGN < 0) ? T2{a.y, -a.x} : T2{-a.y, a.x};
}

// exp(SIGN 2 pi i q / 16) from exact values of the cosine at multiples of
// pi/8: cos(pi/8) = sqrt(2 + sqrt 2)/2, cos(pi/4) = sqrt(2)/2, sin(pi/8) =
// sqrt(2 - sqrt 2)/2
template <int SIGN, typename T2 = float2>
__host__ __device__ __forceinline__ T2 w16(int q) {
  using T = typename ScalarOf<T2>::t;
  constexpr T c1 = (T)0.92387953251128675613, c2 = (T)0.70710678118654752440, c3 = (T)0.38268343236508977173;
  const T cs[16] = {1, c1, c2, c3, 0, -c3, -c2, -c1, -1, -c1, -c2, -c3, 0, c3, c2, c1};
  const T sn[16] = {0, c3, c2, c1, 1, c1, c2, c3, 0, -c3, -c2, -c1, -1, -c1, -c2, -c3};
  return T2{cs[q & 15], (SIGN < 0) ? -sn[q & 15] : sn[q & 15]};
}

template <int SIGN, typename T2>
__host__ __device__ __forceinline__ void dft4(T2 &v0, T2 &v1, T2 &v2, T2 &v3) {
  const T2 a0 = cadd(v0, v2), a1 = csub(v0, v2), a2 = cadd(v1, v3), a3 = rot90<SIGN>(csub(v1, v3));
  v0 = cadd(a0, a2); v1 = cadd(a1, a3); v2 = csub(a0, a2); v3 = csub(a1, a3);
}

// in-register DFT of R points, natural order in and out
template <int R, int SIGN, typename T2>
__host__ __device__ __forceinline__ void dftr(T2 (&v)[R]) {
  using T = typename ScalarOf<T2>::t;
  if constexpr (R == 2) {
    const T2 a = v[0], b = v[1];
    v[0] = cadd(a, b); v[1] = csub(a, b);
  } else if constexpr (R == 3) {
    const T s32 = (T)0.86602540378443864676;   // sin(pi/3) = sqrt(3)/2
    const T2 t1 = cadd(v[1], v[2]);
    const T2 t2 = T2{v[0].x - (T)0.5 * t1.x, v[0].y - (T)0.5 * t1.y};
    const T dx = v[1].x - v[2].x, dy = v[1].y - v[2].y;
    const T2 t3 = (SIGN < 0) ? T2{s32 * dy, -s32 * dx} : T2{-s32 * dy, s32 * dx};
    v[0] = cadd(v[0], t1); v[1] = cadd(t2, t3); v[2] = csub(t2, t3);
  } else if constexpr (R == 4) {
    dft4<SIGN>(v[0], v[1], v[2], v[3]);
  } else if constexpr (R == 8) {
    // 2 x 4: even / odd halves, then W8^k twiddles
    T2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
    T2 o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
    dft4<SIGN>(e0, e1, e2, e3);
    dft4<SIGN>(o0, o1, o2, o3);
    o1 = cmulf(o1, w16<SIGN, T2>(2));
    o2 = rot90<SIGN>(o2);
    o3 = cmulf(o3, w16<SIGN, T2>(6));
    v[0] = cadd(e0, o0); v[4] = csub(e0, o0);
    v[1] = cadd(e1, o1); v[5] = csub(e1, o1);
    v[2] = cadd(e2, o2); v[6] = csub(e2, o2);
    v[3] = cadd(e3, o3); v[7] = csub(e3, o3);
  } else {
    static_assert(R == 16, "radix");
    // 4 x 4: n = 4 n1 + n2, k = k1 + 4 k2
    T2 a[4][4];
#pragma unroll
    for (int n2 = 0; n2 < 4; n2++) {
      a[n2][0] = v[n2]; a[n2][1] = v[4 + n2]; a[n2][2] = v[8 + n2]; a[n2][3] = v[12 + n2];
      dft4<SIGN>(a[n2][0], a[n2][1], a[n2][2], a[n2][3]);   // over n1 -> k1
    }
#pragma unroll
    for (int n2 = 1; n2 < 4; n2++)
#pragma unroll
      for (int k1 = 1; k1 < 4; k1++) a[n2][k1] = cmulf(a[n2][k1], w16<SIGN, T2>(n2 * k1));
#pragma unroll
    for (int k1 = 0; k1 < 4; k1++) {
      T2 b0 = a[0][k1], b1 = a[1][k1], b2 = a[2][k1], b3 = a[3][k1];
      dft4<SIGN>(b0, b1, b2, b3);                              // over n2 -> k2
      v[k1] = b0; v[k1 + 4] = b1; v[k1 + 8] = b2; v[k1 + 12] = b3;
    }
  }
}

template <int N, int R, int NS, int NF, int SIGN>
__device__ __forceinline__ void fft_pass(const float2 *__restrict__ x, float2 *__restrict__ y,
                                         const float2 *__restrict__ tw) {
  constexpr int NB = N / R, NP = Plan3x2<N>::NP;
  for (int idx = threadIdx.x; idx < NF * NB; idx += blockDim.x) {
    const int f = idx / NB, j = idx - f * NB;
    const int k = j % NS;
    const float2 *xf = x + f * NP;
    float2 v[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
      float2 a = xf[fpad(j + r * NB)];
      if (NS > 1 && r > 0) {
        float2 w = tw[(r - 1) * NS + k];
        if (SIGN > 0) w.y = -w.y;
        a = cmulf(a, w);
      }
      v[r] = a;
    }
    dftr<R, SIGN>(v);
    float2 *yf = y + f * NP;
    const int d = (j / NS) * NS * R + k;
#pragma unroll
    for (int r = 0; r < R; r++) yf[fpad(d + r * NS)] = v[r];
  }
  __syncthreads();
}

// all stages from `st` on; returns the buffer holding the result
template <int N, int NF, int SIGN, int ST>
__device__ __forceinline__ float2 *fft_passes(float2 *x, float2 *y, const float2 *tw) {
  using P = Plan3x2<N>;
  if constexpr (ST >= P::nst()) {
    return x;
  } else {
    fft_pass<N, P::radix(ST), P::ns(ST), NF, SIGN>(x, y, tw + P::off(ST));
    return fft_passes<N, NF, SIGN, ST + 1>(y, x, tw);
  }
}

// The fused row kernel for N = 3 * 2^b (see k_fft_products_g for the data
// flow).  Staging rows are padded to an odd stride so the transposes between
// the (m, element) order of HBM and the (element, m) order of the FFT rows
// are free of bank conflicts.
template <int N>
__global__ void __launch_bounds__(512, 2)
k_fft_products_t(int L, MLayout fin, MLayout fout, const float2 *__restrict__ twp, ProdCoef pc) {
  extern __shared__ __align__(16) unsigned char smraw[];
  using P = Plan3x2<N>;
  constexpr int NP = P::NP;
  static_assert(P::ntw() <= N, "twiddle table");
  float2 *A = reinterpret_cast<float2 *>(smraw);   // 7 x NP
  float2 *B = A + 7 * NP;                           // 7 x NP
  float2 *TW = B + 7 * NP;                          // per-stage twiddles (ntw)
  const int M1 = L + 1, MP = M1 | 1;                // padded (odd) staging stride
  float *S = reinterpret_cast<float *>(B);          // [c * 2 + s][MP]
  const int th = blockIdx.x / fin.nr, k = blockIdx.x % fin.nr;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarp = blockDim.x >> 5;
  for (int e = tid; e < P::ntw(); e += blockDim.x) TW[e] = twp[e];
  // input: one warp per order m, lane j < 26 reads element j of the 10 + 16 run
  {
    int cs = 0;
    if (lane < 26) { int c, sg; m_comp_of_in(lane, c, sg); cs = c * 2 + sg; }
    const float *src = (lane < 10) ? fin.P + (size_t)th * fin.sP() + (size_t)k * 10 + lane
                                   : fin.D + (size_t)th * fin.sD() + (size_t)k * 16 + (lane - 10);
    const size_t mst = (size_t)fin.nth * ((lane < 10) ? fin.sP() : fin.sD());
    if (lane < 26)
      for (int m = warp; m <= L; m += nwarp) S[cs * MP + m] = __ldg(src + m * mst);
  }
  __syncthreads();
  // Hermitian rows z = x + i y of the 7 pairs: one thread per (pair, m) fills
  // n = m and n = N - m; the orders above L are zero
  for (int p = 0; p < 7; p++) {
    const int c0 = 2 * p, c1 = 2 * p + 1;
    const bool has1 = c1 < 13;
    float2 *Z = A + p * NP;
    for (int m = tid; m <= L; m += blockDim.x) {
      const float a0 = S[(c0 * 2) * MP + m], a1 = has1 ? S[(c1 * 2) * MP + m] : 0.0f;
      if (m == 0) {
        Z[0] = float2{a0, a1};
      } else {
        const float b0 = S[(c0 * 2 + 1) * MP + m], b1 = has1 ? S[(c1 * 2 + 1) * MP + m] : 0.0f;
        const float xr = 0.5f * a0, xi = -0.5f * b0, yr = 0.5f * a1, yi = -0.5f * b1;
        Z[fpad(m)] = float2{xr - yi, xi + yr};
        Z[fpad(N - m)] = float2{xr + yi, -xi + yr};
      }
    }
    for (int n = L + 1 + tid; n < N - L; n += blockDim.x) Z[fpad(n)] = float2{0.0f, 0.0f};
  }
  __syncthreads();
  float2 *g = fft_passes<N, 7, +1, 0>(A, B, TW);
  float2 *hb = (g == A) ? B : A;
  const float cv = (float)pc.cv, cl = (float)pc.cl, ci = (float)pc.ci, ct = (float)pc.ct;
  for (int qq = tid; qq < N; qq += blockDim.x) {
    const int q = fpad(qq);
    const float2 p0 = g[0 * NP + q], p1 = g[1 * NP + q], p2 = g[2 * NP + q], p3 = g[3 * NP + q];
    const float2 p4 = g[4 * NP + q], p5 = g[5 * NP + q], p6 = g[6 * NP + q];
    const float ur = p0.x, ut = p0.y, up = p1.x, wr = p1.y, wt = p2.x, wp = p2.y;
    const float br = p3.x, bt = p3.y, bp = p4.x, jr = p4.y, jt = p5.x, jp = p5.y, tt = p6.x;
    hb[0 * NP + q] = float2{(wt * up - wp * ut) * cv, (wp * ur - wr * up) * cv};
    hb[1 * NP + q] = float2{(wr * ut - wt * ur) * cv, (jt * bp - jp * bt) * cl};
    hb[2 * NP + q] = float2{(jp * br - jr * bp) * cl, (jr * bt - jt * br) * cl};
    hb[3 * NP + q] = float2{(ut * bp - up * bt) * ci, (up * br - ur * bp) * ci};
    hb[4 * NP + q] = float2{(ur * bt - ut * br) * ci, ur * tt * ct};
    hb[5 * NP + q] = float2{ut * tt * ct, up * tt * ct};
  }
  __syncthreads();
  float2 *zf = fft_passes<N, 6, -1, 0>(hb, g, TW);
  // (a_m, b_m) of both components of a pair from Z[m], Z[N - m]: one thread
  // per (pair, m), into the staging rows O[c * 2 + s][MP]
  float *O = reinterpret_cast<float *>((zf == A) ? B : A);
  const float an = 1.0f / (float)N;
  for (int p = 0; p < 6; p++) {
    const float2 *Z = zf + p * NP;
    float *o0 = O + (2 * p) * 2 * MP, *o1 = O + (2 * p + 1) * 2 * MP;
    for (int m = tid; m <= L; m += blockDim.x) {
      if (m == 0) {
        const float2 z0 = Z[0];
        o0[0] = an * z0.x; o0[MP] = 0.0f; o1[0] = an * z0.y; o1[MP] = 0.0f;
      } else {
        const float2 zk = Z[fpad(m)], zn = Z[fpad(N - m)];
        o0[m] = an * (zk.x + zn.x); o0[MP + m] = -an * (zk.y - zn.y);
        o1[m] = an * (zk.y + zn.y); o1[MP + m] = an * (zk.x - zn.x);
      }
    }
  }
  __syncthreads();
  // output: one warp per m, lane j < 24 writes element j of the 8 + 16 run
  {
    int cs = 0;
    if (lane < 24) { int c, sg; m_comp_of_out(lane, c, sg); cs = c * 2 + sg; }
    float *dst = (lane < 8) ? fout.P + (size_t)th * fout.sP() + (size_t)k * 8 + lane
                            : fout.D + (size_t)th * fout.sD() + (size_t)k * 16 + (lane - 8);
    const size_t mst = (size_t)fout.nth * ((lane < 8) ? fout.sP() : fout.sD());
    if (lane < 24)
      for (int m = warp; m <= L; m += nwarp) dst[m * mst] = O[cs * MP + m];
  }
}

// ---------------------------------------------------------------------------
// Four-step products kernel for N = 3 M, M = R1 R2 = L + 1 (the standard
// nphi = 3 (L + 1) grids).  One CTA per (theta, radial level) as above; 24
// groups of 16 threads, group (pair p, residue r) owns the M-point transform
// of the colatitude samples phi_j with j = 3 j' + r:
//   backward (spectrum -> grid, exponent +): the orders above L vanish, so
//     z(3 j' + r) = sum_{m < M} e^{2 pi i m j'/M} e^{2 pi i m r/N}
//                   (Z[m] + e^{4 pi i r/3} Z[N - (M - m)])
//   forward (grid -> spectrum, exponent -): F_r = M-point DFT of h(3 j' + r),
//     Z[m] = sum_r e^{-2 pi i m r/N} F_r[m],
//     Z[N - m] = sum_r e^{+2 pi i m r/N} F_r[(M - m) mod M].
// The M-point DFT is R1 x R2: n = n1 R2 + n2, k = k1 + R1 k2; a thread holds
// one n2 column (R1 values, DFT over n1 in registers, twiddle
// e^{+-2 pi i n2 k1/M}), a transpose through shared memory, then one k1 row
// (R2 values, DFT over n2).  The Hermitian pair rows are built on the fly
// from the staged (a_m, b_m) without the 1/2 of z = x + i y: the products
// are bilinear, so their coefficients carry the 1/4 instead (exact).
// A group is R2 threads, one per column of the first step; in the second
// each takes R1 / R2 rows, so every thread of the 21 (18) groups holds R1
// values in both steps.  With 16 threads a group whatever R1 and R2, half to
// three quarters of them idled at M < 256, in CTAs of 384 threads: float32
// M = 128 (18624 rows) 477 -> 379 us, M = 64 (6240 rows) 110 -> 70, float64
// M = 32 (2352 rows) 116 -> 36.
constexpr int F4_THREADS = 384;   // the tuning value that selects these kernels
template <int R2> __host__ __device__ constexpr int f4_threads() { return 24 * R2; }

template <int R1, int R2>
struct F4Plan {
  static constexpr int M = R1 * R2, N = 3 * M;
  static constexpr int TP = R2 + 1;            // transpose row pitch (complex)
  // the block of a group (complex): its transposes, then its grid samples,
  // then its F_r.  Half a warp is 16 / R2 groups, whose blocks start R2
  // elements apart modulo 16, so that the groups' accesses fall on different
  // banks.
  static constexpr int T0 = (R1 * TP > M) ? R1 * TP : M;
  static constexpr int TG = T0 + (R2 == 16 ? 0 : (R2 + 16 - T0 % 16) % 16);
  static constexpr int X = 21 * TG;            // work buffer (complex)
  static constexpr int MP2 = M + 1;            // staging row pitch (complex)
  static constexpr int WP = R1 + 1;            // twiddle row pitch (complex)
  // tables: [2][TWP] e^{2 pi i m r/N} of r = 1, 2, then [R2][WP] e^{2 pi i n2 k1/M}
  static constexpr int TWP = M + 8, NTW = 2 * TWP + R2 * WP;
  // staging (floats): 7 rows x MP2 (Z[m], Z[N - (M - m)]) in, later 12 rows x
  // MP2 complex out
  static constexpr int SF = 28 * MP2;
  static constexpr size_t smem() { return (size_t)SF * 4 + ((size_t)X + NTW) * 8; }
};

template <typename T2>
__device__ __forceinline__ T2 cmulc(T2 a, T2 w) {   // a * conj(w)
  return T2{a.x * w.x + a.y * w.y, a.y * w.x - a.x * w.y};
}


// pmax (optional): the forward Legendre row scales' raw material, the
// largest |a_m| w(theta) of each output element over each block of 16
// orders, [theta][m / 16][element] with the elements of the output layout
// (P block k 8 + j, then D block sP + k 16 + j).
template <int R1, int R2>
__global__ void __launch_bounds__(f4_threads<R2>(), R2 == 16 ? 2 : R1 == 16 ? 4 : R2 == 8 ? 5 : 10)
k_fft_products_4s(MLayout fin, MLayout fout, const float2 *__restrict__ tables, ProdCoef pc,
                  float *__restrict__ pmax, const float *__restrict__ wgt) {
  using P = F4Plan<R1, R2>;
  constexpr int NT = f4_threads<R2>(), RU = R1 / R2;
  static_assert(R1 % R2 == 0, "rows of the second step");
  constexpr int M = P::M, N = P::N, TP = P::TP, TG = P::TG, MP2 = P::MP2, WP = P::WP;
  extern __shared__ __align__(16) unsigned char smraw[];
  // input staging [7 pairs][MP2] of (2 Z[m], 2 Z[N - (M - m)])
  float2 *S2 = reinterpret_cast<float2 *>(smraw);
  float2 *X = reinterpret_cast<float2 *>(smraw + (size_t)P::SF * 4);   // [21 groups][TG]
  float2 *TW3 = X + P::X;                                          // [2][TWP]: r = 1, 2
  float2 *TWM = TW3 + 2 * P::TWP;                                  // [R2][WP]
  const int th = blockIdx.x / fin.nr, k = blockIdx.x % fin.nr;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarp = NT / 32;
  const int grp = tid / R2, lt = tid % R2;
  // tables by asynchronous 16-byte copies
  for (int e = 2 * tid; e < 2 * M + R2 * WP; e += 2 * NT) {
    const int to = (e < M) ? e : (e < 2 * M) ? P::TWP + e - M : 2 * P::TWP + e - 2 * M;
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(TW3 + to);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(tables + M + e) : "memory");
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  // input: at one (theta, k) an order m has 13 (cos, sin) pairs, a run of 5
  // in the P block and one of 8 in the D block.  A thread takes a pair of
  // components at the orders m and M - m, which make both rows' entries of
  // the complex transform there, once for the three residues.
  {
    constexpr int IT = (4 * M + NT - 1) / NT;
    const int p = tid & 7;
    auto comp = [&](int c, const float *&src, size_t &mst) {
      const int v = c / 3, s = c - 3 * v;
      if (s == 0) {
        src = fin.P + (size_t)th * fin.sP() + (size_t)k * 10 + 2 * v;
        mst = (size_t)fin.nth * fin.sP();
      } else {
        src = fin.D + (size_t)th * fin.sD() + (size_t)k * 16 + 2 * (2 * v + s - 1);
        mst = (size_t)fin.nth * fin.sD();
      }
    };
    const float *s0, *s1;
    size_t t0, t1;
    comp(min(2 * p, 12), s0, t0);
    comp(min(2 * p + 1, 12), s1, t1);
    float2 a[IT], b[IT], c[IT], d[IT];
#pragma unroll
    for (int i = 0; i < IT; i++) {
      const int mi = (tid + i * NT) >> 3, mj = mi ? M - mi : M / 2;
      const bool on = p < 7 && mi < M / 2;
      const float2 z{0.0f, 0.0f};
      a[i] = on ? __ldg(reinterpret_cast<const float2 *>(s0 + mi * t0)) : z;
      c[i] = on ? __ldg(reinterpret_cast<const float2 *>(s0 + mj * t0)) : z;
      b[i] = (on && p < 6) ? __ldg(reinterpret_cast<const float2 *>(s1 + mi * t1)) : z;
      d[i] = (on && p < 6) ? __ldg(reinterpret_cast<const float2 *>(s1 + mj * t1)) : z;
    }
    float4 *row = reinterpret_cast<float4 *>(S2) + p * MP2;
#pragma unroll
    for (int i = 0; i < IT; i++) {
      const int mi = (tid + i * NT) >> 3, mj = mi ? M - mi : M / 2;
      if (p < 7 && mi < M / 2) {
        const float4 za{a[i].x + b[i].y, b[i].x - a[i].y, c[i].x - d[i].y, c[i].y + d[i].x};
        const float4 zc{c[i].x + d[i].y, d[i].x - c[i].y, a[i].x - b[i].y, a[i].y + b[i].x};
        // m = 0: 2 Z[0] = 2 (a_0, a'_0) and no partner; m = M / 2 is its own
        row[mi] = mi ? za : float4{2.0f * a[i].x, 2.0f * b[i].x, 0.0f, 0.0f};
        row[mj] = mi ? zc : float4{zc.x, zc.y, za.z, za.w};
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  const int gp = grp / 3, gr = grp - 3 * gp;   // pair, residue of this group
  float2 *W = X + grp * TG;                    // its block
  // ---- backward, step 1: column n2 = lt, pair rows built from the staging
  if (grp < 21) {
    const float4 *xy = reinterpret_cast<const float4 *>(S2) + gp * MP2;
    const float2 om = (gr == 0) ? float2{1.0f, 0.0f}
                    : float2{-0.5f, (gr == 1) ? -0.86602540378443864676f : 0.86602540378443864676f};
    const float2 *tw = TW3 + (gr == 2 ? P::TWP : 0);
    float2 v[R1];
#pragma unroll
    for (int n1 = 0; n1 < R1; n1++) {
      const int m = n1 * R2 + lt;
      const float4 z = xy[m];
      const float2 zm{z.x, z.y}, zp{z.z, z.w};
      float2 t{1.0f, 0.0f};
      if (gr) t = tw[m];
      // (zm + om zp) t with the rounding written out: it does not hang on how
      // the compiler contracts it here
      const float2 q{__fadd_rn(zm.x, __fmaf_rn(om.x, zp.x, -__fmul_rn(om.y, zp.y))),
                     __fadd_rn(zm.y, __fmaf_rn(om.x, zp.y, __fmul_rn(om.y, zp.x)))};
      v[n1] = float2{__fmaf_rn(q.x, t.x, -__fmul_rn(q.y, t.y)), __fmaf_rn(q.x, t.y, __fmul_rn(q.y, t.x))};
    }
    dftr<R1, +1>(v);
#pragma unroll
    for (int k1 = 0; k1 < R1; k1++) W[k1 * TP + lt] = (k1 == 0) ? v[0] : cmulf(v[k1], TWM[lt * WP + k1]);
  }
  // the block W of a group is written and read by the group's own R2 threads,
  // which sit in one warp
  __syncwarp();
  // ---- backward, step 2: row k1 = lt -> grid samples j = 3 (k1 + R1 k2) + r
  float2 w[RU][R2];
  if (grp < 21) {
#pragma unroll
    for (int u = 0; u < RU; u++) {
      const float2 *T = W + (lt + R2 * u) * TP;
#pragma unroll
      for (int n2 = 0; n2 < R2; n2++) w[u][n2] = T[n2];
      dftr<R2, +1>(w[u]);
    }
  }
  __syncwarp();
  if (grp < 21) {
#pragma unroll
    for (int u = 0; u < RU; u++) {
#pragma unroll
      for (int k2 = 0; k2 < R2; k2++) W[lt + R2 * u + R1 * k2] = w[u][k2];
    }
  }
  __syncthreads();
  // ---- products at every grid point (in place: 7 pair rows in, 6 out)
  {
    const float cv = 0.25f * (float)pc.cv, cl = 0.25f * (float)pc.cl, ci = 0.25f * (float)pc.ci,
                ct = 0.25f * (float)pc.ct;
    for (int q = tid; q < N; q += NT) {
      float2 *G = X + (q / M) * TG + q % M;
      constexpr int PT = 3 * TG;
      const float2 p0 = G[0 * PT], p1 = G[1 * PT], p2 = G[2 * PT], p3 = G[3 * PT];
      const float2 p4 = G[4 * PT], p5 = G[5 * PT], p6 = G[6 * PT];
      const float ur = p0.x, ut = p0.y, up = p1.x, wr = p1.y, wt = p2.x, wp = p2.y;
      const float br = p3.x, bt = p3.y, bp = p4.x, jr = p4.y, jt = p5.x, jp = p5.y, tt = p6.x;
      G[0 * PT] = float2{(wt * up - wp * ut) * cv, (wp * ur - wr * up) * cv};
      G[1 * PT] = float2{(wr * ut - wt * ur) * cv, (jt * bp - jp * bt) * cl};
      G[2 * PT] = float2{(jp * br - jr * bp) * cl, (jr * bt - jt * br) * cl};
      G[3 * PT] = float2{(ut * bp - up * bt) * ci, (up * br - ur * bp) * ci};
      G[4 * PT] = float2{(ur * bt - ut * br) * ci, ur * tt * ct};
      G[5 * PT] = float2{ut * tt * ct, up * tt * ct};
    }
  }
  __syncthreads();
  // ---- forward, step 1: column n2 = lt of the samples j = 3 (n1 R2 + n2) + r
  float2 v[R1];
  if (grp < 18) {
#pragma unroll
    for (int n1 = 0; n1 < R1; n1++) v[n1] = W[n1 * R2 + lt];
    dftr<R1, -1>(v);
#pragma unroll
    for (int k1 = 1; k1 < R1; k1++) v[k1] = cmulc(v[k1], TWM[lt * WP + k1]);
  }
  __syncwarp();
  if (grp < 18) {
#pragma unroll
    for (int k1 = 0; k1 < R1; k1++) W[k1 * TP + lt] = v[k1];
  }
  __syncwarp();
  // ---- forward, step 2: row k1 = lt -> F_r[k1 + R1 k2]
  if (grp < 18) {
#pragma unroll
    for (int u = 0; u < RU; u++) {
      const float2 *T = W + (lt + R2 * u) * TP;
#pragma unroll
      for (int n2 = 0; n2 < R2; n2++) w[u][n2] = T[n2];
      dftr<R2, -1>(w[u]);
    }
  }
  __syncwarp();
  if (grp < 18) {
#pragma unroll
    for (int u = 0; u < RU; u++) {
#pragma unroll
      for (int k2 = 0; k2 < R2; k2++) W[lt + R2 * u + R1 * k2] = w[u][k2];
    }
  }
  __syncthreads();
  // ---- combine the residues: Z[m], Z[N - m] -> (a_m, b_m) of both
  // components of each pair, into the output staging rows [c][MP2] of
  // (a_m, b_m) pairs.  A thread takes the orders m and M - m together: both
  // read the same six F values.
  float2 *O2 = S2;
  {
    const float an = 1.0f / (float)N;
    constexpr int MH = M / 2 + 1;
    auto out = [&](float2 *o0, float2 *o1, int m, float2 zk, float2 zn) {
      if (m == 0) {
        o0[0] = float2{an * zk.x, 0.0f}; o1[0] = float2{an * zk.y, 0.0f};
      } else {
        o0[m] = float2{an * (zk.x + zn.x), -an * (zk.y - zn.y)};
        o1[m] = float2{an * (zk.y + zn.y), an * (zk.x - zn.x)};
      }
    };
    for (int idx = tid; idx < 6 * MH; idx += NT) {
      const int p = idx / MH, m = idx - p * MH, mm = (M - m) & (M - 1);
      const float2 *F = X + p * 3 * TG;
      float2 *o0 = O2 + (2 * p) * MP2, *o1 = o0 + MP2;
      const float2 f0 = F[m], f1 = F[TG + m], f2 = F[2 * TG + m];
      const float2 g0 = F[mm], g1 = F[TG + mm], g2 = F[2 * TG + mm];
      {
        const float2 t1 = TW3[m], t2 = TW3[P::TWP + m];
        const float2 zk = cadd(f0, cadd(cmulc(f1, t1), cmulc(f2, t2)));
        const float2 zn = cadd(g0, cadd(cmulf(g1, t1), cmulf(g2, t2)));
        out(o0, o1, m, zk, zn);
      }
      if (m > 0 && mm != m) {   // the partner order M - m
        const float2 t1 = TW3[mm], t2 = TW3[P::TWP + mm];
        const float2 zk = cadd(g0, cadd(cmulc(g1, t1), cmulc(g2, t2)));
        const float2 zn = cadd(f0, cadd(cmulf(f1, t1), cmulf(f2, t2)));
        out(o0, o1, mm, zk, zn);
      }
    }
  }
  __syncthreads();
  // output: 12 (cos, sin) pairs per order, a run of 4 in the P block and one
  // of 8 in the D block; half-warp h of warp w writes the orders
  // 2 (w + nwarp i) + h, lane j < 12 of the half pair j (8-byte stores)
  {
    const int j = lane & 15, hw = lane >> 4;
    int c = 0;
    float *dst = fout.P;
    size_t mst = 0;
    if (j < 4) {
      c = 3 * j;
      dst = fout.P + (size_t)th * fout.sP() + (size_t)k * 8 + 2 * j;
      mst = (size_t)fout.nth * fout.sP();
    } else if (j < 12) {
      const int jd = j - 4;
      c = 3 * (jd >> 1) + 1 + (jd & 1);
      dst = fout.D + (size_t)th * fout.sD() + (size_t)k * 16 + 2 * jd;
      mst = (size_t)fout.nth * fout.sD();
    }
    if (j < 12)
      for (int m = 2 * warp + hw; m < M; m += 2 * nwarp)
        *reinterpret_cast<float2 *>(dst + m * mst) = O2[c * MP2 + m];
  }
  if (pmax) {
    constexpr int MB = M / 16;
    const float wt = __ldg(wgt + th);
    const size_t E = fout.sP() + fout.sD();
    float *pm = pmax + (size_t)th * MB * E;
    for (int t = tid; t < 12 * MB; t += NT) {
      const int c = t % 12, mb = t / 12, v = c / 3, s = c - 3 * v;
      const float2 *row = O2 + c * MP2 + mb * 16;
      float ma = 0.0f, mc = 0.0f;
#pragma unroll
      for (int u = 0; u < 16; u++) {
        const float2 x = row[u];
        ma = fmaxf(ma, fabsf(x.x));
        mc = fmaxf(mc, fabsf(x.y));
      }
      const size_t e = (s == 0) ? (size_t)k * 8 + 2 * v : fout.sP() + (size_t)k * 16 + 2 * (2 * v + s - 1);
      *reinterpret_cast<float2 *>(pm + (size_t)mb * E + e) = float2{ma * wt, mc * wt};
    }
  }
}

// ---------------------------------------------------------------------------
// Input of the float64 four-step kernels, as in k_fft_products_4s: a thread
// takes a pair of components at the orders m and M - m.  rows: [7][M + 1]
// 2 Z[m], then [7][M + 1] 2 Z[N - (M - m)] of the pairs, the second component
// scaled to the first; cmx: [0, 14) the components' maxima, the rest of its
// ncmx entries zero.  Ends with the rows written, not yet a barrier.
template <int M, int NT>
__device__ __forceinline__ void stage_pairs64(const MLayout64 &fin, int th, int k, double2 *S2, PairBits<double>::U *cmx,
                                              int ncmx) {
  using PB = PairBits<double>;
  using U = PB::U;
  constexpr int MP2 = M + 1;
  const int tid = threadIdx.x, lane = tid & 31;
  constexpr int IT = (4 * M + NT - 1) / NT;
  const int p = tid & 7;
  auto comp = [&](int c, const double *&src, size_t &mst) {
    const int v = c / 3, s = c - 3 * v;
    if (s == 0) {
      src = fin.P + (size_t)th * fin.sP() + (size_t)k * 10 + 2 * v;
      mst = (size_t)fin.nth * fin.sP();
    } else {
      src = fin.D + (size_t)th * fin.sD() + (size_t)k * 16 + 2 * (2 * v + s - 1);
      mst = (size_t)fin.nth * fin.sD();
    }
  };
  const double *s0, *s1;
  size_t t0, t1;
  comp(min(2 * p, 12), s0, t0);
  comp(min(2 * p + 1, 12), s1, t1);
  double2 a[IT], b[IT], c[IT], d[IT];
#pragma unroll
  for (int i = 0; i < IT; i++) {
    const int mi = (tid + i * NT) >> 3, mj = mi ? M - mi : M / 2;
    const bool on = p < 7 && mi < M / 2;
    const double2 z{0.0, 0.0};
    a[i] = on ? __ldg(reinterpret_cast<const double2 *>(s0 + mi * t0)) : z;
    c[i] = on ? __ldg(reinterpret_cast<const double2 *>(s0 + mj * t0)) : z;
    b[i] = (on && p < 6) ? __ldg(reinterpret_cast<const double2 *>(s1 + mi * t1)) : z;
    d[i] = (on && p < 6) ? __ldg(reinterpret_cast<const double2 *>(s1 + mj * t1)) : z;
  }
  if (tid < ncmx) cmx[tid] = 0;
  __syncthreads();
  U m0 = 0, m1 = 0;
#pragma unroll
  for (int i = 0; i < IT; i++) {
    m0 = max(max(m0, max(PB::abs_bits(a[i].x), PB::abs_bits(a[i].y))), max(PB::abs_bits(c[i].x), PB::abs_bits(c[i].y)));
    m1 = max(max(m1, max(PB::abs_bits(b[i].x), PB::abs_bits(b[i].y))), max(PB::abs_bits(d[i].x), PB::abs_bits(d[i].y)));
  }
#pragma unroll
  for (int o = 8; o <= 16; o *= 2) {
    m0 = max(m0, __shfl_xor_sync(0xffffffffu, m0, o));
    m1 = max(m1, __shfl_xor_sync(0xffffffffu, m1, o));
  }
  if (lane < 7) {
    atomicMax(cmx + 2 * p, m0);
    atomicMax(cmx + 2 * p + 1, m1);
  }
  __syncthreads();
  const double sy = (p < 6) ? PB::factor(cmx[2 * p], cmx[2 * p + 1], false) : 1.0;
  double2 *rm = S2 + p * MP2, *rp = S2 + (7 + p) * MP2;
#pragma unroll
  for (int i = 0; i < IT; i++) {
    const int mi = (tid + i * NT) >> 3, mj = mi ? M - mi : M / 2;
    if (p < 7 && mi < M / 2) {
      const double2 A = a[i], C = c[i], B{b[i].x * sy, b[i].y * sy}, D{d[i].x * sy, d[i].y * sy};
      // m = 0: 2 Z[0] = 2 (a_0, a'_0) and no partner; m = M / 2 is its own
      rm[mi] = mi ? double2{A.x + B.y, B.x - A.y} : double2{2.0 * A.x, 2.0 * B.x};
      rp[mi] = mi ? double2{C.x - D.y, C.y + D.x} : double2{0.0, 0.0};
      rm[mj] = double2{C.x + D.y, D.x - C.y};
      rp[mj] = mi ? double2{A.x - B.y, A.y + B.x} : double2{C.x - D.y, C.y + D.x};
    }
  }
}

// The float64 four-step products kernel (the plain path's step): the data
// flow of k_fft_products_4s on the float64 Fourier rows, with the pair
// scaling of k_fft_products_g (the second row of each pair, inputs and
// products, brought to the size of the first), so every row keeps float64
// precision whatever the sizes of the fields.  One CTA per (theta, k).
template <int R1, int R2>
struct F4Plan64 {
  static constexpr int M = R1 * R2, N = 3 * M;
  static constexpr int TP = R2 + 1;
  // a group's block; 16-byte accesses go eight lanes at a time, two groups of
  // four at R2 = 4, whose blocks then start four elements apart modulo 8
  static constexpr int T0 = (R1 * TP > M) ? R1 * TP : M;
  static constexpr int TG = T0 + (R2 >= 8 ? 0 : (R2 + 8 - T0 % 8) % 8);
  static constexpr int X = 21 * TG;
  static constexpr int MP2 = M + 1;            // staging row pitch
  static constexpr int WP = R1 + 1;
  static constexpr int TWP = M + 4, NTW = 2 * TWP + R2 * WP;
  static constexpr int SC = 14 * MP2;          // staging: Z[m], Z[N - (M - m)] of 7 pairs in, then 12 rows out
  static constexpr size_t smem() { return ((size_t)SC + X + NTW) * sizeof(double2) + 32 * sizeof(double); }
};

template <int R1, int R2>
__global__ void __launch_bounds__(f4_threads<R2>(), R2 == 16 ? 1 : R1 == 16 ? 2 : R2 == 8 ? 4 : 8)
k_fft_products_4s64(MLayout64 fin, MLayout64 fout, const double2 *__restrict__ tables, ProdCoef pc) {
  using P = F4Plan64<R1, R2>;
  using PB = PairBits<double>;
  using U = PB::U;
  constexpr int NT = f4_threads<R2>(), RU = R1 / R2;
  constexpr int M = P::M, N = P::N, TP = P::TP, TG = P::TG, MP2 = P::MP2, WP = P::WP;
  extern __shared__ __align__(16) unsigned char smraw[];
  double2 *S2 = reinterpret_cast<double2 *>(smraw);   // [7][MP2] 2 Z[m], [7][MP2] 2 Z[N - (M - m)]; later [12][MP2] out
  double2 *X = S2 + P::SC;                             // [21 groups][TG]
  double2 *TW3 = X + P::X;                             // [2][TWP]: r = 1, 2
  double2 *TWM = TW3 + 2 * P::TWP;                     // [R2][WP]
  U *cmx = reinterpret_cast<U *>(TWM + R2 * WP);      // [0, 14) input maxima, [14, 26) products
  const int th = blockIdx.x / fin.nr, k = blockIdx.x % fin.nr;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarp = NT / 32;
  const int grp = tid / R2, lt = tid % R2;
  // tables by asynchronous copies
  for (int e = tid; e < 2 * M + R2 * WP; e += NT) {
    const int to = (e < M) ? e : (e < 2 * M) ? P::TWP + e - M : 2 * P::TWP + e - 2 * M;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(TW3 + to)),
                 "l"(tables + M + e) : "memory");
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  stage_pairs64<M, NT>(fin, th, k, S2, cmx, 26);
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  const int gp = grp / 3, gr = grp - 3 * gp;
  double2 *W = X + grp * TG;   // the group's block, written and read by its own threads (one warp)
  // ---- backward, step 1: column n2 = lt
  if (grp < 21) {
    const double2 *rm = S2 + gp * MP2, *rp = S2 + (7 + gp) * MP2;
    const double2 om = (gr == 0) ? double2{1.0, 0.0}
                     : double2{-0.5, (gr == 1) ? -0.86602540378443864676 : 0.86602540378443864676};
    const double2 *tw = TW3 + (gr == 2 ? P::TWP : 0);
    double2 v[R1];
#pragma unroll
    for (int n1 = 0; n1 < R1; n1++) {
      const int m = n1 * R2 + lt;
      double2 t{1.0, 0.0};
      if (gr) t = tw[m];
      v[n1] = cmulf(cadd(rm[m], cmulf(om, rp[m])), t);
    }
    dftr<R1, +1>(v);
#pragma unroll
    for (int k1 = 0; k1 < R1; k1++) W[k1 * TP + lt] = (k1 == 0) ? v[0] : cmulf(v[k1], TWM[lt * WP + k1]);
  }
  __syncwarp();
  // ---- backward, step 2: row k1 = lt -> grid samples j = 3 (k1 + R1 k2) + r
  {
    double2 w[RU][R2];
    if (grp < 21) {
#pragma unroll
      for (int u = 0; u < RU; u++) {
        const double2 *T = W + (lt + R2 * u) * TP;
#pragma unroll
        for (int n2 = 0; n2 < R2; n2++) w[u][n2] = T[n2];
        dftr<R2, +1>(w[u]);
      }
    }
    __syncwarp();
    if (grp < 21) {
#pragma unroll
      for (int u = 0; u < RU; u++) {
#pragma unroll
        for (int k2 = 0; k2 < R2; k2++) W[lt + R2 * u + R1 * k2] = w[u][k2];
      }
    }
  }
  __syncthreads();
  // ---- products at every grid point (the second rows unscaled on the way
  // in), with the largest magnitude of each product row
  {
    const double cv = 0.25 * pc.cv, cl = 0.25 * pc.cl, ci = 0.25 * pc.ci, ct = 0.25 * pc.ct;
    double iy[6];
#pragma unroll
    for (int p = 0; p < 6; p++) iy[p] = PB::factor(cmx[2 * p], cmx[2 * p + 1], true);
    U hm[12];
#pragma unroll
    for (int c = 0; c < 12; c++) hm[c] = 0;
    for (int q = tid; q < N; q += NT) {
      double2 *G = X + (q / M) * TG + q % M;
      constexpr int PT = 3 * TG;
      const double2 p0 = G[0 * PT], p1 = G[1 * PT], p2 = G[2 * PT], p3 = G[3 * PT];
      const double2 p4 = G[4 * PT], p5 = G[5 * PT], p6 = G[6 * PT];
      const double ur = p0.x, ut = p0.y * iy[0], up = p1.x, wr = p1.y * iy[1], wt = p2.x, wp = p2.y * iy[2];
      const double br = p3.x, bt = p3.y * iy[3], bp = p4.x, jr = p4.y * iy[4], jt = p5.x, jp = p5.y * iy[5];
      const double tt = p6.x;
      const double2 hv[6] = {double2{(wt * up - wp * ut) * cv, (wp * ur - wr * up) * cv},
                             double2{(wr * ut - wt * ur) * cv, (jt * bp - jp * bt) * cl},
                             double2{(jp * br - jr * bp) * cl, (jr * bt - jt * br) * cl},
                             double2{(ut * bp - up * bt) * ci, (up * br - ur * bp) * ci},
                             double2{(ur * bt - ut * br) * ci, ur * tt * ct},
                             double2{ut * tt * ct, up * tt * ct}};
#pragma unroll
      for (int p = 0; p < 6; p++) {
        G[p * PT] = hv[p];
        hm[2 * p] = max(hm[2 * p], PB::abs_bits(hv[p].x));
        hm[2 * p + 1] = max(hm[2 * p + 1], PB::abs_bits(hv[p].y));
      }
    }
#pragma unroll
    for (int c = 0; c < 12; c++) {
      const U v = __reduce_max_sync(0xffffffffu, hm[c]);
      if (lane == 0) atomicMax(cmx + 14 + c, v);
    }
  }
  __syncthreads();
  // ---- forward, step 1: column n2 = lt of the samples j = 3 (n1 R2 + n2) + r,
  // the second row of the pair scaled on the way in
  {
    double2 v[R1];
    if (grp < 18) {
      const double sy = PB::factor(cmx[14 + 2 * gp], cmx[15 + 2 * gp], false);
#pragma unroll
      for (int n1 = 0; n1 < R1; n1++) {
        v[n1] = W[n1 * R2 + lt];
        v[n1].y *= sy;
      }
      dftr<R1, -1>(v);
#pragma unroll
      for (int k1 = 1; k1 < R1; k1++) v[k1] = cmulc(v[k1], TWM[lt * WP + k1]);
    }
    __syncwarp();
    if (grp < 18) {
#pragma unroll
      for (int k1 = 0; k1 < R1; k1++) W[k1 * TP + lt] = v[k1];
    }
  }
  __syncwarp();
  // ---- forward, step 2: row k1 = lt -> F_r[k1 + R1 k2]
  {
    double2 w[RU][R2];
    if (grp < 18) {
#pragma unroll
      for (int u = 0; u < RU; u++) {
        const double2 *T = W + (lt + R2 * u) * TP;
#pragma unroll
        for (int n2 = 0; n2 < R2; n2++) w[u][n2] = T[n2];
        dftr<R2, -1>(w[u]);
      }
    }
    __syncwarp();
    if (grp < 18) {
#pragma unroll
      for (int u = 0; u < RU; u++) {
#pragma unroll
        for (int k2 = 0; k2 < R2; k2++) W[lt + R2 * u + R1 * k2] = w[u][k2];
      }
    }
  }
  __syncthreads();
  // ---- combine the residues: (a_m, b_m) of both rows of each pair (the
  // second unscaled), into the staging rows [c][MP2]
  {
    const double an = 1.0 / (double)N;
    for (int idx = tid; idx < 6 * M; idx += NT) {
      const int p = idx / M, m = idx - p * M, mm = (M - m) & (M - 1);
      const double2 *F = X + p * 3 * TG;
      const double2 t1 = TW3[m], t2 = TW3[P::TWP + m];
      const double2 zk = cadd(F[m], cadd(cmulc(F[TG + m], t1), cmulc(F[2 * TG + m], t2)));
      const double2 zn = cadd(F[mm], cadd(cmulf(F[TG + mm], t1), cmulf(F[2 * TG + mm], t2)));
      const double ay = an * PB::factor(cmx[14 + 2 * p], cmx[15 + 2 * p], true);
      double2 *o0 = S2 + (2 * p) * MP2, *o1 = S2 + (2 * p + 1) * MP2;
      if (m == 0) {
        o0[0] = double2{an * zk.x, 0.0};
        o1[0] = double2{ay * zk.y, 0.0};
      } else {
        o0[m] = double2{an * (zk.x + zn.x), -an * (zk.y - zn.y)};
        o1[m] = double2{ay * (zk.y + zn.y), ay * (zk.x - zn.x)};
      }
    }
  }
  __syncthreads();
  {
    const int j = lane & 15, hw = lane >> 4;
    int c = 0;
    double *dst = fout.P;
    size_t mst = 0;
    if (j < 4) {
      c = 3 * j;
      dst = fout.P + (size_t)th * fout.sP() + (size_t)k * 8 + 2 * j;
      mst = (size_t)fout.nth * fout.sP();
    } else if (j < 12) {
      const int jd = j - 4;
      c = 3 * (jd >> 1) + 1 + (jd & 1);
      dst = fout.D + (size_t)th * fout.sD() + (size_t)k * 16 + 2 * jd;
      mst = (size_t)fout.nth * fout.sD();
    }
    if (j < 12)
      for (int m = 2 * warp + hw; m < M; m += 2 * nwarp)
        *reinterpret_cast<double2 *>(dst + m * mst) = S2[c * MP2 + m];
  }
}

// The same transform one residue after another, for M = 256: the grid samples
// of the three residues do not meet until the orders are combined, so a CTA
// needs the transposes and grid rows of one (30 KB instead of 91) and two CTAs
// share an SM, one computing while the other moves data through shared memory;
// the (a_m, b_m) of the 12 products add up in registers.  The product rows are
// scaled pair by pair within each residue.  The three residues side by side in
// one CTA of 384 threads and 166 KB took 5.7 ms at L255 / Nr129 (49536 rows).
template <int R1, int R2>
struct F4Plan64R {
  static constexpr int M = R1 * R2, N = 3 * M, NT = 8 * R2;
  static constexpr int TP = R2 + 1, TG = R1 * TP, X = 7 * TG;   // transposes / 7 M grid samples / 6 M orders
  static constexpr int MP2 = M + 1, WP = R1 + 1, NTW = 3 * M + R2 * WP, SC = 14 * MP2;
  static constexpr int MH = 6 * M / NT;                          // (pair, order) sums of a thread
  static constexpr size_t smem() { return ((size_t)SC + X + NTW) * sizeof(double2) + 56 * sizeof(unsigned); }
};

template <int R1, int R2>
__global__ void __launch_bounds__(F4Plan64R<R1, R2>::NT, 2)
k_fft_products_4s64r(MLayout64 fin, MLayout64 fout, const double2 *__restrict__ tables, ProdCoef pc) {
  using P = F4Plan64R<R1, R2>;
  using PB = PairBits<double>;
  using U = PB::U;
  static_assert(R1 == R2, "one row of the second step a thread");
  constexpr int M = P::M, N = P::N, NT = P::NT, TP = P::TP, TG = P::TG, MP2 = P::MP2, WP = P::WP, MH = P::MH;
  extern __shared__ __align__(16) unsigned char smraw[];
  double2 *S2 = reinterpret_cast<double2 *>(smraw);   // [14][MP2] (a_m, b_m); last [12][MP2] out
  double2 *X = S2 + P::SC;
  double2 *TW3 = X + P::X;                             // [3][M]
  double2 *TWM = TW3 + 3 * M;                          // [R2][WP]
  U *cmx = reinterpret_cast<U *>(TWM + R2 * WP);      // [0, 13) input maxima, 16 + 12 r: products of residue r
  const int th = blockIdx.x / fin.nr, k = blockIdx.x % fin.nr;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarp = NT / 32;
  const int gp = tid / R2, lt = tid % R2;              // pair (7: idle), column / row
  for (int e = tid; e < 14; e += NT) S2[e * MP2 + M] = double2{0.0, 0.0};
  for (int e = tid; e < M; e += NT) S2[13 * MP2 + e] = double2{0.0, 0.0};
  for (int e = tid; e < 52; e += NT) cmx[e] = 0;
  auto cp16 = [](double2 *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
  };
  for (int e = tid; e < P::NTW; e += NT) cp16(TW3 + e, tables + e);
  {
    const int j = lane & 15, hw = lane >> 4;
    int c = 0;
    const double *src = fin.P;
    size_t mst = 0;
    if (j < 5) {
      c = (j < 4) ? 3 * j : 12;
      src = fin.P + (size_t)th * fin.sP() + (size_t)k * 10 + 2 * j;
      mst = (size_t)fin.nth * fin.sP();
    } else if (j < 13) {
      const int jd = j - 5;
      c = 3 * (jd >> 1) + 1 + (jd & 1);
      src = fin.D + (size_t)th * fin.sD() + (size_t)k * 16 + 2 * jd;
      mst = (size_t)fin.nth * fin.sD();
    }
    if (j < 13)
      for (int m = 2 * warp + hw; m < M; m += 2 * nwarp) cp16(S2 + c * MP2 + m, src + m * mst);
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
  }
  __syncthreads();
  for (int c = warp; c < 13; c += nwarp) {
    U mx = 0;
    for (int m = lane; m < M; m += 32) {
      const double2 v = S2[c * MP2 + m];
      mx = max(mx, max(PB::abs_bits(v.x), PB::abs_bits(v.y)));
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane == 0) cmx[c] = mx;
  }
  __syncthreads();
  // (a_m, b_m) of the two components of pair p, (p, m) = tid + i NT
  double2 o0[MH], o1[MH];
#pragma unroll
  for (int i = 0; i < MH; i++) o0[i] = o1[i] = double2{0.0, 0.0};
#pragma unroll 1
  for (int r = 0; r < 3; r++) {
    const double2 *tw = TW3 + r * M;
    double2 v[R1];
    // ---- backward, step 1: column n2 = lt, pair rows from the staging
    if (gp < 7) {
      const double2 *x0 = S2 + (2 * gp) * MP2, *y0 = S2 + (2 * gp + 1) * MP2;
      const double sy = (gp < 6) ? PB::factor(cmx[2 * gp], cmx[2 * gp + 1], false) : 1.0;
      const double2 om = (r == 0) ? double2{1.0, 0.0}
                       : double2{-0.5, (r == 1) ? -0.86602540378443864676 : 0.86602540378443864676};
#pragma unroll
      for (int n1 = 0; n1 < R1; n1++) {
        const int m = n1 * R2 + lt, mq = M - m;
        const double2 a = x0[m], c = x0[mq];
        const double2 b = double2{y0[m].x * sy, y0[m].y * sy}, d = double2{y0[mq].x * sy, y0[mq].y * sy};
        double2 zm = double2{a.x + b.y, b.x - a.y};           // 2 Z[m]
        const double2 zp = double2{c.x - d.y, c.y + d.x};     // 2 Z[N - (M - m)] (zero at m = 0)
        if (n1 == 0 && lt == 0) zm = double2{2.0 * a.x, 2.0 * b.x};
        v[n1] = cmulf(cadd(zm, cmulf(om, zp)), tw[m]);
      }
      dftr<R1, +1>(v);
      double2 *T = X + gp * TG;
#pragma unroll
      for (int k1 = 0; k1 < R1; k1++) T[k1 * TP + lt] = (k1 == 0) ? v[0] : cmulf(v[k1], TWM[lt * WP + k1]);
    }
    __syncwarp();   // the group's own transpose block
    // ---- step 2: row k1 = lt -> samples j' = k1 + R1 k2
    if (gp < 7) {
      const double2 *T = X + gp * TG + lt * TP;
#pragma unroll
      for (int n2 = 0; n2 < R2; n2++) v[n2] = T[n2];
      dftr<R2, +1>(v);
    }
    __syncthreads();
    if (gp < 7) {
      double2 *G = X + gp * M + lt;
#pragma unroll
      for (int k2 = 0; k2 < R2; k2++) G[R1 * k2] = v[k2];
    }
    __syncthreads();
    // ---- products at the residue's samples, in place
    {
      const double cv = 0.25 * pc.cv, cl = 0.25 * pc.cl, ci = 0.25 * pc.ci, ct = 0.25 * pc.ct;
      double iy[6];
#pragma unroll
      for (int p = 0; p < 6; p++) iy[p] = PB::factor(cmx[2 * p], cmx[2 * p + 1], true);
      U hm[12];
#pragma unroll
      for (int c = 0; c < 12; c++) hm[c] = 0;
#pragma unroll 1
      for (int q = tid; q < M; q += NT) {
        const double2 p0 = X[0 * M + q], p1 = X[1 * M + q], p2 = X[2 * M + q], p3 = X[3 * M + q];
        const double2 p4 = X[4 * M + q], p5 = X[5 * M + q], p6 = X[6 * M + q];
        const double ur = p0.x, ut = p0.y * iy[0], up = p1.x, wr = p1.y * iy[1], wt = p2.x, wp = p2.y * iy[2];
        const double br = p3.x, bt = p3.y * iy[3], bp = p4.x, jr = p4.y * iy[4], jt = p5.x, jp = p5.y * iy[5];
        const double tt = p6.x;
        const double2 hv[6] = {double2{(wt * up - wp * ut) * cv, (wp * ur - wr * up) * cv},
                               double2{(wr * ut - wt * ur) * cv, (jt * bp - jp * bt) * cl},
                               double2{(jp * br - jr * bp) * cl, (jr * bt - jt * br) * cl},
                               double2{(ut * bp - up * bt) * ci, (up * br - ur * bp) * ci},
                               double2{(ur * bt - ut * br) * ci, ur * tt * ct},
                               double2{ut * tt * ct, up * tt * ct}};
#pragma unroll
        for (int p = 0; p < 6; p++) {
          X[p * M + q] = hv[p];
          hm[2 * p] = max(hm[2 * p], PB::abs_bits(hv[p].x));
          hm[2 * p + 1] = max(hm[2 * p + 1], PB::abs_bits(hv[p].y));
        }
      }
#pragma unroll
      for (int c = 0; c < 12; c++) {
        const U u = __reduce_max_sync(0xffffffffu, hm[c]);
        if (lane == 0) atomicMax(cmx + 16 + 12 * r + c, u);
      }
    }
    __syncthreads();
    // ---- forward, step 1: column n2 = lt of the samples n1 R2 + n2
    const U *pmx = cmx + 16 + 12 * r;
    if (gp < 6) {
      const double2 *G = X + gp * M + lt;
      const double sy = PB::factor(pmx[2 * gp], pmx[2 * gp + 1], false);
#pragma unroll
      for (int n1 = 0; n1 < R1; n1++) {
        v[n1] = G[R2 * n1];
        v[n1].y *= sy;
      }
      dftr<R1, -1>(v);
#pragma unroll
      for (int k1 = 1; k1 < R1; k1++) v[k1] = cmulc(v[k1], TWM[lt * WP + k1]);
    }
    __syncthreads();
    if (gp < 6) {
      double2 *T = X + gp * TG;
#pragma unroll
      for (int k1 = 0; k1 < R1; k1++) T[k1 * TP + lt] = v[k1];
    }
    __syncwarp();
    // ---- step 2: row k1 = lt -> F_r[k1 + R1 k2]
    if (gp < 6) {
      const double2 *T = X + gp * TG + lt * TP;
#pragma unroll
      for (int n2 = 0; n2 < R2; n2++) v[n2] = T[n2];
      dftr<R2, -1>(v);
    }
    __syncthreads();
    if (gp < 6) {
      double2 *F = X + gp * M + lt;
#pragma unroll
      for (int k2 = 0; k2 < R2; k2++) F[R1 * k2] = v[k2];
    }
    __syncthreads();
    // ---- this residue's part of Z[m], Z[N - m], taken apart into the
    // (a_m, b_m) of both rows of each pair (the second unscaled)
#pragma unroll
    for (int i = 0; i < MH; i++) {
      const int idx = tid + i * NT, p = idx / M, m = idx % M, mm = (M - m) & (M - 1);
      const double2 t = tw[m];
      const double2 zk = cmulc(X[p * M + m], t), zn = cmulf(X[p * M + mm], t);
      const double ay = PB::factor(pmx[2 * p], pmx[2 * p + 1], true);
      if (m == 0) {
        o0[i].x += zk.x;
        o1[i].x += ay * zk.y;
      } else {
        o0[i].x += zk.x + zn.x; o0[i].y -= zk.y - zn.y;
        o1[i].x += ay * (zk.y + zn.y); o1[i].y += ay * (zk.x - zn.x);
      }
    }
    __syncthreads();   // X holds the next residue's transposes
  }
  const double an = 1.0 / (double)N;
#pragma unroll
  for (int i = 0; i < MH; i++) {
    const int idx = tid + i * NT, p = idx / M, m = idx % M;
    S2[(2 * p) * MP2 + m] = double2{an * o0[i].x, an * o0[i].y};
    S2[(2 * p + 1) * MP2 + m] = double2{an * o1[i].x, an * o1[i].y};
  }
  __syncthreads();
  {
    const int j = lane & 15, hw = lane >> 4;
    int c = 0;
    double *dst = fout.P;
    size_t mst = 0;
    if (j < 4) {
      c = 3 * j;
      dst = fout.P + (size_t)th * fout.sP() + (size_t)k * 8 + 2 * j;
      mst = (size_t)fout.nth * fout.sP();
    } else if (j < 12) {
      const int jd = j - 4;
      c = 3 * (jd >> 1) + 1 + (jd & 1);
      dst = fout.D + (size_t)th * fout.sD() + (size_t)k * 16 + 2 * jd;
      mst = (size_t)fout.nth * fout.sD();
    }
    if (j < 12)
      for (int m = 2 * warp + hw; m < M; m += 2 * nwarp)
        *reinterpret_cast<double2 *>(dst + m * mst) = S2[c * MP2 + m];
  }
}

// ---------------------------------------------------------------------------
// The general products kernel, either precision and any N = 2^a 3^b (the grids
// that are not nphi = 3 (L + 1) with L + 1 = 32 .. 256).  Stockham stages of
// radix 3, 4 and 2 over the seven (six) rows of a (theta, k), two stages a pass
// through shared memory: the R2 butterflies of the first stage whose outputs a
// second-stage butterfly reads are R2 rows of a thread's registers, so fusing
// changes no operation and no result.  Index divisions are multiplications,
// rows carry one pad element per 16, the input comes by cp.async, and the
// scaling of the product rows is applied where the first forward pass reads
// them.  Bound by latency: a few hundred butterflies a pass and barrier.  With
// a stage a pass, run-time radices and divisions -> now: float64 nphi = 256 /
// L85 / Nr65 (8320 rows) 1056 -> 334 us; single 614 -> 194 us there, 2600 ->
// 1107 us at nphi = 576 / L191 / Nr65 (18720 rows), 252 -> 76 us at nphi = 216 /
// L63 / Nr33.
struct GStage {
  int R1, R2, Ns;           // radices of the two stages (R2 = 1: one stage), product of the radices before
  int n12, nb1, ts1, ts2;   // N / (R1 R2), N / R1, N / (Ns R1), N / (Ns R1 R2)
  FastDiv d12, dNs;
};
struct GPlan {
  int n, np, nst;           // points, padded row length, passes
  int psh;                  // index i lies at i + (i >> psh)
  int mp;                   // pitch of a staging row of L + 1 orders
  GStage st[12];
  __device__ __forceinline__ int pad(int i) const { return i + (i >> psh); }
};

template <typename T>
static size_t gplan_bytes(int np) { return 14 * (size_t)np * 2 * sizeof(T) + 32 * sizeof(double); }

template <typename T>
static GPlan make_gplan(int n, int L) {
  GPlan p{};
  p.n = n;
  // the largest float64 grids fit without the padding only, the smallest grids
  // with an even staging pitch only
  p.psh = gplan_bytes<T>(n + n / 16 + 1) <= 227 * 1024 ? 4 : 31;
  p.np = p.psh == 4 ? n + n / 16 + 1 : n;
  p.mp = 13 * ((L + 1) | 1) <= 7 * p.np ? (L + 1) | 1 : L + 1;
  int rad[24], nr = 0, m = n, Ns = 1;
  while (m % 3 == 0) { rad[nr++] = 3; m /= 3; }
  while (m % 4 == 0) { rad[nr++] = 4; m /= 4; }
  if (m % 2 == 0) rad[nr++] = 2;
  for (int i = 0; i < nr; i += 2) {
    const int R1 = rad[i], R2 = (i + 1 < nr) ? rad[i + 1] : 1;
    p.st[p.nst++] = GStage{R1, R2, Ns, n / (R1 * R2), n / R1, n / (Ns * R1), n / (Ns * R1 * R2), FastDiv(n / (R1 * R2)),
                           FastDiv(Ns)};
    Ns *= R1 * R2;
  }
  return p;
}

// Products and sums of two products, in single precision with the rounding
// written out: the results do not depend on how the compiler contracts them
// where the passes are inlined (they are those of one stage a pass, bit for bit).
__device__ __forceinline__ float2 gmul(float2 a, float2 b) {
  return float2{__fmaf_rn(a.x, b.x, -__fmul_rn(a.y, b.y)), __fmaf_rn(a.y, b.x, __fmul_rn(a.x, b.y))};
}
__device__ __forceinline__ double2 gmul(double2 a, double2 b) { return cmul(a, b); }
__device__ __forceinline__ float gdet(float a, float b, float c, float d) {   // a b - c d
  return __fmaf_rn(a, b, -__fmul_rn(c, d));
}
__device__ __forceinline__ double gdet(double a, double b, double c, double d) { return a * b - c * d; }
__device__ __forceinline__ float gfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double gfma(double a, double b, double c) { return fma(a, b, c); }

// butterfly of R points, natural order in and out
template <int R, int SIGN, typename T2>
__device__ __forceinline__ void gbf(T2 (&v)[R]) {
  using T = typename ScalarOf<T2>::t;
  T2 o[R];
  if constexpr (R == 4) {
    T2 a0, a1, a2, a3;
    a0.x = v[0].x + v[2].x; a0.y = v[0].y + v[2].y;
    a1.x = v[0].x - v[2].x; a1.y = v[0].y - v[2].y;
    a2.x = v[1].x + v[3].x; a2.y = v[1].y + v[3].y;
    T dx = v[1].x - v[3].x, dy = v[1].y - v[3].y;
    if (SIGN < 0) { a3.x = dy; a3.y = -dx; } else { a3.x = -dy; a3.y = dx; }
    o[0].x = a0.x + a2.x; o[0].y = a0.y + a2.y;
    o[1].x = a1.x + a3.x; o[1].y = a1.y + a3.y;
    o[2].x = a0.x - a2.x; o[2].y = a0.y - a2.y;
    o[3].x = a1.x - a3.x; o[3].y = a1.y - a3.y;
  } else if constexpr (R == 2) {
    o[0].x = v[0].x + v[1].x; o[0].y = v[0].y + v[1].y;
    o[1].x = v[0].x - v[1].x; o[1].y = v[0].y - v[1].y;
  } else if constexpr (R == 3) {
    const T s32 = (T)(0.5 * sqrt(3.0));
    T2 t1, t2;
    t1.x = v[1].x + v[2].x; t1.y = v[1].y + v[2].y;
    t2.x = v[0].x - (T)0.5 * t1.x; t2.y = v[0].y - (T)0.5 * t1.y;
    const T dx = v[1].x - v[2].x, dy = v[1].y - v[2].y, sx = SIGN < 0 ? s32 : -s32;
    o[0].x = v[0].x + t1.x; o[0].y = v[0].y + t1.y;
    o[1].x = gfma(sx, dy, t2.x); o[1].y = gfma(-sx, dx, t2.y);
    o[2].x = gfma(-sx, dy, t2.x); o[2].y = gfma(sx, dx, t2.y);
  } else {
    o[0] = v[0];
  }
#pragma unroll
  for (int r = 0; r < R; r++) v[r] = o[r];
}

// one pass.  The butterflies j0 + r' n12 (r' < R2) of the first stage have one
// k = j0 mod Ns and feed the second stage's butterflies k + r Ns (r < R1) of
// the same block.  mx (first pass of the forward transform): maxima of the
// rows, the second row of each pair scaled to the first on the way in.
template <int R1, int R2, int SIGN, typename T2>
__device__ __forceinline__ void g_pass(const T2 *x, T2 *y, int nf, const GPlan &pl, const GStage &st,
                                       const T2 *__restrict__ tw, const unsigned *mx) {
  using T = typename ScalarOf<T2>::t;
  const int Ns = st.Ns;
  for (int idx = threadIdx.x; idx < nf * st.n12; idx += blockDim.x) {
    const int f = st.d12.div(idx), j0 = idx - f * st.n12, J = st.dNs.div(j0), k = j0 - J * Ns;
    const T2 *xf = x + f * pl.np;
    T2 v[R2][R1], w[R1];
#pragma unroll
    for (int r = 1; r < R1; r++) {
      w[r] = __ldg(tw + r * k * st.ts1);
      if (SIGN > 0) w[r].y = -w[r].y;
    }
    T sy = (T)1;
    if (SIGN < 0 && mx) sy = PairBits<T>::factor(mx[2 * f], mx[2 * f + 1], false);
#pragma unroll
    for (int q = 0; q < R2; q++) {
#pragma unroll
      for (int r = 0; r < R1; r++) {
        T2 a = xf[pl.pad(j0 + q * st.n12 + r * st.nb1)];
        if (SIGN < 0 && mx) a.y *= sy;
        if (r > 0 && k > 0) a = gmul(a, w[r]);
        v[q][r] = a;
      }
      gbf<R1, SIGN>(v[q]);
    }
    T2 *yf = y + f * pl.np;
    const int d = J * Ns * (R1 * R2);
#pragma unroll
    for (int r = 0; r < R1; r++) {
      const int kk = k + r * Ns;
      T2 u[R2];
#pragma unroll
      for (int q = 0; q < R2; q++) {
        T2 a = v[q][r];
        if (q > 0 && kk > 0) {
          T2 z = __ldg(tw + q * kk * st.ts2);
          if (SIGN > 0) z.y = -z.y;
          a = gmul(a, z);
        }
        u[q] = a;
      }
      gbf<R2, SIGN>(u);
#pragma unroll
      for (int q = 0; q < R2; q++) yf[pl.pad(d + kk + q * Ns * R1)] = u[q];
    }
  }
  __syncthreads();
}

template <int SIGN, typename T2>
__device__ __forceinline__ T2 *g_fft(T2 *x, T2 *y, int nf, const GPlan &pl, const T2 *__restrict__ tw,
                                     const unsigned *mx = nullptr) {
  for (int s = 0; s < pl.nst; s++) {
    const GStage &st = pl.st[s];
    const unsigned *m0 = (s == 0) ? mx : nullptr;
    switch (st.R1 * 8 + st.R2) {
      case 3 * 8 + 3: g_pass<3, 3, SIGN>(x, y, nf, pl, st, tw, m0); break;
      case 3 * 8 + 4: g_pass<3, 4, SIGN>(x, y, nf, pl, st, tw, m0); break;
      case 3 * 8 + 2: g_pass<3, 2, SIGN>(x, y, nf, pl, st, tw, m0); break;
      case 3 * 8 + 1: g_pass<3, 1, SIGN>(x, y, nf, pl, st, tw, m0); break;
      case 4 * 8 + 4: g_pass<4, 4, SIGN>(x, y, nf, pl, st, tw, m0); break;
      case 4 * 8 + 2: g_pass<4, 2, SIGN>(x, y, nf, pl, st, tw, m0); break;
      case 4 * 8 + 1: g_pass<4, 1, SIGN>(x, y, nf, pl, st, tw, m0); break;
      default: g_pass<2, 1, SIGN>(x, y, nf, pl, st, tw, m0); break;
    }
    T2 *t = x; x = y; y = t;
  }
  return x;
}

template <typename T>
__global__ void __launch_bounds__(512)
k_fft_products_g(const __grid_constant__ GPlan pl, int L, MLayoutT<T> fin, MLayoutT<T> fout,
                 const typename C2<T>::t *__restrict__ tw, ProdCoef pc) {
  using T2 = typename C2<T>::t;
  using PB = PairBits<T>;
  using U = unsigned;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int N = pl.n, NP = pl.np, MP = pl.mp;
  T2 *A = reinterpret_cast<T2 *>(smraw);      // 7 rows
  T2 *B = A + 7 * NP;                          // 7 rows; first the input, last the output staging
  U *cmx = reinterpret_cast<U *>(B + 7 * NP);  // [0, 13) input maxima, [13, 25) products
  T2 *S = B;                                   // [c][MP] (a_m, b_m)
  const int th = blockIdx.x / fin.nr, k = blockIdx.x % fin.nr;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarp = blockDim.x >> 5;
  if (tid < 12) cmx[13 + tid] = 0;
  // input: an order's 13 (cos, sin) pairs, a run of 5 in the P block and one of
  // 8 in the D block; half-warp h of warp w copies the orders 2 (w + nwarp i) + h
  {
    const int j = lane & 15, hw = lane >> 4;
    int c = 0;
    const T *src = fin.P;
    size_t mst = 0;
    if (j < 5) {
      c = (j < 4) ? 3 * j : 12;
      src = fin.P + (size_t)th * fin.sP() + (size_t)k * 10 + 2 * j;
      mst = (size_t)fin.nth * fin.sP();
    } else if (j < 13) {
      const int jd = j - 5;
      c = 3 * (jd >> 1) + 1 + (jd & 1);
      src = fin.D + (size_t)th * fin.sD() + (size_t)k * 16 + 2 * jd;
      mst = (size_t)fin.nth * fin.sD();
    }
    if (j < 13)
      for (int m = 2 * warp + hw; m <= L; m += 2 * nwarp)
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((uint32_t)__cvta_generic_to_shared(S + c * MP + m)),
                     "l"(src + m * mst), "n"(sizeof(T2))
                     : "memory");
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
  }
  __syncthreads();
  // pair scaling (pair_exp): the largest coefficient of each component
  for (int c = warp; c < 13; c += nwarp) {
    U mx = 0;
    for (int m = lane; m <= L; m += 32) {
      const T2 v = S[c * MP + m];
      mx = max(mx, max(PB::abs_bits(v.x), PB::abs_bits(v.y)));
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane == 0) cmx[c] = mx;
  }
  __syncthreads();
  // Hermitian rows z = x + i y of the 7 pairs, the second row scaled
  const int mmax = min(L, (N + 1) / 2 - 1);
  for (int p = 0; p < 7; p++) {
    const bool has1 = p < 6;
    const T sy = has1 ? PB::factor(cmx[2 * p], cmx[2 * p + 1], false) : (T)1;
    const T2 *x0 = S + (2 * p) * MP, *y0 = has1 ? x0 + MP : x0;
    T2 *Z = A + p * NP;
    for (int m = tid; m <= mmax; m += blockDim.x) {
      const T2 ab = x0[m], cd = y0[m];
      const T a1 = has1 ? cd.x * sy : (T)0, b1 = has1 ? cd.y * sy : (T)0;
      if (m == 0) {
        Z[0] = T2{ab.x, a1};
      } else {
        const T xr = (T)0.5 * ab.x, xi = (T)-0.5 * ab.y, yr = (T)0.5 * a1, yi = (T)-0.5 * b1;
        Z[pl.pad(m)] = T2{xr - yi, xi + yr};
        Z[pl.pad(N - m)] = T2{xr + yi, -xi + yr};
      }
    }
    for (int n = mmax + 1 + tid; n < N - mmax; n += blockDim.x) Z[pl.pad(n)] = T2{0, 0};
  }
  __syncthreads();
  T2 *g = g_fft<+1>(A, B, 7, pl, tw);
  T2 *h = (g == A) ? B : A;
  {
    const T cv = (T)pc.cv, cl = (T)pc.cl, ci = (T)pc.ci, ct = (T)pc.ct;
    T iy[6];
#pragma unroll
    for (int p = 0; p < 6; p++) iy[p] = PB::factor(cmx[2 * p], cmx[2 * p + 1], true);
    U hm[12];
#pragma unroll
    for (int c = 0; c < 12; c++) hm[c] = 0;
    for (int qq = tid; qq < N; qq += blockDim.x) {
      const int q = pl.pad(qq);
      const T2 p0 = g[0 * NP + q], p1 = g[1 * NP + q], p2 = g[2 * NP + q], p3 = g[3 * NP + q];
      const T2 p4 = g[4 * NP + q], p5 = g[5 * NP + q], p6 = g[6 * NP + q];
      const T ur = p0.x, ut = p0.y * iy[0], up = p1.x, wr = p1.y * iy[1], wt = p2.x, wp = p2.y * iy[2];
      const T br = p3.x, bt = p3.y * iy[3], bp = p4.x, jr = p4.y * iy[4], jt = p5.x, jp = p5.y * iy[5], tt = p6.x;
      const T2 hv[6] = {T2{gdet(wt, up, wp, ut) * cv, gdet(wp, ur, wr, up) * cv},
                        T2{gdet(wr, ut, wt, ur) * cv, gdet(jt, bp, jp, bt) * cl},
                        T2{gdet(jp, br, jr, bp) * cl, gdet(jr, bt, jt, br) * cl},
                        T2{gdet(ut, bp, up, bt) * ci, gdet(up, br, ur, bp) * ci},
                        T2{gdet(ur, bt, ut, br) * ci, ur * tt * ct},
                        T2{ut * tt * ct, up * tt * ct}};
#pragma unroll
      for (int p = 0; p < 6; p++) {
        h[p * NP + q] = hv[p];
        hm[2 * p] = max(hm[2 * p], PB::abs_bits(hv[p].x));
        hm[2 * p + 1] = max(hm[2 * p + 1], PB::abs_bits(hv[p].y));
      }
    }
#pragma unroll
    for (int c = 0; c < 12; c++) {
      const U v = __reduce_max_sync(0xffffffffu, hm[c]);
      if (lane == 0) atomicMax(cmx + 13 + c, v);
    }
  }
  __syncthreads();
  const T2 *zf = g_fft<-1>(h, g, 6, pl, tw, cmx + 13);
  T2 *O = (zf == A) ? B : A;   // [c][MP] (a_m, b_m)
  const T an = (T)(1.0 / (double)N);
  for (int p = 0; p < 6; p++) {
    const T2 *Z = zf + p * NP;
    T2 *o0 = O + (2 * p) * MP, *o1 = o0 + MP;
    const T ay = an * PB::factor(cmx[13 + 2 * p], cmx[14 + 2 * p], true);
    for (int m = tid; m <= L; m += blockDim.x) {
      if (m == 0) {
        o0[0] = T2{an * Z[0].x, (T)0};
        o1[0] = T2{ay * Z[0].y, (T)0};
      } else {
        const T2 zk = Z[pl.pad(m % N)], zn = Z[pl.pad((N - m) % N)];
        o0[m] = T2{an * (zk.x + zn.x), -an * (zk.y - zn.y)};
        o1[m] = T2{ay * (zk.y + zn.y), ay * (zk.x - zn.x)};
      }
    }
  }
  __syncthreads();
  // output: 12 pairs an order, a run of 4 in the P block and one of 8 in the D block
  {
    const int j = lane & 15, hw = lane >> 4;
    int c = 0;
    T *dst = fout.P;
    size_t mst = 0;
    if (j < 4) {
      c = 3 * j;
      dst = fout.P + (size_t)th * fout.sP() + (size_t)k * 8 + 2 * j;
      mst = (size_t)fout.nth * fout.sP();
    } else if (j < 12) {
      const int jd = j - 4;
      c = 3 * (jd >> 1) + 1 + (jd & 1);
      dst = fout.D + (size_t)th * fout.sD() + (size_t)k * 16 + 2 * jd;
      mst = (size_t)fout.nth * fout.sD();
    }
    if (j < 12)
      for (int m = 2 * warp + hw; m <= L; m += 2 * nwarp) *reinterpret_cast<T2 *>(dst + m * mst) = O[c * MP + m];
  }
}

// order-major Fourier rows -> grid (float64), for the standalone transform API.
// The rows lie far apart in m, so a (cos, sin) pair is one access, made once:
// the pairs wait in the other buffer of the transform for the pair scaling.
// Bound by the latency of the passes (block_fft): in float64 eight blocks an SM,
// as many as without the pair scaling.  13 components at nphi = 384 / L127 / Nr33
// 852 us (the pairs read twice, five blocks) -> 629 us, and the way back 768 ->
// 632 (six).
template <typename T> constexpr int kGridBlocks = sizeof(T) == 8 ? 8 : 6;
template <typename T>
__global__ void __launch_bounds__(256, kGridBlocks<T>)
k_fft_to_grid_m(FFTPlan pl, int L, MLayoutT<T> fin, double *grid, const typename C2<T>::t *tw) {
  using T2 = typename C2<T>::t;
  using PB = PairBits<T>;
  using U = typename PB::U;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int N = pl.n, nc = 3 * fin.nvec + fin.nscal, nr = fin.nr, nth = fin.nth;
  T2 *Z0 = reinterpret_cast<T2 *>(smraw), *Z1 = Z0 + N;
  const int th = blockIdx.x / nr, k = blockIdx.x % nr;
  const int mmax = min(L, (N + 1) / 2 - 1);
  __shared__ U pmx[2];
  for (int c = 0; c < nc; c += 2) {
    const bool has1 = c + 1 < nc;
    if (threadIdx.x < 2) pmx[threadIdx.x] = 0;
    for (int q = threadIdx.x; q < N; q += blockDim.x) Z0[q] = T2{0, 0};
    __syncthreads();
    // pair scaling (pair_exp): the second row, if there is one, brought to the
    // size of the first
    T sy = (T)1, iy = (T)1;
    {
      U mx = 0, my = 0;
      for (int m = threadIdx.x; m <= mmax; m += blockDim.x) {
        const T2 v = __ldg(reinterpret_cast<const T2 *>(fin.at(m, th, k, c, 0)));
        const T2 w = has1 ? __ldg(reinterpret_cast<const T2 *>(fin.at(m, th, k, c + 1, 0))) : T2{0, 0};
        Z1[2 * m] = v;
        Z1[2 * m + 1] = w;
        mx = max(mx, max(PB::abs_bits(v.x), PB::abs_bits(v.y)));
        my = max(my, max(PB::abs_bits(w.x), PB::abs_bits(w.y)));
      }
      if (has1) {
        mx = __reduce_max_sync(0xffffffffu, mx);
        my = __reduce_max_sync(0xffffffffu, my);
        if ((threadIdx.x & 31) == 0) { atomicMax(pmx, mx); atomicMax(pmx + 1, my); }
        __syncthreads();
        sy = PB::factor(pmx[0], pmx[1], false);
        iy = PB::factor(pmx[0], pmx[1], true);
      }
    }
    for (int m = threadIdx.x; m <= mmax; m += blockDim.x) {
      const T2 v = Z1[2 * m], w = Z1[2 * m + 1];   // this thread's own
      const T a0 = v.x, b0 = v.y, a1 = w.x * sy, b1 = w.y * sy;
      if (m == 0) {
        Z0[0] = T2{a0, a1};
      } else {
        const T xr = (T)0.5 * a0, xi = (T)-0.5 * b0, yr = (T)0.5 * a1, yi = (T)-0.5 * b1;
        Z0[m] = T2{xr - yi, xi + yr};
        Z0[N - m] = T2{xr + yi, -xi + yr};
      }
    }
    __syncthreads();
    T2 *z = block_fft<T, T2>(Z0, Z1, pl, tw, +1);
    for (int q = threadIdx.x; q < N; q += blockDim.x) {
      grid[(((size_t)c * nr + k) * nth + th) * N + q] = (double)z[q].x;
      if (has1) grid[(((size_t)(c + 1) * nr + k) * nth + th) * N + q] = (double)(z[q].y * iy);
    }
    __syncthreads();
  }
}

// grid (float64) -> order-major Fourier rows
template <typename T>
__global__ void __launch_bounds__(256, kGridBlocks<T>)
k_grid_to_fft_m(FFTPlan pl, int L, const double *grid, MLayoutT<T> fout, const typename C2<T>::t *tw) {
  using T2 = typename C2<T>::t;
  using PB = PairBits<T>;
  using U = typename PB::U;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int N = pl.n, nc = 3 * fout.nvec + fout.nscal, nr = fout.nr, nth = fout.nth;
  T2 *Z0 = reinterpret_cast<T2 *>(smraw), *Z1 = Z0 + N;
  const int th = blockIdx.x / nr, k = blockIdx.x % nr;
  const T an = (T)(1.0 / (double)N);
  __shared__ U pmx[2];
  for (int c = 0; c < nc; c += 2) {
    const bool has1 = c + 1 < nc;
    if (threadIdx.x < 2) pmx[threadIdx.x] = 0;
    __syncthreads();
    U mx = 0, my = 0;
    for (int q = threadIdx.x; q < N; q += blockDim.x) {
      const T x = (T)grid[(((size_t)c * nr + k) * nth + th) * N + q];
      const T y = has1 ? (T)grid[(((size_t)(c + 1) * nr + k) * nth + th) * N + q] : (T)0;
      Z0[q] = T2{x, y};
      mx = max(mx, PB::abs_bits(x));
      my = max(my, PB::abs_bits(y));
    }
    if (has1) {
      mx = __reduce_max_sync(0xffffffffu, mx);
      my = __reduce_max_sync(0xffffffffu, my);
      if ((threadIdx.x & 31) == 0) { atomicMax(pmx, mx); atomicMax(pmx + 1, my); }
    }
    __syncthreads();
    // pair scaling (pair_exp): the second row, if there is one, brought to the
    // size of the first
    T ay = an;
    if (has1) {
      const T sy = PB::factor(pmx[0], pmx[1], false);
      if (sy != (T)1) {
        for (int q = threadIdx.x; q < N; q += blockDim.x) Z0[q].y *= sy;
        __syncthreads();
      }
      ay = an * PB::factor(pmx[0], pmx[1], true);
    }
    const T2 *z = block_fft<T, T2>(Z0, Z1, pl, tw, -1);
    for (int m = threadIdx.x; m <= L; m += blockDim.x) {
      T a0, b0, a1, b1;
      if (m == 0) {
        a0 = an * z[0].x; b0 = (T)0; a1 = ay * z[0].y; b1 = (T)0;
      } else {
        const T2 zk = z[m % N], zn = z[(N - m) % N];
        const T xr = (T)0.5 * (zk.x + zn.x), xi = (T)0.5 * (zk.y - zn.y);
        const T yr = (T)0.5 * (zk.y + zn.y), yi = (T)-0.5 * (zk.x - zn.x);
        a0 = (T)2 * an * xr; b0 = (T)-2 * an * xi; a1 = (T)2 * ay * yr; b1 = (T)-2 * ay * yi;
      }
      *reinterpret_cast<T2 *>(fout.at(m, th, k, c, 0)) = T2{a0, b0};
      if (has1) *reinterpret_cast<T2 *>(fout.at(m, th, k, c + 1, 0)) = T2{a1, b1};
    }
    __syncthreads();
  }
}

__global__ void k_twiddles(int n, double2 *tw, float2 *tw32) {
  int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  double s, c;
  sincospi(2.0 * (double)e / (double)n, &s, &c);
  tw[e] = make_double2(c, -s);
  tw32[e] = make_float2((float)c, (float)-s);
}

static FFTPlan make_plan(int n) {
  FFTPlan p{};
  p.n = n;
  int m = n;
  while (m % 3 == 0) { p.rad[p.nst++] = 3; m /= 3; }
  while (m % 4 == 0) { p.rad[p.nst++] = 4; m /= 4; }
  while (m % 2 == 0) { p.rad[p.nst++] = 2; m /= 2; }
  if (m != 1) p.nst = -1;
  return p;
}

template <int N>
static size_t smem_fft_t() { return (14 * (size_t)Plan3x2<N>::NP + N) * sizeof(float2); }

// smem attribute and the per-stage twiddle table w^(r k) of Plan3x2<N>
template <int N>
static int attr_fft_t(Ctx &c) {
  using P = Plan3x2<N>;
  CB2_CUDA(raise_smem_limit(k_fft_products_t<N>, (int)smem_fft_t<N>()));
  std::vector<float2> t(P::ntw());
  const double pi = 3.14159265358979323846;
  for (int st = 0; st < P::nst(); st++) {
    const int R = P::radix(st), NS = P::ns(st), tstr = N / (NS * R);
    for (int r = 1; r < R; r++)
      for (int k = 0; k < NS; k++) {
        const double ang = -2.0 * pi * (double)(r * k * tstr) / (double)N;
        t[P::off(st) + (r - 1) * NS + k] = float2{(float)std::cos(ang), (float)std::sin(ang)};
      }
  }
  CB2_CUDA(cudaMalloc(&c.d_twp32, t.size() * sizeof(float2)));
  CB2_CUDA(cudaMemcpyAsync(c.d_twp32, t.data(), t.size() * sizeof(float2), cudaMemcpyHostToDevice, c.stream));
  return 0;
}

// smem attribute and the tables of the four-step kernel:
// [3][M] e^{2 pi i m r/N} (row 0 ones), [R2][R1 + 1] e^{2 pi i n2 k1/M}
template <int R1, int R2>
static int attr_fft_4s(Ctx &c) {
  using P = F4Plan<R1, R2>;
  CB2_CUDA(raise_smem_limit(k_fft_products_4s<R1, R2>, (int)P::smem()));
  std::vector<float2> t(3 * P::M + R2 * P::WP, float2{0.0f, 0.0f});
  const double pi = 3.14159265358979323846;
  for (int r = 0; r < 3; r++)
    for (int m = 0; m < P::M; m++) {
      const double ang = 2.0 * pi * (double)(m * r) / (double)P::N;
      t[r * P::M + m] = float2{(float)std::cos(ang), (float)std::sin(ang)};
    }
  for (int n2 = 0; n2 < R2; n2++)
    for (int k1 = 0; k1 < R1; k1++) {
      const double ang = 2.0 * pi * (double)(n2 * k1) / (double)P::M;
      t[3 * P::M + n2 * P::WP + k1] = float2{(float)std::cos(ang), (float)std::sin(ang)};
    }
  CB2_CUDA(cudaMalloc(&c.d_twf4, t.size() * sizeof(float2)));
  CB2_CUDA(cudaMemcpyAsync(c.d_twf4, t.data(), t.size() * sizeof(float2), cudaMemcpyHostToDevice, c.stream));
  return 0;
}

template <int R1, int R2>
static int attr_fft_4s64(Ctx &c) {
  using P = F4Plan64<R1, R2>;
  if constexpr (R2 == 16) CB2_CUDA(raise_smem_limit(k_fft_products_4s64r<R1, R2>, F4Plan64R<R1, R2>::smem()));
  else CB2_CUDA(raise_smem_limit(k_fft_products_4s64<R1, R2>, P::smem()));
  std::vector<double2> t(3 * P::M + R2 * P::WP, double2{0.0, 0.0});
  const double pi = 3.14159265358979323846;
  for (int r = 0; r < 3; r++)
    for (int m = 0; m < P::M; m++) {
      const double ang = 2.0 * pi * (double)(m * r) / (double)P::N;
      t[r * P::M + m] = double2{std::cos(ang), std::sin(ang)};
    }
  for (int n2 = 0; n2 < R2; n2++)
    for (int k1 = 0; k1 < R1; k1++) {
      const double ang = 2.0 * pi * (double)(n2 * k1) / (double)P::M;
      t[3 * P::M + n2 * P::WP + k1] = double2{std::cos(ang), std::sin(ang)};
    }
  CB2_CUDA(cudaMalloc(&c.d_twf4_64, t.size() * sizeof(double2)));
  CB2_CUDA(cudaMemcpyAsync(c.d_twf4_64, t.data(), t.size() * sizeof(double2), cudaMemcpyHostToDevice, c.stream));
  return 0;
}

int fft_setup(Ctx &c) {
  FFTPlan p = make_plan(c.nph);
  if (p.nst < 0) {
    set_error("ngrid_zonal_ctl must be of the form 3^a 2^b");
    return CB2_ERR_ARG;
  }
  CB2_CUDA(cudaMalloc(&c.d_tw_fft, (size_t)c.nph * sizeof(double2)));
  CB2_CUDA(cudaMalloc(&c.d_tw_fft32, (size_t)c.nph * sizeof(float2)));
  k_twiddles<<<cdiv(c.nph, 256), 256, 0, c.stream>>>(c.nph, (double2 *)c.d_tw_fft,
                                                     (float2 *)c.d_tw_fft32);
  CB2_CUDA(cudaGetLastError());
  if (14 * (size_t)c.nph * sizeof(double2) + 32 * sizeof(double) > 227 * 1024) {
    set_error("ngrid_zonal_ctl too large for the fused FFT kernel");
    return CB2_ERR_ARG;
  }
  if (c.prec == CB2_PREC_FP64) CB2_CUDA(raise_smem_limit(k_fft_products_g<double>, gplan_bytes<double>(make_gplan<double>(c.nph, c.L).np)));
  else CB2_CUDA(raise_smem_limit(k_fft_products_g<float>, gplan_bytes<float>(make_gplan<float>(c.nph, c.L).np)));
  {
    int rc = 0;
    switch (c.nph) {
      case 768: rc = attr_fft_t<768>(c); break;
      case 384: rc = attr_fft_t<384>(c); break;
      case 192: rc = attr_fft_t<192>(c); break;
      case 96: rc = attr_fft_t<96>(c); break;
      default: break;
    }
    if (rc) return rc;
    if (c.nph == 3 * (c.L + 1)) {
      switch (c.nph) {
        case 768: rc = attr_fft_4s<16, 16>(c); break;
        case 384: rc = attr_fft_4s<16, 8>(c); break;
        case 192: rc = attr_fft_4s<8, 8>(c); break;
        case 96: rc = attr_fft_4s<8, 4>(c); break;
        default: break;
      }
      if (rc) return rc;
      switch (c.nph) {
        case 768: rc = attr_fft_4s64<16, 16>(c); break;
        case 384: rc = attr_fft_4s64<16, 8>(c); break;
        case 192: rc = attr_fft_4s64<8, 8>(c); break;
        case 96: rc = attr_fft_4s64<8, 4>(c); break;
        default: break;
      }
      if (rc) return rc;
    }
  }
  if (26 * (size_t)(c.L + 1) * sizeof(float) > 7 * (size_t)c.nph * sizeof(float2)) {
    set_error("ngrid_zonal_ctl too small for the staging of the fused FFT kernel");
    return CB2_ERR_ARG;
  }
  return 0;
}

template <typename T>
static const typename C2<T>::t *twid(Ctx &c) {
  if (sizeof(T) == 8) return (const typename C2<T>::t *)c.d_tw_fft;
  return (const typename C2<T>::t *)c.d_tw_fft32;
}

template <typename T>
static void launch_fft_g(Ctx &c, const MLayoutT<T> &in, const MLayoutT<T> &out, const ProdCoef &pc) {
  const GPlan pl = make_gplan<T>(c.nph, c.L);
  // about a thread per pair-stage butterfly of the seven rows
  const int threads = std::min(512, std::max(96, 32 * cdiv(7 * c.nph, 16 * 32)));
  k_fft_products_g<T><<<(unsigned)(c.nth * c.nr), threads, gplan_bytes<T>(pl.np), c.stream>>>(pl, c.L, in, out,
                                                                                               twid<T>(c), pc);
}

template <int R1, int R2>
static void launch_fft_4s64(Ctx &c, const MLayout64 &in, const MLayout64 &out, const ProdCoef &pc) {
  if constexpr (R2 == 16)
    k_fft_products_4s64r<R1, R2><<<(unsigned)(c.nth * c.nr), F4Plan64R<R1, R2>::NT, F4Plan64R<R1, R2>::smem(),
                                   c.stream>>>(in, out, (const double2 *)c.d_twf4_64, pc);
  else k_fft_products_4s64<R1, R2><<<(unsigned)(c.nth * c.nr), f4_threads<R2>(), F4Plan64<R1, R2>::smem(), c.stream>>>(
      in, out, (const double2 *)c.d_twf4_64, pc);
}

void fft_products64(Ctx &c, const MLayout64 &in, const MLayout64 &out) {
  const ProdCoef pc{c.p.coef_velo, c.p.coef_lor, c.p.coef_induct, c.p.coef_temp};
  // tuning value F4_THREADS selects the four-step kernel where it applies
  if (c.d_twf4_64 && c.tune[TUNE_FFT_THREADS] == F4_THREADS) {
    switch (c.nph) {
      case 768: launch_fft_4s64<16, 16>(c, in, out, pc); return;
      case 384: launch_fft_4s64<16, 8>(c, in, out, pc); return;
      case 192: launch_fft_4s64<8, 8>(c, in, out, pc); return;
      case 96: launch_fft_4s64<8, 4>(c, in, out, pc); return;
      default: break;
    }
  }
  launch_fft_g<double>(c, in, out, pc);
}

template <typename T>
void fft_backward_grid(Ctx &c, const MLayoutT<T> &in, double *grid) {
  const size_t sm = 2 * (size_t)c.nph * sizeof(typename C2<T>::t);
  k_fft_to_grid_m<T><<<(unsigned)(c.nth * c.nr), 256, sm, c.stream>>>(make_plan(c.nph), c.L, in, grid, twid<T>(c));
}

template <typename T>
void fft_forward_grid(Ctx &c, const double *grid, const MLayoutT<T> &out) {
  const size_t sm = 2 * (size_t)c.nph * sizeof(typename C2<T>::t);
  k_grid_to_fft_m<T><<<(unsigned)(c.nth * c.nr), 256, sm, c.stream>>>(make_plan(c.nph), c.L, grid, out, twid<T>(c));
}

template <int N>
static void launch_fft_t(Ctx &c, const MLayout &in, const MLayout &out, const ProdCoef &pc) {
  const size_t sm = smem_fft_t<N>();
  const int nt = c.tune[TUNE_FFT_THREADS];
  const int threads = (nt == 128 || nt == 256) ? nt : 512;
  k_fft_products_t<N><<<(unsigned)(c.nth * c.nr), threads, sm, c.stream>>>(c.L, in, out, (const float2 *)c.d_twp32,
                                                                          pc);
}

template <int R1, int R2>
static bool launch_fft_4s(Ctx &c, const MLayout &in, const MLayout &out, const ProdCoef &pc, float *pmax) {
  k_fft_products_4s<R1, R2><<<(unsigned)(c.nth * c.nr), f4_threads<R2>(), F4Plan<R1, R2>::smem(), c.stream>>>(
      in, out, (const float2 *)c.d_twf4, pc, pmax, pmax ? mixed_weights32(c) : nullptr);
  return pmax != nullptr;
}

bool fft_products_m(Ctx &c, const MLayout &in, const MLayout &out, float *pmax) {
  ProdCoef pc{c.p.coef_velo, c.p.coef_lor, c.p.coef_induct, c.p.coef_temp};
  // tuning value F4_THREADS selects the four-step kernel where it applies
  if (c.d_twf4 && c.tune[TUNE_FFT_THREADS] == F4_THREADS) {
    switch (c.nph) {
      case 768: return launch_fft_4s<16, 16>(c, in, out, pc, pmax);
      case 384: return launch_fft_4s<16, 8>(c, in, out, pc, pmax);
      case 192: return launch_fft_4s<8, 8>(c, in, out, pc, pmax);
      case 96: return launch_fft_4s<8, 4>(c, in, out, pc, pmax);
      default: break;
    }
  }
  switch (c.nph) {
    case 768: launch_fft_t<768>(c, in, out, pc); return false;
    case 384: launch_fft_t<384>(c, in, out, pc); return false;
    case 192: launch_fft_t<192>(c, in, out, pc); return false;
    case 96: launch_fft_t<96>(c, in, out, pc); return false;
    default: break;
  }
  launch_fft_g<float>(c, in, out, pc);
  return false;
}

template void fft_backward_grid<double>(Ctx &, const MLayout64 &, double *);
template void fft_backward_grid<float>(Ctx &, const MLayout &, double *);
template void fft_forward_grid<double>(Ctx &, const double *, const MLayout64 &);
template void fft_forward_grid<float>(Ctx &, const double *, const MLayout &);

}  // namespace cb2
