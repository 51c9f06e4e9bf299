// cb2_legendre_f64.cu -- float64 Legendre transforms (the plain path) on the
// float64 tensor cores (mma.sync m16n8k4, f64 in and out).
//
// Definition: PARALLEL_src/SPH_SHELL_src/legendre_bwd_trans_org.f90:45-209 and
// legendre_fwd_trans_org.f90:45-169 of the reference, evaluated with the
// equatorial symmetry that its SYMMETRIC_MATMUL variant uses
// (cal_vr_rtm_by_matmul.f90, cal_sp_rlm_by_matmul.f90):
//   P_l^m(pi - theta) = (-1)^(l-m) P_l^m(theta),
//   dP_l^m/dtheta (pi - theta) = -(-1)^(l-m) dP_l^m/dtheta (theta).
//
// Per order m both transforms are products of the basis tables with columns:
//   P block  (k, field, s): the poloidal / r component of a vector or a scalar
//   D block  (k, vector, q): the two tangential parts of a vector,
//            spectra   X = [D+, D-, T+, T-]  (D = dS/dr, T toroidal; +-m),
//            grid rows X = [t+, t-, p+, p-]  (theta, phi components),
// in the order of the Fourier rows (MLayout64: [m][theta][(k, element)]), so a
// tile of 64 columns is a run of 512 bytes of a row.  A column q of the D
// block takes the dP products of X[q] and the m P / sin(theta) products of
// X[3 - q] = X[q ^ 3]: within an 8-column fragment that is the value of the
// lane 12 away, so one staged copy of X serves both.
//
// Bounds: at L255 / Nr129 the sums are 6.8e10 flop backward (4 vectors + 1
// scalar) and 6.5e10 forward (4 vectors), 1.84 and 1.76 ms at the 37 TF/s that
// mma f64 (and DFMA) reach on a B200; the traffic is 0.55 ms.  The earlier kernels (a block per 2 radial levels over
// theta-major rows, whose 16-byte pieces of an order lie 53 KB apart, the B
// matrices of both products built in shared memory for each chunk) took 7.3 ms
// backward and 8.8 ms forward; these take 3.02 ms and 3.28 ms, 61 % and 54 %
// of that rate in useful flops, the matrix pipe 64 % and 60 % busy (padding of
// the tiles counted).
#include <algorithm>

#include "cb2_internal.cuh"

namespace cb2 {

namespace {

constexpr int LTH = 128;     // threads of a block: 4 warps, 16 columns each
constexpr int LNB = 64;      // columns of a block
constexpr int LST = 3;       // cp.async stages
constexpr int MAXF = 13;     // fields (vectors + scalars) of a launch

// asynchronous copies global -> shared; n = 0 fills zeros and reads nothing
__device__ inline void cp_async8(double *dst, const double *src, int n) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(n)
               : "memory");
}
__device__ inline void cp_async16(double *dst, const double *src, int n) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(n)
               : "memory");
}
__device__ inline void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// every group but the newest LST - 2 has landed
__device__ inline void cp_async_wait_stage() { asm volatile("cp.async.wait_group %0;" ::"n"(LST - 2) : "memory"); }

__device__ __forceinline__ void dmma16n8k4(double (&d)[4], double a0, double a1, double b0) {
  asm volatile("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
               : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
               : "d"(a0), "d"(a1), "d"(b0));
}

struct LegArgs {
  int L, nr, nth, nh, jmax, nvec, nscal, tilesP;
  int slot[MAXF];           // first rj slot of each field
  const int *moff;
  const size_t *poff;
  const double *Plt, *dPlt, *asin_t, *wgt;
  const double *g6, *g7, *r, *ar1;
  double *f;                // rj fields
  size_t fs;                // slot stride
  MLayout64 four;
};

// the columns of a block: where column c of its 64 lies in the spectra (offset
// of degree l = m; -1: a zero column, not stored), its radial factor and kind
struct LegCols {
  long long off[LNB];
  double fac[LNB];
  int kind[LNB];            // 1: the poloidal part of a vector, 0: a scalar, 2: D block
};

// rp1: the factor of the tangential parts (1 / r backward, r forward); the
// poloidal part takes its square.  The products of the columns q >= 2 are
// formed with the opposite sign.
__device__ inline void leg_columns(const LegArgs &a, int m, bool isD, int c0, const double *rp1, LegCols &t) {
  const int G = a.nvec + a.nscal, per = isD ? 4 * a.nvec : 2 * G, ncols = a.nr * per, nl = a.L + 1 - m;
  for (int i = threadIdx.x; i < LNB; i += LTH) {
    const int c = c0 + i;
    long long off = -1;
    double fac = 0.0;
    int kind = 2;
    if (c < ncols) {
      const int k = c / per, x = c - k * per, g = isD ? x >> 2 : x >> 1, s = x & 1;
      const int slot = a.slot[g] + (isD ? 1 + ((x & 3) >> 1) : 0);
      const double rr = rp1[k];
      if (isD) {
        fac = ((x & 3) >= 2) ? -rr : rr;
      } else {
        kind = (g < a.nvec) ? 1 : 0;
        fac = kind ? rr * rr : 1.0;
      }
      if (!(m == 0 && s == 1))
        off = (long long)slot * (long long)a.fs + (long long)k * a.jmax + a.moff[m] + s * nl;
    }
    t.off[i] = off; t.fac[i] = fac; t.kind[i] = kind;
  }
}

// ---------------------------------------------------------------------------
// Backward: rows 16 MF south nodes (and their mirrors), columns 64, K the
// degrees of one order in chunks of 16, 8 of each reflection parity.  The sums
// of each parity stay apart: south = sigma 0 + sigma 1, mirror = sigma 0 -
// sigma 1; P and m P / sin add to sigma = p, dP to 1 - p.  The spectra are
// staged straight from the field slots ([column][parity][degree]: runs of 16
// degrees), l(l+1) and m / sin(theta) applied to the fragments, 1 / r in the
// epilogue.  MF = 3 (48 nodes) divides the hemispheres of the standard grids
// (24 2^i colatitudes); up to 32 nodes take MF = 2.  Pitches of 4 mod 16
// doubles keep the fragment reads free of bank conflicts.
template <int MF>
struct BwdTileSz {
  static constexpr int NM = 16 * MF, AP = NM + 4, BP = 20;
  static constexpr int SA = 16 * AP, SB = LNB * BP, STG = 2 * SA + SB;
  static constexpr size_t smem() { return LST * (size_t)STG * sizeof(double) + sizeof(LegCols); }
};

template <int MF>
__global__ void __launch_bounds__(LTH, 3)
k_leg_bwd_f64(const __grid_constant__ LegArgs a) {
  using Z = BwdTileSz<MF>;
  constexpr int NM = Z::NM, AP = Z::AP, BP = Z::BP;
  extern __shared__ __align__(16) double smb[];
  LegCols &tc = *reinterpret_cast<LegCols *>(smb + LST * Z::STG);
  const int m = blockIdx.z, i0 = blockIdx.x * NM;
  const bool isD = (int)blockIdx.y >= a.tilesP;
  const int c0 = ((int)blockIdx.y - (isD ? a.tilesP : 0)) * LNB;
  const int tid = threadIdx.x, lane = tid & 31, wc = tid >> 5, gq = lane >> 2, tq = lane & 3;
  const int nl = a.L + 1 - m;
  leg_columns(a, m, isD, c0, a.ar1, tc);
  __syncthreads();
  const size_t po = a.poff[m];
  const bool pair16 = (a.nh & 1) == 0;   // else a table row starts off a 16-byte boundary
  auto issue = [&](int ch) {
    const int lc0 = ch * 16;
    if (lc0 < nl) {
      double *Ps = smb + (ch % LST) * Z::STG, *dPs = Ps + Z::SA, *B = dPs + Z::SA;
      if (pair16) {
        for (int e = tid; e < 16 * (NM / 2); e += LTH) {
          const int lc = e / (NM / 2), nd = (e % (NM / 2)) * 2, t = lc0 + lc, i = i0 + nd;
          const bool in = t < nl && i < a.nh;
          const size_t at = in ? po + (size_t)t * a.nh + i : 0;
          const int o = ((lc & 1) * 8 + (lc >> 1)) * AP + nd;
          cp_async16(Ps + o, a.Plt + at, in ? 16 : 0);
          if (isD) cp_async16(dPs + o, a.dPlt + at, in ? 16 : 0);
        }
      } else {
        for (int e = tid; e < 16 * NM; e += LTH) {
          const int lc = e / NM, nd = e % NM, t = lc0 + lc, i = i0 + nd;
          const bool in = t < nl && i < a.nh;
          const size_t at = in ? po + (size_t)t * a.nh + i : 0;
          const int o = ((lc & 1) * 8 + (lc >> 1)) * AP + nd;
          cp_async8(Ps + o, a.Plt + at, in ? 8 : 0);
          if (isD) cp_async8(dPs + o, a.dPlt + at, in ? 8 : 0);
        }
      }
#pragma unroll
      for (int e = tid; e < 16 * LNB; e += LTH) {
        const int lc = e & 15, c = e >> 4;
        const long long so = tc.off[c];
        const bool in = so >= 0 && lc0 + lc < nl;
        cp_async8(B + c * BP + (lc & 1) * 8 + (lc >> 1), in ? a.f + so + lc0 + lc : a.f, in ? 8 : 0);
      }
    }
    cp_async_commit();
  };
  double acc[2][MF][2][4];   // [sigma][node tile][column tile]
#pragma unroll
  for (int p = 0; p < 2; p++)
#pragma unroll
    for (int i = 0; i < MF; i++)
#pragma unroll
      for (int j = 0; j < 2; j++)
#pragma unroll
        for (int u = 0; u < 4; u++) acc[p][i][j][u] = 0.0;
  double am[MF][2];          // m / sin(theta) of this thread's fragment rows
#pragma unroll
  for (int i = 0; i < MF; i++)
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int n = i0 + 16 * i + 8 * h + gq;
      am[i][h] = (n < a.nh) ? (double)m * a.asin_t[n] : 0.0;
    }
  const int nb = wc * 16 + gq;                       // column of the first fragment's B value
  const bool vec0 = tc.kind[nb] == 1, vec1 = tc.kind[nb + 8] == 1;
  const bool neg = ((gq & 3) == 1) || ((gq & 3) == 2);   // sign of the m P / sin products of column q
  const int nch = (nl + 15) / 16;
#pragma unroll
  for (int s = 0; s < LST - 1; s++) issue(s);
  for (int ch = 0; ch < nch; ch++) {
    cp_async_wait_stage();
    __syncthreads();
    issue(ch + LST - 1);   // into the stage the last chunk has finished with
    const double *Ps = smb + (ch % LST) * Z::STG, *dPs = Ps + Z::SA, *B = dPs + Z::SA;
    const int lc0 = ch * 16;
#pragma unroll
    for (int p = 0; p < 2; p++)
#pragma unroll
      for (int ks = 0; ks < 2; ks++) {
        if (lc0 + 8 * ks + p >= nl) continue;        // all four degrees beyond the truncation
        const int j = p * 8 + ks * 4 + tq, ao = j * AP + gq;
        double pa[MF][2];
#pragma unroll
        for (int i = 0; i < MF; i++) { pa[i][0] = Ps[ao + 16 * i]; pa[i][1] = Ps[ao + 16 * i + 8]; }
        if (!isD) {
          const int l = m + lc0 + 2 * (ks * 4 + tq) + p;
          const double lf = (l == 0) ? 0.5 : (double)l * (double)(l + 1);
#pragma unroll
          for (int c = 0; c < 2; c++) {
            double b = B[(nb + 8 * c) * BP + j];
            if (c ? vec1 : vec0) b *= lf;
#pragma unroll
            for (int i = 0; i < MF; i++) dmma16n8k4(acc[p][i][c], pa[i][0], pa[i][1], b);
          }
        } else {
          double da[MF][2];
#pragma unroll
          for (int i = 0; i < MF; i++) {
            da[i][0] = dPs[ao + 16 * i]; da[i][1] = dPs[ao + 16 * i + 8];
            pa[i][0] *= am[i][0]; pa[i][1] *= am[i][1];
          }
#pragma unroll
          for (int c = 0; c < 2; c++) {
            const double b = B[(nb + 8 * c) * BP + j];
            double bx = B[((nb ^ 3) + 8 * c) * BP + j];
            bx = neg ? -bx : bx;
#pragma unroll
            for (int i = 0; i < MF; i++) {
              dmma16n8k4(acc[p ^ 1][i][c], da[i][0], da[i][1], b);
              dmma16n8k4(acc[p][i][c], pa[i][0], pa[i][1], bx);
            }
          }
        }
      }
  }
  // fragment rows gq, gq + 8, columns 2 tq, 2 tq + 1 (the orders +m, -m)
  const int ncols = a.nr * (isD ? 4 * a.nvec : 2 * (a.nvec + a.nscal));
  double *base = isD ? a.four.D : a.four.P;
  const size_t st = isD ? a.four.sD() : a.four.sP();
#pragma unroll
  for (int c = 0; c < 2; c++) {
    const int lc = wc * 16 + 8 * c + 2 * tq;
    if (c0 + lc >= ncols) continue;
    const double fac = tc.fac[lc];
    double *out = base + (size_t)m * a.nth * st + c0 + lc;
#pragma unroll
    for (int i = 0; i < MF; i++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int n = i0 + 16 * i + 8 * h + gq;
        if (n >= a.nh) continue;
        const double e0 = acc[0][i][c][2 * h], e1 = acc[0][i][c][2 * h + 1];
        const double o0 = acc[1][i][c][2 * h], o1 = acc[1][i][c][2 * h + 1];
        *reinterpret_cast<double2 *>(out + (size_t)n * st) =
            make_double2((e0 + o0) * fac, m == 0 ? 0.0 : (e1 + o1) * fac);
        *reinterpret_cast<double2 *>(out + (size_t)(a.nth - 1 - n) * st) =
            make_double2((e0 - o0) * fac, m == 0 ? 0.0 : (e1 - o1) * fac);
      }
  }
}

// ---------------------------------------------------------------------------
// Forward: rows 64 degrees (32 of each reflection parity), columns 64, K the
// south nodes in chunks of 8 with their mirrors.  A column's symmetric and
// antisymmetric sums (f(i) +- f(i')) w_i are formed once a lane, in the
// fragment; the rows of parity p take the sums of p ("same") through P and
// the others through dP.  A block's degree tiles run together (x fastest), so
// the Fourier rows come from HBM once.
struct FwdTileSz {
  static constexpr int NC = 8, AP = NC + 4, BP = LNB + 4;
  static constexpr int SA = 64 * AP, SB = 2 * NC * BP, STG = 2 * SA + SB;
  // nh: south nodes whose weights are staged
  static size_t smem(int nh) {
    return LST * (size_t)STG * sizeof(double) + sizeof(LegCols) + (size_t)((nh + NC - 1) / NC * NC) * sizeof(double2);
  }
};

// WSM: the weights of the south nodes sit in shared memory, which has room for
// 10,512 of them; beyond that they are read where they are used.
template <bool WSM>
__global__ void __launch_bounds__(LTH, 3)
k_leg_fwd_f64(const __grid_constant__ LegArgs a) {
  using Z = FwdTileSz;
  constexpr int NC = Z::NC, AP = Z::AP, BP = Z::BP;
  extern __shared__ __align__(16) double smf[];
  LegCols &tc = *reinterpret_cast<LegCols *>(smf + LST * Z::STG);
  double2 *wa = reinterpret_cast<double2 *>(&tc + 1);
  const int m = blockIdx.z, t0 = blockIdx.x * 64, nl = a.L + 1 - m;
  if (t0 >= nl) return;
  const bool isD = (int)blockIdx.y >= a.tilesP;
  const int c0 = ((int)blockIdx.y - (isD ? a.tilesP : 0)) * LNB;
  const int tid = threadIdx.x, lane = tid & 31, wc = tid >> 5, gq = lane >> 2, tq = lane & 3;
  const int ncols = a.nr * (isD ? 4 * a.nvec : 2 * (a.nvec + a.nscal));
  leg_columns(a, m, isD, c0, a.r, tc);
  const int nchk = (a.nh + NC - 1) / NC;
  // (w, m / sin(theta)) of a south node, zero beyond
  auto weight = [&](int i) {
    return (i < a.nh) ? make_double2(a.wgt[i], (double)m * a.asin_t[i]) : make_double2(0.0, 0.0);
  };
  if (WSM)
    for (int i = tid; i < nchk * NC; i += LTH) wa[i] = weight(i);
  const size_t po = a.poff[m], st = isD ? a.four.sD() : a.four.sP();
  const double *rows = (isD ? a.four.D : a.four.P) + (size_t)m * a.nth * st + c0;
  const bool pair16 = (a.nh & 1) == 0;
  auto issue = [&](int ch) {
    const int ib = ch * NC;
    if (ib < a.nh) {
      double *Ps = smf + (ch % LST) * Z::STG, *dPs = Ps + Z::SA, *B = dPs + Z::SA;
      // table rows r = 32 p + j: degree t0 + 2 j + p
      if (pair16) {
#pragma unroll
        for (int e = tid; e < 64 * (NC / 2); e += LTH) {
          const int r = e / (NC / 2), nd = (e % (NC / 2)) * 2, t = t0 + 2 * (r & 31) + (r >> 5), i = ib + nd;
          const bool in = t < nl && i < a.nh;
          const size_t at = in ? po + (size_t)t * a.nh + i : 0;
          cp_async16(Ps + r * AP + nd, a.Plt + at, in ? 16 : 0);
          if (isD) cp_async16(dPs + r * AP + nd, a.dPlt + at, in ? 16 : 0);
        }
      } else {
        for (int e = tid; e < 64 * NC; e += LTH) {
          const int r = e / NC, nd = e % NC, t = t0 + 2 * (r & 31) + (r >> 5), i = ib + nd;
          const bool in = t < nl && i < a.nh;
          const size_t at = in ? po + (size_t)t * a.nh + i : 0;
          cp_async8(Ps + r * AP + nd, a.Plt + at, in ? 8 : 0);
          if (isD) cp_async8(dPs + r * AP + nd, a.dPlt + at, in ? 8 : 0);
        }
      }
      // grid rows [south, mirror][node][column], two columns (+m, -m) a copy
#pragma unroll
      for (int e = tid; e < 2 * NC * (LNB / 2); e += LTH) {
        const int x = (e % (LNB / 2)) * 2, hn = e / (LNB / 2), i = ib + (hn % NC);
        const bool in = i < a.nh && c0 + x < ncols;
        const size_t th = (hn >= NC) ? (size_t)(a.nth - 1 - i) : (size_t)i;
        cp_async16(B + hn * BP + x, in ? rows + th * st + x : a.f, in ? 16 : 0);
      }
    }
    cp_async_commit();
  };
  double acc[2][2][2][4];   // [parity][16-row tile][column tile]
#pragma unroll
  for (int p = 0; p < 2; p++)
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
      for (int j = 0; j < 2; j++)
#pragma unroll
        for (int u = 0; u < 4; u++) acc[p][i][j][u] = 0.0;
  const int nb = wc * 16 + gq;
  const double sg = ((gq & 3) == 0 || (gq & 3) == 3) ? -1.0 : 1.0;   // sign of the m P / sin products of column q
  const bool two = t0 + 32 < nl;                                      // the second row tiles hold a degree
#pragma unroll
  for (int s = 0; s < LST - 1; s++) issue(s);
  for (int ch = 0; ch < nchk; ch++) {
    cp_async_wait_stage();
    __syncthreads();
    issue(ch + LST - 1);
    const double *Ps = smf + (ch % LST) * Z::STG, *dPs = Ps + Z::SA, *B = dPs + Z::SA;
#pragma unroll
    for (int ks = 0; ks < NC / 4; ks++) {
      const int kk = ks * 4 + tq;
      const double2 w = WSM ? wa[ch * NC + kk] : weight(ch * NC + kk);
      double sym[2], ant[2];
#pragma unroll
      for (int c = 0; c < 2; c++) {
        const double f0 = B[kk * BP + nb + 8 * c], f1 = B[(NC + kk) * BP + nb + 8 * c];
        sym[c] = (f0 + f1) * w.x;
        ant[c] = (f0 - f1) * w.x;
      }
      double sx[2], ax[2];
      if (isD) {
        const double ms = w.y * sg;
#pragma unroll
        for (int c = 0; c < 2; c++) {
          sx[c] = __shfl_xor_sync(0xffffffffu, sym[c], 12) * ms;
          ax[c] = __shfl_xor_sync(0xffffffffu, ant[c], 12) * ms;
        }
      }
#pragma unroll
      for (int p = 0; p < 2; p++)
#pragma unroll
        for (int i = 0; i < 2; i++) {
          if (i && !two) continue;
          const int ro = (32 * p + 16 * i + gq) * AP + kk;
          const double pa = Ps[ro], pb = Ps[ro + 8 * AP];
          if (!isD) {
#pragma unroll
            for (int c = 0; c < 2; c++) dmma16n8k4(acc[p][i][c], pa, pb, p ? ant[c] : sym[c]);
          } else {
            const double da = dPs[ro], db = dPs[ro + 8 * AP];
#pragma unroll
            for (int c = 0; c < 2; c++) {
              dmma16n8k4(acc[p][i][c], da, db, p ? sym[c] : ant[c]);
              dmma16n8k4(acc[p][i][c], pa, pb, p ? ax[c] : sx[c]);
            }
          }
        }
    }
  }
  const int j0 = a.moff[m];
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
      for (int p = 0; p < 2; p++) {
        const int t = t0 + 2 * (16 * i + 8 * h + gq) + p;
        if (t >= nl) continue;
        const double g7 = __ldg(a.g7 + j0 + t), g6 = __ldg(a.g6 + j0 + t);
#pragma unroll
        for (int c = 0; c < 2; c++)
#pragma unroll
          for (int s = 0; s < 2; s++) {
            const int lc = wc * 16 + 8 * c + 2 * tq + s;
            const long long so = tc.off[lc];
            if (so >= 0) a.f[so + t] = acc[p][i][c][2 * h + s] * (tc.fac[lc] * (tc.kind[lc] ? g7 : g6));
          }
      }
}

LegArgs leg_args(Ctx &c, const MLayout64 &four, const int *slots) {
  LegArgs a{};
  a.L = c.L; a.nr = c.nr; a.nth = c.nth; a.nh = c.nh; a.jmax = c.jmax;
  a.nvec = four.nvec; a.nscal = four.nscal;
  a.tilesP = cdiv((long)c.nr * four.rpP(), LNB);
  for (int g = 0; g < four.nvec + four.nscal && g < MAXF; g++) a.slot[g] = slots[g];
  a.moff = c.d_moff; a.poff = c.d_poff;
  a.Plt = c.d_Plt; a.dPlt = c.d_dPlt;
  a.asin_t = c.d_asin; a.wgt = c.d_wgt;
  a.g6 = c.d_g6; a.g7 = c.d_g7; a.r = c.d_r; a.ar1 = c.d_ar1;
  a.f = c.d_f; a.fs = c.fsize();
  a.four = four;
  return a;
}

template <int MF>
void launch_bwd(Ctx &c, const LegArgs &a, int tiles) {
  const size_t sm = BwdTileSz<MF>::smem();
  raise_smem_limit(k_leg_bwd_f64<MF>, sm);
  k_leg_bwd_f64<MF><<<dim3(cdiv(c.nh, 16 * MF), tiles, c.L + 1), LTH, sm, c.stream>>>(a);
}

template <bool WSM>
void launch_fwd(Ctx &c, const LegArgs &a, int tiles) {
  const size_t sm = FwdTileSz::smem(WSM ? c.nh : 0);
  raise_smem_limit(k_leg_fwd_f64<WSM>, sm);
  k_leg_fwd_f64<WSM><<<dim3(cdiv(c.L + 1, 64), tiles, c.L + 1), LTH, sm, c.stream>>>(a);
}

}  // namespace

// order-major float64 Fourier rows over a buffer of (L+1) nth nr (6 nvec + 2
// nscal) doubles
MLayout64 mlayout64(const Ctx &c, void *buf, int nvec, int nscal) {
  MLayout64 l;
  l.nvec = nvec; l.nscal = nscal; l.nr = c.nr; l.nth = c.nth;
  l.P = static_cast<double *>(buf);
  l.D = l.P + (size_t)(c.L + 1) * c.nth * l.sP();
  return l;
}

void leg_bwd_f64(Ctx &c, const int *slots, const MLayout64 &out) {
  const LegArgs a = leg_args(c, out, slots);
  const int tiles = a.tilesP + cdiv((long)c.nr * out.rpD(), LNB);
  if (c.nh <= 32) launch_bwd<2>(c, a, tiles);
  else launch_bwd<3>(c, a, tiles);
}

void leg_fwd_f64(Ctx &c, const MLayout64 &in, const int *slots) {
  const LegArgs a = leg_args(c, in, slots);
  const int tiles = a.tilesP + cdiv((long)c.nr * in.rpD(), LNB);
  if (FwdTileSz::smem(c.nh) <= 227 * 1024) launch_fwd<true>(c, a, tiles);
  else launch_fwd<false>(c, a, tiles);
}

}  // namespace cb2
