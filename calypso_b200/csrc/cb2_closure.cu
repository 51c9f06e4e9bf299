// cb2_closure.cu -- learned spectral subgrid closure (no counterpart in the
// reference: its SGS hooks, MHD_src/sph_MHD/cal_explicit_terms.f90:70-95,
// have no call sites on the spherical-shell path).
//
// A low-resolution shell (truncation L_lo) misses the part of its nonlinear
// terms that comes from the modes it does not carry.  The closure predicts
// that part per radial level and per (l, m) from local spectral features:
//   tau(k, l, m) = P_lo[N(u_hi)](k, l, m) - N_lo(P_lo u_hi)(k, l, m)
// for the five explicit nonlinear terms of the evolved equations (curl of
// the forces S and T, induction S and T, heat advection).  P_lo truncates
// to l <= L_lo and restricts to the low-resolution radial points (which must
// be a subset of the high-resolution Chebyshev points).
//
// Network: MLP nin -> nhid -> nhid -> nout, SiLU activations, weights kept
// in bfloat16 for every product (float32 master copy for the optimiser),
// float32 activations and accumulation.  Kernels: for the widths of fused_ok
// one each for the forward pass, the data gradients and the weight gradients;
// for others a tiled GEMM with either operand transposed (split-K with float32
// atomics for the weight gradients), bias + activation, its derivative and
// column sums; and Adam.
// Training runs on the GPU through these kernels; the oracle restates the
// same forward and backward in float64 (numpy) to check the gradients.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <vector>

#include "cb2_internal.cuh"
#include "cb2_tc.cuh"

namespace cb2 {
namespace {

constexpr int NF = 16;   // features per (k, l, m)
constexpr int NO = 5;    // predicted tendencies

struct Slots16 {
  int s[16];
};

// field slots read as features and the slots the closure adds to
Slots16 feat_slots() {
  return Slots16{{VELO, VELO + 1, VELO + 2, VORT, VORT + 1, VORT + 2, MAGNE, MAGNE + 1, MAGNE + 2, CURRENT,
                  CURRENT + 1, CURRENT + 2, TEMP, 0, 0, 0}};
}
Slots16 out_slots() { return Slots16{{FORCES, FORCES + 2, INDUCT, INDUCT + 2, HADV, 0}}; }

// ---------------------------------------------------------------------------
// filtering between shells: dst(k, l, m) = src(k * stride, l, m), l <= L_dst
__global__ void k_filter(int nr_dst, int jmax_dst, int jmax_src, int Lsrc, int stride, const int *jl, const int *jm,
                         const int *moff_src, const double *src, size_t fs_src, double *dst, size_t fs_dst,
                         Slots16 ss, Slots16 sd, int nslots, int to_buffer) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (size_t)nr_dst * jmax_dst) return;
  const int k = (int)(i / jmax_dst), jj = (int)(i - (size_t)k * jmax_dst);
  const int l = jl[jj], m = jm[jj], am = m < 0 ? -m : m;
  const int jjs = moff_src[am] + (m < 0 ? (Lsrc + 1 - am) : 0) + (l - am);
  const size_t at_s = (size_t)(k * stride) * jmax_src + jjs;
  for (int q = 0; q < nslots; q++) {
    const double v = src[(size_t)ss.s[q] * fs_src + at_s];
    if (to_buffer) dst[(size_t)q * fs_dst + i] = v;
    else dst[(size_t)sd.s[q] * fs_dst + i] = v;
  }
}

// features X[row][16], row = k * jmax + jj: the 13 evolved / derived field
// coefficients, l / L, m / L (negative for the sin part), r mapped to [-1, 1]
__global__ void k_features(int nr, int jmax, int L, const int *jl, const int *jm, const double *r, double ri,
                           double ro, const double *f, size_t fs, Slots16 fsl, float *X) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (size_t)nr * jmax) return;
  const int k = (int)(i / jmax), jj = (int)(i - (size_t)k * jmax);
  float *x = X + i * NF;
#pragma unroll
  for (int q = 0; q < 13; q++) x[q] = (float)f[(size_t)fsl.s[q] * fs + i];
  x[13] = (float)jl[jj] / (float)L;
  x[14] = (float)jm[jj] / (float)L;
  x[15] = (float)((2.0 * r[k] - (ri + ro)) / (ro - ri));
}

// normalised features: (x - mean[k]) / std[k] per radial level k
__global__ void k_normalise(size_t n, int jmax, const float *X, const float *mean, const float *istd, float *Xn) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n * NF) return;
  const size_t row = i / NF;
  const int q = (int)(i - row * NF), k = (int)(row / jmax);
  Xn[i] = (X[i] - mean[k * NF + q]) * istd[k * NF + q];
}

// targets Y[row][5] = hi[c][row] - lo slot c (row)
__global__ void k_targets(size_t n, const double *hi, const double *f, size_t fs, Slots16 osl, float *Y) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
#pragma unroll
  for (int c = 0; c < NO; c++) Y[i * NO + c] = (float)(hi[(size_t)c * n + i] - f[(size_t)osl.s[c] * fs + i]);
}

// slot c (row) += Y[row][c] * scale[k][c] at the interior radial levels
// (the wall levels are set by the boundary conditions and left alone)
__global__ void k_add_tendency(size_t n, int nr, int jmax, const float *Y, const float *scale, double *f, size_t fs,
                               Slots16 osl) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int k = (int)(i / jmax);
  if (k == 0 || k == nr - 1) return;
#pragma unroll
  for (int c = 0; c < NO; c++) f[(size_t)osl.s[c] * fs + i] += (double)(Y[i * NO + c] * scale[k * NO + c]);
}

// ---------------------------------------------------------------------------
// GEMM on the tensor cores: C[M][N] (+)= sum_k opA[m][k] opB[k][n];
//   opA[m][k] = TA ? A[k * lda + m] : A[m * lda + k]
//   opB[k][n] = TB ? B[n * ldb + k] : B[k * ldb + n]
// One CTA (128 threads) per tile of 128 rows x NT <= 256 columns and per
// chunk of K (blockIdx.z, partial sums added with float32 atomics when
// `atomic`).  K runs in blocks of 32: the threads load both operand tiles,
// split float32 values into bfloat16 hi + lo (x = hi + lo to 16 bits;
// bfloat16 weights are one exact term) and write them K-major, 64-byte
// swizzled, into one of two shared-memory stages; one thread issues
// tcgen05.mma kind::f16 with bf16 operands (hi*hi', hi*lo', lo*hi': the
// products that reach 2^-16 of the result) into a float32 TMEM accumulator
// and commits to the stage's mbarrier, which the loads of the stage after
// next wait on.  Every wait is bounded; a wait that runs out sets bit 2 of
// *status and the CTA drains its MMAs, frees its TMEM and returns.
constexpr int GK = 32;                        // K per stage (64-byte rows)
constexpr uint32_t GA_BYTES = 128 * GK * 2;   // one bf16 term of the A tile

template <typename T> struct Terms { static constexpr int n = 2; };
template <> struct Terms<__nv_bfloat16> { static constexpr int n = 1; };

__device__ inline float to_f(float x) { return x; }
__device__ inline float to_f(__nv_bfloat16 x) { return __bfloat162float(x); }

// 8 consecutive K values of one row -> nt bf16 terms, 16 bytes each
template <int NT_>
__device__ inline void put_row8(unsigned char *tile, uint32_t term_bytes, int row, int chunk, const float v[8]) {
  uint32_t hi[4], lo[4];
#pragma unroll
  for (int e = 0; e < 8; e += 2) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(v[e], v[e + 1]);
    const float2 f = __bfloat1622float2(h);
    const __nv_bfloat162 l = __floats2bfloat162_rn(v[e] - f.x, v[e + 1] - f.y);
    hi[e >> 1] = *reinterpret_cast<const uint32_t *>(&h);
    lo[e >> 1] = *reinterpret_cast<const uint32_t *>(&l);
  }
  const uint32_t off = tc::sw64_chunk(row, chunk);
  *reinterpret_cast<uint4 *>(tile + off) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
  if (NT_ > 1) *reinterpret_cast<uint4 *>(tile + term_bytes + off) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
}

template <typename TAT, typename TBT, bool TA, bool TB>
__global__ void __launch_bounds__(128)
k_tc_gemm(int M, int N, int NT, int K, const TAT *__restrict__ A, int lda, const TBT *__restrict__ B, int ldb,
          float *C, int ldc, int kchunk, int atomic, uint32_t tmem_cols, int *status, unsigned long long wait_ns) {
  constexpr int NA = Terms<TAT>::n, NBT = Terms<TBT>::n;
  extern __shared__ unsigned char g_smem_raw[];
  unsigned char *base = tc::smem_base_1024(g_smem_raw);
  const uint32_t b_bytes = (uint32_t)NT * GK * 2;               // one bf16 term of the B tile
  const uint32_t stage_bytes = ((NA * GA_BYTES + NBT * b_bytes) + 1023u) & ~1023u;
  uint64_t *bar = reinterpret_cast<uint64_t *>(base + 2 * stage_bytes);   // [2] stage done, [2] final
  uint32_t *tslot = reinterpret_cast<uint32_t *>(bar + 3);
  int *abort = reinterpret_cast<int *>(tslot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.y * 128, n0 = blockIdx.x * NT;
  const int kb = blockIdx.z * kchunk, ke = min(K, kb + kchunk);
  if (tid == 0) {
    tc::mbar_init(&bar[0], 1); tc::mbar_init(&bar[1], 1); tc::mbar_init(&bar[2], 1);
    *abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tc::tmem_alloc(tslot, tmem_cols);
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = *tslot;
  const uint32_t idesc = tc::idesc_bf16_f32(128, NT);
  const int nblk = (ke - kb + GK - 1) / GK;
  bool bad = false;
  for (int ib = 0; ib < nblk; ib++) {
    const int st = ib & 1, k0 = kb + ib * GK;
    unsigned char *ta = base + st * stage_bytes, *tbp = ta + NA * GA_BYTES;
    // the stage's previous MMAs (block ib - 2) must have read it
    if (ib >= 2 && !tc::mbar_wait(&bar[st], ((ib - 2) >> 1) & 1, wait_ns)) bad = true;
    if (__syncthreads_or(bad)) { bad = true; break; }
    // A tile: thread = row
    {
      const int m = m0 + tid;
#pragma unroll
      for (int c = 0; c < GK / 8; c++) {
        float v[8];
#pragma unroll
        for (int e = 0; e < 8; e++) {
          const int k = k0 + c * 8 + e;
          v[e] = (m < M && k < ke) ? to_f(TA ? A[(size_t)k * lda + m] : A[(size_t)m * lda + k]) : 0.0f;
        }
        put_row8<NA>(ta, GA_BYTES, tid, c, v);
      }
    }
    // B tile: rows n of the column tile
    for (int r = tid; r < NT; r += 128) {
      const int n = n0 + r;
#pragma unroll
      for (int c = 0; c < GK / 8; c++) {
        float v[8];
#pragma unroll
        for (int e = 0; e < 8; e++) {
          const int k = k0 + c * 8 + e;
          v[e] = (n < N && k < ke) ? to_f(TB ? B[(size_t)n * ldb + k] : B[(size_t)k * ldb + n]) : 0.0f;
        }
        put_row8<NBT>(tbp, b_bytes, r, c, v);
      }
    }
    tc::fence_proxy_async();
    __syncthreads();
    if (tid == 0) {
      tc::tc_fence_after();
#pragma unroll
      for (int ks = 0; ks < GK / 16; ks++) {
        const uint64_t o = (uint64_t)(ks * 2);
        const uint64_t ah = tc::smem_desc_sw64(ta) + o, bh = tc::smem_desc_sw64(tbp) + o;
        tc::mma_f16(tmem, ah, bh, idesc, (ib == 0 && ks == 0) ? 0u : 1u);
        if (NBT > 1) tc::mma_f16(tmem, ah, tc::smem_desc_sw64(tbp + b_bytes) + o, idesc, 1u);
        if (NA > 1) tc::mma_f16(tmem, tc::smem_desc_sw64(ta + GA_BYTES) + o, bh, idesc, 1u);
      }
      tc::mma_commit(&bar[st]);
    }
  }
  // every MMA has completed before the accumulator is read and freed
  if (tid == 0) {
    if (nblk > 0) tc::mma_commit(&bar[2]);
  }
  __syncthreads();
  const bool done = nblk == 0 || tc::mbar_wait(&bar[2], 0, tc::kWaitNs);
  if (!done || bad) {
    if (tid == 0) atomicOr(status, CB2_STATUS_PIPE_TIMEOUT);
    *abort = 1;
  }
  __syncthreads();
  tc::tc_fence_after();
  if (!*abort && nblk > 0) {
    // epilogue: warp w holds TMEM lanes 32 w .. 32 w + 31 (tile rows), a
    // thread 64 columns of its row per load; through the warp's 32 x 65
    // staging (the stage buffers are free now) a store then writes 32
    // consecutive columns of one row
    float *stg = reinterpret_cast<float *>(base) + warp * 32 * 65;
    for (int c0 = 0; c0 < NT; c0 += 64) {
      float va[32], vb[32];
      const uint32_t ta = tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0;
      tc::tmem_ld32x2(ta, ta + 32, va, vb);
#pragma unroll
      for (int j = 0; j < 32; j++) { stg[lane * 65 + j] = va[j]; stg[lane * 65 + 32 + j] = vb[j]; }
      __syncwarp();
      for (int r = 0; r < 32; r++) {
        const int m = m0 + warp * 32 + r;
        if (m >= M) break;
#pragma unroll
        for (int hh = 0; hh < 2; hh++) {
          const int cc = c0 + 32 * hh + lane, n = n0 + cc;
          if (cc < NT && n < N) {
            float *cp = C + (size_t)m * ldc + n;
            const float v = stg[r * 65 + 32 * hh + lane];
            if (atomic) atomicAdd(cp, v); else *cp = v;
          }
        }
      }
      __syncwarp();
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, tmem_cols);
}

// ---------------------------------------------------------------------------
// The network in one kernel a pass (k_mlp_fwd), its data gradient in one
// (k_mlp_bwd) and every weight and bias gradient in one (k_mlp_wgrad), for
// the sizes of fused_ok: F <= 32 inputs, H a multiple of 32 up to 256, O <= 8.
// Three GEMMs with the activations between them in memory moved 1.6 GB for
// 266240 rows (2031 us: the GEMMs, whose threads read a row each, 1510, bias
// and SiLU 505); kept in tensor and shared memory the pass reads 64 and
// writes 20 bytes a row and takes 187 us, bound by the SiLU epilogue (an
// __expf and a reciprocal per unit and layer) and the operand split.  A
// training pass of 16384 rows: 29 + 39 + 52 + 3 us of kernels, before 500 us.
//
// A training pass forms every product and activation with the terms, the order
// and the rounding of the general kernels (k_tc_gemm, k_bias_act, k_mse,
// k_act_grad), so its loss and gradients do not depend on which of the two a
// network's widths select: they are equal bit for bit but for the order of the
// float32 atomics that add the weight gradients' row chunks and of the float64
// sums of the bias gradients.  That matters
// because an optimiser carries a difference on: an Adam step is +- lr where a
// gradient is far above eps, whatever its size, and one weight that rounds the
// other way to bfloat16 moves the next gradient by 1e-5.
//
// A CTA keeps the bfloat16 weights in shared memory and walks tiles of 128
// rows.  Warps 0-11 are the epilogue: warp w reads tensor-memory lanes
// 32 (w & 3) .. + 31, one row a thread, the four warps of group w >> 2 every
// third chunk of 32 columns (with two groups the SiLU chains leave the
// schedulers idle: a ninth longer at 266240 rows).  A chunk of an activation is
// split into bfloat16 hi + lo and written as the next product's A operand
// into one of ML_ST stages; the last warp issues the MMAs of a chunk as soon as
// it is there, so the second product runs behind the first one's epilogue.  The
// last layer (OC = 5 or 8 columns) is float32 FMAs on the thread's row; in
// training it is a third product over the same stages, whose 16 columns of sums
// take the place of the first layer's.
//
// The stages' empty barriers are waited on by phase parity, so whoever fills
// use q of a stage must know that use q - 2 ML_ST has been released.  Within a
// layer a group fills every ML_G-th use and has seen its own last use's
// predecessor released, q - ML_G - ML_ST: hence ML_G <= ML_ST.  The first uses
// of a layer follow a wait for the accumulator before them (d1, d2, d3), which
// the MMA thread commits once use q - ML_ST has been filled, and whoever filled
// that one had seen use q - 2 ML_ST released; a next tile's input that goes in
// front of the last epilogue follows its group's last chunk.
constexpr int ML_G = 3, ML_EPI = 128 * ML_G, ML_THREADS = ML_EPI + 32, ML_ST = 3, ML_O = 8;
static_assert(ML_G <= ML_ST, "a group may not run two phases ahead of a stage");
constexpr uint32_t ML_STAGE = 2 * GA_BYTES;   // hi and lo of 128 rows x 32 columns
constexpr uint32_t W3_TILE = 16 * 64;          // 16 outputs x 32 units of W3
static_assert(W3_TILE == 32 * ML_O * 4, "the tile takes the place of the float weights");

struct MlpArgs {
  long long n;
  int F, H, O, vec;              // vec: rows of X can be read 16 bytes at a time
  const float *X, *b1, *b2, *b3;
  const __nv_bfloat16 *W1, *W2, *W3;
  float *Y;                      // forward output, n x O
  // training: targets, n O, pre-activations, dL/dY, loss partial sums (4 a
  // tile), and the data gradients of the hidden layers
  const float *T;
  float count;
  float *Z1, *Z2, *dY, *dZ2, *dZ1;
  double *part;
  int *status;
  unsigned long long wait_ns;
};

struct MlpBars {
  uint64_t full[ML_ST], empty[ML_ST], d1, d2, d3, fin;
  uint32_t tmem;
  int abort;
};

struct MlpLayout {
  uint32_t w2, w1, st, w3, b1, b2, yp, bar, total;
};
__host__ __device__ inline MlpLayout mlp_layout(int H) {
  MlpLayout o;
  uint32_t p = 0;
  o.w2 = p; p += (uint32_t)H * H * 2;
  o.w1 = p; p += (uint32_t)H * 64;
  o.st = p; p += ML_ST * ML_STAGE;
  o.w3 = p; p += (uint32_t)H * ML_O * 4;   // float [H][ML_O], or the bfloat16 tile of 16 outputs (W3_TILE a chunk)
  o.b1 = p; p += (uint32_t)H * 4;
  o.b2 = p; p += (uint32_t)H * 4;
  o.yp = p; p += (ML_G - 1) * 128 * ML_O * 4;
  o.bar = p; p += 128;
  o.total = p;
  return o;
}

// The sigmoid with an IEEE division.  The fused passes take it apart: for
// z >= kSigmLow the divisor lies in [1, 2^126), where one step of Newton's
// iteration from the approximate reciprocal rounds as 1.0f / x does (compared
// for every float of that range), without the division's range check a value,
// which kept the 32 chains of a thread apart (closure forward of 266240 rows:
// 333 us with 1.0f / x, 196 so, 187 two values a time).
__device__ inline float sigm(float z) { return 1.0f / (1.0f + __expf(-z)); }
constexpr float kSigmLow = -87.0f;
// two values a time: the packed operations round each as the scalar ones
__device__ inline float2 sigm_mid(float2 z) {
  const float2 x = __fadd2_rn(float2{1.0f, 1.0f}, float2{__expf(-z.x), __expf(-z.y)});
  float2 y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y.x) : "f"(x.x));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y.y) : "f"(x.y));
  return __ffma2_rn(y, __ffma2_rn(float2{-x.x, -x.y}, y, float2{1.0f, 1.0f}), y);
}
template <int N>
__device__ inline bool all_mid(const float *z) {
  float lo = z[0];
#pragma unroll
  for (int j = 1; j < N; j++) lo = fminf(lo, z[j]);
  return !(lo < kSigmLow);
}
// z = SiLU(z), and d = d SiLU'(z), of N values, rounded as in k_bias_act and
// k_act_grad
template <int N>
__device__ inline void silu(float *z) {
  if (all_mid<N>(z)) {
#pragma unroll
    for (int j = 0; j < N; j += 2) {
      const float2 v{z[j], z[j + 1]}, h = __fmul2_rn(v, sigm_mid(v));
      z[j] = h.x;
      z[j + 1] = h.y;
    }
  } else {
#pragma unroll
    for (int j = 0; j < N; j++) z[j] = __fmul_rn(z[j], sigm(z[j]));
  }
}
__device__ inline float act_grad(float d, float z, float s) {
  return __fmul_rn(__fmul_rn(d, s), __fmaf_rn(z, 1.0f - s, 1.0f));
}
template <int N>
__device__ inline void act_grad(float *d, const float *z) {
  if (all_mid<N>(z)) {
#pragma unroll
    for (int j = 0; j < N; j += 2) {
      const float2 s = sigm_mid(float2{z[j], z[j + 1]});
      d[j] = act_grad(d[j], z[j], s.x);
      d[j + 1] = act_grad(d[j + 1], z[j + 1], s.y);
    }
  } else {
#pragma unroll
    for (int j = 0; j < N; j++) d[j] = act_grad(d[j], z[j], sigm(z[j]));
  }
}

// barrier of the epilogue threads; true when any of them passes true
__device__ inline bool epi_any(bool v) {
  int r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.s32 p, %1, 0;\n\t"
      "barrier.cta.red.or.pred q, 1, %2, p;\n\t"
      "selp.s32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"((int)v), "n"(ML_EPI)
      : "memory");
  return r != 0;
}

__device__ inline void tmem_ld32(uint32_t ta, float v[32]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(ta)
      : "memory");
#pragma unroll
  for (int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]);
}

// 32 columns of one row into a stage, hi at 0 and lo at GA_BYTES
__device__ inline void put_chunk(unsigned char *stage, int row, const float v[32]) {
#pragma unroll
  for (int c = 0; c < 4; c++) put_row8<2>(stage, GA_BYTES, row, c, v + 8 * c);
}

__device__ inline void store32(float *dst, const float v[32]) {
#pragma unroll
  for (int j = 0; j < 32; j += 4) *reinterpret_cast<float4 *>(dst + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
}
// d *= SiLU'(z) for 32 columns of a row, kept and stored
__device__ inline void act_grad32(float d[32], const float *z, float *dst) {
#pragma unroll
  for (int j = 0; j < 32; j += 8) {
    const float4 x = __ldg(reinterpret_cast<const float4 *>(z + j));
    const float4 y = __ldg(reinterpret_cast<const float4 *>(z + j + 4));
    const float v[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
    act_grad<8>(d + j, v);
  }
  store32(dst, d);
}

// one thread: acc (+)= (hi + lo) of `stage` times the bfloat16 tile `b`, ks
// steps of 16 columns
__device__ inline void mma_chunk(uint32_t acc, const unsigned char *stage, const unsigned char *b, uint32_t idesc, int ks,
                                 bool first) {
  const uint64_t ah = tc::smem_desc_sw64(stage), al = tc::smem_desc_sw64(stage + GA_BYTES), bd = tc::smem_desc_sw64(b);
  for (int q = 0; q < ks; q++) {
    const uint64_t o = (uint64_t)(q * 2);
    tc::mma_f16(acc, ah + o, bd + o, idesc, (first && q == 0) ? 0u : 1u);
    tc::mma_f16(acc, al + o, bd + o, idesc, 1u);
  }
}

// shared set-up of the two row kernels: barriers and, for the forward pass,
// the biases and the last layer's weights (as floats, or as tiles of 16 outputs
// x 32 units)
enum MlpPass { ML_FORWARD, ML_TRAIN, ML_BACKWARD };
template <MlpPass PASS>
__device__ inline void mlp_setup(const MlpArgs &a, unsigned char *base, const MlpLayout &lay, MlpBars *sb) {
  const int tid = threadIdx.x;
  if (tid == 0) {
    for (int q = 0; q < ML_ST; q++) { tc::mbar_init(&sb->full[q], 4); tc::mbar_init(&sb->empty[q], 1); }
    tc::mbar_init(&sb->d1, 1); tc::mbar_init(&sb->d2, 1); tc::mbar_init(&sb->d3, 1); tc::mbar_init(&sb->fin, 1);
    sb->abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if constexpr (PASS == ML_BACKWARD) return;
  float *b1 = reinterpret_cast<float *>(base + lay.b1), *b2 = reinterpret_cast<float *>(base + lay.b2);
  for (int c = tid; c < a.H; c += ML_THREADS) {
    b1[c] = a.b1[c];
    b2[c] = a.b2[c];
  }
  if constexpr (PASS == ML_TRAIN) {
    for (int e = tid; e < 16 * (a.H / 8); e += ML_THREADS) {
      const int o = e & 15, c8 = e >> 4;   // 8 units from 8 c8
      __nv_bfloat16 v[8];
#pragma unroll
      for (int u = 0; u < 8; u++) v[u] = (o < a.O) ? a.W3[(size_t)o * a.H + c8 * 8 + u] : __float2bfloat16_rn(0.0f);
      *reinterpret_cast<uint4 *>(base + lay.w3 + (c8 >> 2) * W3_TILE + tc::sw64_chunk(o, c8 & 3)) =
          *reinterpret_cast<const uint4 *>(v);
    }
  } else {
    float *w3 = reinterpret_cast<float *>(base + lay.w3);
    for (int c = tid; c < a.H; c += ML_THREADS)
#pragma unroll
      for (int o = 0; o < ML_O; o++) w3[c * ML_O + o] = (o < a.O) ? __bfloat162float(a.W3[(size_t)o * a.H + c]) : 0.0f;
  }
}

// releases tensor memory once every MMA has completed; a wait that ran out
// is reported in *status
__device__ inline void mlp_finish(const MlpArgs &a, MlpBars *sb, uint32_t tmem, bool bad) {
  if (bad) sb->abort = 1;
  tc::tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && sb->abort) atomicOr(a.status, CB2_STATUS_PIPE_TIMEOUT);
  if (threadIdx.x >> 5 == 0) tc::tmem_dealloc(tmem, 512);
}

template <bool TRAIN, int OC>
__global__ void __launch_bounds__(ML_THREADS, 1)
k_mlp_fwd(const __grid_constant__ MlpArgs a) {
  extern __shared__ unsigned char g_smem_raw[];
  unsigned char *base = tc::smem_base_1024(g_smem_raw);
  const MlpLayout lay = mlp_layout(a.H);
  MlpBars *sb = reinterpret_cast<MlpBars *>(base + lay.bar);
  unsigned char *W2s = base + lay.w2, *W1s = base + lay.w1, *st0 = base + lay.st;
  const float *b1 = reinterpret_cast<float *>(base + lay.b1), *b2 = reinterpret_cast<float *>(base + lay.b2);
  const float *w3 = reinterpret_cast<float *>(base + lay.w3);
  float *yp = reinterpret_cast<float *>(base + lay.yp);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, H = a.H, nch = H / 32;
  const int seq = TRAIN ? 2 * nch + 1 : nch + 1;   // stage uses of a tile
  mlp_setup<TRAIN ? ML_TRAIN : ML_FORWARD>(a, base, lay, sb);
  if (warp == 0) tc::tmem_alloc(&sb->tmem, 512);
  // W1 [n = unit][k = input] as one chunk, W2 [n][k] as H / 32 chunks
  for (int e = tid; e < H * 4; e += ML_THREADS) {
    const int r = e >> 2, c = e & 3;
    __nv_bfloat16 v[8];
#pragma unroll
    for (int u = 0; u < 8; u++) v[u] = (c * 8 + u < a.F) ? a.W1[(size_t)r * a.F + c * 8 + u] : __float2bfloat16_rn(0.0f);
    *reinterpret_cast<uint4 *>(W1s + tc::sw64_chunk(r, c)) = *reinterpret_cast<const uint4 *>(v);
  }
  for (int e = tid; e < H * (H / 8); e += ML_THREADS) {
    const int r = e / (H / 8), c8 = e - r * (H / 8);
    *reinterpret_cast<uint4 *>(W2s + (size_t)(c8 >> 2) * H * 64 + tc::sw64_chunk(r, c8 & 3)) =
        *reinterpret_cast<const uint4 *>(a.W2 + (size_t)r * H + c8 * 8);
  }
  tc::fence_proxy_async();
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = sb->tmem;
  const long long ntile = (a.n + 127) / 128;
  bool bad = false;
  if (warp == ML_EPI / 32) {
    if (lane == 0) {
      const uint32_t idesc = tc::idesc_bf16_f32(128, H), idesc3 = tc::idesc_bf16_f32(128, 16);
      uint32_t q = 0;
      for (long long t = blockIdx.x; t < ntile && !bad; t += gridDim.x)
        for (int c = -1; c < seq - 1; c++, q++) {   // c = -1: the input rows; from nch on: the last layer
          const uint32_t s = q % ML_ST;
          if (!tc::mbar_wait(&sb->full[s], (q / ML_ST) & 1, a.wait_ns)) { bad = true; break; }
          tc::tc_fence_after();
          unsigned char *st = st0 + s * ML_STAGE;
          if (c < 0) mma_chunk(tmem, st, W1s, idesc, (a.F + 15) / 16, true);
          else if (c < nch) mma_chunk(tmem + 256, st, W2s + (size_t)c * H * 64, idesc, 2, c == 0);
          else mma_chunk(tmem, st, base + lay.w3 + (c - nch) * W3_TILE, idesc3, 2, c == nch);
          tc::mma_commit(&sb->empty[s]);
          if (c < 0) tc::mma_commit(&sb->d1);
          else if (c == nch - 1) tc::mma_commit(&sb->d2);
          else if (TRAIN && c == seq - 2) tc::mma_commit(&sb->d3);
        }
      tc::mma_commit(&sb->fin);
      if (!tc::mbar_wait(&sb->fin, 0)) bad = true;
    }
  } else {
    const int qd = warp & 3, g = warp >> 2, r = qd * 32 + lane;
    const uint32_t tl = tmem + ((uint32_t)(qd * 32) << 16);
    // stage of sequence number q, once its last MMAs have read it
    auto stage = [&](uint32_t q) {
      if (q >= ML_ST && !bad && !tc::mbar_wait(&sb->empty[q % ML_ST], ((q / ML_ST) - 1) & 1, a.wait_ns)) bad = true;
      bad = __any_sync(0xffffffffu, bad);
      return st0 + (q % ML_ST) * ML_STAGE;
    };
    auto publish = [&](uint32_t q) {
      tc::fence_proxy_async();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&sb->full[q % ML_ST]);
    };
    auto put_input = [&](long long t, uint32_t q) {
      const long long row = t * 128 + r;
      float x[32];
#pragma unroll
      for (int j = 0; j < 32; j += 4) {
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (row < a.n && j < a.F) {
          const float *p = a.X + row * a.F + j;
          if (a.vec) v = __ldg(reinterpret_cast<const float4 *>(p));
          else v = make_float4(p[0], j + 1 < a.F ? p[1] : 0.0f, j + 2 < a.F ? p[2] : 0.0f, j + 3 < a.F ? p[3] : 0.0f);
        }
        x[j] = v.x; x[j + 1] = v.y; x[j + 2] = v.z; x[j + 3] = v.w;
      }
      unsigned char *s = stage(q);
      if (!bad) put_chunk(s, r, x);
      publish(q);
    };
    uint32_t q0 = 0;
    if (g == 0) put_input(blockIdx.x, 0);
    int i = 0;
    for (long long t = blockIdx.x; t < ntile; t += gridDim.x, i++, q0 += seq) {
      const long long row = t * 128 + r;
      const bool in = row < a.n;
      if (!bad && !tc::mbar_wait(&sb->d1, i & 1, a.wait_ns)) bad = true;
      bad = __any_sync(0xffffffffu, bad);
      tc::tc_fence_after();
      for (int c = g; c < nch; c += ML_G) {
        float z[32];
        tmem_ld32(tl + c * 32, z);
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
          const float4 bv = *reinterpret_cast<const float4 *>(b1 + c * 32 + j);
          z[j] += bv.x; z[j + 1] += bv.y; z[j + 2] += bv.z; z[j + 3] += bv.w;
        }
        if (TRAIN && in) store32(a.Z1 + row * H + c * 32, z);
        silu<32>(z);
        unsigned char *s = stage(q0 + 1 + c);
        if (!bad) put_chunk(s, r, z);
        tc::tc_fence_before();
        publish(q0 + 1 + c);
      }
      // the next tile's input goes in front of this tile's last epilogue (in
      // training its product would overwrite the last layer's sums: after them)
      if (!TRAIN && g == 0 && t + gridDim.x < ntile) put_input(t + gridDim.x, q0 + seq);
      if (!bad && !tc::mbar_wait(&sb->d2, i & 1, a.wait_ns)) bad = true;
      bad = __any_sync(0xffffffffu, bad);
      tc::tc_fence_after();
      float y[OC];
#pragma unroll
      for (int o = 0; o < OC; o++) y[o] = 0.0f;
      for (int c = g; c < nch; c += ML_G) {
        float z[32];
        tmem_ld32(tl + 256 + c * 32, z);
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
          const float4 bv = *reinterpret_cast<const float4 *>(b2 + c * 32 + j);
          z[j] += bv.x; z[j + 1] += bv.y; z[j + 2] += bv.z; z[j + 3] += bv.w;
        }
        if (TRAIN && in) store32(a.Z2 + row * H + c * 32, z);
        silu<32>(z);
        if constexpr (TRAIN) {
          unsigned char *s = stage(q0 + 1 + nch + c);
          if (!bad) put_chunk(s, r, z);
          tc::tc_fence_before();
          publish(q0 + 1 + nch + c);
        } else {
#pragma unroll
          for (int j = 0; j < 32; j++) {
            const float h = z[j];
            const float4 wa = *reinterpret_cast<const float4 *>(w3 + (c * 32 + j) * ML_O);
            y[0] += h * wa.x; y[1] += h * wa.y; y[2] += h * wa.z; y[3] += h * wa.w;
            if constexpr (OC == 5) {
              y[4] += h * w3[(c * 32 + j) * ML_O + 4];
            } else {
              const float4 wb = *reinterpret_cast<const float4 *>(w3 + (c * 32 + j) * ML_O + 4);
              y[4] += h * wb.x; y[5] += h * wb.y; y[6] += h * wb.z; y[7] += h * wb.w;
            }
          }
        }
      }
      if (!TRAIN && g > 0) {
#pragma unroll
        for (int o = 0; o < OC; o++) yp[((g - 1) * 128 + r) * ML_O + o] = y[o];
      }
      if (TRAIN && g == 0) {   // the sums of the last layer, over the first one's
        if (!bad && !tc::mbar_wait(&sb->d3, i & 1, a.wait_ns)) bad = true;
        bad = __any_sync(0xffffffffu, bad);
        tc::tc_fence_after();
        float z[32];
        tmem_ld32(tl, z);
#pragma unroll
        for (int o = 0; o < OC; o++) y[o] = z[o];
        tc::tc_fence_before();
        if (t + gridDim.x < ntile) put_input(t + gridDim.x, q0 + seq);
      }
      // every group has read the accumulators: the next tile may refill them
      tc::tc_fence_before();
      bad = epi_any(bad);
      if (bad) break;
      if (g == 0) {
        double e = 0.0;
#pragma unroll
        for (int o = 0; o < OC; o++)
          if (in && o < a.O) {
            float v = y[o];
            if (!TRAIN) {
#pragma unroll
              for (int u = 0; u < ML_G - 1; u++) v += yp[(u * 128 + r) * ML_O + o];
              a.Y[row * a.O + o] = v + a.b3[o];
            } else {
              const float d = v + a.b3[o] - a.T[row * a.O + o];
              a.dY[row * a.O + o] = 2.0f * d / a.count;
              e += (double)d * (double)d;
            }
          }
        if (TRAIN) {
          for (int u = 16; u > 0; u >>= 1) e += __shfl_xor_sync(0xffffffffu, e, u);
          if (lane == 0) a.part[t * 4 + qd] = e;
        }
      }
    }
  }
  mlp_finish(a, sb, tmem, bad);
}

// Data gradients of the hidden layers: dH2 = dY W3, dZ2 = dH2 SiLU'(Z2),
// written out and, a chunk of 32 columns at a time, the A operand of
// dH1 = dZ2 W2; then dZ1 = dH1 SiLU'(Z1).  The CTA holds W2 and W3 transposed
// ([n = input unit][k = output unit], K of W3 padded to 16); dY goes through a
// stage as the input rows of k_mlp_fwd do.  The same roles and hand-overs as
// there, dH2 in the first half of tensor memory and dH1 in the second.
__global__ void __launch_bounds__(ML_THREADS, 1)
k_mlp_bwd(const __grid_constant__ MlpArgs a) {
  extern __shared__ unsigned char g_smem_raw[];
  unsigned char *base = tc::smem_base_1024(g_smem_raw);
  const MlpLayout lay = mlp_layout(a.H);
  MlpBars *sb = reinterpret_cast<MlpBars *>(base + lay.bar);
  unsigned char *W2s = base + lay.w2, *W3s = base + lay.w1, *st0 = base + lay.st;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, H = a.H, nch = H / 32;
  mlp_setup<ML_BACKWARD>(a, base, lay, sb);
  if (warp == 0) tc::tmem_alloc(&sb->tmem, 512);
  for (int e = tid; e < H * (H / 8); e += ML_THREADS) {
    const int r = e % H, c8 = e / H;   // lanes along the input units: coalesced reads of W2's rows
    __nv_bfloat16 v[8];
#pragma unroll
    for (int u = 0; u < 8; u++) v[u] = a.W2[(size_t)(c8 * 8 + u) * H + r];
    *reinterpret_cast<uint4 *>(W2s + (size_t)(c8 >> 2) * H * 64 + tc::sw64_chunk(r, c8 & 3)) =
        *reinterpret_cast<const uint4 *>(v);
  }
  for (int e = tid; e < 2 * H; e += ML_THREADS) {
    const int r = e % H, c = e / H;
    __nv_bfloat16 v[8];
#pragma unroll
    for (int u = 0; u < 8; u++) v[u] = (c * 8 + u < a.O) ? a.W3[(size_t)(c * 8 + u) * H + r] : __float2bfloat16_rn(0.0f);
    *reinterpret_cast<uint4 *>(W3s + tc::sw64_chunk(r, c)) = *reinterpret_cast<const uint4 *>(v);
  }
  tc::fence_proxy_async();
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = sb->tmem;
  const long long ntile = (a.n + 127) / 128;
  bool bad = false;
  if (warp == ML_EPI / 32) {
    if (lane == 0) {
      const uint32_t idesc = tc::idesc_bf16_f32(128, H);
      uint32_t q = 0;
      for (long long t = blockIdx.x; t < ntile && !bad; t += gridDim.x)
        for (int c = -1; c < nch; c++, q++) {   // c = -1: the rows of dY
          const uint32_t s = q % ML_ST;
          if (!tc::mbar_wait(&sb->full[s], (q / ML_ST) & 1, a.wait_ns)) { bad = true; break; }
          tc::tc_fence_after();
          if (c < 0) mma_chunk(tmem, st0 + s * ML_STAGE, W3s, idesc, 1, true);
          else mma_chunk(tmem + 256, st0 + s * ML_STAGE, W2s + (size_t)c * H * 64, idesc, 2, c == 0);
          tc::mma_commit(&sb->empty[s]);
          if (c < 0) tc::mma_commit(&sb->d1);
          else if (c == nch - 1) tc::mma_commit(&sb->d2);
        }
      tc::mma_commit(&sb->fin);
      if (!tc::mbar_wait(&sb->fin, 0)) bad = true;
    }
  } else {
    const int qd = warp & 3, g = warp >> 2, r = qd * 32 + lane;
    const uint32_t tl = tmem + ((uint32_t)(qd * 32) << 16);
    // v into the stage of sequence number q, once its last MMAs have read it
    auto put = [&](uint32_t q, const float v[32]) {
      if (q >= ML_ST && !bad && !tc::mbar_wait(&sb->empty[q % ML_ST], ((q / ML_ST) - 1) & 1, a.wait_ns)) bad = true;
      bad = __any_sync(0xffffffffu, bad);
      if (!bad) put_chunk(st0 + (q % ML_ST) * ML_STAGE, r, v);
      tc::tc_fence_before();
      tc::fence_proxy_async();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&sb->full[q % ML_ST]);
    };
    auto put_dy = [&](long long t, uint32_t q) {
      const long long row = t * 128 + r;
      float x[32];
#pragma unroll
      for (int o = 0; o < 32; o++) x[o] = (o < ML_O && o < a.O && row < a.n) ? a.dY[row * a.O + o] : 0.0f;
      put(q, x);
    };
    uint32_t q0 = 0;
    if (g == 0) put_dy(blockIdx.x, 0);
    int i = 0;
    for (long long t = blockIdx.x; t < ntile; t += gridDim.x, i++, q0 += nch + 1) {
      const long long row = t * 128 + r;
      const bool in = row < a.n;
      if (!bad && !tc::mbar_wait(&sb->d1, i & 1, a.wait_ns)) bad = true;
      bad = __any_sync(0xffffffffu, bad);
      tc::tc_fence_after();
      for (int c = g; c < nch; c += ML_G) {
        float d[32];
        tmem_ld32(tl + c * 32, d);
        if (in) act_grad32(d, a.Z2 + row * H + c * 32, a.dZ2 + row * H + c * 32);
        else
#pragma unroll
          for (int j = 0; j < 32; j++) d[j] = 0.0f;
        put(q0 + 1 + c, d);
      }
      // the next tile's dY goes in front of this tile's last epilogue
      if (g == 0 && t + gridDim.x < ntile) put_dy(t + gridDim.x, q0 + nch + 1);
      if (!bad && !tc::mbar_wait(&sb->d2, i & 1, a.wait_ns)) bad = true;
      bad = __any_sync(0xffffffffu, bad);
      tc::tc_fence_after();
      for (int c = g; c < nch; c += ML_G) {
        float d[32];
        tmem_ld32(tl + 256 + c * 32, d);
        if (in) act_grad32(d, a.Z1 + row * H + c * 32, a.dZ1 + row * H + c * 32);
      }
      // every group has read the accumulators: the next tile may refill them
      tc::tc_fence_before();
      bad = epi_any(bad);
      if (bad) break;
    }
  }
  mlp_finish(a, sb, tmem, bad);
}

// Weight and bias gradients: sums over the rows of dZ2^T H1 (W2), dZ1^T X
// (W1) and H2^T dY (W3, transposed), H1 = SiLU(Z1), H2 = SiLU(Z2).  CTA
// (x, y): rows [x kchunk, (x + 1) kchunk), units 128 y .. of the M side.  Per
// block of 32 rows thread m transposes column m of an operand into the
// K-major tiles (the lanes along the columns, so every read is a whole line),
// float32 values as bfloat16 hi + lo: products hi hi', hi lo', lo hi' as in
// k_tc_gemm.  The partial sums are added with 16-byte float32 atomics.
// The bias gradients, sums of up to a whole batch that cancel, are float64
// throughout: per thread, per CTA into `bias`, and over the CTAs in a fixed
// order (k_mlp_sums), so they are rounded once and the same in every run.
// One launch for what three k_tc_gemm launches (96 us at 16384 rows) and
// three column-sum launches (63 us, one block a column) did.
constexpr int WG_THREADS = 512;
struct WgradArgs {
  long long n;
  int F, H, O, kchunk;
  const float *X, *Z1, *Z2, *dY, *dZ1, *dZ2;
  float *gW1, *gW2, *gW3;
  double *bias;              // [x][2 H + ML_O]: column sums of dZ1, dZ2 and dY
  int *status;
  unsigned long long wait_ns;
};
// stage: A tiles dZ2, dZ1, H2 (128 units), B tiles H1 (H units), X and dY
// (32 columns each)
__host__ __device__ inline uint32_t wg_b_bytes(int H) { return (uint32_t)H * 64; }
__host__ __device__ inline uint32_t wg_stage(int H) { return 3 * 2 * GA_BYTES + 2 * wg_b_bytes(H) + 4 * 32 * 64; }

__global__ void __launch_bounds__(WG_THREADS, 1)
k_mlp_wgrad(const __grid_constant__ WgradArgs a) {
  extern __shared__ unsigned char g_smem_raw[];
  unsigned char *base = tc::smem_base_1024(g_smem_raw);
  const int H = a.H, F = a.F, O = a.O, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t bb = wg_b_bytes(H), stage = wg_stage(H);
  uint64_t *bar = reinterpret_cast<uint64_t *>(base + 2 * stage);
  uint32_t *tslot = reinterpret_cast<uint32_t *>(bar + 3);
  if (tid == 0) {
    tc::mbar_init(&bar[0], 1); tc::mbar_init(&bar[1], 1); tc::mbar_init(&bar[2], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tc::tmem_alloc(tslot, 512);
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = *tslot;   // W2 at 0 (H columns), W1 at 256 and W3 at 288 (32 each)
  const int m0 = blockIdx.y * 128;
  const long long k0 = (long long)blockIdx.x * a.kchunk, k1 = min(a.n, k0 + a.kchunk);
  const int nblk = (int)((k1 - k0 + GK - 1) / GK);
  const int NF = ((F + 15) / 16) * 16, NO16 = 16;
  const uint32_t id2 = tc::idesc_bf16_f32(128, H), id1 = tc::idesc_bf16_f32(128, NF), id3 = tc::idesc_bf16_f32(128, NO16);
  double sb1 = 0.0, sb2 = 0.0, sb3 = 0.0;   // column sums of dZ1, dZ2 (thread = unit m0 + (tid & 127)) and dY
  bool bad = false;
  for (int ib = 0; ib < nblk; ib++) {
    const int s = ib & 1;
    const long long kb = k0 + (long long)ib * GK;
    unsigned char *st = base + s * stage;
    if (ib >= 2 && !tc::mbar_wait(&bar[s], ((ib - 2) >> 1) & 1, a.wait_ns)) bad = true;
    if (__syncthreads_or(bad)) { bad = true; break; }
    unsigned char *tB = st + 6 * GA_BYTES, *tX = tB + 2 * bb, *tY = tX + 2 * 32 * 64;
    // A tiles: thread = (unit, chunk of 8 rows)
    {
      const int m = tid & 127, c = tid >> 7, u = m0 + m;
      const bool ok = u < H;
      float v2[8], v1[8], hh[8];
#pragma unroll
      for (int e = 0; e < 8; e++) {
        const long long k = kb + c * 8 + e;
        const bool in = ok && k < k1;
        const size_t at = in ? (size_t)k * H + u : 0;
        v2[e] = in ? __ldg(a.dZ2 + at) : 0.0f;
        v1[e] = in ? __ldg(a.dZ1 + at) : 0.0f;
        hh[e] = in ? __ldg(a.Z2 + at) : 0.0f;
      }
#pragma unroll
      for (int e = 0; e < 8; e++) { sb2 += (double)v2[e]; sb1 += (double)v1[e]; }
      silu<8>(hh);
      put_row8<2>(st, GA_BYTES, m, c, v2);
      put_row8<2>(st + 2 * GA_BYTES, GA_BYTES, m, c, v1);
      put_row8<2>(st + 4 * GA_BYTES, GA_BYTES, m, c, hh);
    }
    // B tile H1: thread = (unit, chunks of 8 rows)
    for (int e0 = tid; e0 < 4 * H; e0 += WG_THREADS) {
      const int u = e0 % H, c = e0 / H;
      float v[8];
#pragma unroll
      for (int e = 0; e < 8; e++) {
        const long long k = kb + c * 8 + e;
        v[e] = (k < k1) ? __ldg(a.Z1 + (size_t)k * H + u) : 0.0f;
      }
      silu<8>(v);
      put_row8<2>(tB, bb, u, c, v);
    }
    // B tiles X and dY: thread = (chunk of 8 rows, column)
    if (tid < 256) {
      const int c = (tid >> 5) & 3, u = tid & 31;
      const bool isx = tid < 128;
      const int w = isx ? F : O;
      const float *src = isx ? a.X : a.dY;
      float v[8];
#pragma unroll
      for (int e = 0; e < 8; e++) {
        const long long k = kb + c * 8 + e;
        v[e] = (u < w && k < k1) ? __ldg(src + (size_t)k * w + u) : 0.0f;
      }
      if (!isx) {
#pragma unroll
        for (int e = 0; e < 8; e++) sb3 += (double)v[e];
      }
      put_row8<2>(isx ? tX : tY, 32 * 64, u, c, v);
    }
    tc::fence_proxy_async();
    __syncthreads();
    if (tid == 0) {
      tc::tc_fence_after();
#pragma unroll
      for (int ks = 0; ks < GK / 16; ks++) {
        const uint64_t o = (uint64_t)(ks * 2);
        const uint32_t first = (ib == 0 && ks == 0) ? 0u : 1u;
        // the cross terms in the order of k_tc_gemm's dZ^T H, dZ^T X and dY^T H (W3: A and B change places)
        auto mul = [&](uint32_t acc, const unsigned char *A, const unsigned char *B, uint32_t lo, uint32_t idesc,
                       bool swapped) {
          const uint64_t ah = tc::smem_desc_sw64(A) + o, al = tc::smem_desc_sw64(A + GA_BYTES) + o;
          const uint64_t bh = tc::smem_desc_sw64(B) + o, bl = tc::smem_desc_sw64(B + lo) + o;
          tc::mma_f16(acc, ah, bh, idesc, first);
          if (swapped) tc::mma_f16(acc, al, bh, idesc, 1u);
          tc::mma_f16(acc, ah, bl, idesc, 1u);
          if (!swapped) tc::mma_f16(acc, al, bh, idesc, 1u);
        };
        mul(tmem, st, tB, bb, id2, false);
        mul(tmem + 256, st + 2 * GA_BYTES, tX, 32 * 64, id1, false);
        mul(tmem + 288, st + 4 * GA_BYTES, tY, 32 * 64, id3, true);
      }
      tc::mma_commit(&bar[s]);
    }
  }
  if (tid == 0) tc::mma_commit(&bar[2]);
  if (!tc::mbar_wait(&bar[2], 0)) bad = true;
  bad = __syncthreads_or(bad);
  tc::tc_fence_after();
  if (bad) {
    if (tid == 0) atomicOr(a.status, CB2_STATUS_PIPE_TIMEOUT);
  } else if (nblk > 0) {
    const int qd = warp & 3, g = warp >> 2, u = m0 + qd * 32 + lane;
    const uint32_t tl = tmem + ((uint32_t)(qd * 32) << 16);
    float v[32];
    for (int c = g; c < H / 32; c += WG_THREADS / 128) {
      tmem_ld32(tl + c * 32, v);
      if (u < H) {
        float4 *d = reinterpret_cast<float4 *>(a.gW2 + (size_t)u * H + c * 32);
#pragma unroll
        for (int j = 0; j < 8; j++) atomicAdd(d + j, make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]));
      }
    }
    if (g == 0) {
      tmem_ld32(tl + 256, v);
#pragma unroll
      for (int j = 0; j < 32; j++)
        if (u < H && j < F) atomicAdd(a.gW1 + (size_t)u * F + j, v[j]);
    } else if (g == 1) {
      tmem_ld32(tl + 288, v);
#pragma unroll
      for (int j = 0; j < ML_O; j++)
        if (u < H && j < O) atomicAdd(a.gW3 + (size_t)j * H + u, v[j]);
    }
    // the four threads of a unit (and of a column of dY), in the stages' memory
    double *red = reinterpret_cast<double *>(base);
    red[tid] = sb1;
    red[WG_THREADS + tid] = sb2;
    if (tid >= 128 && tid < 256) red[2 * WG_THREADS + tid - 128] = sb3;
    __syncthreads();
    double *out = a.bias + (size_t)blockIdx.x * (2 * H + ML_O);
    auto sum4 = [](const double *x, int st) { return ((x[0] + x[st]) + x[2 * st]) + x[3 * st]; };
    if (tid < 256) {
      const int m = tid & 127, which = tid >> 7;
      if (m0 + m < H) out[which * H + m0 + m] = sum4(red + which * WG_THREADS + m, 128);
    } else if (blockIdx.y == 0 && tid < 256 + O) {
      out[2 * H + tid - 256] = sum4(red + 2 * WG_THREADS + tid - 256, 32);
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, 512);
}

// loss = sum of the partial sums / (n O) (one block of 256, fixed order)
__device__ inline void loss_sum(double *sh, long long np, const double *part, double inv, double *out) {
  double s = 0.0;
  for (long long i = threadIdx.x; i < np; i += 256) s += part[i];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int q = 128; q > 0; q >>= 1) {
    if (threadIdx.x < q) sh[threadIdx.x] += sh[threadIdx.x + q];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[0] = sh[0] * inv;
}
__global__ void __launch_bounds__(256)
k_loss_sum(long long np, const double *part, double inv, double *out) {
  __shared__ double sh[256];
  loss_sum(sh, np, part, inv, out);
}

// after k_mlp_wgrad: a block adds 32 columns of its nx partial sums, eight
// threads a column, into the bias gradients; the last block the loss
__global__ void __launch_bounds__(256)
k_mlp_sums(int nx, int H, int O, const double *bias, float *gb1, float *gb2, float *gb3, long long np,
           const double *part, double inv, double *loss) {
  __shared__ double sh[256];
  if (blockIdx.x == gridDim.x - 1) {
    loss_sum(sh, np, part, inv, loss);
    return;
  }
  const int c = blockIdx.x * 32 + (threadIdx.x & 31);
  double s = 0.0;
  if (c < 2 * H + O)
    for (int x = threadIdx.x >> 5; x < nx; x += 8) s += bias[(size_t)x * (2 * H + ML_O) + c];
  sh[threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.x >= 32 || c >= 2 * H + O) return;
  for (int q = 1; q < 8; q++) s += sh[32 * q + threadIdx.x];
  float *g = (c < H) ? gb1 + c : (c < 2 * H) ? gb2 + c - H : gb3 + c - 2 * H;
  *g = (float)s;
}

// Z += b (per column); H = SiLU(Z) (act != 0) or Z
__global__ void k_bias_act(size_t n, int w, float *Z, const float *b, float *H, int act) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n * w) return;
  const float z = Z[i] + b[i % w];
  Z[i] = z;
  H[i] = act ? z * sigm(z) : z;
}

// dZ = dH * SiLU'(Z)
__global__ void k_act_grad(size_t n, const float *Z, const float *dH, float *dZ) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float s = sigm(Z[i]);
  dZ[i] = dH[i] * s * (1.0f + Z[i] * (1.0f - s));
}

// dY = 2 (Y - T) / (n nout); partial loss sums (float64) per block
__global__ void k_mse(size_t n, int w, const float *Y, const float *T, float *dY, double *part) {
  __shared__ double sh[256];
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  double e = 0.0;
  if (i < n * w) {
    const float d = Y[i] - T[i];
    dY[i] = 2.0f * d / (float)(n * (size_t)w);
    e = (double)d * (double)d;
  }
  sh[threadIdx.x] = e;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = sh[0];
}

// column sums of X[n][w] into out[w] (one block per column, float64 partials)
__global__ void k_colsum(size_t n, int w, const float *X, float *out) {
  __shared__ double sh[256];
  const int c = blockIdx.x;
  double s = 0.0;
  for (size_t i = threadIdx.x; i < n; i += blockDim.x) s += X[i * w + c];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int q = blockDim.x / 2; q > 0; q >>= 1) {
    if (threadIdx.x < q) sh[threadIdx.x] += sh[threadIdx.x + q];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[c] = (float)sh[0];
}

// one Adam step of the float32 master parameters and their bfloat16 copy
__global__ void k_adam(size_t n, float *p, const float *g, float *m, float *v, float lr, float b1, float b2,
                       float eps, float c1, float c2, __nv_bfloat16 *w) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.0f - b1) * gi, vi = b2 * v[i] + (1.0f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  const float pi = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  p[i] = pi;
  w[i] = __float2bfloat16_rn(pi);
}

__global__ void k_to_bf16(size_t n, const float *src, __nv_bfloat16 *dst) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = __float2bfloat16_rn(src[i]);
}

inline unsigned blocks(size_t n, int t = 256) { return (unsigned)((n + t - 1) / t); }

}  // namespace
}  // namespace cb2

using namespace cb2;

// ---------------------------------------------------------------------------
// the network
constexpr size_t kTailBytes = 16;
struct ClosureState;
struct cb2_mlp {
  int F = 0, H = 0, O = 0;
  size_t oW1 = 0, ob1 = 0, oW2 = 0, ob2 = 0, oW3 = 0, ob3 = 0, np = 0;
  float *master = nullptr, *grad = nullptr, *m = nullptr, *v = nullptr;
  __nv_bfloat16 *w = nullptr;   // bfloat16 copy of every parameter (the products use W1, W2, W3)
  int t = 0;
  // the work buffers below, in two allocations: rows x H, and the small ones
  float *work = nullptr, *work_small = nullptr;
  size_t cap = 0;               // their rows
  float *Z1 = nullptr, *H1 = nullptr, *Z2 = nullptr, *H2 = nullptr, *Yp = nullptr, *dY = nullptr;
  float *dH = nullptr, *dZ = nullptr;
  double *part = nullptr;       // loss partial sums
  double *bias = nullptr;       // bias gradients' partial sums (fused passes)
  // behind the gradient in its allocation, read together: the loss of the
  // last fused training pass and the status word of the products (bit 2: a
  // wait ran out)
  double *loss = nullptr;
  int *status = nullptr;
  size_t ycap = 0;              // rows of Yp
  // budget of each wait inside the products (ns), CB2_PIPE_WAIT_NS as for a context
  unsigned long long wait_ns = tc::kWaitNs;
  cudaStream_t stream = nullptr;
  // the parameters are written on `stream` and read there and on the streams of
  // the contexts the network is attached to: `written` follows their last
  // change, and each user's `read` its last pass
  cudaEvent_t written = nullptr;
  std::vector<ClosureState *> users;
};

namespace cb2 {
namespace {

// the sizes the one-kernel passes take: tensor memory holds two accumulators
// of 256 columns, shared memory W2 and the operand stages (208 KB at H = 256),
// the last layer sits in registers; W2's rows are copied 16 bytes at a time
bool fused_ok(const cb2_mlp *n) {
  return n->F <= 32 && n->H % 32 == 0 && n->H >= 64 && n->H <= 256 && n->O <= ML_O && n->oW2 % 8 == 0;
}

// chunks (at most) and rows of a chunk of a sum over n rows into `tiles` output tiles: at
// least 256 rows, and the chunks cover the SMs about twice
long long split_chunks(long long n, int tiles) {
  return std::max<long long>(1, std::min<long long>((n + 255) / 256, (2 * 148 + tiles - 1) / tiles));
}
int split_chunk(long long n, int tiles) {
  const long long nz = split_chunks(n, tiles);
  return (int)(((n + nz - 1) / nz + GK - 1) / GK * GK);
}

// Work buffers of `rows` rows.  The fused passes keep the activations on the
// chip: inference needs none of these, training Z1, Z2 and the gradients dY, dZ2
// (in dZ) and dZ1 (in dH).  The few that are not rows x H have an allocation of
// their own: with them at the end of the large one, the next network took longer
// to make once this one was freed (made with its batch, first trained and freed at
// 16384 rows: 1.2 + 0.7 + 0.8 ms, so 0.8 - 0.95 + 0.75 + 0.5).
int mlp_reserve(cb2_mlp *n, size_t rows, bool train) {
  const bool fused = fused_ok(n);
  if ((fused && !train) || rows <= n->cap) return 0;
  const size_t w = (rows * n->H + 63) / 64 * 64, wy = (rows * n->O + 63) / 64 * 64;
  const size_t pc = std::max((size_t)blocks(rows * n->O), 4 * ((rows + 127) / 128)) + 1;
  const size_t bc = fused ? (size_t)split_chunks(rows, (n->H + 127) / 128) * (2 * n->H + ML_O) : 0;
  n->cap = 0;
  if (n->work) cudaFree(n->work);
  if (n->work_small) cudaFree(n->work_small);
  n->work = n->work_small = nullptr;
  CB2_CUDA(cudaMalloc(&n->work, (fused ? 4 : 6) * w * sizeof(float)));
  CB2_CUDA(cudaMalloc(&n->work_small, wy * sizeof(float) + (pc + bc) * sizeof(double)));
  n->Z1 = n->work; n->Z2 = n->Z1 + w; n->dH = n->Z2 + w; n->dZ = n->dH + w;
  n->H1 = n->dZ + w; n->H2 = n->H1 + w;   // the general passes only
  n->dY = n->work_small;
  n->part = reinterpret_cast<double *>(n->dY + wy);
  n->bias = n->part + pc;
  n->cap = rows;
  return 0;
}

// the output buffer of passes that have none of the caller's
int mlp_reserve_y(cb2_mlp *n, size_t rows) {
  if (rows <= n->ycap) return 0;
  n->ycap = 0;
  if (n->Yp) cudaFree(n->Yp);
  n->Yp = nullptr;
  CB2_CUDA(cudaMalloc(&n->Yp, rows * n->O * sizeof(float)));
  n->ycap = rows;
  return 0;
}

MlpArgs mlp_args(const cb2_mlp *n, const float *X, size_t rows, int *status) {
  MlpArgs a{};
  a.n = (long long)rows; a.F = n->F; a.H = n->H; a.O = n->O;
  a.X = X;
  a.vec = n->F % 4 == 0 && (reinterpret_cast<uintptr_t>(X) & 15) == 0;
  a.b1 = n->master + n->ob1; a.b2 = n->master + n->ob2; a.b3 = n->master + n->ob3;
  a.W1 = n->w + n->oW1; a.W2 = n->w + n->oW2; a.W3 = n->w + n->oW3;
  a.count = (float)(rows * (size_t)n->O);
  a.status = status;
  a.wait_ns = n->wait_ns;
  return a;
}

// one CTA per SM over the row tiles
template <typename K>
int launch_rows(K *kernel, const MlpArgs &a, cudaStream_t st) {
  const size_t smem = mlp_layout(a.H).total + 1024;
  CB2_CUDA(raise_smem_limit(kernel, smem));
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  kernel<<<(unsigned)std::min<long long>(sms, (a.n + 127) / 128), ML_THREADS, smem, st>>>(a);
  CB2_CUDA(cudaGetLastError());
  return 0;
}

// C = opA opB on the tensor cores (k_tc_gemm).  split_k: K is cut into
// chunks so that the grid covers the SMs about twice, C is cleared and the
// chunks' partial products are added with atomics.
struct GemmRun {
  cudaStream_t st;
  int *status;
  unsigned long long wait_ns;
};
template <typename TAT, typename TBT, bool TA, bool TB>
void gemm(const GemmRun &run, int M, int N, int K, const TAT *A, int lda, const TBT *B, int ldb, float *C, int ldc,
          bool split_k) {
  const cudaStream_t st = run.st;
  constexpr int NA = Terms<TAT>::n, NBT = Terms<TBT>::n;
  const int NT = std::min(256, ((N + 15) / 16) * 16);
  uint32_t cols = 64;
  while ((int)cols < NT) cols *= 2;
  const uint32_t stage = ((NA * GA_BYTES + NBT * (uint32_t)NT * GK * 2) + 1023u) & ~1023u;
  const size_t smem = 2 * (size_t)stage + 64 + 1024;
  static bool attr_set = false;
  if (!attr_set) {
    cudaFuncSetAttribute(k_tc_gemm<TAT, TBT, TA, TB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         2 * (2 * GA_BYTES + 2 * 256 * GK * 2) + 64 + 1024);
    attr_set = true;
  }
  const int tiles = ((N + NT - 1) / NT) * ((M + 127) / 128);
  int kchunk = K, nz = 1;
  if (split_k) {
    kchunk = split_chunk(K, tiles);
    nz = (K + kchunk - 1) / kchunk;
    cudaMemsetAsync(C, 0, (size_t)M * ldc * sizeof(float), st);
  }
  dim3 grid((N + NT - 1) / NT, (M + 127) / 128, nz);
  k_tc_gemm<TAT, TBT, TA, TB><<<grid, 128, smem, st>>>(M, N, NT, K, A, lda, B, ldb, C, ldc, kchunk,
                                                        split_k ? 1 : 0, cols, run.status, run.wait_ns);
}

// forward pass of n rows of X (normalised features) into Y, on stream st
int mlp_forward(cb2_mlp *nt, const float *X, size_t n, float *Y, cudaStream_t st, int *status = nullptr) {
  if (!status) status = nt->status;
  if (fused_ok(nt)) {
    MlpArgs a = mlp_args(nt, X, n, status);
    a.Y = Y;
    return nt->O <= 5 ? launch_rows(k_mlp_fwd<false, 5>, a, st) : launch_rows(k_mlp_fwd<false, 8>, a, st);
  }
  int rc = mlp_reserve(nt, n, false);
  if (rc) return rc;
  const int F = nt->F, H = nt->H, O = nt->O;
  const GemmRun run{st, status, nt->wait_ns};
  gemm<float, __nv_bfloat16, false, true>(run, (int)n, H, F, X, F, nt->w + nt->oW1, F, nt->Z1, H, false);
  k_bias_act<<<blocks(n * H), 256, 0, st>>>(n, H, nt->Z1, nt->master + nt->ob1, nt->H1, 1);
  gemm<float, __nv_bfloat16, false, true>(run, (int)n, H, H, nt->H1, H, nt->w + nt->oW2, H, nt->Z2, H,
                                          false);
  k_bias_act<<<blocks(n * H), 256, 0, st>>>(n, H, nt->Z2, nt->master + nt->ob2, nt->H2, 1);
  gemm<float, __nv_bfloat16, false, true>(run, (int)n, O, H, nt->H2, H, nt->w + nt->oW3, H, Y, O,
                                          false);
  k_bias_act<<<blocks(n * O), 256, 0, st>>>(n, O, Y, nt->master + nt->ob3, Y, 0);
  CB2_CUDA(cudaGetLastError());
  return 0;
}

// the fused training pass: loss (left in nt->loss) and gradients
int mlp_backward_fused(cb2_mlp *nt, const float *X, const float *T, size_t n) {
  cudaStream_t st = nt->stream;
  MlpArgs a = mlp_args(nt, X, n, nt->status);
  a.T = T; a.Z1 = nt->Z1; a.Z2 = nt->Z2; a.dY = nt->dY; a.dZ2 = nt->dZ; a.dZ1 = nt->dH; a.part = nt->part;
  CB2_CUDA(cudaMemsetAsync(nt->grad, 0, nt->np * sizeof(float), st));
  int rc = nt->O <= 5 ? launch_rows(k_mlp_fwd<true, 5>, a, st) : launch_rows(k_mlp_fwd<true, 8>, a, st);
  if (rc) return rc;
  if ((rc = launch_rows(k_mlp_bwd, a, st))) return rc;
  WgradArgs w{};
  w.n = a.n; w.F = a.F; w.H = a.H; w.O = a.O;
  w.X = X; w.Z1 = nt->Z1; w.Z2 = nt->Z2; w.dY = nt->dY; w.dZ1 = nt->dH; w.dZ2 = nt->dZ;
  w.gW1 = nt->grad + nt->oW1; w.gW2 = nt->grad + nt->oW2; w.gW3 = nt->grad + nt->oW3;
  w.bias = nt->bias;
  w.status = nt->status; w.wait_ns = nt->wait_ns;
  const int ny = (a.H + 127) / 128;
  w.kchunk = split_chunk(a.n, ny);
  const size_t smem = 2 * (size_t)wg_stage(a.H) + 64 + 1024;
  CB2_CUDA(raise_smem_limit(k_mlp_wgrad, smem));
  const unsigned nx = (unsigned)((a.n + w.kchunk - 1) / w.kchunk);
  k_mlp_wgrad<<<dim3(nx, ny), WG_THREADS, smem, st>>>(w);
  k_mlp_sums<<<cdiv(2 * a.H + a.O, 32) + 1, 256, 0, st>>>((int)nx, a.H, a.O, nt->bias, nt->grad + nt->ob1,
                                                          nt->grad + nt->ob2, nt->grad + nt->ob3,
                                                          4 * ((a.n + 127) / 128), nt->part,
                                                          1.0 / ((double)n * nt->O), nt->loss);
  CB2_CUDA(cudaGetLastError());
  return 0;
}

// loss (nt->loss) and gradients (grad <- dL/dparams) of the mean squared error over n rows
int mlp_backward(cb2_mlp *nt, const float *X, const float *T, size_t n) {
  cudaStream_t st = nt->stream;
  int rc = mlp_reserve(nt, n, true);
  if (rc) return rc;
  if (fused_ok(nt)) {
    if ((rc = mlp_backward_fused(nt, X, T, n))) return rc;
    return 0;
  }
  if ((rc = mlp_reserve_y(nt, n)) || (rc = mlp_forward(nt, X, n, nt->Yp, st))) return rc;
  const int F = nt->F, H = nt->H, O = nt->O;
  const GemmRun run{st, nt->status, nt->wait_ns};
  const unsigned nb = blocks(n * O);
  k_mse<<<nb, 256, 0, st>>>(n, O, nt->Yp, T, nt->dY, nt->part);
  // layer 3
  gemm<float, float, true, false>(run, O, H, (int)n, nt->dY, O, nt->H2, H, nt->grad + nt->oW3, H, true);
  k_colsum<<<O, 256, 0, st>>>(n, O, nt->dY, nt->grad + nt->ob3);
  gemm<float, __nv_bfloat16, false, false>(run, (int)n, H, O, nt->dY, O, nt->w + nt->oW3, H, nt->dH, H, false);
  k_act_grad<<<blocks(n * H), 256, 0, st>>>(n * H, nt->Z2, nt->dH, nt->dZ);
  // layer 2
  gemm<float, float, true, false>(run, H, H, (int)n, nt->dZ, H, nt->H1, H, nt->grad + nt->oW2, H, true);
  k_colsum<<<H, 256, 0, st>>>(n, H, nt->dZ, nt->grad + nt->ob2);
  gemm<float, __nv_bfloat16, false, false>(run, (int)n, H, H, nt->dZ, H, nt->w + nt->oW2, H, nt->dH, H, false);
  k_act_grad<<<blocks(n * H), 256, 0, st>>>(n * H, nt->Z1, nt->dH, nt->dZ);
  // layer 1
  gemm<float, float, true, false>(run, H, F, (int)n, nt->dZ, H, X, F, nt->grad + nt->oW1, F, true);
  k_colsum<<<H, 256, 0, st>>>(n, H, nt->dZ, nt->grad + nt->ob1);
  CB2_CUDA(cudaGetLastError());
  k_loss_sum<<<1, 256, 0, st>>>(nb, nt->part, 1.0 / ((double)n * O), nt->loss);
  CB2_CUDA(cudaGetLastError());
  return 0;
}

}  // namespace
}  // namespace cb2

// closure state of a context
struct ClosureState {
  cb2_mlp *net = nullptr;
  float *norm = nullptr;     // [nr][16 mean], [nr][16 1/std], [nr][5 out scale]
  float *X = nullptr, *Xn = nullptr;
  size_t rows = 0;
  cudaEvent_t read = nullptr;   // after the last pass that read the network's parameters
};

namespace cb2 {
// An event between a context's stream and the network's.  Where the step is
// being captured into a graph, the wait and the record become nodes of the
// graph, which each launch runs anew.
static int event_on(cudaStream_t st, cudaEvent_t e, bool wait) {
  cudaStreamCaptureStatus cap;
  CB2_CUDA(cudaStreamIsCapturing(st, &cap));
  const bool graph = cap == cudaStreamCaptureStatusActive;
  if (wait) CB2_CUDA(cudaStreamWaitEvent(st, e, graph ? cudaEventWaitExternal : cudaEventWaitDefault));
  else CB2_CUDA(cudaEventRecordWithFlags(e, st, graph ? cudaEventRecordExternal : cudaEventRecordDefault));
  return 0;
}

// called by the time step after the explicit nonlinear terms are formed
int closure_apply(Ctx &c) {
  ClosureState *cs = static_cast<ClosureState *>(c.closure);
  if (!cs || !cs->net) return 0;
  const size_t n = cs->rows;
  k_features<<<blocks(n), 256, 0, c.stream>>>(c.nr, c.jmax, c.L, c.d_jl, c.d_jm, c.d_r, c.h_r[c.kin],
                                              c.h_r[c.kout], c.d_f, c.fsize(), feat_slots(), cs->X);
  const size_t nn = (size_t)c.nr * NF;
  k_normalise<<<blocks(n * NF), 256, 0, c.stream>>>(n, c.jmax, cs->X, cs->norm, cs->norm + nn, cs->Xn);
  int rc = event_on(c.stream, cs->net->written, true);
  if (rc || (rc = mlp_forward(cs->net, cs->Xn, n, cs->net->Yp, c.stream, c.d_status))) return rc;
  if ((rc = event_on(c.stream, cs->read, false))) return rc;
  k_add_tendency<<<blocks(n), 256, 0, c.stream>>>(n, c.nr, c.jmax, cs->net->Yp, cs->norm + 2 * nn, c.d_f, c.fsize(),
                                                  out_slots());
  return 0;
}

void closure_free(Ctx &c) {
  ClosureState *cs = static_cast<ClosureState *>(c.closure);
  if (!cs) return;
  if (cs->norm) cudaFree(cs->norm);
  if (cs->X) cudaFree(cs->X);
  if (cs->Xn) cudaFree(cs->Xn);
  if (cs->read) cudaEventDestroy(cs->read);
  if (cs->net) {
    auto &u = cs->net->users;
    u.erase(std::remove(u.begin(), u.end(), cs), u.end());
  }
  delete cs;
  c.closure = nullptr;
}
}  // namespace cb2

extern "C" {

int cb2_mlp_create(int nin, int nhid, int nout, unsigned seed, cb2_mlp **out) {
  if (!out || nin <= 0 || nhid <= 0 || nout <= 0) { set_error("cb2_mlp_create: bad argument"); return CB2_ERR_ARG; }
  *out = nullptr;
  cb2_mlp *n = new cb2_mlp();
  n->F = nin; n->H = nhid; n->O = nout;
  if (const char *pw = getenv("CB2_PIPE_WAIT_NS")) n->wait_ns = strtoull(pw, nullptr, 10);
  n->oW1 = 0; n->ob1 = n->oW1 + (size_t)nhid * nin; n->oW2 = n->ob1 + nhid;
  n->ob2 = n->oW2 + (size_t)nhid * nhid; n->oW3 = n->ob2 + nhid; n->ob3 = n->oW3 + (size_t)nout * nhid;
  n->np = n->ob3 + nout;
  // He-style uniform initialisation, biases zero (host generator: splitmix64)
  std::vector<float> p(n->np, 0.0f);
  unsigned long long s = 0x9E3779B97F4A7C15ULL ^ ((unsigned long long)seed << 21);
  auto uni = [&]() {
    unsigned long long z = (s += 0x9E3779B97F4A7C15ULL);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    z ^= z >> 31;
    return (double)(z >> 11) * (1.0 / 9007199254740992.0);
  };
  auto fill = [&](size_t off, size_t cnt, int fan_in) {
    const double a = std::sqrt(3.0 / fan_in);
    for (size_t q = 0; q < cnt; q++) p[off + q] = (float)((2.0 * uni() - 1.0) * a);
  };
  fill(n->oW1, (size_t)nhid * nin, nin);
  fill(n->oW2, (size_t)nhid * nhid, nhid);
  fill(n->oW3, (size_t)nout * nhid, nhid);
  auto fail = [&](int rc) { cb2_mlp_destroy(n); return rc; };
  const size_t gtail = (n->np + 3) / 4 * 4;
  if (cudaStreamCreateWithFlags(&n->stream, cudaStreamNonBlocking) != cudaSuccess ||
      cudaEventCreateWithFlags(&n->written, cudaEventDisableTiming) != cudaSuccess ||
      cudaMalloc(&n->master, n->np * sizeof(float)) != cudaSuccess ||
      cudaMalloc(&n->grad, gtail * sizeof(float) + kTailBytes) != cudaSuccess ||
      cudaMalloc(&n->m, n->np * sizeof(float)) != cudaSuccess ||
      cudaMalloc(&n->v, n->np * sizeof(float)) != cudaSuccess ||
      cudaMalloc(&n->w, n->np * sizeof(__nv_bfloat16)) != cudaSuccess)
    return fail(cuda_fail(cudaGetLastError(), "cb2_mlp_create"));
  n->loss = reinterpret_cast<double *>(n->grad + gtail);
  n->status = reinterpret_cast<int *>(n->loss + 1);
  // all on the network's stream, which does not wait for the default one
  cudaMemcpyAsync(n->master, p.data(), n->np * sizeof(float), cudaMemcpyHostToDevice, n->stream);
  cudaMemsetAsync(n->grad, 0, gtail * sizeof(float) + kTailBytes, n->stream);
  cudaMemsetAsync(n->m, 0, n->np * sizeof(float), n->stream);
  cudaMemsetAsync(n->v, 0, n->np * sizeof(float), n->stream);
  k_to_bf16<<<blocks(n->np), 256, 0, n->stream>>>(n->np, n->master, n->w);
  cudaEventRecord(n->written, n->stream);
  if (cudaStreamSynchronize(n->stream) != cudaSuccess) return fail(cuda_fail(cudaGetLastError(), "cb2_mlp_create"));
  *out = n;
  return 0;
}

int cb2_mlp_destroy(cb2_mlp *n) {
  if (!n) return 0;
  if (n->stream) cudaStreamSynchronize(n->stream);
  for (ClosureState *cs : n->users) cs->net = nullptr;
  void *ptrs[] = {n->master, n->grad, n->m, n->v, n->w, n->work, n->work_small, n->Yp};
  for (void *q : ptrs)
    if (q) cudaFree(q);
  if (n->written) cudaEventDestroy(n->written);
  if (n->stream) cudaStreamDestroy(n->stream);
  delete n;
  return 0;
}

int cb2_mlp_num_params(const cb2_mlp *n) { return n ? (int)n->np : -1; }

// float32 master parameters: W1 [H][F], b1 [H], W2 [H][H], b2 [H], W3 [O][H], b3 [O]
int cb2_mlp_get_params(cb2_mlp *n, float *host) {
  if (!n || !host) return CB2_ERR_ARG;
  // behind the updates queued on the network's stream
  CB2_CUDA(cudaMemcpyAsync(host, n->master, n->np * sizeof(float), cudaMemcpyDeviceToHost, n->stream));
  CB2_CUDA(cudaStreamSynchronize(n->stream));
  return 0;
}

// the network's stream behind every pass of an attached context, which reads the
// parameters and uses the work buffers of the general kernels and Yp: before
// either is written
static int after_users(cb2_mlp *n) {
  for (ClosureState *cs : n->users) CB2_CUDA(cudaStreamWaitEvent(n->stream, cs->read, cudaEventWaitDefault));
  return 0;
}

int cb2_mlp_set_params(cb2_mlp *n, const float *host) {
  if (!n || !host) return CB2_ERR_ARG;
  if (int rc = after_users(n)) return rc;
  CB2_CUDA(cudaMemcpyAsync(n->master, host, n->np * sizeof(float), cudaMemcpyHostToDevice, n->stream));
  k_to_bf16<<<blocks(n->np), 256, 0, n->stream>>>(n->np, n->master, n->w);
  CB2_CUDA(cudaEventRecord(n->written, n->stream));
  CB2_CUDA(cudaStreamSynchronize(n->stream));
  return 0;
}

// the status word (and the last loss) after the stream has drained: a
// pipeline wait that ran out is reported (and the word cleared)
static int mlp_status(cb2_mlp *n, double *loss = nullptr) {
  struct { double loss; int st; int pad; } tail;
  static_assert(sizeof(tail) == kTailBytes, "gradient tail");
  CB2_CUDA(cudaMemcpyAsync(&tail, n->loss, sizeof(tail), cudaMemcpyDeviceToHost, n->stream));
  CB2_CUDA(cudaStreamSynchronize(n->stream));
  if (tail.st) {
    CB2_CUDA(cudaMemsetAsync(n->status, 0, sizeof(int), n->stream));
    set_error("closure network: a tensor-core pipeline wait ran out");
    return CB2_ERR_TIMEOUT;
  }
  if (loss) *loss = tail.loss;
  return 0;
}

int cb2_mlp_forward(cb2_mlp *n, const float *dev_x, long long rows, float *dev_y) {
  if (!n || !dev_x || !dev_y || rows <= 0) return CB2_ERR_ARG;
  // the fused pass writes the rows of a tile while other tiles are still to be
  // read: an output that overlaps the input goes through a buffer (the
  // general kernels have read the input when their last layer writes)
  const size_t nx = (size_t)rows * n->F, ny = (size_t)rows * n->O;
  const std::less<const float *> before;
  const bool overlap = fused_ok(n) && before(dev_x, dev_y + ny) && before(dev_y, dev_x + nx);
  float *y = dev_y;
  if (overlap || !fused_ok(n))
    if (int rc = after_users(n)) return rc;
  if (overlap) {
    if (int rc = mlp_reserve_y(n, (size_t)rows)) return rc;
    y = n->Yp;
  }
  if (int rc = mlp_forward(n, dev_x, (size_t)rows, y, n->stream)) return rc;
  if (overlap) CB2_CUDA(cudaMemcpyAsync(dev_y, y, ny * sizeof(float), cudaMemcpyDeviceToDevice, n->stream));
  return mlp_status(n);
}

// mean squared error of rows x (normalised features) against t, and its
// gradient (kept for cb2_mlp_adam_step; copied to host_grad when not NULL)
int cb2_mlp_loss_grad(cb2_mlp *n, const float *dev_x, const float *dev_t, long long rows, double *loss,
                      float *host_grad) {
  if (!n || !dev_x || !dev_t || rows <= 0) return CB2_ERR_ARG;
  double l = 0.0;
  int rc = fused_ok(n) ? 0 : after_users(n);
  if (rc || (rc = mlp_backward(n, dev_x, dev_t, (size_t)rows)) || (rc = mlp_status(n, &l))) return rc;
  if (loss) *loss = l;
  if (host_grad) CB2_CUDA(cudaMemcpy(host_grad, n->grad, n->np * sizeof(float), cudaMemcpyDeviceToHost));
  return 0;
}

int cb2_mlp_adam_step(cb2_mlp *n, float lr, float beta1, float beta2, float eps) {
  if (!n) return CB2_ERR_ARG;
  if (int rc = after_users(n)) return rc;
  n->t += 1;
  const float c1 = 1.0f - std::pow(beta1, (float)n->t), c2 = 1.0f - std::pow(beta2, (float)n->t);
  k_adam<<<blocks(n->np), 256, 0, n->stream>>>(n->np, n->master, n->grad, n->m, n->v, lr, beta1, beta2, eps, c1, c2, n->w);
  CB2_CUDA(cudaGetLastError());
  CB2_CUDA(cudaEventRecord(n->written, n->stream));
  return 0;
}

int cb2_mlp_sync(cb2_mlp *n) {
  if (!n) return CB2_ERR_ARG;
  return mlp_status(n);
}

// dst's 13 state fields (velocity, vorticity, magnetic field, current,
// temperature) := src's, truncated to dst's L and restricted to dst's
// radial points; then dst's derived fields and nonlinear terms are rebuilt
// (cb2_start).  dst's radial points must be every stride-th point of src's.
static int filter_check(const cb2_ctx *s, const cb2_ctx *d, int *stride) {
  if (!s || !d) { set_error("filter: null context"); return CB2_ERR_ARG; }
  if (d->L > s->L || d->device != s->device || (s->nr - 1) % (d->nr - 1) != 0) {
    set_error("filter: destination needs L <= source L, the same device and a radial grid whose points are "
              "a subset of the source's");
    return CB2_ERR_ARG;
  }
  *stride = (s->nr - 1) / (d->nr - 1);
  for (int k = 0; k < d->nr; k++)
    if (std::fabs(d->h_r[k] - s->h_r[k * *stride]) > 1e-12 * std::fabs(s->h_r[k * *stride])) {
      set_error("filter: radial points of the destination are not points of the source");
      return CB2_ERR_ARG;
    }
  return 0;
}

int cb2_filter_fields(cb2_ctx *src, cb2_ctx *dst) {
  int stride = 1, rc = filter_check(src, dst, &stride);
  if (rc) return rc;
  CB2_CUDA(cudaStreamSynchronize(src->stream));
  Slots16 ss = feat_slots();
  k_filter<<<blocks((size_t)dst->nr * dst->jmax), 256, 0, dst->stream>>>(
      dst->nr, dst->jmax, src->jmax, src->L, stride, dst->d_jl, dst->d_jm, src->d_moff, src->d_f, src->fsize(),
      dst->d_f, dst->fsize(), ss, ss, 13, 0);
  CB2_CUDA(cudaGetLastError());
  return cb2_start(dst);
}

// src's five explicit nonlinear terms (curl of forces S, T; induction S, T;
// heat advection), filtered onto dst's shape: dev_out = 5 x nr x jmax
// (dst's device order, float64)
int cb2_filter_terms(cb2_ctx *src, cb2_ctx *dst, double *dev_out) {
  int stride = 1, rc = filter_check(src, dst, &stride);
  if (rc) return rc;
  if (!dev_out) return CB2_ERR_ARG;
  CB2_CUDA(cudaStreamSynchronize(src->stream));
  Slots16 so = out_slots();
  k_filter<<<blocks((size_t)dst->nr * dst->jmax), 256, 0, dst->stream>>>(
      dst->nr, dst->jmax, src->jmax, src->L, stride, dst->d_jl, dst->d_jm, src->d_moff, src->d_f, src->fsize(),
      dev_out, dst->fsize(), so, so, NO, 1);
  CB2_CUDA(cudaGetLastError());
  CB2_CUDA(cudaStreamSynchronize(dst->stream));
  return 0;
}

// raw features of ctx's state: dev_x = (nr * jmax) x 16 float32
int cb2_closure_features(cb2_ctx *c, float *dev_x) {
  if (!c || !dev_x) return CB2_ERR_ARG;
  const size_t n = c->fsize();
  k_features<<<blocks(n), 256, 0, c->stream>>>(c->nr, c->jmax, c->L, c->d_jl, c->d_jm, c->d_r, c->h_r[c->kin],
                                               c->h_r[c->kout], c->d_f, c->fsize(), feat_slots(), dev_x);
  CB2_CUDA(cudaGetLastError());
  CB2_CUDA(cudaStreamSynchronize(c->stream));
  return 0;
}

// targets: dev_y = (nr * jmax) x 5 float32 = dev_hi (cb2_filter_terms) minus
// ctx's own five nonlinear terms
int cb2_closure_targets(cb2_ctx *c, const double *dev_hi, float *dev_y) {
  if (!c || !dev_hi || !dev_y) return CB2_ERR_ARG;
  const size_t n = c->fsize();
  k_targets<<<blocks(n), 256, 0, c->stream>>>(n, dev_hi, c->d_f, c->fsize(), out_slots(), dev_y);
  CB2_CUDA(cudaGetLastError());
  CB2_CUDA(cudaStreamSynchronize(c->stream));
  return 0;
}

// attach (net != NULL) or detach the closure: every step then adds
// MLP((features - mean[k]) / std[k]) * scale[k] to the five nonlinear terms
// at the interior radial levels k.  norm (host floats) = nr x 16 means,
// nr x 16 standard deviations, nr x 5 output scales.  The network must have
// 16 inputs and 5 outputs and outlive the attachment.
int cb2_closure_attach(cb2_ctx *c, cb2_mlp *net, const float *norm) {
  if (!c) return CB2_ERR_ARG;
  if (c->graph_exec) { set_error("cb2_closure_attach: the step graph is already captured"); return CB2_ERR_STATE; }
  closure_free(*c);
  if (!net) return 0;
  if (net->F != NF || net->O != NO || !norm) {
    set_error("cb2_closure_attach: the network needs 16 inputs and 5 outputs, and norm nr x 37 floats");
    return CB2_ERR_ARG;
  }
  ClosureState *cs = new ClosureState();
  c->closure = cs;
  cs->net = net;
  net->users.push_back(cs);
  CB2_CUDA(cudaEventCreateWithFlags(&cs->read, cudaEventDisableTiming));
  cs->rows = c->fsize();
  const size_t nn = (size_t)c->nr * NF;
  std::vector<float> hn(norm, norm + 2 * nn + (size_t)c->nr * NO);
  for (size_t q = 0; q < nn; q++) hn[nn + q] = hn[nn + q] > 0.0f ? 1.0f / hn[nn + q] : 1.0f;
  CB2_CUDA(cudaMalloc(&cs->norm, hn.size() * sizeof(float)));
  CB2_CUDA(cudaMemcpyAsync(cs->norm, hn.data(), hn.size() * sizeof(float), cudaMemcpyHostToDevice, c->stream));
  CB2_CUDA(cudaMalloc(&cs->X, cs->rows * NF * sizeof(float)));
  CB2_CUDA(cudaMalloc(&cs->Xn, cs->rows * NF * sizeof(float)));
  if (int rc = mlp_reserve(net, cs->rows, false)) return rc;
  return mlp_reserve_y(net, cs->rows);
}

}  // extern "C"
