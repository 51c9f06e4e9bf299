// cb2_boundary.cu -- routine-level entry points on the reference's buffers.
//
// The reference reaches its Legendre and FFT stages through
//   sel_backward_legendre_trans / sel_forward_legendre_trans
//     (PARALLEL_src/SPH_SHELL_src/legendre_transform_select.f90:309-439):
//     spectra sp_rlm(comp + ncomp ((k-1) istep_rlm(1) + (j-1) istep_rlm(2)))
//     <-> Fourier coefficients vr_rtm(comp + ncomp ((k-1) istep_rtm(1)
//          + (l-1) istep_rtm(2) + (mp-1) istep_rtm(3)))
//     (legendre_bwd_trans_org.f90:45-209, legendre_fwd_trans_org.f90:45-169)
//   back_MHD_FFT_sel_from_recv / fwd_MHD_FFT_sel_from_recv
//     (MHD_src/sph_MHD/MHD_FFT_selector.F90:185-249): Fourier coefficients
//     <-> grid fld_rtp(inod, comp), inod = (k-1) istep_rtp(1)
//          + (l-1) istep_rtp(2) + (p-1) istep_rtp(3) + 1.
// Here the same buffers (host or device memory) go through the library's
// own layouts: the spectra into work slots of the field array (device
// m-major order), the Fourier coefficients into the Fourier rows of the
// context's precision, the grid into [comp][k][theta][phi].  The index
// permutations are the reference's rj <-> rlm and rtm <-> rtp transposes,
// done on the device.  Components are processed in chunks that fit the
// context's Fourier buffers.
#include <algorithm>
#include <cstring>
#include <memory>
#include <vector>

#include "cb2_internal.cuh"

namespace cb2 {

namespace {

bool is_device_ptr(const void *p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
}

int grow(void **buf, size_t *have, size_t need) {
  if (*have >= need) return 0;
  if (*buf) cudaFree(*buf);
  *buf = nullptr;
  *have = 0;
  CB2_CUDA(cudaMalloc(buf, need));
  *have = need;
  return 0;
}

// Device tables of a call.  jo: (j_rlm, jj) in the order of jj, the library's
// m-major index, so that consecutive entries are consecutive in the field
// slots; mo: (mp, |m|, s, -) in the order of (|m|, s), so that the two orders
// of a Fourier row follow each other; mpos: [|m|][s] -> mp (the last one the
// table lists) or -1; mq: by mp.
struct DevTab {
  const int2 *jo = nullptr;  // nidx_rlm(2)
  const int *mq = nullptr;   // nidx_rtm(3) x 2: |m|, s (0 cos / order +m, 1 sin / order -m)
  const int4 *mo = nullptr;  // nidx_rtm(3)
  const int *mpos = nullptr; // (L + 1) x 2
};

// The device tables of the last call stay while a call's own tables hold the
// same values: (l, m) of every j_rlm, m of every mp (the strides do not enter
// the tables).  Checking, sorting and uploading 65536 modes took 0.35 ms of a
// 1.6 ms call at L255; comparing the values takes about 0.02 ms.
bool same_rlm(const Ctx &c, const cb2_sph_tables *t) {
  const size_t n = 2 * (size_t)t->nidx_rlm[1];
  return c.bnd_rlm_key.size() == n &&
         std::memcmp(c.bnd_rlm_key.data(), t->idx_gl_1d_rlm_j + t->nidx_rlm[1], n * sizeof(int)) == 0;
}
bool same_rtm(const Ctx &c, const cb2_sph_tables *t) {
  const size_t n = (size_t)t->nidx_rtm[2];
  return c.bnd_rtm_key.size() == n && std::memcmp(c.bnd_rtm_key.data(), t->idx_gl_1d_rtm_m + n, n * sizeof(int)) == 0;
}

int check_tables(const Ctx &c, const cb2_sph_tables *t, bool need_rlm, bool need_rtp) {
  if (!t) { set_error("null index tables"); return CB2_ERR_ARG; }
  if (t->nidx_rtm[0] != c.nr || t->nidx_rtm[1] != c.nth || t->nidx_rtm[2] < 1 || t->nidx_rtm[2] > 2 * c.L + 1 ||
      !t->idx_gl_1d_rtm_m) {
    set_error("rtm tables: need nidx_rtm = (nr, nth, 1..2L+1) and idx_gl_1d_rtm_m");
    return CB2_ERR_ARG;
  }
  for (int q = 0; q < 3; q++)
    if (t->istep_rtm[q] < 1) { set_error("istep_rtm must be positive"); return CB2_ERR_ARG; }
  const bool known_m = same_rtm(c, t);
  for (int mp = 0; !known_m && mp < t->nidx_rtm[2]; mp++) {
    const int m = t->idx_gl_1d_rtm_m[t->nidx_rtm[2] + mp];
    if (m < -c.L || m > c.L) { set_error("idx_gl_1d_rtm_m: order outside -L..L"); return CB2_ERR_ARG; }
  }
  if (need_rlm) {
    if (t->nidx_rlm[0] != c.nr || t->nidx_rlm[1] < 1 || t->nidx_rlm[1] > c.jmax || !t->idx_gl_1d_rlm_j ||
        t->istep_rlm[0] < 1 || t->istep_rlm[1] < 1) {
      set_error("rlm tables: need nidx_rlm = (nr, 1..(L+1)^2), positive istep_rlm and idx_gl_1d_rlm_j");
      return CB2_ERR_ARG;
    }
    const int nj = t->nidx_rlm[1];
    const bool known = same_rlm(c, t);
    for (int j = 0; !known && j < nj; j++) {
      const int l = t->idx_gl_1d_rlm_j[nj + j], m = t->idx_gl_1d_rlm_j[2 * nj + j];
      if (l < 0 || l > c.L || m < -l || m > l) {
        set_error("idx_gl_1d_rlm_j: (l, m) outside the truncation");
        return CB2_ERR_ARG;
      }
    }
  }
  if (need_rtp) {
    if (t->nidx_rtp[0] != c.nr || t->nidx_rtp[1] != c.nth || t->nidx_rtp[2] != c.nph || t->istep_rtp[0] < 1 ||
        t->istep_rtp[1] < 1 || t->istep_rtp[2] < 1) {
      set_error("rtp tables: need nidx_rtp = (nr, nth, nph) and positive istep_rtp");
      return CB2_ERR_ARG;
    }
    const size_t top = (size_t)(c.nr - 1) * t->istep_rtp[0] + (size_t)(c.nth - 1) * t->istep_rtp[1] +
                       (size_t)(c.nph - 1) * t->istep_rtp[2];
    if (top >= (size_t)c.nr * c.nth * c.nph) {
      set_error("istep_rtp: index beyond nnod_rtp = nr nth nph");
      return CB2_ERR_ARG;
    }
  }
  return 0;
}

// largest index + 1 of the rlm / rtm buffers for ncomp components
size_t rlm_extent(const cb2_sph_tables *t, int ncomp) {
  return (size_t)ncomp * ((size_t)(t->nidx_rlm[0] - 1) * t->istep_rlm[0] +
                          (size_t)(t->nidx_rlm[1] - 1) * t->istep_rlm[1] + 1);
}
size_t rtm_extent(const cb2_sph_tables *t, int ncomp) {
  return (size_t)ncomp * ((size_t)(t->nidx_rtm[0] - 1) * t->istep_rtm[0] +
                          (size_t)(t->nidx_rtm[1] - 1) * t->istep_rtm[1] +
                          (size_t)(t->nidx_rtm[2] - 1) * t->istep_rtm[2] + 1);
}

int jj_host(const Ctx &c, int l, int m) {
  const int am = std::abs(m);
  return c.h_moff[am] + ((m < 0) ? (c.L + 1 - am) : 0) + (l - am);
}

// both device tables, one allocation of the largest the checks let through
int tables_alloc(Ctx &c) {
  if (c.d_bnd_tab) return 0;
  const size_t M1 = c.L + 1, rlm = (2 * (size_t)c.jmax + 3) / 4 * 4, rtm = 6 * (2 * M1 - 1) + 2 * M1;
  CB2_CUDA(cudaMalloc(&c.d_bnd_tab, (rlm + rtm) * sizeof(int)));
  c.d_bnd_mtab = c.d_bnd_tab + rlm;
  return 0;
}

int upload_rlm(Ctx &c, const cb2_sph_tables *t) {
  const int nj = t->nidx_rlm[1];
  const int *lm = t->idx_gl_1d_rlm_j + nj;   // l of every j, then m
  // Every mode once: the entry of jj is its place in the table.  A first call
  // pays for this on the host, 0.1 - 0.5 ms at L255; the sort below, with its
  // lists, takes 0.3 - 1.0 ms.
  std::unique_ptr<int[]> pairs(new int[2 * (size_t)nj]);
  bool once = nj == c.jmax;
  if (once) {
    std::memset(pairs.get(), 0xff, 2 * (size_t)nj * sizeof(int));
    for (int j = 0; j < nj && once; j++) {
      const int jj = jj_host(c, lm[j], lm[nj + j]);
      once = pairs[2 * (size_t)jj] < 0;
      pairs[2 * (size_t)jj] = j;
      pairs[2 * (size_t)jj + 1] = jj;
    }
  }
  if (!once) {
    // entries of equal key keep the table's order (a table may list a mode twice)
    std::vector<int> head(c.jmax, -1), next(nj);
    for (int j = nj - 1; j >= 0; j--) {
      const int jj = jj_host(c, lm[j], lm[nj + j]);
      next[j] = head[jj];
      head[jj] = j;
    }
    size_t at = 0;
    for (int jj = 0; jj < c.jmax; jj++)
      for (int j = head[jj]; j >= 0; j = next[j]) { pairs[at++] = j; pairs[at++] = jj; }
  }
  c.bnd_rlm_key.clear();   // no key while the device table changes
  if (int rc = tables_alloc(c)) return rc;
  CB2_CUDA(cudaMemcpyAsync(c.d_bnd_tab, pairs.get(), 2 * (size_t)nj * sizeof(int), cudaMemcpyHostToDevice, c.stream));
  c.bnd_rlm_key.assign(lm, lm + 2 * (size_t)nj);
  c.bnd_rlm_full = once;
  return 0;
}

// [mo: nm x 4][mq: nm x 2][mpos: (L + 1) x 2]
int upload_rtm(Ctx &c, const cb2_sph_tables *t) {
  const int nm = t->nidx_rtm[2], M1 = c.L + 1;
  const int *om = t->idx_gl_1d_rtm_m + nm;
  std::vector<int> head(2 * M1, -1), next(nm), mpos(2 * (size_t)M1, -1), h;
  for (int mp = nm - 1; mp >= 0; mp--) {
    const int key = 2 * std::abs(om[mp]) + (om[mp] < 0);
    next[mp] = head[key];
    head[key] = mp;
    if (mpos[key] < 0) mpos[key] = mp;
  }
  h.reserve(6 * (size_t)nm + mpos.size());
  for (int key = 0; key < 2 * M1; key++)
    for (int mp = head[key]; mp >= 0; mp = next[mp]) {
      h.push_back(mp); h.push_back(key >> 1); h.push_back(key & 1); h.push_back(0);
    }
  for (int mp = 0; mp < nm; mp++) { h.push_back(std::abs(om[mp])); h.push_back((om[mp] < 0) ? 1 : 0); }
  h.insert(h.end(), mpos.begin(), mpos.end());
  c.bnd_rtm_key.clear();
  if (int rc = tables_alloc(c)) return rc;
  CB2_CUDA(cudaMemcpyAsync(c.d_bnd_mtab, h.data(), h.size() * sizeof(int), cudaMemcpyHostToDevice, c.stream));
  c.bnd_rtm_key.assign(om, om + nm);
  return 0;
}

int device_tables(Ctx &c, const cb2_sph_tables *t, bool rlm, DevTab *d) {
  if (rlm && !same_rlm(c, t))
    if (int rc = upload_rlm(c, t)) return rc;
  if (!same_rtm(c, t))
    if (int rc = upload_rtm(c, t)) return rc;
  const int nm = t->nidx_rtm[2];
  d->jo = reinterpret_cast<const int2 *>(c.d_bnd_tab);
  d->mo = reinterpret_cast<const int4 *>(c.d_bnd_mtab);
  d->mq = c.d_bnd_mtab + 4 * (size_t)nm;
  d->mpos = d->mq + 2 * (size_t)nm;
  return 0;
}

// nidx x istep cover 0 .. product - 1 without a gap or an overlap
bool dense3(const int *n, const int *st) {
  int q[3] = {0, 1, 2};
  std::sort(q, q + 3, [&](int a, int b) { return st[a] != st[b] ? st[a] < st[b] : n[a] < n[b]; });
  long long want = 1;
  for (int i = 0; i < 3; i++) {
    if (n[q[i]] > 1 && st[q[i]] != want) return false;
    want *= n[q[i]];
  }
  return true;
}

// the caller's buffer on the device: itself, or a copy in staging buffer `which`
int device_in(Ctx &c, const double *p, size_t n, int which, const double **out) {
  if (is_device_ptr(p)) { *out = p; return 0; }
  double **b = which ? &c.d_bnd_b : &c.d_bnd_a;
  size_t *have = which ? &c.bnd_b_bytes : &c.bnd_a_bytes;
  if (int rc = grow((void **)b, have, n * sizeof(double))) return rc;
  CB2_CUDA(cudaMemcpyAsync(*b, p, n * sizeof(double), cudaMemcpyHostToDevice, c.stream));
  *out = *b;
  return 0;
}

int device_out(Ctx &c, double *p, size_t n, int which, double **out) {
  if (is_device_ptr(p)) { *out = p; return 0; }
  double **b = which ? &c.d_bnd_b : &c.d_bnd_a;
  size_t *have = which ? &c.bnd_b_bytes : &c.bnd_a_bytes;
  if (int rc = grow((void **)b, have, n * sizeof(double))) return rc;
  *out = *b;
  return 0;
}

// result to the caller's buffer; the stream drains here unless the caller
// reads the status word next, which waits for it anyway
int finish_out(Ctx &c, double *host, const double *dev, size_t n, bool drain = true) {
  if (host != dev) CB2_CUDA(cudaMemcpyAsync(host, dev, n * sizeof(double), cudaMemcpyDeviceToHost, c.stream));
  if (drain) CB2_CUDA(cudaStreamSynchronize(c.stream));
  return 0;
}

// one chunk of components: comp0.. of the caller's numbering, the first nv
// of them vectors (3 components each), then ns scalars
struct Chunk {
  int comp0, nv, ns;
  int nc() const { return 3 * nv + ns; }
};

// chunks that fit the Fourier buffers: float64 rows hold 13 components;
// the mixed transforms take at most 4 vectors and 8 fields with 6 nv + 2 ns
// <= 26 floats per radial level
std::vector<Chunk> chunks(int prec, int nvec, int nscal) {
  std::vector<Chunk> out;
  int comp = 0, v = 0, s = 0;
  while (v < nvec || s < nscal) {
    Chunk ch{comp, 0, 0};
    ch.nv = std::min(4, nvec - v);
    int room = (prec == CB2_PREC_FP64) ? 13 - 3 * ch.nv : std::min(8 - ch.nv, (26 - 6 * ch.nv) / 2);
    ch.ns = (ch.nv == nvec - v) ? std::min(room, nscal - s) : 0;
    v += ch.nv;
    s += ch.ns;
    comp += ch.nc();
    out.push_back(ch);
  }
  return out;
}

constexpr int kBnd = 256;

// rlm buffer <-> work slots (device order).  The slots run along jj, the
// rlm buffer along the nq components of a mode (a run of 8 nq bytes): a block
// takes JT modes of consecutive jj at JK radial levels and turns them round
// in shared memory, so both sides move in whole runs: bound by the runs'
// partial sectors.  At L255 / Nr65 / 11 components 150 us inwards (5.0 TB/s);
// a thread per mode, whose 8-byte slot writes scattered over the orders, took
// 482 us.  Outwards at L170 / Nr49 / 12 components 73 us against 176.
constexpr int JT = 64;
constexpr int JK = 4;   // radial levels a block: that many independent loads a thread and mode

template <bool TO_SLOTS>
__global__ void __launch_bounds__(kBnd)
k_rlm_slots(int nj, int nr, int ncomp, int is0, int is1, int comp0, FastDiv nq, int slot0,
            const int2 *__restrict__ jo, double *__restrict__ rlm, double *__restrict__ f, size_t fs, int jmax) {
  extern __shared__ double tile[];   // [JK][JT][nq | 1]
  __shared__ int2 ent[JT];
  const int i0 = blockIdx.x * JT, k0 = blockIdx.y * JK, nt = min(JT, nj - i0), nk = min(JK, nr - k0);
  const int n = (int)nq.n, pitch = n | 1, kp = JT * pitch;
  if (threadIdx.x < nt) ent[threadIdx.x] = jo[i0 + threadIdx.x];
  __syncthreads();
  const size_t rk = (size_t)ncomp * is0;
  double *r0 = rlm + (size_t)k0 * rk + comp0;
  double *f0 = f + (size_t)slot0 * fs + (size_t)k0 * jmax;
  auto along_rlm = [&](bool load) {
    for (int e = threadIdx.x; e < nt * n; e += kBnd) {
      const int i = nq.div(e), q = e - i * n;
      double *g = r0 + (size_t)ncomp * ent[i].x * is1 + q, *t = tile + i * pitch + q;
#pragma unroll
      for (int k = 0; k < JK; k++)
        if (k < nk) {
          if (load) t[k * kp] = __ldg(g + k * rk);
          else g[k * rk] = t[k * kp];
        }
    }
  };
  auto along_slots = [&](bool load) {
    for (int e = threadIdx.x; e < JT * n; e += kBnd) {
      const int q = e / JT, i = e % JT;
      if (i >= nt) continue;
      double *g = f0 + (size_t)q * fs + ent[i].y, *t = tile + i * pitch + q;
#pragma unroll
      for (int k = 0; k < JK; k++)
        if (k < nk) {
          if (load) t[k * kp] = __ldg(g + (size_t)k * jmax);
          else g[(size_t)k * jmax] = t[k * kp];
        }
    }
  };
  if (TO_SLOTS) along_rlm(true);
  else along_slots(true);
  __syncthreads();
  if (TO_SLOTS) along_slots(false);
  else along_rlm(false);
}

// Order-major Fourier rows <-> rtm buffer where the radius runs faster than
// the order (istep_rtm(1) <= istep_rtm(3), the reference's own order): a
// block takes one order at RTH colatitudes outwards (one inwards), the lanes
// along the buffer's (k, component) runs.  One thread per (theta, k) and order with its
// components in a loop (k_four_to_rtm / k_rtm_to_four, which stay for the
// other stride orders) wrote 8 bytes of every line at a time: 1112 us
// outwards at L255 / Nr65 / 11 components, now 295 us (5.6 TB/s); 323 us
// inwards at L170 / Nr49 / 12, now 140 us; float64 at L106 / Nr41 / 11 inwards
// 264 us, now 54.  Bound by HBM.
struct CompOff {
  int off[13];     // element offset of component c (s = 0) within its block's radial level
  int inD;         // bit c: component c sits in the D block
};

constexpr int RTH = 8;   // colatitudes a block: that many independent loads a thread

template <typename T>
__global__ void __launch_bounds__(kBnd)
k_rows_to_rtm(MLayoutT<T> ml, CompOff co, FastDiv nc, int ncomp, int is0, int is1, int is2, int comp0,
              const int4 *__restrict__ mo, double *__restrict__ WS) {
  __shared__ int off[13];
  const int4 me = mo[blockIdx.x];   // mp, |m|, s
  const int th0 = blockIdx.y * RTH, nt = min(RTH, ml.nth - th0), n = (int)nc.n;
  if (threadIdx.x < 13) off[threadIdx.x] = co.off[threadIdx.x];
  __syncthreads();
  const T *P = ml.P + ((size_t)me.y * ml.nth + th0) * ml.sP() + me.z;
  const T *D = ml.D + ((size_t)me.y * ml.nth + th0) * ml.sD() + me.z;
  const int rP = ml.rpP(), rD = ml.rpD();
  double *w = WS + (size_t)ncomp * ((size_t)th0 * is1 + (size_t)me.x * is2) + comp0;
  const size_t wt = (size_t)ncomp * is1;
  for (int e = threadIdx.x; e < ml.nr * n; e += kBnd) {
    const int k = nc.div(e), c = e - k * n;
    const bool d = co.inD >> c & 1;
    const T *src = d ? D + k * rD + off[c] : P + k * rP + off[c];
    const size_t st = d ? ml.sD() : ml.sP();
    double *o = w + (size_t)ncomp * k * is0 + c;
    T v[RTH];
#pragma unroll
    for (int i = 0; i < RTH; i++) v[i] = (i < nt) ? __ldg(src + i * st) : (T)0;
#pragma unroll
    for (int i = 0; i < RTH; i++)
      if (i < nt) o[i * wt] = (double)v[i];
  }
}

// every element of the order's rows, both signs: an order the table does not
// list is zero, as are the sine part of m = 0 and the padding
template <typename T>
__global__ void __launch_bounds__(kBnd)
k_rtm_to_rows(MLayoutT<T> ml, int ncomp, int is0, int is1, int is2, int comp0, FastDiv rP, FastDiv rD,
              const int *__restrict__ mpos, const double *__restrict__ WR) {
  const int m = blockIdx.x, th = blockIdx.y, nr = ml.nr, nv = ml.nvec;
  const int mp0 = mpos[2 * m], mp1 = (m > 0) ? mpos[2 * m + 1] : -1;
  const double *w0 = WR + (size_t)ncomp * ((size_t)th * is1 + (size_t)max(mp0, 0) * is2) + comp0;
  const double *w1 = WR + (size_t)ncomp * ((size_t)th * is1 + (size_t)max(mp1, 0) * is2) + comp0;
  const size_t ks = (size_t)ncomp * is0;
  T *P = ml.P + ((size_t)m * ml.nth + th) * ml.sP();
  const int eP = nr * (int)rP.n, eP4 = (int)ml.sP(), eD = nr * (int)rD.n, eD4 = (int)ml.sD();
  for (int e = threadIdx.x; e < eP4; e += kBnd) {
    const int k = rP.div(e), x = e - k * (int)rP.n, fl = x >> 1, c = (fl < nv) ? 3 * fl : 2 * nv + fl;
    T v = (T)0;
    if (e < eP && ((x & 1) ? mp1 : mp0) >= 0) v = (T)__ldg(((x & 1) ? w1 : w0) + k * ks + c);
    P[e] = v;
  }
  if (nv == 0) return;
  T *D = ml.D + ((size_t)m * ml.nth + th) * ml.sD();
  for (int e = threadIdx.x; e < eD4; e += kBnd) {
    const int k = rD.div(e), x = e - k * (int)rD.n, c = 3 * (x >> 2) + 1 + ((x & 3) >> 1);
    T v = (T)0;
    if (e < eD && ((x & 1) ? mp1 : mp0) >= 0) v = (T)__ldg(((x & 1) ? w1 : w0) + k * ks + c);
    D[e] = v;
  }
}

// Fourier rows of the context, in its precision: one thread per (theta, k) and
// order with the components in a loop, for the stride orders the row kernels
// above do not take
struct FourView {
  int nc = 0;
  bool f64 = false;
  MLayout ml;
  MLayout64 md;
  __device__ double get(int m, int th, int k, int c, int s) const {
    return f64 ? *md.at(m, th, k, c, s) : (double)*ml.at(m, th, k, c, s);
  }
  __device__ void put(int m, int th, int k, int c, int s, double v) const {
    if (f64) *md.at(m, th, k, c, s) = v;
    else *ml.at(m, th, k, c, s) = (float)v;
  }
};

__global__ void k_four_to_rtm(FourView fv, int nth, int nr, int ncomp, int is0, int is1, int is2, int comp0,
                              const int *mq, double *WS) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, mp = blockIdx.y;
  if (i >= nth * nr) return;
  const int th = i / nr, k = i - th * nr;
  const int m = mq[2 * mp], s = mq[2 * mp + 1];
  const size_t dst = (size_t)ncomp * ((size_t)k * is0 + (size_t)th * is1 + (size_t)mp * is2) + comp0;
  for (int q = 0; q < fv.nc; q++) WS[dst + q] = (m == 0 && s == 1) ? 0.0 : fv.get(m, th, k, q, s);
}

// rows of orders the table does not list stay zero (cleared before)
__global__ void k_rtm_to_four(FourView fv, int nth, int nr, int ncomp, int is0, int is1, int is2, int comp0,
                              const int *mq, const double *WR) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, mp = blockIdx.y;
  if (i >= nth * nr) return;
  const int th = i / nr, k = i - th * nr;
  const int m = mq[2 * mp], s = mq[2 * mp + 1];
  const size_t src = (size_t)ncomp * ((size_t)k * is0 + (size_t)th * is1 + (size_t)mp * is2) + comp0;
  for (int q = 0; q < fv.nc; q++) fv.put(m, th, k, q, s, (m == 0 && s == 1) ? 0.0 : WR[src + q]);
}

// grid [c][k][theta][phi] <-> fld_rtp(inod, comp), one thread per grid point
__global__ void k_grid_to_rtp(int nc, int nr, int nth, int nph, int is0, int is1, int is2, int comp0,
                              size_t nnod, const double *grid, double *fld) {
  const size_t n = (size_t)nr * nth * nph;
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int p = (int)(i % nph);
  const size_t t = i / nph;
  const int th = (int)(t % nth), k = (int)(t / nth);
  const size_t inod = (size_t)k * is0 + (size_t)th * is1 + (size_t)p * is2;
  for (int q = 0; q < nc; q++) fld[inod + nnod * (comp0 + q)] = grid[(size_t)q * n + i];
}

__global__ void k_rtp_to_grid(int nc, int nr, int nth, int nph, int is0, int is1, int is2, int comp0,
                              size_t nnod, const double *fld, double *grid) {
  const size_t n = (size_t)nr * nth * nph;
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int p = (int)(i % nph);
  const size_t t = i / nph;
  const int th = (int)(t % nth), k = (int)(t / nth);
  const size_t inod = (size_t)k * is0 + (size_t)th * is1 + (size_t)p * is2;
  for (int q = 0; q < nc; q++) grid[(size_t)q * n + i] = fld[inod + nnod * (comp0 + q)];
}

FourView four_view(Ctx &c, int nv, int ns, void *buf = nullptr) {
  if (!buf) buf = c.d_four;
  FourView fv;
  fv.nc = 3 * nv + ns;
  fv.f64 = c.prec == CB2_PREC_FP64;
  if (fv.f64) fv.md = mlayout64(c, buf, nv, ns);
  else fv.ml = mlayout(c, buf, nv, ns);
  return fv;
}

size_t four_bytes(const Ctx &c) {
  return (c.prec == CB2_PREC_FP64) ? (size_t)c.nth * c.nr * c.NS * 13 * sizeof(double)
                                   : mlayout_floats(c) * sizeof(float);
}

// the row kernels of one chunk, where the radius runs faster than the order;
// false: the strides are another kind, nothing done
template <typename T>
bool rows_out_k(Ctx &c, const cb2_sph_tables *t, const DevTab &dt, const MLayoutT<T> &ml, int ncomp, int comp0,
                double *dWS) {
  const int *is = t->istep_rtm, nm = t->nidx_rtm[2], nc = 3 * ml.nvec + ml.nscal;
  if (is[0] > is[2] || c.nr * nc >= (1 << 16) || c.nth >= (1 << 16)) return false;
  CompOff co{};
  for (int q = 0; q < nc; q++) {
    const int v = q / 3, cc = q - 3 * v;
    if (q >= 3 * ml.nvec) co.off[q] = 2 * (ml.nvec + q - 3 * ml.nvec);
    else if (cc == 0) co.off[q] = 2 * v;
    else { co.off[q] = 4 * v + 2 * (cc - 1); co.inD |= 1 << q; }
  }
  k_rows_to_rtm<T><<<dim3(nm, cdiv(c.nth, RTH)), kBnd, 0, c.stream>>>(ml, co, FastDiv(nc), ncomp, is[0], is[1], is[2],
                                                                      comp0, dt.mo, dWS);
  return true;
}

template <typename T>
bool rows_in_k(Ctx &c, const cb2_sph_tables *t, const DevTab &dt, const MLayoutT<T> &ml, int ncomp, int comp0,
               const double *dWR) {
  const int *is = t->istep_rtm;
  if (is[0] > is[2] || ml.sP() >= (1u << 16) || ml.sD() >= (1u << 16) || c.nth >= (1 << 16)) return false;
  k_rtm_to_rows<T><<<dim3(c.L + 1, c.nth), kBnd, 0, c.stream>>>(ml, ncomp, is[0], is[1], is[2], comp0,
                                                                FastDiv(ml.rpP()), FastDiv(std::max(1, ml.rpD())),
                                                                dt.mpos, dWR);
  return true;
}

// Fourier rows -> rtm buffer of one chunk
void rows_out(Ctx &c, const cb2_sph_tables *t, const DevTab &dt, const FourView &fv, int ncomp, int comp0, double *dWS) {
  if (fv.f64 ? rows_out_k(c, t, dt, fv.md, ncomp, comp0, dWS) : rows_out_k(c, t, dt, fv.ml, ncomp, comp0, dWS)) return;
  const int *is = t->istep_rtm;
  k_four_to_rtm<<<dim3(cdiv((long)c.nth * c.nr, kBnd), t->nidx_rtm[2]), kBnd, 0, c.stream>>>(
      fv, c.nth, c.nr, ncomp, is[0], is[1], is[2], comp0, dt.mq, dWS);
}

// rtm buffer -> every element of the Fourier rows of one chunk
int rows_in(Ctx &c, const cb2_sph_tables *t, const DevTab &dt, const FourView &fv, int ncomp, int comp0,
            const double *dWR) {
  if (fv.f64 ? rows_in_k(c, t, dt, fv.md, ncomp, comp0, dWR) : rows_in_k(c, t, dt, fv.ml, ncomp, comp0, dWR)) return 0;
  const int *is = t->istep_rtm;
  CB2_CUDA(cudaMemsetAsync(fv.f64 ? (void *)fv.md.P : (void *)fv.ml.P, 0, four_bytes(c), c.stream));
  k_rtm_to_four<<<dim3(cdiv((long)c.nth * c.nr, kBnd), t->nidx_rtm[2]), kBnd, 0, c.stream>>>(
      fv, c.nth, c.nr, ncomp, is[0], is[1], is[2], comp0, dt.mq, dWR);
  return 0;
}

// clears what a call will not write of an rtm (rlm) buffer of n values: the
// whole buffer, or only its tail where the tables cover the rest densely
int clear_rtm(Ctx &c, const cb2_sph_tables *t, int ncomp, int nwritten, size_t n, double *dWS) {
  const size_t ext = rtm_extent(t, ncomp);
  const size_t from = (ncomp == nwritten && dense3(t->nidx_rtm, t->istep_rtm)) ? ext : 0;
  if (from < n) CB2_CUDA(cudaMemsetAsync(dWS + from, 0, (n - from) * sizeof(double), c.stream));
  return 0;
}
int clear_rlm(Ctx &c, const cb2_sph_tables *t, int ncomp, int nwritten, size_t n, double *dWS) {
  const size_t ext = rlm_extent(t, ncomp);
  const int nn[3] = {t->nidx_rlm[0], t->nidx_rlm[1], 1}, st[3] = {t->istep_rlm[0], t->istep_rlm[1], 1 << 30};
  const size_t from = (ncomp == nwritten && dense3(nn, st)) ? ext : 0;
  if (from < n) CB2_CUDA(cudaMemsetAsync(dWS + from, 0, (n - from) * sizeof(double), c.stream));
  return 0;
}

int leg_args_ok(const Ctx &c, int ncomp, int nvec, int nscal) {
  if (nvec < 0 || nscal < 0 || nvec + nscal == 0 || ncomp < 3 * nvec + nscal) {
    set_error("Legendre transform: need nvector, nscalar >= 0, at least one field, ncomp >= 3 nvector + nscalar");
    return CB2_ERR_ARG;
  }
  if (3 * nvec + nscal > NSLOT - MADV) {
    set_error("Legendre transform: at most 38 components per call");
    return CB2_ERR_ARG;
  }
  return 0;
}

}  // namespace

}  // namespace cb2

using namespace cb2;

extern "C" {

int cb2_leg_bwd(cb2_ctx *c, const cb2_sph_tables *t, int ncomp, int nvector, int nscalar, size_t n_WR,
                size_t n_WS, const double *WR, double *WS) {
  if (!c || !WR || !WS) { set_error("null argument"); return CB2_ERR_ARG; }
  if (int rc = leg_args_ok(*c, ncomp, nvector, nscalar)) return rc;
  if (int rc = check_tables(*c, t, true, false)) return rc;
  if (n_WR < rlm_extent(t, ncomp) || n_WS < rtm_extent(t, ncomp)) {
    set_error("cb2_leg_bwd: n_WR or n_WS smaller than the tables' extent");
    return CB2_ERR_ARG;
  }
  DevTab dt;
  const double *dWR;
  double *dWS;
  int rc;
  if ((rc = device_tables(*c, t, true, &dt)) || (rc = device_in(*c, WR, n_WR, 0, &dWR)) ||
      (rc = device_out(*c, WS, n_WS, 1, &dWS)))
    return rc;
  // the callee clears WS, as the reference's backward transforms do
  if ((rc = clear_rtm(*c, t, ncomp, 3 * nvector + nscalar, n_WS, dWS))) return rc;
  const int nj = t->nidx_rlm[1];
  for (const Chunk &ch : chunks(c->prec, nvector, nscalar)) {
    const int nc = ch.nc();
    // vectors occupy three slots each from MADV, scalars follow
    int slots[13];
    for (int g = 0; g < ch.nv; g++) slots[g] = MADV + 3 * g;
    for (int s = 0; s < ch.ns; s++) slots[ch.nv + s] = MADV + 3 * ch.nv + s;
    // modes the table leaves out are zero (one that lists a mode twice leaves
    // another out, however long it is)
    if (!c->bnd_rlm_full)
      CB2_CUDA(cudaMemsetAsync(c->fld(MADV), 0, (size_t)nc * c->fsize() * sizeof(double), c->stream));
    k_rlm_slots<true><<<dim3(cdiv(nj, JT), cdiv(c->nr, JK)), kBnd, JK * JT * (nc | 1) * sizeof(double), c->stream>>>(
        nj, c->nr, ncomp, t->istep_rlm[0], t->istep_rlm[1], ch.comp0, FastDiv(nc), MADV, dt.jo, const_cast<double *>(dWR),
        c->d_f, c->fsize(), c->jmax);
    if (c->prec == CB2_PREC_FP64) {
      leg_bwd_f64(*c, slots, mlayout64(*c, c->d_four, ch.nv, ch.ns));
    } else {
      const MLayout l = mlayout(*c, c->d_four, ch.nv, ch.ns);
      if ((rc = leg_bwd_mixed(*c, slots, l))) return rc;
    }
    rows_out(*c, t, dt, four_view(*c, ch.nv, ch.ns), ncomp, ch.comp0, dWS);
  }
  CB2_CUDA(cudaGetLastError());
  if ((rc = finish_out(*c, WS, dWS, n_WS, false))) return rc;
  return check_status(*c);
}

int cb2_leg_fwd(cb2_ctx *c, const cb2_sph_tables *t, int ncomp, int nvector, int nscalar, size_t n_WR,
                size_t n_WS, const double *WR, double *WS) {
  if (!c || !WR || !WS) { set_error("null argument"); return CB2_ERR_ARG; }
  if (int rc = leg_args_ok(*c, ncomp, nvector, nscalar)) return rc;
  if (int rc = check_tables(*c, t, true, false)) return rc;
  if (n_WR < rtm_extent(t, ncomp) || n_WS < rlm_extent(t, ncomp)) {
    set_error("cb2_leg_fwd: n_WR or n_WS smaller than the tables' extent");
    return CB2_ERR_ARG;
  }
  DevTab dt;
  const double *dWR;
  double *dWS;
  int rc;
  if ((rc = device_tables(*c, t, true, &dt)) || (rc = device_in(*c, WR, n_WR, 0, &dWR)) ||
      (rc = device_out(*c, WS, n_WS, 1, &dWS)))
    return rc;
  if ((rc = clear_rlm(*c, t, ncomp, 3 * nvector + nscalar, n_WS, dWS))) return rc;
  const int nj = t->nidx_rlm[1];
  for (const Chunk &ch : chunks(c->prec, nvector, nscalar)) {
    const int nc = ch.nc();
    int slots[13];
    for (int g = 0; g < ch.nv; g++) slots[g] = MADV + 3 * g;
    for (int s = 0; s < ch.ns; s++) slots[ch.nv + s] = MADV + 3 * ch.nv + s;
    if ((rc = rows_in(*c, t, dt, four_view(*c, ch.nv, ch.ns), ncomp, ch.comp0, dWR))) return rc;
    if (c->prec == CB2_PREC_FP64) {
      leg_fwd_f64(*c, mlayout64(*c, c->d_four, ch.nv, ch.ns), slots);
    } else {
      const MLayout l = mlayout(*c, c->d_four, ch.nv, ch.ns);
      if ((rc = leg_fwd_mixed(*c, l, slots))) return rc;
    }
    k_rlm_slots<false><<<dim3(cdiv(nj, JT), cdiv(c->nr, JK)), kBnd, JK * JT * (nc | 1) * sizeof(double), c->stream>>>(
        nj, c->nr, ncomp, t->istep_rlm[0], t->istep_rlm[1], ch.comp0, FastDiv(nc), MADV, dt.jo, dWS, c->d_f, c->fsize(),
        c->jmax);
  }
  CB2_CUDA(cudaGetLastError());
  if ((rc = finish_out(*c, WS, dWS, n_WS, false))) return rc;
  return check_status(*c);
}

int cb2_fft_bwd(cb2_ctx *c, const cb2_sph_tables *t, int ncomp, size_t n_WR, const double *WR, double *fld_rtp) {
  if (!c || !WR || !fld_rtp || ncomp < 1) { set_error("null argument or ncomp < 1"); return CB2_ERR_ARG; }
  if (int rc = check_tables(*c, t, false, true)) return rc;
  if (n_WR < rtm_extent(t, ncomp)) { set_error("cb2_fft_bwd: n_WR smaller than the tables' extent"); return CB2_ERR_ARG; }
  const size_t nnod = (size_t)c->nr * c->nth * c->nph, nout = nnod * ncomp;
  DevTab dt;
  const double *dWR;
  double *dF;
  int rc;
  if ((rc = device_tables(*c, t, false, &dt)) || (rc = device_in(*c, WR, n_WR, 0, &dWR)) ||
      (rc = device_out(*c, fld_rtp, nout, 1, &dF)))
    return rc;
  if ((rc = grow((void **)&c->d_bnd_grid, &c->bnd_grid_bytes, 13 * nnod * sizeof(double)))) return rc;
  for (int c0 = 0; c0 < ncomp; c0 += 13) {
    const int nc = std::min(13, ncomp - c0);
    FourView fv = four_view(*c, 0, nc);
    if ((rc = rows_in(*c, t, dt, fv, ncomp, c0, dWR))) return rc;
    if (fv.f64) fft_backward_grid<double>(*c, fv.md, c->d_bnd_grid);
    else fft_backward_grid<float>(*c, fv.ml, c->d_bnd_grid);
    k_grid_to_rtp<<<cdiv((long)nnod, kBnd), kBnd, 0, c->stream>>>(nc, c->nr, c->nth, c->nph, t->istep_rtp[0],
                                                                  t->istep_rtp[1], t->istep_rtp[2], c0, nnod,
                                                                  c->d_bnd_grid, dF);
  }
  CB2_CUDA(cudaGetLastError());
  return finish_out(*c, fld_rtp, dF, nout);
}

int cb2_fft_products(cb2_ctx *c, const cb2_sph_tables *t, size_t n_WR, const double *WR, size_t n_WS,
                     double *WS) {
  if (!c || !WR || !WS) { set_error("null argument"); return CB2_ERR_ARG; }
  if (int rc = check_tables(*c, t, false, false)) return rc;
  if (n_WR < rtm_extent(t, 13) || n_WS < rtm_extent(t, 12)) {
    set_error("cb2_fft_products: n_WR (13 components) or n_WS (12) smaller than the tables' extent");
    return CB2_ERR_ARG;
  }
  DevTab dt;
  const double *dWR;
  double *dWS;
  int rc;
  if ((rc = device_tables(*c, t, false, &dt)) || (rc = device_in(*c, WR, n_WR, 0, &dWR)) ||
      (rc = device_out(*c, WS, n_WS, 1, &dWS)))
    return rc;
  if ((rc = clear_rtm(*c, t, 12, 12, n_WS, dWS))) return rc;
  const FourView fin = four_view(*c, 4, 1), fout = four_view(*c, 4, 0, c->d_four2);
  if ((rc = rows_in(*c, t, dt, fin, 13, 0, dWR))) return rc;
  if (fin.f64) fft_products64(*c, fin.md, fout.md);
  else fft_products_m(*c, fin.ml, fout.ml);
  rows_out(*c, t, dt, fout, 12, 0, dWS);
  CB2_CUDA(cudaGetLastError());
  return finish_out(*c, WS, dWS, n_WS);
}

int cb2_fft_fwd(cb2_ctx *c, const cb2_sph_tables *t, int ncomp, const double *frc_rtp, size_t n_WS, double *WS) {
  if (!c || !WS || !frc_rtp || ncomp < 1) { set_error("null argument or ncomp < 1"); return CB2_ERR_ARG; }
  if (int rc = check_tables(*c, t, false, true)) return rc;
  if (n_WS < rtm_extent(t, ncomp)) { set_error("cb2_fft_fwd: n_WS smaller than the tables' extent"); return CB2_ERR_ARG; }
  const size_t nnod = (size_t)c->nr * c->nth * c->nph, nin = nnod * ncomp;
  DevTab dt;
  const double *dF;
  double *dWS;
  int rc;
  if ((rc = device_tables(*c, t, false, &dt)) || (rc = device_in(*c, frc_rtp, nin, 0, &dF)) ||
      (rc = device_out(*c, WS, n_WS, 1, &dWS)))
    return rc;
  if ((rc = grow((void **)&c->d_bnd_grid, &c->bnd_grid_bytes, 13 * nnod * sizeof(double)))) return rc;
  if ((rc = clear_rtm(*c, t, ncomp, ncomp, n_WS, dWS))) return rc;
  for (int c0 = 0; c0 < ncomp; c0 += 13) {
    const int nc = std::min(13, ncomp - c0);
    k_rtp_to_grid<<<cdiv((long)nnod, kBnd), kBnd, 0, c->stream>>>(nc, c->nr, c->nth, c->nph, t->istep_rtp[0],
                                                                  t->istep_rtp[1], t->istep_rtp[2], c0, nnod, dF,
                                                                  c->d_bnd_grid);
    FourView fv = four_view(*c, 0, nc);
    if (fv.f64) fft_forward_grid<double>(*c, c->d_bnd_grid, fv.md);
    else fft_forward_grid<float>(*c, c->d_bnd_grid, fv.ml);
    rows_out(*c, t, dt, fv, ncomp, c0, dWS);
  }
  CB2_CUDA(cudaGetLastError());
  return finish_out(*c, WS, dWS, n_WS);
}

}  // extern "C"
