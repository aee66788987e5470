// ccp_kspace_fixed.cu -- reciprocal-space Ewald sum (kspace_ewald, ewald.f90:754-1173) for
// callers that cannot let the library allocate device memory.
//
// Same kernels as the context form (k_krows.cu, k_kspace.cu mode 0), but every temporary -- k-vector
// list, structure factors, per-site phase tables, packed positions, compact forces and the
// energy accumulators -- is carved out of one file-scope device array of fixed size
// (kFixedScratchBytes).  The entry point allocates no device or host memory on its success
// path and never synchronises: all work is enqueued on the caller's stream.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <mutex>
#include <string>

#include "ccp_device.cuh"
#include "ccp_internal.h"

using namespace ccp;

namespace {

constexpr size_t kFixedScratchBytes = size_t(16) << 20;  // 16 MiB per device
constexpr int kMaxDevices = 64;

}  // namespace

// The scratch itself: one array per device that loads this library, kept until exit.  Host
// code must not pass its name to a kernel (that is a host-side stand-in); the device address
// comes from cudaGetSymbolAddress below.
static __device__ __align__(256) unsigned char g_kspace_scratch[kFixedScratchBytes];

namespace {

std::mutex g_addr_mu;
unsigned char *g_addr[kMaxDevices] = {};

size_t up256(size_t b) { return (b + 255) & ~size_t(255); }

// Half-space k-vectors inside the sphere l^2+m^2+n^2 <= min(kmax)^2, in the reference's loop
// order (ewald.f90:936-1050): l ascending; for l = 0, m >= 0 and, for m = 0, n >= 1.
__host__ __device__ inline bool kvec_kept(int l, int m, int n, int klmsq) {
  if (l == 0 && (m < 0 || (m == 0 && n < 1))) return false;
  return l * l + m * m + n * n <= klmsq;
}

int count_kvecs(int lmax, int mmax, int nmax) {
  const int klm = std::min(lmax, std::min(mmax, nmax));
  int nk = 0;
  for (int l = 0; l <= lmax; l++)
    for (int m = -mmax; m <= mmax; m++)
      for (int n = -nmax; n <= nmax; n++) nk += kvec_kept(l, m, n, klm * klm);
  return nk;
}

int count_rows(int lmax, int mmax, int nmax) {
  const int klm = std::min(lmax, std::min(mmax, nmax));
  int n = 0;
  for (int l = 0; l <= lmax; l++)
    for (int m = -mmax; m <= mmax; m++)
      n += (l > 0 || m >= 0) && l * l + m * m + (l == 0 && m == 0) <= klm * klm;
  return n;
}

// Block 0 writes the ordered k-vector list and, with `rows`, its rows (one per (l, m), KRow) and
// the z components rn[n + nmax]: a thread counts the k-vectors and rows of a run of (l, m), an
// exclusive scan gives the runs their places, and then the block's threads take the (l, m, n)
// candidates in turn.  The other blocks build the charged sites' phase tables (as k_ktab) and
// clear the compact forces, the energy/virial accumulators and the structure factors (all summed
// into with atomics).
constexpr int kSetupThreads = 512, kMaxK = 64;
__global__ void __launch_bounds__(kSetupThreads)
    k_fixed_setup(int lmax, int mmax, int nmax, double alp, double box, KVec *kv, KRow *rows,
                  double *rn, int nk, const double *__restrict__ x, const double *__restrict__ y,
                  const double *__restrict__ z, const double *__restrict__ xs,
                  const double *__restrict__ ys, const double *__restrict__ zs, int nm, int ld,
                  SiteSets S, int k1, double2 *tab, double *f, double *sk, double *scal) {
  if (blockIdx.x > 0) {
    const int t = (blockIdx.x - 1) * blockDim.x + threadIdx.x, stride = (gridDim.x - 1) * blockDim.x;
    const int n = nm * S.nq;
    if (t < n) {
      const int i = t / S.nq, r = t % S.nq;
      const size_t o = (size_t)i * ld + S.qsite[r];
      const double p[3] = {x[i] + xs[o], y[i] + ys[o], z[i] + zs[o]};
      for (int a = 0; a < 3; a++) {
        double2 *T = tab + (size_t)a * k1 * n + t;
        double c1, s1;
        sincos(2.0 * ccpd::kPi * p[a] / box, &s1, &c1);
        double2 v = make_double2(1.0, 0.0);
        for (int l = 0; l < k1; l++) {
          T[(size_t)l * n] = v;
          v = l == 0 ? make_double2(c1, s1) : make_double2(v.x * c1 - v.y * s1, v.y * c1 + v.x * s1);
        }
        f[(size_t)a * n + t] = 0.0;
      }
    }
    if (t < S_COUNT) scal[t] = 0.0;
    for (int u = t; u < 4 * nk; u += stride) sk[u] = 0.0;
    return;
  }
  __shared__ int2 scan[kSetupThreads];
  __shared__ int first[(kMaxK + 1) * (2 * kMaxK + 1)];  // of each (l, m), in the list
  const int M = 2 * mmax + 1, N = 2 * nmax + 1, nlm = (lmax + 1) * M;
  const int klm = min(lmax, min(mmax, nmax)), klmsq = klm * klm;
  const double twopi = 2.0 * ccpd::kPi, volmi = box * box * box;
  auto reach = [&](int l, int m) {  // the largest n of (l, m), -1 for none
    const int left = klmsq - l * l - m * m;
    if (left < 0 || (l == 0 && m < 0)) return -1;
    int n = (int)sqrtf((float)left);
    while (n * n > left) n--;
    while ((n + 1) * (n + 1) <= left) n++;
    return l == 0 && m == 0 && n < 1 ? -1 : n;
  };
  const int per = (nlm + blockDim.x - 1) / blockDim.x;
  const int c0 = min(nlm, (int)threadIdx.x * per), c1 = min(nlm, c0 + per);
  int2 kept = make_int2(0, 0);
  for (int c = c0; c < c1; c++) {
    const int l = c / M, m = c % M - mmax, n = reach(l, m);
    kept.x += n < 0 ? 0 : (l == 0 && m == 0 ? n : 2 * n + 1);
    kept.y += n >= 0;
  }
  scan[threadIdx.x] = kept;
  __syncthreads();
  for (int off = 1; off < (int)blockDim.x; off <<= 1) {
    const int2 v = threadIdx.x >= (unsigned)off ? scan[threadIdx.x - off] : make_int2(0, 0);
    __syncthreads();
    scan[threadIdx.x].x += v.x;
    scan[threadIdx.x].y += v.y;
    __syncthreads();
  }
  int2 o = scan[threadIdx.x];
  o.x -= kept.x;
  o.y -= kept.y;
  for (int c = c0; c < c1; c++) {
    const int l = c / M, m = c % M - mmax, n = reach(l, m);
    first[c] = o.x;
    if (n < 0) continue;
    const int nlo = l == 0 && m == 0 ? 1 : -n, len = n - nlo + 1;
    if (rows) rows[o.y] = {twopi * l / box, twopi * m / box, o.x, len, nlo, c};
    o.x += len;
    o.y++;
  }
  if (rows)
    for (int n = threadIdx.x; n < N; n += blockDim.x) rn[n] = twopi * (n - nmax) / box;
  __syncthreads();
  for (int c = threadIdx.x; c < nlm * N; c += blockDim.x) {
    const int lm = c / N, l = lm / M, m = lm - l * M - mmax, n = c - lm * N - nmax;
    if (!kvec_kept(l, m, n, klmsq)) continue;
    const int nlo = l == 0 && m == 0 ? 1 : -reach(l, m);
    KVec k;
    k.rl = twopi * l / box;
    k.rm = twopi * m / box;
    k.rn = twopi * n / box;
    const double rksq = k.rl * k.rl + k.rm * k.rm + k.rn * k.rn;
    k.ak = twopi / volmi * exp(-0.25 * rksq / (alp * alp)) / rksq;
    k.l = l;
    k.m = m;
    k.n = n;
    k.pad = 0;
    kv[first[lm] + n - nlo] = k;
  }
}

// Adds the compact charged-site forces into the caller's (molecule, ld) arrays and writes
// the energy (kcal/mol) and virial contribution with the reference's prefactors
// (ewald.f90:1151-1160).
__global__ void k_fixed_finish(const double *__restrict__ f, int nm, int ld, SiteSets S,
                               const double *__restrict__ scal, double *fxs, double *fys,
                               double *fzs, double *qkcpe, double *vir) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int n = nm * S.nq;
  if (t < n) {
    const int i = t / S.nq, r = t % S.nq;
    const size_t o = (size_t)i * ld + S.qsite[r];
    fxs[o] += f[t];
    fys[o] += f[(size_t)n + t];
    fzs[o] += f[2 * (size_t)n + t];
  }
  if (t == 0) {
    *qkcpe = 2.0 * ccpd::kR4pie0 * scal[S_KC_E] / 418.4;
    *vir += 2.0 * ccpd::kR4pie0 * scal[S_KC_VIR];
  }
}

int fail(int code, const std::string &msg) {
  set_error("ccp_kspace_ewald_fixed: " + msg);
  return code;
}

}  // namespace

extern "C" int ccp_kspace_ewald_fixed(const ccp_model *m, int nm, const double *x,
                                      const double *y, const double *z, const double *xs,
                                      const double *ys, const double *zs, int ld, int lmax,
                                      int mmax, int nmax, double alp, double box, double *qkcpe,
                                      double *fxs, double *fys, double *fzs, double *vir,
                                      void *stream) {
  if (!m || !x || !y || !z || !xs || !ys || !zs || !qkcpe || !fxs || !fys || !fzs || !vir)
    return fail(CCP_ERR_BAD_INPUT, "null argument");
  if (nm < 1 || ld < m->ns) return fail(CCP_ERR_BAD_INPUT, "need nm >= 1 and ld >= sites per molecule");
  if (lmax < 1 || mmax < 1 || nmax < 1) return fail(CCP_ERR_BAD_INPUT, "k-max must be >= 1");
  if (!(box > 0.0) || !(alp > 0.0)) return fail(CCP_ERR_BAD_INPUT, "box and alpha must be > 0");
  if (lmax > kMaxK || mmax > kMaxK || nmax > kMaxK) return fail(CCP_ERR_CAPACITY, "k-max above 64");

  // charged sites only: the compact site set (active slot = charged slot)
  SiteSets S;
  std::memset(&S, 0, sizeof(S));
  for (int s = 0; s < m->ns; s++) {
    if (m->charge[s] == 0.0) continue;
    if (S.nq >= ccpd::kMaxQ) return fail(CCP_ERR_BAD_INPUT, "too many charged sites per molecule");
    S.qsite[S.nq] = s;
    S.a_of_q[S.nq] = S.nq;
    S.asite[S.nq] = S.nq;
    S.q[S.nq] = m->charge[s];
    S.p_of_a[S.nq] = -1;
    S.nq++;
  }
  S.na = S.nq;
  S.ns = S.nq;  // compact force layout: (molecule, charged slot)
  if (S.nq == 0) return fail(CCP_ERR_BAD_INPUT, "model has no charged sites");

  const int nk = count_kvecs(lmax, mmax, nmax);
  const int k1 = std::max(std::max(std::max(lmax, mmax), nmax) + 1, 2);
  const size_t nq = (size_t)nm * S.nq;
  const size_t b_kv = up256(sizeof(KVec) * (size_t)nk), b_sk = up256(sizeof(double) * 4 * (size_t)nk);
  const size_t b_com = up256(sizeof(double4) * (size_t)nm), b_act = up256(sizeof(double4) * nq);
  const size_t b_tab = up256(sizeof(double2) * 3 * (size_t)k1 * nq);
  const size_t b_f = up256(sizeof(double) * 3 * nq), b_scal = up256(sizeof(double) * S_COUNT);
  const size_t need = b_kv + b_sk + b_com + b_act + b_tab + b_f + b_scal;
  if (need > kFixedScratchBytes)
    return fail(CCP_ERR_CAPACITY, "needs " + std::to_string(need) + " bytes of scratch for " +
                                      std::to_string(nm) + " molecules and " + std::to_string(nk) +
                                      " k-vectors; the fixed scratch holds " +
                                      std::to_string(kFixedScratchBytes) + " bytes");

  // by rows of the k-vector list (k_krows.cu) where the form applies and the scratch has room
  // for its rows and weights
  const int nrow = count_rows(lmax, mmax, nmax);
  const size_t b_row = up256(sizeof(KRow) * (size_t)nrow);
  const size_t b_rn = up256(sizeof(double) * (2 * (size_t)nmax + 1));
  const size_t b_w = up256(sizeof(double2) * krow_weight_len(nrow, nmax));
  const bool krows = iter_rows_fit(nmax) && need + b_row + b_rn + b_w <= kFixedScratchBytes;

  // The launch checks below read the thread's last CUDA error.  An error that earlier work of
  // the caller left pending would be reported as this call's own, so such a call is refused
  // before anything is launched, and the pending error is left in place for its owner.
  cudaError_t e = cudaPeekAtLastError();
  if (e != cudaSuccess)
    return fail(CCP_ERR_CUDA, std::string("a CUDA error from earlier work is pending (nothing "
                                          "launched): ") + cudaGetErrorString(e));
  int dev = 0;
  e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return fail(CCP_ERR_CUDA, std::string("cudaGetDevice: ") + cudaGetErrorString(e));
  if (dev < 0 || dev >= kMaxDevices) return fail(CCP_ERR_BAD_INPUT, "device ordinal above 63");
  unsigned char *base;
  {
    std::lock_guard<std::mutex> lock(g_addr_mu);
    if (!g_addr[dev]) {
      void *p = nullptr;
      e = cudaGetSymbolAddress(&p, g_kspace_scratch);
      if (e != cudaSuccess)
        return fail(CCP_ERR_CUDA, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
      g_addr[dev] = static_cast<unsigned char *>(p);
    }
    base = g_addr[dev];
  }
  KVec *kv = reinterpret_cast<KVec *>(base);
  double *sk = reinterpret_cast<double *>(base + b_kv);
  double2 *tab = reinterpret_cast<double2 *>(base + b_kv + b_sk + b_com + b_act);
  double *f = reinterpret_cast<double *>(base + b_kv + b_sk + b_com + b_act + b_tab);
  double *scal = reinterpret_cast<double *>(base + b_kv + b_sk + b_com + b_act + b_tab + b_f);

  cudaStream_t st = static_cast<cudaStream_t>(stream);
  KRow *rows = reinterpret_cast<KRow *>(base + need);
  double *rn = reinterpret_cast<double *>(base + need + b_row);
  double2 *w = reinterpret_cast<double2 *>(base + need + b_row + b_rn);
  const size_t nthr = std::max(nq, (size_t)S_COUNT);  // nq >= nm
  k_fixed_setup<<<1 + (unsigned)((nthr + kSetupThreads - 1) / kSetupThreads), kSetupThreads, 0, st>>>(
      lmax, mmax, nmax, alp, box, kv, krows ? rows : nullptr, rn, nk, x, y, z, xs, ys, zs, nm, ld, S,
      k1, tab, f, sk, scal);
  e = cudaGetLastError();
  if (krows) {  // the gather adds to the caller's forces
    SiteSets Sr = S;
    for (int r = 0; r < S.nq; r++) Sr.asite[r] = S.qsite[r];
    const KRowArgs R = {kv, rows, nrow, rn, tab, nm, lmax, mmax, nmax, Sr, sk, w};
    if (e == cudaSuccess) e = launch_krow_sums(false, R, nullptr, st);
    if (e == cudaSuccess) e = launch_krow_weights(false, R, alp, 1, scal, st);
    if (e == cudaSuccess)
      e = launch_krow_gather(false, R, 0, nullptr, nullptr, {fxs, fys, fzs, ld, qkcpe, vir, scal}, st);
    return e == cudaSuccess ? CCP_OK : fail(CCP_ERR_CUDA, cudaGetErrorString(e));
  } else {
    if (e == cudaSuccess)
      e = launch_kspace_sums(0, kv, nk, tab, nm, S, lmax, mmax, nmax, nullptr, sk, st);
    if (e == cudaSuccess) e = launch_kspace_energy(0, kv, nk, sk, alp, scal, st);
    if (e == cudaSuccess)
      e = launch_kspace_gather(0, kv, nk, tab, nm, S, lmax, mmax, nmax, nullptr, sk, nullptr, f, st);
  }
  if (e != cudaSuccess) return fail(CCP_ERR_CUDA, cudaGetErrorString(e));
  k_fixed_finish<<<(int)((nq + 255) / 256), 256, 0, st>>>(
      f, nm, ld, S, scal, fxs, fys, fzs, qkcpe, vir);
  if ((e = cudaGetLastError()) != cudaSuccess) return fail(CCP_ERR_CUDA, cudaGetErrorString(e));
  return CCP_OK;
}
