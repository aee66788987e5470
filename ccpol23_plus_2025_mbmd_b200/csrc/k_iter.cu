// k_iter.cu -- one Jacobi step of the induced-dipole solve as two kernels (sm_100a, FP64).
//
// iteridm (nb_induction_model.f90:1193-1407) updates every polarisable dipole from the field
//   E = T.mu (real space + short-range + intramolecular)  +  E_k(mu) (reciprocal)  +  E0.
// The geometry is fixed during the solve, so besides the dipole tensors (k_induction.cu) the
// phases exp(i k.r_s) of the polarisable sites are prepared once per evaluation, factored as
// exp(i(l x + m y)) for every (l, m) and exp(i n z) for every n of each site (the product
// order of the reference's recurrence, ewald.f90:960-1010): a (site, k-vector) phase is then
// one complex product of two table entries, and the tables (nlm + nz per site) stay in L2
// where the full (site, k) matrix would not.  Each iteration then is
//   A  blocks [0, nA):  T.mu, two warps per polarisable site, lanes over its (neighbour, site)
//                       tensor entries (contiguous, so the loads coalesce); these blocks also
//                       clear the S(k) buffer of the other step parity;
//      blocks [nA, ..): dipole structure factors -4 a(k) S(k), S(k) = sum_s (k.mu_s)
//                       e^{ik.r_s}, one thread per k over a chunk of sites, merged with FP64
//                       atomics into this step's buffer;
//   B  one warp per polarisable site: reciprocal field sum_k k g(k, s) (lanes over k), the
//      update mu' = alpha (E_real + E_k + E0) in place, the |mu - mu'|^2 and energy sums;
//      the last block to finish (atomic ticket) closes the iteration: it records the
//      iteration count, change and energy, clears the accumulators for the next iteration,
//      marks the solve finished when it has converged (state[3]: a later B in the same pass
//      of a graph body that unrolls several steps then returns at once) and, inside the
//      graph, sets the WHILE node's condition.  S(k) alternates between two buffers by step
//      parity, so no block has to clear it after the gather.
// Small boxes run the whole solve in one cluster instead (k_dip_cluster), middle ones in one
// cooperative grid (k_dip_grid).  The step normally
// runs in the row form (k_iter_a_rows, k_iter_b_rows below), which takes the
// reciprocal sums as matrix products over the rows of the k-vector list.  k_iter_a and k_iter_b
// take them k-vector by k-vector (k_max above the row form's, or by option), from the factor
// tables or, where it fits in half of the L2, from the full phase matrix [site][k].
#include <cooperative_groups.h>

#include <algorithm>
#include <type_traits>

#include "ccp_device.cuh"

using namespace ccpd;

namespace {

constexpr int kThreads = 128;  // small blocks fit beside two FS3 blocks on an SM (see the step kernels)

// Programmatic dependent launch (sm_90+): `launch_dependents` lets the next kernel in the
// stream (launched with programmatic stream serialization) start its blocks once every block
// of this one has executed it; `wait` blocks until the preceding kernel has completed and its
// writes are visible.  Both are no-ops in a kernel launched without the attribute.
__device__ __forceinline__ void pdl_launch_dependents() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
constexpr int kWarps = kThreads / 32;
// threads of a gather/update block (k_iter_b): they split the k-vectors, so the block's
// serial chain of dependent loads is nk / kGatherThreads iterations long
#ifndef CCP_GATHER_THREADS
#define CCP_GATHER_THREADS 128
#endif
constexpr int kGatherThreads = CCP_GATHER_THREADS;
constexpr int kGatherWarps = kGatherThreads / 32;
constexpr int kSumSitesMax = 128;  // polarisable sites per structure-factor block (A.sum_sites)
// polarisable sites per gather/update block: a template argument, 2, 3, 4, 6 or 8 (A.gather_sites)

// Phase factors of polarisable site w from the per-axis tables tab[axis][l][site] (ewald.f90:
// 960-1010): XY[w][l][m] = exp(i l x) exp(+-i |m| y) in the reference's product order, and
// Z[w][n] = exp(i |n| z), conjugated for n < 0, so that the phase of k = (l, m, n) is
// XY[l][m] * Z[n] exactly as the reference's final product.
__global__ void k_phase_factors(const double2 *__restrict__ tab, int nm, SiteSets S, int k1,
                                int lmax, int mmax, int nmax, double2 *XY, double2 *Z) {
  const int nw = nm * S.np;
  const int M = 2 * mmax + 1, nlm = (lmax + 1) * M, nz = 2 * nmax + 1;
  const size_t N = (size_t)nm * S.na;
  const size_t total = (size_t)nw * (nlm + nz);
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total;
       t += (size_t)gridDim.x * blockDim.x) {
    const int w = (int)(t / (nlm + nz)), u = (int)(t - (size_t)w * (nlm + nz));
    const int i = w / S.np, p = w % S.np;
    const size_t st = (size_t)i * S.na + S.a_of_p[p];
    if (u < nlm) {
      const int l = u / M, m = u % M - mmax;
      const double2 el = tab[(size_t)(0 * k1 + l) * N + st];
      const double2 em = tab[(size_t)(1 * k1 + (m < 0 ? -m : m)) * N + st];
      double clm, slm;
      if (m >= 0) {
        clm = el.x * em.x - el.y * em.y;
        slm = el.y * em.x + em.y * el.x;
      } else {
        clm = el.x * em.x + el.y * em.y;
        slm = el.y * em.x - em.y * el.x;
      }
      XY[(size_t)w * nlm + u] = make_double2(clm, slm);
    } else {
      const int n = u - nlm - nmax;
      const double2 en = tab[(size_t)(2 * k1 + (n < 0 ? -n : n)) * N + st];
      Z[(size_t)w * nz + (u - nlm)] = make_double2(en.x, n < 0 ? -en.y : en.y);
    }
  }
}

// The factor tables of the row form: XYt[row tile of 8][w][row in tile] = exp(i(l x + m y)) of
// the k-vector rows (KRow, lm = l (2 mmax + 1) + m + mmax), formed as k_phase_factors forms XY,
// zero past the last row; and Zc[w][2 n + {0, 1}] = (cos, sin)(n z), n = 0 .. zs / 2 - 1, zero
// past nmax.  A tile's rows are the fastest index, so that an operand fragment of 8 rows x 4
// sites is 512 contiguous bytes.
__global__ void k_phase_rows(const double2 *__restrict__ tab, int nm, SiteSets S, int k1,
                             int mmax, int nmax, const KRow *__restrict__ rows, int nrow, int zs,
                             double2 *XYt, double2 *Zc) {
  const int nw = nm * S.np;
  const int M = 2 * mmax + 1, nt8 = (nrow + 7) / 8;
  const size_t N = (size_t)nm * S.na;
  const size_t nxy = (size_t)nt8 * nw * 8, total = nxy + (size_t)nw * (zs / 2);
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total;
       t += (size_t)gridDim.x * blockDim.x) {
    if (t < nxy) {
      const size_t u = t >> 3;
      const int rt = (int)(u / nw), w = (int)(u - (size_t)rt * nw), r = rt * 8 + (int)(t & 7);
      double2 xy = make_double2(0.0, 0.0);
      if (r < nrow) {
        const int i = w / S.np, p = w % S.np;
        const size_t st = (size_t)i * S.na + S.a_of_p[p];
        const int lm = rows[r].lm, l = lm / M, m = lm % M - mmax;
        const double2 el = tab[(size_t)(0 * k1 + l) * N + st];
        const double2 em = tab[(size_t)(1 * k1 + (m < 0 ? -m : m)) * N + st];
        xy = m >= 0 ? make_double2(el.x * em.x - el.y * em.y, el.y * em.x + em.y * el.x)
                    : make_double2(el.x * em.x + el.y * em.y, el.y * em.x - em.y * el.x);
      }
      XYt[t] = xy;
    } else {
      const size_t u = t - nxy;
      const int w = (int)(u / (zs / 2)), n = (int)(u - (size_t)w * (zs / 2));
      const int i = w / S.np, p = w % S.np;
      const size_t st = (size_t)i * S.na + S.a_of_p[p];
      Zc[u] = n <= nmax ? tab[(size_t)(2 * k1 + n) * N + st] : make_double2(0.0, 0.0);
    }
  }
}

// phase of k = (l, m, n) at site w from its factor rows
__device__ __forceinline__ double2 kphase(const double2 *__restrict__ xyw,
                                          const double2 *__restrict__ zw, int lm, int ni) {
  const double2 a = xyw[lm], b = zw[ni];
  return make_double2(a.x * b.x - a.y * b.y, a.y * b.x + a.x * b.y);
}

// Phase of k-vector k (rows lm, ni of the factor tables) at polarisable site w: with the
// phase matrix one coalesced load of row w, else the product of the two factor entries.
template <bool PM>
__device__ __forceinline__ double2 site_phase(const IterArgs &A, int w, int k, int lm, int ni) {
  if constexpr (PM) return A.PM[(size_t)w * A.nk + k];
  return kphase(A.XY + (size_t)w * A.nlm, A.Z + (size_t)w * A.nz, lm, ni);
}

// The phase matrix PM[w][k] = XY[w][lm(k)] * Z[w][n(k)] (kphase, the same product the step
// kernels form without it), one coalesced row of nk phases per polarisable site.
__global__ void k_phase_matrix(const KGather *__restrict__ kg, int nk, int nw, int nlm, int nz,
                               const double2 *__restrict__ XY, const double2 *__restrict__ Z,
                               double2 *PM) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nk) return;
  const int lmni = kg[k].lmni, lm = lmni >> 8, ni = lmni & 255;
  for (int w = blockIdx.y; w < nw; w += gridDim.y)
    PM[(size_t)w * nk + k] = kphase(XY + (size_t)w * nlm, Z + (size_t)w * nz, lm, ni);
}

// The vector a T.mu product reads: the dipoles themselves (Jacobi).
struct MuIn {
  const double *__restrict__ mu;
  __device__ __forceinline__ double3 operator()(size_t site, int) const {
    const double *m = mu + site * 3;
    return make_double3(m[0], m[1], m[2]);
  }
};

// Preconditioned conjugate gradients (the mixed form's dipole solve) for the same linear
// system as the Jacobi step: A mu = E0 with A mu = mu / alpha - F(mu), F(mu) the field of the
// dipoles (T.mu real space + reciprocal + intramolecular corrections, which is symmetric), and
// the preconditioner M^-1 = diag(alpha), so that the preconditioned residual u = alpha (E0 -
// A x) = alpha (E0 + F(x)) - x is exactly the Jacobi update at the iterate x.  The recurrences
// are Chronopoulos and Gear's one-reduction form (Chronopoulos & Gear, J. Comput. Appl. Math.
// 25 (1989) 153-168): with w = A u and s = A p,
//   p = u + beta p,  s = w + beta s,  x += alpha p,  u -= alpha M^-1 s,  w = A u,
//   gamma = (u, M u), delta = (w, u), beta' = gamma' / gamma,
//   alpha' = gamma' / (delta' - beta' gamma' / alpha),
// so one step is one product A u and one merged reduction, as a Jacobi step is.  The new u
// of a site is needed by every reader of the product before the update kernel can store it,
// so readers form it where they read it (pcg_s, pcg_u) from the stored u, w and s and the two
// scalars of the step; the update kernel forms the same values with the same operations
// (explicit roundings, no contraction), so all of them see the same u.
__device__ __forceinline__ double pcg_s(double w, double s, double beta) {
  return __fma_rn(beta, s, w);
}
__device__ __forceinline__ double pcg_u(double u, double s_new, double apol, double alpha) {
  return __fma_rn(-alpha, __dmul_rn(apol, s_new), u);
}
struct PcgIn {
  const double *__restrict__ u;
  const double *__restrict__ w;
  const double *__restrict__ s;
  double alpha, beta, a0, a1, a2, a3;  // step scalars; polarisabilities of sites 0..3
  __device__ __forceinline__ double apol(int q) const {
    return q == 0 ? a0 : (q == 1 ? a1 : (q == 2 ? a2 : a3));
  }
  __device__ __forceinline__ double comp(size_t o, double ap) const {
    return pcg_u(u[o], pcg_s(w[o], s[o], beta), ap, alpha);
  }
  __device__ __forceinline__ double3 operator()(size_t site, int q) const {
    const double ap = apol(q);
    const size_t o = site * 3;
    return make_double3(comp(o, ap), comp(o + 1, ap), comp(o + 2, ap));
  }
};

__device__ __forceinline__ PcgIn pcg_in(const IterArgs &A) {
  PcgIn in;
  in.u = A.cu;
  in.w = A.cw;
  in.s = A.cs;
  in.alpha = A.state[kIterAlpha];
  in.beta = A.state[kIterBeta];
  in.a0 = A.S.apol[0];
  in.a1 = A.np > 1 ? A.S.apol[1] : 0.0;
  in.a2 = A.np > 2 ? A.S.apol[2] : 0.0;
  in.a3 = A.np > 3 ? A.S.apol[3] : 0.0;
  return in;
}

// T.mu of polarisable site w = (i, p): entries T4/TB[i][p][n][q] for the neighbours n of i and
// the polarisable sites q of each, plus the intramolecular entries S4/SB[i][p][q].  Called by
// whole warps; the sum is returned to every lane.  `in` gives the vector multiplied.
template <typename In>
__device__ __forceinline__ void tmu_warp(int w, int lane, const int *__restrict__ nbr,
                                         const int *__restrict__ ncnt, int cap, int np,
                                         const double4 *__restrict__ T4,
                                         const double *__restrict__ TB,
                                         const double4 *__restrict__ S4,
                                         const double *__restrict__ SB, const In &in,
                                         double &ex, double &ey, double &ez) {
  const int i = w / np;
  const int cnt = ncnt[i];
  const size_t base = (size_t)w * cap * np;
  ex = ey = ez = 0.0;
  const int n_ent = cnt * np;
#pragma unroll 4
  for (int e = lane; e < n_ent; e += 32) {
    const int n = e / np, q = e - n * np;
    const int j = nbr[(size_t)i * cap + n];
    const double4 t = T4[base + e];
    const double b = TB[base + e];
    const double3 m = in((size_t)j * np + q, q);
    const double mx = m.x, my = m.y, mz = m.z;
    const double dm = t.w * (t.x * mx + t.y * my + t.z * mz);
    ex += dm * t.x - b * mx;
    ey += dm * t.y - b * my;
    ez += dm * t.z - b * mz;
  }
  if (lane < np) {
    const size_t o = (size_t)w * np + lane;
    const double4 t = S4[o];
    const double b = SB[o];
    const double3 m = in((size_t)i * np + lane, lane);
    const double mx = m.x, my = m.y, mz = m.z;
    const double dm = t.w * (t.x * mx + t.y * my + t.z * mz);
    ex += dm * t.x - b * mx;
    ey += dm * t.y - b * my;
    ez += dm * t.z - b * mz;
  }
  ex = warp_sum(ex);
  ey = warp_sum(ey);
  ez = warp_sum(ez);
}

// One warp per polarisable site (the fallback path's real-space part).
__global__ void __launch_bounds__(kThreads)
    k_tmu(const int *__restrict__ nbr, const int *__restrict__ ncnt, int cap, int nw, int np,
          const double4 *__restrict__ T4, const double *__restrict__ TB,
          const double4 *__restrict__ S4, const double *__restrict__ SB,
          const double *__restrict__ mu, double *eim) {
  const int w = blockIdx.x * kWarps + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (w >= nw) return;
  double ex, ey, ez;
  tmu_warp(w, lane, nbr, ncnt, cap, np, T4, TB, S4, SB, MuIn{mu}, ex, ey, ez);
  if (lane == 0) {
    eim[(size_t)w * 3 + 0] = ex;
    eim[(size_t)w * 3 + 1] = ey;
    eim[(size_t)w * 3 + 2] = ez;
  }
}

// Blocks [0, nA) of a step's first kernel: T.mu, two warps per polarisable site; they also
// clear the S(k) buffer of the other step parity, whose last reader, the previous step's
// gather, has finished.  The tensor entries are fixed during the solve, so a lane's first
// kTmuPre entries (all of them at 9 A: 306 per site) and their source sites are loaded before
// the wait for the previous step's dipoles; after it only the dipoles are.
constexpr int kTmuWarps = 2, kTmuPre = 5;
constexpr int kTmuSites = kWarps / kTmuWarps;  // sites per block
__host__ __device__ constexpr int tmu_blocks(int nw) { return (nw + kTmuSites - 1) / kTmuSites; }
template <bool PCG>
__device__ __forceinline__ void iter_a_tmu(const IterArgs &A, int block, int nA) {
  const int w = block * kTmuSites + threadIdx.x / (32 * kTmuWarps);
  const int lane = threadIdx.x % (32 * kTmuWarps);
  const bool on = w < A.nw;
  const int i = on ? w / A.np : 0, n_ent = on ? A.ncnt[i] * A.np : 0;
  const size_t base = (size_t)w * A.cap * A.np;
  const int *nb = A.nbr + (size_t)i * A.cap;
  double4 t[kTmuPre + 1];
  double b[kTmuPre + 1];
  int src[kTmuPre + 1], q[kTmuPre + 1];
#pragma unroll
  for (int u = 0; u < kTmuPre; u++) {
    const int e = lane + 32 * kTmuWarps * u;
    t[u] = make_double4(0.0, 0.0, 0.0, 0.0);
    b[u] = 0.0;
    src[u] = q[u] = 0;
    if (e < n_ent) {
      const int n = e / A.np;
      q[u] = e - n * A.np;
      t[u] = A.T4[base + e];
      b[u] = A.TB[base + e];
      src[u] = nb[n] * A.np + q[u];
    }
  }
  // the intramolecular entries
  t[kTmuPre] = make_double4(0.0, 0.0, 0.0, 0.0);
  b[kTmuPre] = 0.0;
  src[kTmuPre] = q[kTmuPre] = 0;
  if (on && lane < A.np) {
    t[kTmuPre] = A.S4[(size_t)w * A.np + lane];
    b[kTmuPre] = A.SB[(size_t)w * A.np + lane];
    src[kTmuPre] = i * A.np + lane;
    q[kTmuPre] = lane;
  }
  pdl_wait();  // the previous step's dipoles (and its gather's last use of the S(k) buffer)
  PcgIn pin;
  if constexpr (PCG) pin = pcg_in(A);
  auto mu = [&](int s, int qs) {
    if constexpr (PCG) return pin((size_t)s, qs);
    else return MuIn{A.mu}((size_t)s, qs);
  };
  double ex = 0.0, ey = 0.0, ez = 0.0;
  auto add = [&](const double4 &T, double B, const double3 &m) {
    const double dm = T.w * (T.x * m.x + T.y * m.y + T.z * m.z);
    ex += dm * T.x - B * m.x;
    ey += dm * T.y - B * m.y;
    ez += dm * T.z - B * m.z;
  };
  double3 m[kTmuPre + 1];
#pragma unroll
  for (int u = 0; u <= kTmuPre; u++) m[u] = mu(src[u], q[u]);  // site 0's where there is no entry
#pragma unroll
  for (int u = 0; u <= kTmuPre; u++) add(t[u], b[u], m[u]);
#pragma unroll kTmuPre
  for (int e = lane + 32 * kTmuWarps * kTmuPre; e < n_ent; e += 32 * kTmuWarps) {
    const int n = e / A.np, qe = e - n * A.np;
    add(A.T4[base + e], A.TB[base + e], mu(nb[n] * A.np + qe, qe));
  }
  double2 *other = reinterpret_cast<double2 *>(A.sk) + (A.par ^ 1);
  for (int k = block * kThreads + threadIdx.x; k < A.nk; k += nA * kThreads)
    other[2 * (size_t)k] = make_double2(0.0, 0.0);
  // the next kernel may launch once every block is this far: late enough that its blocks
  // do not hold SM slots (which concurrent kernels could use) for long while they wait
  pdl_launch_dependents();
  ex = warp_sum(ex);
  ey = warp_sum(ey);
  ez = warp_sum(ez);
  __shared__ double part[kWarps][3];
  const int wid = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    part[wid][0] = ex;
    part[wid][1] = ey;
    part[wid][2] = ez;
  }
  __syncthreads();
  if (on && lane < 3) {
    double v = 0.0;
#pragma unroll
    for (int u = 0; u < kTmuWarps; u++) v += part[wid + u][lane];
    A.eim[(size_t)w * 3 + lane] = v;
  }
}

// Without rows T.mu takes one warp per polarisable site: iter_a_tmu's entries held ahead cost the
// sums' blocks of the same kernel their occupancy (96 registers a thread against 56, PCG 128
// against 72), and those are most of this step.
template <bool PCG, bool PM>
__global__ void __launch_bounds__(kThreads)
    k_iter_a(IterArgs A) {
  // no test of the finished flag here: a step after the finish only rewrites the T.mu
  // scratch and S(k), which the next use clears, and it saves a dependent load per step
  pdl_wait();  // the previous step's dipoles (and its gather's last use of the S(k) buffer)
  const int nA = (A.nw + kWarps - 1) / kWarps;
  PcgIn pin;
  if constexpr (PCG) pin = pcg_in(A);
  if ((int)blockIdx.x < nA) {
    // these blocks also clear the S(k) buffer of the other step parity
    double2 *other = reinterpret_cast<double2 *>(A.sk) + (A.par ^ 1);
    for (int k = blockIdx.x * kThreads + threadIdx.x; k < A.nk; k += nA * kThreads)
      other[2 * (size_t)k] = make_double2(0.0, 0.0);
    const int w = blockIdx.x * kWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (w >= A.nw) return;
    double ex, ey, ez;
    if constexpr (PCG)
      tmu_warp(w, lane, A.nbr, A.ncnt, A.cap, A.np, A.T4, A.TB, A.S4, A.SB, pin, ex, ey, ez);
    else
      tmu_warp(w, lane, A.nbr, A.ncnt, A.cap, A.np, A.T4, A.TB, A.S4, A.SB, MuIn{A.mu}, ex, ey, ez);
    pdl_launch_dependents();  // as late as in iter_a_tmu
    if (lane < 3) A.eim[(size_t)w * 3 + lane] = lane == 0 ? ex : (lane == 1 ? ey : ez);
    return;
  }
  // structure factors: block b covers k-vectors [kt*256, kt*256+256) and sites of chunk sc
  extern __shared__ double smu[];  // A.sum_sites x 3 dipole components
  const int b = blockIdx.x - nA;
  const int nkt = (A.nk + kThreads - 1) / kThreads;
  const int kt = b % nkt, sc = b / nkt;
  const int s0 = sc * A.sum_sites, cnt = min(A.sum_sites, A.nw - s0);
  for (int u = threadIdx.x; u < cnt * 3; u += kThreads) {
    if constexpr (PCG) {
      const int site = s0 + u / 3;
      smu[u] = pin.comp((size_t)s0 * 3 + u, pin.apol(site % A.np));
    } else {
      smu[u] = A.mu[(size_t)s0 * 3 + u];
    }
  }
  __syncthreads();
  const int k = kt * kThreads + threadIdx.x;
  if (k >= A.nk) return;
  const KVec K = A.kv[k];
  const int lm = K.l * (2 * A.mmax + 1) + K.m + A.mmax, ni = K.n + A.nmax;
  double a0 = 0.0, a1 = 0.0;
#pragma unroll 4
  for (int s = 0; s < cnt; s++) {
    const double2 ph = site_phase<PM>(A, s0 + s, k, lm, ni);
    const double dk = K.rl * smu[3 * s] + K.rm * smu[3 * s + 1] + K.rn * smu[3 * s + 2];
    a0 += dk * ph.x;
    a1 += dk * ph.y;
  }
  pdl_launch_dependents();
  // kspace_efield_idm's weight (nb_induction_model.f90:2560-2600), applied before the merge
  const double g = -4.0 * K.ak;
  atomicAdd(&A.sk[(size_t)k * 4 + 2 * A.par], g * a0);
  atomicAdd(&A.sk[(size_t)k * 4 + 2 * A.par + 1], g * a1);
}

// The PCG step's update for the GS sites of a block, after the reciprocal field of
// u is in `part`: the vectors of the step (s, p, x, u, w = A u) in place, the partial sums
// of (u, M u), (w, u), |u|^2 and the energy -1/2 x.E0 (the reference's energy expression at
// the iterate), and in the last block to finish the step's scalars and the convergence test
// on sum |u|^2, the Jacobi update's norm at the iterate.
// ek(g, c) gives component c of the reciprocal field at the block's site g; the updating
// threads (one per site) are all in warp 0.
template <typename EK>
__device__ __forceinline__ void pcg_update(const IterArgs &A, int w0, int ns_blk, const EK &ekf) {
  double gam = 0.0, del = 0.0, ch = 0.0, en = 0.0;
  if ((int)threadIdx.x < ns_blk) {
    const int g = threadIdx.x, w = w0 + g;
    double ek[3];
    for (int c = 0; c < 3; c++) ek[c] = ekf(g, c);
    const double ap = A.S.apol[w % A.np];
    const double ca = A.state[kIterAlpha], cb = A.state[kIterBeta];
    for (int c = 0; c < 3; c++) {
      const size_t o = (size_t)w * 3 + c;
      const double u0 = A.cu[o];
      const double s = pcg_s(A.cw[o], A.cs[o], cb);
      const double p = __fma_rn(cb, A.cp[o], u0);
      const double x = __fma_rn(ca, p, A.mu[o]);
      const double u = pcg_u(u0, s, ap, ca);
      const double wv = u / ap - (A.eim[o] + ek[c]);
      A.cs[o] = s;
      A.cp[o] = p;
      A.mu[o] = x;
      A.cu[o] = u;
      A.cw[o] = wv;
      gam += u * u / ap;
      del += wv * u;
      ch += u * u;
      en += -0.5 * x * A.e0[o];
    }
  }
  gam = warp_sum(gam);  // the updating threads are all in warp 0
  del = warp_sum(del);
  ch = warp_sum(ch);
  en = warp_sum(en);
  __shared__ bool last;
  double *acc = A.state + kIterAcc;
  if (threadIdx.x == 0) {
    atomicAdd(acc + 0, gam);
    atomicAdd(acc + 1, del);
    atomicAdd(acc + 2, ch);
    atomicAdd(acc + 3, en);
    __threadfence();
    last = atomicAdd(A.ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  if (threadIdx.x == 0) {
    const double g1 = atomicAdd(acc + 0, 0.0), d1 = atomicAdd(acc + 1, 0.0);
    const double chg = atomicAdd(acc + 2, 0.0), ene = atomicAdd(acc + 3, 0.0);
    for (int k = 0; k < 4; k++) acc[k] = 0.0;
    *A.ticket = 0u;
    int it = (int)A.state[kIterIters] + 1;
    A.state[kIterChange] = chg;
    A.state[kIterEnergy] = ene;
    bool more = chg > A.thr && it < A.maxit;
    if (more) {
      const double beta = it == 1 ? 0.0 : g1 / A.state[kIterGamma];
      const double alpha = it == 1 ? g1 / d1 : g1 / (d1 - beta * g1 / A.state[kIterAlpha]);
      if (alpha > 0.0 && alpha < 1e300) {
        A.state[kIterAlpha] = alpha;
        A.state[kIterBeta] = beta;
        A.state[kIterGamma] = g1;
      } else {  // breakdown (not positive definite): reported as no convergence
        it = A.maxit;
        more = false;
      }
    }
    A.state[kIterIters] = (double)it;
    if (!more) A.state[kIterFinished] = 1.0;
    if (A.use_graph) cudaGraphSetConditional(A.handle, more ? 1u : 0u);
  }
}

// The Jacobi update of the block's sites (nb_induction_model.f90:1317-1359) from their
// reciprocal field ek(g, c), the change and energy sums, and in the last block to finish the
// step's close (iteration count, convergence test, the graph's condition).  The updating
// threads (one per site) are all in warp 0.
template <typename EK>
__device__ __forceinline__ void jacobi_update(const IterArgs &A, int w0, int ns_blk,
                                              const EK &ekf) {
  double ch = 0.0, en = 0.0;
  if ((int)threadIdx.x < ns_blk) {
    const int g = threadIdx.x, w = w0 + g;
    double ek[3];
    for (int c = 0; c < 3; c++) ek[c] = ekf(g, c);
    const double polr = A.S.apol[w % A.np];
    double Et[3], E0[3];
    for (int c = 0; c < 3; c++) {
      const size_t o = (size_t)w * 3 + c;
      E0[c] = A.e0[o];
      Et[c] = (A.eim[o] + ek[c]) + E0[c];
      const double m = polr * Et[c];
      const double d = A.mu[o] - m;
      ch += d * d;
      A.mu[o] = m;
    }
    en = -0.5 * polr * (Et[0] * E0[0] + Et[1] * E0[1] + Et[2] * E0[2]);
  }
  ch = warp_sum(ch);  // the updating threads are all in warp 0
  en = warp_sum(en);
  __shared__ bool last;
  if (threadIdx.x == 0) {
    atomicAdd(&A.scal[S_IND_CHANGE], ch);
    atomicAdd(&A.scal[S_IND_ENERGY], en);
    __threadfence();
    last = atomicAdd(A.ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  // every other block has added its sums
  __threadfence();
  if (threadIdx.x == 0) {
    const double chg = atomicAdd(&A.scal[S_IND_CHANGE], 0.0);
    const double ene = atomicAdd(&A.scal[S_IND_ENERGY], 0.0);
    const int it = (int)A.state[kIterIters] + 1;
    A.state[kIterIters] = (double)it;
    A.state[kIterChange] = chg;
    A.state[kIterEnergy] = ene;
    A.scal[S_IND_CHANGE] = 0.0;
    A.scal[S_IND_ENERGY] = 0.0;
    *A.ticket = 0u;
    const bool more = chg > A.thr && it < A.maxit;
    if (!more) A.state[kIterFinished] = 1.0;
    if (A.use_graph) cudaGraphSetConditional(A.handle, more ? 1u : 0u);
  }
}

template <bool PCG, bool PM, int GS>
__global__ void __launch_bounds__(kGatherThreads)
    k_iter_b(IterArgs A) {
  // GS polarisable sites per block; the warps split the k-vectors, so every
  // k-vector's weights are loaded once per block and reused for all its sites
  pdl_wait();  // T.mu, S(k) and the step scalars of this step's first kernel
  if (A.state[kIterFinished] != 0.0) return;  // finished in an earlier step of this pass
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int w0 = blockIdx.x * GS;
  const int ns_blk = min(GS, A.nw - w0);
  double acc[GS][3];
#pragma unroll
  for (int g = 0; g < GS; g++) acc[g][0] = acc[g][1] = acc[g][2] = 0.0;
  const double2 *skp = reinterpret_cast<const double2 *>(A.sk) + A.par;
  // the next k-vector's record and S(k) are loaded one iteration ahead, so that an iteration
  // waits for its phase loads only, not for the record that indexes them first
  KGather Kn{};
  double2 fn = make_double2(0.0, 0.0);
  if ((int)threadIdx.x < A.nk) {
    Kn = A.kg[threadIdx.x];
    fn = skp[2 * (size_t)threadIdx.x];
  }
#pragma unroll 2
  for (int k = threadIdx.x; k < A.nk; k += kGatherThreads) {
    const KGather K = Kn;
    const double2 f = fn;
    if (k + kGatherThreads < A.nk) {
      Kn = A.kg[k + kGatherThreads];
      fn = skp[2 * (size_t)(k + kGatherThreads)];
    }
    const int lm = K.lmni >> 8, ni = K.lmni & 255;
    // kspace_efield_idm gather (nb_induction_model.f90:2560-2600): g = -4 a_k (c S_re + s S_im)
    const double f0 = f.x, f1 = f.y;
#pragma unroll
    for (int g = 0; g < GS; g++) {
      if (g < ns_blk) {
        const double2 ph = site_phase<PM>(A, w0 + g, k, lm, ni);
        const double t = ph.x * f0 + ph.y * f1;
        acc[g][0] += K.rl * t;
        acc[g][1] += K.rm * t;
        acc[g][2] += K.rn * t;
      }
    }
  }
  pdl_launch_dependents();  // the gather, the bulk of the kernel, is done
  __shared__ double part[kGatherWarps][GS * 3];
#pragma unroll
  for (int g = 0; g < GS; g++)
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const double v = warp_sum(acc[g][c]);
      if (lane == 0) part[wid][g * 3 + c] = v;
    }
  __syncthreads();
  const auto ek = [&](int g, int c) {
    double v = 0.0;
    for (int u = 0; u < kGatherWarps; u++) v += part[u][g * 3 + c];
    return v;
  };
  if constexpr (PCG)
    pcg_update(A, w0, ns_blk, ek);
  else
    jacobi_update(A, w0, ns_blk, ek);
}

// ------------------------------------------------------------------ the row form
// The step's two reciprocal sums regrouped by the rows of the k-vector list (one (l, m), a run
// of n), which makes them small matrix products for the FP64 tensor cores:
//   structure factors  S(k) = sum_w Z(w, n) (B(w, r) + k_n C(w, r)),
//                      B = XY(w, r) (k_l mu_x + k_m mu_y),  C = XY(w, r) mu_z:
//     the real and imaginary parts of B and C (8 rows x sites) times (cos, sin)(n z) (sites x n
//     >= 0); +n and -n come from the same four real sums;
//   gather             E(w) = sum_r Re[XY(w, r) (k_l Q, k_m Q, Q_z)],
//                      Q = sum_n Z(w, n) conj F(k),  Q_z = sum_n k_n Z(w, n) conj F(k):
//     (cos, sin)(n z) (8 sites x n) times F's combinations over +-n (n x rows), F(k) the
//     weighted S(k) of the step.
// Both read the factor tables once per step (3 MB at 512 waters, where the phase matrix takes
// 38 MB twice), and XY serves 2 n_max + 1 k-vectors per load.  These are k_iter_a's and
// k_iter_b's sums with the products reassociated (equal to rounding).

// D = A (8x4) B (4x8) + C in FP64: lane l holds A[l/4][l%4], B[l%4][l/4] and C, D
// [l/4][2 (l%4) + {0, 1}].
__device__ __forceinline__ void dmma(double2 &d, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(d.x), "+d"(d.y)
      : "d"(a), "d"(b));
}

constexpr int kRowSteps = 6;  // steps of four sites whose XY a warp loads before it waits
constexpr int kRowWarps = 8;  // warps of a gather block, taking row tiles in turn

// the largest n of the rows of a lane's tile (rows sorted by length: only the row (0, 0), which
// has no n < 1, can reach further than its neighbours)
__device__ __forceinline__ int warp_max(int v) { return __reduce_max_sync(0xffffffffu, v); }

// Structure factors: block b (after the T.mu blocks) covers row tile b % nt8 and the sites of
// chunk b / nt8 (A.row_sites of them), its four warps a quarter each.  A lane forms the four
// operands (Re, Im of B and C) of its row and site from one XY load; J tiles of four n.  The
// warps' partial sums meet in shared memory, and one thread per (row, n) combines them into
// S(r, n) and S(r, -n), merged with FP64 atomics as in k_iter_a.  The first steps' XY are
// loaded before the wait for the previous step (the tables are fixed during the solve).
template <bool PCG, int J, bool ZS>
__global__ void __launch_bounds__(kThreads) k_iter_a_rows(IterArgs A) {
  // the sums' blocks first: they run longest.  The loop took 594 / 3682 us with T.mu's blocks
  // first, 565 / 3560 with the two alternating and 561 / 3400 so (512 / 2048 waters).
  const int nA = tmu_blocks(A.nw), nR = gridDim.x - nA;
  if ((int)blockIdx.x >= nR) {
    iter_a_tmu<PCG>(A, blockIdx.x - nR, nA);
    return;
  }
  // A.row_sites dipoles; the sites' Zc (rows of 8 J + 2: no bank conflicts between the four
  // sites of a step), and in the same place at the end the warps' sums
  extern __shared__ double4 smu4[];
  constexpr int kZs = 8 * J + 2;
  double *zsm = reinterpret_cast<double *>(smu4 + A.row_sites);
  double2(*red)[4 * J][32] = reinterpret_cast<double2(*)[4 * J][32]>(zsm);
  const int b = blockIdx.x, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int nt8 = (A.nrow + 7) / 8, rt = b % nt8, s0 = b / nt8 * A.row_sites;
  const int r = min(rt * 8 + (lane >> 2), A.nrow - 1);
  const KRow R = A.rows[r];
  const int jt = warp_max(R.nlo + R.len - 1) / 4 + 1;  // n tiles of the row tile
  const int q0 = wid * (A.row_sites / 4) + (lane & 3);  // lane's site in the chunk, step 0
  const int steps = min(A.row_sites / 16, (A.nw - s0 - wid * (A.row_sites / 4) + 3) / 4);
  const double2 *xyt = A.XYr + (size_t)rt * A.nw * 8 + (lane >> 2);
  double2 xy[kRowSteps];
#pragma unroll
  for (int t = 0; t < kRowSteps; t++)
    xy[t] = xyt[(size_t)min(s0 + q0 + 4 * t, A.nw - 1) * 8];
  if constexpr (ZS)
    for (int u = threadIdx.x; u < A.row_sites * 4 * J; u += kThreads) {
      const int q = u / (4 * J), c = u - q * (4 * J);
      reinterpret_cast<double2 *>(zsm + q * kZs)[c] =
          reinterpret_cast<const double2 *>(A.Zc + (size_t)min(s0 + q, A.nw - 1) * A.zs)[c];
    }
  pdl_wait();  // the previous step's dipoles (and its gather's last use of the S(k) buffer)
  PcgIn pin;
  if constexpr (PCG) pin = pcg_in(A);
  for (int u = threadIdx.x; u < A.row_sites; u += kThreads) {
    double4 m = make_double4(0.0, 0.0, 0.0, 0.0);
    if (s0 + u < A.nw) {
      const size_t o = (size_t)(s0 + u) * 3;
      if constexpr (PCG) {
        const double ap = pin.apol((s0 + u) % A.np);
        m = make_double4(pin.comp(o, ap), pin.comp(o + 1, ap), pin.comp(o + 2, ap), 0.0);
      } else {
        m = make_double4(A.mu[o], A.mu[o + 1], A.mu[o + 2], 0.0);
      }
    }
    smu4[u] = m;
  }
  __syncthreads();
  double2 acc[4][J];
#pragma unroll
  for (int c = 0; c < 4; c++)
#pragma unroll
    for (int j = 0; j < J; j++) acc[c][j] = make_double2(0.0, 0.0);
  for (int t0 = 0; t0 < steps; t0 += kRowSteps) {
#pragma unroll
    for (int t = 0; t < kRowSteps; t++) {
      if (t0 + t < steps) {  // warp-uniform
        const int q = q0 + 4 * (t0 + t);  // mu = 0 past the last site
        const double *z = (ZS ? zsm + q * kZs
                              : A.Zc + (size_t)min(s0 + q, A.nw - 1) * A.zs) + (lane >> 2);
        double zf[J];
#pragma unroll
        for (int j = 0; j < J; j++) zf[j] = j < jt ? z[8 * j] : 0.0;
        const double4 m = smu4[q];
        const double d = R.rl * m.x + R.rm * m.y;
        const double a[4] = {xy[t].x * d, xy[t].y * d, xy[t].x * m.z, xy[t].y * m.z};
#pragma unroll
        for (int j = 0; j < J; j++)
          if (j < jt)
#pragma unroll
            for (int c = 0; c < 4; c++) dmma(acc[c][j], a[c], zf[j]);
      }
    }
    if (t0 + kRowSteps < steps)
#pragma unroll
      for (int t = 0; t < kRowSteps; t++)
        xy[t] = xyt[(size_t)min(s0 + q0 + 4 * (t0 + kRowSteps + t), A.nw - 1) * 8];
  }
  pdl_launch_dependents();
  if constexpr (ZS) __syncthreads();  // every warp has read its sites' Zc
#pragma unroll
  for (int c = 0; c < 4; c++)
#pragma unroll
    for (int j = 0; j < J; j++) red[wid][c * J + j][lane] = acc[c][j];
  __syncthreads();
  // lane l of a warp's results is row l / 4 and n = 4 j + l % 4: (cos, sin) sums of each part
  for (int u = threadIdx.x; u < jt * 32; u += kThreads) {
    const int j = u >> 5, l = u & 31, row = rt * 8 + (l >> 2), n = 4 * j + (l & 3);
    if (row >= A.nrow || n > A.nmax) continue;
    double2 v[4];
#pragma unroll
    for (int c = 0; c < 4; c++) {
      v[c] = red[0][c * J + j][l];
#pragma unroll
      for (int w = 1; w < kWarps; w++) {
        const double2 x = red[w][c * J + j][l];
        v[c].x += x.x;
        v[c].y += x.y;
      }
    }
    const KRow K = A.rows[row];
    const double kn = A.rn[n + A.nmax];
    // B + k_n C (n), B - k_n C (-n), times cos +- i sin
    const double pr = (v[0].x - v[1].y) + kn * (v[2].x - v[3].y);
    const double pi = (v[0].y + v[1].x) + kn * (v[2].y + v[3].x);
    const double mr = (v[0].x + v[1].y) - kn * (v[2].x + v[3].y);
    const double mi = (v[1].x - v[0].y) - kn * (v[3].x - v[2].y);
    // kspace_efield_idm's weight (nb_induction_model.f90:2560-2600), applied before the merge
    const int kp = n - K.nlo, km = -n - K.nlo;
    if (kp >= 0 && kp < K.len) {
      const int k = K.kbeg + kp;
      const double g = -4.0 * A.kv[k].ak;
      atomicAdd(&A.sk[(size_t)k * 4 + 2 * A.par], g * pr);
      atomicAdd(&A.sk[(size_t)k * 4 + 2 * A.par + 1], g * pi);
    }
    if (n > 0 && km >= 0 && km < K.len) {
      const int k = K.kbeg + km;
      const double g = -4.0 * A.kv[k].ak;
      atomicAdd(&A.sk[(size_t)k * 4 + 2 * A.par], g * mr);
      atomicAdd(&A.sk[(size_t)k * 4 + 2 * A.par + 1], g * mi);
    }
  }
}

// Gather and update: a block takes MT tiles of 8 sites, its warps the tiles of four rows in turn.
// Per tile a lane builds the operands of its row and n (columns Re, Im of Q and of Q_z) from
// S(n) and S(-n), loaded a tile ahead; then lane l holds Q and Q_z of site l / 4 and row l % 4
// and contracts them with XY.  The sites' (cos, sin)(n z) stay in registers; they and the first
// tile's XY and row are loaded before the wait for the step's first kernel, and the values of
// the update right after it.  The update is k_iter_b's.
template <bool PCG, int J, int MT>
__global__ void __launch_bounds__(kRowWarps * 32) k_iter_b_rows(IterArgs A) {
  constexpr int KS = 2 * J;  // steps of two n
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int w0 = blockIdx.x * (8 * MT), ns_blk = min(8 * MT, A.nw - w0);
  double zf[MT][KS];
  int ws[MT];
#pragma unroll
  for (int m = 0; m < MT; m++) {
    ws[m] = min(w0 + 8 * m + (lane >> 2), A.nw - 1);
    const double *z = A.Zc + (size_t)ws[m] * A.zs + (lane & 3);
#pragma unroll
    for (int k = 0; k < KS; k++) zf[m][k] = z[4 * k];
  }
  const int nt4 = (A.nrow + 3) / 4;
  // operand element: row lane / 8 of the tile, column part ri (Re, Im), factor part cs (cos, sin)
  const int ri = (lane >> 2) & 1, cs = lane & 1, n0 = (lane >> 1) & 1;
  const double *sk = A.sk + 2 * A.par + (ri ^ cs);  // the part of S that the element combines
  double kn[KS];  // k_n, with the sign of the element's Q_z
  const double sg = cs == 0 && ri == 1 ? -1.0 : 1.0;
#pragma unroll
  for (int k = 0; k < KS; k++) kn[k] = sg * A.rn[min(2 * k + n0, A.nmax) + A.nmax];
  double2 xy[MT];
  double rl = 0.0, rm = 0.0;
  KRow K{};
  int ks_next = 0;
  auto load_rows = [&](int t) {  // fixed during the solve
    const KRow &R = A.rows[min(4 * t + (lane & 3), A.nrow - 1)];
    rl = R.rl;
    rm = R.rm;
#pragma unroll
    for (int m = 0; m < MT; m++)
      xy[m] = A.XYr[((size_t)(t >> 1) * A.nw + ws[m]) * 8 + 4 * (t & 1) + (lane & 3)];
  };
  auto load_row = [&](int t) {
    const int r = 4 * t + (lane >> 3);
    K = A.rows[min(r, A.nrow - 1)];
    ks_next = warp_max(K.nlo + K.len - 1) / 2 + 1;
    if (r >= A.nrow) K.len = 0;
  };
  double p[KS], q[KS];  // S(n) and S(-n)
  auto load_s = [&]() {
#pragma unroll
    for (int k = 0; k < KS; k++) {
      const int n = 2 * k + n0, kp = n - K.nlo, km = -n - K.nlo;
      p[k] = kp >= 0 && kp < K.len ? sk[(size_t)(K.kbeg + kp) * 4] : 0.0;
      q[k] = n > 0 && km >= 0 && km < K.len ? sk[(size_t)(K.kbeg + km) * 4] : 0.0;
    }
  };
  if (wid < nt4) {
    load_row(wid);
    load_rows(wid);
  }
  pdl_wait();  // T.mu, S(k) and the step scalars of this step's first kernel
  const double finished = A.state[kIterFinished];
  if (wid < nt4) load_s();
  if (finished != 0.0) return;  // finished in an earlier step of this pass
  double ex[MT], ey[MT], ez[MT];
#pragma unroll
  for (int m = 0; m < MT; m++) ex[m] = ey[m] = ez[m] = 0.0;
  for (int t = wid; t < nt4; t += kRowWarps) {
    const int ks = ks_next;
    double bq[KS], bz[KS];
#pragma unroll
    for (int k = 0; k < KS; k++) {
      const double a = p[k] + q[k], d = p[k] - q[k];
      bq[k] = sg * (cs == 0 ? a : d);
      bz[k] = kn[k] * (cs == 0 ? d : a);
    }
    double2 x[MT];
#pragma unroll
    for (int m = 0; m < MT; m++) x[m] = xy[m];
    const double l = rl, mm = rm;
    if (t + kRowWarps < nt4) {
      load_row(t + kRowWarps);
      load_s();
      load_rows(t + kRowWarps);
    }
    double2 Q[MT], Z[MT];
#pragma unroll
    for (int m = 0; m < MT; m++) Q[m] = Z[m] = make_double2(0.0, 0.0);
#pragma unroll
    for (int k = 0; k < KS; k++)
      if (k < ks)
#pragma unroll
        for (int m = 0; m < MT; m++) {
          dmma(Q[m], zf[m][k], bq[k]);
          dmma(Z[m], zf[m][k], bz[k]);
        }
#pragma unroll
    for (int m = 0; m < MT; m++) {  // rows past the last have XY = 0
      const double a = x[m].x * Q[m].x - x[m].y * Q[m].y;
      ex[m] += l * a;
      ey[m] += mm * a;
      ez[m] += x[m].x * Z[m].x - x[m].y * Z[m].y;
    }
  }
  pdl_launch_dependents();  // the gather, the bulk of the kernel, is done
  __shared__ double part[kRowWarps][3][8 * MT];
#pragma unroll
  for (int m = 0; m < MT; m++) {
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
      ex[m] += __shfl_xor_sync(0xffffffffu, ex[m], o);
      ey[m] += __shfl_xor_sync(0xffffffffu, ey[m], o);
      ez[m] += __shfl_xor_sync(0xffffffffu, ez[m], o);
    }
    if ((lane & 3) == 0) {
      part[wid][0][8 * m + (lane >> 2)] = ex[m];
      part[wid][1][8 * m + (lane >> 2)] = ey[m];
      part[wid][2][8 * m + (lane >> 2)] = ez[m];
    }
  }
  __syncthreads();
  const auto ek = [&](int g, int c) {
    double v = 0.0;
    for (int u = 0; u < kRowWarps; u++) v += part[u][c][g];
    return v;
  };
  if constexpr (PCG)
    pcg_update(A, w0, ns_blk, ek);
  else
    jacobi_update(A, w0, ns_blk, ek);
}

// ------------------------------------------------------------------ the solve in one cluster
// Small boxes: the whole Jacobi solve as one kernel, a thread-block cluster whose blocks own ns
// polarisable sites each.  A step of so few sites is a chain of latencies (two launches, the
// loads after them, atomics and a ticket: 10.5 us at 37 waters, of which the sums take less
// than one).  Here every block holds what it needs of the tables for the whole solve in shared
// memory (its sites' tensor entries and phase factors, one row tile's phase factors of all
// sites), all dipoles and all S(k) combinations; it receives the other blocks' parts of those
// by distributed shared memory, and a step has two cluster barriers:
//   - four warps take the block's (row tile, n tile), a share of the sites each, as in
//     k_iter_a_rows; the others take T.mu of the block's sites;
//   - barrier; the gather of the block's sites, a tile of four rows per warp, as in
//     k_iter_b_rows, and the update; barrier.
// The change of a step is summed beside the next step's first half, which is thrown away after
// the last one.  Every block forms the total from the blocks' sums in the same order, so all
// leave together.
// 37 waters, 27 steps: 139 us (275 as step kernels); what remains is latency, 5 us a step, of
// which 1.8 are the two barriers with the stores that they wait for.  The form ends where a
// block's tables no longer fit its shared memory (some 45 waters): with the tables left in
// global memory a step took longer than its two kernels (473 us against 327 at 128 waters).
constexpr int kCluThreads = 512, kCluWarps = kCluThreads / 32, kCluRowWarps = 4;
constexpr int kCluTiles = 2;  // site tiles of 8 per block, at most
constexpr int kCluMax = 16;   // blocks of the cluster
static_assert(kCluMax * kCluTiles <= 32, "a lane per block and tile");
constexpr size_t kCluSmem = 227 * 1024 - 64;

__host__ __device__ constexpr int clu_sites(int nw) { return ((nw + kCluMax - 1) / kCluMax + 7) / 8 * 8; }
constexpr int kCluRed = kCluWarps * 3 * 8 * kCluTiles > kCluRowWarps * 4 * 64
                            ? kCluWarps * 3 * 8 * kCluTiles
                            : kCluRowWarps * 4 * 64;
struct CluSmem {  // offsets in doubles
  int ld, nwp, mu, ad, red, xyt, zt, xy, z, t4, tb, src, eim, slot, total;
  __host__ __device__ CluSmem(int J, int nw, int nrow) {
    const int ns = clu_sites(nw), nr8 = (nrow + 7) / 8 * 8;
    ld = 16 * J + 8;  // 64 bytes past a multiple of 128: two rows' elements in distinct banks
    nwp = (nw + 31) / 32 * 32;  // sites and tensor entries, padded with zeros
    mu = 0;                              // double4 [nwp]
    t4 = mu + 4 * nwp;                   // double4 [ns][nwp]: a site's entries, at most one per site
    ad = t4 + 4 * ns * nwp;              // [nr8][ld]: (S(n) + S(-n), S(n) - S(-n))
    red = ad + nr8 * ld;                 // the warps' sums, of either half step
    xyt = red + kCluRed;                 // double2 [nw][8]: the row tile's
    zt = xyt + 16 * nw;                  // [nw][8]: the n tile's
    xy = zt + 8 * nw;         // double2 [nr8][ns]: the block's sites'
    z = xy + 2 * nr8 * ns;               // [ns][8 J + 2]
    tb = z + ns * (8 * J + 2);           // [ns][nwp]
    src = tb + ns * nwp;                 // int [ns][nwp]
    eim = src + ns * nwp / 2;            // [ns][4]
    slot = eim + 4 * ns;                 // [2][32] change by step parity, [32] energy, the flag
    total = slot + 3 * 32 + 2;
  }
};

template <int J>
__global__ void __launch_bounds__(kCluThreads) k_dip_cluster(IterArgs A) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  extern __shared__ double4 clu4[];
  double *sm = reinterpret_cast<double *>(clu4);
  const int me = (int)cl.block_rank();
  const CluSmem L(J, A.nw, A.nrow);
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nw = A.nw;
  const int ns = clu_sites(nw), w0 = me * ns, nloc = min(max(nw - w0, 0), ns);
  const int nt8 = (A.nrow + 7) / 8, nt4 = (A.nrow + 3) / 4, mt = ns / 8;
  double4 *mu = clu4, *T4 = reinterpret_cast<double4 *>(sm + L.t4);
  double *AD = sm + L.ad, *Zt = sm + L.zt, *Zs = sm + L.z, *TB = sm + L.tb, *eim = sm + L.eim;
  double2(*red)[4][32] = reinterpret_cast<double2(*)[4][32]>(sm + L.red);
  double(*part)[3][8 * kCluTiles] = reinterpret_cast<double(*)[3][8 * kCluTiles]>(sm + L.red);
  double2 *XYt = reinterpret_cast<double2 *>(sm + L.xyt), *XYs = reinterpret_cast<double2 *>(sm + L.xy);
  int *src = reinterpret_cast<int *>(sm + L.src);
  double *slot = sm + L.slot;
  volatile int *more = reinterpret_cast<int *>(slot + 3 * 32);
  constexpr int kZs = 8 * J + 2, KS = 2 * J;
  const int rt = me % nt8, jn = me / nt8;  // the block's row tile and n tile
  const bool rows_here = jn < J;

  // ---- the tables, and the first step from mu = 0 (as k_dip_first) in every block alike
  double ch = 0.0, en = 0.0;
  for (int w = tid; w < L.nwp; w += kCluThreads) {
    double m[3] = {0.0, 0.0, 0.0};
    if (w < nw) {
      const double polr = A.S.apol[w % A.np];
      double E0[3];
      for (int c = 0; c < 3; c++) {
        E0[c] = A.e0[(size_t)w * 3 + c];
        m[c] = polr * E0[c];
        ch += m[c] * m[c];
      }
      en += -0.5 * polr * (E0[0] * E0[0] + E0[1] * E0[1] + E0[2] * E0[2]);
    }
    mu[w] = make_double4(m[0], m[1], m[2], 0.0);
  }
  ch = warp_sum(ch);
  en = warp_sum(en);
  double *wsum = sm + L.red;
  if (lane == 0) {
    wsum[wid] = ch;
    wsum[kCluWarps + wid] = en;
  }
  for (int g = wid; g < nloc; g += kCluWarps) {
    const int w = w0 + g, i = w / A.np;
    const int n_ent = min(A.ncnt[i] * A.np, nw - A.np);
    const size_t base = (size_t)w * A.cap * A.np;
    for (int e = lane; e < L.nwp; e += 32) {
      double4 t = make_double4(0.0, 0.0, 0.0, 0.0);
      double b = 0.0;
      int q = 0;
      if (e < A.np) {  // the intramolecular entries first
        t = A.S4[(size_t)w * A.np + e];
        b = A.SB[(size_t)w * A.np + e];
        q = i * A.np + e;
      } else if (e - A.np < n_ent) {
        const int n = (e - A.np) / A.np;
        t = A.T4[base + e - A.np];
        b = A.TB[base + e - A.np];
        q = A.nbr[(size_t)i * A.cap + n] * A.np + (e - A.np) - n * A.np;
      }
      T4[g * L.nwp + e] = t;
      TB[g * L.nwp + e] = b;
      src[g * L.nwp + e] = q;
    }
  }
  if (rows_here) {
    for (int u = tid; u < nw * 8; u += kCluThreads) XYt[u] = A.XYr[(size_t)rt * nw * 8 + u];
    for (int u = tid; u < nw * 8; u += kCluThreads) Zt[u] = A.Zc[(size_t)(u >> 3) * A.zs + 8 * jn + (u & 7)];
  }
  for (int u = tid; u < nt8 * 8 * ns; u += kCluThreads) {
    const int r = u / ns, g = u - r * ns;
    XYs[u] = A.XYr[((size_t)(r >> 3) * nw + min(w0 + g, nw - 1)) * 8 + (r & 7)];
  }
  for (int u = tid; u < ns * 8 * J; u += kCluThreads) {
    const int g = u / (8 * J), c = u - g * (8 * J);
    Zs[g * kZs + c] = A.Zc[(size_t)min(w0 + g, nw - 1) * A.zs + c];
  }
  for (int u = tid; u < nt8 * 8 * L.ld; u += kCluThreads) AD[u] = 0.0;
  // structure factors: the lane's row, the warp's sites, and the thread's (row, n) at the end
  double rl = 0.0, rm = 0.0, kn_a = 0.0, gp = 0.0, gm = 0.0;
  const int fin_row = rt * 8 + (lane >> 2), fin_n = 4 * jn + (lane & 3);
  bool fin = false;
  if (rows_here && wid < kCluRowWarps) {
    const KRow R = A.rows[min(fin_row, A.nrow - 1)];
    rl = R.rl;
    rm = R.rm;
    fin = fin_row < A.nrow && fin_n <= A.nmax;
    if (fin) {
      const int kp = fin_n - R.nlo, km = -fin_n - R.nlo;
      kn_a = A.rn[fin_n + A.nmax];
      // kspace_efield_idm's weights (nb_induction_model.f90:2560-2600)
      if (kp >= 0 && kp < R.len) gp = -4.0 * A.kv[R.kbeg + kp].ak;
      if (fin_n > 0 && km >= 0 && km < R.len) gm = -4.0 * A.kv[R.kbeg + km].ak;
    }
  }
  const int spw = ((nw + kCluRowWarps - 1) / kCluRowWarps + 3) / 4 * 4;  // sites of a row warp
  const int q0 = wid * spw + (lane & 3);
  const int steps = wid < kCluRowWarps ? min(spw, max(nw - wid * spw, 0) + 3) / 4 : 0;
  // gather: the warp's tile of four rows
  const int ri = (lane >> 2) & 1, cs = lane & 1, n0 = (lane >> 1) & 1;
  const double sg = cs == 0 && ri == 1 ? -1.0 : 1.0;
  const double *ad = AD + (4 * wid + (lane >> 3)) * L.ld + 4 * n0 + (ri ^ cs);
  double gl = 0.0, gmm = 0.0, kn[KS];
  int ks = 0;
  if (wid < nt4) {
    const KRow K = A.rows[min(4 * wid + (lane >> 3), A.nrow - 1)];
    ks = warp_max(K.nlo + K.len - 1) / 2 + 1;
    const KRow R = A.rows[min(4 * wid + (lane & 3), A.nrow - 1)];
    gl = R.rl;
    gmm = R.rm;
  }
#pragma unroll
  for (int k = 0; k < KS; k++) kn[k] = sg * A.rn[min(2 * k + n0, A.nmax) + A.nmax];
  // update: warp m takes site tile m, lane (component, site)
  const int uc = lane >> 3, ug = 8 * wid + (lane & 7), uw = w0 + ug;
  const bool upd = wid < mt && uc < 3 && ug < nloc;
  const double polr = upd ? A.S.apol[uw % A.np] : 0.0;
  const double e0 = upd ? A.e0[(size_t)uw * 3 + uc] : 0.0;
  __syncthreads();
  double chg = 0.0, ene = 0.0;  // of step `it`
  for (int u = 0; u < kCluWarps; u++) {
    chg += wsum[u];
    ene += wsum[kCluWarps + u];
  }
  int it = 1;
  double e_up = 0.0;  // the lane's part of the energy of its last update
  cl.sync();  // every block runs and has its combinations cleared
  while (it > 1 || (chg > A.thr && it < A.maxit)) {
    if (wid < kCluRowWarps) {
      if (rows_here) {
        double2 acc[4];
#pragma unroll
        for (int c = 0; c < 4; c++) acc[c] = make_double2(0.0, 0.0);
#pragma unroll 4
        for (int t = 0; t < steps; t++) {
          const int q = q0 + 4 * t, w = min(q, nw - 1);  // mu = 0 past the last site
          const double2 xy = XYt[w * 8 + (lane >> 2)];
          const double zf = Zt[w * 8 + (lane >> 2)];
          const double4 m = mu[q];
          const double d = rl * m.x + rm * m.y;
          dmma(acc[0], xy.x * d, zf);
          dmma(acc[1], xy.y * d, zf);
          dmma(acc[2], xy.x * m.z, zf);
          dmma(acc[3], xy.y * m.z, zf);
        }
#pragma unroll
        for (int c = 0; c < 4; c++) red[wid][c][lane] = acc[c];
        asm volatile("bar.sync 1, %0;" ::"n"(kCluRowWarps * 32) : "memory");
        if (fin) {  // in every row warp alike, which serves a share of the blocks
          double2 v[4];
#pragma unroll
          for (int c = 0; c < 4; c++) {
            double2 x[kCluRowWarps];
#pragma unroll
            for (int w = 0; w < kCluRowWarps; w++) x[w] = red[w][c][lane];
            v[c].x = (x[0].x + x[1].x) + (x[2].x + x[3].x);
            v[c].y = (x[0].y + x[1].y) + (x[2].y + x[3].y);
          }
          // B + k_n C (n), B - k_n C (-n), times cos +- i sin
          const double pr = gp * ((v[0].x - v[1].y) + kn_a * (v[2].x - v[3].y));
          const double pi = gp * ((v[0].y + v[1].x) + kn_a * (v[2].y + v[3].x));
          const double mr = gm * ((v[0].x + v[1].y) - kn_a * (v[2].x + v[3].y));
          const double mi = gm * ((v[1].x - v[0].y) - kn_a * (v[3].x - v[2].y));
          const double4 o = make_double4(pr + mr, pi + mi, pr - mr, pi - mi);
          double4 *at = reinterpret_cast<double4 *>(AD + fin_row * L.ld + 4 * fin_n);
#pragma unroll
          for (int b = 0; b < kCluMax; b += kCluRowWarps) *cl.map_shared_rank(at, b + wid) = o;
        }
      }
    } else {
      for (int g = wid - kCluRowWarps; g < nloc; g += kCluWarps - kCluRowWarps) {
        double ex = 0.0, ey = 0.0, ez = 0.0;
#pragma unroll 4
        for (int e = lane; e < L.nwp; e += 32) {
          const double4 T = T4[g * L.nwp + e], m = mu[src[g * L.nwp + e]];
          const double B = TB[g * L.nwp + e], dm = T.w * (T.x * m.x + T.y * m.y + T.z * m.z);
          ex += dm * T.x - B * m.x;
          ey += dm * T.y - B * m.y;
          ez += dm * T.z - B * m.z;
        }
        ex = warp_sum(ex);
        ey = warp_sum(ey);
        ez = warp_sum(ez);
        if (lane == 0) {
          eim[4 * g] = ex;
          eim[4 * g + 1] = ey;
          eim[4 * g + 2] = ez;
        }
      }
    }
    cl.sync();  // all combinations are here, and no block reads the dipoles any more
    {
      double bq[KS], bz[KS];
#pragma unroll
      for (int k = 0; k < KS; k++) {
        const double a = wid < nt4 ? ad[8 * k] : 0.0, d = wid < nt4 ? ad[8 * k + 2] : 0.0;
        bq[k] = sg * (cs == 0 ? a : d);
        bz[k] = kn[k] * (cs == 0 ? d : a);
      }
#pragma unroll
      for (int m = 0; m < kCluTiles; m++) {
        if (m < mt) {
          const int g = 8 * m + (lane >> 2);
          const double *z = Zs + g * kZs + (lane & 3);
          double2 Q = make_double2(0.0, 0.0), Z = Q;
#pragma unroll
          for (int k = 0; k < KS; k++)
            if (k < ks) {
              const double zf = z[4 * k];
              dmma(Q, zf, bq[k]);
              dmma(Z, zf, bz[k]);
            }
          double2 x = make_double2(0.0, 0.0);  // and 0 past the last row
          if (wid < nt4) x = XYs[(4 * wid + (lane & 3)) * ns + g];
          const double a = x.x * Q.x - x.y * Q.y;
          double ex = gl * a, ey = gmm * a, ez = x.x * Z.x - x.y * Z.y;
#pragma unroll
          for (int o = 1; o < 4; o <<= 1) {
            ex += __shfl_xor_sync(0xffffffffu, ex, o);
            ey += __shfl_xor_sync(0xffffffffu, ey, o);
            ez += __shfl_xor_sync(0xffffffffu, ez, o);
          }
          if ((lane & 3) == 0) {
            part[wid][0][g] = ex;
            part[wid][1][g] = ey;
            part[wid][2][g] = ez;
          }
        }
      }
    }
    if (it > 1 && wid == kCluWarps - 1) {  // the change of the last update
      double v = lane < kCluMax * mt ? slot[32 * (it & 1) + lane] : 0.0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      chg = v;
      if (lane == 0) *more = v > A.thr && it < A.maxit;
    }
    __syncthreads();
    if (it > 1 && !*more) break;
    double c = 0.0;
    if (upd) {
      double p[kCluWarps];
#pragma unroll
      for (int u = 0; u < kCluWarps; u++) p[u] = part[u][uc][ug];
#pragma unroll
      for (int o = kCluWarps / 2; o > 0; o >>= 1)
#pragma unroll
        for (int u = 0; u < o; u++) p[u] += p[u + o];
      double *at = reinterpret_cast<double *>(mu + uw) + uc;
      const double Et = (eim[4 * ug + uc] + p[0]) + e0, m = polr * Et, d = *at - m;
#pragma unroll
      for (int b = 0; b < kCluMax; b++) *cl.map_shared_rank(at, b) = m;
      c = d * d;
      e_up = -0.5 * polr * (Et * e0);
    }
    it++;
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    if (wid < mt) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
      // read after the next step's first barrier, which orders it; by parity, since a slow
      // block may still be reading the previous step's
      if (lane < kCluMax) *cl.map_shared_rank(slot + 32 * (it & 1) + me * mt + wid, lane) = c;
    }
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");  // the new dipoles are here
  }
  if (it > 1) {  // the last update's sums: the change is warp kCluWarps - 1's
    if (wid < mt) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) e_up += __shfl_xor_sync(0xffffffffu, e_up, o);
      if (lane == 0) *cl.map_shared_rank(slot + 64 + me * mt + wid, 0) = e_up;
    }
    cl.sync();
  }
  for (int u = tid; u < nloc * 3; u += kCluThreads) {
    const double4 m = mu[w0 + u / 3];
    A.mu[(size_t)w0 * 3 + u] = u % 3 == 0 ? m.x : (u % 3 == 1 ? m.y : m.z);
  }
  if (me == 0 && tid == kCluThreads - 32) {
    if (it > 1) {
      ene = 0.0;
      for (int u = 0; u < kCluMax * mt; u++) ene += slot[64 + u];
    }
    A.state[kIterIters] = (double)it;
    A.state[kIterChange] = chg;
    A.state[kIterEnergy] = ene;
    A.state[kIterFinished] = 1.0;
  }
}

// ------------------------------------------------------------------ the solve in one grid
// Middle sizes: the whole solve as one cooperative kernel, a block per SM that owns ns sites.
// A step as two kernels costs 5 us per kernel before any work (launch, first loads, the
// reduction's end), and beside the three-body kernels, whose blocks fill the SMs, each launch
// also waits for its blocks' slots; here the blocks keep half of every SM for the solve, the
// constant operands of a step are under way before the step begins, and a step has two grid
// barriers.  Warps 0-3 of a block take (row tile, site chunk) units of the structure factors,
// as k_iter_a_rows, warps 4-7 T.mu of the block's sites; after the barrier all gather the
// block's sites over the rows, as k_iter_b_rows, and update them.  S(k) is kept as the
// combinations that the gather takes, AD[row][n][(re), (im)] = (S(n) + S(-n), S(n) - S(-n)).
// Data of other blocks is read past L1 (__ldcg).  A barrier's wait is bounded: a block that
// waits longer marks the solve as failed and leaves, and the host takes the step kernels.
// Loop, alone / in the evaluation: 128 waters (29 steps) 327 / 421 us as step kernels, 247 / 329
// here; 512 (28 steps) 562 / 1220, 424 / 506; 512, PCG 293 / 972, 205 / 255.  Of a step's 15 us
// at 512 waters the vector and T.mu take 6.8, the gather 3.7 and the two barriers 3.8 (release
// and acquire through L2; polls without acquire took longer).  The form ends where the vector
// and the operands no longer fit in shared memory.
constexpr int kGridThreads = 256, kGridWarps = kGridThreads / 32, kGridRowWarps = 4;
constexpr int kGridSub = 16;     // sites that a row warp stages at a time
constexpr int kGridStages = 4;  // stages of its ring, where a step's operands do not all stay
constexpr int kGridEnt = 5;     // tensor entries that a lane has under way
constexpr int kGridXs = 18;                    // doubles per staged site's XY (8 rows + padding)

struct GridSmem {  // offsets in doubles
  int v, ring, red, part, z, rn, eim, own, src, total, ns8;
  __host__ __device__ GridSmem(int J, int nw, int ns, int ent, int stages) {
    const int kz = 8 * J + 2;
    ns8 = (ns + 7) / 8 * 8;
    v = 0;                                                   // [nw + 64][3] the multiplied vector
    ring = (3 * (nw + 64) + 1) / 2 * 2;                      // [warp][stage][16][kGridXs + kz]
    red = ring + kGridRowWarps * stages * kGridSub * (kGridXs + kz);
    part = red + kGridRowWarps * 4 * J * 64;                 // [warps][3][16]
    z = part + kGridWarps * 3 * 16;                          // [ns8][kz]
    rn = z + ns8 * kz;                                       // [4 J]
    eim = rn + 4 * J;                                        // [ns][3]
    own = eim + 3 * ns;                                      // [ns][3] reciprocal field
    src = own + 3 * ns;                                      // 16 bits [ns][ent], then int [ns]
    total = src + (ns * ent + 3) / 4 + (ns + 1) / 2;
  }
};

__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   (unsigned)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// All blocks' writes before are visible to all blocks after; false when the wait ran out, after
// `polls` of about half a us each.
__device__ __forceinline__ bool grid_barrier(unsigned *bar, unsigned target, unsigned polls,
                                             int *ok) {
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
    unsigned seen = 0, spins = 0;
    do {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(bar) : "memory");
    } while (seen < target && ++spins < polls);
    *ok = seen >= target;
  }
  __syncthreads();
  return *ok != 0;
}

template <bool PCG, int J>
__global__ void __launch_bounds__(kGridThreads, 2) k_dip_grid(IterArgs A, GridArgs G) {
  constexpr int KS = 2 * J, kZs = 8 * J + 2, kStage = kGridSub * (kGridXs + kZs), kN4 = 4 * J;
  extern __shared__ double4 smu4[];
  double *sm = reinterpret_cast<double *>(smu4);
  __shared__ int ok;
  const int ns = G.ns;
  const int ent = A.cap * A.np;
  const GridSmem L(J, A.nw, ns, ent, G.stages);
  double *v = sm + L.v, *Zs = sm + L.z, *eim = sm + L.eim, *own = sm + L.own, *rn = sm + L.rn;
  unsigned short *src = reinterpret_cast<unsigned short *>(sm + L.src);
  int *n_ent = reinterpret_cast<int *>(sm + L.src + (ns * ent + 3) / 4);
  __shared__ int ticket;
  double2(*red)[4 * J][32] = reinterpret_cast<double2(*)[4 * J][32]>(sm + L.red);
  double(*part)[3][16] = reinterpret_cast<double(*)[3][16]>(sm + L.part);
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int w0 = blockIdx.x * ns, nloc = min(max(A.nw - w0, 0), ns);
  const int nt8 = (A.nrow + 7) / 8, nt4 = (A.nrow + 3) / 4, nr8 = 8 * nt8;
  const int n_unit = nt8 * G.nchunk;
  const size_t ad_len = (size_t)nr8 * kN4 * 4;
  unsigned target = 0;

  for (int u = tid; u < L.ns8 * 4 * J; u += kGridThreads) {
    const int g = u / (4 * J), c = u - g * (4 * J);
    *reinterpret_cast<double2 *>(Zs + g * kZs + 2 * c) = reinterpret_cast<const double2 *>(
        A.Zc + (size_t)min(w0 + g, A.nw - 1) * A.zs)[c];
  }
  for (int n = tid; n < 4 * J; n += kGridThreads) rn[n] = A.rn[min(n, A.nmax) + A.nmax];
  for (int u = 3 * A.nw + tid; u < 3 * (A.nw + 64); u += kGridThreads) v[u] = 0.0;
  for (int g = wid; g < nloc; g += kGridWarps) {  // source sites of the block's tensor entries
    const int i = (w0 + g) / A.np, n = min(A.ncnt[i], A.cap) * A.np;
    for (int e = lane; e < n; e += 32)
      src[g * ent + e] = (unsigned short)(A.nbr[(size_t)i * A.cap + e / A.np] * A.np + e % A.np);
    if (lane == 0) n_ent[g] = n;
  }
  // the block's sites at the start: the first Jacobi step (as k_dip_first), or PCG's zero
  // iterate (as k_pcg_first)
  {
    double ch = 0.0, en = 0.0;
    for (int u = tid; u < 3 * nloc; u += kGridThreads) {
      const size_t o = (size_t)w0 * 3 + u;
      const double e0 = A.e0[o], m = A.S.apol[(w0 + u / 3) % A.np] * e0;
      if (PCG) {
        A.mu[o] = A.cw[o] = A.cs[o] = A.cp[o] = 0.0;
        A.cu[o] = m;
      } else {
        A.mu[o] = m;
        ch += m * m;
        en += -0.5 * m * e0;
      }
    }
    if (!PCG) {
      ch = warp_sum(ch);
      en = warp_sum(en);
      if (lane == 0 && 32 * wid < 3 * nloc) {
        atomicAdd(&G.acc[4 + 0], ch);
        atomicAdd(&G.acc[4 + 1], en);
      }
    }
  }
  // row warps: the constant operands of 16 sites (step sub of a unit) into a stage of the ring
  double *ring = sm + L.ring + wid * G.stages * kStage;
  auto fetch = [&](int unit, int sub, int stage) {
    const int rt = unit / G.nchunk, s0 = (unit - rt * G.nchunk) * G.chunk + sub * 4 * kGridSub + wid * kGridSub;
    double *d = ring + stage * kStage;
    const double2 *xy = A.XYr + (size_t)rt * A.nw * 8;
    for (int u = lane; u < kGridSub * 8; u += 32) {
      const int w = min(s0 + (u >> 3), A.nw - 1);
      cp_async16(d + (u >> 3) * kGridXs + 2 * (u & 7), xy + (size_t)w * 8 + (u & 7));
    }
    for (int u = lane; u < kGridSub * 4 * J; u += 32) {
      const int q = u / (4 * J), c = u - q * (4 * J), w = min(s0 + q, A.nw - 1);
      cp_async16(d + kGridSub * kGridXs + q * kZs + 2 * c, A.Zc + (size_t)w * A.zs + 2 * c);
    }
  };
  const int subs = (G.chunk + 4 * kGridSub - 1) / (4 * kGridSub);
  // what the ring takes next: the unit's next sites, the block's next unit and, as the tables
  // stay, the next step's first
  int next_unit = blockIdx.x, next_sub = 0, stage = 0;
  auto fetch_next = [&](int st) {
    fetch(next_unit, next_sub, st);
    cp_async_commit();
    if (++next_sub == subs) {
      next_sub = 0;
      next_unit += gridDim.x;
      if (next_unit >= n_unit) next_unit = blockIdx.x;
    }
  };
  if (wid < kGridRowWarps && (int)blockIdx.x < n_unit) {
    for (int st = 0; st < G.stages; st++) fetch_next(st);
    if (G.stay) cp_async_wait<0>();
  }
  double alpha = 0.0, beta = 0.0, gamma = 0.0, chg = 0.0, ene = 0.0;
  int it = PCG ? 0 : 1;
  bool more = !PCG || A.maxit >= 1;
  const bool started = grid_barrier(G.bar, target += gridDim.x, G.polls, &ok);
  while (started && more) {
    const int par = it & 1;
    double *ad = G.ad + par * ad_len;
    double chg_t = 0.0, ene_t = 0.0;
    if (!PCG) {  // of the last update; the test is below, past the loads that follow
      chg_t = __ldcg(&G.acc[4 * (it % 3)]);
      ene_t = __ldcg(&G.acc[4 * (it % 3) + 1]);
    }
    // the whole vector
    if (PCG) {
      const int m3 = 3 * A.np, dc = kGridThreads % m3;
      int c = tid % m3;  // component in the molecule
#pragma unroll 6
      for (int u = tid; u < 3 * A.nw; u += kGridThreads) {
        v[u] = pcg_u(__ldcg(A.cu + u), pcg_s(__ldcg(A.cw + u), __ldcg(A.cs + u), beta),
                     A.S.apol[c / 3], alpha);
        c += dc;
        if (c >= m3) c -= m3;
      }
    } else {
      for (int u = tid; u < 3 * A.nw / 2; u += kGridThreads)
        cp_async16(v + 2 * u, A.mu + 2 * u);
      cp_async_commit();
      if (tid == 0 && (A.nw & 1)) v[3 * A.nw - 1] = __ldcg(A.mu + 3 * A.nw - 1);
    }
    // the other parity's combinations, last read by the previous step's gather
    for (size_t u = (size_t)blockIdx.x * kGridThreads + tid; u < ad_len / 2;
         u += (size_t)gridDim.x * kGridThreads)
      reinterpret_cast<double2 *>(G.ad + (par ^ 1) * ad_len)[u] = make_double2(0.0, 0.0);
    if (blockIdx.x == 0 && tid < 4) G.acc[4 * ((it + 2) % 3) + tid] = 0.0;
    if (tid == 0) ticket = 0;
    if (!PCG) cp_async_wait<0>();
    __syncthreads();
    if (!PCG) {
      chg = chg_t;
      ene = ene_t;
      if (!(chg > A.thr && it < A.maxit)) break;
    }
    if (wid < kGridRowWarps) {
      for (int unit = blockIdx.x; unit < n_unit; unit += gridDim.x) {
        const int rt = unit / G.nchunk, c0 = (unit - rt * G.nchunk) * G.chunk;
        const int row = rt * 8 + (lane >> 2);
        const KRow R = A.rows[min(row, A.nrow - 1)];
        const int jt = warp_max(R.nlo + R.len - 1) / 4 + 1;
        // kspace_efield_idm's weights (nb_induction_model.f90:2560-2600) of (row, n)
        auto weights = [&](int n, double &gp, double &gm, double &kn) {
          const int kp = n - R.nlo, km = -n - R.nlo;
          gp = kp >= 0 && kp < R.len ? -4.0 * A.kv[R.kbeg + kp].ak : 0.0;
          gm = n > 0 && km >= 0 && km < R.len ? -4.0 * A.kv[R.kbeg + km].ak : 0.0;
          kn = A.rn[min(n, A.nmax) + A.nmax];
        };
        double gp0, gm0, kn0;  // the warp's n tile is wid (and 4 + wid)
        weights(4 * wid + (lane & 3), gp0, gm0, kn0);
        double2 acc[4][J];
#pragma unroll
        for (int c = 0; c < 4; c++)
#pragma unroll
          for (int j = 0; j < J; j++) acc[c][j] = make_double2(0.0, 0.0);
#pragma unroll 1
        for (int sub = 0; sub < subs; sub++) {
          if (!G.stay) {
            cp_async_wait<kGridStages - 1>();
            __syncwarp();
          }
          const double *d = ring + stage * kStage, *xs = d + (lane & 3) * kGridXs + 2 * (lane >> 2),
                       *zs = d + kGridSub * kGridXs + (lane & 3) * kZs + (lane >> 2);
          const int q0 = sub * 4 * kGridSub + wid * kGridSub + (lane & 3);  // in the chunk
          // by the row tile's n tiles: no branch between the products
          auto run = [&](auto jc) {
            constexpr int JT = decltype(jc)::value;
#pragma unroll
            for (int t = 0; t < kGridSub / 4; t++) {
              const int q = q0 + 4 * t;
              const double *m = v + 3 * (q < G.chunk ? min(c0 + q, A.nw) : A.nw);  // zeros past the end
              const double2 xy = *reinterpret_cast<const double2 *>(xs + 4 * t * kGridXs);
              const double dl = R.rl * m[0] + R.rm * m[1], mz = m[2];
              const double a[4] = {xy.x * dl, xy.y * dl, xy.x * mz, xy.y * mz};
#pragma unroll
              for (int j = 0; j < JT; j++) {
                const double z = zs[4 * t * kZs + 8 * j];
#pragma unroll
                for (int c = 0; c < 4; c++) dmma(acc[c][j], a[c], z);
              }
            }
          };
          if (J == 1 || jt == J) run(std::integral_constant<int, J>());
          else if (J == 2 || jt == J - 1) run(std::integral_constant<int, (J > 1 ? J - 1 : 1)>());
          else if (J == 3 || jt == J - 2) run(std::integral_constant<int, (J > 2 ? J - 2 : 1)>());
          else run(std::integral_constant<int, (J > 3 ? J - 3 : 1)>());
          if (!G.stay) {
            __syncwarp();
            fetch_next(stage);
          }
          if (++stage == G.stages) stage = 0;
        }
#pragma unroll
        for (int c = 0; c < 4; c++)
#pragma unroll
          for (int j = 0; j < J; j++) red[wid][c * J + j][lane] = acc[c][j];
        asm volatile("bar.sync 1, %0;" ::"n"(kGridRowWarps * 32) : "memory");
        for (int u = tid; u < jt * 32; u += kGridRowWarps * 32) {
          const int j = u >> 5, n = 4 * j + (lane & 3);
          if (row >= A.nrow || n > A.nmax) continue;
          double2 s[4];
#pragma unroll
          for (int c = 0; c < 4; c++) {
            double2 x[kGridRowWarps];
#pragma unroll
            for (int w = 0; w < kGridRowWarps; w++) x[w] = red[w][c * J + j][lane];
            s[c].x = (x[0].x + x[1].x) + (x[2].x + x[3].x);
            s[c].y = (x[0].y + x[1].y) + (x[2].y + x[3].y);
          }
          double gp = gp0, gm = gm0, kn = kn0;
          if (j != wid) weights(n, gp, gm, kn);
          const double pr = gp * ((s[0].x - s[1].y) + kn * (s[2].x - s[3].y));
          const double pi = gp * ((s[0].y + s[1].x) + kn * (s[2].y + s[3].x));
          const double mr = gm * ((s[0].x + s[1].y) - kn * (s[2].x + s[3].y));
          const double mi = gm * ((s[1].x - s[0].y) - kn * (s[3].x - s[2].y));
          double *o = ad + ((size_t)row * kN4 + n) * 4;
          atomicAdd(o, pr + mr);
          atomicAdd(o + 1, pr - mr);
          atomicAdd(o + 2, pi + mi);
          atomicAdd(o + 3, pi - mi);
        }
        asm volatile("bar.sync 1, %0;" ::"n"(kGridRowWarps * 32) : "memory");
      }
    }
    // T.mu of the block's sites, drawn by the warps one by one
    for (;;) {
      int g = 0;
      if (lane == 0) g = atomicAdd(&ticket, 1);
      g = __shfl_sync(0xffffffffu, g, 0);
      if (g >= nloc) break;
      const int w = w0 + g, n = n_ent[g];
      const double4 *T4 = A.T4 + (size_t)w * ent;
      const double *TB = A.TB + (size_t)w * ent;
      const unsigned short *sg = src + g * ent;
      double ex = 0.0, ey = 0.0, ez = 0.0;
      auto add = [&](const double4 &T, double B, const double *m) {
        const double dm = T.w * (T.x * m[0] + T.y * m[1] + T.z * m[2]);
        ex += dm * T.x - B * m[0];
        ey += dm * T.y - B * m[1];
        ez += dm * T.z - B * m[2];
      };
      if (lane < A.np)
        add(A.S4[(size_t)w * A.np + lane], A.SB[(size_t)w * A.np + lane],
            v + 3 * (w / A.np * A.np + lane));
      for (int e0 = lane; e0 < n + lane; e0 += 32 * kGridEnt) {  // all lanes alike
        double4 t[kGridEnt];
        double b[kGridEnt];
        int q[kGridEnt];
#pragma unroll
        for (int u = 0; u < kGridEnt; u++) {
          const int e = e0 + 32 * u;
          t[u] = make_double4(0.0, 0.0, 0.0, 0.0);
          b[u] = 0.0;
          q[u] = 0;
          if (e < n) {
            t[u] = T4[e];
            b[u] = TB[e];
            q[u] = sg[e];
          }
        }
#pragma unroll
        for (int u = 0; u < kGridEnt; u++) add(t[u], b[u], v + 3 * q[u]);
      }
      ex = warp_sum(ex);
      ey = warp_sum(ey);
      ez = warp_sum(ez);
      if (lane == 0) {
        eim[3 * g] = ex;
        eim[3 * g + 1] = ey;
        eim[3 * g + 2] = ez;
      }
    }
    if (!grid_barrier(G.bar, target += gridDim.x, G.polls, &ok)) break;
    // ---- gather, two tiles of 8 sites at a time
    const int ri = (lane >> 2) & 1, cs = lane & 1, n0 = (lane >> 1) & 1, x = ri ^ cs;
    const double sg = cs == 0 && ri == 1 ? -1.0 : 1.0;
    for (int g0 = 0; g0 < nloc; g0 += 16) {
      const bool two = g0 + 8 < nloc;
      const int wa = min(w0 + g0 + (lane >> 2), A.nw - 1), wb = min(w0 + g0 + 8 + (lane >> 2), A.nw - 1);
      double e[2][3] = {{0.0, 0.0, 0.0}, {0.0, 0.0, 0.0}};
      double2 f[KS], xa, xb;
      double rl = 0.0, rm = 0.0;
      int ks = 0;
      auto load = [&](int t) {
        const double2 *p = reinterpret_cast<const double2 *>(
                               ad + ((size_t)(4 * t + (lane >> 3)) * kN4 + n0) * 4) + x;
#pragma unroll
        for (int k = 0; k < KS; k++) f[k] = __ldcg(p + 4 * k);
        const KRow &Rb = A.rows[min(4 * t + (lane >> 3), A.nrow - 1)];
        ks = Rb.nlo + Rb.len - 1;
        const KRow &Ra = A.rows[min(4 * t + (lane & 3), A.nrow - 1)];
        rl = Ra.rl;
        rm = Ra.rm;
        const double2 *xy = A.XYr + (size_t)(t >> 1) * A.nw * 8 + 4 * (t & 1) + (lane & 3);
        xa = xy[(size_t)wa * 8];
        xb = xy[(size_t)wb * 8];
      };
      if (wid < nt4) load(wid);
      for (int t = wid; t < nt4; t += kGridWarps) {
        const int kl = warp_max(ks) / 2 + 1;
        double bq[KS], bz[KS];
#pragma unroll
        for (int k = 0; k < KS; k++) {
          const double kn = rn[2 * k + n0];
          bq[k] = sg * (cs == 0 ? f[k].x : f[k].y);
          bz[k] = kn * (sg * (cs == 0 ? f[k].y : f[k].x));
        }
        const double2 ya = xa, yb = xb;
        const double l = rl, m = rm;
        if (t + kGridWarps < nt4) load(t + kGridWarps);
        const double *za = Zs + (g0 + (lane >> 2)) * kZs + (lane & 3), *zb = za + 8 * kZs;
        double2 Qa = make_double2(0.0, 0.0), Za = Qa, Qb = Qa, Zb = Qa;
        auto run = [&](auto kc) {  // by two steps of n: no branch between the products
          constexpr int KT = decltype(kc)::value;
          if (two) {
#pragma unroll
            for (int k = 0; k < KT; k++) {
              const double z = za[4 * k], z2 = zb[4 * k];
              dmma(Qa, z, bq[k]);
              dmma(Za, z, bz[k]);
              dmma(Qb, z2, bq[k]);
              dmma(Zb, z2, bz[k]);
            }
          } else {
#pragma unroll
            for (int k = 0; k < KT; k++) {
              const double z = za[4 * k];
              dmma(Qa, z, bq[k]);
              dmma(Za, z, bz[k]);
            }
          }
        };
        if (J == 1 || kl > KS - 2) run(std::integral_constant<int, KS>());
        else if (J == 2 || kl > KS - 4) run(std::integral_constant<int, (J > 1 ? KS - 2 : KS)>());
        else if (J == 3 || kl > KS - 6) run(std::integral_constant<int, (J > 2 ? KS - 4 : KS)>());
        else run(std::integral_constant<int, (J > 3 ? KS - 6 : KS)>());
        const double a = ya.x * Qa.x - ya.y * Qa.y, b = yb.x * Qb.x - yb.y * Qb.y;
        e[0][0] += l * a;
        e[0][1] += m * a;
        e[0][2] += ya.x * Za.x - ya.y * Za.y;
        e[1][0] += l * b;
        e[1][1] += m * b;
        e[1][2] += yb.x * Zb.x - yb.y * Zb.y;
      }
#pragma unroll
      for (int h = 0; h < 2; h++)
#pragma unroll
        for (int c = 0; c < 3; c++) {
#pragma unroll
          for (int o = 1; o < 4; o <<= 1) e[h][c] += __shfl_xor_sync(0xffffffffu, e[h][c], o);
          if ((lane & 3) == 0) part[wid][c][8 * h + (lane >> 2)] = e[h][c];
        }
      __syncthreads();
      if (tid < 48) {
        const int g = g0 + tid / 3, c = tid - tid / 3 * 3;
        if (g < nloc) {
          double s = 0.0;
#pragma unroll
          for (int u = 0; u < kGridWarps; u++) s += part[u][c][tid / 3];
          own[3 * g + c] = s;
        }
      }
      __syncthreads();
    }
    // ---- update of the block's sites, a thread per component
    {
      double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
      for (int u = tid; u < 3 * nloc; u += kGridThreads) {
        const size_t o = (size_t)w0 * 3 + u;
        const double ap = A.S.apol[(w0 + u / 3) % A.np], e0 = A.e0[o];
        if (PCG) {  // the operations of pcg_update
          const double u0 = A.cu[o], sn = pcg_s(A.cw[o], A.cs[o], beta);
          const double p = __fma_rn(beta, A.cp[o], u0), xx = __fma_rn(alpha, p, A.mu[o]);
          const double un = pcg_u(u0, sn, ap, alpha), wv = un / ap - (eim[u] + own[u]);
          A.cs[o] = sn;
          A.cp[o] = p;
          A.mu[o] = xx;
          A.cu[o] = un;
          A.cw[o] = wv;
          s0 += un * un / ap;
          s1 += wv * un;
          s2 += un * un;
          s3 += -0.5 * xx * e0;
        } else {
          const double Et = (eim[u] + own[u]) + e0, m = ap * Et, d = v[o] - m;
          A.mu[o] = m;
          s0 += d * d;
          s1 += -0.5 * ap * (Et * e0);
        }
      }
      if (32 * wid < 3 * nloc) {
        double *acc = G.acc + 4 * ((it + 1) % 3);
        s0 = warp_sum(s0);
        s1 = warp_sum(s1);
        if (PCG) {
          s2 = warp_sum(s2);
          s3 = warp_sum(s3);
        }
        if (lane == 0) {
          atomicAdd(acc, s0);
          atomicAdd(acc + 1, s1);
          if (PCG) {
            atomicAdd(acc + 2, s2);
            atomicAdd(acc + 3, s3);
          }
        }
      }
    }
    it++;
    if (!grid_barrier(G.bar, target += gridDim.x, G.polls, &ok)) break;
    if (PCG) {  // every block closes the step alike (pcg_update)
      const double *acc = G.acc + 4 * (it % 3);
      const double g1 = __ldcg(acc), d1 = __ldcg(acc + 1);
      chg = __ldcg(acc + 2);
      ene = __ldcg(acc + 3);
      more = chg > A.thr && it < A.maxit;
      if (more) {
        const double b = it == 1 ? 0.0 : g1 / gamma;
        const double a = it == 1 ? g1 / d1 : g1 / (d1 - b * g1 / alpha);
        if (a > 0.0 && a < 1e300) {
          alpha = a;
          beta = b;
          gamma = g1;
        } else {  // breakdown (not positive definite): reported as no convergence
          it = A.maxit;
          more = false;
        }
      }
    }
  }
  cp_async_wait<0>();
  if (tid == 0) {
    if (!ok) {
      A.state[kIterFinished] = -1.0;
    } else if (blockIdx.x == 0) {
      A.state[kIterIters] = (double)it;
      A.state[kIterChange] = chg;
      A.state[kIterEnergy] = ene;
      A.state[kIterFinished] = 1.0;
    }
  }
}

// The first Jacobi step from mu = 0 (nb_induction_model.f90:1317-1359), where T.mu and the
// reciprocal field are zero: mu = alpha E0, with the change and energy sums the full step
// forms, in one block.  It records iteration 1 in the state and, inside the graph, sets the
// WHILE node's condition, so the loop starts at the second step.
constexpr int kFirstThreads = 1024;
__global__ void __launch_bounds__(kFirstThreads) k_dip_first(IterArgs A) {
  double ch = 0.0, en = 0.0;
  for (int w = threadIdx.x; w < A.nw; w += kFirstThreads) {
    const double polr = A.S.apol[w % A.np];
    double Et[3], E0[3];
    for (int c = 0; c < 3; c++) {
      const size_t o = (size_t)w * 3 + c;
      E0[c] = A.e0[o];
      Et[c] = (0.0 + 0.0) + E0[c];
      const double m = polr * Et[c];
      const double d = 0.0 - m;
      ch += d * d;
      A.mu[o] = m;
    }
    en += -0.5 * polr * (Et[0] * E0[0] + Et[1] * E0[1] + Et[2] * E0[2]);
  }
  __shared__ double red[2][kFirstThreads / 32];
  ch = warp_sum(ch);
  en = warp_sum(en);
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = ch;
    red[1][threadIdx.x >> 5] = en;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double chg = 0.0, ene = 0.0;
    for (int u = 0; u < kFirstThreads / 32; u++) {
      chg += red[0][u];
      ene += red[1][u];
    }
    A.state[kIterIters] = 1.0;
    A.state[kIterChange] = chg;
    A.state[kIterEnergy] = ene;
    const bool more = chg > A.thr && 1 < A.maxit;
    A.state[kIterFinished] = more ? 0.0 : 1.0;
    if (A.use_graph) cudaGraphSetConditional(A.handle, more ? 1u : 0u);
  }
}

// The start of the PCG solve: x = 0, u = alpha E0 (the Jacobi first step's dipoles), w, s
// and p zero and the step scalars zero, so that the first step forms w = A u and its scalars
// from them (k_iter_a/k_iter_b with PCG); inside the graph it lets the WHILE node run.
__global__ void __launch_bounds__(kFirstThreads) k_pcg_first(IterArgs A) {
  for (int o = threadIdx.x; o < A.nw * 3; o += kFirstThreads) {
    A.mu[o] = 0.0;
    A.cu[o] = A.S.apol[(o / 3) % A.np] * A.e0[o];
    A.cw[o] = 0.0;
    A.cs[o] = 0.0;
    A.cp[o] = 0.0;
  }
  if (threadIdx.x == 0) {
    for (int k = 0; k < kIterStateLen; k++) A.state[k] = 0.0;
    if (A.maxit < 1) A.state[kIterFinished] = 1.0;
    if (A.use_graph) cudaGraphSetConditional(A.handle, A.maxit >= 1 ? 1u : 0u);
  }
}

}  // namespace

cudaError_t launch_dip_first(const IterArgs &A, cudaStream_t st) {
  k_dip_first<<<1, kFirstThreads, 0, st>>>(A);
  return cudaGetLastError();
}

cudaError_t launch_pcg_first(const IterArgs &A, cudaStream_t st) {
  k_pcg_first<<<1, kFirstThreads, 0, st>>>(A);
  return cudaGetLastError();
}

namespace {
template <int J>
void clu_config(const IterArgs &A, cudaLaunchConfig_t &cfg, cudaLaunchAttribute *at) {
  cfg.gridDim = dim3(kCluMax);
  cfg.blockDim = dim3(kCluThreads);
  cfg.dynamicSmemBytes = sizeof(double) * CluSmem(J, A.nw, A.nrow).total;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = kCluMax;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
}
template <int J>
bool clu_fits(const IterArgs &A) {
  // a block per (row tile, n tile), a warp per tile of four rows
  if (clu_sites(A.nw) > 8 * kCluTiles || (A.nrow + 7) / 8 * J > kCluMax || A.nrow > 4 * kCluWarps ||
      sizeof(double) * CluSmem(J, A.nw, A.nrow).total > kCluSmem)
    return false;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  clu_config<J>(A, cfg, at);
  int n = 0;
  const auto k = k_dip_cluster<J>;
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCluSmem) ==
          cudaSuccess &&
      cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
      cudaOccupancyMaxActiveClusters(&n, k, &cfg) == cudaSuccess && n > 0)
    return true;
  (void)cudaGetLastError();  // no such cluster on this device: the step kernels run
  return false;
}
template <int J>
cudaError_t launch_clu_t(const IterArgs &A, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  clu_config<J>(A, cfg, at);
  cfg.stream = st;
  return cudaLaunchKernelEx(&cfg, k_dip_cluster<J>, A);
}
}  // namespace

bool dip_cluster_fits(const IterArgs &A) {
  if (!A.rows || A.cu || A.nw < 1 || A.nw > 8 * kCluTiles * kCluMax) return false;
  switch (iter_row_tiles(A.nmax)) {
    case 1: return clu_fits<1>(A);
    case 2: return clu_fits<2>(A);
    case 3: return clu_fits<3>(A);
    default: return false;
  }
}

cudaError_t launch_dip_cluster(const IterArgs &A, cudaStream_t st) {
  switch (iter_row_tiles(A.nmax)) {
    case 1: return launch_clu_t<1>(A, st);
    case 2: return launch_clu_t<2>(A, st);
    case 3: return launch_clu_t<3>(A, st);
    default: return cudaErrorInvalidValue;
  }
}

namespace {
constexpr size_t kGridStay = 176 * 1024;
template <bool PCG, int J>
int grid_blocks_t(const IterArgs &A, int nsm) {
  const int nb = std::min(nsm, (A.nw + 7) / 8), ns = (A.nw + nb - 1) / nb;
  const size_t smem = sizeof(double) * GridSmem(J, A.nw, ns, A.cap * A.np, kGridStages).total;
  const auto k = k_dip_grid<PCG, J>;
  int per_sm = 0;
  if (smem > kCluSmem || A.nw > 65535 ||  // 16-bit site numbers
      cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCluSmem) !=
          cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kGridThreads, smem) != cudaSuccess ||
      per_sm < 1) {
    (void)cudaGetLastError();
    return 0;
  }
  return (A.nw + ns - 1) / ns;
}
template <bool PCG, int J>
cudaError_t launch_grid_t(const IterArgs &A, GridArgs G, int blocks, cudaStream_t st) {
  // all operands of a block's one unit stay where they fit beside the rest
  const int subs = G.chunk / (kGridRowWarps * kGridSub), ent = A.cap * A.np;
  G.stay = (A.nrow + 7) / 8 * G.nchunk <= blocks &&
           sizeof(double) * GridSmem(J, A.nw, G.ns, ent, subs).total <= kGridStay;
  G.stages = G.stay ? subs : kGridStages;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(kGridThreads);
  cfg.dynamicSmemBytes = sizeof(double) * GridSmem(J, A.nw, G.ns, ent, G.stages).total;
  cfg.stream = st;
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_dip_grid<PCG, J>, A, G);
}
}  // namespace

int dip_grid_blocks(const IterArgs &A, int nsm) {
  if (!A.rows || A.nrow < 1 || A.nw < 1) return 0;
  switch (iter_row_tiles(A.nmax)) {
    case 1: return A.cu ? grid_blocks_t<true, 1>(A, nsm) : grid_blocks_t<false, 1>(A, nsm);
    case 2: return A.cu ? grid_blocks_t<true, 2>(A, nsm) : grid_blocks_t<false, 2>(A, nsm);
    case 3: return A.cu ? grid_blocks_t<true, 3>(A, nsm) : grid_blocks_t<false, 3>(A, nsm);
    case 4: return A.cu ? grid_blocks_t<true, 4>(A, nsm) : grid_blocks_t<false, 4>(A, nsm);
    default: return 0;
  }
}

size_t dip_grid_scratch(const IterArgs &A) {  // doubles: counter, sums, combinations
  return 16 + 2 * (size_t)((A.nrow + 7) / 8 * 8) * 4 * iter_row_tiles(A.nmax) * 4;
}

cudaError_t launch_dip_grid(const IterArgs &A, int blocks, unsigned polls, double *scratch,
                            cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(scratch, 0, sizeof(double) * dip_grid_scratch(A), st);
  if (e != cudaSuccess) return e;
  GridArgs G = {};
  G.bar = reinterpret_cast<unsigned *>(scratch);
  G.polls = polls;
  G.acc = scratch + 4;
  G.ad = scratch + 16;
  G.ns = (A.nw + blocks - 1) / blocks;
  // sites per unit: the fewest steps of the busiest block, where a unit costs some six besides
  const int nt8 = (A.nrow + 7) / 8, sub = kGridRowWarps * kGridSub, most = (A.nw + sub - 1) / sub;
  long long best = -1;
  for (int n = 1; n <= most; n++) {
    const int nchunk = (most + n - 1) / n;
    const long long cost = (long long)((nt8 * nchunk + blocks - 1) / blocks) * (n * (kGridSub / 4) + 6);
    if (best < 0 || cost < best) {
      best = cost;
      G.chunk = n * sub;
      G.nchunk = nchunk;
    }
  }
  switch (iter_row_tiles(A.nmax)) {
    case 1: return A.cu ? launch_grid_t<true, 1>(A, G, blocks, st) : launch_grid_t<false, 1>(A, G, blocks, st);
    case 2: return A.cu ? launch_grid_t<true, 2>(A, G, blocks, st) : launch_grid_t<false, 2>(A, G, blocks, st);
    case 3: return A.cu ? launch_grid_t<true, 3>(A, G, blocks, st) : launch_grid_t<false, 3>(A, G, blocks, st);
    case 4: return A.cu ? launch_grid_t<true, 4>(A, G, blocks, st) : launch_grid_t<false, 4>(A, G, blocks, st);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_phase_factors(const double2 *tab, int nm, SiteSets S, int kl, int km, int kn,
                                 double2 *XY, double2 *Z, cudaStream_t st) {
  int k1 = kl > km ? kl : km;
  k1 = (k1 > kn ? k1 : kn) + 1;
  if (k1 < 2) k1 = 2;
  const size_t total = (size_t)nm * S.np * ((size_t)(kl + 1) * (2 * km + 1) + 2 * kn + 1);
  if (total == 0) return cudaSuccess;
  size_t blocks = (total + 255) / 256;
  if (blocks > 148 * 32) blocks = 148 * 32;
  k_phase_factors<<<(unsigned)blocks, 256, 0, st>>>(tab, nm, S, k1, kl, km, kn, XY, Z);
  return cudaGetLastError();
}

cudaError_t launch_tmu(const int *nbr, const int *ncnt, int cap, int nm, int np, const double4 *T4,
                       const double *TB, const double4 *S4, const double *SB, const double *mu,
                       double *eim, cudaStream_t st) {
  const int nw = nm * np;
  k_tmu<<<(nw + kWarps - 1) / kWarps, kThreads, 0, st>>>(nbr, ncnt, cap, nw, np, T4, TB, S4, SB,
                                                         mu, eim);
  return cudaGetLastError();
}

// Launches a step kernel, with programmatic stream serialization when A.pdl is set.
template <typename Kernel>
cudaError_t launch_step(Kernel kernel, int blocks, const IterArgs &A, cudaStream_t st,
                        size_t smem = 0, int threads = kThreads) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = A.pdl ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, A);
}

// n tiles of four of the row form; it runs up to kRowTilesMax of them (k_max 19)
int iter_row_tiles(int nmax) { return nmax / 4 + 1; }
bool iter_rows_fit(int nmax) { return iter_row_tiles(nmax) <= kRowTilesMax; }

// Up to this many sites per block, their Zc fit the shared memory that the warps' sums take
// at the end; longer blocks read them from memory, where they overlap with the products.
constexpr int kRowStage = 96;
// Shared memory of k_iter_a_rows with `tiles` n tiles: the dipoles, and the sums or the staged Zc.
constexpr size_t iter_rows_smem(int sites, int tiles) {
  const size_t sums = sizeof(double2) * kWarps * 4 * tiles * 32,
               zc = sites <= kRowStage ? sizeof(double) * sites * (8 * tiles + 2) : 0;
  return sizeof(double4) * sites + (sums > zc ? sums : zc);
}
constexpr size_t kRowSmemMax = 226 * 1024;  // 1 KB for the static arrays
static_assert(iter_rows_smem(kRowStage, kRowTilesMax) <= kRowSmemMax, "the smallest blocks fit");

// Sites of a structure-factor block: 96 (six steps per warp, their XY loaded ahead) while that
// makes no more than a few waves of blocks, so that the atomics stay few; 48 in small boxes,
// where blocks are too few otherwise.  Larger boxes take as many as fit in shared memory (3072
// with five n tiles) and more waves.
int iter_row_sites(int nw, int nrow, int nmax) {
  const int nt8 = (nrow + 7) / 8, tiles = iter_row_tiles(nmax);
  int cs = nw <= 512 ? 48 : 96;
  while ((long long)nt8 * ((nw + cs - 1) / cs) > 148 * 8 &&
         iter_rows_smem(2 * cs, tiles) <= kRowSmemMax)
    cs *= 2;
  return cs;
}

template <int J>
cudaError_t launch_iter_a_rows(const IterArgs &A, int nb, cudaStream_t st) {
  const bool zs = A.row_sites <= kRowStage;
  const size_t smem = iter_rows_smem(A.row_sites, J);
  const auto k = zs ? (A.cu ? k_iter_a_rows<true, J, true> : k_iter_a_rows<false, J, true>)
                    : (A.cu ? k_iter_a_rows<true, J, false> : k_iter_a_rows<false, J, false>);
  if (smem > 48 * 1024) {
    // the same value from every thread: the limit belongs to the kernel, and another context's
    // may be launched between this call and the launch
    cudaError_t e =
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRowSmemMax);
    if (e != cudaSuccess) return e;
  }
  return launch_step(k, nb, A, st, smem);
}

cudaError_t launch_iter_a(const IterArgs &A, cudaStream_t st) {
  if (A.sum_sites < 1 || A.sum_sites > kSumSitesMax) return cudaErrorInvalidValue;
  const int nsc = (A.nw + A.sum_sites - 1) / A.sum_sites;
  if (A.rows) {
    const int nb = tmu_blocks(A.nw) + (A.nrow + 7) / 8 * ((A.nw + A.row_sites - 1) / A.row_sites);
    switch (iter_row_tiles(A.nmax)) {
      case 1: return launch_iter_a_rows<1>(A, nb, st);
      case 2: return launch_iter_a_rows<2>(A, nb, st);
      case 3: return launch_iter_a_rows<3>(A, nb, st);
      case 4: return launch_iter_a_rows<4>(A, nb, st);
      case 5: return launch_iter_a_rows<5>(A, nb, st);
      default: return cudaErrorInvalidValue;
    }
  }
  const size_t smem = sizeof(double) * 3 * A.sum_sites;
  const int nkt = (A.nk + kThreads - 1) / kThreads;
  const int nb = (A.nw + kWarps - 1) / kWarps + nkt * nsc;
  if (A.PM)
    return A.cu ? launch_step(k_iter_a<true, true>, nb, A, st, smem)
                : launch_step(k_iter_a<false, true>, nb, A, st, smem);
  return A.cu ? launch_step(k_iter_a<true, false>, nb, A, st, smem)
              : launch_step(k_iter_a<false, false>, nb, A, st, smem);
}

template <int GS>
cudaError_t launch_iter_b_gs(const IterArgs &A, cudaStream_t st) {
  const int nb = (A.nw + GS - 1) / GS;
  constexpr int T = kGatherThreads;
  if (A.PM)
    return A.cu ? launch_step(k_iter_b<true, true, GS>, nb, A, st, 0, T)
                : launch_step(k_iter_b<false, true, GS>, nb, A, st, 0, T);
  return A.cu ? launch_step(k_iter_b<true, false, GS>, nb, A, st, 0, T)
              : launch_step(k_iter_b<false, false, GS>, nb, A, st, 0, T);
}

template <int J>
cudaError_t launch_iter_b_rows(const IterArgs &A, cudaStream_t st) {
  // 16 sites per block once 8 make more than three waves of blocks: an operand then serves both
  if (A.nw > 8 * 148 * 3)
    return launch_step(A.cu ? k_iter_b_rows<true, J, 2> : k_iter_b_rows<false, J, 2>,
                       (A.nw + 15) / 16, A, st, 0, kRowWarps * 32);
  return launch_step(A.cu ? k_iter_b_rows<true, J, 1> : k_iter_b_rows<false, J, 1>, (A.nw + 7) / 8,
                     A, st, 0, kRowWarps * 32);
}

cudaError_t launch_iter_b(const IterArgs &A, cudaStream_t st) {
  if (A.rows) {
    switch (iter_row_tiles(A.nmax)) {
      case 1: return launch_iter_b_rows<1>(A, st);
      case 2: return launch_iter_b_rows<2>(A, st);
      case 3: return launch_iter_b_rows<3>(A, st);
      case 4: return launch_iter_b_rows<4>(A, st);
      case 5: return launch_iter_b_rows<5>(A, st);
      default: return cudaErrorInvalidValue;
    }
  }
  switch (A.gather_sites) {
    case 2: return launch_iter_b_gs<2>(A, st);
    case 3: return launch_iter_b_gs<3>(A, st);
    case 4: return launch_iter_b_gs<4>(A, st);
    case 6: return launch_iter_b_gs<6>(A, st);
    case 8: return launch_iter_b_gs<8>(A, st);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_phase_rows(const double2 *tab, int nm, SiteSets S, int kl, int km, int kn,
                              const KRow *rows, int nrow, int zs, double2 *XYt, double *Zc,
                              cudaStream_t st) {
  int k1 = kl > km ? kl : km;
  k1 = (k1 > kn ? k1 : kn) + 1;
  if (k1 < 2) k1 = 2;
  const size_t total = (size_t)nm * S.np * ((size_t)(nrow + 7) / 8 * 8 + zs / 2);
  if (total == 0) return cudaSuccess;
  size_t blocks = (total + 255) / 256;
  if (blocks > 148 * 32) blocks = 148 * 32;
  k_phase_rows<<<(unsigned)blocks, 256, 0, st>>>(tab, nm, S, k1, km, kn, rows, nrow, zs, XYt,
                                                 reinterpret_cast<double2 *>(Zc));
  return cudaGetLastError();
}

cudaError_t launch_phase_matrix(const KGather *kg, int nk, int nw, int nlm, int nz,
                                const double2 *XY, const double2 *Z, double2 *PM,
                                cudaStream_t st) {
  if (nk <= 0 || nw <= 0) return cudaSuccess;
  const dim3 grid((nk + 127) / 128, nw < 1024 ? nw : 1024);
  k_phase_matrix<<<grid, 128, 0, st>>>(kg, nk, nw, nlm, nz, XY, Z, PM);
  return cudaGetLastError();
}
