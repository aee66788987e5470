// k_krows.cu -- the Ewald reciprocal sums by rows of the k-vector list (sm_100a, FP64 tensor
// cores).
//
// A row is one (l, m) with its run of n (KRow).  With XY = exp(i(l x + m y)) and Z(n) =
// exp(i n z) of a site the sums of k_kspace.cu regroup into small matrix products:
//   structure factors  S(k) = sum_s q XY Z(n):  Re and Im of q XY (8 rows x sites) times
//                      (cos, sin)(n z) (sites x n >= 0); +n and -n come from the same four real
//                      sums.  Dipoles: B = XY (k_l mu_x + k_m mu_y) and C = XY mu_z instead of
//                      q XY, D(k) = sum_s Z (B + k_n C);
//   gathers            E(s) = sum_r Re[XY (k_l Q, k_m Q, Q')], Q = sum_n Z(n) conj F(k), Q' =
//                      sum_n k_n Z(n) conj F(k): (cos, sin)(n z) (8 sites x n) times the
//                      combinations of F(n) and F(-n) (n x rows), for
//     the field of the charges, F = 4 a(k) (-Im S, Re S) (kspace_ewald, ewald.f90:754-1173, as
//     q E, and kspace_efield_stat, nb_induction_model.f90:597-975), and
//     the induction forces (kspace_forces, nb_induction_model.f90:4171-4839), the sum of
//     k (q Re[phase conj A] + mu.k Re[phase conj B]), A = f D, B = f (Im D - Re S, -(Im S +
//     Re D)), f = -4 a(k), which takes Q and Q' of A and of B and Q'' (k_n^2) of B.
// k_kspace.cu forms every (site, k) phase, some eight FP64 operations and two 16-byte
// shared-memory loads per pair; here a pair costs one FP64 multiply-add per real sum.  The
// evaluation's reciprocal phases at 512 / 2048 waters: Ewald sums and forces 56 / 513 us there,
// 25 / 49 here; static field and tensors 45 / 235, 40 / 117 (the field's gather also gives the
// Ewald forces); induction forces with the pair kernel 150 / 1167, 118 / 446.
#include "ccp_device.cuh"

using namespace ccpd;

namespace {

constexpr int kT = 256, kWarps = kT / 32;
constexpr int kCh = 32;        // sites of a staged chunk
constexpr int kLd = kCh + 4;   // 64 bytes of padding: neighbouring l in other banks

// D = A (8x4) B (4x8) + C in FP64: lane l holds A[l/4][l%4], B[l%4][l/4] and C, D
// [l/4][2 (l%4) + {0, 1}].
__device__ __forceinline__ void dmma(double2 &d, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(d.x), "+d"(d.y)
      : "d"(a), "d"(b));
}
__device__ __forceinline__ int warp_max(int v) { return __reduce_max_sync(0xffffffffu, v); }

// Structure factors of the charges (DIP false, into sk[k][0..1]) or of the dipoles (DIP, into
// sk[k][2..3]).  Warp w of block (x, y) takes the row tile 8 y + w over the sites of split x;
// the block stages 32 sites' tables at a time.  J tiles of four n.
template <bool DIP, int J>
__global__ void __launch_bounds__(kT)
    k_krow_sums(const KRow *__restrict__ rows, int nrow, const double2 *__restrict__ tab, int nm,
                SiteSets S, int k1, int mmax, int nmax, const double *__restrict__ rn,
                const double *__restrict__ mu, int split, double *sk) {
  extern __shared__ __align__(16) double4 smem4[];
  double4 *W = smem4;                                  // [kCh] (mu, q)
  double2 *T = reinterpret_cast<double2 *>(W + kCh);   // [3 k1][kLd]
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int per = DIP ? S.np : S.nq, N = nm * S.na;
  const int s_end = min(nm * per, ((int)blockIdx.x + 1) * split);
  const int rt = blockIdx.y * kWarps + wid;
  const bool on = rt * 8 < nrow;
  const KRow R = rows[min(rt * 8 + (lane >> 2), nrow - 1)];
  const int jt = warp_max(R.nlo + R.len - 1) / 4 + 1;
  const int M = 2 * mmax + 1, l = R.lm / M, m = R.lm - l * M - mmax;
  const double2 *Tl = T + l * kLd + (lane & 3), *Tm = T + (k1 + abs(m)) * kLd + (lane & 3);
  // column lane / 4 of the n tiles: n = 4 j + lane / 8, cos or sin
  const double *Tz = reinterpret_cast<const double *>(T + (2 * k1 + (lane >> 3)) * kLd + (lane & 3)) +
                     ((lane >> 2) & 1);
  constexpr int C = DIP ? 4 : 2;
  double2 acc[C][J];
#pragma unroll
  for (int c = 0; c < C; c++)
#pragma unroll
    for (int j = 0; j < J; j++) acc[c][j] = make_double2(0.0, 0.0);
  for (int s0 = blockIdx.x * split; s0 < s_end; s0 += kCh) {
    __syncthreads();
    {
      const int g = s0 + lane, i = g / per, r = g - i * per;
      const bool in = g < s_end;
      const int a = in ? (DIP ? S.a_of_p[r] : S.a_of_q[r]) : 0;
      // tables of every n tile's last n may lie above n_max: their products are not used, but
      // must be finite
      for (int u = wid; u < 2 * k1 + 4 * J; u += kWarps)
        T[u * kLd + lane] = in && (u < 2 * k1 || u - 2 * k1 <= nmax)
                                ? tab[(size_t)u * N + (size_t)i * S.na + a]
                                : make_double2(0.0, 0.0);
      if (wid == 0) {
        double4 w = make_double4(0.0, 0.0, 0.0, 0.0);
        if (in) {
          if (DIP) {
            const size_t o = (size_t)g * 3;
            w = make_double4(mu[o], mu[o + 1], mu[o + 2], 0.0);
          } else {
            w.w = S.q[a];
          }
        }
        W[lane] = w;
      }
    }
    __syncthreads();
    if (!on) continue;
#pragma unroll 2
    for (int t = 0; t < kCh / 4; t++) {
      double2 el = Tl[4 * t], em = Tm[4 * t];
      if (m < 0) em.y = -em.y;
      const double2 xy = make_double2(el.x * em.x - el.y * em.y, el.y * em.x + em.y * el.x);
      const double4 w = W[4 * t + (lane & 3)];
      double a[C];
      if constexpr (DIP) {
        const double d = R.rl * w.x + R.rm * w.y;
        a[0] = xy.x * d;
        a[1] = xy.y * d;
        a[2] = xy.x * w.z;
        a[3] = xy.y * w.z;
      } else {
        a[0] = xy.x * w.w;
        a[1] = xy.y * w.w;
      }
#pragma unroll
      for (int j = 0; j < J; j++)
        if (j < jt) {
          const double z = Tz[2 * (4 * j * kLd + 4 * t)];
#pragma unroll
          for (int c = 0; c < C; c++) dmma(acc[c][j], a[c], z);
        }
    }
  }
  // the lane's row and n = 4 j + lane % 4: (cos, sin) sums of each part
  if (!on || rt * 8 + (lane >> 2) >= nrow) return;
#pragma unroll
  for (int j = 0; j < J; j++) {
    const int n = 4 * j + (lane & 3);
    if (n > nmax) continue;
    double pr = acc[0][j].x - acc[1][j].y, pi = acc[0][j].y + acc[1][j].x;
    double mr = acc[0][j].x + acc[1][j].y, mi = acc[1][j].x - acc[0][j].y;
    if constexpr (DIP) {
      const double kn = rn[n + nmax];
      pr += kn * (acc[2][j].x - acc[3][j].y);
      pi += kn * (acc[2][j].y + acc[3][j].x);
      mr -= kn * (acc[2][j].x + acc[3][j].y);
      mi -= kn * (acc[3][j].x - acc[2][j].y);
    }
    const int kp = n - R.nlo, km = -n - R.nlo;
    double *o = sk + (DIP ? 2 : 0);
    if (kp >= 0 && kp < R.len) {
      atomicAdd(o + (size_t)(R.kbeg + kp) * 4, pr);
      atomicAdd(o + (size_t)(R.kbeg + kp) * 4 + 1, pi);
    }
    if (n > 0 && km >= 0 && km < R.len) {
      atomicAdd(o + (size_t)(R.kbeg + km) * 4, mr);
      atomicAdd(o + (size_t)(R.kbeg + km) * 4 + 1, mi);
    }
  }
}

// The gathers' weights as the combinations F(n) + F(-n), F(n) - F(-n) that their products take,
// w[row][n][(re), (im)] = (sum, difference) for n = 0 .. nn - 1 (IND: of A, then of B), zero
// where the list has no such k; and, with `energy`, the energy and virial of the sums per k
// (ewald.f90:1043-1045; nb_induction_model.f90:4579-4581).
template <bool IND>
__global__ void k_krow_weights(const KVec *__restrict__ kv, const KRow *__restrict__ rows, int nrow,
                               int nn, const double *__restrict__ sk, double alpha, int energy,
                               double2 *w, double *scal) {
  double e = 0.0, vir = 0.0;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < nrow * nn; t += gridDim.x * blockDim.x) {
    const int r = t / nn, n = t - r * nn;
    const KRow R = rows[r];
    double F[2][4] = {{0.0, 0.0, 0.0, 0.0}, {0.0, 0.0, 0.0, 0.0}};  // of n and of -n
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int u = (h ? -n : n) - R.nlo;
      if ((h && n == 0) || u < 0 || u >= R.len) continue;
      const KVec K = kv[R.kbeg + u];
      const double4 s = *reinterpret_cast<const double4 *>(sk + (size_t)(R.kbeg + u) * 4);
      const double f = (IND ? -4.0 : 4.0) * K.ak;
      if (IND) {
        F[h][0] = f * s.z;
        F[h][1] = f * s.w;
        F[h][2] = f * (s.w - s.x);
        F[h][3] = -f * (s.y + s.z);
      } else {
        F[h][0] = -f * s.y;
        F[h][1] = f * s.x;
      }
      if (energy) {
        const double rksq = K.rl * K.rl + K.rm * K.rm + K.rn * K.rn;
        const double fac = 1.0 - 0.5 * rksq / (alpha * alpha);
        if (IND) {
          const double x1 = s.z * s.y - s.w * s.x, x2 = s.z * s.z + s.w * s.w;
          vir -= 2.0 * K.ak * (x1 + x2 + 0.5 * (2.0 * x1 + x2) * fac);
        } else {
          const double s2 = s.x * s.x + s.y * s.y;
          e += K.ak * s2;
          vir -= fac * K.ak * s2;
        }
      }
    }
#pragma unroll
    for (int c = 0; c < (IND ? 4 : 2); c++)
      w[(size_t)t * (IND ? 4 : 2) + c] = make_double2(F[0][c] + F[1][c], F[0][c] - F[1][c]);
  }
  if (!energy) return;
  e = warp_sum(e);
  vir = warp_sum(vir);
  if ((threadIdx.x & 31) == 0) {
    if (IND) {
      atomicAdd(&scal[S_IND_VIR_K], vir);
    } else {
      atomicAdd(&scal[S_KC_E], e);
      atomicAdd(&scal[S_KC_VIR], vir);
    }
  }
}

// Gathers: a block takes MT tiles of 8 sites, its warps the tiles of four rows in turn.  Lane l
// ends up with the row sums of site l / 4 and row l % 4 and contracts them with XY.  Field form
// (IND false): E into e0k of the polarisable sites (if set) and q E into the forces of the
// charged ones (if F.x is set); sites: all active ones, or the polarisable ones only (pol).  With
// F.e the field form also writes the Ewald energy (kcal/mol) and adds the virial, from the sums
// that k_krow_weights left in scal, with the reference's prefactors (ewald.f90:1151-1160).
template <bool IND, int J, int MT>
__global__ void __launch_bounds__(kT)
    k_krow_gather(const KRow *__restrict__ rows, int nrow, const double2 *__restrict__ wt,
                  const double2 *__restrict__ tab, int nm, SiteSets S, int pol, int k1, int mmax,
                  int nmax, const double *__restrict__ rn, const double *__restrict__ mu,
                  double *e0k, KRowForces F) {
  constexpr int KS = 2 * J, kZs = 8 * J + 2, NS = 8 * MT, G = IND ? 4 : 2;
  extern __shared__ __align__(16) double4 smem4[];
  double2 *T = reinterpret_cast<double2 *>(smem4);        // [2 k1][NS]
  double *Zs = reinterpret_cast<double *>(T + 2 * k1 * NS);  // [NS][kZs]
  __shared__ double part[kWarps][3][NS];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int per = pol ? S.np : S.na, N = nm * S.na, total = nm * per, g0 = blockIdx.x * NS;
  auto slot = [&](int g) {  // active site of target g
    const int i = g / per, r = g - i * per;
    return i * S.na + (pol ? S.a_of_p[r] : r);
  };
  {
    const int s = threadIdx.x % NS, st = slot(min(g0 + s, total - 1));
    for (int u = threadIdx.x / NS; u < 2 * k1; u += kT / NS) T[u * NS + s] = tab[(size_t)u * N + st];
    for (int n = threadIdx.x / NS; n < 4 * J; n += kT / NS)
      *reinterpret_cast<double2 *>(Zs + s * kZs + 2 * n) =
          n <= nmax ? tab[(size_t)(2 * k1 + n) * N + st] : make_double2(0.0, 0.0);
  }
  double q[MT], mx[MT], my[MT], mz[MT];
#pragma unroll
  for (int m = 0; m < MT; m++) {
    q[m] = mx[m] = my[m] = mz[m] = 0.0;
    if (IND) {
      const int st = slot(min(g0 + 8 * m + (lane >> 2), total - 1)), i = st / S.na, a = st - i * S.na;
      q[m] = S.q[a];
      const int p = S.p_of_a[a];
      if (p >= 0) {
        const size_t o = ((size_t)i * S.np + p) * 3;
        mx[m] = mu[o];
        my[m] = mu[o + 1];
        mz[m] = mu[o + 2];
      }
    }
  }
  __syncthreads();
  const int M = 2 * mmax + 1, nt4 = (nrow + 3) / 4;
  // operand element: row lane / 8 of the tile, column part ri (Re, Im), factor part cs (cos, sin)
  const int ri = (lane >> 2) & 1, cs = lane & 1, n0 = (lane >> 1) & 1, x = ri ^ cs;
  const double sg = cs == 0 && ri == 1 ? -1.0 : 1.0;
  double kn[KS];
#pragma unroll
  for (int k = 0; k < KS; k++) kn[k] = rn[min(2 * k + n0, nmax) + nmax];
  double ex[MT], ey[MT], ez[MT];
#pragma unroll
  for (int m = 0; m < MT; m++) ex[m] = ey[m] = ez[m] = 0.0;
  for (int t = wid; t < nt4; t += kWarps) {
    const int rb = min(4 * t + (lane >> 3), nrow - 1), ra = min(4 * t + (lane & 3), nrow - 1);
    const KRow Rb = rows[rb], R = rows[ra];
    const int ks = warp_max(Rb.nlo + Rb.len - 1) / 2 + 1;
    const double2 *w = wt + ((size_t)rb * (4 * J) + n0) * G + x;
    double2 Q[MT], Q1[MT], P[MT], P1[MT], P2[MT];
#pragma unroll
    for (int m = 0; m < MT; m++) Q[m] = Q1[m] = P[m] = P1[m] = P2[m] = make_double2(0.0, 0.0);
#pragma unroll
    for (int k = 0; k < KS; k++)
      if (k < ks) {
        const double2 A = w[2 * k * G];
        const double b0 = sg * (cs == 0 ? A.x : A.y), b1 = kn[k] * (sg * (cs == 0 ? A.y : A.x));
        double c0 = 0.0, c1 = 0.0, c2 = 0.0;
        if constexpr (IND) {
          const double2 B = w[2 * k * G + 2];
          c0 = sg * (cs == 0 ? B.x : B.y);
          c1 = kn[k] * (sg * (cs == 0 ? B.y : B.x));
          c2 = kn[k] * (kn[k] * c0);
        }
#pragma unroll
        for (int m = 0; m < MT; m++) {
          const double z = Zs[(8 * m + (lane >> 2)) * kZs + 4 * k + (lane & 3)];
          dmma(Q[m], z, b0);
          dmma(Q1[m], z, b1);
          if constexpr (IND) {
            dmma(P[m], z, c0);
            dmma(P1[m], z, c1);
            dmma(P2[m], z, c2);
          }
        }
      }
    const int l = R.lm / M, mm = R.lm - l * M - mmax;
#pragma unroll
    for (int m = 0; m < MT; m++) {
      const double2 el = T[l * NS + 8 * m + (lane >> 2)];
      double2 em = T[(k1 + abs(mm)) * NS + 8 * m + (lane >> 2)];
      if (mm < 0) em.y = -em.y;
      const double2 xy = make_double2(el.x * em.x - el.y * em.y, el.y * em.x + em.y * el.x);
      double a = xy.x * Q[m].x - xy.y * Q[m].y, az = xy.x * Q1[m].x - xy.y * Q1[m].y;
      if constexpr (IND) {
        const double d = R.rl * mx[m] + R.rm * my[m];
        const double p0 = xy.x * P[m].x - xy.y * P[m].y, p1 = xy.x * P1[m].x - xy.y * P1[m].y,
                     p2 = xy.x * P2[m].x - xy.y * P2[m].y;
        a = q[m] * a + (d * p0 + mz[m] * p1);
        az = q[m] * az + (d * p1 + mz[m] * p2);
      }
      if (4 * t + (lane & 3) < nrow) {  // not a row past the last
        ex[m] += R.rl * a;
        ey[m] += R.rm * a;
        ez[m] += az;
      }
    }
  }
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
  if (threadIdx.x < 3 * NS) {
    const int c = threadIdx.x / NS, s = threadIdx.x - c * NS, g = g0 + s;
    if (g < total) {
      double v = 0.0;
#pragma unroll
      for (int u = 0; u < kWarps; u++) v += part[u][c][s];
      const int st = slot(g), i = st / S.na, a = st - i * S.na;
      double *f = c == 0 ? F.x : (c == 1 ? F.y : F.z);
      const size_t o = (size_t)i * F.ld + S.asite[a];
      if (IND) {
        atomicAdd(&f[o], kR4pie0 * v);
      } else {
        if (f && S.q[a] != 0.0) atomicAdd(&f[o], kR4pie0 * S.q[a] * v);
        if (e0k && S.p_of_a[a] >= 0) e0k[((size_t)i * S.np + S.p_of_a[a]) * 3 + c] = v;
      }
    }
  }
  if (!IND && F.e && blockIdx.x == 0 && threadIdx.x == 0) {
    *F.e = 2.0 * kR4pie0 * F.scal[S_KC_E] / 418.4;
    *F.vir += 2.0 * kR4pie0 * F.scal[S_KC_VIR];
  }
}

inline int k1_of(int kl, int km, int kn) {
  int k1 = kl > km ? kl : km;
  k1 = (k1 > kn ? k1 : kn) + 1;
  return k1 < 2 ? 2 : k1;
}

// Lets the kernel take `smem` bytes.  The same value from every thread, since the limit belongs to
// the kernel: what the gather's static arrays (3 KB) leave, enough for k_max 190 in l and m.
template <typename F>
cudaError_t set_smem(F kern, size_t smem) {
  constexpr size_t kMax = 224 * 1024;
  if (smem > kMax) return cudaErrorInvalidValue;
  if (smem > 48 * 1024)
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMax);
  return cudaSuccess;
}

template <bool DIP, int J>
cudaError_t sums_t(const KRowArgs &A, const double *mu, cudaStream_t st) {
  const int k1 = k1_of(A.kl, A.km, A.kn), total = A.nm * (DIP ? A.S.np : A.S.nq);
  if (total <= 0) return cudaErrorInvalidConfiguration;  // no such site: a grid of no blocks
  const int ny = ((A.nrow + 7) / 8 + kWarps - 1) / kWarps, chunks = (total + kCh - 1) / kCh;
  // blocks for two per SM; each keeps its row tiles' sums over all chunks of its split
  int nx = (148 * 2 + ny - 1) / ny;
  if (nx > chunks) nx = chunks;
  const int split = (chunks + nx - 1) / nx * kCh;
  const size_t smem = sizeof(double4) * kCh + sizeof(double2) * (2 * k1 + 4 * J) * kLd;
  cudaError_t e = set_smem(k_krow_sums<DIP, J>, smem);
  if (e != cudaSuccess) return e;
  k_krow_sums<DIP, J><<<dim3((total + split - 1) / split, ny), kT, smem, st>>>(
      A.rows, A.nrow, A.tab, A.nm, A.S, k1, A.km, A.kn, A.rn, mu, split, A.sk);
  return cudaGetLastError();
}

template <bool IND, int J, int MT>
cudaError_t gather_mt(const KRowArgs &A, int pol, const double *mu, double *e0k, const KRowForces &F,
                      cudaStream_t st) {
  const int k1 = k1_of(A.kl, A.km, A.kn), total = A.nm * (pol ? A.S.np : A.S.na), NS = 8 * MT;
  const size_t smem = sizeof(double2) * 2 * k1 * NS + sizeof(double) * NS * (8 * J + 2);
  cudaError_t e = set_smem(k_krow_gather<IND, J, MT>, smem);
  if (e != cudaSuccess) return e;
  k_krow_gather<IND, J, MT><<<(total + NS - 1) / NS, kT, smem, st>>>(
      A.rows, A.nrow, A.w, A.tab, A.nm, A.S, pol, k1, A.km, A.kn, A.rn, mu, e0k, F);
  return cudaGetLastError();
}
template <bool IND, int J>
cudaError_t gather_t(const KRowArgs &A, int pol, const double *mu, double *e0k, const KRowForces &F,
                     cudaStream_t st) {
  // 16 sites per block once 8 make more than three waves: an operand then serves both tiles
  const int total = A.nm * (pol ? A.S.np : A.S.na);
  return total > 8 * 148 * 6 ? gather_mt<IND, J, 2>(A, pol, mu, e0k, F, st)
                             : gather_mt<IND, J, 1>(A, pol, mu, e0k, F, st);
}

}  // namespace

size_t krow_weight_len(int nrow, int kn) { return (size_t)nrow * 4 * iter_row_tiles(kn) * 4; }

cudaError_t launch_krow_sums(bool dip, const KRowArgs &A, const double *mu, cudaStream_t st) {
  if (A.nrow <= 0) return cudaSuccess;
  switch (iter_row_tiles(A.kn)) {
    case 1: return dip ? sums_t<true, 1>(A, mu, st) : sums_t<false, 1>(A, mu, st);
    case 2: return dip ? sums_t<true, 2>(A, mu, st) : sums_t<false, 2>(A, mu, st);
    case 3: return dip ? sums_t<true, 3>(A, mu, st) : sums_t<false, 3>(A, mu, st);
    case 4: return dip ? sums_t<true, 4>(A, mu, st) : sums_t<false, 4>(A, mu, st);
    case 5: return dip ? sums_t<true, 5>(A, mu, st) : sums_t<false, 5>(A, mu, st);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_krow_weights(bool ind, const KRowArgs &A, double alpha, int energy, double *scal,
                                cudaStream_t st) {
  if (A.nrow <= 0) return cudaSuccess;
  const int nn = 4 * iter_row_tiles(A.kn), blocks = (A.nrow * nn + 127) / 128;
  const int nb = blocks < 148 * 4 ? blocks : 148 * 4;
  if (ind)
    k_krow_weights<true><<<nb, 128, 0, st>>>(A.kv, A.rows, A.nrow, nn, A.sk, alpha, energy, A.w, scal);
  else
    k_krow_weights<false><<<nb, 128, 0, st>>>(A.kv, A.rows, A.nrow, nn, A.sk, alpha, energy, A.w, scal);
  return cudaGetLastError();
}

cudaError_t launch_krow_gather(bool ind, const KRowArgs &A, int pol, const double *mu, double *e0k,
                               const KRowForces &F, cudaStream_t st) {
  if (A.nrow <= 0) return cudaSuccess;
  switch (iter_row_tiles(A.kn)) {
    case 1: return ind ? gather_t<true, 1>(A, pol, mu, e0k, F, st) : gather_t<false, 1>(A, pol, mu, e0k, F, st);
    case 2: return ind ? gather_t<true, 2>(A, pol, mu, e0k, F, st) : gather_t<false, 2>(A, pol, mu, e0k, F, st);
    case 3: return ind ? gather_t<true, 3>(A, pol, mu, e0k, F, st) : gather_t<false, 3>(A, pol, mu, e0k, F, st);
    case 4: return ind ? gather_t<true, 4>(A, pol, mu, e0k, F, st) : gather_t<false, 4>(A, pol, mu, e0k, F, st);
    case 5: return ind ? gather_t<true, 5>(A, pol, mu, e0k, F, st) : gather_t<false, 5>(A, pol, mu, e0k, F, st);
    default: return cudaErrorInvalidValue;
  }
}
