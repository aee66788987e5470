// k_vdw.cu -- the ccpol23plus 2-body term (vdw_ccpol23plus.f90:174-477) on sm_100a, FP64.
//
// For every molecule pair with COM distance below rcut (the reference's exact minimum-image
// test, from the neighbour list) and every pair of sites whose names have a parameter row:
//   u = e^{-beta r} (c0 + c1 r + c2 r^2 + c3 r^3) / (1 + e^{-gamma (r - r0)})
//     + r4pie0 (f1(d1 r) - 1) q_a q_b / r
//     - f6(d6 r) c6 / r^6 - f8(d8 r) c8 / r^8 - f10(d10 r) c10 / r^10,
// f_n the Tang-Toennies damping, gamma = 20/bohr2a, r0 = 1.4 bohr2a.  Molecule i handles half
// of its neighbour pairs: the pair (i, j) goes to i when i < j and i + j is odd or i > j and
// i + j is even, so that every molecule has about half its neighbours (with j > i alone the
// low-numbered molecules carried twice the average and the launch ran in two waves); kSplit
// blocks share a molecule's pairs.  A pair is cut into items that the warps take in turn:
//   - kJs sites js of j, lane = site is of i, the exponential term: i's site forces accumulate
//     in registers, and the 3 kJs force components of the js are summed over the lanes together
//     (16 exchanges for 15 sums instead of 75);
//   - the site pairs with a charge product or dispersion (25 of 625, listed by the host), one per
//     lane: in the first kind's warps, most lanes would idle through those series.
// Each exponential is evaluated once and serves the damping and its derivative; that of the
// short-range damping, which has no effect in double precision from 1.2 A past r0 on, only where
// a lane is nearer.  512 waters: 260 us (402 with one site of j per warp and step).
#include "ccp_device.cuh"

using namespace ccpd;

namespace {

constexpr int kThreads = 128;
// blocks per molecule: each takes every kSplit-th pair of the molecule's share, so that more
// warps are in flight (a molecule's pairs are independent; its site forces are added
// atomically)
#ifndef CCP_VDW_SPLIT
#define CCP_VDW_SPLIT 4
#endif
constexpr int kSplit = CCP_VDW_SPLIT;
constexpr int kWarps = kThreads / 32;

// Tang-Toennies f_N(delta r) and its derivative (utility.f90:89-125) from one exponential.
// The series' divisions by i are products with the reciprocals 1/i (compile-time constants):
// FP64 divisions would dominate the kernel.
template <int N>
__device__ __forceinline__ void tt_both(double delta, double r, double &f, double &df) {
  const double dr = delta * r, ex = exp(-dr);
  double term = 1.0, sum = 1.0;
#pragma unroll
  for (int i = 1; i <= N; i++) {
    term = term * dr * (1.0 / (double)i);
    sum += term;
  }
  f = 1.0 - ex * sum;
  df = delta * ex * term;  // term = (delta r)^N / N!
}

constexpr int kJs = 5;  // sites of j per item

// Sum over the warp of 16 values per lane: lane l returns that of value l / 2.
__device__ __forceinline__ double warp_sum16(double (&g)[16], int lane) {
#pragma unroll
  for (int o = 16, n = 8; o > 1; o >>= 1, n >>= 1)
#pragma unroll
    for (int u = 0; u < n; u++) {
      const bool up = lane & o;
      const double keep = up ? g[u + n] : g[u], give = up ? g[u] : g[u + n];
      g[u] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  return g[0] + __shfl_xor_sync(0xffffffffu, g[0], 1);
}

__global__ void __launch_bounds__(kThreads)
    k_vdw(const double *__restrict__ xs, const double *__restrict__ ys,
          const double *__restrict__ zs, int ld, const int *__restrict__ nbr,
          const double4 *__restrict__ nbrv, const int *__restrict__ ncnt, int cap, int ns,
          double rcutsd, const int *__restrict__ row, const double *__restrict__ qq,
          const double *__restrict__ par, int nrows, const int *__restrict__ vsite, int nv,
          const int2 *__restrict__ spec, int nspec, double *f, double *scal, int nm) {
  __shared__ double P[kVdwPar][kVdwMaxRows];
  __shared__ signed char krow[32][32];  // [js][is], as indices of vsite
  __shared__ double fi[kWarps][32][3];
  __shared__ double red[2][kWarps];
  __shared__ int n_pair;
  extern __shared__ int pairs[];  // places in i's neighbour list
  const int i = blockIdx.x / kSplit, part = blockIdx.x % kSplit;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (threadIdx.x == 0) n_pair = 0;
  for (int u = threadIdx.x; u < nrows * kVdwPar; u += kThreads) P[u % kVdwPar][u / kVdwPar] = par[u];
  for (int u = threadIdx.x; u < nv * 32; u += kThreads)
    krow[u >> 5][u & 31] = (u & 31) < nv ? (signed char)row[vsite[u & 31] * ns + vsite[u >> 5]] : -1;
  __syncthreads();
  const int cnt = min(ncnt[i], cap);
  for (int n = part + kSplit * threadIdx.x; n < cnt; n += kSplit * kThreads) {
    const int j = nbr[(size_t)i * cap + n];
    if (j == i || (j > i) != (((i + j) & 1) != 0)) continue;  // the pair is j's
    if (nbrv[(size_t)i * cap + n].w < rcutsd) pairs[atomicAdd(&n_pair, 1)] = n;
  }
  __syncthreads();
  const double gamma = 20.0 / kBohr2a, sqr0 = 1.4 * kBohr2a;
  const bool lact = lane < nv;
  const int is = lact ? vsite[lane] : 0;
  const size_t oi = (size_t)i * ld + is;
  const double sxi = lact ? xs[oi] : 0.0, syi = lact ? ys[oi] : 0.0, szi = lact ? zs[oi] : 0.0;
  double fx = 0.0, fy = 0.0, fz = 0.0, e = 0.0, v = 0.0;
  // the listed site pairs' force on i, of list chunk `cur`
  double lx = 0.0, ly = 0.0, lz = 0.0;
  int cur = -1;
  const size_t nfs = (size_t)nm * ns;
  auto flush = [&]() {
    if (cur >= 0 && 32 * cur + lane < nspec) {
      const size_t o = (size_t)i * ns + spec[32 * cur + lane].x;
      atomicAdd(&f[o], lx);
      atomicAdd(&f[nfs + o], ly);
      atomicAdd(&f[2 * nfs + o], lz);
    }
    lx = ly = lz = 0.0;
  };
  const int nj = (nv + kJs - 1) / kJs, per = nj + (nspec + 31) / 32, total = n_pair * per;
  for (int t = wid; t < total; t += kWarps) {
    const int pi = t / per, part_t = t - pi * per, n = pairs[pi];
    const int j = nbr[(size_t)i * cap + n];
    const double4 c = nbrv[(size_t)i * cap + n];
    if (part_t < nj) {
      double g[16];
      g[15] = 0.0;
#pragma unroll
      for (int q = 0; q < kJs; q++) {
        const int jv = part_t * kJs + q;
        double gx = 0.0, gy = 0.0, gz = 0.0;
        if (jv < nv) {
          const size_t oj = (size_t)j * ld + vsite[jv];
          const int k = krow[jv][lane];
          const double rsx = c.x + sxi - xs[oj], rsy = c.y + syi - ys[oj], rsz = c.z + szi - zs[oj];
          const double sqr = sqrt(rsx * rsx + rsy * rsy + rsz * rsz);
          // exchange-repulsion with the short-range damping
          const double x0 = gamma * (sqr - sqr0);
          double eg = 0.0, fdamp = 1.0;
          if (__any_sync(0xffffffffu, k >= 0 && x0 < 45.0)) {
            eg = exp(-x0);
            fdamp = 1.0 / (1.0 + eg);
          }
          if (k >= 0) {
            const double beta = P[0][k], c1 = P[2][k], c2 = P[3][k], c3 = P[4][k];
            const double eks = exp(-beta * sqr);
            const double poly = P[1][k] + sqr * (c1 + sqr * (c2 + sqr * c3));
            const double u = eks * poly * fdamp;
            const double du = -beta * u * fdamp + eks * fdamp * (c1 + sqr * (2.0 * c2 + 3.0 * c3 * sqr)) +
                              gamma * eg * fdamp * fdamp * u;
            e += u;
            const double vf = -du / sqr;
            gx = rsx * vf;
            gy = rsy * vf;
            gz = rsz * vf;
            v -= rsx * gx + rsy * gy + rsz * gz;
          }
        }
        fx += gx;
        fy += gy;
        fz += gz;
        g[3 * q] = gx;
        g[3 * q + 1] = gy;
        g[3 * q + 2] = gz;
      }
      const double s = warp_sum16(g, lane);
      const int w = lane >> 1, jv = part_t * kJs + w / 3;
      if (!(lane & 1) && w < 3 * kJs && jv < nv)
        atomicAdd(&f[(w % 3) * nfs + (size_t)j * ns + vsite[jv]], -s);
    } else {
      if (part_t - nj != cur) {
        flush();
        cur = part_t - nj;
      }
      const int u0 = 32 * cur + lane;
      if (u0 < nspec) {
        const int2 ab = spec[u0];
        const size_t oa = (size_t)i * ld + ab.x, ob = (size_t)j * ld + ab.y;
        const int k = row[ab.x * ns + ab.y];
        const double c6 = P[5][k], c8 = P[6][k], c10 = P[7][k];
        const double rsx = c.x + xs[oa] - xs[ob], rsy = c.y + ys[oa] - ys[ob],
                     rsz = c.z + zs[oa] - zs[ob];
        const double sqr = sqrt(rsx * rsx + rsy * rsy + rsz * rsz);
        const double ir = 1.0 / sqr, ir2 = ir * ir;  // one division serves every 1/r^n
        double u = 0.0, du = 0.0;
        // short-range Coulomb correction; q_a q_b of the site pair
        const double qab = qq[ab.x * ns + ab.y];
        if (qab != 0.0) {
          double f1, df1;
          tt_both<1>(P[8][k], sqr, f1, df1);
          u += kR4pie0 * (f1 - 1.0) * qab * ir;
          du += -kR4pie0 * qab * ((f1 - 1.0) * ir2 - df1 * ir);
        }
        const double ir6 = ir2 * ir2 * ir2, ir8 = ir2 * ir6, ir10 = ir2 * ir8;
        if (c6 != 0.0) {
          double f6, df6;
          tt_both<6>(P[9][k], sqr, f6, df6);
          u += -f6 * c6 * ir6;
          du += -df6 * c6 * ir6 + 6.0 * f6 * c6 * ir6 * ir;
        }
        if (c8 != 0.0) {
          double f8, df8;
          tt_both<8>(P[10][k], sqr, f8, df8);
          u += -f8 * c8 * ir8;
          du += -df8 * c8 * ir8 + 8.0 * f8 * c8 * ir8 * ir;
        }
        if (c10 != 0.0) {
          double f10, df10;
          tt_both<10>(P[11][k], sqr, f10, df10);
          u += -f10 * c10 * ir10;
          du += -df10 * c10 * ir10 + 10.0 * f10 * c10 * ir10 * ir;
        }
        e += u;
        const double vf = -du * ir, gx = rsx * vf, gy = rsy * vf, gz = rsz * vf;
        lx += gx;
        ly += gy;
        lz += gz;
        v -= rsx * gx + rsy * gy + rsz * gz;
        const size_t o = (size_t)j * ns + ab.y;
        atomicAdd(&f[o], -gx);
        atomicAdd(&f[nfs + o], -gy);
        atomicAdd(&f[2 * nfs + o], -gz);
      }
    }
  }
  flush();
  fi[wid][lane][0] = fx;
  fi[wid][lane][1] = fy;
  fi[wid][lane][2] = fz;
  e = warp_sum(e);
  v = warp_sum(v);
  if (lane == 0) {
    red[0][wid] = e;
    red[1][wid] = v;
  }
  __syncthreads();
  if (threadIdx.x < 32 && lact) {
    double sx = 0.0, sy = 0.0, sz = 0.0;
    for (int w = 0; w < kWarps; w++) {
      sx += fi[w][lane][0];
      sy += fi[w][lane][1];
      sz += fi[w][lane][2];
    }
    const size_t o = (size_t)i * ns + is;
    atomicAdd(&f[o], sx);
    atomicAdd(&f[nfs + o], sy);
    atomicAdd(&f[2 * nfs + o], sz);
  }
  if (threadIdx.x == 0) {
    double se = 0.0, sv = 0.0;
    for (int w = 0; w < kWarps; w++) {
      se += red[0][w];
      sv += red[1][w];
    }
    atomicAdd(&scal[S_VDW_E], se);
    atomicAdd(&scal[S_VDW_VIR], sv);
  }
}

}  // namespace

cudaError_t launch_vdw(const double *xs, const double *ys, const double *zs, int ld,
                       const int *nbr, const double4 *nbrv, const int *ncnt, int cap, int nm,
                       int ns, double rcutsd, const int *row, const double *qq,
                       const double *par, int nrows, const int *vsite, int nv, const int2 *spec,
                       int nspec, double *f, double *scal, cudaStream_t st) {
  if (nv < 1 || nv > 32 || nrows < 1 || nrows > kVdwMaxRows) return cudaErrorInvalidValue;
  const size_t smem = sizeof(int) * ((cap + kSplit - 1) / kSplit);
  k_vdw<<<nm * kSplit, kThreads, smem, st>>>(xs, ys, zs, ld, nbr, nbrv, ncnt, cap, ns, rcutsd, row,
                                             qq, par, nrows, vsite, nv, spec, nspec, f, scal, nm);
  return cudaGetLastError();
}
