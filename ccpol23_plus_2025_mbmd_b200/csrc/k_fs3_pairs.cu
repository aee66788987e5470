// k_fs3_pairs.cu -- FS3 by molecule pairs on the FP64 tensor-core path (sm_100a).
//
// The FS3 sum of a molecular triple (threebody_potential.f90:676-2062; see k_fs3.cu for the
// sum itself) is trilinear in the tables (e, e d) of its three molecule pairs,
//     S = sum_{abc} sum_{pqr} c(ta, tb, tc; r, q, p) U_p(a, b) V_q(a, c) W_r(b, c),
// U, V, W the tables of the pairs (A, B), (A, C), (B, C), and its coefficients are symmetric
// under a common permutation of the molecules (fill, threebody_potential.f90:2064-2131).  The
// weight of a site pair (a, b) of molecules A, B in the forces is the derivative of the sum
// over ALL third molecules C by U(a, b),
//     q_p(a, b) = sum_{C, c, q, r} c w_C V_q(a, c) W_r(b, c),    w_C the triple's weight,
// so one block takes one molecule pair and runs over its third molecules ("visits"):
//   - the tables are made once per molecule pair (fs3_tables), not once per triple and pair;
//   - the products of a visit are small matrix products over the sites c of one type, and
//     they accumulate over the visits in registers as sum_C w_C V_q W_r per type of c: the
//     contraction with the coefficients is done once per pair, not once per triple;
//   - forces and the virial are formed once per pair.
// The triples' energy sums S, which the damping and switch forces need one by one, come from a
// second kernel, one warp per triple (k_fs3_energy).
//
// Work of a visit (sites 1..16 of a molecule are numbered 0..15 in the code, in the types
// [0,1] [2,3] [4..7] [8..11] [12..15]; site 0 is a type of its own): a block's four warps take
// an 8 x 8 tile of the 16 x 16 site pairs each, as mma.m8n8k4 per type of c and power pair.
// The types of four sites fill the instruction's K; the two of two sites share a fragment and
// are padded with zeros (20 instructions per tile where 16 would do, without a branch); the one
// site of type 0 is multiplied out.  The 33 pairs with a site 0 come from the operand fragments that the warps
// hold anyway, as products with the other molecule's row of site 0 (one of the four 8-site
// edges per warp).  No warp waits for another: each adds its own tile's forces.
// DFMA and DMMA share one pipe on this part (36.8 TFLOP/s DMMA, 34 DFMA); DMMA is taken for
// its operand reuse: two 16-byte loads per lane feed 32 DFMA's worth.
//
// FS3 with its lists at 512 / 2048 waters: 1220 / 6928 us by triples, 750 / 4190 here (at 512:
// lists and tables 67, pair kernel 483, energies 204; four blocks of four warps per SM, 128
// registers a thread).  The pair kernel keeps the FP64 pipe 42 % busy: it waits for its
// own short dependent chains and loads that hit L1 (half of its sectors; the other warps'
// prefetch brings them).  Measured and worse: table stages by TMA or by the block with barriers
// (0.54 to 1.7 ms), 3 or 5 blocks per SM, prefetching two visits ahead (547) or the next pass's
// first visit (494).  The energy kernel keeps it 55 % busy; runs of triples per block, for their
// shared tables' sake, took 218.
#include "ccp_device.cuh"

// Pair blocks per SM that the register allocation targets.
#ifndef CCP_FS3_PAIR_BLOCKS
#define CCP_FS3_PAIR_BLOCKS 4
#endif
#ifndef CCP_FS3_ENERGY_BLOCKS
#define CCP_FS3_ENERGY_BLOCKS 4
#endif

using namespace ccpd;

namespace {

constexpr int kTab = 289;              // site pairs of two molecules
constexpr int kNt = 6;
constexpr int kCoef = kNt * kNt * kNt * 8;
constexpr int kPT = 128;               // threads of a pair block
constexpr int kCs = 10;                // doubles between coefficient entries in shared memory:
                                       // 80 bytes spread neighbouring types over the banks

// A table holds the pair's entries with the sites of one of its molecules as rows and is kept
// for both (tab[pair][rows: lower, higher][SR, LR]), so that every visit reads the third
// molecule's sites as columns.  Rows x and columns c in 0..15 (sites 1..16) lie in operand
// fragments of 8 rows x 4 columns, lane r * 4 + ci of a fragment holding (8 rt + r, 4 cb + ci):
// 512 contiguous bytes per load.  Then (x, site 0), (site 0, c) and (site 0, site 0), padded to
// whole 128-byte lines.
constexpr int kCol0 = 256, kRow0 = 272, k00 = 288;
constexpr int kTabS = kFs3PairTab;
__host__ __device__ constexpr int frag_of(int x, int c) {
  return (x >> 3) * 128 + (c >> 2) * 32 + (x & 7) * 4 + (c & 3);
}
__device__ __forceinline__ int entry_of(int a, int b) {  // sites 0..16, rows a
  if (a && b) return frag_of(a - 1, b - 1);
  return a ? kCol0 + a - 1 : (b ? kRow0 + b - 1 : k00);
}
// type of site 1 + x
__host__ __device__ constexpr int type16(int x) { return x < 4 ? 1 + (x >> 1) : 2 + (x >> 2); }

// ------------------------------------------------------------------ near lists and pairs
// One warp per molecule i: the neighbours within FS3's cut-off in increasing order (near),
// how many of them are below i, and one pair (i, j) with its vector per neighbour above i.
// The radius is widened by 1e-9: a triple whose j-k distance passes the cut-off test by the
// reference's consistent-image vector must find its pair although the minimum-image vector's
// rounding differs.  Every triple is still tested exactly (k_fs3_visits).
__global__ void k_fs3_near(const double4 *__restrict__ comb, const int *__restrict__ nbr,
                           const int *__restrict__ ncnt, int cap, int nm, Fs3Params P, int *near,
                           int4 *head, double4 *pairv, int2 *pairij, int *vcnt, int pair_cap,
                           int *icnt) {
  const int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (i >= nm) return;
  const double4 ci = comb[i];
  const double rc2 = P.rc2 * (1.0 + 1e-9);
  const int cnt = ncnt[i];
  int n = 0, below = 0;
  for (int pass = 0, base = 0; pass < 2; pass++) {
    int m = 0;
    for (int n0 = 0; n0 < cnt; n0 += 32) {
      const int t = n0 + lane;
      bool keep = false;
      int j = 0;
      double x = 0, y = 0, z = 0, r2 = 0;
      if (t < cnt) {
        j = nbr[(size_t)i * cap + t];
        const double4 cj = comb[j];
        x = minimg(xsub(ci.x, cj.x), P.boxb);
        y = minimg(xsub(ci.y, cj.y), P.boxb);
        z = minimg(xsub(ci.z, cj.z), P.boxb);
        r2 = norm2x(x, y, z);
        keep = r2 < rc2;
      }
      const unsigned bal = __ballot_sync(0xffffffffu, keep);
      const int pos = m + __popc(bal & ((1u << lane) - 1u));
      if (pass == 0) {
        if (keep) near[(size_t)i * cap + pos] = j;
        below += __popc(__ballot_sync(0xffffffffu, keep && j < i));
      } else if (keep && j > i) {
        const int p = base + pos - below;
        if (p < pair_cap) {
          pairv[p] = make_double4(x, y, z, r2);
          pairij[p] = make_int2(i, j);
          vcnt[p * 2] = vcnt[p * 2 + 1] = 0;
        }
      }
      m += __popc(bal);
    }
    if (pass == 0) {
      n = m;
      if (lane == 0) {
        base = atomicAdd(&icnt[C_NPAIR_FS3], n - below);
        head[i] = make_int4(n, below, base, 0);
      }
      base = __shfl_sync(0xffffffffu, base, 0);
    }
  }
}

// --------------------------------------------------------------------- pair tables
// (e, e d) of every site pair of every molecule pair, SR and LR, by rows of either molecule, and
// the force-weight factors (e l / d, e l + e / d), l = d ln e / dr, by rows of the lower.
__device__ __forceinline__ void fs3_tables(int block, int nblocks,
                                           const double4 *__restrict__ pairv,
                                           const int2 *__restrict__ pairij, const int *icnt,
                                           int pair_cap, const double4 *__restrict__ s17,
                                           const double *__restrict__ bgr, double2 *tab,
                                           double2 *wtab) {
  const int np = min(icnt[C_NPAIR_FS3], pair_cap);
  const long long total = (long long)np * kTab;
  for (long long t = block * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)nblocks * blockDim.x) {
    const int p = (int)(t / kTab), q = (int)(t - (long long)p * kTab);
    const int a = q / kNs3, b = q - a * kNs3, e0 = entry_of(a, b), e1 = entry_of(b, a);
    const double4 R = pairv[p];
    const int2 ij = pairij[p];
    const double4 sa = s17[(size_t)ij.x * kNs3 + a], sb = s17[(size_t)ij.y * kNs3 + b];
    const double vx = R.x + (sa.x - sb.x), vy = R.y + (sa.y - sb.y), vz = R.z + (sa.z - sb.z);
    const double r = sqrt(vx * vx + vy * vy + vz * vz);
#pragma unroll
    for (int v = 0; v < 2; v++) {
      const double *g = bgr + v * 3 * kTab;
      const double bb = g[q], gg = g[kTab + q], r0 = g[2 * kTab + q];
      const double ex = exp(-gg * (r - r0));
      // one division gives both the damping 1/(1+x) and 1/r
      const double w = 1.0 / ((1.0 + ex) * r);
      const double eor = exp(-bb * r) * w;  // e / r
      const double ee = eor * r;
      const double dln = -bb + gg * ex * (w * r);
      const double2 u = make_double2(ee, ee * r);
      tab[((size_t)p * 4 + v) * kTabS + e0] = u;
      tab[((size_t)p * 4 + 2 + v) * kTabS + e1] = u;
      wtab[((size_t)p * 2 + v) * kTabS + e0] = make_double2(eor * dln, ee * dln + eor);
    }
  }
}

// ------------------------------------------------------------------------ visits
struct Visit {
  unsigned tv, tw;  // first entries of the tables of (A, C) by rows A and of (B, C) by rows B
  double w;    // the triple's weight in this variant
};
// A triple: molecules, pairs (ij, ik, jk) and the weights of its SR and LR sums in the energy and
// in the COM forces (a variant that the triple does not take has w = 0).
struct Triple {
  int mol[3], pair[3], branch, pad;
  double w[2], wc[2];
};

// Position of j among the pairs of i (i < j), or -1.
__device__ __forceinline__ int pair_of(const int *__restrict__ near, const int4 &h, int cap, int i,
                                       int j) {
  const int *l = near + (size_t)i * cap;
  int lo = h.y, hi = h.x;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (l[mid] < j) lo = mid + 1;
    else hi = mid;
  }
  return lo < h.x && l[lo] == j ? h.z + lo - h.y : -1;
}

// One block per molecule i: the triples i < j < k with the reference's exact cut-off tests
// (threebody_potential.f90:860-892, as k_fs3_enum), each added to the visit lists (SR, LR) of
// its three pairs.
__device__ __forceinline__ void fs3_visits(int i, const double4 *__restrict__ comb,
                                           const int *__restrict__ near,
                                           const int4 *__restrict__ head, int cap,
                                           const Fs3Params &P, Visit *vis, int *vcnt, int vcap,
                                           int pair_cap, Triple *tri, int tri_cap, int *icnt) {
  extern __shared__ unsigned char smem_raw[];
  double *lx = reinterpret_cast<double *>(smem_raw);
  double *ly = lx + cap, *lz = ly + cap;
  int *lj = reinterpret_cast<int *>(lz + cap), *lr = lj + cap;
  __shared__ int nl, wcount[32];
  const int4 hi = head[i];
  if (threadIdx.x == 0) nl = 0;
  __syncthreads();
  const double4 ci = comb[i];
  for (int n0 = hi.y; n0 < hi.x; n0 += blockDim.x) {
    const int n = n0 + threadIdx.x;
    bool keep = false;
    int j = 0;
    double xij = 0, yij = 0, zij = 0;
    if (n < hi.x) {
      j = near[(size_t)i * cap + n];
      const double4 cj = comb[j];
      xij = minimg(xsub(ci.x, cj.x), P.boxb);
      yij = minimg(xsub(ci.y, cj.y), P.boxb);
      zij = minimg(xsub(ci.z, cj.z), P.boxb);
      keep = norm2x(xij, yij, zij) < P.rc2;
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const unsigned bal = __ballot_sync(0xffffffffu, keep);
    if (lane == 0) wcount[wid] = __popc(bal);
    __syncthreads();
    int off = nl;
    for (int w = 0; w < wid; w++) off += wcount[w];
    if (keep) {
      const int pos = off + __popc(bal & ((1u << lane) - 1u));
      lj[pos] = j;
      lr[pos] = hi.z + n - hi.y;
      lx[pos] = xij;
      ly[pos] = yij;
      lz[pos] = zij;
    }
    __syncthreads();
    if (threadIdx.x == 0)
      for (int w = 0; w < (int)(blockDim.x >> 5); w++) nl += wcount[w];
    __syncthreads();
  }
  const int L = nl;
  const double b = P.boxb;
  const int npairs = L * (L - 1) / 2;
  for (int t = threadIdx.x; t < npairs; t += blockDim.x) {
    const double h = 2.0 * L - 1.0;
    int a = (int)floor(0.5 * (h - sqrt(h * h - 8.0 * t)));
    while (a > 0 && a * L - a * (a + 1) / 2 > t) a--;
    while ((a + 1) * L - (a + 1) * (a + 2) / 2 <= t) a++;
    const int c = t - (a * L - a * (a + 1) / 2) + a + 1;
    const int j = lj[a], k = lj[c];
    const double4 cj = comb[j], ck = comb[k];
    const double dxik = xsub(ci.x, ck.x), dyik = xsub(ci.y, ck.y), dzik = xsub(ci.z, ck.z);
    // xjk = dxjk + box*nint(dxij/box) - box*nint(dxik/box)  (threebody_potential.f90:883-885)
    const double dxij = xsub(ci.x, cj.x), dyij = xsub(ci.y, cj.y), dzij = xsub(ci.z, cj.z);
    const double xjk = xsub(xadd(xsub(cj.x, ck.x), xmul(b, round(__ddiv_rn(dxij, b)))),
                            xmul(b, round(__ddiv_rn(dxik, b))));
    const double yjk = xsub(xadd(xsub(cj.y, ck.y), xmul(b, round(__ddiv_rn(dyij, b)))),
                            xmul(b, round(__ddiv_rn(dyik, b))));
    const double zjk = xsub(xadd(xsub(cj.z, ck.z), xmul(b, round(__ddiv_rn(dzij, b)))),
                            xmul(b, round(__ddiv_rn(dzik, b))));
    const double djk2 = norm2x(xjk, yjk, zjk);
    if (!(djk2 < P.rc2)) continue;
    const double rij = sqrt(norm2x(lx[a], ly[a], lz[a])), rik = sqrt(norm2x(lx[c], ly[c], lz[c])),
                 rjk = sqrt(djk2);
    const double ravg = (rij + rjk + rik) / 3.0;  // threebody_potential.f90:894-898
    const int branch = ravg <= P.rmin ? 0 : (ravg >= P.rmax ? 1 : 2);
    if (branch == 2) atomicAdd(&icnt[C_NBLEND_FS3], 1);
    const int slot = atomicAdd(&icnt[C_NTRI_FS3], 1);
    if (slot >= tri_cap) continue;  // the host grows the list and re-runs
    const int pij = lr[a], pik = lr[c], pjk = pair_of(near, head[j], cap, j, k);
    if (pjk < 0 || max(max(pij, pik), pjk) >= pair_cap) {
      // no such pair within the widened radius (the host takes the triple form), or no room for
      // one of the pairs (it grows the list): the evaluation is repeated.  Every counted record
      // is written all the same, this one with the valid indices 0 and no weight: a reader of
      // the list must not meet what the memory held before.
      if (pjk < 0) atomicAdd(&icnt[C_FS3_MISS], 1);
      tri[slot] = Triple{};
      continue;
    }
    // global damping and switch (threebody_potential.f90:898-904, 1418-1423)
    const double pom = exp(P.alp3 * (ravg - P.r0dmp));
    const double ppom = 1.0 / (1.0 + pom);
    const double fdmp = pow(ppom, P.delta33);
    const double dfdmp = -P.alp3 * P.delta33 * pom * ppom * fdmp * (1.0 / 3.0);
    const double cfact = (ravg - P.rmin) / (P.rmax - P.rmin);
    const double smfun = 1.0 + 2.0 * cfact * cfact * cfact - 3.0 * cfact * cfact;
    const double cf = 2.0 / (P.rmax - P.rmin) * (cfact * cfact - cfact);
    Triple T;
    T.mol[0] = i;
    T.mol[1] = j;
    T.mol[2] = k;
    T.pair[0] = pij;
    T.pair[1] = pik;
    T.pair[2] = pjk;
    T.branch = branch;
    T.pad = 0;
    // pairs ij, ik, jk with third molecule k, j, i
    const int tv[3] = {2 * pik, 2 * pij, 2 * pij + 1}, tw[3] = {2 * pjk, 2 * pjk + 1, 2 * pik + 1};
    for (int v = 0; v < 2; v++) {
      const double sw = branch == 2 ? (v == 0 ? smfun : 1.0 - smfun) : (branch == v ? 1.0 : 0.0);
      T.w[v] = fdmp * sw;
      T.wc[v] = dfdmp * sw + (branch != 2 ? 0.0 : (v == 0 ? fdmp * cf : -fdmp * cf));
      if (branch == 1 - v) continue;
      for (int role = 0; role < 3; role++) {
        const int list = T.pair[role] * 2 + v;
        Visit V;
        V.tv = (unsigned)(tv[role] * 2 + v) * kTabS;
        V.tw = (unsigned)(tw[role] * 2 + v) * kTabS;
        V.w = T.w[v];
        const int pos = atomicAdd(&vcnt[list], 1);
        if (pos < vcap)
          vis[(size_t)list * vcap + pos] = V;
        else
          atomicMax(&icnt[C_FS3_VMAX], pos + 1);
      }
    }
    tri[slot] = T;
  }
}

// Blocks [0, nm): the visits of a molecule's triples; the others: the tables.  One launch, since
// neither fills the GPU's pipes by itself (atomics and stores) and neither needs the other.
__global__ void __launch_bounds__(128)
    k_fs3_lists(const double4 *__restrict__ comb, const int *__restrict__ near,
                const int4 *__restrict__ head, int cap, int nm, Fs3Params P, Visit *vis, int *vcnt,
                int vcap, int pair_cap, Triple *tri, int tri_cap,
                const double4 *__restrict__ pairv, const int2 *__restrict__ pairij,
                const double4 *__restrict__ s17, const double *__restrict__ bgr, double2 *tab,
                double2 *wtab, int *icnt) {
  if ((int)blockIdx.x < nm)
    fs3_visits(blockIdx.x, comb, near, head, cap, P, vis, vcnt, vcap, pair_cap, tri, tri_cap, icnt);
  else
    fs3_tables(blockIdx.x - nm, gridDim.x - nm, pairv, pairij, icnt, pair_cap, s17, bgr, tab, wtab);
}

// Whether the lists hold every pair, visit and triple that was found.  If not, the host repeats
// the evaluation and the kernels that use the lists have nothing to do.
__device__ __forceinline__ bool fs3_lists_whole(const int *__restrict__ icnt, int pair_cap) {
  return icnt[C_NPAIR_FS3] <= pair_cap && icnt[C_FS3_VMAX] == 0 && icnt[C_FS3_MISS] == 0 &&
         icnt[C_OVERFLOW] == 0;
}

// D = A (8x4) B (4x8) + C in FP64: lane l holds A[l/4][l%4], B[l%4][l/4] and C, D
// [l/4][2 (l%4) + {0, 1}].
__device__ __forceinline__ double2 dmma(double a, double b, double2 c) {
  double2 d;
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%4, %5};"
      : "=d"(d.x), "=d"(d.y)
      : "d"(a), "d"(b), "d"(c.x), "d"(c.y));
  return d;
}

__device__ __forceinline__ void fma2(double2 &a, double s, const double2 &m) {
  a.x += s * m.x;
  a.y += s * m.y;
}

// Extra shared memory of the parameter-gradient form: the block's sums of dS/d(coefficient
// table entry), every triple counted from its three pairs, and of dS/d(b, g, r0).
struct PairGrad {
  double gc[2][kCoef];
  double gb[2][3][kTab];
};

// Constants of a lane: r = lane / 4, ci = lane % 4.  Its operand fragments are V(8 at + r, c)
// and W(8 bt + r, c), c = 4 cb + ci, and their column of site 0; its results the pairs (8 at +
// r, 8 bt + 2 ci + {0, 1}).
struct Lane {
  int a, b;    // rows of the V and W fragments
  int fa, fb;  // places of the first fragments
  int b0;      // first of the two columns
  int r, ci, wid;  // wid: the warp's tile, 0..3
};

// Accumulators over the visits, sum_C w_C V_q W_r: m[type of the half][2 q + r] of the lane's
// two pairs; edge products own_i zero_j per fragment of the half, e[f][i] over j; the pair
// (site 0, site 0), z[i] over j, from one fragment.
struct Acc {
  double2 m[3][4];
  double2 e[3][2];
  double2 z[2];
};

__device__ __forceinline__ double2 mask2(bool on, const double2 &v) {
  return on ? v : make_double2(0.0, 0.0);
}

// One type of one visit: the four power pairs of the tile.
__device__ __forceinline__ void tile_products(const double2 &v, const double2 &u, double2 (&m)[4]) {
  m[0] = dmma(v.x, u.x, m[0]);
  m[1] = dmma(v.x, u.y, m[1]);
  m[2] = dmma(v.y, u.x, m[2]);
  m[3] = dmma(v.y, u.y, m[3]);
}
// Products of one fragment with a row of site 0.
__device__ __forceinline__ void edge_products(const double2 &own, const double2 &zero,
                                              double2 (&m)[2]) {
  fma2(m[0], own.x, zero);
  fma2(m[1], own.y, zero);
}
__device__ __forceinline__ double2 scaled(double w, const double2 &v) {
  return make_double2(w * v.x, w * v.y);
}

// The operands of one fragment of a visit: V's and W's and the edge's row of site 0; of site 0
// itself W's entries of the lane's two columns (x) beside that of its row (u).
struct Frag {
  double2 v, u, z, x[2];
};
// Fragment F of a half: HALF 0 has site 0 (F = 0) and the two-site types (1), HALF 1 the types
// 3..5.  COL: the warp's edge is the pairs (a, site 0), products of V with W's row of site 0,
// else (site 0, b), of W with V's.
template <int HALF, bool COL, int F>
__device__ __forceinline__ Frag load_frag(const double2 *__restrict__ V,
                                          const double2 *__restrict__ W, const Lane &L) {
  const double2 *Z = COL ? W : V;
  Frag X;
  if (HALF == 0 && F == 0) {
    X.v = __ldg(V + kCol0 + L.a);
    if (!COL) X.u = __ldg(W + kCol0 + L.b);
    X.z = __ldg(Z + k00);
    X.x[0] = __ldg(W + kCol0 + L.b0);
    X.x[1] = __ldg(W + kCol0 + L.b0 + 1);
  } else {
    constexpr int cb = HALF == 0 ? 0 : F + 1;
    X.v = __ldg(V + L.fa + 32 * cb);
    X.u = __ldg(W + L.fb + 32 * cb);
    X.z = __ldg(Z + kRow0 + 4 * cb + L.ci);
  }
  return X;
}

// Its products with the visit's weight w, which goes on the edge's operand: the tile and the
// edge share it.
template <int HALF, bool COL, int F>
__device__ __forceinline__ void use_frag(const Frag &X, double w, const Lane &L, Acc &A) {
  if (HALF == 0 && F == 0) {  // one site: each lane's two pairs multiplied out
    const double2 s = scaled(w, X.v);
    fma2(A.m[0][0], s.x, make_double2(X.x[0].x, X.x[1].x));
    fma2(A.m[0][1], s.x, make_double2(X.x[0].y, X.x[1].y));
    fma2(A.m[0][2], s.y, make_double2(X.x[0].x, X.x[1].x));
    fma2(A.m[0][3], s.y, make_double2(X.x[0].y, X.x[1].y));
    edge_products(mask2(L.ci == 0, COL ? s : scaled(w, X.u)), X.z, A.e[0]);
    return;
  }
  const double2 s = scaled(w, COL ? X.v : X.u);
  if (HALF == 0) {
    const bool lo = L.ci < 2;
    const double2 sl = mask2(lo, s), sh = mask2(!lo, s);
    tile_products(COL ? sl : X.v, COL ? X.u : sl, A.m[1]);
    tile_products(COL ? sh : X.v, COL ? X.u : sh, A.m[2]);
  } else {
    tile_products(COL ? s : X.v, COL ? X.u : s, A.m[F]);
  }
  edge_products(s, X.z, A.e[F]);
}

// The pair (site 0, site 0): one fragment per warp.
template <int HALF, bool COL>
__device__ __forceinline__ void use_zero(const double2 *__restrict__ V,
                                         const double2 *__restrict__ W, double w, const Lane &L,
                                         Acc &A) {
  if (HALF == 0 ? L.wid >= 2 : L.wid == 3) return;
  const int c = HALF == 1 ? kRow0 + 4 * (L.wid + 1) + L.ci : (L.wid == 0 ? k00 : kRow0 + L.ci);
  const bool on = L.r == 0 && (HALF == 1 || L.wid == 1 || L.ci == 0);
  edge_products(mask2(on, scaled(w, __ldg(V + c))), __ldg(W + c), A.z);
}

// Asks for the lines of the next visit's tables that this half reads: the block's warps share
// them, warp 0 asks for V's and warp 1 for W's.  A load then finds them in L1 instead of
// waiting for L2.  line: the lane's line, or -1: lines 0-3, 16-19 (fragments 0) and 32-36 (site
// 0) in HALF 0; 4-15, 20-31 (fragments 1-3) and 34, 35 (the row of site 0) in HALF 1.
template <int HALF>
__device__ __forceinline__ int prefetch_line(int lane, int wid) {
  if (wid > 1 || lane >= (HALF == 0 ? 13 : 26)) return -1;
  if (HALF == 0) return lane < 4 ? lane : (lane < 8 ? 12 + lane : 24 + lane);
  return lane < 12 ? 4 + lane : (lane < 24 ? 8 + lane : 10 + lane);
}
__device__ __forceinline__ void prefetch_l1(const double2 *p) {
  asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}

// The 8 coefficients of a type triple, index 4 r + 2 q + p.
struct Coef {
  double c[8];
};
__device__ __forceinline__ Coef load_coef(const double *__restrict__ C, int ta, int tb, int tc,
                                          int stride = 8) {
  Coef k;
  const double2 *p =
      reinterpret_cast<const double2 *>(C + ((ta * kNt + tb) * kNt + tc) * stride);
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const double2 v = p[i];
    k.c[2 * i] = v.x;
    k.c[2 * i + 1] = v.y;
  }
  return k;
}
// (q0, q1) += c_(o, o+1) m
__device__ __forceinline__ void unfold(double2 &q, const Coef &k, int o, double m) {
  q.x += k.c[o] * m;
  q.y += k.c[o + 1] * m;
}
// Coefficient offset of power pair n = 2 q + r.  An edge's n = 2 i + j has (q, r) = (i, j)
// when its own table is V, else (j, i): offset 2 i + 4 j or 4 i + 2 j.
__host__ __device__ constexpr int off_qr(int n) { return 4 * (n & 1) + 2 * (n >> 1); }
// (q0, q1) of a tile's two site pairs from the products of one type.
__device__ __forceinline__ void unfold_tile(double2 (&q)[2], const Coef &k, const double2 (&m)[4]) {
#pragma unroll
  for (int n = 0; n < 4; n++) {
    unfold(q[0], k, off_qr(n), m[n].x);
    unfold(q[1], k, off_qr(n), m[n].y);
  }
}
// The same of an edge (or of site pair (0, 0), with own_v).
__device__ __forceinline__ void unfold_edge(double2 &q, const Coef &k, bool own_v,
                                            const double2 (&m)[2]) {
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int p = 0; p < 2; p++) {
      const double a = own_v ? k.c[2 * i + p] : k.c[4 * i + p];
      const double b = own_v ? k.c[2 * i + 4 + p] : k.c[4 * i + 2 + p];
      double &t = p ? q.y : q.x;
      t += a * m[i].x;
      t += b * m[i].y;
    }
}

// Sum over the lanes that differ in the given lane bits and hold the same site types (s1, s2,
// s3: whether this lane takes part in each step), added by the leading lane.  The warp owns
// the entry within its block, so a plain addition is enough.
__device__ __forceinline__ void grad_add(double *g, double v, int b1, bool s1, int b2, bool s2,
                                         int b3, bool s3, bool lead) {
  double t = __shfl_xor_sync(0xffffffffu, v, b1);
  if (s1) v += t;
  t = __shfl_xor_sync(0xffffffffu, v, b2);
  if (s2) v += t;
  t = __shfl_xor_sync(0xffffffffu, v, b3);
  if (s3) v += t;
  if (lead) *g += v;
}

// What the visits of one variant leave of a pair: (q0, q1) of the lane's two site pairs, its
// share of the edge pair's and of (site 0, site 0).
struct Result {
  double2 m[2], e, z;
};

// A pair's n visits in one variant, types of one half.
template <int HALF, bool COL, bool GRAD>
__device__ __forceinline__ void half_pass(const Visit *__restrict__ vis, int n,
                                          const double2 *__restrict__ tab, int v,
                                          const double2 *__restrict__ U,
                                          const double *__restrict__ C, const Lane &L, double *gc,
                                          Result &R) {
  constexpr int kF = HALF == 0 ? 2 : 3;
  const int b0 = 8 * (L.wid & 1) + 2 * L.ci;  // first of the lane's two columns
  const int ta = type16(L.a), tb = type16(b0), x = COL ? L.a : L.b, tx = type16(x);
  const int ea = COL ? tx : 0, eb = COL ? 0 : tx;
  // type of the lane's site c in fragment f
  auto edge_type = [&](int f) { return HALF == 1 ? 3 + f : (f == 0 ? 0 : (L.ci < 2 ? 1 : 2)); };
  const int zt = HALF == 1 ? 3 + (L.wid < 3 ? L.wid : 0) : (L.wid == 0 ? 0 : (L.ci < 2 ? 1 : 2));
  Acc A;
#pragma unroll
  for (int t = 0; t < 3; t++) {
#pragma unroll
    for (int k = 0; k < 4; k++) A.m[t][k] = make_double2(0.0, 0.0);
    A.e[t][0] = A.e[t][1] = make_double2(0.0, 0.0);
  }
  A.z[0] = A.z[1] = make_double2(0.0, 0.0);
  // a visit's record is loaded two visits ahead, its tables' lines are asked for one ahead
  const int line = prefetch_line<HALF>(threadIdx.x & 31, L.wid);
  uint2 h = __ldg(reinterpret_cast<const uint2 *>(vis));
  double w = __ldg(&vis->w);
  const Visit *q = vis + (n > 1 ? 1 : 0);
  uint2 h1 = __ldg(reinterpret_cast<const uint2 *>(q));
  double w1 = __ldg(&q->w);
#pragma unroll 1
  for (int t = 0; t < n; t++) {
    const double2 *V = tab + h.x, *W = tab + h.y;
    const double wt = w;
    h = h1;
    w = w1;
    if (line >= 0) prefetch_l1(tab + (L.wid == 0 ? h.x : h.y) + 8 * line);
    if (t + 2 < n) q++;
    h1 = __ldg(reinterpret_cast<const uint2 *>(q));
    w1 = __ldg(&q->w);
    const Frag X = load_frag<HALF, COL, 0>(V, W, L), Y = load_frag<HALF, COL, 1>(V, W, L);
    if (HALF == 1) {
      const Frag Z = load_frag<HALF, COL, 2>(V, W, L);
      use_frag<HALF, COL, 0>(X, wt, L, A);
      use_frag<HALF, COL, 1>(Y, wt, L, A);
      use_frag<HALF, COL, HALF == 1 ? 2 : 1>(Z, wt, L, A);
    } else {
      use_frag<HALF, COL, 0>(X, wt, L, A);
      use_frag<HALF, COL, 1>(Y, wt, L, A);
    }
    use_zero<HALF, COL>(V, W, wt, L, A);
  }
#pragma unroll
  for (int t = 0; t < 3; t++) unfold_tile(R.m, load_coef(C, ta, tb, 3 * HALF + t), A.m[t]);
#pragma unroll
  for (int f = 0; f < kF; f++) unfold_edge(R.e, load_coef(C, ea, eb, edge_type(f)), COL, A.e[f]);
  const bool zon = HALF == 1 ? L.wid < 3 : L.wid < 2;
  if (zon) unfold_edge(R.z, load_coef(C, 0, 0, zt), true, A.z);
  if (GRAD) {
    const int ek = (COL ? kCol0 : kRow0) + x, mk = frag_of(L.a, b0);
    const double2 u0 = __ldg(U + mk), u1 = __ldg(U + mk + 1), ue = __ldg(U + ek),
                  uz = __ldg(U + k00);
    {
      const bool r2 = (L.r & 4) || L.wid >= 2, c1 = (L.ci & 2) || (L.wid & 1);
      const bool lead = !(L.r & 1) && !(r2 && (L.r & 2)) && !(c1 && (L.ci & 1));
#pragma unroll
      for (int t = 0; t < 3; t++)
#pragma unroll
        for (int q = 0; q < 4; q++) {
          double *g = gc + ((ta * kNt + tb) * kNt + 3 * HALF + t) * 8 + off_qr(q);
          const double2 m = A.m[t][q];
          grad_add(g, u0.x * m.x + u1.x * m.y, 4, true, 8, r2, 1, c1, lead);
          grad_add(g + 1, u0.y * m.x + u1.y * m.y, 4, true, 8, r2, 1, c1, lead);
        }
    }
    // edges: the four lanes of a row hold the sites c of one type (fragment c0: one lane), or
    // in fragment 0 two types; rows of one type are summed
    {
      const bool r2 = x >= 4;
#pragma unroll
      for (int f = 0; f < kF; f++) {
        const bool one = HALF == 1 || f == 0;
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
          for (int j = 0; j < 2; j++) {
            const double m = j ? A.e[f][i].y : A.e[f][i].x;
#pragma unroll
            for (int k = 0; k < 2; k++) {
              double s = (k ? ue.y : ue.x) * m;
              s += __shfl_xor_sync(0xffffffffu, s, 1);
              const double t = __shfl_xor_sync(0xffffffffu, s, 2);
              if (one) s += t;
              double *g = gc + ((ea * kNt + eb) * kNt + edge_type(f)) * 8 +
                          (COL ? 2 * i + 4 * j : 4 * i + 2 * j) + k;
              const bool lead = !(L.ci & 1) && !(one && (L.ci & 2)) && !(L.r & 1) &&
                                !(r2 && (L.r & 2));
              grad_add(g, s, 4, true, 8, r2, 16, false, lead);
            }
          }
      }
      if (zon) {
        const bool one = HALF == 1 || L.wid == 0;
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
          for (int j = 0; j < 2; j++) {
            const double m = j ? A.z[i].y : A.z[i].x;
#pragma unroll
            for (int k = 0; k < 2; k++) {
              double s = (k ? uz.y : uz.x) * m;  // lanes beyond row 0 hold zeros
              s += __shfl_xor_sync(0xffffffffu, s, 1);
              const double t = __shfl_xor_sync(0xffffffffu, s, 2);
              if (one) s += t;
              if (L.r == 0 && !(L.ci & 1) && !(one && (L.ci & 2)))
                gc[zt * 8 + 2 * i + 4 * j + k] += s;
            }
          }
      }
    }
  }
}

__device__ __forceinline__ double sum_bits(double v, int b0, int b1) {
  for (int b = b0; b < b1; b <<= 1) v += __shfl_xor_sync(0xffffffffu, v, b);
  return v;
}

template <bool GRAD>
__global__ void __launch_bounds__(kPT, GRAD ? 2 : CCP_FS3_PAIR_BLOCKS)
    k_fs3_pair(const double4 *__restrict__ pairv, const int2 *__restrict__ pairij,
               const Visit *__restrict__ vis, const int *__restrict__ vcnt, int vcap, int pair_cap,
               const double2 *__restrict__ tab, const double2 *__restrict__ wtab,
               const double4 *__restrict__ s17, const double *__restrict__ coef,
               const double *__restrict__ bgr, int nm, int ns, double *f,
               double *vpart, double *gfs3, const int *__restrict__ icnt) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  PairGrad *GS = reinterpret_cast<PairGrad *>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int np = min(icnt[C_NPAIR_FS3], pair_cap);
  if (!fs3_lists_whole(icnt, pair_cap)) return;
  if (GRAD) {
    for (int t = tid; t < 2 * kCoef; t += kPT) (&GS->gc[0][0])[t] = 0.0;
    for (int t = tid; t < 2 * 3 * kTab; t += kPT) (&GS->gb[0][0][0])[t] = 0.0;
    __syncthreads();
  }
  Lane L;
  L.r = lane >> 2;
  L.ci = lane & 3;
  L.wid = wid;
  L.a = 8 * (wid >> 1) + L.r;
  L.b = 8 * (wid & 1) + L.r;
  L.fa = 128 * (wid >> 1) + lane;
  L.fb = 128 * (wid & 1) + lane;
  const bool col = (wid >> 1) == (wid & 1);
  const int b0 = 8 * (wid & 1) + 2 * L.ci, mk = frag_of(L.a, b0);
  L.b0 = b0;
  const int x = col ? L.a : L.b, ek = (col ? kCol0 : kRow0) + x;
  for (int p = blockIdx.x; p < np; p += gridDim.x) {
    double g0 = 0.0, g1 = 0.0, ge = 0.0, gz = 0.0;  // force weights (ge, gz: this lane's share)
    bool any = false;
#pragma unroll 1
    for (int v = 0; v < 2; v++) {
      const int n = min(__ldg(&vcnt[p * 2 + v]), vcap);
      if (n == 0) continue;
      any = true;
      const Visit *lv = vis + ((size_t)p * 2 + v) * vcap;
      const double2 *U = tab + ((size_t)p * 4 + v) * kTabS;
      const double *C = coef + v * kCoef;
      double *gc = GRAD ? GS->gc[v] : nullptr;
      Result R;
      R.m[0] = R.m[1] = R.e = R.z = make_double2(0.0, 0.0);
      if (col) {
        half_pass<0, true, GRAD>(lv, n, tab, v, U, C, L, gc, R);
        half_pass<1, true, GRAD>(lv, n, tab, v, U, C, L, gc, R);
      } else {
        half_pass<0, false, GRAD>(lv, n, tab, v, U, C, L, gc, R);
        half_pass<1, false, GRAD>(lv, n, tab, v, U, C, L, gc, R);
      }
      // G = (e l / d) q0 + (e l + e / d) q1
      const double2 *Wt = wtab + ((size_t)p * 2 + v) * kTabS;
      const double2 w0 = __ldg(Wt + mk), w1 = __ldg(Wt + mk + 1), we = __ldg(Wt + ek),
                    wz = __ldg(Wt + k00);
      g0 += w0.x * R.m[0].x + w0.y * R.m[0].y;
      g1 += w1.x * R.m[1].x + w1.y * R.m[1].y;
      ge += we.x * R.e.x + we.y * R.e.y;
      gz += wz.x * R.z.x + wz.y * R.z.y;
      if (GRAD) {
        // dS/de = P = q0 + d q1; de/db = -d e, de/dg = (d - r0) e x, de/dr0 = -g e x with
        // x = exp(-g (d - r0)) / (1 + exp(-g (d - r0)))
        const double4 Rv = pairv[p];
        const int2 ij = pairij[p];
        auto param = [&](int a, int b, double2 q, double e, bool lead, bool shared) {
          const double4 sa = s17[(size_t)ij.x * kNs3 + a], sb = s17[(size_t)ij.y * kNs3 + b];
          const double vx = Rv.x + (sa.x - sb.x), vy = Rv.y + (sa.y - sb.y),
                       vz = Rv.z + (sa.z - sb.z);
          const double d = sqrt(vx * vx + vy * vy + vz * vz);
          const int c = a * kNs3 + b;
          const double *B = bgr + v * 3 * kTab;
          const double gg = B[kTab + c], rr = B[2 * kTab + c], ex = exp(-gg * (d - rr));
          const double xx = ex / (1.0 + ex), pe = (q.x + d * q.y) * e;
          const double t[3] = {-pe * d, pe * (d - rr) * xx, -pe * gg * xx};
          if (lead)
            for (int k = 0; k < 3; k++) {
              if (shared) atomicAdd(&GS->gb[v][k][c], t[k]);
              else GS->gb[v][k][c] += t[k];
            }
        };
        param(1 + L.a, 1 + b0, R.m[0], __ldg(&U[mk].x), true, false);
        param(1 + L.a, 2 + b0, R.m[1], __ldg(&U[mk + 1].x), true, false);
        const double2 qe = make_double2(sum_bits(R.e.x, 1, 4), sum_bits(R.e.y, 1, 4));
        param(col ? 1 + x : 0, col ? 0 : 1 + x, qe, __ldg(&U[ek].x), L.ci == 0, false);
        const double2 qz = make_double2(warp_sum(R.z.x), warp_sum(R.z.y));
        param(0, 0, qz, __ldg(&U[k00].x), lane == 0, true);
      }
    }
    // site forces: F_A = -sum_b G r, F_B = +sum_a G r, r the vector of the site pair; each
    // warp adds its own tile's, edge's and share of (0, 0)
    double vir = 0.0;
    if (any) {
      const double4 Rv = pairv[p];
      const int2 ij = pairij[p];
      const double4 *sA = s17 + (size_t)ij.x * kNs3, *sB = s17 + (size_t)ij.y * kNs3;
      const double4 a = sA[1 + L.a], a0 = sA[0], p0 = sB[1 + b0], p1 = sB[2 + b0], z0 = sB[0];
      const double ax = Rv.x + a.x, ay = Rv.y + a.y, az = Rv.z + a.z;
      double m0[3] = {ax - p0.x, ay - p0.y, az - p0.z}, m1[3] = {ax - p1.x, ay - p1.y, az - p1.z};
      double ze[3] = {Rv.x + (a0.x - z0.x), Rv.y + (a0.y - z0.y), Rv.z + (a0.z - z0.z)};
      double ve[3];
      if (col) {
        ve[0] = ax - z0.x;
        ve[1] = ay - z0.y;
        ve[2] = az - z0.z;
      } else {
        const double4 b = sB[1 + L.b];
        ve[0] = Rv.x + (a0.x - b.x);
        ve[1] = Rv.y + (a0.y - b.y);
        ve[2] = Rv.z + (a0.z - b.z);
      }
      const double conv = kH2kcal * 418.4 / kBohr2a;
      const size_t nfs = (size_t)nm * ns, fa = (size_t)ij.x * ns, fb = (size_t)ij.y * ns;
#pragma unroll
      for (int k = 0; k < 3; k++) {
        double h0 = g0 * m0[k], h1 = g1 * m1[k], he = ge * ve[k], hz = gz * ze[k];
        vir += h0 * m0[k] + h1 * m1[k] + he * ve[k] + hz * ze[k];
        double fr = h0 + h1 + (col ? he : 0.0);  // on the row's site of A (negative)
        fr = sum_bits(fr, 1, 4);
        if (L.ci == 0) atomicAdd(&f[k * nfs + fa + 1 + L.a], -fr * conv);
        h0 = sum_bits(h0, 4, 32);
        h1 = sum_bits(h1, 4, 32);
        if (L.r == 0) {
          atomicAdd(&f[k * nfs + fb + 1 + b0], h0 * conv);
          atomicAdd(&f[k * nfs + fb + 2 + b0], h1 * conv);
        }
        he = sum_bits(he, 1, 4);
        if (!col && L.ci == 0) atomicAdd(&f[k * nfs + fb + 1 + L.b], he * conv);
        he = sum_bits(he, 4, 32);
        hz = warp_sum(hz);
        if (lane == 0) {
          const double on_a = hz + (col ? 0.0 : he), on_b = hz + (col ? he : 0.0);
          atomicAdd(&f[k * nfs + fa], -on_a * conv);
          atomicAdd(&f[k * nfs + fb], on_b * conv);
        }
      }
      vir = warp_sum(vir);
    }
    if (lane == 0) vpart[(size_t)p * kFs3PairWarps + wid] = vir;
  }
  if (GRAD) {
    __syncthreads();
    for (int t = tid; t < 2 * kCoef; t += kPT) {
      const double g = (&GS->gc[0][0])[t] * (1.0 / 3.0);
      if (g != 0.0) atomicAdd(&gfs3[t], g);
    }
    for (int t = tid; t < 2 * 3 * kTab; t += kPT) {
      const double g = (&GS->gb[0][0][0])[t];
      if (g != 0.0) atomicAdd(&gfs3[2 * kCoef + t], g);
    }
  }
}

// Energies, and the damping and switch COM forces (threebody_potential.f90:1092-1120) and
// their virial: one warp per triple (i, j, k), in turn.  With U, V, W the tables of (ij), (ik),
// (jk), S is the sum over the site pairs (a, b) of U0 q0 + U1 q1, (q0, q1) from the same products
// as a visit's: four 8 x 8 tiles, the edges with a site 0 and (site 0, site 0).  The
// coefficients come from shared memory.  The pairs' virial is added up here as well.
constexpr int kET = 128;
__global__ void __launch_bounds__(kET, CCP_FS3_ENERGY_BLOCKS)
    k_fs3_energy(const double4 *__restrict__ comb, const Triple *__restrict__ tri, int tri_cap,
                 const double2 *__restrict__ tab, const double *__restrict__ coef,
                 const double *__restrict__ vpart, int pair_cap, Fs3Params P, int nm, double *fc3,
                 double *scal, int *icnt) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  if (!fs3_lists_whole(icnt, pair_cap)) return;
  double *Cs = reinterpret_cast<double *>(smem_raw);  // [2][216][kCs]
  for (int t = threadIdx.x; t < 2 * kCoef / 2; t += kET) {
    const double2 c = __ldg(reinterpret_cast<const double2 *>(coef) + t);
    *reinterpret_cast<double2 *>(Cs + (t >> 2) * kCs + 2 * (t & 3)) = c;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, r = lane >> 2, ci = lane & 3;
  const int w0 = blockIdx.x * (kET / 32) + (threadIdx.x >> 5), nw = gridDim.x * (kET / 32);
  const int nt = min(icnt[C_NTRI_FS3], tri_cap);
  const int nv = min(icnt[C_NPAIR_FS3], pair_cap) * kFs3PairWarps;
  const double conv = kH2kcal * 418.4 / kBohr2a;
  const bool c0 = ci == 0, lo = ci < 2;
  CompSum e_tot, v_tot;
  for (int t = blockIdx.x * kET + threadIdx.x; t < nv; t += gridDim.x * kET) v_tot.add(vpart[t]);
#pragma unroll 1
  for (int t = w0; t < nt;) {
    // the next triple, in the order of the warps' need: triples take one or two sums
    int next = 0;
    if (lane == 0) next = nw + atomicAdd(&icnt[C_FS3_TICKET], 1);
    const Triple &T = tri[t];
    double S[2] = {0.0, 0.0};
#pragma unroll 1
    for (int v = 0; v < 2; v++) {
      if (__ldg(&T.branch) == 1 - v) continue;
      const double2 *U = tab + ((size_t)__ldg(&T.pair[0]) * 4 + v) * kTabS;
      const double2 *V = tab + ((size_t)__ldg(&T.pair[1]) * 4 + v) * kTabS;
      const double2 *W = tab + ((size_t)__ldg(&T.pair[2]) * 4 + v) * kTabS;
      const double *C = Cs + v * kNt * kNt * kNt * kCs;
      double e = 0.0;
      double2 qz = make_double2(0.0, 0.0);
      // W's fragments stay in registers for both row tiles of V
      double2 wf[2][5];
#pragma unroll
      for (int bt = 0; bt < 2; bt++) {
#pragma unroll
        for (int f = 0; f < 4; f++) wf[bt][f] = __ldg(W + 128 * bt + 32 * f + lane);
        wf[bt][4] = __ldg(W + kCol0 + 8 * bt + r);
      }
#pragma unroll
      for (int bt = 0; bt < 2; bt++) {  // edge (site 0, b): W against V's row of site 0
        double2 q = make_double2(0.0, 0.0);
        const int b = 8 * bt + r, tb = type16(b);
#pragma unroll
        for (int f = 0; f < 5; f++) {
          const double2 z = __ldg(V + (f == 4 ? k00 : kRow0 + 4 * f + ci));
          const double2 o = f == 4 ? mask2(c0, wf[bt][f]) : wf[bt][f];
          const double2 M[2] = {make_double2(o.x * z.x, o.x * z.y),
                                make_double2(o.y * z.x, o.y * z.y)};
          const int tc = f == 4 ? 0 : (f ? 2 + f : (lo ? 1 : 2));
          unfold_edge(q, load_coef(C, 0, tb, tc, kCs), false, M);
        }
        const double2 u = __ldg(U + kRow0 + b);
        e += u.x * q.x + u.y * q.y;
      }
#pragma unroll 1
      for (int at = 0; at < 2; at++) {
        const int a = 8 * at + r, ta = type16(a);
        double2 vf[5];
        vf[4] = __ldg(V + kCol0 + a);
#pragma unroll
        for (int f = 0; f < 4; f++) vf[f] = __ldg(V + 128 * at + 32 * f + lane);
        {  // edge (a, site 0): V against W's row of site 0
          double2 q = make_double2(0.0, 0.0);
#pragma unroll
          for (int f = 0; f < 5; f++) {
            const double2 z = __ldg(W + (f == 4 ? k00 : kRow0 + 4 * f + ci));
            const double2 y = f == 4 ? mask2(c0, vf[f]) : vf[f];
            const double2 M[2] = {make_double2(y.x * z.x, y.x * z.y),
                                  make_double2(y.y * z.x, y.y * z.y)};
            const int tc = f == 4 ? 0 : (f ? 2 + f : (lo ? 1 : 2));
            unfold_edge(q, load_coef(C, ta, 0, tc, kCs), true, M);
          }
          const double2 u = __ldg(U + kCol0 + a);
          e += u.x * q.x + u.y * q.y;
        }
#pragma unroll
        for (int bt = 0; bt < 2; bt++) {
          const int b0 = 8 * bt + 2 * ci, tb = type16(b0), mk = frag_of(a, b0);
          const double2 u0 = __ldg(U + mk), u1 = __ldg(U + mk + 1), o = make_double2(0.0, 0.0);
          double2 q[2] = {o, o};
          {  // site 0: the lane's two pairs multiplied out
            const double2 x0 = __ldg(W + kCol0 + b0), x1 = __ldg(W + kCol0 + b0 + 1), y = vf[4];
            const double2 M[4] = {make_double2(y.x * x0.x, y.x * x1.x), make_double2(y.x * x0.y, y.x * x1.y),
                                  make_double2(y.y * x0.x, y.y * x1.x), make_double2(y.y * x0.y, y.y * x1.y)};
            unfold_tile(q, load_coef(C, ta, tb, 0, kCs), M);
          }
#pragma unroll
          for (int tc = 1; tc < 6; tc++) {
            const int f = tc < 3 ? 0 : tc - 2;
            const double2 x = tc == 1 ? mask2(lo, vf[0]) : (tc == 2 ? mask2(!lo, vf[0]) : vf[f]);
            const double2 M[4] = {dmma(x.x, wf[bt][f].x, o), dmma(x.x, wf[bt][f].y, o),
                                  dmma(x.y, wf[bt][f].x, o), dmma(x.y, wf[bt][f].y, o)};
            unfold_tile(q, load_coef(C, ta, tb, tc, kCs), M);
          }
          e += (u0.x * q[0].x + u0.y * q[0].y) + (u1.x * q[1].x + u1.y * q[1].y);
        }
      }
      // (site 0, site 0): lane c is third site c
      if (lane < kNs3) {
        const double2 x = __ldg(V + (lane ? kRow0 + lane - 1 : k00));
        const double2 z = __ldg(W + (lane ? kRow0 + lane - 1 : k00));
        const double2 M[2] = {make_double2(x.x * z.x, x.x * z.y), make_double2(x.y * z.x, x.y * z.y)};
        unfold_edge(qz, load_coef(C, 0, 0, lane ? type16(lane - 1) : 0, kCs), true, M);
        const double2 u = __ldg(U + k00);
        e += u.x * qz.x + u.y * qz.y;
      }
      S[v] = warp_sum(e);
    }
    // lanes 0..2: component of the forces on the three molecules
    const int m0 = __ldg(&T.mol[0]), m1 = __ldg(&T.mol[1]), m2 = __ldg(&T.mol[2]);
    const double wc0 = __ldg(&T.wc[0]), wc1 = __ldg(&T.wc[1]);
    const double4 ci4 = comb[m0], cj4 = comb[m1], ck4 = comb[m2];
    const double comc = wc0 * S[0] + wc1 * S[1], b = P.boxb;
    const double x[3] = {minimg(xsub(ci4.x, cj4.x), b), minimg(xsub(ci4.x, ck4.x), b),
                         minimg(xsub(cj4.x, ck4.x), b)};
    const double y[3] = {minimg(xsub(ci4.y, cj4.y), b), minimg(xsub(ci4.y, ck4.y), b),
                         minimg(xsub(cj4.y, ck4.y), b)};
    const double z[3] = {minimg(xsub(ci4.z, cj4.z), b), minimg(xsub(ci4.z, ck4.z), b),
                         minimg(xsub(cj4.z, ck4.z), b)};
    double rr[3], u[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
      rr[k] = sqrt(norm2x(x[k], y[k], z[k]));
      u[k] = comc * conv / rr[k] * (lane == 0 ? x[k] : (lane == 1 ? y[k] : z[k]));
    }
    if (lane < 3) {
      double *f = fc3 + (size_t)lane * nm;
      atomicAdd(f + m0, -(u[0] + u[1]));
      atomicAdd(f + m1, u[0] - u[2]);
      atomicAdd(f + m2, u[1] + u[2]);
    }
    if (lane == 0) {
      e_tot.add(__ldg(&T.w[0]) * S[0] + __ldg(&T.w[1]) * S[1]);
      v_tot.add(comc * (rr[0] + rr[1] + rr[2]));
    }
    t = __shfl_sync(0xffffffffu, next, 0);
  }
  const double vs = warp_sum(v_tot.value());
  if (lane == 0) {
    const double es = e_tot.value();
    if (es != 0.0) atomicAdd(&scal[S_FS3_E], es);
    if (vs != 0.0) atomicAdd(&scal[S_FS3_VIR], vs);
  }
}

template <bool GRAD>
cudaError_t launch_pair_t(const Fs3PairBufs &B, const int *icnt, const double4 *s17,
                          const double *coef, const double *bgr, int nm, int ns, double *f,
                          int nsm, double *gfs3, cudaStream_t st) {
  const size_t smem = GRAD ? sizeof(PairGrad) : 0;
  cudaError_t e = cudaFuncSetAttribute(k_fs3_pair<GRAD>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  // one short block per pair, so that blocks retire often and concurrent kernels take their
  // slots; the gradient form flushes per-block sums, so its blocks stay
  const int grid = GRAD ? 2 * nsm : B.pair_cap;
  k_fs3_pair<GRAD><<<grid, kPT, smem, st>>>(
      B.pairv, B.pairij, static_cast<const Visit *>(B.vis), B.vcnt, B.vcap, B.pair_cap, B.tab,
      B.wtab, s17, coef, bgr, nm, ns, f, B.vpart, gfs3, icnt);
  return cudaGetLastError();
}

}  // namespace

size_t fs3_visit_bytes() { return sizeof(Visit); }
// Shared memory of k_fs3_lists: a molecule's neighbours within the cut-off, at most its list.
static size_t fs3_lists_smem(int cap) { return (size_t)cap * (3 * sizeof(double) + 2 * sizeof(int)); }
constexpr size_t kListsSmemMax = 226 * 1024;  // 1 KB for the static arrays
bool fs3_pair_lists_fit(int cap) { return fs3_lists_smem(cap) <= kListsSmemMax; }
static_assert(sizeof(Triple) == 64, "triple record");

cudaError_t launch_fs3_pair_lists(const Fs3PairBufs &B, const double4 *comb, const int *nbr,
                                  const int *ncnt, int cap, int nm, Fs3Params P,
                                  const double4 *s17, const double *bgr, void *tri, int tri_cap,
                                  int *icnt, int nsm, cudaStream_t st) {
  k_fs3_near<<<(nm + 3) / 4, 128, 0, st>>>(comb, nbr, ncnt, cap, nm, P, B.near, B.head, B.pairv,
                                           B.pairij, B.vcnt, B.pair_cap, icnt);
  const size_t smem = fs3_lists_smem(cap);
  if (smem > 48 * 1024) {  // the same value from every thread: the limit is the kernel's
    cudaError_t e = cudaFuncSetAttribute(k_fs3_lists, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kListsSmemMax);
    if (e != cudaSuccess) return e;
  }
  k_fs3_lists<<<nm + nsm * 12, 128, smem, st>>>(
      comb, B.near, B.head, cap, nm, P, static_cast<Visit *>(B.vis), B.vcnt, B.vcap, B.pair_cap,
      static_cast<Triple *>(tri), tri_cap, B.pairv, B.pairij, s17, bgr, B.tab, B.wtab, icnt);
  return cudaGetLastError();
}

cudaError_t launch_fs3_pair(const Fs3PairBufs &B, const int *icnt, const double4 *comb,
                            const double4 *s17, const double *coef, const double *bgr, Fs3Params P,
                            int nm, int ns, double *f, double *fc3, double *scal, void *tri,
                            int tri_cap, int nsm, double *gfs3, cudaStream_t st) {
  cudaError_t e =
      gfs3 ? launch_pair_t<true>(B, icnt, s17, coef, bgr, nm, ns, f, nsm, gfs3, st)
           : launch_pair_t<false>(B, icnt, s17, coef, bgr, nm, ns, f, nsm, nullptr, st);
  if (e != cudaSuccess) return e;
  // one wave of blocks, each taking its share of the triples
  const size_t smem = sizeof(double) * 2 * kNt * kNt * kNt * kCs;
  e = cudaFuncSetAttribute(k_fs3_energy, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  k_fs3_energy<<<nsm * CCP_FS3_ENERGY_BLOCKS, kET, smem, st>>>(
      comb, static_cast<const Triple *>(tri), tri_cap, B.tab, coef, B.vpart, B.pair_cap, P, nm, fc3,
      scal, const_cast<int *>(icnt));
  return cudaGetLastError();
}
