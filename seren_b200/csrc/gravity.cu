// gravity.cu - Barnes-Hut gravity walk with the geometric MAC, quadrupole
// cell terms and the kernel-softened grad-h near field; direct sink gravity.
//
// Two arithmetic forms share one walk:
//  * FP64: the reference's cell and pair terms (BHtree/BHgrav_accel.F90:146-226,
//    gravity/gravity_gradh.F90:57-86) in FP64, with FMA and one reciprocal square
//    root per term.
//  * mixed: the walk, the MAC test (drsqd > dminsqd) and the separations stay
//    FP64, so exactly the same cells are accepted and the same pairs visited;
//    the separation is then cast to FP32 and the cell/pair term evaluated in
//    FP32, with the M4 softening kernel evaluated at the reference's table bin;
//    terms are summed in FP32 with Kahan compensation and added to the FP64
//    result once.
#include <algorithm>
#include <type_traits>

#include "ctx.cuh"
#include "warp.cuh"

namespace seren {

namespace {

struct GravTree {
  const int4* link;
  const double4* gA;   // COM, m
  const double4* gB;   // q1..q4
  const double2* gC;   // q5, dminsqd
  const int* nkids;    // children per cell
  int ctot;
};

// ---------------------------------------------------------------------------
// FP64 terms
// BHgrav_accel.F90:159-189 (1/r once and FMA, as the mixed form below), d = r_p -
// r_c; q5z = (q5, -(q1 + q3))
__device__ __forceinline__ void cell_term64(double d0, double d1, double d2, double m,
                                            const double4& q, const double2& q5z, double& ax,
                                            double& ay, double& az, double& pot) {
  const double inv = rsqrt(fma(d2, d2, fma(d1, d1, fma(d0, d0, SMALL_NUMBER))));
  const double inv2 = inv * inv;
  const double n0 = d0 * inv, n1 = d1 * inv, n2 = d2 * inv;
  const double qx = fma(q.w, n2, fma(q.y, n1, q.x * n0));
  const double qy = fma(q5z.x, n2, fma(q.z, n1, q.y * n0));
  const double qz = fma(q5z.y, n2, fma(q5z.x, n1, q.w * n0));
  const double nqn = fma(qz, n2, fma(qy, n1, qx * n0)) * inv2;
  const double g = fma(-2.5, nqn, -m);
  ax = fma(inv2, fma(g, n0, qx * inv2), ax);
  ay = fma(inv2, fma(g, n1, qy * inv2), ay);
  az = fma(inv2, fma(g, n2, qz * inv2), az);
  pot = fma(inv, fma(0.5, nqn, m), pot);
}

// gravity/gravity_gradh.F90:11-95, d = r_q - r_p, zz = zeta/h^2 of each side, mh
// = m_q/2.  r = sqrt(r^2) + SMALL_NUMBER and 1/r come from one rsqrt: the root
// corrected by its residual (one Newton step), the SMALL_NUMBER to first order (below 1e-12,
// where that would not do, from the reference's own expressions).
__device__ __forceinline__ void pair_term64(double d0, double d1, double d2, double ihp,
                                            double zzp, double mh, double hq, double ihq,
                                            double zzq, const double4* __restrict__ tabG,
                                            double& ax, double& ay, double& az, double& pot) {
  const double r2 = fma(d2, d2, fma(d1, d1, d0 * d0));
  double r, inv;
  if (r2 > 1.0e-24) {
    const double y = rsqrt(r2);
    const double x = r2 * y;
    r = fma(0.5 * y, fma(-x, x, r2), x) + SMALL_NUMBER;
    inv = fma(-(SMALL_NUMBER * y), y, y);
  } else {
    r = sqrt(r2) + SMALL_NUMBER;
    inv = 1.0 / r;
  }
  double grav = inv * inv, dpot = inv;
  const double inv2 = grav;
  if (inv > INVKERNRANGE * ihp) {
    const double4 w = tabG[min((int)((HALFKERNTOT * r) * ihp), KERNTOT)];
    grav = (ihp * ihp) * fma(zzp, w.y, w.x);
    dpot = ihp * w.z;
  }
  if (r < KERNRANGE * hq) {
    const double4 w = tabG[min((int)((HALFKERNTOT * r) * ihq), KERNTOT)];
    grav = fma(ihq * ihq, fma(zzq, w.y, w.x), grav);
    dpot = fma(ihq, w.z, dpot);
  } else {
    grav = grav + inv2;
    dpot = dpot + inv;
  }
  const double f = (mh * inv) * grav;
  ax = fma(f, d0, ax);
  ay = fma(f, d1, ay);
  az = fma(f, d2, az);
  pot = fma(mh, dpot, pot);
}

// gravity/gravity_meanh.F90:12-69
__device__ __forceinline__ void meanh_term64(double d0, double d1, double d2, double hmean, double mq,
                                             const double4* __restrict__ tabG, double& ax,
                                             double& ay, double& az, double& pot) {
  const double drsqd = (d0 * d0 + d1 * d1) + d2 * d2;
  const double drmag = sqrt(drsqd) + SMALL_NUMBER;
  const double invdrmag = 1.0 / drmag;
  double grav, dpot;
  if (drmag < KERNRANGE * hmean) {
    const double invhmean = 1.0 / hmean;
    int kern = (int)((HALFKERNTOT * drmag) * invhmean);
    kern = min(kern, KERNTOT);
    const double4 w = tabG[kern];
    grav = ((invdrmag * invhmean) * invhmean) * w.x;
    dpot = invhmean * w.z;
  } else {
    grav = invdrmag * (invdrmag * invdrmag);
    dpot = invdrmag;
  }
  const double f = mq * grav;
  ax = ax + f * d0; ay = ay + f * d1; az = az + f * d2;
  pot = pot + mq * dpot;
}

// ---------------------------------------------------------------------------
// FP32 terms (mixed form)
struct Kahan4 {
  float s[4] = {0.f, 0.f, 0.f, 0.f};
  float c[4] = {0.f, 0.f, 0.f, 0.f};
  __device__ __forceinline__ void add(int k, float x) {
    const float y = x - c[k];
    const float t = s[k] + y;
    c[k] = (t - s[k]) - y;
    s[k] = t;
  }
  __device__ __forceinline__ double get(int k) const { return (double)s[k] - (double)c[k]; }
};

__device__ __forceinline__ void count_add(unsigned long long* counts, unsigned long long ncell,
                                          unsigned long long npair) {
  // warp-aggregated interaction counters
  for (int o = 16; o > 0; o >>= 1) {
    ncell += __shfl_down_sync(0xffffffffu, ncell, o);
    npair += __shfl_down_sync(0xffffffffu, npair, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(counts + 0, ncell);
    atomicAdd(counts + 1, npair);
  }
}

// ---------------------------------------------------------------------------
// Frontier walk.  One warp walks the tree for 32 consecutive active particles
// (tree order: spatially adjacent) with the reference's per-particle decisions
// intact.  The walk state is a per-warp stack of entries (cell, mask): the
// cell, and the lanes whose walk reaches it (every ancestor was opened for
// them).  Each step pops up to 32 entries; the lanes load those cells in
// parallel, then every lane runs the reference's MAC test drsqd > dminsqd for
// its own particle against each popped cell in its mask.  That test runs first
// in FP32 on root-relative coordinates against a bracket [lo, hi] around
// dminsqd that covers the FP32 rounding; inside the bracket it is redone in
// FP64 exactly as BHgrav_accel.F90:146-155 does, so every decision equals the
// FP64 one.  Accepted cells go to a cell list with the mask of lanes that took
// them; opened leaves put their particles on a near-field list
// (BHgrav_accel.F90:128-136, :242-253); opened branch cells push their children
// with the mask of lanes that opened them.  Each cell is reached at most once
// per group, so a group processes at most ctot+1 entries.  Full lists are
// flushed by all lanes together (lane-parallel record preparation, then
// broadcast loads and a per-lane predicate).
constexpr int GW_THREADS = 128;
constexpr int GW_WARPS = GW_THREADS / 32;
constexpr int GW_STACK = 8192;   // frontier entries per warp (at most ctot+1 are ever live)
constexpr unsigned FULLMASK = 0xffffffffu;

// Near-field record of a particle in the mixed form (k_grav_prep): position,
// m/2, 1/h and zeta/h^2/pi (w4 without its 1/pi), 48 bytes.
struct __align__(16) GravRec {
  double x, y, z;
  float mh, ih, zz, pad0, pad1, pad2;
};

__global__ void k_grav_prep(int n, const double4* __restrict__ pm, const double2* __restrict__ hz,
                            GravRec* __restrict__ prec) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const double4 P = pm[p];
  const double2 H = hz[p];
  const double ih = 1.0 / H.x;
  prec[p] = GravRec{P.x, P.y, P.z, (float)(0.5 * P.w), (float)ih,
                    (float)(((H.y * ih) * ih) * INVPI), 0.0f, 0.0f, 0.0f};
}

struct GravWalk {
  // two float4 per cell: (FP32 COM relative to the root centre, hi bracket),
  // (lo bracket, first particle of a leaf / first child of a branch, leaf
  // count / -children, 0) as int bits
  const float4* wN;
  const double4* gA;
  const double4* gB;
  const double2* gC;
  int ctot;
  int scap;             // stack entries per warp
  double rootx, rooty, rootz;
  int root;             // root cell of the walks
  const CloudInfo* cl;  // a forest of ncl trees (NULL: one tree)
  int ncl;
};

// gravity_gradh.F90:57-86 in FP32 for one pair, d = r_q - r_p: each side's
// softened-gravity functions w5, w4, w6 (setup/kernel.F90:80-81, :99-102) at the
// centre of the reference's table bin int(5000 r/h), evaluated in place with
// the p side in the low half and the q side in the high half.  Inside h the
// reference's polynomials; between h and 2h, with u = 2 - s, the same functions
// as the mass outside s: w5 = (1 - T)/s^2 and w6 = (1 - T)/s + u^4 (1/2 - u/5),
// T = u^4 (1 - 4u/5 + u^2/6), which have no cancellation (the reference's
// expansion in s loses a factor 40 near s = 2).  ih = (1/h_p, 1/h_q), zz =
// zeta/h^2/pi of each side (w4 without its 1/pi), mh = m_q/2.
__device__ __forceinline__ void pair32(float d0, float d1, float d2, f2 ih, f2 zz, float mh,
                                       float& ax, float& ay, float& az, float& ap) {
  const float r2 = fmaxf(fmaf(d2, d2, fmaf(d1, d1, d0 * d0)), 1.0e-30f);
  const float inv = rsqrt_n(r2);
  const float inv2 = inv * inv;
  const f2 x = mul2(pk1(r2 * inv), ih);
  // floor(5000 x) by rounding towards minus infinity at 2^23
  const f2 kf = add2(fma2_rm(x, pk1(5000.0f), pk1(8388608.0f)), pk1(-8388608.0f));
  const f2 s = fma2(kf, pk1(2.0e-4f), pk1(1.0e-4f));
  const f2 s2 = mul2(s, s);
  const f2 w5i = mul2(s, fma2(s2, fma2(s, pk1(0.5f), pk1(-1.2f)), pk1(4.0f / 3.0f)));
  const f2 w6i = fma2(s2, fma2(s2, fma2(s, pk1(-0.1f), pk1(0.3f)), pk1(-2.0f / 3.0f)), pk1(1.4f));
  const f2 w4i = mul2(s, fma2(s, pk1(2.25f), pk1(-3.0f)));
  const f2 u = fma2(s, pk1(-1.0f), pk1(2.0f));
  const f2 u2 = mul2(u, u);
  const f2 u4 = mul2(u2, u2);
  const f2 nT = mul2(u4, fma2(u, fma2(u, pk1(-1.0f / 6.0f), pk1(0.8f)), pk1(-1.0f)));
  float sl, sh;
  unpk(s, sl, sh);
  const f2 is = pk(rcp_n(sl), rcp_n(sh));
  const f2 mi = fma2(nT, is, is);                        // (1 - T)/s
  const f2 w5o = mul2(mi, is);
  const f2 w6o = fma2(u4, fma2(u, pk1(-0.2f), pk1(0.5f)), mi);
  const f2 w4o = mul2(u2, pk1(-0.75f));
  float i5l, i5h, i6l, i6h, i4l, i4h, o5l, o5h, o6l, o6h, o4l, o4h, xl, xh;
  unpk(w5i, i5l, i5h); unpk(w6i, i6l, i6h); unpk(w4i, i4l, i4h);
  unpk(w5o, o5l, o5h); unpk(w6o, o6l, o6h); unpk(w4o, o4l, o4h);
  unpk(x, xl, xh);
  const bool il = sl < 1.0f, ihi = sh < 1.0f;            // bin below KERNTOT/2
  const f2 w5 = pk(il ? i5l : o5l, ihi ? i5h : o5h);
  const f2 w6 = pk(il ? i6l : o6l, ihi ? i6h : o6h);
  const f2 w4 = pk(il ? i4l : o4l, ihi ? i4h : o4h);
  const f2 g = mul2(mul2(ih, ih), fma2(zz, w4, w5));
  const f2 ph = mul2(ih, w6);
  float gl, gh, pl, phh;
  unpk(g, gl, gh);
  unpk(ph, pl, phh);
  const bool nl = xl < KERNRANGE, nh = xh < KERNRANGE;
  const float grav = (nl ? gl : inv2) + (nh ? gh : inv2);
  const float dpot = (nl ? pl : inv) + (nh ? phh : inv);
  const float f = mh * inv * grav;
  ax = fmaf(f, d0, ax);
  ay = fmaf(f, d1, ay);
  az = fmaf(f, d2, az);
  ap = fmaf(mh, dpot, ap);
}

// BHgrav_accel.F90:159-189 in FP32 for two cells at once (one per half), d =
// r_p - r_c, on: which of the two the lane takes; nm = -m, q holds q1..q5 and qz =
// -(q1 + q3).  Written with the unit vector n = d/r so that no power of 1/r above
// the second is formed: with Qn = Q.n and nQn = n.Q.n,
//   a = (1/r^2) [ n (-m - 2.5 nQn/r^2) + Qn/r^2 ],  phi = (1/r) (m + nQn/(2 r^2)),
// the reference's -m dr/r^3 + (Q.dr)/r^5 - 2.5 (dr.Q.dr) dr/r^7 and
// m/r + (dr.Q.dr)/(2 r^5).  |Q|/r^2 is of order m theta^2 for an accepted cell,
// so every FP32 intermediate stays in range however small the cell and its
// distance (1/r^7 alone overflows FP32 below r ~ 4e-6).  A cell the lane does
// not take gets 1/r = 0, so its terms vanish.  np accumulates -phi.
struct Cell2 {
  float4 a;   // x0 x1 y0 y1: r_ref - COM of the two cells
  float4 b;   // z0 z1, -m0 -m1
  float4 c;   // q1 q1, q2 q2
  float4 d;   // q3 q3, q4 q4
  float4 e;   // q5 q5, qz qz
};

__device__ __forceinline__ void cell32x2(f2 d0, f2 d1, f2 d2, bool on0, bool on1, f2 nm,
                                         const float4& qc, const float4& qd, const float4& qe,
                                         f2& ax, f2& ay, f2& az, f2& np) {
  const f2 q1 = pk(qc.x, qc.y), q2 = pk(qc.z, qc.w), q3 = pk(qd.x, qd.y), q4 = pk(qd.z, qd.w),
           q5 = pk(qe.x, qe.y), qz = pk(qe.z, qe.w);
  // the 1.2e-37 keeps the argument of rsqrt normal; it is lost in any
  // separation above 1e-15
  const f2 r2 = fma2(d2, d2, fma2(d1, d1, fma2(d0, d0, pk1(1.2e-37f))));
  float r2l, r2h;
  unpk(r2, r2l, r2h);
  const f2 inv = pk(on0 ? rsqrt_n(r2l) : 0.0f, on1 ? rsqrt_n(r2h) : 0.0f);
  const f2 inv2 = mul2(inv, inv);
  const f2 n0 = mul2(d0, inv), n1 = mul2(d1, inv), n2 = mul2(d2, inv);
  const f2 qx = fma2(q4, n2, fma2(q2, n1, mul2(q1, n0)));
  const f2 qy = fma2(q5, n2, fma2(q3, n1, mul2(q2, n0)));
  const f2 qw = fma2(qz, n2, fma2(q5, n1, mul2(q4, n0)));
  const f2 nqn = mul2(fma2(qw, n2, fma2(qy, n1, mul2(qx, n0))), inv2);
  const f2 g = fma2(pk1(-2.5f), nqn, nm);
  ax = fma2(inv2, fma2(g, n0, mul2(qx, inv2)), ax);
  ay = fma2(inv2, fma2(g, n1, mul2(qy, inv2)), ay);
  az = fma2(inv2, fma2(g, n2, mul2(qw, inv2)), az);
  np = fma2(inv, fma2(pk1(-0.5f), nqn, nm), np);
}

// Per-warp shared state: the interaction lists, and one area that holds, in
// turn, the popped cells of a walk step, the prepared cell records of a flush
// and the prepared near-field items of a flush.
// CAPV: accepted-cell entries per list (the cell-list tile; a tuning knob of
// the mixed-precision kernel, 64 for the FP64 one).
constexpr int GW_LLIST = 128;   // opened leaves per list
template <bool MIXED>
struct GwItems;
template <>
struct GwItems<true> {
  static constexpr int B = 128;    // near-field items per batch
  static constexpr int LS = B + 4; // list stride: an odd number of words
  float4 a[B];                     // r_q - r_ref, m/2
  float2 b[B];                     // 1/h, zeta/h^2/pi
  int id[B];
  union {
    unsigned mask[B];              // lanes that opened the item's leaf
    unsigned char pick[32 * LS];   // each particle's items
  };
};
template <>
struct GwItems<false> {
  static constexpr int B = 96;
  static constexpr int LS = B + 4;
  double4 a[B];                    // r_q, m
  double h[B], ih[B], z[B];
  int id[B];
  union {
    unsigned mask[B];
    unsigned char pick[32 * LS];
  };
};
template <bool MIXED, int CAPV>
struct GwCells;
template <int CAPV>
struct GwCells<true, CAPV> {
  Cell2 rec[CAPV / 2];
};
template <int CAPV>
struct GwCells<false, CAPV> {
  double4 a[CAPV];                 // COM, m
  double4 q[CAPV];                 // q1..q4
  double2 q5[CAPV];                // q5, -(q1 + q3)
};
struct __align__(16) GwPop {       // the popped cells the group test leaves undecided, packed
  float x[32], y[32], z[32];       // FP32 COM relative to the root centre
  float lo[32], hi[32];            // MAC bracket
  unsigned test[32];               // lanes that test the cell
  int cell[32];
};
template <bool MIXED, int CAPV>
struct GwRec {
  using R = typename std::conditional<MIXED, float, double>::type;
  union {
    GwItems<MIXED> it;
    GwCells<MIXED, CAPV> c;
    GwPop f;
  };
  int cid[CAPV];
  unsigned cmask[CAPV];
  int lcode[GW_LLIST];             // opened leaves: first particle * 8 + count - 1
  unsigned lmask[GW_LLIST];
  R gx[32], gy[32], gz[32], gih[32], gzz[32];   // the group's particles: position, 1/h, zeta
  int gp[32];
  int cnt[32];                     // items of each particle in the batch
  double ref[3];                   // the group's reference point
  R part[32][4];                   // near-field sums of a batch
};

__device__ __forceinline__ int warp_incl(int v, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(FULLMASK, v, o);
    if (lane >= o) v += y;
  }
  return v;
}

// A warp takes a group of PW = 2^lpw particles (32, 16, 8 or 4), 32/PW lanes each:
// lane l has particle l % PW and, in the cell lists, every (32/PW)-th pair of
// entries.  groups (a forest): offset/4 and lpw of each group; else the groups
// follow one another in the active list.
//
// Bound by issue slots (the tree and the particles stay in L2).  On a 1M-particle
// core, mixed, B200: 4.75 ms (6.08 ms with one cell entry per step, one item of
// the near field per step for all lanes, and the softening kernel gathered from
// its table); of it the walk 1.0, cell records and terms 1.8, near field 2.0.
// FP64, same core: 8.4-9.0 ms (13.1 ms with the reference's divisions and roots and
// one item per step).  Four blocks per SM at 128 registers: five at 96 spill the
// pair term's constants (5.3 ms).  Splitting the pairs inside 2h from those
// beyond, to skip the softening kernel for the latter, cost more than it saved
// (5.7 ms).
template <bool MIXED, int CAPV>
__global__ void __launch_bounds__(GW_THREADS, 4)
k_grav_walk(int nact, const int* __restrict__ act, int ngroups, const int* __restrict__ groups,
            int lpw, const double4* __restrict__ pm,
            const double2* __restrict__ hz, const GravRec* __restrict__ prec, GravWalk t,
            const double4* __restrict__ tabG, double* __restrict__ acc,
            double* __restrict__ gpot, const double* abase, double* amap, double* __restrict__ gmap,
            int nsink, const double* __restrict__ sinks,
            int2* __restrict__ stacks, int* work, DevError* err, unsigned long long* counts) {
  constexpr int CAP = CAPV;
  using Items = GwItems<MIXED>;
  using Rec = GwRec<MIXED, CAPV>;
  extern __shared__ __align__(32) unsigned char gw_smem[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  Rec& R = reinterpret_cast<Rec*>(gw_smem)[w];
  int2* const S = stacks + (size_t)(blockIdx.x * GW_WARPS + w) * t.scap;
  const unsigned lt = (1u << lane) - 1u, lbit = 1u << lane;
  unsigned long long ncell = 0, npair = 0, nent = 0;
  unsigned ce_all = 0, ce_full = 0, pi_all = 0, pi_full = 0;   // list fill statistics

  while (true) {
    int g = 0;
    if (lane == 0) g = atomicAdd(work, 1);
    g = __shfl_sync(FULLMASK, g, 0);
    if (g >= ngroups) break;
    int i0 = g << lpw;
    if (groups) {
      const int code = groups[g];
      i0 = (code >> 3) * 4;
      lpw = code & 7;
    }
    const int PW = 1 << lpw, SUB = 32 >> lpw;
    const int pl = lane & (PW - 1), sub = lane >> lpw;
    const unsigned PMASK = FULLMASK >> (32 - PW);
    const int i = i0 + pl;
    // act[i] < 0 pads a cloud's last group in a forest; dead lanes take lane
    // 0's particle (always live)
    int p = i < nact ? (act ? act[i] : i) : -1;
    const bool live = p >= 0;
    const int p0 = __shfl_sync(FULLMASK, p, 0);        // every lane takes part
    p = live ? p : p0;
    // the lanes' tree (a forest: their cloud's), as locals so that t stays a
    // kernel parameter
    int root = t.root;
    double rootx = t.rootx, rooty = t.rooty, rootz = t.rootz;
    if (t.cl) {
      const CloudInfo& C = t.cl[cloud_of(t.cl, t.ncl, p)];
      root = C.cell;
      rootx = C.root[0];
      rooty = C.root[1];
      rootz = C.root[2];
    }
    const double4 P = pm[p];
    const double hp = hz[p].x;
    // warp reference point (lane 0 is always live)
    const double rx = __shfl_sync(FULLMASK, P.x, 0);
    const double ry = __shfl_sync(FULLMASK, P.y, 0);
    const double rz = __shfl_sync(FULLMASK, P.z, 0);
    const float px32 = (float)(P.x - rootx), py32 = (float)(P.y - rooty),
                pz32 = (float)(P.z - rootz);
    const float ux = (float)(P.x - rx), uy = (float)(P.y - ry), uz = (float)(P.z - rz);
    // A separation formed in FP32 from two offsets to the reference point
    // (d = a - u) carries an error of order 2^-24 |u|, relative 2^-23 |u|/|d|;
    // the FP64 particle is used instead when some lane lies more than 64
    // smoothing lengths (the group's least) from the reference point, e.g. a
    // group that straddles a dense clump and its sparse surroundings (within
    // that bound a pair at distance h is off by less than 1e-5 relative).
    bool wide = false;
    if constexpr (MIXED) {
      float umax = live ? sqrtf(fmaf(uz, uz, fmaf(uy, uy, ux * ux))) : 0.0f;
      float hmin = live ? (float)hp : 3.0e38f;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        umax = fmaxf(umax, __shfl_xor_sync(FULLMASK, umax, o));
        hmin = fminf(hmin, __shfl_xor_sync(FULLMASK, hmin, o));
      }
      wide = umax > 64.0f * hmin;
    }
    // the group's bounding sphere in the walk's FP32 coordinates: centre the
    // middle of the live lanes' bounding box, radius the farthest live lane's
    // distance from it, rounded up
    float gx, gy, gz;
    {
      const float x0 = __shfl_sync(FULLMASK, px32, 0), y0 = __shfl_sync(FULLMASK, py32, 0),
                  z0 = __shfl_sync(FULLMASK, pz32, 0);
      float lox = live ? px32 : x0, loy = live ? py32 : y0, loz = live ? pz32 : z0;
      float hix = lox, hiy = loy, hiz = loz;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        lox = fminf(lox, __shfl_xor_sync(FULLMASK, lox, o));
        loy = fminf(loy, __shfl_xor_sync(FULLMASK, loy, o));
        loz = fminf(loz, __shfl_xor_sync(FULLMASK, loz, o));
        hix = fmaxf(hix, __shfl_xor_sync(FULLMASK, hix, o));
        hiy = fmaxf(hiy, __shfl_xor_sync(FULLMASK, hiy, o));
        hiz = fmaxf(hiz, __shfl_xor_sync(FULLMASK, hiz, o));
      }
      gx = 0.5f * (lox + hix);
      gy = 0.5f * (loy + hiy);
      gz = 0.5f * (loz + hiz);
    }
    float grad;
    {
      const float e0 = px32 - gx, e1 = py32 - gy, e2 = pz32 - gz;
      float r2 = live ? fmaf(e2, e2, fmaf(e1, e1, e0 * e0)) : 0.0f;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) r2 = fmaxf(r2, __shfl_xor_sync(FULLMASK, r2, o));
      grad = sqrtf(r2) * 1.00001f;
    }
    const float npx = -px32, npy = -py32, npz = -pz32;
    const unsigned rootmask = __ballot_sync(FULLMASK, live);
    __syncwarp();                                      // the previous group's reads are done
    if (lane < PW) {
      const double ih = 1.0 / hp, zt = hz[p].y;
      if constexpr (MIXED) {
        R.gx[lane] = ux; R.gy[lane] = uy; R.gz[lane] = uz;
        R.gih[lane] = (float)ih;
        R.gzz[lane] = (float)(((zt * ih) * ih) * INVPI);
      } else {
        R.gx[lane] = P.x; R.gy[lane] = P.y; R.gz[lane] = P.z;
        R.gih[lane] = ih;
        R.gzz[lane] = (zt * ih) * ih;
      }
      R.gp[lane] = p;
    }
    if (lane == 0) {
      R.ref[0] = rx; R.ref[1] = ry; R.ref[2] = rz;
    }
    Kahan4 kc;
    double cx = 0.0, cy = 0.0, cz = 0.0, cp = 0.0, qx = 0.0, qy = 0.0, qz = 0.0, qp = 0.0;
    int nc = 0, nl = 0;

    // The accepted cells: records prepared lane-parallel (FP64 to FP32), then
    // every lane takes two entries per step, broadcast loads, the entries not
    // in its walk with weight zero.
    auto flush_cells = [&]() {
      __syncwarp();
      for (int e = lane; e < nc; e += 32) {
        const int cid = R.cid[e];
        const double4 a = t.gA[cid];
        const double4 q = t.gB[cid];
        const double q5 = t.gC[cid].x;
        ncell += __popc(R.cmask[e] & PMASK);                 // the terms this entry gives
        if constexpr (MIXED) {
          float* c2 = reinterpret_cast<float*>(&R.c.rec[e >> 1]) + (e & 1);
          c2[0] = (float)(R.ref[0] - a.x);
          c2[2] = (float)(R.ref[1] - a.y);
          c2[4] = (float)(R.ref[2] - a.z);
          c2[6] = (float)-a.w;
          c2[8] = (float)q.x;
          c2[10] = (float)q.y;
          c2[12] = (float)q.z;
          c2[14] = (float)q.w;
          c2[16] = (float)q5;
          c2[18] = (float)(-(q.x + q.z));
        } else {
          R.c.a[e] = a;
          R.c.q[e] = q;
          R.c.q5[e] = make_double2(q5, -(q.x + q.z));
        }
      }
      if constexpr (MIXED) {
        if ((nc & 1) && lane == 0) {                         // an odd count: an entry of no lane
          float* c2 = reinterpret_cast<float*>(&R.c.rec[nc >> 1]) + 1;
#pragma unroll
          for (int k = 0; k < 20; k += 2) c2[k] = k < 6 ? 1.0f : 0.0f;
          R.cmask[nc] = 0u;
        }
      }
      __syncwarp();
      if constexpr (MIXED) {
        f2 sx = 0ull, sy = 0ull, sz = 0ull, np = 0ull;
        const int n2 = (nc + 1) >> 1;
        if (!wide) {
          const f2 ux2 = pk1(ux), uy2 = pk1(uy), uz2 = pk1(uz);
#pragma unroll 2
          for (int e = sub; e < n2; e += SUB) {
            const uint2 m = *reinterpret_cast<const uint2*>(&R.cmask[2 * e]);
            const Cell2& c = R.c.rec[e];
            const float4 a = c.a, b = c.b;
            cell32x2(add2(ux2, pk(a.x, a.y)), add2(uy2, pk(a.z, a.w)), add2(uz2, pk(b.x, b.y)),
                     m.x & lbit, m.y & lbit, pk(b.z, b.w), c.c, c.d, c.e, sx, sy, sz, np);
          }
        } else {
          const double4 P = pm[p];
          for (int e = sub; e < n2; e += SUB) {
            const uint2 m = *reinterpret_cast<const uint2*>(&R.cmask[2 * e]);
            const Cell2& c = R.c.rec[e];
            const double4 A = t.gA[R.cid[2 * e]];
            const double4 B = t.gA[R.cid[min(2 * e + 1, nc - 1)]];
            cell32x2(pk((float)(P.x - A.x), (float)(P.x - B.x)),
                     pk((float)(P.y - A.y), (float)(P.y - B.y)),
                     pk((float)(P.z - A.z), (float)(P.z - B.z)), m.x & lbit, m.y & lbit,
                     pk(c.b.z, c.b.w), c.c, c.d, c.e, sx, sy, sz, np);
          }
        }
        kc.add(0, sum2(sx)); kc.add(1, sum2(sy)); kc.add(2, sum2(sz)); kc.add(3, -sum2(np));
      } else {
        const double4 P = pm[p];
        for (int e = sub; e < nc; e += SUB) {
          if (R.cmask[e] & lbit) {
            const double4 a = R.c.a[e];
            cell_term64(P.x - a.x, P.y - a.y, P.z - a.z, a.w, R.c.q[e], R.c.q5[e], cx, cy, cz, cp);
          }
        }
      }
      nc = 0;
      __syncwarp();
    };
    // The near field of a batch of np items (R.it.id, R.it.mask; zero masks past
    // the last one, np a multiple of 32): each item's record is prepared by one
    // lane; the item-by-particle bits are transposed, so that each particle's
    // lane lists the items that particle opened; then 8 lanes share one
    // particle's list, four particles at a time.  Every lane has work whatever
    // share of the items each particle opened (a quarter of them on average).
    auto do_items = [&](int np) {
      __syncwarp();
      constexpr int NW = Items::B / 32;
      unsigned word[NW];
#pragma unroll
      for (int c = 0; c < NW; ++c) word[c] = 32 * c < np ? R.it.mask[32 * c + lane] : 0u;
      // two records in flight per lane
#pragma unroll
      for (int c0 = 0; c0 < NW; c0 += 2) {
        if (32 * c0 < np) {
          int q[2];
#pragma unroll
          for (int u = 0; u < 2; ++u)
            if (c0 + u < NW) q[u] = word[c0 + u] != 0u ? R.it.id[32 * (c0 + u) + lane] : p0;
          if constexpr (MIXED) {
            GravRec Q[2];
#pragma unroll
            for (int u = 0; u < 2; ++u)
              if (c0 + u < NW) Q[u] = prec[q[u]];
#pragma unroll
            for (int u = 0; u < 2 && c0 + u < NW; ++u) {
              const int e = 32 * (c0 + u) + lane;
              R.it.a[e] = make_float4((float)(Q[u].x - R.ref[0]), (float)(Q[u].y - R.ref[1]),
                                      (float)(Q[u].z - R.ref[2]), Q[u].mh);
              R.it.b[e] = make_float2(Q[u].ih, Q[u].zz);
            }
          } else {
            double4 Q[2];
            double2 H[2];
#pragma unroll
            for (int u = 0; u < 2 && c0 + u < NW; ++u) {
              Q[u] = pm[q[u]];
              H[u] = hz[q[u]];
            }
#pragma unroll
            for (int u = 0; u < 2 && c0 + u < NW; ++u) {
              const int e = 32 * (c0 + u) + lane;
              const double ih = 1.0 / H[u].x;
              R.it.a[e] = make_double4(Q[u].x, Q[u].y, Q[u].z, 0.5 * Q[u].w);
              R.it.h[e] = H[u].x;
              R.it.ih[e] = ih;
              R.it.z[e] = (H[u].y * ih) * ih;
            }
          }
        }
      }
#pragma unroll
      for (int c = 0; c < NW; ++c) {
        npair += __popc(word[c] & PMASK);
        if (32 * c < np) word[c] = warp_transpose(word[c], lane);
      }
      __syncwarp();                                          // the masks are read
      int n = 0;
      if (lane < PW) {
        unsigned char* row = R.it.pick + lane * Items::LS;
#pragma unroll
        for (int c = 0; c < Items::B / 32; ++c) {
          if (32 * c < np) {
            for (unsigned wd = word[c]; wd != 0u;) {
              const int b = 31 - __clz(wd);
              row[n++] = (unsigned char)(32 * c + b);
              wd ^= 1u << b;
            }
          }
        }
        R.cnt[lane] = n;
      }
      __syncwarp();
#pragma unroll 1
      for (int j0 = 0; j0 < PW; j0 += 4) {
        const int j = j0 + (lane >> 3);
        const int cnt = R.cnt[j];
        unsigned char* row = R.it.pick + j * Items::LS;
        const int pj = R.gp[j];
        typename Rec::R sx = 0, sy = 0, sz = 0, sp = 0;
        const typename Rec::R ihp = R.gih[j], zzp = R.gzz[j];
        if constexpr (MIXED) {
          if (!wide) {
            const float xj = R.gx[j], yj = R.gy[j], zj = R.gz[j];
#pragma unroll 2
            for (int k = lane & 7; k < cnt; k += 8) {
              const int e = row[k];
              const float4 a = R.it.a[e];
              const float2 b = R.it.b[e];
              const float mh = R.it.id[e] != pj ? a.w : 0.0f;   // not the particle itself
              pair32(a.x - xj, a.y - yj, a.z - zj, pk(ihp, b.x), pk(zzp, b.y), mh, sx, sy, sz, sp);
            }
          } else {
            const double4 Pj = pm[pj];
            for (int k = lane & 7; k < cnt; k += 8) {
              const int e = row[k];
              const int q = R.it.id[e];
              const double4 Q = pm[q];
              const float2 b = R.it.b[e];
              pair32((float)(Q.x - Pj.x), (float)(Q.y - Pj.y), (float)(Q.z - Pj.z), pk(ihp, b.x),
                     pk(zzp, b.y), q != pj ? R.it.a[e].w : 0.0f, sx, sy, sz, sp);
            }
          }
        } else {
          const double xj = R.gx[j], yj = R.gy[j], zj = R.gz[j];
          for (int k = lane & 7; k < cnt; k += 8) {
            const int e = row[k];
            const double4 a = R.it.a[e];
            if (R.it.id[e] != pj)
              pair_term64(a.x - xj, a.y - yj, a.z - zj, ihp, zzp, a.w, R.it.h[e], R.it.ih[e],
                          R.it.z[e], tabG, sx, sy, sz, sp);
          }
        }
        __syncwarp();
        const typename Rec::R v = sum4_by8(sx, sy, sz, sp, lane);
        if ((lane & 1) == 0) R.part[j][(lane & 7) >> 1] = v;
      }
      __syncwarp();
      if (live && lane < PW) {
        if constexpr (MIXED) {
          kc.add(0, R.part[lane][0]); kc.add(1, R.part[lane][1]);
          kc.add(2, R.part[lane][2]); kc.add(3, R.part[lane][3]);
        } else {
          qx += R.part[lane][0]; qy += R.part[lane][1];
          qz += R.part[lane][2]; qp += R.part[lane][3];
        }
      }
      __syncwarp();
    };
    // The opened leaves' particles, expanded 32 leaves at a time into batches
    // of items
    auto flush_leaves = [&]() {
      int nb = 0, l0 = 0, done = 0;
      while (true) {
        __syncwarp();
        int code = 0, cnt = 0;
        unsigned m = 0u;
        if (l0 + lane < nl) {
          code = R.lcode[l0 + lane];
          m = R.lmask[l0 + lane];
          cnt = (code & 7) + 1;
        }
        const int inc = warp_incl(cnt, lane);
        // the lanes whose particles fit into what is left of the batch; those
        // before them (done particles) are in earlier batches
        const unsigned fit = __ballot_sync(FULLMASK, inc > done && inc - done <= Items::B - nb);
        const int upto = fit ? __shfl_sync(FULLMASK, inc, 31 - __clz(fit)) : done;
        if ((fit >> lane) & 1u) {
          const int o = nb + inc - done - cnt;
          for (int q = 0; q < cnt; ++q) {
            R.it.id[o + q] = (code >> 3) + q;
            R.it.mask[o + q] = m;
          }
        }
        nb += upto - done;
        done = upto;
        const bool all = done == __shfl_sync(FULLMASK, inc, 31);   // these 32 leaves are in
        if (all) {
          l0 += 32;
          done = 0;
        }
        const bool last = l0 >= nl;
        if (!all || last) {                                  // the batch is full, or the list done
          const int np = (nb + 31) & ~31;
          if (nb + lane < np) R.it.mask[nb + lane] = 0u;
          do_items(np);
          nb = 0;
          if (last) break;
        }
      }
      nl = 0;
      __syncwarp();
    };

    if (lane == 0) S[0] = make_int2(root, (int)rootmask);
    int sp = 1;
    long long gent = 0;
    bool over = false;
    while (true) {
      __syncwarp();
      const int k = min(32, sp);
      sp -= k;
      gent += k;
      int cc = 0, cnt = 0, base = 0;     // cnt: leaf particles, or -children of a branch
      unsigned m = 0;
      // group test of the popped cell: 1 when every lane's FP32 prefilter
      // would pass it (d2s > hi: nearest possible lane beyond the bracket),
      // 2 when none would reach the bracket (d2s < lo for the farthest
      // possible lane, or a one-particle leaf, which has no MAC test), 0 when
      // each lane tests it; margins of 1e-5 cover every FP32 rounding, so the
      // decisions are the per-lane ones
      int dec = 2;
      float4 na, nb2;
      if (lane < k) {
        const int2 ent = S[sp + lane];
        cc = ent.x;
        m = (unsigned)ent.y;
        na = t.wN[2 * cc];
        nb2 = t.wN[2 * cc + 1];
        cnt = __float_as_int(nb2.z);
        base = __float_as_int(nb2.y);
        if (cnt != 1) {
          const float e0 = gx - na.x, e1 = gy - na.y, e2 = gz - na.z;
          const float D = sqrtf(fmaf(e2, e2, fmaf(e1, e1, e0 * e0)));
          const float dn = fmaf(D, 0.99999f, -grad);      // at most the nearest lane's distance
          const float df = fmaf(D, 1.00001f, grad);       // at least the farthest lane's
          if (dn > 0.0f && (dn * dn) * 0.99999f > na.w) dec = 1;
          else if (!((df * df) * 1.00001f < nb2.x)) dec = 0;
        }
      }
      unsigned macc = dec == 1 ? m : 0u;
      const unsigned und = __ballot_sync(FULLMASK, dec == 0);
      const int ku = __popc(und);
      const int upos = __popc(und & lt);
      if (dec == 0) {
        R.f.x[upos] = na.x; R.f.y[upos] = na.y; R.f.z[upos] = na.z;
        R.f.lo[upos] = nb2.x; R.f.hi[upos] = na.w;
        R.f.test[upos] = m;
        R.f.cell[upos] = cc;
      }
      if (lane < (-ku & 3)) {                              // up to a multiple of four
        R.f.x[ku + lane] = 0.0f; R.f.y[ku + lane] = 0.0f; R.f.z[ku + lane] = 0.0f;
        R.f.lo[ku + lane] = 0.0f; R.f.hi[ku + lane] = 0.0f;
        R.f.test[ku + lane] = 0u;
      }
      __syncwarp();
      // each lane's MAC test on the undecided cells, four at a time (two per
      // packed operation); a lane inside the FP32 bracket takes the exact FP64
      // test (rare, a warp-uniform branch)
      for (int e0 = 0; e0 < ku; e0 += 4) {
        const float4 X = *reinterpret_cast<const float4*>(&R.f.x[e0]);
        const float4 Y = *reinterpret_cast<const float4*>(&R.f.y[e0]);
        const float4 Z = *reinterpret_cast<const float4*>(&R.f.z[e0]);
        const float4 lo = *reinterpret_cast<const float4*>(&R.f.lo[e0]);
        const float4 hi = *reinterpret_cast<const float4*>(&R.f.hi[e0]);
        const uint4 mt = *reinterpret_cast<const uint4*>(&R.f.test[e0]);
        const f2 ax = add2(pk(X.x, X.y), pk1(npx)), bx = add2(pk(X.z, X.w), pk1(npx));
        const f2 ay = add2(pk(Y.x, Y.y), pk1(npy)), by = add2(pk(Y.z, Y.w), pk1(npy));
        const f2 az = add2(pk(Z.x, Z.y), pk1(npz)), bz = add2(pk(Z.z, Z.w), pk1(npz));
        float d[4];
        unpk(fma2(az, az, fma2(ay, ay, mul2(ax, ax))), d[0], d[1]);
        unpk(fma2(bz, bz, fma2(by, by, mul2(bx, bx))), d[2], d[3]);
        const float lov[4] = {lo.x, lo.y, lo.z, lo.w}, hiv[4] = {hi.x, hi.y, hi.z, hi.w};
        const unsigned mv[4] = {mt.x, mt.y, mt.z, mt.w};
        unsigned amb = 0u;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const bool mine = mv[u] & lbit;
          const bool out = d[u] > hiv[u];
          const unsigned b = __ballot_sync(FULLMASK, mine && out);
          if (dec == 0 && upos == e0 + u) macc = b;
          if (mine && !out && d[u] >= lov[u]) amb |= 1u << u;
        }
        if (__any_sync(FULLMASK, amb != 0u)) {             // exact test, :146-155
#pragma unroll 1
          for (int u = 0; u < 4; ++u) {
            bool a2 = false;
            if ((amb >> u) & 1u) {
              const int ce = R.f.cell[e0 + u];
              const double4 a = t.gA[ce];
              const double4 P = pm[p];
              const double e0d = P.x - a.x, e1d = P.y - a.y, e2d = P.z - a.z;
              a2 = ((e0d * e0d + e1d * e1d) + e2d * e2d) > t.gC[ce].y;
            }
            const unsigned b = __ballot_sync(FULLMASK, a2);
            if (dec == 0 && upos == e0 + u) macc |= b;
          }
        }
      }
      const unsigned mopn = m & ~macc;
      // accepted cells
      const unsigned bc = __ballot_sync(FULLMASK, macc != 0u);
      if (macc != 0u) {
        const int o = nc + __popc(bc & lt);
        R.cid[o] = cc;
        R.cmask[o] = macc;
        ++ce_all;
        ce_full += macc == rootmask;
      }
      nc += __popc(bc);
      // opened leaves join the near-field list
      const bool lf = cnt > 0 && mopn != 0u;
      const unsigned bl = __ballot_sync(FULLMASK, lf);
      if (lf) {
        const int o = nl + __popc(bl & lt);
        R.lcode[o] = base * 8 + (cnt - 1);
        R.lmask[o] = mopn;
        pi_all += cnt;
        pi_full += mopn == rootmask ? cnt : 0;
      }
      nl += __popc(bl);
      // opened branch cells: children onto the stack
      const int nch = (cnt < 0 && mopn != 0u) ? -cnt : 0;
      const int cin = warp_incl(nch, lane);
      const int ctotal = __shfl_sync(FULLMASK, cin, 31);
      if (sp + ctotal > t.scap || gent > (long long)t.ctot + 1) {
        if (lane == 0) set_error(err, SEREN_GPU_ERR_WALK, MIXED ? KID_GRAV_MIXED : KID_GRAV, p, cc);
        over = true;
      } else {
        for (int q = 0; q < nch; ++q) S[sp + cin - nch + q] = make_int2(base + q, (int)mopn);
        sp += ctotal;
      }
      const bool last = sp == 0 || over;
      if (nc > CAP - 32 || last) flush_cells();
      if (nl > GW_LLIST - 32 || last) flush_leaves();
      if (last) break;
    }
    nent += gent;
    npair -= live && sub == 0 ? 1u : 0u;                    // the particle itself
    double ax, ay, az, pot;
    if constexpr (MIXED) {
      ax = kc.get(0); ay = kc.get(1); az = kc.get(2); pot = kc.get(3);
    } else {
      ax = cx + qx; ay = cy + qy; az = cz + qz; pot = cp + qp;
    }
    for (int o = PW; o < 32; o <<= 1) {                     // the lanes of a particle
      ax += __shfl_xor_sync(FULLMASK, ax, o);
      ay += __shfl_xor_sync(FULLMASK, ay, o);
      az += __shfl_xor_sync(FULLMASK, az, o);
      pot += __shfl_xor_sync(FULLMASK, pot, o);
    }
    if (live && sub == 0) {
      double* a = acc + (size_t)p * 3;
      // the acceleration gravity adds to: acc, or a mapped host buffer
      const double* ab = abase ? abase + (size_t)p * 3 : a;
      a[0] = ab[0] + ax;
      a[1] = ab[1] + ay;
      a[2] = ab[2] + az;
      if (nsink > 0) {                                       // sinks/direct_sink_gravity.F90
        const double4 P = pm[p];
        const double hp = hz[p].x;
        double sx = 0.0, sy = 0.0, sz = 0.0, sp2 = 0.0;
        for (int s = 0; s < nsink; ++s) {
          const double* sr = sinks + s * 5;
          meanh_term64(sr[0] - P.x, sr[1] - P.y, sr[2] - P.z, 0.5 * (hp + sr[4]), sr[3], tabG,
                       sx, sy, sz, sp2);
        }
        a[0] = a[0] + sx;
        a[1] = a[1] + sy;
        a[2] = a[2] + sz;
        pot = pot + sp2;
      }
      gpot[p] = pot;
      // host buffers mapped into the device address space: the results
      // cross PCIe while the other groups still compute
      if (amap) {
        amap[(size_t)p * 3] = a[0];
        amap[(size_t)p * 3 + 1] = a[1];
        amap[(size_t)p * 3 + 2] = a[2];
      }
      if (gmap) gmap[p] = pot;
    }
  }
  count_add(counts, ncell, npair);
  count_add(counts + 9, ce_all, ce_full);
  count_add(counts + 11, pi_all, pi_full);
  if (lane == 0) atomicAdd(counts + 2, nent);
}


// sph_sim/sph_sink_forces.F90:49-110: BHgrav_accel(-s) with gravity_meanh
// near field (BHgrav_accel.F90:299-314), then the other sinks directly.  One block
// per sink walks breadth first, a thread per cell of a level (one thread alone
// took 0.35 ms a sink on a 50000-particle disc); its sums are added in a fixed order.
constexpr int SW_T = 256;
__global__ void __launch_bounds__(SW_T) k_sink_walk(
    int s0, int nsink, const double* __restrict__ sinks, const double4* __restrict__ pm,
    const double2* __restrict__ hz, GravTree t, const double4* __restrict__ tabG,
    int* __restrict__ scratch, int cap, double* __restrict__ out, DevError* err) {
  __shared__ int wsum[SW_T / 32];
  __shared__ double red[SW_T / 32][4];
  const int s = s0 + blockIdx.x;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const double* sr = sinks + s * 5;
  const double rx = sr[0], ry = sr[1], rz = sr[2];
  const double invhp = 1.0 / sr[4];
  const double hp = 1.0 / invhp;
  double cx = 0.0, cy = 0.0, cz = 0.0, cp = 0.0, px = 0.0, py = 0.0, pz = 0.0, pp = 0.0;
  int* fa = scratch + (size_t)blockIdx.x * 2 * cap;
  int* fb = fa + cap;
  if (threadIdx.x == 0) fa[0] = 0;
  __syncthreads();
  int nf = 1;
  while (nf > 0) {
    int nnext = 0;
    for (int base = 0; base < nf; base += SW_T) {
      int nk = 0, kid = 0;
      if (base + threadIdx.x < nf) {
        const int c = fa[base + threadIdx.x];
        const int4 lk = t.link[c];
        bool open = lk.x == 1;                       // a one-particle leaf has no MAC test
        if (!open) {
          const double4 a = t.gA[c];
          const double d0 = rx - a.x, d1 = ry - a.y, d2 = rz - a.z;
          const double2 cc = t.gC[c];
          open = !((d0 * d0 + d1 * d1) + d2 * d2 > cc.y);
          if (!open) {
            const double4 q = t.gB[c];
            cell_term64(d0, d1, d2, a.w, q, make_double2(cc.x, -(q.x + q.z)), cx, cy, cz, cp);
          }
        }
        if (open) {
          for (int k = 0; k < lk.x; ++k) {
            const double4 Q = pm[lk.w + k];
            meanh_term64(Q.x - rx, Q.y - ry, Q.z - rz, 0.5 * (hp + hz[lk.w + k].x), Q.w, tabG, px,
                         py, pz, pp);
          }
          if (lk.x == 0) {
            nk = t.nkids[c];
            kid = lk.z;
          }
        }
      }
      const int inc = warp_incl(nk, lane);
      if (lane == 31) wsum[w] = inc;
      __syncthreads();
      int o = nnext + inc - nk, tot = 0;
      for (int ww = 0; ww < SW_T / 32; ++ww) {
        if (ww < w) o += wsum[ww];
        tot += wsum[ww];
      }
      for (int k = 0; k < nk; ++k)
        if (o + k < cap) fb[o + k] = kid + k;
      nnext += tot;
      __syncthreads();
    }
    if (nnext > cap) {                               // (a level has at most ctot + 1 cells)
      if (threadIdx.x == 0) set_error(err, SEREN_GPU_ERR_WALK, KID_SINK, s, nnext);
      break;
    }
    int* tmp = fa;
    fa = fb;
    fb = tmp;
    nf = nnext;
  }
  double v[4] = {cx + px, cy + py, cz + pz, cp + pp};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(FULLMASK, v[k], o);
    if (lane == 0) red[w][k] = v[k];
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  double ax = 0.0, ay = 0.0, az = 0.0, pot = 0.0;
  for (int ww = 0; ww < SW_T / 32; ++ww) {
    ax += red[ww][0];
    ay += red[ww][1];
    az += red[ww][2];
    pot += red[ww][3];
  }
  double sx = 0.0, sy = 0.0, sz = 0.0, sp = 0.0;
  for (int ss = 0; ss < nsink; ++ss) {
    if (ss == s) continue;
    const double* o = sinks + ss * 5;
    meanh_term64(o[0] - rx, o[1] - ry, o[2] - rz, 0.5 * (sr[4] + o[4]), o[3], tabG, sx, sy, sz, sp);
  }
  out[s * 4 + 0] = ax + sx;
  out[s * 4 + 1] = ay + sy;
  out[s * 4 + 2] = az + sz;
  out[s * 4 + 3] = pot + sp;
}

inline int nb(long n, int t) { return (int)((n + t - 1) / t); }

GravTree grav_tree(const Ctx& c) { return GravTree{c.link, c.gA, c.gB, c.gC, c.nkids, c.info.ctot}; }

}  // namespace

// A variant of the walk (FP64; mixed with a cell-list tile of 64 or 96
// entries): its kernel, the shared memory of a block and the resident blocks
// per SM (its dynamic shared-memory limit is raised on first use per device).
struct GravVariant {
  void (*kern)(int, const int*, int, const int*, int, const double4*, const double2*,
               const GravRec*, GravWalk, const double4*, double*, double*, const double*, double*,
               double*, int, const double*, int2*, int*, DevError*, unsigned long long*);
  size_t smem;
  int bps;
};
static GravVariant grav_variant(int dev, bool mixed, int cap) {
  static int occ[16][3] = {};
  int dummy = 0;
  const int which = !mixed ? 0 : (cap > 64 ? 2 : 1);
  GravVariant v;
  if (which == 0) v = {k_grav_walk<false, 64>, sizeof(GwRec<false, 64>) * GW_WARPS, 0};
  else if (which == 1) v = {k_grav_walk<true, 64>, sizeof(GwRec<true, 64>) * GW_WARPS, 0};
  else v = {k_grav_walk<true, 96>, sizeof(GwRec<true, 96>) * GW_WARPS, 0};
  int& r = dev >= 0 && dev < 16 ? occ[dev][which] : dummy;
  if (r == 0) {
    cudaFuncSetAttribute(v.kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)v.smem);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&r, v.kern, GW_THREADS, v.smem);
    if (r < 1) r = 1;
  }
  v.bps = r;
  return v;
}

static int sm_count(const Ctx& c) {
  int nsm = 148;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, c.dev);
  return nsm;
}

int grav_walk_slots(const Ctx& c) {
  const int b = std::max(std::max(grav_variant(c.dev, true, 64).bps,
                                  grav_variant(c.dev, true, 96).bps),
                         grav_variant(c.dev, false, 64).bps);
  return sm_count(c) * b * GW_WARPS;
}

// log2 of the particles per walk group for n particles walked together.  A group
// of 32 costs the least in all, but its walk and lists are one warp's serial
// work, and few particles leave the GPU waiting for a few warps: a smaller
// group gives each particle more lanes and a shorter list.  Measured with
// groups of 32 / 16 / 8 / 4 (us): 777 particles FP64 229 / 135 / 90 / 63, 32768 FP64
// 639 / 496 / 430 / 461, 50000 mixed 559 / 344 / 385 / 485, 200003 mixed 1325 / 1327 /
// 1633 / 2273.  The width follows the number of particles walked (the active ones
// of a list), in a forest the size of the cloud, not of the forest, and not the
// precision: so a cloud has the same groups, and the same sums bit for bit, alone
// and in a forest.  A forest of many small clouds pays for that (64 clouds of 4096,
// mixed, ms: 0.77 / 0.87 / 1.13 / 1.63).
int grav_lpw(int n) { return n <= 4096 ? 2 : n <= 16384 ? 3 : n <= 65536 ? 4 : 5; }

int grav_walk_stack_cap(const Ctx& c) { return std::min(GW_STACK, c.cmax + 1); }

void launch_grav(Ctx& c, int nact, int nsink, const double* d_sinks, double* amap,
                 double* gmap, const double* abase) {
  if (nact <= 0) return;
  unsigned long long* counts = reinterpret_cast<unsigned long long*>(c.d_counts);
  const GravWalk gw{c.wA, c.gA, c.gB, c.gC, c.info.ctot, c.wstack_cap,
                    c.info.root[0], c.info.root[1], c.info.root[2], 0,
                    c.ncloud > 1 ? c.d_clouds : nullptr, c.ncloud};
  const bool mixed = c.prm.precision != 0;
  // in a forest with every particle active the groups follow the clouds, each
  // cloud's with the width it has alone (its results are the same bit for bit)
  const int* gl = c.act;
  const int* groups = nullptr;
  int lpw = grav_lpw(nact);
  int ng = nb(nact, 1 << lpw);
  if (!c.act && c.ncloud > 1) {
    gl = c.gact;
    nact = c.ngact;
    groups = c.ggrp;
    ng = c.nggrp;
  }
  // the tuning knobs: cell-list tile (mixed) and resident blocks per SM
  const GravVariant v = grav_variant(c.dev, mixed, mixed && c.tune.grav_cap > 64 ? 96 : 64);
  const int bps = c.tune.grav_bps > 0 ? std::min(v.bps, c.tune.grav_bps) : v.bps;
  const int blocks = std::min(sm_count(c) * bps, nb(ng, GW_WARPS));
  GravRec* prec = nullptr;
  if (mixed) {
    if (hydro_records(c)) return;
    prec = reinterpret_cast<GravRec*>(c.hrec);
    k_grav_prep<<<nb(c.ptot, 256), 256, 0, c.st>>>(c.ptot, c.pm, c.hz, prec);
    ++c.nlaunch;
  }
  cudaMemsetAsync(c.work, 0, sizeof(int), c.st);
  v.kern<<<blocks, GW_THREADS, v.smem, c.st>>>(nact, gl, ng, groups, lpw, c.pm, c.hz, prec, gw,
                                               c.tabG, c.acc, c.gpot, abase, amap, gmap, nsink,
                                               d_sinks, c.wstack, c.work, c.d_err, counts);
  ++c.nlaunch;
}

void launch_sink_walk(Ctx& c, int nsink, const double* d_sinks, double* d_out) {
  if (nsink <= 0) return;
  // two frontiers per sink in the walk stacks; the sinks in as many rounds as
  // frontiers of a whole level each allow
  const long room = 2l * c.wstack_slots * c.wstack_cap;
  const int cap = (int)std::min<long>(room / 2, c.info.ctot + 1);
  const int per = (int)std::min<long>(nsink, std::max(1l, room / (2l * cap)));
  for (int s0 = 0; s0 < nsink; s0 += per) {
    k_sink_walk<<<std::min(per, nsink - s0), SW_T, 0, c.st>>>(
        s0, nsink, d_sinks, c.pm, c.hz, grav_tree(c), c.tabG, reinterpret_cast<int*>(c.wstack), cap,
        d_out, c.d_err);
    ++c.nlaunch;
  }
}

}  // namespace seren
