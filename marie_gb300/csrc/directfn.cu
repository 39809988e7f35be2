// DIRECTFN weakly singular integrals on the device, FP64.
//
// The reference computes the five singular square-square integrals of
// exp(-j ko R)/R that nearby_correct.m substitutes (ST, EAc, EAo, VAc, VAo)
// by splitting each square face into two triangles and calling the DIRECTFN
// cores for constant basis functions on triangle pairs
// (src_vie/src_operators/cubatures/singular_st.m:14-17, singular_ea.m:17-28,
// singular_va.m:20-34) at Np_1D = 20 Gauss-Legendre points per dimension
// (assembly_nop.m:16):
//   coincident triangles       mexcubatures/directfn_ws_st_const.cpp:48-183
//   edge-adjacent triangles    mexcubatures/directfn_ws_ea_const.cpp:48-182
//   vertex-adjacent triangles  mexcubatures/directfn_ws_va_const.cpp:47-243
// The method (Polimeridis & Mosig, IJNME 83, 2010; Polimeridis, Vipiana,
// Mosig & Wilton, IEEE TAP 61(6), 2013) maps both triangles onto the
// equilateral triangle (eta, xi) with vertices (-1,0), (1,0), (0,sqrt 3),
// changes to polar-type relative coordinates, splits the angular ranges into
// subdomains in which the radial limit is one straight edge, and integrates
// all four dimensions with Gauss-Legendre rules.  Here the two outer
// dimensions of each subdomain (and the sub-triangle or sign branch) form one
// work item, whose inner two dimensions a few lanes sum, and a second kernel
// adds the blocks' sums of each output in a fixed order, so results repeat bit
// for bit.  The subdomain limits, the nesting of the rules and the
// MEX gateways' vertex order (the EA gateway hands the core the second
// triangle as (r4, r2, r1), directfn_ws_ea_const_mex.cpp:50; the VA gateway
// as (r4, r5, r1), directfn_ws_va_const_mex.cpp:51) are the reference's: they
// define the quadrature, and another split changes its value at Np_1D = 20 by
// up to 3e-5.
#include <algorithm>
#include <array>
#include <cmath>
#include <vector>

#include "plan.h"

namespace marie {

namespace {

constexpr double kSq3 = 1.7320508075688772935;
constexpr double kPi = 3.14159265358979323846;

// one triangle-pair call of a DIRECTFN core
struct DfnPair {
  double p[3][3], q[3][3];  // vertices in the order the core receives them
  double map[3][5];         // p(ep, xp) - q(eq, xq) per coordinate: 1, ep, xp, eq, xq
  double jac;               // (area_p / sqrt 3) * (area_q / sqrt 3), times the pairs it stands for
  double reach;             // largest distance between a vertex of P and one of Q
  int kind;                 // 0 coincident, 1 edge-adjacent, 2 vertex-adjacent
  int slot;                 // output the pair adds to
  long long first;          // its first block
};

__host__ __device__ inline long long items_of(int kind, int n) {
  const long long n2 = (long long)n * n;
  return kind == 0 ? 24 * n2 : kind == 1 ? 18 * n2 : 2 * n2;
}

// Lanes per work item: each takes a quarter of its third dimension, so that an
// item's trigonometry serves n^2/4 points and the 42400 items of the square
// pairs at order 20 still give 35 warps per SM.
constexpr int kParts = 4;
constexpr int kItemThreads = 128;
__host__ __device__ inline long long blocks_of(int kind, int n) {
  return (kParts * items_of(kind, n) + kItemThreads - 1) / kItemThreads;
}

// exp(-j ko R).  SMALL: every ko R is within the series' range
template <bool SMALL>
struct Phase {
  SmallPhase series;
  double ko;
  explicit Phase(double ko_) : series(ko_), ko(ko_) {}
  // acc += w exp(-j ko R)
  __device__ __forceinline__ void add(double R, double w, double2& acc) const {
    double sn, cs;
    if (SMALL)
      series.sincos(R, sn, cs);
    else
      sincos(ko * R, &sn, &cs);
    acc.x = fma(w, cs, acc.x);
    acc.y = fma(-w, sn, acc.y);
  }
};

// The rule on [0, 1]: nodes u, weights v, and the weights with the radial
// Jacobian's powers of u.
struct Rule {
  double u[kDirectfnMaxOrder], v[kDirectfnMaxOrder], vu2[kDirectfnMaxOrder], vu3[kDirectfnMaxOrder];
};

// Every pair's innermost dimension is a length lam = Lam u along a fixed
// direction of the four parameters, and both points are affine in those
// (set_map): the difference of the points is d0 + lam d1.  So a point of the
// innermost rule takes the difference, one reciprocal square root and the phase
// (27 FP64 instructions with the series), and everything else belongs to the
// loops around it.
template <bool SMALL>
__device__ __forceinline__ double2 ray(const Phase<SMALL>& ph, int n, const double* u, const double* wu,
                                       const double (&d0)[3], const double (&d1)[3], double Lam) {
  double2 acc = mk<double2>(0.0, 0.0);
  for (int b = 0; b < n; ++b) {
    const double lam = Lam * u[b];
    const double x = fma(lam, d1[0], d0[0]), y = fma(lam, d1[1], d0[1]), z = fma(lam, d1[2], d0[2]);
    const double R2 = fma(x, x, fma(y, y, z * z));
    const double ir = rsqrt(R2);
    ph.add(R2 * ir, wu[b] * ir, acc);
  }
  return acc;
}

// Work items: the two outer dimensions of a subdomain (and the sub-triangle or
// sign branch).  Each returns the sum over the points [a0, a1) of its third
// dimension and all of the fourth, all weights applied.

// coincident triangles; loc = ((kk * 8 + m) * n + i) * n + j: sub-triangle kk,
// subdomain m, psi_i, eta_j
template <bool SMALL>
__device__ double2 item_st(const DfnPair& t, const Phase<SMALL>& ph, int n, const Rule& r, long long loc, int a0,
                           int a1) {
  const int j = (int)(loc % n), i = (int)((loc / n) % n);
  const int m = (int)((loc / ((long long)n * n)) % 8), kk = (int)(loc / (8LL * n * n));
  // psi ranges in units of pi/3 (directfn_ws_st_const.cpp:189-229)
  const int pa = (m == 0 || m == 4 || m == 5) ? 0 : (m == 1 || m == 6) ? 1 : 2;
  const double lps = kPi / 3.0;
  const double psi = lps * (pa + r.u[i]);
  const double wps = lps * r.v[i];
  // eta ranges (:233-287)
  double eA, eB;
  switch (m) {
    case 0: case 1: eA = 0.0; eB = 1.0; break;
    case 2: case 3: {
      const double b1 = tan(kPi - psi) / kSq3, h1 = (1.0 - b1) / (1.0 + b1);
      if (m == 2) { eA = h1; eB = 1.0; } else { eA = 0.0; eB = h1; }
      break;
    }
    case 4: case 5: {
      const double b2 = tan(psi) / kSq3, h2 = -(1.0 - b2) / (1.0 + b2);
      if (m == 4) { eA = h2; eB = 0.0; } else { eA = -1.0; eB = h2; }
      break;
    }
    default: eA = -1.0; eB = 0.0;
  }
  const double eta = fma(eB - eA, r.u[j], eA);
  const double wet = (eB - eA) * r.v[j];
  double sp, cp;
  sincos(psi, &sp, &cp);
  // radial limit (:291-464): L1 for m = 0, 4; L2 for 1, 2; L3 for 3, 7; L4 for 5, 6
  double Lam;
  if (m == 0 || m == 4) Lam = (1.0 - eta) / cp;
  else if (m == 1 || m == 2) Lam = kSq3 * (1.0 - eta) / sp;
  else if (m == 3 || m == 7) Lam = -(1.0 + eta) / cp;
  else Lam = kSq3 * (1.0 + eta) / sp;
  // The points are rho apart in the direction (cp, -sp), turned with the
  // sub-triangle (:519-538), so R = rho D and neither eta nor xi matters.
  double de = cp, dx = -sp;
  if (kk == 1) {
    de = -0.5 * cp + 0.5 * kSq3 * sp;
    dx = 0.5 * kSq3 * cp + 0.5 * sp;
  } else if (kk == 2) {
    de = -0.5 * cp - 0.5 * kSq3 * sp;
    dx = -0.5 * kSq3 * cp + 0.5 * sp;
  }
  double D2 = 0.0;
  for (int c = 0; c < 3; ++c) {
    const double d = fma(t.map[c][3], de, t.map[c][4] * dx);
    D2 = fma(d, d, D2);
  }
  const double iD = rsqrt(D2), D = D2 * iD;
  // inner lambda x rho rule (:468-515): rho in [0, lambda], Jacobian rho, which
  // cancels 1/R
  double2 acc = mk<double2>(0.0, 0.0);
  for (int a = a0; a < a1; ++a) {
    const double lam = Lam * r.u[a];
    double2 s = mk<double2>(0.0, 0.0);
    for (int b = 0; b < n; ++b) ph.add(lam * D * r.u[b], r.v[b], s);
    acc = cadd(acc, cscale(s, r.v[a] * lam));
  }
  return cscale(acc, t.jac * wps * wet * sp * Lam * iD);
}

// edge-adjacent triangles; loc = ((piece * 2 + B) * n + i) * n + j: eta piece of
// a subdomain, sign branch B, theta_i, psi_j
template <bool SMALL>
__device__ double2 item_ea(const DfnPair& t, const Phase<SMALL>& ph, int n, const Rule& r, long long loc, int a0,
                           int a1) {
  const int j = (int)(loc % n), i = (int)((loc / n) % n);
  const int B = (int)((loc / ((long long)n * n)) % 2), piece = (int)(loc / (2LL * n * n));
  // pieces: subdomains 1, 2, 3 have two eta pieces each, 4, 5, 6 one
  const int m = piece < 6 ? piece / 2 : piece - 3;  // 0-based subdomain
  const int half = piece < 6 ? (piece & 1) : 0;
  // theta ranges (directfn_ws_ea_const.cpp:188-218)
  const double h2 = 0.5 * kPi, h3 = kPi / 3.0;
  const double thA = (m == 0 || m == 4) ? 0.0 : (m == 1 || m == 2) ? h3 : h2;
  const double thB = m == 0 ? h3 : (m == 1 || m == 2 || m == 4) ? h2 : kPi;
  const double th = fma(thB - thA, r.u[i], thA);
  const double wth = (thB - thA) * r.v[i];
  double st, ct;
  sincos(th, &st, &ct);
  // psi ranges (:224-260)
  const double PsA = atan(st - kSq3 * ct), PsB = atan(st + kSq3 * ct);
  double pA, pB;
  switch (m) {
    case 0: pA = 0.0; pB = PsB; break;
    case 1: pA = PsA; pB = PsB; break;
    case 2: case 3: pA = 0.0; pB = PsA; break;
    case 4: pA = PsB; pB = h2; break;
    default: pA = PsA; pB = h2;
  }
  const double psi = fma(pB - pA, r.u[j], pA);
  const double wps = (pB - pA) * r.v[j];
  double sp, cp;
  sincos(psi, &sp, &cp);
  // eta pieces and their radial limits (:266-456)
  double eA = 0.0, eB = 1.0;
  int lim;  // 1: L1, 2: L2, 3: L3
  if (m <= 1) {
    const double g = tan(psi) / (st + kSq3 * ct), hs = (1.0 - g) / (1.0 + g);
    if (half == 0) { eB = hs; lim = 3; } else { eA = hs; lim = 2; }
  } else if (m == 2) {
    const double hs = kSq3 / tan(th);
    if (half == 0) { eB = hs; lim = 3; } else { eA = hs; lim = 1; }
  } else if (m == 3) {
    lim = 1;
  } else {
    lim = 2;
  }
  // Lam = limit * (1 + eta) for L3, limit * (1 - |eta|) else
  const double limit =
      kSq3 / (lim == 3 ? cp * (st + kSq3 * ct) : lim == 2 ? sp : cp * (st - kSq3 * ct));
  const double sgn = B == 0 ? 1.0 : -1.0;
  // parameter points (:504-546): ep = sgn eta, xp = lam sp,
  // eq = sgn (lam cp ct - eta), xq = lam cp st; Jacobian lambda^2 (:462-498)
  double de[3], d1[3];
  for (int c = 0; c < 3; ++c) {
    de[c] = sgn * (t.map[c][1] - t.map[c][3]);
    d1[c] = fma(t.map[c][2], sp, cp * fma(t.map[c][3], sgn * ct, t.map[c][4] * st));
  }
  double2 acc = mk<double2>(0.0, 0.0);
  for (int a = a0; a < a1; ++a) {
    const double eta = fma(eB - eA, r.u[a], eA);
    const double Lam = limit * (lim == 3 ? 1.0 + eta : 1.0 - fabs(eta));
    double d0[3];
    for (int c = 0; c < 3; ++c) d0[c] = fma(eta, de[c], t.map[c][0]);
    acc = cadd(acc, cscale(ray(ph, n, r.u, r.vu2, d0, d1, Lam), r.v[a] * Lam * Lam * Lam));
  }
  return cscale(acc, t.jac * wth * wps * cp * (eB - eA));
}

// vertex-adjacent triangles; loc = (part * n + i) * n + j: psi part, theta_p
// index i, theta_q index j (directfn_ws_va_const.cpp:129-228)
template <bool SMALL>
__device__ double2 item_va(const DfnPair& t, const Phase<SMALL>& ph, int n, const Rule& r, long long loc, int a0,
                           int a1) {
  const int j = (int)(loc % n), i = (int)((loc / n) % n), part = (int)(loc / ((long long)n * n));
  const double h = kPi / 3.0;  // thetas in [0, pi/3]
  double stp, ctp, stq, ctq;
  sincos(h * r.u[i], &stp, &ctp);
  sincos(h * r.u[j], &stq, &ctq);
  const double Lp = 2.0 * kSq3 / (stp + kSq3 * ctp), Lq = 2.0 * kSq3 / (stq + kSq3 * ctq);
  const double split = atan(Lq / Lp);
  const double pA = part == 0 ? 0.0 : split, pB = part == 0 ? split : 0.5 * kPi;
  // parameter points (:249-266): ep = lam cp ctp - 1, xp = lam cp stp,
  // eq = lam sp ctq - 1, xq = lam sp stq; Jacobian lambda^3 sin(psi) cos(psi)
  double d0[3], dp[3], dq[3];
  for (int c = 0; c < 3; ++c) {
    d0[c] = t.map[c][0] - t.map[c][1] - t.map[c][3];
    dp[c] = fma(t.map[c][1], ctp, t.map[c][2] * stp);
    dq[c] = fma(t.map[c][3], ctq, t.map[c][4] * stq);
  }
  double2 acc = mk<double2>(0.0, 0.0);
  for (int a = a0; a < a1; ++a) {
    double sp, cp;
    sincos(fma(pB - pA, r.u[a], pA), &sp, &cp);
    const double Lam = part == 0 ? Lp / cp : Lq / sp;
    double d1[3];
    for (int c = 0; c < 3; ++c) d1[c] = fma(cp, dp[c], sp * dq[c]);
    const double L2 = Lam * Lam;
    acc = cadd(acc, cscale(ray(ph, n, r.u, r.vu3, d0, d1, Lam), r.v[a] * sp * cp * (L2 * L2)));
  }
  return cscale(acc, t.jac * (h * r.v[i]) * (h * r.v[j]) * (pB - pA));
}

__device__ __forceinline__ double2 warp_sum(double2 v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
    v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
  }
  return v;
}


// A block's lanes belong to one pair, neighbours to neighbouring items of one
// subdomain; one partial sum per block.  The FP64 pipe is the limit.  Measured on
// GB300 for the 18 pairs of order 20: 0.86 ms, where a
// warp per item, with every point from its four parameters, took 2.9 ms.
template <bool SMALL>
__global__ void __launch_bounds__(kItemThreads) k_directfn_items(const DfnPair* __restrict__ pairs, int npairs,
                                                                 Phase<SMALL> ph, int n, const double* __restrict__ x,
                                                                 const double* __restrict__ w,
                                                                 double2* __restrict__ part) {
  __shared__ Rule r;
  __shared__ DfnPair t;
  __shared__ double2 ws[kItemThreads / 32];
  if (threadIdx.x == 0) {
    int k = 0;
    while (k + 1 < npairs && pairs[k + 1].first <= blockIdx.x) ++k;
    t = pairs[k];
  }
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double u = 0.5 * x[i] + 0.5, v = 0.5 * w[i];
    r.u[i] = u;
    r.v[i] = v;
    r.vu2[i] = v * u * u;
    r.vu3[i] = v * u * u * u;
  }
  __syncthreads();
  const long long items = items_of(t.kind, n), g = (blockIdx.x - t.first) * (long long)blockDim.x + threadIdx.x;
  double2 v = mk<double2>(0.0, 0.0);
  if (g < kParts * items) {
    const int q = (int)(g / items);
    const long long loc = g - q * items;
    const int a0 = q * n / kParts, a1 = (q + 1) * n / kParts;
    if (t.kind == 0) v = item_st(t, ph, n, r, loc, a0, a1);
    else if (t.kind == 1) v = item_ea(t, ph, n, r, loc, a0, a1);
    else v = item_va(t, ph, n, r, loc, a0, a1);
  }
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double2 s = ws[0];
    for (int i = 1; i < kItemThreads / 32; ++i) s = cadd(s, ws[i]);
    part[blockIdx.x] = s;
  }
}

// one block per output: the blocks of every pair of that slot, fixed order
__global__ void __launch_bounds__(256) k_directfn_sum(const DfnPair* __restrict__ pairs, int npairs, int n,
                                                       const double2* __restrict__ part, double2* __restrict__ out) {
  const int slot = blockIdx.x;
  double2 acc = mk<double2>(0.0, 0.0);
  for (int k = 0; k < npairs; ++k) {
    if (pairs[k].slot != slot) continue;
    const long long f = pairs[k].first, cnt = blocks_of(pairs[k].kind, n);
    for (long long i = threadIdx.x; i < cnt; i += blockDim.x) acc = cadd(acc, part[f + i]);
  }
  acc = warp_sum(acc);
  __shared__ double2 ws[8];
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double2 s = mk<double2>(0.0, 0.0);
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) s = cadd(s, ws[i]);
    out[slot] = s;
  }
}

double tri_jac(const double v[3][3]) {
  double a[3], b[3];
  for (int c = 0; c < 3; ++c) {
    a[c] = v[1][c] - v[0][c];
    b[c] = v[2][c] - v[0][c];
  }
  const double cx = a[1] * b[2] - a[2] * b[1], cy = a[2] * b[0] - a[0] * b[2], cz = a[0] * b[1] - a[1] * b[0];
  return 0.5 * std::sqrt(cx * cx + cy * cy + cz * cz) / kSq3;
}

// r(eta, xi) = (v0 + v1)/2 + eta (v1 - v0)/2 + xi (2 v2 - v0 - v1)/(2 sqrt 3):
// the equilateral triangle's corners (-1, 0), (1, 0), (0, sqrt 3) go to v0, v1, v2
void set_map(DfnPair& t) {
  for (int c = 0; c < 3; ++c) {
    const double p0 = t.p[0][c], p1 = t.p[1][c], p2 = t.p[2][c], q0 = t.q[0][c], q1 = t.q[1][c], q2 = t.q[2][c];
    t.map[c][0] = 0.5 * ((p0 + p1) - (q0 + q1));
    t.map[c][1] = 0.5 * (p1 - p0);
    t.map[c][2] = (2.0 * p2 - p0 - p1) / (2.0 * kSq3);
    t.map[c][3] = -0.5 * (q1 - q0);
    t.map[c][4] = -(2.0 * q2 - q0 - q1) / (2.0 * kSq3);
  }
}

using Vec3 = std::array<double, 3>;

DfnPair make_pair(int kind, int slot, const Vec3& p1, const Vec3& p2, const Vec3& p3, const Vec3& q1, const Vec3& q2,
                  const Vec3& q3) {
  DfnPair t{};
  const Vec3* P[3] = {&p1, &p2, &p3};
  const Vec3* Q[3] = {&q1, &q2, &q3};
  for (int i = 0; i < 3; ++i)
    for (int c = 0; c < 3; ++c) {
      t.p[i][c] = (*P[i])[c];
      t.q[i][c] = (*Q[i])[c];
    }
  t.jac = tri_jac(t.p) * tri_jac(t.q);
  set_map(t);
  t.reach = 0;
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) {
      double d2 = 0;
      for (int c = 0; c < 3; ++c) d2 += (t.p[i][c] - t.q[j][c]) * (t.p[i][c] - t.q[j][c]);
      t.reach = std::max(t.reach, std::sqrt(d2));
    }
  t.kind = kind;
  t.slot = slot;
  return t;
}

// the MEX gateways' vertex orders (directfn_ws_{st,ea,va}_const_mex.cpp)
DfnPair gw_st(int slot, const Vec3& r1, const Vec3& r2, const Vec3& r3) {
  return make_pair(0, slot, r1, r2, r3, r1, r2, r3);
}
DfnPair gw_ea(int slot, const Vec3& r1, const Vec3& r2, const Vec3& r3, const Vec3& r4) {
  return make_pair(1, slot, r1, r2, r3, r4, r2, r1);
}
DfnPair gw_va(int slot, const Vec3& r1, const Vec3& r2, const Vec3& r3, const Vec3& r4, const Vec3& r5) {
  return make_pair(2, slot, r1, r2, r3, r4, r5, r1);
}

int run_pairs(std::vector<DfnPair>& pairs, int nslots, double ko, int n, double2* out, cudaStream_t st) {
  long long total = 0;
  for (auto& t : pairs) {
    t.first = total;
    total += blocks_of(t.kind, n);
  }
  std::vector<double> x, w;
  gauss_legendre(n, x, w);
  const size_t pb = pairs.size() * sizeof(DfnPair);
  DBuf dp, dxw, dpart, dout;
  MARIE_TRY(dp.alloc(pb, st));
  MARIE_TRY(dxw.alloc(2 * n * sizeof(double), st));
  MARIE_TRY(dpart.alloc(total * sizeof(double2), st));
  MARIE_TRY(dout.alloc(nslots * sizeof(double2), st));
  std::vector<double> xw(x);
  xw.insert(xw.end(), w.begin(), w.end());
  MARIE_CUDA_TRY(cudaMemcpyAsync(dp.p, pairs.data(), pb, cudaMemcpyHostToDevice, st));
  MARIE_CUDA_TRY(cudaMemcpyAsync(dxw.p, xw.data(), xw.size() * sizeof(double), cudaMemcpyHostToDevice, st));
  double reach = 0;
  for (const auto& t : pairs) reach = std::max(reach, t.reach);
  auto launch = [&](auto phase, auto items) {
    items<<<(unsigned)total, kItemThreads, 0, st>>>(dp.as<DfnPair>(), (int)pairs.size(), phase, n, dxw.as<double>(),
                                                    dxw.as<double>() + n, dpart.as<double2>());
  };
  if (std::fabs(ko) * reach <= kSmallPhase)
    launch(Phase<true>(ko), k_directfn_items<true>);
  else
    launch(Phase<false>(ko), k_directfn_items<false>);
  count_launch();
  MARIE_CUDA_TRY(cudaGetLastError());
  k_directfn_sum<<<nslots, 256, 0, st>>>(dp.as<DfnPair>(), (int)pairs.size(), n, dpart.as<double2>(),
                                        dout.as<double2>());
  count_launch();
  MARIE_CUDA_TRY(cudaGetLastError());
  std::vector<double2> h(nslots);
  MARIE_CUDA_TRY(cudaMemcpyAsync(h.data(), dout.p, nslots * sizeof(double2), cudaMemcpyDeviceToHost, st));
  MARIE_CUDA_TRY(cudaStreamSynchronize(st));
  for (int s = 0; s < nslots; ++s) out[s] = h[s];
  return MARIE_OK;
}

}  // namespace

bool directfn_order_ok(int n) { return n >= 1 && n <= kDirectfnMaxOrder; }

// Pairs whose quadratures are equal term by term are kept once, with their
// count in jac.  The integrand knows the vertices only through the distances
// between the points, so two pairs with the same distances between all six
// vertices are the same sum; a coincident pair is the same under a rotation of
// its vertices, which only renames its three sub-triangles.
static std::vector<DfnPair> merged(const std::vector<DfnPair>& pairs, double d) {
  auto dist2 = [](const DfnPair& t, int rot, int i, int j) {
    double r = 0;
    for (int c = 0; c < 3; ++c) {
      const double a = i < 3 ? t.p[(i + rot) % 3][c] : t.q[(i + rot) % 3][c];
      const double b = j < 3 ? t.p[(j + rot) % 3][c] : t.q[(j + rot) % 3][c];
      r += (a - b) * (a - b);
    }
    return r;
  };
  std::vector<DfnPair> out;
  for (const DfnPair& t : pairs) {
    bool found = false;
    for (DfnPair& o : out) {
      if (found || o.kind != t.kind || o.slot != t.slot) continue;
      for (int rot = 0; rot < (t.kind == 0 ? 3 : 1) && !found; ++rot) {
        bool same = true;
        for (int i = 0; i < 6; ++i)
          for (int j = 0; j < i; ++j)
            same = same && std::fabs(dist2(o, 0, i, j) - dist2(t, rot, i, j)) < 1e-12 * d * d;
        if (same) {
          o.jac += t.jac;
          found = true;
        }
      }
    }
    if (!found) out.push_back(t);
  }
  return out;
}

// The 20 triangle-pair calls of singular_st/ea/va.m for cubic voxels of edge
// d, each adding to its output slot (0 ST, 1 EAc, 2 EAo, 3 VAc, 4 VAo); 18 of
// them differ (the two halves of the ST square are mirror images).
static std::vector<DfnPair> square_pairs(double d) {
  const Vec3 r1{0, 0, 0}, r2{d, 0, 0}, r3{d, d, 0}, r4{0, d, 0};
  std::vector<DfnPair> P;
  // ST, singular_st.m:14-17
  P.push_back(gw_st(0, r1, r2, r3));
  P.push_back(gw_ea(0, r1, r3, r2, r4));
  P.push_back(gw_ea(0, r1, r3, r4, r2));
  P.push_back(gw_st(0, r1, r3, r4));
  // EAc, EAo, singular_ea.m:17-28
  const Vec3 e5{2 * d, 0, 0}, e6{2 * d, d, 0}, e5o{d, 0, d}, e6o{d, d, d};
  for (int o = 0; o < 2; ++o) {
    const Vec3& a = o ? e5o : e5;
    const Vec3& b = o ? e6o : e6;
    P.push_back(gw_ea(1 + o, r2, r3, r1, a));
    P.push_back(gw_va(1 + o, r3, r1, r2, a, b));
    P.push_back(gw_va(1 + o, r3, r4, r1, r2, a));
    P.push_back(gw_va(1 + o, r3, r4, r1, a, b));
  }
  // VAc, VAo, singular_va.m:20-34
  const Vec3 v5{2 * d, d, 0}, v6{2 * d, 2 * d, 0}, v7{d, 2 * d, 0};
  const Vec3 v5o{d, d, d}, v6o{d, 2 * d, d}, v7o{d, 2 * d, 0};
  for (int o = 0; o < 2; ++o) {
    const Vec3& a = o ? v5o : v5;
    const Vec3& b = o ? v6o : v6;
    const Vec3& c = o ? v7o : v7;
    P.push_back(gw_va(3 + o, r3, r1, r2, a, b));
    P.push_back(gw_va(3 + o, r3, r1, r2, b, c));
    P.push_back(gw_va(3 + o, r3, r4, r1, a, b));
    P.push_back(gw_va(3 + o, r3, r4, r1, b, c));
  }
  return merged(P, d);
}

int directfn_integrals(double ko, double dx, int n, double2 out[5], cudaStream_t st) {
  if (!directfn_order_ok(n)) return set_error(MARIE_EINVAL, "Np_1D must be in [1, %d]", kDirectfnMaxOrder);
  std::vector<DfnPair> P = square_pairs(dx);
  return run_pairs(P, 5, ko, n, out, st);
}

int directfn_single(char kind, const double* r, double ko, int n, double2* out, cudaStream_t st) {
  if (!directfn_order_ok(n)) return set_error(MARIE_EINVAL, "Np_1D must be in [1, %d]", kDirectfnMaxOrder);
  Vec3 v[5];
  const int nv = kind == 'S' ? 3 : kind == 'E' ? 4 : kind == 'V' ? 5 : 0;
  if (!nv) return set_error(MARIE_EINVAL, "kind must be 'S', 'E' or 'V'");
  for (int i = 0; i < nv; ++i) v[i] = Vec3{r[3 * i], r[3 * i + 1], r[3 * i + 2]};
  std::vector<DfnPair> P;
  if (kind == 'S') P.push_back(gw_st(0, v[0], v[1], v[2]));
  else if (kind == 'E') P.push_back(gw_ea(0, v[0], v[1], v[2], v[3]));
  else P.push_back(gw_va(0, v[0], v[1], v[2], v[3], v[4]));
  return run_pairs(P, 1, ko, n, out, st);
}

}  // namespace marie

using namespace marie;

extern "C" int marie_directfn(char kind, const double* vertices, double ko, int np_1d, double* out2) {
  if (!vertices || !out2) return set_error(MARIE_EINVAL, "NULL argument");
  double2 v;
  MARIE_TRY(directfn_single(kind, vertices, ko, np_1d, &v, 0));
  out2[0] = v.x;
  out2[1] = v.y;
  return MARIE_OK;
}
