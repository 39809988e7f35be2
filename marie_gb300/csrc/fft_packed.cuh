// FP32 transforms of two columns at once.
//
// sm_100 and later execute f32x2 instructions: one add, multiply or FMA on a
// pair of FP32 values per lane and issue slot.  A complex value as (re, im) can
// use them for additions only; here a value is a pair of re parts and a pair of
// im parts, of the same element in two neighbouring columns, so that every
// addition, twiddle product and FMA of a transform is packed, quarter turns are
// renamings of registers, and the two columns share twiddles and addresses.
#pragma once
#include "fft.cuh"

namespace marie {

// two FP32 values in a register pair
struct pk {
  unsigned long long v;
  pk() = default;
  __device__ __forceinline__ pk(float f) { asm("mov.b64 %0, {%1, %1};" : "=l"(v) : "f"(f)); }
  __device__ __forceinline__ pk(float a, float b) { asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b)); }
  __device__ __forceinline__ void get(float& a, float& b) const { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
};
__device__ __forceinline__ pk operator+(pk a, pk b) {
  pk r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ pk operator-(pk a, pk b) {
  pk r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ pk operator*(pk a, pk b) {
  pk r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ pk pfma(pk a, pk b, pk c) {
  pk r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ pk neg(pk a) {
  a.v ^= 0x8000000080000000ull;
  return a;
}

// a complex value in each of two columns
struct __align__(16) cpk {
  pk x, y;
};
__device__ __forceinline__ cpk cadd(cpk a, cpk b) { return cpk{a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ cpk csub(cpk a, cpk b) { return cpk{a.x - b.x, a.y - b.y}; }
__device__ __forceinline__ cpk cmul(cpk a, cpk b) { return cpk{a.x * b.x - a.y * b.y, pfma(a.x, b.y, a.y * b.x)}; }
__device__ __forceinline__ cpk cmulc(cpk a, cpk b) { return cpk{pfma(a.x, b.x, a.y * b.y), a.y * b.x - a.x * b.y}; }
__device__ __forceinline__ cpk cneg(cpk a) { return cpk{neg(a.x), neg(a.y)}; }
// a + rot90<INV>(d) (rot90: -i, INV +i); a - rot90<INV>(d) is add_rot<!INV>
template <bool INV> __device__ __forceinline__ cpk add_rot(cpk a, cpk d) {
  return INV ? cpk{a.x - d.y, a.y + d.x} : cpk{a.x + d.y, a.y - d.x};
}
// (re, im) of two columns as loaded {re0, im0, re1, im1}, and back
__device__ __forceinline__ cpk pack2(float4 v) { return cpk{pk(v.x, v.z), pk(v.y, v.w)}; }
__device__ __forceinline__ float4 unpack2(cpk a) {
  float4 v;
  a.x.get(v.x, v.z);
  a.y.get(v.y, v.w);
  return v;
}

template <int R, bool INV> struct PDFT;

template <bool INV> struct PDFT<2, INV> {
  __device__ __forceinline__ static void run(cpk* v) {
    const cpk a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
  }
};

template <bool INV> struct PDFT<4, INV> {
  __device__ __forceinline__ static void run(cpk* v) {
    const cpk t0 = cadd(v[0], v[2]), t1 = csub(v[0], v[2]);
    const cpk t2 = cadd(v[1], v[3]), d = csub(v[1], v[3]);
    v[0] = cadd(t0, t2);
    v[2] = csub(t0, t2);
    v[1] = add_rot<INV>(t1, d);
    v[3] = add_rot<!INV>(t1, d);
  }
  __device__ __forceinline__ static void run_half(cpk* v) {
    const cpk a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[2] = csub(a, b);
    v[1] = add_rot<INV>(a, b);
    v[3] = add_rot<!INV>(a, b);
  }
};

template <bool INV> struct PDFT<3, INV> {
  __device__ __forceinline__ static void run(cpk* v) {
    const pk s(0.86602540378443864676f), half(-0.5f);
    const cpk t1 = cadd(v[1], v[2]), d = csub(v[1], v[2]);
    const cpk t2 = cpk{pfma(half, t1.x, v[0].x), pfma(half, t1.y, v[0].y)};
    const cpk e = cpk{s * d.x, s * d.y};
    v[0] = cadd(v[0], t1);
    v[1] = add_rot<INV>(t2, e);
    v[2] = add_rot<!INV>(t2, e);
  }
};

template <bool INV> struct PDFT<5, INV> {
  __device__ __forceinline__ static void run(cpk* v) {
    const pk c1(0.30901699437494742410f), c2(-0.80901699437494742410f);
    const pk s1(0.95105651629515357212f), s2(0.58778525229247312917f), ns1(-0.95105651629515357212f);
    const cpk t1 = cadd(v[1], v[4]), t2 = cadd(v[2], v[3]), t3 = csub(v[1], v[4]), t4 = csub(v[2], v[3]);
    const cpk a1 = cpk{pfma(c2, t2.x, pfma(c1, t1.x, v[0].x)), pfma(c2, t2.y, pfma(c1, t1.y, v[0].y))};
    const cpk a2 = cpk{pfma(c1, t2.x, pfma(c2, t1.x, v[0].x)), pfma(c1, t2.y, pfma(c2, t1.y, v[0].y))};
    const cpk b1 = cpk{pfma(s2, t4.x, s1 * t3.x), pfma(s2, t4.y, s1 * t3.y)};
    const cpk b2 = cpk{pfma(ns1, t4.x, s2 * t3.x), pfma(ns1, t4.y, s2 * t3.y)};
    v[0] = cadd(v[0], cadd(t1, t2));
    v[1] = add_rot<INV>(a1, b1);
    v[4] = add_rot<!INV>(a1, b1);
    v[2] = add_rot<INV>(a2, b2);
    v[3] = add_rot<!INV>(a2, b2);
  }
};

template <bool INV> struct PDFT<8, INV> {
  // from the sums a and differences b of the halves
  __device__ __forceinline__ static void halves(cpk* a, const cpk* b, cpk* v) {
    const pk h(0.70710678118654752440f), nh(-0.70710678118654752440f);
    PDFT<4, INV>::run(a);
    const cpk t0 = add_rot<INV>(b[0], b[2]), t1 = add_rot<!INV>(b[0], b[2]);
    // b1 w and b3 w^3, w = (1 -+ i)/sqrt 2, without the factor 1/sqrt 2
    const pk p1 = b[1].x + b[1].y, p3 = b[3].x + b[3].y;
    cpk u, d;
    if (INV) {
      const pk m1 = b[1].x - b[1].y, m3 = b[3].x - b[3].y;
      u = cpk{m1 - p3, p1 + m3};
      d = cpk{m1 + p3, p1 - m3};
    } else {
      const pk q1 = b[1].y - b[1].x, q3 = b[3].y - b[3].x;
      u = cpk{p1 + q3, q1 - p3};
      d = cpk{p1 - q3, q1 + p3};
    }
    v[0] = a[0];
    v[2] = a[1];
    v[4] = a[2];
    v[6] = a[3];
    v[1] = cpk{pfma(h, u.x, t0.x), pfma(h, u.y, t0.y)};
    v[5] = cpk{pfma(nh, u.x, t0.x), pfma(nh, u.y, t0.y)};
    v[3] = INV ? cpk{pfma(nh, d.y, t1.x), pfma(h, d.x, t1.y)} : cpk{pfma(h, d.y, t1.x), pfma(nh, d.x, t1.y)};
    v[7] = INV ? cpk{pfma(h, d.y, t1.x), pfma(nh, d.x, t1.y)} : cpk{pfma(nh, d.y, t1.x), pfma(h, d.x, t1.y)};
  }
  __device__ __forceinline__ static void run(cpk* v) {
    cpk a[4], b[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      a[k] = cadd(v[k], v[k + 4]);
      b[k] = csub(v[k], v[k + 4]);
    }
    halves(a, b, v);
  }
  // the upper half of the inputs is zero
  __device__ __forceinline__ static void run_half(cpk* v) {
    cpk a[4], b[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) a[k] = b[k] = v[k];
    halves(a, b, v);
  }
};

template <bool INV> struct PDFT<16, INV> {
  // v * exp(-+ 2 pi i k / 16), k odd: (c, s) and its negated sine as constants
  __device__ __forceinline__ static cpk turn(cpk v, pk c, pk s, pk ns) {
    // exp(-+): (x c +- y s, y c -+ x s)
    return INV ? cpk{pfma(v.y, ns, v.x * c), pfma(v.x, s, v.y * c)} : cpk{pfma(v.y, s, v.x * c), pfma(v.x, ns, v.y * c)};
  }
  __device__ __forceinline__ static void halves(cpk* a, cpk* b, cpk* v) {
    const float C = 0.92387953251128675613f, S = 0.38268343236508977173f, H = 0.70710678118654752440f;
    const pk c(C), s(S), ns(-S), nc(-C), h(H), nh(-H);
    b[1] = turn(b[1], c, s, ns);
    b[3] = turn(b[3], s, c, nc);
    b[5] = turn(b[5], ns, c, nc);
    b[7] = turn(b[7], nc, s, ns);
    // k = 2, 6: (1 -+ i)/sqrt 2 and (-1 -+ i)/sqrt 2; k = 4: a quarter turn
    const pk p2 = b[2].x + b[2].y, p6 = b[6].x + b[6].y;
    if (INV) {
      b[2] = cpk{h * (b[2].x - b[2].y), h * p2};
      b[6] = cpk{nh * p6, h * (b[6].x - b[6].y)};
      b[4] = cpk{neg(b[4].y), b[4].x};
    } else {
      b[2] = cpk{h * p2, h * (b[2].y - b[2].x)};
      b[6] = cpk{h * (b[6].y - b[6].x), nh * p6};
      b[4] = cpk{b[4].y, neg(b[4].x)};
    }
    PDFT<8, INV>::run(a);
    PDFT<8, INV>::run(b);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      v[2 * q] = a[q];
      v[2 * q + 1] = b[q];
    }
  }
  __device__ __forceinline__ static void run(cpk* v) {
    cpk a[8], b[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      a[k] = cadd(v[k], v[k + 8]);
      b[k] = csub(v[k], v[k + 8]);
    }
    halves(a, b, v);
  }
  __device__ __forceinline__ static void run_half(cpk* v) {
    cpk a[8], b[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) a[k] = b[k] = v[k];
    halves(a, b, v);
  }
};

// the pass recursion's butterflies on packed values
template <int R, bool INV, bool HALF> __device__ __forceinline__ void butterfly(cpk* v) {
  if constexpr (R == 10 || R == 12 || R == 20)
    DFT<R, INV>::run(v);
  else if constexpr (HALF && (R == 4 || R == 8 || R == 16))
    PDFT<R, INV>::run_half(v);
  else
    PDFT<R, INV>::run(v);
}

}  // namespace marie
