// fft2.cuh — the Stockham transforms of fft.cuh on two fields at once.
//
// A Cx2 holds one complex element of two radii: the pair of real parts and
// the pair of imaginary parts, each in one 64-bit register pair, so that every
// addition, product and fused multiply-add is one packed instruction
// (add/sub/mul/fma.rn.f32x2) for both radii, and every load, store, twiddle and
// address serves both.  A packed instruction occupies the FP32 pipe as long as
// two scalar ones (measured: 39.1 T scalar FMA/s, 18.8-19.6 T packed ones), but
// takes one issue slot: the transforms are bound by instruction issue, not by
// the FP32 pipe.
//
// The arithmetic of each half is that of fft.cuh operation by operation, with
// the fusions the compiler makes there (a product by sqrt(1/2) or sqrt(3)/2 is
// fused into the additions that follow) written out, so each radius comes out
// with the same bits as from the one-field transforms.
#pragma once
#include "fft.cuh"

namespace prc {

typedef unsigned long long f32x2;  // (low, high) floats in one register pair

__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 a) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
  return r;
}
__device__ __forceinline__ f32x2 dup2(float a) { return pack2(a, a); }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// negation half by half: an operand modifier of the packed instruction that
// uses it (measured at no cost; an XOR of the sign bits is not folded)
__device__ __forceinline__ f32x2 neg2(f32x2 a) {
  const float2 v = unpack2(a);
  return pack2(-v.x, -v.y);
}

struct Cx2 {
  f32x2 re, im;
};
__device__ __forceinline__ Cx2 cadd(Cx2 a, Cx2 b) { return {add2(a.re, b.re), add2(a.im, b.im)}; }
__device__ __forceinline__ Cx2 csub(Cx2 a, Cx2 b) { return {sub2(a.re, b.re), sub2(a.im, b.im)}; }
// a + s i b and a - s i b, s = +1 (INV) or -1
template <bool INV> __device__ __forceinline__ Cx2 cadd_i(Cx2 a, Cx2 b) {
  return INV ? Cx2{sub2(a.re, b.im), add2(a.im, b.re)} : Cx2{add2(a.re, b.im), sub2(a.im, b.re)};
}
template <bool INV> __device__ __forceinline__ Cx2 csub_i(Cx2 a, Cx2 b) { return cadd_i<!INV>(a, b); }
// a * w, w given as the two factors dup2(w.x), dup2(w.y)
__device__ __forceinline__ Cx2 cmul(Cx2 a, f32x2 wx, f32x2 wy) {
  return {fma2(a.re, wx, neg2(mul2(a.im, wy))), fma2(a.re, wy, mul2(a.im, wx))};
}
// the twiddle conjugated for the forward direction
template <bool INV> __device__ __forceinline__ Cx2 ctwid(Cx2 a, float2 w) {
  return cmul(a, dup2(w.x), dup2(INV ? w.y : -w.y));
}

// ---------------------------------------------------------------- small DFTs
// PRE: the first layer is done (scaled_layer): the inputs are the sums and
// differences (radix 16: a[m] and a[m + 8]; radix 12: see Dft2x<3>).
template <int R, bool INV, bool PRE = false> struct Dft2x;

template <bool INV> struct Dft2x<2, INV> {
  static __device__ __forceinline__ void run(Cx2* a) {
    const Cx2 t = a[1];
    a[1] = csub(a[0], t);
    a[0] = cadd(a[0], t);
  }
};

// PRE: a[0] = a0 + (a1 + a2), a[1] = a0 - (a1 + a2)/2, a[2] = a1 - a2
template <bool INV, bool PRE> struct Dft2x<3, INV, PRE> {
  static __device__ __forceinline__ void run(Cx2* a) {
    const f32x2 c = dup2(PRC_SQRT3_2), mc = dup2(-PRC_SQRT3_2);
    Cx2 t2 = a[1], d = a[2];
    if constexpr (!PRE) {
      const f32x2 mh = dup2(-0.5f);
      const Cx2 t1 = cadd(a[1], a[2]);
      d = csub(a[1], a[2]);
      t2 = {fma2(mh, t1.re, a[0].re), fma2(mh, t1.im, a[0].im)};
      a[0] = cadd(a[0], t1);
    }
    // t2 +- s i c d
    a[INV ? 1 : 2] = {fma2(d.im, mc, t2.re), fma2(d.re, c, t2.im)};
    a[INV ? 2 : 1] = {fma2(d.im, c, t2.re), fma2(d.re, mc, t2.im)};
  }
};

template <bool INV, bool PRE> struct Dft2x<4, INV, PRE> {
  static __device__ __forceinline__ void run(Cx2* a) {
    const Cx2 t0 = PRE ? a[0] : cadd(a[0], a[2]), t1 = PRE ? a[2] : csub(a[0], a[2]);
    const Cx2 t2 = PRE ? a[1] : cadd(a[1], a[3]), d = PRE ? a[3] : csub(a[1], a[3]);
    a[0] = cadd(t0, t2);
    a[2] = csub(t0, t2);
    a[1] = cadd_i<INV>(t1, d);
    a[3] = csub_i<INV>(t1, d);
  }
};

template <bool INV, bool PRE> struct Dft2x<12, INV, PRE> {
  static __device__ __forceinline__ void run(Cx2* a) {
    Cx2 y[4][3];
#pragma unroll
    for (int n2 = 0; n2 < 4; ++n2) {
      Cx2 b[3] = {a[(3 * n2) % 12], a[(4 + 3 * n2) % 12], a[(8 + 3 * n2) % 12]};
      Dft2x<3, INV, PRE>::run(b);
#pragma unroll
      for (int k1 = 0; k1 < 3; ++k1) y[n2][k1] = b[k1];
    }
#pragma unroll
    for (int k1 = 0; k1 < 3; ++k1) {
      Cx2 c[4] = {y[0][k1], y[1][k1], y[2][k1], y[3][k1]};
      Dft2x<4, INV>::run(c);
#pragma unroll
      for (int k2 = 0; k2 < 4; ++k2) a[(4 * k1 + 9 * k2) % 12] = c[k2];
    }
  }
};

// lo, hi = e +- w8 o and e +- w8^3 o: the sums of o's parts first, their
// product by sqrt(1/2) fused into the additions
template <bool INV> __device__ __forceinline__ void comb_w8_1(Cx2& lo, Cx2& hi, Cx2 e, Cx2 o) {
  const f32x2 c = dup2(PRC_SQRT1_2), mc = dup2(-PRC_SQRT1_2);
  const f32x2 d = sub2(o.re, o.im), s = add2(o.re, o.im);
  const f32x2 tr = INV ? d : s;  // t = o + s i o
  if constexpr (INV) {
    lo = {fma2(tr, c, e.re), fma2(s, c, e.im)};
    hi = {fma2(tr, mc, e.re), fma2(s, mc, e.im)};
  } else {
    lo = {fma2(tr, c, e.re), fma2(d, mc, e.im)};
    hi = {fma2(tr, mc, e.re), fma2(d, c, e.im)};
  }
}
template <bool INV> __device__ __forceinline__ void comb_w8_3(Cx2& lo, Cx2& hi, Cx2 e, Cx2 o) {
  const f32x2 c = dup2(PRC_SQRT1_2), mc = dup2(-PRC_SQRT1_2);
  const f32x2 d = sub2(o.re, o.im), s = add2(o.re, o.im);
  // t = s i o - o: INV (-(re + im), re - im), else (im - re, -(re + im))
  if constexpr (INV) {
    lo = {fma2(s, mc, e.re), fma2(d, c, e.im)};
    hi = {fma2(s, c, e.re), fma2(d, mc, e.im)};
  } else {
    lo = {fma2(d, mc, e.re), fma2(s, mc, e.im)};
    hi = {fma2(d, c, e.re), fma2(s, c, e.im)};
  }
}

template <bool INV, bool PRE> struct Dft2x<8, INV, PRE> {
  static __device__ __forceinline__ void run(Cx2* a) {
    Cx2 e[4] = {a[0], a[2], a[4], a[6]};
    Cx2 o[4] = {a[1], a[3], a[5], a[7]};
    Dft2x<4, INV, PRE>::run(e);
    Dft2x<4, INV, PRE>::run(o);
    a[0] = cadd(e[0], o[0]);
    a[4] = csub(e[0], o[0]);
    comb_w8_1<INV>(a[1], a[5], e[1], o[1]);
    a[2] = cadd_i<INV>(e[2], o[2]);
    a[6] = csub_i<INV>(e[2], o[2]);
    comb_w8_3<INV>(a[3], a[7], e[3], o[3]);
  }
};

template <bool INV, bool PRE> struct Dft2x<16, INV, PRE> {
  static __device__ __forceinline__ void run(Cx2* a) {
    Cx2 e[8], o[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      e[k] = a[2 * k];
      o[k] = a[2 * k + 1];
    }
    Dft2x<8, INV, PRE>::run(e);
    Dft2x<8, INV, PRE>::run(o);
    auto pm = [&](int k, Cx2 t) {
      a[k] = cadd(e[k], t);
      a[k + 8] = csub(e[k], t);
    };
    pm(0, o[0]);
    pm(1, ctwid<INV>(o[1], make_float2(PRC_COS_PI8, PRC_SIN_PI8)));
    comb_w8_1<INV>(a[2], a[10], e[2], o[2]);
    pm(3, ctwid<INV>(o[3], make_float2(PRC_SIN_PI8, PRC_COS_PI8)));
    a[4] = cadd_i<INV>(e[4], o[4]);
    a[12] = csub_i<INV>(e[4], o[4]);
    pm(5, ctwid<INV>(o[5], make_float2(-PRC_SIN_PI8, PRC_COS_PI8)));
    comb_w8_3<INV>(a[6], a[14], e[6], o[6]);
    pm(7, ctwid<INV>(o[7], make_float2(-PRC_COS_PI8, PRC_SIN_PI8)));
  }
};

// The 16-point DFT whose last layer's sums and differences change places where
// s = -1 (s = +1: Dft2x<16>): a[k] = e[k] + s t[k], a[k + 8] = e[k] - s t[k].
// The products by s are exact, so the values keep their bits.
template <bool INV> __device__ __forceinline__ void dft16_signed(Cx2* a, float s) {
  const f32x2 p = dup2(s), m = dup2(-s), c = dup2(s * PRC_SQRT1_2), mc = dup2(-s * PRC_SQRT1_2);
  Cx2 e[8], o[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    e[k] = a[2 * k];
    o[k] = a[2 * k + 1];
  }
  Dft2x<8, INV>::run(e);
  Dft2x<8, INV>::run(o);
  auto pm = [&](int k, Cx2 t) {
    a[k] = {fma2(t.re, p, e[k].re), fma2(t.im, p, e[k].im)};
    a[k + 8] = {fma2(t.re, m, e[k].re), fma2(t.im, m, e[k].im)};
  };
  // e +- s w8 o, e +- s w8^3 o: comb_w8_1 and comb_w8_3 with c for sqrt(1/2)
  auto w81 = [&](int k) {
    const f32x2 d = sub2(o[k].re, o[k].im), q = add2(o[k].re, o[k].im);
    a[k] = INV ? Cx2{fma2(d, c, e[k].re), fma2(q, c, e[k].im)} : Cx2{fma2(q, c, e[k].re), fma2(d, mc, e[k].im)};
    a[k + 8] = INV ? Cx2{fma2(d, mc, e[k].re), fma2(q, mc, e[k].im)} : Cx2{fma2(q, mc, e[k].re), fma2(d, c, e[k].im)};
  };
  auto w83 = [&](int k) {
    const f32x2 d = sub2(o[k].re, o[k].im), q = add2(o[k].re, o[k].im);
    a[k] = INV ? Cx2{fma2(q, mc, e[k].re), fma2(d, c, e[k].im)} : Cx2{fma2(d, mc, e[k].re), fma2(q, mc, e[k].im)};
    a[k + 8] = INV ? Cx2{fma2(q, c, e[k].re), fma2(d, mc, e[k].im)} : Cx2{fma2(d, c, e[k].re), fma2(q, c, e[k].im)};
  };
  pm(0, o[0]);
  pm(1, ctwid<INV>(o[1], make_float2(PRC_COS_PI8, PRC_SIN_PI8)));
  w81(2);
  pm(3, ctwid<INV>(o[3], make_float2(PRC_SIN_PI8, PRC_COS_PI8)));
  // s i o[4] and its negative
  const f32x2 ip = INV ? p : m, im = INV ? m : p;
  a[4] = {fma2(o[4].im, im, e[4].re), fma2(o[4].re, ip, e[4].im)};
  a[12] = {fma2(o[4].im, ip, e[4].re), fma2(o[4].re, im, e[4].im)};
  pm(5, ctwid<INV>(o[5], make_float2(-PRC_SIN_PI8, PRC_COS_PI8)));
  w83(6);
  pm(7, ctwid<INV>(o[7], make_float2(-PRC_COS_PI8, PRC_SIN_PI8)));
}

// The second and third stage of a <16, 16, 2> plan of length 512 whose lanes j
// and j ^ 16 are lanes of one warp (lane ^ 16).  v: the second stage's inputs
// j + 32*m with their twiddles applied.  The last butterflies join positions k
// and k + 256, which the second stage leaves in lanes u and u + 16: each keeps
// eight of its values and gives the other eight to its partner by shuffles (no
// exchange through shared memory: 5.07 -> 4.32 ms where the exchange inside
// the warp through memory took 4.64, the window pass of 32 radii at 512^3).
// With the sums and differences of lane u + 16 changed places, those given are
// v[8..15] in both lanes.  Out: v[r + 8*q] is position u + 128*(j / 16) + 16*r
// + 256*q.
template <bool INV> __device__ __forceinline__ void last_two_stages(Cx2 (&v)[16], int j, const float2* tws) {
  const int u = j & 15, h = j >> 4;
  dft16_signed<INV>(v, h ? -1.f : 1.f);
  auto swap = [](f32x2 x) {
    const float2 f = unpack2(x);
    return pack2(__shfl_xor_sync(0xffffffffu, f.x, 16), __shfl_xor_sync(0xffffffffu, f.y, 16));
  };
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const Cx2 got = {swap(v[r + 8].re), swap(v[r + 8].im)}, kept = v[r];
    Cx2 a[2] = {h ? got : kept, h ? kept : got};
    a[1] = ctwid<INV>(a[1], tws[240 + 128 * h + 16 * r + u]);
    Dft2x<2, INV>::run(a);
    v[r] = a[0];
    v[r + 8] = a[1];
  }
}

// The first layer of the first stage (radix R0, E elements a lane) on real
// multiples x[m] * w[m] of complex numbers x[m].  The compiler fuses these
// products into the additions in the one-field kernel; the same ones are fused
// here: the first operand's with radices 4 and 16, the second's with radix 12.
template <int E, int R0, class X, class W> __device__ __forceinline__ void scaled_layer(Cx2* v, X x, W w) {
  auto scale = [](float2 a, float2 k) { return Cx2{pack2(a.x * k.x, a.x * k.y), pack2(a.y * k.x, a.y * k.y)}; };
  auto fused = [](float2 a, float2 k, Cx2 c) {
    const f32x2 kk = pack2(k.x, k.y);
    return Cx2{fma2(dup2(a.x), kk, c.re), fma2(dup2(a.y), kk, c.im)};
  };
  if constexpr (R0 == 12) {
    static_assert(E == 12, "one radix-12 butterfly a lane");
    const f32x2 mh = dup2(-0.5f);
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      const int i0 = (3 * n) % 12, i1 = (4 + 3 * n) % 12, i2 = (8 + 3 * n) % 12;
      const float2 a0 = x(i0), a1 = x(i1), a2 = x(i2), w2 = w(i2);
      const Cx2 z = scale(a0, w(i0)), p = scale(a1, w(i1));
      const Cx2 t1 = fused(a2, w2, p);
      v[i2] = fused(make_float2(-a2.x, -a2.y), w2, p);
      v[i1] = {fma2(mh, t1.re, z.re), fma2(mh, t1.im, z.im)};
      v[i0] = cadd(z, t1);
    }
  } else {
    static_assert(R0 % 4 == 0 && E % R0 == 0, "first layer: elements m and m + E/2");
#pragma unroll
    for (int m = 0; m < E / 2; ++m) {
      const float2 a = x(m), wa = w(m);
      const Cx2 q = scale(x(m + E / 2), w(m + E / 2));
      v[m] = fused(a, wa, q);
      v[m + E / 2] = fused(a, wa, Cx2{neg2(q.re), neg2(q.im)});
    }
  }
}

// The same for the adjoint's sources A * (h0 + i h1), h0 and h1 pairs of reals.
template <int E, int R0> __device__ __forceinline__ void adj_layer(Cx2* v, float A, const float2* h0, const float2* h1) {
  const f32x2 aa = dup2(A);
  auto pk = [](float2 h) { return pack2(h.x, h.y); };
  // (scalar products: packed ones would be fused into a packed addition)
  auto sc = [&](float2 h) { return pack2(__fmul_rn(A, h.x), __fmul_rn(A, h.y)); };
  auto scale = [&](int m) { return Cx2{sc(h0[m]), sc(h1[m])}; };
  auto fused = [&](int m, Cx2 c) { return Cx2{fma2(aa, pk(h0[m]), c.re), fma2(aa, pk(h1[m]), c.im)}; };
  auto minus = [](Cx2 c) { return Cx2{neg2(c.re), neg2(c.im)}; };
  if constexpr (R0 == 12) {
    const f32x2 mh = dup2(-0.5f);
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      const int i0 = (3 * n) % 12, i1 = (4 + 3 * n) % 12, i2 = (8 + 3 * n) % 12;
      const Cx2 z = scale(i0), p = scale(i1);
      const Cx2 t1 = fused(i2, p);
      v[i2] = minus(fused(i2, minus(p)));
      v[i1] = {fma2(mh, t1.re, z.re), fma2(mh, t1.im, z.im)};
      v[i0] = cadd(z, t1);
    }
  } else {
#pragma unroll
    for (int m = 0; m < E / 2; ++m) {
      const Cx2 q = scale(m + E / 2);
      v[m] = fused(m, q);
      v[m + E / 2] = fused(m, minus(q));
    }
  }
}

// ---------------------------------------------------------------- Stockham
// As Stages in fft.cuh.  Buf addresses are sums: off(p) is the offset of
// position p, and off(a + b) = off(a) + off(b) for the splits used here (a
// thread part a and a compile-time part b), so every access is a per-thread
// base plus a constant.  A stage with span Ns and G lanes splits its store
// positions that way when one of Ns and G divides the other; otherwise (12-
// point stages) the base is formed per butterfly.
template <int L, int E, bool INV, bool PRE, int Ns, int OFF, int... Rs> struct Stages2x;

template <int L, int E, bool INV, bool PRE, int Ns, int OFF> struct Stages2x<L, E, INV, PRE, Ns, OFF> {
  template <class Buf, class Sync>
  static __device__ __forceinline__ void run(Cx2 (&)[E], const Buf&, int, const float2*, const Sync&) {}
};

template <int L, int E, bool INV, bool PRE, int Ns, int OFF, int R, int... Rest>
struct Stages2x<L, E, INV, PRE, Ns, OFF, R, Rest...> {
  template <class Buf, class Sync>
  static __device__ __forceinline__ void run(Cx2 (&v)[E], const Buf& buf, int t, const float2* tws, const Sync& sync) {
    constexpr int G = L / E, Q = E / R;
    constexpr bool last = (Ns * R == L);
    constexpr bool low = Ns <= G && G % Ns == 0;   // t/Ns, t%Ns and q*G*R
    constexpr bool high = Ns > G && Ns % G == 0;   // t and the rest constant
    constexpr int NG = high ? Ns / G : 1;
    int hw = 0;
    if constexpr (!last && low) hw = Buf::off((t / Ns) * Ns * R + (t % Ns));
    if constexpr (!last && high) hw = Buf::off(t);
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int j = t + G * q;
      const int k = (Ns == 1) ? 0 : (j % Ns);
      Cx2 a[R];
#pragma unroll
      for (int r = 0; r < R; ++r) a[r] = v[q + r * Q];
      if constexpr (Ns > 1) {
#pragma unroll
        for (int r = 1; r < R; ++r) a[r] = ctwid<INV>(a[r], tws[OFF + (r - 1) * Ns + k]);
      }
      Dft2x<R, INV, PRE>::run(a);
      if constexpr (last) {
#pragma unroll
        for (int r = 0; r < R; ++r) v[q + r * Q] = a[r];
      } else if constexpr (low || high) {
#pragma unroll
        for (int r = 0; r < R; ++r)
          buf.put(hw, low ? (q * G * R + r * Ns) : ((q / NG) * Ns * R + G * (q % NG) + r * Ns), a[r]);
      } else {
        const int base = Buf::off((j / Ns) * Ns * R + k);
#pragma unroll
        for (int r = 0; r < R; ++r) buf.put(base, r * Ns, a[r]);
      }
    }
    if constexpr (!last) {
      sync();
      if constexpr (Buf::READ_POS) {
#pragma unroll
        for (int m = 0; m < E; ++m) v[m] = buf.get_pos(t + G * m);
      } else {
        const int hr = Buf::off(t);
#pragma unroll
        for (int m = 0; m < E; ++m) v[m] = buf.get(hr, G * m);
      }
      if constexpr (sizeof...(Rest) > 1) sync();  // another exchange follows
      Stages2x<L, E, INV, false, Ns * R, OFF + (Ns > 1 ? (R - 1) * Ns : 0), Rest...>::run(v, buf, t, tws, sync);
    }
  }
};

// The caller synchronises between the last reads of a transform and the next
// use of its buffer.
template <class P> struct PlanRun2x;
template <int E, int... R> struct PlanRun2x<Plan<E, R...>> {
  template <bool INV, bool PRE = false, class Buf, class Sync>
  static __device__ __forceinline__ void run(Cx2 (&v)[E], const Buf& buf, int t, const float2* tws, const Sync& sync) {
    Stages2x<Prod<R...>::v, E, INV, PRE, 1, 0, R...>::run(v, buf, t, tws, sync);
  }
};

}  // namespace prc
