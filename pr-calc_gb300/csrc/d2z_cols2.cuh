// d2z_cols2.cuh — column passes on pairs of radii (fft2.cuh).
//
// The slots of radii 2p and 2p + 1 of a sweep share one pair slot: an element
// holds (re a, re b, im a, im b), 16 bytes, so that one 16-byte load or store
// moves both radii and the packed arithmetic needs no register moves.  A sweep of an odd number of radii fills the last
// pair's second half with a copy of the last radius, whose barrier never wins.
//
// A tile is T columns x N rows as in k_col; thread (t, c) holds rows t + G*m of
// column c.  With T = 8 a row of the tile is 128 bytes and the eight lanes of a
// quarter-warp (one shared-memory wavefront of 16-byte accesses) are the eight
// columns of one row, so every exchange access is conflict-free without a
// swizzle and every shared address is a per-thread base plus a constant.
#pragma once
#include "d2z_cols.cuh"
#include "fft2.cuh"

namespace prc {

// Tile width and resident CTAs per SM of the pair passes (plans as in CCfg).
// Twelve elements a lane leave room for a third y CTA of 256 threads (80
// registers): 384^3 x 24 1.98 -> 1.83 ms, 768^3 x 16 12.6 -> 11.6; a fifth window CTA
// of 128 at 192 (x 41 0.306 -> 0.295 ms).  (Ten at 128 would gain 0.001 ms there.)
// At 1024 shared memory holds two y CTAs whatever MINB says; 80 registers took
// 18.0 ms for 12 radii, 128 18.4.  With sixteen elements elsewhere the same only
// spills (512^3 x 32: y 5.44 -> 5.51, window 4.12 -> 4.27).
// The accumulating x pass (MINBACC) holds a tile's values and windows at once:
// sixteen CTAs spill it at 32 and 64, and eight take 42.9 us against 55.2 (32^3 x
// 64) and 45.0 against 59.9 (64^3 x 64; twelve 47.1).  Elsewhere it takes what the
// window pass does, also where that spills: 192^3 x 41 five CTAs (52 bytes) 303.9,
// four 308.6; 512^3 x 32 four (16 bytes) 3753, three 3891; 96^3 x 32 eight or six
// 42.9; 128^3 x 32 eight 61.9, seven 63.5; 256^3 x 32 four 418, three 441; 384^3 x
// 24 four 1842, three 1930.
template <int N> struct C2Cfg { static constexpr bool on = false; };
template <> struct C2Cfg<32> { static constexpr bool on = true; static constexpr int T = 16, MINB = 16, TWIN = 16, MINBWIN = 16, MINBACC = 8, XB = 8; };
template <> struct C2Cfg<64> { static constexpr bool on = true; static constexpr int T = 8, MINB = 16, TWIN = 8, MINBWIN = 16, MINBACC = 8, XB = 8; };
template <> struct C2Cfg<96> { static constexpr bool on = true; static constexpr int T = 8, MINB = 8, TWIN = 8, MINBWIN = 8, MINBACC = 8, XB = 8; };
template <> struct C2Cfg<128> { static constexpr bool on = true; static constexpr int T = 8, MINB = 8, TWIN = 8, MINBWIN = 8, MINBACC = 8, XB = 8; };
template <> struct C2Cfg<192> { static constexpr bool on = true; static constexpr int T = 8, MINB = 5, TWIN = 8, MINBWIN = 5, MINBACC = 5, XB = 8; };
template <> struct C2Cfg<256> { static constexpr bool on = true; static constexpr int T = 8, MINB = 4, TWIN = 8, MINBWIN = 4, MINBACC = 4, XB = 8; };
template <> struct C2Cfg<384> { static constexpr bool on = true; static constexpr int T = 8, MINB = 3, TWIN = 4, MINBWIN = 4, MINBACC = 4, XB = 8; };
template <> struct C2Cfg<512> { static constexpr bool on = true; static constexpr int T = 8, MINB = 2, TWIN = 4, MINBWIN = 4, MINBACC = 4, XB = 4; };
template <> struct C2Cfg<768> { static constexpr bool on = true; static constexpr int T = 4, MINB = 3, TWIN = 4, MINBWIN = 2, MINBACC = 2, XB = 4; };
template <> struct C2Cfg<1024> { static constexpr bool on = true; static constexpr int T = 4, MINB = 3, TWIN = 8, MINBWIN = 1, MINBACC = 1, XB = 4; };

// Layout of a pair slot's main array: blocks of XB planes ix, in a block the
// order (iy, kz / T, ix % XB, kz % T) with T the window pass's tile width, so
// that the XB rows of a tile in one block are one contiguous piece.  (A tile's
// rows of 128 bytes, 2 MB apart in the single slot's order, are written at
// 5.0 TB/s at 512^3, pieces of 512 bytes or more at 6.5.)  The inverse y pass
// sees rows of XB * H contiguous elements, in any order; a z line is H / T
// pieces.
template <int N> struct PairSlot {
  static constexpr int H = N / 2, T = C2Cfg<N>::TWIN, XB = C2Cfg<N>::XB;
  static_assert(N % XB == 0 && H % T == 0, "whole blocks");
  // element (ix, iy, kz)
  static __device__ __forceinline__ long long at(int ix, int iy, int kz) {
    return (long long)((ix / XB) * N + iy) * (H * XB) + ix % XB * T + along(kz);
  }
  static __device__ __forceinline__ constexpr int along(int kz) { return kz / T * (XB * T) + kz % T; }
};

// Exchange buffer: row p of column c at p*T + c (16-byte elements).  T = 4: a
// quarter-warp holds two rows of four columns, FFT lanes t and t + 1; one row
// of padding after every PD keeps the two in opposite bank halves in every
// read (rows t + G*m) and first store (rows R0*t + r).  PD divides the strides
// that follow a lane's part of a position, so offsets add.
template <int T, int PD> struct PairCol {
  static constexpr bool READ_POS = false;
  ulonglong2* b;
  static __device__ __forceinline__ constexpr int off(int p) { return T == 4 ? (p + p / PD) * T : p * T; }
  __device__ __forceinline__ Cx2 get(int h, int cp) const {
    const ulonglong2 q = b[h + off(cp)];
    return {q.x, q.y};
  }
  __device__ __forceinline__ void put(int h, int cp, Cx2 v) const { b[h + off(cp)] = make_ulonglong2(v.re, v.im); }
};

template <int N, int MODE> struct CK2 {
  using P = typename CCfg<N>::P;
  static constexpr bool XP = MODE == TM_WIN || MODE == TM_ACC;  // an x pass: tiles of the slot's pieces
  static constexpr int H = N / 2, T = XP ? C2Cfg<N>::TWIN : C2Cfg<N>::T;
  static constexpr int E = P::E, G = N / E, THREADS = T * G, EH = E / 2;
  static constexpr int MINB = MODE == TM_ACC ? C2Cfg<N>::MINBACC : XP ? C2Cfg<N>::MINBWIN : C2Cfg<N>::MINB;
  static_assert(T == 16 || (T == 8 && G >= 4) || (T == 4 && G >= 8), "lane layouts");
  static_assert(THREADS % 32 == 0 && H % T == 0, "whole warps, whole tiles");
  static constexpr int TW = (PlanRun<P>::TW + 1) & ~1;
  static constexpr int PD = FirstRadix<P>::v == 12 ? 4 : 16;
  using Buf = PairCol<T, PD>;
  static constexpr int ROWS = T == 4 ? N + N / PD : N;
  // y passes: the tile by cp.async (16 bytes, past the L1 cache) instead
  // of loads into registers.  What such loads have in flight needs room in the
  // L1; at 256^3 a carve-out that another stream's kernel has enlarged slows
  // the pass from 0.635 to 0.94 ms for 32 radii, and at 1024^3 two CTAs' shared
  // memory leaves too little of it alone (22.1 ms against 18.5 for 12 radii).
  // The copies take one more trip through shared memory: 0.642 against 0.635
  // ms at 256 with the GPU to itself, 0.381 against 0.356 at 192^3 x 41, so 192
  // and the smaller ones load into registers; so does 384, where the two are
  // equal (three CTAs an SM, 24 radii: 1.822 against 1.830 ms, the adjoint's y
  // pass 1.827 against 1.825).
  static constexpr bool ASYNC = (MODE == TM_INV || MODE == TM_FWD) && N >= 256 && N != 384;
  // stage twiddles, exchange buffer, (x passes) the spectrum tile or the sums
  static constexpr size_t bytes = (size_t)TW * 8 + (size_t)ROWS * T * 16 + (XP ? (size_t)N * T * 8 : 0);
};

template <int THREADS> struct CtaSync2 {
  __device__ __forceinline__ void operator()() const {
    if constexpr (THREADS == 32) __syncwarp();
    else __syncthreads();
  }
};

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}

// Copies a per-radius parameter array into shared memory (the arguments are
// __grid_constant__, so a runtime index reads the constant bank).
__device__ __forceinline__ void stage_params_all(float* dst, const float (&src)[kMaxBatch]) {
  for (int i = threadIdx.x; i < kMaxBatch; i += blockDim.x) dst[i] = src[i];
}

// The column transform of one lane and the rows it ends up with: register e
// holds row base + rows(e) afterwards.  In general these are the rows t + G*m
// that the lane began with.  Plans <16, 16, R2> (512, 1024) end in a stage
// whose butterflies join positions k + 256*q, q < R2, which the second stage
// left in lanes u + 16*q: with those R2 lanes in one warp the last exchange
// stays inside the warp and needs no CTA barrier.  A lane writes its 16 values
// to the rows that it wrote in the first exchange, so no other warp touches
// them before the next transform's barrier.
template <int N, class P> struct ColFft {
  static constexpr bool TAIL = false;
  static constexpr int E = P::E, G = N / E;
  static __device__ __forceinline__ constexpr int rows(int e) { return G * e; }
};
template <int N, int R2> struct ColFft<N, Plan<16, 16, 16, R2>> {
  static constexpr bool TAIL = true;
  static constexpr int E = 16, G = N / 16, K = 16 / R2;  // K values of each quarter (half) a lane
  static_assert(N == 256 * R2 && G == 16 * R2, "<16, 16, R2>");
  static __device__ __forceinline__ constexpr int rows(int e) { return 16 * (e % K) + 256 * (e / K); }
};

// W(k R) for the two radii of a pair, tophat_big's operations half by half
// (rintf as the addition and subtraction of 1.5 * 2^23, exact for |y| < 2^22).
__device__ __forceinline__ f32x2 tophat_big2(float kq, float kra, float krb) {
  const float xa = kq * kra, xb = kq * krb;
  const f32x2 x = pack2(xa, xb), magic = dup2(12582912.0f);
  // (scalar products: a packed one is fused into the packed addition, which
  // decides ties differently)
  const f32x2 y = pack2(__fmul_rn(xa, 0.159154943091895336f), __fmul_rn(xb, 0.159154943091895336f));
  const f32x2 k = sub2(add2(y, magic), magic);
  f32x2 r = fma2(neg2(k), dup2(6.28318548202514648f), x);
  r = fma2(neg2(k), dup2(-1.74845560e-07f), r);
  const float2 rr = unpack2(r);
  const f32x2 s = pack2(__sinf(rr.x), __sinf(rr.y)), c = pack2(__cosf(rr.x), __cosf(rr.y));
  const f32x2 ix = pack2(rcp_approx(xa), rcp_approx(xb));
  return mul2(mul2(dup2(3.0f), fma2(neg2(x), c, s)), mul2(mul2(ix, ix), ix));
}

// MODE: TM_INV, TM_FWD (blockIdx.y: the pair), TM_WIN (the spectrum tile stays
// in shared memory, each thread's own elements, for all pairs of the sweep) or
// TM_ACC (per pair: forward transform, W times it added to the tile's sums,
// which stay in shared memory likewise; one read-modify-write of the output).
// MB: grouped launch, as in k_col; a.nvb counts boxes per pair there.
template <int N, int MODE, bool MB = false>
__global__ void __launch_bounds__(CK2<N, MODE>::THREADS, CK2<N, MODE>::MINB) k_col2(const __grid_constant__ TileArgs a) {
  using KK = CK2<N, MODE>;
  using P = typename KK::P;
  using L = PairSlot<N>;
  // the window's products are fused into the first stage's additions
  constexpr bool PRE = MODE == TM_WIN;
  constexpr bool INV = MODE == TM_INV || MODE == TM_WIN, XP = KK::XP;
  constexpr int H = N / 2, E = KK::E, G = KK::G, T = KK::T, EH = KK::EH, TH = KK::THREADS;
  static_assert(!MB || INV, "no grouped adjoint passes");
  extern __shared__ float4 smem4[];
  float2* tws = reinterpret_cast<float2*>(smem4);
  ulonglong2* xbuf = reinterpret_cast<ulonglong2*>(tws + KK::TW);
  float2* raw = reinterpret_cast<float2*>(xbuf + KK::ROWS * T) + threadIdx.x;  // element m at raw[m * TH]
  __shared__ float s_kr[kMaxBatch];
  if constexpr (XP && !MB) stage_params_all(s_kr, a.kr);
  PlanRun<P>::template fill<1>(tws, a.tw);
  pdl_wait();
  __syncthreads();
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, c = lane & (T - 1);
  // (TM_ACC needs the mirrors of its final rows in the same warp: rows t + G*m,
  // or at 512 those of the lanes u below, which leave out an exchange: 4.68 ->
  // 4.33 ms for 32 radii)
  using F = ColFft<N, typename std::conditional<MODE == TM_ACC && N != 512, Plan<P::E>, P>::type>;
  constexpr bool ACC_TAIL = MODE == TM_ACC && F::TAIL;
  // FFT lane t of the first stage.  A warp holds lanes and their mirrors G - t
  // (lane ^ 16; t = 0 pairs with G/2), for the window.
  int t;
  if constexpr (T == 16) {
    t = (lane < 16) ? wp : (wp == 0 ? G / 2 : G - wp);
  } else if constexpr (T == 4) {
    const int u = 4 * wp + ((lane >> 2) & 3);
    t = (lane < 16) ? u : (u == 0 ? G / 2 : G - u);
  } else {
    // lanes w, w + G/4 and their mirrors G - w, G - G/4 - w (w = 0: G/2)
    constexpr int Q = G / 4;
    const int sl = (lane >> 3) & 1;
    t = (lane < 16) ? (sl ? wp + Q : wp) : (sl ? G - Q - wp : (wp ? G - wp : G / 2));
  }
  // FFT lane j of the later stages: (TAIL) u + 16*q, q < R2, of a warp's u
  int j = t;
  if constexpr (F::TAIL) {
    constexpr int R2 = N / 256, U = 32 / T / R2;  // values of u a warp
    const int s = lane / T;
    int u = wp * U + s % U;
    if constexpr (ACC_TAIL) {
      // u and 16 - u in one warp: 2 wp, 2 wp + 1 and their mirrors (0 and 8
      // are their own)
      static_assert(U == 4, "two values of u and their mirrors");
      const int i = s % U;
      u = i < 2 ? 2 * wp + i : (wp == 0 && i == 2 ? 8 : 18 - 2 * wp - i);
    }
    j = (s / U) * 16 + u;
  }
  const int row0 = F::TAIL ? (j & 15) + (j >> 4) * (256 / (F::TAIL ? N / 256 : 1)) : t;  // first of the lane's final rows
  using Buf = typename KK::Buf;
  const Buf buf{xbuf + c};
  const CtaSync2<TH> sync;
  const long long yoff = XP ? 0 : (long long)blockIdx.y * a.slot_stride;
  const int tiles0 = a.seg[0].n_outer * a.seg[0].tpo;
  const int tpb = tiles0 + a.seg[1].n_outer * a.seg[1].tpo;
  const int tiles = !MB ? tpb : tpb * (MODE == TM_INV ? a.nvb[blockIdx.y] : a.nbox);

  struct Where {
    int sn, outer, tc, bx;
    long long off;
  };
  auto where = [&](int ti) {
    Where w;
    w.bx = 0;
    if constexpr (MB) {
      w.bx = ti / tpb;
      ti -= w.bx * tpb;
    }
    w.sn = ti >= tiles0;
    const int tl = w.sn ? ti - tiles0 : ti;
    const int tpo = w.sn ? a.seg[1].tpo : a.seg[0].tpo;
    w.outer = tl / tpo;
    w.tc = tl - w.outer * tpo;
    w.off = (long long)w.outer * (w.sn ? a.seg[1].outer_stride : a.seg[0].outer_stride) + (long long)w.tc * T;
    return w;
  };
  auto seg_in = [&](const Where& w) -> const float2* {
    if constexpr (MB) return w.sn ? a.box[w.bx].in1 : a.box[w.bx].in0;
    else return w.sn ? a.seg[1].in : a.seg[0].in;
  };
  auto seg_out = [&](const Where& w) -> ulonglong2* {
    float2* o;
    if constexpr (MB) o = w.sn ? a.box[w.bx].out1 : a.box[w.bx].out0;
    else o = w.sn ? a.seg[1].out : a.seg[0].out;
    return reinterpret_cast<ulonglong2*>(o);
  };
  auto seg_rs = [&](const Where& w) { return w.sn ? a.seg[1].row_stride : a.seg[0].row_stride; };
  auto transform = [&](Cx2 (&v)[E]) {
    if constexpr (!F::TAIL) {
      PlanRun2x<P>::template run<INV, PRE>(v, buf, t, tws, sync);
    } else {
      constexpr int R2 = N / 256, K = 16 / R2, U = 32 / T / R2;
      const int own = Buf::off(16 * t);
      Dft2x<16, INV, PRE>::run(v);
#pragma unroll
      for (int r = 0; r < 16; ++r) buf.put(own, r, v[r]);
      sync();
      const int hr = Buf::off(j);
#pragma unroll
      for (int m = 0; m < 16; ++m) v[m] = buf.get(hr, G * m);
      if constexpr (R2 > 2) sync();  // every lane has read: the rows may be written again
      const int u = j & 15;
#pragma unroll
      for (int r = 1; r < 16; ++r) v[r] = ctwid<INV>(v[r], tws[(r - 1) * 16 + u]);
      if constexpr (R2 == 2) {
        last_two_stages<INV>(v, j, tws);
        return;
      }
      Dft2x<16, INV>::run(v);
#pragma unroll
      for (int r = 0; r < 16; ++r) buf.put(own, r, v[r]);
      __syncwarp();
      // rows 16 t of the warp's lanes u + 16*q: lane slots U apart
      int src[R2];
#pragma unroll
      for (int q = 0; q < R2; ++q)
        src[q] = __shfl_sync(0xffffffffu, own, (q * U + (lane / T) % U) * T + c) + Buf::off(K * (j >> 4));
#pragma unroll
      for (int r = 0; r < K; ++r) {
        Cx2 a[R2];
#pragma unroll
        for (int q = 0; q < R2; ++q) a[q] = buf.get(src[q], r);
        const int k = K * 16 * (j >> 4) + 16 * r + u;
#pragma unroll
        for (int q = 1; q < R2; ++q) a[q] = ctwid<INV>(a[q], tws[240 + (q - 1) * 256 + k]);
        Dft2x<R2, INV>::run(a);
#pragma unroll
        for (int q = 0; q < R2; ++q) v[r + K * q] = a[q];
      }
    }
  };
  // the previous transform's last exchange through memory has been read by its
  // readers: the CTA, or (R2 = 4) this warp alone
  auto reuse = [&]() {
    if constexpr (F::TAIL && N > 512) __syncwarp();
    else sync();
  };
  auto gstore = [&](const Where& w, ulonglong2* dst, const Cx2 (&v)[E]) {
    if (w.sn ? a.seg[1].transpose : a.seg[0].transpose) {
      ulonglong2* q = dst + (long long)w.outer * (w.sn ? a.seg[1].outer_stride : a.seg[0].outer_stride) +
                      (long long)(w.tc * T + c) * N + row0;
#pragma unroll
      for (int m = 0; m < E; ++m) q[F::rows(m)] = make_ulonglong2(v[m].re, v[m].im);
    } else if (MODE == TM_WIN && !w.sn) {
      static_assert(MODE != TM_WIN || L::T == T, "the slot's pieces are the window pass's rows");
      ulonglong2* q = dst + c;
      if constexpr (F::rows(1) % L::XB == 0) {  // every row step crosses whole blocks
        q += L::at(row0, w.outer, w.tc * T);
#pragma unroll
        for (int m = 0; m < E; ++m) q[(long long)F::rows(m) * N * H] = make_ulonglong2(v[m].re, v[m].im);
      } else {
#pragma unroll
        for (int m = 0; m < E; ++m) q[L::at(row0 + F::rows(m), w.outer, w.tc * T)] = make_ulonglong2(v[m].re, v[m].im);
      }
    } else {
      const int rs = seg_rs(w);
      ulonglong2* q = dst + w.off + (long long)row0 * rs + c;
#pragma unroll
      for (int m = 0; m < E; ++m) q[(long long)F::rows(m) * rs] = make_ulonglong2(v[m].re, v[m].im);
    }
  };

  // |k| of rows t + G*m (TM_ACC: of the final rows), m <= E/2, of this thread's
  // column (-1: k = 0); returns the warp's smallest
  auto kmag = [&](const Where& w, float (&kq)[EH + 1]) {
    const int col = w.tc * T + c;
    const int syz = (w.sn ? a.seg[1].nyq : a.seg[0].nyq) ? fsq(col, N) + H * H : fsq(w.outer, N) + col * col;
#pragma unroll
    for (int m = 0; m <= EH; ++m) {
      const int m2 = fsq(MODE == TM_ACC ? row0 + F::rows(m) : t + G * m, N) + syz;
      kq[m] = (m2 == 0) ? -1.f : sqrtf((float)m2);
    }
    float kmin = kq[0];
#pragma unroll
    for (int m = 1; m <= EH; ++m) kmin = fminf(kmin, kq[m]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) kmin = fminf(kmin, __shfl_xor_sync(0xffffffffu, kmin, o));
    return kmin;
  };
  // W(|k| R) of all E rows for the two radii
  auto windows = [&](const float (&kq)[EH + 1], float kmin, float kra, float krb, float2 (&wm)[E]) {
    f32x2 wv[EH + 1];
#pragma unroll
    for (int m = 0; m <= EH; ++m) wv[m] = tophat_big2(kq[m], kra, krb);
    if (kmin * fminf(kra, krb) < 1.0f) {
      // some lane of the warp needs the series (or W(0) = 0)
#pragma unroll
      for (int m = 0; m <= EH; ++m) {
        const float xa = kq[m] * kra, xb = kq[m] * krb;
        float2 ww = unpack2(wv[m]);
        if (xa < 1.0f) ww.x = kq[m] < 0.f ? 0.f : tophat_small(xa);
        if (xb < 1.0f) ww.y = kq[m] < 0.f ? 0.f : tophat_small(xb);
        wv[m] = pack2(ww.x, ww.y);
      }
    }
    // rows m > E/2 mirror rows of the partner lane (lane ^ 16, FFT lane
    // G - t, register E-1-m), or of this lane (t = 0: E-m; t = G/2:
    // E-1-m; both in the first warp)
#pragma unroll
    for (int m = 0; m <= EH; ++m) wm[m] = unpack2(wv[m]);
    if constexpr (ACC_TAIL) {
      // row u + 128 h + 16 r + 256 q mirrors that of 16 - u, 1 - h and register
      // E-1-m; u = 0: of 0, 1 - h and E-m (but for r = 0, evaluated here)
      const int u = j & 15, from = lane ^ (u % 8 ? 24 : 16);
#pragma unroll
      for (int m = EH + 1; m < E; ++m) {
        const float2 s = u ? wm[E - 1 - m] : wm[E - m];
        wm[m] = make_float2(__shfl_sync(0xffffffffu, s.x, from), __shfl_sync(0xffffffffu, s.y, from));
      }
      return;
    }
#pragma unroll
    for (int m = EH + 1; m < E; ++m) {
      const float2 s = wm[E - 1 - m];
      float2 o = make_float2(__shfl_xor_sync(0xffffffffu, s.x, 16), __shfl_xor_sync(0xffffffffu, s.y, 16));
      if (wp == 0) {
        if (t == 0) o = wm[E - m];
        if (t == G / 2) o = s;
      }
      wm[m] = o;
    }
  };

  if constexpr (MODE == TM_INV || MODE == TM_FWD) {
    auto src = [&](const Where& w) {
      return reinterpret_cast<const ulonglong2*>(seg_in(w)) + yoff + w.off + (long long)t * seg_rs(w) + c;
    };
    if constexpr (KK::ASYNC || MB) {
      // A tile arrives by cp.async in the exchange buffer itself, every thread
      // copying the elements that it reads, the next tile's as soon as the
      // last exchange of this one has been read.
      const int own = Buf::off(t);
      auto load = [&](int ti) {
        const Where w = where(ti);
        const ulonglong2* p = src(w);
        const long long step = (long long)G * seg_rs(w);
#pragma unroll
        for (int m = 0; m < E; ++m) cp_async16(buf.b + own + Buf::off(G * m), p + m * step);
      };
      int ti = blockIdx.x;
      if (ti < tiles) load(ti);
      for (; ti < tiles; ti += gridDim.x) {
        const Where w = where(ti);
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        Cx2 v[E];
#pragma unroll
        for (int m = 0; m < E; ++m) v[m] = buf.get(own, G * m);
        sync();  // every thread has its elements: the buffer is free for the exchanges
        transform(v);
        sync();  // the last exchange has been read
        if (ti + (int)gridDim.x < tiles) load(ti + gridDim.x);
        gstore(w, seg_out(w) + yoff, v);
      }
    } else {
      for (int ti = blockIdx.x; ti < tiles; ti += gridDim.x) {
        const Where w = where(ti);
        const ulonglong2* p = src(w);
        const long long step = (long long)G * seg_rs(w);
        Cx2 v[E];
#pragma unroll
        for (int m = 0; m < E; ++m) {
          const ulonglong2 q = p[m * step];
          v[m] = {q.x, q.y};
        }
        reuse();
        transform(v);
        gstore(w, seg_out(w) + yoff, v);
      }
    }
  } else if constexpr (MODE == TM_ACC) {
    // The sums of a tile (raw) and its exchange buffer; a pair's tile is copied
    // into the exchange buffer by cp.async like the y passes' tiles, the next
    // one when the last exchange of this one has been read.
    const int own = Buf::off(t);
    auto load = [&](const Where& w, int p) {
      const ulonglong2* base = reinterpret_cast<const ulonglong2*>(seg_in(w)) + (long long)p * a.slot_stride + c;
      const int rs = seg_rs(w);
      if constexpr (G % L::XB == 0) {
        const ulonglong2* q = base + (w.sn ? w.off + (long long)t * rs : L::at(t, w.outer, w.tc * T));
        const long long step = w.sn ? (long long)G * rs : (long long)G * N * H;
#pragma unroll
        for (int m = 0; m < E; ++m) cp_async16(buf.b + own + Buf::off(G * m), q + m * step);
      } else {
#pragma unroll
        for (int m = 0; m < E; ++m)
          cp_async16(buf.b + own + Buf::off(G * m),
                     base + (w.sn ? w.off + (long long)(t + G * m) * rs : L::at(t + G * m, w.outer, w.tc * T)));
      }
    };
    const int np = (a.nb + 1) >> 1;
    int ti = blockIdx.x;
    if (ti < tiles) load(where(ti), 0);
    for (; ti < tiles; ti += gridDim.x) {
      const Where w = where(ti);
      float kq[EH + 1];
      const float kmin = kmag(w, kq);
#pragma unroll
      for (int m = 0; m < E; ++m) raw[m * TH] = make_float2(0.f, 0.f);
      for (int p = 0; p < np; ++p) {
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        Cx2 v[E];
#pragma unroll
        for (int m = 0; m < E; ++m) v[m] = buf.get(own, G * m);
        sync();  // every thread has its elements: the buffer is free for the exchanges
        transform(v);
        sync();  // the last exchange has been read
        if (p + 1 < np) load(w, p + 1);
        else if (ti + (int)gridDim.x < tiles) load(where(ti + gridDim.x), 0);
        float2 wm[E];
        windows(kq, kmin, s_kr[2 * p], s_kr[2 * p + 1], wm);
        const bool two = 2 * p + 1 < a.nb;
#pragma unroll
        for (int m = 0; m < E; ++m) {
          const float2 re = unpack2(v[m].re), im = unpack2(v[m].im);
          float2 s = raw[m * TH];
          s.x = fmaf(wm[m].x, re.x, s.x);
          s.y = fmaf(wm[m].x, im.x, s.y);
          if (two) {
            s.x = fmaf(wm[m].y, re.y, s.x);
            s.y = fmaf(wm[m].y, im.y, s.y);
          }
          raw[m * TH] = s;
        }
      }
      const int rs = seg_rs(w);
      float2* q = (w.sn ? a.seg[1].out : a.seg[0].out) + w.off + (long long)row0 * rs + c;
#pragma unroll
      for (int m = 0; m < E; ++m) {
        float2* const qm = q + (long long)F::rows(m) * rs;
        const float2 o = a.first ? make_float2(0.f, 0.f) : *qm, s = raw[m * TH];
        *qm = make_float2(o.x + s.x, o.y + s.y);
      }
    }
  } else {
    auto load_raw = [&](int ti) {
      const Where w = where(ti);
      const int rs = seg_rs(w);
      const float2* p = seg_in(w) + w.off + (long long)t * rs + c;
      const long long step = (long long)G * rs;
#pragma unroll
      for (int m = 0; m < E; ++m) cp_async8(raw + m * TH, p + m * step);
    };
    int ti = blockIdx.x;
    if (ti < tiles) load_raw(ti);
    cp_async_commit();
    for (; ti < tiles; ti += gridDim.x) {
      const Where w = where(ti);
      float kq[EH + 1];
      const float kmin = kmag(w, kq);
      cp_async_wait<0>();
      int p0 = 0, p1;
      if constexpr (MB) p1 = (__ldg(&a.box[w.bx].nb) + 1) >> 1;
      else if constexpr (kWinRadiusSplit<N>) radius_range((a.nb + 1) >> 1, p0, p1);
      else p1 = (a.nb + 1) >> 1;
      ulonglong2* const out = seg_out(w);
      for (int p = p0; p < p1; ++p) {
        float kra, krb;
        if constexpr (MB) {
          kra = __ldg(&a.box[w.bx].kr[2 * p]);
          krb = __ldg(&a.box[w.bx].kr[2 * p + 1]);
        } else {
          kra = s_kr[2 * p];
          krb = s_kr[2 * p + 1];
        }
        float2 wm[E];
        windows(kq, kmin, kra, krb, wm);
        Cx2 v[E];
        scaled_layer<E, FirstRadix<P>::v>(v, [&](int m) { return raw[m * TH]; }, [&](int m) { return wm[m]; });
        if (p == p1 - 1) {
          // this thread has read its spectrum elements for the last time: the
          // next tile's come in under the transform and the stores
          if (ti + (int)gridDim.x < tiles) load_raw(ti + gridDim.x);
          cp_async_commit();
        }
        reuse();
        transform(v);
        gstore(w, out + (long long)p * a.slot_stride, v);
      }
    }
    cp_async_wait<0>();
  }
  pdl_release();
}

}  // namespace prc
