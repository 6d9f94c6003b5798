// d2z_lines2.cuh — the inverse z pass on pairs of radii: k_c2r_zp's packing,
// transform, barrier and running max (d2z_lines.cuh) for two radii per step
// with the packed arithmetic of fft2.cuh, from the pair slots of d2z_cols2.cuh.
//
// A warp works alone on 32 / G lines: every lane copies the sixteen-byte
// elements that it needs itself (its mirror pairs X[k], X[H-k]) with cp.async
// into its own column of a staging area, the next step's as soon as this
// step's are in registers, and the copies complete on the warp's mbarrier.
// So no CTA barrier separates the steps, and the warps of an SM drift apart:
// one transforms while others wait for copies.  The transform's exchange runs
// in the warp's own buffer, padded by one element every PD positions so that
// the first stage's stores (stride: the first radix) hit distinct banks.
#pragma once
#include "d2z_cols2.cuh"
#include "d2z_lines.cuh"

namespace prc {

// PD: padding period, MINB: resident CTAs per SM, SP: warps that share a set of
// lines and split the pairs of a sweep
template <int N> struct P2Cfg { static constexpr bool on = false; };
template <> struct P2Cfg<32> { static constexpr bool on = true; static constexpr int PD = 8, MINB = 5, SP = 4; };
template <> struct P2Cfg<64> { static constexpr bool on = true; static constexpr int PD = 8, MINB = 5, SP = 4; };
template <> struct P2Cfg<96> { static constexpr bool on = true; static constexpr int PD = 24, MINB = 4, SP = 4; };
template <> struct P2Cfg<128> { static constexpr bool on = true; static constexpr int PD = 8, MINB = 5, SP = 4; };
template <> struct P2Cfg<192> { static constexpr bool on = true; static constexpr int PD = 24, MINB = 4, SP = 1; };
template <> struct P2Cfg<256> { static constexpr bool on = true; static constexpr int PD = 16, MINB = 3, SP = 1; };
template <> struct P2Cfg<384> { static constexpr bool on = true; static constexpr int PD = 24, MINB = 4, SP = 1; };
template <> struct P2Cfg<512> { static constexpr bool on = true; static constexpr int PD = 16, MINB = 3, SP = 1; };
template <> struct P2Cfg<768> { static constexpr bool on = true; static constexpr int PD = 24, MINB = 4, SP = 1; };
template <> struct P2Cfg<1024> { static constexpr bool on = true; static constexpr int PD = 16, MINB = 3, SP = 1; };

template <int N, bool MB = false> struct PK2 {
  using P = typename PCfg<N>::P;
  static constexpr int H = N / 2, E = P::E, G = H / E, PD = P2Cfg<N>::PD, MINB = P2Cfg<N>::MINB;
  static constexpr int SP = MB ? 1 : P2Cfg<N>::SP;  // (many boxes have lines enough)
  static constexpr int THREADS = 128, NL = THREADS / G, NG = NL / SP;  // line buffers, lines per CTA step
  static_assert(THREADS >= kMaxBatch && NG * SP * G == THREADS, "per-radius sums need a thread per radius");
  static_assert(SP == 1 || (SP == THREADS / 32 && E % SP == 0), "all warps of a CTA or one share lines");
  static_assert(PlanRun<P>::L == H && E % 2 == 0 && G >= 2 && G <= 32 && 32 % G == 0, "paired line shape");
  static constexpr int TW = (PlanRun<P>::TW + 1) & ~1;
  // 16-byte elements of one line's exchange buffer: padded, and G bank groups
  // on from the next line's where several lines share a wavefront
  static constexpr int pads = H + H / PD;
  static constexpr int LS = G >= 8 ? pads : pads + ((G - pads % 8) % 8 + 8) % 8;
  // quarter of the N-table, stage twiddles, exchange buffers, every lane's E staged elements,
  // every line's X[H/2]
  static constexpr int QT = N / 4 + 2;  // e^{2 pi i k/N}, k <= N/4 (even, for alignment)
  static constexpr size_t bytes = (size_t)(QT + TW) * 8 + (size_t)(NL * LS + E * THREADS + NL) * 16;
};

// The transform of a line and the positions it leaves in a lane: register m
// holds position pos(t) + step(m).  A <16, 16, 2> plan on 32 lanes (1024) ends
// without its second exchange (last_two_stages), but for the per-radius sums
// (SIG), which add up the cells of a lane in a fixed order.
template <class P, bool SIG> struct LineFft {
  static constexpr int L = PlanRun<P>::L, G = L / P::E;
  static __device__ __forceinline__ int pos(int t) { return t; }
  static __device__ __forceinline__ constexpr int step(int m) { return G * m; }
  template <class Buf, class Sync>
  static __device__ __forceinline__ void run(Cx2 (&v)[P::E], const Buf& buf, int t, const float2* tws, const Sync& sync) {
    PlanRun2x<P>::template run<true>(v, buf, t, tws, sync);
  }
};
template <> struct LineFft<Plan<16, 16, 16, 2>, false> {
  static __device__ __forceinline__ int pos(int t) { return (t & 15) + 128 * (t >> 4); }
  static __device__ __forceinline__ constexpr int step(int m) { return 16 * (m % 8) + 256 * (m / 8); }
  template <class Buf, class Sync>
  static __device__ __forceinline__ void run(Cx2 (&v)[16], const Buf& buf, int t, const float2* tws, const Sync& sync) {
    Dft2x<16, true>::run(v);
    const int hw = Buf::off(16 * t), hr = Buf::off(t);
#pragma unroll
    for (int r = 0; r < 16; ++r) buf.put(hw, r, v[r]);
    sync();
#pragma unroll
    for (int m = 0; m < 16; ++m) v[m] = buf.get(hr, 32 * m);
#pragma unroll
    for (int r = 1; r < 16; ++r) v[r] = ctwid<true>(v[r], tws[(r - 1) * 16 + (t & 15)]);
    last_two_stages<true>(v, t, tws);
  }
};

// Offsets add except where reads of a 12-point plan (PD = 24) meet a lane's
// position t: there each is formed by itself (Stages2x: get_pos).
template <int PD> struct PairLine {
  static constexpr bool READ_POS = PD == 24;
  ulonglong2* b;
  static __device__ __forceinline__ constexpr int off(int p) { return p + p / PD; }
  __device__ __forceinline__ Cx2 get(int h, int cp) const {
    const ulonglong2 q = b[h + off(cp)];
    return {q.x, q.y};
  }
  __device__ __forceinline__ Cx2 get_pos(int p) const {
    const ulonglong2 q = b[off(p)];
    return {q.x, q.y};
  }
  __device__ __forceinline__ void put_pos(int p, Cx2 v) const { b[off(p)] = make_ulonglong2(v.re, v.im); }
  __device__ __forceinline__ void put(int h, int cp, Cx2 v) const { b[h + off(cp)] = make_ulonglong2(v.re, v.im); }
};

// arrival of this thread at the barrier once all its cp.async so far are done
__device__ __forceinline__ void cp_async_arrive(uint64_t* bar) {
  const unsigned b = (unsigned)__cvta_generic_to_shared(bar);
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];\n" ::"r"(b) : "memory");
}

// AM and SIG as in k_c2r_zp, MB as in k_col2.  A warp takes its line groups in
// turn and of each the pairs sub, sub + SP, ...  With SP > 1 the CTA's warps
// share the lines of a group: small grids have too few lines to give every
// scheduler warps, and the warps' running maxima are merged at the end (the
// larger value wins, of equal ones the smaller radius, as in the serial
// order).  A wait that runs out of polls sets *a.err and ends the warp's work
// (it still takes part in the merges); its own copies are waited for
// (cp.async.wait_all) before it leaves.
// a.withhold (a test hook) makes the first warp of CTA 0 skip its first copies
// and their arrival, so that its first wait runs out with nothing in flight.
template <int N, bool AM, bool SIG, bool MB = false>
__global__ void __launch_bounds__(PK2<N, MB>::THREADS, PK2<N, MB>::MINB) k_c2r_zp2(const __grid_constant__ SweepArgs a) {
  static_assert(!(MB && SIG), "no per-radius sums in grouped launches");
  using KK = PK2<N, MB>;
  using P = typename KK::P;
  using L = PairSlot<N>;
  using F = LineFft<P, SIG>;
  constexpr int H = N / 2, E = KK::E, G = KK::G, NG = KK::NG, EH = E / 2, LS = KK::LS, TH = KK::THREADS;
  constexpr int SP = KK::SP;
  constexpr long long NN = (long long)N * N;
  static_assert(NN % NG == 0 && (NG % L::XB == 0 || L::XB % NG == 0), "whole line groups");
  extern __shared__ float4 smem4[];
  float2* tw = reinterpret_cast<float2*>(smem4);
  float2* tws = tw + KK::QT;
  ulonglong2* xbuf = reinterpret_cast<ulonglong2*>(tws + KK::TW);
  ulonglong2* stage = xbuf + KK::NL * LS + threadIdx.x;  // element i of this lane at stage[i * TH]
  ulonglong2* mid = xbuf + KK::NL * LS + E * TH + threadIdx.x / G;
  load_tw(tw, a.tw, N / 4 + 1);
  PlanRun<P>::template fill<2>(tws, a.tw);
  __shared__ double red[kMaxBatch];
  __shared__ float s_cb[kMaxBatch];
  if constexpr (!MB) stage_params_all(s_cb, a.cb);
  if (threadIdx.x < kMaxBatch) red[threadIdx.x] = 0.0;
  const int lb = threadIdx.x / G, t = threadIdx.x % G;  // line buffer, FFT lane
  const int sub = SP == 1 ? 0 : threadIdx.x >> 5;       // first pair
  const int g = SP == 1 ? lb : lb % NG;                 // line of the group
  const GroupSync<G> sync(lb);
  const int partner = (G - t) & (G - 1);
  const int t0 = F::pos(t);  // first cell pair of the lane after the transform
  constexpr int lgpb = (int)(NN / NG);  // line groups of one box
  const long long lg_all = MB ? (long long)lgpb * a.nbox : lgpb;
  const int nsteps_l = (int)((lg_all - blockIdx.x + gridDim.x - 1) / gridDim.x);
  auto box_of = [&](int lg) { return MB ? (int)(((long long)blockIdx.x + (long long)lg * gridDim.x) / lgpb) : 0; };
  // this lane group's line of line group lg: the block's planes first, then iy
  // (their pieces are neighbours in the slot); with SIG in file order, as in
  // k_c2r_zp, so that a warp adds up the same lines
  auto line_of = [&](int lg, int bx, int& ix, int& iy) {
    const int s = (int)((long long)blockIdx.x + (long long)lg * gridDim.x - (long long)bx * lgpb) * NG + g;
    const int xi = SIG ? 0 : s % L::XB, q = SIG ? s : s / L::XB;
    iy = q % N;
    ix = SIG ? q / N : (q / N) * L::XB + xi;
  };

  __shared__ __align__(8) uint64_t s_bar[TH / 32];
  uint64_t* const bar = &s_bar[threadIdx.x >> 5];
  if ((threadIdx.x & 31) == 0) {
    mbar_init(bar, 32);
    mbar_init_fence();
  }
  pdl_wait();
  __syncthreads();

  // copies of step (line group lg of this CTA, pair p): lane t's pairs (X[k],
  // X[H-k]), k = t + G*m, m < E/2; lane 0 takes the Nyquist element for X[H]
  // and X[H/2] besides
  const bool withheld = a.withhold && blockIdx.x == 0 && threadIdx.x < 32;
  auto issue = [&](int lg, int p) {
    if (lg < nsteps_l && !(withheld && lg == 0 && p == sub)) {
      const int bx = box_of(lg);
      int ix, iy;
      line_of(lg, bx, ix, iy);
      const ulonglong2* slot =
          reinterpret_cast<const ulonglong2*>(MB ? a.box[bx].slots : a.slots) + (long long)p * a.slot_stride;
      const ulonglong2* nyq = slot + NN * H + (long long)iy * N + ix;
      // position t + x, x a multiple of G, lies along(x) after position t
      static_assert(G % L::T == 0 || L::T % G == 0, "a lane's positions split");
      const ulonglong2* line = slot + L::at(ix, iy, 0);
      const ulonglong2* lo = line + L::along(t);
      const ulonglong2* hi = line + L::along(G - t);  // t > 0
#pragma unroll
      for (int m = 0; m < EH; ++m) {
        cp_async16(stage + m * TH, lo + L::along(G * m));
        cp_async16(stage + (EH + m) * TH,
                   t ? hi + L::along(H - G * (m + 1)) : (m ? line + L::along(H - G * m) : nyq));
      }
      if (t == 0) cp_async16(mid, line + L::along(H / 2));
      cp_async_arrive(bar);
    }
  };

  auto pairs_of = [&](int lg) { return ((MB ? a.box[box_of(lg)].nb : a.nb) + 1) >> 1; };
  int lg_next = 0, p_next = sub, np_next = pairs_of(0), i = 0;
  // moves (lg_next, p_next) on to a step that there is
  auto seek = [&]() {
    while (p_next >= np_next && ++lg_next < nsteps_l) {
      p_next = sub;
      np_next = pairs_of(lg_next);
    }
  };
  if constexpr (SP > 1) seek();
  issue(lg_next, p_next);
  bool dead = false;  // a wait ran out
  for (int lg = 0; lg < nsteps_l && (SP > 1 || !dead); ++lg) {
    const int bx = box_of(lg);
    const BoxLine* bp = MB ? a.box + bx : nullptr;
    const int np = pairs_of(lg);
    auto line = [&]() {  // this lane group's line in file order
      int ix, iy;
      line_of(lg, bx, ix, iy);
      return (long long)ix * N + iy;
    };
    float2 zr[E];
    uint32_t am[AM ? EH : 1];  // argmax bytes of cells 2p, 2p+1 of elements 2j (low half) and 2j+1
    if (MB ? bp->first : a.first) {
#pragma unroll
      for (int m = 0; m < E; ++m) zr[m] = make_float2(0.f, 0.f);
      if constexpr (AM) {
#pragma unroll
        for (int j = 0; j < EH; ++j) am[j] = 0xFFFFFFFFu;
      }
    } else {
      const long long l = line();
      const float2* zline = reinterpret_cast<const float2*>((MB ? bp->zreion : a.zreion) + l * N);
#pragma unroll
      for (int m = 0; m < E; ++m) zr[m] = zline[t0 + F::step(m)];
      if constexpr (AM) {
        const uint16_t* aline = reinterpret_cast<const uint16_t*>((MB ? bp->argmax : a.argmax) + l * N);
#pragma unroll
        for (int j = 0; j < EH; ++j)
          am[j] = (uint32_t)aline[t0 + F::step(2 * j)] | ((uint32_t)aline[t0 + F::step(2 * j + 1)] << 16);
      }
    }
    for (int p = sub; p < np && (SP == 1 || !dead); p += SP, ++i) {
      // step i is the barrier's i-th phase
      const bool late = !mbar_wait(bar, (unsigned)(i & 1), (withheld && i == 0) ? kWithheldPolls : kWaitPolls);
      if (__any_sync(0xffffffffu, late)) {
        if ((threadIdx.x & 31) == 0 && a.err) *reinterpret_cast<volatile int*>(a.err) = 1;  // may be mapped host memory
        dead = true;
        break;
      }
      Cx2 v[E];
#pragma unroll
      for (int m = 0; m < EH; ++m) {
        const ulonglong2 q = stage[m * TH], qp = stage[(EH + m) * TH];
        Cx2 x = {q.x, q.y}, xp = {qp.x, qp.y};
        if (m == 0 && t == 0) x.im = xp.im = 0;
        const Cx2 xe = {add2(x.re, xp.re), sub2(x.im, xp.im)};
        const Cx2 xo = ctwid<true>(Cx2{sub2(x.re, xp.re), add2(x.im, xp.im)}, tw[t + G * m]);
        v[m] = {sub2(xe.re, xo.im), add2(xe.im, xo.re)};
        // Z[H-k] to the lane that owns it (lane G-t, register E-1-m)
        const float2 mr = unpack2(add2(xe.re, xo.im)), mi = unpack2(sub2(xo.re, xe.im));
        v[E - 1 - m].re = pack2(__shfl_sync(0xffffffffu, mr.x, partner, G), __shfl_sync(0xffffffffu, mr.y, partner, G));
        v[E - 1 - m].im = pack2(__shfl_sync(0xffffffffu, mi.x, partner, G), __shfl_sync(0xffffffffu, mi.y, partner, G));
      }
      if (t == 0) {
        // lane 0 received its own mirrors Z[G*(E-m)] one register low
#pragma unroll
        for (int j = E - 1; j > EH; --j) v[j] = v[j - 1];
        const ulonglong2 q = *mid;
        const Cx2 x = {q.x, q.y};
        const Cx2 xe = {add2(x.re, x.re), sub2(x.im, x.im)};
        const Cx2 xo = ctwid<true>(Cx2{sub2(x.re, x.re), add2(x.im, x.im)}, tw[H / 2]);
        v[EH] = {sub2(xe.re, xo.im), add2(xe.im, xo.re)};
      }
      // the staged elements are in registers (the shuffles have used them), and
      // the previous exchange of this warp has been read
      sync();
      if constexpr (SP == 1) {  // every line group has a pair
        p_next = p + 1 < np ? p + 1 : 0;
        lg_next = p + 1 < np ? lg : lg + 1;
      } else {
        p_next += SP;
        seek();
      }
      issue(lg_next, p_next);
      const PairLine<KK::PD> buf{xbuf + lb * LS};
      F::run(v, buf, t, tws, sync);
      const f32x2 as = dup2(MB ? bp->as : a.as);
      const f32x2 cb = MB ? pack2(__ldg(&bp->cb[2 * p]), __ldg(&bp->cb[2 * p + 1])) : pack2(s_cb[2 * p], s_cb[2 * p + 1]);
      const uint32_t rid = (uint32_t)((MB ? bp->r0 : a.r0) + 2 * p);
      f32x2 ss = 0;
#pragma unroll
      for (int m = 0; m < E; ++m) {
        const float2 z0 = unpack2(fma2(as, v[m].re, cb)), z1 = unpack2(fma2(as, v[m].im, cb));
        if constexpr (AM) {
          const int sh = 16 * (m & 1);
          // the pair's larger value (the first radius's of equal ones; fmaxf
          // drops a NaN), then the strict comparison with the running maximum
          auto win = [&](float2 z, float& best, int s) {
            const float zm = fmaxf(z.x, z.y);
            const uint32_t who = (z.x == zm ? rid : rid + 1) << s;
            if (zm > best) am[m >> 1] = (am[m >> 1] & ~(0xFFu << s)) | who;
            best = fmaxf(best, zm);
          };
          win(z0, zr[m].x, sh);
          win(z1, zr[m].y, sh + 8);
        } else {
          // fmaxf: as in k_c2r_zp
          zr[m].x = fmaxf(fmaxf(zr[m].x, z0.x), z0.y);
          zr[m].y = fmaxf(fmaxf(zr[m].y, z1.x), z1.y);
        }
        if constexpr (SIG) ss = fma2(v[m].re, v[m].re, fma2(v[m].im, v[m].im, ss));
      }
      if constexpr (SIG) {
        float2 s = unpack2(ss);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
          s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
        }
        if ((threadIdx.x & 31) == 0) {
          atomicAdd(&red[2 * p], (double)s.x);
          atomicAdd(&red[2 * p + 1], (double)s.y);  // (the filler of an odd sweep: never read)
        }
      }
    }
    const long long l = line();
    float2* zout = reinterpret_cast<float2*>((MB ? bp->zreion_out : a.zreion_out) + l * N);
    uint16_t* aout = AM ? reinterpret_cast<uint16_t*>((MB ? bp->argmax_out : a.argmax_out) + l * N) : nullptr;
    if constexpr (SP == 1) {
      if (!dead) {
#pragma unroll
        for (int m = 0; m < E; ++m) zout[t0 + F::step(m)] = zr[m];
        if constexpr (AM) {
#pragma unroll
          for (int m = 0; m < E; ++m) aout[t0 + F::step(m)] = (uint16_t)(am[m >> 1] >> (16 * (m & 1)));
        }
      }
    } else {
      // merge the warps' maxima through their exchange buffers: warp w writes
      // its values, then merges and stores elements m = w*E/SP ...
      constexpr int LANES = 32, WB = (KK::NL / SP) * LS * 16;  // bytes of a warp's buffers
      static_assert(E * LANES * 10 <= WB, "room for the maxima");
      char* const base = reinterpret_cast<char*>(xbuf);
      auto zb = [&](int w) { return reinterpret_cast<float2*>(base + w * WB) + (threadIdx.x & 31); };
      auto ab = [&](int w) { return reinterpret_cast<uint16_t*>(base + w * WB + E * LANES * 8) + (threadIdx.x & 31); };
      __syncwarp();  // the warp's last exchange has been read
#pragma unroll
      for (int m = 0; m < E; ++m) {
        zb(sub)[m * LANES] = zr[m];
        if constexpr (AM) ab(sub)[m * LANES] = (uint16_t)(am[m >> 1] >> (16 * (m & 1)));
      }
      __syncthreads();
#pragma unroll
      for (int k = 0; k < E / SP; ++k) {
        const int m = sub * (E / SP) + k;
        float2 z = zb(0)[m * LANES];
        uint32_t w0 = AM ? ab(0)[m * LANES] : 0u;
        uint32_t x = w0 & 0xFFu, y = w0 >> 8;
#pragma unroll
        for (int w = 1; w < SP; ++w) {
          const float2 o = zb(w)[m * LANES];
          if constexpr (AM) {
            const uint32_t q = ab(w)[m * LANES], qx = q & 0xFFu, qy = q >> 8;
            if (o.x > z.x || (o.x == z.x && qx < x)) x = qx;
            if (o.y > z.y || (o.y == z.y && qy < y)) y = qy;
          }
          z.x = fmaxf(z.x, o.x);
          z.y = fmaxf(z.y, o.y);
        }
        zout[t0 + F::step(m)] = z;
        if constexpr (AM) aout[t0 + F::step(m)] = (uint16_t)(x | (y << 8));
      }
      __syncthreads();  // the buffers are free again
    }
  }
  pdl_release();
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  if constexpr (SIG) {
    __syncthreads();
    if (threadIdx.x < a.nb) atomicAdd(&a.sig_acc[a.r0 + threadIdx.x], red[threadIdx.x]);
  }
}

}  // namespace prc
