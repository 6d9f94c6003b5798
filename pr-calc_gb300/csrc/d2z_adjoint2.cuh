// d2z_adjoint2.cuh — the adjoint's z pass on pairs of radii (k_adj_z of
// d2z_adjoint.cuh on fft2.cuh): h_R = A dL/dz [argmax == R] along z, its
// half-complex spectrum into the pair slot, and the sums for dL/dB_R.
//
// A warp works alone: a line's dL/dz and argmax are
// read once and kept in registers for all pairs of the sweep, and only the
// transform's exchanges and the upper half of Z go through shared memory: the
// lane that holds Z[k], k < H/2, fetches Z[H-k] and forms X[k] and X[H-k] from
// the two (5.12 -> 4.63 ms for 32 radii at 512^3, 1.20 -> 1.09 for 64 at 256^3,
// against every lane fetching a mirror for each of its values).
#pragma once
#include "d2z_adjoint.cuh"
#include "d2z_lines2.cuh"

namespace prc {

template <int N> struct AK2 {
  using P = typename ACfg<N>::P;
  static constexpr int H = N / 2, E = P::E, G = H / E, THREADS = 128, NG = THREADS / G;
  static constexpr int MINB = E >= 12 ? 3 : 4;  // CTAs per SM (12 or 16 elements a lane: 168 registers)
  static constexpr int PD = E == 12 ? 24 : E;
  static constexpr int pads = H + H / PD;
  static constexpr int LS = G >= 8 ? pads : pads + ((G - pads % 8) % 8 + 8) % 8;
  static constexpr int TW = (PlanRun<P>::TW + 1) & ~1;
  static constexpr size_t bytes = (size_t)(H + TW) * 8 + (size_t)NG * LS * 16;
  static_assert(G >= 2 && G <= 64 && NG * G == THREADS, "whole lines");
};

template <int N>
__global__ void __launch_bounds__(AK2<N>::THREADS, AK2<N>::MINB) k_adj_z2(const __grid_constant__ AdjArgs a) {
  using KK = AK2<N>;
  using P = typename KK::P;
  using L = PairSlot<N>;
  using Buf = PairLine<KK::PD>;
  constexpr int H = N / 2, E = KK::E, G = KK::G, NG = KK::NG;
  constexpr long long NN = (long long)N * N;
  // a lane's positions t + G*m split into a part of the lane and a constant,
  // in the exchange buffer and in the slot
  constexpr bool SPLIT = G % KK::PD == 0, SPLITS = G % L::T == 0;
  static_assert(NN % NG == 0 && (G % L::T == 0 || L::T % G == 0), "whole line groups");
  extern __shared__ float4 smem4[];
  float2* tw = reinterpret_cast<float2*>(smem4);  // e^{2 pi i k/N}, k < H
  float2* tws = tw + H;
  ulonglong2* xbuf = reinterpret_cast<ulonglong2*>(tws + KK::TW);
  load_tw(tw, a.tw, H);
  PlanRun<P>::template fill<2>(tws, a.tw);
  __shared__ double red[kMaxBatch];
  if (threadIdx.x < kMaxBatch) red[threadIdx.x] = 0.0;
  pdl_wait();
  __syncthreads();
  const int g = threadIdx.x / G, t = threadIdx.x % G;
  const Buf buf{xbuf + g * KK::LS};
  const GroupSync<G> sync(g);
  const bool want_db = a.dB != nullptr;
  // sums for dL/dB_R (ACfg): 16 lanes i (own) keep those of radius a of the pairs
  // i and i + 16, the other 16 (up) radius b's
  constexpr bool HALF = E != 16 || G == 32;
  const int lane = threadIdx.x & 31, up = HALF ? lane >> 4 : (lane >> 3) & 1;
  const int own = HALF ? lane & 15 : (lane & 7) | (lane >> 4) * 8;
  double acc0 = 0.0, acc1 = 0.0;
  static_assert(kMaxBatch <= 64, "two pairs a lane");
  const int np = (a.nb + 1) >> 1;
  // A unit is the W consecutive lines (iy) of a warp, which its sums for
  // dL/dB_R run over; units take the planes of a block first, so that the
  // pieces written next to one another are written at the same time.
  constexpr int W = G < 32 ? 32 / G : 1, UPC = NG / W;
  for (int s = blockIdx.x; s < (int)(NN / NG); s += gridDim.x) {
    const int u0 = s * UPC + g / W, xi = u0 % L::XB, q0 = u0 / L::XB;
    const int ix = q0 / (N / W) * L::XB + xi, iy = q0 % (N / W) * W + g % W;
    const int l = ix * N + iy;
    const float2* gl = reinterpret_cast<const float2*>(a.g + (long long)l * N);
    const uchar2* al = reinterpret_cast<const uchar2*>(a.am + (long long)l * N);
    float2 gv[E];
    uchar2 u[E];
#pragma unroll
    for (int m = 0; m < E; ++m) {
      gv[m] = gl[t + G * m];
      u[m] = al[t + G * m];
    }
    float mine = 0.f, mine2 = 0.f;
    for (int p = 0; p < np; ++p) {
      // (no argmax byte is 256: the second half of an odd sweep's last pair)
      const int ra = a.r0 + 2 * p, rb = 2 * p + 1 < a.nb ? ra + 1 : 256;
      Cx2 v[E];
      f32x2 part = 0, odd = 0;
      {
        float2 h0[E], h1[E];  // (radius a, radius b) of cells 2p and 2p + 1
#pragma unroll
        for (int m = 0; m < E; ++m) {
          h0[m] = make_float2(u[m].x == ra ? gv[m].x : 0.f, u[m].x == rb ? gv[m].x : 0.f);
          h1[m] = make_float2(u[m].y == ra ? gv[m].y : 0.f, u[m].y == rb ? gv[m].y : 0.f);
          f32x2& sum = E == 16 && m % 2 ? odd : part;
          sum = add2(sum, add2(pack2(h0[m].x, h0[m].y), pack2(h1[m].x, h1[m].y)));
        }
        adj_layer<E, FirstRadix<P>::v>(v, a.A, h0, h1);
      }
      if (want_db) {
        // each lane keeps one radius's sum and gives the other away
        auto split = [&](f32x2 x, int o) {
          const float2 q = unpack2(x);
          return (up ? q.y : q.x) + __shfl_xor_sync(0xffffffffu, up ? q.x : q.y, o);
        };
        float sum;
        if constexpr (E != 16) {
          sum = split(part, 16);
          sum += __shfl_xor_sync(0xffffffffu, sum, 8);
        } else if constexpr (G == 32) {  // (8 lanes keep the even elements', 8 the odd ones')
          const float e = split(part, 16), f = split(odd, 16);
          sum = (lane & 8 ? f : e) + __shfl_xor_sync(0xffffffffu, lane & 8 ? e : f, 8);
        } else if constexpr (G == 16) {
          sum = split(add2(part, odd), 8);
        } else {
          static_assert(G == 8, "four lines a warp");
          sum = split(part, 8) + split(odd, 8);
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if constexpr (E != 16) {
          if (own == (p & 15)) (p < 16 ? acc0 : acc1) += (double)sum;
        } else {
          const float sum2 = __shfl_xor_sync(0xffffffffu, sum, HALF ? 8 : 16);
          if (own == (p & 15)) {
            mine = sum;
            mine2 = sum2;
          }
          if ((p & 15) == 15 || p == np - 1) {  // in double, for 16 pairs at once
            (p < 16 ? acc0 : acc1) += (double)mine + (double)mine2;
            mine = mine2 = 0.f;
          }
        }
      }
      // Z = DFT_H of (even + i odd cells); X[k] = Ze[k] + e^{-2 pi i k/N} Zo[k]
      PlanRun2x<P>::template run<false, true>(v, buf, t, tws, sync);
      sync();  // the last exchange has been read
      if constexpr (G % KK::PD == 0 || KK::PD % G == 0) {
        const int h = Buf::off(t);
#pragma unroll
        for (int m = E / 2; m < E; ++m) buf.put(h, G * m, v[m]);
      } else {
#pragma unroll
        for (int m = E / 2; m < E; ++m) buf.put_pos(t + G * m, v[m]);
      }
      sync();
      ulonglong2* const slot = reinterpret_cast<ulonglong2*>(a.slots) + (long long)p * a.slot_stride;
      ulonglong2* const line = slot + L::at(ix, iy, 0);
      // positions k = t + G*m from lo on, their mirrors H - k = (t ? G - t : G)
      // + (H - G*(m+1)) from hi on
      ulonglong2* const lo = line + L::along(t);
      ulonglong2* const hi = line + L::along(t ? G - t : G);
      const int hm = Buf::off(t ? G - t : G);
      const f32x2 half = dup2(0.5f), mhalf = dup2(-0.5f);
      auto out = [&](Cx2 ze, Cx2 zo, int k) {
        const float2 w = tw[k];
        const f32x2 wx = dup2(w.x), wy = dup2(w.y);
        return make_ulonglong2(add2(ze.re, fma2(wx, zo.re, mul2(wy, zo.im))),
                               add2(ze.im, fma2(wx, zo.im, neg2(mul2(wy, zo.re)))));
      };
#pragma unroll
      for (int m = 0; m < E / 2; ++m) {
        const int k = t + G * m;
        const Cx2 z = v[m];
        Cx2 q;
        if constexpr (!SPLIT) q = k ? buf.get_pos(H - k) : z;
        else if (m == 0) q = t ? buf.get_pos(H - t) : z;
        else q = buf.get(hm, H - G * (m + 1));
        const f32x2 er = mul2(add2(z.re, q.re), half), orr = mul2(add2(z.im, q.im), half);
        const Cx2 ze = {er, mul2(sub2(z.im, q.im), half)}, zo = {orr, mul2(sub2(z.re, q.re), mhalf)};
        lo[L::along(G * m)] = out(ze, zo, k);
        if (m || t) {
          const Cx2 me = {er, mul2(sub2(q.im, z.im), half)}, mo = {orr, mul2(sub2(q.re, z.re), mhalf)};
          const ulonglong2 x = out(me, mo, H - k);
          if constexpr (SPLITS) hi[L::along(H - G * (m + 1))] = x;
          else line[L::along(H - k)] = x;
        } else {
          // X[H] = Ze[0] - Zo[0], into the transposed scratch plane, and H/2,
          // its own mirror
          slot[NN * (H + 1) + (long long)iy * N + ix] = make_ulonglong2(sub2(ze.re, zo.re), 0ull);
          const Cx2 c = v[E / 2];
          const Cx2 ce = {mul2(add2(c.re, c.re), half), mul2(sub2(c.im, c.im), half)};
          const Cx2 co = {mul2(add2(c.im, c.im), half), mul2(sub2(c.re, c.re), mhalf)};
          line[L::along(H / 2)] = out(ce, co, H / 2);
        }
      }
      sync();  // the mirrors have been read
    }
  }
  pdl_release();
  if (want_db) {
    const int r = 2 * own + up;
    if (r < a.nb) atomicAdd(&red[r], acc0);
    if (r + 32 < a.nb) atomicAdd(&red[r + 32], acc1);
    __syncthreads();
    if (threadIdx.x < a.nb) atomicAdd(&a.dB[a.r0 + threadIdx.x], (double)a.A * red[threadIdx.x]);
  }
}

}  // namespace prc
