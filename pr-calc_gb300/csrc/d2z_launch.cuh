// d2z_launch.cuh — host launchers for one grid size; included by inst_*.cu.
#pragma once
#include "d2z_adjoint2.cuh"
#include "d2z_cols.cuh"
#include "d2z_dispatch.h"
#include "d2z_kernels.cuh"
#include "d2z_lines.cuh"
#include "d2z_lines2.cuh"

namespace prc {

static_assert(kWinVariants == kMaxWinVariants, "window variant table size");

// Launch with the programmatic-dependent-launch attribute; only for kernels
// that call pdl_wait before they touch the previous kernel's data.
template <class... P, class... A>
void launch_pdl(void (*f)(P...), dim3 grid, int threads, size_t bytes, cudaStream_t st, const A&... args) {
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = dim3((unsigned)threads);
  c.dynamicSmemBytes = bytes;
  c.stream = st;
  c.attrs = &at;
  c.numAttrs = 1;
  cudaLaunchKernelEx(&c, f, static_cast<P>(args)...);
}

// Column passes: k_col (one lane per column) where CCfg<N> has a plan, else
// k_tile (shared-memory staged tiles).
template <int N, bool COL = CCfg<N>::on> struct ColLaunch;

template <int N> struct ColLaunch<N, false> {
  using TT = TK<N>;
  static constexpr int THREADS = TT::THREADS, T = TT::T;
  static constexpr size_t TS = (size_t)TT::smem_f2 * sizeof(float2);    // one tile
  static constexpr size_t TS2 = (size_t)TT::smem2_f2 * sizeof(float2);  // two tiles (TM_WIN)
  template <int MODE> static void* fn() { return reinterpret_cast<void*>(&k_tile<N, MODE>); }
  static void* faithful_fn() { return reinterpret_cast<void*>(&k_tile<N, TM_WIN>); }
  static constexpr size_t FS = TS2;
  static constexpr int FTHREADS = THREADS;
  static size_t bytes(int mode) { return mode == TM_WIN ? TS2 : TS; }
  static int threads(int) { return THREADS; }
  static constexpr int T_ACC = T;
  // one window variant: the staged tile kernel
  static int win(int v, void** f = nullptr, int* thr = nullptr, size_t* by = nullptr, int* tw = nullptr) {
    if (v == 0) {
      if (f) *f = reinterpret_cast<void*>(&k_tile<N, TM_WIN>);
      if (thr) *thr = THREADS;
      if (by) *by = TS2;
      if (tw) *tw = T;
    }
    return 1;
  }
  static constexpr bool GROUPED = false;
  static void launch(int mode, dim3 grid, cudaStream_t st, const TileArgs& a) {
    switch (mode) {
      case TM_FWD: k_tile<N, TM_FWD><<<grid, THREADS, TS, st>>>(a); break;
      case TM_INV: k_tile<N, TM_INV><<<grid, THREADS, TS, st>>>(a); break;
      case TM_WIN: k_tile<N, TM_WIN><<<grid, THREADS, TS2, st>>>(a); break;
      default: k_tile<N, TM_ACC><<<grid, THREADS, TS, st>>>(a); break;
    }
  }
};

template <int N> struct ColLaunch<N, true> {
  using CC = typename ColK<N, TM_INV, 0>::type;
  using CA = typename ColK<N, TM_ACC, 0>::type;
  static constexpr int THREADS = CC::THREADS, T = CC::T;
  static constexpr int T_ACC = CA::T;
  static constexpr size_t CS = (size_t)CC::smem_f2 * sizeof(float2);
  static constexpr size_t CSA = (size_t)CA::smem_f2 * sizeof(float2);
  // window-pass variant v (when compiled for this N)
  template <int V> struct Win {
    static constexpr bool on = WinVar<N, V>::on;
    using K = typename ColK<N, TM_WIN, V>::type;
  };
  template <int MODE> static void* fn() { return reinterpret_cast<void*>(&k_col<N, MODE>); }
  static size_t bytes(int mode) { return mode == TM_ACC ? CSA : CS; }
  static int threads(int mode) { return mode == TM_ACC ? CA::THREADS : THREADS; }
  template <int V> static void win_info(int v, int* n, void** f, int* thr, size_t* by, int* tw) {
    if constexpr (V < kWinVariants) {
      if constexpr (Win<V>::on) {
        if (v == V) {
          *f = reinterpret_cast<void*>(&k_col<N, TM_WIN, V>);
          *thr = Win<V>::K::THREADS;
          *by = (size_t)Win<V>::K::smem_f2 * sizeof(float2);
          *tw = Win<V>::K::T;
        }
        *n = V + 1;
      }
      win_info<V + 1>(v, n, f, thr, by, tw);
    }
  }
  // number of window variants and, for variant v, its kernel, threads, bytes, tile width
  static int win(int v, void** f = nullptr, int* thr = nullptr, size_t* by = nullptr, int* tw = nullptr) {
    int n = 0, t0 = 0, w0 = 0;
    void* f0 = nullptr;
    size_t b0 = 0;
    win_info<0>(v, &n, f ? f : &f0, thr ? thr : &t0, by ? by : &b0, tw ? tw : &w0);
    return n;
  }
  using WF = typename ColK<N, TM_WIN, kWinFaithful>::type;
  static void* faithful_fn() { return reinterpret_cast<void*>(&k_col<N, TM_WIN, kWinFaithful>); }
  static constexpr size_t FS = (size_t)WF::smem_f2 * sizeof(float2);
  static constexpr int FTHREADS = WF::THREADS;
  template <int V> static void launch_win(int v, dim3 grid, cudaStream_t st, const TileArgs& a) {
    if (V == 0 && a.faithful) {
      k_col<N, TM_WIN, kWinFaithful><<<grid, FTHREADS, FS, st>>>(a);
      return;
    }
    if constexpr (V < kWinVariants) {
      if constexpr (Win<V>::on) {
        if (v == V) {
          k_col<N, TM_WIN, V><<<grid, Win<V>::K::THREADS, (size_t)Win<V>::K::smem_f2 * sizeof(float2), st>>>(a);
          return;
        }
      }
      launch_win<V + 1>(v, grid, st, a);
    }
  }
  static void launch(int mode, dim3 grid, cudaStream_t st, const TileArgs& a) {
    switch (mode) {
      case TM_FWD: launch_pdl(&k_col<N, TM_FWD>, grid, THREADS, CS, st, a); break;
      case TM_INV: k_col<N, TM_INV><<<grid, THREADS, CS, st>>>(a); break;
      case TM_WIN: launch_win<0>(a.win_var, grid, st, a); break;
      default: k_col<N, TM_ACC><<<grid, CA::THREADS, CSA, st>>>(a); break;
    }
  }
  // grouped launches (several boxes of this size per launch; window variant 0)
  static constexpr bool GROUPED = N <= 256 && PCfg<N>::on;
  using W0 = typename Win<0>::K;
  static constexpr size_t WS0 = (size_t)W0::smem_f2 * sizeof(float2);
  template <int MODE> static void* fn_mb() { return reinterpret_cast<void*>(&k_col<N, MODE, 0, true>); }
  static void launch_mb(int mode, dim3 grid, cudaStream_t st, const TileArgs& a) {
    if constexpr (GROUPED) {
      switch (mode) {
        case TM_FWD: launch_pdl(&k_col<N, TM_FWD, 0, true>, grid, THREADS, CS, st, a); break;
        case TM_INV: k_col<N, TM_INV, 0, true><<<grid, THREADS, CS, st>>>(a); break;
        default: k_col<N, TM_WIN, 0, true><<<grid, W0::THREADS, WS0, st>>>(a); break;
      }
    }
  }
};

// Inverse z pass: k_c2r_zp (mirror pairs in one lane) where PCfg<N> has a
// plan, else k_c2r_z.
template <int N, bool PAIR = PCfg<N>::on> struct C2rLaunch {
  static constexpr int THREADS = LK<N>::THREADS, NG = LK<N>::NG;
  static constexpr size_t BYTES = (size_t)LK<N>::smem_f2 * sizeof(float2);
  static constexpr int NFN = 1;
  static void* fn(int) { return reinterpret_cast<void*>(&k_c2r_z<N>); }
  static void launch(int grid, cudaStream_t st, const SweepArgs& a) { k_c2r_z<N><<<grid, THREADS, BYTES, st>>>(a); }
};
template <int N> struct C2rLaunch<N, true> {
  static constexpr int THREADS = PK<N>::THREADS, NG = PK<N>::NG;
  static constexpr size_t BYTES = (size_t)PK<N>::smem_f2 * sizeof(float2);
  template <bool AM, bool SIG> static void* f() { return reinterpret_cast<void*>(&k_c2r_zp<N, AM, SIG>); }
  static constexpr int NFN = 4;
  static void* fn(int i) { return i == 0 ? f<false, false>() : i == 1 ? f<true, false>() : i == 2 ? f<false, true>() : f<true, true>(); }
  static void launch(int grid, cudaStream_t st, const SweepArgs& a) {
    if (a.sig_acc) {
      if (a.argmax) k_c2r_zp<N, true, true><<<grid, THREADS, BYTES, st>>>(a);
      else k_c2r_zp<N, false, true><<<grid, THREADS, BYTES, st>>>(a);
    } else {
      if (a.argmax) k_c2r_zp<N, true, false><<<grid, THREADS, BYTES, st>>>(a);
      else k_c2r_zp<N, false, false><<<grid, THREADS, BYTES, st>>>(a);
    }
  }
  // grouped: a.argmax != null means every box of the launch records its argmax
  template <bool AM> static void* f_mb() { return reinterpret_cast<void*>(&k_c2r_zp<N, AM, false, true>); }
  static void launch_mb(int grid, cudaStream_t st, const SweepArgs& a) {
    if (a.argmax) k_c2r_zp<N, true, false, true><<<grid, THREADS, BYTES, st>>>(a);
    else k_c2r_zp<N, false, false, true><<<grid, THREADS, BYTES, st>>>(a);
  }
};

// The sweep's passes on pairs of radii (grids with both a column and a z-line
// plan): window + inverse x, inverse y, inverse z (MB: grouped launches), and
// the adjoint's z, forward y and accumulating x passes.
template <int N, bool ON = C2Cfg<N>::on> struct PairLaunch {
  static constexpr bool on = false;
};
template <int N> struct PairLaunch<N, true> {
  static constexpr bool on = true;
  using KW = CK2<N, TM_WIN>;
  using KI = CK2<N, TM_INV>;
  using KZ = PK2<N>;
  using KZM = PK2<N, true>;
  template <bool MB> static void* win_fn() { return reinterpret_cast<void*>(&k_col2<N, TM_WIN, MB>); }
  using KF = CK2<N, TM_FWD>;
  using KA = CK2<N, TM_ACC>;
  using KS = AK2<N>;
  static void* fwd_fn() { return reinterpret_cast<void*>(&k_col2<N, TM_FWD>); }
  static void* acc_fn() { return reinterpret_cast<void*>(&k_col2<N, TM_ACC>); }
  static void* adj_fn() { return reinterpret_cast<void*>(&k_adj_z2<N>); }
  static void tile_adj(int mode, dim3 grid, cudaStream_t st, const TileArgs& a) {
    if (mode == TM_FWD) launch_pdl(&k_col2<N, TM_FWD>, grid, KF::THREADS, KF::bytes, st, a);
    else launch_pdl(&k_col2<N, TM_ACC>, grid, KA::THREADS, KA::bytes, st, a);
  }
  static void adj_z(int grid, cudaStream_t st, const AdjArgs& a) {
    launch_pdl(&k_adj_z2<N>, grid, KS::THREADS, KS::bytes, st, a);
  }
  template <bool MB> static void* inv_fn() { return reinterpret_cast<void*>(&k_col2<N, TM_INV, MB>); }
  template <bool AM, bool SIG, bool MB> static void* z_fn() { return reinterpret_cast<void*>(&k_c2r_zp2<N, AM, SIG, MB>); }
  template <bool MB> static void tile(int mode, dim3 grid, cudaStream_t st, const TileArgs& a) {
    if (mode == TM_WIN) launch_pdl(&k_col2<N, TM_WIN, MB>, grid, KW::THREADS, KW::bytes, st, a);
    else launch_pdl(&k_col2<N, TM_INV, MB>, grid, KI::THREADS, KI::bytes, st, a);
  }
  static void c2r(int grid, cudaStream_t st, const SweepArgs& a) {
    if (a.sig_acc) {
      if (a.argmax) launch_pdl(&k_c2r_zp2<N, true, true>, grid, KZ::THREADS, KZ::bytes, st, a);
      else launch_pdl(&k_c2r_zp2<N, false, true>, grid, KZ::THREADS, KZ::bytes, st, a);
    } else {
      if (a.argmax) launch_pdl(&k_c2r_zp2<N, true, false>, grid, KZ::THREADS, KZ::bytes, st, a);
      else launch_pdl(&k_c2r_zp2<N, false, false>, grid, KZ::THREADS, KZ::bytes, st, a);
    }
  }
  static void c2r_mb(int grid, cudaStream_t st, const SweepArgs& a) {
    if (a.argmax) launch_pdl(&k_c2r_zp2<N, true, false, true>, grid, KZM::THREADS, KZM::bytes, st, a);
    else launch_pdl(&k_c2r_zp2<N, false, false, true>, grid, KZM::THREADS, KZM::bytes, st, a);
  }
};

template <int N> struct Launchers {
  using PL = PairLaunch<N>;
  using CL = ColLaunch<N>;
  using CR = C2rLaunch<N>;
  using LL = LK<N>;
  static constexpr size_t LS = (size_t)LL::smem_f2 * sizeof(float2);
  static constexpr size_t AS = (size_t)ALK<N>::smem_f2 * sizeof(float2);

  template <class F> static cudaError_t smem(F fn, size_t bytes) {
    return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  }
  template <class F> static cudaError_t occ(int* dst, F fn, int threads, size_t bytes) {
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(dst, fn, threads, bytes);
    if (*dst < 1) *dst = 1;
    return e;
  }
  static cudaError_t init(KernelSet* ks) {
    void* tf = CL::template fn<TM_FWD>();
    void* ti = CL::template fn<TM_INV>();
    void* ta = CL::template fn<TM_ACC>();
    cudaError_t e;
    if ((e = smem(tf, CL::bytes(TM_FWD))) != cudaSuccess) return e;
    if ((e = smem(ti, CL::bytes(TM_INV))) != cudaSuccess) return e;
    if ((e = smem(ta, CL::bytes(TM_ACC))) != cudaSuccess) return e;
    // window-pass variants
    ks->n_win_var = CL::win(0);
    for (int v = 0; v < ks->n_win_var; ++v) {
      void* f = nullptr;
      int thr = 0, tw = 0;
      size_t by = 0;
      CL::win(v, &f, &thr, &by, &tw);
      if ((e = smem(f, by)) != cudaSuccess) return e;
      if ((e = occ(&ks->occ_winv[v], f, thr, by)) != cudaSuccess) return e;
      ks->tile_w_winv[v] = tw;
    }
    ks->occ_tile_win = ks->occ_winv[0];
    ks->tile_w_win = ks->tile_w_winv[0];
    if constexpr (PL::on) {
      void* w = PL::template win_fn<false>();
      void* v = PL::template inv_fn<false>();
      void* z[4] = {PL::template z_fn<false, false, false>(), PL::template z_fn<true, false, false>(),
                    PL::template z_fn<false, true, false>(), PL::template z_fn<true, true, false>()};
      if ((e = smem(w, PL::KW::bytes)) != cudaSuccess) return e;
      if ((e = smem(v, PL::KI::bytes)) != cudaSuccess) return e;
      for (void* f : z)
        if ((e = smem(f, PL::KZ::bytes)) != cudaSuccess) return e;
      if ((e = smem(PL::fwd_fn(), PL::KF::bytes)) != cudaSuccess) return e;
      if ((e = smem(PL::acc_fn(), PL::KA::bytes)) != cudaSuccess) return e;
      if ((e = smem(PL::adj_fn(), PL::KS::bytes)) != cudaSuccess) return e;
      if ((e = occ(&ks->occ_pair_fwd, PL::fwd_fn(), PL::KF::THREADS, PL::KF::bytes)) != cudaSuccess) return e;
      if ((e = occ(&ks->occ_pair_acc, PL::acc_fn(), PL::KA::THREADS, PL::KA::bytes)) != cudaSuccess) return e;
      if ((e = occ(&ks->occ_pair_adj, PL::adj_fn(), PL::KS::THREADS, PL::KS::bytes)) != cudaSuccess) return e;
      if ((e = occ(&ks->occ_pair_win, w, PL::KW::THREADS, PL::KW::bytes)) != cudaSuccess) return e;
      if ((e = occ(&ks->occ_pair_inv, v, PL::KI::THREADS, PL::KI::bytes)) != cudaSuccess) return e;
      if ((e = occ(&ks->occ_pair_c2r, z[1], PL::KZ::THREADS, PL::KZ::bytes)) != cudaSuccess) return e;
    }
    if constexpr (CL::GROUPED) {
      KernelSet::Grouped &one = ks->mb[0], &two = ks->mb[1];
      void* fm = CL::template fn_mb<TM_FWD>();
      void* i1 = CL::template fn_mb<TM_INV>();
      void* w1 = CL::template fn_mb<TM_WIN>();
      void* i2 = PL::template inv_fn<true>();
      void* w2 = PL::template win_fn<true>();
      void* z1[2] = {CR::template f_mb<false>(), CR::template f_mb<true>()};
      void* z2[2] = {PL::template z_fn<false, false, true>(), PL::template z_fn<true, false, true>()};
      if ((e = smem(fm, CL::CS)) != cudaSuccess) return e;
      if ((e = smem(i1, CL::CS)) != cudaSuccess) return e;
      if ((e = smem(w1, CL::WS0)) != cudaSuccess) return e;
      if ((e = smem(i2, PL::KI::bytes)) != cudaSuccess) return e;
      if ((e = smem(w2, PL::KW::bytes)) != cudaSuccess) return e;
      for (int k = 0; k < 2; ++k) {
        if ((e = smem(z1[k], CR::BYTES)) != cudaSuccess) return e;
        if ((e = smem(z2[k], PL::KZM::bytes)) != cudaSuccess) return e;
      }
      if ((e = smem(&k_r2c_z<N, true>, LS)) != cudaSuccess) return e;
      if ((e = occ(&ks->occ_mb_tile, fm, CL::THREADS, CL::CS)) != cudaSuccess) return e;
      if ((e = occ(&one.occ_inv, i1, CL::THREADS, CL::CS)) != cudaSuccess) return e;
      if ((e = occ(&one.occ_win, w1, CL::W0::THREADS, CL::WS0)) != cudaSuccess) return e;
      if ((e = occ(&one.occ_c2r, z1[1], CR::THREADS, CR::BYTES)) != cudaSuccess) return e;
      if ((e = occ(&two.occ_inv, i2, PL::KI::THREADS, PL::KI::bytes)) != cudaSuccess) return e;
      if ((e = occ(&two.occ_win, w2, PL::KW::THREADS, PL::KW::bytes)) != cudaSuccess) return e;
      if ((e = occ(&two.occ_c2r, z2[1], PL::KZM::THREADS, PL::KZM::bytes)) != cudaSuccess) return e;
      if ((e = occ(&ks->occ_mb_r2c, &k_r2c_z<N, true>, LL::THREADS, LS)) != cudaSuccess) return e;
    }
    if ((e = smem(CL::faithful_fn(), CL::FS)) != cudaSuccess) return e;
    if ((e = occ(&ks->occ_win_faithful, CL::faithful_fn(), CL::FTHREADS, CL::FS)) != cudaSuccess) return e;
    if ((e = smem(&k_r2c_z<N>, LS)) != cudaSuccess) return e;
    for (int i = 0; i < CR::NFN; ++i)
      if ((e = smem(CR::fn(i), CR::BYTES)) != cudaSuccess) return e;
    if ((e = smem(&k_adj_z<N>, AS)) != cudaSuccess) return e;
    if ((e = smem(&k_c2r_plain<N>, LS)) != cudaSuccess) return e;
    if ((e = occ(&ks->occ_tile, ti, CL::THREADS, CL::bytes(TM_INV))) != cudaSuccess) return e;
    if ((e = occ(&ks->occ_tile_acc, ta, CL::threads(TM_ACC), CL::bytes(TM_ACC))) != cudaSuccess) return e;
    if ((e = occ(&ks->occ_r2c, &k_r2c_z<N>, LL::THREADS, LS)) != cudaSuccess) return e;
    if ((e = occ(&ks->occ_c2r, CR::fn(0), CR::THREADS, CR::BYTES)) != cudaSuccess) return e;
    if ((e = occ(&ks->occ_c2r_plain, &k_c2r_plain<N>, LL::THREADS, LS)) != cudaSuccess) return e;
    if ((e = occ(&ks->occ_adj_z, &k_adj_z<N>, ALK<N>::THREADS, AS)) != cudaSuccess) return e;
    return cudaSuccess;
  }
  static void r2c_z(const KernelSet&, int grid, cudaStream_t st, const float* d, float dinit, float2* S,
                    float2* Qt, const float2* tw) {
    launch_pdl(&k_r2c_z<N>, grid, LL::THREADS, LS, st, d, dinit, S, Qt, tw, (const BoxR2c*)nullptr, 0);
  }
  static void r2c_z_mb(const KernelSet&, int grid, cudaStream_t st, const BoxR2c* box, int nbox, const float2* tw) {
    if constexpr (CL::GROUPED) launch_pdl(&k_r2c_z<N, true>, grid, LL::THREADS, LS, st, (const float*)nullptr, 1.f, (float2*)nullptr, (float2*)nullptr,
                                               tw, box, nbox);
  }
  static void tile_mb(const KernelSet&, dim3 grid, cudaStream_t st, const TileArgs& a) {
    if constexpr (CL::GROUPED) CL::launch_mb(TM_FWD, grid, st, a);
  }
  template <bool PAIR> static void sweep_mb(const KernelSet&, int mode, dim3 grid, cudaStream_t st, const TileArgs& a) {
    if constexpr (CL::GROUPED) {
      if constexpr (PAIR) PL::template tile<true>(mode, grid, st, a);
      else CL::launch_mb(mode, grid, st, a);
    }
  }
  template <bool PAIR> static void c2r_z_mb(const KernelSet&, int grid, cudaStream_t st, const SweepArgs& a) {
    if constexpr (CL::GROUPED) {
      if constexpr (PAIR) PL::c2r_mb(grid, st, a);
      else CR::launch_mb(grid, st, a);
    }
  }
  static void pair_tile(const KernelSet&, int mode, dim3 grid, cudaStream_t st, const TileArgs& a) {
    if constexpr (PL::on) {
      if (mode == TM_FWD || mode == TM_ACC) PL::tile_adj(mode, grid, st, a);
      else PL::template tile<false>(mode, grid, st, a);
    }
  }
  static void pair_adj_z(const KernelSet&, int grid, cudaStream_t st, const AdjArgs& a) {
    if constexpr (PL::on) PL::adj_z(grid, st, a);
  }
  static void pair_c2r(const KernelSet&, int grid, cudaStream_t st, const SweepArgs& a) {
    if constexpr (PL::on) PL::c2r(grid, st, a);
  }
  static void tile(const KernelSet&, int mode, dim3 grid, cudaStream_t st, const TileArgs& a) {
    CL::launch(mode, grid, st, a);
  }
  static void c2r_z(const KernelSet&, int grid, cudaStream_t st, const SweepArgs& a) { CR::launch(grid, st, a); }
  static void adj_z(const KernelSet&, int grid, cudaStream_t st, const AdjArgs& a) {
    k_adj_z<N><<<grid, ALK<N>::THREADS, AS, st>>>(a);
  }
  static void c2r_plain(const KernelSet&, int grid, cudaStream_t st, const AdjArgs& a) {
    k_c2r_plain<N><<<grid, LL::THREADS, LS, st>>>(a);
  }
  static KernelSet make() {
    KernelSet ks{};
    ks.N = N;
    ks.tile_threads = CL::THREADS;
    ks.tile_w = CL::T;
    ks.tile_w_acc = CL::T_ACC;
    ks.n_win_var = CL::win(0);
    ks.line_threads = LL::THREADS;
    ks.line_groups = LL::NG;
    ks.c2r_lines = CR::NG;
    ks.tile_smem = CL::bytes(TM_INV);
    ks.line_smem = LS;
    ks.init = &init;
    ks.r2c_z = &r2c_z;
    ks.tile = &tile;
    ks.c2r_z = &c2r_z;
    ks.adj_z = &adj_z;
    ks.c2r_plain = &c2r_plain;
    if constexpr (PL::on) {
      ks.pair = 1;
      ks.pair_xb = PairSlot<N>::XB;
      ks.pair_tile_w = PL::KI::T;
      ks.pair_tile_w_win = PL::KW::T;
      ks.pair_lines = PL::KZ::NG;
      ks.pair_adj_lines = PL::KS::NG;
      ks.pair_adj_z = &pair_adj_z;
      ks.pair_tile = &pair_tile;
      ks.pair_c2r = &pair_c2r;
    }
    if constexpr (CL::GROUPED) {
      ks.grouped = 1;
      ks.mb[0] = {CL::W0::T, CL::T, CR::NG, 0, 0, 0, &sweep_mb<false>, &c2r_z_mb<false>};
      ks.mb[1] = {PL::KW::T, PL::KI::T, PL::KZM::NG, 0, 0, 0, &sweep_mb<true>, &c2r_z_mb<true>};
      ks.r2c_z_mb = &r2c_z_mb;
      ks.tile_mb = &tile_mb;
    }
    return ks;
  }
};

}  // namespace prc

#define PRC_INSTANTIATE(NV)                      \
  namespace prc {                                \
  const KernelSet* kernel_set_##NV() {           \
    static KernelSet ks = Launchers<NV>::make(); \
    return &ks;                                  \
  }                                              \
  }
