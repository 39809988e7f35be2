// Definitions of the matvec launchers; included only by the two translation
// units that instantiate them (matvec_f32.cu, matvec_f64.cu).
#pragma once
#include <cstring>

#include "matvec_fused.cuh"
#include "matvec_launch.cuh"
#include "matvec_zpack.cuh"

namespace marie {

// Launches a pass as a programmatic dependent of the kernel before it (the
// passes wait before they read anything that kernel writes).
template <typename... P, typename... A>
static cudaError_t launch_pass(void (*kern)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, P(args)...);
}

template <typename T> struct MatvecImpl {
  using V = cplx<T>;

  template <int NL, int THR, typename IO>
  static cudaError_t xfwd_nt(const IO* J, long long js, const int* inv, Prologue pro, V* A, long long as,
                            const Dims& d, const V* tw, int nrhs, cudaStream_t st) {
    if constexpr (sizeof(T) == 4) {
      using X = XRow<NL, THR>;
      cudaError_t e = opt_in_smem(k_xfwd_rows<NL, THR, IO>, X::bytes);
      if (e != cudaSuccess) return e;
      dim3 grid((d.M * d.N * 3 + X::S - 1) / X::S, nrhs);
      return launch_pass(k_xfwd_rows<NL, THR, IO>, grid, RowCfg<V, NL, THR>::THREADS, X::bytes, st, J, js, inv, pro, A,
                         as, d, tw);
    } else {
      constexpr int S = RowCfg<cplx<T>, NL, THR>::S;
      const size_t smem = (size_t)(NL + NL * (S + 1)) * sizeof(V);
      cudaError_t e = opt_in_smem(k_xfwd<T, NL, THR, IO>, smem);
      if (e != cudaSuccess) return e;
      const int rows = d.M * d.N * 3;
      dim3 grid((rows + S - 1) / S, nrhs);
      return launch_pass(k_xfwd<T, NL, THR, IO>, grid, RowCfg<cplx<T>, NL, THR>::THREADS, smem, st, J, js, inv, pro, A, as,
                         d, tw);
    }
  }
  template <int NL, int THR, typename IO>
  static cudaError_t xinv_nt(const V* A, long long as, const IO* J, long long js, const int* inv, Epilogue ep,
                            IO* out, long long os, const Dims& d, const V* tw, int nrhs, cudaStream_t st) {
    if constexpr (sizeof(T) == 4) {
      using X = XRow<NL, THR>;
      cudaError_t e = opt_in_smem(k_xinv_rows<NL, THR, IO>, X::bytes);
      if (e != cudaSuccess) return e;
      dim3 grid((d.M * d.N * 3 + X::S - 1) / X::S, nrhs);
      return launch_pass(k_xinv_rows<NL, THR, IO>, grid, RowCfg<V, NL, THR>::THREADS, X::bytes, st, A, as, J, js, inv,
                         ep, out, os, d, tw);
    } else {
      constexpr int S = RowCfg<cplx<T>, NL, THR>::S;
      const size_t smem = (size_t)(NL + NL * (S + 1)) * sizeof(V);
      cudaError_t e = opt_in_smem(k_xinv<T, NL, THR, IO>, smem);
      if (e != cudaSuccess) return e;
      const int rows = d.M * d.N * 3;
      dim3 grid((rows + S - 1) / S, nrhs);
      return launch_pass(k_xinv<T, NL, THR, IO>, grid, RowCfg<cplx<T>, NL, THR>::THREADS, smem, st, A, as, J, js, inv, ep,
                         out, os, d, tw);
    }
  }
  // An x pass of 256-thread CTAs is taken when it fills the chip four times over;
  // below that, CTAs of a quarter the rows spread the work over all SMs.
  // First and last pass of a 40^3 FP64 grid 46 -> 32 and 51 -> 37 us; of a 12 x 8
  // x 20 grid, two CTAs before, 34 -> 15 and 47 -> 18 us.
  template <int NL> static bool many_rows(const Dims& d, int nrhs) {
    constexpr int S = RowCfg<cplx<T>, NL>::S;
    return ((long long)d.M * d.N * 3 + S - 1) / S * nrhs >= 4LL * sm_count();
  }
  template <int NL, typename IO>
  static cudaError_t xfwd_n(const IO* J, long long js, const int* inv, Prologue pro, V* A, long long as,
                            const Dims& d, const V* tw, int nrhs, cudaStream_t st) {
    return many_rows<NL>(d, nrhs) ? xfwd_nt<NL, 256, IO>(J, js, inv, pro, A, as, d, tw, nrhs, st)
                                  : xfwd_nt<NL, 64, IO>(J, js, inv, pro, A, as, d, tw, nrhs, st);
  }
  template <int NL, typename IO>
  static cudaError_t xinv_n(const V* A, long long as, const IO* J, long long js, const int* inv, Epilogue ep,
                            IO* out, long long os, const Dims& d, const V* tw, int nrhs, cudaStream_t st) {
    return many_rows<NL>(d, nrhs) ? xinv_nt<NL, 256, IO>(A, as, J, js, inv, ep, out, os, d, tw, nrhs, st)
                                  : xinv_nt<NL, 64, IO>(A, as, J, js, inv, ep, out, os, d, tw, nrhs, st);
  }
  template <int NC, bool INV>
  static cudaError_t cols_n(const V* in, long long in_w, long long in_rhs, int n_in, V* out, long long out_w,
                            long long out_rhs, int n_out, int Lp, int nw, const V* tw, int nrhs, cudaStream_t st,
                            const int* stop, int step) {
    constexpr int S = ColS<T>::S;
    const size_t smem = (size_t)(NC + NC * (S + 1)) * sizeof(V);
    cudaError_t e = opt_in_smem(k_cols<T, NC, INV>, smem);
    if (e != cudaSuccess) return e;
    dim3 grid((Lp + S - 1) / S, nw, nrhs);
    return launch_pass(k_cols<T, NC, INV>, grid, S * FFT<V, NC, INV>::T, smem, st, in, in_w, in_rhs, n_in, out, out_w,
                       out_rhs, n_out, Lp, tw, stop, step);
  }
  template <int NZ, int KIND>
  static cudaError_t zmul_nk(V* B, long long bs, const V* fN, int oct, const Dims& d, const V* tw, int nrhs,
                             cudaStream_t st) {
    using ZC = ZS<T, NZ, KIND>;
    constexpr int S = ZC::S;  // S columns, 3 component buffers, operator tile
    cudaError_t e = opt_in_smem(k_zmul<T, NZ, KIND>, ZC::bytes);
    if (e != cudaSuccess) return e;
    return launch_pass(k_zmul<T, NZ, KIND>, dim3((d.Lp + S - 1) / S, d.Mp, nrhs), ZC::THREADS, ZC::bytes, st, B, bs,
                       fN, oct, d, tw);
  }
  // the z pass on column pairs (FP32, a tile by bulk copy)
  template <int NZ>
  static cudaError_t zmul_pairs(float2* B, long long bs, const Dims& d, const float2* tw, int nrhs, cudaStream_t st,
                                const ZTile* zt) {
    using Z = ZP<NZ>;
    const int tma = take_tile_timeout_injection() ? 2 : 1;  // 2: a test, a wait that runs out
    cudaError_t e = opt_in_smem(k_zmul_pairs<NZ>, Z::bytes);
    if (e != cudaSuccess) return e;
    return launch_pass(k_zmul_pairs<NZ>, dim3(d.Lp / Z::S, d.Mp, nrhs), Z::THREADS, Z::bytes, st, B, bs, d, tw, zt->map,
                       tma, zt->err);
  }
  template <int NZ>
  static cudaError_t zmul_n(V* B, long long bs, const V* fN, int oct, const Dims& d, const V* tw, int nrhs,
                            cudaStream_t st, int kind, const ZTile* zt) {
    if (kind == 1) return zmul_nk<NZ, 1>(B, bs, fN, oct, d, tw, nrhs, st);
    if constexpr (sizeof(T) == 4 && ZP<NZ>::ok)
      if (oct && zt && zt->ok) return zmul_pairs<NZ>(B, bs, d, tw, nrhs, st, zt);
    return zmul_nk<NZ, 0>(B, bs, fN, oct, d, tw, nrhs, st);
  }

  template <typename IO>
  static cudaError_t xfwd(const IO* J, long long js, const int* inv, Prologue pro, V* A, long long as,
                          const Dims& d, const V* tw, int nrhs, cudaStream_t st) {
    switch (d.Lp) {
#define MARIE_CASE(n_) case n_: return xfwd_n<n_, IO>(J, js, inv, pro, A, as, d, tw, nrhs, st);
      MARIE_FFT_LENGTHS(MARIE_CASE)
#undef MARIE_CASE
    }
    return cudaErrorInvalidValue;
  }
  template <typename IO>
  static cudaError_t xinv(const V* A, long long as, const IO* J, long long js, const int* inv, Epilogue ep,
                          IO* out, long long os, const Dims& d, const V* tw, int nrhs, cudaStream_t st) {
    switch (d.Lp) {
#define MARIE_CASE(n_) case n_: return xinv_n<n_, IO>(A, as, J, js, inv, ep, out, os, d, tw, nrhs, st);
      MARIE_FFT_LENGTHS(MARIE_CASE)
#undef MARIE_CASE
    }
    return cudaErrorInvalidValue;
  }
  static cudaError_t cols(bool inv, int NC, const V* in, long long in_w, long long in_rhs, int n_in, V* out,
                          long long out_w, long long out_rhs, int n_out, int Lp, int nw, const V* tw, int nrhs,
                          cudaStream_t st, const int* stop, int step) {
    if (inv) {
      switch (NC) {
#define MARIE_CASE(n_) \
  case n_: return cols_n<n_, true>(in, in_w, in_rhs, n_in, out, out_w, out_rhs, n_out, Lp, nw, tw, nrhs, st, stop, step);
        MARIE_FFT_LENGTHS(MARIE_CASE)
#undef MARIE_CASE
      }
    } else {
        switch (NC) {
#define MARIE_CASE(n_) \
  case n_: return cols_n<n_, false>(in, in_w, in_rhs, n_in, out, out_w, out_rhs, n_out, Lp, nw, tw, nrhs, st, stop, step);
          MARIE_FFT_LENGTHS(MARIE_CASE)
#undef MARIE_CASE
        }
    }
    return cudaErrorInvalidValue;
  }
  static cudaError_t zmul(V* B, long long bs, const V* fN, int oct, const Dims& d, const V* tw, int nrhs,
                          cudaStream_t st, int kind, const ZTile* zt) {
    switch (d.Np) {
#define MARIE_CASE(n_) case n_: return zmul_n<n_>(B, bs, fN, oct, d, tw, nrhs, st, kind, zt);
      MARIE_FFT_LENGTHS(MARIE_CASE)
#undef MARIE_CASE
    }
    return cudaErrorInvalidValue;
  }
};


// (2L, 2M, cluster size) of the grids with fused x+y passes.  Only the smallest
// of them gains (64 x 64: three launches of 37.6 us against five of 40.5 us in
// all); the separate passes are faster from 96 x 96 on (96^3 grid: 318 us
// against 429 us; 128^3 with every voxel a DOF 593 against 607 us).
#define MARIE_FUSED_PAIRS(X) X(64, 64, 2)

template <typename T> struct FusedImpl {
  using V = cplx<T>;
  template <int NL, int NM, int CS> static constexpr bool usable() {
    using C = XYCfg<T, NL, NM, CS>;
    // FP64 is FP64-pipe bound on GB300: the fused kernels' lower occupancy costs
    // more than the saved spectrum traffic, so FP64 keeps the five-pass path.
    return sizeof(T) == 4 && C::ok && C::fwd_smem <= 220 * 1024 && C::inv_smem <= 220 * 1024;
  }
  template <typename K>
  static cudaError_t launch(K kern, int CS, int nblocks, int nrhs, size_t smem, cudaStream_t st, void** args) {
    cudaError_t e = opt_in_smem(kern, smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nblocks, nrhs, 1);
    cfg.blockDim = dim3(256, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)CS;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    // the pass waits (griddepcontrol) before reading the previous pass's output
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelExC(&cfg, (const void*)kern, args);
  }
  template <int NL, int NM, int CS, typename IO>
  static cudaError_t xyfwd_n(const IO* J, long long js, const int* inv, Prologue pro, V* B, long long bs,
                             Dims d, const V* twx, const V* twy, int nrhs, cudaStream_t st) {
    if constexpr (usable<NL, NM, CS>()) {
      void* args[] = {(void*)&J, (void*)&js, (void*)&inv, (void*)&pro, (void*)&B, (void*)&bs, (void*)&d,
                      (void*)&twx, (void*)&twy};
      return launch(k_xyfwd<T, NL, NM, CS, IO>, CS, CS * 3 * d.N, nrhs, XYCfg<T, NL, NM, CS>::fwd_smem, st, args);
    } else {
        return cudaErrorNotSupported;
    }
  }
  template <int NL, int NM, int CS, typename IO>
  static cudaError_t yxinv_n(const V* B, long long bs, const IO* J, long long js, const int* inv, Epilogue ep,
                             IO* out, long long os, Dims d, const V* twx, const V* twy, int nrhs,
                             cudaStream_t st) {
    if constexpr (usable<NL, NM, CS>()) {
      void* args[] = {(void*)&B, (void*)&bs, (void*)&J, (void*)&js, (void*)&inv, (void*)&ep, (void*)&out,
                      (void*)&os, (void*)&d, (void*)&twx, (void*)&twy};
      return launch(k_yxinv<T, NL, NM, CS, IO>, CS, CS * 3 * d.N, nrhs, XYCfg<T, NL, NM, CS>::inv_smem, st, args);
    } else {
        return cudaErrorNotSupported;
    }
  }
};

template <typename T> bool MatvecLaunch<T>::fused(const Dims& d) {
#define MARIE_CASE(a_, b_, c_) \
  if (d.Lp == a_ && d.Mp == b_) return FusedImpl<T>::template usable<a_, b_, c_>();
  MARIE_FUSED_PAIRS(MARIE_CASE)
#undef MARIE_CASE
  return false;
}
template <typename T>
template <typename IO>
cudaError_t MatvecLaunch<T>::xyfwd(const IO* J, long long js, const int* inv, Prologue pro, V* B, long long bs,
                                   const Dims& d, const V* twx, const V* twy, int nrhs, cudaStream_t st) {
#define MARIE_CASE(a_, b_, c_)    \
  if (d.Lp == a_ && d.Mp == b_) \
    return FusedImpl<T>::template xyfwd_n<a_, b_, c_, IO>(J, js, inv, pro, B, bs, d, twx, twy, nrhs, st);
  MARIE_FUSED_PAIRS(MARIE_CASE)
#undef MARIE_CASE
  return cudaErrorNotSupported;
}
template <typename T>
template <typename IO>
cudaError_t MatvecLaunch<T>::yxinv(const V* B, long long bs, const IO* J, long long js, const int* inv,
                                   Epilogue ep, IO* out, long long os, const Dims& d, const V* twx, const V* twy,
                                   int nrhs, cudaStream_t st) {
#define MARIE_CASE(a_, b_, c_)    \
  if (d.Lp == a_ && d.Mp == b_) \
    return FusedImpl<T>::template yxinv_n<a_, b_, c_, IO>(B, bs, J, js, inv, ep, out, os, d, twx, twy, nrhs, st);
  MARIE_FUSED_PAIRS(MARIE_CASE)
#undef MARIE_CASE
  return cudaErrorNotSupported;
}

template <typename T>
template <typename IO>
cudaError_t MatvecLaunch<T>::xfwd(const IO* J, long long js, const int* inv, Prologue pro, V* A, long long as,
                                  const Dims& d, const V* tw, int nrhs, cudaStream_t st) {
  return MatvecImpl<T>::template xfwd<IO>(J, js, inv, pro, A, as, d, tw, nrhs, st);
}
template <typename T>
template <typename IO>
cudaError_t MatvecLaunch<T>::xinv(const V* A, long long as, const IO* J, long long js, const int* inv,
                                  Epilogue ep, IO* out, long long os, const Dims& d, const V* tw, int nrhs,
                                  cudaStream_t st) {
  return MatvecImpl<T>::template xinv<IO>(A, as, J, js, inv, ep, out, os, d, tw, nrhs, st);
}
template <typename T>
cudaError_t MatvecLaunch<T>::cols(bool inv, int NC, const V* in, long long in_w, long long in_rhs, int n_in, V* out,
                                  long long out_w, long long out_rhs, int n_out, int Lp, int nw, const V* tw,
                                  int nrhs, cudaStream_t st, const int* stop, int step) {
  return MatvecImpl<T>::cols(inv, NC, in, in_w, in_rhs, n_in, out, out_w, out_rhs, n_out, Lp, nw, tw, nrhs, st, stop,
                             step);
}
template <typename T>
cudaError_t MatvecLaunch<T>::zmul(V* B, long long bs, const V* fN, int oct, const Dims& d, const V* tw, int nrhs,
                                  cudaStream_t st, int kind, const ZTile* zt) {
  return MatvecImpl<T>::zmul(B, bs, fN, oct, d, tw, nrhs, st, kind, zt);
}

}  // namespace marie
