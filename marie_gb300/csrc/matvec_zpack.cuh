// The FP32 z pass on two columns per thread (fft_packed.cuh): forward z
// transforms of the three components, the symmetric product with the operator
// and the inverse transforms, in place in B, for operators whose tile arrives
// by a bulk tensor copy.
#pragma once
#include "fft_packed.cuh"
#include "matvec_kernels.cuh"

namespace marie {

template <int NZ> struct ZP {
  static constexpr bool W = HasWide<NZ>::value;
  using FF = FFT<cpk, NZ, false, W>;
  using FI = FFT<cpk, NZ, true, W>;
  static constexpr int S = 8, P = S / 2;  // columns and column pairs per CTA
  static constexpr int T = FF::T;
  static constexpr int THREADS = 3 * P * T;
  // one component's exchange buffer: rows of four pairs (64 B), half a line
  // inserted after every 16 rows
  static constexpr int BUF = NZ * P + (NZ / 16 + 1) * P;
  static constexpr int NO = NZ / 2 + 1;
  static constexpr int TILE = 6 * NO * P;
  static constexpr size_t bytes = (size_t)(NZ + 3 * BUF + TILE) * sizeof(cpk) + 128;
  static constexpr bool ok = NO <= 256 && bytes <= 220 * 1024;
  // CTAs per SM that shared memory and a register budget for the held values allow
  static constexpr int REGS = FF::E <= 8 ? 80 : FF::E <= 16 ? 128 : 216;
  static constexpr int BY_SMEM = (int)(227 * 1024 / (bytes + 1024)), BY_REGS = 65536 / (THREADS * REGS);
  static constexpr int MOST = BY_SMEM < BY_REGS ? BY_SMEM : BY_REGS;
  static constexpr int CTAS = MOST < 1 ? 1 : MOST > 16 ? 16 : MOST;
  __device__ static SAddr addr() { return SAddr(P, false, P); }
};

// Waits for a bulk copy's barrier, at most `limit` ns of global time, after
// which *err is set and the pass goes on (its values are wrong, the status word
// tells the host).
__device__ __forceinline__ void tile_wait(unsigned bar, unsigned long long limit, int* err) {
  unsigned long long t_start;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_start));
  for (;;) {
    unsigned done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar)
        : "memory");
    if (done) return;
    unsigned long long t_now;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_now));
    if (t_now - t_start > limit) {
      if (err) atomicExch(err, 1);
      return;
    }
  }
}

// Thread group c transforms component c of the CTA's 4 column pairs.  The
// operator's reflections in y and z act as N -> D N D, D = diag(1, -1, 1) for a
// y-reflected column and diag(1, 1, -1) for positions kz > NZ/2 (the odd
// components of the symmetric tensor are the ones that change sign): the
// component's spectrum and its row of the product change sign there, and the
// tile is read as it is.  The tile holds the two columns of a pair as {re, re,
// im, im}.
//
// tma = 2: a test of the bounded wait (see k_zmul).
//
// Bound by shared memory (about 40 16-byte accesses per thread and 16 points:
// exchanges, the other components' spectra, the tile) and by DRAM next; issue
// slots bound the one-column form (packed FP32 instructions are additions only
// there).  Measured against
// the one-column form: 128-point columns of a 64^3 grid 33.0 -> 30.4 us, 160 of
// 80^3 99 -> 73 us, 192 of 96^3 144 -> 118 us (both with the prime-factor
// schedules), 256 of 128^3 241 -> 217 us.  Persistent CTAs that load the next
// columns and tile during the inverse transforms were no faster (256 points 229
// us, 128 32 us): the phases overlap across the resident CTAs already.
template <int NZ>
__global__ void __launch_bounds__(ZP<NZ>::THREADS, ZP<NZ>::CTAS)
k_zmul_pairs(float2* __restrict__ B, long long b_rhs, Dims d, const float2* __restrict__ tw,
             const __grid_constant__ CUtensorMap tmap, int tma, int* err) {
  if (rhs_skipped(d, blockIdx.z)) return;
  using Z = ZP<NZ>;
  using FF = typename Z::FF;
  using FI = typename Z::FI;
  constexpr int P = Z::P, NH = NZ / 2, NO = Z::NO, E = FF::E, R0 = FF::R0, RL = FF::RL, RLI = FI::RL;
  static_assert(FI::R0 == FF::RL, "inverse must start where the forward transform ended");
  const SAddr ad = Z::addr();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  // the tile first, on a 128-byte boundary (the bulk copy's destination)
  cpk* tile = reinterpret_cast<cpk*>(
      smem_raw + ((128u - ((unsigned)__cvta_generic_to_shared(smem_raw) & 127u)) & 127u));
  cpk* tw_s = tile + Z::TILE;
  cpk* buf = tw_s + NZ;
  const int kx0 = blockIdx.x * Z::S;
  // rows in the order 0, M, 1, 2M-1, 2, ...: the two that share a tile adjacent
  const int gy = blockIdx.y;
  const int ky = gy == 0 ? 0 : gy == 1 ? d.Mp / 2 : (gy & 1) ? d.Mp - (gy >> 1) : (gy >> 1);
  const bool fy = ky > d.Mp / 2;
  const int oy = fy ? d.Mp - ky : ky;
  const long long plane = (long long)d.Lp * d.Mp;
  const int c = threadIdx.x / (P * FF::T);
  const int rem = threadIdx.x - c * P * FF::T;
  const int s = rem % P, t = rem / P;
  __shared__ __align__(8) unsigned long long tile_bar;
  const unsigned bar = (unsigned)__cvta_generic_to_shared(&tile_bar);
  if (threadIdx.x == 0) {
    // box origin (kx0, oy, 0, 0), kx0 a multiple of 8: a 16-byte boundary; the
    // box 8 x 1 x NO x 6 lies inside the (Lp, M+1, N+1, 6) tensor
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar));
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    const unsigned bytes = (unsigned)(Z::TILE * sizeof(cpk)) + (tma == 2 ? 16u : 0u);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, "
        "%5}], [%6];" ::"r"((unsigned)__cvta_generic_to_shared(tile)),
        "l"(reinterpret_cast<unsigned long long>(&tmap)), "r"(kx0), "r"(oy), "r"(0), "r"(0), "r"(bar)
        : "memory");
  }
  for (int i = threadIdx.x; i < NZ; i += Z::THREADS) {
    const float2 w = tw[i];
    tw_s[i] = cpk{pk(w.x), pk(w.y)};
  }
  pdl_wait();  // the spectrum B is the previous pass's output
  float2* Bp = after_wait(B) + blockIdx.z * b_rhs + c * plane * d.N + (long long)ky * d.Lp + kx0 + 2 * s;
  float4 in[E / R0 * (R0 / 2)];
#pragma unroll
  for (int b = 0; b < E / R0; ++b)
#pragma unroll
    for (int r = 0; r < R0 / 2; ++r) {
      const int p = FF::in_pos(t, b, r);
      in[b * (R0 / 2) + r] =
          p < d.N ? __ldcg(reinterpret_cast<const float4*>(Bp + p * plane)) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  __syncthreads();  // twiddles staged, barrier initialised
  cpk reg[E];
#pragma unroll
  for (int b = 0; b < E / R0; ++b)
#pragma unroll
    for (int r = 0; r < R0; ++r)
      reg[b * R0 + r] = r < R0 / 2 ? pack2(in[b * (R0 / 2) + (r < R0 / 2 ? r : 0)]) : mk<cpk>(0, 0);
  cpk* my = buf + c * Z::BUF + s;
  FF::run_half(reg, my, ad, t, tw_s);
  auto reflect = [&]() {
    if (c == 1 && fy) {
#pragma unroll
      for (int i = 0; i < E; ++i) reg[i] = cneg(reg[i]);
    }
    if (c == 2) {
#pragma unroll
      for (int b = 0; b < E / RL; ++b)
#pragma unroll
        for (int r = 0; r < RL; ++r)
          if (FF::out_pos(t, b, r) > NH) reg[b * RL + r] = cneg(reg[b * RL + r]);
    }
  };
  reflect();
  __syncthreads();
  FF::store(reg, my, ad, t);
  tile_wait(bar, tma == 2 ? 5000000ull : 2000000000ull, err);
  __syncthreads();
  // row c of the symmetric product: own component from registers, the others' spectra
  auto comp = [](int a, int b) { return a == 0 ? b : a + b + 1; };  // a <= b: xx xy xz yy yz zz
  const int o1 = c == 0 ? 1 : 0, o2 = c == 2 ? 1 : 2;
  const cpk* n0 = tile + comp(c, c) * NO * P + s;
  const cpk* n1 = tile + (c < o1 ? comp(c, o1) : comp(o1, c)) * NO * P + s;
  const cpk* n2 = tile + (c < o2 ? comp(c, o2) : comp(o2, c)) * NO * P + s;
  const cpk* b1 = buf + o1 * Z::BUF + s;
  const cpk* b2 = buf + o2 * Z::BUF + s;
#pragma unroll
  for (int b = 0; b < E / RL; ++b)
#pragma unroll
    for (int r = 0; r < RL; ++r) {
      const int kz = FF::out_pos(t, b, r);
      const int o = (kz > NH ? NZ - kz : kz) * P, e = ad(kz);
      const cpk u = n0[o], v1 = n1[o], v2 = n2[o], x0 = reg[b * RL + r], x1 = b1[e], x2 = b2[e];
      const pk re = pfma(v2.x, x2.x, pfma(v1.x, x1.x, u.x * x0.x));
      const pk im = pfma(v2.y, x2.y, pfma(v1.y, x1.y, u.y * x0.y));
      const pk cr = pfma(v2.x, x2.y, pfma(v1.x, x1.y, u.x * x0.y));
      reg[b * RL + r] = cpk{re - im, pfma(v2.y, x2.x, pfma(v1.y, x1.x, pfma(u.y, x0.x, cr)))};
    }
  reflect();
  pdl_trigger();
  FI::run(reg, my, ad, t, tw_s);
#pragma unroll
  for (int b = 0; b < E / RLI; ++b)
#pragma unroll
    for (int r = 0; r < RLI; ++r) {
      const int z = FI::out_pos(t, b, r);
      if (z < d.N) *reinterpret_cast<float4*>(Bp + z * plane) = unpack2(reg[b * RLI + r]);
    }
}

}  // namespace marie
