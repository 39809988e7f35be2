// The system's operator on the smallest transform grid that holds the body.
//
// The matvec multiplies by the block-Toeplitz operator T(i - j) through a
// circulant of the whole grid, but only differences between DOFs ever meet:
// when the DOFs lie in a box of bx x by x bz voxels, a circulant of the next
// transform lengths >= 2 bx, 2 by, 2 bz gives the same products.  A body rarely
// fills its grid (the 20 x 15 x 25 cm phantom takes 100 x 75 x 125 voxels at 2
// mm, of 128^3 or of 256 x 192 x 160), and every pass, spectrum and operator
// read scales with the padded volume.
//
// The smaller spectrum comes from the plan's FP64 octant by one real matrix per
// axis: back to Toeplitz entries, cut to the box's offsets, forward at the new
// length, composed.  With P = 2n and P' = 2n' the matrix entry is
//   R(k', k) = c_k / (2P') * [D(t-) +- D(t+)],   t+- = 2 pi (k'/P' +- k/P),
//   D(t) = sin((n' - 1/2) t) / sin(t/2) = sum_{|m| < n'} exp(i m t),
// + for components even along the axis, - for odd ones, c_k = 1 at k = 0, n and
// 2 between.  The angles are reduced as integers, so the entries carry a few
// ulp and the new spectrum is as good as a new FFT (no FFT is cheaper here: the
// matrices are at most 257 square and run at the FP64 pipe's rate).
// Measured with ellipsoid phantoms (whole grid -> box): FP64 product of a 96 x
// 80 x 64 grid 2.24 -> 0.61 ms, FP32 product of 256 x 192 x 160 3.15 -> 0.41 ms,
// BiCGSTAB solve of 48^3 in FP64 217 -> 138 ms.
//
// The maps are FP64 work (31 GFLOP from 256 x 192 x 160 to 128 x 80 x 128): a
// plan's first solve or bind on a box, and every one after a body of another box,
// takes 30 ms more there, 4.3 ms more for 128^3 (to 128 x 80 x 128) and 1.0 ms
// more for 96 x 80 x 64; a bind on the box that the plan holds takes 0.5 to 0.7
// ms in all.  A solve's first use pays for it; a bound FP32 product does after 11
// applications at 256 x 192 x 160 and about 24 at 128^3, an FP64 one of 96 x 80 x
// 64 after one.
#include <algorithm>
#include <cstring>
#include <vector>

#include "matvec_launch.cuh"
#include "plan.h"

namespace marie {

namespace {

// Products below this many voxels are bound by launches, not by the padded
// volume.
constexpr long long kCropMinVoxels = 30000;
// Crop when the padded volume, to which the passes' time is proportional, falls
// to this share or less: building the smaller operator costs up to a few FP64
// products, and a solve takes tens to hundreds.
constexpr double kCropShare = 0.8;
// sin(pi m / d), the angle reduced to the first quarter turn as an integer
__device__ __forceinline__ double sin_ratio(long long m, long long d) {
  m %= 2 * d;
  const bool neg = m >= d;
  if (neg) m -= d;
  if (2 * m > d) m = d - m;
  const double v = sinpi((double)m / (double)d);
  return neg ? -v : v;
}

// sin((n2 - 1/2) t) / sin(t/2) at t = 2 pi a / d
__device__ __forceinline__ double dirichlet(long long a, long long d, int n2) {
  a %= d;
  if (a < 0) a += d;
  return a == 0 ? 2.0 * n2 - 1.0 : sin_ratio((2LL * n2 - 1) * a, d) / sin_ratio(a, d);
}

// R[parity][k][k2] for k <= n, k2 <= n2
__global__ void k_axis_matrix(int n, int n2, double* __restrict__ R) {
  const int K = n + 1, K2 = n2 + 1;
  const long long P = 2LL * n, P2 = 2LL * n2, PP = P * P2;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < (long long)K * K2;
       i += (long long)gridDim.x * blockDim.x) {
    const long long k = i / K2, k2 = i - k * K2;
    const double dm = dirichlet(k2 * P - k * P2, PP, n2), dp = dirichlet(k2 * P + k * P2, PP, n2);
    const double c = (k == 0 || k == n ? 0.5 : 1.0) / (double)P2;
    R[i] = c * (dm + dp);
    R[(long long)K * K2 + i] = c * (dm - dp);
  }
}

// out[o][k2][i] = sum_k R[parity(q)][k][k2] in[o][k][i], o = (q, outer), i <
// inner.  FP64-pipe bound: a warp holds 32 columns (o, i) and 8 outputs per
// thread, so each shared-memory read feeds 2 to 16 FP64 FMAs.
constexpr int AM_KT = 16, AM_OUT = 64;
__global__ void __launch_bounds__(256) k_axis_map(const double2* __restrict__ in, double2* __restrict__ out,
                                                  const double* __restrict__ R, int axis, int K, int K2,
                                                  long long inner, long long outer) {
  __shared__ double2 xs[AM_KT][33];
  __shared__ double rs[AM_KT][AM_OUT];
  const int q = blockIdx.z;
  const double* Rq = R + (OpKind<0>::odd(q, axis) ? (long long)K * K2 : 0);
  const long long cols = inner * outer;
  const long long col0 = blockIdx.x * 32LL;
  const int lane = threadIdx.x & 31, group = threadIdx.x >> 5;
  const int k20 = blockIdx.y * AM_OUT;
  const double2* inq = in + q * cols * K;
  double2* outq = out + q * cols * K2;
  double2 acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = mk<double2>(0, 0);
  const bool busy = k20 + 8 * group < K2;
  for (int k0 = 0; k0 < K; k0 += AM_KT) {
    for (int e = threadIdx.x; e < AM_KT * 32; e += 256) {
      // along x (inner = 1) consecutive threads read consecutive k
      const int kk = inner == 1 ? e % AM_KT : e / 32, c = inner == 1 ? e / AM_KT : e % 32;
      const long long j = col0 + c;
      double2 v = mk<double2>(0, 0);
      if (j < cols && k0 + kk < K) {
        const long long o = j / inner, i = j - o * inner;
        v = inq[(o * K + k0 + kk) * inner + i];
      }
      xs[kk][c] = v;
    }
    for (int e = threadIdx.x; e < AM_KT * AM_OUT; e += 256) {
      const int kk = e / AM_OUT, j = e % AM_OUT;
      rs[kk][j] = (k0 + kk < K && k20 + j < K2) ? Rq[(long long)(k0 + kk) * K2 + k20 + j] : 0.0;
    }
    __syncthreads();
    if (busy) {
#pragma unroll 4
      for (int kk = 0; kk < AM_KT; ++kk) {
        const double2 v = xs[kk][lane];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const double r = rs[kk][8 * group + j];
          acc[j].x = fma(r, v.x, acc[j].x);
          acc[j].y = fma(r, v.y, acc[j].y);
        }
      }
    }
    __syncthreads();
  }
  const long long j = col0 + lane;
  if (!busy || j >= cols) return;
  const long long o = j / inner, i = j - o * inner;
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const int k2 = k20 + 8 * group + r;
    if (k2 < K2) outq[(o * K2 + k2) * inner + i] = acc[r];
  }
}

// box[0..2] = max(-x, -y, -z), box[3..5] = max(x, y, z) over the voxels of the
// DOFs (1-based idx into L x M x N x 3, or outside: skipped)
__global__ void k_dof_box(const int64_t* __restrict__ idx, long long n, int L, int M, long long V,
                          int* __restrict__ box) {
  int b[6] = {INT_MIN, INT_MIN, INT_MIN, INT_MIN, INT_MIN, INT_MIN};
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const long long g = idx[i] - 1;
    if (g < 0 || g >= 3 * V) continue;
    const int v = (int)(g % V);
    const int c[3] = {v % L, (v / L) % M, v / (L * M)};
    for (int a = 0; a < 3; ++a) {
      b[a] = max(b[a], -c[a]);
      b[3 + a] = max(b[3 + a], c[a]);
    }
  }
  box_reduce(b, box);
}

// inv (3 x N' x M' x L', preset to -1) of the DOFs on the box's grid
__global__ void k_inverse_box(const int64_t* __restrict__ idx, long long n, int L, int M, long long V, int x0, int y0,
                              int z0, int L2, int M2, int N2, int* __restrict__ inv) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const long long g = idx[i] - 1;
    const int c = (int)(g / V), v = (int)(g % V);
    const int x = v % L - x0, y = (v / L) % M - y0, z = v / (L * M) - z0;
    inv[x + (long long)L2 * (y + (long long)M2 * (z + (long long)N2 * c))] = (int)i;
  }
}

}  // namespace

bool crop_possible(const marie_plan* p) {
  // the smaller operator is derived from the FP64 octant
  return p->has_op && p->oct && p->fN64 && !p->profile && !p->whole_grid && p->d.V >= kCropMinVoxels;
}

int dof_box(marie_plan* p, const int64_t* idx_dev, long long n, int box[6]) {
  DBuf b;
  MARIE_TRY(b.alloc(6 * sizeof(int), p->stream));
  MARIE_CUDA_TRY(cudaMemsetAsync(b.p, 0x80, 6 * sizeof(int), p->stream));
  k_dof_box<<<grid_stride_blocks(n, 4), 256, 0, p->stream>>>(idx_dev, n, p->d.L, p->d.M, p->d.V, b.as<int>());
  count_launch();
  MARIE_CUDA_TRY(cudaGetLastError());
  MARIE_CUDA_TRY(cudaMemcpyAsync(box, b.p, 6 * sizeof(int), cudaMemcpyDeviceToHost, p->stream));
  MARIE_CUDA_TRY(cudaStreamSynchronize(p->stream));
  return MARIE_OK;
}

static void free_crop(marie_plan* q) {
  if (!q) return;
  cudaStreamSynchronize(q->stream);
  if (q->wsB) cudaFreeAsync(q->wsB, q->stream);
  if (q->arena) cudaFreeAsync(q->arena, q->stream);
  if (q->pinned) cudaFreeHost(q->pinned);
  delete q;
}

// The operator of p on an L2 x M2 x N2 grid; null when memory or a launch
// fails (the caller keeps the whole grid).
static std::shared_ptr<marie_plan> build_crop(marie_plan* p, int L2, int M2, int N2) {
  cudaStream_t st = p->stream;
  std::shared_ptr<marie_plan> q(new marie_plan(), free_crop);
  q->stream = st;
  q->device = p->device;
  q->precision = p->precision;
  q->d.L = L2; q->d.M = M2; q->d.N = N2;
  q->d.Lp = 2 * L2; q->d.Mp = 2 * M2; q->d.Np = 2 * N2;
  q->d.V = (long long)L2 * M2 * N2;
  q->kerr = p->kerr;
  const int from[3] = {p->d.L, p->d.M, p->d.N}, to[3] = {L2, M2, N2};
  const long long O = (long long)(L2 + 1) * (M2 + 1) * (N2 + 1);
  const bool f32 = p->fN32 != nullptr;
  // one allocation: fN64, fN32, fN32x, twiddles (FP64 then FP32)
  std::vector<size_t> off;
  size_t total = 0;
  auto take = [&](size_t bytes) {
    total = (total + 255) / 256 * 256;
    off.push_back(total);
    total += bytes;
  };
  take(6 * O * sizeof(double2));
  take(f32 ? 6 * O * sizeof(float2) : 0);
  take(f32 ? fullx_elems(q->d) * sizeof(float2) : 0);
  std::vector<double2> tw;
  for (int a = 0; a < 3; ++a)
    for (int k = 0; k < 2 * to[a]; ++k) {
      const double t = 2.0 * M_PI * (double)k / (double)(2 * to[a]);
      tw.push_back(mk<double2>(std::cos(t), -std::sin(t)));
    }
  std::vector<float2> tw32;
  for (const double2& t : tw) tw32.push_back(mk<float2>((float)t.x, (float)t.y));
  take(tw.size() * sizeof(double2));
  take(tw.size() * sizeof(float2));
  DBuf arena, t0, t1, R;
  if (!arena.try_alloc(total, st)) return nullptr;
  q->arena = arena.p;
  arena.p = nullptr;
  char* base = static_cast<char*>(q->arena);
  q->fN64 = reinterpret_cast<double2*>(base + off[0]);
  if (f32) q->fN32 = reinterpret_cast<float2*>(base + off[1]);
  double2* tw64_d = reinterpret_cast<double2*>(base + off[3]);
  float2* tw32_d = reinterpret_cast<float2*>(base + off[4]);
  if (cudaMemcpyAsync(tw64_d, tw.data(), tw.size() * sizeof(double2), cudaMemcpyHostToDevice, st) != cudaSuccess ||
      cudaMemcpyAsync(tw32_d, tw32.data(), tw32.size() * sizeof(float2), cudaMemcpyHostToDevice, st) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  for (int a = 0, o = 0; a < 3; o += 2 * to[a], ++a) {
    q->tw64[a] = tw64_d + o;
    if (f32) q->tw32[a] = tw32_d + o;
  }
  // the axes that shrink, the strongest reduction first (the least work left)
  std::vector<int> axes;
  for (int a = 0; a < 3; ++a)
    if (to[a] < from[a]) axes.push_back(a);
  std::sort(axes.begin(), axes.end(), [&](int a, int b) {
    return (double)to[a] / from[a] < (double)to[b] / from[b];
  });
  int cur[3] = {from[0], from[1], from[2]};
  const double2* src = p->fN64;
  for (size_t s = 0; s < axes.size(); ++s) {
    const int a = axes[s];
    const int K = cur[a] + 1, K2 = to[a] + 1;
    const long long inner = a == 0 ? 1 : a == 1 ? cur[0] + 1 : (long long)(cur[0] + 1) * (cur[1] + 1);
    const long long outer = a == 0 ? (long long)(cur[1] + 1) * (cur[2] + 1) : a == 1 ? cur[2] + 1 : 1;
    DBuf& tmp = (s & 1) ? t1 : t0;
    double2* dst = q->fN64;
    if (s + 1 < axes.size()) {
      if (!tmp.try_alloc((size_t)6 * inner * outer * K2 * sizeof(double2), st)) return nullptr;
      dst = tmp.as<double2>();
    }
    if (R.p) {
      cudaFreeAsync(R.p, st);
      R.p = nullptr;
    }
    if (!R.try_alloc((size_t)2 * K * K2 * sizeof(double), st)) return nullptr;
    k_axis_matrix<<<grid_stride_blocks((long long)K * K2, 8), 256, 0, st>>>(cur[a], to[a], R.as<double>());
    const dim3 grid((unsigned)((inner * outer + 31) / 32), (K2 + AM_OUT - 1) / AM_OUT, 6);
    k_axis_map<<<grid, 256, 0, st>>>(src, dst, R.as<double>(), a, K, K2, inner, outer);
    count_launch(2);
    if (cudaGetLastError() != cudaSuccess) return nullptr;
    cur[a] = to[a];
    src = dst;
  }
  if (f32 && store_crop_f32(q.get(), reinterpret_cast<float2*>(base + off[2])) != MARIE_OK) return nullptr;
  if (cudaStreamSynchronize(st) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  q->oct = 1;
  q->has_op = true;
  return q;
}

std::shared_ptr<marie_plan> crop_plan(marie_plan* p, const int box[6], int origin[3]) {
  if (!crop_possible(p)) return nullptr;
  const int n[3] = {p->d.L, p->d.M, p->d.N};
  int need[3];
  for (int a = 0; a < 3; ++a) {
    origin[a] = -box[a];
    need[a] = box[3 + a] + box[a] + 1;
    if (origin[a] < 0 || need[a] < 1 || origin[a] + need[a] > n[a]) return nullptr;
  }
  int best[3];
  for (int a = 0; a < 3; ++a)
    for (best[a] = need[a]; !fft_length_supported(2 * best[a]); ++best[a]) {
    }
  if ((double)best[0] * best[1] * best[2] > kCropShare * (double)p->d.V) return nullptr;
  std::shared_ptr<marie_plan> q = p->crop;
  if (!q || q->d.L != best[0] || q->d.M != best[1] || q->d.N != best[2]) {
    // the last one stays with the plan: its size depends on the body's box only
    p->crop.reset();
    q = build_crop(p, best[0], best[1], best[2]);
    p->crop = q;
  }
  if (q) crop_settings(p, q.get());
  return q;
}

void crop_settings(const marie_plan* p, marie_plan* q) {
  q->stream = p->stream;
  q->nrhs_max = p->nrhs_max;
  q->fuse = p->fuse;
  q->inner_prec = p->inner_prec;
  q->inner_restart = p->inner_restart;
  q->batch_groups = p->batch_groups;
  q->graph_refine = p->graph_refine;
}

void drain(cudaStream_t st) {
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusActive;
  if (cudaStreamIsCapturing(st, &capturing) == cudaSuccess && capturing == cudaStreamCaptureStatusNone)
    cudaStreamSynchronize(st);
  cudaGetLastError();
}

bool give_crop_back(marie_plan* p) {
  if (!p->crop && !p->bnd_crop) return false;
  p->crop.reset();
  p->bnd_crop.reset();  // (bnd_inv serves the whole grid)
  cudaFree(p->bnd_inv_crop);
  p->bnd_inv_crop = nullptr;
  trim_pool(p->stream);
  return true;
}

// The body seldom fills its transform grid either (98 x 72 x 122 voxels of 128 x
// 80 x 128): the passes run over its rows and planes only.  Measured with
// ellipsoid phantoms: FP64 product of a 96 x 80 x 64 grid 538 -> 519 us, FP32
// product of 128^3 335 -> 322, of 256 x 192 x 160 341 -> 332, mixed solve of
// 128^3 194.5 -> 189.7 ms, batch of 8 at 64^3 123.2 -> 120.7.
Extent box_extent(const marie_plan* q, const int box[6]) {
  Extent e;
  // the fused x+y kernels are compiled for all rows
  e.M = MatvecLaunch<float>::fused(q->d) ? q->d.M : box[4] + box[1] + 1;
  e.N = box[5] + box[2] + 1;
  return e;
}

int build_inverse_box(marie_plan* p, marie_plan* q, const int origin[3], const Extent& ext, const int64_t* idx_dev,
                      long long n, int* inv) {
  const Dims& d = q->d;
  MARIE_CUDA_TRY(cudaMemsetAsync(inv, 0xff, 3LL * d.L * ext.M * ext.N * sizeof(int), p->stream));
  k_inverse_box<<<grid_stride_blocks(n, 8), 256, 0, p->stream>>>(idx_dev, n, p->d.L, p->d.M, p->d.V, origin[0],
                                                                 origin[1], origin[2], d.L, ext.M, ext.N, inv);
  count_launch();
  MARIE_CUDA_TRY(cudaGetLastError());
  return MARIE_OK;
}

}  // namespace marie
