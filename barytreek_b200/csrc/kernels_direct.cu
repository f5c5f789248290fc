// FP64 direct sum over every (target, source) pair, target == source included
// (src/direct_sum_impl.hpp:9-94). Used for accuracy measurement against the
// treecode (the reference's examples do the same, e.g.
// examples/example_poisson_3d.cpp:163-183). Its reciprocal square roots and
// quotients are rounded to FP64 (a cubic step on the FP32 seed, a remainder),
// where the treecode takes one Newton step; the 2-D logarithm is the treecode's
// (log_fp64_pos, checked by itself in test_gpu_log2d.py).
//
// Bound: FP64 issue (18 FP64 operations a potential + gradient pair). A block
// of 4 warps owns 64 targets, two per lane, and one slice of the sources, a
// quarter of it per warp; a second kernel adds the slices. One thread per
// target over all sources left 108 of 148 SMs idle at 10,000 targets. Each
// warp stages 32 sources at a time through its own 1 KB of shared memory, the
// next 32 in flight in registers. Warps and slices are added in a fixed order,
// so a result depends on the counts and the GPU's SM count alone. 10,000
// targets x 1M sources, potential + gradient: 147.8 -> 12.8 ms (with slices
// spread over thread-block clusters instead of a second kernel 15.6 ms: too few
// clusters of 8 fit at a time).
#include <algorithm>

#include "device_math.cuh"
#include "kernels.cuh"

namespace btk {

namespace {

constexpr int kDirectWarps = 4;
constexpr int kDirectTile = 64;
constexpr int kDirectBlocksPerSm = 4;  // 123 registers without spills: 12.8 ms; 5 blocks 15.8, 6 blocks 14.1 (spills)
// Coordinates up to here keep r^2 inside the seeds' range, charges the
// quotients' remainders finite; a call with larger ones (or infinities) takes
// IEEE square roots, divisions and CUDA's log.
constexpr double kDirectCoordMax = 1.0e18, kDirectChargeMax = 1.0e200;

// 1 / sqrt(x) rounded to FP64: the seed of rsqrt_fp64_scaled (relative error e
// below 2e-7) and a step with error e^3.
__device__ __forceinline__ double rsqrt_full(double x) {
  float yf;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(yf) : "f"(fp32_seed_arg(x)));
  const double y = (double)yf;
  const double e = fma(-x, y * y, 1.0);
  return fma(y, e * fma(e, 0.375, 0.5), y);
}
// w / x rounded to FP64: rcp_fp64_pos (error 4e-14) and the quotient's remainder.
// |w| <= kDirectChargeMax, so nothing overflows. A rounded reciprocal times w has
// one rounding more and one operation less: 10,000 targets x 1M sources, vector
// kernel 10.3 -> 11.4 ms, 2-D potential + gradient 17.9 -> 18.9 ms.
__device__ __forceinline__ double quotient(double w, double x) {
  const double y = rcp_fp64_pos(x), q = w * y;
  return fma(fma(-x, q, w), y, q);
}

// One pair; sums without the constant factor, as eval_fp64's. FAST: r^2 inside
// the seeds' range.
template <int DIM, int KIND, bool FAST>
__device__ __forceinline__ void direct_pair(double tx, double ty, double tz, const double4& s, double eps2,
                                            const double* log_table, double* acc) {
  const double dx = tx - s.x, dy = ty - s.y, dz = DIM == 3 ? tz - s.z : 0.0;
  double r2 = fma(dx, dx, fma(dy, dy, eps2));
  if (DIM == 3) r2 = fma(dz, dz, r2);
  if (DIM == 2) {
    float yf = 0.f;
    acc[0] = fma(FAST ? log_fp64_pos(r2, log_table, yf) : log(r2), s.w, acc[0]);
    if (KIND == BTK_KIND_FIELD) {
      const double g = FAST ? quotient(s.w, r2) : s.w / r2;
      acc[1] = fma(dx, g, acc[1]);
      acc[2] = fma(dy, g, acc[2]);
    }
  } else if (KIND == BTK_KIND_VEL) {
    const double g = FAST ? quotient(s.w, r2) : s.w / r2;
    acc[0] = fma(dx, g, acc[0]);
    acc[1] = fma(dy, g, acc[1]);
    acc[2] = fma(dz, g, acc[2]);
  } else {
    const double ri = FAST ? rsqrt_full(r2) : 1.0 / sqrt(r2);
    if (KIND == BTK_KIND_POT) {
      acc[0] = fma(ri, s.w, acc[0]);
    } else {
      const double wr = s.w * ri;
      acc[0] += wr;
      const double g = wr * (ri * ri);
      acc[1] = fma(dx, g, acc[1]);
      acc[2] = fma(dy, g, acc[2]);
      acc[3] = fma(dz, g, acc[3]);
    }
  }
}

// A warp's slice [s0, s1) of the sources against its lanes' two targets.
template <int DIM, int KIND, bool FAST, int NC>
__device__ __forceinline__ void direct_slice(const double4* src, long long s0, long long s1, double4* stage,
                                             const double* tx, const double* ty, const double* tz, double eps2,
                                             const double* log_table, double (*acc)[NC]) {
  const int lane = threadIdx.x & 31;
  double4 next = s0 + lane < s1 ? src[s0 + lane] : make_double4(0.0, 0.0, 0.0, 0.0);
  for (long long b = s0; b < s1; b += 32) {
    __syncwarp();
    stage[lane] = next;
    __syncwarp();
    if (b + 32 + lane < s1) next = src[b + 32 + lane];
    const int cnt = (int)min(32ll, s1 - b);
#pragma unroll 4
    for (int j = 0; j < cnt; ++j) {
      const double4 s = stage[j];
      direct_pair<DIM, KIND, FAST>(tx[0], ty[0], tz[0], s, eps2, log_table, acc[0]);
      direct_pair<DIM, KIND, FAST>(tx[1], ty[1], tz[1], s, eps2, log_table, acc[1]);
    }
  }
}

// The constant factor of component c.
template <int DIM>
__device__ __forceinline__ double direct_scale(int c) {
  const double pi = 3.141592653589793238462643383279502884;
  return DIM == 3 ? -1.0 / (4.0 * pi) : (c == 0 ? 1.0 / (4.0 * pi) : -1.0 / (2.0 * pi));
}

// Block (tile, slice). partial: [slice][component][target], or null (one
// slice): the results go to out.
template <int DIM, int KIND>
__global__ void __launch_bounds__(kDirectWarps * 32, kDirectBlocksPerSm)
    k_direct(double eps2, int nt, const double* xt, const double* yt, const double* zt, int ns, const double4* src,
             const int* large, double* partial, double* out) {
  constexpr int NC = KIND == BTK_KIND_POT ? 1 : (KIND == BTK_KIND_VEL ? 3 : 1 + DIM);
  constexpr int kVals = NC * kDirectTile;
  __shared__ double4 stage[kDirectWarps][32];
  __shared__ double red[kDirectWarps][kVals];
  __shared__ double s_log[DIM == 2 ? kLogTable : 1];
  const int tile = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (DIM == 2) {
    log_table_fill(s_log);
    __syncthreads();
  }
  double tx[2], ty[2], tz[2], acc[2][NC];
  bool big = *large != 0;
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int i = min(tile * kDirectTile + 32 * u + lane, nt - 1);
    tx[u] = xt[i];
    ty[u] = yt[i];
    tz[u] = DIM == 3 ? zt[i] : 0.0;
    big |= !(fmax(fabs(tx[u]), fmax(fabs(ty[u]), fabs(tz[u]))) <= kDirectCoordMax);
#pragma unroll
    for (int c = 0; c < NC; ++c) acc[u][c] = 0.0;
  }
  const long long parts = (long long)gridDim.y * kDirectWarps, k = (long long)blockIdx.y * kDirectWarps + warp;
  const long long s0 = ns * k / parts, s1 = ns * (k + 1) / parts;
  if (__any_sync(0xffffffffu, big) || !(eps2 >= kSeedMin && eps2 <= 1.0e37))
    direct_slice<DIM, KIND, false, NC>(src, s0, s1, stage[warp], tx, ty, tz, eps2, s_log, acc);
  else
    direct_slice<DIM, KIND, true, NC>(src, s0, s1, stage[warp], tx, ty, tz, eps2, s_log, acc);
#pragma unroll
  for (int u = 0; u < 2; ++u)
#pragma unroll
    for (int c = 0; c < NC; ++c) red[warp][c * kDirectTile + 32 * u + lane] = acc[u][c];
  __syncthreads();
  for (int v = threadIdx.x; v < kVals; v += blockDim.x) {
    double s = red[0][v];
#pragma unroll
    for (int w = 1; w < kDirectWarps; ++w) s += red[w][v];
    const int c = v / kDirectTile, i = tile * kDirectTile + v % kDirectTile;
    if (i >= nt) continue;
    if (partial)
      partial[((size_t)blockIdx.y * NC + c) * nt + i] = s;
    else
      out[(size_t)c * nt + i] = direct_scale<DIM>(c) * s;
  }
}

// out = the slices' partial sums in slice order, scaled.
template <int DIM>
__global__ void k_direct_reduce(int slices, int nc, int nt, const double* partial, double* out) {
  const size_t v = (size_t)blockIdx.x * blockDim.x + threadIdx.x, n = (size_t)nc * nt;
  if (v >= n) return;
  double s = partial[v];
  for (int k = 1; k < slices; ++k) s += partial[k * n + v];
  out[v] = direct_scale<DIM>((int)(v / nt)) * s;
}

// Packs (x, y, z, q) into double4 in the original source order; *large is set
// when a coordinate exceeds kDirectCoordMax or a charge kDirectChargeMax.
__global__ void k_pack_sources(int n, const double* x, const double* y, const double* z, const double* q,
                               double4* out, int* large) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double4 s = make_double4(x[i], y[i], z ? z[i] : 0.0, q[i]);
  out[i] = s;
  if (!(fmax(fabs(s.x), fmax(fabs(s.y), fabs(s.z))) <= kDirectCoordMax) || !(fabs(s.w) <= kDirectChargeMax)) *large = 1;
}

}  // namespace

cudaError_t launch_pack_sources(int n, const double* x, const double* y, const double* z, const double* q,
                                double4* out, int* large, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(large, 0, sizeof(int), s);
  if (e != cudaSuccess || n <= 0) return e;
  k_pack_sources<<<(n + 255) / 256, 256, 0, s>>>(n, x, y, z, q, out, large);
  count_launch();
  return cudaGetLastError();
}

// Slices of the sources: the count with the fewest waves of the grid per unit
// of a slice's work (a last wave that is mostly empty costs a whole one), the
// smallest of equals; at least 32 sources a warp, and partial sums of at most
// kDirectScratch doubles.
int direct_slices(int dim, int kind, int nt, int ns) {
  int dev = 0, sms = 1;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    sms = 1;
  const long long tiles = (nt + kDirectTile - 1) / kDirectTile, slots = (long long)sms * kDirectBlocksPerSm;
  const int nc = kind == BTK_KIND_POT ? 1 : (kind == BTK_KIND_VEL ? 3 : 1 + dim);
  const long long most = std::min<long long>(std::min<long long>(kDirectScratch / std::max<long long>(1, (long long)nc * nt),
                                                                 ns / (kDirectWarps * 32)), 1024);
  int best = 1;
  double t_best = (double)((tiles + slots - 1) / slots);
  for (int k = 2; k <= most; ++k) {
    const double t = (double)((tiles * k + slots - 1) / slots) / k;
    if (t < 0.99 * t_best) {
      t_best = t;
      best = k;
    }
  }
  return best;
}

cudaError_t launch_direct(int dim, int kind, double eps, int nt, const double* xt, const double* yt, const double* zt,
                          int ns, const double4* src, const int* large, int slices, double* partial, double* out,
                          cudaStream_t s) {
  if (nt <= 0) return cudaSuccess;
  const dim3 grid((nt + kDirectTile - 1) / kDirectTile, slices);
  const int threads = kDirectWarps * 32;
  const double e2 = eps * eps;
  double* p = slices > 1 ? partial : nullptr;
  if (dim == 2) {
    if (kind == BTK_KIND_POT) k_direct<2, BTK_KIND_POT><<<grid, threads, 0, s>>>(e2, nt, xt, yt, zt, ns, src, large, p, out);
    else k_direct<2, BTK_KIND_FIELD><<<grid, threads, 0, s>>>(e2, nt, xt, yt, zt, ns, src, large, p, out);
  } else {
    if (kind == BTK_KIND_POT) k_direct<3, BTK_KIND_POT><<<grid, threads, 0, s>>>(e2, nt, xt, yt, zt, ns, src, large, p, out);
    else if (kind == BTK_KIND_VEL) k_direct<3, BTK_KIND_VEL><<<grid, threads, 0, s>>>(e2, nt, xt, yt, zt, ns, src, large, p, out);
    else k_direct<3, BTK_KIND_FIELD><<<grid, threads, 0, s>>>(e2, nt, xt, yt, zt, ns, src, large, p, out);
  }
  count_launch();
  if (p) {
    const int nc = kind == BTK_KIND_POT ? 1 : (kind == BTK_KIND_VEL ? 3 : 1 + dim);
    const unsigned blocks = (unsigned)(((size_t)nc * nt + 255) / 256);
    if (dim == 2)
      k_direct_reduce<2><<<blocks, 256, 0, s>>>(slices, nc, nt, p, out);
    else
      k_direct_reduce<3><<<blocks, 256, 0, s>>>(slices, nc, nt, p, out);
    count_launch();
  }
  return cudaGetLastError();
}

}  // namespace btk
