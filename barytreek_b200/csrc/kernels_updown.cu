// Upward and downward passes, gathers and proxy materialisation (FP64).
//
// These kernels follow the reference's functors (src/upward_pass_impl.hpp,
// src/downward_pass_impl.hpp) but are gather-shaped: each output row (a leaf's
// modified charges, a parent's anterpolated charges, a child's interpolated
// potentials, a target's value) is produced by one thread block, so no atomics
// are needed and results are bit-reproducible. The (n+1)^d x (n+1)^d
// child<->parent transfers are applied as d one-dimensional (n+1)x(n+1)
// contractions (the tensor-product basis factorises), which is the same linear
// map as the reference's nested loops with (n+1)^d fewer operations.
#include <algorithm>

#include "device_math.cuh"
#include "kernels.cuh"

namespace btk {

namespace {

constexpr double kDblEps = 2.220446049250313e-16;  // numeric_limits<double>::epsilon()

// Barycentric weights 1/2, (-1)^i, (-1)^n/2 (src/bli_impl.hpp:26-32).
template <int M>
__device__ __forceinline__ double bary_weight(int i) {
  double w = (i & 1) ? -1.0 : 1.0;
  return (i == 0 || i == M - 1) ? 0.5 * w : w;
}

// interp_vals_bli (src/bli_impl.hpp:9-63) on precomputed nodes:
// the absolute near-node test, then w_i/(x-x_i) normalised by their sum.
template <int M>
__device__ __forceinline__ void bary_basis(double (&L)[M], double x, const double* node) {
  int hit = -1;
#pragma unroll
  for (int i = 0; i < M; ++i)
    if (hit < 0 && fabs(x - node[i]) < kDblEps) hit = i;
  if (hit >= 0) {
#pragma unroll
    for (int i = 0; i < M; ++i) L[i] = (i == hit) ? 1.0 : 0.0;
    return;
  }
  double denom = 0.0;
#pragma unroll
  for (int i = 0; i < M; ++i) {
    L[i] = bary_weight<M>(i) / (x - node[i]);
    denom += L[i];
  }
#pragma unroll
  for (int i = 0; i < M; ++i) L[i] = L[i] / denom;
}

// The same basis for many points of one leaf: reciprocals from the FP32 unit
// with a cubic step (1e-7 of a rounding from the rounded value) instead of 2 M
// divisions, and quotients by the sum corrected by their remainders: the
// division form's errors (0.85 to 1.36 roundings rms for 3 to 13 nodes; without
// the correction 0.07 to 0.1 more). The basis does not change when x and the nodes are scaled, so
// they come times `scale`, a power of two that makes the node range 1 to 2 and
// keeps every difference inside the FP32 unit's range; a point nearer than that
// to a node, or within the near-node test, and a panel without a usable scale
// (basis_scale 0) take bary_basis.
__device__ __forceinline__ double basis_scale(double range) {  // range >= 0
  const int e = __double2hiint(range) >> 20;                     // biased exponent
  return e >= 1 && e < 2046 ? __hiloint2double((2046 - e) << 20, 0) : 0.0;
}
__device__ __forceinline__ double rcp_signed(double d) {
  float yf;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(yf) : "f"((float)d));
  const double y = (double)yf, e = fma(-d, y, 1.0);
  return fma(y, fma(e, e, e), y);
}
template <int M>
__device__ __forceinline__ void bary_basis_fast(double (&L)[M], double x, const double* node, const double* node_scaled,
                                                double scale) {
  const double xs = x * scale, near = fmax(kDblEps * scale, 1.0e-30);
  bool slow = !(scale > 0.0);
  double denom = 0.0;
#pragma unroll
  for (int i = 0; i < M; ++i) {
    const double d = xs - node_scaled[i];
    slow |= !(fabs(d) >= near);
    L[i] = bary_weight<M>(i) * rcp_signed(d);
    denom += L[i];
  }
  if (slow) {
    bary_basis<M>(L, x, node);
    return;
  }
  const double r = rcp_signed(denom);
#pragma unroll
  for (int i = 0; i < M; ++i) {
    const double q = L[i] * r;
    L[i] = fma(fma(-q, denom, L[i]), r, q);
  }
}

// A panel's nodes and their scaled form in shared memory (all threads call it,
// DIM * M of them at least; the caller synchronises).
template <int DIM, int M>
__device__ __forceinline__ void load_nodes(const double* nd, double (*node)[kMaxNodes], double (*node_scaled)[kMaxNodes],
                                           double* scale) {
  const int t = threadIdx.x;
  if (t < DIM * M) {
    const int d = t / M, i = t % M;
    const double* row = nd + d * kNodeStride;
    const double sc = basis_scale(fabs(row[0] - row[M - 1]));
    node[d][i] = row[i];
    node_scaled[d][i] = row[i] * sc;
    if (i == 0) scale[d] = sc;
  }
}

template <int M, int DIM>
__host__ __device__ constexpr int ipow_c() {
  return DIM == 2 ? M * M : M * M * M;
}

// ---- per-panel geometry ---------------------------------------------------
// One thread per (panel, axis, node): nodes_shift/nodes_interp, then (second
// kernel) the transfer rows L^{parent}_a(node_shift^child_i).
__global__ void k_panel_nodes(int dim, int m, int P, const DevPanel* panels, const double* ucos_shift,
                              const double* ucos_interp, double* nodes_shift, double* nodes_interp) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  int total = P * dim * m;
  if (t >= total) return;
  int i = t % m, d = (t / m) % dim, p = t / (m * dim);
  double lo = panels[p].lo[d], hi = panels[p].hi[d];
  double range = __dmul_rn(0.5, __dsub_rn(hi, lo));
  double mid = __dmul_rn(0.5, __dadd_rn(hi, lo));
  nodes_shift[(size_t)p * kPanelNodes + d * kNodeStride + i] = __dadd_rn(__dmul_rn(ucos_shift[i], range), mid);
  nodes_interp[(size_t)p * kPanelNodes + d * kNodeStride + i] = __dadd_rn(__dmul_rn(ucos_interp[i], range), mid);
}

template <int M>
__global__ void k_panel_xfer(int dim, int P, const DevPanel* panels, const double* nodes_shift,
                             const double* nodes_interp, double* xfer) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  int total = P * dim * M;
  if (t >= total) return;
  int i = t % M, d = (t / M) % dim, c = t / (M * dim);
  int par = panels[c].parent;
  double* row = xfer + (size_t)c * kPanelXfer + (d * kMaxNodes + i) * kMaxNodes;
  if (par < 0) {
    for (int a = 0; a < M; ++a) row[a] = 0.0;
    return;
  }
  double L[M];
  bary_basis<M>(L, nodes_shift[(size_t)c * kPanelNodes + d * kNodeStride + i],
                nodes_interp + (size_t)par * kPanelNodes + d * kNodeStride);
#pragma unroll
  for (int a = 0; a < M; ++a) row[a] = L[a];
}

// ---- gathers ---------------------------------------------------------------
__global__ void k_perm_from_inside(const int* leaves, const int* leaf_begin, const int* point_count,
                                   const int* inside, int thresh, int* perm) {
  int L = leaves[blockIdx.x];
  int b = leaf_begin[L], n = point_count[L];
  for (int j = threadIdx.x; j < n; j += blockDim.x) perm[b + j] = inside[(size_t)L * thresh + j];
}

__global__ void k_gather(int n, const int* perm, const double* x, const double* y, const double* z,
                         const double* w, double4* out) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  int i = perm[k];
  out[k] = make_double4(x[i], y[i], z ? z[i] : 0.0, w ? w[i] : 0.0);
}

// A solve's gathers and clears (SolveBegin): seven launches' worth of work that
// a small solve spent 20 us of its 104 launching (1,000 points).
__global__ void __launch_bounds__(256) k_begin(SolveBegin b) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x, n = (long long)gridDim.x * blockDim.x;
  if (t < b.n_words) b.words[t] = 0;
  for (long long k = t; k < b.ns; k += n) {
    const int i = b.perm_s[k];
    const double x = b.xs[i], y = b.ys[i], z = b.zs ? b.zs[i] : 0.0;
    b.S4[k] = make_double4(x, y, z, b.q[i]);
    if (!b.xt) b.T4[k] = make_double4(x, y, z, 0.0);
  }
  for (long long k = t; b.xt && k < b.nt; k += n) {
    const int i = b.perm_t[k];
    b.T4[k] = make_double4(b.xt[i], b.yt[i], b.zt ? b.zt[i] : 0.0, 0.0);
  }
#pragma unroll
  for (int c = 0; c < 4; ++c)
    for (long long k = t; k < b.n_zero[c]; k += n) b.zero[c][k] = 0.0;
}

// ---- upward pass -----------------------------------------------------------
// base_pots (src/upward_pass_impl.hpp:90-132): a leaf's modified charges
// W[a,b,c] = sum_p q_p Lx_a(x_p) Ly_b(y_p) Lz_c(z_p), one block per leaf. Thread
// (a, b) of a group of M^2 threads keeps W[a][b][0..M-1] (2-D: W[a][b]); G
// groups take every G-th point of a chunk and their partial sums are added at
// the end. Per point a thread reads Lx_a q, Ly_b and the M values Lz_c (two per
// load, broadcasts) for M + 1 FP64 operations. The basis of PCH points is
// formed by one thread a point and axis; with M divisions and M more to
// normalise it took most of the kernel (1M, n = 8: 299 -> 188 us; 1.6M points
// in a batch, n = 6: 383 -> 229 us).
template <int DIM, int M>
__global__ void __launch_bounds__(256, M <= 9 ? 4 : 3) k_leaf_moments(const int* leaves, const int* leaf_begin, const int* point_count,
                                                      const double4* pts, const double* nodes_interp, double* psw) {
  constexpr int IPC = ipow_c<M, DIM>();
  constexpr int PCH = 64;
  constexpr int NZ = DIM == 3 ? M : 1;       // values a thread keeps
  constexpr int MP = (M + 1) & ~1;           // padded to 16 bytes
  constexpr int G = 256 / (M * M) > 0 ? 256 / (M * M) : 1;
  __shared__ __align__(16) double sb[DIM][PCH][MP];
  __shared__ double snode[3][kMaxNodes], snode_s[3][kMaxNodes], sscale[3];
  __shared__ double red[G > 1 ? IPC : 1];
  const int L = leaves[blockIdx.x];
  const int b = leaf_begin[L], cnt = point_count[L];
  const int t = threadIdx.x;
  const int grp = t / (M * M), ab = t % (M * M);
  const bool active = grp < G;
  const int ia = ab / M, ib = ab % M;
  load_nodes<DIM, M>(nodes_interp + (size_t)L * kPanelNodes, snode, snode_s, sscale);
  double acc[NZ];
#pragma unroll
  for (int c = 0; c < NZ; ++c) acc[c] = 0.0;
  __syncthreads();
  for (int p0 = 0; p0 < cnt; p0 += PCH) {
    const int np = min(PCH, cnt - p0);
    for (int v = t; v < DIM * np; v += 256) {
      const int d = v / np, pp = v - d * np;
      const double4 pt = pts[b + p0 + pp];
      double Lv[M];
      bary_basis_fast<M>(Lv, d == 0 ? pt.x : (d == 1 ? pt.y : pt.z), snode[d], snode_s[d], sscale[d]);
      // the charge is folded into the x factor (changes only the last bit
      // against the reference's product order, upward_pass_impl.hpp:164)
#pragma unroll
      for (int i = 0; i < M; ++i) sb[d][pp][i] = d == 0 ? Lv[i] * pt.w : Lv[i];
    }
    __syncthreads();
    if (active) {
      for (int pp = grp; pp < np; pp += G) {
        const double v = sb[0][pp][ia] * sb[1][pp][ib];
        if (DIM == 2) {
          acc[0] += v;
        } else {
          const double2* z = reinterpret_cast<const double2*>(sb[DIM - 1][pp]);
#pragma unroll
          for (int c = 0; c < NZ; c += 2) {
            const double2 zc = z[c / 2];
            acc[c] = fma(v, zc.x, acc[c]);
            if (c + 1 < NZ) acc[c + 1 < NZ ? c + 1 : 0] = fma(v, zc.y, acc[c + 1 < NZ ? c + 1 : 0]);
          }
        }
      }
    }
    __syncthreads();
  }
  // groups added in order
  for (int g = 1; g < G; ++g) {
    if (grp == g) {
#pragma unroll
      for (int c = 0; c < NZ; ++c) red[ab * NZ + c] = acc[c];
    }
    __syncthreads();
    if (grp == 0) {
#pragma unroll
      for (int c = 0; c < NZ; ++c) acc[c] += red[ab * NZ + c];
    }
    __syncthreads();
  }
  if (grp == 0) {
#pragma unroll
    for (int c = 0; c < NZ; ++c) psw[(size_t)L * IPC + ab * NZ + c] += acc[c];
  }
}

// Applies the 1-D factors along axis AX of one tensor in shared memory, in
// place, by threads t, t + threads, ...: out[..i..] = sum_j A(i, j) in[..j..]. A
// thread owns whole lines along the axis and takes the factors as broadcasts,
// where one output a thread read both operands of every multiply-add from
// shared memory; it sums all M outputs at once (j outermost), so no multiply-add
// waits for the one before (two outputs at a time: 1,000 points, n = 6, parent
// to child 11.1 -> 9.3 us; 1M, n = 8, child to parent 91 -> 83 us). A at
// X[j * kXStride + i]. Elements (a, b, c) at ((a M) + b) S + c with an odd S
// (2-D: a S + b), so lines along the last axis do not share banks.
constexpr int kXStride = (kMaxNodes + 1) & ~1;
template <int M>
__host__ __device__ constexpr int line_stride() {
  return M | 1;
}
template <int DIM, int M>
__host__ __device__ constexpr int tensor_doubles() {
  return DIM == 2 ? M * line_stride<M>() : M * M * line_stride<M>();
}
template <int DIM, int M>
__device__ __forceinline__ int tensor_at(int o) {  // o: index in tensor order
  return o + (o / M) * (line_stride<M>() - M);
}
template <int DIM, int M, int AX>
__device__ __forceinline__ void apply_axis(double* buf, const double* X, int t, int threads) {
  constexpr int S = line_stride<M>();
  constexpr int LINES = DIM == 2 ? M : M * M;
  constexpr int STEP = AX == DIM - 1 ? 1 : (AX == DIM - 2 ? S : M * S);
  for (int l = t; l < LINES; l += threads) {
    int base;
    if (DIM == 2)
      base = AX == 0 ? l : l * S;
    else
      base = AX == 0 ? (l / M) * S + l % M : (AX == 1 ? (l / M) * M * S + l % M : l * S);
    double s[M];
#pragma unroll
    for (int i = 0; i < M; ++i) s[i] = 0.0;
#pragma unroll 3
    for (int j = 0; j < M; ++j) {
      const double v = buf[base + j * STEP];
      const double2* row = reinterpret_cast<const double2*>(X + j * kXStride);
#pragma unroll
      for (int i = 0; i < M; i += 2) {
        const double2 x = row[i / 2];
        s[i] = fma(x.x, v, s[i]);
        if (i + 1 < M) s[i + 1 < M ? i + 1 : 0] = fma(x.y, v, s[i + 1 < M ? i + 1 : 0]);
      }
    }
#pragma unroll
    for (int i = 0; i < M; ++i) buf[base + i * STEP] = s[i];
  }
}

// child_to_parent (src/upward_pass_impl.hpp:134-188): one block per parent,
// W_parent[a,b,c] += sum_children sum_{i,j,k} X[i][a] Y[j][b] Z[k][c] W_child[i,j,k].
// The children are transformed at the same time, kChildThreads threads each,
// and added in child order (one after the other by the whole block the upper
// levels, a block or a few, took 20 us a level). With `proxies` (the parents'
// places among the source proxies) the block also writes its parent's proxies
// as point sources: {node_x[a], node_y[b], node_z[c], W[k]}. 1,000 points, n = 6, 42 -> 14
// us; 1M, n = 8, 141 -> 81 us; 262k, n = 10, 251 -> 74 us.
constexpr int kChildThreads = 64;
template <int DIM, int M>
__global__ void __launch_bounds__(kChildThreads << DIM) k_c2p(const int* parents, const int* child, const double* xfer,
                                                            double* psw, const double* nodes_shift, double4* proxies) {
  constexpr int IPC = ipow_c<M, DIM>();
  constexpr int NCH = 1 << DIM, TD = tensor_doubles<DIM, M>();
  constexpr int XD = DIM * M * kXStride;
  extern __shared__ __align__(16) double c2p_smem[];  // per child: factors, tensor
  const int p = parents[blockIdx.x];
  const int ch = threadIdx.x / kChildThreads, t = threadIdx.x % kChildThreads;
  double* sX = c2p_smem + (size_t)ch * XD;
  double* buf = c2p_smem + (size_t)NCH * XD + (size_t)ch * TD;
  const int c = child[(size_t)p * NCH + ch];
  for (int o = t; o < IPC; o += kChildThreads) buf[tensor_at<DIM, M>(o)] = psw[(size_t)c * IPC + o];
  for (int o = t; o < DIM * M * M; o += kChildThreads) {
    const int d = o / (M * M), i = (o / M) % M, a = o % M;  // A(a, i) = X[i][a]
    sX[(d * M + i) * kXStride + a] = xfer[(size_t)c * kPanelXfer + (d * kMaxNodes + i) * kMaxNodes + a];
  }
  __syncthreads();
  apply_axis<DIM, M, 0>(buf, sX, t, kChildThreads);
  __syncthreads();
  apply_axis<DIM, M, 1>(buf, sX + M * kXStride, t, kChildThreads);
  __syncthreads();
  if constexpr (DIM == 3) {
    apply_axis<DIM, M, 2>(buf, sX + 2 * M * kXStride, t, kChildThreads);
    __syncthreads();
  }
  const double* all = c2p_smem + (size_t)NCH * XD;
  for (int o = threadIdx.x; o < IPC; o += blockDim.x) {
    const int at = tensor_at<DIM, M>(o);
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < NCH; ++k) s += all[(size_t)k * TD + at];
    s += psw[(size_t)p * IPC + o];
    psw[(size_t)p * IPC + o] = s;
    if (proxies) {
      const double* nd = nodes_shift + (size_t)p * kPanelNodes;
      const int c3 = o % M, b3 = (o / M) % M, a3 = o / (M * M);
      proxies[(size_t)blockIdx.x * IPC + o] =
          DIM == 3 ? make_double4(nd[a3], nd[kNodeStride + b3], nd[2 * kNodeStride + c3], s)
                   : make_double4(nd[b3], nd[kNodeStride + c3], 0.0, s);
    }
  }
}

// Source proxies as point sources: {node_x[a], node_y[b], node_z[c], W[k]}.
template <int DIM, int M>
__global__ void k_src_proxies(const int* cluster_panels, const double* nodes_shift, const double* psw, double4* out) {
  constexpr int IPC = ipow_c<M, DIM>();
  const int P = cluster_panels[blockIdx.x];
  const double* nd = nodes_shift + (size_t)P * kPanelNodes;
  for (int k = threadIdx.x; k < IPC; k += blockDim.x) {
    int a, b, c = 0;
    if (DIM == 2) {
      a = k / M;
      b = k % M;
    } else {
      a = k / (M * M);
      b = (k / M) % M;
      c = k % M;
    }
    out[(size_t)blockIdx.x * IPC + k] =
        make_double4(nd[a], nd[kNodeStride + b], DIM == 3 ? nd[2 * kNodeStride + c] : 0.0, psw[(size_t)P * IPC + k]);
  }
}

template <int DIM, int M>
__global__ void k_tgt_proxies(const int* cluster_panels, const double* nodes_shift, double4* out, int* out_index) {
  constexpr int IPC = ipow_c<M, DIM>();
  const int P = cluster_panels[blockIdx.x];
  const double* nd = nodes_shift + (size_t)P * kPanelNodes;
  for (int k = threadIdx.x; k < IPC; k += blockDim.x) {
    int a, b, c = 0;
    if (DIM == 2) {
      a = k / M;
      b = k % M;
    } else {
      a = k / (M * M);
      b = (k / M) % M;
      c = k % M;
    }
    out[(size_t)blockIdx.x * IPC + k] =
        make_double4(nd[a], nd[kNodeStride + b], DIM == 3 ? nd[2 * kNodeStride + c] : 0.0, 0.0);
    out_index[(size_t)blockIdx.x * IPC + k] = P * IPC + k;
  }
}

// ---- downward pass ---------------------------------------------------------
// parent_to_child (src/downward_pass_impl.hpp:109-191): one block per child and
// component (1M, potential + gradient, n = 8: 240 -> 151 us), Phi_child[i,j,k] += sum_{a,b,c} X[i][a] Y[j][b] Z[k][c] Phi_parent[a,b,c].
constexpr int kP2cThreads = 128;
template <int DIM, int M>
__global__ void __launch_bounds__(kP2cThreads) k_p2c(const int* children, const int* parent_of, const double* xfer,
                                                     Ptr4 ptw) {
  constexpr int IPC = ipow_c<M, DIM>();
  __shared__ __align__(16) double sX[DIM * M * kXStride];
  __shared__ double buf[tensor_doubles<DIM, M>()];
  const int c = children[blockIdx.x];
  const int p = parent_of[c], t = threadIdx.x;
  double* W = ptw.p[blockIdx.y];
  for (int o = t; o < IPC; o += kP2cThreads) buf[tensor_at<DIM, M>(o)] = W[(size_t)p * IPC + o];
  for (int o = t; o < DIM * M * M; o += kP2cThreads) {
    const int d = o / (M * M), i = (o / M) % M, a = o % M;  // A(i, a) = X[i][a]
    sX[(d * M + a) * kXStride + i] = xfer[(size_t)c * kPanelXfer + (d * kMaxNodes + i) * kMaxNodes + a];
  }
  __syncthreads();
  apply_axis<DIM, M, 0>(buf, sX, t, kP2cThreads);
  __syncthreads();
  apply_axis<DIM, M, 1>(buf, sX + M * kXStride, t, kP2cThreads);
  __syncthreads();
  if constexpr (DIM == 3) {
    apply_axis<DIM, M, 2>(buf, sX + 2 * M * kXStride, t, kP2cThreads);
    __syncthreads();
  }
  for (int o = t; o < IPC; o += kP2cThreads) W[(size_t)c * IPC + o] += buf[tensor_at<DIM, M>(o)];
}

// leaf_to_point (src/downward_pass_impl.hpp:193-237, 327-379) on every leaf:
// out[t] += sum_{a,b,c} Phi[a,b,c] Lx_a(x) Ly_b(y) Lz_c(z), one block per leaf.
// A thread takes a point; the leaf's weights come from shared memory two at a
// time (16-byte broadcasts of rows padded to an even length): with 8-byte loads
// the kernel was bound by them and by the basis' divisions (1M, n = 8, four
// components: 571 -> 447 us; 262k, n = 10, three: 326 -> 211 us; two points a
// thread leave too few warps, 502 us).
template <int DIM, int M>
__global__ void __launch_bounds__(128, M <= 8 ? 5 : 4) k_l2p(int ncomp, const int* leaves, const int* leaf_begin,
                                                             const int* point_count, const double4* pts,
                                                             const int* perm, const double* nodes_interp, Ptr4 ptw,
                                                             Ptr4 out) {
  constexpr int IPC = ipow_c<M, DIM>();
  constexpr int MP = (M + 1) & ~1, ROWS = IPC / M;
  extern __shared__ __align__(16) double sP[];  // [ncomp][ROWS][MP]
  __shared__ double snode[3][kMaxNodes], snode_s[3][kMaxNodes], sscale[3];
  const int L = leaves[blockIdx.x];
  const int b = leaf_begin[L], cnt = point_count[L];
  for (int comp = 0; comp < ncomp; ++comp)
    for (int o = threadIdx.x; o < IPC; o += blockDim.x)
      sP[(comp * ROWS + o / M) * MP + o % M] = ptw.p[comp][(size_t)L * IPC + o];
  load_nodes<DIM, M>(nodes_interp + (size_t)L * kPanelNodes, snode, snode_s, sscale);
  __syncthreads();
  for (int j = threadIdx.x; j < cnt; j += blockDim.x) {
    const double4 pt = pts[b + j];
    const int orig = perm[b + j];
    double Lx[M], Ly[M], Lz[DIM == 3 ? M : 1];
    bary_basis_fast<M>(Lx, pt.x, snode[0], snode_s[0], sscale[0]);
    bary_basis_fast<M>(Ly, pt.y, snode[1], snode_s[1], sscale[1]);
    if constexpr (DIM == 3) bary_basis_fast<M>(Lz, pt.z, snode[2], snode_s[2], sscale[2]);
    for (int comp = 0; comp < ncomp; ++comp) {
      const double* P = sP + comp * ROWS * MP;
      double phi = 0.0;
#pragma unroll
      for (int a = 0; a < M; ++a) {
        double ta = 0.0;
#pragma unroll
        for (int bb = 0; bb < M; ++bb) {
          double v;
          if constexpr (DIM == 2) {
            v = P[a * MP + bb];
          } else {
            const double2* row = reinterpret_cast<const double2*>(P + (a * M + bb) * MP);
            v = 0.0;
#pragma unroll
            for (int c = 0; c < M; c += 2) {
              const double2 w = row[c / 2];
              v = fma(w.x, Lz[c], v);
              if (c + 1 < M) v = fma(w.y, Lz[c + 1 < M ? c + 1 : 0], v);
            }
          }
          ta = fma(Ly[bb], v, ta);
        }
        phi = fma(Lx[a], ta, phi);
      }
      out.p[comp][orig] += phi;
    }
  }
}

}  // namespace

#define BTK_DISPATCH_M(degree, ...)         \
  switch (degree) {                          \
    case 1: { constexpr int M = 2; __VA_ARGS__; } break;   \
    case 2: { constexpr int M = 3; __VA_ARGS__; } break;   \
    case 3: { constexpr int M = 4; __VA_ARGS__; } break;   \
    case 4: { constexpr int M = 5; __VA_ARGS__; } break;   \
    case 5: { constexpr int M = 6; __VA_ARGS__; } break;   \
    case 6: { constexpr int M = 7; __VA_ARGS__; } break;   \
    case 7: { constexpr int M = 8; __VA_ARGS__; } break;   \
    case 8: { constexpr int M = 9; __VA_ARGS__; } break;   \
    case 9: { constexpr int M = 10; __VA_ARGS__; } break;  \
    case 10: { constexpr int M = 11; __VA_ARGS__; } break; \
    case 11: { constexpr int M = 12; __VA_ARGS__; } break; \
    case 12: { constexpr int M = 13; __VA_ARGS__; } break; \
    default: return cudaErrorInvalidValue;   \
  }

static inline int blocks_for(long long n, int t) { return (int)((n + t - 1) / t); }

cudaError_t launch_panel_geometry(int dim, int degree, int P, const DevPanel* panels, const double* ucos_shift,
                                  const double* ucos_interp, double* nodes_shift, double* nodes_interp, double* xfer,
                                  cudaStream_t s) {
  if (P <= 0) return cudaSuccess;
  const int m = degree + 1;
  k_panel_nodes<<<blocks_for((long long)P * dim * m, 256), 256, 0, s>>>(dim, m, P, panels, ucos_shift, ucos_interp,
                                                                        nodes_shift, nodes_interp);
  count_launch();
  BTK_DISPATCH_M(degree, k_panel_xfer<M><<<blocks_for((long long)P * dim * M, 128), 128, 0, s>>>(
                             dim, P, panels, nodes_shift, nodes_interp, xfer));
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_perm_from_inside(int n_leaves, const int* leaves, const int* leaf_begin, const int* point_count,
                                    const int* inside, int thresh, int* perm, cudaStream_t s) {
  if (n_leaves <= 0) return cudaSuccess;
  k_perm_from_inside<<<n_leaves, 128, 0, s>>>(leaves, leaf_begin, point_count, inside, thresh, perm);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_gather(int n, const int* perm, const double* x, const double* y, const double* z,
                          const double* w, double4* out, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_gather<<<blocks_for(n, 256), 256, 0, s>>>(n, perm, x, y, z, w, out);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_begin(const SolveBegin& b, int sms, cudaStream_t s) {
  long long most = std::max<long long>(b.ns, b.nt);
  for (int c = 0; c < 4; ++c) most = std::max(most, b.n_zero[c]);
  const int grid = (int)std::max<long long>(1, std::min<long long>((most + 255) / 256, (long long)sms * 8));
  k_begin<<<grid, 256, 0, s>>>(b);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_leaf_moments(int dim, int degree, int n_leaves, const int* leaves, const int* leaf_begin,
                                const int* point_count, const double4* pts, const double* nodes_interp, double* psw,
                                cudaStream_t s) {
  if (n_leaves <= 0) return cudaSuccess;
  if (dim == 2) {
    BTK_DISPATCH_M(degree, k_leaf_moments<2, M><<<n_leaves, 256, 0, s>>>(leaves, leaf_begin, point_count, pts,
                                                                         nodes_interp, psw));
  } else {
    BTK_DISPATCH_M(degree, k_leaf_moments<3, M><<<n_leaves, 256, 0, s>>>(leaves, leaf_begin, point_count, pts,
                                                                         nodes_interp, psw));
  }
  count_launch();
  return cudaGetLastError();
}

template <int DIM, int M>
static void launch_c2p_one(int n_parents, const int* parents, const int* child, const double* xfer, double* psw,
                           const double* nodes_shift, double4* proxies, cudaStream_t s) {
  const int shm = (int)sizeof(double) * (1 << DIM) * (DIM * M * kXStride + tensor_doubles<DIM, M>());
  cudaFuncSetAttribute(k_c2p<DIM, M>, cudaFuncAttributeMaxDynamicSharedMemorySize, shm);
  k_c2p<DIM, M><<<n_parents, kChildThreads << DIM, shm, s>>>(parents, child, xfer, psw, nodes_shift, proxies);
}

cudaError_t launch_c2p(int dim, int degree, int n_parents, const int* parents, const int* child, const double* xfer,
                       double* psw, const double* nodes_shift, double4* proxies, cudaStream_t s) {
  if (n_parents <= 0) return cudaSuccess;
  if (dim == 2) {
    BTK_DISPATCH_M(degree, (launch_c2p_one<2, M>(n_parents, parents, child, xfer, psw, nodes_shift, proxies, s)));
  } else {
    BTK_DISPATCH_M(degree, (launch_c2p_one<3, M>(n_parents, parents, child, xfer, psw, nodes_shift, proxies, s)));
  }
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_src_proxies(int dim, int degree, int n_clusters, const int* cluster_panels,
                               const double* nodes_shift, const double* psw, double4* out, cudaStream_t s) {
  if (n_clusters <= 0) return cudaSuccess;
  if (dim == 2) {
    BTK_DISPATCH_M(degree, k_src_proxies<2, M><<<n_clusters, 256, 0, s>>>(cluster_panels, nodes_shift, psw, out));
  } else {
    BTK_DISPATCH_M(degree, k_src_proxies<3, M><<<n_clusters, 256, 0, s>>>(cluster_panels, nodes_shift, psw, out));
  }
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_tgt_proxies(int dim, int degree, int n_clusters, const int* cluster_panels,
                               const double* nodes_shift, double4* out, int* out_index, cudaStream_t s) {
  if (n_clusters <= 0) return cudaSuccess;
  if (dim == 2) {
    BTK_DISPATCH_M(degree, k_tgt_proxies<2, M><<<n_clusters, 256, 0, s>>>(cluster_panels, nodes_shift, out, out_index));
  } else {
    BTK_DISPATCH_M(degree, k_tgt_proxies<3, M><<<n_clusters, 256, 0, s>>>(cluster_panels, nodes_shift, out, out_index));
  }
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_p2c(int dim, int degree, int ncomp, int n_children, const int* children, const int* parent_of,
                       const double* xfer, Ptr4 ptw, int /*ptw_stride*/, cudaStream_t s) {
  if (n_children <= 0) return cudaSuccess;
  if (dim == 2) {
    BTK_DISPATCH_M(degree, (k_p2c<2, M><<<dim3(n_children, ncomp), kP2cThreads, 0, s>>>(children, parent_of, xfer, ptw)));
  } else {
    BTK_DISPATCH_M(degree, (k_p2c<3, M><<<dim3(n_children, ncomp), kP2cThreads, 0, s>>>(children, parent_of, xfer, ptw)));
  }
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_l2p(int dim, int degree, int ncomp, int n_leaves, const int* leaves, const int* leaf_begin,
                       const int* point_count, const double4* pts, const int* perm, const double* nodes_interp,
                       Ptr4 ptw, Ptr4 out, cudaStream_t s) {
  if (n_leaves <= 0) return cudaSuccess;
  const int m = degree + 1;
  const size_t shm = sizeof(double) * ncomp * (dim == 2 ? m : m * m) * ((m + 1) & ~1);
  if (dim == 2) {
    BTK_DISPATCH_M(degree, {
      cudaFuncSetAttribute(k_l2p<2, M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm);
      k_l2p<2, M><<<n_leaves, 128, shm, s>>>(ncomp, leaves, leaf_begin, point_count, pts, perm, nodes_interp, ptw, out);
    });
  } else {
    BTK_DISPATCH_M(degree, {
      cudaFuncSetAttribute(k_l2p<3, M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm);
      k_l2p<3, M><<<n_leaves, 128, shm, s>>>(ncomp, leaves, leaf_begin, point_count, pts, perm, nodes_interp, ptw, out);
    });
  }
  count_launch();
  return cudaGetLastError();
}

}  // namespace btk
