// learned.cu -- training and use of the learned initializer.
//
// The network predicts a correction to the graph's pivot-MDS shape y (input
// features 0 and 1): the start is p = y + net(features), scaled to a
// predicted mean edge length.
//
// Training (bl_learned_train): the graphs of a training set form one
// block-diagonal graph on the device; their features come from one
// multi-source BFS and a pivot MDS per graph (features.cu).  Each target
// layout (what algo 4 produced for that graph) is centred and fitted to y by
// the similarity (scale times the Procrustes rotation or reflection) that
// minimises the squared distance; the network learns the residual
// fit(target) - y.  Full-batch Adam on sum_g mean_v |net_v - residual_v|^2 / G
// with the tcgen05 kernels of mpnn.cu.  A least-squares model
// log l = a + b log n + c log(mean degree) of the targets' mean edge length l
// gives the scale at inference.
//
// Use (bl_learned_init): features, one forward pass, p = y + net, scaled to
// the predicted mean edge length.  bl_learned_layout adds the refinement by Barnes-Hut
// iterations until a target energy is reached, and falls back to the greedy
// DFS start with the plain iteration count when the refined energy stays
// above the target.
#include <algorithm>
#include <chrono>
#include <cstdio>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/batchlayout_gb300.h"
#include "learned.h"
#include "mpnn.h"

namespace bl {

namespace {

// p = y + net (unscaled start) into pos
__global__ void residual_start_kernel(const float *__restrict__ net, const float *__restrict__ feat, int n,
                                      float2 *__restrict__ pos) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v < n) pos[v] = make_float2(net[2 * v] + feat[(size_t)v * kFeat], net[2 * v + 1] + feat[(size_t)v * kFeat + 1]);
}

// per block: sum over the CSR entries of |p_v - p_u| (each edge twice).  Bound
// by FP64, so the entries are dealt out in runs of kEdgeRun instead of by row:
// a warp with a row a lane works as long as its longest row (400,000 vertices
// of a geometric graph: 205 us by rows, 81 by runs).
constexpr int kEdgeRun = 8;

__global__ void edge_length_kernel(int n, const int *__restrict__ rowptr, const int *__restrict__ colids,
                                   const float2 *__restrict__ pos, double *part) {
  __shared__ double red[8];
  const int nnz = rowptr[n];
  double s = 0.0;
  for (long long e0 = (long long)kEdgeRun * (blockIdx.x * blockDim.x + threadIdx.x); e0 < nnz;
       e0 += (long long)kEdgeRun * gridDim.x * blockDim.x) {
    const int e1 = (int)min(e0 + kEdgeRun, (long long)nnz);
    int lo = 0, hi = n;  // the row of e0: rowptr[lo] <= e0 < rowptr[hi]
    while (hi - lo > 1) {
      const int mid = lo + ((hi - lo) >> 1);
      if (rowptr[mid] <= e0) lo = mid;
      else hi = mid;
    }
    int end = rowptr[lo + 1];
    float2 p = pos[lo];
    for (int e = (int)e0; e < e1; e++) {
      while (e >= end) {
        lo++;
        end = rowptr[lo + 1];
        p = pos[lo];
      }
      const float2 q = pos[colids[e]];
      s += sqrt((double)(p.x - q.x) * (p.x - q.x) + (double)(p.y - q.y) * (p.y - q.y));
    }
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += red[w];
    part[blockIdx.x] = t;
  }
}

// per block: sum_v A_v . R_v and sum_v |A_v|^2 with A_v the FR attraction
// sum_u W |p_u - p_v| (p_u - p_v) (algorithms.cpp:1056-1058) and R_v the
// Barnes-Hut sum of unit vectors towards the cells (BarnesHut.h:69-86).
// Bound by FP64: a warp takes 32 consecutive rows and forms the terms of their
// entries a lane each, kFitEntries at a time, so that the root and the products
// run in full warps; a lane then adds its row's terms in row order: 155 us for
// 400,000 vertices of a geometric graph, 272 with the whole row a lane's.
constexpr int kFitEntries = 192, kFitWarps = 8;

__global__ void __launch_bounds__(32 * kFitWarps) scale_fit_kernel(int n, const int *__restrict__ rowptr,
                                                                   const int *__restrict__ colids,
                                                                   const float2 *__restrict__ pos,
                                                                   const float2 *__restrict__ rep, float W,
                                                                   double *part) {
  __shared__ double red[2][8];
  __shared__ double2 term[kFitWarps][kFitEntries];
  __shared__ int first[kFitWarps][33];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double ar = 0.0, aa = 0.0;
  for (int v0 = 32 * (blockIdx.x * kFitWarps + warp); v0 < n; v0 += 32 * gridDim.x * kFitWarps) {
    const int v = v0 + lane, e0 = rowptr[min(v, n)], e1 = rowptr[min(v + 1, n)];
    __syncwarp();
    first[warp][lane] = e0;
    if (lane == 31) first[warp][32] = e1;
    __syncwarp();
    // (unsigned: a step past the last of 2^31 - 1 entries is compared too)
    const unsigned int base = first[warp][0], end = first[warp][32];
    double ax = 0.0, ay = 0.0;
    for (unsigned int c0 = base; c0 < end; c0 += kFitEntries) {
      const unsigned int c1 = min(c0 + kFitEntries, end);
      for (unsigned int e = c0 + lane; e < c1; e += 32) {
        int lo = 0;  // the row of e: first[lo] <= e < first[lo + 1]
#pragma unroll
        for (int h = 16; h > 0; h >>= 1)
          if ((unsigned int)first[warp][lo + h] <= e) lo += h;
        const float2 p = pos[v0 + lo], q = pos[colids[e]];
        const double dx = (double)q.x - p.x, dy = (double)q.y - p.y;
        const double sc = (double)W * sqrt(dx * dx + dy * dy);
        term[warp][e - c0] = make_double2(sc * dx, sc * dy);
      }
      __syncwarp();
      for (unsigned int e = max((unsigned int)e0, c0); e < min((unsigned int)e1, c1); e++) {
        const double2 t = term[warp][e - c0];
        ax += t.x;
        ay += t.y;
      }
      __syncwarp();
    }
    if (v < n) {
      const float2 r = rep[v];
      ar += ax * r.x + ay * r.y;
      aa += ax * ax + ay * ay;
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    ar += __shfl_xor_sync(0xffffffffu, ar, o);
    aa += __shfl_xor_sync(0xffffffffu, aa, o);
  }
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = ar;
    red[1][threadIdx.x >> 5] = aa;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double t0 = 0.0, t1 = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) {
      t0 += red[0][w];
      t1 += red[1][w];
    }
    part[2 * blockIdx.x] = t0;
    part[2 * blockIdx.x + 1] = t1;
  }
}

__global__ void scale_pos_kernel(float2 *pos, int n, float s) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v < n) pos[v] = make_float2(pos[v].x * s, pos[v].y * s);
}

__global__ void f32_to_bf16_kernel(const float *__restrict__ in, __nv_bfloat16 *__restrict__ out, long long n) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = __float2bfloat16_rn(in[i]);
}

// ---- the training set on the device ----------------------------------------------
//
// The graphs' edges joined into one CSR, and every target layout fitted to its
// graph's shape y = features 0 and 1.  A block takes a chunk of one graph, up
// to kFitChunk vertices or kEdgeChunk CSR entries (entries, not rows: the long
// rows of a power-law graph are neighbours).  Sums in FP64 in a fixed order
// (threads, warps, then chunks).  Twelve graphs of 207,796 vertices: the joined
// CSR 0.8 ms, the fit 0.2 (on the host 3.5, and 15.7 with its copies).
constexpr int kFitThreads = 256;
constexpr int kFitChunk = 512;
constexpr int kEdgeChunk = 4096;

struct FitArgs {
  const int4 *chunk;    // {graph, first vertex, end, -}
  const int *gchunk;    // first chunk of each graph, then their number
  const int4 *echunk;   // {graph, first CSR entry, end, -}
  const int *voff;
  const int *rowptr;    // joined
  int *colids;          // local ids, then joined
  const double2 *layout;
  const float *feat;
  double *sums;    // per chunk {x, y}
  double *length;  // per entry chunk: sum of the lengths
  double *cross;   // per chunk t^T y, row-major
  double *scales;  // per chunk {tR . y, |tR|^2}
  float2 *target;
  float *vweight;
  int num_graphs;
  int *bad;  // set when a colid is out of range
};

// every thread's v[K] summed over the block, in every thread
template <int K>
__device__ __forceinline__ void block_total(double (&v)[K]) {
  __shared__ double red[kFitThreads / 32][K];
  __syncthreads();
#pragma unroll
  for (int k = 0; k < K; k++) {
    for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][k] = v[k];
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < K; k++) {
    v[k] = 0.0;
    for (int w = 0; w < kFitThreads / 32; w++) v[k] += red[w][k];
  }
}

// the sum of a graph's chunks' K partials
template <int K>
__device__ __forceinline__ void graph_total(const FitArgs &a, int g, const double *part, double (&v)[K]) {
#pragma unroll
  for (int k = 0; k < K; k++) v[k] = 0.0;
  for (int c = a.gchunk[g] + threadIdx.x; c < a.gchunk[g + 1]; c += kFitThreads)
#pragma unroll
    for (int k = 0; k < K; k++) v[k] += part[(size_t)c * K + k];
  block_total<K>(v);
}

template <int K>
__device__ __forceinline__ void chunk_store(double (&v)[K], double *part) {
  block_total<K>(v);
  if (threadIdx.x == 0)
#pragma unroll
    for (int k = 0; k < K; k++) part[(size_t)blockIdx.x * K + k] = v[k];
}

__global__ void __launch_bounds__(kFitThreads) join_colids_kernel(FitArgs a) {
  const int4 c = a.echunk[blockIdx.x];
  const int v0 = a.voff[c.x], n = a.voff[c.x + 1] - v0;
  bool bad = false;
  for (unsigned int e = c.y + threadIdx.x; e < (unsigned int)c.z; e += kFitThreads) {
    const int u = a.colids[e];
    bad |= u < 0 || u >= n;
    a.colids[e] = v0 + u;
  }
  if (bad) *a.bad = 1;
}

__global__ void __launch_bounds__(kFitThreads) fit_length_kernel(FitArgs a) {
  const int4 c = a.echunk[blockIdx.x];
  constexpr int kRun = kEdgeChunk / kFitThreads;  // consecutive entries of a thread
  const unsigned int e0 = c.y + threadIdx.x * kRun, e1 = min(e0 + kRun, (unsigned int)c.z);
  double s[1] = {0.0};
  if (e0 < e1) {
    int lo = a.voff[c.x], hi = a.voff[c.x + 1];  // the row of e0: rowptr[lo] <= e0 < rowptr[hi]
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if ((unsigned int)a.rowptr[mid] <= e0) lo = mid;
      else hi = mid;
    }
    unsigned int end = a.rowptr[lo + 1];
    double2 p = a.layout[lo];
    for (unsigned int e = e0; e < e1; e++) {
      while (e >= end) {
        lo++;
        end = a.rowptr[lo + 1];
        p = a.layout[lo];
      }
      const double2 q = a.layout[a.colids[e]];
      const double dx = p.x - q.x, dy = p.y - q.y, d2 = fma(dx, dx, dy * dy);
      s[0] += d2 > 1e-280 && d2 < 1e300 ? sqrt(d2) : hypot(dx, dy);  // half the FP64 operations where it is safe
    }
  }
  chunk_store<1>(s, a.length);
}

__global__ void __launch_bounds__(kFitThreads) fit_sums_kernel(FitArgs a) {
  const int4 c = a.chunk[blockIdx.x];
  double s[2] = {0.0, 0.0};
  for (int v = c.y + threadIdx.x; v < c.z; v += kFitThreads) {
    const double2 p = a.layout[v];
    s[0] += p.x;
    s[1] += p.y;
  }
  chunk_store<2>(s, a.sums);
}

__device__ __forceinline__ double2 fit_mean(const FitArgs &a, int g) {
  double m[2];
  graph_total<2>(a, g, a.sums, m);
  const int n = a.voff[g + 1] - a.voff[g];
  return make_double2(m[0] / n, m[1] / n);
}

// orthogonal R (rotation or reflection) maximising tr(R^T M), M 2x2 row-major
__device__ __forceinline__ void fit_rotation(const FitArgs &a, int g, double R[4]) {
  double M[4];
  graph_total<4>(a, g, a.cross, M);
  __shared__ double rot[4];
  if (threadIdx.x == 0) {  // one warp's FP64 work, not the block's
    const double rs = M[2] - M[1], rc = M[0] + M[3], fs = M[1] + M[2], fc = M[0] - M[3];
    const double vr = hypot(rs, rc), vf = hypot(fs, fc);
    if (vr >= vf) {
      const double c = vr > 0.0 ? rc / vr : 1.0, s = vr > 0.0 ? rs / vr : 0.0;
      rot[0] = c; rot[1] = -s;
      rot[2] = s; rot[3] = c;
    } else {
      const double c = fc / vf, s = fs / vf;
      rot[0] = c; rot[1] = s;
      rot[2] = s; rot[3] = -c;
    }
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 4; k++) R[k] = rot[k];
}

__global__ void __launch_bounds__(kFitThreads) fit_cross_kernel(FitArgs a) {
  const int4 c = a.chunk[blockIdx.x];
  const double2 mean = fit_mean(a, c.x);
  double M[4] = {0.0, 0.0, 0.0, 0.0};
  for (int v = c.y + threadIdx.x; v < c.z; v += kFitThreads) {
    const double2 p = a.layout[v];
    const double tx = p.x - mean.x, ty = p.y - mean.y;
    const double y0 = a.feat[(size_t)v * kFeat], y1 = a.feat[(size_t)v * kFeat + 1];
    M[0] += tx * y0;
    M[1] += tx * y1;
    M[2] += ty * y0;
    M[3] += ty * y1;
  }
  chunk_store<4>(M, a.cross);
}

__global__ void __launch_bounds__(kFitThreads) fit_scale_kernel(FitArgs a) {
  const int4 c = a.chunk[blockIdx.x];
  const double2 mean = fit_mean(a, c.x);
  double R[4];
  fit_rotation(a, c.x, R);
  double s[2] = {0.0, 0.0};
  for (int v = c.y + threadIdx.x; v < c.z; v += kFitThreads) {
    const double2 p = a.layout[v];
    const double tx = p.x - mean.x, ty = p.y - mean.y;
    const double rx = tx * R[0] + ty * R[2], ry = tx * R[1] + ty * R[3];
    s[0] += rx * a.feat[(size_t)v * kFeat] + ry * a.feat[(size_t)v * kFeat + 1];
    s[1] += rx * rx + ry * ry;
  }
  chunk_store<2>(s, a.scales);
}

__global__ void __launch_bounds__(kFitThreads) fit_target_kernel(FitArgs a) {
  const int4 c = a.chunk[blockIdx.x];
  const double2 mean = fit_mean(a, c.x);
  double R[4], s[2];
  fit_rotation(a, c.x, R);
  graph_total<2>(a, c.x, a.scales, s);
  const double sc = s[1] > 0.0 ? s[0] / s[1] : 0.0;
  const float w = (float)(1.0 / ((double)a.num_graphs * (a.voff[c.x + 1] - a.voff[c.x])));
  for (int v = c.y + threadIdx.x; v < c.z; v += kFitThreads) {
    const double2 p = a.layout[v];
    const double tx = p.x - mean.x, ty = p.y - mean.y;
    const double rx = sc * (tx * R[0] + ty * R[2]), ry = sc * (tx * R[1] + ty * R[3]);
    a.target[v] = make_float2((float)(rx - a.feat[(size_t)v * kFeat]), (float)(ry - a.feat[(size_t)v * kFeat + 1]));
    a.vweight[v] = w;
  }
}

double wall_s() {
  using namespace std::chrono;
  return duration<double>(steady_clock::now().time_since_epoch()).count();
}

double predict_edge_length(const double *sm, int n, double mean_degree) {
  return std::exp(sm[0] + sm[1] * std::log((double)std::max(n, 1)) + sm[2] * std::log(std::max(mean_degree, 1e-3)));
}

}  // namespace

constexpr int kEdgeParts = 608;  // blocks of the two kernels over all entries

// Learned coordinates for the context's graph into ctx->pos.
int learned_init(bl_ctx *ctx, const float *params, const double *scale_model, int seed) {
  const int n = ctx->g.n;
  if (n < 2) return bl_fail(ctx, BL_ERR_ARG, "learned init needs at least two vertices");
  if (int rc = mpnn_set_params_device(ctx, params)) return rc;
  if (int rc = mpnn_prepare(ctx, n)) return rc;
  float *d_f = nullptr;
  unsigned short *d_d = nullptr;
  BL_CUDA(ctx, cudaMalloc(&d_f, sizeof(float) * kFeat * (size_t)n));
  if (cudaMalloc(&d_d, sizeof(unsigned short) * kPivots * (size_t)n) != cudaSuccess) {
    cudaFree(d_f);
    return bl_fail(ctx, BL_ERR_CUDA, "cudaMalloc");
  }
  int piv[kPivots];
  choose_pivots(n, (uint64_t)seed, piv);
  const int voff[2] = {0, n};
  int max_row = 0;
  for (int v = 0; v < n; v++) max_row = std::max(max_row, ctx->h_rowptr[v + 1] - ctx->h_rowptr[v]);
  int rc = compute_features(ctx, 1, voff, n, &max_row, ctx->g.rowptr, ctx->g.colids, piv, d_f, d_d);
  if (!rc) {
    f32_to_bf16_kernel<<<(int)((16LL * n + 255) / 256), 256, 0, ctx->stream>>>(d_f, mpnn_input(ctx), 16LL * n);
    ctx->launches++;
    rc = mpnn_forward(ctx, n, max_row, ctx->g.rowptr, ctx->g.colids, false);
  }
  if (!rc) {
    residual_start_kernel<<<(n + 255) / 256, 256, 0, ctx->stream>>>(mpnn_output(ctx), d_f, n, ctx->pos);
    double *d_part = nullptr;
    std::vector<double> part(kEdgeParts);
    if (cudaMalloc(&d_part, sizeof(double) * kEdgeParts) != cudaSuccess) rc = bl_fail(ctx, BL_ERR_CUDA, "cudaMalloc");
    if (!rc) {
      edge_length_kernel<<<kEdgeParts, 256, 0, ctx->stream>>>(n, ctx->g.rowptr, ctx->g.colids, ctx->pos, d_part);
      if (cudaMemcpyAsync(part.data(), d_part, sizeof(double) * kEdgeParts, cudaMemcpyDeviceToHost, ctx->stream) !=
              cudaSuccess ||
          cudaStreamSynchronize(ctx->stream) != cudaSuccess)
        rc = bl_fail(ctx, BL_ERR_CUDA, "learned init");
    }
    cudaFree(d_part);
    if (!rc) {
      double tot = 0.0;
      for (double x : part) tot += x;
      const double mean_len = ctx->g.nnz > 0 ? tot / (double)ctx->g.nnz : 0.0;
      const double want = predict_edge_length(scale_model, n, (double)ctx->g.nnz / n);
      const float sc = mean_len > 0.0 ? (float)(want / mean_len) : 1.0f;
      scale_pos_kernel<<<(n + 255) / 256, 256, 0, ctx->stream>>>(ctx->pos, n, sc);
      ctx->launches += 3;
    }
    // Energy-optimal scale of this shape: the Barnes-Hut repulsion R is
    // invariant under scaling (unit vectors, scale-free opening test) while
    // the attraction A grows with the square of the scale, so
    // sum_v |k^2 A_v - R_v|^2 is least at k^2 = sum A.R / sum |A|^2.
    if (!rc) rc = ensure_bh_scratch(ctx);
    if (!rc) rc = bh_build(ctx, ctx->pos, 1.2);
    if (!rc) rc = bh_traverse(ctx, 1.2, false, 0);
    if (!rc) {
      double *d_p2 = nullptr;
      std::vector<double> p2(2 * kEdgeParts);
      if (cudaMalloc(&d_p2, sizeof(double) * 2 * kEdgeParts) != cudaSuccess) rc = bl_fail(ctx, BL_ERR_CUDA, "cudaMalloc");
      if (!rc) {
        scale_fit_kernel<<<kEdgeParts, 32 * kFitWarps, 0, ctx->stream>>>(n, ctx->g.rowptr, ctx->g.colids, ctx->pos, ctx->s.rep,
                                                          (float)ctx->weight, d_p2);
        ctx->launches++;
        if (cudaMemcpyAsync(p2.data(), d_p2, sizeof(double) * 2 * kEdgeParts, cudaMemcpyDeviceToHost, ctx->stream) !=
                cudaSuccess ||
            cudaStreamSynchronize(ctx->stream) != cudaSuccess)
          rc = bl_fail(ctx, BL_ERR_CUDA, "learned init scale");
      }
      cudaFree(d_p2);
      if (!rc) {
        double ar = 0.0, aa = 0.0;
        for (int b = 0; b < kEdgeParts; b++) {
          ar += p2[2 * b];
          aa += p2[2 * b + 1];
        }
        if (ar > 0.0 && aa > 0.0) {
          scale_pos_kernel<<<(n + 255) / 256, 256, 0, ctx->stream>>>(ctx->pos, n, (float)std::sqrt(ar / aa));
          ctx->launches++;
        }
      }
    }
    if (!rc && cudaStreamSynchronize(ctx->stream) != cudaSuccess) rc = bl_fail(ctx, BL_ERR_CUDA, "learned init");
  }
  if (!rc) rc = bl_check_status(ctx);
  cudaFree(d_f);
  cudaFree(d_d);
  return rc;
}

}  // namespace bl

extern "C" {

int bl_learned_train(bl_ctx *ctx, int num_graphs, const int *vertex_offset, const long long *edge_offset,
                     const int *rowptr, const int *colids, const double *layouts, int epochs, double lr, int seed,
                     float *params, double *scale_model, double *loss_history) try {
  using namespace bl;
  if (!ctx || num_graphs < 1 || !vertex_offset || !edge_offset || !rowptr || !layouts || !params || !scale_model ||
      epochs < 0 || !(lr > 0))
    return BL_ERR_ARG;
  if (vertex_offset[0] != 0) return bl_fail(ctx, BL_ERR_ARG, "vertex_offset[0] must be 0");
  if (edge_offset[0] != 0 || edge_offset[num_graphs] < 0 || edge_offset[num_graphs] > 2147483647LL)
    return bl_fail(ctx, BL_ERR_ARG, "edge_offset must start at 0 and end within int32");
  if (edge_offset[num_graphs] > 0 && !colids) return bl_fail(ctx, BL_ERR_ARG, "null colids");
  for (int g = 0; g < num_graphs; g++)  // before the offsets size anything
    if ((long long)vertex_offset[g + 1] - vertex_offset[g] < 2)
      return bl_fail(ctx, BL_ERR_ARG, "graph " + std::to_string(g) + " has fewer than two vertices");
  BL_CUDA(ctx, cudaSetDevice(ctx->device));
  const int N = vertex_offset[num_graphs];
  const long long nnz = edge_offset[num_graphs];
  std::vector<int> grp(N + 1);
  std::vector<int> piv((size_t)num_graphs * kPivots);
  std::vector<double> logn(num_graphs), logd(num_graphs);
  std::vector<int> max_row(num_graphs, 0), gchunk(num_graphs + 1, 0);
  std::vector<int4> chunk, echunk;
  grp[0] = 0;
  for (int g = 0; g < num_graphs; g++) {
    const int v0 = vertex_offset[g], v1 = vertex_offset[g + 1], n = v1 - v0;
    if (n < 2) return bl_fail(ctx, BL_ERR_ARG, "graph " + std::to_string(g) + " has fewer than two vertices");
    const int *rp = rowptr + v0 + g;
    const long long e0 = edge_offset[g], m = edge_offset[g + 1] - e0;
    if (rp[0] != 0 || rp[n] != m) return bl_fail(ctx, BL_ERR_ARG, "rowptr does not match edge_offset");
    for (int v = 0; v < n; v++) {
      if (rp[v + 1] < rp[v]) return bl_fail(ctx, BL_ERR_ARG, "rowptr decreases");
      max_row[g] = std::max(max_row[g], rp[v + 1] - rp[v]);
      grp[v0 + v + 1] = (int)(e0 + rp[v + 1]);
    }
    for (int v = v0; v < v1; v += kFitChunk) chunk.push_back(make_int4(g, v, std::min(v + kFitChunk, v1), 0));
    gchunk[g + 1] = (int)chunk.size();
    for (long long e = e0; e < e0 + m; e += kEdgeChunk)
      echunk.push_back(make_int4(g, (int)e, (int)std::min(e + kEdgeChunk, e0 + m), 0));
    choose_pivots(n, (uint64_t)seed + (uint64_t)g, &piv[(size_t)g * kPivots]);
    for (int s = 0; s < kPivots; s++) piv[(size_t)g * kPivots + s] += v0;
    logn[g] = std::log((double)n);
    logd[g] = std::log(std::max((double)m / n, 1e-3));
  }
  const int nchunk = (int)chunk.size(), nechunk = (int)echunk.size();
  if (!ctx->s.status) {
    BL_CUDA(ctx, cudaMalloc(&ctx->s.status, sizeof(DevStatus)));
    BL_CUDA(ctx, cudaMemset(ctx->s.status, 0, sizeof(DevStatus)));
  }
  int *d_rp = nullptr, *d_ci = nullptr, *d_meta = nullptr;
  float *d_f = nullptr;
  double *d_lay = nullptr;
  unsigned short *d_d = nullptr;
  int rc = 0;
  auto ck = [&](cudaError_t e, const char *w) {
    if (e != cudaSuccess && !rc) rc = bl_cuda_fail(ctx, e, w);
  };
  FitArgs fit{};
  std::vector<double> logsig(num_graphs);
  const size_t meta = 4 * ((size_t)nchunk + nechunk) + 2 * ((size_t)num_graphs + 1) + 1;  // chunks, offsets, the flag
  ck(cudaMalloc(&d_rp, sizeof(int) * (N + 1)), "cudaMalloc");
  ck(cudaMalloc(&d_ci, sizeof(int) * (size_t)std::max<long long>(nnz, 1)), "cudaMalloc");
  ck(cudaMalloc(&d_meta, sizeof(int) * meta), "cudaMalloc");
  ck(cudaMalloc(&d_lay, sizeof(double) * (2 * (size_t)N + 8 * (size_t)nchunk + nechunk)), "cudaMalloc");
  if (!rc) {
    fit.chunk = reinterpret_cast<const int4 *>(d_meta);
    int4 *d_echunk = reinterpret_cast<int4 *>(d_meta) + nchunk;
    fit.echunk = d_echunk;
    int *d_gchunk = reinterpret_cast<int *>(d_echunk + nechunk), *d_voff = d_gchunk + num_graphs + 1;
    fit.gchunk = d_gchunk;
    fit.voff = d_voff;
    fit.bad = d_voff + num_graphs + 1;
    fit.rowptr = d_rp;
    fit.colids = d_ci;
    fit.layout = reinterpret_cast<const double2 *>(d_lay);
    fit.sums = d_lay + 2 * (size_t)N;
    fit.cross = fit.sums + 2 * (size_t)nchunk;
    fit.scales = fit.cross + 4 * (size_t)nchunk;
    fit.length = fit.scales + 2 * (size_t)nchunk;
    fit.num_graphs = num_graphs;
    ck(cudaMemcpyAsync(d_rp, grp.data(), sizeof(int) * (N + 1), cudaMemcpyHostToDevice, ctx->stream), "H2D");
    if (nnz) ck(cudaMemcpyAsync(d_ci, colids, sizeof(int) * (size_t)nnz, cudaMemcpyHostToDevice, ctx->stream), "H2D");
    ck(cudaMemcpyAsync(d_meta, chunk.data(), sizeof(int4) * nchunk, cudaMemcpyHostToDevice, ctx->stream), "H2D");
    if (nechunk)
      ck(cudaMemcpyAsync(d_echunk, echunk.data(), sizeof(int4) * nechunk, cudaMemcpyHostToDevice, ctx->stream), "H2D");
    ck(cudaMemcpyAsync(d_gchunk, gchunk.data(), sizeof(int) * (num_graphs + 1), cudaMemcpyHostToDevice, ctx->stream),
       "H2D");
    ck(cudaMemcpyAsync(d_voff, vertex_offset, sizeof(int) * (num_graphs + 1), cudaMemcpyHostToDevice, ctx->stream),
       "H2D");
    ck(cudaMemsetAsync(fit.bad, 0, sizeof(int), ctx->stream), "memset");
    int bad = 0;
    if (!rc && nechunk) join_colids_kernel<<<nechunk, kFitThreads, 0, ctx->stream>>>(fit);
    ctx->launches++;
    ck(cudaMemcpyAsync(&bad, fit.bad, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream), "D2H");
    ck(cudaStreamSynchronize(ctx->stream), "training set");
    if (!rc && bad) rc = bl_fail(ctx, BL_ERR_ARG, "colid out of range");
  }
  if (!rc) rc = mpnn_set_params_device(ctx, params);
  if (!rc) rc = mpnn_prepare(ctx, N);
  if (!rc) {
    ck(cudaMalloc(&d_f, sizeof(float) * kFeat * (size_t)N), "cudaMalloc");
    ck(cudaMalloc(&d_d, sizeof(unsigned short) * kPivots * (size_t)N), "cudaMalloc");
    ck(cudaMemcpyAsync(d_lay, layouts, sizeof(double) * 2 * (size_t)N, cudaMemcpyHostToDevice, ctx->stream), "H2D");
  }
  if (!rc)
    rc = compute_features(ctx, num_graphs, vertex_offset, N, max_row.data(), d_rp, d_ci, piv.data(), d_f, d_d);
  if (!rc) {
    fit.feat = d_f;
    fit.target = reinterpret_cast<float2 *>(mpnn_targets(ctx));
    fit.vweight = mpnn_vweights(ctx);
    if (nechunk) fit_length_kernel<<<nechunk, kFitThreads, 0, ctx->stream>>>(fit);
    fit_sums_kernel<<<nchunk, kFitThreads, 0, ctx->stream>>>(fit);
    fit_cross_kernel<<<nchunk, kFitThreads, 0, ctx->stream>>>(fit);
    fit_scale_kernel<<<nchunk, kFitThreads, 0, ctx->stream>>>(fit);
    fit_target_kernel<<<nchunk, kFitThreads, 0, ctx->stream>>>(fit);
    ctx->launches += 5;
    f32_to_bf16_kernel<<<(int)((16LL * N + 255) / 256), 256, 0, ctx->stream>>>(d_f, mpnn_input(ctx), 16LL * N);
    ctx->launches++;
    ck(cudaGetLastError(), "target fit");
  }
  const int longest = *std::max_element(max_row.begin(), max_row.end());
  for (int e = 0; e < epochs && !rc; e++) {
    const double lr_e = lr * 0.5 * (1.0 + std::cos(M_PI * e / std::max(epochs, 1)));
    rc = mpnn_forward(ctx, N, longest, d_rp, d_ci, true);
    if (!rc) rc = mpnn_backward(ctx, N, longest, d_rp, d_ci);
    double loss = 0.0;
    if (!rc && loss_history) rc = mpnn_loss(ctx, N, &loss);
    if (!rc && loss_history) loss_history[e] = loss;
    if (!rc) rc = mpnn_adam_step(ctx, lr_e);
  }
  // mean edge length of the targets (the scale model's data)
  std::vector<double> length(nechunk), el(num_graphs, 0.0);
  if (!rc && nechunk)
    ck(cudaMemcpyAsync(length.data(), fit.length, sizeof(double) * nechunk, cudaMemcpyDeviceToHost, ctx->stream), "D2H");
  if (!rc) ck(cudaStreamSynchronize(ctx->stream), "training");
  for (int c = 0; c < nechunk && !rc; c++) el[echunk[c].x] += length[c];
  for (int g = 0; g < num_graphs && !rc; g++) {
    const long long m = edge_offset[g + 1] - edge_offset[g];
    logsig[g] = std::log(std::max(m > 0 ? el[g] / (double)m : 1.0, 1e-300));
  }
  if (!rc) rc = bl_check_status(ctx);
  if (!rc) rc = bl_mpnn_get_params(ctx, params);
  if (!rc) {
    // log l = a + b log n + c log(mean degree), least squares (3x3 normal equations)
    double A[9] = {0}, bb[3] = {0};
    for (int g = 0; g < num_graphs; g++) {
      const double x[3] = {1.0, logn[g], logd[g]};
      for (int i = 0; i < 3; i++) {
        bb[i] += x[i] * logsig[g];
        for (int j = 0; j < 3; j++) A[i * 3 + j] += x[i] * x[j];
      }
    }
    for (int i = 0; i < 3; i++) A[i * 3 + i] += 1e-9 * (A[0] + 1.0);  // ridge for singular sets
    // Gaussian elimination with partial pivoting
    int p[3] = {0, 1, 2};
    for (int c = 0; c < 3; c++) {
      int best = c;
      for (int r = c + 1; r < 3; r++)
        if (std::fabs(A[p[r] * 3 + c]) > std::fabs(A[p[best] * 3 + c])) best = r;
      std::swap(p[c], p[best]);
      for (int r = c + 1; r < 3; r++) {
        const double f = A[p[r] * 3 + c] / A[p[c] * 3 + c];
        for (int k = c; k < 3; k++) A[p[r] * 3 + k] -= f * A[p[c] * 3 + k];
        bb[p[r]] -= f * bb[p[c]];
      }
    }
    double sol[3];
    for (int c = 2; c >= 0; c--) {
      double s = bb[p[c]];
      for (int k = c + 1; k < 3; k++) s -= A[p[c] * 3 + k] * sol[k];
      sol[c] = s / A[p[c] * 3 + c];
    }
    for (int i = 0; i < 3; i++) scale_model[i] = sol[i];
  }
  cudaFree(d_rp);
  cudaFree(d_ci);
  cudaFree(d_meta);
  cudaFree(d_lay);
  cudaFree(d_f);
  cudaFree(d_d);
  return rc;
} catch (...) {
  return bl_host_exception(ctx);
}

int bl_learned_load_model(const char *path, float *params, double *scale_model) try {
  if (!path || !params || !scale_model) return BL_ERR_ARG;
  FILE *f = std::fopen(path, "rb");
  if (!f) return BL_ERR_IO;
  char magic[8];
  unsigned char cnt[4];
  int rc = BL_OK;
  if (std::fread(magic, 1, 8, f) != 8 || std::memcmp(magic, "BLMPNN01", 8) != 0 || std::fread(cnt, 1, 4, f) != 4)
    rc = BL_ERR_IO;
  // little-endian fields, read byte by byte so the host's byte order does not matter
  const unsigned count = cnt[0] | (cnt[1] << 8) | (cnt[2] << 16) | ((unsigned)cnt[3] << 24);
  if (!rc && count != (unsigned)bl::kMpnnParams) rc = BL_ERR_IO;
  for (int i = 0; i < bl::kMpnnParams && !rc; i++) {
    unsigned char b[4];
    if (std::fread(b, 1, 4, f) != 4) {
      rc = BL_ERR_IO;
      break;
    }
    const uint32_t u = b[0] | (b[1] << 8) | (b[2] << 16) | ((uint32_t)b[3] << 24);
    std::memcpy(&params[i], &u, 4);
  }
  for (int i = 0; i < 3 && !rc; i++) {
    unsigned char b[8];
    if (std::fread(b, 1, 8, f) != 8) {
      rc = BL_ERR_IO;
      break;
    }
    uint64_t u = 0;
    for (int k = 7; k >= 0; k--) u = (u << 8) | b[k];
    std::memcpy(&scale_model[i], &u, 8);
  }
  std::fclose(f);
  // a non-finite weight or scale would give a start of NaNs: not a model
  for (int i = 0; i < bl::kMpnnParams && !rc; i++)
    if (!std::isfinite(params[i])) rc = BL_ERR_IO;
  for (int i = 0; i < 3 && !rc; i++)
    if (!std::isfinite(scale_model[i])) rc = BL_ERR_IO;
  return rc;
} catch (...) {
  return bl_host_exception(nullptr);
}

int bl_learned_init(bl_ctx *ctx, const float *params, const double *scale_model, int seed) try {
  if (!ctx || !params || !scale_model) return BL_ERR_ARG;
  BL_CUDA(ctx, cudaSetDevice(ctx->device));
  if (ctx->g.n < 2) return bl_fail(ctx, BL_ERR_STATE, "bl_learned_init needs a context with a graph");
  return bl::learned_init(ctx, params, scale_model, seed);
} catch (...) {
  return bl_host_exception(ctx);
}

int bl_learned_layout(bl_ctx *ctx, const float *params, const double *scale_model, int seed, int max_iterations,
                      int batch, double theta, double target_energy, double step0, double *out) try {
  using namespace bl;
  if (!ctx || !params || !scale_model || !out || max_iterations < 1 || batch < 1 || !(theta > 0) || !(step0 > 0))
    return BL_ERR_ARG;
  BL_CUDA(ctx, cudaSetDevice(ctx->device));
  if (ctx->g.n < 2) return bl_fail(ctx, BL_ERR_STATE, "bl_learned_layout needs a context with a graph");
  const double t0 = wall_s();
  if (int rc = learned_init(ctx, params, scale_model, seed)) return rc;
  const double t_init = wall_s() - t0;
  double e = HUGE_VAL, step = step0;
  int it = 0;
  while (it < max_iterations) {
    if (int rc = bh_run(ctx, 1, batch, theta, &step, &e)) return rc;  // STEP times 0.999
    it++;
    if (e <= target_energy) break;
  }
  int fell_back = 0;
  if (!(e <= target_energy)) {
    // the plain run: greedy DFS start, STEP from 1 (algorithms.cpp:1020-1072)
    if (int rc = bl_init_dfs(ctx)) return rc;
    step = 1.0;
    if (int rc = bh_run(ctx, max_iterations, batch, theta, &step, &e)) return rc;
    fell_back = 1;
  }
  BL_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  out[0] = e;
  out[1] = wall_s() - t0;
  out[2] = it;
  out[3] = fell_back;
  out[4] = t_init;
  return BL_OK;
} catch (...) {
  return bl_host_exception(ctx);
}

}  // extern "C"
