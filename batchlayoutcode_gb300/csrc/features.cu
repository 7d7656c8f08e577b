// features.cu -- the 16 input features of the learned initializer.
//
// A 3-layer message-passing network sees only 3 hops, so the features have
// to carry the global shape: they are pivot-MDS coordinates (Brandes & Pich,
// "Eigensolver methods for progressive multidimensional scaling of large
// data", 2006) from 16 pivots, plus degree features:
//   f[0..11]  the first 12 component scores of the double-centred squared
//             hop distances to the pivots, scaled so that component 1 has
//             unit mean square;
//   f[12]     log2(1 + deg), f[13] 1 / (1 + deg),
//   f[14]     mean of log2(1 + deg) over the neighbours,
//   f[15]     log2(n) / 20.
// Hop distances.  A graph with rows of at most 64 entries gets one block per
// pivot, which runs that breadth-first search by itself, the frontier and (up
// to 1.3 million vertices) the visited bits in shared memory, one block barrier
// a level: the graphs this engine lays out are mostly mesh-like, with hundreds
// to thousands of levels and frontiers of hundreds of vertices, where a level
// is a chain of round trips (400,000-vertex random geometric graph: 8.8 ms
// with one grid barrier a level over the whole device, 2.6 ms this way).
// Graphs with longer rows, and all graphs when a frontier outgrows a block's
// queue, take the device-wide form: one multi-source BFS over their pivots (a
// 16-bit visited mask per vertex, one level per grid-barrier step, the
// vertices of the level's frontier push their new source bits to their
// neighbours, which join the next frontier list the first time a bit reaches
// them); a block gathers its new frontier vertices in shared memory and
// reserves room for them in the global list with one atomic per level.
// Distances to pivots that a vertex cannot reach count as one more than the
// pivot's largest finite distance.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/batchlayout_gb300.h"
#include "learned.h"

namespace bl {

namespace {

constexpr int kP = kPivots;
constexpr unsigned short kUnreached = 0xFFFF;

__global__ void bfs_init_kernel(int n, unsigned int *visited, unsigned int *fr0, unsigned int *fr1) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= n) return;
  visited[v] = 0u;
  fr0[v] = 0u;
  fr1[v] = 0u;
}

// pivots[g * 16 + s]: global vertex of pivot s of graph g; the distinct pivot
// vertices of the listed graphs form the frontier list of level 0
__global__ void bfs_seed_kernel(int count, const int *list, const int *pivots, unsigned int *visited,
                                unsigned int *fr0, unsigned short *dist, int *wl0, unsigned int *cnt) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const int s = i % kP, p = pivots[list[i / kP] * kP + s];
  atomicOr(&visited[p], 1u << s);
  dist[(size_t)p * kP + s] = 0;
  if (atomicOr(&fr0[p], 1u << s) == 0u) wl0[atomicAdd(&cnt[0], 1u)] = p;
}

struct BfsArgs {
  int n;
  const int *rowptr, *colids;
  unsigned int *visited;
  unsigned int *fr[2];   // frontier masks: bits that reached the vertex at the level
  int *wl[2];            // frontier lists
  unsigned int *cnt;     // [3] list lengths, rotating by level
  unsigned short *dist;
  DevStatus *st;
  int max_levels;
};

constexpr int kBfsBuf = 2048;  // new frontier vertices a block gathers per level before spilling

// One cooperative launch, one level per bounded grid barrier.  Level L reads
// the list of level L-1 (fr[(L-1)&1], wl[(L-1)&1], cnt[(L-1)%3]) and builds
// the list of level L; a frontier vertex's mask is cleared once pushed, so a
// mask buffer holds only its own list's vertices.  Lists and masks written by
// other blocks are read through L2 (__ldcg) after the barrier.
__global__ void __launch_bounds__(512) msbfs_kernel(BfsArgs a) {
  __shared__ unsigned int s_count, s_n, s_base;
  __shared__ int s_buf[kBfsBuf];
  unsigned int epoch = 0;
  const unsigned int lane = threadIdx.x & 31u;
  const unsigned int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const unsigned int nwarps = (gridDim.x * blockDim.x) >> 5;
  for (int L = 1; L <= a.max_levels; L++) {
    const int cb = (L - 1) & 1, nbuf = L & 1;
    // one read per block; all appends preceded the barrier, so every block
    // sees the same value
    if (threadIdx.x == 0) {
      s_count = ld_acquire_gpu(&a.cnt[(L - 1) % 3]);
      s_n = 0u;
    }
    __syncthreads();
    const unsigned int count = s_count;
    if (count == 0u) break;
    if (blockIdx.x == 0 && threadIdx.x == 0) a.cnt[(L + 1) % 3] = 0u;  // untouched during this level
    // a warp per frontier vertex, a lane per neighbour: a level costs one
    // neighbour's chain of dependent L2 round trips, not deg of them
    for (unsigned int idx = wid; idx < count; idx += nwarps) {
      const int u = __ldcg(&a.wl[cb][idx]);
      const unsigned int m = __ldcg(&a.fr[cb][u]);
      const int e0 = a.rowptr[u], e1 = a.rowptr[u + 1];
      __syncwarp();
      if (lane == 0) a.fr[cb][u] = 0u;
      for (int e = e0 + lane; e < e1; e += 32) {
        const int v = a.colids[e];
        const unsigned int got = m & ~atomicOr(&a.visited[v], m);
        if (!got) continue;
        unsigned int b = got;
        while (b) {
          const int s = __ffs(b) - 1;
          b &= b - 1u;
          a.dist[(size_t)v * kP + s] = (unsigned short)min(L, 65534);
        }
        if (atomicOr(&a.fr[nbuf][v], got) == 0u) {
          const unsigned int slot = atomicAdd(&s_n, 1u);
          if (slot < (unsigned int)kBfsBuf) s_buf[slot] = v;
          else a.wl[nbuf][atomicAdd(&a.cnt[L % 3], 1u)] = v;  // rare spill
        }
      }
    }
    __syncthreads();
    const unsigned int mine = min(s_n, (unsigned int)kBfsBuf);
    if (threadIdx.x == 0 && mine) s_base = atomicAdd(&a.cnt[L % 3], mine);
    __syncthreads();
    for (unsigned int k = threadIdx.x; k < mine; k += blockDim.x) a.wl[nbuf][s_base + k] = s_buf[k];
    if (!grid_barrier(a.st, epoch)) return;
  }
}

// ---- one block per (graph, pivot) --------------------------------------------

constexpr int kBlockThreads = 1024;
// vertices of a frontier; a level of 8,192 vertices costs one block about
// what a level costs the whole device (10 us)
constexpr int kBlockQueue = 8192;
constexpr int kBlockEdges = 8;  // row entries a lane loads at a time, two lanes a row
// longest row taken: the level waits for the longest row of its frontier
constexpr int kBlockRow = 64;

struct BlockBfsArgs {
  const int *rowptr, *colids;
  const int *voff;    // [graphs + 1]
  const int *pivots;  // [graphs * 16]
  const int *list;    // graph of each 16 blocks
  unsigned short *dist;
  int *wide;  // set when a frontier outgrows the queue
  int bits;   // visited bits that fit in shared memory
};

struct BlockBfsSmem {
  int queue[2][kBlockQueue];
  int count[3];  // frontier sizes, rotating by level
};

__device__ __forceinline__ void prefetch_l1(const void *p) {
  asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}

// Bound by latency: per level one L2 round trip for the row entries (the row
// pointers are prefetched when a vertex is found), the shared-memory tests and
// appends of a row's entries side by side, one block barrier.
template <bool kBits>
__device__ __forceinline__ void bfs_block(const BlockBfsArgs &a, BlockBfsSmem &S, unsigned int *vis, int v0, int n,
                                          int pivot, int s) {
  const int tid = threadIdx.x, lane = tid & 31;
  const unsigned int lt = (1u << lane) - 1u;
  if (kBits)
    for (int k = tid; k < (n + 31) / 32; k += kBlockThreads) vis[k] = 0u;
  __syncthreads();
  if (tid == 0) {
    if (kBits) vis[pivot >> 5] = 1u << (pivot & 31);
    a.dist[(size_t)(v0 + pivot) * kP + s] = 0;
    S.queue[0][0] = pivot;
    S.count[0] = 1;
    S.count[1] = S.count[2] = 0;
  }
  __syncthreads();
  unsigned short *const dist = a.dist + (size_t)v0 * kP + s;
  int cur = 0, nxt = 1, third = 2;
  // every vertex enters the frontier once: at most n levels
  for (int L = 1; L <= n; L++) {
    const int count = S.count[cur];
    if (count == 0) return;
    if (count > kBlockQueue) {  // every thread sees the same count
      if (tid == 0) atomicExch(a.wide, 1);
      return;
    }
    if ((L & 63) == 0) {  // another block gave up
      if (__syncthreads_or(tid == 0 && ld_volatile_u32(reinterpret_cast<const unsigned int *>(a.wide)) != 0u)) return;
    }
    if (tid == 0) S.count[third] = 0;  // read as `cur` one level ago, appended to in the next one
    const int *q = S.queue[(L - 1) & 1];
    int *out = S.queue[L & 1];
    const unsigned short d = (unsigned short)min(L, 65534);
    for (int i0 = 0; i0 < 2 * count; i0 += kBlockThreads) {
      const int idx = (i0 + tid) >> 1;
      int e = 0, left = 0;  // the lane's next entry of its row, entries from there to the row's end
      if (idx < count) {
        const int u = v0 + q[idx];
        e = __ldg(&a.rowptr[u]) + (tid & 1);
        left = __ldg(&a.rowptr[u + 1]) - e;
      }
      while (__any_sync(0xffffffffu, left > 0)) {
        int v[kBlockEdges];
        unsigned int fresh = 0;
#pragma unroll
        for (int k = 0; k < kBlockEdges; k++) v[k] = 2 * k < left ? __ldg(&a.colids[(size_t)(unsigned int)e + 2 * k]) - v0 : -1;
        if (kBits) {
          unsigned int old[kBlockEdges];
#pragma unroll
          for (int k = 0; k < kBlockEdges; k++) old[k] = v[k] >= 0 ? vis[v[k] >> 5] : 0xffffffffu;
#pragma unroll
          for (int k = 0; k < kBlockEdges; k++)
            if (((old[k] >> (v[k] & 31)) & 1u) == 0u) old[k] = atomicOr(&vis[v[k] >> 5], 1u << (v[k] & 31));
#pragma unroll
          for (int k = 0; k < kBlockEdges; k++)
            if (((old[k] >> (v[k] & 31)) & 1u) == 0u) {
              fresh |= 1u << k;
              dist[(size_t)v[k] * kP] = d;
            }
        } else {
          unsigned short old[kBlockEdges];
#pragma unroll
          for (int k = 0; k < kBlockEdges; k++) {
            old[k] = 0;
            if (v[k] >= 0) old[k] = atomicCAS(&dist[(size_t)v[k] * kP], kUnreached, d);
          }
#pragma unroll
          for (int k = 0; k < kBlockEdges; k++)
            if (old[k] == kUnreached) fresh |= 1u << k;
        }
        // appended to the next frontier, one shared atomic a warp
        unsigned int b[kBlockEdges];
        int total = 0;
#pragma unroll
        for (int k = 0; k < kBlockEdges; k++) {
          b[k] = __ballot_sync(0xffffffffu, (fresh >> k) & 1u);
          total += __popc(b[k]);
        }
        if (total) {
          int slot = 0;
          if (lane == 0) slot = atomicAdd(&S.count[nxt], total);
          slot = __shfl_sync(0xffffffffu, slot, 0);
#pragma unroll
          for (int k = 0; k < kBlockEdges; k++) {
            const int x = slot + __popc(b[k] & lt);
            if (((fresh >> k) & 1u) && x < kBlockQueue) {
              out[x] = v[k];
              prefetch_l1(&a.rowptr[v0 + v[k]]);
            }
            slot += __popc(b[k]);
          }
        }
        e = (int)((unsigned int)e + 2 * kBlockEdges);
        left -= 2 * kBlockEdges;
      }
    }
    __syncthreads();
    const int t = cur;
    cur = nxt;
    nxt = third;
    third = t;
  }
}

__global__ void __launch_bounds__(kBlockThreads, 1) bfs_block_kernel(BlockBfsArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  BlockBfsSmem &S = *reinterpret_cast<BlockBfsSmem *>(smem_raw);
  unsigned int *vis = reinterpret_cast<unsigned int *>(smem_raw + sizeof(BlockBfsSmem));
  const int g = a.list[blockIdx.x / kP], s = blockIdx.x % kP;
  const int v0 = a.voff[g], n = a.voff[g + 1] - v0;
  const int pivot = a.pivots[g * kP + s] - v0;
  if (n <= a.bits) bfs_block<true>(a, S, vis, v0, n, pivot, s);
  else bfs_block<false>(a, S, vis, v0, n, pivot, s);
}

// ---- pivot MDS of one graph (vertices [v0, v1)) ---------------------------
// The squared distance: squared as an integer (at most 65,535 hops) and made a
// double by its bits above 2^52, one FP64 operation instead of a conversion and
// a product: FP64 runs at two lanes a cycle and SM here and bounds these kernels.
__device__ __forceinline__ double hop2(unsigned int d, int s, const int *maxd) {
  const unsigned int h = d == kUnreached ? (unsigned int)(maxd[s] + 1) : d;
  return __hiloint2double(0x43300000, (int)(h * h)) - 4503599627370496.0;
}

// a vertex's 16 hop counts, two loads
__device__ __forceinline__ void hops(const unsigned short *dist, int v, unsigned int (&d)[kP]) {
  const uint4 *row = reinterpret_cast<const uint4 *>(dist + (size_t)v * kP);
  const uint4 x[2] = {row[0], row[1]};
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const unsigned int w[4] = {x[k].x, x[k].y, x[k].z, x[k].w};
#pragma unroll
    for (int i = 0; i < 4; i++) {
      d[8 * k + 2 * i] = w[i] & 0xffffu;
      d[8 * k + 2 * i + 1] = w[i] >> 16;
    }
  }
}

// The pivot MDS of a slice of graphs: blockIdx.y is the graph of the slice,
// mds_blocks(n) blocks of blockIdx.x work on its n vertices.  Everything
// between the distances and the 16 x 16 eigenproblem stays on the device, all
// graphs at once: 1.0 ms for twelve graphs, the eigenproblems included (2.3
// with a host reduction and its synchronisation after each of three kernels a
// graph).
constexpr int kMdsBlocks = 256;
constexpr int kMdsSlice = 64;        // graphs a launch: bounds the partials' memory
constexpr int kGram = kP * (kP + 1) / 2;
constexpr int kMean = kP + 1;        // a graph's column means, then their mean

__host__ __device__ __forceinline__ int mds_blocks(int n) {
  const int b = (n + 255) / 256;
  return b < kMdsBlocks ? b : kMdsBlocks;
}

// hop maxima of every pivot into maxd (zero before)
__global__ void mds_max_kernel(const int *voff, const unsigned short *dist, int *maxd) {
  const int g = blockIdx.y, v0 = voff[g], v1 = voff[g + 1], blocks = mds_blocks(v1 - v0);
  if ((int)blockIdx.x >= blocks) return;
  __shared__ int smax[kP];
  if (threadIdx.x < kP) smax[threadIdx.x] = 0;
  __syncthreads();
  int m[kP];
#pragma unroll
  for (int s = 0; s < kP; s++) m[s] = 0;
  for (int v = v0 + blockIdx.x * blockDim.x + threadIdx.x; v < v1; v += blocks * blockDim.x) {
    unsigned int h[kP];
    hops(dist, v, h);
#pragma unroll
    for (int s = 0; s < kP; s++) {
      if (h[s] != kUnreached) m[s] = max(m[s], (int)h[s]);
    }
  }
#pragma unroll
  for (int s = 0; s < kP; s++) atomicMax(&smax[s], m[s]);
  __syncthreads();
  if (threadIdx.x < kP) atomicMax(&maxd[g * kP + threadIdx.x], smax[threadIdx.x]);
}

__device__ void block_sum_doubles(double *vals, int count, double *scratch, double *out) {
  // scratch: blockDim.x / 32 * count doubles; out: count doubles (thread 0 writes)
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int k = 0; k < count; k++) {
    double v = vals[k];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) scratch[w * count + k] = v;
  }
  __syncthreads();
  for (int k = threadIdx.x; k < count; k += blockDim.x) {
    double s = 0.0;
    for (int j = 0; j < nw; j++) s += scratch[j * count + k];
    out[k] = s;
  }
}

// per block: column sums of the squared distances
__global__ void __launch_bounds__(256) mds_colsum_kernel(const int *voff, const unsigned short *dist, const int *maxds,
                                                         double *part) {
  const int g = blockIdx.y, v0 = voff[g], v1 = voff[g + 1], blocks = mds_blocks(v1 - v0);
  if ((int)blockIdx.x >= blocks) return;
  const int *maxd = maxds + g * kP;
  __shared__ double scratch[8 * kP];
  double c[kP];
#pragma unroll
  for (int s = 0; s < kP; s++) c[s] = 0.0;
  for (int v = v0 + blockIdx.x * blockDim.x + threadIdx.x; v < v1; v += blocks * blockDim.x) {
    unsigned int h[kP];
    hops(dist, v, h);
#pragma unroll
    for (int s = 0; s < kP; s++) c[s] += hop2(h[s], s, maxd);
  }
  block_sum_doubles(c, kP, scratch, part + ((size_t)g * kMdsBlocks + blockIdx.x) * kP);
}

// the means from the blocks' sums, added in block order
__global__ void mds_mean_kernel(const int *voff, const double *part, double *mean) {
  const int g = blockIdx.x, n = voff[g + 1] - voff[g], blocks = mds_blocks(n), s = threadIdx.x;
  __shared__ double m[kP];
  if (s < kP) {
    double t = 0.0;
#pragma unroll 8
    for (int b = 0; b < blocks; b++) t += part[((size_t)g * kMdsBlocks + b) * kP + s];
    m[s] = t / n;
    mean[g * kMean + s] = m[s];
  }
  __syncthreads();
  if (s == 0) {
    double grand = 0.0;
    for (int k = 0; k < kP; k++) grand += m[k];
    mean[g * kMean + kP] = grand / kP;
  }
}

// per block: Gram matrix sum_v C_v C_v^T of the double-centred rows
// C[v][s] = -0.5 (D2[v][s] - r_v - c_s + g), upper triangle (136 values):
// a tile of 256 rows is staged in shared memory, thread t < 136 owns entry t.
__global__ void __launch_bounds__(256) mds_gram_kernel(const int *voff, const unsigned short *dist, const int *maxds,
                                                       const double *mean, double *part) {
  const int g = blockIdx.y, v0 = voff[g], v1 = voff[g + 1], blocks = mds_blocks(v1 - v0);
  if ((int)blockIdx.x >= blocks) return;
  const int *maxd = maxds + g * kP;
  const double *colmean = mean + g * kMean;
  const double grand = colmean[kP];
  __shared__ double cbuf[256][kP + 1];
  const int tid = threadIdx.x;
  int pi = 0, pj = 0;
  if (tid < kGram) {
    int k = tid, i = 0;
    while (k >= kP - i) {
      k -= kP - i;
      i++;
    }
    pi = i;
    pj = i + k;
  }
  double acc = 0.0;
  for (int base = v0 + blockIdx.x * 256; base < v1; base += blocks * 256) {
    const int v = base + tid;
    if (v < v1) {
      double d2[kP], r = 0.0;
      unsigned int h[kP];
      hops(dist, v, h);
#pragma unroll
      for (int s = 0; s < kP; s++) {
        d2[s] = hop2(h[s], s, maxd);
        r += d2[s];
      }
      r *= 1.0 / kP;
#pragma unroll
      for (int s = 0; s < kP; s++) cbuf[tid][s] = d2[s] - r - colmean[s] + grand;  // x -0.5 at the end: exact
    } else {
#pragma unroll
      for (int s = 0; s < kP; s++) cbuf[tid][s] = 0.0;
    }
    __syncthreads();
    if (tid < kGram)
      for (int rr = 0; rr < 256; rr++) acc = fma(cbuf[rr][pi], cbuf[rr][pj], acc);
    __syncthreads();
  }
  if (tid < kGram) part[((size_t)g * kMdsBlocks + blockIdx.x) * kGram + tid] = 0.25 * acc;
}

// the Gram matrices from the blocks' sums, added in block order
__global__ void mds_gram_sum_kernel(const int *voff, const double *part, double *gram) {
  const int g = blockIdx.x, blocks = mds_blocks(voff[g + 1] - voff[g]), k = threadIdx.x;
  if (k >= kGram) return;
  double t = 0.0;
#pragma unroll 8
  for (int b = 0; b < blocks; b++) t += part[((size_t)g * kMdsBlocks + b) * kGram + k];
  gram[g * kGram + k] = t;
}

struct ProjectArgs {
  const int *voff;    // of the slice's graphs
  const int *rowptr;  // global CSR
  const int *colids;
  const unsigned short *dist;
  const int *maxd;
  const double *mean;  // column means, then their mean
  const double *V;     // 16 x 12 and the scale's inverse: column j = eigenvector j
  float *features;     // global n x 16
};
constexpr int kProj = kP * 12 + 1;

__global__ void mds_project_kernel(ProjectArgs a) {
  const int g = blockIdx.y, n_graph = a.voff[g + 1] - a.voff[g];
  const int v = a.voff[g] + blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= a.voff[g + 1]) return;
  a.maxd += g * kP;
  a.mean += g * kMean;
  a.V += (size_t)g * kProj;
  const double inv_scale = -0.5 * a.V[kP * 12];
  double d2[kP], r = 0.0;
  unsigned int h[kP];
  hops(a.dist, v, h);
#pragma unroll
  for (int s = 0; s < kP; s++) {
    d2[s] = hop2(h[s], s, a.maxd);
    r += d2[s];
  }
  r *= 1.0 / kP;
  double c[kP];
#pragma unroll
  for (int s = 0; s < kP; s++) c[s] = d2[s] - r - a.mean[s] + a.mean[kP];  // x -0.5 below: exact
  float f[kFeat];
#pragma unroll
  for (int j = 0; j < 12; j++) {
    double y = 0.0;
#pragma unroll
    for (int s = 0; s < kP; s++) y = fma(c[s], a.V[s * 12 + j], y);
    f[j] = (float)(y * inv_scale);
  }
  const int e0 = a.rowptr[v], e1 = a.rowptr[v + 1];
  const int deg = e1 - e0;
  float m = 0.f;
  for (int e = 0; e < deg; e += 8) {  // eight neighbours' loads together, added in row order
    int u[8], d[8];
#pragma unroll
    for (int q = 0; q < 8; q++) u[q] = e + q < deg ? a.colids[e0 + e + q] : v;
#pragma unroll
    for (int q = 0; q < 8; q++) d[q] = a.rowptr[u[q] + 1] - a.rowptr[u[q]];
#pragma unroll
    for (int q = 0; q < 8; q++)
      if (e + q < deg) m += log2f(1.0f + (float)d[q]);
  }
  f[12] = log2f(1.0f + (float)deg);
  f[13] = 1.0f / (1.0f + (float)deg);
  f[14] = deg > 0 ? m / (float)deg : 0.0f;
  f[15] = log2f((float)n_graph) / 20.0f;
  float4 *out = reinterpret_cast<float4 *>(a.features + (size_t)v * kFeat);
#pragma unroll
  for (int k = 0; k < kFeat / 4; k++) out[k] = make_float4(f[4 * k], f[4 * k + 1], f[4 * k + 2], f[4 * k + 3]);
}

}  // namespace

// splitmix64 (Steele, Lea & Flood, "Fast splittable pseudorandom number
// generators", 2014)
static uint64_t splitmix64(uint64_t &x) {
  uint64_t z = (x += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

void choose_pivots(int n, uint64_t seed, int *out) {
  uint64_t x = seed;
  int k = 0;
  if (n <= kP) {
    for (int s = 0; s < kP; s++) out[s] = s % n;
    return;
  }
  while (k < kP) {
    const int p = (int)(splitmix64(x) % (uint64_t)n);
    bool dup = false;
    for (int j = 0; j < k; j++) dup |= out[j] == p;
    if (!dup) out[k++] = p;
  }
}

// Cyclic Jacobi eigenvalue iteration (Golub & Van Loan, "Matrix Computations",
// section 8.5) for a symmetric m x m matrix; eigenvalues descending, column j
// of V the eigenvector of eigenvalue j with its largest-magnitude entry
// positive.
void jacobi_eigen(int m, std::vector<double> A, std::vector<double> &lam, std::vector<double> &V) {
  V.assign(m * m, 0.0);
  for (int i = 0; i < m; i++) V[i * m + i] = 1.0;
  for (int sweep = 0; sweep < 100; sweep++) {
    double off = 0.0, tot = 0.0;
    for (int i = 0; i < m; i++)
      for (int j = 0; j < m; j++) {
        tot += A[i * m + j] * A[i * m + j];
        if (i != j) off += A[i * m + j] * A[i * m + j];
      }
    if (off <= 1e-30 * tot || off == 0.0) break;
    for (int p = 0; p < m; p++)
      for (int q = p + 1; q < m; q++) {
        const double apq = A[p * m + q];
        if (apq == 0.0) continue;
        const double theta = (A[q * m + q] - A[p * m + p]) / (2.0 * apq);
        const double t = (theta >= 0 ? 1.0 : -1.0) / (std::fabs(theta) + std::sqrt(theta * theta + 1.0));
        const double c = 1.0 / std::sqrt(t * t + 1.0), s = t * c;
        for (int k = 0; k < m; k++) {
          const double akp = A[k * m + p], akq = A[k * m + q];
          A[k * m + p] = c * akp - s * akq;
          A[k * m + q] = s * akp + c * akq;
        }
        for (int k = 0; k < m; k++) {
          const double apk = A[p * m + k], aqk = A[q * m + k];
          A[p * m + k] = c * apk - s * aqk;
          A[q * m + k] = s * apk + c * aqk;
        }
        for (int k = 0; k < m; k++) {
          const double vkp = V[k * m + p], vkq = V[k * m + q];
          V[k * m + p] = c * vkp - s * vkq;
          V[k * m + q] = s * vkp + c * vkq;
        }
      }
  }
  std::vector<int> idx(m);
  for (int i = 0; i < m; i++) idx[i] = i;
  std::stable_sort(idx.begin(), idx.end(), [&](int x, int y) { return A[x * m + x] > A[y * m + y]; });
  std::vector<double> V2(m * m);
  lam.assign(m, 0.0);
  for (int j = 0; j < m; j++) {
    const int c = idx[j];
    lam[j] = A[c * m + c];
    int arg = 0;
    for (int k = 1; k < m; k++)
      if (std::fabs(V[k * m + c]) > std::fabs(V[arg * m + c])) arg = k;
    const double sg = V[arg * m + c] < 0 ? -1.0 : 1.0;
    for (int k = 0; k < m; k++) V2[k * m + j] = sg * V[k * m + c];
  }
  V = V2;
}

// Features of the graphs [voff[g], voff[g+1]) of a block-diagonal device CSR.
// max_row[g]: the graph's longest row.
int compute_features(bl_ctx *ctx, int num_graphs, const int *voff, int n, const int *max_row, const int *d_rowptr,
                     const int *d_colids, const int *pivots, float *d_features, unsigned short *d_dist) {
  cudaStream_t st = ctx->stream;
  const int P = num_graphs * kP;
  unsigned int *visited = nullptr, *fr0 = nullptr, *fr1 = nullptr, *cnt = nullptr;
  int *d_piv = nullptr, *d_maxd = nullptr, *wl0 = nullptr, *wl1 = nullptr, *d_voff = nullptr;
  double *d_part = nullptr, *d_mean = nullptr, *d_gram = nullptr, *d_V = nullptr;
  const int slice = std::min(num_graphs, kMdsSlice);
  int rc = 0;
  auto cleanup = [&]() {
    cudaFree(visited); cudaFree(fr0); cudaFree(fr1); cudaFree(cnt); cudaFree(wl0); cudaFree(wl1);
    cudaFree(d_piv); cudaFree(d_maxd); cudaFree(d_voff);
    cudaFree(d_part); cudaFree(d_mean); cudaFree(d_gram); cudaFree(d_V);
  };
  auto ck = [&](cudaError_t e, const char *w) {
    if (e != cudaSuccess && !rc) rc = bl_cuda_fail(ctx, e, w);
    return rc == 0;
  };
  // graphs by the form of their search: blocks first
  std::vector<int> list;
  for (int k = 0; k < 2; k++)
    for (int g = 0; g < num_graphs; g++)
      if ((max_row[g] <= kBlockRow) == (k == 0)) list.push_back(g);
  int nblock = 0, largest = 0;
  for (int g = 0; g < num_graphs; g++)
    if (max_row[g] <= kBlockRow) {
      nblock++;
      largest = std::max(largest, voff[g + 1] - voff[g]);
    }
  ck(cudaMalloc(&cnt, 4 * sizeof(unsigned int)), "cudaMalloc");
  ck(cudaMalloc(&d_voff, sizeof(int) * (2 * num_graphs + 1)), "cudaMalloc");
  ck(cudaMalloc(&d_piv, sizeof(int) * P), "cudaMalloc");
  ck(cudaMalloc(&d_maxd, sizeof(int) * kP * slice), "cudaMalloc");
  ck(cudaMalloc(&d_part, sizeof(double) * kMdsBlocks * kGram * (size_t)slice), "cudaMalloc");
  ck(cudaMalloc(&d_mean, sizeof(double) * kMean * slice), "cudaMalloc");
  ck(cudaMalloc(&d_gram, sizeof(double) * kGram * slice), "cudaMalloc");
  ck(cudaMalloc(&d_V, sizeof(double) * kProj * slice), "cudaMalloc");
  if (rc) {
    cleanup();
    return rc;
  }
  ck(cudaMemcpyAsync(d_piv, pivots, sizeof(int) * P, cudaMemcpyHostToDevice, st), "H2D");
  int *d_list = d_voff + num_graphs + 1;
  ck(cudaMemcpyAsync(d_voff, voff, sizeof(int) * (num_graphs + 1), cudaMemcpyHostToDevice, st), "H2D");
  ck(cudaMemcpyAsync(d_list, list.data(), sizeof(int) * num_graphs, cudaMemcpyHostToDevice, st), "H2D");
  ck(cudaMemsetAsync(cnt, 0, 4 * sizeof(unsigned int), st), "memset");  // list lengths, then the give-up flag
  ck(cudaMemsetAsync(d_dist, 0xff, sizeof(unsigned short) * kP * (size_t)n, st), "memset");
  if (!rc && nblock > 0) {
    int optin = 0, wide = 0;
    ck(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device), "attribute");
    const int room = (optin - 1024 - (int)sizeof(BlockBfsSmem)) / 4;  // words of visited bits
    const int words = std::min(room, (largest + 31) / 32);
    const size_t smem = sizeof(BlockBfsSmem) + 4 * (size_t)words;
    ck(cudaFuncSetAttribute(bfs_block_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), "attribute");
    BlockBfsArgs b{d_rowptr, d_colids, d_voff, d_piv, d_list, d_dist, reinterpret_cast<int *>(cnt + 3), 32 * words};
    bl_time_begin(ctx, "msbfs_kernel");
    if (!rc) bfs_block_kernel<<<nblock * kP, kBlockThreads, smem, st>>>(b);
    bl_time_end(ctx, "msbfs_kernel");
    ctx->launches++;
    ck(cudaGetLastError(), "BFS launch");
    ck(cudaMemcpyAsync(&wide, cnt + 3, sizeof(int), cudaMemcpyDeviceToHost, st), "D2H");
    ck(cudaStreamSynchronize(st), "BFS");
    if (!rc && wide) {  // a frontier outgrew a block's queue: every graph device-wide, from the start
      nblock = 0;
      ck(cudaMemsetAsync(d_dist, 0xff, sizeof(unsigned short) * kP * (size_t)n, st), "memset");
    }
  }
  if (!rc && nblock < num_graphs) {
    ck(cudaMalloc(&visited, sizeof(unsigned int) * n), "cudaMalloc");
    ck(cudaMalloc(&fr0, sizeof(unsigned int) * n), "cudaMalloc");
    ck(cudaMalloc(&fr1, sizeof(unsigned int) * n), "cudaMalloc");
    ck(cudaMalloc(&wl0, sizeof(int) * n), "cudaMalloc");
    ck(cudaMalloc(&wl1, sizeof(int) * n), "cudaMalloc");
    if (rc) {
      cleanup();
      return rc;
    }
    const int seeds = (num_graphs - nblock) * kP;
    bfs_init_kernel<<<(n + 255) / 256, 256, 0, st>>>(n, visited, fr0, fr1);
    bfs_seed_kernel<<<(seeds + 255) / 256, 256, 0, st>>>(seeds, d_list + nblock, d_piv, visited, fr0, d_dist, wl0,
                                                         cnt);
    ck(cudaMemsetAsync(&ctx->s.status->barrier, 0, sizeof(unsigned int), st), "memset");
    ctx->launches += 2;
    int occ = 0;
    ck(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, msbfs_kernel, 512, 0), "occupancy");
    if (!rc && occ < 1) rc = bl_fail(ctx, BL_ERR_TOO_LARGE, "BFS kernel cannot be resident");
    BfsArgs b{n, d_rowptr, d_colids, visited, {fr0, fr1}, {wl0, wl1}, cnt, d_dist, ctx->s.status, n + 1};
    void *args[] = {&b};
    bl_time_begin(ctx, "msbfs_kernel");
    if (!rc)
      ck(cudaLaunchCooperativeKernel((const void *)msbfs_kernel, dim3(ctx->num_sms * std::min(occ, 2)), dim3(512),
                                     args, 0, st),
         "BFS launch");
    bl_time_end(ctx, "msbfs_kernel");
    ctx->launches++;
  }
  if (!rc) ck(cudaStreamSynchronize(st), "BFS");
  if (!rc) rc = bl_check_status(ctx);
  std::vector<double> gram((size_t)slice * kGram), V12((size_t)slice * kProj);
  for (int g0 = 0; g0 < num_graphs && !rc; g0 += slice) {
    const int gs = std::min(slice, num_graphs - g0);
    const int *vo = d_voff + g0;
    int widest = 1;
    for (int g = g0; g < g0 + gs; g++) widest = std::max(widest, mds_blocks(voff[g + 1] - voff[g]));
    ck(cudaMemsetAsync(d_maxd, 0, sizeof(int) * kP * gs, st), "memset");
    mds_max_kernel<<<dim3(widest, gs), 256, 0, st>>>(vo, d_dist, d_maxd);
    mds_colsum_kernel<<<dim3(widest, gs), 256, 0, st>>>(vo, d_dist, d_maxd, d_part);
    mds_mean_kernel<<<gs, 32, 0, st>>>(vo, d_part, d_mean);
    mds_gram_kernel<<<dim3(widest, gs), 256, 0, st>>>(vo, d_dist, d_maxd, d_mean, d_part);
    mds_gram_sum_kernel<<<gs, 256, 0, st>>>(vo, d_part, d_gram);
    ctx->launches += 5;
    ck(cudaMemcpyAsync(gram.data(), d_gram, sizeof(double) * kGram * gs, cudaMemcpyDeviceToHost, st), "D2H");
    ck(cudaStreamSynchronize(st), "sync");
    for (int g = 0; g < gs && !rc; g++) {
      std::vector<double> S(kP * kP, 0.0), lam, V;
      const double *t = gram.data() + (size_t)g * kGram;
      for (int i = 0; i < kP; i++)
        for (int j = i; j < kP; j++) S[i * kP + j] = S[j * kP + i] = *t++;
      jacobi_eigen(kP, S, lam, V);
      for (int s = 0; s < kP; s++)
        for (int j = 0; j < 12; j++) V12[(size_t)g * kProj + s * 12 + j] = V[s * kP + j];
      V12[(size_t)g * kProj + kP * 12] = lam[0] > 0 ? 1.0 / std::sqrt(lam[0] / (voff[g0 + g + 1] - voff[g0 + g])) : 0.0;
    }
    ck(cudaMemcpyAsync(d_V, V12.data(), sizeof(double) * kProj * gs, cudaMemcpyHostToDevice, st), "H2D");
    int most = 1;
    for (int g = g0; g < g0 + gs; g++) most = std::max(most, (voff[g + 1] - voff[g] + 255) / 256);
    ProjectArgs pa{vo, d_rowptr, d_colids, d_dist, d_maxd, d_mean, d_V, d_features};
    mds_project_kernel<<<dim3(most, gs), 256, 0, st>>>(pa);
    ctx->launches++;
    ck(cudaGetLastError(), "MDS kernels");
    if (g0 + gs < num_graphs) ck(cudaStreamSynchronize(st), "MDS");  // V12 is filled again
  }
  if (!rc) ck(cudaStreamSynchronize(st), "features");
  cleanup();
  return rc;
}

}  // namespace bl

extern "C" {

int bl_learned_features(bl_ctx *ctx, int n, const int *rowptr, const int *colids, int seed, const int *pivots,
                        float *features, unsigned short *dist, int *pivots_out) try {
  using namespace bl;
  if (!ctx || n < 1 || !rowptr || !features) return BL_ERR_ARG;
  BL_CUDA(ctx, cudaSetDevice(ctx->device));
  const long long nnz = rowptr[n];
  for (int v = 0; v < n; v++)
    if (rowptr[v + 1] < rowptr[v]) return bl_fail(ctx, BL_ERR_ARG, "rowptr decreases");
  int max_row = 0;
  for (int v = 0; v < n; v++) max_row = std::max(max_row, rowptr[v + 1] - rowptr[v]);
  for (long long e = 0; e < nnz; e++)
    if (colids[e] < 0 || colids[e] >= n) return bl_fail(ctx, BL_ERR_ARG, "colid out of range");
  int piv[kPivots];
  if (pivots) {
    for (int s = 0; s < kPivots; s++) {
      if (pivots[s] < 0 || pivots[s] >= n) return bl_fail(ctx, BL_ERR_ARG, "pivot out of range");
      piv[s] = pivots[s];
    }
  } else {
    choose_pivots(n, (uint64_t)seed, piv);
  }
  if (pivots_out) std::memcpy(pivots_out, piv, sizeof(piv));
  if (!ctx->s.status) {
    BL_CUDA(ctx, cudaMalloc(&ctx->s.status, sizeof(DevStatus)));
    BL_CUDA(ctx, cudaMemset(ctx->s.status, 0, sizeof(DevStatus)));
  }
  int *d_rp = nullptr, *d_ci = nullptr;
  float *d_f = nullptr;
  unsigned short *d_d = nullptr;
  int rc = 0;
  auto ck = [&](cudaError_t e, const char *w) {
    if (e != cudaSuccess && !rc) rc = bl_cuda_fail(ctx, e, w);
  };
  ck(cudaMalloc(&d_rp, sizeof(int) * (n + 1)), "cudaMalloc");
  ck(cudaMalloc(&d_ci, sizeof(int) * std::max<long long>(nnz, 1)), "cudaMalloc");
  ck(cudaMalloc(&d_f, sizeof(float) * kFeat * (size_t)n), "cudaMalloc");
  ck(cudaMalloc(&d_d, sizeof(unsigned short) * kPivots * (size_t)n), "cudaMalloc");
  if (!rc) {
    ck(cudaMemcpy(d_rp, rowptr, sizeof(int) * (n + 1), cudaMemcpyHostToDevice), "H2D");
    if (nnz) ck(cudaMemcpy(d_ci, colids, sizeof(int) * nnz, cudaMemcpyHostToDevice), "H2D");
  }
  const int voff[2] = {0, n};
  if (!rc) rc = compute_features(ctx, 1, voff, n, &max_row, d_rp, d_ci, piv, d_f, d_d);
  if (!rc) ck(cudaMemcpy(features, d_f, sizeof(float) * kFeat * (size_t)n, cudaMemcpyDeviceToHost), "D2H");
  if (!rc && dist) ck(cudaMemcpy(dist, d_d, sizeof(unsigned short) * kPivots * (size_t)n, cudaMemcpyDeviceToHost), "D2H");
  cudaFree(d_rp);
  cudaFree(d_ci);
  cudaFree(d_f);
  cudaFree(d_d);
  return rc;
} catch (...) {
  return bl_host_exception(ctx);
}

}  // extern "C"
