// barnes_hut.cu -- Barnes-Hut minibatch layout (algo 4) on the device.
//
// Reference: sample/algorithms.cpp:1038-1072 (iteration), sample/MortonCode.h
// (frame, quantisation, order), sample/BarnesHut.h:114-225 (sort, quadtree
// build, opening test, unit-vector repulsion).
//
// Per iteration:
//   1. bbox of the positions; Morton frame {minX, minY, MAXMIN} and 64-bit keys
//      (y-major interleave of the two 32-bit quantised coordinates, quantised
//      in FP64 exactly as the reference: (uint32)(4294967295.0*(x-minX)/MAXMIN)).
//   2. stable LSD radix sort of the keys on the high 32 bits (4 passes of 8
//      bits), then each run of equal high halves sorted on its own (they are
//      rare); 1 and 2 are one cooperative launch.
//   3. binary radix tree over the sorted keys (Karras 2012), then a bottom-up
//      pass that merges the x-bit level into the y-bit level of the same
//      digit, giving exactly the reference quadtree without its single-child
//      chain nodes; centroids are the unweighted means of the children summed
//      in quadrant order, in FP64, bit-identical to the reference, computed
//      bottom-up by the last-arriving child of every node (no barriers).
//   4. pre-order layout with skip links: 16-byte records {x, y, D^2, skip}
//      walked without a stack.
//   5. repulsion of every vertex in Morton order (coherent warps).  A vertex
//      is only moved by its own batch, so its query position and the tree
//      snapshot are both the iteration-start positions: all n traversals are
//      independent.  The opening test D/dist < theta is evaluated in FP32 and
//      re-evaluated in FP64 when the FP32 margin is within its error bound,
//      so every decision equals the reference's FP64 decision.
//   6. attraction + update.  Vertex i reads the new position of a neighbour j
//      from an earlier batch and the iteration-start position otherwise, so
//      the batch order only constrains i after its earlier-batch neighbours:
//      vertices are grouped into dependency levels (computed once per graph
//      and batch size) and each level is one parallel launch.  This produces
//      the same values as the reference's sequential batch loop.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>

#include "bh_device.cuh"

namespace bl {
namespace {

constexpr int kQuadLevels = 33;  // quad levels 0..31, 32 for runs of identical keys


// ---- box, keys and order: one cooperative launch --------------------------------
//
// Bounding box of the positions (MortonCode.h:42-58), the FP64 frame
// {minX, minY, MAXMIN, 1/MAXMIN}, the high half of every point's 64-bit Morton
// key, and a stable LSD radix sort of (high half, vertex) words on it (four
// 8-bit digits).  The points are cut into tiles of r * 512 (r such that one
// tile per resident block covers them where r <= 16 does); a block takes tiles
// b, b + grid, ...  Per digit pass:
//   - a tile's keys are ranked stably: warp w owns r * 32 consecutive keys and
//     counts with warp-private counters, so no block barrier sits in the
//     ranking; the keys are placed in shared memory grouped by digit (with
//     more than one tile a block, then written back where they were read);
//     the tile's digit counts go to hist[tile][256] and are added to the
//     totals of the tile's group (16 groups);
//   - grid barrier;
//   - a tile's offset of a digit = the digit's global offset + the groups
//     before + the tiles before in its group: 16 + tiles / 16 loads a thread,
//     all independent, in place of a scan over all tiles;
//   - the grouped keys are written out, each digit's run of the tile as whole
//     sectors;
//   - grid barrier.
// Bound by the nine barriers and the L2 round trips between them at small
// sizes (2 us of the 3 us a half pass takes at 100,000 points) and by the
// ranking's shared-memory traffic at large ones (9,000 of a pass's 25,000
// cycles at a million).  As sixteen launches (frame and keys, three a digit
// pass, two for the runs, a gather) the stage up to the sorted positions took
// 104 us at 4,000 points, 103 at 100,000, 160 at 1,000,000 and 346 at
// 3,000,000; it takes 43, 51, 90 and 206.  One cluster of 16 blocks that keeps
// everything in shared memory took 26 us at 4,000 but 97 at 100,000.
constexpr int kSortThreads = 512;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSortItems = 16;
constexpr int kSortTile = kSortThreads * kSortItems;
constexpr int kSortGroups = 16;

__device__ __forceinline__ unsigned int hi32(u64 k) { return (unsigned int)(k >> 32); }

struct SortSmem {
  u64 key[kSortTile];                     // a tile's words grouped by digit
  unsigned short rank[kSortTile];         // of a key among its warp's and its digit's
  unsigned int wcnt[kSortWarps][256];     // per-warp digit counts, then offsets within the digit
  // first key of each digit: position in the tile; global position less that
  unsigned int base[256], loc[256];
  unsigned int ws[kSortWarps];
  unsigned int box[kSortWarps][4];
  KeyFrame frame;
  unsigned int ok;
};

struct SortArgs {
  const float2 *pos;
  int n, items, ntiles, group;  // keys per thread, tiles, tiles per group
  // all bits set before the launch: {min x, ~max x, min y, ~max y} as ordered
  // integers, barrier arrivals
  unsigned int *ctl;
  double *frame;
  KeyFrame *kframe;
  double inv_theta2;
  float *ztab;
  u64 *pairs0, *pairs1;  // (high half << 32) | vertex; a pass reads one and writes the other
  unsigned int *hist;    // [tiles][256]
  unsigned int *gtot;    // [4 passes][kSortGroups][256]
  int *runs;             // count of the long runs (cleared)
  int *zero0, *zero1;    // cleared for the tree kernels
  int nzero0, nzero1;
  DevStatus *st;
};

// Grid barrier `k` (1, 2, ...) of a launch; false when the kernel has to end.
__device__ __forceinline__ bool sort_barrier(const SortArgs &a, SortSmem &S, unsigned int k) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicSub(&a.ctl[4], 1u);
    const unsigned int target = 0xffffffffu - k * gridDim.x;
    const unsigned long long t0 = dev_globaltimer();
    unsigned int ok = 1, polls = 0;
    while (ld_acquire_gpu(&a.ctl[4]) > target) {
      if ((++polls & 127u) == 0u) {
        if (ld_volatile_u32(&a.st->code) != 0u) {
          ok = 0;
          break;
        }
        if (dev_globaltimer() - t0 > kBarrierTimeoutNs) {
          dev_record_error(a.st, DEV_TIMEOUT_GRID_BARRIER);
          ok = 0;
          break;
        }
      }
    }
    S.ok = ok;
  }
  __syncthreads();
  return S.ok != 0u;
}

// Lanes of the warp with the same digit (256: none).  Eight ballots: with
// a __match_any_sync the ranking of a million keys took 16,600 cycles a pass,
// so it takes 12,000 with the placing.
__device__ __forceinline__ unsigned int digit_peers(unsigned int d) {
  unsigned int peers = __ballot_sync(0xffffffffu, d < 256u);
#pragma unroll
  for (int b = 0; b < 8; b++) {
    const bool one = (d >> b) & 1u;
    const unsigned int m = __ballot_sync(0xffffffffu, one);
    peers &= one ? m : ~m;
  }
  return peers;
}

// Exclusive scan over the first 256 threads; every thread of the block calls it.
__device__ __forceinline__ unsigned int sort_scan256(unsigned int v, SortSmem &S) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned int x = v;
  if (tid < 256) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) S.ws[warp] = x;
  }
  __syncthreads();
  unsigned int pre = 0;
  if (tid < 256)
    for (int w = 0; w < warp; w++) pre += S.ws[w];
  __syncthreads();
  return pre + x - v;
}

// A tile of the pass's input grouped by digit in S.key (stable), the first
// position of each digit in S.loc; returns the digit counts to threads
// 0..255.
__device__ __forceinline__ unsigned int sort_rank_tile(const SortArgs &a, SortSmem &S, const u64 *in, int shift,
                                                       int tile) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const unsigned int lt = (1u << lane) - 1u;
#pragma unroll
  for (int k = 0; k < 256 / 32; k++) S.wcnt[warp][k * 32 + lane] = 0u;
  __syncwarp();
  const int first = warp * a.items * 32, i0 = tile * a.items * kSortThreads + first;
  for (int r0 = 0; r0 < a.items; r0 += 4) {
    unsigned int dg[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {  // four loads in flight
      const int i = i0 + (r0 + q) * 32 + lane;
      dg[q] = r0 + q < a.items && i < a.n ? ((unsigned int)(__ldcg(&in[i]) >> shift) & 255u) : 256u;
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
      if (r0 + q >= a.items) break;
      const unsigned int d = dg[q];
      const unsigned int peers = digit_peers(d);
      unsigned int old = 0;
      if (d < 256u) old = S.wcnt[warp][d];
      __syncwarp();
      if (d < 256u && (peers & lt) == 0u) S.wcnt[warp][d] = old + __popc(peers);
      __syncwarp();
      S.rank[first + (r0 + q) * 32 + lane] = (unsigned short)(old + __popc(peers & lt));
    }
  }
  __syncthreads();
  unsigned int run = 0;
  if (tid < 256) {
#pragma unroll
    for (int w = 0; w < kSortWarps; w++) {
      const unsigned int c = S.wcnt[w][tid];
      S.wcnt[w][tid] = run;
      run += c;
    }
  }
  const unsigned int loff = sort_scan256(run, S);
  if (tid < 256) S.loc[tid] = loff;
  __syncthreads();
  for (int r0 = 0; r0 < a.items; r0 += 4) {
    u64 k[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int i = i0 + (r0 + q) * 32 + lane;
      if (r0 + q < a.items && i < a.n) k[q] = __ldcg(&in[i]);
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int i = i0 + (r0 + q) * 32 + lane;
      if (r0 + q < a.items && i < a.n) {
        const unsigned int d = (unsigned int)(k[q] >> shift) & 255u;
        S.key[S.loc[d] + S.wcnt[warp][d] + S.rank[first + (r0 + q) * 32 + lane]] = k[q];
      }
    }
  }
  return run;
}

__global__ void __launch_bounds__(kSortThreads, 2) morton_sort_kernel(SortArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SortSmem &S = *reinterpret_cast<SortSmem *>(smem_raw);
  if (!block_status_ok(a.st)) return;  // every block sees the same value: no barrier is left waiting
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tsize = a.items * kSortThreads;
  const bool single = a.ntiles <= (int)gridDim.x;  // one tile a block: its ranks stay
  unsigned int nbar = 0;
  // box
  unsigned int bb[4] = {0xffffffffu, 0xffffffffu, 0xffffffffu, 0xffffffffu};
  for (int tile = blockIdx.x; tile < a.ntiles; tile += gridDim.x)
#pragma unroll 4
    for (int r = 0; r < a.items; r++) {
      const int i = tile * tsize + r * kSortThreads + tid;
      if (i < a.n) {
        const float2 p = a.pos[i];
        const unsigned int ux = f2ord(p.x), uy = f2ord(p.y);
        bb[0] = min(bb[0], ux);
        bb[1] = min(bb[1], ~ux);
        bb[2] = min(bb[2], uy);
        bb[3] = min(bb[3], ~uy);
      }
    }
#pragma unroll
  for (int c = 0; c < 4; c++) {
    bb[c] = __reduce_min_sync(0xffffffffu, bb[c]);
    if (lane == 0) S.box[warp][c] = bb[c];
  }
  // what this launch and the tree kernels count from zero
  const int gid = blockIdx.x * kSortThreads + tid, gsz = gridDim.x * kSortThreads;
  for (int k = gid; k < 4 * kSortGroups * 256; k += gsz) a.gtot[k] = 0u;
  for (int k = gid; k < a.nzero0; k += gsz) a.zero0[k] = 0;
  for (int k = gid; k < a.nzero1; k += gsz) a.zero1[k] = 0;
  if (gid == 0) a.runs[0] = 0;
  __syncthreads();
  if (tid < 4) {
    unsigned int v = 0xffffffffu;
#pragma unroll
    for (int w = 0; w < kSortWarps; w++) v = min(v, S.box[w][tid]);
    atomicMin(&a.ctl[tid], v);
  }
  if (!sort_barrier(a, S, ++nbar)) return;
  if (tid == 0) {
    unsigned int box[4];
    box[0] = ld_volatile_u32(&a.ctl[0]);
    box[1] = ~ld_volatile_u32(&a.ctl[1]);
    box[2] = ld_volatile_u32(&a.ctl[2]);
    box[3] = ~ld_volatile_u32(&a.ctl[3]);
    double minX, minY, maxmin;
    frame_from_bbox(box, minX, minY, maxmin);
    S.frame = key_frame(minX, minY, maxmin);
    if (blockIdx.x == 0) {
      a.frame[0] = minX;
      a.frame[1] = minY;
      a.frame[2] = maxmin;
      a.frame[3] = S.frame.inv;
      *a.kframe = S.frame;
    }
  }
  __syncthreads();
  const KeyFrame &frame = S.frame;
  // keys; the records' z by quad level: D^2 / theta^2 with D = MAXMIN / 2^level
  if (blockIdx.x == 0 && tid < kQuadLevels) a.ztab[tid] = bh_record_z(ldexp(frame.maxmin, -tid), a.inv_theta2);
  for (int tile = blockIdx.x; tile < a.ntiles; tile += gridDim.x)
#pragma unroll 2
    for (int r = 0; r < a.items; r++) {
      const int i = tile * tsize + r * kSortThreads + tid;
      if (i < a.n)
        __stcg(&a.pairs1[i], ((u64)morton_halves(a.pos[i], frame).y << 32) | (unsigned int)i);
    }
  __syncthreads();  // a block ranks its own tiles' keys
  for (int pass = 0; pass < 4; pass++) {
    const int shift = 32 + 8 * pass;
    unsigned int *gt = a.gtot + pass * kSortGroups * 256;
    u64 *in = (pass & 1) ? a.pairs0 : a.pairs1, *out = (pass & 1) ? a.pairs1 : a.pairs0;
    for (int tile = blockIdx.x; tile < a.ntiles; tile += gridDim.x) {
      const unsigned int mine = sort_rank_tile(a, S, in, shift, tile);
      if (tid < 256) {
        __stcg(&a.hist[(size_t)tile * 256 + tid], mine);
        if (mine) atomicAdd(&gt[(tile / a.group) * 256 + tid], mine);
      }
      if (!single) {  // back to where the tile's keys were read
        __syncthreads();
        const int cnt = min(tsize, a.n - tile * tsize);
        for (int x = tid; x < cnt; x += kSortThreads) __stcg(&in[tile * tsize + x], S.key[x]);
        __syncthreads();
      }
    }
    if (!sort_barrier(a, S, ++nbar)) return;
    for (int tile = blockIdx.x; tile < a.ntiles; tile += gridDim.x) {
      unsigned int all = 0, before = 0;
      if (tid < 256) {
        const int g = tile / a.group;
#pragma unroll
        for (int q = 0; q < kSortGroups; q++) {
          const unsigned int c = __ldcg(&gt[q * 256 + tid]);
          all += c;
          if (q < g) before += c;
        }
#pragma unroll 8
        for (int t = g * a.group; t < tile; t++) before += __ldcg(&a.hist[(size_t)t * 256 + tid]);
      }
      if (!single) {
        const unsigned int mine = tid < 256 ? __ldcg(&a.hist[(size_t)tile * 256 + tid]) : 0u;
        const unsigned int loff = sort_scan256(mine, S);
        if (tid < 256) S.loc[tid] = loff;
      }
      const unsigned int goff = sort_scan256(all, S);
      if (tid < 256) S.base[tid] = goff + before - S.loc[tid];
      __syncthreads();
      const int cnt = min(tsize, a.n - tile * tsize);
#pragma unroll 4
      for (int x = tid; x < cnt; x += kSortThreads) {
        const u64 k = single ? S.key[x] : __ldcg(&in[tile * tsize + x]);
        const unsigned int g = S.base[(unsigned int)(k >> shift) & 255u] + (unsigned int)x;
        if (g < (unsigned int)a.n) __stcg(&out[g], k);
      }
      if (!single) __syncthreads();
    }
    if (pass < 3 && !sort_barrier(a, S, ++nbar)) return;
  }
}

// ---- sorted keys, vertices and positions; the low 32 bits -----------------------
//
// The four LSD passes on bits 32..63 leave the keys ordered by their high
// halves and, within a run of equal high halves, by vertex id (the passes are
// stable and the keys started in vertex order).  A run means two points in
// the same cell of a 65,536 x 65,536 grid over the frame: rare (a uniform
// million points give ~100 runs of two).  So each run is finished on its own,
// by (key, vertex id): runs of up to 32 keys by one thread (insertion sort),
// longer ones by one block each (bitonic network in shared memory up to
// kRunCap keys, beyond that stable 8-bit LSD passes through global memory).
// The result is the stable order of the full 64-bit keys.
constexpr int kRunThreads = 512;
constexpr int kRunShort = 32;
constexpr int kRunCap = 2048;

struct RunSmem {
  union {
    struct {
      u64 k[kRunCap];
      int v[kRunCap];
    } b;
    struct {
      unsigned int cnt[kRunThreads / 32][256];
      unsigned int base[256];
      unsigned int carry[256];
      unsigned int tot[256];
    } c;
  } u;
  unsigned int ws[kRunThreads / 32];
};

// Exclusive scan of x over the first 256 threads; all threads call.
__device__ __forceinline__ unsigned int run_scan256(unsigned int x, RunSmem &S) {
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  unsigned int inc = x;
  if (tid < 256) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned int y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += y;
    }
    if (lane == 31) S.ws[w] = inc;
  }
  __syncthreads();
  unsigned int pre = 0;
  if (tid < 256)
    for (int q = 0; q < w; q++) pre += S.ws[q];
  __syncthreads();
  return pre + inc - x;
}

// The run [start, start + len) sorted by one block.
__device__ __noinline__ void sort_run(u64 *keys, int *vals, u64 *kalt, int *valt, int start, int len, RunSmem &S) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (len <= kRunCap) {
    int m = 2;
    while (m < len) m <<= 1;
    for (int q = tid; q < m; q += kRunThreads) {
      S.u.b.k[q] = q < len ? keys[start + q] : ~0ull;
      S.u.b.v[q] = q < len ? vals[start + q] : INT_MAX;
    }
    __syncthreads();
    for (int size = 2; size <= m; size <<= 1) {
      for (int stride = size >> 1; stride > 0; stride >>= 1) {
        for (int i = tid; i < (m >> 1); i += kRunThreads) {
          const int lo = ((i & ~(stride - 1)) << 1) | (i & (stride - 1));
          const int hi = lo + stride;
          const bool up = (lo & size) == 0;
          const u64 ka = S.u.b.k[lo], kb = S.u.b.k[hi];
          const int va = S.u.b.v[lo], vb = S.u.b.v[hi];
          if ((ka > kb || (ka == kb && va > vb)) == up) {
            S.u.b.k[lo] = kb;
            S.u.b.k[hi] = ka;
            S.u.b.v[lo] = vb;
            S.u.b.v[hi] = va;
          }
        }
        __syncthreads();
      }
    }
    for (int q = tid; q < len; q += kRunThreads) {
      keys[start + q] = S.u.b.k[q];
      vals[start + q] = S.u.b.v[q];
    }
    __syncthreads();
    return;
  }
  // a long run: four stable 8-bit passes on the low 32 bits through
  // global memory (keys <-> the same range of kalt), chunk by chunk
  const unsigned int lt = (1u << lane) - 1u;
  for (int pass = 0; pass < 4; pass++) {
    const u64 *ks = (pass & 1) ? kalt + start : keys + start;
    const int *vs = (pass & 1) ? valt + start : vals + start;
    u64 *kd = (pass & 1) ? keys + start : kalt + start;
    int *vd = (pass & 1) ? vals + start : valt + start;
    const int shift = 8 * pass;
    if (tid < 256) S.u.c.carry[tid] = 0;
    __syncthreads();
    for (int q = tid; q < len; q += kRunThreads) atomicAdd(&S.u.c.carry[(unsigned int)(ks[q] >> shift) & 255u], 1u);
    __syncthreads();
    const unsigned int pre = run_scan256(tid < 256 ? S.u.c.carry[tid] : 0u, S);
    if (tid < 256) {
      S.u.c.base[tid] = pre;
      S.u.c.carry[tid] = 0;
    }
    __syncthreads();
    for (int c0 = 0; c0 < len; c0 += kRunThreads) {  // one key per thread and chunk
      for (int q = tid; q < (kRunThreads / 32) * 256; q += kRunThreads) (&S.u.c.cnt[0][0])[q] = 0;
      __syncthreads();
      const int q = c0 + tid;
      const bool valid = q < len;
      const u64 key = valid ? ks[q] : 0ull;
      const int val = valid ? vs[q] : 0;
      const unsigned int d = valid ? ((unsigned int)(key >> shift) & 255u) : 256u;
      const unsigned int peers = __match_any_sync(0xffffffffu, d);
      const unsigned int rank = __popc(peers & lt);
      if (d < 256u && lane == __ffs(peers) - 1) S.u.c.cnt[warp][d] = __popc(peers);
      __syncthreads();
      if (tid < 256) {
        unsigned int run = 0;
        for (int w = 0; w < kRunThreads / 32; w++) {
          const unsigned int c = S.u.c.cnt[w][tid];
          S.u.c.cnt[w][tid] = run;
          run += c;
        }
        S.u.c.tot[tid] = run;
      }
      __syncthreads();
      if (d < 256u) {
        const unsigned int p = S.u.c.base[d] + S.u.c.carry[d] + S.u.c.cnt[warp][d] + rank;
        kd[p] = key;
        vd[p] = val;
      }
      __syncthreads();
      if (tid < 256) S.u.c.carry[tid] += S.u.c.tot[tid];
      __syncthreads();
    }
  }
  // four passes end where they started (keys/vals)
}

// One thread per sorted position: full key, vertex and position, from the
// position that is fetched by vertex anyway (the sort carries high halves
// only).  A thread of a kernel of its own, not of the sort: the random 8-byte
// fetches need many of them in flight, and beside the sort's 200 KB of shared
// memory the first-level cache leaves few: there a million points took 27 us,
// here 9.
__global__ void __launch_bounds__(256) morton_emit_kernel(const float2 *__restrict__ pos, int n,
                                                          const u64 *__restrict__ pairs, const KeyFrame *__restrict__ frame,
                                                          u64 *__restrict__ keys, int *__restrict__ vals,
                                                          float2 *__restrict__ spos, int *runs, int runs_cap,
                                                          DevStatus *st) {
  if (!block_status_ok(st)) return;
  const int k = blockIdx.x * 256 + threadIdx.x;
  if (k >= n) return;
  const KeyFrame &F = *frame;
  const u64 w = pairs[k];
  const unsigned int h = hi32(w);
  const unsigned int before = k > 0 ? hi32(pairs[k - 1]) : ~h, after = k + 1 < n ? hi32(pairs[k + 1]) : ~h;
  const float2 p = pos[(unsigned int)w];
  int len = 1;
  if (before == h || after == h) {  // in a run
    int first = k;
    while (first > 0 && k - first < kRunShort && hi32(pairs[first - 1]) == h) first--;
    len = k + 1 - first;
    while (first + len < n && len <= kRunShort && hi32(pairs[first + len]) == h) len++;
    if (len <= kRunShort) {
      if (first != k) return;  // the run's first thread writes all of it
    } else if (before != h) {
      while (k + len < n && hi32(pairs[k + len]) == h) len++;  // the whole run
      const int slot = atomicAdd(&runs[0], 1);
      if (slot < runs_cap) {
        runs[1 + 2 * slot] = k;
        runs[2 + 2 * slot] = len;
      } else {
        dev_record_error(st, DEV_BAD_INDEX);  // cannot happen (see runs_cap)
      }
      len = 1;
    } else {
      len = 1;
    }
  }
  keys[k] = ((u64)h << 32) | morton_halves(p, F).x;
  vals[k] = (int)(unsigned int)w;
  spos[k] = p;
  // a short run: insertion by (key, vertex id); the rest arrive in vertex order
  for (int x = k + 1; x < k + len; x++) {
    const unsigned int vx = (unsigned int)pairs[x];
    const float2 px = pos[vx];
    const u64 kx = ((u64)h << 32) | morton_halves(px, F).x;
    int b = x - 1;
    for (; b >= k && keys[b] > kx; b--) {
      keys[b + 1] = keys[b];
      vals[b + 1] = vals[b];
      spos[b + 1] = spos[b];
    }
    keys[b + 1] = kx;
    vals[b + 1] = (int)vx;
    spos[b + 1] = px;
  }
}

// The queued long runs, one block each, and their positions.
__global__ void __launch_bounds__(kRunThreads) run_sort_kernel(u64 *keys, int *vals, u64 *kalt, int *valt,
                                                               const int *runs, int runs_cap,
                                                               const float2 *__restrict__ pos, float2 *spos,
                                                               DevStatus *st) {
  __shared__ RunSmem S;
  const int nruns = min(runs[0], runs_cap);
  if ((int)blockIdx.x >= nruns || !block_status_ok(st)) return;
  for (int q = blockIdx.x; q < nruns; q += gridDim.x) {
    const int start = runs[1 + 2 * q], len = runs[2 + 2 * q];
    __syncthreads();
    sort_run(keys, vals, kalt, valt, start, len, S);
    __syncthreads();
    for (int k = threadIdx.x; k < len; k += kRunThreads) spos[start + k] = pos[vals[start + k]];
  }
}

// ---- binary radix tree (Karras 2012) ----------------------------------------
__device__ __forceinline__ int kdelta(const u64 *__restrict__ K, int n, int i, int j) {
  if (j < 0 || j >= n) return -1;
  const u64 x = K[i] ^ K[j];
  return x ? __clzll((long long)x) : 64 + __clz(i ^ j);
}

// internal node i in [0, n-2]; leaf k encoded as ~k in child links; the root
// is internal node 0.  A node is 32 bytes of bnode, ints {first, last, prefix
// length, left; right, parent, -, -}: its own words are two stores of one
// sector, the parent word is written by the parent's thread.  range and dlt
// repeat the first words for the kernels that want only those; leaf_parent[k]
// is the parent of leaf k.  Bound by issue (the searches): 1,000,000 points 30
// us, 3,000,000 72; with the words stored one by one and a child and a parent
// array beside them 33 and 76.
__global__ void radix_tree_kernel(const u64 *__restrict__ K, int n, int2 *range, int *dlt, int *leaf_parent,
                                  int *bnode) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n - 1) return;
  const u64 ki = K[i];
  const int dnext = kdelta(K, n, i, i + 1), dprev = kdelta(K, n, i, i - 1);
  const int d = dnext - dprev >= 0 ? 1 : -1;
  const int dmin = min(dnext, dprev);
  // The searches ask whether a prefix with key i is longer than m bits: for
  // m < 64 whether the keys' difference is below 2^(63 - m), one comparison
  // where the prefix itself takes a count, a select and the tie's rule (with
  // which 1,000,000 points took 8 us more, 3,000,000 25).
  auto longer = [&](int q, int m, u64 lim) {
    return m < 64 ? (unsigned int)q < (unsigned int)n && (ki ^ K[q]) <= lim : kdelta(K, n, i, q) > m;
  };
  auto limit = [](int m) { return m < 0 ? ~0ull : (1ull << (63 - min(m, 63))) - 1ull; };
  const u64 lmin = limit(dmin);
  int lmax = 2;
  while (longer(i + lmax * d, dmin, lmin)) lmax <<= 1;
  int l = 0;
  for (int t = lmax >> 1; t >= 1; t >>= 1)
    if (longer(i + (l + t) * d, dmin, lmin)) l += t;
  const int j = i + l * d;
  const int dnode = kdelta(K, n, i, j);
  const u64 lnode = limit(dnode);
  int s = 0;
  for (int t = l; t > 1;) {
    t = (t + 1) >> 1;  // l / 2, l / 4, ... rounded up
    if (longer(i + (s + t) * d, dnode, lnode)) s += t;
  }
  const int gamma = i + s * d + min(d, 0);
  const int first = min(i, j), last = max(i, j);
  const int left = (first == gamma) ? ~gamma : gamma;
  const int right = (last == gamma + 1) ? ~(gamma + 1) : gamma + 1;
  range[i] = make_int2(first, last);
  dlt[i] = dnode;
  int *b = bnode + 8 * (size_t)i;
  *reinterpret_cast<int4 *>(b) = make_int4(first, last, dnode, left);
  b[4] = right;
  if (i == 0) b[5] = -1;
  if (left >= 0) bnode[8 * (size_t)left + 5] = i;
  else leaf_parent[~left] = i;
  if (right >= 0) bnode[8 * (size_t)right + 5] = i;
  else leaf_parent[~right] = i;
}

struct TreeArgs {
  int n;
  const float2 *spos;
  const int2 *range;
  const int *dlt;
  const int *leaf_parent;
  int4 *qkids;          // quad children of a quad node, kNoChild-padded
  double2 *qcen;
  int *qbelow;
  int *startcnt;
  int *qpar;     // quad parent of internal node i (index i) and of leaf k (index n-1+k); -1 for the root
  int *qnchild;  // children of a quad node
  // quad nodes whose range spans centroid blocks, by level (0..32):
  // span_cnt[level] (zero before the pass), span_list[level * span_cap + slot]
  int *span_cnt;
  int *span_list;
  int span_cap;
  int *span_pos;  // position of a listed node (span_stage_kernel)
  double2 *stage_val;  // staged listed nodes (span_stage_kernel -> centroid_top_kernel)
  int4 *stage_pend;
  int4 *stage_meta;
  // pre-order records: quad nodes starting before each centroid block
  // (chain_kernel adds them up, block_base_kernel turns them into offsets),
  // startbase[k] = quad nodes starting before sorted position k
  int *blocktot;
  int *startbase;
  // quad nodes that span exactly one block boundary, by boundary b (between
  // blocks b and b+1): their levels (bit mask) and ids (chain_node[b * 33 +
  // level])
  unsigned long long *chain_mask;
  int *chain_node;
  const float *ztab;  // the records' z = D^2 / theta^2 by quad level (morton_sort_kernel)
  float4 *nodes;
  double2 *nodes_c64;
  unsigned char *nodes_lvl;
  const int4 *bnode;  // packed internal nodes, two int4 each (radix_tree_kernel)
  DevStatus *st;
};

constexpr int kNoChild = INT_MIN;
constexpr int kCenSpanC = 1024;  // sorted points per centroid block

__device__ __forceinline__ int quad_level(int p) { return p >= 64 ? 32 : (p >> 1); }


// Structure of the quadtree, one thread per sorted position k.  The binary
// nodes whose range starts at k form the left-child chain above leaf k; the
// chains of different k are disjoint, so each thread owns its nodes and no
// synchronisation is needed.  For every quad node on the chain it records the
// number of quad nodes below it on the chain (qbelow), its quad children, their
// count, and itself as their quad parent; startcnt[k] counts the quad nodes
// starting at k.
__device__ __forceinline__ int chain_walk(const TreeArgs &t, int k);

__global__ void __launch_bounds__(256) chain_kernel(TreeArgs t) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  const int cnt = k < t.n ? chain_walk(t, k) : 0;
  // quad nodes starting in this warp's 32 positions (one centroid block)
  const int sum = __reduce_add_sync(0xffffffffu, cnt);
  if ((threadIdx.x & 31) == 0 && sum) atomicAdd(&t.blocktot[(k & ~31) / kCenSpanC], sum);
}

__device__ __forceinline__ int chain_walk(const TreeArgs &t, int k) {
  int cnt = 0;
  int cur = t.leaf_parent[k];
  if (k == 0) t.qpar[0] = -1;  // the root
  const int4 none = make_int4(-1, -1, -1, -1);
  int4 ra = none;  // cur's packed record
  int2 rb = make_int2(-1, -1);
  auto second = [&](int node) { return __ldg(reinterpret_cast<const int2 *>(&t.bnode[2 * node + 1])); };
  if (cur >= 0) {
    ra = __ldg(&t.bnode[2 * cur]);
    rb = second(cur);
  }
  // bounded by the tree height: every step moves to a parent.  The parent's
  // record and the children's are loaded together, one round trip a step.
  while (cur >= 0 && ra.x == k) {
    const int par = rb.y;
    int4 pa = none;
    int2 pb = make_int2(-1, -1);
    if (par >= 0) {
      pa = __ldg(&t.bnode[2 * par]);
      pb = second(par);
    }
    const int p = ra.z;
    const int sides[2] = {ra.w, rb.x};
    int4 ca[2] = {none, none};
    int2 cb[2];
#pragma unroll
    for (int h = 0; h < 2; h++)
      if (p < 64 && sides[h] >= 0) {
        ca[h] = __ldg(&t.bnode[2 * sides[h]]);
        cb[h] = second(sides[h]);
      }
    // cur is merged into its parent's quad node: the x-bit split of the digit
    // whose y-bit split is the parent, or any split inside a run below its top
    const bool sub = cur > 0 && (p >= 64 ? pa.z >= 64 : ((p & 1) && pa.z == p - 1));
    if (!sub) {
      t.qbelow[cur] = cnt++;
      int kids[4] = {kNoChild, kNoChild, kNoChild, kNoChild};
      int m = 0;
      if (p < 64) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int c = sides[h];
          const int pc = ca[h].z;  // the child's prefix length; its parent is cur
          const bool csub = c > 0 && (pc >= 64 ? p >= 64 : ((pc & 1) && p == pc - 1));
          if (c >= 0 && csub) {
            kids[m++] = ca[h].w;
            kids[m++] = cb[h].x;
          } else {
            kids[m++] = c;
          }
        }
        for (int c = 0; c < m; c++) t.qpar[kids[c] >= 0 ? kids[c] : t.n - 1 + ~kids[c]] = cur;
      } else {
        // run of identical keys: every point of the range is a child
        for (int q = ra.x; q <= ra.y; q++) t.qpar[t.n - 1 + q] = cur;
        m = ra.y - ra.x + 1;
      }
      t.qkids[cur] = make_int4(kids[0], kids[1], kids[2], kids[3]);
      t.qnchild[cur] = m;
    } else {
      t.qnchild[cur] = 0;  // merged into its parent: not a quad node
    }
    cur = (cur == 0) ? -1 : par;
    ra = pa;
    rb = pb;
  }
  t.startcnt[k] = cnt;
  return cnt;
}

// Exclusive offsets of the centroid blocks' quad-node counts, in place
// (tot[nb] = the number of quad nodes), and startbase[n] = the same.  One
// block of 1024 threads.
__global__ void __launch_bounds__(1024) block_base_kernel(int *tot, int nb, int *startbase_n) {
  __shared__ int ws[32];
  __shared__ int carry;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  if (tid == 0) carry = 0;
  __syncthreads();
  for (int c0 = 0; c0 < nb; c0 += 1024) {
    const int b = c0 + tid;
    const int v = b < nb ? tot[b] : 0;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) ws[w] = x;
    __syncthreads();
    int wpre = 0, total = 0;
    for (int q = 0; q < 32; q++) {
      const int u = ws[q];
      if (q < w) wpre += u;
      total += u;
    }
    const int base = carry;
    if (b < nb) tot[b] = base + wpre + x - v;
    __syncthreads();
    if (tid == 0) carry = base + total;
    __syncthreads();
  }
  if (tid == 0) {
    tot[nb] = carry;
    *startbase_n = carry;
  }
}

// Pre-order record of quad node `node` (BarnesHut.h:114-225 as a flat walk):
// the record after the quad nodes starting before position lo = range.x and
// the deeper quad nodes starting at lo; its skip link is the first record
// after its range.  sc_lo = quad nodes starting at lo, sb_lo / sb_hi =
// startbase at lo and at hi = range.y + 1, qb = quad nodes below it starting
// at lo.  False (and DEV_BAD_INDEX) for offsets that cannot be.
__device__ __forceinline__ bool node_record_slot(const TreeArgs &t, int lo, int hi, int qb, int sc_lo, int sb_lo,
                                                 int sb_hi, int &idx, int &skip) {
  const int cap = 2 * t.n - 1;  // records: n leaves + at most n-1 quad nodes
  const int rank = sc_lo - 1 - qb;
  idx = lo + sb_lo + rank;
  skip = hi + sb_hi;
  if (rank < 0 || idx < 0 || idx >= cap || skip <= idx || skip > cap) {
    dev_record_error(t.st, DEV_BAD_INDEX);
    return false;
  }
  return true;
}

// {x, y, D^2 / theta^2, skip} with the FP64 centroid and the level beside it
// (the walk's FP64 re-test reads those two).
__device__ __forceinline__ void write_node_record(const TreeArgs &t, int idx, int skip, int lvl, double2 c) {
  t.nodes[idx] = make_float4(d2f_int(c.x), d2f_int(c.y), t.ztab[lvl], __int_as_float(skip));
  t.nodes_c64[idx] = c;
  t.nodes_lvl[idx] = (unsigned char)lvl;
}

// The same from global memory (startbase of the whole range written).
__device__ __forceinline__ void write_node_record_global(const TreeArgs &t, int node, double2 c) {
  const int2 rg = t.range[node];
  int idx, skip;
  if (node_record_slot(t, rg.x, rg.y + 1, t.qbelow[node], t.startcnt[rg.x], t.startbase[rg.x],
                       t.startbase[rg.y + 1], idx, skip))
    write_node_record(t, idx, skip, quad_level(t.dlt[node]), c);
}

// Centroids bottom-up.  The centroid of a quad node is the unweighted mean of
// its children summed in quadrant order in FP64 (BarnesHut.h:197-217),
// bit-identical to the reference; it can be computed once every child is
// done.  Three passes by how many block boundaries a node's range contains:
// * none — centroid_kernel: a block owns kCenSpan consecutive sorted points;
//   a binary node whose range lies inside them has its index there too (a
//   Karras node's index is one of its range ends), so the block loads those
//   nodes' structure and its points into shared memory with coalesced reads,
//   and processes the nodes in rounds: the nodes whose children are all done
//   form a queue, handled one node per thread so that the FP64 work (a small
//   fraction of the FP32 rate on this part, charged per warp instruction)
//   runs in full warps, and a node's last arriving child appends it to the
//   next round's queue.  The block also lists the spanning nodes whose index
//   it holds.
// * one — boundary_chain_kernel: the nodes containing boundary b and no other
//   are nested, one per level; one warp computes them from the deepest up.
// * more — span_stage_kernel gathers their children over the whole device;
//   centroid_top_kernel, one thread-block cluster, computes them level by
//   level from the deepest, a cluster barrier between levels (a node's
//   children are one level deeper at least).  At one level the quad nodes'
//   ranges are disjoint and each of these contains a block boundary, so a
//   level lists fewer nodes than there are blocks.
// On a uniform 1M-point tree ~5,200 nodes span blocks (15 levels), 341 of
// them (5 levels) more than one boundary.  (A climb by the last arriving child
// through device-scope counters did the spanning nodes before: one serial
// chain of L2 round trips per level, 58 us of the pass.)
constexpr int kCenThreads = 512;
constexpr int kCenSpan = kCenSpanC;

struct CenSmem {
  double2 cen[kCenSpan];
  int4 kids[kCenSpan];
  float2 pts[kCenSpan];
  int dlt[kCenSpan];
  int par[kCenSpan];       // quad parent of the local node at this index
  int leafpar[kCenSpan];   // quad parent of the point at this index
  int arrive[kCenSpan];
  int queue[2][kCenSpan];
  unsigned short need[kCenSpan];  // children of the local quad node here (<= kCenSpan), 0 if none
  int qn[2];
};

// Centroid of quad node `node` from global memory: its children's centroids
// were written by an earlier launch or before the last cluster barrier (read
// through L2).
__device__ double2 quad_centroid_global(const TreeArgs &t, int node) {
  double cx = 0.0, cy = 0.0;
  int cnt = 0;
  if (t.dlt[node] >= 64) {
    const int2 rg = t.range[node];
    for (int q = rg.x; q <= rg.y; q++) {
      const float2 v = t.spos[q];
      cx = cnt ? __dadd_rn(cx, f2d_int(v.x)) : zero_plus(f2d_int(v.x));
      cy = cnt ? __dadd_rn(cy, f2d_int(v.y)) : zero_plus(f2d_int(v.y));
      cnt++;
    }
  } else {
    const int4 kk = t.qkids[node];
    const int kids[4] = {kk.x, kk.y, kk.z, kk.w};
    double vx[4], vy[4];
#pragma unroll
    for (int c = 0; c < 4; c++) {  // the loads first, then the ordered sum
      const int ch = kids[c];
      vx[c] = vy[c] = 0.0;
      if (ch == kNoChild) continue;
      if (ch < 0) {
        const float2 v = t.spos[~ch];
        vx[c] = f2d_int(v.x);
        vy[c] = f2d_int(v.y);
      } else {
        const double2 v = __ldcg(&t.qcen[ch]);
        vx[c] = v.x;
        vy[c] = v.y;
      }
    }
#pragma unroll
    for (int c = 0; c < 4; c++) {
      if (kids[c] == kNoChild) break;
      cx = c ? __dadd_rn(cx, vx[c]) : zero_plus(vx[c]);
      cy = c ? __dadd_rn(cy, vy[c]) : zero_plus(vy[c]);
      cnt++;
    }
  }
  return make_double2(div_count_int(cx, cnt), div_count_int(cy, cnt));
}

// Centroids of the quad nodes that contain boundary b and no other (one
// warp).  They are nested, one per level, each the parent of the
// next deeper one; their other children lie inside block b or b+1 (done) or
// are points.  Lane i takes the i-th deepest node: its structure and its done
// children are loaded in parallel, then the nodes are summed from the deepest
// up, each taking the one below from the lane before it.
__device__ __forceinline__ void chain_centroids(const TreeArgs &t, int b) {
  const int lane = threadIdx.x & 31;
  const unsigned long long mask = __ldcg(&t.chain_mask[b]);
  const int cnt = __popcll(mask);
  if (cnt == 0) return;
  if (cnt > 32) {  // every level: one lane, in order (the others wait at the shuffle-free path)
    if (lane == 0)
      for (int lvl = kQuadLevels - 1; lvl >= 0; lvl--)
        if ((mask >> lvl) & 1ull) {
          const int node = __ldcg(&t.chain_node[b * kQuadLevels + lvl]);
          t.qcen[node] = quad_centroid_global(t, node);
        }
    __syncwarp();
    return;
  }
  // lane i: the level of the (i+1)-th highest set bit
  int lvl = -1;
  {
    int seen = 0;
    for (int l = kQuadLevels - 1; l >= 0; l--)
      if ((mask >> l) & 1ull) {
        if (seen == lane) lvl = l;
        seen++;
      }
  }
  const bool mine = lane < cnt;
  const int node = mine ? __ldcg(&t.chain_node[b * kQuadLevels + lvl]) : -1;
  const int below = __shfl_up_sync(0xffffffffu, node, 1);  // the next deeper chain node
  double2 v[4] = {make_double2(0.0, 0.0), make_double2(0.0, 0.0), make_double2(0.0, 0.0), make_double2(0.0, 0.0)};
  int nc = 0, from_below = -1;
  double2 run = make_double2(0.0, 0.0);
  bool is_run = false;
  if (mine) {
    const int p = t.dlt[node];
    if (p >= 64) {  // a run: points only
      is_run = true;
      run = quad_centroid_global(t, node);
    } else {
      const int4 kk = t.qkids[node];
      const int kids[4] = {kk.x, kk.y, kk.z, kk.w};
#pragma unroll
      for (int c = 0; c < 4; c++) {
        const int ch = kids[c];
        if (ch == kNoChild) continue;
        nc = c + 1;
        if (lane > 0 && ch == below) {
          from_below = c;
        } else if (ch < 0) {
          const float2 pt = t.spos[~ch];
          v[c] = make_double2(f2d_int(pt.x), f2d_int(pt.y));
        } else {
          v[c] = __ldcg(&t.qcen[ch]);
        }
      }
    }
  }
  double2 prev = make_double2(0.0, 0.0), mine_c = make_double2(0.0, 0.0);
  for (int i = 0; i < cnt; i++) {
    if (lane == i) {
      if (is_run) {
        mine_c = run;
      } else {
        double cx = 0.0, cy = 0.0;
#pragma unroll
        for (int c = 0; c < 4; c++) {
          if (c >= nc) break;
          const double2 u = c == from_below ? prev : v[c];
          cx = c ? __dadd_rn(cx, u.x) : zero_plus(u.x);
          cy = c ? __dadd_rn(cy, u.y) : zero_plus(u.y);
        }
        mine_c = make_double2(div_count_int(cx, nc), div_count_int(cy, nc));
      }
    }
    prev.x = __shfl_sync(0xffffffffu, mine_c.x, i);
    prev.y = __shfl_sync(0xffffffffu, mine_c.y, i);
  }
  if (mine) t.qcen[node] = mine_c;
}

// One warp per block boundary (boundaries 0 .. nb-2).
constexpr int kChainThreads = 128;
__global__ void __launch_bounds__(kChainThreads) boundary_chain_kernel(TreeArgs t, int nbound) {
  if (!block_status_ok(t.st)) return;
  const int b = blockIdx.x * (kChainThreads / 32) + (threadIdx.x >> 5);
  if (b < nbound) chain_centroids(t, b);
}

__global__ void __launch_bounds__(kCenThreads) centroid_kernel(TreeArgs t) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  CenSmem &S = *reinterpret_cast<CenSmem *>(smem_raw);
  if (!block_status_ok(t.st)) return;
  const int tid = threadIdx.x;
  const int lo = blockIdx.x * kCenSpan, hi = min(t.n, lo + kCenSpan);
  // the block's points and local quad nodes, coalesced
  for (int j = lo + tid; j < hi; j += kCenThreads) {
    const int q = j - lo;
    S.pts[q] = t.spos[j];
    S.leafpar[q] = t.qpar[t.n - 1 + j];
    S.arrive[q] = 0;
    int need = 0;
    if (j < t.n - 1) {
      const int m = t.qnchild[j];
      const int2 rg = t.range[j];
      if (m > 0 && rg.x >= lo && rg.y < hi) {
        need = m;
        S.kids[q] = t.qkids[j];
        S.dlt[q] = t.dlt[j];
        S.par[q] = t.qpar[j];
      } else if (m > 0) {  // spans blocks
        const int lvl = quad_level(t.dlt[j]);
        const int bl = rg.x / kCenSpan;
        if (rg.y / kCenSpan == bl + 1) {  // one boundary: boundary_chain_kernel
          t.chain_node[bl * kQuadLevels + lvl] = j;
          atomicOr(&t.chain_mask[bl], 1ull << lvl);
        } else {  // more: centroid_top_kernel
          const int slot = atomicAdd(&t.span_cnt[lvl], 1);
          if (slot < t.span_cap) t.span_list[lvl * t.span_cap + slot] = j;
          else dev_record_error(t.st, DEV_BAD_INDEX);  // cannot happen (see above)
        }
      }
    }
    S.need[q] = (unsigned short)need;
  }
  if (tid < 2) S.qn[tid] = 0;
  __syncthreads();
  auto is_local = [&](int node) { return node >= lo && node < hi && S.need[node - lo] != 0; };
  // round 0: every point arrives at its quad parent
  for (int k = lo + tid; k < hi; k += kCenThreads) {
    const int par = S.leafpar[k - lo];
    if (par < 0 || !is_local(par)) continue;  // a spanning parent is listed by its own block
    if (atomicAdd(&S.arrive[par - lo], 1) == (int)S.need[par - lo] - 1) S.queue[0][atomicAdd(&S.qn[0], 1)] = par;
  }
  __syncthreads();
  // rounds: the ready local nodes, one per thread (bounded by the depth of
  // the block's subtrees: every round moves up one node)
  for (int cur = 0;; cur ^= 1) {
    const int cnt = S.qn[cur];
    if (cnt == 0) break;
    if (tid == 0) S.qn[cur ^ 1] = 0;
    __syncthreads();
    for (int q = tid; q < cnt; q += kCenThreads) {
      const int node = S.queue[cur][q];
      const int ln = node - lo;
      double cx = 0.0, cy = 0.0;
      int nc = 0;
      if (S.dlt[ln] >= 64) {
        // run of identical keys: every point is a child (the reference
        // recurses without end here; see the oracle's note)
        const int2 rg = t.range[node];
        for (int k = rg.x; k <= rg.y; k++) {
          const float2 v = S.pts[k - lo];
          cx = nc ? __dadd_rn(cx, f2d_int(v.x)) : zero_plus(f2d_int(v.x));
          cy = nc ? __dadd_rn(cy, f2d_int(v.y)) : zero_plus(f2d_int(v.y));
          nc++;
        }
      } else {
        const int4 kk = S.kids[ln];
        const int kids[4] = {kk.x, kk.y, kk.z, kk.w};
#pragma unroll
        for (int c = 0; c < 4; c++) {
          const int ch = kids[c];
          if (ch == kNoChild) break;
          double vx, vy;
          if (ch < 0) {  // a point of this block
            const float2 v = S.pts[~ch - lo];
            vx = f2d_int(v.x);
            vy = f2d_int(v.y);
          } else {  // a local node, done in an earlier round
            const double2 v = S.cen[ch - lo];
            vx = v.x;
            vy = v.y;
          }
          cx = c ? __dadd_rn(cx, vx) : zero_plus(vx);
          cy = c ? __dadd_rn(cy, vy) : zero_plus(vy);
          nc++;
        }
      }
      const double2 c2 = make_double2(div_count_int(cx, nc), div_count_int(cy, nc));
      S.cen[ln] = c2;
      t.qcen[node] = c2;
      const int up = S.par[ln];
      if (up < 0 || !is_local(up)) continue;
      if (atomicAdd(&S.arrive[up - lo], 1) == (int)S.need[up - lo] - 1)
        S.queue[cur ^ 1][atomicAdd(&S.qn[cur ^ 1], 1)] = up;
    }
    __syncthreads();
  }
  // startbase over the block (the round queues are free now): the blocks
  // before it plus an exclusive scan of startcnt inside it
  __syncthreads();
  const int span = hi - lo;
  const int q0 = 2 * tid, q1 = 2 * tid + 1;  // kCenSpan == 2 * kCenThreads
  const int c0 = q0 < span ? t.startcnt[lo + q0] : 0, c1 = q1 < span ? t.startcnt[lo + q1] : 0;
  const int bbase = t.blocktot[blockIdx.x];
  int x = c0 + c1;
  const int lane = tid & 31, w = tid >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  int *wsum = S.queue[0];
  if (lane == 31) wsum[w] = x;
  __syncthreads();
  int wpre = 0;
  for (int q = 0; q < w; q++) wpre += wsum[q];
  const int excl = bbase + wpre + x - (c0 + c1);
  if (q0 < span) t.startbase[lo + q0] = excl;
  if (q1 < span) t.startbase[lo + q1] = excl + c0;
}

// Pre-order records of the points and of the quad nodes inside one centroid
// block, one thread per sorted position (the nodes that span blocks are
// written by boundary_chain_kernel and centroid_top_kernel, beside which this
// kernel runs).
__global__ void __launch_bounds__(256) layout_local_kernel(TreeArgs t) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (!block_status_ok(t.st)) return;
  const int cap = 2 * t.n - 1;  // records: n leaves + at most n-1 quad nodes
  // every load that depends only on i first, then the range ends' offsets
  const bool leaf = i < t.n, inner = i < t.n - 1;
  const int sb = leaf ? t.startbase[i] : 0, sc = leaf ? t.startcnt[i] : 0;
  const float2 pt = leaf ? t.spos[i] : make_float2(0.f, 0.f);
  const int m = inner ? t.qnchild[i] : 0;
  const int2 rg = inner ? t.range[i] : make_int2(0, 0);
  const int qb = inner ? t.qbelow[i] : 0;
  const int p = inner ? t.dlt[i] : 0;
  const double2 c = inner ? t.qcen[i] : make_double2(0.0, 0.0);
  // a quad node (binary internal node i) inside one block or spanning one
  // boundary; the nodes spanning more are written by centroid_top_kernel
  const bool node = m > 0 && rg.y / kCenSpan - rg.x / kCenSpan <= 1;
  int sc_lo = 0, sb_lo = 0, sb_hi = 0;
  if (node) {
    sc_lo = t.startcnt[rg.x];
    sb_lo = t.startbase[rg.x];
    sb_hi = t.startbase[rg.y + 1];
  }
  if (leaf) {  // leaf (sorted point) i, after the quad nodes starting at i
    const int idx = i + sb + sc;
    if (idx < 0 || idx >= cap) {
      dev_record_error(t.st, DEV_BAD_INDEX);
      return;
    }
    // a leaf's z = -inf is never in doubt: no FP64 centroid or level needed
    t.nodes[idx] = make_float4(pt.x, pt.y, kLeafZ, __int_as_float(idx + 1));
  }
  int idx, skip;
  if (node && node_record_slot(t, rg.x, rg.y + 1, qb, sc_lo, sb_lo, sb_hi, idx, skip))
    write_node_record(t, idx, skip, quad_level(p), c);
}

constexpr int kTopCtas = 8;  // one cluster (the portable maximum size)
constexpr int kTopThreads = 1024;
constexpr int kTopCap = 1024;  // listed nodes per block held in shared memory (104 KB)
constexpr int kStageThreads = 128;

__device__ __forceinline__ void top_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ unsigned int top_cluster_rank() {
  unsigned int r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}

// v = the double2 at `p` in the shared memory of block `rank` of the cluster.
__device__ __forceinline__ double2 ld_cluster_double2(const double2 *p, unsigned int rank) {
  const unsigned int a = (unsigned int)__cvta_generic_to_shared(p);
  unsigned int ra;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(a), "r"(rank));
  double x, y;
  asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(x), "=d"(y) : "r"(ra));
  return make_double2(x, y);
}

// Position g of a listed node: level lvl's nodes follow the deeper levels'
// (off[lvl] = the deeper levels' count), node q of a level at g = off + q.
// In the cluster, block g % kTopCtas holds it in slot g / kTopCtas; its staged
// record sits at (g % kTopCtas) * kTopCap + g / kTopCtas.
struct SpanLevels {
  int cnt[kQuadLevels], off[kQuadLevels], total;
};

// Every thread of the block calls it.
__device__ __forceinline__ void span_levels(const TreeArgs &t, SpanLevels &L) {
  if (threadIdx.x < kQuadLevels) L.cnt[threadIdx.x] = max(0, min(t.span_cnt[threadIdx.x], t.span_cap));
  __syncthreads();
  if (threadIdx.x == 0) {
    int o = 0;
    for (int lvl = kQuadLevels - 1; lvl >= 0; lvl--) {
      L.off[lvl] = o;
      o += L.cnt[lvl];
    }
    L.total = o;
  }
  __syncthreads();
}

__device__ __forceinline__ int span_level_of(const SpanLevels &L, int g) {
  int lvl = 0;
  while (lvl < kQuadLevels - 1 && g < L.off[lvl]) lvl++;
  return lvl;
}

// Staging of the listed nodes, one thread each, over the whole device (the
// gathers of a node's children are scattered loads; on the cluster's few SMs
// alone they queue): the node's position, its record's place, and per child
// its centroid when it is final (a point, or a node within one block or
// spanning one boundary) or its node id when it is a listed node itself.  A run of identical keys (children: points only) is
// computed here.  Nothing is staged when the cluster cannot hold the nodes.
__global__ void __launch_bounds__(kStageThreads) span_stage_kernel(TreeArgs t) {
  __shared__ SpanLevels L;
  if (!block_status_ok(t.st)) return;
  span_levels(t, L);
  const int total = L.total;
  const int g = blockIdx.x * kStageThreads + threadIdx.x;
  if (total > kTopCtas * kTopCap || g >= total) return;
  const int lvl = span_level_of(L, g);
  const int idx = (g % kTopCtas) * kTopCap + g / kTopCtas;
  const int node = t.span_list[lvl * t.span_cap + (g - L.off[lvl])];
  if (node < 0 || node >= t.n - 1) {
    dev_record_error(t.st, DEV_BAD_INDEX);
    t.stage_meta[idx] = make_int4(-1, 0, -1, 0);
    t.stage_pend[idx] = make_int4(-1, -1, -1, -1);
    t.stage_val[idx] = make_double2(0.0, 0.0);
    return;
  }
  t.span_pos[node] = g;
  const int p = t.dlt[node];
  const int4 kk = t.qkids[node];
  const int2 nr = t.range[node];
  const int qb = t.qbelow[node];
  // its record's place (startbase of the whole range was written by centroid_kernel)
  int ridx, skip;
  if (!node_record_slot(t, nr.x, nr.y + 1, qb, t.startcnt[nr.x], t.startbase[nr.x], t.startbase[nr.y + 1], ridx,
                        skip))
    ridx = -1;
  const int lvl8 = quad_level(p) << 8;
  if (p >= 64) {  // a run
    t.stage_val[idx] = quad_centroid_global(t, node);
    t.stage_meta[idx] = make_int4(node, lvl8, ridx, skip);
    t.stage_pend[idx] = make_int4(-1, -1, -1, -1);
    return;
  }
  const int kids[4] = {kk.x, kk.y, kk.z, kk.w};
  int2 rg[4];
  double2 qc[4];
  float2 pt[4];
#pragma unroll
  for (int c = 0; c < 4; c++) {  // independent loads issued together
    const int ch = kids[c];
    rg[c] = make_int2(0, 0);
    qc[c] = make_double2(0.0, 0.0);
    pt[c] = make_float2(0.f, 0.f);
    if (ch == kNoChild) continue;
    if (ch < 0) {
      pt[c] = t.spos[~ch];
    } else {
      rg[c] = t.range[ch];
      qc[c] = __ldcg(&t.qcen[ch]);  // used only when the child is done (at most one boundary)
    }
  }
  int pend[4] = {-1, -1, -1, -1};
  int nc = 0;
#pragma unroll
  for (int c = 0; c < 4; c++) {
    const int ch = kids[c];
    if (ch == kNoChild) break;
    nc++;
    double2 v = make_double2(0.0, 0.0);
    if (ch < 0) v = make_double2(f2d_int(pt[c].x), f2d_int(pt[c].y));
    else if (rg[c].y / kCenSpan - rg[c].x / kCenSpan >= 2) pend[c] = ch;  // listed
    else v = qc[c];
    t.stage_val[(size_t)c * kTopCtas * kTopCap + idx] = v;
  }
  t.stage_pend[idx] = make_int4(pend[0], pend[1], pend[2], pend[3]);
  t.stage_meta[idx] = make_int4(node, nc | lvl8, ridx, skip);
}

struct TopSmem {
  double2 val[4][kTopCap];  // the children's centroids in quadrant order
  double2 cen[kTopCap];     // the node's centroid (read by the other blocks)
  int4 pend[kTopCap];       // cluster position of a listed child, -1 otherwise
  int node[kTopCap];
  int nc[kTopCap];          // children; 0 for a run (done when staged) or a bad entry
};

// The listed nodes, level by level from the deepest, in one cluster: each
// block loads its staged records and the positions of their listed children,
// then one level per round, a listed child read from the shared memory of the
// block holding it, a cluster barrier after every round.  Every thread reads
// the same level counts, so all take the same cluster barriers; every block
// reads the error record before the first barrier and this kernel records
// errors only after it, so all blocks leave together or none.  Each block
// then writes its nodes' centroids and pre-order records.  More listed nodes
// than the blocks can hold: the same rounds through global memory.
__global__ void __cluster_dims__(kTopCtas, 1, 1) __launch_bounds__(kTopThreads, 1)
    centroid_top_kernel(TreeArgs t) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  TopSmem &S = *reinterpret_cast<TopSmem *>(smem_raw);
  __shared__ SpanLevels L;
  __shared__ unsigned int s_code;
  const int tid = threadIdx.x;
  if (tid == 0) s_code = ld_volatile_u32(&t.st->code);
  top_cluster_sync();
  if (s_code != 0u) return;  // the tree of this iteration is not valid
  span_levels(t, L);
  const int total = L.total;
  if (total > kTopCtas * kTopCap) {
    for (int lvl = kQuadLevels - 1; lvl >= 0; lvl--) {
      const int cnt = L.cnt[lvl];
      if (cnt == 0) continue;
      for (int q = blockIdx.x * kTopThreads + tid; q < cnt; q += kTopCtas * kTopThreads) {
        const int node = t.span_list[lvl * t.span_cap + q];
        if (node < 0 || node >= t.n - 1) {
          dev_record_error(t.st, DEV_BAD_INDEX);
          continue;
        }
        const double2 c = quad_centroid_global(t, node);
        t.qcen[node] = c;  // read by the next levels
        write_node_record_global(t, node, c);
      }
      top_cluster_sync();
    }
    return;
  }
  const int crank = (int)top_cluster_rank();
  const int nslots = total > crank ? (total - crank + kTopCtas - 1) / kTopCtas : 0;
  for (int l = tid; l < nslots; l += kTopThreads) {
    const int idx = crank * kTopCap + l;
    const int4 meta = t.stage_meta[idx];
    const int4 pk = t.stage_pend[idx];
    int pend[4] = {pk.x, pk.y, pk.z, pk.w};
    int gc[4];
#pragma unroll
    for (int c = 0; c < 4; c++) gc[c] = pend[c] >= 0 ? __ldcg(&t.span_pos[pend[c]]) : -1;
#pragma unroll
    for (int c = 0; c < 4; c++) {
      if (pend[c] >= 0 && (gc[c] < 0 || gc[c] >= total)) {
        dev_record_error(t.st, DEV_BAD_INDEX);
        gc[c] = -1;
      }
      S.val[c][l] = t.stage_val[(size_t)c * kTopCtas * kTopCap + idx];
    }
    S.pend[l] = make_int4(gc[0], gc[1], gc[2], gc[3]);
    S.node[l] = meta.x;
    S.nc[l] = meta.y & 255;
    if ((meta.y & 255) == 0) S.cen[l] = S.val[0][l];  // a run (or a bad entry: zero)
  }
  top_cluster_sync();  // every block's staged records (and runs) in place
  // this thread's positions of level lvl: g = first + k * kTopCtas * kTopThreads
  auto first_of = [&](int lvl) {
    const int off = L.off[lvl];
    return off + (crank - off % kTopCtas + kTopCtas) % kTopCtas + kTopCtas * tid;
  };
  // the rounds (runs, level 32, were done when staged)
  for (int lvl = kQuadLevels - 2; lvl >= 0; lvl--) {
    if (L.cnt[lvl] == 0) continue;
    const int end = L.off[lvl] + L.cnt[lvl];
    for (int g = first_of(lvl); g < end; g += kTopCtas * kTopThreads) {
      const int l = g / kTopCtas;
      const int nc = S.nc[l];
      if (nc == 0) continue;
      const int4 pk = S.pend[l];
      const int pend[4] = {pk.x, pk.y, pk.z, pk.w};
      double2 v[4];
#pragma unroll
      for (int c = 0; c < 4; c++) {
        v[c] = S.val[c][l];
        if (c < nc && pend[c] >= 0) v[c] = ld_cluster_double2(&S.cen[pend[c] / kTopCtas], pend[c] % kTopCtas);
      }
      double cx = 0.0, cy = 0.0;
#pragma unroll
      for (int c = 0; c < 4; c++) {
        if (c >= nc) break;
        cx = c ? __dadd_rn(cx, v[c].x) : zero_plus(v[c].x);
        cy = c ? __dadd_rn(cy, v[c].y) : zero_plus(v[c].y);
      }
      S.cen[l] = make_double2(div_count_int(cx, nc), div_count_int(cy, nc));
    }
    // no global store is pending here, so the barrier's release has only
    // this round's shared-memory stores to order; it also keeps every
    // block's shared memory alive while the others read it
    top_cluster_sync();
  }
  for (int l = tid; l < nslots; l += kTopThreads) {
    const int4 meta = t.stage_meta[crank * kTopCap + l];
    if (meta.x < 0) continue;
    t.qcen[meta.x] = S.cen[l];  // every quad node's centroid stays readable by node id
    if (meta.z >= 0) write_node_record(t, meta.z, meta.w, meta.y >> 8, S.cen[l]);
  }
}

struct TraverseArgs {
  int n;
  DevStatus *st;
  const float4 *nodes;
  const double2 *nodes_c64;
  const unsigned char *nodes_lvl;
  const double *frame;
  const float2 *spos;
  const int *perm;
  float2 *rep;
  double theta;
  unsigned long long *stats;  // [visits, fp64 decisions] or null
  // the attraction of the neighbours that have not moved yet in this
  // iteration (unmoved_attraction_kernel); the walk adds minus the
  // repulsion; null to skip
  float4 *f0;
};

// FR attraction (algorithms.cpp:1056-1058) of the neighbours of v that have
// not moved before v in the iteration (same or later batch), float-float, by
// vertex id.  It needs no tree, so it runs on the second stream beside the
// sort and the tree; the walk then adds minus the repulsion.
// A thread takes a row of up to kHubRow neighbours, a warp a longer one: its
// lanes fetch 32 neighbours at once and form the factors, which every lane
// then multiplies and adds in CSR order, so the sum is the thread's bit for bit.
// A thread alone is bound by its fetches, two dependent L2 round trips per four
// neighbours: 100,003 vertices, the longest row 633 neighbours, 155 us by
// threads only (longer than the sort and the tree beside it), 49 with the
// warps.  The vertices with long rows often have neighbouring ids, so a block
// takes groups of 8 vertices from all over the range (8 keep the rows' offsets
// and the results in whole sectors) and its warps share the long rows among
// them.
constexpr int kHubRow = 32;
constexpr int kAttractThreads = 256;

__device__ __forceinline__ float4 hub_unmoved_attraction(int v, const int *__restrict__ rowptr,
                                                         const int *__restrict__ colids, const float2 *pold, int batch,
                                                         float W) {
  const int lane = threadIdx.x & 31;
  const float2 pv = pold[v];
  const int batch_lo = (v / batch) * batch;
  const unsigned int e0 = rowptr[v], e1 = rowptr[v + 1];  // (unsigned: two chunks past the end are compared too)
  auto column = [&](unsigned int e) { return e < e1 ? colids[e] : -1; };
  auto position = [&](int j) { return j >= batch_lo ? pold[j] : pv; };
  float hx = 0.f, lx = 0.f, hy = 0.f, ly = 0.f;
  int j = column(e0 + lane), jn = column(e0 + 32 + lane);
  float2 p = position(j);
  for (unsigned int e = e0; e < e1; e += 32) {  // positions one chunk ahead, columns two
    const float2 pn = position(jn);
    const int j2 = column(e + 64 + lane);
    const float dx = p.x - pv.x, dy = p.y - pv.y;
    const float sc = W * sqrtf(fmaf(dx, dx, dy * dy));
    const unsigned int m = __ballot_sync(0xffffffffu, j >= batch_lo);  // past the row's end j is -1
#pragma unroll 8
    for (int q = 0; q < 32; q++) {
      const float x = __shfl_sync(0xffffffffu, dx, q), y = __shfl_sync(0xffffffffu, dy, q);
      const float s = __shfl_sync(0xffffffffu, sc, q);
      if ((m >> q) & 1u) {  // the products here, as in bh_attract: the sums take them unrounded
        ff_add(hx, lx, x * s);
        ff_add(hy, ly, y * s);
      }
    }
    j = jn;
    jn = j2;
    p = pn;
  }
  return make_float4(hx, hy, lx, ly);
}

__global__ void __launch_bounds__(kAttractThreads) unmoved_attraction_kernel(int n, const int *__restrict__ rowptr,
                                                                             const int *__restrict__ colids,
                                                                             const float2 *pold, int batch, float W,
                                                                             float4 *f0) {
  __shared__ int hub[kAttractThreads];
  __shared__ int nhub;
  if (threadIdx.x == 0) nhub = 0;
  __syncthreads();
  const long long v = 8ll * ((threadIdx.x >> 3) * (long long)gridDim.x + blockIdx.x) + (threadIdx.x & 7);
  if (v < n) {
    if (rowptr[v + 1] - rowptr[v] <= kHubRow) f0[v] = bh_unmoved_attraction((int)v, rowptr, colids, pold, batch, W);
    else hub[atomicAdd(&nhub, 1)] = (int)v;
  }
  __syncthreads();
  for (int h = threadIdx.x >> 5; h < nhub; h += kAttractThreads / 32) {
    const float4 f = hub_unmoved_attraction(hub[h], rowptr, colids, pold, batch, W);
    if ((threadIdx.x & 31) == 0) f0[hub[h]] = f;
  }
}

// 128 threads per block: measured 1.5 % faster than 256 and 512 on the 1M
// graph (finer blocks, smaller tail); 64 is no better.
constexpr int kTravThreads = 128;

template <bool kStats>
__global__ void __launch_bounds__(kTravThreads) traverse_kernel(TraverseArgs a) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (!block_status_ok(a.st)) return;  // the tree of this iteration is not valid
  if (k >= a.n) return;
  const float2 q = a.spos[k];
  // record 0 is the root; its skip link is the number of records
  int total = __float_as_int(__ldg(&a.nodes[0]).w);
  if (total < 0 || total > 2 * a.n - 1) {
    dev_record_error(a.st, DEV_BAD_INDEX);
    total = 0;
  }
  unsigned int visits = 0, exact = 0;
  const float2 rep = bh_repulsion<true, kStats>(a.nodes, a.nodes_c64, a.nodes_lvl, a.frame[2], a.theta,
                                                total, q, visits, exact);
  const int v = a.perm[k];
  a.rep[v] = rep;
  // minus the repulsion into v's sum of unmoved neighbours' attraction
  if (a.f0) a.f0[v] = bh_minus_repulsion(a.f0[v], rep);
  if (kStats) {  // one atomic per group of converged lanes, not per thread
    const unsigned int m = __activemask();
    const unsigned int sv = __reduce_add_sync(m, visits), se = __reduce_add_sync(m, exact);
    if ((threadIdx.x & 31u) == (unsigned int)(__ffs(m) - 1)) {
      atomicAdd(&a.stats[0], (unsigned long long)sv);
      if (se) atomicAdd(&a.stats[1], (unsigned long long)se);
    }
  }
}

struct SweepArgs {
  const int *order;        // vertices grouped by dependency level
  const int *group_start;  // groups + 1 offsets into order
  const int *early_off;  // per level-order slot: earlier-batch neighbours
  const int *early_col;
  int groups;
  const float4 *f0;      // attraction of unmoved neighbours minus repulsion (float-float)
  float4 *f0out;         // the same array: the final float-float force when write_out
  const float2 *pold;
  float2 *pnew;          // every entry kUnmoved before the launch
  int write_out;
  float W;
  float step;
  DevStatus *st;
};

constexpr int kSweepThreads = 1024;
constexpr unsigned int kSweepSleep = 100;  // ns

// A new position not yet written: both coordinates NaN, all bits set
// (no layout coordinate is NaN).  pnew is filled with it before the sweep.
constexpr unsigned long long kUnmoved = 0xffffffffffffffffull;

__device__ __forceinline__ unsigned long long ld_relaxed_u64(const float2 *p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void st_relaxed_u64(float2 *p, float2 v) {
  const unsigned long long b =
      (unsigned long long)__float_as_uint(v.x) | ((unsigned long long)__float_as_uint(v.y) << 32);
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(b) : "memory");
}

__device__ __forceinline__ float2 unpack_pos(unsigned long long b) {
  return make_float2(__uint_as_float((unsigned int)b), __uint_as_float((unsigned int)(b >> 32)));
}

// A vertex's data that does not change during the sweep: its slot in the
// level order, id, iteration-start position, f0, earlier-batch neighbour
// range and the first four of those neighbours (most vertices have no more).
struct SweepVertex {
  int t, i;
  float2 pi;
  float4 f;
  int e0, e1;
  int c[4];
};

__device__ __forceinline__ void sweep_load(const SweepArgs &a, int t, SweepVertex &v) {
  v.t = t;
  v.i = a.order[t];
  v.pi = a.pold[v.i];
  v.f = a.f0[v.i];
  v.e0 = a.early_off[t];
  v.e1 = a.early_off[t + 1];
#pragma unroll
  for (int q = 0; q < 4; q++) v.c[q] = (v.e0 + q < v.e1) ? a.early_col[v.e0 + q] : 0;
}

// The vertices of a warp (one a lane, has: the lane has one): adds the
// attraction of the neighbours that moved earlier in this iteration (earlier
// batches, their new positions) to f0, then the unit-step update
// (algorithms.cpp:1056-1066).  FP32 terms, float-float sum in neighbour
// order, FP32 unit vector.
// A neighbour's new position, which an earlier dependency level writes, is an
// 8-byte word that is its own ready flag (a single-copy atomic 64-bit access):
// one load both tests and reads it.  The warp stays converged: in every round
// each lane loads the words of its next four neighbours (only the first while
// it waits for that one), takes those that are there and, with the last,
// publishes its own position.  So a row of many moved neighbours costs a round
// trip per four of them, all lanes at once; a lane that waits alone and then
// loads its neighbours one by one holds up the warp and every level after it
// (the sweep of 100,003 vertices of a power-law graph, 32 levels, up to 22 moved
// neighbours, 118 us that way, 94 this; of 1,000,000 of a geometric one 77 and
// 58).  The wait is bounded; false when it ran out or another thread recorded
// an error (the same in every lane).
__device__ __forceinline__ bool sweep_group(const SweepArgs &a, const SweepVertex &v, bool has) {
  float hx = v.f.x, hy = v.f.y, lx = v.f.z, ly = v.f.w;
  int c[4] = {v.c[0], v.c[1], v.c[2], v.c[3]};
  int e = v.e0;
  bool more = has, wide = true;
  unsigned long long t0 = 0;
  for (unsigned int round = 0;; round++) {
    const int left = more ? v.e1 - e : 0, ask = wide ? left : min(left, 1);
    unsigned long long b[4];
#pragma unroll
    for (int q = 0; q < 4; q++) b[q] = q < ask ? ld_relaxed_u64(&a.pnew[c[q]]) : kUnmoved;
    int got = 0;
#pragma unroll
    for (int q = 0; q < 4; q++)
      if (got == q && b[q] != kUnmoved) {
        bh_attract(unpack_pos(b[q]), v.pi, a.W, hx, lx, hy, ly);
        got = q + 1;
      }
    if (more && got == left) {  // all are in (left > 4 never equals got)
      more = false;
      const float2 np = bh_step(v.pi, hx, lx, hy, ly, a.step);
      // the force's float-float sums replace f0 (read above, not needed again);
      // bh_forces_kernel turns them into the FP64 force and |f|^2 in full warps
      if (a.write_out) a.f0out[v.i] = make_float4(hx, hy, lx, ly);
      st_relaxed_u64(&a.pnew[v.i], np);  // publishes the position: later levels wait for this word
    }
    if (!__any_sync(0xffffffffu, more)) return true;
    wide = got > 0;
    if (more && got > 0) {
      e += got;
#pragma unroll
      for (int q = 0; q < 4; q++) c[q] = e + q < v.e1 ? a.early_col[e + q] : 0;
    }
    if (!__any_sync(0xffffffffu, got > 0)) {
      __nanosleep(kSweepSleep);  // fewer polls queued at L2 while the writers work
      if ((round & 63u) == 63u) {
        const unsigned long long now = dev_globaltimer();
        if (t0 == 0) t0 = now;
        bool quit = ld_volatile_u32(&a.st->code) != 0u;
        if (!quit && now - t0 > kBarrierTimeoutNs) {
          dev_record_error(a.st, DEV_TIMEOUT_SWEEP);
          quit = true;
        }
        if (__any_sync(0xffffffffu, quit)) return false;
      }
    }
  }
}

// All dependency levels of an iteration in one launch, without barriers: a
// vertex waits only for the new positions of its own earlier-batch
// neighbours (bounded waits on their position words).  The slots of each
// level are cut into 32-slot groups, numbered across the levels in level
// order, and group G goes to warp G mod W (W warps in the grid, numbered so
// that consecutive groups land on different SMs): every warp gets about the
// same number of groups, and takes them in level order.  A warp finishes a
// group before it starts the next, so a slot waits only on slots
// of lower levels held by other warps or by this warp's finished groups; with
// every block resident (a cooperative launch) the warp holding the lowest
// unfinished slot can always proceed, so the sweep cannot deadlock.  A thread
// loads its next slot's vertex data before it waits on the current slot's
// neighbours.  Bound by the levels: each is a round trip to see the position,
// the update and the store; 72 us for the 100,003 vertices above, 48 for the
// 1,000,000.  The groups' first slots are a table made with the levels: found
// here (a walk over the levels' ends, 64-bit remainders) they took 22 and 10 us
// more.  Blocks of 512 threads are 4 us faster at 100,003 vertices, 11 slower
// at 1,000,000 and 45 at 3,000,000.
__global__ void __launch_bounds__(kSweepThreads, 1) sweep_kernel(SweepArgs a) {
  if (!block_status_ok(a.st)) return;
  const int W = gridDim.x * (blockDim.x >> 5);
  const int lane = threadIdx.x & 31;
  const int w = ((int)threadIdx.x >> 5) * (int)gridDim.x + (int)blockIdx.x;
  auto load = [&](int g, SweepVertex &v) {  // whether the lane has a vertex in group g
    if (g >= a.groups) return false;
    const int t = a.group_start[g] + lane;
    if (t >= a.group_start[g + 1]) return false;
    sweep_load(a, t, v);
    return true;
  };
  SweepVertex cur{};
  bool has = load(w, cur);
  for (int g = w; g < a.groups; g += W) {
    SweepVertex nxt{};
    const bool nhas = load(g + W, nxt);
    if (!sweep_group(a, cur, has)) return;  // the group is done before the warp's next one starts
    cur = nxt;
    has = nhas;
  }
}

// The FP64 force f = hi + lo of each vertex (exact conversions, one addition
// per component) and |f|^2, from the float-float sums the sweep left: the
// values the reference's prevCoordinates and energy take, computed in full
// warps by vertex id.
__global__ void bh_forces_kernel(const float4 *__restrict__ ff, int n, double2 *__restrict__ force,
                                 double *__restrict__ e) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 v = ff[i];
  const double fx = __dadd_rn(f2d_int(v.x), f2d_int(v.z)), fy = __dadd_rn(f2d_int(v.y), f2d_int(v.w));
  force[i] = make_double2(fx, fy);
  e[i] = __fma_rn(fx, fx, __dmul_rn(fy, fy));
}

inline int nblk(long long n, int t) { return (int)((n + t - 1) / t); }

// `missing` blocks never arrive; the others wait at the sort's grid barrier.
__global__ void __launch_bounds__(kSortThreads) sort_barrier_selftest_kernel(SortArgs a, int missing) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  if ((int)blockIdx.x >= missing) sort_barrier(a, *reinterpret_cast<SortSmem *>(smem_raw), 1);
}

}  // namespace

int sort_wait_selftest(bl_ctx *ctx, bool complete) {
  if (!ctx->s.bbox) return bl_fail(ctx, -7, "no graph loaded");
  BL_CUDA(ctx, cudaFuncSetAttribute(sort_barrier_selftest_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)sizeof(SortSmem)));
  BL_CUDA(ctx, cudaMemsetAsync(ctx->s.bbox, 0xff, 5 * sizeof(unsigned int), ctx->stream));
  SortArgs a{};
  a.ctl = ctx->s.bbox;
  a.st = ctx->s.status;
  int missing = complete ? 0 : 1;
  void *args[] = {&a, &missing};
  BL_CUDA(ctx, cudaLaunchCooperativeKernel((const void *)sort_barrier_selftest_kernel, dim3(8), dim3(kSortThreads),
                                           args, sizeof(SortSmem), ctx->stream));
  return 0;
}

int ensure_bh_scratch(bl_ctx *ctx) {
  const size_t n = (size_t)ctx->g.n;
  Scratch &s = ctx->s;
  if (s.bh_n >= n && s.keys) return 0;
  auto fr = [](void *p) { if (p) cudaFree(p); };
  fr(s.keys); fr(s.keys_alt); fr(s.perm); fr(s.perm_alt); fr(s.hist); fr(s.spos);
  fr(s.bparent); fr(s.brange); fr(s.bdelta); fr(s.qkids); fr(s.qpar); fr(s.qnchild);
  fr(s.span); fr(s.span_stage); fr(s.ztab); fr(s.chain); fr(s.qcen);
  fr(s.qbelow); fr(s.startcnt); fr(s.startbase); fr(s.nodes); fr(s.nodes_c64);
  fr(s.nodes_lvl); fr(s.rep); fr(s.f0); fr(s.pos_alt); fr(s.runs); fr(s.bnode); fr(s.pairs);
  const size_t m = std::max<size_t>(n, 2);
  BL_CUDA(ctx, cudaMalloc(&s.keys, m * 8));
  BL_CUDA(ctx, cudaMalloc(&s.keys_alt, m * 8));
  BL_CUDA(ctx, cudaMalloc(&s.perm, m * 4));
  BL_CUDA(ctx, cudaMalloc(&s.perm_alt, m * 4));
  BL_CUDA(ctx, cudaMalloc(&s.pairs, 2 * m * 8));
  BL_CUDA(ctx, cudaMalloc(&s.spos, m * sizeof(float2)));
  BL_CUDA(ctx, cudaMalloc(&s.bparent, m * sizeof(int)));
  BL_CUDA(ctx, cudaMalloc(&s.brange, m * sizeof(int2)));
  BL_CUDA(ctx, cudaMalloc(&s.bnode, 2 * m * sizeof(int4)));
  BL_CUDA(ctx, cudaMalloc(&s.bdelta, m * sizeof(int)));
  BL_CUDA(ctx, cudaMalloc(&s.qkids, m * sizeof(int4)));
  BL_CUDA(ctx, cudaMalloc(&s.qpar, 2 * m * sizeof(int)));
  BL_CUDA(ctx, cudaMalloc(&s.qnchild, m * sizeof(int)));
  BL_CUDA(ctx, cudaMalloc(&s.ztab, kQuadLevels * sizeof(float)));
  {
    const size_t cap = (size_t)nblk((long long)m, kCenSpan);
    BL_CUDA(ctx, cudaMalloc(&s.chain, cap * (sizeof(unsigned long long) + kQuadLevels * sizeof(int))));
  }
  s.span_cap = nblk((long long)m, kCenSpan);
  BL_CUDA(ctx, cudaMalloc(&s.span, (kQuadLevels + (s.span_cap + 1) + (size_t)kQuadLevels * s.span_cap + m) *
                                        sizeof(int)));
  BL_CUDA(ctx, cudaMalloc(&s.span_stage, (size_t)kTopCtas * kTopCap * (4 * sizeof(double2) + 2 * sizeof(int4))));
  BL_CUDA(ctx, cudaMalloc(&s.qcen, m * sizeof(double2)));
  BL_CUDA(ctx, cudaMalloc(&s.qbelow, m * sizeof(int)));
  BL_CUDA(ctx, cudaMalloc(&s.startcnt, (m + 1) * sizeof(int)));
  BL_CUDA(ctx, cudaMalloc(&s.startbase, (m + 1) * sizeof(int)));
  BL_CUDA(ctx, cudaMalloc(&s.nodes, 2 * m * sizeof(float4)));
  BL_CUDA(ctx, cudaMalloc(&s.nodes_c64, 2 * m * sizeof(double2)));
  BL_CUDA(ctx, cudaMalloc(&s.nodes_lvl, 2 * m));
  BL_CUDA(ctx, cudaMalloc(&s.rep, m * sizeof(float2)));
  BL_CUDA(ctx, cudaMalloc(&s.f0, m * sizeof(float4)));
  BL_CUDA(ctx, cudaMalloc(&s.pos_alt, m * sizeof(float2)));
  s.runs_cap = (int)(m / (kRunShort + 1) + 1);  // runs longer than kRunShort: at most n / (kRunShort + 1)
  BL_CUDA(ctx, cudaMalloc(&s.runs, (2 * (size_t)s.runs_cap + 1) * sizeof(int)));
  // the sort's tiles: one a resident block where 16 keys a thread are enough
  // (they then stay in shared memory between the ranking and the scatter),
  // else an even number of tiles a block
  BL_CUDA(ctx, cudaFuncSetAttribute(morton_sort_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)sizeof(SortSmem)));
  int occ = 0;
  BL_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, morton_sort_kernel, kSortThreads,
                                                             sizeof(SortSmem)));
  if (occ < 1) return bl_fail(ctx, -5, "sort kernel cannot be resident");
  const int resident = ctx->num_sms * occ;
  const long long per_wave = (long long)resident * kSortThreads;
  const int waves = (int)((m + per_wave * kSortItems - 1) / (per_wave * kSortItems));
  s.sort_items = (int)((m + per_wave * waves - 1) / (per_wave * waves));
  s.sort_tiles = nblk((long long)m, s.sort_items * kSortThreads);
  s.sort_grid = std::min(s.sort_tiles, resident);
  BL_CUDA(ctx, cudaMalloc(&s.hist, ((size_t)s.sort_tiles + 4 * kSortGroups) * 256 * sizeof(unsigned int)));
  // set here, outside any stream capture of the iteration
  BL_CUDA(ctx, cudaFuncSetAttribute(centroid_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)sizeof(CenSmem)));
  BL_CUDA(ctx, cudaFuncSetAttribute(centroid_top_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)sizeof(TopSmem)));
  s.bh_n = n;
  return 0;
}

// Steps 1-4 for the positions `pos`; leaves the pre-order records in
// ctx->s.nodes (total = n + number of quad nodes, read back by callers that
// need it via startbase[n]).
int bh_build(bl_ctx *ctx, const float2 *pos, double theta, int attract_batch) {
  const int n = ctx->g.n;
  Scratch &s = ctx->s;
  cudaStream_t st = ctx->stream;
  if (n < 2) return 0;
  const int ncb = nblk(n, kCenSpan);  // centroid blocks
  // the walk's attraction part (for the iteration that follows) needs no
  // tree: on the second stream (lower priority) beside the sort
  if (attract_batch > 0) {
    const bool side = ctx->side && ctx->ev_fork && ctx->ev_join;
    if (side) {
      BL_CUDA(ctx, cudaEventRecord(ctx->ev_fork, st));
      BL_CUDA(ctx, cudaStreamWaitEvent(ctx->side, ctx->ev_fork, 0));
    }
    unmoved_attraction_kernel<<<nblk(n, kAttractThreads), kAttractThreads, 0, side ? ctx->side : st>>>(
        n, ctx->g.rowptr, ctx->g.colids, pos, attract_batch, (float)ctx->weight, s.f0);
    ctx->launches++;
  }
  bl_time_begin(ctx, "morton_sort");
  BL_CUDA(ctx, cudaMemsetAsync(s.bbox, 0xff, 5 * sizeof(unsigned int), st));
  {
    SortArgs a;
    a.pos = pos;
    a.n = n;
    a.items = s.sort_items;
    a.ntiles = s.sort_tiles;
    a.group = (s.sort_tiles + kSortGroups - 1) / kSortGroups;
    a.ctl = s.bbox;
    a.frame = s.frame;
    a.kframe = reinterpret_cast<KeyFrame *>(s.frame + 4);
    a.inv_theta2 = 1.0 / (theta * theta);
    a.ztab = s.ztab;
    a.pairs0 = s.pairs;
    a.pairs1 = s.pairs + std::max(n, 2);
    a.hist = s.hist;
    a.gtot = s.hist + (size_t)s.sort_tiles * 256;
    a.runs = s.runs;
    // span_cnt, the block totals and the boundary chains' level masks
    a.zero0 = s.span;
    a.nzero0 = kQuadLevels + ncb + 1;
    a.zero1 = reinterpret_cast<int *>(s.chain);
    a.nzero1 = 2 * ncb;
    a.st = s.status;
    void *args[] = {&a};
    BL_CUDA(ctx, cudaLaunchCooperativeKernel((const void *)morton_sort_kernel, dim3(s.sort_grid), dim3(kSortThreads),
                                             args, sizeof(SortSmem), st));
    ctx->launches++;
  }
  morton_emit_kernel<<<nblk(n, 256), 256, 0, st>>>(pos, n, s.pairs + std::max(n, 2),
                                                   reinterpret_cast<const KeyFrame *>(s.frame + 4), s.keys, s.perm, s.spos,
                                                   s.runs, s.runs_cap, s.status);
  ctx->launches++;
  run_sort_kernel<<<std::min(s.runs_cap, ctx->num_sms), kRunThreads, 0, st>>>(
      s.keys, s.perm, s.keys_alt, s.perm_alt, s.runs, s.runs_cap, pos, s.spos, s.status);
  ctx->launches++;
  bl_time_end(ctx, "morton_sort");
  bl_time_begin(ctx, "radix_tree");
  radix_tree_kernel<<<nblk(n - 1, 256), 256, 0, st>>>(s.keys, n, s.brange, s.bdelta, s.bparent,
                                                       reinterpret_cast<int *>(s.bnode));
  bl_time_end(ctx, "radix_tree");
  TreeArgs t;
  t.n = n;
  t.spos = s.spos;
  t.range = s.brange;
  t.dlt = s.bdelta;
  t.leaf_parent = s.bparent;
  t.qkids = s.qkids;
  t.qcen = s.qcen;
  t.qbelow = s.qbelow;
  t.startcnt = s.startcnt;
  t.qpar = s.qpar;
  t.qnchild = s.qnchild;
  t.span_cnt = s.span;
  t.blocktot = s.span + kQuadLevels;
  t.span_list = t.blocktot + s.span_cap + 1;
  t.span_cap = s.span_cap;
  t.span_pos = t.span_list + (size_t)kQuadLevels * s.span_cap;
  t.startbase = s.startbase;
  t.ztab = s.ztab;
  t.chain_mask = reinterpret_cast<unsigned long long *>(s.chain);
  t.chain_node = reinterpret_cast<int *>(t.chain_mask + s.span_cap);
  t.nodes = s.nodes;
  t.nodes_c64 = s.nodes_c64;
  t.nodes_lvl = s.nodes_lvl;
  t.stage_val = reinterpret_cast<double2 *>(s.span_stage);
  t.stage_pend = reinterpret_cast<int4 *>(t.stage_val + 4 * kTopCtas * kTopCap);
  t.stage_meta = reinterpret_cast<int4 *>(t.stage_pend + kTopCtas * kTopCap);
  t.bnode = s.bnode;
  t.st = s.status;
  bl_time_begin(ctx, "chain_kernel");
  chain_kernel<<<nblk(n, 256), 256, 0, st>>>(t);
  block_base_kernel<<<1, 1024, 0, st>>>(t.blocktot, ncb, s.startbase + n);
  ctx->launches++;
  bl_time_end(ctx, "chain_kernel");
  bl_time_begin(ctx, "centroid_kernel");
  centroid_kernel<<<nblk(n, kCenSpan), kCenThreads, sizeof(CenSmem), st>>>(t);
  // the quad nodes spanning one boundary (one warp per boundary); then on the
  // side stream (at the lower priority) the records of the points and of the
  // nodes spanning at most one boundary, beside the nodes spanning more (one
  // cluster, which leaves most SMs free)
  const bool fork = ctx->side && ctx->ev_fork && ctx->ev_join;
  const bool spans = ncb > 1;  // one block has no spanning node
  bl_time_begin(ctx, "centroid_top");
  if (spans) {
    boundary_chain_kernel<<<nblk(ncb - 1, kChainThreads / 32), kChainThreads, 0, st>>>(t, ncb - 1);
    ctx->launches++;
  }
  if (fork) {
    BL_CUDA(ctx, cudaEventRecord(ctx->ev_fork, st));
    BL_CUDA(ctx, cudaStreamWaitEvent(ctx->side, ctx->ev_fork, 0));
  }
  layout_local_kernel<<<nblk(n, 256), 256, 0, fork ? ctx->side : st>>>(t);
  ctx->launches++;
  if (fork) BL_CUDA(ctx, cudaEventRecord(ctx->ev_join, ctx->side));
  if (spans) {
    span_stage_kernel<<<kTopCtas * kTopCap / kStageThreads, kStageThreads, 0, st>>>(t);
    centroid_top_kernel<<<kTopCtas, kTopThreads, sizeof(TopSmem), st>>>(t);
    ctx->launches += 2;
  }
  if (fork) BL_CUDA(ctx, cudaStreamWaitEvent(st, ctx->ev_join, 0));
  bl_time_end(ctx, "centroid_top");
  bl_time_end(ctx, "centroid_kernel");
  ctx->launches += 4;
  BL_CUDA(ctx, cudaGetLastError());
  return 0;
}

int bh_traverse(bl_ctx *ctx, double theta, bool want_stats, int batch) {
  const int n = ctx->g.n;
  Scratch &s = ctx->s;
  if (n < 2) {  // one vertex: no repulsion and no neighbour
    BL_CUDA(ctx, cudaMemsetAsync(s.rep, 0, sizeof(float2) * std::max(n, 1), ctx->stream));
    if (batch > 0) BL_CUDA(ctx, cudaMemsetAsync(s.f0, 0, sizeof(float4) * std::max(n, 1), ctx->stream));
    return 0;
  }
  TraverseArgs a;
  a.n = n;
  a.nodes = s.nodes;
  a.nodes_c64 = s.nodes_c64;
  a.nodes_lvl = s.nodes_lvl;
  a.frame = s.frame;
  a.spos = s.spos;
  a.perm = s.perm;
  a.rep = s.rep;
  a.theta = theta;
  a.stats = want_stats ? s.stats : nullptr;
  a.st = s.status;
  a.f0 = batch > 0 ? s.f0 : nullptr;
  if (want_stats) BL_CUDA(ctx, cudaMemsetAsync(s.stats, 0, 2 * sizeof(unsigned long long), ctx->stream));
  bl_time_begin(ctx, "traverse_kernel");
  if (want_stats) traverse_kernel<true><<<nblk(n, kTravThreads), kTravThreads, 0, ctx->stream>>>(a);
  else traverse_kernel<false><<<nblk(n, kTravThreads), kTravThreads, 0, ctx->stream>>>(a);
  bl_time_end(ctx, "traverse_kernel");
  ctx->launches++;
  BL_CUDA(ctx, cudaGetLastError());
  return 0;
}

int bh_iteration(bl_ctx *ctx, int batch, double theta, double step, bool want_energy,
                 double *energy_out) {
  if (int rc = ensure_bh_scratch(ctx)) return rc;
  const LevelSchedule *ls = level_schedule(ctx, batch);
  if (!ls) return -2;
  float2 *pold = ctx->pos, *pnew = ctx->s.pos_alt;
  if (int rc = bh_build(ctx, pold, theta, batch)) return rc;  // with the unmoved neighbours' attraction
  if (int rc = bh_traverse(ctx, theta, false, batch)) return rc;
  SweepArgs a;
  a.order = ls->order;
  a.group_start = ls->d_groups;
  a.early_off = ls->early_off;
  a.early_col = ls->early_col;
  a.groups = ls->groups;
  a.f0 = ctx->s.f0;
  a.f0out = ctx->s.f0;
  a.pold = pold;
  a.pnew = pnew;
  a.write_out = want_energy ? 1 : 0;
  a.W = (float)ctx->weight;
  a.step = (float)step;
  a.st = ctx->s.status;
  int occ = 0;
  BL_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, sweep_kernel, kSweepThreads, 0));
  if (occ < 1) return bl_fail(ctx, -5, "sweep kernel cannot be resident");
  const int sweep_grid = ctx->num_sms * std::min(occ, 2);
  // every new position starts as "not written": the sweep's waits read it
  BL_CUDA(ctx, cudaMemsetAsync(pnew, 0xff, (size_t)ctx->g.n * sizeof(float2), ctx->stream));
  void *args[] = {&a};
  bl_time_begin(ctx, "sweep_kernel");
  BL_CUDA(ctx, cudaLaunchCooperativeKernel((const void *)sweep_kernel, dim3(sweep_grid), dim3(kSweepThreads),
                                           args, 0, ctx->stream));
  bl_time_end(ctx, "sweep_kernel");
  ctx->launches++;
  std::swap(ctx->pos, ctx->s.pos_alt);
  if (want_energy) {
    bh_forces_kernel<<<nblk(ctx->g.n, 256), 256, 0, ctx->stream>>>(ctx->s.f0, ctx->g.n, ctx->force, ctx->e);
    ctx->launches++;
    if (int rc = energy_reduce(ctx, energy_out)) return rc;
    // without a destination (a captured iteration) the energy stays in
    // s.energy for the caller to read after the replay
    return energy_out ? bl_check_status(ctx) : 0;
  }
  return 0;
}

// ---- CUDA-graph replay of the iteration ------------------------------------
// One Barnes-Hut iteration without the energy read-back is a fixed sequence
// of about 15 launches and memsets on fixed buffers; only the positions
// alternate between two buffers and STEP changes.  It is captured once per
// parity of the position buffers and replayed, STEP being set on the sweep's
// kernel node before each replay.
// Captured iterations: [variant][parity], variant 1 also writes the forces
// and |f|^2 and reduces the energy into s.energy; parity p reads the
// position buffer that is ctx->pos when (ctx->pos == pos0) == (p == 0).
// Each is captured the first time it is needed.
struct BhGraph {
  int batch = -1;
  double theta = 0.0;
  float2 *pos0 = nullptr;  // ctx->pos of parity 0
  cudaGraph_t graph[2][2] = {{nullptr, nullptr}, {nullptr, nullptr}};
  cudaGraphExec_t exec[2][2] = {{nullptr, nullptr}, {nullptr, nullptr}};
  cudaGraphNode_t sweep[2][2] = {{nullptr, nullptr}, {nullptr, nullptr}};
  SweepArgs args[2][2];
  cudaKernelNodeParams params[2][2];
  long long kernels[2][2] = {{0, 0}, {0, 0}};
};

void bh_graph_free(BhGraph *g) {
  if (!g) return;
  for (int v = 0; v < 2; v++)
    for (int p = 0; p < 2; p++) {
      if (g->exec[v][p]) cudaGraphExecDestroy(g->exec[v][p]);
      if (g->graph[v][p]) cudaGraphDestroy(g->graph[v][p]);
    }
  delete g;
}

namespace {

// Capture variant v of the iteration that reads ctx->pos (the parity the
// context is at).  Returns 0, or 1 when the iteration cannot be captured
// (nothing has run).
int bh_graph_capture(bl_ctx *ctx, BhGraph &G, int v, int p, int batch, double theta) {
  float2 *save_pos = ctx->pos, *save_alt = ctx->s.pos_alt;
  const std::string save_timed = ctx->timed_kernel;
  const long long save_launches = ctx->launches;
  ctx->timed_kernel.clear();  // no timing events inside the graph
  if (cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
    cudaGetLastError();
    ctx->timed_kernel = save_timed;
    return 1;
  }
  const int rc = bh_iteration(ctx, batch, theta, 1.0, v == 1, nullptr);
  cudaGraph_t graph = nullptr;
  const cudaError_t e = cudaStreamEndCapture(ctx->stream, &graph);
  ctx->pos = save_pos;
  ctx->s.pos_alt = save_alt;
  ctx->timed_kernel = save_timed;
  G.kernels[v][p] = ctx->launches - save_launches;
  ctx->launches = save_launches;
  if (rc || e != cudaSuccess || !graph) {
    if (graph) cudaGraphDestroy(graph);
    cudaGetLastError();
    return 1;
  }
  size_t count = 0;
  cudaGraphGetNodes(graph, nullptr, &count);
  std::vector<cudaGraphNode_t> nodes(count);
  cudaGraphGetNodes(graph, nodes.data(), &count);
  cudaGraphNode_t sweep = nullptr;
  for (cudaGraphNode_t nd : nodes) {
    cudaGraphNodeType t;
    if (cudaGraphNodeGetType(nd, &t) != cudaSuccess || t != cudaGraphNodeTypeKernel) continue;
    cudaKernelNodeParams kp;
    if (cudaGraphKernelNodeGetParams(nd, &kp) != cudaSuccess) continue;
    if (kp.func == (void *)sweep_kernel) {
      sweep = nd;
      G.params[v][p] = kp;
      G.args[v][p] = *static_cast<SweepArgs *>(kp.kernelParams[0]);
    }
  }
  cudaGraphExec_t exec = nullptr;
  if (!sweep || cudaGraphInstantiate(&exec, graph, 0) != cudaSuccess) {
    cudaGraphDestroy(graph);
    cudaGetLastError();
    return 1;
  }
  G.graph[v][p] = graph;
  G.exec[v][p] = exec;
  G.sweep[v][p] = sweep;
  return 0;
}

// The context's graphs for (batch, theta), dropped and started afresh when
// they or the position buffers changed.
BhGraph *bh_graph_for(bl_ctx *ctx, int batch, double theta) {
  BhGraph *G = ctx->bh_graph;
  const bool fresh = !G || G->batch != batch || G->theta != theta ||
                     (G->pos0 != ctx->pos && G->pos0 != ctx->s.pos_alt);
  if (fresh) {
    bh_graph_free(G);
    G = ctx->bh_graph = new BhGraph();
    G->batch = batch;
    G->theta = theta;
    G->pos0 = ctx->pos;
  }
  return G;
}

// One replay of variant v with STEP `step`; 1 when it cannot be captured.
int bh_graph_replay(bl_ctx *ctx, BhGraph *G, int v, int batch, double theta, double step) {
  const int p = (ctx->pos == G->pos0) ? 0 : 1;
  if (!G->exec[v][p] && bh_graph_capture(ctx, *G, v, p, batch, theta)) return 1;
  G->args[v][p].step = (float)step;
  void *kargs[] = {&G->args[v][p]};
  cudaKernelNodeParams kp = G->params[v][p];
  kp.kernelParams = kargs;
  BL_CUDA(ctx, cudaGraphExecKernelNodeSetParams(G->exec[v][p], G->sweep[v][p], &kp));
  BL_CUDA(ctx, cudaGraphLaunch(G->exec[v][p], ctx->stream));
  ctx->launches += G->kernels[v][p];
  std::swap(ctx->pos, ctx->s.pos_alt);
  return 0;
}

}  // namespace

// `count` iterations without energy read-back by graph replay, STEP from
// *step (multiplied by 0.999 after each).  Returns 0, an error code, or 1
// when the iteration cannot be captured (nothing has run; launch directly).
int bh_graph_iterations(bl_ctx *ctx, int batch, double theta, double *step, int count) {
  if (count <= 0) return 0;
  if (int rc = ensure_bh_scratch(ctx)) return rc;
  if (!level_schedule(ctx, batch)) return -2;
  BhGraph *G = bh_graph_for(ctx, batch, theta);
  for (int k = 0; k < count; k++) {
    const int r = bh_graph_replay(ctx, G, 0, batch, theta, *step);
    if (r) return k == 0 ? r : -5;  // a parity that cannot be captured after one that could: not expected
    *step *= 0.999;
  }
  return 0;
}

// One iteration with its energy (as bh_iteration with want_energy) by graph
// replay.  Returns 0, an error code, or 1 when it cannot be captured.
int bh_graph_energy_iteration(bl_ctx *ctx, int batch, double theta, double step, double *energy_out) {
  if (int rc = ensure_bh_scratch(ctx)) return rc;
  if (!level_schedule(ctx, batch)) return -2;
  BhGraph *G = bh_graph_for(ctx, batch, theta);
  if (int r = bh_graph_replay(ctx, G, 1, batch, theta, step)) return r;
  // the energy and the device status in one wait
  DevStatus st;
  BL_CUDA(ctx, cudaMemcpyAsync(energy_out, ctx->s.energy, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  BL_CUDA(ctx, cudaMemcpyAsync(&st, ctx->s.status, sizeof(DevStatus), cudaMemcpyDeviceToHost, ctx->stream));
  BL_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return st.code == 0u ? 0 : bl_check_status(ctx);
}

// `iterations` Barnes-Hut iterations from STEP *step (times 0.999 after
// each); the last one's energy into *energy when it is not null.  In graph
// mode the iterations replay captured graphs (the last one the variant that
// reduces the energy); an iteration that cannot be captured is launched
// directly.
int bh_run(bl_ctx *ctx, int iterations, int batch, double theta, double *step, double *energy) {
  if (batch < 1) return bl_fail(ctx, -1, "batch must be >= 1");  // BL_ERR_ARG
  int it = 0;
  const int replay = energy ? iterations - 1 : iterations;
  if (ctx->graph_mode && replay > 0) {
    const int r = bh_graph_iterations(ctx, batch, theta, step, replay);
    if (r < 0) return r;
    if (r == 0) it = replay;
  }
  for (; it < iterations; it++) {
    const bool last = energy && it == iterations - 1;
    int r = 1;
    if (last && ctx->graph_mode) {
      r = bh_graph_energy_iteration(ctx, batch, theta, *step, energy);
      if (r < 0) return r;
    }
    if (r == 1)
      if (int rc = bh_iteration(ctx, batch, theta, *step, last, last ? energy : nullptr)) return rc;
    *step = *step * 0.999;
  }
  return 0;
}

int bh_canonical_tree(bl_ctx *ctx, int cap, int *lo, int *hi, int *depth, int *nchild,
                      double *centroid) {
  const int n = ctx->g.n;
  if (n < 2) return 0;
  if (int rc = ensure_bh_scratch(ctx)) return rc;
  if (n < 2) return 0;
  if (int rc = bh_build(ctx, ctx->pos, 1.2)) return rc;  // (theta enters only the records)
  // copy the binary tree back and emit quad nodes in pre-order (host walk)
  std::vector<int2> range(n - 1);
  std::vector<int4> node(2 * (size_t)(n - 1));  // as radix_tree_kernel packs them
  std::vector<int> dlt(n - 1);
  std::vector<double2> qcen(n - 1);
  cudaStream_t st = ctx->stream;
  BL_CUDA(ctx, cudaMemcpyAsync(node.data(), ctx->s.bnode, node.size() * sizeof(int4), cudaMemcpyDeviceToHost, st));
  BL_CUDA(ctx, cudaMemcpyAsync(range.data(), ctx->s.brange, (n - 1) * sizeof(int2), cudaMemcpyDeviceToHost, st));
  BL_CUDA(ctx, cudaMemcpyAsync(dlt.data(), ctx->s.bdelta, (n - 1) * sizeof(int), cudaMemcpyDeviceToHost, st));
  BL_CUDA(ctx, cudaMemcpyAsync(qcen.data(), ctx->s.qcen, (n - 1) * sizeof(double2), cudaMemcpyDeviceToHost, st));
  BL_CUDA(ctx, cudaStreamSynchronize(st));
  if (int rc = bl_check_status(ctx)) return rc;
  auto left = [&](int v) { return node[2 * (size_t)v].w; };
  auto right = [&](int v) { return node[2 * (size_t)v + 1].x; };
  auto sub = [&](int v) {
    if (v <= 0) return false;
    const int p = dlt[v], pp = dlt[node[2 * (size_t)v + 1].y];
    if (p >= 64) return pp >= 64;
    return (p & 1) && pp == p - 1;
  };
  int count = 0;
  std::vector<int> stack{0};
  while (!stack.empty()) {
    const int v = stack.back();
    stack.pop_back();
    std::vector<int> kids;
    if (dlt[v] >= 64) {
      kids.clear();
    } else {
      const int sides[2] = {left(v), right(v)};
      for (int c : sides) {
        if (c >= 0 && sub(c)) {
          kids.push_back(left(c));
          kids.push_back(right(c));
        } else {
          kids.push_back(c);
        }
      }
    }
    if (count < cap) {
      lo[count] = range[v].x;
      hi[count] = range[v].y + 1;
      depth[count] = dlt[v] >= 64 ? 32 : dlt[v] / 2;
      nchild[count] = dlt[v] >= 64 ? (range[v].y - range[v].x + 1) : (int)kids.size();
      centroid[2 * count] = qcen[v].x;
      centroid[2 * count + 1] = qcen[v].y;
    }
    count++;
    for (int q = (int)kids.size() - 1; q >= 0; q--)
      if (kids[q] >= 0) stack.push_back(kids[q]);
  }
  return count;
}

// Dependency levels of the attraction sweep for batch size `batch`:
// level(i) = 0 without neighbours in earlier batches, else 1 + the largest
// level among them.  Cached per batch size.
const LevelSchedule *level_schedule(bl_ctx *ctx, int batch) {
  for (auto &ls : ctx->schedules)
    if (ls.batch == batch) return &ls;
  const int n = ctx->g.n;
  const std::vector<int> &rp = ctx->h_rowptr, &ci = ctx->h_colids;
  std::vector<int> lev(n, 0);
  int maxl = 0;
  for (int i = 0; i < n; i++) {
    const int bi = i / batch;
    int l = -1;
    for (int e = rp[i]; e < rp[i + 1]; e++) {
      const int j = ci[e];
      if (j / batch < bi) l = std::max(l, lev[j]);
    }
    lev[i] = l + 1;
    maxl = std::max(maxl, l + 1);
  }
  LevelSchedule ls;
  ls.batch = batch;
  ls.levels = n > 0 ? maxl + 1 : 0;
  ls.offsets.assign(ls.levels + 1, 0);
  for (int i = 0; i < n; i++) ls.offsets[lev[i] + 1]++;
  for (int l = 0; l < ls.levels; l++) ls.offsets[l + 1] += ls.offsets[l];
  std::vector<int> start;  // the sweep's groups: up to 32 slots of one level
  for (int l = 0; l < ls.levels; l++)
    for (int t = ls.offsets[l]; t < ls.offsets[l + 1]; t += 32) start.push_back(t);
  ls.groups = (int)start.size();
  start.push_back(n);
  std::vector<int> order(std::max(n, 1));
  std::vector<int> fill(ls.offsets.begin(), ls.offsets.end() - 1);
  for (int i = 0; i < n; i++) order[fill[lev[i]]++] = i;
  if (cudaMalloc(&ls.order, order.size() * sizeof(int)) != cudaSuccess ||
      cudaMalloc(&ls.d_groups, start.size() * sizeof(int)) != cudaSuccess) {
    bl_fail(ctx, -2, "cudaMalloc level schedule");
    return nullptr;
  }
  if (cudaMemcpy(ls.d_groups, start.data(), start.size() * sizeof(int), cudaMemcpyHostToDevice) != cudaSuccess) {
    bl_fail(ctx, -2, "cudaMemcpy level schedule");
    return nullptr;
  }
  if (cudaMemcpy(ls.order, order.data(), order.size() * sizeof(int), cudaMemcpyHostToDevice) != cudaSuccess) {
    bl_fail(ctx, -2, "cudaMemcpy level schedule");
    return nullptr;
  }
  // neighbours in earlier batches, per level-order slot, in CSR order
  std::vector<int> eoff(std::max(n, 1) + 1, 0), ecol;
  ecol.reserve(ci.size() / 2 + 1);
  for (int t = 0; t < n; t++) {
    const int i = order[t];
    const int blo = (i / batch) * batch;
    for (int e = rp[i]; e < rp[i + 1]; e++)
      if (ci[e] < blo) ecol.push_back(ci[e]);
    eoff[t + 1] = (int)ecol.size();
  }
  if (ecol.empty()) ecol.push_back(0);
  if (cudaMalloc(&ls.early_off, eoff.size() * sizeof(int)) != cudaSuccess ||
      cudaMalloc(&ls.early_col, ecol.size() * sizeof(int)) != cudaSuccess ||
      cudaMemcpy(ls.early_off, eoff.data(), eoff.size() * sizeof(int), cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemcpy(ls.early_col, ecol.data(), ecol.size() * sizeof(int), cudaMemcpyHostToDevice) != cudaSuccess) {
    bl_fail(ctx, -2, "level schedule neighbour lists");
    return nullptr;
  }
  ctx->schedules.push_back(std::move(ls));
  return &ctx->schedules.back();
}

}  // namespace bl
