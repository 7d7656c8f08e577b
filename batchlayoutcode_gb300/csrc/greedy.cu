// greedy.cu -- algo 5, greedy approximation, first phase
// (approxForceDirectedAlgorithm, sample/algorithms.cpp:1085-1190).
//
// For the first (int)(0.8 * ITERATIONS) + 1 iterations the reference gives
// every vertex i the attraction W|d|d of its CSR neighbours and the
// repulsion -d/|d|^2 of the vertices a bounded depth-first walk reaches
// (:1126-1170): the stack starts with i's neighbours in CSR order; popping u
// scans u's row and every entry v outside {i} u N(i) repels, is pushed and
// spends one unit of a budget of 200; the walk ends after the row that spends
// the budget, or when the stack is empty.  Reached vertices are not marked,
// so a walk visits few distinct vertices many times (about 22 distinct among
// ~200 on the benchmark graphs).
//
// GB300 design.  The walk depends on the graph only, so it runs once per
// graph instead of once per vertex and iteration: walk_kernel (a warp per
// vertex, the stack in HBM, each popped row scanned 32 entries at a time,
// pushes kept in CSR order by a ballot) merges repeated sources in shared
// memory and stores each vertex's walk as (source, count) pairs, in a
// count pass and a fill pass around a prefix sum.  An iteration is then a
// sparse gather over a per-vertex term list (CSR entries, then walk pairs):
// greedy_iteration_kernel runs all first-phase iterations in one persistent
// launch without barriers.  A warp takes a vertex, a lane a term; a position
// word is its own ready flag, so a vertex waits only for the sources it reads
// (Gauss-Seidel across batches, Jacobi inside a batch) and vertices of many
// batches, and of two iterations, are in work at once.
//
// Summation order differs from the reference's (pairs instead of walk
// order, FP32 terms summed exactly in units of 2^-28 instead of in FP64):
// results agree within FP32 rounding.
#include <algorithm>
#include <cstring>
#include <numeric>
#include <vector>

#include "../../include/batchlayout_gb300.h"
#include "bl_device.cuh"

namespace bl {
namespace {

constexpr int kGreedyBudget = 200;  // countNodes (algorithms.cpp:1147)

// ---- walk construction ---------------------------------------------------------

constexpr int kWalkThreads = 256;
constexpr int kWalkWarps = kWalkThreads / 32;
constexpr int kUniq = 128;  // distinct sources merged per walk in shared memory

struct WalkArgs {
  int n;
  const int *rowptr, *colids;          // the CSR (push order)
  const int *srt_rowptr, *srt_colids;  // rows sorted (membership test)
  int *stack;
  long long stack_cap;                 // ints per warp
  long long *count;                    // count pass: pairs per vertex
  const long long *off;                // fill pass: first pair of each vertex
  int2 *pairs;
  DevStatus *st;
};

// v in N(i): binary search of the sorted row [m0, m1)
__device__ __forceinline__ bool row_contains(const int *srt, int m0, int m1, int v) {
  while (m0 < m1) {
    const int mid = (m0 + m1) >> 1;
    const int c = __ldg(&srt[mid]);
    if (c == v) return true;
    if (c < v) m0 = mid + 1;
    else m1 = mid;
  }
  return false;
}

template <bool kFill>
__global__ void __launch_bounds__(kWalkThreads) walk_kernel(WalkArgs a) {
  __shared__ int uv[kWalkWarps][kUniq];
  __shared__ int um[kWalkWarps][kUniq];
  if (!block_status_ok(a.st)) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long gw = (long long)blockIdx.x * kWalkWarps + warp;
  const long long nw = (long long)gridDim.x * kWalkWarps;
  int *stack = a.stack + gw * a.stack_cap;
  int *myv = uv[warp], *mym = um[warp];
  const unsigned lt = (1u << lane) - 1u;
  for (long long ii = gw; ii < a.n; ii += nw) {
    const int i = (int)ii;
    const int r0 = __ldg(&a.rowptr[i]), r1 = __ldg(&a.rowptr[i + 1]);
    const int m0 = __ldg(&a.srt_rowptr[i]), m1 = __ldg(&a.srt_rowptr[i + 1]);
    // the stack starts with N(i) in CSR order (:1130-1144); the capacity
    // covers deg(i) + 199 + max degree entries
    for (int k = lane; k < r1 - r0; k += 32) stack[k] = __ldg(&a.colids[r0 + k]);
    long long sp = r1 - r0;
    int nu = 0, budget = kGreedyBudget;
    long long nover = 0;  // pairs stored directly once the table is full
    const long long obase = kFill ? a.off[i] : 0;
    long long pops = 0;
    bool bad = false;
    __syncwarp();
    while (sp > 0) {
      // every pop either pushes (spending budget) or shrinks the stack, so
      // the walk ends after at most stack_cap pops; the check is a guard
      if (++pops > a.stack_cap + 1) {
        bad = true;
        break;
      }
      const int u = stack[sp - 1];
      sp--;
      const int u0 = __ldg(&a.rowptr[u]), u1 = __ldg(&a.rowptr[u + 1]);
      int pushed = 0;
      for (int e0 = u0; e0 < u1; e0 += 32) {
        const int e = e0 + lane;
        int v = -1;
        bool push = false;
        if (e < u1) {
          v = __ldg(&a.colids[e]);
          push = v != i && !row_contains(a.srt_colids, m0, m1, v);
        }
        unsigned mask = __ballot_sync(0xffffffffu, push);
        const long long at = sp + __popc(mask & lt);
        if (push) {
          if (at < a.stack_cap) stack[at] = v;
          else bad = true;
        }
        sp += __popc(mask);
        pushed += __popc(mask);
        // merge the pushed sources, in push order
        while (mask) {
          const int src = __ffs(mask) - 1;
          mask &= mask - 1u;
          const int cv = __shfl_sync(0xffffffffu, v, src);
          int found = -1;
          for (int q = lane; q < nu; q += 32)
            if (myv[q] == cv) found = q;
          const unsigned fm = __ballot_sync(0xffffffffu, found >= 0);
          if (fm) {
            if (lane == __ffs(fm) - 1) mym[found]++;
          } else if (nu < kUniq) {
            if (lane == 0) {
              myv[nu] = cv;
              mym[nu] = 1;
            }
            nu++;
          } else {
            if (kFill && lane == 0) a.pairs[obase + nover] = make_int2(cv, 1);
            nover++;
          }
          __syncwarp();
        }
      }
      if (__any_sync(0xffffffffu, bad)) break;
      __syncwarp();
      budget -= pushed;
      if (budget <= 0) break;  // :1167
    }
    if (__any_sync(0xffffffffu, bad)) {
      if (lane == 0) dev_record_error(a.st, DEV_BAD_INDEX);
      return;
    }
    if (!kFill) {
      if (lane == 0) a.count[i] = nover + nu;
    } else {
      for (int q = lane; q < nu; q += 32) a.pairs[obase + nover + q] = make_int2(myv[q], mym[q]);
    }
    __syncwarp();
  }
}

// ---- first-phase iterations ----------------------------------------------------

// Term list of a vertex i, at term_off[i] = rowptr[i] + walk_off[i]: its CSR
// entries as (neighbour, 0) -- attraction -- then its walk pairs as
// (source, count) -- count x repulsion.
__global__ void term_list_kernel(int n, const int *__restrict__ rowptr, const int *__restrict__ colids,
                                 const long long *__restrict__ walk_off, const int2 *__restrict__ walk_pairs,
                                 int2 *__restrict__ terms) {
  const int warp = (int)((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (warp >= n) return;
  const int i = warp;
  const int r0 = rowptr[i], r1 = rowptr[i + 1];
  const long long w0 = walk_off[i], w1 = walk_off[i + 1];
  const long long q0 = (long long)r0 + w0;
  for (int k = r0 + lane; k < r1; k += 32) terms[q0 + (k - r0)] = make_int2(colids[k], 0);
  const long long qa = q0 + (r1 - r0);
  for (long long k = w0 + lane; k < w1; k += 32) terms[qa + (k - w0)] = walk_pairs[k];
}

constexpr int kIterThreads = 896;
constexpr int kIterWarps = kIterThreads / 32;
constexpr int kPosBufs = 5;

// Fixed-point force sums (units of 2^-28, the minibatch sweep's format):
// exact, so they do not depend on the order of the terms.  A term or a lane's
// sum beyond +-2^34 is reported instead of wrapping.
constexpr float kFix = 268435456.0f;
constexpr double kFixInv = 1.0 / 268435456.0;
constexpr float kFixLimit = 17179869184.0f;

// Batches above some 7,200 (this many bytes a vertex within a block's shared
// memory) are refused.  Nothing here needs the bound; algo 5's second phase
// takes 4,096 at most, and a run it cannot end is better refused before the
// first phase has moved anything.
constexpr size_t kBatchBytes = 2 * sizeof(long long) + 2 * sizeof(float2);

// A position not yet written: both coordinates NaN, all bits set.
constexpr unsigned long long kNoPos = 0xffffffffffffffffull;

struct IterArgs {
  int n, batch, iterations, energy_last;
  float W;
  double step0, decay;
  const long long *term_off;  // per vertex
  const int2 *terms;
  float2 *buf;         // kPosBufs arrays of n positions: after m moves in array m % kPosBufs
  unsigned int *done;  // [4]: blocks whose warps have all left iteration k, in word k & 3
  double2 *force;
  double *e;
  DevStatus *st;
};

__device__ __forceinline__ unsigned long long ld_word(const float2 *p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void st_word(float2 *p, unsigned long long b) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(b) : "memory");
}

__device__ __forceinline__ float2 word_pos(unsigned long long b) {
  return make_float2(__uint_as_float((unsigned int)b), __uint_as_float((unsigned int)(b >> 32)));
}

__device__ __forceinline__ unsigned long long pos_word(float2 p) {
  return (unsigned long long)__float_as_uint(p.x) | ((unsigned long long)__float_as_uint(p.y) << 32);
}

// Array 0: the start; arrays 1 and 2: not written; no warp has left an
// iteration.  (Arrays 3 and 4 are cleared by iterations 0 and 1.)
__global__ void greedy_start_kernel(IterArgs a, const float2 *__restrict__ pos) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < 4) a.done[i] = 0u;
  if (i >= a.n) return;
  unsigned long long b = pos_word(pos[i]);
  if (b == kNoPos) b = 0x7fffffff7fffffffull;  // a NaN that is not the flag
  st_word(&a.buf[i], b);
  st_word(&a.buf[(size_t)a.n + i], kNoPos);
  st_word(&a.buf[2 * (size_t)a.n + i], kNoPos);
}

// The positions after the last move, unless the run ended in an error: then
// some were never written and the context keeps the start.
__global__ void greedy_finish_kernel(int n, const float2 *__restrict__ moved, float2 *__restrict__ pos,
                                     const DevStatus *st) {
  if (!block_status_ok(st)) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) pos[i] = moved[i];
}

// The sum over the warp of one signed 64-bit value a lane (|v| < 2^62), by
// three 27-bit limbs; false when it leaves 64 bits.
__device__ __forceinline__ bool warp_sum_ll(long long v, long long &sum) {
  const unsigned int lo = __reduce_add_sync(0xffffffffu, (unsigned int)v & 0x7ffffffu);
  const unsigned int mid = __reduce_add_sync(0xffffffffu, (unsigned int)(v >> 27) & 0x7ffffffu);
  const int hi = __reduce_add_sync(0xffffffffu, (int)(v >> 54));
  sum = ((long long)hi << 54) + ((long long)mid << 27) + (long long)lo;
  return hi > -500 && hi < 500;
}

// Whether a warp may go on waiting: false once `since` (0: the first call) is
// too long ago or another warp recorded an error; the same in every lane.
__device__ __forceinline__ bool keep_waiting(DevStatus *st, unsigned long long &since) {
  const unsigned long long t = dev_globaltimer();
  if (since == 0) since = t;
  bool quit = ld_volatile_u32(&st->code) != 0u;
  if (!quit && t - since > kBarrierTimeoutNs) {
    dev_record_error(st, DEV_TIMEOUT_SWEEP);
    quit = true;
  }
  return !__any_sync(0xffffffffu, quit);
}

// All iterations of the first phase in one cooperative launch.
//
// Task (it, i) moves vertex i in iteration it; warp w of W takes tasks w,
// w + W, ... in (it, i) order, warps numbered so that consecutive vertices
// land on different SMs.  A lane holds two terms at a time: it reads its
// sources' position words, of a vertex in an earlier batch after this
// iteration's move, of any other before it, and waits (bounded) for those not
// written yet.  Every word a task waits for is written by a task before it in
// the order and all blocks are resident, so the first unfinished task can
// always proceed.  The terms whose words are there are added first, so that
// only the latest source's term lies between its move and this one.  The lanes'
// fixed-point sums meet in warp reductions and the new position is one 8-byte
// store that later tasks see as ready.
// Positions after m moves live in array m % 5.  A task of iteration it clears
// its word of array (it + 3) % 5, whose old content (after it - 2 moves) only
// iterations it - 3 and it - 2 read: a warp enters iteration it when all warps
// have left it - 2, so at most two iterations are in work, and the words are
// clear before iteration it + 2 begins to read them.
// Bound by the dependency chain across the batches (73 links an iteration on
// the power-law graph below; a link is a load that sees the position, 600-700
// cycles, the term, the reductions and the store) and, with few links, by
// instruction issue.  One cluster of 16 blocks with a barrier a batch takes
// 2.6 us a batch whatever it depends on and leaves 136 SMs idle: nine
// iterations of 100,000 vertices 9,200 us, this way 1,070 (power law) and 530
// (geometric).  28 warps a block: 32 spill registers, 24 and 16 take 3 and
// 11 % longer.
__global__ void __launch_bounds__(kIterThreads, 1) greedy_iteration_kernel(IterArgs a) {
  __shared__ unsigned int left[4];
  if (threadIdx.x < 4) left[threadIdx.x] = 0u;
  if (!block_status_ok(a.st)) return;
  const int lane = threadIdx.x & 31;
  const int W = gridDim.x * kIterWarps, w = (int)(threadIdx.x >> 5) * (int)gridDim.x + (int)blockIdx.x;
  const int wrap = W / a.n, rest = W % a.n;  // from a task to the warp's next: iterations, vertices
  double step = a.step0;
  int entered = 0;  // the iteration the warp is in, its positions before and after the move
  const float2 *now = a.buf;
  float2 *next = a.buf + a.n;
  auto array_after = [&](float2 *p, int m) {  // m arrays on, cyclically
    return p + (p + m * (size_t)a.n >= a.buf + kPosBufs * (size_t)a.n ? m - kPosBufs : m) * (long long)a.n;
  };
  // Leaves iterations until `target` is the current one; false when a wait ran
  // out or another warp recorded an error.
  auto enter = [&](int target) {
    while (entered < target) {
      __syncwarp();
      bool ok = true;
      if (lane == 0) {
        __threadfence();
        // the block's last warp tells the others (a warp is at most two
        // iterations ahead: four words are enough)
        if (atomicAdd(&left[entered & 3], 1u) % kIterWarps == kIterWarps - 1) {
          __threadfence();
          atomicAdd(&a.done[entered & 3], 1u);
        }
      }
      entered++;
      step = step * a.decay;
      now = next;
      next = array_after(next, 1);
      if (entered >= 2 && entered < a.iterations) {
        if (lane == 0) {
          const int k = entered - 2;
          const unsigned int want = gridDim.x * (unsigned int)(k / 4 + 1);
          const unsigned long long t0 = dev_globaltimer();
          for (unsigned int polls = 1; (int)(ld_acquire_gpu(&a.done[k & 3]) - want) < 0; polls++) {
            __nanosleep(100);
            if ((polls & 63u) != 0u) continue;
            if (ld_volatile_u32(&a.st->code) != 0u) ok = false;
            else if (dev_globaltimer() - t0 > kBarrierTimeoutNs) {
              dev_record_error(a.st, DEV_TIMEOUT_SWEEP);
              ok = false;
            }
            if (!ok) break;
          }
        }
        // the other lanes' position loads come after lane 0's acquire (a shuffle
        // orders no memory)
        __syncwarp();
        if (!__shfl_sync(0xffffffffu, ok ? 1 : 0, 0)) return false;
      }
    }
    return true;
  };
  int it = w / a.n, i = w % a.n;
  int off = i % a.batch;  // i's place in its batch
  const int rest_off = rest % a.batch;
  // the graph's part of the tasks ahead: offsets two tasks, terms one task
  int inext = i + rest;
  if (inext >= a.n) inext -= a.n;
  struct Terms {
    const int2 *at;
    int count;
  };
  auto terms_of = [&](int v) {
    const long long q = __ldg(&a.term_off[v]);
    return Terms{a.terms + q, (int)(__ldg(&a.term_off[v + 1]) - q)};
  };
  auto term = [&](const Terms &t, int k) { return k < t.count ? __ldg(&t.at[k]) : make_int2(-1, 0); };
  Terms cur = terms_of(i), coming = terms_of(inext);
  int2 t0 = term(cur, lane), t1 = term(cur, 32 + lane);
  while (it < a.iterations) {
    if (!enter(it)) return;
    const int batch_lo = i - off;
    // the words of this task, then the graph's part of the tasks ahead
    auto source = [&](int j) { return (j < batch_lo ? next : now) + j; };
    unsigned long long bi = ld_word(&now[i]);
    unsigned long long b0 = t0.x >= 0 ? ld_word(source(t0.x)) : 0ull;
    unsigned long long b1 = t1.x >= 0 ? ld_word(source(t1.x)) : 0ull;
    int iahead = inext + rest;
    if (iahead >= a.n) iahead -= a.n;
    const Terms ahead = terms_of(iahead);
    const int2 u0 = term(coming, lane), u1 = term(coming, 32 + lane);
    // polls until no lane misses its word; false when that takes too long
    auto wait = [&](unsigned long long &b, const float2 *at) {
      unsigned long long since = 0;
      for (unsigned int polls = 1; __any_sync(0xffffffffu, b == kNoPos); polls++) {
        if (b == kNoPos) b = ld_word(at);
        if ((polls & 255u) == 0u && !keep_waiting(a.st, since)) return false;
      }
      return true;
    };
    if (!wait(bi, &now[i])) return;  // its own position before this iteration
    const float2 pi = word_pos(bi);
    long long ax = 0, ay = 0;
    unsigned int wide = 0u;
    auto add = [&](int count, unsigned long long b) {
      const float2 pj = word_pos(b);
      float fx = 0.f, fy = 0.f;
      if (count == 0) {
        attract_pair(MODEL_FR, a.W, pj.x, pj.y, pi.x, pi.y, fx, fy);
      } else {
        rep_pair(pj.x, pj.y, pi.x, pi.y, fx, fy);
        fx *= (float)count;
        fy *= (float)count;
      }
      if (!(fmaxf(fabsf(fx), fabsf(fy)) < kFixLimit && fx == fx && fy == fy)) wide = 0x80000000u;
      ax += __float2ll_rn(fx * kFix);
      ay += __float2ll_rn(fy * kFix);
      // the sign of `wide` stays set once a sum leaves 63 bits (|sum| < 2^62
      // before and |term| <= 2^62 do not wrap)
      const unsigned int hx = (unsigned int)(ax >> 32), hy = (unsigned int)(ay >> 32);
      wide |= (hx ^ (hx << 1)) | (hy ^ (hy << 1));
    };
    // the terms whose words are there, in any order (the sums are exact); the
    // others' places are noted: bit k for the lane's k-th term
    unsigned long long pend = 0ull;
    for (int k = 0; 64ll * k < cur.count; k++) {
      const int q = 64 * (k + 1) + lane;
      const int2 v0 = term(cur, q), v1 = term(cur, q + 32);
      if (k >= 32) {  // no bits left: wait here
        if (!wait(b0, source(max(t0.x, 0))) || !wait(b1, source(max(t1.x, 0)))) return;
      }
      if (t0.x >= 0) {
        if (b0 != kNoPos) add(t0.y, b0);
        else pend |= 1ull << (2 * k);
      }
      if (t1.x >= 0) {
        if (b1 != kNoPos) add(t1.y, b1);
        else pend |= 2ull << (2 * k);
      }
      t0 = v0;
      t1 = v1;
      b0 = t0.x >= 0 ? ld_word(source(t0.x)) : 0ull;
      b1 = t1.x >= 0 ? ld_word(source(t1.x)) : 0ull;
    }
    // the rest as they come, each lane its first one
    if (__any_sync(0xffffffffu, pend != 0ull)) {
      auto first = [&]() {
        return pend ? __ldg(&cur.at[32 * (__ffsll((long long)pend) - 1) + lane]) : make_int2(-1, 0);
      };
      int2 tm = first();
      unsigned long long since = 0;
      for (unsigned int polls = 1; __any_sync(0xffffffffu, tm.x >= 0); polls++) {
        const unsigned long long b = tm.x >= 0 ? ld_word(source(tm.x)) : kNoPos;
        if (b != kNoPos) {
          add(tm.y, b);
          pend &= pend - 1ull;
          tm = first();
        }
        if ((polls & 255u) == 0u && !keep_waiting(a.st, since)) return;
      }
    }
    long long sx, sy;
    const bool fits = warp_sum_ll(ax, sx) & warp_sum_ll(ay, sy);
    if (!__all_sync(0xffffffffu, (int)wide >= 0 && fits)) {
      if (lane == 0) dev_record_error(a.st, DEV_FORCE_RANGE);
      return;
    }
    // the move (:1171-1177), the same in every lane
    const float fx = __ll2float_rn(sx) * (float)kFixInv, fy = __ll2float_rn(sy) * (float)kFixInv;
    const float stepf = (float)step;
    const float m2 = fmaf(fx, fx, fy * fy);
    float2 np = pi;
    if (m2 >= 1.17549435e-38f && m2 <= 3.0e38f) {
      const float rm = rsqrt_approx(m2);
      np.x = fmaf(stepf, fx * rm, np.x);
      np.y = fmaf(stepf, fy * rm, np.y);
    } else {
      np = unit_step(pi, (double)sx * kFixInv, (double)sy * kFixInv, stepf);
    }
    if (lane == 0) {
      unsigned long long b = pos_word(np);
      if (b == kNoPos) b = 0x7fffffff7fffffffull;
      st_word(&next[i], b);
      st_word(&array_after(next, 2)[i], kNoPos);
      if (it == a.iterations - 1) {
        const double dfx = (double)sx * kFixInv, dfy = (double)sy * kFixInv;
        a.force[i] = make_double2(dfx, dfy);
        if (a.energy_last) a.e[i] = dfx * dfx + dfy * dfy;
      }
    }
    off += rest_off;
    if (off >= a.batch) off -= a.batch;
    it += wrap;
    if (inext < i) {  // past the last vertex
      it++;
      off = inext % a.batch;
    }
    i = inext;
    inext = iahead;
    cur = coming;
    coming = ahead;
    t0 = u0;
    t1 = u1;
  }
  enter(a.iterations);
}

}  // namespace

int ensure_sorted_csr(bl_ctx *ctx) {
  if (ctx->g.max_degree >= 0) return 0;
  const int n = ctx->g.n;
  const std::vector<int> &rp = ctx->h_rowptr, &ci = ctx->h_colids;
  bool sorted = true;
  int maxd = 0;
  for (int i = 0; i < n; i++) {
    maxd = std::max(maxd, rp[i + 1] - rp[i]);
    for (int k = rp[i] + 1; k < rp[i + 1] && sorted; k++)
      if (ci[k] < ci[k - 1]) sorted = false;
  }
  if (sorted) {
    ctx->g.srt_rowptr = ctx->g.rowptr;
    ctx->g.srt_colids = ctx->g.colids;
  } else {
    std::vector<int> sc(ci);
    for (int i = 0; i < n; i++) std::sort(sc.begin() + rp[i], sc.begin() + rp[i + 1]);
    BL_CUDA(ctx, cudaMalloc(&ctx->g.srt_rowptr, (size_t)(n + 1) * sizeof(int)));
    BL_CUDA(ctx, cudaMalloc(&ctx->g.srt_colids, std::max<size_t>(sc.size(), 1) * sizeof(int)));
    BL_CUDA(ctx, cudaMemcpy(ctx->g.srt_rowptr, rp.data(), (size_t)(n + 1) * sizeof(int), cudaMemcpyHostToDevice));
    if (!sc.empty())
      BL_CUDA(ctx, cudaMemcpy(ctx->g.srt_colids, sc.data(), sc.size() * sizeof(int), cudaMemcpyHostToDevice));
  }
  ctx->g.max_degree = maxd;
  return 0;
}

int greedy_walks_build(bl_ctx *ctx) {
  if (ctx->s.walk_total >= 0) return 0;
  if (int rc = ensure_sorted_csr(ctx)) return rc;
  const int n = ctx->g.n;
  // stack bound: deg(i) + (199 + the degree of the row that spends the budget)
  const long long cap = 2LL * ctx->g.max_degree + 256;
  long long blocks = std::min<long long>((n + kWalkWarps - 1) / kWalkWarps, (long long)ctx->num_sms * 8);
  const long long max_warps = std::max<long long>(kWalkWarps, (512LL << 20) / (cap * (long long)sizeof(int)));
  blocks = std::max<long long>(1, std::min(blocks, max_warps / kWalkWarps));
  int *stack = nullptr;
  long long *count = nullptr;
  BL_CUDA(ctx, cudaMalloc(&stack, (size_t)(blocks * kWalkWarps * cap) * sizeof(int)));
  cudaError_t e = cudaMalloc(&count, (size_t)n * sizeof(long long));
  if (e != cudaSuccess) {
    cudaFree(stack);
    return bl_cuda_fail(ctx, e, "cudaMalloc");
  }
  auto cleanup = [&]() {
    cudaFree(stack);
    cudaFree(count);
  };
  WalkArgs a;
  a.n = n;
  a.rowptr = ctx->g.rowptr;
  a.colids = ctx->g.colids;
  a.srt_rowptr = ctx->g.srt_rowptr;
  a.srt_colids = ctx->g.srt_colids;
  a.stack = stack;
  a.stack_cap = cap;
  a.count = count;
  a.off = nullptr;
  a.pairs = nullptr;
  a.st = ctx->s.status;
  bl_time_begin(ctx, "walk_kernel");
  walk_kernel<false><<<(unsigned)blocks, kWalkThreads, 0, ctx->stream>>>(a);
  bl_time_end(ctx, "walk_kernel");
  ctx->launches++;
  std::vector<long long> off(n + 1, 0);
  e = cudaMemcpyAsync(off.data() + 1, count, (size_t)n * sizeof(long long), cudaMemcpyDeviceToHost, ctx->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
  if (e != cudaSuccess) {
    cleanup();
    return bl_cuda_fail(ctx, e, "walk count");
  }
  if (int rc = bl_check_status(ctx)) {
    cleanup();
    return rc;
  }
  std::partial_sum(off.begin(), off.end(), off.begin());
  const long long total = off[n];
  if (!ctx->s.walk_off) {
    e = cudaMalloc(&ctx->s.walk_off, (size_t)(n + 1) * sizeof(long long));
    if (e != cudaSuccess) {
      cleanup();
      return bl_cuda_fail(ctx, e, "cudaMalloc");
    }
  }
  if (ctx->s.walk_pairs) cudaFree(ctx->s.walk_pairs);  // left by a failed build
  ctx->s.walk_pairs = nullptr;
  e = cudaMalloc(&ctx->s.walk_pairs, (size_t)std::max<long long>(total, 1) * sizeof(int2));
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(ctx->s.walk_off, off.data(), (size_t)(n + 1) * sizeof(long long), cudaMemcpyHostToDevice,
                        ctx->stream);
  if (e != cudaSuccess) {
    cleanup();
    return bl_cuda_fail(ctx, e, "walk pairs");
  }
  a.count = nullptr;
  a.off = ctx->s.walk_off;
  a.pairs = ctx->s.walk_pairs;
  bl_time_begin(ctx, "walk_kernel");
  walk_kernel<true><<<(unsigned)blocks, kWalkThreads, 0, ctx->stream>>>(a);
  bl_time_end(ctx, "walk_kernel");
  ctx->launches++;
  e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
  cleanup();
  if (e != cudaSuccess) return bl_cuda_fail(ctx, e, "walk fill");
  if (int rc = bl_check_status(ctx)) return rc;
  ctx->s.walk_total = total;
  return 0;
}

int greedy_terms_build(bl_ctx *ctx) {
  if (ctx->s.terms) return 0;
  if (int rc = greedy_walks_build(ctx)) return rc;
  const int n = ctx->g.n;
  const long long total = ctx->g.nnz + ctx->s.walk_total;
  // term offsets = CSR offsets + walk offsets
  std::vector<long long> woff(n + 1);
  BL_CUDA(ctx, cudaMemcpy(woff.data(), ctx->s.walk_off, (size_t)(n + 1) * sizeof(long long), cudaMemcpyDeviceToHost));
  for (int i = 0; i <= n; i++) woff[i] += ctx->h_rowptr[i];
  BL_CUDA(ctx, cudaMalloc(&ctx->s.term_off, (size_t)(n + 1) * sizeof(long long)));
  BL_CUDA(ctx, cudaMemcpy(ctx->s.term_off, woff.data(), (size_t)(n + 1) * sizeof(long long), cudaMemcpyHostToDevice));
  BL_CUDA(ctx, cudaMalloc(&ctx->s.terms, (size_t)std::max<long long>(total, 1) * sizeof(int2)));
  const long long threads = 32LL * n;
  term_list_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, ctx->stream>>>(
      n, ctx->g.rowptr, ctx->g.colids, ctx->s.walk_off, ctx->s.walk_pairs, ctx->s.terms);
  ctx->launches++;
  BL_CUDA(ctx, cudaGetLastError());
  return 0;
}

int greedy_walk_run(bl_ctx *ctx, int batch, int iterations, double step0, double decay, bool want_energy,
                    double *energy_out) {
  const int n = ctx->g.n;
  if (batch < 1) return bl_fail(ctx, BL_ERR_ARG, "batch must be >= 1");
  if (iterations <= 0) return 0;
  if (int rc = greedy_terms_build(ctx)) return rc;
  if (int rc = bl_check_status(ctx)) return rc;
  batch = std::min(batch, n);
  int smem_optin = 0;
  cudaDeviceGetAttribute(&smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device);
  if (batch * kBatchBytes + 1024 > (size_t)smem_optin) return bl_fail(ctx, BL_ERR_TOO_LARGE, "algo 5: batch too large");
  if (!ctx->s.greedy_pos) {
    BL_CUDA(ctx, cudaMalloc(&ctx->s.greedy_pos, (size_t)kPosBufs * std::max(n, 2) * sizeof(float2) + 4 * sizeof(int)));
  }
  IterArgs a;
  a.n = n;
  a.batch = batch;
  a.iterations = iterations;
  a.energy_last = want_energy ? 1 : 0;
  a.W = (float)ctx->weight;
  a.step0 = step0;
  a.decay = decay;
  a.term_off = ctx->s.term_off;
  a.terms = ctx->s.terms;
  a.buf = ctx->s.greedy_pos;
  a.done = reinterpret_cast<unsigned int *>(a.buf + (size_t)kPosBufs * std::max(n, 2));
  a.force = ctx->force;
  a.e = ctx->e;
  a.st = ctx->s.status;
  int occ = 0;
  BL_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, greedy_iteration_kernel, kIterThreads, 0));
  if (occ < 1) return bl_fail(ctx, BL_ERR_TOO_LARGE, "algo 5: the iteration kernel cannot be resident");
  const int grid = std::min(ctx->num_sms, (n + kIterWarps - 1) / kIterWarps);  // no more warps than vertices need
  greedy_start_kernel<<<(std::max(n, 4) + 255) / 256, 256, 0, ctx->stream>>>(a, ctx->pos);
  ctx->launches++;
  bl_time_begin(ctx, "greedy_iteration_kernel");
  void *args[] = {&a};
  BL_CUDA(ctx, cudaLaunchCooperativeKernel((const void *)greedy_iteration_kernel, dim3(grid), dim3(kIterThreads), args, 0,
                                           ctx->stream));
  bl_time_end(ctx, "greedy_iteration_kernel");
  ctx->launches++;
  greedy_finish_kernel<<<(n + 255) / 256, 256, 0, ctx->stream>>>(n, a.buf + (size_t)(iterations % kPosBufs) * n,
                                                                 ctx->pos, ctx->s.status);
  ctx->launches++;
  BL_CUDA(ctx, cudaGetLastError());
  if (want_energy) {
    if (int rc = energy_reduce(ctx, energy_out)) return rc;
  } else {
    BL_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  }
  return bl_check_status(ctx);
}

}  // namespace bl

extern "C" int bl_greedy_walks(bl_ctx *ctx, long long *offsets, int *sources, int *counts, long long cap,
                               long long *total) try {
  if (!ctx || !offsets || !total || cap < 0 || (cap > 0 && (!sources || !counts))) return BL_ERR_ARG;
  BL_CUDA(ctx, cudaSetDevice(ctx->device));
  if (int rc = bl::greedy_walks_build(ctx)) return rc;
  const int n = ctx->g.n;
  *total = ctx->s.walk_total;
  BL_CUDA(ctx, cudaMemcpy(offsets, ctx->s.walk_off, (size_t)(n + 1) * sizeof(long long), cudaMemcpyDeviceToHost));
  const long long m = std::min(cap, ctx->s.walk_total);
  if (m > 0) {
    std::vector<int2> p((size_t)m);
    BL_CUDA(ctx, cudaMemcpy(p.data(), ctx->s.walk_pairs, (size_t)m * sizeof(int2), cudaMemcpyDeviceToHost));
    for (long long k = 0; k < m; k++) {
      sources[k] = p[k].x;
      counts[k] = p[k].y;
    }
  }
  return BL_OK;
} catch (...) {
  return bl_host_exception(ctx);
}
