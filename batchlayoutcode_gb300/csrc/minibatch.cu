// minibatch.cu -- all-pairs stochastic minibatch update (algo 2 / 3 / 8, and
// algo 7 and the second phase of algo 5).
//
// Reference: sample/algorithms.cpp:739-783 (FR), :894-936 (LinLog),
// :967-1009 (FA), :536-590 (algo 7: attraction over every CSR neighbour, the
// neighbours' repulsion removed), :1112-1125 (algo 5 after 80 % of the
// iterations: repulsion -d/|d| instead of -d/|d|^2).  Vertices are processed in consecutive batches of `batch`
// ids; every force of a batch uses the positions at the start of that batch
// (Jacobi inside a batch) and the batch then moves by STEP * f/|f| before the
// next batch starts (Gauss-Seidel across batches).  f_i is attraction over
// the neighbours matched by the sorted-CSR cursor (kindex, :758-762) plus
// repulsion -d/|d|^2 over every other vertex with |d| > 0.
//
// GB300 design: one persistent cooperative kernel, one 1,024-thread block per
// SM, runs every iteration and batch without a grid barrier.  Batches are
// numbered through the run (q = 0, 1, ...).  The sequential chain (a batch's
// forces need the batch before it moved) only touches the pairs with the last
// few batches, so two kinds of blocks share the work:
//
// * Sweepers own a contiguous slice of the source vertices in shared memory
//   and add up, for batch q, the repulsion of their sources except those in
//   the `lag` (two) batches before q, which may still be moving: one FP32
//   partial force per target, stored to global memory.  They need only batch
//   q - lag - 1 to have moved, so they run up to `lag` batches ahead of the
//   chain.  Two 512-thread teams take alternate batches, so one team's waits,
//   partial sums and stores overlap the other's sweep.
// * Movers (the first M blocks) each move a fixed share of every batch.
//   Three teams work side by side: P adds up the sweepers' partials, N the
//   neighbour corrections (remove the repulsion, add the model's attraction
//   -- the decomposition the reference's own algo 7 uses, :553-579; of long rows
//   with P), and the critical team the pairs with the last `lag` batches; it receives the batch
//   before as 8-byte words {coordinate, batch tag} the other movers write (one
//   L2 hop, no barrier), moves its share and publishes it the same way.
//
// So a batch costs max(sweep, chain); with a grid barrier a batch it costs their
// sum and the barrier.  Bound of the sweep: the MUFU reciprocal, 16 a clock and
// SM; its loop runs at 14.9 pairs a clock.  Bound of the chain: instruction
// latency of about 400 dependent instructions and one L2 round trip.  us a
// batch, with a barrier / so: 100,000 vertices and batch 256 10.8 (6.9 of them
// the sweep) / 6.8; 4,096 vertices 5.2 / 3.0; 20,000 and batch 200 5.4 / 3.5;
// 31,000 and batch 512 12.3 / 5.8.  Every sum has a fixed order, so results are
// deterministic.
//
// Algorithmic work: 10 flops per ordered pair (2 sub, 3 for |d|^2, 1 rcp,
// 2 FMA x 2 components counted as 4), n*n pairs per iteration.
#include <cooperative_groups.h>

#include <algorithm>
#include <cfloat>
#include <climits>
#include <cmath>
#include <cstddef>
#include <mutex>

#include "../../include/batchlayout_gb300.h"
#include "bl_device.cuh"

namespace bl {
namespace {

constexpr int kThreads = 1024;
constexpr int kTeam = 512;                  // sweeper team
constexpr int kGroups = 4;                  // source groups of a team
constexpr int kGroup = kTeam / kGroups;     // 128 threads, two targets each
constexpr int kChunk = 2 * kGroup;          // targets per pass of a team
constexpr int kCWarps = 16;                 // mover: critical team
constexpr int kNWarps = 7;                  // mover: neighbours
constexpr int kPWarps = 8;                  // mover: sweepers' partials (and one warp that watches for them)
constexpr int kRows = 16;                   // sums per target that N and P leave (row kNWarps stays zero)
constexpr int kMoveTile = 32;               // targets a mover handles at a time
constexpr int kPartLoads = 5;               // partials a P lane loads at a time
constexpr int kMaxMovers = 64;              // more than 32 for graphs of long rows only (minibatch_shape)
constexpr double kDense = 100.0;            // mean row length from which they are considered
constexpr int kMaxLag = 2;
constexpr int kExchange = 4;                // slots of the exchange and of the moved counts (two would do)
constexpr int kNear = 16;                   // staged neighbours in the batch before
constexpr int kFlatBlock = 64 * kNWarps;    // entries that team N takes at once where it shares them evenly
constexpr int kFlatJoin = 2 * kFlatBlock;   // more of them: team P takes its part
constexpr unsigned int kNearMore = 0x80000000u;
constexpr int kMaxBatch = 4096;

// A force component beyond +-2^34 (coincident-but-for-rounding vertices) or
// not a number is reported as an error; the vertex keeps its position.
constexpr float kForceLimit = 17179869184.0f;  // 2^34

// Control words of a launch (zero before it).
struct MbControl {
  // movers that stored the new positions of batch q, in word q % kExchange: one
  // mover's count is at most two batches ahead of another's, so a full word
  // tells that every mover is done with its batch (one sum over all batches
  // would not: a mover ahead makes up for one behind)
  unsigned int moved[kExchange];
  unsigned int stop;    // converged runs: the movers ended
  unsigned int ready;   // movers whose first loads are done
  unsigned int pad;
  unsigned int arrive[kMaxLag + 2];  // sweepers that stored a batch's partials, per slot
  // energy per mover, tagged by iteration: {low word, tag}, {high word, tag}
  alignas(16) ulonglong2 energy[2][kMaxMovers];
};
static_assert(offsetof(MbControl, energy) % 16 == 0 && alignof(MbControl) == 16, "16-byte accesses");

struct MinibatchArgs {
  int n, batch, nbatches, model, lag, movers, sweepers;
  int late;  // the movers' early teams start on a batch one batch later (one buffer instead of two)
  float W;
  const int *eff_rowptr, *eff_colids;
  float2 *pos;
  double2 *force;
  double *e;
  float2 *part;             // [lag + 1][sweepers][batch rounded up to even] partial forces
  ulonglong2 *exchange;     // [kExchange][batch] new positions {x, tag}, {y, tag}
  MbControl *ctl;
  double *energy;           // energy of the last iteration (device)
  long long *loops;         // iterations run (device, 1 value)
  DevStatus *st;
  int iterations;
  double step0, decay;
  int converged;
  double engt;
  long long max_loops;
};

// ---- waits and named barriers ------------------------------------------------

__device__ __forceinline__ void bar_sync(int id, int count) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int count) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(count) : "memory");
}

__device__ __forceinline__ void red_add(unsigned int *p, unsigned int v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Bounded poll step: false when the wait has to end (time-out, or an error
// recorded elsewhere).
struct Poll {
  unsigned long long t0;
  unsigned int polls;
  __device__ __forceinline__ Poll() : t0(0), polls(0) {}
  __device__ __forceinline__ bool again(DevStatus *st) {
    if ((++polls & 63u) == 0u) {
      if (ld_volatile_u32(&st->code) != 0u) return false;
      const unsigned long long t = dev_globaltimer();
      if (t0 == 0) t0 = t;
      if (t - t0 > kBarrierTimeoutNs) {
        dev_record_error(st, DEV_TIMEOUT_GRID_BARRIER);
        return false;
      }
    }
    return true;
  }
};

// counters are monotone modulo 2^32
__device__ __forceinline__ bool reached(unsigned int v, unsigned int target) { return (int)(v - target) >= 0; }

__device__ __forceinline__ bool wait_count(const unsigned int *p, unsigned int target, DevStatus *st) {
  Poll w;
#pragma unroll 1
  while (!reached(ld_acquire_gpu(p), target))
    if (!w.again(st)) return false;
  return true;
}

__device__ __forceinline__ unsigned long long tagged(float v, unsigned int tag) {
  return (unsigned long long)__float_as_uint(v) | ((unsigned long long)tag << 32);
}

__device__ __forceinline__ ulonglong2 ld_relaxed_pair(const ulonglong2 *p) {
  ulonglong2 v;
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void st_relaxed_pair(ulonglong2 *p, unsigned long long x, unsigned long long y) {
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(x), "l"(y) : "memory");
}

// ---- packed FP32 pairs -----------------------------------------------------------
//
// Two sources at a time through the packed FP32 instructions (the same
// operations per lane as the scalar form; half the issue slots, which leaves
// room for the reciprocals: 4,307 against 3,788 pairs per ns on 152 SMs with
// 656 sources and 256 targets each).  Sharing one reciprocal between two
// pairs was slower (3,209-3,980): the extra products cost more than the
// shared unit saves.

__device__ __forceinline__ unsigned long long pack2(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float &a, float &b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ unsigned long long sub2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

template <int kRep>
__device__ __forceinline__ float rep_scale(float d2) {
  return kRep == REP_UNIT ? rsqrt_approx(d2) : rcp_approx(d2);
}

// A target and its packed force sums.
struct Target {
  unsigned long long x, y, fx, fy;
  __device__ __forceinline__ void set(float2 p) {
    x = pack2(p.x, p.x);
    y = pack2(p.y, p.y);
    fx = fy = 0ull;  // two +0
  }
  // repulsion of the source pair q = (x0, x1, y0, y1)
  template <int kRep>
  __device__ __forceinline__ void pair(float4 q) {
    const unsigned long long dx = sub2(x, pack2(q.x, q.y)), dy = sub2(y, pack2(q.z, q.w));
    const unsigned long long d2 = fma2(dx, dx, fma2(dy, dy, pack2(kTinyD2, kTinyD2)));
    float a, b;
    unpack2(d2, a, b);
    const unsigned long long r = pack2(rep_scale<kRep>(a), rep_scale<kRep>(b));
    fx = fma2(dx, r, fx);
    fy = fma2(dy, r, fy);
  }
  // repulsion of one source
  template <int kRep>
  __device__ __forceinline__ void single(float sx, float sy) {
    float px, py, t, ax, bx, ay, by;
    unpack2(x, px, t);
    unpack2(y, py, t);
    unpack2(fx, ax, bx);
    unpack2(fy, ay, by);
    rep_law_pair<kRep>(sx, sy, px, py, ax, ay);
    fx = pack2(ax, bx);
    fy = pack2(ay, by);
  }
  __device__ __forceinline__ float2 sum() const {
    float ax, bx, ay, by;
    unpack2(fx, ax, bx);
    unpack2(fy, ay, by);
    return make_float2(ax + bx, ay + by);
  }
};

// Points in shared memory, two per float4 (x0, x1, y0, y1).
__device__ __forceinline__ void put_point(float4 *a, int k, float2 p) {
  float *f = reinterpret_cast<float *>(a + (k >> 1)) + (k & 1);
  f[0] = p.x;
  f[2] = p.y;
}
__device__ __forceinline__ float2 get_point(const float4 *a, int k) {
  const float *f = reinterpret_cast<const float *>(a + (k >> 1)) + (k & 1);
  return make_float2(f[0], f[2]);
}

// Targets of a batch that one mover moves (even, so that pairs of partials
// load as float4).
__host__ __device__ __forceinline__ int mover_share(int batch, int movers) {
  return 2 * ((batch + 2 * movers - 1) / (2 * movers));
}

// Sources of sweeper s: [lo, hi), lo even.
__device__ __forceinline__ void slice_of(int n, int sweepers, int s, int &lo, int &hi) {
  const long long half = (n + 1) / 2;
  lo = 2 * (int)(half * s / sweepers);
  hi = min(n, 2 * (int)(half * (s + 1) / sweepers));
}

// ---- sweeper -----------------------------------------------------------------------

// Slice-local sources [a, b) on two targets.
template <int kRep>
__device__ __forceinline__ void sweep_range(const float4 *slice, int a, int b, Target &t0, Target &t1) {
  if (a >= b) return;
  if (a & 1) {
    const float2 q = get_point(slice, a);
    t0.single<kRep>(q.x, q.y);
    t1.single<kRep>(q.x, q.y);
    a++;
  }
  const int p1 = b >> 1;
#pragma unroll 4
  for (int p = a >> 1; p < p1; p++) {
    const float4 q = slice[p];
    t0.pair<kRep>(q);
    t1.pair<kRep>(q);
  }
  if ((b & 1) && a < b) {
    const float2 q = get_point(slice, b - 1);
    t0.single<kRep>(q.x, q.y);
    t1.single<kRep>(q.x, q.y);
  }
}

// Part g of kGroups of [a, b), cut at even sources.
__device__ __forceinline__ int cut(int a, int b, int g) {
  if (g == 0) return a;
  if (g == kGroups) return b;
  return max(a, (a + (int)((long long)(b - a) * g / kGroups)) & ~1);
}

template <int kRep>
__device__ __forceinline__ void sweeper(const MinibatchArgs &a, unsigned char *smem) {
  const int s = (int)blockIdx.x - a.movers;
  int slo, shi;
  slice_of(a.n, a.sweepers, s, slo, shi);
  const int len = shi - slo;
  float4 *slice = reinterpret_cast<float4 *>(smem);
  const int tid = threadIdx.x % kTeam, team = threadIdx.x / kTeam;
  float2 *gsum = reinterpret_cast<float2 *>(slice + (len + 1) / 2) + team * kGroups * kChunk;
  __shared__ int s_go[2];
  const int grp = tid / kGroup, gl = tid % kGroup;
#pragma unroll 1
  for (int k = threadIdx.x; k < len; k += kThreads) put_point(slice, k, __ldcg(&a.pos[slo + k]));
  __syncthreads();
  const int nb = a.nbatches, B = a.batch, slots = a.lag + 1, stride = (B + 1) & ~1;
  long long left = (a.converged ? LLONG_MAX : (long long)a.iterations * nb) - team;
  // next batch whose new positions this team takes over into the slice
  // (batch numbers modulo 2^32)
  unsigned int fresh = 0;
  int fresh_b = 0;
  int b = team % nb, slot = team % slots;
  // the first targets of the team's next batch are loaded ahead when they
  // cannot move before the current one is done
  const bool ahead = nb >= a.lag + 3;
  float2 p0 = make_float2(0.f, 0.f), p1 = p0;
  bool have = false;
  bool started = false;  // a batch has to have moved
  // batch q - lag - 1, the last that has to have: its word of `moved`, full at
  // `target` (0 and a word of a batch before the run at first)
  int word = (team - a.lag - 1) & (kExchange - 1);
  unsigned int target = team - a.lag - 1 < 0 ? 0u : (unsigned int)a.movers;
  for (unsigned int q = (unsigned int)team; left > 0; q += 2, left -= 2) {
    const unsigned int need = q - (unsigned int)a.lag;  // batches that have moved
    started = started || (int)need > 0;
    if (tid == 0) {
      int go = 1;
      if (started) {
        Poll w;
#pragma unroll 1
        while (!reached(ld_acquire_gpu(&a.ctl->moved[word]), target)) {
          if ((a.converged && ld_volatile_u32(&a.ctl->stop) != 0u) || !w.again(a.st)) {
            go = 0;
            break;
          }
        }
      }
      s_go[team] = go;
    }
    word += 2;
    if (word >= kExchange) {
      word -= kExchange;
      target += (unsigned int)a.movers;
    }
    bar_sync(1 + team, kTeam);
    if (!s_go[team]) return;
    // the batches up to q - lag - 1 have moved: their new positions into the slice
    bool changed = false;
#pragma unroll 1
    for (; started && fresh != need; fresh++) {
      const int lo = fresh_b * B;
      const int f0 = max(slo, lo), f1 = min(shi, min(a.n, lo + B));
#pragma unroll 1
      for (int i = f0 + tid; i < f1; i += kTeam) put_point(slice, i - slo, __ldcg(&a.pos[i]));
      changed |= f0 < f1;
      if (++fresh_b == nb) fresh_b = 0;
    }
    const int base = b * B, cnt = min(B, a.n - base);
    if (!have) {
      p0 = gl < cnt ? __ldcg(&a.pos[base + gl]) : make_float2(0.f, 0.f);
      p1 = gl + kGroup < cnt ? __ldcg(&a.pos[base + gl + kGroup]) : make_float2(0.f, 0.f);
    }
    if (changed) bar_sync(1 + team, kTeam);
    // this team's next batch
    int nxt = b + 2;
    while (nxt >= nb) nxt -= nb;
    // allowed sources: all but batches b - lag .. b - 1 (cyclically)
    const int e = b - a.lag;
    int a0, a1, c0 = 0, c1 = 0;
    if (e >= 0) {
      a0 = 0;
      a1 = min(len, e * B - slo);
      c0 = max(0, base - slo);
      c1 = len;
      if (a.lag == 0) {
        a1 = len;
        c0 = len;
      }
    } else {
      a0 = max(0, base - slo);
      a1 = min(len, (nb + e) * B - slo);
    }
    const int ga0 = cut(a0, max(a0, a1), grp), ga1 = cut(a0, max(a0, a1), grp + 1);
    const int gc0 = cut(c0, max(c0, c1), grp), gc1 = cut(c0, max(c0, c1), grp + 1);
    float2 *out = a.part + ((size_t)slot * a.sweepers + s) * stride;
    for (int t0 = 0; t0 < cnt; t0 += kChunk) {
      Target u, v;
      u.set(p0);
      v.set(p1);
      // the next targets: of this batch, else of the team's next one
      {
        const bool more = t0 + kChunk < cnt;
        const int nbase = more ? base + t0 + kChunk : nxt * B;
        const int ncnt = more ? cnt - t0 - kChunk : min(B, a.n - nbase);
        if (more || ahead) {
          if (gl < ncnt) p0 = __ldcg(&a.pos[nbase + gl]);
          if (gl + kGroup < ncnt) p1 = __ldcg(&a.pos[nbase + gl + kGroup]);
        }
      }
      sweep_range<kRep>(slice, ga0, ga1, u, v);
      sweep_range<kRep>(slice, gc0, gc1, u, v);
      if (t0 > 0) bar_sync(1 + team, kTeam);  // gsum of the chunk before is read
      gsum[grp * kChunk + gl] = u.sum();
      gsum[grp * kChunk + gl + kGroup] = v.sum();
      bar_sync(1 + team, kTeam);
      if (tid < kChunk && t0 + tid < cnt) {
        float2 f = gsum[tid];
#pragma unroll
        for (int g = 1; g < kGroups; g++) {
          const float2 w = gsum[g * kChunk + tid];
          f.x += w.x;
          f.y += w.y;
        }
        __stcg(&out[t0 + tid], f);
      }
    }
    have = ahead;
    bar_sync(1 + team, kTeam);
    if (tid == 0) {
      __threadfence();
      red_add(&a.ctl->arrive[slot], 1u);
    }
    b = nxt;
    slot += 2;
    while (slot >= slots) slot -= slots;
  }
}

// ---- mover --------------------------------------------------------------------------

// The model's attraction of neighbour pj on pi with the pair's repulsion (the
// same FP32 operations) taken back (algorithms.cpp:758-768).
template <int kRep>
__device__ __forceinline__ float2 neighbour_force(int model, float W, float2 pj, float2 pi) {
  const float dx = pj.x - pi.x, dy = pj.y - pi.y;
  const float r = rep_scale<kRep>(fmaf(dx, dx, fmaf(dy, dy, kTinyD2)));
  float fx = dx * r, fy = dy * r;
  attract_pair(model, W, pj.x, pj.y, pi.x, pi.y, fx, fy);
  return make_float2(fx, fy);
}

// Float-float sums of (x, y) in packed form.
struct Sum2 {
  unsigned long long hi, lo;
  __device__ __forceinline__ void add(unsigned long long t) {  // Knuth's TwoSum, as ff_add
    const unsigned long long sum = add2(hi, t);
    const unsigned long long bb = sub2(sum, hi);
    const unsigned long long err = add2(sub2(hi, sub2(sum, bb)), sub2(t, bb));
    hi = sum;
    lo = add2(lo, err);
  }
  __device__ __forceinline__ void add(float x, float y) { add(pack2(x, y)); }
  __device__ __forceinline__ void merge(Sum2 s) {
    add(s.hi);
    lo = add2(lo, s.lo);
  }
  __device__ __forceinline__ Sum2 from_xor(int o) const {
    return Sum2{__shfl_xor_sync(0xffffffffu, hi, o), __shfl_xor_sync(0xffffffffu, lo, o)};
  }
  __device__ __forceinline__ Sum2 from_up(int o) const {
    return Sum2{__shfl_up_sync(0xffffffffu, hi, o), __shfl_up_sync(0xffffffffu, lo, o)};
  }
};

struct MoverSmem {
  float4 *ring;        // [lag + 1][pairs]: positions of the last batches, slot = q % (lag + 1)
  ulonglong2 *rows;    // [2, 1 when late][chunks][kRows][kMoveTile]: N's and P's sums, float-float
  float4 *moved;       // [2][share]: the forces of the share {hi x, hi y, lo x, lo y}
  float2 *tile;        // [tiles][stride]: positions of batches q .. q + 2 (q + 1 when late) before they move
  int *near;           // [2][share][kNear]: neighbours in the batch before (unless late)
  unsigned int *mask;  // [2][share]: which of them are set
  int2 *range;         // [2][share]: where in a long row they are (first above last: not noted; unless late)
  int pairs, stride, share, chunks, tiles;
};

constexpr int kBarC = 1, kBarRing = 2, kBarEarly = 4, kBarPub = 6;
constexpr int kCThreads = kCWarps * 32;
constexpr int kEarlyThreads = kCThreads + (kNWarps + kPWarps) * 32;  // C with N and P

struct MoverFlags {
  // fail, end and gone are set once and stay: they end waits
  volatile int fail;           // a wait ran out or a force left the range
  volatile unsigned int end;   // batches from this one on do not exist (0: not known yet)
  volatile unsigned int seen;  // batches whose partials all sweepers have stored
  volatile int gone;           // the watching warp, whose waits are bounded, has returned
  volatile int last[2];        // by parity of the batch: 1 no batch follows, 2 not even this one
  volatile double step;
  volatile float stepf;
  volatile double energy;  // of the iteration before
  volatile int settled;    // converged runs: the energy changed by no more than engt
  volatile long long loop;  // iterations finished
  volatile int last_loop;   // this iteration is the last one
  double e_lane[32];       // this iteration's energy so far, per lane of the warp that adds it up
};

__device__ __forceinline__ ulonglong2 *rows_of(const MinibatchArgs &a, const MoverSmem &S, int par, int ch) {
  return S.rows + ((a.late ? 0 : par * S.chunks) + ch) * (kRows * kMoveTile);
}

// The critical team's signal that batch q - 2 (q - 1 when late) is in the
// ring, which also means that the sums of that batch are used up; false: there
// is no batch q.
__device__ __forceinline__ bool ring_ready(const MinibatchArgs &a, MoverFlags &F, int par) {
  if (a.late) {
    bar_sync(kBarRing + par, kEarlyThreads);
    return true;
  }
  bar_sync(kBarRing + (par ^ 1), kEarlyThreads);
  return F.last[par ^ 1] == 0;
}

// A lane of team N or P waits until the watching warp has seen `batches`
// batches' partials.  Bounded by that warp: it ends for a run that is over
// (end), one that failed (fail), and at the latest when the warp is gone.
__device__ __forceinline__ void wait_seen(MoverFlags &F, unsigned int batches) {
#pragma unroll 1
  while (!reached(F.seen, batches)) {
    const unsigned int end = F.end;
    if ((end != 0u && reached(batches, end + 1u)) || F.fail || F.gone) break;
  }
}

// One warp: announces in shared memory which batches' partials are complete,
// a round trip ahead of the team that reads them.
__device__ __forceinline__ void mover_watch(const MinibatchArgs &a, MoverFlags &F) {
  unsigned int q = 0, round = 1;
  for (int slot = 0;; q++) {
    Poll p;
#pragma unroll 1
    while (!reached(ld_acquire_gpu(&a.ctl->arrive[slot]), round * (unsigned int)a.sweepers)) {
      const unsigned int end = F.end;
      if ((end != 0u && reached(q, end)) || F.fail) return;
      if (!p.again(a.st)) {
        F.fail = 1;
        return;
      }
    }
    __threadfence_block();
    F.seen = q + 1u;
    if (++slot > a.lag) {
      slot = 0;
      round++;
    }
  }
}

// Where team N finds the neighbours of batch q = `b` of the iteration: batch
// q - d holds vertex j as its vertex t; far: in a batch further back, in global
// memory.
struct Places {
  int slot, slots, batch;
  int w0, w1;  // batches q - slots .. q (cyclically) start at these ids (w1: where they wrap)
  unsigned int span;
  float inv_b;
  int tile;  // where the tile holds the batch's positions before it moves (-1: they are in the ring)
  __device__ __forceinline__ Places(const MinibatchArgs &a, const MoverSmem &S, int b, int slot_, int tslot)
      : slot(slot_), slots(a.lag + 1), batch(a.batch) {
    w0 = (b - slots) * batch;
    w1 = b < slots ? (a.nbatches + b - slots) * batch : INT_MAX;
    span = (slots + 1) * batch;
    inv_b = 1.0f / (float)batch;
    tile = a.nbatches == slots ? -1 : tslot * S.stride;
  }
  __device__ __forceinline__ bool far(int j) const {
    return (unsigned int)(j - w0) >= span && (unsigned int)(j - w1) >= span;
  }
  // of a vertex that is not far
  __device__ __forceinline__ void find(int j, int &d, int &t) const {
    const unsigned int rel = (unsigned int)(j - w0) < span ? j - w0 : j - w1;
    const int k = (int)(((float)rel + 0.5f) * inv_b);  // exact: rel < 2^16
    d = slots - k;
    t = (int)rel - k * batch;
  }
  __device__ __forceinline__ float2 target(const MoverSmem &S, int t) const {
    return tile >= 0 ? S.tile[tile + t] : get_point(S.ring + slot * S.pairs, t);
  }
  // a position that the mover holds (d <= slots)
  __device__ __forceinline__ float2 held(const MoverSmem &S, int d, int t) const {
    if (d == 0) return target(S, t);
    int ss = slot - d;
    if (ss < 0) ss += slots;
    return get_point(S.ring + ss * S.pairs, t);
  }
};

// The row of vertex t of batch b when it is in the share that starts at t0, else an empty one.
__device__ __forceinline__ void row_of(const MinibatchArgs &a, const MoverSmem &S, int b, int t, int t0, int &r0, int &r1) {
  const int i = b * a.batch + t;
  const bool valid = t < min(a.batch, t0 + S.share) && i < a.n;
  r0 = valid ? __ldg(&a.eff_rowptr[i]) : 0;
  r1 = valid ? __ldg(&a.eff_rowptr[i + 1]) : 0;
}

// A neighbour in the batch before, vertex jt of it, entry x of the row of
// staged target t2: the critical team adds it.
__device__ __forceinline__ void stage_near(const MoverSmem &S, int t2, int x, int jt) {
  x &= kNear - 1;
  S.near[t2 * kNear + x] = jt;
  const unsigned int old = atomicOr(&S.mask[t2], 1u << x);
  if ((old >> x) & 1u) atomicOr(&S.mask[t2], kNearMore);
}

// The corrections of a tile of targets in which a row is long (a row a lane,
// [r0, r1), empty where there is no target, `total` entries in all; the first
// target is the share's `off`-th): the seven warps share the tile's entries,
// consecutive in memory, evenly, whatever rows they belong to.  A warp takes 64
// entries at a time, two consecutive ones a lane, with the ids of the next on
// their way.  While all 64 are of one row a lane adds its own until the row
// ends; else a segmented scan over the lanes adds up the rows' parts.  `ready`
// is called once, before the first position is read; false when it was.
template <int kRep, typename Ready>
__device__ __forceinline__ bool neighbours_flat(const MinibatchArgs &a, const MoverSmem &S, int b, int slot, int tslot,
                                                int par, int off, int r0, int r1, int total, int w, Ready ready) {
  const int lane = threadIdx.x & 31, parts = total > kFlatJoin ? kNWarps + kPWarps : kNWarps;
  const Places P(a, S, b, slot, tslot);
  // the tile's entries and the warp's (unsigned: a few past the end are compared too)
  const unsigned int e0 = __shfl_sync(0xffffffffu, r0, 0), e1 = e0 + total;
  const unsigned int each = (total + 64 * parts - 1) / (64 * parts) * 64;
  unsigned int x0 = e0 + (w > kNWarps ? w - 1 : w) * each;
  const unsigned int hi = min(e1, x0 + each);
  int j[2];
  auto fetch = [&](unsigned int x) {
    x += 2 * lane;
#pragma unroll
    for (int u = 0; u < 2; u++) j[u] = x + u < hi ? __ldg(&a.eff_colids[x + u]) : -1;
  };
  fetch(x0);
  // the rows that have entries, numbered through: lane k holds the first entry
  // and the target of the k-th (those beyond: behind all entries)
  unsigned int start = r1 > r0 ? r0 : e1;
  int target = lane;
  const unsigned int some = __ballot_sync(0xffffffffu, start < e1);
  const int nrows = __popc(some);
  if (some & (some + 1u)) {
    target = (int)__fns(some, 0, lane + 1);
    start = __shfl_sync(0xffffffffu, start, target & 31);
    if (target < 0 || target > 31) start = e1;
    target &= 31;
  }
  if (!ready()) return false;
  auto rows = [&]() { return rows_of(a, S, par, off / kMoveTile) + w * kMoveTile; };
  if (w < kNWarps) rows()[lane] = make_ulonglong2(0ull, 0ull);  // (team P's holds its partials)
  __syncwarp();
  auto append = [&](int t, Sum2 s) {  // one lane a target
    ulonglong2 *at = rows() + t;
    Sum2 z = {at->x, at->y};
    z.merge(s);
    *at = make_ulonglong2(z.hi, z.lo);
  };
  // the force of entry x of the row of target t, whose position is p where it
  // is far; nothing where it is staged or no neighbour (an id outside the graph)
  auto force = [&](bool far, float2 p, int t, int x) {
    if (!far) {
      const int id = __float_as_int(p.x);
      if (id < 0) return make_float2(0.f, 0.f);
      int d, jt;
      P.find(id, d, jt);
      if (d == 1 && !a.late) {
        const int t2 = par * S.share + off + t;
        stage_near(S, t2, x, jt);
        atomicMin(&S.range[t2].x, x);
        atomicMax(&S.range[t2].y, x);
        return make_float2(0.f, 0.f);
      }
      p = P.held(S, d, jt);
    }
    return neighbour_force<kRep>(a.model, a.W, p, P.target(S, (int)blockIdx.x * S.share + off + t));
  };
  Sum2 acc = {0ull, 0ull};  // the lane's part of target `cur`
  int cur = -1;
  auto flush = [&]() {
    if (cur < 0) return;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc.merge(acc.from_xor(o));
    if (lane == 0) append(cur, acc);
    __syncwarp();
    acc.hi = acc.lo = 0ull;
    cur = -1;
  };
#pragma unroll 1
  for (; x0 < hi; x0 += 64) {
    bool far[2];
    float2 p[2];
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const bool known = (unsigned int)j[u] < (unsigned int)a.n;
      far[u] = known && P.far(j[u]);
      if (far[u]) p[u] = __ldcg(&a.pos[j[u]]);
      else p[u].x = __int_as_float(known ? j[u] : -1);
    }
    fetch(x0 + 64);
    // the entries' rows: of those that start behind x0 a bit each
    const int first = __popc(__ballot_sync(0xffffffffu, start <= x0)) - 1;  // the row of entry x0
    const unsigned int rel = start - x0;
    const unsigned int lower = __reduce_or_sync(0xffffffffu, rel - 1u < 31u ? 1u << rel : 0u);
    const unsigned int upper = __reduce_or_sync(0xffffffffu, rel - 32u < 32u ? 1u << (rel - 32u) : 0u);
    if ((lower | upper) == 0u) {  // all of one
      const int t = __shfl_sync(0xffffffffu, target, first);
      const int x = (int)(x0 + 2 * lane - __shfl_sync(0xffffffffu, start, first));
      if (cur != t) {
        flush();
        cur = t;
      }
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const float2 f = force(far[u], p[u], t, x + u);
        acc.add(f.x, f.y);
      }
      continue;
    }
    flush();
    const unsigned long long starts = (unsigned long long)upper << 32 | lower;
    int row[2], tgt[2];
    Sum2 s[2];
#pragma unroll
    for (int u = 0; u < 2; u++) {
      row[u] = first + __popcll(starts << (63 - 2 * lane - u));
      tgt[u] = __shfl_sync(0xffffffffu, target, row[u]);
      const float2 f = force(far[u], p[u], tgt[u], (int)(x0 + 2 * lane + u - __shfl_sync(0xffffffffu, start, row[u])));
      s[u].hi = pack2(f.x, f.y);
      s[u].lo = 0ull;
    }
    // the lane's last row, from its first entry on when that is of the same one
    Sum2 run = s[1];
    if (row[0] == row[1]) run.add(s[0].hi);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const Sum2 up = run.from_up(o);
      if (__shfl_up_sync(0xffffffffu, row[1], o) == row[1] && lane >= o) run.merge(up);
    }
    const Sum2 up = run.from_up(1);
    const int last = __shfl_up_sync(0xffffffffu, row[1], 1), next = __shfl_down_sync(0xffffffffu, row[0], 1);
    if (row[0] != row[1]) {  // the row that ends with the first entry
      if (lane > 0 && last == row[0]) s[0].merge(up);
      append(tgt[0], s[0]);
    }
    __syncwarp();
    // (places behind the last entry are of no row)
    if ((lane == 31 || next != row[1]) && row[1] < nrows) append(tgt[1], run);
    __syncwarp();
  }
  flush();
  return true;
}

// Team P's part of a tile: the sweepers' partials of its targets.
__device__ __forceinline__ Sum2 partial_sums(const MinibatchArgs &a, const MoverSmem &S, int w, int slot, int t, int t1) {
  // lane: targets t = 2 (lane % 16) and the next of sweepers 2 w + lane / 16 + 16 k
  const int lane = threadIdx.x & 31;
  const float2 *col = a.part + (size_t)slot * a.sweepers * S.stride + t;
  Sum2 f0 = {0ull, 0ull}, f1 = {0ull, 0ull};
#pragma unroll 1
  for (int s0 = w * 2 + (lane >> 4); s0 < a.sweepers; s0 += 2 * kPWarps * kPartLoads) {
    float4 v[kPartLoads];
#pragma unroll
    for (int k = 0; k < kPartLoads; k++) {
      v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (t < t1 && s0 + 2 * kPWarps * k < a.sweepers)
        v[k] = __ldcg(reinterpret_cast<const float4 *>(&col[(size_t)(s0 + 2 * kPWarps * k) * S.stride]));
    }
#pragma unroll
    for (int k = 0; k < kPartLoads; k++) {
      f0.add(v[k].x, v[k].y);
      f1.add(v[k].z, v[k].w);
    }
  }
  __syncwarp();
  // the other half-warp's sweepers: lanes 0-15 keep the first target, 16-31 the second
  const bool up = lane & 16;
  Sum2 keep = up ? f1 : f0;
  const unsigned long long gh = __shfl_xor_sync(0xffffffffu, up ? f0.hi : f1.hi, 16);
  const unsigned long long gl = __shfl_xor_sync(0xffffffffu, up ? f0.lo : f1.lo, 16);
  keep.add(gh);
  keep.lo = add2(keep.lo, gl);
  return keep;
}

// Teams N and P, seven and eight warps.
// P: the sweepers' partials of the share, and the positions of batch q + 2 (q + 1
// when late) before it moves: N starts on a batch when the critical team has
// finished the second (first) batch before it.
// N: the neighbour corrections of the share, those in batch q - 1 staged
// for the critical team (unless late: the ring holds it then).
// A row is a lane's, of every seventh entry in each of N's warps, one position
// in flight: 0.33 us for seven entries of the longest row.  Where that takes
// longer than the tile's entries shared evenly (neighbours_flat: as 21 entries
// of a row to start with and as 14 for every kFlatBlock) they are shared, above
// kFlatJoin by P's warps too.  us a batch, by lanes only / by this rule: power-
// law graphs of 100,000 vertices and mean degree 10, ids by weight 6.9 / 6.8,
// ids shuffled 11.9 / 7.1, mean degree 40 shuffled 35 / 7.8; 10,000 vertices of
// mean degree 65 shuffled 44 / 6.3; 4,096 vertices of 400 neighbours each 28 /
// 7.8, a grid 3.39 / 3.43.  P looks at its tile's total only: with all rows'
// lengths the grid took 3.48.
// What N reads from global memory moved before batch q - lag - 1, which the
// sweepers saw before they stored the partials of batch q - 1: it waits for
// the watching warp to have seen those (long since).
template <int kRep>
__device__ __forceinline__ void mover_early(const MinibatchArgs &a, const MoverSmem &S, MoverFlags &F, int m) {
  const int w = (int)(threadIdx.x >> 5) - kCWarps, lane = threadIdx.x & 31;  // N: 0 .., P: kNWarps + 1 ..
  const bool sums = w > kNWarps;  // team P
  const int t0 = m * S.share;
  int b = 0, slot = 0;
  // N: this lane's row; P: where the tile's rows start (lane 0) and end (the
  // others); of the share's first tile a batch ahead
  int r0, r1 = 0;
  auto rows_of_tile = [&](int off) {
    if (!sums) {
      row_of(a, S, b, t0 + off + lane, t0, r0, r1);
    } else {
      const int base = b * a.batch, end = min(min(a.batch, a.n - base), min(t0 + S.share, t0 + off + kMoveTile));
      r0 = __ldg(&a.eff_rowptr[base + (lane == 0 ? min(t0 + off, end) : end)]);
    }
  };
  rows_of_tile(0);
  for (unsigned int q = 0;; q++) {
    const int par = (int)(q & 1), tslot = (int)q & (S.tiles - 1);
#pragma unroll 1
    for (int ch = 0; ch < S.chunks; ch++) {
      const int off = ch * kMoveTile;
      if (ch > 0) rows_of_tile(off);
      // waits for the positions (of the share's first tile: the others find them there)
      auto ready = [&]() {
        if (ch > 0 || sums) return true;
        if (!ring_ready(a, F, par)) return false;
        if (lane == 0) wait_seen(F, q);
        __syncwarp();
        __threadfence_block();
        return true;
      };
      if (sums) {
        const int pt = (int)threadIdx.x - (kCWarps + kNWarps + 1) * 32;
        int nbase = -1, ncnt = 0;
        float2 nt[2];
        if (ch == 0) {
          if (lane == 0) wait_seen(F, q + 1u);
          __syncwarp();
          __threadfence_block();
          if (a.nbatches > a.lag + 1) {  // (else every batch is in the ring)
            int fb = b + S.tiles / 2;
            if (fb >= a.nbatches) fb -= a.nbatches;
            nbase = fb * a.batch;
            ncnt = min(a.batch, a.n - nbase);
#pragma unroll
            for (int k = 0; k < 2; k++) {
              const int x = pt + k * kPWarps * 32;
              if (x < ncnt) nt[k] = __ldcg(&a.pos[nbase + x]);
            }
          }
        }
        const int t = t0 + off + 2 * (lane & 15);
        const Sum2 keep = partial_sums(a, S, w - kNWarps - 1, slot, t, min(min(a.batch, a.n - b * a.batch), t0 + S.share));
        if (ch == 0) {
          if (!ring_ready(a, F, par)) return;
          float2 *dst = S.tile + ((tslot + S.tiles / 2) & (S.tiles - 1)) * S.stride;
#pragma unroll
          for (int k = 0; k < 2; k++) {
            const int x = pt + k * kPWarps * 32;
            if (x < ncnt) dst[x] = nt[k];
          }
#pragma unroll 1
          for (int x = pt + 2 * kPWarps * 32; x < ncnt; x += kPWarps * 32) dst[x] = __ldcg(&a.pos[nbase + x]);
        }
        rows_of(a, S, par, ch)[w * kMoveTile + 2 * (lane & 15) + (lane >> 4)] = make_ulonglong2(keep.hi, keep.lo);
        __syncwarp();
      }
      if (sums) {
        if (__shfl_sync(0xffffffffu, r0, 31) - __shfl_sync(0xffffffffu, r0, 0) <= kFlatJoin) continue;
        row_of(a, S, b, t0 + off + lane, t0, r0, r1);
      }
      bool flat = __any_sync(0xffffffffu, r1 - r0 > 5 * kNWarps);
      int total = 0;
      if (__builtin_expect(flat, 0)) {
        total = __reduce_max_sync(0xffffffffu, r1) - __shfl_sync(0xffffffffu, r0, 0);
        flat = __any_sync(0xffffffffu, r1 - r0 > (3 + 2 * ((total + kFlatBlock - 1) / kFlatBlock)) * kNWarps);
      }
      if (__builtin_expect(flat, 0)) {
        if (!neighbours_flat<kRep>(a, S, b, slot, tslot, par, off, r0, r1, total, w, ready)) return;
      } else if (!sums) {
        // (unsigned: places behind the last of 2^31 - 1 entries are compared too)
        unsigned int e = r0 + w;
        const unsigned int end = r1;
        int j0 = e < end ? __ldg(&a.eff_colids[e]) : -1;
        if (!ready()) return;
        const Places P(a, S, b, slot, tslot);
        const float2 p = r0 < r1 ? P.target(S, t0 + off + lane) : make_float2(0.f, 0.f);
        Sum2 f = {0ull, 0ull};
#pragma unroll 1
        for (int j1; e < end; j0 = j1, e += kNWarps) {
          j1 = e + kNWarps < end ? __ldg(&a.eff_colids[e + kNWarps]) : -1;
          // a list handed in on the device is not checked: other ids are no neighbours
          if ((unsigned int)j0 >= (unsigned int)a.n) continue;
          float2 pj;
          if (P.far(j0)) {
            pj = __ldcg(&a.pos[j0]);
          } else {
            int d, jt;
            P.find(j0, d, jt);
            if (d == 1 && !a.late) {  // the batch before: the critical team's
              stage_near(S, par * S.share + off + lane, e - r0, jt);
              continue;
            }
            pj = P.held(S, d, jt);
          }
          const float2 v = neighbour_force<kRep>(a.model, a.W, pj, p);
          f.add(v.x, v.y);
        }
        rows_of(a, S, par, ch)[w * kMoveTile + lane] = make_ulonglong2(f.hi, f.lo);
      }
    }
    bar_arrive(kBarEarly + par, kEarlyThreads);
    if (a.late && F.last[par]) return;
    if (++b == a.nbatches) b = 0;
    if (++slot > a.lag) slot = 0;
    rows_of_tile(0);
  }
}

// A half-warp's sum over the neighbours of vertex i in the batch at `pbase`
// when there are more than were staged: its row again, between the first and
// the last of them where those were noted (`range`), four entries a lane in
// flight.
template <int kRep>
__device__ __noinline__ float2 near_row(const MinibatchArgs &a, const float4 *prev, int pbase, int i, float2 pi,
                                        int2 range) {
  const int r0 = __ldg(&a.eff_rowptr[i]), r1 = __ldg(&a.eff_rowptr[i + 1]);
  const unsigned int pcnt = min(a.batch, a.n - pbase);
  const int lo = range.x <= range.y ? range.x : 0, hi = range.x <= range.y ? range.y + 1 : r1 - r0;
  float2 f = make_float2(0.f, 0.f);
#pragma unroll 1
  for (int x = lo + ((int)threadIdx.x & 15); x < hi; x += 64) {
    unsigned int jt[4];
#pragma unroll
    for (int u = 0; u < 4; u++)
      jt[u] = x + 16 * u < hi ? (unsigned int)__ldg(&a.eff_colids[r0 + x + 16 * u]) - (unsigned int)pbase : ~0u;
#pragma unroll
    for (int u = 0; u < 4; u++) {
      if (jt[u] >= pcnt) continue;
      const float2 g = neighbour_force<kRep>(a.model, a.W, get_point(prev, (int)jt[u]), pi);
      f.x += g.x;
      f.y += g.y;
    }
  }
  return f;
}

// The step when |f|^2 is outside the FP32 range.
__device__ __noinline__ float2 step_fp64(float2 p, float hx, float hy, float lx, float ly, double step) {
  const double dx = (double)hx + (double)lx, dy = (double)hy + (double)ly;
  const double mag = sqrt(dx * dx + dy * dy);
  return make_float2((float)((double)p.x + (dx / mag) * step), (float)((double)p.y + (dy / mag) * step));
}

// One thread's part of the movers' energy exchange: publishes this mover's
// energy of iteration `loop` and, when asked, adds up all of them in order.
__device__ __noinline__ double exchange_energy(const MinibatchArgs &a, MoverFlags &F, int m, long long loop, double v,
                                               bool total) {
  const unsigned long long bits = (unsigned long long)__double_as_longlong(v);
  const unsigned long long tag = (unsigned long long)(unsigned int)(loop + 1);
  ulonglong2 *ce = a.ctl->energy[loop & 1];
  st_relaxed_pair(&ce[m], (bits & 0xffffffffull) | (tag << 32), (bits >> 32) | (tag << 32));
  double tot = 0.0;
#pragma unroll 1
  for (int k = 0; total && k < a.movers; k++) {
    Poll p;
    ulonglong2 x = ld_relaxed_pair(&ce[k]);
#pragma unroll 1
    while ((x.x >> 32) != tag || (x.y >> 32) != tag) {
      if (!p.again(a.st)) {
        F.fail = 1;
        break;
      }
      x = ld_relaxed_pair(&ce[k]);
    }
    tot += __longlong_as_double((long long)((x.x & 0xffffffffull) | (x.y << 32)));
  }
  return tot;
}

// The FP64 forces and |f|^2 of a mover's share (one warp) and, at the end of
// an iteration, its energy: lanes in a fixed tree, movers in order.
__device__ __noinline__ void mover_outputs(const MinibatchArgs &a, const MoverSmem &S, MoverFlags &F, int m, int par,
                                           int base, int count, bool iteration_end) {
  const int lane = threadIdx.x & 31, t0 = m * S.share;
  double e_sum = F.e_lane[lane];
#pragma unroll 1
  for (int t = lane; t < count; t += 32) {
    const float4 f = S.moved[par * S.share + t];
    const double dx = (double)f.x + (double)f.z, dy = (double)f.y + (double)f.w;
    const double e = dx * dx + dy * dy;
    a.force[base + t0 + t] = make_double2(dx, dy);
    a.e[base + t0 + t] = e;
    e_sum += e;
  }
  if (iteration_end) {
    for (int o = 16; o > 0; o >>= 1) e_sum += __shfl_xor_sync(0xffffffffu, e_sum, o);
    if (lane == 0) {
      const double tot = exchange_energy(a, F, m, F.loop, e_sum, a.converged || m == 0);
      if (m == 0) a.energy[0] = tot;
      F.settled = !(fabs(F.energy - tot) / F.energy > a.engt) ? 1 : 0;
      F.energy = tot;
    }
    e_sum = 0.0;
  }
  F.e_lane[lane] = e_sum;
}

// Critical team: the pairs with the last batches, the move, its publication.
// While the batch before is on its way from the other movers, the team adds
// the pairs with the older ones.  The last warp also announces the moved
// batch to the sweepers and turns the share's forces into the FP64 outputs,
// in full warps (the FP64 pipe is charged by the warp instruction), off the
// other warps' path.
template <int kRep>
__device__ __forceinline__ void mover_critical(const MinibatchArgs &a, const MoverSmem &S, MoverFlags &F, int m) {
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int nb = a.nbatches, B = a.batch, slots = a.lag + 1;
  const bool closed = nb == slots;
  const int t0 = m * S.share;
  bool stop = false, started = false;
  int b = 0, slot = 0, tslot = 0;
  if (!a.late) bar_arrive(kBarRing + 1, kEarlyThreads);  // for batch 0 of the early teams: batch -2 is in the ring
  for (unsigned int q = 0;; q++) {
    const int par = (int)(q & 1);
    const int base = b * B;
    const int t1 = min(min(B, a.n - base), t0 + S.share);
    int last = 0;
#pragma unroll 1
    for (int ch = 0; ch < S.chunks; ch++) {
      const int ta = t0 + ch * kMoveTile + 2 * w;
      auto target_at = [&](int t) {
        return t >= t1 ? make_float2(0.f, 0.f)
                       : closed ? get_point(S.ring + slot * S.pairs, t) : S.tile[tslot * S.stride + t];
      };
      Target u, v;  // (without a lag no pair is added)
      u.set(target_at(ta));
      v.set(target_at(ta + 1));
#pragma unroll 1
      for (int d = max(a.lag, 1); d >= 1; d--) {  // batch q - d
        int sb = b - d, ss = slot - d;
        if (sb < 0) sb += nb;
        if (ss < 0) ss += slots;
        float4 *src = S.ring + ss * S.pairs;
        const int scnt = min(B, a.n - sb * B);
        if (d == 1 && ch == 0) {
          // the batch before, from the other movers into the ring
          if (started && !stop) {
            const ulonglong2 *ex = a.exchange + (size_t)((q - 1) & (kExchange - 1)) * B;
#pragma unroll 1
            for (int t = tid; t < scnt; t += kCThreads) {
              Poll p;
              ulonglong2 x = ld_relaxed_pair(&ex[t]);
#pragma unroll 1
              while ((unsigned int)(x.x >> 32) != q || (unsigned int)(x.y >> 32) != q) {
                if (!p.again(a.st)) {
                  F.fail = 1;
                  break;
                }
                x = ld_relaxed_pair(&ex[t]);
              }
              put_point(src, t, make_float2(__uint_as_float((unsigned int)x.x), __uint_as_float((unsigned int)x.y)));
            }
          }
          if (tid == kCThreads - 1) {
            if (!started && !wait_count(&a.ctl->ready, (unsigned int)a.movers, a.st)) F.fail = 1;
            const int l = (stop || F.fail) ? 2 : (F.last_loop && b == nb - 1) ? 1 : 0;
            F.last[par] = l;
            // (a converged run's end is known since its last iteration's end, a
            // failed one's waits end by `fail`: what a wait has seen stays)
            if (l == 1) F.end = q + 1u;
          }
          bar_sync(kBarC, kCThreads);
          last = F.last[par];
          bar_arrive(kBarRing + par, kEarlyThreads);
          if (last == 2) {  // the early teams finish the batch they are in
            bar_sync(kBarEarly + par, kEarlyThreads);
            return;
          }
        }
        if (a.lag >= 1 && ta < t1) {
          // one source pair a lane, the warp's two targets
#pragma unroll 4
          for (int k = lane; k < (scnt >> 1); k += 32) {
            const float4 x = src[k];
            u.pair<kRep>(x);
            v.pair<kRep>(x);
          }
          if ((scnt & 1) && lane == 0) {
            const float2 x = get_point(src, scnt - 1);
            u.single<kRep>(x.x, x.y);
            v.single<kRep>(x.x, x.y);
          }
        }
      }
      if (ch == 0) bar_sync(kBarEarly + par, kEarlyThreads);
      if (ta >= t1) continue;  // a small share leaves warps without targets
      // lanes 0-15 go on with the first target, 16-31 with the second
      const int up = lane >> 4, t = ta + up;
      const float2 pi = target_at(t);
      float fx, fy;
      {
        const float2 fu = u.sum(), fv = v.sum();
        fx = (up ? fv.x : fu.x) + __shfl_xor_sync(0xffffffffu, up ? fu.x : fv.x, 16);
        fy = (up ? fv.y : fu.y) + __shfl_xor_sync(0xffffffffu, up ? fu.y : fv.y, 16);
      }
      // neighbours in the batch before
      if (!a.late) {
        const int x = par * S.share + (t - t0);
        const unsigned int mask = t < t1 ? S.mask[x] : 0u;
        if (__any_sync(0xffffffffu, mask != 0u)) {
          const float4 *prev = S.ring + (slot == 0 ? slots - 1 : slot - 1) * S.pairs;
          const int pbase = b == 0 ? (nb - 1) * B : base - B;
          if (mask & kNearMore) {
            const float2 g = near_row<kRep>(a, prev, pbase, base + t, pi, S.range[x]);
            fx += g.x;
            fy += g.y;
          } else if ((mask >> (lane & 15)) & 1u) {
            const float2 g = neighbour_force<kRep>(a.model, a.W, get_point(prev, S.near[x * kNear + (lane & 15)]), pi);
            fx += g.x;
            fy += g.y;
          }
          __syncwarp();
          if ((lane & 15) == 0 && mask != 0u) {  // for batch q + 2
            S.mask[x] = 0u;
            S.range[x] = make_int2(INT_MAX, -1);
          }
        }
      }
      // with N's and P's sums (a row per lane), a fixed tree over the 16 lanes
      Sum2 s;
      {
        const ulonglong2 row = rows_of(a, S, par, ch)[(lane & 15) * kMoveTile + 2 * w + up];
        s.hi = row.x;
        s.lo = row.y;
      }
      s.add(fx, fy);
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) {
        const unsigned long long h = __shfl_down_sync(0xffffffffu, s.hi, o, 16);
        const unsigned long long l = __shfl_down_sync(0xffffffffu, s.lo, o, 16);
        s.add(h);
        s.lo = add2(s.lo, l);
      }
      if ((lane & 15) == 0 && t < t1) {
        float hx, hy, lx, ly;
        unpack2(s.hi, hx, hy);
        unpack2(s.lo, lx, ly);
        fx = hx + lx;
        fy = hy + ly;
        float2 np = pi;
        const float m2 = fmaf(fx, fx, fy * fy);
        if (m2 >= 1.17549435e-38f && m2 <= 3.0e38f) {
          const float rm = rsqrt_approx(m2), stepf = F.stepf;
          np.x = fmaf(stepf, fx * rm, pi.x);
          np.y = fmaf(stepf, fy * rm, pi.y);
        } else if (fx != 0.f || fy != 0.f) {
          np = step_fp64(pi, hx, hy, lx, ly, F.step);
        }
        const bool in_range = fabsf(fx) < kForceLimit && fabsf(fy) < kForceLimit;
        if (!in_range) np = pi;
        st_relaxed_pair(&a.exchange[(size_t)(q & (kExchange - 1)) * B + t], tagged(np.x, q + 1u), tagged(np.y, q + 1u));
        __stcg(&a.pos[base + t], np);
        if (!in_range) {
          dev_record_error(a.st, DEV_FORCE_RANGE);
          F.fail = 1;
        }
        S.moved[par * S.share + (t - t0)] = make_float4(hx, hy, lx, ly);
      }
    }
    // the last warp learns that the share is stored
    if (w < kCWarps - 1) {
      bar_arrive(kBarPub, kCThreads);
    } else {
      bar_sync(kBarPub, kCThreads);
      if (lane == 0) {
        __threadfence();
        red_add(&a.ctl->moved[q & (kExchange - 1)], 1u);
      }
      if (a.converged || F.last_loop) mover_outputs(a, S, F, m, par, base, t1 - t0, b == nb - 1);
    }
    if (b == nb - 1) {  // end of an iteration
      bar_sync(kBarC, kCThreads);
      const long long loop = F.loop + 1;
      if (a.converged && (F.settled || loop >= a.max_loops)) {
        stop = true;
        F.end = q + 1u;
        if (m == 0 && tid == 0) atomicExch(&a.ctl->stop, 1u);
      }
      bar_sync(kBarC, kCThreads);
      if (tid == kCThreads - 1) {
        F.loop = loop;
        F.last_loop = !a.converged && loop == a.iterations - 1;
        F.step = F.step * a.decay;
        F.stepf = (float)F.step;
        if (m == 0) *a.loops = loop;
      }
    }
    if (last) return;
    started = true;
    if (++b == nb) b = 0;
    if (++slot == slots) slot = 0;
    tslot = (tslot + 1) & (S.tiles - 1);
  }
}

template <int kRep>
__device__ __forceinline__ void mover(const MinibatchArgs &a, unsigned char *smem) {
  __shared__ MoverFlags F;
  __shared__ MoverSmem S;
  const int m = (int)blockIdx.x, B = a.batch, slots = a.lag + 1, nb = a.nbatches;
  const int tid = threadIdx.x;
  if (tid == 0) {
    S.pairs = (B + 1) / 2;
    S.stride = 2 * S.pairs;
    S.share = mover_share(B, a.movers);
    S.chunks = (S.share + kMoveTile - 1) / kMoveTile;
    S.tiles = a.late ? 2 : 4;
    S.ring = reinterpret_cast<float4 *>(smem);
    S.rows = reinterpret_cast<ulonglong2 *>(S.ring + slots * S.pairs);
    S.moved = reinterpret_cast<float4 *>(S.rows + (a.late ? 1 : 2) * S.chunks * kRows * kMoveTile);
    S.tile = reinterpret_cast<float2 *>(S.moved + 2 * S.share);
    S.mask = reinterpret_cast<unsigned int *>(S.tile + S.tiles * S.stride);
    S.near = reinterpret_cast<int *>(S.mask + 2 * S.share);
    S.range = reinterpret_cast<int2 *>(S.near + 2 * S.share * kNear);
    F.fail = 0;
    F.end = 0;
    F.seen = 0;
    F.gone = 0;
    F.last[0] = F.last[1] = 0;
    F.step = a.step0;
    F.stepf = (float)a.step0;
    F.energy = 0.0;
    F.settled = 0;
    F.loop = 0;
    F.last_loop = !a.converged && a.iterations == 1;
  }
  if (tid < 32) F.e_lane[tid] = 0.0;
  __syncthreads();
  // batches -1 .. -slots (the run's first batch has them before it), the first targets
#pragma unroll 1
  for (int d = 1; d <= slots; d++) {
    const int sb = nb - d;
    const int cnt = min(B, a.n - sb * B);
#pragma unroll 1
    for (int t = tid; t < cnt; t += kThreads) put_point(S.ring + (slots - d) * S.pairs, t, __ldcg(&a.pos[sb * B + t]));
  }
  if (nb > slots)  // else every batch is in the ring
#pragma unroll 1
    for (int k = 0; k < S.tiles / 2; k++)
#pragma unroll 1
      for (int t = tid; t < min(B, a.n - k * B); t += kThreads) S.tile[k * S.stride + t] = __ldcg(&a.pos[k * B + t]);
#pragma unroll 1
  for (int t = tid; t < 2 * S.share; t += kThreads) {
    S.mask[t] = 0u;
    if (!a.late) S.range[t] = make_int2(INT_MAX, -1);
  }
#pragma unroll 1
  for (int k = tid; k < (a.late ? 1 : 2) * S.chunks * kMoveTile; k += kThreads)
    S.rows[(k / kMoveTile * kRows + kNWarps) * kMoveTile + k % kMoveTile] = make_ulonglong2(0ull, 0ull);
  __syncthreads();
  // no mover moves a vertex before every mover has its first positions
  if (tid == 0) red_add(&a.ctl->ready, 1u);
  if (tid < kCThreads) mover_critical<kRep>(a, S, F, m);
  else if (tid / 32 != kCWarps + kNWarps) mover_early<kRep>(a, S, F, m);
  else if ((tid & 31) == 0) {
    mover_watch(a, F);
    F.gone = 1;
  }
}

template <int kRep>
__global__ void __launch_bounds__(kThreads, 1) minibatch_kernel(MinibatchArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  if (a.converged && (!(1.0 > a.engt) || a.max_loops < 1)) {  // (DBL_MAX - 0) / DBL_MAX > engt before the first loop
    if (blockIdx.x == 0 && threadIdx.x == 0) *a.loops = 0;
    return;
  }
  if ((int)blockIdx.x < a.movers) mover<kRep>(a, smem_raw);
  else sweeper<kRep>(a, smem_raw);
}

// ---- launch shape ---------------------------------------------------------------------

struct MinibatchShape {
  int movers = 1, sweepers = 1, lag = 0, late = 1;
  size_t smem = 0, part_bytes = 0, exchange_bytes = 0;
  // scratch: control words and exchange (zero before a launch), then partials
  size_t control_bytes() const { return ((sizeof(MbControl) + 255) / 256) * 256 + exchange_bytes; }
  void carve(void *base, MinibatchArgs &a) const {
    unsigned char *p = static_cast<unsigned char *>(base);
    a.ctl = reinterpret_cast<MbControl *>(p);
    a.exchange = reinterpret_cast<ulonglong2 *>(p + ((sizeof(MbControl) + 255) / 256) * 256);
    a.part = reinterpret_cast<float2 *>(p + control_bytes());
    a.lag = lag;
    a.late = late;
    a.movers = movers;
    a.sweepers = sweepers;
  }
};

// Blocks and shared memory for `movers` movers and a lag.
MinibatchShape shape_of(int n, int batch, int num_sms, int movers, int lag) {
  MinibatchShape s;
  const int nb = (n + batch - 1) / batch;
  s.movers = movers;
  s.sweepers = std::max(1, std::min(num_sms - movers, (n + 63) / 64));
  s.lag = std::min(lag, nb - 1);
  if (s.lag > 0 && nb == s.lag + 2) s.lag--;  // every batch in the ring, or the next two outside it
  const size_t slice = (size_t)(2 * (((n + 1) / 2 + s.sweepers - 1) / s.sweepers) + 2);
  const size_t sweeper = slice * sizeof(float2) + 16 + (size_t)2 * kGroups * kChunk * sizeof(float2);
  const size_t share = (size_t)mover_share(batch, s.movers), stride = (size_t)(batch + 1) / 2 * 2;
  const size_t chunks = (share + kMoveTile - 1) / kMoveTile;
  s.late = s.lag == 0 || chunks > 2 ? 1 : 0;
  const size_t mover = (s.lag + 1) * (stride / 2) * sizeof(float4) +
                       (s.late ? 1 : 2) * chunks * kRows * kMoveTile * sizeof(ulonglong2) +
                       2 * share * sizeof(float4) + (s.late ? 2 : 4) * stride * sizeof(float2) +
                       2 * share * (s.late ? 1 : kNear + 3) * sizeof(int);
  s.smem = std::max(sweeper, mover);
  s.part_bytes = (size_t)(s.lag + 1) * s.sweepers * stride * sizeof(float2);
  s.exchange_bytes = (size_t)kExchange * batch * sizeof(ulonglong2);
  return s;
}

// The number of movers with the smallest time per batch, the larger of the
// chain's (2.6 us and the pairs of a share with the `lag` batches before at
// 15,600 a us) and the sweep's (28,500 pairs a us and SM, and 1 us).
// Measured, us per batch with 8 / 16 / 32 movers: 4,096 vertices, batch 256
// 4.0 / 3.2 / 2.9; 100,000, batch 256 6.8 / 7.1 / 7.9; 31,000, batch 512
// 9.1 / 5.8 / 6.1; 30,000, batch 1,000 21.5 / 12.0 / 9.8; 90,000, batch 1,000
// 25.1 / 24.5 / 26.8.  A lag of 2 was best or within 3 % everywhere (4,096
// vertices 1 / 2 / 3 / 4: 3.7 / 2.9 / 3.1 / 3.3; 31,000: 7.8 / 5.8 / 5.9 /
// 6.6); a smaller one where shared memory does not hold the batches.
// Rows (`row`: their mean length, 0 if not known) come beside the chain, or on
// top of it where they start a batch later: 1 us and 1.3 us for every 960
// entries of a share.  That matters from some hundred entries a row on, so in a
// dense graph up to 64 movers, down to two targets each, and every lag are
// considered; elsewhere rows change nothing.  False when a slice does not fit
// a block's shared memory.
bool minibatch_shape(int n, int batch, double row, int num_sms, int smem_optin, MinibatchShape &s) {
  // the largest graph taken: 3.5 million vertices at batch 256, 2.3 million at 4,096
  if ((((n + num_sms - 1) / num_sms + 5) & ~3) * 8LL + 16LL * batch + 44032 > smem_optin) return false;
  bool found = false;
  const bool dense = row >= kDense;
  double best = 0.0;
  for (int lag = 2; lag >= 0 && (!found || dense); lag--) {
    for (int movers = dense ? kMaxMovers : kMaxMovers / 2; movers >= 1; movers /= 2) {
      if (movers > 1 && (movers > (dense ? (batch + 1) / 2 : (batch + 7) / 8) || movers > num_sms / (dense ? 2 : 4)))
        continue;
      const int share = mover_share(batch, movers);
      if (movers < 16 && share > kMoveTile && movers < num_sms / 4) continue;  // several passes a batch
      const MinibatchShape t = shape_of(n, batch, num_sms, movers, lag);
      if (t.smem + 1024 > (size_t)smem_optin) continue;
      const double chain = 2.6 + (double)std::max(t.lag, 1) * batch * share / 15600.0;
      const double sweep = 1.0 + (double)batch * n / (28500.0 * t.sweepers);
      const double rows = dense ? 1.0 + row * share / 740.0 : 0.0;
      const double us = t.late ? (t.lag == 0 ? chain + sweep : std::max(chain, sweep)) + rows
                               : std::max(std::max(chain, sweep), rows);
      if (!found || us < best) {
        best = us;
        s = t;
        found = true;
      }
    }
  }
  return found;
}

// One thread waits for the count as the movers do.
__global__ void count_wait_selftest_kernel(const unsigned int *count, unsigned int target, DevStatus *st) {
  wait_count(count, target, st);
}

}  // namespace

int count_wait_selftest(bl_ctx *ctx, bool complete) {
  // a zero word that nothing counts in
  count_wait_selftest_kernel<<<1, 1, 0, ctx->stream>>>(&ctx->s.status->pad, complete ? 0u : 1u, ctx->s.status);
  BL_CUDA(ctx, cudaGetLastError());
  return 0;
}

int minibatch_run(bl_ctx *ctx, int model, int batch, int iterations, double step0,
                  double decay, bool converged, double engt, long long max_loops,
                  double *energy_out, long long *loops_out) {
  const int n = ctx->g.n;
  if (batch < 1) return bl_fail(ctx, -1, "batch must be >= 1");
  if (n < 1) return bl_fail(ctx, -7, "no graph loaded");
  batch = std::min(batch, n);  // a batch larger than n is one Jacobi batch
  if (batch > kMaxBatch)
    return bl_fail(ctx, -5, "minibatch path supports batch <= 4096 (got " + std::to_string(batch) + ")");
  if (!converged && iterations <= 0) {
    if (energy_out) *energy_out = 0.0;
    if (loops_out) *loops_out = 0;
    return 0;
  }
  // model 2 / 3 / 8: the cursor-matched neighbours, inverse-distance
  // repulsion; 7 (algo 7): FR over every CSR neighbour; 5 (algo 5, second
  // phase): FR over the cursor-matched neighbours, unit-vector repulsion
  const int attract = (model == MODEL_SD || model == MODEL_GREEDY_EXACT) ? (int)MODEL_FR : model;
  const bool unit_rep = model == MODEL_GREEDY_EXACT;
  const bool full_rows = model == MODEL_SD;
  if (full_rows)
    if (int rc = ensure_sorted_csr(ctx)) return rc;
  int dev_smem_optin = 0;
  cudaDeviceGetAttribute(&dev_smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device);
  MinibatchShape sh;
  if (!minibatch_shape(n, batch, (double)ctx->g.nnz / n, ctx->num_sms, dev_smem_optin, sh))
    return bl_fail(ctx, -5, "graph too large for the shared-memory source slices of the minibatch path");
  void (*kernel)(MinibatchArgs) = unit_rep ? minibatch_kernel<REP_UNIT> : minibatch_kernel<REP_INV>;
  const int grid = sh.movers + sh.sweepers;
  BL_CUDA(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh.smem));
  int occ = 0;
  BL_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, kThreads, sh.smem));
  if (occ < 1 || grid > occ * ctx->num_sms)
    return bl_fail(ctx, -5, "minibatch kernel cannot be co-resident");
  const size_t need = sh.control_bytes() + sh.part_bytes;
  if (ctx->s.partials_bytes < need) {
    if (ctx->s.partials) cudaFree(ctx->s.partials);
    ctx->s.partials = nullptr;
    ctx->s.partials_bytes = 0;
    BL_CUDA(ctx, cudaMalloc(&ctx->s.partials, need));
    ctx->s.partials_bytes = need;
  }
  BL_CUDA(ctx, cudaMemsetAsync(ctx->s.status, 0, sizeof(DevStatus), ctx->stream));
  BL_CUDA(ctx, cudaMemsetAsync(ctx->s.partials, 0, sh.control_bytes(), ctx->stream));

  MinibatchArgs a;
  a.n = n;
  a.batch = batch;
  a.nbatches = (n + batch - 1) / batch;
  a.model = attract;
  a.W = (float)ctx->weight;
  a.eff_rowptr = full_rows ? ctx->g.srt_rowptr : ctx->g.eff_rowptr;
  a.eff_colids = full_rows ? ctx->g.srt_colids : ctx->g.eff_colids;
  a.pos = ctx->pos;
  a.force = ctx->force;
  a.e = ctx->e;
  sh.carve(ctx->s.partials, a);
  a.energy = ctx->s.energy;
  a.loops = reinterpret_cast<long long *>(ctx->s.energy + 1);
  a.st = ctx->s.status;
  a.iterations = iterations;
  a.step0 = step0;
  a.decay = decay;
  a.converged = converged ? 1 : 0;
  a.engt = engt;
  a.max_loops = max_loops;
  void *args[] = {&a};
  bl_time_begin(ctx, "minibatch_kernel");
  BL_CUDA(ctx, cudaLaunchCooperativeKernel((const void *)kernel, dim3(grid), dim3(kThreads), args, sh.smem,
                                           ctx->stream));
  bl_time_end(ctx, "minibatch_kernel");
  ctx->launches++;
  double host[2];
  DevStatus st;
  BL_CUDA(ctx, cudaMemcpyAsync(host, ctx->s.energy, 2 * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  BL_CUDA(ctx, cudaMemcpyAsync(&st, ctx->s.status, sizeof(st), cudaMemcpyDeviceToHost, ctx->stream));
  BL_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  if (st.code != DEV_OK)
    if (int rc = bl_check_status(ctx)) return rc;
  long long loops;
  memcpy(&loops, &host[1], sizeof(loops));
  if (energy_out) *energy_out = host[0];
  if (loops_out) *loops_out = loops;
  return 0;
}

}  // namespace bl

// ---------------------------------------------------------------------------
// Allocation-free entry point.
//
// Some callers cannot allocate device memory once they are running: services
// that reserve all GPU memory up front in their own pool, real-time loops
// that forbid allocation after start-up, or code that enqueues work on a
// stream another component owns.  bl_minibatch_iteration_noalloc runs the
// same minibatch kernel as bl_minibatch_iteration, but every scratch buffer
// it needs (partial forces, control words, the device status word) lives
// in the fixed array below, so the call allocates nothing.  The caller passes
// its inputs and outputs as device pointers.
//
// Limits: batch <= 256 and at most 160 blocks (one per SM); the scratch is a
// fixed 1 MiB (partial forces of the batches in flight, control words, status).
// The array exists once per device for the lifetime of the process and every
// call on that device shares it: calls that overlap on the GPU (different
// streams, or host threads that do not serialise) race and give wrong
// results.  The first call on a device looks up the array's device address
// (cudaGetSymbolAddress) with that device current; make that first call
// before any stream capture.
// ---------------------------------------------------------------------------
namespace bl {
namespace {

constexpr int kNoAllocMaxBatch = 256;
constexpr int kNoAllocMaxGrid = 160;
constexpr int kNoAllocMaxLag = kMaxLag;
constexpr size_t kNoAllocBytes = 1024 * 1024;
static_assert(256 + ((sizeof(MbControl) + 255) / 256) * 256 + (size_t)kExchange * kNoAllocMaxBatch * sizeof(ulonglong2) +
                      (size_t)(kNoAllocMaxLag + 1) * kNoAllocMaxGrid * kNoAllocMaxBatch * sizeof(float2) <=
                  kNoAllocBytes,
              "no-alloc scratch too small");

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mutex;
unsigned char *g_noalloc_ptr[kMaxDevices] = {nullptr};

}  // namespace
}  // namespace bl

extern "C" int bl_minibatch_iteration_noalloc(int n, const int *d_rowptr, const int *d_colids,
                                              float *d_xy, double *d_force, double *d_vertex_energy,
                                              int model, int batch, double weight, double step,
                                              double *energy_out, void *stream) try {
  using namespace bl;
  if (n < 1 || !d_rowptr || !d_colids || !d_xy || !d_force || !d_vertex_energy)
    return BL_ERR_ARG;
  if (model != MODEL_FR && model != MODEL_LINLOG && model != MODEL_FA) return BL_ERR_ARG;
  if (batch < 1) return BL_ERR_ARG;
  batch = std::min(batch, n);
  if (batch > kNoAllocMaxBatch) return BL_ERR_TOO_LARGE;  // scratch holds batch <= 256
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= kMaxDevices) return BL_ERR_CUDA;
  unsigned char *base = nullptr;
  {
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_ptr[device]) {
      void *p = nullptr;
      if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p) return BL_ERR_CUDA;
      g_noalloc_ptr[device] = static_cast<unsigned char *>(p);
    }
    base = g_noalloc_ptr[device];
  }
  int num_sms = 0, smem_optin = 0;
  cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, device);
  cudaDeviceGetAttribute(&smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
  // same blocks and shared-memory sizing as the context path
  MinibatchShape sh;
  if (!minibatch_shape(n, batch, 0.0, std::min(num_sms, kNoAllocMaxGrid), smem_optin, sh)) return BL_ERR_TOO_LARGE;
  const int grid = sh.movers + sh.sweepers;
  if (cudaFuncSetAttribute(minibatch_kernel<REP_INV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh.smem) !=
      cudaSuccess)
    return BL_ERR_CUDA;
  int occ = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, minibatch_kernel<REP_INV>, kThreads, sh.smem) !=
          cudaSuccess ||
      occ < 1 || grid > occ * num_sms)
    return BL_ERR_TOO_LARGE;
  // the scratch: status | energy + loops | control words, exchange, partials.
  // The first two and the control words and exchange start at zero.  Partials
  // may be loaded unwritten (the second of a pair of targets when their number
  // is odd, those of a batch past the end) and are not used then.
  DevStatus *status = reinterpret_cast<DevStatus *>(base);
  double *energy = reinterpret_cast<double *>(base + sizeof(DevStatus));
  unsigned char *scratch = base + 256;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (cudaMemsetAsync(base, 0, 256 + sh.control_bytes(), st) != cudaSuccess) return BL_ERR_CUDA;
  MinibatchArgs a;
  a.n = n;
  a.batch = batch;
  a.nbatches = (n + batch - 1) / batch;
  a.model = model;
  a.W = (float)weight;
  a.eff_rowptr = d_rowptr;
  a.eff_colids = d_colids;
  a.pos = reinterpret_cast<float2 *>(d_xy);
  a.force = reinterpret_cast<double2 *>(d_force);
  a.e = d_vertex_energy;
  sh.carve(scratch, a);
  a.energy = energy;
  a.loops = reinterpret_cast<long long *>(energy + 1);
  a.st = status;
  a.iterations = 1;
  a.step0 = step;
  a.decay = 1.0;
  a.converged = 0;
  a.engt = 0.0;
  a.max_loops = 0;
  void *args[] = {&a};
  if (cudaLaunchCooperativeKernel((const void *)minibatch_kernel<REP_INV>, dim3(grid), dim3(kThreads), args, sh.smem,
                                  st) !=
      cudaSuccess)
    return BL_ERR_CUDA;
  double host_energy = 0.0;
  DevStatus host_status;
  if (cudaMemcpyAsync(&host_energy, energy, sizeof(double), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaMemcpyAsync(&host_status, status, sizeof(DevStatus), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return BL_ERR_CUDA;
  if (host_status.code != DEV_OK) return BL_ERR_DEVICE_TIMEOUT;
  if (energy_out) *energy_out = host_energy;
  return BL_OK;
} catch (...) {
  return bl_host_exception(nullptr);
}
