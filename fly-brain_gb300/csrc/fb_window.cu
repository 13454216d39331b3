// The brain step in windows of the synaptic delay: a batch of brains, each advanced H steps
// between grid barriers instead of one. Semantics are those of lif_step (src/wasm/lif.c:29-80),
// bit for bit.
//
// A spike of step s arrives D = nslots - 1 steps later (lif.c:44-45, 77-79), so everything that
// arrives in the window of steps [t, t + H), H <= D, was emitted before t: the window's deliveries
// can all be made first, and then every neuron can run its H steps on its own, its state in
// registers, with no exchange between neurons at all. H is also at most the shortest time between
// two spikes of a neuron (its refractory steps), so within a window a neuron fires at most once
// and each of its edges delivers at most once: a target's contributions of a window fit in a
// region of its in-degree, and one shared counter per target and window replaces one per step.
//
// Per window:
//  P  deliver  the log's spikes that arrive in the window: blocks take batches of arrivals, form
//              each one's amplitude (sign * res, lif.c:37; res recovered to the arrival step), and
//              deal their rows to warps 32 edges at a time; a contribution goes to its target's
//              region keyed by (window step, arrival rank, repeat, inhibitory).
//  -- grid barrier --
//  F, D  one block per brain runs the generator step by step, because the number of draws of a step
//     is the number of driven neurons not refractory (lif.c:49-52); see below. The outputs of
//     xorshift32 are its states, so the draws of a whole window are generated into shared memory
//     ahead of time and a step only looks up draw (base + rank).
//  U  every other neuron, one thread each, all H steps: contributions in key order (lif.c's
//     order), membrane and decays (lif.c:53-72), threshold (lif.c:73-76). With background events
//     (drawn from the same stream) U waits for D.
//  -- grid barrier --
// Spikes are appended to the brain's log. The delay ring of lif.c (its sorted lists) is rebuilt
// from the log when it is asked for.
//
// What bounds it. One brain: a window is a chain of round trips to L2 -- the deliveries (log entry,
// edge, slot claim, barrier: 6.5 us), the driven neurons' free run (7 us beside U), the chain of
// their draws (0.34 us a step), their spikes and state (3.6 us), the last barrier -- 26 us per 18
// steps at 165,122 neurons and 2,000 driven ones, 1.5 us a step against 4.1 with one synchronised
// step at a time, and 0.9 at 20,000 and 200. Many brains: U, latency of the state's loads at 32 warps
// an SM (96 full brains: 780 tiles of 32 neurons per microsecond, 634 us of a window's 970; state
// crosses HBM once per window instead of once per step; the whole launch keeps 45% of the issue slots
// and a sixth of DRAM busy), then the deliveries' slot claims (19e9 a second).
//
// Not covered (the grid kernel runs these): presynaptic inhibition, sequential and fast delivery. One
// brain whose windows would be a few steps long is faster on the lagged kernel (fb_lagged.cu; lag_better
// in fb_api.cu has the rule).
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "fb_window.cuh"

// Compiled once per block width: this file for batches, fb_window_narrow.cu for one brain.
#ifndef FB_WINDOW_WIDTH
#define FB_WINDOW_WIDTH kWinWide
#define FB_WINDOW_NAME wide
#endif

namespace fb {
namespace FB_WINDOW_NAME {

constexpr int kWT = FB_WINDOW_WIDTH;
constexpr int kWinRun = window_run(kWT);
constexpr uint32_t kNone = 0xffffffffu;  // key past a target's last contribution (step bits 31)

__device__ __forceinline__ bool win_timeout(const WinArgs &a, uint64_t t0, uint32_t &it) {
  if ((++it & 63u) == 0) {
    if (ld_volatile(a.err) != 0) return true;
    if (global_ns() - t0 > (uint64_t)a.timeoutNs || it > (1u << 30)) {
      atomicCAS(a.err, 0, FB_ETIMEOUT);
      return true;
    }
  }
  return false;
}

// Grid barrier: every block adds one to a counter that never goes back (the host passes its value
// at launch) and waits until all have (target: its value then); an arrival is a release without a return trip. Bounded, and
// every block leaves once an error is set.
__device__ __noinline__ bool win_sync(const WinArgs &a, uint32_t target) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    int ok = 1;
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.barCount) : "memory");
    const uint64_t t0 = global_ns();
    uint32_t it = 0;
    while ((int32_t)(ld_acquire(a.barCount) - target) < 0)
      if (win_timeout(a, t0, it)) {
        ok = 0;
        break;
      }
    if (ok && ld_volatile(a.err) != 0) ok = 0;
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// ---- a target's contributions of the window, in key order ----------------------------------
struct List {
  const uint2 *p;  // sorted entries, `stride` apart
  int stride;
  uint32_t left;   // entries after the current one
  uint32_t key;    // the current entry (kNone: none)
  float val;
};

__device__ __forceinline__ void list_next(List &l) {
  if (l.left) {
    l.p += l.stride;
    l.left--;
    l.key = l.p->x;
    l.val = __uint_as_float(l.p->y);
  } else {
    l.key = kNone;
  }
}

// Heap sort in place by key, one thread (the region is its target's until the next barrier).
__device__ __noinline__ void heap_sort(uint2 *e, uint32_t n) {
  auto sift = [&](uint32_t root, uint32_t end) {
    const uint2 x = e[root];
    for (;;) {
      uint32_t c = 2 * root + 1;
      if (c >= end) break;
      uint2 y = e[c];
      if (c + 1 < end) {
        const uint2 z = e[c + 1];
        if (z.x > y.x) {
          y = z;
          c++;
        }
      }
      if (y.x <= x.x) break;
      e[root] = y;
      root = c;
    }
    e[root] = x;
  };
  for (uint32_t r = n / 2; r-- > 0;) sift(r, n);
  for (uint32_t end = n - 1; end > 0; end--) {
    const uint2 x = e[end];
    e[end] = e[0];
    e[0] = x;
    sift(0, end);
  }
}

// Sort in place by key, one warp: every lane counts the keys below its own (up to 4 of them, so up
// to 128 entries; longer ones by lane 0 alone). Keys are unique.
__device__ __noinline__ void warp_sort(uint2 *e, uint32_t n) {
  constexpr int kM = 4;
  const uint32_t lane = threadIdx.x & 31u;
  if (n > 32 * kM) {
    if (lane == 0) heap_sort(e, n);
    __syncwarp();
    return;
  }
  uint2 x[kM];
  uint32_t rank[kM];
#pragma unroll
  for (int m = 0; m < kM; m++) {
    const uint32_t k = lane + 32 * m;
    x[m] = k < n ? ldcg(e + k) : make_uint2(kNone, 0u);
    rank[m] = 0;
  }
#pragma unroll
  for (int g = 0; g < kM; g++) {
    if (32u * g >= n) break;
    for (int l = 0; l < 32; l++) {
      const uint32_t y = __shfl_sync(0xffffffffu, x[g].x, l);
#pragma unroll
      for (int m = 0; m < kM; m++) rank[m] += y < x[m].x;
    }
  }
  __syncwarp();
#pragma unroll
  for (int m = 0; m < kM; m++)
    if (lane + 32 * m < n) e[rank[m]] = x[m];
  __syncwarp();
}

// The n contributions at e as a sorted list, every lane of the warp its own target's: up to
// kWinSort are sorted by insertion into `stage` (shared memory, entries 32 apart: one bank pair per
// lane), more in place by the whole warp.
// first: e[0], loaded before.
__device__ __forceinline__ List make_list(uint2 *e, uint32_t n, uint2 *stage, uint2 first) {
  for (uint32_t big = __ballot_sync(0xffffffffu, n > (uint32_t)kWinSort); big; big &= big - 1) {
    const int src = __ffs(big) - 1;
    uint2 *p = (uint2 *)__shfl_sync(0xffffffffu, (unsigned long long)e, src);
    warp_sort(p, __shfl_sync(0xffffffffu, n, src));
  }
  List l;
  l.left = 0;
  l.key = kNone;
  l.p = e;
  l.stride = 1;
  l.val = 0.f;
  if (n == 0) return l;
  if (n > 1 && n <= (uint32_t)kWinSort) {
    for (uint32_t u0 = 0; u0 < n; u0 += 4) {
      uint2 x[4];
#pragma unroll
      for (int c = 0; c < 4; c++) x[c] = u0 + c == 0 ? first : u0 + c < n ? ldcg(e + u0 + c) : make_uint2(kNone, 0u);
#pragma unroll
      for (int c = 0; c < 4; c++) {
        if (u0 + c >= n) break;
        uint32_t w = u0 + c;
        while (w > 0) {
          const uint2 y = stage[(w - 1) * 32];
          if (y.x < x[c].x) break;
          stage[w * 32] = y;
          w--;
        }
        stage[w * 32] = x[c];
      }
    }
    l.p = stage;
    l.stride = 32;
  }
  const uint2 x = n == 1 ? first : *l.p;
  l.key = x.x;
  l.val = __uint_as_float(x.y);
  l.left = n - 1;
  return l;
}

// Phase timer (fb_profile): thread 0 of block 0 and of the last block add the time since their
// last lap to slot k0 and k1 (-1: none).
__device__ __forceinline__ void win_lap(const WinArgs &a, int k0, int k1, uint64_t &tp) {  // tp: shared
  if (a.prof == nullptr || threadIdx.x != 0 || (blockIdx.x != 0 && blockIdx.x != gridDim.x - 1)) return;
  const uint64_t now = global_ns();
  const int k = blockIdx.x == 0 ? k0 : k1;
  if (k >= 0) atomicAdd(a.prof + k, (unsigned long long)(now - tp));
  tp = now;
}

struct Neuron {
  float v, ge, gi, r, ad, rs;
};

// The header constants of a neuron's step, in registers.
struct Model {
  float vRest, vReset, kM, dt, dE, tRef;                                          // every brain
  float vThresh, dA, kRec, adaptInc, depU, bgAmp, eExc, eInh, cE, cI;
  int coba;
};
template <int GEN>
__device__ __forceinline__ Model model_of(const Trial &T) {
  Model m;
  m.vRest = T.vRest; m.vReset = T.vReset; m.kM = T.kM; m.dt = T.dt; m.dE = T.dE; m.tRef = T.tRef;
  if (GEN) {
    m.vThresh = T.vThresh; m.dA = T.dA; m.kRec = T.kRec; m.adaptInc = T.adaptInc; m.depU = T.depU; m.bgAmp = T.bgAmp;
    m.eExc = T.eExc; m.eInh = T.eInh; m.cE = T.cE; m.cI = T.cI; m.coba = T.coba;
  }
  return m;
}

// One step of one neuron, after its forced spike, if any, was applied. First its inputs: the
// contributions, background hits (lif.c:48), its own depression (lif.c:37-39). Then membrane and
// decays (lif.c:55-72) and threshold (lif.c:73-76). One IEEE f32 operation per C operation, in C
// order. GEN 0 leaves out what the brain's flags make constant: adapt 0, res 1, current-based, no
// background, no depression (thB = vThresh + adapt + thr then does not change either).
template <int GEN>
__device__ __forceinline__ void neuron_inputs(const Model &T, Neuron &x, List &l, int j, uint32_t hits, bool depress, float sign) {
  while ((l.key >> 27) == (uint32_t)j) {
    if (l.key & 1u) x.gi = __fadd_rn(x.gi, l.val);
    else x.ge = __fadd_rn(x.ge, l.val);
    list_next(l);
  }
  if (GEN) {
    for (uint32_t u = 0; u < hits; u++) x.ge = __fadd_rn(x.ge, T.bgAmp);
    if (depress && !(__fmul_rn(sign, x.rs) == 0.f)) x.rs = __fsub_rn(x.rs, __fmul_rn(T.depU, x.rs));
  }
}

// Returns whether the neuron crossed its threshold.
template <int GEN>
__device__ __forceinline__ bool neuron_step(const Model &T, Neuron &x, float bias, float thr, float thB) {
  float acc = __fsub_rn(T.vRest, x.v);
  if (GEN && T.coba) {
    acc = __fadd_rn(acc, __fmul_rn(__fmul_rn(x.ge, __fsub_rn(T.eExc, x.v)), T.cE));
    acc = __fadd_rn(acc, __fmul_rn(__fmul_rn(x.gi, __fsub_rn(x.v, T.eInh)), T.cI));
  } else {
    acc = __fadd_rn(acc, x.ge);
    acc = __fadd_rn(acc, x.gi);
  }
  acc = __fadd_rn(acc, bias);
  const float dv = __fmul_rn(acc, T.kM);
  const bool refractory = x.r > 0;
  x.v = refractory ? T.vReset : __fadd_rn(x.v, dv);
  x.r = refractory ? __fsub_rn(x.r, T.dt) : x.r;
  x.ge = __fmul_rn(x.ge, T.dE);
  x.gi = __fmul_rn(x.gi, T.dE);
  if (GEN) {
    x.ad = __fmul_rn(x.ad, T.dA);
    x.rs = __fadd_rn(x.rs, __fmul_rn(__fsub_rn(1.f, x.rs), T.kRec));
    thB = __fadd_rn(__fadd_rn(T.vThresh, x.ad), thr);
  }
  if (x.v >= thB && x.r <= 0) {
    x.v = T.vReset;
    x.r = T.tRef;
    if (GEN) x.ad = __fadd_rn(x.ad, T.adaptInc);
    return true;
  }
  return false;
}

// Appends the warp's spikes (lanes with step >= 0) to brain b's log and counts those of the
// launch's last step.
__device__ __forceinline__ void log_append(const Trial &T, const WinBrain &C, WinBrain *W, Trial *G, int step, uint64_t g0, int t0, int steps,
                                           int32_t id, uint32_t rank) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t on = __ballot_sync(0xffffffffu, step >= 0);
  if (!on) return;
  const uint32_t r0 = __ldg(T.indptr + id), r1 = __ldg(T.indptr + id + 1);
  uint32_t base = 0;
  if (lane == (uint32_t)__ffs(on) - 1) base = atomicAdd(&W->logTop, (uint32_t)__popc(on));
  base = __shfl_sync(0xffffffffu, base, __ffs(on) - 1);
  if (step >= 0) {
    const uint32_t at = base + __popc(on & ((1u << lane) - 1u));
    const uint32_t e = (uint32_t)(g0 + (uint64_t)step) & 255u;
    C.log[at & C.logMask] = make_uint4((uint32_t)id | (e << 24), rank, r0, r1);
    if (t0 + step == steps - 1) atomicAdd(&G->nFired, 1);
  }
}

// lif.c:57-60's trace over the window: decayed every step, 1 at a spike. A forced spike (before
// the step's decay) still decays in its own step.
__device__ __forceinline__ float trace_window(float tr, float dTr, int h, int fired, bool forced) {
  int k = 0;
  if (fired >= 0) {
    tr = 1.f;
    k = forced ? fired : fired + 1;
  }
  for (; k < h; k++) tr = __fmul_rn(tr, dTr);
  return tr;
}

// What the parts of the kernel share: the brains' headers (a single brain's in shared memory) and
// the launch's and window's per-brain words.
struct WinCtx {
  const Trial *tr;      // headers
  const WinBrain *win;  // sizes and pointers
  const int64_t *done;
  const int32_t *steps;
  uint32_t *pre;
  // window w of brain b: steps t0 .. t0 + h - 1 of the launch
  __device__ __forceinline__ int t0(int b, int w) const { return w * win[b].H; }
  __device__ __forceinline__ int h(int b, int w) const { return min(win[b].H, steps[b] - w * win[b].H); }
};
// What a warp needs of the brain whose tiles it takes, in its own words of shared memory: read once
// per brain instead of through L1, which the block's shared memory leaves too small to hold it.
struct WarpBrain {
  float *v;           // the state's fields are one allocation: v gE gI refr trace adapt res bias thr,
  uint32_t f;         // f apart
  int32_t N, flags, nD, h, t0, steps;
  uint32_t e0, logMask;  // the window's first step (low bits)
  float dTr, vThresh;
  Model K;
  const uint32_t *inOff, *indptr;
  const int32_t *drvPos;
  uint32_t *wcnt, *spikeCount, *bgMask, *bgHit;
  uint2 *wbuf;
  uint4 *log;
  uint8_t *arr;
  const float *sign;
  uint32_t *logTop;
  int32_t *nFired;
};
struct DrivenShared {
  uint4 cnt[2][2];             // live entries per warp, a byte each, by step parity
  uint32_t base[kWinMax + 1];  // draws before each step's first
  uint32_t nbg[kWinMax + 1];
  uint32_t events;
  uint64_t tp;  // phase timer
  float acc;    // the background accumulator after the window
  int changed;
};

struct SpikeRec {  // an arrival a block delivers
  uint32_t lo, hi, key;
  uint32_t id;
  int32_t b;
};

struct WinShared {
  uint32_t scan[33];
  uint32_t jump[kWinJumpWords];
  DrivenShared dr;
  union {
    struct {
      SpikeRec rec[kWinSpikes];
      uint32_t pre[kWinSpikes + 1];
    };
  };
  WarpBrain wb[kWT > 512 ? kWT / 32 : 1][2];
  WinArgs a;
  WinCtx ctx;
  Trial tr;  // a single brain's headers
  WinBrain win;
};

// The block's shared memory: named here, so that every part addresses it as such. s_pool: D's draws
// and entry words, or the sort staging of F and U; then the per-brain words of WinCtx.
__shared__ WinShared s_win;
extern __shared__ __align__(16) uint32_t s_pool[];

__device__ __forceinline__ uint2 *sort_stage() {
  return (uint2 *)s_pool + (size_t)(threadIdx.x >> 5) * 32 * kWinSort + (threadIdx.x & 31);
}

__device__ __forceinline__ bool plain_brain(const Trial &T) {
  return (T.flags & (kAdaptZero | kResRest | kHasBg | kHasDep)) == (kAdaptZero | kResRest) && !T.coba;
}

__device__ __forceinline__ int find_brain(const uint32_t *pre, int B, uint32_t x) {  // pre[b] <= x < pre[b+1]
  int lo = 0, hi = B;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (pre[mid] <= x) lo = mid;
    else hi = mid;
  }
  return lo;
}

// ---- U: the other neurons, the whole window ---------------------------------------------------
//
// A warp takes tiles of 32 neurons, and the steps between two contributions to any of them run
// without looking at the lists: about 14 instructions per neuron and step. Bound by the latency of
// the state's loads and by instructions: the other warps' steps are what hides a tile's loads. Measured
// on 96 full brains, a window's U: 769 us when a warp also loaded
// its next tile ahead (the registers for it spill, and the block's shared memory leaves little L1 to
// spill to), 641 us with a tile at a time and the other 31 warps to hide its loads, 592 us now; with
// the next two tiles copied to shared memory ahead no less.
struct Tile {
  int32_t i;  // this lane's neuron (0 where it has none)
  int32_t pos;  // its place in the driven list (-1: not driven)
  uint32_t o, o1, end;  // its region of wbuf, the end of its contributions
  Neuron x;
  float tr, bias, thr;
  uint32_t ar;
};

// By one thread, before the window's first barrier.
__device__ __forceinline__ void make_brain(WarpBrain &B, const WinArgs &a, const WinCtx &c, int w, int b) {
  const Trial &T = c.tr[b];
  const WinBrain &C = c.win[b];
  B.v = T.v;
  B.f = (uint32_t)(T.gE - T.v);
  B.N = T.N;
  B.flags = T.flags;
  B.nD = a.B == 1 ? T.nDriven : ldcg(&a.trials[b].nDriven);
  B.h = c.h(b, w);
  B.t0 = c.t0(b, w);
  B.steps = c.steps[b];
  B.e0 = (uint32_t)(c.done[b] + B.t0);
  B.logMask = C.logMask;
  B.dTr = T.dTr;
  B.vThresh = T.vThresh;
  B.K = model_of<1>(T);
  B.inOff = C.inOff;
  B.indptr = T.indptr;
  B.drvPos = C.drvPos;
  B.wcnt = C.wcnt;
  B.spikeCount = T.spikeCount;
  B.bgMask = C.bgMask;
  B.bgHit = C.bgHit;
  B.wbuf = C.wbuf;
  B.log = C.log;
  B.arr = C.arr;
  B.sign = T.sign;
  B.logTop = &a.win[b].logTop;
  B.nFired = &a.trials[b].nFired;
}
// Into the warp's own words: a thread that reads the headers one by one takes microseconds.
__device__ __forceinline__ void copy_brain(WarpBrain &B, const WarpBrain *src) {
  static_assert(sizeof(WarpBrain) <= kWarpBrainBytes && sizeof(WarpBrain) % 4 == 0, "room in the launch's table");
  __syncwarp();
#pragma unroll
  for (uint32_t k = threadIdx.x & 31u; k < sizeof(WarpBrain) / 4; k += 32) ((uint32_t *)&B)[k] = ldcg((const uint32_t *)src + k);
  __syncwarp();
}


// Only loads: nothing here waits for one.
template <int GEN>
__device__ __forceinline__ void tile_load(const WarpBrain &T, int32_t i, Tile &t) {
  const int32_t q = i < T.N ? i : 0;
  t.i = q;
  const uint32_t f = T.f;
  const float *p = T.v + q;
  t.pos = ldcg(T.drvPos + q);
  t.o = __ldg(T.inOff + q);
  t.o1 = __ldg(T.inOff + q + 1);
  t.end = ldcg(T.wcnt + q);
  t.x.v = ldcg(p);
  t.x.ge = ldcg(p + f);
  t.x.gi = ldcg(p + 2 * f);
  t.x.r = ldcg(p + 3 * f);
  t.tr = ldcg(p + 4 * f);
  t.x.ad = GEN ? ldcg(p + 5 * f) : 0.f;
  t.x.rs = GEN ? ldcg(p + 6 * f) : 1.f;
  t.bias = (T.flags & kBiasZero) ? 0.f : ldcg(p + 7 * f);
  t.thr = (T.flags & kThrZero) ? 0.f : ldcg(p + 8 * f);
  t.ar = (GEN && (T.flags & kHasDep)) ? (uint32_t)ldcg(T.arr + q) : 0u;
}

// own: the lane has a neuron of its own here; n, first: its contributions and the first of them.
template <int GEN>
__device__ __forceinline__ void tile_run(const WarpBrain &T, const Tile &t, bool own, uint32_t n, uint2 first, uint2 *stage) {
  const int h = T.h;
  const int ar = (int)t.ar - 1;
  const uint32_t bg = (GEN && (T.flags & kHasBg) && own) ? ldcg(T.bgMask + t.i) : 0u;
  const float sign = (GEN && ar >= 0) ? __ldg(T.sign + t.i) : 0.f;
  List l = make_list(T.wbuf + t.o, n, stage, first);
  const Model K = T.K;
  Neuron x = t.x;
  // words that provably keep their bits are not stored: a conductance of +0 without input, a
  // refractory count of 0 or less and a trace of +0 without a spike
  const bool geKeeps = __float_as_uint(x.ge) == 0u && n == 0 && bg == 0, giKeeps = __float_as_uint(x.gi) == 0u && n == 0;
  const bool rKeeps = !(x.r > 0), trKeeps = __float_as_uint(t.tr) == 0u;
  const float thB = __fadd_rn(__fadd_rn(T.vThresh, x.ad), t.thr);
  int fired = -1;
  if (GEN) {
    for (int j = 0; j < h; j++) {
      uint32_t hits = (bg >> j) & 1u;
      if (hits && (bg >> 31)) {  // further hits of some step
        uint32_t *ph = T.bgHit + (int64_t)j * T.N + t.i;
        hits += ldcg(ph);
        *ph = 0;
      }
      neuron_inputs<1>(K, x, l, j, hits, ar == j, sign);
      if (neuron_step<1>(K, x, t.bias, t.thr, thB)) fired = j;
    }
  } else {
    int j = 0;
    if (kWT > 512 && !__any_sync(0xffffffffu, K.vReset >= thB || x.r != x.r)) {
      // The refractory count as the step it ends before: a neuron that fires stays refractory to the
      // window's end, and while it is it cannot cross a threshold above vReset. (A count that is not a
      // number lets the neuron integrate but never fire: the other path.) Four instructions fewer per
      // step: 96 brains 641 -> 617 us a window; one brain gains nothing (its warps have two tiles at
      // most).
      int silent = 0;
      float r = x.r;
      for (int q = 0; q < h && __any_sync(0xffffffffu, r > 0); q++)
        if (r > 0) {
          r = __fsub_rn(r, K.dt);
          silent = q + 1;
        }
      while (j < h) {
        neuron_inputs<0>(K, x, l, j, 0, false, 0.f);
        // steps until any lane's next contribution
        const int e = min(h, (int)__reduce_min_sync(0xffffffffu, l.key >> 27));
        do {  // neuron_step<0>
          const float acc = __fadd_rn(__fadd_rn(__fadd_rn(__fsub_rn(K.vRest, x.v), x.ge), x.gi), t.bias);
          const float v = __fadd_rn(x.v, __fmul_rn(acc, K.kM));
          const bool cross = j >= silent && v >= thB;
          x.v = j < silent || cross ? K.vReset : v;
          silent = cross ? kWinMax + 1 + j : silent;
          x.ge = __fmul_rn(x.ge, K.dE);
          x.gi = __fmul_rn(x.gi, K.dE);
        } while (++j < e);
      }
      fired = silent - (kWinMax + 1);
      x.r = r;
      if (__any_sync(0xffffffffu, fired >= 0)) {
        if (fired >= 0) x.r = K.tRef;
        for (int q = 1; q < h; q++)
          if (fired >= 0 && q > fired) x.r = __fsub_rn(x.r, K.dt);
      }
    }
    while (j < h) {
      neuron_inputs<0>(K, x, l, j, 0, false, 0.f);
      const int e = min(h, (int)__reduce_min_sync(0xffffffffu, l.key >> 27));
      do {
        if (neuron_step<0>(K, x, t.bias, t.thr, thB)) fired = j;
      } while (++j < e);
    }
  }
  if (!own) fired = -1;
  const bool spiked = fired >= 0;
  const uint32_t on = __ballot_sync(0xffffffffu, spiked);
  if (on) {
    const uint32_t lane = threadIdx.x & 31u, lead = (uint32_t)__ffs(on) - 1;
    uint32_t base = 0;
    if (lane == lead) base = atomicAdd(T.logTop, (uint32_t)__popc(on));
    const uint32_t r0 = __ldg(T.indptr + t.i), r1 = __ldg(T.indptr + t.i + 1);
    base = __shfl_sync(0xffffffffu, base, lead);
    if (spiked) {
      T.log[(base + __popc(on & ((1u << lane) - 1u))) & T.logMask] =
          make_uint4((uint32_t)t.i | (((T.e0 + (uint32_t)fired) & 255u) << 24), (uint32_t)(T.nD + t.i), r0, r1);
      if (T.t0 + fired == T.steps - 1) atomicAdd(T.nFired, 1);
      atomicAdd(T.spikeCount + t.i, 1u);
    }
  }
  if (!own) return;
  const uint32_t f = T.f;
  float *p = T.v + t.i;
  if (__float_as_uint(x.v) != __float_as_uint(t.x.v)) *p = x.v;
  if (!geKeeps) p[f] = x.ge;
  if (!giKeeps) p[2 * f] = x.gi;
  if (!rKeeps || spiked) p[3 * f] = x.r;
  if (!trKeeps || spiked) p[4 * f] = trace_window(t.tr, T.dTr, h, fired, false);
  if (GEN) {
    if (!(T.flags & kAdaptZero)) p[5 * f] = x.ad;
    if (!(T.flags & kResRest)) p[6 * f] = x.rs;
  }
  if (n) T.wcnt[t.i] = t.o;
  if (GEN && bg) T.bgMask[t.i] = 0;
  if (GEN && ar >= 0) T.arr[t.i] = 0;
}

// This warp's share of the tiles of all brains (`total`, numbered through the prefix c.pre). Few
// tiles per warp: dealt. Many: three quarters dealt as runs of a warp (a run stays within few brains), the
// rest taken by tickets from a counter, so that blocks that come late from a driven list take fewer:
// four tiles a ticket, the last ones singly, as the warps of a block take 6 us for a tile.
// meet: where not 0, the target of the grid barrier that U waits at, after the first loads.
template <int GEN>
__device__ __noinline__ bool update_tiles(int w, uint32_t total, uint32_t first,
                                          uint32_t nWarps, uint32_t meet) {
  const WinArgs &a = s_win.a;
  const WinCtx &c = s_win.ctx;
  WarpBrain *wb = s_win.wb[kWT > 512 ? threadIdx.x >> 5 : 0];  // one brain: one for the block
  uint2 *stage = sort_stage();
  const uint32_t lane = threadIdx.x & 31u;
  constexpr uint32_t kGrab = 4;
  const bool dyn = total >= 16 * nWarps;
  const uint32_t run = total / nWarps * 3 / 4, dealt = dyn ? run * nWarps : total;
  const uint32_t grabs = (total - dealt) / kGrab - min((total - dealt) / kGrab, nWarps / kGrab);  // tickets of four
  uint32_t g = dyn ? first * run : first, end = dyn ? g + run : total;
  // tiles first + k nWarps of every brain's, or of a run: two brains at most are in use at a time
  uint32_t lo = 0, hi = 0, cur = 0;
  Tile t;
  auto load = [&](Tile &x) {
    if (kWT > 512 && (g < lo || g >= hi)) {
      const int b = find_brain(c.pre, a.B, g);
      lo = c.pre[b];
      hi = c.pre[b + 1];
      cur ^= 1u;
      copy_brain(wb[cur], (const WarpBrain *)(a.brains + (size_t)b * kWarpBrainBytes));
    }
    tile_load<GEN>(wb[cur], (int32_t)((g - lo) * 32 + lane), x);
  };
  if (g < total) load(t);
  if (meet && !win_sync(a, meet)) return false;
  while (g < total) {
    const WarpBrain &T = wb[cur];
    const bool own = t.pos < 0 && (g - lo) * 32 + lane < (uint32_t)T.N;
    uint32_t n = own ? t.end - t.o : 0u;
    if (n > t.o1 - t.o) {  // two spikes of one neuron in a window
      atomicCAS(a.err, 0, FB_EOVERFLOW);
      n = 0;
    }
    uint2 head = make_uint2(kNone, 0u);
    if (n) head = ldcg(T.wbuf + t.o);
    g += dyn ? 1 : nWarps;
    if (dyn && g >= end) {
      uint32_t x = 0;
      if (lane == 0) x = atomicAdd(a.uNext + (w & 1), 1u);
      x = __shfl_sync(0xffffffffu, x, 0);
      g = dealt + (x < grabs ? x * kGrab : grabs * kGrab + (x - grabs));
      end = min(total, g + (x < grabs ? kGrab : 1u));
    }
    const bool more = g < total;
    tile_run<GEN>(T, t, own, n, head, stage);
    __syncwarp();
    if (more) load(t);
  }
  return true;
}

// ---- F and D: the driven neurons and the generator -------------------------------------------
//
// A step's draws go to the driven neurons not refractory then, in list order, so where each draw
// lands depends on every earlier spike of the list: a chain over the window's steps. Only that is
// done step by step, by one block per brain. First (F, tiles of 32 spread over all blocks, so no
// one SM makes all the gathers) every driven neuron runs the window as if nothing were drawn for
// it: that is its state unless it is forced, and gives the steps in which it would be live (one
// bit each). The chain (D) then counts live bits, looks the draws up and cuts a neuron's bits at
// its forced spike, after which it is refractory for the rest of the window; conductances and res
// do not depend on the neuron's own spikes, so only v, refr, trace and adapt need setting again.
// Background hits on driven neurons come from the same stream: they are looked up under the chain's
// positions, the neurons that were hit run again, and if that changed any live bit the chain is
// repeated with the new ones (the steps before the first change stay right, so this ends).
// The next `need` outputs of the stream after state s into sm[0 .. need): each thread jumps to
// its run (by warp, then by lane) and takes it one generator step at a time.
__device__ __forceinline__ void fill_stream(uint32_t s, uint32_t need) {
  const uint32_t *jump = s_win.jump;
  uint32_t *sm = s_pool;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t k0 = threadIdx.x * kWinRun;
  if (warp * 32 * kWinRun >= need) return;
  uint32_t b = s;
  for (uint32_t i = 0; i < 5; i++)
    if ((warp >> i) & 1u) b = xs_apply(jump + i * 128, b);
  const uint32_t *off = jump + 5 * 128;
  uint32_t x = 0;
#pragma unroll
  for (int n = 0; n < 8; n++) x ^= off[((uint32_t)n * 16 + ((b >> (4 * n)) & 15u)) * 32 + lane];
#pragma unroll 4
  for (uint32_t k = 0; k < kWinRun; k++) {
    x = xs_next(x);
    if (k0 + k < need) sm[k0 + k] = x;
  }
}

// Draws the window may need (the host keeps it within kWinStream).
__device__ __forceinline__ uint32_t stream_need(const Trial &T, int nD, int h) {
  const uint32_t per = (uint32_t)nD + ((T.flags & kHasBg) ? (uint32_t)T.bgEvents + 2u : 0u);
  return min(per * (uint32_t)h, (uint32_t)kWinStream);
}

// A driven neuron's window without a forced spike, from state x.
struct DrivenRun {
  uint32_t live;  // steps it is live in
  int fired;
};
template <int GEN>
__device__ __forceinline__ DrivenRun driven_run(const Trial &T, const WinBrain &C, Neuron &x, List &l, int32_t i, int h,
                                                int ar, bool hit) {
  const uint32_t bg = GEN && hit ? ldcg(C.bgMask + i) : 0u;
  const float bias = (T.flags & kBiasZero) ? 0.f : ldcg(T.bias + i);
  const float thr = (T.flags & kThrZero) ? 0.f : ldcg(T.thr + i);
  const float sign = (GEN && ar >= 0) ? __ldg(T.sign + i) : 0.f;
  const float thB = __fadd_rn(__fadd_rn(T.vThresh, x.ad), thr);
  const Model K = model_of<GEN>(T);
  DrivenRun d;
  d.live = 0;
  d.fired = -1;
  for (int j = 0; j < h; j++) {
    if (!(x.r > 0)) d.live |= 1u << j;  // lif.c:50: refractory entries draw nothing
    uint32_t hits = (bg >> j) & 1u;
    if (GEN && hits && (bg >> 31)) hits += ldcg(C.bgHit + (int64_t)j * T.N + i);
    neuron_inputs<GEN>(K, x, l, j, hits, ar == j, sign);
    if (neuron_step<GEN>(K, x, bias, thr, thB)) d.fired = j;
  }
  return d;
}

template <int GEN>
__device__ __forceinline__ void driven_store(const Trial &T, int32_t i, const Neuron &x, float tr) {
  T.v[i] = x.v;
  T.gE[i] = x.ge;
  T.gI[i] = x.gi;
  T.refr[i] = x.r;
  T.trace[i] = tr;
  if (GEN) {
    T.adapt[i] = x.ad;
    T.res[i] = x.rs;
  }
}

// One brain: each warp's first tile of F is the same in every window, and its state does not depend
// on the deliveries. Its neurons and regions stay in the warp's words of the pool, and the state is
// copied there while P runs (words of 32 lanes: id, region, its end, v, gE, gI, refr, trace, adapt,
// res).
constexpr int kEarlyWords = 10;
__device__ __forceinline__ uint32_t *early_words() {
  return s_pool + kWinPool - (kWT / 32) * 32 * kEarlyWords + (threadIdx.x >> 5) * 32 * kEarlyWords + (threadIdx.x & 31);
}
static_assert((kWT / 32) * 32 * (kWinSort * 2 + kEarlyWords) <= kWinPool, "beside the sort staging");
__device__ __forceinline__ void copy_async4(uint32_t *dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void early_load(uint32_t tile, bool once) {
  const Trial &T = s_win.tr;
  const int k = (int)tile * 32 + (int)(threadIdx.x & 31);
  uint32_t *p = early_words();
  if (once) {
    const int32_t i = k < T.nDriven ? ldcg(T.driven + k) : 0;
    p[0] = (uint32_t)i;
    p[32] = __ldg(s_win.win.inOff + i);
    p[64] = __ldg(s_win.win.inOff + i + 1);
  }
  const int32_t i = (int32_t)p[0];
  copy_async4(p + 3 * 32, T.v + i);
  copy_async4(p + 4 * 32, T.gE + i);
  copy_async4(p + 5 * 32, T.gI + i);
  copy_async4(p + 6 * 32, T.refr + i);
  copy_async4(p + 7 * 32, T.trace + i);
  copy_async4(p + 8 * 32, T.adapt + i);
  copy_async4(p + 9 * 32, T.res + i);
}

// F: 32 entries of the driven list, one per lane. early: their state is in early_words().
template <int GEN>
__device__ __forceinline__ void free_warp(const WinArgs &a, const Trial &T, const WinBrain &C, WinBrain *W, int k, int nD,
                                          int h, uint2 *stage, bool early) {
  const bool on = k < nD;
  int32_t i;
  uint32_t o, o1;
  Neuron x;
  float tr;
  if (early) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    const uint32_t *p = early_words();
    i = (int32_t)p[0];
    o = p[32];
    o1 = p[64];
    x.v = __uint_as_float(p[3 * 32]);
    x.ge = __uint_as_float(p[4 * 32]);
    x.gi = __uint_as_float(p[5 * 32]);
    x.r = __uint_as_float(p[6 * 32]);
    tr = __uint_as_float(p[7 * 32]);
    x.ad = GEN ? __uint_as_float(p[8 * 32]) : 0.f;
    x.rs = GEN ? __uint_as_float(p[9 * 32]) : 1.f;
  } else {
    i = on ? ldcg(T.driven + k) : 0;
    o = __ldg(C.inOff + i);
    o1 = __ldg(C.inOff + i + 1);
    x.v = ldcg(T.v + i);
    x.ge = ldcg(T.gE + i);
    x.gi = ldcg(T.gI + i);
    x.r = ldcg(T.refr + i);
    tr = ldcg(T.trace + i);
    x.ad = GEN ? ldcg(T.adapt + i) : 0.f;
    x.rs = GEN ? ldcg(T.res + i) : 1.f;
  }
  uint32_t n = ldcg(C.wcnt + i) - o;
  const int ar = (GEN && (T.flags & kHasDep)) ? (int)ldcg(C.arr + i) - 1 : -1;
  if (!on) n = 0;
  if (n > o1 - o) {
    atomicCAS(a.err, 0, FB_EOVERFLOW);
    n = 0;
  }
  List l = make_list(C.wbuf + o, n, stage, n ? ldcg(C.wbuf + o) : make_uint2(kNone, 0u));
  if (on) {
    if (GEN) {  // the window's start, for a neuron that runs again: one row, read in one go
      float4 *row = C.dSave + 3 * k;
      row[0] = make_float4(x.v, x.ge, x.gi, x.r);
      row[1] = make_float4(x.ad, x.rs, tr, __int_as_float(ar));
      row[2] = make_float4(__uint_as_float(n), __uint_as_float(o), __uint_as_float(l.key), l.val);
    }
    if (GEN && (T.flags & kHasBg) && n > 1 && n <= (uint32_t)kWinSort)
      for (uint32_t u = 0; u < n; u++) C.wbuf[o + u] = stage[u * 32];  // in order, for the same
    const DrivenRun d = driven_run<GEN>(T, C, x, l, i, h, ar, false);
    C.dLive[k] = d.live;
    C.dFired[k] = (uint8_t)(d.fired + 1);
    driven_store<GEN>(T, i, x, trace_window(tr, T.dTr, h, d.fired, false));
    if (n) C.wcnt[i] = o;
    if (GEN && ar >= 0) C.arr[i] = 0;
  }
  __syncwarp();
  if ((threadIdx.x & 31) == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&W->fDone) : "memory");
}

// Per-entry words of a driven item, behind the draws in the block's pool (kWinPool words).
struct DrivenWords {
  uint32_t *live;          // live bits
  int32_t *id;
  uint32_t *lim;           // the largest draw that forces a spike
  uint16_t *event;         // entries that fire in the window (after the chain, in live's place)
  uint8_t *forced, *own;   // forced step or 255; 1 + the step of its own spike without one
  uint8_t *mark;           // ran again for background hits
};
__device__ __forceinline__ DrivenWords driven_words(int nD) {
  DrivenWords d;
  uint32_t *p = s_pool + kWinPool - window_entry_words(nD);
  d.live = p;
  d.id = (int32_t *)(p + nD);
  d.lim = p + 2 * nD;
  d.event = (uint16_t *)d.live;
  d.forced = (uint8_t *)(p + 3 * nD);
  d.own = d.forced + nD;
  d.mark = d.own + nD;
  return d;
}

// The chain: for each step the live entries' ranks, their draws, the forced spikes. A warp owns M
// consecutive words of 32 entries, so it publishes one count per step (a byte per four words); the
// warps in use meet at one named barrier a step and add up the 16 V bytes (dp4a: one shared load and
// no exchange between lanes).
template <int M, int V, bool BG>
__device__ __noinline__ void draw_chain(int nD, int h) {
  DrivenShared &sh = s_win.dr;
  const DrivenWords E = driven_words(nD);
  const uint32_t *sm = s_pool;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, lt = (1u << lane) - 1u;
  const uint32_t nW = max(1u, (uint32_t)(nD + 32 * M - 1) / (32 * M));
  if (warp >= nW) return;
  uint32_t mask[M], lim[M], f[M];
#pragma unroll
  for (int m = 0; m < M; m++) {
    const int k = (int)(warp * M + m) * 32 + (int)lane;
    mask[m] = k < nD ? E.live[k] : 0u;
    lim[m] = k < nD ? E.lim[k] : 0u;
    f[m] = 255u;
  }
  constexpr int kBytes = M > 4 ? 2 : 1;  // four words' live entries per byte
  uint32_t below[4 * V];                 // a one in the bytes of the warps before this one
#pragma unroll
  for (int q = 0; q < 4 * V; q++) {
    const int n = min(max((int)warp * kBytes - 4 * q, 0), 4);
    below[q] = n == 0 ? 0u : 0x01010101u >> (32 - 8 * n);
  }
  uint32_t base = 0;
  for (int j = 0; j < h; j++) {
    uint4 *cnt = sh.cnt[j & 1];
    if (BG) base += sh.nbg[j];
    uint32_t live[M], mine[2] = {0, 0};
#pragma unroll
    for (int m = 0; m < M; m++) {
      live[m] = __ballot_sync(0xffffffffu, mask[m] & 1u);
      mine[m / 4] += (uint32_t)__popc(live[m]);
    }
    if (lane < kBytes) ((uint8_t *)cnt)[warp * kBytes + lane] = (uint8_t)(lane ? mine[1] : mine[0]);
    asm volatile("bar.sync 2, %0;" ::"r"(nW * 32) : "memory");
    uint32_t at = base;  // the counts of the warps before this one, and of all
    if (BG && warp == 0 && lane == 0) sh.base[j] = base;
#pragma unroll
    for (int v = 0; v < V; v++) {
      const uint4 c = cnt[v];
      at = __dp4a(c.x, below[4 * v], at);
      at = __dp4a(c.y, below[4 * v + 1], at);
      at = __dp4a(c.z, below[4 * v + 2], at);
      at = __dp4a(c.w, below[4 * v + 3], at);
      base = __dp4a(c.x, 0x01010101u, base);
      base = __dp4a(c.y, 0x01010101u, base);
      base = __dp4a(c.z, 0x01010101u, base);
      base = __dp4a(c.w, 0x01010101u, base);
    }
    uint32_t x[M];  // every lane's next draw, whether it takes it or not: the loads overlap
#pragma unroll
    for (int m = 0; m < M; m++) {
      x[m] = sm[at + (uint32_t)__popc(live[m] & lt)];
      at += (uint32_t)__popc(live[m]);
    }
#pragma unroll
    for (int m = 0; m < M; m++) {
      const bool hit = (mask[m] & 1u) && x[m] <= lim[m];
      f[m] = hit ? (uint32_t)j : f[m];
      mask[m] = hit ? 0u : mask[m] >> 1;
    }
  }
  if (warp == 0 && lane == 0) sh.base[h] = base;
#pragma unroll
  for (int m = 0; m < M; m++) {
    const int k = (int)(warp * M + m) * 32 + (int)lane;
    if (k < nD) E.forced[k] = (uint8_t)f[m];
  }
}

// A driven neuron that background events hit, run again from its state at the window's start.
template <int GEN>
__device__ __noinline__ uint32_t driven_again(const Trial &T, const WinBrain &C, int k, int32_t i, int h, uint8_t &own) {
  const float4 *row = C.dSave + 3 * k;
  const float4 r0 = ldcg(row), r1 = ldcg(row + 1), r2 = ldcg(row + 2);
  Neuron x;
  x.v = r0.x;
  x.ge = r0.y;
  x.gi = r0.z;
  x.r = r0.w;
  x.ad = r1.x;
  x.rs = r1.y;
  const float tr = r1.z;
  const int ar = __float_as_int(r1.w);
  const uint32_t n = __float_as_uint(r2.x);
  List l;  // in key order already
  l.p = C.wbuf + __float_as_uint(r2.y);
  l.stride = 1;
  l.left = n ? n - 1 : 0;
  l.key = __float_as_uint(r2.z);
  l.val = r2.w;
  const DrivenRun d = driven_run<GEN>(T, C, x, l, i, h, ar, true);
  own = (uint8_t)(d.fired + 1);
  driven_store<GEN>(T, i, x, trace_window(tr, T.dTr, h, d.fired, false));
  return d.live;
}

// The window's background draws under the chain's positions: f(step, target).
template <typename F>
__device__ __forceinline__ void each_hit(int h, uint32_t N, F f) {
  const DrivenShared &sh = s_win.dr;
  uint32_t total = 0;
  for (int j = 0; j < h; j++) total += sh.nbg[j];
  for (uint32_t t = threadIdx.x; t < total; t += kWT) {
    int j = 0;
    uint32_t d = t;
    while (d >= sh.nbg[j]) d -= sh.nbg[j++];
    f(j, s_pool[sh.base[j] - sh.nbg[j] + d] % N);
  }
}

constexpr int kChainMax = kWinDriven / kWT;  // words per warp when every warp is in use
static_assert(kChainMax <= 8 && kWT / 32 * (kChainMax > 4 ? 2 : 1) <= 32, "the counts fit in 32 bytes");

// D: the chain and the background hits. sm: the pool, the window's draws first.
template <int GEN>
__device__ __noinline__ void driven_window(int b, int w, int nD, int h, bool keep) {
  const WinArgs &a = s_win.a;
  const Trial &T = s_win.ctx.tr[b];
  const WinBrain &C = s_win.ctx.win[b];
  WinBrain *W = a.win + b;
  DrivenShared &sh = s_win.dr;
  const int tid = threadIdx.x, N = T.N;
  const bool bg = GEN && (T.flags & kHasBg);
  const DrivenWords E = driven_words(nD);
  float acc = ldcg(&W->bgAcc);
  // a block that only serves one list keeps these words from window to window
  if (!(keep && w > 0))
#pragma unroll 4
  for (int k = tid; k < nD; k += kWT) {
    const int32_t i = ldcg(T.driven + k);
    E.id[k] = i;
    // x <= lim for u < p: u = (x >> 8) 2^-24 < p = f32(drive dtS) iff x >> 8 is below p 2^24 rounded
    // up; a draw x is never 0
    const float p = __fmul_rn(ldcg(T.drive + i), T.dtS);
    const uint32_t t = p >= 1.f ? 1u << 24 : (uint32_t)ceilf(p * 16777216.f);
    E.lim[k] = t ? (t << 8) - 1u : 0u;
  }
  if (tid == 0) {
    for (int j = 0; j < h; j++) {  // lif.c:46-47 (f32)
      uint32_t n = 0;
      if (bg) {
        acc = __fadd_rn(acc, T.bgEvents);
        const int32_t nb = (int32_t)acc;
        acc = __fsub_rn(acc, (float)nb);
        n = (uint32_t)nb;
      }
      sh.nbg[j] = n;
    }
    sh.acc = acc;
    sh.events = 0;
    sh.cnt[0][0] = sh.cnt[0][1] = sh.cnt[1][0] = sh.cnt[1][1] = make_uint4(0, 0, 0, 0);
    const uint32_t want = (uint32_t)(nD + 31) / 32;  // the brain's tiles of F
    if (ld_acquire(&W->fDone) != want) {
      const uint64_t q0 = global_ns();
      uint32_t it = 0;
      while (ld_acquire(&W->fDone) != want)
        if (win_timeout(a, q0, it)) break;
    }
    W->fDone = 0;
  }
  __syncthreads();
#pragma unroll 4
  for (int k = tid; k < nD; k += kWT) {
    E.live[k] = ldcg(C.dLive + k);
    E.own[k] = ldcg(C.dFired + k);
    if (bg) E.mark[k] = 0;
  }
  __syncthreads();
  win_lap(a, 2, -1, sh.tp);
  for (int it = 0; it <= h; it++) {
    if (nD <= 256) draw_chain<1, 1, GEN != 0>(nD, h);
    else if (nD <= 1024) draw_chain<2, 1, GEN != 0>(nD, h);
    else if (nD <= 2048) draw_chain<4, 1, GEN != 0>(nD, h);
    else draw_chain<kChainMax, 2, GEN != 0>(nD, h);
    if (tid == 0) sh.changed = 0;
    __syncthreads();
    if (!bg) break;
    each_hit(h, (uint32_t)N, [&](int j, uint32_t q) {  // lif.c:48
      const int32_t k = nD ? ldcg(C.drvPos + q) : -1;
      if ((atomicOr(C.bgMask + q, 1u << j) >> j) & 1u) {  // the step's second hit and further ones
        atomicAdd(C.bgHit + (int64_t)j * N + q, 1u);
        atomicOr(C.bgMask + q, 1u << 31);
      }
      if (k >= 0) E.mark[k] = 1;
    });
    __syncthreads();
    for (int k = tid; k < nD; k += kWT)
      if (E.mark[k]) {
        const uint32_t live = driven_again<GEN>(T, C, k, E.id[k], h, E.own[k]);
        if (live != E.live[k]) {
          E.live[k] = live;
          sh.changed = 1;
        }
      }
    __syncthreads();
    const bool again = sh.changed != 0;
    if (again)  // the positions move: these hits are taken back
      each_hit(h, (uint32_t)N, [&](int j, uint32_t q) {
        C.bgHit[(int64_t)j * N + q] = 0;
        C.bgMask[q] = 0;
      });
    __syncthreads();
    if (!again) break;
  }
  win_lap(a, 3, -1, sh.tp);
}

// D, the rest: the generator's state after the window, the spikes and the forced neurons' state.
template <int GEN>
__device__ __noinline__ void driven_finish(int b, int nD, int h, int t0, int steps, uint64_t g0) {
  const WinArgs &a = s_win.a;
  const Trial &T = s_win.ctx.tr[b];
  const WinBrain &C = s_win.ctx.win[b];
  Trial *G = a.trials + b;
  WinBrain *W = a.win + b;
  DrivenShared &sh = s_win.dr;
  const uint32_t *sm = s_pool;
  const int tid = threadIdx.x, N = T.N;
  const bool bg = GEN && (T.flags & kHasBg);
  const DrivenWords E = driven_words(nD);
  if (tid == 0) {
    const float acc = sh.acc;
    const uint32_t used = sh.base[h], s1 = used ? sm[used - 1] : ldcg(&W->rng);
    W->rng = s1;
    W->bgAcc = acc;
    if (t0 + h >= steps) {
      const uint64_t e = g0 + (uint64_t)h;
      G->rngP[e & 1] = s1;
      G->bgAccP[e & 1] = acc;
      const int ns = T.nslots, head = (int)((ldcg(&G->head) + (int64_t)steps) % ns);
      G->head = head;
      G->stepsDone = (int64_t)e;
      G->lastSlot = (head + ns - 2) % ns;  // the last step's list arrives last
    }
  }
  const uint32_t lane = tid & 31u;
  for (int k0 = 0; k0 < nD; k0 += kWT) {  // the entries that fire, gathered so that one pass serves them
    const int k = k0 + tid;
    const uint32_t on = __ballot_sync(0xffffffffu, k < nD && (E.forced[k] != 255 || E.own[k]));
    if (on) {
      uint32_t at = 0;
      if (lane == 0) at = atomicAdd(&sh.events, (uint32_t)__popc(on));
      at = __shfl_sync(0xffffffffu, at, 0) + (uint32_t)__popc(on & ((1u << lane) - 1u));
      if ((on >> lane) & 1u) E.event[at] = (uint16_t)k;
    }
    if (bg && k < nD && E.mark[k]) {
      if (ldcg(C.bgMask + E.id[k]) >> 31)
        for (int j = 0; j < h; j++) C.bgHit[(int64_t)j * N + E.id[k]] = 0;
      C.bgMask[E.id[k]] = 0;
    }
  }
  __syncthreads();
  const int nE = (int)sh.events;
  for (int e0 = 0; e0 < nE; e0 += kWT) {
    const bool on = e0 + tid < nE;
    const int k = on ? E.event[e0 + tid] : 0;
    const int32_t i = E.id[k];
    const int f = on && E.forced[k] != 255 ? E.forced[k] : -1;
    log_append(T, C, W, G, !on ? -1 : f >= 0 ? f : (int)E.own[k] - 1, g0, t0, steps, i,
               f >= 0 ? (uint32_t)k : (uint32_t)(nD + i));
    if (!on) continue;
    atomicAdd(T.spikeCount + i, 1u);
    if (f >= 0) {  // lif.c:51-52, then refractory to the window's end (lif.c:61-64)
      float r = __fadd_rn(T.tRef, T.dt), ad = GEN ? ldcg(&C.dSave[3 * k + 1].x) : 0.f;
      for (int j = f; j < h; j++) r = r > 0 ? __fsub_rn(r, T.dt) : r;
      T.v[i] = T.vReset;
      T.refr[i] = r;
      T.trace[i] = trace_window(1.f, T.dTr, h, f, true);
      if (GEN) {
        for (int j = 0; j < h; j++) {
          if (j == f) ad = __fadd_rn(ad, T.adaptInc);
          ad = __fmul_rn(ad, T.dA);
        }
        T.adapt[i] = ad;
      }
    }
  }
}

// ---- the kernel --------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t wprefix_sum(const WinArgs &a, const WinCtx &c, uint32_t *scan, uint32_t mine, int b0,
                                                uint32_t carry) {
  const int b = b0 + (int)threadIdx.x;
  uint32_t tot;
  const uint32_t ex = block_exclusive_scan(b < a.B ? mine : 0u, &tot, scan);
  if (b < a.B) c.pre[b] = carry + ex;
  return carry + tot;
}
// Exclusive prefix of f(b) over the brains into c.pre; returns the sum. One brain: f(0) alone (pre
// stays {0, all ones}, under which every number is brain 0's).
template <typename F>
__device__ __forceinline__ uint32_t brain_prefix(const WinArgs &a, const WinCtx &c, uint32_t *scan, F f) {
  if (a.B == 1) return f(0);
  uint32_t carry = 0;
  for (int b0 = 0; b0 < a.B; b0 += kWT) {
    const int b = b0 + (int)threadIdx.x;
    carry = wprefix_sum(a, c, scan, b < a.B ? f(b) : 0u, b0, carry);
  }
  if (threadIdx.x == 0) c.pre[a.B] = carry;
  __syncthreads();
  return carry;
}
__device__ __forceinline__ int driven_count(const WinArgs &a, const WinCtx &c, int b) {
  return a.B == 1 ? c.tr[0].nDriven : ldcg(&a.trials[b].nDriven);
}

// ---- P: the log's spikes that arrive in the window ----------------------------------------------
__device__ __noinline__ void deliver(int w, uint32_t off, uint32_t nb) {
  const WinArgs &a = s_win.a;
  const WinCtx &c = s_win.ctx;
  WinShared &sh = s_win;
  const int tid = threadIdx.x, warp = tid >> 5;
  const uint32_t lane = tid & 31u;
  // The log entries from the window that emitted step t0 - D on (those of other steps are skipped).
  // Blocks take every nb-th entry, so one brain's first entries can be loaded before their number is
  // known.
  uint32_t total;
  uint4 early = make_uint4(0, 0, 0, 0);
  if (a.B == 1) {
    const int64_t e = c.done[0] + c.t0(0, w) - c.win[0].D;
    const uint32_t lo = ldcg(&a.win->ls[(uint64_t)e & (kWinRing - 1)]);
    if (tid < kWinSpikes / 8) early = ldcg(c.win[0].log + ((lo + off + nb * tid) & c.win[0].logMask));
    total = ldcg(&a.win->logTop) - lo;
    if (total > c.win[0].logMask + 1) {
      atomicCAS(a.err, 0, FB_EOVERFLOW);  // more spikes than the refractory time allows
      total = c.win[0].logMask + 1;
    }
  } else {
    total = brain_prefix(a, c, sh.scan, [&](int b) -> uint32_t {
      if (c.h(b, w) <= 0) return 0u;
      const WinBrain *W = a.win + b;
      const int64_t e = c.done[b] + c.t0(b, w) - c.win[b].D;
      const uint32_t n = ldcg(&W->logTop) - ldcg(&W->ls[(uint64_t)e & (kWinRing - 1)]);
      if (n > c.win[b].logMask + 1) atomicCAS(a.err, 0, FB_EOVERFLOW);
      return min(n, c.win[b].logMask + 1);
    });
  }
  const uint32_t mine = total > off ? (total - off + nb - 1) / nb : 0u;
  for (uint32_t c0 = 0; c0 < mine; c0 += kWinSpikes) {
    const uint32_t m = min(mine - c0, (uint32_t)kWinSpikes);
    uint32_t nch = 0;
    if ((uint32_t)tid < m) {
      SpikeRec r;
      r.lo = r.hi = 0;
      r.key = r.id = 0;
      const uint32_t x = off + nb * (c0 + tid);
      r.b = a.B == 1 ? 0 : find_brain(c.pre, a.B, x);
      const WinBrain *W = a.win + r.b;
      const WinBrain &C = c.win[r.b];
      const Trial &T = c.tr[r.b];
      const int64_t g0 = c.done[r.b] + c.t0(r.b, w);
      uint4 s = early;
      if (a.B != 1 || c0 != 0 || tid >= kWinSpikes / 8) {
        const uint32_t at = ldcg(&W->ls[(uint64_t)(g0 - C.D) & (kWinRing - 1)]) + (a.B == 1 ? x : x - c.pre[r.b]);
        s = ldcg(C.log + (at & C.logMask));
      }
      const uint32_t id = s.x & 0xffffffu;
      int j = (int)(((s.x >> 24) + (uint32_t)C.D - (uint32_t)g0) & 255u);
      FB_GUARD(a, id < (uint32_t)T.N && (int64_t)s.w <= T.E, 21, id, s.y, j = 256);
      if (j < c.h(r.b, w)) {
        r.id = id;
        if (T.flags & kHasDep) C.arr[id] = (uint8_t)(j + 1);
        r.lo = s.z;
        r.hi = s.w;
        r.key = ((uint32_t)j << 27) | (s.y << 3);
        nch = (r.hi - r.lo + 31) / 32;
      }
      sh.rec[tid] = r;
    }
    uint32_t chunks;
    const uint32_t ex = block_exclusive_scan(nch, &chunks, sh.scan);
    if ((uint32_t)tid < m) sh.pre[tid] = ex;
    if (tid == 0) sh.pre[m] = chunks;
    __syncthreads();
    for (uint32_t q0 = warp; q0 < chunks; q0 += kWT / 32) {
      const uint32_t k = (uint32_t)find_brain(sh.pre, (int)m, q0);
      const SpikeRec r = sh.rec[k];
      const uint32_t e = r.lo + (q0 - sh.pre[k]) * 32 + lane;
      if (e < r.hi) {  // the amplitude's loads and the edge's in one round trip
        const Trial &T = c.tr[r.b];
        const WinBrain &C = c.win[r.b];
        const uint32_t q = __ldg(T.indices + e);
        const float we = __ldg(T.W + e), sign = __ldg(T.sign + r.id);
        float rs = 1.f;
        if (!(T.flags & kResRest)) {  // res at the arrival step (at most one arrival per window)
          rs = ldcg(T.res + r.id);
          for (uint32_t k = 0; k < r.key >> 27; k++) rs = __fadd_rn(rs, __fmul_rn(__fsub_rn(1.f, rs), T.kRec));
        }
        const float amp = __fmul_rn(sign, rs);  // lif.c:37
        if (amp == 0.f) continue;
        const float wt = __fmul_rn(we, amp);  // lif.c:41-42, one rounding
        const uint32_t key = r.key | (amp > 0 ? 0u : 1u) | (T.dup ? (uint32_t)__ldg(T.dup + e) << 1 : 0u);
        const uint32_t pos = atomicAdd(C.wcnt + q, 1u);  // the counter starts at the target's region
        if ((int64_t)pos < T.E) C.wbuf[pos] = make_uint2(key, __float_as_uint(wt));
      }
    }
    __syncthreads();
  }
}

// F: this block's tiles of the driven lists.
__device__ __noinline__ void free_tiles(int w, uint32_t off, uint32_t nb) {
  const WinArgs &a = s_win.a;
  const WinCtx &c = s_win.ctx;
  WinShared &sh = s_win;
  uint2 *stage = sort_stage();
  const uint32_t total = brain_prefix(a, c, sh.scan, [&](int b) -> uint32_t {
    return c.h(b, w) > 0 ? (uint32_t)(driven_count(a, c, b) + 31) / 32 : 0u;
  });
  for (uint32_t t = off + nb * (threadIdx.x >> 5); t < total; t += nb * (kWT / 32)) {
    const int b = find_brain(c.pre, a.B, t);
    const Trial &T = c.tr[b];
    const int k = (int)(t - c.pre[b]) * 32 + (int)(threadIdx.x & 31), nD = driven_count(a, c, b);
    const bool early = a.B == 1 && t == off + nb * (threadIdx.x >> 5);
    if (plain_brain(T)) free_warp<0>(a, T, c.win[b], a.win + b, k, nD, c.h(b, w), stage, early);
    else free_warp<1>(a, T, c.win[b], a.win + b, k, nD, c.h(b, w), stage, early);
  }
  __syncthreads();
}

__global__ void __launch_bounds__(kWT, 1) window_kernel(const WinArgs args) {
  WinShared &sh = s_win;
  int64_t *sDone = (int64_t *)(s_pool + kWinPool);
  int32_t *sSteps = (int32_t *)(sDone + args.B);
  uint32_t *sPre = (uint32_t *)(sSteps + args.B);  // [B + 1]
  const int tid = threadIdx.x;
  for (int k = tid; k < kWinJumpWords; k += kWT) sh.jump[k] = args.jump[k];
  if (args.B == 1) {
    const uint32_t *src = (const uint32_t *)args.trials;
    for (int k = tid; k < (int)(sizeof(Trial) / 4); k += kWT) ((uint32_t *)&sh.tr)[k] = ldcg(src + k);
    const uint32_t *win = (const uint32_t *)args.win;
    for (int k = tid; k < (int)(sizeof(WinBrain) / 4); k += kWT) ((uint32_t *)&sh.win)[k] = ldcg(win + k);
  }
  if (tid < 2) sPre[tid] = tid ? 0xffffffffu : 0u;
  for (int b = tid; b < args.B; b += kWT) {
    sDone[b] = ldcg(&args.trials[b].stepsDone);
    sSteps[b] = args.steps[b];
  }
  if (tid == 0) {
    sh.a = args;
    sh.ctx = WinCtx{args.B == 1 ? &sh.tr : args.trials, args.B == 1 ? &sh.win : args.win, sDone, sSteps, sPre};
    sh.dr.tp = global_ns();
  }
  __syncthreads();
  const WinArgs &a = sh.a;
  const WinCtx &c = sh.ctx;
  uint32_t target = args.barBase;  // of the next grid barrier
  auto lap = [&](int k0, int k1) { win_lap(a, k0, k1, sh.dr.tp); };
  const int own = (int)blockIdx.x;
  const int nServe = args.dedicated ? args.B : 0;  // blocks that leave P, F and U to the others
  for (int w = 0; w < args.nWin; w++) {
    // ---------------- P ----------------
    for (int b = own; b < args.B; b += gridDim.x) {  // the brains whose driven lists this block serves
      const int t0 = c.t0(b, w), h = c.h(b, w);
      if (h <= 0) continue;
      WinBrain *W = args.win + b;
      if (tid < h) W->ls[(c.done[b] + t0 + tid) & (kWinRing - 1)] = ldcg(&W->logTop);
      if (tid == 0) {
        if (w == 0) {  // the header's generator state
          W->rng = ldcg(&args.trials[b].rngP[c.done[b] & 1]);
          W->bgAcc = ldcg(&args.trials[b].bgAccP[c.done[b] & 1]);
        }
        if (t0 + h >= c.steps[b]) args.trials[b].nFired = 0;
      }
      if (kWT > 512 && tid == kWT - 1) make_brain(*(WarpBrain *)(args.brains + (size_t)b * kWarpBrainBytes), a, c, w, b);
      if (own < nServe) {  // one brain, and P left to the others: its draws now
        __syncthreads();
        fill_stream(ldcg(&W->rng), stream_need(c.tr[b], driven_count(a, c, b), h));
      }
    }
    if (kWT <= 512 && tid == kWT - 1) make_brain(sh.wb[0][0], a, c, w, 0);
    if (blockIdx.x == gridDim.x - 1 && tid == 0) args.uNext[w & 1] = 0;
    if (own >= nServe) {
      if (args.B == 1) {
        const uint32_t tile = (own - nServe) + (gridDim.x - nServe) * (tid >> 5);
        if (tile * 32 < (uint32_t)sh.tr.nDriven) early_load(tile, w == 0);
      }
      deliver(w, own - nServe, gridDim.x - nServe);
    }
    lap(0, 6);
    if (!win_sync(a, target += gridDim.x)) return;
    lap(1, 7);
    // ---------------- F ----------------
    if (own >= nServe) free_tiles(w, own - nServe, gridDim.x - nServe);
    // ---------------- D ----------------
    if (args.anyBg) target += gridDim.x;  // the barrier between the background hits and U
    bool met = false;
    for (int b = own; b < args.B; b += gridDim.x) {
      const int t0 = c.t0(b, w), h = c.h(b, w);
      if (h <= 0) continue;
      if (args.tripStep >= t0 && args.tripStep < t0 + h && b == 0) {  // test hook: a wait nothing ends
        __shared__ int never;
        if (tid == 0) {
          never = 0;
          const uint64_t q0 = global_ns();
          uint32_t it = 0;
          while (*(volatile int *)&never == 0)
            if (win_timeout(a, q0, it)) break;
        }
        __syncthreads();
      }
      const Trial &T = c.tr[b];
      WinBrain *W = args.win + b;
      const int nD = driven_count(a, c, b);
      const uint64_t g0 = (uint64_t)(c.done[b] + t0);
      if (own >= nServe) {
        fill_stream(ldcg(&W->rng), stream_need(T, nD, h));
        __syncthreads();
      }
      const bool plain = plain_brain(T);
      if (plain) driven_window<0>(b, w, nD, h, own < nServe);
      else driven_window<1>(b, w, nD, h, own < nServe);
      // U waits for the background hits only, so a block's last driven list finishes beside it
      if (args.anyBg && b + (int)gridDim.x >= args.B) {
        if (!win_sync(a, target)) return;
        met = true;
        lap(5, 9);
      }
      if (plain) driven_finish<0>(b, nD, h, t0, c.steps[b], g0);
      else driven_finish<1>(b, nD, h, t0, c.steps[b], g0);
      __syncthreads();
      lap(4, -1);
    }
    lap(-1, 8);
    const uint32_t meet = args.anyBg && !met ? target : 0u;
    // ---------------- U ----------------
    if (own < nServe) {
      if (meet && !win_sync(a, meet)) return;
    } else {
      const uint32_t total = brain_prefix(a, c, sh.scan, [&](int b) -> uint32_t {
        return c.h(b, w) > 0 ? (uint32_t)(c.tr[b].N + 31) / 32 : 0u;
      });
      const uint32_t nWarps = (gridDim.x - nServe) * (kWT / 32), first = (own - nServe) * (kWT / 32) + (tid >> 5);
      if (!(args.allPlain ? update_tiles<0>(w, total, first, nWarps, meet)
                          : update_tiles<1>(w, total, first, nWarps, meet)))
        return;
    }
    lap(-1, 10);
    if (w + 1 < args.nWin && !win_sync(a, target += gridDim.x)) return;
    lap(5, 11);
  }
}

}  // namespace FB_WINDOW_NAME

#ifdef FB_WINDOW_IS_NARROW
const void *window_kernel_narrow() { return (const void *)narrow::window_kernel; }
}  // namespace fb
#else
const void *window_kernel_wide() { return (const void *)wide::window_kernel; }

extern __shared__ __align__(16) uint32_t s_sort[];

// ---- the log and the ring ----------------------------------------------------------------------

// The log's spikes of step e, in rank order, to out[0 .. ) (at most cap entries are stored);
// returns their number. A thread each: ranks are counted against each other; more: marked in a bitmap,
// 32 kSortWords at a time.
constexpr int kSortThreads = 512;
constexpr int kSortWords = 8192;
__device__ uint32_t sorted_list(const Trial &T, const WinBrain *W, int64_t e, int32_t *out, int64_t cap, uint32_t *bits,
                                uint32_t *scan, uint32_t *s_n) {
  const uint32_t tid = threadIdx.x;
  const uint32_t lo = W->ls[(uint64_t)e & (kWinRing - 1)], hi = W->logTop, e8 = (uint32_t)e & 255u;
  if (e < 0) return 0;
  if (tid == 0) *s_n = 0;
  __syncthreads();
  uint2 *few = (uint2 *)bits;  // {rank, id} of the first kSortThreads
  for (uint32_t k = lo + tid; k - lo < hi - lo; k += kSortThreads) {
    const uint4 s = W->log[k & W->logMask];
    if ((s.x >> 24) != e8) continue;
    const uint32_t at = atomicAdd(s_n, 1u);
    if (at < kSortThreads) few[at] = make_uint2(s.y, s.x & 0xffffffu);
  }
  __syncthreads();
  const uint32_t n = *s_n;
  if (n <= kSortThreads) {
    const uint2 s = tid < n ? few[tid] : make_uint2(0u, 0u);
    uint32_t at = 0;
    for (uint32_t k = 0; k < n; k++) at += few[k].x < s.x;
    if (tid < n && (int64_t)at < cap) out[at] = (int32_t)s.y;
    __syncthreads();
    return n;
  }
  uint32_t done = 0;
  constexpr uint32_t kPer = kSortWords / kSortThreads;
  for (uint32_t r0 = 0; done < n && r0 < 2u * (uint32_t)T.N; r0 += kSortWords * 32u) {
    for (uint32_t k = tid; k < kSortWords; k += kSortThreads) bits[k] = 0;
    __syncthreads();
    for (uint32_t k = lo + tid; k - lo < hi - lo; k += kSortThreads) {
      const uint4 s = W->log[k & W->logMask];
      const uint32_t r = s.y - r0;
      if ((s.x >> 24) == e8 && r < kSortWords * 32u) atomicOr(bits + r / 32, 1u << (r & 31));
    }
    __syncthreads();
    uint32_t c = 0;
    for (uint32_t k = 0; k < kPer; k++) c += __popc(bits[tid * kPer + k]);
    uint32_t tot;
    const uint32_t ex = block_exclusive_scan(c, &tot, scan);
    uint32_t *pre = bits + kSortWords;  // per thread run
    pre[tid] = ex;
    __syncthreads();
    for (uint32_t k = lo + tid; k - lo < hi - lo; k += kSortThreads) {
      const uint4 s = W->log[k & W->logMask];
      const uint32_t r = s.y - r0;
      if ((s.x >> 24) != e8 || r >= kSortWords * 32u) continue;
      const uint32_t wd = r / 32, run = wd / kPer;
      uint32_t at = done + pre[run] + __popc(bits[wd] & ((1u << (r & 31)) - 1u));
      for (uint32_t k2 = run * kPer; k2 < wd; k2++) at += __popc(bits[k2]);
      if ((int64_t)at < cap) out[at] = (int32_t)(s.x & 0xffffffu);
    }
    done += tot;
    __syncthreads();
  }
  return n;
}

__global__ void __launch_bounds__(kSortThreads) log_export_kernel(Trial *trials, WinBrain *win, int b0, int lastOnly) {
  uint32_t *bits = s_sort;
  __shared__ uint32_t scan[33], s_n;
  Trial *G = trials + b0 + blockIdx.y;
  const WinBrain *W = win + b0 + blockIdx.y;
  const Trial &T = *G;
  const int D = W->D, j = lastOnly ? D - 1 : (int)blockIdx.x;
  if (j >= D) return;
  const int slot = (T.head + j) % T.nslots;
  const uint32_t n = sorted_list(T, W, T.stepsDone + j - D, T.ring + (int64_t)slot * T.N, T.N, bits, scan, &s_n);
  if (threadIdx.x == 0) {
    T.ringCount[slot] = (int32_t)n;
    if (j == D - 1 && !lastOnly) T.ringCount[(T.head + D) % T.nslots] = 0;  // delivered (lif.c:44)
  }
}

// One block per slot in flight and brain; the log starts over. Two steps and one step in turn, 20,000
// neurons: 120 us a pair with one block for all slots of a brain and bitmaps for every list, 110 now.
__global__ void __launch_bounds__(256) log_import_kernel(const Trial *trials, WinBrain *win) {
  __shared__ uint32_t s_top, s_end;
  const Trial &T = trials[blockIdx.y];
  WinBrain *W = win + blockIdx.y;
  const int D = W->D, j = (int)blockIdx.x;  // D <= 32
  if (j >= D) return;
  if (threadIdx.x < 32) {
    const int k = (int)threadIdx.x;
    const uint32_t n = k < D ? (uint32_t)T.ringCount[(T.head + k) % T.nslots] : 0u;
    const uint32_t before = __reduce_add_sync(0xffffffffu, k < j ? n : 0u), own = __shfl_sync(0xffffffffu, n, j);
    if (k == 0) {
      s_top = before;
      s_end = before + own;
    }
  }
  __syncthreads();
  const uint32_t top = s_top, n = s_end - top;
  const int64_t e = T.stepsDone + j - D;
  const int32_t *list = T.ring + (int64_t)((T.head + j) % T.nslots) * T.N;
  for (uint32_t k = threadIdx.x; k < n; k += blockDim.x) {
    const int32_t i = list[k];
    W->log[(top + k) & W->logMask] = make_uint4((uint32_t)i | (((uint32_t)e & 255u) << 24), k, T.indptr[i], T.indptr[i + 1]);
  }
  if (threadIdx.x == 0) {
    W->ls[(uint64_t)e & (kWinRing - 1)] = top;
    if (j == D - 1) W->logTop = top + n;
  }
}

__global__ void log_clear_kernel(WinBrain *win, int b0) {
  WinBrain *W = win + b0 + blockIdx.x;
  W->ls[threadIdx.x] = W->logTop;
}

// One block: the fired counts and lists of the last n steps of brain 0, after the step record so far.
__global__ void __launch_bounds__(kSortThreads) log_record_kernel(Trial *G, const WinBrain *W, int n) {
  uint32_t *bits = s_sort;
  __shared__ uint32_t scan[33], s_n;
  const Trial &T = *G;
  int64_t len = T.logRasterLen[(T.stepsDone - n) & 1];
  for (int k = n; k > 0; k--) {
    const int64_t e = T.stepsDone - k;
    const int64_t room = T.logRaster && len < T.logRasterCap ? T.logRasterCap - len : 0;
    const uint32_t m = sorted_list(T, W, e, T.logRaster + (room ? len : 0), room, bits, scan, &s_n);
    __syncthreads();
    const int64_t row = e - T.logStart;
    if (threadIdx.x == 0) {
      if (T.logCount && row >= 0 && row < T.logCap) T.logCount[row] = (int32_t)m;
    }
    len += m;
  }
  if (threadIdx.x == 0) G->logRasterLen[T.stepsDone & 1] = len;
}

__global__ void in_degree_kernel(const uint32_t *indices, int64_t E, uint32_t *off) {
  for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < E; j += (int64_t)gridDim.x * blockDim.x)
    atomicAdd(off + indices[j], 1u);
}
__global__ void __launch_bounds__(1024) exclusive_prefix_kernel(uint32_t *off, int32_t n) {  // n counts -> n + 1 offsets
  __shared__ uint32_t scan[33];
  uint32_t carry = 0;
  for (int32_t k0 = 0; k0 <= n; k0 += 1024) {
    const int32_t k = k0 + threadIdx.x;
    uint32_t tot;
    const uint32_t ex = block_exclusive_scan(k < n ? off[k] : 0u, &tot, scan);
    if (k <= n) off[k] = carry + ex;
    carry += tot;
  }
}
// Places in the driven lists: the entries of the list before out, the present ones in. One block per brain
// and one launch; clearing every neuron's place first took a second one (1,501 neurons, drives switched on
// and off and two steps: 76 us with both, 72 now).
__global__ void __launch_bounds__(1024) driven_pos_kernel(const Trial *trials, WinBrain *win) {
  const Trial &T = trials[blockIdx.x];
  WinBrain &W = win[blockIdx.x];
  const int was = W.nPlaced, n = min(T.nDriven, kWinDriven);
  for (int k = threadIdx.x; k < was; k += blockDim.x) W.drvPos[W.placed[k]] = -1;
  __syncthreads();
  for (int k = threadIdx.x; k < n; k += blockDim.x) {
    const int32_t i = T.driven[k];
    W.drvPos[i] = k;
    W.placed[k] = i;
  }
  if (threadIdx.x == 0) W.nPlaced = n;
}

// ---- launch glue ---------------------------------------------------------------------------------
size_t window_smem_bytes(int B) {
  return (size_t)kWinPool * 4 + (size_t)B * (8 + 4 + 4) + 16;
}

void window_jump_tables(int threads, uint32_t *tab) {
  const int kWinRun = window_run(threads);
  uint32_t one[32], m[32], p[32];  // columns of M, of M^run, of the power at hand
  for (int b = 0; b < 32; b++) {
    uint32_t x = 1u << b;
    x ^= x << 13;
    x ^= x >> 17;
    x ^= x << 5;
    one[b] = x;
    m[b] = 1u << b;
  }
  auto apply = [](const uint32_t *c, uint32_t x) {
    uint32_t y = 0;
    for (int b = 0; b < 32; b++)
      if (x >> b & 1u) y ^= c[b];
    return y;
  };
  for (int k = 0; k < kWinRun; k++)
    for (int b = 0; b < 32; b++) m[b] = apply(one, m[b]);
  for (int b = 0; b < 32; b++) p[b] = 1u << b;
  uint32_t *lane = tab + 5 * 128;
  for (int l = 0; l < 32; l++) {
    for (int n = 0; n < 8; n++)
      for (uint32_t v = 0; v < 16; v++) lane[(n * 16 + v) * 32 + l] = apply(p, v << (4 * n));
    for (int b = 0; b < 32; b++) p[b] = apply(m, p[b]);
  }
  for (int i = 0; i < 5; i++) {  // p = M^(run * 32 * 2^i)
    for (int n = 0; n < 8; n++)
      for (uint32_t v = 0; v < 16; v++) tab[i * 128 + n * 16 + v] = apply(p, v << (4 * n));
    uint32_t q[32];
    for (int b = 0; b < 32; b++) q[b] = apply(p, p[b]);
    for (int b = 0; b < 32; b++) p[b] = q[b];
  }
}

static const void *window_kernel_of(int B) { return window_threads(B) == kWinNarrow ? window_kernel_narrow() : window_kernel_wide(); }

static cudaError_t window_attr(int B, size_t bytes) {
  static std::mutex mu;
  static size_t limit[2][64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lk(mu);
  size_t &cur = limit[B == 1][dev & 63];
  if (bytes <= cur) return cudaSuccess;
  e = cudaFuncSetAttribute(window_kernel_of(B), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(log_export_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (kSortWords + kSortThreads) * 4);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(log_record_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (kSortWords + kSortThreads) * 4);
  if (e == cudaSuccess) cur = bytes;
  return e;
}

int window_blocks_per_sm(int B, size_t smem) {
  int n = 0;
  if (window_attr(B, smem) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, window_kernel_of(B), window_threads(B), smem) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

cudaError_t launch_window(const WinArgs &a, int grid, size_t smem, cudaStream_t st) {
  const cudaError_t e = window_attr(a.B, smem);
  if (e != cudaSuccess) return e;
  void *args[] = {(void *)&a};
  return cudaLaunchCooperativeKernel(window_kernel_of(a.B), dim3(grid), dim3(window_threads(a.B)), args, smem, st);
}

cudaError_t launch_in_offsets(const uint32_t *indices, int32_t N, int64_t E, uint32_t *off, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(off, 0, (size_t)(N + 1) * 4, st);
  if (e != cudaSuccess) return e;
  if (E) in_degree_kernel<<<1216, 256, 0, st>>>(indices, E, off);
  exclusive_prefix_kernel<<<1, 1024, 0, st>>>(off, N);
  return cudaGetLastError();
}

cudaError_t launch_driven_pos(const Trial *trials, WinBrain *win, int B, cudaStream_t st) {
  driven_pos_kernel<<<B, 1024, 0, st>>>(trials, win);
  return cudaGetLastError();
}

cudaError_t launch_log_import(const Trial *trials, WinBrain *win, int B, int maxD, cudaStream_t st) {
  log_import_kernel<<<dim3(maxD, B), 256, 0, st>>>(trials, win);
  return cudaGetLastError();
}
cudaError_t launch_log_export(Trial *trials, WinBrain *win, int b0, int b1, int maxD, bool lastOnly, cudaStream_t st) {
  log_export_kernel<<<dim3(lastOnly ? 1 : maxD, b1 - b0), kSortThreads, (kSortWords + kSortThreads) * 4, st>>>(trials, win, b0, lastOnly);
  return cudaGetLastError();
}
cudaError_t launch_log_clear(WinBrain *win, int b0, int b1, cudaStream_t st) {
  log_clear_kernel<<<b1 - b0, kWinRing, 0, st>>>(win, b0);
  return cudaGetLastError();
}
cudaError_t launch_log_record(Trial *trials, WinBrain *win, int n, cudaStream_t st) {
  log_record_kernel<<<1, kSortThreads, (kSortWords + kSortThreads) * 4, st>>>(trials, win, n);
  return cudaGetLastError();
}

}  // namespace fb
#endif
