// The adjoint's forward, replay and reverse sweep in windows of the synaptic delay (included by
// fb_adjoint.cu). One launch of each kernel covers h steps instead of one:
//
//  - A spike arrives D = nslots - 1 steps after it is emitted, so with h <= D everything that
//    arrives in steps [t0, t0 + h) is on the tape before them: one k_wdeliver pushes the window's
//    contributions, one k_wupdate runs every neuron through the window with its state in registers.
//  - In the reverse sweep the adjoint of a spike reaches the neuron's step D steps earlier: the
//    window's h reverse neuron steps need only arrivals of later windows (k_wbneuron), and the
//    window's arrivals only the conductance adjoints those steps leave (kept per step), so one
//    k_wbarrival follows.
// h is also at most the steps a neuron stays silent after a spike, so a neuron spikes, and its row
// arrives, at most once in a window: a target's contributions fit in a region of its in-degree, and
// every edge and presynaptic accumulator still has one writer per kernel, in time order. Hard
// spikes only (a soft neuron spikes in every step); the per-step kernels run the rest.
//
// Arithmetic and its order are the per-step kernels'. What a step leaves for its reverse is less:
// the integrated potential u instead of v, gE, gI (current-based), no adaptation where it is 0,
// the spike in a bit of the mode -- 5 bytes per neuron and step instead of 21 in the current-based
// float case. The res adjoint, which only its own arrivals read, decays when one does.
#pragma once
#include "fb_window.cuh"

namespace fb {

constexpr int kWSort = 8;          // contributions per target sorted in shared memory
constexpr int kWindowMax = 31;     // steps per window (five key bits)
constexpr uint32_t kWNone = 0xffffffffu;

// A contribution: key {step << 27 | arrival rank << 1 | inhibitory}, edge, the amount (float bits,
// or a double's two words).
__device__ __forceinline__ bool w_before(const uint4 &p, const uint4 &q) { return p.x < q.x || (p.x == q.x && p.y < q.y); }

// Sort in place by (key, edge), one warp: each lane counts the entries before its own (up to 4 of
// them); longer lists by insertion, lane 0.
__device__ __noinline__ void w_warp_sort(uint4 *e, uint32_t n) {
  constexpr int kM = 4;
  const uint32_t lane = threadIdx.x & 31u;
  if (n > 32 * kM) {
    if (lane == 0)
      for (uint32_t gap = n / 2; gap > 0; gap /= 2)  // Shell sort
        for (uint32_t u = gap; u < n; u++) {
          const uint4 x = e[u];
          uint32_t w = u;
          while (w >= gap) {
            const uint4 y = e[w - gap];
            if (w_before(y, x)) break;
            e[w] = y;
            w -= gap;
          }
          e[w] = x;
        }
    __syncwarp();
    return;
  }
  uint4 x[kM];
  uint32_t rank[kM];
#pragma unroll
  for (int m = 0; m < kM; m++) {
    const uint32_t k = lane + 32 * m;
    x[m] = k < n ? e[k] : make_uint4(kWNone, kWNone, 0, 0);
    rank[m] = 0;
  }
#pragma unroll
  for (int g = 0; g < kM; g++) {
    if (32u * g >= n) break;
    for (int l = 0; l < 32; l++) {
      uint4 y = x[g];
      y.x = __shfl_sync(0xffffffffu, y.x, l);
      y.y = __shfl_sync(0xffffffffu, y.y, l);
#pragma unroll
      for (int m = 0; m < kM; m++) rank[m] += w_before(y, x[m]);
    }
  }
  __syncwarp();
#pragma unroll
  for (int m = 0; m < kM; m++)
    if (lane + 32 * m < n) e[rank[m]] = x[m];
  __syncwarp();
}

// A target's contributions of the window in order.
struct WList {
  const uint4 *p;
  int stride;
  uint32_t left;
  uint4 c;  // the current one (key kWNone: none)
};
__device__ __forceinline__ void wl_next(WList &l) {
  if (l.left) {
    l.p += l.stride;
    l.left--;
    l.c = *l.p;
  } else {
    l.c.x = kWNone;
  }
}
// Every lane its own target's; stage: this lane's column of shared memory (entries 32 apart).
__device__ __forceinline__ WList wl_make(uint4 *e, uint32_t n, uint4 *stage) {
  for (uint32_t big = __ballot_sync(0xffffffffu, n > (uint32_t)kWSort); big; big &= big - 1) {
    const int src = __ffs(big) - 1;
    uint4 *p = (uint4 *)__shfl_sync(0xffffffffu, (unsigned long long)e, src);
    w_warp_sort(p, __shfl_sync(0xffffffffu, n, src));
  }
  WList l;
  l.p = e;
  l.stride = 1;
  l.left = n ? n - 1 : 0;
  l.c = make_uint4(kWNone, 0, 0, 0);
  if (n > 1 && n <= (uint32_t)kWSort) {
    for (uint32_t u = 0; u < n; u++) {
      const uint4 x = e[u];
      uint32_t w = u;
      while (w > 0) {
        const uint4 y = stage[(w - 1) * 32];
        if (w_before(y, x)) break;
        stage[w * 32] = y;
        w--;
      }
      stage[w * 32] = x;
    }
    l.p = stage;
    l.stride = 32;
  }
  if (n) l.c = *l.p;
  return l;
}

// The instance's steps of window [t0, t1), and its arrivals: tape entries [a0, a1) with the first
// entry of each emission step (off[k]: step e0 + k).
struct WSpan {
  int h, e0, ne;
  int64_t a0, a1;
};
__device__ __forceinline__ WSpan w_span(const DiffDev &D, int t0, int t1, int64_t *off) {
  WSpan s;
  s.h = min(t1, D.steps) - t0;
  const int d = D.nslots - 1;
  s.e0 = max(0, t0 - d);
  s.ne = s.h > 0 ? max(0, t0 + s.h - d - s.e0) : 0;
  if (s.ne > 0 && (int)threadIdx.x <= s.ne) off[threadIdx.x] = min(D.tOff[s.e0 + threadIdx.x], D.tapeCap);
  __syncthreads();
  s.a0 = s.ne ? off[0] : 0;
  s.a1 = s.ne ? off[s.ne] : 0;
  return s;
}
__device__ __forceinline__ int w_step_of(const WSpan &s, const int64_t *off, int64_t a) {  // k with off[k] <= a < off[k+1]
  int lo = 0, hi = s.ne;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (off[mid] <= a) lo = mid;
    else hi = mid;
  }
  return lo;
}

// Delivery of the window's arrivals (k_deliver for h steps), `parts` warps per arrival; in a replay
// (row >= 0) also the forced spikes' marks from the tape. The amplitude's res is the window's first
// one recovered to the arrival step.
template <typename R>
__global__ void __launch_bounds__(kDB, 4) k_wdeliver(const DiffDev *Ds, DP<R> P, int32_t t0, int32_t t1, int32_t row,
                                                    int32_t parts) {
  __shared__ DiffDev D;
  __shared__ int64_t off[kWindowMax + 1];
  load_dev(Ds, D);
  const WSpan S = w_span(D, t0, t1, off);
  if (S.h <= 0) return;
  const int lane = threadIdx.x & 31, d = D.nslots - 1;
  const int64_t th = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, nth = (int64_t)gridDim.x * blockDim.x;
  if (row < 0 && th < kWindowMax) D.wSpikes[th] = 0;  // a forward's spike counts of the window
  if (row >= 0)
    for (int j = 0; j < S.h; j++) {
      const int64_t base = D.tOff[t0 + j], nf = tape_count(D, base, base + D.tForced[t0 + j]);
      for (int64_t k = th; k < nf; k += nth) D.wForced[D.tIdx[base + k]] = (uint8_t)(j + 1);
    }
  const int64_t work = (S.a1 - S.a0) * parts;
  for (int64_t w = th >> 5; w < work; w += nth >> 5) {
    const int64_t a = S.a0 + w / parts;
    const int part = (int)(w % parts);
    const int ek = w_step_of(S, off, a), j = S.e0 + ek + d - t0;
    const uint32_t k = (uint32_t)(a - off[ek]);
    const int32_t pre = D.tIdx[a];
    const float sg = D.sign[pre];
    float r = D.res[pre];
    if (sg == 0) continue;
    for (int q = 0; q < j; q++) r = (float)((R)r + (R(1) - (R)r) * P.kRec);
    if (row >= 0 && part == 0 && lane == 0) D.resAt[(int64_t)(row + j) * D.maxArr + k] = r;
    const R eff = (R)sg * P.wSyn * d_out<R>(D, pre) * exp((R)D.logGain[pre]) * (R)r * (R)D.tAmp[a];
    if (part == 0 && lane == 0) D.wArr[pre] = (uint8_t)(j + 1);
    const bool inh = !(eff > 0);
    const uint32_t key = ((uint32_t)j << 27) | (k << 1) | (inh ? 1u : 0u);
    const uint32_t lo = D.indptr[pre], hi = D.indptr[pre + 1];
    for (uint32_t j0 = lo + 32u * kEdgeILP * part + lane; j0 < hi; j0 += 32u * kEdgeILP * parts) {
      bool on[kEdgeILP];
      uint32_t q[kEdgeILP], pos[kEdgeILP];
      uint4 c[kEdgeILP];
#pragma unroll
      for (int u = 0; u < kEdgeILP; u++) {
        const uint32_t e = j0 + 32u * u;
        on[u] = e < hi && D.gate[e];
        if (on[u]) q[u] = D.indices[e];
      }
      if (row >= 0)
#pragma unroll
        for (int u = 0; u < kEdgeILP; u++) on[u] = on[u] && D.wNeed[q[u]];
#pragma unroll
      for (int u = 0; u < kEdgeILP; u++) {
        const uint32_t e = j0 + 32u * u;
        if (!on[u]) continue;
        c[u] = make_uint4(key, e, 0u, 0u);
        if (sizeof(R) == 8) {
          const R p = (R)D.P[e], x = inh ? p * P.inhGain * eff : p * eff;
          const long long b = __double_as_longlong((double)x);
          c[u].z = (uint32_t)b;
          c[u].w = (uint32_t)(b >> 32);
        } else {
          const R p = (R)D.Pf[e];
          c[u].z = __float_as_uint((float)(inh ? p * P.inhGain * eff : p * eff));
        }
      }
#pragma unroll
      for (int u = 0; u < kEdgeILP; u++)
        if (on[u]) pos[u] = atomicAdd(D.wCnt + q[u], 1u);  // the counter starts at the target's region
#pragma unroll
      for (int u = 0; u < kEdgeILP; u++)
        if (on[u] && (int64_t)pos[u] < D.E) D.wBuf[pos[u]] = c[u];
    }
  }
}

// A neuron's state and its window. REPLAY: its forced step `frc` comes from the tape, and what the
// reverse needs goes to the arena (CUBA: current-based, u alone is kept); otherwise the window runs
// without a forced spike, and the steps it is live in (not refractory, so that a driven neuron draws)
// and the step it fires in (-1) are returned.
struct WNeuron {
  float v, ge, gi, refr, ad, res;
};
__device__ __forceinline__ WNeuron wn_load(const DiffDev &D, int i) {
  WNeuron x;
  x.v = D.v[i];
  x.ge = D.gE[i];
  x.gi = D.gI[i];
  x.refr = D.refr[i];
  x.ad = D.adapt[i];
  x.res = D.res[i];
  return x;
}
__device__ __forceinline__ void wn_store(const DiffDev &D, int i, const WNeuron &x) {
  D.v[i] = x.v;
  D.gE[i] = x.ge;
  D.gI[i] = x.gi;
  D.refr[i] = x.refr;
  D.adapt[i] = x.ad;
  D.res[i] = x.res;
}
template <typename R, bool REPLAY, bool CUBA>
__device__ __forceinline__ int wn_run(const DiffDev &D, const DP<R> &P, int i, bool own, int h, int row, WNeuron &x, WList &l,
                                      int arr, int frc, uint32_t *live) {
  const int N = D.N;
  const float thrO = D.thrOffset[i];
  const R bias = d_bias<R>(D, P, i, nullptr), kc = d_kc<R>(D, P, i);
  R *aU = (R *)D.aV;
  const bool hasAd = P.adaptInc != 0;
  int fired = -1;
  bool wild = false;
  for (int j = 0; j < h; j++) {
    while ((l.c.x >> 27) == (uint32_t)j) {
      const R c = sizeof(R) == 8 ? (R)__longlong_as_double((long long)(((unsigned long long)l.c.w << 32) | l.c.z))
                                 : (R)__uint_as_float(l.c.z);
      if (l.c.x & 1u) x.gi = (float)((R)x.gi + c);
      else x.ge = (float)((R)x.ge + c);
      wl_next(l);
    }
    if (arr == j) x.res = (float)((R)x.res - P.depU * (R)x.res);
    if (REPLAY && frc == j) {
      x.refr = (float)(P.tRef + P.dt);
      x.ad = (float)((R)x.ad + P.adaptInc);
    }
    const R ge = x.ge, gi = x.gi;
    const int64_t at = REPLAY ? (int64_t)(row + j) * N + i : 0;
    R vi = x.v;
    int md = 0, s = 0;
    const bool wasRefr = x.refr > 0;
    if (wasRefr) {
      x.refr = (float)((R)x.refr - P.dt);
      vi = P.vReset;
      md = frc == j ? 2 : 1;
    } else {
      if (!REPLAY) *live |= 1u << j;
      vi = d_u<R>(D, P, vi, ge, gi, bias);
      if (REPLAY && own) {
        if (CUBA) {
          aU[at] = vi;
        } else {
          D.aV[at] = x.v;
          D.aGE[at] = x.ge;
          D.aGI[at] = x.gi;
        }
      }
    }
    x.ge = (float)(ge * P.dE);
    x.gi = (float)(gi * P.dE);
    x.ad = (float)((R)x.ad * P.dA);
    x.res = (float)((R)x.res + (R(1) - (R)x.res) * P.kRec);
    if (REPLAY && own && hasAd && !wasRefr) D.aAd[at] = x.ad;
    if (!wasRefr) {
      const R thr = P.vThresh + (R)x.ad + kc + (R)thrO;
      wild |= !(fabs(vi - thr) <= (R)3e38);
      if (vi >= thr) {
        s = 1;
        fired = j;
        vi = R(1) * P.vReset + (R(1) - R(1)) * vi;
        x.refr = (float)P.tRef;
        x.ad = (float)((R)x.ad + R(1) * P.adaptInc);
      }
    }
    if (REPLAY && own) D.aMode[at] = (uint8_t)(md | s << 2);
    x.v = (float)vi;
  }
  if (own && wild) (REPLAY ? D.wAct : D.wWild)[i] = 1;  // zero times infinity
  return fired;
}

// The window's contributions of neuron i (none unless own).
__device__ __forceinline__ uint32_t wn_count(const DiffDev &D, int i, bool own, uint32_t &o) {
  o = D.cscPtr[i];
  const uint32_t end = D.cscPtr[i + 1];
  uint32_t n = own ? D.wCnt[i] - o : 0u;
  if (n > end - o) {  // two spikes of one neuron in a window
    atomicCAS(D.err, 0, FB_EOVERFLOW);
    n = 0;
  }
  return n;
}

// The neurons whose replay the reverse sweep reads (all: every one): those whose adjoint may not be
// zero, and those with a spike on the tape in steps [e0, e1) -- the segment's, the D steps' before
// it, whose spikes arrive in it, and the next segment's, whose sweep runs beside this replay: only a
// neuron with such a spike can be handed an adjoint from then on. A neuron's own trajectory needs
// the tape's spikes and nothing else of the others'. Two launches: 0 copies the marks, 1 adds the
// spikes'.
__global__ void k_wneed(const DiffDev *Ds, int32_t e0, int32_t e1, int32_t all, int32_t spikes) {
  __shared__ DiffDev D;
  load_dev(Ds, D);
  const int64_t s0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, ns = (int64_t)gridDim.x * blockDim.x;
  if (!spikes) {
    for (int64_t i = s0; i < D.N; i += ns) D.wNeed[i] = all || D.wAct[i];
    return;
  }
  e0 = min(e0, D.steps);
  e1 = min(e1, D.steps);
  const int64_t a1 = min(D.tOff[e1], D.tapeCap);
  for (int64_t a = D.tOff[e0] + s0; a < a1; a += ns) D.wNeed[D.tIdx[a]] = 1;
}

// Replay of the window (k_update for h steps of a replay) for the needed neurons of each tile of
// 256, gathered so that they fill warps, a neuron per lane.
template <typename R, bool CUBA>
__global__ void __launch_bounds__(kDB, 4) k_wreplay(const DiffDev *Ds, DP<R> P, int32_t t0, int32_t t1, int32_t row) {
  __shared__ DiffDev D;
  __shared__ uint4 stage[kDB / 32][kWSort * 32];
  __shared__ uint16_t mark[kDB];
  __shared__ uint32_t nMark;
  load_dev(Ds, D);
  const int h = min(t1, D.steps) - t0;
  if (h <= 0) return;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const int N = D.N;
  for (int tile = blockIdx.x * kDB; tile < N; tile += gridDim.x * kDB) {
    __syncthreads();
    if (threadIdx.x == 0) nMark = 0;
    __syncthreads();
    if (tile + (int)threadIdx.x < N && D.wNeed[tile + threadIdx.x]) mark[atomicAdd(&nMark, 1u)] = (uint16_t)threadIdx.x;
    __syncthreads();
    if (warp * 32 >= nMark) continue;
    const bool own = threadIdx.x < nMark;
    const int i = tile + mark[own ? threadIdx.x : warp * 32];
    uint32_t o;
    WNeuron x = wn_load(D, i);
    const int arr = (int)D.wArr[i] - 1, frc = (int)D.wForced[i] - 1;
    const uint32_t n = wn_count(D, i, own, o);
    WList l = wl_make(D.wBuf + o, n, stage[warp] + lane);
    __syncwarp();
    wn_run<R, true, CUBA>(D, P, i, own, h, row, x, l, arr, frc, nullptr);
    if (!own) continue;
    wn_store(D, i, x);
    if (n) D.wCnt[i] = o;
    if (arr >= 0) D.wArr[i] = 0;
    if (frc >= 0) D.wForced[i] = 0;
  }
}

// ---- the forward ----------------------------------------------------------------------------------
// As in the brain step's windows (fb_window.cu): the driven neurons first run the window as if
// nothing were drawn for them (k_wforward, its driven part), one block per instance follows the chain
// of draws (k_wchain), the other neurons run beside it (k_wforward), and the window's spikes go to
// the tape from per-step bitmaps (k_wemit). A window lies within a checkpoint interval and a drive
// epoch.

// Places in the live drivenSet (wDrv, -1: not driven), at the start of a pass and after an epoch's edits.
__global__ void k_wplaces(const DiffDev *Ds, int32_t set) {
  __shared__ DiffDev D;
  load_dev(Ds, D);
  const int n = set ? *D.nLive : D.N;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    if (set) D.wDrv[D.drivenLive[k]] = k;
    else D.wDrv[k] = -1;
  }
}

// driven 0: the neurons that are not driven; 1: the driven list, without its draws.
template <typename R>
__global__ void __launch_bounds__(kDB, 4) k_wforward(const DiffDev *Ds, DP<R> P, int32_t t0, int32_t t1, int32_t driven) {
  __shared__ DiffDev D;
  __shared__ uint4 stage[kDB / 32][kWSort * 32];
  load_dev(Ds, D);
  const int h = min(t1, D.steps) - t0;
  if (h <= 0) return;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const int M = driven ? *D.nLive : D.N, nW = (M + 31) / 32;
  for (int wt = blockIdx.x * (kDB / 32) + warp; wt < nW; wt += gridDim.x * (kDB / 32)) {
    const int k = wt * 32 + (int)lane, kk = k < M ? k : M - 1;
    const int i = driven ? D.drivenLive[kk] : kk;
    const bool own = k < M && (driven || D.wDrv[i] < 0);
    uint32_t o, live = 0;
    WNeuron x = wn_load(D, i);
    const float ad0 = x.ad;
    const int arr = (int)D.wArr[i] - 1;
    const uint32_t n = wn_count(D, i, own, o);
    WList l = wl_make(D.wBuf + o, n, stage[warp] + lane);
    __syncwarp();
    int fired = wn_run<R, false, false>(D, P, i, own, h, 0, x, l, arr, -1, &live);
    if (!own) fired = -1;
    if (own) {
      wn_store(D, i, x);
      if (n) D.wCnt[i] = o;
      if (arr >= 0) D.wArr[i] = 0;
    }
    if (driven) {
      if (own) {
        D.wLive[k] = live;
        D.wOwn[k] = (uint8_t)(fired + 1);
        D.wAd0[k] = ad0;
      }
      continue;
    }
    if (fired >= 0) {
      atomicOr(D.wBits + (int64_t)fired * nW + wt, 1u << lane);
      atomicAdd(D.wSpikes + fired, 1);
      D.spikeCount[i] = (float)((R)D.spikeCount[i] + R(1));
    }
  }
}

constexpr int kChainThreads = kWinNarrow;
constexpr int kChainRun = window_run(kChainThreads);
constexpr int kChainDriven = 8 * kChainThreads;  // driven neurons per instance at most

// For each step the live entries' ranks, their draws, the forced spikes (draw_chain of fb_window.cu:
// a warp owns M words of 32 entries and publishes a byte per four of them and step). sm: the
// window's draws; returns the number used.
template <int M>
__device__ __forceinline__ uint32_t wc_chain(int n, int h, uint32_t *sLive, const uint32_t *sLim, const uint32_t *sm,
                                             uint4 (*cnt)[2]) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, lt = (1u << lane) - 1u;
  constexpr int kBytes = M > 4 ? 2 : 1, V = kBytes;
  uint32_t below[4 * V];
#pragma unroll
  for (int q = 0; q < 4 * V; q++) {
    const int m = min(max((int)warp * kBytes - 4 * q, 0), 4);
    below[q] = m == 0 ? 0u : 0x01010101u >> (32 - 8 * m);
  }
  uint32_t mask[M], lim[M], f[M];
#pragma unroll
  for (int m = 0; m < M; m++) {
    const int k = (int)(warp * M + m) * 32 + (int)lane;
    mask[m] = k < n ? sLive[k] : 0u;
    lim[m] = k < n ? sLim[k] : 0u;
    f[m] = 255u;
  }
  uint32_t base = 0;
  for (int j = 0; j < h; j++) {
    uint32_t live[M], mine[2] = {0, 0};
#pragma unroll
    for (int m = 0; m < M; m++) {
      live[m] = __ballot_sync(0xffffffffu, mask[m] & 1u);
      mine[m / 4] += (uint32_t)__popc(live[m]);
    }
    if (lane < kBytes) ((uint8_t *)cnt[j & 1])[warp * kBytes + lane] = (uint8_t)(lane ? mine[1] : mine[0]);
    __syncthreads();
    uint32_t at = base;
#pragma unroll
    for (int v = 0; v < V; v++) {
      const uint4 c = cnt[j & 1][v];
      at = __dp4a(c.x, below[4 * v], at);
      at = __dp4a(c.y, below[4 * v + 1], at);
      at = __dp4a(c.z, below[4 * v + 2], at);
      at = __dp4a(c.w, below[4 * v + 3], at);
      base = __dp4a(c.x, 0x01010101u, base);
      base = __dp4a(c.y, 0x01010101u, base);
      base = __dp4a(c.z, 0x01010101u, base);
      base = __dp4a(c.w, 0x01010101u, base);
    }
    uint32_t x[M];
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
  __syncthreads();
#pragma unroll
  for (int m = 0; m < M; m++) {
    const int k = (int)(warp * M + m) * 32 + (int)lane;
    if (k < n) sLive[k] = f[m];  // the forced step from here on
  }
  return base;
}

// The window's draws and forced spikes of one instance per block; the forced neurons' state and the
// driven ones' own spikes.
template <typename R>
__global__ void __launch_bounds__(kChainThreads, 1) k_wchain(const DiffDev *Ds, DP<R> P, int32_t t0, int32_t t1,
                                                            const uint32_t *jumpTab) {
  extern __shared__ __align__(16) uint32_t pool[];  // lane tables, live bits, draw limits, draws
  __shared__ DiffDev D;
  __shared__ uint4 cnt[2][2];
  __shared__ int nForced[kWindowMax];
  __shared__ uint32_t nEvents;
  load_dev(Ds, D);
  const int h = min(t1, D.steps) - t0;
  if (h <= 0) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = *D.nLive;
  uint32_t *jump = pool, *sLive = pool + kWinJumpWords, *sLim = sLive + n, *sm = sLim + n;
  for (int k = tid; k < kWinJumpWords; k += kChainThreads) jump[k] = jumpTab[k];
  if (tid < 4) cnt[tid >> 1][tid & 1] = make_uint4(0, 0, 0, 0);
  if (tid < kWindowMax) nForced[tid] = 0;
  if (tid == 0) nEvents = 0;
#pragma unroll 4
  for (int k = tid; k < n; k += kChainThreads) {
    sLive[k] = D.wLive[k];
    // x <= lim for u < p: u = (x >> 8) 2^-24, p = drive dt/1000 in R; a draw x is never 0
    const R p = (R)d_drive(D, D.drivenLive[k], t0) * P.dtS;
    const uint32_t t = p >= R(1) ? 1u << 24 : (uint32_t)ceil((double)p * 16777216.0);
    sLim[k] = t ? (t << 8) - 1u : 0u;
  }
  const uint32_t s0 = *D.rng;
  __syncthreads();
  const uint32_t need = (uint32_t)n * (uint32_t)h;  // the host keeps it within the pool
  if ((uint32_t)warp * 32 * kChainRun < need) {
    uint32_t b = s0, x = 0;
    for (int q = 0; q < 5; q++)
      if ((warp >> q) & 1) b = xs_apply(jump + q * 128, b);
    const uint32_t *off = jump + 5 * 128;
#pragma unroll
    for (int q = 0; q < 8; q++) x ^= off[((uint32_t)q * 16 + ((b >> (4 * q)) & 15u)) * 32 + lane];
    for (uint32_t k = (uint32_t)tid * kChainRun, e = min(need, k + kChainRun); k < e; k++) {
      x = xs_next(x);
      sm[k] = x;
    }
  }
  __syncthreads();
  uint32_t used;
  if (n <= kChainThreads) used = wc_chain<1>(n, h, sLive, sLim, sm, cnt);
  else if (n <= 4 * kChainThreads) used = wc_chain<4>(n, h, sLive, sLim, sm, cnt);
  else used = wc_chain<8>(n, h, sLive, sLim, sm, cnt);
  __syncthreads();
  if (tid == 0 && used) *D.rng = sm[used - 1];
  // the entries that fire, gathered so that one pass serves them (in the place of the limits)
  uint32_t *event = sLim;
  for (int k0 = 0; k0 < n; k0 += kChainThreads) {
    const int k = k0 + tid;
    uint32_t f = 255u;
    int own = -1;
    if (k < n) {
      f = sLive[k];
      own = (int)D.wOwn[k] - 1;
      D.wFs[k] = (uint8_t)f;
    }
    const bool on = f != 255u || own >= 0;
    const uint32_t m = __ballot_sync(0xffffffffu, on);
    uint32_t at = 0;
    if (m && lane == 0) at = atomicAdd(&nEvents, (uint32_t)__popc(m));
    at = __shfl_sync(0xffffffffu, at, 0) + (uint32_t)__popc(m & ((1u << lane) - 1u));
    if (on) event[at] = (uint32_t)k | (f << 16) | ((uint32_t)(own + 1) << 24);
  }
  __syncthreads();
  const uint32_t nE = nEvents;
  for (uint32_t q = tid; q < nE; q += kChainThreads) {
    const uint32_t ev = event[q], f = (ev >> 16) & 255u;
    const int k = (int)(ev & 0xffffu), own = (int)(ev >> 24) - 1;
    const int i = D.drivenLive[k];
    D.spikeCount[i] = (float)((R)D.spikeCount[i] + R(1));
    if (f == 255u) {
      atomicOr(D.wBits + (int64_t)own * ((D.N + 31) / 32) + (i >> 5), 1u << (i & 31));
      atomicAdd(D.wSpikes + own, 1);
      continue;
    }
    atomicAdd(&nForced[f], 1);
    // refractory from the forced spike to the window's end
    float r = (float)(P.tRef + P.dt), ad = D.wAd0[k];
    for (int j = 0; j < h; j++) {
      if (j >= (int)f && r > 0) r = (float)((R)r - P.dt);
      if (j == (int)f) ad = (float)((R)ad + P.adaptInc);
      ad = (float)((R)ad * P.dA);
    }
    D.v[i] = (float)P.vReset;
    D.refr[i] = r;
    D.adapt[i] = ad;
  }
  __syncthreads();
  if (tid < h) D.tForced[t0 + tid] = nForced[tid];
}

// The tape of step t0 + blockIdx.x: its forced spikes in list order, then its threshold spikes
// ascending, after the window's steps before it.
__global__ void __launch_bounds__(1024) k_wemit(const DiffDev *Ds, int32_t t0, int32_t t1) {
  __shared__ DiffDev D;
  __shared__ uint32_t scan[33];
  load_dev(Ds, D);
  const int h = min(t1, D.steps) - t0, j = blockIdx.x, tid = threadIdx.x;
  if (j >= h) return;
  int64_t o = D.tOff[t0];
  for (int q = 0; q < j; q++) o += D.tForced[t0 + q] + D.wSpikes[q];
  auto put = [&](int64_t at, int32_t i) {
    if (at < D.tapeCap) {
      D.tIdx[at] = i;
      D.tAmp[at] = 1.f;
    } else {
      atomicCAS(D.err, 0, FB_EOVERFLOW);
    }
  };
  const int n = *D.nLive;
  for (int k0 = 0; k0 < n; k0 += 1024) {
    const int k = k0 + tid;
    const uint32_t on = k < n && D.wFs[k] == j ? 1u : 0u;
    uint32_t tot;
    const uint32_t at = block_exclusive_scan(on, &tot, scan);
    if (on) put(o + at, D.drivenLive[k]);
    o += tot;
  }
  const int nW = (D.N + 31) / 32, per = (nW + 1023) / 1024, w0 = min(nW, tid * per), w1 = min(nW, w0 + per);
  uint32_t c = 0, tot;
  uint32_t *words = D.wBits + (int64_t)j * nW;
  for (int w = w0; w < w1; w++) c += (uint32_t)__popc(words[w]);
  int64_t at = o + block_exclusive_scan(c, &tot, scan);
  if (c)
    for (int w = w0; w < w1; w++) {
      uint32_t bits = words[w];
      if (!bits) continue;
      words[w] = 0;
      for (; bits; bits &= bits - 1) put(at++, w * 32 + __ffs(bits) - 1);
    }
  if (tid == 0) D.tOff[t0 + j + 1] = o + tot;
}

// A gradient accumulator over a window's steps (kWA..kWEI). A double runs at two lanes per clock and
// SM here, so the sums of floats are kept as three floats, in wSum from window to window, whose sum
// is exact but for the last one's rounding (TwoSum: Knuth, The Art of Computer Programming,
// 4.2.2): 72 bits against a double's 53. Addends past 2^100, infinities and NaN go to the double;
// k_wsums adds the floats to it at the pass's end.
enum { kWA, kWV, kWB, kWEI, kWSums };
static_assert(3 * kWSums == kWSumRows, "three floats per accumulator");
__device__ __forceinline__ double *w_acc(const DiffDev &D, int k) {
  return k == kWA ? D.accA : k == kWV ? D.accV : k == kWB ? D.gBias : D.accEI;
}
template <typename R, int k>
struct WSum {
  double s;
  __device__ void load(const DiffDev &D, int i) { s = w_acc(D, k)[i]; }
  __device__ void add(const DiffDev &, int, R x) { s += x; }
  __device__ void store(const DiffDev &D, int i) const { w_acc(D, k)[i] = s; }
};
template <int k>
struct WSum<float, k> {
  float a, b, c;
  __device__ void load(const DiffDev &D, int i) {
    const float *p = D.wSum + (int64_t)3 * k * D.N + i;
    a = p[0], b = p[D.N], c = p[2 * (int64_t)D.N];
  }
  __device__ static float two(float &s, float x) {  // s + x as s and what it lost
    const float t = s + x, z = t - s, e = (s - (t - z)) + (x - z);
    s = t;
    return e;
  }
  __device__ void add(const DiffDev &D, int i, float x) {
    if (!(fabsf(x) <= 0x1p100f)) w_acc(D, k)[i] += (double)x;
    else c += two(b, two(a, x));
  }
  __device__ void store(const DiffDev &D, int i) const {
    float *p = D.wSum + (int64_t)3 * k * D.N + i;
    p[0] = a, p[D.N] = b, p[2 * (int64_t)D.N] = c;
  }
};
// The accumulators complete: the floats' part, and the two that are sums of the same addends over
// part of the neurons (kcThreshold, laminaBias).
template <typename R>
__global__ void k_wsums(const DiffDev *Ds, DP<R> P) {
  __shared__ DiffDev D;
  load_dev(Ds, D);
  const int64_t N = D.N;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
    if (sizeof(R) == 4)
      for (int k = 0; k < kWSums; k++) {
        const float *p = D.wSum + 3 * k * N + i;
        w_acc(D, k)[i] += (double)p[0] + ((double)p[N] + (double)p[2 * N]);
      }
    if (D.thrMask && D.thrMask[i]) D.accKc[i] = D.accV[i];
    R lam;
    d_bias<R>(D, P, i, &lam);
    if (lam != 0) D.accLa[i] = D.gBias[i];
  }
}

// The reverse sweep leaves out what is zero. A neuron's adjoint is zero until a loss gradient or an
// arrival reversed at one of its targets reaches it, and a step of the sweep keeps it so (every
// term is a product with it). wAct marks the neurons that may have one: at the pass's start those
// with a loss gradient, then those k_wbarrival hands one to; also every neuron whose products with
// zero need not be zero (a potential, threshold or surrogate width that is not finite, `dense` for
// the parameters, wWild the recorded forward's). The others' rows of wE and wI stay zero. 1% of the neurons of a full brain with
// 1,000 readouts are ever marked.
template <typename R>
__global__ void k_wactive(const DiffDev *Ds, DP<R> P, int32_t dense, int32_t fromForward) {
  __shared__ DiffDev D;
  load_dev(Ds, D);
  const int64_t N = D.N, s0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, ns = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = s0; i < N; i += ns) {
    const bool loss = D.dL && (D.roMap ? D.roMap[i] >= 0 : !(D.dL[i] == 0.f));
    const float thr = D.thrOffset[i];
    D.wAct[i] = dense || loss || (fromForward && D.wWild[i]) || thr != thr || !(d_beta<R>(D, P, (int)i) > R(1e-30));
  }
  for (int64_t k = s0; k < 2 * D.wRows * N; k += ns) D.wE[k] = 0.f;  // and wI behind it
}

// The reverse neuron pass of the window's steps, last first (bneuron for h steps), over the marked
// neurons of each tile of 256, gathered so that they fill warps; the conductance adjoints after
// each step go to wE / wI for the window's arrivals.
template <typename R, bool CUBA>
__global__ void __launch_bounds__(kDB, 4) k_wbneuron(const DiffDev *Ds, DP<R> P, int32_t t0, int32_t t1, int32_t row,
                                                    int32_t lossFrom) {
  __shared__ DiffDev D;
  load_dev(Ds, D);
  const int h = min(t1, D.steps) - t0;
  if (h <= 0) return;
  const int N = D.N;
  const R *aU = (const R *)D.aV;
  const bool hasAd = P.adaptInc != 0;
  const R c = P.adjClip;
  auto cl = [c](float x) { return c > 0 ? (float)((R)x > c ? c : ((R)x < -c ? -c : (R)x)) : x; };
  __shared__ uint16_t mark[kDB];
  __shared__ uint32_t nMark;
  for (int tile = blockIdx.x * kDB; tile < N; tile += gridDim.x * kDB) {
    __syncthreads();
    if (threadIdx.x == 0) nMark = 0;
    __syncthreads();
    if (tile + (int)threadIdx.x < N && D.wAct[tile + threadIdx.x]) mark[atomicAdd(&nMark, 1u)] = (uint16_t)threadIdx.x;
    __syncthreads();
    if (threadIdx.x >= nMark) continue;
    const int i = tile + mark[threadIdx.x];
    float lv = D.lv[i], lgE = D.lgE[i], lgI = D.lgI[i], lad = D.lad[i];
    WSum<R, kWA> sA;
    WSum<R, kWV> sV;
    WSum<R, kWB> sB;
    WSum<R, kWEI> sEI;
    sA.load(D, i);
    sV.load(D, i);
    sB.load(D, i);
    if (!CUBA) sEI.load(D, i);
    const R bias = d_bias<R>(D, P, i, nullptr), kc = d_kc<R>(D, P, i), beta = d_beta<R>(D, P, i);
    const float thrO = D.thrOffset[i];
    const int ro = D.dL && D.roMap ? D.roMap[i] : -1;
    const int slotD = D.gDrive ? D.dSlot[i] : -1;
    const bool lossAll = D.dL && !D.roMap, lossRo = ro >= 0;
    // a step's inputs, loaded a step ahead: mode, spike adjoint, potential, loss gradient
    struct In {
      int m;
      float ls, v, ge, gi, ad, dl;
      R u;
    };
    auto load = [&](int j) {
      In x;
      const int t = t0 + j;
      const int64_t at = (int64_t)(row + j) * N + i;
      x.m = D.aMode[at];
      x.ls = D.lsRing[(int64_t)(t % D.nslots) * N + i];
      x.v = x.ge = x.gi = 0.f;
      x.u = 0;
      if (CUBA) {
        x.u = aU[at];
      } else {
        x.v = D.aV[at];
        x.ge = D.aGE[at];
        x.gi = D.aGI[at];
      }
      x.ad = hasAd ? D.aAd[at] : 0.f;
      x.dl = t >= lossFrom && (lossAll || lossRo) ? (lossRo ? D.dL[(int64_t)t * D.nro + ro] : D.dL[i]) : 0.f;
      return x;
    };
    In next = load(h - 1);
    for (int j = h - 1; j >= 0; j--) {
      const int t = t0 + j;
      const In in = next;
      if (j > 0) next = load(j - 1);
      const int m = in.m, md = m & 3;
      const R lpA = lad;
      const R lE = (R)lgE * P.dE, lI = (R)lgI * P.dE, lA = lpA * P.dA;
      float lgEF = (float)lE, lgIF = (float)lI, ladF = (float)lA;
      if (md == 1) {
        lv = 0.f;
      } else {
        const float lsv = in.ls;
        const R dl = in.dl;
        float *gDrv = slotD >= 0 ? D.gDrive + (int64_t)(t / D.driveEpoch) * D.nDS + slotD : nullptr;
        if (__float_as_uint(lsv) != 0u) D.lsRing[(int64_t)(t % D.nslots) * N + i] = 0.f;
        if (md == 2) {
          if (lA != R(0)) sA.add(D, i, lA);
          if (gDrv) *gDrv = (float)((R)*gDrv + (lA * P.adaptInc + ((R)lsv + dl)) * P.dtS);
          lv = 0.f;
        } else {
          const R vv = in.v, gEv = in.ge, gIv = in.gi;
          const R uu = CUBA ? in.u : d_u<R>(D, P, vv, gEv, gIv, bias);
          const R thr = P.vThresh + (R)in.ad + kc + (R)thrO;
          const R d = uu - thr;
          const R s = (m & 4) ? R(1) : R(0);
          const R tt = R(1) + fabs(d) / beta;
          const R sg = R(1) / (beta * tt * tt);
          const R lspike = (R)lsv + dl;
          const R lvNew = lv;
          const R lsTot = (P.vReset - uu) * lvNew + lpA * P.adaptInc + lspike;
          const R lt = lsTot * (R(1) - R(0)) * sg;
          const R lu = lvNew * (R(1) - s) + lt;
          const R lthr = -lt;
          if (gDrv) *gDrv = (float)((R)*gDrv + lsTot * (R(1) - s) * P.dtS);
          const R aA = lpA * s, aB = lu * P.kM;
          if (aA != R(0)) sA.add(D, i, aA);
          if (lthr != R(0)) sV.add(D, i, lthr);
          ladF = (float)(lA + lthr * P.dA);
          if (CUBA) {
            lv = (float)(lu * (R(1) - P.kM));
            lgEF = (float)(lE + lu * P.kM);
            lgIF = (float)(lI + lu * P.kM);
          } else {
            lv = (float)(lu * (R(1) + P.kM * (R(-1) - gEv * P.cE + gIv * P.cI)));
            lgEF = (float)(lE + lu * P.kM * (P.eExc - vv) * P.cE);
            lgIF = (float)(lI + lu * P.kM * (vv - P.eInh) * P.cI);
            const R aE = lu * P.kM * gIv * P.cI * (R(-1) + (vv - P.eInh) * P.cI);
            if (aE != R(0)) sEI.add(D, i, aE);
          }
          if (aB != R(0)) sB.add(D, i, aB);
        }
      }
      lv = cl(lv);
      lgE = cl(lgEF);
      lgI = cl(lgIF);
      lad = cl(ladF);
      D.wE[(int64_t)j * N + i] = lgE;
      D.wI[(int64_t)j * N + i] = lgI;
    }
    D.lv[i] = lv;
    D.lgE[i] = lgE;
    D.lgI[i] = lgI;
    D.lad[i] = lad;
    sA.store(D, i);
    sV.store(D, i);
    sB.store(D, i);
    if (!CUBA) sEI.store(D, i);
  }
}

// Reverse of the window's deliveries (k_barrival for h steps), warp per arrival.
template <typename R>
__global__ void __launch_bounds__(kDB, 2) k_wbarrival(const DiffDev *Ds, DP<R> P, int32_t t0, int32_t t1, int32_t row,
                                                      int32_t dense) {
  __shared__ DiffDev D;
  __shared__ int64_t off[kWindowMax + 1];
  load_dev(Ds, D);
  const WSpan S = w_span(D, t0, t1, off);
  if (S.h <= 0) return;
  const bool wild = dense || *D.wild;
  const int lane = threadIdx.x & 31, dd = D.nslots - 1;
  const int64_t w0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t a = S.a0 + w0; a < S.a1; a += nw) {
    const int ek = w_step_of(S, off, a), e = S.e0 + ek, t = e + dd, j = t - t0;
    const int32_t pre = D.tIdx[a];
    const R sgn = D.sign[pre];
    if (sgn == 0) continue;
    const R amp = D.tAmp[a];
    const R resAtv = D.resAt[(int64_t)(row + j) * D.maxArr + (a - off[ek])];
    const R gain = exp((R)D.logGain[pre]) * d_out<R>(D, pre);
    const R base = sgn * P.wSyn * gain * resAtv;
    const R eff = base * amp;
    const bool exc = eff > 0;
    const float *lg0 = (exc ? D.wE : D.wI) + (int64_t)j * D.N;
    const uint32_t lo = D.indptr[pre], hi = D.indptr[pre + 1];
    const bool all = wild || !(fabs(eff) <= (R)3e38) || !(fabs(base) <= (R)3e38);
    R lraw = 0;
    for (uint32_t j0 = lo + lane; j0 < hi; j0 += 32 * kEdgeILP) {
      bool on[kEdgeILP];
      uint32_t q[kEdgeILP];
      float cnt[kEdgeILP], eg[kEdgeILP], lgv[kEdgeILP], ins[kEdgeILP];
      double old[kEdgeILP];
#pragma unroll
      for (int u = 0; u < kEdgeILP; u++) {
        const uint32_t ed = j0 + 32u * u;
        on[u] = ed < hi && D.gate[ed];
        if (on[u]) q[u] = D.indices[ed];
      }
#pragma unroll
      for (int u = 0; u < kEdgeILP; u++)
        if (on[u]) lgv[u] = lg0[q[u]];
#pragma unroll
      for (int u = 0; u < kEdgeILP; u++) {  // a zero adjoint adds zeros
        const uint32_t ed = j0 + 32u * u;
        on[u] = on[u] && (all || lgv[u] != 0.f);
        if (on[u]) {
          cnt[u] = D.counts[ed];
          eg[u] = D.edgeGain ? D.edgeGain[ed] : 1.f;
          old[u] = D.gEdge[ed];
          ins[u] = D.inScale[q[u]];
        }
      }
#pragma unroll
      for (int u = 0; u < kEdgeILP; u++) {
        if (on[u]) {
          const R lg = lgv[u];
          const R cw = (R)cnt[u] * (R)eg[u];
          lraw += exc ? lg * cw * (R)ins[u] : lg * cw * (R)ins[u] * P.inhGain;
          D.gEdge[j0 + 32u * u] = old[u] + (double)(lg * eff);
        }
      }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) lraw += __shfl_xor_sync(0xffffffffu, lraw, o);
    if (lane == 0 && (all || lraw != 0 || D.lres[pre] != 0.f)) {
      float *target = D.lsRing + (int64_t)(e % D.nslots) * D.N;
      D.accW[pre] += (double)(lraw * sgn * gain * resAtv * amp);
      D.gLog[pre] += (double)(lraw * eff);
      float x = (float)((R)target[pre] + lraw * base);
      if (P.adjClip > 0) x = (float)fmin(P.adjClip, fmax(-P.adjClip, (R)x));
      target[pre] = x;
      if (x != 0.f) D.wAct[pre] = 1;  // NaN != 0
      // the res adjoint decays once per step down to this one (its clip bounds what an arrival left)
      float lr = D.lres[pre];
      if (lr != 0.f)
        for (int s = D.wResT[pre] - t; s > 0; s--) lr = (float)((R)lr * (R(1) - P.kRec));
      const R lresAfter = lr;
      D.accD[pre] += (double)(-lresAfter * resAtv);
      float y = (float)(lresAfter * (R(1) - P.depU) + lraw * sgn * P.wSyn * gain * amp);
      if (P.adjClip > 0) y = (float)fmin(P.adjClip, fmax(-P.adjClip, (R)y));
      D.lres[pre] = y;
      D.wResT[pre] = t;
    }
  }
}

}  // namespace fb
