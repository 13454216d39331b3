// The delay-windowed step kernel (fb_window.cu): device records, arguments and launch glue.
#pragma once
#include "fb_internal.cuh"

namespace fb {

// Threads per block (one block per SM), by the number of brains. Many brains: as many warps as the
// registers allow, a tile's loads are hidden by other warps only (96 full brains, U of a window: 634
// us with 32 warps, 1,039 with 16). One brain: the window is a chain of round trips and block
// barriers, which 16 warps with twice the registers run faster (60,013 conductance-based neurons,
// window of 4 steps: 32.6 us with 32 warps, 27.3 with 16; the full graph, 18 steps: 28.2 and 26.1).
// Few brains share the wide form, since the narrow one keeps a single brain's headers: 200 steps of
// 2 / 4 / 8 brains of 20,000 neurons 303 / 311 / 370 us (one brain 242), on the grid kernel 2,436 /
// 2,528 / 2,881.
constexpr int kWinWide = 1024, kWinNarrow = 512;
inline int window_threads(int B) { return B == 1 ? kWinNarrow : kWinWide; }
constexpr int kWinMax = 31;         // steps per window at most (five key bits; 31 marks "no entry")
constexpr int kWinRing = 64;        // per-step log positions kept (a power of two >= delay + window)
constexpr int kWinSort = 16;        // contributions per target sorted in shared memory
constexpr int kWinStream = 37888;   // draws of a window at most, in shared memory
// Generator words per thread (odd: the threads' runs start in different banks).
constexpr int window_run(int threads) { return (kWinStream + threads - 1) / threads | 1; }
constexpr int kWarpBrainBytes = 384;
constexpr int kWinPool = 44032;     // words of that memory: a window's draws and its driven entries
// Words a driven list's entries take of it.
__host__ __device__ constexpr int window_entry_words(int nD) { return 3 * nD + (3 * nD + 3) / 4; }
// Driven neurons per brain at most: the chain's warps hold eight words of 32 entries each, and their
// entries share the block's memory with a window's draws. A brain beyond that, and its batch, goes to
// the grid kernel: 20,000 neurons, 200 steps, 4,090 driven 852 us, 4,097 driven 3,593.
constexpr int kWinDriven = 4096;
constexpr int kWinSaved = 12;       // words kept of a driven entry at the window's start
constexpr int kWinBrains = 512;     // brains per launch at most (per-brain words in shared memory)
constexpr int kWinSpikes = 256;     // arrivals a block delivers at a time
constexpr int32_t kWinIds = 1 << 23;  // neurons at most: ids and ranks (driven + id) of 24 bits

// One brain's window state. The spike log holds its spikes in flight in emission order (no order
// within a window): {id | step << 24 (8 bits), rank, its row's first and last edge + 1}; ranks order the spikes of a step as lif.c's
// fired list does (driven-list position, then driven count + id). ls[s & 63] is the log position
// at the start of the window that emitted step s.
struct WinBrain {
  int32_t D, H;        // arrival delay in steps; window length
  uint32_t logMask;    // log capacity - 1
  int32_t nPlaced;     // neurons with a place in drvPos, and which (kWinDriven at most)
  int32_t *placed;
  const uint32_t *inOff;  // [N+1] in-degree prefix: where a target's contributions start in wbuf
  int32_t *drvPos;     // [N] place in the driven list, -1 if not driven
  uint32_t *wcnt;      // [N] end of each target's contributions of the window in wbuf (inOff: none)
  uint2 *wbuf;         // [E] {step << 27 | rank << 3 | repeat << 1 | inhibitory, f32 bits}
  uint4 *log;
  uint8_t *arr;        // [N] 1 + the window step at which the neuron's own spike arrives (depression)
  uint32_t *bgMask;    // [N] window steps with background hits; bit 31: some step has several
  uint32_t *bgHit;     // [H][N] hits of a step after its first
  // driven entries (kWinDriven each): the window's live bits and 1 + the step of the neuron's own spike (both without a forced one), the state at the
  // window's start (v gE gI refr, adapt res trace, own arrival, contributions)
  uint32_t *dLive;
  uint8_t *dFired;
  float4 *dSave;       // 3 per entry
  uint32_t fDone;      // tiles of the driven list that have run the window
  uint32_t logTop;
  uint32_t ls[kWinRing];
  uint32_t rng;        // generator and background accumulator at the window's start
  float bgAcc;
};

struct WinArgs {
  Trial *trials;
  WinBrain *win;
  int32_t B, nWin;           // brains; windows of the longest-running brain
  const int32_t *steps;      // [B] steps of this launch
  int32_t anyBg, dedicated;  // background in any brain; blocks 0..B-1 only serve driven lists
  int32_t allPlain, pad;     // every brain: current-based, adapt 0, res 1, no background
  const uint32_t *jump;      // window_jump_tables(window_threads(B))
  uint32_t *barCount;        // grid barrier arrivals, barBase of them at launch
  uint32_t *uNext;           // [2] tiles dealt, by window parity
  int32_t *err;
  int64_t timeoutNs;
  int32_t tripStep;
  uint32_t barBase;
  unsigned long long *prof;
  uint32_t *dbg;
  char *brains;              // [B] kWarpBrainBytes: what U's warps need of each brain (written per window)
};

// M^(32 run 2^i) for i < 5 (8 nibble tables of 16 words each), then M^(run l) for l < 32 as word
// (n * 16 + nibble) * 32 + l, M the generator's map and run = window_run(threads).
constexpr int kWinJumpWords = 5 * 128 + 32 * 128;
void window_jump_tables(int threads, uint32_t *tab);
size_t window_smem_bytes(int B);
int window_blocks_per_sm(int B, size_t smem);
cudaError_t launch_window(const WinArgs &a, int grid, size_t smem, cudaStream_t st);
// The kernel of one width (fb_window.cu, compiled once per width).
const void *window_kernel_wide();
const void *window_kernel_narrow();
// In-degree prefix of a topology (off: [N+1]).
cudaError_t launch_in_offsets(const uint32_t *indices, int32_t N, int64_t E, uint32_t *off, cudaStream_t st);
// drvPos of every brain from its driven list (at most kWinDriven entries).
cudaError_t launch_driven_pos(const Trial *trials, WinBrain *win, int B, cudaStream_t st);
// The ring's spikes in flight into the log (import), the log's into the ring (export: every slot
// in flight, or the last step's list only), the log emptied (brains b0 .. b1-1).
cudaError_t launch_log_import(const Trial *trials, WinBrain *win, int B, int maxD, cudaStream_t st);
cudaError_t launch_log_export(Trial *trials, WinBrain *win, int b0, int b1, int maxD, bool lastOnly, cudaStream_t st);
cudaError_t launch_log_clear(WinBrain *win, int b0, int b1, cudaStream_t st);
// Appends the fired lists of the last n steps (at most the window's) to the per-step record.
cudaError_t launch_log_record(Trial *trials, WinBrain *win, int n, cudaStream_t st);

}  // namespace fb
