// The flyvis optic-lobe rate network (src/wasm/lif.c:82-93, src/flyvis.js, src/flyvisgpu.js) on
// sm_103a: B instances (the eyes of one or many flies) sharing one model, advanced together.
//
//   acc[i] = sum over edges (j -> i) with v[j] > 0 of weight * v[j]
//   v[i]  += kdt[i] * (-v[i] + bias[i] + acc[i] + x[i])
//
// lif.c scatters by source (acc[target[k]] += weight[k] * v[j], sources ascending, each row in
// CSR order); per target that is its in-edges in ascending edge id. Here every (target, instance)
// pair gathers its in-edges in that order from a transposed copy of the graph built once, so the
// sums are lif.c's bit for bit with no atomics (the WGSL port rounds to 1/65536 fixed point
// instead). State is instance-minor ([N][B]). A step gathers the rectified activity r (v where v > 0,
// else 0) that the step before left in rows padded to whole vectors, double-buffered; a call's first
// step gathers v itself, which may have been written from outside, and leaves the new one in the
// other of two v buffers. Either way every target sees the previous step's activity, as with
// lif.c's separate scatter and update passes.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <vector>

#include "fb_internal.cuh"

namespace fb {
int set_error(int code, const char *msg);
}
using namespace fb;

namespace {

int fvfail(int code, const char *fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  return set_error(code, buf);
}

#define FVCU(call)                                                                            \
  do {                                                                                        \
    cudaError_t e_ = (call);                                                                  \
    if (e_ != cudaSuccess)                                                                    \
      return fvfail(e_ == cudaErrorMemoryAllocation ? FB_ENOMEM : FB_ECUDA, "%s: %s", #call, \
                    cudaGetErrorString(e_));                                                  \
  } while (0)

constexpr int kFvThreads = 256;       // the other kernels
constexpr int kFvStepThreads = 1024;
constexpr int kFvWidth = 64;  // words per chunk at most

// V instances of a row of r.
template <int V>
struct FvVec {
  float a[V];
};
template <int V>
__device__ __forceinline__ FvVec<V> fv_load(const float *p) {
  FvVec<V> x;
  if constexpr (V == 4) {
    const float4 q = *(const float4 *)p;
    x.a[0] = q.x, x.a[1] = q.y, x.a[2] = q.z, x.a[3] = q.w;
  } else if constexpr (V == 2) {
    const float2 q = *(const float2 *)p;
    x.a[0] = q.x, x.a[1] = q.y;
  } else {
    x.a[0] = *p;
  }
  return x;
}
template <int V>
__device__ __forceinline__ void fv_store(float *p, const FvVec<V> &x) {
  if constexpr (V == 4) *(float4 *)p = make_float4(x.a[0], x.a[1], x.a[2], x.a[3]);
  else if constexpr (V == 2) *(float2 *)p = make_float2(x.a[0], x.a[1]);
  else *p = x.a[0];
}
// Two records {source, weight bits}; each is read once per step, so they are not kept in L1.
__device__ __forceinline__ int4 fv_records(const int4 *p) {
  int4 q;
  asm volatile("ld.global.nc.L1::no_allocate.v4.s32 {%0, %1, %2, %3}, [%4];"
               : "=r"(q.x), "=r"(q.y), "=r"(q.z), "=r"(q.w)
               : "l"(p));
  return q;
}
// acc += w * r, two roundings per instance (lif.c:90-91), two instances per instruction. A source
// that is skipped there (v <= 0) has r = 0 and adds a zero here, which leaves the sum as it is (a
// sum that starts at +0 is never -0) unless the weight is not finite: then it is skipped. The
// product is a packed fma with an addend of -0 that the compiler does not know (`nz`): it contracts
// a packed mul and add to one fma, whatever rounding they name.
enum { kFvV, kFvR, kFvFinite };  // gathers v; r; r, every weight finite
template <int V, int MODE>
__device__ __forceinline__ void fv_add(FvVec<V> &acc, float w, const FvVec<V> &r, float nz) {
  if constexpr (MODE == kFvFinite && V >= 2) {
#pragma unroll
    for (int u = 0; u < V; u += 2)
      asm("{\n\t.reg .b64 a, w, r, z;\n\tmov.b64 a, {%0, %1};\n\tmov.b64 w, {%2, %2};\n\tmov.b64 r, {%3, %4};\n\t"
          "mov.b64 z, {%5, %5};\n\tfma.rn.f32x2 r, w, r, z;\n\tadd.rn.f32x2 a, a, r;\n\tmov.b64 {%0, %1}, a;\n\t}"
          : "+f"(acc.a[u]), "+f"(acc.a[u + 1])
          : "f"(w), "f"(r.a[u]), "f"(r.a[u + 1]), "f"(nz));
  } else {
#pragma unroll
    for (int u = 0; u < V; u++)
      if (MODE == kFvFinite || (MODE == kFvR ? r.a[u] != 0.f : !(r.a[u] <= 0.f))) acc.a[u] = __fadd_rn(acc.a[u], __fmul_rn(w, r.a[u]));
  }
}

// The update of V instances of a target (lif.c:92: v += kdt * (-v + bias + acc + x), one rounding per
// operation in C order) and the r that the next step gathers.
template <int V>
__device__ __forceinline__ void fv_update(int32_t i, int32_t b0, int32_t B, int32_t pitch, const FvVec<V> &acc,
                                          const float *bias, const float *kdt, float *rout, const float *vin, float *vout,
                                          const float *x) {
  const float bi = __ldg(bias + i), kd = __ldg(kdt + i);
  const int64_t o = (int64_t)i * B + b0;
  FvVec<V> v0, xi, out;
  const bool whole = B % V == 0;  // v and x in vectors: their rows are whole ones
  if (whole) {
    v0 = fv_load<V>(vin + o);
    xi = fv_load<V>(x + o);
  }
#pragma unroll
  for (int u = 0; u < V; u++) {
    if (!whole) v0.a[u] = b0 + u < B ? vin[o + u] : 0.f, xi.a[u] = b0 + u < B ? x[o + u] : 0.f;
    const float s = __fadd_rn(__fadd_rn(__fadd_rn(-v0.a[u], bi), acc.a[u]), xi.a[u]);
    v0.a[u] = __fadd_rn(v0.a[u], __fmul_rn(kd, s));
    if (!whole && b0 + u < B) vout[o + u] = v0.a[u];
    out.a[u] = v0.a[u] <= 0.f || b0 + u >= B ? 0.f : v0.a[u];
  }
  if (whole) fv_store<V>(vout + o, v0);
  if (rout) fv_store<V>(rout + (int64_t)i * pitch + b0, out);
}

// One step, bound by the L1's wavefronts and the latency of its misses. A lane takes V instances of a
// target: wider gathers mean fewer of them (64 eyes of the full network: 38 us a step; a thread per
// instance, its load and issue slots full, took 74; 16 eyes 18.5 and 24.6), where there are enough
// of them to fill the lanes (fv_width). The instances are cut into `chunks` of `width` vectors, and
// each block takes a run of neighbouring targets in one chunk, so that the sources that a block's
// targets share stay in its L1. Rows of `gin` hold `pitch` words, rows of `rout` `rpitch`.
template <int V, int MODE>
__global__ void __launch_bounds__(kFvStepThreads, 1)
    fv_step_kernel(int32_t N, int32_t B, int32_t pitch, int32_t rpitch, int32_t width, int32_t chunks,
                   const uint32_t *__restrict__ ptr, const int4 *__restrict__ rec, const float *__restrict__ bias,
                   const float *__restrict__ kdt, const float *__restrict__ gin, float *__restrict__ rout, const float *vin, float *vout,
                   const float *__restrict__ x, float nz) {
  const int64_t row = (int64_t)N * width, per = (row * chunks + gridDim.x - 1) / gridDim.x;
  const int64_t t0 = per * blockIdx.x, t1 = min(t0 + per, row * chunks);
  int32_t ch = (int32_t)(t0 / row);
  int64_t k = t0 + threadIdx.x - ch * row;
  for (int64_t t = t0 + threadIdx.x; t < t1; t += blockDim.x, k += blockDim.x) {
    for (; k >= row; k -= row) ch++;
    const int32_t i = row >> 32 ? (int32_t)(k / width) : (int32_t)((uint32_t)k / (uint32_t)width);
    const int32_t b0 = (ch * width + (int32_t)(k - (int64_t)i * width)) * V;
    if (b0 >= B) continue;
    const float *src = gin + b0;
    FvVec<V> acc;
#pragma unroll
    for (int u = 0; u < V; u++) acc.a[u] = 0.f;
    const uint32_t hi = __ldg(ptr + i + 1);
    uint32_t g = __ldg(ptr + i);  // in units of four records
    // eight in-edges per round: their loads are issued together, the sum stays in edge order
    for (; g + 2 <= hi; g += 2) {
      int4 q[4];
      FvVec<V> r[8];
#pragma unroll
      for (int u = 0; u < 4; u++) q[u] = fv_records(rec + 2 * (size_t)g + u);
#pragma unroll
      for (int u = 0; u < 4; u++) {
        r[2 * u] = fv_load<V>(src + (int64_t)q[u].x * pitch);
        r[2 * u + 1] = fv_load<V>(src + (int64_t)q[u].z * pitch);
      }
#pragma unroll
      for (int u = 0; u < 4; u++) {
        fv_add<V, MODE>(acc, __int_as_float(q[u].y), r[2 * u], nz);
        fv_add<V, MODE>(acc, __int_as_float(q[u].w), r[2 * u + 1], nz);
      }
    }
    if (g < hi) {
      int4 q[2];
      FvVec<V> r[4];
#pragma unroll
      for (int u = 0; u < 2; u++) q[u] = fv_records(rec + 2 * (size_t)g + u);
#pragma unroll
      for (int u = 0; u < 2; u++) {
        r[2 * u] = fv_load<V>(src + (int64_t)q[u].x * pitch);
        r[2 * u + 1] = fv_load<V>(src + (int64_t)q[u].z * pitch);
      }
#pragma unroll
      for (int u = 0; u < 2; u++) {
        fv_add<V, MODE>(acc, __int_as_float(q[u].y), r[2 * u], nz);
        fv_add<V, MODE>(acc, __int_as_float(q[u].w), r[2 * u + 1], nz);
      }
    }
    fv_update<V>(i, b0, B, rpitch, acc, bias, kdt, rout, vin, vout, x);
  }
}

// r of the state as it is now (it can be written from outside between calls).
__global__ void fv_rectify_kernel(int32_t N, int32_t B, int32_t pitch, const float *v, float *r) {
  const int64_t total = (int64_t)N * pitch;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int32_t i = (int32_t)(t / pitch), b = (int32_t)(t - (int64_t)i * pitch);
    const float a = b < B ? v[(int64_t)i * B + b] : 0.f;
    r[t] = a <= 0.f ? 0.f : a;
  }
}

// v[b] = bias (src/flyvis.js:24), every instance when b < 0.
__global__ void fv_reset_kernel(int32_t N, int32_t B, int32_t b, const float *bias, float *v) {
  const int64_t total = (int64_t)N * B;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int32_t i = (int32_t)(t / B), c = (int32_t)(t - (int64_t)i * B);
    if (b < 0 || c == b) v[t] = bias[i];
  }
}

// x[idx[k]] of instance b = values[k] (src/flyvis.js:21). The reference loop leaves a repeated
// index at its last value: each index's last list position is claimed first (win[], reset to -1
// by the writes).
__global__ void fv_claim_kernel(int32_t N, int32_t n, const int32_t *idx, int32_t *win, int32_t *err) {
  for (int32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    const int32_t i = idx[k];
    if (i < 0 || i >= N) atomicCAS(err, 0, FB_EINVAL);
    else atomicMax(win + i, k);
  }
}
__global__ void fv_input_kernel(int32_t N, int32_t B, int32_t b, int32_t n, const int32_t *idx, const float *values,
                                float *x, int32_t *win) {
  for (int32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    const int32_t i = idx[k];
    if (i < 0 || i >= N || win[i] != k) continue;
    x[(int64_t)i * B + b] = values[k];
    win[i] = -1;  // ready for the next list (only the winner of i gets here)
  }
}

// Both for a list that one block holds in registers, read from the host's pinned copy: idx, then
// values, then the error word that it sets.
constexpr int kFvListThreads = 1024, kFvListEach = 8, kFvList = kFvListThreads * kFvListEach;
__global__ void __launch_bounds__(kFvListThreads) fv_list_kernel(int32_t N, int32_t B, int32_t b, int32_t n, const int32_t *list,
                                                                 float *x, int32_t *win, int32_t *err) {
  int32_t idx[kFvListEach];
  float val[kFvListEach];
#pragma unroll
  for (int m = 0; m < kFvListEach; m++) {
    const int k = threadIdx.x + m * kFvListThreads;
    idx[m] = k < n ? list[k] : -1;
    val[m] = k < n ? __int_as_float(list[n + k]) : 0.f;
    if (k < n && (idx[m] < 0 || idx[m] >= N)) {
      *err = FB_EINVAL;
      idx[m] = -1;
    }
  }
#pragma unroll
  for (int m = 0; m < kFvListEach; m++)
    if (idx[m] >= 0) atomicMax(win + idx[m], (int)threadIdx.x + m * kFvListThreads);
  __syncthreads();
#pragma unroll
  for (int m = 0; m < kFvListEach; m++) {
    if (idx[m] < 0 || __ldcg(win + idx[m]) != (int)threadIdx.x + m * kFvListThreads) continue;
    x[(int64_t)idx[m] * B + b] = val[m];
  }
  __syncthreads();
#pragma unroll
  for (int m = 0; m < kFvListEach; m++)
    if (idx[m] >= 0) win[idx[m]] = -1;
}

// Instance b's N values out of (or into) the instance-minor layout.
__global__ void fv_gather_kernel(int32_t N, int32_t B, int32_t b, const float *src, float *dst) {
  for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) dst[i] = src[(int64_t)i * B + b];
}
__global__ void fv_scatter_kernel(int32_t N, int32_t B, int32_t b, const float *src, float *dst) {
  for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) dst[(int64_t)i * B + b] = src[i];
}

}  // namespace

struct fb_flyvis {
  int32_t N = 0, B = 0;
  int64_t E = 0;
  uint32_t *ptr = nullptr;  // per target: its records, in units of four
  int4 *rec = nullptr;      // two records {source, weight} each; row N is the padding's source
  float *bias = nullptr, *kdt = nullptr;
  float *v[2] = {nullptr, nullptr};       // [N + 1][B]; v[cur] is the state, row N zero
  float *r[2] = {nullptr, nullptr};       // [N + 1][pitch], row N zero; null without room for them
  float *x = nullptr, *scratch = nullptr; // [N][B], [N]
  int32_t vec = 1, pitch = 1;             // instances per lane, words per row of r
  bool finite = true;                     // every weight is
  int32_t *idxBuf = nullptr, *err = nullptr, *win = nullptr;
  int64_t idxCap = 0;
  int32_t *list = nullptr;  // pinned: kFvList indices and values, the error word; null: none yet
  int32_t lists = 0;        // host lists set until it was there; kFvPinAfter: none to be had
  int cur = 0, grid = 0, sms = 0;
  cudaStream_t st = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  float lastMs = 0.f;
};

extern "C" int fb_flyvis_destroy(fb_flyvis *f) {
  if (!f) return FB_OK;
  if (f->st) cudaStreamSynchronize(f->st);
  for (void *p : {(void *)f->ptr, (void *)f->rec, (void *)f->bias, (void *)f->kdt, (void *)f->v[0], (void *)f->v[1], (void *)f->r[0],
                  (void *)f->r[1], (void *)f->x, (void *)f->scratch, (void *)f->idxBuf, (void *)f->err, (void *)f->win})
    if (p) cudaFree(p);
  if (f->list) cudaFreeHost(f->list);
  if (f->ev0) cudaEventDestroy(f->ev0);
  if (f->ev1) cudaEventDestroy(f->ev1);
  if (f->st) cudaStreamDestroy(f->st);
  delete f;
  return FB_OK;
}

extern "C" int fb_flyvis_create(int32_t N, int64_t E, const int32_t *indptr, const int32_t *target, const float *weight,
                                const float *bias, const float *kdt, int32_t B, fb_flyvis **out) {
  if (!out || N <= 0 || E < 0 || B <= 0 || !indptr || (E && (!target || !weight)) || !bias || !kdt)
    return fvfail(FB_EINVAL, "fb_flyvis_create: bad arguments (N=%d E=%lld B=%d)", N, (long long)E, B);
  if (E > INT32_MAX) return fvfail(FB_EINVAL, "fb_flyvis_create: %lld edges (at most 2^31 - 1)", (long long)E);
  *out = nullptr;
  // the transposed graph, in-edges of each target in ascending edge id (lif.c's summation order)
  // (each target's list padded to whole groups of four with zero weights from the zero row N)
  std::vector<int32_t> ip(N + 1), tg((size_t)std::max<int64_t>(E, 1)), deg(N, 0);
  std::vector<float> w((size_t)std::max<int64_t>(E, 1));
  std::vector<uint32_t> cp(N + 1, 0);
  bool finite = true;
  auto copy_in = [](void *dst, const void *src, size_t bytes) {
    return cudaMemcpy(dst, src, bytes, cudaMemcpyDefault) == cudaSuccess;
  };
  if (!copy_in(ip.data(), indptr, (size_t)(N + 1) * 4) || (E && (!copy_in(tg.data(), target, (size_t)E * 4) ||
                                                                 !copy_in(w.data(), weight, (size_t)E * 4))))
    return fvfail(FB_ECUDA, "fb_flyvis_create: reading the model failed");
  if (ip[0] != 0 || ip[N] != E) return fvfail(FB_EINVAL, "fb_flyvis_create: indptr[0]=%d indptr[N]=%d E=%lld", ip[0], ip[N], (long long)E);
  for (int32_t j = 0; j < N; j++)
    if (ip[j + 1] < ip[j]) return fvfail(FB_EINVAL, "fb_flyvis_create: indptr decreases at %d", j);
  for (int64_t k = 0; k < E; k++) {
    if (tg[k] < 0 || tg[k] >= N) return fvfail(FB_EINVAL, "fb_flyvis_create: target[%lld]=%d", (long long)k, tg[k]);
    deg[tg[k]]++;
    finite = finite && std::isfinite(w[k]);
  }
  for (int32_t i = 0; i < N; i++) cp[i + 1] = cp[i] + (uint32_t)((deg[i] + 3) / 4);
  std::vector<int2> rec((size_t)std::max<uint32_t>(cp[N], 1) * 4, make_int2(N, 0));
  {
    std::vector<size_t> fill(N);
    for (int32_t i = 0; i < N; i++) fill[i] = (size_t)cp[i] * 4;
    for (int32_t j = 0; j < N; j++)
      for (int32_t k = ip[j]; k < ip[j + 1]; k++) {
        int32_t bits;
        memcpy(&bits, &w[k], 4);
        rec[fill[tg[k]]++] = make_int2(j, bits);
      }
  }
  fb_flyvis *f = new fb_flyvis;
  f->N = N;
  f->B = B;
  f->E = E;
  f->finite = finite;
  f->vec = B >= 3 ? 4 : B;
  f->pitch = (B + f->vec - 1) / f->vec * f->vec;
  auto bail = [&](int rc) {
    fb_flyvis_destroy(f);
    return rc;
  };
  const size_t nb = (size_t)N * B;
  const size_t rb = (size_t)(N + 1) * f->pitch * 4, vb = nb * 4 + (size_t)B * 4;
  if (cudaMalloc(&f->ptr, (size_t)(N + 1) * 4) != cudaSuccess || cudaMalloc(&f->rec, rec.size() * 8) != cudaSuccess ||
      cudaMalloc(&f->bias, (size_t)N * 4) != cudaSuccess || cudaMalloc(&f->kdt, (size_t)N * 4) != cudaSuccess ||
      cudaMalloc(&f->v[0], vb) != cudaSuccess || cudaMalloc(&f->v[1], vb) != cudaSuccess ||
      cudaMalloc(&f->x, nb * 4) != cudaSuccess ||
      cudaMalloc(&f->scratch, (size_t)N * 4) != cudaSuccess || cudaMalloc(&f->err, 4) != cudaSuccess ||
      cudaMalloc(&f->win, (size_t)N * 4) != cudaSuccess)
    return bail(fvfail(FB_ENOMEM, "fb_flyvis_create: device allocation failed (N=%d E=%lld B=%d)", N, (long long)E, B));
  if (cudaMemcpy(f->ptr, cp.data(), (size_t)(N + 1) * 4, cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemcpy(f->rec, rec.data(), rec.size() * 8, cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemset(f->v[0], 0, vb) != cudaSuccess || cudaMemset(f->v[1], 0, vb) != cudaSuccess ||
      cudaMemcpy(f->bias, bias, (size_t)N * 4, cudaMemcpyDefault) != cudaSuccess ||
      cudaMemcpy(f->kdt, kdt, (size_t)N * 4, cudaMemcpyDefault) != cudaSuccess || cudaMemset(f->x, 0, nb * 4) != cudaSuccess ||
      cudaMemset(f->win, 0xff, (size_t)N * 4) != cudaSuccess ||
      cudaMemset(f->err, 0, 4) != cudaSuccess)
    return bail(fvfail(FB_ECUDA, "fb_flyvis_create: upload failed"));
  if (cudaStreamCreateWithFlags(&f->st, cudaStreamNonBlocking) != cudaSuccess || cudaEventCreate(&f->ev0) != cudaSuccess ||
      cudaEventCreate(&f->ev1) != cudaSuccess)
    return bail(fvfail(FB_ECUDA, "fb_flyvis_create: stream setup failed"));
  // without room for r every step gathers v
  if (cudaMalloc(&f->r[0], rb) != cudaSuccess || cudaMalloc(&f->r[1], rb) != cudaSuccess) {
    if (f->r[0]) cudaFree(f->r[0]);
    f->r[0] = f->r[1] = nullptr;
    cudaGetLastError();
  } else if (cudaMemset(f->r[0], 0, rb) != cudaSuccess || cudaMemset(f->r[1], 0, rb) != cudaSuccess) {
    return bail(fvfail(FB_ECUDA, "fb_flyvis_create: clearing the state failed"));
  }
  int dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&f->sms, cudaDevAttrMultiProcessorCount, dev);
  const int64_t blocks = ((int64_t)nb + kFvThreads - 1) / kFvThreads;
  f->grid = (int)std::max<int64_t>(1, std::min<int64_t>(blocks, (int64_t)f->sms * 8));
  fv_reset_kernel<<<f->grid, kFvThreads, 0, f->st>>>(N, B, -1, f->bias, f->v[0]);
  if (cudaStreamSynchronize(f->st) != cudaSuccess) return bail(fvfail(FB_ECUDA, "fb_flyvis_create: reset failed"));
  *out = f;
  return FB_OK;
}

static int fv_check(fb_flyvis *f, int32_t b, const char *fn, bool allowAll = false) {
  if (!f) return fvfail(FB_EINVAL, "%s: null handle", fn);
  if (b >= f->B || (b < 0 && !allowAll)) return fvfail(FB_EINVAL, "%s: instance %d out of range [0, %d)", fn, b, f->B);
  return FB_OK;
}

static int fv_sync_err(fb_flyvis *f, const char *fn) {
  int32_t err = 0;
  FVCU(cudaMemcpyAsync(&err, f->err, 4, cudaMemcpyDeviceToHost, f->st));
  FVCU(cudaStreamSynchronize(f->st));
  if (err) {
    cudaMemset(f->err, 0, 4);
    return fvfail(err, "%s: an index out of range was skipped", fn);
  }
  return FB_OK;
}

extern "C" int fb_flyvis_reset(fb_flyvis *f, int32_t b) {
  int rc = fv_check(f, b, "fb_flyvis_reset", true);
  if (rc) return rc;
  fv_reset_kernel<<<f->grid, kFvThreads, 0, f->st>>>(f->N, f->B, b, f->bias, f->v[f->cur]);
  FVCU(cudaGetLastError());
  FVCU(cudaStreamSynchronize(f->st));
  return FB_OK;
}

// The pinned copy costs 300 us and saves a list 5 to 9: it comes with this many lists. (A model of 100
// neurons, created and given one list: 670 us with a copy made at creation, now 390.)
constexpr int32_t kFvPinAfter = 32;

// Whether p is plain host memory.
static bool fv_host(const void *p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeUnregistered || a.type == cudaMemoryTypeHost;
}

extern "C" int fb_flyvis_set_input(fb_flyvis *f, int32_t b, int32_t n, const int32_t *idx, const float *values) {
  int rc = fv_check(f, b, "fb_flyvis_set_input");
  if (rc) return rc;
  if (n < 0 || (n && (!idx || !values))) return fvfail(FB_EINVAL, "fb_flyvis_set_input: bad list");
  if (n == 0) return FB_OK;
  // one kernel that reads the pinned copy, where a block holds the list (5,768 values: 31 us a call,
  // with two copies, two kernels and the error word's copy 36)
  const bool small = n <= kFvList && fv_host(idx) && fv_host(values);
  if (small && f->lists < kFvPinAfter && ++f->lists == kFvPinAfter &&
      cudaHostAlloc((void **)&f->list, (2 * kFvList + 1) * 4, cudaHostAllocDefault) != cudaSuccess) {
    f->list = nullptr;
    cudaGetLastError();
  }
  if (f->list && small) {
    int32_t *err = f->list + 2 * n;
    memcpy(f->list, idx, (size_t)n * 4);
    memcpy(f->list + n, values, (size_t)n * 4);
    *err = 0;
    fv_list_kernel<<<1, kFvListThreads, 0, f->st>>>(f->N, f->B, b, n, f->list, f->x, f->win, err);
    FVCU(cudaGetLastError());
    FVCU(cudaStreamSynchronize(f->st));
    if (*err) return fvfail(*err, "fb_flyvis_set_input: an index out of range was skipped");
    return FB_OK;
  }
  if (n > f->idxCap) {
    if (f->idxBuf) cudaFree(f->idxBuf);
    f->idxBuf = nullptr;
    FVCU(cudaMalloc(&f->idxBuf, (size_t)n * 8));
    f->idxCap = n;
  }
  float *vals = (float *)(f->idxBuf + n);
  FVCU(cudaMemcpyAsync(f->idxBuf, idx, (size_t)n * 4, cudaMemcpyDefault, f->st));
  FVCU(cudaMemcpyAsync(vals, values, (size_t)n * 4, cudaMemcpyDefault, f->st));
  const int g = std::max(1, std::min(f->grid, (n + 255) / 256));
  fv_claim_kernel<<<g, 256, 0, f->st>>>(f->N, n, f->idxBuf, f->win, f->err);
  fv_input_kernel<<<g, 256, 0, f->st>>>(f->N, f->B, b, n, f->idxBuf, vals, f->x, f->win);
  FVCU(cudaGetLastError());
  return fv_sync_err(f, "fb_flyvis_set_input");
}

extern "C" int fb_flyvis_write(fb_flyvis *f, int32_t field, int32_t b, const float *values) {
  int rc = fv_check(f, b, "fb_flyvis_write");
  if (rc) return rc;
  if (!values || (field != FB_FV_V && field != FB_FV_X)) return fvfail(FB_EINVAL, "fb_flyvis_write: bad field %d", field);
  FVCU(cudaMemcpyAsync(f->scratch, values, (size_t)f->N * 4, cudaMemcpyDefault, f->st));
  fv_scatter_kernel<<<std::min(f->grid, (f->N + 255) / 256), 256, 0, f->st>>>(f->N, f->B, b, f->scratch,
                                                                            field == FB_FV_V ? f->v[f->cur] : f->x);
  FVCU(cudaGetLastError());
  FVCU(cudaStreamSynchronize(f->st));
  return FB_OK;
}

extern "C" int fb_flyvis_read(fb_flyvis *f, int32_t field, int32_t b, float *out) {
  int rc = fv_check(f, b, "fb_flyvis_read");
  if (rc) return rc;
  if (!out || (field != FB_FV_V && field != FB_FV_X)) return fvfail(FB_EINVAL, "fb_flyvis_read: bad field %d", field);
  fv_gather_kernel<<<std::min(f->grid, (f->N + 255) / 256), 256, 0, f->st>>>(f->N, f->B, b,
                                                                           field == FB_FV_V ? f->v[f->cur] : f->x, f->scratch);
  FVCU(cudaGetLastError());
  FVCU(cudaMemcpyAsync(out, f->scratch, (size_t)f->N * 4, cudaMemcpyDefault, f->st));
  FVCU(cudaStreamSynchronize(f->st));
  return FB_OK;
}

// Instances per lane, at most `most`: one while all (target, instance) pairs take a third of the chip's
// 311,296 resident threads, two until they take all of them, then four. Microseconds for 20 steps at
// 1 / 2 / 4: 3,000 neurons and 4 eyes 136 / 175 / 217, 6,000 and 16 (96,000 pairs) 167 / 175 / 177, 20,000
// and 6 (120,000) 214 / 202 / 263, 24,000 and 8 (192,000) 219 / 216 / 226, 45,669 and 6 (274,000) 299 / 283 /
// 298, 24,000 and 13 (312,000) 299 / 299 / 295, 45,669 and 8 (365,000) 341 / 328 / 299, 45,669 and 64 1,332 /
// 919 / 785.
static int32_t fv_width(const fb_flyvis *f, int32_t most) {
  const int64_t pairs = (int64_t)f->N * f->B;
  return pairs <= 100000 ? 1 : std::min(most, pairs <= 300000 ? 2 : 4);
}

// One step from `gin` (rows of `pitch` words). The lanes are those of the instances, not of the rows'
// padding (20,000 neurons and 5 eyes, 20 steps 265 us with lanes for it, 198 without). A chunk is at most
// kFvWidth words wide whatever the lane's width: in chunks of 16 words a row of 17 eyes was read in two
// parts (the full network, a call of one step: 43 us, now 37). Blocks of 1,024 threads, one per SM, leave
// one block to balance a run of targets in; with fewer lanes than that, blocks of 256 spread them over the
// SMs (8 eyes of the full network 14.5 us a step against 18.6, 24 eyes 22.7 against 20.9).
static void fv_launch(fb_flyvis *f, int V, int mode, int32_t pitch, const float *gin, float *rout, float *vout) {
  const int32_t vecs = (f->B + V - 1) / V, chunks = (vecs * V + kFvWidth - 1) / kFvWidth, width = (vecs + chunks - 1) / chunks;
  const int64_t lanes = (int64_t)f->N * width * chunks;
  const int threads = lanes <= (int64_t)f->sms * kFvStepThreads ? 256 : kFvStepThreads;
  const int grid = (int)std::min<int64_t>((lanes + threads - 1) / threads, (int64_t)f->sms * (kFvStepThreads / threads));
#define FV_PICK(V_)                                                                                        \
  (mode == kFvFinite ? fv_step_kernel<V_, kFvFinite> : mode == kFvR ? fv_step_kernel<V_, kFvR> : fv_step_kernel<V_, kFvV>)
  auto kernel = V == 4 ? FV_PICK(4) : V == 2 ? FV_PICK(2) : FV_PICK(1);
#undef FV_PICK
  kernel<<<grid, threads, 0, f->st>>>(f->N, f->B, pitch, f->pitch, width, chunks, f->ptr, f->rec, f->bias, f->kdt, gin, rout,
                                      f->v[f->cur], vout, f->x, -0.f);
}

extern "C" int fb_flyvis_step(fb_flyvis *f, int32_t nsteps) {
  int rc = fv_check(f, 0, "fb_flyvis_step");
  if (rc) return rc;
  if (nsteps < 0) return fvfail(FB_EINVAL, "fb_flyvis_step: nsteps=%d", nsteps);
  FVCU(cudaEventRecord(f->ev0, f->st));
  // instances per lane from r, and from v, whose rows hold whole vectors of this many
  const int32_t vecR = fv_width(f, f->vec), vecV = fv_width(f, f->B % 4 == 0 ? 4 : f->B % 2 == 0 ? 2 : 1);
  // a first step that would gather one instance per lane where r allows more: the pass that makes r
  // repays itself from some 2.2 million pairs on (the full network, calls of one step without / with it: 35
  // eyes 53 / 53 us, 49 eyes 65 / 63, 97 eyes 118 / 102); two per lane do as well without (66 eyes 66 / 84)
  const bool pass = f->r[0] && vecV == 1 && vecV < vecR && (int64_t)f->N * f->B >= 2200000;
  for (int32_t s = 0, in = 0; s < nsteps; s++) {
    const bool more = f->r[0] && s + 1 < nsteps;
    if (!f->r[0] || (s == 0 && !pass)) {
      fv_launch(f, vecV, kFvV, f->B, f->v[f->cur], more ? f->r[0] : nullptr, f->v[f->cur ^ 1]);
      f->cur ^= 1;
    } else {
      if (s == 0) {
        const int64_t words = (int64_t)f->N * f->pitch;
        const int g = (int)std::min<int64_t>((words + kFvThreads - 1) / kFvThreads, (int64_t)f->sms * 8);
        fv_rectify_kernel<<<g, kFvThreads, 0, f->st>>>(f->N, f->B, f->pitch, f->v[f->cur], f->r[0]);
      }
      fv_launch(f, vecR, f->finite ? kFvFinite : kFvR, f->pitch, f->r[in], more ? f->r[in ^ 1] : nullptr, f->v[f->cur]);
      in ^= 1;
    }
  }
  FVCU(cudaEventRecord(f->ev1, f->st));
  FVCU(cudaGetLastError());
  FVCU(cudaStreamSynchronize(f->st));
  cudaEventElapsedTime(&f->lastMs, f->ev0, f->ev1);
  return FB_OK;
}

extern "C" int fb_flyvis_last_ms(fb_flyvis *f, float *ms) {
  if (!f || !ms) return fvfail(FB_EINVAL, "fb_flyvis_last_ms: null argument");
  *ms = f->lastMs;
  return FB_OK;
}

extern "C" int fb_flyvis_state(fb_flyvis *f, float **v, float **x, int32_t *layout_b) {
  if (!f) return fvfail(FB_EINVAL, "fb_flyvis_state: null handle");
  if (v) *v = f->v[f->cur];
  if (x) *x = f->x;
  if (layout_b) *layout_b = f->B;
  return FB_OK;
}
