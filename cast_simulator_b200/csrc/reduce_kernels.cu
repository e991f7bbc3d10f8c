// Statevector reductions: norm^2 (FP64 accumulation) and scaling.
//
// Replaces src/cpp/cuda/cuda_kernels.cu of narix10yc/cast_simulator
// (normSqPass1/2 at :124-167, scaleKernel at :171-196, C wrappers at :244-254).
// Per-block FP64 partial sums over 128-bit loads go into a device scratch array;
// the launch's last block folds them in a fixed order and writes the result into
// page-locked host memory: one launch and one wait a call (norm of a 16-qubit
// complex128 state 17 us; 27 with a fold kernel and a copy back behind it).
// cast_cuda_norm_squared and cast_cuda_scale run on the legacy default stream, as
// the reference's do (cuda_kernels.cu:236-238), so they order after earlier work
// on blocking streams.
#include "../../include/ffi_cuda.h"
#include "internal.hpp"

#include <mutex>
#include <type_traits>
#include <vector>

namespace cb2 {

namespace {

constexpr int kRedThreads = 256;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// Block-wide sum; result valid in thread 0.
__device__ __forceinline__ double block_sum(double v) {
  __shared__ double part[kRedThreads / 32];
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
  __syncthreads();
  v = threadIdx.x < kRedThreads / 32 ? part[threadIdx.x] : 0.0;
  if (threadIdx.x < 32) v = warp_sum(v);
  return v;
}

__device__ __forceinline__ double sq4(float4 v) {
  return (double)v.x * v.x + (double)v.y * v.y + (double)v.z * v.z + (double)v.w * v.w;
}
__device__ __forceinline__ double sq4(double2 v) { return v.x * v.x + v.y * v.y; }

template <typename T> struct V16;
template <> struct V16<float> { using type = float4; static constexpr int N = 4; };
template <> struct V16<double> { using type = double2; static constexpr int N = 2; };

// Called by every block once its partials are written: true in the block that
// comes last, for which all partials are then visible.  `done` counts the blocks of
// the running launch; the last one puts it back to 0.
__device__ __forceinline__ bool last_block(unsigned *done) {
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    last = atomicAdd(done, 1u) == gridDim.x - 1;
    if (last) *done = 0;
  }
  __syncthreads();
  if (last) __threadfence();
  return last;
}

// out[c] = sum over blocks r of partial[r * cols + c], in a fixed order: the whole
// block a column while they are few, else one warp a column.
__device__ __forceinline__ void fold_columns(const double *partial, int rows, int cols, double *out) {
  if (cols <= 2) {
    for (int c = 0; c < cols; ++c) {
      double v = 0;
      for (int r = threadIdx.x; r < rows; r += kRedThreads) v += __ldcg(&partial[(size_t)r * cols + c]);
      v = block_sum(v);
      if (threadIdx.x == 0) out[c] = v;
      __syncthreads();
    }
    return;
  }
  for (int c = threadIdx.x >> 5; c < cols; c += kRedThreads / 32) {
    double v = 0;
    for (int r = threadIdx.x & 31; r < rows; r += 32) v += __ldcg(&partial[(size_t)r * cols + c]);
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) out[c] = v;
  }
}

// out[0] = sum of squares.
template <typename T>
__global__ void __launch_bounds__(kRedThreads) k_norm(const T *__restrict__ x, uint64_t n,
                                                     double *partial, unsigned *done,
                                                     double *__restrict__ out) {
  using V = typename V16<T>::type;
  constexpr int N = V16<T>::N;
  const V *xv = reinterpret_cast<const V *>(x);
  const uint64_t nv = n / N;
  const uint64_t stride = (uint64_t)gridDim.x * kRedThreads;
  uint64_t i = (uint64_t)blockIdx.x * kRedThreads + threadIdx.x;
  double a0 = 0, a1 = 0, a2 = 0, a3 = 0;
  for (; i + 3 * stride < nv; i += 4 * stride) {
    const V v0 = xv[i], v1 = xv[i + stride], v2 = xv[i + 2 * stride], v3 = xv[i + 3 * stride];
    a0 += sq4(v0);
    a1 += sq4(v1);
    a2 += sq4(v2);
    a3 += sq4(v3);
  }
  for (; i < nv; i += stride) a0 += sq4(xv[i]);
  double acc = (a0 + a1) + (a2 + a3);
  // scalar tail (n not a multiple of the vector width)
  if (blockIdx.x == 0 && threadIdx.x < n - nv * N) {
    const double t = (double)x[nv * N + threadIdx.x];
    acc += t * t;
  }
  acc = block_sum(acc);
  if (threadIdx.x == 0) partial[blockIdx.x] = acc;
  if (last_block(done)) fold_columns(partial, (int)gridDim.x, 1, out);
}

template <typename T>
__global__ void __launch_bounds__(kRedThreads) k_scale(T *__restrict__ x, uint64_t n, T s) {
  using V = typename V16<T>::type;
  constexpr int N = V16<T>::N;
  V *xv = reinterpret_cast<V *>(x);
  const uint64_t nv = n / N;
  const uint64_t stride = (uint64_t)gridDim.x * kRedThreads;
  for (uint64_t i = (uint64_t)blockIdx.x * kRedThreads + threadIdx.x; i < nv; i += stride) {
    V v = xv[i];
    if constexpr (N == 4) {
      v.x *= s; v.y *= s; v.z *= s; v.w *= s;
    } else {
      v.x *= s; v.y *= s;
    }
    xv[i] = v;
  }
  if (blockIdx.x == 0 && threadIdx.x < n - nv * N) x[nv * N + threadIdx.x] *= s;
}

// Scratch of one device: per-block partials, the count of finished blocks and a
// page-locked result buffer that kernels write straight into.  (The count by pointer
// and the checks cost 0.3 us of a 19 us call against a count in a device variable,
// which outlived failed calls.)  Allocated on first use
// and grown on demand (the reference keeps the same kind of process-wide scratch,
// cuda_kernels.cu:203-230).  The mutex serialises its users, each until its result
// has arrived.
std::mutex g_scratch_mu;
constexpr int kMaxScratchDevices = 64;
constexpr int kMaxResult = 4096;  // doubles: the largest marginal
constexpr size_t kCountBytes = 256;
struct Scratch {
  double *partial = nullptr;
  int len = 0;
  unsigned *done = nullptr;  // 0 between launches
  double *result = nullptr;  // page-locked, mapped
};
Scratch g_scratch_dev[kMaxScratchDevices];

Scratch *ensure_scratch(int len, cudaStream_t stream, std::string &err) {
  // a reduction waits for its result, which a stream under capture cannot give; said
  // before anything is enqueued, it leaves the caller's capture (and this scratch) valid
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  if (!cuda_ok(cudaStreamIsCapturing(stream, &capturing), "cudaStreamIsCapturing (reduction)", err)) return nullptr;
  if (capturing != cudaStreamCaptureStatusNone) {
    err = "a reduction cannot run on a stream that is being captured";
    return nullptr;
  }
  int dev = 0;
  if (!cuda_ok(cudaGetDevice(&dev), "cudaGetDevice", err)) return nullptr;
  if (dev < 0 || dev >= kMaxScratchDevices) {
    err = "reduction scratch: device index out of range";
    return nullptr;
  }
  Scratch &s = g_scratch_dev[dev];
  if (!s.result && !cuda_ok(cudaHostAlloc((void **)&s.result, sizeof(double) * kMaxResult,
                                          cudaHostAllocMapped | cudaHostAllocPortable),
                            "cudaHostAlloc (reduction result)", err)) {
    s.result = nullptr;
    return nullptr;
  }
  if (!s.partial || s.len < len) {
    if (s.partial) cudaFree(s.done);
    s.partial = nullptr;
    s.done = nullptr;
    s.len = 0;
    char *base = nullptr;  // the count, then the partials
    if (!cuda_ok(cudaMalloc((void **)&base, kCountBytes + sizeof(double) * len), "cudaMalloc (norm scratch)", err))
      return nullptr;
    // ahead of the caller's launch on this stream, which it waits for
    if (!cuda_ok(cudaMemsetAsync(base, 0, kCountBytes, stream), "cudaMemsetAsync (reduction count)", err)) {
      cudaFree(base);
      return nullptr;
    }
    s.done = reinterpret_cast<unsigned *>(base);
    s.partial = reinterpret_cast<double *>(base + kCountBytes);
    s.len = len;
  }
  return &s;
}

// Launch status and the wait for the result in s.result: always both, since a kernel
// still running would go on using the scratch after the mutex is free.  Where the
// wait itself fails nothing says that the kernel has ended or what it leaves in the
// count: the scratch is given up (not freed) and the next reduction makes its own.
bool fetch_result(Scratch &s, cudaStream_t stream, const char *what, std::string &err) {
  const cudaError_t launched = cudaGetLastError();
  const cudaError_t waited = cudaStreamSynchronize(stream);
  if (waited != cudaSuccess) s = Scratch{};
  return cuda_ok(launched, what, err) && cuda_ok(waited, what, err);
}

unsigned red_grid(uint64_t nv) {
  const uint64_t want = (nv + kRedThreads - 1) / kRedThreads;
  const uint64_t cap = 4ull * sm_count();
  return (unsigned)std::max<uint64_t>(1, std::min(want, cap));
}

template <typename T>
bool norm_sq_impl(const void *x, uint64_t n, double *out, cudaStream_t s, std::string &err) {
  std::lock_guard<std::mutex> lock(g_scratch_mu);
  const unsigned grid = red_grid(n / V16<T>::N);
  Scratch *const sc = ensure_scratch((int)grid, s, err);
  if (!sc) return false;
  k_norm<T><<<grid, kRedThreads, 0, s>>>(static_cast<const T *>(x), n, sc->partial, sc->done,
                                         sc->result);
  if (!fetch_result(*sc, s, "norm", err)) return false;
  *out = sc->result[0];
  return true;
}

template <typename T>
bool scale_impl(void *x, uint64_t n, double scale, cudaStream_t s, std::string &err) {
  const unsigned grid = red_grid(n / V16<T>::N);
  k_scale<T><<<grid, kRedThreads, 0, s>>>(static_cast<T *>(x), n, (T)scale);
  return cuda_ok(cudaGetLastError(), "scale kernel launch", err);
}


// One 16-byte vector of a and b: 2 amplitudes in FP32, 1 in FP64.
__device__ __forceinline__ void inner_add(float4 x, float4 y, double &re, double &im) {
  re += (double)x.x * y.x + (double)x.y * y.y;
  im += (double)x.x * y.y - (double)x.y * y.x;
  re += (double)x.z * y.z + (double)x.w * y.w;
  im += (double)x.z * y.w - (double)x.w * y.z;
}
__device__ __forceinline__ void inner_add(double2 x, double2 y, double &re, double &im) {
  re += x.x * y.x + x.y * y.y;
  im += x.x * y.y - x.y * y.x;
}

// out = <a|b> (re, im).  Bound by the two streams: four 16-byte loads of each in
// flight a thread (one amplitude a time took 556 us for two 27-qubit complex64
// states, 0.60 of the copy peak; now 356 us).
template <typename T>
__global__ void __launch_bounds__(kRedThreads) k_inner(const T *__restrict__ a, const T *__restrict__ b,
                                                      uint64_t n_vec, double *partial, unsigned *done,
                                                      double *__restrict__ out) {
  using V = typename V16<T>::type;
  const V *av = reinterpret_cast<const V *>(a);
  const V *bv = reinterpret_cast<const V *>(b);
  double re[4] = {}, im[4] = {};
  const uint64_t stride = (uint64_t)gridDim.x * kRedThreads;
  uint64_t i = (uint64_t)blockIdx.x * kRedThreads + threadIdx.x;
  for (; i + 3 * stride < n_vec; i += 4 * stride) {
    V x[4], y[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      x[u] = av[i + u * stride];
      y[u] = bv[i + u * stride];
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) inner_add(x[u], y[u], re[u], im[u]);
  }
  for (; i < n_vec; i += stride) inner_add(av[i], bv[i], re[0], im[0]);
  if (n_vec == 0 && blockIdx.x == 0 && threadIdx.x == 0) {  // one complex64 amplitude: half a vector
    re[0] = (double)a[0] * b[0] + (double)a[1] * b[1];
    im[0] = (double)a[0] * b[1] - (double)a[1] * b[0];
  }
  const double r = block_sum((re[0] + re[1]) + (re[2] + re[3]));
  __syncthreads();
  const double m = block_sum((im[0] + im[1]) + (im[2] + im[3]));
  if (threadIdx.x == 0) {
    partial[2 * blockIdx.x] = r;
    partial[2 * blockIdx.x + 1] = m;
  }
  if (last_block(done)) fold_columns(partial, (int)gridDim.x, 2, out);
}

constexpr int kMaxPopQubits = 40;

// |a|^2 of the amplitudes of a 16-byte vector: two in FP32, one in FP64.
__device__ __forceinline__ double prob_lo(float4 v) { return (double)v.x * v.x + (double)v.y * v.y; }
__device__ __forceinline__ double prob_hi(float4 v) { return (double)v.z * v.z + (double)v.w * v.w; }
__device__ __forceinline__ double prob_lo(double2 v) { return v.x * v.x + v.y * v.y; }
__device__ __forceinline__ double prob_hi(double2) { return 0.0; }

// The state as rows of kRedThreads 16-byte vectors: bits of an amplitude's index
// are [row | thread | place in the vector].
template <typename T> constexpr uint32_t vec_bits() { return sizeof(T) == 4 ? 1 : 0; }
template <typename T> constexpr uint32_t row_bits() { return 8 + vec_bits<T>(); }
constexpr uint32_t kPopRowBits = 3;  // rows a thread takes at once, all loads in flight

// Per-qubit populations P(q = 1) and the total norm in one pass, for states of at
// least one chunk of 8 rows.  A thread's place in a row is fixed, so its total
// serves every qubit that indexes threads, at the end; the three lowest row bits
// are split inside a chunk; the chunk's total is added once for every set bit of
// the chunk's index.  That is about five FP64 operations an amplitude, which the
// loads (128 bytes in flight a thread) cover.  27-qubit complex64: 498 -> 190
// us (a thread took 8 consecutive amplitudes, 128 bytes apart from its
// neighbour's).
template <typename T>
__global__ void __launch_bounds__(kRedThreads, 2) k_populations(const T *__restrict__ x, uint32_t n,
                                                               double *partial, unsigned *done,
                                                               double *__restrict__ out) {
  using V = typename V16<T>::type;
  constexpr uint32_t VB = vec_bits<T>(), CB = row_bits<T>() + kPopRowBits;
  constexpr int R = 1 << kPopRowBits;
  const V *xv = reinterpret_cast<const V *>(x);
  const uint64_t n_chunks = 1ull << (n - CB);
  double odd = 0, row[kPopRowBits] = {}, tot = 0, high[kMaxPopQubits - CB] = {};
  for (uint64_t c = blockIdx.x; c < n_chunks; c += gridDim.x) {
    V v[R];
#pragma unroll
    for (int u = 0; u < R; ++u) v[u] = xv[(c * R + u) * kRedThreads + threadIdx.x];
    double s[R];
#pragma unroll
    for (int u = 0; u < R; ++u) {
      s[u] = prob_lo(v[u]);
      if (VB) {
        const double h = prob_hi(v[u]);
        odd += h;
        s[u] += h;
      }
    }
    const double p01 = s[0] + s[1], p23 = s[2] + s[3], p45 = s[4] + s[5], p67 = s[6] + s[7];
    row[0] += (s[1] + s[3]) + (s[5] + s[7]);
    row[1] += p23 + p67;
    const double top = p45 + p67, all = (p01 + p23) + top;
    row[2] += top;
    tot += all;
#pragma unroll
    for (uint32_t q = 0; q < kMaxPopQubits - CB; ++q)
      if ((c >> q) & 1) high[q] += all;
  }
  // columns of this block's partial row: qubits 0 .. n - 1, then the norm
  __shared__ double red[kRedThreads / 32];
  double *mine = partial + (size_t)blockIdx.x * (n + 1);
  auto put = [&](uint32_t column, double v) {
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
      double t = 0;
      for (int w = 0; w < kRedThreads / 32; ++w) t += red[w];
      mine[column] = t;
    }
    __syncthreads();
  };
  if (VB) put(0, odd);
#pragma unroll
  for (uint32_t b = 0; b < 8; ++b) put(VB + b, (threadIdx.x >> b) & 1 ? tot : 0.0);
#pragma unroll
  for (uint32_t b = 0; b < kPopRowBits; ++b) put(row_bits<T>() + b, row[b]);
#pragma unroll
  for (uint32_t q = 0; q < kMaxPopQubits - CB; ++q)
    if (CB + q < n) put(CB + q, high[q]);
  put(n, tot);
  if (last_block(done)) fold_columns(partial, (int)gridDim.x, (int)n + 1, out);
}

// The same for a state below one chunk: one block, amplitude by amplitude.
template <typename T>
__global__ void __launch_bounds__(kRedThreads) k_populations_small(const T *__restrict__ x, uint32_t n,
                                                                  double *__restrict__ out) {
  using V = typename std::conditional<sizeof(T) == 8, double2, float2>::type;
  const V *xv = reinterpret_cast<const V *>(x);
  const int lane = threadIdx.x & 31;
  // a warp a column
  for (uint32_t c = threadIdx.x >> 5; c <= n; c += kRedThreads / 32) {
    double acc = 0;
    for (uint32_t i = lane; i < (1u << n); i += 32)
      if (c == n || ((i >> c) & 1)) {
        const V v = xv[i];
        acc += (double)v.x * v.x + (double)v.y * v.y;
      }
    acc = warp_sum(acc);
    if (lane == 0) out[c] = acc;
  }
}

// Marginal probabilities over m distinct measured qubits (ascending).  A block
// takes rows of one value of the measured row bits (`high`), so a thread's bin
// never changes while it sums: no atomics.  At the end lanes that differ only in
// unmeasured lane bits are summed by shuffles, warps that differ only in
// unmeasured warp bits through shared memory, and the block writes one partial
// per value of the measured bits inside a row.  One FP64 shared atomic an
// amplitude, as before, took 3.2 ms for 5 qubits of a 27-qubit complex64 state
// and 13.4 ms for one high qubit; now 185 and 195 us.
struct MarginalArgs {
  uint64_t row_mask;   // measured bits of the row index
  uint32_t thread_mask;  // measured bits of the thread index
  uint32_t vec_measured;  // the place in the vector is measured
  uint32_t n_rows_log2;
  uint32_t segs_log2;  // blocks that share a value of the measured row bits
  uint32_t high_bits, in_bits;  // popcounts: row_mask; thread_mask + vec
};

__device__ __forceinline__ uint64_t deposit(uint64_t v, uint64_t mask) {
  uint64_t r = 0;
  for (; mask; mask &= mask - 1, v >>= 1)
    if (v & 1) r |= mask & (~mask + 1);
  return r;
}

template <typename T>
__global__ void __launch_bounds__(kRedThreads) k_marginal_rows(const T *__restrict__ x, uint32_t n,
                                                              const MarginalArgs a,
                                                              double *__restrict__ partial) {
  using V = typename V16<T>::type;
  constexpr uint32_t VB = vec_bits<T>();
  const V *xv = reinterpret_cast<const V *>(x);
  const uint64_t high = blockIdx.x >> a.segs_log2, seg = blockIdx.x & ((1u << a.segs_log2) - 1);
  const uint64_t free_mask = ((1ull << a.n_rows_log2) - 1) & ~a.row_mask;
  const uint64_t per = 1ull << (a.n_rows_log2 - a.high_bits - a.segs_log2);  // rows of this block
  // rows in ascending order of their unmeasured bits
  uint64_t r = deposit(seg * per, free_mask);
  const uint64_t fixed = deposit(high, a.row_mask);
  double lo[2] = {}, hi[2] = {};
  const bool live = ((uint64_t)threadIdx.x << VB) < (1ull << n);
  if (live) {
    uint64_t k = 0;
    for (; k + 8 <= per; k += 8) {
      V v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        v[u] = xv[(r | fixed) * kRedThreads + threadIdx.x];
        r = ((r | ~free_mask) + 1) & free_mask;
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        lo[u & 1] += prob_lo(v[u]);
        if (VB) hi[u & 1] += prob_hi(v[u]);
      }
    }
    for (; k < per; ++k) {
      const V v = xv[(r | fixed) * kRedThreads + threadIdx.x];
      r = ((r | ~free_mask) + 1) & free_mask;
      lo[0] += prob_lo(v);
      if (VB) hi[0] += prob_hi(v);
    }
  }
  double p[2] = {lo[0] + lo[1], hi[0] + hi[1]};
  if (!a.vec_measured) p[0] += p[1];
  __shared__ double sm[2][kRedThreads];
#pragma unroll
  for (int v = 0; v < 2; ++v) {
#pragma unroll
    for (int b = 0; b < 5; ++b) {
      const double other = __shfl_xor_sync(0xffffffffu, p[v], 1 << b);
      if (!((a.thread_mask >> b) & 1)) p[v] += other;
    }
    sm[v][threadIdx.x] = p[v];
  }
  __syncthreads();
  const uint32_t warp_free = 0xe0u & ~a.thread_mask;
  for (uint32_t o = threadIdx.x; o < (1u << a.in_bits); o += kRedThreads) {
    const uint32_t v = a.vec_measured ? o & 1 : 0;
    const uint32_t t = (uint32_t)deposit(a.vec_measured ? o >> 1 : o, a.thread_mask);
    double sum = 0;
    uint32_t w = 0;
    do {
      sum += sm[v][t | w];
      w = ((w | ~warp_free) + 1) & warp_free;
    } while (w);
    partial[((uint64_t)blockIdx.x << a.in_bits) + o] = sum;
  }
}

// out[bin] = sum over the segments that share it (bins: measured row bits above
// the measured bits inside a row).
__global__ void __launch_bounds__(kRedThreads) k_marginal_fold(const double *__restrict__ partial,
                                                              uint32_t bins, uint32_t in_bits,
                                                              uint32_t segs_log2, double *__restrict__ out) {
  for (uint32_t b = blockIdx.x * (kRedThreads / 32) + (threadIdx.x >> 5); b < bins;
       b += gridDim.x * (kRedThreads / 32)) {
    const uint32_t high = b >> in_bits, in = b & ((1u << in_bits) - 1);
    double acc = 0;
    for (uint32_t s = threadIdx.x & 31; s < (1u << segs_log2); s += 32)
      acc += partial[((((uint64_t)high << segs_log2) + s) << in_bits) + in];
    acc = warp_sum(acc);
    if ((threadIdx.x & 31) == 0) out[b] = acc;
  }
}

// A table of powers indexed by a popcount (0 .. kMaxPopQubits), passed to the
// kernels by value (328 bytes of kernel parameters).
struct PopcTable {
  double v[kMaxPopQubits + 1];
};

// Amplitude-damping sums on a qubit mask: per block (T, D) with
// T = sum |a_i|^2 and D = sum |a_i|^2 * w^popc(i & mask), w = 1 - gamma
// (the probability weight of "no jump on any masked qubit"); tab.v[c] = w^c.
template <typename T>
__global__ void __launch_bounds__(kRedThreads) k_damp_sums(const T *__restrict__ x, uint32_t n,
                                                          uint64_t mask, const PopcTable tab,
                                                          double *partial, unsigned *done,
                                                          double *__restrict__ out) {
  using V = typename std::conditional<sizeof(T) == 8, double2, float2>::type;
  const V *xv = reinterpret_cast<const V *>(x);
  const uint64_t n_amps = 1ull << n;
  const uint64_t stride = (uint64_t)gridDim.x * kRedThreads;
  double t = 0, d = 0;
  for (uint64_t i = (uint64_t)blockIdx.x * kRedThreads + threadIdx.x; i < n_amps; i += stride) {
    const V v = xv[i];
    const double p = (double)v.x * v.x + (double)v.y * v.y;
    t += p;
    d += p * tab.v[__popcll(i & mask)];
  }
  t = block_sum(t);
  __syncthreads();
  d = block_sum(d);
  if (threadIdx.x == 0) {
    partial[2 * blockIdx.x] = t;
    partial[2 * blockIdx.x + 1] = d;
  }
  if (last_block(done)) fold_columns(partial, (int)gridDim.x, 2, out);
}

// x_i *= scale * s^popc(i & mask): the no-jump branch of amplitude damping on
// the masked qubits (s = sqrt(1 - gamma)) with its renormalisation folded in.
// tab.v[c] = scale * s^c, computed in FP64 on the host.
template <typename T>
__global__ void __launch_bounds__(kRedThreads) k_scale_popc(T *__restrict__ x, uint32_t n, uint64_t mask,
                                                           const PopcTable tab) {
  using V = typename std::conditional<sizeof(T) == 8, double2, float2>::type;
  V *xv = reinterpret_cast<V *>(x);
  const uint64_t n_amps = 1ull << n;
  const uint64_t stride = (uint64_t)gridDim.x * kRedThreads;
  for (uint64_t i = (uint64_t)blockIdx.x * kRedThreads + threadIdx.x; i < n_amps; i += stride) {
    V v = xv[i];
    const T f = (T)tab.v[__popcll(i & mask)];
    v.x *= f;
    v.y *= f;
    xv[i] = v;
  }
}

template <typename T>
__global__ void k_dm_diag(const T *__restrict__ rho, uint32_t n, double *__restrict__ out) {
  const uint64_t dim = 1ull << n;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < dim;
       i += (uint64_t)gridDim.x * blockDim.x)
    out[i] = (double)rho[2 * (i | (i << n))];
}

template <typename T>
bool inner_impl(const void *a, const void *b, uint32_t n, double *re, double *im, cudaStream_t s,
                std::string &err) {
  std::lock_guard<std::mutex> lock(g_scratch_mu);
  const uint64_t vec = (1ull << n) >> vec_bits<T>();
  const unsigned grid = red_grid(vec);
  Scratch *const sc = ensure_scratch(2 * (int)grid, s, err);
  if (!sc) return false;
  k_inner<T><<<grid, kRedThreads, 0, s>>>(static_cast<const T *>(a), static_cast<const T *>(b), vec,
                                          sc->partial, sc->done, sc->result);
  if (!fetch_result(*sc, s, "inner product", err)) return false;
  *re = sc->result[0];
  *im = sc->result[1];
  return true;
}

template <typename T>
bool pop_impl(const void *x, uint32_t n, double *p1, double *norm, cudaStream_t s,
              std::string &err) {
  std::lock_guard<std::mutex> lock(g_scratch_mu);
  constexpr uint32_t CB = row_bits<T>() + kPopRowBits;
  const uint64_t chunks = n >= CB ? 1ull << (n - CB) : 1;
  const unsigned grid = (unsigned)std::min<uint64_t>(chunks, 2ull * sm_count());
  Scratch *const sc = ensure_scratch((int)((n + 1) * grid), s, err);
  if (!sc) return false;
  if (n >= CB)
    k_populations<T><<<grid, kRedThreads, 0, s>>>(static_cast<const T *>(x), n, sc->partial, sc->done,
                                                  sc->result);
  else
    k_populations_small<T><<<1, kRedThreads, 0, s>>>(static_cast<const T *>(x), n, sc->result);
  if (!fetch_result(*sc, s, "populations", err)) return false;
  for (uint32_t q = 0; q < n; ++q) p1[q] = sc->result[q];
  if (norm) *norm = sc->result[n];
  return true;
}

template <typename T>
bool marg_impl(const void *x, uint32_t n, const uint32_t *measured, uint32_t m, double *out,
               cudaStream_t s, std::string &err) {
  // the distinct measured qubits, ascending; the caller's order (and any qubit
  // listed twice) is restored from their bins at the end
  uint64_t mask = 0;
  for (uint32_t j = 0; j < m; ++j) mask |= 1ull << measured[j];
  constexpr uint32_t VB = vec_bits<T>(), RB = row_bits<T>();
  MarginalArgs a{};
  a.vec_measured = VB ? (uint32_t)(mask & 1) : 0;
  a.thread_mask = (uint32_t)((mask >> VB) & (kRedThreads - 1));
  a.row_mask = mask >> RB;
  a.n_rows_log2 = n > RB ? n - RB : 0;
  a.high_bits = (uint32_t)__builtin_popcountll(a.row_mask);
  a.in_bits = (uint32_t)__builtin_popcountll(mask) - a.high_bits;
  // about 8 blocks an SM, each with at least 8 rows where there are that many
  const uint32_t free_rows = a.n_rows_log2 - a.high_bits;
  uint32_t want = 0;
  while ((1u << (a.high_bits + want)) < 8u * (uint32_t)sm_count()) ++want;
  a.segs_log2 = std::min(want, free_rows > 3 ? free_rows - 3 : 0);
  const uint32_t bins = 1u << (a.high_bits + a.in_bits);
  const unsigned grid = 1u << (a.high_bits + a.segs_log2);
  std::lock_guard<std::mutex> lock(g_scratch_mu);
  Scratch *const sc = ensure_scratch((int)(grid << a.in_bits), s, err);
  if (!sc) return false;
  k_marginal_rows<T><<<grid, kRedThreads, 0, s>>>(static_cast<const T *>(x), n, a, sc->partial);
  k_marginal_fold<<<std::min<uint32_t>((bins + 7) / 8, 512), kRedThreads, 0, s>>>(
      sc->partial, bins, a.in_bits, a.segs_log2, sc->result);
  if (!fetch_result(*sc, s, "marginal", err)) return false;
  // out[i]: the bin whose bits are i's at the measured qubits' places
  uint32_t bin[1u << 12], place[12];
  bool listed_once = true;
  for (uint32_t j = 0; j < m; ++j) {
    place[j] = (uint32_t)__builtin_popcountll(mask & ((1ull << measured[j]) - 1));
    for (uint32_t l = 0; l < j; ++l) listed_once = listed_once && measured[l] != measured[j];
  }
  bin[0] = 0;
  out[0] = sc->result[0];
  for (uint32_t i = 1; i < (1u << m); ++i) {
    bin[i] = bin[i & (i - 1)] | 1u << place[__builtin_ctz(i)];
    out[i] = sc->result[bin[i]];
  }
  if (!listed_once)  // bits of one qubit that disagree never occur
    for (uint32_t i = 0; i < (1u << m); ++i)
      for (uint32_t j = 0; j < m; ++j)
        if (((i >> j) & 1) != ((bin[i] >> place[j]) & 1)) out[i] = 0.0;
  return true;
}

PopcTable powers(double base, double first) {
  PopcTable t;
  double f = first;
  for (int c = 0; c <= kMaxPopQubits; ++c) {
    t.v[c] = f;
    f *= base;
  }
  return t;
}

template <typename T>
bool damp_sums_impl(const void *x, uint32_t n, uint64_t mask, double gamma, double *tot, double *wsum,
                    cudaStream_t s, std::string &err) {
  std::lock_guard<std::mutex> lock(g_scratch_mu);
  const unsigned grid = red_grid(1ull << n);
  Scratch *const sc = ensure_scratch(2 * (int)grid, s, err);
  if (!sc) return false;
  k_damp_sums<T><<<grid, kRedThreads, 0, s>>>(static_cast<const T *>(x), n, mask, powers(1.0 - gamma, 1.0),
                                              sc->partial, sc->done, sc->result);
  if (!fetch_result(*sc, s, "damping sums", err)) return false;
  *tot = sc->result[0];
  *wsum = sc->result[1];
  return true;
}

template <typename T>
bool scale_popc_impl(void *x, uint32_t n, uint64_t mask, double sfac, double scale, cudaStream_t s,
                     std::string &err) {
  k_scale_popc<T><<<red_grid(1ull << n), kRedThreads, 0, s>>>(static_cast<T *>(x), n, mask,
                                                               powers(sfac, scale));
  return cuda_ok(cudaGetLastError(), "popcount scale launch", err);
}

template <typename T>
bool dm_impl(const void *rho, uint32_t n, double *out, cudaStream_t s, std::string &err) {
  // into the reductions' scratch: a stream-ordered allocation here is handed back at
  // the synchronise and mapped again by the next call
  std::lock_guard<std::mutex> lock(g_scratch_mu);
  const uint64_t dim = 1ull << n;
  Scratch *const sc = ensure_scratch((int)dim, s, err);
  if (!sc) return false;
  const unsigned grid = (unsigned)std::min<uint64_t>((dim + 255) / 256, 4ull * sm_count());
  k_dm_diag<T><<<grid, 256, 0, s>>>(static_cast<const T *>(rho), n, sc->partial);
  const bool copied =
      cuda_ok(cudaGetLastError(), "dm diagonal launch", err) &&
      cuda_ok(cudaMemcpyAsync(out, sc->partial, sizeof(double) << n, cudaMemcpyDeviceToHost, s),
              "cudaMemcpyAsync (dm diagonal)", err);
  return fetch_result(*sc, s, "dm diagonal", err) && copied;
}

}  // namespace

bool damping_sums(const void *x, uint32_t n, uint8_t precision, uint64_t mask, double gamma,
                  double *tot, double *wsum, cudaStream_t s, std::string &err) {
  if (!aligned16(reinterpret_cast<uint64_t>(x), "statevector pointer", err)) return false;
  if (n == 0 || n > kMaxSvQubits || precision > 1 || !(gamma >= 0.0 && gamma <= 1.0)) {
    err = "damping sums: invalid statevector size, precision or gamma";
    return false;
  }
  return precision == 0 ? damp_sums_impl<float>(x, n, mask, gamma, tot, wsum, s, err)
                        : damp_sums_impl<double>(x, n, mask, gamma, tot, wsum, s, err);
}

bool scale_popc(void *x, uint32_t n, uint8_t precision, uint64_t mask, double sfac, double scale,
                cudaStream_t s, std::string &err) {
  if (!aligned16(reinterpret_cast<uint64_t>(x), "statevector pointer", err)) return false;
  if (n == 0 || n > kMaxSvQubits || precision > 1) {
    err = "popcount scale: invalid statevector size or precision";
    return false;
  }
  return precision == 0 ? scale_popc_impl<float>(x, n, mask, sfac, scale, s, err)
                        : scale_popc_impl<double>(x, n, mask, sfac, scale, s, err);
}

bool norm_squared(const void *x, uint64_t n_scalars, uint8_t precision, double *out,
                  cudaStream_t s, std::string &err) {
  if (!aligned16(reinterpret_cast<uint64_t>(x), "statevector pointer", err)) return false;
  return precision == 0 ? norm_sq_impl<float>(x, n_scalars, out, s, err)
                        : norm_sq_impl<double>(x, n_scalars, out, s, err);
}

bool scale(void *x, uint64_t n_scalars, uint8_t precision, double factor, cudaStream_t s,
           std::string &err) {
  if (!aligned16(reinterpret_cast<uint64_t>(x), "statevector pointer", err)) return false;
  return precision == 0 ? scale_impl<float>(x, n_scalars, factor, s, err)
                        : scale_impl<double>(x, n_scalars, factor, s, err);
}

bool inner_product(const void *a, const void *b, uint32_t n, uint8_t precision, double *re,
                   double *im, cudaStream_t s, std::string &err) {
  if (!aligned16(reinterpret_cast<uint64_t>(a), "first statevector pointer", err) ||
      !aligned16(reinterpret_cast<uint64_t>(b), "second statevector pointer", err))
    return false;
  return precision == 0 ? inner_impl<float>(a, b, n, re, im, s, err)
                        : inner_impl<double>(a, b, n, re, im, s, err);
}

bool qubit_populations(const void *x, uint32_t n, uint8_t precision, double *p1, double *norm,
                       cudaStream_t s, std::string &err) {
  if (!aligned16(reinterpret_cast<uint64_t>(x), "statevector pointer", err)) return false;
  if (n > kMaxPopQubits) {
    err = "populations support at most 40 qubits";
    return false;
  }
  return precision == 0 ? pop_impl<float>(x, n, p1, norm, s, err)
                        : pop_impl<double>(x, n, p1, norm, s, err);
}

bool marginal_probabilities(const void *x, uint32_t n, uint8_t precision, const uint32_t *measured,
                            uint32_t m, double *out, cudaStream_t s, std::string &err) {
  if (!aligned16(reinterpret_cast<uint64_t>(x), "statevector pointer", err)) return false;
  if (m == 0 || m > 12) {
    err = "between 1 and 12 measured qubits are supported";
    return false;
  }
  for (uint32_t j = 0; j < m; ++j)
    if (measured[j] >= n) {
      err = "measured qubit out of range";
      return false;
    }
  return precision == 0 ? marg_impl<float>(x, n, measured, m, out, s, err)
                        : marg_impl<double>(x, n, measured, m, out, s, err);
}

bool dm_populations(const void *rho, uint32_t n, uint8_t precision, double *out, cudaStream_t s,
                    std::string &err) {
  if (!aligned16(reinterpret_cast<uint64_t>(rho), "density-matrix pointer", err)) return false;
  if (2 * n > kMaxSvQubits) {
    err = "density matrix too large";
    return false;
  }
  return precision == 0 ? dm_impl<float>(rho, n, out, s, err) : dm_impl<double>(rho, n, out, s, err);
}

}  // namespace cb2

extern "C" {

int cast_cuda_norm_squared(uint64_t dptr, size_t n_elements, uint8_t precision, double *out_norm_sq,
                           char *err_buf, size_t err_buf_len) {
  if (!out_norm_sq) {
    cb2::write_err(err_buf, err_buf_len, "out_norm_sq must not be null");
    return 1;
  }
  std::string err;
  if (!cb2::norm_squared(reinterpret_cast<const void *>(dptr), n_elements, precision, out_norm_sq,
                         nullptr, err)) {
    cb2::write_err(err_buf, err_buf_len, err);
    return 1;
  }
  cb2::clear_err(err_buf, err_buf_len);
  return 0;
}

int cast_cuda_scale(uint64_t dptr, size_t n_elements, uint8_t precision, double scale,
                    char *err_buf, size_t err_buf_len) {
  std::string err;
  if (!cb2::scale(reinterpret_cast<void *>(dptr), n_elements, precision, scale, nullptr, err)) {
    cb2::write_err(err_buf, err_buf_len, err);
    return 1;
  }
  cb2::clear_err(err_buf, err_buf_len);
  return 0;
}

}  // extern "C"
