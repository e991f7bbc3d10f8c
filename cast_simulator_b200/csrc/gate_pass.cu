// Merged gate passes: several gates of a program applied to the statevector for
// one read and one write of it: dense gates of up to 4 qubits and sparse ones of 5
// to 7, in both precisions.  complex128 first, complex64 below.
//
// A CTA owns a tile: the 2^tb amplitudes whose non-tile qubits are fixed
// (pass_plan.hpp chooses the tile's qubits and its gates).  The tile is copied to
// shared memory with cp.async, every gate of the pass is applied there, one CTA
// barrier between gates, and the tile is written back coalesced.
//
// A pass of two or more gates is bound by the FP64 pipe, not HBM (48 FP64
// multiply-adds an amplitude for a 4-qubit gate in the three-product form, 64 a
// clock and SM).  The gate is therefore a small GEMM on the FP64 tensor pipe
// (mma.sync m8n8k4): the matrix is A (its fragments stay in registers for the
// whole gate), eight gather groups are the N columns of B.  Each amplitude is
// read and written once a gate in shared memory, and a warp issues 24
// instructions per 128 amplitudes of arithmetic where scalar FMAs would take 192
// with a constant-bank operand each, which could not index a list of matrices.
// 30 qubits, depth 20, fused at 4 (88 gates, 18 passes): 481 -> 293 ms; the FP64
// pipe's floor is 217 ms at 1.965 GHz, the passes' traffic 95 ms.  Without any
// global traffic the kernel takes 268 ms, so what is left is the pipe and its
// feeding, not HBM: two tiles a CTA with the next one's copy in flight took 335 ms
// (half the tile), 256 threads a CTA 321, staggered CTAs 294, two blocks a warp at
// once 291, larger MMA shapes (m16n8k8, m16n8k16) 294.
#include "gate_tile.cuh"
#include "pass_plan.hpp"
#include "plan_buffers.hpp"

#include <memory>
#include <mutex>

#include <cuda_pipeline.h>

namespace cb2 {

namespace {

constexpr int kPassThreads = 128;
constexpr int kPassWarps = kPassThreads / 32;
constexpr uint32_t kPassMaxTile = 12;
constexpr uint32_t kPassMinTile = kTileMin64;
constexpr uint32_t kPassLow = 3;      // lowest qubits every tile holds: 128-byte runs

struct PassArgs {
  uint64_t stride[kPassMaxTile];  // tile bit -> amplitude stride
  uint32_t tb, n_gates;
  PassGateArgs g[kMaxPassGates];
};

// NARROW: the pass has gates of 1 or 2 qubits.  Their code and the tests that lead to
// it cost the other gates of small states 25 to 40 ns each (17 qubits, fused at 3:
// 96 -> 105 us), so passes without them run without it.
template <bool NARROW>
__global__ void __launch_bounds__(kPassThreads, 3)
    k_gate_pass(double2 *__restrict__ psi, const double *__restrict__ pool,
                const __grid_constant__ PassArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2 *s = reinterpret_cast<double2 *>(smem_raw);
  const uint32_t tile = 1u << a.tb;
  // where the tile starts: the block index spread over the non-tile qubits
  uint64_t base = blockIdx.x;
  for (uint32_t j = 0; j < a.tb; ++j) {
    const uint64_t lo = a.stride[j] - 1;
    base = ((base & ~lo) << 1) | (base & lo);
  }
  // amplitude offset of tile index i: the strides of its set bits
  uint64_t off = base;
#pragma unroll
  for (int b = 0; b < 7; ++b)
    if ((threadIdx.x >> b) & 1) off += a.stride[b];
  const uint32_t rounds = tile / kPassThreads;
  auto round_off = [&](uint32_t u) {
    uint64_t o = off;
#pragma unroll
    for (int b = 7; b < (int)kPassMaxTile; ++b)
      if ((u >> (b - 7)) & 1) o += a.stride[b];
    return o;
  };
#pragma unroll 8
  for (uint32_t u = 0; u < rounds; ++u)
    __pipeline_memcpy_async(&s[pass_swz(threadIdx.x + u * kPassThreads)], &psi[round_off(u)], 16);
  __pipeline_commit();
  __pipeline_wait_prior(0);
  __syncthreads();
  // the same in every lane, and known to be
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  for (uint32_t gi = 0; gi < a.n_gates; ++gi) {
    const PassGateArgs &g = a.g[gi];
    if (NARROW && g.k == 2) pass_small<kPassWarps, 2, 2>(s, pool + g.mat, g, tile >> 6, warp, lane);
    else if (NARROW && g.k == 1) pass_small<kPassWarps, 1, 4>(s, pool + g.mat, g, tile >> 6, warp, lane);
    else if (g.k == 4) pass_gate4<kPassWarps>(s, pool + g.mat, g, tile >> 7, warp, lane);
    else if (g.k > 4)
      pass_sparse<kPassWarps>(s, reinterpret_cast<const double2 *>(pool + g.mat), g.k, g.sp, a.tb, warp, lane);
    else pass_gate3<kPassWarps>(s, pool + g.mat, g, tile >> 6, warp, lane);
    __syncthreads();
  }
#pragma unroll 8
  for (uint32_t u = 0; u < rounds; ++u) psi[round_off(u)] = s[pass_swz(threadIdx.x + u * kPassThreads)];
}

// ── complex64 ────────────────────────────────────────────────────────────────
//
// The same passes in FP32, bound by the FP32 pipe (59% busy) and shared memory
// (78 to 86% of its wavefronts): 24 packed pair FMAs
// (__ffma2_rn, two rows at once) an amplitude and 4-qubit gate.  A thread takes U
// gather groups and, of a 4-qubit gate, half the rows (its partner for the other
// half is in the same warp and reads the same amplitudes: a broadcast).  It walks
// the columns with all its sums in registers; per column it reads U amplitudes
// from the tile and its rows of the matrix, staged in shared memory one gate
// ahead, at addresses the lanes share.  Whole rows of two groups a thread
// with the matrix read through L1 ran at 0.71 of this (28 qubits, fused at 4:
// 64.3 against 46.8 ms; one gate a pass 56.0).  30 qubits, complex64, depth 20,
// fused at 4: 232 -> 200 ms; 26 qubits fused at 3: 21.4 -> 12.3 ms, at 2: 40.4 ->
// 22.9 ms.  Every row is the same FMA sequence as in the one-gate kernels.
constexpr uint32_t kPass32MaxTile = 13;  // 64 KB: three CTAs an SM
constexpr uint32_t kPass32MinTile = 8;
constexpr uint32_t kPass32Low = 4;       // 128-byte runs

struct PassArgs32 {
  uint64_t stride[kPass32MaxTile];
  uint32_t tb, n_gates;
  PassGateArgs32 g[kMaxPassGates];
};

// NARROW: the pass has 1-qubit gates.
template <bool NARROW>
__global__ void __launch_bounds__(kPassThreads, 3)
    k_gate_pass32(float2 *__restrict__ psi, const float *__restrict__ pool,
                  const __grid_constant__ PassArgs32 a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float *mat = reinterpret_cast<float *>(smem_raw);  // two gates' matrices
  float2 *s = reinterpret_cast<float2 *>(smem_raw + 2 * kPass32MatBytes);
  auto fetch_matrix = [&](uint32_t gi) {
    if (a.g[gi].k > 4) return;  // a sparse gate's entries go to registers
    const float *from = pool + a.g[gi].mat;
    float *to = mat + (gi & 1) * (kPass32MatBytes / 4);
    for (uint32_t i = 4 * threadIdx.x; i < 3u << (2 * a.g[gi].k); i += 4 * kPassThreads)
      __pipeline_memcpy_async(to + i, from + i, 16);
  };
  uint64_t base = blockIdx.x;
  for (uint32_t j = 0; j < a.tb; ++j) {
    const uint64_t lo = a.stride[j] - 1;
    base = ((base & ~lo) << 1) | (base & lo);
  }
  // a thread copies pairs of amplitudes: tile bits 1..7 are its thread index
  uint64_t off = base;
#pragma unroll
  for (int b = 0; b < 7; ++b)
    if ((threadIdx.x >> b) & 1) off += a.stride[b + 1];
  const uint32_t rounds = (1u << a.tb) / (2 * kPassThreads);
  auto round_off = [&](uint32_t u) {
    uint64_t o = off;
#pragma unroll
    for (int b = 8; b < (int)kPass32MaxTile; ++b)
      if ((u >> (b - 8)) & 1) o += a.stride[b];
    return o;
  };
#pragma unroll 8
  for (uint32_t u = 0; u < rounds; ++u)
    __pipeline_memcpy_async(&s[pass_swz32(2 * (threadIdx.x + u * kPassThreads))], &psi[round_off(u)], 16);
  fetch_matrix(0);
  for (uint32_t gi = 0; gi < a.n_gates; ++gi) {
    __pipeline_commit();
    __pipeline_wait_prior(0);
    __syncthreads();  // the gate before is done; this one's matrix (and the tile) are here
    if (gi + 1 < a.n_gates) fetch_matrix(gi + 1);
    const PassGateArgs32 &g = a.g[gi];
    const float *m = mat + (gi & 1) * (kPass32MatBytes / 4);
    if (NARROW && g.k == 1) {
      if (a.tb > 9) pass_gate32<kPassThreads, 1, 1, 4, false>(s, m, g, a.tb);
      else pass_gate32<kPassThreads, 1, 1, 2, false>(s, m, g, a.tb);  // 2 groups a thread at most
    } else if (g.k == 4) pass_gate32<kPassThreads, 4, 2, 2, true>(s, m, g, a.tb);
    else if (g.k > 4)
      pass_sparse<kPassWarps>(s, reinterpret_cast<const float2 *>(pool + g.mat), g.k, g.sp, a.tb,
                              __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), (int)threadIdx.x & 31);
    else if (g.k == 3) pass_gate32<kPassThreads, 3, 1, 4, false>(s, m, g, a.tb);
    else pass_gate32<kPassThreads, 2, 1, 4, false>(s, m, g, a.tb);
  }
  __syncthreads();
#pragma unroll 8
  for (uint32_t u = 0; u < rounds; ++u)
    *reinterpret_cast<float4 *>(&psi[round_off(u)]) =
        *reinterpret_cast<const float4 *>(&s[pass_swz32(2 * (threadIdx.x + u * kPassThreads))]);
}

// ── host side ────────────────────────────────────────────────────────────────

// Allocating, freeing and copying on a private stream is safe while a stream is
// captured; say so, or the capture would refuse it (and be invalid from then on).
struct RelaxedCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

// The runtime calls behind plan_buffers.hpp; a call that fails says why in `err`.
struct PlanApi {
  using Event = cudaEvent_t;
  using Stream = cudaStream_t;
  std::string &err;
  bool done(Event e) { return cudaEventQuery(e) == cudaSuccess; }
  bool record(Event e, Stream s) { return cuda_ok(cudaEventRecord(e, s), "cudaEventRecord (gate pass)", err); }
  bool create(Event &e) {
    return cuda_ok(cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "cudaEventCreate (gate pass)", err);
  }
  void destroy(Event e) { cudaEventDestroy(e); }
  bool id(Stream s, unsigned long long &id) {
    return cuda_ok(cudaStreamGetId(s, &id), "cudaStreamGetId (gate pass)", err);
  }
  bool allocate(size_t bytes, char *&p) {
    return cuda_ok(cudaMalloc((void **)&p, bytes), "cudaMalloc (gate pass matrices)", err);
  }
  void release(char *p) {
    RelaxedCapture relaxed;  // a program may be dropped at any time
    cudaFree(p);
  }
};

PlanBufferPool<PlanApi> &buffer_pool() {
  static auto *p = new PlanBufferPool<PlanApi>(size_t(64) << 20);  // outlives programs destroyed at exit
  return *p;
}

// Copies `bytes` to the device on a stream of its own and waits for that copy
// only: a caller's stream may have long work queued, and the destination is read
// by launches on streams that would not wait for the legacy stream's copy.
bool upload_now(void *dst, const void *src, size_t bytes, std::string &err) {
  static std::mutex mu;
  static std::vector<std::pair<int, cudaStream_t>> streams;
  int dev = 0;
  if (!cuda_ok(cudaGetDevice(&dev), "cudaGetDevice", err)) return false;
  std::lock_guard<std::mutex> lock(mu);
  cudaStream_t s = nullptr;
  for (auto &x : streams)
    if (x.first == dev) s = x.second;
  if (!s) {
    if (!cuda_ok(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking), "cudaStreamCreate", err)) return false;
    streams.emplace_back(dev, s);
  }
  return cuda_ok(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s),
                 "cudaMemcpyAsync (gate pass matrices)", err) &&
         cuda_ok(cudaStreamSynchronize(s), "cudaStreamSynchronize (gate pass matrices)", err);
}

}  // namespace

struct PassPlan {
  std::vector<Pass> passes;
  std::vector<PassArgs> args;   // one per merged pass (complex128)
  std::vector<PassArgs32> args32;  // the same in complex64
  std::vector<int> arg_of;      // pass -> its entry of args, -1 for a single gate
  std::vector<double> pool;     // matrices of every merged gate, as its kernel reads them
  std::vector<float> pool32;    // the same in complex64
  PlanCopies<PlanApi> copies;   // of the matrices, one a device
};

// Tile bits by register size.  Small registers need tiles for every SM more than
// gates in a tile (12 qubits, complex128, fused at 4: 41 us with 2^9 amplitudes a
// tile, 92 with 2^12); large ones take the most that leaves three CTAs an SM.
// The lines are where the measured times of neighbouring sizes cross (brickwork
// of depth 20 fused at 2, 3 and 4, replayed as a graph).
uint32_t pass_tile_bits(uint32_t n, uint8_t precision) {
  if (precision) return n >= 22 ? kPassMaxTile : std::min(n, std::min(11u, std::max(9u, n > 8 ? n - 8 : 0u)));
  return n >= 23 ? kPass32MaxTile : std::min(n, n >= 19 ? 12u : n == 18 ? 11u : 10u);
}

// Which gates may share a pass, and what each saves: dense ones of up to 4 qubits
// and sparse ones (CSR) with few nonzeros a row, whose kernel nothing chose from
// outside.
//
// A complex64 pass is bound by the FP32 pipe, so merging pays only where one-gate
// kernels wait for memory or launches.  Not 4-qubit gates of states of 21 to 23
// qubits, which stay in L2 (22 qubits: 545 us one gate a pass, 646 merged; 20
// qubits 204 and 196; 24 qubits 2934 and 2575).  From 24 qubits a merged pass
// costs about 1.4 one-gate passes for its copy and start plus 0.6 a 4-qubit and
// 0.4 a smaller gate (28 qubits: 14 passes of 83 gates 46.8 ms, 17 passes 49.7 ms,
// one-gate pass 0.67 ms), so it has to save that much.  In complex128 two gates
// already pay (their one-gate passes are nearer to HBM's rate than to the pipe's).
PassGate pass_gate_of(const GateData &g, uint32_t n) {
  PassGate p;
  for (uint32_t b = 0; b < g.k; ++b) p.qubits |= 1ull << g.qubits[b];
  const uint32_t least = g.precision ? kPassMinTile : kPass32MinTile;
  if (n < least || g.d_tc || gate_choice_forced(g)) return p;
  if (g.d_sparse) {  // little arithmetic: a merged gate saves its whole pass
    p.mergeable = sparse_most(g) != 0;
    return p;
  }
  if (g.k > 4) return p;
  p.mergeable = g.precision || g.k < 4 || n <= 20 || n >= 24;
  p.saves = g.precision || n < 24 ? 10 : g.k == 4 ? 4 : 6;
  return p;
}

uint32_t pass_cost(uint32_t n, uint8_t precision) { return precision || n < 24 ? 11 : 14; }

std::vector<Pass> program_passes(const std::vector<GateData> &gates, uint32_t n) {
  if (gates.empty()) return {};
  const uint8_t precision = gates[0].precision;  // one a program
  std::vector<PassGate> g;
  g.reserve(gates.size());
  for (const GateData &x : gates) g.push_back(pass_gate_of(x, n));
  return plan_passes(g, n, pass_tile_bits(n, precision), precision ? kPassLow : kPass32Low, kMaxPassGates,
                     pass_cost(n, precision));
}

PassPlan *make_pass_plan(const std::vector<GateData> &gates, uint32_t n) {
  std::unique_ptr<PassPlan> p(new PassPlan);
  p->passes = program_passes(gates, n);
  const bool f64 = !gates.empty() && gates[0].precision == 1;
  size_t scalars = 0, merged = 0;
  for (const Pass &x : p->passes)
    if (x.tile) {
      ++merged;
      for (uint32_t i : x.gates)
        scalars += gates[i].k > 4 ? (size_t)416 << (gates[i].k - 5) : gates[i].k == 4 ? 3 * 256 : 3 * 64;
    }
  if (f64) {
    p->pool.reserve(scalars);
    p->args.reserve(merged);
  } else {
    p->pool32.reserve(scalars);
    p->args32.reserve(merged);
  }
  int next = 0;
  for (const Pass &x : p->passes) {
    if (!x.tile) {
      p->arg_of.push_back(-1);
      continue;
    }
    std::vector<uint32_t> qubits;
    for (uint32_t q = 0; q < n; ++q)
      if ((x.tile >> q) & 1) qubits.push_back(q);
    const uint32_t tb = (uint32_t)qubits.size();
    if (f64) {
      p->args.emplace_back();
      PassArgs &a = p->args.back();
      std::memset(&a, 0, sizeof(a));
      a.tb = tb;
      a.n_gates = (uint32_t)x.gates.size();
      for (uint32_t j = 0; j < tb; ++j) a.stride[j] = 1ull << qubits[j];
      for (uint32_t i = 0; i < a.n_gates; ++i) {
        const GateData &g = gates[x.gates[i]];
        if (g.k > 4) {
          a.g[i].k = (uint16_t)g.k;
          pack_sparse(g, qubits, pass_swz, p->pool, a.g[i].mat, a.g[i].sp);
        } else {
          pack_gate(place_gate(g, qubits), tb, g.k == 4, p->pool, a.g[i]);
        }
      }
    } else {
      p->args32.emplace_back();
      PassArgs32 &a = p->args32.back();
      std::memset(&a, 0, sizeof(a));
      a.tb = tb;
      a.n_gates = (uint32_t)x.gates.size();
      for (uint32_t j = 0; j < tb; ++j) a.stride[j] = 1ull << qubits[j];
      for (uint32_t i = 0; i < a.n_gates; ++i) {
        const GateData &g = gates[x.gates[i]];
        if (g.k > 4) {
          a.g[i].k = (uint16_t)g.k;
          pack_sparse(g, qubits, pass_swz32, p->pool32, a.g[i].mat, a.g[i].sp);
        } else {
          pack_gate32(place_gate(g, qubits), tb, g.k == 4, p->pool32, a.g[i]);
        }
      }
    }
    p->arg_of.push_back(next++);
  }
  return p.release();
}

void free_pass_plan(PassPlan *p) {
  if (!p) return;
  std::string err;
  PlanApi api{err};
  p->copies.give_all(api, buffer_pool());
  delete p;
}

bool upload_pass_plan(PassPlan &p, std::string &err) {
  const size_t bytes = p.pool.size() * sizeof(double) + p.pool32.size() * sizeof(float);
  int dev = 0;
  if (!bytes) return true;
  if (!cuda_ok(cudaGetDevice(&dev), "cudaGetDevice", err)) return false;
  if (p.copies.on(dev)) return true;
  const void *src = p.pool.empty() ? (const void *)p.pool32.data() : (const void *)p.pool.data();
  RelaxedCapture relaxed;
  // the shared-memory limit is a kernel's on one device; tiles that launch without
  // raising it do not wait for the calls
  auto opt_in = [&](auto kernel, size_t most) {
    return cuda_ok(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most),
                   "cudaFuncSetAttribute(gate pass kernel)", err);
  };
  constexpr size_t most64 = sizeof(double2) << kPassMaxTile;
  constexpr size_t most32 = 2 * kPass32MatBytes + (sizeof(float2) << kPass32MaxTile);
  size_t most = 0;
  for (const PassArgs &a : p.args) most = std::max(most, sizeof(double2) << a.tb);
  for (const PassArgs32 &a : p.args32) most = std::max(most, 2 * kPass32MatBytes + (sizeof(float2) << a.tb));
  if (most > 48 * 1024 &&
      (p.pool.empty() ? !opt_in(k_gate_pass32<false>, most32) || !opt_in(k_gate_pass32<true>, most32)
                      : !opt_in(k_gate_pass<false>, most64) || !opt_in(k_gate_pass<true>, most64)))
    return false;
  PlanApi api{err};
  PlanBuffer<PlanApi> b;
  if (!buffer_pool().take(api, dev, bytes, b)) return false;
  if (!upload_now(b.ptr, src, bytes, err)) {
    buffer_pool().give(api, std::move(b));
    return false;
  }
  p.copies.add(std::move(b));
  return true;
}

bool launch_pass_plan(PassPlan &p, const std::vector<GateData> &gates, void *sv, uint32_t n,
                      cudaStream_t s, std::string &err) {
  int dev = 0;
  if (!cuda_ok(cudaGetDevice(&dev), "cudaGetDevice", err)) return false;
  const PlanBuffer<PlanApi> *const mats = p.copies.on(dev);
  for (size_t i = 0; i < p.passes.size(); ++i) {
    if (p.arg_of[i] < 0) {
      if (!launch_gate(gates[p.passes[i].gates[0]], sv, n, s, err)) return false;
      continue;
    }
    if (!mats) {
      err = "gate pass matrices are not on the current device";
      return false;
    }
    const uint32_t tb = p.args.empty() ? p.args32[p.arg_of[i]].tb : p.args[p.arg_of[i]].tb;
    const uint64_t tiles = 1ull << (n - tb);
    if (tiles > 0x7fffffffull) {
      err = "statevector too large for the gate pass kernel grid";
      return false;
    }
    auto narrow = [](const auto &a, uint32_t below) {
      return std::any_of(a.g, a.g + a.n_gates, [&](const auto &g) { return g.k < below; });
    };
    if (p.args.empty()) {
      const PassArgs32 &a = p.args32[p.arg_of[i]];
      const auto kernel = narrow(a, 2) ? k_gate_pass32<true> : k_gate_pass32<false>;
      kernel<<<(unsigned)tiles, kPassThreads, 2 * kPass32MatBytes + (sizeof(float2) << tb), s>>>(
          static_cast<float2 *>(sv), reinterpret_cast<const float *>(mats->ptr), a);
    } else {
      const PassArgs &a = p.args[p.arg_of[i]];
      const auto kernel = narrow(a, 3) ? k_gate_pass<true> : k_gate_pass<false>;
      kernel<<<(unsigned)tiles, kPassThreads, sizeof(double2) << tb, s>>>(
          static_cast<double2 *>(sv), reinterpret_cast<const double *>(mats->ptr), a);
    }
    if (!cuda_ok(cudaGetLastError(), "gate pass kernel launch", err)) return false;
  }
  return true;
}

bool mark_pass_plan(PassPlan &p, cudaStream_t s, std::string &err) {
  int dev = 0;
  if (!cuda_ok(cudaGetDevice(&dev), "cudaGetDevice", err)) return false;
  PlanBuffer<PlanApi> *const mats = p.copies.on(dev);
  if (!mats) return true;
  RelaxedCapture relaxed;
  PlanApi api{err};
  if (mats->mark(api, s)) return true;
  cudaStreamSynchronize(s);  // nothing keeps the buffer for what is queued: wait for it here
  return false;
}

}  // namespace cb2
