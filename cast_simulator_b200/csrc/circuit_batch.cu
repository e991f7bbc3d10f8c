// Many small circuits in one persistent launch.
//
// The reference simulates one circuit at a time: Simulator::simulate launches
// one kernel per gate on the whole device and synchronises
// (src/simulator/mod.rs:523-547; cuda_exec.cpp:302-335).  For circuits of up to
// ~16 qubits a gate pass is a few microseconds of work spread over 148 SMs, so
// such a stream is bound by launches and host round trips.  Here a batch of
// independent circuits - different qubit counts, depths and precisions - runs
// in ONE launch:
//
//  * a persistent grid of CTAs; each CTA claims the next circuit from a device
//    work counter, so long and short circuits balance (the host orders the batch
//    longest first);
//  * a circuit whose state fits (complex128 7..13 qubits, complex64 3..14) lives in
//    shared memory from its first gate to its last: every fused gate (k <= 4) is
//    applied there with the tile code of the merged passes (gate_tile.cuh), the
//    next gate's matrix and walk copied in behind it, and the state is written to
//    the caller's buffer once.  Gate after gate through L1 and L2, as the larger
//    circuits still run, a gate waits for its loads and for a matrix entry from
//    shared memory for every four FMAs: 256 circuits of 8..13 qubits took 700 us,
//    now 238 (kernel 246 -> 140);
//  * the others run every gate in place on the caller's device buffer (at most 2^20
//    amplitudes: 16 MiB in complex128), one thread per gather group;
//  * optionally a circuit starts from |0...0> (written by the CTA itself);
//  * at the end the CTA reduces, in FP64 and in a fixed order, the norm and
//    P(q = 1) of every qubit, and writes <Z_q> = (norm - 2 P(q = 1)) / norm.
//
// Matrices are snapped with the plain path's zero / +-1 rule
// (src/cpp/cuda/cuda_gen.cpp:84-103) and stored in the circuit's precision.
// The circuit table, op list and matrices go to the device at the first run after
// a change of the batch, ahead of its launch on the same stream; a run resets the work counter, launches, and copies the
// <Z> table back: three operations on one stream.
#include "../../include/cast_b200.h"
#include "gate_tile.cuh"

#include <algorithm>
#include <cstring>
#include <exception>
#include <mutex>
#include <numeric>
#include <vector>

#include <cuda_pipeline.h>

namespace {

using cb2::cuda_ok;
using cb2::write_err;
using cb2::clear_err;

// Threads a CTA: 256 when every circuit of a batch is resident (two CTAs an SM for
// small states), 512 when one streams its state from memory (loads in flight).
constexpr int kBResidentThreads = 256, kBThreads = 512;
constexpr uint32_t kBatchMaxQubits = 20;
constexpr uint32_t kBatchMaxGate = 4;
constexpr uint32_t kBatchMagic = 0xB47C4001u;

struct BCircuit {
  uint64_t sv;      // device statevector (interleaved re/im)
  uint32_t n;       // qubits
  uint32_t prec;    // 0 = F32, 1 = F64
  uint32_t op_begin;
  uint32_t n_ops;
  uint32_t init_zero;
  uint32_t z_off;   // first <Z> slot of this circuit
  uint32_t resident;  // the state is held in shared memory
  uint32_t pad;
};

struct alignas(16) BOp {
  uint32_t mat;  // where the matrix starts in the pool, in units of 16 bytes
  uint32_t mat_bytes;
  uint32_t k;
  uint32_t q[kBatchMaxGate];
  union {  // resident circuits: the walk of the tile
    cb2::PassGateArgs a64;
    cb2::PassGateArgs32 a32;
  };
};

// Shared memory: two gates' matrices (the resident form's 4-qubit matrix in
// complex128 is the largest) and their ops, then a resident circuit's state.
constexpr uint32_t kBMatBytes = 2 * 256 * sizeof(double);
constexpr uint32_t kBStateOffset = 2 * kBMatBytes + 2 * ((sizeof(BOp) + 15) & ~15u);

// Sizes whose state is held in shared memory: at least the tile code's smallest
// tile, at most 128 KB.
bool resident_size(uint32_t n, uint32_t prec) {
  return prec ? n >= cb2::kTileMin64 && n <= cb2::kTileMax64 : n >= 3 && n <= cb2::kTileMax32;
}

struct BHeader {
  uint32_t next;  // work counter (zero in every upload)
  uint32_t n_circuits;
  uint32_t n_ops;
  uint32_t pad;
};

template <typename T> struct C2;
template <> struct C2<float> { using type = float2; };
template <> struct C2<double> { using type = double2; };

template <typename V> __device__ __forceinline__ V cmac(V m, V x, V acc) {
  acc.x = fma(m.x, x.x, acc.x);
  acc.x = fma(-m.y, x.y, acc.x);
  acc.y = fma(m.x, x.y, acc.y);
  acc.y = fma(m.y, x.x, acc.y);
  return acc;
}

// One fused k-qubit gate applied in place: thread t takes groups t, t + NT, ...
template <int NT, typename T, int K>
__device__ __noinline__ void batch_gate(typename C2<T>::type *sv, uint32_t n, const uint32_t *q,
                                        const typename C2<T>::type *M) {
  using V = typename C2<T>::type;
  constexpr int D = 1 << K;
  uint32_t lo[K];
#pragma unroll
  for (int b = 0; b < K; ++b) lo[b] = (1u << q[b]) - 1;
  const uint32_t ng = 1u << (n - K);
  for (uint32_t g = threadIdx.x; g < ng; g += NT) {
    uint32_t base = g;
#pragma unroll
    for (int b = 0; b < K; ++b) base = ((base & ~lo[b]) << 1) | (base & lo[b]);
    V x[D];
#pragma unroll
    for (int a = 0; a < D; ++a) {
      uint32_t o = base;
#pragma unroll
      for (int b = 0; b < K; ++b)
        if ((a >> b) & 1) o += lo[b] + 1;
      x[a] = sv[o];
    }
#pragma unroll
    for (int r = 0; r < D; ++r) {
      V acc;
      acc.x = 0;
      acc.y = 0;
#pragma unroll
      for (int c = 0; c < D; ++c) acc = cmac(M[r * D + c], x[c], acc);
      uint32_t o = base;
#pragma unroll
      for (int b = 0; b < K; ++b)
        if ((r >> b) & 1) o += lo[b] + 1;
      sv[o] = acc;
    }
  }
}

struct BShared {
  double red[kBThreads / 32][6 + kBatchMaxQubits];
  BCircuit circ;
  uint32_t claim;
};

// <Z_q> of a state of 2^n amplitudes with probabilities prob(i), i = u RT + thread,
// by the first RT threads of the CTA (a resident circuit gives the same bits
// whatever the CTA's size).  A thread's low index bits are fixed, so its total
// serves their qubits.
template <int RT, typename P>
__device__ __forceinline__ void reduce_z(BShared &S, uint32_t n, P prob, double *__restrict__ out_z) {
  constexpr uint32_t TB = RT == 512 ? 9 : 8;
  static_assert(RT == 1 << TB, "a power of two of threads");
  constexpr uint32_t HIGH = kBatchMaxQubits - TB;
  double tot = 0.0, high[HIGH];
#pragma unroll
  for (uint32_t q = 0; q < HIGH; ++q) high[q] = 0.0;
  for (uint32_t u = 0; threadIdx.x < RT && (u << TB) + threadIdx.x < (1u << n); ++u) {
    const double p = prob((u << TB) + threadIdx.x);
    tot += p;
#pragma unroll
    for (uint32_t q = 0; q < HIGH; ++q)
      if ((u >> q) & 1) high[q] += p;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto put = [&](uint32_t slot, double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) S.red[warp][slot] = v;
  };
#pragma unroll
  for (uint32_t b = 0; b < 5; ++b) put(b, (lane >> b) & 1 ? tot : 0.0);
  put(5, tot);
#pragma unroll
  for (uint32_t q = 0; q < HIGH; ++q)
    if (TB + q < n) put(6 + q, high[q]);
  __syncthreads();
  if (threadIdx.x < n) {
    const uint32_t q = threadIdx.x;
    double all = 0.0, p1 = 0.0;
    for (uint32_t w = 0; w < RT / 32; ++w) {
      all += S.red[w][5];
      p1 += q < 5 ? S.red[w][q] : q < TB ? ((w >> (q - 5)) & 1 ? S.red[w][5] : 0.0) : S.red[w][6 + q - TB];
    }
    out_z[q] = all > 0.0 ? (all - 2.0 * p1) / all : 0.0;
  }
  __syncthreads();
}

// A circuit whose state stays in device memory.
template <int NT, typename T>
__device__ void run_streamed(BShared &S, unsigned char *smem, const BOp *__restrict__ ops,
                             const char *__restrict__ pool, double *__restrict__ out_z) {
  using V = typename C2<T>::type;
  const BCircuit c = S.circ;
  V *sv = reinterpret_cast<V *>(c.sv);
  const uint32_t N = 1u << c.n;
  if (c.init_zero) {
    for (uint32_t i = threadIdx.x; i < N; i += NT) {
      V v;
      v.x = i == 0 ? (T)1 : (T)0;
      v.y = 0;
      sv[i] = v;
    }
    __syncthreads();
  }
  V *Msm = reinterpret_cast<V *>(smem);
  for (uint32_t oi = 0; oi < c.n_ops; ++oi) {
    const BOp &op = ops[c.op_begin + oi];
    const V *Mg = reinterpret_cast<const V *>(pool + (size_t)op.mat * 16);
    const uint32_t k = op.k, entries = 1u << (2 * k);
    for (uint32_t i = threadIdx.x; i < entries; i += NT) Msm[i] = Mg[i];
    __syncthreads();
    switch (k) {
    case 1: batch_gate<NT, T, 1>(sv, c.n, op.q, Msm); break;
    case 2: batch_gate<NT, T, 2>(sv, c.n, op.q, Msm); break;
    case 3: batch_gate<NT, T, 3>(sv, c.n, op.q, Msm); break;
    default: batch_gate<NT, T, 4>(sv, c.n, op.q, Msm); break;
    }
    __syncthreads();
  }
  reduce_z<NT>(S, c.n, [&](uint32_t i) {
    const V v = sv[i];
    return (double)v.x * v.x + (double)v.y * v.y;
  }, out_z + c.z_off);
}

// A circuit whose state is held in shared memory.
template <int NT, typename T>
__device__ void run_resident(BShared &S, unsigned char *smem, const BOp *__restrict__ ops,
                             const char *__restrict__ pool, double *__restrict__ out_z) {
  using V = typename C2<T>::type;
  constexpr bool F64 = sizeof(T) == 8;
  const BCircuit c = S.circ;
  V *sv = reinterpret_cast<V *>(c.sv);
  V *s = reinterpret_cast<V *>(smem + kBStateOffset);
  BOp *const slots = reinterpret_cast<BOp *>(smem + 2 * kBMatBytes);
  auto place = [](uint32_t i) { return F64 ? cb2::pass_swz(i) : cb2::pass_swz32(i); };
  const uint32_t N = 1u << c.n;
  for (uint32_t i = threadIdx.x; i < N; i += NT) {
    V v;
    v.x = i == 0 ? (T)1 : (T)0;
    v.y = 0;
    s[place(i)] = c.init_zero ? v : sv[i];
  }
  const BOp *const op = ops + c.op_begin;
  // the copies of gate i's matrix and walk, given where its matrix is
  auto fetch = [&](uint32_t i, uint2 where) {
    unsigned char *to = smem + (i & 1) * kBMatBytes;
    for (uint32_t b = 16 * threadIdx.x; b < where.y; b += 16 * NT)
      __pipeline_memcpy_async(to + b, pool + (size_t)where.x * 16 + b, 16);
    if (threadIdx.x < sizeof(BOp) / 16)
      __pipeline_memcpy_async(reinterpret_cast<char *>(&slots[i & 1]) + 16 * threadIdx.x,
                              reinterpret_cast<const char *>(op + i) + 16 * threadIdx.x, 16);
  };
  auto where = [&](uint32_t i) { return *reinterpret_cast<const uint2 *>(op + i); };
  if (c.n_ops) fetch(0, where(0));
  uint2 next = c.n_ops > 1 ? where(1) : make_uint2(0, 0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (uint32_t oi = 0; oi < c.n_ops; ++oi) {
    __pipeline_commit();
    __pipeline_wait_prior(0);
    __syncthreads();  // the gate before is done; this one's matrix and walk are here
    if (oi + 1 < c.n_ops) fetch(oi + 1, next);
    if (oi + 2 < c.n_ops) next = where(oi + 2);
    const unsigned char *mat = smem + (oi & 1) * kBMatBytes;
    const BOp &o = slots[oi & 1];
    if constexpr (F64) {
      const double *m = reinterpret_cast<const double *>(mat);
      switch (o.k) {
      case 4: cb2::pass_gate4_full<NT / 32>(s, m, o.a64, N >> 7, warp, lane); break;
      case 3: cb2::pass_gate3<NT / 32>(s, m, o.a64, N >> 6, warp, lane); break;
      case 2: cb2::pass_small<NT / 32, 2, 2>(s, m, o.a64, N >> 6, warp, lane); break;
      default: cb2::pass_small<NT / 32, 1, 2>(s, m, o.a64, N >> 6, warp, lane);
      }
    } else {
      const float *m = reinterpret_cast<const float *>(mat);
      switch (o.k) {
      case 4: cb2::pass_gate32<NT, 4, 2, 2, false>(s, m, o.a32, c.n); break;
      case 3: cb2::pass_gate32<NT, 3, 1, 2, false>(s, m, o.a32, c.n); break;
      case 2: cb2::pass_gate32<NT, 2, 1, 4, false>(s, m, o.a32, c.n); break;
      default: cb2::pass_gate32<NT, 1, 1, 4, false>(s, m, o.a32, c.n);
      }
    }
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < N; i += NT) sv[i] = s[place(i)];
  reduce_z<kBResidentThreads>(S, c.n, [&](uint32_t i) {
    const V v = s[place(i)];
    return (double)v.x * v.x + (double)v.y * v.y;
  }, out_z + c.z_off);
}

template <int NT>
__global__ void __launch_bounds__(NT, NT == kBResidentThreads ? 2 : 1)
    k_circuit_batch(BHeader *__restrict__ hdr, const BCircuit *__restrict__ circs,
                    const BOp *__restrict__ ops, const char *__restrict__ pool,
                    double *__restrict__ out_z) {
  __shared__ BShared S;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const uint32_t n_circ = hdr->n_circuits;
  while (true) {
    if (threadIdx.x == 0) {
      S.claim = atomicAdd(&hdr->next, 1u);
      if (S.claim < n_circ) S.circ = circs[S.claim];
    }
    __syncthreads();
    if (S.claim >= n_circ) return;
    if (S.circ.resident) {
      if (S.circ.prec == 1) run_resident<NT, double>(S, smem_raw, ops, pool, out_z);
      else run_resident<NT, float>(S, smem_raw, ops, pool, out_z);
    } else {
      if (S.circ.prec == 1) run_streamed<NT, double>(S, smem_raw, ops, pool, out_z);
      else run_streamed<NT, float>(S, smem_raw, ops, pool, out_z);
    }
  }
}

// ── host side ────────────────────────────────────────────────────────────────

struct Batch {
  uint32_t magic = kBatchMagic;
  std::mutex mu;
  std::vector<BCircuit> circs;
  std::vector<BOp> ops;
  std::vector<char> pool;   // matrices as the kernel reads them, each 16-byte aligned
  size_t matrix_bytes = 0;  // of the gates' matrices by themselves: what the limit is on
  std::vector<uint64_t> cost;  // work estimate per circuit (ordering)
  std::vector<char> tables;    // header, circuits and ops of the last upload
  uint32_t n_z = 0;
  bool uploaded = false;  // the device buffer holds the circuits as they are now
  // device and pinned buffers, grown on demand and reused across runs
  char *dev = nullptr;
  size_t dev_cap = 0;
  double *host_z = nullptr;
  size_t host_z_cap = 0;
  int device = -1;

  ~Batch() {
    if (dev) cudaFree(dev);
    if (host_z) cudaFreeHost(host_z);
  }
};

Batch *as_batch(void *p) {
  Batch *b = static_cast<Batch *>(p);
  return b && b->magic == kBatchMagic ? b : nullptr;
}

size_t align16(size_t x) { return (x + 15) & ~size_t(15); }

// Takes back what a refused circuit has appended.
struct Appended {
  Batch &b;
  const size_t ops = b.ops.size(), pool = b.pool.size(), matrices = b.matrix_bytes;
  bool keep = false;
  ~Appended() {
    if (keep) return;
    b.ops.resize(ops);
    b.pool.resize(pool);
    b.matrix_bytes = matrices;
  }
};

// gate(i, k, q) gives gate i's width, targets and matrix (interleaved complex128,
// read before the next call), or null for one it has no matrix of.  Everything is
// appended where it stays: a serving loop builds a batch for one run, so what adding
// a circuit costs counts like the run.  256 circuits of 8..13 qubits (4259 gates of
// up to 4 qubits) in complex128: 8.2 ms through copies of the whole circuit, now 5.6.
template <class Gate>
bool add_circuit(Batch &b, uint64_t sv, uint32_t n, uint8_t prec, uint32_t n_gates, Gate gate, int init_zero,
                 double ztol, double otol, std::string &err) {
  if (!sv) {
    err = "statevector must not be null";
    return false;
  }
  if (!cb2::aligned16(sv, "statevector pointer", err)) return false;
  if (prec > 1 || n == 0 || n > kBatchMaxQubits) {
    err = "batched circuits: precision 0 / 1 and 1.." + std::to_string(kBatchMaxQubits) + " qubits";
    return false;
  }
  BCircuit c{};
  c.sv = sv;
  c.n = n;
  c.prec = prec;
  c.op_begin = (uint32_t)b.ops.size();
  c.n_ops = n_gates;
  c.init_zero = init_zero ? 1 : 0;
  c.z_off = b.n_z;
  c.resident = resident_size(n, prec) ? 1 : 0;
  std::vector<uint32_t> tile_qubits(n);
  std::iota(tile_qubits.begin(), tile_qubits.end(), 0u);
  std::vector<double> frag64;
  std::vector<float> frag32;
  Appended appended{b};
  cb2::GateData g;
  g.precision = prec;
  uint64_t cost = 0;
  for (uint32_t i = 0; i < n_gates; ++i) {
    uint32_t k = 0, q[cb2::kMaxGateQubits] = {0};
    const double *const m = gate(i, k, q);
    if (k == 0 || k > kBatchMaxGate || k > n) {
      err = "batched circuits take gates of 1.." + std::to_string(kBatchMaxGate) +
            " qubits within the circuit (gate " + std::to_string(i) + ")";
      return false;
    }
    if (!m) {
      err = "gate arrays must not be null";
      return false;
    }
    g.k = k;
    BOp op{};
    op.k = k;
    for (uint32_t j = 0; j < k; ++j) {
      if (q[j] >= n || (j && q[j - 1] >= q[j])) {
        err = "gate " + std::to_string(i) + ": qubits must be ascending and below the circuit's size";
        return false;
      }
      op.q[j] = g.qubits[j] = q[j];
    }
    const size_t entries = 1ull << (2 * k);
    cb2::snap_matrix(g, m, ztol, otol);
    size_t bytes = entries * (prec ? 16 : 8);
    if (b.matrix_bytes + bytes > 0xFFFFFFF0ull) {
      err = "batch matrix pool exceeds 4 GiB";
      return false;
    }
    b.matrix_bytes += bytes;
    const void *from = prec ? (const void *)g.m64.data() : (const void *)g.m32.data();
    if (c.resident) {
      const cb2::PlacedGate placed = cb2::place_gate(g, tile_qubits);
      frag64.clear();
      frag32.clear();
      if (prec) cb2::pack_gate(placed, n, false, frag64, op.a64);
      else cb2::pack_gate32(placed, n, false, frag32, op.a32);
      bytes = prec ? frag64.size() * sizeof(double) : frag32.size() * sizeof(float);
      from = prec ? (const void *)frag64.data() : (const void *)frag32.data();
    }
    static_assert(sizeof(float2) * 4 % 16 == 0, "the smallest matrix keeps the pool 16-byte aligned");
    op.mat = (uint32_t)(b.pool.size() / 16);  // laid out, at most 1.5 times 4 GiB
    op.mat_bytes = (uint32_t)bytes;
    const char *const at = static_cast<const char *>(from);
    b.uploaded = false;
    b.pool.insert(b.pool.end(), at, at + bytes);
    b.ops.push_back(op);
    cost += (uint64_t)entries << (n - k);  // complex multiply-adds of the pass
  }
  b.uploaded = false;
  b.circs.push_back(c);
  b.cost.push_back(cost + (2ull << n));
  b.n_z += n;
  appended.keep = true;
  return true;
}

size_t smem_most() { return kBStateOffset + (sizeof(double2) << cb2::kTileMax64); }

bool run_batch(Batch &b, double *out_z, cudaStream_t s, std::string &err) {
  const uint32_t nc = (uint32_t)b.circs.size();
  if (nc == 0) return true;
  int dev = 0;
  if (!cuda_ok(cudaGetDevice(&dev), "cudaGetDevice", err)) return false;
  if (b.device != dev) {  // buffers belong to the device they were made on
    if (b.dev) cudaFree(b.dev);
    b.dev = nullptr;
    b.dev_cap = 0;
    b.device = dev;
    b.uploaded = false;
  }
  const size_t off_c = align16(sizeof(BHeader));
  const size_t off_o = align16(off_c + sizeof(BCircuit) * nc);
  const size_t off_p = align16(off_o + sizeof(BOp) * b.ops.size());
  const size_t off_z = align16(off_p + b.pool.size());
  const size_t total = off_z + sizeof(double) * b.n_z;
  if (b.dev_cap < total) {
    if (b.dev) cudaFree(b.dev);
    b.dev = nullptr;
    b.uploaded = false;
    const size_t cap = std::max(total, b.dev_cap * 2);
    if (!cuda_ok(cudaMalloc(&b.dev, cap), "cudaMalloc (circuit batch)", err)) {
      b.dev_cap = 0;
      return false;
    }
    b.dev_cap = cap;
  }
  if (b.host_z_cap < b.n_z) {
    if (b.host_z) cudaFreeHost(b.host_z);
    b.host_z = nullptr;
    const size_t cap = std::max<size_t>(b.n_z, b.host_z_cap * 2);
    if (!cuda_ok(cudaMallocHost(&b.host_z, cap * sizeof(double)), "cudaMallocHost (batch <Z>)", err)) {
      b.host_z_cap = 0;
      return false;
    }
    b.host_z_cap = cap;
  }
  if (!b.uploaded) {
    // longest first: the work counter hands them out in this order
    std::vector<uint32_t> order(nc);
    std::iota(order.begin(), order.end(), 0u);
    std::stable_sort(order.begin(), order.end(),
                     [&](uint32_t a, uint32_t c) { return b.cost[a] > b.cost[c]; });
    std::vector<char> &tables = b.tables;
    tables.assign(off_p, 0);
    const BHeader h{0u, nc, (uint32_t)b.ops.size(), 0u};
    std::memcpy(tables.data(), &h, sizeof(h));
    BCircuit *hc = reinterpret_cast<BCircuit *>(tables.data() + off_c);
    for (uint32_t i = 0; i < nc; ++i) hc[i] = b.circs[order[i]];
    if (!b.ops.empty()) std::memcpy(tables.data() + off_o, b.ops.data(), sizeof(BOp) * b.ops.size());
    // pageable memory, which is staged before these calls return
    if (!cuda_ok(cudaMemcpyAsync(b.dev, tables.data(), off_p, cudaMemcpyHostToDevice, s),
                 "cudaMemcpyAsync (batch upload)", err) ||
        (!b.pool.empty() && !cuda_ok(cudaMemcpyAsync(b.dev + off_p, b.pool.data(), b.pool.size(),
                                                     cudaMemcpyHostToDevice, s),
                                     "cudaMemcpyAsync (batch matrices)", err))) {
      cudaStreamSynchronize(s);
      return false;
    }
    b.uploaded = true;
  }
  // 256 threads a CTA when every circuit is resident; shared memory for the largest
  uint32_t state = 0;
  bool all_resident = true;
  for (const BCircuit &c : b.circs) {
    if (c.resident) state = std::max(state, (c.prec ? 16u : 8u) << c.n);
    else all_resident = false;
  }
  const size_t smem = kBStateOffset + state;
  const auto kernel = all_resident ? k_circuit_batch<kBResidentThreads> : k_circuit_batch<kBThreads>;
  const int threads = all_resident ? kBResidentThreads : kBThreads;
  int per_sm = 1;
  if (!cuda_ok(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_most()),
               "cudaFuncSetAttribute (circuit batch)", err) ||
      !cuda_ok(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem),
               "cudaOccupancyMaxActiveBlocksPerMultiprocessor", err))
    return false;
  const uint32_t slots = (uint32_t)std::max(1, per_sm) * (uint32_t)std::max(1, cb2::sm_count());
  const unsigned grid = (unsigned)std::min<uint32_t>(nc, slots);
  bool ok = cuda_ok(cudaMemsetAsync(b.dev, 0, sizeof(uint32_t), s), "cudaMemsetAsync (work counter)", err);
  if (ok) {
    kernel<<<grid, threads, smem, s>>>(
        reinterpret_cast<BHeader *>(b.dev), reinterpret_cast<const BCircuit *>(b.dev + off_c),
        reinterpret_cast<const BOp *>(b.dev + off_o), b.dev + off_p,
        reinterpret_cast<double *>(b.dev + off_z));
    ok = cuda_ok(cudaGetLastError(), "circuit batch launch", err) &&
         cuda_ok(cudaMemcpyAsync(b.host_z, b.dev + off_z, sizeof(double) * b.n_z,
                                 cudaMemcpyDeviceToHost, s),
                 "cudaMemcpyAsync (batch <Z>)", err);
  }
  // the pinned buffer is reused by the next run: wait for the copy either way
  std::string e2;
  const bool synced = cuda_ok(cudaStreamSynchronize(s), "cudaStreamSynchronize (circuit batch)", e2);
  if (ok && !synced) err = e2;
  ok = ok && synced;
  if (ok && out_z) std::memcpy(out_z, b.host_z, sizeof(double) * b.n_z);
  return ok;
}

bool check_distinct(const Batch &b, std::string &err) {
  std::vector<std::pair<uint64_t, uint64_t>> spans;  // [begin, end) bytes of each statevector
  for (const BCircuit &c : b.circs)
    spans.emplace_back(c.sv, c.sv + ((uint64_t)(c.prec ? 16 : 8) << c.n));
  std::sort(spans.begin(), spans.end());
  for (size_t i = 1; i < spans.size(); ++i)
    if (spans[i].first < spans[i - 1].second) {
      err = "two circuits of a batch share statevector memory";
      return false;
    }
  return true;
}

}  // namespace

extern "C" {

void *cast_b200_batch_create(char *err_buf, size_t err_buf_len) {
  try {
    Batch *b = new Batch;
    clear_err(err_buf, err_buf_len);
    return b;
  } catch (const std::exception &ex) {
    write_err(err_buf, err_buf_len, ex.what());
    return nullptr;
  }
}

void cast_b200_batch_destroy(void *batch) {
  Batch *b = as_batch(batch);
  if (!b) return;
  b->magic = 0;
  delete b;
}

int cast_b200_batch_add(void *batch, uint64_t sv_dptr, uint32_t n_qubits, uint8_t precision,
                        uint32_t n_gates, const uint32_t *gate_k, const uint32_t *qubits,
                        const cast_complex64_t *matrices, int init_zero, double ztol, double otol,
                        char *err_buf, size_t err_buf_len) {
  Batch *b = as_batch(batch);
  if (!b) {
    write_err(err_buf, err_buf_len, "invalid batch handle");
    return 1;
  }
  try {
    std::lock_guard<std::mutex> lock(b->mu);
    std::string err;
    const double *m = reinterpret_cast<const double *>(matrices);
    auto gate = [&](uint32_t i, uint32_t &k, uint32_t *q) -> const double * {
      k = gate_k[i];
      if (k > kBatchMaxGate) return nullptr;  // refused by its width
      std::copy(qubits, qubits + k, q);
      qubits += k;
      const double *const at = m;
      m += (size_t)2 << (2 * k);
      return at;
    };
    if (n_gates && (!gate_k || !qubits || !matrices)) err = "gate arrays must not be null";
    if (!err.empty() ||
        !add_circuit(*b, sv_dptr, n_qubits, precision, n_gates, gate, init_zero, ztol, otol, err)) {
      write_err(err_buf, err_buf_len, err);
      return 1;
    }
  } catch (const std::exception &ex) {
    write_err(err_buf, err_buf_len, ex.what());
    return 1;
  }
  clear_err(err_buf, err_buf_len);
  return 0;
}

int cast_b200_batch_add_fused(void *batch, uint64_t sv_dptr, uint32_t n_qubits, uint8_t precision,
                              const void *fused, int init_zero, double ztol, double otol,
                              char *err_buf, size_t err_buf_len) {
  Batch *b = as_batch(batch);
  if (!b || !fused) {
    write_err(err_buf, err_buf_len, "invalid batch or fused-circuit handle");
    return 1;
  }
  try {
    const uint32_t ng = cast_b200_fused_num_gates(fused);
    for (uint32_t i = 0; i < ng; ++i) {
      uint32_t k = 0;
      if (cast_b200_fused_gate(fused, i, &k, nullptr, nullptr) || k == 0 || k > kBatchMaxGate) {
        write_err(err_buf, err_buf_len,
                  "fused gate " + std::to_string(i) + " is wider than the batch kernel's " +
                      std::to_string(kBatchMaxGate) + " qubits (fuse with size_max <= 4)");
        return 1;
      }
    }
    cast_complex64_t m[1u << (2 * kBatchMaxGate)];
    auto gate = [&](uint32_t i, uint32_t &k, uint32_t *q) -> const double * {
      return cast_b200_fused_gate(fused, i, &k, q, m) ? nullptr : reinterpret_cast<const double *>(m);
    };
    std::lock_guard<std::mutex> lock(b->mu);
    std::string err;
    if (!add_circuit(*b, sv_dptr, n_qubits, precision, ng, gate, init_zero, ztol, otol, err)) {
      write_err(err_buf, err_buf_len, err);
      return 1;
    }
  } catch (const std::exception &ex) {
    write_err(err_buf, err_buf_len, ex.what());
    return 1;
  }
  clear_err(err_buf, err_buf_len);
  return 0;
}

uint32_t cast_b200_batch_num_circuits(const void *batch) {
  const Batch *b = static_cast<const Batch *>(batch);
  return b && b->magic == kBatchMagic ? (uint32_t)b->circs.size() : 0;
}

uint32_t cast_b200_batch_num_z(const void *batch) {
  const Batch *b = static_cast<const Batch *>(batch);
  return b && b->magic == kBatchMagic ? b->n_z : 0;
}

void cast_b200_batch_clear(void *batch) {
  Batch *b = as_batch(batch);
  if (!b) return;
  std::lock_guard<std::mutex> lock(b->mu);
  b->circs.clear();
  b->ops.clear();
  b->pool.clear();
  b->matrix_bytes = 0;
  b->cost.clear();
  b->uploaded = false;
  b->n_z = 0;
}

int cast_b200_batch_run(void *batch, double *out_z, void *stream, char *err_buf,
                        size_t err_buf_len) {
  Batch *b = as_batch(batch);
  if (!b) {
    write_err(err_buf, err_buf_len, "invalid batch handle");
    return 1;
  }
  try {
    std::lock_guard<std::mutex> lock(b->mu);
    std::string err;
    if (!check_distinct(*b, err) || !run_batch(*b, out_z, static_cast<cudaStream_t>(stream), err)) {
      write_err(err_buf, err_buf_len, err);
      return 1;
    }
  } catch (const std::exception &ex) {
    write_err(err_buf, err_buf_len, ex.what());
    return 1;
  }
  clear_err(err_buf, err_buf_len);
  return 0;
}

}  // extern "C"
