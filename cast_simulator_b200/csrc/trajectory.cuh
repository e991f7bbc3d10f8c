// Batched Monte-Carlo quantum-jump trajectories in one persistent kernel.
//
// Replaces the reference's ensemble simulation (src/simulator/trajectory.rs:
// simulate_ensemble at :180-265 branches deterministically on fixed weights
// p_i and launches one kernel per gate per member, syncing with the host at
// every noisy gate) with quantum-jump trajectories sampled on the device:
//
//  * one CTA (512 or 1024 threads) owns one trajectory at a time; its 2^n
//    complex64 statevector lives in a per-CTA slice of a workspace in global
//    memory (148 CTAs x 512 KiB = 74 MiB at 16 qubits, resident in the 126 MB
//    L2); the CTA loops over trajectories blockIdx.x, blockIdx.x + gridDim.x, ...
//  * GATE ops are fused unitary blocks (k <= 4).  Pieces of a run of them up to the
//    next DAMP or CHAN op are segments (seg_plan.cpp): when none of a segment's ERR
//    sites fires (their draws do not depend on the state), its blocks share passes as
//    a gate program's gates do (pass_plan.hpp, gate_tile.cuh), tiles of up to 2^13
//    amplitudes in shared memory with the next tile's copy in flight; otherwise, and
//    for programs without such segments, the blocks are applied one after the other
//    in place;
//  * ERR ops are state-independent Pauli errors (depolarizing): a Philox draw
//    decides; when one fires, the Pauli propagated to the end of its fused
//    block (U P U^dagger, precomputed on the host) is applied as a gate;
//  * DAMP ops are amplitude damping on a set of qubits.  The no-jump branch has
//    probability D/T with T = sum |a_i|^2 and D = sum |a_i|^2 (1-g)^popc(i&mask),
//    both FP64 sums computed by the preceding gate pass as it stores; on a
//    no-jump draw the diagonal prod_q K0_q and the 1/sqrt(D) renormalisation are
//    folded into the next pass's loads.  Otherwise the jump pattern is sampled
//    exactly, qubit by qubit, conditioned on at least one jump;
//  * CHAN ops are general single-qubit channels: FP64 branch norms
//    ||K_j psi||^2, one draw, K_j / sqrt(p_j) applied.
// At the end each trajectory writes <Z_q> for every qubit and one measured
// bitstring sampled from |psi|^2.  Branch sums, renormalisation factors and the
// final reductions are FP64; amplitudes and gate arithmetic are FP32.
//
// This file is the device side.  The plain kernels (trajectory.cu) and the one for
// programs with segments (trajectory_seg.cu) are compiled apart: in one translation
// unit the functions they share are laid out for both, and the ops of states of 4
// to 7 qubits took 7% longer.
#pragma once

#include "gate_tile.cuh"
#include "pass_plan.hpp"
#include "philox.cuh"

#include <cuda_pipeline.h>

#include <algorithm>

namespace cb2 {

// Enqueues the kernel of trajectory_seg.cu.  ops, run and segs: TOp, TRun and TSegs
// as below (each translation unit has its own copy of these types).
cudaError_t launch_trajectory_segments(unsigned grid, cudaStream_t s, const void *ops, uint32_t n_ops,
                                       const float2 *pool, float2 *ws, uint32_t n, const void *run,
                                       double *z, uint32_t *sample, const void *segs);

}  // namespace cb2

namespace {

// A CTA has 512 or 1024 threads (the kernel is instantiated for both).
constexpr int kTMinThreads = 512, kTMaxThreads = 1024;
constexpr uint32_t kTrajMaxQubits = 22;
constexpr uint32_t kTrajMaxGate = 4;

enum : uint32_t { T_GATE = 0, T_ERR = 1, T_DAMP = 2, T_CHAN = 3 };

struct TOp {
  uint32_t type;
  uint32_t k;
  uint32_t q[kTrajMaxGate];
  uint32_t mat;    // complex offset into the matrix pool
  uint32_t nk;     // CHAN: number of Kraus operators (<= 4)
  uint32_t mask;   // DAMP: qubits
  uint32_t stats;  // GATE: accumulate (T, D) for the DAMP op that follows
  uint32_t nerr;   // GATE: number of ERR ops that directly follow it
  uint32_t smask;  // GATE stats: damping mask of that op
  float prob;      // ERR: firing probability
  float gamma;     // DAMP: damping rate
  float sgamma;    // GATE stats: damping rate of that op
};

// A run of GATE ops (and the ERR ops that follow them) grouped into passes.
struct TSeg {
  uint32_t end_op;           // first op after it
  uint32_t pass0, n_passes;
  uint32_t err0, n_err;      // its ERR ops, in order (entries of the site list)
  uint32_t stats, smask;     // the DAMP op behind it, if any (as TOp)
  float sgamma;
};
struct TSegPass {
  uint32_t tb, n_gates;
  uint32_t gate0;            // first entry of the gate list
  uint32_t mat, mat_bytes;   // its gates' matrices, one after the other
  uint32_t stride[13];       // tile bit -> amplitude stride
};
constexpr uint32_t kSegMaxTile = 13, kSegLow = 4;
constexpr uint32_t kSegMinQubits = 8;  // below, a pass costs what its gates do (6 qubits: 1.26 against 1.20 ms)

struct TSegs {  // device arrays of a program's segments
  const TSeg *segs;
  const TSegPass *passes;
  const cb2::PassGateArgs32 *gates;
  const uint32_t *sites;     // op index of every ERR op of a segment
  const uint32_t *starts;    // per op: 1 + the segment that starts there, or 0
  const float *mats;
  uint32_t mat_cap;          // bytes kept for a pass's matrices
};

struct TRun {  // device-resident, rewritten before each launch
  uint32_t n_traj;
  uint32_t first;  // index of the first trajectory (its Philox stream), for ranges
  uint64_t seed;
};

// Philox-4x32-10 (philox.cuh): counter (event, 0, trajectory, 0x5eed5eed),
// key = the 64-bit seed.
__device__ __forceinline__ double philox_uniform(uint64_t seed, uint32_t traj, uint32_t event) {
  uint32_t x[4] = {event, 0u, traj, 0x5eed5eedu};
  cb2::philox4x32_10(x, (uint32_t)seed, (uint32_t)(seed >> 32));
  return cb2::philox_unit(x);
}

struct Shared {
  double red[3][kTMaxThreads / 32];
  double vals[4];
  float dtab[kTrajMaxQubits + 1];  // pending diagonal: scale * s^popc
  double stab[kTrajMaxQubits + 1]; // damping weights (1 - g)^popc for the sums
  uint32_t pmask;
  int pend;
};

__device__ __forceinline__ float2 cmul_add(float2 m, float2 x, float2 acc) {
  acc.x = fmaf(m.x, x.x, acc.x);
  acc.x = fmaf(-m.y, x.y, acc.x);
  acc.y = fmaf(m.x, x.y, acc.y);
  acc.y = fmaf(m.y, x.x, acc.y);
  return acc;
}

// Shared memory kept for a pass's gate arguments.
constexpr uint32_t kSegArgBytes = (cb2::kMaxPassGates * sizeof(cb2::PassGateArgs32) + 15) & ~15u;

// The device side of one trajectory, for CTAs of NT threads.  512-thread CTAs
// get 128 registers a thread, so the fused gates run without spills (their passes
// are bound by instruction issue); 1024-thread CTAs keep twice the loads in flight,
// which is what narrow blocks need on L2-resident states (plain_threads, seg_plan.cpp).
template <int NT>
struct Traj {
  static constexpr int kTThreads = NT;
  static constexpr uint32_t kTLogThreads = NT == 1024 ? 10 : 9;

  // Block sum of up to three doubles; every thread gets the results.
  static __device__ void block_sum3(Shared &S, double &a, double &b, double &c) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      a += __shfl_down_sync(0xffffffffu, a, o);
      b += __shfl_down_sync(0xffffffffu, b, o);
      c += __shfl_down_sync(0xffffffffu, c, o);
    }
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) {
      S.red[0][w] = a;
      S.red[1][w] = b;
      S.red[2][w] = c;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      double x = 0, y = 0, z = 0;
      for (int i = 0; i < kTThreads / 32; ++i) {
        x += S.red[0][i];
        y += S.red[1][i];
        z += S.red[2][i];
      }
      S.vals[0] = x;
      S.vals[1] = y;
      S.vals[2] = z;
    }
    __syncthreads();
    a = S.vals[0];
    b = S.vals[1];
    c = S.vals[2];
    __syncthreads();
  }

  static __device__ void fill_stab(Shared &S, double g) {
    if (threadIdx.x == 0) {
      double f = 1.0;
      for (uint32_t c = 0; c <= kTrajMaxQubits; ++c) {
        S.stab[c] = f;
        f *= 1.0 - g;
      }
    }
    __syncthreads();
  }

  static __device__ __forceinline__ float2 pend_load(const float2 *sv, uint32_t i, const Shared &S) {
    float2 v = sv[i];
    if (S.pend) {
      const float f = S.dtab[__popc(i & S.pmask)];
      v.x *= f;
      v.y *= f;
    }
    return v;
  }

  // Fused-gate pass (k = K).  PEND: the pending diagonal (scale * s^popc(i & pmask))
  // is applied to every loaded amplitude.  With op.stats the pass also sums, over
  // its outputs, t += |o|^2 and d += |o|^2 (1-g)^popc(i & smask) for the damping op
  // that follows.
  //
  // k = 1 gates take two groups a thread, so every matrix load serves both.
  template <int K>
  static constexpr int groups_per_thread() { return K == 1 ? 2 : 1; }

  template <int K, bool PEND>
  static __device__ __noinline__ void gate_pass(float2 *sv, uint32_t n, const TOp &op, const float2 *M,
                                         const Shared &S, double &t, double &d) {
    constexpr int D = 1 << K;
    constexpr int U = groups_per_thread<K>();
    uint32_t lo[K];
#pragma unroll
    for (int b = 0; b < K; ++b) lo[b] = (1u << op.q[b]) - 1;
    const uint32_t ng = 1u << (n - K);
    const bool stats = op.stats != 0;
    const uint32_t smask = op.smask;
    const uint32_t pmask = S.pmask;
    double lt = 0, ld = 0;
    for (uint32_t g0 = threadIdx.x; g0 < ng; g0 += kTThreads * U) {
      uint32_t base[U];
      float2 x[U][D];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint32_t g = g0 + u * kTThreads;
        uint32_t bb = g < ng ? g : 0;
#pragma unroll
        for (int b = 0; b < K; ++b) bb = ((bb & ~lo[b]) << 1) | (bb & lo[b]);
        base[u] = bb;
#pragma unroll
        for (int a = 0; a < D; ++a) {
          uint32_t o = bb;
#pragma unroll
          for (int b = 0; b < K; ++b)
            if ((a >> b) & 1) o += lo[b] + 1;
          float2 v = make_float2(0.f, 0.f);
          if (g < ng) v = sv[o];
          if (PEND) {
            const float f = S.dtab[__popc(o & pmask)];
            v.x *= f;
            v.y *= f;
          }
          x[u][a] = v;
        }
      }
#pragma unroll
      for (int r = 0; r < D; ++r) {
        float2 acc[U];
#pragma unroll
        for (int u = 0; u < U; ++u) acc[u] = make_float2(0.f, 0.f);
#pragma unroll
        for (int c = 0; c < D; ++c) {
          const float2 m = M[r * D + c];
#pragma unroll
          for (int u = 0; u < U; ++u) acc[u] = cmul_add(m, x[u][c], acc[u]);
        }
        uint32_t roff = 0;
#pragma unroll
        for (int b = 0; b < K; ++b)
          if ((r >> b) & 1) roff += lo[b] + 1;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (g0 + u * kTThreads < ng) {
            const uint32_t o = base[u] + roff;
            sv[o] = acc[u];
            if (stats) {
              const double p = (double)acc[u].x * acc[u].x + (double)acc[u].y * acc[u].y;
              lt += p;
              ld += p * S.stab[__popc(o & smask)];
            }
          }
        }
      }
    }
    t += lt;
    d += ld;
  }

  static __device__ void dispatch_gate(float2 *sv, uint32_t n, const TOp &op, const float2 *M, Shared &S,
                                double &t, double &d) {
    if (S.pend) {
      switch (op.k) {
      case 1: gate_pass<1, true>(sv, n, op, M, S, t, d); break;
      case 2: gate_pass<2, true>(sv, n, op, M, S, t, d); break;
      case 3: gate_pass<3, true>(sv, n, op, M, S, t, d); break;
      default: gate_pass<4, true>(sv, n, op, M, S, t, d); break;
      }
    } else {
      switch (op.k) {
      case 1: gate_pass<1, false>(sv, n, op, M, S, t, d); break;
      case 2: gate_pass<2, false>(sv, n, op, M, S, t, d); break;
      case 3: gate_pass<3, false>(sv, n, op, M, S, t, d); break;
      default: gate_pass<4, false>(sv, n, op, M, S, t, d); break;
      }
    }
  }

  // Stage a 2^k x 2^k matrix into shared memory.
  static __device__ void stage_matrix(float2 *Msm, const float2 *pool, uint32_t off, uint32_t entries) {
    for (uint32_t i = threadIdx.x; i < entries; i += kTThreads) Msm[i] = pool[off + i];
    __syncthreads();
  }

  // Materialise the pending diagonal (and optionally compute sums):
  // t = sum |a|^2, d = sum |a|^2 * w(i) with w = (1-g)^popc(i & mask), j = g * sum_{bit q} |a|^2.
  static __device__ __noinline__ void stats_pass(float2 *sv, uint32_t n, Shared &S, uint32_t mask, double g, uint32_t q,
                             double &t, double &d, double &j) {
    t = d = j = 0;
    fill_stab(S, g);
    const uint32_t N = 1u << n;
    for (uint32_t i = threadIdx.x; i < N; i += kTThreads) {
      float2 v = sv[i];
      if (S.pend) {
        const float f = S.dtab[__popc(i & S.pmask)];
        v.x *= f;
        v.y *= f;
        sv[i] = v;
      }
      const double p = (double)v.x * v.x + (double)v.y * v.y;
      t += p;
      d += p * S.stab[__popc(i & mask)];
      if ((i >> q) & 1) j += p;
    }
    __syncthreads();
    if (threadIdx.x == 0) S.pend = 0;
    block_sum3(S, t, d, j);
    j *= g;
  }

  static __device__ void set_pending(Shared &S, uint32_t mask, double gamma, double scale) {
    if (threadIdx.x == 0) {
      S.pend = 1;
      S.pmask = mask;
      const double s = sqrt(1.0 - gamma);
      double f = scale;
      for (uint32_t c = 0; c <= kTrajMaxQubits; ++c) {
        S.dtab[c] = (float)f;
        f *= s;
      }
    }
    __syncthreads();
  }

  // Elementwise single-qubit damping branch on qubit q: jump -> x0 = sqrt(g) x1, x1 = 0;
  // no jump -> x1 *= sqrt(1 - g).
  static __device__ __noinline__ void damp_apply(float2 *sv, uint32_t n, uint32_t q, double g, bool jump) {
    const uint32_t npair = 1u << (n - 1);
    const uint32_t lo = (1u << q) - 1;
    const float sj = (float)sqrt(g), sn = (float)sqrt(1.0 - g);
    for (uint32_t p = threadIdx.x; p < npair; p += kTThreads) {
      const uint32_t i0 = ((p & ~lo) << 1) | (p & lo), i1 = i0 | (1u << q);
      const float2 x1 = sv[i1];
      if (jump) {
        sv[i0] = make_float2(sj * x1.x, sj * x1.y);
        sv[i1] = make_float2(0.f, 0.f);
      } else {
        sv[i1] = make_float2(sn * x1.x, sn * x1.y);
      }
    }
    __syncthreads();
  }

  // General single-qubit channel: p_j = ||K_j psi||^2 (FP64), pick j, apply K_j / sqrt(p_j).
  static __device__ __noinline__ void chan_op(float2 *sv, uint32_t n, const TOp &op, const float2 *pool,
                                       float2 *Msm, Shared &S, uint64_t seed, uint32_t traj,
                                       uint32_t &ev) {
    const uint32_t N = 1u << n;
    stage_matrix(Msm, pool, op.mat, 4 * op.nk);
    const uint32_t q = op.q[0];
    const uint32_t lo = (1u << q) - 1;
    double pj[4] = {0, 0, 0, 0};
    for (uint32_t p = threadIdx.x; p < N / 2; p += kTThreads) {
      const uint32_t i0 = ((p & ~lo) << 1) | (p & lo), i1 = i0 | (1u << q);
      const float2 x0 = pend_load(sv, i0, S), x1 = pend_load(sv, i1, S);
      for (uint32_t b = 0; b < op.nk; ++b) {
        const float2 y0 = cmul_add(Msm[4 * b + 1], x1, cmul_add(Msm[4 * b], x0, make_float2(0, 0)));
        const float2 y1 = cmul_add(Msm[4 * b + 3], x1, cmul_add(Msm[4 * b + 2], x0, make_float2(0, 0)));
        pj[b] += (double)y0.x * y0.x + (double)y0.y * y0.y + (double)y1.x * y1.x + (double)y1.y * y1.y;
      }
    }
    double a = pj[0], b = pj[1], c = pj[2];
    block_sum3(S, a, b, c);
    double d3 = pj[3], z0 = 0, z1 = 0;
    block_sum3(S, d3, z0, z1);
    const double tot[4] = {a, b, c, d3};
    double sum = 0;
    for (uint32_t bb = 0; bb < op.nk; ++bb) sum += tot[bb];
    const double v = philox_uniform(seed, traj, ev++) * sum;
    uint32_t pick = op.nk - 1;
    double acc = 0;
    for (uint32_t bb = 0; bb < op.nk; ++bb) {
      acc += tot[bb];
      if (v < acc) {
        pick = bb;
        break;
      }
    }
    const float sc = (float)(tot[pick] > 0 ? 1.0 / sqrt(tot[pick]) : 0.0);
    const float2 *K = Msm + 4 * pick;
    for (uint32_t p = threadIdx.x; p < N / 2; p += kTThreads) {
      const uint32_t i0 = ((p & ~lo) << 1) | (p & lo), i1 = i0 | (1u << q);
      const float2 x0 = pend_load(sv, i0, S), x1 = pend_load(sv, i1, S);
      const float2 y0 = cmul_add(K[1], x1, cmul_add(K[0], x0, make_float2(0, 0)));
      const float2 y1 = cmul_add(K[3], x1, cmul_add(K[2], x0, make_float2(0, 0)));
      sv[i0] = make_float2(y0.x * sc, y0.y * sc);
      sv[i1] = make_float2(y1.x * sc, y1.y * sc);
    }
    __syncthreads();
    if (threadIdx.x == 0) S.pend = 0;
    __syncthreads();
  }

  // Applies a Pauli error op (one of three k-qubit matrices) as a gate pass.
  static __device__ __noinline__ void err_apply(float2 *sv, uint32_t n, const TOp &op, double u,
                                         const float2 *pool, float2 *Msm, Shared &S) {
    const uint32_t which = min(2u, (uint32_t)(u / (double)op.prob * 3.0));
    const uint32_t e = 1u << (2 * op.k);
    stage_matrix(Msm, pool, op.mat + which * e, e);
    TOp g = op;
    g.stats = 0;
    double t = 0, d = 0;
    dispatch_gate(sv, n, g, Msm, S, t, d);
    __syncthreads();
    if (threadIdx.x == 0) S.pend = 0;
    __syncthreads();
  }

  // Amplitude damping on op.mask: exact sampling of the joint jump pattern.
  static __device__ __noinline__ void damp_op(float2 *sv, uint32_t n, const TOp &op, Shared &S,
                                       uint64_t seed, uint32_t traj, uint32_t &ev, double T,
                                       double Dd, bool stats_valid) {
    const double g = (double)op.gamma;
    if (!stats_valid) {
      double j;
      stats_pass(sv, n, S, op.mask, g, 0, T, Dd, j);
    }
    const double u = philox_uniform(seed, traj, ev++);
    if (u * T < Dd) {  // no jump on any qubit of the mask
      set_pending(S, op.mask, g, 1.0 / sqrt(Dd));
      return;
    }
    // at least one jump: sample qubit by qubit, conditioned on a jump occurring
    if (S.pend) {
      double a, b, c;
      stats_pass(sv, n, S, 0, 0.0, 0, a, b, c);
    }
    bool need = true;
    for (uint32_t q = 0; q < n; ++q) {
      if (!((op.mask >> q) & 1)) continue;
      const uint32_t rem = op.mask & ~((1u << q) - 1);
      double t, zsum, j;
      stats_pass(sv, n, S, rem, g, q, t, zsum, j);
      const double p1 = need ? (t - zsum > 0 ? j / (t - zsum) : 1.0) : (t > 0 ? j / t : 0.0);
      const double v = philox_uniform(seed, traj, ev++);
      const bool jump = v < p1;
      damp_apply(sv, n, q, g, jump);
      if (jump) need = false;
    }
    double t, a, b;
    stats_pass(sv, n, S, 0, 0.0, 0, t, a, b);
    set_pending(S, 0, 0.0, t > 0 ? 1.0 / sqrt(t) : 1.0);
  }

  // The passes of a segment.  A block in place costs its loads' latency through L2
  // and a matrix entry from shared memory for every four FMAs: 27 us a block of a
  // 16-qubit state, whose arithmetic takes 4 to 9.  2048 trajectories of 16 qubits and
  // depth 30 (fused at 3): 87.5 -> 73 ms; 18 qubits, depth 20 (296): 54 -> 37 ms; 12
  // qubits (2048): 5.8 -> 4.8 ms.  What is left is latency: 16 warps issue 0.45
  // instructions a clock and scheduler, waiting for shared memory and for each other.
  // The first applies the pending diagonal as its tiles
  // arrive, the last sums t and d (as gate_pass does) as its tiles leave.  Two tile
  // buffers: the next tile is copied in while this one is computed.
  static __device__ __noinline__ void run_segment(float2 *sv, uint32_t n, const TSeg &seg, const TSegs &G,
                                                  unsigned char *smem, const Shared &S, double &t,
                                                  double &d) {
    float *const mats = reinterpret_cast<float *>(smem);
    cb2::PassGateArgs32 *const args = reinterpret_cast<cb2::PassGateArgs32 *>(smem + G.mat_cap);
    const bool pend = S.pend != 0;
    const uint32_t pmask = S.pmask;
    for (uint32_t pi = 0; pi < seg.n_passes; ++pi) {
      const TSegPass &P = G.passes[seg.pass0 + pi];
      const uint32_t tb = P.tb, tile = 1u << tb, n_tiles = 1u << (n - tb), n_gates = P.n_gates;
      float2 *const buf = reinterpret_cast<float2 *>(smem + G.mat_cap + kSegArgBytes);
      for (uint32_t i = threadIdx.x; i < n_gates * sizeof(cb2::PassGateArgs32) / 4; i += NT)
        reinterpret_cast<uint32_t *>(args)[i] = reinterpret_cast<const uint32_t *>(G.gates + P.gate0)[i];
      for (uint32_t i = 16 * threadIdx.x; i < P.mat_bytes; i += 16 * NT)
        __pipeline_memcpy_async(smem + i, reinterpret_cast<const char *>(G.mats + P.mat) + i, 16);
      // pairs of amplitudes: tile bits 1 .. kTLogThreads are the thread index, the
      // bits above the rounds; where each starts, and the tiles' first amplitudes in
      // ascending order of the other qubits
      constexpr uint32_t R = (1u << kSegMaxTile) / (2 * NT);
      uint32_t at[R], tmask = 0;
      for (uint32_t b = 0; b < tb; ++b) tmask |= P.stride[b];
      uint32_t off = 0;
#pragma unroll
      for (uint32_t b = 0; b < kTLogThreads; ++b)
        if (b + 1 < tb && ((threadIdx.x >> b) & 1)) off += P.stride[b + 1];
#pragma unroll
      for (uint32_t u = 0; u < R; ++u) {
        at[u] = off;
#pragma unroll
        for (uint32_t b = kTLogThreads + 1; b < kSegMaxTile; ++b)
          if (b < tb && ((u >> (b - kTLogThreads - 1)) & 1)) at[u] += P.stride[b];
      }
      const uint32_t rounds = 2 * threadIdx.x < tile ? (tile + 2 * NT - 1) / (2 * NT) : 0;
      uint32_t base = 0, next = 0;  // of this tile and the next one to fetch
      auto fetch = [&](float2 *to) {
#pragma unroll
        for (uint32_t u = 0; u < R; ++u)
          if (u < rounds)
            __pipeline_memcpy_async(&to[cb2::pass_swz32(2 * (threadIdx.x + u * NT))], &sv[next + at[u]], 16);
        next = ((next | tmask) + 1) & ~tmask;
      };
      fetch(buf);
      __pipeline_commit();
      for (uint32_t tl = 0; tl < n_tiles; ++tl) {
        float2 *s = buf + (tl & 1) * tile;
        if (tl + 1 < n_tiles) fetch(buf + ((tl + 1) & 1) * tile);
        __pipeline_commit();
        __pipeline_wait_prior(1);
        if (pend && pi == 0) {  // a thread scales what it copied
#pragma unroll
          for (uint32_t u = 0; u < R; ++u)
            if (u < rounds) {
              const uint32_t i = base + at[u];
              float4 *v = reinterpret_cast<float4 *>(&s[cb2::pass_swz32(2 * (threadIdx.x + u * NT))]);
              const float f0 = S.dtab[__popc(i & pmask)], f1 = S.dtab[__popc((i | 1) & pmask)];
              float4 x = *v;
              x.x *= f0;
              x.y *= f0;
              x.z *= f1;
              x.w *= f1;
              *v = x;
            }
        }
        __syncthreads();
        const float *m = mats;
        for (uint32_t gi = 0; gi < n_gates; ++gi) {
          const cb2::PassGateArgs32 &g = args[gi];
          if (g.k == 4) {
            cb2::pass_gate32<NT, 4, 2, 2, false>(s, m, g, tb);
            m += 3 * 256;
          } else if (g.k == 3) {
            cb2::pass_gate32<NT, 3, 1, 2, false>(s, m, g, tb);
            m += 3 * 64;
          } else if (g.k == 2) {
            cb2::pass_gate32<NT, 2, 1, 4, false>(s, m, g, tb);
            m += 3 * 16;
          } else {
            cb2::pass_gate32<NT, 1, 1, 4, false>(s, m, g, tb);
            m += 3 * 4;
          }
          __syncthreads();
        }
        const bool sum = seg.stats && pi + 1 == seg.n_passes;
#pragma unroll
        for (uint32_t u = 0; u < R; ++u)
          if (u < rounds) {
            const uint32_t i = base + at[u];
            const float4 v = *reinterpret_cast<const float4 *>(&s[cb2::pass_swz32(2 * (threadIdx.x + u * NT))]);
            *reinterpret_cast<float4 *>(&sv[i]) = v;
            if (sum) {
              const double p0 = (double)v.x * v.x + (double)v.y * v.y;
              const double p1 = (double)v.z * v.z + (double)v.w * v.w;
              t += p0 + p1;
              d += p0 * S.stab[__popc(i & seg.smask)] + p1 * S.stab[__popc((i | 1) & seg.smask)];
            }
          }
        base = ((base | tmask) + 1) & ~tmask;
        __syncthreads();  // the buffer is read out, the state written
      }
    }
  }

  // End of a trajectory: <Z_q> for every qubit and one sampled bitstring.
  static __device__ __noinline__ void finish(float2 *sv, uint32_t n, Shared &S, double *csum, uint64_t seed,
                                      uint32_t traj, double *z_row, uint32_t *sample_slot) {
    const uint32_t N = 1u << n;
    const uint32_t c = n > kTLogThreads ? n - kTLogThreads : 0;  // bits inside a thread's chunk
    const uint32_t chunk = 1u << c;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // The pending diagonal stays pending: every read below applies it.
    if (c >= 5) {
      // one coalesced pass: a warp sums a chunk, so a lane's place in it is fixed and
      // its total serves the five lowest qubits (not a chunk a thread, which reads
      // 32 lines a warp, again for every three of its qubits)
      constexpr int HIGH = (int)kTrajMaxQubits - (int)kTLogThreads - 5;
      double tot = 0, high[HIGH];
#pragma unroll
      for (int q = 0; q < HIGH; ++q) high[q] = 0;
      for (uint32_t ch = warp; ch < (uint32_t)NT; ch += NT / 32) {
        double sum = 0;
        for (uint32_t j = 0; j < chunk >> 5; ++j) {
          const float2 v = pend_load(sv, (ch << c) + (j << 5) + lane, S);
          const double p = (double)v.x * v.x + (double)v.y * v.y;
          sum += p;
#pragma unroll
          for (int q = 0; q < HIGH; ++q)
            if ((j >> q) & 1) high[q] += p;
        }
        tot += sum;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
        if (lane == 0) csum[ch] = sum;
      }
      for (uint32_t q0 = 0; q0 < c; q0 += 3) {
        double acc[3];
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          const int q = (int)q0 + j;
          acc[j] = q < 5 && ((lane >> q) & 1) ? tot : 0.0;
#pragma unroll
          for (int h = 0; h < HIGH; ++h)
            if (q == 5 + h) acc[j] = high[h];
        }
        block_sum3(S, acc[0], acc[1], acc[2]);
        if (threadIdx.x < 3 && q0 + threadIdx.x < c) z_row[q0 + threadIdx.x] = acc[threadIdx.x];
      }
    } else {
      const bool active = (threadIdx.x << c) < N;
      const uint32_t base = threadIdx.x << c;
      double my = 0;
      if (active)
        for (uint32_t i = 0; i < chunk; ++i) {
          const float2 v = pend_load(sv, base + i, S);
          my += (double)v.x * v.x + (double)v.y * v.y;
        }
      csum[threadIdx.x] = my;
      __syncthreads();
      // qubits inside a chunk, three per block reduction
      for (uint32_t q0 = 0; q0 < c; q0 += 3) {
        double acc[3] = {0, 0, 0};
        if (active)
          for (uint32_t i = 0; i < chunk; ++i) {
            const float2 v = pend_load(sv, base + i, S);
            const double p = (double)v.x * v.x + (double)v.y * v.y;
            for (uint32_t j = 0; j < 3; ++j)
              if (q0 + j < c && ((i >> (q0 + j)) & 1)) acc[j] += p;
          }
        block_sum3(S, acc[0], acc[1], acc[2]);
        if (threadIdx.x < 3 && q0 + threadIdx.x < c) z_row[q0 + threadIdx.x] = acc[threadIdx.x];
      }
    }
    __syncthreads();
    // qubits that index the threads: thread j sums the chunk sums with bit j set
    const uint32_t nthr = N >> c;
    if (threadIdx.x < n - c) {
      double x = 0;
      for (uint32_t tt = 0; tt < nthr; ++tt)
        if ((tt >> threadIdx.x) & 1) x += csum[tt];
      z_row[c + threadIdx.x] = x;
    }
    __syncthreads();  // the sums over csum are done
    if (threadIdx.x == 0) {
      double tot = 0;
      for (uint32_t tt = 0; tt < nthr; ++tt) tot += csum[tt];
      S.vals[3] = tot;
      // inverse-CDF sample: find the chunk, then the amplitude (a target that
      // rounding leaves past the end takes the last one of nonzero weight)
      const double target = philox_uniform(seed, traj, 0xFFFFFFF0u) * tot;
      double acc = 0, acc_t = 0;
      uint32_t tsel = nthr;
      for (uint32_t tt = 0; tt < nthr; ++tt) {
        if (csum[tt] > 0) {
          tsel = tt;
          acc_t = acc;
        }
        if (acc + csum[tt] > target) break;
        acc += csum[tt];
      }
      S.vals[0] = target;
      S.vals[1] = acc_t;
      S.vals[2] = (double)(tsel == nthr ? 0 : tsel);  // an all-zero state (cannot arise from normalised branches)
    }
    __syncthreads();
    const uint32_t first = (uint32_t)S.vals[2] << c;
    // the chosen chunk's probabilities, NT at a time
    double acc = S.vals[1];
    const double target = S.vals[0];
    uint32_t isel = first;
    for (uint32_t part = 0; part < chunk; part += NT) {
      const uint32_t len = min(chunk - part, (uint32_t)NT);
      if (threadIdx.x < len) {
        const float2 v = pend_load(sv, first + part + threadIdx.x, S);
        csum[threadIdx.x] = (double)v.x * v.x + (double)v.y * v.y;
      }
      __syncthreads();
      if (threadIdx.x == 0)
        for (uint32_t i = 0; i < len && !(acc > target); ++i) {
          const double p = csum[i];
          if (p > 0) isel = first + part + i;
          acc += p;
        }
      __syncthreads();
    }
    if (threadIdx.x == 0 && sample_slot) *sample_slot = isel;
    __syncthreads();
    const double tot = S.vals[3];
    if (threadIdx.x < n) {
      const double p1 = z_row[threadIdx.x];
      z_row[threadIdx.x] = tot > 0 ? 1.0 - 2.0 * p1 / tot : 0.0;
    }
    __syncthreads();
  }

  // The same in programs without segments, mostly small states whose chunks are a few
  // amplitudes: the pending diagonal is materialised first.
  static __device__ __noinline__ void finish_plain(float2 *sv, uint32_t n, Shared &S, double *csum, uint64_t seed,
                                      uint32_t traj, double *z_row, uint32_t *sample_slot) {
    {
      double t, a, b;
      stats_pass(sv, n, S, 0, 0.0, 0, t, a, b);  // materialise the pending diagonal
    }
    const uint32_t N = 1u << n;
    const uint32_t c = n > kTLogThreads ? n - kTLogThreads : 0;  // bits inside a thread's chunk
    const uint32_t chunk = 1u << c;
    const bool active = (threadIdx.x << c) < N;
    const uint32_t base = threadIdx.x << c;
    double my = 0;
    if (active)
      for (uint32_t i = 0; i < chunk; ++i) {
        const float2 v = sv[base + i];
        my += (double)v.x * v.x + (double)v.y * v.y;
      }
    csum[threadIdx.x] = my;
    __syncthreads();
    // qubits inside a chunk, three per block reduction
    for (uint32_t q0 = 0; q0 < c; q0 += 3) {
      double acc[3] = {0, 0, 0};
      if (active)
        for (uint32_t i = 0; i < chunk; ++i) {
          const float2 v = sv[base + i];
          const double p = (double)v.x * v.x + (double)v.y * v.y;
          for (uint32_t j = 0; j < 3; ++j)
            if (q0 + j < c && ((i >> (q0 + j)) & 1)) acc[j] += p;
        }
      block_sum3(S, acc[0], acc[1], acc[2]);
      if (threadIdx.x < 3 && q0 + threadIdx.x < c) z_row[q0 + threadIdx.x] = acc[threadIdx.x];
    }
    // qubits that index the threads: thread j sums the chunk sums with bit j set
    const uint32_t nthr = N >> c;
    if (threadIdx.x < n - c) {
      double x = 0;
      for (uint32_t tt = 0; tt < nthr; ++tt)
        if ((tt >> threadIdx.x) & 1) x += csum[tt];
      z_row[c + threadIdx.x] = x;
    }
    if (threadIdx.x == 0) {
      double tot = 0;
      for (uint32_t tt = 0; tt < nthr; ++tt) tot += csum[tt];
      S.vals[3] = tot;
      // inverse-CDF sample: find the chunk, then the amplitude (a target that
      // rounding leaves past the end takes the last one of nonzero weight)
      const double target = philox_uniform(seed, traj, 0xFFFFFFF0u) * tot;
      double acc = 0, acc_t = 0;
      uint32_t tsel = nthr;
      for (uint32_t tt = 0; tt < nthr; ++tt) {
        if (csum[tt] > 0) {
          tsel = tt;
          acc_t = acc;
        }
        if (acc + csum[tt] > target) break;
        acc += csum[tt];
      }
      acc = acc_t;
      if (tsel == nthr) tsel = 0;  // an all-zero state (cannot arise from normalised branches)
      uint32_t isel = tsel << c;
      for (uint32_t i = 0; i < chunk; ++i) {
        const float2 v = sv[(tsel << c) + i];
        const double p = (double)v.x * v.x + (double)v.y * v.y;
        if (p > 0) isel = (tsel << c) + i;
        acc += p;
        if (acc > target) break;
      }
      if (sample_slot) *sample_slot = isel;
    }
    __syncthreads();
    const double tot = S.vals[3];
    if (threadIdx.x < n) {
      const double p1 = z_row[threadIdx.x];
      z_row[threadIdx.x] = tot > 0 ? 1.0 - 2.0 * p1 / tot : 0.0;
    }
    __syncthreads();
  }
};

// SEG: the program has segments.
template <int NT, bool SEG>
__device__ __forceinline__ void trajectories(const TOp *__restrict__ ops, uint32_t n_ops,
                                             const float2 *__restrict__ pool, float2 *__restrict__ ws,
                                             uint32_t n, const TRun *__restrict__ run,
                                             double *__restrict__ out_z,
                                             uint32_t *__restrict__ out_sample, const TSegs &segs,
                                             unsigned char *seg_smem) {
  __shared__ Shared S;
  __shared__ float2 Msm[1 << (2 * kTrajMaxGate)];
  __shared__ double csum[NT];
  using Tr = Traj<NT>;
  const uint32_t n_traj = run->n_traj;
  const uint64_t seed = run->seed;
  const uint32_t N = 1u << n;
  float2 *sv = ws + ((size_t)blockIdx.x << n);
  for (uint32_t lt = blockIdx.x; lt < n_traj; lt += gridDim.x) {
    const uint32_t traj = run->first + lt;  // draws depend on the global index only
    for (uint32_t i = threadIdx.x; i < N; i += NT)
      sv[i] = make_float2(i == 0 ? 1.f : 0.f, 0.f);
    if (threadIdx.x == 0) S.pend = 0;
    __syncthreads();
    uint32_t ev = 0;
    bool stats_valid = false;
    double T = 1.0, Dd = 1.0;
    for (uint32_t oi = 0; oi < n_ops; ++oi) {
      if constexpr (SEG) {
        if (const uint32_t start = segs.starts[oi]) {
          const TSeg seg = segs.segs[start - 1];
          int fired = 0;
          for (uint32_t e = threadIdx.x; e < seg.n_err; e += NT)
            fired |= philox_uniform(seed, traj, ev + e) < (double)ops[segs.sites[seg.err0 + e]].prob;
          if (!__syncthreads_or(fired)) {
            if (seg.stats) Tr::fill_stab(S, (double)seg.sgamma);
            double t = 0, d = 0, z = 0;
            Tr::run_segment(sv, n, seg, segs, seg_smem, S, t, d);
            if (threadIdx.x == 0) S.pend = 0;
            if (seg.stats) {
              Tr::block_sum3(S, t, d, z);
              T = t;
              Dd = d;
            } else {
              __syncthreads();
            }
            stats_valid = seg.stats != 0;
            ev += seg.n_err;
            oi = seg.end_op - 1;
            continue;
          }
        }
      }
      const TOp op = ops[oi];
      if (op.type == T_GATE) {
        if (op.stats) Tr::fill_stab(S, (double)op.sgamma);
        Tr::stage_matrix(Msm, pool, op.mat, 1u << (2 * op.k));
        double t = 0, d = 0, z = 0;
        Tr::dispatch_gate(sv, n, op, Msm, S, t, d);
        __syncthreads();
        if (threadIdx.x == 0) S.pend = 0;
        if (op.stats) {
          Tr::block_sum3(S, t, d, z);
          T = t;
          Dd = d;
        } else {
          __syncthreads();
        }
        stats_valid = op.stats != 0;
        if (op.nerr) {
          // all error sites of this block decide in parallel (event ev + e for site e)
          int fired = 0;
          if (threadIdx.x < op.nerr)
            fired = philox_uniform(seed, traj, ev + threadIdx.x) < (double)ops[oi + 1 + threadIdx.x].prob;
          if (__syncthreads_or(fired)) {
            for (uint32_t e = 0; e < op.nerr; ++e) {
              const TOp eo = ops[oi + 1 + e];
              const double u = philox_uniform(seed, traj, ev + e);
              if (u < (double)eo.prob) {
                Tr::err_apply(sv, n, eo, u, pool, Msm, S);
                stats_valid = false;
              }
            }
          }
          ev += op.nerr;
          oi += op.nerr;
        }
      } else if (op.type == T_ERR) {  // not preceded by a gate block (kept for completeness)
        const double u = philox_uniform(seed, traj, ev++);
        if (u < (double)op.prob) {
          Tr::err_apply(sv, n, op, u, pool, Msm, S);
          stats_valid = false;
        }
      } else if (op.type == T_DAMP) {
        Tr::damp_op(sv, n, op, S, seed, traj, ev, T, Dd, stats_valid);
        stats_valid = false;
      } else if (op.type == T_CHAN) {
        Tr::chan_op(sv, n, op, pool, Msm, S, seed, traj, ev);
        stats_valid = false;
      }
    }
    if constexpr (SEG) {
      Tr::finish(sv, n, S, csum, seed, traj, out_z + (size_t)lt * n, out_sample ? out_sample + lt : nullptr);
    } else {
      Tr::finish_plain(sv, n, S, csum, seed, traj, out_z + (size_t)lt * n, out_sample ? out_sample + lt : nullptr);
    }
  }
}

}  // namespace
