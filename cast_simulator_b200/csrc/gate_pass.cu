// Merged gate passes: several gates of a program applied to the statevector for
// one read and one write of it (complex128, k <= 4).
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
//
// Which tile bits the lanes walk is free: members (K order), rows and groups may
// be taken in any order.  The host picks them so that the eight lanes of a
// 16-byte shared-memory wavefront fall into different bank groups under the
// tile's XOR swizzle (bank group = XOR of the index's 3-bit fields).
#include "internal.hpp"
#include "pass_plan.hpp"

#include <algorithm>
#include <cstring>
#include <memory>
#include <mutex>

#include <cuda_pipeline.h>

namespace cb2 {

namespace {

constexpr int kPassThreads = 128;
constexpr int kPassWarps = kPassThreads / 32;
constexpr uint32_t kPassMaxTile = 12;
constexpr uint32_t kPassMinTile = 7;  // a 4-qubit gate and the 8 groups of a fragment
constexpr uint32_t kPassLow = 3;      // lowest qubits every tile holds: 128-byte runs

// One gate of a pass.  Index contributions are swizzled tile offsets; XOR of the
// contributions of an index's set bits is its place in shared memory.
struct PassGateArgs {
  uint32_t mat;          // first double of its fragments in the pool
  uint16_t k;            // 3 or 4
  uint16_t ld_lane[5];   // load: lane bits 0, 1 -> member bits 0, 1; 2..4 -> group bits 0..2
  uint16_t ld_k[2];      // load: member bits 2, 3 (the k steps)
  uint16_t st_lane[5];   // store: lane bits 0, 1 -> group bits 1, 2; 2..4 -> row bits 0..2
  uint16_t st_row;       // store: row bit 3 (k = 4)
  uint16_t st_col;       // store: group bit 0 (the fragment's register index)
  uint16_t blk[kPassMaxTile - 6];  // group bits 3, 4, ...
};

struct PassArgs {
  uint64_t stride[kPassMaxTile];  // tile bit -> amplitude stride
  uint32_t tb, n_gates;
  PassGateArgs g[kMaxPassGates];
};

__host__ __device__ inline uint32_t pass_swz(uint32_t i) {
  return i ^ (((i >> 3) ^ (i >> 6) ^ (i >> 9)) & 7u);
}

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

__device__ __forceinline__ uint32_t lane_bits(const uint16_t (&c)[5], int lane) {
  uint32_t x = 0;
#pragma unroll
  for (int b = 0; b < 5; ++b)
    if ((lane >> b) & 1) x ^= c[b];
  return x;
}

template <int NB>
__device__ __forceinline__ uint32_t block_bits(const PassGateArgs &g, uint32_t blk) {
  uint32_t x = 0;
#pragma unroll
  for (int b = 0; b < NB; ++b)
    if ((blk >> b) & 1) x ^= g.blk[b];
  return x;
}

// 4-qubit gate, three real products: S1 += c (a + b), S2 += (d - c) a,
// S3 += (c + d) b, Re = S1 - S3, Im = S1 + S2.  (Accumulating Re and Im on top of
// S1 saves their eight adds a block, which share the pipe, and 5% of the time at 30
// qubits, but moves the state 10% further from its 64-bit value: not done.)
__device__ __forceinline__ void pass_gate4(double2 *s, const double *__restrict__ pool,
                                           const PassGateArgs &g, uint32_t n_blk, int warp, int lane) {
  double a[3][2][4];
  const double *m = pool + g.mat + lane;
#pragma unroll
  for (int p = 0; p < 3; ++p)
#pragma unroll
    for (int rb = 0; rb < 2; ++rb)
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) a[p][rb][ks] = __ldg(m + 32 * ((p * 2 + rb) * 4 + ks));
  const uint32_t ld = lane_bits(g.ld_lane, lane), st = lane_bits(g.st_lane, lane);
  for (uint32_t blk = warp; blk < n_blk; blk += kPassWarps) {
    const uint32_t bx = block_bits<kPassMaxTile - 7>(g, blk);
    double2 x[4];
#pragma unroll
    for (int ks = 0; ks < 4; ++ks)
      x[ks] = s[bx ^ ld ^ (ks & 1 ? g.ld_k[0] : 0) ^ (ks & 2 ? g.ld_k[1] : 0)];
    double c[3][2][2] = {};
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      const double sum = x[ks].x + x[ks].y;
#pragma unroll
      for (int rb = 0; rb < 2; ++rb) {
        dmma(c[0][rb], a[0][rb][ks], sum);
        dmma(c[1][rb], a[1][rb][ks], x[ks].x);
        dmma(c[2][rb], a[2][rb][ks], x[ks].y);
      }
    }
#pragma unroll
    for (int rb = 0; rb < 2; ++rb)
#pragma unroll
      for (int i = 0; i < 2; ++i)
        s[bx ^ st ^ (rb ? g.st_row : 0) ^ (i ? g.st_col : 0)] =
            make_double2(c[0][rb][i] - c[2][rb][i], c[0][rb][i] + c[1][rb][i]);
  }
}

// 3-qubit gate, four real products: Re = C a - D b, Im = D a + C b.  U group
// blocks at once give the tensor pipe independent accumulators.
template <int U>
__device__ __forceinline__ void pass_gate3_blocks(double2 *s, const double (&c)[2], const double (&d)[2],
                                                  const PassGateArgs &g, uint32_t ld, uint32_t st,
                                                  uint32_t blk) {
  uint32_t bx[U];
  double2 x[U][2];
  double re[U][2] = {}, im[U][2] = {};
#pragma unroll
  for (int u = 0; u < U; ++u) {
    bx[u] = block_bits<kPassMaxTile - 6>(g, blk + u * kPassWarps);
    x[u][0] = s[bx[u] ^ ld];
    x[u][1] = s[bx[u] ^ ld ^ g.ld_k[0]];
  }
#pragma unroll
  for (int ks = 0; ks < 2; ++ks)
#pragma unroll
    for (int u = 0; u < U; ++u) {
      dmma(re[u], c[ks], x[u][ks].x);
      dmma(im[u], c[ks], x[u][ks].y);
      dmma(re[u], -d[ks], x[u][ks].y);
      dmma(im[u], d[ks], x[u][ks].x);
    }
#pragma unroll
  for (int u = 0; u < U; ++u)
#pragma unroll
    for (int i = 0; i < 2; ++i) s[bx[u] ^ st ^ (i ? g.st_col : 0)] = make_double2(re[u][i], im[u][i]);
}

__device__ __forceinline__ void pass_gate3(double2 *s, const double *__restrict__ pool,
                                           const PassGateArgs &g, uint32_t n_blk, int warp, int lane) {
  const double *m = pool + g.mat + lane;
  const double c[2] = {__ldg(m), __ldg(m + 32)}, d[2] = {__ldg(m + 64), __ldg(m + 96)};
  const uint32_t ld = lane_bits(g.ld_lane, lane), st = lane_bits(g.st_lane, lane);
  uint32_t blk = warp;
  for (; blk + 3 * kPassWarps < n_blk; blk += 4 * kPassWarps)
    pass_gate3_blocks<4>(s, c, d, g, ld, st, blk);
  for (; blk < n_blk; blk += kPassWarps) pass_gate3_blocks<1>(s, c, d, g, ld, st, blk);
}

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
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (uint32_t gi = 0; gi < a.n_gates; ++gi) {
    const PassGateArgs &g = a.g[gi];
    if (g.k == 4) pass_gate4(s, pool, g, tile >> 7, warp, lane);
    else pass_gate3(s, pool, g, tile >> 6, warp, lane);
    __syncthreads();
  }
#pragma unroll 8
  for (uint32_t u = 0; u < rounds; ++u) psi[round_off(u)] = s[pass_swz(threadIdx.x + u * kPassThreads)];
}

// ── complex64 ────────────────────────────────────────────────────────────────
//
// The same passes in FP32, bound by the FP32 pipe: 24 packed pair FMAs
// (__ffma2_rn, two rows at once) an amplitude and 4-qubit gate.  A thread takes U
// gather groups and, of a 4-qubit gate, half the rows (its partner for the other
// half is in the same warp and reads the same amplitudes: a broadcast).  It walks
// the columns with all its sums in registers; per column it reads U amplitudes
// from the tile and its rows of the matrix, staged in shared memory one gate
// ahead, at addresses the lanes share.  The FMA pipe is 59% busy (register
// operands: three 64-bit reads a packed FMA); whole rows of two groups a thread
// with the matrix read through L1 ran at 0.71 of this (28 qubits, fused at 4:
// 64.3 against 46.8 ms; one gate a pass 56.0).  30 qubits, complex64, depth 20,
// fused at 4: 232 -> 200 ms; 26 qubits fused at 3: 21.4 -> 12.3 ms, at 2: 40.4 ->
// 22.9 ms.  Every row is the same FMA sequence as in the one-gate kernels.
constexpr uint32_t kPass32MaxTile = 13;  // 64 KB: three CTAs an SM
constexpr uint32_t kPass32MinTile = 8;
constexpr uint32_t kPass32Low = 4;       // 128-byte runs

constexpr uint32_t kPass32MatBytes = 3 * 256 * sizeof(float);

struct PassGateArgs32 {
  uint32_t mat;           // first float of its columns in the pool
  uint16_t k;             // 3 or 4
  uint16_t member[4];     // gate bits
  uint16_t group[kPass32MaxTile - 3];  // group bits
};

struct PassArgs32 {
  uint64_t stride[kPass32MaxTile];
  uint32_t tb, n_gates;
  PassGateArgs32 g[kMaxPassGates];
};

// 16-byte units of two amplitudes; bank group = XOR of the unit's 3-bit fields.
__host__ __device__ inline uint32_t pass_swz32(uint32_t i) {
  const uint32_t u = i >> 1;
  return ((u ^ (((u >> 3) ^ (u >> 6) ^ (u >> 9)) & 7u)) << 1) | (i & 1u);
}

template <int K>
__device__ __forceinline__ uint32_t member_bits32(const PassGateArgs32 &g, int a) {
  uint32_t o = 0;
#pragma unroll
  for (int b = 0; b < K; ++b)
    if ((a >> b) & 1) o ^= g.member[b];
  return o;
}

// Rows of part `half` of 1 / H of a gate for U groups at tile offsets gb.  Column c
// of the matrix holds six floats a row pair: k = 4 (c_0, c_1, (d-c)_0, (d-c)_1,
// (c+d)_0, (c+d)_1), three products; k = 3 (re_0, re_1, im_0, im_1, -im_0, -im_1),
// four.  A thread that is not `live` takes part in the barrier only.
template <int K, int H, int U>
__device__ __forceinline__ void pass_groups32(float2 *s, const float *mat, const PassGateArgs32 &g,
                                              const uint32_t (&gb)[U], uint32_t half, bool live) {
  constexpr int D = 1 << K, P = D / 2 / H, S = K == 4 ? 3 : 2;  // row pairs, sums a row pair
  const float4 *m = reinterpret_cast<const float4 *>(mat) + half * (3 * P / 2);
  float2 acc[U][S][P];
#pragma unroll
  for (int u = 0; u < U; ++u)
#pragma unroll
    for (int i = 0; i < S; ++i)
#pragma unroll
      for (int p = 0; p < P; ++p) acc[u][i][p] = make_float2(0.f, 0.f);
#pragma unroll
  for (int c = 0; c < D; ++c) {
    float2 xr[U], xi[U], xs[U];
    const uint32_t off = member_bits32<K>(g, c);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const float2 x = s[gb[u] ^ off];
      xr[u] = make_float2(x.x, x.x);
      xi[u] = make_float2(x.y, x.y);
      const float sum = x.x + x.y;
      xs[u] = make_float2(sum, sum);
    }
#pragma unroll
    for (int h = 0; h < P / 2; ++h) {  // two row pairs: three 16-byte loads
      const float4 *mc = m + 3 * (c * (D / 4) + h);
      const float4 m0 = mc[0], m1 = mc[1], m2 = mc[2];
      const float2 e[2][3] = {{make_float2(m0.x, m0.y), make_float2(m0.z, m0.w), make_float2(m1.x, m1.y)},
                              {make_float2(m1.z, m1.w), make_float2(m2.x, m2.y), make_float2(m2.z, m2.w)}};
#pragma unroll
      for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int p = 2 * h + q;
          if constexpr (K == 4) {
            acc[u][0][p] = __ffma2_rn(e[q][0], xs[u], acc[u][0][p]);
            acc[u][1][p] = __ffma2_rn(e[q][1], xr[u], acc[u][1][p]);
            acc[u][2][p] = __ffma2_rn(e[q][2], xi[u], acc[u][2][p]);
          } else {
            acc[u][0][p] = __ffma2_rn(e[q][2], xi[u], __ffma2_rn(e[q][0], xr[u], acc[u][0][p]));
            acc[u][1][p] = __ffma2_rn(e[q][1], xr[u], __ffma2_rn(e[q][0], xi[u], acc[u][1][p]));
          }
        }
    }
  }
  if constexpr (H > 1) {
    __syncwarp();  // the partner has read this group
    if (!live) return;
  }
  uint32_t top = 0;  // the half's row bits
  if constexpr (H == 2) top = half ? g.member[K - 1] : 0;
#pragma unroll
  for (int u = 0; u < U; ++u)
#pragma unroll
    for (int p = 0; p < P; ++p) {
      float2 re = acc[u][0][p], im = acc[u][1][p];
      if constexpr (K == 4) {
        const float2 s3 = acc[u][S - 1][p];
        im = __fadd2_rn(re, im);
        re = __fadd2_rn(re, make_float2(-s3.x, -s3.y));
      }
      s[gb[u] ^ top ^ member_bits32<K>(g, 2 * p)] = make_float2(re.x, im.x);
      s[gb[u] ^ top ^ member_bits32<K>(g, 2 * p + 1)] = make_float2(re.y, im.y);
    }
}

// A gate on the whole tile; H threads share a group, lane bit 4 telling them apart.
template <int K, int H, int U>
__device__ __forceinline__ void pass_gate32(float2 *s, const float *mat, const PassGateArgs32 &g,
                                            uint32_t tb) {
  constexpr uint32_t GT = kPassThreads / H;  // groups the CTA takes at once
  constexpr int TB = H == 2 ? 6 : 7;
  const uint32_t half = H == 2 ? (threadIdx.x >> 4) & 1 : 0;
  const uint32_t gt = H == 2 ? (threadIdx.x & 15) | (threadIdx.x >> 5) << 4 : threadIdx.x;
  auto offset = [&](uint32_t group) {
    uint32_t o = 0;
#pragma unroll
    for (int b = 0; b < (int)kPass32MaxTile - 3; ++b)
      if ((group >> b) & 1) o ^= g.group[b];
    return o;
  };
  const uint32_t groups = 1u << (tb - K), t = offset(gt);
  if (groups >= U * GT) {
    for (uint32_t it = 0; it < groups >> TB; it += U) {
      uint32_t gb[U];
#pragma unroll
      for (int u = 0; u < U; ++u) gb[u] = t ^ offset((it + u) << TB);
      pass_groups32<K, H, U>(s, mat, g, gb, half, true);
    }
  } else {
    for (uint32_t it = 0; it * GT < groups; ++it) {
      const bool live = it * GT + gt < groups;
      const uint32_t gb[1] = {live ? t ^ offset(it << TB) : 0};
      if (H > 1 || live) pass_groups32<K, H, 1>(s, mat, g, gb, half, live);
    }
  }
}

__global__ void __launch_bounds__(kPassThreads, 3)
    k_gate_pass32(float2 *__restrict__ psi, const float *__restrict__ pool,
                  const __grid_constant__ PassArgs32 a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float *mat = reinterpret_cast<float *>(smem_raw);  // two gates' matrices
  float2 *s = reinterpret_cast<float2 *>(smem_raw + 2 * kPass32MatBytes);
  auto fetch_matrix = [&](uint32_t gi) {
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
    if (g.k == 4) pass_gate32<4, 2, 2>(s, m, g, a.tb);
    else pass_gate32<3, 1, 4>(s, m, g, a.tb);
  }
  __syncthreads();
#pragma unroll 8
  for (uint32_t u = 0; u < rounds; ++u)
    *reinterpret_cast<float4 *>(&psi[round_off(u)]) =
        *reinterpret_cast<const float4 *>(&s[pass_swz32(2 * (threadIdx.x + u * kPassThreads))]);
}

// ── host side ────────────────────────────────────────────────────────────────

// The gate on k' = max(3, k) tile positions: positions (ascending, member bit b
// at pos[b]) and the matrix, padded with the identity on spare positions.
struct PlacedGate {
  uint32_t k = 0;
  uint32_t pos[4] = {0};
  const double *m = nullptr;   // interleaved, 2^k x 2^k: the gate's own, or `padded`
  std::vector<double> padded;
};

PlacedGate place_gate(const GateData &g, const std::vector<uint32_t> &tile_qubits) {
  PlacedGate p;
  auto position = [&](uint32_t q) {
    return (uint32_t)(std::lower_bound(tile_qubits.begin(), tile_qubits.end(), q) - tile_qubits.begin());
  };
  uint32_t pos[4] = {0}, used = 0;
  for (uint32_t b = 0; b < g.k; ++b) used |= 1u << (pos[b] = position(g.qubits[b]));
  for (uint32_t c = (uint32_t)tile_qubits.size(); __builtin_popcount(used) < 3 && c-- > 0;) used |= 1u << c;
  for (uint32_t c = 0; c < tile_qubits.size(); ++c)
    if ((used >> c) & 1) p.pos[p.k++] = c;
  if (p.k == g.k) {
    p.m = g.m64.data();
    return p;
  }
  const uint32_t D = 1u << p.k;
  uint32_t gate_bit[4] = {0}, gate_mask = 0;  // bit of the padded index holding gate bit b
  for (uint32_t b = 0; b < g.k; ++b) {
    gate_bit[b] = (uint32_t)__builtin_popcount(used & ((1u << pos[b]) - 1));
    gate_mask |= 1u << gate_bit[b];
  }
  p.padded.assign(2 * D * D, 0.0);
  for (uint32_t r = 0; r < D; ++r)
    for (uint32_t c = 0; c < D; ++c) {
      if ((r ^ c) & ~gate_mask) continue;
      uint32_t gr = 0, gc = 0;
      for (uint32_t b = 0; b < g.k; ++b) {
        gr |= ((r >> gate_bit[b]) & 1) << b;
        gc |= ((c >> gate_bit[b]) & 1) << b;
      }
      const size_t src = 2 * (((size_t)gr << g.k) + gc), dst = 2 * ((size_t)r * D + c);
      p.padded[dst] = g.m64[src];
      p.padded[dst + 1] = g.m64[src + 1];
    }
  p.m = p.padded.data();
  return p;
}

// How lanes walk the tile for one gate, as orders of its targets and of the
// other positions.  Tile bit p feeds bank-group bit p % 3, so a wavefront's
// three lane bits are conflict-free when their positions differ mod 3: members
// 0, 1 and group bit 0 on loads, group bits 1, 2 and row bit 0 on stores.
struct LaneOrder {
  uint8_t member[4], row[4];      // gate bit (index into pos) by member / row bit
  uint8_t group[kPassMaxTile];    // tile position by group bit
};

LaneOrder lane_order(const PlacedGate &p, uint32_t tb) {
  uint32_t rest[kPassMaxTile], n_rest = 0, taken = 0;
  for (uint32_t b = 0; b < p.k; ++b) taken |= 1u << p.pos[b];
  for (uint32_t c = 0; c < tb; ++c)
    if (!((taken >> c) & 1)) rest[n_rest++] = c;
  auto distinct = [](uint32_t x, uint32_t y, uint32_t z) {
    return (uint32_t)__builtin_popcount((1u << (x % 3)) | (1u << (y % 3)) | (1u << (z % 3)));
  };
  // the load triple, then the store triple from what is left; taking each best in
  // turn is enough: a tile has several free positions of every class
  uint32_t best = 0, ma = 0, mb = 1, ga = 0;
  for (uint32_t a = 0; a < p.k && best < 3; ++a)
    for (uint32_t b = a + 1; b < p.k && best < 3; ++b)
      for (uint32_t x = 0; x < n_rest && best < 3; ++x) {
        const uint32_t d = distinct(p.pos[a], p.pos[b], rest[x]);
        if (d > best) best = d, ma = a, mb = b, ga = x;
      }
  uint32_t gb = n_rest, gc = n_rest, ra = 0;
  best = 0;
  for (uint32_t y = 0; y < n_rest && best < 3; ++y)
    for (uint32_t z = y + 1; z < n_rest && best < 3; ++z) {
      if (y == ga || z == ga) continue;
      for (uint32_t r = 0; r < p.k && best < 3; ++r) {
        const uint32_t d = distinct(rest[y], rest[z], p.pos[r]);
        if (d > best) best = d, gb = y, gc = z, ra = r;
      }
    }
  LaneOrder o{};
  uint32_t at = 2;
  o.member[0] = (uint8_t)ma;
  o.member[1] = (uint8_t)mb;
  for (uint32_t b = 0; b < p.k; ++b)
    if (b != ma && b != mb) o.member[at++] = (uint8_t)b;
  at = 1;
  o.row[0] = (uint8_t)ra;
  for (uint32_t b = 0; b < p.k; ++b)
    if (b != ra) o.row[at++] = (uint8_t)b;
  at = 3;
  o.group[0] = (uint8_t)rest[ga];
  o.group[1] = (uint8_t)rest[gb];
  o.group[2] = (uint8_t)rest[gc];
  for (uint32_t c = 0; c < n_rest; ++c)
    if (c != ga && c != gb && c != gc) o.group[at++] = (uint8_t)rest[c];
  return o;
}

// Appends a gate's A fragments to the pool (lane l holds row l / 4 and column
// l % 4 of an 8 x 4 block) and fills its launch arguments.
void pack_gate(const PlacedGate &p, uint32_t tb, std::vector<double> &pool, PassGateArgs &out) {
  const LaneOrder o = lane_order(p, tb);
  const uint32_t D = 1u << p.k;
  uint32_t row_of[16], col_of[16];
  for (uint32_t i = 0; i < D; ++i) {
    row_of[i] = col_of[i] = 0;
    for (uint32_t b = 0; b < p.k; ++b)
      if ((i >> b) & 1) {
        row_of[i] |= 1u << o.row[b];
        col_of[i] |= 1u << o.member[b];
      }
  }
  std::memset(&out, 0, sizeof(out));
  out.mat = (uint32_t)pool.size();
  out.k = (uint16_t)p.k;
  const uint32_t products = p.k == 4 ? 3 : 2, row_blocks = D / 8, k_steps = D / 4;
  pool.resize(pool.size() + (size_t)products * D * D);
  double *to = pool.data() + out.mat;
  for (uint32_t prod = 0; prod < products; ++prod)
    for (uint32_t rb = 0; rb < row_blocks; ++rb)
      for (uint32_t ks = 0; ks < k_steps; ++ks)
        for (uint32_t lane = 0; lane < 32; ++lane) {
          const double *e = &p.m[2 * ((size_t)row_of[8 * rb + lane / 4] * D + col_of[4 * ks + lane % 4])];
          *to++ = prod == 0 ? e[0] : p.k == 3 ? e[1] : prod == 1 ? e[1] - e[0] : e[0] + e[1];
        }
  auto at = [](uint32_t position) { return (uint16_t)pass_swz(1u << position); };
  for (uint32_t b = 0; b < 2; ++b) out.ld_lane[b] = at(p.pos[o.member[b]]);
  for (uint32_t b = 0; b < 3; ++b) out.ld_lane[2 + b] = at(o.group[b]);
  for (uint32_t b = 2; b < p.k; ++b) out.ld_k[b - 2] = at(p.pos[o.member[b]]);
  for (uint32_t b = 0; b < 2; ++b) out.st_lane[b] = at(o.group[1 + b]);
  for (uint32_t b = 0; b < 3; ++b) out.st_lane[2 + b] = at(p.pos[o.row[b]]);
  if (p.k == 4) out.st_row = at(p.pos[o.row[3]]);
  out.st_col = at(o.group[0]);
  for (uint32_t b = 3; b < tb - p.k; ++b) out.blk[b - 3] = at(o.group[b]);
}

// A complex64 gate: its columns in row pairs appended to the pool, and the walk of
// the tile.  A half-warp's 16 eight-byte accesses are conflict-free when one lane
// bit is tile bit 0 and three others differ mod 3 as bits of the 16-byte unit's
// index; when bit 0 is a target they take two wavefronts.
void pack_gate32(const PlacedGate &p, uint32_t tb, std::vector<float> &pool, PassGateArgs32 &out) {
  std::memset(&out, 0, sizeof(out));
  out.mat = (uint32_t)pool.size();
  out.k = (uint16_t)p.k;
  uint32_t order[kPass32MaxTile], n_order = 0, used = 0;
  for (uint32_t b = 0; b < p.k; ++b) used |= 1u << p.pos[b];
  auto take = [&](uint32_t c) {
    order[n_order++] = c;
    used |= 1u << c;
  };
  if (!(used & 1)) take(0);
  for (uint32_t cls = 0; cls < 3; ++cls)
    for (uint32_t c = 1 + cls; c < tb; c += 3)
      if (!((used >> c) & 1)) {
        take(c);
        break;
      }
  for (uint32_t c = 0; c < tb; ++c)
    if (!((used >> c) & 1)) take(c);
  auto at = [](uint32_t position) { return (uint16_t)pass_swz32(1u << position); };
  for (uint32_t b = 0; b < n_order; ++b) out.group[b] = at(order[b]);
  for (uint32_t b = 0; b < p.k; ++b) out.member[b] = at(p.pos[b]);
  const uint32_t D = 1u << p.k;
  pool.resize(pool.size() + 3 * (size_t)D * D);
  for (uint32_t r = 0; r < D; ++r)
    for (uint32_t c = 0; c < D; ++c) {
      const double re = p.m[2 * (r * D + c)], im = p.m[2 * (r * D + c) + 1];
      float *to = &pool[out.mat + 6 * (c * (D / 2) + r / 2) + (r & 1)];
      to[0] = (float)re;
      to[2] = (float)(p.k == 4 ? im - re : im);
      to[4] = (float)(p.k == 4 ? re + im : -im);
    }
}

// Device buffers of plans.  A plan's buffer may still be read by launches in
// flight when its program is destroyed, so it comes back with the events recorded
// behind those launches and is handed out again (or freed) only once they have
// completed.  At most kPoolBytes wait here; a buffer beyond that is freed, which
// waits for the device.
constexpr size_t kPoolBytes = size_t(64) << 20;

struct PoolBuffer {
  int device = 0;
  char *ptr = nullptr;
  size_t bytes = 0;
  std::vector<cudaEvent_t> events;
};

struct BufferPool {
  std::mutex mu;
  std::vector<PoolBuffer> idle;
  size_t total = 0;
};

BufferPool &buffer_pool() {
  static BufferPool *p = new BufferPool;  // outlives programs destroyed at exit
  return *p;
}

bool settled(PoolBuffer &b) {
  while (!b.events.empty()) {
    if (cudaEventQuery(b.events.back()) == cudaErrorNotReady) return false;
    cudaEventDestroy(b.events.back());
    b.events.pop_back();
  }
  return true;
}

bool take_buffer(size_t bytes, PoolBuffer &out, std::string &err) {
  size_t cap = size_t(64) << 10;
  while (cap < bytes) cap <<= 1;
  int dev = 0;
  if (!cuda_ok(cudaGetDevice(&dev), "cudaGetDevice", err)) return false;
  {
    BufferPool &p = buffer_pool();
    std::lock_guard<std::mutex> lock(p.mu);
    for (size_t i = 0; i < p.idle.size(); ++i)
      if (p.idle[i].device == dev && p.idle[i].bytes == cap && settled(p.idle[i])) {
        out = p.idle[i];
        p.total -= cap;
        p.idle.erase(p.idle.begin() + (std::ptrdiff_t)i);
        return true;
      }
  }
  out = PoolBuffer{};
  out.device = dev;
  out.bytes = cap;
  return cuda_ok(cudaMalloc((void **)&out.ptr, cap), "cudaMalloc (gate pass matrices)", err);
}

void give_buffer(PoolBuffer &b) {
  if (!b.ptr) return;
  {
    BufferPool &p = buffer_pool();
    std::lock_guard<std::mutex> lock(p.mu);
    if (p.total + b.bytes <= kPoolBytes) {
      p.total += b.bytes;
      p.idle.push_back(std::move(b));
      b = PoolBuffer{};
      return;
    }
  }
  cudaFree(b.ptr);  // waits for the device
  for (cudaEvent_t e : b.events) cudaEventDestroy(e);
  b = PoolBuffer{};
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

// Allocating and copying on a private stream is safe while another thread
// captures; say so, or that thread's capture would refuse it.
struct RelaxedCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

}  // namespace

struct PassPlan {
  std::vector<Pass> passes;
  std::vector<PassArgs> args;   // one per merged pass (complex128)
  std::vector<PassArgs32> args32;  // the same in complex64
  std::vector<int> arg_of;      // pass -> its entry of args, -1 for a single gate
  std::vector<double> pool;     // matrices of every merged gate, as its kernel reads them
  std::vector<float> pool32;    // the same in complex64
  PoolBuffer buf;
  std::vector<cudaEvent_t> events;  // behind launches that read the buffer
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
// whose kernel nothing chose from outside.
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
  if (n < least || g.k > 4 || g.d_tc || g.d_sparse || gate_choice_forced(g)) return p;
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
      for (uint32_t i : x.gates) scalars += gates[i].k == 4 ? 3 * 256 : 3 * 64;
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
      for (uint32_t i = 0; i < a.n_gates; ++i)
        pack_gate(place_gate(gates[x.gates[i]], qubits), tb, p->pool, a.g[i]);
    } else {
      p->args32.emplace_back();
      PassArgs32 &a = p->args32.back();
      std::memset(&a, 0, sizeof(a));
      a.tb = tb;
      a.n_gates = (uint32_t)x.gates.size();
      for (uint32_t j = 0; j < tb; ++j) a.stride[j] = 1ull << qubits[j];
      for (uint32_t i = 0; i < a.n_gates; ++i)
        pack_gate32(place_gate(gates[x.gates[i]], qubits), tb, p->pool32, a.g[i]);
    }
    p->arg_of.push_back(next++);
  }
  return p.release();
}

void free_pass_plan(PassPlan *p) {
  if (!p) return;
  p->buf.events = std::move(p->events);
  give_buffer(p->buf);
  delete p;
}

bool upload_pass_plan(PassPlan &p, std::string &err) {
  const size_t bytes = p.pool.size() * sizeof(double) + p.pool32.size() * sizeof(float);
  if (p.buf.ptr || !bytes) return true;
  const void *src = p.pool.empty() ? (const void *)p.pool32.data() : (const void *)p.pool.data();
  RelaxedCapture relaxed;
  static std::once_flag once;
  static cudaError_t attr_rc = cudaSuccess;
  std::call_once(once, [] {
    attr_rc = cudaFuncSetAttribute(k_gate_pass, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)(sizeof(double2) << kPassMaxTile));
    if (attr_rc == cudaSuccess)
      attr_rc = cudaFuncSetAttribute(k_gate_pass32, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)(2 * kPass32MatBytes + (sizeof(float2) << kPass32MaxTile)));
  });
  if (!cuda_ok(attr_rc, "cudaFuncSetAttribute(gate pass kernel)", err)) return false;
  PoolBuffer b;
  if (!take_buffer(bytes, b, err)) return false;
  if (!upload_now(b.ptr, src, bytes, err)) {
    give_buffer(b);
    return false;
  }
  p.buf = std::move(b);
  return true;
}

bool launch_pass_plan(PassPlan &p, const std::vector<GateData> &gates, void *sv, uint32_t n,
                      cudaStream_t s, std::string &err) {
  for (size_t i = 0; i < p.passes.size(); ++i) {
    if (p.arg_of[i] < 0) {
      if (!launch_gate(gates[p.passes[i].gates[0]], sv, n, s, err)) return false;
      continue;
    }
    const uint32_t tb = p.args.empty() ? p.args32[p.arg_of[i]].tb : p.args[p.arg_of[i]].tb;
    const uint64_t tiles = 1ull << (n - tb);
    if (tiles > 0x7fffffffull) {
      err = "statevector too large for the gate pass kernel grid";
      return false;
    }
    if (p.args.empty())
      k_gate_pass32<<<(unsigned)tiles, kPassThreads, 2 * kPass32MatBytes + (sizeof(float2) << tb), s>>>(
          static_cast<float2 *>(sv), reinterpret_cast<const float *>(p.buf.ptr), p.args32[p.arg_of[i]]);
    else
      k_gate_pass<<<(unsigned)tiles, kPassThreads, sizeof(double2) << tb, s>>>(
          static_cast<double2 *>(sv), reinterpret_cast<const double *>(p.buf.ptr), p.args[p.arg_of[i]]);
    if (!cuda_ok(cudaGetLastError(), "gate pass kernel launch", err)) return false;
  }
  return true;
}

bool mark_pass_plan(PassPlan &p, cudaStream_t s, std::string &err) {
  if (!p.buf.ptr) return true;
  RelaxedCapture relaxed;
  // an event that has completed is recorded again, so the list is as long as the
  // most runs ever in flight at once
  cudaEvent_t ev = nullptr;
  for (size_t i = 0; i < p.events.size() && i < 8 && !ev; ++i)
    if (cudaEventQuery(p.events[i]) == cudaSuccess) ev = p.events[i];
  if (!ev) {
    if (!cuda_ok(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming), "cudaEventCreate", err)) return false;
    p.events.push_back(ev);
  }
  return cuda_ok(cudaEventRecord(ev, s), "cudaEventRecord (gate pass)", err);
}

}  // namespace cb2
