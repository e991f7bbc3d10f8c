// Gates applied to a tile of amplitudes in shared memory: device code shared by the
// merged passes (gate_pass.cu) and the circuit batch (circuit_batch.cu), and the
// host code that lays a gate out for it.
//
// complex128: a gate is a small GEMM on the FP64 tensor pipe (mma.sync m8n8k4).
// The matrix is A, its fragments in registers for the whole gate; eight gather
// groups are the N columns of B.  complex64: packed FP32 FMAs.
//
// Which tile bits the lanes walk is free: members (K order), rows and groups may
// be taken in any order.  The host picks them so that the lanes of a shared-memory
// wavefront fall into different bank groups under the tile's XOR swizzle (bank
// group = XOR of the 3-bit fields of the index in 16-byte units).
#pragma once

#include "internal.hpp"

#include <algorithm>
#include <cstring>
#include <vector>

namespace cb2 {

namespace {

constexpr uint32_t kTileMax64 = 13, kTileMax32 = 14;  // bits of the largest tiles
constexpr uint32_t kTileMin64 = 7;  // a 4-qubit gate and the 8 groups of a fragment

// Sparse gates (k = 5..7, few nonzeros a row): a lane owns 2^k / 32 rows of every
// group its warp takes.
constexpr uint32_t kSparseMost = 8;  // rows times nonzeros a lane holds

struct SparseGateArgs {
  uint16_t most;      // entries a row is given (1, 2 or 4)
  uint16_t full;      // every row has that many
  uint16_t group[9];  // group bits
};

// One gate of a pass.  Index contributions are swizzled tile offsets; XOR of the
// contributions of an index's set bits is its place in shared memory.
// k = 1, 2: ld_k holds the member bits, ld_lane (4 of it for k = 2) and blk the group
// bits; the st_ fields are unused.
struct PassGateArgs {
  uint32_t mat;          // first double of its fragments in the pool
  uint16_t k;            // 1..4; 5..7 for a sparse gate
  uint16_t ld_lane[5];   // load: lane bits 0, 1 -> member bits 0, 1; 2..4 -> group bits 0..2
  uint16_t ld_k[2];      // load: member bits 2, 3 (the k steps)
  uint16_t st_lane[5];   // store: lane bits 0, 1 -> group bits 1, 2; 2..4 -> row bits 0..2
  uint16_t st_row;       // store: row bit 3 (k = 4)
  uint16_t st_col;       // store: group bit 0 (the fragment's register index)
  uint16_t blk[kTileMax64 - 6];  // group bits 3, 4, ...
  SparseGateArgs sp;     // k >= 5
};

__host__ __device__ inline uint32_t pass_swz(uint32_t i) {
  return i ^ (((i >> 3) ^ (i >> 6) ^ (i >> 9) ^ (i >> 12)) & 7u);
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

template <int W> constexpr int log2_warps() { return W == 16 ? 4 : W == 8 ? 3 : 2; }

// Group bits 3.. of block warp + W * round: the warp's share once a gate, then the
// round's.
template <int W>
__device__ __forceinline__ uint32_t warp_bits(const PassGateArgs &g, int warp) {
  static_assert(W == 1 << log2_warps<W>(), "a power of two of warps");
  uint32_t x = 0;
#pragma unroll
  for (int b = 0; b < log2_warps<W>(); ++b)
    if ((warp >> b) & 1) x ^= g.blk[b];
  return x;
}

template <int W>
__device__ __forceinline__ uint32_t round_bits(const PassGateArgs &g, uint32_t round) {
  uint32_t x = 0;
#pragma unroll
  for (int b = log2_warps<W>(); b < (int)kTileMax64 - 6; ++b)
    if ((round >> (b - log2_warps<W>())) & 1) x ^= g.blk[b];
  return x;
}

// 4-qubit gate, three real products: S1 += c (a + b), S2 += (d - c) a,
// S3 += (c + d) b, Re = S1 - S3, Im = S1 + S2.  (Accumulating Re and Im on top of
// S1 saves their eight adds a block, which share the pipe, and 5% of the time at 30
// qubits, but moves the state 10% further from its 64-bit value: not done.)
// `m`: the gate's fragments, in global or shared memory.
template <int W>
__device__ __forceinline__ void pass_gate4(double2 *s, const double *mat, const PassGateArgs &g, uint32_t n_blk, int warp, int lane) {
  double a[3][2][4];
  const double *m = mat + lane;
#pragma unroll
  for (int p = 0; p < 3; ++p)
#pragma unroll
    for (int rb = 0; rb < 2; ++rb)
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) a[p][rb][ks] = m[32 * ((p * 2 + rb) * 4 + ks)];
  const uint32_t ld = lane_bits(g.ld_lane, lane), st = lane_bits(g.st_lane, lane);
  const uint32_t wb = warp_bits<W>(g, warp);
  for (uint32_t round = 0; round * W + warp < n_blk; ++round) {
    const uint32_t bx = wb ^ round_bits<W>(g, round);
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

// The same with four real products (Re = C a - D b, Im = D a + C b), for callers
// whose results have always been formed that way.
template <int W>
__device__ __forceinline__ void pass_gate4_full(double2 *s, const double *mat, const PassGateArgs &g,
                                                uint32_t n_blk, int warp, int lane) {
  double c[2][4], d[2][4];
  const double *m = mat + lane;
#pragma unroll
  for (int rb = 0; rb < 2; ++rb)
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      c[rb][ks] = m[32 * (rb * 4 + ks)];
      d[rb][ks] = m[32 * (8 + rb * 4 + ks)];
    }
  const uint32_t ld = lane_bits(g.ld_lane, lane), st = lane_bits(g.st_lane, lane);
  const uint32_t wb = warp_bits<W>(g, warp);
  for (uint32_t round = 0; round * W + warp < n_blk; ++round) {
    const uint32_t bx = wb ^ round_bits<W>(g, round);
    double2 x[4];
#pragma unroll
    for (int ks = 0; ks < 4; ++ks)
      x[ks] = s[bx ^ ld ^ (ks & 1 ? g.ld_k[0] : 0) ^ (ks & 2 ? g.ld_k[1] : 0)];
    double re[2][2] = {}, im[2][2] = {};
#pragma unroll
    for (int ks = 0; ks < 4; ++ks)
#pragma unroll
      for (int rb = 0; rb < 2; ++rb) {
        dmma(re[rb], c[rb][ks], x[ks].x);
        dmma(im[rb], c[rb][ks], x[ks].y);
        dmma(re[rb], -d[rb][ks], x[ks].y);
        dmma(im[rb], d[rb][ks], x[ks].x);
      }
#pragma unroll
    for (int rb = 0; rb < 2; ++rb)
#pragma unroll
      for (int i = 0; i < 2; ++i)
        s[bx ^ st ^ (rb ? g.st_row : 0) ^ (i ? g.st_col : 0)] = make_double2(re[rb][i], im[rb][i]);
  }
}

// 3-qubit gate, four real products: Re = C a - D b, Im = D a + C b.  U group
// blocks at once give the tensor pipe independent accumulators.
template <int W, int U>
__device__ __forceinline__ void pass_gate3_blocks(double2 *s, const double (&c)[2], const double (&d)[2],
                                                  const PassGateArgs &g, uint32_t ld, uint32_t st,
                                                  uint32_t wb, uint32_t round) {
  uint32_t bx[U];
  double2 x[U][2];
  double re[U][2] = {}, im[U][2] = {};
#pragma unroll
  for (int u = 0; u < U; ++u) {
    bx[u] = wb ^ round_bits<W>(g, round + u);
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

template <int W>
__device__ __forceinline__ void pass_gate3(double2 *s, const double *mat, const PassGateArgs &g, uint32_t n_blk, int warp, int lane) {
  const double *m = mat + lane;
  const double c[2] = {m[0], m[32]}, d[2] = {m[64], m[96]};
  const uint32_t ld = lane_bits(g.ld_lane, lane), st = lane_bits(g.st_lane, lane);
  const uint32_t wb = warp_bits<W>(g, warp);
  uint32_t round = 0;
  for (; (round + 3) * W + warp < n_blk; round += 4)
    pass_gate3_blocks<W, 4>(s, c, d, g, ld, st, wb, round);
  for (; round * W + warp < n_blk; ++round) pass_gate3_blocks<W, 1>(s, c, d, g, ld, st, wb, round);
}

// 1- and 2-qubit gates: a lane a gather group, or half the rows of one (2 qubits: two
// lanes of a warp read the same amplitudes, and hold half a matrix each), the fma
// sequence of the one-gate kernels.  (Padded with the identity to the 3-qubit form they
// took twice the arithmetic, and its zeros spread an infinity to amplitudes the gate
// leaves alone.)  U rounds at once keep loads in flight.
template <int W, int K, int U>
__device__ __forceinline__ void pass_small_rounds(double2 *s, const double2 (&m)[K == 1 ? 4 : 8],
                                                  const PassGateArgs &g, uint32_t lb, uint32_t top,
                                                  uint32_t round) {
  constexpr int D = 1 << K, R = 2;  // rows a lane
  uint32_t off[D], bx[U];
  double2 x[U][D];
#pragma unroll
  for (int a = 0; a < D; ++a) off[a] = (a & 1 ? g.ld_k[0] : 0) ^ (a & 2 ? g.ld_k[1] : 0);
#pragma unroll
  for (int u = 0; u < U; ++u) {
    bx[u] = lb ^ round_bits<W>(g, round + u);
#pragma unroll
    for (int a = 0; a < D; ++a) x[u][a] = s[bx[u] ^ off[a]];
  }
  if (K == 2) __syncwarp();  // the partner has read these groups
#pragma unroll
  for (int u = 0; u < U; ++u)
#pragma unroll
    for (int r = 0; r < R; ++r) {
      double re = 0.0, im = 0.0;
#pragma unroll
      for (int c = 0; c < D; ++c) {
        const double2 e = m[r * D + c];
        re = fma(e.x, x[u][c].x, re);
        re = fma(-e.y, x[u][c].y, re);
        im = fma(e.x, x[u][c].y, im);
        im = fma(e.y, x[u][c].x, im);
      }
      s[bx[u] ^ top ^ off[r]] = make_double2(re, im);
    }
}

// n_blk: blocks of 32 groups (k = 1) or 16 (k = 2).
template <int W, int K, int U>
__device__ __forceinline__ void pass_small(double2 *s, const double *mat, const PassGateArgs &g, uint32_t n_blk, int warp, int lane) {
  constexpr int E = K == 1 ? 4 : 8;
  const bool half = K == 2 && lane >= 16;
  double2 m[E];
#pragma unroll
  for (int e = 0; e < E; ++e) m[e] = reinterpret_cast<const double2 *>(mat)[e + (half ? E : 0)];
  const uint32_t lb = lane_bits(g.ld_lane, lane) ^ warp_bits<W>(g, warp), top = half ? g.ld_k[1] : 0;
  uint32_t round = 0;
  for (; (round + U - 1) * W + warp < n_blk; round += U) pass_small_rounds<W, K, U>(s, m, g, lb, top, round);
  if (U > 1)
    for (; round * W + warp < n_blk; ++round) pass_small_rounds<W, K, 1>(s, m, g, lb, top, round);
}

constexpr uint32_t kPass32MatBytes = 3 * 256 * sizeof(float);

struct PassGateArgs32 {
  uint32_t mat;           // first float of its columns in the pool
  uint16_t k;             // 1..4; 5..7 for a sparse gate
  uint16_t member[4];     // gate bits
  uint16_t group[kTileMax32 - 1];  // group bits (a 1-qubit gate has the most)
  SparseGateArgs sp;      // k >= 5
};

// 16-byte units of two amplitudes; bank group = XOR of the unit's 3-bit fields.
__host__ __device__ inline uint32_t pass_swz32(uint32_t i) {
  const uint32_t u = i >> 1;
  return ((u ^ (((u >> 3) ^ (u >> 6) ^ (u >> 9) ^ (u >> 12)) & 7u)) << 1) | (i & 1u);
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
// of the matrix holds six floats a row pair: for three products (M3) c_0, c_1,
// (d-c)_0, (d-c)_1, (c+d)_0, (c+d)_1; for four re_0, re_1, im_0, im_1, -im_0, -im_1.  A thread that is not `live` takes part in the barrier only.
template <int K, int H, int U, bool M3>
__device__ __forceinline__ void pass_groups32(float2 *s, const float *mat, const PassGateArgs32 &g,
                                              const uint32_t (&gb)[U], uint32_t half, bool live) {
  constexpr int D = 1 << K, P = D / 2 / H, S = M3 ? 3 : 2;  // row pairs, sums a row pair
  const float2 *m = reinterpret_cast<const float2 *>(mat) + half * (3 * P);
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
    constexpr int Q = P < 2 ? 1 : 2;  // row pairs at once: two are three 16-byte loads
#pragma unroll
    for (int h = 0; h < P / Q; ++h) {
      const float2 *mc = m + 3 * (c * (D / 2) + Q * h);
      float2 e[Q][3];
      if constexpr (Q == 2) {
        const float4 *m4 = reinterpret_cast<const float4 *>(mc);
        const float4 m0 = m4[0], m1 = m4[1], m2 = m4[2];
        e[0][0] = make_float2(m0.x, m0.y), e[0][1] = make_float2(m0.z, m0.w), e[0][2] = make_float2(m1.x, m1.y);
        e[1][0] = make_float2(m1.z, m1.w), e[1][1] = make_float2(m2.x, m2.y), e[1][2] = make_float2(m2.z, m2.w);
      } else {  // a 1-qubit gate
        e[0][0] = mc[0], e[0][1] = mc[1], e[0][2] = mc[2];
      }
#pragma unroll
      for (int q = 0; q < Q; ++q)
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int p = Q * h + q;
          if constexpr (M3) {
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
      if constexpr (M3) {
        const float2 s3 = acc[u][S - 1][p];
        im = __fadd2_rn(re, im);
        re = __fadd2_rn(re, make_float2(-s3.x, -s3.y));
      }
      s[gb[u] ^ top ^ member_bits32<K>(g, 2 * p)] = make_float2(re.x, im.x);
      s[gb[u] ^ top ^ member_bits32<K>(g, 2 * p + 1)] = make_float2(re.y, im.y);
    }
}

// A gate on the whole tile; H threads share a group, lane bit 4 telling them apart.
template <int NT, int K, int H, int U, bool M3>
__device__ __forceinline__ void pass_gate32(float2 *s, const float *mat, const PassGateArgs32 &g,
                                            uint32_t tb) {
  constexpr uint32_t GT = NT / H;  // groups the CTA takes at once
  constexpr int TB = GT == 512 ? 9 : GT == 256 ? 8 : GT == 128 ? 7 : 6;
  static_assert(GT == 1u << TB, "a power of two of groups");
  const uint32_t half = H == 2 ? (threadIdx.x >> 4) & 1 : 0;
  const uint32_t gt = H == 2 ? (threadIdx.x & 15) | (threadIdx.x >> 5) << 4 : threadIdx.x;
  constexpr int LAST = (int)kTileMax32 - K;  // group bits of the largest tile
  auto offset = [&](uint32_t group, int from, int to) {  // group bits from .. to - 1
    uint32_t o = 0;
#pragma unroll
    for (int b = 0; b < LAST; ++b)
      if (b >= from && b < to && ((group >> b) & 1)) o ^= g.group[b];
    return o;
  };
  constexpr int LU = U == 4 ? 2 : U == 2 ? 1 : 0;
  static_assert(U == 1 << LU, "a power of two of groups");
  const uint32_t groups = 1u << (tb - K), t = offset(gt, 0, TB);
  if (groups >= U * GT) {
    for (uint32_t it = 0; it < groups >> TB; it += U) {
      const uint32_t ib = t ^ offset(it << TB, TB + LU, LAST);
      uint32_t gb[U];
#pragma unroll
      for (int u = 0; u < U; ++u) gb[u] = ib ^ offset((uint32_t)u << TB, TB, TB + LU);
      pass_groups32<K, H, U, M3>(s, mat, g, gb, half, true);
    }
  } else {
    for (uint32_t it = 0; it * GT < groups; ++it) {
      const bool live = it * GT + gt < groups;
      const uint32_t gb[1] = {live ? t ^ offset(it << TB, TB, LAST) : 0};
      if (H > 1 || live) pass_groups32<K, H, 1, M3>(s, mat, g, gb, half, live);
    }
  }
}

// A sparse gate on a tile (either precision).  The entries of a lane's rows stay in
// registers for the whole gate: per group it reads their amplitudes, waits for the
// warp (the group is this warp's alone) and writes its rows.  An absent entry has
// the place kNoEntry.  The same fma sequence a row as the one-gate CSR kernels.
// A gate costs two shared-memory accesses an amplitude, so what counts is the
// instructions around them: with the group's place formed once for U groups
// instead of bit by bit for each, the 22-qubit QFT (CX form, complex128, 37 gates in
// 14 passes) takes 561 us, 904 before; one gate a pass 909.  26 qubits: 19.4 ->
// 10.8 ms in complex128, 11.3 -> 6.8 in complex64.
constexpr uint32_t kNoEntry = 0xffffffffu;

template <int ROWS, int M, int U, typename V>
__device__ __forceinline__ void sparse_groups(V *s, const V (&m)[ROWS][M], const uint32_t (&at)[ROWS][M],
                                              const uint32_t (&own)[ROWS], bool full,
                                              const uint32_t (&gb)[U]) {
  V out[U][ROWS];
#pragma unroll
  for (int u = 0; u < U; ++u)
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      if (full) {  // every row has its M entries
        V x = s[gb[u] ^ at[r][0]];
        out[u][r].x = fma(m[r][0].x, x.x, -m[r][0].y * x.y);
        out[u][r].y = fma(m[r][0].x, x.y, m[r][0].y * x.x);
#pragma unroll
        for (int j = 1; j < M; ++j) {
          x = s[gb[u] ^ at[r][j]];
          out[u][r].x = fma(m[r][j].x, x.x, fma(-m[r][j].y, x.y, out[u][r].x));
          out[u][r].y = fma(m[r][j].x, x.y, fma(m[r][j].y, x.x, out[u][r].y));
        }
      } else {
        out[u][r].x = out[u][r].y = 0;
#pragma unroll
        for (int j = 0; j < M; ++j)
          if (at[r][j] != kNoEntry) {
            const V x = s[gb[u] ^ at[r][j]];
            out[u][r].x = fma(m[r][j].x, x.x, fma(-m[r][j].y, x.y, out[u][r].x));
            out[u][r].y = fma(m[r][j].x, x.y, fma(m[r][j].y, x.x, out[u][r].y));
          }
      }
    }
  __syncwarp();
#pragma unroll
  for (int u = 0; u < U; ++u)
#pragma unroll
    for (int r = 0; r < ROWS; ++r) s[gb[u] ^ own[r]] = out[u][r];
}

template <int W, int ROWS, int M, typename V>
__device__ __forceinline__ void pass_sparse_rows(V *s, const V *__restrict__ vals, const SparseGateArgs &g,
                                                 uint32_t n_groups, int warp, int lane) {
  const uint32_t *places = reinterpret_cast<const uint32_t *>(vals + 32 * ROWS * M);
  V m[ROWS][M];
  uint32_t at[ROWS][M], own[ROWS];
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
#pragma unroll
    for (int j = 0; j < M; ++j) {
      m[r][j] = vals[32 * (r * M + j) + lane];
      at[r][j] = places[32 * (r * M + j) + lane];
    }
    own[r] = places[32 * (ROWS * M + r) + lane];
  }
  // group bits: the warp, then the U groups taken at once, then the rounds
  constexpr int LU = ROWS * M >= 8 ? 0 : ROWS * M >= 4 ? 1 : 2, U = 1 << LU;
  constexpr int LW = log2_warps<W>();
  uint32_t wb = 0;
#pragma unroll
  for (int b = 0; b < LW; ++b)
    if ((warp >> b) & 1) wb ^= g.group[b];
  if (n_groups >= (uint32_t)(U * W)) {
    for (uint32_t it = 0; it < n_groups / (U * W); ++it) {
      uint32_t ib = wb;
#pragma unroll
      for (int b = LW + LU; b < 9; ++b)
        if ((it >> (b - LW - LU)) & 1) ib ^= g.group[b];
      uint32_t gb[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        gb[u] = ib;
#pragma unroll
        for (int b = 0; b < LU; ++b)
          if ((u >> b) & 1) gb[u] ^= g.group[LW + b];
      }
      sparse_groups<ROWS, M, U>(s, m, at, own, g.full, gb);
    }
  } else {
    for (uint32_t group = warp; group < n_groups; group += W) {
      uint32_t gb[1] = {wb};
#pragma unroll
      for (int b = LW; b < 9; ++b)
        if ((group >> b) & 1) gb[0] ^= g.group[b];
      sparse_groups<ROWS, M, 1>(s, m, at, own, g.full, gb);
    }
  }
}

template <int W, typename V>
__device__ __forceinline__ void pass_sparse(V *s, const V *__restrict__ vals, uint32_t k,
                                            const SparseGateArgs &g, uint32_t tb, int warp, int lane) {
  const uint32_t n = 1u << (tb - k);
  if (k == 5) {
    if (g.most == 1) pass_sparse_rows<W, 1, 1>(s, vals, g, n, warp, lane);
    else pass_sparse_rows<W, 1, 4>(s, vals, g, n, warp, lane);
  } else if (k == 6) {
    if (g.most == 1) pass_sparse_rows<W, 2, 1>(s, vals, g, n, warp, lane);
    else pass_sparse_rows<W, 2, 4>(s, vals, g, n, warp, lane);
  } else {
    if (g.most == 1) pass_sparse_rows<W, 4, 1>(s, vals, g, n, warp, lane);
    else pass_sparse_rows<W, 4, 2>(s, vals, g, n, warp, lane);
  }
}

// Entries a row of a sparse gate is given in its tile form, 0 when it has too many
// nonzeros for one.
inline uint32_t sparse_most(const GateData &g) {
  const size_t most = gate_row_nnz_max(g);
  const uint32_t rows = 1u << (g.k - 5), cap = g.k == 7 ? 2 : 4;
  if (most > cap || rows * cap > kSparseMost) return 0;
  return most <= 1 ? 1 : cap;
}

// A sparse gate's entries appended to the pool (T: its scalars) and its walk; `swz`
// maps a tile index to its place.
template <typename T, typename S>
inline void pack_sparse(const GateData &g, const std::vector<uint32_t> &tile_qubits, S swz,
                        std::vector<T> &pool, uint32_t &mat, SparseGateArgs &out) {
  const uint32_t D = 1u << g.k, tb = (uint32_t)tile_qubits.size(), rows = D / 32;
  const uint32_t M = out.most = (uint16_t)sparse_most(g);
  uint32_t pos[kMaxGateQubits], taken = 0;
  for (uint32_t b = 0; b < g.k; ++b) {
    pos[b] = (uint32_t)(std::lower_bound(tile_qubits.begin(), tile_qubits.end(), g.qubits[b]) -
                        tile_qubits.begin());
    taken |= 1u << pos[b];
  }
  uint32_t at = 0;
  for (uint32_t c = 0; c < tb; ++c)
    if (!((taken >> c) & 1)) out.group[at++] = (uint16_t)swz(1u << c);
  while (pool.size() % 4) pool.push_back(T(0));  // 16-byte aligned
  mat = (uint32_t)pool.size();
  const size_t entries = 32 * (size_t)rows * M;
  pool.resize(pool.size() + 2 * entries + (entries + D) * sizeof(uint32_t) / sizeof(T));
  T *vals = pool.data() + mat;
  uint32_t *places = reinterpret_cast<uint32_t *>(vals + 2 * entries);
  for (size_t e = 0; e < entries; ++e) places[e] = kNoEntry;
  uint32_t member[1u << kMaxGateQubits];  // place of a member in its group
  for (uint32_t i = 0; i < D; ++i) {
    member[i] = 0;
    for (uint32_t b = 0; b < g.k; ++b)
      if ((i >> b) & 1) member[i] ^= swz(1u << pos[b]);
  }
  uint8_t cols[1u << kMaxGateQubits][4], n_cols[1u << kMaxGateQubits];
  out.full = 1;
  for (uint32_t r = 0; r < D; ++r) {
    n_cols[r] = 0;
    for (uint32_t c = 0; c < D; ++c)
      if (g.m64[2 * ((size_t)r * D + c)] != 0.0 || g.m64[2 * ((size_t)r * D + c) + 1] != 0.0)
        cols[r][n_cols[r]++] = (uint8_t)c;
    if (n_cols[r] != M) out.full = 0;
  }
  // Rows are dealt to lanes wavefront by wavefront (8 lanes of 16-byte amplitudes or
  // 16 of 8-byte ones), each time the row whose own place and inputs meet the fewest
  // taken banks: a permutation's rows and columns rarely suit the same plain order.
  constexpr uint32_t WF = 128 / (2 * sizeof(T));
  bool dealt[1u << kMaxGateQubits] = {};
  for (uint32_t first = 0; first < D; first += WF) {
    uint8_t used[1 + 4][16] = {};  // own place, then each entry's; by bank slot
    for (uint32_t i = first; i < first + WF; ++i) {
      uint32_t row = D, least = ~0u;
      for (uint32_t r = 0; r < D && least; ++r) {
        if (dealt[r]) continue;
        uint32_t clash = used[0][member[r] % WF];
        for (uint32_t j = 0; j < n_cols[r]; ++j) clash += used[1 + j][member[cols[r][j]] % WF];
        if (clash < least) least = clash, row = r;
      }
      dealt[row] = true;
      ++used[0][member[row] % WF];
      places[entries + i] = member[row];
      for (uint32_t j = 0; j < n_cols[row]; ++j) {
        const uint32_t c = cols[row][j];
        ++used[1 + j][member[c] % WF];
        const size_t e = 32 * ((size_t)(i / 32) * M + j) + i % 32, from = 2 * ((size_t)row * D + c);
        vals[2 * e] = (T)g.m64[from];
        vals[2 * e + 1] = (T)g.m64[from + 1];
        places[e] = member[c];
      }
    }
  }
}

// The gate's places in the tile (ascending, member bit b at pos[b]) and its matrix.
struct PlacedGate {
  uint32_t k = 0;
  uint32_t pos[4] = {0};
  const double *m = nullptr;   // interleaved, 2^k x 2^k
};

inline PlacedGate place_gate(const GateData &g, const std::vector<uint32_t> &tile_qubits) {
  PlacedGate p;
  p.k = g.k;
  p.m = g.m64.data();
  for (uint32_t b = 0; b < g.k; ++b)
    p.pos[b] = (uint32_t)(std::lower_bound(tile_qubits.begin(), tile_qubits.end(), g.qubits[b]) - tile_qubits.begin());
  return p;
}

// How lanes walk the tile for one gate, as orders of its targets and of the
// other positions.  Tile bit p feeds bank-group bit p % 3, so a wavefront's
// three lane bits are conflict-free when their positions differ mod 3: members
// 0, 1 and group bit 0 on loads, group bits 1, 2 and row bit 0 on stores.
struct LaneOrder {
  uint8_t member[4], row[4];      // gate bit (index into pos) by member / row bit
  uint8_t group[kTileMax64];    // tile position by group bit
};

inline LaneOrder lane_order(const PlacedGate &p, uint32_t tb) {
  uint32_t rest[kTileMax64], n_rest = 0, taken = 0;
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

// A 1- or 2-qubit gate: its matrix as it is, and group bits such that the 8 lanes of a
// wavefront fall into different bank groups (three lane bits that differ mod 3).
inline void pack_small(const PlacedGate &p, uint32_t tb, std::vector<double> &pool, PassGateArgs &out) {
  std::memset(&out, 0, sizeof(out));
  out.mat = (uint32_t)pool.size();
  out.k = (uint16_t)p.k;
  pool.insert(pool.end(), p.m, p.m + ((size_t)2 << (2 * p.k)));
  uint32_t order[kTileMax64], n_order = 0, used = 0;
  for (uint32_t b = 0; b < p.k; ++b) used |= 1u << p.pos[b];
  auto take = [&](uint32_t c) {
    order[n_order++] = c;
    used |= 1u << c;
  };
  for (uint32_t cls = 0; cls < 3; ++cls)
    for (uint32_t c = cls; c < tb; c += 3)
      if (!((used >> c) & 1)) {
        take(c);
        break;
      }
  for (uint32_t c = 0; c < tb; ++c)
    if (!((used >> c) & 1)) take(c);
  auto at = [](uint32_t position) { return (uint16_t)pass_swz(1u << position); };
  const uint32_t lanes = p.k == 1 ? 5 : 4;
  for (uint32_t b = 0; b < n_order; ++b) (b < lanes ? out.ld_lane[b] : out.blk[b - lanes]) = at(order[b]);
  for (uint32_t b = 0; b < p.k; ++b) out.ld_k[b] = at(p.pos[b]);
}

// Appends a gate's A fragments to the pool (lane l holds row l / 4 and column
// l % 4 of an 8 x 4 block) and fills its launch arguments.
// `three`: the three-product form (4-qubit gates).
inline void pack_gate(const PlacedGate &p, uint32_t tb, bool three, std::vector<double> &pool, PassGateArgs &out) {
  if (p.k < 3) return pack_small(p, tb, pool, out);
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
  const uint32_t products = three ? 3 : 2, row_blocks = D / 8, k_steps = D / 4;
  pool.resize(pool.size() + (size_t)products * D * D);
  double *to = pool.data() + out.mat;
  for (uint32_t prod = 0; prod < products; ++prod)
    for (uint32_t rb = 0; rb < row_blocks; ++rb)
      for (uint32_t ks = 0; ks < k_steps; ++ks)
        for (uint32_t lane = 0; lane < 32; ++lane) {
          const double *e = &p.m[2 * ((size_t)row_of[8 * rb + lane / 4] * D + col_of[4 * ks + lane % 4])];
          *to++ = prod == 0 ? e[0] : !three ? e[1] : prod == 1 ? e[1] - e[0] : e[0] + e[1];
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
inline void pack_gate32(const PlacedGate &p, uint32_t tb, bool three, std::vector<float> &pool,
                        PassGateArgs32 &out) {
  std::memset(&out, 0, sizeof(out));
  out.mat = (uint32_t)pool.size();
  out.k = (uint16_t)p.k;
  uint32_t order[kTileMax32], n_order = 0, used = 0;
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
      to[2] = (float)(three ? im - re : im);
      to[4] = (float)(three ? re + im : -im);
    }
}

}  // namespace

}  // namespace cb2
