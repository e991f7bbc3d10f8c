// Batched Monte-Carlo quantum-jump trajectories: programs, their upload and runs
// (the kernels' device side is trajectory.cuh).
#include "../../include/cast_b200.h"
#include "seg_plan.hpp"
#include "trajectory.cuh"

#include <algorithm>
#include <cmath>
#include <exception>
#include <map>
#include <mutex>
#include <vector>

namespace {

using cb2::cuda_ok;

template <int NT>
__global__ void __launch_bounds__(NT, 1)
    k_trajectories(const TOp *__restrict__ ops, uint32_t n_ops, const float2 *__restrict__ pool,
                   float2 *__restrict__ ws, uint32_t n, const TRun *__restrict__ run,
                   double *__restrict__ out_z, uint32_t *__restrict__ out_sample) {
  trajectories<NT, false>(ops, n_ops, pool, ws, n, run, out_z, out_sample, TSegs{}, nullptr);
}

constexpr uint32_t kTrajMagic = 0xCB2077A1u;

// Trajectories in flight when the program does not fix them: one per SM, unless
// the slices of one per SM overflow L2 while those of at least half as many
// still fit in 89% of it (17 qubits: 112 CTAs x 1 MB instead of 148, 1.8x the
// throughput); beyond that the passes stream from HBM either way.
unsigned auto_ctas(uint32_t n) {
  const unsigned sms = (unsigned)cb2::sm_count();
  int dev = 0, l2 = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, dev) != cudaSuccess || l2 <= 0) {
    cudaGetLastError();
    return sms;
  }
  const uint64_t slice = sizeof(float2) << n;
  const uint64_t fit = (uint64_t)l2 * 89 / 100 / slice;
  return fit >= sms || fit < sms / 2 ? sms : (unsigned)fit;
}

// No access-policy window: a persisting-L2 set-aside sized for the workspace
// gave the trajectories 4% at 16 qubits but, being a limit of the whole
// context, cut every later streaming gate pass of the process from 6.3 to
// 2.8 TB/s until it was set back to 0.
cudaError_t launch_trajectories(unsigned grid, unsigned threads, cudaStream_t s, const TOp *ops,
                                uint32_t n_ops, const float2 *pool, float2 *ws, uint32_t n,
                                const TRun *run, double *z, uint32_t *sample, TSegs segs) {
  if (threads != (unsigned)kTMinThreads) segs.segs = nullptr;  // segments need 128 registers a thread
  if (segs.segs) return cb2::launch_trajectory_segments(grid, s, ops, n_ops, pool, ws, n, run, z, sample, &segs);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = s;
  if (threads == 1024)
    return cudaLaunchKernelEx(&cfg, k_trajectories<1024>, ops, n_ops, pool, ws, n, run, z, sample);
  return cudaLaunchKernelEx(&cfg, k_trajectories<512>, ops, n_ops, pool, ws, n, run, z, sample);
}

// Device buffers of trajectory programs come from a process-wide cache keyed by
// (device, exact size).  cudaFree synchronises the whole device, and a serving
// loop creates and drops one program per noisy request while other requests
// run on other streams.  A dropped program's buffers are idle (cast_b200_traj_run
// returns only after its work completes), so they wait here for reuse, up to
// 8 GiB in all; beyond that they are freed.  The device of a returned buffer is
// read from the pointer itself, so a process that switches devices with
// cast_b200_set_device never receives another device's memory.
std::mutex g_buf_mu;
std::multimap<std::pair<int, size_t>, void *> g_buf_cache;
size_t g_buf_cached = 0;
constexpr size_t kBufCacheMax = 8ull << 30;

cudaError_t buf_alloc(void **p, size_t bytes) {
  int dev = 0;
  const cudaError_t rc = cudaGetDevice(&dev);
  if (rc != cudaSuccess) return rc;
  {
    std::lock_guard<std::mutex> lock(g_buf_mu);
    auto it = g_buf_cache.find({dev, bytes});
    if (it != g_buf_cache.end()) {
      *p = it->second;
      g_buf_cache.erase(it);
      g_buf_cached -= bytes;
      return cudaSuccess;
    }
  }
  return cudaMalloc(p, bytes);
}

void buf_free(void *p, size_t bytes) {
  if (!p) return;
  cudaPointerAttributes attr{};
  if (cudaPointerGetAttributes(&attr, p) == cudaSuccess && attr.type == cudaMemoryTypeDevice) {
    std::lock_guard<std::mutex> lock(g_buf_mu);
    if (g_buf_cached + bytes <= kBufCacheMax) {
      g_buf_cache.emplace(std::make_pair(attr.device, bytes), p);
      g_buf_cached += bytes;
      return;
    }
  }
  cudaFree(p);
}

struct TrajProgram {
  uint32_t magic = kTrajMagic;
  uint32_t n = 0;
  std::vector<TOp> ops;
  std::vector<float2> pool;
  bool dirty = true;
  TOp *d_ops = nullptr;
  float2 *d_pool = nullptr;
  float2 *d_ws = nullptr;
  size_t ws_ctas = 0;
  size_t ops_bytes = 0, pool_bytes = 0, ws_bytes = 0, z_bytes = 0, sample_bytes = 0;
  void *d_segs = nullptr;     // the segments' arrays, one buffer
  size_t segs_bytes = 0;
  TSegs segs{};
  double width = 0;           // mean qubits of the GATE ops
  TRun *d_run = nullptr;
  double *d_z = nullptr;
  uint32_t *d_sample = nullptr;
  size_t out_cap = 0;
  cudaGraphExec_t graph = nullptr;
  void *graph_stream = nullptr;
  unsigned graph_grid = 0;
  unsigned threads = 0;  // threads per CTA: 512, 1024, or 0 for the size's own
  unsigned max_ctas = 0; // CTAs (trajectories in flight), or 0 for auto_ctas(n)
  unsigned graph_threads = 0;
  std::mutex mu;

  ~TrajProgram() {
    if (graph) cudaGraphExecDestroy(graph);
    buf_free(d_ops, ops_bytes);
    buf_free(d_pool, pool_bytes);
    buf_free(d_ws, ws_bytes);
    buf_free(d_segs, segs_bytes);
    buf_free(d_run, sizeof(TRun));
    buf_free(d_z, z_bytes);
    buf_free(d_sample, sample_bytes);
  }

  uint32_t push_matrix(const cast_complex64_t *m, size_t entries) {
    const uint32_t off = (uint32_t)pool.size();
    for (size_t i = 0; i < entries; ++i) pool.push_back(make_float2((float)m[i].re, (float)m[i].im));
    return off;
  }

  void mark_stats() {
    for (auto &o : ops) o.stats = o.nerr = 0;
    for (size_t i = 0; i < ops.size(); ++i) {
      if (ops[i].type != T_GATE) continue;
      uint32_t e = 0;
      while (i + 1 + e < ops.size() && ops[i + 1 + e].type == T_ERR && e < (uint32_t)kTMinThreads) ++e;
      ops[i].nerr = e;
    }
    for (size_t i = 0; i < ops.size(); ++i) {
      if (ops[i].type != T_DAMP) continue;
      size_t j = i;
      while (j > 0 && ops[j - 1].type == T_ERR) --j;
      if (j > 0 && ops[j - 1].type == T_GATE) {
        ops[j - 1].stats = 1;
        ops[j - 1].smask = ops[i].mask;
        ops[j - 1].sgamma = ops[i].gamma;
      }
    }
  }

  // Plans the program's segments (seg_plan.cpp) and uploads them.
  bool build_segments(std::string &err) {
    std::vector<TSeg> sg;
    std::vector<TSegPass> ps;
    std::vector<cb2::PassGateArgs32> gs;
    std::vector<uint32_t> sites;
    std::vector<float> mats;
    uint32_t mat_cap = 0;
    const uint32_t tb_most = std::min(n, kSegMaxTile);
    std::vector<cb2::SegBlock> blocks;
    std::vector<uint32_t> at;  // block -> its op
    for (size_t i = 0; i < ops.size(); ++i) {
      if (ops[i].type == T_GATE) {
        cb2::SegBlock b;
        for (uint32_t j = 0; j < ops[i].k; ++j) b.qubits |= 1ull << ops[i].q[j];
        b.follows = i > 0 && (ops[i - 1].type == T_GATE || ops[i - 1].type == T_ERR);
        blocks.push_back(b);
        at.push_back((uint32_t)i);
      } else if (ops[i].type == T_ERR && !blocks.empty()) {
        blocks.back().quiet *= 1.0 - (double)ops[i].prob;
      }
    }
    width = cb2::mean_width(blocks);
    std::vector<cb2::Segment> plan;
    if (n >= kSegMinQubits) plan = cb2::plan_segments(blocks, n, tb_most, kSegLow);
    std::vector<uint32_t> starts(ops.size(), 0);
    for (const cb2::Segment &seg : plan) {
      std::vector<cb2::GateData> gates;
      TSeg g{};
      g.err0 = (uint32_t)sites.size();
      const uint32_t first_op = at[seg.first];
      uint32_t end = first_op;
      for (; end < ops.size() && (ops[end].type == T_ERR || gates.size() < seg.count); ++end) {
        if (ops[end].type == T_ERR) {
          sites.push_back(end);
          continue;
        }
        cb2::GateData x;
        x.k = ops[end].k;
        for (uint32_t b = 0; b < x.k; ++b) x.qubits[b] = ops[end].q[b];
        const size_t entries = size_t(1) << (2 * x.k);
        x.m64.reserve(2 * entries);
        for (size_t e = 0; e < entries; ++e) {
          x.m64.push_back(pool[ops[end].mat + e].x);
          x.m64.push_back(pool[ops[end].mat + e].y);
        }
        if (ops[end].stats) {
          g.stats = 1;
          g.smask = ops[end].smask;
          g.sgamma = ops[end].sgamma;
        }
        gates.push_back(std::move(x));
      }
      g.n_err = (uint32_t)sites.size() - g.err0;
      g.end_op = end;
      g.pass0 = (uint32_t)ps.size();
      g.n_passes = (uint32_t)seg.passes.size();
      for (const cb2::Pass &x : seg.passes) {
        uint64_t tile = x.tile ? x.tile : blocks[seg.first + x.gates[0]].qubits | ((1ull << std::min(n, kSegLow)) - 1);
        for (uint32_t b = 0; b < n && (uint32_t)__builtin_popcountll(tile) < tb_most; ++b) tile |= 1ull << b;
        std::vector<uint32_t> qubits;
        for (uint32_t q = 0; q < n; ++q)
          if ((tile >> q) & 1) qubits.push_back(q);
        TSegPass t{};
        t.tb = (uint32_t)qubits.size();
        t.n_gates = (uint32_t)x.gates.size();
        t.gate0 = (uint32_t)gs.size();
        t.mat = (uint32_t)mats.size();
        for (uint32_t j = 0; j < t.tb; ++j) t.stride[j] = 1u << qubits[j];
        for (const uint32_t j : x.gates) {
          cb2::PassGateArgs32 a;
          cb2::pack_gate32(cb2::place_gate(gates[j], qubits), t.tb, false, mats, a);
          gs.push_back(a);
        }
        t.mat_bytes = (uint32_t)((mats.size() - t.mat) * sizeof(float));
        mat_cap = std::max(mat_cap, t.mat_bytes);
        ps.push_back(t);
      }
      starts[first_op] = (uint32_t)sg.size() + 1;
      sg.push_back(g);
    }
    buf_free(d_segs, segs_bytes);
    d_segs = nullptr;
    segs_bytes = 0;
    segs = TSegs{};
    if (sg.empty()) return true;
    auto align = [](size_t x) { return (x + 255) & ~size_t(255); };
    const size_t at_p = align(sg.size() * sizeof(TSeg)), at_g = at_p + align(ps.size() * sizeof(TSegPass)),
                 at_s = at_g + align(gs.size() * sizeof(gs[0])), at_o = at_s + align(sites.size() * 4 + 4),
                 at_m = at_o + align(starts.size() * 4),
                 bytes = at_m + align(mats.size() * sizeof(float));
    std::vector<char> host(bytes, 0);
    std::memcpy(host.data(), sg.data(), sg.size() * sizeof(TSeg));
    std::memcpy(host.data() + at_p, ps.data(), ps.size() * sizeof(TSegPass));
    std::memcpy(host.data() + at_g, gs.data(), gs.size() * sizeof(gs[0]));
    if (!sites.empty()) std::memcpy(host.data() + at_s, sites.data(), sites.size() * 4);
    std::memcpy(host.data() + at_o, starts.data(), starts.size() * 4);
    std::memcpy(host.data() + at_m, mats.data(), mats.size() * sizeof(float));
    if (!cuda_ok(buf_alloc(&d_segs, bytes), "cudaMalloc (trajectory segments)", err)) return false;
    segs_bytes = bytes;
    if (!cuda_ok(cudaMemcpy(d_segs, host.data(), bytes, cudaMemcpyHostToDevice),
                 "cudaMemcpy (trajectory segments)", err))
      return false;
    const char *base = static_cast<const char *>(d_segs);
    segs.segs = reinterpret_cast<const TSeg *>(base);
    segs.passes = reinterpret_cast<const TSegPass *>(base + at_p);
    segs.gates = reinterpret_cast<const cb2::PassGateArgs32 *>(base + at_g);
    segs.sites = reinterpret_cast<const uint32_t *>(base + at_s);
    segs.starts = reinterpret_cast<const uint32_t *>(base + at_o);
    segs.mats = reinterpret_cast<const float *>(base + at_m);
    segs.mat_cap = (mat_cap + 15) & ~15u;
    return true;
  }

  bool upload(std::string &err) {
    if (!dirty) return true;
    mark_stats();
    if (!build_segments(err)) return false;
    if (graph) {
      cudaGraphExecDestroy(graph);
      graph = nullptr;
    }
    buf_free(d_ops, ops_bytes);
    buf_free(d_pool, pool_bytes);
    d_ops = nullptr;
    d_pool = nullptr;
    ops_bytes = pool_bytes = 0;
    const size_t ob = sizeof(TOp) * std::max<size_t>(1, ops.size());
    const size_t pb = sizeof(float2) * std::max<size_t>(1, pool.size());
    if (!cuda_ok(buf_alloc(reinterpret_cast<void **>(&d_ops), ob), "cudaMalloc (trajectory ops)", err))
      return false;
    ops_bytes = ob;
    if (!cuda_ok(buf_alloc(reinterpret_cast<void **>(&d_pool), pb), "cudaMalloc (trajectory matrices)", err))
      return false;
    pool_bytes = pb;
    if (!ops.empty() &&
        !cuda_ok(cudaMemcpy(d_ops, ops.data(), sizeof(TOp) * ops.size(), cudaMemcpyHostToDevice),
                 "cudaMemcpy (trajectory ops)", err))
      return false;
    if (!pool.empty() &&
        !cuda_ok(cudaMemcpy(d_pool, pool.data(), sizeof(float2) * pool.size(),
                            cudaMemcpyHostToDevice),
                 "cudaMemcpy (trajectory matrices)", err))
      return false;
    dirty = false;
    return true;
  }
};

TrajProgram *as_traj(void *p) {
  TrajProgram *t = static_cast<TrajProgram *>(p);
  return t && t->magic == kTrajMagic ? t : nullptr;
}

bool check_qubits(const TrajProgram &p, const uint32_t *q, uint32_t k, std::string &err) {
  if (!q || k == 0 || k > kTrajMaxGate) {
    err = "trajectory gates act on 1.." + std::to_string(kTrajMaxGate) + " qubits";
    return false;
  }
  for (uint32_t b = 0; b < k; ++b) {
    if (q[b] >= p.n) {
      err = "qubit out of range";
      return false;
    }
    if (b && q[b - 1] >= q[b]) {
      err = "qubits must be distinct and ascending";
      return false;
    }
  }
  return true;
}

}  // namespace

extern "C" {

void *cast_b200_traj_create(uint32_t n_qubits, char *err_buf, size_t err_buf_len) {
  if (n_qubits == 0 || n_qubits > kTrajMaxQubits) {
    cb2::write_err(err_buf, err_buf_len,
                   "trajectory statevectors support 1.." + std::to_string(kTrajMaxQubits) + " qubits");
    return nullptr;
  }
  try {
    TrajProgram *p = new TrajProgram;
    p->n = n_qubits;
    cb2::clear_err(err_buf, err_buf_len);
    return p;
  } catch (const std::exception &e) {
    cb2::write_err(err_buf, err_buf_len, e.what());
    return nullptr;
  }
}

void cast_b200_traj_destroy(void *prog) {
  TrajProgram *p = as_traj(prog);
  if (!p) return;
  p->magic = 0;
  delete p;
}

int cast_b200_traj_add_gate(void *prog, const cast_complex64_t *matrix, const uint32_t *qubits,
                            uint32_t k, char *err_buf, size_t err_buf_len) {
  TrajProgram *p = as_traj(prog);
  std::string err;
  if (!p || !matrix) err = "invalid trajectory program or matrix";
  else if (check_qubits(*p, qubits, k, err)) {
    std::lock_guard<std::mutex> lock(p->mu);
    TOp o{};
    o.type = T_GATE;
    o.k = k;
    for (uint32_t b = 0; b < k; ++b) o.q[b] = qubits[b];
    o.mat = p->push_matrix(matrix, 1ull << (2 * k));
    p->ops.push_back(o);
    p->dirty = true;
    cb2::clear_err(err_buf, err_buf_len);
    return 0;
  }
  cb2::write_err(err_buf, err_buf_len, err);
  return 1;
}

int cast_b200_traj_add_pauli_error(void *prog, double prob, const cast_complex64_t *mats,
                                   char *err_buf, size_t err_buf_len) {
  TrajProgram *p = as_traj(prog);
  if (!p || !mats || prob < 0.0 || prob > 1.0) {
    cb2::write_err(err_buf, err_buf_len, "invalid trajectory program, matrices or probability");
    return 1;
  }
  std::lock_guard<std::mutex> lock(p->mu);
  if (p->ops.empty() || (p->ops.back().type != T_GATE && p->ops.back().type != T_ERR)) {
    cb2::write_err(err_buf, err_buf_len, "a Pauli error must follow the gate block it belongs to");
    return 1;
  }
  size_t gi = p->ops.size() - 1;
  while (p->ops[gi].type != T_GATE) --gi;
  TOp o = p->ops[gi];
  o.type = T_ERR;
  o.prob = (float)prob;
  o.mat = p->push_matrix(mats, 3ull << (2 * o.k));
  p->ops.push_back(o);
  p->dirty = true;
  cb2::clear_err(err_buf, err_buf_len);
  return 0;
}

int cast_b200_traj_add_damping(void *prog, uint32_t mask, double gamma, char *err_buf,
                               size_t err_buf_len) {
  TrajProgram *p = as_traj(prog);
  if (!p || gamma < 0.0 || gamma >= 1.0 || mask == 0 || (p->n < 32 && (mask >> p->n) != 0)) {
    cb2::write_err(err_buf, err_buf_len, "invalid damping mask or rate");
    return 1;
  }
  std::lock_guard<std::mutex> lock(p->mu);
  TOp o{};
  o.type = T_DAMP;
  o.mask = mask;
  o.gamma = (float)gamma;
  p->ops.push_back(o);
  p->dirty = true;
  cb2::clear_err(err_buf, err_buf_len);
  return 0;
}

int cast_b200_traj_add_channel(void *prog, uint32_t qubit, const cast_complex64_t *kraus,
                               uint32_t n_kraus, char *err_buf, size_t err_buf_len) {
  TrajProgram *p = as_traj(prog);
  if (!p || !kraus || n_kraus == 0 || n_kraus > 4 || qubit >= p->n) {
    cb2::write_err(err_buf, err_buf_len, "invalid channel (1..4 Kraus operators on one qubit)");
    return 1;
  }
  std::lock_guard<std::mutex> lock(p->mu);
  TOp o{};
  o.type = T_CHAN;
  o.k = 1;
  o.q[0] = qubit;
  o.nk = n_kraus;
  o.mat = p->push_matrix(kraus, 4ull * n_kraus);
  p->ops.push_back(o);
  p->dirty = true;
  cb2::clear_err(err_buf, err_buf_len);
  return 0;
}

int cast_b200_traj_set_launch(void *prog, uint32_t threads, uint32_t max_ctas, char *err_buf,
                              size_t err_buf_len) {
  TrajProgram *p = as_traj(prog);
  if (!p || (threads != 0 && threads != 512 && threads != 1024)) {
    cb2::write_err(err_buf, err_buf_len, "threads per CTA must be 512, 1024 or 0 (by state size)");
    return 1;
  }
  std::lock_guard<std::mutex> lock(p->mu);
  p->threads = threads;
  p->max_ctas = max_ctas;
  cb2::clear_err(err_buf, err_buf_len);
  return 0;
}

uint32_t cast_b200_traj_num_qubits(const void *prog) {
  const TrajProgram *p = static_cast<const TrajProgram *>(prog);
  return p && p->magic == kTrajMagic ? p->n : 0;
}

int cast_b200_traj_get_op(const void *prog, uint32_t index, uint32_t *out_type, uint32_t *out_k,
                          uint32_t *out_qubits, double *out_prob, uint32_t *out_mask,
                          uint32_t *out_n_mats, cast_complex64_t *out_mats, size_t out_mats_len) {
  const TrajProgram *p = static_cast<const TrajProgram *>(prog);
  if (!p || p->magic != kTrajMagic || index >= p->ops.size()) return 1;
  const TOp &o = p->ops[index];
  size_t entries = 0;
  uint32_t nm = 0;
  double prob = 0;
  switch (o.type) {
  case T_GATE: nm = 1; entries = 1ull << (2 * o.k); break;
  case T_ERR: nm = 3; entries = 3ull << (2 * o.k); prob = o.prob; break;
  case T_DAMP: prob = o.gamma; break;
  default: nm = o.nk; entries = 4ull * o.nk; break;
  }
  if (out_type) *out_type = o.type;
  if (out_k) *out_k = o.k;
  if (out_qubits)
    for (uint32_t b = 0; b < o.k && b < kTrajMaxGate; ++b) out_qubits[b] = o.q[b];
  if (out_prob) *out_prob = prob;
  if (out_mask) *out_mask = o.mask;
  if (out_n_mats) *out_n_mats = nm;
  if (out_mats) {
    if (out_mats_len < entries) return 1;
    for (size_t e = 0; e < entries; ++e)
      out_mats[e] = {p->pool[o.mat + e].x, p->pool[o.mat + e].y};
  }
  return 0;
}

uint32_t cast_b200_traj_num_ops(const void *prog) {
  const TrajProgram *p = static_cast<const TrajProgram *>(prog);
  return p && p->magic == kTrajMagic ? (uint32_t)p->ops.size() : 0;
}

int cast_b200_traj_run(void *prog, uint32_t n_traj, uint64_t seed, double *out_z,
                       uint32_t *out_samples, void *stream, int use_graph, char *err_buf,
                       size_t err_buf_len) {
  return cast_b200_traj_run_range(prog, 0, n_traj, seed, out_z, out_samples, stream, use_graph,
                                  err_buf, err_buf_len);
}

int cast_b200_traj_run_range(void *prog, uint32_t first, uint32_t n_traj, uint64_t seed,
                             double *out_z, uint32_t *out_samples, void *stream, int use_graph,
                             char *err_buf, size_t err_buf_len) {
  TrajProgram *p = as_traj(prog);
  if (p && (uint64_t)first + n_traj > 0xFFFFFFFFull) {
    cb2::write_err(err_buf, err_buf_len, "trajectory range exceeds 2^32 indices");
    return 1;
  }
  if (!p || !out_z || n_traj == 0) {
    cb2::write_err(err_buf, err_buf_len, "invalid trajectory program, output or count");
    return 1;
  }
  try {
    std::lock_guard<std::mutex> lock(p->mu);
    std::string err;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (!p->upload(err)) {
      cb2::write_err(err_buf, err_buf_len, err);
      return 1;
    }
    const unsigned ctas = p->max_ctas ? p->max_ctas : auto_ctas(p->n);
    const unsigned grid = (unsigned)std::min<uint64_t>(n_traj, ctas);
    // a program with segments: 512, for their tiles in shared memory and the registers
    const unsigned threads = p->threads ? p->threads
                             : p->segs.segs ? (unsigned)kTMinThreads : cb2::plain_threads(p->n, p->width);
    if (p->ws_ctas < grid) {
      buf_free(p->d_ws, p->ws_bytes);
      p->d_ws = nullptr;
      p->ws_bytes = 0;
      if (!cuda_ok(buf_alloc(reinterpret_cast<void **>(&p->d_ws), (sizeof(float2) << p->n) * grid),
                   "cudaMalloc (trajectory workspace)", err)) {
        cb2::write_err(err_buf, err_buf_len, err);
        return 1;
      }
      p->ws_ctas = grid;
      p->ws_bytes = (sizeof(float2) << p->n) * grid;
      if (p->graph) {
        cudaGraphExecDestroy(p->graph);
        p->graph = nullptr;
      }
    }
    if (!p->d_run &&
        !cuda_ok(buf_alloc(reinterpret_cast<void **>(&p->d_run), sizeof(TRun)), "cudaMalloc (run)", err)) {
      cb2::write_err(err_buf, err_buf_len, err);
      return 1;
    }
    if (p->out_cap < n_traj) {
      buf_free(p->d_z, p->z_bytes);
      buf_free(p->d_sample, p->sample_bytes);
      p->d_z = nullptr;
      p->d_sample = nullptr;
      p->z_bytes = p->sample_bytes = 0;
      if (!cuda_ok(buf_alloc(reinterpret_cast<void **>(&p->d_z), sizeof(double) * n_traj * p->n),
                   "cudaMalloc (z)", err)) {
        cb2::write_err(err_buf, err_buf_len, err);
        return 1;
      }
      p->z_bytes = sizeof(double) * n_traj * p->n;
      if (!cuda_ok(buf_alloc(reinterpret_cast<void **>(&p->d_sample), sizeof(uint32_t) * n_traj),
                   "cudaMalloc (samples)", err)) {
        cb2::write_err(err_buf, err_buf_len, err);
        return 1;
      }
      p->sample_bytes = sizeof(uint32_t) * n_traj;
      p->out_cap = n_traj;
      if (p->graph) {
        cudaGraphExecDestroy(p->graph);
        p->graph = nullptr;
      }
    }
    TRun r{n_traj, first, seed};
    if (!cuda_ok(cudaMemcpyAsync(p->d_run, &r, sizeof(r), cudaMemcpyHostToDevice, s),
                 "cudaMemcpyAsync (run parameters)", err)) {
      cb2::write_err(err_buf, err_buf_len, err);
      return 1;
    }
    const uint32_t n_ops = (uint32_t)p->ops.size();
    if (use_graph && s) {
      if (p->graph && (p->graph_stream != stream || p->graph_grid != grid || p->graph_threads != threads)) {
        cudaGraphExecDestroy(p->graph);
        p->graph = nullptr;
      }
      if (!p->graph) {
        cudaGraph_t gph = nullptr;
        if (!cuda_ok(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal),
                     "cudaStreamBeginCapture", err)) {
          cb2::write_err(err_buf, err_buf_len, err);
          return 1;
        }
        const cudaError_t lrc = launch_trajectories(grid, threads, s, p->d_ops, n_ops, p->d_pool,
                                                    p->d_ws, p->n, p->d_run, p->d_z, p->d_sample, p->segs);
        const cudaError_t erc = cudaStreamEndCapture(s, &gph);
        if (!cuda_ok(lrc, "trajectory kernel capture", err) ||
            !cuda_ok(erc, "cudaStreamEndCapture", err) ||
            !cuda_ok(cudaGraphInstantiate(&p->graph, gph, 0), "cudaGraphInstantiate", err)) {
          if (gph) cudaGraphDestroy(gph);
          cb2::write_err(err_buf, err_buf_len, err);
          return 1;
        }
        cudaGraphDestroy(gph);
        p->graph_stream = stream;
        p->graph_grid = grid;
        p->graph_threads = threads;
      }
      if (!cuda_ok(cudaGraphLaunch(p->graph, s), "cudaGraphLaunch", err)) {
        cb2::write_err(err_buf, err_buf_len, err);
        return 1;
      }
    } else {
      if (!cuda_ok(launch_trajectories(grid, threads, s, p->d_ops, n_ops, p->d_pool, p->d_ws, p->n,
                                       p->d_run, p->d_z, p->d_sample, p->segs),
                   "trajectory kernel launch", err)) {
        cb2::write_err(err_buf, err_buf_len, err);
        return 1;
      }
    }
    if (!cuda_ok(cudaMemcpyAsync(out_z, p->d_z, sizeof(double) * n_traj * p->n,
                                 cudaMemcpyDeviceToHost, s),
                 "cudaMemcpyAsync (z)", err) ||
        (out_samples &&
         !cuda_ok(cudaMemcpyAsync(out_samples, p->d_sample, sizeof(uint32_t) * n_traj,
                                  cudaMemcpyDeviceToHost, s),
                  "cudaMemcpyAsync (samples)", err)) ||
        !cuda_ok(cudaStreamSynchronize(s), "cudaStreamSynchronize (trajectories)", err)) {
      // The kernel may already be queued: let it finish before returning, so
      // that no buffer of this program is handed on (buffer cache) in use.
      cudaStreamSynchronize(s);
      cb2::write_err(err_buf, err_buf_len, err);
      return 1;
    }
    cb2::clear_err(err_buf, err_buf_len);
    return 0;
  } catch (const std::exception &e) {
    cb2::write_err(err_buf, err_buf_len, e.what());
    return 1;
  }
}

}  // extern "C"
