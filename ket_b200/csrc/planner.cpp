// planner.cpp -- gate lowering and the fusion planner (host, C++20).
//
// Lowering follows ket's gate definitions (src/simulator.cpp:38-254 for the
// matrices, :259-338 for the dispatch).  Planning replaces ket's Fuser
// (src/simulator.cpp:400-477):
//   * FUSE_NONE       one specialised kernel per gate (the plain method);
//   * FUSE_REFERENCE  ket's own rule -- a gate joins the open block only if
//                     its qubits are a subset of the block's first gate's;
//   * FUSE_GREEDY     blocks of up to k qubits grown over the gate DAG (a
//                     gate may join past gates on other qubits, never past a
//                     pending gate on one of its own qubits), kept only when a
//                     static byte model says one dense pass beats the
//                     specialised kernels it replaces;
//   * FUSE_LEARNED    the same candidate generator, with block costs from the
//                     MLP cost model and the partition chosen by predicted time.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <functional>
#include <numeric>
#include <string>
#include <thread>
#include <vector>

#include "internal.h"

namespace kb {

bool is_unitary(int type) { return type >= KETGPU_H && type <= KETGPU_CSWAP; }

int gate_arity(int type) {
  if (type < 0) return -1;
  if (type <= KETGPU_U) return 1;
  if (type <= KETGPU_SWAP) return 2;
  if (type <= KETGPU_CSWAP) return 3;
  return 0;
}

void validate_ops(int n, const ketgpu_op* ops, uint64_t nops) {
  for (uint64_t i = 0; i < nops; ++i) {
    const ketgpu_op& o = ops[i];
    if (o.type < 0 || o.type > KETGPU_PROBE)
      fail(KETGPU_ERR_INVALID, "ket: unknown gate code " + std::to_string(o.type));
    if (o.type == KETGPU_COMPOSITE)
      fail(KETGPU_ERR_INVALID, "ket: composite blocks must be flattened before the device call");
    const int a = is_unitary(o.type) ? gate_arity(o.type) : (o.type == KETGPU_MEASURE ? 1 : 0);
    for (int j = 0; j < a; ++j) {
      if (o.q[j] < 0 || o.q[j] >= n)
        fail(KETGPU_ERR_OUT_OF_RANGE, "ket: qubit index " + std::to_string(o.q[j]) +
                                          " is out of range for a " + std::to_string(n) +
                                          "-qubit circuit");
      for (int k = 0; k < j; ++k)
        if (o.q[j] == o.q[k])
          fail(KETGPU_ERR_INVALID,
               "ket: a gate cannot act on qubit " + std::to_string(o.q[j]) + " more than once");
    }
  }
}

void single_matrix(int type, const double* p, cplx m[4]) {
  const double r = 1.0 / std::sqrt(2.0);
  double c = 0, sn = 0;
  if (type == KETGPU_RX || type == KETGPU_RY || type == KETGPU_RZ || type == KETGPU_U ||
      type == KETGPU_CRX || type == KETGPU_CRY || type == KETGPU_CRZ || type == KETGPU_CU) {
    c = std::cos(p[0] / 2.0);
    sn = std::sin(p[0] / 2.0);
  }
  switch (type) {
    case KETGPU_H: case KETGPU_CH: m[0] = r; m[1] = r; m[2] = r; m[3] = -r; return;
    case KETGPU_X: case KETGPU_CX: case KETGPU_CCX: m[0] = 0; m[1] = 1; m[2] = 1; m[3] = 0; return;
    case KETGPU_Y: case KETGPU_CY: m[0] = 0; m[1] = cplx(0, -1); m[2] = cplx(0, 1); m[3] = 0; return;
    case KETGPU_Z: m[0] = 1; m[1] = 0; m[2] = 0; m[3] = -1; return;
    case KETGPU_S: m[0] = 1; m[1] = 0; m[2] = 0; m[3] = cplx(0, 1); return;
    case KETGPU_SDG: m[0] = 1; m[1] = 0; m[2] = 0; m[3] = cplx(0, -1); return;
    case KETGPU_T: m[0] = 1; m[1] = 0; m[2] = 0; m[3] = cplx(r, r); return;
    case KETGPU_TDG: m[0] = 1; m[1] = 0; m[2] = 0; m[3] = cplx(r, -r); return;
    case KETGPU_RX: case KETGPU_CRX:
      m[0] = c; m[1] = cplx(0, -sn); m[2] = cplx(0, -sn); m[3] = c; return;
    case KETGPU_RY: case KETGPU_CRY: m[0] = c; m[1] = -sn; m[2] = sn; m[3] = c; return;
    case KETGPU_RZ: case KETGPU_CRZ: m[0] = cplx(c, -sn); m[1] = 0; m[2] = 0; m[3] = cplx(c, sn); return;
    case KETGPU_U: case KETGPU_CU:
      m[0] = cplx(c, 0.0);
      m[1] = -std::polar(sn, p[2]);
      m[2] = std::polar(sn, p[1]);
      m[3] = std::polar(c, p[1] + p[2]);
      return;
    default:
      fail(KETGPU_ERR_LOGIC, "single_matrix: not a 1-qubit gate");
  }
}

namespace {

void set_fixed(Pass& p, std::initializer_list<int> qs) {
  p.nfixed = 0;
  for (int q : qs) p.fixed[p.nfixed++] = q;
  std::sort(p.fixed, p.fixed + p.nfixed);
}

}  // namespace

Pass lower_gate(const ketgpu_op& op) {
  Pass p;
  const int t = op.type;
  const auto bit = [&](int j) { return uint64_t{1} << op.q[j]; };
  if (gate_arity(t) == 1) {
    single_matrix(t, op.p, p.m);
    if (t == KETGPU_Z || t == KETGPU_S || t == KETGPU_SDG || t == KETGPU_T || t == KETGPU_TDG) {
      p.kind = PassKind::Phase;
      set_fixed(p, {op.q[0]});
      p.p0 = bit(0);
      p.m[0] = p.m[3];
    } else {
      p.kind = PassKind::Pair;
      set_fixed(p, {op.q[0]});
      p.p0 = 0;
      p.p1 = bit(0);
      p.mode = (t == KETGPU_X) ? kPairSwap : (t == KETGPU_RZ) ? kPairDiag : kPairGeneral;
    }
    return p;
  }
  switch (t) {
    case KETGPU_CZ: case KETGPU_CP:
      p.kind = PassKind::Phase;
      set_fixed(p, {op.q[0], op.q[1]});
      p.p0 = bit(0) | bit(1);
      p.m[0] = (t == KETGPU_CZ) ? cplx(-1.0, 0.0) : cplx(std::cos(op.p[0]), std::sin(op.p[0]));
      return p;
    case KETGPU_SWAP:
      p.kind = PassKind::Pair;
      p.mode = kPairSwap;
      set_fixed(p, {op.q[0], op.q[1]});
      p.p0 = bit(0);
      p.p1 = bit(1);
      return p;
    case KETGPU_CCX:
      p.kind = PassKind::Pair;
      p.mode = kPairSwap;
      set_fixed(p, {op.q[0], op.q[1], op.q[2]});
      p.p0 = bit(0) | bit(1);
      p.p1 = bit(0) | bit(1) | bit(2);
      return p;
    case KETGPU_CSWAP:
      p.kind = PassKind::Pair;
      p.mode = kPairSwap;
      set_fixed(p, {op.q[0], op.q[1], op.q[2]});
      p.p0 = bit(0) | bit(1);
      p.p1 = bit(0) | bit(2);
      return p;
    default: {  // controlled 2x2: CH, CX, CY, CRx, CRy, CRz, CU
      single_matrix(t, op.p, p.m);
      p.kind = PassKind::Pair;
      p.mode = (t == KETGPU_CX) ? kPairSwap : (t == KETGPU_CRZ) ? kPairDiag : kPairGeneral;
      set_fixed(p, {op.q[0], op.q[1]});
      p.p0 = bit(0);
      p.p1 = bit(0) | bit(1);
      return p;
    }
  }
}

double gate_traffic_fraction(const ketgpu_op& op) {
  switch (op.type) {  // the gates lower_gate makes phase passes
    case KETGPU_Z: case KETGPU_S: case KETGPU_SDG: case KETGPU_T: case KETGPU_TDG: return 0.5;
    case KETGPU_CZ: case KETGPU_CP: return 0.25;
    default: return std::ldexp(1.0, 1 - gate_arity(op.type));
  }
}

namespace {

// Apply a lowered pass to a small dense vector (host, FP64).
void apply_small(const Pass& p, cplx* v, int nloc) {
  const uint64_t dim = uint64_t{1} << nloc;
  const uint64_t count = dim >> p.nfixed;
  for (uint64_t i = 0; i < count; ++i) {
    uint64_t b = i;
    for (int j = 0; j < p.nfixed; ++j) {
      const int f = p.fixed[j];
      b = ((b >> f) << (f + 1)) | (b & ((uint64_t{1} << f) - 1));
    }
    if (p.kind == PassKind::Phase) {
      v[b | p.p0] *= p.m[0];
      continue;
    }
    const cplx a = v[b | p.p0], c = v[b | p.p1];
    if (p.mode == kPairSwap) {
      v[b | p.p0] = c;
      v[b | p.p1] = a;
    } else {
      v[b | p.p0] = p.m[0] * a + p.m[1] * c;
      v[b | p.p1] = p.m[2] * a + p.m[3] * c;
    }
  }
}

}  // namespace

std::vector<Pass> lower_block(const ketgpu_op* ops, const std::vector<int>& gates, const int* qubits, int k) {
  std::vector<Pass> local;
  local.reserve(gates.size());
  for (int gi : gates) {
    ketgpu_op o = ops[gi];
    for (int j = 0; j < gate_arity(o.type); ++j) {
      int li = -1;
      for (int b = 0; b < k; ++b)
        if (qubits[b] == o.q[j]) li = b;
      if (li < 0) fail(KETGPU_ERR_LOGIC, "lower_block: gate outside block");
      o.q[j] = li;
    }
    local.push_back(lower_gate(o));
  }
  return local;
}

std::vector<cplx> block_matrix(const ketgpu_op* ops, const std::vector<int>& gates, const int* qubits, int k) {
  const int dim = 1 << k;
  const std::vector<Pass> local = lower_block(ops, gates, qubits, k);
  std::vector<cplx> mat((size_t)dim * dim);
  std::vector<cplx> col(dim);
  for (int c = 0; c < dim; ++c) {
    std::fill(col.begin(), col.end(), cplx(0.0, 0.0));
    col[c] = 1.0;
    for (const Pass& p : local) apply_small(p, col.data(), k);
    for (int r = 0; r < dim; ++r) mat[(size_t)r * dim + c] = col[r];
  }
  return mat;
}

PlanOptions resolve_options(const ketgpu_options* opt) {
  PlanOptions o;
  if (!opt) return o;
  if (opt->precision != KETGPU_C64 && opt->precision != KETGPU_C128)
    fail(KETGPU_ERR_INVALID, "precision must be KETGPU_C64 or KETGPU_C128");
  if (opt->fusion < KETGPU_FUSE_NONE || opt->fusion > KETGPU_FUSE_LEARNED)
    fail(KETGPU_ERR_INVALID, "unknown fusion mode");
  o.precision = opt->precision;
  o.fusion = opt->fusion;
  // default block size: 6 qubits for complex64 on the tensor cores (their
  // 3xFP16 blocks stay memory-bound at k = 6, so fewer passes win), 5 for
  // the SIMT blocks, whose arithmetic grows with 2^k per amplitude
  o.max_k = opt->max_block_qubits ? opt->max_block_qubits
                                  : (opt->precision == KETGPU_C64 && opt->tensor_cores ? 6 : 5);
  if (o.max_k < 1 || o.max_k > 6) fail(KETGPU_ERR_INVALID, "max_block_qubits must be in [1, 6]");
  o.tensor = opt->tensor_cores != 0;
  o.renormalize = opt->renormalize;
  return o;
}

namespace {

struct Block {
  std::vector<int> gates;  // op indices, program order
  std::vector<int> qubits; // sorted
  bool diag = false;       // a run of diagonal gates: one Diagonal pass
};

uint64_t qubit_mask(const ketgpu_op& o) {
  uint64_t m = 0;
  for (int j = 0; j < gate_arity(o.type); ++j) m |= uint64_t{1} << o.q[j];
  return m;
}

// Cost (in full-state passes) of a dense k-qubit block pass: one HBM pass,
// plus the compute that outgrows it at large k.
double fused_cost_static(int k, int precision, bool tensor) {
  if (precision == KETGPU_C128) return k <= 4 ? 1.0 : (k == 5 ? 1.35 : 2.7);
  if (tensor && k >= 4 && k <= 6) return 1.0;
  return k <= 4 ? 1.0 : (k == 5 ? 1.45 : 2.9);
}

// Predicted gain (fraction of the greedy plan's predicted time) the learned
// planner needs before it departs from the greedy plan.
constexpr double kLearnedMargin = 0.02;

bool block_on_tensor_cores(int n, int k, const PlanOptions& opt) {
  return opt.precision == KETGPU_C64 && opt.tensor && tc_supported(k) && n >= k + 7;
}

// A partition in flat arrays: the planner grows many and keeps one.
struct Partition {
  std::vector<int> gates;        // op indices, block after block
  std::vector<size_t> end;       // where each block ends in them
  std::vector<uint64_t> qubits;  // masks
  std::vector<char> diag;
  void close(uint64_t q, bool d) {
    end.push_back(gates.size());
    qubits.push_back(q);
    diag.push_back(d);
  }
};

// Greedy DAG-aware block growth over the gates `order` of `ops`.  With
// diag_runs, whenever the next gate to place is diagonal, every diagonal gate
// that can be moved to the front of what is left (no earlier non-diagonal
// gate shares a qubit with it) is collected; if that run spans more qubits
// than one block holds, it becomes a single Diagonal pass.
Partition grow_blocks(int n, const ketgpu_op* ops, const std::vector<int>& order, int max_k, bool diag_runs) {
  const size_t G = order.size();
  Partition part;
  part.gates.reserve(G);
  // gates left, a linked list in order; qubit sets as masks
  std::vector<uint64_t> mask(G);
  std::vector<char> diag(G);
  std::vector<size_t> next(G + 1);
  for (size_t i = 0; i < G; ++i) {
    mask[i] = qubit_mask(ops[order[i]]);
    diag[i] = is_diagonal_gate(ops[order[i]].type);
  }
  std::iota(next.begin(), next.end(), size_t{0});  // next[j]: the gate after position j - 1
  size_t& first = next[0];
  const uint64_t all = n >= 64 ? ~uint64_t{0} : ((uint64_t{1} << n) - 1);
  std::vector<size_t> run;
  while (first < G) {
    if (diag_runs && diag[first]) {
      run.clear();
      uint64_t blk = 0, span = 0;
      for (size_t i = first; i < G && blk != all; i = next[i + 1]) {
        if (diag[i] && !(mask[i] & blk)) {
          run.push_back(i);
          span |= mask[i];
        } else {
          blk |= mask[i];
        }
      }
      if (run.size() >= 2 && __builtin_popcountll(span) > max_k) {
        size_t r = 0;
        for (size_t prev = 0; r < run.size();) {
          const size_t i = next[prev];
          if (i == run[r]) {
            part.gates.push_back(order[i]);
            next[prev] = next[i + 1];
            ++r;
          } else {
            prev = i + 1;
          }
        }
        part.close(span, true);
        continue;
      }
    }
    uint64_t blocked = 0, inq = 0;
    const size_t start = part.gates.size();
    for (size_t prev = 0, i; (i = next[prev]) < G;) {
      const uint64_t m = mask[i];
      if (part.gates.size() == start || (!(m & blocked) && __builtin_popcountll(inq | m) <= max_k)) {
        inq |= m;
        part.gates.push_back(order[i]);
        next[prev] = next[i + 1];
      } else {
        blocked |= m;
        if (blocked == all) break;
        // nothing more can join once every block qubit is blocked and the
        // block is full
        if (__builtin_popcountll(inq) == max_k && !(inq & ~blocked)) break;
        prev = i + 1;
      }
    }
    part.close(inq, false);
  }
  return part;
}

struct Dependencies {  // of a segment's gates
  std::vector<int> depth, lowest, indegree;  // ASAP depth, lowest qubit, direct predecessors
  std::vector<int> succ_at, succ;            // successors of gate i: succ[succ_at[i] .. succ_at[i + 1])
};

Dependencies dependencies(const ketgpu_op* ops, const std::vector<int>& seg, int n) {
  const size_t G = seg.size();
  Dependencies d;
  d.depth.assign(G, 0);
  d.lowest.assign(G, 0);
  d.indegree.assign(G, 0);
  d.succ_at.assign(G + 1, 0);
  std::vector<int> last(n, -1), from, to;
  for (size_t i = 0; i < G; ++i) {
    const ketgpu_op& o = ops[seg[i]];
    int dep = 0, lo = n;
    for (int j = 0; j < gate_arity(o.type); ++j) {
      const int q = o.q[j];
      lo = std::min(lo, q);
      if (last[q] >= 0) {
        dep = std::max(dep, d.depth[last[q]] + 1);
        from.push_back(last[q]);
        to.push_back((int)i);
        ++d.succ_at[last[q] + 1];
        ++d.indegree[i];
      }
      last[q] = (int)i;
    }
    d.depth[i] = dep;
    d.lowest[i] = lo;
  }
  std::partial_sum(d.succ_at.begin(), d.succ_at.end(), d.succ_at.begin());
  d.succ.resize(from.size());
  std::vector<int> at(d.succ_at.begin(), d.succ_at.end() - 1);
  for (size_t e = 0; e < from.size(); ++e) d.succ[at[from[e]]++] = to[e];
  return d;
}

// Topological orders of a segment's gates for the greedy block growth.  The
// program order is one; a "band" order of width w sorts the gates by
// ((ASAP depth + offset) / w, lowest qubit, depth), subject to every dependency, so
// growth from the first gate follows a few neighbouring qubits through w
// levels of the circuit before moving on: light-cone-shaped blocks.  On the
// 30-qubit, 40-layer brick wall at k = 5 the best band order needs 119
// passes against 154 in program order.  Returns op indices.
std::vector<int> band_order(const std::vector<int>& seg, const Dependencies& d, int w, int off) {
  const size_t G = seg.size();
  // (band, lowest qubit, depth, gate), smallest first
  struct Key {
    uint64_t hi;
    uint32_t depth;
    int gate;
    bool operator>(const Key& o) const {
      return hi != o.hi ? hi > o.hi : depth != o.depth ? depth > o.depth : gate > o.gate;
    }
  };
  std::vector<int> indeg = d.indegree, out;
  std::vector<Key> heap;
  out.reserve(G);
  auto key = [&](int i) {
    return Key{((uint64_t)((d.depth[i] + off) / w) << 8) | (uint64_t)d.lowest[i], (uint32_t)d.depth[i], i};
  };
  for (size_t i = 0; i < G; ++i)
    if (!indeg[i]) heap.push_back(key((int)i));
  std::make_heap(heap.begin(), heap.end(), std::greater<Key>());
  while (!heap.empty()) {
    std::pop_heap(heap.begin(), heap.end(), std::greater<Key>());
    const int i = heap.back().gate;
    heap.pop_back();
    out.push_back(seg[i]);
    for (int e = d.succ_at[i]; e < d.succ_at[i + 1]; ++e)
      if (--indeg[d.succ[e]] == 0) {
        heap.push_back(key(d.succ[e]));
        std::push_heap(heap.begin(), heap.end(), std::greater<Key>());
      }
  }
  return out;
}

// Band widths the planner tries besides the program order, each at every
// offset (the band boundaries shifted by 0 .. w-1 levels).
constexpr int kBandWidths[] = {3, 4, 5, 6, 7, 8};

// Static cost of a partition in full-state passes: each block fused or as
// its separate gates, whichever is cheaper; a diagonal run is one pass.
// fraction: of each gate, from op index `from` on.
double partition_cost(const std::vector<double>& fraction, int from, const Partition& part, const PlanOptions& opt) {
  double total = 0;
  size_t g = 0;
  for (size_t b = 0; b < part.end.size(); ++b) {
    const size_t count = part.end[b] - g;
    double separate = 0;
    for (; g < part.end[b]; ++g) separate += fraction[part.gates[g] - from];
    if (part.diag[b]) total += 1.0;
    else
      total += count > 1 ? std::min(separate, fused_cost_static(__builtin_popcountll(part.qubits[b]), opt.precision,
                                                                 opt.tensor))
                         : separate;
  }
  return total;
}

// Greedy growth over the program order and every band order (width,
// offset); the partition with the least static cost, the earliest candidate
// on ties.  The candidates are grown on up to 16 host threads.
std::vector<Block> best_partition(int n, const ketgpu_op* ops, const std::vector<int>& seg,
                                  const PlanOptions& opt) {
  std::vector<std::pair<int, int>> cands{{0, 0}};  // (0, 0): the program order
  for (int w : kBandWidths)
    for (int off = 0; off < w; ++off) cands.push_back({w, off});
  const size_t C = cands.size();
  std::vector<Partition> parts(C);
  std::vector<double> cost(C, 0.0);
  const Dependencies deps = dependencies(ops, seg, n);
  // of the segment's span alone: a circuit may have as many segments as gates
  const auto [from, last] = std::minmax_element(seg.begin(), seg.end());
  const int first_op = seg.empty() ? 0 : *from;
  std::vector<double> fraction(seg.empty() ? 0 : *last - first_op + 1, 0.0);
  for (int gi : seg) fraction[gi - first_op] = gate_traffic_fraction(ops[gi]);
  auto work = [&](size_t c) {
    parts[c] = grow_blocks(n, ops, cands[c].first ? band_order(seg, deps, cands[c].first, cands[c].second) : seg,
                           std::max(1, opt.max_k), true);
    cost[c] = partition_cost(fraction, first_op, parts[c], opt);
  };
  const unsigned nt = seg.size() < 256 ? 1u : std::min<unsigned>(16u, std::max(1u, std::thread::hardware_concurrency()));
  if (nt <= 1) {
    for (size_t c = 0; c < C; ++c) work(c);
  } else {
    std::atomic<size_t> next{0};
    std::vector<std::thread> th;
    for (unsigned t = 0; t < nt; ++t)
      th.emplace_back([&] {
        for (size_t c; (c = next.fetch_add(1)) < C;) work(c);
      });
    for (auto& x : th) x.join();
  }
  size_t best = 0;
  for (size_t c = 1; c < C; ++c)
    if (cost[c] < cost[best] - 1e-9) best = c;
  const Partition& p = parts[best];
  std::vector<Block> blocks(p.end.size());
  for (size_t b = 0, g = 0; b < blocks.size(); g = p.end[b++]) {
    blocks[b].gates.assign(p.gates.begin() + (std::ptrdiff_t)g, p.gates.begin() + (std::ptrdiff_t)p.end[b]);
    for (int q = 0; q < n; ++q)
      if ((p.qubits[b] >> q) & 1) blocks[b].qubits.push_back(q);
    blocks[b].diag = p.diag[b];
  }
  return blocks;
}

// ket's Fuser block rule on one barrier-free segment.
std::vector<Block> reference_blocks(const ketgpu_op* ops, const std::vector<int>& order) {
  std::vector<Block> blocks;
  Block cur;
  std::vector<int> first_qubits;
  for (int idx : order) {
    const ketgpu_op& o = ops[idx];
    const int a = gate_arity(o.type);
    bool subset = !cur.gates.empty();
    for (int j = 0; j < a && subset; ++j)
      if (std::find(first_qubits.begin(), first_qubits.end(), o.q[j]) == first_qubits.end()) subset = false;
    if (!cur.gates.empty() && !subset) {
      blocks.push_back(std::move(cur));
      cur = Block();
    }
    if (cur.gates.empty()) {
      first_qubits.assign(o.q, o.q + a);
      cur.qubits = first_qubits;
    }
    cur.gates.push_back(idx);
  }
  if (!cur.gates.empty()) blocks.push_back(std::move(cur));
  return blocks;
}

void emit_single(Plan& plan, const ketgpu_op& o, int idx) {
  Pass p = lower_gate(o);
  p.first_op = idx;
  p.n_gates = 1;
  p.gates = {idx};
  plan.passes.push_back(p);
}

void emit_run(Plan& plan, const ketgpu_op* ops, const std::vector<int>& gates) {
  std::vector<Pass> lowered;
  for (int gi : gates) lowered.push_back(lower_gate(ops[gi]));
  Pass p;
  p.kind = PassKind::SharedRun;
  p.run_index = plan.runs.size();
  p.first_op = gates.front();
  p.n_gates = (int)gates.size();
  p.gates = gates;
  plan.runs.push_back(std::move(lowered));
  plan.passes.push_back(p);
}

void emit_diagonal(Plan& plan, int n, const ketgpu_op* ops, const Block& b) {
  DiagPoly poly;
  poly.a.assign(n, 0.0);
  poly.b.assign((size_t)n * n, 0.0);
  for (int gi : b.gates) add_diagonal_gate(ops[gi], poly, n);
  Pass p;
  p.kind = PassKind::Diagonal;
  p.k = (int)b.qubits.size();
  p.diag_index = plan.diags.size();
  p.first_op = b.gates.front();
  p.n_gates = (int)b.gates.size();
  p.gates = b.gates;
  plan.diags.push_back(std::move(poly));
  plan.passes.push_back(p);
}

void emit_fused(Plan& plan, int n, const ketgpu_op* ops, const Block& b, const PlanOptions& opt) {
  std::vector<int> qs = b.qubits;
  std::sort(qs.begin(), qs.end());
  // complex64 on the tensor cores: a 2- or 3-qubit block is padded to 4
  // qubits (identity on the highest free qubits, so the block's group bits
  // stay low) and runs at HBM speed instead of on the SIMT block kernel.
  if (qs.size() >= 2 && qs.size() < 4 && !block_on_tensor_cores(n, (int)qs.size(), opt) &&
      block_on_tensor_cores(n, 4, opt)) {
    for (int q = n - 1; q >= 0 && qs.size() < 4; --q)
      if (std::find(qs.begin(), qs.end(), q) == qs.end()) qs.push_back(q);
    std::sort(qs.begin(), qs.end());
  }
  // complex128: a 2-qubit block likewise runs as a 3-qubit one (the FP64
  // matrix instructions work on 16 rows of the block's real embedding).
  if (opt.precision == KETGPU_C128 && qs.size() == 2 && f64_supported(n, 3)) {
    for (int q = n - 1; q >= 0 && qs.size() < 3; --q)
      if (std::find(qs.begin(), qs.end(), q) == qs.end()) qs.push_back(q);
    std::sort(qs.begin(), qs.end());
  }
  const int k = (int)qs.size();
  Pass p;
  p.first_op = b.gates.front();
  p.n_gates = (int)b.gates.size();
  p.gates = b.gates;
  if (k == 1) {  // one 2x2 through the streaming pair kernel
    const std::vector<cplx> mat = block_matrix(ops, b.gates, qs.data(), k);
    p.kind = PassKind::Pair;
    p.mode = kPairGeneral;
    p.nfixed = 1;
    p.fixed[0] = qs[0];
    p.p0 = 0;
    p.p1 = uint64_t{1} << qs[0];
    for (int j = 0; j < 4; ++j) p.m[j] = mat[j];
    plan.passes.push_back(p);
    return;
  }
  p.kind = PassKind::Fused;
  p.k = k;
  for (int j = 0; j < k; ++j) p.qubits[j] = qs[j];
  p.tensor = block_on_tensor_cores(n, k, opt);
  plan.passes.push_back(p);
}

// Orders the passes, under every dependency (passes that share a qubit keep
// their order), so that qubits become active late: of the passes that can go
// next, the one that leaves the fewest qubits active, the earliest on ties.
// A run from |0...0> touches 2^active amplitudes a pass (PassRunner).  Once
// every qubit that a pass activates is active the rest keep their order.
// A pass can go next when it is the first one left on each of its qubits, so
// at most n are looked at a step: a circuit of 60,000 lone gates that leaves a
// qubit idle is planned in 1.0 s (2.3 with a search through all that are left).
void order_passes(Plan& plan, const ketgpu_op* ops, int n) {
  const size_t P = plan.passes.size();
  std::vector<uint64_t> touch(P, 0), grow(P, 0);
  uint64_t grown = 0;
  for (size_t i = 0; i < P; ++i) {
    for (int gi : plan.passes[i].gates) {
      touch[i] |= qubit_mask(ops[gi]);
      if (!is_diagonal_gate(ops[gi].type)) grow[i] |= qubit_mask(ops[gi]);
    }
    grown |= grow[i];
  }
  std::vector<std::vector<size_t>> on(n);  // passes of each qubit, in order
  std::vector<int> behind(P, 0);           // qubits on which an earlier pass is left
  for (size_t i = 0; i < P; ++i)
    for (uint64_t m = touch[i]; m; m &= m - 1) {
      std::vector<size_t>& list = on[__builtin_ctzll(m)];
      behind[i] += !list.empty();
      list.push_back(i);
    }
  std::vector<size_t> at(n, 0), ready, order;  // ready: ascending
  std::vector<char> done(P, 0);
  for (size_t i = 0; i < P; ++i)
    if (!behind[i]) ready.push_back(i);
  uint64_t active = 0;
  while (!ready.empty() && active != grown) {
    auto best = ready.begin();
    int best_count = 65;
    for (auto r = ready.begin(); r != ready.end(); ++r) {
      const int c = __builtin_popcountll(active | grow[*r]);
      if (c < best_count) {
        best_count = c;
        best = r;
      }
    }
    const size_t i = *best;
    ready.erase(best);
    active |= grow[i];
    order.push_back(i);
    done[i] = 1;
    for (uint64_t m = touch[i]; m; m &= m - 1) {
      const int q = __builtin_ctzll(m);
      if (++at[q] == on[q].size()) continue;
      const size_t next = on[q][at[q]];
      if (--behind[next] == 0) ready.insert(std::upper_bound(ready.begin(), ready.end(), next), next);
    }
  }
  for (size_t i = 0; i < P; ++i)
    if (!done[i]) order.push_back(i);
  std::vector<Pass> sorted;
  sorted.reserve(P);
  for (size_t i : order) sorted.push_back(std::move(plan.passes[i]));
  plan.passes = std::move(sorted);
}

}  // namespace

// 48 features: scale (n, bytes), pass kind, block geometry (k, span, low /
// high qubits, runs of adjacent qubits, coalescing), gate content (counts by
// kind), precision and an L2-residency flag.  Index layout is fixed; the
// trained cost model depends on it.
void pass_features(int n, int precision, const std::vector<const ketgpu_op*>& gates,
                   const std::vector<int>& qubits, bool fused, bool tensor, float* f) {
  for (int i = 0; i < kFeatures; ++i) f[i] = 0.f;
  const double amp = precision == KETGPU_C64 ? 8.0 : 16.0;
  const double state = amp * std::ldexp(1.0, n);
  double frac = 1.0;
  if (!fused && gates.size() == 1) frac = gate_traffic_fraction(*gates[0]);
  const int k = (int)qubits.size();
  int lo = n, hi = -1, runs = 0, low7 = 0;
  std::vector<int> qs = qubits;
  std::sort(qs.begin(), qs.end());
  for (size_t i = 0; i < qs.size(); ++i) {
    lo = std::min(lo, qs[i]);
    hi = std::max(hi, qs[i]);
    if (i == 0 || qs[i] != qs[i - 1] + 1) ++runs;
    if (qs[i] < 7) ++low7;
  }
  f[0] = (float)n / 32.f;
  f[1] = (float)(std::log2(2.0 * state * frac) / 40.0);
  f[2] = fused ? 1.f : 0.f;
  f[3] = tensor ? 1.f : 0.f;
  f[4] = (float)k / 6.f;
  f[5] = (float)gates.size() / 64.f;
  f[6] = k ? (float)lo / (float)n : 0.f;
  f[7] = k ? (float)hi / (float)n : 0.f;
  f[8] = k ? (float)(hi - lo + 1) / (float)n : 0.f;
  f[9] = (k && lo == 0) ? 1.f : 0.f;
  f[10] = (float)low7 / 6.f;
  f[11] = (float)runs / 6.f;
  f[12] = (float)frac;
  f[13] = precision == KETGPU_C128 ? 1.f : 0.f;
  if (k >= 1 && k <= 6) f[13 + k] = 1.f;  // 14..19
  for (const ketgpu_op* g : gates) {
    int slot;
    switch (g->type) {
      case KETGPU_H: slot = 0; break;
      case KETGPU_S: case KETGPU_SDG: case KETGPU_Z: case KETGPU_T: case KETGPU_TDG: slot = 1; break;
      case KETGPU_RX: slot = 2; break;
      case KETGPU_RY: slot = 3; break;
      case KETGPU_RZ: slot = 4; break;
      case KETGPU_U: case KETGPU_X: case KETGPU_Y: slot = 5; break;
      case KETGPU_CX: case KETGPU_CY: slot = 6; break;
      case KETGPU_CZ: slot = 7; break;
      case KETGPU_CP: slot = 8; break;
      case KETGPU_CRX: case KETGPU_CRY: case KETGPU_CRZ: case KETGPU_CU: case KETGPU_CH: slot = 9; break;
      case KETGPU_SWAP: slot = 10; break;
      case KETGPU_CCX: slot = 11; break;
      case KETGPU_CSWAP: slot = 12; break;
      default: slot = 13; break;
    }
    f[20 + slot] += 1.f / 16.f;  // 20..33
  }
  for (int q : qs) {
    if (q < 8) f[34 + q] = 1.f;                    // 34..41
    if (q >= n - 4) f[42 + (n - 1 - q)] = 1.f;      // 42..45
  }
  f[46] = state <= 126e6 ? 1.f : 0.f;
  f[47] = 1.f;
}

void build_plan(Plan& plan, int n, const ketgpu_op* ops, uint64_t nops, const PlanOptions& opt) {
  plan.n = n;
  plan.precision = opt.precision;
  plan.ops.assign(ops, ops + nops);
  plan.passes.clear();
  uint64_t n_gates = 0;
  double predicted = 0;
  const size_t amp = opt.precision == KETGPU_C64 ? 8 : 16;
  // Split at structural ops: they are fusion barriers (simulator.cpp:496).
  std::vector<int> seg;
  auto flush = [&]() {
    if (seg.empty()) return;
    if (opt.fusion == KETGPU_FUSE_NONE) {
      // One kernel per gate, except that consecutive gates on qubits below
      // kRunBits are staged through shared memory as one pass.
      const int bits = std::min(n, kRunBits);
      size_t i = 0;
      while (i < seg.size()) {
        size_t j = i;
        while (j < seg.size() && j - i < (size_t)kRunMaxGates && (qubit_mask(ops[seg[j]]) >> bits) == 0) ++j;
        if (j - i >= 2) {
          emit_run(plan, ops, std::vector<int>(seg.begin() + i, seg.begin() + j));
          i = j;
        } else {
          emit_single(plan, ops[seg[i]], seg[i]);
          ++i;
        }
      }
    } else if (opt.fusion == KETGPU_FUSE_REFERENCE) {
      for (const Block& b : reference_blocks(ops, seg)) {
        if (b.gates.size() == 1) emit_single(plan, ops[b.gates[0]], b.gates[0]);
        else emit_fused(plan, n, ops, b, opt);
      }
    } else if (opt.fusion == KETGPU_FUSE_LEARNED && learned_model_attached()) {
      // Candidate partitions (greedy growth at k = 3..6); every block scored
      // fused and as its separate gates by the cost model in one batched
      // inference; the partition with the least predicted time wins, each
      // block taking its cheaper form.
      const int kmin_cand = std::min(3, std::max(1, opt.max_k));
      const int kmax_cap = std::max(kmin_cand, std::min(6, opt.max_k + 1));
      // per k: the greedy partition of least static cost over the program
      // order and the band orders (what FUSE_GREEDY would emit at that k)
      std::vector<std::vector<Block>> cands;
      for (int kc = kmin_cand; kc <= kmax_cap; ++kc) {
        PlanOptions ok = opt;
        ok.max_k = kc;
        cands.push_back(best_partition(n, ops, seg, ok));
      }
      std::vector<float> rows;
      float fr[kFeatures];
      // single-gate rows, one per gate of the segment
      std::vector<size_t> single_row(nops, 0);
      for (int gi : seg) {
        std::vector<int> q1(ops[gi].q, ops[gi].q + gate_arity(ops[gi].type));
        pass_features(n, opt.precision, {&ops[gi]}, q1, false, false, fr);
        single_row[gi] = rows.size() / kFeatures;
        rows.insert(rows.end(), fr, fr + kFeatures);
      }
      std::vector<std::vector<size_t>> fused_row(cands.size());
      for (size_t c = 0; c < cands.size(); ++c)
        for (const Block& b : cands[c]) {
          if (b.diag) {
            // A Diagonal pass streams the whole state once: scored as the
            // model's time of a dense one-qubit pass on the run's top qubit.
            ketgpu_op proxy{};
            proxy.type = KETGPU_U;
            proxy.nq = 1;
            proxy.q[0] = b.qubits.back();
            pass_features(n, opt.precision, {&proxy}, {proxy.q[0]}, false, false, fr);
            fused_row[c].push_back(rows.size() / kFeatures);
            rows.insert(rows.end(), fr, fr + kFeatures);
            continue;
          }
          std::vector<const ketgpu_op*> gs;
          for (int gi : b.gates) gs.push_back(&ops[gi]);
          pass_features(n, opt.precision, gs, b.qubits, true,
                        block_on_tensor_cores(n, (int)b.qubits.size(), opt), fr);
          fused_row[c].push_back(rows.size() / kFeatures);
          rows.insert(rows.end(), fr, fr + kFeatures);
        }
      std::vector<float> us;
      learned_predict(rows, us);
      size_t best = 0;
      double best_t = 1e300;
      std::vector<std::vector<char>> choice(cands.size());
      for (size_t c = 0; c < cands.size(); ++c) {
        double tot = 0;
        for (size_t bi = 0; bi < cands[c].size(); ++bi) {
          const Block& b = cands[c][bi];
          if (b.diag) {
            choice[c].push_back(2);
            tot += us[fused_row[c][bi]];
            continue;
          }
          double sep = 0;
          for (int gi : b.gates) sep += us[single_row[gi]];
          const double fu = us[fused_row[c][bi]];
          const bool fuse = b.gates.size() > 1 && fu < sep;
          choice[c].push_back(fuse ? 1 : 0);
          tot += fuse ? fu : sep;
        }
        if (tot < best_t) {
          best_t = tot;
          best = c;
        }
      }
      // The greedy plan (growth at max_k, static fuse rule), scored by the
      // same model: the learned choice replaces it only when the model
      // predicts a clear gain, so model error on near-equal plans cannot
      // make the learned plan slower than greedy.
      const size_t gk = (size_t)(std::max(kmin_cand, std::min(opt.max_k, kmax_cap)) - kmin_cand);
      double greedy_t = 0;
      std::vector<char> greedy_choice;
      for (size_t bi = 0; bi < cands[gk].size(); ++bi) {
        const Block& b = cands[gk][bi];
        char ch;
        if (b.diag) {
          ch = 2;
          greedy_t += us[fused_row[gk][bi]];
        } else {
          double sep = 0, frac = 0;
          for (int gi : b.gates) {
            sep += us[single_row[gi]];
            frac += gate_traffic_fraction(ops[gi]);
          }
          ch = b.gates.size() > 1 && fused_cost_static((int)b.qubits.size(), opt.precision, opt.tensor) < frac;
          greedy_t += ch ? us[fused_row[gk][bi]] : sep;
        }
        greedy_choice.push_back(ch);
      }
      if (!(best_t < (1.0 - kLearnedMargin) * greedy_t)) {
        best = gk;
        best_t = greedy_t;
        choice[gk] = greedy_choice;
      }
      predicted += best_t;
      for (size_t bi = 0; bi < cands[best].size(); ++bi) {
        const Block& b = cands[best][bi];
        if (choice[best][bi] == 2) emit_diagonal(plan, n, ops, b);
        else if (choice[best][bi]) emit_fused(plan, n, ops, b, opt);
        else
          for (int gi : b.gates) emit_single(plan, ops[gi], gi);
      }
    } else {
      // greedy growth over the program order and every band order; the
      // partition with the least static cost wins (the program order on ties)
      std::vector<Block> best = best_partition(n, ops, seg, opt);
      for (const Block& b : best) {
        if (b.diag) {
          emit_diagonal(plan, n, ops, b);
          continue;
        }
        if (b.gates.size() == 1) {
          emit_single(plan, ops[b.gates[0]], b.gates[0]);
          continue;
        }
        const int k = (int)b.qubits.size();
        double separate = 0;
        for (int gi : b.gates) separate += gate_traffic_fraction(ops[gi]);
        if (fused_cost_static(k, opt.precision, opt.tensor) < separate) {
          emit_fused(plan, n, ops, b, opt);
        } else {
          for (int gi : b.gates) emit_single(plan, ops[gi], gi);
        }
      }
    }
    seg.clear();
  };
  for (uint64_t i = 0; i < nops; ++i) {
    if (is_unitary(ops[i].type)) {
      seg.push_back((int)i);
      ++n_gates;
    } else {
      flush();
    }
  }
  flush();
  if (opt.fusion == KETGPU_FUSE_GREEDY || opt.fusion == KETGPU_FUSE_LEARNED) order_passes(plan, ops, n);
  for (uint64_t i = 0; i < nops && plan.finite; ++i)
    if (is_unitary(ops[i].type))
      for (double v : ops[i].p) plan.finite = plan.finite && std::isfinite(v);
  bool any_tensor = false;
  for (const Pass& p : plan.passes) any_tensor |= p.tensor;
  if ((opt.renormalize == 0 && any_tensor) || (opt.renormalize > 0 && !plan.passes.empty())) {
    Pass cap, res;
    cap.kind = PassKind::NormCapture;
    res.kind = PassKind::NormRestore;
    // a tensor-core block right before the restore sums the norm as it stores
    if (!plan.passes.empty() && plan.passes.back().kind == PassKind::Fused && plan.passes.back().tensor) {
      plan.passes.back().norm_out = true;
      res.norm_out = true;
    }
    plan.passes.insert(plan.passes.begin(), cap);
    plan.passes.push_back(res);
  }
  ketgpu_plan_stats& st = plan.stats;
  st = ketgpu_plan_stats{};
  st.n_gates = n_gates;
  st.n_passes = plan.passes.size();
  for (const Pass& p : plan.passes) {
    st.bytes += p.bytes(n, amp);
    if (p.kind == PassKind::Fused) {
      ++st.n_fused;
      if (p.tensor) ++st.n_tensor;
      st.flops += 8.0 * (double)(1 << p.k) * (double)(uint64_t{1} << n);
    }
  }
  st.predicted_us = predicted;
}

}  // namespace kb
