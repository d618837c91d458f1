// tables.cu -- the device tables of a plan (block matrices, tensor-core
// operands, diagonal phase tables), built on the device.
//
// ket multiplies the gates of a block into its matrix on the host
// (src/simulator.cpp:420-470).  Here a plan uploads its gates (96 bytes each)
// in one copy and one launch builds every table, a CTA each: for a block, its
// 2^k columns start as the identity in shared memory and the gates act on them
// in turn, in FP64, as they act on a state; the result is written in the form
// the block's kernel reads -- transposed FP64 or FP32, or the fp16 hi / lo
// images of the real embedding (build_tc_image's layout).  For a diagonal run
// it is the phase table of the low index bits.
// Bound: shared memory, two 16-byte accesses each way per pair and gate
// (about 0.5 us a gate at k = 6), all blocks at once; the host threads that
// built the matrices and images, and the copy of the images, took 2.9 ms for
// the 51 blocks of a 24-qubit circuit over the full gate mix (a call of 8.7 ms,
// now 5.2).
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <vector>

#include "internal.h"
#include "tc_layout.cuh"

namespace kb {
namespace {

enum TableKind : int32_t { kTable64 = 0, kTable32 = 1, kTableTc = 2, kTableDiag64 = 3, kTableDiag32 = 4 };

struct TableJob {
  int32_t kind, k;     // k: block qubits; diagonal: tabulated low bits
  uint64_t src;        // byte offset of its gates (diagonal: coefficients)
  uint64_t dst;        // byte offset of its table
  uint64_t count;      // gates; diagonal: FP64 coefficients to append to the table
  uint64_t pairs;      // diagonal: byte offset of the low pair terms, k x k
};

// A gate lowered onto its block's bits.
struct TableGate {
  int32_t kind;  // 0 pair, 1 phase
  int32_t mode;
  int32_t nfixed;
  int32_t fixed[3];
  uint32_t p0, p1;
  double2 m[4];
};

constexpr int kTableThreads = 256;
constexpr int kGateChunk = 32;

__device__ __forceinline__ double2 zmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 zmul_add(double2 a, double2 b, double2 c, double2 d) {
  return make_double2(a.x * b.x - a.y * b.y + (c.x * d.x - c.y * d.y), a.x * b.y + a.y * b.x + (c.x * d.y + c.y * d.x));
}

// exponent e with |v| in [2^(e-1), 2^e) (frexp's), v finite and nonzero
__device__ __forceinline__ int exponent_of(double v) {
  const int f = (int)((__double_as_longlong(v) >> 52) & 0x7ff);
  if (f) return f - 1022;
  return (int)((__double_as_longlong(v * 18014398509481984.0) >> 52) & 0x7ff) - 1022 - 54;  // subnormal: * 2^54
}

__device__ void build_block(const TableJob& jb, unsigned char* block, double2* v) {
  __shared__ TableGate gates[kGateChunk];
  __shared__ double wmax[kTableThreads / 32];
  const int tid = threadIdx.x, k = jb.k, dim = 1 << k;
  for (int i = tid; i < dim * dim; i += kTableThreads)  // v[c][r]
    v[i] = make_double2((i >> k) == (i & (dim - 1)) ? 1.0 : 0.0, 0.0);
  const TableGate* src = reinterpret_cast<const TableGate*>(block + jb.src);
  for (uint64_t g0 = 0; g0 < jb.count; g0 += kGateChunk) {
    const int cnt = (int)min((unsigned long long)kGateChunk, (unsigned long long)(jb.count - g0));
    __syncthreads();
    for (int i = tid; i < cnt * (int)(sizeof(TableGate) / 4); i += kTableThreads)
      reinterpret_cast<uint32_t*>(gates)[i] = reinterpret_cast<const uint32_t*>(src + g0)[i];
    __syncthreads();
    for (int gi = 0; gi < cnt; ++gi) {
      const TableGate& g = gates[gi];
      const int sh = k - g.nfixed;  // 2^sh pairs (or elements) a column
      for (int i = tid; i < dim << sh; i += kTableThreads) {
        uint32_t b = (uint32_t)(i & ((1 << sh) - 1));
        for (int j = 0; j < g.nfixed; ++j) {
          const int f = g.fixed[j];
          b = ((b >> f) << (f + 1)) | (b & ((1u << f) - 1));
        }
        double2* col = v + ((size_t)(i >> sh) << k);
        double2* x = col + (b | g.p0);
        if (g.kind == 1) {
          *x = zmul(g.m[0], *x);
          continue;
        }
        double2* y = col + (b | g.p1);
        const double2 a = *x, c = *y;
        if (g.mode == kPairSwap) {
          *x = c;
          *y = a;
        } else if (g.mode == kPairDiag) {
          *x = zmul(g.m[0], a);
          *y = zmul(g.m[3], c);
        } else {
          *x = zmul_add(g.m[0], a, g.m[1], c);
          *y = zmul_add(g.m[2], a, g.m[3], c);
        }
      }
      __syncthreads();
    }
  }
  __syncthreads();
  if (jb.kind == kTable64) {
    double2* out = reinterpret_cast<double2*>(block + jb.dst);
    for (int i = tid; i < dim * dim; i += kTableThreads) out[i] = v[i];
    return;
  }
  if (jb.kind == kTable32) {
    float2* out = reinterpret_cast<float2*>(block + jb.dst);
    for (int i = tid; i < dim * dim; i += kTableThreads) out[i] = make_float2((float)v[i].x, (float)v[i].y);
    return;
  }
  // tensor-core operand: scale 2^sb that brings the largest entry into
  // [2^14, 2^15), hi and lo images, sb
  double m = 0.0;
  for (int i = tid; i < dim * dim; i += kTableThreads) m = fmax(m, fmax(fabs(v[i].x), fabs(v[i].y)));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((tid & 31) == 0) wmax[tid >> 5] = m;
  __syncthreads();
  m = 0.0;
  for (int w = 0; w < kTableThreads / 32; ++w) m = fmax(m, wmax[w]);
  const int sb = m > 0.0 ? max(-24, min(24, 15 - exponent_of(m))) : 14;
  const double scale = __longlong_as_double((long long)(1023 + sb) << 52);
  const int N = 2 * dim, atoms = (2 * dim + 63) / 64;
  unsigned char* hi = block + jb.dst;
  unsigned char* lo = hi + (size_t)atoms * N * 128;
  // one 4-byte word (K entries 2c and 2c + 1) of row n at a time; whole atoms,
  // zeros beyond K
  for (int i = tid; i < N * atoms * 32; i += kTableThreads) {
    const int c = i & (atoms * 32 - 1), n = i / (atoms * 32), r = n >> 1;
    double a = 0.0, b = 0.0;
    if (c < dim) {
      const double2 z = v[((size_t)c << k) + r];
      a = scale * ((n & 1) ? z.y : z.x);
      b = scale * ((n & 1) ? z.x : -z.y);
    }
    const __half ha = __double2half(a), hb = __double2half(b);
    const __half la = __double2half(a - (double)__half2float(ha)), lb = __double2half(b - (double)__half2float(hb));
    const uint32_t off = sw128_offset_h(n, 2 * c, N);
    *reinterpret_cast<__half2*>(hi + off) = __halves2half2(ha, hb);
    *reinterpret_cast<__half2*>(lo + off) = __halves2half2(la, lb);
  }
  if (tid == 0) *reinterpret_cast<int32_t*>(lo + (size_t)atoms * N * 128) = sb;
}

// exp(i q(x)) for the 2^L low index patterns, q(x) the sum of the pair terms
// among x's set bits, then the coefficients as they are.
__device__ void build_diag(const TableJob& jb, unsigned char* block) {
  const int L = jb.k, n = 1 << L;
  const double* pairs = reinterpret_cast<const double*>(block + jb.pairs);
  for (int x = threadIdx.x; x < n; x += kTableThreads) {
    double q = 0.0;
    for (int j = 1; j < L; ++j)
      if ((x >> j) & 1)
        for (int i = 0; i < j; ++i)
          if ((x >> i) & 1) q += pairs[i * L + j];
    double s, c;
    sincos(q, &s, &c);
    if (jb.kind == kTableDiag64) reinterpret_cast<double2*>(block + jb.dst)[x] = make_double2(c, s);
    else reinterpret_cast<float2*>(block + jb.dst)[x] = make_float2((float)c, (float)s);
  }
  double* out = reinterpret_cast<double*>(block + jb.dst + ((uint64_t)n << (jb.kind == kTableDiag64 ? 4 : 3)));
  const double* prm = reinterpret_cast<const double*>(block + jb.src);
  for (uint64_t i = threadIdx.x; i < jb.count; i += kTableThreads) out[i] = prm[i];
}

__global__ void __launch_bounds__(kTableThreads) build_tables(unsigned char* block, uint64_t jobs) {
  extern __shared__ __align__(16) double2 table_matrix[];
  const TableJob jb = reinterpret_cast<const TableJob*>(block + jobs)[blockIdx.x];
  if (jb.kind >= kTableDiag64) build_diag(jb, block);
  else build_block(jb, block, table_matrix);
}

}  // namespace

// Device tables of a plan on `device` (current), once per plan: one block of
// memory, one copy, one launch, on `stream`; waited for unless the plan runs
// on that stream alone.
void upload_plan_tables(Plan& plan, int device, cudaStream_t stream, bool one_stream) {
  std::lock_guard<std::mutex> lk(plan.mu);
  if (plan.device == device) return;
  if (plan.device >= 0) fail(KETGPU_ERR_INVALID, "plan was prepared for another device");
  const bool c64 = plan.precision == KETGPU_C64;
  // [norm][tables][job records, gates, coefficients and run records: copied]
  std::vector<unsigned char> up;
  std::vector<TableJob> jobs;
  auto append = [&](const void* p, size_t bytes) -> size_t {
    while (up.size() % 16) up.push_back(0);
    const size_t at = up.size();
    const unsigned char* b = static_cast<const unsigned char*>(p);
    up.insert(up.end(), b, b + bytes);
    return at;
  };
  size_t tables = 0;
  auto place = [&](size_t bytes) -> size_t {
    const size_t at = tables;
    tables += (bytes + 255) / 256 * 256;
    return at;
  };
  for (const Pass& p : plan.passes)
    if (p.kind == PassKind::NormCapture && tables == 0) place(sizeof(double) * (2 + kNormBlocks));
  const bool norm = tables > 0;
  int max_k = 0;
  std::vector<TableGate> gates;
  std::vector<unsigned char> run;
  std::vector<double> prm;
  std::vector<size_t> run_at;  // SharedRun passes: offsets in the copied part
  for (Pass& p : plan.passes) {
    TableJob jb{};
    if (p.kind == PassKind::Fused) {
      gates.clear();
      for (const Pass& l : lower_block(plan.ops.data(), p.gates, p.qubits, p.k)) {
        TableGate g{};
        g.kind = l.kind == PassKind::Phase ? 1 : 0;
        g.mode = l.mode;
        g.nfixed = l.nfixed;
        for (int j = 0; j < 3; ++j) g.fixed[j] = l.fixed[j];
        g.p0 = (uint32_t)l.p0;
        g.p1 = (uint32_t)l.p1;
        for (int j = 0; j < 4; ++j) g.m[j] = make_double2(l.m[j].real(), l.m[j].imag());
        gates.push_back(g);
      }
      const size_t dim = size_t{1} << p.k;
      jb.kind = !c64 ? kTable64 : p.tensor ? kTableTc : kTable32;
      jb.k = p.k;
      jb.src = append(gates.data(), gates.size() * sizeof(TableGate));
      jb.count = gates.size();
      p.table = jb.dst = place(p.tensor ? tc_image_bytes(p.k) : dim * dim * (c64 ? 8 : 16));
      max_k = std::max(max_k, p.k);
    } else if (p.kind == PassKind::Diagonal) {
      const DiagPoly& poly = plan.diags[p.diag_index];
      const int L = std::min(plan.n, kDiagLowBits);
      jb.kind = c64 ? kTableDiag32 : kTableDiag64;
      jb.k = L;
      diag_coefficients(poly, plan.n, prm);
      jb.src = append(prm.data(), prm.size() * sizeof(double));
      jb.count = prm.size();
      std::vector<double> low((size_t)L * L);
      for (int i = 0; i < L; ++i)
        for (int j = 0; j < L; ++j) low[(size_t)i * L + j] = poly.b[(size_t)i * plan.n + j];
      jb.pairs = append(low.data(), low.size() * sizeof(double));
      p.table = jb.dst = place(((size_t{1} << L) * (c64 ? 8 : 16)) + prm.size() * sizeof(double));
    } else {
      if (p.kind == PassKind::SharedRun) {
        run_device_data(plan.runs[p.run_index], plan.precision, run);
        p.table = append(run.data(), run.size());
      }
      continue;
    }
    jobs.push_back(jb);
  }
  for (TableJob& jb : jobs) {
    jb.src += tables;
    jb.pairs += tables;
  }
  for (Pass& p : plan.passes)
    if (p.kind == PassKind::SharedRun) p.table += tables;
  const size_t jobs_at = tables + append(jobs.data(), jobs.size() * sizeof(TableJob));
  if (tables + up.size()) {
    DeviceBlock block(tables + up.size(), device, stream);
    if (!up.empty())
      KB_CUDA(cudaMemcpyAsync(static_cast<char*>(block.p) + tables, up.data(), up.size(), cudaMemcpyHostToDevice,
                              stream));
    if (!jobs.empty()) {
      const size_t smem = max_k ? sizeof(double2) << (2 * max_k) : 0;
      static OncePerDevice attr;
      attr(device, [] {
        KB_CUDA(cudaFuncSetAttribute(build_tables, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)(sizeof(double2) << 12)));
      });
      build_tables<<<(unsigned)jobs.size(), kTableThreads, smem, stream>>>(static_cast<unsigned char*>(block.p),
                                                                            jobs_at);
      count_launch();
      KB_CUDA(cudaGetLastError());
    }
    if (!one_stream) KB_CUDA(cudaStreamSynchronize(stream));
    plan.block = std::move(block);
  }
  plan.d_norm = norm ? static_cast<double*>(plan.block.p) : nullptr;
  plan.device = device;
}

}  // namespace kb
