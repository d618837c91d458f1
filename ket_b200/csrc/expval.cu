// expval.cu -- Pauli-string expectations of a state, all terms of a sum at
// once (ket::expval, src/observable.cpp:18-91).
//
// Term t has a flip mask f, a sign mask s and a phase i^q:
//     <P> = sum_x Re(i^q (-1)^|x & s| psi[x] conj(psi[x ^ f])).
// x and x ^ f contribute the same value, so a term with f != 0 needs half of
// the indices, each pair of amplitudes once.
//
// Flips (f != 0).  The flips of up to five terms that are linearly independent
// over GF(2) generate cosets of 2^R indices (R <= 5).  A thread takes one
// coset, 2^R amplitudes, converts them to FP64 once and holds them in
// registers; in the coset's coordinates each term's flip is one coordinate
// bit, so every pair of every term of the group is in the thread's registers:
// one read of the state serves R flips (a kernel that read the partner of
// every amplitude for every term moved the state once a term).  A flip has up
// to two terms in a group (XX and YY on the same pair share it).  Signs are
// linear in the coset's coordinates: one parity a thread and term, then a
// signed tree over the pairs.  The next coset's copies (cp.async into the
// thread's own shared-memory slots) run under the arithmetic.
// Bound: HBM, ceil(flips / R) reads of the state, next to 3 FP64 operations a
// pair and term and 2 FP32 -> FP64 conversions an amplitude and group.
// Measured, 64 random strings on 27 qubits, complex64: 2.61 ms (13 groups of
// 200 us; one read of the state takes 164), against 32.4 ms for a kernel that
// read every partner for every term; without the copies under the arithmetic
// 3.64 ms, R = 4 4.6 ms.  complex128, 32 strings on 26 qubits: 1.15 ms, seven
// reads of the state at 6.5 TB/s.
//
// Diagonal terms (f = 0).  A CTA takes 4096 consecutive probabilities and
// forms their Walsh-Hadamard transform (three radix-16 steps in registers);
// coefficient s mod 4096 of it, with the sign of the chunk's own index, is the
// chunk's sum for the term of sign mask s.  12 additions an amplitude whatever
// the number of terms; one read of the state (26 qubits, complex64: 0.19 ms).
//
// Everything is FP64 and in a fixed order: per thread, per block, and over the
// blocks' partials in index order.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <vector>

#include "internal.h"

namespace kb {
namespace {

constexpr int kMaxR = 5;       // flips a group
constexpr int kPerFlip = 2;    // terms of a flip a group
constexpr int kFlipThreads = 128;

struct FlipGroup {
  uint64_t gen[kMaxR];
  uint64_t s[kMaxR * kPerFlip];
  int piv[kMaxR];                       // pivot bits, ascending
  int out[kMaxR * kPerFlip];            // term, -1: none
  unsigned char sg[kMaxR * kPerFlip];   // bit j: parity(gen[j] & s)
  unsigned char odd[kMaxR * kPerFlip];  // q odd: imaginary part
};

struct DiagTerm {
  uint64_t s;
  int out;
  int pad;
};

struct TermFinish {
  double scale;
  int blocks;
  int pad;
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// Signed sum over the coset's pairs along coordinate I: the pair (m, m | 2^I)
// counts with the product of sg[j] over the set bits j of m.
template <int R, int I, bool ODD, int LV, int M>
__device__ __forceinline__ double pair_tree(const double* re, const double* im, const double* sg) {
  if constexpr (LV < 0) {
    constexpr int P = M | (1 << I);
    if constexpr (ODD) return im[M] * re[P] - re[M] * im[P];
    else return re[M] * re[P] + im[M] * im[P];
  } else if constexpr (LV == I) {
    return pair_tree<R, I, ODD, LV - 1, M>(re, im, sg);
  } else {
    const double a = pair_tree<R, I, ODD, LV - 1, M>(re, im, sg);
    const double b = pair_tree<R, I, ODD, LV - 1, M | (1 << LV)>(re, im, sg);
    return fma(sg[LV], b, a);
  }
}

template <int R, int I>
__device__ __forceinline__ void flip_terms(const FlipGroup& g, uint64_t x0, const double* re, const double* im,
                                           double* acc) {
  if constexpr (I < R) {
#pragma unroll
    for (int j = 0; j < kPerFlip; ++j) {
      constexpr int T = I * kPerFlip;
      if (g.out[T + j] >= 0) {
        double sg[R];
#pragma unroll
        for (int b = 0; b < R; ++b) sg[b] = (g.sg[T + j] >> b) & 1 ? -1.0 : 1.0;
        const double v = g.odd[T + j] ? pair_tree<R, I, true, R - 1, 0>(re, im, sg)
                                      : pair_tree<R, I, false, R - 1, 0>(re, im, sg);
        acc[(T + j) * kFlipThreads] += __popcll(x0 & g.s[T + j]) & 1 ? -v : v;
      }
    }
    flip_terms<R, I + 1>(g, x0, re, im, acc);
  }
}

template <typename T, int R>
__global__ void __launch_bounds__(kFlipThreads, R == 5 ? 3 : 4)
    expval_flips(const T* __restrict__ s, int n, const FlipGroup* __restrict__ groups, double* __restrict__ part,
                 uint64_t stride) {
  __shared__ FlipGroup g;
  __shared__ double sh[kFlipThreads / 32][kMaxR * kPerFlip];
  for (int i = threadIdx.x; i < (int)(sizeof(FlipGroup) / 4); i += kFlipThreads)
    reinterpret_cast<uint32_t*>(&g)[i] = reinterpret_cast<const uint32_t*>(groups + blockIdx.y)[i];
  __syncthreads();
  // the thread's sums, in shared memory: its registers hold the coset
  __shared__ double sums[R * kPerFlip * kFlipThreads];
  double* acc = sums + threadIdx.x;
#pragma unroll
  for (int t = 0; t < R * kPerFlip; ++t) acc[t * kFlipThreads] = 0.0;
  uint64_t gen[R];
#pragma unroll
  for (int j = 0; j < R; ++j) gen[j] = g.gen[j];
  // The next coset's copies into the thread's own shared-memory slots are in
  // flight while this one is worked on.
  extern __shared__ __align__(16) unsigned char flip_smem[];
  T* slots = reinterpret_cast<T*>(flip_smem) + threadIdx.x;
  const uint32_t slot_addr = (uint32_t)__cvta_generic_to_shared(slots);
  const uint64_t count = uint64_t{1} << (n - R), step = (uint64_t)gridDim.x * kFlipThreads;
  auto member = [&](uint64_t i) -> uint64_t {  // the coset's member with zero pivot bits
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const int f = g.piv[j];
      i = ((i >> f) << (f + 1)) | (i & ((uint64_t{1} << f) - 1));
    }
    return i;
  };
  auto fetch = [&](uint64_t x0) {
#pragma unroll
    for (int m = 0; m < (1 << R); ++m) {
      uint64_t c = 0;
#pragma unroll
      for (int j = 0; j < R; ++j)
        if ((m >> j) & 1) c ^= gen[j];
      if constexpr (sizeof(T) == 8)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(slot_addr + m * kFlipThreads * 8),
                     "l"(s + (x0 ^ c))
                     : "memory");
      else
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(slot_addr + m * kFlipThreads * 16),
                     "l"(s + (x0 ^ c))
                     : "memory");
    }
  };
  uint64_t i = (uint64_t)blockIdx.x * kFlipThreads + threadIdx.x;
  uint64_t next = member(i);
  if (i < count) fetch(next);
  for (; i < count; i += step) {
    const uint64_t x0 = next;
    asm volatile("cp.async.wait_all;" ::: "memory");
    double re[1 << R], im[1 << R];
#pragma unroll
    for (int m = 0; m < (1 << R); ++m) {
      const T v = slots[m * kFlipThreads];
      re[m] = (double)v.x;
      im[m] = (double)v.y;
    }
    next = member(i + step);
    if (i + step < count) fetch(next);
    flip_terms<R, 0>(g, x0, re, im, acc);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int t = 0; t < R * kPerFlip; ++t) {
    const double r = warp_sum(acc[t * kFlipThreads]);
    if (lane == 0) sh[warp][t] = r;
  }
  __syncthreads();
  if (threadIdx.x < R * kPerFlip && g.out[threadIdx.x] >= 0) {
    double r = 0.0;
    for (int w = 0; w < kFlipThreads / 32; ++w) r += sh[w][threadIdx.x];
    part[(uint64_t)g.out[threadIdx.x] * stride + blockIdx.x] = r;
  }
}

constexpr int kWalshBits = 12;
constexpr int kWalshThreads = 256;
constexpr int kWalshTerms = 4;  // terms a thread; 1024 a CTA

__device__ __forceinline__ void walsh16(double* v) {
#pragma unroll
  for (int h = 1; h < 16; h <<= 1)
#pragma unroll
    for (int i = 0; i < 16; ++i)
      if (!(i & h)) {
        const double a = v[i], b = v[i | h];
        v[i] = a + b;
        v[i | h] = a - b;
      }
}

template <typename T>
__global__ void __launch_bounds__(kWalshThreads, 2)
    expval_diagonal(const T* __restrict__ s, uint64_t dim, uint64_t n_chunks, const DiagTerm* __restrict__ terms,
                    int n_terms, double* __restrict__ part, uint64_t stride) {
  __shared__ double w[(1 << kWalshBits) / 16 * 17];  // 17 doubles a row of 16
  const int tid = threadIdx.x;
  auto at = [&](int e) -> double& { return w[e + (e >> 4)]; };
  uint64_t mask[kWalshTerms];
  int out[kWalshTerms];
  double acc[kWalshTerms];
#pragma unroll
  for (int k = 0; k < kWalshTerms; ++k) {
    const int t = (blockIdx.y * kWalshTerms + k) * kWalshThreads + tid;
    out[k] = t < n_terms ? terms[t].out : -1;
    mask[k] = t < n_terms ? terms[t].s : 0;
    acc[k] = 0.0;
  }
  T a[16];  // the next chunk's amplitudes, loaded while this one is transformed
  auto fetch = [&](uint64_t c) {
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const uint64_t x = (c << kWalshBits) + tid + j * kWalshThreads;
      a[j].x = a[j].y = 0;
      if (x < dim) a[j] = s[x];
    }
  };
  fetch(blockIdx.x);
  for (uint64_t c = blockIdx.x; c < n_chunks; c += gridDim.x) {
    const uint64_t base = c << kWalshBits;
    double v[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = (double)a[j].x * (double)a[j].x + (double)a[j].y * (double)a[j].y;
    fetch(c + gridDim.x);
    walsh16(v);  // bits 8..11
    __syncthreads();  // the previous chunk's coefficients have been read
#pragma unroll
    for (int j = 0; j < 16; ++j) at(tid + j * kWalshThreads) = v[j];
    __syncthreads();
    const int mid = (tid & 15) | ((tid >> 4) << 8);
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = at(mid | (j << 4));
    walsh16(v);  // bits 4..7
#pragma unroll
    for (int j = 0; j < 16; ++j) at(mid | (j << 4)) = v[j];
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = at((tid << 4) | j);
    walsh16(v);  // bits 0..3
#pragma unroll
    for (int j = 0; j < 16; ++j) at((tid << 4) | j) = v[j];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kWalshTerms; ++k)
      if (out[k] >= 0) {
        const double r = at((int)(mask[k] & ((1u << kWalshBits) - 1)));
        acc[k] += __popcll(base & mask[k]) & 1 ? -r : r;
      }
  }
#pragma unroll
  for (int k = 0; k < kWalshTerms; ++k)
    if (out[k] >= 0) part[(uint64_t)out[k] * stride + blockIdx.x] = acc[k];
}

// One block a term: its partials in a fixed tree, times its scale.
__global__ void expval_finish(const double* __restrict__ part, uint64_t stride, const TermFinish* __restrict__ fin,
                              double* __restrict__ out) {
  __shared__ double sh[8];
  const TermFinish f = fin[blockIdx.x];
  const double* p = part + (uint64_t)blockIdx.x * stride;
  double acc = 0.0;
  for (int i = threadIdx.x; i < f.blocks; i += blockDim.x) acc += p[i];
  acc = warp_sum(acc);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double r = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) r += sh[w];
    out[blockIdx.x] = r * f.scale;
  }
}

template <typename T, int R>
void launch_flips_r(dim3 grid, int device, cudaStream_t st, const T* s, int n, const FlipGroup* g, double* part,
                    uint64_t stride) {
  constexpr int smem = (int)sizeof(T) * kFlipThreads << R;
  if constexpr (smem > 16 * 1024) {
    static OncePerDevice attr;
    attr(device, [] {
      KB_CUDA(cudaFuncSetAttribute(expval_flips<T, R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)sizeof(T) * kFlipThreads << R));
    });
  }
  expval_flips<T, R><<<grid, kFlipThreads, smem, st>>>(s, n, g, part, stride);
}

template <typename T>
void launch_flips(int r, dim3 grid, int device, cudaStream_t st, const T* s, int n, const FlipGroup* g, double* part,
                  uint64_t stride) {
  switch (r) {
    case 1: launch_flips_r<T, 1>(grid, device, st, s, n, g, part, stride); break;
    case 2: launch_flips_r<T, 2>(grid, device, st, s, n, g, part, stride); break;
    case 3: launch_flips_r<T, 3>(grid, device, st, s, n, g, part, stride); break;
    case 4: launch_flips_r<T, 4>(grid, device, st, s, n, g, part, stride); break;
    default: launch_flips_r<T, 5>(grid, device, st, s, n, g, part, stride); break;
  }
}

// Independent flips of one group, reduced: basis[i] has its highest bit
// cleared in no earlier element (echelon by highest bit).
struct Echelon {
  uint64_t row[kMaxR];
  int count = 0;
  uint64_t reduce(uint64_t v) const {
    for (int i = 0; i < count; ++i)
      if ((v ^ row[i]) < v) v ^= row[i];
    return v;
  }
  bool add(uint64_t v) {
    v = reduce(v);
    if (!v) return false;
    int i = count++;
    for (; i > 0 && row[i - 1] < v; --i) row[i] = row[i - 1];  // descending
    row[i] = v;
    return true;
  }
};

// Flips a group holds.  A wider group reads the state less often but has
// fewer threads (2^(n - R)); below 2^17 of them the chip is not filled, and
// the state is in L2 anyway (14 qubits, 55 terms of a chain: 119 us a call,
// nearly all of it the call itself; 764 us with a finishing launch a term).
int flips_per_group(int n) { return std::clamp(n - 17, 1, std::min(kMaxR, std::max(n, 1))); }

}  // namespace

void expval_terms(const State& st, const std::vector<uint64_t>& flip, const std::vector<uint64_t>& sign,
                  const std::vector<int>& phase, double* out) {
  const int T = (int)flip.size();
  if (T == 0) return;
  const int n = st.n, r = flips_per_group(n);
  std::vector<FlipGroup> groups;
  std::vector<Echelon> bases;
  std::vector<int> gens;  // generators of each group
  std::vector<DiagTerm> diag;
  std::vector<TermFinish> fin(T);
  // terms in order of their flips, so that terms of one flip meet
  std::vector<int> order(T);
  for (int t = 0; t < T; ++t) order[t] = t;
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return flip[a] < flip[b]; });
  size_t open = 0;  // groups before it are full
  uint64_t last_flip = 0;  // the flip placed last, and its group
  size_t last = 0;
  for (int i = 0; i < T;) {
    const uint64_t f = flip[order[i]];
    if (!f) {
      const int t = order[i++];
      diag.push_back({sign[t], t, 0});
      fin[t].scale = 1.0;  // no X or Y: no factor i
      continue;
    }
    int cnt = 1;
    while (cnt < kPerFlip && i + cnt < T && flip[order[i + cnt]] == f) ++cnt;
    while (open < groups.size() && gens[open] == r) ++open;
    // the groups up to the last one of this flip hold it, span it or are full
    size_t gi = f == last_flip ? std::max(open, last + 1) : open;
    for (; gi < groups.size(); ++gi)
      if (gens[gi] < r && bases[gi].reduce(f)) break;
    if (gi == groups.size()) {
      groups.emplace_back();
      std::memset(&groups.back(), 0, sizeof(FlipGroup));
      std::fill(groups.back().out, groups.back().out + kMaxR * kPerFlip, -1);
      bases.emplace_back();
      gens.push_back(0);
    }
    last_flip = f;
    last = gi;
    bases[gi].add(f);
    FlipGroup& g = groups[gi];
    const int c = gens[gi]++;
    g.gen[c] = f;
    for (int j = 0; j < cnt; ++j) {
      const int t = order[i + j], slot = c * kPerFlip + j;
      g.out[slot] = t;
      g.s[slot] = sign[t];
      g.odd[slot] = (unsigned char)(phase[t] & 1);
      fin[t].scale = (phase[t] == 0 || phase[t] == 3) ? 2.0 : -2.0;
    }
    i += cnt;
  }
  for (size_t gi = 0; gi < groups.size(); ++gi) {
    FlipGroup& g = groups[gi];
    for (int q = n - 1; q >= 0 && gens[gi] < r; --q)  // fill up with single-bit flips without terms
      if (bases[gi].add(uint64_t{1} << q)) g.gen[gens[gi]++] = uint64_t{1} << q;
    for (int j = 0; j < r; ++j) g.piv[j] = 63 - __builtin_clzll(bases[gi].row[r - 1 - j]);
    for (int slot = 0; slot < r * kPerFlip; ++slot)
      for (int j = 0; j < r; ++j)
        if (__builtin_popcountll(g.gen[j] & g.s[slot]) & 1) g.sg[slot] |= (unsigned char)(1 << j);
  }
  const uint64_t n_chunks = st.dim() > (uint64_t{1} << kWalshBits) ? st.dim() >> kWalshBits : 1;
  const uint64_t cosets = uint64_t{1} << (n >= r ? n - r : 0);
  const uint64_t need = (cosets + kFlipThreads - 1) / kFlipThreads;
  // eight CTAs an SM in all, each group an equal share of them (one resident
  // wave of CTAs was no better: 2.61 ms for 64 strings at 27 qubits both ways,
  // and 1.26 against 1.15 ms for 32 strings of a 26-qubit complex128 state)
  const uint64_t share = groups.empty() ? 1 : std::max<uint64_t>(1, 148 * 8 / groups.size());
  const int gx = (int)std::min(need, share), gd = (int)std::min<uint64_t>(n_chunks, 148 * 2);
  const uint64_t stride = (uint64_t)std::max(gx, diag.empty() ? 1 : gd);
  for (int t = 0; t < T; ++t) fin[t].blocks = gx;
  for (const DiagTerm& d : diag) fin[d.out].blocks = gd;
  const size_t b_groups = groups.size() * sizeof(FlipGroup), b_diag = diag.size() * sizeof(DiagTerm),
               b_fin = fin.size() * sizeof(TermFinish);
  const size_t meta = b_groups + b_diag + b_fin;
  StreamScratch sc(meta + sizeof(double) * (stride * T + T), st.device, st.stream);
  char* base = static_cast<char*>(sc.p);
  std::vector<char> host(meta);
  if (b_groups) std::memcpy(host.data(), groups.data(), b_groups);
  if (b_diag) std::memcpy(host.data() + b_groups, diag.data(), b_diag);
  std::memcpy(host.data() + b_groups + b_diag, fin.data(), b_fin);
  KB_CUDA(cudaMemcpyAsync(base, host.data(), meta, cudaMemcpyHostToDevice, st.stream));
  const FlipGroup* d_groups = reinterpret_cast<const FlipGroup*>(base);
  const DiagTerm* d_diag = reinterpret_cast<const DiagTerm*>(base + b_groups);
  const TermFinish* d_fin = reinterpret_cast<const TermFinish*>(base + b_groups + b_diag);
  double* d_part = reinterpret_cast<double*>(base + meta);
  double* d_out = d_part + stride * T;
  static_assert(sizeof(FlipGroup) % 8 == 0 && sizeof(DiagTerm) % 8 == 0 && sizeof(TermFinish) % 8 == 0, "alignment");
  constexpr size_t kMaxY = 65535;
  for (size_t y = 0; y < groups.size(); y += kMaxY) {
    const dim3 grid(gx, (unsigned)std::min(kMaxY, groups.size() - y));
    if (st.precision == KETGPU_C64)
      launch_flips(r, grid, st.device, st.stream, static_cast<const float2*>(st.amps), n, d_groups + y, d_part, stride);
    else
      launch_flips(r, grid, st.device, st.stream, static_cast<const double2*>(st.amps), n, d_groups + y, d_part, stride);
    count_launch();
  }
  if (!diag.empty()) {
    constexpr int kPerCta = kWalshTerms * kWalshThreads;
    const dim3 grid(gd, (unsigned)((diag.size() + kPerCta - 1) / kPerCta));
    if (st.precision == KETGPU_C64)
      expval_diagonal<float2><<<grid, kWalshThreads, 0, st.stream>>>(static_cast<const float2*>(st.amps), st.dim(),
                                                                     n_chunks, d_diag, (int)diag.size(), d_part,
                                                                     stride);
    else
      expval_diagonal<double2><<<grid, kWalshThreads, 0, st.stream>>>(static_cast<const double2*>(st.amps), st.dim(),
                                                                      n_chunks, d_diag, (int)diag.size(), d_part,
                                                                      stride);
    count_launch();
  }
  expval_finish<<<T, 128, 0, st.stream>>>(d_part, stride, d_fin, d_out);
  count_launch();
  KB_CUDA(cudaGetLastError());
  KB_CUDA(cudaMemcpyAsync(out, d_out, sizeof(double) * T, cudaMemcpyDeviceToHost, st.stream));
  KB_CUDA(cudaStreamSynchronize(st.stream));
}

}  // namespace kb
