// adjoint.cu -- reverse-sweep (adjoint) gradients of <psi(theta)|H|psi(theta)>
// for a batch of parameter sets, H a Pauli sum.
//
// No ket counterpart: ket evaluates ket::expval(run(circuit), PauliSum)
// (src/observable.cpp:85-91) and has no derivatives.  The algebra follows
// ket's gate matrices (src/simulator.cpp:73-89 for Rx/Ry/Rz, :166-189 for the
// controlled rotations, :322-324 for CP) and Pauli actions
// (src/observable.cpp:68-118):
//   forward   psi_N = U_N ... U_1 |0>, checkpoints at layer boundaries
//   lambda    lambda = H psi_N,   <H> = Re <psi_N|lambda>
//   reverse   for i = N..1:  g_i = Im <lambda|G_i|psi_i>  (U_i = exp(-i t G_i / 2))
//                            psi <- U_i^dag psi, lambda <- U_i^dag lambda
// For CP(t) = diag(1,1,1,e^{it}) the term is -2 Im <lambda|P11|psi>.
// Three forms: up to 11 qubits one CTA a parameter set holds both states and
// runs everything in one launch (adjoint_resident); larger states go tile by
// tile, a block of gates a pass (tile_sweep and its compiled form); and one
// kernel per gate, on request, does the inner-product partial sums (FP64) and
// the two inverse applications in a single pass over psi and lambda.  All
// parameter sets of a chunk share every launch.  Layers are the
// barrier-delimited runs of ops; with checkpoint_every = m the forward state
// is stored every m layers and the reverse sweep restarts psi from it, so
// the uncomputation error does not accumulate across segments.
#include <cuda_runtime.h>
#include <dlfcn.h>

#include <algorithm>
#include <cstdio>
#include <map>
#include <mutex>
#include <cmath>
#include <cstring>
#include <memory>
#include <queue>
#include <string>
#include <type_traits>
#include <utility>
#include <vector>

#include "internal.h"
#include "adj_tile.cuh"

#define KB_API extern "C" __attribute__((visibility("default")))

namespace kb {
State* create_state(int n, int precision);
void destroy_state(State* s);

namespace {

template <typename R>
struct C2T;
template <>
struct C2T<float> {
  using T = float2;
};
template <>
struct C2T<double> {
  using T = double2;
};

constexpr int kAThreads = 256;

struct GateGeom {
  uint64_t count;  // pairs (or phase elements) per state
  uint64_t p0, p1;
  int fixed[3];
  int nfixed;
  int kind;   // 0 pair general, 1 pair swap, 2 phase
  int gen;    // generator for the gradient: 0 none, 1 X, 2 Y, 3 Z, 4 P11 (phase)
  int pslot;  // gradient slot (parameter index) or -1
};

__device__ __forceinline__ uint64_t spread3(uint64_t i, const int* fixed, int nfixed) {
#pragma unroll
  for (int j = 0; j < 3; ++j)
    if (j < nfixed) {
      const int f = fixed[j];
      i = ((i >> f) << (f + 1)) | (i & ((uint64_t{1} << f) - 1));
    }
  return i;
}

// Forward application of one gate to every state of the chunk: mats holds a
// 2x2 (or the phase in slot 0) per state, FP64 interleaved.
template <typename R>
__global__ void fwd_gate(typename C2T<R>::T* __restrict__ states, uint64_t dim, GateGeom g,
                         const double* __restrict__ mats) {
  using T = typename C2T<R>::T;
  T* s = states + (uint64_t)blockIdx.y * dim;
  const double* m = mats + (size_t)blockIdx.y * 8;
  const R m0r = (R)m[0], m0i = (R)m[1], m1r = (R)m[2], m1i = (R)m[3];
  const R m2r = (R)m[4], m2i = (R)m[5], m3r = (R)m[6], m3i = (R)m[7];
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < g.count;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t b = spread3(i, g.fixed, g.nfixed);
    if (g.kind == 2) {
      const T a = s[b | g.p0];
      T r;
      r.x = m0r * a.x - m0i * a.y;
      r.y = m0r * a.y + m0i * a.x;
      s[b | g.p0] = r;
      continue;
    }
    const T a = s[b | g.p0], c = s[b | g.p1];
    if (g.kind == 1) {
      s[b | g.p0] = c;
      s[b | g.p1] = a;
      continue;
    }
    T x, y;
    x.x = m0r * a.x - m0i * a.y + m1r * c.x - m1i * c.y;
    x.y = m0r * a.y + m0i * a.x + m1r * c.y + m1i * c.x;
    y.x = m2r * a.x - m2i * a.y + m3r * c.x - m3i * c.y;
    y.y = m2r * a.y + m2i * a.x + m3r * c.y + m3i * c.x;
    s[b | g.p0] = x;
    s[b | g.p1] = y;
  }
}

// Reverse step: partial Im <lambda|G|psi> (FP64) for this gate, then
// psi <- U^dag psi and lambda <- U^dag lambda.  mats holds U (not U^dag).
template <typename R>
__global__ void __launch_bounds__(kAThreads)
    rev_gate(typename C2T<R>::T* __restrict__ psi, typename C2T<R>::T* __restrict__ lam, uint64_t dim, GateGeom g,
             const double* __restrict__ mats, double* __restrict__ partial /* [set][blocks] */) {
  using T = typename C2T<R>::T;
  __shared__ double sh[32];
  T* s = psi + (uint64_t)blockIdx.y * dim;
  T* l = lam + (uint64_t)blockIdx.y * dim;
  const double* m = mats + (size_t)blockIdx.y * 8;
  // U^dag entries
  const R d0r = (R)m[0], d0i = (R)-m[1], d1r = (R)m[4], d1i = (R)-m[5];
  const R d2r = (R)m[2], d2i = (R)-m[3], d3r = (R)m[6], d3i = (R)-m[7];
  double acc = 0.0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < g.count;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t b = spread3(i, g.fixed, g.nfixed);
    if (g.kind == 2) {
      const T a = s[b | g.p0], lv = l[b | g.p0];
      if (g.gen == 4) acc += (double)lv.x * (double)a.y - (double)lv.y * (double)a.x;  // Im(conj(l) a)
      T r, q;
      r.x = d0r * a.x - d0i * a.y;
      r.y = d0r * a.y + d0i * a.x;
      q.x = d0r * lv.x - d0i * lv.y;
      q.y = d0r * lv.y + d0i * lv.x;
      s[b | g.p0] = r;
      l[b | g.p0] = q;
      continue;
    }
    const T a0 = s[b | g.p0], a1 = s[b | g.p1];
    const T l0 = l[b | g.p0], l1 = l[b | g.p1];
    if (g.gen) {
      // G psi restricted to the pair
      double g0r, g0i, g1r, g1i;
      if (g.gen == 1) {  // X
        g0r = a1.x; g0i = a1.y; g1r = a0.x; g1i = a0.y;
      } else if (g.gen == 2) {  // Y: (-i a1, i a0)
        g0r = a1.y; g0i = -(double)a1.x; g1r = -(double)a0.y; g1i = a0.x;
      } else {  // Z
        g0r = a0.x; g0i = a0.y; g1r = -(double)a1.x; g1i = -(double)a1.y;
      }
      // Im(conj(l0) g0 + conj(l1) g1)
      acc += (double)l0.x * g0i - (double)l0.y * g0r + (double)l1.x * g1i - (double)l1.y * g1r;
    }
    if (g.kind == 1) {
      s[b | g.p0] = a1;
      s[b | g.p1] = a0;
      l[b | g.p0] = l1;
      l[b | g.p1] = l0;
      continue;
    }
    T x, y;
    x.x = d0r * a0.x - d0i * a0.y + d1r * a1.x - d1i * a1.y;
    x.y = d0r * a0.y + d0i * a0.x + d1r * a1.y + d1i * a1.x;
    y.x = d2r * a0.x - d2i * a0.y + d3r * a1.x - d3i * a1.y;
    y.y = d2r * a0.y + d2i * a0.x + d3r * a1.y + d3i * a1.x;
    s[b | g.p0] = x;
    s[b | g.p1] = y;
    x.x = d0r * l0.x - d0i * l0.y + d1r * l1.x - d1i * l1.y;
    x.y = d0r * l0.y + d0i * l0.x + d1r * l1.y + d1i * l1.x;
    y.x = d2r * l0.x - d2i * l0.y + d3r * l1.x - d3i * l1.y;
    y.y = d2r * l0.y + d2i * l0.x + d3r * l1.y + d3i * l1.x;
    l[b | g.p0] = x;
    l[b | g.p1] = y;
  }
  if (g.gen == 0) return;
  // fixed-order block reduction
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if (lane == 0) sh[warp] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += sh[w];
    partial[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = t;
  }
}

// lambda = H psi for every state of the chunk (FP64 accumulation per
// amplitude), and per-block partials of Re <psi|lambda>.
template <typename R>
__global__ void __launch_bounds__(kAThreads)
    ham_apply(const typename C2T<R>::T* __restrict__ psi, typename C2T<R>::T* __restrict__ lam, uint64_t dim,
              const uint64_t* __restrict__ flips, const uint64_t* __restrict__ signs, const int* __restrict__ qs,
              const double* __restrict__ coeffs, int nterms, double* __restrict__ partial) {
  using T = typename C2T<R>::T;
  __shared__ double sh[32];
  const T* s = psi + (uint64_t)blockIdx.y * dim;
  T* l = lam + (uint64_t)blockIdx.y * dim;
  double e = 0.0;
  for (uint64_t y = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; y < dim;
       y += (uint64_t)gridDim.x * blockDim.x) {
    double re = 0.0, im = 0.0;
    for (int t = 0; t < nterms; ++t) {
      const uint64_t x = y ^ flips[t];
      const T a = s[x];
      // phase i^q times (-1)^popcount(x & sign)
      double ar = a.x, ai = a.y, vr, vi;
      switch (qs[t]) {
        case 0: vr = ar; vi = ai; break;
        case 1: vr = -ai; vi = ar; break;
        case 2: vr = -ar; vi = -ai; break;
        default: vr = ai; vi = -ar; break;
      }
      const double c = (__popcll(x & signs[t]) & 1) ? -coeffs[t] : coeffs[t];
      re += c * vr;
      im += c * vi;
    }
    T out;
    out.x = (R)re;
    out.y = (R)im;
    l[y] = out;
    const T p = s[y];
    e += (double)p.x * re + (double)p.y * im;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) e += __shfl_down_sync(0xffffffffu, e, o);
  if (lane == 0) sh[warp] = e;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += sh[w];
    partial[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = t;
  }
}

// lambda = H psi, split by the top qubit for states larger than L2.  A Pauli
// term maps output half h to source half h ^ (flip's top bit), so the terms
// are grouped by that bit and each output half is built in two passes: first
// from the terms that read the same half, then (adding to lambda) from those
// that read the other half.  Each pass gathers from one half (67 MB at 24
// qubits, complex64), which stays in L2 while the pass's terms revisit it.
// The grid (CTAs per set x sets) covers about one set at a time.  The last
// pass of a half adds Re <psi|lambda> over it into per-CTA partials.
//
// What bounds it is the work per term and amplitude, not the gathers (L2 at a
// quarter of its rate), so that is cut to the two conversions and two FP64
// multiply-adds it needs: a thread takes the outputs of a whole 16-byte word
// (two of complex64) from one 16-byte load a term; i^q c is real or
// imaginary, and terms are sorted by that and by whether they swap the word's
// halves; a term's sign on output y is the parity of y & sign, linear in y's
// bits, so it is the thread's own bit (a mask of 32 terms, made once) XOR that
// of the tile's base (a ballot per 32 terms and tile).
// 64 terms, 24 qubits, complex64: 1.69 ms for two sets, against 3.44 with one output a
// thread, two POPC and a complex coefficient a term.
constexpr int kHamSmemTerms = 1024;
struct HamTerm {
  uint64_t flip, sign;
  double c0, c1;  // coefficient for the outputs of the word (their own signs in)
};
struct HamClasses {
  int end[4];  // terms of class imaginary * 2 + swapped end here
};

template <bool IMAG>
__device__ __forceinline__ void ham_add(double c, double ar, double ai, double& re, double& im) {
  if (IMAG) {
    re = fma(-c, ai, re);
    im = fma(c, ar, im);
  } else {
    re = fma(c, ar, re);
    im = fma(c, ai, im);
  }
}

__device__ __forceinline__ double flip_sign(double c, uint32_t top_bit) {
  return __hiloint2double(__double2hiint(c) ^ (int)top_bit, __double2loint(c));
}

template <typename R>
__global__ void __launch_bounds__(kAThreads)
    ham_half(const typename C2T<R>::T* __restrict__ psi, typename C2T<R>::T* __restrict__ lam, uint64_t dim, int h,
             int first, int last, const HamTerm* __restrict__ terms, const HamClasses cls,
             double* __restrict__ epart) {
  using T = typename C2T<R>::T;
  constexpr int PER = 16 / (int)sizeof(T);  // outputs a thread
  struct alignas(16) Word {
    T v[PER];
  };
  __shared__ double sh[32];
  extern __shared__ __align__(16) unsigned char hsm[];
  const int nterms = cls.end[3], chunks = (nterms + 31) / 32, tid = threadIdx.x, lane = tid & 31;
  HamTerm* st = reinterpret_cast<HamTerm*>(hsm);
  uint32_t* own = reinterpret_cast<uint32_t*>(st + nterms) + tid;  // [chunk][thread]
  for (int i = tid; i < nterms; i += kAThreads) st[i] = terms[i];
  __syncthreads();
  for (int c = 0; c < chunks; ++c) {
    uint32_t m = 0;
    for (int t = 32 * c; t < min(nterms, 32 * c + 32); ++t)
      m |= (uint32_t)(__popcll((uint64_t)(PER * tid) & st[t].sign) & 1) << (t & 31);
    own[c * kAThreads] = m;
  }
  const T* s = psi + (uint64_t)blockIdx.y * dim;
  T* l = lam + (uint64_t)blockIdx.y * dim;
  const uint64_t half = dim >> 1, lo = h ? half : 0, hi = h ? dim : half;
  double e = 0.0;
  for (uint64_t base = lo + (uint64_t)blockIdx.x * (kAThreads * PER); base < hi;
       base += (uint64_t)gridDim.x * (kAThreads * PER)) {
    const uint64_t y = base + (uint64_t)(PER * tid);
    const bool in = y < hi;
    double re[PER] = {}, im[PER] = {};
    if (!first && in) {  // lambda and psi[y] stream through (evict-first) so
                         // the gathered half keeps L2
      const float4 w = __ldcs(reinterpret_cast<const float4*>(l + y));
      const Word p = *reinterpret_cast<const Word*>(&w);
#pragma unroll
      for (int u = 0; u < PER; ++u) {
        re[u] = p.v[u].x;
        im[u] = p.v[u].y;
      }
    }
    const uint64_t ys = in ? y : lo;  // a thread beyond the half reads, and adds nothing
    uint32_t mask = 0;
    int t = 0;
    auto run = [&](auto imag, auto swapped, int end) {
      constexpr bool IMAG = decltype(imag)::value, SW = decltype(swapped)::value;
      auto refill = [&]() {
        const int j = (t & ~31) + lane;
        const bool odd = j < nterms && (__popcll(base & st[j].sign) & 1);
        mask = __ballot_sync(0xffffffffu, odd) ^ own[(t >> 5) * kAThreads];
      };
      while (t < end) {
        if ((t & 31) == 0 || t == 0) refill();
        const int stop = min(end, (t | 31) + 1);  // to the end of the 32 terms
        for (; t + 4 <= stop; t += 4) {
          Word a[4];
#pragma unroll
          for (int u = 0; u < 4; ++u)
            a[u] = *reinterpret_cast<const Word*>(s + ((ys ^ st[t + u].flip) & ~(uint64_t)(PER - 1)));
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const uint32_t neg = (mask << (31 - ((t + u) & 31))) & 0x80000000u;
#pragma unroll
            for (int k = 0; k < PER; ++k) {
              const T& v = a[u].v[SW ? PER - 1 - k : k];
              ham_add<IMAG>(flip_sign(k ? st[t + u].c1 : st[t + u].c0, neg), (double)v.x, (double)v.y, re[k], im[k]);
            }
          }
        }
        for (; t < stop; ++t) {
          const Word a = *reinterpret_cast<const Word*>(s + ((ys ^ st[t].flip) & ~(uint64_t)(PER - 1)));
          const uint32_t neg = (mask << (31 - (t & 31))) & 0x80000000u;
#pragma unroll
          for (int k = 0; k < PER; ++k) {
            const T& v = a.v[SW ? PER - 1 - k : k];
            ham_add<IMAG>(flip_sign(k ? st[t].c1 : st[t].c0, neg), (double)v.x, (double)v.y, re[k], im[k]);
          }
        }
      }
    };
    run(std::false_type{}, std::false_type{}, cls.end[0]);
    run(std::false_type{}, std::true_type{}, cls.end[1]);
    run(std::true_type{}, std::false_type{}, cls.end[2]);
    run(std::true_type{}, std::true_type{}, cls.end[3]);
    if (in) {
      Word o;
#pragma unroll
      for (int u = 0; u < PER; ++u) {
        o.v[u].x = (R)re[u];
        o.v[u].y = (R)im[u];
      }
      __stcs(reinterpret_cast<float4*>(l + y), *reinterpret_cast<const float4*>(&o));
      if (last) {
        const float4 w = __ldcs(reinterpret_cast<const float4*>(s + y));
        const Word p = *reinterpret_cast<const Word*>(&w);
#pragma unroll
        for (int u = 0; u < PER; ++u) e += (double)p.v[u].x * re[u] + (double)p.v[u].y * im[u];
      }
    }
  }
  if (!last) return;
  const int warp = tid >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) e += __shfl_down_sync(0xffffffffu, e, o);
  if (lane == 0) sh[warp] = e;
  __syncthreads();
  if (tid == 0) {
    double v = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) v += sh[w];
    epart[((size_t)blockIdx.y * 2 + h) * gridDim.x + blockIdx.x] += v;
  }
}

// ---------------------------------------------------------------------------
// Resident form, for states that fit the shared memory of one CTA: one CTA a
// parameter set runs the whole circuit forwards, H psi (where that is little
// work, else between two launches) and the reverse sweep with psi and lambda
// in shared memory, one barrier a gate.  The arithmetic of a gate is that of
// the per-gate kernels.
//
// What bounds it is the chain of gates: a gate of a small state is a few
// hundred cycles of shared-memory reads, products and a barrier, against a
// launch (about 3 us on the device, 5 us in the stream) in the per-gate form.
// So everything that a gate needs is staged ahead (records and matrices, 64
// gates at a time), and the FP64 partial sums of a gradient stay one per
// thread until 16 gates have them, when each warp sums whole rows.
// A call with 4 layers and 16 terms, 8 sets: 8 qubits complex64 1255 -> 493
// us, 10 qubits 1459 -> 538, 10 qubits complex128 1440 -> 508 (per gate
// before), of which some 400 us are the host's.  256 threads a CTA: with 512
// or 1024 a few sets take as long, 1024 sets of 11 qubits 2.33 and 2.25 ms
// against 1.97.  Up to 11 qubits: at 12 (complex64) one tile holds a state too, and the
// tiled sweeps, with 16 amplitudes a thread in registers, take 776 us against 786 (8
// sets) and 1116 against 1094 (256 sets); at 11 (complex128) they take 683
// against 600 and, for 1024 sets, 2.36 against 2.18 ms.
constexpr int kResThreads = 256;  // at most
constexpr int kResGates = 64;     // gates staged at a time
constexpr int kResRows = 16;      // gradient rows between two sums
constexpr int kResMaxQubits = 11;
// H psi by the set's own CTA up to this many amplitudes x terms; there (11
// qubits, 128 terms) it takes as long as the launches that spread it over the
// chip: 8 sets 778 against 730 us, 512 sets 1126 against 1117.
constexpr uint64_t kResHamWork = 1u << 18;

struct ResGate {
  uint32_t p0, p1;
  int32_t ck;  // the state after this gate is this checkpoint (0: none)
  int16_t fixed[3];
  uint8_t nfixed, kind, gen, grad;  // grad: has a row of gradient partials
};

struct ResTerm {
  uint32_t flip, sign;
  double c;  // real: c, imaginary: i c
  uint32_t imag, pad;
};

enum { kResForward = 1, kResHam = 2, kResReverse = 4 };

__device__ __forceinline__ uint32_t res_index(const ResGate& g, uint32_t i) {
#pragma unroll
  for (int j = 0; j < 3; ++j)
    if (j < g.nfixed) i = ((i >> g.fixed[j]) << (g.fixed[j] + 1)) | (i & ((1u << g.fixed[j]) - 1));
  return i;
}

template <typename R>
struct ResMat {
  R r[4], i[4];
};

template <typename R, typename T>
__device__ __forceinline__ T res_mul(R mr, R mi, T a) {
  T o;
  o.x = mr * a.x - mi * a.y;
  o.y = mr * a.y + mi * a.x;
  return o;
}

template <typename R, typename T>
__device__ __forceinline__ void res_pair(const ResMat<R>& m, T a, T c, T& x, T& y) {
  x.x = m.r[0] * a.x - m.i[0] * a.y + m.r[1] * c.x - m.i[1] * c.y;
  x.y = m.r[0] * a.y + m.i[0] * a.x + m.r[1] * c.y + m.i[1] * c.x;
  y.x = m.r[2] * a.x - m.i[2] * a.y + m.r[3] * c.x - m.i[3] * c.y;
  y.y = m.r[2] * a.y + m.i[2] * a.x + m.r[3] * c.y + m.i[3] * c.x;
}

size_t resident_smem(size_t state_bytes, int threads, size_t real_bytes) {
  return 2 * state_bytes + sizeof(double) * kResRows * (size_t)threads + kResGates * (sizeof(ResGate) + 8 * real_bytes);
}

template <typename R>
__global__ void __launch_bounds__(kResThreads)
    adjoint_resident(typename C2T<R>::T* __restrict__ psi, typename C2T<R>::T* __restrict__ lam,
                     typename C2T<R>::T* __restrict__ ck, int n, const ResGate* __restrict__ gates, int ngates,
                     const double* __restrict__ mats, uint64_t chunk, const ResTerm* __restrict__ terms, int nterms,
                     int phases, double* __restrict__ gpart, double* __restrict__ vpart) {
  using T = typename C2T<R>::T;
  extern __shared__ __align__(16) unsigned char rsm[];
  __shared__ double wsum[kResThreads / 32];
  const uint32_t dim = 1u << n, tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5;
  const uint64_t set = blockIdx.x;
  T* s = reinterpret_cast<T*>(rsm);
  T* l = s + dim;
  double* rows = reinterpret_cast<double*>(l + dim);  // [row][thread]
  R* cm = reinterpret_cast<R*>(rows + kResRows * nt);
  ResGate* cg = reinterpret_cast<ResGate*>(cm + 8 * kResGates);
  auto stage = [&](int first, int count) {
    __syncthreads();
    for (int i = (int)tid; i < 8 * count; i += (int)nt)
      cm[i] = (R)mats[((uint64_t)(first + (i >> 3)) * chunk + set) * 8 + (i & 7)];
    for (int i = (int)tid; i < count; i += (int)nt) cg[i] = gates[first + i];
    __syncthreads();
  };
  auto count_of = [&](const ResGate& g) { return dim >> g.nfixed; };

  if (phases & kResForward) {
    for (uint32_t i = tid; i < dim; i += nt) {
      T z;
      z.x = i == 0 ? (R)1 : (R)0;
      z.y = (R)0;
      s[i] = z;
    }
    for (int c0 = 0; c0 < ngates; c0 += kResGates) {
      const int cn = min(kResGates, ngates - c0);
      stage(c0, cn);
      for (int k = 0; k < cn; ++k) {
        const ResGate g = cg[k];
        const R* e = cm + 8 * k;
        ResMat<R> m;
#pragma unroll
        for (int j = 0; j < 4; ++j) m.r[j] = e[2 * j], m.i[j] = e[2 * j + 1];
        const uint32_t count = count_of(g);
        if (g.kind == 2) {
          for (uint32_t i = tid; i < count; i += nt) {
            const uint32_t b = res_index(g, i) | g.p0;
            s[b] = res_mul<R, T>(m.r[0], m.i[0], s[b]);
          }
        } else {
          for (uint32_t i = tid; i < count; i += nt) {
            const uint32_t b = res_index(g, i);
            const T a = s[b | g.p0], c = s[b | g.p1];
            T x = c, y = a;
            if (g.kind == 0) res_pair<R, T>(m, a, c, x, y);
            s[b | g.p0] = x;
            s[b | g.p1] = y;
          }
        }
        __syncthreads();
        if (g.ck) {  // the same thread reads it back
          T* o = ck + ((uint64_t)g.ck * chunk + set) * dim;
          for (uint32_t i = tid; i < dim; i += nt) o[i] = s[i];
          __syncthreads();
        }
      }
    }
    __syncthreads();
    if (!(phases & kResHam))
      for (uint32_t i = tid; i < dim; i += nt) psi[set * dim + i] = s[i];
  } else {
    for (uint32_t i = tid; i < dim; i += nt) {
      s[i] = psi[set * dim + i];
      l[i] = lam[set * dim + i];
    }
  }

  if (phases & kResHam) {
    double e = 0.0;
    for (uint32_t y = tid; y < dim; y += nt) {
      double re = 0.0, im = 0.0;
#pragma unroll 4
      for (int t = 0; t < nterms; ++t) {
        const ResTerm h = terms[t];
        const uint32_t x = y ^ h.flip;
        const T a = s[x];
        const double c = (__popc(x & h.sign) & 1) ? -h.c : h.c;
        const double ar = a.x, ai = a.y;
        re = fma(c, h.imag ? -ai : ar, re);
        im = fma(c, h.imag ? ar : ai, im);
      }
      T o;
      o.x = (R)re;
      o.y = (R)im;
      l[y] = o;
      const T p = s[y];
      e += (double)p.x * re + (double)p.y * im;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) e += __shfl_down_sync(0xffffffffu, e, o);
    if (lane == 0) wsum[warp] = e;
    __syncthreads();
    if (tid == 0) {
      double v = 0.0;
      for (uint32_t w = 0; w < nt / 32; ++w) v += wsum[w];
      vpart[set] = v;
    }
  }

  if (phases & kResReverse) {
    int row = 0;
    int32_t row_gate[kResRows];
    auto sum_rows = [&]() {  // row r of `rows` belongs to gate row_gate[r]
      __syncthreads();
#pragma unroll
      for (int r = 0; r < kResRows; ++r) {
        if (r < row && (uint32_t)r % (nt / 32) == warp) {
          double v = 0.0;
          for (uint32_t i = lane; i < nt; i += 32) v += rows[r * nt + i];
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
          if (lane == 0) gpart[(uint64_t)row_gate[r] * chunk + set] = v;
        }
      }
      __syncthreads();
      row = 0;
    };
    for (int c0 = (ngates - 1) / kResGates * kResGates; c0 >= 0 && ngates > 0; c0 -= kResGates) {
      const int cn = min(kResGates, ngates - c0);
      stage(c0, cn);
      for (int k = cn; k-- > 0;) {
        const ResGate g = cg[k];
        const R* e = cm + 8 * k;
        ResMat<R> m;  // U^dag
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int d = (j & 1) * 2 + (j >> 1);
          m.r[j] = e[2 * d], m.i[j] = -e[2 * d + 1];
        }
        if (g.ck) {
          const T* o = ck + ((uint64_t)g.ck * chunk + set) * dim;
          for (uint32_t i = tid; i < dim; i += nt) s[i] = o[i];
          __syncthreads();
        }
        const uint32_t count = count_of(g);
        double acc = 0.0;
        if (g.kind == 2) {
          for (uint32_t i = tid; i < count; i += nt) {
            const uint32_t b = res_index(g, i) | g.p0;
            const T a = s[b], v = l[b];
            if (g.gen == 4) acc += (double)v.x * (double)a.y - (double)v.y * (double)a.x;
            s[b] = res_mul<R, T>(m.r[0], m.i[0], a);
            l[b] = res_mul<R, T>(m.r[0], m.i[0], v);
          }
        } else {
          for (uint32_t i = tid; i < count; i += nt) {
            const uint32_t b = res_index(g, i);
            const T a0 = s[b | g.p0], a1 = s[b | g.p1], l0 = l[b | g.p0], l1 = l[b | g.p1];
            if (g.gen) {  // Im(conj(l0) (G psi)_0 + conj(l1) (G psi)_1)
              const T u = g.gen == 3 ? a0 : a1, w = g.gen == 3 ? a1 : a0;
              const double ur = u.x, ui = u.y, wr = w.x, wi = w.y;
              const double p0r = l0.x, p0i = l0.y, p1r = l1.x, p1i = l1.y;
              if (g.gen == 1) acc += p0r * ui - p0i * ur + p1r * wi - p1i * wr;
              else if (g.gen == 2) acc += -p0r * ur - p0i * ui + p1r * wr + p1i * wi;  // (-i a1, i a0)
              else acc += p0r * ui - p0i * ur - p1r * wi + p1i * wr;
            }
            T x = a1, y = a0;
            if (g.kind == 0) res_pair<R, T>(m, a0, a1, x, y);
            s[b | g.p0] = x;
            s[b | g.p1] = y;
            x = l1, y = l0;
            if (g.kind == 0) res_pair<R, T>(m, l0, l1, x, y);
            l[b | g.p0] = x;
            l[b | g.p1] = y;
          }
        }
        if (g.grad) {
#pragma unroll
          for (int r = 0; r < kResRows; ++r)
            if (r == row) row_gate[r] = c0 + k;
          rows[row * nt + tid] = acc;
          ++row;
        }
        if (row == kResRows) sum_rows();
        else __syncthreads();
      }
    }
    if (row) sum_rows();
  }
}

// Matrices of the circuit's gates for every parameter set, [gate][set][8].
// A gate without a parameter has the same one for all sets (made on the host);
// a parameterised one is formed here from its set's angle, with ket's
// formulas.  The host loop over gates and sets, and the copy of its result,
// were most of a small call.
struct AdjGate {
  double m[8];   // kind 0: the matrix
  int32_t kind;  // 0 fixed, 1 Rx, 2 Ry, 3 Rz (or their controlled forms), 4 CP,
                 // 5 Rz without its global phase: diag(1, e^{it})
  int32_t pslot;
};

template <typename R>
__global__ void gate_matrices(const AdjGate* __restrict__ gates, int ngates, const double* __restrict__ params,
                              uint64_t nparams, uint64_t nsets, uint64_t stride, int diag_phase,
                              R* __restrict__ out) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (uint64_t)ngates * nsets) return;
  const uint64_t gi = i / nsets, set = i % nsets;
  const AdjGate& g = gates[gi];
  double m[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) m[j] = g.m[j];
  if (g.kind) {
    const double t = params[set * nparams + g.pslot];
    double s, c;
    sincos(g.kind >= 4 ? t : t / 2.0, &s, &c);
#pragma unroll
    for (int j = 0; j < 8; ++j) m[j] = 0.0;
    if (g.kind == 1) {
      m[0] = m[6] = c;
      m[3] = m[5] = -s;
    } else if (g.kind == 2) {
      m[0] = m[6] = c;
      m[2] = -s;
      m[4] = s;
    } else if (g.kind == 3) {
      m[0] = m[6] = c;
      m[1] = -s;
      m[7] = s;
    } else if (diag_phase) {  // the tiled sweeps take a phase as diag(1, phase)
      m[0] = 1.0;
      m[6] = c;
      m[7] = s;
    } else {
      m[0] = c;
      m[1] = s;
    }
  }
  R* o = out + (gi * stride + set) * 8;
#pragma unroll
  for (int j = 0; j < 8; ++j) o[j] = (R)m[j];
}

// One warp a result: the sum of its partials, scaled, over its pieces (gates
// that share a parameter).  Fixed order: lane-strided per piece, then a tree.
struct AdjPiece {
  uint64_t at;      // first partial of set 0
  uint64_t stride;  // from set to set
  double scale;
};

__global__ void sum_partials(const double* __restrict__ part, const AdjPiece* __restrict__ pieces,
                             const int32_t* __restrict__ first /* [nresults + 1] */, int nresults, uint64_t nsets,
                             int count, double* __restrict__ out) {
  const uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (w >= (uint64_t)nresults * nsets) return;
  const int lane = threadIdx.x & 31;
  const uint64_t set = w / nresults, r = w % nresults;
  double v = 0.0;
  for (int k = first[r]; k < first[r + 1]; ++k) {
    const double* p = part + pieces[k].at + set * pieces[k].stride;
    double a = 0.0;
    for (int i = lane; i < count; i += 32) a += p[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    v += pieces[k].scale * a;
  }
  if (lane == 0) out[set * nresults + r] = v;
}

template <typename R>
__global__ void ground_batch(typename C2T<R>::T* states, uint64_t dim) {
  typename C2T<R>::T one;
  one.x = 1;
  one.y = 0;
  states[(uint64_t)blockIdx.x * dim] = one;
}


// ---------------------------------------------------------------------------
// Tiled sweeps.  The per-gate kernels above stream psi (and lambda) through
// HBM once per gate.  The tiled form groups consecutive gates into blocks
// whose qubits fit one tile of TB qubits (always including qubits 0-4, so a
// warp's 32 consecutive tile elements are 32 consecutive amplitudes), loads
// each tile of psi and lambda into shared memory once, and runs the whole
// block there: the forward applications, or in the reverse sweep the
// gradient inner products and the inverse applications of every gate of the
// block.  Inside a block, gates are run in phases: a phase names RB tile bits
// that each thread holds in registers (2^RB amplitudes of each state), so
// every gate whose target bits are among them is register arithmetic; a
// diagonal gate needs no register bits at all.  Gradient partial sums are
// formed per thread over its pairs in the state's precision, reduced across
// the warp in FP64 and accumulated per warp and gate in shared memory (FP64),
// then summed in fixed order over warps, CTAs and blocks (sum_partials).

// TileCfg, TGate, TPhase, TileGeom, the swizzle, the asynchronous copy and
// the packed complex64 gate code live in adj_tile.cuh, shared with the
// per-block kernels compiled at run time.
using namespace kbt;

template <typename R>
struct CM2 {
  R r[4], i[4];
};

// m (U, row-major, 8 values re/im interleaved) or its conjugate transpose.
template <typename R, bool DAG>
__device__ __forceinline__ CM2<R> load_cm2(const R* m) {
  CM2<R> c;
  if (!DAG) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      c.r[k] = m[2 * k];
      c.i[k] = m[2 * k + 1];
    }
  } else {
    c.r[0] = m[0], c.i[0] = -m[1];
    c.r[1] = m[4], c.i[1] = -m[5];
    c.r[2] = m[2], c.i[2] = -m[3];
    c.r[3] = m[6], c.i[3] = -m[7];
  }
  return c;
}

template <typename T, typename R>
__device__ __forceinline__ void mul2(const CM2<R>& c, T& a, T& b) {
  T x, y;
  x.x = c.r[0] * a.x - c.i[0] * a.y + c.r[1] * b.x - c.i[1] * b.y;
  x.y = c.r[0] * a.y + c.i[0] * a.x + c.r[1] * b.y + c.i[1] * b.x;
  y.x = c.r[2] * a.x - c.i[2] * a.y + c.r[3] * b.x - c.i[3] * b.y;
  y.y = c.r[2] * a.y + c.i[2] * a.x + c.r[3] * b.y + c.i[3] * b.x;
  a = x;
  b = y;
}

template <typename T, typename R>
__device__ __forceinline__ void mul2_real(const CM2<R>& c, T& a, T& b) {
  T x, y;
  x.x = c.r[0] * a.x + c.r[1] * b.x;
  x.y = c.r[0] * a.y + c.r[1] * b.y;
  y.x = c.r[2] * a.x + c.r[3] * b.x;
  y.y = c.r[2] * a.y + c.r[3] * b.y;
  a = x;
  b = y;
}

template <typename T, typename R>
__device__ __forceinline__ void cmul(T& a, R pr, R pi) {
  const R x = pr * a.x - pi * a.y;
  a.y = pr * a.y + pi * a.x;
  a.x = x;
}

template <typename T, typename R>
__device__ __forceinline__ void tswap(T& a, T& b) {
  const T t = a;
  a = b;
  b = t;
}

// Im <l|G|a> on one pair for the generators X (1), Y (2), Z (3).
template <typename T, typename R>
__device__ __forceinline__ R pair_grad(int gen, const T& a0, const T& a1, const T& l0, const T& l1) {
  if (gen == 1) return (l0.x * a1.y - l0.y * a1.x) + (l1.x * a0.y - l1.y * a0.x);
  if (gen == 2) return (l1.x * a0.x + l1.y * a0.y) - (l0.x * a1.x + l0.y * a1.y);
  return (l0.x * a0.y - l0.y * a0.x) - (l1.x * a1.y - l1.y * a1.x);
}

// Gate bodies.  A thread holds the 2^RB register elements j of its group; S
// (A, B) are register slots known at compile time; RC says whether some
// control bits are register bits (then each j is tested against cm_r).
// Forward (REV = false) applies U to p; reverse adds the gradient term and
// applies U^dag to p and q.  What a gate is (its generator, a real matrix, a
// unit entry) is decided once a gate, not once a pair: with the tests inside
// the unrolled loops four of five instructions of a block were not arithmetic.

template <typename R, int RB, int S, bool REV, bool RC>
__device__ __forceinline__ R tile_pair(typename C2T<R>::T* p, typename C2T<R>::T* q, const TGate& g,
                                       const R* m) {
  R part = 0;
  if constexpr (S < RB) {
    if (g.kind == kTPairSwap) {
#pragma unroll
      for (int j = 0; j < (1 << RB); ++j) {
        if (j & (1 << S)) continue;
        if (RC && (j & g.cm_r) != g.cm_r) continue;
        tswap<typename C2T<R>::T, R>(p[j], p[j | (1 << S)]);
        if (REV) tswap<typename C2T<R>::T, R>(q[j], q[j | (1 << S)]);
      }
      return part;
    }
    const CM2<R> c = load_cm2<R, REV>(m);
    auto body = [&](auto real, auto generator) {
      constexpr bool REAL = decltype(real)::value;
      constexpr int GEN = decltype(generator)::value;
#pragma unroll
      for (int j = 0; j < (1 << RB); ++j) {
        if (j & (1 << S)) continue;
        const int j1 = j | (1 << S);
        if (RC && (j & g.cm_r) != g.cm_r) continue;
        if (REV && GEN) part += pair_grad<typename C2T<R>::T, R>(GEN, p[j], p[j1], q[j], q[j1]);
        if constexpr (REAL) {
          mul2_real(c, p[j], p[j1]);
          if (REV) mul2_real(c, q[j], q[j1]);
        } else {
          mul2(c, p[j], p[j1]);
          if (REV) mul2(c, q[j], q[j1]);
        }
      }
    };
    using std::integral_constant;
    const int gen = REV ? g.gen : 0;
    if (g.real) {
      if (REV && gen == 2) body(std::true_type{}, integral_constant<int, 2>{});
      else body(std::true_type{}, integral_constant<int, 0>{});  // (only Y's rotations are real)
    } else {
      if (REV && gen == 1) body(std::false_type{}, integral_constant<int, 1>{});
      else if (REV && gen == 2) body(std::false_type{}, integral_constant<int, 2>{});
      else if (REV && gen) body(std::false_type{}, integral_constant<int, 3>{});
      else body(std::false_type{}, integral_constant<int, 0>{});
    }
  }
  return part;
}

template <typename R, int RB, int A, int B, bool REV, bool RC>
__device__ __forceinline__ void tile_swap2(typename C2T<R>::T* p, typename C2T<R>::T* q, const TGate& g) {
  if constexpr (A < RB && B < RB && A < B) {
#pragma unroll
    for (int j = 0; j < (1 << RB); ++j) {
      if (!(j & (1 << A)) || (j & (1 << B))) continue;
      if (RC && (j & g.cm_r) != g.cm_r) continue;
      const int j1 = j ^ (1 << A) ^ (1 << B);
      tswap<typename C2T<R>::T, R>(p[j], p[j1]);
      if (REV) tswap<typename C2T<R>::T, R>(q[j], q[j1]);
    }
  }
}

// Diagonal gate whose target is register slot S: diag(m0, m3).
template <typename R, int RB, int S, bool REV, bool RC>
__device__ __forceinline__ R tile_diag_reg(typename C2T<R>::T* p, typename C2T<R>::T* q, const TGate& g,
                                           const R* m) {
  R part = 0;
  if constexpr (S < RB) {
    const R m0r = m[0], m0i = REV ? -m[1] : m[1], m3r = m[6], m3i = REV ? -m[7] : m[7];
    auto body = [&](auto unit, auto generator) {
      constexpr bool UNIT = decltype(unit)::value;  // the entry of target bit 0 is 1
      constexpr int GEN = decltype(generator)::value;
#pragma unroll
      for (int j = 0; j < (1 << RB); ++j) {
        if (RC && (j & g.cm_r) != g.cm_r) continue;
        const bool bit = (j >> S) & 1;
        if (REV && (GEN == 3 || (GEN == 4 && bit))) {  // Z, P11: Im(conj(l) a)
          const R im = q[j].x * p[j].y - q[j].y * p[j].x;
          part += GEN == 3 && bit ? -im : im;
        }
        if (UNIT && !bit) continue;
        cmul(p[j], bit ? m3r : m0r, bit ? m3i : m0i);
        if (REV) cmul(q[j], bit ? m3r : m0r, bit ? m3i : m0i);
      }
    };
    using std::integral_constant;
    const int gen = REV ? g.gen : 0;
    if (g.real) {
      if (REV && gen == 3) body(std::true_type{}, integral_constant<int, 3>{});
      else if (REV && gen) body(std::true_type{}, integral_constant<int, 4>{});
      else body(std::true_type{}, integral_constant<int, 0>{});
    } else {
      if (REV && gen == 3) body(std::false_type{}, integral_constant<int, 3>{});
      else if (REV && gen) body(std::false_type{}, integral_constant<int, 4>{});
      else body(std::false_type{}, integral_constant<int, 0>{});
    }
  }
  return part;
}

// Diagonal gate whose target is a group bit: one phase for all of the
// thread's elements.
template <typename R, int RB, bool REV, bool RC>
__device__ __forceinline__ R tile_diag_grp(typename C2T<R>::T* p, typename C2T<R>::T* q, const TGate& g,
                                           const R* m, bool bit) {
  R part = 0;
  const R pr = bit ? m[6] : m[0];
  const R pi = REV ? -(bit ? m[7] : m[1]) : (bit ? m[7] : m[1]);
  const int gen = REV ? g.gen : 0;
  if (REV && gen) {
#pragma unroll
    for (int j = 0; j < (1 << RB); ++j) {
      if (RC && (j & g.cm_r) != g.cm_r) continue;
      part += q[j].x * p[j].y - q[j].y * p[j].x;
    }
    part = gen == 3 ? (bit ? -part : part) : (bit ? part : R(0));
  }
  if (!bit && g.real) return part;  // times 1
#pragma unroll
  for (int j = 0; j < (1 << RB); ++j) {
    if (RC && (j & g.cm_r) != g.cm_r) continue;
    cmul(p[j], pr, pi);
    if (REV) cmul(q[j], pr, pi);
  }
  return part;
}

template <typename R, int RB, bool REV, bool RC>
__device__ __forceinline__ R tile_gate_rc(typename C2T<R>::T* p, typename C2T<R>::T* q, const TGate& g,
                                          const R* m, int gbase) {
  if (g.kind == kTDiag) {
    switch (g.tslot) {
      case 0: return tile_diag_reg<R, RB, 0, REV, RC>(p, q, g, m);
      case 1: return tile_diag_reg<R, RB, 1, REV, RC>(p, q, g, m);
      case 2: return tile_diag_reg<R, RB, 2, REV, RC>(p, q, g, m);
      case 3: return tile_diag_reg<R, RB, 3, REV, RC>(p, q, g, m);
      default: return tile_diag_grp<R, RB, REV, RC>(p, q, g, m, (gbase >> g.tbit) & 1);
    }
  }
  if (g.kind == kTSwap2) {
    switch (g.s0 * 4 + g.s1) {
      case 1: tile_swap2<R, RB, 0, 1, REV, RC>(p, q, g); break;
      case 2: tile_swap2<R, RB, 0, 2, REV, RC>(p, q, g); break;
      case 3: tile_swap2<R, RB, 0, 3, REV, RC>(p, q, g); break;
      case 6: tile_swap2<R, RB, 1, 2, REV, RC>(p, q, g); break;
      case 7: tile_swap2<R, RB, 1, 3, REV, RC>(p, q, g); break;
      case 11: tile_swap2<R, RB, 2, 3, REV, RC>(p, q, g); break;
      default: break;
    }
    return 0;
  }
  switch (g.s0) {
    case 0: return tile_pair<R, RB, 0, REV, RC>(p, q, g, m);
    case 1: return tile_pair<R, RB, 1, REV, RC>(p, q, g, m);
    case 2: return tile_pair<R, RB, 2, REV, RC>(p, q, g, m);
    default: return tile_pair<R, RB, 3, REV, RC>(p, q, g, m);
  }
}

template <typename R, int RB, bool REV>
__device__ __forceinline__ R tile_gate(typename C2T<R>::T* p, typename C2T<R>::T* q, const TGate& g,
                                       const R* m, int gbase) {
  if ((gbase & g.cm_g) != g.cm_g) return 0;  // a group-bit control is 0 for this thread
  return g.cm_r ? tile_gate_rc<R, RB, REV, true>(p, q, g, m, gbase)
                : tile_gate_rc<R, RB, REV, false>(p, q, g, m, gbase);
}


// Forward (REV = false: psi only, gates in order) or reverse (REV = true:
// psi and lambda, gates in reverse order, gradient partials) over one block,
// for every tile of every parameter set of the chunk (gridDim.y = set); the
// complex128 form.  Two CTAs per SM: forwards the next tile streams into a
// second buffer with cp.async while the current one is processed; in reverse
// one buffer holds psi and lambda, and one CTA's copies run under the other's
// gates.  Shared memory: the tile buffers, the block's gate records and this
// set's matrices, then the gradient sums (reverse), eight lanes a warp.
// What bounds it is instruction issue, half busy with two CTAs (a third with
// one): of a gate's instructions a quarter is FP64 arithmetic, the rest moves of
// 64 registers between the gate bodies and the bodies' selection.  20 qubits, 8 sets, 4 layers:
// 8.5 -> 6.0 ms a call against one CTA with two buffers, full warp sums a
// gradient and a gate's tests inside its loops.
template <typename R, bool REV>
__global__ void __launch_bounds__(kTileThreads, 2)
    tile_sweep(typename C2T<R>::T* __restrict__ psi, typename C2T<R>::T* __restrict__ lam, uint64_t dim,
               TileGeom tg, const TGate* __restrict__ gates, int ngates, const TPhase* __restrict__ phases,
               int nph, const R* __restrict__ mats, uint64_t mat_stride, int ngrad, double* __restrict__ partial) {
  using T = typename C2T<R>::T;
  constexpr int TB = TileCfg<R>::TB, RB = TileCfg<R>::RB, NR = 1 << RB, TILE = 1 << TB;
  extern __shared__ __align__(16) unsigned char tsm[];
  T* bufs = reinterpret_cast<T*>(tsm);  // two of psi, or one of psi and one of lambda
  TGate* sg = reinterpret_cast<TGate*>(tsm + 2 * TILE * sizeof(T));
  R* smat = reinterpret_cast<R*>(sg + ngates);
  double* acc = reinterpret_cast<double*>(smat + 8 * (size_t)ngates);  // [gradient][warp][8 lanes]
  // offset of tile element tid + 256 r: off[tid] + off[256 + r]
  __shared__ uint64_t off[kTileThreads + NR];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int set = blockIdx.y;
  T* s = psi + (uint64_t)set * dim;
  T* l = REV ? lam + (uint64_t)set * dim : nullptr;

  static_assert(kTileThreads << RB == TILE && kTileThreads == 256, "tile elements a thread");
  {
    uint64_t o = 0;
#pragma unroll
    for (int b = 0; b < 8; ++b)
      if ((tid >> b) & 1) o |= uint64_t{1} << tg.pos[b];
    off[tid] = o;
    if (tid < NR) {
      o = 0;
#pragma unroll
      for (int b = 0; b < RB; ++b)
        if ((tid >> b) & 1) o |= uint64_t{1} << tg.pos[8 + b];
      off[kTileThreads + tid] = o;
    }
  }
  for (int i = tid; i < ngates; i += kTileThreads) {
    const TGate g = gates[i];
    sg[i] = g;
    const R* src = mats + ((uint64_t)g.mat * mat_stride + set) * 8;
#pragma unroll
    for (int k = 0; k < 8; ++k) smat[8 * i + k] = src[k];
  }
  if (REV)
    for (int i = tid; i < 8 * kTileWarps * ngrad; i += kTileThreads) acc[i] = 0.0;
  __syncthreads();

  auto tile_base = [&](uint64_t t) {
    uint64_t base = t;
#pragma unroll
    for (int b = 0; b < TB; ++b) {
      const int f = tg.pos[b];
      base = ((base >> f) << (f + 1)) | (base & ((uint64_t{1} << f) - 1));
    }
    return base;
  };
  const int ptid = tphys<R>(tid);
  auto prefetch = [&](uint64_t at, T* buf) {
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      const uint64_t o = at + off[kTileThreads + r];
      T* d = buf + (ptid ^ tphys<R>(r * kTileThreads));
      tile_cp_async(d, s + o);
      if (REV) tile_cp_async(d + TILE, l + o);
    }
  };

  int cur = 0;
  uint64_t at = 0, next_at = 0;  // where this thread's first element of a tile is
  if (blockIdx.x < tg.n_tiles) {
    next_at = tile_base(blockIdx.x) + off[tid];
    if (!REV) prefetch(next_at, bufs);
  }
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  for (uint64_t t = blockIdx.x; t < tg.n_tiles; t += gridDim.x) {
    T* sp = REV ? bufs : bufs + cur * TILE;
    T* sl = bufs + TILE;  // (reverse)
    at = next_at;
    if (t + gridDim.x < tg.n_tiles) next_at = tile_base(t + gridDim.x) + off[tid];
    if (REV) prefetch(at, bufs);
    else if (t + gridDim.x < tg.n_tiles) prefetch(next_at, bufs + (cur ^ 1) * TILE);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    if (REV) asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    else asm volatile("cp.async.wait_group 1;\n" ::: "memory");  // this tile's copies are done
    __syncthreads();
    for (int k = 0; k < nph; ++k) {
      const TPhase P = phases[REV ? nph - 1 - k : k];
      // group bits of this thread: tid with zeros at the register bits, from
      // the lowest up
      static_assert(RB == 3, "three register bits");
      const int r_lo = min(min(P.r[0], P.r[1]), P.r[2]), r_hi = max(max(P.r[0], P.r[1]), P.r[2]);
      const int r_mid = P.r[0] + P.r[1] + P.r[2] - r_lo - r_hi;
      auto open = [](int x, int b) { return ((x >> b) << (b + 1)) | (x & ((1 << b) - 1)); };
      const int gbase = open(open(open(tid, r_lo), r_mid), r_hi);
      // the swizzle is XOR-linear and gbase, rdep(j) have disjoint bits, so
      // the address of element j is tphys(gbase) ^ tphys(rdep(j))
      const int pg = tphys<R>(gbase);
      int pb[RB];
#pragma unroll
      for (int b = 0; b < RB; ++b) pb[b] = tphys<R>(1 << P.r[b]);
      T p[NR], q[NR];
#pragma unroll
      for (int j = 0; j < NR; ++j) {
        int a = pg;
#pragma unroll
        for (int b = 0; b < RB; ++b)
          if (j & (1 << b)) a ^= pb[b];
        p[j] = sp[a];
        if (REV) q[j] = sl[a];
      }
      for (int c = 0; c < P.count; ++c) {
        const int gi = REV ? P.first + P.count - 1 - c : P.first + c;
        const TGate g = sg[gi];
        const R part = tile_gate<R, RB, REV>(p, q, g, smat + 8 * gi, gbase);
        if (REV && g.grad >= 0) {
          double v = (double)part;
#pragma unroll
          for (int o = 16; o > 4; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
          if (lane < 8) acc[(g.grad * kTileWarps + warp) * 8 + lane] += v;
        }
      }
      {
        // element addresses again, from a fresh read of the phase record (so
        // that the 2^RB addresses are not held in registers across the gates)
        unsigned rw;
        asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(rw) : "l"(&phases[REV ? nph - 1 - k : k]));
        const int pg2 = tphys<R>(gbase);
        int pb2[RB];
#pragma unroll
        for (int b = 0; b < RB; ++b) pb2[b] = tphys<R>(1 << ((rw >> (8 * b)) & 0xff));
#pragma unroll
        for (int j = 0; j < NR; ++j) {
          int a = pg2;
#pragma unroll
          for (int b = 0; b < RB; ++b)
            if (j & (1 << b)) a ^= pb2[b];
          sp[a] = p[j];
          if (REV) sl[a] = q[j];
        }
      }
      __syncthreads();
    }
    {
      const volatile uint64_t* voff = off;
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        const uint64_t o = at + voff[kTileThreads + r];
        const int e = ptid ^ tphys<R>(r * kTileThreads);
        s[o] = sp[e];
        if (REV) l[o] = sl[e];
      }
    }
    __syncthreads();
    cur ^= 1;
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  if (REV) {
    __syncthreads();
    for (int g = warp; g < ngrad; g += kTileWarps) {
      double v = acc[g * 64 + lane] + acc[g * 64 + 32 + lane];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) partial[((uint64_t)set * ngrad + g) * gridDim.x + blockIdx.x] = v;
    }
  }
}


// The complex64 form of tile_sweep (same grid, pipeline and partials).
template <bool REV>
__global__ void __launch_bounds__(kTileThreads, 1)
    tile_sweep_c64(float2* __restrict__ psi, float2* __restrict__ lam, uint64_t dim, TileGeom tg,
                   const TGate* __restrict__ gates, int ngates, const TPhase* __restrict__ phases, int nph,
                   const float* __restrict__ mats, uint64_t mat_stride, int ngrad, double* __restrict__ partial) {
  constexpr int TB = TileCfg<float>::TB, RB = TileCfg<float>::RB, TILE = 1 << TB;
  static_assert(RB == 4, "8 packs of 2 amplitudes per state");
  constexpr int BUF = (REV ? 2 : 1) * TILE;
  extern __shared__ __align__(16) unsigned char tsm[];
  float2* bufs = reinterpret_cast<float2*>(tsm);
  f2* spk = reinterpret_cast<f2*>(tsm + 2 * BUF * sizeof(float2));  // [gate][16]
  TGate* sg = reinterpret_cast<TGate*>(spk + 16 * (size_t)ngates);
  double* acc = reinterpret_cast<double*>(sg + ngates);  // [warp][ngrad]
  __shared__ uint8_t sop[kMaxBlockGates];
  __shared__ uint64_t off_lo[64], off_hi[64];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int set = blockIdx.y;
  float2* s = psi + (uint64_t)set * dim;
  float2* l = REV ? lam + (uint64_t)set * dim : nullptr;

  if (tid < 128) {
    const int half = tid >> 6, e = tid & 63;
    uint64_t off = 0;
    for (int b = 0; b < 6; ++b) {
      const int tb = 6 * half + b;
      if (tb < TB && ((e >> b) & 1)) off |= uint64_t{1} << tg.pos[tb];
    }
    (half ? off_hi : off_lo)[e] = off;
  }
  for (int i = tid; i < ngates; i += kTileThreads) {
    const TGate g = gates[i];
    sg[i] = g;
    sop[i] = (uint8_t)pk_opcode(g, REV);
    const float* m = mats + ((uint64_t)g.mat * mat_stride + set) * 8;
    // U or U^dag, row-major (re, im) of entries 0..3
    float cr[4], ci[4];
    if (!REV) {
      for (int k = 0; k < 4; ++k) cr[k] = m[2 * k], ci[k] = m[2 * k + 1];
    } else {
      cr[0] = m[0], ci[0] = -m[1];
      cr[1] = m[4], ci[1] = -m[5];
      cr[2] = m[2], ci[2] = -m[3];
      cr[3] = m[6], ci[3] = -m[7];
    }
    f2* c = spk + 16 * i;
    for (int k = 0; k < 4; ++k) {
      c[2 * k] = pk2(cr[k], cr[k]);
      c[2 * k + 1] = pk2(ci[k], ci[k]);
      c[8 + k] = pk2(-ci[k], -ci[k]);
    }
    c[12] = pk2(cr[0], cr[3]);
    c[13] = pk2(ci[0], ci[3]);
    c[14] = pk2(-ci[0], -ci[3]);
    c[15] = 0;
  }
  if (REV)
    for (int i = tid; i < kTileWarps * ngrad; i += kTileThreads) acc[i] = 0.0;
  __syncthreads();

  auto tile_base = [&](uint64_t t) {
    uint64_t base = t;
#pragma unroll
    for (int b = 0; b < TB; ++b) {
      const int f = tg.pos[b];
      base = ((base >> f) << (f + 1)) | (base & ((uint64_t{1} << f) - 1));
    }
    return base;
  };
  auto prefetch = [&](uint64_t t, float2* buf) {
    const uint64_t base = tile_base(t);
#pragma unroll 2
    for (int r = 0; r < (1 << RB); ++r) {
      const int e = tid + r * kTileThreads;
      const uint64_t o = base + (off_lo[e & 63] | off_hi[e >> 6]);
      tile_cp_async(buf + tphys<float>(e), s + o);
      if (REV) tile_cp_async(buf + TILE + tphys<float>(e), l + o);
    }
  };

  int cur = 0;
  if (blockIdx.x < tg.n_tiles) prefetch(blockIdx.x, bufs);
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  for (uint64_t t = blockIdx.x; t < tg.n_tiles; t += gridDim.x) {
    float2* sp = bufs + cur * BUF;
    float2* sl = sp + TILE;
    if (t + gridDim.x < tg.n_tiles) prefetch(t + gridDim.x, bufs + (cur ^ 1) * BUF);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    __syncthreads();
    for (int k = 0; k < nph; ++k) {
      const TPhase P = phases[REV ? nph - 1 - k : k];
      int rmask = 0;
#pragma unroll
      for (int b = 0; b < RB; ++b) rmask |= 1 << P.r[b];
      int gbase = 0;
      {
        int kk = 0;
#pragma unroll
        for (int b = 0; b < TB; ++b)
          if (!((rmask >> b) & 1)) {
            gbase |= ((tid >> kk) & 1) << b;
            ++kk;
          }
      }
      const int pg = tphys<float>(gbase);
      int pb[RB];
#pragma unroll
      for (int b = 0; b < RB; ++b) pb[b] = tphys<float>(1 << P.r[b]);
      PackState A, L;
#pragma unroll
      for (int jo = 0; jo < 8; ++jo) {
        int a0 = pg;
#pragma unroll
        for (int b = 1; b < RB; ++b)
          if (jo & (1 << (b - 1))) a0 ^= pb[b];
        const int a1 = a0 ^ pb[0];
        const float2 x = sp[a0], y = sp[a1];
        A.r[jo] = pk2(x.x, y.x);
        A.i[jo] = pk2(x.y, y.y);
        if (REV) {
          const float2 u = sl[a0], v = sl[a1];
          L.r[jo] = pk2(u.x, v.x);
          L.i[jo] = pk2(u.y, v.y);
        }
      }
      for (int c = 0; c < P.count; ++c) {
        const int gi = REV ? P.first + P.count - 1 - c : P.first + c;
        const TGate g = sg[gi];
        float part = 0.f;
        if ((gbase & g.cm_g) == g.cm_g) part = pk_dispatch<REV>(sop[gi], A, L, g, spk + 16 * gi, gbase);
        if (REV && g.grad >= 0) {
          double v = (double)part;
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
          if (lane == 0) acc[warp * ngrad + g.grad] += v;
        }
      }
      {
        // addresses again from a fresh read of the phase record (not held
        // in registers across the gates)
        unsigned rw;
        asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(rw) : "l"(&phases[REV ? nph - 1 - k : k]));
        const int pg2 = tphys<float>(gbase);
        int pb2[RB];
#pragma unroll
        for (int b = 0; b < RB; ++b) pb2[b] = tphys<float>(1 << ((rw >> (8 * b)) & 0xff));
#pragma unroll
        for (int jo = 0; jo < 8; ++jo) {
          int a0 = pg2;
#pragma unroll
          for (int b = 1; b < RB; ++b)
            if (jo & (1 << (b - 1))) a0 ^= pb2[b];
          const int a1 = a0 ^ pb2[0];
          float xr, yr, xi, yi;
          upk2(A.r[jo], xr, yr);
          upk2(A.i[jo], xi, yi);
          sp[a0] = make_float2(xr, xi);
          sp[a1] = make_float2(yr, yi);
          if (REV) {
            upk2(L.r[jo], xr, yr);
            upk2(L.i[jo], xi, yi);
            sl[a0] = make_float2(xr, xi);
            sl[a1] = make_float2(yr, yi);
          }
        }
      }
      __syncthreads();
    }
    {
      const uint64_t base = tile_base(t);
      const volatile uint64_t* vlo = off_lo;
      const volatile uint64_t* vhi = off_hi;
#pragma unroll 2
      for (int r = 0; r < (1 << RB); ++r) {
        const int e = tid + r * kTileThreads;
        const uint64_t o = base + (vlo[e & 63] | vhi[e >> 6]);
        s[o] = sp[tphys<float>(e)];
        if (REV) l[o] = sl[tphys<float>(e)];
      }
    }
    __syncthreads();
    cur ^= 1;
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  if (REV)
    for (int g = tid; g < ngrad; g += kTileThreads) {
      double v = 0.0;
      for (int w = 0; w < kTileWarps; ++w) v += acc[w * ngrad + g];
      partial[((uint64_t)set * ngrad + g) * gridDim.x + blockIdx.x] = v;
    }
}

// Host plan of the tiled sweeps.
struct TBlock {
  TileGeom geom;
  int layer = 0;
  int gate_first = 0, n_gates = 0;    // into the concatenated TGate array
  int phase_first = 0, n_phases = 0;  // into the concatenated TPhase array
  std::vector<int> grad_gate;         // gradient slot -> gate list index
  size_t part_off = 0;                // into the gradient partials (doubles)
  uint64_t active_tiles = 0;          // tiles that can be nonzero after the block
};

struct TilePlan {
  std::vector<TBlock> blocks;
  std::vector<TGate> gates;
  std::vector<TPhase> phases;
};

// Target tile bits, controls and kind of a lowered gate, in tile bits.
struct TileOp {
  uint8_t kind;
  int targets[2];
  int ntargets;
  int tgt_diag;  // kTDiag: target tile bit
  int cmask;     // controls (tile bits)
};

TileOp tile_op_of(const Pass& p, const int* tpos_of_qubit) {
  TileOp t{};
  auto tile_mask = [&](uint64_t m) {
    int r = 0;
    for (int q = 0; q < 64; ++q)
      if ((m >> q) & 1) r |= 1 << tpos_of_qubit[q];
    return r;
  };
  if (p.kind == PassKind::Phase) {
    // all fixed bits must be 1: the highest is the target, the rest controls
    const int top = p.fixed[p.nfixed - 1];
    t.kind = kTDiag;
    t.tgt_diag = tpos_of_qubit[top];
    t.cmask = tile_mask(p.p0 & ~(uint64_t{1} << top));
    t.ntargets = 0;
    return t;
  }
  const uint64_t diff = p.p0 ^ p.p1;
  if (p.mode == kPairDiag) {
    t.kind = kTDiag;
    t.tgt_diag = tpos_of_qubit[__builtin_ctzll(diff)];
    t.cmask = tile_mask(p.p0);
    t.ntargets = 0;
    return t;
  }
  if (__builtin_popcountll(diff) == 2) {
    t.kind = kTSwap2;
    const int a = __builtin_ctzll(diff), b = 63 - __builtin_clzll(diff);
    t.targets[0] = tpos_of_qubit[a];
    t.targets[1] = tpos_of_qubit[b];
    t.ntargets = 2;
    t.cmask = tile_mask(p.p0 & p.p1);
    return t;
  }
  t.kind = p.mode == kPairSwap ? kTPairSwap : kTPair;
  t.targets[0] = tpos_of_qubit[__builtin_ctzll(diff)];
  t.ntargets = 1;
  t.cmask = tile_mask(p.p0);
  return t;
}

template <typename R>
TilePlan plan_tiles(int n, const ketgpu_op* ops, const std::vector<int>& gate_ops, const std::vector<int>& layer_of,
                    const std::vector<GateGeom>& geo, const std::vector<uint8_t>& real, int seg_layers,
                    bool kPacked) {
  constexpr int TB = TileCfg<R>::TB, RB = TileCfg<R>::RB;
  TilePlan tp;
  const int G = (int)gate_ops.size();
  std::vector<uint64_t> qmask(G);
  for (int i = 0; i < G; ++i) {
    const ketgpu_op& o = ops[gate_ops[i]];
    uint64_t m = 0;
    for (int j = 0; j < gate_arity(o.type); ++j) m |= uint64_t{1} << o.q[j];
    qmask[i] = m;
  }
  int i0 = 0;
  while (i0 < G) {
    // one checkpoint segment (seg_layers layers) at a time: blocks may run
    // across the layers of a segment but never across its ends
    int i1 = i0;
    while (i1 < G && layer_of[i1] / seg_layers == layer_of[i0] / seg_layers) ++i1;
    // A topological order of the layer that sweeps the qubits upwards: among
    // the gates whose predecessors (earlier gates sharing a qubit) are
    // placed, take the one with the lowest highest qubit.  Chains such as a
    // CX ring then fall into consecutive tiles instead of being cut by the
    // single-qubit gates listed before them.
    std::vector<int> rem;
    {
      std::vector<std::vector<int>> on_qubit(n);
      for (int i = i0; i < i1; ++i)
        for (int q = 0; q < n; ++q)
          if ((qmask[i] >> q) & 1) on_qubit[q].push_back(i);
      std::vector<size_t> head(n, 0);
      auto ready = [&](int i) {
        for (int q = 0; q < n; ++q)
          if (((qmask[i] >> q) & 1) && on_qubit[q][head[q]] != i) return false;
        return true;
      };
      using Key = std::pair<int, int>;  // (highest qubit, original index)
      std::priority_queue<Key, std::vector<Key>, std::greater<Key>> pq;
      std::vector<uint8_t> queued(G, 0);
      auto offer = [&](int i) {
        if (!queued[i] && ready(i)) {
          queued[i] = 1;
          pq.push({63 - __builtin_clzll(qmask[i]), i});
        }
      };
      for (int q = 0; q < n; ++q)
        if (!on_qubit[q].empty()) offer(on_qubit[q][0]);
      while (!pq.empty()) {
        const int i = pq.top().second;
        pq.pop();
        rem.push_back(i);
        for (int q = 0; q < n; ++q)
          if ((qmask[i] >> q) & 1) {
            ++head[q];
            if (head[q] < on_qubit[q].size()) offer(on_qubit[q][head[q]]);
          }
      }
    }
    while (!rem.empty()) {
      uint64_t S = 0x1f, blocked = 0;
      std::vector<int> take, keep;
      int ngrad = 0;
      for (int i : rem) {
        const bool grad = geo[i].gen && geo[i].pslot >= 0;
        const uint64_t u = S | qmask[i];
        if ((qmask[i] & blocked) || __builtin_popcountll(u) > TB || (int)take.size() >= kMaxBlockGates ||
            (grad && ngrad >= kMaxBlockGrads)) {
          blocked |= qmask[i];
          keep.push_back(i);
          continue;
        }
        S = u;
        take.push_back(i);
        ngrad += grad;
      }
      rem.swap(keep);
      for (int q = 0; q < n && __builtin_popcountll(S) < TB; ++q) S |= uint64_t{1} << q;
      TBlock b;
      b.layer = layer_of[i0];
      int tpos[64];
      for (int q = 0, k = 0; q < n; ++q)
        if ((S >> q) & 1) {
          b.geom.pos[k] = q;
          tpos[q] = k++;
        }
      for (int k = TB; k < 12; ++k) b.geom.pos[k] = 0;
      b.geom.n_tiles = uint64_t{1} << (n - TB);
      // phases: runs of gates whose target bits fit RB register bits
      std::vector<TileOp> top(take.size());
      for (size_t k = 0; k < take.size(); ++k) top[k] = tile_op_of(lower_gate(ops[gate_ops[take[k]]]), tpos);
      b.gate_first = (int)tp.gates.size();
      b.phase_first = (int)tp.phases.size();
      size_t k0 = 0;
      const int all_bits = (1 << TB) - 1;
      while (k0 < take.size()) {
        int rmask = 0;
        size_t k1 = k0;
        TPhase ph{};
        int slot_of[12];
        if (kPacked) {
          // complex64: register slot 0 is the pack bit, a tile bit that no
          // gate of the phase targets (pair kinds) or uses as a control;
          // the targets take at most the other RB - 1 slots
          int forbid = 0;
          for (; k1 < take.size(); ++k1) {
            int need = 0;
            for (int t = 0; t < top[k1].ntargets; ++t) need |= 1 << top[k1].targets[t];
            const int f = forbid | need | top[k1].cmask;
            if (__builtin_popcount(rmask | need) > RB - 1 || (f & all_bits) == all_bits) break;
            rmask |= need;
            forbid = f;
          }
          int pack = 0;
          while ((forbid >> pack) & 1) ++pack;
          for (int t = 0; t < TB && __builtin_popcount(rmask) < RB - 1; ++t)
            if (t != pack) rmask |= 1 << t;
          ph.r[0] = (uint8_t)pack;
          slot_of[pack] = 0;
          for (int t = 0, k = 1; t < TB; ++t)
            if ((rmask >> t) & 1) {
              ph.r[k] = (uint8_t)t;
              slot_of[t] = k++;
            }
          rmask |= 1 << pack;
        } else {
          for (; k1 < take.size(); ++k1) {
            int need = 0;
            for (int t = 0; t < top[k1].ntargets; ++t) need |= 1 << top[k1].targets[t];
            if (__builtin_popcount(rmask | need) > RB) break;
            rmask |= need;
          }
          for (int t = 0; t < TB && __builtin_popcount(rmask) < RB; ++t) rmask |= 1 << t;
          for (int t = 0, k = 0; t < TB; ++t)
            if ((rmask >> t) & 1) {
              ph.r[k] = (uint8_t)t;
              slot_of[t] = k++;
            }
        }
        ph.first = (int)tp.gates.size() - b.gate_first;  // relative to the block's first gate
        ph.count = (int)(k1 - k0);
        for (size_t k = k0; k < k1; ++k) {
          const TileOp& o = top[k];
          const int gi = take[k];
          TGate g{};
          g.kind = o.kind;
          g.mat = gi;
          g.gen = geo[gi].pslot >= 0 ? (uint8_t)geo[gi].gen : 0;
          g.real = real[gi];
          g.tslot = -1;
          int cm_r = 0, cm_g = 0;
          for (int t = 0; t < TB; ++t)
            if ((o.cmask >> t) & 1) {
              if ((rmask >> t) & 1) cm_r |= 1 << slot_of[t];
              else cm_g |= 1 << t;
            }
          g.cm_r = (uint8_t)cm_r;
          g.cm_g = (uint16_t)cm_g;
          if (o.kind == kTDiag) {
            g.tbit = (uint8_t)o.tgt_diag;
            if ((rmask >> o.tgt_diag) & 1) g.tslot = (int8_t)slot_of[o.tgt_diag];
          } else if (o.kind == kTSwap2) {
            const int a = slot_of[o.targets[0]], c = slot_of[o.targets[1]];
            g.s0 = (uint8_t)std::min(a, c);
            g.s1 = (uint8_t)std::max(a, c);
          } else {
            g.s0 = (uint8_t)slot_of[o.targets[0]];
          }
          g.grad = -1;
          if (g.gen) {
            g.grad = (int16_t)b.grad_gate.size();
            b.grad_gate.push_back(gi);
          }
          tp.gates.push_back(g);
        }
        tp.phases.push_back(ph);
        k0 = k1;
      }
      b.n_gates = (int)tp.gates.size() - b.gate_first;
      b.n_phases = (int)tp.phases.size() - b.phase_first;
      tp.blocks.push_back(std::move(b));
    }
    i0 = i1;
  }
  return tp;
}

// packed: the phases of the interpreted complex64 sweep, whose packs hold two
// amplitudes (slot 0 is the pack bit); otherwise all slots are targets.  The
// blocks and their gates are the same.
//
// The tiled plan with blocks per layer, or per checkpoint segment of m
// layers when that needs fewer blocks (fewer HBM passes; a block that spans
// layers holds more gates and register phases, so on a tie the per-layer
// plan is kept).
template <typename R>
TilePlan plan_tiles_best(int n, const ketgpu_op* ops, const std::vector<int>& gate_ops,
                         const std::vector<int>& layer_of, const std::vector<GateGeom>& geo,
                         const std::vector<uint8_t>& real, int m, bool packed = sizeof(R) == 4) {
  TilePlan per_layer = plan_tiles<R>(n, ops, gate_ops, layer_of, geo, real, 1, packed);
  if (m <= 1) return per_layer;
  TilePlan per_seg = plan_tiles<R>(n, ops, gate_ops, layer_of, geo, real, m, packed);
  return per_seg.blocks.size() < per_layer.blocks.size() ? std::move(per_seg) : std::move(per_layer);
}

// A call's device memory, from the library's pool, freed in stream order.
struct DevBuf : StreamScratch {
  using StreamScratch::StreamScratch;
  template <typename T>
  T* as() const {
    return static_cast<T*>(p);
  }
};

int gen_of(int type) {
  switch (type) {
    case KETGPU_RX: case KETGPU_CRX: return 1;
    case KETGPU_RY: case KETGPU_CRY: return 2;
    case KETGPU_RZ: case KETGPU_CRZ: return 3;
    case KETGPU_CP: return 4;
    default: return 0;
  }
}

// ---------------------------------------------------------------------------
// Per-block complex64 kernels compiled at run time.  The compiled sweep
// (tile_sweep_c64) interprets each block's gate records: every gate goes
// through a switch, and the register moves at its merge points dominate the
// instruction count.  Here the block's phases and gates become compile-time
// constants of a kernel generated from adj_tile.cuh: a swap is a renaming,
// each gate is straight-line arithmetic.  The kernels are compiled
// with NVRTC for sm_100a (loaded with dlopen on first use), loaded with the
// runtime's library API and cached by their source text, so a layer
// structure that repeats is compiled once per process.  When NVRTC cannot
// be loaded or a compile fails, the compiled sweep runs instead.

const char* const kTileSource =
#include "adj_tile_src.inc"
    ;

struct Nvrtc {
  using Create = int (*)(void**, const char*, const char*, int, const char* const*, const char* const*);
  using Compile = int (*)(void*, int, const char* const*);
  using SizeOf = int (*)(void*, size_t*);
  using Get = int (*)(void*, char*);
  using Destroy = int (*)(void**);
  Create create = nullptr;
  Compile compile = nullptr;
  SizeOf log_size = nullptr, cubin_size = nullptr;
  Get log = nullptr, cubin = nullptr;
  Destroy destroy = nullptr;
  bool ok = false;
  Nvrtc() {
    const char* names[] = {"libnvrtc.so.12", "libnvrtc.so", "/usr/local/cuda/lib64/libnvrtc.so.12"};
    void* h = nullptr;
    for (const char* n : names)
      if ((h = dlopen(n, RTLD_NOW | RTLD_LOCAL))) break;
    if (!h) return;
    create = reinterpret_cast<Create>(dlsym(h, "nvrtcCreateProgram"));
    compile = reinterpret_cast<Compile>(dlsym(h, "nvrtcCompileProgram"));
    log_size = reinterpret_cast<SizeOf>(dlsym(h, "nvrtcGetProgramLogSize"));
    log = reinterpret_cast<Get>(dlsym(h, "nvrtcGetProgramLog"));
    cubin_size = reinterpret_cast<SizeOf>(dlsym(h, "nvrtcGetCUBINSize"));
    cubin = reinterpret_cast<Get>(dlsym(h, "nvrtcGetCUBIN"));
    destroy = reinterpret_cast<Destroy>(dlsym(h, "nvrtcDestroyProgram"));
    ok = create && compile && log_size && log && cubin_size && cubin && destroy;
  }
};

Nvrtc& nvrtc() {
  static Nvrtc n;
  return n;
}

// AUTO uses the per-block kernels from this many qubits up.
constexpr int kJitMinQubits = 16;

std::mutex g_jit_mu;
std::map<std::string, cudaKernel_t> g_jit;  // source -> kernel (nullptr: failed)
std::string g_jit_last_log;

// Compile (once) and return the kernel "kb_tile_jit" of `src`, or nullptr.
cudaKernel_t jit_kernel(const std::string& src) {
  std::lock_guard<std::mutex> lock(g_jit_mu);
  auto it = g_jit.find(src);
  if (it != g_jit.end()) return it->second;
  cudaKernel_t k = nullptr;
  Nvrtc& nv = nvrtc();
  if (nv.ok) {
    const std::string full = std::string("#define KB_JIT 1\n") + kTileSource + src;
    void* prog = nullptr;
    if (nv.create(&prog, full.c_str(), "kb_tile_jit.cu", 0, nullptr, nullptr) == 0) {
      const char* opts[] = {"--gpu-architecture=sm_100a", "-std=c++17"};
      const int rc = nv.compile(prog, 2, opts);
      size_t ls = 0;
      nv.log_size(prog, &ls);
      std::string lg(ls, '\0');
      if (ls) nv.log(prog, &lg[0]);
      g_jit_last_log = lg;
      size_t cs = 0;
      if (rc == 0 && nv.cubin_size(prog, &cs) == 0 && cs) {
        std::vector<char> cubin(cs);
        if (nv.cubin(prog, cubin.data()) == 0) {
          cudaLibrary_t lib = nullptr;
          if (cudaLibraryLoadData(&lib, cubin.data(), nullptr, nullptr, 0, nullptr, nullptr, 0) == cudaSuccess &&
              cudaLibraryGetKernel(&k, lib, "kb_tile_jit") != cudaSuccess)
            k = nullptr;
        }
      }
      nv.destroy(&prog);
    }
  }
  cudaGetLastError();  // a failed load leaves no sticky error behind
  g_jit[src] = k;
  return k;
}

int tphys_host(int e) { return e ^ (((e >> 4) ^ (e >> 8)) & 15); }

// The kernel of one complex64 block: phases (in sweep order) and their gates
// as constants.  Parameters as tile_sweep_c64, without the phase table.
// Gradient slots per thread for a reverse block with `ngrad` gradients: the
// odd stride of the per-thread FP32 sums, or 0 for the per-tile warp
// reduction into per-warp FP64 sums (blocks with many gradients, whose
// per-thread slots would not leave room for two CTAs per SM).
constexpr int kThreadGradMax = 31;
int grad_slot_stride(int ngrad) { return ngrad > 0 && ngrad <= kThreadGradMax ? (ngrad | 1) : 0; }

std::string jit_source(const std::vector<TPhase>& phases, const std::vector<TGate>& gates, bool rev) {
  std::string o;
  auto line = [&](const std::string& x) { o += x + "\n"; };
  int ngrad_block = 0;
  for (const TGate& g : gates)
    if (g.grad >= 0) ngrad_block = std::max(ngrad_block, (int)g.grad + 1);
  const int gs = rev ? grad_slot_stride(ngrad_block) : 0;
  // Reverse: two CTAs per SM with one tile buffer each (load, compute,
  // store) beat one CTA with two buffers: the other CTA's work covers the
  // loads.  Forward: two CTAs, each prefetching its next tile.
  line("extern \"C\" __global__ void __launch_bounds__(256, 2)");
  line("kb_tile_jit(float2* psi, const float2* psi_src, float2* __restrict__ lam, uint64_t dim, kbt::TileGeom tg,");
  line("            const kbt::TGate* __restrict__ gates, int ngates, const float* __restrict__ mats,");
  line("            uint64_t mat_stride, int ngrad, double* __restrict__ partial) {");
  line("  using namespace kbt;");
  line(std::string("  constexpr bool REV = ") + (rev ? "true" : "false") + ";");
  line("  constexpr int TILE = 1 << TileCfg<float>::TB, BUF = (REV ? 2 : 1) * TILE;");
  line("  constexpr bool SINGLE = REV;  // one tile buffer");
  line("  extern __shared__ __align__(16) unsigned char tsm[];");
  line("  float2* bufs = reinterpret_cast<float2*>(tsm);");
  line("  f2* spk = reinterpret_cast<f2*>(tsm + (SINGLE ? 1 : 2) * BUF * sizeof(float2));");
  line("  float* accf = reinterpret_cast<float*>(spk + 16 * ngates);");
  line("  double* acc = reinterpret_cast<double*>(accf);");
  line("  constexpr int GS = " + std::to_string(gs) + ";  // per-thread gradient slots (0: per-warp sums)");
  line("  __shared__ uint64_t off[kTileThreads + 16];");
  line("  const int tid = threadIdx.x;");
  line("  const int set = blockIdx.y;");
  line("  float2* s = psi + (uint64_t)set * dim;  // tiles are stored here");
  line("  const float2* sin = psi_src + (uint64_t)set * dim;  // and loaded from here (psi, or a checkpoint)");
  line("  float2* l = REV ? lam + (uint64_t)set * dim : nullptr;");
  line("  c64_setup<REV>(tg, gates, ngates, mats, mat_stride, set, GS ? kTileThreads * GS : 2 * kTileWarps * ngrad,");
  line("                 off, spk, accf);");
  line("  __syncthreads();");
  line("  int cur = 0;");
  line("  if (!SINGLE && blockIdx.x < tg.n_tiles) c64_prefetch<REV>(tg, off, blockIdx.x, bufs, sin, l);");
  line("  asm volatile(\"cp.async.commit_group;\\n\" ::: \"memory\");");
  line("  for (uint64_t t = blockIdx.x; t < tg.n_tiles; t += gridDim.x) {");
  line("    float2* sp = bufs + (SINGLE ? 0 : cur) * BUF;");
  line("    float2* sl = sp + TILE;");
  line("    if (SINGLE) c64_prefetch<REV>(tg, off, t, bufs, sin, l);");
  line("    else if (t + gridDim.x < tg.n_tiles)");
  line("      c64_prefetch<REV>(tg, off, t + gridDim.x, bufs + (cur ^ 1) * BUF, sin, l);");
  line("    asm volatile(\"cp.async.commit_group;\\n\" ::: \"memory\");");
  line("    if (SINGLE) asm volatile(\"cp.async.wait_group 0;\\n\" ::: \"memory\");");
  line("    else asm volatile(\"cp.async.wait_group 1;\\n\" ::: \"memory\");");
  line("    __syncthreads();");
  constexpr int TB = TileCfg<float>::TB;
  const int nph = (int)phases.size();
  for (int k = 0; k < nph; ++k) {
    const TPhase& P = phases[rev ? nph - 1 - k : k];
    int rmask = 0;
    for (int b = 0; b < 4; ++b) rmask |= 1 << P.r[b];
    std::string gb = "0";
    for (int b = 0, kk = 0; b < TB; ++b)
      if (!((rmask >> b) & 1)) gb += " | (((tid >> " + std::to_string(kk++) + ") & 1) << " + std::to_string(b) + ")";
    line("    {");
    line("      const int gbase = " + gb + ";");
    line("      const int pg = tphys<float>(gbase);");
    line("      NatState A, L;");
    std::string pb;
    for (int b = 0; b < 4; ++b) pb += ", " + std::to_string(tphys_host(1 << P.r[b]));
    line("      c64_load_phase<REV>(sp, sl, pg" + pb + ", A, L);");
    for (int c = 0; c < P.count; ++c) {
      const int gi = rev ? P.first + P.count - 1 - c : P.first + c;
      const TGate& g = gates[gi];
      char buf[512];
      std::snprintf(buf, sizeof buf,
                    "      { constexpr TGate g{%d, %d, %d, %d, %d, %d, %d, %d, %d, %d, %d}; float part = 0.f;",
                    (int)g.kind, (int)g.s0, (int)g.s1, (int)g.tslot, (int)g.tbit, (int)g.cm_r, (int)(rev ? g.gen : 0),
                    (int)g.real, (int)g.cm_g, (int)g.grad, 0);  // mat: read from the gate table at set-up
      line(buf);
      const auto num = [](int v) { return std::to_string(v); };
      const int gen = rev ? g.gen : 0;
      const std::string coef = "spk + 16 * " + num(gi);
      std::string call;
      if (g.kind == kTPair)
        call = "part = nk_pair<" + num(g.s0) + ", " + (g.real ? "true" : "false") + ", " + num(gen) + ", REV>(A, L, g, " +
               coef + ");";
      else if (g.kind == kTPairSwap) call = "part = nk_swap<" + num(g.s0) + ", REV>(A, L, g);";
      else if (g.kind == kTSwap2) call = "part = nk_swap2<" + num(g.s0) + ", " + num(g.s1) + ", REV>(A, L, g);";
      else
        call = "part = nk_diag<" + num(g.tslot) + ", " + num(gen == 3 || gen == 4 ? gen : 0) + ", REV>(A, L, g, " + coef +
               ", gbase);";
      if (g.cm_g) line("        if ((gbase & " + std::to_string((int)g.cm_g) + ") == " + std::to_string((int)g.cm_g) +
                       ") " + call);
      else line("        " + call);
      if (rev && g.grad >= 0) {
        if (gs) line("        c64_grad_slot(accf, GS, " + std::to_string((int)g.grad) + ", part);");
        else line("        c64_grad(acc, ngrad, " + std::to_string((int)g.grad) + ", part);");
      }
      line("        (void)part; }");
    }
    line("      c64_store_phase<REV>(sp, sl, pg" + pb + ", A, L);");
    line("      __syncthreads();");
    line("    }");
  }
  line("    c64_store_tile<REV>(tg, off, t, sp, sl, s, l);");
  line("    __syncthreads();");
  line("    cur ^= 1;");
  line("  }");
  line("  asm volatile(\"cp.async.wait_all;\\n\" ::: \"memory\");");
  if (gs) line("  __syncthreads();");
  line(gs ? "  c64_flush_slots(accf, GS, ngrad, partial, set);" : "  if (REV) c64_flush(acc, ngrad, partial, set);");
  line("}");
  return o;
}

size_t jit_smem(bool rev, int ngates, int ngrad) {
  // forward: two buffers of psi; reverse: one buffer of psi and lambda, and
  // the gradient sums (per-thread FP32 slots or per-warp FP64)
  const int gs = grad_slot_stride(ngrad);
  const size_t acc = !rev ? 0 : gs ? (size_t)kTileThreads * gs * 4 : (size_t)kTileWarps * ngrad * 8;
  return 2 * (size_t{1} << TileCfg<float>::TB) * sizeof(float2) + (size_t)ngates * 16 * sizeof(f2) + acc;
}

// Dynamic shared memory of one tiled sweep launch (see the kernels).
template <typename R>
size_t tile_smem(bool rev, int ngates, int ngrad) {
  using T = typename C2T<R>::T;
  const size_t tile = (size_t{1} << TileCfg<R>::TB) * sizeof(T);
  if (sizeof(R) == 8)
    return 2 * tile + (size_t)ngates * (sizeof(TGate) + 8 * sizeof(R)) + (rev ? (size_t)kTileWarps * ngrad * 64 : 0);
  return (rev ? 4 : 2) * tile + (size_t)ngates * (16 * sizeof(f2) + sizeof(TGate)) +
         (rev ? (size_t)kTileWarps * ngrad * 8 : 0);
}

std::atomic<uint64_t> g_jit_launches{0};

template <typename R, bool REV>
void launch_tile(dim3 grid, cudaStream_t st, typename C2T<R>::T* psi, typename C2T<R>::T* lam, uint64_t dim,
                 const TBlock& b, const TGate* gates, const TPhase* phases, const R* mats, uint64_t chunk,
                 double* partial, cudaKernel_t jit = nullptr, const typename C2T<R>::T* psi_src = nullptr,
                 bool all_tiles = false) {
  TileGeom tg = b.geom;
  if (!all_tiles) tg.n_tiles = std::min(tg.n_tiles, b.active_tiles);
  const int ngrad = REV ? (int)b.grad_gate.size() : 0;
  if constexpr (sizeof(R) == 4) {
    if (jit) {
      float2* a0 = psi;
      const float2* asrc = psi_src ? psi_src : psi;
      float2* a1 = lam;
      uint64_t d = dim;
      const TGate* gp = gates + b.gate_first;
      int ng = b.n_gates;
      const float* mp = mats;
      uint64_t ms = chunk;
      int ngr = ngrad;
      double* pp = partial;
      void* args[] = {&a0, &asrc, &a1, &d, &tg, &gp, &ng, &mp, &ms, &ngr, &pp};
      KB_CUDA(cudaLaunchKernel(reinterpret_cast<const void*>(jit), grid, dim3(kTileThreads), args,
                               jit_smem(REV, b.n_gates, ngrad), st));
      count_launch();
      g_jit_launches.fetch_add(1, std::memory_order_relaxed);
      return;
    }
  }
  if (psi_src && psi_src != psi)  // the interpreted sweeps load in place only
    KB_CUDA(cudaMemcpyAsync(psi, psi_src, dim * sizeof(typename C2T<R>::T) * grid.y, cudaMemcpyDeviceToDevice, st));
  const size_t smem = tile_smem<R>(REV, b.n_gates, ngrad);
  if constexpr (sizeof(R) == 4)
    tile_sweep_c64<REV><<<grid, kTileThreads, smem, st>>>(psi, lam, dim, tg, gates + b.gate_first, b.n_gates,
                                                          phases + b.phase_first, b.n_phases, mats, chunk, ngrad,
                                                          partial);
  else
    tile_sweep<R, REV><<<grid, kTileThreads, smem, st>>>(psi, lam, dim, tg, gates + b.gate_first, b.n_gates,
                                                         phases + b.phase_first, b.n_phases, mats, chunk, ngrad,
                                                         partial);
  count_launch();
}

// The terms and, per 32 of them, a mask a thread.
size_t ham_smem(int nterms) {
  return sizeof(HamTerm) * (size_t)nterms + sizeof(uint32_t) * kAThreads * (size_t)((nterms + 31) / 32);
}

template <typename R>
void run_adjoint(int n, const ketgpu_op* ops, uint64_t nops, const int32_t* pidx, const double* params,
                 uint64_t nparams, uint64_t batch, const std::vector<uint64_t>& flip,
                 const std::vector<uint64_t>& sign, const std::vector<int>& phq, const double* coeffs,
                 int ckpt_every, int method, double* values, double* grads) {
  using T = typename C2T<R>::T;
  constexpr int TB = TileCfg<R>::TB;
  const uint64_t dim = uint64_t{1} << n;
  const int T_ = (int)flip.size();
  const bool resident = method == KETGPU_ADJOINT_AUTO && n <= kResMaxQubits;
  const bool tiled = method == KETGPU_ADJOINT_TILED || method == KETGPU_ADJOINT_TILED_JIT ||
                     (method == KETGPU_ADJOINT_AUTO && n >= TB && !resident);
  const bool ham_inside = resident && dim * (uint64_t)T_ <= kResHamWork;
  // per-block compiled kernels: complex64, asked for, or chosen at sizes
  // where the sweeps take long enough to repay a compile
  const bool want_jit = sizeof(R) == 4 && tiled &&
                        (method == KETGPU_ADJOINT_TILED_JIT || (method == KETGPU_ADJOINT_AUTO && n >= kJitMinQubits));
  if (tiled && n < TB)
    fail(KETGPU_ERR_INVALID, "adjoint: the tiled sweep needs at least " + std::to_string(TB) + " qubits");
  // gates (unitary ops) and layer boundaries (barriers)
  std::vector<int> gate_ops;
  std::vector<int> layer_of;
  int layer = 0;
  for (uint64_t i = 0; i < nops; ++i) {
    if (ops[i].type == KETGPU_BARRIER) {
      ++layer;
      continue;
    }
    if (!is_unitary(ops[i].type)) continue;
    gate_ops.push_back((int)i);
    layer_of.push_back(layer);
  }
  const int n_layers = layer + 1;
  const int m = ckpt_every > 0 ? ckpt_every : n_layers;
  const int n_ckpt = (n_layers + m - 1) / m;  // segment starts at layers 0, m, 2m, ...
  const size_t G = gate_ops.size();

  // memory: chunk of the batch that fits in ~60% of free memory (not asked
  // for when the states take little)
  const size_t per_set = dim * sizeof(T) * (2 + (size_t)n_ckpt);
  uint64_t chunk = batch;
  if (batch && per_set > kPoolKeep / batch) {
    size_t free_b = 0, total_b = 0;
    KB_CUDA(cudaMemGetInfo(&free_b, &total_b));
    if ((uint64_t)((free_b * 0.6) / per_set) < batch) {  // first take back what is kept between calls
      release_kept();
      KB_CUDA(cudaMemGetInfo(&free_b, &total_b));
    }
    chunk = std::max<uint64_t>(1, (uint64_t)((free_b * 0.6) / per_set));
  }
  chunk = std::min<uint64_t>(chunk, batch);
  chunk = std::min<uint64_t>(chunk, 65535);

  int dev = 0;
  KB_CUDA(cudaGetDevice(&dev));
  // psi, lambda and the checkpoints of every set of the chunk (ends after the
  // lease, which waits for the stream)
  Workspace work(per_set * chunk, dev);
  StreamLease lease(dev);
  const cudaStream_t st = lease.s;
  T* const psi = static_cast<T*>(work.p);
  T* const lam = psi + dim * chunk;
  T* const ck = lam + dim * chunk;
  const int blocks = resident ? 1
                              : (int)std::min<uint64_t>(std::max<uint64_t>(1, (dim / 2 + kAThreads - 1) / kAThreads), 592);
  const int ham_blocks = (int)std::min<uint64_t>(std::max<uint64_t>(1, (dim / 2 + kAThreads - 1) / kAThreads), 592);
  // the gates' matrices in the precision their sweep reads
  DevBuf mats((tiled ? sizeof(R) : sizeof(double)) * 8 * chunk * std::max<size_t>(G, 1), dev, st);
  DevBuf hmeta(sizeof(uint64_t) * 2 * T_ + sizeof(int) * T_ + sizeof(double) * T_ + 64, dev, st);
  if (ham_inside) {  // the terms as the resident form takes them, i^q folded in
    static_assert(sizeof(ResTerm) <= 28, "the room of a term");
    std::vector<ResTerm> h(T_);
    for (int t = 0; t < T_; ++t) {
      const int q = phq[t] & 3;
      h[t] = {(uint32_t)flip[t], (uint32_t)sign[t], q >= 2 ? -coeffs[t] : coeffs[t], (uint32_t)(q & 1), 0};
    }
    KB_CUDA(cudaMemcpyAsync(hmeta.p, h.data(), sizeof(ResTerm) * h.size(), cudaMemcpyHostToDevice, st));
  } else {
    std::vector<char> h(sizeof(uint64_t) * 2 * T_ + sizeof(int) * T_ + sizeof(double) * T_);
    std::memcpy(h.data(), flip.data(), 8 * T_);
    std::memcpy(h.data() + 8 * T_, sign.data(), 8 * T_);
    std::memcpy(h.data() + 16 * T_, coeffs, 8 * T_);  // 8-byte values first, whatever T_ is
    std::memcpy(h.data() + 24 * T_, phq.data(), 4 * T_);
    KB_CUDA(cudaMemcpyAsync(hmeta.p, h.data(), h.size(), cudaMemcpyHostToDevice, st));
  }
  // the terms for ham_half: grouped by the top qubit of their flip (0: same
  // half, 1: other half), sorted by class within a group, the phase i^q and
  // the signs that do not depend on the output folded into the coefficients
  constexpr int kHamPer = 16 / (int)sizeof(T);
  std::unique_ptr<DevBuf> d_ham;
  HamClasses hcls[2] = {};
  const bool ham_split = !ham_inside && T_ <= kHamSmemTerms && dim >= 2 * (uint64_t)kHamPer;
  if (ham_split) {
    std::vector<HamTerm> ht;
    for (int pass = 0; pass < 2; ++pass) {
      const size_t begin = ht.size();
      for (int c = 0; c < 4; ++c) {
        for (int t = 0; t < T_; ++t) {
          if ((int)((flip[t] >> (n - 1)) & 1) != pass) continue;
          const int q = phq[t] & 3;  // i^q: 1, i, -1, -i
          if (2 * (q & 1) + (kHamPer > 1 ? (int)(flip[t] & 1) : 0) != c) continue;
          HamTerm x;
          x.flip = flip[t];
          x.sign = sign[t];
          const bool neg = (q >= 2) != (bool)(__builtin_popcountll(flip[t] & sign[t]) & 1);
          x.c0 = neg ? -coeffs[t] : coeffs[t];
          x.c1 = (sign[t] & 1) ? -x.c0 : x.c0;
          ht.push_back(x);
        }
        hcls[pass].end[c] = (int)(ht.size() - begin);
      }
    }
    d_ham = std::make_unique<DevBuf>(sizeof(HamTerm) * std::max(T_, 1), dev, st);
    KB_CUDA(cudaMemcpyAsync(d_ham->p, ht.data(), sizeof(HamTerm) * T_, cudaMemcpyHostToDevice, st));
    static OncePerDevice ham_attr;  // one for each R
    ham_attr(dev, [] {
      KB_CUDA(cudaFuncSetAttribute(ham_half<R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)ham_smem(kHamSmemTerms)));
    });
  }
  // ham_half grid: about one set's worth of resident CTAs per half
  const uint64_t ham_words = dim / 2 / kHamPer;
  const int ham_ctas = (int)std::min<uint64_t>(std::max<uint64_t>(1, (ham_words + kAThreads - 1) / kAThreads), 148ull * 8);
  const uint64_t* d_flip = hmeta.as<uint64_t>();
  const uint64_t* d_sign = d_flip + T_;
  const double* d_coef = reinterpret_cast<const double*>(d_sign + T_);
  const int* d_q = reinterpret_cast<const int*>(d_coef + T_);

  // geometry of every gate (independent of the parameters)
  std::vector<GateGeom> geo(G);
  for (size_t gi = 0; gi < G; ++gi) {
    const ketgpu_op& o = ops[gate_ops[gi]];
    const Pass p = lower_gate(o);
    GateGeom& g = geo[gi];
    g.nfixed = p.nfixed;
    for (int j = 0; j < 3; ++j) g.fixed[j] = p.fixed[j];
    g.count = dim >> p.nfixed;
    g.p0 = p.p0;
    g.p1 = p.p1;
    g.kind = p.kind == PassKind::Phase ? 2 : (p.mode == kPairSwap ? 1 : 0);
    const int32_t pi = pidx ? pidx[gate_ops[gi]] : -1;
    g.gen = pi >= 0 ? gen_of(o.type) : 0;
    g.pslot = pi;
    if (pi >= 0 && g.gen == 0) fail(KETGPU_ERR_INVALID, "adjoint: parameterised op must be Rx/Ry/Rz/CRx/CRy/CRz/CP");
    if (pi >= (int32_t)nparams) fail(KETGPU_ERR_OUT_OF_RANGE, "adjoint: parameter index out of range");
  }
  if (!batch) return;  // no sets: the arguments have been checked

  // the gates as gate_matrices takes them: 2x2 U, row-major, FP64
  // interleaved; the tiled sweep stores a phase gate as diag(1, phase)
  std::vector<AdjGate> agates(G);
  std::vector<uint8_t> real(G, 0);  // the matrix is real for every set
  for (size_t gi = 0; gi < G; ++gi) {
    const ketgpu_op& o = ops[gate_ops[gi]];
    AdjGate& a = agates[gi];
    a = AdjGate{};
    a.pslot = geo[gi].pslot;
    if (a.pslot >= 0) {
      a.kind = geo[gi].gen;  // 1 X, 2 Y, 3 Z, 4 P11
      real[gi] = a.kind == 2;
      continue;
    }
    const Pass p = lower_gate(o);
    cplx mm[4] = {p.m[0], p.m[1], p.m[2], p.m[3]};
    if (tiled && p.kind == PassKind::Phase) {
      mm[3] = p.m[0];
      mm[0] = cplx(1.0, 0.0);
      mm[1] = mm[2] = cplx(0.0, 0.0);
    }
    bool r = true;
    for (int j = 0; j < 4; ++j) {
      a.m[2 * j] = mm[j].real();
      a.m[2 * j + 1] = mm[j].imag();
      r = r && mm[j].imag() == 0.0;
    }
    real[gi] = r;
  }
  if (tiled) {
    // An uncontrolled Rz loses its phase e^{-it/2}: a phase common to psi and
    // lambda = H psi drops out of the expectation and of every gradient, and
    // diag(1, e^{it}) leaves half of the amplitudes alone.  Diagonal gates
    // with a 1 for target bit 0 are marked for the sweeps.
    for (size_t gi = 0; gi < G; ++gi) {
      const int type = ops[gate_ops[gi]].type;
      AdjGate& a = agates[gi];
      if (type == KETGPU_RZ) {
        if (a.pslot >= 0) {
          a.kind = 5;
        } else {
          const double t = ops[gate_ops[gi]].p[0];
          a.m[0] = 1.0;
          a.m[1] = 0.0;
          a.m[6] = std::cos(t);
          a.m[7] = std::sin(t);
        }
      }
      if (is_diagonal_gate(type)) real[gi] = type != KETGPU_CRZ;
    }
  }
  DevBuf d_agates(sizeof(AdjGate) * std::max<size_t>(G, 1), dev, st);
  if (G) KB_CUDA(cudaMemcpyAsync(d_agates.p, agates.data(), sizeof(AdjGate) * G, cudaMemcpyHostToDevice, st));
  DevBuf d_params(sizeof(double) * std::max<uint64_t>(chunk * nparams, 1), dev, st);

  // the gates as the resident form takes them
  std::unique_ptr<DevBuf> d_res;
  const int res_threads = (int)std::min<uint64_t>(kResThreads, std::max<uint64_t>(32, dim / 4));
  const size_t res_smem = resident_smem(dim * sizeof(T), res_threads, sizeof(R));
  if (resident) {
    std::vector<ResGate> rg(G);
    for (size_t gi = 0; gi < G; ++gi) {
      const GateGeom& g = geo[gi];
      ResGate& r = rg[gi];
      r = ResGate{};
      r.p0 = (uint32_t)g.p0;
      r.p1 = (uint32_t)g.p1;
      for (int j = 0; j < g.nfixed; ++j) r.fixed[j] = (int16_t)g.fixed[j];
      r.nfixed = (uint8_t)g.nfixed;
      r.kind = (uint8_t)g.kind;
      r.gen = (uint8_t)g.gen;
      r.grad = g.pslot >= 0;
      // the state after the last gate of a segment starts the next one
      const int seg = layer_of[gi] / m;
      if (gi + 1 < G && layer_of[gi + 1] / m != seg && seg + 1 < n_ckpt) r.ck = seg + 1;
    }
    d_res = std::make_unique<DevBuf>(sizeof(ResGate) * std::max<size_t>(G, 1), dev, st);
    if (G) KB_CUDA(cudaMemcpyAsync(d_res->p, rg.data(), sizeof(ResGate) * G, cudaMemcpyHostToDevice, st));
    // the most that any size takes: calls of other sizes may be between here
    // and their launch on other threads
    static OncePerDevice res_attr;  // one for each R
    res_attr(dev, [] {
      KB_CUDA(cudaFuncSetAttribute(adjoint_resident<R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)resident_smem(sizeof(T) << kResMaxQubits, kResThreads, sizeof(R))));
    });
  }

  // tiled plan
  TilePlan tp;
  std::vector<cudaKernel_t> jit_fwd, jit_rev;
  std::unique_ptr<DevBuf> d_tgates, d_tphases;
  int gx = 1;
  size_t grad_doubles = 0;
  if (tiled) {
    tp = plan_tiles_best<R>(n, ops, gate_ops, layer_of, geo, real, m);
    d_tgates = std::make_unique<DevBuf>(sizeof(TGate) * std::max<size_t>(tp.gates.size(), 1), dev, st);
    d_tphases = std::make_unique<DevBuf>(sizeof(TPhase) * std::max<size_t>(tp.phases.size(), 1), dev, st);
    if (!tp.gates.empty())
      KB_CUDA(cudaMemcpyAsync(d_tgates->p, tp.gates.data(), sizeof(TGate) * tp.gates.size(),
                              cudaMemcpyHostToDevice, st));
    if (!tp.phases.empty())
      KB_CUDA(cudaMemcpyAsync(d_tphases->p, tp.phases.data(), sizeof(TPhase) * tp.phases.size(),
                              cudaMemcpyHostToDevice, st));
    if (want_jit && nvrtc().ok) {
      jit_fwd.assign(tp.blocks.size(), nullptr);
      jit_rev.assign(tp.blocks.size(), nullptr);
      const TilePlan tj = plan_tiles_best<R>(n, ops, gate_ops, layer_of, geo, real, m, false);
      for (size_t bi = 0; bi < tj.blocks.size(); ++bi) {
        const TBlock& b = tj.blocks[bi];
        const std::vector<TPhase> ph(tj.phases.begin() + b.phase_first,
                                     tj.phases.begin() + b.phase_first + b.n_phases);
        const std::vector<TGate> gs(tj.gates.begin() + b.gate_first, tj.gates.begin() + b.gate_first + b.n_gates);
        jit_fwd[bi] = jit_kernel(jit_source(ph, gs, false));
        jit_rev[bi] = jit_kernel(jit_source(ph, gs, true));
        if (jit_fwd[bi])
          KB_CUDA(cudaFuncSetAttribute(reinterpret_cast<const void*>(jit_fwd[bi]),
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)jit_smem(false, kMaxBlockGates, 0)));
        if (jit_rev[bi])
          KB_CUDA(cudaFuncSetAttribute(reinterpret_cast<const void*>(jit_rev[bi]),
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)std::max(jit_smem(true, kMaxBlockGates, kMaxBlockGrads),
                                                     jit_smem(true, kMaxBlockGates, kThreadGradMax))));
      }
    }
    const uint64_t n_tiles = uint64_t{1} << (n - TB);
    // From |0...0>, psi after block b is zero beyond the indices below the
    // highest qubit that gates have acted on so far, and the reverse sweep
    // needs lambda only where psi is nonzero: block b runs on that many tiles
    // (with finite numbers: 0 * inf).  At 24 qubits the first layer's three
    // blocks cover 1, 64 and all 4096 tiles.
    bool finite = true;
    for (uint64_t i = 0; i < batch * nparams && finite; ++i) finite = std::isfinite(params[i]);
    for (int t = 0; t < T_ && finite; ++t) finite = std::isfinite(coeffs[t]);
    for (int gi : gate_ops)
      for (double v : ops[gi].p) finite = finite && std::isfinite(v);
    int top = 0;
    for (TBlock& b : tp.blocks) {
      for (int k = 0; k < b.n_gates; ++k) {
        const ketgpu_op& o = ops[gate_ops[tp.gates[b.gate_first + k].mat]];
        for (int j = 0; j < gate_arity(o.type); ++j) top = std::max(top, o.q[j] + 1);
      }
      int outside = 0;  // qubits below `top` that are not in the tile
      for (int q = 0; q < top; ++q) outside += std::find(b.geom.pos, b.geom.pos + TB, q) == b.geom.pos + TB;
      b.active_tiles = finite ? uint64_t{1} << outside : n_tiles;
    }
    // About eight rounds of every resident CTA (two per SM) over the chunk's
    // sets, in whole rounds where the set count allows: a grid of 10 x 64
    // CTAs on 296 slots ran two full rounds and a third of 48 CTAs, leaving
    // most SMs idle for a third of each sweep.
    int sms = 148;
    KB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const uint64_t slots = 2ull * (uint64_t)sms;
    gx = (int)std::min<uint64_t>(n_tiles, std::max<uint64_t>(1, (8 * slots + chunk / 2) / chunk));
    for (TBlock& b : tp.blocks) {
      b.part_off = grad_doubles;
      grad_doubles += b.grad_gate.size() * chunk * (size_t)gx;
    }
    static OncePerDevice tile_attr;  // one for each R
    tile_attr(dev, [] {
      const int smem_rev = (int)tile_smem<R>(true, kMaxBlockGates, kMaxBlockGrads);
      const int smem_fwd = (int)tile_smem<R>(false, kMaxBlockGates, 0);
      if constexpr (sizeof(R) == 4) {
        KB_CUDA(cudaFuncSetAttribute(tile_sweep_c64<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_rev));
        KB_CUDA(cudaFuncSetAttribute(tile_sweep_c64<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_fwd));
      } else {
        KB_CUDA(cudaFuncSetAttribute(tile_sweep<R, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_rev));
        KB_CUDA(cudaFuncSetAttribute(tile_sweep<R, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_fwd));
      }
    });
  }
  const int per_value = ham_inside ? 1 : ham_split ? 2 * ham_ctas : ham_blocks;
  const size_t ham_doubles = chunk * (size_t)per_value;
  // gradient partials (tiled: per block; per-gate: [gate][set][block]), then
  // the expectation partials
  const size_t grad_region = tiled ? grad_doubles : (size_t)G * chunk * blocks;
  DevBuf part(sizeof(double) * (grad_region + ham_doubles), dev, st);
  double* d_ham_part = part.as<double>() + grad_region;

  // The pieces of every parameter's gradient, then those of the expectation.
  // (A gate's partials: [gate][set][CTA] tiled within its block, per gate
  // [gate][set][CTA].)
  const int per_grad = tiled ? gx : blocks;
  std::vector<AdjPiece> pieces;
  std::vector<int32_t> first(nparams + 3, 0);
  {
    std::vector<std::vector<AdjPiece>> by_param(nparams);
    auto add = [&](size_t gi, uint64_t at, uint64_t stride) {
      by_param[geo[gi].pslot].push_back({at, stride, geo[gi].gen == 4 ? -2.0 : 1.0});
    };
    if (tiled) {
      for (const TBlock& blk : tp.blocks) {
        const size_t ng = blk.grad_gate.size();
        for (size_t k = 0; k < ng; ++k)
          add((size_t)blk.grad_gate[k], blk.part_off + k * (size_t)gx, (uint64_t)ng * gx);
      }
    } else {
      for (size_t gi = 0; gi < G; ++gi)
        if (geo[gi].pslot >= 0) add(gi, (uint64_t)gi * chunk * blocks, (uint64_t)blocks);
    }
    for (uint64_t k = 0; k < nparams; ++k) {
      pieces.insert(pieces.end(), by_param[k].begin(), by_param[k].end());
      first[k + 1] = (int32_t)pieces.size();
    }
    // the expectation, as a one-result list of its own
    first[nparams + 1] = (int32_t)pieces.size();
    pieces.push_back({(uint64_t)grad_region, (uint64_t)per_value, 1.0});
    first[nparams + 2] = (int32_t)pieces.size();
  }
  DevBuf d_pieces(sizeof(AdjPiece) * pieces.size() + sizeof(int32_t) * first.size(), dev, st);
  const AdjPiece* dp = d_pieces.as<AdjPiece>();
  const int32_t* df = reinterpret_cast<const int32_t*>(dp + pieces.size());
  KB_CUDA(cudaMemcpyAsync(d_pieces.p, pieces.data(), sizeof(AdjPiece) * pieces.size(), cudaMemcpyHostToDevice, st));
  KB_CUDA(cudaMemcpyAsync(const_cast<int32_t*>(df), first.data(), sizeof(int32_t) * first.size(),
                          cudaMemcpyHostToDevice, st));
  DevBuf d_result(sizeof(double) * chunk * (nparams + 1), dev, st);
  std::vector<double> hresult;
  for (uint64_t b0 = 0; b0 < batch; b0 += chunk) {
    const uint64_t nb = std::min(chunk, batch - b0);
    if (nparams)
      KB_CUDA(cudaMemcpyAsync(d_params.p, params + b0 * nparams, sizeof(double) * nb * nparams,
                              cudaMemcpyHostToDevice, st));
    if (G) {
      const unsigned mb = (unsigned)((G * nb + 127) / 128);
      if (tiled)
        gate_matrices<R><<<mb, 128, 0, st>>>(d_agates.as<AdjGate>(), (int)G, d_params.as<double>(), nparams, nb,
                                             chunk, 1, mats.as<R>());
      else
        gate_matrices<double><<<mb, 128, 0, st>>>(d_agates.as<AdjGate>(), (int)G, d_params.as<double>(), nparams, nb,
                                                  chunk, 0, mats.as<double>());
      count_launch();
    }
    // With every block compiled, checkpoints cost no copies: the block
    // before a checkpoint writes its tiles into the checkpoint, the next
    // block reads them from there and writes psi (and in the reverse sweep
    // the first block of a segment reads psi from its checkpoint).
    bool ck_direct = tiled && !jit_fwd.empty();
    for (size_t bi = 0; ck_direct && bi < jit_fwd.size(); ++bi) ck_direct = jit_fwd[bi] && jit_rev[bi];
    auto ck_at = [&](int k) { return ck + (size_t)k * chunk * dim; };
    // forward
    T* ground = ck_direct ? ck_at(0) : psi;
    // (a block that runs on part of the tiles leaves the rest of psi as it is)
    if (ck_direct) KB_CUDA(cudaMemsetAsync(psi, 0, dim * sizeof(T) * nb, st));
    if (!resident) {
      KB_CUDA(cudaMemsetAsync(ground, 0, dim * sizeof(T) * nb, st));
      ground_batch<R><<<(unsigned)nb, 1, 0, st>>>(ground, dim);
      count_launch();
    }
    auto run_resident = [&](int phases) {
      adjoint_resident<R><<<(unsigned)nb, res_threads, res_smem, st>>>(
          psi, lam, ck, n, d_res->as<ResGate>(), (int)G, mats.as<double>(), chunk, hmeta.as<ResTerm>(), T_, phases,
          part.as<double>(), d_ham_part);
      count_launch();
    };
    // checkpoint k = the state at the start of layer k*m
    int next_ck = 0;
    auto store_ck = [&]() {
      KB_CUDA(cudaMemcpyAsync(ck + (size_t)next_ck * chunk * dim, psi, dim * sizeof(T) * nb,
                              cudaMemcpyDeviceToDevice, st));
      ++next_ck;
    };
    if (resident) {
      run_resident(ham_inside ? kResForward | kResHam | kResReverse : kResForward);
    } else if (ck_direct) {
      const int B = (int)tp.blocks.size();
      const T* cur = ground;  // where the state lives now
      next_ck = 1;            // checkpoint 0 is the ground state
      for (int bi = 0; bi < B; ++bi) {
        const TBlock& b = tp.blocks[bi];
        if (cur != psi && next_ck < n_ckpt && next_ck * m <= b.layer) {
          // more checkpoints due here than blocks between them
          KB_CUDA(cudaMemcpyAsync(psi, cur, dim * sizeof(T) * nb, cudaMemcpyDeviceToDevice, st));
          cur = psi;
        }
        while (cur == psi && next_ck < n_ckpt && next_ck * m <= b.layer) store_ck();
        T* out = psi;
        if (bi + 1 < B && next_ck < n_ckpt && next_ck * m <= tp.blocks[bi + 1].layer) out = ck_at(next_ck++);
        dim3 grid((unsigned)gx, (unsigned)nb);
        launch_tile<R, false>(grid, st, out, nullptr, dim, b, d_tgates->as<TGate>(), d_tphases->as<TPhase>(),
                              mats.as<R>(), chunk, nullptr, jit_fwd[bi], cur, out != psi);
        cur = out;
      }
      if (cur != psi)
        KB_CUDA(cudaMemcpyAsync(psi, cur, dim * sizeof(T) * nb, cudaMemcpyDeviceToDevice, st));
    } else if (tiled) {
      for (const TBlock& b : tp.blocks) {
        while (next_ck < n_ckpt && next_ck * m <= b.layer) store_ck();
        dim3 grid((unsigned)gx, (unsigned)nb);
        launch_tile<R, false>(grid, st, psi, nullptr, dim, b, d_tgates->as<TGate>(), d_tphases->as<TPhase>(),
                              mats.as<R>(), chunk, nullptr,
                              jit_fwd.empty() ? nullptr : jit_fwd[&b - tp.blocks.data()]);
      }
    } else {
      for (size_t gi = 0; gi < G; ++gi) {
        while (next_ck < n_ckpt && next_ck * m <= layer_of[gi]) store_ck();
        dim3 grid((unsigned)blocks, (unsigned)nb);
        fwd_gate<R><<<grid, kAThreads, 0, st>>>(psi, dim, geo[gi], mats.as<double>() + gi * chunk * 8);
        count_launch();
      }
    }
    while (!resident && next_ck < n_ckpt) store_ck();
    KB_CUDA(cudaGetLastError());
    // lambda = H psi and <H>
    if (!ham_inside) {
      if (ham_split) {
        KB_CUDA(cudaMemsetAsync(d_ham_part, 0, sizeof(double) * ham_doubles, st));
        const int g0 = hcls[0].end[3], g1 = hcls[1].end[3];
        dim3 hgrid((unsigned)ham_ctas, (unsigned)nb);
        for (int h = 0; h < 2; ++h) {
          if (g0 > 0) {
            ham_half<R><<<hgrid, kAThreads, ham_smem(g0), st>>>(psi, lam, dim, h, 1, g1 == 0 ? 1 : 0,
                                                                d_ham->as<HamTerm>(), hcls[0], d_ham_part);
            count_launch();
          }
          if (g1 > 0) {
            ham_half<R><<<hgrid, kAThreads, ham_smem(g1), st>>>(psi, lam, dim, h, g0 == 0 ? 1 : 0, 1,
                                                                d_ham->as<HamTerm>() + g0, hcls[1], d_ham_part);
            count_launch();
          }
        }
      } else {
        dim3 grid((unsigned)ham_blocks, (unsigned)nb);
        ham_apply<R><<<grid, kAThreads, 0, st>>>(psi, lam, dim, d_flip, d_sign, d_q, d_coef, T_,
                                                 d_ham_part);
        count_launch();
      }
    }
    // reverse sweep; at the last gate (block) of each segment, walking
    // backwards, psi is reset to the checkpoint of the segment's end
    if (resident) {
      if (!ham_inside) run_resident(kResReverse);
    } else if (tiled) {
      const int B = (int)tp.blocks.size();
      for (int bi = B; bi-- > 0;) {
        const TBlock& b = tp.blocks[bi];
        const int seg = b.layer / m;
        const T* src = psi;
        if (bi + 1 < B && tp.blocks[bi + 1].layer / m != seg && seg + 1 < n_ckpt) {
          if (ck_direct) src = ck_at(seg + 1);
          else
            KB_CUDA(cudaMemcpyAsync(psi, ck + (size_t)(seg + 1) * chunk * dim, dim * sizeof(T) * nb,
                                    cudaMemcpyDeviceToDevice, st));
        }
        dim3 grid((unsigned)gx, (unsigned)nb);
        launch_tile<R, true>(grid, st, psi, lam, dim, b, d_tgates->as<TGate>(),
                             d_tphases->as<TPhase>(), mats.as<R>(), chunk, part.as<double>() + b.part_off,
                             jit_rev.empty() ? nullptr : jit_rev[bi], src);
      }
    } else {
      for (size_t gi = G; gi-- > 0;) {
        const int seg = layer_of[gi] / m;
        if (gi + 1 < G && layer_of[gi + 1] / m != seg && seg + 1 < n_ckpt) {
          KB_CUDA(cudaMemcpyAsync(psi, ck + (size_t)(seg + 1) * chunk * dim, dim * sizeof(T) * nb,
                                  cudaMemcpyDeviceToDevice, st));
        }
        dim3 grid((unsigned)blocks, (unsigned)nb);
        rev_gate<R><<<grid, kAThreads, 0, st>>>(psi, lam, dim, geo[gi],
                                                mats.as<double>() + gi * chunk * 8,
                                                part.as<double>() + gi * chunk * blocks);
        count_launch();
      }
    }
    KB_CUDA(cudaGetLastError());
    auto sums = [&](const int32_t* list, int nresults, int count, double* out) {
      const uint64_t warps = (uint64_t)nresults * nb;
      sum_partials<<<(unsigned)((warps + 3) / 4), 128, 0, st>>>(part.as<double>(), dp, list, nresults, nb, count, out);
      count_launch();
    };
    double* d_values = d_result.as<double>() + chunk * nparams;
    if (nparams) sums(df, (int)nparams, per_grad, d_result.as<double>());
    sums(df + nparams + 1, 1, per_value, d_values);
    KB_CUDA(cudaGetLastError());
    hresult.resize(nb * (nparams + 1));
    if (nparams)
      KB_CUDA(cudaMemcpyAsync(hresult.data(), d_result.p, sizeof(double) * nb * nparams, cudaMemcpyDeviceToHost, st));
    KB_CUDA(cudaMemcpyAsync(hresult.data() + nb * nparams, d_values, sizeof(double) * nb, cudaMemcpyDeviceToHost, st));
    KB_CUDA(cudaStreamSynchronize(st));
    std::copy(hresult.begin(), hresult.begin() + (std::ptrdiff_t)(nb * nparams), grads + b0 * nparams);
    std::copy(hresult.begin() + (std::ptrdiff_t)(nb * nparams), hresult.end(), values + b0);
  }
}

}  // namespace
}  // namespace kb

using namespace kb;

namespace {
int adjoint_entry(int32_t n, const ketgpu_op* ops, uint64_t n_ops, const int32_t* param_index, const double* params,
                  uint64_t n_params, uint64_t batch, const double* coeffs, const char* const* paulis,
                  uint64_t n_terms, int32_t precision, int32_t checkpoint_every, int32_t method, double* values,
                  double* grads) {
  try {
    if (n < 1 || n > 34) fail(KETGPU_ERR_INVALID, "adjoint: n_qubits must be in [1, 34]");
    if (!ops || !values || !grads || (n_params && !params) || !coeffs || !paulis || n_terms == 0)
      fail(KETGPU_ERR_INVALID, "adjoint: null argument");
    if (method < KETGPU_ADJOINT_AUTO || method > KETGPU_ADJOINT_TILED_JIT) fail(KETGPU_ERR_INVALID, "adjoint: bad method");
    validate_ops(n, ops, n_ops);
    std::vector<uint64_t> flip(n_terms), sign(n_terms);
    std::vector<int> q(n_terms);
    for (uint64_t t = 0; t < n_terms; ++t) pauli_masks(n, paulis[t], flip[t], sign[t], q[t]);
    if (precision == KETGPU_C64)
      run_adjoint<float>(n, ops, n_ops, param_index, params, n_params, batch, flip, sign, q, coeffs,
                         checkpoint_every, method, values, grads);
    else if (precision == KETGPU_C128)
      run_adjoint<double>(n, ops, n_ops, param_index, params, n_params, batch, flip, sign, q, coeffs,
                          checkpoint_every, method, values, grads);
    else
      fail(KETGPU_ERR_INVALID, "adjoint: bad precision");
    return KETGPU_OK;
  } catch (const Error& e) {
    kb::set_last_error(e.what());
    return e.code;
  } catch (const std::exception& e) {
    kb::set_last_error(e.what());
    return KETGPU_ERR_LOGIC;
  }
}
}  // namespace

KB_API int ketgpu_adjoint(int32_t n, const ketgpu_op* ops, uint64_t n_ops, const int32_t* param_index,
                          const double* params, uint64_t n_params, uint64_t batch, const double* coeffs,
                          const char* const* paulis, uint64_t n_terms, int32_t precision, int32_t checkpoint_every,
                          double* values, double* grads) {
  return adjoint_entry(n, ops, n_ops, param_index, params, n_params, batch, coeffs, paulis, n_terms, precision,
                       checkpoint_every, KETGPU_ADJOINT_AUTO, values, grads);
}

KB_API int ketgpu_adjoint_ex(int32_t n, const ketgpu_op* ops, uint64_t n_ops, const int32_t* param_index,
                             const double* params, uint64_t n_params, uint64_t batch, const double* coeffs,
                             const char* const* paulis, uint64_t n_terms, int32_t precision,
                             int32_t checkpoint_every, int32_t method, double* values, double* grads) {
  return adjoint_entry(n, ops, n_ops, param_index, params, n_params, batch, coeffs, paulis, n_terms, precision,
                       checkpoint_every, method, values, grads);
}

// Plan of the tiled sweeps as flat int32 records, for inspection and for
// checking the plan on the host: [n_blocks] then per block
// [layer, pos[12], n_phases, n_gates, phases (r0 r1 r2 r3 first count) ...,
//  gates (kind s0 s1 tslot tbit cm_r cm_g gen real grad op_index) ...],
// phase.first relative to the block's first gate.  Angles are taken from
// the ops as given (the real flag is per those angles).
KB_API int ketgpu_adjoint_plan_describe(int32_t n, const ketgpu_op* ops, uint64_t n_ops,
                                        const int32_t* param_index, int32_t precision, int32_t checkpoint_every,
                                        int32_t* out, uint64_t capacity, uint64_t* length) {
  try {
    if (!ops || !length) fail(KETGPU_ERR_INVALID, "adjoint_plan_describe: null argument");
    validate_ops(n, ops, n_ops);
    const int TB = precision == KETGPU_C64 ? TileCfg<float>::TB : TileCfg<double>::TB;
    if (n < TB) fail(KETGPU_ERR_INVALID, "adjoint_plan_describe: fewer qubits than a tile");
    std::vector<int> gate_ops, layer_of;
    int layer = 0;
    for (uint64_t i = 0; i < n_ops; ++i) {
      if (ops[i].type == KETGPU_BARRIER) {
        ++layer;
        continue;
      }
      if (!is_unitary(ops[i].type)) continue;
      gate_ops.push_back((int)i);
      layer_of.push_back(layer);
    }
    std::vector<GateGeom> geo(gate_ops.size());
    std::vector<uint8_t> real(gate_ops.size(), 0);
    for (size_t gi = 0; gi < gate_ops.size(); ++gi) {
      const ketgpu_op& o = ops[gate_ops[gi]];
      const int32_t pi = param_index ? param_index[gate_ops[gi]] : -1;
      geo[gi].pslot = pi;
      geo[gi].gen = pi >= 0 ? gen_of(o.type) : 0;
      const Pass p = lower_gate(o);
      bool r = true;
      for (int j = 0; j < 4; ++j) r = r && p.m[j].imag() == 0.0;
      real[gi] = r && p.kind == PassKind::Pair;
    }
    const int m = checkpoint_every > 0 ? checkpoint_every : layer + 1;
    const TilePlan tp = precision == KETGPU_C64 ? plan_tiles_best<float>(n, ops, gate_ops, layer_of, geo, real, m)
                                                : plan_tiles_best<double>(n, ops, gate_ops, layer_of, geo, real, m);
    std::vector<int32_t> v;
    v.push_back((int32_t)tp.blocks.size());
    for (const TBlock& b : tp.blocks) {
      v.push_back(b.layer);
      for (int k = 0; k < 12; ++k) v.push_back(b.geom.pos[k]);
      v.push_back(b.n_phases);
      v.push_back(b.n_gates);
      for (int k = 0; k < b.n_phases; ++k) {
        const TPhase& ph = tp.phases[b.phase_first + k];
        for (int j = 0; j < 4; ++j) v.push_back(ph.r[j]);
        v.push_back(ph.first);
        v.push_back(ph.count);
      }
      for (int k = 0; k < b.n_gates; ++k) {
        const TGate& g = tp.gates[b.gate_first + k];
        v.insert(v.end(), {g.kind, g.s0, g.s1, g.tslot, g.tbit, g.cm_r, g.cm_g, g.gen, g.real, g.grad,
                           gate_ops[g.mat]});
      }
    }
    *length = v.size();
    if (out) {
      if (capacity < v.size()) fail(KETGPU_ERR_INVALID, "adjoint_plan_describe: buffer too small");
      std::memcpy(out, v.data(), v.size() * sizeof(int32_t));
    }
    return KETGPU_OK;
  } catch (const Error& e) {
    kb::set_last_error(e.what());
    return e.code;
  } catch (const std::exception& e) {
    kb::set_last_error(e.what());
    return KETGPU_ERR_LOGIC;
  }
}

// Per-block compiled adjoint kernels: whether NVRTC could be loaded, how
// many distinct kernels are cached and how many launches used one.
KB_API int ketgpu_adjoint_jit_info(int32_t* available, uint64_t* kernels, uint64_t* launches) {
  try {
    if (available) *available = nvrtc().ok ? 1 : 0;
    if (kernels) {
      std::lock_guard<std::mutex> lock(g_jit_mu);
      uint64_t c = 0;
      for (const auto& kv : g_jit) c += kv.second != nullptr;
      *kernels = c;
    }
    if (launches) *launches = g_jit_launches.load();
    return KETGPU_OK;
  } catch (const std::exception& e) {
    kb::set_last_error(e.what());
    return KETGPU_ERR_LOGIC;
  }
}
