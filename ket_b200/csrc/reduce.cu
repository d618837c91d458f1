// reduce.cu -- FP64 reductions over the state: norm, inner product and the
// fixed-tree Born-rule sampler (Pauli expectations are in expval.cu).
//
// Replaces
//   ket::measure(State, rng)         src/measurement.cpp:12-21
// The reference runs one O(2^n) scan per shot.  Sampling here builds one FP64
// CDF tree per state and answers all shots with a short descent each.
// All sums are deterministic: fixed per-thread order, fixed warp/block trees,
// block partials reduced in index order by a second kernel.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <mutex>
#include <random>
#include <type_traits>
#include <cstring>
#include <vector>

#include "internal.h"

namespace kb {
namespace {

constexpr int kRThreads = 256;

template <typename T>
struct AmpT;
template <>
struct AmpT<float2> {
  static __device__ __forceinline__ double re(float2 v) { return (double)v.x; }
  static __device__ __forceinline__ double im(float2 v) { return (double)v.y; }
};
template <>
struct AmpT<double2> {
  static __device__ __forceinline__ double re(double2 v) { return v.x; }
  static __device__ __forceinline__ double im(double2 v) { return v.y; }
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// Block sum in a fixed tree; result valid in thread 0.
__device__ __forceinline__ double block_sum(double v, double* sh) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  v = warp_sum(v);
  if (lane == 0) sh[warp] = v;
  __syncthreads();
  double r = 0;
  if (warp == 0) {
    r = lane < (int)(blockDim.x >> 5) ? sh[lane] : 0.0;
    r = warp_sum(r);
  }
  __syncthreads();
  return r;
}

template <typename T>
__global__ void norm_partial(const T* __restrict__ s, Extent extent, double* __restrict__ part) {
  __shared__ double sh[32];
  const uint64_t dim = extent.count();
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  // 16-byte loads, eight in flight, a sum each (one 8-byte load at a time:
  // 77 us for 24 qubits, complex64)
  constexpr int PER = 16 / (int)sizeof(T);
  struct alignas(16) Vec {
    T v[PER];
  };
  const Vec* p = reinterpret_cast<const Vec*>(s);
  const uint64_t nv = dim / PER;
  double a[8] = {};
  auto square = [](const Vec& v) {
    double r = 0;
#pragma unroll
    for (int q = 0; q < PER; ++q) {
      const double x = AmpT<T>::re(v.v[q]), y = AmpT<T>::im(v.v[q]);
      r += x * x + y * y;
    }
    return r;
  };
  for (; i + 7 * stride < nv; i += 8 * stride) {
    Vec v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = p[i + u * stride];
#pragma unroll
    for (int u = 0; u < 8; ++u) a[u] += square(v[u]);
  }
  for (; i < nv; i += stride) a[0] += square(p[i]);
  if (PER > 1 && (dim & 1) && blockIdx.x == 0 && threadIdx.x == 0) {  // a 1-amplitude state
    const double x = AmpT<T>::re(s[dim - 1]), y = AmpT<T>::im(s[dim - 1]);
    a[1] += x * x + y * y;
  }
  const double acc = ((a[0] + a[1]) + (a[2] + a[3])) + ((a[4] + a[5]) + (a[6] + a[7]));
  const double r = block_sum(acc, sh);
  if (threadIdx.x == 0) part[blockIdx.x] = r;
}

template <typename T>
__global__ void inner_partial(const T* __restrict__ a, const T* __restrict__ b, uint64_t dim,
                              double* __restrict__ part) {
  __shared__ double sh[32];
  double re = 0, im = 0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < dim;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const T u = a[i], v = b[i];
    const double ur = AmpT<T>::re(u), ui = AmpT<T>::im(u);
    const double vr = AmpT<T>::re(v), vi = AmpT<T>::im(v);
    re += ur * vr + ui * vi;  // conj(u) * v
    im += ur * vi - ui * vr;
  }
  const double r0 = block_sum(re, sh);
  const double r1 = block_sum(im, sh);
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = r0;
    part[2 * blockIdx.x + 1] = r1;
  }
}

// Mixed-precision comparison: max |a-b| and the sums <a|b>, <a|a>, <b|b>.
template <typename TA, typename TB>
__global__ void compare_partial(const TA* __restrict__ a, const TB* __restrict__ b, uint64_t dim,
                                double* __restrict__ part /* 5 per block */) {
  __shared__ double sh[32];
  double re = 0, im = 0, na = 0, nb = 0, mx = 0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < dim;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const TA u = a[i];
    const TB v = b[i];
    const double ur = AmpT<TA>::re(u), ui = AmpT<TA>::im(u);
    const double vr = AmpT<TB>::re(v), vi = AmpT<TB>::im(v);
    re += ur * vr + ui * vi;
    im += ur * vi - ui * vr;
    na += ur * ur + ui * ui;
    nb += vr * vr + vi * vi;
    mx = fmax(mx, fmax(fabs(ur - vr), fabs(ui - vi)));
  }
  const double r0 = block_sum(re, sh), r1 = block_sum(im, sh), r2 = block_sum(na, sh), r3 = block_sum(nb, sh);
  // block max
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_down_sync(0xffffffffu, mx, o));
  if (lane == 0) sh[warp] = mx;
  __syncthreads();
  if (threadIdx.x == 0) {
    double m = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) m = fmax(m, sh[w]);
    part[5 * blockIdx.x + 0] = m;
    part[5 * blockIdx.x + 1] = r0;
    part[5 * blockIdx.x + 2] = r1;
    part[5 * blockIdx.x + 3] = r2;
    part[5 * blockIdx.x + 4] = r3;
  }
}

// Sum `count` partials of `width` interleaved values each, in index order.
__global__ void finish_partials(const double* __restrict__ part, int count, int width,
                                double* __restrict__ out) {
  __shared__ double sh[32];
  for (int w = 0; w < width; ++w) {
    double acc = 0;
    for (int i = threadIdx.x; i < count; i += blockDim.x) acc += part[(size_t)i * width + w];
    const double r = block_sum(acc, sh);
    if (threadIdx.x == 0) out[w] = r;
  }
}

// ---------------------------------------------------------------------------
// Fixed-tree sampler.  p_i = re*re + im*im in FP64 (round-to-nearest on each
// product and the sum, no fused multiply-add).  Level 1 holds sequential sums
// of 32 consecutive p_i; level l+1 holds sequential sums of 32 consecutive
// level-l values; the top level has at most 32 entries.  Carries are then
// folded top-down in place: F_l[j] = F_{l+1}[parent-1] (or 0) + V_l[first
// child] + ... + V_l[j], each addition rounded in order.  A draw descends:
// at each level the first child with u < F, else the last child.
constexpr int kSeg = 32;
constexpr int kSegThreads = 128;  // 4 warps: 4 x 32 x 33 doubles of staging

__device__ __forceinline__ double prob(float2 v) {
  const double x = (double)v.x, y = (double)v.y;
  return __dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y));
}
__device__ __forceinline__ double prob(double2 v) {
  return __dadd_rn(__dmul_rn(v.x, v.x), __dmul_rn(v.y, v.y));
}

// One warp produces 32 segment sums; each lane folds one segment from shared
// memory after a coalesced, transposing load.
template <typename T, bool LEAF>
__global__ void __launch_bounds__(kSegThreads)
    seg_sums(const T* __restrict__ src, uint64_t n_src, double* __restrict__ dst, uint64_t n_dst) {
  __shared__ double sh[kSegThreads / 32][32][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint64_t warps_total = (uint64_t)gridDim.x * (kSegThreads / 32);
  for (uint64_t wseg = (uint64_t)blockIdx.x * (kSegThreads / 32) + warp; wseg * 32 < n_dst;
       wseg += warps_total) {
    const uint64_t base = wseg * 32 * kSeg;
    if (base + 32 * kSeg <= n_src) {
      // 16-byte loads, eight in flight a lane (one 8-byte load at a time, four
      // in flight: 463 us for 28 qubits, complex64; now 396)
      constexpr int PER = 16 / (int)sizeof(T);  // values a load
      struct alignas(16) Vec {
        T v[PER];
      };
      const Vec* p = reinterpret_cast<const Vec*>(src + base) + lane;
#pragma unroll
      for (int h = 0; h < 32 / PER; h += 8) {
        Vec x[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) x[r] = p[(h + r) * 32];
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const int e = ((h + r) * 32 + lane) * PER;
#pragma unroll
          for (int q = 0; q < PER; ++q) {
            if constexpr (LEAF) sh[warp][e >> 5][(e & 31) + q] = prob(x[r].v[q]);
            else sh[warp][e >> 5][(e & 31) + q] = x[r].v[q];
          }
        }
      }
    } else {
      for (int r = 0; r < 32; ++r) {
        const uint64_t i = base + (uint64_t)r * 32 + lane;
        double v = 0;
        if (i < n_src) {
          if constexpr (LEAF) v = prob(src[i]);
          else v = src[i];
        }
        sh[warp][r][lane] = v;
      }
    }
    __syncwarp();
    const uint64_t j = wseg * 32 + lane;
    if (j < n_dst) {
      double acc = 0;
      const uint64_t lo = j * kSeg;
      for (int c = 0; c < kSeg; ++c)
        if (lo + c < n_src) acc = __dadd_rn(acc, sh[warp][lane][c]);
      dst[j] = acc;
    }
    __syncwarp();
  }
}

__global__ void top_fold(double* v, uint64_t n) {
  double c = 0;
  for (uint64_t j = 0; j < n; ++j) {
    c = __dadd_rn(c, v[j]);
    v[j] = c;
  }
}

// Fold carries into level l (in place) from the inclusive carries of level l+1.
__global__ void __launch_bounds__(kSegThreads)
    down_fold(double* __restrict__ v, uint64_t n, const double* __restrict__ parent, uint64_t n_parent) {
  __shared__ double sh[kSegThreads / 32][32][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint64_t warps_total = (uint64_t)gridDim.x * (kSegThreads / 32);
  for (uint64_t wp = (uint64_t)blockIdx.x * (kSegThreads / 32) + warp; wp * 32 < n_parent;
       wp += warps_total) {
    const uint64_t base = wp * 32 * kSeg;
    for (int r = 0; r < 32; ++r) {
      const uint64_t i = base + (uint64_t)r * 32 + lane;
      sh[warp][r][lane] = i < n ? v[i] : 0.0;
    }
    __syncwarp();
    const uint64_t jp = wp * 32 + lane;
    if (jp < n_parent) {
      double c = jp == 0 ? 0.0 : parent[jp - 1];
      const uint64_t lo = jp * kSeg;
      for (int k = 0; k < kSeg; ++k)
        if (lo + k < n) {
          c = __dadd_rn(c, sh[warp][lane][k]);
          sh[warp][lane][k] = c;
        }
    }
    __syncwarp();
    for (int r = 0; r < 32; ++r) {
      const uint64_t i = base + (uint64_t)r * 32 + lane;
      if (i < n) v[i] = sh[warp][r][lane];
    }
    __syncwarp();
  }
}

struct Levels {
  int L;
  uint64_t size[24];
  uint64_t off[24];  // offset (in doubles) of level l >= 1 in the buffer
};

// The uniform of two successive words of std::mt19937, as libstdc++'s
// uniform_real_distribution<double>(0, 1) forms it (its generate_canonical:
// lo + hi * 2^32 in double, over 2^64, below 1).
__device__ __forceinline__ double canonical(uint2 w) {
  const double r = __dadd_rn((double)w.x, (double)w.y * 4294967296.0) * 5.42101086242752217e-20;
  return r < 1.0 ? r : __longlong_as_double(0x3fefffffffffffffll);
}
__device__ __forceinline__ double canonical(double u) { return u; }

// std::mt19937's output words, by one CTA.  With f the twist of two words,
//     x[k] = x[k - 227] ^ f(x[k - 624], x[k - 623])
// gives 227 words at a time; put into itself once,
//     x[k] = x[k - 454] ^ f(x[k - 851], x[k - 850]) ^ f(x[k - 624], x[k - 623])
// gives 454, from a ring of 2048 words in shared memory.  A step's output is
// tempered and stored during the next step's loads.
// Bound: a barrier and a shared-memory round trip a step, 4405 steps for 10^6
// draws (0.78 ms; 1.03 with 227-word steps and the tempering in line, 5.2 on the
// host); it runs beside the passes that read the state.
struct MtState {
  uint32_t x[624];
};
constexpr int kMtThreads = 480, kMtStep = 454;

__device__ __forceinline__ uint32_t mt_twist(uint32_t a, uint32_t b) {
  const uint32_t y = (a & 0x80000000u) | (b & 0x7fffffffu);
  return (y >> 1) ^ (b & 1 ? 0x9908b0dfu : 0u);
}
__device__ __forceinline__ uint32_t mt_temper(uint32_t v) {
  v ^= v >> 11;
  v ^= (v << 7) & 0x9d2c5680u;
  v ^= (v << 15) & 0xefc60000u;
  return v ^ (v >> 18);
}

__global__ void __launch_bounds__(kMtThreads)
    mt19937_words(const __grid_constant__ MtState init, uint32_t words, uint32_t* __restrict__ out) {
  __shared__ uint32_t ring[2048];
  const uint32_t tid = threadIdx.x;
  for (uint32_t i = tid; i < 624; i += kMtThreads) ring[i] = init.x[i];
  __syncthreads();
  if (tid < 227) {  // words 0..226, x[624 .. 850]
    const uint32_t v = ring[tid + 397] ^ mt_twist(ring[tid], ring[tid + 1]);
    ring[tid + 624] = v;
    if (tid < words) out[tid] = mt_temper(v);
  }
  __syncthreads();
  uint32_t last = 0, at = 0xffffffffu;  // the previous step's word and its place
  for (uint32_t w0 = 227; w0 < words; w0 += kMtStep) {
    const uint32_t k = w0 + 624 + tid;
    uint32_t v = 0;
    if (tid < kMtStep) {
      const uint32_t a = ring[(k - 851) & 2047], b = ring[(k - 850) & 2047], c = ring[(k - 624) & 2047],
                     d = ring[(k - 623) & 2047];
      v = ring[(k - 454) & 2047];
      if (at < words) out[at] = mt_temper(last);
      v ^= mt_twist(a, b) ^ mt_twist(c, d);
      ring[k & 2047] = v;
      last = v;
      at = w0 + tid;
    }
    __syncthreads();
  }
  if (at < words) out[at] = mt_temper(last);
}

template <typename T, typename U>
__global__ void sample_kernel(const T* __restrict__ s, const double* __restrict__ buf, Levels lv,
                              const U* __restrict__ u, uint64_t count, uint64_t* __restrict__ out) {
  const uint64_t d = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (d >= count) return;
  const double x = canonical(u[d]);
  double carry = 0;
  uint64_t lo = 0, hi = lv.size[lv.L];
  for (int l = lv.L; l >= 1; --l) {
    const double* F = buf + lv.off[l];
    // first j in [lo, hi) with x < F[j] (F non-decreasing within the range)
    uint64_t a = lo, b = hi;
    while (a < b) {
      const uint64_t m = (a + b) >> 1;
      if (x < F[m]) b = m;
      else a = m + 1;
    }
    const uint64_t pick = a < hi ? a : hi - 1;
    if (pick != lo) carry = F[pick - 1];
    lo = pick * kSeg;
    hi = lo + kSeg < lv.size[l - 1] ? lo + kSeg : lv.size[l - 1];
  }
  uint64_t pick = hi - 1;
  double c = carry;
  if (hi - lo == (uint64_t)kSeg) {
    // eight amplitudes' loads in flight, then their sums in order (one
    // dependent load at a time: 296 us for 10^6 draws at 28 qubits, now about 200)
    bool found = false;
    for (uint64_t i = lo; i < hi && !found; i += 8) {
      T a[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) a[j] = s[i + j];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        c = __dadd_rn(c, prob(a[j]));
        if (!found && x < c) {
          pick = i + j;
          found = true;
        }
      }
    }
  } else {
    for (uint64_t i = lo; i < hi; ++i) {
      c = __dadd_rn(c, prob(s[i]));
      if (x < c) {
        pick = i;
        break;
      }
    }
  }
  out[d] = pick;
}

int grid_for(uint64_t work, int per_block) {
  uint64_t g = (work + per_block - 1) / per_block;
  if (g > 148ull * 16) g = 148ull * 16;
  if (g < 1) g = 1;
  return (int)g;
}

template <typename T>
__global__ void rescale_kernel(T* __restrict__ s, Extent extent, const double* __restrict__ target,
                               const double* __restrict__ current) {
  const uint64_t dim = extent.count();
  const double c = current[0];
  const double f = c > 0.0 ? sqrt(target[0] / c) : 1.0;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if constexpr (std::is_same_v<T, float2>) {
    // complex64: two amplitudes per 16-byte access, four accesses in flight;
    // x * f = fma(x, f - 1, x) in FP32 rounds once, like the FP64 product
    // rounded to FP32 (f - 1 is small, so its own FP32 rounding is far below
    // an ulp of x)
    const float d = (float)(f - 1.0);
    float4* s4 = reinterpret_cast<float4*>(s);
    const uint64_t n4 = dim / 2;
    auto scale = [d](float4 v) {
      return make_float4(fmaf(v.x, d, v.x), fmaf(v.y, d, v.y), fmaf(v.z, d, v.z), fmaf(v.w, d, v.w));
    };
    for (; i + 3 * stride < n4; i += 4 * stride) {
      float4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = s4[i + u * stride];
#pragma unroll
      for (int u = 0; u < 4; ++u) s4[i + u * stride] = scale(v[u]);
    }
    for (; i < n4; i += stride) s4[i] = scale(s4[i]);
    if ((dim & 1) && blockIdx.x == 0 && threadIdx.x == 0) {  // a 1-amplitude state
      s[dim - 1].x = fmaf(s[dim - 1].x, d, s[dim - 1].x);
      s[dim - 1].y = fmaf(s[dim - 1].y, d, s[dim - 1].y);
    }
  } else {
    for (; i < dim; i += stride) {
      T v = s[i];
      v.x = v.x * f;
      v.y = v.y * f;
      s[i] = v;
    }
  }
}

}  // namespace

void norm_to_device(const State& st, const Extent& dim, double* partials, double* out, int blocks) {
  double* part = blocks == 1 ? out : partials;
  if (st.precision == KETGPU_C64)
    norm_partial<float2><<<blocks, kRThreads, 0, st.stream>>>(static_cast<const float2*>(st.amps), dim, part);
  else
    norm_partial<double2><<<blocks, kRThreads, 0, st.stream>>>(static_cast<const double2*>(st.amps), dim, part);
  count_launch();
  if (blocks > 1) {
    finish_partials<<<1, kRThreads, 0, st.stream>>>(partials, blocks, 1, out);
    count_launch();
  }
  KB_CUDA(cudaGetLastError());
}

void norm_from_partials(const State& st, const double* partials, double* out) {
  finish_partials<<<1, kRThreads, 0, st.stream>>>(partials, kNormBlocks, 1, out);
  count_launch();
  KB_CUDA(cudaGetLastError());
}

void rescale_state(const State& st, const Extent& dim, const double* target, const double* current) {
  if (st.precision == KETGPU_C64)
    rescale_kernel<float2><<<kNormBlocks, kRThreads, 0, st.stream>>>(static_cast<float2*>(st.amps), dim,
                                                                     target, current);
  else
    rescale_kernel<double2><<<kNormBlocks, kRThreads, 0, st.stream>>>(static_cast<double2*>(st.amps), dim,
                                                                      target, current);
  count_launch();
  KB_CUDA(cudaGetLastError());
}

namespace {
// Bit patterns other than those of |0...0> (a negative zero counts).
__global__ void not_ground(const uint64_t* __restrict__ w, uint64_t words, uint64_t first, unsigned* flag) {
  bool bad = false;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  const ulonglong2* w2 = reinterpret_cast<const ulonglong2*>(w);
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < words / 2; i += stride) {
    const ulonglong2 v = w2[i];
    bad |= (i == 0 ? v.x != first : v.x != 0) || v.y != 0;
  }
  if ((words & 1) && blockIdx.x == 0 && threadIdx.x == 0) bad |= words == 1 ? w[0] != first : w[words - 1] != 0;
  if (bad) *flag = 1u;
}
}  // namespace

const unsigned* find_not_ground(const State& st) {
  if (!st.word.p) st.word = DeviceBlock(sizeof(unsigned), st.device, st.stream);
  unsigned* d = static_cast<unsigned*>(st.word.p);
  KB_CUDA(cudaMemsetAsync(d, 0, sizeof(unsigned), st.stream));
  const bool c64 = st.precision == KETGPU_C64;
  const uint64_t words = st.dim() * (c64 ? 1 : 2);
  not_ground<<<grid_for(words, kRThreads * 16), kRThreads, 0, st.stream>>>(
      static_cast<const uint64_t*>(st.amps), words, c64 ? 0x3f800000ull : 0x3ff0000000000000ull, d);
  count_launch();
  KB_CUDA(cudaGetLastError());
  return d;
}

double reduce_norm(const State& st) {
  const int blocks = grid_for(st.dim(), kRThreads * 8);
  StreamScratch part(sizeof(double) * (blocks + 1), st.device, st.stream);
  double* d = static_cast<double*>(part.p);
  const Extent all{st.dim(), st.dim(), nullptr};
  if (st.precision == KETGPU_C64)
    norm_partial<float2><<<blocks, kRThreads, 0, st.stream>>>(static_cast<const float2*>(st.amps), all, d);
  else
    norm_partial<double2><<<blocks, kRThreads, 0, st.stream>>>(static_cast<const double2*>(st.amps), all, d);
  finish_partials<<<1, kRThreads, 0, st.stream>>>(d, blocks, 1, d + blocks);
  count_launch(2);
  KB_CUDA(cudaGetLastError());
  double h = 0;
  KB_CUDA(cudaMemcpyAsync(&h, d + blocks, sizeof(double), cudaMemcpyDeviceToHost, st.stream));
  KB_CUDA(cudaStreamSynchronize(st.stream));
  return h;
}

cplx reduce_inner(const State& a, const State& b) {
  const int blocks = grid_for(a.dim(), kRThreads * 8);
  StreamScratch part(sizeof(double) * 2 * (blocks + 1), a.device, a.stream);
  double* d = static_cast<double*>(part.p);
  if (b.stream != a.stream) KB_CUDA(cudaStreamSynchronize(b.stream));
  if (a.precision == KETGPU_C64)
    inner_partial<float2><<<blocks, kRThreads, 0, a.stream>>>(static_cast<const float2*>(a.amps),
                                                              static_cast<const float2*>(b.amps), a.dim(), d);
  else
    inner_partial<double2><<<blocks, kRThreads, 0, a.stream>>>(static_cast<const double2*>(a.amps),
                                                               static_cast<const double2*>(b.amps), a.dim(), d);
  finish_partials<<<1, kRThreads, 0, a.stream>>>(d, blocks, 2, d + 2 * blocks);
  count_launch(2);
  KB_CUDA(cudaGetLastError());
  double h[2];
  KB_CUDA(cudaMemcpyAsync(h, d + 2 * blocks, sizeof h, cudaMemcpyDeviceToHost, a.stream));
  KB_CUDA(cudaStreamSynchronize(a.stream));
  return {h[0], h[1]};
}

void compare_states(const State& a, const State& b, double out[5]) {
  const int blocks = grid_for(a.dim(), kRThreads * 8);
  StreamScratch part(sizeof(double) * 5 * blocks, a.device, a.stream);
  double* d = static_cast<double*>(part.p);
  KB_CUDA(cudaStreamSynchronize(b.stream));
  const bool a64 = a.precision == KETGPU_C64, b64 = b.precision == KETGPU_C64;
  if (a64 && b64)
    compare_partial<float2, float2><<<blocks, kRThreads, 0, a.stream>>>(
        static_cast<const float2*>(a.amps), static_cast<const float2*>(b.amps), a.dim(), d);
  else if (a64)
    compare_partial<float2, double2><<<blocks, kRThreads, 0, a.stream>>>(
        static_cast<const float2*>(a.amps), static_cast<const double2*>(b.amps), a.dim(), d);
  else if (b64)
    compare_partial<double2, float2><<<blocks, kRThreads, 0, a.stream>>>(
        static_cast<const double2*>(a.amps), static_cast<const float2*>(b.amps), a.dim(), d);
  else
    compare_partial<double2, double2><<<blocks, kRThreads, 0, a.stream>>>(
        static_cast<const double2*>(a.amps), static_cast<const double2*>(b.amps), a.dim(), d);
  count_launch();
  KB_CUDA(cudaGetLastError());
  std::vector<double> h((size_t)5 * blocks);
  KB_CUDA(cudaMemcpyAsync(h.data(), d, h.size() * sizeof(double), cudaMemcpyDeviceToHost, a.stream));
  KB_CUDA(cudaStreamSynchronize(a.stream));
  for (int w = 0; w < 5; ++w) out[w] = 0;
  for (int bl = 0; bl < blocks; ++bl) {
    out[0] = std::max(out[0], h[5 * bl]);
    for (int w = 1; w < 5; ++w) out[w] += h[5 * bl + w];
  }
}

std::atomic<uint64_t> g_tree_builds{0};

uint64_t sample_tree_builds() { return g_tree_builds.load(); }

namespace {

Levels tree_levels(const State& st, uint64_t* total) {
  Levels lv{};
  lv.size[0] = st.dim();
  *total = 0;
  while (lv.size[lv.L] > (uint64_t)kSeg) {
    lv.size[lv.L + 1] = (lv.size[lv.L] + kSeg - 1) / kSeg;
    ++lv.L;
    lv.off[lv.L] = *total;
    *total += lv.size[lv.L];
  }
  return lv;
}

// What draws make on demand in a state, its tree and its second stream, is made
// by one thread: several may draw from a state at once.
std::mutex g_draw_mu;

// The state's tree, built on its stream if the amplitudes changed, or may have:
// a graph's replays are not seen.
Levels build_tree(const State& st) {
  uint64_t total = 0;
  const Levels lv = tree_levels(st, &total);
  std::lock_guard<std::mutex> lk(g_draw_mu);
  // The tree lives with the state (1/31 of a complex128 state's size, 1/15
  // of a complex64 one) and is rebuilt only after the amplitudes changed.
  if (total && !st.tree) {
    allocate("cudaMalloc(sampling tree)", [&] { return cudaMalloc(&st.tree, sizeof(double) * total); });
    st.tree_doubles = total;
  }
  if (!total || (st.tree_version == st.version && !st.captured)) return lv;
  double* buf = st.tree;
  g_tree_builds.fetch_add(1);
  for (int l = 1; l <= lv.L; ++l) {
    const uint64_t nd = lv.size[l];
    const int blocks = grid_for(nd, kSegThreads);  // one warp -> 32 outputs
    if (l == 1) {
      if (st.precision == KETGPU_C64)
        seg_sums<float2, true><<<blocks, kSegThreads, 0, st.stream>>>(static_cast<const float2*>(st.amps),
                                                                      lv.size[0], buf + lv.off[1], nd);
      else
        seg_sums<double2, true><<<blocks, kSegThreads, 0, st.stream>>>(static_cast<const double2*>(st.amps),
                                                                       lv.size[0], buf + lv.off[1], nd);
    } else {
      seg_sums<double, false><<<blocks, kSegThreads, 0, st.stream>>>(buf + lv.off[l - 1], lv.size[l - 1],
                                                                     buf + lv.off[l], nd);
    }
    count_launch();
  }
  top_fold<<<1, 1, 0, st.stream>>>(buf + lv.off[lv.L], lv.size[lv.L]);
  count_launch();
  for (int l = lv.L - 1; l >= 1; --l) {
    const int blocks = grid_for(lv.size[l + 1], kSegThreads);
    down_fold<<<blocks, kSegThreads, 0, st.stream>>>(buf + lv.off[l], lv.size[l], buf + lv.off[l + 1],
                                                   lv.size[l + 1]);
    count_launch();
  }
  KB_CUDA(cudaGetLastError());
  st.tree_version = st.version;
  return lv;
}

template <typename U>
void draw(const State& st, const Levels& lv, const U* d_u, uint64_t count, uint64_t* d_out, uint64_t* out) {
  const unsigned blocks = (unsigned)((count + kRThreads - 1) / kRThreads);
  if (st.precision == KETGPU_C64)
    sample_kernel<<<blocks, kRThreads, 0, st.stream>>>(static_cast<const float2*>(st.amps), st.tree, lv, d_u, count,
                                                       d_out);
  else
    sample_kernel<<<blocks, kRThreads, 0, st.stream>>>(static_cast<const double2*>(st.amps), st.tree, lv, d_u, count,
                                                       d_out);
  count_launch();
  KB_CUDA(cudaGetLastError());
  fetch_bytes(d_out, sizeof(uint64_t) * count, out, st.stream);
}

cudaStream_t side_stream(const State& st) {
  std::lock_guard<std::mutex> lk(g_draw_mu);
  if (!st.side) {
    int least = 0, greatest = 0;
    KB_CUDA(cudaDeviceGetStreamPriorityRange(&least, &greatest));
    KB_CUDA(cudaStreamCreateWithPriority(&st.side, cudaStreamNonBlocking, greatest));
  }
  return st.side;
}

// Draws from which the uniforms are made on the device.  A call of 8192 draws
// at 12 qubits takes 79 us with them made on the device and 120 on the host;
// one of 1000 takes 61 us on the host.
constexpr uint64_t kDeviceDraws = 2048;
constexpr uint64_t kMostDeviceDraws = uint64_t{1} << 30;  // 32-bit word indices

}  // namespace

void sample_tree(const State& st, const double* u, uint64_t count, uint64_t* out) {
  const Levels lv = build_tree(st);
  if (!count) {
    KB_CUDA(cudaStreamSynchronize(st.stream));
    return;
  }
  StreamScratch sc((sizeof(double) + sizeof(uint64_t)) * count, st.device, st.stream);
  double* d_u = static_cast<double*>(sc.p);
  KB_CUDA(cudaMemcpyAsync(d_u, u, sizeof(double) * count, cudaMemcpyHostToDevice, st.stream));
  draw(st, lv, d_u, count, reinterpret_cast<uint64_t*>(d_u + count), out);
}

void sample_tree_seeded(const State& st, uint32_t seed, uint64_t count, uint64_t* out) {
  if (count < kDeviceDraws || count > kMostDeviceDraws) {
    std::vector<double> u(count);
    std::mt19937 rng{seed};
    std::uniform_real_distribution<double> dist(0.0, 1.0);
    for (double& v : u) v = dist(rng);
    sample_tree(st, u.data(), count, out);
    return;
  }
  // the words on the second stream, beside whatever the first one still does
  // to the amplitudes and the tree's building
  const cudaStream_t side = side_stream(st);
  StreamScratch words(sizeof(uint2) * count, st.device, side);
  MtState mt;
  mt.x[0] = seed;
  for (uint32_t i = 1; i < 624; ++i) mt.x[i] = 1812433253u * (mt.x[i - 1] ^ (mt.x[i - 1] >> 30)) + i;
  mt19937_words<<<1, kMtThreads, 0, side>>>(mt, (uint32_t)(2 * count), static_cast<uint32_t*>(words.p));
  count_launch();
  KB_CUDA(cudaGetLastError());
  const Levels lv = build_tree(st);
  cudaEvent_t made;
  KB_CUDA(cudaEventCreateWithFlags(&made, cudaEventDisableTiming));
  cudaError_t e = cudaEventRecord(made, side);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(st.stream, made, 0);
  cudaEventDestroy(made);
  check_cuda(e, "sample_tree_seeded");
  StreamScratch sc(sizeof(uint64_t) * count, st.device, st.stream);
  uint64_t* d_out = static_cast<uint64_t*>(sc.p);
  draw(st, lv, static_cast<const uint2*>(words.p), count, d_out, out);
}

}  // namespace kb
