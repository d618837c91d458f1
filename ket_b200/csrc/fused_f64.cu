// fused_f64.cu -- dense k-qubit block apply for complex128 states on the
// FP64 tensor instructions.
//
// The complex128 counterpart of fused_tc.cu (ket's apply_matrix,
// src/simulator.cpp:357-393), k = 3..6.  A tile is 2^k target combinations x
// G groups (the lowest non-target qubits); the block matrix's real embedding
// E (2^(k+1) x 2^(k+1)) multiplies the tile's columns, one column per group:
//     out[2r + p][g] = sum_{c, p'} E[2r + p][2c + p'] in[2c + p'][g].
// Products and sums are FP64 (mma.sync m16n8k16 .f64): the same operations as
// the scalar kernel, in another order.
//
// What bounds it: 4 * 2^k FP64 multiply-adds per amplitude against 32 bytes.
// At the measured 36.9 TFLOP/s of this instruction (the FP64 rate of the
// chip; scalar DFMA reaches 35.1) and 6548 GB/s, k = 5 is bound by
// arithmetic (0.93 ms of a 27-qubit pass, memory 0.66 ms) and k <= 4 by
// memory.  The scalar kernel this replaces read both operands of every
// multiply-add from shared memory and reached 6.4 TFLOP/s.
//
// Split.  A warp owns 16 rows of E and keeps them in registers for the whole
// launch (its A fragments, 2^(k+1) / 2 doubles a thread), so shared memory
// holds only the tile and each amplitude is read once per row block as one
// conflict-free 16-byte load.  The K order of the fragments is permuted so
// that a thread's two consecutive K entries are the (re, im) of one
// amplitude, and the row order so that its two accumulator halves are the
// (re, im) of one output: results leave straight from registers in whole
// 32-byte sectors.  One CTA an SM holds five teams of four warps (k <= 5),
// each with its own double-buffered tiles (cp.async), so that one's loads
// overlap another's arithmetic; the teams take tiles from a counter in shared
// memory (five separate CTAs with equal shares: 1.27 ms, since the scheduler
// favours the oldest and the others finish late, alone).
// Measured, 27 qubits, k = 5: 1.10 ms a pass (31.3 TFLOP/s, 0.85 of the
// instruction's rate) against 5.37 ms for the scalar kernel; k = 4: 0.80 ms
// (5.4 TB/s) against 3.61 ms.
// The launch overlaps the previous pass (programmatic dependent launch): the
// matrix fragments are read before the wait on it.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "internal.h"

namespace kb {
namespace {

constexpr int kMaxTileBits = 10;  // 16 KB a stage
constexpr int kStages = 2;
constexpr int kLoadsPerStep = 4;  // copies of the next tile a thread issues per column-block pair

template <int KQ>
struct F64Cfg {
  static constexpr int DIM = 1 << KQ;
  static constexpr int RB = 2 * DIM / 16;         // 16-row blocks of E
  static constexpr int NW = RB < 4 ? 4 : RB;      // warps
  static constexpr int CW = NW / RB;              // warps sharing a row block
  static constexpr int KK = 2 * DIM / 16;         // K = 16 steps
  static constexpr int TEAM = NW * 32;            // threads of a team
  static constexpr int TEAMS = KQ <= 5 ? 5 : 2;
  static constexpr int THREADS = TEAMS * TEAM;
};

struct F64Geom {
  int tb, k;            // tile bits, block qubits
  int q0_group;         // qubit 0 is group bit 0: 32-byte stores
  int gpos[kMaxTileBits];  // qubits of the group bits, ascending
  int tpos[6];          // the block's qubits, ascending
  int is_target[kMaxTileBits];
  int tile_pos[kMaxTileBits];
  // A tile's base is its index spread over the active qubits outside the tile:
  // run by run of adjacent ones, the index shifted and masked ([1]: where
  // nothing is known, over all qubits outside the tile).  One thread of a team
  // forms it while the others wait (inserting a zero bit at a time, positions
  // picked by what is known: 27 qubits, depth 20, 38.1 ms a circuit, now 37.0;
  // 20 qubits 501 us, now 475).  At most 20 runs in 40 qubits.
  int nruns[2];
  unsigned char shift[2][20];
  uint64_t run[2][20];
  Extent tiles;
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mma_f64(double* c, const double* a, double b0, double b1, double b2, double b3) {
  asm("mma.sync.aligned.m16n8k16.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7,%8,%9,%10,%11}, "
      "{%12,%13,%14,%15}, {%0,%1,%2,%3};"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(a[4]), "d"(a[5]), "d"(a[6]), "d"(a[7]), "d"(b0), "d"(b1),
        "d"(b2), "d"(b3));
}

// A group's combinations are stored permuted by XOR with f(group): the 8
// lanes of a 16-byte read phase (4 combinations x 2 groups) and of a write
// phase (8 consecutive groups, or 8 combinations) touch all 8 bank groups.
__device__ __forceinline__ int slot_swizzle(int group) { return ((group & 1) << 2) | ((group >> 1) & 3); }

template <int KQ>
__global__ void __launch_bounds__(F64Cfg<KQ>::THREADS, 1)
    fused_f64_kernel(double2* __restrict__ s, const __grid_constant__ F64Geom g, const double2* __restrict__ mat_t) {
  using Cfg = F64Cfg<KQ>;
  constexpr int DIM = Cfg::DIM, KK = Cfg::KK;
  extern __shared__ __align__(128) double2 f64_tile[];  // kStages stages of 2^tb
  const int team = threadIdx.x / Cfg::TEAM, tid = threadIdx.x % Cfg::TEAM, lane = tid & 31, warp = tid >> 5;
  const int gid = lane >> 2, tig = lane & 3;
  const int rb = warp % Cfg::RB, cw = warp / Cfg::RB;
  const int tile = 1 << g.tb;
  const int nt_total = tile >> (KQ + 3);  // 8-group column blocks

  // A fragments: step kk covers combinations 8 kk + tig and 8 kk + 4 + tig
  double a[KK][8];
  const int r = 8 * rb + gid;
#pragma unroll
  for (int kk = 0; kk < KK; ++kk)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const double2 m = mat_t[(8 * kk + 4 * j + tig) * DIM + r];
      a[kk][4 * j + 0] = m.x;   // (re row, re column)
      a[kk][4 * j + 1] = m.y;   // (im, re)
      a[kk][4 * j + 2] = -m.y;  // (re, im)
      a[kk][4 * j + 3] = m.x;   // (im, im)
    }

  // this thread's part of a tile load: amplitude e = tid + i * THREADS of the
  // tile in address order goes to its (group, combination) slot; offsets and
  // slots are XOR-linear in e
  auto place = [&](int e, uint64_t* off, uint32_t* slot) {
    uint64_t o = 0;
    int grp = 0, comb = 0, gb = 0, cb = 0;
    for (int j = 0; j < g.tb; ++j) {
      const int bit = (e >> j) & 1;
      if (g.is_target[j]) comb |= bit << cb++;
      else grp |= bit << gb++;
      if (bit) o |= uint64_t{1} << g.tile_pos[j];
    }
    *off = o;
    *slot = (uint32_t)(grp * DIM + (comb ^ slot_swizzle(grp)));
  };
  __shared__ uint64_t ld_off[8];  // 2^10 amplitudes / 128 threads
  __shared__ uint32_t ld_slot[8];
  __shared__ uint64_t nt_off[32];  // state offset of column block nt's first group
  const int per = (tile + Cfg::TEAM - 1) / Cfg::TEAM;
  __shared__ unsigned long long team_base[Cfg::TEAMS][2];
  __shared__ unsigned int taken;
  if (threadIdx.x == 0) taken = Cfg::TEAMS * (kStages - 1);
  if (threadIdx.x < 8) {
    uint64_t o;
    uint32_t sl;
    place(tid * Cfg::TEAM & (tile - 1), &o, &sl);
    ld_off[tid] = o;
    ld_slot[tid] = sl;
  }
  if (threadIdx.x >= 32 && threadIdx.x < 64) {
    uint64_t o = 0;
    for (int b = 0; b < 5; ++b)
      if (((tid - 32) >> b) & 1 && 3 + b < g.tb - KQ) o |= uint64_t{1} << g.gpos[3 + b];
    nt_off[tid - 32] = o;
  }
  uint64_t my_off;
  uint32_t my_slot;
  place(tid & (tile - 1), &my_off, &my_slot);
  // this thread's output: row r of groups 8 nt + 2 tig and + 1
  uint64_t out_off = 0;
#pragma unroll
  for (int b = 0; b < KQ; ++b)
    if ((r >> b) & 1) out_off |= uint64_t{1} << g.tpos[b];
  if (tig & 1) out_off |= uint64_t{1} << g.gpos[1];
  if (tig & 2) out_off |= uint64_t{1} << g.gpos[2];
  const uint64_t out_next = uint64_t{1} << g.gpos[0];
  const int o0 = tig ^ slot_swizzle(gid), o1 = (4 + tig) ^ slot_swizzle(gid);

  // Set before the run's first pass, so it can be read ahead of the wait too.
  const int whole = g.tiles.unknown && *g.tiles.unknown;
  const uint64_t n_tiles = whole ? g.tiles.all : g.tiles.known;
  auto tile_base = [&](uint64_t t) -> uint64_t {
    uint64_t b = 0;
    for (int j = 0; j < g.nruns[whole]; ++j) b |= (t << g.shift[whole][j]) & g.run[whole][j];
    return b;
  };
  const int mine = tid < tile ? per : 0;
  auto stage_at = [&](int stage) { return f64_tile + ((size_t)(team * kStages + stage) << g.tb); };
  auto copy = [&](uint64_t at, uint32_t dst, int i) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + ((my_slot ^ ld_slot[i]) << 4)),
                 "l"(s + at + (my_off ^ ld_off[i]))
                 : "memory");
  };

  __syncthreads();
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");

  // Tile i of this CTA is tile i * gridDim.x + blockIdx.x; the teams take
  // them from a shared counter, so no team is left with the last ones.
  constexpr unsigned long long kNone = ~0ull;
  auto base_of = [&](unsigned i) -> unsigned long long {
    const uint64_t t = (uint64_t)i * gridDim.x + blockIdx.x;
    return t < n_tiles ? tile_base(t) : kNone;
  };
  auto team_sync = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "n"(Cfg::TEAM) : "memory"); };
  // kStages - 1 tiles in flight; the barrier that publishes a tile also says
  // that the one before it has been read, so the next load takes its stage
  uint64_t base[kStages];
#pragma unroll
  for (int i = 0; i < kStages - 1; ++i) {
    base[i] = base_of(i * Cfg::TEAMS + team);
    if (base[i] != kNone)
      for (int c = 0; c < mine; ++c) copy(base[i], smem_addr(stage_at(i)), c);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  if (tid == 0) team_base[team][0] = base_of(atomicAdd(&taken, 1u));
  int odd = 0;
  for (int stage = 0;;) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
    team_sync();
    base[kStages - 1] = team_base[team][odd];
    odd ^= 1;
    if (tid == 0) team_base[team][odd] = base_of(atomicAdd(&taken, 1u));
    if (base[0] == kNone) break;
    // the next tile's copies go out between the column blocks: issued all at
    // once they hold the team's warps for as long as the copies queue (1.20
    // against 1.10 ms a pass at 27 qubits, k = 5)
    const uint64_t next = base[kStages - 1];
    const uint32_t next_dst = smem_addr(stage_at(stage == 0 ? kStages - 1 : stage - 1));
    const int copies = next != kNone ? mine : 0;
    int copied = 0;
    const double2* buf = stage_at(stage) + gid * DIM;
    // two column blocks at a time: two independent accumulator chains
    for (int nt = cw; nt < nt_total; nt += 2 * Cfg::CW) {
      const bool two = nt + Cfg::CW < nt_total;
      const double2* in = buf + nt * 8 * DIM;
      const double2* in2 = buf + (two ? nt + Cfg::CW : nt) * 8 * DIM;
      for (int z = 0; z < kLoadsPerStep && copied < copies; ++z, ++copied) copy(next, next_dst, copied);
      double c[2][4] = {};
#pragma unroll
      for (int kk = 0; kk < KK; ++kk) {
        const double2 x = in[8 * kk + o0], y = in[8 * kk + o1];
        mma_f64(c[0], a[kk], x.x, x.y, y.x, y.y);
        const double2 x2 = in2[8 * kk + o0], y2 = in2[8 * kk + o1];
        mma_f64(c[1], a[kk], x2.x, x2.y, y2.x, y2.y);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (h && !two) break;
        double2* out = s + (base[0] | out_off | nt_off[nt + h * Cfg::CW]);
        if (g.q0_group) {
          asm volatile("st.global.v4.f64 [%0], {%1,%2,%3,%4};" ::"l"(out), "d"(c[h][0]), "d"(c[h][2]), "d"(c[h][1]),
                       "d"(c[h][3])
                       : "memory");
        } else {
          out[0] = make_double2(c[h][0], c[h][2]);
          out[out_next] = make_double2(c[h][1], c[h][3]);
        }
      }
    }
    for (; copied < copies; ++copied) copy(next, next_dst, copied);
    asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll
    for (int i = 0; i + 1 < kStages; ++i) base[i] = base[i + 1];
    stage = stage == kStages - 1 ? 0 : stage + 1;
  }
}

template <int KQ>
void launch_k(const State& st, const F64Geom& g, const double2* mat_t, bool overlap) {
  using Cfg = F64Cfg<KQ>;
  const size_t smem = sizeof(double2) * Cfg::TEAMS * kStages * ((size_t)1 << g.tb);
  static OncePerDevice attr;  // one for each KQ
  attr(st.device, [] {
    KB_CUDA(cudaFuncSetAttribute(fused_f64_kernel<KQ>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(sizeof(double2) * Cfg::TEAMS * kStages << kMaxTileBits)));
  });
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)std::min<uint64_t>(g.tiles.most(), 148));
  cfg.blockDim = dim3(Cfg::THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st.stream;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = overlap ? 1 : 0;
  KB_CUDA(cudaLaunchKernelEx(&cfg, fused_f64_kernel<KQ>, static_cast<double2*>(st.amps), g, mat_t));
  count_launch();
}

}  // namespace

// A k-qubit complex128 block needs whole 8-group column blocks.
bool f64_supported(int n, int k) { return k >= 3 && k <= 6 && n >= k + 3; }

void launch_fused_f64(const State& st, const Pass& p, const void* mat_t, const Reach& reach, bool overlap) {
  F64Geom g{};
  g.k = p.k;
  // 1024-amplitude tiles, fewer amplitudes where that leaves teams without a
  // tile: 2^11 tiles or more, down to one column block
  uint64_t span = reach.active;  // index bits of the amplitudes the launch covers
  for (int b = 0; b < p.k; ++b) span |= uint64_t{1} << p.qubits[b];
  g.tb = std::clamp(__builtin_popcountll(span) - 11, p.k + 3, kMaxTileBits);
  uint64_t tmask = 0;
  for (int b = 0; b < p.k; ++b) {
    tmask |= uint64_t{1} << p.qubits[b];
    g.tpos[b] = p.qubits[b];
  }
  uint64_t tile_mask = tmask;
  int extra = g.tb - p.k, j = 0, gb = 0;
  for (int q = 0; q < st.n && extra > 0; ++q)
    if (!((tmask >> q) & 1)) {
      tile_mask |= uint64_t{1} << q;
      --extra;
    }
  span |= tile_mask;
  for (int q = 0; q < st.n; ++q) {
    if ((tile_mask >> q) & 1) {
      g.tile_pos[j] = q;
      g.is_target[j] = (int)((tmask >> q) & 1);
      if (!g.is_target[j]) g.gpos[gb++] = q;
      ++j;
    }
    for (int w = 0; w < 2; ++w) {
      const uint64_t zero = w ? tile_mask : tile_mask | ~span;
      if ((zero >> q) & 1) continue;
      const int below = q - __builtin_popcountll(~zero & ((uint64_t{1} << q) - 1));
      int& r = g.nruns[w];
      if (!r || g.shift[w][r - 1] != below) g.shift[w][r++] = (unsigned char)below;
      g.run[w][r - 1] |= uint64_t{1} << q;
    }
  }
  g.q0_group = g.gpos[0] == 0;
  g.tiles = {uint64_t{1} << (__builtin_popcountll(span) - g.tb), st.dim() >> g.tb, reach.unknown};
  const double2* m = static_cast<const double2*>(mat_t);
  switch (p.k) {
    case 3: launch_k<3>(st, g, m, overlap); break;
    case 4: launch_k<4>(st, g, m, overlap); break;
    case 5: launch_k<5>(st, g, m, overlap); break;
    case 6: launch_k<6>(st, g, m, overlap); break;
    default: fail(KETGPU_ERR_LOGIC, "launch_fused_f64: unsupported block size");
  }
}

}  // namespace kb
