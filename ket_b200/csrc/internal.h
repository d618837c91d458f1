// internal.h -- shared host-side declarations of the B200 state-vector
// backend (not installed; the public surface is include/ket_b200.h).
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <complex>
#include <cstdint>
#include <memory>
#include <mutex>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/ket_b200.h"

namespace kb {

using cplx = std::complex<double>;

// ---- errors ----------------------------------------------------------------
// Thrown inside the library, turned into KETGPU_ERR_* at the ABI boundary.
struct Error : std::runtime_error {
  int code;
  Error(int c, const std::string& m) : std::runtime_error(m), code(c) {}
};
[[noreturn]] void fail(int code, const std::string& msg);
void check_cuda(cudaError_t e, const char* what);
void set_last_error(const char* msg);
#define KB_CUDA(x) ::kb::check_cuda((x), #x)

extern std::atomic<uint64_t> g_launches;
inline void count_launch(uint64_t k = 1) { g_launches.fetch_add(k, std::memory_order_relaxed); }

// Switch to a device for the lifetime of the guard.
struct DeviceGuard {
  int prev = -1;
  explicit DeviceGuard(int dev);
  ~DeviceGuard();
};

// Gives back what the library keeps between calls: idle states, workspaces,
// scratch.
void release_kept();
// Kernel attributes are a device's: `set` on the first call for each device.
// One object for each set of attributes.
class OncePerDevice {
 public:
  template <class F>
  void operator()(int device, F&& set) {
    const bool noted = device >= 0 && device < 64;
    if (noted && done_[device].load(std::memory_order_acquire)) return;
    set();
    if (noted) done_[device].store(true, std::memory_order_release);
  }

 private:
  std::atomic<bool> done_[64] = {};
};

// Device memory: `alloc` (returning a cudaError_t), once more after what is
// kept between calls has been given back if there is no room.
template <class F>
void allocate(const char* what, F&& alloc) {
  cudaError_t e = alloc();
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    release_kept();
    e = alloc();
  }
  check_cuda(e, what);
}

// Device scratch of one call, stream-ordered, from the library's own pool on
// the device.  The pool keeps up to kPoolKeep bytes between calls (taking them
// back from the driver at each synchronisation cost 0.1 ms and more a call);
// release_pools gives them back.
constexpr uint64_t kPoolKeep = uint64_t{64} << 20;
struct StreamScratch {
  void* p = nullptr;
  cudaStream_t st;
  StreamScratch(size_t bytes, int device, cudaStream_t stream);
  ~StreamScratch();
  StreamScratch(const StreamScratch&) = delete;
  StreamScratch& operator=(const StreamScratch&) = delete;
};
void release_pools();
// Device memory from the same pool that outlives the call that made it.  Its
// owner frees it when nothing on the device uses it any more.
struct DeviceBlock {
  void* p = nullptr;
  DeviceBlock() = default;
  DeviceBlock(size_t bytes, int device, cudaStream_t stream);
  DeviceBlock(DeviceBlock&& o) noexcept : p(o.p) { o.p = nullptr; }
  DeviceBlock& operator=(DeviceBlock&& o) noexcept;
  ~DeviceBlock();
};

// ---- state -----------------------------------------------------------------
struct State {
  int n = 0;
  int precision = KETGPU_C64;
  int device = 0;
  void* amps = nullptr;  // float2[2^n] or double2[2^n]
  cudaStream_t stream = nullptr;
  // Bumped by every write the library makes to the amplitudes (touch()).
  mutable uint64_t version = 0;
  // The sampling tree (FP64 level sums with folded carries) of the state at
  // tree_version, kept for the next draws; built by sample_tree on demand.
  mutable double* tree = nullptr;
  mutable uint64_t tree_doubles = 0;
  mutable uint64_t tree_version = ~uint64_t{0};
  // A second stream, above the first in priority, for work that does not need
  // the amplitudes (the draws of sample_tree_seeded); made on demand.
  mutable cudaStream_t side = nullptr;
  // version right after set_ground: while version still equals it, the state
  // is |0...0> and its squared norm is exactly 1
  mutable uint64_t ground_version = ~uint64_t{0};
  // The index bits that can be set in a nonzero amplitude, known while
  // version equals active_version (see Activity): 0 after set_ground.
  mutable uint64_t active = 0;
  mutable uint64_t active_version = ~uint64_t{0};
  // The amplitudes' address has been handed out, or a plan has been captured
  // into a graph: they may change without a touch(), so what is known about
  // them is checked on the device before use.
  mutable bool exposed = false;
  // A plan has been captured into a graph: the tree is built for each call.
  mutable bool captured = false;
  // Device word of the check for |0...0> (find_not_ground), made on demand and
  // kept: memory of the pool that each run gave back behind its own passes made
  // the pool's next users wait for this stream (14 qubits, complex128, adjoint:
  // 870 us a call beside 16 MB states, now 805).
  mutable DeviceBlock word;
  uint64_t dim() const { return uint64_t{1} << n; }
  size_t amp_bytes() const { return precision == KETGPU_C64 ? 8 : 16; }
  void touch() const { ++version; }
};

// ---- passes ----------------------------------------------------------------
// One kernel launch of a plan.
enum class PassKind : int {
  Pair,      // 2x2 on (k0, k1) = (base|P0, base|P1), base ranges over the
             // indices with zeros at the fixed positions
  Phase,     // multiply the amplitudes with all fixed bits set by a phase
  Fused,     // dense 2^k x 2^k complex matrix on k qubits
  NormCapture,  // record the state's squared norm (FP64) on the device
  NormRestore,  // rescale the state to the recorded squared norm
  Diagonal,     // multiply amplitude x by exp(i phi(x)), phi a quadratic
                // polynomial in the index bits (a run of diagonal gates)
  SharedRun,    // consecutive gates on qubits below kRunBits, applied one
                // after another to chunks of 2^kRunBits amplitudes held in
                // shared memory (one HBM pass for the run)
};
// Chunk bits of a shared-memory run: its gates act on qubits 0..kRunBits-1.
constexpr int kRunBits = 11;
constexpr int kRunMaxGates = 128;
enum PairMode : int { kPairGeneral = 0, kPairSwap = 1, kPairDiag = 2 };

// Index bits of the lowest indices that hold every amplitude within `active`.
inline int active_bits(uint64_t active) { return active ? 64 - __builtin_clzll(active) : 0; }

struct Pass {
  PassKind kind = PassKind::Pair;
  int mode = kPairGeneral;
  int nfixed = 0;
  int fixed[3] = {0, 0, 0};  // sorted ascending
  uint64_t p0 = 0, p1 = 0;   // bit patterns of element 0 / element 1
  cplx m[4];                 // 2x2 (Pair) ; m[0] = phase (Phase)
  // Fused
  int k = 0;
  int qubits[6] = {0, 0, 0, 0, 0, 0};  // sorted ascending; matrix bit b <-> qubits[b]
  size_t table = 0;                    // Fused, Diagonal, SharedRun: its table's offset in Plan::block
  bool tensor = false;                 // tcgen05 path
  // tcgen05 block directly before the plan's NormRestore: it also writes
  // per-CTA FP64 sums of |out|^2 into the plan's norm partials, and the
  // restore (norm_out set there too) takes the norm from them
  bool norm_out = false;
  size_t diag_index = 0;               // Diagonal: into Plan::diags
  size_t run_index = 0;                // SharedRun: into Plan::runs
  int first_op = 0, n_gates = 0;       // provenance
  std::vector<int> gates;              // op indices of the gates this pass applies
  double bytes(int n, size_t amp) const;
};

// Phase polynomial of a run of diagonal gates: the amplitude with index bits
// x_0..x_{n-1} is multiplied by exp(i phi(x)),
//   phi(x) = c0 + sum_i a[i] x_i + sum_{i<j} b[i*n + j] x_i x_j.
struct DiagPoly {
  double c0 = 0.0;
  std::vector<double> a;  // n
  std::vector<double> b;  // n x n, upper triangle used
};
// Low index bits whose pair terms are tabulated by the diagonal kernel.
constexpr int kDiagLowBits = 12;

struct Plan {
  int n = 0;
  int precision = KETGPU_C64;
  std::vector<ketgpu_op> ops;  // the circuit the plan was built from
  bool finite = true;          // every gate parameter is a finite number
  std::vector<Pass> passes;
  std::vector<DiagPoly> diags;          // Diagonal passes (host)
  std::vector<std::vector<Pass>> runs;  // SharedRun passes: each gate lowered (host)
  // Device tables (tables.cu), made at the first execution: block matrices
  // (transposed FP64 or FP32) or tensor-core operands, diagonal tables with
  // their coefficients, gate records of shared-memory runs.
  DeviceBlock block;
  double* d_norm = nullptr;  // [captured, current, block partials...]
  int device = -1;
  bool idle = false;  // nothing that reads the tables is in flight
  std::mutex mu;      // guards the tables' making
  ketgpu_plan_stats stats{};
  ~Plan();
};

// ---- gate lowering -----------------------------------------------------------
bool is_unitary(int type);
int gate_arity(int type);
void validate_ops(int n, const ketgpu_op* ops, uint64_t nops);
// The 2x2 matrix of a 1-qubit gate (or the target block of a controlled
// rotation), built with ket's formulas (simulator.cpp:38-97, 166-200).
void single_matrix(int type, const double* p, cplx m[4]);
// Lower one gate to its specialised pass.
Pass lower_gate(const ketgpu_op& op);
// Per-gate cost in state passes (fraction of the state each pass moves).
double gate_traffic_fraction(const ketgpu_op& op);
// The gates ops[gates[i]] lowered onto the bits of a block (bit b <-> qubits[b]).
std::vector<Pass> lower_block(const ketgpu_op* ops, const std::vector<int>& gates, const int* qubits, int k);
// Their dense matrix, on the host.
std::vector<cplx> block_matrix(const ketgpu_op* ops, const std::vector<int>& gates, const int* qubits, int k);

// ---- planner ---------------------------------------------------------------
struct PlanOptions {
  int precision = KETGPU_C64;
  int fusion = KETGPU_FUSE_GREEDY;
  int max_k = 5;
  bool tensor = true;
  int renormalize = 0;
};
constexpr int kNormBlocks = 592;  // 4 x 148 SMs
PlanOptions resolve_options(const ketgpu_options* opt);
void build_plan(Plan& plan, int n, const ketgpu_op* ops, uint64_t nops,
                const PlanOptions& o);
// Cost-model features of one pass: a dense block over `qubits` (fused) or
// one gate through its specialised kernel (gates.size() == 1, !fused).
constexpr int kFeatures = 48;
void pass_features(int n, int precision, const std::vector<const ketgpu_op*>& gates,
                   const std::vector<int>& qubits, bool fused, bool tensor, float* out);
// Learned-planner hooks (mlp.cu): the attached model, and batched
// predictions of pass times (microseconds) for feature rows.
bool learned_model_attached();
void learned_predict(const std::vector<float>& rows, std::vector<float>& us);

// ---- kernel launchers (gates.cu / fused_*.cu / reduce.cu) ------------------
// The part of a state that a pass works on: the amplitudes whose set index
// bits all lie within `active`.  unknown (null: that is certain) points to a
// device word; where it holds nonzero, the pass works on the whole state.
struct Reach {
  uint64_t active;
  const unsigned* unknown = nullptr;
};
// How many of something (tiles, chunks, pairs, amplitudes) a launch works on.
struct Extent {
  uint64_t known, all;
  const unsigned* unknown;
  uint64_t most() const { return unknown ? all : known; }
#ifdef __CUDACC__
  __device__ __forceinline__ uint64_t count() const { return unknown && *unknown ? all : known; }
#endif
};
// Runs a plan's passes in order on the part of the state that can be nonzero.
//
// From |0...0> only amplitudes whose set index bits lie within the qubits
// acted on so far are nonzero, so a pass before all qubits are active runs on
// 2^|active| amplitudes instead of 2^n (dense blocks exactly; the streaming
// kernels on the indices below the highest active qubit).  The other
// amplitudes are zeros and stay so.  Planned in an order that activates
// qubits late (order_passes), the 30-qubit depth-40 brick wall moves 47.1
// states' worth of blocks instead of 63.
// Nothing is assumed of a plan with non-finite parameters (0 * inf) and under
// stream capture (a graph may replay on another state).  A state whose address
// was handed out, or whose stream was captured before (a replay writes it), is
// looked at on the device after a reset: a kernel sets a word if it is not
// |0...0>, and each pass takes the part of the state that it works on by that
// word, so the host waits for nothing.
class PassRunner {
 public:
  PassRunner(const State& s, const Plan& plan);
  ~PassRunner();
  void launch(const Pass& p);

 private:
  Extent amplitudes() const;  // the lowest indices that hold all active ones

  const State& s_;
  const Plan& plan_;
  uint64_t active_;
  bool keep_;  // what is known outlives the run
  const unsigned* word_ = nullptr;  // set by the device: not |0...0> at the start
  bool first_ = true;
};
// Enqueues one read of the state; returns the device word that it sets if that
// differs from |0...0>.
const unsigned* find_not_ground(const State& s);
// one_stream: the plan runs on `stream` only (the tables are not waited for).
void upload_plan_tables(Plan& plan, int device, cudaStream_t stream, bool one_stream);
// norm_partials: null, or kNormBlocks doubles that receive the per-CTA sums
// of |out|^2 (zero beyond the grid).  reach (here and below): the index bits
// that can be set in a nonzero amplitude, the pass's gates' qubits included.
// overlap (and below): the launch may start under the one before it.
void launch_fused_tc(const State& s, const Pass& p, const void* b_image, double* norm_partials, const Reach& reach,
                     bool overlap);
// complex128 dense blocks (fused_f64.cu): mat_t = the FP64 matrix,
// transposed ([c][r], re/im).
bool f64_supported(int n, int k);
void launch_fused_f64(const State& s, const Pass& p, const void* mat_t, const Reach& reach, bool overlap);
// Host only: the producer and epilogue forms a tensor-core launch of pass p
// on an n-qubit state takes (tma_dims = tensor-map dimensions, 0 for the
// cp.async producers; direct = register-to-HBM stores), given the tensor-map
// encoder of the driver.
void tc_form(int n, const Pass& p, int* tma_dims, int* direct);
// Diagonal pass: device data = table (2^L complex, state precision) then FP64
// coefficients.
void launch_diag(const State& s, const Pass& p, const void* data, const Reach& reach);
// SharedRun pass: device gate records laid out by run_device_data (gates.cu).
void launch_run(const State& s, const Pass& p, const void* data, const Reach& reach);
void run_device_data(const std::vector<Pass>& gates, int precision, std::vector<unsigned char>& out);
// The coefficients the diagonal kernel reads after its table (diag.cu).
void diag_coefficients(const DiagPoly& poly, int n, std::vector<double>& out);
bool is_diagonal_gate(int type);
// Add one diagonal gate's phase terms to a polynomial.
void add_diagonal_gate(const ketgpu_op& op, DiagPoly& poly, int n);
// Size in bytes of one tcgen05 B image for a k-qubit block.
size_t tc_image_bytes(int k);
void build_tc_image(const std::vector<cplx>& mat, int k, std::vector<uint32_t>& out);
bool tc_supported(int k);

void set_ground(const State& s);
// Squared norm of the first amplitudes into a device scalar (partials:
// kNormBlocks doubles), by `blocks` CTAs.
void norm_to_device(const State& s, const Extent& dim, double* partials, double* out, int blocks = kNormBlocks);
// The same from partials a tensor-core block already wrote (in index order).
void norm_from_partials(const State& s, const double* partials, double* out);
// Look up (and so load) the no-allocation entry point's scratch array and
// kernels on `device`, which must be current; once per device, at the first
// state created there.
void noalloc_prepare(int device);
// Free the device state that ketgpu_run keeps between calls (if any).
void release_run_state();
// Free the destroyed states kept for reuse.
void release_idle_states();
// Device memory for one call that may be large: the last call's is kept for
// the next when it is at most kWorkspaceKeep (allocating and freeing 400 MB
// took half of a call; the stream-ordered pool maps 50 GB far more slowly
// than cudaMalloc).  The owner's work on it is done when it ends.
constexpr uint64_t kWorkspaceKeep = uint64_t{4} << 30;
struct Workspace {
  void* p = nullptr;
  size_t bytes;
  int device;
  Workspace(size_t bytes, int dev);
  ~Workspace();
  Workspace(const Workspace&) = delete;
  Workspace& operator=(const Workspace&) = delete;
};
void release_workspaces();
// A non-blocking stream for one call, from a few kept per device (making and
// destroying one costs about 50 us).
struct StreamLease {
  cudaStream_t s = nullptr;
  int device;
  explicit StreamLease(int dev);
  ~StreamLease();  // waits for the stream's work
  StreamLease(const StreamLease&) = delete;
  StreamLease& operator=(const StreamLease&) = delete;
};
// The first amplitudes *= sqrt(target[0] / current[0]), factor read on the
// device.
void rescale_state(const State& s, const Extent& dim, const double* target, const double* current);
double reduce_norm(const State& s);
cplx reduce_inner(const State& a, const State& b);
void compare_states(const State& a, const State& b, double out[5]);
// Expectations of Pauli strings (expval.cu); phase[t] = number of Y's mod 4.
void expval_terms(const State& s, const std::vector<uint64_t>& flip,
                  const std::vector<uint64_t>& sign, const std::vector<int>& phase,
                  double* out);
// Born-rule draws for host uniforms; builds the state's sampling tree only
// when the amplitudes changed since the last build (State::version).
void sample_tree(const State& s, const double* u, uint64_t count, uint64_t* out);
// The same for the draws of std::mt19937{seed}.
void sample_tree_seeded(const State& s, uint32_t seed, uint64_t count, uint64_t* out);
// Copy device memory to a host buffer, ordered on and waiting for `stream`
// (abi.cpp; large copies go through pinned staging).
void fetch_bytes(const void* src, uint64_t bytes, void* out, cudaStream_t stream);
// Number of sampling-tree builds since load (all states).
uint64_t sample_tree_builds();

// Pauli-string masks (observable.cpp:68-113); throws Error(INVALID).
void pauli_masks(int n, const char* pauli, uint64_t& flip, uint64_t& sign, int& phase_q);

}  // namespace kb
