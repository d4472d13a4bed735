// Internal declarations shared by the libfmpt translation units.
#pragma once

#include <cuda_runtime.h>
#include <cusolverDn.h>

#include <cstdint>
#include <cstdio>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/fmpt.h"

struct fmpt_handle {
  int device = 0;
  cudaStream_t stream = nullptr;       // stream in use
  cudaStream_t own_stream = nullptr;   // stream created by fmpt_create
  cusolverDnHandle_t solver = nullptr;
  uint64_t launches = 0;
  std::string err;
  // small pinned host staging area for scalars read back by the solvers
  double* pinned = nullptr;
  size_t pinned_len = 0;
  // Lanczos solve: the ends of its two latest steps, and pinned memory their kernels write
  // (alpha, beta) pairs to while the staging area above serves the calls in between (both
  // created on first use)
  cudaEvent_t step_event[2] = {nullptr, nullptr};
  double* step_host = nullptr;
  int sm_count = 0;
  // device timers (fmpt_profile_*)
  bool prof = false;
  std::vector<std::pair<cudaEvent_t, cudaEvent_t>> prof_ev[FMPT_K_COUNT];
  std::vector<cudaEvent_t> ev_pool;
  // status word of the grouped block-sparse launches (1 = a grid barrier timed
  // out); allocated on first use, read and cleared by gp_check_status
  int* gstatus = nullptr;
  // auxiliary streams with their own cuSOLVER handles for independent
  // factorisations (created on first use): fork/join through events on `stream`
  std::vector<cudaStream_t> aux_stream;
  std::vector<cusolverDnHandle_t> aux_solver;
  std::vector<cudaEvent_t> aux_event;   // [0] fork, [1 + i] join of aux stream i
  // CUDA graphs for the Krylov solvers of block-sparse operators (fmpt_set_graphs)
  bool graphs = true;
  // Krylov exponentials: one cooperative launch per Arnoldi orthogonalisation step
  // (fmpt_set_fused_krylov; the six separate launches give bit-identical results)
  int fused_gs = 1;
  // thin QR of small tall panels on one thread-block cluster (fmpt_set_cluster_qr)
  int cluster_qr = 1;
  int svd_method = 0;          // 0 gesvd (bidiagonalisation), 1 gesvdp (polar decomposition)
  int tc_tile = 0;             // tcgen05 GEMM tile: 0 CTA pair where it applies, 1 one CTA
  // split-K workspace of the FP64 GEMM, grown outside stream capture only (stream-ordered
  // reuse on h->stream)
  void* gemm_ws = nullptr;
  size_t gemm_ws_bytes = 0;
  // per-tile arrival counts of the split FP64 GEMM (zero between launches)
  void* gemm_cnt = nullptr;
  size_t gemm_cnt_bytes = 0;
  // partial tiles and arrival counters of the BF16 pair GEMM's K-split last round
  void* tc_ws = nullptr;
  size_t tc_ws_bytes = 0;
  // counters of the split tiles: zero between launches (the last piece of a tile resets its own,
  // in a launch that gives up too)
  void* tc_cnt = nullptr;
  size_t tc_cnt_bytes = 0;
  // FP64 GEMMs on the BF16 tensor cores (Ozaki scheme: residue planes, exponents,
  // the product's residues):
  // f64_tc 1 routes every FP64 GEMM of this handle there when its cost model says it is
  // faster than the CUDA-core kernel (fmpt_set_f64_engine)
  int f64_tc = 0;
  // set while fmpt_lanczos_ground runs: its tensor-core FP64 GEMMs are the digit products of
  // ozaki_digits.cu (see there), not the residue products of ozaki.cu
  int oz_digits = 0;
  // device flag of the Lanczos solve that is running, set while it queues a step ahead of its
  // stopping test: nonzero once the solve has stopped, and that step's GEMMs return at once
  const int* gate = nullptr;
  // 1 while an Arnoldi basis is built: small complex FP64 GEMMs may add K pieces (gemm_f64.cu)
  int k_pieces = 0;
  // failure-detection test hook (fmpt_set_wait_test): bound of the grouped kernel's barrier
  // waits (0: 2 s) and extra arrivals they wait for (0 in normal use)
  int64_t wait_test_ns = 0;
  int wait_test_hold = 0;
  void* oz_ws = nullptr;
  size_t oz_ws_bytes = 0;
  // row maxima of the residue GEMM's operands: zero between calls (its last kernel zeroes what
  // the call used) unless a call failed half-way (oz_mx_dirty)
  void* oz_mx = nullptr;
  size_t oz_mx_bytes = 0;
  bool oz_mx_dirty = true;
  cudaGraphExec_t lanczos_exec = nullptr;   // reused through cudaGraphExecUpdate
  uint64_t graph_launches = 0;
  // grouped-kernel tile autotuner (fmpt_set_tuning): 0 measure, 1 force the
  // 32x32 tile, 2 force 64x64; cache: (program kind, work bucket) -> variant
  int tune_mode = 0;
  std::map<int, int> tune_cache;
  uint64_t tune_runs = 0;
};

namespace fmpt {

int set_error(fmpt_handle* h, int status, const char* fmt, ...);

#define FMPT_CUDA(h, expr)                                                              \
  do {                                                                                  \
    cudaError_t _e = (expr);                                                            \
    if (_e != cudaSuccess)                                                              \
      return ::fmpt::set_error((h), _e == cudaErrorMemoryAllocation ? FMPT_ERR_NOMEM    \
                                                                    : FMPT_ERR_CUDA,    \
                               "%s:%d %s: %s", __FILE__, __LINE__, #expr,              \
                               cudaGetErrorString(_e));                                 \
  } while (0)

#define FMPT_TRY(expr)          \
  do {                          \
    int _s = (expr);            \
    if (_s != FMPT_OK) return _s; \
  } while (0)

#define FMPT_LAUNCHED(h)                                                                \
  do {                                                                                  \
    (h)->launches++;                                                                    \
    cudaError_t _e = cudaGetLastError();                                                \
    if (_e != cudaSuccess)                                                              \
      return ::fmpt::set_error((h), FMPT_ERR_CUDA, "%s:%d launch: %s", __FILE__,        \
                               __LINE__, cudaGetErrorString(_e));                       \
  } while (0)

// Kernels that follow one another in a stream overlap their launches (programmatic dependent
// launch): launch_chain lets the kernel be launched while its predecessor still runs, and
// chain_begin, before its first access to global memory, waits until every earlier kernel
// has completed with its writes visible (a plain launch of the same kernel waits for nothing
// there).  The predecessors do not release their successors early: blocks that wait beside a
// running grid start unevenly spread over the SMs, and a D = 64 Krylov exponential took 1.42 ms
// instead of 1.30 (1.42 with plain launches too).  An H_eff*x at D = 32, three kernels, 18.4 us
// with plain launches and 11.3 with these.
#ifdef __CUDACC__
__device__ __forceinline__ void chain_begin() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// The first statement of a kernel with a gate (fmpt_handle::gate): nothing is to be done.  Uniform
// for the whole grid, since an earlier kernel sets the flag.  Before the kernel's own chain_begin:
// read after it, the parameter alone cost 0.05 us per launch.
__device__ __forceinline__ bool gate_closed(const int* gate) {
  if (!gate) return false;
  chain_begin();
  return *gate != 0;
}

// 8 bytes by cp.async, zeros if !in
__device__ __forceinline__ void cp_async8z(double* dst, const double* src, bool in) {
  const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src),
               "r"(in ? 8 : 0)
               : "memory");
}

// Conversions between FP32 and FP64 on the integer pipe: a conversion instruction runs on the
// FP64 pipe of GB300, 64 cycles of its SM sub-partition, and the epilogues and layout kernels
// that widen or narrow every element were bound by it.  Zeros and normal numbers here; the rest
// (rare) through the instruction.
__device__ __forceinline__ bool widen_rare(uint32_t b) {     // denormal, Inf, NaN
  const uint32_t mag = b & 0x7fffffffu;
  return mag - 1u < 0x007fffffu || mag >= 0x7f800000u;
}
__device__ __forceinline__ double widen_common(uint32_t b) {
  const uint32_t mag = b & 0x7fffffffu;
  const uint32_t hi = (b & 0x80000000u) | (mag ? (mag >> 3) + 0x38000000u : 0u);
  double r;
  asm("mov.b64 %0, {%1, %2};" : "=d"(r) : "r"(b << 29), "r"(hi));
  return r;
}
__device__ __forceinline__ double widen(float v) {
  const uint32_t b = __float_as_uint(v);
  return widen_rare(b) ? (double)v : widen_common(b);
}
__device__ __forceinline__ bool is_one(double v) {           // an FP64 comparison takes the pipe too
  uint32_t lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "d"(v));
  return lo == 0u && hi == 0x3ff00000u;
}
__device__ __forceinline__ double xor_high(double v, uint32_t mask) {
  uint32_t lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "d"(v));
  asm("mov.b64 %0, {%1, %2};" : "=d"(v) : "r"(lo), "r"(hi ^ mask));
  return v;
}
// round to nearest even
__device__ __forceinline__ float narrow(double v) {
  uint32_t lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "d"(v));
  const uint32_t mag = hi & 0x7fffffffu;
  const uint32_t hm = mag - 0x38000000u;                     // exponent rebased
  if ((mag | lo) == 0u) return __uint_as_float(hi);
  if (hm - 0x00100000u >= 0x0fe00000u) return (float)v;      // below the normal range, above it
  uint32_t f = __funnelshift_l(lo, hm, 3);
  f += ((lo & 0x1fffffffu) + 0x0fffffffu + (f & 1u)) >> 29;
  return __uint_as_float(f | (hi & 0x80000000u));
}
inline void chain_attr(cudaLaunchAttribute& a) {
  a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  a.val.programmaticStreamSerializationAllowed = 1;
}
template <class... P, class... A>
cudaError_t launch_chain(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem,
                         cudaStream_t stream, A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  chain_attr(attr[0]);
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
#endif

// What a kernel needs to know or have set once per device (attributes, resident clusters), in N
// slots.  Handles of several host threads may ask at the same time.
template <int N = 1>
class PerDevice {
  static constexpr int kDevices = 64;
  std::mutex mu_;
  int value_[kDevices][N] = {};
  bool done_[kDevices][N] = {};

 public:
  // value = what find(value) has found for h's device; an error of find is returned and not kept
  template <class Find>
  int get(fmpt_handle* h, int slot, int& value, Find find) {
    if (h->device < 0 || h->device >= kDevices) return find(value);
    std::lock_guard<std::mutex> lock(mu_);
    if (!done_[h->device][slot]) {
      FMPT_TRY(find(value_[h->device][slot]));
      done_[h->device][slot] = true;
    }
    value = value_[h->device][slot];
    return FMPT_OK;
  }
};

// Stream-ordered device scratch owned by a C++ scope.
struct DevBuf {
  fmpt_handle* h = nullptr;
  void* p = nullptr;
  size_t bytes = 0;
  DevBuf() = default;
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
  ~DevBuf() { release(); }
  int alloc(fmpt_handle* hh, size_t nbytes);
  void release();
  double* d() const { return static_cast<double*>(p); }
};

int ensure_pinned(fmpt_handle* h, size_t n_doubles);
// the FP64 one-/two-site operator application in two halves (heff.cu): head = GEMM 1 and
// the MPO step into the operator's scratch, tail = GEMM 2 into y
int op_fp64_head(fmpt_op* op, const double* x);
int op_fp64_tail(fmpt_op* op, double* y);
// Q (m x n) and R (n x n) of a small tall panel (m >= n) on one thread-block cluster;
// FMPT_ERR_UNSUPPORTED (nothing launched) outside its range (qr_cluster.cu)
int qr_small_cluster(fmpt_handle* h, int cplx, int m, int n, const double* M, double* Q,
                     double* R);
// a device buffer of at least `bytes` held in *buf / *cap (stream-ordered on h->stream);
// growing it while h->stream is being captured returns FMPT_ERR_UNSUPPORTED
int grow_buffer(fmpt_handle* h, void** buf, size_t* cap, size_t bytes);
// At least n auxiliary streams/solvers; aux_fork makes them wait for the work
// queued so far on h->stream, aux_join makes h->stream wait for them.
int ensure_aux(fmpt_handle* h, int n);
int aux_fork(fmpt_handle* h, int n);
int aux_join(fmpt_handle* h, int n);

// Scoped device timer for one launch of a kernel class (no-op unless profiling).
struct ProfScope {
  fmpt_handle* h;
  int cls;
  cudaEvent_t b = nullptr, e = nullptr;
  ProfScope(fmpt_handle* hh, int c);
  ~ProfScope();
};

// Residue planes and exponents of one FP64 GEMM operand for the tensor-core FP64 engine,
// kept across calls by an owner whose operand does not change between them (a prepared
// operator's environments): built on first use, reused while src and shape match.
struct OzCache {
  const double* src = nullptr;
  int64_t key[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  void* buf = nullptr;
  size_t bytes = 0;
  bool valid = false;
};
void oz_cache_free(fmpt_handle* h, OzCache& c);

// -------- generic FP64 / split-complex GEMM (gemm_f64.cu)
// C = alpha op(A) op(B) + beta C ; planes: element offsets between re and im planes.
struct GemmArgs {
  int cplx;                 // 0 real, 1 split complex
  int ta, tb;               // fmpt_trans
  int m, n, k;
  double alpha[2], beta[2];
  const double* A; int64_t lda; int64_t planeA;
  const double* B; int64_t ldb; int64_t planeB;
  double* C; int64_t ldc; int64_t planeC;
  int batch;                // batched over blockIdx.z with the strides below
  int64_t strideA, strideB, strideC;
  int nosplit;              // 1: never split K (no workspace allocation)
  int engine;               // 0: the handle's FP64 engine, 1: tensor cores where faster
  OzCache* cacheA;          // optional residue-plane caches of A / B (tensor-core engine)
  OzCache* cacheB;
  // optional row maxima of op(A) (bit patterns of |.|, one per row of the real embedding), formed
  // by the kernel that wrote A; the residue GEMM zeroes them after use and then sets *maxA_clean
  unsigned long long* maxA;
  bool* maxA_clean;
  const int* gate;          // the handle's (filled in by gemm_f64)
};
int gemm_f64(fmpt_handle* h, const GemmArgs& g);
// the Ozaki-scheme FP64 GEMM on the BF16 tensor cores (ozaki.cu): whether it applies to g
// (engine requested, shape large enough to win), and the call itself
int gemm_f64_ozaki_possible(fmpt_handle* h, const GemmArgs& g);
bool gemm_f64_ozaki_takes_maxima(fmpt_handle* h, const GemmArgs& g);   // would use g.maxA
int gemm_f64_ozaki(fmpt_handle* h, const GemmArgs& g);
// the same by digit products (ozaki_digits.cu), inside the Lanczos solve
int gemm_f64_digits_possible(fmpt_handle* h, const GemmArgs& g);
int gemm_f64_digits(fmpt_handle* h, const GemmArgs& g);
// the handle's device status word (1: a bounded device wait timed out), read and cleared by
// gp_check_status / fmpt_synchronize
int gp_status_word(fmpt_handle* h, int** out);
inline bool prec_is_f64(int precision) {
  return precision == FMPT_PREC_FP64 || precision == FMPT_PREC_FP64_TC;
}

// -------- block-sparse MPO "middle" contraction (heff.cu)
// out[o1, o2, wo, so] = sum_{blocks (wi -> wo)} sum_si coef[so, si] in[o1, o2, wi, si]
constexpr int MS_MAX_OUT = 128, MS_MAX_T = 512;   // sparse MPO-step table capacity
struct MidSchedule {
  int nw_in = 0, nw_out = 0, p_in = 0, p_out = 0, cplx = 0;
  std::vector<int> blk_win;      // per block: input w
  std::vector<int> wout_start;   // nw_out + 1 prefix offsets into the blocks (sorted by wo)
  std::vector<double> coef;      // per block: p_out x p_in (row-major so, si), re then im if cplx
  // the nonzero terms per output (wo, so): prefix offsets, wi * 16 + si, coefficients (re, im
  // pairs if cplx); empty when they exceed the by-value table of the sparse kernel
  std::vector<int> sp_start, sp_idx;
  std::vector<double> sp_coef;
  // device copies
  int* d_win = nullptr;
  int* d_wstart = nullptr;
  double* d_coef = nullptr;
  int nblocks() const { return (int)blk_win.size(); }
};
int mid_upload(fmpt_handle* h, MidSchedule& s);
void mid_free(fmpt_handle* h, MidSchedule& s);
struct MidStrides { int64_t o1, o2, w, s; };
// mx: optionally the maxima over (wo, o2) of |out| per row o1 + n1 so of the real embedding (a
// complex product's rows appear twice); only with a by-value table (sp_start not empty)
int mid_apply(fmpt_handle* h, const MidSchedule& s, const double* in, int64_t plane_in,
              MidStrides si, double* out, int64_t plane_out, MidStrides so, int n1, int n2,
              unsigned long long* mx = nullptr);

// Schedules from dense host MPO tensors (W[wl, s_out, wr, s_in]).
int schedule_ac2(fmpt_handle* h, int cplx, const double* W1, const double* W2, int d1, int d2,
                 int wl, int wm, int wr, MidSchedule& s);
// the host part of schedule_ac2: fills s.blk_win / s.wout_start / s.coef, uploads nothing
void schedule_ac2_host(int cplx, const double* W1, const double* W2, int d1, int d2, int wl,
                       int wm, int wr, MidSchedule& s);
int schedule_ac(fmpt_handle* h, int cplx, const double* W, int d, int wl, int wr, MidSchedule& s);
// updateright maps the right index w2 (input) to the left index w (output)
int schedule_env(fmpt_handle* h, int cplx, const double* W, int d, int wl, int wr, bool right,
                 MidSchedule& s);

// -------- grouped persistent block-sparse engine (grouped.cu)
constexpr int GP_MAX_PHASES = 4, GP_SLOTS = 8;
// variants 0-3: (tile, schedule), v & 1 -> 32x32 / 64x64 tiles of a block, v >> 1 -> schedule;
// GP_WARP: 8x4 tiles of a warp
constexpr int GP_VARIANTS = 5, GP_WARP = 4;
enum { GP_GEMM = 0, GP_SUM = 1 };
// One output block: C (m x n, column-major with ldc) at c_off in the phase's C slot.
struct GProblem {
  int64_t c_off, ldc;
  int m, n, seg0, seg1;
};
// One term of a block: coef * op(A) op(B) (GEMM, inner extent k) or coef * A (SUM).
struct GSegment {
  int64_t a_off, lda, b_off, ldb;
  double coef;
  int k, pad;
};
// GP_WARP: a block in its phase's order with the number of tiles before it
struct GWarpProb {
  GProblem p;
  int tile0, pad;
};
struct GPhaseDesc {
  int type, ta, tb, a_slot, b_slot, c_slot, tile0, tile1;
};
struct GroupedProgram {
  std::vector<GPhaseDesc> phases;
  std::vector<int> phase_prob0;
  std::vector<GProblem> probs;
  std::vector<GSegment> segs;
  std::vector<int> tile_prob, tile_mn;           // the tiles of variants 0-3, one after another
  std::vector<int> vtile0[GP_VARIANTS], vtile1[GP_VARIANTS];   // per variant and phase
  int vgrid[GP_VARIANTS] = {0, 0, 0, 0, 0};
  int variant = GP_WARP;                          // the one gp_run launches by default
  double flops = 0.0;       // 2 m n k over the GEMM segments
  double sum_elems = 0.0;   // output elements x terms of the SUM phases
  int64_t slot_elems[GP_SLOTS] = {-1, -1, -1, -1, -1, -1, -1, -1};  // operand extents
  DevBuf dev;
  GProblem* d_probs = nullptr;
  GSegment* d_segs = nullptr;
  int* d_tile_prob = nullptr;
  int* d_tile_mn = nullptr;
  GWarpProb* d_wprob = nullptr;                   // GP_WARP: blocks by descending work
  int* d_ctl = nullptr;
  bool ready = false;
};
// Builder: a phase, then its problems, each followed by its segments.
void gp_phase(GroupedProgram& g, int type, int ta, int tb, int a_slot, int b_slot, int c_slot);
int gp_problem(GroupedProgram& g, int64_t c_off, int64_t ldc, int m, int n);
void gp_segment(GroupedProgram& g, int64_t a_off, int64_t lda, int64_t b_off, int64_t ldb, int k,
                double coef);
// Declares how many doubles operand slot `slot` holds; gp_finalize checks every
// block footprint against it (host side, before anything reaches the GPU).
void gp_slot(GroupedProgram& g, int slot, int64_t elems);
int gp_finalize(fmpt_handle* h, GroupedProgram& g);   // bounds check + tiles + upload
// gate: optional device flag; when it is nonzero at launch time every CTA
// returns at once (a solver step after convergence inside a CUDA graph)
int gp_run(fmpt_handle* h, const GroupedProgram& g, double* const* slots, int nslots,
           const int* gate = nullptr, int variant = -1);
int gp_prepare(fmpt_handle* h);   // allocations gp_run needs, done before a stream capture
// Picks g.variant: the handle's cached choice for (kind, work bucket), else
// (tune mode 0) times every variant on these slots -- the program must be
// safe to run repeatedly on them -- and caches the fastest.
enum { GP_KIND_HEFF = 1, GP_KIND_ENV = 2, GP_KIND_OTHER = 3 };
int gp_autotune(fmpt_handle* h, GroupedProgram& g, double* const* slots, int nslots, int kind);
int gp_check_status(fmpt_handle* h);                  // synchronises; FMPT_ERR_TIMEOUT if set

// -------- dense helpers shared with the sector code (linalg.cu)
int copy_mat(fmpt_handle* h, int cplx, int rows, int cols, const double* src, int64_t s_ld,
             int64_t s_plane, int trans, int conj, double* dst, int64_t d_ld, int64_t d_plane);
int svd_tall(fmpt_handle* h, int cplx, int m, int n, double* Awork, double* S, double* U,
             double* VT);

// -------- vector kernels (krylov.cu)
int vec_dot_dev(fmpt_handle* h, int cplx, int64_t n, const double* x, const double* y,
                double* out_dev /* re, im */);
int vec_nrm2_dev(fmpt_handle* h, int cplx, int64_t n, const double* x, double* out_dev);

}  // namespace fmpt

// The opaque operator type of the C ABI.
struct fmpt_op {
  fmpt_handle* h = nullptr;
  int kind = 0;          // 0 ac2, 1 ac, 2 c
  int dtype = FMPT_F64;
  int precision = FMPT_PREC_FP64;
  int Dl = 0, Dr = 0, d1 = 1, d2 = 1, wl = 1, wm = 1, wr = 1;
  const double* hleft = nullptr;
  const double* hright = nullptr;
  fmpt::MidSchedule sched;
  int64_t n = 0;          // vector length (complex elements for C128)
  void* tc = nullptr;     // tensor-core state (mixed precision), owned
  void* u1 = nullptr;     // U(1) block-sparse state (grouped program + scratch), owned
  bool defer_right = false;  // mixed precision: the right environment is converted later
  // FP64 intermediates of one application (T1/T3 or T), grown outside stream capture only
  double* scratch = nullptr;
  // residue planes of the environments for the tensor-core FP64 engine (FP64_TC operators)
  fmpt::OzCache oz_left, oz_right;
  fmpt::OzCache ozd_left, ozd_right;   // digit planes (the Lanczos solve's engine)
  size_t scratch_bytes = 0;
  // row maxima of T3 behind it in the scratch: formed by the last head; zero (which they are
  // again after a tail unless the zeros were only recorded, mx_keep)
  bool mx_ready = false, mx_clean = false, mx_keep = false;
  // projectors of the excited-state sweeps: after every application
  // y -= dot(y, p) p for each p in order (device vectors of n elements, not owned)
  std::vector<const double*> proj;
  double* proj_part = nullptr;   // 2 * proj_G block partials, owned
  int proj_G = 0;
};

namespace fmpt {
int op_apply_fp64(fmpt_op* op, const double* x, double* y);
int op_tc_prepare(fmpt_op* op);
int op_tc_apply(fmpt_op* op, const double* x, double* y);
// split application of a real tensor-core two-site operator (host-buffer pipeline):
// head = x conversion, GEMM 1 and MPO step; tail = GEMM 2; prepare_right converts the
// right environment of an operator created with defer_right
// (x null: its operand planes, op_tc_planes, have been written already)
int op_tc_apply_head(fmpt_op* op, const double* x);
// where a real tensor-core operator keeps the operand planes of x: element i of x at element i of
// hi (and, for 3xTF32, lo); mode < 0 where the layout is another one
struct TcPlanes { int mode = -1; void* hi = nullptr; void* lo = nullptr; };
TcPlanes op_tc_planes(fmpt_op* op);
int op_apply_planes(fmpt_op* op, double* y);   // fmpt_op_apply on those planes
int op_tc_apply_tail(fmpt_op* op, double* y);
int op_tc_prepare_right(fmpt_op* op);
// the same for the rows b' in [r0, r1) of the right environment / columns of y
int op_tc_prepare_right_rows(fmpt_op* op, int r0, int r1);
int op_tc_apply_tail_rows(fmpt_op* op, double* y, int r0, int r1);
int op_tc_check(fmpt_op* op);   // reads the device timeout flag (synchronises)
// mixed-precision environment update (real data), FP64 output in the reference layout
int env_update_tc(fmpt_handle* h, bool right, int precision, const double* hold, const double* A,
                  const double* W, const double* B, double* hnew, int Dl, int d, int Dr, int wl,
                  int wr);
void op_tc_free(fmpt_op* op);
int op_u1_apply(fmpt_op* op, const double* x, double* y, const int* gate = nullptr);
// the projections of op->proj applied to y in place (no-op without projectors)
int op_project(fmpt_op* op, double* y, const int* gate = nullptr);
void op_u1_free(fmpt_op* op);

// K-major tensor-core operand: TF32 (float storage) or BF16 plane, optional
// TF32 low plane (3xTF32), row stride and batch stride in elements.
struct TcOperand {
  const void* hi;
  const void* lo;
  int64_t ld;
  int64_t bstride;
};
// C[m, n] (+ batch) = sum_k A[m, k] B[n, k] on tcgen05; mode 0 TF32, 1 3xTF32, 2 BF16;
// C is FP32 (out_f64 = 0), FP64 (1) or, in BF16 mode, BF16 (2); column-major with ldc.
int tc_gemm(fmpt_handle* h, int mode, int M, int N, int K, int batch, const TcOperand& A,
            const TcOperand& B, void* C, int out_f64, int64_t ldc, int64_t strideC, int* err_dev);
}  // namespace fmpt
