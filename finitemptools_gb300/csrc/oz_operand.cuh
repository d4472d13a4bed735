// Operands of the FP64 GEMMs on the BF16 tensor cores (ozaki.cu, ozaki_digits.cu): the index
// space of op(X), tiles of FP64 bit patterns, and the row maxima that set the exponents.
#pragma once
#include "tc_ptx.cuh"

namespace fmpt {
namespace {

// op(X)(r, c) of a GEMM operand, real index space: X[r * sr + c * sc] (+ batch stride).
// Complex operands are embedded as real matrices with doubled extents: the A side as
// rows [Re, -Im] over [Im, Re], the B side (rows = output columns) as [Re, Im].
struct SliceSrc {
  const double* p;
  int64_t plane;        // offset of the imaginary plane
  int64_t sr, sc;       // element strides of row and column index
  int64_t bstride;      // batch stride
  int rows, cols;       // real extents of op(X)
  int cplx, role, conj; // role 0: A side, 1: B side
};

__device__ __forceinline__ uint64_t src_bits(const SliceSrc& s, int z, int r2, int c2) {
  int r = r2, c = c2, hr = 0, hc = 0;
  if (s.cplx) {
    if (s.role == 0 && r >= s.rows) { r -= s.rows; hr = 1; }
    if (c >= s.cols) { c -= s.cols; hc = 1; }
  }
  // the imaginary part sits at (hr, hc) = (0, 1) with a minus sign and at (1, 0) on the
  // A side, at hc = 1 on the B side; conj flips its sign once more
  bool im = false, neg = false;
  if (s.cplx) {
    if (s.role == 0) {
      im = hr != hc;
      neg = hr == 0 && hc == 1;
    } else {
      im = hc == 1;
    }
    if (im && s.conj) neg = !neg;
  }
  const double* b = s.p + (int64_t)z * s.bstride + (int64_t)r * s.sr + (int64_t)c * s.sc;
  uint64_t v = __ldg(reinterpret_cast<const unsigned long long*>(b + (im ? s.plane : 0)));
  if (neg) v ^= 0x8000000000000000ull;
  return v;
}

constexpr int SL_ROWS = 32;           // rows of a slicing block
constexpr int SL_KCH = 512;           // K columns of a slicing block (8 tiles of 64)

// A 32 x 64 tile of op(X) bit patterns: element e = t + 256 q of thread t (q < 8) is
// (row, column) = (e & 31, e >> 5) when rows are contiguous in the source and
// (e >> 6, e & 63) otherwise, so that every warp load is contiguous; zeros outside the
// operand.  The loads go to registers first, so that a block can fetch its next tile
// while it works on the current one.
__device__ __forceinline__ void tile_pos(bool rowfast, int e, int& lr, int& lc) {
  if (rowfast) { lr = e & 31; lc = e >> 5; } else { lc = e & 63; lr = e >> 6; }
}

__device__ __forceinline__ void fetch_tile(const SliceSrc& src, int z, int r0, int c0, int rows_out,
                                           int k_out, uint64_t (&v)[8]) {
  const int t = threadIdx.x;
  const bool rowfast = src.sr == 1;
#pragma unroll
  for (int q = 0; q < 8; q++) {
    int lr, lc;
    tile_pos(rowfast, t + 256 * q, lr, lc);
    const int r = r0 + lr, c = c0 + lc;
    v[q] = (r < rows_out && c < k_out) ? src_bits(src, z, r, c) : 0ull;
  }
}

// Row maxima of |X| on the bit patterns (non-negative IEEE doubles order as their bits):
// block (strip, K chunk, batch) reduces its 32 x SL_KCH part and folds it into mx with an
// atomic max (mx zeroed beforehand).
__global__ void __launch_bounds__(256, 4) oz_rowmax(SliceSrc src, int rows_out, int k_out,
                                                 unsigned long long* __restrict__ mx) {
  chain_begin();
  __shared__ unsigned long long smax[SL_ROWS];
  const int r0 = blockIdx.x * SL_ROWS, kc0 = blockIdx.y * SL_KCH, z = blockIdx.z;
  const int t = threadIdx.x;
  const bool rowfast = src.sr == 1;
  if (t < SL_ROWS) smax[t] = 0ull;
  // rows of this thread's elements: one row (rowfast) or rows (t >> 6) + 4 q
  uint64_t m[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  const int c1 = min(kc0 + SL_KCH, k_out);
  uint64_t v[8];
  if (kc0 < c1) fetch_tile(src, z, r0, kc0, rows_out, k_out, v);
  for (int c0 = kc0; c0 < c1; c0 += 64) {
    uint64_t cur[8];
#pragma unroll
    for (int q = 0; q < 8; q++) cur[q] = v[q] & 0x7fffffffffffffffull;
    if (c0 + 64 < c1) fetch_tile(src, z, r0, c0 + 64, rows_out, k_out, v);
#pragma unroll
    for (int q = 0; q < 8; q++) m[q] = cur[q] > m[q] ? cur[q] : m[q];
  }
  __syncthreads();
  if (rowfast) {
    uint64_t a = m[0];
#pragma unroll
    for (int q = 1; q < 8; q++) a = m[q] > a ? m[q] : a;
    if (a) atomicMax(&smax[t & 31], (unsigned long long)a);
  } else {
    // the 64 threads of a row group share their rows: fold across the warp's halves
#pragma unroll
    for (int q = 0; q < 8; q++) {
      uint64_t a = m[q];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint64_t y = __shfl_xor_sync(0xffffffffu, a, o);
        a = y > a ? y : a;
      }
      if ((t & 31) == 0 && a) atomicMax(&smax[(t >> 6) + 4 * q], (unsigned long long)a);
    }
  }
  __syncthreads();
  const int r = r0 + t;
  if (t < SL_ROWS && r < rows_out && smax[t] != 0) atomicMax(mx + (int64_t)z * rows_out + r, smax[t]);
}

// ------------------------------------------------------------ fast conversion of real operands
// Real operands whose row or K index has unit stride take these kernels instead of the generic
// ones above: eight independent loads in flight per thread and no shared-memory staging for the
// row maxima, the residues of a K-contiguous operand straight from registers.  The generic
// kernels are bound by memory latency (long-scoreboard stalls, 22-37% of DRAM bandwidth).
// V = 2: 16-byte loads, for 16-byte aligned rows or columns and an even extent along the
// unit-stride index; V = 1: 8-byte loads, for the rest.  Loaded as integers: from doubles, the
// compiler turns the masking of the sign into an FP64 instruction per element (kfast 37 -> 23 us
// at 2048 x 8192).
constexpr int RK_KCH = 1024;          // K columns per block, K-contiguous row maxima

template <int V>
struct OzBits {
  uint64_t x[V];
};
// V doubles' bits without their signs; zeros if !in
template <int V>
__device__ __forceinline__ OzBits<V> oz_load_abs(const double* p, bool in) {
  constexpr uint64_t kAbs = 0x7fffffffffffffffull;
  OzBits<V> r{};
  if constexpr (V == 2) {
    const ulonglong2 v =
        in ? __ldg(reinterpret_cast<const ulonglong2*>(p)) : make_ulonglong2(0, 0);
    r.x[0] = v.x & kAbs;
    r.x[1] = v.y & kAbs;
  } else {
    r.x[0] = in ? __ldg(reinterpret_cast<const unsigned long long*>(p)) & kAbs : 0ull;
  }
  return r;
}

// rows r .. r + V - 1 of a row-contiguous operand (element (r, c) at p[r + c ld])
template <int V>
__global__ void __launch_bounds__(128) oz_rowmax_rowfast(const double* __restrict__ p, int64_t ld,
                                                         int64_t bstride, int rows, int k, int kch,
                                                         unsigned long long* __restrict__ mx) {
  chain_begin();
  const int z = blockIdx.z;
  const int r = (blockIdx.x * 128 + threadIdx.x) * V;
  const int c0 = blockIdx.y * kch, c1 = min(c0 + kch, k);
  if (r >= rows) return;
  const double* b = p + (int64_t)z * bstride + r;
  uint64_t m[V] = {};
  for (int c = c0; c < c1; c += 8) {
    OzBits<V> v[8];
#pragma unroll
    for (int u = 0; u < 8; u++) v[u] = oz_load_abs<V>(b + (int64_t)(c + u) * ld, c + u < c1);
#pragma unroll
    for (int u = 0; u < 8; u++)
#pragma unroll
      for (int q = 0; q < V; q++) m[q] = v[u].x[q] > m[q] ? v[u].x[q] : m[q];
  }
#pragma unroll
  for (int q = 0; q < V; q++)
    if (m[q]) atomicMax(mx + (int64_t)z * rows + r + q, (unsigned long long)m[q]);
}

// one warp per row of a K-contiguous operand (element (r, c) at p[r ld + c])
template <int V>
__global__ void __launch_bounds__(256) oz_rowmax_kfast(const double* __restrict__ p, int64_t ld,
                                                       int64_t bstride, int rows, int k,
                                                       unsigned long long* __restrict__ mx) {
  chain_begin();
  const int z = blockIdx.z, lane = threadIdx.x & 31;
  const int r = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (r >= rows) return;                                   // uniform over the warp
  const int c0 = blockIdx.y * RK_KCH, c1 = min(c0 + RK_KCH, k);
  const double* b = p + (int64_t)z * bstride + (int64_t)r * ld;
  uint64_t m = 0;
  for (int c = c0 + V * lane; c < c1; c += 32 * V * 8) {
    OzBits<V> v[8];
#pragma unroll
    for (int u = 0; u < 8; u++) v[u] = oz_load_abs<V>(b + c + 32 * V * u, c + 32 * V * u < c1);
#pragma unroll
    for (int u = 0; u < 8; u++)
#pragma unroll
      for (int q = 0; q < V; q++) m = v[u].x[q] > m ? v[u].x[q] : m;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const uint64_t y = __shfl_xor_sync(0xffffffffu, m, o);
    m = y > m ? y : m;
  }
  if (lane == 0 && m) atomicMax(mx + (int64_t)z * rows + r, (unsigned long long)m);
}

// 8-byte cp.async ring of a row-contiguous operand's tiles
constexpr int DR_STAGES = 3;
constexpr size_t DR_SMEM = (size_t)DR_STAGES * SL_ROWS * 65 * sizeof(uint64_t);

__device__ __forceinline__ void cp_async8(uint64_t* dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(tc::smem_u32(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}


// 16-byte loads along the unit-stride index (extent n, other stride ld)
inline bool oz_aligned(const SliceSrc& x, int64_t ld, int n) {
  return (reinterpret_cast<uintptr_t>(x.p) & 15) == 0 && (ld & 1) == 0 && (x.bstride & 1) == 0 &&
         (n & 1) == 0;
}
inline bool oz_kfast(const SliceSrc& x) { return !x.cplx && x.sc == 1; }

// Row maxima of |op(X)| (bit patterns) into mx, zeroed by the caller.
inline int oz_row_maxima(fmpt_handle* h, const SliceSrc& x, int rows, int k, int batch,
                         unsigned long long* mx) {
  if (!x.cplx && x.sr == 1) {
    const bool two = oz_aligned(x, x.sc, rows);
    // K columns per block (a multiple of the eight loads in flight): short enough for about
    // 16 blocks per SM, so that a small operand is spread out (1024 x 1280: 35 us on 20
    // blocks) and a large one ends evenly, at most 128
    const int gx = (rows / (two ? 2 : 1) + 127) / 128;
    const int64_t want = (int64_t)k * gx * batch / (16LL * std::max(1, h->sm_count));
    const int kc = (int)std::max<int64_t>(8, std::min<int64_t>(128, want) / 8 * 8);
    const dim3 g1((unsigned)gx, (unsigned)((k + kc - 1) / kc), (unsigned)batch);
    if (two)
      FMPT_CUDA(h, launch_chain(oz_rowmax_rowfast<2>, g1, 128, 0, h->stream, x.p, x.sc, x.bstride,
                                rows, k, kc, mx));
    else
      FMPT_CUDA(h, launch_chain(oz_rowmax_rowfast<1>, g1, 128, 0, h->stream, x.p, x.sc, x.bstride,
                                rows, k, kc, mx));
  } else if (oz_kfast(x)) {
    const dim3 g1((unsigned)((rows + 7) / 8), (unsigned)((k + RK_KCH - 1) / RK_KCH),
                  (unsigned)batch);
    if (oz_aligned(x, x.sr, k))
      FMPT_CUDA(h, launch_chain(oz_rowmax_kfast<2>, g1, 256, 0, h->stream, x.p, x.sr, x.bstride,
                                rows, k, mx));
    else
      FMPT_CUDA(h, launch_chain(oz_rowmax_kfast<1>, g1, 256, 0, h->stream, x.p, x.sr, x.bstride,
                                rows, k, mx));
  } else {
    const dim3 g1((unsigned)((rows + SL_ROWS - 1) / SL_ROWS),
                  (unsigned)((k + SL_KCH - 1) / SL_KCH), (unsigned)batch);
    FMPT_CUDA(h, launch_chain(oz_rowmax, g1, 256, 0, h->stream, x, rows, k, mx));
  }
  FMPT_LAUNCHED(h);
  return FMPT_OK;
}

// op(A) (m x k) as the A side, op(B)^T (n x k) as the B side
inline SliceSrc oz_side_a(const GemmArgs& g) {
  SliceSrc s{};
  s.p = g.A; s.plane = g.planeA; s.bstride = g.strideA; s.rows = g.m; s.cols = g.k;
  s.cplx = g.cplx ? 1 : 0; s.role = 0; s.conj = (g.ta == FMPT_C || g.ta == FMPT_R);
  if (g.ta == FMPT_N || g.ta == FMPT_R) { s.sr = 1; s.sc = g.lda; } else { s.sr = g.lda; s.sc = 1; }
  return s;
}
inline SliceSrc oz_side_b(const GemmArgs& g) {
  SliceSrc s{};
  s.p = g.B; s.plane = g.planeB; s.bstride = g.strideB; s.rows = g.n; s.cols = g.k;
  s.cplx = g.cplx ? 1 : 0; s.role = 1; s.conj = (g.tb == FMPT_C || g.tb == FMPT_R);
  // op(B)(c, n) = B[c + n ldb] (N, R) or B[n + c ldb] (T, C)
  if (g.tb == FMPT_N || g.tb == FMPT_R) { s.sr = g.ldb; s.sc = 1; } else { s.sr = 1; s.sc = g.ldb; }
  return s;
}

// whether an operand's cached planes are those of (src, key)
inline bool oz_cache_hit(const OzCache* c, const double* src, const int64_t* key) {
  if (!c || !c->valid || c->src != src) return false;
  for (int i = 0; i < 8; i++)
    if (c->key[i] != key[i]) return false;
  return true;
}

}  // namespace
}  // namespace fmpt
