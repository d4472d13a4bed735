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
// Real operands whose row or K index has unit stride (with 16-byte aligned rows or columns)
// take these kernels instead of the generic ones above: 16-byte loads, eight independent
// loads in flight per thread and no shared-memory staging for the row maxima, the residues
// of a K-contiguous operand straight from registers.  The generic kernels are bound by
// memory latency (long-scoreboard stalls, 22-37% of DRAM bandwidth).
constexpr int RK_KCH = 1024;          // K columns per block, K-contiguous row maxima

// Loaded as integers: from doubles, the compiler turns the masking of the sign into an FP64
// instruction per element (kfast 37 -> 23 us at 2048 x 8192).
// rows r, r + 1 of a row-contiguous operand (element (r, c) at p[r + c ld])
__global__ void __launch_bounds__(128) oz_rowmax_rowfast(const double* __restrict__ p, int64_t ld,
                                                         int64_t bstride, int rows, int k, int kch,
                                                         unsigned long long* __restrict__ mx) {
  chain_begin();
  const int z = blockIdx.z;
  const int r = (blockIdx.x * 128 + threadIdx.x) * 2;
  const int c0 = blockIdx.y * kch, c1 = min(c0 + kch, k);
  if (r >= rows) return;
  const double* b = p + (int64_t)z * bstride + r;
  uint64_t m0 = 0, m1 = 0;
  for (int c = c0; c < c1; c += 8) {
    ulonglong2 v[8];
#pragma unroll
    for (int u = 0; u < 8; u++)
      v[u] = c + u < c1 ? __ldg(reinterpret_cast<const ulonglong2*>(b + (int64_t)(c + u) * ld))
                        : make_ulonglong2(0, 0);
#pragma unroll
    for (int u = 0; u < 8; u++) {
      const uint64_t a0 = v[u].x & 0x7fffffffffffffffull, a1 = v[u].y & 0x7fffffffffffffffull;
      m0 = a0 > m0 ? a0 : m0;
      m1 = a1 > m1 ? a1 : m1;
    }
  }
  if (m0) atomicMax(mx + (int64_t)z * rows + r, (unsigned long long)m0);
  if (m1) atomicMax(mx + (int64_t)z * rows + r + 1, (unsigned long long)m1);
}

// one warp per row of a K-contiguous operand (element (r, c) at p[r ld + c])
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
  for (int c = c0 + 2 * lane; c < c1; c += 64 * 8) {
    ulonglong2 v[8];
#pragma unroll
    for (int u = 0; u < 8; u++)
      v[u] = c + 64 * u < c1 ? __ldg(reinterpret_cast<const ulonglong2*>(b + c + 64 * u))
                             : make_ulonglong2(0, 0);
#pragma unroll
    for (int u = 0; u < 8; u++) {
      const uint64_t a0 = v[u].x & 0x7fffffffffffffffull, a1 = v[u].y & 0x7fffffffffffffffull;
      m = a0 > m ? a0 : m;
      m = a1 > m ? a1 : m;
    }
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


// Row maxima of |op(X)| (bit patterns) into mx, zeroed by the caller.  The fast kernels need
// a real operand with a unit-stride index, 16-byte aligned rows or columns and an even
// extent along the unit-stride index.
inline bool oz_aligned(const SliceSrc& x, int64_t ld) {
  return !x.cplx && (reinterpret_cast<uintptr_t>(x.p) & 15) == 0 && (ld & 1) == 0 &&
         (x.bstride & 1) == 0;
}
inline bool oz_kfast(const SliceSrc& x, int k) {
  return x.sc == 1 && oz_aligned(x, x.sr) && (k & 1) == 0;
}
inline int oz_row_maxima(fmpt_handle* h, const SliceSrc& x, int rows, int k, int batch,
                         unsigned long long* mx) {
  if (x.sr == 1 && oz_aligned(x, x.sc) && (rows & 1) == 0) {
    // K columns per block (a multiple of the eight loads in flight): short enough for about
    // 16 blocks per SM, so that a small operand is spread out (1024 x 1280: 35 us on 20
    // blocks) and a large one ends evenly, at most 128
    const int gx = (rows / 2 + 127) / 128;
    const int64_t want = (int64_t)k * gx * batch / (16LL * std::max(1, h->sm_count));
    const int kc = (int)std::max<int64_t>(8, std::min<int64_t>(128, want) / 8 * 8);
    const dim3 g1((unsigned)gx, (unsigned)((k + kc - 1) / kc), (unsigned)batch);
    FMPT_CUDA(h, launch_chain(oz_rowmax_rowfast, g1, 128, 0, h->stream, x.p, x.sc, x.bstride, rows, k, kc, mx));
  } else if (oz_kfast(x, k)) {
    const dim3 g1((unsigned)((rows + 7) / 8), (unsigned)((k + RK_KCH - 1) / RK_KCH),
                  (unsigned)batch);
    FMPT_CUDA(h, launch_chain(oz_rowmax_kfast, g1, 256, 0, h->stream, x.p, x.sr, x.bstride, rows, k, mx));
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
