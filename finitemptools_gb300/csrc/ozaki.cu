// FP64-accurate GEMM on the BF16 tensor cores (residue number system).
//
// GB300 runs FP64 on the CUDA cores at about 2 DFMA per clock per SM (~1.2 TFLOP/s for
// the whole chip) while its BF16 tensor cores run three orders of magnitude faster.  The
// FP64-accurate contractions therefore use the modular technique of Ozaki, Uchino and
// Imamura ("Ozaki scheme II", arXiv:2504.08009, 2025):
//
//   1. every row r of op(A) (and every column n of op(B)) gets an exponent e with
//      max |row| < 2^e, and its entries become integers
//        X(r, k) = round(x(r, k) 2^(t - e)),   |X| <= 2^t,
//      t >= 53 bits below the row maximum (every FP64 entry in the top binade of its row is
//      represented exactly);
//   2. the integer product sum_k A(r, k) B(n, k) is below P / 2 in magnitude, P the product
//      of NMOD pairwise coprime moduli p <= 256, so its residues modulo the p determine it.
//      A residue in [-128, 128] is an exact BF16 value, and the tensor cores multiply the
//      residue planes of each modulus (tcgen05.mma kind::f16, BF16 x BF16 -> FP32): over a
//      K chunk of 1024 the sums stay within 2^24, so the FP32 accumulation is exact.  After
//      each chunk the epilogue warps reduce the accumulator modulo p; what remains of a
//      tile is one byte per entry and modulus;
//   3. the Chinese remainder theorem gives X / P = frac(sum_i c_i w_i), w_i the rational
//      (P / p_i)^-1 mod p_i over p_i, summed in 96-bit fixed point with integer
//      instructions, and the FP64 result is put together from the top 64 bits of X: one
//      rounding, no FP64 instruction.
//
// The products and sums are exact, so the error is that of step 1 (2^-54 of the row or
// column maximum per entry, or less) and one rounding.  t follows from K: with 15 moduli
// (P = 2^118.0) t >= 53 up to K = 2048, with 16 (2^125.6) t = 56 up to K = 6295 and 55 at
// K = 10240; more moduli are not needed, fewer do not hold two 53-bit factors.  That is 15
// or 16 BF16 multiply-adds per FP64 one, against 45 of the digit products (ozaki_digits.cu):
// a two-site H_eff*x at w = 5 takes 7.8 ms at D = 2048 (17.6 ms there), 0.076 ms at D = 256
// (0.25).  Error of a product of random matrices relative to its norm, against 113-bit
// references: 2.6e-16 at K = 2048 (15 moduli), 5e-17 at K = 5120 (16); of the digit form, which
// drops the products below 2^-60 of the row and column maxima, 1.2e-15 and 1.9e-15.  The GEMM
// runs 1.73 to 1.75 PFLOP/s of BF16 work at D = 2048, 0.98 to 0.99 of the sustained cuBLAS rate.
// Complex operands use the real embedding [Re -Im; Im Re] x [Re; Im].
//
// Kernels: oz_rowmax* / oz_residues* (FP64 operand -> row exponents and NMOD K-major BF16
// residue planes), oz_gemm_pair (CTA-pair tcgen05 GEMM over (modulus, tile) items with the
// modular epilogue), oz_crt (bytes -> FP64 output, alpha / beta).
#include <algorithm>
#include <cmath>

#include "oz_operand.cuh"

namespace fmpt {
namespace oz {

using namespace tc;

constexpr int MAXMOD = 16;
constexpr int STAGES = 6;
constexpr int KELEMS = 64;            // BF16 elements per 128-byte K slice
constexpr int KCHUNK = 16;            // K slices per exactness chunk: 1024 * 128^2 = 2^24
constexpr int KMAX = 1 << 17;         // largest K of one launch (chunk sums fit 16 bits)
constexpr int GH = 8;                 // tile rows per group of the tile order
constexpr int E_BAD = 1 << 20;        // exponent of a row or column holding Inf / NaN
constexpr int TILE = 256;             // pair tile edge
constexpr int EPI_WARPS = 8;
constexpr int NTHR = 64 + 32 * EPI_WARPS;   // producer, MMA issuer, epilogue warps

// ------------------------------------------------------------ moduli and their constants
// the 15 and 16 pairwise coprime numbers up to 256 of the largest product (a search over all)
__host__ __device__ constexpr int modulus(int i) {
  constexpr int p[MAXMOD] = {256, 253, 251, 249, 247, 241, 239, 235,
                             233, 229, 227, 223, 217, 211, 199, 197};
  return p[i];
}
// log2 of the product of the first n moduli, rounded down to 1/100
constexpr double log2_product(int n) { return n == 15 ? 118.00 : 125.62; }

// 2^e mod p, balanced
__host__ __device__ constexpr int pow2_mod(int e, int p) {
  int r = 1;
  for (int k = 0; k < e; k++) r = r * 2 % p;
  return r > p / 2 ? r - p : r;
}

typedef unsigned __int128 u128;

template <int NMOD>
struct Crt {
  uint32_t w[NMOD][3];        // round(2^96 frac(y_i / p_i)), low word first
  uint64_t phat;              // top 64 bits of P, P = phat 2^pexp
  int pexp;
  // k-th 16-bit limb of weight i, 0 beyond the moduli
  __host__ __device__ constexpr uint32_t limb(int i, int k) const {
    return i < NMOD ? (w[i < NMOD ? i : 0][k >> 1] >> (16 * (k & 1))) & 0xffffu : 0u;
  }
};

template <int NMOD>
constexpr Crt<NMOD> make_crt() {
  Crt<NMOD> c{};
  u128 P = 1;
  for (int i = 0; i < NMOD; i++) P *= (u128)modulus(i);
  for (int i = 0; i < NMOD; i++) {
    const int p = modulus(i);
    int q = 1;                                   // P / p mod p
    for (int j = 0; j < NMOD; j++)
      if (j != i) q = q * (modulus(j) % p) % p;
    int y = 0;
    for (int v = 1; v < p; v++)
      if (q * v % p == 1) y = v;
    const u128 f = ((((u128)y) << 96) + (u128)(p / 2)) / (u128)p;
    for (int k = 0; k < 3; k++) c.w[i][k] = (uint32_t)(f >> (32 * k));
  }
  int e = 0;
  while (P >> 64) {
    P >>= 1;
    e++;
  }
  c.phat = (uint64_t)P;
  c.pexp = e;
  return c;
}

// ------------------------------------------------------------ residue planes
// exponent of a row from its maximum's bit pattern (max < 2^e), and whether the row holds
// Inf / NaN; the subnormal exponent field 0 behaves as 1 with no implicit bit
__device__ __forceinline__ int row_exponent(uint64_t mx, bool& bad) {
  const int exm = (int)(mx >> 52);
  bad = exm == 0x7ff;
  return mx == 0 ? 0 : (exm == 0 ? -1021 : exm - 1022);
}

// Residues of 8 consecutive K entries of one row: 16-byte stores at out + cb, one per
// modulus.  N = round(|x| 2^(t - e)) (below 2^57) is cut into four 15-bit limbs, held as
// exact FP32 integers with the entry's sign; limb sums weighted by 2^(15 j) mod p stay below
// 2^24, so three FFMA give an exact v = N mod p, and v - p round(v / p) is in [-128, 128]:
// six FP32 instructions per entry and modulus.  A BF16 value of such an integer is the
// upper half of its FP32 encoding.  The kernels are bound by the planes' writes (2 NMOD B
// per entry against 8 read).
template <int NMOD>
__device__ __forceinline__ void residues8_store(const uint64_t (&bits8)[8], int t_minus_e, bool bad,
                                                uint16_t* __restrict__ out, int64_t plane_stride,
                                                int cb) {
  float l[8][4];
#pragma unroll
  for (int q = 0; q < 8; q++) {
    const uint64_t bits = bad ? 0ull : bits8[q];
    const int ex = (int)((bits >> 52) & 0x7ff);
    uint64_t N = bits & 0xfffffffffffffull;
    if (ex) N |= 1ull << 52;
    const int sh = (ex ? ex : 1) - 1075 + t_minus_e;    // x = N 2^(max(ex, 1) - 1075)
    if (sh >= 0) N <<= sh;                              // sh <= t - 53 <= 4
    else N = sh <= -54 ? 0 : ((N >> (-sh - 1)) + 1) >> 1;
    const uint32_t sgn = (uint32_t)(bits >> 32) & 0x80000000u;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const uint32_t u = (uint32_t)(N >> (15 * j)) & 0x7fffu;
      const float f = __uint_as_float(0x4B000000u | u) - 8388608.0f;
      l[q][j] = __uint_as_float(__float_as_uint(f) ^ sgn);
    }
  }
#pragma unroll
  for (int i = 0; i < NMOD; i++) {
    const int p = modulus(i);
    const float c1 = (float)pow2_mod(15, p), c2 = (float)pow2_mod(30, p),
                c3 = (float)pow2_mod(45, p);
    const float inv = 1.0f / (float)p;
    uint32_t fb[8];
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const float v = fmaf(l[q][3], c3, fmaf(l[q][2], c2, fmaf(l[q][1], c1, l[q][0])));
      const float n = fmaf(v, inv, 12582912.0f) - 12582912.0f;
      fb[q] = __float_as_uint(fmaf(-(float)p, n, v));
    }
    *reinterpret_cast<uint4*>(out + i * plane_stride + cb) =
        make_uint4(__byte_perm(fb[0], fb[1], 0x7632), __byte_perm(fb[2], fb[3], 0x7632),
                   __byte_perm(fb[4], fb[5], 0x7632), __byte_perm(fb[6], fb[7], 0x7632));
  }
}

// Residue planes: block (strip, K chunk, batch) writes NMOD BF16 planes of its 32 x kch
// part (zeros in the padding up to ldk); the chunk-0 blocks write the row exponents.
// S[(z NMOD + i) rows_out + r][ldk] (K-major), E[z rows_out + r].  Each 32 x 64 tile goes
// through a double-buffered shared tile (one barrier per tile); thread (rr, part) then
// turns 8 consecutive K entries of row rr into 16-byte stores, one per plane.
template <int NMOD>
__global__ void __launch_bounds__(256, 2) oz_residues(SliceSrc src, int rows_out, int k_out, int ldk,
                                                   int kch, int tbits,
                                                   const unsigned long long* __restrict__ mxa,
                                                   uint16_t* __restrict__ S, int* __restrict__ E) {
  chain_begin();
  __shared__ uint64_t tile[2][SL_ROWS][65];
  const int r0 = blockIdx.x * SL_ROWS, kc0 = blockIdx.y * kch, z = blockIdx.z;
  const int t = threadIdx.x, rr = t >> 3, part = t & 7;
  const bool rowfast = src.sr == 1;
  const int r = r0 + rr;
  bool bad = false;
  const int e = r < rows_out ? row_exponent(mxa[(int64_t)z * rows_out + r], bad) : 0;
  if (blockIdx.y == 0 && part == 0 && r < rows_out) E[(int64_t)z * rows_out + r] = bad ? E_BAD : e;
  const int64_t plane_stride = (int64_t)rows_out * ldk;
  uint16_t* out = S + ((int64_t)z * NMOD * rows_out + r) * ldk;
  const int c1 = min(kc0 + kch, ldk);
  uint64_t v[8];
  if (kc0 < c1) fetch_tile(src, z, r0, kc0, rows_out, k_out, v);
  int buf = 0;
  for (int c0 = kc0; c0 < c1; c0 += 64, buf ^= 1) {
#pragma unroll
    for (int q = 0; q < 8; q++) {
      int lr, lc;
      tile_pos(rowfast, t + 256 * q, lr, lc);
      tile[buf][lr][lc] = v[q];
    }
    __syncthreads();
    if (c0 + 64 < c1) fetch_tile(src, z, r0, c0 + 64, rows_out, k_out, v);
    const int cb = c0 + part * 8;
    if (r < rows_out && cb < ldk) {
      uint64_t bits8[8];
#pragma unroll
      for (int q = 0; q < 8; q++) bits8[q] = tile[buf][rr][part * 8 + q];
      residues8_store<NMOD>(bits8, tbits - e, bad, out, plane_stride, cb);
    }
  }
}

// Residues of a K-contiguous operand: thread (rr, part) of a block owns row r0 + rr and, per
// 64-column tile, the 8 entries from part * 8, by 16-byte (V = 2) or 8-byte loads.
template <int NMOD, int V>
__global__ void __launch_bounds__(256, 2) oz_residues_kfast(const double* __restrict__ p, int64_t ld,
                                                       int64_t bstride, int rows_out, int k_out,
                                                       int ldk, int kch, int tbits,
                                                       const unsigned long long* __restrict__ mxa,
                                                       uint16_t* __restrict__ S,
                                                       int* __restrict__ E) {
  chain_begin();
  const int r0 = blockIdx.x * SL_ROWS, kc0 = blockIdx.y * kch, z = blockIdx.z;
  const int t = threadIdx.x, rr = t >> 3, part = t & 7;
  const int r = r0 + rr;
  if (r >= rows_out) return;
  bool bad;
  const int e = row_exponent(mxa[(int64_t)z * rows_out + r], bad);
  if (blockIdx.y == 0 && part == 0) E[(int64_t)z * rows_out + r] = bad ? E_BAD : e;
  const int64_t plane_stride = (int64_t)rows_out * ldk;
  uint16_t* out = S + ((int64_t)z * NMOD * rows_out + r) * ldk;
  const double* b = p + (int64_t)z * bstride + (int64_t)r * ld;
  const int c1 = min(kc0 + kch, ldk);
  for (int cb = kc0 + part * 8; cb < c1; cb += 64) {
    uint64_t bits8[8];
#pragma unroll
    for (int u = 0; u < 8; u += V) {
      const int cc = cb + u;
      if constexpr (V == 2) {
        const ulonglong2 v = cc < k_out ? __ldg(reinterpret_cast<const ulonglong2*>(b + cc))
                                        : make_ulonglong2(0, 0);
        bits8[u] = v.x;
        bits8[u + 1] = v.y;
      } else {
        bits8[u] = cc < k_out ? __ldg(reinterpret_cast<const unsigned long long*>(b + cc)) : 0ull;
      }
    }
    residues8_store<NMOD>(bits8, tbits - e, bad, out, plane_stride, cb);
  }
}

// Residues of a row-contiguous operand (element (r, c) at p[r + c ld]): the 32 x 64 tiles of
// the block's K chunk stream into a 3-stage shared-memory ring by 8-byte cp.async copies
// (two tiles in flight, no registers held for them), and thread (rr, part) turns 8
// consecutive K entries of row rr into one 16-byte store per plane.
template <int NMOD>
__global__ void __launch_bounds__(256, 2) oz_residues_rowfast(const double* __restrict__ p, int64_t ld,
                                                         int64_t bstride, int rows_out,
                                                         int k_out, int ldk, int kch, int tbits,
                                                         const unsigned long long* __restrict__ mxa,
                                                         uint16_t* __restrict__ S,
                                                         int* __restrict__ E) {
  chain_begin();
  extern __shared__ __align__(16) uint64_t dr_smem[];
  auto tile = [&](int st, int lr, int lc) -> uint64_t& {
    return dr_smem[((size_t)st * SL_ROWS + lr) * 65 + lc];
  };
  const int r0 = blockIdx.x * SL_ROWS, kc0 = blockIdx.y * kch, z = blockIdx.z;
  const int t = threadIdx.x, rr = t >> 3, part = t & 7;
  const int r = r0 + rr;
  bool bad = false;
  const int e = r < rows_out ? row_exponent(mxa[(int64_t)z * rows_out + r], bad) : 0;
  if (blockIdx.y == 0 && part == 0 && r < rows_out) E[(int64_t)z * rows_out + r] = bad ? E_BAD : e;
  const int64_t plane_stride = (int64_t)rows_out * ldk;
  uint16_t* out = S + ((int64_t)z * NMOD * rows_out + r) * ldk;
  const double* b = p + (int64_t)z * bstride;
  const int c1 = min(kc0 + kch, ldk);
  const int ntile = (c1 - kc0 + 63) / 64;
  // tile j of the chunk into stage j % DR_STAGES: lanes run along rows (contiguous)
  auto issue = [&](int j) {
    if (j < ntile) {
      const int c0 = kc0 + 64 * j, st = j % DR_STAGES;
#pragma unroll
      for (int q = 0; q < 8; q++) {
        const int e2 = t + 256 * q, lr = e2 & 31, lc = e2 >> 5;
        const int rg = r0 + lr, cg = c0 + lc;
        if (rg < rows_out && cg < k_out)
          cp_async8(&tile(st, lr, lc), b + rg + (int64_t)cg * ld);
        else
          tile(st, lr, lc) = 0ull;
      }
    }
    cp_async_commit();                      // one group per tile slot (empty past the end)
  };
  issue(0);
  issue(1);
  for (int j = 0; j < ntile; j++) {
    issue(j + 2);
    cp_async_wait<2>();                     // this thread's copies of tile j have landed
    __syncthreads();                        // and every thread's
    const int cb = kc0 + 64 * j + part * 8;
    if (r < rows_out && cb < c1) {
      uint64_t bits8[8];
#pragma unroll
      for (int q = 0; q < 8; q++) bits8[q] = tile(j % DR_STAGES, rr, part * 8 + q);
      residues8_store<NMOD>(bits8, tbits - e, bad, out, plane_stride, cb);
    }
    __syncthreads();                        // stage j % 3 is refilled by issue(j + 3)
  }
}

// ------------------------------------------------------------ GEMM kernel
struct OzEpi {
  uint8_t* res;         // residues [modulus][unit][64 column groups][256 rows][4 columns]
  int M, N;
  int* err;
};

// tile unit -> (mt2, nt, z): groups of GH tile rows, column by column inside a group, so the
// clusters running at the same time share the residue planes of few A row blocks and few B
// column blocks in L2
__host__ __device__ inline void oz_tile(int u, int tiles_m2, int tiles_n, int& mt2, int& nt,
                                        int& z) {
  const int per = tiles_m2 * tiles_n;
  z = u / per;
  const int r = u - z * per;
  const int g = r / (GH * tiles_n);
  const int rows = min(GH, tiles_m2 - g * GH);
  const int idx = r - g * GH * tiles_n;
  mt2 = g * GH + idx % rows;
  nt = idx / rows;
}
// the place u of tile (mt2, nt, z) in that order
__device__ __forceinline__ int oz_tile_index(int mt2, int nt, int z, int tiles_m2, int tiles_n) {
  const int g = mt2 / GH, rows = min(GH, tiles_m2 - g * GH);
  return (z * tiles_m2 + g * GH) * tiles_n + nt * rows + (mt2 - g * GH);
}

// chunk ch of nch equal chunks of the nk K slices (nch = ceil(nk / KCHUNK), so every chunk
// is at most KCHUNK long and none is a short tail)
__device__ __forceinline__ int chunk_edge(int nk, int nch, int ch) {
  return (int)((int64_t)nk * ch / nch);
}

// v - p round(v / p) of an integer-valued |v| <= 2^24; |result| <= 130 (the quotient's
// rounding can be off by 2^-6)
__device__ __forceinline__ float mod_balanced(float v, float p, float inv) {
  const float n = fmaf(v, inv, 12582912.0f) - 12582912.0f;
  return fmaf(-p, n, v);
}

// Persistent over work items (modulus, tile unit), modulus-major: the clusters that run at
// one time read ONE modulus's planes (at D = 2048, w = 5: 75 MB for GEMM 1, which stay in
// L2).  Cluster c of two CTAs takes items c, c + ncl..  Each K chunk accumulates in one of
// two TMEM buffers; the epilogue warps (two per 32 tile rows, 128 columns each) reduce it
// modulo p while the next chunk or item is multiplied, keep the chunk sums as packed 16-bit
// integers, and store one byte per entry at the end.
__global__ void __launch_bounds__(NTHR, 1)
    oz_gemm_pair(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB,
                 int K, int tiles_m2, int tiles_n, int batch, int nmod, OzEpi ep) {
  constexpr int A_BYTES = BM * 128, B_BYTES = 128 * 128;
  constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  constexpr int TMEM_COLS = 256;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
  uint64_t* acc_full = bars + 2 * STAGES;
  uint64_t* acc_empty = bars + 2 * STAGES + 2;
  uint64_t* drainb = bars + 2 * STAGES + 4;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 5);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const uint32_t rank = cluster_rank();
  const bool lead = rank == 0;
  const int cl = blockIdx.x >> 1, ncl = gridDim.x >> 1;
  const int nk = (K + KELEMS - 1) / KELEMS;
  const int nch = (nk + KCHUNK - 1) / KCHUNK;
  const int units = tiles_m2 * tiles_n * batch;
  const int num_items = units * nmod;
  auto stageA = [&](int s) { return smem + s * STAGE_BYTES; };
  auto stageB = [&](int s) { return stageA(s) + A_BYTES; };

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; s++) {
      mbar_init(smem_u32(&bars[s]), 1);
      mbar_init(smem_u32(&bars[STAGES + s]), 1);
    }
    for (int b = 0; b < 2; b++) {
      mbar_init(smem_u32(&acc_full[b]), 1);
      mbar_init(smem_u32(&acc_empty[b]), 2 * EPI_WARPS);
    }
    mbar_init(smem_u32(drainb), 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&mapA)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&mapB)) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(2 * TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  chain_begin();

  if (warp == 0) {
    if (lane == 0) {
      int it = 0, last = -1;
      bool stop = false;
      for (int item = cl; item < num_items && !stop && !*abort_flag; item += ncl) {
        const int i = item / units, u = item - i * units;
        int mt2, nt, z;
        oz_tile(u, tiles_m2, tiles_n, mt2, nt, z);
        const int m0 = min(mt2 * 2 * BM + (int)rank * BM, ep.M - 1);
        const int n0 = min(nt * TILE + (int)rank * 128, ep.N - 1);
        const int zp = z * nmod + i;
        for (int kb = 0; kb < nk; kb++, it++) {
          const int s = it % STAGES;
          const uint32_t ph = (it / STAGES) & 1;
          if (!mbar_wait(smem_u32(&bars[STAGES + s]), ph ^ 1, abort_flag, ep.err)) {
            stop = true;
            break;
          }
          const uint32_t full = smem_u32(&bars[s]);
          if (lead) mbar_expect_tx(full, 2 * STAGE_BYTES);
          const uint32_t full_lead = cluster_addr(full, 0);
          const int kc = kb * KELEMS;
          tma_load_3d_pair(smem_u32(stageA(s)), &mapA, full_lead, kc, m0, zp);
          tma_load_3d_pair(smem_u32(stageB(s)), &mapB, full_lead, kc, n0, zp);
          last = it;
        }
      }
      if (*abort_flag && last >= 0) {
        const unsigned long long t0 = globaltimer();
        if (lead) {
          for (int j = max(0, last - STAGES + 1); j <= last; j++) {
            const uint32_t bar = smem_u32(&bars[j % STAGES]);
            while (!mbar_try(bar, (j / STAGES) & 1) && globaltimer() - t0 < WAIT_NS) {
            }
          }
        } else {
          while (globaltimer() - t0 < 1000000ull) {
          }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && lead) {
      constexpr uint32_t idesc = make_idesc(BF16, 2 * BM, TILE);
      int it = 0, local = 0;
      bool stop = false;
      for (int item = cl; item < num_items && !stop && !*abort_flag; item += ncl) {
        for (int ch = 0; ch < nch && !stop; ch++, local++) {
          const int kb0 = chunk_edge(nk, nch, ch), kb1 = chunk_edge(nk, nch, ch + 1);
          const int buf = local & 1;
          const uint32_t use = (uint32_t)(local >> 1);
          if (!mbar_wait(smem_u32(&acc_empty[buf]), (use & 1) ^ 1, abort_flag, ep.err)) {
            stop = true;
            break;
          }
          tc_fence_after();
          const uint32_t tacc = tmem + buf * TMEM_COLS;
          for (int kb = kb0; kb < kb1; kb++, it++) {
            const int s = it % STAGES;
            const uint32_t ph = (it / STAGES) & 1;
            if (!mbar_wait(smem_u32(&bars[s]), ph, abort_flag, ep.err)) {
              stop = true;
              break;
            }
            tc_fence_after();
            const uint32_t a0 = smem_u32(stageA(s)), b0 = smem_u32(stageB(s));
#pragma unroll
            for (int ks = 0; ks < 4; ks++)
              mma_pair<BF16>(tacc, smem_desc(a0 + ks * 32), smem_desc(b0 + ks * 32), idesc,
                             (kb > kb0 || ks > 0) ? 1u : 0u);
            mma_commit_pair(smem_u32(&bars[STAGES + s]), 3);
          }
          if (!stop) mma_commit_pair(smem_u32(&acc_full[buf]), 3);
        }
      }
    }
  } else {
    const int q = warp & 3;                  // the TMEM lanes (tile rows) this warp may read
    const int half = (warp - 2) >> 2;        // its 128 columns
    const int rloc = (int)rank * BM + 32 * q + lane;
    int local = 0;
    bool stop = false;
    for (int item = cl; item < num_items && !stop; item += ncl) {
      const int i = item / units;
      const float p = (float)modulus(i), inv = 1.0f / p;
      uint32_t acc[64];                      // column pairs' chunk sums, each + 256 per chunk
      uint8_t* out = ep.res + ((int64_t)item * 64 + 32 * half) * (TILE * 4) + rloc * 4;
      for (int ch = 0; ch < nch; ch++, local++) {
        const int buf = local & 1;
        const uint32_t use = (uint32_t)(local >> 1);
        const bool ok = mbar_wait(smem_u32(&acc_full[buf]), use & 1, abort_flag, ep.err);
        if (!ok || *abort_flag) {
          stop = true;
          break;
        }
        tc_fence_after();
        const uint32_t tbase =
            tmem + buf * TMEM_COLS + 128 * half + ((uint32_t)(32 * q) << 16);
#pragma unroll
        for (int c0 = 0; c0 < 128; c0 += 32) {
          uint32_t r[32];
          tmem_ld32_async(tbase + c0, r);
          tmem_wait_ld(r);
#pragma unroll
          for (int j = 0; j < 32; j += 2) {
            // r + 256 >= 0 in the low mantissa bits of 2^23 + 256 + r
            const uint32_t a = __float_as_uint(
                mod_balanced(__uint_as_float(r[j]), p, inv) + 8388864.0f);
            const uint32_t b = __float_as_uint(
                mod_balanced(__uint_as_float(r[j + 1]), p, inv) + 8388864.0f);
            const uint32_t ab = __byte_perm(a, b, 0x5410);
            acc[(c0 + j) / 2] = ch == 0 ? ab : acc[(c0 + j) / 2] + ab;
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(cluster_addr(smem_u32(&acc_empty[buf]), 0));
      }
      if (stop) break;
      // total mod p in [0, 255]: the bias is taken out, a negative remainder lifted by p
      const float bias = 8388608.0f + 256.0f * (float)nch;
#pragma unroll
      for (int g = 0; g < 32; g++) {
        uint32_t by[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const uint32_t lohi = __byte_perm(acc[2 * g + (j >> 1)], 0x4B00u, (j & 1) ? 0x5432 : 0x5410);
          const float v = mod_balanced(__uint_as_float(lohi) - bias, p, inv);
          by[j] = __float_as_uint((v < 0.0f ? v + p : v) + 8388608.0f);
        }
        *reinterpret_cast<uint32_t*>(out + (int64_t)g * (TILE * 4)) =
            __byte_perm(__byte_perm(by[0], by[1], 0x0040), __byte_perm(by[2], by[3], 0x0040),
                        0x5410);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1 && lead) {
    tc_fence_after();
    if (lane == 0) {
      mma_commit_pair(smem_u32(drainb), 1);
      const unsigned long long t0 = globaltimer();
      while (!mbar_try(smem_u32(drainb), 0) && globaltimer() - t0 < WAIT_NS) {
      }
    }
    __syncwarp();
  }
  cluster_sync();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(2 * TMEM_COLS)
                 : "memory");
  }
}

// ------------------------------------------------------------ Chinese remainder
struct CrtArgs {
  const uint8_t* res;
  double* C;
  int64_t ldc, strideC, planeC;
  int M, N, mh;         // rows >= mh of the real embedding go to the imaginary plane
  int units, tiles_m2, tiles_n;
  const int* ea;        // [batch][M] row exponents
  const int* eb;        // [batch][N] column exponents
  int tbits;
  double alpha[2], beta[2];
  int m, cplx;
  int mt0;              // first row of tiles of this launch
  unsigned long long* zero[2];   // row maxima that the call has used, to be zeroed
  int64_t nzero[2];
};

// The sums of the residues times the six 16-bit limbs of the weights, two moduli per instruction
// (dp2a): 48 instructions per value where 32-bit words take 16 multiply-adds and 32 wide ones
// at half their rate.  The integer pipes bound this kernel (151 instructions per value, 194
// before; D = 1024, 15 moduli: 158 -> 119 us, 74 at the copy bandwidth).  Four columns at a
// time, so that a weight is put into a register once for four values.  c[j][q]: residues of
// moduli 4 q .. 4 q + 3 in column j.
template <int NMOD>
__device__ __forceinline__ void crt_limbs(const uint32_t (&c)[4][4], uint32_t (&L)[4][6]) {
  constexpr Crt<NMOD> T = make_crt<NMOD>();
#pragma unroll
  for (int j = 0; j < 4; j++)
#pragma unroll
    for (int k = 0; k < 6; k++) L[j][k] = 0u;     // below 16 * 255 * 2^16 in the end
#pragma unroll
  for (int i = 0; i < MAXMOD; i += 2)
#pragma unroll
    for (int k = 0; k < 6; k++) {
      const uint32_t w = T.limb(i, k) | (T.limb(i + 1, k) << 16);
#pragma unroll
      for (int j = 0; j < 4; j++)
        L[j][k] = (i & 2) ? __dp2a_hi(w, c[j][i / 4], L[j][k]) : __dp2a_lo(w, c[j][i / 4], L[j][k]);
    }
}

// The cases that crt_value leaves out: X = 0 or below 2^-33 P, results outside the range of
// normal numbers, rows or columns that hold Inf / NaN (exponents from E_BAD on).  |S| in words.
__device__ __noinline__ double crt_rare(uint32_t s0, uint32_t s1, uint32_t s2, uint32_t sgn, int E,
                                        uint64_t phat, int pexp) {
  if (E >= E_BAD / 2) return __longlong_as_double(0x7ff8000000000000ll);
  int n = 0;
  for (int k = 0; k < 2 && s2 == 0u; k++) { s2 = s1; s1 = s0; s0 = 0u; n += 32; }
  if (s2 == 0u) return 0.0;
  const int lz = __clz(s2);
  const uint64_t hi =
      ((uint64_t)__funnelshift_l(s1, s2, lz) << 32) | __funnelshift_l(s0, s1, lz);
  const uint64_t m = __umul64hi(hi, phat);
  const int top = (int)(m >> 63);
  const double v = ldexp((double)(((m >> (9 + top)) + 1) >> 1), E + pexp - n - lz + top + 10);
  return sgn ? -v : v;
}

// The FP64 value of the limb sums L, scaled by 2^E.  S = sum c_i w_i mod 2^96 is X / P as a
// signed 96-bit fraction (error below 2^-85, and exactly 0 for X = 0), and X 2^E is rounded
// once, to 53 bits.  One branch: what is rare is left to crt_rare.
template <int NMOD>
__device__ __forceinline__ double crt_value(const uint32_t (&L)[6], int E) {
  constexpr Crt<NMOD> T = make_crt<NMOD>();
  const uint64_t a = ((uint64_t)L[1] << 16) + L[0], b = ((uint64_t)L[3] << 16) + L[2];
  const uint64_t a1 = (a >> 32) + (uint32_t)b;
  uint32_t s0 = (uint32_t)a, s1 = (uint32_t)a1;
  uint32_t s2 = (L[5] << 16) + L[4] + (uint32_t)(b >> 32) + (uint32_t)(a1 >> 32);
  const uint32_t sgn = s2 & 0x80000000u, neg = (uint32_t)((int32_t)s2 >> 31);
  // |S|: the complement plus one if negative
  asm("{\n\t"
      "xor.b32 %0, %0, %3;\n\txor.b32 %1, %1, %3;\n\txor.b32 %2, %2, %3;\n\t"
      "sub.cc.u32 %0, %0, %3;\n\tsubc.cc.u32 %1, %1, %3;\n\tsubc.u32 %2, %2, %3;\n\t}"
      : "+r"(s0), "+r"(s1), "+r"(s2)
      : "r"(neg));
  // the top 64 bits, normalised: |S| = hi 2^(32 - lz)
  const int lz = __clz(s2);
  const uint64_t hi =
      ((uint64_t)__funnelshift_l(s1, s2, lz) << 32) | __funnelshift_l(s0, s1, lz);
  // |X| = hi 2^(32 - lz) 2^-96 phat 2^pexp = m 2^(pexp - lz), m = high half of hi phat, whose
  // top bit is bit 63 or 62
  const uint64_t m = __umul64hi(hi, T.phat);
  const int top = (int)(m >> 63);
  // 53 bits and the rounding carry, which may run on into the exponent
  const uint64_t mant = ((m >> (9 + top)) + 1) >> 1;
  const int be1 = E + (T.pexp + 10 + 52 + 1022) - lz + top;      // biased exponent less 1
  if (s2 == 0u || (uint32_t)be1 > 2045u) return crt_rare(s0, s1, s2, sgn, E, T.phat, T.pexp);
  return __hiloint2double((int)(((uint32_t)(mant >> 32) + ((uint32_t)be1 << 20)) | sgn),
                          (int)(uint32_t)mant);
}

// Thread = one tile row of a 4-column group: one 4-byte load per modulus (a warp reads 128
// contiguous bytes), 4 outputs (a warp writes 256 contiguous bytes per column).  Four columns
// rather than sixteen keep the loaded residues in 16 registers, so that enough warps are
// resident to hide the loads behind the integer work of the others; the grid's axes are the
// tile's coordinates, so that a thread needs no division.  GENERAL applies alpha / beta in FP64.
template <int NMOD, bool GENERAL>
__global__ void __launch_bounds__(256, 5) oz_crt(CrtArgs a) {
  chain_begin();
  const int mt2 = a.mt0 + blockIdx.y, z = blockIdx.z;
  for (int q = 0; q < 2; q++) {
    const int64_t t = ((int64_t)z * a.tiles_m2 + mt2) * (gridDim.x * 256LL) + blockIdx.x * 256 +
                      threadIdx.x;
    if (t < a.nzero[q]) a.zero[q][t] = 0ull;
  }
  const int row = mt2 * TILE + threadIdx.x, col0 = blockIdx.x * 4;
  if (row >= a.M) return;
  // 4-column groups of all tiles in the tile order, 1 KB per modulus each
  const int64_t grp = (int64_t)oz_tile_index(mt2, blockIdx.x >> 6, z, a.tiles_m2, a.tiles_n) * 64 +
                      (blockIdx.x & 63);
  const uint8_t* base = a.res + (grp * TILE + threadIdx.x) * 4;
  const int64_t mstep = (int64_t)a.units * (TILE * TILE);
  uint32_t v[MAXMOD];
#pragma unroll
  for (int i = 0; i < MAXMOD; i++)
    v[i] = i < NMOD ? __ldcs(reinterpret_cast<const uint32_t*>(base + i * mstep)) : 0u;
  const int e0 = __ldg(a.ea + (int64_t)z * a.M + row) - 2 * a.tbits;
  const int* eb = a.eb + (int64_t)z * a.N + col0;
  const bool im = row >= a.mh;
  double* p = a.C + (int64_t)z * a.strideC + (im ? a.planeC + row - a.mh : (int64_t)row) +
              (int64_t)col0 * a.ldc;
  // bytes by column: c[j][q] holds the residues of moduli 4 q .. 4 q + 3 in column j
  uint32_t c[4][4], L[4][6];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const uint32_t* x = v + 4 * q;
    const uint32_t a0 = __byte_perm(x[0], x[1], 0x5140), a1 = __byte_perm(x[0], x[1], 0x7362);
    const uint32_t b0 = __byte_perm(x[2], x[3], 0x5140), b1 = __byte_perm(x[2], x[3], 0x7362);
    c[0][q] = __byte_perm(a0, b0, 0x5410);
    c[1][q] = __byte_perm(a0, b0, 0x7632);
    c[2][q] = __byte_perm(a1, b1, 0x5410);
    c[3][q] = __byte_perm(a1, b1, 0x7632);
  }
  crt_limbs<NMOD>(c, L);
#pragma unroll
  for (int j = 0; j < 4; j++, p += a.ldc) {
    if (col0 + j >= a.N) break;
    double x = crt_value<NMOD>(L[j], e0 + __ldg(eb + j));
    if (GENERAL) {
      x *= a.alpha[0];
      if (a.beta[0] != 0.0) x += a.beta[0] * *p;
    }
    *p = x;
  }
}

// C = alpha T + beta C of a complex product T (split planes, ld m) with general alpha, beta
__global__ void oz_axpby_cplx(int m, int64_t n, const double* __restrict__ T, int64_t planeT,
                              CrtArgs a, int batch) {
  chain_begin();
  const int64_t mn = (int64_t)m * n, total = mn * batch;
  const bool has_beta = a.beta[0] != 0.0 || a.beta[1] != 0.0;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t z = t / mn, rem = t - z * mn;
    const double sr = T[2 * z * planeT + rem], si = T[(2 * z + 1) * planeT + rem];
    double* C = a.C + z * a.strideC + rem % m + (rem / m) * a.ldc;
    double re = a.alpha[0] * sr - a.alpha[1] * si, im = a.alpha[0] * si + a.alpha[1] * sr;
    if (has_beta) {
      const double cr = C[0], ci = C[a.planeC];
      re += a.beta[0] * cr - a.beta[1] * ci;
      im += a.beta[0] * ci + a.beta[1] * cr;
    }
    C[0] = re;
    C[a.planeC] = im;
  }
}

// ------------------------------------------------------------ host side
constexpr int SMEM = STAGES * (BM * 128 + 128 * 128) + 1024 + 256;
static_assert(SMEM <= 227 * 1024, "shared memory");

// moduli and bits per operand entry for inner extent K: K 2^(2 t) < P / 2 with t >= 53
struct Plan {
  int nmod = MAXMOD, tbits = 53;
};
static Plan oz_plan(int64_t K) {
  const double lk = std::log2((double)std::max<int64_t>(K, 2));
  Plan p;
  p.tbits = (int)std::floor((log2_product(15) - 1.0 - lk) / 2.0);
  if (p.tbits >= 53) {
    p.nmod = 15;
  } else {
    p.nmod = 16;
    p.tbits = (int)std::floor((log2_product(16) - 1.0 - lk) / 2.0);
  }
  p.tbits = std::min(p.tbits, 57);
  return p;
}

}  // namespace oz

// estimated device seconds of the residue GEMM on `cl` resident clusters
static double oz_seconds(int64_t M2, int64_t N, int64_t K2, int batch, int cl) {
  using namespace oz;
  const Plan p = oz_plan(std::min<int64_t>(K2, KMAX));
  const int64_t tiles = ((M2 + TILE - 1) / TILE) * ((N + TILE - 1) / TILE) * batch;
  const int64_t rounds = (tiles * p.nmod + cl - 1) / cl;
  const double kpad = (double)((K2 + KELEMS - 1) / KELEMS * KELEMS);
  // a pair tile of one modulus: 256 x 256 x K on two SMs at ~1.75 PFLOP/s / 76 pairs, at
  // least the epilogue of one tile
  const double item = std::max(2.0 * TILE * TILE * kpad / (1.75e15 / 76.0), 1.2e-6);
  double t = rounds * item;
  // planes: FP64 read twice, 2 B per entry and modulus written; bytes and FP64 per output
  t += (double)(M2 + N) * K2 * batch * (16.0 + 2.0 * p.nmod) / 4e12;
  t += (double)tiles * TILE * TILE * (2.0 * p.nmod + 8.0) / 4e12;
  return t + 20e-6;                                     // launches
}

int gemm_f64_ozaki_possible(fmpt_handle* h, const GemmArgs& g) {
  if (!h->f64_tc && !g.engine) return 0;
  if (g.m < 32 || g.n < 32 || g.k < 16) return 0;
  const int cp = g.cplx ? 2 : 1;
  const double flops = 2.0 * g.m * g.n * (double)g.k * g.batch * cp * cp;
  const double t_simt = flops / 1.1e12;
  return oz_seconds((int64_t)g.m * cp, g.n, (int64_t)g.k * cp, g.batch,
                    std::max(1, h->sm_count / 2)) < t_simt
             ? 1
             : 0;
}

bool gemm_f64_ozaki_takes_maxima(fmpt_handle* h, const GemmArgs& g) {
  return !h->oz_digits && g.batch == 1 && (int64_t)g.k * (g.cplx ? 2 : 1) <= oz::KMAX &&
         gemm_f64_ozaki_possible(h, g);
}

namespace oz {
// kernels by modulus count
typedef void (*ResGeneric)(SliceSrc, int, int, int, int, int, const unsigned long long*, uint16_t*, int*);
typedef void (*ResFast)(const double*, int64_t, int64_t, int, int, int, int, int,
                        const unsigned long long*, uint16_t*, int*);
static ResGeneric residues_kernel(int nmod) {
  return nmod == 15 ? oz_residues<15> : oz_residues<16>;
}
static ResFast residues_rowfast_kernel(int nmod) {
  return nmod == 15 ? oz_residues_rowfast<15> : oz_residues_rowfast<16>;
}
static ResFast residues_kfast_kernel(int nmod, bool two) {
  if (two) return nmod == 15 ? oz_residues_kfast<15, 2> : oz_residues_kfast<16, 2>;
  return nmod == 15 ? oz_residues_kfast<15, 1> : oz_residues_kfast<16, 1>;
}
}  // namespace oz

int gemm_f64_ozaki(fmpt_handle* h, const GemmArgs& g) {
  using namespace oz;
  const int cp = g.cplx ? 1 : 0;
  if ((int64_t)g.k * (cp ? 2 : 1) > KMAX) {
    // K beyond one launch's chunk sums: K ranges accumulated through beta = 1
    const int half = (g.k / 2 + 7) / 8 * 8;
    GemmArgs lo = g, hi = g;
    lo.k = half;
    hi.k = g.k - half;
    hi.A += (g.ta == FMPT_N || g.ta == FMPT_R) ? (int64_t)half * g.lda : (int64_t)half;
    hi.B += (g.tb == FMPT_N || g.tb == FMPT_R) ? (int64_t)half : (int64_t)half * g.ldb;
    hi.beta[0] = 1.0;
    hi.beta[1] = 0.0;
    lo.cacheA = lo.cacheB = hi.cacheA = hi.cacheB = nullptr;
    lo.maxA = hi.maxA = nullptr;           // they are those of the whole K
    FMPT_TRY(gemm_f64_ozaki(h, lo));
    return gemm_f64_ozaki(h, hi);
  }
  const int M2 = g.m * (cp ? 2 : 1), K2 = g.k * (cp ? 2 : 1), N = g.n;
  const int ldk = (K2 + 7) / 8 * 8;
  const int batch = g.batch;
  const Plan plan = oz_plan(K2);
  const int nmod = plan.nmod;
  if ((int64_t)batch * nmod > INT32_MAX / 2) return set_error(h, FMPT_ERR_SHAPE, "ozaki: batch");
  // workspace: residue planes of A and B, exponents, row maxima, then the product's residues
  const size_t planesA = (size_t)batch * nmod * M2 * ldk * 2, planesB = (size_t)batch * nmod * N * ldk * 2;
  const size_t expA = (size_t)batch * M2 * 4, expB = (size_t)batch * N * 4;
  auto al = [](size_t b) { return (b + 255) / 256 * 256; };
  const int tiles_m2 = (M2 + TILE - 1) / TILE, tiles_n = (N + TILE - 1) / TILE;
  const int64_t units = (int64_t)tiles_m2 * tiles_n * batch;
  if (units > INT32_MAX / 128) return set_error(h, FMPT_ERR_SHAPE, "ozaki: too many tiles");
  // resident clusters of the kernel
  static PerDevice<> resident;
  int clusters = 0;
  cudaLaunchConfig_t cfg{};
  cfg.blockDim = dim3(NTHR);
  cfg.dynamicSmemBytes = SMEM;
  cfg.stream = h->stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  FMPT_TRY(resident.get(h, 0, clusters, [&](int& found) -> int {
    for (int n : {15, 16})
      FMPT_CUDA(h, cudaFuncSetAttribute(residues_rowfast_kernel(n),
                                        cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DR_SMEM));
    FMPT_CUDA(h, cudaFuncSetAttribute(oz_gemm_pair, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
    cfg.gridDim = dim3(2 * std::max(1, h->sm_count / 2));
    if (cudaOccupancyMaxActiveClusters(&found, oz_gemm_pair, &cfg) != cudaSuccess) {
      (void)cudaGetLastError();
      found = 0;
    }
    return FMPT_OK;
  }));
  if (clusters <= 0) return set_error(h, FMPT_ERR_UNSUPPORTED, "ozaki: no 2-CTA cluster fits");
  const size_t resb = (size_t)nmod * units * TILE * TILE;
  const size_t mxb = (size_t)batch * (M2 + N) * sizeof(uint64_t);
  // a complex product with a complex alpha or beta, or with an old C, goes through a copy
  const bool via_copy = cp && (g.alpha[1] != 0.0 || g.beta[0] != 0.0 || g.beta[1] != 0.0);
  const size_t copyb = via_copy ? (size_t)batch * 2 * g.m * N * sizeof(double) : 0;
  // an operand with a cache keeps its planes there (built once while its key holds)
  const int64_t keyA[8] = {M2, K2, ldk, g.ta, cp, batch, g.lda, g.strideA};
  const int64_t keyB[8] = {N, K2, ldk, g.tb, cp, batch, g.ldb, g.strideB};
  const bool hitA = oz_cache_hit(g.cacheA, g.A, keyA), hitB = oz_cache_hit(g.cacheB, g.B, keyB);
  const bool inA = g.cacheA != nullptr, inB = g.cacheB != nullptr;
  const size_t need = (inA ? 0 : al(planesA) + al(expA)) + (inB ? 0 : al(planesB) + al(expB)) +
                      al(resb) + copyb;
  FMPT_TRY(grow_buffer(h, &h->oz_ws, &h->oz_ws_bytes, need));
  if (h->oz_mx_bytes < mxb) h->oz_mx_dirty = true;
  FMPT_TRY(grow_buffer(h, &h->oz_mx, &h->oz_mx_bytes, al(mxb)));
  bool clean = true;                       // zero again once this call's kernels have run
  if (h->oz_mx_dirty) {
    FMPT_CUDA(h, cudaMemsetAsync(h->oz_mx, 0, h->oz_mx_bytes, h->stream));
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    clean = cudaStreamIsCapturing(h->stream, &cs) == cudaSuccess && cs == cudaStreamCaptureStatusNone;
  }
  h->oz_mx_dirty = true;
  for (int side = 0; side < 2; side++) {
    OzCache* c = side == 0 ? g.cacheA : g.cacheB;
    if (!c || (side == 0 ? hitA : hitB)) continue;
    const size_t want = side == 0 ? al(planesA) + al(expA) : al(planesB) + al(expB);
    c->valid = false;
    FMPT_TRY(grow_buffer(h, &c->buf, &c->bytes, want));
  }
  char* base = static_cast<char*>(h->oz_ws);
  char* pa = inA ? static_cast<char*>(g.cacheA->buf) : base;
  if (!inA) base += al(planesA) + al(expA);
  char* pb = inB ? static_cast<char*>(g.cacheB->buf) : base;
  if (!inB) base += al(planesB) + al(expB);
  uint16_t* SA = reinterpret_cast<uint16_t*>(pa);
  int* EA = reinterpret_cast<int*>(pa + al(planesA));
  uint16_t* SBp = reinterpret_cast<uint16_t*>(pb);
  int* EB = reinterpret_cast<int*>(pb + al(planesB));
  unsigned long long* MX = static_cast<unsigned long long*>(h->oz_mx);
  uint8_t* RES = reinterpret_cast<uint8_t*>(base);
  double* COPY = reinterpret_cast<double*>(base + al(resb));

  const SliceSrc sa = oz_side_a(g), sb = oz_side_b(g);
  if (!hitA || !hitB) {
    ProfScope prof(h, FMPT_K_CONVERT);
    auto convert = [&](const SliceSrc& x, int rows, unsigned long long* mx, uint16_t* planes,
                       int* ex) -> int {
      // K columns per block: 512 where that leaves four blocks per SM, else down to one
      // 64-column tile (a 1024 x 256 operand on 32 blocks took 12 us, its FP64 data 0.3)
      const int strips = (rows + SL_ROWS - 1) / SL_ROWS;
      int kch = SL_KCH;
      while (kch > 64 && (int64_t)strips * ((ldk + kch - 1) / kch) * batch < 4LL * h->sm_count)
        kch /= 2;
      const dim3 grid(strips, (ldk + kch - 1) / kch, batch);
      if (mx != g.maxA) FMPT_TRY(oz_row_maxima(h, x, rows, K2, batch, mx));
      if (oz_kfast(x))
        FMPT_CUDA(h, launch_chain(residues_kfast_kernel(nmod, oz_aligned(x, x.sr, K2)), grid, 256, 0,
                                  h->stream, x.p, x.sr, x.bstride, rows, K2, ldk, kch, plan.tbits,
                                  mx, planes, ex));
      else if (x.sr == 1 && !x.cplx)
        FMPT_CUDA(h, launch_chain(residues_rowfast_kernel(nmod), grid, 256, DR_SMEM, h->stream, x.p, x.sc, x.bstride, rows, K2, ldk, kch, plan.tbits, mx, planes, ex));
      else
        FMPT_CUDA(h, launch_chain(residues_kernel(nmod), grid, 256, 0, h->stream, x, rows, K2, ldk, kch, plan.tbits, mx,
                                                           planes, ex));
      FMPT_LAUNCHED(h);
      return FMPT_OK;
    };
    if (!hitA) FMPT_TRY(convert(sa, M2, g.maxA ? g.maxA : MX, SA, EA));
    if (!hitB) FMPT_TRY(convert(sb, N, MX + (size_t)batch * M2, SBp, EB));
  }
  for (int side = 0; side < 2; side++) {
    OzCache* c = side == 0 ? g.cacheA : g.cacheB;
    if (!c || (side == 0 ? hitA : hitB)) continue;
    c->src = side == 0 ? g.A : g.B;
    for (int i = 0; i < 8; i++) c->key[i] = side == 0 ? keyA[i] : keyB[i];
    c->valid = true;
  }
  CUtensorMap ma, mb;
  FMPT_TRY(make_map(h, &ma, SA, BF16, K2, M2, ldk, (int64_t)batch * nmod, (int64_t)M2 * ldk, BM));
  FMPT_TRY(make_map(h, &mb, SBp, BF16, K2, N, ldk, (int64_t)batch * nmod, (int64_t)N * ldk, 128));

  OzEpi ep{};
  ep.M = M2;
  ep.N = N;
  ep.res = RES;
  FMPT_TRY(gp_status_word(h, &ep.err));
  cfg.gridDim = dim3((unsigned)(2 * std::min<int64_t>(units * nmod, clusters)));
  {
    ProfScope prof(h, FMPT_K_TC_GEMM);
    chain_attr(attr[1]);
    cfg.numAttrs = 2;
    FMPT_CUDA(h, cudaLaunchKernelEx(&cfg, oz_gemm_pair, ma, mb, K2, tiles_m2, tiles_n, batch, nmod,
                                    ep));
    FMPT_LAUNCHED(h);
  }
  CrtArgs ca{};
  ca.res = RES;
  ca.M = M2;
  ca.N = N;
  ca.mh = cp ? g.m : INT32_MAX;
  ca.units = (int)units;
  ca.tiles_m2 = tiles_m2;
  ca.tiles_n = tiles_n;
  ca.ea = EA;
  ca.eb = EB;
  ca.tbits = plan.tbits;
  if (via_copy) {
    ca.C = COPY;
    ca.ldc = g.m;
    ca.planeC = (int64_t)g.m * N;
    ca.strideC = 2 * ca.planeC;
    ca.alpha[0] = 1.0;
  } else {
    ca.C = g.C;
    ca.ldc = g.ldc;
    ca.strideC = g.strideC;
    ca.planeC = g.planeC;
    ca.alpha[0] = g.alpha[0];
    ca.beta[0] = g.beta[0];
  }
  const bool general = ca.alpha[0] != 1.0 || ca.beta[0] != 0.0;
  ProfScope prof(h, FMPT_K_CONVERT);
  ca.zero[0] = MX;
  ca.nzero[0] = (int64_t)batch * (M2 + N);
  ca.zero[1] = g.maxA;
  ca.nzero[1] = g.maxA ? M2 : 0;
  for (ca.mt0 = 0; ca.mt0 < tiles_m2; ca.mt0 += 65535) {
    const dim3 blocks((unsigned)((N + 3) / 4), (unsigned)std::min(65535, tiles_m2 - ca.mt0),
                      (unsigned)batch);
    if (nmod == 15) {
      if (general) FMPT_CUDA(h, launch_chain(oz_crt<15, true>, blocks, 256, 0, h->stream, ca));
      else FMPT_CUDA(h, launch_chain(oz_crt<15, false>, blocks, 256, 0, h->stream, ca));
    } else {
      if (general) FMPT_CUDA(h, launch_chain(oz_crt<16, true>, blocks, 256, 0, h->stream, ca));
      else FMPT_CUDA(h, launch_chain(oz_crt<16, false>, blocks, 256, 0, h->stream, ca));
    }
    FMPT_LAUNCHED(h);
  }
  if (clean) h->oz_mx_dirty = false;
  if (g.maxA && g.maxA_clean) *g.maxA_clean = true;
  if (via_copy) {
    CrtArgs cc = ca;
    cc.C = g.C;
    cc.ldc = g.ldc;
    cc.strideC = g.strideC;
    cc.planeC = g.planeC;
    for (int i = 0; i < 2; i++) {
      cc.alpha[i] = g.alpha[i];
      cc.beta[i] = g.beta[i];
    }
    const int64_t total = (int64_t)g.m * N * batch;
    const int nb = (int)std::max<int64_t>(1, std::min<int64_t>((total + 255) / 256, 8LL * h->sm_count));
    FMPT_CUDA(h, launch_chain(oz_axpby_cplx, nb, 256, 0, h->stream, g.m, N, COPY, ca.planeC, cc, batch));
    FMPT_LAUNCHED(h);
  }
  return FMPT_OK;
}

void oz_cache_free(fmpt_handle* h, OzCache& c) {
  if (c.buf) cudaFreeAsync(c.buf, h->stream);
  c.buf = nullptr;
  c.bytes = 0;
  c.valid = false;
  c.src = nullptr;
}

}  // namespace fmpt
