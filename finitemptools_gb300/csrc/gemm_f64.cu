// Plain FP64 (and split-plane complex FP64) GEMM on the CUDA cores.
//
// GB300's FP64 rate is small: a warp's FMA occupies its SM sub-partition for 64 to
// 77 cycles, dependent or not, so these kernels are FP64-pipe bound for every shape
// that matters, and what decides their speed is how evenly they spread the
// multiply-adds over the 608 sub-partitions.  Large problems use a 64x64 tile with a
// 4x4 register block per thread (gemm_kernel).  Small ones (the D <= 128
// contractions of TDVP and of the first DMRG bonds) give every warp an 8x4 tile and a
// cp.async ring of its own (gemm_warp) and may split K over the grid.  Every split writes its
// partial product to a workspace; the last split of a tile to finish (an atomic
// count per tile) sums the tile's partials in split order, so the result does
// not depend on scheduling, applies alpha/beta and resets the count.  Where no
// count is available (a stream capture before the counts exist) a second kernel
// does the same sum.
#include "internal.h"

namespace fmpt {
namespace {

constexpr int BK = 8, NT = 256;

// op(X)(r, c) with trans code: 0 N, 1 T, 2 C, 3 R(conj, no transpose)
__device__ __forceinline__ int64_t a_index(int t, int r, int c, int64_t ld) {
  return (t == 0 || t == 3) ? (int64_t)r + (int64_t)c * ld : (int64_t)c + (int64_t)r * ld;
}

// C (or the split workspace) = op(A) op(B) over k in [k_lo, k_hi).
// gridDim.z = batch * splits; with splits > 1 (batch == 1) the raw partial
// product goes to ws + split * plane_ws (re, then im plane at + m*n).
template <bool CPLX>
__global__ void __launch_bounds__(NT) gemm_kernel(GemmArgs g, int splits, int kchunk,
                                                  double* __restrict__ ws,
                                                  int* __restrict__ tile_cnt) {
  if (gate_closed(g.gate)) return;
  chain_begin();
  constexpr int BMN = 64;                      // tile edge
  constexpr int TPR = BMN / 16;                // outputs per thread along each dimension
  __shared__ double As[2][BK][BMN + 1];
  __shared__ double Bs[2][BK][BMN + 1];
  const int tid = threadIdx.x;
  const int tx = tid % 16, ty = tid / 16;
  const int m0 = blockIdx.x * BMN, n0 = blockIdx.y * BMN;
  const int zb = blockIdx.z / splits, sp = blockIdx.z % splits;
  const int k_lo = sp * kchunk;
  const int k_hi = min(g.k, k_lo + kchunk);
  const double* A = g.A + zb * g.strideA;
  const double* B = g.B + zb * g.strideB;
  const bool conjA = (g.ta == 2 || g.ta == 3);
  const bool conjB = (g.tb == 2 || g.tb == 3);
  const bool a_mfast = (g.ta == 0 || g.ta == 3);   // op(A) rows contiguous
  const bool b_kfast = (g.tb == 0 || g.tb == 3);   // op(B) rows (k) contiguous

  double acc[TPR][TPR], acci[TPR][TPR];
#pragma unroll
  for (int i = 0; i < TPR; i++)
#pragma unroll
    for (int j = 0; j < TPR; j++) { acc[i][j] = 0.0; acci[i][j] = 0.0; }

  // The K slab k0 .. k0 + BK of A and B goes global -> registers -> shared memory; the
  // next slab's loads are issued before the current one is multiplied, so that their
  // latency overlaps the FMAs (a small GEMM runs one block per SM and has nothing else to
  // hide it behind).  The products are summed in the same order as without it.
  constexpr int NE = (BMN * BK + NT - 1) / NT;       // slab elements per thread and operand
  double ra[NE][2], rb[NE][2];
  auto load_slab = [&](int k0) {
#pragma unroll
    for (int q = 0; q < NE; q++) {
      const int e = tid + q * NT;
      ra[q][0] = ra[q][1] = rb[q][0] = rb[q][1] = 0.0;
      if (e >= BMN * BK) continue;
      int mm, kk;
      if (a_mfast) { mm = e % BMN; kk = e / BMN; } else { kk = e % BK; mm = e / BK; }
      int gm = m0 + mm, gk = k0 + kk;
      if (gm < g.m && gk < k_hi) {
        const int64_t idx = a_index(g.ta, gm, gk, g.lda);
        ra[q][0] = __ldg(A + idx);
        if (CPLX) { ra[q][1] = __ldg(A + g.planeA + idx); if (conjA) ra[q][1] = -ra[q][1]; }
      }
      int nn;
      if (b_kfast) { kk = e % BK; nn = e / BK; } else { nn = e % BMN; kk = e / BMN; }
      const int gn = n0 + nn;
      gk = k0 + kk;
      if (gn < g.n && gk < k_hi) {
        const int64_t idx = a_index(g.tb, gk, gn, g.ldb);
        rb[q][0] = __ldg(B + idx);
        if (CPLX) { rb[q][1] = __ldg(B + g.planeB + idx); if (conjB) rb[q][1] = -rb[q][1]; }
      }
    }
  };
  auto store_slab = [&]() {
#pragma unroll
    for (int q = 0; q < NE; q++) {
      const int e = tid + q * NT;
      if (e >= BMN * BK) continue;
      int mm, kk;
      if (a_mfast) { mm = e % BMN; kk = e / BMN; } else { kk = e % BK; mm = e / BK; }
      As[0][kk][mm] = ra[q][0];
      if (CPLX) As[1][kk][mm] = ra[q][1];
      int nn;
      if (b_kfast) { kk = e % BK; nn = e / BK; } else { nn = e % BMN; kk = e / BMN; }
      Bs[0][kk][nn] = rb[q][0];
      if (CPLX) Bs[1][kk][nn] = rb[q][1];
    }
  };
  if (k_lo < k_hi) load_slab(k_lo);
  for (int k0 = k_lo; k0 < k_hi; k0 += BK) {
    store_slab();
    __syncthreads();
    if (k0 + BK < k_hi) load_slab(k0 + BK);
#pragma unroll
    for (int kk = 0; kk < BK; kk++) {
      double a[TPR], b[TPR], ai[TPR], bi[TPR];
#pragma unroll
      for (int i = 0; i < TPR; i++) {
        a[i] = As[0][kk][tx + 16 * i];
        b[i] = Bs[0][kk][ty + 16 * i];
        if (CPLX) { ai[i] = As[1][kk][tx + 16 * i]; bi[i] = Bs[1][kk][ty + 16 * i]; }
      }
#pragma unroll
      for (int i = 0; i < TPR; i++)
#pragma unroll
        for (int j = 0; j < TPR; j++) {
          if (CPLX) {
            acc[i][j] = fma(a[i], b[j], acc[i][j]);
            acc[i][j] = fma(-ai[i], bi[j], acc[i][j]);
            acci[i][j] = fma(a[i], bi[j], acci[i][j]);
            acci[i][j] = fma(ai[i], b[j], acci[i][j]);
          } else {
            acc[i][j] = fma(a[i], b[j], acc[i][j]);
          }
        }
    }
    __syncthreads();
  }
  // ---- epilogue
  if (splits > 1) {
    const int64_t mn = (int64_t)g.m * g.n;
    double* W = ws + (int64_t)sp * mn * (CPLX ? 2 : 1);
#pragma unroll
    for (int i = 0; i < TPR; i++) {
      const int gm = m0 + tx + 16 * i;
      if (gm >= g.m) continue;
#pragma unroll
      for (int j = 0; j < TPR; j++) {
        const int gn = n0 + ty + 16 * j;
        if (gn >= g.n) continue;
        const int64_t idx = (int64_t)gm + (int64_t)gn * g.m;
        W[idx] = acc[i][j];
        if (CPLX) W[mn + idx] = acci[i][j];
      }
    }
    if (!tile_cnt) return;                 // the reduction kernel sums the splits
    // the last split of this tile to arrive sums the partials in split order
    __shared__ int s_last;
    __threadfence();
    __syncthreads();
    const int tile = (blockIdx.y * gridDim.x + blockIdx.x) + (int)(gridDim.x * gridDim.y) * zb;
    if (tid == 0) {
      const int prev = atomicAdd(tile_cnt + tile, 1);
      s_last = prev == splits - 1;
      if (s_last) tile_cnt[tile] = 0;      // ready for the next launch (stream order)
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const bool has_beta = (g.beta[0] != 0.0 || g.beta[1] != 0.0);
    double* C = g.C + zb * g.strideC;
#pragma unroll
    for (int i = 0; i < TPR; i++) {
      const int gm = m0 + tx + 16 * i;
      if (gm >= g.m) continue;
#pragma unroll
      for (int j = 0; j < TPR; j++) {
        const int gn = n0 + ty + 16 * j;
        if (gn >= g.n) continue;
        const int64_t t = (int64_t)gm + (int64_t)gn * g.m;
        double sr = 0.0, si = 0.0;
        for (int q = 0; q < splits; q++) {
          const double* Wq = ws + (int64_t)q * mn * (CPLX ? 2 : 1);
          sr += __ldcg(Wq + t);
          if (CPLX) si += __ldcg(Wq + mn + t);
        }
        const int64_t idx = (int64_t)gm + (int64_t)gn * g.ldc;
        if (CPLX) {
          double r = g.alpha[0] * sr - g.alpha[1] * si;
          double im = g.alpha[0] * si + g.alpha[1] * sr;
          if (has_beta) {
            const double cr = C[idx], ci = C[g.planeC + idx];
            r += g.beta[0] * cr - g.beta[1] * ci;
            im += g.beta[0] * ci + g.beta[1] * cr;
          }
          C[idx] = r;
          C[g.planeC + idx] = im;
        } else {
          double r = g.alpha[0] * sr;
          if (has_beta) r += g.beta[0] * C[idx];
          C[idx] = r;
        }
      }
    }
    return;
  }
  double* C = g.C + zb * g.strideC;
  const bool has_beta = (g.beta[0] != 0.0 || g.beta[1] != 0.0);
#pragma unroll
  for (int i = 0; i < TPR; i++) {
    const int gm = m0 + tx + 16 * i;
    if (gm >= g.m) continue;
#pragma unroll
    for (int j = 0; j < TPR; j++) {
      const int gn = n0 + ty + 16 * j;
      if (gn >= g.n) continue;
      const int64_t idx = (int64_t)gm + (int64_t)gn * g.ldc;
      if (CPLX) {
        double r = g.alpha[0] * acc[i][j] - g.alpha[1] * acci[i][j];
        double im = g.alpha[0] * acci[i][j] + g.alpha[1] * acc[i][j];
        if (has_beta) {
          const double cr = C[idx], ci = C[g.planeC + idx];
          r += g.beta[0] * cr - g.beta[1] * ci;
          im += g.beta[0] * ci + g.beta[1] * cr;
        }
        C[idx] = r;
        C[g.planeC + idx] = im;
      } else {
        double r = g.alpha[0] * acc[i][j];
        if (has_beta) r += g.beta[0] * C[idx];
        C[idx] = r;
      }
    }
  }
}

// Small problems: one warp per 8 x 4 tile of C (complex: one for the real and one for the
// imaginary part), one output per lane, two warps per block: the small unit of work fills
// the 608 sub-partitions evenly.  A 16x16 tile per block of eight warps left a D = 64
// contraction (320 x 256 x 64) on 3 blocks or 2 per SM, with two barriers and a load latency
// per 8-deep slab.  Here the operands stream through a ring of WST slabs of WK by cp.async
// (the whole K of a small contraction is in flight at once: one latency, not one per slab).
// Each output is the same chain of FMAs over k as in gemm_kernel.  Per contraction, D = 64:
// real 16.1 and 20.4 -> 14.6 and 17.8 us (FP64 pipe 80% busy), complex 24.2 and 22.8 ->
// 17.7 and 18.2 us.
constexpr int WM = 8, WN = 4, WWARPS = 2, WK1 = 32, WST1 = 4;

// KP > 1 (complex, Arnoldi only): KP pairs of warps take a K piece of the tile each, and the
// pieces are added in order.  At D <= 32 a tile's chain of multiply-adds is longer than
// everything else (K = 96: 192 of them, 64 cycles each) while most sub-partitions are idle.
// The sum's order differs from the other forms', so the Lanczos solve (whose eigenvector's sign
// hangs on a last bit) and the plain GEMM keep to KP = 1.  Exponential of 20 vectors: D = 16
// 689 -> 615 us, D = 22 790 -> 708, D = 32 923 -> 800, D = 8 574 -> 553; from D = 40 on the
// pieces do not fit the idle sub-partitions.
template <bool CPLX, int KP>
__global__ void __launch_bounds__(32 * WWARPS * KP) gemm_warp(GemmArgs g, int splits, int kchunk,
                                                              double* __restrict__ ws,
                                                              int* __restrict__ tile_cnt) {
  static_assert(KP == 1 || CPLX, "K pieces of complex tiles");
  if (gate_closed(g.gate)) return;
  chain_begin();
  constexpr int NP = CPLX ? 2 : 1;                       // planes
  constexpr int WK = KP > 1 ? 16 : WK1, WST = KP > 1 ? 3 : WST1;
  // the ring belongs to a warp (real) or to the two warps of a tile and piece (complex)
  constexpr int T = CPLX ? 64 : 32, RINGS = CPLX ? KP : WWARPS;
  __shared__ double As[RINGS][WST][NP][WK][WM], Bs[RINGS][WST][NP][WK][WN];
  const int lane = threadIdx.x & 31, wid = CPLX ? (threadIdx.x >> 5) & 1 : threadIdx.x >> 5;
  const int piece = CPLX ? threadIdx.x >> 6 : 0;
  const int t = threadIdx.x % T, ring = CPLX ? piece : wid;
  const int comp = CPLX ? wid : 0;                       // the part of C this warp forms
  const int mt = CPLX ? blockIdx.x : blockIdx.x * WWARPS + wid;
  const int m0 = mt * WM, n0 = blockIdx.y * WN;
  const int lm = lane & 7, ln = lane >> 3;
  const int gm = m0 + lm, gn = n0 + ln;
  const int zb = blockIdx.z / splits, sp = blockIdx.z % splits;
  const int kp = KP > 1 ? (g.k + KP - 1) / KP : 0;       // KP > 1: splits is 1
  const int k_lo = KP > 1 ? min(g.k, piece * kp) : sp * kchunk;
  const int k_hi = min(g.k, k_lo + (KP > 1 ? kp : kchunk));
  const int K = max(0, k_hi - k_lo), nslab = (K + WK - 1) / WK;
  const bool live = gm < g.m && gn < g.n;
  // This thread's elements of a slab: (mm, kk) of A, (kk, nn) of B, the first ones here and
  // the next ones a fixed step on, so that lanes run along the contiguous index.
  const bool a_mfast = g.ta == 0 || g.ta == 3, b_kfast = g.tb == 0 || g.tb == 3;
  const int amm = a_mfast ? t % WM : t / WK, akk = a_mfast ? t / WM : t % WK;
  const int adm = a_mfast ? 0 : T / WK, adk = a_mfast ? T / WM : 0;
  const int bnn = b_kfast ? t / WK : t % WN, bkk = b_kfast ? t % WK : t / WN;
  const int bdn = b_kfast ? T / WK : 0, bdk = b_kfast ? 0 : T / WN;
  const int64_t sam = a_mfast ? 1 : g.lda, sak = a_mfast ? g.lda : 1;
  const int64_t sbk = b_kfast ? 1 : g.ldb, sbn = b_kfast ? g.ldb : 1;
  const double* A = g.A + zb * g.strideA + (m0 + amm) * sam + (k_lo + akk) * sak;
  const double* B = g.B + zb * g.strideB + (n0 + bnn) * sbn + (k_lo + bkk) * sbk;
  const int64_t ai_step = adm * sam + adk * sak, bi_step = bdn * sbn + bdk * sbk;
  auto issue = [&](int j) {
    if (j < nslab) {
      const int st = j % WST, k0 = j * WK;
      const double* pa = A + k0 * sak;
      const double* pb = B + k0 * sbk;
#pragma unroll
      for (int e = 0; e < WM * WK / T; e++) {
        const int mm = amm + e * adm, kk = akk + e * adk;
        const bool in = m0 + mm < g.m && k0 + kk < K;
        const double* q = in ? pa + e * ai_step : g.A;
#pragma unroll
        for (int c = 0; c < NP; c++) cp_async8z(&As[ring][st][c][kk][mm], q + (in ? c * g.planeA : 0), in);
      }
#pragma unroll
      for (int e = 0; e < WN * WK / T; e++) {
        const int nn = bnn + e * bdn, kk = bkk + e * bdk;
        const bool in = n0 + nn < g.n && k0 + kk < K;
        const double* q = in ? pb + e * bi_step : g.B;
#pragma unroll
        for (int c = 0; c < NP; c++) cp_async8z(&Bs[ring][st][c][kk][nn], q + (in ? c * g.planeB : 0), in);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");   // one group per slab slot
  };
  auto ring_sync = [&]() {
    if (KP > 1) asm volatile("bar.sync %0, 64;" ::"r"(1 + piece) : "memory");
    else if (CPLX) __syncthreads();
    else __syncwarp();
  };
  // real part: a b - ai bi; imaginary part: a bi + ai b; conj(op) flips the sign of ai, bi
  const bool conj_a = g.ta == 2 || g.ta == 3, conj_b = g.tb == 2 || g.tb == 3;
  const uint64_t kSign = 1ull << 63;
  const uint64_t na = (conj_a != (comp == 0)) ? kSign : 0ull;    // sign of ai as used
  const uint64_t nb = conj_b ? kSign : 0ull;
  auto flip = [](double x, uint64_t m) {
    return __longlong_as_double(__double_as_longlong(x) ^ (long long)m);
  };
  double acc = 0.0;
#pragma unroll
  for (int j = 0; j < WST - 1; j++) issue(j);
  for (int j = 0; j < nslab; j++) {
    issue(j + WST - 1);
    asm volatile("cp.async.wait_group %0;" ::"n"(WST - 1) : "memory");
    ring_sync();
    const int st = j % WST, kn = min(WK, K - j * WK);
#pragma unroll 8
    for (int kk = 0; kk < kn; kk++) {
      const double a = As[ring][st][0][kk][lm], b = Bs[ring][st][0][kk][ln];
      if (CPLX) {
        const double ai = flip(As[ring][st][NP - 1][kk][lm], na);
        const double bi = flip(Bs[ring][st][NP - 1][kk][ln], nb);
        acc = fma(a, comp ? bi : b, acc);
        acc = fma(ai, comp ? b : bi, acc);
      } else {
        acc = fma(a, b, acc);
      }
    }
    if (j + WST < nslab) ring_sync();                    // stage j % WST is refilled next
  }
  double* C = g.C + zb * g.strideC;
  const int64_t idx = (int64_t)gm + (int64_t)gn * g.ldc;
  const bool has_beta = g.beta[0] != 0.0 || g.beta[1] != 0.0;
  __shared__ double part[32 * WWARPS * KP];              // complex: the other part's value
  if constexpr (KP > 1) {                                // the pieces' sums, in order
    part[threadIdx.x] = acc;
    __syncthreads();
    if (piece > 0) return;
#pragma unroll
    for (int q = 1; q < KP; q++) acc += part[64 * q + threadIdx.x];
    if (g.alpha[0] == 1.0 && g.alpha[1] == 0.0 && !has_beta) {
      if (live) C[comp * g.planeC + idx] = acc;
      return;
    }
    asm volatile("bar.sync 1, 64;" ::: "memory");        // part is written again
  }
  if (KP == 1 && splits > 1) {
    const int64_t mn = (int64_t)g.m * g.n, t = (int64_t)gm + (int64_t)gn * g.m;
    if (live) ws[(int64_t)sp * mn * (CPLX ? 2 : 1) + comp * mn + t] = acc;
    if (!tile_cnt) return;                               // the reduction kernel sums the splits
    // the last split of this tile to arrive sums the partials in split order
    __shared__ int s_last[WWARPS];
    const int tiles_x = CPLX ? gridDim.x : gridDim.x * WWARPS;
    if (CPLX) __syncthreads(); else __syncwarp();        // both parts are written
    if (CPLX ? threadIdx.x == 0 : lane == 0) {
      __threadfence();
      int* cnt = tile_cnt + ((int64_t)zb * gridDim.y + blockIdx.y) * tiles_x + mt;
      const bool last = atomicAdd(cnt, 1) == splits - 1;
      if (last) *cnt = 0;                                // ready for the next launch
      __threadfence();
      s_last[wid] = last;
    }
    if (CPLX) __syncthreads(); else __syncwarp();
    if (!s_last[CPLX ? 0 : wid]) return;
    acc = 0.0;
    if (live)
      for (int q = 0; q < splits; q++) acc += __ldcg(ws + (int64_t)q * mn * (CPLX ? 2 : 1) + comp * mn + t);
  }
  if (CPLX) {
    if (g.alpha[0] != 1.0 || g.alpha[1] != 0.0 || has_beta) {
      part[threadIdx.x] = acc;
      if (KP > 1) asm volatile("bar.sync 1, 64;" ::: "memory"); else __syncthreads();
      const double sr = part[lane], si = part[32 + lane];
      double r = comp ? g.alpha[0] * si + g.alpha[1] * sr : g.alpha[0] * sr - g.alpha[1] * si;
      if (has_beta && live) {
        const double cr = C[idx], ci = C[g.planeC + idx];
        r += comp ? g.beta[0] * ci + g.beta[1] * cr : g.beta[0] * cr - g.beta[1] * ci;
      }
      if (KP > 1) asm volatile("bar.sync 1, 64;" ::: "memory"); else __syncthreads();   // both have read the old C
      acc = r;
    }
    if (live) C[comp * g.planeC + idx] = acc;
  } else if (live) {
    double r = g.alpha[0] * acc;
    if (has_beta) r += g.beta[0] * C[idx];
    C[idx] = r;
  }
}

// C = alpha * sum_{s < splits} W_s + beta * C, summed in split order
template <bool CPLX>
__global__ void split_reduce(GemmArgs g, int splits, const double* __restrict__ ws) {
  if (g.gate && *g.gate) return;
  const int64_t mn = (int64_t)g.m * g.n;
  const bool has_beta = (g.beta[0] != 0.0 || g.beta[1] != 0.0);
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < mn;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int gm = (int)(t % g.m), gn = (int)(t / g.m);
    double sr = 0.0, si = 0.0;
    for (int s = 0; s < splits; s++) {
      const double* W = ws + (int64_t)s * mn * (CPLX ? 2 : 1);
      sr += W[t];
      if (CPLX) si += W[mn + t];
    }
    const int64_t idx = (int64_t)gm + (int64_t)gn * g.ldc;
    if (CPLX) {
      double r = g.alpha[0] * sr - g.alpha[1] * si;
      double im = g.alpha[0] * si + g.alpha[1] * sr;
      if (has_beta) {
        const double cr = g.C[idx], ci = g.C[g.planeC + idx];
        r += g.beta[0] * cr - g.beta[1] * ci;
        im += g.beta[0] * ci + g.beta[1] * cr;
      }
      g.C[idx] = r;
      g.C[g.planeC + idx] = im;
    } else {
      double r = g.alpha[0] * sr;
      if (has_beta) r += g.beta[0] * g.C[idx];
      g.C[idx] = r;
    }
  }
}

// Per-tile split counters (zeroed once, left zero by every launch): enough for any grid
// the cost model below may choose with a split.
constexpr int kMaxSplitTiles = 1 << 14;

template <bool CPLX>
int launch(fmpt_handle* h, const GemmArgs& g) {
  const int sms = h->sm_count > 0 ? h->sm_count : 1;
  // The K split: the one that, in square tiles of the best of three edges, puts the fewest
  // multiply-adds on the busiest SM; a split adds the partials' round trip, priced as that many
  // multiply-adds.  It is a rule about the order of the sums, not a model of the kernel below: the
  // 32 and 16 wide tiles it was made for have become warp tiles, and a Lanczos vector's sign
  // hangs on the last bit of the sums, so it stays as it was.
  const double cm = CPLX ? 4.0 : 1.0;
  int splits = 1;
  double best = 1e300;
  for (int e : {64, 32, 16}) {
    const int64_t t = (int64_t)((g.m + e - 1) / e) * ((g.n + e - 1) / e) * g.batch;
    for (int s = 1; s <= 64; s *= 2) {
      if (s > 1 && (g.batch != 1 || g.nosplit || g.k < 4 * BK || g.k / s < 2 * BK)) break;
      const int kc = s > 1 ? ((g.k + s - 1) / s + BK - 1) / BK * BK : g.k;
      const int64_t blocks = t * ((g.k + kc - 1) / kc);
      const int64_t per_sm = (blocks + sms - 1) / sms;
      double cost = (double)per_sm * e * e * kc * cm;
      if (s > 1) cost += 2.0e4 * cm + (double)s * e * e * cm * 4.0;
      if (e == 16) cost *= 1.15;               // (more loads per FMA)
      if (cost < best * 0.98) {
        best = cost;
        splits = s;
      }
    }
  }
  int kchunk = splits > 1 ? ((g.k + splits - 1) / splits + BK - 1) / BK * BK : g.k;
  if (splits > 1) splits = (g.k + kchunk - 1) / kchunk;
  const size_t wsb = (size_t)splits * g.m * g.n * sizeof(double) * (CPLX ? 2 : 1);
  if (splits > 1 && h->gemm_ws_bytes < wsb) {
    // the workspace cannot grow inside a stream capture: K stays whole
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(h->stream, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) {
      cudaGetLastError();
      splits = 1;
      kchunk = g.k;
    }
  }
  // The kernel: 8x4 tiles per warp where they put fewer multiply-adds on the busiest
  // sub-partition than 64x64 tiles do on the busiest SM, those otherwise.  The split stays
  // as it is, so the sums do not depend on this choice; the warps' operand reads come to
  // 1.5 TB/s whatever the shape.
  const int64_t wx = (g.m + WM - 1) / WM, wy = (g.n + WN - 1) / WN;
  const int64_t warps = wx * wy * g.batch * splits * (CPLX ? 2 : 1);
  const double cost_warp = (double)((warps + 4 * sms - 1) / (4 * sms)) * 4.0 * WM * WN * kchunk *
                           (CPLX ? 2.0 : 1.0);
  const int64_t tiles64 = (int64_t)((g.m + 63) / 64) * ((g.n + 63) / 64) * g.batch * splits;
  const double cost64 = (double)((tiles64 + sms - 1) / sms) * 4096.0 * kchunk * cm;
  const bool warp_tiles = wy <= 65535 && cost_warp < 0.95 * cost64;
  dim3 grid((g.m + 63) / 64, (g.n + 63) / 64, g.batch * splits);
  if (warp_tiles)
    grid = dim3((unsigned)(CPLX ? wx : (wx + WWARPS - 1) / WWARPS), (unsigned)wy, g.batch * splits);
  if (grid.y > 65535 || grid.z > 65535)
    return set_error(h, FMPT_ERR_SHAPE, "gemm: grid too large (%d x %d x %d)", grid.x, grid.y,
                     grid.z);
  // the split partials live in the handle's workspace (reused in stream order)
  double* ws = nullptr;
  int* cnt = nullptr;
  if (splits > 1) {
    FMPT_TRY(grow_buffer(h, &h->gemm_ws, &h->gemm_ws_bytes, wsb));
    ws = static_cast<double*>(h->gemm_ws);
    const int64_t tiles = (int64_t)grid.x * (warp_tiles && !CPLX ? WWARPS : 1) * grid.y * g.batch;
    if (tiles <= kMaxSplitTiles) {
      cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
      if (!h->gemm_cnt && cudaStreamIsCapturing(h->stream, &cs) == cudaSuccess &&
          cs == cudaStreamCaptureStatusNone) {
        // created outside a stream capture only; inside one the reduction kernel runs
        FMPT_TRY(grow_buffer(h, &h->gemm_cnt, &h->gemm_cnt_bytes, kMaxSplitTiles * sizeof(int)));
        FMPT_CUDA(h, cudaMemsetAsync(h->gemm_cnt, 0, kMaxSplitTiles * sizeof(int), h->stream));
      }
      cudaGetLastError();
      cnt = static_cast<int*>(h->gemm_cnt);
    }
  }
  ProfScope prof(h, FMPT_K_F64_GEMM);
  // four K pieces per tile while the sub-partitions (four per SM) have room for them all
  constexpr int KP = CPLX ? 4 : 1;
  if (CPLX && warp_tiles && h->k_pieces && splits == 1 && g.k >= 16 && warps * KP <= 4LL * sms)
    FMPT_CUDA(h, launch_chain(gemm_warp<CPLX, KP>, grid, 32 * WWARPS * KP, 0, h->stream, g, splits,
                              kchunk, ws, cnt));
  else if (warp_tiles)
    FMPT_CUDA(h, launch_chain(gemm_warp<CPLX, 1>, grid, 32 * WWARPS, 0, h->stream, g, splits, kchunk,
                              ws, cnt));
  else
    FMPT_CUDA(h, launch_chain(gemm_kernel<CPLX>, grid, NT, 0, h->stream, g, splits, kchunk, ws,
                              cnt));
  FMPT_LAUNCHED(h);
  if (splits > 1 && !cnt) {
    const int64_t mn = (int64_t)g.m * g.n;
    const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((mn + 255) / 256, 4LL * sms));
    split_reduce<CPLX><<<blocks, 256, 0, h->stream>>>(g, splits, ws);
    FMPT_LAUNCHED(h);
  }
  return FMPT_OK;
}

}  // namespace

int gemm_f64(fmpt_handle* h, const GemmArgs& g) {
  if (g.m < 0 || g.n < 0 || g.k < 0 || g.batch < 1)
    return set_error(h, FMPT_ERR_SHAPE, "gemm: negative extent");
  if (g.m == 0 || g.n == 0) return FMPT_OK;
  if (g.k == 0 && g.beta[0] == 1.0 && g.beta[1] == 0.0) return FMPT_OK;
  if (g.k > 0 && !g.nosplit &&
      (h->oz_digits ? gemm_f64_digits_possible(h, g) : gemm_f64_ozaki_possible(h, g))) {
    const int st = h->oz_digits ? gemm_f64_digits(h, g) : gemm_f64_ozaki(h, g);
    // FMPT_ERR_UNSUPPORTED: nothing launched (no cluster fits, or its workspace would have
    // to grow inside a stream capture); the CUDA-core kernel runs instead
    if (st != FMPT_ERR_UNSUPPORTED) return st;
  }
  GemmArgs gated = g;
  gated.gate = h->gate;
  return g.cplx ? launch<true>(h, gated) : launch<false>(h, gated);
}

}  // namespace fmpt
