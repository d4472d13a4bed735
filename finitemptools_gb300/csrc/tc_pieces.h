// Work items of the pair GEMM (tc_gemm.cu) and the walk of an epilogue warp over them.  Plain C++
// apart from the function qualifier, so that the walk also compiles for the host.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define FMPT_PIECES_FN __device__ __forceinline__
#else
#define FMPT_PIECES_FN inline
#endif

namespace fmpt {
namespace tc {

// Work items of the pair kernel: `full` whole tiles (units) and, when the last round of tiles
// would leave clusters idle, the `tail` units after them, each cut into S pieces along K.  The
// pieces are the first tail S items: their sums, a round trip through L2, then lie beside the
// whole tiles' products instead of behind the last round (H_eff*x at D = 512: BF16 47.0 -> 42.2
// us, TF32 57.0 -> 51.2, 3xTF32 90.8 -> 78.7; D = 1200: 149 -> 135, 230 -> 215, 517 -> 500; a
// part of it because the counters no longer take a memset per GEMM).  Piece p sums K-slices
// [p nk / S, (p+1) nk / S) and writes its FP32 partial tile to ws; the last piece of a
// tile to finish (per CTA half and epilogue warp, counted in cnt) adds the S partials in
// piece order and stores the tile, so the result does not depend on which piece ends last.
struct PairSched {
  int full, tail, S;
  float* ws;          // [tail * S][256 columns][256 rows]
  int* cnt;           // [tail][2 CTAs][4 warps], zero at launch, reset by the last piece
};

FMPT_PIECES_FN void pair_item(const PairSched& sp, int item, int nk, int& u,
                                          int& kb0, int& kb1, int& t) {
  const int pieces = sp.tail * sp.S;
  if (item >= pieces) {
    u = item - pieces;
    kb0 = 0;
    kb1 = nk;
    t = -1;
  } else {
    t = item;
    const int p = t % sp.S;
    u = sp.full + t / sp.S;
    kb0 = (int)((int64_t)p * nk / sp.S);
    kb1 = (int)((int64_t)(p + 1) * nk / sp.S);
  }
}

// The items of cluster cl of ncl in order, for one epilogue warp.  ready(local) waits for the
// accumulator of its local-th item and says whether it came; drain(local, u, t) stores it;
// count(ut) counts a piece of split tile ut and says whether it was the last; sum(ut, u) adds the
// pieces; reset(ut) zeroes the count.  A warp that has given up waiting leaves its results out
// (the launch's error flag is set) but still counts every piece, so that the counts are zero
// again when the launch ends, whatever happened in it: they serve every later launch of the
// handle, which does not look at this one's flag.
template <class Ready, class Drain, class Count, class Sum, class Reset>
FMPT_PIECES_FN void pair_epilogue(const PairSched& sp, int cl, int ncl, int nk, Ready ready,
                                  Drain drain, Count count, Sum sum, Reset reset) {
  const int num_items = sp.full + sp.tail * sp.S;
  bool live = true;
  int local = 0;
  for (int item = cl; item < num_items; item += ncl, local++) {
    int u, kb0, kb1, t;
    pair_item(sp, item, nk, u, kb0, kb1, t);
    if (live) live = ready(local);
    if (live) drain(local, u, t);
    if (t < 0 || !count(u - sp.full)) continue;
    if (live) sum(u - sp.full, u);
    reset(u - sp.full);
  }
}

}  // namespace tc
}  // namespace fmpt
