// gemm_plan.cuh -- which of the tensor-core GEMMs runs a product, in which shape, and its launch.  The engine and the
// single-kernel entry points go through the same two functions, so that a test of a product runs what a decode runs.
#pragma once
#include <cstring>

#include "gemm_tc.cuh"
#include "gemm_tc_pair.cuh"
#include "gemm_tc_rows.cuh"

namespace linmt {
namespace tc {

// What the caller's device and buffers allow.
struct GemmLimits {
  int n_sm = 148;
  int parts = 1;          // products that run side by side, each shaped for its share of the SMs (encoder wavefront)
  size_t ws_floats = 0;   // split-K workspace and its tile counters, of this product alone
  int max_tiles = 0;
  bool beside = false;    // few rows: the next product's CTAs are to find room beside this one's
  bool rows = true, pair = true, persist = true;    // kernel forms that may be used (tests switch them off)
};

enum class GemmKernel { kTile, kRows, kPair, kPersist, kPersistPair };
struct GemmPlan {
  GemmKernel kernel = GemmKernel::kTile;
  Shape sh{};                // every kernel but kRows
  RowsShape rs{};            // kRows
  int bk = 64;               // depth of a tensor map's box, and the rows of A's and of W's
  int a_box = BM, b_box = 0;
  int stat_tile = 0, stat_part = 0;   // block statistics of a row: four blocks of `part` columns per tile of `tile` (0: none)
  bool on_pairs() const { return kernel == GemmKernel::kPair || kernel == GemmKernel::kPersistPair; }
};

// C[M][N] = A[M][K] . W[N][K]^T on `nt` planes of format `fmt`.  drain: k-blocks of 32 between drains of the leading
// accumulator (0: the default; K / 32 and more: one chain).  a_row0: the product's first row in A's tensor map.
template <class Epi>
inline GemmPlan plan_gemm(int M, int N, int K, int nt, int fmt, int drain, int a_row0, const GemmLimits& lim) {
  GemmPlan p;
  // Few rows: the weight-streaming kernel (gemm_tc_rows.cuh), where the rows are the narrow side of the MMA.  Its gain
  // shrinks as the rows fill the 128-row tile (gate product, us against the one-tile kernel: 8.7 / 13.8 at 12
  // rows, 10.2 / 14.8 at 32, 11.4 / 15.8 at 64; bf16 6.3 / 13.0 at 12, 9.0 / 13.0 at 64); a product of many column
  // tiles and one k slice is finished by too few warps for more than 48 rows of the f16 pair (one plane, vocabulary with
  // block statistics in the decode: 12.7 us at 12 rows, 18.9 at 64 against 19.6 in the one-tile kernel).
  if (lim.rows && lim.parts == 1 && M <= kRowsMax && (nt == 1 || M <= 48 || N <= 128 * lim.n_sm) &&
      make_shape_rows(M, N, K, nt, fmt, lim.n_sm, drain >= K / 32, lim.beside, &p.rs)) {
    p.kernel = GemmKernel::kRows;
    p.a_box = p.rs.rp; p.b_box = BM;
    if (Epi::kHasPmax) { p.stat_tile = BM; p.stat_part = 32; }
    return p;
  }
  // The encoder runs its L layers as a wavefront on L streams: a GEMM sized for the whole machine would only
  // queue behind its neighbours, so there each one is shaped for its share of the SMs and they run side by side.
  const int sm_budget = lim.parts > 1 ? (lim.n_sm / lim.parts > 0 ? lim.n_sm / lim.parts : 1) : lim.n_sm;
  int bn = 0, splits = 1;
  pick_shape(M, N, K, nt, sm_budget, lim.ws_floats, lim.max_tiles, &bn, &splits, fmt);
  // one plane (bf16 precision): 64-deep stages with 128-byte rows halve the per-k-block overheads
  // (measured 1.5x on the gate GEMMs); with split operands only 32-deep stages leave room for a ring
  // the f16 pair: 64-deep stages as well, except for a weight matrix far larger than L2 under
  // the widest tiles, where only two such stages fit and four 32-deep ones hide DRAM latency better
  // (vocabulary GEMM: 143 us against 149 us)
  p.bk = nt == 1 ? 64 : 32;
  if (fmt == 1 && nt == 2 && K % 64 == 0) p.bk = (bn >= 240 && (size_t)N * K * 4 > ((size_t)96 << 20)) ? 32 : 64;
  const int mt = (M + BM - 1) / BM;
  // (a row offset is for the few-rows kernel and the one-tile kernel: the encoder's positions, a single row tile where the
  // former declines them, and its input parts of eight positions, up to eight row tiles shaped for a share of the SMs)
  const bool alone = lim.parts == 1 && a_row0 == 0;
  const bool whole_k = splits == 1 && p.bk == 64;
  // The many-wave one-plane logits GEMM has a persistent pair form (measured at K = 1024, against one tile per CTA:
  // N = 30016 23.6 / 29.5 us at 256 rows, 51 / 57 at 640, 55 / 71 at 768; N = 80000 104 / 124 at 512; three row tiles, a
  // quarter of the pair idle, are equal), with 208-wide tiles.
  const bool one_plane_logits = nt == 1 && Epi::kHasPmax;   // the fp32-output GEMMs: vocabulary projection
  // (the block statistics depend on the tile width, so the width is the pair's whether or not pairs may run)
  bool ppair = false;
  if (one_plane_logits && whole_k && mt >= 2 && alone && (long)mt * ((N + bn - 1) / bn) > lim.n_sm &&
      (long)((mt + 1) / 2) * ((N + 207) / 208) > lim.n_sm / 2) {
    ppair = lim.pair && lim.persist;
    bn = 208;
  }
  // ... and the gate product of one plane, where one tile per CTA is more than one wave (beyond 1024 rows; measured at N =
  // 4096, K = 2048: 22.4 / 28.3 us at 1280 rows, 25.7 / 30.6 at 1536): rounds of 3.9 + 0.0215 * width us, and a prologue
  // and last epilogue of 4 + 0.033 * width.
  if (Epi::kHasBlock && !Epi::kHasPmax && lim.pair && lim.persist && nt == 1 && whole_k && mt > 8 && alone) {
    double best = 1e30;
    for (int w = 96; w <= 256; w += 16) {
      const long t = (long)((mt + 1) / 2) * ((N + w - 1) / w), rounds = (t + lim.n_sm / 2 - 1) / (lim.n_sm / 2);
      const double cost = 4.0 + 0.033 * w + rounds * (3.9 + 0.0215 * w) * K / 2048.0;
      if (cost < best) { best = cost; bn = w; }
    }
    ppair = true;
  }
  const long ntile_cols = (N + bn - 1) / bn;
  // block statistics: four column blocks per tile; not from the split-K fix-up path
  if (Epi::kHasPmax && splits == 1) { p.stat_tile = bn; p.stat_part = ((bn >> 4) + 3) / 4 * 16; }
  // CTA pairs (gemm_tc_pair.cuh) where the one-tile shape has room for two stages only: an even number of row
  // tiles (an odd one is rounded up, which must still fit one wave), split operands, 64-deep stages, K not split
  if (ppair) {
    p.kernel = GemmKernel::kPersistPair;
    p.sh = make_shape_persist_pair(bn, fmt);
  } else if (Epi::kHasPmax && lim.persist && splits == 1 && a_row0 == 0 && mt * ntile_cols > lim.n_sm &&
             ((nt == 2 && drain >= K / 32) || one_plane_logits)) {
    // many waves of tiles whose leading product is one chain: one persistent CTA per SM
    p.kernel = GemmKernel::kPersist;
    p.sh = nt == 1 ? make_shape_persist(bn, nt, p.bk, fmt)    // a ring of one stage less, staging areas of its own
                   : make_shape(bn, nt, p.bk, fmt);
  } else if (lim.pair && fmt == 1 && nt == 2 && whole_k && mt >= 2 && bn % 16 == 0 && make_shape(bn, nt, p.bk, fmt).stages < 3 &&
             (long)((mt + 1) & ~1) * ntile_cols <= lim.n_sm && alone) {
    p.kernel = GemmKernel::kPair;
    p.sh = make_shape_pair(bn, nt, p.bk, fmt);
  } else {
    p.sh = make_shape(bn, nt, p.bk, fmt);
  }
  p.sh.splits = splits;
  if (drain > 0) p.sh.drain = drain;
  p.b_box = p.on_pairs() ? bn / 2 : bn;
  return p;
}

// The tensor maps of `tm` have the plan's boxes; ws and counters are those the limits were given for.  late: the next kernel may
// start only once this one is past its wait (the few-rows kernel's offer, with fp32 results).
template <class Epi>
inline cudaError_t launch_planned(const GemmPlan& p, const TmapSet& tm, int M, int N, int K, int nt, int fmt, bool pdl, const Epi& e, int* err_flag,
                                  cudaStream_t st, int n_sm, float* ws, int* counters, int a_row0 = 0, bool late = false) {
  Shape sh = p.sh;
  sh.pdl = pdl ? 1 : 0;
  switch (p.kernel) {
    case GemmKernel::kRows: {
      RowsShape rs = p.rs;
      rs.pdl = pdl ? 1 : 0;
      if (nt == 2) return launch_gemm_tc_rows<2, 1, Epi>(tm, M, N, K, rs, e, err_flag, st, a_row0, late);
      if (fmt == 1) return launch_gemm_tc_rows<1, 1, Epi>(tm, M, N, K, rs, e, err_flag, st, a_row0, late);
      return launch_gemm_tc_rows<1, 0, Epi>(tm, M, N, K, rs, e, err_flag, st, a_row0, late);
    }
    case GemmKernel::kPersistPair:
      if constexpr (Epi::kHasBlock) {
        if (fmt == 1) return launch_gemm_tc_persist_pair<1, Epi>(tm, M, N, K, sh, e, err_flag, st, n_sm);
        return launch_gemm_tc_persist_pair<0, Epi>(tm, M, N, K, sh, e, err_flag, st, n_sm);
      }
      return cudaErrorInvalidValue;
    case GemmKernel::kPersist:
      if constexpr (Epi::kHasPmax) return launch_gemm_tc_persist(tm, M, N, K, sh, e, err_flag, st, n_sm);
      return cudaErrorInvalidValue;
    case GemmKernel::kPair:
      return launch_gemm_tc_pair<2, 64, 1, Epi>(tm, M, N, K, sh, e, err_flag, st, nullptr, nullptr);
    default:
      return launch_gemm_tc(tm, M, N, K, sh, e, err_flag, st, ws, counters, a_row0);
  }
}

}  // namespace tc
}  // namespace linmt
