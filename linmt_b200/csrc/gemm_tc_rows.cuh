// gemm_tc_rows.cuh -- the tensor-core GEMM for FEW activation rows (a decoder step of a sentence or a small batch).
//
//   C[R][N] = A[R][K] . Wt[N][K]^T   with R <= 128 (one plane: 64), N and K in the thousands
//
// With few rows the product is a stream of weights: every weight byte comes in once and meets R rows.  The kernel of
// gemm_tc.cuh puts the rows on the 128-wide M side of the MMA, holds a whole SM's shared memory and joins K slices
// through global memory with a ticket; at 12 rows that is 13.4 us per 33.5 MB layer (5.1 us of HBM time).  Here
//   * the WEIGHTS are the M operand (128 rows of Wt per tile) and the activations the N operand, R rounded up to 16;
//   * a CTA needs half an SM (<= 114 KB of shared memory, 256 TMEM columns), so that the next kernel's CTAs move in
//     beside this one's and have their first weight tiles requested before this kernel has finished (programmatic
//     dependent launch: weights depend on nothing);
//   * the K slices of a tile are the CTAs of one cluster; every CTA of the cluster owns some of the rows, and the others
//     write their partial sums of those rows into its shared memory (st.async, bytes counted on a barrier there).
// Rows are owned in units of four rows x 32 columns; a warp finishes a unit, four columns of one row to a lane, so that
// an LSTM cell's four gates meet in one lane.
//
// Accumulators.  With split operands (the f16 pair) the leading product is kept to short chains as in gemm_tc.cuh
// (the tensor core truncates on every accumulate): the K range of a CTA is dealt to `leads` accumulators, each chain
// at most three k-blocks, and the cross terms have columns of their own.  All of them are added in fp32 registers.
#pragma once
#include <type_traits>

#include "gemm_tc.cuh"
#include "gemm_tc_pair.cuh"

namespace linmt {
namespace tc {

constexpr int kRowsThreads = 256;       // warp 0 TMA, warps 1 and 2 issue MMAs, then all eight finish rows
constexpr int kRowsMax = 128;
constexpr int rows_max(int nt) { return nt == 1 ? 64 : 128; }    // (one plane, 96 rows: 9.5 us in the one-tile kernel, 10.5 here)
constexpr int kRowsMaxLeads = 4;
// Shared memory of a CTA that shares its SM with one of the next kernel's (SM: 228 KB, 1 KB of it per CTA reserved), and
// the least it asks for: with less, a third CTA would fit whose TMEM allocation waits for the other two, and CTAs of one
// cluster waiting on several SMs for CTAs of another could wait for each other.
constexpr int kRowsSmemHalf = 113 * 1024;
constexpr int kRowsSmemMin = 78 * 1024;
constexpr int kRowsSmemWhole = 224 * 1024;     // a CTA that has the SM to itself
// A CTA that takes all of an SM's TMEM asks for so much shared memory that none of the others fits beside it, as the other
// kernels with 512 columns do (their staging area alone): a CTA never waits for TMEM that a CTA of another stream holds, whose
// cluster might in turn wait for one that this CTA's cluster keeps out elsewhere.
constexpr int kRowsSmemWholeMin = 150 * 1024;
constexpr int kSmemPerSm = 228 * 1024, kSmemReserved = 1024;       // of an SM; of every block
static_assert(3 * (kRowsSmemMin + kSmemReserved) > kSmemPerSm && kRowsSmemWholeMin + kRowsSmemMin + 2 * kSmemReserved > kSmemPerSm &&
              kEpiStagingBytes + kRowsSmemMin + 2 * kSmemReserved > kSmemPerSm, "two CTAs of half the TMEM on an SM, or one of all of it");
constexpr int kRowsBarBytes = 384;

struct RowsShape {
  int rp, units;       // rows rounded up to 16 = N of the MMA; rows rounded up to 4 = units of 4 rows x 32 columns
  int wstages, xstages, recv_bytes, smem_bytes;   // rings of weight and activation k-blocks
  int splits;          // K slices = cluster size
  int leads, acc_stride, stacked, tmem_cols;
  int alias;           // the partial sums' buffer lies in the rings (and waits until the whole cluster is done with them)
  int pdl;
  int ahead;           // (several products in a launch) reads nothing of the kernel before it, and waits for that only at its end
};

// Everything that follows from the split.
inline bool rows_set_splits(RowsShape* s, int K, int nt) {
  // partial sums: the units are dealt to the CTAs of the cluster, 512 bytes a slice
  s->recv_bytes = (s->units + s->splits - 1) / s->splits * s->splits * 512;
  const int w = nt * BM * 128, x = nt * s->rp * 128;
  const int nkb = (K / 64 + s->splits - 1) / s->splits;
  for (s->alias = 0; s->alias < 2; ++s->alias) {
    const int room = (s->tmem_cols == 512 ? kRowsSmemWhole : kRowsSmemHalf) - (s->alias ? 0 : s->recv_bytes) - kRowsBarBytes;
    s->wstages = (room - 2 * x) / w;
    if (s->wstages > nkb) s->wstages = nkb;
    if (s->wstages > kMaxStages) s->wstages = kMaxStages;
    if (s->wstages < 1) continue;
    s->xstages = (room - s->wstages * w) / x;
    if (s->xstages > s->wstages) s->xstages = s->wstages;
    if (s->wstages >= 2 || nkb == 1 || s->alias) break;
  }
  if (s->alias > 1) return false;
  const int rings = s->wstages * w + s->xstages * x;
  if (s->alias && rings < s->recv_bytes) return false;
  s->smem_bytes = rings + (s->alias ? 0 : s->recv_bytes) + kRowsBarBytes;
  const int least = s->tmem_cols == 512 ? kRowsSmemWholeMin : kRowsSmemMin;
  if (s->smem_bytes < least) s->smem_bytes = least;
  return s->wstages >= 1 && s->xstages >= 1;
}

// one_chain: the leading product may be one long chain per accumulator (logits, see gemm_tc_persist_kernel)
// beside: a CTA per SM at most, so that the next product's are all in flight beside them, their rings full, when this one's
// results arrive (4096 x 1024 and 3072 x 1024 in a chain, 12 rows: 80 against 84 us a step with 256 and 192 CTAs, which take turns)
inline bool make_shape_rows(int rows, int N, int K, int nt, int fmt, int n_sm, bool one_chain, bool beside, RowsShape* out) {
  if (rows < 1 || rows > rows_max(nt) || K % 64 || K < 64 || N % 16) return false;
  if (!(nt == 1 || (nt == 2 && fmt == 1))) return false;
  RowsShape s{};
  s.rp = (rows + 15) & ~15; s.units = (rows + 3) & ~3;
  const int tiles = (N + BM - 1) / BM, nkb = K / 64;
  // One 128-column tile per cluster; K slices to fill the machine once.  CTAs of half an SM: measured best with as many
  // slices as a portable cluster has (4096 x 2048 at 12 rows: 10.2, 9.1, 8.7 us at 4, 6, 8 slices -- the more of the
  // weights are in flight when the activations arrive); CTAs of a whole SM: clusters of four are the largest of which
  // the device holds enough at once (8.1 us at 4, 14 us at 6 slices, 3072 x 1024 at 64 rows) -- for more rows than the
  // accumulators of half an SM's TMEM serve.  One plane and few rows: a CTA's slice fits its ring whole at half as many
  // slices (4096 x 2048 at 12 rows: 6.2 us at 4, 6.6 at 8; at 64 rows 9.5 and 8.0).
  for (int whole = 0; whole < 2; ++whole) {
    s.splits = (whole || beside || (nt == 1 && s.rp <= 32) ? n_sm : 2 * n_sm) / tiles;
    s.splits = s.splits < 1 ? 1 : (s.splits > (whole ? 4 : 8) ? (whole ? 4 : 8) : s.splits);
    if (s.splits > nkb) s.splits = nkb;
    s.tmem_cols = whole ? 512 : 256;
    // f16 pair: w0 meets both planes of the activations in ONE instruction (N = 2 rp, the planes lie one behind the
    // other), so an accumulator holds w0 x0 | w0 x1; beyond 64 rows an instruction per product takes as long, and the
    // columns are better spent on short chains
    // (or not, where that gives short enough chains in half an SM's columns and the SM is to be shared)
    for (s.stacked = nt == 2 && s.rp <= 64; s.stacked >= 0; --s.stacked) {
      s.acc_stride = s.stacked ? 2 * s.rp : (s.rp + 31) & ~31;
      s.leads = nt == 1 ? 1 : (s.tmem_cols - s.rp) / s.acc_stride;
      if (s.leads > kRowsMaxLeads) s.leads = kRowsMaxLeads;
      const bool chains = nt == 1 || one_chain || (nkb + s.splits - 1) / s.splits <= 3 * s.leads;   // a chain is at most three k-blocks
      if (s.leads >= 1 && chains && rows_set_splits(&s, K, nt)) {
        *out = s;
        return true;
      }
      if (!beside) break;
    }
  }
  return false;
}

// The shape of `segs` products of few rows that run beside other kernels (Engine::recurrent_ahead): as many K slices as fit
// beside a few whole-SM blocks at once, each with a long stream of weights, where make_shape_rows would have the whole product in
// flight (three products of 4096 x 1024 as launches of 256 CTAs each behind one another: 24 us more a step than these beside the
// attention and the softmax, 12 rows).  Half an SM each, so that the next kernel's CTAs find room.
constexpr int kRowsAhead = 60;
// (The f16 pair only: one plane keeps its order of sums.)
inline bool make_shape_ahead(int rows, int N, int K, int n_sm, int segs, RowsShape* out) {
  if (rows < 1 || rows > kRowsAhead || K % 64 || K < 64 || N % 16) return false;
  RowsShape s{};
  s.rp = (rows + 15) & ~15; s.units = (rows + 3) & ~3;
  s.tmem_cols = 256;
  const int tiles = (N + BM - 1) / BM * segs, nkb = K / 64, places = n_sm * 4 / 3;
  s.splits = 8;
  while (s.splits > 1 && tiles * s.splits > places) s.splits >>= 1;
  for (; s.splits <= 8; s.splits *= 2) {
    if (s.splits > nkb) s.splits = nkb;
    for (s.stacked = 1; s.stacked >= 0; --s.stacked) {     // (not stacked: more and shorter chains)
      s.acc_stride = s.stacked ? 2 * s.rp : (s.rp + 31) & ~31;
      s.leads = (s.tmem_cols - s.rp) / s.acc_stride;
      if (s.leads > kRowsMaxLeads) s.leads = kRowsMaxLeads;
      const bool chains = (nkb + s.splits - 1) / s.splits <= 3 * s.leads;   // a chain is at most three k-blocks
      if (chains && rows_set_splits(&s, K, 2)) {
        *out = s;
        return true;
      }
    }
    if (s.splits == nkb) break;
  }
  return false;
}

// four floats into the shared memory of a CTA of the cluster, their bytes counted on a barrier there
__device__ __forceinline__ void st_async4(uint32_t addr, uint32_t bar, float a, float b, float c, float d) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1,%2,%3,%4}, [%5];"
               ::"r"(addr), "f"(a), "f"(b), "f"(c), "f"(d), "r"(bar) : "memory");
}
// eight accumulator columns of this lane's row, not waited for
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// Several products of the same shape in one launch: blockIdx.y chooses the operands' maps, and Epi::of(blockIdx.y) the result.
template <int SEGS>
struct TmapSets { TmapSet s[SEGS]; };

// LATE: the next kernel may start only once this one is past its wait.  (Template parameters: a kernel's word to the next one is its
// first instruction, ahead of the first read of its parameters, which cost 1 to 3 % of a chain of small products.)
template <int NT, int FMT, class Epi, int SEGS, bool LATE>
__global__ void __launch_bounds__(kRowsThreads, 2)
gemm_tc_rows_kernel(const __grid_constant__ TmapSets<SEGS> tms, int M, int N, int K, int x_row0, RowsShape sh, Epi epi_of,
                    int* __restrict__ err_flag) {
  auto chosen = [&]() -> std::conditional_t<(SEGS > 1), Epi, const Epi&> {
    if constexpr (SEGS > 1) return epi_of.of(blockIdx.y);
    else return epi_of;
  };
  const Epi& epi = chosen();
  const TmapSet& tm = tms.s[SEGS > 1 ? blockIdx.y : 0];
  constexpr int PC = product_code(NT, FMT);
  static_assert(NT == 1 || PC == kF16PairCode, "one plane or the f16 pair");
  constexpr int W_BYTES = BM * 128;            // one plane of a weight k-block (64 deep)
  extern __shared__ __align__(1024) unsigned char rows_smem[];
  const uint32_t base = smem_u32(rows_smem);
  const int X_BYTES = sh.rp * 128;             // one plane of an activation k-block
  const int WS = sh.wstages, XS = sh.xstages;
  const uint32_t xbase = base + (uint32_t)(WS * NT * W_BYTES);
  const uint32_t rings_end = xbase + (uint32_t)(XS * NT * X_BYTES);
  const uint32_t recv = sh.alias ? base : rings_end;
  const uint32_t bars = rings_end + (sh.alias ? 0u : (uint32_t)sh.recv_bytes);   // W full[WS], W empty[WS], X full[XS], X empty[XS], accum, recv
  const uint32_t xbars = bars + 16u * WS, accum_bar = xbars + 16u * XS, recv_bar = accum_bar + 8u;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(rows_smem + (recv_bar + 8u - base));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(rows_smem + (recv_bar + 12u - base));

  if (!LATE) pdl_launch_dependents();
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int n0 = blockIdx.x * BM;
  const int splits = sh.splits, rank = blockIdx.z;
  const int nkb_total = K / 64;
  const int kb0 = nkb_total * rank / splits;
  const int nkb = nkb_total * (rank + 1) / splits - kb0;
  constexpr int issuers = NT;
  // units of 4 rows x 32 columns: unit u = 4 * (row group) + (column quarter) belongs to CTA u % splits of the cluster
  const int units = (M + 3) & ~3;
  const int n_own = rank < units ? (units - rank + splits - 1) / splits : 0;

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < WS; ++s) { mbar_init(bars + 8u * s, 1); mbar_init(bars + 8u * (WS + s), issuers); }
    for (int s = 0; s < XS; ++s) { mbar_init(xbars + 8u * s, 1); mbar_init(xbars + 8u * (XS + s), issuers); }
    mbar_init(accum_bar, issuers);
    mbar_init(recv_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    mbar_expect_tx(recv_bar, (uint32_t)(n_own * (splits - 1) * 512));   // the neighbours' share
  }
  const bool one = elect_one();
  const uint64_t policy = warp == 0 ? weight_policy(tm.stream_b) : 0;
  auto load_w = [&](int kb, int stage) {
#pragma unroll
    for (int t = 0; t < NT; ++t) tma_load_2d(base + (uint32_t)((stage * NT + t) * W_BYTES), &tm.b[t], (kb0 + kb) * 64, n0, bars + 8u * stage, policy);
  };
  auto load_x = [&](int kb, int stage) {
#pragma unroll
    for (int t = 0; t < NT; ++t) tma_load_2d(xbase + (uint32_t)((stage * NT + t) * X_BYTES), &tm.a[t], (kb0 + kb) * 64, x_row0, xbars + 8u * stage);
  };
  const int prew = nkb < WS ? nkb : WS, prex = nkb < XS ? nkb : XS;
  if (warp == 0) {
    if (one) {
#pragma unroll
      for (int t = 0; t < NT; ++t) asm volatile("prefetch.tensormap [%0];" ::"l"(&tm.a[t]) : "memory");   // there when the wait ends
      for (int kb = 0; kb < prew; ++kb) {
        mbar_expect_tx(bars + 8u * kb, (uint32_t)(NT * W_BYTES));
        load_w(kb, kb);
      }
      for (int kb = 0; kb < prex; ++kb) mbar_expect_tx(xbars + 8u * kb, (uint32_t)(NT * X_BYTES));
    }
    __syncwarp();
  } else if (warp == 1) {
    tmem_alloc(recv_bar + 8u, (uint32_t)sh.tmem_cols);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (splits > 1) cluster_arrive();     // the barriers above exist (waited for before the first remote write)
  const uint32_t tmem = *tmem_slot;

  if (SEGS == 1 || !sh.ahead) pdl_wait();    // from here on the previous kernel's results are visible
  if (LATE) pdl_launch_dependents();
  if (warp == 0 && one)
    for (int kb = 0; kb < prex; ++kb) load_x(kb, kb);
  // what the epilogue of this warp's first unit reads is requested now and used after the accumulators are complete
  auto unit_row = [&](int i) { return ((rank + splits * i) >> 2) * 4 + (lane & 3); };
  auto unit_col = [&](int i) { return n0 + ((rank + splits * i) & 3) * 32 + (lane & ~3); };    // of the lane's four columns
  typename Epi::Pre pre{};
  if (warp < n_own && unit_row(warp) < M && unit_col(warp) < N) pre = epi.preload(unit_row(warp), unit_col(warp));

  if (warp == 0) {
    int ws = prew == WS ? 0 : prew, xs = prex == XS ? 0 : prex;
    uint32_t wph = prew == WS ? 1u : 0u, xph = prex == XS ? 1u : 0u;
    int kw = prew, kx = prex;
    while (kw < nkb || kx < nkb) {
      // the ring that is behind goes first (with equal depths: alternately)
      const bool do_w = kx >= nkb || (kw < nkb && kw <= kx);
      if (do_w) {
        if (!mbar_wait(bars + 8u * (WS + ws), wph ^ 1u, abort_flag)) break;
        if (one) { mbar_expect_tx(bars + 8u * ws, (uint32_t)(NT * W_BYTES)); load_w(kw, ws); }
        ++kw;
        if (++ws == WS) { ws = 0; wph ^= 1u; }
      } else {
        if (!mbar_wait(xbars + 8u * (XS + xs), xph ^ 1u, abort_flag)) break;
        if (one) { mbar_expect_tx(xbars + 8u * xs, (uint32_t)(NT * X_BYTES)); load_x(kx, xs); }
        ++kx;
        if (++xs == XS) { xs = 0; xph ^= 1u; }
      }
    }
  } else if (warp <= issuers) {
    // warp 1: w0 times the activations (both planes of the f16 pair if stacked), warp 2 (f16 pair): w1 x0, and w0 x1 if not
    const uint32_t idesc = make_idesc(BM, sh.stacked && warp == 1 ? 2 * sh.rp : sh.rp, FMT);
    const int chain = NT == 1 ? nkb : (nkb + sh.leads - 1) / sh.leads;   // k-blocks per leading accumulator
    int ws = 0, xs = 0, in_chain = 0;
    uint32_t wph = 0, xph = 0;
    uint32_t acc = warp == 1 ? tmem : tmem + (uint32_t)(sh.leads * sh.acc_stride);
    const uint32_t woff = warp == 1 ? 0u : (uint32_t)W_BYTES;
    for (int kb = 0; kb < nkb; ++kb) {
      if (!mbar_wait(bars + 8u * ws, wph, abort_flag) || !mbar_wait(xbars + 8u * xs, xph, abort_flag)) break;
      tc_fence_after();
      const uint64_t w0 = make_desc<64>(base + (uint32_t)(ws * NT * W_BYTES) + woff), x0 = make_desc<64>(xbase + (uint32_t)(xs * NT * X_BYTES));
      if (warp == 1 && in_chain == chain) { in_chain = 0; acc += (uint32_t)sh.acc_stride; }
      if (one) {
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) umma_bf16(acc, w0 + (uint64_t)(ks * 2), x0 + (uint64_t)(ks * 2), idesc, (in_chain | ks) ? 1u : 0u);
        if (NT == 2 && warp == 2 && !sh.stacked) {      // w0 x1
          const uint64_t wl = w0 - (uint64_t)(W_BYTES >> 4), x1 = x0 + (uint64_t)(X_BYTES >> 4);
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) umma_bf16(acc, wl + (uint64_t)(ks * 2), x1 + (uint64_t)(ks * 2), idesc, 1u);
        }
        umma_commit(bars + 8u * (WS + ws));
        umma_commit(xbars + 8u * (XS + xs));
      }
      ++in_chain;
      if (++ws == WS) { ws = 0; wph ^= 1u; }
      if (++xs == XS) { xs = 0; xph ^= 1u; }
    }
    if (one) umma_commit(accum_bar);
  }
  __syncwarp();

  // Accumulators -> the owners' shared memory: a warp has 32 columns (its TMEM lanes) of every other block of eight rows.
  // Partial sums of a unit: [slice][32 columns][4 rows].
  const int q = warp & 3, half = warp >> 2;
  if (splits > 1) cluster_wait();
  const bool done = mbar_wait(accum_bar, 0, abort_flag);
  if (sh.alias) {        // nobody writes into a ring that is still being read
    __syncwarp();
    if (splits > 1) cluster_sync_all(); else __syncthreads();
  }
  if (done) {
    tc_fence_after();
    const int chain = (nkb + sh.leads - 1) / sh.leads;
    const int used = NT == 1 ? 1 : (nkb + chain - 1) / chain;
    constexpr int ML = NT == 1 ? 1 : kRowsMaxLeads;
    for (int rb = half * 8; rb < M; rb += 16) {
      const uint32_t at = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)rb;
      uint32_t lead[ML][8], cross[ML + 1][8];
#pragma unroll
      for (int a = 0; a < ML; ++a)
        if (a < used) {
          tmem_ld8(at + (uint32_t)(a * sh.acc_stride), lead[a]);
          if (NT > 1 && sh.stacked) tmem_ld8(at + (uint32_t)(a * sh.acc_stride + sh.rp), cross[a]);
        }
      if (NT > 1) tmem_ld8(at + (uint32_t)(sh.leads * sh.acc_stride), cross[ML]);
      tmem_wait_ld();
      float v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        v[i] = __uint_as_float(lead[0][i]);
        if (NT > 1) {
          float c = __uint_as_float(cross[ML][i]);
#pragma unroll
          for (int a = 0; a < ML; ++a)
            if (a < used) {
              if (a > 0) v[i] += __uint_as_float(lead[a][i]);
              if (sh.stacked) c += __uint_as_float(cross[a][i]);
            }
          v[i] = fmaf(c, kF16PairInvScale, v[i]);
        }
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int u = rb + 4 * h + q;      // 4 * (row group) + quarter
        if (rb + 4 * h < M) {
          const int owner = u % splits, slot = u / splits;
          const int at_unit = (slot * splits + rank) * 32 + lane;
          // (st.async is for another CTA's shared memory only; what stays here is ordered by the barrier below)
          if (owner == rank) reinterpret_cast<float4*>(rows_smem + (recv - base))[at_unit] = make_float4(v[4 * h], v[4 * h + 1], v[4 * h + 2], v[4 * h + 3]);
          else st_async4(cluster_map(recv + (uint32_t)(at_unit * 16), (uint32_t)owner), cluster_map(recv_bar, (uint32_t)owner), v[4 * h], v[4 * h + 1], v[4 * h + 2], v[4 * h + 3]);
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, (uint32_t)sh.tmem_cols);

  if (n_own > 0 && mbar_wait(recv_bar, 0, abort_flag)) {
    const float4* part = reinterpret_cast<const float4*>(rows_smem + (recv - base)) + lane;
    for (int i = warp; i < n_own; i += kRowsThreads / 32) {
      const int row = unit_row(i), col = unit_col(i);
      const bool valid = row < M && col < N;
      if (i != warp && valid) pre = epi.preload(row, col);
      float4 v = part[(i * splits) * 32];
      for (int z = 1; z < splits; ++z) {
        const float4 w = part[(i * splits + z) * 32];
        v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
      }
      // four rows of one column -> four columns of one row, within four lanes
      {
        const bool o = lane & 1, p = lane & 2;
        const float a = __shfl_xor_sync(0xffffffffu, o ? v.x : v.y, 1), b = __shfl_xor_sync(0xffffffffu, o ? v.z : v.w, 1);
        if (o) { v.x = a; v.z = b; } else { v.y = a; v.w = b; }
        const float c = __shfl_xor_sync(0xffffffffu, p ? v.x : v.z, 2), d = __shfl_xor_sync(0xffffffffu, p ? v.y : v.w, 2);
        if (p) { v.x = c; v.y = d; } else { v.z = c; v.w = d; }
      }
      epi.finish_row(valid, row, col, lane, v, pre);
    }
  }
  if (threadIdx.x == 0 && *abort_flag) atomicExch(err_flag, 1);
  if (SEGS > 1 && sh.ahead) pdl_wait();     // (who waits for this kernel waits for the one before it as well)
}

// x_row0: first row of the product in the activations' tensor map
template <int NT, int FMT, class Epi, int SEGS, bool LATE>
inline cudaError_t launch_gemm_tc_rows_of(const TmapSets<SEGS>& tms, int segs, int M, int N, int K, const RowsShape& sh, const Epi& epi,
                                          int* err_flag, cudaStream_t st, int x_row0) {
  static std::atomic<bool> optin_done[kMaxDevices] = {};
  if (cudaError_t e = ensure_smem_optin(gemm_tc_rows_kernel<NT, FMT, Epi, SEGS, LATE>, optin_done, kRowsSmemWhole); e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((N + BM - 1) / BM, segs, sh.splits); cfg.blockDim = dim3(kRowsThreads);
  cfg.dynamicSmemBytes = (size_t)sh.smem_bytes; cfg.stream = st;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (sh.splits > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = 1; attr[na].val.clusterDim.y = 1; attr[na].val.clusterDim.z = sh.splits;
    ++na;
  }
  if (sh.pdl) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  return cudaLaunchKernelEx(&cfg, gemm_tc_rows_kernel<NT, FMT, Epi, SEGS, LATE>, tms, M, N, K, x_row0, sh, epi, err_flag);
}
template <int NT, int FMT, class Epi>
inline cudaError_t launch_gemm_tc_rows(const TmapSet& tm, int M, int N, int K, const RowsShape& sh, const Epi& epi, int* err_flag, cudaStream_t st,
                                       int x_row0 = 0, bool late = false) {
  if constexpr (Epi::kLate)
    if (late) return launch_gemm_tc_rows_of<NT, FMT, Epi, 1, true>(TmapSets<1>{{tm}}, 1, M, N, K, sh, epi, err_flag, st, x_row0);
  return launch_gemm_tc_rows_of<NT, FMT, Epi, 1, false>(TmapSets<1>{{tm}}, 1, M, N, K, sh, epi, err_flag, st, x_row0);
}

}  // namespace tc
}  // namespace linmt
