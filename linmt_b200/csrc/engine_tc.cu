// engine_tc.cu -- the tensor-core path of the engine: operands as bf16 planes, every GEMM a
// tcgen05/TMEM kernel fed by TMA, LSTM cell / tanh / bias fused into the epilogues.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <algorithm>

#include "encoder_form.h"
#include "engine.h"
#include "gemm_plan.cuh"
#include "gemm_tc.cuh"
#include "step_kernels.cuh"
#include "weight_stream.h"

namespace linmt {

#define LAUNCHED() (++stats.kernel_launches)

int Engine::alloc_planes(tc::Planes& p, size_t rows, int ld) {
  p = tc::Planes{};
  p.ld = ld;
  p.fmt = fmt_;
  for (int t = 0; t < nt_; ++t) {
    void* q = nullptr;
    const size_t bytes = rows * (size_t)ld * sizeof(__nv_bfloat16);
    if (int rc = device_memory(&q, bytes, "operand planes")) return rc;
    allocs_.push_back(q);
    // (on the engine's stream, whose kernels do not wait for the legacy one: scoring makes its panels in the middle of a call)
    if (cudaMemsetAsync(q, 0, bytes, stream) != cudaSuccess) return fail(LINMT_ECUDA, "cudaMemsetAsync failed (operand planes)");
    p.p[t] = static_cast<__nv_bfloat16*>(q);
  }
  return LINMT_OK;
}

// fp32 host matrix -> device -> bf16 planes (the split runs on the GPU).
int Engine::to_planes(const std::vector<float>& host, size_t rows, int ld, tc::Planes& dst) {
  int rc = alloc_planes(dst, rows, ld);
  if (rc) return rc;
  float* tmp = nullptr;
  const size_t n = rows * (size_t)ld;
  if (host.size() < n) return fail(LINMT_EINVAL, "internal: packed matrix smaller than its planes");
  if ((rc = device_memory(reinterpret_cast<void**>(&tmp), n * sizeof(float), "weight staging"))) return rc;
  // stream-ordered copy: the split kernel must not start before the last byte has landed
  cudaError_t e = cudaMemcpyAsync(tmp, host.data(), n * sizeof(float), cudaMemcpyHostToDevice, stream);
  if (e == cudaSuccess) {
    tc::split_planes_kernel<<<2048, 256, 0, stream>>>(tmp, dst, nt_, n);
    LAUNCHED();
    e = cudaStreamSynchronize(stream);
  }
  cudaFree(tmp);
  if (e != cudaSuccess) return fail(LINMT_ECUDA, std::string("weight split: ") + cudaGetErrorString(e));
  return LINMT_OK;
}

int Engine::alloc_state_tc(TcState& s) {
  int rc;
  for (int i = 0; i < 2; ++i) {
    if ((rc = alloc_planes(s.panel1[i], R, 3 * Hp))) return rc;
    s.panel[i].resize(L);
    for (int l = 1; l < L; ++l)
      if ((rc = alloc_planes(s.panel[i][l], R, 2 * Hp))) return rc;
  }
  if ((rc = alloc_planes(s.panel_top, R, 2 * Hp))) return rc;
  if ((rc = alloc_planes(s.panel_ht, R, Hp))) return rc;
  if (att_fold_ && !states16() && (rc = alloc_planes(s.hs_planes, (size_t)B * opt.max_src_len, Hp))) return rc;
  if (enc_rows_) {
    if ((rc = alloc_planes(s.enc_in, enc_rows_, Hp))) return rc;
    s.enc_seq.resize(L);
    for (int l = 0; l < L; ++l)
      if ((rc = alloc_planes(s.enc_seq[l], (size_t)enc_rows_ + tc::kRowsMax, Hp))) return rc;
  }
  for (int i = 0; i < 2; ++i) {
    s.encp[i].resize(L);
    for (int l = 0; l < L; ++l)
      if ((rc = alloc_planes(s.encp[i][l], B, 2 * Hp))) return rc;
  }
  return LINMT_OK;
}

// Tensor maps are built once per (buffer view, box) and reused by every launch.
const CUtensorMap* Engine::maps(const tc::Planes& p, int col0, int rows, int K, int box_rows, int bk) {
  auto key = std::make_tuple((const void*)(p.p[0] + col0), rows, K, p.ld, box_rows + 1000 * bk);
  auto it = tmap_cache_.find(key);
  if (it == tmap_cache_.end()) {
    std::array<CUtensorMap, 3> m{};
    for (int t = 0; t < nt_; ++t)
      if (!tc::make_tmap(&m[t], p.p[t] + col0, rows, K, p.ld, box_rows, bk)) return nullptr;
    it = tmap_cache_.emplace(key, m).first;
  }
  return it->second.data();
}

// Products of a device batch that others run beside: up to 64 rows in CTAs of half an SM, as few of them as leave room for another
// product's; beyond, in tiles for half of the SMs.  4 x 1000 / 30k, ms a call shaped for the whole chip / so: 300 sentences greedily,
// 64 rows in a batch, 36.2 / 31.4; four batches, greedily 128 rows 25.3 / 21.5; beam 4, 128 rows 23.7 / 20.4, 256 rows 28.6 / 27.1;
// beam 8, 512 rows 42.5 / 41.2; scoring 128 15.9 / 13.8.  (Products of all positions fill the chip.  One plane: shaped for the whole
// chip, see Engine::Several.)
static constexpr int kSeveralFew = 64, kSeveralMost = 512;

// C[M][N] = A[:, a_col0 : a_col0+K] . W[N][K]^T on the kernel and in the shape that plan_gemm chooses.
template <class Epi>
int Engine::tc_gemm(const tc::Planes& A, int a_col0, int a_rows_cap, const tc::Planes& W, int M, int N, int K, const Epi& e_in, int nt, int drain, int x_row0) {
  Epi e = e_in;
  if (nt <= 0 || nt > nt_) nt = nt_;
  tc::GemmLimits lim;
  lim.beside = beside_ || several_;
  lim.n_sm = n_sm_; lim.parts = plan_parts_ ? plan_parts_ : ws_parts_;
  if (several_ && lim.parts == 1 && M > kSeveralFew && M <= kSeveralMost) lim.parts = 2;
  lim.rows = rows_; lim.pair = pair_; lim.persist = persist_;
  // a layer's slice of the split-K workspace: whole 256-byte units, so that every slice starts aligned for the
  // 16-byte partial-tile stores whatever the number of layers sharing it
  lim.ws_floats = (kSplitKWsFloats / ws_parts_) & ~(size_t)63;
  lim.max_tiles = kSplitKMaxTiles / ws_parts_;
  const tc::GemmPlan plan = tc::plan_gemm<Epi>(M, N, K, nt, fmt_, drain, x_row0, lim);
  got_late_ = want_late_ && plan.kernel == tc::GemmKernel::kRows;
  want_late_ = false;
  const CUtensorMap* am = maps(A, a_col0, a_rows_cap, K, plan.a_box, plan.bk);
  const CUtensorMap* bm = maps(W, 0, N, K, plan.b_box, plan.bk);
  if (!am || !bm) return fail(LINMT_ECUDA, "cuTensorMapEncodeTiled failed");
  tc::TmapSet tm;
  std::memcpy(tm.a, am, sizeof(tm.a));
  std::memcpy(tm.b, bm, sizeof(tm.b));
  // (one plane and many rows: tensor-bound, and its row tiles read the weights several times over: 1536 rows 29.5 -> 29.9 ms a
  // call as a stream)
  tm.stream_b = stream_weights_ && (nt > 1 || M <= 256);
  if constexpr (Epi::kHasPmax) {
    if (e.pmax) {
      blocks_ = logit_blocks(e.pmax, e.psum, e.pmax_ld, N, K, plan.stat_tile, plan.stat_part);
      e.pmax = blocks_.max; e.psum = blocks_.sum;
    }
  }
  CK(tc::launch_planned(plan, tm, M, N, K, nt, fmt_, pdl_ && pdl_gemm_, e, d_tc_err_, stream, n_sm_, d_splitk_ws_ + (size_t)ws_part_ * lim.ws_floats,
                        d_splitk_counters_ + ws_part_ * lim.max_tiles, x_row0, got_late_));
  LAUNCHED();
  if (plan.on_pairs()) ++stats.pair_launches;
  return LINMT_OK;
}

// The weights of a step are loaded as a stream (weight_stream.h).
bool Engine::step_streams(bool scoring, int rows) const {
  return weights_stream(StepWeights{L, Hp, Vp, n_models, nt_, nt_vocab_}, (size_t)l2_bytes_, scoring, rows);
}

bool Engine::pairs_available() { return tc::max_resident_pairs<2, 64, 1, tc::TcEpiLstm>() > 0; }

static tc::Planes no_planes() { return tc::Planes{}; }

// Input-term table of the first decoder layer: dec_xw[v][:] = W_x . embedding(v) for every target word, computed
// once with the same tensor GEMM (W_x = the first Hp of the K columns of the layer's weight planes).
int Engine::build_xw_tables() {
  for (int mi = 0; mi < n_models; ++mi) {
    DevModel& m = models_[mi];
    void* q = nullptr;
    const size_t bytes = (size_t)desc.vocab_tgt * 4 * Hp * sizeof(float);
    if (int rc = device_memory(&q, bytes, "input-term table")) return rc;
    allocs_.push_back(q);
    m.dec_xw = static_cast<float*>(q);
    tc::TcEpiF32 e{nullptr, m.dec_xw, 4 * Hp, 0};
    pdl_gemm_ = false;
    int rc = tc_gemm(m.p_emb_tgt, 0, desc.vocab_tgt, m.p_dec_w[0], desc.vocab_tgt, 4 * Hp, Hp, e);
    if (rc) return rc;
  }
  CK(cudaStreamSynchronize(stream));
  int herr = 0;
  CK(cudaMemcpy(&herr, d_tc_err_, sizeof(int), cudaMemcpyDeviceToHost));
  if (herr) return fail(LINMT_ECUDA, "a tensor-core GEMM gave up waiting on a barrier while building the input-term table");
  return LINMT_OK;
}

static constexpr int kEncRing = 4;
int Engine::encoder_streams() {
  if (enc_start_ev_) return LINMT_OK;      // (the last to be made)
  enc_streams_.resize(L);
  enc_events_.resize(L, std::vector<cudaEvent_t>(kEncRing));
  for (int l = 0; l < L; ++l) {
    if (!enc_streams_[l]) CK(cudaStreamCreateWithFlags(&enc_streams_[l], cudaStreamNonBlocking));
    for (int r = 0; r < kEncRing; ++r)
      if (!enc_events_[l][r]) CK(cudaEventCreateWithFlags(&enc_events_[l][r], cudaEventDisableTiming));
  }
  CK(cudaEventCreateWithFlags(&enc_start_ev_, cudaEventDisableTiming));
  return LINMT_OK;
}

// Encoder, tensor-core path (see Engine::run_encoder for the reference procedure).  Panel of
// layer l at position p: encp[p&1][l] = (input from below | h_prev).  The epilogue writes h to
// the next position's h_prev slot and to the next layer's input slot of this position.
//
// (layer l, position p) depends on (l-1, p) and (l, p-1) only, and each launch fills about half
// the SMs (64 rows = one row tile), so the layers run as a wavefront: one stream per layer,
// events for the cross-layer edges.  Besides the true dependencies, (l, p) waits for (l+1, p-2),
// the last reader of the double-buffered input slot it overwrites.
// Which form, and in which shapes: encoder_form.h.
int Engine::run_encoder_tc(int n, int Smax) {
  const EncoderModel model{L, Hp, n_models, nt_ > 1};
  const bool side = encoder_layers_beside(model, n, Smax, several_);
  stream_weights_ = false; beside_ = encoder_leaves_room(model, n, side);
  if (enc_rows_)
    switch (encoder_form(model, n, Smax)) {
      case EncoderForm::kLayers: return side ? run_encoder_pipeline_tc(n, Smax, true) : run_encoder_layers_tc(n, Smax);
      case EncoderForm::kPipelined: return run_encoder_pipeline_tc(n, Smax, false);
      case EncoderForm::kWavefront: break;
    }
  constexpr int kRing = kEncRing;
  hs_sent_ = opt.max_src_len; hs_pos_ = 1; enc_final_row_ = -1;
  if (int rc = encoder_streams()) return rc;
  cudaStream_t main_stream = stream;
  pdl_gemm_ = false;
  for (int mi = 0; mi < n_models; ++mi) {
    DevModel& m = models_[mi];
    DevState& s = states_[mi];
    TcState& ts = tc_states_[mi];
    for (int l = 0; l < L; ++l) {
      CK(cudaMemsetAsync(s.enc_c[0][l], 0, sizeof(float) * (size_t)B * Hp, main_stream));
      for (int t = 0; t < nt_; ++t)  // h_prev = 0 at the first position
        CK(cudaMemset2DAsync(ts.encp[0][l].p[t] + Hp, (size_t)2 * Hp * 2, 0, (size_t)Hp * 2, B, main_stream));
    }
    CK(cudaEventRecord(enc_start_ev_, main_stream));
    for (int l = 0; l < L; ++l) CK(cudaStreamWaitEvent(enc_streams_[l], enc_start_ev_, 0));
    int rc = LINMT_OK;
    for (int pos = 0; pos < Smax && rc == LINMT_OK; ++pos) {
      const int in = pos & 1, out = in ^ 1;
      for (int l = 0; l < L && rc == LINMT_OK; ++l) {
        cudaStream_t sl = enc_streams_[l];
        if (l > 0) CK(cudaStreamWaitEvent(sl, enc_events_[l - 1][pos % kRing], 0));
        if (l + 1 < L && pos >= 2) CK(cudaStreamWaitEvent(sl, enc_events_[l + 1][(pos - 2) % kRing], 0));
        if (l == 0) {
          dim3 grid(n, nt_);
          enc_embed_planes_kernel<<<grid, 128, 0, sl>>>(cur_ids_, d_off_, d_len_, m.p_emb_src, desc.vocab_src, ts.encp[in][0], Hp, pos);
          LAUNCHED();
        }
        tc::TcEpiLstm e{};
        e.bias = m.enc_b[l]; e.c_prev = s.enc_c[in][l]; e.ldc = Hp; e.c_out = s.enc_c[out][l];
        e.h_out1 = ts.encp[out][l]; e.h1_col0 = Hp;
        if (l + 1 < L) { e.h_out2 = ts.encp[in][l + 1]; e.h2_col0 = 0; } else { e.h_out2 = s.hs16; e.h_out2.ld = (int)opt.max_src_len * Hp; e.h2_col0 = pos * Hp; }
        e.h_prev = ts.encp[in][l]; e.hp_col0 = Hp;
        e.h_f32 = (l == L - 1 && s.hs) ? s.hs + (size_t)pos * Hp : nullptr;
        e.hf_row_stride = (long long)opt.max_src_len * Hp;
        e.row_len = d_len_; e.pos = pos; e.nt = nt_;
        stream = sl;  // tc_gemm launches on the member stream, with this layer's slice of the split-K workspace
        ws_part_ = l; ws_parts_ = L;
        rc = tc_gemm(ts.encp[in][l], 0, B, m.p_enc_w[l], n, 4 * Hp, 2 * Hp, e);
        stream = main_stream; ws_part_ = 0; ws_parts_ = 1;
        if (rc == LINMT_OK) CK(cudaEventRecord(enc_events_[l][pos % kRing], sl));
      }
    }
    // the decoder (main stream) starts after the last launch of every layer
    for (int l = 0; l < L; ++l)
      if (Smax > 0) CK(cudaStreamWaitEvent(main_stream, enc_events_[l][(Smax - 1) % kRing], 0));
    if (rc != LINMT_OK) return rc;
    if (att_fold_) {
      // W_c1 applied to every encoder state of the batch, once: the decoder's attention then sums these rows and
      // needs no output GEMM of its own (see AttFold in step_kernels.cuh).  Rows past a sentence's length hold
      // whatever an earlier batch left there; nothing reads their products.
      const size_t rows_all = (size_t)n * opt.max_src_len;
      if (s.hs) {
        tc::split_planes_kernel<<<1024, 256, 0, main_stream>>>(s.hs, ts.hs_planes, nt_, rows_all * Hp);
        LAUNCHED();
      }
      tc::TcEpiF32 e{nullptr, s.hs_wc1, Hp, 0};
      if ((rc = tc_gemm(s.hs ? ts.hs_planes : s.hs16, 0, B * (int)opt.max_src_len, m.p_att_out_w, (int)rows_all, Hp, Hp, e))) return rc;
    }
  }
  return LINMT_OK;
}

// Encoder for few sentences, layer by layer.  A layer's input part W_x . x_p of ALL positions is one GEMM; what is left of the
// recurrence per position is W_h . h (half of the layer's weights, which then stay in L2 from one position to the next) in the
// few-rows kernel, or for wide models in the one-tile kernel, with the input part added in the epilogue.  L x S short launches
// instead of S rounds of L launches on L streams that each read the whole layer from HBM: one sentence of 30 words 1.28 -> 0.75
// ms.  Block p of a layer's sequence panel holds its states after p positions (block 0 the state before): operand of the next
// position and, as a whole, of the next layer's input GEMM.  Sources longer than the panels are taken in chunks.
int Engine::run_encoder_layers_tc(int n, int Smax) {
  hs_sent_ = 1; hs_pos_ = n;
  const int per = enc_rows_ / n;               // positions per chunk
  pdl_gemm_ = true;
  enc_final_row_ = (Smax - (Smax - 1) / per * per) * n;     // (of the last chunk)
  return each_member(n, [&](int mi) { return encode_member_layers(mi, n, Smax, per); });
}

// Positions pos0 .. pos0 + np of layer l, whose input parts are in `pre`: W_h . h in the few-rows kernel or in the one-tile
// kernel, with the input part added in the epilogue.  Their states go into the layer's sequence panel from block `block` on.
int Engine::encode_positions(int mi, int l, int n, int pos0, int np, float* pre, int block) {
  DevModel& m = models_[mi];
  DevState& s = states_[mi];
  const tc::Planes& seq = tc_states_[mi].enc_seq[l];
  tc::Planes wh = m.p_enc_w[l];
  for (int t = 0; t < nt_; ++t) wh.p[t] += Hp;
  for (int q = 0; q < np; ++q) {
    const int pos = pos0 + q;
    tc::TcEpiLstm e{};
    e.bias = m.enc_b[l]; e.c_prev = s.enc_c[pos & 1][l]; e.ldc = Hp; e.c_out = s.enc_c[(pos & 1) ^ 1][l];
    e.xw = pre + (size_t)q * n * 4 * Hp; e.x_ld = 4 * Hp;
    e.h_out1 = seq; e.h1_col0 = 0;
    e.h_prev = seq; e.hp_col0 = 0;
    for (int t = 0; t < nt_; ++t) { e.h_out1.p[t] += (size_t)(block + q + 1) * n * Hp; e.h_prev.p[t] += (size_t)(block + q) * n * Hp; }
    e.h_out2 = l == L - 1 ? s.hs16 : no_planes(); e.h2_col0 = 0;
    if (e.h_out2.p[0]) e.h_out2.p[0] += (size_t)pos * n * Hp;
    e.h_f32 = (l == L - 1 && s.hs) ? s.hs + (size_t)pos * n * Hp : nullptr;
    e.hf_row_stride = Hp;
    e.row_len = d_len_; e.pos = pos; e.nt = nt_;
    if (int rc = tc_gemm(seq, 0, enc_rows_ + tc::kRowsMax, wh, n, 4 * Hp, Hp, e, 0, 0, (block + q) * n)) return rc;
  }
  return LINMT_OK;
}

// Encoder for more sentences and longer sources (`few`: few sentences): the layers side by side on a stream each, every one kEncLag
// positions behind the layer below.
// As in the form above, the input parts of that many positions are one product, and what is left of the recurrence reads
// half of a layer's weights, which all layers' together (67 MB in fp32 precision) stay in L2; but every layer's products are
// shaped for their share of the SMs and run beside the others'.  Sources longer than the panels are taken in chunks: the
// layers fall in line at the end of one, and the next starts from the states it ended with (4 x 1000, 500 words, two chunks,
// against one position after another: 40 sentences 14.2 / 19.7 ms, 64 15.6 / 20.7).
// few: the products of few sentences are those of the form above (encoder_layers_beside).
int Engine::run_encoder_pipeline_tc(int n, int Smax, bool few) {
  if (int rc = encoder_streams()) return rc;
  hs_sent_ = 1; hs_pos_ = n;
  const int per = enc_rows_ / n;               // positions per chunk
  enc_final_row_ = (Smax - (Smax - 1) / per * per) * n;     // (of the last chunk)
  const int share = enc_rows_ / L, lag = std::max(1, std::min(kEncLag, share / n));
  const cudaStream_t main_stream = stream;
  pdl_gemm_ = true;
  for (int mi = 0; mi < n_models; ++mi) {
    DevModel& m = models_[mi];
    DevState& s = states_[mi];
    TcState& ts = tc_states_[mi];
    for (int l = 0; l < L; ++l) {
      CK(cudaMemsetAsync(s.enc_c[0][l], 0, sizeof(float) * (size_t)n * Hp, stream));
      for (int t = 0; t < nt_; ++t) CK(cudaMemsetAsync(ts.enc_seq[l].p[t], 0, sizeof(uint16_t) * (size_t)n * Hp, stream));
    }
    for (int c0 = 0; c0 < Smax; c0 += per) {
      const int len = std::min(per, Smax - c0);
      if (c0 > 0)   // the states the previous chunk ended with
        for (int l = 0; l < L; ++l)
          for (int t = 0; t < nt_; ++t)
            CK(cudaMemcpyAsync(ts.enc_seq[l].p[t], ts.enc_seq[l].p[t] + (size_t)per * n * Hp, sizeof(uint16_t) * (size_t)n * Hp, cudaMemcpyDeviceToDevice, stream));
      enc_embed_seq_kernel<<<dim3(n, len, nt_), 128, 0, stream>>>(cur_ids_, d_off_, d_len_, m.p_emb_src, desc.vocab_src, ts.enc_in, Hp, c0);
      LAUNCHED();
      CK(cudaEventRecord(enc_start_ev_, main_stream));
      for (int l = 0; l < L; ++l) CK(cudaStreamWaitEvent(enc_streams_[l], enc_start_ev_, 0));
      int rc = LINMT_OK;
      for (int p0 = 0; p0 < len && rc == LINMT_OK; p0 += lag) {
        const int np = std::min(lag, len - p0);
        for (int l = 0; l < L && rc == LINMT_OK; ++l) {
          if (l > 0) CK(cudaStreamWaitEvent(enc_streams_[l], enc_events_[l - 1][0], 0));
          stream = enc_streams_[l];       // (tc_gemm: on the layer's stream, with its slice of the split-K workspace)
          ws_part_ = l; ws_parts_ = L; plan_parts_ = few ? 1 : L;
          float* pre = s.enc_pre + (size_t)l * share * 4 * Hp;
          tc::TcEpiF32 ei{nullptr, pre, 4 * Hp, 0};
          rc = l == 0 ? tc_gemm(ts.enc_in, 0, enc_rows_, m.p_enc_w[0], np * n, 4 * Hp, Hp, ei, 0, 0, p0 * n)
                      : tc_gemm(ts.enc_seq[l - 1], 0, enc_rows_ + tc::kRowsMax, m.p_enc_w[l], np * n, 4 * Hp, Hp, ei, 0, 0, (p0 + 1) * n);
          if (rc == LINMT_OK) rc = encode_positions(mi, l, n, c0 + p0, np, pre, p0);
          stream = main_stream;
          ws_part_ = 0; ws_parts_ = 1; plan_parts_ = 0;
          CK(cudaEventRecord(enc_events_[l][0], enc_streams_[l]));
        }
      }
      for (int l = 0; l < L; ++l) CK(cudaStreamWaitEvent(main_stream, enc_events_[l][0], 0));
      if (rc != LINMT_OK) return rc;
      if (att_fold_) {      // W_c1 applied to the encoder states, once (see AttFold in step_kernels.cuh)
        tc::Planes top = ts.enc_seq[L - 1];       // (past block 0; a row offset would keep the product off CTA pairs)
        for (int t = 0; t < nt_; ++t) top.p[t] += (size_t)n * Hp;
        tc::TcEpiF32 e{nullptr, s.hs_wc1 + (size_t)c0 * n * Hp, Hp, 0};
        if ((rc = tc_gemm(top, 0, enc_rows_, m.p_att_out_w, len * n, Hp, Hp, e))) return rc;
      }
    }
  }
  return LINMT_OK;
}

// One member, in chunks of `per` positions.
int Engine::encode_member_layers(int mi, int n, int Smax, int per) {
  DevModel& m = models_[mi];
  DevState& s = states_[mi];
  TcState& ts = tc_states_[mi];
  for (int l = 0; l < L; ++l) {
    CK(cudaMemsetAsync(s.enc_c[0][l], 0, sizeof(float) * (size_t)n * Hp, stream));
    for (int t = 0; t < nt_; ++t) CK(cudaMemsetAsync(ts.enc_seq[l].p[t], 0, sizeof(uint16_t) * (size_t)n * Hp, stream));
  }
  for (int p0 = 0; p0 < Smax; p0 += per) {
    const int np = std::min(per, Smax - p0);
    enc_embed_seq_kernel<<<dim3(n, np, nt_), 128, 0, stream>>>(cur_ids_, d_off_, d_len_, m.p_emb_src, desc.vocab_src, ts.enc_in, Hp, p0);
    LAUNCHED();
    for (int l = 0; l < L; ++l) {
      const tc::Planes& seq = ts.enc_seq[l];
      if (p0 > 0)   // the state the previous chunk ended with
        for (int t = 0; t < nt_; ++t)
          CK(cudaMemcpyAsync(seq.p[t], seq.p[t] + (size_t)per * n * Hp, sizeof(uint16_t) * (size_t)n * Hp, cudaMemcpyDeviceToDevice, stream));
      tc::Planes in = l == 0 ? ts.enc_in : ts.enc_seq[l - 1];
      if (l > 0) for (int t = 0; t < nt_; ++t) in.p[t] += (size_t)n * Hp;
      tc::TcEpiF32 ei{nullptr, s.enc_pre, 4 * Hp, 0};
      if (int rc = tc_gemm(in, 0, enc_rows_, m.p_enc_w[l], np * n, 4 * Hp, Hp, ei)) return rc;
      if (int rc = encode_positions(mi, l, n, p0, np, s.enc_pre, 0)) return rc;
      if (l == L - 1 && att_fold_) {
        // W_c1 applied to the encoder states, once: the attention sums these rows (see AttFold in step_kernels.cuh)
        tc::Planes top = seq;
        for (int t = 0; t < nt_; ++t) top.p[t] += (size_t)n * Hp;
        tc::TcEpiF32 e{nullptr, s.hs_wc1 + (size_t)p0 * n * Hp, Hp, 0};
        if (int rc = tc_gemm(top, 0, enc_rows_, m.p_att_out_w, np * n, Hp, Hp, e)) return rc;
      }
    }
  }
  return LINMT_OK;
}

// One decoder forward, tensor-core path (see Engine::run_decoder_step).
int Engine::run_decoder_step_tc(int mi, int t, int rows, const ScoreStep* sc, int rows_next) {
  DevModel& m = models_[mi];
  DevState& s = states_[mi];
  TcState& ts = tc_states_[mi];
  const bool feed = desc.feed_input && t > 0;
  pdl_gemm_ = true;
  stream_weights_ = step_streams(sc != nullptr, rows);
  // scoring: one row per sentence continues itself, its tokens are given, and every step's htilde is kept
  const int kb = sc ? 1 : k;
  const int32_t* tok = sc ? sc->tok : d_tok_;
  const tc::Planes ht = sc ? sc->ht[mi] : ts.panel_ht;
  // Rows that continue themselves (one beam slot, scoring) need no copy of their states between two steps: there are two sets
  // of panels, and a step writes its states into the other set's h_prev and htilde_prev columns as well, while its own are
  // being read.  A launch less in a chain of eight to nine.
  const bool self = sc || self_rows();
  const int now = self ? t & 1 : 0, next = now ^ 1;
  const int32_t* parent = self ? nullptr : d_parent_;
  // The recurrent half of every layer's product was made behind the last step (recurrent_ahead); `next`'s first panel takes the
  // operand of the next one's.
  const bool have_rec = rec_ready_ && !sc, want_rec = rows_next > 0 && !sc;
  rec_ready_ = false;
  beside_ = have_rec;
  tc::Planes ht_next = no_planes();      // htilde_prev of the next step
  if ((self || want_rec) && desc.feed_input) {
    ht_next = ts.panel1[next];
    for (int p = 0; p < nt_; ++p) ht_next.p[p] += 2 * Hp;
  }
  // where h_cur of layer l lives after its GEMM: the input slot of the consumer panel
  auto hcur_planes = [&](int l) -> const tc::Planes& { return (l + 1 < L) ? ts.panel[now][l + 1] : ts.panel_top; };
  auto hcur_col0 = [&](int l) { return (l + 1 < L) ? 0 : Hp; };
  auto hprev_of = [&](int set, int l) -> const tc::Planes& { return l == 0 ? ts.panel1[set] : ts.panel[set][l]; };
  auto hprev_planes = [&](int l) -> const tc::Planes& { return hprev_of(now, l); };
  // 1. gather states through the parents into the h_prev slots, look up embeddings
  if (!have_rec) {
    GatherJobs jobs{};
    int nj = 0;
    auto add = [&](const void* src, long long sstride, void* dst, long long dstride, int bytes, int kind) {
      jobs.j[nj++] = GatherJob{static_cast<const unsigned char*>(src), sstride, static_cast<unsigned char*>(dst), dstride, bytes, kind};
    };
    const int fb = enc_final_buf_;
    for (int l = 0; l < L && !(self && t > 0); ++l) {
      for (int p = 0; p < nt_; ++p) {
        const __nv_bfloat16* src;
        long long sst;
        if (t == 0 && enc_final_row_ >= 0) { src = ts.enc_seq[l].p[p] + (size_t)enc_final_row_ * Hp; sst = (long long)Hp * 2; }
        else if (t == 0) { src = ts.encp[fb][l].p[p] + Hp; sst = (long long)ts.encp[fb][l].ld * 2; }
        else { src = hcur_planes(l).p[p] + hcur_col0(l); sst = (long long)hcur_planes(l).ld * 2; }
        add(src, sst, hprev_planes(l).p[p] + Hp, (long long)hprev_planes(l).ld * 2, Hp * 2, 0);
      }
      // the cell state is copied only at the first step (from the encoder); afterwards the LSTM epilogue
      // reads it through the parent index and the two buffers swap roles every step
      if (t == 0) add(s.enc_c[fb][l], (long long)Hp * 4, s.c_prev[l], (long long)Hp * 4, Hp * 4, 0);
    }
    if (feed && !self)
      for (int p = 0; p < nt_; ++p)
        add(ts.panel_ht.p[p], (long long)ts.panel_ht.ld * 2, ts.panel1[0].p[p] + 2 * Hp, (long long)ts.panel1[0].ld * 2, Hp * 2, 0);
    if (!m.dec_xw)   // with the input-term table the embedding never enters the GEMM
      for (int p = 0; p < nt_; ++p)
        add(m.p_emb_tgt.p[p], (long long)m.p_emb_tgt.ld * 2, ts.panel1[now].p[p], (long long)ts.panel1[now].ld * 2, Hp * 2, 1);
    jobs.n = nj;
    if (nj > 0) {
      dim3 grid(rows, (nj + kGatherJobsPerBlock - 1) / kGatherJobsPerBlock);
      if (int rc = kt(KC_GATHER)) return rc;
      CK(tc::launch_k(pdl_, row_gather_kernel, grid, dim3(128), 0, stream, jobs, parent, tok, V, kb, t == 0 ? 1 : 0));
      LAUNCHED();
    }
  }
  // 2. LSTM stack
  for (int l = 0; l < L; ++l) {
    if (int rc = kt(KC_LSTM)) return rc;
    tc::TcEpiLstm e{};
    e.bias = m.dec_b[l]; e.ldc = Hp;
    if (t == 0) { e.c_prev = s.c_prev[l]; e.c_out = s.c_cur[l]; }
    else {
      e.c_prev = (t & 1) ? s.c_cur[l] : s.c_prev[l];
      e.c_out = (t & 1) ? s.c_prev[l] : s.c_cur[l];
      e.c_parent = parent; e.c_k = kb;
    }
    e.h_out1 = hcur_planes(l); e.h1_col0 = hcur_col0(l);
    e.h_out2 = self || (want_rec && l == 0) ? hprev_of(next, l) : no_planes(); e.h2_col0 = Hp;
    e.h_prev = no_planes(); e.hp_col0 = 0;
    e.h_f32 = (l == L - 1 && opt.attention_mode == LINMT_ATT_GLOBAL_DOT) ? s.h_cur[l] : nullptr;
    e.hf_row_stride = Hp;
    e.row_len = nullptr; e.pos = 0; e.nt = nt_;
    int K = (l == 0 && feed) ? 3 * Hp : 2 * Hp;
    int rc;
    if (have_rec && l == 0) {
      e.xw = m.dec_xw; e.x_tok = tok; e.x_ld = 4 * Hp; e.x_vocab = V; e.x_unk = kUnk;
      const float *pre = s.rec, *fed = desc.feed_input ? s.rec + (size_t)kRecFeed * rec_rows_ * 4 * Hp : nullptr;
      CK(tc::launch_k(pdl_, lstm_cell_kernel, dim3(rows, (Hp + 127) / 128), dim3(128), 0, stream, e, pre, fed, Hp));
      LAUNCHED();
      rc = LINMT_OK;
    } else if (have_rec) {
      e.xw = s.rec + (size_t)rec_slot(l) * rec_rows_ * 4 * Hp; e.x_ld = 4 * Hp; e.x_parent = true;
      rc = tc_gemm(hprev_planes(l), 0, R, m.p_dec_w[l], rows, 4 * Hp, Hp, e);
    } else if (l == 0 && m.dec_xw) {
      // K columns (h_prev | htilde_prev) only: the x columns of panel and weights are skipped, their term comes from the table
      tc::Planes wrest = m.p_dec_w[0];
      for (int p = 0; p < 3; ++p) if (wrest.p[p]) wrest.p[p] += Hp;
      e.xw = m.dec_xw; e.x_tok = tok; e.x_ld = 4 * Hp; e.x_vocab = V; e.x_unk = kUnk;
      K -= Hp;
      rc = tc_gemm(hprev_planes(0), Hp, R, wrest, rows, 4 * Hp, K, e);
    } else {
      rc = tc_gemm(hprev_planes(l), 0, R, m.p_dec_w[l], rows, 4 * Hp, K, e);
    }
    if (rc) return rc;
    if (kernel_timing) rec_flops_ += 2.0 * rows * 4.0 * H * (double)((have_rec ? (l > 0) : K / Hp) * H);
  }
  // 3. attention projections: tanh(W_p h) | W_a^T h
  if (int rc = kt(KC_PROJ)) return rc;
  got_late_ = false;
  want_late_ = want_rec && L > 2;
  const float* u_alt = (opt.attention_mode == LINMT_ATT_GLOBAL_DOT) ? s.h_cur[L - 1] : nullptr;
  if (att_merge_) {
    // ... | W_c2 h: the half of the attention output's pre-activation that needs h_top only (global dot
    // attention uses no projection, so only those rows run)
    const int n0 = (opt.attention_mode == LINMT_ATT_GLOBAL_DOT) ? 2 * Hp : 0;
    tc::Planes w = m.p_att_proj_w;
    for (int p = 0; p < 3; ++p) if (w.p[p]) w.p[p] += (size_t)n0 * w.ld;
    tc::TcEpiF32 e{nullptr, s.proj + n0, 3 * Hp, n0 ? 0 : Hp};
    int rc = tc_gemm(ts.panel_top, Hp, R, w, rows, 3 * Hp - n0, Hp, e);
    if (rc) return rc;
  } else if (opt.attention_mode != LINMT_ATT_GLOBAL_DOT) {
    tc::TcEpiF32 e{nullptr, s.proj, 2 * Hp, Hp};
    int rc = tc_gemm(ts.panel_top, Hp, R, m.p_att_proj_w, rows, 2 * Hp, Hp, e);
    if (rc) return rc;
  }
  want_late_ = false;
  // 4. scores, softmax x Gaussian, context (written into the attention-output panel)
  {
    const bool rec = d_rec_align_ && !sc;
    float* ra = rec ? d_rec_align_ + (size_t)t * R * rec_win : nullptr;
    int32_t* rl = rec ? d_rec_lo_ + (size_t)t * R : nullptr;
    int32_t* rv = rec ? d_rec_vit_ + (size_t)t * R : nullptr;
    if (int rc = kt(KC_ATTENTION)) return rc;
    if (int rc = launch_attention(mi, t, rows, kb, u_alt, nullptr, att_fold_ ? ht : ts.panel_top, nt_, ra, rl, rv, att_fold_, att_fold_ ? ht_next : no_planes())) return rc;
    if (want_rec)
      if (int rc = recurrent_ahead(Ahead::kBetween, mi, t, rows_next)) return rc;
  }
  // 5. htilde = tanh(W_c1 ctx + W_c2 h + b) (with the fold the attention kernel has written it already)
  if (!att_fold_) {
    tc::TcEpiBiasTanh e{m.att_bout, ht, 0, nt_};
    e.out2 = ht_next;
    if (int rc0 = kt(KC_ATTOUT)) return rc0;
    int rc;
    if (att_merge_) {
      // W_c1 ctx over the first Hp of the K columns; W_c2 h comes in as a precomputed row
      e.add = s.proj + 2 * Hp; e.ld_add = 3 * Hp;
      rc = tc_gemm(ts.panel_top, 0, R, m.p_att_out_w, rows, Hp, Hp, e);
    } else {
      rc = tc_gemm(ts.panel_top, 0, R, m.p_att_out_w, rows, Hp, 2 * Hp, e);
    }
    if (rc) return rc;
  }
  beside_ = false;
  // 6. logits
  if (sc) return LINMT_OK;
  if (int rc = kt(KC_VOCAB)) return rc;
  return vocab_gemm(mi, ts.panel_ht, R, rows, s.logits, s.logits16, d_pmax_ + (size_t)mi * R * pmax_ld_, d_psum_ + (size_t)mi * R * pmax_ld_);
}

// The recurrent halves of the next step's LSTM products, W_h . h of every layer (and W_feed . htilde of the first), of the rows
// as they are: which row continues which is not needed for them, only for their sum with the rest, whose epilogue reads the
// parent's row.  With few rows a step is a chain of launches that wait for each other, and the weights' stream stands still
// while the attention, the softmax and the selection run on a few SMs; these products run beside them, those of the layers
// between beside the attention, the rest beside the softmax.  What is left of the chain is half a product a layer, none of the
// first (lstm_cell_kernel adds up its terms), and no state is gathered.  48 steps, ms a call without / with: 4 x 1000 / 30k 1 row
// 3.92 / 3.81, 12 rows 4.74 / 4.02, 24 4.88 / 4.34; 2 x 1000 12 rows 3.55 / 3.08, 48 3.69 / 3.46;
// 3 x 250 / 5k 12 rows 2.50 / 2.36.  (Up to how many rows: init_state.)
//
// They start without a wait for the kernel before them in the stream (RowsShape::ahead).  Before the attention that is where the
// projections have let the attention start only behind their own wait, and it these products: the layers' states are complete.
// Before the softmax, where that has let them start only behind its wait: all of the step is.  (The LATE instances; got_late_ says
// whether the launch was one of them.)  At their end they do wait, for those who wait for them.
bool Engine::ahead_ok(int rows) const {
  tc::RowsShape sh;
  return rows > 0 && rows <= rec_rows_ && tc::make_shape_ahead(rows, 4 * Hp, Hp, n_sm_, 1, &sh);   // (more products: fewer slices each, see there)
}

int Engine::recurrent_ahead(Ahead which, int mi, int t, int rows) {
  DevModel& m = models_[mi];
  DevState& s = states_[mi];
  TcState& ts = tc_states_[mi];
  const int now = self_rows() ? t & 1 : 0, next = now ^ 1;     // the sets of panels, see run_decoder_step_tc
  constexpr int kSegs = 3;      // (at most five layers)
  struct Part { tc::Planes a; int a_col0, layer, w_col0; } part[kSegs];
  int segs = 0, slot = 0;
  if (which == Ahead::kBetween) {
    slot = rec_slot(1);
    for (int l = 1; l + 1 < L; ++l) part[segs++] = Part{ts.panel[now][l + 1], 0, l, Hp};
  } else {
    part[segs++] = Part{ts.panel1[next], Hp, 0, Hp};
    part[segs++] = Part{ts.panel_top, Hp, L - 1, Hp};
    if (desc.feed_input) part[segs++] = Part{ts.panel1[next], 2 * Hp, 0, 2 * Hp};
  }
  if (segs == 0) return LINMT_OK;
  tc::RowsShape sh;
  if (!tc::make_shape_ahead(rows, 4 * Hp, Hp, n_sm_, segs, &sh)) return fail(LINMT_EINVAL, "internal: no shape for the recurrent products");
  sh.pdl = pdl_ ? 1 : 0;
  sh.ahead = pdl_ && got_late_ ? 1 : 0;
  tc::TmapSets<kSegs> tms{};
  for (int i = 0; i < segs; ++i) {
    tc::Planes w = m.p_dec_w[part[i].layer];
    for (int p = 0; p < nt_; ++p) w.p[p] += part[i].w_col0;
    const CUtensorMap* am = maps(part[i].a, part[i].a_col0, R, Hp, sh.rp, 64);
    const CUtensorMap* bm = maps(w, 0, 4 * Hp, Hp, tc::BM, 64);
    if (!am || !bm) return fail(LINMT_ECUDA, "cuTensorMapEncodeTiled failed");
    std::memcpy(tms.s[i].a, am, sizeof(tms.s[i].a));
    std::memcpy(tms.s[i].b, bm, sizeof(tms.s[i].b));
    tms.s[i].stream_b = stream_weights_;
  }
  const size_t stride = (size_t)rec_rows_ * 4 * Hp;
  const tc::TcEpiParts e{s.rec + slot * stride, (long long)stride, 4 * Hp};
  if (int rc = kt(KC_LSTM)) return rc;
  if (kernel_timing) rec_flops_ += 2.0 * rows * 4.0 * H * (double)(segs * H);
  CK((tc::launch_gemm_tc_rows_of<2, 1, tc::TcEpiParts, kSegs, false>(tms, segs, rows, 4 * Hp, Hp, sh, e, d_tc_err_, stream, 0)));
  LAUNCHED();
  return LINMT_OK;
}

// Logits of `rows` attentional states.
int Engine::vocab_gemm(int mi, const tc::Planes& ht, int rows_cap, int rows, float* logits, __half* logits16, float* pmax, float* psum) {
  DevModel& m = models_[mi];
  tc::TcEpiF32 e{m.voc_b, logits, Vp, 0};
  if (logits16_) e.out16 = logits16;   // the softmax of this step is their only reader
  blocks_ = LogitBlocks{};
  if (pmax_on_ && pmax) { e.pmax = pmax; e.psum = psum; e.pmax_ld = pmax_ld_; e.n_valid = V; }
  // Logits feed only the softmax of their own step: the tensor core's truncation bias over one
  // K = Hp chain (~32 ulp of the accumulator, 2e-7 relative on a log-probability) does not
  // accumulate over steps as it does through the recurrent products, so this GEMM runs its
  // leading product as one chain (no intermediate drains: 5 % faster).
  return tc_gemm(ht, 0, rows_cap, m.p_voc_w, rows, Vp, Hp, e, nt_vocab_, Hp / 32);
}

// Scores of given targets, tensor-core path: one device batch of n sentences, longest target first.  Nothing of a step
// depends on the step's logits, so only the recurrence runs step by step, on ONE row per sentence (a forced decode ran a
// row per beam slot), and the vocabulary product, its softmax and the given tokens' log-probabilities follow for all
// positions together.
//   n_act[t] sentences run step t; d_tok [steps][n] the tokens read (START first); d_gold / d_logp the tokens asked for
//   (EOS last) and their log-probabilities, packed: the first n_act[t] sentences of step 0, of step 1, ...
int Engine::score_core_tc(int n, int Smax, const std::vector<int>& n_act, const int32_t* d_tok, const int32_t* d_gold, float* d_logp) {
  const int steps = (int)n_act.size();
  size_t rows_all = 0;
  for (int a : n_act) rows_all += a;
  if (int rc = reserve_score(rows_all)) return rc;
  if (int rc = run_encoder_tc(n, Smax)) return rc;
  enc_final_buf_ = Smax & 1;
  std::vector<tc::Planes> cur = score_ht_;
  size_t row = 0;
  for (int t = 0; t < steps; ++t) {
    for (int mi = 0; mi < n_models; ++mi)
      for (int p = 0; p < nt_; ++p) cur[mi].p[p] = score_ht_[mi].p[p] + row * Hp;
    const ScoreStep sc{d_tok + (size_t)t * n, cur.data()};
    if (int rc = each_member(n_act[t], [&](int mi) { return run_decoder_step_tc(mi, t, n_act[t], &sc); })) return rc;
    row += n_act[t];
    stats.decoder_row_steps += n_act[t];
    stats.sentence_steps += n_act[t];
  }
  stream_weights_ = step_streams(false, 0);
  for (size_t r0 = 0; r0 < rows_all; r0 += score_q_) {
    const int rows = (int)std::min<size_t>(score_q_, rows_all - r0);
    TopkOut o{score_idx_, score_candp_, score_eos_, score_stats_};
    TopkRefine rf{};
    for (int mi = 0; mi < n_models; ++mi) {
      tc::Planes a = score_ht_[mi];
      for (int p = 0; p < nt_; ++p) a.p[p] += r0 * Hp;
      if (mi == 0 && refine_) rf = refinement(a);
      if (int rc = vocab_gemm(mi, a, (int)std::min<size_t>(score_q_, score_rows_ - r0), rows, score_logits_[mi], score_logits16_, n_models == 1 ? score_pmax_ : nullptr, score_psum_)) return rc;
    }
    const float* logits = score_logits_[0];
    int normalise = 1;
    if (n_models > 1) {
      EnsembleRows er{};
      for (int mi = 0; mi < n_models; ++mi) er.logits[mi] = score_logits_[mi];
      er.n = n_models;
      CK(tc::launch_k(pdl_, ensemble_combine_kernel, dim3(rows), dim3(256), 0, stream, er, Vp, V, (int)opt.ensemble_mode, score_combined_));
      LAUNCHED();
      logits = score_combined_;
      normalise = opt.ensemble_mode == LINMT_ENS_PROB_MEAN ? 1 : 0;
    }
    CK(softmax_topk(logits, score_logits16_, rows, o, normalise, refine_ ? &rf : nullptr, SelectArgs{}));
    LAUNCHED();
    CK(tc::launch_k(pdl_, gold_logp_kernel, dim3((rows + 7) / 8), dim3(256), 0, stream, d_gold + r0, rows, logits, Vp, V, (const float*)score_stats_, rf, d_logp + r0));
    LAUNCHED();
  }
  return LINMT_OK;
}

// Workspace of score_core_tc, kept between calls: attentional states of every position, and logits of as many rows at a
// time as 64 Mi values hold.
int Engine::reserve_score(size_t rows) {
  int rc;
  if (rows > score_rows_) {
    for (auto& p : score_ht_)
      for (int t = 0; t < nt_; ++t) release(p.p[t]);
    tmap_cache_.clear();      // (maps of the released panels)
    score_rows_ = 0;
    score_ht_.assign(n_models, tc::Planes{});
    for (int mi = 0; mi < n_models; ++mi)
      if ((rc = alloc_planes(score_ht_[mi], rows, Hp))) return rc;
    score_rows_ = rows;
  }
  if (score_q_) return LINMT_OK;
  const size_t cap = std::max<size_t>(128, (((size_t)64 << 20) / Vp) & ~(size_t)127);
  // (one request for all parts)
  size_t at = 0;
  auto part = [&](bool wanted, size_t bytes) {
    const size_t here = at;
    if (wanted) at += (bytes + kMemoryUnit - 1) / kMemoryUnit * kMemoryUnit;
    return here;
  };
  const size_t logits16 = part(logits16_, cap * Vp * 2), logits = part(!logits16_, (size_t)n_models * cap * Vp * 4),
               combined = part(n_models > 1, cap * Vp * 4), idx = part(true, cap * kk * 4), candp = part(true, cap * kk * 4), eos = part(true, cap * 4), statistics = part(true, cap * 8),
               pmax = part(true, cap * pmax_ld_ * 4), psum = part(true, cap * pmax_ld_ * 4);
  char* ws = nullptr;
  if ((rc = dalloc_bytes(&ws, at))) return rc;
  auto floats = [&](size_t offset) { return reinterpret_cast<float*>(ws + offset); };
  score_logits_.assign(n_models, nullptr);
  if (logits16_) score_logits16_ = reinterpret_cast<__half*>(ws + logits16);
  else
    for (int mi = 0; mi < n_models; ++mi) score_logits_[mi] = floats(logits) + (size_t)mi * cap * Vp;
  if (n_models > 1) score_combined_ = floats(combined);
  score_idx_ = reinterpret_cast<int32_t*>(ws + idx);
  score_candp_ = floats(candp); score_eos_ = floats(eos); score_stats_ = floats(statistics); score_pmax_ = floats(pmax); score_psum_ = floats(psum);
  score_q_ = (int)cap;
  return LINMT_OK;
}

}  // namespace linmt
