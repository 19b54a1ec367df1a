// engine.h -- the decoding engine behind the C ABI (host side, C++).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>
#include <vector>

#include "../../include/linmt_decoder.h"
#include "encoder_form.h"
#include "step_kernels.cuh"
#include "gemm_tc.cuh"
#include <array>
#include <functional>
#include <map>
#include <memory>
#include <tuple>

namespace linmt {

inline int round_up(int x, int m) { return (x + m - 1) / m * m; }

// Packed weights of one ensemble member in device memory.  Every dense operand is stored
// K-major ("[out][in]", in padded to Hp) so both GEMM operands are K-contiguous.
struct DevModel {
  float* emb_src = nullptr;              // [Vs][Hp]
  float* emb_tgt = nullptr;              // [V][Hp]
  std::vector<float*> enc_w, enc_b;      // [4Hp][2Hp], [4Hp]   gate-interleaved rows 4j+g
  std::vector<float*> dec_w, dec_b;      // layer 0: [4Hp][3Hp] (x | h' | htilde'), others [4Hp][2Hp]
  std::vector<int> dec_ldw;
  float* att_proj_w = nullptr;           // [2Hp][Hp]: rows < Hp = W_p, rows >= Hp = W_a^T (tensor path: [3Hp][Hp], rows >= 2Hp = W_c2)
  float* att_out_w = nullptr;            // [Hp][2Hp]: (ctx | h_top)
  float* att_bout = nullptr;             // [Hp]
  float* vp = nullptr;                   // [Hp]
  float* voc_w = nullptr;                // [Vp][Hp]
  float* voc_b = nullptr;                // [Vp]
  float* dec_xw = nullptr;               // [V][4Hp] W_x . embedding(v) of the first decoder layer (tensor path, optional)
  float voc_wnorm_max = 0.f;             // largest 2-norm of a vocabulary weight row
  float voc_babs_max = 0.f;              // largest magnitude of a vocabulary bias
  // the same operands as bf16 planes for the tensor-core path (fp32 copies are then not kept)
  tc::Planes p_emb_src{}, p_emb_tgt{}, p_att_proj_w{}, p_att_out_w{}, p_voc_w{};
  std::vector<tc::Planes> p_enc_w, p_dec_w;
};

// Activation panels of the tensor-core path: every GEMM reads ONE K-contiguous panel, so the
// producers write straight into the column range of the panel that consumes them.
struct TcState {
  // (two of each: rows that continue themselves take turns, see run_decoder_step_tc)
  tc::Planes panel1[2];              // [R][3Hp]  x | h_prev(layer 0) | htilde_prev
  std::vector<tc::Planes> panel[2];  // l = 1..L-1: [R][2Hp]  h_cur(l-1) | h_prev(l)
  tc::Planes panel_top{};            // [R][2Hp]  ctx | h_cur(L-1)
  tc::Planes panel_ht{};             // [R][Hp]   htilde
  tc::Planes hs_planes{};            // [B * max_src][Hp]  the encoder's top states as operand planes (attention fold)
  std::vector<tc::Planes> encp[2];   // [L] x [B][2Hp]  below | h_prev, double buffered over positions
  // encoder layer by layer (few sentences): block p of n rows = the state after p positions of the chunk
  tc::Planes enc_in{};               // [rows][Hp] the first layer's input
  std::vector<tc::Planes> enc_seq;   // [L] x [rows + n][Hp]
};

struct DevState {
  float* x = nullptr;                        // [R][Hp]
  std::vector<float*> h_cur, c_cur, h_prev, c_prev;  // [L] x [R][Hp]
  float *htilde = nullptr, *htilde_prev = nullptr;   // [R][Hp]
  float *proj = nullptr, *ctx = nullptr;             // [R][2Hp or 3Hp], [R][Hp]
  float* logits = nullptr;                           // [R][Vp]
  __half* logits16 = nullptr;                        // [R][Vp]  the same in fp16 (one-product logits whose candidates are recomputed)
  float* hs = nullptr;                               // [B][max_src][Hp]
  tc::Planes hs16{};                                 // the same in bf16 (one plane: instead of hs)
  float* hs_wc1 = nullptr;                           // [B][max_src][Hp]  W_c1 . hs (tensor path with the attention fold)
  // [L + 1][rec_rows_][4Hp]  recurrent products of the step before, by its rows (Engine::recurrent_ahead), in the order of rec_slot
  float* rec = nullptr;
  float* enc_x = nullptr;                            // [B][Hp]
  float* enc_pre = nullptr;                          // [rows][4Hp]  W_x . input of every position (encoder layer by layer)
  std::vector<float*> enc_h[2], enc_c[2];            // [L] x [B][Hp], double buffered
};

// A call of the CUDA runtime in an Engine's method, which returns where it fails.
#define CK(call)                                                             \
  do {                                                                       \
    const cudaError_t e_ = (call);                                           \
    if (e_ != cudaSuccess) return cuda_failed(e_, __FILE__, __LINE__);       \
  } while (0)

// Kernel classes of a decoder step, in launch order (linmt_kernel_times reports one entry per class).
enum KernelClass { KC_GATHER = 0, KC_LSTM, KC_PROJ, KC_ATTENTION, KC_ATTOUT, KC_VOCAB, KC_COMBINE, KC_SOFTMAX, KC_SELECT, KC_COUNT, KC_END = KC_COUNT };

class Engine {
 public:
  float class_ms[KC_COUNT] = {};      // device time per kernel class in the last timed decode
  int class_launches[KC_COUNT] = {};
  Engine() = default;
  ~Engine();
  int init(const linmt_model_desc& d, const float* const* blobs, int n_models, size_t blob_floats, const linmt_options& o);
  // A lane: an engine on the device of `of` with its weights, which it must not outlive, and state, stream and workspaces of its own.
  // Those are made by `ready`, in the thread that is going to use them; one that could not be is `broken` and of no use.
  explicit Engine(const Engine* of) : lane_of_(of), broken_(true) { opt = of->opt; }
  int ready();
  // After an exception or an error in the middle of a call: waits for what is under way, and the engine is as between two calls.
  void recover();
  // Runs `call`; an exception is its error (for host memory).
  int guarded(const std::function<int()>& call);
  bool planned() const { return lane_of_ != nullptr; }
  bool broken() const { return broken_ && !lane_of_; }
  // While one lives, the engine's device batch is one of a call's that run at once on a device, and its products leave room for others.
  // That goes by the engines that the call has, not by what runs at the moment: a sentence's last bits do not depend on time.  (Not in one
  // plane: in other shapes the sums are in another order, which rounds a state to the other bf16 neighbour now and then.  A
  // sentence has the bits there that it has in a batch by itself.)
  struct Several {
    Engine& g;
    Several(Engine& e, bool on) : g(e) { g.several_ = on && g.nt_ > 1; }
    ~Several() { g.several_ = false; }
  };
  // Device batches of a call that are worth running at once, of this engine's `rows` each.
  int lanes_for(int rows) const;
  // Whether the device can spare what so many lanes take: a quarter of its free memory at most, for calls grow an engine's buffers and
  // others use the device as well.
  bool room_for_lanes(int n) const;
  int decode_core(const int32_t* d_ids, const int32_t* off_host, int n, const int32_t* steps_host, int max_len,
                  int32_t* d_out_tok, int32_t* d_out_len, float* d_out_score, int32_t* d_out_vit, float* d_out_align,
                  const linmt_trace* trace_dev, int trace_Tm);
  int finish_timing();
  // a decode call's arrays (linmt_decode_batch)
  struct HostJob {
    const int32_t *src_ids, *src_off, *steps; int max_len;
    int32_t *out_tok, *out_len; float* out_score; int32_t* out_vit; float* out_align;
  };
  int decode_chunk(const HostJob& jb, const int* idx, int cn, const linmt_trace* trace_dev, int Tm_all);
  // a scoring call's arrays (linmt_score_batch), and one device batch of it: sentences idx[0..cn), longest target first
  struct ScoreJob {
    const int32_t *src_ids, *src_off, *tgt_ids, *tgt_off;
    float *out_logprob, *out_token_logp; int max_tgt;
  };
  int score_chunk(const ScoreJob& jb, const int* idx, int cn);
  bool scores_rows() const { return use_tc_; }    // (the CUDA-core path scores through a forced decode)
  int decode_host(const int32_t* src_ids, const int32_t* src_off, int n, const int32_t* steps, int max_len,
                  int32_t* out_tok, int32_t* out_len, float* out_score, int32_t* out_vit, float* out_align,
                  const linmt_trace* trace);

  std::string err;
  linmt_model_desc desc{};
  linmt_options opt{};
  int k = 0, kk = 0, H = 0, Hp = 0, V = 0, Vp = 0, L = 0, B = 0, R = 0, win = 0, rec_win = 0, Tcap = 0, fin_cap = 0;
  int n_models = 0;
  cudaStream_t stream = nullptr;
  linmt_stats stats{};
  bool kernel_timing = false;

  // sentence front-end (filled by the config-file constructor)
  std::vector<std::string> tgt_words;
  std::vector<std::pair<std::string, int>> src_words_sorted;
  int longest_sentence = 0;
  int print_align_scores = 0;
  int src_unk_id = 0;   // id unknown source words read: the source map's "UNK" entry, 0 when it has none
  std::string result_buf;

 private:
  int init_lane(const Engine& of);
  int init_state(const Engine* of, const float* const* blobs);
  const Engine* lane_of_ = nullptr;      // a lane that is not made yet
  bool broken_ = false;
  int fail(int code, const std::string& msg) { err = msg; return code; }
  int cuda_failed(cudaError_t e, const char* file, int line);
  // role of member mi in the alignment record of a step: 0 = single model, 1 / 2 / 3 = first / middle / last member
  int ens_member_code(int mi) const { return n_models == 1 ? 0 : (mi == 0 ? 1 : (mi == n_models - 1 ? 3 : 2)); }
  int pack_model(const float* blob, DevModel& m);
  int alloc_state(DevState& s);
  // one plane: the encoder's states are rounded to bf16, and kept as that (a sentence's, numbered in 32 bits)
  bool states16() const { return use_tc_ && nt_ == 1 && (long long)opt.max_src_len * Hp < (1ll << 31); }
  int run_encoder(int n, int Smax);
  int run_decoder_step(int mi, int t, int rows);
  int run_encoder_tc(int n, int Smax);
  int run_encoder_layers_tc(int n, int Smax);   // few sentences: layer by layer
  int encode_member_layers(int mi, int n, int Smax, int per);
  int run_encoder_pipeline_tc(int n, int Smax, bool few);   // more sentences: the layers side by side, a few positions behind each other
  int encoder_streams();
  int encode_positions(int mi, int l, int n, int pos0, int np, float* pre, int block);
  int each_member(int rows, const std::function<int(int)>& work);
  // a step of scoring: the tokens read, and where every member's htilde goes
  struct ScoreStep { const int32_t* tok; const tc::Planes* ht; };
  int run_decoder_step_tc(int mi, int t, int rows, const ScoreStep* sc = nullptr, int rows_next = 0);
  bool ahead_ok(int rows) const;
  enum class Ahead { kBetween, kEnds };      // which of the recurrent products: the layers' between first and last, those two's
  // where they are in DevState::rec: the first layer's states, the last one's, the first layer's feed-input, the layers between
  static constexpr int kRowsAheadSelf = 32, kRowsAheadWide = 48;      // (see init_state; kRowsAhead otherwise)
  static constexpr size_t kWideLayers = (size_t)2 << 20;              // layers x units x units
  static constexpr int kRecFeed = 2;
  int rec_slot(int l) const { return l == 0 ? 0 : l == L - 1 ? 1 : l + 2; }
  int recurrent_ahead(Ahead which, int mi, int t, int rows);
  // rows that continue themselves: one beam slot (scoring aside)
  bool self_rows() const { return k == 1 && !trace_dev_.force_tok; }
  int vocab_gemm(int mi, const tc::Planes& ht, int rows_cap, int rows, float* logits, __half* logits16, float* pmax, float* psum);
  cudaError_t softmax_topk(const float* logits, const __half* logits16, int rows, const TopkOut& o, int normalise, const TopkRefine* rf, const SelectArgs& sel,
                           bool late = false);
  int score_core_tc(int n, int Smax, const std::vector<int>& n_act, const int32_t* d_tok, const int32_t* d_gold, float* d_logp);
  int reserve_score(size_t rows);
  TopkRefine refinement(const tc::Planes& ht) const;    // of one-product logits of these attentional states
  int step_tail(int t, int rows, bool ahead);
  bool step_streams(bool scoring, int rows) const;
  bool pairs_available();   // clusters of two GEMM CTAs can be scheduled on the current device (engine_tc.cu)
  int launch_attention(int mi, int t, int rows, int kb, const float* u_alt, float* ctx, const tc::Planes& ctx_planes, int nt,
                       float* rec_align, int32_t* rec_lo, int32_t* rec_vit, bool fold = false, const tc::Planes& ctx2 = tc::Planes{});
  int alloc_state_tc(TcState& s);
  int build_xw_tables();   // dec_xw of every model (tensor path, xw_table_)
  int alloc_planes(tc::Planes& p, size_t rows, int ld);
  int to_planes(const std::vector<float>& host, size_t rows, int ld, tc::Planes& dst);
  const CUtensorMap* maps(const tc::Planes& p, int col0, int rows, int K, int box_rows, int bk);
  template <class Epi>
  int tc_gemm(const tc::Planes& A, int a_col0, int a_rows_cap, const tc::Planes& W, int M, int N, int K, const Epi& e, int nt = 0, int drain = 0, int x_row0 = 0);

  bool use_tc_ = false;
  cudaStream_t main_stream_ = nullptr;     // `stream`, but for a layer's or a member's work
  // encoder wavefront: one stream per layer, a small ring of events per layer
  std::vector<cudaStream_t> enc_streams_;
  std::vector<std::vector<cudaEvent_t>> enc_events_;
  cudaEvent_t enc_start_ev_ = nullptr;
  int nt_ = 3;
  bool pdl_ = false;  // decoder-step kernels launched with programmatic stream serialization (tensor path)
  bool xw_table_ = false;  // first decoder layer: embedding term from a per-vocabulary table instead of the GEMM
  bool refine_ = false;    // one-product vocabulary GEMM + accurate recomputation of the candidates in the softmax kernel
  bool logits16_ = false;  // one-product logits stored as fp16 (only with the accurate recomputation of the candidates; LINMT_LOGITS16=0: test knob)
  bool att_fold_ = false;  // tensor path: W_c1 applied to the encoder states once per batch, attention writes htilde (LINMT_ATT_FOLD=0: test knob)
  bool att_merge_ = false; // tensor path: W_c2 . h_top computed with the attention projections (LINMT_ATT_MERGE=0: test knob)
  bool pmax_on_ = true;    // vocabulary GEMM hands block maxima to the softmax (LINMT_PMAX=0: test knob)
  bool pair_ = true;       // CTA pairs for the GEMM shapes that are down to two stages (LINMT_TC_PAIR=0: test knob)
  bool stream_weights_ = false;  // the products issued are a step's (or scoring's vocabulary products), whose weights do not fit L2
  int l2_bytes_ = 0;
  bool rows_ = true;       // weight-streaming kernel for few rows (LINMT_TC_ROWS=0: test knob)
  bool ahead_ = true;      // recurrent products behind the step before (LINMT_AHEAD=0: test knob)
  bool several_ = false;   // see Several
  bool lanes_ = true;      // device batches of a call at once (LINMT_LANES=0: test knob)
  bool persist_ = true;    // persistent kernel for the many-wave vocabulary GEMM (LINMT_TC_PERSIST=0: test knob)
  bool beside_ = false;      // the products issued leave room for the next one's CTAs (GemmLimits::beside)
  bool want_late_ = false, got_late_ = false;   // the next product is asked to let its successor start only behind its wait; the last one asked does
  bool rec_ready_ = false;   // the last step's recurrent products are made (recurrent_ahead)
  int rec_rows_ = 0;         // rows they have room for
  bool pdl_gemm_ = false;  // true while the decoder step issues its GEMMs (the encoder's wavefront does not take part)
  int fmt_ = 0;       // plane format of every operand: 0 = bf16 planes, 1 = f16 pair
  int nt_vocab_ = 0;  // planes used by the vocabulary GEMM (0 = nt_)
  int n_sm_ = 148;
  int* d_tc_err_ = nullptr;
  float* d_splitk_ws_ = nullptr;      // split-K partial tiles
  int* d_splitk_counters_ = nullptr;  // one arrival counter per output tile
  static constexpr size_t kSplitKWsFloats = (size_t)16 << 20;  // 64 MiB
  // ensembles: a stream per member (see each_member)
  std::vector<cudaStream_t> mem_streams_;
  std::vector<cudaEvent_t> mem_events_;
  int plan_parts_ = 0;                // products that run side by side, for the choice of their shapes (0: ws_parts_)
  int ws_part_ = 0, ws_parts_ = 1;    // slice of the workspace a launch may use (concurrent encoder layers get one each)
  static constexpr int kSplitKMaxTiles = 4096;
  std::vector<TcState> tc_states_;
  std::map<std::tuple<const void*, int, int, int, int>, std::array<CUtensorMap, 3>> tmap_cache_;

  const int32_t* cur_ids_ = nullptr;
  // row of the encoder states of sentence b after position p: b * hs_sent_ + p * hs_pos_
  int hs_sent_ = 0, hs_pos_ = 1;
  int enc_rows_ = 0;                    // rows (positions x sentences) of the layers' panels (0: position by position only)
  int enc_final_row_ = -1;              // the final states in the panels: first row in enc_seq (-1: position by position)
  TraceDev trace_dev_{};
  size_t trace_pt_member_stride_ = 0;   // floats between two members' p_t records in the device trace buffer
  int enc_final_buf_ = 0;
  std::vector<DevModel> models_;
  std::vector<DevState> states_;
  std::vector<void*> allocs_;
  // device memory requested so far, in whole units; what the handle's creation took of it beside the weights
  static constexpr size_t kMemoryUnit = 512;
  size_t asked_bytes_ = 0, lane_bytes_ = 0;
  // A lane's creation takes all that in one request, and its buffers from there: a request costs 0.3 to 2 ms, whatever its size.
  char* arena_ = nullptr;
  size_t arena_used_ = 0, arena_bytes_ = 0;
  int device_memory(void** p, size_t bytes, const char* what);
  int host_memory(void** p, size_t bytes, const char* what);      // (pinned)
  template <class T> int dalloc(T** p, size_t count);
  template <class T> int regrow(T** p, size_t count, size_t* cap);

  // batch metadata (device) and pinned staging
  int32_t *d_off_ = nullptr, *d_len_ = nullptr, *d_steps_ = nullptr, *d_orig_ = nullptr;
  int32_t* h_meta_ = nullptr;  // pinned [4][B+1], then the error flag
  int32_t* h_err_ = nullptr;
  // beam state
  int32_t *d_tok_ = nullptr, *d_parent_ = nullptr, *d_hist_tok_ = nullptr, *d_hist_parent_ = nullptr;
  float* d_score_ = nullptr;
  int32_t *d_fin_t_ = nullptr, *d_fin_b_ = nullptr, *d_fin_n_ = nullptr;
  int32_t* d_rows_done_ = nullptr;   // per sentence: rows whose softmax of this step is done (SelectArgs)
  float *d_fin_score_ = nullptr, *d_fin_final_ = nullptr;
  float* d_combined_ = nullptr;  // [R][Vp] ensemble-combined log-values (n_models > 1)
  int32_t* d_cand_idx_ = nullptr;
  float *d_cand_logp_ = nullptr, *d_eos_logp_ = nullptr, *d_row_stats_ = nullptr;
  float* d_pmax_ = nullptr;   // [members][R][pmax_ld_] block maxima of the logits, by-product of the vocabulary GEMM ...
  float* d_psum_ = nullptr;   // ... and the blocks' sums of exp(z - maximum)
  int pmax_ld_ = 0;
  LogitBlocks blocks_{};      // what the last vocabulary GEMM left of them
  // alignment records (print_info)
  float* d_rec_align_ = nullptr;
  int32_t *d_rec_lo_ = nullptr, *d_rec_vit_ = nullptr;
  // host staging for decode_host
  int32_t* d_ids_ = nullptr;
  size_t d_ids_cap_ = 0;
  int32_t* d_out_ = nullptr;      // results of a device batch: len | score | tok | vit | align
  size_t out_cap_ = 0;
  int32_t* h_stage_ = nullptr;    // pinned: ids of a batch, then its results
  size_t h_stage_cap_ = 0;
  int reserve_host(size_t bytes);
  // scoring workspace, made at the first call and kept
  std::vector<tc::Planes> score_ht_;
  size_t score_rows_ = 0;
  int score_q_ = 0;
  std::vector<float*> score_logits_;
  __half* score_logits16_ = nullptr;
  float *score_combined_ = nullptr, *score_candp_ = nullptr, *score_eos_ = nullptr, *score_stats_ = nullptr, *score_pmax_ = nullptr, *score_psum_ = nullptr;
  int32_t *score_idx_ = nullptr, *score_io_ = nullptr;
  size_t score_io_cap_ = 0;
  template <class T> int dalloc_bytes(T** p, size_t bytes) {
    void* q = nullptr;
    if (int rc = device_memory(&q, bytes, "scoring workspace")) return rc;
    allocs_.push_back(q);
    *p = static_cast<T*>(q);
    return LINMT_OK;
  }
  // (buffers that are made when they are needed; those of the creation stay)
  void release(void* p) {
    for (auto it = allocs_.begin(); p && it != allocs_.end(); ++it)
      if (*it == p) { allocs_.erase(it); cudaFree(p); return; }
  }
  // trace buffers (device), sized on demand
  std::vector<void*> trace_allocs_;
  cudaEvent_t ev0_ = nullptr, ev1_ = nullptr;
  // kernel timing (off by default): an event before every kernel of the decoder steps, tagged with the kernel's
  // class; the time to the next event is booked to that class.  The events end the overlap of consecutive
  // kernels, so a timed decode is a measurement pass, not the number to report as throughput.
  std::vector<cudaEvent_t> kt_ev_;
  std::vector<int> kt_cls_;
  size_t kt_used_ = 0;
  double rec_flops_ = 0.0;
  int kt(int cls);
};

// host-side weight packing
void pack_gate_weights(const float* const* mats, int nseg, int H, int Hp, float* out /*[4Hp][nseg*Hp]*/);

}  // namespace linmt

// The opaque handle of the C ABI: the engine on the first device and, for a handle created on several
// devices, one replica of the same models per further device.  Sentences are independent, so a job is
// dealt to the devices in device batches, one host thread per device, with no traffic between them.
struct linmt_engine {
  linmt::Engine eng;
  std::vector<std::unique_ptr<linmt::Engine>> replicas;
  // Further engines on the devices above, with their weights: a call of several device batches runs some at once (Engine::lanes_for).
  // Made when such a call first wants them, beside the batches that it has begun with, and kept, unless memory is short (with_lanes).
  std::vector<std::unique_ptr<linmt::Engine>> lanes;
  bool no_more_lanes = false;
  // Runs `call`, which may use the lanes; where it fails for memory, which they hold some of or were refused, it runs once more from its
  // start without them, as every later one does.
  int with_lanes(const std::function<int()>& call);
  // the engines that share `items` device batches of `rows` rows, on the first device alone or on all
  std::vector<linmt::Engine*> workers(size_t items, int rows, bool first_device);
  int n_engines() const { return 1 + (int)replicas.size(); }
  linmt::Engine& engine(int i) { return i == 0 ? eng : *replicas[i - 1]; }
};

namespace linmt {
std::vector<int> batch_order(const int32_t* src_off, int n, const int32_t* steps);
// Runs work(engine, item) for item = order[0], order[1], ... on engines of a handle (linmt_engine::workers), one host thread per
// engine, each taking the next item when it is free.  Returns the first error; engine 0's `err` names it.
int run_on_engines(linmt_engine* h, const std::vector<Engine*>& workers, const std::vector<int>& order, const std::function<int(Engine&, int)>& work);
}  // namespace linmt
