// step_kernels.cuh -- the non-GEMM kernels of the decoding step loop: embedding gather and
// beam reorder, attention, log-softmax + per-beam top-(k+1), beam selection, finalisation.
// All beam state lives on the device; the host only launches.
#pragma once
#include <cuda_runtime.h>
#include <float.h>
#include <math.h>
#include <stdint.h>

#include "gemm_tc.cuh"

namespace linmt {

constexpr int kMaxBeam = 31;          // kk = beam + 1 <= 32, the lanes that a threshold is ranked on
constexpr int kStart = 0, kEos = 1, kUnk = 2;  // src/input_file_preprocess.cc:549-567
constexpr float kDeadScore = -1e30f;  // score of a hypothesis created when candidates run out

// ---------------------------------------------------------------------------------------
// Encoder input: x[b] = E_src[ids_rev[b][pos]] (SparseLookupKernel,
// src/deep_rnn_kernel.h:248-255); the sentence is read back to front
// (src/decoder_sentence.cu:68).  Rows past their length get zeros.
// grid = (B), block = 256
static __global__ void enc_embed_kernel(const int32_t* __restrict__ ids, const int32_t* __restrict__ off,
                                 const int32_t* __restrict__ len, const float* __restrict__ emb, int vocab,
                                 float* __restrict__ x, int Hp, int pos) {
  const int b = blockIdx.x;
  const int S = len[b];
  float4* dst = reinterpret_cast<float4*>(x + (size_t)b * Hp);
  if (pos < S) {
    int tok = ids[off[b] + (S - 1 - pos)];
    if (tok < 0 || tok >= vocab) tok = 0;  // out-of-range ids read <UNK> (src/decoder_sentence.cu:61-62)
    const float4* src = reinterpret_cast<const float4*>(emb + (size_t)tok * Hp);
    for (int i = threadIdx.x; i < Hp / 4; i += blockDim.x) dst[i] = src[i];
  } else {
    for (int i = threadIdx.x; i < Hp / 4; i += blockDim.x) dst[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

// ---------------------------------------------------------------------------------------
// Start of a decoder step: gathers every state row through the parent chosen by the last
// beam selection and looks up the new token's embedding.  Replaces SwapDecodingStates +
// TargetCopyPrevStates (src/deep_rnn.h:1842-1872, 2L(k+1)+k+2L cudaMemcpy calls) and the
// embedding lookup of src/node_input_to_hidden.h:243.  At step 0 the source rows are the
// encoder's final states, one per sentence (src/deep_rnn.h:1766-1789).
//   src[a], dst[a]: n_arr state arrays [rows][Hp]; src_per_sentence = 1 at step 0.
// grid = (rows, n_arr + 1), block = 256; blockIdx.y == n_arr is the embedding.
struct PrepArrays {
  const float* src[12];
  float* dst[12];
  int n_arr;
};
static __global__ void dec_prep_kernel(PrepArrays arr, const int32_t* __restrict__ parent, const int32_t* __restrict__ tok,
                                const float* __restrict__ emb, int vocab, float* __restrict__ x, int Hp, int k,
                                int src_per_sentence) {
  const int r = blockIdx.x;
  const int a = blockIdx.y;
  const float4* src;
  float4* dst;
  if (a == arr.n_arr) {
    int t = tok[r];
    if (t < 0 || t >= vocab) t = kUnk;
    src = reinterpret_cast<const float4*>(emb + (size_t)t * Hp);
    dst = reinterpret_cast<float4*>(x + (size_t)r * Hp);
  } else {
    const int sent = r / k;
    const int srow = src_per_sentence ? sent : sent * k + parent[r];
    src = reinterpret_cast<const float4*>(arr.src[a] + (size_t)srow * Hp);
    dst = reinterpret_cast<float4*>(arr.dst[a] + (size_t)r * Hp);
  }
  for (int i = threadIdx.x; i < Hp / 4; i += blockDim.x) dst[i] = src[i];
}

// ---------------------------------------------------------------------------------------
// The same step start for the tensor-core path, where states live as bf16 planes inside the
// operand panels: a list of byte-row copy jobs.  kind 0: state row gathered through the parent
// (or, at step 0, the sentence's encoder row); kind 1: embedding row of the slot's token.
// grid = (rows, n_jobs), block = 128
struct GatherJob {
  const unsigned char* src; long long src_stride;   // bytes
  unsigned char* dst; long long dst_stride;
  int row_bytes;   // multiple of 16
  int kind;
};
struct GatherJobs {
  GatherJob j[32];
  int n;
};
constexpr int kGatherJobsPerBlock = 4;   // a full step (768 rows x 10 jobs) is then 2304 blocks: one wave of resident CTAs
static __global__ void row_gather_kernel(GatherJobs jobs, const int32_t* __restrict__ parent, const int32_t* __restrict__ tok,
                                         int vocab, int k, int src_per_sentence) {
  tc::pdl_launch_dependents();   // see gemm_tc.cuh: the next kernel of the step may start its prologue
  tc::pdl_wait();                // nothing below runs before the previous kernel's results are visible
  const int r = blockIdx.x;
  const int j0 = blockIdx.y * kGatherJobsPerBlock;
  const int sent = r / k;
  const long long prow = src_per_sentence ? sent : parent ? sent * k + parent[r] : r;
  // every thread moves 16 bytes of up to four jobs at a time: all loads first, then the stores
  const unsigned char* src[kGatherJobsPerBlock];
  unsigned char* dst[kGatherJobsPerBlock];
  int nchunk[kGatherJobsPerBlock];
  int most = 0;
#pragma unroll
  for (int q = 0; q < kGatherJobsPerBlock; ++q) {
    nchunk[q] = 0; src[q] = nullptr; dst[q] = nullptr;
    if (j0 + q < jobs.n) {
      const GatherJob& jb = jobs.j[j0 + q];
      long long srow = prow;
      if (jb.kind == 1) {
        int t = tok[r];
        if (t < 0 || t >= vocab) t = kUnk;
        srow = t;
      }
      src[q] = jb.src + srow * jb.src_stride;
      dst[q] = jb.dst + (long long)r * jb.dst_stride;
      nchunk[q] = jb.row_bytes / 16;
      most = nchunk[q] > most ? nchunk[q] : most;
    }
  }
  for (int c = threadIdx.x; c < most; c += blockDim.x) {
    uint4 v[kGatherJobsPerBlock];
#pragma unroll
    for (int q = 0; q < kGatherJobsPerBlock; ++q)
      if (c < nchunk[q]) v[q] = reinterpret_cast<const uint4*>(src[q])[c];
#pragma unroll
    for (int q = 0; q < kGatherJobsPerBlock; ++q)
      if (c < nchunk[q]) reinterpret_cast<uint4*>(dst[q])[c] = v[q];
  }
}

// First decoder layer of a step whose recurrent products are there already (Engine::recurrent_ahead): gates of row r = row
// parent[r] of `pre` (its second part `feed` behind it, or null) plus the input term of its token, which the epilogue's preload looks
// up.  A thread per hidden unit; grid = (rows, Hp / 128).
static __global__ void __launch_bounds__(128) lstm_cell_kernel(tc::TcEpiLstm e, const float* __restrict__ pre, const float* __restrict__ feed,
                                                               int Hp) {
  tc::pdl_launch_dependents();
  tc::pdl_wait();
  const int row = blockIdx.x, col = (blockIdx.y * 128 + threadIdx.x) * 4;
  if (col >= 4 * Hp) return;
  const size_t at = (size_t)e.c_src_row(row) * 4 * Hp + col;
  const tc::TcEpiLstm::Pre p = e.preload(row, col);
  float4 v = *reinterpret_cast<const float4*>(pre + at);
  if (feed) {
    const float4 f = *reinterpret_cast<const float4*>(feed + at);
    v.x += f.x; v.y += f.y; v.z += f.z; v.w += f.w;
  }
  e.finish_row(true, row, col, 0, v, p);
}

// Encoder input for the tensor-core path: embedding planes of the token at reversed position
// `pos` into columns [0, Hp) of the layer-0 panel; zeros past the sentence.
// grid = (B, nt), block = 128
static __global__ void enc_embed_planes_kernel(const int32_t* __restrict__ ids, const int32_t* __restrict__ off,
                                               const int32_t* __restrict__ len, tc::Planes emb, int vocab,
                                               tc::Planes dst, int Hp, int pos) {
  const int b = blockIdx.x, t = blockIdx.y;
  const int S = len[b];
  uint4* d = reinterpret_cast<uint4*>(dst.p[t] + (size_t)b * dst.ld);
  if (pos < S) {
    int tok = ids[off[b] + (S - 1 - pos)];
    if (tok < 0 || tok >= vocab) tok = 0;
    const uint4* src = reinterpret_cast<const uint4*>(emb.p[t] + (size_t)tok * emb.ld);
    for (int i = threadIdx.x; i < Hp / 8; i += blockDim.x) d[i] = src[i];
  } else {
    for (int i = threadIdx.x; i < Hp / 8; i += blockDim.x) d[i] = make_uint4(0, 0, 0, 0);
  }
}

// The same for every position at once (encoder layer by layer): row (pos * n + b) of dst.  grid = (n, positions, nt).
static __global__ void enc_embed_seq_kernel(const int32_t* __restrict__ ids, const int32_t* __restrict__ off, const int32_t* __restrict__ len,
                                            tc::Planes emb, int vocab, tc::Planes dst, int Hp, int pos0) {
  tc::pdl_launch_dependents();
  tc::pdl_wait();
  const int b = blockIdx.x, t = blockIdx.z, pos = pos0 + blockIdx.y;
  const int S = len[b];
  uint4* d = reinterpret_cast<uint4*>(dst.p[t] + (size_t)(blockIdx.y * gridDim.x + b) * dst.ld);
  int tok = pos < S ? ids[off[b] + (S - 1 - pos)] : 0;
  if (tok < 0 || tok >= vocab) tok = 0;
  const uint4* src = reinterpret_cast<const uint4*>(emb.p[t] + (size_t)tok * emb.ld);
  for (int i = threadIdx.x; i < Hp / 8; i += blockDim.x) d[i] = src[i];
}

// ---------------------------------------------------------------------------------------
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// ---------------------------------------------------------------------------------------
// Attention of a step (AttentionNode::ForwardProp, src/layer_attention.h:243-483,
// kernels k12-k20: Sgemm m=1, SigmoidKernel, AlignmentPosKernel, LowerUpperKernel,
// CreateIndicesKernel, LoadInHSKernel, ElemReduceKernelLarge, AlignmentReductionKernel,
// CreateCTKernel).
//   proj [rows][2*Hp]: tanh(W_p h) | W_a^T h      (global_dot: `u` = h_top itself)
//   hs   row sent * hs_sent + p * hs_pos: top encoder state of a sentence after consuming reversed position p, in T
//   ctx  [rows][Hp] fp32 and/or ctx_planes (bf16 planes, columns [0,Hp) of the panel) and ctx2 (a second place for the same)
//   rec_align [rows][rec_win] / rec_lo [rows] / rec_vit [rows]: alignment record of this step
//   (may be null).  win = 2D+1 for local attention, max_src for the global modes.
//   ens = 0: one model; the record is the window (rec_win = win) and its first position rec_lo.
//   ens = 1, 2, 3: first / middle / last member of an ensemble; the record is dense over the source
//   (rec_win = max_src, rec_lo = 0), the first member writes it, the others add to it in member order,
//   and the last one takes the vote: the position of the largest summed score, the search starting from
//   "none, 0" (EnsembleFactory::EnsemblesModels, src/decoder.h:1934-1964).
// Optional record of the attention centre p_t of every row of a forward (local attention): the parity tests
// use it to tell a window that was cut on the other side of an integer apart from an error.
struct AttTrace {
  float* pt;            // [n][T1][k] by the caller's sentence index, or null
  const int32_t* orig;  // batch slot -> caller's sentence index
  int T1;               // forwards per sentence in the record (longest step count + 1)
  int t;                // this forward
};
// Optional fold of the attention output layer into this kernel.  htilde = tanh(W_c1 ctx + W_c2 h + b) and
// ctx = sum_j a_j hs_j, so W_c1 ctx = sum_j a_j (W_c1 hs_j): with `cs` = the encoder states already multiplied by
// W_c1 (once per batch), the weighted sum IS the first term, `add` carries the row's W_c2 h (computed with the
// attention projections) and the kernel writes the attentional state itself -- a dependent GEMM launch less per
// step.  cs == nullptr: plain context.
struct AttFold {
  const float* cs;      // [B][max_src][Hp] like hs
  const float* add; int ld_add;   // element (row, j) at add[row * ld_add + j]
  const float* bias;    // [Hp]
};
// A CTA serves G beams of a sentence (a group): their windows overlap almost everywhere, so an encoder state is read once
// for all of them -- for the scores by a warp per position, for the context by a thread per four columns -- and meets G
// vectors, the scores' in shared memory.  The kernel is a chain of L2 round trips (centre, scores, context), so a group
// costs little more time than one row, while the rows of a step become fewer waves of CTAs.  Against a CTA of 256 threads
// per row: 1536 rows, window 21 44 -> 32 us per step; 640 rows, whole sources of up to 100 words 49 -> 28; 768 rows 26 -> 19.
// G = 1, THREADS = 1024 for a step whose rows leave SMs empty: one position per warp and the context in four ranges of
// positions (one sentence: 18.1 us per step with 256 threads, 10 so).  grid = sentences * groups, dynamic smem =
// attention_smem
// T: the states as they are stored, fp32 or (one plane: they are rounded to it anyhow) bf16.  The kernel's time beyond its chain
// is reading them out of L2 twice, for the scores and for the context.
__device__ __forceinline__ float4 state4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float2 state2(const float* p) { return *reinterpret_cast<const float2*>(p); }
__device__ __forceinline__ float2 state2(uint32_t q) { return make_float2(__uint_as_float(q << 16), __uint_as_float(q & 0xffff0000u)); }
__device__ __forceinline__ float2 state2(const __nv_bfloat16* p) { return state2(*reinterpret_cast<const uint32_t*>(p)); }
__device__ __forceinline__ float4 state4(const __nv_bfloat16* p) {
  const uint2 q = *reinterpret_cast<const uint2*>(p);
  const float2 a = state2(q.x), b = state2(q.y);
  return make_float4(a.x, a.y, b.x, b.y);
}
template <int G, int THREADS, class T>
static __global__ void __launch_bounds__(THREADS, THREADS == 512 ? 2 : 1) attention_kernel(const float* __restrict__ proj, int ldp, const float* __restrict__ u_alt, int ldu,
                                 const float* __restrict__ vp, const T* __restrict__ hs,
                                 const int32_t* __restrict__ src_len, float* __restrict__ ctx, int H, int Hp,
                                 int k, int groups, int hs_sent, int hs_pos, int mode, int D, float* __restrict__ rec_align,
                                 int32_t* __restrict__ rec_lo, int32_t* __restrict__ rec_vit, tc::Planes ctx_planes, tc::Planes ctx2, int nt,
                                 int rec_win, int ens, AttTrace at, AttFold fold) {
  tc::pdl_launch_dependents();   // see gemm_tc.cuh: the next kernel of the step may start its prologue
  constexpr int kWarps = THREADS / 32;
  constexpr int kRanges = THREADS > 512 ? THREADS / 256 : 1;    // of positions, in the context sum
  constexpr int GP = G == 3 ? 4 : G;                            // beams per position in e, for vector loads
  const int sent = blockIdx.x / groups, q = blockIdx.x - sent * groups;
  const int per = (k + groups - 1) / groups, b0 = q * per;
  const int nb = k - b0 < per ? k - b0 : per;          // beams of this group, 1 .. G
  if (THREADS > 512) {
    // Few rows: the weights of a step have displaced the encoder's states from L2.  While the projection runs, the CTAs
    // of a sentence ask for them again.  A hint: no state is read here, and the length this goes by may be an earlier
    // batch's (or the zero it starts as), which names rows of the same buffer; the one that counts is read below.
    const int S = src_len[sent];
    const char* h0 = reinterpret_cast<const char*>(hs + (size_t)sent * hs_sent * Hp);
    const char* c0 = fold.cs ? reinterpret_cast<const char*>(fold.cs + (size_t)sent * hs_sent * Hp) : nullptr;
    const int lines = Hp / 32;         // (of fp32 rows; every other one where the states are half as wide)
    for (int i = q * THREADS + threadIdx.x; i < S * lines; i += groups * THREADS) {
      const int pos = i / lines, line = i - pos * lines;
      const size_t row = (size_t)pos * hs_pos * Hp;
      if (sizeof(T) == 4 || line % 2 == 0) asm volatile("prefetch.global.L2 [%0];" ::"l"(h0 + row * sizeof(T) + (size_t)line * (32 * sizeof(T))));
      if (c0) asm volatile("prefetch.global.L2 [%0];" ::"l"(c0 + row * 4 + (size_t)line * 128));
    }
  }
  tc::pdl_wait();                // nothing below runs before the previous kernel's results are visible
  int S;      // (from L2 and not moved: the value above may be in L1)
  asm volatile("ld.global.cg.s32 %0, [%1];" : "=r"(S) : "l"(src_len + sent) : "memory");
  extern __shared__ __align__(16) float sm[];
  float* su = sm;                                           // [G][Hp] what the states are multiplied with, and then
  float4* csum = reinterpret_cast<float4*>(sm);             // [kRanges - 1][256] partial contexts (G = 1)
  float* e = sm + G * (Hp > (kRanges - 1) * 1024 ? Hp : (kRanges - 1) * 1024);    // [positions][GP], from the first position of all windows on
  __shared__ float s_red[G][kWarps];
  __shared__ float s_pt[G];
  __shared__ int s_lo[G], s_hi[G];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int r0 = sent * k + b0;
  const T* hsb = hs + (size_t)sent * hs_sent * Hp;
  auto row_of = [&](int g) { return r0 + (g < nb ? g : nb - 1); };

#pragma unroll
  for (int g = 0; g < G; ++g) {
    const float* u = u_alt ? (u_alt + (size_t)row_of(g) * ldu) : (proj + (size_t)row_of(g) * ldp + Hp);
    for (int j = tid * 4; j < Hp; j += THREADS * 4) *reinterpret_cast<float4*>(su + g * Hp + j) = *reinterpret_cast<const float4*>(u + j);
  }
  if (mode == 0) {
    // each 256 threads take every other beam
    constexpr int kPart = THREADS / 256, kMine = (G + kPart - 1) / kPart;
    const int first = G > 1 ? tid >> 8 : 0;
    constexpr int kStep = G > 1 ? 256 : THREADS;
    float part[kMine] = {};
    for (int j = G > 1 ? tid & 255 : tid; j < H; j += kStep) {
      const float v = vp[j];
#pragma unroll
      for (int i = 0; i < kMine; ++i) part[i] = fmaf(v, proj[(size_t)row_of(first + i * kPart) * ldp + j], part[i]);
    }
#pragma unroll
    for (int i = 0; i < kMine; ++i) {
      const int g = first + i * kPart;
      part[i] = warp_sum(part[i]);
      if (lane == 0 && g < G) s_red[g][G > 1 ? warp & 7 : warp] = part[i];
    }
    __syncthreads();
    if (warp < nb) {
      float dot = 0.f;
      if (G > 1) {
        for (int i = 0; i < 8; ++i) dot += s_red[warp][i];
      } else {
        dot = warp_sum(lane < kWarps ? s_red[0][lane] : 0.f);
      }
      if (lane == 0) {
        const float sg = (float)(1.0 / (1.0 + exp(-1.0 * (double)dot)));  // SigmoidKernel, deep_rnn_kernel.h:1075-1080
        const float pt = (float)S * sg;
        s_pt[warp] = pt;
        s_lo[warp] = (0 > (int)pt - D) ? 0 : ((int)pt - D);                       // LowerUpperKernel, :1094-1100
        s_hi[warp] = ((S - 1) < (int)pt + D) ? (S - 1) : ((int)pt + D);
        if (at.pt) at.pt[((size_t)at.orig[sent] * at.T1 + at.t) * k + b0 + warp] = pt;
      }
    }
  } else if (tid < nb) {
    s_pt[tid] = 0.f; s_lo[tid] = 0; s_hi[tid] = S - 1;
  }
  __syncthreads();
  int lo = s_lo[0], hi = s_hi[0];     // of all windows
#pragma unroll
  for (int g = 1; g < G; ++g)
    if (g < nb) { lo = min(lo, s_lo[g]); hi = max(hi, s_hi[g]); }
  const int W = hi - lo + 1;
  // scores: two positions at a time meet the vectors read from shared memory, which would otherwise be the bound
  constexpr int kAtOnce = G > 1 ? 2 : 1;
  for (int w = warp; w < W; w += kWarps * kAtOnce) {
    const int w2 = kAtOnce > 1 && w + kWarps < W ? w + kWarps : w;
    const T* ha = hsb + (size_t)(S - 1 - (lo + w)) * hs_pos * Hp;
    const T* hb = hsb + (size_t)(S - 1 - (lo + w2)) * hs_pos * Hp;
    float acc[kAtOnce][G] = {};
    auto dot4 = [&](int j) {
      float4 a[kAtOnce];
      a[0] = state4(ha + j);
      if (kAtOnce > 1) a[kAtOnce - 1] = state4(hb + j);
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const float4 b = *reinterpret_cast<const float4*>(su + g * Hp + j);
#pragma unroll
        for (int p = 0; p < kAtOnce; ++p) {
          float& c = acc[p][g];
          c = fmaf(a[p].x, b.x, c); c = fmaf(a[p].y, b.y, c); c = fmaf(a[p].z, b.z, c); c = fmaf(a[p].w, b.w, c);
        }
      }
    };
#pragma unroll (THREADS > 512 ? 8 : G > 1 ? 2 : 4)
    for (int j = lane * 4; j < Hp; j += 128) dot4(j);
#pragma unroll
    for (int p = 0; p < kAtOnce; ++p)
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const float v = warp_sum(acc[p][g]);
        if (lane == 0) e[(p ? w2 : w) * GP + g] = v;
      }
  }
  __syncthreads();
  if (warp < nb) {
    // AlignmentReductionKernel, deep_rnn_kernel.h:1197-1241 (max starts at 0, no renormalisation
    // after the Gaussian), one lane per window position instead of one thread per beam
    const int g = warp, wlo = s_lo[g], whi = s_hi[g];
    const int w0 = wlo - lo, w1 = whi - lo + 1;     // its window among the positions
    float* eg = e + g;
    float mx = 0.f;
    for (int w = w0 + lane; w < w1; w += 32) mx = fmaxf(mx, eg[w * GP]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    float sum = 0.f;
    for (int w = w0 + lane; w < w1; w += 32) { const float ev = expf(eg[w * GP] - mx); eg[w * GP] = ev; sum += ev; }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const float sigma_sq = ((float)D * (float)D) / 4.0f;
    const float pt = s_pt[g];
    float best = 0.f; int besti = 0x7fffffff;
    for (int w = w0 + lane; w < w1; w += 32) {
      float a = eg[w * GP];
      if (mode == 0) {
        const float d = pt - (float)(lo + w);
        const float tmp = expf(-(d * d) / (2 * sigma_sq));
        if (0 != sum) a = (a / sum) * tmp;
      } else if (0 != sum) a = a / sum;
      eg[w * GP] = a;
      if (a > best) { best = a; besti = lo + w; }  // viterbi vote, src/decoder.h:1948-1962 (first maximum)
    }
    if (G > 1)
      for (int w = lane; w < W; w += 32)
        if (w < w0 || w >= w1) eg[w * GP] = 0.f;
    if (rec_lo && ens == 0) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, besti, o);
        if (ob > best || (ob == best && oi < besti)) { best = ob; besti = oi; }
      }
    }
    if (lane == 0 && rec_lo && ens == 0) { rec_lo[r0 + g] = wlo; rec_vit[r0 + g] = (best > 0.f) ? besti : -1; }
  } else if (G > 1 && warp < G) {
    for (int w = lane; w < W; w += 32) e[w * GP + warp] = 0.f;
  }
  __syncthreads();
  if (rec_align)
    for (int g = 0; g < nb; ++g) {
      float* row = rec_align + (size_t)(r0 + g) * rec_win;
      const float* eg = e + g;
      const int wlo = s_lo[g], whi = s_hi[g];
      if (ens == 0) {
        for (int w = tid; w < rec_win; w += THREADS) row[w] = (wlo + w <= whi) ? eg[(wlo - lo + w) * GP] : 0.f;
        continue;
      }
      for (int sp = tid; sp < rec_win; sp += THREADS) {
        const float a = (sp >= wlo && sp <= whi) ? eg[(sp - lo) * GP] : 0.f;
        row[sp] = (ens == 1) ? (0.f + a) : (row[sp] + a);
      }
      if (ens == 3) {
        __syncthreads();
        if (warp == 0) {
          float best = 0.f; int besti = 0x7fffffff;
          for (int sp = lane; sp < rec_win; sp += 32) {
            const float a = row[sp];
            if (a > best) { best = a; besti = sp; }
          }
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) {
            const float ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, besti, o);
            if (ob > best || (ob == best && oi < besti)) { best = ob; besti = oi; }
          }
          if (lane == 0) { rec_lo[r0 + g] = 0; rec_vit[r0 + g] = (best > 0.f) ? besti : -1; }
        }
      }
    }
  // context: CreateCTKernel, deep_rnn_kernel.h:1250-1260
  auto context = [&](const auto* csb) {
  const auto* col0 = csb + (size_t)(S - 1 - lo) * hs_pos * Hp;
  const size_t step = (size_t)hs_pos * Hp;
  if constexpr (kRanges == 1) {
    // a thread has two columns of every beam and sums the positions in order
    for (int j = tid * 2; j < Hp; j += THREADS * 2) {
      float2 acc[G];
#pragma unroll
      for (int g = 0; g < G; ++g) acc[g] = make_float2(0.f, 0.f);
      const auto* col = col0 + j;
#pragma unroll 6
      for (int w = 0; w < W; ++w) {
        const float2 h = state2(col - w * step);
        float a[GP];
        if constexpr (GP == 4) {
          *reinterpret_cast<float4*>(a) = *reinterpret_cast<const float4*>(e + w * GP);
        } else if constexpr (GP == 2) {
          *reinterpret_cast<float2*>(a) = *reinterpret_cast<const float2*>(e + w * GP);
        } else {
          a[0] = e[w];
        }
#pragma unroll
        for (int g = 0; g < G; ++g) { acc[g].x += a[g] * h.x; acc[g].y += a[g] * h.y; }
      }
#pragma unroll
      for (int g = 0; g < G; ++g) {
        if (g >= nb) break;
        const int r = r0 + g;
        float2 c = acc[g];
        if (fold.cs) {
          // the attentional state: the sums of TcEpiBiasTanh in its order, (W_c1 ctx + W_c2 h) + b
          const float2 a = *reinterpret_cast<const float2*>(fold.add + (size_t)r * fold.ld_add + j);
          const float2 b = *reinterpret_cast<const float2*>(fold.bias + j);
          c.x = tc::tanh_fast((c.x + a.x) + b.x); c.y = tc::tanh_fast((c.y + a.y) + b.y);
        }
        if (ctx) *reinterpret_cast<float2*>(ctx + (size_t)r * Hp + j) = c;
        if (ctx_planes.p[0])    // tensor-core path: the context goes straight into its operand panel
          tc::split_store2(ctx_planes, nt, (size_t)r * ctx_planes.ld + j, c.x, c.y);
        if (ctx2.p[0]) tc::split_store2(ctx2, nt, (size_t)r * ctx2.ld + j, c.x, c.y);
      }
    }
  } else {
    const int range = tid >> 8, c = tid & 255, w0 = W * range / kRanges, w1 = W * (range + 1) / kRanges;
    for (int j0 = 0; j0 < Hp; j0 += 1024) {
      const int j = j0 + c * 4;
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      if (j < Hp) {
        const auto* col = col0 + j;
#pragma unroll 6
        for (int w = w0; w < w1; ++w) {
          const float a = e[w];
          const float4 h4 = state4(col - w * step);
          acc.x += a * h4.x; acc.y += a * h4.y; acc.z += a * h4.z; acc.w += a * h4.w;
        }
      }
      if (j0 > 0) __syncthreads();      // (the previous pass's partial contexts have been read)
      if (range > 0 && j < Hp) csum[(range - 1) * 256 + c] = acc;
      __syncthreads();
      if (range == 0 && j < Hp) {
#pragma unroll
        for (int o = 0; o < kRanges - 1; ++o) {
          const float4 p = csum[o * 256 + c];
          acc.x += p.x; acc.y += p.y; acc.z += p.z; acc.w += p.w;
        }
        if (fold.cs) {
          const float4 a = *reinterpret_cast<const float4*>(fold.add + (size_t)r0 * fold.ld_add + j);
          const float4 b = *reinterpret_cast<const float4*>(fold.bias + j);
          acc.x = tc::tanh_fast((acc.x + a.x) + b.x); acc.y = tc::tanh_fast((acc.y + a.y) + b.y);
          acc.z = tc::tanh_fast((acc.z + a.z) + b.z); acc.w = tc::tanh_fast((acc.w + a.w) + b.w);
        }
        if (ctx) *reinterpret_cast<float4*>(ctx + (size_t)r0 * Hp + j) = acc;
        if (ctx_planes.p[0]) tc::split_store4(ctx_planes, nt, (size_t)r0 * ctx_planes.ld + j, acc.x, acc.y, acc.z, acc.w);
        if (ctx2.p[0]) tc::split_store4(ctx2, nt, (size_t)r0 * ctx2.ld + j, acc.x, acc.y, acc.z, acc.w);
      }
    }
  }
  };
  const float* folded = fold.cs ? fold.cs + (size_t)sent * hs_sent * Hp : nullptr;
  if constexpr (sizeof(T) == 4) context(folded ? folded : hsb);
  else if (folded) context(folded);
  else context(hsb);
}

// `positions`: the window of one beam, the whole source where windows are joined.  Wide models and global attention over
// sources of more than about 9000 words pass 48 KB and are launched with the opt-in (tc::allow_smem): up to 54,000
// floats for the widest vector and the window of a row together.
inline size_t attention_smem(int G, int threads, int Hp, int positions) {
  const int parts = threads > 512 ? (threads / 256 - 1) * 1024 : 0, gp = G == 3 ? 4 : G;
  return sizeof(float) * (size_t)(G * (Hp > parts ? Hp : parts) + gp * positions);
}

// ---------------------------------------------------------------------------------------
// Log-softmax statistics and per-row top-kk of the logits in ONE pass over HBM.
// Replaces MatrixBiasKernel's consumer OutputdistOverflowPreventionKernel
// (src/deep_rnn_kernel.h:352-429, three passes), the V x k device-to-host copy
// (src/decoder.h:1413) and the host scan that keeps the k+1 best per beam
// (src/decoder.h:401-410).  Order: value descending, vocabulary index ascending -- what the
// strict-greater replacement of the reference keeps.  log p = (z - max) - log(sum exp).
// grid = rows, block = 256.
struct TopkOut {
  int32_t* idx;    // [rows][kk]
  float* logp;     // [rows][kk]
  float* eos_logp; // [rows]
  float* row_stats; // [rows][2] = (max, log sum exp(z - max)) of the row, may be null
};
__device__ __forceinline__ bool better(float va, int ia, float vb, int ib) { return va > vb || (va == vb && ia < ib); }

// Refinement of a row whose logits came from a ONE-product (plain fp16) vocabulary GEMM: the row's
// activations and the vocabulary weights as fp16 pairs, from which the few logits that matter are
// recomputed at fp32-class accuracy.  eps_coef * |a|_2 bounds the error of a one-product logit
// (both operands rounded to 11 bits: relative 2^-10 on every term, Cauchy-Schwarz over the row,
// largest weight-row norm of the model folded into eps_coef).
struct TopkRefine {
  const __half* a0; const __half* a1; int lda;   // activations [rows][lda], planes of the fp16 pair
  const __half* b0; const __half* b1; int ldb;   // vocabulary weights [V][ldb]
  const float* bias;                             // [V]
  int K;
  float eps_coef;
};
constexpr float kPairInv = 1.0f / 2048.0f;
inline float refine_eps(float w_norm_max) { return 1.1f * (1.0f / 1024.0f) * w_norm_max; }

// ---------------------------------------------------------------------------------------
// Beam selection for one sentence and one step, all on the device.  Replaces
// Decoder<T>::ExpandHypothesis (src/decoder.h:355-480) and, on a sentence's last step,
// Decoder<T>::FinishCurrentHypotheses (src/decoder.h:502-525).
// Candidate order = (score desc, beam asc, vocab asc), the defined order of the reference's
// global heap.  START is skipped, EOS goes to the finished list without using a slot.
struct BeamState {
  int32_t* tok;        // [R] current token of each slot
  float* score;        // [R]
  int32_t* parent;     // [R] parent slot chosen by the last selection
  int32_t* hist_tok;   // [Tcap][R]
  int32_t* hist_parent;// [Tcap][R]
  int32_t* fin_t;      // [B][fin_cap] step at which EOS was produced
  int32_t* fin_b;      // [B][fin_cap] slot whose history the hypothesis continues
  float* fin_score;    // [B][fin_cap]
  int32_t* fin_n;      // [B]
  int fin_cap;
  int R;
};
struct TraceDev {
  int32_t* cand_tok; float* cand_logp; int32_t* surv_tok; int32_t* surv_parent; float* surv_score; float* final_logp;
  const int32_t* force_tok; const int32_t* force_parent; const float* force_score;
  int Tm;
  float* pt;                 // [n][Tm+1][k] attention centre of every forward (member 0), or null
  float* gold_logp;          // [n][Tm][k] log-probability of the forced token of every slot (scoring)
  const float* logits; int ld_logits; const float* row_stats;   // what gold_logp is computed from
  TopkRefine rf;             // set when the logits are one-product values: the forced token's logit is recomputed accurately
};
// The selection runs inside the softmax kernels: the CTA that finishes a sentence's last row (a counter per sentence)
// goes on with the sentence's selection, which as a kernel of its own cost a launch and a round trip per step for a
// microsecond of work (7.7 us per step at one sentence).
struct SelectArgs {
  BeamState bs;
  const int32_t* steps;    // null: no selection (the kernel is called for its own result)
  const int32_t* orig;
  int* done;               // [B] rows of the sentence finished in this step; left at zero
  int t, k;
  float penalty, diversity;
  TraceDev tr;
};
constexpr int kSelectSmem = kMaxBeam * (kMaxBeam + 1) * 16;   // its shared memory: candidates of the widest beam
// Candidates of the whole sentence in shared memory, then the walk over them in order, 32 candidates at a time.
template <int THREADS>
__device__ __forceinline__ void beam_select_block(const SelectArgs& a, const TopkOut& cand, int sent, int T, int osent, int nf0, unsigned char* smraw) {
  const BeamState& bs = a.bs;
  const TraceDev& tr = a.tr;
  const int k = a.k, kk = k + 1, t = a.t;
  const int r0 = sent * k;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (t > T) return;
  if (t == T) {
    if (warp == 0) {
      const int n0 = nf0;
      if (lane < k) {
        const float lp = __ldcg(cand.eos_logp + r0 + lane);
        if (tr.final_logp) tr.final_logp[(size_t)osent * k + lane] = lp;
        const int n = n0 + lane;
        if (n < bs.fin_cap) {
          bs.fin_t[(size_t)sent * bs.fin_cap + n] = t;
          bs.fin_b[(size_t)sent * bs.fin_cap + n] = lane;
          bs.fin_score[(size_t)sent * bs.fin_cap + n] = bs.score[r0 + lane] + (lp + a.penalty);
        }
      }
      __syncwarp();
      if (lane == 0) bs.fin_n[sent] = n0 + k < bs.fin_cap ? n0 + k : bs.fin_cap;
    }
    return;
  }
  unsigned long long* key = reinterpret_cast<unsigned long long*>(smraw);   // sortable (score, beam, vocabulary id)
  unsigned long long* listed = key + k * kk;                                // those that may be among the survivors
  const int cols = (t == 0) ? 1 : k;
  const int n = cols * kk;
  __shared__ int s_special[THREADS / 32];      // a warp's candidates that take no slot
  int special = 0;
  for (int c = tid; c < n; c += THREADS) {
    const int b = c / kk, q = c - b * kk;
    const float lp = __ldcg(cand.logp + (size_t)(r0 + b) * kk + q);    // (other CTAs' results)
    const int v = __ldcg(cand.idx + (size_t)(r0 + b) * kk + q);
    const float rank_penalty = (float)(q + 1) * a.diversity;
    const float sc = (lp + bs.score[r0 + b]) - rank_penalty;
    // one 64-bit key, larger = earlier: score descending, then beam ascending, then vocabulary id ascending
    const unsigned int fb = __float_as_uint(sc);
    const unsigned int ord = (fb & 0x80000000u) ? ~fb : (fb | 0x80000000u);
    const unsigned int low = 0xFFFFFFFFu - (((unsigned int)b << 24) | ((unsigned int)v & 0xFFFFFFu));
    key[c] = ((unsigned long long)ord << 32) | low;
    special += v < 0 || v == kStart || v == kEos ? 1 : 0;
    if (tr.cand_tok) {
      const size_t off = ((((size_t)osent * tr.Tm + t) * k + b) * kk) + q;
      tr.cand_tok[off] = v; tr.cand_logp[off] = lp;
    }
  }
  special = __reduce_add_sync(0xffffffffu, special);
  if (lane == 0) s_special[warp] = special;
  __syncthreads();
  // Only as many candidates as there are slots, and those that take none (START, EOS), have to be in order: the `need` best.
  // The need-th best of every row's first two (of its first, beyond 16 rows) is a bound that they all reach; what reaches it,
  // some tens of n, is listed and ranked.  (All n against all n: 2.5 us of the last CTA at 156 candidates, whatever the
  // threads; 768 rows 29.4 -> 25.3 us a launch, 1536 rows 30.9 -> 25.1.)
  __shared__ unsigned long long s_bound;
  __shared__ int s_listed;
  // so few are ranked as they are (a beam of 7: 56 of them by the bound 4.33 -> 4.38 ms in a call of 69 steps; 12: 156 gain by it,
  // as above; nothing between was measured)
  constexpr int kDirect = 64;
  int n_order = n;
  const unsigned long long* ranked = key;
  unsigned long long* order = listed;      // the result, in order
  if (n > kDirect) {
    if (warp == 0) {
      const int need = k + __reduce_add_sync(0xffffffffu, lane < THREADS / 32 ? s_special[lane] : 0);
      const int firsts = cols > 16 ? 1 : 2, m = firsts * cols;
      const int b = firsts == 2 ? lane >> 1 : lane, q = firsts == 2 ? lane & 1 : 0;
      const unsigned long long f = lane < m ? key[b * kk + q] : 0ull;
      int rank = 0;
#pragma unroll 4
      for (int j = 0; j < m; ++j) {
        const unsigned long long o = __shfl_sync(0xffffffffu, f, j);
        rank += o > f || (o == f && j < lane) ? 1 : 0;
      }
      if (lane == 0) { s_listed = 0; if (need > m) s_bound = 0ull; }
      if (lane < m && rank == need - 1) s_bound = f;
    }
    __syncthreads();
    const unsigned long long bound = s_bound;
    for (int c = tid; c < n; c += THREADS) {
      const unsigned long long kc = key[c];
      if (kc >= bound) listed[atomicAdd(&s_listed, 1)] = kc;
    }
    __syncthreads();
    n_order = s_listed;
    ranked = listed;
    order = key;
  }
  // a thread counts the candidates before its own; four of a large block share one
  const int share = THREADS > 256 && n_order <= THREADS / 4 ? 4 : 1;
  for (int c0 = 0; c0 < n_order; c0 += THREADS / share) {
    const int c = c0 + tid / share;
    const unsigned long long kc = c < n_order ? ranked[c] : 0ull;
    int p = 0;
    if (c < n_order) {
#pragma unroll 4
      for (int d = tid & (share - 1); d < n_order; d += share) {
        const unsigned long long kd = ranked[d];
        p += (kd > kc || (kd == kc && d < c)) ? 1 : 0;
      }
    }
    if (share > 1) {
      p += __shfl_xor_sync(0xffffffffu, p, 1);
      p += __shfl_xor_sync(0xffffffffu, p, 2);
    }
    if (c < n_order && (tid & (share - 1)) == 0) order[p] = kc;
  }
  __syncthreads();
  __shared__ int s_ntok[kMaxBeam + 1], s_npar[kMaxBeam + 1];
  __shared__ float s_nscore[kMaxBeam + 1];
  if (warp == 0) {
    // START is skipped, EOS leaves the beam without taking a slot as long as slots are free
    int ns = 0, nf = nf0;
    for (int p0 = 0; p0 < n_order && ns < k; p0 += 32) {
      const int p = p0 + lane;
      const unsigned long long ko = p < n_order ? order[p] : 0ull;
      const unsigned int low = 0xFFFFFFFFu - (unsigned int)ko, ord = (unsigned int)(ko >> 32);
      const int v = p < n_order && (low & 0xFFFFFFu) != 0xFFFFFFu ? (int)(low & 0xFFFFFFu) : -1, b = (int)(low >> 24);
      const float sc = __uint_as_float((ord & 0x80000000u) ? (ord & 0x7FFFFFFFu) : ~ord);
      const unsigned take = __ballot_sync(0xffffffffu, v >= 0 && v != kStart && v != kEos);
      const unsigned below = (1u << lane) - 1u;
      const int slot = ns + __popc(take & below);            // free slots used before this candidate
      const bool eos = v == kEos && slot < k;
      const unsigned ends = __ballot_sync(0xffffffffu, eos);
      if (((take >> lane) & 1u) && slot < k) { s_ntok[slot] = v; s_npar[slot] = b; s_nscore[slot] = sc + a.penalty; }
      const int f = nf + __popc(ends & below);
      if (eos && f < bs.fin_cap) {
        bs.fin_t[(size_t)sent * bs.fin_cap + f] = t;
        bs.fin_b[(size_t)sent * bs.fin_cap + f] = b;
        bs.fin_score[(size_t)sent * bs.fin_cap + f] = sc + a.penalty;
      }
      ns += __popc(take);
      nf += __popc(ends);
    }
    for (int q = ns + lane; q < k; q += 32) { s_ntok[q] = kUnk; s_npar[q] = 0; s_nscore[q] = kDeadScore; }
    if (lane == 0 && nf > nf0) bs.fin_n[sent] = nf < bs.fin_cap ? nf : bs.fin_cap;
  }
  // Scoring (force-decoding): log-probability of the forced token of every slot under its parent's row.
  // With one-product logits the token's logit is recomputed from both planes of both operands, like the
  // candidates in the softmax kernel; one warp per slot.
  __shared__ float s_gold[kMaxBeam + 1];
  if (tr.force_tok && tr.gold_logp && tr.logits) {
    for (int b = warp; b < k; b += THREADS / 32) {
      const size_t off = ((size_t)osent * tr.Tm + t) * k + b;
      const int npar = tr.force_parent[off];
      const int prow = r0 + (npar >= 0 && npar < k ? npar : 0);
      const int gt = tr.force_tok[off] >= 0 ? tr.force_tok[off] : 0;
      float zv = 0.f;
      if (tr.rf.a0) {
        const __half* a0 = tr.rf.a0 + (size_t)prow * tr.rf.lda;
        const __half* a1 = tr.rf.a1 + (size_t)prow * tr.rf.lda;
        const __half* w0 = tr.rf.b0 + (size_t)gt * tr.rf.ldb;
        const __half* w1 = tr.rf.b1 + (size_t)gt * tr.rf.ldb;
        float acc = 0.f;
        for (int j = lane; j < tr.rf.K; j += 32) {
          const float x = fmaf(__half2float(a1[j]), kPairInv, __half2float(a0[j]));
          const float w = fmaf(__half2float(w1[j]), kPairInv, __half2float(w0[j]));
          acc = fmaf(x, w, acc);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        zv = acc + (tr.rf.bias ? tr.rf.bias[gt] : 0.f);
      } else if (lane == 0) {
        zv = tr.logits[(size_t)prow * tr.ld_logits + gt];
      }
      if (lane == 0) s_gold[b] = (zv - __ldcg(tr.row_stats + 2 * prow)) - __ldcg(tr.row_stats + 2 * prow + 1);
    }
  }
  __syncthreads();
  if (tid < k) {
    const int b = tid;
    int ntok = s_ntok[b], npar = s_npar[b];
    float nscore = s_nscore[b];
    const size_t off = ((size_t)osent * tr.Tm + t) * k + b;
    if (tr.surv_tok) { tr.surv_tok[off] = ntok; tr.surv_parent[off] = npar; tr.surv_score[off] = nscore; }
    if (tr.force_tok) {
      ntok = tr.force_tok[off]; npar = tr.force_parent[off]; nscore = tr.force_score[off];
      if (tr.gold_logp && tr.logits) tr.gold_logp[off] = s_gold[b];
    }
    bs.tok[r0 + b] = ntok; bs.parent[r0 + b] = npar; bs.score[r0 + b] = nscore;
    bs.hist_tok[(size_t)t * bs.R + r0 + b] = ntok;
    bs.hist_parent[(size_t)t * bs.R + r0 + b] = npar;
  }
}
// End of a softmax kernel: row r's results are written; the last row of its sentence selects.
template <int THREADS>
__device__ __forceinline__ void select_if_last(const SelectArgs& a, const TopkOut& cand, int r, unsigned char* smraw) {
  if (!a.steps) return;
  __shared__ int s_last;
  const int sent = r / a.k;
  // what the selection reads first is on its way while the counter answers
  const int T = a.steps[sent], osent = a.orig[sent], nf0 = a.bs.fin_n[sent];
  __syncthreads();
  bool last = true;        // (a greedy sentence has one row)
  if (a.k > 1) {
    if (threadIdx.x == 0) {
      int before;            // releases this row's candidates (all threads', by the barrier) and acquires the other rows'
      asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;" : "=r"(before) : "l"(a.done + sent) : "memory");
      s_last = before == a.k - 1;
      if (s_last) a.done[sent] = 0;
    }
    __syncthreads();
    last = s_last;
  }
  if (last) beam_select_block<THREADS>(a, cand, sent, T, osent, nf0, smraw);
}

// Pass 1 finds the row maximum and, from 32 maxima over groups of threads, a threshold that at least
// kk elements reach (the kk-th largest of them).  Pass 2 (the row is L2/L1 resident by
// then) sums exp(z - max) and collects the few elements at or above the threshold, which are
// then ranked exactly.  If more elements than the candidate buffer holds reach the threshold
// (e.g. a row of equal logits) the block falls back to kk exact arg-best sweeps.
constexpr int kTopkCap = 1024;
// What both softmax kernels do once the candidates of a row are listed (sh.cv, sh.ci, sh.count) and each thread holds its
// share `ssum` of the sum of exp(z - rmax): log-sum, accurate values of the candidates (refinement), exact ranking.
struct TopkShared {
  float cv[kTopkCap];
  int ci[kTopkCap];
  float cd[kTopkCap];   // refinement: change of exp(z - max) per candidate, in buffer order ...
  float co[kTopkCap];   // ... and in vocabulary order
  float red[32];
  int redi[32];
  float part[32];       // the warps' shares of the sum
  int count, n_blocks;
  float lse, eos, eos_delta, eos_half[2];
};
// (once a row's results are written, the selection has the memory)
union TopkSmem {
  TopkShared sh;
  unsigned char sel[kSelectSmem];
};
template <int THREADS>
__device__ __forceinline__ void topk_finish(TopkShared& sh, int r, float ssum, float rmax, const float* __restrict__ z, const __half* __restrict__ zh,
                                            int V, int kk, const TopkOut& out, int normalise, const TopkRefine& rf, const float* s_a) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  auto zat = [&](int i) { return zh ? __half2float(zh[i]) : z[i]; };
  ssum = warp_sum(ssum);
  if (lane == 0) sh.part[warp] = ssum;
  const float z_eos = !rf.a0 && warp == 0 ? zat(kEos) : 0.f;
  int n = sh.count;
  if (rf.a0 && n > kTopkCap) {
    // More elements than the buffer holds reach the widened threshold (a nearly flat row): pick the kk best
    // of the one-product logits by exact sweeps and make those the candidates.  Their values are refined
    // like any others below; an element within the error bound just beyond the kk-th can be missed here,
    // which on a row this flat is a tie within the tolerance.
    float last_v = INFINITY;
    int last_i = -1;
    for (int round = 0; round < kk; ++round) {
      float bv = -INFINITY;
      int bi = 0x7fffffff;
      for (int i = tid; i < V; i += THREADS) {
        const float v = zat(i);
        const bool after = (v < last_v) || (v == last_v && i > last_i);
        if (after && better(v, i, bv, bi)) { bv = v; bi = i; }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (better(ov, oi, bv, bi)) { bv = ov; bi = oi; }
      }
      __syncthreads();
      if (lane == 0) { sh.red[warp] = bv; sh.redi[warp] = bi; }
      __syncthreads();
      bv = sh.red[0]; bi = sh.redi[0];
      for (int w = 1; w < THREADS / 32; ++w) if (better(sh.red[w], sh.redi[w], bv, bi)) { bv = sh.red[w]; bi = sh.redi[w]; }
      if (tid == 0) { sh.cv[round] = bv; sh.ci[round] = bi; }
      last_v = bv; last_i = bi;
    }
    __syncthreads();
    n = 0;
    while (n < kk && sh.ci[n] != 0x7fffffff) ++n;   // fewer than kk elements in the row
    __syncthreads();
    if (tid == 0) sh.count = n;
  }
  if (rf.a0) {
    // accurate values for the candidates (and for EOS, whose log-probability is always reported): one
    // warp per candidate, fp32 FMAs over the two planes of both operands.  Each also yields the term by
    // which the row's sum of exponentials changes when the accurate value replaces the one-product one:
    // on a peaked row the few dominant logits ARE the normaliser, and their fp16-product error would
    // otherwise go straight into every log-probability of the row.
    const int nc = n;
    // the dot product of a stretch of the row with the same stretch of weight row v, eight values to a lane and load
    auto dot = [&](int v, int j0, int j1) {
      const __half* w0 = rf.b0 + (size_t)v * rf.ldb;
      const __half* w1 = rf.b1 + (size_t)v * rf.ldb;
      float acc = 0.f;
#pragma unroll 2
      for (int j = j0 + lane * 8; j < j1; j += 256) {
        const uint4 q0 = *reinterpret_cast<const uint4*>(w0 + j), q1 = *reinterpret_cast<const uint4*>(w1 + j);
        const uint32_t u0[4] = {q0.x, q0.y, q0.z, q0.w}, u1[4] = {q1.x, q1.y, q1.z, q1.w};
        const float4 x[2] = {*reinterpret_cast<const float4*>(s_a + j), *reinterpret_cast<const float4*>(s_a + j + 4)};
        const float* xs = reinterpret_cast<const float*>(x);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 f0 = __half22float2(*reinterpret_cast<const __half2*>(&u0[i])), f1 = __half22float2(*reinterpret_cast<const __half2*>(&u1[i]));
          acc = fmaf(xs[2 * i], fmaf(f1.x, kPairInv, f0.x), acc);
          acc = fmaf(xs[2 * i + 1], fmaf(f1.y, kPairInv, f0.y), acc);
        }
      }
      return warp_sum(acc);
    };
    auto done = [&](int c, float acc, float bias, float za) {
      const float zv = acc + bias;
      const float delta = __expf(zv - rmax) - __expf(za - rmax);
      if (c < nc) { sh.cv[c] = zv; sh.cd[c] = delta; }
      else { sh.eos = zv; sh.eos_delta = delta; }
    };
    if constexpr (THREADS > 256) {
      // Few rows: the weight rows come from HBM, and their latency is most of the time.  Two warps share a candidate, so that
      // all that a lane wants is in flight at once (K = 1024: four loads of 16 bytes): 5.2 us with a warp each.
      float bias = 0.f, za = 0.f;      // (a thread completes a candidate; what it needs for that is requested first)
      if (tid <= nc) {
        const int v = tid < nc ? sh.ci[tid] : kEos;
        bias = rf.bias ? rf.bias[v] : 0.f;
        za = tid < nc ? sh.cv[tid] : zat(kEos);
      }
      const int half = warp & 1, mid = (rf.K >> 1) & ~7;
      for (int c = warp >> 1; c <= nc; c += THREADS / 64) {
        const float acc = dot(c < nc ? sh.ci[c] : kEos, half ? mid : 0, half ? rf.K : mid);
        if (lane == 0) { if (c < nc) (half ? sh.co : sh.cd)[c] = acc; else sh.eos_half[half] = acc; }
      }
      __syncthreads();
      if (tid <= nc) done(tid, tid < nc ? sh.cd[tid] + sh.co[tid] : sh.eos_half[0] + sh.eos_half[1], bias, za);
      if (nc == THREADS && tid == 0) done(nc, sh.eos_half[0] + sh.eos_half[1], rf.bias ? rf.bias[kEos] : 0.f, zat(kEos));
    } else {
      for (int c = warp; c <= nc; c += THREADS / 32) {
        const int v = (c < nc) ? sh.ci[c] : kEos;
        // (what the sum is completed with is requested together with the weights)
        const float bias = rf.bias ? rf.bias[v] : 0.f;
        const float za = (c < nc) ? sh.cv[c] : zat(kEos);
        const float acc = dot(v, 0, rf.K);
        if (lane == 0) done(c, acc, bias, za);
      }
    }
  }
  __syncthreads();
  // The rest is a warp's work while the candidates are no more than its lanes (13 to 17 at a beam of 12): in registers,
  // without a barrier.  The correction is summed in vocabulary order, so the result does not depend on the order in
  // which the candidates happened to enter the buffer.
  if (n <= 32) {
    if (warp != 0) return;
    const bool in = lane < n;
    const float v = in ? sh.cv[lane] : -INFINITY;
    const int i = in ? sh.ci[lane] : 0x7fffffff;
    float sum = warp_sum(lane < THREADS / 32 ? sh.part[lane] : 0.f);
    int pos = 0, rank = 0;
#pragma unroll 4
    for (int d = 0; d < n; ++d) {
      const float ov = __shfl_sync(0xffffffffu, v, d);
      const int oi = __shfl_sync(0xffffffffu, i, d);
      pos += oi < i ? 1 : 0;
      rank += better(ov, oi, v, i) ? 1 : 0;
    }
    float eos = z_eos;
    if (rf.a0) {
      if (in) sh.co[pos] = sh.cd[lane];
      __syncwarp();
      float corr = warp_sum(in ? sh.co[lane] : 0.f);
      if (!__any_sync(0xffffffffu, in && i == kEos)) corr += sh.eos_delta;
      if (sum + corr > 0.f) sum += corr;
      eos = sh.eos;
    }
    const float lse = normalise ? logf(sum) : -rmax;   // normalise = 0: the row already holds log-probabilities
    if (in && rank < kk) {
      out.idx[(size_t)r * kk + rank] = i;
      out.logp[(size_t)r * kk + rank] = (v - rmax) - lse;
    }
    if (n + lane < kk) {       // fewer than kk elements in the row
      out.idx[(size_t)r * kk + n + lane] = -1;
      out.logp[(size_t)r * kk + n + lane] = -INFINITY;
    }
    if (lane == 0) {
      if (out.eos_logp) out.eos_logp[r] = (eos - rmax) - lse;
      if (out.row_stats) { out.row_stats[2 * r] = rmax; out.row_stats[2 * r + 1] = lse; }
    }
    return;
  }
  if (rf.a0 && n <= kTopkCap) {
    for (int c = tid; c < n; c += THREADS) {
      const int i = sh.ci[c];
      int pos = 0;
      for (int d = 0; d < n; ++d) pos += (sh.ci[d] < i) ? 1 : 0;
      sh.co[pos] = sh.cd[c];
    }
    __syncthreads();
  }
  if (warp == 0) {
    float sum = warp_sum(lane < THREADS / 32 ? sh.part[lane] : 0.f);
    float eos = z_eos;
    if (rf.a0) {
      float corr = 0.f;
      bool eos_listed = false;
      for (int c = lane; c < n; c += 32) { corr += sh.co[c]; eos_listed = eos_listed || (sh.ci[c] == kEos); }
      corr = warp_sum(corr);
      if (!__any_sync(0xffffffffu, eos_listed)) corr += sh.eos_delta;
      if (sum + corr > 0.f) sum += corr;
      eos = sh.eos;
    }
    if (lane == 0) {
      sh.lse = normalise ? logf(sum) : -rmax;
      if (out.eos_logp) out.eos_logp[r] = (eos - rmax) - sh.lse;
      if (out.row_stats) { out.row_stats[2 * r] = rmax; out.row_stats[2 * r + 1] = sh.lse; }
    }
  }
  __syncthreads();
  const float rlse = sh.lse;
  if (n <= kTopkCap) {
    // exact ranking of the candidates: value descending, index ascending
    for (int c = tid; c < n; c += THREADS) {
      const float v = sh.cv[c];
      const int i = sh.ci[c];
      int rank = 0;
      for (int d = 0; d < n; ++d) rank += better(sh.cv[d], sh.ci[d], v, i) ? 1 : 0;
      if (rank < kk) {
        out.idx[(size_t)r * kk + rank] = i;
        out.logp[(size_t)r * kk + rank] = (v - rmax) - rlse;
      }
    }
    for (int q = n + tid; q < kk; q += THREADS) {  // fewer than kk elements in the row
      out.idx[(size_t)r * kk + q] = -1;
      out.logp[(size_t)r * kk + q] = -INFINITY;
    }
    return;
  }
  // ---- fallback: kk sweeps, each picking the best element after the previous pick ----
  float last_v = INFINITY;
  int last_i = -1;
  for (int round = 0; round < kk; ++round) {
    float bv = -INFINITY;
    int bi = 0x7fffffff;
    for (int i = tid; i < V; i += THREADS) {
      const float v = zat(i);
      const bool after = (v < last_v) || (v == last_v && i > last_i);
      if (after && better(v, i, bv, bi)) { bv = v; bi = i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (better(ov, oi, bv, bi)) { bv = ov; bi = oi; }
    }
    __syncthreads();
    if (lane == 0) { sh.red[warp] = bv; sh.redi[warp] = bi; }
    __syncthreads();
    bv = sh.red[0]; bi = sh.redi[0];
    for (int w = 1; w < THREADS / 32; ++w) if (better(sh.red[w], sh.redi[w], bv, bi)) { bv = sh.red[w]; bi = sh.redi[w]; }
    if (tid == 0) {
      const bool valid = bi != 0x7fffffff;
      out.idx[(size_t)r * kk + round] = valid ? bi : -1;
      out.logp[(size_t)r * kk + round] = valid ? ((bv - rmax) - rlse) : -INFINITY;
    }
    last_v = bv; last_i = bi;
  }
}

static __global__ void __launch_bounds__(256, 6) softmax_topk_kernel(const float* __restrict__ logits, int ld, int V, int kk, TopkOut out,
                                                                  int normalise, const float* __restrict__ pmax, int pmax_ld, int n_slots, TopkRefine rf,
                                                                  const __half* __restrict__ logits16, const __grid_constant__ SelectArgs sel) {
  extern __shared__ __align__(16) float s_a[];   // [rf.K] the row's activations in fp32 (refinement only)
  tc::pdl_launch_dependents();   // see gemm_tc.cuh: the next kernel of the step may start its prologue
  tc::pdl_wait();                // nothing below runs before the previous kernel's results are visible
  __shared__ float s_tmax[256];
  __shared__ __align__(16) unsigned char s_union[sizeof(TopkSmem)];
  TopkShared& sh = *reinterpret_cast<TopkShared*>(s_union);
  __shared__ float s_tau, s_max;
  const int r = blockIdx.x, tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31;
  const float* z = logits + (size_t)r * ld;
  // fp16 logits (refinement mode only: the candidates' values are recomputed, the rest only enter the sum)
  const __half* zh = logits16 ? logits16 + (size_t)r * ld : nullptr;
  const int V4 = V & ~3;
  // ---- pass 1: maxima (four independent 16-byte loads in flight per thread) -- or, when the GEMM that
  // produced the logits left the maxima of disjoint column blocks of every row (pmax), just those ----
  float m = -INFINITY;
  if (pmax) {
    for (int s = tid; s < n_slots; s += 256) m = fmaxf(m, pmax[(size_t)r * pmax_ld + s]);
  } else if (zh) {
    for (int i = tid; i < V; i += 256) m = fmaxf(m, __half2float(zh[i]));
  } else {
    float m0 = -INFINITY, m1 = -INFINITY, m2 = -INFINITY, m3 = -INFINITY;
    int i = tid * 4;
    for (; i + 3 * 1024 < V4; i += 4 * 1024) {
      const float4 q0 = *reinterpret_cast<const float4*>(z + i);
      const float4 q1 = *reinterpret_cast<const float4*>(z + i + 1024);
      const float4 q2 = *reinterpret_cast<const float4*>(z + i + 2048);
      const float4 q3 = *reinterpret_cast<const float4*>(z + i + 3072);
      m0 = fmaxf(fmaxf(m0, q0.x), fmaxf(q0.y, fmaxf(q0.z, q0.w)));
      m1 = fmaxf(fmaxf(m1, q1.x), fmaxf(q1.y, fmaxf(q1.z, q1.w)));
      m2 = fmaxf(fmaxf(m2, q2.x), fmaxf(q2.y, fmaxf(q2.z, q2.w)));
      m3 = fmaxf(fmaxf(m3, q3.x), fmaxf(q3.y, fmaxf(q3.z, q3.w)));
    }
    for (; i < V4; i += 1024) {
      const float4 q = *reinterpret_cast<const float4*>(z + i);
      m0 = fmaxf(fmaxf(m0, q.x), fmaxf(q.y, fmaxf(q.z, q.w)));
    }
    m = fmaxf(fmaxf(m0, m1), fmaxf(m2, m3));
    for (int i = V4 + tid; i < V; i += 256) m = fmaxf(m, z[i]);
  }
  s_tmax[tid] = m;
  if (tid == 0) sh.count = 0;
  __syncthreads();
  // Threshold from 32 group maxima (group = the 8 threads with the same lane): each is an
  // element of the row and the groups are disjoint, so at least kk (at most 32) elements reach the kk-th
  // largest of them; it is a little lower than the kk-th largest thread maximum (a few more
  // candidates to rank) and costs one warp ~100 instructions instead of 256 x 256 compares.
  if (warp == 0) {
    float g = -INFINITY;
#pragma unroll
    for (int w = 0; w < 8; ++w) g = fmaxf(g, s_tmax[w * 32 + lane]);
    float bm = g;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) bm = fmaxf(bm, __shfl_xor_sync(0xffffffffu, bm, o));
    int rank = 0;
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      const float o = __shfl_sync(0xffffffffu, g, j);
      rank += (o > g || (o == g && j < lane)) ? 1 : 0;
    }
    if (rank == kk - 1) s_tau = g;
    if (lane == 0) s_max = bm;
  }
  __syncthreads();
  if (pmax) {
    // The threshold from 32 group maxima admits a few dozen elements.  A tighter one costs little here: the
    // block maxima that reach it are few, each is an element of the row, the blocks are disjoint, and the
    // kk-th largest of them is still reached by at least kk elements.
    const float tau0 = s_tau;
    for (int sl = tid; sl < n_slots; sl += 256) {
      const float v = pmax[(size_t)r * pmax_ld + sl];
      if (v >= tau0) {
        const int pos = atomicAdd(&sh.count, 1);
        if (pos < kTopkCap) sh.cv[pos] = v;
      }
    }
    __syncthreads();
    const int m2 = sh.count;
    if (m2 <= kTopkCap)
      for (int c = tid; c < m2; c += 256) {
        const float v = sh.cv[c];
        int rank = 0;
        for (int d = 0; d < m2; ++d) rank += (sh.cv[d] > v || (sh.cv[d] == v && d < c)) ? 1 : 0;
        if (rank == kk - 1) s_tau = v;
      }
    __syncthreads();
    if (tid == 0) sh.count = 0;
    __syncthreads();
  }
  float tau = s_tau;
  const float rmax = s_max;
  if (rf.a0) {
    // Every logit in this row is within eps of its accurate value, so the accurate top-kk all lie at or
    // above (kk-th largest approximate value) - 2 eps, and tau is no larger than that kk-th value.
    float ss = 0.f;
    for (int j = tid; j < rf.K; j += 256) {
      const float a = __half2float(rf.a0[(size_t)r * rf.lda + j]) + __half2float(rf.a1[(size_t)r * rf.lda + j]) * kPairInv;
      s_a[j] = a;
      ss = fmaf(a, a, ss);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (lane == 0) sh.red[warp] = ss;
    __syncthreads();
    float tot = 0.f;
    for (int w = 0; w < 8; ++w) tot += sh.red[w];
    tau -= 2.0f * (rf.eps_coef * sqrtf(tot) + 1e-5f);   // + fp16 subnormals and the accumulator's own rounding
    if (zh) tau -= 2.0f * 4.9e-4f * fmaxf(fabsf(rmax), fabsf(tau));   // and the rounding of the stored value (2^-11 relative)
    __syncthreads();
  }
  // ---- pass 2: sum of exponentials, candidates ----
  float ssum = 0.f;
  auto visit = [&](float v, int i) {
    ssum += __expf(v - rmax);  // arguments in [-few, 0]: ~1e-7 relative on the sum of V terms
    if (v >= tau) {
      const int pos = atomicAdd(&sh.count, 1);
      if (pos < kTopkCap) { sh.cv[pos] = v; sh.ci[pos] = i; }
    }
  };
  {
    // four independent 16-byte loads in flight per thread; candidates are rare, so a group of four is
    // first tested as a whole against the threshold
    auto group = [&](const float4& q, int i) {
      ssum += __expf(q.x - rmax) + __expf(q.y - rmax);
      ssum += __expf(q.z - rmax) + __expf(q.w - rmax);
      if (fmaxf(fmaxf(q.x, q.y), fmaxf(q.z, q.w)) >= tau) {
        const float v[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (v[u] >= tau) {
            const int pos = atomicAdd(&sh.count, 1);
            if (pos < kTopkCap) { sh.cv[pos] = v[u]; sh.ci[pos] = i + u; }
          }
      }
    };
    if (zh) {
      // eight values per 16-byte load, blocks of 2048 columns, from the last one down
      auto group8 = [&](const uint4& q, int i) {
        const __half2* h = reinterpret_cast<const __half2*>(&q);
        const float2 a = __half22float2(h[0]), b = __half22float2(h[1]), c = __half22float2(h[2]), d = __half22float2(h[3]);
        group(make_float4(a.x, a.y, b.x, b.y), i);
        group(make_float4(c.x, c.y, d.x, d.y), i + 4);
      };
      const int V8 = V & ~7;
      const int top8 = V8 & ~2047;
      if (top8 + tid * 8 < V8) group8(*reinterpret_cast<const uint4*>(zh + top8 + tid * 8), top8 + tid * 8);
      int i = top8 - 2048 + tid * 8;
      for (; i - 3 * 2048 >= 0; i -= 4 * 2048) {
        const uint4 q0 = *reinterpret_cast<const uint4*>(zh + i);
        const uint4 q1 = *reinterpret_cast<const uint4*>(zh + i - 2048);
        const uint4 q2 = *reinterpret_cast<const uint4*>(zh + i - 4096);
        const uint4 q3 = *reinterpret_cast<const uint4*>(zh + i - 6144);
        group8(q0, i); group8(q1, i - 2048); group8(q2, i - 4096); group8(q3, i - 6144);
      }
      for (; i >= 0; i -= 2048) group8(*reinterpret_cast<const uint4*>(zh + i), i);
      for (int j = V8 + tid; j < V; j += 256) visit(__half2float(zh[j]), j);
    } else {
    // From the last column block down: the GEMM that wrote the logits walked the column tiles upwards, so the
    // highest columns of every row are the ones still in L2 (all rows are swept at the same time).
    const int top = V4 & ~1023;                       // start of the last, possibly partial, block of 1024
    if (top + tid * 4 < V4) group(*reinterpret_cast<const float4*>(z + top + tid * 4), top + tid * 4);
    int i = top - 1024 + tid * 4;
    for (; i - 3 * 1024 >= 0; i -= 4 * 1024) {
      const float4 q0 = *reinterpret_cast<const float4*>(z + i);
      const float4 q1 = *reinterpret_cast<const float4*>(z + i - 1024);
      const float4 q2 = *reinterpret_cast<const float4*>(z + i - 2048);
      const float4 q3 = *reinterpret_cast<const float4*>(z + i - 3072);
      group(q0, i); group(q1, i - 1024); group(q2, i - 2048); group(q3, i - 3072);
    }
    for (; i >= 0; i -= 1024) group(*reinterpret_cast<const float4*>(z + i), i);
    for (int j = V4 + tid; j < V; j += 256) visit(z[j], j);
    }
  }
  __syncthreads();
  topk_finish<256>(sh, r, ssum, rmax, z, zh, V, kk, out, normalise, rf, s_a);
  select_if_last<256>(sel, out, r, s_union);
}

// The same result when the GEMM that produced the logits left, for every block of up to 64 columns of a row, the block's
// maximum AND its sum of exp(z - maximum) (TcEpiF32): the row itself is not swept.  The maximum, the sum and the threshold
// come from the blocks (580 or 940 pairs for 30,000 classes), and only blocks whose maximum reaches the threshold are
// looked into.  THREADS = 1024 for few rows, whose one CTA each has an SM to itself and is bound by the chain of its memory
// round trips (one sentence at 12 rows, 30k classes: 22.2 us per step sweeping, 13.1 so); 256 otherwise, where the sweep
// read what the GEMM had just written.
// grid = rows, dynamic smem = topk_blocks_smem
// The block statistics of a row and its activations lie in shared memory beside the candidate lists (18 or 21 KB, of the 48
// a launch may use unasked): rows that need more than this are swept, which includes 80,000 classes in the few-rows kernel's
// blocks of 32 columns (2500 pairs, 24.1 KB with the activations of 1024 units, 20.0 without).
constexpr int kBlocksSmemMax = 23 * 1024;
struct LogitBlocks {
  float* max; float* sum; int ld; int n;
  int tile, part;     // columns of a GEMM tile and of one of its four blocks (the last one of a tile may be narrower)
};
inline size_t topk_blocks_smem(int n_blocks, int refine_K) { return sizeof(float) * (size_t)(2 * n_blocks + refine_K); }
// LATE: the next kernel runs beside this one and reads what this one has waited for, without a wait of its own: it may start
// only behind that wait.
template <int THREADS, bool LATE>
static __global__ void __launch_bounds__(THREADS, THREADS == 256 ? 6 : 1) topk_blocks_kernel(const float* __restrict__ logits, const __half* __restrict__ logits16, int ld, int V, int kk,
                                                                           TopkOut out, int normalise, LogitBlocks bl, TopkRefine rf, const __grid_constant__ SelectArgs sel) {
  if (!LATE) tc::pdl_launch_dependents();
  tc::pdl_wait();
  if (LATE) tc::pdl_launch_dependents();
  extern __shared__ __align__(16) float dyn[];
  float* s_m = dyn;                  // [n] block maxima
  float* s_q = dyn + bl.n;           // [n] block sums
  float* s_a = dyn + 2 * bl.n;       // [rf.K] activations (refinement)
  __shared__ __align__(16) unsigned char s_union[sizeof(TopkSmem)];
  TopkShared& sh = *reinterpret_cast<TopkShared*>(s_union);
  __shared__ float s_tmax[THREADS];
  __shared__ float s_tau, s_max, s_eps;
  const int r = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const float* z = logits ? logits + (size_t)r * ld : nullptr;
  const __half* zh = logits16 ? logits16 + (size_t)r * ld : nullptr;
  // (the activations are requested before the blocks are waited for; K is a multiple of 64)
  uint2 q0 = make_uint2(0u, 0u), q1 = make_uint2(0u, 0u);
  auto act_load = [&](int j) {
    q0 = *reinterpret_cast<const uint2*>(rf.a0 + (size_t)r * rf.lda + j);
    q1 = *reinterpret_cast<const uint2*>(rf.a1 + (size_t)r * rf.lda + j);
  };
  if (rf.a0 && tid * 4 < rf.K) act_load(tid * 4);
  float m = -INFINITY;
  for (int b = tid; b < bl.n; b += THREADS) {
    const float v = bl.max[(size_t)r * bl.ld + b];
    s_q[b] = bl.sum[(size_t)r * bl.ld + b];
    s_m[b] = v;
    m = fmaxf(m, v);
  }
  s_tmax[tid] = m;
  if (tid == 0) { sh.count = 0; sh.n_blocks = 0; s_tau = -INFINITY; }
  if (rf.a0) {
    float ss = 0.f;
    for (int j = tid * 4; j < rf.K; j += THREADS * 4) {
      if (j >= THREADS * 4) act_load(j);
      const float2 f0 = __half22float2(*reinterpret_cast<const __half2*>(&q0.x)), f1 = __half22float2(*reinterpret_cast<const __half2*>(&q0.y));
      const float2 g0 = __half22float2(*reinterpret_cast<const __half2*>(&q1.x)), g1 = __half22float2(*reinterpret_cast<const __half2*>(&q1.y));
      const float4 a = make_float4(f0.x + g0.x * kPairInv, f0.y + g0.y * kPairInv, f1.x + g1.x * kPairInv, f1.y + g1.y * kPairInv);
      s_a[j] = a.x; s_a[j + 1] = a.y; s_a[j + 2] = a.z; s_a[j + 3] = a.w;
      ss = fmaf(a.x, a.x, ss); ss = fmaf(a.y, a.y, ss); ss = fmaf(a.z, a.z, ss); ss = fmaf(a.w, a.w, ss);
    }
    ss = warp_sum(ss);
    if (lane == 0) sh.red[warp] = ss;
  }
  __syncthreads();
  if (warp == 0) {
    // threshold from 32 group maxima, as in softmax_topk_kernel (kk <= 32)
    float g = -INFINITY;
#pragma unroll
    for (int w = 0; w < THREADS / 32; ++w) g = fmaxf(g, s_tmax[w * 32 + lane]);
    float bm = g;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) bm = fmaxf(bm, __shfl_xor_sync(0xffffffffu, bm, o));
    int rank = 0;
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      const float o = __shfl_sync(0xffffffffu, g, j);
      rank += (o > g || (o == g && j < lane)) ? 1 : 0;
    }
    if (rank == kk - 1) s_tau = g;
    const float tot = rf.a0 ? warp_sum(lane < THREADS / 32 ? sh.red[lane] : 0.f) : 0.f;
    if (lane == 0) { s_max = bm; s_eps = rf.a0 ? 2.0f * (rf.eps_coef * sqrtf(tot) + 1e-5f) : 0.f; }
  }
  __syncthreads();
  const float rmax = s_max, tau0 = s_tau, eps = s_eps;
  // refinement: every logit is within eps of its accurate value (see softmax_topk_kernel)
  auto lowered = [&](float t) {
    if (!rf.a0) return t;
    t -= eps;
    return zh ? t - 2.0f * 4.9e-4f * fmaxf(fabsf(rmax), fabsf(t)) : t;
  };
  // the sum, and the list of the blocks that reach the (lowered) threshold: sh.cd their maxima, sh.co their numbers
  float* lv = sh.cd;
  int* lb = reinterpret_cast<int*>(sh.co);
  float ssum = 0.f;
  float tau = lowered(tau0);
  for (int b = tid; b < bl.n; b += THREADS) {
    const float v = s_m[b];
    if (v > -INFINITY) ssum = fmaf(s_q[b], __expf(v - rmax), ssum);
    if (v >= tau) {
      const int pos = atomicAdd(&sh.n_blocks, 1);
      if (pos < kTopkCap) { lv[pos] = v; lb[pos] = b; }
    }
  }
  __syncthreads();
  const int n_list = sh.n_blocks;
  // tighter: the kk-th largest of those maxima is still reached by kk elements (a warp ranks a block)
  if (n_list <= kTopkCap)
    for (int c = warp; c < n_list; c += THREADS / 32) {
      const float v = lv[c];
      int rank = 0;
      for (int d0 = 0; d0 < n_list; d0 += 32) {
        const int d = d0 + lane;
        const float o = d < n_list ? lv[d] : -INFINITY;
        rank += __popc(__ballot_sync(0xffffffffu, d < n_list && (o > v || (o == v && d < c))));
      }
      if (rank == kk - 1 && lane == 0) s_tau = v;
    }
  __syncthreads();
  tau = lowered(s_tau);
  // a warp reads a block
  auto read_block = [&](int b) {
    const int in_tile = (b & 3) * bl.part, c0 = (b >> 2) * bl.tile + in_tile;
    const int end = c0 + (bl.tile - in_tile < bl.part ? bl.tile - in_tile : bl.part);
    float v[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int i = c0 + lane + 32 * u;
      v[u] = i < end && i < V ? (zh ? __half2float(zh[i]) : z[i]) : -INFINITY;
    }
#pragma unroll
    for (int u = 0; u < 2; ++u)
      if (v[u] >= tau && v[u] > -INFINITY) {
        const int pos = atomicAdd(&sh.count, 1);
        if (pos < kTopkCap) { sh.cv[pos] = v[u]; sh.ci[pos] = c0 + lane + 32 * u; }
      }
  };
  if (n_list <= kTopkCap) {
    for (int c = warp; c < n_list; c += THREADS / 32)
      if (lv[c] >= tau) read_block(lb[c]);
  } else {
    for (int b = warp; b < bl.n; b += THREADS / 32)
      if (s_m[b] >= tau) read_block(b);
  }
  __syncthreads();     // (the list has been read by every warp)
  topk_finish<THREADS>(sh, r, ssum, rmax, z, zh, V, kk, out, normalise, rf, s_a);
  select_if_last<THREADS>(sel, out, r, s_union);
}

inline cudaError_t launch_softmax_topk(const float* logits, int ld, int V, int kk, int rows, const TopkOut& out, int normalise,
                                       cudaStream_t st, bool pdl = false, const float* pmax = nullptr, int pmax_ld = 0, int n_slots = 0,
                                       const TopkRefine* refine = nullptr, const __half* logits16 = nullptr, const SelectArgs& sel = SelectArgs{}) {
  if (n_slots <= 0) pmax = nullptr;
  TopkRefine rf{};
  if (refine) rf = *refine;
  const size_t smem = rf.a0 ? sizeof(float) * (size_t)rf.K : 0;
  // (models of more than 7680 hidden units)
  if (cudaError_t e = tc::allow_smem<softmax_topk_kernel>(smem); e != cudaSuccess) return e;
  return tc::launch_k(pdl, softmax_topk_kernel, dim3(rows), dim3(256), smem, st, logits, ld, V, kk, out, normalise, pmax, pmax_ld, n_slots, rf, refine ? logits16 : (const __half*)nullptr, sel);
}

// What block statistics a logits GEMM of N columns is going to leave in rows of `ld` values: four blocks of `part` columns
// per tile of `tile`.  n = 0: none, sum = null: the maxima only.
inline LogitBlocks logit_blocks(float* max, float* sum, int ld, int N, int K, int tile, int part) {
  const int slots = tile > 0 ? 4 * ((N + tile - 1) / tile) : 0;
  if (!max || slots < 1 || slots > ld) return LogitBlocks{};
  if (topk_blocks_smem(slots, K) > (size_t)kBlocksSmemMax) sum = nullptr;
  return LogitBlocks{max, sum, ld, slots, tile, part};
}
// Values a row of block statistics has room for: four column blocks per tile, tiles at least 48 wide.
inline int logit_blocks_ld(int N) { return 4 * ((N + 47) / 48) + 4; }

// Softmax statistics and top-k (and the selection) of rows of logits, from their block statistics where they have them.  late: see
// topk_blocks_kernel, where topk_late says that the launch can.
inline bool topk_late(const LogitBlocks& bl, int rows, int n_sm) { return bl.sum && rows <= n_sm; }
inline cudaError_t launch_topk(const float* logits, const __half* logits16, int ld, int V, int kk, int rows, int n_sm, const TopkOut& o, int normalise,
                               const LogitBlocks& bl, const TopkRefine* rf, const SelectArgs& sel, cudaStream_t st, bool pdl, bool late = false) {
  if (!bl.sum) return launch_softmax_topk(logits, ld, V, kk, rows, o, normalise, st, pdl, bl.max, bl.ld, bl.n, rf, logits16, sel);
  const bool wide = rows <= n_sm;
  auto* kernel = !wide ? topk_blocks_kernel<256, false> : late ? topk_blocks_kernel<1024, true> : topk_blocks_kernel<1024, false>;
  return tc::launch_k(pdl, kernel, dim3(rows), dim3(wide ? 1024 : 256), topk_blocks_smem(bl.n, rf ? rf->K : 0), st,
                      logits, logits16, ld, V, kk, o, normalise, bl, rf ? *rf : TopkRefine{}, sel);
}

// Log-probability of one given token per row (scoring), from the row's softmax statistics; with one-product logits the
// token's logit is recomputed from both planes of both operands, like the candidates above.  One warp per row.
static __global__ void __launch_bounds__(256) gold_logp_kernel(const int32_t* __restrict__ gold, int rows, const float* __restrict__ logits, int ld, int V,
                                                               const float* __restrict__ row_stats, TopkRefine rf, float* __restrict__ out) {
  tc::pdl_launch_dependents();
  tc::pdl_wait();
  const int r = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (r >= rows) return;
  int g = gold[r];
  if (g < 0) g = 0;
  if (g >= V) g = kUnk;
  float zv = 0.f;
  if (rf.a0) {
    const __half *a0 = rf.a0 + (size_t)r * rf.lda, *a1 = rf.a1 + (size_t)r * rf.lda;
    const __half *w0 = rf.b0 + (size_t)g * rf.ldb, *w1 = rf.b1 + (size_t)g * rf.ldb;
    float acc = 0.f;
    for (int j = lane; j < rf.K; j += 32) {
      const float x = fmaf(__half2float(a1[j]), kPairInv, __half2float(a0[j]));
      const float w = fmaf(__half2float(w1[j]), kPairInv, __half2float(w0[j]));
      acc = fmaf(x, w, acc);
    }
    zv = warp_sum(acc) + (rf.bias ? rf.bias[g] : 0.f);
  } else {
    zv = logits[(size_t)r * ld + g];
  }
  if (lane == 0) out[r] = (zv - row_stats[2 * r]) - row_stats[2 * r + 1];
}

// ---------------------------------------------------------------------------------------
// Ensemble of up to 8 members for one row: out[v] = log(mean_m softmax(z_m)[v]) (mode 0, the
// reference's rule, src/decoder.h:1913-1921 -- its renormalisation, :1923-1931, is the
// log-softmax the next kernel applies to this row) or mean_m log softmax(z_m)[v] (mode 1).
// Two sweeps over the members' rows (HBM-bound: each row of logits is read twice, the combined row
// written once): running (max, sum of exponentials) per member, then the combination.
// grid = rows, block = 256
struct EnsembleRows {
  const float* logits[8];
  int n;
};
static __global__ void __launch_bounds__(256) ensemble_combine_kernel(EnsembleRows er, int ld, int V, int mode, float* __restrict__ out) {
  tc::pdl_launch_dependents();   // see gemm_tc.cuh: the next kernel of the step may start its prologue
  tc::pdl_wait();                // nothing below runs before the previous kernel's results are visible
  __shared__ float s_m[8][8], s_s[8][8];   // [member][warp] partial (max, sum of exp relative to it)
  __shared__ float s_max[8], s_lse[8];
  const int r = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int V4 = V & ~3;
  // one sweep per member: running maximum and sum of exponentials relative to it (16-byte loads, two in flight)
  for (int m = 0; m < er.n; ++m) {
    const float* z = er.logits[m] + (size_t)r * ld;
    float mx = -INFINITY, sum = 0.f;
    auto take = [&](float x) {
      if (x > mx) { sum = sum * __expf(mx - x) + 1.0f; mx = x; }
      else sum += __expf(x - mx);
    };
    int i = tid * 4;
    for (; i + 1024 < V4; i += 2048) {
      const float4 q0 = *reinterpret_cast<const float4*>(z + i);
      const float4 q1 = *reinterpret_cast<const float4*>(z + i + 1024);
      take(q0.x); take(q0.y); take(q0.z); take(q0.w);
      take(q1.x); take(q1.y); take(q1.z); take(q1.w);
    }
    for (; i < V4; i += 1024) {
      const float4 q = *reinterpret_cast<const float4*>(z + i);
      take(q.x); take(q.y); take(q.z); take(q.w);
    }
    for (int j = V4 + tid; j < V; j += 256) take(z[j]);
    // combine (max, sum) pairs in a fixed order: lanes by shuffle tree, then the warps one after the other
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float om = __shfl_xor_sync(0xffffffffu, mx, o);
      const float os = __shfl_xor_sync(0xffffffffu, sum, o);
      const float nm = fmaxf(mx, om);
      sum = (nm == -INFINITY) ? 0.f : sum * __expf(mx - nm) + os * __expf(om - nm);
      mx = nm;
    }
    if (lane == 0) { s_m[m][warp] = mx; s_s[m][warp] = sum; }
  }
  __syncthreads();
  if (tid < er.n) {
    float mx = s_m[tid][0], sum = s_s[tid][0];
    for (int w = 1; w < 8; ++w) {
      const float om = s_m[tid][w], os = s_s[tid][w];
      const float nm = fmaxf(mx, om);
      sum = (nm == -INFINITY) ? 0.f : sum * __expf(mx - nm) + os * __expf(om - nm);
      mx = nm;
    }
    s_max[tid] = mx; s_lse[tid] = logf(sum);
  }
  __syncthreads();
  // second sweep: the members' probabilities (or log-probabilities) of four classes at a time, accumulated in
  // double like the reference's loop (src/decoder.h:1913-1921)
  float* o = out + (size_t)r * ld;
  for (int i = tid * 4; i < V4; i += 1024) {
    double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
    for (int m = 0; m < er.n; ++m) {
      const float4 q = *reinterpret_cast<const float4*>(er.logits[m] + (size_t)r * ld + i);
      const float c = s_max[m] + s_lse[m];
      const float l0 = q.x - c, l1 = q.y - c, l2 = q.z - c, l3 = q.w - c;   // (z - max) - lse up to one rounding
      if (mode == 0) { a0 += (double)expf(l0); a1 += (double)expf(l1); a2 += (double)expf(l2); a3 += (double)expf(l3); }
      else { a0 += (double)l0; a1 += (double)l1; a2 += (double)l2; a3 += (double)l3; }
    }
    float4 w;
    if (mode == 0) w = make_float4(logf((float)(a0 / er.n)), logf((float)(a1 / er.n)), logf((float)(a2 / er.n)), logf((float)(a3 / er.n)));
    else w = make_float4((float)(a0 / er.n), (float)(a1 / er.n), (float)(a2 / er.n), (float)(a3 / er.n));
    *reinterpret_cast<float4*>(o + i) = w;
  }
  for (int j = V4 + tid; j < V; j += 256) {
    double acc = 0.0;
    for (int m = 0; m < er.n; ++m) {
      const float lp = er.logits[m][(size_t)r * ld + j] - (s_max[m] + s_lse[m]);
      acc += (mode == 0) ? (double)expf(lp) : (double)lp;
    }
    acc /= er.n;
    o[j] = (mode == 0) ? logf((float)acc) : (float)acc;
  }
}

// Ensembles: combination, log-softmax and top-kk of a row in one pass over the members' logits.  A member's maximum and
// log-sum come from its block statistics if the GEMM left them (otherwise from a sweep of its own); the pass then forms the
// combined value of every class -- mean of the probabilities (mode 0) or of the log-probabilities (mode 1), accumulated
// in double like the reference's loop -- keeps the maximum of every 128 classes and the sum, and only the blocks that reach
// the threshold are formed again to list their candidates.  The combined row itself is never written, and the logits are
// read once: (M + 1/16) x V x 4 bytes a row instead of (2 M + 2) x V x 4.  M = 4 at up to 384 rows, 30k classes: the two
// kernels took 224 us per step, this one 91, and 76 with the next block's loads in flight.
// THREADS = 1024 for rows that leave SMs empty.  grid = rows, dynamic smem = ceil(V / 128) floats.
template <int THREADS>
static __global__ void __launch_bounds__(THREADS, THREADS == 256 ? 3 : 1) ensemble_topk_kernel(const __grid_constant__ EnsembleRows er, int ld, int V, int kk, int mode, TopkOut out, LogitBlocks bl,
                                                                                             long long bl_member, float* __restrict__ combined, const __grid_constant__ SelectArgs sel) {
  tc::pdl_launch_dependents();
  tc::pdl_wait();
  constexpr int kWarps = THREADS / 32;
  extern __shared__ float s_bm[];            // [ceil(V / 128)] block maxima of the combined values
  __shared__ __align__(16) unsigned char s_union[sizeof(TopkSmem)];
  TopkShared& sh = *reinterpret_cast<TopkShared*>(s_union);
  __shared__ float s_m[8][kWarps], s_s[8][kWarps];
  __shared__ float s_c[8];                   // maximum + log-sum of a member
  __shared__ float s_tmax[THREADS], s_tau, s_eos[2];
  const int r = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int m = 0; m < er.n; ++m) {
    float mx = -INFINITY, sum = 0.f;
    auto join = [&](float om, float os) {
      const float nm = fmaxf(mx, om);
      sum = (nm == -INFINITY) ? 0.f : sum * __expf(mx - nm) + os * __expf(om - nm);
      mx = nm;
    };
    if (bl.n > 0) {
      const float* bm = bl.max + m * bl_member + (size_t)r * bl.ld;
      const float* bs = bl.sum + m * bl_member + (size_t)r * bl.ld;
      for (int b = tid; b < bl.n; b += THREADS) join(bm[b], bs[b]);
    } else {
      const float* z = er.logits[m] + (size_t)r * ld;
      for (int i = tid * 4; i < V; i += THREADS * 4) {
        const float4 q = *reinterpret_cast<const float4*>(z + i);     // (rows are padded)
        const float v[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int u = 0; u < 4; ++u) if (i + u < V) join(v[u], 1.f);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float om = __shfl_xor_sync(0xffffffffu, mx, o), os = __shfl_xor_sync(0xffffffffu, sum, o);
      join(om, os);
    }
    if (lane == 0) { s_m[m][warp] = mx; s_s[m][warp] = sum; }
  }
  if (tid == 0) sh.count = 0;
  __syncthreads();
  if (tid < er.n) {
    float mx = s_m[tid][0], sum = s_s[tid][0];
    for (int w = 1; w < kWarps; ++w) {
      const float om = s_m[tid][w], os = s_s[tid][w];
      const float nm = fmaxf(mx, om);
      sum = (nm == -INFINITY) ? 0.f : sum * __expf(mx - nm) + os * __expf(om - nm);
      mx = nm;
    }
    s_c[tid] = mx + logf(sum);
  }
  __syncthreads();
  // four classes from i on; what is compared is the mean probability (mode 0) or the mean log-probability (mode 1)
  const double n_members = er.n;
  const bool pow2 = (er.n & (er.n - 1)) == 0;        // then the division is an exact product
  const double inv_members = 1.0 / n_members;
  auto load4 = [&](int i, float4* q) {      // the first four members' loads, in flight together
#pragma unroll
    for (int m = 0; m < 4; ++m)
      if (m < er.n) q[m] = *reinterpret_cast<const float4*>(er.logits[m] + (size_t)r * ld + i);
  };
  auto combine4 = [&](int i, float4* q) {
    double a[4] = {0.0, 0.0, 0.0, 0.0};
    auto add = [&](int m, const float4& v) {
      const float c = s_c[m];
      const float l[4] = {v.x - c, v.y - c, v.z - c, v.w - c};
#pragma unroll
      for (int u = 0; u < 4; ++u) a[u] += mode == 0 ? (double)expf(l[u]) : (double)l[u];
    };
#pragma unroll
    for (int m = 0; m < 4; ++m)
      if (m < er.n) add(m, q[m]);
#pragma unroll 1
    for (int m = 4; m < er.n; ++m) add(m, *reinterpret_cast<const float4*>(er.logits[m] + (size_t)r * ld + i));
    if (pow2) return make_float4((float)(a[0] * inv_members), (float)(a[1] * inv_members), (float)(a[2] * inv_members), (float)(a[3] * inv_members));
    return make_float4((float)(a[0] / n_members), (float)(a[1] / n_members), (float)(a[2] / n_members), (float)(a[3] / n_members));
  };
  float tmax = -INFINITY, psum = 0.f;
  // (the next block's loads are in flight while a block is combined: its latency was most of the kernel)
  float4 next[4] = {};
  if (warp * 128 + lane * 4 < V) load4(warp * 128 + lane * 4, next);
  for (int b = warp; b * 128 < V; b += kWarps) {
    const int i = b * 128 + lane * 4;
    float bm = -INFINITY;
    float4 q[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) q[m] = next[m];
    if (i + kWarps * 128 < V) load4(i + kWarps * 128, next);
    if (i < V) {
      const float4 w = combine4(i, q);
      const float v[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (i + u < V) {
          bm = fmaxf(bm, v[u]);
          psum += v[u];
          if (i + u == kEos) s_eos[kEos] = mode == 0 ? logf(v[u]) : v[u];
        }
    }
    tmax = fmaxf(tmax, bm);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) bm = fmaxf(bm, __shfl_xor_sync(0xffffffffu, bm, o));
    if (lane == 0) s_bm[b] = bm;
  }
  // threshold: the kk-th largest of 32 maxima over disjoint classes (kk <= 32), reached by kk classes
  s_tmax[tid] = tmax;
  __syncthreads();
  if (warp == 0) {
    float g = -INFINITY;
    for (int w = 0; w < kWarps; ++w) g = fmaxf(g, s_tmax[w * 32 + lane]);
    int rank = 0;
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      const float o = __shfl_sync(0xffffffffu, g, j);
      rank += (o > g || (o == g && j < lane)) ? 1 : 0;
    }
    if (rank == kk - 1) s_tau = g;
  }
  __syncthreads();
  // (probabilities that differ may have the same logarithm, and then the lower index is the better one)
  const float tau = mode == 0 ? s_tau * (1.0f - 1e-6f) : s_tau;
  for (int b = warp; b * 128 < V; b += kWarps) {
    if (s_bm[b] < tau) continue;
    const int i = b * 128 + lane * 4;
    if (i >= V) continue;
    float4 q[4];
    load4(i, q);
    const float4 w = combine4(i, q);
    const float v[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (i + u < V && v[u] >= tau) {
        const int pos = atomicAdd(&sh.count, 1);
        if (pos < kTopkCap) { sh.cv[pos] = mode == 0 ? logf(v[u]) : v[u]; sh.ci[pos] = i + u; }
      }
  }
  __syncthreads();
  const float* z = s_eos;     // (of the row, only EOS is asked for by index ...)
  if (sh.count > kTopkCap) {  // ... unless more classes than the list holds reach the threshold: then it is swept
    float* row = combined + (size_t)r * ld;
    for (int i = tid * 4; i < V; i += THREADS * 4) {
      float4 q[4];
      load4(i, q);
      const float4 w = combine4(i, q);
      *reinterpret_cast<float4*>(row + i) = mode == 0 ? make_float4(logf(w.x), logf(w.y), logf(w.z), logf(w.w)) : w;
    }
    __threadfence_block();
    __syncthreads();
    z = row;
  }
  topk_finish<THREADS>(sh, r, psum, 0.f, z, nullptr, V, kk, out, mode == 0 ? 1 : 0, TopkRefine{}, nullptr);
  select_if_last<THREADS>(sel, out, r, s_union);
}

// ---------------------------------------------------------------------------------------
// Final scoring and n-best extraction for one sentence.  Replaces
// Decoder<T>::ObtainOneBestHypothesis (src/decoder.h:703-859) up to the numeric result:
// length normalisation (:708-713), coverage penalty (:716-759), minimum-ratio filter
// (:762-765), n-best with strictly-greater replacement (:766-773), then the hypothesis is
// rebuilt from the back-pointers.
struct FinalizeArgs {
  BeamState bs;
  const int32_t* steps;     // [B]
  const int32_t* src_len;   // [B]
  const int32_t* orig;      // [B] caller's sentence index
  const float* rec_align;   // [Tcap][R][win] or null
  const int32_t* rec_lo;    // [Tcap][R]
  const int32_t* rec_vit;   // [Tcap][R]
  float* fin_final;         // [B][fin_cap] scratch: final score, -inf if filtered
  int win;
  int k;
  int nbest;
  int max_len;
  int max_src;
  float lp_alpha, cp_beta, min_ratio;
  int32_t* out_tok;   // [n][nbest][max_len]
  int32_t* out_len;   // [n][nbest]
  float* out_score;   // [n][nbest]
  int32_t* out_vit;   // [n][nbest][max_len] or null
  float* out_align;   // [n][nbest][max_len][max_src] or null
};
// grid = sentences, block and dynamic smem = finalize_shape: 1 to 16 warps, a path and row sums of max_len entries for each
// of them, and the sentence's back-pointers where they fit.
// The kernel is a chain of memory round trips: following the back-pointers of a hypothesis through global memory was one
// per step (54 us for 85 steps), and the coverage of a hypothesis two per step.  The sentence's back-pointers come into
// shared memory first (a byte each), and the coverage reads four steps at a time.
// Before: 570 us for sentences of up to 100 words with a coverage penalty, 54 us for one of 50 without.
constexpr int kFinalizeSmem = 46 * 1024;
struct FinalizeShape { int warps, par_bytes; size_t smem; };
inline FinalizeShape finalize_shape(int max_len, int k) {
  FinalizeShape f{16, 0, 0};
  const size_t per = 2 * sizeof(int) * (size_t)max_len;     // path and row sums of a hypothesis
  while (f.warps > 1 && f.warps * per > kFinalizeSmem / 2) f.warps >>= 1;
  f.smem = f.warps * per;
  if (f.smem + (size_t)max_len * k <= (size_t)kFinalizeSmem) { f.par_bytes = max_len * k; f.smem += f.par_bytes; }
  return f;
}
static __global__ void __launch_bounds__(512) finalize_kernel(FinalizeArgs a, int par_bytes) {
  extern __shared__ unsigned char smraw[];
  const int sent = blockIdx.x;
  const int S = a.src_len[sent];
  const int k = a.k, R = a.bs.R;
  const int nf = a.bs.fin_n[sent];
  const int r0 = sent * k;
  const int32_t* ft = a.bs.fin_t + (size_t)sent * a.bs.fin_cap;
  const int32_t* fb = a.bs.fin_b + (size_t)sent * a.bs.fin_cap;
  const float* fs = a.bs.fin_score + (size_t)sent * a.bs.fin_cap;
  float* ff = a.fin_final + (size_t)sent * a.bs.fin_cap;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nw = blockDim.x >> 5;
  int* path = reinterpret_cast<int*>(smraw) + warp * a.max_len;     // path[p] = slot that ran the forward producing position p
  float* sums = reinterpret_cast<float*>(smraw) + (nw + warp) * a.max_len;
  unsigned char* par = smraw + 8 * (size_t)nw * a.max_len;          // [steps][k] back-pointers
  int last = 0;             // the longest hypothesis' last step
  if (par_bytes) {
    for (int q = lane; q < nf; q += 32) last = max(last, ft[q]);
    last = __reduce_max_sync(0xffffffffu, last);
    for (int i = threadIdx.x; i < last * k; i += blockDim.x) {
      const int tt = i / k;
      const int p = a.bs.hist_parent[(size_t)tt * R + r0 + (i - tt * k)];
      par[i] = p >= 0 && p < k ? (unsigned char)p : 0;       // (a forced search may name anything)
    }
    __syncthreads();
  }
  auto follow = [&](int q) {        // by one lane
    const int t = ft[q];
    int slot = fb[q];
    path[t + 1] = slot;
    for (int tt = t - 1; tt >= 0; --tt) {
      slot = par_bytes ? par[tt * k + slot] : a.bs.hist_parent[(size_t)tt * R + r0 + slot];
      path[tt + 1] = slot;
    }
  };
  const bool tracked = a.rec_align != nullptr;

  if (!tracked || a.cp_beta == 0.f) {
    for (int q = threadIdx.x; q < nf; q += blockDim.x) {
      const int n = ft[q] + 2;
      float sc = fs[q];
      if (0 != a.lp_alpha) {
        const float lp = powf((float)(5 + n), a.lp_alpha) / powf((float)(5 + 1), a.lp_alpha);
        sc /= lp;
      }
      if (0 != a.cp_beta) {
        // alignments are all zero when they are not tracked: every position becomes the
        // uniform row (0 + 0.01) / sum; same loops as the reference, in fp32
        float sum = 0.f;
        const float one = (float)(0.0f + 0.01);
        for (int s = 0; s < S; ++s) sum += one;
        const float u = one / sum;
        float c1 = 0.f;
        for (int j = 1; j < n - 1; ++j) c1 += u;
        float cp = 0.f;
        const float lg = logf(fminf(c1, 1.0f));
        for (int s = 0; s < S; ++s) cp += lg;
        cp *= a.cp_beta;
        if (cp < -20) cp = -20;
        sc += cp;
      }
      const float ratio = ((float)n) / S;
      ff[q] = (ratio > a.min_ratio) ? sc : -INFINITY;
    }
  } else {
    // tracked alignments: one warp per hypothesis, lanes over source positions
    for (int q = warp; q < nf; q += nw) {
      const int t = ft[q];
      const int n = t + 2;
      float sc = fs[q];
      if (0 != a.lp_alpha) {
        const float lp = powf((float)(5 + n), a.lp_alpha) / powf((float)(5 + 1), a.lp_alpha);
        sc /= lp;
      }
      if (lane == 0) follow(q);
      __syncwarp();
      auto at = [&](size_t row, int lo, int s) {
        const int w = s - lo;
        return ((w >= 0 && w < a.win) ? a.rec_align[row * a.win + w] : 0.f) + 0.01f;
      };
      for (int p0 = 2; p0 <= n - 1; p0 += 4) {
        size_t row[4];
        int lo[4];
        float part[4] = {};
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int p = min(p0 + u, n - 1);
          row[u] = (size_t)(p - 1) * R + r0 + path[p];
          lo[u] = a.rec_lo[row[u]];
        }
        for (int s = lane; s < S; s += 32) {
#pragma unroll
          for (int u = 0; u < 4; ++u) part[u] += at(row[u], lo[u], s);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          part[u] = warp_sum(part[u]);
          if (lane == 0 && p0 + u <= n - 1) sums[p0 + u] = part[u];
        }
      }
      __syncwarp();
      float cp = 0.f;
      for (int s = lane; s < S; s += 32) {
        float cov = 0.f;
#pragma unroll 4
        for (int p = 2; p <= n - 1; ++p) {
          const size_t row = (size_t)(p - 1) * R + r0 + path[p];
          cov += at(row, a.rec_lo[row], s) / sums[p];
        }
        cp += logf(fminf(cov, 1.0f));
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) cp += __shfl_xor_sync(0xffffffffu, cp, o);
      cp *= a.cp_beta;
      if (cp < -20) cp = -20;
      sc += cp;
      const float ratio = ((float)n) / S;
      if (lane == 0) ff[q] = (ratio > a.min_ratio) ? sc : -INFINITY;
      __syncwarp();
    }
  }
  __syncthreads();
  // n-best in creation order with strictly-greater replacement, then descending
  __shared__ int s_best[32];
  __shared__ int s_nb;
  if (threadIdx.x == 0) {
    int nb = 0;
    for (int q = 0; q < nf; ++q) {
      const float sc = ff[q];
      if (sc == -INFINITY) continue;
      if (nb < a.nbest) s_best[nb++] = q;
      else {
        int worst = 0;
        for (int z = 1; z < nb; ++z)
          if (ff[s_best[z]] < ff[s_best[worst]] || (ff[s_best[z]] == ff[s_best[worst]] && s_best[z] > s_best[worst])) worst = z;
        if (ff[s_best[worst]] < sc) s_best[worst] = q;
      }
    }
    for (int i = 1; i < nb; ++i) {  // insertion sort: score desc, creation order asc
      const int q = s_best[i];
      int j = i - 1;
      while (j >= 0 && (ff[s_best[j]] < ff[q] || (ff[s_best[j]] == ff[q] && s_best[j] > q))) { s_best[j + 1] = s_best[j]; --j; }
      s_best[j + 1] = q;
    }
    s_nb = nb;
  }
  __syncthreads();
  const int osent = a.orig[sent];
  for (int q0 = 0; q0 < a.nbest; q0 += nw) {
    const int q = q0 + warp;
    if (q < a.nbest) {
    const size_t ob = (size_t)osent * a.nbest + q;
    // positions past the hypothesis (all of them when fewer than nbest passed the filter) read START / "no
    // alignment", so that a result does not carry what an earlier decode left in the buffer
    const int n_used = (q >= s_nb) ? 0 : ft[s_best[q]] + 2;
    for (int j = n_used + lane; j < a.max_len; j += 32) {
      a.out_tok[ob * a.max_len + j] = kStart;
      if (a.out_vit) a.out_vit[ob * a.max_len + j] = -20;
    }
    if (a.out_align)
      for (size_t j = (size_t)n_used * a.max_src + lane; j < (size_t)a.max_len * a.max_src; j += 32)
        a.out_align[ob * a.max_len * a.max_src + j] = 0.f;
    if (q >= s_nb && lane == 0) { a.out_len[ob] = 0; a.out_score[ob] = 0.f; }
    if (q < s_nb) {
    const int h = s_best[q];
    const int t = ft[h];
    const int n = t + 2;
    int32_t* ot = a.out_tok + ob * a.max_len;
    int32_t* ov = a.out_vit ? a.out_vit + ob * a.max_len : nullptr;
    if (lane == 0) {
      a.out_len[ob] = n;
      a.out_score[ob] = ff[h];
      ot[0] = kStart; ot[t + 1] = kEos;
      if (ov) ov[0] = -20;
      follow(h);
    }
    __syncwarp();
    for (int p = 1 + lane; p <= t + 1; p += 32) {
      if (p <= t) ot[p] = a.bs.hist_tok[(size_t)(p - 1) * R + r0 + path[p + 1]];      // the word chosen after forward p - 1
      if (ov) ov[p] = a.rec_vit ? a.rec_vit[(size_t)(p - 1) * R + r0 + path[p]] : -1;
    }
    }
    }
    if (!a.out_align || !tracked) continue;
    // alignments: the steps of this round's hypotheses are dealt to all warps
    __syncthreads();
    for (int z = 0; z < nw && q0 + z < s_nb; ++z) {
      const int n = ft[s_best[q0 + z]] + 2;
      const int* zpath = reinterpret_cast<int*>(smraw) + z * a.max_len;
      float* oa = a.out_align + ((size_t)osent * a.nbest + q0 + z) * a.max_len * a.max_src;
      for (int p = warp; p < n; p += nw) {
        float part = 0.f;
        const bool norm = (a.cp_beta != 0.f) && p >= 2;
        size_t row = 0; int lo = 0;
        if (p >= 1) { row = (size_t)(p - 1) * R + r0 + zpath[p]; lo = a.rec_lo[row]; }
        if (norm) {
          for (int s = lane; s < S; s += 32) {
            const int w = s - lo;
            part += ((w >= 0 && w < a.win) ? a.rec_align[row * a.win + w] : 0.f) + 0.01f;
          }
          part = warp_sum(part);
        }
        for (int s = lane; s < a.max_src; s += 32) {
          float v = 0.f;
          if (p >= 1 && s < S) {
            const int w = s - lo;
            v = (w >= 0 && w < a.win) ? a.rec_align[row * a.win + w] : 0.f;
            if (norm) v = (v + 0.01f) / part;
          }
          oa[(size_t)p * a.max_src + s] = v;
        }
      }
    }
    __syncthreads();
  }
}

}  // namespace linmt
