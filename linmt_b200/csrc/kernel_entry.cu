// kernel_entry.cu -- single-kernel entry points of the C ABI (host pointers), used by the
// parity tests to check one kernel at a time against the CPU oracle.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "engine.h"
#include "gemm_plan.cuh"
#include "gemm_simt.cuh"
#include "step_kernels.cuh"

namespace {
struct DevBuf {
  void* p = nullptr;
  ~DevBuf() { if (p) cudaFree(p); }
  cudaError_t alloc(size_t bytes) {
    const cudaError_t e = cudaMalloc(&p, bytes ? bytes : 1);
    if (e != cudaSuccess) cudaGetLastError();      // (or the next launch that is checked reports it again)
    return e;
  }
  template <class T> T* as() { return static_cast<T*>(p); }
};
#define KCK(x) do { if ((x) != cudaSuccess) return LINMT_ECUDA; } while (0)
// What a handle made now would allow its products (LINMT_TC_PAIR=0, LINMT_TC_ROWS=0, LINMT_TC_PERSIST=0 as there).
linmt::tc::GemmLimits limits_from_env(int device) {
  auto allowed = [](const char* name) { const char* v = std::getenv(name); return !(v && std::atoi(v) == 0); };
  linmt::tc::GemmLimits lim;
  if (cudaDeviceGetAttribute(&lim.n_sm, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) lim.n_sm = 0;
  lim.ws_floats = (size_t)16 << 20; lim.max_tiles = 4096;
  lim.rows = allowed("LINMT_TC_ROWS"); lim.persist = allowed("LINMT_TC_PERSIST");
  lim.pair = allowed("LINMT_TC_PAIR") && linmt::tc::max_resident_pairs<2, 64, 1, linmt::tc::TcEpiF32>() > 0;
  return lim;
}
}  // namespace

extern "C" {

int linmt_k_gemm(const float* X, const float* W, float* Y, int32_t R, int32_t K, int32_t N, int32_t gemm_path,
                 int32_t precision, int32_t device) {
  using namespace linmt;
  if (!X || !W || !Y || R < 1 || K < 1 || N < 1) return LINMT_EINVAL;
  if (gemm_path == LINMT_GEMM_SIMT && precision != LINMT_PREC_FP32) return LINMT_EINVAL;
  if (gemm_path != LINMT_GEMM_SIMT && gemm_path != LINMT_GEMM_TENSOR && gemm_path != LINMT_GEMM_TENSOR2 &&
      gemm_path != LINMT_GEMM_TENSOR3) return LINMT_EINVAL;
  KCK(cudaSetDevice(device));
  const int Kp = round_up(K, 64), Np = round_up(N, 128);
  std::vector<float> xp((size_t)R * Kp, 0.f), wt((size_t)Np * Kp, 0.f);
  for (int r = 0; r < R; ++r) std::memcpy(&xp[(size_t)r * Kp], X + (size_t)r * K, sizeof(float) * K);
  for (int n = 0; n < N; ++n)
    for (int k = 0; k < K; ++k) wt[(size_t)n * Kp + k] = W[(size_t)k * N + n];
  DevBuf dx, dw, dy;
  KCK(dx.alloc(xp.size() * 4)); KCK(dw.alloc(wt.size() * 4)); KCK(dy.alloc((size_t)R * Np * 4));
  KCK(cudaMemcpy(dx.p, xp.data(), xp.size() * 4, cudaMemcpyHostToDevice));
  KCK(cudaMemcpy(dw.p, wt.data(), wt.size() * 4, cudaMemcpyHostToDevice));
  if (gemm_path == LINMT_GEMM_SIMT) {
    ASegs a{}; a.ptr[0] = dx.as<float>(); a.ld[0] = Kp; a.nseg = 1; a.seg_k = Kp;
    EpiBias e{nullptr, dy.as<float>(), Np};
    KCK(gemm_simt(a, dw.as<float>(), Kp, R, Np, Kp, e, 0));
    KCK(cudaDeviceSynchronize());
  } else {
    const int fmt = (precision == LINMT_PREC_FP32 && gemm_path == LINMT_GEMM_TENSOR) ? 1 : 0;
    const int nt = (precision == LINMT_PREC_BF16) ? 1 : (gemm_path == LINMT_GEMM_TENSOR3 ? 3 : 2);
    DevBuf pa[3], pb[3], derr;
    tc::Planes A{}, B{};
    A.ld = Kp; B.ld = Kp; A.fmt = fmt; B.fmt = fmt;
    for (int t = 0; t < nt; ++t) {
      KCK(pa[t].alloc(xp.size() * 2)); KCK(pb[t].alloc(wt.size() * 2));
      A.p[t] = pa[t].as<__nv_bfloat16>(); B.p[t] = pb[t].as<__nv_bfloat16>();
    }
    KCK(derr.alloc(4));
    KCK(cudaMemset(derr.p, 0, 4));
    tc::split_planes_kernel<<<256, 256>>>(dx.as<float>(), A, nt, xp.size());
    tc::split_planes_kernel<<<1024, 256>>>(dw.as<float>(), B, nt, wt.size());
    KCK(cudaGetLastError());
    const tc::GemmLimits lim = limits_from_env(device);      // the engine's choice of kernel and shape
    if (lim.n_sm < 1) return LINMT_ECUDA;
    tc::TcEpiF32 e{nullptr, dy.as<float>(), Np, 0};
    const tc::GemmPlan plan = tc::plan_gemm<tc::TcEpiF32>(R, Np, Kp, nt, fmt, 0, 0, lim);
    tc::TmapSet tm{};
    for (int t = 0; t < nt; ++t)
      if (!tc::make_tmap(&tm.a[t], A.p[t], R, Kp, Kp, plan.a_box, plan.bk) || !tc::make_tmap(&tm.b[t], B.p[t], Np, Kp, Kp, plan.b_box, plan.bk)) return LINMT_ECUDA;
    DevBuf dws, dcnt;
    KCK(dws.alloc(lim.ws_floats * 4)); KCK(dcnt.alloc(lim.max_tiles * 4)); KCK(cudaMemset(dcnt.p, 0, lim.max_tiles * 4));
    const cudaError_t le = tc::launch_planned(plan, tm, R, Np, Kp, nt, fmt, false, e, derr.as<int>(), 0, lim.n_sm, dws.as<float>(), dcnt.as<int>());
    KCK(le);
    KCK(cudaDeviceSynchronize());
    int herr = 0;
    KCK(cudaMemcpy(&herr, derr.p, 4, cudaMemcpyDeviceToHost));
    if (herr) return LINMT_ECUDA;
  }
  std::vector<float> yp((size_t)R * Np);
  KCK(cudaMemcpy(yp.data(), dy.p, yp.size() * 4, cudaMemcpyDeviceToHost));
  for (int r = 0; r < R; ++r) std::memcpy(Y + (size_t)r * N, &yp[(size_t)r * Np], sizeof(float) * N);
  return LINMT_OK;
}

int linmt_k_logits(const float* X, const float* W, const float* bias, int32_t R, int32_t K, int32_t V, int32_t gemm_path, int32_t precision, int32_t kk,
                   float* Y, float* block_max, float* block_sum, int32_t* info, int32_t* idx, float* logp, float* eos_logp, int32_t device) {
  using namespace linmt;
  if (!X || !W || !bias || !Y || !block_max || !block_sum || !info || !idx || !logp || !eos_logp || R < 1 || K < 1 || V < 4 || kk < 1 || kk > kMaxBeam + 1 || kk > V)
    return LINMT_EINVAL;
  if ((gemm_path != LINMT_GEMM_AUTO && gemm_path != LINMT_GEMM_TENSOR) || (precision != LINMT_PREC_FP32 && precision != LINMT_PREC_BF16)) return LINMT_EINVAL;
  KCK(cudaSetDevice(device));
  const int Kp = round_up(K, 64), Vp = round_up(V, 128), ld = logit_blocks_ld(Vp);
  const int fmt = precision == LINMT_PREC_FP32 ? 1 : 0, planes = fmt ? 2 : 1;
  const bool refine = fmt && gemm_path == LINMT_GEMM_AUTO;     // one fp16 product, the candidates recomputed
  const int nt = refine ? 1 : planes;
  std::vector<float> xp((size_t)R * Kp, 0.f), wt((size_t)Vp * Kp, 0.f), bp(Vp, 0.f);
  for (int r = 0; r < R; ++r) std::memcpy(&xp[(size_t)r * Kp], X + (size_t)r * K, sizeof(float) * K);
  double norm = 0.0;
  for (int v = 0; v < V; ++v) {
    double ss = 0.0;
    for (int k = 0; k < K; ++k) { const float w = W[(size_t)k * V + v]; wt[(size_t)v * Kp + k] = w; ss += (double)w * w; }
    norm = std::max(norm, ss);
  }
  std::memcpy(bp.data(), bias, sizeof(float) * V);
  DevBuf dx, dw, db, pa[2], pb[2], dy, dmax, dsum, derr, dws, dcnt, di, dp, de;
  KCK(dx.alloc(xp.size() * 4)); KCK(dw.alloc(wt.size() * 4)); KCK(db.alloc(bp.size() * 4));
  KCK(cudaMemcpy(dx.p, xp.data(), xp.size() * 4, cudaMemcpyHostToDevice));
  KCK(cudaMemcpy(dw.p, wt.data(), wt.size() * 4, cudaMemcpyHostToDevice));
  KCK(cudaMemcpy(db.p, bp.data(), bp.size() * 4, cudaMemcpyHostToDevice));
  tc::Planes A{}, B{};
  A.ld = B.ld = Kp; A.fmt = B.fmt = fmt;
  for (int t = 0; t < planes; ++t) {
    KCK(pa[t].alloc(xp.size() * 2)); KCK(pb[t].alloc(wt.size() * 2));
    A.p[t] = pa[t].as<__nv_bfloat16>(); B.p[t] = pb[t].as<__nv_bfloat16>();
  }
  tc::split_planes_kernel<<<256, 256>>>(dx.as<float>(), A, planes, xp.size());
  tc::split_planes_kernel<<<1024, 256>>>(dw.as<float>(), B, planes, wt.size());
  KCK(cudaGetLastError());
  KCK(derr.alloc(4)); KCK(cudaMemset(derr.p, 0, 4));
  KCK(dy.alloc((size_t)R * Vp * 4)); KCK(dmax.alloc((size_t)R * ld * 4)); KCK(dsum.alloc((size_t)R * ld * 4));
  const tc::GemmLimits lim = limits_from_env(device);
  if (lim.n_sm < 1) return LINMT_ECUDA;
  const tc::GemmPlan plan = tc::plan_gemm<tc::TcEpiF32>(R, Vp, Kp, nt, fmt, Kp / 32, 0, lim);
  tc::TmapSet tm{};
  for (int t = 0; t < nt; ++t)
    if (!tc::make_tmap(&tm.a[t], A.p[t], R, Kp, Kp, plan.a_box, plan.bk) || !tc::make_tmap(&tm.b[t], B.p[t], Vp, Kp, Kp, plan.b_box, plan.bk)) return LINMT_ECUDA;
  KCK(dws.alloc(lim.ws_floats * 4)); KCK(dcnt.alloc(lim.max_tiles * 4)); KCK(cudaMemset(dcnt.p, 0, lim.max_tiles * 4));
  const LogitBlocks bl = logit_blocks(dmax.as<float>(), dsum.as<float>(), ld, Vp, Kp, plan.stat_tile, plan.stat_part);
  tc::TcEpiF32 e{db.as<float>(), dy.as<float>(), Vp, 0};
  if (refine) e.out16 = dy.as<__half>();
  e.pmax = bl.max; e.psum = bl.sum; e.pmax_ld = ld; e.n_valid = V;
  KCK(tc::launch_planned(plan, tm, R, Vp, Kp, nt, fmt, false, e, derr.as<int>(), 0, lim.n_sm, dws.as<float>(), dcnt.as<int>()));
  TopkRefine rf{};
  if (refine) {
    rf.a0 = pa[0].as<__half>(); rf.a1 = pa[1].as<__half>(); rf.lda = Kp;
    rf.b0 = pb[0].as<__half>(); rf.b1 = pb[1].as<__half>(); rf.ldb = Kp;
    rf.bias = db.as<float>(); rf.K = Kp; rf.eps_coef = refine_eps((float)std::sqrt(norm));
  }
  KCK(di.alloc((size_t)R * kk * 4)); KCK(dp.alloc((size_t)R * kk * 4)); KCK(de.alloc((size_t)R * 4));
  TopkOut o{di.as<int32_t>(), dp.as<float>(), de.as<float>(), nullptr};
  KCK(launch_topk(refine ? (const float*)nullptr : dy.as<float>(), refine ? dy.as<__half>() : nullptr, Vp, V, kk, R, lim.n_sm, o, 1, bl, refine ? &rf : nullptr, SelectArgs{}, 0, false));
  KCK(cudaDeviceSynchronize());
  int herr = 0;
  KCK(cudaMemcpy(&herr, derr.p, 4, cudaMemcpyDeviceToHost));
  if (herr) return LINMT_ECUDA;
  info[0] = (int32_t)plan.kernel; info[1] = bl.n; info[2] = bl.tile; info[3] = bl.part; info[4] = bl.sum ? 1 : 0;
  if (refine) {
    std::vector<__half> yh((size_t)R * Vp);
    KCK(cudaMemcpy(yh.data(), dy.p, yh.size() * 2, cudaMemcpyDeviceToHost));
    for (int r = 0; r < R; ++r)
      for (int v = 0; v < V; ++v) Y[(size_t)r * V + v] = __half2float(yh[(size_t)r * Vp + v]);
  } else {
    KCK(cudaMemcpy2D(Y, (size_t)V * 4, dy.p, (size_t)Vp * 4, (size_t)V * 4, R, cudaMemcpyDeviceToHost));
  }
  if (bl.n) KCK(cudaMemcpy(block_max, dmax.p, (size_t)R * ld * 4, cudaMemcpyDeviceToHost));
  if (bl.sum) KCK(cudaMemcpy(block_sum, dsum.p, (size_t)R * ld * 4, cudaMemcpyDeviceToHost));
  KCK(cudaMemcpy(idx, di.p, (size_t)R * kk * 4, cudaMemcpyDeviceToHost));
  KCK(cudaMemcpy(logp, dp.p, (size_t)R * kk * 4, cudaMemcpyDeviceToHost));
  KCK(cudaMemcpy(eos_logp, de.p, (size_t)R * 4, cudaMemcpyDeviceToHost));
  return LINMT_OK;
}

int linmt_k_softmax_topk(const float* logits, int32_t R, int32_t V, int32_t kk, int32_t* idx, float* logp,
                         float* eos_logp, int32_t device) {
  using namespace linmt;
  if (!logits || !idx || !logp || R < 1 || V < 2 || kk < 1 || kk > kMaxBeam + 1) return LINMT_EINVAL;
  KCK(cudaSetDevice(device));
  const int Vp = round_up(V, 4);
  std::vector<float> lp((size_t)R * Vp, 0.f);
  for (int r = 0; r < R; ++r) std::memcpy(&lp[(size_t)r * Vp], logits + (size_t)r * V, sizeof(float) * V);
  DevBuf dl, di, dp, de;
  KCK(dl.alloc(lp.size() * 4)); KCK(di.alloc((size_t)R * kk * 4)); KCK(dp.alloc((size_t)R * kk * 4)); KCK(de.alloc((size_t)R * 4));
  KCK(cudaMemcpy(dl.p, lp.data(), lp.size() * 4, cudaMemcpyHostToDevice));
  TopkOut o{di.as<int32_t>(), dp.as<float>(), de.as<float>(), nullptr};
  KCK(launch_softmax_topk(dl.as<float>(), Vp, V, kk, R, o, 1, 0));
  KCK(cudaDeviceSynchronize());
  KCK(cudaMemcpy(idx, di.p, (size_t)R * kk * 4, cudaMemcpyDeviceToHost));
  KCK(cudaMemcpy(logp, dp.p, (size_t)R * kk * 4, cudaMemcpyDeviceToHost));
  if (eos_logp) KCK(cudaMemcpy(eos_logp, de.p, (size_t)R * 4, cudaMemcpyDeviceToHost));
  return LINMT_OK;
}

}  // extern "C"
