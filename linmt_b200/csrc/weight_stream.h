// weight_stream.h -- whether a step's weights are loaded as a stream that L2 gives up first (weight_policy in gemm_tc.cuh).
// Plain C++, so that the rule can be checked without a device.
#pragma once
#include <cstddef>

namespace linmt {

struct StepWeights {
  int layers, hp, vp;            // sizes rounded up to their tiles
  int members;                   // of the ensemble
  int planes, vocab_planes;      // 16-bit planes of the recurrent and attention products, and of the vocabulary product
};

// What a step reads of them: a scoring step ends with the attentional state, its vocabulary products follow for all positions.
inline size_t step_weight_bytes(const StepWeights& w, bool scoring) {
  const size_t hh = (size_t)w.hp * w.hp, recurrent = (8 * (size_t)w.layers + 4) * hh, vocab = (size_t)w.vp * w.hp;
  return 2 * w.members * (w.planes * recurrent + (scoring ? 0 : w.vocab_planes * vocab));
}

// A step reads more weights than L2 has room for beside the states (three quarters of it): they are a stream.  Scoring with
// recurrent weights that L2 holds, bf16, as ordinary loads / as a stream, ms a call: 4 x 1000 / 30k 4 rows 2.24 / 2.31, 16
// 2.48 / 2.54, 32 2.89 / 2.93, 64 3.74 / 3.73, 80 3.94 / 3.81, 128 4.22 / 4.05, 256 5.40 / 5.19; 2 x 1000 / 60k 1.37 / 1.44,
// 1.57 / 1.63, 1.86 / 1.91, 2.43 / 2.46, 2.96 / 2.99, 3.31 / 3.30, 4.50 / 4.39; in fp32 precision 2 x 1000 / 30k 1.77 /
// 1.85, 2.11 / 2.28, 2.56 / 2.62, 3.18 / 3.21.  So from 65 rows on, which one plane runs in the one-tile kernel,
// scoring goes by the same sum as decoding.
inline bool weights_stream(const StepWeights& w, size_t l2_bytes, bool scoring, int rows) {
  return step_weight_bytes(w, scoring && rows <= 64) > l2_bytes / 4 * 3;
}

}  // namespace linmt
