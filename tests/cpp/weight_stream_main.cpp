// Prints, for every line "layers hp vp members planes vocab_planes l2_bytes scoring rows" of its input, the bytes that a step
// reads and whether they are a stream (csrc/weight_stream.h).
#include <cstdio>

#include "weight_stream.h"

int main() {
  linmt::StepWeights w;
  size_t l2;
  int scoring, rows;
  while (std::scanf("%d %d %d %d %d %d %zu %d %d", &w.layers, &w.hp, &w.vp, &w.members, &w.planes, &w.vocab_planes, &l2, &scoring, &rows) == 9)
    std::printf("%zu %d\n", linmt::step_weight_bytes(w, scoring != 0), static_cast<int>(linmt::weights_stream(w, l2, scoring != 0, rows)));
}
