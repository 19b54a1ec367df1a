// Prints encoder_layers_beside and encoder_leaves_room (csrc/encoder_form.h) for every line "layers hp members split sentences words
// shared" of its input.
#include <cstdio>

#include "encoder_form.h"

int main() {
  linmt::EncoderModel m;
  int split, n, words, shared;
  while (std::scanf("%d %d %d %d %d %d %d", &m.layers, &m.hp, &m.members, &split, &n, &words, &shared) == 7) {
    m.split = split != 0;
    const bool beside = linmt::encoder_layers_beside(m, n, words, shared != 0);
    std::printf("%d %d\n", beside, linmt::encoder_leaves_room(m, n, beside));
  }
}
