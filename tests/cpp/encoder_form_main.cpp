// Prints the encoder's form (csrc/encoder_form.h) for every line "layers hp members split sentences words" of its input.
#include <cstdio>

#include "encoder_form.h"

int main() {
  linmt::EncoderModel m;
  int split, n, words;
  const char* names[] = {"wavefront", "layers", "pipelined"};
  while (std::scanf("%d %d %d %d %d %d", &m.layers, &m.hp, &m.members, &split, &n, &words) == 6) {
    m.split = split != 0;
    std::puts(names[static_cast<int>(linmt::encoder_form(m, n, words))]);
  }
}
