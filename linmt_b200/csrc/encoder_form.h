// encoder_form.h -- which form of the tensor-core encoder takes a batch.  Plain C++, so that the rule can be checked without
// a device.
#pragma once
#include <algorithm>

namespace linmt {

// kWavefront   position by position: a layer's whole product per position, a stream per layer
// kLayers      layer by layer: the input parts of all positions in one product, then W_h . h position by position
// kPipelined   the layers side by side, each kEncLag positions behind the layer below, with input parts of that many positions
enum class EncoderForm { kWavefront, kLayers, kPipelined };

// most sentences that are encoded layer by layer, and with the layers side by side; 32 fill a quarter of the row tile that the
// latter's products take, and are always faster in the few-rows kernel of the former
constexpr int kEncLayers = 64, kEncPipelined = 128, kEncFew = 32;
constexpr int kEncLag = 8;     // positions (4 x 1000, 64 sentences of 80 words: 3.32, 3.06, 3.20 ms with 4, 8, 14)

struct EncoderModel {
  int layers, hp;      // hidden size, rounded up to 64
  int members;         // of the ensemble (its members are encoded side by side already)
  bool split;          // fp32 weights (the f16 pair)
};

// n sentences, the longest of S words, on a handle that has the layers' panels.
inline EncoderForm encoder_form(const EncoderModel& m, int n, int S) {
  const EncoderForm other = n <= kEncLayers ? EncoderForm::kLayers : EncoderForm::kWavefront;
  // (One plane stays with the layers up to 64: another order of sums rounds a state to the other bf16 neighbour now and then,
  // and a near tie of two hypotheses is decided by that.)
  if (n <= kEncFew || n > kEncPipelined || !m.split || m.members > 1 || m.layers < 2) return other;
  // Measured with 2 to 5 layers of 128 to 2048 units and 16 to 96 words (ms of a call with two decoder steps).  A pipeline of L
  // layers is filled and drained, and pays where the sources are long for that.  Against the wavefront (65 to 128 sentences,
  // n = 96, pipelined / wavefront at 32, 64 and 96 words): 2 x 1000 1.09 / 1.26, 1.81 / 2.17, 2.56 / 3.07; 3 x 1000 1.48 / 1.51,
  // 2.36 / 2.63, 3.22 / 3.73; 4 x 1000 1.76 / 1.68, 2.77 / 2.89, 3.69 / 4.35; 5 x 1000 2.27 / 1.90, 3.47 / 3.31, 4.63 / 4.83.
  if (n > kEncLayers) return S >= kEncLag * std::max(4, 3 * (m.layers - 2)) ? EncoderForm::kPipelined : other;
  // Against the layers (33 to 64 sentences, n = 33, pipelined / layers): 2 x 128 0.55 / 0.61, 0.88 / 1.02, 1.03 / 1.43; 2 x 1000
  // 0.97 / 0.76, 1.60 / 1.31, 2.21 / 1.86; 4 x 512 1.00 / 1.01, 1.50 / 1.78, 1.97 / 2.56; 4 x 1000 1.57 / 1.36, 2.44 / 2.43, 3.24 /
  // 3.52; 5 x 768 1.52 / 1.44, 2.24 / 2.59, 3.01 / 3.76.  Fitted, in us a position: side by side, the longer of issuing L launches
  // and a product on 1/L of the SMs; one after another, L products of the few-rows kernel, which take a quarter longer from 49
  // rows on and go from 8.4 to 14 us between 1024 and 1088 units.  What the fit takes is at most 6 % slower than the other.
  const double h = m.hp / 1024.0, L = m.layers;
  const double side = std::max(3.2 * L, 8 + 9 * h + 3.5 * h * h * h * (L - 1));
  const double turn = L * (m.hp <= 1024 ? std::max(6.1, 3.0 + 5.85 * h) : 13.5 + 10 * (h - 1)) * (n > 48 ? 1.22 : 1.0);
  return S >= 4 * kEncLag && (S + 6 * (L - 1)) * side < S * turn ? EncoderForm::kPipelined : other;
}

// Whether the layers of EncoderForm::kLayers run side by side all the same: the products of few sentences in CTAs of half an SM that
// leave room for the other layers'.  Encoder and two scored words, ms, layer by layer / so, at 20, 32 and 100 words: 4 x 1000 1 sentence
// 0.71 / 0.66, 0.96 / 0.82, 2.42 / 1.82, 16 0.82 / 0.79, 1.10 / 1.01, 2.81 / 2.37, 48 (20 and 32 words) 1.13 / 0.98, 1.63 / 1.24; 5 x 768 4
// 0.78 / 0.72, 1.07 / 0.92, 2.63 / 2.08; 2 x 512 4 0.34 / 0.33, 0.45 / 0.41, 1.04 / 0.86; of 8 words 2 to 8 % slower.  Not
// * one sentence of a narrow model, until it is longer: its products are over before the next layer's start (2 x 512 20 words 0.333 /
//   0.348, 32 0.437 / 0.454, 50 0.588 / 0.517);
// * from 49 sentences on at 769 to 1024 units, where a layer's product fills the chip, in CTAs that leave no room (2 x 1000 64 sentences of 20
//   and 50 words 0.726 / 0.745, 1.38 / 1.42; 4 x 1000 20 and 24 words 1.24 / 1.26, 1.44 / 1.42; 512, 768 and 1280 units gain 3 to 14 %);
// * below 512 units (3 x 250 with 1 to 30 sentences of 40 words gained 2 to 3 % of a call, and lost 2 % with 11 ragged ones);
// * where the batch shares the device with others (`shared`);
// * in one plane, which keeps its order of sums (see encoder_form).
constexpr int kEncBesideWords = 20, kEncBesideWordsOne = 40, kEncBesideHidden = 512, kEncRoomSentences = 48;
inline bool encoder_layers_beside(const EncoderModel& m, int n, int S, bool shared) {
  if (!m.split || m.members > 1 || m.layers < 2 || m.hp < kEncBesideHidden || shared) return false;
  if (n > kEncRoomSentences && m.hp > 768 && m.hp <= 1024) return false;
  return S >= (n == 1 && m.hp < 768 ? kEncBesideWordsOne : kEncBesideWords);
}

// Whether the encoder's products of a position are shaped like a step's, so that the next one's weights are under way: up to 48
// sentences whose layers run side by side (4 x 1000, 20 words, ms as above with / without: 1 sentence 0.66 / 0.76, 40 0.96 / 1.08), up to 32
// one layer after another (1 sentence 0.71 / 0.72; 40 of 10 words 0.73 / 0.70).  One plane: as above.
inline bool encoder_leaves_room(const EncoderModel& m, int n, bool beside) { return m.split && n <= (beside ? kEncRoomSentences : kEncFew); }

// Sentences that the layers' panels of a handle are made for: those of the forms that its batches, of at most max_batch
// sentences and max_words words, can take.
inline int encoder_panel_sentences(const EncoderModel& m, int max_batch, int max_words) {
  if (max_batch > kEncLayers && encoder_form(m, kEncLayers + 1, max_words) == EncoderForm::kPipelined) return std::min(max_batch, kEncPipelined);
  return std::min(max_batch, kEncLayers);
}

}  // namespace linmt
