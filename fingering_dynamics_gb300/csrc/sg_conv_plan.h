// Tiles and ring of the persistent tcgen05 convolutions (sg_conv.cu), plain C++ so
// that they can be checked without a GPU.
#pragma once

#include <algorithm>

namespace sg {

constexpr int kConvPixels = 128;  // operand rows of an MMA

// The tile of a width: W in equal parts (the last may be shorter), as many rows as
// fit 128 operand rows at a pitch of the part plus `gap`; the parts that give the
// fewest tiles.
inline void tile_box(int H, int W, int gap, int& bw, int& rows) {
  long long best = 0;
  const int least = (W + kConvPixels - 1) / kConvPixels;
  for (int k = least; k <= std::max(least, 16) && k <= W; ++k) {
    const int w = (W + k - 1) / k, r = std::min((kConvPixels + gap) / (w + gap), 254);
    const long long tiles = (long long)((W + w - 1) / w) * ((H + r - 1) / r);
    if (best == 0 || tiles < best) {
      best = tiles;
      bw = w;
      rows = r;
    }
  }
}

// Ring of input boxes of `a` bytes and weights of `b` bytes a chunk, nk chunks, in
// `room` bytes: the weights stay where two stages of the ring fit beside them (or
// all the chunks there are); else they share the stages.
struct ConvRing {
  int resident, stages;
};
inline ConvRing conv_ring(int nk, int a, int b, int room, int most) {
  ConvRing r;
  r.resident = nk * b + (nk < 2 ? 1 : 2) * a <= room;
  r.stages = std::min(most, (room - (r.resident ? nk * b : 0)) / (a + (r.resident ? 0 : b)));
  return r;
}

}  // namespace sg
