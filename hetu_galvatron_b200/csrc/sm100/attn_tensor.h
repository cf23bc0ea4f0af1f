// Tensor descriptor of the attention entry points (mirrored by ``AttnTensor`` in ops/_lib.py): base pointer, strides
// (elements) over s and b, number of head slots in a token row, and the head -> slot map (gs, hs, off).
#pragma once

struct HgAttnTensor {
  void* ptr;
  long long ss, sb;
  int slots;
  int gs, hs, off;
};

// Most pieces of scratch that the backward keeps dS in.
constexpr int kHgDsPieces = 64;
