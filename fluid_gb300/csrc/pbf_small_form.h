// Which form of the whole-step kernel (pbf_small.cu) serves a scene: the rule on sizes, and the choice
// among the forms that a device accepts. Host code without CUDA.
#pragma once

#include <cstddef>

namespace pbf {

struct SmallFormSize {
  unsigned threads, per_block;  // threads and particles of a block
  unsigned on_sm;               // blocks on an SM
  bool cluster;                 // one thread block cluster of kClusterBlocks blocks
};
constexpr unsigned kClusterBlocks = 16;
constexpr unsigned kSmallTile = 1024;  // grid cells of a scan tile
constexpr int kSmallForms = 4;
constexpr SmallFormSize kSmallForm[kSmallForms + 1] = {
    {0, 0, 0, false}, {512, 64, 1, true}, {256, 32, 2, false}, {128, 128, 1, false}, {256, 256, 1, false}};

// Form 1 is one cluster of 16 blocks of 64 particles, 8 lanes each; 2 the same over the grid while two
// blocks of 32 particles fit on every SM; 3 and 4 one lane a particle with one block on an SM. Steps
// (us, no statistics) of 8 lanes over the grid / 1 lane / per-phase kernels: 512 particles
// 59 / 75 / 77, 4,096 65 / 85 / 96, 8,000 73 / 87 / 101; 19k - / 89 / 105, 33k - / 89 / 109; with a
// second block on some SMs the gain is gone (51k: 115 / 118). 4 lanes a particle over the grid: 8,000
// 77, 14k 93 (1 lane 89).
inline bool small_form_serves(int form, size_t n, size_t n_cells, size_t sms) {
  const SmallFormSize& f = kSmallForm[form];
  const size_t room = f.cluster ? kClusterBlocks : f.on_sm * sms;
  const size_t tiles = (n_cells + kSmallTile - 1) / kSmallTile;
  return (n + f.per_block - 1) / f.per_block <= room && tiles <= room;
}

// The first form that serves the scene and that the device takes (takes(form): asked only for the
// forms that serve it, and for no form after the first taken); 0: the per-phase kernels.
template <typename F>
inline int small_form_for(size_t n, size_t n_cells, size_t sms, F&& takes) {
  if (n == 0 || sms == 0) return 0;
  for (int form = 1; form <= kSmallForms; ++form)
    if (small_form_serves(form, n, n_cells, sms) && takes(form)) return form;
  return 0;
}

}  // namespace pbf
