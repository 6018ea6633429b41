// wave_shape.h — how the lock-step sweep kernel lays a block size out (no CUDA).
#pragma once
#include "wave_plan.h"

namespace bsp {

constexpr int kWaveWarps = 8;   // compute warps of a set
constexpr int kSlots = 8;       // steps staged ahead
constexpr int kRing = 8;        // steps whose results stay in shared memory

// Lanes and CTA shape of a block size.  Sizes 1, 2, 4, 8, 16: row-major
// blocks, lane l of a block's G holds pieces q * G + l of V values, those of PR
// block rows.  Others (3, 5, 6): column-major blocks, lane r holds block row r.
// A step begins with the operand reads of its 8 warps all at once, and the
// lanes that hold different rows of a block read the same operands again, so a
// block is spread over as few lanes as its registers allow.  8 x 8 over 16 lanes, two rows each, two items
// side by side, against a warp an item and two items in turn: 64^3 application
// 321 -> 300 us, 160 x 160 (IChol0) 298 -> 267, batched sweeps with 4
// right-hand sides 258 -> 175 us.  16 x 16 in one warp, four rows a lane in
// FP64, against two warps: 48^3 363 -> 351 us, 80 x 80 (IChol0) 1159 -> 607.  With
// several right-hand sides the registers do not suffice for that.
template <int BS, int R = 1> struct WaveDim {
  static constexpr bool kChunk = (BS & (BS - 1)) == 0;
  static constexpr int G = BS == 1 ? 1 : BS == 2 ? 2 : BS == 3 ? 4 : BS < 8 ? 8 : BS == 8 ? 16 : 32;  // lanes of a warp per item
  static constexpr int WPI = BS == 16 && R > 1 ? 2 : 1;                               // warps per item
  static constexpr int IPW = 32 / G;                                                   // items side by side in a warp
  static constexpr bool kItemMajor = BS >= 4;                                          // order of a step's blocks
  static constexpr int W = kWaveWarps * IPW / WPI;
  static constexpr int ECAP = W >= 128 ? 64 : W >= 64 ? 32 : W >= 16 ? 16 : 8;
  // three turns of polls in flight keep up with the short steps of small blocks
  // (24 x 20 rows of 2 x 2 blocks 42.7 -> 39.4 us, 40 x 36 x 44 of 4 x 4 133 -> 125);
  // larger ones need the registers (64^3 of 8 x 8: 321 -> 327 us with three)
  static constexpr int kFetchWarps = R == 1 && BS <= 4 ? 3 : 2;
  // measured on systems of one super-task (a line, a band); several right-hand
  // sides: on batches of 2D grids
  static constexpr double kStepUs = R > 1      ? (BS == 4 ? 0.45 : BS == 8 ? 0.65 : 1.2)
                                    : BS <= 2  ? 0.26
                                    : BS <= 4  ? 0.3
                                    : BS == 5  ? 0.36
                                    : BS == 8  ? 0.36
                                               : 0.42;
};
// External rows of a step with R right-hand sides: with more than one, what the
// tile of a 3D grid needs (the fetch warps hold them in registers).
template <int BS, int R> constexpr int wave_ecap() { return R == 1 ? WaveDim<BS>::ECAP : BS == 4 ? 12 : 8; }

template <int BS, int R> inline WaveShape wave_shape_of() {
  WaveShape s;
  s.W = WaveDim<BS, R>::W;
  s.ecap = wave_ecap<BS, R>();
  s.ring = kRing;
  s.slots = kSlots;
  s.item_major = WaveDim<BS>::kItemMajor;
  s.fetch = WaveDim<BS, R>::kFetchWarps;
  s.step_us = WaveDim<BS, R>::kStepUs;
  return s;
}

// Block sizes the lock-step kernel takes (FP64 vectors), and the shape of one
// (the plans for 2 and 4 right-hand sides are the same); W = 0: not taken.
#define BSP_WAVE_SIZES(X) X(1) X(2) X(3) X(4) X(5) X(6) X(8) X(16)
inline WaveShape wave_shape(int bs, int nrhs) {
  switch (bs) {
#define BSP_WAVE_CASE(B) \
  case B: return nrhs == 1 ? wave_shape_of<B, 1>() : wave_shape_of<B, 2>();
    BSP_WAVE_SIZES(BSP_WAVE_CASE)
#undef BSP_WAVE_CASE
    default: return WaveShape{};
  }
}
inline bool wave_supported(int bs) { return wave_shape(bs, 1).W > 0; }

}  // namespace bsp
