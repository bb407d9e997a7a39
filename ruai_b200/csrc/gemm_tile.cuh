// Sizes of the prefill GEMM's tiles (gemm_tc.cu): warps, rings in shared memory, tensor memory.  Plain C++, so that the rings' reuse can
// be checked on the host.
#pragma once
#include <cstddef>
#include <cstdint>

namespace gemm_tc {

// CB column blocks of 128 x NT rows of x per CTA.  Warps: 0 copies W, 1 and 2 issue MMAs, 3 copies x, then, with one column block,
// four that expand and four per 64 rows that drain; with two, sixteen that do both (96 registers for twenty warps are what the
// register file holds).  The A operand lies in tensor memory: from shared memory its reads, the writes of the expanding warps and the
// copies together took more than the 128 bytes per clock there are (measured: a stage's MMAs 1,900 clocks instead of 1,024).  Shared
// memory: a ring of packed stages (the scales of int4 in one of their own) and a ring of stages of x.
template <int BITS, int CB, int NT>
struct Tile {
  static constexpr int kCols = CB * 128;
  static constexpr int kDrains = CB * NT / 64;                           // draining warpgroups
  static constexpr bool kBoth = CB == 2;                                 // the draining warps expand as well
  static constexpr int kDrain0 = kBoth ? 4 : 8;                          // first draining warp
  static constexpr int kExpanders = kBoth ? 4 * kDrains : 4;             // warps
  static constexpr int kThreads = 32 * kDrain0 + 128 * kDrains;
  static constexpr uint32_t kWChunk = kCols * 16;                        // one 16-byte chunk of every column
  static constexpr int kChunks = BITS == 4 ? 2 : 4;                      // chunks per stage
  static constexpr uint32_t kWBytes = kChunks * kWChunk;
  static constexpr int kWSlots = CB == 2 ? 4 : 6;
  static constexpr uint32_t kPiece = NT * 128;                           // one piece of x of a stage
  static constexpr uint32_t kX = 2 * kPiece;                             // both
  // Tensor memory: three buffers of sums, then the A operand, 32 words per column block and stage.
  // A wait for a phase of a barrier by its parity also returns while the phase before is open, so whoever waits must know that one to be
  // over.  The buffers are used in turn, but by two issuing threads and two column blocks' draining warps: with a barrier per buffer one
  // party meets every other phase only.  With six, units u and u + 6 of a barrier belong to the same column block, or to the same
  // issuing thread; and where two threads take stages in turn (int4, one column block), a thread's units are at most five apart and
  // the read-out goes in order, so that the phase before its own (unit u - 9) is over.
  static constexpr uint32_t kUnitBars = 6;
  static constexpr uint32_t kACol0 = 3 * NT;
  static constexpr int kABufs = 4 / CB;
  static constexpr uint32_t kTmem = 512;
  static constexpr uint32_t kScale = BITS == 4 ? 2 * kCols * 4 : 0;      // scales of a stage
  // Scales of a stage are read when its sums are, and no barrier of their own says so.  A free packed slot for stage i means that stage
  // i - kWSlots is expanded, so that the MMAs of S = i - kWSlots - kABufs are done, and those waited for the read-out of every unit but
  // the last three up to S's own last.  With two column blocks a stage is two units at least: all of S - 2 has been read.  With one
  // column block and 32 k a stage is one unit: S - 3.  (A tile's last stage of one group between stages of two: S - 2.)
  static constexpr int kScaleSlots = kWSlots + kABufs + (CB == 1 ? 3 : 2);
  static constexpr uint32_t kFixed = kWSlots * kWBytes + kScaleSlots * kScale;
  static constexpr int kFit = (int)((230400 - 1024 - kFixed) / kX);
  static constexpr int kXSlots = kFit < 8 ? kFit : 8;
  static constexpr uint32_t off_w = kXSlots * kX, off_scale = off_w + kWSlots * kWBytes;
  static constexpr size_t kRed = (size_t)(NT + 8) * kCols * 4;           // split k: partial sums of this CTA's rows
  static constexpr size_t kRing = (size_t)kFixed + (size_t)kXSlots * kX;
  static constexpr size_t kSmem = 1024 + (kRing > kRed ? kRing : kRed);
  static_assert(kXSlots >= 3, "ring too short");
};

}  // namespace gemm_tc
