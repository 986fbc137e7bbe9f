// What the host hands to world_reduce_kernel (world_reduce.cu): one pass over the copies of all ranks of a world that
// lives on one device.  Programs are built by planner/world_program.hpp.
#pragma once
#include <stdint.h>

namespace ftk {

constexpr int kWorldRanks = 16;      // ranks, and entries of a program, that fit the kernel's parameters
constexpr int kMaxRounds = 4;        // copies that may be finished after one step
constexpr int kWorldGroup = 8;       // steps whose sources the kernel looks up together, also behind the last one
constexpr uint8_t kNoStore = 0xff;

// Take the next value: start an accumulator with it (a running one is put aside) or add it.  Then `rounds` times:
// round the accumulator to the element type as a stage of the plan does when it stores a copy, store it as rank
// store[i]'s copy if that is how the copy ends; between two rounds, and after the last one if `pop`, add the
// accumulator to the one put aside last.
struct WorldStep {
  uint8_t rank, start, rounds, pop;
  uint8_t store[kMaxRounds];
};
// One block's program: its steps, and the ranks that get the result.
struct WorldEntry {
  uint16_t block, first, nsteps, scaled;   // scaled: the result is multiplied by the call's scale (float types)
  uint64_t mask;
};

// What is left of a step in the kernel's parameters besides the pointer: start | pop << 1 | rounds << 2.
// One table of pointers: of step k the copy it takes, and from kSteps on the ranks' results.  The kernel looks the sources
// up in groups, past an entry's last step, without reading them: behind the last step of all lies rank 0's input or
// these.  (56 bytes more for that cost every call 0.24 us: 1048 bytes of parameters 2.58 us, 1104 bytes 2.82.)
template <int RANKS>
struct WorldArgs {
  static constexpr int kSteps = RANKS * RANKS;
  WorldEntry entry[RANKS];
  const void* ptr[kSteps + RANKS];
  uint8_t code[kSteps];
  uint8_t store[kSteps][kMaxRounds];
  uint64_t total_bytes, block_bytes;
  uint32_t es;
  float scale;
  static_assert(RANKS >= kWorldGroup - 1, "a group that starts with the last step ends inside the table");
};

}  // namespace ftk
