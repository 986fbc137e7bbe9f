// What the host hands to the kernels that run one pass over the copies of all ranks of a world that lives on one device:
// of up to eight ranks world_tree_kernel (world_tree.cu) for floating sums, and for integers wherever whole sums are stored (a
// flat sum then, whatever the plan), and world_copy_kernel for copies; for the rest world_reduce_kernel (world_reduce.cu), which
// interprets its program.  Programs are built by planner/world_program.hpp.
#pragma once
#include <stddef.h>
#include <stdint.h>

#include "nway_layout.h"

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
// these.
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

// ---- programs the tree kernel is compiled for -----------------------------------------------------------------------
// A program's steps as one word: start | pop << 1 | rounds << 2 of step k in bits 4k .. 4k + 3.  As text: S starts, a
// adds, r is a round, p a pop.
constexpr int kTreeThreads = 128;
constexpr int kTreeRanks = 8, kTreeRounds = 6;   // ranks, and rounds of one entry, of a program in this form
constexpr uint32_t tree_code(const char* s) {
  uint32_t code = 0;
  for (int k = -1; *s; ++s) {
    if (*s == 'S') code |= 1u << (4 * ++k);
    else if (*s == 'a') ++k;
    else if (*s == 'r') code += 4u << (4 * k);
    else if (*s == 'p') code |= 2u << (4 * k);
  }
  return code;
}
// The shapes that the planner proposes for two to eight ranks: flat, trees of two or three levels, rings, and the trees
// with lonely ranks (whose blocks follow two codes, by the group a lonely rank joins).
struct WorldTree {
  int ranks;
  uint32_t code[2];   // in ascending order; the same twice where all blocks follow one
};
constexpr WorldTree tree(int ranks, const char* a, const char* b = nullptr) {
  const uint32_t x = tree_code(a), y = b ? tree_code(b) : x;
  return x < y ? WorldTree{ranks, {x, y}} : WorldTree{ranks, {y, x}};
}
constexpr WorldTree kWorldTrees[] = {
    tree(2, "S a"), tree(3, "S a a"), tree(4, "S a a a"), tree(5, "S a a a a"), tree(6, "S a a a a a"), tree(7, "S a a a a a a"),
    tree(8, "S a a a a a a a"),
    tree(4, "S ar S arp"),                                        // 2*2
    tree(6, "S ar S arp S arp"), tree(6, "S a ar S a arp"),       // 2*3, 3*2
    tree(8, "S ar S arp S arp S arp"), tree(8, "S a a ar S a a arp"), tree(8, "S ar S arr S ar S arrp"),   // 2*4, 4*2, 2*2*2
    tree(3, "S ar a"), tree(4, "S ar ar a"), tree(5, "S ar ar ar a"), tree(6, "S ar ar ar ar a"), tree(7, "S ar ar ar ar ar a"),
    tree(8, "S ar ar ar ar ar ar a"),                             // rings
    tree(5, "S a ar S arp", "S ar S a arp"),                      // 2*2+1
    tree(7, "S a ar S arp S arp", "S ar S a arp S arp"),          // 2*3+1
    tree(7, "S a a ar S a arp", "S a ar S a a arp"),              // 3*2+1
    tree(8, "S a ar S a arp S arp", "S ar S a arp S a arp"),      // 2*3+2
};
constexpr int kFlatTrees = kTreeRanks - 1;   // the first ones: 2 .. 8 ranks in one sum
constexpr int kWorldTreeCount = sizeof kWorldTrees / sizeof kWorldTrees[0];

// One block's program beside its code: the rank of step k in bits 3k .. 3k + 2, the ranks that get the result in bits
// 24 .. 31, the block in 32 .. 34, which of the two codes in 35, and from 36 on four bits a round: the rank whose copy ends
// there, or 15.
constexpr int kTreeMask = 24, kTreeBlock = 32, kTreeWhich = 35, kTreeStore = 36;

// 224 bytes, looked up by few and short chains: the interpreter's 1 KB of tables costs each launch one miss of the constant
// cache after the other.
struct WorldTreeArgs {
  uint64_t entry[kTreeRanks];
  const void* in[kTreeRanks];
  void* out[kTreeRanks];
  uint64_t total_bytes, block_bytes;
  float scale;
  Seam seam;        // (nway_layout.h); CTAs counted along the blocks first
  uint8_t es;
  uint8_t streams;  // what is read, and by a gather written, leaves L2 before other data (halves_stream)
};

// Whether a half of an all-reduce tells L2 (126 MB) that what it reads, and as a gather what it writes, may leave first.
// `copies`: bytes of all ranks' copies.
// What the reduce-scatter leaves is what the gather reads; everything else it touches has served.  Worth saying only where the
// copies take a good part of L2: both halves of four ranks of 6 MB took 7.0 us, 7.6 with it.
// The gather's copies are read by whoever comes behind, and are found in L2 as long as that holds them all: with an update of
// the owned blocks between the halves and a sum over every copy behind them, us with neither / the reduce-scatter / both saying it:
//   copies   58 MB               84 MB               100 MB              112 MB              128 MB
//   2 ranks  57.6 / 57.1 / 59.9  71.7 / 70.5 / 73.1  86.8 / 82.1 / 80.1  96.3 / 88.1 / 86.1  107.7/100.9/ 95.6
//   4 ranks  74.0 / 73.7 / 80.6  90.8 / 88.8 / 93.1  103.2/ 98.1/100.1   112.9/108.1/104.7   123.7/116.1/112.3
//   8 ranks  115.6/114.8/121.4   129.5/126.8/135.9   139.9/136.4/141.4   151.1/143.9/145.6   163.1/155.8/153.7
// The halves alone, nobody between or behind them, 4 ranks: 19.7 / 19.7 / 18.4, 27.8 / 27.2 / 26.0, 32.9 / 32.8 / 30.6, 36.9 / 36.1 /
// 34.4, 43.0 / 42.1 / 39.5.
inline bool halves_stream(bool gather, uint64_t copies) { return copies >= (gather ? 100u << 20 : 32u << 20); }

}  // namespace ftk
