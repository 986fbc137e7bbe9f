// A plan as one pass over the data of every rank, for worlds whose ranks share a device.
//
// A plan is element-wise: what a rank's copy of block b becomes depends on the other ranks' copies of block b at the
// same offset only.  So the whole plan (or one half of it) for one offset is an expression over the ranks' inputs,
// and one thread that holds the `world` values of an offset can evaluate it and store every copy the plan changes:
// each input is read once and each result written once, where running the stages one after another moves the
// intermediate copies through memory as well.
//
// build_world_program() executes the plan symbolically and linearises each block's expression, keeping the order of
// the additions and the places where a copy is stored - and rounded to the element type - between two stages, so
// that the results are the same bits.  Plans it cannot linearise (a block that ends in two different expressions, a
// nesting deeper than the kernel's stack) come back with ok = false and are run stage by stage.
#pragma once
#include <algorithm>
#include <cstdint>
#include <list>
#include <map>
#include <mutex>
#include <vector>

#include "../kernels/world_dev.h"
#include "../runtime/dev_plan.hpp"
#include "plan.hpp"

namespace ft {

struct WorldProgram {
  bool ok = false;
  int depth = 0;                             // 0: plain sums; else the accumulators put aside at the same time, at least 1
  std::vector<ftk::WorldEntry> entries;      // one per block and pass over it
  std::vector<ftk::WorldStep> steps;         // entries[i] uses steps [first, first + nsteps)
  // The same for the kernels with programs compiled in, where there is one for this program (compact_world_program).
  int tree = -1;                             // index into kWorldTrees
  bool copies = false;                       // every entry is one step: copies only
  bool partial = false;                      // some copy ends as a part of the sum
  std::vector<uint64_t> words;               // WorldTreeArgs::entry
};

// Finds the compiled form of a finished program: all entries take every rank's copy once and follow one or two codes of
// kWorldTrees, or are copies.  Leaves tree = -1 and copies = false where there is none.
inline void compact_world_program(int world, WorldProgram* wp) {
  if (!wp->ok || world > ftk::kTreeRanks || wp->entries.empty() || wp->entries.size() > (std::size_t)ftk::kTreeRanks) return;
  std::vector<uint32_t> codes;
  std::vector<uint64_t> words;
  bool copies = true, whole = true, partial = false;
  for (const ftk::WorldEntry& e : wp->entries) {
    uint64_t word = (uint64_t)(e.mask & 0xff) << ftk::kTreeMask | (uint64_t)e.block << ftk::kTreeBlock;
    uint32_t code = 0;
    int rounds = 0;
    copies = copies && e.nsteps == 1 && !e.scaled && wp->steps[e.first].rounds == 0;
    whole = whole && e.nsteps == world && e.scaled;
    if (e.nsteps > ftk::kTreeRanks || e.block >= ftk::kTreeRanks) return;
    for (int k = 0; k < e.nsteps; ++k) {
      const ftk::WorldStep& s = wp->steps[e.first + k];
      if (s.rounds > 3 || rounds + s.rounds > ftk::kTreeRounds) return;
      word |= (uint64_t)s.rank << (3 * k);
      code |= (uint32_t)(s.start | s.pop << 1 | s.rounds << 2) << (4 * k);
      for (int r = 0; r < s.rounds; ++r) {
        partial = partial || s.store[r] != ftk::kNoStore;
        word |= (uint64_t)(s.store[r] == ftk::kNoStore ? 15 : s.store[r]) << (ftk::kTreeStore + 4 * rounds++);
      }
    }
    words.push_back(word);
    codes.push_back(code);
  }
  if (copies) {
    wp->copies = true;
    wp->words = words;
    return;
  }
  const uint32_t lo = *std::min_element(codes.begin(), codes.end()), hi = *std::max_element(codes.begin(), codes.end());
  for (std::size_t i = 0; i < codes.size(); ++i) {
    if (codes[i] != lo && codes[i] != hi) return;
    if (codes[i] != lo) words[i] |= 1ull << ftk::kTreeWhich;
  }
  for (int t = 0; whole && t < ftk::kWorldTreeCount; ++t)
    if (ftk::kWorldTrees[t].ranks == world && ftk::kWorldTrees[t].code[0] == lo && ftk::kWorldTrees[t].code[1] == hi) {
      wp->tree = t;
      wp->partial = partial;
      wp->words = words;
    }
}

// What the tree and copy kernels get of it for the tensors of a call.
inline void fill_tree_args(const WorldProgram& wp, int world, const void* const* in, void* const* out, ftk::WorldTreeArgs* a) {
  for (int r = 0; r < ftk::kTreeRanks; ++r) {
    a->entry[r] = r < (int)wp.words.size() ? wp.words[r] : 0;
    a->in[r] = r < world ? in[r] : nullptr;
    a->out[r] = r < world ? out[r] : nullptr;
  }
}

// What the kernel gets of a program for the tensors of a call.  False: more than its parameters hold.
template <int RANKS>
bool fill_world_args(const WorldProgram& wp, int world, const void* const* in, void* const* out, ftk::WorldArgs<RANKS>* a) {
  constexpr std::size_t cap = ftk::WorldArgs<RANKS>::kSteps;
  if (world > RANKS || wp.entries.size() > (std::size_t)RANKS || wp.steps.size() > cap) return false;
  std::copy(wp.entries.begin(), wp.entries.end(), a->entry);
  std::size_t k = 0;
  for (const ftk::WorldStep& s : wp.steps) {
    a->ptr[k] = in[s.rank];
    a->code[k] = (uint8_t)(s.start | s.pop << 1 | s.rounds << 2);
    std::copy(s.store, s.store + ftk::kMaxRounds, a->store[k]);
    ++k;
  }
  for (const std::size_t end = std::min(cap, k + ftk::kWorldGroup - 1); k < end; ++k) a->ptr[k] = in[0];
  for (int r = 0; r < RANKS; ++r) a->ptr[cap + r] = r < world ? out[r] : nullptr;
  return true;
}

enum class WorldPhase { all, reduce_scatter, all_gather };

class WorldProgramBuilder {
 public:
  explicit WorldProgramBuilder(int world) : world_(world) {
    for (int r = 0; r < world; ++r) nodes_.push_back(Node{{}, r, false});
  }

  WorldProgram run(const Plan& p, WorldPhase phase) {
    WorldProgram out;
    const int half = p.num_stages / 2, begin = phase == WorldPhase::all_gather ? half : 0;
    const int end = phase == WorldPhase::reduce_scatter ? half : p.num_stages;
    for (int b = 0; b < world_; ++b) {
      std::vector<int> val(world_);
      for (int r = 0; r < world_; ++r) val[r] = r;   // node r: rank r's copy before the call
      for (int s = begin; s < end; ++s) {
        const std::vector<int> before = val;   // a plan reads nothing in a stage that the stage writes
        for (int r = 0; r < world_; ++r)
          for (const Pull& pl : p.stages[r][s].pulls) {
            if (pl.block != b) continue;
            if (!pl.reduce) { val[r] = before[pl.srcs[0]]; continue; }
            std::vector<int> kids{val[r]};
            for (int q : pl.srcs) kids.push_back(before[q]);
            val[r] = make(kids, s == half - 1);
          }
      }
      if (!(phase == WorldPhase::all_gather ? gather(b, val, &out) : reduce(b, val, phase, &out))) return WorldProgram{};
    }
    out.ok = true;
    return out;
  }

  // All copies summed in the order first, first + 1, ... (modulo the world) in one go; every rank gets the result.
  void flat(int block, int first, WorldProgram* out) const {
    ftk::WorldEntry e{};
    e.block = (uint16_t)block;
    e.first = (uint16_t)out->steps.size();
    e.nsteps = (uint16_t)world_;
    e.scaled = 1;
    e.mask = everyone();
    for (int k = 0; k < world_; ++k) out->steps.push_back(step((first + k) % world_, k == 0));
    add(e, out);
    out->ok = true;
  }

 private:
  struct Node {
    std::vector<int> kids;   // empty: the copy of rank `rank`
    int rank;
    bool scaled;             // made in the stage that finishes the reduction
  };
  static void add(const ftk::WorldEntry& e, WorldProgram* out) {
    out->entries.push_back(e);
  }
  uint64_t everyone() const { return world_ >= 64 ? ~0ull : (1ull << world_) - 1; }
  static ftk::WorldStep step(int rank, bool start) {
    ftk::WorldStep s{};
    s.rank = (uint8_t)rank;
    s.start = start ? 1 : 0;
    for (uint8_t& d : s.store) d = ftk::kNoStore;
    return s;
  }
  // Equal expressions are one node: ranks that compute the same sum the same way agree.
  int make(const std::vector<int>& kids, bool scaled) {
    const auto key = std::make_pair(kids, scaled);
    auto it = known_.find(key);
    if (it != known_.end()) return it->second;
    nodes_.push_back(Node{kids, -1, scaled});
    return known_[key] = (int)nodes_.size() - 1;
  }
  int count(int node, std::vector<int>* leaves) const {
    if (nodes_[node].kids.empty()) { ++(*leaves)[node]; return 1; }
    int n = 0;
    for (int k : nodes_[node].kids) n += count(k, leaves);
    return n;
  }
  bool contains(int root, int node) const {
    if (root == node) return true;
    for (int k : nodes_[root].kids)
      if (contains(k, node)) return true;
    return false;
  }

  // Copies only: one entry per source rank that some other rank takes the block from.
  bool gather(int b, const std::vector<int>& val, WorldProgram* out) const {
    std::vector<uint64_t> mask(world_, 0);
    for (int r = 0; r < world_; ++r) {
      if (val[r] == r) continue;
      if (val[r] >= world_ || val[val[r]] != val[r]) return false;   // not a copy of a rank that keeps its own
      mask[val[r]] |= 1ull << r;
    }
    for (int q = 0; q < world_; ++q) {
      if (!mask[q]) continue;
      ftk::WorldEntry e{};
      e.block = (uint16_t)b;
      e.first = (uint16_t)out->steps.size();
      e.nsteps = 1;
      e.mask = mask[q];
      out->steps.push_back(step(q, true));
      add(e, out);
    }
    return true;
  }

  // One sum; copies that end as part of it are stored where they arise.
  bool reduce(int b, const std::vector<int>& val, WorldPhase phase, WorldProgram* out) {
    int root = 0;
    std::size_t most = 0;
    for (int r = 0; r < world_; ++r) {
      std::vector<int> leaves(world_, 0);
      const std::size_t n = (std::size_t)count(val[r], &leaves);
      if (n > most) { most = n; root = val[r]; }
    }
    std::vector<int> leaves(world_, 0);
    count(root, &leaves);
    for (int n : leaves)
      if (n != 1) return false;
    if (!nodes_[root].scaled) return false;
    ftk::WorldEntry e{};
    e.block = (uint16_t)b;
    e.first = (uint16_t)out->steps.size();
    e.scaled = 1;
    std::map<int, int> partial;   // node -> the rank whose copy ends as it
    for (int r = 0; r < world_; ++r) {
      if (val[r] == root) { e.mask |= 1ull << r; continue; }
      if (val[r] < world_) {
        if (val[r] != r) return false;   // takes another rank's input: not a reduction's doing
        continue;
      }
      if (phase == WorldPhase::all || !contains(root, val[r]) || nodes_[val[r]].scaled || !partial.emplace(val[r], r).second) return false;
    }
    if (phase == WorldPhase::all && e.mask != everyone()) return false;
    open_ = false;
    stack_ = 0;
    if (!eval(root, root, partial, out)) return false;
    e.nsteps = (uint16_t)(out->steps.size() - e.first);
    add(e, out);
    return true;
  }

  // Append the steps of `node`.  An accumulator that is running already when it starts is put aside.
  bool eval(int node, int root, const std::map<int, int>& partial, WorldProgram* out) {
    std::vector<int> kids = nodes_[node].kids;
    // x + y is y + x: the nested operand first needs no place to put the other one aside (the ring is a chain of these)
    if (kids.size() == 2 && nodes_[kids[0]].kids.empty() && !nodes_[kids[1]].kids.empty()) std::swap(kids[0], kids[1]);
    bool first = true;
    for (int k : kids) {
      const bool leaf = nodes_[k].kids.empty();
      if (leaf) {
        if (first) begin(out, k);
        else out->steps.push_back(step(k, false));
      } else {
        if (!eval(k, root, partial, out)) return false;
        if (!first) {   // fold the finished operand into the accumulator that was put aside for it
          out->steps.back().pop = 1;
          --stack_;
        }
      }
      first = false;
    }
    if (node == root) return true;
    ftk::WorldStep& last = out->steps.back();
    if (last.rounds >= ftk::kMaxRounds) return false;
    if (out->depth < 1) out->depth = 1;
    auto it = partial.find(node);
    last.store[last.rounds++] = it == partial.end() ? ftk::kNoStore : (uint8_t)it->second;
    last.pop = 0;
    return true;
  }
  void begin(WorldProgram* out, int leaf) {
    if (open_) {
      ++stack_;
      if (stack_ > out->depth) out->depth = stack_;
    }
    open_ = true;
    out->steps.push_back(step(leaf, true));
  }

  int world_, stack_ = 0;
  bool open_ = false;
  std::vector<Node> nodes_;
  std::map<std::pair<std::vector<int>, bool>, int> known_;
};

// What a call asks for: a plan, all copies summed in one order, or each block summed from its owner on.
enum class WorldForm { plan, flat, rotated };

// The programs of one world, each built by the first call that asks for it and kept: as many as shapes and phases in
// use.  Calls may come from several threads.
class WorldProgramCache {
 public:
  struct Entry {
    WorldForm form;
    WorldPhase phase;
    Shape shape;
    uint32_t nslots;   // receive slots of the plan's tagged-word form, whose limit holds for a call in one pass too
    WorldProgram program;
  };

  // Null where there is no such plan, or none that runs in one pass; nothing is kept of those.
  const Entry* get(int world, WorldForm form, WorldPhase phase, const int* widths, int nw, int lonely, bool ring) {
    std::lock_guard<std::mutex> lock(mu_);
    for (const Entry& e : entries_)
      if (e.form == form && e.phase == phase && e.shape.lonely == lonely && e.shape.ring == ring && (int)e.shape.widths.size() == nw &&
          std::equal(e.shape.widths.begin(), e.shape.widths.end(), widths))
        return &e;
    Entry e{form, phase, Shape{std::vector<int>(widths, widths + nw), lonely, ring}, 0, {}};
    WorldProgramBuilder builder(world);
    if (form == WorldForm::plan) {
      const Plan p = build_plan(world, nw > 0 ? e.shape : Shape::flat(world));
      if (!p.ok()) return nullptr;
      e.program = builder.run(p, phase);
      e.nslots = build_dev_plan(p, 0).plan.nslots;
    } else {
      for (int b = 0; b < (form == WorldForm::rotated ? world : 1); ++b) builder.flat(b, b, &e.program);
    }
    if (!e.program.ok) return nullptr;
    compact_world_program(world, &e.program);
    entries_.push_back(std::move(e));
    return &entries_.back();
  }
  std::size_t size() {
    std::lock_guard<std::mutex> lock(mu_);
    return entries_.size();
  }

 private:
  std::mutex mu_;
  std::list<Entry> entries_;   // their addresses stay
};

}  // namespace ft
