// Work list of a tensor-core prefill call: units of query rows, cut along their keys where that pays, dealt to
// clusters.  Host code only.
#pragma once
#include <stddef.h>
#include <stdint.h>

#include <algorithm>
#include <utility>
#include <vector>

namespace kpx {

constexpr int kTile = 128;          // query rows of an item, keys of a tile
constexpr int kMaxPartSlots = 320;  // slots for parts in the work area
constexpr int kMaxMerges = kMaxPartSlots / 2;
constexpr int kMaxParts = 8;

// A unit: `ntok` tokens of sequence `seq` from query row `tok0` on (cache position pos0), query heads
// group * group_heads and on, and its share [tile0, tile1) of the key tiles.  Item 0 has the first
// `tokens an item`, item 1 the rest; where they fit one item, it is item 1.  part >= 0: the keys were
// cut, and the unnormalised rows go to that slot.
struct alignas(16) Unit {
  int32_t seq, group, tok0, ntok, pos0, tile0, tile1, part;
};
// A unit whose keys were cut: `parts` slots from slot0 on.
struct alignas(16) Merge {
  int32_t group, tok0, ntok, slot0, parts, pad[3];
};

// What a call launches: units order[start[c]] .. order[start[c + 1] - 1] are cluster c's.
struct WorkList {
  std::vector<Unit> units;
  std::vector<int32_t> order, start;
  std::vector<Merge> merges;
};

// The units of a call, their keys whole: 2 * item_tokens tokens each, for every group of query heads.
inline std::vector<Unit> whole_units(const int32_t* cu_q_lens, const int32_t* start_pos, int batch, int groups,
                                     int item_tokens) {
  std::vector<Unit> units;
  units.reserve(size_t(cu_q_lens[batch] / (2 * item_tokens) + batch) * size_t(groups));
  for (int32_t b = 0; b < batch; ++b) {
    const int32_t n = cu_q_lens[b + 1] - cu_q_lens[b];
    for (int32_t t = 0; t < n; t += 2 * item_tokens) {
      const int ntok = std::min(2 * item_tokens, n - t), pos = start_pos[b] + t, end = (pos + ntok - 1) / kTile + 1;
      for (int32_t h = 0; h < groups; ++h) units.push_back(Unit{b, h, cu_q_lens[b] + t, ntok, pos, 0, end, -1});
    }
  }
  return units;
}

// Unit indexes, longest first (units of a length in their order).  Lengths are counted, not compared: a tile
// for every 128 cached tokens, and a call makes its list while the GPU waits.
inline std::vector<int32_t> longest_first(const std::vector<Unit>& units) {
  int most = 0;
  for (const Unit& d : units) most = std::max(most, d.tile1 - d.tile0);
  std::vector<int32_t> at(size_t(most) + 2, 0), order(units.size(), 0);
  for (const Unit& d : units) ++at[size_t(most - (d.tile1 - d.tile0)) + 1];
  for (int i = 0; i <= most; ++i) at[size_t(i) + 1] += at[size_t(i)];
  for (size_t i = 0; i < units.size(); ++i) order[size_t(at[size_t(most - (units[i].tile1 - units[i].tile0))]++)] = int32_t(i);
  return order;
}

// Units dealt to `clusters` clusters, longest first to the least loaded; fills order (unit indexes,
// cluster by cluster) and start.  Returns the largest load.  A unit costs its tiles and kUnitCost.
constexpr int kUnitCost = 1;
inline int deal_units(const std::vector<Unit>& units, int clusters, std::vector<int32_t>& order, std::vector<int32_t>& start) {
  const int n = int(units.size());
  const std::vector<int32_t> by_length = longest_first(units);
  std::vector<int32_t> owner(size_t(n), 0), load(size_t(clusters), 0), heap(size_t(clusters), 0);
  auto cost = [&](int i) { return units[size_t(i)].tile1 - units[size_t(i)].tile0 + kUnitCost; };
  for (int c = 0; c < clusters; ++c) heap[size_t(c)] = c;  // a heap with the least loaded on top (ties: lowest index)
  auto less = [&](int a, int b) { return load[size_t(a)] != load[size_t(b)] ? load[size_t(a)] < load[size_t(b)] : a < b; };
  start.assign(size_t(clusters) + 1, 0);
  int longest = 0;
  for (int i : by_length) {
    const int c = heap[0];
    owner[size_t(i)] = c;
    load[size_t(c)] += cost(i);
    longest = std::max(longest, load[size_t(c)]);
    ++start[size_t(c) + 1];
    for (int at = 0;;) {  // sift down
      int child = 2 * at + 1;
      if (child >= clusters) break;
      if (child + 1 < clusters && less(heap[size_t(child) + 1], heap[size_t(child)])) ++child;
      if (!less(heap[size_t(child)], heap[size_t(at)])) break;
      std::swap(heap[size_t(at)], heap[size_t(child)]);
      at = child;
    }
  }
  for (int c = 0; c < clusters; ++c) start[size_t(c) + 1] += start[size_t(c)];
  std::vector<int32_t> at(start.begin(), start.end() - 1);
  order.assign(size_t(n), 0);
  for (int i : by_length) order[size_t(at[size_t(owner[size_t(i)])]++)] = i;
  return longest;
}

// Cuts unit d along its keys into k parts, slots from `slot` on.
inline void cut_unit(const Unit& d, int k, int& slot, std::vector<Unit>& units, std::vector<Merge>& merges) {
  const int tiles = d.tile1 - d.tile0;
  k = std::min(k, tiles);
  if (k < 2 || slot + k > kMaxPartSlots || int(merges.size()) >= kMaxMerges) {
    units.push_back(d);
    return;
  }
  merges.push_back(Merge{d.group, d.tok0, d.ntok, slot, k, {0, 0, 0}});
  for (int j = 0; j < k; ++j) {
    Unit c = d;
    c.tile0 = d.tile0 + int(int64_t(tiles) * j / k);
    c.tile1 = d.tile0 + int(int64_t(tiles) * (j + 1) / k);
    c.part = slot++;
    units.push_back(c);
  }
}

// What a cut costs, in tiles: a second launch, the parts' rows written and read in fp32, and the clock, which rises
// where a last round leaves clusters idle and no longer does when they share its work.  Fitted to calls cut and whole
// (us, parts, tiles of the fullest cluster): 28/4 heads, 4 x 512 tokens behind 1536 79.7 / 70.5 (72, 52 / 61); 32/8, 20 x
// 64 behind 1500 51.9 / 53.9 (72, 32 / 42); 8/8, 10 x 128 behind 1000 25.4 / 27.5 (48, 13 / 20); 32/8, 448 behind 6000
// 65.7 / 60.0 (280, 44 / 52); 64/8, 512 behind 16384 301 / 307 (216, 233 / 263); 8/8, 16 x 128 behind 8192 164.4 / 162.2
// (216, 118 / 132).
constexpr int cut_cost(int64_t parts, int64_t load) { return int(4 + parts / 24 + load / 20); }

// The work list of whole units (a cluster can take any number of them).  split: -1 cut where it pays, 0 never, 2..4
// always, into that many parts (tests).
inline WorkList plan_units(std::vector<Unit> units, int clusters, int split) {
  WorkList w;
  const int n = int(units.size());
  if (split >= 2) {  // test knob: always cut
    int slot = 0;
    for (const Unit& d : units) cut_unit(d, std::min(split, 4), slot, w.units, w.merges);
    deal_units(w.units, clusters, w.order, w.start);
    return w;
  }
  int64_t tiles = 0;
  int longest = 0;
  for (const Unit& d : units) {
    tiles += d.tile1;
    longest = std::max(longest, d.tile1);
  }
  w.units.swap(units);
  int load = deal_units(w.units, clusters, w.order, w.start);
  // Cut along the keys where whole units leave many clusters idle for long.
  const int64_t even = (tiles + int64_t(n) * kUnitCost + clusters - 1) / clusters;
  const int idle = load - int(even);
  if (split == 0 || idle <= cut_cost(0, 0) || idle * int64_t(8) <= even) return w;
  const std::vector<Unit> whole = w.units;
  const std::vector<int32_t> by_length = longest_first(whole);
  // The rules below go by means.  Each gives the best cut that has a slot for every part and, where a finer one would
  // be better, that one with the longest units cut first; what is kept is what the dealing bears out.  (Chosen as if
  // slots had no end, the longest units stayed whole and the cut was for nothing: 512 tokens, 28/4 heads behind 7168
  // tokens 86 us against 67 uncut, 32/8 behind 10752 119 against 104, behind 32768 335 against 308.)
  auto parts_of = [](const WorkList& cut) {
    int64_t n = 0;
    for (const Merge& m : cut.merges) n += m.parts;
    return n;
  };
  auto keep_if_shorter = [&](WorkList&& cut) {
    if (cut.merges.empty()) return;
    const int of_parts = deal_units(cut.units, clusters, cut.order, cut.start);
    const int with_cut = of_parts + cut_cost(parts_of(cut), of_parts);
    if (with_cut >= load) return;
    load = with_cut;
    w = std::move(cut);
  };
  if (longest > even) {
    // A few long units: no part longer than a k-th of the longest, k by the rounds that the parts make.  (Cut to
    // an even share instead, whatever the rounds: 512 tokens behind 3584, 32/8 heads, 64 units on 74 clusters, 51 us
    // against 42; 256 behind 8192, 28/4, 71 against 59; 256 behind 3840, 32/8, 41 against 36.)
    int cap = 0, best = load, cap_slots = 0, best_slots = load;  // of all k; of those with a slot for every part
    for (int k = 2; k <= kMaxParts; ++k) {
      const int c = (longest + k - 1) / k;
      int64_t count = 0, slots = 0, cuts = 0;
      for (const Unit& d : whole) {
        const int parts = (d.tile1 + c - 1) / c;
        count += parts;
        slots += parts > 1 ? parts : 0;
        cuts += parts > 1;
      }
      const int64_t rounds = (count + clusters - 1) / clusters, mean = (tiles + count * kUnitCost + count - 1) / count;
      const int64_t of_parts = std::max<int64_t>(c + kUnitCost, rounds * mean);
      const int cost = int(of_parts) + cut_cost(std::min<int64_t>(slots, kMaxPartSlots), of_parts);
      if (cost < best) {
        best = cost;
        cap = c;
      }
      if (cost < best_slots && slots <= kMaxPartSlots && cuts <= kMaxMerges) {
        best_slots = cost;
        cap_slots = c;
      }
    }
    auto cut_to = [&](int c) {  // the longest first: those beyond the slots stay whole
      WorkList cut;
      cut.units.reserve(whole.size() + kMaxPartSlots);
      int slot = 0;
      for (int32_t i : by_length)
        cut_unit(whole[size_t(i)], std::min(kMaxParts, (whole[size_t(i)].tile1 + c - 1) / c), slot, cut.units, cut.merges);
      return cut;
    };
    if (cap_slots > 0) keep_if_shorter(cut_to(cap_slots));
    if (cap > 0 && cap != cap_slots) keep_if_shorter(cut_to(cap));
  } else {  // many units of like length and a thin last round: the shortest, a round's remainder, are cut
    const int rest = n % clusters;
    const int t = whole[size_t(by_length[size_t(n - 1)])].tile1 + 1, before = load - t;
    int k = 1, best = (t + kUnitCost) * 8, k_slots = 1;  // eighths of a tile
    for (int c = 2; c <= kMaxParts && rest > 0; ++c) {
      const int rounds = (rest * c + clusters - 1) / clusters;
      const int of_parts = rounds * (t * 8 / c + 8 * kUnitCost);
      const int cost = of_parts + 8 * cut_cost(std::min(rest * c, kMaxPartSlots), before + of_parts / 8);
      if (cost < best) {
        best = cost;
        k = c;
        if (rest * c <= kMaxPartSlots) k_slots = c;
      }
    }
    auto cut_rest = [&](int c) {
      WorkList cut;
      cut.units.reserve(whole.size() + kMaxPartSlots);
      int slot = 0;
      for (int i = 0; i < n - rest; ++i) cut.units.push_back(whole[size_t(by_length[size_t(i)])]);
      for (int i = n - rest; i < n; ++i) cut_unit(whole[size_t(by_length[size_t(i)])], c, slot, cut.units, cut.merges);
      return cut;
    };
    if (k_slots > 1) keep_if_shorter(cut_rest(k_slots));
    if (k > k_slots) keep_if_shorter(cut_rest(k));
  }
  return w;
}

}  // namespace kpx
