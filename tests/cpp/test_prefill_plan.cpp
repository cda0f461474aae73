// The work list of tensor-core prefill calls: every unit's keys are there once, parts have a slot each, and a call is
// cut only where that shortens its fullest cluster by more than the cut costs.
#include <cstdio>
#include <set>

#include "kpx_prefill_plan.h"

using namespace kpx;

static int bad = 0;
#define EXPECT(what)                                                       \
  do {                                                                     \
    if (!(what) && ++bad <= 20) std::printf("%s: not %s\n", label, #what); \
  } while (0)

struct Call {
  int q_heads, kv_heads;
  std::vector<int> lens, starts;
};

static int fullest(const WorkList& w, int clusters) {
  int most = 0;
  for (int c = 0; c < clusters; ++c) {
    int load = 0;
    for (int i = w.start[size_t(c)]; i < w.start[size_t(c) + 1]; ++i) {
      const Unit& d = w.units[size_t(w.order[size_t(i)])];
      load += d.tile1 - d.tile0 + kUnitCost;
    }
    most = std::max(most, load);
  }
  return most;
}

static void check(const Call& call, int clusters, int split) {
  char label[160];
  std::snprintf(label, sizeof label, "%d/%d heads, %zu sequences, first %d tokens behind %d, %d clusters, split %d", call.q_heads,
                call.kv_heads, call.lens.size(), call.lens[0], call.starts[0], clusters, split);
  const int mul = call.q_heads / call.kv_heads, item_tokens = kTile / mul;
  std::vector<int32_t> cu{0}, start(call.starts.begin(), call.starts.end());
  for (int n : call.lens) cu.push_back(cu.back() + n);
  const std::vector<Unit> whole = whole_units(cu.data(), start.data(), int(call.lens.size()), call.kv_heads, item_tokens);
  const WorkList uncut = plan_units(whole, clusters, 0), w = plan_units(whole, clusters, split);
  EXPECT(uncut.merges.empty() && uncut.units.size() == whole.size());

  EXPECT(w.order.size() == w.units.size() && w.start.size() == size_t(clusters) + 1);
  EXPECT(w.start[0] == 0 && w.start[size_t(clusters)] == int(w.units.size()));
  EXPECT(std::set<int32_t>(w.order.begin(), w.order.end()).size() == w.units.size());
  EXPECT(w.merges.size() <= size_t(kMaxMerges));

  int64_t tiles = 0, tiles_whole = 0;
  std::set<int> slots;
  size_t parts = 0;
  for (const Unit& d : whole) tiles_whole += d.tile1;
  for (const Unit& d : w.units) {
    EXPECT(d.tile0 < d.tile1);
    tiles += d.tile1 - d.tile0;
    if (d.part < 0) continue;
    ++parts;
    EXPECT(d.part < kMaxPartSlots);
    slots.insert(d.part);
  }
  EXPECT(tiles == tiles_whole && slots.size() == parts);
  for (const Merge& m : w.merges) {  // its slots hold parts that follow one another, of its rows
    EXPECT(m.parts >= 2 && m.parts <= kMaxParts);
    int at = 0;
    for (const Unit& d : w.units)
      if (d.part >= m.slot0 && d.part < m.slot0 + m.parts) {
        EXPECT(d.tile0 == at && d.tok0 == m.tok0 && d.group == m.group && d.ntok == m.ntok);
        at = d.tile1;
      }
    EXPECT(at > 0);
    parts -= size_t(m.parts);
  }
  EXPECT(parts == 0);

  int cut_parts = 0;
  for (const Merge& m : w.merges) cut_parts += m.parts;
  if (split < 0) {
    const int before = fullest(uncut, clusters), after = fullest(w, clusters);
    if (w.merges.empty()) EXPECT(w.units.size() == whole.size() && after == before);
    else EXPECT(after + cut_cost(cut_parts, after) < before);
  }
}

int main() {
  // many long units: more parts wanted than there are slots
  for (int behind : {3584, 7168, 10752, 15872, 16384, 32768, 65536, 131072})
    for (int clusters : {74, 66, 16}) {
      check({32, 8, {512}, {behind}}, clusters, -1);
      check({28, 4, {512}, {behind}}, clusters, -1);
      check({64, 8, {256}, {behind}}, clusters, -1);
      check({16, 2, {1024}, {behind}}, clusters, -1);
      check({32, 8, {128, 128, 128, 128}, {behind, behind, behind, behind}}, clusters, -1);
    }
  // a remainder of 45 units and more
  for (int n = 1; n < 74; ++n) check({8, 8, std::vector<int>(size_t(n), 256), std::vector<int>(size_t(n), 8000)}, 74, -1);
  uint64_t x = 1;
  auto draw = [&](int lo, int hi) {
    x = x * 6364136223846793005ull + 1442695040888963407ull;
    return lo + int((x >> 33) % uint64_t(hi - lo + 1));
  };
  const int heads[][2] = {{32, 8}, {28, 4}, {12, 2}, {16, 2}, {40, 8}, {64, 8}, {14, 2}, {8, 8}, {128, 1}};
  for (int i = 0; i < 4000; ++i) {
    const int* h = heads[draw(0, 8)];
    Call call{h[0], h[1], {}, {}};
    const int batch = draw(1, draw(1, 24)), top = 1 << draw(4, 11), far = 1 << draw(0, 16);
    for (int b = 0; b < batch; ++b) {
      call.lens.push_back(draw(1, top));
      call.starts.push_back(draw(0, far));
    }
    check(call, i % 4 ? 74 : draw(1, 96), i % 5 ? -1 : draw(2, 4));
  }
  if (bad) std::printf("%d expectations failed\n", bad);
  return bad != 0;
}
