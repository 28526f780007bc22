// One issuing warp of the attention kernel against a model of what is around it: the K / V ring, its Q
// tile, the items and the epilogue. Barriers are what the hardware has, a phase count of which a wait
// sees one bit; copies land in any order; the other Q tile's warp releases a stage at once. Every step
// of the warp is checked against what is really there.
#include <cstdint>
#include <random>
#include <vector>

#include "attention_issue.cuh"

namespace {

enum Wrong { NONE, LAPPED, OVERWRITTEN, RELEASED_TWICE, ORDER, DEADLOCK, UNFINISHED };

struct Item {
  int n, lo, hi;
};
struct Fill {
  int item, visit;
  bool k, issued = false, landed = false, released = false;
};

struct World {
  std::mt19937_64 rng;
  std::vector<Item> items;
  std::vector<Fill> fills;
  std::vector<int> first;  // fill of each item
  Wrong wrong = NONE;
  int lazy = 0;            // a copy into this stage lands only when nothing else can happen
  // producer
  int item = 0, next_fill = 0;
  bool q_pending = false;
  int published = 0, read = 0;
  int q_issued = 0, q_landed = 0, q_done = 0, q_waited = 0;
  int landed[trx::AP_STAGES] = {};
  // O and the epilogue
  int o_done = 0, o_free = 0, o_waited = 0;
  std::vector<int> scores, products;  // 1000 * item + visit

  bool keyed(int i) const { return items[i].hi > items[i].lo; }

  bool publish() {
    if (item >= static_cast<int>(items.size()) || published > item) return false;
    if (item >= 2 && read < item - 1) return false;
    published = item + 1;
    q_pending = keyed(item);
    return true;
  }
  bool issue_q() {
    if (published <= item || !q_pending) return false;
    if (next_fill == first[item] && item > 0) return false;  // its first K tile goes ahead
    if (q_done < q_issued) return false;
    ++q_issued;
    q_pending = false;
    return true;
  }
  bool issue_fill() {
    if (published <= item || next_fill == first[item + 1]) return false;
    if (q_pending && (item == 0 || next_fill > first[item])) return false;
    if (next_fill >= trx::AP_STAGES && !fills[next_fill - trx::AP_STAGES].released) return false;
    fills[next_fill++].issued = true;
    return true;
  }
  bool next_item() {
    if (published <= item || q_pending || next_fill < first[item + 1]) return false;
    ++item;
    return publish();
  }
  bool land(bool lazy_too) {
    std::vector<int> flying;
    for (int f = 0; f < next_fill; ++f)
      if (!fills[f].landed && (lazy_too || f % trx::AP_STAGES != lazy)) flying.push_back(f);
    if (flying.empty()) return false;
    const int f = flying[rng() % flying.size()];
    fills[f].landed = true;
    ++landed[f % trx::AP_STAGES];
    return true;
  }
  bool land_q() {
    if (q_landed == q_issued) return false;
    ++q_landed;
    return true;
  }
  bool epilogue() {
    if (o_free == o_done) return false;
    ++o_free;
    return true;
  }
  bool step() {  // something around the warp happens
    for (int i = 0; i < 12; ++i) switch (rng() % 6) {
        case 0: if (issue_fill()) return true; break;
        case 1: if (issue_q()) return true; break;
        case 2: if (next_item() || publish()) return true; break;
        case 3: if (land(false)) return true; break;
        case 4: if (land_q()) return true; break;
        default: if (epilogue()) return true;
      }
    return issue_fill() || issue_q() || next_item() || publish() || land(false) || land_q() ||
           epilogue() || land(true);
  }
  void some_steps() {
    for (int i = rng() % 4; i > 0; --i) step();
  }
  bool fail(Wrong w) {
    if (wrong == NONE) wrong = w;
    return false;
  }
  // A wait for a phase of which one bit is compared; `phase` is the one that is meant.
  template <class Count>
  bool wait(Count count, int phase) {
    some_steps();
    while ((count() & 1) == (phase & 1))
      if (!step()) return fail(DEADLOCK);
    return count() == phase + 1 ? true : fail(LAPPED);
  }
  template <class Count>
  bool there(Count count, int phase) {
    some_steps();
    if ((count() & 1) == (phase & 1)) return false;
    if (count() != phase + 1) fail(LAPPED);
    return true;
  }
  bool wait_fill(int f) {
    return wait([&] { return landed[f % trx::AP_STAGES]; }, f / trx::AP_STAGES);
  }
  void use(int f, bool k) {
    if (!fills[f].landed || fills[f].k != k) fail(ORDER);
    const int later = f + trx::AP_STAGES;
    if (later < static_cast<int>(fills.size()) && fills[later].issued) fail(OVERWRITTEN);
  }
};

}  // namespace

extern "C" int issue_model(int count, const int* n, const int* lo, const int* hi, uint64_t seed) {
  World w;
  w.rng.seed(seed);
  w.lazy = static_cast<int>(w.rng() % trx::AP_STAGES);
  std::vector<int> visits;
  for (int i = 0; i < count; ++i) {
    w.items.push_back({n[i], lo[i], hi[i]});
    w.first.push_back(static_cast<int>(w.fills.size()));
    // K(0), K(1), V(0), K(2), V(1), .. V(n - 1)
    for (int v = 0; v < n[i]; ++v) {
      w.fills.push_back({i, v, true});
      if (v > 0) w.fills.push_back({i, v - 1, false});
    }
    if (n[i] > 0) w.fills.push_back({i, n[i] - 1, false});
    for (int v = lo[i]; v < hi[i]; ++v) visits.push_back(1000 * i + v);
  }
  w.first.push_back(static_cast<int>(w.fills.size()));
  w.publish();

  trx::PlainSteps steps{
      [&](trx::PlainCursor& c, int item, bool& ok) {
        if (item < count)
          while (w.published <= item)
            if (!w.step()) return ok = w.fail(DEADLOCK);
        if (item >= count) return false;
        c = {lo[item], hi[item], n[item], item, 0};
        w.read = item + 1;
        return true;
      },
      [&](int item) { w.some_steps(); return item >= count || w.published > item; },
      [&](int f) { return w.wait_fill(f); },
      [&](int f) { return w.there([&] { return w.landed[f % trx::AP_STAGES]; }, f / trx::AP_STAGES); },
      [&](int f) {
        if (w.fills[f].released) w.fail(RELEASED_TWICE);
        if (!w.fills[f].landed) w.fail(LAPPED);
        w.fills[f].released = true;
      },
      [&](unsigned parity) {
        if (parity != (w.q_waited & 1u)) return w.fail(ORDER);
        return w.wait([&] { return w.q_landed; }, w.q_waited++);
      },
      [&](unsigned) { return w.there([&] { return w.q_landed; }, w.q_waited); },
      [&](int f) {
        w.use(f, true);
        if (w.scores.size() != w.products.size()) w.fail(ORDER);  // its P is not used up yet
        w.scores.push_back(1000 * w.fills[f].item + w.fills[f].visit);
      },
      [&] { ++w.q_done; },
      [&](unsigned parity) {
        if (parity != (w.o_waited & 1u)) return w.fail(ORDER);
        return w.wait([&] { return w.o_free; }, w.o_waited++);
      },
      [&](int f, unsigned acc) {
        w.use(f, false);
        const int v = w.fills[f].visit, i = w.fills[f].item;
        if ((acc == 0) != (v == lo[i]) || w.scores.size() != w.products.size() + 1 ||
            (acc == 0 && w.o_free != w.o_done))
          w.fail(ORDER);
        w.products.push_back(1000 * i + v);
        w.some_steps();
        return w.wrong == NONE;
      },
      [&] { ++w.o_done; }};
  trx::plain_issue(steps);
  if (w.wrong == NONE) {
    if (w.scores != visits || w.products != visits) w.fail(UNFINISHED);
    for (const Fill& f : w.fills)
      if (!f.released) w.fail(UNFINISHED);
  }
  return w.wrong;
}
