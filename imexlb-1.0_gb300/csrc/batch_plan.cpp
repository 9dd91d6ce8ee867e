// Parts and chains of a batch of cases (batch.h).
#include <algorithm>
#include <cstdint>
#include <vector>

#include "batch.h"

namespace imx {

// Largest first into the first part with room, so that there are few parts: a
// part is one launch an iteration, and cases of one size or many small ones
// wait for launches more than for anything else. All that fits is therefore
// one part, even if that leaves a chain idle (8 lattices of 48x24 to 99x49 in
// FP32, 200 iterations: 0.78 ms, on two chains 1.5; 300 of them in 3 parts of up to
// 128: 3.0, in 19 of up to 16: 9.0), and as many parts as chains
// are made alike in size (64 lattices of 96x64, 63 + 1 and 32 + 32: 1.65 and 1.35).
BatchPlan plan_batch(const std::vector<int64_t>& bytes, int64_t room, int cap, int chains) {
  struct Part {
    std::vector<int> cases;
    int64_t used = 0;
  };
  std::vector<int> order(bytes.size());
  for (size_t i = 0; i < order.size(); ++i) order[i] = (int)i;
  std::stable_sort(order.begin(), order.end(),
                   [&](int x, int y) { return bytes[(size_t)x] > bytes[(size_t)y]; });
  std::vector<Part> parts;
  auto put = [&](Part& p, int i) {
    p.cases.push_back(i);
    p.used += bytes[(size_t)i];
  };
  auto full = [&](const Part& p) { return p.cases.size() == (size_t)cap; };
  size_t open = 0;  // the parts before it have all their cases
  for (int i : order) {
    while (open < parts.size() && full(parts[open])) ++open;
    size_t k = open;
    while (k < parts.size() && (full(parts[k]) || parts[k].used + bytes[(size_t)i] > room)) ++k;
    if (k == parts.size()) parts.emplace_back();
    put(parts[k], i);
  }
  if (parts.size() == (size_t)chains) {
    for (Part& p : parts) p = Part{};
    for (int i : order) {
      Part* to = nullptr;  // the smallest so far
      for (Part& p : parts)
        if (!full(p) && (!to || p.used < to->used)) to = &p;
      put(*to, i);
    }
  }
  // to the chain with the least to do, largest part first
  std::stable_sort(parts.begin(), parts.end(), [](const Part& x, const Part& y) { return x.used > y.used; });
  BatchPlan plan((size_t)chains);
  std::vector<int64_t> load((size_t)chains, 0);
  for (Part& p : parts) {
    const size_t to = (size_t)(std::min_element(load.begin(), load.end()) - load.begin());
    load[to] += p.used;
    plan[to].push_back(std::move(p.cases));
  }
  return plan;
}

}  // namespace imx
