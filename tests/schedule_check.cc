// Test harness of schedule_units (csrc/host_math.h): the schedule of the given runs, and the longest block's cost that
// giving each unit, longest first, to the least loaded block reaches.
#include <algorithm>
#include <queue>

#include "host_math.h"

using namespace leapgb;

extern "C" long long schedule_check(int nruns, const long long* cost, const int* shape, int grid, int* out, long long capacity) {
  std::vector<UnitRun> runs;
  for (int i = 0; i < nruns; ++i)
    runs.push_back(UnitRun{cost[i], shape[4 * i], shape[4 * i + 1], shape[4 * i + 2], shape[4 * i + 3]});
  std::vector<int32_t> order;
  schedule_units(runs, grid, order);
  if (static_cast<long long>(order.size()) > capacity) return -1;
  std::copy(order.begin(), order.end(), out);
  return static_cast<long long>(order.size());
}

extern "C" long long greedy_makespan(int nruns, const long long* cost, const int* shape, int grid) {
  std::vector<long long> units;
  for (int i = 0; i < nruns; ++i) units.insert(units.end(), shape[4 * i + 1], cost[i]);
  std::sort(units.rbegin(), units.rend());
  std::priority_queue<long long, std::vector<long long>, std::greater<>> load;
  for (int b = 0; b < grid; ++b) load.push(0);
  long long most = 0;
  for (long long c : units) {
    const long long l = load.top() + c;
    load.pop();
    load.push(l);
    most = std::max(most, l);
  }
  return most;
}
