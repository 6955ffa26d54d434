// Test driver: solve_batch's host passes (solver.cpp) with the GPU entry points as stubs, and the threads
// that they start, counted by a pthread_create of its own (tests/test_batch_threads.py). Prints that number and
// the scenarios' fingerprints.
#include <dlfcn.h>
#include <pthread.h>

#include <atomic>
#include <cstdio>
#include <stdexcept>
#include <vector>

#include "batch.hpp"
#include "solver.hpp"

static std::atomic<int> started{0};

extern "C" int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* arg) noexcept {
  using Create = int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
  static const Create real = reinterpret_cast<Create>(dlsym(RTLD_NEXT, "pthread_create"));
  ++started;
  return real(t, a, f, arg);
}

namespace b200 {
EngineResult run_engine_host(const HostModelView&, const EngineOptions&, HostOutputs&) {
  throw std::runtime_error("no engine here");
}
const char* status_name(Status) { return "?"; }
void require_device() {}
std::vector<BatchOutcome> run_batch_host(const HostModelView&, const std::vector<BatchScenarioView>& scenarios,
                                         const std::vector<int>&, const EngineOptions&,
                                         std::chrono::steady_clock::time_point) {
  return std::vector<BatchOutcome>(scenarios.size());
}
}  // namespace b200

int main() {
  using namespace b200;
  Model m;
  m.num_rows = 1, m.num_cols = 2;
  m.obj = {1.0, 2.0}, m.col_lower = {0.0, 0.0}, m.col_upper = {1.0, 1.0}, m.row_lower = {0.5}, m.row_upper = {2.0};
  m.col_start = {0, 1, 2}, m.row_index = {0, 0}, m.value = {1.0, 1.0};
  std::vector<Scenario> scenarios(40);
  for (std::size_t k = 1; k < scenarios.size(); ++k) scenarios[k].obj = {1.0, static_cast<double>(k)};
  const std::vector<Solution> got = solve_batch(m, scenarios, Options{});
  std::printf("%d\n", started.load());
  for (const Solution& s : got) std::printf("%s\n", s.model_fingerprint.c_str());
}
