#include "tcpxb/cpu_budget.h"

#include <limits.h>
#include <sched.h>
#include <stdio.h>
#include <stdlib.h>

#include <algorithm>
#include <sstream>
#include <vector>

namespace tcpxb {

namespace {

// First up to two numbers of a file; false when it cannot be read or does not start with a number ("max").
bool readNumbers(const std::string& path, long long* a, long long* b) {
  FILE* f = fopen(path.c_str(), "r");
  if (f == nullptr) return false;
  *b = 0;
  const int n = fscanf(f, "%lld %lld", a, b);
  fclose(f);
  return n >= 1;
}

int cores(long long quota_us, long long period_us) {
  if (quota_us <= 0 || period_us <= 0) return INT_MAX;
  return (int)std::min<long long>(std::max<long long>(quota_us / period_us, 1), INT_MAX);
}

bool listed(const std::string& list, const char* name) {
  std::istringstream in(list);
  for (std::string s; std::getline(in, s, ',');)
    if (s == name) return true;
  return false;
}

}  // namespace

int cgroupCpuLimit(const std::string& membership, const std::string& root) {
  int limit = INT_MAX;
  std::istringstream lines(membership);
  for (std::string line; std::getline(lines, line);) {  // hierarchy:controllers:path
    const size_t c1 = line.find(':'), c2 = c1 == std::string::npos ? c1 : line.find(':', c1 + 1);
    if (c2 == std::string::npos) continue;
    const std::string controllers = line.substr(c1 + 1, c2 - c1 - 1);
    const bool v2 = controllers.empty();
    if (!v2 && !listed(controllers, "cpu")) continue;
    std::vector<std::string> mounts{root};
    if (!v2) mounts = {root + "/cpu", root + "/" + controllers};
    std::string path = line.substr(c2 + 1);
    while (!path.empty() && path.back() == '/') path.pop_back();
    for (;;) {  // the group itself, then every group above it
      for (const std::string& m : mounts) {
        long long quota = 0, period = 0, none = 0;
        if (v2) {
          if (readNumbers(m + path + "/cpu.max", &quota, &period)) limit = std::min(limit, cores(quota, period));
        } else if (readNumbers(m + path + "/cpu.cfs_quota_us", &quota, &none) && readNumbers(m + path + "/cpu.cfs_period_us", &period, &none)) {
          limit = std::min(limit, cores(quota, period));
        }
      }
      if (path.empty()) break;
      path.resize(path.rfind('/') == std::string::npos ? 0 : path.rfind('/'));
    }
  }
  return limit;
}

int usableCores() {
  cpu_set_t set;
  CPU_ZERO(&set);
  if (sched_getaffinity(0, sizeof set, &set) != 0) return 1;
  std::string membership;
  if (FILE* f = fopen("/proc/self/cgroup", "r")) {
    char buf[4096];
    for (size_t n; (n = fread(buf, 1, sizeof buf, f)) > 0;) membership.append(buf, n);
    fclose(f);
  }
  return std::max(1, std::min(CPU_COUNT(&set), cgroupCpuLimit(membership, "/sys/fs/cgroup")));
}

int localRanks(int gpus_per_node, int seen) {
  const char* v = getenv("LOCAL_WORLD_SIZE");
  return std::max({1, v != nullptr ? atoi(v) : 1, gpus_per_node, seen});
}

// The line at 16 cores was measured (kSpareCoreSpinUs in the engine) with 32 helper threads, which nap when they have
// nothing to do; with more of them it moves up in proportion.
bool spareCores(int cores, int local_ranks, int helper_threads) {
  const int mine = cores / std::max(1, local_ranks);
  return mine >= 16 && 2 * mine >= helper_threads;
}

}  // namespace tcpxb
