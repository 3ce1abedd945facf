// How many cores a rank has to itself, for idle policies that spin.
#ifndef TCPXB_CPU_BUDGET_H_
#define TCPXB_CPU_BUDGET_H_

#include <string>

namespace tcpxb {

// Whole cores' worth of time that the CPU quotas of this process's control groups allow: the least of the group and
// its ancestors, INT_MAX without a quota.  `membership` is the content of /proc/self/cgroup, `root` the mount point
// (/sys/fs/cgroup); both cgroup versions are understood, and groups that cannot be seen are passed over.
int cgroupCpuLimit(const std::string& membership, const std::string& root);

// Cores this process may run on (affinity mask), no more than its CPU quota.  At least 1.
int usableCores();

// Ranks that share those cores: the most that anyone claims, the launcher's LOCAL_WORLD_SIZE among them.
int localRanks(int gpus_per_node, int seen);

// Whether a driving thread that spins takes nothing from `helper_threads` of its own rank.
bool spareCores(int cores, int local_ranks, int helper_threads);

}  // namespace tcpxb

#endif  // TCPXB_CPU_BUDGET_H_
