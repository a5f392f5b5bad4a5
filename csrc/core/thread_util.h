// Thread placement helpers (reference: rust/thread-lib/src/lib.rs:4-16).
#pragma once

#include <string>
#include <vector>

namespace pplx {

// Pins the calling thread to one logical CPU. Throws pplx::Error on failure.
void pin_cpu(int cpu);
// CPUs the calling thread may run on.
std::vector<int> current_affinity();
void set_thread_name(const std::string& name);

// A CPU for one busy-polling thread of this process: of `candidates` the one with the fewest
// leases, the first of them on a tie. Two such threads on one core take turns by the scheduler's
// time slice, milliseconds each, whatever they are waiting for. Given back by the destructor.
class CpuLease {
 public:
  CpuLease() = default;
  explicit CpuLease(const std::vector<int>& candidates);
  ~CpuLease();
  CpuLease(CpuLease&& o) noexcept : cpu_(o.cpu_) { o.cpu_ = -1; }
  CpuLease& operator=(CpuLease&& o) noexcept;
  int cpu() const { return cpu_; }   // -1: no candidates

 private:
  int cpu_ = -1;
};

}  // namespace pplx
