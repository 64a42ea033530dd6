#include "launch.hpp"

#include <atomic>
#include <cstdlib>

#include "log.hpp"

namespace mccl {

namespace {
// Launches per kernel-name literal, counted without a lock: a launch costs the host two or three microseconds, and a mutex,
// a string and a map lookup were a tenth of that.  Every call site passes the same literal every time, so the pointer is
// the key; equal names from different sites are added up when somebody asks.
constexpr int kSlots = 256;
struct Slot {
  std::atomic<const char*> name{nullptr};
  std::atomic<uint64_t> count{0};
};
Slot g_slots[kSlots];
std::atomic<uint64_t> g_total{0};

void count(const char* kernel) {
  size_t at = (reinterpret_cast<uintptr_t>(kernel) >> 3) % kSlots;
  for (int i = 0; i < kSlots; ++i, at = (at + 1) % kSlots) {
    const char* have = g_slots[at].name.load(std::memory_order_acquire);
    if (have == nullptr && g_slots[at].name.compare_exchange_strong(have, kernel, std::memory_order_acq_rel)) have = kernel;
    if (have == kernel) {
      g_slots[at].count.fetch_add(1, std::memory_order_relaxed);
      return;
    }
  }
}
thread_local cudaError_t t_first_error = cudaSuccess;

// "(gemm_persistent_kernel<BN, STAGES, kAMn, kBMn>)" -> "gemm_persistent_kernel"
std::string short_name(const char* kernel) {
  std::string s(kernel);
  size_t b = 0;
  while (b < s.size() && (s[b] == '(' || s[b] == ' ')) ++b;
  size_t e = b;
  while (e < s.size() && s[e] != '<' && s[e] != ')' && s[e] != ' ') ++e;
  return s.substr(b, e - b);
}
}  // namespace

cudaError_t launch_record(const char* kernel, const char* file, int line, dim3 grid, dim3 block, size_t smem, cudaStream_t stream) {
  const cudaError_t rc = cudaGetLastError();
  g_total.fetch_add(1, std::memory_order_relaxed);
  count(kernel);
  if (rc != cudaSuccess) {
    if (t_first_error == cudaSuccess) t_first_error = rc;
    MCCL_ERROR("launch of " << kernel << " at " << file << ":" << line << " failed: " << cudaGetErrorString(rc) << " (grid " << grid.x
                            << "x" << grid.y << "x" << grid.z << ", block " << block.x << ", smem " << smem << ")");
  } else if (log_level() <= LogLevel::TRACE) {
    const char* base = file;
    for (const char* p = file; *p; ++p)
      if (*p == '/') base = p + 1;
    MCCL_TRACE("launch " << short_name(kernel) << " @" << base << ":" << line << " grid " << grid.x << "x" << grid.y << " block "
                         << block.x << " smem " << smem << " stream " << static_cast<const void*>(stream));
  }
  return rc;
}

bool pdl_enabled() {
  static const bool on = [] {
    // MCCL_PDL=0 switches it off.  Measured with the trigger behind the wait (see launch.hpp): training step of the
    // 2-layer model 159 -> 139 us, of the 70M model on 1600 tokens 2.57 -> 2.39 ms, on 4096 tokens 3.54 -> 3.47 ms; 37-token
    // scoring 880 -> 616 us.
    const char* v = std::getenv("MCCL_PDL");
    return !(v && v[0] == '0');
  }();
  return on;
}

cudaError_t launch_status() {
  const cudaError_t rc = t_first_error;
  t_first_error = cudaSuccess;
  return rc;
}

std::map<std::string, uint64_t> launch_counts() {
  std::map<std::string, uint64_t> out;
  for (const Slot& slot : g_slots) {
    const char* name = slot.name.load(std::memory_order_acquire);
    const uint64_t n = slot.count.load(std::memory_order_relaxed);
    if (name && n) out[short_name(name)] += n;
  }
  return out;
}
void launch_counts_reset() {
  for (Slot& slot : g_slots) slot.count.store(0);
  g_total.store(0);
}
uint64_t launch_total() { return g_total.load(); }

}  // namespace mccl
