// checked_launch (csrc/runtime.h) against fakes of the runtime calls around it.
// Prints, per scenario, the launches made, the status returned and the error
// left unread.  stdin is not read; no GPU takes part.
#include <cstdio>
#include <vector>

#include "runtime.h"

static int g_launches = 0, g_raised = 0;
static cudaError_t g_last = cudaSuccess;
static std::vector<cudaError_t> g_answers;  // of the launches to come (then success)

extern "C" {
cudaError_t cudaGetLastError(void) {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
}

namespace tridi {
static DeviceInfo g_dev;
const DeviceInfo* current_device() { return &g_dev; }
static bool g_allowed = true;  // the kernel's limit is raised
bool smem_allowed(const void*, size_t) { return g_allowed; }
cudaError_t raise_smem_limit(const void*, const DeviceInfo&) {
  ++g_raised;
  g_allowed = true;
  return cudaSuccess;
}
}  // namespace tridi

static void scenario(bool allowed, cudaError_t unread, std::vector<cudaError_t> answers, size_t smem) {
  tridi::g_allowed = allowed;
  g_launches = g_raised = 0;
  g_last = unread;
  g_answers = answers;
  const auto launch = [] {
    ++g_launches;
    if (g_answers.empty()) return;
    if (g_answers.front() != cudaSuccess) g_last = g_answers.front();
    g_answers.erase(g_answers.begin());
  };
  const cudaError_t e = tridi::checked_launch(launch, nullptr, smem);
  std::printf("%d %d %d %d\n", g_launches, g_raised, (int)e, (int)g_last);
}

int main() {
  const cudaError_t bad = cudaErrorInvalidValue, other = cudaErrorMemoryAllocation;
  scenario(true, cudaSuccess, {}, 100000);
  scenario(true, bad, {}, 100000);  // the caller's unread error
  scenario(true, other, {}, 100000);
  scenario(false, cudaSuccess, {bad}, 100000);       // the limit was dropped
  scenario(false, other, {bad}, 100000);
  scenario(false, cudaSuccess, {bad, bad}, 100000);  // and does not help
  scenario(true, cudaSuccess, {bad}, 100000);        // not the limit
  scenario(true, cudaSuccess, {bad}, 1000);
  scenario(true, cudaSuccess, {other}, 100000);
}
