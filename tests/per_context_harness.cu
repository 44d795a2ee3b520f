// Host-side harness of the objects kept per context (csrc/piv_per_context.h) with
// a fake runtime, for the CPU tests.
#include "../openpiv-python-gpu_gb300/csrc/piv_per_context.h"

namespace {
int g_device = 0, g_resets[64] = {0}, g_pools = 0, g_trimmed[256] = {0};
bool g_fail = false;
struct Fake {
  using Value = int;  // 1, 2, ... in the order of creation
  struct OnDevice {
    int before = g_device;
    explicit OnDevice(int dev) { g_device = dev; }
    ~OnDevice() { g_device = before; }
  };
  static unsigned long long context() { return 1 + g_device + 64ull * g_resets[g_device]; }
  static bool create(Value* pool) { return g_fail ? false : (*pool = ++g_pools, true); }
};
piv::PerContext<Fake> g_set;
}  // namespace

extern "C" {
void fake_device(int dev) { g_device = dev; }
void fake_reset(int dev) { ++g_resets[dev]; }
void fake_fail(int fail) { g_fail = fail != 0; }
int fake_trimmed(int pool) { return g_trimmed[pool]; }
int pool_get() { return g_set.get(); }
void pool_trim(int dev) {
  g_set.with(dev, [](int pool) { ++g_trimmed[pool]; });
}
}
