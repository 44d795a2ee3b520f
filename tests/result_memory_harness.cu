// Host-side harness of the rule that sends a run's results through a kernel or
// through copies (memory_of_device in csrc/piv_internal.h), for the CPU tests.
#include "../openpiv-python-gpu_gb300/csrc/piv_internal.h"

extern "C" int memory_of_device(int type, int at_device, int device) {
  cudaPointerAttributes at = {};
  at.type = (cudaMemoryType)type;
  at.device = at_device;
  return piv::memory_of_device(at, device) ? 1 : 0;
}
