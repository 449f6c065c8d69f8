// The word in which bounded waits record that they gave up (sm100.cuh), one per device.  Static storage: it is there, and zero, before the
// first kernel that wants it, also where that is launched into a graph, whose pool (and whose every replay) an allocated word would belong to.
#include <cuda_runtime.h>

namespace sb {
__device__ unsigned int g_status_word;
}

// Address of the current device's word.
extern "C" int sb_status_word(void** out) { return cudaGetSymbolAddress(out, sb::g_status_word) == cudaSuccess ? 0 : -2; }
