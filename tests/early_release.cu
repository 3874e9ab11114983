// A kernel that lets the next one of its stream in at once and then goes on for a given time, for
// tests/test_wait_runs_out.py. It waits for the clock alone, and for at most 1 << 20 looks at it.
#include <cuda_runtime.h>

__global__ void early_release(unsigned long long ns) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  unsigned long long start, now;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(start));
  for (int i = 0; i < 1 << 20; ++i) {
    __nanosleep(1000);
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
    if (now - start >= ns) break;
  }
}

extern "C" int launch_early_release(unsigned long long ns, void* stream) {
  early_release<<<148, 32, 0, static_cast<cudaStream_t>(stream)>>>(ns);
  return static_cast<int>(cudaGetLastError());
}
