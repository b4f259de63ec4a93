/* A launch that lets the one behind it start at once and moves the cursor only some microseconds
 * later: what the single-token append reads while its dependency is open is then out of date. */
#include <cuda_runtime.h>

static __global__ void late_cursor_kernel(int *cursor, int value, long long clocks) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const long long t0 = clock64();
  while (clock64() - t0 < clocks) {
  }
  *cursor = value;
}

extern "C" int late_cursor(void *cursor, int value, long long clocks, void *stream) {
  late_cursor_kernel<<<1, 1, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<int *>(cursor), value, clocks);
  return static_cast<int>(cudaGetLastError());
}
