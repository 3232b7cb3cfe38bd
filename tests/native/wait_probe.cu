// Kernels for tests/test_gpu_waits.py: the bounded waits of common.cuh made to run out, and a predecessor that lets its
// dependents start early and then stays busy.  Every loop here ends by the SM clock.
#include "../../sglang_b200/csrc/common.cuh"

namespace {

// One warp waits for a barrier that nothing arrives at.  out[0]: what the wait returned, out[1]: cycles it took.
__global__ void wait_out_kernel(int form, int* slot, long long* out) {
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) {
    b200::mbar_init(&bar, 1);
    b200::fence_mbar_init();
  }
  __syncthreads();
  const long long t0 = clock64();
  const bool ok = form == 0 ? b200::mbar_wait(&bar, 0, slot, 77) : b200::sa::wait(b200::smem_u32(&bar), 0, slot, 77);
  if (threadIdx.x == 0) {
    out[0] = ok;
    out[1] = clock64() - t0;
  }
}

__global__ void early_trigger_kernel(long long cycles) {
  b200::pdl_trigger();
  const long long t0 = clock64();
  while (clock64() - t0 < cycles) __nanosleep(1000);
}

}  // namespace

extern "C" int probe_wait_out(int form, void* slot, void* out, void* stream) {
  wait_out_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(form, static_cast<int*>(slot), static_cast<long long*>(out));
  return static_cast<int>(cudaGetLastError());
}

extern "C" int probe_early_trigger(long long cycles, void* stream) {
  early_trigger_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(cycles);
  return static_cast<int>(cudaGetLastError());
}
