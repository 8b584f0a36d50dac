// Self-test of the bounded waits: a wait that nothing will ever satisfy has to give up, record its status
// code and let the kernel finish, so that the context stays usable.  The kernels of this library wait on
// mbarriers that asynchronous copies complete (async.cuh); here one warp arms such a barrier for bytes that
// no copy delivers and waits on it with a short poll limit, in each of the ways that the kernels wait.  Nothing is
// faulted, trapped or left spinning.
// A second self-test stands for the opposite: a kernel that is merely slow is no reason to give up.
// The reference has no counterpart (its only error path is exit(1), csrc/include/common.cuh:44-51).
#include <cuda_runtime.h>

#include "../../include/matgptq_b200.h"
#include "async.cuh"
#include "kernels.h"

namespace mg {

// The warp waits with mbar_wait_bounded, then with mbar_wait_chain, where the odd lanes ask for a barrier whose phase is
// complete: a warp has one answer there, so these give up as well.  *gave_up is set when every lane gave up both times.
__global__ void __launch_bounds__(32, 1) wait_timeout_probe_kernel(int code, unsigned polls, unsigned chain_polls, int *gave_up) {
  __shared__ __align__(8) unsigned long long bar_storage[2];
  const uint32_t open = smem_u32(&bar_storage[0]), complete = smem_u32(&bar_storage[1]);
  if (threadIdx.x == 0) {
    mbar_init(open, 1);
    mbar_init(complete, 1);
    mbar_init_fence();
  }
  __syncwarp();
  if (threadIdx.x == 0) {
    mbar_arrive_expect_tx(open, 64);  // 64 bytes are expected; no copy is issued
    mbar_arrive(complete);
  }
  __syncwarp();
  const bool bounded = mbar_wait_bounded(open, 0, polls);
  __syncwarp();
  const bool chain = mbar_wait_chain((threadIdx.x & 1) ? complete : open, 0, chain_polls);
  __syncwarp();
  if (__all_sync(0xffffffffu, !bounded && !chain)) {
    report_status(code);
    if (threadIdx.x == 0 && gave_up) *gave_up = 1;
  }
}

int selftest_wait_timeout_launch(int code, unsigned polls, unsigned chain_polls, int *gave_up, cudaStream_t stream) {
  wait_timeout_probe_kernel<<<1, 32, 0, stream>>>(code, polls, chain_polls, gave_up);
  return cudaGetLastError() == cudaSuccess ? MG_OK : MG_ERR_CUDA;
}

// The kernel before a product in a launch chain that takes its time: lets the next kernel start at once, rests for `rest_ns`
// nanoseconds and only then writes what that kernel reads.
__global__ void __launch_bounds__(1024, 1) late_writer_kernel(const uint16_t *__restrict__ src, uint16_t *__restrict__ dst, long long n,
                                                            unsigned long long rest_ns) {
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  unsigned long long start, now;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(start));
  for (unsigned it = 0; it < (1u << 24); ++it) {  // at least a fifth of a microsecond each
    __nanosleep(1000);
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
    if (now - start >= rest_ns) break;
  }
  for (long long i = threadIdx.x; i < n; i += blockDim.x) dst[i] = src[i];
}

MG_DEFINE_STATUS_ACCESSOR(selftest_device_status)

}  // namespace mg

extern "C" int matgptq_b200_selftest_wait_timeout(int status_code, int *gave_up_flag, void *stream) {
  if (status_code != mg::kStatusWeightCopyTimeout && status_code != mg::kStatusActivationCopyTimeout &&
      status_code != mg::kStatusMmaTimeout)
    return MG_ERR_BAD_ARG;
  // 4096 polls of about 40 ns each and the hardware's own try_wait time-out, then 256 polls of at most 20 us: well under a second
  return mg::selftest_wait_timeout_launch(status_code, 4096u, 256u, gave_up_flag, static_cast<cudaStream_t>(stream));
}

extern "C" int matgptq_b200_selftest_late_writer(const void *src, void *dst, int64_t n, int rest_ms, void *stream) {
  if (!src || !dst || n <= 0 || rest_ms < 0 || rest_ms > 4000) return MG_ERR_BAD_ARG;
  mg::late_writer_kernel<<<1, 1024, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const uint16_t *>(src), static_cast<uint16_t *>(dst), n, static_cast<unsigned long long>(rest_ms) * 1000000ull);
  return cudaGetLastError() == cudaSuccess ? MG_OK : MG_ERR_CUDA;
}
