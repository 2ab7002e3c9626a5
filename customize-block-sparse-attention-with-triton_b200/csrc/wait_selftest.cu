// Self-test of the bounded waits the attention kernels are built on: a wait that nothing will ever
// satisfy has to run out, report through the status word and leave by the ordinary end of the
// kernel, with the context usable afterwards.  One CTA, two warps; no tensor memory, no TMA.
#include "host_common.h"
#include "sm100_ptx.cuh"

namespace bsa {

__global__ void __launch_bounds__(64, 1) wait_selftest_kernel(int32_t* status, int32_t* report) {
  __shared__ uint64_t bar;
  __shared__ int abort_flag;
  const int warp = uniform_warp_index();
  const int lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&bar), 1);  // one arrival expected; none is ever made
    abort_flag = 0;
    mbar_fence_init();
  }
  __syncthreads();
  volatile int* flag = &abort_flag;
  const uint64_t t0 = global_timer_ns();
  if (warp == 0) {
    // runs out after the wait limit, then raises the CTA's flag like a role of a kernel does
    const bool ok = mbar_wait_warp(smem_u32(&bar), 0);
    if (!ok && lane == 0) {
      abort_flag = 1;
      report_status(status, 99);
    }
    if (lane == 0) report[0] = ok ? 1 : 0;
  } else {
    // the wait for an item, begun a second later, so that it leaves because the other warp raised the flag and not by its
    // own limit
#pragma unroll 1
    for (int i = 0; i < 2000 && global_timer_ns() - t0 < 1000000000ull; ++i) __nanosleep(1000000u);
    const bool ok = mbar_wait_warp_item(smem_u32(&bar), 0, flag);
    if (lane == 0) report[1] = ok ? 1 : 0;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    report[2] = 1;  // both warps reached the end of the kernel
    report[3] = static_cast<int32_t>((global_timer_ns() - t0) / 1000000ull);  // milliseconds waited
  }
}

// What two warps make of a wait when half of their lanes look at a barrier that is complete and the others at
// one that never will be: the second warp waits as for an item, and the first one raises the flag
// after 20 ms; the third one makes all of its tries.
__global__ void __launch_bounds__(96, 1) give_up_selftest_kernel(int32_t* report) {
  __shared__ uint64_t bar[2];
  __shared__ int abort_flag;
  const int warp = uniform_warp_index();
  const int lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&bar[0]), 1);
    mbar_init(smem_u32(&bar[1]), 1);
    abort_flag = 0;
    mbar_fence_init();
    mbar_arrive(smem_u32(&bar[0]));
  }
  __syncthreads();
  volatile int* flag = &abort_flag;
  const uint64_t t0 = global_timer_ns();
  if (warp == 0) {
#pragma unroll 1
    for (int i = 0; i < 20; ++i) __nanosleep(1000000u);  // (at most a millisecond each)
    if (lane == 0) *flag = 1;
  } else {
    const bool ok = warp == 1 ? mbar_wait_warp_item(smem_u32(&bar[lane & 1]), 0, flag)
                              : mbar_wait_warp(smem_u32(&bar[lane & 1]), 0);
    const unsigned went_on = __ballot_sync(0xffffffffu, ok);
    if (lane == 0) {
      report[2 * warp - 2] = __popc(went_on);
      report[2 * warp - 1] = static_cast<int32_t>((global_timer_ns() - t0) / 1000000ull);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) report[4] = 1;
}

// How long the forms of a wait last on barriers that nothing ever completes, one warp each: on one barrier, on two at
// once, on three at once, for an item, and for an item when the sixth warp raises the flag after 100 ms.
__global__ void __launch_bounds__(192, 1) wait_limits_selftest_kernel(int32_t* report) {
  __shared__ uint64_t bar[3];
  __shared__ int flags[2];
  const int warp = uniform_warp_index();
  const int lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < 3; ++i) mbar_init(smem_u32(&bar[i]), 1);
    flags[0] = flags[1] = 0;
    mbar_fence_init();
  }
  __syncthreads();
  volatile int* flag = flags;
  const uint32_t b0 = smem_u32(&bar[0]), b1 = smem_u32(&bar[1]), b2 = smem_u32(&bar[2]);
  const uint64_t t0 = global_timer_ns();
  bool ok = false;
  if (warp == 0) {
    ok = mbar_wait_warp(b0, 0);
  } else if (warp == 1) {
    ok = mbar_wait_warp2(b0, 0, b1, 0);
  } else if (warp == 2) {
    ok = mbar_wait_warp3(b0, 0, b1, 0, b2, 0);
  } else if (warp < 5) {
    ok = mbar_wait_warp_item(b0, 0, flag + (warp - 3));
  } else {
#pragma unroll 1
    for (int i = 0; i < 100; ++i) __nanosleep(1000000u);  // (at most a millisecond each)
    if (lane == 0) flag[1] = 1;
  }
  const unsigned went_on = __ballot_sync(0xffffffffu, ok);
  if (lane == 0) {
    report[2 * warp] = __popc(went_on);
    report[2 * warp + 1] = static_cast<int32_t>((global_timer_ns() - t0) / 1000000ull);
  }
}

// The loop of a role of four warps that wait for their items one by one, as the attention kernels' write-out does:
// items 0, 2, 3 and 6 have work, 1, 4 and 5 have none, 7 is the end, and the wait of warp w for item run_out[w] runs out
// (not at all if there is no such item).  report[w]: after how many items with work the warp went on, 100 more once it has left.
__global__ void __launch_bounds__(128, 1) role_vote_selftest_kernel(int4 run_out, int32_t* report) {
  const int warp = uniform_warp_index();
  const int mine = warp == 0 ? run_out.x : warp == 1 ? run_out.y : warp == 2 ? run_out.z : run_out.w;
  int done = 0;
#pragma unroll 1
  for (int i = 0;; ++i) {
    const bool ok = i != mine;
    if (ok && i == 7) {
      named_barrier_sync(2, 128);
      role_leaves(2, 128, false);
      break;
    }
    if (ok && (i == 1 || i == 4 || i == 5)) continue;
    named_barrier_sync(2, 128);
    if (role_leaves(2, 128, !ok)) break;
    ++done;
  }
  if ((threadIdx.x & 31) == 0) report[warp] = done + 100;
}

// Lets its dependents in at once and ends after so many milliseconds.
__global__ void __launch_bounds__(32, 1) early_selftest_kernel(int milliseconds) {
  grid_dependents_launch();
  const uint64_t t0 = global_timer_ns();
#pragma unroll 1
  for (int i = 0; i < 100 * milliseconds && global_timer_ns() - t0 < 1000000ull * milliseconds; ++i)
    __nanosleep(100000u);
}

}  // namespace bsa

extern "C" int bsa_selftest_early_kernel(int milliseconds, void* stream) {
  if (milliseconds < 0 || milliseconds > 10000) return BSA_ERR_BAD_SHAPE;
  int rc;
  if ((rc = bsa::check_device_sm100()) != BSA_OK) return rc;
  bsa::early_selftest_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(milliseconds);
  return cudaGetLastError() == cudaSuccess ? BSA_OK : BSA_ERR_CUDA;
}

extern "C" int bsa_selftest_wait_limits(int32_t* report, void* stream) {
  if (!report) return BSA_ERR_BAD_POINTER;
  int rc;
  if ((rc = bsa::check_device_sm100()) != BSA_OK) return rc;
  bsa::wait_limits_selftest_kernel<<<1, 192, 0, static_cast<cudaStream_t>(stream)>>>(report);
  return cudaGetLastError() == cudaSuccess ? BSA_OK : BSA_ERR_CUDA;
}

extern "C" int bsa_selftest_launch_registers(int more) {
  int rc;
  if ((rc = bsa::check_device_sm100()) != BSA_OK) return rc;
  const void* kernel = reinterpret_cast<const void*>(bsa::role_vote_selftest_kernel);
  cudaFuncAttributes attr;
  if (cudaFuncGetAttributes(&attr, kernel) != cudaSuccess) return BSA_ERR_CUDA;
  return bsa::check_launch_registers(kernel, attr.numRegs + more);
}

extern "C" int bsa_selftest_role_vote(int item0, int item1, int item2, int item3, int32_t* report, void* stream) {
  if (!report) return BSA_ERR_BAD_POINTER;
  int rc;
  if ((rc = bsa::check_device_sm100()) != BSA_OK) return rc;
  bsa::role_vote_selftest_kernel<<<1, 128, 0, static_cast<cudaStream_t>(stream)>>>(make_int4(item0, item1, item2, item3),
                                                                                   report);
  return cudaGetLastError() == cudaSuccess ? BSA_OK : BSA_ERR_CUDA;
}

extern "C" int bsa_selftest_give_up(int32_t* report, void* stream) {
  if (!report) return BSA_ERR_BAD_POINTER;
  int rc;
  if ((rc = bsa::check_device_sm100()) != BSA_OK) return rc;
  bsa::give_up_selftest_kernel<<<1, 96, 0, static_cast<cudaStream_t>(stream)>>>(report);
  return cudaGetLastError() == cudaSuccess ? BSA_OK : BSA_ERR_CUDA;
}

extern "C" int bsa_selftest_bounded_wait(int32_t* status, int32_t* report, void* stream) {
  if (!report) return BSA_ERR_BAD_POINTER;
  int rc;
  if ((rc = bsa::check_device_sm100()) != BSA_OK) return rc;
  bsa::wait_selftest_kernel<<<1, 64, 0, static_cast<cudaStream_t>(stream)>>>(status, report);
  return cudaGetLastError() == cudaSuccess ? BSA_OK : BSA_ERR_CUDA;
}
