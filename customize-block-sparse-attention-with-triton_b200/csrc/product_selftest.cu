// Self-test of the product that P V, dV, dK and dQ are made of: A in tensor memory, M = 64 in the "weight stationary"
// form, two tiles beside one another in B (umma_ws_ts).  Ordinary use of the form has the same 64 rows of A in both lane
// halves; the attention kernels rest on each half reading its own.  One CTA of four warps.
#include "host_common.h"
#include "sm100_ptx.cuh"

namespace bsa {

constexpr uint32_t kProductCols = 128;  // TMEM: the result in columns [0, 64), A as 16-bit pairs in [64, 96)

// a [128][64], b [2][64][64] 16-bit, out [128][64]: out[r] = a[r] b[r / 64].
template <bool kBf16>
__global__ void __launch_bounds__(128, 1)
half_products_selftest_kernel(const uint32_t* a, const uint4* b, float* out, int32_t* status) {
  __shared__ __align__(1024) uint8_t tiles[2][64 * 128];
  __shared__ uint64_t done;
  __shared__ uint32_t tmem_base;
  const int warp = uniform_warp_index();
  const int lane = threadIdx.x & 31;
  const int row = threadIdx.x;  // of A and of the result: TMEM lane
  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&done), 1);
    mbar_fence_init();
  }
  if (warp == 0) {
    tmem_alloc(smem_u32(&tmem_base), kProductCols);
    tmem_relinquish();
  }
  // B as TMA would leave it: rows of 128 bytes, 16-byte pieces exchanged by the row's place in its group of eight
#pragma unroll 1
  for (int i = threadIdx.x; i < 2 * 64 * 8; i += 128) {
    const int r = i >> 3;  // of both tiles
    *reinterpret_cast<uint4*>(&tiles[r >> 6][(r & 63) * 128 + (((i & 7) ^ (r & 7)) << 4)]) = b[i];
  }
  async_proxy_fence();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base;
  const uint32_t lanes = tmem + (static_cast<uint32_t>(warp * 32) << 16);
  {
    uint32_t mine[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) mine[j] = a[row * 32 + j];
    tmem_st_32x32b_x32(lanes + 64, mine);
    tc_wait_st();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) {
    constexpr uint32_t idesc = umma_idesc(kBf16, 0, 1, 64, 128);
    const uint64_t desc = smem_desc_sw128(smem_u32(tiles[0]), 8192, 1024);
    if (elect_one()) {
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) umma_ws_ts(tmem, tmem + 64 + 8 * kk, desc + 128 * kk, idesc, kk > 0);
      tc_commit(smem_u32(&done));
    }
    __syncwarp();
  }
  const bool ok = mbar_wait_warp(smem_u32(&done), 0);
  tc_fence_after();
  if (ok) {
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
      uint32_t sums[32];
      tmem_ld_32x32b_x32(lanes + 32 * half, sums);
      tc_wait_ld();
#pragma unroll
      for (int j = 0; j < 32; ++j) out[row * 64 + 32 * half + j] = __uint_as_float(sums[j]);
    }
  } else if (lane == 0) {
    report_status(status, 98);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, kProductCols);
  }
}

}  // namespace bsa

extern "C" int bsa_selftest_half_products(const void* a, const void* b, float* out, int dtype, int32_t* status,
                                          void* stream) {
  if (!a || !b || !out || !bsa::is_aligned(a, 16) || !bsa::is_aligned(b, 16) || !bsa::is_aligned(out, 16))
    return BSA_ERR_BAD_POINTER;
  if (dtype != BSA_F16 && dtype != BSA_BF16) return BSA_ERR_BAD_DTYPE;
  int rc;
  if ((rc = bsa::check_device_sm100()) != BSA_OK) return rc;
  auto kernel = dtype == BSA_BF16 ? bsa::half_products_selftest_kernel<true> : bsa::half_products_selftest_kernel<false>;
  kernel<<<1, 128, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const uint32_t*>(a), static_cast<const uint4*>(b),
                                                           out, status);
  return cudaGetLastError() == cudaSuccess ? BSA_OK : BSA_ERR_CUDA;
}
