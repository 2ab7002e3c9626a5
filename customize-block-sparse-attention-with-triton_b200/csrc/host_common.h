// Host-side helpers shared by the entry points: argument checks, per-device set-up, and TMA
// tensor-map encoding through a driver entry point resolved at run time (the library does not
// link libcuda).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/bsattn.h"

namespace bsa {

constexpr int kBlock = 64;     // tokens per mask block (semantic: the reference's BLOCK_M = BLOCK_N)
constexpr int kHeadDim = 64;   // the kernels' row width; narrower heads are zero-filled to it on load

inline bool head_dim_ok(int D) { return D == 16 || D == 32 || D == kHeadDim; }

inline bool is_aligned(const void* p, size_t a) { return (reinterpret_cast<uintptr_t>(p) % a) == 0; }

// 0 when the current device is compute capability 10.x, else a negative status.
int check_device_sm100();

// Validates a [B,H,N,D] 16-bit operand for TMA: base 16-byte aligned, last stride 1, the other
// strides positive multiples of 8 elements.
int check_qkv_operand(const void* p, const int64_t s[4]);

// Encodes a 4-D tile map over a [B,H,N,D] 16-bit tensor with element strides s[4]:
// box = box_rows x 64 elements, 128-byte swizzle, out-of-range rows and columns read as zero.
int make_qkv_tmap(CUtensorMap* out, const void* base, const int64_t s[4], int B, int H, int N,
                  int D, int dtype, int box_rows);

// The same with 64-row boxes out of a small per-thread cache of recent operands: encoding a map takes
// the driver about a microsecond, a forward and backward need seven, and a model calls the op with the
// same few buffers over and over.
int cached_qkv_tmap(CUtensorMap* out, const void* base, const int64_t s[4], int B, int H, int N, int D,
                    int dtype);

// Number of SMs of the current device (cached per device).
int sm_count(int* out);

// Launches a kernel that may begin while the previous one of the stream is still running (see
// grid_dependency_wait): its set-up and the launch itself, 2 to 4 us, then cost nothing between kernels
// that follow one another.
template <typename... Params, typename... Args>
int launch_dependent(void (*kernel)(Params...), dim3 grid, unsigned threads, size_t smem, cudaStream_t stream,
                     const Args&... args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...) == cudaSuccess ? BSA_OK : BSA_ERR_CUDA;
}

// bsa_tile_lists_places; together: beside the kernel before it in the stream, which has let it in after it
// has itself seen the end of everything earlier, the mask included.
int launch_lists_places(const uint8_t* block, const int64_t s[4], int B, int H, int nb, int32_t* row_cnt,
                        int32_t* col_idx, int32_t* col_cnt, int32_t* row_idx, bool together, void* stream);

// Raises a kernel's dynamic shared-memory limit; done once per (kernel, device) and remembered.  launch_regs: what
// its roles share out a thread, 0 if they share out nothing; see check_launch_registers.
int ensure_dynamic_smem(const void* kernel, size_t bytes, int launch_regs = 0);

// BSA_OK if the kernel is launched with just so many registers a thread, else BSA_ERR_REGISTERS.  The shares of a
// kernel whose roles exchange registers are constants, the number at launch is the compiler's: with fewer than they
// add up to, the roles that take some would wait for them, and that wait has no limit.
int check_launch_registers(const void* kernel, int launch_regs);

}  // namespace bsa
