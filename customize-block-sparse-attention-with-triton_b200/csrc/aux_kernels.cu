// HBM-bound helpers around the attention kernels:
//   bsa_attn_bwd_delta   delta = rowsum(O * dO) in fp32
//   bsa_reorder / bsa_inv_reorder   head-wise permutation of the (F, H, W) token grid
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <atomic>
#include <string.h>

#include "host_common.h"
#include "sm100_ptx.cuh"

namespace bsa {

// ---------------------------------------------------------------------------------------------
// delta
// ---------------------------------------------------------------------------------------------
// Eight lanes own one 128-byte row (64 16-bit values): a warp covers 4 rows per step and a CTA of
// 8 warps covers 128 rows with 4 independent steps in flight per thread.
constexpr int kDeltaThreads = 256;

template <bool kBf16>
__device__ __forceinline__ float dot8(const uint4& a, const uint4& b) {
  const uint32_t aw[4] = {a.x, a.y, a.z, a.w};
  const uint32_t bw[4] = {b.x, b.y, b.z, b.w};
  float acc = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 fa, fb;
    if constexpr (kBf16) {
      fa = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&aw[i]));
      fb = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&bw[i]));
    } else {
      fa = __half22float2(*reinterpret_cast<const __half2*>(&aw[i]));
      fb = __half22float2(*reinterpret_cast<const __half2*>(&bw[i]));
    }
    acc = fmaf(fa.x, fb.x, acc);
    acc = fmaf(fa.y, fb.y, acc);
  }
  return acc;
}

// A row of D elements takes D / 8 lanes, 16 bytes each; four rows of a lane are in flight.  O and dO have
// strides of their own.
template <bool kBf16, int kD>
__global__ void __launch_bounds__(kDeltaThreads)
bwd_delta_kernel(const uint16_t* __restrict__ o, int64_t o_sb, int64_t o_sh, int64_t o_sn,
                 const uint16_t* __restrict__ dout, int64_t d_sb, int64_t d_sh, int64_t d_sn,
                 float* __restrict__ delta, int H, int N, int64_t rows) {
  constexpr int kLanes = kD / 8, kStep = 32 / kLanes;  // lanes of a row, rows of a warp at a time
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sub = lane / kLanes, chunk = lane % kLanes;
  // A warp's rows (16, 32 or 64) lie in one (batch, head): N is a multiple of 64 and the warp starts at
  // a multiple of their number, so the division is done once per thread, not once per row.
  const int64_t warp_row =
      (static_cast<int64_t>(blockIdx.x) * (kDeltaThreads / 32) + warp) * (4 * kStep);
  const int64_t row0 = warp_row + sub;
  const int64_t bh = warp_row / N;
  const int64_t n0 = warp_row - bh * N + sub;
  const int64_t b = bh / H, h = bh - b * H;
  const uint16_t* po = o + b * o_sb + h * o_sh + chunk * 8;
  const uint16_t* pd = dout + b * d_sb + h * d_sh + chunk * 8;
  grid_dependents_launch();
  grid_dependency_wait();
  uint4 xo[4], xd[4];
  bool live[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    live[i] = row0 + kStep * i < rows;
    if (live[i]) {
      xo[i] = __ldg(reinterpret_cast<const uint4*>(po + (n0 + kStep * i) * o_sn));
      xd[i] = __ldg(reinterpret_cast<const uint4*>(pd + (n0 + kStep * i) * d_sn));
    } else {
      xo[i] = make_uint4(0, 0, 0, 0);
      xd[i] = make_uint4(0, 0, 0, 0);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float acc = dot8<kBf16>(xo[i], xd[i]);
#pragma unroll
    for (int x = 1; x < kLanes; x *= 2) acc += __shfl_xor_sync(0xffffffffu, acc, x);
    if (chunk == 0 && live[i]) delta[row0 + kStep * i] = acc;
  }
}

template <int kD>
static int launch_delta(bool bf16, const void* o, const int64_t* os, const void* dout, const int64_t* ds,
                         float* delta, int H, int N, int64_t rows, cudaStream_t stream) {
  constexpr int64_t kRows = kDeltaThreads / 32 * 4 * (32 / (kD / 8));  // of a CTA
  const unsigned blocks = static_cast<unsigned>((rows + kRows - 1) / kRows);
  auto kern = bf16 ? bwd_delta_kernel<true, kD> : bwd_delta_kernel<false, kD>;
  return launch_dependent(kern, dim3(blocks), kDeltaThreads, 0, stream, static_cast<const uint16_t*>(o), os[0],
                          os[1], os[2], static_cast<const uint16_t*>(dout), ds[0], ds[1], ds[2], delta, H, N,
                          rows);
}

// ---------------------------------------------------------------------------------------------
// head-wise token reorder
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ int pick3(int sel, int v0, int v1, int v2) {
  return sel == 0 ? v0 : (sel == 1 ? v1 : (sel == 2 ? v2 : 0));
}

// Destination token of source token t for head order (p0,p1,p2) over a grid of extents
// (e0,e1,e2): the coordinates are re-laid-out in the order (p0,p1,p2).
__device__ __forceinline__ int permuted_token(int t, int e0, int e1, int e2, int p0, int p1,
                                              int p2) {
  const int plane = e1 * e2;
  const int c_f = t / plane;
  const int rem = t - c_f * plane;
  const int c_h = rem / e2;
  const int c_w = rem - c_h * e2;
  const int c0 = pick3(p0, c_f, c_h, c_w);
  const int c1 = pick3(p1, c_f, c_h, c_w);
  const int c2 = pick3(p2, c_f, c_h, c_w);
  const int d1 = pick3(p1, e0, e1, e2);
  const int d2 = pick3(p2, e0, e1, e2);
  return c0 * (d1 * d2) + c1 * d2 + c2;
}

constexpr int kReorderThreads = 256;
constexpr int kReorderPieces = 4;  // independent loads in flight per thread

// A CTA moves kReorderThreads * kReorderPieces Vec-sized pieces of the token rows of one
// (batch, head) (blockIdx.y, strided if the grid's y extent is smaller than batch * heads): all
// index arithmetic is 32-bit and the head's axis order is read once per CTA.  Every thread issues
// its loads before its stores.  kInverse: the source grid has the extents permuted by `orders`,
// and `inv_orders` lays the coordinates back out.
template <typename Vec, bool kInverse>
__global__ void __launch_bounds__(kReorderThreads)
reorder_kernel(const uint8_t* __restrict__ in, uint8_t* __restrict__ out, int64_t sb, int64_t sh,
               int64_t st, int64_t ob, int64_t oh, int64_t ot, const int32_t* __restrict__ orders,
               const int32_t* __restrict__ inv_orders, int heads, int n_bh, int T, int F, int Hh,
               int W, int vec_per_row) {
  const uint32_t per_head = static_cast<uint32_t>(T) * static_cast<uint32_t>(vec_per_row);
  const uint32_t first = blockIdx.x * (kReorderThreads * kReorderPieces) + threadIdx.x;
  for (int bh = blockIdx.y; bh < n_bh; bh += gridDim.y) {
    const int h = bh % heads;
    const int b = bh / heads;
    const int o0 = __ldg(orders + 3 * h), o1 = __ldg(orders + 3 * h + 1),
              o2 = __ldg(orders + 3 * h + 2);
    int e0 = F, e1 = Hh, e2 = W, p0 = o0, p1 = o1, p2 = o2;
    if constexpr (kInverse) {
      e0 = pick3(o0, F, Hh, W);
      e1 = pick3(o1, F, Hh, W);
      e2 = pick3(o2, F, Hh, W);
      p0 = __ldg(inv_orders + 3 * h);
      p1 = __ldg(inv_orders + 3 * h + 1);
      p2 = __ldg(inv_orders + 3 * h + 2);
    }
    // An order row that is not a permutation of (0, 1, 2) would send tokens past the end of the
    // head (the reference has no check either): such a head's rows are left unwritten.
    const bool valid = ((1 << p0) | (1 << p1) | (1 << p2)) == 7 && (p0 | p1 | p2) >= 0 &&
                       (!kInverse || (((1 << o0) | (1 << o1) | (1 << o2)) == 7 && (o0 | o1 | o2) >= 0));
    if (!valid) continue;
    const uint8_t* src = in + b * sb + h * sh;  // byte offsets
    uint8_t* dst = out + b * ob + h * oh;
    Vec val[kReorderPieces];
    int64_t to[kReorderPieces];
#pragma unroll
    for (int i = 0; i < kReorderPieces; ++i) {
      const uint32_t idx = first + i * kReorderThreads;
      to[i] = -1;
      if (idx < per_head) {
        const int t = static_cast<int>(idx / static_cast<uint32_t>(vec_per_row));
        const int piece = static_cast<int>(idx - static_cast<uint32_t>(t) * vec_per_row);
        val[i] = *reinterpret_cast<const Vec*>(src + t * st + piece * sizeof(Vec));
        to[i] = permuted_token(t, e0, e1, e2, p0, p1, p2) * ot + piece * sizeof(Vec);
      }
    }
#pragma unroll
    for (int i = 0; i < kReorderPieces; ++i)
      if (to[i] >= 0) *reinterpret_cast<Vec*>(dst + to[i]) = val[i];
  }
}

template <bool kInverse>
static int launch_reorder(const void* in, const int64_t s[4], void* out, const int64_t so[4],
                          const int32_t* orders, const int32_t* inv_orders, int B, int heads, int T, int D, int F, int Hh,
                          int W, int elem_bytes, void* stream) {
  if (B <= 0 || heads <= 0 || T <= 0 || D <= 0 || F <= 0 || Hh <= 0 || W <= 0 ||
      static_cast<int64_t>(F) * Hh * W != T)
    return BSA_ERR_BAD_SHAPE;
  if (elem_bytes != 1 && elem_bytes != 2 && elem_bytes != 4 && elem_bytes != 8)
    return BSA_ERR_BAD_DTYPE;
  if (!in || !out || !orders || (kInverse && !inv_orders)) return BSA_ERR_BAD_POINTER;
  if (!s || !so) return BSA_ERR_BAD_POINTER;
  if (s[3] != 1 || s[0] < 0 || s[1] < 0 || s[2] < 0) return BSA_ERR_BAD_STRIDE;
  if (so[3] != 1 || so[0] < 0 || so[1] < 0 || so[2] < 0) return BSA_ERR_BAD_STRIDE;
  const int64_t row_bytes = static_cast<int64_t>(D) * elem_bytes;
  const int64_t sb = s[0] * elem_bytes, sh = s[1] * elem_bytes, st = s[2] * elem_bytes;
  const int64_t ob = so[0] * elem_bytes, oh = so[1] * elem_bytes, ot = so[2] * elem_bytes;
  // widest piece that divides the row and keeps every access aligned
  int vec = 16;
  auto fits = [&](int v) {
    return row_bytes % v == 0 && sb % v == 0 && sh % v == 0 && st % v == 0 && ob % v == 0 &&
           oh % v == 0 && ot % v == 0 && is_aligned(in, v) && is_aligned(out, v);
  };
  while (vec > elem_bytes && !fits(vec)) vec >>= 1;
  if (!fits(vec)) return BSA_ERR_BAD_POINTER;
  const int vec_per_row = static_cast<int>(row_bytes / vec);
  const int64_t per_head = static_cast<int64_t>(T) * vec_per_row;
  const int64_t n_bh = static_cast<int64_t>(B) * heads;
  if (per_head > 0x7fffffffLL || n_bh > 0x7fffffffLL) return BSA_ERR_TOO_LARGE;
  constexpr int kPerCta = kReorderThreads * kReorderPieces;
  const dim3 g(static_cast<unsigned>((per_head + kPerCta - 1) / kPerCta),
               static_cast<unsigned>(n_bh < 65535 ? n_bh : 65535));
  cudaStream_t cs = static_cast<cudaStream_t>(stream);
  const uint8_t* pi = static_cast<const uint8_t*>(in);
  uint8_t* po = static_cast<uint8_t*>(out);
#define BSA_LAUNCH_REORDER(V)                                                                      \
  reorder_kernel<V, kInverse><<<g, kReorderThreads, 0, cs>>>(pi, po, sb, sh, st, ob, oh, ot,       \
                                                             orders, inv_orders, heads,            \
                                                             static_cast<int>(n_bh), T, F, Hh, W,  \
                                                             vec_per_row)
  switch (vec) {
    case 16: BSA_LAUNCH_REORDER(uint4); break;
    case 8: BSA_LAUNCH_REORDER(uint2); break;
    case 4: BSA_LAUNCH_REORDER(uint32_t); break;
    case 2: BSA_LAUNCH_REORDER(uint16_t); break;
    default: BSA_LAUNCH_REORDER(uint8_t); break;
  }
#undef BSA_LAUNCH_REORDER
  return cudaGetLastError() == cudaSuccess ? BSA_OK : BSA_ERR_CUDA;
}

// ---------------------------------------------------------------------------------------------
// head-wise token reorder in place
// ---------------------------------------------------------------------------------------------
// One cluster of CTAs reorders one column chunk (64 bytes or more of every row) of one head: every CTA
// gathers its share of the destination rows into shared memory, the cluster waits until all of it has been
// read, and every CTA stores its share.  Bound by HBM: each byte is read once and written once, where a
// gather into a second tensor and a copy back move it twice and allocate that tensor.  Shared
// memory holds 72 KB a CTA, so that three CTAs share an SM and one's loads run under the others' stores; a
// cluster of 16 holds 18,432 rows of 64 bytes, the reference's 13 x 30 x 45 grid among them.  More tokens than that
// are refused, and the caller goes back to the gather and the copy.
// B200, D = 64, 16 bit, q, k, v and output of 2 x 48 heads of that grid, orders drawn from all six:
// 0.69 ms with the gather and the copy, 0.31 with the rows in registers (two CTAs an SM), 0.28 in shared
// memory.  q, k, v alone, 5/6 of the heads with an order to move (1.08 GB read and written): 0.49, 0.22 and
// 0.20 ms, 5.5 TB/s.  A grid of 16 x 33 x 47, too large, stays at 2.2 TB/s by that count.
constexpr int kPermThreads = 512;
constexpr int kPermPieces = 9;  // 16-byte pieces a thread holds
constexpr int kPermTensors = 3;

struct PermuteArgs {
  uint8_t* base[kPermTensors];
  int64_t sb[kPermTensors], sh[kPermTensors], st[kPermTensors];  // bytes
  const void* plan;       // the axis order of a head, as an index into the six of permute_kernel
  int64_t plan_stride;    // in elements
  int plan_is_64;
  int32_t* status;        // optional
  int B, heads, T, chunks, chunk_bytes, pieces_per_cta;
  int ext[3];             // F, Hh, W
  // floor(n / d) = umulhi(n, m) for n * d < 2^32: m = floor(2^32 / d) + 1
  uint32_t m_vec;         // d = pieces of a row's chunk
  uint32_t m_ext[3];      // d = ext[i]
  uint32_t m_plane[3];    // d = product of the other two extents
};

__device__ __forceinline__ uint32_t div_by(uint32_t n, uint32_t d, uint32_t m) {
  return d == 1 ? n : __umulhi(n, m);
}

// (indexing of PermuteArgs with constants only, so that nothing goes through local memory)
__device__ __forceinline__ uint32_t pick3u(int sel, uint32_t v0, uint32_t v1, uint32_t v2) {
  return sel == 0 ? v0 : (sel == 1 ? v1 : v2);
}

template <bool kInverse>
__global__ void __launch_bounds__(kPermThreads, 3) permute_kernel(const __grid_constant__ PermuteArgs a) {
  extern __shared__ __align__(16) uint8_t s_pieces[];  // piece i of thread t at (i * kPermThreads + t) * 16
  grid_dependents_launch();
  grid_dependency_wait();
  int unit = blockIdx.y;
  const int chunk = unit % a.chunks;
  unit /= a.chunks;
  const int h = unit % a.heads;
  unit /= a.heads;
  const int b = unit % a.B, which = unit / a.B;
  int64_t order = a.plan_is_64 ? static_cast<const int64_t*>(a.plan)[h * a.plan_stride]
                               : static_cast<const int32_t*>(a.plan)[h * a.plan_stride];
  if (order < 0) order += 6;
  // nothing to do for the order (0,1,2); an index that is none leaves the head alone and is reported.
  // The same for every CTA of the cluster.
  if (order <= 0 || order > 5) {
    if (order != 0 && blockIdx.x == 0 && threadIdx.x == 0) report_status(a.status, BSA_REPORT_BAD_ORDER);
    return;
  }
  // axis orders 1..5: (0,2,1), (1,2,0), (1,0,2), (2,1,0), (2,0,1)
  const int p0 = order >= 4 ? 2 : (order == 1 ? 0 : 1);
  const int p1 = order == 1 || order == 2 ? 2 : (order == 4 ? 1 : 0);
  const int p2 = 3 - p0 - p1;
  const uint32_t e0 = a.ext[0], e1 = a.ext[1], e2 = a.ext[2];
  const uint32_t d1 = pick3u(p1, e0, e1, e2), d2 = pick3u(p2, e0, e1, e2);
  // the destination is walked in its own axis order; its token splits into coordinates along the axes
  // q0, q1, q2 (the permuted ones, or, laying back, the grid's own)
  const uint32_t g1 = kInverse ? e1 : d1, g2 = kInverse ? e2 : d2;
  const uint32_t m_plane = kInverse ? a.m_plane[0] : pick3u(p0, a.m_plane[0], a.m_plane[1], a.m_plane[2]);
  const uint32_t m_last = kInverse ? a.m_ext[2] : pick3u(p2, a.m_ext[0], a.m_ext[1], a.m_ext[2]);
  // weight of each of those coordinates in the source token
  uint32_t w0, w1, w2;
  if (kInverse) {  // source: grid in the order (p0, p1, p2)
    const uint32_t s0 = d1 * d2, s1 = d2;
    w0 = p0 == 0 ? s0 : (p1 == 0 ? s1 : 1u);
    w1 = p0 == 1 ? s0 : (p1 == 1 ? s1 : 1u);
    w2 = p0 == 2 ? s0 : (p1 == 2 ? s1 : 1u);
  } else {         // source: the grid's own order
    w0 = pick3u(p0, e1 * e2, e2, 1u);
    w1 = pick3u(p1, e1 * e2, e2, 1u);
    w2 = pick3u(p2, e1 * e2, e2, 1u);
  }
  const int64_t st = which == 0 ? a.st[0] : (which == 1 ? a.st[1] : a.st[2]);
  uint8_t* const base =
      (which == 0 ? a.base[0] + b * a.sb[0] + h * a.sh[0]
                  : (which == 1 ? a.base[1] + b * a.sb[1] + h * a.sh[1] : a.base[2] + b * a.sb[2] + h * a.sh[2])) +
      static_cast<int64_t>(chunk) * a.chunk_bytes;
  const uint32_t vec = static_cast<uint32_t>(a.chunk_bytes) >> 4;
  const uint32_t first = blockIdx.x * a.pieces_per_cta + threadIdx.x;
  const uint32_t end = min(static_cast<uint32_t>(a.T) * vec, (blockIdx.x + 1) * a.pieces_per_cta);
  uint4* const mine = reinterpret_cast<uint4*>(s_pieces) + threadIdx.x;
#pragma unroll
  for (int i = 0; i < kPermPieces; ++i) {
    const uint32_t idx = first + i * kPermThreads;
    if (idx < end) {
      const uint32_t t = div_by(idx, vec, a.m_vec), piece = idx - t * vec;
      const uint32_t c0 = div_by(t, g1 * g2, m_plane), rem = t - c0 * (g1 * g2);
      const uint32_t c1 = div_by(rem, g2, m_last), c2 = rem - c1 * g2;
      const uint32_t from = c0 * w0 + c1 * w1 + c2 * w2;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(mine + i * kPermThreads)),
                   "l"(base + from * st + piece * 16u) : "memory");
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  // every CTA of the cluster has read its share before any of them stores
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < kPermPieces; ++i) {
    const uint32_t idx = first + i * kPermThreads;
    if (idx < end) {
      const uint32_t t = div_by(idx, vec, a.m_vec), piece = idx - t * vec;
      *reinterpret_cast<uint4*>(base + t * st + piece * 16u) = mine[i * kPermThreads];
    }
  }
}

template <bool kInverse>
static int launch_permute(PermuteArgs& a, int n_tensors, int cluster, cudaStream_t stream) {
  auto kern = permute_kernel<kInverse>;
  constexpr size_t kSmem = kPermThreads * kPermPieces * 16;
  const int smem_rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), kSmem);
  if (smem_rc != BSA_OK) return smem_rc;
  static std::atomic<int> ready[64];  // per device: 0 unknown, 1 clusters of 16 fit, 2 they do not
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return BSA_ERR_CUDA;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(cluster);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  const int64_t units = static_cast<int64_t>(n_tensors) * a.B * a.heads * a.chunks;
  if (units > 65535) return BSA_ERR_TOO_LARGE;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(cluster), static_cast<unsigned>(units), 1);
  cfg.blockDim = dim3(kPermThreads, 1, 1);
  cfg.dynamicSmemBytes = kSmem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  if (cluster > 8) {
    int r = ready[dev].load(std::memory_order_relaxed);
    if (r == 0) {
      int n = 0;
      const bool ok = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                      cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess && n > 0;
      if (!ok) (void)cudaGetLastError();
      r = ok ? 1 : 2;
      ready[dev].store(r, std::memory_order_relaxed);
    }
    if (r == 2) return BSA_ERR_TOO_LARGE;
  }
  return cudaLaunchKernelEx(&cfg, kern, a) == cudaSuccess ? BSA_OK : BSA_ERR_CUDA;
}

}  // namespace bsa

extern "C" int bsa_attn_bwd_delta_strided(const void* o, const int64_t o_strides[4], const void* dout,
                                          const int64_t do_strides[4], float* delta, int dtype, int B,
                                          int H, int N, int D, void* stream) {
  using namespace bsa;
  if (B <= 0 || H <= 0 || N <= 0 || !head_dim_ok(D)) return BSA_ERR_BAD_SHAPE;
  if (dtype != BSA_F16 && dtype != BSA_BF16) return BSA_ERR_BAD_DTYPE;
  if (!delta || !o_strides || !do_strides) return BSA_ERR_BAD_POINTER;
  int rc;
  if ((rc = check_qkv_operand(o, o_strides)) != BSA_OK) return rc;
  if ((rc = check_qkv_operand(dout, do_strides)) != BSA_OK) return rc;
  const int64_t rows = static_cast<int64_t>(B) * H * N;
  if (rows / 128 >= 0x7fffffffLL) return BSA_ERR_TOO_LARGE;
  const bool bf16 = dtype == BSA_BF16;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (D == 64) return launch_delta<64>(bf16, o, o_strides, dout, do_strides, delta, H, N, rows, st);
  if (D == 32) return launch_delta<32>(bf16, o, o_strides, dout, do_strides, delta, H, N, rows, st);
  return launch_delta<16>(bf16, o, o_strides, dout, do_strides, delta, H, N, rows, st);
}

extern "C" int bsa_attn_bwd_delta(const void* o, const void* dout, const int64_t s[4], float* delta,
                                  int dtype, int B, int H, int N, int D, void* stream) {
  return bsa_attn_bwd_delta_strided(o, s, dout, s, delta, dtype, B, H, N, D, stream);
}

extern "C" int bsa_permute_in_place(void* const tensors[], const int64_t* strides, int n_tensors,
                                    const void* plan, int plan_elem_bytes, int64_t plan_stride,
                                    int inverse, int B, int heads, int T, int D, int F, int Hh, int W,
                                    int elem_bytes, void* stream) {
  return bsa_permute_in_place_status(tensors, strides, n_tensors, plan, plan_elem_bytes, plan_stride, inverse, B,
                                     heads, T, D, F, Hh, W, elem_bytes, nullptr, stream);
}

extern "C" int bsa_permute_in_place_status(void* const tensors[], const int64_t* strides, int n_tensors,
                                           const void* plan, int plan_elem_bytes, int64_t plan_stride,
                                           int inverse, int B, int heads, int T, int D, int F, int Hh, int W,
                                           int elem_bytes, int32_t* status, void* stream) {
  using namespace bsa;
  if (B <= 0 || heads <= 0 || T <= 0 || D <= 0 || F <= 0 || Hh <= 0 || W <= 0 || n_tensors < 1 ||
      n_tensors > kPermTensors || static_cast<int64_t>(F) * Hh * W != T)
    return BSA_ERR_BAD_SHAPE;
  if ((elem_bytes != 1 && elem_bytes != 2 && elem_bytes != 4 && elem_bytes != 8) ||
      (plan_elem_bytes != 4 && plan_elem_bytes != 8))
    return BSA_ERR_BAD_DTYPE;
  if (!tensors || !strides || !plan) return BSA_ERR_BAD_POINTER;
  PermuteArgs a;
  memset(&a, 0, sizeof(a));
  for (int i = 0; i < n_tensors; ++i) {
    const int64_t* s = strides + 4 * i;
    if (s[3] != 1) return BSA_ERR_BAD_STRIDE;
    for (int k = 0; k < 3; ++k)
      if (s[k] < 0 || (s[k] * elem_bytes) % 16 != 0) return BSA_ERR_BAD_STRIDE;
    if (!tensors[i] || !is_aligned(tensors[i], 16)) return BSA_ERR_BAD_POINTER;
    a.base[i] = static_cast<uint8_t*>(tensors[i]);
    a.sb[i] = s[0] * elem_bytes;
    a.sh[i] = s[1] * elem_bytes;
    a.st[i] = s[2] * elem_bytes;
  }
  const int64_t row_bytes = static_cast<int64_t>(D) * elem_bytes;
  if (row_bytes % 16 != 0 || row_bytes > (1 << 20)) return BSA_ERR_BAD_STRIDE;
  // As few column chunks as a cluster of 16 can hold, none below 64 bytes (two DRAM sectors) unless the
  // row is; then the smallest cluster that holds one.
  constexpr int64_t kCapacity = kPermThreads * kPermPieces * 16;
  int64_t chunk = row_bytes;
  while (T * chunk > 16 * kCapacity && chunk % 32 == 0 && chunk >= 128) chunk /= 2;
  const int64_t pieces = T * (chunk / 16);
  if (pieces * 16 > 16 * kCapacity || pieces * (chunk / 16) >= (1ll << 32) || T >= 65536) return BSA_ERR_TOO_LARGE;
  int cluster = 1;
  while (cluster * kCapacity < pieces * 16) cluster *= 2;
  a.plan = plan;
  a.plan_stride = plan_stride;
  a.plan_is_64 = plan_elem_bytes == 8;
  a.status = status;
  a.B = B;
  a.heads = heads;
  a.T = T;
  a.chunk_bytes = static_cast<int>(chunk);
  a.chunks = static_cast<int>(row_bytes / chunk);
  a.pieces_per_cta = static_cast<int>((pieces + cluster - 1) / cluster);
  a.ext[0] = F;
  a.ext[1] = Hh;
  a.ext[2] = W;
  const auto magic = [](int64_t d) { return static_cast<uint32_t>((1ll << 32) / d + 1); };
  a.m_vec = magic(chunk / 16);
  for (int i = 0; i < 3; ++i) {
    a.m_ext[i] = magic(a.ext[i]);
    a.m_plane[i] = magic(T / a.ext[i]);
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  return inverse ? launch_permute<true>(a, n_tensors, cluster, st) : launch_permute<false>(a, n_tensors, cluster, st);
}

extern "C" int bsa_reorder(const void* in, void* out, const int64_t strides[4],
                           const int32_t* orders, int B, int heads, int T, int D, int F, int Hh,
                           int W, int elem_bytes, void* stream) {
  return bsa::launch_reorder<false>(in, strides, out, strides, orders, nullptr, B, heads, T, D, F,
                                    Hh, W, elem_bytes, stream);
}

extern "C" int bsa_reorder_strided(const void* in, const int64_t in_strides[4], void* out,
                                   const int64_t out_strides[4], const int32_t* orders, int B,
                                   int heads, int T, int D, int F, int Hh, int W, int elem_bytes,
                                   void* stream) {
  return bsa::launch_reorder<false>(in, in_strides, out, out_strides, orders, nullptr, B, heads, T,
                                    D, F, Hh, W, elem_bytes, stream);
}

extern "C" int bsa_inv_reorder(const void* in, void* out, const int64_t strides[4],
                               const int32_t* orders, const int32_t* inv_orders, int B, int heads,
                               int T, int D, int F, int Hh, int W, int elem_bytes, void* stream) {
  return bsa::launch_reorder<true>(in, strides, out, strides, orders, inv_orders, B, heads, T, D, F,
                                   Hh, W, elem_bytes, stream);
}

extern "C" int bsa_inv_reorder_strided(const void* in, const int64_t in_strides[4], void* out,
                                       const int64_t out_strides[4], const int32_t* orders,
                                       const int32_t* inv_orders, int B, int heads, int T, int D,
                                       int F, int Hh, int W, int elem_bytes, void* stream) {
  return bsa::launch_reorder<true>(in, in_strides, out, out_strides, orders, inv_orders, B, heads,
                                   T, D, F, Hh, W, elem_bytes, stream);
}
