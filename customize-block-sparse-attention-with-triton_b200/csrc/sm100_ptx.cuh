// Thin inline-PTX wrappers for the sm_100a features the attention kernels use:
// mbarrier, TMA tile loads (never multicast), tcgen05 MMA / TMEM alloc / ld / st / commit / fences,
// and the shared-memory and instruction descriptors of tcgen05.mma.kind::f16.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace bsa {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// One lane of a converged warp; the same lane on every call.  Code that feeds tcgen05 / TMA
// instructions runs warp-wide (so addresses and descriptors stay warp-uniform) and only the issue
// itself is guarded by this predicate.
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile(
      "{\n\t.reg .pred P;\n\t"
      "elect.sync _|P, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, P;\n\t}"
      : "=r"(pred));
  return pred != 0;
}
__device__ __forceinline__ int uniform_warp_index() {
  return __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
}
__device__ __forceinline__ void named_barrier_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// Counts as one of the threads that named_barrier_sync waits for, without waiting.
__device__ __forceinline__ void named_barrier_arrive(int id, int threads) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// Register split between the warpgroups of a block: executed by all four warps of one.  The shares
// must add up to no more than the registers the block was launched with.
template <int kRegs>
__device__ __forceinline__ void give_registers() {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegs));
}
template <int kRegs>
__device__ __forceinline__ void take_registers() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegs));
}

// Named barrier that also ORs a predicate over the participating threads.
__device__ __forceinline__ bool named_barrier_or(int id, int threads, bool pred) {
  uint32_t out;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %3, 0;\n\t"
      "bar.red.or.pred q, %1, %2, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(out)
      : "r"(id), "r"(threads), "r"(static_cast<uint32_t>(pred))
      : "memory");
  return out != 0;
}

// The vote of a role of several warps that meet at a named barrier in their items.  Each of them waits for the item by
// itself, and a wait may run out in one warp while the others still see what it waited for: an item, one that
// needs no barrier, or the end of the work.  So whenever they have met, for an item, because a wait has run out, or
// at the end of the work, they vote: all of them go on, or none does.
__device__ __forceinline__ bool role_leaves(int id, int threads, bool gave_up) {
  return named_barrier_or(id, threads, gave_up);
}

// Programmatic dependent launch: the attention kernels, delta, the lists with places and the in-place reorder are
// launched so that they may begin while the previous kernel of the stream is still running, do their set-up,
// and wait here, in every role, before they touch memory that another kernel may write or read, until that one
// has ended and its writes are visible.  (The mask reduction, the CSR lists and the out-of-place reorder are
// ordinary launches; without the attribute on the launch both instructions are no-ops.)
// Two kernels read before they wait: dQ beside dK/dV, and the tile lists of a training forward beside the forward.
// What they read was written before the kernel that they run beside, which lets them in from a thread that has
// itself waited for those writes.  That they see them too holds on B200 (steps on new data in the same buffers,
// called and replayed, are tested bit for bit); the programming model promises it only after a wait of their own.
__device__ __forceinline__ void grid_dependency_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
// The next kernel of the stream may be launched as soon as all CTAs have said so or ended.
__device__ __forceinline__ void grid_dependents_launch() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

__device__ __forceinline__ uint64_t global_timer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Records a give-up code in the optional status word unless one is there already.  Plain loads
// and stores on purpose: the word may live in pinned host memory that the device reaches over
// PCIe, and which of several simultaneous reports wins does not matter.
__device__ __forceinline__ void report_status(int32_t* status, int code) {
  if (status != nullptr) {
    volatile int32_t* w = status;
    if (*w == 0) *w = code;
    __threadfence_system();
  }
}

// ---------------------------------------------------------------------------------------------
// mbarrier
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
// A warp's lanes initialise n <= 32 barriers at once (one after the other takes 30 cycles each).
__device__ __forceinline__ void mbar_init_warp(uint64_t* bars, int n, uint32_t count, int lane) {
  if (lane < n) mbar_init(smem_u32(bars + lane), count);
}
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

// One lane's bounded look-out for the end of a phase.  False: it gave up, after so many tries, each of which the
// hardware suspends for up to 4 us (75 ns when the lanes of a warp have parted).  Lanes may disagree and come back one by one: the warp has to vote on
// the verdict before any other .sync.aligned instruction.
constexpr int kWaitTries = 1 << 19;  // 2 seconds in all
__device__ __forceinline__ bool mbar_poll(uint32_t bar, uint32_t parity, int tries) {
#pragma unroll 1
  while (!mbar_try_wait(bar, parity))
    if (--tries == 0) break;
  return tries != 0;
}

// Bounded wait of a whole (converged) warp, with one way out and one verdict for all of its lanes.  On give-up
// the caller records the code, raises the CTA's flag and leaves through the normal tear-down path so TMEM is
// always released.
// (This code is inlined at every wait of every role and run through at every superstep, mostly on barriers
// that are long complete.  Against a way out for each verdict and no vote, which lets lanes go on without
// the others: forward 0.3 to 1 %, training steps 1 to 2 %.  A vote, a look at the flag, a parked form of
// the wait or %globaltimer in every try cost 2 to 6 %, a look at the flag every 1024 tries 1 to 4 %.)
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, int tries = kWaitTries) {
  return __all_sync(0xffffffffu, mbar_poll(bar, parity, tries));
}

// Several barriers, one after the other, which share one limit.  The warp is together whenever it begins to look at one:
// its limit would be 0.04 s otherwise.
__device__ __forceinline__ void mbar_poll_shared(uint32_t bar, uint32_t parity, int* tries) {
#pragma unroll 1
  while (!mbar_try_wait(bar, parity))
    if (--*tries <= 0) break;
  __syncwarp();
}
__device__ __forceinline__ bool mbar_wait_warp_in_turn(uint32_t bar0, uint32_t parity0, uint32_t bar1, uint32_t parity1) {
  int tries = kWaitTries;
  mbar_poll_shared(bar0, parity0, &tries);
  mbar_poll_shared(bar1, parity1, &tries);
  return __all_sync(0xffffffffu, tries > 0);
}

// Two barriers at once: both looks are on their way together.  (A look takes 150 to 250 cycles while the tensor cores
// read their operands from shared memory, and one after the other cost the backward's S/dP issuers 450 cycles a
// superstep of 950: 2 x 16 heads, N = 16384, causal, a quarter, forward and backward 1,402 -> 1,378 us.  The forward's S
// issuer, which has time for them, takes them in turn: N = 17536, everything listed 107.2 us so, 106.5 in turn.)
__device__ __forceinline__ bool mbar_wait_warp2(uint32_t bar0, uint32_t parity0, uint32_t bar1, uint32_t parity1) {
  const bool seen0 = mbar_try_wait(bar0, parity0), seen1 = mbar_try_wait(bar1, parity1);
  if (__all_sync(0xffffffffu, seen0 && seen1)) return true;
  return mbar_wait_warp_in_turn(bar0, parity0, bar1, parity1);
}

__device__ __forceinline__ bool mbar_wait_warp3(uint32_t bar0, uint32_t parity0, uint32_t bar1, uint32_t parity1,
                                                uint32_t bar2, uint32_t parity2) {
  const bool seen0 = mbar_try_wait(bar0, parity0), seen1 = mbar_try_wait(bar1, parity1), seen2 = mbar_try_wait(bar2, parity2);
  if (__all_sync(0xffffffffu, seen0 && seen1 && seen2)) return true;
  int tries = kWaitTries;
  mbar_poll_shared(bar0, parity0, &tries);
  mbar_poll_shared(bar1, parity1, &tries);
  mbar_poll_shared(bar2, parity2, &tries);
  return __all_sync(0xffffffffu, tries > 0);
}

// The same for the beginning of an item, where a role comes that still had work when another one gave up: it
// looks at the CTA's flag every quarter of a second.  (The forward's write-out slept between its looks, 128 to 256 ns:
// one head, N = 1024 5.22 us, so 5.12.)
constexpr int kItemBatches = 8;
__device__ __forceinline__ bool mbar_wait_warp_item(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
#pragma unroll 1
  for (int batch = 0; batch < kItemBatches; ++batch) {
    if (mbar_wait_warp(bar, parity, kWaitTries / kItemBatches)) return true;
    if (__any_sync(0xffffffffu, *abort_flag != 0)) break;
  }
  return false;
}

// ---------------------------------------------------------------------------------------------
// TMA (cp.async.bulk.tensor), tile mode, 4-D, no multicast
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void tma_prefetch_desc(const void* tmap) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(tmap)) : "memory");
}
__device__ __forceinline__ void tma_load_4d(uint32_t dst_smem, const void* tmap, uint32_t bar,
                                            int c0, int c1, int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(dst_smem), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(bar), "r"(c0), "r"(c1), "r"(c2),
      "r"(c3)
      : "memory");
}
// Untiled bulk copy global -> shared; both addresses 16-byte aligned, bytes a multiple of 16.
__device__ __forceinline__ void bulk_load_1d(uint32_t dst_smem, const void* src, uint32_t bytes,
                                             uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
      ::"r"(dst_smem), "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(bar)
      : "memory");
}

// ---------------------------------------------------------------------------------------------
// tcgen05: TMEM allocation
// ---------------------------------------------------------------------------------------------
// Whole warp; writes the TMEM base address to *dst_smem.
__device__ __forceinline__ void tmem_alloc(uint32_t dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}

// ---------------------------------------------------------------------------------------------
// tcgen05: fences, commit, waits
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// The mbarrier receives one arrival once every tcgen05.mma issued so far by this thread is done.
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   bar)
               : "memory");
}
// What this thread has written to shared memory may be read by MMAs and bulk copies after the next barrier.
__device__ __forceinline__ void async_proxy_fence() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void tc_wait_ld() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_wait_st() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// ---------------------------------------------------------------------------------------------
// tcgen05.mma.kind::f16 (fp16/bf16 inputs, fp32 accumulate), one CTA
// ---------------------------------------------------------------------------------------------
// D[tmem] (+)= A[smem desc] * B[smem desc] with M = 64 rows of A in the "weight stationary" form: columns [0, N/2) of the result
// go to TMEM lanes 0..63, columns [N/2, N) to lanes 64..127 of the same N/2 TMEM columns, so all
// lanes are used (the ordinary M = 64 form runs at half rate).
__device__ __forceinline__ void umma_ws_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                           uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.ws.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem desc] in the same form with A in tensor memory: lanes 0..63 of D are their own
// rows of A times columns [0, N/2) of B, lanes 64..127 their own rows of A times columns [N/2, N).  With two tiles
// beside one another in B (MN-major, the leading byte offset is the way from one to the other) that is two
// products of 64 rows at once.  (Ordinary use has the same 64 rows in both lane halves.  That each half reads its own
// is how B200 does it and not promised anywhere; product_selftest.cu checks it element by element.)  Two products of 64 x 64
// with 64 columns: 176 cycles; as two M = 128 products, each with one lane half of the result switched off, 256.
// Both halves are always written: where there is no second tile, its rows of A and its part of B are zeros.
__device__ __forceinline__ void umma_ws_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc,
                                           uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.ws.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Shared-memory matrix descriptor for a tile stored as rows of 128 bytes with the 128-byte
// swizzle (what a TMA SWIZZLE_128B load of a [rows][64 x 16-bit] box produces; the tile base must
// be 1024-byte aligned).  Bits: [0,14) address>>4, [16,30) leading byte offset>>4, [32,46) stride
// byte offset>>4, [46,48) version = 1, [61,64) layout = 2 (SWIZZLE_128B).
//  * K-major use (the 64 contiguous elements are the contraction axis): one MMA consumes 16
//    elements = 32 bytes of every row; the next k-step starts 32 bytes further; 8-row groups are
//    1024 bytes apart (stride byte offset).
//  * MN-major use (the 64 contiguous elements are the M/N axis, rows are the contraction axis):
//    one MMA consumes 16 rows = 2 groups of 8 rows, groups 1024 bytes apart (stride byte offset);
//    the next k-step starts 2048 bytes further.  The leading byte offset is the way to the second
//    64-element chunk of the M/N axis: all accumulating products have N = 128, two tiles 8192 bytes apart.
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t smem_addr, uint32_t lbo_bytes,
                                                    uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr >> 4) & 0x3FFFu);
  d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFFu) << 16;
  d |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFFu) << 32;
  d |= 1ull << 46;
  d |= 2ull << 61;
  return d;
}

// Instruction descriptor of tcgen05.mma.kind::f16 with fp32 accumulation.
// Bits: [4,6) D format (1 = f32), [7,10) A format, [10,13) B format (0 = f16, 1 = bf16),
// 15 A major, 16 B major (0 = K-major, 1 = MN-major), [17,23) N>>3, [24,29) M>>4.
__host__ __device__ constexpr uint32_t umma_idesc(int is_bf16, int a_mn_major, int b_mn_major,
                                                  int M, int N) {
  return (1u << 4) | (static_cast<uint32_t>(is_bf16) << 7) | (static_cast<uint32_t>(is_bf16) << 10) |
         (static_cast<uint32_t>(a_mn_major) << 15) | (static_cast<uint32_t>(b_mn_major) << 16) |
         (static_cast<uint32_t>(N >> 3) << 17) | (static_cast<uint32_t>(M >> 4) << 24);
}

// ---------------------------------------------------------------------------------------------
// tcgen05.ld / tcgen05.st, shape 32x32b: thread i of the warp touches TMEM lane (lane_base + i),
// register j touches column (col_base + j).  A warp may only touch the 32 lanes of its own
// quarter: lane_base = 32 * (warp index % 4).
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void tmem_ld_32x32b_x32(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_32x32b_x16(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st_32x32b_x32(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]),
      "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]),
      "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]),
      "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]),
      "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st_32x32b_x16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]),
      "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]),
      "r"(r[15])
      : "memory");
}

__device__ __forceinline__ void tmem_st_32x32b_x4(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr), "r"(r[0]),
               "r"(r[1]), "r"(r[2]), "r"(r[3])
               : "memory");
}
__device__ __forceinline__ void tmem_ld_32x32b_x8(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
      : "r"(taddr)
      : "memory");
}

// Shapes 16x256b / 16x128b: 16 lanes (lane_base a multiple of 16 inside the warp's quarter) by 8 / 4 columns, N times
// beside one another.  Thread i holds, of each 8 columns, columns 2 (i % 4) and 2 (i % 4) + 1 of lanes i / 4
// (registers 0, 1) and i / 4 + 8 (registers 2, 3); of each 4, column i % 4 of the same two lanes.  So what it has read
// as two columns of fp32 it can store as one of 16-bit pairs.
__device__ __forceinline__ void tmem_ld_16x256b_x2(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st_16x128b_x2(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.16x128b.x2.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr), "r"(r[0]),
               "r"(r[1]), "r"(r[2]), "r"(r[3])
               : "memory");
}

// One 32-byte store (a whole sector) instead of two 16-byte ones; the address must be 32-byte
// aligned.
__device__ __forceinline__ void st_global_v8(void* p, const uint32_t* w) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(w[0]),
               "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
               : "memory");
}

// Two fp32 operations in one instruction (sm_100 packed forms; same rounding as the scalar ones).
__device__ __forceinline__ uint64_t pack_f32x2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack_f32x2(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t add_f32x2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// ---------------------------------------------------------------------------------------------
// small numeric helpers
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float lg2_approx(float x) {
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// Pack two floats into one 32-bit word of 16-bit values: `lo` in bits [0,16), `hi` in [16,32).
template <bool kBf16>
__device__ __forceinline__ uint32_t pack_2x16(float lo, float hi) {
  uint32_t r;
  if constexpr (kBf16) {
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  } else {
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  }
  return r;
}

}  // namespace bsa
