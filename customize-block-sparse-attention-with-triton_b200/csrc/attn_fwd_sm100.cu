// Forward block-sparse attention for sm_100a.
//
// Persistent kernel: one CTA per SM.  A work item is ONE query block (64 rows) of one (batch, head)
// with its list of key blocks; CTA c starts with item c and then draws further items from an
// optional work counter (or walks a fixed stride).  The list is taken FOUR key tiles at a time
// ("supersteps": tiles a, b, c, d in list order).  The 128 TMEM lanes are split between the
// tiles: lanes 0..63 own tiles a and c, lanes 64..127 own tiles b and d, so that every SM
// sub-partition (32 lanes) has the same amount of exp2 work whatever the sparsity pattern.
//
// S of a superstep is ONE product of 64 query rows with 256 keys: the M = 64 "weight stationary"
// form of the MMA puts columns [0, 128) of its result into lanes 0..63 and columns [128, 256) into
// lanes 64..127 of the same 128 TMEM columns, which is just the split above.  (An M = 128
// instruction can only fill the lanes that way with half of its rows multiplied by zeros.)  P V
// takes tiles a and b, then c and d, in one product each: in the same form every lane half multiplies its own P
// with its own half of the columns of [V_a | V_b].  A pair whose second tile does not exist has zeros in its place, in P
// and in V.  Measured on one SM, in cycles per tile: S 80 (128 with the M = 128 form, both bound by the operand
// reads from shared memory at 128 B per cycle), P V 88 (128 as two M = 128 products with half of the lanes
// switched off each).
//
// The supersteps alternate between two softmax teams of four warps, each with its own accumulator,
// so that one team exponentiates while the other waits for its products.  Three S slots rotate;
// the probabilities go over the logits of their slot, which is held from the S product until P V
// is complete.
//
// What bounds it: with everything listed a tile takes 320 active SM cycles, of which the exp2 unit
// is busy 256 (4096 exponentials at 16 per cycle).  The softmax warps wait for nothing: of a team's 2,600 cycles a superstep
// 2,000 lie between its logits and its last exponential (64 columns take a warp 730 cycles alone and 1,160 beside
// the other team's, 512 being the unit's limit), the rest are a look at a barrier, two loads, a store and an
// arrival, 60 to 120 cycles each.  MMA operand reads (144 cycles a tile) and arriving tiles (128) take most of shared
// memory's port.  With short lists the way of an item comes first: ticket and list 2,000 cycles, first tiles 1,600, from the
// last product to the last store 2,300; and the instruction cache: all roles run at the same time, and with 86 KB of
// code (most of it unrolled by the compiler; 50 KB now) the instruction caches of a GPC were 73 % busy.  So what is
// executed per item or per superstep is kept short, waits included, and no loop is unrolled without a reason.
// B200, D = 64, public calls back to back on inputs that rotate: fp16 N = 17536 with one head, all blocks
// 106 us (115 with products of one tile each, shared memory not aligned and a write-out warp for lister, in turn on one
// GPU), a tenth of them 17.1 us (18.5); 8 heads, a tenth 100 us (111); bf16 N = 32000, 32 heads, a tenth 1.180 ms
// (1.280), at the power cap.
//
// Roles (17 warps of 20); every role walks the same item sequence, so set-up of item i+1 and write-out
// of item i-1 overlap the arithmetic of item i:
//   warps 0..7  : online softmax (team = warp / 4, TMEM lane quarter = warp % 4; superstep g is team
//                 g % 2's).  A warp loads its tiles' 128 logits, exponentiates them, packs P to 16 bit
//                 and stores it over the logits (first tile in columns [0, 32) of the slot, second
//                 one in [32, 64)).
//   warp 8      : K producer — TMA-loads Q and the listed K tiles of every item into a 3-deep ring of
//                 superstages (4 tiles, held until S is complete), one lane per tile, and tells the lister
//                 when to set up the next item
//   warp 9      : S issuer and TMEM owner
//   warp 10     : P V issuer — O[team] += P_t V_t for the tiles t of the superstep, two at a time.  P is read
//                 from TMEM, V is an MN-major shared-memory operand.  Row r of an accumulator sums products
//                 of tiles a and c, row r+64 of tiles b and d.
//   warp 11     : V producer — TMA-loads the listed V tiles in pairs into a 5-deep ring (held until
//                 their P V is complete); they land on the barrier that P arrives on.  Only listed tiles
//                 are ever loaded.
//   warps 12..15: write-out — merge the four partial results (m, l, O) of every query row (teams x
//                 lanes r / r+64), normalise, store O, LSE and the row maximum
//   warp 18     : lister — draws the items, lists their key blocks (from the mask row, or copies the CSR row)
//                 into the next of three list buffers and publishes them
// The lister was one of the write-out warps: ticket, list and write-out one after the other took 4,100 cycles an item,
// more than an item of three supersteps does.  With a warp of its own, and an item there as soon as the one before the
// one before the previous one has been written out: 24 heads, N = 4160, D = 32, a quarter 46.1 -> 42.6 us; bf16
// 2 x 16 heads, N = 16384, causal, a quarter 412 -> 390; 8 heads, N = 17536, a tenth 99.2 -> 97.6; lists of one item a CTA the
// same.  It matters which quarter of the SM it runs in, beside the K producer (warp 16), the S issuer (17), the P V
// issuer (18) or the V producer (19): 32 heads, N = 32000 1,152 / 1,149 / 1,141 / 1,139 us (1,142 before).  (The K
// producer as lister: 8 heads 99 -> 103.)
// TMEM (512 columns): S/P slots 3 x 128, accumulators 2 x 64.
//
// Head dimensions 16 and 32 run on the same 128-byte rows: the tensor maps are D wide, so TMA fills
// the other columns of a tile with zeros without reading them, and S takes D / 16 K steps instead of
// four.
//
// Numerics follow the reference's loop (fa2_custom_mask/fa2_fwd.py:150-196): logits scaled by
// sm_scale*log2(e), exp2 domain, fp32 row sums of the fp32 probabilities, P rounded to the input
// dtype before P V.  The reference maximum of a row comes from its first 32 logits and moves only
// when later ones would make probabilities too large for 16 bit (sum of a superstep above 4096; then to
// the maximum of that superstep), which leaves O = acc / l unchanged because both use the same reference.  Which partial result a tile
// goes into depends on its position in the row's list alone, so results do not depend on which CTA
// computes an item.
//
// Every wait is bounded.  A role that gives up leaves its loops and raises a CTA-wide flag, which the waits for an
// item and of the write-out look at; a role in the middle of an item runs out by itself, within the same
// 2 seconds or so.  TMEM is always released.  Every
// barrier is waited on only by warps that see each of its phases, or that know the barrier to be
// at most one phase behind (a parity wait cannot tell a phase from the one two before it).
#include <math.h>

#include "host_common.h"
#include "sm100_ptx.cuh"

namespace bsa {

constexpr int kKStages = 3;     // K superstages (4 tiles) in flight: held from load to S complete
constexpr int kVStages = 5;     // pairs of V tiles in flight: held from load to P V complete
constexpr int kSlots = 3;       // S/P slots (128 TMEM columns): held from S issue to P V complete
constexpr int kLists = 3;       // items set up at a time: one being worked on, one written out, one to come
constexpr int kSoftmaxWarps = 8;
constexpr int kTeamWarps = kSoftmaxWarps / 2;
constexpr int kProducerWarp = 8, kSWarp = 9, kPvWarp = 10, kVProducerWarp = 11;
constexpr int kListerWarp = 18;
constexpr int kFwdThreads = 32 * 20;  // whole warpgroups: one warp at the end fills one
// Registers by warpgroup: 2 softmax, producers and issuers, write-out, lister.  All waits are bounded but the one for
// registers that the block was not launched with; and a share above what a warp has is taken, not given.  (kLaunchRegs
// is what the compiler makes of the launch bounds; the host compares before the first launch.)
constexpr int kLaunchRegs = 96, kSoftmaxRegs = 160, kIssuerRegs = 40, kWriteRegs = 88, kListerRegs = 32;
static_assert(2 * kSoftmaxRegs + kIssuerRegs + kWriteRegs + kListerRegs <= kLaunchRegs * kFwdThreads / 128);
static_assert(kSoftmaxRegs >= kLaunchRegs && kIssuerRegs <= kLaunchRegs && kWriteRegs <= kLaunchRegs &&
              kListerRegs <= kLaunchRegs);
constexpr int kGoBefore = 2;         // supersteps before an item's end at which the next is set up
constexpr uint32_t kTileBytes = 64 * 64 * 2;       // one Q, K or V tile
constexpr uint32_t kFwdTmemCols = 512;
// TMEM columns: slot r at 128 r; accumulator of softmax team T at 384 + 64 T.
constexpr uint32_t kTmemO = 384;
constexpr float kRescaleThreshold = 8.0f;
// Largest sum of a row's probabilities in a superstep (hence largest probability) that may go into P
// against a reference maximum that was not checked: far below fp16's 65504.
constexpr float kMaxRowSum = 4096.0f;
constexpr int kFrontRounds = 4, kFrontRows = 8;  // see fwd_item
constexpr int kFwdMaxTiles = 2048;  // key blocks per row that a CTA can list (N <= 131072)
constexpr uint16_t kColPartial = 0x8000;  // list entry in shared memory: the tile has masked elements
constexpr uint16_t kColIndex = 0x7fff;

struct FwdSmem {
  uint8_t q[2][kTileBytes];                   // by parity of the non-empty items
  uint8_t k[kKStages][4][kTileBytes];         // tiles in the order a, c, b, d
  uint8_t v[kVStages][2][kTileBytes];
  // write-out: what lanes 0..63 and 64..127 hand to each other, 16 columns of 64 rows at a time (rows
  // of 20 floats: eight lanes' 16-byte accesses then fall into different banks)
  float xfer[2][64][20];
  uint16_t cols[kLists][kFwdMaxTiles];        // ring over the items: the item's key-block list (| kColPartial)
  int4 item[kLists];                          // the item: batch (-1 = no more work), head, query block, tile count
  float mref[kLists][2][128];                 // by list buffer of the item, softmax team, lane
  float lsum[kLists][2][128];
  float mtrue[kLists][2][128];
  uint64_t list_full[kLists];                 // lister -> everyone: list and header ready
  uint64_t list_free[kLists];                 // everyone is through with list, header and statistics
  uint64_t setup_go[2];                       // producer -> lister: time to set up the next item
  uint64_t q_free[2];                         // S of the item complete
  uint64_t k_full[kKStages];                  // the superstep's K tiles (and, with an item's first, its Q) are there
  uint64_t k_empty[kKStages];                 // S of the superstep complete
  uint64_t s_full[2 * kSlots];                // S of the superstep complete; one per (team, slot), so
                                              // that the team that waits on it sees each phase
  uint64_t p_full[kSlots];                    // the team's four warps stored P of the superstep, its V has landed
  uint64_t pv_done[kSlots];                   // P V of the superstep complete: slot and V places free, O current
  uint64_t o_full[2];                         // last P V of the item done
  uint64_t stats_full[kLists];                // softmax warps published (m, l) of the item
  uint64_t o_free[2];                         // write-out has read accumulators, stats and header
  uint32_t tmem_base;
  int abort_flag;
};
static_assert(sizeof(FwdSmem) <= 232448, "FwdSmem exceeds the shared memory of one CTA");

struct FwdParams {
  const int32_t* row_ptr;   // list mode: CSR row lists
  const int32_t* col_idx;
  const uint8_t* block;     // mask mode (block != nullptr): the kernel lists the mask rows itself
  int64_t ms0, ms1, ms2, ms3;
  const uint8_t* dense;     // optional element-level mask for the tiles marked partial
  int64_t ds0, ds1, ds2;
  void* o;
  int64_t o_sb, o_sh, o_sn;
  float* lse2;     // optional
  float* rowmax;   // optional
  int B, H, N, D, nb;
  int row_begin, nrows;     // the query-block rows [row_begin, row_begin + nrows) of every head
  int list_b_stride, list_h_stride;
  int items;                // B * H * nrows
  float scale_log2;
  int32_t* status;
  int32_t* ticket;          // optional work counter (0 at kernel start, left 0): dynamic item hand-out
  int front, front_items;   // so many first rows of every head come before all others
  int wide_stores;          // rows of O start on 32-byte boundaries
  int successor_early;      // what follows in the stream may begin before this kernel ends, and knows it
};

enum FwdFail : int { kFailProducer = 1, kFailMma = 2, kFailSoftmax = 3, kFailOut = 4 };

__device__ __forceinline__ void fwd_give_up(FwdSmem* sm, int32_t* status, int code) {
  sm->abort_flag = 1;
  report_status(status, code);
}

// exp2 of 32 columns of S against the row's reference maximum: packs the probabilities to 16 bit and
// adds them (fp32) to two pairs of running sums.  The scale-and-subtract and the sums take two
// columns per instruction.
template <bool kBf16>
__device__ __forceinline__ void exp_chunk(const uint32_t* sr, float c, float neg_m, uint32_t* pk,
                                          uint64_t& l0, uint64_t& l1) {
  const uint64_t c2 = pack_f32x2(c, c), m2 = pack_f32x2(neg_m, neg_m);
#pragma unroll
  for (int i = 0; i < 32; i += 4) {
    float z0, z1, z2, z3;
    unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(sr[i]), __uint_as_float(sr[i + 1])), c2, m2),
                 z0, z1);
    unpack_f32x2(
        fma_f32x2(pack_f32x2(__uint_as_float(sr[i + 2]), __uint_as_float(sr[i + 3])), c2, m2), z2,
        z3);
    const float p0 = ex2_approx(z0), p1 = ex2_approx(z1), p2 = ex2_approx(z2), p3 = ex2_approx(z3);
    l0 = add_f32x2(l0, pack_f32x2(p0, p1));
    l1 = add_f32x2(l1, pack_f32x2(p2, p3));
    pk[i / 2] = pack_2x16<kBf16>(p0, p1);
    pk[i / 2 + 1] = pack_2x16<kBf16>(p2, p3);
  }
}

__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));  // one instruction on sm_100
  return d;
}

__device__ __forceinline__ float max_chunk(const uint32_t* sr) {
  float mx0 = __uint_as_float(sr[0]), mx1 = __uint_as_float(sr[1]);
#pragma unroll
  for (int i = 2; i < 30; i += 4) {
    mx0 = max3(mx0, __uint_as_float(sr[i]), __uint_as_float(sr[i + 1]));
    mx1 = max3(mx1, __uint_as_float(sr[i + 2]), __uint_as_float(sr[i + 3]));
  }
  return max3(mx0, mx1, fmaxf(__uint_as_float(sr[30]), __uint_as_float(sr[31])));
}

// 32 logits of one row: those whose mask byte is zero become -inf, so that they take no part in the
// maximum and exponentiate to 0.
__device__ __forceinline__ void mask_chunk(uint32_t* sr, const uint8_t* mask) {
  uint4 mw[2];
#pragma unroll
  for (int j = 0; j < 2; ++j) mw[j] = __ldg(reinterpret_cast<const uint4*>(mask) + j);
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const uint32_t w4[4] = {mw[j].x, mw[j].y, mw[j].z, mw[j].w};
#pragma unroll
    for (int q4 = 0; q4 < 4; ++q4) {
      const uint32_t nz = __vcmpne4(w4[q4], 0u);  // 0xff in every byte that keeps its element
#pragma unroll
      for (int bb = 0; bb < 4; ++bb) {
        const uint32_t keep = __byte_perm(nz, 0u, 0x1111u * bb);
        const int i = 16 * j + 4 * q4 + bb;
        sr[i] = (sr[i] & keep) | (0xff800000u & ~keep);
      }
    }
  }
}

// Takes a superstep's scaled row maximum into a lane's running ones; returns the factor by which the lane's
// rows of O have to be rescaled (1: not at all).  The reference moves when the maximum lies more than
// `slack` above it.  (A row with nothing kept so far keeps m_ref = -inf: its logits are all -inf, and
// against a zero in place of the maximum they exponentiate to 0 instead of NaN.)
__device__ __forceinline__ float fwd_new_max(float zmax, float slack, float& m_ref, float& m_true, float& l) {
  float alpha = 1.f;
  m_true = fmaxf(m_true, zmax);
  if (m_ref == -INFINITY) {
    m_ref = zmax;  // first tile of this lane in this item: O and l are still zero
  } else if (zmax > m_ref + slack) {
    alpha = ex2_approx(m_ref - zmax);
    l *= alpha;
    m_ref = zmax;
  }
  return alpha;
}

// Multiplies the warp's rows of an accumulator (64 columns) with a factor per lane.
__device__ __forceinline__ void fwd_rescale(uint32_t o_addr, float alpha) {
#pragma unroll 1
  for (int part = 0; part < 4; ++part) {
    uint32_t orow[16];
    tmem_ld_32x32b_x16(o_addr + 16 * part, orow);
    tc_wait_ld();
#pragma unroll
    for (int j = 0; j < 16; ++j) orow[j] = __float_as_uint(__uint_as_float(orow[j]) * alpha);
    tmem_st_32x32b_x16(o_addr + 16 * part, orow);
  }
}

// Work item w -> (batch, head, query block).  Late (long, if causal) query blocks of a head come first, but where a
// CTA has few items (kFrontRounds at most) the first kFrontRows query blocks of every head come before all
// others: those of global tokens keep everything, and a kernel ends with the CTA that draws a long item last.
// Where they are short it makes no difference.  (With many items it matters less, and heads beside one another
// would share the L2 cache.)  B200, public calls, with / without: two heads, 30 % of the blocks, the first 8 query
// blocks full, N = 9600 31.8 / 46.8 us, N = 14976 63.1 / 84.0; all rows alike, a tenth, 15.3 / 15.4 and 25.6 / 25.3;
// N = 6400, 4 heads, causal, a quarter 17.1 / 17.2.  All heads' blocks in turn: 15.8 and 26.4.
// (An order by length, which every CTA has to work out: 41.3 and 65.5; all rows alike 19.3 and 35.7.  That one
// also found long rows elsewhere, 8 evenly spread at N = 9600: 41.5, with this order 46.0.  Columns of items, the
// longest first, read at every draw: 33.3 there, all rows alike 18.5 and 29.0.)
struct FwdItem {
  int b, h, mb;
};
__device__ __forceinline__ FwdItem fwd_item(int w, const FwdParams& p) {
  const int late = w - p.front_items;  // >= 0: not one of the front ones
  const int each = late < 0 ? p.front : p.nrows - p.front, bh = (late < 0 ? w : late) / each;
  FwdItem it;
  it.mb = p.row_begin + (late < 0 ? w - bh * each : p.nrows - 1 - (late - bh * each));
  it.b = bh / p.H;
  it.h = bh - it.b * p.H;
  return it;
}

// Mask row of a work item (mask mode); list_*_stride are 0 for a broadcast axis and 1 otherwise.
__device__ __forceinline__ const uint8_t* fwd_mask_row(const FwdItem& it, const FwdParams& p) {
  return p.block + (it.b * p.list_b_stride) * p.ms0 + (it.h * p.list_h_stride) * p.ms1 +
         static_cast<int64_t>(it.mb) * p.ms2;
}

// Lists the key blocks of work item w into list buffer `at` (one warp), with the item itself.
template <bool kElementMask>
__device__ __forceinline__ void fwd_list_item(FwdSmem* sm, const FwdParams& p, int w, int at,
                                              int lane) {
  const FwdItem it = fwd_item(w, p);
  uint16_t* cols = sm->cols[at];
  int n_tiles = 0;
  if (p.block != nullptr) {
    // mask mode: the kept blocks of mask row (b, h, mb) in order
    const uint8_t* mrow = fwd_mask_row(it, p);
    if (p.ms3 == 1) {
      // 128 columns per pass, four per lane: a 4-byte word of memory, the row beginning in the first one.  (So the
      // first and the last word may reach three bytes beyond the row, and beyond the caller's mask; an aligned
      // word never reaches beyond what was allocated, and the C interface says so.)  The words of four passes are
      // on their way at a time, so that a row costs one round trip to memory up to N = 32,000
      const int off = static_cast<int>(reinterpret_cast<uintptr_t>(mrow) & 3u), words = (off + p.nb + 3) >> 2;
      const uint32_t* word = reinterpret_cast<const uint32_t*>(mrow - off) + lane;
      uint32_t next[4] = {0u, 0u, 0u, 0u};
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (32 * j + lane < words) next[j] = __ldg(word + 32 * j);
#pragma unroll 1
      for (int i = lane, col = 4 * lane - off; i - lane < words; i += 32, col += 128, word += 32) {
        uint32_t v = next[0];
#pragma unroll
        for (int j = 0; j < 3; ++j) next[j] = next[j + 1];
        next[3] = 0u;
        if (i + 128 < words) next[3] = __ldg(word + 128);
        // bytes of other rows at both ends
        if (col < 0) v &= 0xffffffffu << (8 * off);
        if (i == words - 1) v &= 0xffffffffu >> (8 * (col + 4 - p.nb));
        uint16_t* out = cols + n_tiles;
        uint32_t kept[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          kept[j] = __ballot_sync(0xffffffffu, (v & (0xffu << (8 * j))) != 0);
          out += __popc(kept[j] & ((1u << lane) - 1u));
          n_tiles += __popc(kept[j]);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t byte = v >> (8 * j) & 0xffu;
          if (byte != 0) *out++ = static_cast<uint16_t>((col + j) | (kElementMask && byte == 2 ? kColPartial : 0));
        }
      }
    } else {
#pragma unroll 1
      for (int c0 = 0; c0 < p.nb; c0 += 32) {
        const int c = c0 + lane, byte = c < p.nb ? mrow[c * p.ms3] : 0;
        const unsigned bal = __ballot_sync(0xffffffffu, byte != 0);
        if (byte != 0)
          cols[n_tiles + __popc(bal & ((1u << lane) - 1u))] =
              static_cast<uint16_t>(c | (kElementMask && byte == 2 ? kColPartial : 0));
        n_tiles += __popc(bal);
      }
    }
  } else {
    const int64_t li =
        static_cast<int64_t>(it.b * p.list_b_stride + it.h * p.list_h_stride) * p.nb + it.mb;
    const int beg = __ldg(p.row_ptr + li);
    n_tiles = __ldg(p.row_ptr + li + 1) - beg;
#pragma unroll 1
    for (int jj = lane; jj < n_tiles; jj += 32) {
      const int e = __ldg(p.col_idx + beg + jj);
      cols[jj] = static_cast<uint16_t>(
          (e & kColIndex) | (kElementMask && (e & BSA_LIST_PARTIAL_FLAG) ? kColPartial : 0));
    }
  }
  if (lane == 0) sm->item[at] = make_int4(it.b, it.h, it.mb, n_tiles);
}

// A role's walk over the items: waits for the next one to be published and reads its header.
struct FwdWalk {
  int at = 0, ph = 0;  // list buffer, phase of its barrier
  int4 it;             // batch (< 0: no more work), head, query block, tile count
  // The first item is published after the end of the kernel before, which may take any time (one that lets its
  // successor in early and then waits for a peer, say): a role's limited waits begin when that has ended.
  __device__ __forceinline__ FwdWalk() { grid_dependency_wait(); }
  __device__ __forceinline__ bool wait(FwdSmem* sm) {
    if (!mbar_wait_warp_item(smem_u32(&sm->list_full[at]), ph, &sm->abort_flag)) return false;
    it = sm->item[at];
    return true;
  }
  __device__ __forceinline__ void next() {
    if (++at == kLists) { at = 0; ph ^= 1; }
  }
};

// kElementMask: the instantiation that applies a dense mask inside the tiles marked partial; the
// plain one carries none of that code.
template <bool kBf16, bool kElementMask>
__global__ void __launch_bounds__(kFwdThreads, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                const __grid_constant__ CUtensorMap tm_v, const FwdParams p) {
  // (Aligned by declaration: every address in it is a constant then.  Rounded up at run time, all roles carried a
  // base and added to it at every barrier: N = 17536, a tenth, one head 19.15 -> 17.94 us, 8 heads 107.6 -> 102.5;
  // everything listed 108.9 -> 104.0.)
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  FwdSmem* sm = reinterpret_cast<FwdSmem*>(smem_raw);

  // (the lister's warps come first: the first list is what all others wait for)
  const int hw_warp = uniform_warp_index(), warp = hw_warp >= 4 ? hw_warp - 4 : hw_warp + 16;
  const int lane = threadIdx.x & 31;
  const int stride = gridDim.x;
  const int n2 = p.items - stride;  // items beyond the first round

  // ---- set-up ----
  if (warp == 0) {
    mbar_init_warp(sm->setup_go, 2, 1, lane);
    mbar_init_warp(sm->q_free, 2, 1, lane);
    mbar_init_warp(sm->o_full, 2, 1, lane);
    mbar_init_warp(sm->stats_full, kLists, kSoftmaxWarps, lane);
    mbar_init_warp(sm->o_free, 2, 4, lane);  // one arrival per write-out warp
    mbar_init_warp(sm->k_full, kKStages, 1, lane);
    mbar_init_warp(sm->k_empty, kKStages, 1, lane);
    mbar_init_warp(sm->s_full, 2 * kSlots, 1, lane);
    mbar_init_warp(sm->p_full, kSlots, kTeamWarps + 1, lane);
    mbar_init_warp(sm->pv_done, kSlots, 1, lane);
    mbar_init_warp(sm->list_full, kLists, 1, lane);
    mbar_init_warp(sm->list_free, kLists, 8, lane);  // two producers, two issuers, four write-out warps
    if (lane == 0) sm->abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == kSWarp) {
    tmem_alloc(smem_u32(&sm->tmem_base), kFwdTmemCols);
    tmem_relinquish();
  }
  if (warp == kProducerWarp && lane == 0) {
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_v);
  }
  tc_fence_before();
  if (warp == kListerWarp) {
    // Lists the CTA's first item while the others set up and get as far as their first barrier.  (With the list
    // from the lister's own loop, behind the jumps to the roles and instructions that no cache held yet, the
    // first tiles were asked for 2,200 cycles later.)  Everything that touches memory that an earlier
    // kernel may use comes after this.
    grid_dependency_wait();
    if (p.successor_early) grid_dependents_launch();
    fwd_list_item<kElementMask>(sm, p, blockIdx.x, 0, lane);
    named_barrier_sync(1, kFwdThreads);  // the barriers are there
    if (lane == 0) mbar_arrive(smem_u32(&sm->list_full[0]));
  } else {
    named_barrier_arrive(1, kFwdThreads);
    named_barrier_sync(3, kFwdThreads - 32);
  }
  tc_fence_after();
  const uint32_t tmem = sm->tmem_base;
  volatile int* abort_flag = &sm->abort_flag;

  // 640 threads are launched with 96 registers: the softmax warps, which hold 64 logits and 128 probabilities each,
  // take what the others do without (2 x 160 + 40 + 88 + 32 = 5 x 96).  The write-out needs its 88: with 80 or 72 short
  // lists are 1 or 2 % slower.
  if (warp >= kSoftmaxWarps && warp < kSoftmaxWarps + 4) {
  give_registers<kIssuerRegs>();
  if (warp == kProducerWarp) {
    // =========================== K producer ===========================
    bool ok = true;
    // Loads Q and the K tiles of the listed key blocks from the list the lister published, and
    // tells the lister when to set up the next item: kGoBefore supersteps of loads before the end, so that
    // a CTA draws its next item when it is about to need it.  (Set up as soon as an item begins: four heads,
    // N = 6400, causal, a quarter of the blocks 19.3 us against 18.6, the same with many items.  Items
    // beyond the first round longest first, which every CTA had to work out for itself: 22.0 us; and with
    // one head, N = 17536, a tenth: 20.2 us against 19.2.)
    int ks = 0, kph = 1;  // ring position, parity to wait for
    int qi = 0;           // non-empty items so far (Q buffer position)
    FwdWalk walk;
#pragma unroll 1
    for (int i = 0; ok; ++i, walk.next()) {
      const int par = i & 1;
      ok = walk.wait(sm);
      if (!ok || walk.it.x < 0) break;  // (no more work)
      const int n_tiles = walk.it.w;
      const uint16_t* cols = sm->cols[walk.at];
      const int n_super = (n_tiles + 3) >> 2;
      const int u_go = max(n_super - kGoBefore, 0);
      if (n_super == 0 && lane == 0) mbar_arrive(smem_u32(&sm->setup_go[par]));
      // One lane per tile issues its load: a single thread can start a tile load only every couple
      // of hundred cycles.
#pragma unroll 1
      for (int u = 0; u < n_super; ++u) {
        if (u == u_go && lane == 0) mbar_arrive(smem_u32(&sm->setup_go[par]));
        const int nt = min(4, n_tiles - 4 * u);
        const int qpar = qi & 1;
        // (the item before the previous one is through with its Q as long as this one lasts)
        ok = mbar_wait_warp2(smem_u32(&sm->k_empty[ks]), kph, smem_u32(&sm->q_free[qpar]), ((qi >> 1) & 1) ^ 1);
        if (!ok) break;
        const uint32_t bar = smem_u32(&sm->k_full[ks]);
        if (lane == 0) {
          mbar_expect_tx(bar, kTileBytes * (nt + (u == 0)));
          if (u == 0) tma_load_4d(smem_u32(sm->q[qpar]), &tm_q, bar, 0, walk.it.z * 64, walk.it.y, walk.it.x);
        }
        __syncwarp();
        if (lane < nt) {  // in shared memory a, c, b, d; only a, b: next to each other
          const int at = nt > 2 ? ((lane & 1) << 1) | (lane >> 1) : lane;
          tma_load_4d(smem_u32(sm->k[ks][at]), &tm_k, bar, 0,
                      static_cast<int>(cols[4 * u + lane] & kColIndex) * 64, walk.it.y, walk.it.x);
        }
        if (++ks == kKStages) { ks = 0; kph ^= 1; }
      }
      if (n_super > 0) ++qi;
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&sm->list_free[walk.at]));
    }
    if (!ok) fwd_give_up(sm, p.status, kFailProducer);
  } else if (warp == kVProducerWarp) {
    // =========================== V producer ===========================
    // Loads the V tiles of the listed key blocks, one lane per tile; a warp of its own, so that
    // waiting for a free V stage (P V complete) never holds back the K tiles of a later superstep.
    // Superstep g has the pairs 2 g and 2 g + 1 of the ring, whether it needs both or not: they were those
    // of supersteps g - 3 and g - 2.  Its tiles land on the barrier that P arrives on, so that P V has
    // one wait (a look at a barrier that is long complete costs its issuer 150 cycles and more).
    bool ok = true;
    int vs = 0, slot = 0, ph = 1;
    FwdWalk walk;
#pragma unroll 1
    for (; ok; walk.next()) {
      ok = walk.wait(sm);
      if (!ok || walk.it.x < 0) break;  // (no more work)
      const int n_tiles = walk.it.w;
      const uint16_t* cols = sm->cols[walk.at];
#pragma unroll 1
      for (int u = 0; 4 * u < n_tiles; ++u) {
        const int nt = min(4, n_tiles - 4 * u);
        const int at = lane < 2 ? vs : vs + 1 < kVStages ? vs + 1 : 0;
        // whole pairs: a tile that does not exist is read behind the last row, which gives zeros
        const int n_load = (nt + 1) & ~1;
        const int row = lane < nt ? static_cast<int>(cols[4 * u + lane] & kColIndex) * 64 : p.N;
        const uint32_t dst = smem_u32(sm->v[at][lane & 1]), bar = smem_u32(&sm->p_full[slot]);
        // (for the first users these ask for the phase before the first one, which counts as complete)
        ok = mbar_wait_warp(smem_u32(&sm->pv_done[slot]), ph);
        if (!ok) break;
        if (lane == 0) mbar_expect_tx(bar, kTileBytes * n_load);
        __syncwarp();
        if (lane < 2) tma_load_4d(dst, &tm_v, bar, 0, row, walk.it.y, walk.it.x);
        const int next = slot + 1 < kSlots ? slot + 1 : 0;
        ok = mbar_wait_warp(smem_u32(&sm->pv_done[next]), next > 0 ? ph : ph ^ 1);
        if (!ok) break;
        if (lane >= 2 && lane < n_load) tma_load_4d(dst, &tm_v, bar, 0, row, walk.it.y, walk.it.x);
        vs += 2;
        if (vs >= kVStages) vs -= kVStages;
        slot = next;
        if (slot == 0) ph ^= 1;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&sm->list_free[walk.at]));
    }
    if (!ok) fwd_give_up(sm, p.status, kFailProducer);
  } else if (warp == kSWarp) {
    // =========================== S issuer ===========================
    constexpr uint32_t idesc_s4 = umma_idesc(kBf16, 0, 0, 64, 256);
    constexpr uint32_t idesc_s2 = umma_idesc(kBf16, 0, 0, 64, 128);
    const bool leader = elect_one();
    const uint64_t desc_q0 = smem_desc_sw128(smem_u32(sm->q[0]), 16, 1024);
    const uint64_t desc_k0 = smem_desc_sw128(smem_u32(sm->k[0][0]), 16, 1024);
    constexpr uint64_t kTileDesc = kTileBytes >> 4;  // one tile further, in descriptor units
    const int k_steps = p.D >> 4;
    bool ok = true;
    int ks = 0, kph = 0, qi = 0;
    int slot = 0, slot_ph = 1, bar_s = 0;  // (bar_s: superstep number mod 2 kSlots)
    FwdWalk walk;
#pragma unroll 1
    for (; ok; walk.next()) {
      ok = walk.wait(sm);
      if (!ok || walk.it.x < 0) break;  // (no more work)
      const int n_tiles = walk.it.w;
      const int n_super = (n_tiles + 3) >> 2;
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&sm->list_free[walk.at]));
      if (n_super == 0) continue;
      const int qpar = qi & 1;
      const uint64_t desc_q = desc_q0 + static_cast<uint64_t>(qpar) * kTileDesc;
#pragma unroll 1
      for (int u = 0; u < n_super; ++u) {
        // the slot's previous user, three supersteps ago, must have had its P V completed (for the
        // first users this asks for the phase before the first one, which counts as complete)
        ok = mbar_wait_warp_in_turn(smem_u32(&sm->k_full[ks]), kph, smem_u32(&sm->pv_done[slot]), slot_ph);
        if (!ok) break;
        tc_fence_after();
        if (leader) {
          // an odd number of tiles multiplies with whatever the rest of the stage holds: those
          // logits are nobody's
          const uint32_t d = tmem + 128 * slot;
          const uint64_t desc_k = desc_k0 + static_cast<uint64_t>(ks * 4) * kTileDesc;
          const uint32_t idesc = n_tiles - 4 * u > 2 ? idesc_s4 : idesc_s2;
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)
            if (kk < k_steps) umma_ws_ss(d, desc_q + 2 * kk, desc_k + 2 * kk, idesc, kk > 0);
          tc_commit(smem_u32(&sm->s_full[bar_s]));
          tc_commit(smem_u32(&sm->k_empty[ks]));
          if (u == n_super - 1) tc_commit(smem_u32(&sm->q_free[qpar]));
        }
        if (++ks == kKStages) { ks = 0; kph ^= 1; }
        if (++slot == kSlots) { slot = 0; slot_ph ^= 1; }
        if (++bar_s == 2 * kSlots) bar_s = 0;
      }
      ++qi;
    }
    if (!ok) fwd_give_up(sm, p.status, kFailMma);
  } else if (warp == kPvWarp) {
    // =========================== P V issuer ===========================
    constexpr uint32_t idesc_pv = umma_idesc(kBf16, 0, 1, 64, 128);  // P (TMEM) x V (MN-major)
    const bool leader = elect_one();
    const uint64_t desc_v0 = smem_desc_sw128(smem_u32(sm->v[0][0]), 8192, 1024);
    bool ok = true;
    int vs = 0, slot = 0, slot_ph = 0, team = 0;
    FwdWalk walk;
#pragma unroll 1
    for (int i = 0; ok; ++i, walk.next()) {
      const int par = i & 1;
      ok = walk.wait(sm);
      if (!ok || walk.it.x < 0) break;  // (no more work)
      const int n_tiles = walk.it.w;
      const int n_super = (n_tiles + 3) >> 2;
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&sm->list_free[walk.at]));
      // the accumulators are free once the previous item has been read out; the softmax warps
      // meanwhile work ahead
      if (i >= 1)
        ok = mbar_wait_warp(smem_u32(&sm->o_free[par ^ 1]), ((i - 1) >> 1) & 1);
      if (!ok) break;
      if (n_super == 0) {
        if (leader) mbar_arrive(smem_u32(&sm->o_full[par]));
        continue;
      }
#pragma unroll 1
      for (int u = 0; u < n_super && ok; ++u, team ^= 1) {
        const int nt = min(4, n_tiles - 4 * u);
        const int vs1 = vs + 1 < kVStages ? vs + 1 : 0;
        ok = mbar_wait_warp(smem_u32(&sm->p_full[slot]), slot_ph);  // P and V
        if (!ok) break;
        tc_fence_after();
        // Tiles a and b have their P in columns [0, 32) of the slot, a in lanes 0..63 and b in lanes
        // 64..127; c and d in columns [32, 64).  The team's first product of an item starts its accumulator
        // afresh, in all lanes.  (N = 17536, everything listed 114.1 -> 110.8 us, 8 heads, a tenth 111.4 -> 109.1,
        // bf16 N = 32000, 32 heads, a tenth 1288 -> 1249, against a product for each tile; D = 32, where those are
        // 32 columns wide, 49.3 -> 49.5.)
        const uint32_t o_acc = tmem + kTmemO + 64 * team;
        if (leader) {
#pragma unroll
          for (int t = 0; t < 4; t += 2) {
            if (t >= nt) break;
            const uint32_t p_cols = tmem + 128 * slot + 16 * t;
            const uint64_t desc_v = desc_v0 + static_cast<uint64_t>((t < 2 ? vs : vs1) * 2) * (kTileBytes >> 4);
            const uint32_t started = u > 1 || t > 1;
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
              umma_ws_ts(o_acc, p_cols + 8 * kk, desc_v + 128 * kk, idesc_pv, started | (kk > 0));
          }
        }
        if (leader) {
          tc_commit(smem_u32(&sm->pv_done[slot]));
          if (u == n_super - 1) tc_commit(smem_u32(&sm->o_full[par]));
        }
        vs += 2;
        if (vs >= kVStages) vs -= kVStages;
        if (++slot == kSlots) { slot = 0; slot_ph ^= 1; }
      }
    }
    if (!ok) fwd_give_up(sm, p.status, kFailMma);
  }
  } else if (warp < kSoftmaxWarps) {
    // =========================== softmax ===========================
    take_registers<kSoftmaxRegs>();
    const int team = warp >> 2;
    const int quarter = warp & 3;     // TMEM lane quarter this warp may touch
    const int half = quarter >> 1;    // lanes 0..63 own tiles a, c of a superstep, 64..127 b, d
    const int lane_row = quarter * 32 + lane;  // TMEM lane
    const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
    const uint32_t o_addr = tmem + lane_base + kTmemO + 64 * team;
    const float c = p.scale_log2;
    const bool want_max = p.rowmax != nullptr;
    bool ok = true;
    int g = 0;        // supersteps of earlier items; this team takes those with g % 2 == team
    int next = team;  // its next one, with the slot next % kSlots and the barrier next % (2 kSlots)
    int slot = team, bar_s = team, bar_ph = 0;
    FwdWalk walk;
#pragma unroll 1
    for (int i = 0; ok; ++i, walk.next()) {
      ok = walk.wait(sm);
      if (!ok || walk.it.x < 0) break;  // (no more work)
      const int n_tiles = walk.it.w;
      const int n_super = (n_tiles + 3) >> 2;
      const uint16_t* cols = sm->cols[walk.at];
      float m_ref = -INFINITY, m_true = -INFINITY, l = 0.f;
      // this lane's row of the element-level mask, if there is one
      const uint8_t* mask_row = nullptr;
      if constexpr (kElementMask)
        mask_row = p.dense + walk.it.x * p.ds0 + walk.it.y * p.ds1 +
                   static_cast<int64_t>(walk.it.z * 64 + (quarter & 1) * 32 + lane) * p.ds2;

#pragma unroll 1
      for (; next < g + n_super; next += 2) {
        const int u = next - g;
        const uint32_t s_addr = tmem + lane_base + 128 * slot;
        const int mine = n_tiles - 4 * u - half;  // > 0: this lane's first tile exists, > 2: both
        ok = mbar_wait_warp(smem_u32(&sm->s_full[bar_s]), bar_ph);
        if (!ok) break;
        tc_fence_after();
        // The row maximum is looked up only where it is needed: when the caller wants it, and with
        // element masks as long as one of the warp's rows has nothing yet.  The first superstep of the
        // team takes the maximum of the 32 logits that it holds anyway for a reference, and logits are
        // exponentiated against that as it is; a row whose sum shows that it was too low (or not finite)
        // makes the warp do the superstep again with the maximum of all its logits.  S is still in tensor
        // memory then: P goes over it last.
        bool with_max = want_max;
        if constexpr (kElementMask) with_max |= u >= 2 && __any_sync(0xffffffffu, m_ref == -INFINITY);
        if (mine > 0) {
          const bool two = mine > 2;  // both tiles exist (warp-uniform)
          const auto masked = [&](uint32_t* sr, int col) {
            if constexpr (kElementMask) {
              const uint16_t entry = cols[4 * u + (col >> 6) * 2 + half];
              if (entry & kColPartial)
                mask_chunk(sr, mask_row + (entry & kColIndex) * 64 + (col & 32));
            }
          };
          uint32_t pk[64];
          float sum, slack = kRescaleThreshold;
#pragma unroll 1
          while (true) {
            uint32_t sa[32], sb[32];
            if (with_max) {
              float zmax = -INFINITY;
#pragma unroll 1
              for (int col = 0; col < (two ? 128 : 64); col += 32) {
                tmem_ld_32x32b_x32(s_addr + col, sa);
                tc_wait_ld();
                masked(sa, col);
                zmax = fmaxf(zmax, max_chunk(sa));
              }
              const float alpha = fwd_new_max(zmax * c, slack, m_ref, m_true, l);
              if (__any_sync(0xffffffffu, alpha != 1.f)) {
                // the previous product of this team, two supersteps ago, must be in O
                const int prev = slot == 2 ? 0 : slot + 1;  // (slot - 2) % 3
                ok = mbar_wait_warp(smem_u32(&sm->pv_done[prev]),
                                    static_cast<uint32_t>((next - 2) / kSlots) & 1u);
                if (!ok) break;
                tc_fence_after();
                fwd_rescale(o_addr, alpha);
              }
            }
            uint64_t l0 = pack_f32x2(0.f, 0.f), l1 = l0;
            tmem_ld_32x32b_x32(s_addr, sa);
            tmem_ld_32x32b_x32(s_addr + 32, sb);
            tc_wait_ld();
            masked(sa, 0);
            masked(sb, 32);
            if (u < 2 && !with_max) {
              m_ref = max_chunk(sa) * c;
              if (kElementMask && __any_sync(0xffffffffu, m_ref == -INFINITY)) {
                with_max = true;  // a row has nothing among those 32
                m_ref = -INFINITY;
                continue;
              }
            }
            const float neg_m = (kElementMask && m_ref == -INFINITY) ? 0.f : -m_ref;
            exp_chunk<kBf16>(sa, c, neg_m, pk, l0, l1);
            if (two) {
              tmem_ld_32x32b_x32(s_addr + 64, sa);
              exp_chunk<kBf16>(sb, c, neg_m, pk + 16, l0, l1);
              tmem_ld_32x32b_x32(s_addr + 96, sb);
              tc_wait_ld();
              masked(sa, 64);
              masked(sb, 96);
              exp_chunk<kBf16>(sa, c, neg_m, pk + 32, l0, l1);
              exp_chunk<kBf16>(sb, c, neg_m, pk + 48, l0, l1);
            } else {
              exp_chunk<kBf16>(sb, c, neg_m, pk + 16, l0, l1);
#pragma unroll
              for (int j = 32; j < 64; ++j) pk[j] = 0u;
            }
            float a0, a1;
            unpack_f32x2(add_f32x2(l0, l1), a0, a1);
            sum = a0 + a1;
            if (with_max || !__any_sync(0xffffffffu, !(sum <= kMaxRowSum))) break;
            with_max = true;
            // The maximum becomes the reference however little it lies above it: many logits a few units
            // above would fail the test in every later superstep of the row as well (N = 17536, everything
            // listed, keys from the second eighth on 6.3 above: 194 us, 107 with the move; 102 if level).
            slack = 0.f;
            if (u < 2) m_ref = -INFINITY;  // nothing is summed against it yet
          }
          if (!ok) break;
          l += sum;
          // this lane's first tile in columns [0, 32) of the slot, its second one in [32, 64); zeros for one that
          // does not exist while the other lane half has it
          tmem_st_32x32b_x32(s_addr, pk);
          if (n_tiles - 4 * u > 2) tmem_st_32x32b_x32(s_addr + 32, pk + 32);
        } else {
          uint32_t zero[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) zero[j] = 0u;
          tmem_st_32x32b_x32(s_addr, zero);
        }
        tc_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&sm->p_full[slot]));
        slot = slot >= 1 ? slot - 1 : kSlots - 1;  // (slot + 2) % 3
        bar_s += 2;
        if (bar_s >= 2 * kSlots) { bar_s -= 2 * kSlots; bar_ph ^= 1; }
      }
      if (!ok) break;
      g += n_super;

      // publish this item's (m, l) of the warp's lanes (that this item is there means that the one that had its list
      // buffer has been written out)
      sm->mref[walk.at][team][lane_row] = m_ref;
      sm->lsum[walk.at][team][lane_row] = l;
      if (want_max) sm->mtrue[walk.at][team][lane_row] = m_true;
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&sm->stats_full[walk.at]));
    }
    if (!ok) fwd_give_up(sm, p.status, kFailSoftmax);
  } else if (warp < kSoftmaxWarps + 8) {
    // =========================== write-out ===========================
    // Merges the four partial results of every query row (first / second team of the item x lanes
    // r / r+64).  A warp reads both accumulators of its own lanes from TMEM; lanes 64..127 hand
    // their weighted rows to each other through shared memory, 16 columns at a time.  Each time
    // takes two named barriers, also after a give-up, the second one with the give-up vote (role_leaves); a warp
    // that is told that there is no more work comes to both before it leaves.
    give_registers<kWriteRegs>();
    const int quarter = warp & 3;  // lane quarter a warp may touch = its index mod 4
    bool ok = true;
    const int half = quarter >> 1;
    const int r_blk = (quarter & 1) * 32 + lane;  // row of the query block
    const uint32_t o_lanes = tmem + (static_cast<uint32_t>(quarter * 32) << 16) + kTmemO;
    int g = 0;  // supersteps of earlier items
    FwdWalk walk;
#pragma unroll 1
    for (int i = 0;; ++i) {
      const int par = i & 1;
      if (ok) ok = mbar_wait_warp_item(smem_u32(&sm->list_full[walk.at]), walk.ph, abort_flag);
      walk.it = ok ? sm->item[walk.at] : make_int4(0, 0, 0, 0);
      if (walk.it.x < 0) {  // no more work
        named_barrier_sync(2, 128);
        role_leaves(2, 128, false);
        break;
      }
      const int n_tiles = walk.it.w;
      if (ok) ok = mbar_wait_warp_item(smem_u32(&sm->stats_full[walk.at]), walk.ph, abort_flag);
      // The weights of the four partial results need the statistics only, which the softmax warps
      // publish before the item's last P V is complete.
      const int t0 = g & 1;  // the team with the item's first superstep
      g += (n_tiles + 3) >> 2;
      float m_all = -INFINITY, l_all = 0.f, mt = -INFINITY, w0 = 0.f, w1 = 0.f;
      if (ok) {
        // (A lane and team that has nothing has m = -inf and l = 0, hence weight 0; if none has anything, against a
        // zero in place of the maximum.  Everything between two items is kept short: 50 KB of code against an
        // instruction cache of 32 KB on an SM.  With a select at every use here, and masks at every word of a row in
        // the lister: N = 17536, a tenth 17.87 / 17.70 us, 24 heads of N = 4160, D = 32 45.4 / 44.9.)
        const float *m_at = &sm->mref[walk.at][t0][r_blk], *l_at = &sm->lsum[walk.at][t0][r_blk];
        const int other = t0 ? -128 : 128;  // the other team's
        const float m0 = m_at[0], m1 = m_at[other], m2 = m_at[64], m3 = m_at[other + 64];
        m_all = fmaxf(fmaxf(m0, m1), fmaxf(m2, m3));
        const float top = m_all == -INFINITY ? 0.f : m_all;
        const float e0 = ex2_approx(m0 - top), e1 = ex2_approx(m1 - top), e2 = ex2_approx(m2 - top), e3 = ex2_approx(m3 - top);
        l_all = e0 * l_at[0];
        l_all += e1 * l_at[other];
        l_all += e2 * l_at[64];
        l_all += e3 * l_at[other + 64];
        if (p.rowmax) {
          const float* t_at = &sm->mtrue[walk.at][0][r_blk];
          mt = fmaxf(fmaxf(t_at[0], t_at[64]), fmaxf(t_at[128], t_at[192]));
        }
        const float inv = l_all > 0.f ? 1.f / l_all : 0.f;
        w0 = (half ? e2 : e0) * inv;
        w1 = (half ? e3 : e1) * inv;
      }
      if (ok) ok = mbar_wait_warp(smem_u32(&sm->o_full[par]), (i >> 1) & 1);
      tc_fence_after();
      // A team's accumulator holds sums of this item only if the item has a superstep for it.
      const bool live0 = n_tiles > 0, live1 = n_tiles > 4;
      const uint64_t w0w0 = pack_f32x2(w0, w0), w1w1 = pack_f32x2(w1, w1);
      const int row = walk.it.z * 64 + r_blk;
      uint16_t* dst = static_cast<uint16_t*>(p.o) + walk.it.x * p.o_sb + walk.it.y * p.o_sh +
                      static_cast<int64_t>(row) * p.o_sn;
      bool any_failed = false;
      // Lanes 0..63 finish columns [0, 32) of their rows, lanes 64..127 columns [32, 64) of the same
      // rows, 16 columns at a time; each hands the other its sums of the other columns.
#pragma unroll 1
      for (int part = 0; part < 2; ++part) {
        uint64_t keep[8];
        if (ok) {
          uint64_t send[8];
          const uint32_t at_send = o_lanes + 32 * (half ^ 1) + 16 * part, at_keep = o_lanes + 32 * half + 16 * part;
          const auto sum = [&](uint32_t cols, uint64_t* acc) {
            uint32_t a0[16], a1[16];
            tmem_ld_32x32b_x16(cols + 64 * t0, a0);
            tmem_ld_32x32b_x16(cols + 64 * (t0 ^ 1), a1);
            tc_wait_ld();
#pragma unroll
            for (int j = 0; j < 8; ++j)
              acc[j] = mul_f32x2(pack_f32x2(__uint_as_float(a0[2 * j]), __uint_as_float(a0[2 * j + 1])), w0w0);
            if (live1) {
#pragma unroll
              for (int j = 0; j < 8; ++j)
                acc[j] = fma_f32x2(pack_f32x2(__uint_as_float(a1[2 * j]), __uint_as_float(a1[2 * j + 1])), w1w1, acc[j]);
            } else if (!live0) {
#pragma unroll
              for (int j = 0; j < 8; ++j) acc[j] = 0ull;
            }
          };
          sum(at_send, send);
          sum(at_keep, keep);
          ulonglong2* out = reinterpret_cast<ulonglong2*>(sm->xfer[half][r_blk]);
#pragma unroll
          for (int j = 0; j < 4; ++j) out[j] = make_ulonglong2(send[2 * j], send[2 * j + 1]);
          if (part == 1) {
            // Accumulators, statistics and the item's header are in registers now: the next item may
            // use them, while this one is still being merged and stored.
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
              mbar_arrive(smem_u32(&sm->o_free[par]));
              mbar_arrive(smem_u32(&sm->list_free[walk.at]));
            }
          }
        }
        named_barrier_sync(2, 128);
        const int col = 32 * half + 16 * part;
        if (ok && col < p.D) {
          const ulonglong2* in = reinterpret_cast<const ulonglong2*>(sm->xfer[half ^ 1][r_blk]);
          uint32_t pkd[8];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const ulonglong2 x = in[j];
            float f0, f1, f2, f3;
            unpack_f32x2(add_f32x2(keep[2 * j], x.x), f0, f1);
            unpack_f32x2(add_f32x2(keep[2 * j + 1], x.y), f2, f3);
            pkd[2 * j] = pack_2x16<kBf16>(f0, f1);
            pkd[2 * j + 1] = pack_2x16<kBf16>(f2, f3);
          }
          // whole 32-byte sectors when the rows start on such boundaries
          if (p.wide_stores) {
            st_global_v8(dst + col, pkd);
          } else {
            *reinterpret_cast<uint4*>(dst + col) = make_uint4(pkd[0], pkd[1], pkd[2], pkd[3]);
            *reinterpret_cast<uint4*>(dst + col + 8) = make_uint4(pkd[4], pkd[5], pkd[6], pkd[7]);
          }
        }
        // xfer may be overwritten now; all four warps leave together if any gave up
        any_failed = role_leaves(2, 128, !ok);
        if (any_failed) break;
      }
      if (ok && half == 0) {
        const int64_t ri = (static_cast<int64_t>(walk.it.x) * p.H + walk.it.y) * p.N + row;
        if (p.lse2) p.lse2[ri] = l_all > 0.f ? m_all + lg2_approx(l_all) : -INFINITY;
        if (p.rowmax) p.rowmax[ri] = mt;
      }
      if (any_failed) break;
      walk.next();
    }
    if (!ok) fwd_give_up(sm, p.status, kFailOut);
  } else {
  give_registers<kListerRegs>();
  if (warp == kListerWarp) {
    // =========================== lister ===========================
    // Sets up item i+1 when the K producer says so during item i, or publishes that there is none; a wait that gives
    // up leaves ok = false and nothing published.
    bool ok = true;
    bool terminal = p.ticket == nullptr;  // drew a ticket past the end (or draws none)
    int w = blockIdx.x, at = 0;
#pragma unroll 1
    for (int i = 0; w < p.items; ++i) {
      ok = mbar_wait_warp_item(smem_u32(&sm->setup_go[i & 1]), (i >> 1) & 1, abort_flag);
      if (!ok) break;
      // the next ticket when items are handed out dynamically, else a fixed stride
      if (p.ticket != nullptr) {
        int t = 0;
        if (lane == 0) {
          t = atomicAdd(p.ticket, 1);
          // every CTA draws until its first ticket past the end, so the launch draws exactly
          // `items` tickets in all; whoever draws the last one leaves the counter at zero
          if (t == p.items - 1) atomicExch(p.ticket, 0);
        }
        t = __shfl_sync(0xffffffffu, t, 0);
        terminal = t >= n2;
        w = stride + t;
      } else {
        w += stride;
      }
      if (++at == kLists) at = 0;
      // the list buffer was that of item i-2
      if (i >= 2) ok = mbar_wait_warp_item(smem_u32(&sm->list_free[at]), ((i - 2) / kLists) & 1, abort_flag);
      if (!ok) break;
      if (w < p.items)
        fwd_list_item<kElementMask>(sm, p, w, at, lane);
      else if (lane == 0)
        sm->item[at].x = -1;
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&sm->list_full[at]));  // release: list and item are visible
    }
    if (!ok) fwd_give_up(sm, p.status, kFailOut);
    if (!terminal && lane == 0) {
      // gave up before the last draw: draw on (without working) until this CTA's first ticket past
      // the end, so that the launch still draws `items` tickets and the counter returns to zero
      int t;
      do {
        t = atomicAdd(p.ticket, 1);
        if (t == p.items - 1) atomicExch(p.ticket, 0);
      } while (t < n2);
    }
  }
  }

  // ---- tear-down: every role arrives here, also after a give-up ----
  // (by the first role that is through with its work, not by warps without one; let in at the beginning, CTAs of the next kernel that wait
  // on free SMs slowed the working ones down by 3 %, let in by the last role they come 0.5 us late)
  if (warp < kSoftmaxWarps + 8 || warp == kListerWarp) grid_dependents_launch();
  tc_fence_before();
  __syncthreads();
  if (warp == kSWarp) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem, kFwdTmemCols);
  }
}

static int launch_fwd(const void* q, const int64_t q_strides[4], const void* k,
                      const int64_t k_strides[4], const void* v, const int64_t v_strides[4], void* o,
                      const int64_t o_strides[4], float* lse2, float* rowmax,
                      const int32_t* row_ptr, const int32_t* col_idx, const uint8_t* block,
                      const int64_t* block_strides, int list_b_stride, int list_h_stride,
                      float sm_scale, int dtype, int B, int H, int N, int D, int row_begin,
                      int row_end, const uint8_t* dense, const int64_t* dense_strides,
                      int32_t* status, int32_t* ticket, void* stream, bool successor_early = false) {
  if (B <= 0 || H <= 0 || N <= 0 || (N % kBlock) != 0 || !head_dim_ok(D))
    return BSA_ERR_BAD_SHAPE;
  if (!(sm_scale >= 0.f)) return BSA_ERR_BAD_SHAPE;  // the row maximum is taken before scaling
  if (dtype != BSA_F16 && dtype != BSA_BF16) return BSA_ERR_BAD_DTYPE;
  if (block == nullptr && (!row_ptr || !col_idx)) return BSA_ERR_BAD_POINTER;
  if (dense != nullptr) {
    // rows of 64 mask bytes are read as four 16-byte words; -inf times a zero scale would be NaN
    if (!dense_strides || !is_aligned(dense, 16)) return BSA_ERR_BAD_POINTER;
    if (dense_strides[3] != 1 || dense_strides[2] <= 0 || (dense_strides[2] % 16) != 0 ||
        dense_strides[0] < 0 || dense_strides[1] < 0 || (dense_strides[0] % 16) != 0 ||
        (dense_strides[1] % 16) != 0)
      return BSA_ERR_BAD_STRIDE;
    if (!(sm_scale > 0.f)) return BSA_ERR_BAD_SHAPE;
  }
  int rc;
  if ((rc = check_qkv_operand(q, q_strides)) != BSA_OK) return rc;
  if ((rc = check_qkv_operand(k, k_strides)) != BSA_OK) return rc;
  if ((rc = check_qkv_operand(v, v_strides)) != BSA_OK) return rc;
  if ((rc = check_qkv_operand(o, o_strides)) != BSA_OK) return rc;
  if ((rc = check_device_sm100()) != BSA_OK) return rc;

  const int nb = N / kBlock;
  if (nb > kFwdMaxTiles) return BSA_ERR_TOO_LARGE;
  if (row_begin < 0 || row_end > nb || row_begin > row_end) return BSA_ERR_BAD_SHAPE;
  const int nrows = row_end - row_begin;
  if (nrows == 0) return BSA_OK;  // an empty share of the rows: nothing to launch
  if (static_cast<int64_t>(B) * H * nrows > 0x7fffffffLL) return BSA_ERR_TOO_LARGE;

  CUtensorMap tm_q, tm_k, tm_v;
  if ((rc = cached_qkv_tmap(&tm_q, q, q_strides, B, H, N, D, dtype)) != BSA_OK) return rc;
  if ((rc = cached_qkv_tmap(&tm_k, k, k_strides, B, H, N, D, dtype)) != BSA_OK) return rc;
  if ((rc = cached_qkv_tmap(&tm_v, v, v_strides, B, H, N, D, dtype)) != BSA_OK) return rc;

  FwdParams prm;
  prm.row_ptr = row_ptr;
  prm.col_idx = col_idx;
  prm.block = block;
  prm.ms0 = block ? block_strides[0] : 0;
  prm.ms1 = block ? block_strides[1] : 0;
  prm.ms2 = block ? block_strides[2] : 0;
  prm.ms3 = block ? block_strides[3] : 0;
  prm.dense = dense;
  prm.ds0 = dense ? dense_strides[0] : 0;
  prm.ds1 = dense ? dense_strides[1] : 0;
  prm.ds2 = dense ? dense_strides[2] : 0;
  prm.o = o;
  prm.o_sb = o_strides[0];
  prm.o_sh = o_strides[1];
  prm.o_sn = o_strides[2];
  prm.lse2 = lse2;
  prm.rowmax = rowmax;
  prm.B = B;
  prm.H = H;
  prm.N = N;
  prm.D = D;
  prm.nb = nb;
  prm.row_begin = row_begin;
  prm.nrows = nrows;
  prm.list_b_stride = list_b_stride;
  prm.list_h_stride = list_h_stride;
  prm.items = B * H * nrows;
  prm.scale_log2 = sm_scale * 1.4426950408889634f;
  prm.status = status;
  prm.ticket = ticket;
  prm.successor_early = successor_early ? 1 : 0;
  prm.wide_stores =
      ((reinterpret_cast<uintptr_t>(o) |
        static_cast<uintptr_t>((o_strides[0] | o_strides[1] | o_strides[2]) * 2)) & 31u) == 0 ? 1 : 0;
  int sms = 0;
  if ((rc = sm_count(&sms)) != BSA_OK) return rc;

  const size_t smem_bytes = sizeof(FwdSmem);
  auto kern = dense != nullptr
                  ? (dtype == BSA_BF16 ? attn_fwd_kernel<true, true> : attn_fwd_kernel<false, true>)
                  : (dtype == BSA_BF16 ? attn_fwd_kernel<true, false> : attn_fwd_kernel<false, false>);
  if ((rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem_bytes, kLaunchRegs)) != BSA_OK)
    return rc;
  // (no more than an eighth of a head's rows: front < nrows)
  prm.front = prm.items > sms && prm.items <= kFrontRounds * sms ? (nrows / 8 < kFrontRows ? nrows / 8 : kFrontRows) : 0;
  prm.front_items = B * H * prm.front;
  const dim3 grid(static_cast<unsigned>(prm.items < sms ? prm.items : sms));  // one CTA per SM
  return launch_dependent(kern, grid, kFwdThreads, smem_bytes, static_cast<cudaStream_t>(stream), tm_q, tm_k,
                          tm_v, prm);
}

}  // namespace bsa

extern "C" int bsa_attn_fwd_rows(const void* q, const int64_t q_strides[4], const void* k,
                                 const int64_t k_strides[4], const void* v,
                                 const int64_t v_strides[4], void* o, const int64_t o_strides[4],
                                 float* lse2, float* rowmax, const int32_t* row_ptr,
                                 const int32_t* col_idx, int list_b_stride, int list_h_stride,
                                 float sm_scale, int dtype, int B, int H, int N, int D,
                                 int row_begin, int row_end, const uint8_t* dense,
                                 const int64_t dense_strides[4], int32_t* work_counter,
                                 int32_t* status, void* stream) {
  if (!row_ptr || !col_idx || !lse2) return BSA_ERR_BAD_POINTER;
  return bsa::launch_fwd(q, q_strides, k, k_strides, v, v_strides, o, o_strides, lse2, rowmax,
                         row_ptr, col_idx, nullptr, nullptr, list_b_stride, list_h_stride, sm_scale,
                         dtype, B, H, N, D, row_begin, row_end, dense, dense_strides, status,
                         work_counter, stream);
}

extern "C" int bsa_attn_fwd(const void* q, const int64_t q_strides[4], const void* k,
                            const int64_t k_strides[4], const void* v, const int64_t v_strides[4],
                            void* o, const int64_t o_strides[4], float* lse2, float* rowmax,
                            const int32_t* row_ptr, const int32_t* col_idx, int list_b_stride,
                            int list_h_stride, float sm_scale, int dtype, int B, int H, int N,
                            int D, int32_t* work_counter, int32_t* status, void* stream) {
  return bsa_attn_fwd_rows(q, q_strides, k, k_strides, v, v_strides, o, o_strides, lse2, rowmax,
                           row_ptr, col_idx, list_b_stride, list_h_stride, sm_scale, dtype, B, H,
                           N, D, 0, N / bsa::kBlock, nullptr, nullptr, work_counter, status, stream);
}

extern "C" int bsa_attn_fwd_block_mask_rows(
    const void* q, const int64_t q_strides[4], const void* k, const int64_t k_strides[4],
    const void* v, const int64_t v_strides[4], void* o, const int64_t o_strides[4], float* lse2,
    float* rowmax, const uint8_t* block, const int64_t block_strides[4], int Bm, int Hm,
    float sm_scale, int dtype, int B, int H, int N, int D, int row_begin, int row_end,
    const uint8_t* dense, const int64_t dense_strides[4], int32_t* work_counter, int32_t* status,
    void* stream) {
  if (!block || !block_strides || !lse2) return BSA_ERR_BAD_POINTER;
  if ((Bm != 1 && Bm != B) || (Hm != 1 && Hm != H)) return BSA_ERR_BAD_SHAPE;
  for (int i = 0; i < 4; ++i)
    if (block_strides[i] < 0) return BSA_ERR_BAD_STRIDE;
  return bsa::launch_fwd(q, q_strides, k, k_strides, v, v_strides, o, o_strides, lse2, rowmax,
                         nullptr, nullptr, block, block_strides, Bm > 1 ? 1 : 0, Hm > 1 ? 1 : 0,
                         sm_scale, dtype, B, H, N, D, row_begin, row_end, dense, dense_strides,
                         status, work_counter, stream);
}

extern "C" int bsa_attn_fwd_block_mask(const void* q, const int64_t q_strides[4], const void* k,
                                       const int64_t k_strides[4], const void* v,
                                       const int64_t v_strides[4], void* o,
                                       const int64_t o_strides[4], float* lse2, float* rowmax,
                                       const uint8_t* block, const int64_t block_strides[4],
                                       int Bm, int Hm, float sm_scale, int dtype, int B, int H,
                                       int N, int D, int32_t* work_counter, int32_t* status,
                                       void* stream) {
  return bsa_attn_fwd_block_mask_rows(q, q_strides, k, k_strides, v, v_strides, o, o_strides, lse2,
                                      rowmax, block, block_strides, Bm, Hm, sm_scale, dtype, B, H,
                                      N, D, 0, N > 0 ? N / bsa::kBlock : 0, nullptr, nullptr,
                                      work_counter, status, stream);
}

extern "C" int bsa_attn_fwd_block_mask_lists(
    const void* q, const int64_t q_strides[4], const void* k, const int64_t k_strides[4], const void* v,
    const int64_t v_strides[4], void* o, const int64_t o_strides[4], float* lse2, const uint8_t* block,
    const int64_t block_strides[4], int Bm, int Hm, float sm_scale, int dtype, int B, int H, int N, int D,
    const uint8_t* dense, const int64_t dense_strides[4], int32_t* row_cnt, int32_t* col_idx, int32_t* col_cnt,
    int32_t* row_idx, int32_t* work_counter, int32_t* status, void* stream) {
  if (!block || !block_strides || !lse2 || !row_cnt || !col_idx || !col_cnt || !row_idx) return BSA_ERR_BAD_POINTER;
  if ((Bm != 1 && Bm != B) || (Hm != 1 && Hm != H)) return BSA_ERR_BAD_SHAPE;
  for (int i = 0; i < 4; ++i)
    if (block_strides[i] < 0) return BSA_ERR_BAD_STRIDE;
  if (N > 0 && static_cast<int64_t>(Bm) * Hm * (N / bsa::kBlock) * (N / bsa::kBlock) > 0x7fffffffLL)
    return BSA_ERR_TOO_LARGE;
  const int rc = bsa::launch_fwd(q, q_strides, k, k_strides, v, v_strides, o, o_strides, lse2, nullptr, nullptr,
                                 nullptr, block, block_strides, Bm > 1 ? 1 : 0, Hm > 1 ? 1 : 0, sm_scale, dtype,
                                 B, H, N, D, 0, N > 0 ? N / bsa::kBlock : 0, dense, dense_strides, status,
                                 work_counter, stream, true);
  if (rc != BSA_OK) return rc;
  return bsa::launch_lists_places(block, block_strides, Bm, Hm, N / bsa::kBlock, row_cnt, col_idx, col_cnt, row_idx,
                                  true, stream);
}

extern "C" int bsa_attn_fwd_block_mask_output(
    const void* q, const int64_t q_strides[4], const void* k, const int64_t k_strides[4], const void* v,
    const int64_t v_strides[4], void* o, const int64_t o_strides[4], const uint8_t* block,
    const int64_t block_strides[4], int Bm, int Hm, float sm_scale, int dtype, int B, int H, int N, int D,
    const uint8_t* dense, const int64_t dense_strides[4], int32_t* work_counter, int32_t* status, void* stream) {
  if (!block || !block_strides) return BSA_ERR_BAD_POINTER;
  if ((Bm != 1 && Bm != B) || (Hm != 1 && Hm != H)) return BSA_ERR_BAD_SHAPE;
  for (int i = 0; i < 4; ++i)
    if (block_strides[i] < 0) return BSA_ERR_BAD_STRIDE;
  return bsa::launch_fwd(q, q_strides, k, k_strides, v, v_strides, o, o_strides, nullptr, nullptr, nullptr, nullptr,
                         block, block_strides, Bm > 1 ? 1 : 0, Hm > 1 ? 1 : 0, sm_scale, dtype, B, H, N, D, 0,
                         N > 0 ? N / bsa::kBlock : 0, dense, dense_strides, status, work_counter, stream);
}
