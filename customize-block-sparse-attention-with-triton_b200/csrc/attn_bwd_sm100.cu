// Backward block-sparse attention for sm_100a: one kernel template, two instantiations.
//
//   dK/dV (kDKDV = true):  a CTA owns ONE key block (64 keys), keeps its K and V in shared memory and
//       walks the block's list of query blocks (the column lists of the mask) two at a time
//       ("supersteps", tiles a and b):
//         S^T = K [Q_a;Q_b]^T, dP^T = V [dO_a;dO_b]^T                     (SS MMAs, M=64, N=128)
//         P^T = exp2(S^T c - LSE2[q]), dS^T = P^T (dP^T - delta[q])       (one thread per key row)
//         dV += P^T_a dO_a + P^T_b dO_b,  dK += dS^T_a Q_a + dS^T_b Q_b   (TS MMAs, M=64, N=128: A from
//       TMEM, B MN-major from shared memory).
//   dQ    (kDKDV = false): a CTA owns one query block, keeps Q and dO resident and walks the row list
//       of key blocks two at a time:
//         S = Q [K_a;K_b]^T, dP = dO [V_a;V_b]^T;  dS = exp2(S c - LSE2[row]) (dP - delta[row]);
//         dQ += dS_a K_a + dS_b K_b
//
// The M = 64 "weight stationary" form of the MMA puts the columns of tile a into TMEM lanes 0..63 and
// those of tile b into lanes 64..127 of the same 64 columns, so every SM sub-partition has
// exponentials to do whatever the mask is, and no operand is multiplied twice.  The accumulating
// products take both tiles at once in the same form: lanes 0..63 multiply their P or dS with tile a, lanes 64..127
// theirs with tile b.  Lane r sums the tile-a products of row r, lane r+64 its tile-b products; the two are
// added when the block is written out.  A tile b that does not exist is all zeros, in P and dS and in shared
// memory.
//
// Formulas are those of the reference's backward (fa2_custom_mask/fa2_bwd.py:56-74, 116-130) with
// M replaced by a true base-2 log-sum-exp; the iteration space is the tile lists, not the
// reference's causal loops.  dK and dQ carry the factor sm_scale.
//
// Persistent: one CTA per SM starts with block blockIdx.x and draws further blocks from an
// optional work counter (or walks a fixed stride); long lists first when the mask is causal.  dQ may run
// beside dK/dV (see `together`).
// Roles (28 warps; warp 25 has none):
//   warps 0..15 : compute, two teams of eight warps on alternate supersteps (team = warp / 8, TMEM lane
//                 quarter = warp % 4, 32 of a tile's 64 columns = (warp / 4) % 2), so that one team's
//                 barrier round trips and products run under the other one's arithmetic
//   warps 16, 19: TMA producers, one for Q and K (and LSE2), one for dO and V (and delta): an SM starts a
//                 copy only every 190 cycles or so from one warp, and four tiles and four vectors a
//                 superstep from a single one (1,270 cycles) were what the whole kernel waited for
//   warps 17, 26: issue the S/dP MMAs, one for each team (a wait, eight MMAs and their commit take an
//                 issuer longer than the superstep); warp 17 owns TMEM
//   warps 18, 24: issue the accumulating MMAs (dK/dV: one warp for dV, one for dK, since a single issuer of
//                 both spent most of a superstep on its own waits and commits; dQ has one product and one
//                 issuer).  All issuers run warp-wide with one elected lane issuing
//   warp 27     : lister: draws the blocks, looks their lists up and publishes them.  It does so while the block
//                 before is still being loaded.  (By the first producer after its last load, ticket, list and
//                 first entries were three trips to memory one after the other, 3,000 to 4,000 cycles from one
//                 block's last copy to the next one's first, with three supersteps of 1,000 in the ring to bridge
//                 them.  Forward and backward, 2 x 8 heads, N = 4160, causal, a quarter 88.6 -> 84.9 us; 2 x 16
//                 heads, N = 16384 1,646 -> 1,612.  Set up 2 to 5 supersteps before the last load: the same.)
//   warps 20..23: take a block's sums out of tensor memory and store them while the compute warps are
//                 already at work on the next block
// A block's own operands are double-buffered: the next block's are loaded while this one is at work.
// Head dimensions 16 and 32: zero-filled on load by D-wide tensor maps, D / 16 K steps for S and dP.
// S and dP of a superstep have slots in TMEM, and P and dS are stored over S: a slot of S is held until their
// products are complete, one of dP only until the arithmetic is done.
// What bounds it: the way of a superstep through its slots, with no part of it that is the bound alone.
// A dK/dV superstep takes 950 cycles (900 to 1,000 more at a block's end), of which the tensor pipe 756, shared memory's
// port about 1,000 (operands of S and dP 384, of the accumulating products 256, copies arriving 256, LSE2 and delta and the
// looks at barriers 200; part of it at once), the exponentials 512; a dQ superstep 790, of which the tensor pipe 585.  One
// superstep's way is 750 cycles to the logits, 850 for the arithmetic, 220 to the accumulating products, 550 until
// they are complete.  B=2, H=16, N=16384, 25 % of the tiles under a causal mask, forward and backward at the power
// cap: 1,578 us (1,904 with products of one tile each, shared memory not aligned, no lister and the steps below).
// (With S and dP multiplied from tensor memory, which has no room for K and V, the port and the tensor pipe would have
// 128 cycles a superstep less: 3 %.)
// Every wait is bounded, and a role that gives up raises a CTA-wide flag, which the others look at when they wait
// for an item.  Every barrier is waited on by warps that see each of its phases.
#include <math.h>

#include "host_common.h"
#include "sm100_ptx.cuh"

namespace bsa {

// The streamed tiles: ten places of two tiles (16 KB), split into a ring for Q (dK/dV) or K (dQ) and one
// for dO or V.  What an accumulating product reads (Q and dO; K) is held from its load to the end of
// that product, about 4,500 cycles with the arithmetic in between; V only until dP is complete.  With
// rings too short for that the issuers wait for operands (dK/dV, four places each: a third of the time).
constexpr int kRing = 10;
template <bool kDKDV> constexpr int kRing0 = kDKDV ? 5 : 6;
template <bool kDKDV> constexpr int kRing1 = kRing - kRing0<kDKDV>;
constexpr int kCW = 16;                    // compute warps: 2 teams x 4 lane quarters x 2 column halves
constexpr int kTeamW = kCW / 2;
constexpr int kProdWarp = kCW, kXWarp = kCW + 1, kAccWarp = kCW + 2, kProd2Warp = kCW + 3;
constexpr int kX2Warp = 26, kAcc2Warp = 24;           // (warps kCW + 4 .. kCW + 7 write out: lane quarter = warp % 4)
constexpr int kListWarp = 27;
constexpr int kGoBefore = 3;                  // supersteps of loads before an item's end at which the next one is set up
constexpr int kBwdThreads = 32 * (kCW + 12);  // whole warpgroups: one warp at the end only fills one
// Registers by warpgroup: 4 compute, which keep what they are launched with, producers and first issuers, write-out,
// second issuers and lister.  All waits are bounded but the one for registers that the block was not launched
// with.  (kBwdLaunchRegs is what the compiler makes of the launch bounds; the host compares before the first launch.)
constexpr int kBwdLaunchRegs = 72, kBwdIssuerRegs = 40, kBwdWriteRegs = 136;
static_assert((kCW / 4) * kBwdLaunchRegs + 2 * kBwdIssuerRegs + kBwdWriteRegs <= kBwdLaunchRegs * kBwdThreads / 128);
static_assert(kBwdWriteRegs >= kBwdLaunchRegs && kBwdIssuerRegs <= kBwdLaunchRegs);
constexpr uint32_t kBwdTile = 64 * 64 * 2;
constexpr uint32_t kBwdTmemCols = 512;
constexpr int kListIndex = BSA_LIST_PARTIAL_FLAG - 1;  // a list entry without its flag
// TMEM columns: S (or S^T) of superstep g in slot g % kSlots, 64 columns each, dP (or dP^T) behind them in slot
// g % kDpSlots; two fp32 accumulators at the end (dQ: one).  P and dS (as 16-bit pairs) go over the 16 columns of S
// that they come from, P into the first 8 and dS into the last 8 of them (dQ: dS into the first 8): a warp only
// overwrites what it has read itself.  So a dP slot is free as soon as the arithmetic is done, and where there is one
// accumulator S can be four supersteps deep: dQ with everything listed, 2 heads, N = 9600, forward and backward 280 us
// with 3 + 3 slots, 272.5 so, lists of 16 supersteps the same.  (dK/dV with 4 + 2: both teams fall into step, at
// 1,394 us for 2 x 16 heads, N = 16384 against 1,377.)
constexpr int kDpSlots = 3;
template <bool kDKDV> constexpr int kSlots = kDKDV ? 3 : 4;
template <bool kDKDV> constexpr uint32_t kTmDp = 64 * kSlots<kDKDV>;
constexpr uint32_t kTmAcc0 = 384, kTmAcc1 = 448;
static_assert(kTmDp<true> + 64 * kDpSlots <= kTmAcc0 && kTmDp<false> + 64 * kDpSlots <= kTmAcc1);
// Barriers by superstep: an even number, so that the issuers and teams, which see every second superstep, see each
// phase of theirs, and more than there are supersteps between those that look at one and those that complete it.
constexpr int kXBars = 6;
static_assert(kXBars % 2 == 0 && kXBars > kSlots<false> && kXBars > kRing0<true> && kXBars > kRing1<true>);
// dQ: places of a block's LSE2 and delta, which are read at each of its supersteps.  Those of block n are fetched when
// all S/dP of block n-2 are complete, and with that the arithmetic of all but its last kDpSlots supersteps: what
// block n-5 has is not read any more, even if all blocks have a single superstep.
constexpr int kVecPlaces = 5;
static_assert(kVecPlaces >= kDpSlots + 2 && kVecPlaces <= kRing0<true> && kVecPlaces <= kRing1<true>);

struct BwdSmem {
  uint8_t stat[2][2][kBwdTile];             // by block parity: the CTA's own K, V (dK/dV) or Q, dO (dQ)
  uint8_t ring[kRing][2][kBwdTile];         // streamed tiles a, b: Q (dK/dV) or K (dQ), then dO or V
  float lse[kRing0<true>][2][64];           // dK/dV: LSE2 and delta of the streamed query tiles
  float delta[kRing1<true>][2][64];
  // write-out: what lanes 0..63 and 64..127 hand to each other, 32 columns of 64 rows at a time (rows of
  // 36 floats: eight lanes' 16-byte accesses then fall into different banks)
  float xfer[2][64][36];
  // by item parity: the work item
  int4 item[2];                             // batch (-1 = no more work), head, block, list length
  int item_begin[2];                        // where its list begins
  int first[2][32];                         // the first entries of its list
  uint64_t item_full[2], item_free[2];      // published; read by all its readers
  uint64_t setup_go[2];                     // first producer -> lister: time to set up the next one
  uint64_t stat_full[2], stat_free[2];      // own operands loaded; their S/dP instructions complete
  uint64_t acc_done;                        // all accumulating MMAs of the block complete (one arrival per issuer)
  uint64_t acc_free;                        // the write-out warps have read the accumulators
  // a place's tiles have landed: one barrier for each place and team, so that the team's issuer and
  // compute warps, which wait on it, see each of its phases
  uint64_t in_full0[2 * kRing0<false>], in_full1[2 * kRing1<true>];
  uint64_t in_empty0[kRing0<false>];        // dQ: accumulating MMAs that read the place of K complete
  uint64_t in_empty1[kRing1<false>];        // dQ: dP complete, the place of V is free (dK/dV goes by d_free)
  // by superstep modulo kXBars:
  uint64_t x_full[kXBars];                  // S/dP complete (dK/dV: and LSE2 and delta there)
  uint64_t d_full[kXBars];                  // P/dS stored: the slot of dP is free
  uint64_t d_free[kXBars];                  // accumulating MMAs that read P/dS complete: the slot of S is free
  uint32_t tmem_base;
  int abort_flag;                           // a role has given up
};

static_assert(sizeof(BwdSmem) <= 232448, "BwdSmem exceeds the shared memory of one CTA");

struct BwdParams {
  const int32_t* list_ptr;  // dK/dV: column lists (col_ptr/row_idx); dQ: row lists (row_ptr/col_idx)
  const int32_t* list_idx;
  int list_places;          // 0: list_ptr holds offsets; else counts, list u at list_idx + u * list_places
  const uint8_t* dense;     // optional element-level mask for the tiles whose list entry is flagged
  int64_t ds0, ds1, ds2;
  const float* lse2;
  const float* delta;
  void* out0;  // dV (dK/dV kernel only)
  void* out1;  // dK or dQ
  int64_t sb0, sh0, sn0, sb1, sh1, sn1;  // their element strides
  int B, H, N, D, nb;
  int items;  // B * H * nb
  int list_b_stride, list_h_stride;
  float scale_log2;
  float sm_scale;
  int32_t* status;
  int32_t* ticket;  // optional work counter (0 at kernel start, left 0): dynamic item hand-out
  int wide_stores;  // output rows start on 32-byte boundaries
  // dK/dV: dQ of the same call follows in the stream and may begin as soon as SMs are free; dQ: that is
  // what it does (it reads nothing that dK/dV writes)
  int together;
};

__device__ __forceinline__ void bwd_give_up(BwdSmem* sm, int32_t* status, int code) {
  sm->abort_flag = 1;
  report_status(status, code);
}

// At the beginning of every role.  The first item is published after the end of the kernel before, which may take
// any time (one that lets its successor in early and then waits for a peer, say): a role's limited waits
// begin when that has ended.  Together, dQ begins while dK/dV is still running: it is launched when all CTAs of
// dK/dV have passed this point, so what came before dK/dV has ended.  (That dQ sees it without a wait of its
// own is observed, not promised: see grid_dependency_wait.)  It ends after dK/dV (see the end).
template <bool kDKDV>
__device__ __forceinline__ void bwd_begin(const BwdParams& p) {
  if (kDKDV || !p.together) grid_dependency_wait();
}

// A work item as the lister publishes it.
struct BwdItem {
  int b, h, blk, n_tiles;  // b < 0: no more work
  int begin;               // of its list, in list_idx
  __device__ __forceinline__ int supersteps() const { return (n_tiles + 1) >> 1; }
  __device__ __forceinline__ int64_t vec_base(const BwdParams& p) const {  // into lse2 / delta
    return (static_cast<int64_t>(b) * p.H + h) * p.N;
  }
};

// Readers of the items: wait for item i, read it, tell the lister that it was read (first: the lane's own of
// the first 32 entries, for the producers).
__device__ __forceinline__ bool bwd_next_item(BwdSmem* sm, int i, int lane, BwdItem* it, int* first = nullptr) {
  const int par = i & 1;
  if (!mbar_wait_warp_item(smem_u32(&sm->item_full[par]), (i >> 1) & 1, &sm->abort_flag)) return false;
  const int4 h = sm->item[par];
  it->b = h.x;
  it->h = h.y;
  it->blk = h.z;
  it->n_tiles = h.w;
  it->begin = sm->item_begin[par];
  if (first != nullptr) *first = sm->first[par][lane];
  __syncwarp();
  if (lane == 0) mbar_arrive(smem_u32(&sm->item_free[par]));
  return true;
}

// Work item w -> (batch, head, block) and its list (one warp; first: the lane's own of the first 32 entries).
// dQ: long (late) rows first; dK/dV: long (early) key columns first when the mask is causal.
struct BwdFound {
  int4 it;
  int begin, first;
};
template <bool kDKDV>
__device__ __forceinline__ BwdFound bwd_look_up(const BwdParams& p, int w, int lane) {
  BwdFound f{make_int4(-1, 0, 0, 0), 0, 0};
  if (w < p.items) {
    const int bh = w / p.nb;
    f.it.z = kDKDV ? (w - bh * p.nb) : (p.nb - 1 - (w - bh * p.nb));
    f.it.x = bh / p.H;
    f.it.y = bh - f.it.x * p.H;
    const int64_t li = static_cast<int64_t>(f.it.x * p.list_b_stride + f.it.y * p.list_h_stride) * p.nb + f.it.z;
    if (p.list_places > 0) {
      f.begin = static_cast<int>(li * p.list_places);
      if (lane < p.list_places) f.first = __ldg(p.list_idx + f.begin + lane);
      f.it.w = __ldg(p.list_ptr + li);
    } else {
      f.begin = __ldg(p.list_ptr + li);
      f.it.w = __ldg(p.list_ptr + li + 1) - f.begin;
      if (lane < f.it.w) f.first = __ldg(p.list_idx + f.begin + lane);
    }
  }
  return f;
}

// The lister (one warp): draws the items, looks their lists up and publishes them with the first entries,
// kGoBefore supersteps of loads before the producers need them.
template <bool kDKDV>
__device__ __forceinline__ void bwd_list_items(BwdSmem* sm, const BwdParams& p, BwdFound f, int lane) {
  const int stride = gridDim.x;
  bool ok = true;
  bool terminal = p.ticket == nullptr;  // drew a ticket past the end (or draws none)
#pragma unroll 1
  for (int i = 0, w = blockIdx.x;; ++i) {
    const int par = i & 1;
    if (i > 0) {
      ok = mbar_wait_warp_item(smem_u32(&sm->setup_go[par ^ 1]), ((i - 1) >> 1) & 1, &sm->abort_flag);
      if (!ok) break;
      if (p.ticket != nullptr) {
        int t = 0;
        if (lane == 0) {
          t = atomicAdd(p.ticket, 1);
          // every CTA draws until its first ticket past the end, so the launch draws exactly
          // `items` tickets in all; whoever draws the last one leaves the counter at zero
          if (t == p.items - 1) atomicExch(p.ticket, 0);
        }
        w = stride + __shfl_sync(0xffffffffu, t, 0);
        terminal = w >= p.items;
      } else {
        w += stride;
      }
    }
    if (i > 0) f = bwd_look_up<kDKDV>(p, w, lane);
    // item i-2 must have been read by everyone
    if (i >= 2) ok = mbar_wait_warp_item(smem_u32(&sm->item_free[par]), ((i - 2) >> 1) & 1, &sm->abort_flag);
    if (!ok) break;
    sm->first[par][lane] = f.first;
    if (lane == 0) {
      sm->item[par] = f.it;
      sm->item_begin[par] = f.begin;
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&sm->item_full[par]));  // release: the item is visible
    if (f.it.x < 0) break;
  }
  if (!ok) bwd_give_up(sm, p.status, 1);
  if (!terminal && lane == 0) {
    // gave up before the last draw: draw on (without working) until this CTA's first ticket past
    // the end, so that the launch still draws `items` tickets and the counter returns to zero
    int t;
    do {
      t = atomicAdd(p.ticket, 1);
      if (t == p.items - 1) atomicExch(p.ticket, 0);
    } while (stride + t < p.items);
  }
}

// A producer's share of an item's supersteps: the listed tiles a, b of one tensor into its half of the
// ring (and, dK/dV, the tiles' part of one of the two vectors), one lane per copy, copies of one kind in
// one instruction.  In the place of a tile that does not exist comes block `none`, behind the last one: zeros.
// (first: the lane's own of the first 32 entries; those behind them are fetched 32 at a time, ahead of need.)
// go: the barrier on which the lister waits to set up the next item, or 0.
template <int kPlaces, bool kVector>
__device__ __forceinline__ bool bwd_load_tiles(uint8_t* ring, uint64_t* full, uint64_t* empty,
                                               const CUtensorMap* map, float* vec_ring, const float* vec,
                                               const BwdItem& it, const int32_t* ents, int first, int none,
                                               uint32_t go, int lane, int* gs) {
  const int n_super = it.supersteps(), j_go = max(n_super - kGoBefore, 0);
  int mine = first, next = 32 + lane < it.n_tiles ? __ldg(ents + 32 + lane) : 0;
#pragma unroll 1
  for (int j = 0; j < n_super; ++j, ++*gs) {
    if (j == j_go && lane == 0 && go != 0) mbar_arrive(go);
    const int s = *gs % kPlaces;
    const int nt = min(2, it.n_tiles - 2 * j), t = lane & 1;
    if ((j & 15) == 0 && j > 0) {
      mine = next;
      const int at = 2 * j + 32 + lane;
      if (at < it.n_tiles) next = __ldg(ents + at);
    }
    const int entry = __shfl_sync(0xffffffffu, mine, (2 * j + t) & 31);
    const int nj = t < nt ? (entry & kListIndex) : none;
    if (kVector) {
      // dK/dV: the place is free when the products of its previous superstep are (empty: d_free)
      if (*gs >= kPlaces &&
          !mbar_wait_warp(smem_u32(empty + (*gs - kPlaces) % kXBars), ((*gs - kPlaces) / kXBars) & 1))
        return false;
    } else {
      if (!mbar_wait_warp(smem_u32(empty + s), ((*gs / kPlaces) & 1) ^ 1)) return false;
    }
    const uint32_t bar = smem_u32(full + *gs % (2 * kPlaces));
    if (lane == 0) mbar_expect_tx(bar, 2 * kBwdTile + (kVector ? nt * 256u : 0u));
    __syncwarp();
    if (lane < 2)
      tma_load_4d(smem_u32(ring) + (2 * s + t) * kBwdTile, map, bar, 0, nj * 64, it.h, it.b);
    if (kVector && (lane & 30) == 2 && t < nt)
      bulk_load_1d(smem_u32(vec_ring + (2 * s + t) * 64), vec + nj * 64, 256, bar);
  }
  return true;
}

// A producer (one warp): a block's own operand and its share of the streamed tiles.  dQ: the block's part of LSE2
// or delta comes with the operand, into one of kRing0<true> places.
template <bool kDKDV, bool kFirst>
__device__ __forceinline__ void bwd_produce(BwdSmem* sm, const BwdParams& p, const CUtensorMap* own_map,
                                            const CUtensorMap* map, int lane) {
  constexpr int kR0 = kRing0<kDKDV>;
  float* const vec_ring = kFirst ? sm->lse[0][0] : sm->delta[0][0];
  bool ok = true;
  int gs = 0, ni = 0;
  bwd_begin<kDKDV>(p);
  // (by a role that has waited, and by no other: a warp without a role must not let dQ in)
  if (kFirst && kDKDV && p.together) grid_dependents_launch();
#pragma unroll 1
  for (int i = 0; ok; ++i) {
    BwdItem it;
    int first;
    ok = bwd_next_item(sm, i, lane, &it, &first);
    if (!ok || it.b < 0) break;
    const uint32_t go = kFirst ? smem_u32(&sm->setup_go[i & 1]) : 0u;
    if (it.n_tiles == 0) {
      if (kFirst && lane == 0) mbar_arrive(go);
      continue;
    }
    // the S/dP instructions of the block before the previous one must be complete
    const int own = ni & 1;
    if (ni >= 2) ok = mbar_wait_warp(smem_u32(&sm->stat_free[own]), ((ni - 2) >> 1) & 1);
    if (!ok) break;
    const float* vec = (kFirst ? p.lse2 : p.delta) + it.vec_base(p);
    if (lane == 0) {
      const uint32_t bar = smem_u32(&sm->stat_full[own]);
      mbar_expect_tx(bar, kBwdTile + (kDKDV ? 0u : 256u));
      tma_load_4d(smem_u32(sm->stat[own][kFirst ? 0 : 1]), own_map, bar, 0, it.blk * 64, it.h, it.b);
      if constexpr (!kDKDV)
        bulk_load_1d(smem_u32(vec_ring + (ni % kVecPlaces) * 128), vec + it.blk * 64, 256, bar);
    }
    if constexpr (kFirst)
      ok = bwd_load_tiles<kR0, kDKDV>(sm->ring[0][0], sm->in_full0, kDKDV ? sm->d_free : sm->in_empty0, map, vec_ring,
                                      vec, it, p.list_idx + it.begin, first, p.nb, go, lane, &gs);
    else
      ok = bwd_load_tiles<kRing1<kDKDV>, kDKDV>(sm->ring[kR0][0], sm->in_full1, kDKDV ? sm->d_free : sm->in_empty1, map,
                                                vec_ring, vec, it, p.list_idx + it.begin, first, p.nb, 0u, lane, &gs);
    ++ni;
  }
  if (!ok) bwd_give_up(sm, p.status, 1);
}

// Write-out: a lane's 32 sums for the lane that finishes their columns.
__device__ __forceinline__ void bwd_hand_over(float* at, const uint32_t* sums) {
  uint4* to = reinterpret_cast<uint4*>(at);
#pragma unroll
  for (int k = 0; k < 8; ++k) to[k] = make_uint4(sums[4 * k], sums[4 * k + 1], sums[4 * k + 2], sums[4 * k + 3]);
}

// The S/dP instructions of one team's supersteps (one warp).
template <bool kBf16, bool kDKDV>
__device__ __forceinline__ void bwd_issue_x(BwdSmem* sm, const BwdParams& p, uint32_t tmem, int team,
                                            int lane) {
  constexpr uint32_t idesc_x = umma_idesc(kBf16, 0, 0, 64, 128);
  const bool leader = elect_one();
  const uint64_t desc_a0 = smem_desc_sw128(smem_u32(sm->stat[0][0]), 16, 1024);
  const uint64_t desc_b0 = smem_desc_sw128(smem_u32(sm->ring[0][0]), 16, 1024);
  const uint64_t desc_b1 = smem_desc_sw128(smem_u32(sm->ring[kRing0<kDKDV>][0]), 16, 1024);
  constexpr int kR0 = kRing0<kDKDV>, kR1 = kRing1<kDKDV>, kDp = kDpSlots, kS = kSlots<kDKDV>;
  constexpr uint64_t kTileDesc = kBwdTile >> 4;  // one tile further, in descriptor units
  const int k_steps = p.D >> 4;
  bool ok = true;
  int gs = 0, ni = 0;
  bwd_begin<kDKDV>(p);
#pragma unroll 1
  for (int i = 0; ok; ++i) {
    BwdItem it;
    ok = bwd_next_item(sm, i, lane, &it);
    if (!ok || it.b < 0) break;
    const int n_super = it.supersteps();
    if (n_super == 0) continue;
    const int own = ni & 1;
    const uint32_t stat = smem_u32(&sm->stat_full[own]), stat_phase = (ni >> 1) & 1;
    const uint64_t a0 = desc_a0 + static_cast<uint64_t>(2 * own) * kTileDesc;
    int g = gs + ((gs ^ team) & 1);
    gs += n_super;
    if (g >= gs) ok = mbar_wait_warp(stat, stat_phase);  // nothing to do, but the phase has to be seen
#pragma unroll 1
    for (; ok && g < gs; g += 2) {
      const uint32_t s_tmem = tmem + 64 * (g % kS), dp_tmem = tmem + kTmDp<kDKDV> + 64 * (g % kDp);
      const uint32_t x_full = smem_u32(&sm->x_full[g % kXBars]);
      const uint64_t b0 = desc_b0 + static_cast<uint64_t>(2 * (g % kR0)) * kTileDesc;
      const uint64_t b1 = desc_b1 + static_cast<uint64_t>(2 * (g % kR1)) * kTileDesc;
      // the operands, and the accumulating products of the slot's previous superstep must be complete (the first
      // ones ask for the phase before the first one, which counts as complete; the block's own operand stays
      // complete as long as the block lasts, and with a wait of its own 2 x 16 heads, N = 16384, causal, a quarter,
      // forward and backward 1,378 us, 1,368 so)
      ok = mbar_wait_warp3(stat, stat_phase, smem_u32(&sm->in_full0[g % (2 * kR0)]), (g / (2 * kR0)) & 1,
                           smem_u32(&sm->d_free[(g + kXBars - kS) % kXBars]), ((g + kXBars - kS) / kXBars + 1) & 1);
      if (!ok) break;
      tc_fence_after();
      if (leader) {
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          if (kk < k_steps) umma_ws_ss(s_tmem, a0 + 2 * kk, b0 + 2 * kk, idesc_x, kk > 0);
      }
      __syncwarp();
      // the arithmetic on the slot's previous superstep must be done
      ok = mbar_wait_warp2(smem_u32(&sm->in_full1[g % (2 * kR1)]), (g / (2 * kR1)) & 1,
                           smem_u32(&sm->d_full[(g + kXBars - kDp) % kXBars]), ((g + kXBars - kDp) / kXBars + 1) & 1);
      if (!ok) break;
      tc_fence_after();
      if (leader) {
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          if (kk < k_steps) umma_ws_ss(dp_tmem, a0 + kTileDesc + 2 * kk, b1 + 2 * kk, idesc_x, kk > 0);
        tc_commit(x_full);
        mbar_arrive(x_full);  // release: LSE2 and delta have been seen to be there
        if constexpr (!kDKDV) tc_commit(smem_u32(&sm->in_empty1[g % kR1]));  // V is not needed any more
      }
    }
    if (ok && leader) tc_commit(smem_u32(&sm->stat_free[own]));  // this issuer is through with the operands
    ++ni;
  }
  if (!ok) bwd_give_up(sm, p.status, 2);
}

// The accumulating instructions of one warp.  dK/dV: the first warp's sum dV, the second one's dK (each
// accumulator has one issuer, which keeps its products in order); dQ: the first warp's, there is no second one.
template <bool kBf16, bool kDKDV>
__device__ __forceinline__ void bwd_issue_acc(BwdSmem* sm, const BwdParams& p, uint32_t tmem, bool first,
                                              int lane) {
  const bool dv = kDKDV && first;
  constexpr uint32_t idesc = umma_idesc(kBf16, 0, 1, 64, 128);
  const bool leader = elect_one();
  const int places = dv ? kRing1<kDKDV> : kRing0<kDKDV>;
  const uint64_t desc = smem_desc_sw128(smem_u32(sm->ring[dv ? kRing0<kDKDV> : 0][0]), 8192, 1024);
  const uint32_t empty = smem_u32(sm->in_empty0);  // (dQ)
  const uint32_t acc = tmem + (dv ? kTmAcc0 : kTmAcc1), from = tmem + (kDKDV && !dv ? 8 : 0);
  bool ok = true;
  int ni = 0, place = 0, slot = 0, x = 0;
  uint32_t phase = 0;  // of the superstep's barrier
  bwd_begin<kDKDV>(p);
#pragma unroll 1
  for (int i = 0; ok; ++i) {
    BwdItem it;
    ok = bwd_next_item(sm, i, lane, &it);
    if (!ok || it.b < 0) break;
    if (it.n_tiles == 0) continue;
    // the write-out warps must have read the previous block's accumulators (the first one asks for the phase before
    // the first one, which counts as complete)
    ok = mbar_wait_warp(smem_u32(&sm->acc_free), (ni & 1) ^ 1);
#pragma unroll 1
    for (int left = it.n_tiles; ok && left > 0; left -= 2) {
      ok = mbar_wait_warp(smem_u32(&sm->d_full[x]), phase);
      if (!ok) break;
      tc_fence_after();
      if (leader) {
        // rows [16 kk, +16) of a streamed tile: those of P or dS in the first or last 8 of columns [16 kk, +16) of
        // their slot; tile a's in lanes 0..63, tile b's in lanes 64..127.  (A product for each
        // tile, with the other's lanes switched off: bf16 2 x 16 heads, N = 16384, causal, a quarter, forward
        // and backward 1,835 us, 1,785 so; 2 x 8 heads, N = 4160 97.5 and 96.2.)
        const uint32_t cols = from + 64 * slot;
        const uint64_t b0 = desc + static_cast<uint64_t>(2 * place * (kBwdTile >> 4));
        const uint32_t more = left != it.n_tiles;
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          umma_ws_ts(acc, cols + 16 * kk, b0 + 128 * kk, idesc, more | (kk > 0));
        if constexpr (!kDKDV) tc_commit(empty + 8 * place);  // place free
        tc_commit(smem_u32(&sm->d_free[x]));  // P or dS columns free; accumulator updated
        if (left <= 2) tc_commit(smem_u32(&sm->acc_done));  // the block's sums are final
      }
      if (++place == places) place = 0;
      if (++slot == kSlots<kDKDV>) slot = 0;
      if (++x == kXBars) x = 0, phase ^= 1;
    }
    ++ni;
  }
  if (!ok) bwd_give_up(sm, p.status, 2);
}

// Persistent: one CTA per SM.  The lister starts with item blockIdx.x and then draws further
// items from the optional work counter (or walks a fixed stride), and hands them to
// the other roles through shared memory; every role walks the same sequence and counts
// supersteps (gs) and non-empty items (ni) the same way, so barrier phases follow from the counts.

// kElementMask: the instantiation that applies a dense mask inside the tiles whose list entries
// are flagged; the plain one carries none of that code.
template <bool kBf16, bool kDKDV, bool kElementMask>
__global__ void __launch_bounds__(kBwdThreads, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tm_stat0,
                const __grid_constant__ CUtensorMap tm_stat1,
                const __grid_constant__ CUtensorMap tm_str0,
                const __grid_constant__ CUtensorMap tm_str1, const BwdParams p) {
  // (Aligned by declaration: every address in it is a constant then.  Rounded up at run time, all roles carried a
  // base and added to it at every barrier: 2 x 16 heads, N = 16384, causal, a quarter, forward and backward
  // 1,745 -> 1,645 us; 2 x 8 heads, N = 4160 96.0 -> 89.0.)
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  BwdSmem* sm = reinterpret_cast<BwdSmem*>(smem_raw);

  const int warp = uniform_warp_index();
  const int lane = threadIdx.x & 31;

  if (warp == 0) {
    mbar_init_warp(sm->item_full, 2, 1, lane);
    mbar_init_warp(sm->item_free, 2, kCW + 8 + (kDKDV ? 2 : 1), lane);  // all other roles
    mbar_init_warp(sm->setup_go, 2, 1, lane);
    mbar_init_warp(sm->stat_full, 2, 2, lane);        // two producers
    mbar_init_warp(sm->stat_free, 2, 2, lane);        // two S/dP issuers
    mbar_init_warp(sm->d_full, kXBars, kTeamW, lane);  // one arrival per warp
    mbar_init_warp(sm->x_full, kXBars, 2, lane);      // the commit and the issuer
    mbar_init_warp(sm->d_free, kXBars, kDKDV ? 2 : 1, lane);
    mbar_init_warp(sm->in_full0, 2 * kRing0<false>, 1, lane);
    mbar_init_warp(sm->in_full1, 2 * kRing1<true>, 1, lane);
    if constexpr (!kDKDV) {
      mbar_init_warp(sm->in_empty0, kRing0<false>, 1, lane);
      mbar_init_warp(sm->in_empty1, kRing1<false>, 1, lane);
    }
    mbar_init_warp(&sm->acc_done, 1, kDKDV ? 2 : 1, lane);
    mbar_init_warp(&sm->acc_free, 1, 4, lane);  // one arrival per write-out warp
    if (lane == 0) sm->abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == kXWarp) {
    tmem_alloc(smem_u32(&sm->tmem_base), kBwdTmemCols);
    tmem_relinquish();
  }
  if (warp == kProdWarp && lane == 0) {
    tma_prefetch_desc(&tm_stat0);
    tma_prefetch_desc(&tm_stat1);
    tma_prefetch_desc(&tm_str0);
    tma_prefetch_desc(&tm_str1);
  }
  tc_fence_before();
  BwdFound found;
  if (warp == kListWarp) {
    // looks the CTA's first item up while the others set up and get as far as their first wait.  (All of that one after
    // the other, barriers initialised by one thread: forward and backward, 2 x 8 heads, N = 4160 84.9 us, so 84.0.)
    bwd_begin<kDKDV>(p);
    found = bwd_look_up<kDKDV>(p, blockIdx.x, lane);
    named_barrier_sync(1, kBwdThreads);  // the barriers are there
  } else {
    named_barrier_arrive(1, kBwdThreads);
    named_barrier_sync(3, kBwdThreads - 32);
  }
  tc_fence_after();
  const uint32_t tmem = sm->tmem_base;
  // 896 threads are launched with 72 registers: the write-out warps take what the producers and the
  // issuers do without (40 + 136 + 40 = 3 x 72).
  if ((warp >= kCW && warp < kCW + 4) || warp >= kCW + 8) {
    give_registers<kBwdIssuerRegs>();
    if (warp == kProdWarp) {
      bwd_produce<kDKDV, true>(sm, p, &tm_stat0, &tm_str0, lane);
    } else if (warp == kProd2Warp) {
      bwd_produce<kDKDV, false>(sm, p, &tm_stat1, &tm_str1, lane);
    } else if (warp == kListWarp) {
      bwd_list_items<kDKDV>(sm, p, found, lane);
    } else if (warp == kXWarp || warp == kX2Warp) {
      bwd_issue_x<kBf16, kDKDV>(sm, p, tmem, warp == kX2Warp, lane);
    } else if (warp == kAccWarp || (kDKDV && warp == kAcc2Warp)) {
      bwd_issue_acc<kBf16, kDKDV>(sm, p, tmem, warp == kAccWarp, lane);
    }
  } else if (warp < kCW) {
    // =========================== compute warps ===========================
    const int team = warp >> 3;
    const int ch = (warp >> 2) & 1;     // which 32 of the tile's 64 columns
    const int quarter = warp & 3;
    const int t_mine = quarter >> 1;    // lanes 0..63 own tile a of a superstep, 64..127 tile b
    const int r_blk = (quarter & 1) * 32 + lane;  // row of the CTA's block
    const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
    const uint32_t x_base = tmem + lane_base + 32 * ch;
    const float c = p.scale_log2;
    bool ok = true;
    int gs = 0, ni = 0;  // supersteps of earlier items (this team takes those with gs % 2 == team), items with any
    bwd_begin<kDKDV>(p);
#pragma unroll 1
    for (int i = 0; ok; ++i) {
      BwdItem it;
      ok = bwd_next_item(sm, i, lane, &it);
      if (!ok || it.b < 0) break;
      const int n_super = it.supersteps();
      if (n_super == 0) continue;  // (the write-out warps store the zero gradients)
      const int vec_at = (ni++ % kVecPlaces) * 128 + r_blk;  // (dQ)
      const uint8_t* mask_at = nullptr;
      const int32_t* ents = nullptr;
      if constexpr (kElementMask) {
        const int row = it.blk * 64 + r_blk;
        ents = p.list_idx + it.begin + t_mine;
        // element-level mask: where this lane's mask bytes of a tile start (dQ: its query row, 32
        // consecutive keys; dK/dV: its key column, 32 consecutive query rows)
        mask_at = p.dense + it.b * p.ds0 + it.h * p.ds1 +
                  (kDKDV ? static_cast<int64_t>(row) : static_cast<int64_t>(row) * p.ds2);
      }
      int j = (gs ^ team) & 1;
      int g = gs + j;
      gs += n_super;
#pragma unroll 1
      for (; ok && j < n_super; j += 2, g += 2) {
        const bool active = 2 * j + t_mine < it.n_tiles;  // this lane's tile exists (warp-uniform)
        const uint32_t s_at = x_base + 64 * (g % kSlots<kDKDV>), dp_at = x_base + kTmDp<kDKDV> + 64 * (g % kDpSlots);
        // A tile with masked elements inside: fetch this lane's 32 mask bytes while S is on its way
        uint32_t mw[8];
        bool partial = false;
        if (kElementMask && active) {
          const int e = __ldg(ents + 2 * j);
          partial = (e & BSA_LIST_PARTIAL_FLAG) != 0;  // warp-uniform
          if (partial) {
            const int64_t other = static_cast<int64_t>((e & kListIndex) * 64 + 32 * ch);
            if constexpr (kDKDV) {
              // this lane's key row as a bit for each of the 32 query rows, then the rows of the lane's elements
              const uint8_t* mp = mask_at + other * p.ds2;
              uint32_t kept = 0;
#pragma unroll
              for (int q = 0; q < 32; ++q) kept |= (__ldg(mp + q * p.ds2) != 0 ? 1u : 0u) << q;
#pragma unroll
              for (int r = 0; r < 4; ++r) mw[r] = __shfl_sync(0xffffffffu, kept, 8 * r + (lane >> 2)) >> (2 * (lane & 3));
            } else {
              const uint4* mp = reinterpret_cast<const uint4*>(mask_at + other);
#pragma unroll
              for (int q16 = 0; q16 < 2; ++q16) {
                const uint4 a = __ldg(mp + q16);
                mw[4 * q16] = a.x; mw[4 * q16 + 1] = a.y; mw[4 * q16 + 2] = a.z; mw[4 * q16 + 3] = a.w;
              }
            }
          }
        }
        ok = mbar_wait_warp(smem_u32(&sm->x_full[g % kXBars]), (g / kXBars) & 1);
        if (!ok) break;
        tc_fence_after();
        if (active) {
          // 8 columns of 32 rows (dQ) or 16 of 16 (dK/dV) at a time, the next ones on their way from tensor memory
          // meanwhile (straight through all of them the registers do not suffice)
          uint32_t xsb[2][8], xdb[2][8];
          if constexpr (kDKDV) {
            // LSE2 and delta differ from column to column here.  A lane that held all 32 columns of one row read all
            // of both from shared memory, in 16 loads of 16 bytes that all lanes have in common: 347 cycles of
            // shared memory's port a superstep of 1,058.  Two columns in eight of four rows need a quarter.
            const uint64_t* lse2 = reinterpret_cast<const uint64_t*>(&sm->lse[g % kRing0<true>][t_mine][32 * ch + 2 * (lane & 3)]);
            const uint64_t* del2 = reinterpret_cast<const uint64_t*>(&sm->delta[g % kRing1<true>][t_mine][32 * ch + 2 * (lane & 3)]);
            const uint64_t c2 = pack_f32x2(c, c);
            uint64_t neg_l[2], neg_d[2];
            tmem_ld_16x256b_x2(s_at, xsb[0]);
            tmem_ld_16x256b_x2(dp_at, xdb[0]);
#pragma unroll
            for (int n = 0; n < 4; ++n) {  // columns 16 (n / 2), lanes 16 (n % 2)
              uint32_t *xs = xsb[n & 1], *xd = xdb[n & 1], pk_p[4], pk_ds[4];
              if ((n & 1) == 0) {
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                  float l0, l1, d0, d1;
                  unpack_f32x2(lse2[4 * (n + k)], l0, l1);
                  unpack_f32x2(del2[4 * (n + k)], d0, d1);
                  // (-inf: a query row with every element masked.  Every logit it meets is -inf too, and against a
                  // finite stand-in it exponentiates to 0 instead of NaN)
                  if constexpr (kElementMask) l0 = fmaxf(l0, -3.0e38f), l1 = fmaxf(l1, -3.0e38f);
                  neg_l[k] = pack_f32x2(-l0, -l1);
                  neg_d[k] = pack_f32x2(-d0, -d1);
                }
              }
              tc_wait_ld();
              if (partial) {
                // masked elements: logit -inf, so P = 0 and with it dS = 0
#pragma unroll
                for (int e = 0; e < 8; ++e)
                  if ((mw[2 * (n & 1) + ((e >> 1) & 1)] >> (16 * (n >> 1) + 8 * (e >> 2) + (e & 1)) & 1u) == 0) xs[e] = 0xff800000u;
              }
              if (n < 3) {
                const uint32_t next = 16 * ((n + 1) >> 1) + (static_cast<uint32_t>(16 * ((n + 1) & 1)) << 16);
                tmem_ld_16x256b_x2(s_at + next, xsb[(n + 1) & 1]);
                tmem_ld_16x256b_x2(dp_at + next, xdb[(n + 1) & 1]);
              }
#pragma unroll
              for (int e = 0; e < 4; ++e) {  // columns 8 (e / 2), row 8 (e % 2)
                float z0, z1, ds0, ds1;
                unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(xs[2 * e]), __uint_as_float(xs[2 * e + 1])), c2, neg_l[e >> 1]), z0, z1);
                const float p0 = ex2_approx(z0), p1 = ex2_approx(z1);
                const uint64_t diff2 = add_f32x2(pack_f32x2(__uint_as_float(xd[2 * e]), __uint_as_float(xd[2 * e + 1])), neg_d[e >> 1]);
                unpack_f32x2(mul_f32x2(pack_f32x2(p0, p1), diff2), ds0, ds1);
                pk_p[e] = pack_2x16<kBf16>(p0, p1);
                pk_ds[e] = pack_2x16<kBf16>(ds0, ds1);
              }
              const uint32_t to = s_at + 16 * (n >> 1) + (static_cast<uint32_t>(16 * (n & 1)) << 16);
              tmem_st_16x128b_x2(to, pk_p);
              tmem_st_16x128b_x2(to + 8, pk_ds);
            }
          } else {
            // (a row whose elements are all masked has LSE = -inf: as above)
            float my_lse = sm->lse[0][0][vec_at];
            if constexpr (kElementMask) my_lse = fmaxf(my_lse, -3.0e38f);
            const float my_delta = sm->delta[0][0][vec_at];
            tmem_ld_32x32b_x8(s_at, xsb[0]);
            tmem_ld_32x32b_x8(dp_at, xdb[0]);
#pragma unroll
            for (int c8 = 0; c8 < 4; ++c8) {
              uint32_t *xs = xsb[c8 & 1], *xd = xdb[c8 & 1], pk_ds[4];
              tc_wait_ld();
              if (partial) {
#pragma unroll
                for (int q4 = 0; q4 < 2; ++q4) {
                  const uint32_t nz = __vcmpne4(mw[2 * c8 + q4], 0u);
#pragma unroll
                  for (int bb = 0; bb < 4; ++bb) {
                    const uint32_t keep = __byte_perm(nz, 0u, 0x1111u * bb);
                    xs[4 * q4 + bb] = (xs[4 * q4 + bb] & keep) | (0xff800000u & ~keep);
                  }
                }
              }
              if (c8 < 3) {
                tmem_ld_32x32b_x8(s_at + 8 * c8 + 8, xsb[(c8 + 1) & 1]);
                tmem_ld_32x32b_x8(dp_at + 8 * c8 + 8, xdb[(c8 + 1) & 1]);
              }
#pragma unroll
              for (int q = 0; q < 8; q += 2) {
                float z0, z1, ds0, ds1;
                unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(xs[q]), __uint_as_float(xs[q + 1])),
                                       pack_f32x2(c, c), pack_f32x2(-my_lse, -my_lse)),
                             z0, z1);
                const uint64_t diff2 = add_f32x2(pack_f32x2(__uint_as_float(xd[q]), __uint_as_float(xd[q + 1])),
                                                 pack_f32x2(-my_delta, -my_delta));
                unpack_f32x2(mul_f32x2(pack_f32x2(ex2_approx(z0), ex2_approx(z1)), diff2), ds0, ds1);
                pk_ds[q / 2] = pack_2x16<kBf16>(ds0, ds1);
              }
              tmem_st_32x32b_x4(s_at + 16 * (c8 >> 1) + 4 * (c8 & 1), pk_ds);
            }
          }
        } else {
          uint32_t zero[16];
#pragma unroll
          for (int k = 0; k < 16; ++k) zero[k] = 0u;
          tmem_st_32x32b_x16(s_at, zero);
          tmem_st_32x32b_x16(s_at + 16, zero);
        }
        tc_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&sm->d_full[g % kXBars]));
      }
      // (the block's sums are merged and stored by the write-out warps; these warps go straight
      // on to the next block, whose first S/dP is usually complete already)
    }
    if (!ok) bwd_give_up(sm, p.status, 3);
  } else {
    // =========================== write-out ===========================
    // Lane r of an accumulator holds the tile-a sums of row r of the CTA's block, lane r+64 its tile-b
    // sums (zeros when the list has a single tile).  These four warps (lane quarter = warp % 4)
    // take the sums out of tensor memory as soon as the block's last MMAs are complete, so that the
    // next block can start accumulating, then add the two halves, scale, round and store, while the
    // compute warps are already at work on the next block.  dK/dV: lanes 0..63 finish dV and hand
    // over their sums of dK, lanes 64..127 the other way round; dQ: lanes 0..63 finish columns
    // [0, 32), lanes 64..127 columns [32, 64).
    // Each 32 columns take two named barriers, also after a give-up, the second one with the give-up vote
    // (role_leaves); a warp that is told that there is no more work comes to both before it leaves.
    take_registers<kBwdWriteRegs>();
    const int quarter = warp & 3;
    const int half = quarter >> 1;
    const int r_blk = (quarter & 1) * 32 + lane;  // row of the CTA's block
    const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
    constexpr int kKeep = kDKDV ? 64 : 32;        // columns a lane finishes, and hands over
    const uint32_t tm_keep = tmem + lane_base + (kDKDV ? (half ? kTmAcc1 : kTmAcc0) : kTmAcc1 + 32 * half);
    const uint32_t tm_send = tmem + lane_base + (kDKDV ? (half ? kTmAcc0 : kTmAcc1) : kTmAcc1 + 32 - 32 * half);
    const bool first_out = kDKDV && half == 0;    // dV; else dK or dQ
    const float scale = first_out ? 1.0f : p.sm_scale;
    const int col0 = kDKDV ? 0 : 32 * half;
    bool ok = true;
    int ni = 0;
    bwd_begin<kDKDV>(p);
#pragma unroll 1
    for (int i = 0;; ++i) {
      BwdItem it{0, 0, 0, 1, 0};
      if (ok) ok = bwd_next_item(sm, i, lane, &it);
      if (ok && it.b < 0) {  // no more work
        named_barrier_sync(2, 128);
        role_leaves(2, 128, false);
        break;
      }
      const int64_t row = it.blk * 64 + r_blk;
      uint16_t* dst = first_out
                          ? static_cast<uint16_t*>(p.out0) + it.b * p.sb0 + it.h * p.sh0 + row * p.sn0
                          : static_cast<uint16_t*>(p.out1) + it.b * p.sb1 + it.h * p.sh1 + row * p.sn1;
      if (ok && it.n_tiles == 0) {
        // a block with an empty list: zero gradients (the same decision in all four warps)
#pragma unroll 1
        for (int v = col0; v < min(col0 + kKeep, p.D); v += 8)
          *reinterpret_cast<uint4*>(dst + v) = make_uint4(0u, 0u, 0u, 0u);
        continue;
      }
      if (ok) ok = mbar_wait_warp(smem_u32(&sm->acc_done), ni & 1);
      ++ni;
      bool any_failed = false;
      // All sums are taken out of tensor memory before the first exchange, so that the next block may start
      // accumulating.
      uint32_t keep[kKeep], send[32];
      if (ok) {
        tc_fence_after();
#pragma unroll
        for (int q = 0; q < kKeep; q += 32) {
          if (q > 0) bwd_hand_over(sm->xfer[half][r_blk], send);
          tmem_ld_32x32b_x32(tm_send + q, send);
          tmem_ld_32x32b_x32(tm_keep + q, keep + q);
          tc_wait_ld();
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&sm->acc_free));
        if (kKeep == 32) bwd_hand_over(sm->xfer[half][r_blk], send);
      }
#pragma unroll
      for (int q = 0; q < kKeep; q += 32) {
        if (q > 0 && ok) bwd_hand_over(sm->xfer[half][r_blk], send);
        named_barrier_sync(2, 128);
        if (ok) {
          const float4* from = reinterpret_cast<const float4*>(sm->xfer[half ^ 1][r_blk]);
          const int col = col0 + q;
#pragma unroll
          for (int v = 0; v < 32; v += 16) {
            if (col + v < p.D) {
              uint32_t o[8];
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                const float4 x = from[v / 4 + k];
                const uint32_t* mine = keep + q + v + 4 * k;
                o[2 * k] = pack_2x16<kBf16>((__uint_as_float(mine[0]) + x.x) * scale, (__uint_as_float(mine[1]) + x.y) * scale);
                o[2 * k + 1] = pack_2x16<kBf16>((__uint_as_float(mine[2]) + x.z) * scale, (__uint_as_float(mine[3]) + x.w) * scale);
              }
              // 16 columns go out as one whole sector when the rows start on such boundaries
              if (p.wide_stores) {
                st_global_v8(dst + col + v, o);
              } else {
                reinterpret_cast<uint4*>(dst + col + v)[0] = make_uint4(o[0], o[1], o[2], o[3]);
                reinterpret_cast<uint4*>(dst + col + v)[1] = make_uint4(o[4], o[5], o[6], o[7]);
              }
            }
          }
        }
        // xfer may be overwritten now; all four warps leave together on a give-up
        any_failed = role_leaves(2, 128, !ok);
        if (any_failed) break;
      }
      if (any_failed) break;
    }
    if (!ok) bwd_give_up(sm, p.status, 3);
  }

  // The next kernel may come as soon as a role of every CTA gets here, warps without a role at once: it waits
  // itself for the end of this one (from the last role on: 1 us later).  Not so when dQ follows that does not
  // wait: it has been let in above.
  if (!(kDKDV && p.together)) grid_dependents_launch();
  tc_fence_before();
  __syncthreads();
  if (warp == kXWarp) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem, kBwdTmemCols);
  }
  // what follows dQ in the stream waits for dQ alone
  if (!kDKDV && p.together) grid_dependency_wait();
}

struct BwdOperand {
  const void* p;
  const int64_t* strides;
};

// q, k, v, dO and the one or two outputs with strides of their own; out0 = dV (dK/dV only), out1 = dK
// or dQ.
template <bool kDKDV>
static int launch_bwd(BwdOperand q, BwdOperand k, BwdOperand v, BwdOperand dout, const float* lse2,
                      const float* delta, BwdOperand out0, BwdOperand out1, const int32_t* list_ptr,
                      const int32_t* list_idx, int list_places, int list_b_stride, int list_h_stride,
                      float sm_scale, int dtype, int B, int H, int N, int D, const uint8_t* dense,
                      const int64_t* dense_strides, int32_t* ticket, int32_t* status, bool together,
                      void* stream) {
  if (B <= 0 || H <= 0 || N <= 0 || (N % kBlock) != 0 || !head_dim_ok(D)) return BSA_ERR_BAD_SHAPE;
  if (dense != nullptr) {
    if (!dense_strides || !is_aligned(dense, 16)) return BSA_ERR_BAD_POINTER;
    if (dense_strides[3] != 1 || dense_strides[2] <= 0 || (dense_strides[2] % 16) != 0 ||
        dense_strides[0] < 0 || dense_strides[1] < 0 || (dense_strides[0] % 16) != 0 ||
        (dense_strides[1] % 16) != 0)
      return BSA_ERR_BAD_STRIDE;
    if (!(sm_scale > 0.f)) return BSA_ERR_BAD_SHAPE;
  }
  if (dtype != BSA_F16 && dtype != BSA_BF16) return BSA_ERR_BAD_DTYPE;
  if (!lse2 || !delta || !list_ptr || !list_idx || !is_aligned(lse2, 16) || !is_aligned(delta, 16))
    return BSA_ERR_BAD_POINTER;
  int rc;
  if (!kDKDV) out0 = out1;
  for (const BwdOperand& op : {q, k, v, dout, out0, out1})
    if ((rc = check_qkv_operand(op.p, op.strides)) != BSA_OK) return rc;
  if ((rc = check_device_sm100()) != BSA_OK) return rc;
  const int nb = N / kBlock;
  if (list_places != 0 && list_places != nb) return BSA_ERR_BAD_SHAPE;
  if (static_cast<int64_t>(B) * H * nb > 0x7fffffffLL) return BSA_ERR_TOO_LARGE;

  // dK/dV: K, V resident; Q, dO streamed.   dQ: Q, dO resident; K, V streamed.
  CUtensorMap tm_q, tm_k, tm_v, tm_do;
  if ((rc = cached_qkv_tmap(&tm_q, q.p, q.strides, B, H, N, D, dtype)) != BSA_OK) return rc;
  if ((rc = cached_qkv_tmap(&tm_k, k.p, k.strides, B, H, N, D, dtype)) != BSA_OK) return rc;
  if ((rc = cached_qkv_tmap(&tm_v, v.p, v.strides, B, H, N, D, dtype)) != BSA_OK) return rc;
  if ((rc = cached_qkv_tmap(&tm_do, dout.p, dout.strides, B, H, N, D, dtype)) != BSA_OK) return rc;

  BwdParams prm;
  prm.list_ptr = list_ptr;
  prm.list_idx = list_idx;
  prm.list_places = list_places;
  prm.dense = dense;
  prm.ds0 = dense ? dense_strides[0] : 0;
  prm.ds1 = dense ? dense_strides[1] : 0;
  prm.ds2 = dense ? dense_strides[2] : 0;
  prm.lse2 = lse2;
  prm.delta = delta;
  prm.out0 = const_cast<void*>(out0.p);
  prm.out1 = const_cast<void*>(out1.p);
  prm.sb0 = out0.strides[0];
  prm.sh0 = out0.strides[1];
  prm.sn0 = out0.strides[2];
  prm.sb1 = out1.strides[0];
  prm.sh1 = out1.strides[1];
  prm.sn1 = out1.strides[2];
  prm.B = B;
  prm.H = H;
  prm.N = N;
  prm.D = D;
  prm.nb = nb;
  prm.items = B * H * nb;
  prm.list_b_stride = list_b_stride;
  prm.list_h_stride = list_h_stride;
  prm.scale_log2 = sm_scale * 1.4426950408889634f;
  prm.sm_scale = sm_scale;
  prm.status = status;
  prm.ticket = ticket;
  prm.together = together ? 1 : 0;
  {
    // 16 output columns are one 32-byte sector when every row starts on such a boundary
    uintptr_t bits = 0;
    for (const BwdOperand& op : {out0, out1})
      bits |= reinterpret_cast<uintptr_t>(op.p) |
              static_cast<uintptr_t>((op.strides[0] | op.strides[1] | op.strides[2]) * 2);
    prm.wide_stores = (bits & 31u) == 0 ? 1 : 0;
  }

  const size_t smem_bytes = sizeof(BwdSmem);
  auto kern = dense != nullptr ? (dtype == BSA_BF16 ? attn_bwd_kernel<true, kDKDV, true>
                                                    : attn_bwd_kernel<false, kDKDV, true>)
                               : (dtype == BSA_BF16 ? attn_bwd_kernel<true, kDKDV, false>
                                                    : attn_bwd_kernel<false, kDKDV, false>);
  if ((rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem_bytes, kBwdLaunchRegs)) != BSA_OK)
    return rc;
  int sms = 0;
  if ((rc = sm_count(&sms)) != BSA_OK) return rc;
  const dim3 grid(static_cast<unsigned>(prm.items < sms ? prm.items : sms));  // one CTA per SM
  return launch_dependent(kern, grid, kBwdThreads, smem_bytes, static_cast<cudaStream_t>(stream),
                          kDKDV ? tm_k : tm_q, kDKDV ? tm_v : tm_do, kDKDV ? tm_q : tm_k,
                          kDKDV ? tm_do : tm_v, prm);
}

}  // namespace bsa

extern "C" int bsa_attn_bwd_dkdv_strided(
    const void* q, const int64_t q_strides[4], const void* k, const int64_t k_strides[4],
    const void* v, const int64_t v_strides[4], const void* dout, const int64_t do_strides[4],
    const float* lse2, const float* delta, void* dk, const int64_t dk_strides[4], void* dv,
    const int64_t dv_strides[4], const int32_t* col_ptr, const int32_t* row_idx, int list_places,
    int list_b_stride, int list_h_stride, float sm_scale, int dtype, int B, int H, int N, int D, const uint8_t* dense,
    const int64_t dense_strides[4], int32_t* work_counter, int32_t* status, void* stream) {
  if (!q_strides || !k_strides || !v_strides || !do_strides || !dk_strides || !dv_strides)
    return BSA_ERR_BAD_POINTER;
  return bsa::launch_bwd<true>({q, q_strides}, {k, k_strides}, {v, v_strides}, {dout, do_strides},
                               lse2, delta, {dv, dv_strides}, {dk, dk_strides}, col_ptr, row_idx,
                               list_places, list_b_stride, list_h_stride, sm_scale, dtype, B, H, N, D, dense,
                               dense_strides, work_counter, status, false, stream);
}

extern "C" int bsa_attn_bwd_dkdv(const void* q, const void* k, const void* v, const void* dout,
                                 const int64_t strides[4], const float* lse2, const float* delta,
                                 void* dk, void* dv, const int32_t* col_ptr,
                                 const int32_t* row_idx, int list_b_stride, int list_h_stride,
                                 float sm_scale, int dtype, int B, int H, int N, int D,
                                 const uint8_t* dense, const int64_t dense_strides[4],
                                 int32_t* work_counter, int32_t* status, void* stream) {
  return bsa_attn_bwd_dkdv_strided(q, strides, k, strides, v, strides, dout, strides, lse2, delta, dk,
                                   strides, dv, strides, col_ptr, row_idx, 0, list_b_stride,
                                   list_h_stride, sm_scale, dtype, B, H, N, D, dense, dense_strides,
                                   work_counter, status, stream);
}

extern "C" int bsa_attn_bwd_dq_strided(
    const void* q, const int64_t q_strides[4], const void* k, const int64_t k_strides[4],
    const void* v, const int64_t v_strides[4], const void* dout, const int64_t do_strides[4],
    const float* lse2, const float* delta, void* dq, const int64_t dq_strides[4],
    const int32_t* row_ptr, const int32_t* col_idx, int list_places, int list_b_stride, int list_h_stride,
    float sm_scale, int dtype, int B, int H, int N, int D, const uint8_t* dense,
    const int64_t dense_strides[4], int32_t* work_counter, int32_t* status, void* stream) {
  if (!q_strides || !k_strides || !v_strides || !do_strides || !dq_strides) return BSA_ERR_BAD_POINTER;
  return bsa::launch_bwd<false>({q, q_strides}, {k, k_strides}, {v, v_strides}, {dout, do_strides},
                                lse2, delta, {nullptr, nullptr}, {dq, dq_strides}, row_ptr, col_idx,
                                list_places, list_b_stride, list_h_stride, sm_scale, dtype, B, H, N, D, dense,
                                dense_strides, work_counter, status, false, stream);
}

extern "C" int bsa_attn_bwd_dq(const void* q, const void* k, const void* v, const void* dout,
                               const int64_t strides[4], const float* lse2, const float* delta,
                               void* dq, const int32_t* row_ptr, const int32_t* col_idx,
                               int list_b_stride, int list_h_stride, float sm_scale, int dtype,
                               int B, int H, int N, int D, const uint8_t* dense,
                               const int64_t dense_strides[4], int32_t* work_counter,
                               int32_t* status, void* stream) {
  return bsa_attn_bwd_dq_strided(q, strides, k, strides, v, strides, dout, strides, lse2, delta, dq,
                                 strides, row_ptr, col_idx, 0, list_b_stride, list_h_stride, sm_scale,
                                 dtype, B, H, N, D, dense, dense_strides, work_counter, status, stream);
}

extern "C" int bsa_attn_bwd_strided(
    const void* q, const int64_t q_strides[4], const void* k, const int64_t k_strides[4],
    const void* v, const int64_t v_strides[4], const void* dout, const int64_t do_strides[4],
    const float* lse2, const float* delta, void* dq, const int64_t dq_strides[4], void* dk,
    const int64_t dk_strides[4], void* dv, const int64_t dv_strides[4], const int32_t* row_ptr,
    const int32_t* col_idx, const int32_t* col_ptr, const int32_t* row_idx, int list_places,
    int list_b_stride, int list_h_stride, float sm_scale, int dtype, int B, int H, int N, int D,
    const uint8_t* dense, const int64_t dense_strides[4], int32_t* dkdv_counter, int32_t* dq_counter,
    int32_t* status, void* stream) {
  if (!q_strides || !k_strides || !v_strides || !do_strides || !dq_strides || !dk_strides || !dv_strides ||
      (dkdv_counter != nullptr && dkdv_counter == dq_counter))
    return BSA_ERR_BAD_POINTER;
  const int rc = bsa::launch_bwd<true>({q, q_strides}, {k, k_strides}, {v, v_strides}, {dout, do_strides},
                                       lse2, delta, {dv, dv_strides}, {dk, dk_strides}, col_ptr, row_idx,
                                       list_places, list_b_stride, list_h_stride, sm_scale, dtype, B, H, N, D,
                                       dense, dense_strides, dkdv_counter, status, true, stream);
  if (rc != BSA_OK) return rc;
  return bsa::launch_bwd<false>({q, q_strides}, {k, k_strides}, {v, v_strides}, {dout, do_strides}, lse2, delta,
                                {nullptr, nullptr}, {dq, dq_strides}, row_ptr, col_idx, list_places,
                                list_b_stride, list_h_stride, sm_scale, dtype, B, H, N, D, dense, dense_strides,
                                dq_counter, status, true, stream);
}
