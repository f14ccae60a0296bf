// Decode matmul for up to 32 token rows: out = epilogue(alpha * x @ W + add), W block-float in streaming layout,
// and a queue of such matmuls run by ONE launch.
//
// The work is bound by HBM: every packed weight byte is read once, by a bulk (TMA) copy into a ring of
// shared-memory stages, and dequantised in registers on its way into a bf16 MMA with fp32 accumulators.
//
// Lists of small matmuls for a few tokens, where the way from one result to the next is all that counts, have a kernel of
// their own at the end of this file (chain_kernel). All others run in gemv_queue_kernel:
//
// A queue. In decode one matmul's result is the next one's x, so between two of them the GPU has nothing to read
// unless the next weights are already on their way. The kernel therefore takes a list of matmuls (up to kQueueMax
// per launch) and runs them in order with the same persistent CTAs. The weight warp of a CTA walks the whole list:
// weight copies depend on nothing and go out as soon as the ring has room, across the boundary between two matmuls.
// Only x waits: the x warp copies a matmul's activations once the last earlier matmul that this one depends on, and all
// before that one, are complete: every sub-panel reported finished (a counter per matmul in global memory, read with acquire
// semantics; see Gate on the host side, which works out the dependences from the buffer addresses). Matmuls that do not
// depend on one another overlap, two in flight at most. While that report travels, the ring fills with the next weights:
// 190 KB per SM, 28 MB in all, over 4 us of HBM.
//
// Decomposition ("stream-K"). A weight matrix is cut into sub-panels of 4 tile columns (one run of the streaming
// layout). A unit is one tile row of one sub-panel. Units are numbered sub-panel by sub-panel and dealt out in
// contiguous ranges to the CTAs, one per SM: equal shares of all CTAs, so every SM streams the same number of bytes
// whatever the shape, or, for small matmuls, whole sub-panels. A sub-panel that several CTAs share is finished by the
// CTA that holds its last tile row: the others write their fp32 partial sums to scratch, where a word is zero until its
// sum is there; the owner, which takes that sub-panel last, waits for the words (with a limit), adds them in CTA order, so
// results do not depend on timing, and runs the epilogue. Contributors never wait, so the owner's wait always ends; it is bounded
// all the same.
//
// Inside a CTA: two producer warps fill the ring, 16 consumer warps empty it. For one weight matrix a consumer warp has
// one column of the sub-panel and every fourth tile row of a stage; for a gate/up pair one column of one of the two
// matrices and every other tile row. When the CTA's part of a sub-panel ends the warps leave their sums in shared
// memory and all 512 threads add them up and run the epilogue element by element. One CTA of 16 warps per SM rather
// than two of 8: half the reports, polls and partial sums, and twice the bytes per copy. A weight tile is
// four 16x16 faces; a face is one m16n8k16 MMA with the face's 16 output channels as the MMA's rows, 16 input
// channels as its K and up to 8 tokens as its columns. The 16 weights of a face row share an exponent e; how the
// packed bytes become weights is described at tile_mma.
#include "common.cuh"
#include "expand.cuh"
#include "tmap.cuh"
#include <algorithm>
#include <cstring>
#include <mutex>

using namespace bt;

namespace {

constexpr int kWC = kPanel;                 // tile columns of a run of the streaming layout, and of a sub-panel but for small matmuls
constexpr int kCW = 16;                     // consumer warps of the CTA; an SM holds one CTA
constexpr int kConsumers = kCW * 32;
constexpr int kThreads = (kCW + 3) * 32;    // plus two producer warps and a messenger
constexpr int kBars = 16;                   // stages in the ring at most: mbarriers that go round with the stages
constexpr int kMaxCtas = 160;               // one CTA per SM; a B200 has 148
constexpr int kMaxSubPanels = 16384;
constexpr int kQueueMax = 32;               // matmuls per launch; longer lists take several launches
constexpr uint32_t kSpinLimit = 1u << 14;   // attempts of up to 100 us each (mbarriers) or polls x 64 (counters)

// Shared memory of a CTA: mbarriers and notes, the sums on their way through the CTA, then the ring.
constexpr int kSmFull = 0, kSmEmpty = 128;  // mbarriers: a stage's weights and x have landed; it is free again
constexpr int kSmHeld = 256;                // uint32[2][kBars]: ring bytes of each stage in the ring, as each producer warp noted them
constexpr int kSmDead = 384;                // int: a wait on a stage gave up; nobody in this CTA waits for the ring any more
constexpr int kSmEpoch = 388;               // chains: uint32, the launch's number
constexpr int kSmReady = 392, kSmGo = 400, kSmDone = 416;   // chains: mbarriers: the launch's number is there; [2] a matmul may start; [2] its results are stored
constexpr int kSmStages = 512;              // Stage[kBars]: what the weight warp tells the consumers about each stage
constexpr int kSmSums = 1024;               // float[k groups x matrices, or tile rows x matrices][tokens][channels of a sub-panel + 4]
// Floats from one token's channels to the next: 4 past the channels, so that the fragment stores meet no bank twice.
__host__ __device__ constexpr int sum_stride(int lw) { return (32 << lw) + 4; }
constexpr int sums_bytes(int tg) { return 4 * 8 * tg * sum_stride(2) * 4; }
constexpr int kSmallSums = 84 * 1024;       // bytes at most that the sums of a small matmul's tile rows take of the ring
__host__ __device__ constexpr int small_groups(int lw, bool pair) { return kCW >> lw >> (pair ? 1 : 0); }   // warps that share a column (of a matrix)
constexpr int kSmemBytes = 227 * 1024;

// Scratch layout (byte offsets into the caller's workspace). Two matmuls of a queue may be in flight at once, so
// what a matmul uses while it runs exists twice (a set for even and one for odd positions in the queue).
constexpr size_t kWsError = 0;                                   // int: set to nonzero when a wait gave up
constexpr size_t kWsOpsDone = 8;                                 // int[kQueueMax]: finished sub-panels of each matmul of the launch
constexpr size_t kWsAllDone = 144;                               // int: and of all of them
constexpr size_t kWsEpoch = 148;                                 // uint32: launches of chains that used this workspace so far, modulo kEpochs
constexpr size_t kWsSets = 256;                                  // the sets start here
constexpr size_t kSetPanelsDone = 0;                             // int: sub-panels finished (argmax epilogue)
constexpr size_t kSetKeys = 256;                                 // u64[32]: per token the best (value, column) so far (argmax epilogue)
constexpr size_t kSetCounters = 512;                             // int[kMaxSubPanels]: CTAs arrived at a sub-panel
constexpr size_t kSetPartials = kSetCounters + 4 * kMaxSubPanels;
constexpr size_t kSlotFloatsMax = 32 * 2 * 128;                  // 32 tokens x up to two matrices x 128 channels
constexpr size_t kSetBytes = kSetPartials + (size_t)kMaxCtas * kSlotFloatsMax * 4;
constexpr int kSets = 2;                                         // matmuls of a queue in flight at most
constexpr size_t kWsExchange = (kWsSets + kSets * kSetBytes + 255) / 256 * 256;   // kExchanges results on their way to the next matmul of a chain
constexpr int kExchanges = 3, kChainRows = 8;                    // chains are for up to 8 tokens
constexpr size_t kExchangeBytes = (size_t)kMaxCtas * kWC * 2 * kChainRows * 64;
constexpr size_t kWsBytes = kWsExchange + kExchanges * kExchangeBytes;
constexpr uint32_t kEpochs = 1u << 26;

// The shape of a stage for one kind of matmul: format, one matrix or a gate/up pair, token groups of 8 rows, columns of a
// sub-panel (1 << lw).
struct Geometry {
  int tb;        // bytes of a packed tile
  int ups;       // units (tile rows) per stage
  int matrix;    // bytes of one matrix's part of a stage
  int w_bytes;   // all weights of a stage; the x tiles follow
  int xb;        // bytes of an x tile staged: token rows 0-7, 0-15 or all
  int stage;     // bytes of a stage
};
// Tile rows a warp takes per stage. Large stages: a stage costs its waits, arrivals and copies whatever its size, about
// 430 cycles of a warp's time on an 8192 x 28672 matmul, and a ring of three or four stages of 35-55 KB is enough to cover
// the latency of HBM. In narrow sub-panels, whose rows go round more warps, x would outgrow the weights.
__host__ __device__ constexpr int stage_rows_per_warp(int fmt, int tg, int lw) {
  return lw == 2 ? (fmt == BT_BFP4 && tg < 4 ? 4 : 2) : lw == 1 ? (tg == 4 ? 1 : 2) : tg == 1 ? 2 : 1;
}
__host__ __device__ constexpr Geometry geometry(int fmt, bool pair, int tg, int lw) {
  Geometry g{};
  g.tb = tile_bytes(fmt);
  g.ups = (kCW >> lw >> (pair ? 1 : 0)) * stage_rows_per_warp(fmt, tg, lw);
  g.matrix = (g.ups << lw) * g.tb;
  g.w_bytes = (pair ? 2 : 1) * g.matrix;
  g.xb = 512 * tg;
  g.stage = g.w_bytes + g.ups * g.xb;
  return g;
}
static_assert(geometry(BT_BFP8, false, 1, 2).w_bytes % 128 == 0 && geometry(BT_BFP4, true, 4, 2).matrix % 128 == 0 && geometry(BT_BFP4, true, 2, 0).matrix % 128 == 0 &&
              geometry(BT_BFP8, true, 4, 1).matrix % 128 == 0 && geometry(BT_BFP4, true, 4, 0).matrix % 128 == 0, "tiled copies land on 128-byte boundaries");

// One matmul of the queue, as the kernel sees it.
struct alignas(64) GemvParams {
  CUtensorMap xmap;           // x as (16-datum face rows of the staged tokens, faces, tile columns)
  CUtensorMap wmap[2];        // for sub-panels narrower than a run: the weights as (a tile's bytes, the four tiles of a run's tile row, tile rows)
  const uint8_t *w[2];
  const uint16_t *add;
  void *out;
  float *arg_val;
  int *arg_idx;
  float alpha;
  int arg_base, M, KT, TC, epi, out_fp32;
  int fmt, pair, tg;
  int wait_for, wait_panels;  // the last matmul of the launch that must be complete before this one starts (-1: none), and its sub-panels
  int wait_also, also_panels; // the one before it, where its being complete does not follow (see Gate), and its sub-panels
  int turn;                   // CTA c takes the unit range (c + turn) % CTAs
  int lw, panels;             // tile columns of a sub-panel are 1 << lw, and there are so many sub-panels
  int tiled;                  // wmap is used
  int small;                  // every tile row's sums are kept apart and added in order at the end
  int units;                  // tile rows of all sub-panels
  int active;                 // CTAs with a range
  int parts;                  // > 0: every sub-panel is cut into so many ranges; 0: ranges of equal size whatever they straddle,
  int share, extra;           // range b then starts at b * share + min(b, extra), and the last one ends at units
  // what chains have beside it, behind what the general kernel reads (between its fields these cost independent small matmuls 2 %: 2.66 us each for 2.60)
  const uint16_t *x;          // chains read it themselves, where it does not come from an exchange
  int from;                   // chains: x is the result of the matmul before this one and comes from its exchange
  int add_from;               // so does the addend
  int to;                     // chains: the matmul after this one reads the exchange
  int early, early_panels;    // with `from`: what must be complete before this one stores anything, as wait_for and
  int early_also, early_also_panels;   // wait_also without it
};

// The kernel exists for lists with a small matmul in them and for lists without one, which is spared all that sub-panels
// of other widths than four take (as one kernel it cost lists of large matmuls 2-3 %); each for short and for long lists (see
// kQueueShort).
template <bool SMALL> __device__ __forceinline__ int lw_of(const GemvParams &p) { return SMALL ? p.lw : 2; }

// Where sub-panel `sp` lies: 1 << lw tile columns from `col` on, fewer at the end of a matrix, part of a run of `run_width`.
template <bool SMALL> struct Columns {
  int run, run_width, col, width;
  __device__ __forceinline__ Columns(const GemvParams &p, int sp) {
    const int lw = lw_of<SMALL>(p);
    run = sp >> (2 - lw), col = run * kWC + ((sp & ((1 << (2 - lw)) - 1)) << lw);
    run_width = min(kWC, p.TC - run * kWC), width = min(1 << lw, p.TC - col);
  }
};

// Waits for a phase of a stage's mbarrier, with a limit. A wait that gives up marks the CTA: its sums are worthless from
// there on (the error word says so), but every warp still goes through all of its pieces and barriers, without waiting
// for the ring, so that the CTA ends.
__device__ __forceinline__ bool stage_wait(uint32_t smem, uint32_t bar, uint32_t parity, int *error) {
  if (mbar_try_wait(bar, parity, 100000u)) return true;
  for (uint32_t i = 0; i < 2 * kSpinLimit && lds32(smem + kSmDead) == 0; i++)
    if (mbar_try_wait(bar, parity, 100000u)) return true;
  sts32(smem + kSmDead, 1);
  atomicExch(error, 2);
  return false;
}

// What a matmul uses while it runs: the count of finished sub-panels and the per-token best keys (argmax), the
// arrivals per sub-panel (all zero before first use; the kernel leaves them zero) and one slot of partial sums per CTA.
struct Scratch {
  int *panels_done, *counters;
  unsigned long long *keys;   // per token the best (value, column) so far, as an ordered key; zero: nothing yet
  float *partials;
};

// What one launch gets: the matmuls and the scratch they share: a wait-gave-up flag, the counts of finished sub-panels of
// each matmul and of the launch (zero before first use; the kernel leaves them zero) and one or two sets of running scratch.
struct QueueHead {
  int n;
  int sets;                   // kSets: matmuls take the sets in turn, and as many may be in flight; 1: one after the other
  int *error, *ops_done, *all_done;
  uint32_t *epoch;            // the launch's number, with `exchange`
  uint8_t *exchange;          // or null
  int panels;                 // sub-panels of all matmuls
  Scratch set[kSets];
  int slot_floats;            // floats between two CTAs' slots of partial sums
  int ring;                   // where the ring starts in shared memory
  int ring_bytes;
};
// A launch's parameters travel with it, and 16 KB of them cost it about a microsecond, so short lists have a kernel of their own.
constexpr int kQueueShort = 8;
template <int OPS> struct Queue : QueueHead {
  GemvParams op[OPS];
};

// A stage as the consumers see it, written by the weight warp ahead of its arrival on the stage's barrier: where a warp
// goes next is worked out once per CTA, not by 16 warps.
struct alignas(32) Stage {
  uint32_t at;                // shared-memory address of its weights; the x tiles follow the matmul's w_bytes further
  int rows, width;            // tile rows, and tile columns of the sub-panel
  int ends;                   // bits 0-1: 1, the CTA's part of the sub-panel ends with it; 3, and so does its part of the matmul; bit 2: all rows,
                              // four columns; from bit 3 on the first tile row
  int sp, first, cta, end;    // the sub-panel, the first range that shares it, this CTA's and the last one, the owner
};
static_assert(sizeof(Stage) * kBars <= kSmSums - kSmStages, "room for the stages' notes");

__device__ __forceinline__ int range_start(const GemvParams &p, int b) {
  if (p.parts > 0) return b / p.parts * p.KT + b % p.parts * p.KT / p.parts;
  return min(b * p.share + min(b, p.extra), p.units);
}
// The CTA whose (non-empty) range holds unit u.
__device__ __forceinline__ int cta_of(const GemvParams &p, int u) {
  if (p.parts > 0) return u / p.KT * p.parts + ((u % p.KT + 1) * p.parts - 1) / p.KT;
  const int longer = p.extra * (p.share + 1);
  return u < longer ? u / (p.share + 1) : p.extra + (u - longer) / p.share;
}

// One weight tile times the staged x tile. `tile`, `ex` and `xs` are shared-memory addresses that already include
// the lane's own offsets: tile = tile base + 16 * lane; ex = tile base + 16 * t, where the lane's exponents are;
// xs = x tile base + 32 * g + 8 * t (g = lane / 4, t = lane % 4).
//
// A weight byte (offset binary, see stream_layout.cuh) zero-extended into a 16-bit lane is the bf16 number
// byte * 2^-133, so a mask (bytes 0 and 2 of a word: the lane's first k pair) or a byte-permute (bytes 1 and 3: its
// second pair) makes a register of two weights. A face (16 k x 16 n) is one MMA, rows g and g + 8 of it the channels 2g
// and 2g + 1; acc[fs][tg] collects face column fs. A bfp4 byte holds two channels of the
// same k: rows g of its MMA are the whole byte, 16 * high + low, rows g + 8 the masked low nibble, and the high channel
// is the difference, taken once per sub-panel (one mask less per word than two masked nibbles).
//
// Where the face row's power of two goes depends on how many tokens share it. Up to 16 tokens (TG 1 and 2) it goes to
// x: the MMA's two x registers per 8 tokens are multiplied by 2^(e - 127), exactly unless the product with a weight
// of that run leaves bf16's range, and the four weight registers take one multiply-add with constants that makes
// them the signed integers times 2^-6, whatever the run. With 32 tokens eight x
// registers would need it per face and the weights only four, so there the weights carry it: one packed
// multiply-add with s = 2^(e - 64) and with -offset * 2^-133 * s makes them the weights times 2^-64, which the epilogue
// undoes. On shared-memory data alone, 16 warps, an SM does a tile in 23 (8 tokens), 32 (16) and 47-50 cycles
// (32): 68 instructions, of which an MMA holds the tensor pipe for about 10 cycles, so the bound is instructions. Weights
// that carry the scale take 24 / 27 (bfp8 / bfp4) for 8 tokens, x that carries it 52 for 32, and subtracting the offset
// with a second MMA instead of the multiply-adds 26-28 for 8.
constexpr uint32_t kByteLanes = 0x00FF00FFu, kNibbleLanes = 0x000F000Fu, kOddBytes = 0x4341u;
constexpr uint32_t kMinus128 = 0x80808080u;   // two bf16 lanes of -128 * 2^-133 = -2^-126
constexpr uint32_t kMinus136 = 0x80888088u;   // -(128 + 8) * 2^-133: offset of a byte made of two offset nibbles
constexpr uint32_t kMinus8 = 0x80088008u;     // -8 * 2^-133
constexpr uint32_t kTo6 = 0x7F007F00u;                                              // 2^127: code * 2^-133 to code * 2^-6
constexpr uint32_t kOff128 = 0xC000C000u, kOff136 = 0xC008C008u, kOff8 = 0xBE00BE00u;   // the same offsets times 2^-6
__host__ __device__ constexpr bool scale_on_x(int tg) { return tg <= 2; }
__host__ __device__ constexpr float unscale_of(int tg) { return scale_on_x(tg) ? 1.f : 18446744073709551616.f; }   // 2^64
template <int FMT, int TG>
__device__ __forceinline__ void tile_mma(uint32_t tile, uint32_t ex, uint32_t xs, float (&acc)[2][TG][4]) {
  constexpr bool SX = scale_on_x(TG);
  const uint4 ev = lds128(ex);
  const uint32_t ee[4] = {ev.x, ev.y, ev.z, ev.w};
  uint2 bx[2][TG];
#pragma unroll
  for (int h = 0; h < 2; h++) {
#pragma unroll
    for (int tg = 0; tg < TG; tg++) bx[h][tg] = lds64(xs + (TG == 1 ? h * 256 : (tg >> 1) * 1024 + h * 512 + (tg & 1) * 256));
  }
  uint4 wv[2];
  wv[0] = lds128(tile + 64);
  if (FMT == BT_BFP8) wv[1] = lds128(tile + 64 + 512);
#pragma unroll
  for (int h = 0; h < 2; h++) {
#pragma unroll
    for (int fs = 0; fs < 2; fs++) {
      const uint32_t e = ee[2 * h + fs];
      const uint32_t s01 = SX ? (e << 7) & 0x7F807F80u : scale_pair<0>(e), s23 = SX ? (e >> 1) & 0x7F807F80u : scale_pair<1>(e);
      uint32_t a0, a1, a2, a3;
      if (FMT == BT_BFP8) {
        const uint32_t w0 = fs ? wv[h].z : wv[h].x, w1 = fs ? wv[h].w : wv[h].y;   // channels 2g and 2g + 1
        const uint32_t m01 = SX ? kTo6 : s01, m23 = SX ? kTo6 : s23, n01 = SX ? kOff128 : mul_bf16x2(s01, kMinus128), n23 = SX ? kOff128 : mul_bf16x2(s23, kMinus128);
        a0 = fma_bf16x2(w0 & kByteLanes, m01, n01), a1 = fma_bf16x2(w1 & kByteLanes, m01, n01);
        a2 = fma_bf16x2(prmt(w0, 0u, kOddBytes), m23, n23), a3 = fma_bf16x2(prmt(w1, 0u, kOddBytes), m23, n23);
      } else {
        const uint32_t w = h ? (fs ? wv[0].w : wv[0].z) : (fs ? wv[0].y : wv[0].x), w01 = w & kByteLanes, w23 = prmt(w, 0u, kOddBytes);
        const uint32_t m01 = SX ? kTo6 : s01, m23 = SX ? kTo6 : s23;
        a0 = fma_bf16x2(w01, m01, SX ? kOff136 : mul_bf16x2(s01, kMinus136)), a1 = fma_bf16x2(w01 & kNibbleLanes, m01, SX ? kOff8 : mul_bf16x2(s01, kMinus8));
        a2 = fma_bf16x2(w23, m23, SX ? kOff136 : mul_bf16x2(s23, kMinus136)), a3 = fma_bf16x2(w23 & kNibbleLanes, m23, SX ? kOff8 : mul_bf16x2(s23, kMinus8));
      }
#pragma unroll
      for (int tg = 0; tg < TG; tg++) {
        const uint32_t b0 = SX ? mul_bf16x2(bx[h][tg].x, s01) : bx[h][tg].x, b1 = SX ? mul_bf16x2(bx[h][tg].y, s23) : bx[h][tg].y;
        mma_bf16(acc[fs][tg], a0, a1, a2, a3, b0, b1);
      }
    }
  }
}

// (value, column) as one number whose order is the pick's: larger value first, of equal values (-0 equals 0) the lower
// column. Zero is "nothing": a NaN, which never wins, maps to it, and no other value does (-inf maps to 0x007FFFFF in
// the upper half).
__device__ __forceinline__ unsigned long long pick_key(float v, int column) {
  if (v != v) return 0ull;
  uint32_t b = __float_as_uint(v == 0.f ? 0.f : v);
  b ^= b >> 31 ? 0xFFFFFFFFu : 0x80000000u;
  return (unsigned long long)b << 32 | (0xFFFFFFFFu - (uint32_t)column);
}

// ---- a sub-panel's end: the CTA's warps, then the CTAs that share it ---------------------------------------------
// The warps have left their sums in shared memory, [k group][matrix][token][channel]. Every consumer thread takes
// one pair of neighbouring channels and every eighth token (or sixteenth, or thirty-second), adds the k groups in order and either stores the sums
// in the CTA's slot of partial sums (a contributor) or adds the contributors' slots in CTA order, so that results do
// not depend on timing, and runs the epilogue (the sub-panel's owner). Elementwise over 512 threads: one small piece of
// code for every kind of matmul. Everybody waits for it, so what counts is its chain of dependent steps and the
// instructions that 16 warps issue (as plain loops over groups, contributors and all 32 rows it took 3000-5000 cycles).
//
// Partial sums carry their own signal: a word of a slot is zero until it is there (a zero sum is sent as -0, and the
// reader adds +0 at the end), the owner's threads poll the words they need and put zeros back. A counter released by
// the contributor and acquired by the owner took about 1.2 us more.
struct Piece {
  int sp;                  // the sub-panel
  int first, last, me;     // the ranges that share it, and this CTA's
  int toks;                // tokens whose sums are in shared memory: M rounded up to whole groups of 8
};
constexpr int kSlots = 4;  // words of contributors' slots that a thread has in flight together
__device__ __forceinline__ void send(float *to, float2 v) {
  const uint32_t x = __float_as_uint(v.x), y = __float_as_uint(v.y);
  st_relaxed2(to, make_uint2(x ? x : 0x80000000u, y ? y : 0x80000000u));
}
// The rows past M of an owner's tiles are zeros; they need no sums, so the messenger writes them while the others work.
template <bool SMALL> __device__ __forceinline__ void zero_rows(const GemvParams &p, int sp) {
  const int M = p.M, lane = threadIdx.x & 31;
  if (M == 1 || p.epi == BT_EPI_ARGMAX || p.out_fp32 == 2) return;
  const Columns<SMALL> at(p, sp);
  const int per_row = p.out_fp32 ? 4 : 2;                                           // 16-byte words of a face row
  for (int face = 0; face < 4 * at.width; face++) {                                 // two lower and two upper faces of each tile
    uint4 *rows = static_cast<uint4 *>(p.out) + ((size_t)at.col * 4 + face) * 16 * per_row;
    for (int i = max(M - (face & 2) * 8, 0) * per_row + lane; i < 16 * per_row; i += 32) rows[i] = make_uint4(0, 0, 0, 0);
  }
}
// Where the pair of channels `pr` of a sub-panel, in tile column `tcol`, has row r in the result's tiles: a datum's index, as in an addend's.
__device__ __forceinline__ int pair_place(int tcol, int pr, int r) { return tcol * 1024 + ((r >> 4) * 2 + (pr >> 3 & 1)) * 256 + (r & 15) * 16 + (2 * pr & 15); }
// A pair of neighbouring channels of one token to the result; n0 is the first of them. Neighbouring lanes have neighbouring pairs of the same token.
// end_piece is on the way from one matmul to the next, where code and parameters are fetched anew every time, so what it has at hand comes
// as it is: `live` as an expression for every use of it, n0, the pointer. With one flag worked out before and the rest taken from the parameters
// behind the barrier the way between two small matmuls took 0.5 us more (3 rows of 8192 x 64 and back, 6.3 us a matmul against 5.8).
template <class Live> __device__ __forceinline__ void store_pair(const GemvParams &p, char *out, int fp32, int M, int tcol, int pr, int n0, int row, Live live, float2 v) {
  const uint32_t both = bf16_half_up(v.x) | bf16_half_up(v.y) << 16;
  if (fp32 == 2) {
    // row-major fp32, only the rows there are: partial sums on their way to an all-reduce
    if (live()) *reinterpret_cast<float2 *>(out + 4 * ((size_t)row * (p.TC * 32) + n0)) = v;
  } else if (M > 1) {
    if (live() && fp32) *reinterpret_cast<float2 *>(out + 4 * (size_t)pair_place(tcol, pr, row)) = v;
    else if (live()) *reinterpret_cast<uint32_t *>(out + 2 * (size_t)pair_place(tcol, pr, row)) = both;
  } else if (fp32) {
    // a one-row result repeats across its tile
    for (int r = 0; live() && r < 32; r++) *reinterpret_cast<float2 *>(out + 4 * (size_t)pair_place(tcol, pr, r)) = v;
  } else {
    // the same: four lanes put half a face row together, and each of them writes it to eight of the rows
    uint4 half;
    half.x = __shfl_sync(0xFFFFFFFFu, both, 0, 4), half.y = __shfl_sync(0xFFFFFFFFu, both, 1, 4);
    half.z = __shfl_sync(0xFFFFFFFFu, both, 2, 4), half.w = __shfl_sync(0xFFFFFFFFu, both, 3, 4);
    if (live()) {
#pragma unroll
      for (int r = 0; r < 32; r += 4) *reinterpret_cast<uint4 *>(out + 2 * (size_t)(pair_place(tcol, pr, r + (pr & 3)) - 2 * (pr & 3))) = half;
    }
  }
}
template <bool SMALL> __device__ __forceinline__ void end_piece(const GemvParams &p, const Scratch &sc, int slot_floats, const float *sums, const Piece &pc, uint32_t smem, int *error) {
  const Columns<SMALL> at(p, pc.sp);
  const int lw = lw_of<SMALL>(p), pairs = 16 << lw, pr = threadIdx.x & (pairs - 1), M = p.M, epi = p.epi, fp32 = p.out_fp32;
  const bool pair = p.pair, owner = pc.me == pc.last;
  const int others = owner ? pc.last - pc.first : 0;                                  // contributors whose sums are to be added
  const int tcol = at.col + (pr >> 4), n0 = at.col * 32 + 2 * pr;                     // tile column and first channel of the pair
  const bool inside = (pr >> 4) < at.width;
  const float unscale = unscale_of(p.tg) * p.alpha;
  const uint16_t *add = owner && inside ? p.add : nullptr;
  char *out = static_cast<char *>(p.out);
  float *slots = sc.partials + (size_t)(owner ? pc.first : pc.me) * slot_floats + 2 * pr;
  const int rows = kConsumers >> (4 + lw), mine = threadIdx.x >> (4 + lw);            // rows at a time, and this thread's among them
  auto addend = [&](int r) { return add && r < M ? __ldcg(reinterpret_cast<const uint32_t *>(add + pair_place(tcol, pr, r))) : 0u; };
  uint32_t a = addend(mine);
  // what the barrier is waited with is worked out and fetched already
  int KT = p.KT, next = M * sum_stride(lw) * (pair ? 2 : 1);
  float scale = unscale;
  asm volatile("" : "+r"(KT), "+r"(next), "+f"(scale), "+l"(out), "+l"(slots) :: "memory");
  named_barrier(1, kConsumers);                                                       // every warp's sums are in place
  uint32_t patience = others && lds32(smem + kSmDead) ? 1 : kSpinLimit * 64;
  for (int row0 = 0; row0 < M; row0 += rows) {
    const int row = row0 + mine;
    const bool live = row < M;
    float2 v = make_float2(0.f, 0.f), u = v;
    if (SMALL && p.small) {
      // one slab of sums per tile row (and matrix): the last row's, then the others' in order, as if every row were a CTA's
      // share: how a matmul is spread over CTAs and warps then has no say in the last bit of a result
      if (live) {
        const float *from = sums + row * sum_stride(lw) + 2 * pr, *last = from + (KT - 1) * next;
        v = *reinterpret_cast<const float2 *>(last);
        if (!pair) {
#pragma unroll 4
          for (int k = 0; k < KT - 1; k++, from += next) {
            const float2 w = *reinterpret_cast<const float2 *>(from);
            v.x += w.x, v.y += w.y;
          }
        } else {
          u = *reinterpret_cast<const float2 *>(last + next / 2);
#pragma unroll 4
          for (int k = 0; k < KT - 1; k++, from += next) {
            const float2 w = *reinterpret_cast<const float2 *>(from), x = *reinterpret_cast<const float2 *>(from + next / 2);
            v.x += w.x, v.y += w.y, u.x += x.x, u.y += x.y;
          }
        }
      }
    } else if (live) {
      // four slabs: k groups of one matrix, or two of gate and of up by turns
      float2 s[4];
#pragma unroll
      for (int j = 0; j < 4; j++) s[j] = *reinterpret_cast<const float2 *>(sums + (j * pc.toks + row) * sum_stride(2) + 2 * pr);
      u = make_float2(s[1].x + s[3].x, s[1].y + s[3].y), v = make_float2(s[0].x + s[2].x, s[0].y + s[2].y);
      if (!pair) v.x += u.x, v.y += u.y;
    }
    float *slot = slots + (pair ? 2 * row : row) * 128;
    if (!owner) {
      if (live) send(slot, v);
      if (live && pair) send(slot + 128, u);
      continue;
    }
    const int per = pair ? kSlots / 2 : kSlots;                                       // contributors at a time: words of gate and up by turns, or of one matrix
    for (int c = live ? 0 : others; c < others; c += per, slot += per * (size_t)slot_floats) {
      uint2 w[kSlots];
      auto there = [&](int j) { return c + (pair ? j / 2 : j) < others; };
      auto at_slot = [&](int j) { return slot + (size_t)(pair ? j / 2 : j) * slot_floats + (pair ? j % 2 * 128 : 0); };
      bool missing;
      do {                                                                            // all of them in flight together, again until all are there
        missing = false;
#pragma unroll
        for (int j = 0; j < kSlots; j++)
          if (there(j)) w[j] = ld_relaxed2(at_slot(j));
#pragma unroll
        for (int j = 0; j < kSlots; j++)
          if (there(j)) missing |= w[j].x == 0 || w[j].y == 0;
      } while (missing && patience && --patience);
#pragma unroll
      for (int j = 0; j < kSlots; j++)
        if (there(j)) {
          st_relaxed2(at_slot(j), make_uint2(0, 0));
          if (pair && j % 2) u.x += __uint_as_float(w[j].x), u.y += __uint_as_float(w[j].y);
          else v.x += __uint_as_float(w[j].x), v.y += __uint_as_float(w[j].y);
        }
    }
    v.x = v.x * scale + __uint_as_float(a << 16), v.y = v.y * scale + __uint_as_float(a & 0xFFFF0000u);
    a = addend(row + rows);
    if (epi == BT_EPI_RELU) v.x = fmaxf(v.x, 0.f), v.y = fmaxf(v.y, 0.f);
    if (epi == BT_EPI_SILU || pair) v.x = silu(v.x), v.y = silu(v.y);
    if (pair) v.x *= (u.x + 0.f) * scale, v.y *= (u.y + 0.f) * scale;
    if (epi == BT_EPI_ARGMAX) {
      unsigned long long key = inside && live ? max(pick_key(v.x, n0), pick_key(v.y, n0 + 1)) : 0ull;
      for (int d = 1; d < min(pairs, 32); d <<= 1) key = max(key, __shfl_xor_sync(0xFFFFFFFFu, key, d));
      // a maximum over all sub-panels whatever the order they finish in, so the last one to finish has the answer at hand
      if ((threadIdx.x & (min(pairs, 32) - 1)) == 0 && key) atomicMax(sc.keys + row, key);
      continue;
    }
    store_pair(p, out, fp32, M, tcol, pr, n0, row, [&] { return inside && live; }, v);
  }
  if (!patience) {
    sts32(smem + kSmDead, 1);
    atomicExch(error, 3);
  }
}

// The unit ranges of a CTA in the order it takes them. A sub-panel that several CTAs share is finished by the CTA
// that holds its last tile row (its owner); the others hand it their partial sums through global memory. So a CTA
// first takes the sub-panel its range ends in (it is that one's first contributor, and the owner will not need the
// sums for a while), then the sub-panels it has whole, and last the sub-panel its range starts in, which it owns:
// by then the other contributors have long signalled, or are finishing at the same moment. `walk` below goes through
// these pieces sub-panel by sub-panel; everything is a scalar with a fixed place, so it lives in registers.
struct Walk {
  int KT, segs;                      // segments left, the one at hand included
  int a, b, a1, b1, a2, b2;          // units [a, b) of this segment, and the segments after it
  __device__ __forceinline__ void start(const GemvParams &p, int range) {
    const int u0 = range_start(p, range), u1 = range_start(p, range + 1);
    KT = p.KT, segs = 0;
    a = b = a1 = b1 = a2 = b2 = 0;
    const int head_end = min(u1, (u0 / KT + 1) * KT);                  // end of the sub-panel the range starts in
    const bool head_partial = u0 % KT != 0 || head_end - u0 < KT;
    const int tail_start = u1 / KT * KT;                               // start of the sub-panel the range ends in
    const bool tail_partial = u1 % KT != 0 && tail_start >= head_end;  // a tail that is not the head itself
    const int mid_a = head_partial ? head_end : u0, mid_b = tail_partial ? tail_start : u1;
    if (head_partial) push(u0, head_end);
    if (mid_b > mid_a) push(mid_a, mid_b);
    if (tail_partial) push(tail_start, u1);
  }
  __device__ __forceinline__ void push(int from, int to) { a2 = a1, b2 = b1, a1 = a, b1 = b, a = from, b = to, segs++; }
  __device__ __forceinline__ bool more() const { return segs > 0; }
  // the next piece: up to the end of a sub-panel or of the segment
  __device__ __forceinline__ void next(int &sp, int &kt, int &rows) {
    sp = a / KT, kt = a - sp * KT, rows = min(KT - kt, b - a);
    a += rows;
    if (a == b) segs--, a = a1, b = b1, a1 = a2, b1 = b2;
  }
};

// Where the next stage goes, kept in step by the two producers: stages follow one another through the ring's bytes (a
// stage that would run past the end starts over at 0).
struct Ring {
  uint32_t off;     // where the next stage would start
  // The room that the next stage takes: its bytes plus what is skipped when it starts over. Together these may be more than a ring has which
  // is shorter than two stages (a chain's, whose stages may differ in size). Such a stage waits until it is alone in the ring, and then skips nothing.
  template <bool SHORT> __host__ __device__ __forceinline__ uint32_t room(uint32_t bytes, uint32_t ring_bytes, bool *alone) const {
    const uint32_t skipped = off + bytes > ring_bytes ? ring_bytes - off : 0;
    *alone = SHORT && bytes + skipped > ring_bytes;
    return *alone ? bytes : bytes + skipped;
  }
  __host__ __device__ __forceinline__ uint32_t place(uint32_t bytes, uint32_t ring_bytes) {       // byte offset of the next stage
    if (off + bytes > ring_bytes) off = 0;
    const uint32_t at = off;
    off += bytes;
    return at;
  }
};

// ---- producers: two warps walk the whole queue ---------------------------------------------------------------
// One warp copies weights, the other x. Both follow the same stages through the ring and wait for the same room
// (the oldest stage in the ring freed by the consumers), each keeping its own books, so neither waits for the other.
// Weights never depend on an earlier matmul: their copies go out as soon as the ring has room, one bulk copy per
// weight matrix and stage. x is the result of an earlier matmul: the x warp waits (with a limit) until all sub-panels of
// the matmul it depends on are reported finished, then copies each stage's x tiles with ONE tiled TMA copy, which picks
// the token rows that are there out of every tile (8 rows: 256 bytes of each of two faces). An asynchronous copy costs
// its issuer and the copy engine the same whatever its size: with two plain copies of 256 bytes per tile the x
// warp alone held an 8192 x 28672 bfp4 matmul at 46 us, with one of 1 KB at 35, where the weights take 31.
// x may be the result of the launch before this one, or of an earlier matmul of this one: the host has worked out the
// last matmul of the launch that this one must see complete, and every one before that must be complete too (see Gate). A
// whole warp waits, a lane for each of the two counters, so that their loads are in flight together. False: gave up.
__device__ __forceinline__ bool await_turn(const QueueHead &q, int wait_for, int wait_panels, int wait_also, int also_panels, int pause_ns) {
  asm volatile("griddepcontrol.wait;" ::: "memory");     // returns when the previous launch is complete and visible
  const int lane = threadIdx.x & 31, op = lane == 0 ? wait_for : lane == 1 ? wait_also : -1;
  bool ok = true;
  if (op >= 0) {
    const int panels = lane ? also_panels : wait_panels;
    uint32_t spins = 0;
    while (ld_acquire_gpu(q.ops_done + op) < panels) {
      if (++spins > kSpinLimit * 64) { ok = false; break; }
      if (pause_ns) __nanosleep(pause_ns);
    }
  }
  return __all_sync(0xFFFFFFFFu, ok);                    // what either lane acquired is visible to the whole warp
}
__device__ __forceinline__ bool await_turn(const QueueHead &q, const GemvParams &p, int pause_ns) { return await_turn(q, p.wait_for, p.wait_panels, p.wait_also, p.also_panels, pause_ns); }

template <bool WEIGHTS, bool SMALL, bool CHAIN, class Q>
__device__ __forceinline__ void produce(const Q &q, uint8_t *smem, uint32_t sbase, int cta, int ctas) {
  const uint32_t full0 = sbase + kSmFull, empty0 = sbase + kSmEmpty, ring0 = sbase + q.ring, ring_bytes = q.ring_bytes;
  volatile uint32_t *held = reinterpret_cast<volatile uint32_t *>(smem + kSmHeld) + (WEIGHTS ? 0 : kBars);   // ring bytes of each stage in the ring
  const int lane = threadIdx.x & 31;
  if (!WEIGHTS && lane < q.n) tensormap_prefetch(&q.op[lane].xmap);
  if (WEIGHTS && SMALL && lane < q.n && q.op[lane].tiled) {
    tensormap_prefetch(&q.op[lane].wmap[0]);
    if (q.op[lane].pair) tensormap_prefetch(&q.op[lane].wmap[1]);
  }
  Ring ring{0};
  uint32_t count = 0, oldest = 0, used = 0;   // stages placed; first stage not yet known to be free; ring bytes held from there on
  for (int i = 0; i < q.n; i++) {
    const GemvParams &p = q.op[i];
    Geometry g = geometry(p.fmt, p.pair != 0, p.tg, lw_of<SMALL>(p));
    if (CHAIN) g.stage = g.w_bytes;                          // x goes straight to registers
    const int me = (cta + p.turn) % ctas;                    // the range this CTA takes in this matmul
    if (me >= p.active) continue;
    const int KT = p.KT, nw = p.pair ? 2 : 1;
    const uint8_t *w = p.w[lane < nw ? lane : 0];
    Walk walk;
    walk.start(p, me);
    bool gate = !WEIGHTS;                 // the x warp has yet to wait for the matmul before this one
    while (walk.more()) {
      int sp, kt, rows;
      walk.next(sp, kt, rows);
      const Columns<SMALL> at(p, sp);
      const int width = at.width, ends = walk.more() ? 1 : 3;
      const int first = WEIGHTS ? cta_of(p, sp * KT) : 0, end = WEIGHTS ? cta_of(p, (sp + 1) * KT - 1) : 0;
      for (; rows > 0; rows -= g.ups, kt += g.ups) {
        const int n = min(g.ups, rows);
        bool alone;
        const uint32_t need = ring.room<CHAIN>(g.stage, ring_bytes, &alone);
        while (used + need > ring_bytes || count - oldest == kBars || (alone && used)) {
          // asleep in the instruction: a polling loop takes issue slots from the consumers, and the ring is deep enough to
          // hide a late wake-up
          if (!stage_wait(sbase, empty0 + 8 * (oldest % kBars), (oldest / kBars) & 1, q.error)) {
            // the copies in flight land before the CTA may end (with a limit: some of these stages may never get their x)
            for (; oldest != count; oldest++) mbar_wait(full0 + 8 * (oldest % kBars), (oldest / kBars) & 1, 100);
            return;
          }
          used -= held[oldest % kBars], oldest++;
        }
        const uint32_t bar = full0 + 8 * (count % kBars), stage = ring0 + ring.place(g.stage, ring_bytes);
        if (lane == 0) held[count % kBars] = need;
        if (WEIGHTS) {
          const uint32_t bytes = n * width * g.tb;
          if (lane == 0) {
            uint4 *note = reinterpret_cast<uint4 *>(smem + kSmStages) + 2 * (count % kBars);
            note[0] = make_uint4(stage, n, width, (rows <= g.ups ? ends : 0) | (n == g.ups && width == kWC ? 4 : 0) | kt << 3), note[1] = make_uint4(sp, first, me, end);
            mbar_expect_tx(bar, nw * bytes);
          }
          __syncwarp();
          if (!SMALL || width == at.run_width) {
            // one contiguous range of each matrix
            if (lane < nw) bulk_g2s(stage + lane * g.matrix, w + ((size_t)at.run * kWC * KT + (size_t)kt * width) * g.tb, bytes, bar);
          } else if (n == g.ups && at.run_width == kWC) {
            // some columns of a run: a tiled copy of each matrix
            if (lane < nw) tma_load_3d(stage + lane * g.matrix, &p.wmap[lane], 0, at.col & 3, at.run * KT + kt, bar);
          } else {
            // the last, shorter stage of such a piece, or a run shorter than four: a copy per tile row
            for (int j = lane; j < nw * n; j += 32) {
              const int m = j >= n, row = j - m * n;
              bulk_g2s(stage + m * g.matrix + row * width * g.tb, p.w[m] + ((size_t)at.run * kWC * KT + (size_t)(kt + row) * at.run_width + (at.col & 3)) * g.tb, width * g.tb, bar);
            }
          }
        } else {
          if (gate) {
            if (!await_turn(q, p, 0) && lane == 0) atomicExch(q.error, 5);
            // x was written with ordinary stores (by other CTAs of this launch, or by the launch before) and is about to
            // be read by TMA copies: order what the acquire made visible before the asynchronous proxy's reads
            fence_proxy_async();
            gate = false;
          }
          // always a whole stage's box: tile columns past K come as zeros, those past the piece are not looked at
          if (lane == 0) {
            mbar_expect_tx(bar, g.ups * g.xb);
            tma_load_3d(stage + g.w_bytes, &p.xmap, 0, 0, kt, bar);
          }
        }
        __syncwarp();
        used += need, count++;
      }
    }
  }
}

// ---- consumers --------------------------------------------------------------------------------------------------
// A warp's part of one piece: tile rows of a sub-panel, of which the warp takes every second or fourth from `ck` on in
// one column, stage by stage; then its sums go to shared memory. What does not depend on the kind of matmul lives in the
// kernel itself, once, where the matmul's parameters are read from the constant bank (passed on by reference they were
// fetched through global memory, and a sub-panel's end took 4-6 us).
struct Place {
  uint32_t smem;                     // shared memory
  uint32_t count;                    // stages so far
  int cc, ck, mat;                   // this warp's column, first tile row, weight matrix
  int lane;
};
// Fragments to [k group][matrix][token][channel]: lane (g, t) holds tokens 8 tg + 2 t + j and channels 16 fs + 2 g + {0, 1}.
// Tokens from `tokens` on are left out.
template <int FMT, int TG>
__device__ __forceinline__ void leave_sums(const float (&acc)[2][TG][4], float *to, int stride, int tokens, int cc, int lane) {
  const int t = lane & 3, g = lane >> 2;
  to += 2 * t * stride + cc * 32 + 2 * g;
#pragma unroll
  for (int fs = 0; fs < 2; fs++)
#pragma unroll
    for (int tg = 0; tg < TG; tg++)
#pragma unroll
      for (int j = 0; j < 2; j++)
        if (8 * tg + 2 * t + j < tokens)
          *reinterpret_cast<float2 *>(to + (8 * tg + j) * stride + 16 * fs) =
              FMT == BT_BFP8 ? make_float2(acc[fs][tg][j], acc[fs][tg][2 + j]) : make_float2(16.f * acc[fs][tg][2 + j], acc[fs][tg][j] - acc[fs][tg][2 + j]);
}
template <int FMT, int TG, bool PAIR>
__device__ __forceinline__ uint4 stream_rows(Place &w, float *sums, int *error) {
  constexpr int TB = tile_bytes(FMT), T = stage_rows_per_warp(FMT, TG, 2), XB = 512 * TG, GROUPS = PAIR ? 2 : 4;   // warps that share a column
  const int lane = w.lane, ck = w.ck, cc = w.cc;
  const uint32_t matrix0 = w.mat * (GROUPS * T * kWC * TB), x0 = 4 * T * kWC * TB + ck * XB + lane * 8, tile0 = matrix0 + (ck * kWC + cc) * TB;
  float acc[2][TG][4];
#pragma unroll
  for (int i = 0; i < 8 * TG; i++) acc[i / (4 * TG)][i / 4 % TG][i % 4] = 0.f;
  uint4 piece = make_uint4(0, 0, 0, 0);
  for (int last = 0; !last;) {
    const uint32_t slot = w.count & (kBars - 1), bar = w.smem + 8 * slot, note = w.smem + kSmStages + 32 * slot;
    if (!stage_wait(w.smem, bar + kSmFull, w.count / kBars & 1, error)) break;
    const uint4 stage = lds128(note);                                  // at, rows, width, ends
    last = stage.w & 3;
    if (last) piece = lds128(note + 16), piece.x |= (uint32_t)last << 30;
    if (stage.w & 4) {
      // a whole stage of four columns: every offset is a constant
      const uint32_t tile = stage.x + tile0 + lane * 16, ex = stage.x + tile0 + (lane & 3) * 16, xs = stage.x + x0;
#pragma unroll
      for (int j = 0; j < T; j++) tile_mma<FMT, TG>(tile + j * (GROUPS * kWC * TB), ex + j * (GROUPS * kWC * TB), xs + j * (GROUPS * XB), acc);
    } else if (cc < (int)stage.z) {
      uint32_t tile = stage.x + matrix0 + (ck * stage.z + cc) * TB, xs = stage.x + x0;
#pragma unroll 1
      for (int row = ck; row < (int)stage.y; row += GROUPS, tile += GROUPS * stage.z * TB, xs += GROUPS * XB)
        tile_mma<FMT, TG>(tile + lane * 16, tile + (lane & 3) * 16, xs, acc);
    }
    __syncwarp();
    mbar_arrive_if(bar + kSmEmpty, lane == 0);
    w.count++;
  }
  leave_sums<FMT, TG>(acc, sums + (PAIR ? 2 * ck + w.mat : ck) * 8 * TG * sum_stride(2), sum_stride(2), 8 * TG, cc, lane);
  return piece;
}
// The same for small matmuls, whose sub-panels have one, two or four columns and whose tile rows go round up to 16 warps: a
// warp has a few tiles in all, and leaves the sums of each by itself.
template <int FMT, int TG>
__device__ __forceinline__ uint4 stream_small(Place &w, float *sums, int *error, const GemvParams &p) {
  constexpr int TB = tile_bytes(FMT), XB = 512 * TG;
  const int lw = p.lw, M = p.M, matrices = p.pair ? 2 : 1, lane = w.lane, groups = kCW >> lw >> (matrices - 1);
  const Geometry g = geometry(FMT, matrices == 2, TG, lw);
  uint4 piece = make_uint4(0, 0, 0, 0);
  for (int last = 0; !last;) {
    const uint32_t slot = w.count & (kBars - 1), bar = w.smem + 8 * slot, note = w.smem + kSmStages + 32 * slot;
    if (!stage_wait(w.smem, bar + kSmFull, w.count / kBars & 1, error)) break;
    const uint4 stage = lds128(note);
    last = stage.w & 3;
    if (last) piece = lds128(note + 16), piece.x |= (uint32_t)last << 30;
    if (w.cc < (int)stage.z) {
      uint32_t tile = stage.x + w.mat * g.matrix + (w.ck * stage.z + w.cc) * TB, xs = stage.x + g.w_bytes + w.ck * XB + lane * 8;
#pragma unroll 1
      for (int row = w.ck; row < (int)stage.y; row += groups, tile += groups * stage.z * TB, xs += groups * XB) {
        float acc[2][TG][4];
#pragma unroll
        for (int i = 0; i < 8 * TG; i++) acc[i / (4 * TG)][i / 4 % TG][i % 4] = 0.f;
        tile_mma<FMT, TG>(tile + lane * 16, tile + (lane & 3) * 16, xs, acc);
        leave_sums<FMT, TG>(acc, sums + ((((int)stage.w >> 3) + row) * matrices + w.mat) * M * sum_stride(lw), sum_stride(lw), M, w.cc, lane);
      }
    }
    __syncwarp();
    mbar_arrive_if(bar + kSmEmpty, lane == 0);
    w.count++;
  }
  return piece;
}

// ---- the messenger: one warp tells other CTAs and hears from them ------------------------------------------------
// It goes through the CTA's pieces beside the consumers and meets them when they have stored what they had. A release
// takes 1000 to 3000 cycles under load; a consumer warp that did it was that much behind the others at the next barrier.
// Report a sub-panel: its results are visible to the whole GPU before the count moves. A matmul is complete when all
// its sub-panels are: by then every CTA with a part in it has read its x, and is past its look at the counts. It says
// nothing about the matmul before it, of which this CTA may have no part: that is what Gate is about. (Counting
// the CTAs instead, idle ones too, took 148 reports to one address where a small matmul has 5 sub-panels.) The last
// report of the launch therefore finds nobody looking any more, and zeroes the counts for the next launch (and counts a launch of chains:
// reading and writing that number at the end of every launch took 0.35 us).
template <bool CHAIN> __device__ __forceinline__ void report(const QueueHead &q, int i) {
  const int lane = threadIdx.x & 31;
  int end = 0;
  if (lane == 0) {
    red_release_gpu(q.ops_done + i, 1);
    if (atom_add_acq_rel_gpu(q.all_done, 1) == q.panels - 1) {
      for (int j = 0; j < q.n; j++) q.ops_done[j] = 0;
      *q.all_done = 0;
      if (CHAIN && q.exchange) {
        const uint32_t next = (*q.epoch + 1) % kEpochs;
        *q.epoch = next, end = next == 0;
      }
    }
  }
  if (CHAIN && __shfl_sync(0xFFFFFFFFu, end, 0))          // the tags start over
    for (size_t at = lane; at < kExchanges * kExchangeBytes / 16; at += 32) reinterpret_cast<uint4 *>(q.exchange)[at] = make_uint4(0, 0, 0, 0);
}

template <bool SMALL, class Q> __device__ __forceinline__ void carry(const Q &q, int cta, int ctas) {
  const int lane = threadIdx.x & 31;
  for (int i = 0; i < q.n; i++) {
    const GemvParams &p = q.op[i];
    const Scratch &sc = q.set[i % q.sets];
    const int me = (cta + p.turn) % ctas, M = p.M;
    Walk walk{};
    if (me < p.active) {
      walk.start(p, me);
      // the counters and the result are this matmul's only when the ones before it that it must not overtake are done
      if (!await_turn(q, p, 100) && lane == 0) atomicExch(q.error, 5);
    }
    while (walk.more()) {
      int sp, kt, rows;
      walk.next(sp, kt, rows);
      const int first = cta_of(p, sp * p.KT), last = cta_of(p, (sp + 1) * p.KT - 1);
      int *counter = sc.counters + sp;
      if (me == last) zero_rows<SMALL>(p, sp);
      // every contributor is past its last look at the counts of this launch
      if (me == last && first != last && lane == 0) {
        uint32_t spins = 0;
        while (ld_acquire_gpu(counter) < last - first) {
          if (++spins > kSpinLimit * 32) { atomicExch(q.error, 3); break; }
          __nanosleep(100);
        }
        *counter = 0;                            // ready for the next matmul
      }
      __syncwarp();
      named_barrier(2, kConsumers + 32);
      if (me != last) {
        if (lane == 0) atomicAdd(counter, 1);    // the sums themselves say that they are there
        continue;
      }
      if (p.epi == BT_EPI_ARGMAX) {
        // the last sub-panel to finish turns the keys into the answer and leaves the scratch as it found it
        int is_last = 0;
        if (lane == 0) {
          fence_gpu();
          is_last = atomicAdd(sc.panels_done, 1) == p.panels - 1;
        }
        if (__shfl_sync(0xFFFFFFFFu, is_last, 0)) {
          fence_gpu();
          if (lane < M) {
            const unsigned long long key = atomicExch(sc.keys + lane, 0ull);
            uint32_t b = (uint32_t)(key >> 32);
            b ^= b >> 31 ? 0x80000000u : 0xFFFFFFFFu;
            p.arg_val[lane] = key ? __uint_as_float(b) : -INFINITY;
            p.arg_idx[lane] = (key ? (int)(0xFFFFFFFFu - (uint32_t)key) : 0x7FFFFFFF) + p.arg_base;
          }
          if (lane == 0) *sc.panels_done = 0;
        }
        __syncwarp();
      }
      report<false>(q, i);
      __syncwarp();
    }
  }
}

// Piece `n` of range `me` as a stage's note has it: (sub-panel | what ends with it << 30, first range, this one, last one).
__device__ __noinline__ uint4 piece_at(const GemvParams &p, int me, int n) {
  int sp = 0, kt, rows;
  Walk walk;
  walk.start(p, me);
  for (int i = 0; i <= n; i++) walk.next(sp, kt, rows);
  return make_uint4(sp | (walk.more() ? 1u : 3u) << 30, cta_of(p, sp * p.KT), me, cta_of(p, (sp + 1) * p.KT - 1));
}

template <bool SMALL, int OPS>
__global__ void __launch_bounds__(kThreads, 1) gemv_queue_kernel(const __grid_constant__ Queue<OPS> q) {
  extern __shared__ __align__(128) uint8_t smem[];
  const uint32_t sbase = smem_u32(smem);
  const int warp = threadIdx.x >> 5, cta = blockIdx.x, ctas = gridDim.x;
  // The next launch in the stream may start as soon as there is room for its CTAs: what it does before its own
  // griddepcontrol.wait (set up, prefetch weights) does not depend on this launch.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (threadIdx.x == 0) {
    sts32(sbase + kSmDead, 0);
    for (int s = 0; s < kBars; s++) {
      mbar_init(sbase + kSmFull + 8 * s, 2);        // the announcements of the weight bytes and of the x bytes
      mbar_init(sbase + kSmEmpty + 8 * s, kCW);
    }
    mbar_fence_init();
  }
  __syncthreads();
  if (warp >= kCW) {
    if (warp == kCW) produce<true, SMALL, false>(q, smem, sbase, cta, ctas);
    else if (warp == kCW + 1) produce<false, SMALL, false>(q, smem, sbase, cta, ctas);
    else carry<SMALL>(q, cta, ctas);
    return;
  }
  float *sums = reinterpret_cast<float *>(smem + kSmSums);
  Place w;
  w.smem = sbase, w.count = 0, w.lane = threadIdx.x & 31, w.cc = warp & 3;
  for (int i = 0; i < q.n; i++) {
    const GemvParams &p = q.op[i];
    const Scratch &sc = q.set[i % q.sets];
    // a column's tile rows go round the warps that a sub-panel's columns and matrices leave for it: 4 of them for four columns of one matrix
    const int lw = lw_of<SMALL>(p), rest = warp >> lw;
    w.cc = warp & ((1 << lw) - 1), w.mat = p.pair ? rest & 1 : 0, w.ck = p.pair ? rest >> 1 : rest;
    // The ranges go round the CTAs from matmul to matmul: the CTAs that finish shared sub-panels have more to do than
    // the others, and it should not be the same ones every time.
    const int me = (cta + p.turn) % ctas;
    int pieces = 0;
    for (bool more = me < p.active; more; pieces++) {
      uint4 piece;
      if (SMALL && p.small) switch ((p.fmt == BT_BFP4 ? 3 : 0) + (p.tg == 1 ? 0 : p.tg == 2 ? 1 : 2)) {
        case 0: piece = stream_small<BT_BFP8, 1>(w, sums, q.error, p); break;
        case 1: piece = stream_small<BT_BFP8, 2>(w, sums, q.error, p); break;
        case 2: piece = stream_small<BT_BFP8, 4>(w, sums, q.error, p); break;
        case 3: piece = stream_small<BT_BFP4, 1>(w, sums, q.error, p); break;
        case 4: piece = stream_small<BT_BFP4, 2>(w, sums, q.error, p); break;
        default: piece = stream_small<BT_BFP4, 4>(w, sums, q.error, p); break;
      } else switch ((p.fmt == BT_BFP4 ? 6 : 0) + (p.pair ? 3 : 0) + (p.tg == 1 ? 0 : p.tg == 2 ? 1 : 2)) {
        case 0: piece = stream_rows<BT_BFP8, 1, false>(w, sums, q.error); break;
        case 1: piece = stream_rows<BT_BFP8, 2, false>(w, sums, q.error); break;
        case 2: piece = stream_rows<BT_BFP8, 4, false>(w, sums, q.error); break;
        case 3: piece = stream_rows<BT_BFP8, 1, true>(w, sums, q.error); break;
        case 4: piece = stream_rows<BT_BFP8, 2, true>(w, sums, q.error); break;
        case 5: piece = stream_rows<BT_BFP8, 4, true>(w, sums, q.error); break;
        case 6: piece = stream_rows<BT_BFP4, 1, false>(w, sums, q.error); break;
        case 7: piece = stream_rows<BT_BFP4, 2, false>(w, sums, q.error); break;
        case 8: piece = stream_rows<BT_BFP4, 4, false>(w, sums, q.error); break;
        case 9: piece = stream_rows<BT_BFP4, 1, true>(w, sums, q.error); break;
        case 10: piece = stream_rows<BT_BFP4, 2, true>(w, sums, q.error); break;
        default: piece = stream_rows<BT_BFP4, 4, true>(w, sums, q.error); break;
      }
      // ---- this CTA is done with its part of the sub-panel ----
      if (lds32(sbase + kSmDead)) piece = piece_at(p, me, pieces);       // not from the ring's notes
      more = piece.x >> 30 != 3;
      const Piece pc = {(int)(piece.x & 0x3FFFFFFF), (int)piece.y, (int)piece.w, (int)piece.z, 8 * p.tg};
      end_piece<SMALL>(p, sc, q.slot_floats, sums, pc, sbase, q.error);
      named_barrier(2, kConsumers + 32);       // the messenger may tell; the sums may be overwritten
    }
  }
}

// ---- chains of small matmuls --------------------------------------------------------------------------------------
// In a small model's decode step every matmul is small (a sub-panel to a CTA, whole) and reads the one before it. What such a matmul
// costs is the way from one's result to the next one's. In the general kernel that is 4.9 us: the stores have to be acknowledged before the
// report (0.7), the report is seen by polling (0.7-1.0), then the copy of x starts (0.8), and from x to the result there are some 2.7 us of
// instructions, most of them fetched anew for every matmul. So lists of small matmuls with up to 8 tokens have a kernel of their own (where it is the faster one: see chain):
//  * A result also goes to an exchange where every word (two bf16 values) travels with a tag: the launch's number and the matmul's
//    place in it. What has the right tag is there: no report, no copy. A consumer lane fetches the words of its own
//    MMA fragments, straight into registers.
//  * Weights are expanded, scale and all, while x is still on its way, and wait in shared memory as the MMAs take them.
//  * The next matmul runs on other CTAs, which have had the time for that.
// 2.0-2.2 us a matmul for one token (1.0 until x is seen, 0.4 to the sums, 0.6 to add them and publish), 3 for eight, whose words and
// tags are 36 KB to a CTA of a gate/up pair. 30 layers of 576 x 1536 with host values in and out: one token 500 -> 276 us, eight 507 -> 390.
//
// What makes it safe to start before the matmul before is known to be complete: of that matmul only x (and the addend, where it is the
// same tensor) is read, from the exchange. Whatever this one overwrites that the matmul before reads has been
// read by then: a word is published after the values that go into it were read, and every word this matmul stores depends on all of
// its x. (The zero rows, which do not, wait for the counter: the messenger writes them.) Everything else waits for the counters of the
// matmuls before that one (early), and so does every store. kExchanges = 3: matmul i + 3 stores when i + 1, which reads exchange i, is complete.
// A tag comes up once in kEpochs launches, and then the exchanges are cleared.
//
// An exchange: [tile column][left, right face][row < M][8 words with their tags].
__device__ __forceinline__ uint32_t tag_of(uint32_t epoch, int i) { return epoch * 64 + i + 1; }

// A tile's weights as the registers of its four MMAs, [h][fs], exactly: the codes as integers times 2^-6, times 2^(e - 127).
template <int FMT> __device__ __forceinline__ void expand_tile(uint32_t tile, uint32_t ex, uint32_t (&a)[2][2][4]) {
  const uint4 ev = lds128(ex);
  const uint32_t ee[4] = {ev.x, ev.y, ev.z, ev.w};
  uint4 wv[2];
  wv[0] = lds128(tile + 64);
  if (FMT == BT_BFP8) wv[1] = lds128(tile + 64 + 512);
#pragma unroll
  for (int h = 0; h < 2; h++)
#pragma unroll
    for (int fs = 0; fs < 2; fs++) {
      const uint32_t e = ee[2 * h + fs], s01 = (e << 7) & 0x7F807F80u, s23 = (e >> 1) & 0x7F807F80u;
      uint32_t c0, c1, c2, c3, o0, o1;     // codes of rows g and g + 8, first and second k pair, and their offsets
      if (FMT == BT_BFP8) {
        const uint32_t w0 = fs ? wv[h].z : wv[h].x, w1 = fs ? wv[h].w : wv[h].y;
        c0 = w0 & kByteLanes, c1 = w1 & kByteLanes, c2 = prmt(w0, 0u, kOddBytes), c3 = prmt(w1, 0u, kOddBytes), o0 = kOff128, o1 = kOff128;
      } else {
        const uint32_t w = h ? (fs ? wv[0].w : wv[0].z) : (fs ? wv[0].y : wv[0].x);
        c0 = w & kByteLanes, c1 = w & kNibbleLanes, c2 = prmt(w, 0u, kOddBytes), c3 = c2 & kNibbleLanes, o0 = kOff136, o1 = kOff8;
      }
      a[h][fs][0] = mul_bf16x2(fma_bf16x2(c0, kTo6, o0), s01), a[h][fs][1] = mul_bf16x2(fma_bf16x2(c1, kTo6, o1), s01);
      a[h][fs][2] = mul_bf16x2(fma_bf16x2(c2, kTo6, o0), s23), a[h][fs][3] = mul_bf16x2(fma_bf16x2(c3, kTo6, o1), s23);
    }
}

// One matmul's part of a consumer warp: its tile rows, every `groups`-th from ck on. x is asked for kAhead tile rows ahead.
constexpr int kAhead = 3;                            // 48 tile rows of one column: K = 1536
constexpr int kAheadBytes = kAhead * kCW * 2048;     // expanded weights of so many tile rows per warp
struct Link {
  uint32_t smem, count, turn;        // shared memory; stages, and matmuls of this CTA, so far
  int warp, lane;
};
template <int FMT> __device__ __forceinline__ void chain_matmul(const GemvParams &p, const QueueHead &q, int index, int me, Link &w, float *sums, uint32_t expanded) {
  constexpr int TB = tile_bytes(FMT);
  const int lane = w.lane, t = lane & 3, token = lane >> 2, M = p.M, lw = p.lw, KT = p.KT, thread = threadIdx.x;
  const bool from = p.from, pair = p.pair;
  const int rest = w.warp >> lw, cc = w.warp & ((1 << lw) - 1), mat = pair ? rest & 1 : 0, ck = pair ? rest >> 1 : rest, groups = small_groups(lw, pair);
  uint32_t tag = tag_of(lds32(w.smem + kSmEpoch), index) - 1;        // of the matmul before
  // this thread's place in the result: a pair of channels of one token
  const Columns<true> at(p, me);
  const int pr = thread & ((16 << lw) - 1), row = thread >> (4 + lw), tcol = at.col + (pr >> 4);
  const bool live = row < M && (pr >> 4) < at.width;
  const int before = (index + kExchanges - 1) % kExchanges, word = ((tcol * 2 + (pr >> 3 & 1)) * M + row) * 64 + (pr & 7) * 8;
  const uint8_t *x = from ? q.exchange + before * kExchangeBytes + token * 64 + t * 16 : reinterpret_cast<const uint8_t *>(p.x) + token * 32 + t * 8;
  const uint8_t *addend = p.add_from ? q.exchange + before * kExchangeBytes + word : reinterpret_cast<const uint8_t *>(p.add + pair_place(tcol, pr, row));
  const bool add_from = p.add_from && live, add = p.add && !p.add_from && live;
  uint8_t *to = p.to && live ? q.exchange + index % kExchanges * kExchangeBytes + word : nullptr;
  float alpha = p.alpha;
  int epi = p.epi;
  // what the end needs is fetched here, not when it is waited for
  asm volatile("" : "+f"(alpha), "+r"(epi), "+l"(to), "+l"(addend), "+l"(x), "+r"(tag));
  const uint32_t go = w.smem + kSmGo + 8 * (w.turn & 1);
  if (!from) stage_wait(w.smem, go, w.turn >> 1 & 1, q.error);
  const int steps = (KT + groups - 1) / groups, per_stage = stage_rows_per_warp(FMT, 1, lw);
  const uint32_t matrix = (uint32_t)mat * geometry(FMT, pair, 1, lw).matrix;
  expanded += w.warp * 2048 + lane * 16;
  uint32_t patience = kSpinLimit * 64;
  uint2 a = make_uint2(0, tag);
  const int stride = sum_stride(lw), slab = M * stride;
  for (int k0 = 0, in_stage = 0; k0 < steps; k0 += kAhead) {
    const int n = min(steps - k0, kAhead);
    // the weights of up to kAhead tile rows, as the MMAs take them
    uint4 stage = make_uint4(0, 0, 0, 0);
#pragma unroll 1
    for (int j = 0; j < n; j++) {
      const uint32_t slot = w.count & (kBars - 1);
      if (in_stage == 0 || j == 0) {
        const bool ok = stage_wait(w.smem, w.smem + kSmFull + 8 * slot, w.count / kBars & 1, q.error);
        stage = __all_sync(0xFFFFFFFFu, ok) ? lds128(w.smem + kSmStages + 32 * slot) : make_uint4(0, 0, 0, 0);
      }
      const int r = ck + in_stage * groups;
      uint32_t m[2][2][4] = {};
      if (cc < (int)stage.z && r < (int)stage.y) {
        const uint32_t tile = stage.x + matrix + (r * stage.z + cc) * TB;
        expand_tile<FMT>(tile + lane * 16, tile + t * 16, m);
      }
#pragma unroll
      for (int i = 0; i < 4; i++) sts128(expanded + j * (kCW * 2048) + i * 512, make_uint4(m[i / 2][i % 2][0], m[i / 2][i % 2][1], m[i / 2][i % 2][2], m[i / 2][i % 2][3]));
      if (++in_stage == per_stage || k0 + j == steps - 1) {
        in_stage = 0, w.count++;
        __syncwarp();
        mbar_arrive_if(w.smem + kSmEmpty + 8 * slot, lane == 0);
      }
    }
    // their x: upper and lower half of each, what this lane's token has there
    uint4 v[kAhead][2];
#pragma unroll
    for (int j = 0; j < kAhead; j++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int r = ck + (k0 + j) * groups;
        v[j][h] = make_uint4(0, tag, 0, tag);
        if (token < M && r < KT) {
          if (from) v[j][h].y = ~tag;
          else {
            const uint2 u = __ldcg(reinterpret_cast<const uint2 *>(x + r * 2048 + h * 512));
            v[j][h].x = u.x, v[j][h].z = u.y;
          }
        }
      }
    if (k0 == 0) {
      if (from) stage_wait(w.smem, go, w.turn >> 1 & 1, q.error);
      __syncwarp();
      if (add) a.x = __ldcg(reinterpret_cast<const uint32_t *>(addend));
      if (add_from) a.y = ~tag;
    }
    if (from) {
      bool missing;
      do {
        if (lds32(w.smem + kSmDead)) patience = 1;
#pragma unroll
        for (int j = 0; j < kAhead; j++)
#pragma unroll
          for (int h = 0; h < 2; h++)
            if (v[j][h].y != tag || v[j][h].w != tag) v[j][h] = ld_relaxed4(x + ((ck + (k0 + j) * groups) * 2 + h) * M * 64);
        if (a.y != tag) a = ld_relaxed64(addend);
        missing = a.y != tag;
#pragma unroll
        for (int j = 0; j < kAhead; j++) missing |= v[j][0].y != tag || v[j][0].w != tag || v[j][1].y != tag || v[j][1].w != tag;
      } while (__any_sync(0xFFFFFFFFu, missing && patience && --patience));   // the vote keeps the warp together; a lane that has given up stays that way
    }
    // the sums of the matmul before have been read
    if (k0 == 0 && w.turn) stage_wait(w.smem, w.smem + kSmDone + 8 * ((w.turn - 1) & 1), (w.turn - 1) >> 1 & 1, q.error);
    __syncwarp();
#pragma unroll
    for (int j = 0; j < kAhead; j++)
      if (ck + (k0 + j) * groups < KT) {
        float acc[2][1][4];
#pragma unroll
        for (int i = 0; i < 8; i++) acc[i / 4][0][i % 4] = 0.f;
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
          for (int fs = 0; fs < 2; fs++) {
            const uint4 m = lds128(expanded + j * (kCW * 2048) + (2 * h + fs) * 512);
            mma_bf16(acc[fs][0], m.x, m.y, m.z, m.w, v[j][h].x, v[j][h].z);
          }
        leave_sums<FMT, 1>(acc, sums + ((ck + (k0 + j) * groups) * (pair ? 2 : 1) + mat) * slab, stride, M, cc, lane);
      }
  }
  if (!patience) {
    sts32(w.smem + kSmDead, 1);
    atomicExch(q.error, 6);
  }
  // the last tile row's sums, then the others' in order: as in the general kernel, and with the same last bit
  const int next = pair ? 2 * slab : slab;
  const float *from_sum = sums + row * stride + 2 * pr, *last_sum = from_sum + (KT - 1) * next;
  int rows = KT - 1;
  asm volatile("" : "+l"(from_sum), "+l"(last_sum), "+r"(rows) :: "memory");
  named_barrier(1, kConsumers);
  // from here on a pair of channels of a token to a thread
  if (row - (lane >> min(4 + lw, 5)) < M) {                          // (whole warps)
    float2 s = make_float2(0.f, 0.f), u = s;
    if (row < M) {
      s = *reinterpret_cast<const float2 *>(last_sum);
      if (!pair) {
#pragma unroll 8
        for (int i = 0; i < rows; i++, from_sum += next) {
          const float2 y = *reinterpret_cast<const float2 *>(from_sum);
          s.x += y.x, s.y += y.y;
        }
      } else {
        u = *reinterpret_cast<const float2 *>(last_sum + slab);
#pragma unroll 4
        for (int i = 0; i < rows; i++, from_sum += next) {
          const float2 y = *reinterpret_cast<const float2 *>(from_sum), z = *reinterpret_cast<const float2 *>(from_sum + slab);
          s.x += y.x, s.y += y.y, u.x += z.x, u.y += z.y;
        }
      }
    }
    s.x = s.x * alpha + __uint_as_float(a.x << 16), s.y = s.y * alpha + __uint_as_float(a.x & 0xFFFF0000u);
    if (epi == BT_EPI_RELU) s.x = fmaxf(s.x, 0.f), s.y = fmaxf(s.y, 0.f);
    if (epi == BT_EPI_SILU || pair) s.x = silu(s.x), s.y = silu(s.y);
    if (pair) s.x *= (u.x + 0.f) * alpha, s.y *= (u.y + 0.f) * alpha;
    if (to) st_relaxed64(to, make_uint2(bf16_half_up(s.x) | bf16_half_up(s.y) << 16, tag + 1));
    store_pair(p, static_cast<char *>(p.out), p.out_fp32, M, tcol, pr, at.col * 32 + 2 * pr, row, [&] { return live; }, s);
  }
  __syncwarp();
  mbar_arrive_if(w.smem + kSmDone + 8 * (w.turn & 1), lane == 0);
  w.turn++;
}

template <int OPS>
__global__ void __launch_bounds__(kThreads, 1) chain_kernel(const __grid_constant__ Queue<OPS> q) {
  extern __shared__ __align__(128) uint8_t smem[];
  const uint32_t sbase = smem_u32(smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, cta = blockIdx.x, ctas = gridDim.x;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (threadIdx.x == 0) {
    sts32(sbase + kSmDead, 0);
    for (int s = 0; s < kBars; s++) mbar_init(sbase + kSmFull + 8 * s, 1), mbar_init(sbase + kSmEmpty + 8 * s, kCW);
    mbar_init(sbase + kSmReady, 1);
    for (int s = 0; s < 2; s++) mbar_init(sbase + kSmGo + 8 * s, 1), mbar_init(sbase + kSmDone + 8 * s, kCW);
    mbar_fence_init();
  }
  __syncthreads();
  if (warp == kCW) return produce<true, true, true>(q, smem, sbase, cta, ctas);
  if (warp < kCW) {
    Link w = {sbase, 0, 0, warp, lane};
    stage_wait(sbase, sbase + kSmReady, 0, q.error);
    for (int i = 0; i < q.n; i++) {
      const GemvParams &p = q.op[i];
      const int me = (cta + p.turn) % ctas;
      if (me >= p.active) continue;
      if (p.fmt == BT_BFP8) chain_matmul<BT_BFP8>(p, q, i, me, w, reinterpret_cast<float *>(smem + kSmSums + kAheadBytes), sbase + kSmSums);
      else chain_matmul<BT_BFP4>(p, q, i, me, w, reinterpret_cast<float *>(smem + kSmSums + kAheadBytes), sbase + kSmSums);
    }
    return;
  }
  // one warp lets the consumers go ahead, one, the messenger, reports what they have done
  const bool messenger = warp == kCW + 2;
  if (!messenger) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (lane == 0) {
      if (q.exchange) sts32(sbase + kSmEpoch, *reinterpret_cast<volatile int *>(q.epoch));
      mbar_arrive(sbase + kSmReady);
    }
    __syncwarp();
  }
  uint32_t turn = 0;
  for (int i = 0; i < q.n; i++) {
    const GemvParams &p = q.op[i];
    const int me = (cta + p.turn) % ctas;
    if (me >= p.active) continue;
    const bool early = !messenger && p.from;
    if (!await_turn(q, early ? p.early : p.wait_for, early ? p.early_panels : p.wait_panels, early ? p.early_also : p.wait_also, early ? p.early_also_panels : p.also_panels, messenger ? 100 : 0) &&
        lane == 0)
      atomicExch(q.error, 5);
    __syncwarp();
    if (!messenger) mbar_arrive_if(sbase + kSmGo + 8 * (turn & 1), lane == 0);
    else {
      zero_rows<true>(p, me);
      stage_wait(sbase, sbase + kSmDone + 8 * (turn & 1), turn >> 1 & 1, q.error);
      __syncwarp();
      report<true>(q, i);
      __syncwarp();
    }
    turn++;
  }
}

// ---- host side ---------------------------------------------------------------------------------------------------

int check_op(const char *who, int index, const bt_gemv_op &o) {
  BT_REQUIRE(o.fmt == BT_BFP8 || o.fmt == BT_BFP4, "%s: matmul %d: weights must be bfp8 (8) or bfp4 (4), not %d", who, index, o.fmt);
  BT_REQUIRE(o.epilogue >= BT_EPI_NONE && o.epilogue <= BT_EPI_ARGMAX, "%s: matmul %d: unknown epilogue %d", who, index, o.epilogue);
  BT_REQUIRE(o.M >= 1 && o.M <= 32, "%s: matmul %d: takes 1 to 32 rows of x, not %d", who, index, o.M);
  BT_REQUIRE(o.K > 0 && o.N > 0 && o.K % 32 == 0 && o.N % 32 == 0, "%s: matmul %d: K and N must be positive multiples of 32: %d x %d", who, index, o.K, o.N);
  BT_REQUIRE((o.N / 32 + kWC - 1) / kWC <= kMaxSubPanels, "%s: matmul %d: N = %d is past the %d columns one matmul handles", who, index, o.N,
             kMaxSubPanels * kWC * 32);
  BT_REQUIRE(o.x && o.w && o.x % 16 == 0 && o.w % 16 == 0, "%s: matmul %d: x and w must be 16-byte aligned device addresses", who, index);
  BT_REQUIRE((o.epilogue == BT_EPI_GLU) == (o.w2 != 0) && o.w2 % 16 == 0, "%s: matmul %d: w2 goes with the GLU epilogue, and only with it", who, index);
  BT_REQUIRE(o.add % 4 == 0, "%s: matmul %d: the addend must be 4-byte aligned", who, index);
  if (o.epilogue == BT_EPI_ARGMAX) BT_REQUIRE(o.arg_val && o.arg_idx, "%s: matmul %d: the argmax epilogue needs arg_val and arg_idx", who, index);
  else BT_REQUIRE(o.out && o.out % 8 == 0 && (o.out_dtype == BT_BF16 || o.out_dtype == BT_FP32 || o.out_dtype == BT_FP32_ROWS), "%s: matmul %d: needs an 8-byte aligned bf16 or fp32 result", who, index);
  return BT_OK;
}

// The byte ranges a matmul reads and writes. No earlier matmul writes its weights, but a later one may write where they lay: in
// the memory of weights that were freed behind their last use.
struct Range {
  uint64_t a, b;
  bool meets(const Range &o) const { return a < o.b && o.a < b; }
};
int ranges_read(const bt_gemv_op &o, Range *r) {
  int n = 0;
  r[n++] = {o.x, o.x + (uint64_t)(o.K / 32) * 2048};
  if (o.add) r[n++] = {o.add, o.add + (uint64_t)(o.N / 32) * 2048};
  const uint64_t weights = (uint64_t)(o.K / 32) * (o.N / 32) * tile_bytes(o.fmt);
  r[n++] = {o.w, o.w + weights};
  if (o.w2) r[n++] = {o.w2, o.w2 + weights};
  return n;
}
int ranges_written(const bt_gemv_op &o, Range *r) {
  int n = 0;
  if (o.epilogue == BT_EPI_ARGMAX) r[n++] = {o.arg_val, o.arg_val + 4ull * o.M}, r[n++] = {o.arg_idx, o.arg_idx + 4ull * o.M};
  else if (o.out_dtype == BT_FP32_ROWS) r[n++] = {o.out, o.out + 4ull * o.M * o.N};
  else r[n++] = {o.out, o.out + (uint64_t)(o.N / 32) * (o.out_dtype == BT_FP32 ? 4096 : 2048)};
  return n;
}
// `later` must not start before `earlier` is complete: it reads or writes what `earlier` writes, or writes what it reads.
bool depends(const bt_gemv_op &later, const bt_gemv_op &earlier) {
  Range lr[4], lw[2], er[4], ew[2];
  const int nlr = ranges_read(later, lr), nlw = ranges_written(later, lw), ner = ranges_read(earlier, er), new_ = ranges_written(earlier, ew);
  for (int i = 0; i < new_; i++) {
    for (int j = 0; j < nlr; j++) if (ew[i].meets(lr[j])) return true;
    for (int j = 0; j < nlw; j++) if (ew[i].meets(lw[j])) return true;
  }
  for (int i = 0; i < ner; i++)
    for (int j = 0; j < nlw; j++) if (er[i].meets(lw[j])) return true;
  return false;
}

// The last earlier matmul of a launch that matmul `i` of it (ops[i]; the launch starts at ops[0]) must not overtake:
// one whose result it reads (x, the addend) or whose buffers it writes, or that reads what it writes; and, because
// the running scratch exists `sets` times, the matmul `sets` places before it. -1: none.
int wait_for(const bt_gemv_op *ops, int i, int sets) {
  int w = i - sets;
  for (int e = i - 1; e > w && e >= 0; e--)
    if (depends(ops[i], ops[e])) w = e;
  return w < 0 ? -1 : w;
}

// The matmuls whose counters matmul `i` looks at before it starts, so that `last` AND ALL BEFORE IT are complete: it may
// depend on any of those, and any of them may still use its set of scratch. A matmul's counter speaks for that matmul
// alone, since a CTA without a range in it passes it by. What follows from it: matmul j has started everywhere, so what j
// itself waited for is complete, and (by induction over j) that is j's own `last` and all before it. `last` of every
// matmul is at most kSets = 2 places back; so of the matmuls before w = `last`, all up to w - 2 are complete when w is, and
// w - 1 is in doubt unless w waited for it. Then it is looked at too. In a chain it never is.
static_assert(kSets == 2, "one more counter closes the gap that a last matmul two places back leaves");
struct Gate {
  int last, also;             // -1: none
};
Gate gate(const bt_gemv_op *ops, int i, int sets) {
  const int w = wait_for(ops, i, sets);
  return {w, w > 0 && wait_for(ops, w, sets) < w - 1 ? w - 1 : -1};
}

// Whether matmul `i` of a chain takes its x from the exchange of matmul i - 1: x is that one's result, all of it, and nothing
// else stands between them than what the exchange takes care of.
bool exchanged(const bt_gemv_op *ops, int i) {
  if (i < 1) return false;
  const bt_gemv_op &o = ops[i], &e = ops[i - 1];
  if (o.x != e.out || e.out_dtype != BT_BF16 || o.M != e.M || o.K != e.N) return false;
  Range lr[4], lw[2], ew[2];
  ranges_read(o, lr), ranges_written(o, lw), ranges_written(e, ew);
  // an addend that is the same tensor comes from the exchange too, which has no more columns than the matmul before
  return !lw[0].meets(ew[0]) && (!o.add || (o.add == e.out ? o.N <= e.N : !lr[1].meets(ew[0])));
}
// Lists that chain_kernel takes: every matmul small, a sub-panel to a CTA, up to 8 tokens, no pick and no rows for an all-reduce; and it has to be
// the faster kernel. What it gains is the way from one result to the next. A matmul that reads x from memory gains little, and with many tile rows
// it loses, since x is then fetched batch by batch, each behind the weights it goes with; and a launch costs more. us, general kernel and this one (tokens):
//   chains of 24, a matmul: 576 x 1536 and back 5.1 and 2.7 (1), 5.2 and 3.9 (8); 4096 x 256 6.4 and 5.3 (1), 5.4 (3); 8192 x 64 10.9 and 10.4 (1), 11.4 and 13.7 (2); 9000 x 100 8.7 and 10.0 (1)
//   a launch of two: 576 x 576 9.3 and 7.9 (1), 9.0 (3); 2048 x 256 and back 10.5 and 10.3 (1), 11.4 (3), 12.4 (8); of three 15.9 and 13.7 (1), 14.2 (3)
//   not dependent, 24, a matmul: 576 x 576 2.4 and 2.3; 576 x 1536 3.1 and 2.5; 1024 x 768 2.6 and 2.7; 2048 x 512 3.3 and 3.6 (1), 3.4 and 4.5 (8); 4096 x 256 4.1 and 5.0; 100 x 9000 4.6 and 3.2
//   and a few: one of 576 x 1536 5.2 and 5.9, of 100 x 9000 6.6 and 6.3, three of 576 x 576 9.3 and 10.2, four of 576 x 1536 14.4 and 11.6
constexpr float kChainStartUs = 1.f;
float chain_gain_us(const GemvParams &p, bool linked) {
  if (linked) return p.M == 1 ? 2.4f - 0.017f * p.KT : 1.5f - 0.01f * p.KT - 0.03f * max(p.KT - 128, 0);
  return p.KT > 24 ? -0.0175f * p.KT : p.panels >= 32 ? 1.05f - 0.035f * p.KT : 0.1f;
}
bool chain(int n, const GemvParams *op, const bt_gemv_op *ops) {
  float gain = -kChainStartUs;
  for (int i = 0; i < n; i++) {
    if (!op[i].small || op[i].M > kChainRows || op[i].epi == BT_EPI_ARGMAX || op[i].out_fp32 == 2 || op[i].share != op[i].KT || op[i].extra) return false;
    gain += chain_gain_us(op[i], exchanged(ops, i));
  }
  return gain > 0.f;
}

// The ranges of a matmul's units. Sharing a sub-panel costs a hand-over of partial sums, a range that straddles sub-panels
// a second pass through a sub-panel's end, and fewer CTAs than SMs cost time only while the busy ones cannot take in what
// HBM delivers. So the candidates are: every sub-panel cut into 1, 2, ... ranges, as many as there are SMs for; whole
// sub-panels, several to a CTA, when there are more of them than SMs; equal shares of all SMs that straddle. The one
// with the least estimated time is taken, from the rates measured on 8192 x 28672 in steady state: HBM 6.3 TB/s, 50 GB/s
// into one SM, and an SM's time for a tile row of four tiles (row_us). In ranges that straddle, a sub-panel shared by two or
// three CTAs is handed over early: its contributors take it first. 4096 x 4096 is cut 4 ways (128 CTAs), 4096 x 14336 not
// at all (112 CTAs); a gate/up pair of 4096 x 14336 and 8192 x 28672 go in equal shares. The choice depends on the shape only, never on a matmul's place in a queue: the way the sums are grouped,
// and with it the last bit of a result, must not change with how matmuls are batched.
constexpr float kHbmBytesPerUs = 6.3e6f, kSmBytesPerUs = 50e3f, kHandOverUs = 2.f, kEarlyUs = 1.2f, kFourSlotsUs = 0.4f, kStraddleUs = 1.f;
float row_us(int tg) { return tg == 1 ? 0.07f : tg == 2 ? 0.1f : 0.145f; }
// Small matmuls: up to two tile rows of four-column sub-panels per SM. What they cost is the chain from x to the report, so
// nothing is handed over: sub-panels are as narrow as there are SMs for, whole, and their tile rows go round all warps.
// Every tile row's sums are added by themselves (see end_piece), as far as they fit: 84 KB.
bool deal_small(GemvParams &p, int ctas) {
  const int runs = p.TC / kWC, rest = p.TC % kWC, matrices = p.pair ? 2 : 1;
  if (p.units > 2 * ctas) return false;
  for (int lw = 0; lw <= 2; lw++) {
    const int w = 1 << lw, panels = (runs << (2 - lw)) + (rest + w - 1) / w, each = (panels + ctas - 1) / ctas;
    if (each > 1 && lw < 2) continue;
    if (p.KT * matrices * p.M * sum_stride(lw) * 4 > kSmallSums) continue;
    p.lw = lw, p.panels = panels, p.units = panels * p.KT, p.small = 1;
    p.parts = 0, p.share = each * p.KT, p.extra = 0, p.active = (panels + each - 1) / each;
    return true;
  }
  return false;
}
void deal_units(GemvParams &p, int ctas) {
  const int panels = (p.TC + kWC - 1) / kWC, matrices = p.pair ? 2 : 1;
  p.units = panels * p.KT, p.panels = panels, p.lw = 2, p.small = 0;
  if (deal_small(p, ctas)) return;
  const float hbm = (float)p.KT * p.TC * tile_bytes(p.fmt) * matrices / kHbmBytesPerUs;
  const float row = max(row_us(p.tg) * matrices, kWC * tile_bytes(p.fmt) * matrices / kSmBytesPerUs);   // us per tile row, an SM on its own
  auto stream = [&](float rows) { return max(hbm, rows * row); };
  auto shared = [&](int ranges) { return ranges > 1 ? kHandOverUs + kFourSlotsUs * ((ranges - 1 + kSlots - 1) / kSlots) : 0.f; };
  const int each = (panels + ctas - 1) / ctas;
  // whole sub-panels, or equal shares that straddle
  float best = stream((float)each * p.KT);
  p.parts = 0, p.share = each * p.KT, p.extra = 0, p.active = (p.units + p.share - 1) / p.share;
  const int busy = min(ctas, p.units), equal = p.units / busy;
  const float straddling = stream((float)p.units / busy) + kStraddleUs + (p.KT <= 2 * equal ? kEarlyUs : shared(p.KT / equal + 2));
  if (straddling < best) best = straddling, p.active = busy, p.share = equal, p.extra = p.units % busy;
  for (int parts = 2; parts <= p.KT && parts * panels <= ctas; parts++) {
    const float t = stream((float)((p.KT + parts - 1) / parts)) + shared(parts);
    if (t < best) best = t, p.parts = parts, p.active = parts * panels;
  }
}

// A matmul but for its place in a list and its tensor maps.
void describe(GemvParams &p, const bt_gemv_op &o, int ctas) {
  p.x = as_ptr<uint16_t>(o.x), p.w[0] = as_ptr<uint8_t>(o.w), p.w[1] = as_ptr<uint8_t>(o.w2), p.add = as_ptr<uint16_t>(o.add);
  p.out = as_ptr<void>(o.out), p.arg_val = as_ptr<float>(o.arg_val), p.arg_idx = as_ptr<int>(o.arg_idx);
  p.alpha = o.alpha, p.arg_base = o.arg_base, p.M = o.M, p.KT = o.K / 32, p.TC = o.N / 32, p.epi = o.epilogue, p.out_fp32 = o.out_dtype == BT_FP32 ? 1 : o.out_dtype == BT_FP32_ROWS ? 2 : 0;
  p.fmt = o.fmt, p.pair = o.epilogue == BT_EPI_GLU, p.tg = o.M <= 8 ? 1 : o.M <= 16 ? 2 : 4;
  p.from = p.to = p.add_from = 0;
  deal_units(p, ctas);
}
// Which matmuls of a chain take x from the exchange, and what those wait for.
void link(int n, GemvParams *op, const bt_gemv_op *ops, int sets) {
  for (int i = 1; i < n; i++) {
    GemvParams &p = op[i];
    if (!exchanged(ops, i)) continue;
    const int w = i - sets, v = w > 0 && wait_for(ops, w, sets) < w - 1 ? w - 1 : -1;
    p.from = op[i - 1].to = 1, p.add_from = p.add && ops[i].add == ops[i].x;
    p.early = w < 0 ? -1 : w, p.early_panels = w >= 0 ? op[w].panels : 0, p.early_also = v, p.early_also_panels = v >= 0 ? op[v].panels : 0;
  }
}

// The stages that a launch holds: every stage has to fit a chain's ring, and two of them any other's (see Ring).
constexpr int largest_stage(bool chain) {
  int most = 0;
  for (int fmt : {BT_BFP8, BT_BFP4})
    for (int tg = 1; tg <= (chain ? 1 : 4); tg *= 2)
      for (int lw = 0; lw <= 2; lw++)
        for (bool pair : {false, true}) most = std::max(most, chain ? geometry(fmt, pair, tg, lw).w_bytes : geometry(fmt, pair, tg, lw).stage);
  return most;
}
static_assert(kSmSums + kSmallSums + kAheadBytes + largest_stage(true) + 256 <= kSmemBytes, "a chain's ring has room for a stage");
static_assert(kSmSums + std::max(kSmallSums, sums_bytes(4)) + 2 * largest_stage(false) + 256 <= kSmemBytes, "the general kernel's ring has room for two stages");

// What a matmul's sums take of shared memory, and the ring of a launch behind them.
int sums_of(const GemvParams &p) { return p.small ? p.KT * (p.pair ? 2 : 1) * p.M * sum_stride(p.lw) * 4 : sums_bytes(p.tg); }
void lay_out(QueueHead &q, int sums, bool chained) {
  if (chained) sums += kAheadBytes;
  q.ring = kSmSums + (sums + 127) / 128 * 128, q.ring_bytes = (kSmemBytes - q.ring) / 128 * 128;
}
// Where a chain's matmuls run: the next one on other CTAs, which have its weights at hand when its x comes.
void take_turns(int n, GemvParams *op, int ctas) {
  for (int i = 0, start = 0; i < n; start = (start + op[i++].active) % ctas) op[i].turn = (ctas - start) % ctas;
}

// The tensor map of a matmul's x (one tile row of bf16 tiles): the staged token rows of each face are contiguous, a tile
// has its faces 512 bytes apart, and a copy takes the tile columns of one stage. And those of its weights, if sub-panels are
// narrower than the runs of the streaming layout.
int make_maps(GemvParams &p, uint64_t x) {
  const Geometry g = geometry(p.fmt, p.pair != 0, p.tg, p.lw);
  const uint32_t box[3] = {p.tg == 1 ? 128u : 256u, p.tg == 4 ? 4u : 2u, (uint32_t)g.ups};
  const uint64_t dims[3] = {box[0], box[1], (uint64_t)p.KT}, strides[2] = {512, 2048};
  if (int s = make_tmap(&p.xmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, as_ptr<void>(x), dims, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE)) return s;
  p.tiled = p.lw < 2 && p.TC >= kWC && p.KT >= g.ups;                 // else contiguous, or never a whole stage
  if (!p.tiled) return BT_OK;
  // weights in 8-byte elements: a tile is 136 or 72 of them
  const uint32_t wbox[3] = {(uint32_t)g.tb / 8, 1u << p.lw, (uint32_t)g.ups};
  const uint64_t wdims[3] = {wbox[0], kWC, (uint64_t)(p.TC / kWC) * p.KT}, wstrides[2] = {(uint64_t)g.tb, (uint64_t)kWC * g.tb};
  for (int m = 0; m < (p.pair ? 2 : 1); m++)
    if (int s = make_tmap(&p.wmap[m], CU_TENSOR_MAP_DATA_TYPE_UINT64, 3, p.w[m], wdims, wstrides, wbox, CU_TENSOR_MAP_SWIZZLE_NONE)) return s;
  return BT_OK;
}

}  // namespace

// Entry points stamp g_calls when they select their device.
bool bt::follows_matmul(uint64_t stream) {
  static std::mutex lock;
  static struct { uint64_t stream, stamp; } last[64] = {};
  std::lock_guard<std::mutex> hold(lock);
  const uint64_t now = g_calls.load(std::memory_order_relaxed);
  int slot = -1, spare = 0;
  for (int i = 0; i < 64; i++) {
    if (last[i].stamp && last[i].stream == stream) slot = i;
    if (last[i].stamp < last[spare].stamp) spare = i;
  }
  const bool yes = slot >= 0 && last[slot].stamp + 1 == now;
  if (slot < 0) slot = spare;
  last[slot].stream = stream, last[slot].stamp = now;
  return yes;
}

namespace {

// Argument checks and the launches shared by the entry points. `scratch` carries the scratch pointers.
int enqueue(const char *who, int device, int n, const bt_gemv_op *ops, const QueueHead &scratch, uint64_t stream) {
  BT_REQUIRE(n >= 1 && ops, "%s: needs at least one matmul", who);
  for (int i = 0; i < n; i++)
    if (int s = check_op(who, i, ops[i])) return s;
  if (int s = use_device(device)) return s;
  int sms = 0;
  BT_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  // The CTAs of a launch wait for one another, so all of them must fit on the GPU at once.
  static int resident[64] = {};
  if (!resident[device & 63]) {
    auto fits = [&](auto *kernel) -> int {
      BT_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes));
      int per_sm = 0;
      BT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kThreads, kSmemBytes));
      if (per_sm < 1) return fail(BT_DEVICE, "%s: the matmul kernel does not fit an SM of device %d", who, device);
      return BT_OK;
    };
    if (int s = fits(chain_kernel<kQueueShort>)) return s;
    if (int s = fits(chain_kernel<kQueueMax>)) return s;
    if (int s = fits(gemv_queue_kernel<true, kQueueShort>)) return s;
    if (int s = fits(gemv_queue_kernel<true, kQueueMax>)) return s;
    if (int s = fits(gemv_queue_kernel<false, kQueueShort>)) return s;
    if (int s = fits(gemv_queue_kernel<false, kQueueMax>)) return s;
    resident[device & 63] = 1;
  }
  const int ctas = min(sms, kMaxCtas);
  for (int base = 0; base < n; base += kQueueMax) {
    Queue<kQueueMax> q;
    static_cast<QueueHead &>(q) = scratch;
    q.n = min(kQueueMax, n - base);
    q.panels = 0;
    int sums = 0;
    bool small = false;
    for (int i = 0; i < q.n; i++) {
      const bt_gemv_op &o = ops[base + i];
      GemvParams &p = q.op[i];
      describe(p, o, ctas);
      const Gate g = gate(ops + base, i, scratch.sets);
      p.wait_for = g.last, p.wait_also = g.also;
      p.turn = (int)(((long long)(base + i) * 101) % ctas);
      p.wait_panels = g.last >= 0 ? q.op[g.last].panels : 0, p.also_panels = g.also >= 0 ? q.op[g.also].panels : 0;
      q.panels += p.panels;
      small |= p.small;
      if (int s = make_maps(p, o.x)) return s;
      sums = max(sums, sums_of(p));
    }
    const bool chained = scratch.exchange && chain(q.n, q.op, ops + base);
    if (chained) {
      take_turns(q.n, q.op, ctas);
      link(q.n, q.op, ops + base, scratch.sets);
    }
    lay_out(q, sums, chained);
    // Programmatic dependent launch: this grid may begin while the previous launch of the stream is still finishing.
    // It only sets up and prefetches weights until its x warps pass griddepcontrol.wait. Weights read that early must
    // be in place, so the launch overlaps its predecessor only when that was a matmul launch of this file too (which
    // never writes weights): anything else this library queued in between (a cast, a relayout, a copy, a memset)
    // turns the overlap off for the next matmul launch.
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas), cfg.blockDim = dim3(kThreads), cfg.dynamicSmemBytes = kSmemBytes, cfg.stream = as_stream(stream);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr, cfg.numAttrs = base > 0 || follows_matmul(stream) ? 1 : 0;
    if (q.n <= kQueueShort) {
      Queue<kQueueShort> s;
      static_cast<QueueHead &>(s) = q;
      std::copy(q.op, q.op + q.n, s.op);
      BT_CUDA(chained ? cudaLaunchKernelEx(&cfg, chain_kernel<kQueueShort>, s) : small ? cudaLaunchKernelEx(&cfg, gemv_queue_kernel<true, kQueueShort>, s) : cudaLaunchKernelEx(&cfg, gemv_queue_kernel<false, kQueueShort>, s));
    } else BT_CUDA(chained ? cudaLaunchKernelEx(&cfg, chain_kernel<kQueueMax>, q) : small ? cudaLaunchKernelEx(&cfg, gemv_queue_kernel<true, kQueueMax>, q) : cudaLaunchKernelEx(&cfg, gemv_queue_kernel<false, kQueueMax>, q));
    if (int st = launched(chained ? "chain_kernel" : "gemv_queue_kernel")) return st;
  }
  return BT_OK;
}

Scratch scratch_at(unsigned char *set) {
  Scratch s;
  s.panels_done = reinterpret_cast<int *>(set + kSetPanelsDone), s.counters = reinterpret_cast<int *>(set + kSetCounters);
  s.keys = reinterpret_cast<unsigned long long *>(set + kSetKeys);
  s.partials = reinterpret_cast<float *>(set + kSetPartials);
  return s;
}

QueueHead workspace_scratch(uint64_t work) {
  QueueHead q{};
  unsigned char *base = as_ptr<unsigned char>(work);
  q.error = reinterpret_cast<int *>(base + kWsError), q.ops_done = reinterpret_cast<int *>(base + kWsOpsDone), q.all_done = reinterpret_cast<int *>(base + kWsAllDone);
  q.sets = kSets;
  for (int s = 0; s < kSets; s++) q.set[s] = scratch_at(base + kWsSets + s * kSetBytes);
  q.slot_floats = (int)kSlotFloatsMax;
  q.epoch = reinterpret_cast<uint32_t *>(base + kWsEpoch), q.exchange = base + kWsExchange;
  return q;
}

}  // namespace

// ---- the entry point that allocates nothing -------------------------------------------------------------------
// Scratch for bt_gemv_bfp_static lives in this array, inside the library's device image, so a caller that may
// not allocate device memory still has somewhere for the kernel's counters and partial sums. Every device that
// loads the library holds these bytes until the process exits. The layout mirrors the caller-provided workspace
// at reduced limits: up to 8 rows of x, up to kStaticSubPanels sub-panels of 4 tile columns.
namespace {
constexpr int kStaticSubPanels = 4096;                                  // N <= 4096 * 4 * 32 = 524288 columns
constexpr size_t kStaticSlotFloats = 8 * 2 * 128;                       // 8 tokens x up to two matrices x 128 channels
constexpr size_t kStKeys = 256;
constexpr size_t kStCounters = 512;
constexpr size_t kStControlBytes = kStCounters + 4 * (size_t)kStaticSubPanels;   // what must be zero when a call starts
constexpr size_t kStPartials = kStControlBytes;
constexpr size_t kStaticBytes = kStPartials + (size_t)kMaxCtas * kStaticSlotFloats * 4;   // about 1.3 MB
}  // namespace
static __device__ __align__(256) unsigned char g_static_scratch[kStaticBytes];

extern "C" {

int bt_gemv_workspace_bytes(int device, size_t *bytes) {
  BT_REQUIRE(bytes, "bt_gemv_workspace_bytes: null result");
  (void)device;
  *bytes = kWsBytes;
  return BT_OK;
}

int bt_gemv_queue(int device, int n, const bt_gemv_op *ops, uint64_t work, size_t work_bytes, uint64_t stream) {
  BT_REQUIRE(work && work % 16 == 0 && work_bytes >= kWsBytes, "bt_gemv_queue: needs %zu bytes of 16-byte aligned scratch, got %zu", kWsBytes, work_bytes);
  return enqueue("bt_gemv_queue", device, n, ops, workspace_scratch(work), stream);
}

int bt_gemv_queue_plan(int n, const bt_gemv_op *ops, int *waits) {
  BT_REQUIRE(n >= 1 && ops && waits, "bt_gemv_queue_plan: needs at least one matmul and somewhere for the answer");
  for (int i = 0; i < n; i++)
    if (int s = check_op("bt_gemv_queue_plan", i, ops[i])) return s;
  for (int i = 0; i < n; i++) {
    const int base = i / kQueueMax * kQueueMax, w = wait_for(ops + base, i - base, kSets);
    waits[i] = w < 0 ? -1 : base + w;
  }
  return BT_OK;
}

int bt_gemv_queue_gates(int n, const bt_gemv_op *ops, int *gates) {
  BT_REQUIRE(n >= 1 && ops && gates, "bt_gemv_queue_gates: needs at least one matmul and somewhere for the answer");
  for (int i = 0; i < n; i++)
    if (int s = check_op("bt_gemv_queue_gates", i, ops[i])) return s;
  for (int i = 0; i < n; i++) {
    const int base = i / kQueueMax * kQueueMax;
    const Gate g = gate(ops + base, i - base, kSets);
    gates[2 * i] = g.last < 0 ? -1 : base + g.last, gates[2 * i + 1] = g.also < 0 ? -1 : base + g.also;
  }
  return BT_OK;
}

int bt_gemv_queue_links(int sms, int n, const bt_gemv_op *ops, int *links) {
  BT_REQUIRE(sms >= 1 && n >= 1 && ops && links, "bt_gemv_queue_links: needs a GPU's number of SMs, at least one matmul and somewhere for the answer");
  for (int i = 0; i < n; i++)
    if (int s = check_op("bt_gemv_queue_links", i, ops[i])) return s;
  for (int base = 0; base < n; base += kQueueMax) {
    GemvParams op[kQueueMax];
    const int count = min(kQueueMax, n - base);
    for (int i = 0; i < count; i++) describe(op[i], ops[base + i], min(sms, kMaxCtas));
    const bool chained = chain(count, op, ops + base);
    if (chained) link(count, op, ops + base, kSets);
    for (int i = 0; i < count; i++) links[base + i] = chained ? op[i].from : -1;
  }
  return BT_OK;
}

int bt_gemv_queue_rooms(int sms, int n, const bt_gemv_op *ops, int *rooms) {
  BT_REQUIRE(sms >= 1 && n >= 1 && ops && rooms, "bt_gemv_queue_rooms: needs a GPU's number of SMs, at least one matmul and somewhere for the answer");
  for (int i = 0; i < n; i++)
    if (int s = check_op("bt_gemv_queue_rooms", i, ops[i])) return s;
  const int ctas = min(sms, kMaxCtas);
  for (int base = 0; base < n; base += kQueueMax) {
    GemvParams op[kQueueMax];
    QueueHead q{};
    const int count = min(kQueueMax, n - base);
    int sums = 0;
    for (int i = 0; i < count; i++) describe(op[i], ops[base + i], ctas), sums = max(sums, sums_of(op[i])), rooms[2 * (base + i)] = rooms[2 * (base + i) + 1] = 0;
    if (!chain(count, op, ops + base)) continue;
    lay_out(q, sums, true), take_turns(count, op, ctas);
    for (int cta = 0; cta < ctas; cta++) {
      Ring ring{0};
      for (int i = 0; i < count; i++) {
        rooms[2 * (base + i)] = q.ring_bytes;
        if ((cta + op[i].turn) % ctas >= op[i].active) continue;
        const Geometry g = geometry(op[i].fmt, op[i].pair != 0, op[i].tg, op[i].lw);
        for (int k = 0; k < op[i].KT; k += g.ups) {              // (a whole sub-panel: see chain)
          bool alone;
          rooms[2 * (base + i) + 1] = max(rooms[2 * (base + i) + 1], (int)ring.room<true>(g.w_bytes, q.ring_bytes, &alone));
          ring.place(g.w_bytes, q.ring_bytes);
        }
      }
    }
  }
  return BT_OK;
}

int bt_gemv_bfp(int device, int fmt, int epilogue, int M, int K, int N, uint64_t x, uint64_t w, uint64_t w2, uint64_t add,
                float alpha, uint64_t out, int out_dtype, uint64_t arg_val, uint64_t arg_idx, int arg_base, uint64_t work,
                size_t work_bytes, uint64_t stream) {
  BT_REQUIRE(work && work % 16 == 0 && work_bytes >= kWsBytes, "bt_gemv_bfp: needs %zu bytes of 16-byte aligned scratch, got %zu", kWsBytes, work_bytes);
  const bt_gemv_op op = {fmt, epilogue, M, K, N, out_dtype, arg_base, alpha, x, w, w2, add, out, arg_val, arg_idx};
  return enqueue("bt_gemv_bfp", device, 1, &op, workspace_scratch(work), stream);
}

// The device address of g_static_scratch on `device`, looked up once per device. In host code the array's name is
// only a handle for the runtime, not an address a kernel could use, so the address comes from
// cudaGetSymbolAddress, asked with that device current.
static int static_scratch(int device, unsigned char **base) {
  static unsigned char *bases[64] = {};
  BT_REQUIRE(device >= 0 && device < 64, "bt_gemv_bfp_static: device %d is out of range", device);
  if (!bases[device]) {
    if (int s = use_device(device)) return s;
    void *ptr = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&ptr, g_static_scratch);
    if (e != cudaSuccess || !ptr) return fail(BT_DEVICE, "bt_gemv_bfp_static: no address for the built-in scratch on device %d: %s", device, cudaGetErrorString(e));
    bases[device] = static_cast<unsigned char *>(ptr);
  }
  *base = bases[device];
  return BT_OK;
}

int bt_gemv_bfp_static(int device, int fmt, int epilogue, int M, int K, int N, uint64_t x, uint64_t w, uint64_t w2, uint64_t add,
                       float alpha, uint64_t out, int out_dtype, uint64_t arg_val, uint64_t arg_idx, int arg_base, uint64_t stream) {
  BT_REQUIRE(M <= 8, "bt_gemv_bfp_static: the built-in scratch holds up to 8 rows of x, not %d; use bt_gemv_bfp with your own scratch", M);
  BT_REQUIRE(N <= kStaticSubPanels * 128, "bt_gemv_bfp_static: the built-in scratch holds up to %d columns, not %d; use bt_gemv_bfp with your own scratch",
             kStaticSubPanels * 128, N);
  const bt_gemv_op op = {fmt, epilogue, M, K, N, out_dtype, arg_base, alpha, x, w, w2, add, out, arg_val, arg_idx};
  if (int s = check_op("bt_gemv_bfp_static", 0, op)) return s;
  unsigned char *base = nullptr;
  if (int s = static_scratch(device, &base)) return s;
  if (int s = use_device(device)) return s;
  // the array keeps whatever the last call left: the arrival counters must start at zero. The wait-gave-up word at
  // its start is left alone, so that it stays until bt_gemv_check(device, 0, ...) reads it.
  BT_CUDA(cudaMemsetAsync(base + kWsOpsDone, 0, kStControlBytes - kWsOpsDone, as_stream(stream)));
  QueueHead scratch{};
  scratch.error = reinterpret_cast<int *>(base + kWsError), scratch.ops_done = reinterpret_cast<int *>(base + kWsOpsDone), scratch.all_done = reinterpret_cast<int *>(base + kWsAllDone);
  scratch.sets = 1;
  scratch.set[0].panels_done = reinterpret_cast<int *>(base + 192), scratch.set[0].counters = reinterpret_cast<int *>(base + kStCounters);
  scratch.set[0].keys = reinterpret_cast<unsigned long long *>(base + kStKeys);
  scratch.set[0].partials = reinterpret_cast<float *>(base + kStPartials);
  scratch.slot_floats = (int)kStaticSlotFloats;
  return enqueue("bt_gemv_bfp_static", device, 1, &op, scratch, stream);
}

// Nonzero once a bounded wait inside a launch that used this scratch gave up; the results of that launch are
// then unreliable. Reads the flag back (synchronising the stream) and, if it was set, clears it together with the
// counters a launch that gave up may have left half-counted, so that the next launch starts clean. `work` = 0 means
// the built-in scratch of bt_gemv_bfp_static on `device`.
int bt_gemv_check(int device, uint64_t work, uint64_t stream, int *error) {
  BT_REQUIRE(error, "bt_gemv_check: null result");
  unsigned char *base = as_ptr<unsigned char>(work);
  if (!work) {
    if (int s = static_scratch(device, &base)) return s;
  }
  if (int s = use_device(device)) return s;
  BT_CUDA(cudaMemcpyAsync(error, base + kWsError, 4, cudaMemcpyDeviceToHost, as_stream(stream)));
  BT_CUDA(cudaStreamSynchronize(as_stream(stream)));
  if (*error) {
    BT_CUDA(cudaMemsetAsync(base, 0, work ? kWsBytes : kStaticBytes, as_stream(stream)));
  }
  return BT_OK;
}

}  // extern "C"
