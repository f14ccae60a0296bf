// Prefill matmul for many token rows: out = epilogue(alpha * x @ W + add), W block-float in streaming layout.
//
// With hundreds of rows the contraction is dense and belongs on the 5th-generation tensor cores. What bounds it on
// one SM is shared-memory bandwidth, not the tensor pipe: every MMA reads its A and B slabs from shared memory while
// TMA writes the next x tiles and the dequantising warps write the next expanded weights. So two CTAs on neighbouring
// SMs work as a pair (a cluster of two, tcgen05 cta_group::2): one MMA of 256 rows x 256 columns takes 128 rows of
// x from each CTA and 128 weight columns from each CTA, so each CTA stages, expands and feeds only half of the
// weights, and each B slab is read from shared memory once for 256 rows instead of once for every 128.
//
// A pair computes a block of 512 (or, for few rows, 256) rows x 256 MMA columns; each CTA holds its rows' fp32
// accumulators in tensor memory (two halves of 256 columns). For a gate/up pair the 256 MMA columns are 128 columns
// of Wg (CTA 0) next to the same 128 columns of Wu (CTA 1), and the epilogue writes silu(gate) * up for 128 columns.
//
// Per 64-deep K block, in each CTA:
//   warp 0   (producer)  TMA-loads its 128 x 64 tiles of x (row-major bf16, 128-byte swizzle), whose bytes complete
//                        directly on the LEADER CTA's "full" barrier (a cta_group::2 load; the leader arms the barrier
//                        for both CTAs' bytes), and bulk-copies its 8 packed weight tiles (one run of the streaming
//                        layout, two tile rows) into a ring.
//   warps 2-9 (dequant)  (and 10-17, which take every other K block, where a pair has 256 rows: there a K block's expansion
//                        takes longer than its MMAs) each takes one packed tile, expands it to exact bf16 in registers the way the decode kernel
//                        does (a mask or byte permute, then a packed multiply-add with the face row's power of two),
//                        and stores it into the B tile in the K-major 128-byte-swizzled layout the MMA reads. The
//                        weights carry a factor 2^-64, undone in the epilogue. When its tile is stored and fenced
//                        for the tensor core, the warp arrives on the leader CTA's "full" barrier (17 arrivals in
//                        all: 8 warps of each CTA and the leader's producer).
//   warp 1   (MMA)       in the leader CTA one lane issues 2 x 4 tcgen05.mma (256 x 256 x 16 each) and commits to
//                        both CTAs; the commit frees the stage for both producers and all dequant warps.
// After the last K block the dequant warps become the epilogue: tcgen05.ld brings 32 rows x 32 columns per warp into
// registers, the addend and the activation are applied, and bf16 (rounded half up) or fp32 goes out in tile layout.
// N needs no alignment (a last run of fewer than 4 tile columns is staged tile row by tile row, a missing run is
// skipped); K is a multiple of 32 (an odd last tile row issues half the MMAs of a K block).
// Every wait is bounded and reports through the error word instead of hanging; both CTAs meet at a cluster barrier
// before either frees its tensor memory or exits, so neither signals a barrier of a CTA that has gone.
#include "common.cuh"
#include "ptx.cuh"
#include "expand.cuh"
#include "tmap.cuh"
#include <cstring>

using namespace bt;

namespace {

constexpr int kBK = 64;                                  // K block
constexpr int kStagesAB = 3, kStagesP = 4;             // four stages of x and weights measured the same as three
constexpr int kDequantWarps = 8;
constexpr int threads_of(int groups) { return (2 + groups * kDequantWarps) * 32; }
constexpr uint32_t kWaitLimit = 1u << 14;                // attempts of up to 100 us each

constexpr int kABytes = 128 * 128;                       // one 128-row half of this CTA's x for a K block
constexpr int kBBytes = 128 * 128;                       // this CTA's 128 expanded weight columns for a K block
constexpr int kStageAB = 2 * kABytes + kBBytes;          // 48 KiB

struct GemmParams {
  const uint8_t *w[2];       // packed weights by columns; w[1] only for the gate/up pair
  const uint16_t *add;       // addend tiles (bf16), or null
  size_t add_row_stride;     // datums from one tile row of the addend to the next; 0 when the addend is one row
  void *out;
  int *error;
  float alpha;
  int M, KT, TC, epi, out_fp32, pair;
  int row_blocks;            // blocks of 512 rows, or of 256 where `half`
  int half;                  // every pair takes 256 rows
  int splits;                // pairs of CTAs that share a block, each with its part of K; their sums meet in `part`
  int weights_early;         // the launch before this one laid x out by rows
  float *part;               // [split][gate, up][tile_rows * 32][TC * 32] fp32, where splits > 1
  int whole;                 // pairs of CTAs that take a whole block of 512 rows x 256 MMA columns; the pairs after them
};                           // take half a block (256 rows) each, so that the last wave of the grid is a short one

template <int FMT>
struct Layout {
  static constexpr int TB = tile_bytes(FMT);
  static constexpr int P_STAGE = 8 * TB;                  // packed tiles of one K block: 2 tile rows x 4 tile columns
  static constexpr int AB0 = 1024;                        // barriers and the tensor-memory address live below
  static constexpr int P0 = AB0 + kStagesAB * kStageAB;
  static constexpr int BYTES = P0 + kStagesP * P_STAGE;
};

// Shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFF) >> 4) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// Instruction descriptor: fp32 accumulator, bf16 A and B, both K-major, N = 256, M = 256 (128 rows in each CTA).
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(256 >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);

// Expand one packed tile (streaming layout, shared address `tile`) to bf16 and store it as rows [32 c, 32 c + 32) and
// K columns [32 j, 32 j + 32) of the B tile at shared address `b` (K-major, 128-byte rows, 128-byte swizzle: the
// 16-byte chunk index of a row is XORed with the row's index modulo 8).
template <int FMT>
__device__ __forceinline__ void expand_tile(uint32_t tile, uint32_t b, int c, int j, int lane) {
  const int g = lane >> 2, t = lane & 3;
  uint32_t a[2][2][4];
  expand_weights<FMT>(packed_lane<FMT>(tile, lane), a);
#pragma unroll
  for (int h = 0; h < 2; h++)
#pragma unroll
    for (int fs = 0; fs < 2; fs++) {
      const int n0 = 32 * c + 16 * fs + 2 * g;                       // even, so n0 and n0 + 1 share an 8-row group
      const int chunk = 4 * j + 2 * h + (t >> 1);                    // 16-byte chunk of k = 32 j + 16 h + 4 t
      const uint32_t group = b + (n0 >> 3) * 1024 + (t & 1) * 8;
      sts64(group + (n0 & 7) * 128 + ((chunk ^ (n0 & 7)) << 4), a[h][fs][0], a[h][fs][2]);
      sts64(group + ((n0 + 1) & 7) * 128 + ((chunk ^ ((n0 + 1) & 7)) << 4), a[h][fs][1], a[h][fs][3]);
    }
}

// SPLIT: the pairs share K. A kernel of its own, since whole blocks lose 2 % to the K block a pair starts at and the sums that
// go out as they are.
template <int FMT, bool SPLIT, int GROUPS>
__global__ void __launch_bounds__(threads_of(GROUPS), 1) gemm_kernel(const GemmParams p, const __grid_constant__ CUtensorMap amap) {
  using L = Layout<FMT>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);   // swizzled tiles want 1024-byte alignment
  const uint32_t sb = smem_u32(smem);
  const uint32_t full0 = sb, empty0 = sb + 32, pfull0 = sb + 96, pempty0 = sb + 128, acc_full = sb + 160, tmem_slot = sb + 176;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();                          // 0: the leader, which issues the MMAs
  const int KB = (p.KT + 1) / 2;                                    // K blocks of 64; the last may hold one tile row
  const int pair_id = blockIdx.x >> 1;
  const int split = SPLIT ? pair_id % p.splits : 0, kb0 = SPLIT ? KB * split / p.splits : 0, kbs = SPLIT ? KB * (split + 1) / p.splits - kb0 : KB;   // this pair's K blocks
  const int block = SPLIT ? pair_id / p.splits : pair_id < p.whole ? pair_id : p.whole + ((pair_id - p.whole) >> 1);   // blocks go down the rows first
  const int bc = block / p.row_blocks;                              // block column: 128 output columns (pair) or 256
  const bool all_rows = !p.half && (SPLIT || pair_id < p.whole);
  const int pair_m0 = (block % p.row_blocks) * (p.half ? 256 : 512) + (p.half || all_rows ? 0 : ((pair_id - p.whole) & 1) * 256);   // first row of the pair's rows
  const int MH = all_rows && pair_m0 + 256 < p.M ? 2 : 1;           // halves of 256 rows this pair computes
  if (pair_m0 >= p.M) return;                                       // (both CTAs of the pair: nothing here)
  const int run = p.pair ? bc : 2 * bc + (int)rank;                 // this CTA's run of 4 tile columns
  const int width = min(kPanel, p.TC - run * kPanel);               // tile columns it really has; <= 0: none
  const uint8_t *wsrc = (p.pair ? p.w[rank] : p.w[0]) + (size_t)run * kPanel * p.KT * L::TB;
  auto row0 = [&](int mh) { return pair_m0 + (2 * mh + (int)rank) * 128; };   // first row of this CTA's half mh
  auto a_tile = [&](int s, int mh) { return sb + L::AB0 + s * kStageAB + mh * kABytes; };
  auto b_tile = [&](int s) { return sb + L::AB0 + s * kStageAB + 2 * kABytes; };
  auto p_stage = [&](int ps) { return sb + L::P0 + ps * L::P_STAGE; };
  auto wait = [&](uint32_t bar, uint32_t parity, int code) {
    if (!mbar_wait(bar, parity, kWaitLimit)) atomicExch(p.error, code);
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStagesAB; s++) mbar_init(full0 + 8 * s, 1 + 2 * kDequantWarps), mbar_init(empty0 + 8 * s, 1);
    for (int s = 0; s < kStagesP; s++) mbar_init(pfull0 + 8 * s, 1), mbar_init(pempty0 + 8 * s, kDequantWarps);
    mbar_init(acc_full, 1);
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc_pair(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  cluster_sync();                                                   // the peer's barriers exist before anyone signals them
  tc_fence_after();
  // All of that may happen while the launch before this one drains. What that one writes is read, and what it reads written, only
  // behind this wait: x, the addend, the result. Where it is the one that lays x out by rows, everything before it is
  // complete (its blocks wait for that before they let this launch come up), so the weights need not wait, and the first
  // of them are expanded by the time x is there.
  auto in_turn = [] { asm volatile("griddepcontrol.wait;" ::: "memory"); };
  if (!p.weights_early) in_turn();
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(smem + 176);

  if (warp == 0) {
    // ---- producer ----
    if (lane == 0) {
      const uint32_t leader_full = map_to_cta(full0, 0);
      auto packed = [&](int i) {            // the i-th K block's packed tiles of this CTA's run: up to 2 tile rows x 4 tiles
        if (width <= 0) return;
        const int kb = kb0 + i, ps = i % kStagesP, rows = min(2, p.KT - 2 * kb);
        if (i >= kStagesP) wait(pempty0 + 8 * ps, (i / kStagesP - 1) & 1, 11);
        mbar_expect_tx(pfull0 + 8 * ps, rows * width * L::TB);
        const uint8_t *src = wsrc + (size_t)(2 * kb) * width * L::TB;
        if (width == kPanel) bulk_g2s(p_stage(ps), src, rows * kPanel * L::TB, pfull0 + 8 * ps);
        else
          for (int j = 0; j < rows; j++) bulk_g2s(p_stage(ps) + j * kPanel * L::TB, src + (size_t)j * width * L::TB, width * L::TB, pfull0 + 8 * ps);
      };
      for (int i = 0; i < min(kbs, kStagesP - 1); i++) packed(i);
      in_turn();
      for (int i = 0; i < kbs; i++) {
        if (i + kStagesP - 1 < kbs) packed(i + kStagesP - 1);
        const int s = i % kStagesAB;
        if (i >= kStagesAB) wait(empty0 + 8 * s, (i / kStagesAB - 1) & 1, 12);
        // the x tiles of BOTH CTAs complete on the leader's barrier, which the leader arms for all of them
        if (rank == 0) mbar_expect_tx(full0 + 8 * s, 2 * MH * kABytes);
        for (int mh = 0; mh < MH; mh++) tma_load_2d_pair(a_tile(s, mh), &amap, (kb0 + i) * kBK, row0(mh), leader_full + 8 * s);   // past M or K: zeros
      }
    }
  } else if (warp == 1) {
    // ---- MMA issuer: the leader CTA alone ----
    if (lane == 0 && rank == 0) {
      for (int i = 0; i < kbs; i++) {
        const int s = i % kStagesAB, steps = 2 * min(2, p.KT - 2 * (kb0 + i));   // 16-deep MMAs in this K block
        wait(full0 + 8 * s, (i / kStagesAB) & 1, 13);
        tc_fence_after();
        for (int mh = 0; mh < MH; mh++)
          for (int kk = 0; kk < steps; kk++)
            umma_bf16_pair(tmem + mh * 256, smem_desc(a_tile(s, mh) + kk * 32), smem_desc(b_tile(s) + kk * 32), kIdesc, (i | kk) != 0);
        umma_commit_pair(empty0 + 8 * s);
      }
      umma_commit_pair(acc_full);
    }
  } else {
    // ---- dequant warps, then the epilogue ----
    const int d = warp - 2, c = d & 3, j = d >> 2 & 1;                  // this warp's tile column and tile row in a K block
    const uint32_t leader_full0 = map_to_cta(full0, 0);
    for (int i = d / kDequantWarps; i < kbs; i += GROUPS) {
      const int ps = i % kStagesP, s = i % kStagesAB;
      if (width > 0) wait(pfull0 + 8 * ps, (i / kStagesP) & 1, 14);
      if (i >= kStagesAB) wait(empty0 + 8 * s, (i / kStagesAB - 1) & 1, 15);
      tc_fence_after();
      if (c < width && 2 * (kb0 + i) + j < p.KT) expand_tile<FMT>(p_stage(ps) + (j * kPanel + c) * L::TB, b_tile(s), c, j, lane);
      fence_async_shared();
      __syncwarp();
      if (lane == 0) {
        if (width > 0) mbar_arrive(pempty0 + 8 * ps);
        mbar_arrive_cluster(leader_full0 + 8 * s);
      }
    }
    in_turn();
    wait(acc_full, 0, 16);
    tc_fence_after();
    const int q = warp & 3, ch = d >> 2;                            // tensor-memory lane quarter; column half
    const float unscale = kExpandedUnscale * p.alpha;
    const int out_cols = p.pair ? 128 : 256, part = out_cols / (2 * GROUPS);   // this warp's columns
    constexpr int COLS = GROUPS == 1 ? 32 : 16;                     // and how many at a time: 32 need more registers than 18 warps have
    const int tile_rows = (p.M + 31) / 32;
#pragma unroll 1
    for (int mh = 0; mh < MH; mh++) {
      const int row = row0(mh) + 32 * q + lane, tr = row >> 5;
      if (tr >= tile_rows) continue;                                // the whole warp is past the tensor's tile rows
#pragma unroll 1
      for (int col = ch * part; col < (ch + 1) * part; col += COLS) {   // first output column, within the block
        const int tcol = bc * (out_cols / 32) + (col >> 5);         // its tile column
        if (tcol >= p.TC) continue;
        uint32_t v[COLS], u[COLS];
        tmem_ld(tmem + ((uint32_t)(32 * q) << 16) + mh * 256 + col, v);
        if (p.pair) tmem_ld(tmem + ((uint32_t)(32 * q) << 16) + mh * 256 + 128 + col, u);
        tmem_ld_wait();
        if (SPLIT) {
          // sums of a part of K, as they are: reduce_kernel adds the parts
          if (row < p.M) {
            const size_t cols = (size_t)p.TC * 32, plane = (size_t)tile_rows * 32 * cols;
            float *o = p.part + (size_t)split * (p.pair ? 2 : 1) * plane + (size_t)row * cols + tcol * 32 + (col & 16);
#pragma unroll
            for (int i = 0; i < COLS / 4; i++) reinterpret_cast<uint4 *>(o)[i] = make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
            if (p.pair) {
#pragma unroll
              for (int i = 0; i < COLS / 4; i++) reinterpret_cast<uint4 *>(o + plane)[i] = make_uint4(u[4 * i], u[4 * i + 1], u[4 * i + 2], u[4 * i + 3]);
            }
          }
          continue;
        }
        const int in_tile = ((row >> 4) & 1) * 512 + (col & 16) * 16 + (row & 15) * 16;    // datum index of (row, col) in the tile
        uint32_t w[COLS / 2] = {};
        if (p.add) {
          const uint4 *a = reinterpret_cast<const uint4 *>(p.add + (size_t)tr * p.add_row_stride + (size_t)tcol * 1024 + (p.add_row_stride ? in_tile : (col & 16) * 16));
#pragma unroll
          for (int i = 0; i < COLS / 8; i++) {
            const uint4 a4 = a[i / 2 * 32 + i % 2];
            w[4 * i] = a4.x, w[4 * i + 1] = a4.y, w[4 * i + 2] = a4.z, w[4 * i + 3] = a4.w;
          }
        }
        float f[COLS];
#pragma unroll
        for (int i = 0; i < COLS; i++) {
          float x = __uint_as_float(v[i]) * unscale;
          if (p.add) x += __uint_as_float(i % 2 ? w[i / 2] & 0xFFFF0000u : w[i / 2] << 16);
          if (p.pair) x = silu(x) * (__uint_as_float(u[i]) * unscale);
          else if (p.epi == BT_EPI_RELU) x = fmaxf(x, 0.f);
          else if (p.epi == BT_EPI_SILU) x = silu(x);
          f[i] = row < p.M ? x : 0.f;
        }
        const size_t at = ((size_t)tr * p.TC + tcol) * 1024 + in_tile;
        if (p.out_fp32) {
          float4 *o = reinterpret_cast<float4 *>(static_cast<float *>(p.out) + at);
#pragma unroll
          for (int i = 0; i < COLS / 4; i++) o[i / 4 * 64 + i % 4] = make_float4(f[4 * i], f[4 * i + 1], f[4 * i + 2], f[4 * i + 3]);
        } else {
          uint4 *o = reinterpret_cast<uint4 *>(static_cast<uint16_t *>(p.out) + at);
#pragma unroll
          for (int k = 0; k < COLS / 2; k++) w[k] = bf16_half_up(f[2 * k]) | bf16_half_up(f[2 * k + 1]) << 16;
#pragma unroll
          for (int i = 0; i < COLS / 8; i++) o[i / 2 * 32 + i % 2] = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();                                                   // neither CTA frees or leaves while the other may still use it
  if (warp == 1) tmem_dealloc_pair(tmem, 512);
}

// The parts of K added in order, and the epilogue: one thread to four neighbouring columns of a row, 16 bytes of each part
// (which L2 still holds) and 8 or 16 bytes of the result.
__global__ void __launch_bounds__(256) reduce_kernel(const GemmParams p) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int quads = p.TC * 8, tile_rows = (p.M + 31) / 32;
  const unsigned i = blockIdx.x * 256u + threadIdx.x;
  if (i >= (unsigned)tile_rows * 32 * quads) return;
  const int row = i / quads, col = (i - row * quads) * 4, tcol = col >> 5, tr = row >> 5;
  const size_t cols = (size_t)p.TC * 32, plane = (size_t)tile_rows * 32 * cols;
  const float unscale = kExpandedUnscale * p.alpha;
  float f[4] = {0.f, 0.f, 0.f, 0.f}, g[4] = {0.f, 0.f, 0.f, 0.f};
  const int at = ((row >> 4) & 1) * 512 + (row & 15) * 16 + ((col >> 4) & 1) * 256 + (col & 15);   // datum index in the tile
  if (row < p.M) {
    const float *from = p.part + (size_t)row * cols + col;
    for (int s = 0; s < p.splits; s++) {
      const float4 a = __ldcg(reinterpret_cast<const float4 *>(from));
      f[0] += a.x, f[1] += a.y, f[2] += a.z, f[3] += a.w;
      if (p.pair) {
        const float4 b = __ldcg(reinterpret_cast<const float4 *>(from + plane));
        g[0] += b.x, g[1] += b.y, g[2] += b.z, g[3] += b.w;
      }
      from += (p.pair ? 2 : 1) * plane;
    }
    uint2 a = make_uint2(0, 0);
    if (p.add) a = *reinterpret_cast<const uint2 *>(p.add + (size_t)tr * p.add_row_stride + (size_t)tcol * 1024 + (p.add_row_stride ? at : ((col >> 4) & 1) * 256 + (col & 15)));
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const uint32_t w = k < 2 ? a.x : a.y;
      float x = f[k] * unscale;
      if (p.add) x += __uint_as_float(k % 2 ? w & 0xFFFF0000u : w << 16);
      if (p.pair) x = silu(x) * (g[k] * unscale);
      else if (p.epi == BT_EPI_RELU) x = fmaxf(x, 0.f);
      else if (p.epi == BT_EPI_SILU) x = silu(x);
      f[k] = x;
    }
  }
  const size_t o = ((size_t)tr * p.TC + tcol) * 1024 + at;
  if (p.out_fp32) *reinterpret_cast<float4 *>(static_cast<float *>(p.out) + o) = make_float4(f[0], f[1], f[2], f[3]);
  else *reinterpret_cast<uint2 *>(static_cast<uint16_t *>(p.out) + o) = make_uint2(bf16_half_up(f[0]) | bf16_half_up(f[1]) << 16, bf16_half_up(f[2]) | bf16_half_up(f[3]) << 16);
}

// How the blocks of a matmul are dealt out to the `slots` pairs of CTAs that fit on the GPU at once: pairs, and in `p` what
// they do. With at least as many blocks as slots the pairs take whole blocks, and when they do not fill the last wave, the
// blocks of that wave are cut in two, so that it takes half as long (as long as the halves still fit in one wave). With
// fewer, which is what prompts of some hundred rows and few columns have, blocks of 256 rows and blocks whose K is shared
// by several pairs keep more of the GPU busy, at the price of fp32 parts written and read once more. The estimate: a pair
// takes kBlockUs for a K block of 256 rows and kFixedUs for everything else; the parts move at 3 TB/s and cost another
// launch. 2048 rows of 14336 x 4096 stay as they are (64 blocks), 400 rows of 8992 x 2900 (12 blocks of 141 K blocks) go in parts. (Most
// sizes that want parts are the few-rows kernel's by bt_gemm_tiles' rule.)
// Where every pair has 256 rows the MMAs of a K block take 512 cycles and its expansion, one warp's chain of waits, loads,
// arithmetic and stores, 700, so two groups of warps expand K blocks in turn: 40 rows of 4096x14336, gate/up and down, 133 -> 118
// us, 512 rows 202 -> 191. With 512 rows to a pair the MMAs take 1024, one group keeps up, and a second one only
// gets in the way of the MMAs' operands (2048 rows 562 -> 665).
bool two_groups(const GemmParams &p) { return p.half || p.M <= 256; }
constexpr float kBlockUs = 0.42f, kFixedUs = 5.f, kReduceUs = 3.f, kPartBytesPerUs = 3e6f;
int deal_blocks(GemmParams &p, int slots, size_t part_bytes, float *expected_us) {
  const int runs = (p.TC + kPanel - 1) / kPanel, columns = p.pair ? runs : (runs + 1) / 2, KB = (p.KT + 1) / 2, tile_rows = (p.M + 31) / 32;
  p.row_blocks = (p.M + 511) / 512, p.half = 0, p.splits = 1;
  const int blocks = p.row_blocks * columns;
  p.whole = blocks;
  if (blocks >= slots) {
    const int last = blocks % slots;
    if (last > 0 && 2 * last <= slots && p.M > 256) p.whole = blocks - last;
    *expected_us = (p.whole < blocks ? blocks / slots + 0.5f : (float)((blocks + slots - 1) / slots)) * (kFixedUs + KB * kBlockUs * (p.M > 256 ? 2 : 1));
    return p.whole + 2 * (blocks - p.whole);
  }
  float best = 1e30f;
  int pairs = blocks;
  const float plane = (float)tile_rows * 32 * p.TC * 32 * 4 * (p.pair ? 2 : 1);
  for (int half = 0; half <= (p.M > 256 ? 1 : 0); half++) {
    const int rows = half ? (p.M + 255) / 256 : p.row_blocks, b = rows * columns, height = half || p.M <= 256 ? 1 : 2;
    for (int splits = 1; splits == 1 || (b * splits <= slots && splits <= KB && splits * (double)plane <= part_bytes); splits++) {
      const int waves = (b * splits + slots - 1) / slots;
      const float us = waves * (kFixedUs + (KB + splits - 1) / splits * kBlockUs * height) + (splits > 1 ? kReduceUs + 2 * splits * plane / kPartBytesPerUs : 0.f);
      if (us < best) best = us, pairs = b * splits, p.half = half, p.splits = splits, p.row_blocks = rows, p.whole = b;
    }
  }
  *expected_us = best;
  return pairs;
}

// Argument checks of both entry points.
int check(const char *who, int fmt, int epilogue, int M, int K, int N, uint64_t a, uint64_t w, uint64_t w2, uint64_t add, int add_rows, uint64_t out, int out_dtype, uint64_t work) {
  BT_REQUIRE(fmt == BT_BFP8 || fmt == BT_BFP4, "%s: weights must be bfp8 (8) or bfp4 (4), not %d", who, fmt);
  BT_REQUIRE(epilogue >= BT_EPI_NONE && epilogue <= BT_EPI_GLU, "%s: the epilogue is none, relu, silu or glu, not %d", who, epilogue);
  BT_REQUIRE(M >= 1 && K > 0 && N > 0 && K % 32 == 0, "%s: needs M >= 1, N >= 1 and K a positive multiple of 32: %d x %d x %d", who, M, K, N);
  BT_REQUIRE(a && w && out && work && a % 16 == 0 && w % 16 == 0 && out % 16 == 0, "%s: needs 16-byte aligned device addresses", who);
  BT_REQUIRE((epilogue == BT_EPI_GLU) == (w2 != 0) && w2 % 16 == 0, "%s: w2 goes with the GLU epilogue, and only with it", who);
  BT_REQUIRE(add % 16 == 0 && (!add || add_rows == 1 || add_rows == M), "%s: the addend is 16-byte aligned and has 1 or M rows, not %d", who, add_rows);
  BT_REQUIRE(out_dtype == BT_BF16 || out_dtype == BT_FP32, "%s: results are bf16 or fp32", who);
  return BT_OK;
}
// Their launches.
int gemm(const char *who, int device, int fmt, int epilogue, int M, int K, int N, uint64_t a, uint64_t w, uint64_t w2, uint64_t add, int add_rows, float alpha,
         uint64_t out, int out_dtype, uint64_t part, size_t part_bytes, bool weights_early, uint64_t work, uint64_t stream) {
  const bool pair = epilogue == BT_EPI_GLU;
  if (int s = check(who, fmt, epilogue, M, K, N, a, w, w2, add, add_rows, out, out_dtype, work)) return s;
  if (int s = use_device(device)) return s;
  alignas(64) CUtensorMap amap;
  const uint64_t dims[2] = {(uint64_t)K, (uint64_t)M}, strides[1] = {(uint64_t)K * 2};
  const uint32_t box[2] = {kBK, 128};
  if (int s = make_tmap(&amap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, as_ptr<void>(a), dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B)) return s;
  GemmParams p{};
  p.w[0] = as_ptr<uint8_t>(w), p.w[1] = as_ptr<uint8_t>(w2), p.add = as_ptr<uint16_t>(add), p.out = as_ptr<void>(out), p.error = as_ptr<int>(work);
  p.alpha = alpha, p.M = M, p.KT = K / 32, p.TC = (N + 31) / 32, p.epi = epilogue, p.out_fp32 = out_dtype == BT_FP32, p.pair = pair;
  p.add_row_stride = add && add_rows > 1 ? (size_t)p.TC * 1024 : 0;
  p.part = as_ptr<float>(part), p.weights_early = weights_early;
  int sms = 0;
  BT_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  float expected_us;
  const int pairs = deal_blocks(p, sms / 2 > 0 ? sms / 2 : 1, part_bytes, &expected_us);
  using Kernel = void (*)(GemmParams, CUtensorMap);
  static const Kernel kernels[2][2][2] = {{{gemm_kernel<BT_BFP8, false, 1>, gemm_kernel<BT_BFP8, false, 2>}, {gemm_kernel<BT_BFP8, true, 1>, gemm_kernel<BT_BFP8, true, 2>}},
                                          {{gemm_kernel<BT_BFP4, false, 1>, gemm_kernel<BT_BFP4, false, 2>}, {gemm_kernel<BT_BFP4, true, 1>, gemm_kernel<BT_BFP4, true, 2>}}};
  static const int bytes[2] = {Layout<BT_BFP8>::BYTES + 1024, Layout<BT_BFP4>::BYTES + 1024};
  static bool configured[64] = {};
  if (!configured[device & 63]) {
    for (int f = 0; f < 2; f++)
      for (int k = 0; k < 4; k++) BT_CUDA(cudaFuncSetAttribute(kernels[f][k / 2][k % 2], cudaFuncAttributeMaxDynamicSharedMemorySize, bytes[f]));
    configured[device & 63] = true;
  }
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3(2 * pairs);
  const int groups = two_groups(p) ? 2 : 1;
  cfg.blockDim = dim3(threads_of(groups));
  cfg.dynamicSmemBytes = bytes[fmt == BT_BFP4];
  cfg.stream = as_stream(stream);
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr, cfg.numAttrs = 2;
  BT_CUDA(cudaLaunchKernelEx(&cfg, kernels[fmt == BT_BFP4][p.splits > 1][groups - 1], p, amap));
  if (int s = launched("gemm_kernel")) return s;
  if (p.splits == 1) return BT_OK;
  // its blocks come up while the last of gemm_kernel drain, and wait there until that is complete
  cudaLaunchConfig_t add_up{};
  add_up.gridDim = dim3((unsigned)(((size_t)(M + 31) / 32 * 32 * p.TC * 8 + 255) / 256)), add_up.blockDim = dim3(256), add_up.stream = as_stream(stream);
  add_up.attrs = attr + 1, add_up.numAttrs = 1;
  BT_CUDA(cudaLaunchKernelEx(&add_up, reduce_kernel, p));
  return launched("reduce_kernel");
}

// What this kernel is expected to take for x in tiles, laid out by rows first (2.5 us, and x read and written at 5 TB/s).
int expected(int device, int epilogue, int M, int K, int N, size_t part_bytes, float *us) {
  int sms = 0;
  BT_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  GemmParams p{};
  p.M = M, p.KT = K / 32, p.TC = (N + 31) / 32, p.pair = epilogue == BT_EPI_GLU;
  deal_blocks(p, sms / 2 > 0 ? sms / 2 : 1, part_bytes, us);
  if (M <= 256) *us *= 1.1f;                      // one half of 256 rows at a time: a tenth slower than the estimate has it (128 rows of 4096 x 14336 120 us, not 108)
  *us += 2.5f + 4.f * M * K / 5e6f;
  return BT_OK;
}

}  // namespace

extern "C" {

int bt_gemm_bfp(int device, int fmt, int epilogue, int M, int K, int N, uint64_t a, uint64_t w, uint64_t w2, uint64_t add, int add_rows,
                float alpha, uint64_t out, int out_dtype, uint64_t work, uint64_t stream) {
  return gemm("bt_gemm_bfp", device, fmt, epilogue, M, K, N, a, w, w2, add, add_rows, alpha, out, out_dtype, 0, 0, false, work, stream);
}

int bt_gemm_tiles(int device, int fmt, int epilogue, int M, int K, int N, uint64_t x, uint64_t w, uint64_t w2, uint64_t add, int add_rows,
                  float alpha, uint64_t out, int out_dtype, uint64_t scratch, size_t scratch_bytes, uint64_t work, uint64_t stream) {
  BT_REQUIRE(M >= 1 && K > 0 && K % 32 == 0, "bt_gemm_tiles: needs M >= 1 and K a positive multiple of 32: %d x %d", M, K);
  const size_t rows = ((size_t)M * K * 2 + 255) / 256 * 256;
  BT_REQUIRE(x && x % 16 == 0 && scratch && scratch % 256 == 0 && scratch_bytes >= rows, "bt_gemm_tiles: needs x and at least %zu bytes of 256-byte aligned scratch, got %zu", rows, scratch_bytes);
  // The kernel of gemm_few.cu where its estimate is the lower one by 8 % (what the estimates are good for). Gate/up and down together, this kernel and that one: 128 rows of 4096 x 14336 120 and 55 us, 640
  // rows 287 and 228, 1024 rows 333 and 348, 2048 rows 569 and 695; 1024 rows of 2048 x 5632 104 and 89, 1400 rows 127 and 135; 2048 rows of
  // 1024 x 3000 78 and 63. Blocks of 128 x 128 waste less of a last wave and need no parts of K in memory; blocks of 512 x 256 expand a weight a fourth as often.
  if (M > 32) {
    if (int s = check("bt_gemm_tiles", fmt, epilogue, M, K, N, x, w, w2, add, add_rows, out, out_dtype, work)) return s;
    if (int s = use_device(device)) return s;
    float us;
    bool taken;
    if (int s = expected(device, epilogue, M, K, N, scratch_bytes - rows, &us)) return s;
    if (int s = gemm_few(device, fmt, epilogue, M, K, N, x, w, w2, add, add_rows, alpha, out, out_dtype, 0.92f * us, &taken, work, stream)) return s;
    if (taken) return BT_OK;
  }
  if (int s = bt_untilize(device, 2, x, scratch, 1, M, K, stream)) return s;
  return gemm("bt_gemm_tiles", device, fmt, epilogue, M, K, N, scratch, w, w2, add, add_rows, alpha, out, out_dtype, scratch + rows, scratch_bytes - rows, true, work, stream);
}

}  // extern "C"
