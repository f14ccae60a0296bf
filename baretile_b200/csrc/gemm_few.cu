// Prefill matmul for prompts of up to some hundred rows (and longer ones on few columns; see bt_gemm_tiles): out = epilogue(alpha * x @ W + add),
// W block-float in streaming layout, x in tiles as Tensor holds it.
//
// With few rows every weight is used a few dozen times and the work is bound by the stream of packed weights: by
// HBM (an SM's share of it is a tile in 43 cycles in bfp8, 23 in bfp4), by their expansion (25 cycles a tile) and by what a launch
// costs. MMAs with the rows of x as their M would be mostly padding, and expanded weights as a B operand would cross shared memory
// twice (2 KB a tile each way, of 128 bytes a cycle). So the operands change places: the 128 output channels of a sub-panel are the MMA's M,
// the tokens its N (only as many as there are, in sixteens, up to 128), and the expanded weights go from registers to TENSOR MEMORY, from
// where tcgen05.mma takes its A operand; a lane's registers are 16x256b store fragments as they come.
//
// A CTA has a sub-panel of 4 tile columns (of both matrices of a gate/up pair) and a block of up to 128 rows; where these are fewer than SMs a
// cluster of up to 8 CTAs shares one, each with a part of K. At the end the CTAs' fp32 sums are added through distributed shared memory,
// in order, and each CTA of the cluster runs the epilogue for its share of the rows: one launch, no scratch, x not laid out anew.
//
// Per stage of up to 4 tile rows (K = 128):
//   warps 0-15   expand packed tiles into tensor memory, two groups of eight that take the stages in turn (as one group all warps computed at
//                the same time and waited at the same time: 33 rows of 4096 x 14336 52 us against 46); then the epilogue
//   warp 16      copies the packed tiles (a bulk copy per matrix)
//   warp 17      issues the MMAs (128 channels x tokens x 16 each); a commit frees x and the tensor memory of the stage
//   warps 18-21  copy x, a tile row each: 16 tokens x 16 k of a tile are 512 consecutive bytes, a warp's one cp.async, which lands
//                in the 32-byte swizzle, and tells the stage's barrier itself when it has (warps that waited for their copies: 128 rows 58 us against 55)
// Gate/up pair and down projection, against the kernel of gemm.cu with its x laid out by rows and its parts of K added up by another launch:
// 77 rows of 2048 x 5632 (bfp4, bfp8) 43.7 -> 22.1 us, 33 rows of 512 x 1024 23.8 -> 10.6, 33 rows of 4096 x 14336 113 -> 44, 128 rows 120 -> 55,
// 256 rows 124 -> 110, 640 rows 287 -> 228; 512 rows of 1024 x 3000 37.9 -> 24.7.
// A launch costs 5 to 10 us beside its stages: setting up and the first weights and x 3, the sums' way through the cluster and the epilogue 3.
// Every wait on an mbarrier is bounded and reports through the error word; the first that gives up ends the waiting of its CTA. The cluster's two barriers,
// which every CTA reaches that way, have no limit of their own.
#include "common.cuh"
#include "expand.cuh"
#include <algorithm>

namespace bt {
namespace {

constexpr int kRows = 4;                            // tile rows of a stage
constexpr int kExpandWarps = 16, kWeightWarp = 16, kMmaWarp = 17, kXWarp = 18, kXWarps = kRows;
// Groups of warps that take the stages in turn. An mbarrier's parity tells a phase only from its neighbours, so whoever waits for one has to know that the
// phase before is over. A place of the weights' ring therefore belongs to one group: the ring has a multiple of kGroups places. (With three, a group came to a
// place where the other group's weights had not landed yet, and took the phase before that for its own: garbage, and in the end a launch
// failure.) A buffer in tensor memory may go from group to group, up to 4 of them: its phases end in order, and a group has waited for one of the stages
// before.
constexpr int kGroups = 2, kGroupWarps = kExpandWarps / kGroups;
constexpr int kThreads = (kXWarp + kXWarps) * 32;
constexpr int kMaxStages = 8, kMaxBufs = 4, kMaxSplits = 8;
static_assert(kMaxStages % kGroups == 0, "places of the ring belong to groups");
constexpr uint32_t kLimit = 1u << 14;               // attempts of up to 100 us each

// Shared memory: mbarriers, then the rings of packed weights and of x, over which the sums go in the end.
constexpr int kWFull = 0, kWEmpty = 64, kXFull = 128, kXEmpty = 192, kReady = 256, kFree = 288, kDone = 320, kTmem = 328, kDead = 332, kRing = 1024;
constexpr int kSmem = 227 * 1024;
constexpr int kBlockRows = 4;                       // tile rows of a CTA at most: the sums of 128 tokens of a pair and the expanded weights fill tensor memory
constexpr int kSumStride = 132;                     // floats from one token's 128 channels to the next

struct FewParams {
  const uint8_t *w[2];
  const uint8_t *x;
  const uint16_t *add;
  size_t add_row_stride;     // datums from one tile row of the addend to the next; 0 when the addend is one row
  void *out;
  int *error;
  float alpha;
  int M, KT, TC, epi, out_fp32;
  int splits;                // CTAs of a cluster, which share a sub-panel
  int stages, x_stages, bufs;   // of the rings of packed weights and of x, and of expanded weights in tensor memory
  int blocks, block_rows;    // blocks of rows, and tile rows of each but the last
  int tokens;                // rows of a block in sixteens: the MMAs' N
  int weights_early;         // the launch before this one does not write weights
};

// Shared-memory descriptor of x: K-major rows of 32 bytes, 32-byte swizzle, 8-row groups 256 bytes apart.
__device__ __forceinline__ uint64_t x_desc(uint32_t addr) { return (uint64_t)((addr & 0x3FFFF) >> 4) | ((uint64_t)(256 >> 4) << 32) | (1ull << 46) | (6ull << 61); }

template <int FMT, bool PAIR>
__global__ void __launch_bounds__(kThreads, 1) few_rows_kernel(const __grid_constant__ FewParams p) {
  constexpr int TB = tile_bytes(FMT), MATS = PAIR ? 2 : 1, W_STAGE = MATS * kRows * kPanel * TB, BUF = MATS * kRows * 16;   // BUF: tensor-memory columns of a stage's weights
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t sb = smem_u32(smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = p.splits > 1 ? (int)cluster_ctarank() : 0, panel = blockIdx.x / (p.splits * p.blocks);
  const int tr0 = blockIdx.x / p.splits % p.blocks * p.block_rows, M = min(p.M - tr0 * 32, p.block_rows * 32);   // first tile row, and rows
  const int k0 = p.KT * rank / p.splits, kn = p.KT * (rank + 1) / p.splits - k0, steps = (kn + kRows - 1) / kRows;   // this CTA's tile rows
  const int width = min(kPanel, p.TC - panel * kPanel), N = (M + 15) / 16 * 16, stages = p.stages, x_stages = p.x_stages, bufs = p.bufs;
  const int x_row = N * 64, x_stage = kRows * p.tokens * 64;
  const uint32_t x_ring = sb + kRing + stages * W_STAGE;
  // A wait that gives up marks the CTA: from there on its sums are worthless, and every wait takes one attempt, so that the CTA ends in some
  // milliseconds (with a full limit to each of up to 112 stages it held the GPU for minutes).
  auto wait = [&](uint32_t bar, uint32_t parity, int code) {
    bool ok = mbar_try_wait(bar, parity, 100000u);
    for (uint32_t i = 1; !ok && i < kLimit && !lds32(sb + kDead); i++) ok = mbar_try_wait(bar, parity, 100000u);
    if (!ok) sts32(sb + kDead, 1), atomicExch(p.error, code);
    __syncwarp();                                   // whole warps wait, and the tensor-memory instructions that follow want them in step
    return ok;
  };
  if (warp == 0) {                                  // a lane to a place of the rings
    if (lane < kMaxStages) {
      mbar_init(sb + kWFull + 8 * lane, 1), mbar_init(sb + kWEmpty + 8 * lane, kGroupWarps);
      mbar_init(sb + kXFull + 8 * lane, kXWarps * 32), mbar_init(sb + kXEmpty + 8 * lane, 1);
    }
    if (lane < kMaxBufs) mbar_init(sb + kReady + 8 * lane, kGroupWarps), mbar_init(sb + kFree + 8 * lane, 1);
    if (lane == 0) mbar_init(sb + kDone, 1), sts32(sb + kDead, 0);
    mbar_fence_init();
  }
  if (warp == kMmaWarp) tmem_alloc(sb + kTmem, 512);
  tc_fence_before();
  __syncthreads();                                  // the barriers are set up, and the allocation's answer is there for everyone, the warp that asked included
  tc_fence_after();
  // All of that, and the first weights where the launch before writes none, may happen while that launch drains. x, the addend and
  // the result wait.
  auto in_turn = [] { asm volatile("griddepcontrol.wait;" ::: "memory"); };
  if (!p.weights_early) in_turn();
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(smem + kTmem), weights0 = tmem + 512 - bufs * BUF;

  // Every role is one warp's chain of dependent instructions, about 5 cycles each, so what is worked out per stage counts: places in
  // the ring go round by themselves (divisions by a number of stages known only at run time took 400 cycles of 2400 a stage).
  struct Turn {                                      // of a ring of n: the place, and the parity of its round
    int at = 0;
    uint32_t parity = 0;
    __device__ __forceinline__ void next(int n) {
      if (++at == n) at = 0, parity ^= 1;
    }
  };
  if (warp == kWeightWarp) {
    const uint8_t *from = p.w[lane < MATS ? lane : 0] + ((size_t)panel * kPanel * p.KT + (size_t)k0 * width) * TB;
    const uint32_t stage = kRows * width * TB;
    Turn t;
    for (int i = 0; i < steps; i++, t.next(stages), from += stage) {
      if (i >= stages && !__all_sync(0xFFFFFFFFu, wait(sb + kWEmpty + 8 * t.at, t.parity ^ 1, 21))) break;
      const uint32_t bytes = min(kRows, kn - i * kRows) * width * TB, bar = sb + kWFull + 8 * t.at;
      if (lane == 0) mbar_expect_tx(bar, MATS * bytes);
      __syncwarp();
      if (lane < MATS) bulk_g2s(sb + kRing + t.at * W_STAGE + lane * (kRows * kPanel * TB), from, bytes, bar);
    }
    if (lds32(sb + kDead))                           // nobody may be waiting for the copies in flight any more; they land before the CTA ends
      for (int i = 0; i < stages; i++, t.next(stages)) mbar_wait(sb + kWFull + 8 * t.at, t.parity ^ 1, 100);
  } else if (warp == kMmaWarp) {
    {
      const uint32_t leader = elect_one();
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
      const uint64_t x0 = x_desc(x_ring);
      const uint32_t row = x_row >> 4, half = N * 2, stage = x_stage >> 4;   // descriptors count 16 bytes
      auto mmas = [&](uint64_t x, uint32_t a, int r, uint32_t more) {
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
          for (int m = 0; m < MATS; m++) umma_bf16_ts(tmem + m * N, a + m * (kRows * 16) + r * 16 + h * 8, x + h * half, idesc, h ? 1u : more, leader);
      };
      Turn t, u;
      for (int i = 0; i < steps; i++, t.next(x_stages), u.next(bufs)) {
        const int n = min(kRows, kn - i * kRows);
        wait(sb + kXFull + 8 * t.at, t.parity, 22);
        wait(sb + kReady + 8 * u.at, u.parity, 23);
        fence_async_shared();                        // x came with copies of the generic proxy
        tc_fence_after();
        const uint64_t x = x0 + t.at * stage;
        const uint32_t a = weights0 + u.at * BUF;
        mmas(x, a, 0, i != 0);
        if (n == kRows) {
#pragma unroll
          for (int r = 1; r < kRows; r++) mmas(x + r * row, a, r, 1u);
        } else
          for (int r = 1; r < n; r++) mmas(x + r * row, a, r, 1u);
        umma_commit_if(sb + kXEmpty + 8 * t.at, leader);
        umma_commit_if(sb + kFree + 8 * u.at, leader);
      }
      umma_commit_if(sb + kDone, leader);
      wait(sb + kDone, 0, 28);                       // tensor memory is given back by this warp
    }
  } else if (warp >= kXWarp) {
    in_turn();
    const int me = warp - kXWarp;
    const uint32_t place = (lane >> 1) * 32 + (((lane & 1) ^ (lane >> 3 & 1)) << 4);
    Turn t;
    // a warp copies its tile row of the stage, whose barrier hears from every lane when its copies have landed
    const uint8_t *from = p.x + ((size_t)tr0 * p.KT + k0 + me) * 2048 + lane * 16;
    for (int i = 0; i < steps; i++, t.next(x_stages), from += kRows * 2048) {
      if (i >= x_stages) wait(sb + kXEmpty + 8 * t.at, t.parity ^ 1, 24);
      if (me < kn - i * kRows) {
        uint32_t to = x_ring + t.at * x_stage + place + me * x_row;
        const uint8_t *src = from;
        for (int tb = 0; tb < N / 16; tb += 2, to += 1024, src += (size_t)p.KT * 2048) {
          cp_async16(to, src), cp_async16(to + N * 32, src + 512);
          if (tb + 1 < N / 16) cp_async16(to + 512, src + 1024), cp_async16(to + N * 32 + 512, src + 1536);
        }
      }
      cp_async_arrive(sb + kXFull + 8 * t.at);
    }
    cp_async_wait_all();
  } else {
    const int cc = warp & 3, group = warp / kGroupWarps, row = warp % kGroupWarps >> 2;
    const uint32_t lanes = (uint32_t)(32 * cc) << 16, tile0 = sb + kRing + (row * width + cc) * TB, a0 = weights0 + lanes + row * 16;
    Turn t, u;
    for (int i = 0; i < group; i++) t.next(stages), u.next(bufs);
    for (int i = group; i < steps; i += kGroups) {
      wait(sb + kWFull + 8 * t.at, t.parity, 25);
      if (i >= bufs) wait(sb + kFree + 8 * u.at, u.parity ^ 1, 26);
      tc_fence_after();
      {
#pragma unroll
        for (int r = 0; r < kRows; r += kGroupWarps / 4)
#pragma unroll
          for (int m = 0; m < MATS; m++) {           // (rows past a last stage: what lies there, which no MMA takes)
            uint32_t a[2][2][4] = {};                // of a column that the matrix does not have: zeros
            if (cc < width) expand_weights<FMT>(packed_lane<FMT>(tile0 + t.at * W_STAGE + m * (kRows * kPanel * TB) + r * width * TB, lane), a);
            // a lane's two pairs of k are two neighbouring 32-bit columns of rows g and g + 8
#pragma unroll
            for (int fs = 0; fs < 2; fs++) {
              const uint32_t v[8] = {a[0][fs][0], a[0][fs][2], a[0][fs][1], a[0][fs][3], a[1][fs][0], a[1][fs][2], a[1][fs][1], a[1][fs][3]};
              tmem_st_16x256b(a0 + ((uint32_t)(16 * fs) << 16) + u.at * BUF + m * (kRows * 16) + r * 16, v);
            }
          }
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(sb + kWEmpty + 8 * t.at), mbar_arrive(sb + kReady + 8 * u.at);
      for (int g = 0; g < kGroups; g++) t.next(stages), u.next(bufs);
    }
    wait(sb + kDone, 0, 27);
    tc_fence_after();
    // the sums go over the ring: every stage has been used
    const int t0 = 32 * (warp >> 2), ch = 32 * cc + (lane & 16) + 2 * (lane & 7) + (lane >> 3 & 1);
    if (t0 < M) {
#pragma unroll
      for (int m = 0; m < MATS; m++) {
        float *to = reinterpret_cast<float *>(smem + kRing) + (m * M + t0) * kSumStride + ch;
#pragma unroll
        for (int c = 0; c < 32; c += 16)
          if (t0 + c < N) {
            uint32_t v[16];
            tmem_ld(tmem + lanes + m * N + t0 + c, v);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; j++)
              if (t0 + c + j < M) to[(c + j) * kSumStride] = __uint_as_float(v[j]);
          }
      }
    }
  }
  in_turn();
  __syncwarp();
  tc_fence_before();
  if (p.splits > 1) cluster_sync();
  else __syncthreads();
  tc_fence_after();
  if (warp == kMmaWarp) tmem_dealloc(tmem, 512);
  // a warp to a row of 128 channels, a lane to four of them
  const int tile_rows = (M + 31) / 32, first = tile_rows * 32 * rank / p.splits, end = tile_rows * 32 * (rank + 1) / p.splits;
  const int tcol = panel * kPanel + (lane >> 3), in_face = (lane & 4) * 64 + (lane & 3) * 4;   // datum of the lane's first channel in a tile's row 0
  if (lane >> 3 < width) {
    const float unscale = kExpandedUnscale * p.alpha;
    for (int row = first + warp; row < end; row += kThreads / 32) {
      float f[4] = {0.f, 0.f, 0.f, 0.f}, g[4] = {0.f, 0.f, 0.f, 0.f};
      const int tr = tr0 + (row >> 5), at = in_face + (row >> 4 & 1) * 512 + (row & 15) * 16;
      if (row < M) {
        uint2 a = make_uint2(0, 0);
        if (p.add) a = __ldcg(reinterpret_cast<const uint2 *>(p.add + (size_t)tr * p.add_row_stride + (size_t)tcol * 1024 + (p.add_row_stride ? at : in_face)));
        const float *own = reinterpret_cast<const float *>(smem + kRing) + row * kSumStride + lane * 4;
        for (int c = 0; c < p.splits; c += 4) {      // of up to four CTAs in flight together; the way between SMs is narrow, so not this one's own
          float4 v[4], u[4];
#pragma unroll
          for (int j = 0; j < 4; j++) {
            v[j] = u[j] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (c + j == rank) {
              v[j] = *reinterpret_cast<const float4 *>(own);
              if (PAIR) u[j] = *reinterpret_cast<const float4 *>(own + M * kSumStride);
            } else if (c + j < p.splits) {
              const uint32_t from = map_to_cta(smem_u32(own), c + j);
              v[j] = ld_cluster4(from);
              if (PAIR) u[j] = ld_cluster4(from + M * kSumStride * 4);
            }
          }
#pragma unroll
          for (int j = 0; j < 4; j++) {
            f[0] += v[j].x, f[1] += v[j].y, f[2] += v[j].z, f[3] += v[j].w;
            if (PAIR) g[0] += u[j].x, g[1] += u[j].y, g[2] += u[j].z, g[3] += u[j].w;
          }
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const uint32_t w = k < 2 ? a.x : a.y;
          float y = f[k] * unscale;
          if (p.add) y += __uint_as_float(k % 2 ? w & 0xFFFF0000u : w << 16);
          if (PAIR) y = silu(y) * (g[k] * unscale);
          else if (p.epi == BT_EPI_RELU) y = fmaxf(y, 0.f);
          else if (p.epi == BT_EPI_SILU) y = silu(y);
          f[k] = y;
        }
      }
      const size_t o = ((size_t)tr * p.TC + tcol) * 1024 + at;
      if (p.out_fp32) *reinterpret_cast<float4 *>(static_cast<float *>(p.out) + o) = make_float4(f[0], f[1], f[2], f[3]);
      else *reinterpret_cast<uint2 *>(static_cast<uint16_t *>(p.out) + o) = make_uint2(bf16_half_up(f[0]) | bf16_half_up(f[1]) << 16, bf16_half_up(f[2]) | bf16_half_up(f[3]) << 16);
    }
  }
  __syncwarp();
  if (p.splits > 1) cluster_sync();                // nobody leaves while others read its sums
}

constexpr float kStartUs = 2.f, kFixedUs = 4.f;     // a launch's start, a wave's start and end
float tile_us(int tokens) { return 0.02f + 0.0001f * tokens; }   // an SM's time for a packed tile: 0.024 with 48 tokens, 0.032 with 128

}  // namespace

int gemm_few(int device, int fmt, int epilogue, int M, int K, int N, uint64_t x, uint64_t w, uint64_t w2, uint64_t add, int add_rows, float alpha, uint64_t out,
             int out_dtype, float beat_us, bool *taken, uint64_t work, uint64_t stream) {
  const bool pair = epilogue == BT_EPI_GLU;
  FewParams p{};
  p.w[0] = as_ptr<uint8_t>(w), p.w[1] = as_ptr<uint8_t>(w2), p.x = as_ptr<uint8_t>(x), p.add = as_ptr<uint16_t>(add), p.out = as_ptr<void>(out), p.error = as_ptr<int>(work);
  p.alpha = alpha, p.M = M, p.KT = K / 32, p.TC = (N + 31) / 32, p.epi = epilogue, p.out_fp32 = out_dtype == BT_FP32;
  p.add_row_stride = add && add_rows > 1 ? (size_t)p.TC * 1024 : 0;
  const int tile_rows = (M + 31) / 32;
  p.blocks = (tile_rows + kBlockRows - 1) / kBlockRows, p.block_rows = (tile_rows + p.blocks - 1) / p.blocks;
  p.tokens = (std::min(M, p.block_rows * 32) + 15) / 16 * 16;
  const int mats = pair ? 2 : 1, w_stage = kRows * mats * kPanel * tile_bytes(fmt), x_stage = kRows * p.tokens * 64;
  // as many places for x as leave four for the weights (128 tokens and a pair in bfp8: two)
  for (p.x_stages = kMaxStages; p.x_stages > 2 && (kSmem - kRing - p.x_stages * x_stage) / w_stage < 4; p.x_stages--);
  p.stages = std::min(kMaxStages, (kSmem - kRing - p.x_stages * x_stage) / w_stage) / kGroups * kGroups;
  p.bufs = std::min(kMaxBufs, (512 - mats * p.tokens) / (mats * kRows * 16));

  using Kernel = void (*)(FewParams);
  static const Kernel kernels[2][2] = {{few_rows_kernel<BT_BFP8, false>, few_rows_kernel<BT_BFP8, true>}, {few_rows_kernel<BT_BFP4, false>, few_rows_kernel<BT_BFP4, true>}};
  const Kernel kernel = kernels[fmt == BT_BFP4][pair];
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.blockDim = dim3(kThreads), cfg.dynamicSmemBytes = kSmem, cfg.stream = as_stream(stream), cfg.attrs = attr;
  // how many clusters of each size fit on the GPU at once: all four kernels take the same room
  static int clusters[64][kMaxSplits + 1] = {};
  int *fit = clusters[device & 63];
  if (!fit[1]) {
    for (int k = 0; k < 4; k++) BT_CUDA(cudaFuncSetAttribute(kernels[k / 2][k % 2], cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
    for (int s = kMaxSplits; s >= 1; s--) {
      int n = 0;
      attr[1].val.clusterDim.x = s, cfg.gridDim = dim3(s), cfg.numAttrs = 2;
      BT_CUDA(cudaOccupancyMaxActiveClusters(&n, kernels[0][0], &cfg));
      fit[s] = std::max(n, 1);
    }
  }
  // The split with the least estimated time: waves of CTAs, each with its start and end and its tiles. As many CTAs as fit at once, in
  // short: 77 rows of 2048 x 5632 (44 sub-panels, pair) 16.9, 12.7, 12.5, 21 us in 1, 2, 3 and 4 parts, 5632 x 2048 (16)
  // 15.5, 10.4, 10.3, 16.3 in 2, 4, 6 and 8.
  const int panels = (p.TC + kPanel - 1) / kPanel;
  float best = 1e30f;
  int rounds = 1;
  for (int s = 1; s <= std::min(kMaxSplits, p.KT); s++) {
    const int waves = (panels * p.blocks + fit[s] - 1) / fit[s];
    const float us = kStartUs + waves * (kFixedUs + (p.KT + s - 1) / s * kPanel * mats * tile_us(p.tokens)) + (s > 1 ? 0.5f + 0.1f * s : 0.f);
    if (us < best) best = us, p.splits = s, rounds = waves;
  }
  // many waves of 128 x 128 draw more power than the estimate knows of: 2048 rows of 3000 x 8000 291 us where it had 250, the other kernel 278
  *taken = best < (rounds > 2 ? 0.87f : 1.f) * beat_us;
  if (!*taken) return BT_OK;
  p.weights_early = follows_matmul(stream);
  cfg.gridDim = dim3(panels * p.blocks * p.splits), attr[1].val.clusterDim.x = p.splits, cfg.numAttrs = p.splits > 1 ? 2 : 1;
  BT_CUDA(cudaLaunchKernelEx(&cfg, kernel, p));
  return launched("few_rows_kernel");
}

}  // namespace bt
