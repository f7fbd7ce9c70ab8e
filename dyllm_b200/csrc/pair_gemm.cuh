// bf16 GEMM on CTA pairs (tcgen05 cta_group::2) with the weights as the M operand:
//
//   D[n, m] = sum_k W[w_row0(tile) + n, k] * A[m, k]        (fp32 accumulation in tensor memory)
//
// i.e. the transpose of the usual arrangement: weight rows (output columns) fill the tensor cores' M dimension and
// activation rows are the N dimension, in steps of 32.  One kernel then serves every live row count, which only the
// device knows (m_count_dev): few rows make a narrow product whose time is that of streaming the weights, many rows
// make 256-row tiles at full tensor rate.  The launch is always one CTA per SM and needs no row-count estimate.
//
// A tile is (up to 256 rows) x (nb blocks of 128 output columns per CTA, so nb * 256 per pair).  Per k step of 64 a CTA
// loads its own nb * 128 weight rows and half of the tile's activation rows; the pair's product reads both halves.  At
// 256 rows and nb = 2 that is 48 KB per SM for 1024 tensor-core clocks (47 B/clk); the 256 x 256 tile of a single CTA
// needs 64 KB (62 B/clk), more than the ~52 B/clk an SM gets from L2.
//
// Work split: tiles are dealt to the pairs in turn (groups of eight row tiles, so that the tiles in flight share weights
// and activations in L2).  Few rows of a plain product cut the k range into up to four parts: fp32 partial sums go to the
// workspace and the CTA that finishes a tile last adds them in k order (the same sum whoever is last).  The number of
// parts is that of gemm.cuh for the launch's row estimate (set_cut() in ffn.cu) and the live count, whatever the tile shape
// here, so both kernels give the same bits.  (Equal shares
// per pair over all sizes, so that the last wave is always full, were measured too: 280 us against 289 us for a 3277 x
// 4096 x 12288 product, nothing at few rows, and other sums.)
//
// Warp roles (12 warps per CTA):
//   warps 0, 2  producers: weight and activation boxes by TMA (128-byte swizzle), completion counted by the barrier of
//               the pair's first CTA
//   warp 1      tensor memory; in the first CTA: issues the pair's tcgen05.mma, commits to both CTAs' barriers
//   warps 4-11  epilogue: thread = output column, registers = rows; SiLU(gate) * up, bias, row scale, row scatter,
//               column split, or fp32 partial sums.  Neighbouring lanes swap values so that a thread stores two
//               adjacent columns of one row.
// Measured on one B200 (us, against the kernel of gemm.cuh under the fixed estimate of 128 rows that a captured step
// gives; gate/up and down product of a 4096 x 12288 FFN, K/V projection 4096 x 8192):
//   rows      46           100          200          400          800          1500
//   gate/up   41 -> 42     43 -> 48     72 -> 52     115 -> 96    192 -> 145   355 -> 209
//   down      31 -> 30     35 -> 34     55 -> 47     94 -> 73     174 -> 109   254 -> 136
//   K/V       23 -> 23     25 -> 26     35 -> 31     65 -> 43     114 -> 56    177 -> 111
// Library products of the same size: 91 against 107 us at 4096 rows, 182 against 224 at 8192 (4096 x 4096).  At 46 rows the
// weights alone take 31, 15 and 10 us at the HBM rate (6.5 TB/s), so every product spends another 11 to 15 us beside the
// stream (start of the ring, whose round trip spans two CTAs; partial sums; epilogue): gate/up runs at 4.8 TB/s, down at 3.4,
// K/V at 2.9.  Many rows are bound by the power limit (1.3 PFLOP/s at 3277 rows, as the library's products).
// Every wait is bounded; a wait that runs out raises the CTA's abort flag and the device status word.
#pragma once

#include <cooperative_groups.h>

#include "gemm.cuh"   // effective_splits(), open_counter(), last_to_arrive()

namespace dyllm {

struct PairGemmParams;
int launch_pair_gemm(bool swiglu, const PairGemmParams& p, const void* a, int a_rows, int64_t lda, const void* w,
                     int64_t w_total_rows, cudaStream_t stream);

struct PairGemmParams {
  const int32_t* m_count_dev;   // device scalar bounding the live rows; null = M
  int M;                        // upper bound of rows
  const int4* row_tiles;        // grouped product: {first row, rows (<= 256), weight block, 0} per row tile; null = dense rows
  const int32_t* tiles_dev;     // grouped product: [0] number of row tiles, [1] rows of the tallest one
  int K;                        // contraction length, multiple of 64
  int n;                        // output columns per weight block
  int w_rows_per_block;         // weight rows per weight block
  int up_row_offset;            // SwiGLU: row distance from the gate rows to the up rows
  __nv_bfloat16* out;
  int64_t ldc;
  __nv_bfloat16* out2;          // columns >= split_col go here (column - split_col); null = no split
  int64_t ldc2;
  int split_col;                // multiple of 128
  const int32_t* out_row_map;   // destination row per row (negative = drop); null = identity
  const float* row_scale;       // multiplier per row; null = 1
  const __nv_bfloat16* bias;    // [n], at any element; null = none
  int bias_fp32;                // 1: added to the fp32 sum, one rounding; 0: to the rounded result (bf16 + bf16)
  float* partial;               // partial sums [parts][kSplitRows][n] of a cut k range; null = never cut
  unsigned long long* tickets;  // arrival counters of cut tiles, two per tile (one per CTA of a pair)
  unsigned long long launch_id;
  int max_parts;                // parts of a cut k range: effective_splits() of these three and the live count
  int cut_col_tiles;
  int cut_slots;
  int one_tile_pairs;           // pairs that work when all rows fit one row tile (0 = all)
  int* status_word;
};

constexpr int kPgMaxPairs = 96;                  // pairs a launch uses at most (192 SMs)
constexpr int kSplitRows = 512;                  // partial sums are kept for at most this many live rows
constexpr int kMaxSplits = 4;
constexpr int kPgThreads = 384;
constexpr int kPgMaxRows = 256;                  // rows per tile (UMMA N)
constexpr int kPgMaxStages = 10;
constexpr uint32_t kPgWBytes = 128 * 64 * 2;     // one weight box
constexpr uint32_t kPgABytes = 32 * 64 * 2;      // one activation box
constexpr uint32_t kPgSwapBytes = 2 * 32 * 64 * 4;   // narrow SwiGLU tiles: up values on their way to the gate threads
constexpr uint32_t kPgRing = 216 * 1024;
constexpr uint32_t kPgSmem = kPgRing + 1024;
constexpr int kPgRowGroup = 8;                   // row tiles that share the weight tiles in flight

// How a launch's tiles are shared out; the same arithmetic in every thread of the grid.
struct PgSched {
  bool narrow;        // SwiGLU with 64 gate and 64 up rows in the CTA's one weight block (128 columns per pair)
  int kt, nb, tile_n, row_tiles, col_tiles, parts, part_kt, units, pairs, pair, m;
};

struct PgSeg {
  int tile, part, k0, k1;
};

// Rows spread evenly over row tiles of at most kPgMaxRows, in steps of 32.
__host__ __device__ __forceinline__ void pg_row_tiles(int m, int at_least, int& tile_n, int& row_tiles) {
  tile_n = ((m + at_least - 1) / at_least + 31) & ~31;
  row_tiles = (m + tile_n - 1) / tile_n;
}
// More and lower row tiles (the weights come from L2 the second time) give more pairs work.
__host__ __device__ __forceinline__ void pg_lower_tiles(int m, int col_tiles, int parts, int pairs, int& tile_n,
                                                        int& row_tiles) {
  while (tile_n > 64 && 2 * row_tiles * col_tiles * parts <= pairs)
    pg_row_tiles(m, 2 * row_tiles, tile_n, row_tiles);
}
// One or two weight blocks per CTA: two need fewer operand bytes per flop, one gives twice the tiles to fill the waves
// with.  A wave of one-block tiles takes 2/3 to 3/4 of the time of a wave of two-block tiles at 256 rows (62 B/clk of
// operands against 47), and half at few rows.  (K = 12288, 4096 columns: 5000 rows 600 us in five waves of one block, 450 us
// in three of two; 3277 rows three against two waves, which is even.)
__host__ __device__ __forceinline__ int pg_blocks(int row_tiles, int n, int parts, int pairs, int& waves) {
  const int w1 = (row_tiles * ((n + 255) >> 8) * parts + pairs - 1) / pairs;
  const int w2 = (row_tiles * ((n + 511) >> 9) * parts + pairs - 1) / pairs;
  const int nb = w1 * 2 <= w2 * 3 ? 1 : 2;
  waves = nb == 1 ? w1 : w2;
  return nb;
}

__device__ __forceinline__ bool pg_schedule(const PairGemmParams& p, bool swiglu, PgSched& s) {
  s.pairs = gridDim.x >> 1;
  s.pair = blockIdx.x >> 1;
  s.kt = p.K >> 6;
  if (p.row_tiles) {
    s.m = 0;
    s.row_tiles = p.tiles_dev[0];
    s.tile_n = (min(p.tiles_dev[1], kPgMaxRows) + 31) & ~31;
  } else {
    s.m = p.m_count_dev ? min(*p.m_count_dev, p.M) : p.M;
    if (s.m <= 0)
      return false;
    pg_row_tiles(s.m, (s.m + kPgMaxRows - 1) / kPgMaxRows, s.tile_n, s.row_tiles);
  }
  if (s.row_tiles <= 0)
    return false;
  if (!p.row_tiles && s.row_tiles == 1 && p.one_tile_pairs > 0 && p.one_tile_pairs < s.pairs)
    s.pairs = p.one_tile_pairs;
  // Few tiles leave most pairs without work.  SwiGLU tiles of half the width give twice as many (8 experts of 1024 columns
  // with 60 rows each: 32 tiles for 74 pairs).
  s.narrow = swiglu && 2 * s.row_tiles * ((p.n + 255) >> 8) <= s.pairs;
  const int pair_cols = s.narrow ? 128 : 256;
  s.parts = 1;
  if (!swiglu && !p.row_tiles && p.partial && p.max_parts > 1 && s.m <= kSplitRows)
    s.parts = effective_splits((s.m + kGemmBM - 1) / kGemmBM, p.cut_col_tiles, p.cut_slots, p.max_parts, s.kt);
  s.part_kt = (s.kt + s.parts - 1) / s.parts;
  if (!p.row_tiles)
    pg_lower_tiles(s.m, (p.n + pair_cols - 1) / pair_cols, s.parts, s.pairs, s.tile_n, s.row_tiles);
  int waves;
  // grouped tiles up to 128 rows high: one block; higher ones by the waves, too (8 experts of 200 rows each, 2048 columns: 32
  // tiles of two blocks leave more than half of the pairs idle)
  s.nb = swiglu ? (s.narrow ? 1 : 2)
                : p.row_tiles && s.tile_n <= 128 ? 1 : pg_blocks(s.row_tiles, p.n, s.parts, s.pairs, waves);
  const int cols = swiglu ? pair_cols : s.nb * 256;
  s.col_tiles = (p.n + cols - 1) / cols;
  s.units = s.row_tiles * s.col_tiles * s.parts;
  return true;
}

// Piece of work number `u` (pairs take u = pair, pair + pairs, ...); false past the last one.
__device__ __forceinline__ bool pg_unit(const PgSched& s, int u, PgSeg& g) {
  if (u >= s.units)
    return false;
  g.tile = u / s.parts;
  g.part = u - g.tile * s.parts;
  g.k0 = min(g.part * s.part_kt, s.kt);
  g.k1 = min(g.k0 + s.part_kt, s.kt);
  return true;
}

struct PgTile {
  int row0, rows, block, col_tile, n;   // n: UMMA N, rows rounded up to 32
};

__device__ __forceinline__ PgTile pg_tile(const PairGemmParams& p, const PgSched& s, int tile) {
  PgTile t;
  const int per_group = kPgRowGroup * s.col_tiles;
  const int g = tile / per_group, rem = tile - g * per_group;
  const int gr = min(kPgRowGroup, s.row_tiles - g * kPgRowGroup);
  const int r = g * kPgRowGroup + rem % gr;
  t.col_tile = rem / gr;
  if (p.row_tiles) {
    const int4 v = p.row_tiles[r];
    t.row0 = v.x;
    t.rows = v.y;
    t.block = v.z;
  } else {
    t.row0 = r * s.tile_n;
    t.rows = min(s.tile_n, s.m - t.row0);
    t.block = 0;
  }
  t.n = (t.rows + 31) & ~31;
  return t;
}

// ---- cta_group::2 forms of the wrappers in common.cuh ----------------------------------------------------------------
__device__ __forceinline__ uint32_t pair_first_cta_addr(uint32_t smem_addr) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(smem_addr));
  return r;
}
// Box into this CTA's shared memory; `bar` is a shared::cluster address (the first CTA's barrier).
__device__ __forceinline__ void tma_load_2d_pair(uint32_t smem_dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%3, "
      "%4}], [%2];" ::"r"(smem_dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair(uint32_t smem_dst, const CUtensorMap* map, uint32_t bar, int c0, int c1,
                                                 int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%3, %4, "
      "%5}], [%2];" ::"r"(smem_dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void umma_ss_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t"
      "}\n" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// One arrival at the barrier of this offset in both CTAs once every product issued so far has finished.
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
          smem_u32(bar)),
      "h"(static_cast<uint16_t>(3))
      : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// mbar_wait for a barrier that the other CTA of the pair arrives at.
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                                  int* status_word, int where) {
  for (uint32_t spin = 0; spin < kWaitSpinLimit; ++spin) {
    uint32_t ok;
    asm volatile(
        "{\n\t"
        ".reg .pred P;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 P, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, P;\n\t"
        "}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (ok)
      return true;
    if ((spin & 1023u) == 1023u && *abort_flag)
      return false;
  }
  *abort_flag = 1;
  if (status_word)
    atomicCAS(status_word, 0, where);
  return false;
}

template <bool SWIGLU>
__global__ void __launch_bounds__(kPgThreads, 1)
pair_gemm_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_a,
                 const __grid_constant__ CUtensorMap tmap_w2, const __grid_constant__ CUtensorMap tmap_a2_32,
                 const __grid_constant__ CUtensorMap tmap_a2_64, const __grid_constant__ CUtensorMap tmap_w64,
                 const PairGemmParams p) {
  pdl_wait();      // programmatic dependent launch: nothing before this reads an earlier kernel's data
  pdl_trigger();
  namespace cg = cooperative_groups;
  PgSched s;
  if (!pg_schedule(p, SWIGLU, s))
    return;        // no live rows: the whole grid leaves
  if (s.pair >= s.pairs)
    return;        // both CTAs of the pair

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t full_bar[kPgMaxStages];     // used in the first CTA of the pair
  __shared__ uint64_t empty_bar[kPgMaxStages];
  __shared__ uint64_t acc_full[2];
  __shared__ uint64_t acc_empty[2];               // used in the first CTA of the pair
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  __shared__ int last_part;    // this CTA finished the current tile last

  cg::cluster_group cluster = cg::this_cluster();
  const int rank = blockIdx.x & 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // k steps per stage: a stage costs some 500 clocks of barrier round trips between the two CTAs whatever it holds, so
  // narrow products, whose tensor work does not cover that, take two k steps at a time, one 3-D box per operand (46 rows:
  // K/V 36 -> 29 us, gate/up 46 -> 42; rotating the k steps over several accumulators instead made them slower)
  const int kps = s.tile_n <= 64 || (s.nb == 1 && s.tile_n <= 128) ? 2 : 1;
  const CUtensorMap* const tmap_a2 = s.tile_n <= 64 ? &tmap_a2_32 : &tmap_a2_64;   // rows of the activation box
  const uint32_t a_step = ((s.tile_n + 63) >> 6) * kPgABytes;                      // activation bytes per k step
  const uint32_t stage_bytes = kps * (s.nb * kPgWBytes + a_step);
  const int stages = min(kPgMaxStages, static_cast<int>((kPgRing - (s.narrow ? kPgSwapBytes : 0)) / stage_bytes));
  const int accs = 2 * s.nb * s.tile_n <= 512 ? 2 : 1;   // accumulators that fit the tensor memory

  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int i = 0; i < kPgMaxStages; ++i) {
      mbar_init(&full_bar[i], 1);
      mbar_init(&empty_bar[i], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], 16);   // one arrival per epilogue warp of both CTAs
    }
    fence_mbar_init();
    tma_prefetch_desc(kps == 2 ? &tmap_w2 : &tmap_w);
    tma_prefetch_desc(kps == 2 ? tmap_a2 : &tmap_a);
  }
  if (warp == 1) {
    tmem_alloc_pair(&tmem_slot, 512);
    tmem_relinquish_pair();
  }
  tc_fence_before_sync();
  cluster.sync();
  tc_fence_after_sync();
  const uint32_t tmem_base = tmem_slot;

  int u = s.pair;
  PgSeg g;
  if (warp == 0 || warp == 2) {
    // ------------------------------------------------------------------ producers: weights (warp 0), activations (warp 2)
    if (lane == 0) {
      int st = 0;
      uint32_t ph = 0;
      for (; pg_unit(s, u, g); u += s.pairs) {
        const PgTile t = pg_tile(p, s, g.tile);
        const int half = t.n >> 1;
        const int boxes = (half + 31) >> 5;
        const uint32_t pair_bytes = 2 * kps * (s.nb * kPgWBytes + (kps == 2 ? a_step : boxes * kPgABytes));
        const int w_row = t.block * p.w_rows_per_block +
                          (s.narrow ? (t.col_tile * 2 + rank) * 64
                                    : (t.col_tile * (SWIGLU ? 2 : 2 * s.nb) + rank * (SWIGLU ? 1 : s.nb)) * 128);
        const int w_step = SWIGLU ? p.up_row_offset : 128;
        const int a_row = t.row0 + rank * half;
        for (int k = g.k0; k < g.k1; k += kps) {
          mbar_wait(&empty_bar[st], ph ^ 1, &abort_flag, p.status_word, 501);
          if (rank == 0 && warp == 0)
            mbar_arrive_expect_tx(&full_bar[st], pair_bytes);
          const uint32_t bar = pair_first_cta_addr(smem_u32(&full_bar[st]));
          const uint32_t w_dst = smem_u32(smem + st * stage_bytes);
          const uint32_t a_dst = w_dst + kps * s.nb * kPgWBytes;
          if (warp == 0 && SWIGLU && s.narrow) {
            for (int h = 0; h < kps; ++h) {   // gate rows in the upper half of a k step's block, up rows in the lower one
              tma_load_2d_pair(w_dst + h * kPgWBytes, &tmap_w64, bar, (k + h) * 64, w_row);
              tma_load_2d_pair(w_dst + h * kPgWBytes + kPgWBytes / 2, &tmap_w64, bar, (k + h) * 64, w_row + w_step);
            }
          } else if (warp == 0) {
            for (int j = 0; j < s.nb; ++j)
              if (kps == 2)
                tma_load_3d_pair(w_dst + j * 2 * kPgWBytes, &tmap_w2, bar, 0, w_row + j * w_step, k);
              else
                tma_load_2d_pair(w_dst + j * kPgWBytes, &tmap_w, bar, k * 64, w_row + j * w_step);
          } else if (kps == 2) {
            tma_load_3d_pair(a_dst, tmap_a2, bar, 0, a_row, k);
          } else {
            for (int b = 0; b < boxes; ++b)
              tma_load_2d_pair(a_dst + b * kPgABytes, &tmap_a, bar, k * 64, a_row + b * 32);
          }
          if (++st == stages) {
            st = 0;
            ph ^= 1;
          }
        }
      }
      // The first CTA's commits arrive at the second CTA's barriers, too: every stage is seen released before this CTA may
      // end, so that none arrives at the shared memory of a CTA that has left.
      if (warp == 0)
        for (int i = 0; i < stages; ++i) {
          mbar_wait(&empty_bar[st], ph ^ 1, &abort_flag, p.status_word, 506);
          if (++st == stages) {
            st = 0;
            ph ^= 1;
          }
        }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (first CTA of the pair)
    if (rank == 0 && lane == 0) {
      int st = 0, seg = 0;
      uint32_t ph = 0;
      for (; pg_unit(s, u, g); u += s.pairs) {
        const PgTile t = pg_tile(p, s, g.tile);
        const uint32_t idesc = umma_idesc_bf16(256, t.n, 0, 0);
        const int acc = accs == 2 ? (seg & 1) : 0;
        const uint32_t use = accs == 2 ? (seg >> 1) : seg;
        mbar_wait_cluster(&acc_empty[acc], (use & 1) ^ 1, &abort_flag, p.status_word, 502);
        tc_fence_after_sync();
        const uint32_t d0 = tmem_base + acc * s.nb * s.tile_n;
        for (int k = g.k0; k < g.k1; k += kps) {
          mbar_wait(&full_bar[st], ph, &abort_flag, p.status_word, 503);
          tc_fence_after_sync();
          const uint32_t w_addr = smem_u32(smem + st * stage_bytes);
          const uint32_t a_addr = w_addr + kps * s.nb * kPgWBytes;
          for (int h = 0; h < kps && k + h < g.k1; ++h) {
            const uint64_t b_desc = umma_smem_desc_sw128(a_addr + h * a_step, 16, 1024);
            for (int j = 0; j < s.nb; ++j) {
              const uint64_t a_desc = umma_smem_desc_sw128(w_addr + (j * kps + h) * kPgWBytes, 16, 1024);
#pragma unroll
              for (int kk = 0; kk < 4; ++kk)
                umma_ss_pair(d0 + j * s.tile_n, a_desc + 2 * kk, b_desc + 2 * kk, idesc, (k + h > g.k0 || kk != 0) ? 1u : 0u);
            }
          }
          umma_commit_pair(&empty_bar[st]);
          if (++st == stages) {
            st = 0;
            ph ^= 1;
          }
        }
        umma_commit_pair(&acc_full[acc]);
        ++seg;
      }
    }
    __syncwarp();
  } else if (warp >= 4) {
    // ------------------------------------------------------------------ epilogue
    const int q = warp & 3;                  // tensor-memory lane quarter this warp may read
    const int part = (warp - 4) >> 2;        // which of every two 32-row chunks
    const bool odd = lane & 1;
    const uint32_t t_lane = static_cast<uint32_t>(q * 32) << 16;
    int seg = 0;
    for (; pg_unit(s, u, g); u += s.pairs) {
      const PgTile t = pg_tile(p, s, g.tile);
      const int acc = accs == 2 ? (seg & 1) : 0;
      const uint32_t use = accs == 2 ? (seg >> 1) : seg;
      const bool cut = !SWIGLU && s.parts > 1;
      if (cut && threadIdx.x == 128)
        open_counter(p.tickets + g.tile * 2 + rank, p.launch_id);
      mbar_wait(&acc_full[acc], use & 1, &abort_flag, p.status_word, 504);
      tc_fence_after_sync();
      const uint32_t d0 = tmem_base + acc * s.nb * s.tile_n + t_lane;
      const int col_cta = s.narrow ? (t.col_tile * 2 + rank) * 64
                                   : (t.col_tile * (SWIGLU ? 2 : 2 * s.nb) + rank * (SWIGLU ? 1 : s.nb)) * 128;
      const int chunks = (t.rows + 31) >> 5;

      // 32 rows of one block, already final except for bias and scale: bf16 pairs to their rows
      auto store_chunk = [&](int c, int col_block, const float (&v)[32]) {
        const int rl = c * 32 + lane;
        int dest = -1;
        float scale = 1.f;
        if (rl < t.rows) {
          dest = p.out_row_map ? p.out_row_map[t.row0 + rl] : t.row0 + rl;
          if (p.row_scale)
            scale = p.row_scale[t.row0 + rl];
        }
        const int col = col_block + q * 32 + lane;
        const int col2 = col & ~1;
        __nv_bfloat162 bias = __floats2bfloat162_rn(0.f, 0.f);
        float own_bias = 0.f;
        if (p.bias && col2 < p.n) {
          bias = __halves2bfloat162(p.bias[col2], p.bias[col2 + 1]);   // a bias may start at any element
          own_bias = odd ? __bfloat162float(bias.y) : __bfloat162float(bias.x);
        }
        const bool second = p.out2 && col_block >= p.split_col;
        __nv_bfloat16* base = second ? p.out2 + (col2 - p.split_col) : p.out + col2;
        const int64_t ld = second ? p.ldc2 : p.ldc;
#pragma unroll
        for (int r = 0; r < 32; r += 2) {
          float v0 = v[r], v1 = v[r + 1];
          if (p.bias && p.bias_fp32) {
            v0 += own_bias;
            v1 += own_bias;
          }
          if (p.row_scale) {
            v0 *= __shfl_sync(0xffffffffu, scale, r);
            v1 *= __shfl_sync(0xffffffffu, scale, r + 1);
          }
          const float got = __shfl_xor_sync(0xffffffffu, odd ? v0 : v1, 1);
          const int row = __shfl_sync(0xffffffffu, dest, r + (odd ? 1 : 0));
          __nv_bfloat162 h = __floats2bfloat162_rn(odd ? got : v0, odd ? v1 : got);
          if (p.bias && !p.bias_fp32)
            h = __hadd2(h, bias);
          if (row >= 0 && col2 < p.n)
            *reinterpret_cast<__nv_bfloat162*>(base + row * ld) = h;
        }
      };
      const int64_t part_floats = static_cast<int64_t>(kSplitRows) * p.n;
      auto keep_chunk = [&](int c, int col_block, const uint32_t (&r32)[32]) {   // partial sums of one block
        const int col = col_block + q * 32 + lane;
        if (col >= p.n)
          return;
        float* dst = p.partial + g.part * part_floats + static_cast<int64_t>(t.row0 + c * 32) * p.n + col;
        const int live = t.rows - c * 32;
        const bool some = g.k1 > g.k0;   // the last part of a short k range may be empty
#pragma unroll
        for (int r = 0; r < 32; ++r)
          if (r < live)
            __stcg(dst + static_cast<int64_t>(r) * p.n, some ? __uint_as_float(r32[r]) : 0.f);
      };
      if (SWIGLU && s.narrow) {
        // lane quarters 0, 1 hold gate columns, 2, 3 the up values of the same columns: these cross through shared memory
        float* swap = reinterpret_cast<float*>(smem + kPgRing - kPgSwapBytes) + part * (32 * 64) + (q & 1) * 32 + lane;
        for (int c = part; c < chunks; c += 2) {
          uint32_t ra[32];
          tmem_ld_32x32(d0 + c * 32, ra);
          tmem_ld_wait();
          if (q >= 2) {
#pragma unroll
            for (int r = 0; r < 32; ++r)
              swap[r * 64] = __uint_as_float(ra[r]);
          }
          if (part == 0)
            asm volatile("bar.sync 2, 128;" ::: "memory");
          else
            asm volatile("bar.sync 3, 128;" ::: "memory");
          if (q < 2) {
            float a[32];
#pragma unroll
            for (int r = 0; r < 32; ++r)
              a[r] = silu_f(__uint_as_float(ra[r])) * swap[r * 64];
            store_chunk(c, col_cta, a);
          }
          if (part == 0)   // read before the next chunk's values overwrite them
            asm volatile("bar.sync 2, 128;" ::: "memory");
          else
            asm volatile("bar.sync 3, 128;" ::: "memory");
        }
      } else {
        for (int c = part; c < chunks; c += 2) {
          if (SWIGLU) {
            uint32_t ra[32], rb[32];
            tmem_ld_32x32(d0 + c * 32, ra);
            tmem_ld_32x32(d0 + s.tile_n + c * 32, rb);
            tmem_ld_wait();
            float a[32];
#pragma unroll
            for (int r = 0; r < 32; ++r)
              a[r] = silu_f(__uint_as_float(ra[r])) * __uint_as_float(rb[r]);
            store_chunk(c, col_cta, a);
          } else {
#pragma unroll 1
            for (int j = 0; j < s.nb; ++j) {
              uint32_t ra[32];
              tmem_ld_32x32(d0 + j * s.tile_n + c * 32, ra);
              tmem_ld_wait();
              if (cut) {
                keep_chunk(c, col_cta + j * 128, ra);
              } else {
                float a[32];
#pragma unroll
                for (int r = 0; r < 32; ++r)
                  a[r] = __uint_as_float(ra[r]);
                store_chunk(c, col_cta + j * 128, a);
              }
            }
          }
        }
      }
      // the accumulator may be overwritten
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0)
        mbar_arrive_cluster(pair_first_cta_addr(smem_u32(&acc_empty[acc])));

      if (cut) {
        __threadfence();
        asm volatile("bar.sync 1, 256;" ::: "memory");
        if (threadIdx.x == 128)
          last_part = last_to_arrive(p.tickets + g.tile * 2 + rank, s.parts) ? 1 : 0;
        asm volatile("bar.sync 1, 256;" ::: "memory");
        if (last_part) {
          __threadfence();
          // every warp sums whole rows (16 bytes per lane and 128-column block), four rows and all parts at a time with
          // all loads in flight; the parts are added in k order
          constexpr int kRows = 4;
          for (int r0 = warp - 4; r0 < t.rows; r0 += 8 * kRows) {
#pragma unroll 1
            for (int j = 0; j < s.nb; ++j) {
              const int col_block = col_cta + j * 128, col = col_block + lane * 4;
              if (col >= p.n)
                continue;
              float4 v[kMaxSplits][kRows];
#pragma unroll
              for (int z = 0; z < kMaxSplits; ++z)
#pragma unroll
                for (int x = 0; x < kRows; ++x)
                  v[z][x] = z < s.parts ? __ldcg(reinterpret_cast<const float4*>(
                                              p.partial + z * part_floats +
                                              static_cast<int64_t>(t.row0 + min(r0 + 8 * x, t.rows - 1)) * p.n + col))
                                        : make_float4(0.f, 0.f, 0.f, 0.f);
              const bool second = p.out2 && col_block >= p.split_col;
              __nv_bfloat16* base = second ? p.out2 + (col - p.split_col) : p.out + col;
              const int64_t ld = second ? p.ldc2 : p.ldc;
#pragma unroll
              for (int x = 0; x < kRows; ++x) {
                const int r = r0 + 8 * x;
                if (r >= t.rows)
                  continue;
                const int dest = p.out_row_map ? p.out_row_map[t.row0 + r] : t.row0 + r;
                if (dest < 0)
                  continue;
                const float scale = p.row_scale ? p.row_scale[t.row0 + r] : 1.f;
                float a[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int z = 0; z < kMaxSplits; ++z) {
                  a[0] += v[z][x].x;
                  a[1] += v[z][x].y;
                  a[2] += v[z][x].z;
                  a[3] += v[z][x].w;
                }
                if (p.bias && p.bias_fp32) {
#pragma unroll
                  for (int z = 0; z < 4; ++z)
                    a[z] += __bfloat162float(p.bias[col + z]);
                }
                __nv_bfloat162 h[2];
                h[0] = __floats2bfloat162_rn(a[0] * scale, a[1] * scale);
                h[1] = __floats2bfloat162_rn(a[2] * scale, a[3] * scale);
                if (p.bias && !p.bias_fp32) {
#pragma unroll
                  for (int z = 0; z < 2; ++z)
                    h[z] = __hadd2(h[z], __halves2bfloat162(p.bias[col + 2 * z], p.bias[col + 2 * z + 1]));
                }
                *reinterpret_cast<uint2*>(base + dest * ld) = *reinterpret_cast<const uint2*>(h);
              }
            }
          }
        }
        asm volatile("bar.sync 1, 256;" ::: "memory");   // last_part is read before the next tile's ticket
      }
      ++seg;
    }
  }

  __syncwarp();
  tc_fence_before_sync();
  cluster.sync();   // no CTA frees tensor memory or leaves while its pair's products or arrivals are in flight
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem_base, 512);
  }
  cluster.sync();
}

}  // namespace dyllm
