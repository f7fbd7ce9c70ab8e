// Mixture-of-experts FFN on salient rows: softmax top-k router, expert-sorted grouped GEMMs on the
// CTA-pair kernel of pair_gemm.cuh (one weight block per row tile), routing weight folded into the
// down-projection epilogue, per-token sum over the top-k slots.
//
//   route    logits = x[idx[m]] . Wr^T (fp32), softmax over experts, top-k       (one or four rows per block)
//   align    (row, slot) pairs grouped by expert, row tiles of at most 256 rows  (one block)
//   GEMM 1   h = silu(x Wg_e^T) * (x Wu_e^T) for the rows of each tile's expert
//   GEMM 2   y[pair] = w_pair * (h Wd_e^T)
//   combine  out[map[m]] = sum over the owned slots of row m of y[m * k + j]
#include "gemm.cuh"
#include "pair_gemm.cuh"

namespace dyllm {

namespace {

constexpr int kMaxExperts = 256;
constexpr int kMaxTopK = 16;

// Router.  A block takes R rows at a time, its 16 warps share out the experts in pairs, lanes split the hidden
// dimension.  Several rows wait in shared memory, so a weight vector fetched from L2 serves R rows: with one row per block
// 3003 rows read the 256 KB router weight (64 experts, hidden 2048) 3003 times, 88 us.  Few rows are bound by the latency
// of the weight loads instead: R = 1 spreads them over more blocks, and a lane keeps eight loads in flight (150 rows:
// 21 us with one expert and one load at a time).
constexpr int kRouteThreads = 512;
constexpr int kRouteManyRows = 4;

template <int R>
__device__ __forceinline__ void
route_rows(const __nv_bfloat16* __restrict__ x, int64_t ldx, const int32_t* __restrict__ idx, int x_rows, int n,
           const __nv_bfloat16* __restrict__ wr, int hidden, int num_experts, int top_k, int renormalize,
           float* __restrict__ topk_w, int32_t* __restrict__ topk_ids, uint4* s_x, float (*s_all)[kMaxExperts]) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int vecs = hidden / 8;
  for (int m0 = blockIdx.x * R; m0 < n; m0 += gridDim.x * R) {
    const uint4* xr = nullptr;
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const int m = min(m0 + j, n - 1);
      const int r = idx ? min(max(idx[m], 0), x_rows - 1) : m;
      xr = reinterpret_cast<const uint4*>(x + static_cast<int64_t>(r) * ldx);
      if (R > 1)
        for (int v = threadIdx.x; v < vecs; v += kRouteThreads)
          s_x[j * vecs + v] = __ldg(xr + v);
    }
    if (R > 1)
      __syncthreads();
    const int per_warp = num_experts > kRouteThreads / 32 ? 2 : 1;
    for (int e = warp * per_warp; e < num_experts; e += kRouteThreads / 32 * per_warp) {
      const bool two = per_warp == 2 && e + 1 < num_experts;
      const uint4* w0 = reinterpret_cast<const uint4*>(wr + static_cast<int64_t>(e) * hidden);
      const uint4* w1 = two ? w0 + vecs : w0;
      float acc[2][R];
#pragma unroll
      for (int j = 0; j < R; ++j)
        acc[0][j] = acc[1][j] = 0.f;
      for (int v0 = lane; v0 < vecs; v0 += 128) {
        uint4 w[2][4], xa[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int v = v0 + i * 32;
          w[0][i] = v < vecs ? __ldg(w0 + v) : make_uint4(0, 0, 0, 0);
          w[1][i] = two && v < vecs ? __ldg(w1 + v) : make_uint4(0, 0, 0, 0);
          if (R == 1)
            xa[i] = v < vecs ? __ldg(xr + v) : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int v = v0 + i * 32;
          if (v >= vecs)
            break;
#pragma unroll
          for (int j = 0; j < R; ++j) {
            const uint4 a = R > 1 ? s_x[j * vecs + v] : xa[i];
            const __nv_bfloat162* a2 = reinterpret_cast<const __nv_bfloat162*>(&a);
#pragma unroll
            for (int z = 0; z < 2; ++z) {
              const __nv_bfloat162* b2 = reinterpret_cast<const __nv_bfloat162*>(&w[z][i]);
#pragma unroll
              for (int c = 0; c < 4; ++c) {
                const float2 fa = __bfloat1622float2(a2[c]), fb = __bfloat1622float2(b2[c]);
                acc[z][j] = fmaf(fa.x, fb.x, acc[z][j]);
                acc[z][j] = fmaf(fa.y, fb.y, acc[z][j]);
              }
            }
          }
        }
      }
#pragma unroll
      for (int z = 0; z < 2; ++z)
#pragma unroll
        for (int j = 0; j < R; ++j) {
#pragma unroll
          for (int off = 16; off > 0; off >>= 1)
            acc[z][j] += __shfl_xor_sync(0xffffffffu, acc[z][j], off);
          if (lane == 0 && (z == 0 || two))
            s_all[j][e + z] = acc[z][j];
        }
    }
    __syncthreads();
    const int m = m0 + warp;
    if (warp < R && m < n) {
      float* s_logits = s_all[warp];
      // softmax over the experts, then top-k by repeated arg-max (lowest index wins ties).  NaN (a logit that is NaN or
      // +inf) ranks below every number and above the experts already taken (-1), so that a pick is an expert always; the
      // sum, hence every weight of such a row, is NaN.
      float mx = -3.0e38f;
      for (int e = lane; e < num_experts; e += 32)
        mx = fmaxf(mx, s_logits[e]);
#pragma unroll
      for (int off = 16; off > 0; off >>= 1)
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
      float sum = 0.f;
      for (int e = lane; e < num_experts; e += 32) {
        const float pe = expf(s_logits[e] - mx);
        s_logits[e] = pe;
        sum += pe;
      }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1)
        sum += __shfl_xor_sync(0xffffffffu, sum, off);
      __syncwarp();
      const float inv = 1.0f / sum;
      float picked_w = 0.f, total = 0.f;
      int picked_e = 0;
      for (int j = 0; j < top_k; ++j) {
        float best = -1.f;
        int best_e = 0x7fffffff;
        for (int e = lane; e < num_experts; e += 32) {
          const float v = isnan(s_logits[e]) ? -0.5f : s_logits[e];
          if (v > best) {
            best = v;
            best_e = e;
          }
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
          const float ob = __shfl_xor_sync(0xffffffffu, best, off);
          const int oe = __shfl_xor_sync(0xffffffffu, best_e, off);
          if (ob > best || (ob == best && oe < best_e)) {
            best = ob;
            best_e = oe;
          }
        }
        if (lane == 0)
          s_logits[best_e] = -1.f;  // taken
        __syncwarp();
        if (lane == j) {
          picked_w = best * inv;
          picked_e = best_e;
        }
        total += best * inv;
      }
      if (lane < top_k) {
        const float w = renormalize ? picked_w / total : picked_w;
        // the reference hands the routing weights on in the activation dtype (bf16)
        topk_w[static_cast<int64_t>(m) * top_k + lane] = __bfloat162float(__float2bfloat16(w));
        topk_ids[static_cast<int64_t>(m) * top_k + lane] = picked_e;
      }
    }
    __syncthreads();
  }
}

// `shared_rows`: rows that the dynamic shared memory holds (0: always one row per block at a time).
__global__ void __launch_bounds__(kRouteThreads, 2)
moe_route_kernel(const __nv_bfloat16* __restrict__ x, int64_t ldx, const int32_t* __restrict__ idx, int x_rows,
                 int num_rows, const int32_t* __restrict__ num_rows_dev, const __nv_bfloat16* __restrict__ wr,
                 int hidden, int num_experts, int top_k, int renormalize, float* __restrict__ topk_w,
                 int32_t* __restrict__ topk_ids, int shared_rows) {
  pdl_wait();      // programmatic dependent launch: nothing before this reads an earlier kernel's data
  pdl_trigger();
  extern __shared__ uint4 s_x[];                 // [kRouteManyRows][hidden / 8]
  __shared__ float s_all[kRouteManyRows][kMaxExperts];
  const int n = num_rows_dev ? min(num_rows, *num_rows_dev) : num_rows;
  // several rows per block once there are enough rows for more than one turn of the grid
  if (shared_rows >= kRouteManyRows && n > static_cast<int>(gridDim.x))
    route_rows<kRouteManyRows>(x, ldx, idx, x_rows, n, wr, hidden, num_experts, top_k, renormalize, topk_w, topk_ids, s_x, s_all);
  else
    route_rows<1>(x, ldx, idx, x_rows, n, wr, hidden, num_experts, top_k, renormalize, topk_w, topk_ids, s_x, s_all);
}

// Single block: the position of every owned (row, slot) pair when the pairs are grouped by local expert, in pair order
// inside an expert (-1 for a pair of another rank's expert), and the row tiles of every expert (at most 256 rows each,
// spread evenly in steps of 32: the tiles of pair_gemm.cuh).  Every warp owns a contiguous part of the pairs and counts
// it with warp matches, so no counter is shared between warps and the order is the same in every run.  Only the positions
// are written here, coalesced; what lies at a position is scattered by moe_stage_kernel on all SMs (from this one SM the
// scattered stores alone took 25 of 35 us at 24 000 pairs).
constexpr int kAlignWarps = 32;
constexpr int kAlignBatch = 8;   // independent loads in flight per lane

__global__ void __launch_bounds__(kAlignWarps * 32)
moe_align_kernel(const int32_t* __restrict__ topk_ids, int num_rows,
                 const int32_t* __restrict__ num_rows_dev, int top_k, int expert_start, int num_local_experts,
                 int32_t* __restrict__ pair_pos, int4* __restrict__ row_tiles, int32_t* __restrict__ tiles_dev) {
  pdl_wait();      // programmatic dependent launch: nothing before this reads an earlier kernel's data
  pdl_trigger();
  __shared__ int s_next[kAlignWarps][kMaxExperts];   // pairs per warp and expert, then the warp's next position
  __shared__ int s_warp[2][kMaxExperts / 32];
  __shared__ int s_max;
  const int n = num_rows_dev ? min(num_rows, *num_rows_dev) : num_rows;
  const int pairs = n * top_k;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int per_warp = ((pairs + kAlignWarps - 1) / kAlignWarps + 31) & ~31;
  const int p0 = warp * per_warp, p1 = min(pairs, p0 + per_warp);
  const int used = per_warp ? (pairs + per_warp - 1) / per_warp : 0;   // warps that own pairs
  for (int i = threadIdx.x; i < used * kMaxExperts; i += blockDim.x)
    s_next[i / kMaxExperts][i % kMaxExperts] = 0;
  if (threadIdx.x == 0)
    s_max = 0;
  __syncthreads();
  for (int base = p0; base < p1; base += 32 * kAlignBatch) {
    int e[kAlignBatch];
#pragma unroll
    for (int j = 0; j < kAlignBatch; ++j) {
      const int i = base + j * 32 + lane;
      e[j] = i < p1 ? topk_ids[i] - expert_start : -1;
      if (e[j] >= num_local_experts)
        e[j] = -1;
    }
#pragma unroll
    for (int j = 0; j < kAlignBatch; ++j) {
      const unsigned same = __match_any_sync(0xffffffffu, e[j]);
      if (e[j] >= 0 && lane == __ffs(same) - 1)
        s_next[warp][e[j]] += __popc(same);
      __syncwarp();
    }
  }
  __syncthreads();
  // positions: experts in order, warps in order inside an expert
  int count = 0, tiles = 0;
  if (threadIdx.x < kMaxExperts) {
    const int e = threadIdx.x;
    for (int w = 0; w < used; ++w) {
      const int c = s_next[w][e];
      s_next[w][e] = count;
      count += c;
    }
    const int even = (count + kPgMaxRows - 1) / kPgMaxRows;
    const int h = count ? ((count + even - 1) / even + 31) & ~31 : 32;
    tiles = (count + h - 1) / h;
    int c_incl = count, t_incl = tiles;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int oc = __shfl_up_sync(0xffffffffu, c_incl, off), ot = __shfl_up_sync(0xffffffffu, t_incl, off);
      if (lane >= off) {
        c_incl += oc;
        t_incl += ot;
      }
    }
    if (lane == 31) {
      s_warp[0][warp] = c_incl;
      s_warp[1][warp] = t_incl;
    }
    asm volatile("bar.sync 1, 256;" ::: "memory");
    int c_first = c_incl - count, t_first = t_incl - tiles;
    for (int w = 0; w < warp; ++w) {
      c_first += s_warp[0][w];
      t_first += s_warp[1][w];
    }
    for (int w = 0; w < used; ++w)
      s_next[w][e] += c_first;
    if (tiles > 0) {
      for (int t = 0; t < tiles; ++t)
        row_tiles[t_first + t] = make_int4(c_first + t * h, min(h, count - t * h), e, 0);
      atomicMax(&s_max, min(h, count));
    }
    if (e == kMaxExperts - 1)
      tiles_dev[0] = t_first + tiles;
  }
  __syncthreads();
  if (threadIdx.x == 0)
    tiles_dev[1] = s_max;
  for (int base = p0; base < p1; base += 32 * kAlignBatch) {
    int e[kAlignBatch];
#pragma unroll
    for (int j = 0; j < kAlignBatch; ++j) {
      const int i = base + j * 32 + lane;
      e[j] = i < p1 ? topk_ids[i] - expert_start : -1;
      if (e[j] >= num_local_experts)
        e[j] = -1;
    }
#pragma unroll
    for (int j = 0; j < kAlignBatch; ++j) {
      const int i = base + j * 32 + lane;
      const unsigned same = __match_any_sync(0xffffffffu, e[j]);
      int pos = -1;
      if (e[j] >= 0)
        pos = s_next[warp][e[j]] + __popc(same & ((1u << lane) - 1u));
      if (i < p1)
        pair_pos[i] = pos;
      __syncwarp();
      if (e[j] >= 0 && lane == __ffs(same) - 1)
        s_next[warp][e[j]] += __popc(same);
      __syncwarp();
    }
  }
}

// staged[pos] = x row of every owned pair, pair_idx[pos] = pair, pair_w[pos] = its routing weight.  One warp per row of x,
// which it reads once and writes to the row's top_k positions; few rows get a warp per position instead (60 rows: 6.4 us
// with eight copies one after the other, 3.7 without).
__global__ void __launch_bounds__(256)
moe_stage_kernel(const uint4* __restrict__ x, int64_t x_pitch_vecs, const int32_t* __restrict__ idx, int x_rows,
                 const int32_t* __restrict__ pair_pos, const float* __restrict__ topk_w, int num_rows,
                 const int32_t* __restrict__ num_rows_dev, int top_k, uint4* __restrict__ staged, int vecs,
                 int32_t* __restrict__ pair_idx, float* __restrict__ pair_w) {
  pdl_wait();      // programmatic dependent launch: nothing before this reads an earlier kernel's data
  pdl_trigger();
  const int n = num_rows_dev ? min(num_rows, *num_rows_dev) : num_rows;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int slots = n * top_k <= static_cast<int>(gridDim.x) * 8 ? 1 : top_k;   // positions per warp
  const int per_row = top_k / slots;
  for (int item = blockIdx.x * 8 + warp; item < n * per_row; item += gridDim.x * 8) {
    const int m = item / per_row, k0 = item - m * per_row;
    const int r = idx ? min(max(idx[m], 0), x_rows - 1) : m;
    const uint4* src = x + static_cast<int64_t>(r) * x_pitch_vecs;
    const int my_pos = lane < top_k ? pair_pos[static_cast<int64_t>(m) * top_k + lane] : -1;   // top_k <= 16
    if (my_pos >= 0 && k0 == 0) {
      const int i = m * top_k + lane;
      pair_idx[my_pos] = i;
      pair_w[my_pos] = topk_w[i];
    }
    for (int base = 0; base < vecs; base += 128) {   // uniform over the warp
      const int v0 = base + lane;
      uint4 a[4];
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (v0 + j * 32 < vecs)
          a[j] = __ldg(src + v0 + j * 32);
      for (int k = k0; k < k0 + slots; ++k) {
        const int pos = __shfl_sync(0xffffffffu, my_pos, k);
        if (pos < 0)
          continue;
        uint4* dst = staged + static_cast<int64_t>(pos) * vecs;
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (v0 + j * 32 < vecs)
            dst[v0 + j * 32] = a[j];
      }
    }
  }
}

// out[map[m]] = bf16( sum over the owned slots j of y[m * k + j] ), fp32 accumulation in slot order.
__global__ void __launch_bounds__(256)
moe_combine_kernel(const __nv_bfloat16* __restrict__ y, const int32_t* __restrict__ topk_ids, int num_rows,
                   const int32_t* __restrict__ num_rows_dev, int top_k, int expert_start, int num_local_experts,
                   int hidden, __nv_bfloat16* __restrict__ out, int64_t ldo, const int32_t* __restrict__ out_row_map) {
  pdl_wait();      // programmatic dependent launch: nothing before this reads an earlier kernel's data
  pdl_trigger();
  const int n = num_rows_dev ? min(num_rows, *num_rows_dev) : num_rows;
  const int vecs = hidden / 8;
  for (int m = blockIdx.x; m < n; m += gridDim.x) {
    const int dst_row = out_row_map ? out_row_map[m] : m;
    if (dst_row < 0)
      continue;
    for (int v = threadIdx.x; v < vecs; v += blockDim.x) {
      float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      for (int j = 0; j < top_k; ++j) {
        const int e = topk_ids[static_cast<int64_t>(m) * top_k + j] - expert_start;
        if (e < 0 || e >= num_local_experts)
          continue;
        const uint4 a = __ldg(reinterpret_cast<const uint4*>(y + (static_cast<int64_t>(m) * top_k + j) * hidden) + v);
        const __nv_bfloat162* a2 = reinterpret_cast<const __nv_bfloat162*>(&a);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 f = __bfloat1622float2(a2[i]);
          acc[2 * i] += f.x;
          acc[2 * i + 1] += f.y;
        }
      }
      uint4 o = make_uint4(pack_bf16x2(acc[0], acc[1]), pack_bf16x2(acc[2], acc[3]), pack_bf16x2(acc[4], acc[5]),
                           pack_bf16x2(acc[6], acc[7]));
      reinterpret_cast<uint4*>(out + static_cast<int64_t>(dst_row) * ldo)[v] = o;
    }
  }
}

size_t align_up_sz(size_t v, size_t a) { return (v + a - 1) / a * a; }

struct MoeLayout {
  int pairs;           // (row, slot) positions
  size_t off_pos, off_pair_idx, off_pair_w, off_tiles, off_counts, off_staged, off_inter, off_y, total;
};

MoeLayout moe_layout(int max_rows, int top_k, int num_local_experts, int hidden, int inter) {
  MoeLayout l;
  const int64_t pairs = static_cast<int64_t>(max_rows) * top_k;
  l.pairs = static_cast<int>(pairs);
  size_t off = 0;
  l.off_pos = off;         off = align_up_sz(off + pairs * 4, 1024);
  l.off_pair_idx = off;    off = align_up_sz(off + pairs * 4, 1024);
  l.off_pair_w = off;      off = align_up_sz(off + pairs * 4, 1024);
  l.off_tiles = off;       off = align_up_sz(off + (pairs / kPgMaxRows + num_local_experts) * sizeof(int4), 1024);
  l.off_counts = off;      off = align_up_sz(off + 16, 1024);
  l.off_staged = off;      off = align_up_sz(off + static_cast<size_t>(pairs) * hidden * 2, 1024);
  l.off_inter = off;       off = align_up_sz(off + static_cast<size_t>(pairs) * inter * 2, 1024);
  l.off_y = off;           off = align_up_sz(off + static_cast<size_t>(pairs) * hidden * 2, 1024);
  l.total = off;
  return l;
}

}  // namespace
}  // namespace dyllm

using namespace dyllm;

extern "C" {

int dyllm_moe_route(const void* x, int x_rows, int hidden, int64_t ldx, const int32_t* idx, int num_rows,
                    const int32_t* num_rows_dev, const void* router_weight, int num_experts, int top_k,
                    int renormalize, float* topk_weights, int32_t* topk_ids, void* stream) {
  DYLLM_REQUIRE(x_rows >= 0 && num_rows >= 0 && hidden > 0, DYLLM_ERR_INVALID_ARGUMENT, "moe_route: rows %d hidden %d",
                num_rows, hidden);
  DYLLM_REQUIRE(num_experts > 0 && num_experts <= kMaxExperts && top_k > 0 && top_k <= kMaxTopK && top_k <= num_experts,
                DYLLM_ERR_UNSUPPORTED, "moe_route: %d experts (max %d), top-%d (max %d)", num_experts, kMaxExperts,
                top_k, kMaxTopK);
  DYLLM_REQUIRE(hidden % 8 == 0 && ldx % 8 == 0, DYLLM_ERR_UNSUPPORTED, "moe_route: hidden and pitch must be multiples of 8");
  if (num_rows == 0 || x_rows == 0)
    return DYLLM_OK;
  DYLLM_REQUIRE(x && router_weight && topk_weights && topk_ids, DYLLM_ERR_INVALID_ARGUMENT, "moe_route: null pointer");
  // the live count is known on the device only: the kernel chooses between one and several rows per block
  const int shared_rows = num_rows >= kRouteManyRows && kRouteManyRows * hidden * 2 <= 40 * 1024 ? kRouteManyRows : 0;
  const int blocks = min(num_rows, 2 * sm_count());
  DYLLM_LAUNCH(moe_route_kernel, blocks, kRouteThreads, static_cast<size_t>(shared_rows) * hidden * 2,
      static_cast<cudaStream_t>(stream),
      static_cast<const __nv_bfloat16*>(x), ldx, idx, x_rows, num_rows, num_rows_dev,
      static_cast<const __nv_bfloat16*>(router_weight), hidden, num_experts, top_k, renormalize, topk_weights, topk_ids,
      shared_rows);
  return check_launch("moe_route");
}

size_t dyllm_moe_ffn_workspace_bytes(int max_rows, int top_k, int num_local_experts, int hidden, int inter) {
  if (max_rows <= 0 || top_k <= 0 || num_local_experts <= 0 || hidden <= 0 || inter <= 0)
    return 0;
  return moe_layout(max_rows, top_k, num_local_experts, hidden, inter).total;
}

int dyllm_moe_ffn(const void* x, int x_rows, int hidden, int64_t ldx, const int32_t* idx, int num_rows,
                  const int32_t* num_rows_dev, int rows_hint, const float* topk_weights, const int32_t* topk_ids,
                  int top_k, const void* w1, const void* w2, int num_local_experts, int expert_start, int inter,
                  void* out, int64_t ldo, const int32_t* out_row_map, void* workspace, size_t workspace_bytes,
                  void* stream) {
  DYLLM_REQUIRE(x_rows >= 0 && num_rows >= 0 && hidden > 0 && inter > 0, DYLLM_ERR_INVALID_ARGUMENT,
                "moe_ffn: rows %d hidden %d inter %d", num_rows, hidden, inter);
  DYLLM_REQUIRE(num_local_experts > 0 && num_local_experts <= kMaxExperts && top_k > 0 && top_k <= kMaxTopK,
                DYLLM_ERR_UNSUPPORTED, "moe_ffn: %d local experts (max %d), top-%d (max %d)", num_local_experts,
                kMaxExperts, top_k, kMaxTopK);
  DYLLM_REQUIRE(hidden % 64 == 0 && inter % 64 == 0 && ldx % 8 == 0 && ldo % 8 == 0, DYLLM_ERR_UNSUPPORTED,
                "moe_ffn: hidden and inter must be multiples of 64, pitches of 8");
  if (num_rows == 0 || x_rows == 0)
    return DYLLM_OK;
  DYLLM_REQUIRE(x && topk_weights && topk_ids && w1 && w2 && out && workspace, DYLLM_ERR_INVALID_ARGUMENT,
                "moe_ffn: null pointer");
  const MoeLayout l = moe_layout(num_rows, top_k, num_local_experts, hidden, inter);
  DYLLM_REQUIRE(workspace_bytes >= l.total && (reinterpret_cast<uintptr_t>(workspace) & 15) == 0, DYLLM_ERR_WORKSPACE,
                "moe_ffn: needs a 16-byte aligned workspace of %zu bytes (got %zu)", l.total, workspace_bytes);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  int32_t* pair_pos = reinterpret_cast<int32_t*>(ws + l.off_pos);
  int32_t* pair_idx = reinterpret_cast<int32_t*>(ws + l.off_pair_idx);
  float* pair_w = reinterpret_cast<float*>(ws + l.off_pair_w);
  int4* row_tiles = reinterpret_cast<int4*>(ws + l.off_tiles);
  int32_t* tiles_dev = reinterpret_cast<int32_t*>(ws + l.off_counts);
  void* staged = ws + l.off_staged;
  __nv_bfloat16* inter_buf = reinterpret_cast<__nv_bfloat16*>(ws + l.off_inter);
  __nv_bfloat16* y = reinterpret_cast<__nv_bfloat16*>(ws + l.off_y);

  DYLLM_LAUNCH(moe_align_kernel, 1, kAlignWarps * 32, 0, s, topk_ids, num_rows, num_rows_dev, top_k, expert_start,
               num_local_experts, pair_pos, row_tiles, tiles_dev);
  int rc = check_launch("moe_align");
  if (rc != DYLLM_OK)
    return rc;
  const int hint_rows = rows_hint > 0 && rows_hint < num_rows ? rows_hint : num_rows;
  DYLLM_LAUNCH(moe_stage_kernel, static_cast<int>(min(cdiv_l(static_cast<int64_t>(hint_rows) * top_k, 8), static_cast<int64_t>(sm_count()) * 8)), 256, 0, s, static_cast<const uint4*>(x),
               ldx / 8, idx, x_rows, pair_pos, topk_weights, num_rows, num_rows_dev, top_k,
               static_cast<uint4*>(staged), hidden / 8, pair_idx, pair_w);
  rc = check_launch("moe_stage");
  if (rc != DYLLM_OK)
    return rc;
  PairGemmParams g = {};
  g.row_tiles = row_tiles;
  g.tiles_dev = tiles_dev;
  g.K = hidden;
  g.n = inter;
  g.w_rows_per_block = 2 * inter;
  g.up_row_offset = inter;
  g.out = inter_buf;
  g.ldc = inter;
  rc = launch_pair_gemm(true, g, staged, l.pairs, hidden, w1, static_cast<int64_t>(num_local_experts) * 2 * inter, s);
  if (rc != DYLLM_OK)
    return rc;
  g.K = inter;
  g.n = hidden;
  g.w_rows_per_block = hidden;
  g.up_row_offset = 0;
  g.out = y;
  g.ldc = hidden;
  g.out_row_map = pair_idx;
  g.row_scale = pair_w;
  rc = launch_pair_gemm(false, g, inter_buf, l.pairs, inter, w2, static_cast<int64_t>(num_local_experts) * hidden, s);
  if (rc != DYLLM_OK)
    return rc;
  const int blocks = min(hint_rows, sm_count() * 8);
  DYLLM_LAUNCH(moe_combine_kernel, blocks < 1 ? 1 : blocks, 256, 0, s, y, topk_ids, num_rows, num_rows_dev, top_k, expert_start,
                                                            num_local_experts, hidden, static_cast<__nv_bfloat16*>(out),
                                                            ldo, out_row_map);
  return check_launch("moe_combine");
}

}  // extern "C"
