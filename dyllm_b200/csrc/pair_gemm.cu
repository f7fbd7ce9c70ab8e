// Launch of the CTA-pair GEMM (pair_gemm.cuh).
#include <atomic>

#include "pair_gemm.cuh"

namespace dyllm {

namespace {

template <bool SWIGLU>
int launch(const CUtensorMap (&t)[6], const PairGemmParams& p, int pairs, cudaStream_t stream) {
  auto kernel = pair_gemm_kernel<SWIGLU>;
  // one flag per kernel instantiation and device: the opt-in shared-memory size is a per-function attribute
  static std::atomic<bool> smem_set[64];
  int dev = 0;
  cudaGetDevice(&dev);
  dev = (dev < 0 || dev >= 64) ? 0 : dev;
  if (!smem_set[dev].load(std::memory_order_acquire)) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kPgSmem)) != cudaSuccess)
      return set_error(DYLLM_ERR_CUDA, "cudaFuncSetAttribute(%u bytes of shared memory) failed: %s", kPgSmem,
                       cudaGetErrorString(cudaGetLastError()));
    smem_set[dev].store(true, std::memory_order_release);
  }
  launch_pdl_cluster(kernel, dim3(2 * pairs), dim3(kPgThreads), kPgSmem, stream, 2, t[0], t[1], t[2], t[3], t[4], t[5], p);
  return check_launch("pair_gemm");
}

}  // namespace

// `a` holds a_rows rows of pitch lda (p.M dense rows, or the rows that p.row_tiles list); `w` holds w_total_rows rows
// of p.K.  p.status_word, p.tickets and p.launch_id are filled in here.
int launch_pair_gemm(bool swiglu, const PairGemmParams& p_in, const void* a, int a_rows, int64_t lda, const void* w,
                     int64_t w_total_rows, cudaStream_t stream) {
  PairGemmParams p = p_in;
  DYLLM_REQUIRE(p.K > 0 && p.K % 64 == 0, DYLLM_ERR_UNSUPPORTED, "gemm: K = %d is not a multiple of 64", p.K);
  DYLLM_REQUIRE(p.n > 0 && p.n % 64 == 0, DYLLM_ERR_UNSUPPORTED, "gemm: N = %d is not a multiple of 64", p.n);
  DYLLM_REQUIRE(lda % 8 == 0 && p.ldc % 8 == 0 && p.ldc2 % 8 == 0, DYLLM_ERR_UNSUPPORTED,
                "gemm: row pitches must be multiples of 8");
  DYLLM_REQUIRE((reinterpret_cast<uintptr_t>(a) & 15) == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0 &&
                    (reinterpret_cast<uintptr_t>(p.out) & 15) == 0 && (reinterpret_cast<uintptr_t>(p.out2) & 15) == 0,
                DYLLM_ERR_INVALID_ARGUMENT, "gemm: operands must be 16-byte aligned");
  DYLLM_REQUIRE(!p.out2 || (p.split_col > 0 && p.split_col % 128 == 0 && p.split_col < p.n), DYLLM_ERR_INVALID_ARGUMENT,
                "gemm: split column %d must be a multiple of 128 inside (0, %d)", p.split_col, p.n);
  if (p.M <= 0 && !p.row_tiles)
    return DYLLM_OK;
  int pairs = sm_count() / 2;
  pairs = pairs < 1 ? 1 : (pairs > kPgMaxPairs ? kPgMaxPairs : pairs);
  p.status_word = device_status_word();
  // a cut launch has at most 2 * pairs tiles (each part of a tile is a piece of work, and tiles are only made smaller while
  // the pieces do not fill the pairs): two words for each fit
  static_assert(4 * kPgMaxPairs <= kTicketCount, "arrival counters of the cut tiles");
  if (p.partial) {
    p.tickets = reinterpret_cast<unsigned long long*>(reinterpret_cast<uint8_t*>(p.partial) - kTicketBytes);
    p.launch_id = next_launch_id();
  }
  // boxes of one k step (64 columns) and, as 3-D boxes [k step][row][column], of two
  CUtensorMap t[6];
  int rc = encode_tmap_2d_bf16(&t[0], w, w_total_rows, p.K, p.K, 128, 64, true);
  if (rc == DYLLM_OK)
    rc = encode_tmap_2d_bf16(&t[1], a, a_rows, p.K, lda, 32, 64, true);
  if (rc == DYLLM_OK)
    rc = encode_tmap_3d_bf16(&t[2], w, 64, w_total_rows, p.K / 64, static_cast<uint64_t>(p.K) * 2, 128, 64, 128, 2, true);
  if (rc == DYLLM_OK)
    rc = encode_tmap_3d_bf16(&t[3], a, 64, a_rows, p.K / 64, static_cast<uint64_t>(lda) * 2, 128, 64, 32, 2, true);
  if (rc == DYLLM_OK)
    rc = encode_tmap_3d_bf16(&t[4], a, 64, a_rows, p.K / 64, static_cast<uint64_t>(lda) * 2, 128, 64, 64, 2, true);
  t[5] = t[0];
  if (rc == DYLLM_OK && swiglu)
    rc = encode_tmap_2d_bf16(&t[5], w, w_total_rows, p.K, p.K, 64, 64, true);
  if (rc != DYLLM_OK)
    return rc;
  return swiglu ? launch<true>(t, p, pairs, stream) : launch<false>(t, p, pairs, stream);
}

}  // namespace dyllm
