// Which tile a product takes: see gemm_tiles.cuh for the kernel.
#include "gemm_persistent.cuh"
#include "gemm_tiles.cuh"

namespace mccl {
namespace ops {

namespace tiles {
#define MCCL_TILES_EXTERN(A, B, OUT)                                                                        \
  extern template cudaError_t launch_tiles<64, false, A, B, OUT>(const GemmArgs&, int, int, cudaStream_t);  \
  extern template cudaError_t launch_tiles<128, false, A, B, OUT>(const GemmArgs&, int, int, cudaStream_t);
#define MCCL_TILES_EXTERN_PAIR(A, B, OUT)                                                                   \
  MCCL_TILES_EXTERN(A, B, OUT)                                                                              \
  extern template cudaError_t launch_tiles<256, true, A, B, OUT>(const GemmArgs&, int, int, cudaStream_t);  \
  extern template int max_pairs<256, A, B, OUT>();
MCCL_TILES_EXTERN(false, false, OUT_GELU)
MCCL_TILES_EXTERN_PAIR(false, false, OUT_BF16)
MCCL_TILES_EXTERN_PAIR(false, false, OUT_F32)
MCCL_TILES_EXTERN_PAIR(false, true, OUT_BF16)
MCCL_TILES_EXTERN_PAIR(false, true, OUT_F32)
MCCL_TILES_EXTERN_PAIR(true, false, OUT_BF16)
MCCL_TILES_EXTERN_PAIR(true, false, OUT_F32)
MCCL_TILES_EXTERN_PAIR(true, true, OUT_BF16)
MCCL_TILES_EXTERN_PAIR(true, true, OUT_F32)
#undef MCCL_TILES_EXTERN
#undef MCCL_TILES_EXTERN_PAIR

namespace {

struct Plan {
  int bn = 0;         // 64, 128 (one CTA) or 256 (CTA pair)
  int workers = 0;
  int splits = 1;
};

constexpr int ceil_div(int a, int b) { return (a + b - 1) / b; }

// Clocks of a product on one kind of tile.  Fitted to graphs of back-to-back launches (70M to 1.3B shapes):
// per 64 of K a 128 x 64 tile takes 260 clocks, a 128 x 128 tile 350 and a 256 x 256 pair tile 515; an epilogue 1500 /
// 2000 / 4000, hidden behind the next tile's main loop when there is one; launch and set-up 3500, a pair's two cluster
// barriers 2000 more.
double cost(int bn, int m, int n, int k, int workers, int splits, bool gelu) {
  const bool pair = bn == 256;
  const int tiles = ceil_div(m, pair ? 256 : 128) * ceil_div(n, bn) * splits;
  const int rounds = ceil_div(tiles, workers);
  const double per64 = pair ? 515 : (bn == 128 ? 350 : 260);
  double epilogue = pair ? 4000 : (bn == 128 ? 2000 : 1500);
  if (gelu) epilogue *= 2.5;
  const double main_loop = per64 * ceil_div(k, 64) / splits;
  const double round = main_loop > epilogue ? main_loop : epilogue;
  return 3500 + (pair ? 2000 : 0) + (rounds - 1) * round + main_loop + epilogue + (splits > 1 ? 1500 : 0);
}

Plan choose(const GemmArgs& a, int forced, int sms, int pairs, bool gelu, bool splittable) {
  Plan best;
  double best_cost = 0;
  for (int bn : {64, 128, 256}) {
    if (forced ? bn != forced : false) continue;
    if (bn == 256 && (gelu || pairs < 1)) continue;
    const int workers = bn == 256 ? pairs : sms;
    const int tiles = ceil_div(a.m, bn == 256 ? 256 : 128) * ceil_div(a.n, bn);
    const int num_kb = ceil_div(a.k, 64);
    for (int s = 1; s <= 16; s = s < 4 ? s + 1 : s + 2) {
      if (s > 1 && (!splittable || num_kb / s < 4 || tiles * (s - 1) >= 2 * workers)) break;
      const double c = cost(bn, a.m, a.n, a.k, workers, s, gelu);
      if (best.bn == 0 || c < best_cost) {
        best_cost = c;
        best.bn = bn;
        best.splits = s;
        best.workers = tiles * s < workers ? tiles * s : workers;
      }
    }
  }
  return best;
}

template <bool kAMn, bool kBMn, int kOut>
cudaError_t run(const GemmArgs& a, int forced, cudaStream_t stream) {
  int sms = gemm_sm_count(), pairs = kOut == OUT_GELU ? 0 : 1;
  if constexpr (kOut != OUT_GELU) pairs = max_pairs<256, kAMn, kBMn, kOut>();
  const int limit = gemm_cta_limit();
  if (limit > 0) {
    if (limit < sms) sms = limit;
    if (limit / 2 < pairs) pairs = limit / 2;
  }
  const bool splittable = kOut == OUT_F32 && (a.accumulate || a.ldd == a.n);
  const Plan p = choose(a, forced, sms, pairs, kOut == OUT_GELU, splittable);
  if (p.bn == 64) return launch_tiles<64, false, kAMn, kBMn, kOut>(a, p.workers, p.splits, stream);
  if constexpr (kOut != OUT_GELU)
    if (p.bn == 256) return launch_tiles<256, true, kAMn, kBMn, kOut>(a, p.workers, p.splits, stream);
  return launch_tiles<128, false, kAMn, kBMn, kOut>(a, p.workers, p.splits, stream);
}

template <int kOut>
cudaError_t run_majors(const GemmArgs& a, int forced, cudaStream_t stream) {
  if (a.a_mn_major) return a.b_mn_major ? run<true, true, kOut>(a, forced, stream) : run<true, false, kOut>(a, forced, stream);
  return a.b_mn_major ? run<false, true, kOut>(a, forced, stream) : run<false, false, kOut>(a, forced, stream);
}

}  // namespace
}  // namespace tiles

cudaError_t launch_gemm_tiles(const GemmArgs& a, int forced_bn, cudaStream_t stream) {
  const bool gelu = a.epilogue == EPI_BIAS_GELU || a.epilogue == EPI_GELU || a.epilogue == EPI_BIAS_GELU_D || a.epilogue == EPI_GELU_D;
  // What the kernel does not combine takes the one-CTA persistent kernel: two extra inputs, an activation with one or
  // over an MN-major operand, a bias or an extra input with an fp32 output, a bias that is not 16-byte aligned.
  if ((a.mul && a.residual) || (gelu && (a.mul || a.residual || a.a_mn_major || a.b_mn_major)) ||
      (a.d_fp32 && (a.epilogue != EPI_NONE || a.residual)) || (a.bias && (reinterpret_cast<uintptr_t>(a.bias) & 15)))
    return launch_gemm_persistent(a, FusedDev{}, 0, stream);
  (void)cudaGetLastError();   // a stale error of an earlier, unrelated call must not be blamed on this launch
  if (gelu) return tiles::run<false, false, tiles::OUT_GELU>(a, forced_bn == 256 ? 128 : forced_bn, stream);
  if (a.d_fp32) return tiles::run_majors<tiles::OUT_F32>(a, forced_bn, stream);
  return tiles::run_majors<tiles::OUT_BF16>(a, forced_bn, stream);
}

}  // namespace ops
}  // namespace mccl
