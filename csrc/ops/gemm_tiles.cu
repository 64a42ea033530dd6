// Which tile a product takes: see gemm_tiles.cuh for the kernel.
#include "gemm_persistent.cuh"
#include "gemm_tiles.cuh"

namespace mccl {
namespace ops {

namespace tiles {
#define MCCL_TILES_EXTERN(A, B, OUT, MAX)                                                                                     \
  extern template cudaError_t launch_tiles<64, false, A, B, OUT, MAX>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);   \
  extern template cudaError_t launch_tiles<128, false, A, B, OUT, MAX>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
#define MCCL_TILES_EXTERN_PAIR(A, B, OUT, MAX)                                                                                \
  MCCL_TILES_EXTERN(A, B, OUT, MAX)                                                                                           \
  extern template cudaError_t launch_tiles<192, false, A, B, OUT, MAX>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);   \
  extern template cudaError_t launch_tiles<256, true, A, B, OUT, MAX>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);   \
  extern template int max_pairs<256, A, B, OUT, MAX>();
MCCL_TILES_EXTERN(false, false, OUT_GELU, 1)
MCCL_TILES_EXTERN_PAIR(false, false, OUT_BF16, 1)
MCCL_TILES_EXTERN_PAIR(false, false, OUT_F32, 1)
MCCL_TILES_EXTERN_PAIR(false, true, OUT_BF16, 1)
MCCL_TILES_EXTERN_PAIR(false, true, OUT_BF16_SUM, 1)
MCCL_TILES_EXTERN_PAIR(false, true, OUT_BF16_PARTS, 1)
MCCL_TILES_EXTERN_PAIR(false, true, OUT_BF16_SCALED, 1)
MCCL_TILES_EXTERN_PAIR(false, false, OUT_F32_SLABS, 1)
MCCL_TILES_EXTERN_PAIR(false, true, OUT_F32_SLABS, 1)
MCCL_TILES_EXTERN_PAIR(true, true, OUT_F32_SCALED, 1)
MCCL_TILES_EXTERN_PAIR(false, true, OUT_F32, 1)
MCCL_TILES_EXTERN_PAIR(true, false, OUT_BF16, 1)
MCCL_TILES_EXTERN_PAIR(true, false, OUT_F32, 1)
MCCL_TILES_EXTERN_PAIR(true, true, OUT_BF16, 1)
MCCL_TILES_EXTERN_PAIR(true, true, OUT_F32, 1)
MCCL_TILES_EXTERN_PAIR(true, true, OUT_F32, kMaxGroup)
extern template cudaError_t launch_tiles<256, true, false, false, OUT_SWIGLU, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
extern template int max_pairs<256, false, false, OUT_SWIGLU, 1>();
extern template cudaError_t launch_tiles<256, true, false, true, OUT_SWIGLU_GRAD, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
extern template int max_pairs<256, false, true, OUT_SWIGLU_GRAD, 1>();
#undef MCCL_TILES_EXTERN
#undef MCCL_TILES_EXTERN_PAIR

namespace {

struct Plan {
  int bn = 0;         // 64, 128, 192 (one CTA) or 256 (CTA pair)
  int workers = 0;
  int splits = 1;
};

constexpr double kRunsBytes = 80e6;   // of 126 MB of L2, which also holds the output
constexpr int ceil_div(int a, int b) { return (a + b - 1) / b; }

// Clocks of a product on one kind of tile, fitted to graphs of back-to-back launches (70M to 1.3B shapes) and the kernel's
// timeline: per 64 of K a 128 x 64 tile takes 260 clocks, a 128 x 128 tile 350, a 128 x 192 tile 520 and a 256 x 256
// pair tile 515 (its MMAs need 512); an epilogue 1500 / 2000 / 2500 / 3000, fp32 sums added into memory 1800 / 2600 / 3900 / 7000, hidden behind the next tile's
// main loop when there is one; launch and set-up 3500, a pair's two cluster barriers 2000 more.
constexpr double kPer64[4] = {260, 350, 520, 515}, kEpilogue[4] = {1500, 2000, 2500, 3000}, kAdding[4] = {1800, 2600, 3900, 7000};
int kind_of(int bn) { return bn / 64 - 1; }

double cost(int bn, int tiles, int k, int workers, int splits, bool gelu, bool adding) {
  const int kind = kind_of(bn);
  const int rounds = ceil_div(tiles * splits, workers);
  double epilogue = adding ? kAdding[kind] : kEpilogue[kind];
  if (gelu) epilogue *= 2.5;
  const double main_loop = kPer64[kind] * ceil_div(k, 64) / splits;
  const double round = main_loop > epilogue ? main_loop : epilogue;
  return 3500 + (kind == 3 ? 2000 : 0) + (rounds - 1) * round + main_loop + epilogue;
}

Plan choose(const GemmArgs* args, int count, int forced, int sms, int pairs, bool gelu, bool splittable, bool slabs = false) {
  Plan best;
  double best_cost = 0;
  const int k = args[0].k;
  double operand_bytes = 0;
  for (int p = 0; p < count; ++p) operand_bytes += 2.0 * k * (static_cast<double>(args[p].m) + args[p].n);
  for (int bn : {64, 128, 192, 256}) {
    if (forced ? bn != forced : false) continue;
    if ((bn == 256 && (gelu || pairs < 1)) || (bn == 192 && gelu)) continue;
    const int workers = bn == 256 ? pairs : sms;
    int tiles = 0;
    for (int p = 0; p < count; ++p) tiles += ceil_div(args[p].m, bn == 256 ? 256 : 128) * ceil_div(args[p].n, bn);
    const int num_kb = ceil_div(k, 64);
    if (splittable && !slabs && operand_bytes < kRunsBytes && static_cast<long long>(tiles) * num_kb >= 8ll * workers) {
      // Equal runs of k-blocks for every worker: no last round that leaves SMs idle, at the price of up to two more partial
      // tiles per worker.  Workers are then at different places of K, so operands that do not stay in L2 are read several
      // times (the 262 MB of an LM head's gradient: 4096 x 512 x 32000 131 us against 123).
      const double run = kPer64[kind_of(bn)] * (static_cast<double>(tiles) * num_kb / workers);
      const double c = 3500 + (bn == 256 ? 2000 : 0) + run + 1.5 * kAdding[kind_of(bn)];
      if (best.bn == 0 || c < best_cost) {
        best_cost = c;
        best.bn = bn;
        best.splits = 0;
        best.workers = workers;
      }
    }
    for (int s = 1; s <= 16; s = s < 4 ? s + 1 : s + 2) {
      if (s > 1 && (!splittable || num_kb / s < 4 || tiles * (s - 1) >= 2 * workers)) break;
      const double c = cost(bn, tiles, k, workers, s, gelu, splittable && (s > 1 || args[0].accumulate));
      if (best.bn == 0 || c < best_cost) {
        best_cost = c;
        best.bn = bn;
        best.splits = s;
        best.workers = tiles * s < workers ? tiles * s : workers;
      }
    }
  }
  // a tile that was asked for and cannot run (a pair under a cap of one CTA, a wide tile with GELU): one that can
  if (best.bn == 0 && forced) return choose(args, count, 0, sms, pairs, gelu, splittable, slabs);
  return best;
}

template <bool kAMn, bool kBMn, int kOut, int kMax = 1>
cudaError_t run_plan(const GemmArgs* a, int count, const Plan& plan, cudaStream_t stream, const PartSums* sums = nullptr);

template <bool kAMn, bool kBMn, int kOut, int kMax = 1>
cudaError_t run(const GemmArgs* a, int count, int forced, cudaStream_t stream, const PartSums* sums = nullptr) {
  int sms = gemm_sm_count(), pairs = 0;
  if constexpr (kOut != OUT_GELU) pairs = max_pairs<256, kAMn, kBMn, kOut, kMax>();
  const int limit = gemm_cta_limit();
  if (limit > 0) {
    if (limit < sms) sms = limit;
    if (limit / 2 < pairs) pairs = limit / 2;
  }
  bool splittable = fp32_out(kOut);
  for (int p = 0; p < count; ++p) splittable = splittable && (a[p].accumulate || a[p].ldd == a[p].n);
  return run_plan<kAMn, kBMn, kOut, kMax>(a, count, choose(a, count, forced, sms, pairs, kOut == OUT_GELU, splittable), stream, sums);
}

template <bool kAMn, bool kBMn, int kOut, int kMax>
cudaError_t run_plan(const GemmArgs* a, int count, const Plan& plan, cudaStream_t stream, const PartSums* sums) {
  if (plan.bn == 64) return launch_tiles<64, false, kAMn, kBMn, kOut, kMax>(a, count, plan.workers, plan.splits, stream, sums);
  if constexpr (kOut != OUT_GELU)
    if (plan.bn == 192) return launch_tiles<192, false, kAMn, kBMn, kOut, kMax>(a, count, plan.workers, plan.splits, stream, sums);
  if constexpr (kOut != OUT_GELU)
    if (plan.bn == 256) return launch_tiles<256, true, kAMn, kBMn, kOut, kMax>(a, count, plan.workers, plan.splits, stream, sums);
  return launch_tiles<128, false, kAMn, kBMn, kOut, kMax>(a, count, plan.workers, plan.splits, stream, sums);
}

template <int kOut>
cudaError_t run_majors(const GemmArgs& a, int forced, cudaStream_t stream) {
  if (a.a_mn_major) return a.b_mn_major ? run<true, true, kOut>(&a, 1, forced, stream) : run<true, false, kOut>(&a, 1, forced, stream);
  return a.b_mn_major ? run<false, true, kOut>(&a, 1, forced, stream) : run<false, false, kOut>(&a, 1, forced, stream);
}

}  // namespace
}  // namespace tiles

cudaError_t launch_gemm_tiles(const GemmArgs& a, int forced_bn, cudaStream_t stream) {
  const bool gelu = a.epilogue == EPI_BIAS_GELU || a.epilogue == EPI_GELU || a.epilogue == EPI_BIAS_GELU_D || a.epilogue == EPI_GELU_D;
  // What the kernel does not combine takes the one-CTA persistent kernel: two extra inputs, an activation with one or
  // over an MN-major operand, a bias or an extra input with an fp32 output, a bias that is not 16-byte aligned.
  if ((a.mul && a.residual) || (gelu && (a.mul || a.residual || a.a_mn_major || a.b_mn_major)) ||
      (a.d_fp32 && (a.epilogue != EPI_NONE || a.residual)) || (a.bias && (reinterpret_cast<uintptr_t>(a.bias) & 15)))
    return gelu && !a.aux ? cudaErrorNotSupported : launch_gemm_persistent(a, FusedDev{}, 0, stream);
  (void)cudaGetLastError();   // a stale error of an earlier, unrelated call must not be blamed on this launch
  if (a.colsum) {
    if (gelu || a.d_fp32 || a.bias || a.residual || a.a_mn_major || !a.b_mn_major) return cudaErrorInvalidValue;
    return a.colsum_in_order ? tiles::run<false, true, tiles::OUT_BF16_PARTS>(&a, 1, forced_bn, stream)
                             : tiles::run<false, true, tiles::OUT_BF16_SUM>(&a, 1, forced_bn, stream);
  }
  if (a.alpha) {
    if (a.d_fp32 && a.a_mn_major && a.b_mn_major) return tiles::run<true, true, tiles::OUT_F32_SCALED>(&a, 1, forced_bn, stream);
    if (!a.d_fp32 && !a.a_mn_major && a.b_mn_major) return tiles::run<false, true, tiles::OUT_BF16_SCALED>(&a, 1, forced_bn, stream);
    return cudaErrorInvalidValue;
  }
  if (gelu) return tiles::run<false, false, tiles::OUT_GELU>(&a, 1, forced_bn > 128 ? 128 : forced_bn, stream);
  if (a.d_fp32) return tiles::run_majors<tiles::OUT_F32>(a, forced_bn, stream);
  return tiles::run_majors<tiles::OUT_BF16>(a, forced_bn, stream);
}

// Measured on an LM head's input gradient (K 32000): 32 pair tiles (4096 x 512) 108 against 123 us, 48 (4096 x 768) 145 against
// 152; with 64 tiles (4096 x 1024, K 8192) writing, adding and casting the parts cost more than the idle SMs, 67 against 43.
bool gemm_wants_slabs(const GemmArgs& a) {
  if (a.m <= 0 || a.n <= 0 || a.a_mn_major || a.n % 8 != 0 || a.lda % 8 != 0 || a.ldb % 8 != 0 ||
      ((reinterpret_cast<uintptr_t>(a.a) | reinterpret_cast<uintptr_t>(a.b)) & 15u))
    return false;   // gemm_bf16_tn says why
  return a.k >= 4096 && gemm_kernel_choice() >= 0 && tiles::ceil_div(a.m, 256) * tiles::ceil_div(a.n, 256) * 10 <= gemm_sm_count() / 2 * 7;
}

Slabs gemm_slabs(const GemmArgs& a) {
  int sms = gemm_sm_count();
  int pairs = a.b_mn_major ? tiles::max_pairs<256, false, true, tiles::OUT_F32_SLABS, 1>() : tiles::max_pairs<256, false, false, tiles::OUT_F32_SLABS, 1>();
  const int limit = gemm_cta_limit();
  if (limit > 0) {
    sms = limit < sms ? limit : sms;
    pairs = limit / 2 < pairs ? limit / 2 : pairs;
  }
  const int choice = gemm_kernel_choice();
  const tiles::Plan plan = tiles::choose(&a, 1, choice > 0 ? choice : 0, sms, pairs, false, true, true);
  return {plan.splits, static_cast<long long>((a.m + 31) / 32 * 32) * a.n, plan.bn, plan.workers};
}

cudaError_t gemm_to_slabs(const GemmArgs& a, const Slabs& s, cudaStream_t stream) {
  if (a.m <= 0 || a.n <= 0 || a.k <= 0 || a.a_mn_major || a.bias || a.residual || a.mul || a.colsum || a.alpha || a.accumulate || !a.d_fp32 ||
      a.epilogue != EPI_NONE || a.ldd != a.n || s.count < 1 || s.count > tiles::ceil_div(a.k, BK))
    return cudaErrorInvalidValue;
  if (a.n % 8 != 0 || a.lda % 8 != 0 || a.ldb % 8 != 0 ||
      ((reinterpret_cast<uintptr_t>(a.a) | reinterpret_cast<uintptr_t>(a.b) | reinterpret_cast<uintptr_t>(a.d)) & 15u))
    return cudaErrorNotSupported;
  if (s.workers < 1) return cudaErrorInvalidValue;
  tiles::Plan plan;
  plan.bn = s.tile;
  plan.workers = s.workers;
  plan.splits = s.count;
  (void)cudaGetLastError();
  return a.b_mn_major ? tiles::run_plan<false, true, tiles::OUT_F32_SLABS>(&a, 1, plan, stream) : tiles::run_plan<false, false, tiles::OUT_F32_SLABS>(&a, 1, plan, stream);
}

namespace {
// SwiGLU around a product of n (grad) or 2 n columns, on the pair tile only: where the product alone takes another one, tiles of
// 256 rows would leave SMs idle.
template <bool kBMn, int kOut>
cudaError_t run_swiglu(const GemmArgs& a, cudaStream_t stream) {
  if (a.m <= 0 || a.n <= 0 || a.k <= 0 || a.d_fp32 || a.accumulate || a.bias || a.residual || a.mul || a.colsum || a.a_mn_major || a.b_mn_major != kBMn ||
      a.epilogue != EPI_NONE)
    return cudaErrorInvalidValue;
  if (a.n % 32 != 0 || a.lda % 8 != 0 || a.ldb % 8 != 0 || a.ldd % 8 != 0 ||
      ((reinterpret_cast<uintptr_t>(a.a) | reinterpret_cast<uintptr_t>(a.b) | reinterpret_cast<uintptr_t>(a.d) | reinterpret_cast<uintptr_t>(a.aux)) & 15u))
    return cudaErrorNotSupported;
  int sms = gemm_sm_count(), pairs = tiles::max_pairs<256, false, kBMn, kOut, 1>();
  const int limit = gemm_cta_limit();
  if (limit > 0) {
    sms = limit < sms ? limit : sms;
    pairs = limit / 2 < pairs ? limit / 2 : pairs;
  }
  constexpr int kTileN = kOut == tiles::OUT_SWIGLU ? 128 : 256;
  GemmArgs alone = a;
  alone.n = a.n * (256 / kTileN);
  if (tiles::choose(&alone, 1, 0, sms, pairs, false, false).bn != 256) return cudaErrorNotSupported;
  const int tiles = tiles::ceil_div(a.m, 256) * tiles::ceil_div(a.n, kTileN);
  (void)cudaGetLastError();
  return tiles::launch_tiles<256, true, false, kBMn, kOut, 1>(&a, 1, tiles < pairs ? tiles : pairs, 1, stream, nullptr);
}
}  // namespace

cudaError_t gemm_swiglu(const GemmArgs& a, cudaStream_t stream) { return run_swiglu<false, tiles::OUT_SWIGLU>(a, stream); }
cudaError_t gemm_swiglu_grad(const GemmArgs& a, cudaStream_t stream) {
  return a.aux ? run_swiglu<true, tiles::OUT_SWIGLU_GRAD>(a, stream) : cudaErrorInvalidValue;
}

cudaError_t gemm_group(const GemmArgs* args, int count, cudaStream_t stream, const PartSum* sums, int sum_count) {
  PartSums table;
  if (cudaError_t rc = table.set(sums, sum_count); rc != cudaSuccess) return rc;
  for (int p = 0; p < count; ++p) {
    const GemmArgs& a = args[p];
    if (!a.a_mn_major || !a.b_mn_major || !a.d_fp32 || a.epilogue != EPI_NONE || a.residual || a.mul || a.colsum || a.k != args[0].k ||
        a.accumulate != args[0].accumulate || a.m <= 0 || a.n <= 0 || a.k <= 0)
      return cudaErrorInvalidValue;
    if (a.m % 8 != 0 || a.n % 8 != 0 || a.lda % 8 != 0 || a.ldb % 8 != 0 || a.ldd % 4 != 0 ||
        ((reinterpret_cast<uintptr_t>(a.a) | reinterpret_cast<uintptr_t>(a.b) | reinterpret_cast<uintptr_t>(a.d)) & 15u))
      return cudaErrorNotSupported;
  }
  (void)cudaGetLastError();
  for (int p = 0; p < count; p += tiles::kMaxGroup) {
    const int c = count - p < tiles::kMaxGroup ? count - p : tiles::kMaxGroup;
    cudaError_t rc = tiles::run<true, true, tiles::OUT_F32, tiles::kMaxGroup>(args + p, c, 0, stream, p == 0 && sum_count > 0 ? &table : nullptr);
    if (rc != cudaSuccess) return rc;
  }
  return cudaSuccess;
}

}  // namespace ops
}  // namespace mccl
