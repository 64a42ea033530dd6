// Entry point of the bf16 GEMM: operand checks, kernel selection, and the error word every GEMM kernel shares.
//
// The reference has no GEMM of its own (no tensor-core code at all); these kernels exist for the model operators and
// as the core the fused all-gather→GEMM / GEMM→reduce-scatter tensor-parallel kernels build on.
#include "../core/launch.hpp"
#include "gemm_common.cuh"
#include "gemm_persistent.cuh"

#include <atomic>

#include <cstdlib>
#include <string>

namespace mccl {
namespace ops {

namespace {

thread_local const char* t_reason = "";
cudaError_t unsupported(const char* why) {
  t_reason = why;
  return cudaErrorNotSupported;
}

}  // namespace

namespace {
// The tile kernel with a tile of its choosing (0) or a given one (64, 128, 192, 256), or the one-CTA persistent kernel.
constexpr int kPersistent = -1;
std::atomic<int> g_gemm_kernel_override{-2};
int kernel_index(const std::string& s) {
  if (s == "persistent") return kPersistent;
  if (s == "tile64") return 64;
  if (s == "tile128") return 128;
  if (s == "tile192") return 192;
  if (s == "pair256") return 256;
  return 0;
}
}  // namespace

// A name of the list above ("pair" and "tile" are the default kernel); "" returns to MCCL_GEMM_KERNEL / the default.
void set_gemm_kernel(const std::string& name) {
  g_gemm_kernel_override.store(name.empty() ? -2 : kernel_index(name), std::memory_order_relaxed);
}

int gemm_kernel_choice() {
  static const int env_choice = [] {
    const char* v = std::getenv("MCCL_GEMM_KERNEL");
    return kernel_index(v ? v : "");
  }();
  const int forced = g_gemm_kernel_override.load(std::memory_order_relaxed);
  return forced != -2 ? forced : env_choice;
}

const char* gemm_last_reason() { return t_reason; }

cudaError_t gemm_bf16_tn(const GemmArgs& a, cudaStream_t stream) {
  t_reason = "";
  if (a.m <= 0 || a.n <= 0 || a.k <= 0) return cudaErrorInvalidValue;
  // (a contraction may end anywhere: the tile kernel's loads are zero past it)
  if (a.n % 8 != 0) return unsupported("N must be a multiple of 8");
  if (a.lda % 8 != 0 || a.ldb % 8 != 0 || a.ldd % (a.d_fp32 ? 4 : 8) != 0)
    return unsupported("row strides must keep rows 16-byte aligned");
  if ((reinterpret_cast<uintptr_t>(a.a) | reinterpret_cast<uintptr_t>(a.b) | reinterpret_cast<uintptr_t>(a.d)) & 15u)
    return unsupported("operand pointers must be 16-byte aligned");
  if (a.aux && (reinterpret_cast<uintptr_t>(a.aux) & 15u)) return unsupported("aux pointer must be 16-byte aligned");
  if ((a.epilogue == EPI_BIAS || a.epilogue == EPI_BIAS_GELU || a.epilogue == EPI_BIAS_GELU_D) && !a.bias) return cudaErrorInvalidValue;
  if ((a.epilogue == EPI_BIAS_GELU || a.epilogue == EPI_GELU || a.epilogue == EPI_BIAS_GELU_D || a.epilogue == EPI_GELU_D) &&
      a.d_fp32)
    return cudaErrorInvalidValue;
  if (a.accumulate && !a.d_fp32) return cudaErrorInvalidValue;
  if (a.residual && (reinterpret_cast<uintptr_t>(a.residual) & 15u)) return unsupported("residual pointer must be 16-byte aligned");
  if (a.mul && ((reinterpret_cast<uintptr_t>(a.mul) & 15u) || a.d_fp32)) return unsupported("mul must be 16-byte aligned and the output bf16");
  if (a.a_mn_major && a.m % 8 != 0) return unsupported("an MN-major A needs M to be a multiple of 8");
  const int choice = gemm_kernel_choice();
  const bool gelu = a.epilogue == EPI_BIAS_GELU || a.epilogue == EPI_GELU || a.epilogue == EPI_BIAS_GELU_D || a.epilogue == EPI_GELU_D;
  if (a.alpha && (gelu || a.bias || a.residual || a.mul || a.colsum)) return cudaErrorInvalidValue;
  const bool tile_only = a.k % BK != 0 || a.colsum || a.alpha || (gelu && !a.aux);   // what only the tile kernel does
  cudaError_t rc = choice == kPersistent && !tile_only ? launch_gemm_persistent(a, FusedDev{}, 0, stream)
                                                         : launch_gemm_tiles(a, choice > 0 ? choice : 0, stream);
  if (rc == cudaErrorNotSupported) return unsupported("cuTensorMapEncodeTiled rejected an operand");
  return rc;
}

namespace {
__device__ int g_gemm_error = 0;
}

int* gemm_error_device_ptr() {
  static int* ptr = nullptr;
  if (!ptr) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_gemm_error) == cudaSuccess) ptr = static_cast<int*>(p);
  }
  return ptr;
}

int gemm_error_flag() {
  int v = 0;
  cudaMemcpyFromSymbol(&v, g_gemm_error, sizeof(int));
  return v;
}

}  // namespace ops
}  // namespace mccl
