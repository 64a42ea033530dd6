// Instantiations of the GEMM kernel: both operands MN-major (weight gradients).
#include "gemm_tiles.cuh"

namespace mccl {
namespace ops {
namespace tiles {

template cudaError_t launch_tiles<64, false, true, true, OUT_BF16, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<128, false, true, true, OUT_BF16, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<192, false, true, true, OUT_BF16, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<256, true, true, true, OUT_BF16, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template int max_pairs<256, true, true, OUT_BF16, 1>();
template cudaError_t launch_tiles<64, false, true, true, OUT_F32, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<128, false, true, true, OUT_F32, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<192, false, true, true, OUT_F32, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<256, true, true, true, OUT_F32, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template int max_pairs<256, true, true, OUT_F32, 1>();
template cudaError_t launch_tiles<64, false, true, true, OUT_F32_SCALED, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<128, false, true, true, OUT_F32_SCALED, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<192, false, true, true, OUT_F32_SCALED, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<256, true, true, true, OUT_F32_SCALED, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template int max_pairs<256, true, true, OUT_F32_SCALED, 1>();
template cudaError_t launch_tiles<64, false, true, true, OUT_F32, kMaxGroup>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<128, false, true, true, OUT_F32, kMaxGroup>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<192, false, true, true, OUT_F32, kMaxGroup>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<256, true, true, true, OUT_F32, kMaxGroup>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template int max_pairs<256, true, true, OUT_F32, kMaxGroup>();

}  // namespace tiles
}  // namespace ops
}  // namespace mccl
