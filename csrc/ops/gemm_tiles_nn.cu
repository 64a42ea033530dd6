// Instantiations of the GEMM kernel: one operand MN-major (input gradients).
#include "gemm_tiles.cuh"

namespace mccl {
namespace ops {
namespace tiles {

template cudaError_t launch_tiles<64, false, false, true, OUT_BF16, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<128, false, false, true, OUT_BF16, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<192, false, false, true, OUT_BF16, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<256, true, false, true, OUT_BF16, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template int max_pairs<256, false, true, OUT_BF16, 1>();
template cudaError_t launch_tiles<64, false, false, true, OUT_F32, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<128, false, false, true, OUT_F32, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<192, false, false, true, OUT_F32, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<256, true, false, true, OUT_F32, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template int max_pairs<256, false, true, OUT_F32, 1>();
template cudaError_t launch_tiles<64, false, false, true, OUT_BF16_SUM, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<128, false, false, true, OUT_BF16_SUM, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<192, false, false, true, OUT_BF16_SUM, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<256, true, false, true, OUT_BF16_SUM, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template int max_pairs<256, false, true, OUT_BF16_SUM, 1>();
template cudaError_t launch_tiles<64, false, false, true, OUT_BF16_PARTS, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<128, false, false, true, OUT_BF16_PARTS, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<192, false, false, true, OUT_BF16_PARTS, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<256, true, false, true, OUT_BF16_PARTS, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template int max_pairs<256, false, true, OUT_BF16_PARTS, 1>();
template cudaError_t launch_tiles<64, false, false, true, OUT_BF16_SCALED, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<128, false, false, true, OUT_BF16_SCALED, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<192, false, false, true, OUT_BF16_SCALED, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<256, true, false, true, OUT_BF16_SCALED, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template int max_pairs<256, false, true, OUT_BF16_SCALED, 1>();
template cudaError_t launch_tiles<64, false, false, true, OUT_F32_SLABS, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<128, false, false, true, OUT_F32_SLABS, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<192, false, false, true, OUT_F32_SLABS, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<256, true, false, true, OUT_F32_SLABS, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template int max_pairs<256, false, true, OUT_F32_SLABS, 1>();
template cudaError_t launch_tiles<64, false, true, false, OUT_BF16, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<128, false, true, false, OUT_BF16, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<192, false, true, false, OUT_BF16, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<256, true, true, false, OUT_BF16, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template int max_pairs<256, true, false, OUT_BF16, 1>();
template cudaError_t launch_tiles<64, false, true, false, OUT_F32, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<128, false, true, false, OUT_F32, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<192, false, true, false, OUT_F32, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<256, true, true, false, OUT_F32, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template int max_pairs<256, true, false, OUT_F32, 1>();

template cudaError_t launch_tiles<256, true, false, true, OUT_SWIGLU_GRAD, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template int max_pairs<256, false, true, OUT_SWIGLU_GRAD, 1>();

}  // namespace tiles
}  // namespace ops
}  // namespace mccl
