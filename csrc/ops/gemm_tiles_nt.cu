// Instantiations of the GEMM kernel: K-major operands (forward products).
#include "gemm_tiles.cuh"

namespace mccl {
namespace ops {
namespace tiles {

template cudaError_t launch_tiles<64, false, false, false, OUT_BF16, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<128, false, false, false, OUT_BF16, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<192, false, false, false, OUT_BF16, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<256, true, false, false, OUT_BF16, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template int max_pairs<256, false, false, OUT_BF16, 1>();
template cudaError_t launch_tiles<64, false, false, false, OUT_F32, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<128, false, false, false, OUT_F32, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<192, false, false, false, OUT_F32, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<256, true, false, false, OUT_F32, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template int max_pairs<256, false, false, OUT_F32, 1>();
template cudaError_t launch_tiles<64, false, false, false, OUT_F32_SLABS, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<128, false, false, false, OUT_F32_SLABS, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<192, false, false, false, OUT_F32_SLABS, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<256, true, false, false, OUT_F32_SLABS, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template int max_pairs<256, false, false, OUT_F32_SLABS, 1>();
template cudaError_t launch_tiles<256, true, false, false, OUT_SWIGLU, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template int max_pairs<256, false, false, OUT_SWIGLU, 1>();
template cudaError_t launch_tiles<64, false, false, false, OUT_GELU, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);
template cudaError_t launch_tiles<128, false, false, false, OUT_GELU, 1>(const GemmArgs*, int, int, int, cudaStream_t, const PartSums*);

}  // namespace tiles
}  // namespace ops
}  // namespace mccl
