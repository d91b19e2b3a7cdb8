// Pyramid, blur, FAST-9 + Harris score map and NMS for sm_100a.
//
// Each launch covers a batch of frames; a block finds its frame through a
// prefix table of tile counts.  Pyramid layout, guards and the score-map
// format follow the reference (orb.cpp:145-191, orbd.cu:1576-1577) so that
// reads that leave an octave see the same bytes the reference sees.
#include "orbx_stages.cuh"

namespace orbx {

// Kernels take the batch as a grid constant so that, for batches whose frame
// table travels in the launch parameters (INL), the stages read it in place.
template <int TH, bool INL>
__global__ void __launch_bounds__(kPyrThreads, 4) k_pyramid_blur(const __grid_constant__ Batch b) {
  __shared__ PyrSmem<TH> sm;
  chain_wait();
  pyr_tile<false, TH, INL>(b, blockIdx.x, sm);
}

template <bool INL>
__global__ void __launch_bounds__(256, 6) k_detect(const __grid_constant__ Batch b) {
  __shared__ DetSmem sm;
  chain_wait();
  det_tile<false, INL>(b, blockIdx.x, sm);
}

template <bool INL>
__global__ void __launch_bounds__(256, 4) k_nms(const __grid_constant__ Batch b) {
  __shared__ NmsSmem sm;
  __shared__ int s_ticket;
  chain_wait();
  if (threadIdx.x == 0) s_ticket = (int)atomicAdd(b.nms_ticket, 1u);
  __syncthreads();
  nms_strip<false, INL>(b, s_ticket, sm);
}

// Dense reference-layout maps (vmem: f32 scores then i32 octaves,
// orbd.cu:1576-1577) from the sparse ones, for orbd.h callers and debugging.
__global__ void k_expand_score_map(const uint32_t* __restrict__ occ, const float* __restrict__ vmap,
                                   const uint8_t* __restrict__ oct8, float* vmap_dense, int* layer_dense,
                                   long long npx) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < npx;
       i += (long long)gridDim.x * blockDim.x) {
    const bool on = (__ldg(occ + (i >> 5)) >> (i & 31)) & 1u;
    vmap_dense[i] = on ? vmap[i] : 0.f;
    layer_dense[i] = on ? (int)oct8[i] : 0;
  }
}

cudaError_t launch_expand_score_map(const uint32_t* occ, const float* vmap, const uint8_t* oct8, float* vmap_dense,
                                    int* layer_dense, long long npx, cudaStream_t s) {
  k_expand_score_map<<<4 * 148, 256, 0, s>>>(occ, vmap, oct8, vmap_dense, layer_dense, npx);
  return cudaGetLastError();
}

cudaError_t launch_pyramid_blur(const Batch& b, int total_tiles, cudaStream_t s) {
  if (total_tiles <= 0) return cudaSuccess;
  const bool inl = b.n_inline > 0;
  auto run = [&](auto* kernel) { return launch_chained(kernel, total_tiles, kPyrThreads, s, b); };
#define PYR_SHAPE(i) (inl ? run(k_pyramid_blur<kPyrShapeTH[i], true>) : run(k_pyramid_blur<kPyrShapeTH[i], false>))
  switch (b.pyr_shape) {
    case 1: return PYR_SHAPE(1);
    case 2: return PYR_SHAPE(2);
    case 3: return PYR_SHAPE(3);
    default: return PYR_SHAPE(0);
  }
#undef PYR_SHAPE
}

cudaError_t launch_detect(const Batch& b, int total_tiles, cudaStream_t s) {
  if (total_tiles <= 0) return cudaSuccess;
  return launch_chained(b.n_inline > 0 ? k_detect<true> : k_detect<false>, total_tiles, 256, s, b);
}

cudaError_t launch_nms(const Batch& b, int total_strips, cudaStream_t s) {
  if (total_strips <= 0) return cudaSuccess;
  return launch_chained(b.n_inline > 0 ? k_nms<true> : k_nms<false>, total_strips, 256, s, b);
}

}  // namespace orbx
