// persistent_solo_large.cu — k_persistent with large DCT tiles: one placement on every
// co-resident block of the GPU.
#include "persistent_body.cuh"

namespace tgp {

__global__ void __launch_bounds__(2 * kThreads, kBlocksPerSm) k_persistent_large(const __grid_constant__ InstDesc desc) {
  extern __shared__ __align__(16) unsigned char resident[];
  copy_words(&loop_state<2>().inst, &desc);
  __syncthreads();
  run_body<true, 2>((int)blockIdx.x, (int)gridDim.x, reinterpret_cast<Resident*>(resident));
}

const void* persistent_kernel_large() { return (const void*)k_persistent_large; }

}  // namespace tgp
