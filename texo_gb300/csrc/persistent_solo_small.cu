// persistent_solo_small.cu — k_persistent with small DCT tiles: one placement on every
// co-resident block of the GPU.
#include "persistent_body.cuh"

namespace tgp {

__global__ void __launch_bounds__(2 * kThreads, kBlocksPerSm) k_persistent_small(const __grid_constant__ InstDesc desc) {
  extern __shared__ __align__(16) unsigned char resident[];
  copy_words(&loop_state<2>().inst, &desc);
  __syncthreads();
  run_body<false, 2>((int)blockIdx.x, (int)gridDim.x, reinterpret_cast<Resident*>(resident));
}

size_t persistent_shared() { return sizeof(Resident); }
const void* persistent_kernel_small() { return (const void*)k_persistent_small; }

}  // namespace tgp
