// wf_grid.h — grids of the persistent kernels: every block resident at once.
#pragma once
#include <cuda_runtime.h>

namespace wf {

int sm_count();

// Blocks of a grid that fills the GPU with Kernel.  The occupancy is asked for
// once per kernel: instantiations of one template have one type, but registers
// (and so resident blocks: 9 per SM for the binary BLAS layout, 8 for the 4-wide
// ones) of their own, and a block that is not resident holds first rays that
// start only once another block has ended (1M incoherent rays, quantized / exact
// 4-wide: 1,428 / 1,508 us, 1,544 / 1,642 on the binary kernels' grid).
template <auto Kernel, int Block>
inline unsigned persistent_grid() {
    static const int per_sm = [] {
        int n = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, reinterpret_cast<const void*>(Kernel), Block, 0);
        return n > 0 ? n : 1;
    }();
    return (unsigned)(sm_count() * per_sm);
}

}  // namespace wf
