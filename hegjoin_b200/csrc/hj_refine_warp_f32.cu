// hj_refine_warp_f32.cu -- the warp-per-item exact refine for float data.
#include "hj_refine_warp.cuh"

namespace hj {

hj_status refine_warp_f32(const WarpArgs<float>& a, uint32_t d, bool digest, cudaStream_t st) {
    return digest ? dispatch_warp<float, 1, kWarpMaxD32, true>(a, d, st) : dispatch_warp<float, 1, kWarpMaxD32, false>(a, d, st);
}

}  // namespace hj
