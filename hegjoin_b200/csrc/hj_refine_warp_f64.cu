// hj_refine_warp_f64.cu -- the warp-per-item exact refine for double data.
#include "hj_refine_warp.cuh"

namespace hj {

hj_status refine_warp_f64(const WarpArgs<double>& a, uint32_t d, bool digest, cudaStream_t st) {
    return digest ? dispatch_warp<double, 1, kWarpMaxD64, true>(a, d, st) : dispatch_warp<double, 1, kWarpMaxD64, false>(a, d, st);
}

}  // namespace hj
