// In-place y passes with a runtime plan (any length of hqt_lineplan.h)
#include "hqt_line_impl.cuh"

namespace hqt {
using LRt = LineLaunch<double, RGeo, RGeo>;
cudaError_t line_rt_init_y(int max_smem) { return LRt::init_y(max_smem); }
cudaError_t line_rt_launch_y(int kind, const void *args, int nsl, cudaStream_t s) {
    return LRt::launch_y(kind, args, nsl, s);
}
}  // namespace hqt
