// In-place x passes with a runtime plan (any length of hqt_lineplan.h)
#include "hqt_line_impl.cuh"

namespace hqt {
using LRt = LineLaunch<double, RGeo, RGeo>;
cudaError_t line_rt_init_x(int max_smem) { return LRt::init_x(max_smem); }
cudaError_t line_rt_launch_x(int kind, const void *args, cudaStream_t s) {
    return LRt::launch_x(kind, args, s);
}
}  // namespace hqt
