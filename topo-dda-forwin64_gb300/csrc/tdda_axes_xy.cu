// tdda_axes_xy.cu -- the x and y kernels of the x-first A-product for one FFT
// length, TDDA_AXIS; build.py compiles this file once per length of TDDA_XY_AXES
// (tdda_internal.cuh), which keeps the build parallel.
#include "tdda_axes.cuh"

namespace tdda {

#define TDDA_CAT2(a, b) a##b
#define TDDA_CAT(a, b) TDDA_CAT2(a, b)

cudaError_t TDDA_CAT(axis_f32_, TDDA_AXIS)(int op, int mode, int rows, const PassArgs<float>& a) {
    return dev::AxisLaunch<float, TDDA_AXIS>::run(op, mode, rows, a);
}
cudaError_t TDDA_CAT(axis_f64_, TDDA_AXIS)(int op, int mode, int rows, const PassArgs<double>& a) {
    return dev::AxisLaunch<double, TDDA_AXIS>::run(op, mode, rows, a);
}
#if TDDA_AXIS == 40 || TDDA_AXIS == 128 || TDDA_AXIS == 160 || TDDA_AXIS == 192
cudaError_t TDDA_CAT(axis_dd_, TDDA_AXIS)(int op, int mode, int rows, const PassArgs<dd>& a) {
    return dev::AxisLaunch<dd, TDDA_AXIS>::run(op, mode, rows, a);
}
#endif

}  // namespace tdda
