// tdda_axes.cu -- dispatch of the x-first A-product (tdda_axes.cuh) and its z
// kernels; the x, y and plane kernels are compiled per length in
// tdda_axes_xy.cu and tdda_axes_plane.cu.
#include "tdda_axes.cuh"

namespace tdda {

#define TDDA_X(M)                                                                     \
    cudaError_t axis_f32_##M(int op, int mode, int rows, const PassArgs<float>& a);   \
    cudaError_t axis_f64_##M(int op, int mode, int rows, const PassArgs<double>& a);
TDDA_XY_AXES(TDDA_X)
#undef TDDA_X
#define TDDA_X(M) cudaError_t axis_dd_##M(int op, int mode, int rows, const PassArgs<dd>& a);
TDDA_X(40) TDDA_X(128) TDDA_X(160) TDDA_X(192)
#undef TDDA_X
#define TDDA_X(M)                                             \
    cudaError_t plane_##M(int Mz, const PassArgs<float>* a);  \
    bool plane_has_##M(int Mz);
TDDA_PLANE_Y(TDDA_X)
#undef TDDA_X

namespace {
cudaError_t axis_run(int M, int op, int mode, int rows, const PassArgs<float>& a) {
    switch (M) {
#define TDDA_X(L) case L: return axis_f32_##L(op, mode, rows, a);
        TDDA_XY_AXES(TDDA_X)
#undef TDDA_X
        default: return cudaErrorInvalidValue;
    }
}
cudaError_t axis_run(int M, int op, int mode, int rows, const PassArgs<double>& a) {
    switch (M) {
#define TDDA_X(L) case L: return axis_f64_##L(op, mode, rows, a);
        TDDA_XY_AXES(TDDA_X)
#undef TDDA_X
        default: return cudaErrorInvalidValue;
    }
}
cudaError_t axis_run(int M, int op, int mode, int rows, const PassArgs<dd>& a) {
    switch (M) {
#define TDDA_X(L) case L: return axis_dd_##L(op, mode, rows, a);
        TDDA_X(40) TDDA_X(128) TDDA_X(160) TDDA_X(192)
#undef TDDA_X
        default: return cudaErrorInvalidValue;
    }
}
template <typename T> cudaError_t zprod_run(const PassArgs<T>& a) {
    switch (a.g.pz.M) {
#define TDDA_X(L) case L: return dev::ZprodLaunch<T, L>::run(a);
        TDDA_Z_AXES(TDDA_X)
#undef TDDA_X
        default: return cudaErrorInvalidValue;
    }
}
template <> cudaError_t zprod_run<dd>(const PassArgs<dd>& a) {
    switch (a.g.pz.M) {
#define TDDA_X(L) case L: return dev::ZprodLaunch<dd, L>::run(a);
        TDDA_X(20) TDDA_X(32) TDDA_X(40) TDDA_X(48)
#undef TDDA_X
        default: return cudaErrorInvalidValue;
    }
}
bool xy_axis(int M) {
    switch (M) {
#define TDDA_X(L) case L:
        TDDA_XY_AXES(TDDA_X)
#undef TDDA_X
        return true;
        default: return false;
    }
}
bool z_axis(int M) {
    switch (M) {
#define TDDA_X(L) case L:
        TDDA_Z_AXES(TDDA_X)
#undef TDDA_X
        return true;
        default: return false;
    }
}
bool dd_xy(int M) { return M == 40 || M == 128 || M == 160 || M == 192; }
bool dd_z(int M) { return M == 20 || M == 32 || M == 40 || M == 48; }
}  // namespace

bool axes_lengths(const Geom& g) { return xy_axis(g.px.M) && xy_axis(g.py.M) && z_axis(g.pz.M); }
bool dd_lengths(const Geom& g) { return dd_z(g.pz.M) && dd_xy(g.py.M) && dd_xy(g.px.M); }
bool axes_plane(const Geom& g) {
    switch (g.py.M) {
#define TDDA_X(L) case L: return plane_has_##L(g.pz.M);
        TDDA_PLANE_Y(TDDA_X)
#undef TDDA_X
        default: return false;
    }
}
// Lines per block.  A gather changes nothing but the block that transforms a
// line; a sink's block sums are the partials of the solver's dots, so its tile
// depends on the FFT lengths alone and every lattice of a grid shape forms them
// alike, alone or in a cross-lattice batch.  16 lines where that gives every SM
// a block, else 8.
int axis_tile_fwd(const Geom& g) { return g.x_tile ? g.x_tile : axis_tile_inv(g); }
int axis_tile_inv(const Geom& g) {
    const long long cells = (long long)((g.py.M + 1) / 2) * ((g.pz.M + 1) / 2);
    return 3 * cells >= 16 * 152 ? 16 : 8;
}
int axis_sink_blocks(const Geom& g, bool fp32) {
    const int ct = fp32 ? axis_tile_inv(g) : 8;
    return (int)((3LL * g.Ny * g.Nz + ct - 1) / ct);
}

template <typename T> cudaError_t launch_axes(int src, int snk, const PassArgs<T>& a, bool plane, cudaEvent_t* ev) {
    const int Mx = a.g.px.M, My = a.g.py.M;
    const int rows = plane ? 0 : My;  // rows of a component on the work grid: the lattice's, or My
    auto mark = [&](int k) {
        if (ev) cudaEventRecord(ev[k], a.stream);
    };
    mark(0);
    cudaError_t e = axis_run(Mx, AXIS_XFWD, src, rows, a);
    mark(1);
    if (plane) {
        mark(2);
        if constexpr (sizeof(T) == 4) {
            if (e == cudaSuccess) {
                switch (My) {
#define TDDA_X(L) case L: e = plane_##L(a.g.pz.M, &a); break;
                    TDDA_PLANE_Y(TDDA_X)
#undef TDDA_X
                    default: e = cudaErrorInvalidValue;
                }
            }
        }
        mark(3);
        if (e == cudaSuccess) e = axis_run(Mx, AXIS_XINV, snk, rows, a);
        mark(4);
    } else {
        if (e == cudaSuccess) e = axis_run(My, AXIS_YFWD, 0, rows, a);
        mark(2);
        if (e == cudaSuccess) e = zprod_run<T>(a);
        mark(3);
        if (e == cudaSuccess) e = axis_run(My, AXIS_YINV, 0, rows, a);
        mark(4);
        if (e == cudaSuccess) e = axis_run(Mx, AXIS_XINV, snk, rows, a);
    }
    mark(5);
    return e;
}
template cudaError_t launch_axes<float>(int, int, const PassArgs<float>&, bool, cudaEvent_t*);
template cudaError_t launch_axes<double>(int, int, const PassArgs<double>&, bool, cudaEvent_t*);

cudaError_t launch_residual_dd(const Geom& g, int nrhs, const RhsVecs<dd>* rhs, const dd2* green, const dd2* twx,
                               const dd2* twy, const dd2* twz, const int* cellmap, dd2* grid, cudaStream_t stream) {
    if (!dd_lengths(g)) return cudaErrorInvalidValue;
    const PassArgs<dd> a{g, nrhs, rhs, green, twx, twy, twz, cellmap, grid, stream, 0, 0};
    return launch_axes<dd>(SRC_P, SNK_RES, a, false, nullptr);
}

cudaError_t configure_axes() {
    cudaError_t e = cudaSuccess;
#define TDDA_X(L)                                                 \
    if (!e) e = dev::ZprodLaunch<float, L>::configure();          \
    if (!e) e = dev::ZprodLaunch<double, L>::configure();
    TDDA_Z_AXES(TDDA_X)
#undef TDDA_X
#define TDDA_X(L) \
    if (!e) e = dev::ZprodLaunch<dd, L>::configure();
    TDDA_X(20) TDDA_X(32) TDDA_X(40) TDDA_X(48)
#undef TDDA_X
#define TDDA_X(L) \
    if (!e) e = plane_##L(0, nullptr);
    TDDA_PLANE_Y(TDDA_X)
#undef TDDA_X
    return e;
}

}  // namespace tdda
