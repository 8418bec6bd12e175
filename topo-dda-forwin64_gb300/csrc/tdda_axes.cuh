// tdda_axes.cuh -- the A-product in x-first order: transform x while gathering
// the dipole vector, then y, then z with the spectral product, and back.
//
//   k_xfwd   gather (+ the fused vector update of the solver), x forward
//   k_yaxis  y forward / inverse, in place on the work grid
//   k_zprod  z forward, spectral product, z inverse, in place
//   k_xpass2p  (FP32, where three components of a (y, z) plane fit one block's
//            shared memory) the y and z passes and the product in one kernel
//   k_xinv   x inverse, scatter to the dipoles, + al v, the solver's dots
//
// Why this order.  With M = 2N points an axis the zero half of each axis is
// pruned until it is transformed, so the first axis costs N2 N3 lines, the
// second M1 N3 and the last M1 M2: the last axis runs the most lines and
// should be the short one.  Lattices are flat (z is the thickness), so z last
// costs 5 Mz log2 Mz on those lines instead of 5 Mx log2 Mx with x last, and
// the work grid holds [kx][y < Ny][z < Nz] (2N entries a component) between the
// gather, the plane kernel and the scatter, half of a grid kept to x < Nx.
// What it costs is rounding: the inverse that runs last keeps all of its rounding
// errors, while half of an earlier one's go with the halves that later axes drop,
// and now the longest axis is the last.  FP32 products against FP64 ones, z-y-x and
// x-first: 128 x 128 x 32 1.73e-7 and 1.94e-7, 128 x 20 x 10 1.13e-7 and 1.22e-7
// (a float32 model of the same plans in both orders: 1.13e-7 and 1.22e-7), 20 x 20
// x 10 1.29e-7 and 1.28e-7; over 46 boxes 0.97 to 1.12 times, 1.02 in the mean.
// The x lines gather straight from the dipole vectors: cells are contiguous in
// (y, z), so a warp reads and writes whole sectors, and every fused mode of the
// solver lives in the two x kernels, which depend on one length each.
//
// Each axis length M = R1 R2 has a two-stage plan, forward in decimation in
// time and back in decimation in frequency, in place: with n = jj + R2 r and
// k = j + R1 q,
//   forward 1, task jj < R2:  Y[jj R1 + k'] = sum_r x[jj + R2 r] W_R1^(r k')
//   forward 2, task j < R1:   X[j + R1 q]  = sum_r (W_M^(r j) Y[r R1 + j]) W_R2^(r q)
// and the inverse runs the same tasks backwards on conjugate roots.  A task
// writes exactly the slots it read, so one buffer serves every stage and one
// barrier separates two stages.
#pragma once

#include "tdda_passes.cuh"

namespace tdda {
namespace dev {

// ------------------------------------------------------------ plans
// x and y: the gather and the scatter run the tasks of R1, so R1 is the smaller
// one where it can be (few loads in flight per thread, more threads)
__host__ __device__ constexpr int xy_radix1(int M) {
    switch (M) {
        case 12: case 20: case 24: return 4;
        case 14: return 2;
        case 15: case 18: case 21: return 3;
        case 25: return 5;
        case 160: return 10;
        case 192: return 12;
        case 224: return 14;
        case 256: return 16;
        default: return 8;  // 32, 40, 48, 56, 64, 80, 96, 112, 128
    }
}
// z: R2 = 8 where it can be -- a thread of the product holds R2 spectral
// points of three components
__host__ __device__ constexpr int z_radix1(int M) {
    switch (M) {
        case 12: case 15: case 21: case 24: return 3;
        case 14: return 2;
        case 32: return 4;
        case 20: case 25: case 40: return 5;
        case 48: return 6;
        case 56: return 7;
        default: return 8;  // 64
    }
}
__host__ __device__ constexpr int cdiv_i(int a, int b) { return (a + b - 1) / b; }
__host__ __device__ constexpr int round32(int v) { return cdiv_i(v, 32) * 32; }
// one axis: M = R1 R2, at most LX lattice cells (M >= 2N - 1), of which a
// stage-1 task sees the RH inputs x = jj + R2 r < LX
template <int M_, int R1_> struct Axis {
    static constexpr int M = M_, R1 = R1_, R2 = M_ / R1_, LX = (M_ + 1) / 2, RH = cdiv_i(LX, R2);
    static_assert(R1 * R2 == M, "two-stage plan");
};
template <int M> using AxisXY = Axis<M, xy_radix1(M)>;
template <int M> using AxisZ = Axis<M, z_radix1(M)>;

// v[r] times w^(r j) (or its conjugate), r = 1 .. R - 1
template <int R, int SIGN, typename T> __device__ __forceinline__ void twiddle(cx<T>* v, const cx<T>* tw, int j) {
#pragma unroll
    for (int r = 1; r < R; r++) {
        cx<T> t = tw[r * j];
        if (SIGN > 0) t.y = -t.y;
        v[r] = cmul<T>(v[r], t);
    }
}

// A line of the x kernels: one component of one (y, z) cell.  FP32 vectors are
// SoA and their lines component-major; FP64 vectors are AoS and their lines
// cell-major, so that consecutive lines are consecutive entries of either.
template <typename T> constexpr bool kSoa = sizeof(T) == 4;
// entry of the dipole vectors (of an AoS vector: AOS) at cell (x, line), or -1;
// 32 bits hold it (a box has at most 2^28 cells)
template <typename T, bool AOS = false>
__device__ __forceinline__ int line_entry(const Lat& L, int NC, int x, int cell, int c) {
    const int i = L.dense ? x * NC + cell : L.cellmap[x * NC + cell];
    return i < 0 ? -1 : AOS ? 3 * i + c : (int)vec_index<T>(i, c, L.N);
}
// offset of a line in one kx plane of the work grid whose components (SoA) are
// `rows` rows of Nz entries
template <typename T> __device__ __forceinline__ long long line_offset(int line, int c, int cell, int rows, int Nz) {
    return kSoa<T> ? (long long)c * rows * Nz + cell : (long long)line;
}

// Totals of nblk published partials for a block of NW warps (sum_partials: one
// warp per value).  Warp w adds the values w, w + NW, ... together, so their
// loads and additions overlap; lane l takes the partials l, l + 32, ..., then a
// shuffle tree: the order does not depend on the number of warps.
template <int NV, int NW>
__device__ __forceinline__ void sum_partials_nw(const double* part, int nblk, float2* sred, float2 (&tot)[NV]) {
    constexpr int VW = cdiv_i(NV, NW), U = 8 / VW > 2 ? 8 / VW : 2;
    const float2* part2 = reinterpret_cast<const float2*>(part);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp < NV) {
        float2 a[VW];
#pragma unroll
        for (int k = 0; k < VW; k++) a[k] = make_float2(0.f, 0.f);
        for (int i0 = lane; i0 < nblk; i0 += 32 * U) {
            float2 v[VW][U];
#pragma unroll
            for (int k = 0; k < VW; k++)
#pragma unroll
                for (int u = 0; u < U; u++)
                    v[k][u] = i0 + 32 * u < nblk && warp + NW * k < NV
                                  ? __ldcg(part2 + (long long)(warp + NW * k) * nblk + i0 + 32 * u)
                                  : make_float2(0.f, 0.f);
#pragma unroll
            for (int u = 0; u < U; u++)
#pragma unroll
                for (int k = 0; k < VW; k++) a[k] = df_add(a[k], v[k][u]);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int k = 0; k < VW; k++)
                a[k] = df_add(a[k], make_float2(__shfl_down_sync(0xffffffffu, a[k].x, o),
                                                __shfl_down_sync(0xffffffffu, a[k].y, o)));
        if (lane == 0) {
#pragma unroll
            for (int k = 0; k < VW; k++)
                if (warp + NW * k < NV) sred[warp + NW * k] = a[k];
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NV; k++) tot[k] = sred[k];
}

// The step scalars of an FP32 gather (fp32_step_scalars) for any block size.
template <int SRC, int NW>
__device__ __forceinline__ bool step_scalars_nw(const RhsVecs<float>& R, int slot, int prod_nblk, float2* scratch,
                                                float2& alpha, float2& beta, float2& zeta) {
    __shared__ float2 s_sc[3];
    __shared__ int s_stop;
    if constexpr (SRC == SRC_PUPD_DEF) {
        StepIn in = {};
        if (threadIdx.x == 0) in = load_step_in(R.st, slot);
        float2 tot[8];
        sum_partials_nw<8, NW>(R.part, prod_nblk, scratch, tot);
        if (threadIdx.x < 32) {  // the totals are in scratch
            const int status = __shfl_sync(0xffffffffu, in.status, 0);
            if (status != ST_RUNNING) {
                if (threadIdx.x == 0) s_stop = status;
            } else {
                const StepEnd e = step_end_f32(in, scratch);
                if (threadIdx.x == 0) {
                    if (blockIdx.x == 0) write_step_end(R.st, e, slot);
                    s_sc[0] = e.zeta;
                    s_sc[1] = e.beta;
                    s_sc[2] = in.alpha;
                    s_stop = e.stop;
                }
            }
        }
        __syncthreads();
        if (s_stop != ST_RUNNING) return false;
        zeta = s_sc[0];
        beta = s_sc[1];
        alpha = s_sc[2];
    } else {
        float2 rho;
        int status;
        if (threadIdx.x == 0) rho = R.st->rho32[slot], status = R.st->status;
        float2 tot[2];
        sum_partials_nw<2, NW>(R.part, prod_nblk, scratch, tot);
        if (threadIdx.x == 0) {
            const float2 a = fdiv2(rho, make_float2(tot[0].x, tot[1].x));  // DDAModel.cpp:221
            if (status == ST_RUNNING && blockIdx.x == 0) R.st->alpha32[slot] = a;
            s_sc[0] = a;
            s_stop = status;
        }
        __syncthreads();
        if (s_stop != ST_RUNNING) return false;
        alpha = s_sc[0];
    }
    return true;
}

// Block sums of NV values (a power of two) as double-float pairs, published by
// one thread each into part slots k * nblk + bid.  The values are folded while
// the lanes are: each of the first log2 NV shuffle steps halves the values a
// lane holds, so a warp runs NV - 1 + 5 - log2 NV additions instead of 5 NV.
template <int NV>
__device__ __forceinline__ void publish_partials_nw(const float (&v)[NV], double* part, int nblk, int bid,
                                                    float2* sred /* NV x warps */) {
    static_assert((NV & (NV - 1)) == 0 && NV <= 8, "a power of two");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    float2 a[NV];
#pragma unroll
    for (int k = 0; k < NV; k++) a[k] = make_float2(v[k], 0.f);
    int n = NV, mine = 0;  // values held; index of the first one
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        if (n > 1) {
            const int h = n / 2;
            const bool up = lane & o;
#pragma unroll
            for (int k = 0; k < NV / 2; k++) {
                if (k >= h) break;
                const float2 give = up ? a[k] : a[k + h], keep = up ? a[k + h] : a[k];
                const float2 got = make_float2(__shfl_xor_sync(0xffffffffu, give.x, o),
                                               __shfl_xor_sync(0xffffffffu, give.y, o));
                a[k] = df_add(keep, got);
            }
            if (up) mine += h;
            n = h;
        } else {
            a[0] = df_add(a[0], make_float2(__shfl_xor_sync(0xffffffffu, a[0].x, o),
                                            __shfl_xor_sync(0xffffffffu, a[0].y, o)));
        }
    }
    constexpr int kFold = 32 / NV;  // lanes that end with the same value; the lowest one speaks
    if ((lane & (kFold - 1)) == 0) sred[mine * nw + warp] = a[0];
    __syncthreads();
    if (threadIdx.x < NV) {
        float2 t = sred[threadIdx.x * nw];
        for (int w = 1; w < nw; w++) t = df_add(t, sred[threadIdx.x * nw + w]);
        reinterpret_cast<float2*>(part)[(long long)threadIdx.x * nblk + bid] = t;
    }
}

// ------------------------------------------------------------ x kernels
// threads of an x or y kernel: CT lines, one task of the longer stage each
template <int M, int CT> __host__ __device__ constexpr int axis_threads() {
    using A = AxisXY<M>;
    return round32(CT * (A::R1 > A::R2 ? A::R1 : A::R2));
}
// threads of a scatter: FP64 and double-float sinks (diagonal, dots,
// conversions: tens of FP64 instructions an entry) of short lines, whose lattices
// leave SM quarters idle, take one entry per thread whatever the transform's
// tasks; longer lines keep the transform's threads (fewer threads, fewer sums)
template <typename T, int M, int CT> __host__ __device__ constexpr int sink_threads() {
    constexpr int nt = axis_threads<M, CT>(), ne = round32(CT * AxisXY<M>::LX);
    return sizeof(T) == 4 || ne <= nt ? nt : ne <= 256 ? ne : nt < 128 ? 128 : nt;
}
// blocks per SM a gather is compiled for: 512 threads, which may use 128
// registers each (the loads of a task in flight)
template <int M, int CT> __host__ __device__ constexpr int axis_minb() { return 512 / axis_threads<M, CT>(); }
// Shared rows hold CT lines.  With 8 lines an FP32 half warp spans two rows of
// a stage, whose banks must differ by 8 entries: stage 1 steps by R1 rows from
// task to task, so a shift of 8 entries per task is added where R1 is even.
template <typename T, int M, int CT> struct XTile {
    using A = AxisXY<M>;
    static constexpr int SK = (sizeof(T) == 4 && CT == 8 && A::R1 % 2 == 0) ? 8 : 0;
    static constexpr int JS = A::R1 * CT + SK;  // from task jj to jj + 1
    static constexpr size_t smem = sizeof(cx<T>) * (size_t)(M + A::R2 * JS);
};

// The sink of one line: load() issues the loads of its operands, store() forms
// the diagonal term, the stores and the dot-product terms from A v in val.
template <typename T, int SRC, int SNK, int CH> struct SinkIn {
    cx<T> vv[CH], al[CH], q2[CH];
    static constexpr bool kV = SNK != SNK_OUT && SNK != SNK_EXT, kQ = SNK == SNK_AP || SNK == SNK_AT_DEF || SNK == SNK_RES;
    bool unit;  // a Jacobi-preconditioned product adds 1 v (RhsVecs::pre)
    __device__ __forceinline__ void load(const RhsVecs<T>& R, const int (&o)[CH]) {
        const cx<T>* vsrc = SRC == SRC_TUPD ? R.t : (SRC == SRC_P ? R.P : R.p);
        unit = sizeof(T) == 4 && R.pre != nullptr;
#pragma unroll
        for (int q = 0; q < CH; q++) {
            if (o[q] < 0) continue;
            if constexpr (kV) {
                vv[q] = ldv<T>(vsrc, o[q]);
                if (!unit) al[q] = ldv<T>(R.al, o[q]);
            }
            if constexpr (kQ) q2[q] = ldv<T>(SNK == SNK_RES ? R.E : R.r0, o[q]);
        }
    }
    template <int NV>
    __device__ __forceinline__ void store(const RhsVecs<T>& R, const int (&o)[CH], const cx<T>* val,
                                          acc_t<T> (&acc)[NV], double2* ext) const {
#pragma unroll
        for (int q = 0; q < CH; q++) {
            if (o[q] < 0) continue;
            if constexpr (SNK == SNK_EXT) {
                ext[o[q]] = make_double2((double)val[q].x, (double)val[q].y);
            } else if constexpr (SNK == SNK_OUT) {
                R.Ap[o[q]] = val[q];
            } else {
                const cx<T> t = vv[q], w = cadd<T>(val[q], unit ? t : cmul<T>(t, al[q]));
                if constexpr (SNK == SNK_ALB) {
                    R.Ap[o[q]] = w;
                } else if constexpr (SNK == SNK_AP) {
                    R.Ap[o[q]] = w;
                    const cx<T> r0 = q2[q];  // r0 . Ap
                    acc[0] += r0.x * w.x + r0.y * w.y;
                    acc[1] += r0.x * w.y - r0.y * w.x;
                } else if constexpr (SNK == SNK_AT || SNK == SNK_AT_DEF) {
                    R.At[o[q]] = w;
                    acc[0] += w.x * t.x + w.y * t.y;  // At . t
                    acc[1] += w.x * t.y - w.y * t.x;
                    acc[2] += w.x * w.x + w.y * w.y;  // At . At
                    if constexpr (SNK == SNK_AT_DEF) {  // r0 . t, r0 . At, t . t
                        const cx<T> r0 = q2[q];
                        acc[3] += r0.x * t.x + r0.y * t.y;
                        acc[4] += r0.x * t.y - r0.y * t.x;
                        acc[5] += r0.x * w.x + r0.y * w.y;
                        acc[6] += r0.x * w.y - r0.y * w.x;
                        acc[7] += t.x * t.x + t.y * t.y;
                    }
                } else {  // SNK_RES
                    const cx<T> res = csub<T>(q2[q], w);
                    stv<T>(R.r, o[q], res);
                    stv<T>(R.r0, o[q], res);
                    stv<T>(R.p, o[q], res);
                    acc[0] += cnorm2<T>(res);
                }
            }
        }
    }
};

// Gather and x forward of tiles of CT lines.  The loads of a task's cells are
// issued together.  The FP32 step's scalars come from the partials of every
// sink block, so a block forms them once, while its first tile's loads are in
// flight, and then takes every gridDim.x-th tile.
template <typename T, int SRC, int M, int CT>
__global__ void __launch_bounds__(axis_threads<M, CT>(), axis_minb<M, CT>()) k_xfwd(Geom g, const RhsVecs<T>* __restrict__ rhs,
                                                                const cx<T>* __restrict__ twx,
                                                                const int* __restrict__ cellmap,
                                                                cx<T>* __restrict__ grid, int pitch_rows, int slot,
                                                                int prod_nblk, const double2* in_ext) {
    using A = AxisXY<M>;
    using TL = XTile<T, M, CT>;
    constexpr bool kStep32 = sizeof(T) == 4 && (SRC == SRC_PUPD_DEF || SRC == SRC_TUPD);
    constexpr int R1 = A::R1, R2 = A::R2, RH = A::RH, NT = axis_threads<M, CT>();
    static_assert(CT * R1 <= NT && CT * R2 <= NT, "one task of each stage per thread");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cx<T>* stw = reinterpret_cast<cx<T>*>(smem_raw);
    cx<T>* s = stw + M;
    __shared__ float2 s_scratch[kStep32 ? 8 : 1];
    const int b = blockIdx.y;
    const RhsVecs<T> R = rhs[b];
    const Lat L = lattice_of<T>(g, R, cellmap);
    const int NC = L.Ny * L.Nz, NL = 3 * NC;
    const int rows = pitch_rows ? pitch_rows : L.Ny;  // rows of a component on the work grid
    if (blockIdx.x * CT >= NL) return;  // past this right-hand side's lines (cross-lattice batches)
    stage_tw<T>(stw, twx, M);
    grid_dep_wait();  // the vectors, partials and states are the previous kernel's
    if (g.early == 1) grid_dep_release();
    if constexpr (!kStep32) {  // the FP32 step reads the status with its scalars
        if (rhs_done(R.st)) return;
    }
    cx<T> beta, alpha, zeta;
    if constexpr (!kStep32) {
        if (SRC == SRC_PUPD) beta = st_beta<T>(R.st);
        if (SRC == SRC_TUPD) alpha = st_alpha<T>(R.st);
    }
    const cx<T>* src = SRC == SRC_IN ? R.p : R.P;
    const long long kxs = 3LL * rows * L.Nz;
    cx<T>* gb = grid + (long long)b * g.vb;
    const int l = threadIdx.x % CT, j = threadIdx.x / CT;  // line of the tile, task of either stage
    for (int l0 = blockIdx.x * CT; l0 < NL; l0 += gridDim.x * CT) {
        const int line = l0 + l;
        const int c = kSoa<T> ? line / NC : line % 3, cell = kSoa<T> ? line - c * NC : line / 3;
        if (l0 != (int)blockIdx.x * CT) __syncthreads();  // the previous tile's stage 2 has read s
        int o[RH];
#pragma unroll
        for (int r = 0; r < RH; r++) {
            const int x = j + R2 * r;
            o[r] = j < R2 && line < NL && x < L.Nx ? line_entry<T, SRC == SRC_EXT>(L, NC, x, cell, c) : -1;
        }
        cx<T> v[R1];
        if constexpr (SRC == SRC_EXT) {
#pragma unroll
            for (int r = 0; r < RH; r++) v[r] = o[r] >= 0 ? from_d<T>(in_ext[o[r]]) : czero<T>();
        } else if constexpr (is_dd<T>) {
#pragma unroll
            for (int r = 0; r < RH; r++) v[r] = o[r] >= 0 ? ldv<T>(src, o[r]) : czero<T>();
        } else {
            GatherIn<T, SRC, RH> in;
            in.load(R, o, src);
            if constexpr (kStep32) {
                if (l0 == (int)blockIdx.x * CT &&
                    !step_scalars_nw<SRC, NT / 32>(R, slot, prod_nblk, s_scratch, alpha, beta, zeta))
                    return;
            }
            cx<T> u[RH];
            in.combine(R, o, u, alpha, beta, zeta);
#pragma unroll
            for (int r = 0; r < RH; r++) v[r] = u[r];
        }
        if (j < R2) {
            BflyIn<R1, -1, T, RH>::run(v);
#pragma unroll
            for (int q = 0; q < R1; q++) s[j * TL::JS + q * CT + l] = v[q];
        }
        __syncthreads();  // also publishes the twiddles
        if (g.early == 2 && l0 + gridDim.x * CT >= NL) grid_dep_release();  // the next kernel's blocks start
        if (j < R1 && line < NL) {
            cx<T> w[R2];
#pragma unroll
            for (int r = 0; r < R2; r++) w[r] = s[r * TL::JS + j * CT + l];
            twiddle<R2, -1, T>(w, stw, j);
            Bfly<R2, -1, T>::run(w);
            cx<T>* d = gb + line_offset<T>(line, c, cell, rows, L.Nz) + j * kxs;
#pragma unroll
            for (int q = 0; q < R2; q++, d += R1 * kxs) *d = w[q];
        }
    }
}

// Inverse x transform of CT lines and the scatter.  FP32: task j of the last
// stage holds the cells x = j + R2 r of one line and scatters them; the sink's
// operands do not depend on the transform, and their loads are issued before the
// barrier.  FP64 and double-float: the cells go back to shared memory (in place)
// and all threads of the block share them.  The double-float kernel waits for
// memory: registers for 768 threads an SM instead of 512 (96 x 96 x 24, four
// right-hand sides: 213 -> 170 us; 640: 184; 80 x 80 x 20, two: 63 -> 62).
template <typename T, int SRC, int SNK, int M, int CT>
__global__ void __launch_bounds__(sink_threads<T, M, CT>(), is_dd<T> ? 768 / sink_threads<T, M, CT>() : 0) k_xinv(Geom g, const RhsVecs<T>* __restrict__ rhs,
                                                                  const cx<T>* __restrict__ twx,
                                                                  const int* __restrict__ cellmap,
                                                                  const cx<T>* __restrict__ grid, int pitch_rows,
                                                                  double2* out_ext) {
    using A = AxisXY<M>;
    using TL = XTile<T, M, CT>;
    constexpr int R1 = A::R1, R2 = A::R2, RH = A::RH, LX = A::LX, NT = sink_threads<T, M, CT>();
    constexpr int NV = SNK == SNK_AT_DEF ? 8 : SNK == SNK_AT ? 3 : SNK == SNK_AP ? 2 : 1;  // sums of the sink
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cx<T>* stw = reinterpret_cast<cx<T>*>(smem_raw);
    cx<T>* s = stw + M;
    constexpr bool kSums = SNK != SNK_OUT && SNK != SNK_ALB && SNK != SNK_EXT;
    __shared__ double sred[!kSums ? 1 : sizeof(T) == 4 ? NV * (NT / 32) : NV * NT];
    const int b = blockIdx.y;
    const RhsVecs<T> R = rhs[b];
    const Lat L = lattice_of<T>(g, R, cellmap);
    const int NC = L.Ny * L.Nz, NL = 3 * NC;
    const int rows = pitch_rows ? pitch_rows : L.Ny;  // rows of a component on the work grid
    const int l0 = blockIdx.x * CT;
    acc_t<T> acc[NV] = {};
    if (l0 < NL) {
        stage_tw<T>(stw, twx, M);
        grid_dep_wait();  // the grid and the solve's state are the previous kernel's
        if (g.early == 1) grid_dep_release();
        const int l = threadIdx.x % CT, j = threadIdx.x / CT, line = l0 + l;  // line of the tile, task of either stage
        const int c = kSoa<T> ? line / NC : line % 3, cell = kSoa<T> ? line - c * NC : line / 3;
        const long long kxs = 3LL * rows * L.Nz;
        cx<T> w[R2];
        {
            const bool task = j < R1 && line < NL;
            const cx<T>* d = grid + (long long)b * g.vb + line_offset<T>(line, c, cell, rows, L.Nz) + j * kxs;
#pragma unroll
            for (int q = 0; q < R2; q++, d += R1 * kxs) w[q] = task ? *d : czero<T>();
        }
        if (rhs_done(R.st)) return;  // checked after the first loads are issued: nothing is written yet
        __syncthreads();             // publishes the twiddles
        if (j < R1) {
            Bfly<R2, +1, T>::run(w);
            twiddle<R2, +1, T>(w, stw, j);
#pragma unroll
            for (int r = 0; r < R2; r++) s[r * TL::JS + j * CT + l] = w[r];
        }
        if (g.early == 2) grid_dep_release();  // the next kernel's blocks start during the last stage
        if constexpr (sizeof(T) == 4) {
            int o[RH];
#pragma unroll
            for (int r = 0; r < RH; r++) {
                const int x = j + R2 * r;
                o[r] = j < R2 && line < NL && x < L.Nx ? line_entry<T, SNK == SNK_EXT>(L, NC, x, cell, c) : -1;
            }
            SinkIn<T, SRC, SNK, RH> in;
            in.load(R, o);
            __syncthreads();
            if (j < R2) {
                cx<T> v[R1];
#pragma unroll
                for (int q = 0; q < R1; q++) v[q] = s[j * TL::JS + q * CT + l];
                Bfly<R1, +1, T>::run(v);
                in.template store<NV>(R, o, v, acc, out_ext);
            }
        } else {
            __syncthreads();
            if (j < R2) {
                cx<T> v[R1];
#pragma unroll
                for (int q = 0; q < R1; q++) v[q] = s[j * TL::JS + q * CT + l];
                Bfly<R1, +1, T>::run(v);
#pragma unroll
                for (int r = 0; r < RH; r++) s[j * TL::JS + r * CT + l] = v[r];
            }
            // cell x = j + R2 r of line l0 + l; kGroup entries' operands are in flight together,
            // the first group's through the barrier (96 x 96 x 24, eight double-float right-hand
            // sides: 451 -> 389 us with groups of three against one entry at a time)
            constexpr int kGroup = 3;
            SinkIn<T, SRC, SNK, kGroup> in;
            int o[kGroup];
            auto load = [&](int e0) {
#pragma unroll
                for (int k = 0; k < kGroup; k++) {
                    const int e = e0 + k * NT, x = e / CT, ln = l0 + e % CT;
                    o[k] = x < L.Nx && ln < NL ? line_entry<T>(L, NC, x, ln / 3, ln % 3) : -1;
                }
                in.load(R, o);
            };
            load(threadIdx.x);
            __syncthreads();
            for (int e0 = threadIdx.x; e0 < L.Nx * CT; e0 += kGroup * NT) {
                if (e0 != (int)threadIdx.x) load(e0);
                cx<T> v[kGroup];
#pragma unroll
                for (int k = 0; k < kGroup; k++) {
                    const int e = e0 + k * NT, x = e / CT;
                    v[k] = o[k] >= 0 ? s[(x % R2) * TL::JS + (x / R2) * CT + e % CT] : czero<T>();
                }
                in.template store<NV>(R, o, v, acc, out_ext);
            }
        }
    } else {
        // past this right-hand side's lines (cross-lattice batches): its sums take
        // zeros here, after its own blocks' partials, which leaves them unchanged
        if constexpr (!kSums) return;
        grid_dep_wait();
        if (rhs_done(R.st)) return;
    }
    if constexpr (kSums) {
        if constexpr (sizeof(T) == 4) {
            publish_partials_nw<NV>(acc, R.part, gridDim.x, blockIdx.x, reinterpret_cast<float2*>(sred));
        } else {
            tot_t<T> tot[NV];
            const int slot = SNK == SNK_AP ? 0 : (SNK == SNK_AT ? 1 : 2);
            if (!last_block_total<NV>(acc, R.part, gridDim.x, blockIdx.x, R.cnt + slot, sred, tot)) return;
            if (threadIdx.x != 0) return;
            finalize_sink<T, SNK, NV>(R.st, tot);
        }
    }
}

// ------------------------------------------------------------ y axis
// CT columns of the work grid, in place.  A column is one z (and, cell-major,
// component) of one kx (and component): W columns per group of My rows of W.
template <typename T, int SIGN, int M, int CT>
__global__ void __launch_bounds__(axis_threads<M, CT>()) k_yaxis(Geom g, const RhsVecs<T>* __restrict__ rhs,
                                                                 const cx<T>* __restrict__ twy,
                                                                 cx<T>* __restrict__ grid) {
    using A = AxisXY<M>;
    using TL = XTile<T, M, CT>;
    constexpr int R1 = A::R1, R2 = A::R2, RH = A::RH, NT = axis_threads<M, CT>();
    constexpr int T1 = cdiv_i(CT * R2, NT), T2 = cdiv_i(CT * R1, NT);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cx<T>* stw = reinterpret_cast<cx<T>*>(smem_raw);
    cx<T>* s = stw + M;
    const int b = blockIdx.y;
    const SolveState* st = rhs[b].st;
    const int Ny = g.multi ? rhs[b].Ny : g.Ny, Nz = g.multi ? rhs[b].Nz : g.Nz;
    const int W = kSoa<T> ? Nz : 3 * Nz;
    const int ncol = g.px.M * 3 * Nz, c0 = blockIdx.x * CT;
    if (c0 >= ncol) return;
    stage_tw<T>(stw, twy, M);
    cx<T>* gb = grid + (long long)b * g.vb;
    // CT divides the threads' stride, so every task of a thread is on one column
    const int l = threadIdx.x % CT, col = c0 + l, grp = col / W;
    const bool live = col < ncol;
    cx<T>* d = gb + (long long)grp * M * W + (col - grp * W);
    const int j0 = threadIdx.x / CT;
    grid_dep_wait();
    if (g.early == 1) grid_dep_release();
    if constexpr (SIGN < 0) {
#pragma unroll
        for (int k = 0; k < T1; k++) {
            const int jj = j0 + k * (NT / CT);
            if (jj >= R2) break;
            cx<T> v[R1];
#pragma unroll
            for (int r = 0; r < RH; r++) {
                const int y = jj + R2 * r;
                v[r] = live && y < Ny ? d[(long long)y * W] : czero<T>();
            }
            BflyIn<R1, -1, T, RH>::run(v);
#pragma unroll
            for (int q = 0; q < R1; q++) s[jj * TL::JS + q * CT + l] = v[q];
        }
        if (rhs_done(st)) return;
        __syncthreads();
        if (g.early == 2) grid_dep_release();
#pragma unroll
        for (int k = 0; k < T2; k++) {
            const int j = j0 + k * (NT / CT);
            if (j >= R1) break;
            cx<T> v[R2];
#pragma unroll
            for (int r = 0; r < R2; r++) v[r] = s[r * TL::JS + j * CT + l];
            twiddle<R2, -1, T>(v, stw, j);
            Bfly<R2, -1, T>::run(v);
            if (live) {
#pragma unroll
                for (int q = 0; q < R2; q++) d[(long long)(j + R1 * q) * W] = v[q];
            }
        }
    } else {
        __syncthreads();  // publishes the twiddles
#pragma unroll
        for (int k = 0; k < T2; k++) {
            const int j = j0 + k * (NT / CT);
            if (j >= R1) break;
            cx<T> v[R2];
#pragma unroll
            for (int q = 0; q < R2; q++) v[q] = live ? d[(long long)(j + R1 * q) * W] : czero<T>();
            Bfly<R2, +1, T>::run(v);
            twiddle<R2, +1, T>(v, stw, j);
#pragma unroll
            for (int r = 0; r < R2; r++) s[r * TL::JS + j * CT + l] = v[r];
        }
        if (rhs_done(st)) return;
        __syncthreads();
        if (g.early == 2) grid_dep_release();
#pragma unroll
        for (int k = 0; k < T1; k++) {
            const int jj = j0 + k * (NT / CT);
            if (jj >= R2) break;
            cx<T> v[R1];
#pragma unroll
            for (int q = 0; q < R1; q++) v[q] = s[jj * TL::JS + q * CT + l];
            Bfly<R1, +1, T>::run(v);
            if (live) {
#pragma unroll
                for (int r = 0; r < RH; r++) {
                    const int y = jj + R2 * r;
                    if (y < Ny) d[(long long)y * W] = v[r];
                }
            }
        }
    }
}

// ------------------------------------------------------------ z axis and product
// acc + a b
template <typename T> __device__ __forceinline__ cx<T> cfma(cx<T> a, cx<T> b, cx<T> acc) {
    if constexpr (is_dd<T>) {
        return cadd<T>(acc, cmul<T>(a, b));
    } else {  // four fused multiply-adds
        acc.x = fma(a.x, b.x, acc.x);
        acc.y = fma(a.x, b.y, acc.y);
        acc.x = fma(-a.y, b.y, acc.x);
        acc.y = fma(a.y, b.x, acc.y);
        return acc;
    }
}
// The six components at one (kx, ky) row of the folded spectrum, by fz: one
// 64-bit base per row and 32-bit offsets, so a load costs one address
// instruction.  16-byte loads: pairs of components (FP32) or components.
template <typename T> struct GreenRow {
    const float4* p;
    int z, l;
    __device__ __forceinline__ GreenRow(const cx<T>* green, const Geom& g, int fx, int fy) {
        const GreenStride& gs = sizeof(T) == 4 ? g.gs32 : g.gs64;
        p = reinterpret_cast<const float4*>(green) + (fx * gs.x + fy * gs.y);
        z = (int)gs.z;
        l = (int)gs.l;
    }
    static __device__ __forceinline__ cx<T> one(float4 v) {
        if constexpr (is_dd<T>) {
            return dd2(v);
        } else {
            cx<T> c;
            memcpy(&c, &v, sizeof(c));
            return c;
        }
    }
    __device__ __forceinline__ void load(int fz, cx<T> (&a)[6]) const {
        const float4* q = p + fz * z;
        if constexpr (sizeof(T) == 4) {
#pragma unroll
            for (int k = 0; k < 3; k++) {
                const float4 v = __ldg(q + k * l);
                a[2 * k] = mk<T>(v.x, v.y), a[2 * k + 1] = mk<T>(v.z, v.w);
            }
        } else {
#pragma unroll
            for (int k = 0; k < 6; k++) a[k] = one(__ldg(q + k * l));
        }
    }
};
// v with its sign flipped where m = 0x80000000 (m = 0: v)
__device__ __forceinline__ float xor_sign(float v, unsigned m) { return __uint_as_float(__float_as_uint(v) ^ m); }
__device__ __forceinline__ double xor_sign(double v, unsigned m) {
    return __hiloint2double(__double2hiint(v) ^ (int)m, __double2loint(v));
}
__device__ __forceinline__ dd xor_sign(dd v, unsigned m) { return dd(xor_sign(v.hi, m), xor_sign(v.lo, m)); }
// C = A b with the symmetric 3 x 3 tensor at one spectral point; the masks are
// 0x80000000 in the upper half of an axis.  Signs without branches: rows of
// both halves share a warp.
template <typename T>
__device__ __forceinline__ void spectral_point(cx<T> (&a)[6], unsigned mx, unsigned my, unsigned mz, cx<T>& b0,
                                               cx<T>& b1, cx<T>& b2) {
    a[1] = mk<T>(xor_sign(a[1].x, mx ^ my), xor_sign(a[1].y, mx ^ my));  // xy: odd in x and y
    a[2] = mk<T>(xor_sign(a[2].x, mx ^ mz), xor_sign(a[2].y, mx ^ mz));  // xz: odd in x and z
    a[4] = mk<T>(xor_sign(a[4].x, my ^ mz), xor_sign(a[4].y, my ^ mz));  // yz: odd in y and z
    const cx<T> x = b0, y = b1, z = b2;
    b0 = cfma<T>(a[0], x, cfma<T>(a[1], y, cmul<T>(a[2], z)));
    b1 = cfma<T>(a[1], x, cfma<T>(a[3], y, cmul<T>(a[4], z)));
    b2 = cfma<T>(a[2], x, cfma<T>(a[4], y, cmul<T>(a[5], z)));
}
__device__ __forceinline__ unsigned half_mask(int k, int M) { return 2 * k > M ? 0x80000000u : 0u; }
// R2 spectral points of one row, kz = j + R1 q.  For even R2 the upper half is
// q >= R2 / 2, known at compile time (kz = M / 2 counts as upper there: its odd
// components vanish).  The spectrum's loads run kAhead points ahead of their
// use, the first ones issued by the constructor, before the transform of the
// vectors: left to the compiler, they waited for L2 point by point (192 x 48
// planes, eight right-hand sides: 243 -> 181 us; of 2 to 5 points ahead, 5 is
// the fastest or within 3% of it on 29 plane sizes).
template <typename T, int R1, int R2, int M, int kAhead_> struct SpectralRow {
    static constexpr int kAhead = kAhead_;
    GreenRow<T> gr;
    int j;
    cx<T> a[kAhead][6];
    static __device__ __forceinline__ bool upper(int q, int kz) { return R2 % 2 == 0 ? 2 * q >= R2 : 2 * kz > M; }
    __device__ __forceinline__ void load(int q) {
        const int kz = j + R1 * q;
        gr.load(upper(q, kz) ? M - kz : kz, a[q % kAhead]);
    }
    __device__ __forceinline__ SpectralRow(const GreenRow<T>& g, int j_) : gr(g), j(j_) {
#pragma unroll
        for (int q = 0; q < kAhead && q < R2; q++) load(q);
    }
    __device__ __forceinline__ void apply(cx<T> (&X)[3][R2], unsigned mx, unsigned my) {
#pragma unroll
        for (int q = 0; q < R2; q++) {
            spectral_point<T>(a[q % kAhead], mx, my, upper(q, j + R1 * q) ? 0x80000000u : 0u, X[0][q], X[1][q],
                              X[2][q]);
            if (q + kAhead < R2) load(q + kAhead);
        }
    }
};

// FP64 and double-float run the second z stage, the product and the first
// inverse stage as separate phases of small tasks: the FP64 pipe takes one warp
// instruction in 64 cycles on each SM quarter, whatever its active lanes, so
// what counts is full warps spread evenly over the quarters.  FP32 keeps the
// three components of R2 points in registers through all three.
template <typename T> constexpr bool kZFused = sizeof(T) == 4;
template <typename T, int M, int RT> __host__ __device__ constexpr int zprod_threads() {
    return !kZFused<T> ? 128 : round32(RT * AxisZ<M>::R1) < 64 ? 64 : round32(RT * AxisZ<M>::R1);
}
// Rows of a full tile, points the FP32 spectrum's loads run ahead, and the threads
// an SM has to hold (registers): what bounds the FP32 kernel is its loads' latency,
// so the long lengths take smaller tiles, more blocks and loads further ahead
// (steps of 110 x 100 x 24, z length 48: 168 us with 32 rows, 1 ahead and no
// bound, 147 so; 80 x 100 x 28, 56: 139 and 119; 128 x 128 x 32, 64: 246 and 240,
// where the bound costs 3 us; 60 x 128 x 20, 40: 91 and 83 with the bound alone,
// 89 with the small tile).  The lengths below 40 lose with any of the three.
template <typename T, int M> __host__ __device__ constexpr int zprod_wide() { return kZFused<T> && M < 48 ? 32 : 16; }
template <int M, int RT> __host__ __device__ constexpr int zprod_ahead() { return M < 48 || RT < 16 ? 1 : 3; }
template <typename T, int M, int RT> __host__ __device__ constexpr int zprod_minb() {  // 0: unspecified (1 lets the compiler take more registers: 128 x 128 x 32 288 us)
    return kZFused<T> && M >= 40 && M < 64 && RT >= 16 ? 640 / zprod_threads<T, M, RT>() : 0;
}
// RT rows (kx, ky) of three components: row pitch odd, so that consecutive rows
// start in different banks
template <typename T, int M, int RT> struct ZTile {
    static constexpr int ZP = pad_odd(M);
    static constexpr size_t smem = sizeof(cx<T>) * (size_t)(M + 3 * RT * ZP);
};
template <typename T, int M, int RT>
__global__ void __launch_bounds__(zprod_threads<T, M, RT>(), zprod_minb<T, M, RT>())
    k_zprod(Geom g, const RhsVecs<T>* __restrict__ rhs, const cx<T>* __restrict__ green, const cx<T>* __restrict__ twz,
            cx<T>* __restrict__ grid) {
    using A = AxisZ<M>;
    constexpr int R1 = A::R1, R2 = A::R2, RH = A::RH, ZP = ZTile<T, M, RT>::ZP, NT = zprod_threads<T, M, RT>();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cx<T>* stw = reinterpret_cast<cx<T>*>(smem_raw);
    cx<T>* s = stw + M;
    const int b = blockIdx.y;
    const SolveState* st = rhs[b].st;
    const int My = g.py.M, Mx = g.px.M, Nz = g.multi ? rhs[b].Nz : g.Nz;
    if (g.multi) green = rhs[b].green;
    const int row0 = blockIdx.x * RT, nrow = min(RT, Mx * My - row0);
    const int kx0 = row0 / My, ky0 = row0 - kx0 * My;
    stage_tw<T>(stw, twz, M);
    cx<T>* gb = grid + (long long)b * g.vb;
    // element (row, component, z): SoA [kx][c][ky][z], AoS [kx][ky][z][c]
    auto at = [&](int row, int c, int z) -> long long {
        if constexpr (!kSoa<T>) return ((long long)(row0 + row) * Nz + z) * 3 + c;
        int kx = kx0, ky = ky0 + row;
        while (ky >= My) ky -= My, kx++;
        return (((long long)kx * 3 + c) * My + ky) * Nz + z;
    };
    grid_dep_wait();
    if (g.early == 1) grid_dep_release();
    // z forward, stage 1, from the grid: consecutive threads on consecutive entries
    for (int w = threadIdx.x; w < 3 * RT * R2; w += NT) {
        int row, c, j;
        if constexpr (kSoa<T>) j = w % R2, row = (w / R2) % RT, c = w / (R2 * RT);
        else c = w % 3, j = (w / 3) % R2, row = w / (3 * R2);
        cx<T> v[R1];
#pragma unroll
        for (int r = 0; r < RH; r++) {
            const int z = j + R2 * r;
            v[r] = row < nrow && z < Nz ? gb[at(row, c, z)] : czero<T>();
        }
        BflyIn<R1, -1, T, RH>::run(v);
        cx<T>* d = s + (c * RT + row) * ZP + j;
#pragma unroll
        for (int q = 0; q < R1; q++) d[R2 * q] = v[q];
    }
    if (rhs_done(st)) return;
    __syncthreads();
    // the kx, ky of a row of the tile
    auto row_k = [&](int row, int& kx, int& ky) {
        kx = kx0, ky = ky0 + row;
        while (ky >= My) ky -= My, kx++;
    };
    if constexpr (kZFused<T>) {
        // stage 2, product, inverse stage 1: consecutive threads on consecutive rows
        for (int w = threadIdx.x; w < RT * R1; w += NT) {
            const int row = w % RT, j = w / RT;
            int kx, ky;
            row_k(row, kx, ky);
            if (kx >= Mx) continue;
            SpectralRow<T, R1, R2, M, zprod_ahead<M, RT>()> sp(GreenRow<T>(green, g, fold(kx, Mx), fold(ky, My)), j);
            cx<T> X[3][R2];
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const cx<T>* d = s + (c * RT + row) * ZP + R2 * j;
#pragma unroll
                for (int r = 0; r < R2; r++) X[c][r] = d[r];
                twiddle<R2, -1, T>(X[c], stw, j);
                Bfly<R2, -1, T>::run(X[c]);
            }
            sp.apply(X, half_mask(kx, Mx), half_mask(ky, My));
#pragma unroll
            for (int c = 0; c < 3; c++) {
                Bfly<R2, +1, T>::run(X[c]);
                twiddle<R2, +1, T>(X[c], stw, j);
                cx<T>* d = s + (c * RT + row) * ZP + R2 * j;
#pragma unroll
                for (int r = 0; r < R2; r++) d[r] = X[c][r];
            }
        }
    } else {
        for (int w = threadIdx.x; w < 3 * RT * R1; w += NT) {  // stage 2, in place
            const int row = w % (3 * RT), j = w / (3 * RT);    // rows of all components
            cx<T>* d = s + row * ZP + R2 * j;
            cx<T> v[R2];
#pragma unroll
            for (int r = 0; r < R2; r++) v[r] = d[r];
            twiddle<R2, -1, T>(v, stw, j);
            Bfly<R2, -1, T>::run(v);
#pragma unroll
            for (int r = 0; r < R2; r++) d[r] = v[r];
        }
        __syncthreads();
        for (int w = threadIdx.x; w < RT * M; w += NT) {  // entry R2 j + q holds kz = j + R1 q
            const int row = w % RT, e = w / RT, kz = e / R2 + R1 * (e % R2);
            int kx, ky;
            row_k(row, kx, ky);
            if (kx >= Mx) continue;
            cx<T> a[6];
            GreenRow<T>(green, g, fold(kx, Mx), fold(ky, My)).load(fold(kz, M), a);
            cx<T>* d = s + row * ZP + e;
            cx<T> b0 = d[0], b1 = d[RT * ZP], b2 = d[2 * RT * ZP];
            spectral_point<T>(a, half_mask(kx, Mx), half_mask(ky, My), half_mask(kz, M), b0, b1, b2);
            d[0] = b0, d[RT * ZP] = b1, d[2 * RT * ZP] = b2;
        }
        __syncthreads();
        for (int w = threadIdx.x; w < 3 * RT * R1; w += NT) {  // inverse stage 1, in place
            const int row = w % (3 * RT), j = w / (3 * RT);
            cx<T>* d = s + row * ZP + R2 * j;
            cx<T> v[R2];
#pragma unroll
            for (int r = 0; r < R2; r++) v[r] = d[r];
            Bfly<R2, +1, T>::run(v);
            twiddle<R2, +1, T>(v, stw, j);
#pragma unroll
            for (int r = 0; r < R2; r++) d[r] = v[r];
        }
    }
    __syncthreads();
    if (g.early == 2) grid_dep_release();
    for (int w = threadIdx.x; w < 3 * RT * R2; w += NT) {
        int row, c, j;
        if constexpr (kSoa<T>) j = w % R2, row = (w / R2) % RT, c = w / (R2 * RT);
        else c = w % 3, j = (w / 3) % R2, row = w / (3 * R2);
        const cx<T>* d = s + (c * RT + row) * ZP + j;
        cx<T> v[R1];
#pragma unroll
        for (int q = 0; q < R1; q++) v[q] = d[R2 * q];
        Bfly<R1, +1, T>::run(v);
#pragma unroll
        for (int r = 0; r < RH; r++) {
            const int z = j + R2 * r;
            if (row < nrow && z < Nz) gb[at(row, c, z)] = v[r];
        }
    }
}

// ------------------------------------------------------------ fused (y, z) plane
// One block holds the three components of one kx plane in shared memory and
// runs y forward, z forward, the spectral product, z inverse and y inverse in
// place: the plane is read and written once, as its Ny x Nz lattice part.
// y runs the plan MY = B1 8, z the plan MZ = A1 A2 (A2 = 8, or 4 for 20), so
// that a thread can follow the second y stage of the columns z, z + A2, ... with
// their first z stage in registers (and back): five phases, four exchanges.
//   1  y stage 1 from the grid         task (c, jj < 8, z)
//   2  y stage 2, z stage 1            task (c, j < B1, jz < A2): AH columns, 8 rows
//   3  z stage 2, product, z stage 2'  task (ky, j < A1): three components
//   4  z stage 1', y stage 2'          as 2, backwards
//   5  y stage 1' to the grid          as 1, backwards
// Shared rows of ZP entries, ZP = 2 (mod 4): phase 3 reads 16-byte values with
// consecutive threads on rows 16 bytes apart modulo the banks, phases 2 and 4
// take 2 columns x 8 rows to a half warp; both without conflicts.
template <int MY, int MZ> struct Plane {
    using Y = Axis<MY, MY / 8>;
    using Z = AxisZ<MZ>;
    static constexpr int ZP = MZ + (MZ % 4 == 0 ? 2 : 4);
    static constexpr size_t smem = sizeof(float2) * (size_t)(MY + MZ + 3 * MY * ZP);
    // Registers are given to warps in fours, one per SM quarter: 512 threads may
    // use 128, which phase 3 needs.
    static constexpr int NT = MY * MZ <= 1024 ? 256 : 512;
    // a second form with two blocks of 256 threads an SM, where both fit: it overlaps
    // the phases of two planes, but takes longer over one (PlaneLaunch)
    static constexpr bool kPair = NT == 512 && smem <= 113000;
};
constexpr size_t kMaxPlaneSmem = 232448;  // 227 KB, the most one block may use
template <int MY, int MZ> constexpr bool plane_fits() { return Plane<MY, MZ>::smem <= kMaxPlaneSmem; }

// 16-byte shared accesses of N (even) consecutive values
template <int N> __device__ __forceinline__ void load_pairs(const float2* d, float2* v) {
#pragma unroll
    for (int r = 0; r < N; r += 2) {
        const float4 u = *reinterpret_cast<const float4*>(d + r);
        v[r] = make_float2(u.x, u.y), v[r + 1] = make_float2(u.z, u.w);
    }
}
template <int N> __device__ __forceinline__ void store_pairs(float2* d, const float2* v) {
#pragma unroll
    for (int r = 0; r < N; r += 2)
        *reinterpret_cast<float4*>(d + r) = make_float4(v[r].x, v[r].y, v[r + 1].x, v[r + 1].y);
}
// Rows ky and My - ky share their folded spectrum: a warp takes eight
// consecutive rows and their mirror images, so its loads cover half the lines
// (and each quarter warp's rows stay 16 bytes apart modulo the banks).
template <int MY> __device__ __forceinline__ int mirrored_row(int i) {
    if constexpr (MY % 16 != 0) return i;
    const int h = i / 16 * 8 + i % 8;
    return i % 16 < 8 ? h : (h == 0 ? MY / 2 : MY - h);
}

// The plane of the block that follows this one on its SM (`resident` blocks fill
// the device, and blocks start in order) into L2: with a batch the work grid does
// not stay there, and phase 1 would wait for DRAM at the start of every block.
__device__ __forceinline__ void prefetch_plane(const Geom& g, const RhsVecs<float>* rhs, const float2* grid, int kx,
                                               int b, int resident) {
    kx += resident;
    while (kx >= g.px.M) kx -= g.px.M, b++;
    if (b >= (int)gridDim.y) return;
    const long long n = 3LL * (g.multi ? rhs[b].Ny : g.Ny) * (g.multi ? rhs[b].Nz : g.Nz);
    const float2* p = grid + (long long)b * g.vb + kx * n;
    const unsigned long long a = reinterpret_cast<unsigned long long>(p), a16 = a & ~15ull;
    const unsigned bytes = (unsigned)(n * sizeof(float2) + (a - a16)) & ~15u;
    if (bytes) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a16), "r"(bytes) : "memory");
}

template <int MY, int MZ, int NT>
__global__ void __launch_bounds__(NT, NT < Plane<MY, MZ>::NT ? 2 : 0) k_xpass2p(Geom g, const RhsVecs<float>* __restrict__ rhs,
                                                                const float2* __restrict__ green,
                                                                const float2* __restrict__ twy,
                                                                const float2* __restrict__ twz,
                                                                float2* __restrict__ grid) {
    using T = float;
    using PL = Plane<MY, MZ>;
    using Y = typename PL::Y;
    using Z = typename PL::Z;
    constexpr int ZP = PL::ZP, LZ = Z::LX;
    constexpr int B1 = Y::R1, B2 = Y::R2, BH = Y::RH, A1 = Z::R1, A2 = Z::R2, AH = Z::RH;
    constexpr int CS = MY * ZP;  // from component to component
    static_assert(B2 == 8 && A2 % 2 == 0, "plans of the plane");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* s = reinterpret_cast<float2*>(smem_raw);
    float2* stwy = s + 3 * CS;
    float2* stwz = stwy + MY;
    const int b = blockIdx.y, kx = blockIdx.x;
    const SolveState* st = rhs[b].st;
    const int Ny = g.multi ? rhs[b].Ny : g.Ny, Nz = g.multi ? rhs[b].Nz : g.Nz;
    if (g.multi) green = rhs[b].green;
    stage_tw<T>(stwy, twy, MY);
    stage_tw<T>(stwz, twz, MZ);
    const int Mx = g.px.M, fx = fold(kx, Mx);
    float2* gp = grid + (long long)b * g.vb + (long long)kx * 3 * Ny * Nz;
    grid_dep_wait();
    if (g.early == 1) grid_dep_release();
    // not for the small planes, which are several to an SM and whose grid stays in L2 (a
    // prefetch of planes that already run: 64 x 16 x 16, sixteen right-hand sides 107.5 us a
    // step with it, 105.2 without; 40 x 20 x 10 61.9 and 60.7); in pairs the next plane is two
    // blocks an SM away (13 batches: within 0.6% of the distance of one, either way)
    if constexpr (PL::NT == 512) {
        if (threadIdx.x == 0) prefetch_plane(g, rhs, grid, kx, b, NT < PL::NT ? 2 * g.sms : g.sms);
    }
    // 1: rows y = jj + 8 r < Ny of column z
    for (int w = threadIdx.x; w < 3 * B2 * LZ; w += NT) {
        const int z = w % LZ, jj = (w / LZ) % B2, c = w / (LZ * B2);
        const float2* src = gp + (c * Ny + jj) * Nz + z;
        float2 v[B1];
#pragma unroll
        for (int r = 0; r < BH; r++) v[r] = z < Nz && jj + B2 * r < Ny ? src[B2 * r * Nz] : czero<T>();
        BflyIn<B1, -1, T, BH>::run(v);
        float2* d = s + c * CS + jj * B1 * ZP + z;
#pragma unroll
        for (int q = 0; q < B1; q++) d[q * ZP] = v[q];
    }
    if (rhs_done(st)) return;  // checked after the first loads are issued: nothing is written yet
    __syncthreads();
    // 2: rows j + B1 r of the columns jz + A2 k; row j + B1 q is then ky
    for (int w = threadIdx.x; w < 3 * B1 * A2; w += NT) {
        const int j = (w / 2) % B1, c = w / (B1 * A2), jz = w % 2 + 2 * (w / (2 * B1) % (A2 / 2));
        float2* d = s + c * CS + j * ZP + jz;
        float2 v[AH][B2];
#pragma unroll
        for (int k = 0; k < AH; k++) {
            const bool in = AH * A2 == LZ || jz + A2 * k < LZ;
#pragma unroll
            for (int r = 0; r < B2; r++) v[k][r] = in ? d[r * B1 * ZP + A2 * k] : czero<T>();
        }
        float2 tw[B2];
#pragma unroll
        for (int r = 1; r < B2; r++) tw[r] = stwy[r * j];
#pragma unroll
        for (int k = 0; k < AH; k++) {
#pragma unroll
            for (int r = 1; r < B2; r++) v[k][r] = cmul<T>(v[k][r], tw[r]);
            Bfly<B2, -1, T>::run(v[k]);
        }
#pragma unroll
        for (int q = 0; q < B2; q++) {
            float2 u[A1];
#pragma unroll
            for (int k = 0; k < AH; k++) u[k] = v[k][q];
            BflyIn<A1, -1, T, AH>::run(u);
#pragma unroll
            for (int k = 0; k < A1; k++) d[q * B1 * ZP + A2 * k] = u[k];
        }
    }
    __syncthreads();
    // 3: row = ky
    for (int w = threadIdx.x; w < A1 * MY; w += NT) {
        const int row = mirrored_row<MY>(w % MY), j = w / MY;
        SpectralRow<T, A1, A2, MZ, A2 < 5 ? A2 : 5> sp(GreenRow<T>(green, g, fx, fold(row, MY)), j);
        float2* d = s + row * ZP + A2 * j;
        float2 X[3][A2], tw[A2];
#pragma unroll
        for (int r = 1; r < A2; r++) tw[r] = stwz[r * j];
#pragma unroll
        for (int c = 0; c < 3; c++) {
            load_pairs<A2>(d + c * CS, X[c]);
#pragma unroll
            for (int r = 1; r < A2; r++) X[c][r] = cmul<T>(X[c][r], tw[r]);
            Bfly<A2, -1, T>::run(X[c]);
        }
        sp.apply(X, half_mask(kx, Mx), half_mask(row, MY));
#pragma unroll
        for (int c = 0; c < 3; c++) {
            Bfly<A2, +1, T>::run(X[c]);
#pragma unroll
            for (int r = 1; r < A2; r++) X[c][r] = cmulc<T>(tw[r], X[c][r]);
            store_pairs<A2>(d + c * CS, X[c]);
        }
    }
    __syncthreads();
    // 4: columns jz + A2 k < LZ of the rows j + B1 q, then rows j + B1 r
    for (int w = threadIdx.x; w < 3 * B1 * A2; w += NT) {
        const int j = (w / 2) % B1, c = w / (B1 * A2), jz = w % 2 + 2 * (w / (2 * B1) % (A2 / 2));
        float2* d = s + c * CS + j * ZP + jz;
        float2 v[AH][B2];
#pragma unroll
        for (int q = 0; q < B2; q++) {
            float2 u[A1];
#pragma unroll
            for (int k = 0; k < A1; k++) u[k] = d[q * B1 * ZP + A2 * k];
            Bfly<A1, +1, T>::run(u);
#pragma unroll
            for (int k = 0; k < AH; k++) v[k][q] = u[k];
        }
        float2 tw[B2];
#pragma unroll
        for (int r = 1; r < B2; r++) tw[r] = stwy[r * j];
#pragma unroll
        for (int k = 0; k < AH; k++) {
            Bfly<B2, +1, T>::run(v[k]);
#pragma unroll
            for (int r = 1; r < B2; r++) v[k][r] = cmulc<T>(tw[r], v[k][r]);
            if (AH * A2 == LZ || jz + A2 * k < LZ) {
#pragma unroll
                for (int r = 0; r < B2; r++) d[r * B1 * ZP + A2 * k] = v[k][r];
            }
        }
    }
    __syncthreads();
    if (g.early == 2) grid_dep_release();  // the next kernel's blocks start during the last stage
    // 5: rows y = jj + 8 r < Ny of column z
    for (int w = threadIdx.x; w < 3 * B2 * LZ; w += NT) {
        const int z = w % LZ, jj = (w / LZ) % B2, c = w / (LZ * B2);
        const float2* d = s + c * CS + jj * B1 * ZP + z;
        float2 v[B1];
#pragma unroll
        for (int q = 0; q < B1; q++) v[q] = d[q * ZP];
        Bfly<B1, +1, T>::run(v);
        float2* dst = gp + (c * Ny + jj) * Nz + z;
#pragma unroll
        for (int r = 0; r < BH; r++)
            if (z < Nz && jj + B2 * r < Ny) dst[B2 * r * Nz] = v[r];
    }
}

// ------------------------------------------------------------ launchers
inline cudaError_t allow_smem(const void* k, size_t smem) {
    return smem > 48 * 1024 ? cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)
                            : cudaSuccess;
}
// launches on the stream, early where the geometry asks for it
template <typename T, typename... P, typename... A>
cudaError_t launch_axis(const PassArgs<T>& a, void (*k)(Geom, P...), dim3 grid, int nt, size_t smem, A... args) {
    // where the next kernel's blocks start early they take the room the last blocks
    // of this one leave, not an even share of the SMs: a loss for launches of many
    // waves (96 x 96 x 24, eight right-hand sides: 604 us a step without, 625 with)
    // and for the FP64 kernels, which fill the FP64 pipe of the SMs they are on
    // (10 x 17 x 25 product: 104 -> 210 us with it, released after the wait)
    Geom g = early_geom(a.g, (long long)grid.x * grid.y);
    const long long blocks = (long long)grid.x * grid.y;
    if (sizeof(T) == 4 ? blocks > 8LL * g.sms : true) g.early = 0;
    const cudaError_t e = launch_early(g.early != 0, k, grid, dim3(nt), smem, a.stream, g, args...);
    return e != cudaSuccess ? e : cudaGetLastError();
}

// the x and y kernels of one length
template <typename T, int M> struct AxisLaunch {
    static dim3 lines(const PassArgs<T>& a, int ct) {
        return dim3((unsigned)((3LL * a.g.Ny * a.g.Nz + ct - 1) / ct), a.nrhs);
    }
    template <int SRC, int CT> static cudaError_t fwd1(const PassArgs<T>& a, int rows) {
        // tiles per block: all blocks of the launch resident at once
        dim3 grid = lines(a, CT);
        const long long tiles = (long long)grid.x * a.nrhs, room = 152LL * axis_minb<M, CT>();
        const unsigned per = (unsigned)((tiles + room - 1) / room);
        grid.x = (grid.x + per - 1) / per;
        return launch_axis(a, k_xfwd<T, SRC, M, CT>, grid, axis_threads<M, CT>(), XTile<T, M, CT>::smem, a.rhs, a.twx,
                           a.cellmap, a.grid, rows, a.slot, a.prod_nblk, a.in);
    }
    template <int SRC> static cudaError_t fwd(const PassArgs<T>& a, int rows) {
        if constexpr (sizeof(T) == 4) {
            if (axis_tile_fwd(a.g) == 16) return fwd1<SRC, 16>(a, rows);
        }
        return fwd1<SRC, 8>(a, rows);
    }
    template <int SRC, int SNK, int CT> static cudaError_t inv1(const PassArgs<T>& a, int rows) {
        return launch_axis(a, k_xinv<T, SRC, SNK, M, CT>, lines(a, CT), sink_threads<T, M, CT>(), XTile<T, M, CT>::smem,
                           a.rhs, a.twx, a.cellmap, (const cx<T>*)a.grid, rows, a.out);
    }
    template <int SRC, int SNK> static cudaError_t inv(const PassArgs<T>& a, int rows) {
        if constexpr (sizeof(T) == 4) {
            if (axis_tile_inv(a.g) == 16) return inv1<SRC, SNK, 16>(a, rows);
        }
        return inv1<SRC, SNK, 8>(a, rows);
    }
    template <int SIGN> static cudaError_t yaxis(const PassArgs<T>& a) {
        constexpr int CT = sizeof(T) == 4 ? 16 : 8;
        const dim3 grid((unsigned)((3LL * a.g.px.M * a.g.Nz + CT - 1) / CT), a.nrhs);
        return launch_axis(a, k_yaxis<T, SIGN, M, CT>, grid, axis_threads<M, CT>(), XTile<T, M, CT>::smem, a.rhs, a.twy,
                           a.grid);
    }
    // op: AxisOp; mode: SrcMode / SnkMode; rows: AXIS_XFWD / AXIS_XINV
    static cudaError_t run(int op, int mode, int rows, const PassArgs<T>& a) {
        if (op == AXIS_YFWD) return yaxis<-1>(a);
        if (op == AXIS_YINV) return yaxis<+1>(a);
        if constexpr (is_dd<T>) {  // the double-float product forms residuals only
            return op == AXIS_XFWD ? fwd<SRC_P>(a, rows) : inv<SRC_P, SNK_RES>(a, rows);
        } else if constexpr (sizeof(T) == 4) {  // products and the deferred step
            if (op == AXIS_XFWD) {
                switch (mode) {
                    case SRC_EXT: return fwd<SRC_EXT>(a, rows);
                    case SRC_IN: return fwd<SRC_IN>(a, rows);
                    case SRC_TUPD: return fwd<SRC_TUPD>(a, rows);
                    default: return fwd<SRC_PUPD_DEF>(a, rows);
                }
            }
            switch (mode) {
                case SNK_EXT: return inv<SRC_EXT, SNK_EXT>(a, rows);
                case SNK_OUT: return inv<SRC_IN, SNK_OUT>(a, rows);
                case SNK_AP: return inv<SRC_PUPD, SNK_AP>(a, rows);
                default: return inv<SRC_TUPD, SNK_AT_DEF>(a, rows);
            }
        } else {
            if (op == AXIS_XFWD) {
                switch (mode) {
                    case SRC_EXT: return fwd<SRC_EXT>(a, rows);
                    case SRC_IN: return fwd<SRC_IN>(a, rows);
                    case SRC_PUPD: return fwd<SRC_PUPD>(a, rows);
                    case SRC_TUPD: return fwd<SRC_TUPD>(a, rows);
                    default: return fwd<SRC_P>(a, rows);
                }
            }
            switch (mode) {
                case SNK_EXT: return inv<SRC_EXT, SNK_EXT>(a, rows);
                case SNK_OUT: return inv<SRC_IN, SNK_OUT>(a, rows);
                case SNK_ALB: return inv<SRC_IN, SNK_ALB>(a, rows);
                case SNK_AP: return inv<SRC_PUPD, SNK_AP>(a, rows);
                case SNK_AT: return inv<SRC_TUPD, SNK_AT>(a, rows);
                default: return inv<SRC_P, SNK_RES>(a, rows);
            }
        }
    }
};

template <typename T, int M> struct ZprodLaunch {
    template <int RT> static cudaError_t run1(const PassArgs<T>& a) {
        const dim3 grid((unsigned)(((long long)a.g.px.M * a.g.py.M + RT - 1) / RT), a.nrhs);
        return launch_axis(a, k_zprod<T, M, RT>, grid, zprod_threads<T, M, RT>(), ZTile<T, M, RT>::smem, a.rhs, a.green,
                           a.twz, a.grid);
    }
    // rows a block: the full tile where that leaves every SM several blocks, else 8
    static constexpr int kWide = zprod_wide<T, M>();
    static cudaError_t run(const PassArgs<T>& a) {
        const long long rows = (long long)a.g.px.M * a.g.py.M * a.nrhs;
        return rows >= kWide * (kZFused<T> ? 4LL : 2LL) * 152 ? run1<kWide>(a) : run1<8>(a);
    }
    static cudaError_t configure() {
        cudaError_t e = allow_smem((const void*)k_zprod<T, M, kWide>, ZTile<T, M, kWide>::smem);
        return e != cudaSuccess ? e : allow_smem((const void*)k_zprod<T, M, 8>, ZTile<T, M, 8>::smem);
    }
};

template <int MY, int MZ> struct PlaneLaunch {
    using PL = Plane<MY, MZ>;
    template <int NT> static cudaError_t run1(const PassArgs<float>& a) {
        return launch_axis(a, k_xpass2p<MY, MZ, NT>, dim3(a.g.px.M, a.nrhs), NT, PL::smem, a.rhs, a.green, a.twy,
                           a.twz, a.grid);
    }
    // Pairs of blocks where the planes that run side by side (the batch's, over its
    // branches) are more than two an SM: steps of 40 x 40 x 12, eight right-hand sides
    // 75 -> 64 us, of 45 x 33 x 19, four 65 -> 59, of 64 x 64 x 16, four 83 -> 76 and
    // eight 157 -> 144; below, a plane's own time counts (64 x 64 x 16, one 34 -> 40,
    // two 49 -> 54 with pairs).
    static cudaError_t run(const PassArgs<float>& a) {
        if constexpr (PL::kPair) {
            const int sms = a.g.sms > 0 ? a.g.sms : 152;
            const long long planes = (long long)a.g.px.M * std::max(a.nrhs, a.g.batch);
            if (planes > 2LL * sms) return run1<256>(a);
        }
        return run1<PL::NT>(a);
    }
    static cudaError_t configure() {
        cudaError_t e = allow_smem((const void*)k_xpass2p<MY, MZ, PL::NT>, PL::smem);
        if constexpr (PL::kPair) {
            if (e == cudaSuccess) e = allow_smem((const void*)k_xpass2p<MY, MZ, 256>, PL::smem);
        }
        return e;
    }
};

}  // namespace dev
}  // namespace tdda
