// Fused, shared-memory tiled kernels of the pyramid and of one solver level (strict mode).
//
// Each kernel computes a TX x TY tile of its outputs. Intermediate planes live only in shared
// memory, over the tile plus the halo the later stages need, and are recomputed in the halo rather
// than exchanged between CTAs. Every element still takes the reference's own operation order
// (flow/conv.rs for the separable passes, flow.rs for the solver steps), so the results are bit
// identical to the unfused kernels and to the reference CPU path.
#include "kernels.cuh"
#include "level.cuh"
#include "luma.cuh"

namespace tw {
TW_VARIANT_BEGIN

// ---- a step of a pyramid (flow.rs:248-275): blur5, the band and the next size, in one launch ---------------

// flow/extras.rs:64-72: v >= 0.95 gives 1, else 0 (a NaN gives 0)
__device__ __forceinline__ float binarized(float v) { return v >= 0.95f ? 1.0f : 0.0f; }

// The tile of a step: T x T source pixels, their blur with one column and row more (the resample's second
// taps) and the halo of the blur. The row pass takes the rows y and y + HP as a pair (rows a lane apart, so
// that the lanes' loads fall into different banks), the column pass two columns next to each other; 4 outputs
// per thread. Strides keep the scalar accesses free of conflicts and the pairs aligned.
template <int T>
struct PyramidGeom {
    static constexpr int N = 3, HALO = N - 1, R = 4;
    static constexpr int OUT = T + 1, SEG = (OUT + R - 1) / R, RC = T + 8, RS = RC + 1;
    static constexpr int HP = (OUT + 2 * HALO + 1) / 2, HS = R * SEG + 2, HROWS = R * SEG + 2 * HALO;
    static constexpr int CP = (OUT + 1) / 2, VS = 2 * CP + 1, VROWS = R * SEG;
    static constexpr int DEN = R * SEG, CELLS = T + 2;
    static_assert(2 * HP <= HROWS && R * SEG + 2 * HALO <= RC && HS % 2 == 0, "the planes hold every run");
    static constexpr int O_H = 2 * HP * RS, O_V = O_H + HROWS * HS, O_TAB = (O_V + VROWS * VS + 1) / 2 * 2;
    static constexpr int FLOATS = O_TAB + 2 * (2 * DEN + 2 * CELLS);
};

// The region's rows r, r + 1, ... (a warp each) and then its last 8 columns, through at(X, Y)
template <int T, int NT, class At>
__device__ __forceinline__ void pyramid_load(float* s_in, int X0, int Y0, int w, int h, At at) {
    using G = PyramidGeom<T>;
    const int tid = threadIdx.x;
    constexpr int ROWS = 2 * G::HP, PER = NT / T, A = (ROWS + PER - 1) / PER, B = (ROWS * 8 + NT - 1) / NT;
    float v[A + B];
    const int c = tid % T, r0 = tid / T, X = X0 - G::HALO + c;
#pragma unroll
    for (int j = 0; j < A; j++) {
        const int Y = Y0 - G::HALO + r0 + j * PER;
        v[j] = X >= 0 && X < w && Y >= 0 && Y < h ? at(X, Y) : 0.0f;
    }
#pragma unroll
    for (int j = 0; j < B; j++) {
        const int e = tid + j * NT, X1 = X0 - G::HALO + T + e % 8, Y = Y0 - G::HALO + e / 8;
        v[A + j] = e % 8 < G::OUT + 2 * G::HALO - T && X1 < w && Y >= 0 && Y < h ? at(X1, Y) : 0.0f;
    }
#pragma unroll
    for (int j = 0; j < A; j++)
        if (r0 + j * PER < ROWS) s_in[(r0 + j * PER) * G::RS + c] = v[j];
#pragma unroll
    for (int j = 0; j < B; j++) {
        const int e = tid + j * NT;
        if (e < ROWS * 8) s_in[e / 8 * G::RS + T + e % 8] = v[A + j];
    }
}

// One step: blur = blur5(src) (src a plane, or the luma of an engine image computed on the way,
// prep.rs:168-235), band = src - blur and its transpose, and dst = blur resampled to dw x dh
// (sample.rs:91-112): each output belongs to the tile of its first tap; the sizes are such that a step is at
// least 1 (dw = w / 2, and no less than 2). bin_in, bin_out: a mask's pyramid (flow/extras.rs:76-123), src and
// dst binarized. sm: PyramidGeom<T>::FLOATS floats.
template <int T, int NT>
__device__ __forceinline__ void pyramid_step(const PyramidStep& P, float* sm, int X0, int Y0) {
    using G = PyramidGeom<T>;
    constexpr int R = G::R;
    float *s_in = sm, *s_h = sm + G::O_H, *s_v = sm + G::O_V;
    float2 *s_dx = (float2*)(sm + G::O_TAB), *s_dy = s_dx + G::DEN, *s_cx = s_dy + G::DEN, *s_cy = s_cx + G::CELLS;
    const int w = P.w, h = P.h, tid = threadIdx.x;
    if (P.luma_src) {
        const int fmt = P.fmt, mode = P.luma_mode;
        const void* img = P.luma_src;
        auto load = [&](auto at) { pyramid_load<T, NT>(s_in, X0, Y0, w, h, at); };
        // (the plain luma of each depth without the tests of a depth and a mode per sample)
        if (mode == 0 && fmt == 0) load([&](int X, int Y) { return luma_px(img, 0, (long)Y * w + X, 0); });
        else if (mode == 0 && fmt == 1) load([&](int X, int Y) { return luma_px(img, 1, (long)Y * w + X, 0); });
        else if (mode == 0) load([&](int X, int Y) { return luma_px(img, 2, (long)Y * w + X, 0); });
        else load([&](int X, int Y) { return luma_px(img, fmt, (long)Y * w + X, mode); });
    } else if (P.bin_in) {
        pyramid_load<T, NT>(s_in, X0, Y0, w, h, [&](int X, int Y) { return binarized(P.src[(long)Y * w + X]); });
    } else {
        pyramid_load<T, NT>(s_in, X0, Y0, w, h, [&](int X, int Y) { return P.src[(long)Y * w + X]; });
    }
    // the outputs xa .. (nx of them), ya .. (ny) whose first tap can lie in the tile: its ends over the step
    int xa = 0, nx = 0, ya = 0, ny = 0;
    if (P.dst) {
        // (rounded correctly in the fast mode too: a quotient below an output's number would leave it to no tile)
        auto range = [](int at, int len, float step, int n, int& lo, int& count) {
            lo = (int)__fdiv_rn((float)at, step);
            count = min((at + T < len - 1 ? min((int)__fdiv_rn((float)(at + T), step), n - 1) : n - 1) - lo + 1, G::CELLS);
        };
        range(X0, w, P.sx, P.dw, xa, nx);
        range(Y0, h, P.sy, P.dh, ya, ny);
    }
    // the tables: border weights, and the cells of the outputs (first tap in the tile, or -1; fraction)
    auto cell_at = [](int i, float step, int len, int at) {
        int k;
        float f;
        cell((float)i * step, len, k, f);
        k -= at;
        return make_float2(__int_as_float(k >= 0 && k < T ? k : -1), f);
    };
    for (int i = tid; i < G::DEN; i += NT) {
        s_dx[i] = border_den<G::N>(X0 + i, w, P.t.k);
        s_dy[i] = border_den<G::N>(Y0 + i, h, P.t.k);
    }
    for (int i = NT - 1 - tid; i < G::CELLS; i += NT) {
        if (i < nx) s_cx[i] = cell_at(xa + i, P.sx, w, X0);
        if (i < ny) s_cy[i] = cell_at(ya + i, P.sy, h, Y0);
    }
    __syncthreads();
    for (int e = tid; e < G::HP * G::SEG; e += NT) {
        const int seg = e / G::HP, y = e - seg * G::HP;
        const float *a = s_in + y * G::RS + seg * R, *b = a + G::HP * G::RS;
        float2 in[R + 2 * G::N - 2], o[R];
#pragma unroll
        for (int j = 0; j < R + 2 * G::N - 2; j++) in[j] = make_float2(a[j], b[j]);
        single_run<G::N, R, false>(in, X0 + seg * R, w, P.t, s_dx + seg * R, o);
        float* out = s_h + y * G::HS + seg * R;
#pragma unroll
        for (int r = 0; r < R; r++) {
            out[r] = o[r].x;
            out[G::HP * G::HS + r] = o[r].y;
        }
    }
    __syncthreads();
    for (int e = tid; e < G::CP * G::SEG; e += NT) {
        const int seg = e / G::CP, c = e - seg * G::CP;
        float2 in[R + 2 * G::N - 2], o[R];
#pragma unroll
        for (int j = 0; j < R + 2 * G::N - 2; j++) in[j] = *(const float2*)(s_h + (seg * R + j) * G::HS + 2 * c);
        if (P.above_first) single_run<G::N, R, true>(in, Y0 + seg * R, h, P.t, s_dy + seg * R, o);
        else single_run<G::N, R, false>(in, Y0 + seg * R, h, P.t, s_dy + seg * R, o);
#pragma unroll
        for (int r = 0; r < R; r++) {
            s_v[(seg * R + r) * G::VS + 2 * c] = o[r].x;
            s_v[(seg * R + r) * G::VS + 2 * c + 1] = o[r].y;
        }
    }
    __syncthreads();
    const float* centre = s_in + G::HALO * G::RS + G::HALO;
    const int u = tid % T, v0 = tid / T;
    if (P.band && X0 + u < w) {
        float* out = P.band + (long)(Y0 + v0) * w + X0 + u;
#pragma unroll
        for (int j = 0; j < T; j += NT / T)
            if (Y0 + v0 + j < h) out[(long)j * w] = centre[(v0 + j) * G::RS + u] - s_v[(v0 + j) * G::VS + u];
    }
    if (P.band_t && Y0 + u < h) {  // element (x, y) at [x * h + y], for the column sweeps
        float* out = P.band_t + (long)(X0 + v0) * h + Y0 + u;
#pragma unroll
        for (int j = 0; j < T; j += NT / T)
            if (X0 + v0 + j < w) out[(long)j * h] = centre[u * G::RS + v0 + j] - s_v[u * G::VS + v0 + j];
    }
    constexpr int COLS = T / 2 + 2;  // the outputs across a tile at a step of 2
    for (int x0 = 0; x0 < nx; x0 += COLS) {
        for (int e = tid; e < COLS * ny; e += NT) {
            const int y = e / COLS, x = x0 + e - y * COLS;
            if (x >= nx) continue;
            const float2 cx = s_cx[x], cy = s_cy[y];
            const int ix = __float_as_int(cx.x), iy = __float_as_int(cy.x);
            if (ix < 0 || iy < 0) continue;
            const float* q = s_v + iy * G::VS + ix;
            const float top = (q[1] - q[0]) * cx.y + q[0], bot = (q[G::VS + 1] - q[G::VS]) * cx.y + q[G::VS];
            const float r = (bot - top) * cy.y + top;
            P.dst[(long)(ya + y) * P.dw + xa + x] = P.bin_out ? binarized(r) : r;
        }
    }
}

// Bound by issue at the large sizes (130 instructions per 8 bit pixel, 200 before) and by latency at the small
// ones. A step was two launches with the blur's plane stored in between, scalar passes and a test per tap:
// 1920 x 1080 to 960 x 540 22 us, now 17; 480 x 270 11, now 7.
__global__ void __launch_bounds__(PYRAMID_THREADS_32) k_pyramid_step_32(const __grid_constant__ PyramidStep P) {
    __shared__ __align__(16) float sm[PyramidGeom<32>::FLOATS];
    pyramid_step<32, PYRAMID_THREADS_32>(P, sm, blockIdx.x * 32, blockIdx.y * 32);
}
__global__ void __launch_bounds__(PYRAMID_THREADS_16) k_pyramid_step_16(const __grid_constant__ PyramidStep P) {
    __shared__ __align__(16) float sm[PyramidGeom<16>::FLOATS];
    pyramid_step<16, PYRAMID_THREADS_16>(P, sm, blockIdx.x * 16, blockIdx.y * 16);
}

// The last steps of a pyramid, whose planes are one tile of 64 x 64 each: one block, a step after the other
// (each plane but the first is this block's own of the step before).
__global__ void __launch_bounds__(PYRAMID_TAIL_THREADS) k_pyramid_tail(const __grid_constant__ PyramidTail P) {
    extern __shared__ __align__(16) float tail_sm[];
    for (int i = 0; i < P.n; i++) {
        pyramid_step<PYRAMID_TAIL, PYRAMID_TAIL_THREADS>(P.step[i], tail_sm, 0, 0);
        __syncthreads();
    }
}
size_t pyramid_tail_smem() { return PyramidGeom<PYRAMID_TAIL>::FLOATS * sizeof(float); }

// ---- one solver level: the tile geometry of its kernels ----------------------------------------------

// Stores of res[0 .. R-1] along a shared memory line
template <int R, class V>
__device__ __forceinline__ void put_run(V* out, int stride, const V* res) {
#pragma unroll
    for (int r = 0; r < R; r++) out[r * stride] = res[r];
}

// The border weight sums (border_den) of n consecutive line indices from i0 on: entry t of the block's
// table (run_pass reads them for the outputs near the line's ends). Tables are filled one after the
// other by consecutive threads; returns the index past this one.
template <int N>
__device__ __forceinline__ int fill_den(float2* den, int first, int n, int i0, int len, const Taps& k) {
    for (int t = (int)threadIdx.x - first; t < n; t += blockDim.x)
        if (t >= 0) den[t] = border_den<N>(i0 + t, len, k.k);
    return first + n;
}
// Whether a tile of w0 x h0 outputs at (X0, Y0) of a w x h level has border outputs in a filter chain that
// reaches `reach` pixels past it
__device__ __forceinline__ bool at_border(int X0, int Y0, int w0, int h0, int reach, int w, int h) {
    return X0 < reach || Y0 < reach || X0 + w0 > w - reach || Y0 + h0 > h - reach;
}

// ---- one solver level: gradient, tensor and its blur (flow.rs:1275-1277) ---------------------------

template <int TX, int TY>
struct InitGeom {
    static constexpr int HALO = 7, R = 4;
    static constexpr int RW = TX + 2 * HALO, RH = TY + 2 * HALO;
    static constexpr int RS = RW | 1, HS = TX | 1;  // row strides (odd: a warp's lanes on distinct rows hit distinct banks)
    static constexpr int NDEN = TX + TY;
    static constexpr size_t SMEM = sizeof(float2) * (RH * RS + RH * HS + NDEN) + sizeof(float) * (RH * RS + RH * HS);
    static_assert(TX % R == 0 && TY % R == 0, "whole runs");
};

// The tasks of the passes below, each the outputs of one run; false when they are done, true (nothing
// written) when the run needs the general rule: the same task again with SLOW, out of line, so that the
// main path carries no calls.
template <int TX, int TY, bool SLOW>
__device__ __forceinline__ bool init_row(const LevelInitArgs& P, const float2* t, const float* t2, float2* o_h, float* o_h2,
                                         const float2* den, int i0) {
    constexpr int R = InitGeom<TX, TY>::R;
    float2 o[R];
    float o2[R];
    if (h_pass<SLOW, 8, R>(t, i0, P.w, P.g7, den, o)) return true;
    if (h_pass<SLOW, 8, R>(t2, i0, P.w, P.g7, den, o2)) return true;
    put_run<R>(o_h, 1, o);
    put_run<R>(o_h2, 1, o2);
    return false;
}
template <int TX, int TY, bool SLOW>
__device__ __forceinline__ bool init_column(const LevelInitArgs& P, const float2* h, const float* h2, const float2* den,
                                            int x, int y0) {
    using G = InitGeom<TX, TY>;
    constexpr int R = G::R;
    float2 o[R];
    float o2[R];
    if (v_pass<SLOW, 8, R>(h, G::HS, y0, P.h, P.g7, den, P.af, o)) return true;
    if (v_pass<SLOW, 8, R>(h2, G::HS, y0, P.h, P.g7, den, P.af, o2)) return true;
#pragma unroll
    for (int r = 0; r < R; r++)  // with the determinant of new_disp beside the tensor
        if (y0 + r < P.h) P.tensor[(y0 + r) * P.w + x] = make_float4(o[r].x, o[r].y, o2[r], o[r].y * o[r].y - o2[r] * o[r].x);
    return false;
}
template <int TX, int TY>
__device__ __noinline__ void init_row_slow(const LevelInitArgs& P, const float2* t, const float* t2, float2* o_h, float* o_h2,
                                           const float2* den, int i0) {
    init_row<TX, TY, true>(P, t, t2, o_h, o_h2, den, i0);
}
template <int TX, int TY>
__device__ __noinline__ void init_column_slow(const LevelInitArgs& P, const float2* h, const float* h2, const float2* den, int x,
                                              int y0) {
    init_column<TX, TY, true>(P, h, h2, den, x, y0);
}

template <int TX, int TY>
__device__ __forceinline__ void level_init_body(const LevelInitArgs& P) {
    using G = InitGeom<TX, TY>;
    constexpr int N = 8, R = G::R;
    extern __shared__ __align__(16) float sm[];
    float2* s_t = (float2*)sm;            // RH x RS: the tensor's first two channels
    float2* s_h = s_t + G::RH * G::RS;    // RH x HS: their horizontal pass
    float2* den_x = s_h + G::RH * G::HS;  // the weight sums of the tile's columns and rows
    float2* den_y = den_x + TX;
    float* s_t2 = (float*)(den_y + TY);   // the third channel, the same two planes
    float* s_h2 = s_t2 + G::RH * G::RS;
    const int w = P.w, h = P.h;
    const int X0 = blockIdx.x * TX, Y0 = blockIdx.y * TY;
    const int gx0 = X0 - G::HALO, gy0 = Y0 - G::HALO;
    const int nt = blockDim.x;
    if (at_border(X0, Y0, TX, TY, N, w, h)) {
        const int t = fill_den<N>(den_x, 0, TX, X0, w, P.g7);
        fill_den<N>(den_y, t, TY, Y0, h, P.g7);
    }
    // the tile's own pixels: the flow from the coarser level, the gradient, calc_b of the first iteration
    const bool zero = P.src && zero_at_level(P.any, P.l + 1, P.start);
    for (int e = threadIdx.x; e < TX * TY; e += nt) {
        const int r = e / TX, c = e - r * TX;
        const int x = X0 + c, y = Y0 + r;
        if (x >= w || y >= h) continue;
        const int i = y * w + x;
        float2 f;
        if (P.src) {
            f = upsample_at(P.src, P.sw, P.sh, P.up, zero, P.damp_now, P.damp, x, y);
            P.f[i] = f;
        } else {
            f = P.f[i];
        }
        const float2 g = gradient_at(P.img, P.mask_x, w, h, x, y);
        P.grad[i] = g;
        const float i1 = __ldg(P.img + i);
        float2 b;
        calc_b_run<1>(P.i0, P.mask_y, w, h, x, y, &f, &i1, &g, &b);
        P.b_out[(long)y * P.bp + x] = b;
    }
    // the tensor (flow.rs:319-328) over the tile and the blur's halo
    for (int e = threadIdx.x; e < G::RW * G::RH; e += nt) {
        const int r = e / G::RW, c = e - r * G::RW;
        const int x = gx0 + c, y = gy0 + r;
        float2 t = outside_value<float2>();
        float t2 = outside_value<float>();
        if (x >= 0 && x < w && y >= 0 && y < h) {
            const float2 g = gradient_at(P.img, P.mask_x, w, h, x, y);
            t = make_float2(g.x * g.x, g.x * g.y);
            t2 = g.y * g.y;
        }
        s_t[r * G::RS + c] = t;
        s_t2[r * G::RS + c] = t2;
    }
    __syncthreads();
    // blur7 of the tensor: along the region's rows at the tile's columns, a lane per row
    for (int e = threadIdx.x; e < G::RH * (TX / R); e += nt) {
        const int r = e % G::RH, c0 = (e / G::RH) * R;
        const float2* t = s_t + r * G::RS + c0;
        const float* t2 = s_t2 + r * G::RS + c0;
        float2* o = s_h + r * G::HS + c0;
        float* o2 = s_h2 + r * G::HS + c0;
        if (init_row<TX, TY, false>(P, t, t2, o, o2, den_x + c0, X0 + c0)) init_row_slow<TX, TY>(P, t, t2, o, o2, den_x + c0, X0 + c0);
    }
    __syncthreads();
    // then along the tile's columns, a lane per column
    for (int e = threadIdx.x; e < TX * (TY / R); e += nt) {
        const int c = e % TX, r0 = (e / TX) * R;
        if (X0 + c >= w || Y0 + r0 >= h) continue;
        const float2* t = s_h + r0 * G::HS + c;
        const float* t2 = s_h2 + r0 * G::HS + c;
        if (init_column<TX, TY, false>(P, t, t2, den_y + r0, X0 + c, Y0 + r0))
            init_column_slow<TX, TY>(P, t, t2, den_y + r0, X0 + c, Y0 + r0);
    }
}

#define TW_LEVEL_INIT(TX, TY)                                                                            \
    __global__ void __launch_bounds__(LEVEL_INIT_MAX_THREADS, 2) k_level_init_##TX##x##TY(               \
        const __grid_constant__ LevelInitArgs P) {                                                      \
        level_init_body<TX, TY>(P);                                                                     \
    }
TW_LEVEL_INIT(16, 16)
TW_LEVEL_INIT(32, 32)
#undef TW_LEVEL_INIT

size_t level_init_smem(int tile) { return tile == LEVEL_TILE_16x16 ? InitGeom<16, 16>::SMEM : InitGeom<32, 32>::SMEM; }

// ---- one solver iteration (flow.rs:1278-1282): calc_b, blur7 of B, new_disp, blur5 of the flow -----
// mask_y (may be null): the level mask of Y of a layered solve
//
// calc_b depends only on the flow at its own pixel, so it is computed once per pixel where the flow
// is made: k_level_init for the level's first iteration, each iteration's epilogue for the next one
// (k_calc_b_pitched after the level's block matching).
//
// Halos: the flow's blur5 needs new_disp on the tile + 5; new_disp needs blurred B there, which
// needs B on the tile + 12. The tile is TX x TY outputs (a template: the host picks the shape per
// level size). A thread computes R consecutive outputs along a pass (run_pass) with both channels in
// one packed operation. The vertical passes end in registers: blur7's runs go straight into new_disp,
// blur5's into the new flow and calc_b of the next iteration. Horizontal passes give each lane of a
// warp its own row (row strides are odd, so the lanes hit distinct banks), vertical passes its own
// column.
//
// What bounds it: the FP32 pipe and, on levels of few tiles, the latency of its five stages. Per launch
// (back to back launches on random planes, both with calc_b): 960 x 540 18.5 us with 32 x 64 tiles, 1920 x
// 1080 59.5 us; 480 x 270 10.3 us with 32 x 32 (14.4 with 32 x 64, 14.2 with 16 x 16); 240 x 135 and 120 x
// 67 8.3 us with 16 x 16 (10.3 with 32 x 32). Scalar planes with per tap border tests took 31, 19 and 18.6
// us (960 x 540, 480 x 270, the smaller ones).
template <int TX, int TY>
struct IterGeom {
    static constexpr int HB = 12, HD = 5;
    static constexpr int BW = TX + 2 * HB, BH = TY + 2 * HB;  // B region
    static constexpr int DW = TX + 2 * HD, DH = TY + 2 * HD;  // new_disp region
    // outputs per thread of the passes: blur7 along rows and columns, blur5 along rows and columns
    // (short runs for the small tiles, whose time is latency)
    static constexpr int R7H = TX == 16 ? 3 : 6, R7V = TX == 16 ? 2 : 4;
    static constexpr int R5H = TX == 16 ? 2 : 4, R5V = TX == 16 ? 1 : TX * TY == 1024 ? 2 : 4;
    static constexpr int S7H = (DW + R7H - 1) / R7H, S7V = (DH + R7V - 1) / R7V;  // runs of a blur7 line
    // row strides (odd) and the columns / rows a ragged last run reads past its region
    static constexpr int BS = (S7H * R7H + 14) | 1, HS = (S7H * R7H) | 1, DS = DW | 1, FS = TX | 1;
    static constexpr int HH = S7V * R7V + 14;
    // buffer 1: B (BH x BS), then the new_disp flow (DH x DS); buffer 2: blur7's horizontal pass (HH x
    // HS), then blur5's (DH x FS); then the border weight sums
    static constexpr int BUF1 = BH * BS > S7V * R7V * DS ? BH * BS : S7V * R7V * DS;
    static constexpr int BUF2 = HH * HS > DH * FS ? HH * HS : DH * FS;
    static constexpr int NDEN = S7H * R7H + S7V * R7V + TX + TY;
    static constexpr size_t SMEM = sizeof(float2) * (BUF1 + BUF2 + NDEN);
    static_assert(BW % 2 == 0 && HB % 2 == 0 && TX % R5H == 0 && TY % R5V == 0, "aligned pairs, whole blur5 runs");
};

// The tasks of the passes below, as those of k_level_init: the outputs of one run, or true when it needs
// the general rule.
// blur7 of B along a row
template <int TX, int TY, bool SLOW>
__device__ __forceinline__ bool iter_row7(const LevelIterArgs& P, const float2* in, float2* out, const float2* den, int i0) {
    constexpr int R = IterGeom<TX, TY>::R7H;
    float2 o[R];
    if (h_pass<SLOW, 8, R>(in, i0, P.w, P.g7, den, o)) return true;
    put_run<R>(out, 1, o);
    return false;
}
// blur7 of B along column x from row y0 on, and new_disp there (flow.rs:361-371); a pixel outside the image
// leaves what the flow's blur expects there
template <int TX, int TY, bool SLOW>
__device__ __forceinline__ bool iter_column7(const LevelIterArgs& P, const float2* in, float2* out, const float2* den, int x,
                                             int y0, int y_end) {
    using G = IterGeom<TX, TY>;
    constexpr int R = G::R7V;
    float2 b[R], f[R];
    if (v_pass<SLOW, 8, R>(in, G::HS, y0, P.h, P.g7, den, P.af, b)) return true;
    float4 t[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int y = y0 + r;
        f[r] = outside_value<float2>();
        t[r] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (x >= 0 && x < P.w && y >= 0 && y < y_end) {
            t[r] = __ldg(P.tensor + y * P.w + x);
            f[r] = __ldg(P.f + y * P.w + x);
        }
    }
#pragma unroll
    for (int r = 0; r < R; r++) {
        if (fabsf(t[r].w) > 40.0f) {
            f[r].x = (t[r].y * b[r].y - t[r].z * b[r].x) / t[r].w + f[r].x;
            f[r].y = (t[r].y * b[r].x - t[r].x * b[r].y) / t[r].w + f[r].y;
        }
    }
    put_run<R>(out, G::DS, f);
    return false;
}
// blur5 of the flow along a row
template <int TX, int TY, bool SLOW>
__device__ __forceinline__ bool iter_row5(const LevelIterArgs& P, const float2* in, float2* out, const float2* den, int i0) {
    constexpr int R = IterGeom<TX, TY>::R5H;
    float2 o[R];
    if (h_pass<SLOW, 6, R>(in, i0, P.w, P.g5, den, o)) return true;
    put_run<R>(out, 1, o);
    return false;
}
// blur5 of the flow along column x from row y0 on: the new flow, and with b_out calc_b of the next
// iteration there (flow.rs:334-357)
template <int TX, int TY, bool SLOW>
__device__ __forceinline__ bool iter_column5(const LevelIterArgs& P, const float2* in, const float2* den, int x, int y0) {
    using G = IterGeom<TX, TY>;
    constexpr int R = G::R5V;
    float2 f[R], g[R], b[R];
    float i1[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int i = min(y0 + r, P.h - 1) * P.w + x;
        g[r] = make_float2(0.0f, 0.0f);
        i1[r] = 0.0f;
        if (P.b_out) {
            g[r] = __ldg(P.grad + i);
            i1[r] = __ldg(P.i1 + i);
        }
    }
    if (v_pass<SLOW, 6, R>(in, G::FS, y0, P.h, P.g5, den, P.af, f)) return true;
#pragma unroll
    for (int r = 0; r < R; r++)
        if (y0 + r < P.h) P.f_out[(y0 + r) * P.w + x] = f[r];
    if (P.any) {
#pragma unroll
        for (int r = 0; r < R; r++)
            if (y0 + r < P.h) check_range(P.any, x, y0 + r, f[r], P.w, P.h);
    }
    if (P.b_out) {
        calc_b_run<R>(P.i0, P.mask_y, P.w, P.h, x, y0, f, i1, g, b);
#pragma unroll
        for (int r = 0; r < R; r++)
            if (y0 + r < P.h) P.b_out[(long)(y0 + r) * P.bp + x] = b[r];
    }
    return false;
}
template <int TX, int TY>
__device__ __noinline__ void iter_row7_slow(const LevelIterArgs& P, const float2* in, float2* out, const float2* den, int i0) {
    iter_row7<TX, TY, true>(P, in, out, den, i0);
}
template <int TX, int TY>
__device__ __noinline__ void iter_column7_slow(const LevelIterArgs& P, const float2* in, float2* out, const float2* den, int x,
                                               int y0, int y_end) {
    iter_column7<TX, TY, true>(P, in, out, den, x, y0, y_end);
}
template <int TX, int TY>
__device__ __noinline__ void iter_row5_slow(const LevelIterArgs& P, const float2* in, float2* out, const float2* den, int i0) {
    iter_row5<TX, TY, true>(P, in, out, den, i0);
}
template <int TX, int TY>
__device__ __noinline__ void iter_column5_slow(const LevelIterArgs& P, const float2* in, const float2* den, int x, int y0) {
    iter_column5<TX, TY, true>(P, in, den, x, y0);
}

template <int TX, int TY>
__device__ __forceinline__ void level_iter_body(const LevelIterArgs& P) {
    using G = IterGeom<TX, TY>;
    extern __shared__ __align__(16) float sm[];
    float2* s1 = (float2*)sm;
    float2* s2 = s1 + G::BUF1;
    float2* den7x = s2 + G::BUF2;
    float2* den7y = den7x + G::S7H * G::R7H;
    float2* den5x = den7y + G::S7V * G::R7V;
    float2* den5y = den5x + TX;
    const int w = P.w, h = P.h, bp = P.bp;
    const int X0 = blockIdx.x * TX, Y0 = blockIdx.y * TY;
    const int bx0 = X0 - G::HB, by0 = Y0 - G::HB;
    const int dx0 = X0 - G::HD, dy0 = Y0 - G::HD;
    const int nt = blockDim.x;
    // 1. B over the B region: 128-bit loads of two columns (bx0 and the pitch are even, the plane 16-byte
    //    aligned), four per thread in flight before their stores
    {
        constexpr int Q = G::BW / 2, NQ = G::BH * Q;
        for (int e0 = threadIdx.x; e0 < NQ; e0 += 4 * nt) {
            float4 v[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int e = e0 + k * nt;
                const int r = e / Q, q = e - r * Q;
                const int x = bx0 + 2 * q, y = by0 + r;
                v[k] = make_float4(-0.0f, -0.0f, -0.0f, -0.0f);
                if (e < NQ && x >= 0 && x < w && y >= 0 && y < h) {
                    v[k] = __ldg(reinterpret_cast<const float4*>(P.b_in + y * bp + x));
                    if (x + 1 >= w) v[k].z = v[k].w = -0.0f;  // the pitch's padding column
                }
            }
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int e = e0 + k * nt;
                if (e >= NQ) break;
                const int r = e / Q, q = e - r * Q;
                float2* d = s1 + r * G::BS + 2 * q;
                d[0] = make_float2(v[k].x, v[k].y);
                d[1] = make_float2(v[k].z, v[k].w);
            }
        }
        if (at_border(X0, Y0, TX, TY, G::HD + 8 + G::R7H, w, h)) {  // a ragged last run reaches past the region
            int t = fill_den<8>(den7x, 0, G::S7H * G::R7H, dx0, w, P.g7);
            t = fill_den<8>(den7y, t, G::S7V * G::R7V, dy0, h, P.g7);
            t = fill_den<6>(den5x, t, TX, X0, w, P.g5);
            fill_den<6>(den5y, t, TY, Y0, h, P.g5);
        }
    }
    __syncthreads();
    // 2. blur7 of B along the B rows, outputs at the new_disp columns
    for (int e = threadIdx.x; e < G::BH * G::S7H; e += nt) {
        const int r = e % G::BH, c0 = (e / G::BH) * G::R7H;
        const float2* in = s1 + r * G::BS + c0;
        float2* out = s2 + r * G::HS + c0;
        if (iter_row7<TX, TY, false>(P, in, out, den7x + c0, dx0 + c0)) iter_row7_slow<TX, TY>(P, in, out, den7x + c0, dx0 + c0);
    }
    __syncthreads();
    // 3. blur7 along the columns, outputs at the new_disp rows, and new_disp
    for (int e = threadIdx.x; e < G::DW * G::S7V; e += nt) {
        const int c = e % G::DW, r0 = (e / G::DW) * G::R7V;
        const float2* in = s2 + r0 * G::HS + c;
        float2* out = s1 + r0 * G::DS + c;
        const int y_end = min(h, dy0 + G::DH);
        if (iter_column7<TX, TY, false>(P, in, out, den7y + r0, dx0 + c, dy0 + r0, y_end))
            iter_column7_slow<TX, TY>(P, in, out, den7y + r0, dx0 + c, dy0 + r0, y_end);
    }
    __syncthreads();
    // 4. blur5 of the flow along the rows at the tile's columns
    for (int e = threadIdx.x; e < G::DH * (TX / G::R5H); e += nt) {
        const int r = e % G::DH, c0 = (e / G::DH) * G::R5H;
        const float2* in = s1 + r * G::DS + c0;
        float2* out = s2 + r * G::FS + c0;
        if (iter_row5<TX, TY, false>(P, in, out, den5x + c0, X0 + c0)) iter_row5_slow<TX, TY>(P, in, out, den5x + c0, X0 + c0);
    }
    __syncthreads();
    // 5. blur5 along the columns: the new flow and the next iteration's B
    for (int e = threadIdx.x; e < TX * (TY / G::R5V); e += nt) {
        const int c = e % TX, r0 = (e / TX) * G::R5V;
        if (X0 + c >= w || Y0 + r0 >= h) continue;
        const float2* in = s2 + r0 * G::FS + c;
        if (iter_column5<TX, TY, false>(P, in, den5y + r0, X0 + c, Y0 + r0)) iter_column5_slow<TX, TY>(P, in, den5y + r0, X0 + c, Y0 + r0);
    }
}

// The iteration reads B from b_in and, with b_out (same pitch bp), writes the next iteration's B; b_in
// and b_out are different buffers (other tiles still read b_in's halo).
#define TW_LEVEL_ITER(TX, TY)                                                                          \
    __global__ void __launch_bounds__(LEVEL_ITER_MAX_THREADS, 2) k_level_iter_##TX##x##TY(             \
        const __grid_constant__ LevelIterArgs P) {                                                    \
        level_iter_body<TX, TY>(P);                                                                   \
    }
TW_LEVEL_ITER(16, 16)
TW_LEVEL_ITER(32, 32)
TW_LEVEL_ITER(32, 64)
TW_LEVEL_ITER(64, 32)
TW_LEVEL_ITER(64, 64)
#undef TW_LEVEL_ITER

size_t level_iter_smem(int tile) {
    switch (tile) {
        case LEVEL_TILE_64x32: return IterGeom<64, 32>::SMEM;
        case LEVEL_TILE_64x64: return IterGeom<64, 64>::SMEM;
        case LEVEL_TILE_16x16: return IterGeom<16, 16>::SMEM;
        case LEVEL_TILE_32x64: return IterGeom<32, 64>::SMEM;
        default: return IterGeom<32, 32>::SMEM;
    }
}

// calc_b (flow.rs:334-357) of the next iteration where the flow changed outside an iteration (after
// the block matching and the user displacement of the finest level): one thread per pixel, into a plane
// of pitch bp.
__global__ void k_calc_b_pitched(const float* __restrict__ i1, const float* __restrict__ i0,
                                 const float2* __restrict__ grad, const float2* __restrict__ f, int w, int h,
                                 const float* __restrict__ mask_y, float2* __restrict__ b_out, int bp) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
    if (x >= w || y >= h) return;
    const int i = y * w + x;
    const float2 fl = __ldg(f + i), g = __ldg(grad + i);
    const float v = __ldg(i1 + i);
    float2 b;
    calc_b_run<1>(i0, mask_y, w, h, x, y, &fl, &v, &g, &b);
    b_out[(long)y * bp + x] = b;
}

// ---- the end of a level (flow.rs:1292-1303): range reset, damping, then the upsample ---------------

// The coarse field (with the reset and damping of its level applied on the fly) upsampled to the
// next finer level, for the solves whose level starts with a user displacement (the others upsample in
// k_level_init).
__global__ void k_apply_upsample(const float2* __restrict__ src, int sw, int sh, UpsampleScale up,
                                 const int* __restrict__ any, int l, int start, bool damp_now, float damp,
                                 float2* __restrict__ dst, int dw, int dh) {
    int x = blockIdx.x * blockDim.x + threadIdx.x;
    int y = blockIdx.y;
    if (x >= dw || y >= dh) return;
    dst[(long)y * dw + x] = upsample_at(src, sw, sh, up, zero_at_level(any, l, start), damp_now, damp, x, y);
}

// The finest level: reset and damping, then the final negation (flow.rs:1305) into the
// interleaved FlowField; flags a NaN.
__global__ void k_apply_negate(const float2* __restrict__ f, long n, const int* __restrict__ any, int start,
                               bool damp_now, float damp, float2* __restrict__ out, int* __restrict__ nan_flag) {
    long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float2 v = zero_at_level(any, 0, start) ? make_float2(0.0f, 0.0f) : f[i];
    if (damp_now) {
        v.x = damp * v.x;
        v.y = damp * v.y;
    }
    v.x = -1.0f * v.x;
    v.y = -1.0f * v.y;
    out[i] = v;
    if (isnan(v.x) || isnan(v.y)) atomicOr(nan_flag, 1);
}

TW_VARIANT_END
}  // namespace tw

namespace tw {
TW_VARIANT_BEGIN
// flow/extras.rs:64-72 of a plane in place
__global__ void k_binarize(float* __restrict__ p, long n) {
    long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) p[i] = binarized(p[i]);
}
TW_VARIANT_END
}  // namespace tw
