// Warping code 1 (Smart Blend) and the pull-push hole fill, strict mode.
//
// k_compose_smart: the two inverse warps with their coverage (warp.rs:504-561, hold off), the
// Smart Blend composite (smartblend.rs:168-262) and the holes mask (255 - max of the coverages,
// smartblend.rs:335-345), one pixel per thread. The fill (holefill.rs) then goes up a pyramid of the
// values and their weights and down again, a launch per level and direction, every kernel a no-op
// when the mask has no hole (the fill is the identity then). Float images run the fill's operations
// with the NaN rule: for numbers it is the plain arithmetic bit for bit, and an element that comes
// out as a NaN is taken again with the rule, which gives the bits the reference's repeat gives.
#include "kernels.cuh"
#include "level.cuh"
#include "warp.cuh"

namespace tw {

// ---- Smart Blend pixel arithmetic (smartblend.rs:155-262) ------------------------------------------

template <bool RULE> struct Ar;
template <> struct Ar<false> {
    __device__ static float add(float a, float b) { return a + b; }
    __device__ static float sub(float a, float b) { return a - b; }
    __device__ static float mul(float a, float b) { return a * b; }
    __device__ static float div(float a, float b) { return a / b; }
};
template <> struct Ar<true> {
    __device__ static float add(float a, float b) { return nr::add(a, b); }
    __device__ static float sub(float a, float b) { return nr::sub(a, b); }
    __device__ static float mul(float a, float b) { return nr::mul(a, b); }
    __device__ static float div(float a, float b) { return nr::div(a, b); }
};
template <bool RULE> __device__ __forceinline__ float lerp_r(float a, float b, float f) {
    return Ar<RULE>::add(Ar<RULE>::mul(Ar<RULE>::sub(b, a), f), a);
}

template <bool R>
__device__ __forceinline__ void over_r(const float a[4], const float b[4], float white, float o[4]) {
    if (a[0] == 0.0f) { for (int c = 0; c < 4; c++) o[c] = b[c]; return; }
    if (a[0] == white) { for (int c = 0; c < 4; c++) o[c] = a[c]; return; }
    float ia = Ar<R>::sub(1.0f, Ar<R>::div(a[0], white));
    o[0] = Ar<R>::add(Ar<R>::mul(Ar<R>::sub(white, b[0]), Ar<R>::div(a[0], white)), b[0]);
#pragma unroll
    for (int c = 1; c < 4; c++) o[c] = Ar<R>::add(Ar<R>::mul(b[c], ia), a[c]);
}

// returns true for the raw store (the "result alpha is 0" fallback)
template <bool R>
__device__ __forceinline__ bool smart_px(const float p1[4], const float p2[4], float w, float white, float v[4]) {
    float c1[4], c2[4];
    over_r<R>(p1, p2, white, c1);
    over_r<R>(p2, p1, white, c2);
    float amax = p1[0] > p2[0] ? p1[0] : p2[0];
#pragma unroll
    for (int i = 0; i < 4; i++) v[i] = lerp_r<R>(c1[i], c2[i], w);
    if (v[0] == amax) return false;
    if (v[0] == 0.0f) {
        const float* s = c1[0] > c2[0] ? c1 : c2;
        for (int i = 0; i < 4; i++) v[i] = s[i];
        return true;
    }
    float alpha = v[0];
#pragma unroll
    for (int c = 1; c < 4; c++) v[c] = Ar<R>::div(Ar<R>::mul(v[c], amax), alpha);
    v[0] = amax;
    return false;
}

template <bool R>
__device__ __forceinline__ void binary_px(const float p1[4], const float p2[4], float w, float white, float v[4]) {
    float x[4], y[4];
    if (p2[0] == white) {
        float ia = Ar<R>::sub(1.0f, Ar<R>::div(p1[0], white));
        x[0] = p2[0];
        for (int c = 1; c < 4; c++) x[c] = Ar<R>::add(Ar<R>::mul(p2[c], ia), p1[c]);
    } else if (p1[0] == white) {
        for (int c = 0; c < 4; c++) x[c] = p1[c];
    } else {
        for (int c = 0; c < 4; c++) x[c] = 0.0f;
    }
    if (p1[0] == white) {
        float ia = Ar<R>::sub(1.0f, Ar<R>::div(p2[0], white));
        y[0] = p1[0];
        for (int c = 1; c < 4; c++) y[c] = Ar<R>::add(Ar<R>::mul(p1[c], ia), p2[c]);
    } else if (p2[0] == white) {
        for (int c = 0; c < 4; c++) y[c] = p2[c];
    } else {
        for (int c = 0; c < 4; c++) y[c] = 0.0f;
    }
#pragma unroll
    for (int i = 0; i < 4; i++) v[i] = lerp_r<R>(x[i], y[i], w);
}

template <typename P> struct SPx;
template <> struct SPx<uint8_t> {
    static constexpr float WHITE = 255.0f;
    __device__ static uint8_t plain(float x) {
        float y = x + 0.5f;
        if (0.0f > y) return 0;
        if (y > 255.0f) return 255;
        return (uint8_t)__float2int_rz(y);  // (a NaN: 0)
    }
    __device__ static uint8_t raw(float x) { return (uint8_t)cvtt_low(x); }
};
template <> struct SPx<uint16_t> {
    static constexpr float WHITE = 65535.0f;
    __device__ static uint16_t plain(float x) {
        float y = x + 0.5f;
        if (0.0f > y) return 0;
        if (y > 65535.0f) return 65535;
        return (uint16_t)__float2int_rz(y);  // (a NaN: 0)
    }
    __device__ static uint16_t raw(float x) { return (uint16_t)cvtt_low(x); }
};
template <> struct SPx<float> {
    static constexpr float WHITE = 1.0f;
    __device__ static float plain(float x) { return nr::add(x, 0.0f); }
    __device__ static float raw(float x) { return x; }
};

// One Smart Blend pixel (smartblend.rs:268-298): p1 over p2 and p2 over p1 blended at w, or the
// binary alpha variant; the raw store where the blended alpha came out 0, else the plain store.
template <typename P>
__device__ __forceinline__ void smart_blend_px(const float p1[4], const float p2[4], float w, bool binary, float o[4]) {
    float v[4];
    constexpr bool R = sizeof(P) == 4;  // NaN only reaches float images
    bool raw = false;
    if (binary) binary_px<R>(p1, p2, w, SPx<P>::WHITE, v);
    else raw = smart_px<R>(p1, p2, w, SPx<P>::WHITE, v);
    if (raw) {
        for (int k = 0; k < 4; k++) o[k] = (float)SPx<P>::raw(v[k]);
    } else {
        for (int k = 0; k < 4; k++) o[k] = (float)SPx<P>::plain(v[k]);
    }
}

// One pixel of warping code 1. mode 0: Nearest (one warp: pa), 1: Blend (pa = A, pb = B, w = frac).
template <typename P>
__device__ __forceinline__ void compose_smart_px(const WarpParams& pa, const WarpParams& pb, int mode, float w,
                                                 bool binary, void* out, uint8_t* holes, int W, int H, int* any_hole,
                                                 int* bad) {
    int x = blockIdx.x * blockDim.x + threadIdx.x;
    int y = blockIdx.y;
    bool hole = false;
    if (x < W && y < H) {
        float ta[4], tb[4], o[4];
        bool b = false;
        uint8_t c1 = warp_pixel<P>(pa, x, y, W, H, ta, b);
        uint8_t cov = c1;
        if (mode == 0) {
            for (int k = 0; k < 4; k++) o[k] = ta[k];
        } else {
            uint8_t c2 = warp_pixel<P>(pb, x, y, W, H, tb, b);
            cov = c1 > c2 ? c1 : c2;
            smart_blend_px<P>(ta, tb, w, binary, o);
        }
        long i = (long)y * W + x;
        px_store((P*)out + i * 4, o);
        uint8_t m = (uint8_t)(0xff - cov);
        holes[i] = m;
        hole = m != 0;  // a u8 mask value is a hole iff it is not 0 (holefill.rs:124-133)
        if (b) atomicOr(bad, 1);
    }
    if (__syncthreads_or(hole) && threadIdx.x == 0) atomicOr(any_hole, 1);
}

__global__ void k_compose_smart(WarpParams pa, WarpParams pb, int fmt, int mode, float w, bool binary,
                                void* __restrict__ out, uint8_t* __restrict__ holes, int W, int H,
                                int* __restrict__ any_hole, int* __restrict__ bad) {
    if (fmt == 0) compose_smart_px<uint8_t>(pa, pb, mode, w, binary, out, holes, W, H, any_hole, bad);
    else if (fmt == 1) compose_smart_px<uint16_t>(pa, pb, mode, w, binary, out, holes, W, H, any_hole, bad);
    else compose_smart_px<float>(pa, pb, mode, w, binary, out, holes, W, H, any_hole, bad);
}

// smartblend.rs:305-315 on whole images (the stage entry point)
template <typename P>
__device__ __forceinline__ void smart_blend_at(const void* p1, const void* p2, float w, bool binary, void* out, long i) {
    float a[4], b[4], o[4];
    px_floats<P>((const P*)p1 + 4 * i, a);
    px_floats<P>((const P*)p2 + 4 * i, b);
    smart_blend_px<P>(a, b, w, binary, o);
    px_store((P*)out + 4 * i, o);
}
__global__ void k_smart_blend(const void* __restrict__ p1, const void* __restrict__ p2, int fmt, float w, bool binary,
                              void* __restrict__ out, long n) {
    long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (fmt == 0) smart_blend_at<uint8_t>(p1, p2, w, binary, out, i);
    else if (fmt == 1) smart_blend_at<uint16_t>(p1, p2, w, binary, out, i);
    else smart_blend_at<float>(p1, p2, w, binary, out, i);
}

// holefill.rs:124-133: a pixel is a hole when !(eps > m) in double (a NaN float value is a hole);
// eps is the u8 threshold for kind 1, the u16 / f32 one for kinds 2 and 3. Writes the u8 holes
// mask (1 at a hole) and sets *any_hole.
__global__ void k_mask_holes(const void* __restrict__ mask, int kind, uint8_t* __restrict__ holes, long n,
                             int* __restrict__ any_hole) {
    long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    bool hole = false;
    if (i < n) {
        const double u8_eps = __longlong_as_double(0x20202020202020fcll);
        const double wide_eps = __longlong_as_double(0x3f0040bfe3b03e21ll);
        double m;
        if (kind == 1) m = (double)((const uint8_t*)mask)[i];
        else if (kind == 2) m = (double)((const uint16_t*)mask)[i];
        else m = (double)((const float*)mask)[i];
        hole = !((kind == 1 ? u8_eps : wide_eps) > m);
        holes[i] = hole ? 1 : 0;
    }
    if (__syncthreads_or(hole) && threadIdx.x == 0) atomicOr(any_hole, 1);
}

// warp.rs:76-95 then the u8 hole rule (holefill.rs:126-133): the holes of a coverage image, or of the
// per byte maximum of two (Coverage::combine_max), inverted: a hole where 255 - coverage is not 0
__global__ void k_cov_holes(const uint8_t* __restrict__ c1, const uint8_t* __restrict__ c2, uint8_t* __restrict__ holes,
                            long n, int* __restrict__ any_hole) {
    long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    bool hole = false;
    if (i < n) {
        uint8_t c = c1[i];
        if (c2 && c2[i] > c) c = c2[i];
        hole = (uint8_t)(0xffu - c) != 0;
        holes[i] = hole ? 1 : 0;
    }
    if (__syncthreads_or(hole) && threadIdx.x == 0) atomicOr(any_hole, 1);
}

// ---- the hole fill (holefill.rs): its levels in tiles ---------------------------------------------------

// One element of a pass along a line held in shared memory: element t (global index in [0, len)) of
// the line at line[(t - origin) * stride]; the interior chain or the 1 channel border rule (conv.rs:101-137,
// :141-190, :268-301).
template <bool R, int N, bool LEFT_FIRST>
__device__ __forceinline__ float stack_elem(const float* line, int origin, int stride, int len, int i, const Taps& t) {
    if (len >= 2 * N && i >= N && i < len - N) {
        const float* c = line + (i - origin) * stride;
        float r = Ar<R>::mul(c[0], t.k[0]);
#pragma unroll
        for (int j = N - 1; j >= 1; j--) r = Ar<R>::add(r, Ar<R>::mul(Ar<R>::add(c[j * stride], c[-j * stride]), t.k[j]));
        return r;
    }
    float num = Ar<R>::mul(t.k[0], line[(i - origin) * stride]);
    float den = t.k[0];
#pragma unroll
    for (int j = N - 1; j >= 1; j--) {
        float kj = t.k[j];
#pragma unroll
        for (int side = 0; side < 2; side++) {
            bool right = (side == 0) != LEFT_FIRST;
            int tt = right ? i + j : i - j;
            bool inside = tt >= 0 && tt < len;
            float xv = inside ? line[(tt - origin) * stride] : 0.0f;
            float wv = inside ? kj : 0.0f;
            den = den + wv;
            num = Ar<R>::add(num, Ar<R>::mul(xv, wv));
        }
    }
    return Ar<R>::div(num, den);
}

// The NaN rule's results, out of the main path
template <int N, bool LEFT_FIRST>
__device__ __noinline__ float2 fill_rule_elem(const float2* line, int origin, int stride, int len, int i, const Taps& t) {
    const float* f = reinterpret_cast<const float*>(line);
    return make_float2(stack_elem<true, N, LEFT_FIRST>(f, origin, 2 * stride, len, i, t),
                       stack_elem<true, N, LEFT_FIRST>(f + 1, origin, 2 * stride, len, i, t));
}
__device__ __noinline__ float2 fill_rule_mix(float2 a, float2 b, float2 c, float2 d, float fx, float fy) {
    auto mix = [&](float a, float b, float c, float d) {
        return lerp_r<true>(lerp_r<true>(a, b, fx), lerp_r<true>(c, d, fx), fy);
    };
    return make_float2(mix(a.x, b.x, c.x, d.x), mix(a.y, b.y, c.y, d.y));
}
__device__ __noinline__ float2 fill_rule_quot(float2 v, float d) { return make_float2(nr::div(v.x, d), nr::div(v.y, d)); }
__device__ __forceinline__ bool any_nan(float2 v) { return isnan(v.x) || isnan(v.y); }

// v / d: the reciprocal correctly rounded and Markstein's corrections in a pair (level.cuh) for operands within
// 2^60 of 1; others divide. Most weights are 1.
__device__ __forceinline__ float2 fill_quot(float2 v, float d, bool rule) {
    float2 q = v;
    if (d != 1.0f) {
        const float lo = 8.67e-19f, hi = 1.15e18f;  // 2^-60, 2^60
        auto in = [&](float x) { return fabsf(x) > lo && fabsf(x) < hi; };
        if (in(d) && (v.x == 0.0f || in(v.x)) && (v.y == 0.0f || in(v.y))) {
            const float y = __frcp_rn(d);
            const float2 n = make_float2(-d, -d), yy = make_float2(y, y);
            const float2 q0 = __ffma2_rn(v, yy, make_float2(-0.0f, -0.0f));
            q = __ffma2_rn(__ffma2_rn(q0, n, v), yy, q0);
            q = __ffma2_rn(__ffma2_rn(q, n, v), yy, q);
            q = make_float2(v.x == 0.0f ? q0.x : q.x, v.y == 0.0f ? q0.y : q.y);
        } else {
            q = make_float2(v.x / d, v.y / d);
        }
    }
    return rule && any_nan(q) ? fill_rule_quot(v, d) : q;
}

// Four taps a b / c d of a pair mixed (flow/sample.rs:91-112)
__device__ __forceinline__ float2 fill_mix(float2 a, float2 b, float2 c, float2 d, float fx, float fy, float z, bool rule) {
    const float2 fx2 = make_float2(fx, fx), z2 = make_float2(z, z);
    const float2 top = px_lerp(a, a, b, fx2, z2), bot = px_lerp(c, c, d, fx2, z2);
    const float2 r = px_lerp(top, top, bot, make_float2(fy, fy), z2);
    return rule && any_nan(r) ? fill_rule_mix(a, b, c, d, fx, fy) : r;
}

// The tile of a level: 32 x 32 outputs of the blur with N taps (the pull: blur5, one output more each way for the
// resample's second taps; the push: the Gaussian), two channels of a pixel as a pair. 4 outputs per thread,
// rows a lane apart in the row pass and columns a lane apart in the column pass.
template <int N>
struct FillGeom {
    static constexpr int T = 32, R = 4, HALO = N - 1, OUT = N == 3 ? T + 1 : T, SEG = (OUT + R - 1) / R;
    static constexpr int ROWS = OUT + 2 * HALO, RUNS = R * SEG + 2 * HALO, RS = RUNS | 1, HS = R * SEG | 1, VS = OUT | 1;
    static constexpr int EX = N == 3 ? 8 : 16;  // the region's columns right of the first 32 (RUNS - T of them)
    static constexpr int IN = ROWS * RS, MID = RUNS * HS;
    static_assert(RUNS - T <= EX && SEG * R * VS <= IN, "the planes hold every run");
};

// A tile's shared memory
template <int N>
struct FillShared {
    using G = FillGeom<N>;
    float2 in[G::IN], mid[G::MID], dx[G::R * G::SEG], dy[G::R * G::SEG], cx[G::RUNS], cy[G::RUNS];
};
// The threads of a tile: a whole block, or one of a block's groups of FILL_THREADS, with a barrier of its own
struct FillBlock {
    static __device__ __forceinline__ int tid() { return threadIdx.x; }
    static __device__ __forceinline__ void sync() { __syncthreads(); }
};
struct FillGroup {
    static __device__ __forceinline__ int tid() { return threadIdx.x % FILL_THREADS; }
    static __device__ __forceinline__ void sync() {
        asm volatile("bar.sync %0, %1;" ::"r"(1 + (int)threadIdx.x / FILL_THREADS), "n"(FILL_THREADS) : "memory");
    }
};

// The region of a tile at (X0, Y0), at(X, Y) inside the image and 0 outside
template <int N, class At>
__device__ __forceinline__ void fill_region(float2* s_in, int tid, int X0, int Y0, int w, int h, At at) {
    using G = FillGeom<N>;
    const int c = tid % G::T, r0 = tid / G::T;
    constexpr int PER = FILL_THREADS / G::T, A = (G::ROWS + PER - 1) / PER, B = (G::ROWS * G::EX + FILL_THREADS - 1) / FILL_THREADS;
    float2 v[A + B];
    // column and row of the region (no others are looked at: `at` may hold tables of the region's size)
    auto value = [&](int x, int y) {
        const int X = X0 - G::HALO + x, Y = Y0 - G::HALO + y;
        return x < G::RUNS && y < G::ROWS && X >= 0 && X < w && Y >= 0 && Y < h ? at(X, Y) : make_float2(0.0f, 0.0f);
    };
#pragma unroll
    for (int j = 0; j < A; j++) v[j] = value(c, r0 + j * PER);
#pragma unroll
    for (int j = 0; j < B; j++) {
        const int e = tid + j * FILL_THREADS;
        v[A + j] = value(G::T + e % G::EX, e / G::EX);
    }
#pragma unroll
    for (int j = 0; j < A; j++)
        if (r0 + j * PER < G::ROWS) s_in[(r0 + j * PER) * G::RS + c] = v[j];
#pragma unroll
    for (int j = 0; j < B; j++) {
        const int e = tid + j * FILL_THREADS;
        if (e / G::EX < G::ROWS && e % G::EX < G::RUNS - G::T) s_in[e / G::EX * G::RS + G::T + e % G::EX] = v[A + j];
    }
}

// A run of R outputs of a pass: line is the sample at index i0 - (N - 1), `first` the first one held
template <int N, bool LEFT_FIRST>
__device__ __forceinline__ void fill_run(const float2* line, int stride, int i0, int len, int held, const Taps& t,
                                         const float2* den, bool rule, float2* o) {
    constexpr int R = FillGeom<N>::R;
    float2 v[R + 2 * N - 2];
#pragma unroll
    for (int j = 0; j < R + 2 * N - 2; j++) v[j] = line[j * stride];
    single_run<N, R, LEFT_FIRST>(v, i0, len, t, den, o);
    if (rule) {
#pragma unroll
        for (int r = 0; r < R; r++)
            if (any_nan(o[r]) && i0 + r < min(len, held)) o[r] = fill_rule_elem<N, LEFT_FIRST>(line, i0 - (N - 1), stride, len, i0 + r, t);
    }
}

// Both passes of the region in S.in; out(seg, x, values): the 4 outputs of column x from row 4 * seg on
template <int N, class Threads, class Out>
__device__ __forceinline__ void fill_blur(FillShared<N>& S, int X0, int Y0, int w, int h, const Taps& t, bool above_first, bool rule,
                                          Out out) {
    using G = FillGeom<N>;
    for (int e = Threads::tid(); e < G::ROWS * G::SEG; e += FILL_THREADS) {
        const int seg = e / G::ROWS, y = e - seg * G::ROWS;
        float2 o[G::R];
        fill_run<N, false>(S.in + y * G::RS + seg * G::R, 1, X0 + seg * G::R, w, X0 + G::OUT, t, S.dx + seg * G::R, rule, o);
#pragma unroll
        for (int r = 0; r < G::R; r++) S.mid[y * G::HS + seg * G::R + r] = o[r];
    }
    Threads::sync();
    for (int e = Threads::tid(); e < G::OUT * G::SEG; e += FILL_THREADS) {
        const int seg = e / G::OUT, x = e - seg * G::OUT;
        float2 o[G::R];
        const float2* line = S.mid + seg * G::R * G::HS + x;
        if (above_first) fill_run<N, true>(line, G::HS, Y0 + seg * G::R, h, Y0 + G::OUT, t, S.dy + seg * G::R, rule, o);
        else fill_run<N, false>(line, G::HS, Y0 + seg * G::R, h, Y0 + G::OUT, t, S.dy + seg * G::R, rule, o);
        out(seg, x, o);
    }
}

// Channels 2 * pair and 2 * pair + 1 of an image's pixel i (a flow's vector)
template <int FMT>
__device__ __forceinline__ float2 fill_sample(const void* img, long i, int pair) {
    if (FMT == FILL_FLOW) return ((const float2*)img)[i];
    if (FMT == 2) return ((const float2*)img)[2 * i + pair];
    if (FMT == 0) {
        const Px4 q = px_load((const uint8_t*)img + 4 * i);
        return px_value<uint8_t>(pair ? q.b : q.a);
    }
    const Px4 q = px_load((const uint16_t*)img + 4 * i);
    return px_value<uint16_t>(pair ? q.b : q.a);
}

template <int FMT>
__device__ __forceinline__ void fill_pull_image(const FillPull& P, float2* s_in, int X0, int Y0, int pair) {
    const bool weights = 2 * pair == P.nc;
    fill_region<3>(s_in, threadIdx.x, X0, Y0, P.w, P.h, [&](int X, int Y) {
        const long i = (long)Y * P.w + X;
        if (P.holes[i]) return make_float2(0.0f, 0.0f);
        return weights ? make_float2(1.0f, 0.0f) : fill_sample<FMT>(P.img, i, pair);
    });
}

// A level's stack: the pair's planes, or the weights and nothing
__device__ __forceinline__ void fill_pull_planes(const float* vals, float2* s_in, int tid, int X0, int Y0, int w, int h, int nc, int pair) {
    const long n = (long)w * h;
    const float *a = vals + 2 * pair * n, *b = 2 * pair == nc ? nullptr : a + n;
    fill_region<3>(s_in, tid, X0, Y0, w, h, [&](int X, int Y) {
        const long i = (long)Y * w + X;
        return make_float2(a[i], b ? b[i] : 0.0f);
    });
}

// The rest of a pull: the blur of the region and the outputs whose first tap lies in the tile
template <class Threads>
__device__ __forceinline__ void fill_pull_tile(FillShared<3>& S, int X0, int Y0, int w, int h, int dw, int dh, float sx, float sy,
                                               float* dst, int nc, int pair, const Taps& t, bool above_first, bool rule) {
    using G = FillGeom<3>;
    const int tid = Threads::tid();
    // the outputs whose first tap can lie in the tile, from its ends over the step (at least 1)
    auto range = [](int at, int len, float step, int n, int& lo, int& count) {
        lo = (int)((float)at / step);
        count = min((at + G::T < len - 1 ? min((int)((float)(at + G::T) / step), n - 1) : n - 1) - lo + 1, G::T + 2);
    };
    int xa, nx, ya, ny;
    range(X0, w, sx, dw, xa, nx);
    range(Y0, h, sy, dh, ya, ny);
    auto cell_at = [](int i, float step, int len, int at) {
        int k;
        float f;
        cell((float)i * step, len, k, f);
        k -= at;
        return make_float2(__int_as_float(k >= 0 && k < G::T ? k : -1), f);
    };
    if (tid < G::R * G::SEG) {
        S.dx[tid] = border_den<3>(X0 + tid, w, t.k);
        S.dy[tid] = border_den<3>(Y0 + tid, h, t.k);
    }
    const int k = FILL_THREADS - 1 - tid;
    if (k < nx) S.cx[k] = cell_at(xa + k, sx, w, X0);
    if (k < ny) S.cy[k] = cell_at(ya + k, sy, h, Y0);
    Threads::sync();
    float2* s_v = S.in;  // (the column pass reads S.mid alone)
    fill_blur<3, Threads>(S, X0, Y0, w, h, t, above_first, rule, [&](int seg, int x, const float2* o) {
#pragma unroll
        for (int r = 0; r < G::R; r++) s_v[(seg * G::R + r) * G::VS + x] = o[r];
    });
    Threads::sync();
    constexpr int COLS = G::T / 2 + 2;  // the outputs across a tile at a step of 2
    const long dn = (long)dw * dh;
    float *da = dst + 2 * pair * dn, *db = 2 * pair == nc ? nullptr : da + dn;
    for (int x0 = 0; x0 < nx; x0 += COLS) {
        for (int e = tid; e < COLS * ny; e += FILL_THREADS) {
            const int y = e / COLS, x = x0 + e - y * COLS;
            if (x >= nx) continue;
            const float2 cx = S.cx[x], cy = S.cy[y];
            const int ix = __float_as_int(cx.x), iy = __float_as_int(cy.x);
            if (ix < 0 || iy < 0) continue;
            const float2* q = s_v + iy * G::VS + ix;
            const float2 r = fill_mix(q[0], q[1], q[G::VS], q[G::VS + 1], cx.y, cy.y, t.z, rule);
            const long i = (long)(ya + y) * dw + xa + x;
            da[i] = r.x;
            if (db) db[i] = r.y;
        }
    }
}

// One level up (holefill.rs:300-350): blur5 of level k - 1 and the resample to level k, a pair of channels
// or the weights (blockIdx.z); level 0 is the image itself with its holes at zero weight. Each output belongs
// to the tile of its first tap.
//
// Bound by issue. With planes of single channels, a launch for the load, the blur and the resample each and a
// test per tap, a 1080p level 0 took 14 + 50 + 12 us. Flows filled at 1080p: 38 us for a level's
// blur and resample on average, now 19.
__global__ void __launch_bounds__(FILL_THREADS) k_fill_pull(const __grid_constant__ FillPull P) {
    if (!*P.any) return;
    __shared__ FillShared<3> S;
    const int X0 = blockIdx.x * FillGeom<3>::T, Y0 = blockIdx.y * FillGeom<3>::T, pair = blockIdx.z;
    if (P.vals) fill_pull_planes(P.vals, S.in, threadIdx.x, X0, Y0, P.w, P.h, P.nc, pair);
    else if (P.fmt == 0) fill_pull_image<0>(P, S.in, X0, Y0, pair);
    else if (P.fmt == 1) fill_pull_image<1>(P, S.in, X0, Y0, pair);
    else if (P.fmt == 2) fill_pull_image<2>(P, S.in, X0, Y0, pair);
    else fill_pull_image<FILL_FLOW>(P, S.in, X0, Y0, pair);
    fill_pull_tile<FillBlock>(S, X0, Y0, P.w, P.h, P.dw, P.dh, P.sx, P.sy, P.dst, P.nc, pair, P.t, P.above_first, P.rule);
}

// A sample as stored (holefill.rs:379-404)
template <int FMT>
__device__ __forceinline__ void fill_put(void* img, long i, int pair, float2 v) {
    if (FMT == 0) ((uchar2*)img)[2 * i + pair] = make_uchar2(SPx<uint8_t>::plain(v.x), SPx<uint8_t>::plain(v.y));
    else if (FMT == 1) ((ushort2*)img)[2 * i + pair] = make_ushort2(SPx<uint16_t>::plain(v.x), SPx<uint16_t>::plain(v.y));
    else if (FMT == 2) ((float2*)img)[2 * i + pair] = v;
    else ((float2*)img)[i] = v;
}

// The coarser solution (planes of pairs of channels, null: zero) at the region's (X, Y), by the tables of S
__device__ __forceinline__ float2 fill_coarser(const float2* coarse, int cw, int ch, const FillShared<6>& S, int x, int y, int pair,
                                               float z, bool rule) {
    if (!coarse) return make_float2(0.0f, 0.0f);
    const float2 cx = S.cx[x], cy = S.cy[y];
    const float2* q = coarse + (long)pair * cw * ch + (long)__float_as_int(cy.x) * cw + __float_as_int(cx.x);
    return fill_mix(q[0], q[1], q[cw], q[cw + 1], cx.y, cy.y, z, rule);
}

// The tables of a push: the border weights, and the cells of the region in the coarser level
template <class Threads>
__device__ __forceinline__ void fill_push_tables(FillShared<6>& S, int X0, int Y0, int w, int h, int cw, int ch, float sx, float sy,
                                                 const Taps& t) {
    using G = FillGeom<6>;
    const int tid = Threads::tid(), k = FILL_THREADS - 1 - tid;
    if (tid < G::R * G::SEG) {
        S.dx[tid] = border_den<6>(X0 + tid, w, t.k);
        S.dy[tid] = border_den<6>(Y0 + tid, h, t.k);
    }
    if (k < G::RUNS) {
        auto cell_at = [](int i, float step, int len) {
            int c;
            float f;
            cell((float)i * step, len, c, f);
            return make_float2(__int_as_float(c), f);
        };
        S.cx[k] = cell_at(X0 - G::HALO + k, sx, cw);
        S.cy[k] = cell_at(Y0 - G::HALO + k, sy, ch);
    }
    Threads::sync();
}

// A level of planes: the values over their weights or the coarser solution, blurred into out
template <class Threads>
__device__ __forceinline__ void fill_push_planes(FillShared<6>& S, int X0, int Y0, int w, int h, const float* vals, const float2* coarse,
                                                 int cw, int ch, float2* out, int nc, int pair, const Taps& t, bool above_first,
                                                 bool rule) {
    using G = FillGeom<6>;
    const long n = (long)w * h;
    const float *va = vals + 2 * pair * n, *wt = vals + nc * n;
    fill_region<6>(S.in, Threads::tid(), X0, Y0, w, h, [&](int X, int Y) {
        const long i = (long)Y * w + X;
        const float d = wt[i];
        if (d == 0.0f) return fill_coarser(coarse, cw, ch, S, X - X0 + G::HALO, Y - Y0 + G::HALO, pair, t.z, rule);
        return fill_quot(make_float2(va[i], va[n + i]), d, rule);
    });
    Threads::sync();
    fill_blur<6, Threads>(S, X0, Y0, w, h, t, above_first, rule, [&](int seg, int x, const float2* o) {
#pragma unroll
        for (int r = 0; r < G::R; r++) {
            const int X = X0 + x, Y = Y0 + seg * G::R + r;
            if (X < w && Y < h) out[pair * n + (long)Y * w + X] = o[r];
        }
    });
}

// Level 0, the image: the holes take the blurred solution
template <int FMT>
__device__ __forceinline__ void fill_push_image(FillShared<6>& S, const FillPush& P, int X0, int Y0, int pair) {
    using G = FillGeom<6>;
    const int w = P.w, h = P.h;
    fill_region<6>(S.in, threadIdx.x, X0, Y0, w, h, [&](int X, int Y) {
        const long i = (long)Y * w + X;
        if (P.holes[i]) return fill_coarser(P.coarse, P.cw, P.ch, S, X - X0 + G::HALO, Y - Y0 + G::HALO, pair, P.t.z, P.rule);
        return fill_quot(fill_sample<FMT>(P.img, i, pair), 1.0f, P.rule);
    });
    __syncthreads();
    fill_blur<6, FillBlock>(S, X0, Y0, w, h, P.t, P.above_first, P.rule, [&](int seg, int x, const float2* o) {
#pragma unroll
        for (int r = 0; r < G::R; r++) {
            const int X = X0 + x, Y = Y0 + seg * G::R + r;
            if (X >= w || Y >= h) continue;
            const long i = (long)Y * w + X;
            if (P.holes[i]) fill_put<FMT>(P.img, i, pair, o[r]);
        }
    });
}

// One level down (holefill.rs:352-404): the values over their weights, the coarser solution where there is no
// weight, and the Gaussian of it; a pair of channels (blockIdx.z). At level 0 (an image) the holes take it and
// the other pixels stay as they are, but for a NaN that the rule's division by 1 quiets; a tile without a
// hole has nothing to do. A tile's halo may read a sample while its own tile quiets it: the NaN that was there
// and the quieted one give the same bits after the division by 1; a hole's own sample is not looked at.
//
// Bound by issue. The launches of a 1080p level 0 (combine, blur, combine, store) took 10 + 48 + 10 + 15 us.
__global__ void __launch_bounds__(FILL_THREADS) k_fill_push(const __grid_constant__ FillPush P) {
    using G = FillGeom<6>;
    if (!*P.any) return;
    __shared__ FillShared<6> S;
    const int w = P.w, h = P.h, X0 = blockIdx.x * G::T, Y0 = blockIdx.y * G::T, pair = blockIdx.z, tid = threadIdx.x;
    if (P.img) {
        bool hole = false;
        const int X = X0 + tid % G::T;
        for (int Y = Y0 + tid / G::T; Y < min(Y0 + G::T, h); Y += FILL_THREADS / G::T) {
            if (X >= w) continue;
            const long i = (long)Y * w + X;
            if (P.holes[i]) {
                hole = true;
            } else if (P.rule) {
                const float2 v = P.fmt == 2 ? fill_sample<2>(P.img, i, pair) : fill_sample<FILL_FLOW>(P.img, i, pair);
                if (any_nan(v)) {
                    if (P.fmt == 2) fill_put<2>(P.img, i, pair, fill_rule_quot(v, 1.0f));
                    else fill_put<FILL_FLOW>(P.img, i, pair, fill_rule_quot(v, 1.0f));
                }
            }
        }
        if (!__syncthreads_or(hole)) return;
    }
    fill_push_tables<FillBlock>(S, X0, Y0, w, h, P.cw, P.ch, P.sx, P.sy, P.t);
    if (!P.img)
        fill_push_planes<FillBlock>(S, X0, Y0, w, h, P.vals, P.coarse, P.cw, P.ch, P.out, P.nc, pair, P.t, P.above_first, P.rule);
    else if (P.fmt == 0) fill_push_image<0>(S, P, X0, Y0, pair);
    else if (P.fmt == 1) fill_push_image<1>(S, P, X0, Y0, pair);
    else if (P.fmt == 2) fill_push_image<2>(S, P, X0, Y0, pair);
    else fill_push_image<FILL_FLOW>(S, P, X0, Y0, pair);
}

// The levels k0 .. top, of one tile each, up from level k0 and down to it in one block: a group of threads per
// pair of channels and for the weights, the level's planes in global memory (the block's own, and in its L1). A
// level and direction takes some 4 us. (One block over planes in shared memory, a thread per element of a
// plane with a division for its place, took 100 us for these levels and 60 x 33, this and two launches 50.)
union FillTailShared {
    FillShared<3> up;
    FillShared<6> down;
};
__global__ void __launch_bounds__(FILL_TAIL_GROUPS * FILL_THREADS) k_fill_tail(const __grid_constant__ FillTail J) {
    if (!*J.any) return;
    extern __shared__ __align__(16) unsigned char tail_sm[];
    const int pair = threadIdx.x / FILL_THREADS;
    FillTailShared& S = reinterpret_cast<FillTailShared*>(tail_sm)[pair];
    auto step = [](int from, int to) { return ((float)from - 1.0f) / (float)(to - 1); };
    for (int k = J.k0 + 1; k <= J.top; k++) {
        const int w = J.dims[k - 1][0], h = J.dims[k - 1][1], dw = J.dims[k][0], dh = J.dims[k][1];
        if (2 * pair <= J.nc) {
            fill_pull_planes(J.base + J.offs[k - 1], S.up.in, FillGroup::tid(), 0, 0, w, h, J.nc, pair);
            fill_pull_tile<FillGroup>(S.up, 0, 0, w, h, dw, dh, step(w, dw), step(h, dh), J.base + J.offs[k], J.nc, pair, J.b5,
                                      J.above_first, J.rule);
        }
        __syncthreads();
    }
    for (int k = J.top; k >= J.k0; k--) {
        const int w = J.dims[k][0], h = J.dims[k][1], cw = k < J.top ? J.dims[k + 1][0] : 2, ch = k < J.top ? J.dims[k + 1][1] : 2;
        if (2 * pair < J.nc) {
            fill_push_tables<FillGroup>(S.down, 0, 0, w, h, cw, ch, step(cw, w), step(ch, h), J.g5);
            fill_push_planes<FillGroup>(S.down, 0, 0, w, h, J.base + J.offs[k], k < J.top ? J.blurred[(k + 1) & 1] : nullptr, cw, ch,
                                        J.blurred[k & 1], J.nc, pair, J.g5, J.above_first, J.rule);
        }
        __syncthreads();
    }
}
size_t fill_tail_smem() { return FILL_TAIL_GROUPS * sizeof(FillTailShared); }

// a hole in an image with a side of 1 pixel: the fill refuses it (holefill.rs:273-277)
__global__ void k_hole_side1(const int* __restrict__ any_hole, int* __restrict__ flag) {
    if (*any_hole) *flag = 1;
}

}  // namespace tw
