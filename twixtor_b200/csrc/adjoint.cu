// The adjoint of warp + blend (the differentiable twin of compose_vectors' Blend with warping code
// 0): out = ta + (tb - ta) * w with ta = warp(A, F_BA, 1 - wa), tb = warp(B, F_AB, wa), w = 1 - wa,
// where warp(S, F, s)(p) samples S bilinearly at p + F(p r) (s / r) (the flow sampled bilinearly at
// p r, r = (flow size - 1) / (image size - 1) per axis, the step s / r formed once per side as
// warp.rs:636-651 forms sx, sy), the position clamped
// to the image rectangle. One fused kernel per pixel recomputes the forward sample (nothing of the
// forward pass is stored), takes the output gradient (given, or the sign of out - target for the
// photometric L1 loss) and scatters:
//   dA, dB     the bilinear weights times (1 - w) g and w g at the sample's four corners;
//   dF_BA, dF_AB  the image gradient at the sample point times s / r, through the flow's bilinear weights.
// Neighbouring pixels mostly share corners: under a smooth flow a pixel's right corners are the next
// lane's left ones, its lower corners the next row's upper ones, and a row's flow texels those of the
// rows beside it. So a thread goes down 8 rows of a column, takes its left neighbour's share by
// shuffles, carries its lower share to the next row in registers, and adds what is left, some 1.2
// corners and 0.3 texels a pixel and side, to global memory by vector atomics.
// Frames are float RGBA (4 channels, any premultiplication), batch items back to back.
#include "kernels.cuh"

namespace tw {

namespace {

// A pixel as two pairs of channels. The forward's products stay products of their own (z, -0.0, from the kernel's
// arguments: the bits of the library's warp and blend); the gradients' may go into a sum.
struct Px {
    float2 a, b;
};
__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }
__device__ __forceinline__ Px ld4(const float* p, long i) {
    const float4 v = reinterpret_cast<const float4*>(p)[i];
    return {make_float2(v.x, v.y), make_float2(v.z, v.w)};
}
__device__ __forceinline__ float4 whole(Px p) { return make_float4(p.a.x, p.a.y, p.b.x, p.b.y); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, both(-1.0f), a); }
__device__ __forceinline__ Px sub4(Px a, Px b) { return {sub2(a.a, b.a), sub2(a.b, b.b)}; }
__device__ __forceinline__ Px add4(Px a, Px b) { return {__fadd2_rn(a.a, b.a), __fadd2_rn(a.b, b.b)}; }
__device__ __forceinline__ Px scale4(Px a, float s) { return {__fmul2_rn(a.a, both(s)), __fmul2_rn(a.b, both(s))}; }
// a + d * t, the product rounded (the forward) or not
__device__ __forceinline__ float2 step2(float2 a, float2 d, float t, float z) { return __fadd2_rn(a, __ffma2_rn(d, both(t), both(z))); }
__device__ __forceinline__ Px step4(Px a, Px d, float t, float z) { return {step2(a.a, d.a, t, z), step2(a.b, d.b, t, z)}; }
__device__ __forceinline__ Px fused4(Px a, Px d, float t) { return {__ffma2_rn(d.a, both(t), a.a), __ffma2_rn(d.b, both(t), a.b)}; }
__device__ __forceinline__ Px mix4(Px a, Px b, float t, float z) { return step4(a, sub4(b, a), t, z); }
__device__ __forceinline__ float dot4(Px a, Px b) {
    const float2 s = __ffma2_rn(a.b, b.b, __fmul2_rn(a.a, b.a));
    return s.x + s.y;
}

// the bilinear cell of x in a line of n, the last one folded as warp.rs does
__device__ __forceinline__ void cell_of(float x, int n, int& i, float& f) {
    i = (int)floorf(x);
    f = x - (float)i;
    if (i >= n - 1) { i = n - 2; f = 1.0f; }
    if (i < 0) { i = 0; f = 0.0f; }
}

// The cell of a pixel in the flow
struct FlowCell {
    int ix, iy;
    float fx, fy;
};

// One side: the sample of S at p + F(p r) (s / r), sx, sy = s / r, and its derivatives along x and y. Along an axis
// on which the position was clamped there is none: the derivative's first channel holds CLAMPED then, a NaN that no
// operation gives (their NaNs are 0x7fffffff, whatever payload came in).
struct Side {
    int ix, iy;      // top left corner
    float fx, fy;    // fractions
    Px val, dx, dy;
};
constexpr int CLAMPED = 0x7fc00001;
__device__ __forceinline__ float along(Px g, Px d, float s) {
    return __float_as_int(d.a.x) == CLAMPED ? 0.0f : dot4(g, d) * s;
}

__device__ __forceinline__ Side side_at(const float* S, const float* F, const AdjParams& P, const FlowCell& q, int x, int y,
                                        float sx, float sy) {
    Side d;
    const float2* f0 = reinterpret_cast<const float2*>(F) + ((long)q.iy * P.fw + q.ix);
    const float2* f1 = f0 + P.fw;
    const float2 a = f0[0], b = f0[1], c = f1[0], e = f1[1], z2 = both(P.z);
    const float2 top = step2(a, sub2(b, a), q.fx, P.z), bot = step2(c, sub2(e, c), q.fx, P.z);
    const float2 f = __fadd2_rn(__ffma2_rn(top, both(1.0f - q.fy), z2), __ffma2_rn(bot, both(q.fy), z2));
    const float2 at = __fadd2_rn(make_float2((float)x, (float)y), __ffma2_rn(f, make_float2(sx, sy), z2));
    float px = at.x, py = at.y;
    const bool cx = !(px >= 0.0f && px <= (float)(P.w - 1)), cy = !(py >= 0.0f && py <= (float)(P.h - 1));
    px = fminf(fmaxf(px, 0.0f), (float)(P.w - 1));
    py = fminf(fmaxf(py, 0.0f), (float)(P.h - 1));
    cell_of(px, P.w, d.ix, d.fx);
    cell_of(py, P.h, d.iy, d.fy);
    const long i00 = (long)d.iy * P.w + d.ix, i01 = i00 + P.w;
    const Px c00 = ld4(S, i00), c10 = ld4(S, i00 + 1), c01 = ld4(S, i01), c11 = ld4(S, i01 + 1);
    const Px d0 = sub4(c10, c00), d1 = sub4(c11, c01), e0 = sub4(c01, c00), e1 = sub4(c11, c10);
    d.val = mix4(step4(c00, d0, d.fx, P.z), step4(c01, d1, d.fx, P.z), d.fy, P.z);
    d.dx = fused4(d0, sub4(d1, d0), d.fy);
    d.dy = fused4(e0, sub4(e1, e0), d.fx);
    if (cx) d.dx.a.x = __int_as_float(CLAMPED);
    if (cy) d.dy.a.x = __int_as_float(CLAMPED);
    return d;
}

__device__ __forceinline__ void add_pixel(float* dst, const AdjParams& P, int x, int y, Px v) {
    atomicAdd(reinterpret_cast<float4*>(dst) + ((long)y * P.w + x), whole(v));
}

// A lower corner's share, carried to the row below
struct Carry {
    int x = -1, y = -1;
    Px v;
    __device__ __forceinline__ void flush(float* dst, const AdjParams& P) const {
        if (y >= 0) add_pixel(dst, P, x, y, v);
    }
};

// The image gradient of one side's pixel, g its output gradient and lg the left lane's. All lanes of the warp
// take part; `live` ones have a pixel.
__device__ __forceinline__ void add_corners(const Side& s, Px g, Px lg, bool live, float* dst, const AdjParams& P, Carry& c) {
    constexpr unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, ix = live ? s.ix : -9;
    const int lx = __shfl_up_sync(FULL, ix, 1), ly = __shfl_up_sync(FULL, s.iy, 1);
    const float lfx = __shfl_up_sync(FULL, s.fx, 1), lfy = __shfl_up_sync(FULL, s.fy, 1);
    const bool take = lane > 0 && lx + 1 == ix && ly == s.iy;
    const bool given = __shfl_down_sync(FULL, (int)take, 1) != 0 && lane < 31;
    if (!live) return;
    Px top = scale4(g, (1.0f - s.fx) * (1.0f - s.fy)), low = scale4(g, (1.0f - s.fx) * s.fy);
    if (take) {
        top = fused4(top, lg, lfx * (1.0f - lfy));
        low = fused4(low, lg, lfx * lfy);
    }
    if (!given) {
        add_pixel(dst, P, s.ix + 1, s.iy, scale4(g, s.fx * (1.0f - s.fy)));
        add_pixel(dst, P, s.ix + 1, s.iy + 1, scale4(g, s.fx * s.fy));
    }
    if (c.x == s.ix && c.y == s.iy) top = add4(top, c.v);
    else c.flush(dst, P);
    add_pixel(dst, P, s.ix, s.iy, top);
    c.x = s.ix;
    c.y = s.iy + 1;
    c.v = low;
}

// The flow gradient of a column: the sums for the upper and the lower texels of the row's cells (the same rows
// for the whole warp)
struct FlowSums {
    float2 up = {0.0f, 0.0f}, low = {0.0f, 0.0f};
};

// The sums of texel row `row` to the columns of the cell; two lanes of one column go together
__device__ __forceinline__ void add_texels(float2 s, int row, const FlowCell& q, float* dF, const AdjParams& P) {
    constexpr unsigned FULL = 0xffffffffu;
    float2 l = make_float2(s.x * (1.0f - q.fx), s.y * (1.0f - q.fx)), r = make_float2(s.x * q.fx, s.y * q.fx);
    const bool pair = __shfl_xor_sync(FULL, q.ix, 1) == q.ix;
    const float lx = __shfl_xor_sync(FULL, l.x, 1), ly = __shfl_xor_sync(FULL, l.y, 1);
    const float rx = __shfl_xor_sync(FULL, r.x, 1), ry = __shfl_xor_sync(FULL, r.y, 1);
    if (pair) {
        if (threadIdx.x & 1) return;
        l = make_float2(l.x + lx, l.y + ly);
        r = make_float2(r.x + rx, r.y + ry);
    }
    float2* to = reinterpret_cast<float2*>(dF) + ((long)row * P.fw + q.ix);
    if (l.x != 0.0f || l.y != 0.0f) atomicAdd(to, l);
    if (r.x != 0.0f || r.y != 0.0f) atomicAdd(to + 1, r);
}

// On from the cells of row `from` to those of row `to` (-1: the end)
__device__ __forceinline__ void next_texels(FlowSums& s, int from, int to, const FlowCell& q, float* dF, const AdjParams& P) {
    if (to == from) return;
    add_texels(s.up, from, q, dF, P);
    if (to == from + 1) {
        s.up = s.low;
    } else {
        add_texels(s.low, from + 1, q, dF, P);
        s.up = make_float2(0.0f, 0.0f);
    }
    s.low = make_float2(0.0f, 0.0f);
}

__device__ __forceinline__ void sum_texels(FlowSums& s, const Side& d, Px g, const FlowCell& q, float sx, float sy, bool live) {
    if (!live) return;
    // (0 along a clamped axis whatever g is: an infinity times a derivative of 0 would be a NaN)
    const float2 v = make_float2(along(g, d.dx, sx), along(g, d.dy, sy));
    s.up = __ffma2_rn(v, both(1.0f - q.fy), s.up);
    s.low = __ffma2_rn(v, both(q.fy), s.low);
}

}  // namespace

// One CTA per 32 x 32 output tile of a batch item, a warp per 8 rows, a lane per column; nothing is shared between
// warps.
//
// Bound by the gathers' latency at 16 warps an SM (128 registers; 20 warps with 96 spill: 721 us, and 4 rows a
// thread, more corners left over, 774). 16 x 1280 x 720 with the L1 loss: 574 us (612 with the clamped axes in
// flags of their own); floats added to tiles of the gradients in shared memory, a loop of compare and swap each
// and 40 a pixel, took 1.40 ms.
__global__ void __launch_bounds__(ADJ_THREADS, 4) k_warp_blend_adjoint(const __grid_constant__ AdjParams P) {
    constexpr unsigned FULL = 0xffffffffu;
    const int b = blockIdx.z, lane = threadIdx.x & 31;
    const long img = (long)P.w * P.h * 4 * b, flo = (long)P.fw * P.fh * 2 * b;
    const float *A = P.a + img, *B = P.b + img, *Fba = P.f_ba + flo, *Fab = P.f_ab + flo;
    float *da = P.da ? P.da + img : nullptr, *db = P.db ? P.db + img : nullptr;
    float *dba = P.df_ba ? P.df_ba + flo : nullptr, *dab = P.df_ab ? P.df_ab + flo : nullptr;
    const float frac = 1.0f - P.wa;
    // the steps per flow unit of the two sides (A by F_BA at 1 - wa, B by F_AB at wa)
    const float sxa = frac / P.rx, sya = frac / P.ry, sxb = P.wa / P.rx, syb = P.wa / P.ry;
    const bool backward = P.grad_out || P.target;
    const int x = blockIdx.x * ADJ_TX + lane, xs = min(x, P.w - 1), y0 = blockIdx.y * ADJ_TY + threadIdx.x / 32 * ADJ_ROWS;
    const bool live = x < P.w;
    FlowCell q;
    cell_of((float)xs * P.rx, P.fw, q.ix, q.fx);
    q.iy = -1;
    Carry ca, cb;
    FlowSums fa, fb;
    float loss = 0.0f;
#pragma unroll 1
    for (int y = y0; y < min(y0 + ADJ_ROWS, P.h); y++) {  // the same rows for the whole warp
        const int above = q.iy;
        cell_of((float)y * P.ry, P.fh, q.iy, q.fy);
        const long i = (long)y * P.w + xs;
        const float* given = P.target ? P.target : P.grad_out;  // (asked for before the gathers)
        const Px in = backward ? ld4(given + img, i) : Px{};
        const Side sa = side_at(A, Fba, P, q, xs, y, sxa, sya), sb = side_at(B, Fab, P, q, xs, y, sxb, syb);
        const Px out = mix4(sa.val, sb.val, frac, P.z);
        if (P.out && live) reinterpret_cast<float4*>(P.out + img)[i] = whole(out);
        if (!backward) continue;
        Px g;
        if (P.target) {  // the photometric L1 loss: d|out - t| / d out = sign(out - t)
            const float4 r = whole(sub4(out, in));
            if (live) loss += fabsf(r.x) + fabsf(r.y) + fabsf(r.z) + fabsf(r.w);
            auto sign = [](float v) { return v == 0.0f || isnan(v) ? 0.0f : copysignf(1.0f, v); };
            g = {make_float2(sign(r.x), sign(r.y)), make_float2(sign(r.z), sign(r.w))};
        } else {
            g = in;
        }
        const Px ga = scale4(g, 1.0f - frac), gb = scale4(g, frac);
        if (da || db) {
            const Px l = {make_float2(__shfl_up_sync(FULL, g.a.x, 1), __shfl_up_sync(FULL, g.a.y, 1)),
                          make_float2(__shfl_up_sync(FULL, g.b.x, 1), __shfl_up_sync(FULL, g.b.y, 1))};
            if (da) add_corners(sa, ga, scale4(l, 1.0f - frac), live, da, P, ca);
            if (db) add_corners(sb, gb, scale4(l, frac), live, db, P, cb);
        }
        if (dba) {
            if (above >= 0) next_texels(fa, above, q.iy, q, dba, P);
            sum_texels(fa, sa, ga, q, sxa, sya, live);
        }
        if (dab) {
            if (above >= 0) next_texels(fb, above, q.iy, q, dab, P);
            sum_texels(fb, sb, gb, q, sxb, syb, live);
        }
    }
    if (backward && y0 < P.h) {
        if (da) ca.flush(da, P);
        if (db) cb.flush(db, P);
        if (dba) next_texels(fa, q.iy, -1, q, dba, P);
        if (dab) next_texels(fb, q.iy, -1, q, dab, P);
    }
    if (P.loss) {  // the loss of the batch item: a warp shuffle sum, one atomic per warp
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) loss += __shfl_down_sync(FULL, loss, o);
        if (lane == 0 && loss != 0.0f) atomicAdd(P.loss + b, loss);
    }
}

}  // namespace tw
