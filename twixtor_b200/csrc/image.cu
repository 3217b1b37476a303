// Image boundary, luma, inverse warps and blends, strict mode. Each kernel cites the reference
// function (plugins/retime-engine/src/...) whose per-element arithmetic it repeats.
#include "kernels.cuh"
#include "luma.cuh"
#include "warp.cuh"
#include "blend.cuh"

namespace tw {

// ---- wire -> engine (image.rs:178-206, premultiply :276-303) ----------------------------------------

// The wire element of engine element i (w x h, rows bottom up with flip)
__device__ __forceinline__ long wire_at(long i, int w, int h, bool flip) {
    if (!flip) return i;
    const int y = row_of(i, w);
    return (long)(h - 1 - y) * w + (i - (long)y * w);
}

__global__ void k_from_frame_u8(const uint8_t* __restrict__ wire, uint8_t* __restrict__ eng, int w, int h, bool flip) {
    long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    long n = (long)w * h;
    if (i >= n) return;
    float p[4], o[4];  // r, g, b, a
    px_floats<uint8_t>(wire + wire_at(i, w, h, flip) * 4, p);
    float a = p[3] * inv_255();
    o[0] = p[3];
#pragma unroll
    for (int c = 0; c < 3; c++) o[c + 1] = px_rounded(p[c] * a);
    px_store(eng + i * 4, o);
}

__global__ void k_from_frame_u16(const uint16_t* __restrict__ wire, uint16_t* __restrict__ eng, int w, int h, bool flip) {
    long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    long n = (long)w * h;
    if (i >= n) return;
    ushort4 p = reinterpret_cast<const ushort4*>(wire)[wire_at(i, w, h, flip)];
    uint16_t A = u16_to_q15(p.w), R = u16_to_q15(p.x), G = u16_to_q15(p.y), Bc = u16_to_q15(p.z);
    float a = (float)A * premul16_color();
    ushort4 o;
    o.x = (uint16_t)qround((float)A * premul16_alpha());
    o.y = (uint16_t)qround((float)R * a);
    o.z = (uint16_t)qround((float)G * a);
    o.w = (uint16_t)qround((float)Bc * a);
    reinterpret_cast<ushort4*>(eng)[i] = o;
}

__global__ void k_from_frame_f32(const float* __restrict__ wire, float* __restrict__ eng, int w, int h, bool flip) {
    long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    long n = (long)w * h;
    if (i >= n) return;
    long si = wire_at(i, w, h, flip);
    // planes G, B, R, A
    float g = wire[si], b = wire[n + si], r = wire[2 * n + si], a = wire[3 * n + si];
    float o1 = a * r, o2 = a * g, o3 = a * b;
    if (isnan(o1) || isnan(o2) || isnan(o3) || isnan(a)) {
        o1 = nr::mul(a, r);
        o2 = nr::mul(a, g);
        o3 = nr::mul(a, b);
    }
    reinterpret_cast<float4*>(eng)[i] = make_float4(a, o1, o2, o3);
}

// ---- engine -> wire (image.rs:213-245, unpremultiply :306-351) --------------------------------------

// Whole samples a, r, g, b as floats -> r, g, b, a; an opaque pixel's factor is 1
__device__ __forceinline__ void unpremul_u8(const float p[4], float o[4]) {
    o[0] = p[1];
    o[1] = p[2];
    o[2] = p[3];
    o[3] = p[0];
    if (p[0] == 0.0f || p[0] == 255.0f) return;
    const float s = 255.0f / p[0];
#pragma unroll
    for (int c = 0; c < 3; c++) o[c] = px_rounded(fminf(o[c] * s, 255.0f));
}

__device__ __forceinline__ void unpremul_u16(const float p[4], float o[4]) {
    uint32_t q[4] = {(uint32_t)p[1], (uint32_t)p[2], (uint32_t)p[3], (uint32_t)p[0]};
    if (p[0] != 0.0f) {
        const float s = p[0] == 32768.0f ? 1.0f : 32768.0f / p[0];
#pragma unroll
        for (int c = 0; c < 3; c++) q[c] = qround(p[c + 1] * s);
        q[3] = qround(p[0] * unpremul16_alpha());
    }
#pragma unroll
    for (int c = 0; c < 4; c++) o[c] = (float)q15_to_u16((uint16_t)q[c]);
}

__device__ __forceinline__ float4 unpremul_f32(float4 p) {  // -> a, r, g, b (engine order)
    if ((double)p.x < 1e-12) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    // `1.0 / a` keeps a NaN alpha's payload as the x86 divide does (the quieted NaN operand)
    float inv = nr::div(1.0f, p.x);
    float r = p.y * inv, g = p.z * inv, b = p.w * inv;
    if (isnan(r) || isnan(g) || isnan(b) || isnan(p.x)) {
        r = nr::mul(p.y, inv);
        g = nr::mul(p.z, inv);
        b = nr::mul(p.w, inv);
    }
    return make_float4(p.x, r, g, b);
}

__global__ void k_to_frame_u8(const uint8_t* __restrict__ eng, uint8_t* __restrict__ wire, int w, int h, bool flip) {
    long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    long n = (long)w * h;
    if (i >= n) return;
    long si = wire_at(i, w, h, flip);
    float p[4], o[4];
    px_floats<uint8_t>(eng + si * 4, p);
    unpremul_u8(p, o);
    px_store(wire + i * 4, o);
}

__global__ void k_to_frame_u16(const uint16_t* __restrict__ eng, uint16_t* __restrict__ wire, int w, int h, bool flip) {
    long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    long n = (long)w * h;
    if (i >= n) return;
    long si = wire_at(i, w, h, flip);
    float p[4], o[4];
    px_floats<uint16_t>(eng + si * 4, p);
    unpremul_u16(p, o);
    px_store(wire + i * 4, o);
}

__global__ void k_to_frame_f32(const float* __restrict__ eng, float* __restrict__ wire, int w, int h, bool flip) {
    long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    long n = (long)w * h;
    if (i >= n) return;
    long si = wire_at(i, w, h, flip);
    float4 o = unpremul_f32(reinterpret_cast<const float4*>(eng)[si]);
    wire[i] = o.z;          // G
    wire[n + i] = o.w;      // B
    wire[2 * n + i] = o.y;  // R
    wire[3 * n + i] = o.x;  // A
}

// ---- luma (prep.rs:168-235) ------------------------------------------------------------------------

__global__ void k_luma(const void* __restrict__ eng, int fmt, float* __restrict__ out, int w, int h, bool track_alpha,
                       bool video_range) {
    long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    long n = (long)w * h;
    if (i >= n) return;
    out[i] = luma_px(eng, fmt, i, (track_alpha ? LUMA_TRACK_ALPHA : 0) | (video_range ? LUMA_VIDEO_RANGE : 0));
}

template <typename P>
__device__ __forceinline__ void inv_warp_px(const WarpParams& p, void* out, uint8_t* cov, int w, int h, int* bad) {
    int x = blockIdx.x * blockDim.x + threadIdx.x;
    int y = blockIdx.y;
    if (x >= w || y >= h) return;
    float o[4];
    bool b = false;
    uint8_t c = warp_pixel<P>(p, x, y, w, h, o, b);
    px_store((P*)out + ((long)y * w + x) * 4, o);
    if (cov) cov[(long)y * w + x] = c;
    if (b) atomicOr(bad, 1);
}

__global__ void k_inv_warp(WarpParams p, int fmt, void* __restrict__ out, uint8_t* __restrict__ cov, int w, int h,
                           int* __restrict__ bad) {
    if (fmt == 0) inv_warp_px<uint8_t>(p, out, cov, w, h, bad);
    else if (fmt == 1) inv_warp_px<uint16_t>(p, out, cov, w, h, bad);
    else inv_warp_px<float>(p, out, cov, w, h, bad);
}

// ---- blend and lerp (blend.rs) -----------------------------------------------------------------------

__global__ void k_blend(const void* __restrict__ a, const void* __restrict__ b, void* __restrict__ out, int fmt,
                        long nsamples, float w) {
    long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nsamples) return;
    if (fmt == 0) ((uint8_t*)out)[i] = blend_sample<uint8_t>(((const uint8_t*)a)[i], ((const uint8_t*)b)[i], w);
    else if (fmt == 1) ((uint16_t*)out)[i] = blend_sample<uint16_t>(((const uint16_t*)a)[i], ((const uint16_t*)b)[i], w);
    else ((float*)out)[i] = blend_sample<float>(((const float*)a)[i], ((const float*)b)[i], w);
}

template <typename P>
__device__ __forceinline__ void lerp_one(void* first, const void* second, long i, float w) {
    P f[4], s[4];
    P* fp = (P*)first + i * 4;
    const P* sp = (const P*)second + i * 4;
#pragma unroll
    for (int k = 0; k < 4; k++) { f[k] = fp[k]; s[k] = sp[k]; }
    lerp_px<P>(f, s, w);
#pragma unroll
    for (int k = 0; k < 4; k++) fp[k] = f[k];
}

__global__ void k_lerp(void* __restrict__ first, const void* __restrict__ second, int fmt, long npx, float w) {
    long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= npx) return;
    if (fmt == 0) lerp_one<uint8_t>(first, second, i, w);
    else if (fmt == 1) lerp_one<uint16_t>(first, second, i, w);
    else lerp_one<float>(first, second, i, w);
}

// ---- the fused Blend composition of warping code 0 ---------------------------------------------------

// Samples as floats into the engine image, or unpremultiplied into the wire frame
__device__ __forceinline__ void store_px(const float o[4], uint8_t* out, long i, bool to_wire, long npx) {
    float u[4] = {o[0], o[1], o[2], o[3]};
    if (to_wire) unpremul_u8(o, u);
    px_store(out + i * 4, u);
}
__device__ __forceinline__ void store_px(const float o[4], uint16_t* out, long i, bool to_wire, long npx) {
    float u[4] = {o[0], o[1], o[2], o[3]};
    if (to_wire) unpremul_u16(o, u);
    px_store(out + i * 4, u);
}
__device__ __forceinline__ void store_px(const float o[4], float* out, long i, bool to_wire, long npx) {
    if (!to_wire) {
        px_store(out + i * 4, o);
        return;
    }
    float4 u = unpremul_f32(make_float4(o[0], o[1], o[2], o[3]));
    out[i] = u.z;
    out[npx + i] = u.w;
    out[2 * npx + i] = u.y;
    out[3 * npx + i] = u.x;
}

// blend_sample of a pair, samples and result as floats: with 0 <= w <= 1 (the common branch) an integer
// depth's sum is in its range, and a NaN weight's is stored as 0
template <typename P>
__device__ __forceinline__ float2 blend_pair(float2 a, float2 b, float w, float z) {
    float2 t = __fadd2_rn(__ffma2_rn(__ffma2_rn(a, make_float2(-1.0f, -1.0f), b), make_float2(w, w), make_float2(z, z)), a);
    t = __fadd2_rn(t, make_float2(0.5f, 0.5f));
    return make_float2(trunc_biased(fmaxf(t.x, 0.0f)) - PX_BIAS, trunc_biased(fmaxf(t.y, 0.0f)) - PX_BIAS);
}

// Both warps, the blend and the store of a pixel. A thread takes one pixel: a frame has some hundred times the
// threads that the chip holds, and the gathers want many in flight.
template <typename P>
__device__ __forceinline__ void compose_blend_px(const WarpParams& pa, const WarpParams& pb, float wblend, int mode,
                                                 void* out, int w, int h, bool to_wire, bool flip_out, int* bad) {
    int x = blockIdx.x * blockDim.x + threadIdx.x;
    int y = blockIdx.y;
    if (x >= w || y >= h) return;
    // the output pixel (x, y) of the engine image lands on wire row h-1-y when flip_out
    float ta[4], tb[4], o[4];
    bool b = false;
    if (mode != 2) warp_pixel<P>(pa, x, y, w, h, ta, b);
    if (mode != 1) warp_pixel<P>(pb, x, y, w, h, tb, b);
    if (mode == 0 && sizeof(P) < 4) {
        const float2 u = blend_pair<P>(make_float2(ta[0], ta[1]), make_float2(tb[0], tb[1]), wblend, pa.z);
        const float2 v = blend_pair<P>(make_float2(ta[2], ta[3]), make_float2(tb[2], tb[3]), wblend, pa.z);
        o[0] = u.x; o[1] = u.y; o[2] = v.x; o[3] = v.y;
    } else if (mode == 1 || mode == 2) {
#pragma unroll
        for (int k = 0; k < 4; k++) o[k] = mode == 1 ? ta[k] : tb[k];
    } else {
        P qa[4], qb[4], qo[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            qa[k] = (P)ta[k];
            qb[k] = (P)tb[k];
        }
        blend_px<P>(qa, qb, wblend, mode == 3 ? (float)(1.0 - (double)wblend) : 0.0f, mode, qo);
#pragma unroll
        for (int k = 0; k < 4; k++) o[k] = (float)qo[k];
    }
    int oy = flip_out ? h - 1 - y : y;
    store_px(o, (P*)out, (long)oy * w + x, to_wire, (long)w * h);
    if (b) atomicOr(bad, 1);
}

__global__ void k_compose_blend(WarpParams pa, WarpParams pb, int fmt, float wblend, int blend_mode, void* __restrict__ out,
                                int w, int h, bool to_wire, bool flip_out, int* __restrict__ bad) {
    if (fmt == 0) compose_blend_px<uint8_t>(pa, pb, wblend, blend_mode, out, w, h, to_wire, flip_out, bad);
    else if (fmt == 1) compose_blend_px<uint16_t>(pa, pb, wblend, blend_mode, out, w, h, to_wire, flip_out, bad);
    else compose_blend_px<float>(pa, pb, wblend, blend_mode, out, w, h, to_wire, flip_out, bad);
}

// ---- the vector encoder (vectors.rs:57-130) ---------------------------------------------------------
// Per output pixel: the flow sampled with the warps' flow sampler (warp.rs:415-442) at (x sx, y sy),
// scaled by (kx, ky), then the depth's store; zero != 0 writes the zero vector image
// (vectors.rs:148-156). Writes the engine image (A, R, G, B).
__global__ void k_encode_vectors(const float* __restrict__ flow, int fw, int fh, void* __restrict__ out, int W, int H,
                                 int fmt, float sx, float sy, float kx, float ky, int zero) {
    int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
    if (x >= W || y >= H) return;
    float a = 0.0f, b = 0.0f;
    if (!zero) {
        float px = (float)x * sx, py = (float)y * sy;
        int fw1 = fw - 1, fh1 = fh - 1;
        int ix = cvtt32(px), iy = cvtt32(py);
        float fx = px - (float)ix, fy = py - (float)iy;
        if (ix >= fw1) { ix = fw1 - 1; fx = 1.0f; }
        if (iy >= fh1) { iy = fh1 - 1; fy = 1.0f; }
        long i00 = ((long)iy * fw + ix) * 2, i01 = i00 + (long)fw * 2;
        // x86 arithmetic: a NaN vector (a NaN or infinite flow) keeps the reference's bits in the
        // float depth's output
        float o[2];
#pragma unroll
        for (int k = 0; k < 2; k++) {
            float p00 = flow[i00 + k], p10 = flow[i00 + 2 + k], p01 = flow[i01 + k], p11 = flow[i01 + 2 + k];
            float top = x86::add(x86::mul(x86::sub(p10, p00), fx), p00);
            float bot = x86::add(x86::mul(x86::sub(p11, p01), fx), p01);
            o[k] = x86::add(x86::mul(x86::sub(bot, top), fy), top);
        }
        a = x86::mul(o[0], kx);
        b = x86::mul(o[1], ky);
    }
    long i = ((long)y * W + x) * 4;
    if (fmt == 2) {
        float* d = (float*)out + i;
        d[0] = 1.0f;
        d[1] = x86::mul(x86::add(a, 1.0f), 0.5f);
        d[2] = x86::mul(x86::add(b, 1.0f), 0.5f);
        d[3] = 0.0f;
        return;
    }
    if (a > 1.0f) a = 1.0f;  // vectors.rs:133-140: a NaN falls through
    else if (-1.0f > a) a = -1.0f;
    if (b > 1.0f) b = 1.0f;
    else if (-1.0f > b) b = -1.0f;
    a = a + 1.0f;
    b = b + 1.0f;
    if (fmt == 0) {
        uint8_t* d = (uint8_t*)out + i;
        d[0] = 0xff;
        d[1] = (uint8_t)cvtt64d((double)a * 127.0 + 0.5);
        d[2] = (uint8_t)cvtt64d((double)b * 127.0 + 0.5);
        d[3] = 0;
    } else {
        uint16_t* d = (uint16_t*)out + i;
        d[0] = 0xffff;
        d[1] = (uint16_t)cvtt64d((double)a * 32767.0 + 0.5);
        d[2] = (uint16_t)cvtt64d((double)b * 32767.0 + 0.5);
        d[3] = 0;
    }
}

}  // namespace tw
