// The inverse warp of one output pixel (warp.rs:290-561), shared by the warp, Blend and Smart Blend
// kernels. Strict mode: single precision in the reference's order, the NaN rule repeat of the
// float depth, x86 truncations.
//
// Bound by instruction issue: a pixel's four channels go as two packed pairs, a pixel and a flow vector are one
// load each, and integer samples are read as floats biased by 2^23 (a byte permute each; the differences of
// two are exact, so that only the corners that are added drop the bias) and stored by trunc_biased: no
// conversions, no doubles. The Blend composition of a 1080p 8 bit frame, 550 instructions per pixel with scalar
// loads, lerps and conversions, went from 64 to 41 us (each launch between events).
#pragma once
#include "kernels.cuh"

namespace tw {

template <typename P> struct Pix;
template <> struct Pix<uint8_t> {
    __device__ static float f(uint8_t v) { return (float)v; }
    __device__ static uint8_t store(float v) { return sat_u8(v); }
    // warp.rs:152-155: the stored sample scaled by the fade, the add in double
    __device__ static uint8_t faded(float v, float f) { return (uint8_t)cvtt64d((double)((float)sat_u8(v) * f) + 0.5); }
};
template <> struct Pix<uint16_t> {
    __device__ static float f(uint16_t v) { return (float)v; }
    __device__ static uint16_t store(float v) { return sat_u16(v); }
    __device__ static uint16_t faded(float v, float f) { return (uint16_t)cvtt64d((double)((float)sat_u16(v) * f) + 0.5); }
};
template <> struct Pix<float> {
    __device__ static float f(float v) { return v; }
    __device__ static float store(float v) { return v; }
    // a NaN sample keeps its payload through the fade product, as on x86
    __device__ static float faded(float v, float f) { return nr::mul(v, f); }
};

// warp.rs:178-215 (clip_to_rect), bounded like the reference
__device__ __forceinline__ bool clip_to_rect(float x, float y, float& ix, float& iy, float w1, float h1) {
#pragma unroll 1
    for (int it = 0; it < 4096; it++) {
        if (ix < 0.0f) {
            float dy = y - iy, dxs = x - ix, num = x - 0.0f;
            ix = 0.0f;
            iy = y - (num / dxs) * dy;
            continue;
        }
        if (ix > w1) {
            float dy = y - iy, dxs = x - ix, num = x - w1;
            ix = w1;
            iy = y - (num / dxs) * dy;
            continue;
        }
        if (iy < 0.0f) {
            float dyy = y - iy, num = y - 0.0f, dx = x - ix;
            ix = x - (num / dyy) * dx;
            iy = 0.0f;
            continue;
        }
        if (iy > h1) {
            float dyy = y - iy, num = y - h1, dx = x - ix;
            ix = x - (num / dyy) * dx;
            iy = h1;
            continue;
        }
        return true;
    }
    return false;
}

// Four samples of a pixel as two pairs. The integer depths hold them biased by 2^23.
struct Px4 {
    float2 a, b;
};
constexpr float PX_BIAS = 8388608.0f;  // 2^23
__device__ __forceinline__ float biased(uint32_t v, uint32_t sel) { return __uint_as_float(__byte_perm(v, 0x4b000000u, sel)); }
__device__ __forceinline__ Px4 px_load(const uint8_t* p) {
    const uint32_t v = *(const uint32_t*)p;
    return {make_float2(biased(v, 0x7540), biased(v, 0x7541)), make_float2(biased(v, 0x7542), biased(v, 0x7543))};
}
__device__ __forceinline__ Px4 px_load(const uint16_t* p) {
    const uint2 v = *(const uint2*)p;
    return {make_float2(biased(v.x, 0x7410), biased(v.x, 0x7432)), make_float2(biased(v.y, 0x7410), biased(v.y, 0x7432))};
}
__device__ __forceinline__ Px4 px_load(const float* p) {
    const float4 v = *(const float4*)p;
    return {make_float2(v.x, v.y), make_float2(v.z, v.w)};
}
// The samples as they are
template <typename P>
__device__ __forceinline__ float2 px_value(float2 v) {
    return sizeof(P) == 4 ? v : __fadd2_rn(v, make_float2(-PX_BIAS, -PX_BIAS));
}
template <typename P>
__device__ __forceinline__ void px_floats(const P* p, float o[4]) {
    const Px4 v = px_load(p);
    const float2 a = px_value<P>(v.a), b = px_value<P>(v.b);
    o[0] = a.x; o[1] = a.y; o[2] = b.x; o[3] = b.y;
}
// Samples that are floats of whole numbers in the depth's range (float depth: any) into a pixel
__device__ __forceinline__ void px_store(uint8_t* p, const float v[4]) {
    uint32_t b[4];
#pragma unroll
    for (int k = 0; k < 4; k++) b[k] = __float_as_uint(v[k] + PX_BIAS);
    *(uint32_t*)p = __byte_perm(__byte_perm(b[0], b[1], 0x0040), __byte_perm(b[2], b[3], 0x0040), 0x5410);
}
__device__ __forceinline__ void px_store(uint16_t* p, const float v[4]) {
    uint32_t b[4];
#pragma unroll
    for (int k = 0; k < 4; k++) b[k] = __float_as_uint(v[k] + PX_BIAS);
    *(uint2*)p = make_uint2(__byte_perm(b[0], b[1], 0x5410), __byte_perm(b[2], b[3], 0x5410));
}
__device__ __forceinline__ void px_store(float* p, const float v[4]) { *(float4*)p = make_float4(v[0], v[1], v[2], v[3]); }

// qround of 0 <= v < 2^22 as a float
__device__ __forceinline__ float px_rounded(float v) { return trunc_biased(__fadd_rz(v, 0.5f)) - PX_BIAS; }

// a + (b - a) * f of a pair whose `a` without the bias is a0
__device__ __forceinline__ float2 px_lerp(float2 a0, float2 a, float2 b, float2 f, float2 z) {
    return __fadd2_rn(a0, __ffma2_rn(__ffma2_rn(a, make_float2(-1.0f, -1.0f), b), f, z));
}

// warp.rs:339-352 (mix4): the three lerps of four taps, for the float depth repeated with the NaN rule when
// NaN (an integer depth has none: its taps are numbers, and no NaN coordinate comes this far)
template <typename P>
__device__ __forceinline__ void mix4(const P* p00, const P* p10, const P* p01, const P* p11, float fx, float fy, float z,
                                     float o[4]) {
    const Px4 a = px_load(p00), b = px_load(p10), c = px_load(p01), d = px_load(p11);
    const float2 fx2 = make_float2(fx, fx), fy2 = make_float2(fy, fy), z2 = make_float2(z, z);
    auto mix = [&](float2 pa, float2 pb, float2 pc, float2 pd) {
        const float2 top = px_lerp(px_value<P>(pa), pa, pb, fx2, z2), bot = px_lerp(px_value<P>(pc), pc, pd, fx2, z2);
        return px_lerp(top, top, bot, fy2, z2);
    };
    const float2 u = mix(a.a, b.a, c.a, d.a), v = mix(a.b, b.b, c.b, d.b);
    o[0] = u.x; o[1] = u.y; o[2] = v.x; o[3] = v.y;
    if (sizeof(P) == 4 && (isnan(o[0]) || isnan(o[1]) || isnan(o[2]) || isnan(o[3]))) {
        auto rule = [&](float w00, float w10, float w01, float w11) {
            float top = nr::add(w00, nr::mul(nr::sub(w10, w00), fx));
            float bot = nr::add(w01, nr::mul(nr::sub(w11, w01), fx));
            return nr::add(top, nr::mul(nr::sub(bot, top), fy));
        };
        o[0] = rule(a.a.x, b.a.x, c.a.x, d.a.x);
        o[1] = rule(a.a.y, b.a.y, c.a.y, d.a.y);
        o[2] = rule(a.b.x, b.b.x, c.b.x, d.b.x);
        o[3] = rule(a.b.y, b.b.y, c.b.y, d.b.y);
    }
}

// warp.rs:290-360 (bilerp4). z: -0.0, from a kernel's arguments (see mix4's products)
template <typename P>
__device__ __forceinline__ void bilerp4(const P* __restrict__ src, int w, int w1, int h1, float x, float y, float z, float o[4]) {
    int ix = cvtt32(x), iy = cvtt32(y);
    float fx = x - (float)ix, fy = y - (float)iy;
    if (ix >= w1) { ix = w1 - 1; fx = 1.0f; }
    if (iy >= h1) { iy = h1 - 1; fy = 1.0f; }
    const P* p = src + ((long)iy * w + ix) * 4;
    const P* q = p + (long)w * 4;
    mix4<P>(p, p + 4, q, q + 4, fx, fy, z, o);
}

// warp.rs:362-396 (bilerp360): the coordinates already in [0, W) x [0, H); the right neighbour of
// the last column is column 0, below the last row the taps are the last row's shifted by half the
// width
template <typename P>
__device__ __forceinline__ void bilerp360(const P* __restrict__ src, int w, int w1, int h1, float x, float y, float z, float o[4]) {
    int ix = cvtt32(x), iy = cvtt32(y);
    float fx = x - (float)ix, fy = y - (float)iy;
    int x1 = ix + 1 > w1 ? 0 : ix + 1;
    int xc, xd, yc;
    if (iy + 1 > h1) {
        int half = w / 2;
        xc = (half + ix) % w;
        xd = (half + x1) % w;
        yc = h1;
    } else {
        xc = ix;
        xd = x1;
        yc = iy + 1;
    }
    int ya = min(iy, h1);
    xc = max(xc, 0);
    xd = max(xd, 0);
    auto at = [&](int xx, int yy) { return src + ((long)yy * w + xx) * 4; };
    mix4<P>(at(ix, ya), at(x1, ya), at(xc, yc), at(xd, yc), fx, fy, z, o);
}

// warp.rs:563-621 (pixel_360): wrapped by whole turns (at most 2^16 steps, else bad), an odd number
// of vertical wraps reflected over the pole, then the 360 sampler; the coverage stays 255
template <typename P>
__device__ __forceinline__ void pixel_360(const P* src, int w, int h, float ix, float iy, float z, float o[4], bool& bad) {
    const uint32_t WRAP_LIMIT = 1u << 16;
    float wf = (float)w, hf = (float)h;
    uint32_t guard = 0, n = 0;
    while (ix < 0.0f) { ix += wf; if (++guard > WRAP_LIMIT) break; }
    while (wf <= ix) { ix -= wf; if (++guard > WRAP_LIMIT) break; }
    while (iy < 0.0f) { iy += hf; n++; if (++guard > WRAP_LIMIT) break; }
    while (hf <= iy) { iy -= hf; n++; if (++guard > WRAP_LIMIT) break; }
    if (guard > WRAP_LIMIT || !(ix >= 0.0f && ix < wf) || isnan(iy)) {
        bad = true;
#pragma unroll
        for (int k = 0; k < 4; k++) o[k] = 0.0f;
        return;
    }
    if (n & 1) {
        ix = wf * 0.5f + ix;
        if (ix >= wf) ix -= wf;
        if (iy != 0.0f) iy = hf - iy;
    }
    float s[4];
    bilerp360<P>(src, w, w - 1, h - 1, ix, iy, z, s);
#pragma unroll
    for (int k = 0; k < 4; k++) o[k] = (float)Pix<P>::store(s[k]);
}

// warp.rs:415-442 (Flow::bilerp) on a strided field
__device__ __forceinline__ void flow_bilerp(const WarpParams& p, float x, float y, float& du, float& dv) {
    int fw1 = p.fw - 1, fh1 = p.fh - 1;
    int ix = cvtt32(x), iy = cvtt32(y);
    float fx = x - (float)ix, fy = y - (float)iy;
    if (ix >= fw1) { ix = fw1 - 1; fx = 1.0f; }
    if (iy >= fh1) { iy = fh1 - 1; fy = 1.0f; }
    float2 v00, v10, v01, v11;
    if (p.pairs) {
        const float2* q = reinterpret_cast<const float2*>(p.fu) + ((long)iy * p.fw + ix);
        v00 = __ldg(q);
        v10 = __ldg(q + 1);
        v01 = __ldg(q + p.fw);
        v11 = __ldg(q + p.fw + 1);
    } else {
        const long s = p.fstride, i00 = ((long)iy * p.fw + ix) * s, i01 = i00 + (long)p.fw * s;
        v00 = make_float2(__ldg(p.fu + i00), __ldg(p.fv + i00));
        v10 = make_float2(__ldg(p.fu + i00 + s), __ldg(p.fv + i00 + s));
        v01 = make_float2(__ldg(p.fu + i01), __ldg(p.fv + i01));
        v11 = make_float2(__ldg(p.fu + i01 + s), __ldg(p.fv + i01 + s));
    }
    const float2 fx2 = make_float2(fx, fx), z2 = make_float2(p.z, p.z);
    const float2 top = px_lerp(v00, v00, v10, fx2, z2), bot = px_lerp(v01, v01, v11, fx2, z2);
    const float2 r = px_lerp(top, top, bot, make_float2(fy, fy), z2);
    du = r.x;
    dv = r.y;
}

// A bilinear sample of an integer depth as stored: its value is in the depth's range (each lerp of numbers in
// it rounds into it), so the reference's saturations have nothing to do.
template <typename P>
__device__ __forceinline__ float px_stored(float v) {
    return sizeof(P) == 4 ? v : trunc_biased(v + 0.5f) - PX_BIAS;
}

// One output pixel of the inverse warp (warp.rs:466-561, Kernel::row / pixel_hold / pixel_fade).
// Returns the coverage byte, and the stored samples as floats; sets bad for a coordinate the reference
// refuses.
template <typename P>
__device__ __forceinline__ uint8_t warp_pixel(const WarpParams& p, int x, int y, int w, int h, float o[4], bool& bad) {
    const P* src = (const P*)p.src;
    if (p.copy_only) {
        px_floats<P>(src + ((long)y * w + x) * 4, o);
        return 255;
    }
    int w1i = w - 1, h1i = h - 1;
    const float rx = p.rx, ry = p.ry, sx = p.sx, sy = p.sy;  // formed on the host (warp_params)
    float wf = (float)w, hf = (float)h, w1 = (float)w1i, h1 = (float)h1i;
    float xf = (float)x, yf = (float)y;
    float du, dv;
    flow_bilerp(p, xf * rx, yf * ry, du, dv);
    float ix = du * sx + xf;
    float iy = dv * sy + yf;
    float s[4];
    if (p.is360) {
        pixel_360<P>(src, w, h, ix, iy, p.z, o, bad);
        return 255;
    }
    const bool inside = ix >= 0.0f && ix <= w1 && iy >= 0.0f && iy <= h1;
    if (p.hold && !inside && (!clip_to_rect(xf, yf, ix, iy, w1, h1) || isnan(ix) || isnan(iy))) {
        bad = true;
#pragma unroll
        for (int k = 0; k < 4; k++) o[k] = 0.0f;
        return 255;
    }
    if (!p.hold && !(ix > -1.0f && ix < wf && iy > -1.0f && iy < hf)) {
#pragma unroll
        for (int k = 0; k < 4; k++) o[k] = 0.0f;
        return 0;
    }
    if (p.hold || inside) {
        bilerp4<P>(src, w, w1i, h1i, ix, iy, p.z, s);
#pragma unroll
        for (int k = 0; k < 4; k++) o[k] = px_stored<P>(s[k]);
        return 255;
    }
    float f = ix < 0.0f ? ix + 1.0f : (ix <= w1 ? 1.0f : wf - ix);
    if (iy < 0.0f) f *= iy + 1.0f;
    else if (iy > h1) f *= hf - iy;
    if (!clip_to_rect(xf, yf, ix, iy, w1, h1) || isnan(ix) || isnan(iy)) {
        bad = true;
#pragma unroll
        for (int k = 0; k < 4; k++) o[k] = 0.0f;
        return 0;
    }
    bilerp4<P>(src, w, w1i, h1i, ix, iy, p.z, s);
#pragma unroll
    for (int k = 0; k < 4; k++) o[k] = (float)Pix<P>::faded(s[k], f);
    float c = f * 255.0f + 0.5f;
    return c <= 255.0f ? (uint8_t)cvtt64d((double)c) : (uint8_t)255;
}

}  // namespace tw
