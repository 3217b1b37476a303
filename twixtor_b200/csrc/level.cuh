// Per element rules shared by the solver's kernels (the tiled level kernels, block matching and the
// persistent coarse-level solve): the separable filter element with its border rule
// (flow/conv.rs), Block::cost of block matching (flow.rs:474-523) and the range state of a level
// (flow.rs:1292-1300). Each repeats the reference's operation order, so every kernel that calls
// them computes the same bits.
#pragma once
#include "kernels.cuh"

namespace tw {

// ---- packed pairs ------------------------------------------------------------------------------------
// The two channels of B and of the flow (and two of the tensor's three) travel as float2 through the
// separable passes: one packed instruction rounds both lanes as the scalar one does, so the bits are
// the same for half the issue slots (the FP32 pipe takes a packed operation in two cycles: 127 scalar
// results per clock and SM either way, measured).
//
// The assembler contracts a packed multiply and a packed add into one fused operation whatever
// -fmad=false and the .rn say (measured: every one of a million sums differed). So a product is
// written as a * k + z with z = -0.0, which rounds exactly as the product does, zeros and their signs
// included, and z is a value the compiler cannot know: it comes with the kernel's parameters (Taps::z).
__device__ __forceinline__ float2 vadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 vmul(float2 a, float k, float z) {
    return __ffma2_rn(a, make_float2(k, k), make_float2(z, z));
}
__device__ __forceinline__ float2 vmadd(float2 s, float2 a, float k, float z) {  // s + a * k
#ifdef TW_FAST_VARIANT
    return __ffma2_rn(a, make_float2(k, k), s);
#else
    return __fadd2_rn(s, vmul(a, k, z));
#endif
}
__device__ __forceinline__ float vadd(float a, float b) { return a + b; }
__device__ __forceinline__ float vmul(float a, float k, float) { return a * k; }
__device__ __forceinline__ float vmadd(float s, float a, float k, float) { return s + a * k; }
// a / d for a weight sum d (0.05 < d <= 1) and y = 1 / d, both correctly rounded: Markstein's division by
// a known reciprocal (P. Markstein, "Computation of elementary functions on the IBM RISC System/6000
// processor", 1990): q1 = a y corrected by its exact remainder is faithful, and a second correction by the
// exact remainder of q1 rounds it correctly. Two lanes share each step. A zero keeps its sign; an
// operand too near the range's ends for the exact remainders shows in `seen` (its magnitudes' largest and
// smallest but zero), and the caller redoes it by the division. (A division here, even one that is
// never taken, holds up the zero filled rows outside the image in its slow path: 7000 cycles for the
// border rows of a tile, 3100 without.)
struct Magnitudes {
    float hi = 0.0f, lo = 1.0f;
    __device__ __forceinline__ bool safe() const { return hi < 1e30f && lo > 1e-30f; }
};
__device__ __forceinline__ float quot1(float a, float q, Magnitudes& seen) {
    seen.hi = fmaxf(seen.hi, fabsf(a));
    seen.lo = fminf(seen.lo, a == 0.0f ? 1.0f : fabsf(a));
    return a == 0.0f ? a : q;
}
__device__ __forceinline__ float2 vquot(float2 a, float2 dy, Magnitudes& seen) {
    const float2 n = make_float2(-dy.x, -dy.x), y = make_float2(dy.y, dy.y);
    float2 q = __ffma2_rn(a, y, make_float2(0.0f, 0.0f));
    q = __ffma2_rn(__ffma2_rn(q, n, a), y, q);
    q = __ffma2_rn(__ffma2_rn(q, n, a), y, q);
    return make_float2(quot1(a.x, q.x, seen), quot1(a.y, q.y, seen));
}
__device__ __forceinline__ float vquot(float a, float2 dy, Magnitudes& seen) {
    float q = a * dy.y;
    q = __fmaf_rn(__fmaf_rn(q, -dy.x, a), dy.y, q);
    q = __fmaf_rn(__fmaf_rn(q, -dy.x, a), dy.y, q);
    return quot1(a, q, seen);
}
// how far the nearest sample is from the sentinel -1.0 of the border rule (0: it is the sentinel)
__device__ __forceinline__ float from_sentinel(float2 v, float m) {
    const float2 d = __fadd2_rn(v, make_float2(1.0f, 1.0f));
    return fminf(fminf(m, fabsf(d.x)), fabsf(d.y));
}
__device__ __forceinline__ float from_sentinel(float v, float m) { return fminf(m, fabsf(v + 1.0f)); }
template <class V>
__device__ __forceinline__ V outside_value();  // -0.0: adding it times a tap changes no sum, not even a zero's sign
template <>
__device__ __forceinline__ float2 outside_value<float2>() { return make_float2(-0.0f, -0.0f); }
template <>
__device__ __forceinline__ float outside_value<float>() { return -0.0f; }

// An element of a plane in global memory, or (LDG false) in shared memory
template <bool LDG>
__device__ __forceinline__ float plane_load(const float* p) {
    return LDG ? __ldg(p) : *p;
}

// ---- separable pass elements ---------------------------------------------------------------------

// flow/conv.rs:101-137 on a line held in shared memory: element t of the line (global index, inside
// [0, len)) lives at line[(t - origin) * stride].
template <int N, bool LEFT_FIRST>
__device__ __forceinline__ float border_sm(const float* line, int origin, int stride, int len, int i, const float* k) {
    float centre = line[(i - origin) * stride];
    float num = k[0] * centre;
    float den = k[0];
#pragma unroll
    for (int j = N - 1; j >= 1; j--) {
        float kj = k[j];
#pragma unroll
        for (int side = 0; side < 2; side++) {
            bool right = (side == 0) != LEFT_FIRST;
            int t = right ? i + j : i - j;
            bool inside = t >= 0 && t < len;
            float v = inside ? line[(t - origin) * stride] : -1.0f;
            float mask = (v != -1.0f) ? 1.0f : 0.0f;
            float wv = mask * kj;
            den = den + wv;
            num = num + v * wv;
        }
    }
    return num / den;
}

// One output of a pass along a line (conv.rs:141-190 horizontally, :268-301 vertically): the
// interior chain for elements whose taps all lie inside [n, len - n), the border rule otherwise.
template <int N, bool LEFT_FIRST>
__device__ __forceinline__ float pass_elem(const float* line, int origin, int stride, int len, int i, const float* k) {
    if (len >= 2 * N && i >= N && i < len - N) {
        const float* c = line + (i - origin) * stride;
        float s = c[0] * k[0];
#pragma unroll
        for (int j = N - 1; j >= 1; j--) s = s + (c[j * stride] + c[-j * stride]) * k[j];
        return s;
    }
    return border_sm<N, LEFT_FIRST>(line, origin, stride, len, i, k);
}

// The weight sum of the border rule at line index i (conv.rs:101-137) when no sample is the sentinel:
// it depends on the position alone; with its reciprocal. 1 for the interior outputs, which are not
// divided.
template <int N>
__device__ __forceinline__ float2 border_den(int i, int len, const float* k) {
    if (i >= N && i < len - N) return make_float2(1.0f, 1.0f);
    float den = k[0];
#pragma unroll
    for (int j = N - 1; j >= 1; j--) {
        if (i + j >= 0 && i + j < len) den = den + k[j];
        if (i - j >= 0 && i - j < len) den = den + k[j];
    }
    return make_float2(den, __frcp_rn(den));
}

// new_disp (flow.rs:361-371) at R pixels: b the blurred B, t the blurred tensor and its determinant, f the flow,
// updated. Both components divide by the determinant: y = 1 / t once, correctly rounded, and Markstein's
// corrections in pairs (vquot; a zero takes its sign from a y), which hold for operands within 2^60 of 1 (t
// is above 40); others divide.
template <int R>
__device__ __forceinline__ void new_disp_run(const float2* b, const float4* t, float2* f) {
    float2 a[R], q[R];
    bool on[R], plain[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
        on[r] = fabsf(t[r].w) > 40.0f;
        a[r] = make_float2(t[r].y * b[r].y - t[r].z * b[r].x, t[r].y * b[r].x - t[r].x * b[r].y);
        const float d = on[r] ? t[r].w : 64.0f, y = __frcp_rn(d);
        const float lo = 8.67e-19f, hi = 1.15e18f;  // 2^-60, 2^60
        plain[r] = on[r] && !(fabsf(d) < hi && (a[r].x == 0.0f || (fabsf(a[r].x) > lo && fabsf(a[r].x) < hi)) &&
                              (a[r].y == 0.0f || (fabsf(a[r].y) > lo && fabsf(a[r].y) < hi)));
        const float2 n = make_float2(-d, -d), yy = make_float2(y, y);
        const float2 q0 = __ffma2_rn(a[r], yy, make_float2(-0.0f, -0.0f));
        float2 v = __ffma2_rn(__ffma2_rn(q0, n, a[r]), yy, q0);
        v = __ffma2_rn(__ffma2_rn(v, n, a[r]), yy, v);
        q[r] = make_float2(a[r].x == 0.0f ? q0.x : v.x, a[r].y == 0.0f ? q0.y : v.y);
    }
#pragma unroll
    for (int r = 0; r < R; r++) {
        if (plain[r]) q[r] = make_float2(a[r].x / t[r].w, a[r].y / t[r].w);
        if (on[r]) f[r] = make_float2(q[r].x + f[r].x, q[r].y + f[r].y);
    }
}

// One element by the general rule, per channel, out of the main path: the multi channel rule drops
// real samples of exactly -1.0, which run_pass sends here. line: line index `origin` at line[0].
template <int N, bool LEFT_FIRST>
__device__ __noinline__ float slow_elem(const float* line, int origin, int stride, int len, int i, const float* k) {
    return pass_elem<N, LEFT_FIRST>(line, origin, stride, len, i, k);
}
template <int N, bool LEFT_FIRST>
__device__ __forceinline__ float slow_pass(const float* line, int origin, int stride, int len, int i, const float* k) {
    return slow_elem<N, LEFT_FIRST>(line, origin, stride, len, i, k);
}
template <int N, bool LEFT_FIRST>
__device__ __forceinline__ float2 slow_pass(const float2* line, int origin, int stride, int len, int i, const float* k) {
    const float* f = reinterpret_cast<const float*>(line);
    return make_float2(slow_elem<N, LEFT_FIRST>(f, origin, 2 * stride, len, i, k),
                       slow_elem<N, LEFT_FIRST>(f + 1, origin, 2 * stride, len, i, k));
}

// R consecutive outputs of a multi channel pass (conv.rs:141-190 / :268-301) at line indices i0 ..
// i0 + R - 1, from the R + 2N - 2 samples base[0], base[stride], ... (line indices i0 - (N - 1) on),
// each read once. Samples outside the line hold outside_value, so a border output is the plain chain
// of its taps, one side after the other, over the position's weight sum (den[r], border_den of output
// r): no per tap tests. Returns true, with res undefined, for the rare run near the line's ends that
// needs the general rule: a window that holds the sentinel -1.0, or a sum that vquot does not divide; the
// caller then runs slow_run. Outputs outside the line come out as garbage that nobody reads.
template <int N, int R, bool LEFT_FIRST, bool SPLIT, class V>
__device__ __forceinline__ bool run_pass(const V* base, int stride, int i0, int len, const Taps& t, const float2* den,
                                         V* res) {
    constexpr int NV = R + 2 * N - 2;
    V v[NV];
#pragma unroll
    for (int j = 0; j < NV; j++) v[j] = base[j * stride];
    if (i0 >= N && i0 + R - 1 < len - N) {
#pragma unroll
        for (int r = 0; r < R; r++) {
            V s = vmul(v[r + N - 1], t.k[0], t.z);
#pragma unroll
            for (int j = N - 1; j >= 1; j--) s = vmadd(s, vadd(v[r + N - 1 + j], v[r + N - 1 - j]), t.k[j], t.z);
            res[r] = s;
        }
        return false;
    }
    // a run that touches the line's ends: both rules for every output and a select, so that the R chains
    // stay independent (an interior output's weight sum is 1, and a value over 1 is the value). SPLIT: the
    // border rule first, then the interior one in a run that has both. One block whose runs are mostly at a
    // line's ends is faster so; the tiles of a level, which have few such runs, are 13 % slower.
    Magnitudes seen;
    float near4[4] = {1.0f, 1.0f, 1.0f, 1.0f};  // (SPLIT: four chains of minima)
#pragma unroll
    for (int j = 0; j < NV; j++) near4[SPLIT ? j % 4 : 0] = from_sentinel(v[j], near4[SPLIT ? j % 4 : 0]);
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int i = i0 + r;
        V s = vmul(v[r + N - 1], t.k[0], t.z), e = s;
#pragma unroll
        for (int j = N - 1; j >= 1; j--) {
            if (!SPLIT) s = vmadd(s, vadd(v[r + N - 1 + j], v[r + N - 1 - j]), t.k[j], t.z);
            e = vmadd(e, LEFT_FIRST ? v[r + N - 1 - j] : v[r + N - 1 + j], t.k[j], t.z);
            e = vmadd(e, LEFT_FIRST ? v[r + N - 1 + j] : v[r + N - 1 - j], t.k[j], t.z);
        }
        const bool inner = i >= N && i < len - N;
        const V q = vquot(e, den[r], seen);
        res[r] = !SPLIT && inner ? s : q;
    }
    if (SPLIT && i0 + R - 1 >= N && i0 < len - N) {
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int i = i0 + r;
            V s = vmul(v[r + N - 1], t.k[0], t.z);
#pragma unroll
            for (int j = N - 1; j >= 1; j--) s = vmadd(s, vadd(v[r + N - 1 + j], v[r + N - 1 - j]), t.k[j], t.z);
            res[r] = i >= N && i < len - N ? s : res[r];
        }
    }
    const float nearest = fminf(fminf(near4[0], near4[1]), fminf(near4[2], near4[3]));
    return nearest == 0.0f || !seen.safe();
}

// The same outputs by the general rule, one element after the other.
template <int N, int R, bool LEFT_FIRST, class V>
__device__ __forceinline__ void slow_run(const V* base, int stride, int i0, int len, const Taps& t, V* res) {
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int i = i0 + r;
        res[r] = outside_value<V>();
        if (i >= 0 && i < len) res[r] = slow_pass<N, LEFT_FIRST>(base, i0 - (N - 1), stride, len, i, t.k);
    }
}

// run_pass, or with SLOW slow_run, for a pass along the rows or the columns (`above_first`: the tap above
// first).
template <bool SLOW, int N, int R, bool SPLIT = false, class V>
__device__ __forceinline__ bool h_pass(const V* base, int i0, int len, const Taps& t, const float2* den, V* res) {
    if (!SLOW) return run_pass<N, R, false, SPLIT>(base, 1, i0, len, t, den, res);
    slow_run<N, R, false>(base, 1, i0, len, t, res);
    return false;
}
template <bool SLOW, int N, int R, bool SPLIT = false, class V>
__device__ __forceinline__ bool v_pass(const V* base, int stride, int i0, int len, const Taps& t, const float2* den,
                                       bool above_first, V* res) {
    if (!SLOW)
        return above_first ? run_pass<N, R, true, SPLIT>(base, stride, i0, len, t, den, res)
                           : run_pass<N, R, false, SPLIT>(base, stride, i0, len, t, den, res);
    if (above_first) slow_run<N, R, true>(base, stride, i0, len, t, res);
    else slow_run<N, R, false>(base, stride, i0, len, t, res);
    return false;
}

// The single channel border rule by the division, for a run of sums that vquot does not divide.
template <int R>
__device__ __noinline__ void single_slow(float2* e, const float2* den, int i0, int len, int n) {
#pragma unroll 1
    for (int r = 0; r < R; r++)
        if (i0 + r < n || i0 + r >= len - n) e[r] = make_float2(e[r].x / den[r].x, e[r].y / den[r].x);
}

// R outputs of the single channel rule (conv.rs:101-137, :141-190) of a pair of lines, from their R + 2N - 2
// samples v (line indices i0 - (N - 1) on; samples outside the line are 0, which its taps add). The outputs near
// the line's ends are divided by the weights inside it (den: border_den of each output).
template <int N, int R, bool LEFT_FIRST>
__device__ __forceinline__ void single_run(const float2* v, int i0, int len, const Taps& t, const float2* den, float2* res) {
    if (i0 >= N && i0 + R - 1 < len - N) {
#pragma unroll
        for (int r = 0; r < R; r++) {
            float2 s = vmul(v[r + N - 1], t.k[0], t.z);
#pragma unroll
            for (int j = N - 1; j >= 1; j--) s = vmadd(s, vadd(v[r + N - 1 + j], v[r + N - 1 - j]), t.k[j], t.z);
            res[r] = s;
        }
        return;
    }
    Magnitudes seen;
    float2 sums[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int i = i0 + r;
        const bool inner = i >= N && i < len - N;
        const float2 c = vmul(v[r + N - 1], t.k[0], t.z);
        float2 s = c, e = c;
#pragma unroll
        for (int j = N - 1; j >= 1; j--) {
            s = vmadd(s, vadd(v[r + N - 1 + j], v[r + N - 1 - j]), t.k[j], t.z);
            e = vmadd(e, LEFT_FIRST ? v[r + N - 1 - j] : v[r + N - 1 + j], t.k[j], t.z);
            e = vmadd(e, LEFT_FIRST ? v[r + N - 1 + j] : v[r + N - 1 - j], t.k[j], t.z);
        }
        sums[r] = inner ? s : e;
        const float2 q = vquot(e, den[r], seen);
        res[r] = inner ? s : q;
    }
    if (!seen.safe()) {
        single_slow<R>(sums, den, i0, len, N);
#pragma unroll
        for (int r = 0; r < R; r++) res[r] = sums[r];
    }
}

__device__ __forceinline__ bool same_bits(float2 a, float2 b) {
    return __float_as_int(a.x) == __float_as_int(b.x) && __float_as_int(a.y) == __float_as_int(b.y);
}

// One coordinate of a target for Block::cost (flow.rs:474-500) in a level of n >= 4 pixels along it: the
// cost exists for targets in [1, n - 2]; the cell is the target's whole part, but at n - 2 the cell
// before it (with the fraction 1). Any other target is moved into the range and reported as no good.
__device__ __forceinline__ void bm_cell(float t, float top, int last, bool& ok, int& i, float& f) {
    const float c = fminf(fmaxf(t, 1.0f), top);
    ok = ok && c == t;
    i = min(__float2int_rz(c), last);
    f = c - (float)i;
}

// The costs (flow.rs:474-523) of two vectors at one position as the two lanes of packed arithmetic: lane .x
// and lane .y their cells' first elements (at0, at1) and fractions; p: the 3 x 3 patch of A there, row by row. B is
// row major (element (x, y) at [y * w + x]), or with COLS the transpose ([x * h + y]), so that the patches along a
// line are contiguous.
// The products carry negated weights, so that their sum adds to the patch value; the squares are the same
// bits. z: -0.0 (see the packed pairs above).
template <bool COLS, bool LDG = true>
__device__ __forceinline__ float2 bm_cost2(const float* __restrict__ B, int pitch, const float p[9], float2 fx, float2 fy,
                                           int at0, int at1, float z) {
    float2 T[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++)
            T[COLS ? j : i][COLS ? i : j] = make_float2(plane_load<LDG>(B + at0 + i * pitch + j), plane_load<LDG>(B + at1 + i * pitch + j));
    const float2 zz = make_float2(z, z);
    const float2 nx = make_float2(-fx.x, -fx.y), ny = make_float2(-fy.x, -fy.y);
    const float2 w11 = __ffma2_rn(fy, fx, zz), n11 = __ffma2_rn(fy, nx, zz);
    const float2 n10 = __fadd2_rn(w11, nx), n01 = __fadd2_rn(w11, ny);
    const float2 n00 = __fadd2_rn(__fadd2_rn(__fadd2_rn(fx, make_float2(-1.0f, -1.0f)), fy), n11);
    float2 s = zz;
#pragma unroll
    for (int b = 0; b < 3; b++) {
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const int k = b * 3 + a;
#ifdef TW_FAST_VARIANT
            const float2 d = __ffma2_rn(n11, T[b + 1][a + 1], __ffma2_rn(n01, T[b + 1][a], __ffma2_rn(n10, T[b][a + 1],
                             __ffma2_rn(n00, T[b][a], make_float2(p[k], p[k])))));
            s = __ffma2_rn(d, d, s);
#else
            float2 q = __fadd2_rn(__ffma2_rn(n00, T[b][a], zz), __ffma2_rn(n10, T[b][a + 1], zz));
            q = __fadd2_rn(q, __ffma2_rn(n01, T[b + 1][a], zz));
            q = __fadd2_rn(q, __ffma2_rn(n11, T[b + 1][a + 1], zz));
            const float2 d = __fadd2_rn(make_float2(p[k], p[k]), q);
            const float2 sq = __ffma2_rn(d, d, zz);
            s = k == 0 ? sq : k < 8 ? __fadd2_rn(s, sq) : __fadd2_rn(sq, s);
#endif
        }
    }
    return s;
}

// The cost of one vector there, the same bits as a lane of bm_cost2 (in the fast mode too, where the compiler would
// contract the plain sums its own way: a run's test compares the one with the other).
template <bool COLS, bool LDG = true>
__device__ __forceinline__ float bm_cost1(const float* __restrict__ B, int pitch, const float p[9], float fx, float fy, int at) {
    float T[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) T[COLS ? j : i][COLS ? i : j] = plane_load<LDG>(B + at + i * pitch + j);
#ifdef TW_FAST_VARIANT
    const float w11 = __fmul_rn(fy, fx), n10 = __fsub_rn(w11, fx), n01 = __fsub_rn(w11, fy);
    const float n00 = __fsub_rn(__fadd_rn(__fsub_rn(fx, 1.0f), fy), w11);
    float s = -0.0f;
#pragma unroll
    for (int b = 0; b < 3; b++)
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const float d = __fmaf_rn(-w11, T[b + 1][a + 1], __fmaf_rn(n01, T[b + 1][a], __fmaf_rn(n10, T[b][a + 1],
                            __fmaf_rn(n00, T[b][a], p[b * 3 + a]))));
            s = __fmaf_rn(d, d, s);
        }
    return s;
#else
    const float w11 = fy * fx, w10 = fx - w11, w01 = fy - w11, w00 = ((1.0f - fx) - fy) + w11;
    float sq[9];
#pragma unroll
    for (int b = 0; b < 3; b++)
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const float q = ((w00 * T[b][a] + w10 * T[b][a + 1]) + w01 * T[b + 1][a]) + w11 * T[b + 1][a + 1];
            const float d = p[b * 3 + a] - q;
            sq[b * 3 + a] = d * d;
        }
    float s = sq[0] + sq[1];
#pragma unroll
    for (int k = 2; k < 8; k++) s = s + sq[k];
    return sq[8] + s;
#endif
}

// sample.rs:31-41 for a coordinate known to lie in [0, len - 1] (or a NaN): the conversion needs no range
// test and the cell no lower clamp (a NaN gives cell 0 and a NaN fraction, as the general rule does)
__device__ __forceinline__ void cell_inside(float x, int len, int& io, float& fo) {
    int i = __float2int_rz(x);
    float f = x - (float)i;
    if (i >= len - 1) { i = len - 2; f = 1.0f; }
    io = i;
    fo = f;
}

// flow.rs:334-357 (calc_b) at R pixels (x, y + r) whose flow is f[r]: B = (I0(x - u, y - v) - I1) * grad,
// zero where the source point leaves the level, and in a layered solve (mask_y) where the warped mask of
// Y is below 0.999 (flow.rs:777-845). i1, g: I1 and the gradient at the pixels. Levels are at least 2 x
// 2. The gathers of all R pixels are in flight together (a point outside reads pixel 0).
template <int R, bool LDG = true>
__device__ __forceinline__ void calc_b_run(const float* i0, const float* __restrict__ mask_y, int w, int h, int x,
                                           int y, const float2* f, const float* i1, const float2* g, float2* b) {
    bool in[R];
    int at[R];
    float fx[R], fy[R], p[R][4];
#pragma unroll
    for (int r = 0; r < R; r++) {
        const float sx = (float)x - f[r].x, sy = (float)(y + r) - f[r].y;
        in[r] = !(sx < 0.0f || (float)w - 1.0f < sx || sy < 0.0f || (float)h - 1.0f < sy);
        if (in[r] && mask_y) in[r] = bilinear1(mask_y, w, h, sx, sy) >= 0.999f;
        int ix, iy;
        cell_inside(sx, w, ix, fx[r]);
        cell_inside(sy, h, iy, fy[r]);
        at[r] = in[r] ? iy * w + ix : 0;
    }
#pragma unroll
    for (int r = 0; r < R; r++) {
        const float* q = i0 + at[r];
        p[r][0] = plane_load<LDG>(q);
        p[r][1] = plane_load<LDG>(q + 1);
        p[r][2] = plane_load<LDG>(q + w);
        p[r][3] = plane_load<LDG>(q + w + 1);
    }
#pragma unroll
    for (int r = 0; r < R; r++) {
        const float top = (p[r][1] - p[r][0]) * fx[r] + p[r][0];
        const float bot = (p[r][3] - p[r][2]) * fx[r] + p[r][2];
        const float rr = ((bot - top) * fy[r] + top) - i1[r];
        b[r] = in[r] ? make_float2(rr * g[r].x, rr * g[r].y) : make_float2(0.0f, 0.0f);
    }
}

// The gradient of img at (x, y) (flow.rs:283-316): the mean of the one sided differences that exist (a
// half is exact, so the reference's division by 2 is a product), zero in a layered solve where the
// level mask of X is below 0.95 at the pixel or at one of its four neighbours that exist
// (flow.rs:743-761).
template <bool LDG = true>
__device__ __forceinline__ float2 gradient_at(const float* img, const float* __restrict__ mask, int w, int h, int x, int y) {
    const int i = y * w + x;
    const float cc = plane_load<LDG>(img + i);
    float nx = 0.0f, ny = 0.0f;
    if (x >= 1) nx = (cc - plane_load<LDG>(img + i - 1)) + 0.0f;
    if (y >= 1) ny = (cc - plane_load<LDG>(img + i - w)) + 0.0f;
    if (x + 1 <= w - 1) nx = nx + (plane_load<LDG>(img + i + 1) - cc);
    if (y + 1 <= h - 1) ny = ny + (plane_load<LDG>(img + i + w) - cc);
    float2 g = make_float2(x >= 1 && x + 1 <= w - 1 ? nx * 0.5f : nx, y >= 1 && y + 1 <= h - 1 ? ny * 0.5f : ny);
    if (mask) {
        auto off = [&](int j) { return __ldg(mask + j) < 0.95f; };
        if (off(i) || (y >= 1 && off(i - w)) || (y + 1 < h && off(i + w)) || (x >= 1 && off(i - 1)) ||
            (x + 1 < w && off(i + 1)))
            g = make_float2(0.0f, 0.0f);
    }
    return g;
}

// any[k] (k = level) is set when some pixel of level k is in range after its refinement.
// check at level l = no level processed before (start .. l+1) had a pixel in range.
__device__ __forceinline__ bool zero_at_level(const int* any, int l, int start) {
    bool check = true;
    for (int k = start; k > l; k--) check = check && any[k] == 0;
    return check && any[l] == 0;
}

// The range check at pixel (x, y) with flow f (flow.rs:430-442, all_flow_out_of_range, as "some pixel is in
// range"), where a level's last kernel writes the flow: nearly every pixel is in range, so the flag is set within
// the first ones and read by the others.
__device__ __forceinline__ void check_range(int* any, int x, int y, float2 f, int w, int h) {
    const float px = (float)x + f.x, py = (float)y + f.y;
    const bool in = 0.0f <= px && px <= (float)(w - 1) && 0.0f <= py && py <= (float)(h - 1);
    if (in && *(volatile int*)any == 0) atomicOr(any, 1);
}

// flow.rs:376-391 (upsample_flow, bilinear2 of sample.rs:69-86) from a field of sw x sh to one of dw x
// dh: the scales sx, sy and their reciprocals, formed once on the host (the same IEEE operations).
__host__ __device__ inline UpsampleScale upsample_scale(int sw, int sh, int dw, int dh) {
    UpsampleScale u;
    u.sx = ((float)dw - 1.0f) / (float)(sw - 1);
    u.sy = ((float)dh - 1.0f) / (float)(sh - 1);
    u.rx = (float)(1.0 / (double)u.sx);
    u.ry = (float)(1.0 / (double)u.sy);
    return u;
}

// The upsampled flow at output pixel (x, y), with the reset (zero) and the damping of the coarse
// field's level applied to the four gathered samples, which is the same as applying them to the whole
// field first.
__device__ __forceinline__ float2 upsample_at(const float2* src, int sw, int sh, const UpsampleScale& c, bool zero,
                                              bool damp_now, float damp, int x, int y) {
    int ix, iy;
    float fx, fy;
    cell((float)x * c.rx, sw, ix, fx);
    cell((float)y * c.ry, sh, iy, fy);
    const int i = iy * sw + ix;
    float2 q[4] = {src[i], src[i + 1], src[i + sw], src[i + sw + 1]};
#pragma unroll
    for (int m = 0; m < 4; m++) {
        if (zero) q[m] = make_float2(0.0f, 0.0f);
        if (damp_now) q[m] = make_float2(damp * q[m].x, damp * q[m].y);
    }
    float2 r;
    {
        float top = (q[1].x - q[0].x) * fx + q[0].x;
        float bot = (q[3].x - q[2].x) * fx + q[2].x;
        r.x = ((bot - top) * fy + top) * c.sx;
    }
    {
        float top = (q[1].y - q[0].y) * fx + q[0].y;
        float bot = (q[3].y - q[2].y) * fx + q[2].y;
        r.y = ((bot - top) * fy + top) * c.sy;
    }
    return r;
}

}  // namespace tw
