// The persistent coarse-level solve: one CTA walks every coarse level of a solve (flow.rs:1258-1307)
// in a single launch.
//
// The coarse levels of a pyramid are tiny (15 x 8 to 60 x 33 at 1080p) and, launched kernel by
// kernel, they cost about seven launches each whose time is all latency. Here one block keeps every
// solver plane of a level in shared memory (the bands it reads stay in L1) and runs, level after
// level with block barriers between the stages: the gradient and the blurred tensor, the three
// iterations (calc_b, blur7, new_disp, blur5), the four block matching sweeps, the range check and
// the upsample (with the reset and the damping of the level) into the next level; the last one
// writes the flow of the first level the tiled kernels take over. Every element follows the same
// rules as those kernels (level.cuh), so the flow is bit identical. No block waits on another.
//
// The separable passes run on two planes padded with what lies outside the image (run_pass of
// level.cuh), both components of a pixel in one packed operation; the vertical ones end in registers
// (new_disp; the new flow and the next iteration's B).
//
// Block matching: the own cost and S[q] = accept(q, v[q-1]) (the test when q-1 kept its own vector) of
// every position of the level at once, a thread each; then the sweep's recurrence
// v'[q] = accept(q, v'[q-1]) ? v'[q-1] : v[q] is walked run by run, a group of 8 lanes per line: a stretch of
// positions that start their own runs is skipped with ballots over S, and a run that goes on tests its
// vector at the next 8 positions at once (one lane each), the first refusal ending it (most runs end
// within a few positions).
#include "kernels.cuh"
#include "level.cuh"

namespace tw {
TW_VARIANT_BEGIN

namespace {

constexpr int NT = COARSE_THREADS;
constexpr int GL = 8;        // lanes per line of block matching
constexpr int NG = NT / GL;  // lines in flight
constexpr int PAD = 7;       // what the longest filter reads past a line
constexpr int RUN = 2;       // outputs per thread of a pass
// the largest padded plane of a level of at most COARSE_MAX_PIXELS (16 x 128)
constexpr int PLANE = 4800;

// A level in shared memory
struct Coarse {
    float2 *p1, *p2;  // the padded planes: pixel (x, y) at [(y + PAD) * stride + x + PAD]
    float4* tensor;
    float2* grad;
    float2* f;
    float* cost;
    unsigned char* takes;
    float2 *den7x, *den7y, *den5x, *den5y;
    int w, h, stride;
    __device__ __forceinline__ int at(int x, int y) const { return (y + PAD) * stride + x + PAD; }
};

// The pass along the rows, p1 -> p2
template <int N>
__device__ __forceinline__ void rows_pass(const Coarse& C, const Taps& t, const float2* den) {
    const int segs = (C.w + RUN - 1) / RUN;
    for (int e = threadIdx.x; e < C.h * segs; e += NT) {
        const int seg = e / C.h, y = e - seg * C.h, x = seg * RUN;
        float2 o[RUN];
        const float2* in = C.p1 + C.at(x, y) - (N - 1);
        if (h_pass<false, N, RUN>(in, x, C.w, t, den + x, o)) h_pass<true, N, RUN>(in, x, C.w, t, den + x, o);
#pragma unroll
        for (int r = 0; r < RUN; r++)
            if (x + r < C.w) C.p2[C.at(x + r, y)] = o[r];
    }
    __syncthreads();
}

// The pass along the columns of p2, its outputs handed to put(x, y, value)
template <int N, class Put>
__device__ __forceinline__ void columns_pass(const Coarse& C, const Taps& t, const float2* den, bool af, Put put) {
    const int segs = (C.h + RUN - 1) / RUN;
    for (int e = threadIdx.x; e < C.w * segs; e += NT) {
        const int seg = e / C.w, x = e - seg * C.w, y = seg * RUN;
        float2 o[RUN];
        const float2* in = C.p2 + C.at(x, y) - (N - 1) * C.stride;
        if (v_pass<false, N, RUN>(in, C.stride, y, C.h, t, den + y, af, o)) v_pass<true, N, RUN>(in, C.stride, y, C.h, t, den + y, af, o);
#pragma unroll
        for (int r = 0; r < RUN; r++)
            if (y + r < C.h) put(x, y + r, o[r]);
    }
    __syncthreads();
}

// The targets and the patch of a block cost at pixel (x, y) (row major bands)
__device__ __forceinline__ void patch_at(const float* __restrict__ A, int w, int x, int y, float p[9]) {
    const float* a = A + (y - 1) * w + (x - 1);
#pragma unroll
    for (int r = 0; r < 3; r++)
#pragma unroll
        for (int c = 0; c < 3; c++) p[r * 3 + c] = __ldg(a + r * w + c);
}

// Block::step's test at pixel (x, y) for the vector n against c0, the cost of the pixel's own vector (NaN
// when no step can happen there).
__device__ __forceinline__ bool accept_at(const float* __restrict__ A, const float* __restrict__ B, int w, int h, int x, int y,
                                          float2 n, float c0) {
    float p[9];
    patch_at(A, w, x, y, p);
    bool ok = true;
    int ix, iy;
    float fx, fy;
    bm_cell((float)x - n.x, (float)(w - 2), w - 3, ok, ix, fx);
    bm_cell((float)y - n.y, (float)(h - 2), h - 3, ok, iy, fy);
    const float c1 = bm_cost1<false>(B, w, p, fx, fy, (iy - 1) * w + ix - 1);
    return ok && c1 < c0;
}

// One sweep of every row (COLS false) or column of the level, in place on the flow; reverse: from the far
// end.
template <bool COLS>
__device__ __forceinline__ void sweep(const Coarse& C, const float* __restrict__ A, const float* __restrict__ B, bool reverse,
                                      float z) {
    const int w = C.w, h = C.h, iw = w - 2, step = (COLS ? w : 1) * (reverse ? 1 : -1);
    float2* f = C.f;
    // the own cost of every interior position, and S
    for (int k = threadIdx.x; k < iw * (h - 2); k += NT) {
        const int y = 1 + k / iw, x = 1 + k - (y - 1) * iw, e = y * w + x;
        float p[9];
        patch_at(A, w, x, y, p);
        const float2 v = f[e], n = f[e + step];
        bool ok0 = true, ok1 = true;
        int ix0, iy0, ix1, iy1;
        float2 fx, fy;
        bm_cell((float)x - v.x, (float)(w - 2), w - 3, ok0, ix0, fx.x);
        bm_cell((float)y - v.y, (float)(h - 2), h - 3, ok0, iy0, fy.x);
        bm_cell((float)x - n.x, (float)(w - 2), w - 3, ok1, ix1, fx.y);
        bm_cell((float)y - n.y, (float)(h - 2), h - 3, ok1, iy1, fy.y);
        const float2 c = bm_cost2<false>(B, w, p, fx, fy, (iy0 - 1) * w + ix0 - 1, (iy1 - 1) * w + ix1 - 1, z);
        const float ci = ok0 ? c.x : __int_as_float(0x7fc00000);
        C.cost[e] = ci;
        C.takes[e] = ok1 && c.y < ci;
    }
    __syncthreads();
    // the recurrence, a group of lanes per line
    const int grp = threadIdx.x / GL, gl = threadIdx.x % GL, gshift = (threadIdx.x & 31) & ~(GL - 1);
    const unsigned gmask = ((1u << GL) - 1u) << gshift;
    const int len = COLS ? h : w, lines = (COLS ? w : h) - 2;
    auto group_ballot = [&](bool p) { return (__ballot_sync(gmask, p) >> gshift) & ((1u << GL) - 1u); };
    for (int line = 1 + grp; line <= lines; line += NG) {
        auto elem = [&](int q) {  // the element at sweep position q
            const int i = reverse ? len - 1 - q : q;
            return COLS ? i * w + line : line * w + i;
        };
        float2 cur = make_float2(0.0f, 0.0f);  // the vector of the run in progress (uniform over the group)
        bool own = true;                       // position q - 1 kept its own vector
        int q = 1;
        while (q <= len - 2) {
            const int qq = q + gl;
            const bool valid = qq <= len - 2;
            if (own) {
                // the first position >= q that takes the vector before it: the others start runs
                const unsigned m = group_ballot(valid && C.takes[elem(valid ? qq : q)]);
                if (!m) {
                    q += GL;
                    continue;
                }
                const int r = q + __ffs(m) - 1;
                cur = f[elem(r - 1)];
                __syncwarp(gmask);
                if (gl == 0) f[elem(r)] = cur;
                q = r + 1;
                own = false;
            } else {
                // the run goes on while the next positions accept its vector
                bool acc = false;
                if (valid) {
                    const int i = reverse ? len - 1 - qq : qq;
                    acc = accept_at(A, B, w, h, COLS ? line : i, COLS ? i : line, cur, C.cost[elem(qq)]);
                }
                const unsigned va = group_ballot(valid), fails = va & ~group_ballot(acc);
                const int n = fails ? __ffs(fails) - 1 : __popc(va);
                if (valid && gl < n) f[elem(qq)] = cur;
                q += n;
                if (fails) {  // position q starts its own run
                    q++;
                    own = true;
                }
            }
            __syncwarp(gmask);
        }
    }
    __syncthreads();
}

}  // namespace

__global__ void __launch_bounds__(COARSE_THREADS) k_solve_coarse(const __grid_constant__ CoarseJob J) {
    extern __shared__ __align__(16) float4 coarse_sm[];
    constexpr int M = COARSE_MAX_PIXELS;
    Coarse C;
    C.tensor = coarse_sm;
    C.p1 = (float2*)(C.tensor + M);
    C.p2 = C.p1 + PLANE;
    C.grad = C.p2 + PLANE;
    C.f = C.grad + M;
    float2* fn = C.f + M;
    C.den7x = fn + M;
    C.den7y = C.den7x + COARSE_MAX_LINE;
    C.den5x = C.den7y + COARSE_MAX_LINE;
    C.den5y = C.den5x + COARSE_MAX_LINE;
    C.cost = (float*)(C.den5y + COARSE_MAX_LINE);
    C.takes = (unsigned char*)(C.cost + M);
    __shared__ int s_any[32];
    const int tid = threadIdx.x;
    const bool af = J.af;
    if (tid < 32) s_any[tid] = 0;
    for (int l = J.start; l >= J.last; l--) {
        const int w = J.sizes[l][0], h = J.sizes[l][1], n = w * h;
        const float fw = (float)w, fh = (float)h;
        C.w = w;
        C.h = h;
        C.stride = (w + 2 * PAD + RUN) | 1;
        const float* __restrict__ A = J.x + J.offs[l];
        const float* __restrict__ B = J.y + J.offs[l];
        const float* mask_x = J.mx ? J.mx + J.offs[l] : nullptr;
        const float* mask_y = J.my ? J.my + J.offs[l] : nullptr;
        auto user = [&]() {  // the user displacement of the tracking points (flow/extras.rs:198-215)
            if (!J.uww) return;
            for (int i = tid; i < n; i += NT) {
                const float k = __ldg(J.uww + J.offs[l] + i);
                if (k != 0.0f) C.f[i] = make_float2(__ldg(J.udu + J.offs[l] + i) / k, __ldg(J.udv + J.offs[l] + i) / k);
            }
            __syncthreads();
        };
        if (l == J.start)
            for (int i = tid; i < n; i += NT) C.f[i] = make_float2(0.0f, 0.0f);
        for (int i = tid; i < (h + 2 * PAD) * C.stride; i += NT) C.p1[i] = C.p2[i] = outside_value<float2>();
        for (int i = tid; i < w; i += NT) {
            C.den7x[i] = border_den<8>(i, w, J.g7.k);
            C.den5x[i] = border_den<6>(i, w, J.g5.k);
        }
        for (int i = tid; i < h; i += NT) {
            C.den7y[i] = border_den<8>(i, h, J.g7.k);
            C.den5y[i] = border_den<6>(i, h, J.g5.k);
        }
        __syncthreads();
        user();
        // the gradient and the tensor (flow.rs:283-328), its blur7 in two turns: the first two channels, then
        // the third, with the determinant of new_disp and calc_b of the first iteration
        for (int i = tid; i < n; i += NT) {
            const int y = i / w, x = i - y * w;
            const float2 g = gradient_at(A, mask_x, w, h, x, y);
            C.grad[i] = g;
            C.p1[C.at(x, y)] = make_float2(g.x * g.x, g.x * g.y);
        }
        __syncthreads();
        rows_pass<8>(C, J.g7, C.den7x);
        columns_pass<8>(C, J.g7, C.den7y, af, [&](int x, int y, float2 v) {
            const int i = y * w + x;
            C.tensor[i] = make_float4(v.x, v.y, 0.0f, 0.0f);
            const float2 g = C.grad[i];
            C.p1[C.at(x, y)] = make_float2(g.y * g.y, 0.0f);
        });
        rows_pass<8>(C, J.g7, C.den7x);
        auto b_of = [&](int x, int y, float2 f) {
            const int i = y * w + x;
            const float i1 = __ldg(A + i);
            const float2 g = C.grad[i];
            float2 b;
            calc_b_run<1>(B, mask_y, w, h, x, y, &f, &i1, &g, &b);
            return b;
        };
        columns_pass<8>(C, J.g7, C.den7y, af, [&](int x, int y, float2 v) {
            const int i = y * w + x;
            const float4 t = C.tensor[i];
            C.tensor[i] = make_float4(t.x, t.y, v.x, t.y * t.y - v.x * t.x);
            C.p1[C.at(x, y)] = b_of(x, y, C.f[i]);
        });
        for (int it = 0; it < 3; it++) {
            rows_pass<8>(C, J.g7, C.den7x);
            columns_pass<8>(C, J.g7, C.den7y, af, [&](int x, int y, float2 b) {  // new_disp (flow.rs:361-371)
                const float4 t = C.tensor[y * w + x];
                float2 f = C.f[y * w + x];
                if (fabsf(t.w) > 40.0f) {
                    f.x = (t.y * b.y - t.z * b.x) / t.w + f.x;
                    f.y = (t.y * b.x - t.x * b.y) / t.w + f.y;
                }
                C.p1[C.at(x, y)] = f;
            });
            rows_pass<6>(C, J.g5, C.den5x);
            columns_pass<6>(C, J.g5, C.den5y, af, [&](int x, int y, float2 f) {
                C.f[y * w + x] = f;
                if (it < 2) C.p1[C.at(x, y)] = b_of(x, y, f);
            });
        }
        // block matching (flow.rs:551-622): the row sweeps, then the column sweeps; no block has a cost in a
        // level of fewer than 4 x 4 pixels
        if (J.refine && w >= 4 && h >= 4) {
            sweep<false>(C, A, B, false, J.g7.z);
            sweep<false>(C, A, B, true, J.g7.z);
            sweep<true>(C, A, B, false, J.g7.z);
            sweep<true>(C, A, B, true, J.g7.z);
        }
        user();
        // the range check (flow.rs:430-442)
        int in = 0;
        for (int i = tid; i < n; i += NT) {
            int y = i / w, x = i - y * w;
            float px = (float)x + C.f[i].x, py = (float)y + C.f[i].y;
            if (0.0f <= px && px <= fw - 1.0f && 0.0f <= py && py <= fh - 1.0f) in = 1;
        }
        if (__syncthreads_or(in) && tid == 0) {
            s_any[l] = 1;
            J.any[l] = 1;
        }
        __syncthreads();
        // the reset and the damping of the level, then the upsample into the next level
        const int dw = J.sizes[l - 1][0], dh = J.sizes[l - 1][1];
        const bool zero = zero_at_level(s_any, l, J.start);
        const bool damp_now = l == J.start && J.damp_any;
        const UpsampleScale up = upsample_scale(w, h, dw, dh);
        float2* to = l == J.last ? J.f_out : fn;
        for (int i = tid; i < dw * dh; i += NT) {
            int y = i / dw, x = i - y * dw;
            to[i] = upsample_at(C.f, w, h, up, zero, damp_now, J.damp, x, y);
        }
        __syncthreads();
        float2* t = C.f;
        C.f = fn;
        fn = t;
    }
}

size_t coarse_smem_bytes() {
    return (size_t)COARSE_MAX_PIXELS * (sizeof(float4) + 3 * sizeof(float2) + sizeof(float) + 1) +
           (2 * PLANE + 4 * COARSE_MAX_LINE) * sizeof(float2);
}

TW_VARIANT_END
}  // namespace tw
