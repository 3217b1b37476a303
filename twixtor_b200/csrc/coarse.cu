// The persistent coarse-level solve: one CTA walks every coarse level of a solve (flow.rs:1258-1307)
// in a single launch.
//
// The coarse levels of a pyramid are tiny (15 x 8 to 60 x 33 at 1080p) and, launched kernel by
// kernel, they cost about seven launches each whose time is all latency. Here one block keeps every
// plane of a level in shared memory and runs, level after
// level with block barriers between the stages: the gradient and the blurred tensor, the three
// iterations (calc_b, blur7, new_disp, blur5), the four block matching sweeps, the range check and
// the upsample (with the reset and the damping of the level) into the next level; the last one's
// flow is written for the tiled kernels that take over. Every element follows the same
// rules as those kernels (level.cuh), so the flow is bit identical. No block waits on another.
//
// The separable passes run on two planes padded with what lies outside the image (run_pass of
// level.cuh), both components of a pixel in one packed operation; the vertical ones end in registers
// (new_disp; the new flow and the next iteration's B).
//
// Block matching: the own cost and S[q] = accept(q, v[q-1]) (the test when q-1 kept its own vector) of
// every position of the level at once, a thread each; then the sweep's recurrence
// v'[q] = accept(q, v'[q-1]) ? v'[q-1] : v[q] is walked run by run, a group of 4 lanes per segment of a line: a
// stretch of positions that start their own runs is skipped with the bits of S, and a run that goes on
// tests its vector at the next 4 positions at once (one lane each), the first refusal ending it (most runs
// end within a few positions). The segments of a line start together; those that a run of the segment
// before reaches into are walked again until the new vectors meet the old ones.
//
// Bound by the latency of its dependent steps on one SM (the chip's other SMs run other solves). A 1080p
// solve's four levels (7 x 4 to 60 x 33) take 150 us; with passes of scalar elements, own costs evaluated per line
// and bands read through L1 they took 230 us. At 60 x 33 the passes are half of it, block matching the rest.
#include "kernels.cuh"
#include "level.cuh"

namespace tw {
TW_VARIANT_BEGIN

namespace {

constexpr int NT = COARSE_THREADS;
constexpr int GL = 4;        // lanes per segment of a line of block matching
constexpr int NG = NT / GL;  // segments in flight
constexpr int PAD = 7;       // what the longest filter reads past a line
constexpr int RUN = 2;       // outputs per thread of a pass
// e / d for 0 <= e < 4096 and 1 <= d <= COARSE_MAX_LINE, from inverse_of(d)
__device__ __forceinline__ unsigned inverse_of(int d) { return (1u << 20) / (unsigned)d + 1u; }
__device__ __forceinline__ int over_of(int e, unsigned inv) { return (int)((unsigned)e * inv >> 20); }

// A level in shared memory
struct Coarse {
    float2 *p1, *p2;  // the padded planes: pixel (x, y) at [(y + PAD) * stride + x + PAD]
    float *a, *b;     // the bands (block matching's scattered reads cost a bank's turn here, a line's in L1)
    float4* tensor;
    float2* grad;
    float2 *f, *fn;  // the flow and its copy
    float* cost;
    unsigned char* takes;
    float2 *den7x, *den7y, *den5x, *den5y;
    int w, h, stride;
    unsigned winv, hinv, iwinv;  // the reciprocals of w, h and w - 2 (over_of)
    __device__ __forceinline__ int at(int x, int y) const { return (y + PAD) * stride + x + PAD; }
};

// The pass along the rows, p1 -> p2
template <int N>
__device__ __forceinline__ void rows_pass(const Coarse& C, const Taps& t, const float2* den) {
    const int segs = (C.w + RUN - 1) / RUN;
    for (int e = threadIdx.x; e < C.h * segs; e += NT) {
        const int seg = over_of(e, C.hinv), y = e - seg * C.h, x = seg * RUN;
        float2 o[RUN];
        const float2* in = C.p1 + C.at(x, y) - (N - 1);
        if (h_pass<false, N, RUN, true>(in, x, C.w, t, den + x, o)) h_pass<true, N, RUN>(in, x, C.w, t, den + x, o);
#pragma unroll
        for (int r = 0; r < RUN; r++)
            if (x + r < C.w) C.p2[C.at(x + r, y)] = o[r];
    }
    __syncthreads();
}

// The pass along the columns of p2, its outputs handed to put(x, y, n, values): n rows from y on
template <int N, class Put>
__device__ __forceinline__ void columns_pass(const Coarse& C, const Taps& t, const float2* den, bool af, Put put) {
    const int segs = (C.h + RUN - 1) / RUN;
    for (int e = threadIdx.x; e < C.w * segs; e += NT) {
        const int seg = over_of(e, C.winv), x = e - seg * C.w, y = seg * RUN;
        float2 o[RUN];
        const float2* in = C.p2 + C.at(x, y) - (N - 1) * C.stride;
        if (v_pass<false, N, RUN, true>(in, C.stride, y, C.h, t, den + y, af, o))
            v_pass<true, N, RUN>(in, C.stride, y, C.h, t, den + y, af, o);
        put(x, y, min(RUN, C.h - y), o);
    }
    __syncthreads();
}

// The targets and the patch of a block cost at pixel (x, y) (row major bands)
__device__ __forceinline__ void patch_at(const float* A, int w, int x, int y, float p[9]) {
    const float* a = A + (y - 1) * w + (x - 1);
#pragma unroll
    for (int r = 0; r < 3; r++)
#pragma unroll
        for (int c = 0; c < 3; c++) p[r * 3 + c] = a[r * w + c];
}

// Block::step's test at pixel (x, y) for the vector n against c0, the cost of the pixel's own vector (NaN
// when no step can happen there).
__device__ __forceinline__ bool accept_at(const float* A, const float* B, int w, int h, int x, int y,
                                          float2 n, float c0) {
    float p[9];
    patch_at(A, w, x, y, p);
    bool ok = true;
    int ix, iy;
    float fx, fy;
    bm_cell((float)x - n.x, (float)(w - 2), w - 3, ok, ix, fx);
    bm_cell((float)y - n.y, (float)(h - 2), h - 3, ok, iy, fy);
    const float c1 = bm_cost1<false, false>(B, w, p, fx, fy, (iy - 1) * w + ix - 1);
    return ok && c1 < c0;
}

// One sweep of every row (COLS false) or column of the level, from the flow f into fn; reverse: from the
// far end.
template <bool COLS>
__device__ __forceinline__ void sweep(const Coarse& C, bool reverse, float z) {
    const int w = C.w, h = C.h, iw = w - 2, step = (COLS ? w : 1) * (reverse ? 1 : -1);
    const float2* f = C.f;
    const float *A = C.a, *B = C.b;
    // the own cost of every interior position, and S
    for (int k = threadIdx.x; k < iw * (h - 2); k += NT) {
        const int y = 1 + over_of(k, C.iwinv), x = 1 + k - (y - 1) * iw, e = y * w + x;
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
        const float2 c = bm_cost2<false, false>(B, w, p, fx, fy, (iy0 - 1) * w + ix0 - 1, (iy1 - 1) * w + ix1 - 1, z);
        const float ci = ok0 ? c.x : __int_as_float(0x7fc00000);
        C.cost[e] = ci;
        C.takes[e] = ok1 && c.y < ci;
    }
    for (int e = threadIdx.x; e < w * h; e += NT) C.fn[e] = f[e];
    __syncthreads();
    // the recurrence, a group of lanes per segment of a line, as if the position before each segment kept its
    // own vector. The groups of a warp go in step, so that they evaluate their tests together.
    const unsigned FULL = 0xffffffffu;
    const int grp = threadIdx.x / GL, gl = threadIdx.x % GL, gshift = (threadIdx.x & 31) & ~(GL - 1);
    const int len = COLS ? h : w, lines = (COLS ? w : h) - 2;
    int seg = 32;  // positions per segment: as many segments as there are groups for, of 8 positions at least
    while (seg > 8 && lines * ((len - 2 + seg / 2 - 1) / (seg / 2)) <= NG) seg /= 2;
    const int segs = (len - 2 + seg - 1) / seg;
    auto group_ballot = [&](bool p) { return (__ballot_sync(FULL, p) >> gshift) & ((1u << GL) - 1u); };
    auto elem = [&](int line, int q) {  // the element at sweep position q of a line
        const int i = reverse ? len - 1 - q : q;
        return COLS ? i * w + line : line * w + i;
    };
    // how many of the positions q, q + 1, ... < end (at most GL; none with !on) take the vector `cur` carried
    // into q, and whether the next one refused it
    auto taken = [&](bool on, int line, int q, int end, float2 cur, bool& refused) {
        const int qq = q + gl;
        const bool valid = on && qq < end;
        bool acc = false;
        if (valid) {
            const int e = elem(line, qq), y = over_of(e, C.winv);
            acc = accept_at(A, B, w, h, e - y * w, y, cur, C.cost[e]);
        }
        const unsigned va = group_ballot(valid), fails = va & ~group_ballot(acc);
        refused = fails != 0;
        return fails ? __ffs(fails) - 1 : __popc(va);
    };
    for (int job0 = 0; job0 < lines * segs; job0 += NG) {
        const int job = job0 + grp;
        bool live = job < lines * segs;
        const int line = live ? 1 + job / segs : 1, q0 = live ? 1 + (job - (line - 1) * segs) * seg : 1;
        const int q1 = min(q0 + seg, len - 1);
        unsigned takes = 0;  // S of the segment's positions
        for (int j = 0; j < seg / GL; j++) {
            const int q = q0 + j * GL + gl;
            takes |= group_ballot(live && q < q1 && C.takes[elem(line, min(q, len - 2))]) << (j * GL);
        }
        int q = q0;
        bool carry = false;
        float2 cur = make_float2(0.0f, 0.0f);
        // every round passes at least one position of each live segment
        for (int guard = 0; guard <= seg && __any_sync(FULL, live); guard++) {
            if (live && !carry) {
                const unsigned m = q < q1 ? takes & (FULL << (q - q0)) : 0u;
                if (m) {  // the next position that takes the vector before it: a run
                    const int r = q0 + __ffs(m) - 1;
                    cur = f[elem(line, r - 1)];
                    if (gl == 0) C.fn[elem(line, r)] = cur;
                    q = r + 1;
                    carry = true;
                } else {
                    live = false;
                }
            }
            bool refused;
            const int n = taken(live, line, q, q1, cur, refused);
            if (live) {
                if (gl < n) C.fn[elem(line, q + gl)] = cur;
                q += n;
                if (refused) {  // the position keeps its own vector
                    q++;
                    carry = false;
                }
                if (q >= q1) live = false;
            }
        }
    }
    __syncthreads();
    // the segments whose first position met another vector, in order: walked again until the new vectors meet
    // the old ones
    if (segs > 1) {
        for (int line0 = 0; line0 < lines; line0 += NG) {
            bool live = line0 + grp < lines;
            const int line = live ? line0 + 1 + grp : 1;
            int s = 0, q = 0, end = 0;
            bool carry = false;
            float2 cur = make_float2(0.0f, 0.0f);
            // every round passes a segment, or a position of each live line
            for (int guard = 0; guard <= len + segs && __any_sync(FULL, live); guard++) {
                while (live && !carry) {  // the next segment to walk again
                    if (++s == segs) {
                        live = false;
                    } else {
                        q = 1 + s * seg;
                        end = min(q + seg, len - 1);
                        const int e = elem(line, q - 1);
                        cur = C.fn[e];
                        carry = !same_bits(cur, f[e]);
                    }
                }
                bool refused;
                const int n = taken(live, line, q, end, cur, refused);
                const int e = elem(line, min(max(q + gl, 1), len - 2));
                // an accepted position whose vector was this one already: the rest stands
                const unsigned met = group_ballot(live && gl < n && same_bits(C.fn[e], cur));
                // the refusing position keeps its own vector; if it did before, the rest stands. Only the lane that
                // stores it reads it (a ballot orders no memory accesses: another lane could read what was stored).
                const int r = elem(line, min(max(q + n, 1), len - 2));
                const bool changes = group_ballot(gl == 0 && live && refused && !met && !same_bits(C.fn[r], f[r])) != 0;
                if (live) {
                    if (gl < (met ? __ffs(met) - 1 : n)) C.fn[e] = cur;
                    if (met) {
                        carry = false;
                    } else {
                        q += n;
                        if (refused) {
                            cur = f[r];
                            if (changes && gl == 0) C.fn[r] = cur;
                            carry = changes;
                            q++;
                        }
                        if (q >= end) carry = false;
                    }
                }
                __syncwarp();
            }
        }
        __syncthreads();
    }
}

}  // namespace

__global__ void __launch_bounds__(COARSE_THREADS) k_solve_coarse(const __grid_constant__ CoarseJob J) {
    extern __shared__ __align__(16) float4 coarse_sm[];
    // block matching's planes (the flow's copy, the costs and the tests) lie in the tensor's, which it does not need
    const int M = J.pixels, PLANE = J.plane;
    Coarse C;
    C.tensor = coarse_sm;
    C.fn = (float2*)C.tensor;
    C.cost = (float*)(C.fn + M);
    C.takes = (unsigned char*)(C.cost + M);
    C.p1 = (float2*)(C.tensor + M);
    C.p2 = C.p1 + PLANE;
    C.grad = C.p2 + PLANE;
    C.f = C.grad + M;
    C.den7x = C.f + M;
    C.den7y = C.den7x + COARSE_MAX_LINE;
    C.den5x = C.den7y + COARSE_MAX_LINE;
    C.den5y = C.den5x + COARSE_MAX_LINE;
    C.a = (float*)(C.den5y + COARSE_MAX_LINE);
    C.b = C.a + M;
    __shared__ int s_any[32];
    const int tid = threadIdx.x;
    const bool af = J.af;
    auto flip = [&]() {
        float2* t = C.f;
        C.f = C.fn;
        C.fn = t;
    };
    if (tid < 32) s_any[tid] = 0;
    for (int l = J.start; l >= J.last; l--) {
        const int w = J.sizes[l][0], h = J.sizes[l][1], n = w * h;
        const float fw = (float)w, fh = (float)h;
        C.w = w;
        C.h = h;
        C.stride = (w + 2 * PAD + RUN) | 1;
        C.winv = inverse_of(w);
        C.hinv = inverse_of(h);
        C.iwinv = inverse_of(max(w - 2, 1));
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
        for (int i = tid; i < n; i += NT) {
            C.a[i] = __ldg(A + i);
            C.b[i] = __ldg(B + i);
        }
        for (int i = tid; i < (h + 2 * PAD) * C.stride; i += NT) C.p1[i] = C.p2[i] = outside_value<float2>();
        {  // a table each 128 threads
            const int table = tid / COARSE_MAX_LINE, i = tid % COARSE_MAX_LINE;
            if (table == 0 && i < w) C.den7x[i] = border_den<8>(i, w, J.g7.k);
            if (table == 1 && i < h) C.den7y[i] = border_den<8>(i, h, J.g7.k);
            if (table == 2 && i < w) C.den5x[i] = border_den<6>(i, w, J.g5.k);
            if (table == 3 && i < h) C.den5y[i] = border_den<6>(i, h, J.g5.k);
            static_assert(NT == 4 * COARSE_MAX_LINE, "a thread per entry");
        }
        __syncthreads();
        user();
        // the gradient and the tensor (flow.rs:283-328), its blur7 in two turns: the first two channels, then
        // the third, with the determinant of new_disp and calc_b of the first iteration
        for (int i = tid; i < n; i += NT) {
            const int y = over_of(i, C.winv), x = i - y * w;
            const float2 g = gradient_at<false>(C.a, mask_x, w, h, x, y);
            C.grad[i] = g;
            C.p1[C.at(x, y)] = make_float2(g.x * g.x, g.x * g.y);
        }
        __syncthreads();
        rows_pass<8>(C, J.g7, C.den7x);
        columns_pass<8>(C, J.g7, C.den7y, af, [&](int x, int y, int n, const float2* v) {
#pragma unroll
            for (int r = 0; r < RUN; r++) {
                if (r >= n) break;
                const int i = (y + r) * w + x;
                C.tensor[i] = make_float4(v[r].x, v[r].y, 0.0f, 0.0f);
                const float2 g = C.grad[i];
                C.p1[C.at(x, y + r)] = make_float2(g.y * g.y, 0.0f);
            }
        });
        rows_pass<8>(C, J.g7, C.den7x);
        // calc_b of the rows y .. y + n - 1 of column x, whose flow is f, into the padded plane
        auto b_of = [&](int x, int y, int n, const float2* f) {
            float i1[RUN];
            float2 g[RUN], b[RUN];
#pragma unroll
            for (int r = 0; r < RUN; r++) {
                const int i = min(y + r, h - 1) * w + x;
                i1[r] = C.a[i];
                g[r] = C.grad[i];
            }
            calc_b_run<RUN, false>(C.b, mask_y, w, h, x, y, f, i1, g, b);
#pragma unroll
            for (int r = 0; r < RUN; r++)
                if (r < n) C.p1[C.at(x, y + r)] = b[r];
        };
        columns_pass<8>(C, J.g7, C.den7y, af, [&](int x, int y, int n, const float2* v) {
            float2 f[RUN];
#pragma unroll
            for (int r = 0; r < RUN; r++) {
                const int i = min(y + r, h - 1) * w + x;
                f[r] = C.f[i];
                const float4 t = C.tensor[i];
                if (r < n) C.tensor[i] = make_float4(t.x, t.y, v[r].x, t.y * t.y - v[r].x * t.x);
            }
            b_of(x, y, n, f);
        });
        for (int it = 0; it < 3; it++) {
            rows_pass<8>(C, J.g7, C.den7x);
            columns_pass<8>(C, J.g7, C.den7y, af, [&](int x, int y, int n, const float2* b) {
                float4 t[RUN];
                float2 f[RUN];
#pragma unroll
                for (int r = 0; r < RUN; r++) {
                    const int i = min(y + r, h - 1) * w + x;
                    t[r] = C.tensor[i];
                    f[r] = C.f[i];
                }
                new_disp_run<RUN>(b, t, f);
#pragma unroll
                for (int r = 0; r < RUN; r++)
                    if (r < n) C.p1[C.at(x, y + r)] = f[r];
            });
            rows_pass<6>(C, J.g5, C.den5x);
            columns_pass<6>(C, J.g5, C.den5y, af, [&](int x, int y, int n, const float2* f) {
#pragma unroll
                for (int r = 0; r < RUN; r++)
                    if (r < n) C.f[(y + r) * w + x] = f[r];
                if (it < 2) b_of(x, y, n, f);
            });
        }
        // block matching (flow.rs:551-622): the row sweeps, then the column sweeps; no block has a cost in a
        // level of fewer than 4 x 4 pixels
        if (J.refine && w >= 4 && h >= 4) {
            sweep<false>(C, false, J.g7.z);
            flip();
            sweep<false>(C, true, J.g7.z);
            flip();
            sweep<true>(C, false, J.g7.z);
            flip();
            sweep<true>(C, true, J.g7.z);
            flip();
        }
        user();
        // the range check (flow.rs:430-442)
        int in = 0;
        for (int i = tid; i < n; i += NT) {
            int y = over_of(i, C.winv), x = i - y * w;
            float px = (float)x + C.f[i].x, py = (float)y + C.f[i].y;
            if (0.0f <= px && px <= fw - 1.0f && 0.0f <= py && py <= fh - 1.0f) in = 1;
        }
        if (__syncthreads_or(in) && tid == 0) {
            s_any[l] = 1;
            J.any[l] = 1;
        }
        __syncthreads();
        if (l == J.last) break;
        // the reset and the damping of the level, then the upsample into the next level
        const int dw = J.sizes[l - 1][0], dh = J.sizes[l - 1][1];
        const bool zero = zero_at_level(s_any, l, J.start);
        const bool damp_now = l == J.start && J.damp_any;
        const unsigned dinv = inverse_of(dw);
        for (int i = tid; i < dw * dh; i += NT) {
            int y = over_of(i, dinv), x = i - y * dw;
            C.fn[i] = upsample_at(C.f, w, h, J.up[l], zero, damp_now, J.damp, x, y);
        }
        __syncthreads();
        for (int i = tid; i < dw * dh; i += NT) C.f[i] = C.fn[i];
    }
    const int n = J.sizes[J.last][0] * J.sizes[J.last][1];
    for (int i = tid; i < n; i += NT) J.f_out[i] = C.f[i];
}

int coarse_plane(int w, int h) { return (h + 2 * PAD) * ((w + 2 * PAD + RUN) | 1); }
size_t coarse_smem_bytes(int pixels, int plane) {
    return (size_t)pixels * (sizeof(float4) + 2 * sizeof(float2) + 2 * sizeof(float)) +
           (2 * (size_t)plane + 4 * COARSE_MAX_LINE) * sizeof(float2);
}

TW_VARIANT_END
}  // namespace tw
