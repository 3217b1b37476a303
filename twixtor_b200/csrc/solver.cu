// Pyramid filters and the optical flow solver, strict mode. Each kernel cites the reference
// function (plugins/retime-engine/src/...) whose per-element arithmetic it repeats.
#include "kernels.cuh"
#include "level.cuh"

namespace tw {
TW_VARIANT_BEGIN

// flow/conv.rs:101-137 (border_value_ordered): one border element of a line whose element t is
// line[t * stride]. `multi` selects the 2- and 3-channel rule (the -1.0 sentinel decides whether a
// tap exists, so a real sample of exactly -1.0 is dropped too); LEFT_FIRST adds the tap at i - j
// before the tap at i + j.
template <bool LEFT_FIRST, class T>
__device__ __forceinline__ float border_value(const float* __restrict__ line, long stride, int len, int i,
                                              const T& t, bool multi) {
    float centre = (i >= 0 && i < len) ? line[(long)i * stride] : 0.0f;
    float num = t.k[0] * centre;
    float den = t.k[0];
#pragma unroll 1
    for (int j = t.n - 1; j >= 1; j--) {
        float kj = t.k[j];
#pragma unroll
        for (int side = 0; side < 2; side++) {
            bool right = (side == 0) != LEFT_FIRST;
            int tt = right ? i + j : i - j;
            bool inside = tt >= 0 && tt < len;
            float xv, wv;
            if (!multi) {
                xv = inside ? line[(long)tt * stride] : 0.0f;
                wv = inside ? kj : 0.0f;
            } else {
                float v = inside ? line[(long)tt * stride] : -1.0f;
                float mask = (v != -1.0f) ? 1.0f : 0.0f;
                xv = v;
                wv = mask * kj;
            }
            den = den + wv;
            num = num + xv * wv;
        }
    }
    return num / den;
}

// conv.rs:141-190 (hrow + interior_run), one output sample per thread
template <class T>
__device__ __forceinline__ void conv_h_px(const float* __restrict__ src, float* __restrict__ dst, int w, int h,
                                          const T& t, bool multi) {
    int x = blockIdx.x * blockDim.x + threadIdx.x;
    int y = blockIdx.y;
    if (x >= w || y >= h) return;
    const float* row = src + (long)y * w;
    int n = t.n;
    int head = min(n, w);
    int interior = max(w - 2 * n, 0);
    float r;
    if (x >= head && x < head + interior) {
        r = row[x] * t.k[0];
#pragma unroll 1
        for (int j = n - 1; j >= 1; j--) r = r + (row[x + j] + row[x - j]) * t.k[j];
    } else {
        r = border_value<false>(row, 1, w, x, t, multi);
    }
    dst[(long)y * w + x] = r;
}

// conv.rs:268-301 (vrow_ordered); the optional band output is flow.rs:266-267 (band = orig - blur)
template <class T>
__device__ __forceinline__ void conv_v_px(const float* __restrict__ src, float* __restrict__ dst, int w, int h,
                                          const T& t, bool multi, bool above_first, const float* __restrict__ orig,
                                          float* __restrict__ band) {
    int x = blockIdx.x * blockDim.x + threadIdx.x;
    int y = blockIdx.y;
    if (x >= w || y >= h) return;
    int n = t.n;
    int head = min(n, h);
    int interior = max(h - 2 * n, 0);
    float r;
    if (y >= head && y < head + interior) {
        r = src[(long)y * w + x] * t.k[0];
#pragma unroll 1
        for (int j = n - 1; j >= 1; j--) r = r + (src[(long)(y + j) * w + x] + src[(long)(y - j) * w + x]) * t.k[j];
    } else if (above_first) {
        r = border_value<true>(src + x, w, h, y, t, multi);
    } else {
        r = border_value<false>(src + x, w, h, y, t, multi);
    }
    long i = (long)y * w + x;
    dst[i] = r;
    if (band) band[i] = orig[i] - r;
}

__global__ void k_conv_h(const float* __restrict__ src, float* __restrict__ dst, int w, int h, Taps t, bool multi) {
    conv_h_px(src, dst, w, h, t, multi);
}

__global__ void k_conv_v(const float* __restrict__ src, float* __restrict__ dst, int w, int h, Taps t, bool multi,
                         bool above_first, const float* __restrict__ orig, float* __restrict__ band) {
    conv_v_px(src, dst, w, h, t, multi, above_first, orig, band);
}

// the same passes with the wide half kernels of the matte choke (one channel)
__global__ void k_conv_h_wide(const float* __restrict__ src, float* __restrict__ dst, int w, int h, WideTaps t) {
    conv_h_px(src, dst, w, h, t, false);
}

__global__ void k_conv_v_wide(const float* __restrict__ src, float* __restrict__ dst, int w, int h, WideTaps t,
                              bool above_first) {
    conv_v_px(src, dst, w, h, t, false, above_first, (const float*)nullptr, (float*)nullptr);
}

// ---- the 360 mode of the pyramid's filters (prep.rs:261-299, conv.rs:192-400, sample.rs:196-286) ------

// conv.rs:192-244 (hrow_wrapx): s = x[i] k0, then s = s + (x[(i+j) mod w] + x[(i-j) mod w]) k[j] for
// j = n-1 down to 1; the interior run is the same chain without a wrap
__global__ void k_conv_h_wrap(const float* __restrict__ src, float* __restrict__ dst, int w, int h, Taps t) {
    int x = blockIdx.x * blockDim.x + threadIdx.x;
    int y = blockIdx.y;
    if (x >= w || y >= h) return;
    const float* row = src + (long)y * w;
    float r = row[x] * t.k[0];
#pragma unroll 1
    for (int j = t.n - 1; j >= 1; j--) {
        int rr = (x + j) % w;
        int l = ((x - j) % w + w) % w;
        r = r + (row[rr] + row[l]) * t.k[j];
    }
    dst[(long)y * w + x] = r;
}

// conv.rs:326-400 (vpass_sphere): the element of column x at row yy, outside 0..h-1 found by the
// equirectangular walk from the edge row (reflect, and half a turn in x at every reflection)
__device__ __forceinline__ float sphere_at(const float* __restrict__ src, int w, int h, int x, int yy) {
    if (yy >= 0 && yy < h) return src[(long)yy * w + x];
    int half = w / 2;
    int c = x, r, d, steps;
    if (yy < 0) { r = 0; d = -1; steps = -yy; }
    else { r = h - 1; d = 1; steps = yy - h + 1; }
#pragma unroll 1
    for (int m = 0; m < steps; m++) {
        r += d;
        if (r < 0) { r = 0; d = -d; c = (half + c) % w; }
        else if (r >= h) { r = h - 1; d = -d; c = (half + c) % w; }
    }
    return src[(long)r * w + c];
}

// the column pass of the 360 mode: s = g[y] k0, s = s + (g[y+j] + g[y-j]) k[j]; with `band`, the band
// orig - s and its transpose (element (x, y) at [x * h + y]) for the column sweeps (flow.rs:264-267)
__global__ void k_conv_v_sphere(const float* __restrict__ src, float* __restrict__ dst, int w, int h, Taps t,
                                const float* __restrict__ orig, float* __restrict__ band, float* __restrict__ band_t) {
    int x = blockIdx.x * blockDim.x + threadIdx.x;
    int y = blockIdx.y;
    if (x >= w || y >= h) return;
    float r = src[(long)y * w + x] * t.k[0];
#pragma unroll 1
    for (int j = t.n - 1; j >= 1; j--) r = r + (sphere_at(src, w, h, x, y + j) + sphere_at(src, w, h, x, y - j)) * t.k[j];
    long i = (long)y * w + x;
    dst[i] = r;
    if (band) {
        float b = orig[i] - r;
        band[i] = b;
        if (band_t) band_t[(long)x * h + y] = b;
    }
}

// sample.rs:255-286 (bilinear1_sphere)
__device__ __forceinline__ float bilinear1_sphere(const float* __restrict__ img, int w, int h, float x, float y) {
    int w1 = w - 1, h1 = h - 1;
    int tx = cvtt32(x), ty = cvtt32(y);
    int ix = min(max(tx, 0), w1), iy = min(max(ty, 0), h1);
    float fx = x - (float)tx, fy = y - (float)ty;
    int x1 = ix + 1 > w1 ? 0 : ix + 1;
    int xc = ix, xd = x1, yc = iy + 1;
    if (iy + 1 > h1) {
        int half = w / 2;
        xc = (half + ix) % w;
        xd = (half + x1) % w;
        yc = h1;
    }
    float p00 = img[(long)iy * w + ix], p10 = img[(long)iy * w + x1];
    float p01 = img[(long)yc * w + xc], p11 = img[(long)yc * w + xd];
    float top = (p10 - p00) * fx + p00;
    float bot = (p11 - p01) * fx + p01;
    return (bot - top) * fy + top;
}

// sample.rs:205-230 (resample1_wrapx): the steps sw / dw and sh / dh, the equirectangular sampler
__global__ void k_resample_sphere(const float* __restrict__ src, int sw, int sh, float* __restrict__ dst, int dw, int dh) {
    int x = blockIdx.x * blockDim.x + threadIdx.x;
    int y = blockIdx.y;
    if (x >= dw || y >= dh) return;
    float sx = (float)sw / (float)dw, sy = (float)sh / (float)dh;
    dst[(long)y * dw + x] = bilinear1_sphere(src, sw, sh, (float)x * sx, (float)y * sy);
}

// flow/sample.rs:91-112 (resample1): corner aligned bilinear
__global__ void k_resample(const float* __restrict__ src, int sw, int sh, float* __restrict__ dst, int dw, int dh) {
    int x = blockIdx.x * blockDim.x + threadIdx.x;
    int y = blockIdx.y;
    if (x >= dw || y >= dh) return;
    float sx = ((float)sw - 1.0f) / (float)(dw - 1);
    float sy = ((float)sh - 1.0f) / (float)(dh - 1);
    dst[(long)y * dw + x] = bilinear1(src, sw, sh, (float)x * sx, (float)y * sy);
}

// The range check of a level whose flow the tracking points move at its end
__global__ void k_range_any(const float2* __restrict__ f, int w, int h, int* __restrict__ any_in_range) {
    int x = blockIdx.x * blockDim.x + threadIdx.x;
    int y = blockIdx.y;
    if (x < w && y < h) check_range(any_in_range, x, y, f[(long)y * w + x], w, h);
}

__global__ void k_deinterleave(const float* __restrict__ in, long n, float* __restrict__ fu, float* __restrict__ fv) {
    long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    fu[i] = in[2 * i];
    fv[i] = in[2 * i + 1];
}

// =====================================================================================================
// Block matching (flow.rs:447-622).
//
// A sweep is an in-place, loop-carried recurrence along a row (or a column): with v the vectors
// before the sweep, v'[x] = accept(x, v'[x-1]) ? v'[x-1] : v[x], where accept(x, n) holds when the
// target of v[x] lies in the level, its block cost c0 exists, the cost c1 at the target of n
// exists and c1 < c0 (Block::step, flow.rs:529-546). Every v'[x] is therefore the ORIGINAL vector
// of the start s <= x of its run, and a run started at j continues while accept(x, v[j]) holds.
// The kernel evaluates that exactly, in parallel:
//   1. c0[x] and the validity of v[x] for every x of the line;
//   2. end[j] = the first x past j where accept(x, v[j]) fails, for every candidate start j;
//   3. the run starts: 0, end[0], end[end[0]], ... (a chain walked in shared memory);
//   4. v'[x] = v[start of x's run].
// Each cost evaluation is Block::cost bit for bit, so the result equals the sequential sweep.

// Shared memory of one line of length len: u, v, c0 (floats), the three rows of A along the line
// (floats), end and two queues (ints), then 8 counters and two ints per 32-position chunk.
size_t bm_smem_bytes(int len) { return (size_t)len * 4 * (3 + 3 + 3) + (size_t)(8 + 2 * ((len + 31) / 32)) * 4; }

constexpr int BM_STAGES = 3;      // run extension tests made one per queued candidate before the lane groups
constexpr int BM_GROUP = 8;       // lanes per queued candidate after the stages (positions tested per round)
static_assert(BM_GROUP >= 2 && BM_GROUP < 32 && 32 % BM_GROUP == 0, "groups tile a warp");
constexpr int BM_TERM = 1 << 30;  // "past the line" in the chain tables

// The 3x3 patch of A around line position i (flow.rs:454-469) from the three lines of A in shared
// memory (rows y-1..y+1 for a row sweep, columns x-1..x+1 for a column sweep).
template <bool COLS>
__device__ __forceinline__ void bm_patch(const float* s_a, int len, int i, float p[9]) {
#pragma unroll
    for (int r = 0; r < 3; r++)
#pragma unroll
        for (int c = 0; c < 3; c++) p[r * 3 + c] = COLS ? s_a[c * len + (i - 1 + r)] : s_a[r * len + (i - 1 + c)];
}

// accept(i, n) of the sweep at line position i (Block::step, flow.rs:529-546): ci is the cost of the
// current vector (NaN when the step cannot happen at i: no target or no cost).
template <bool COLS>
__device__ __forceinline__ bool bm_accept(const float* s_a, int len, const float* __restrict__ B, int w, int h,
                                          int fixed, int i, float nu, float nv, float ci) {
    float p[9];
    bm_patch<COLS>(s_a, len, i, p);
    const int x = COLS ? fixed : i, y = COLS ? i : fixed;
    bool ok = true;
    int ix, iy;
    float fx, fy;
    bm_cell((float)x - nu, (float)(w - 2), w - 3, ok, ix, fx);
    bm_cell((float)y - nv, (float)(h - 2), h - 3, ok, iy, fy);
    const float c1 = bm_cost1<COLS>(B, COLS ? h : w, p, fx, fy, COLS ? (ix - 1) * h + iy - 1 : (iy - 1) * w + ix - 1);
    return ok && c1 < ci;
}

// The cost ci of the current vector (u, v) at line position i (NaN: no target, or no cost) and accept(i, n)
// for the vector (nu, nv), evaluated together.
template <bool COLS>
__device__ __forceinline__ bool bm_own_accept(const float* s_a, int len, const float* __restrict__ B, int w, int h, int fixed,
                                              int i, float u, float v, float nu, float nv, float z, float& ci) {
    float p[9];
    bm_patch<COLS>(s_a, len, i, p);
    const float x = (float)(COLS ? fixed : i), y = (float)(COLS ? i : fixed);
    const float wtop = (float)(w - 2), htop = (float)(h - 2);
    bool ok0 = true, ok1 = true;
    int ix0, iy0, ix1, iy1;
    float2 fx, fy;
    bm_cell(x - u, wtop, w - 3, ok0, ix0, fx.x);
    bm_cell(y - v, htop, h - 3, ok0, iy0, fy.x);
    bm_cell(x - nu, wtop, w - 3, ok1, ix1, fx.y);
    bm_cell(y - nv, htop, h - 3, ok1, iy1, fy.y);
    const float2 c = bm_cost2<COLS>(B, COLS ? h : w, p, fx, fy, COLS ? (ix0 - 1) * h + iy0 - 1 : (iy0 - 1) * w + ix0 - 1,
                                    COLS ? (ix1 - 1) * h + iy1 - 1 : (iy1 - 1) * w + ix1 - 1, z);
    ci = ok0 ? c.x : __int_as_float(0x7fc00000);
    return ok1 && c.y < ci;
}

// Appends val to q (counter *n) for the lanes of the warp with `want`: one atomic per warp. Every lane
// of the warp calls it.
__device__ __forceinline__ void bm_push(int* q, int* n, bool want, int val) {
    const unsigned m = __ballot_sync(0xffffffffu, want);
    if (m) {
        const int lane = threadIdx.x & 31, lead = __ffs(m) - 1;
        int base = 0;
        if (lane == lead) base = atomicAdd(n, __popc(m));
        base = __shfl_sync(0xffffffffu, base, lead);
        if (want) q[base + __popc(m & ((1u << lane) - 1u))] = val;
    }
}

// One sweep over a line held in shared memory (su, sv: the field along the line, updated in place;
// s_a: the three lines of A across it). The line is the row y (COLS false: pixel (i, y)) or the
// column x (COLS true: pixel (x, i)); len is its length. Forward sweeps run i = 1..len-2 with the
// neighbour i - 1, reverse sweeps i = len-2..1 with the neighbour i + 1. In "sweep order" position
// q (q = i forward, q = len-1-i reverse) both are the same forward recurrence
// v'[q] = accept(q, v'[q-1]) ? v'[q-1] : v[q], so every v'[q] is the vector of its run's start, and
// a run started at j ends at end[j], the first position past j that refuses v[j]. The sweep:
//   1. c0[i], the cost of the current vector, and the test of v[q-1], evaluated as a pair at every q:
//      end[q-1] = q where it refuses, the others queued;
//   2. the queued candidates extended one position per stage (BM_STAGES stages, the survivors
//      compacted after each), then the rest by groups of BM_GROUP lanes testing as many positions at once;
//   3. the chain of run starts 0, end[0], end[end[0]], ... in 32-position chunks, one warp per
//      chunk: the successor tables doubled by shuffles give every position's first chain element
//      past the chunk; one thread walks the chunks from position 0 (their entries and the last start
//      before each);
//   4. the owner of every position (the last start at or before it, by binary lifting over the
//      doubled tables from the chunk's entry), and v[owner] into the line.
// What bounds it: instruction issue on the fine levels, the latency of its stages on the coarse ones. The
// packed evaluation of step 1 (both sweeps; the reverse sweep used to queue and recompute the replaced
// positions' costs) took the launches at 960 x 540 from 81 to 74 us (rows) and 57 to 52 us (columns). Tried
// and slower: a warp of 32 neighbouring lines walking chunks of positions with carried vectors, chunks and
// clusters of blocks put right afterwards (half the instructions, but 64 to 80 us at 960 x 540 and 28 to 47
// us at 120 x 67 against 14: its steps follow one another).
// Every cost is Block::cost bit for bit, so the result equals the sequential sweep. The in place
// update is safe: step 4 reads only run starts, which keep their own vectors.
template <bool COLS>
__device__ void bm_sweep(float* su, float* sv, float* c0, const float* s_a, int* endp, int* qa, int* qb, int* ctl,
                         int* entry, int* prevl, const float* __restrict__ B, int w, int h, int fixed, int len,
                         bool reverse, float z) {
    const unsigned FULL = 0xffffffffu;
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
    auto line_of = [&](int q) -> int { return reverse ? len - 1 - q : q; };  // sweep position -> line index
    // 1. c0 and the test of v[q-1] at q (candidate j = q - 1)
    for (int qb0 = 0; qb0 < len; qb0 += nt) {
        const int q = qb0 + tid, j = q - 1;
        bool more = false;
        if (q >= 1 && q < len) {
            if (q <= len - 2) {
                const int i = line_of(q), jl = line_of(j);
                float ci;
                const bool take = bm_own_accept<COLS>(s_a, len, B, w, h, fixed, i, su[i], sv[i], su[jl], sv[jl], z, ci);
                c0[i] = ci;
                if (!take) endp[j] = q;
                else if (q + 1 <= len - 2) more = true;
                else endp[j] = len - 1;
            } else {
                endp[j] = len - 1;  // j = len - 2: no position left to test
            }
        }
        bm_push(qa, ctl + 0, more, j);
    }
    __syncthreads();
    // 2. stage t tests position j + t + 2 of every queued candidate j (counters rotate over ctl[0..2]:
    //    stage t reads ctl[t % 3], appends to ctl[(t + 1) % 3] and clears ctl[(t + 2) % 3], whose last
    //    reader passed the barrier before this stage)
    int nq = ctl[0];
    int* cur = qa;
    int* nxt = qb;
    int t = 0;
    for (; t < BM_STAGES && nq > 0; t++) {
        if (tid == 0) ctl[(t + 2) % 3] = 0;
        const int step = t + 2;
        for (int kb = 0; kb < nq; kb += nt) {
            const int k = kb + tid;
            bool more = false;
            int j = 0;
            if (k < nq) {
                j = cur[k];
                const int qq = j + step;  // <= len - 2: a candidate is queued only with a position left
                const int jl = line_of(j), il = line_of(qq);
                if (!bm_accept<COLS>(s_a, len, B, w, h, fixed, il, su[jl], sv[jl], c0[il])) endp[j] = qq;
                else if (qq + 1 > len - 2) endp[j] = len - 1;
                else more = true;
            }
            bm_push(nxt, ctl + (t + 1) % 3, more, j);
        }
        __syncthreads();
        nq = ctl[(t + 1) % 3];
        int* sw = cur;
        cur = nxt;
        nxt = sw;
    }
    //    the long runs: a group of BM_GROUP lanes per candidate, BM_GROUP positions per test round
    if (nq > 0) {
        constexpr int GPW = 32 / BM_GROUP;  // groups per warp
        const int g = lane / BM_GROUP, sub = lane % BM_GROUP, step = BM_STAGES + 2;
        for (int kb = warp * GPW; kb < nq; kb += nw * GPW) {
            const int k = kb + g;
            bool live = k < nq;
            const int j = live ? cur[k] : 0;
            const int jl = line_of(j);
            const float nu = live ? su[jl] : 0.0f, nv = live ? sv[jl] : 0.0f;
            int pos = j + step;
            for (int guard = 0; guard <= len && __any_sync(FULL, live); guard += BM_GROUP) {
                const int qq = pos + sub;
                bool refuse = false;
                if (live && qq <= len - 2) {
                    const int il = line_of(qq);
                    refuse = !bm_accept<COLS>(s_a, len, B, w, h, fixed, il, nu, nv, c0[il]);
                }
                const unsigned gm = (__ballot_sync(FULL, refuse) >> (g * BM_GROUP)) & ((1u << BM_GROUP) - 1u);
                if (live) {
                    if (gm) {
                        if (sub == 0) endp[j] = pos + __ffs(gm) - 1;
                        live = false;
                    } else if (pos + BM_GROUP > len - 2) {
                        if (sub == 0) endp[j] = len - 1;
                        live = false;
                    } else {
                        pos += BM_GROUP;
                    }
                }
            }
        }
    }
    __syncthreads();
    // 3. per chunk: J = the successor (end) doubled five times, L = the last start inside the chunk on
    //    the way; the queues are free now and take the two tables
    const int nch = (len + 31) >> 5;
    int* exitq = qa;
    int* lastq = qb;
    for (int c = warp; c < nch; c += nw) {
        const int base = c << 5, q = base + lane;
        int J = q <= len - 2 ? endp[q] : BM_TERM;
        int L = q;
#pragma unroll
        for (int r = 0; r < 5; r++) {
            const int src = J - base;  // > 0: a successor lies past its position
            const int tJ = __shfl_sync(FULL, J, src & 31);
            const int tL = __shfl_sync(FULL, L, src & 31);
            if (src < 32) {
                J = tJ;
                L = tL;
            }
        }
        if (q < len) {
            exitq[q] = J;
            lastq[q] = L;
        }
    }
    __syncthreads();
    //    the walk over the chunks from position 0: entry[c] = the first start in chunk c (-1: none),
    //    prevl[c] = the last start before it
    if (tid == 0) {
        int E = 0, Lp = -1, k = 0;
        for (int guard = 0; guard < len; guard++) {
            const int kE = E >> 5;
            for (; k < kE; k++) {
                entry[k] = -1;
                prevl[k] = Lp;
            }
            entry[kE] = E;
            prevl[kE] = Lp;
            k = kE + 1;
            Lp = lastq[E];
            const int F = exitq[E];
            if (F >= len - 1) break;  // the line's last position, or past it: no start to follow
            E = F;
        }
        for (; k < nch; k++) {
            entry[k] = -1;
            prevl[k] = Lp;
        }
        ctl[0] = ctl[1] = ctl[2] = 0;  // the next sweep's counters
    }
    __syncthreads();
    // 4. owners by binary lifting from the chunk's entry over the doubled tables Jr[r] (2^r successors,
    //    saturated at the chunk's end), then the scatter
    for (int c = warp; c < nch; c += nw) {
        const int base = c << 5, q = base + lane;
        int Jr[5];
        Jr[0] = q <= len - 2 ? endp[q] : BM_TERM;
#pragma unroll
        for (int r = 1; r < 5; r++) {
            const int src = Jr[r - 1] - base;
            const int tv = __shfl_sync(FULL, Jr[r - 1], src & 31);
            Jr[r] = src < 32 ? tv : Jr[r - 1];
        }
        const int e = entry[c];
        int own = prevl[c];
        if (e >= 0) {  // the same for the whole warp
            int x = e;
#pragma unroll
            for (int r = 4; r >= 0; r--) {
                const int y = __shfl_sync(FULL, Jr[r], (x - base) & 31);
                if (y <= q) x = y;
            }
            if (q >= e) own = x;
        }
        const bool moved = q >= 1 && q <= len - 2 && own != q;
        const int i = line_of(q);
        if (moved) {
            const int o = line_of(own);
            su[i] = su[o];
            sv[i] = sv[o];
        }
    }
    __syncthreads();
}

// The two sweeps of a line (flow.rs:551-622: left to right then right to left, or top to bottom
// then bottom to top), with the field, A's three lines and the tables in shared memory. The line is
// read contiguously from src (row y of the row-major field, or column x of the transposed one; a
// column's two end elements, which no sweep changes, from the row-major field ends) and its swept
// interior written across: element i of line `fixed` to dst[i * other + fixed], other = h for a row
// (into the transposed field the column sweeps read) and w for a column (back into the row-major
// field). So no transpose of the field runs between the row and the column sweeps; the reference
// transposes its field for the column sweeps (flow.rs:583-621). A and B of a column sweep are the
// transposed planes (element (x, y) at [x * h + y]) so that the line's patches stay contiguous.
template <bool COLS>
__device__ void bm_line(const float* __restrict__ A, const float* __restrict__ B, const float2* src, const float2* ends,
                        float2* dst, int w, int h, int fixed, float z, int* any) {
    extern __shared__ float sm[];
    const int len = COLS ? h : w, other = COLS ? w : h;
    if (len < 3) return;  // no interior position
    const int nch = (len + 31) >> 5;
    float* su = sm;
    float* sv = su + len;
    float* c0 = sv + len;
    float* s_a = c0 + len;  // 3 * len
    int* endp = (int*)(s_a + 3 * len);
    int* qa = endp + len;
    int* qb = qa + len;
    int* ctl = qb + len;  // 8 counters
    int* entry = ctl + 8;
    int* prevl = entry + nch;
    for (int i = threadIdx.x; i < len; i += blockDim.x) {
        const float2 f = COLS && (i == 0 || i == len - 1) ? ends[(long)i * w + fixed] : src[(long)fixed * len + i];
        su[i] = f.x;
        sv[i] = f.y;
#pragma unroll
        for (int o = 0; o < 3; o++)  // A at offset o-1 across the line: rows y-1..y+1, or columns x-1..x+1
            s_a[o * len + i] = __ldg(A + (long)(fixed - 1 + o) * len + i);
    }
    if (threadIdx.x < 8) ctl[threadIdx.x] = 0;
    __syncthreads();
    bm_sweep<COLS>(su, sv, c0, s_a, endp, qa, qb, ctl, entry, prevl, B, w, h, fixed, len, false, z);
    bm_sweep<COLS>(su, sv, c0, s_a, endp, qa, qb, ctl, entry, prevl, B, w, h, fixed, len, true, z);
    for (int i = threadIdx.x + 1; i <= len - 2; i += blockDim.x) {
        dst[(long)i * other + fixed] = make_float2(su[i], sv[i]);
    }
    if (COLS && any) {  // the range check of the level: this column, and the end ones, which are not swept
        for (int i = threadIdx.x; i < len; i += blockDim.x) {
            check_range(any, fixed, i, make_float2(su[i], sv[i]), w, h);
            if (fixed == 1) check_range(any, 0, i, dst[(long)i * w], w, h);
            if (fixed == w - 2) check_range(any, w - 1, i, dst[(long)i * w + w - 1], w, h);
        }
    }
}

// Two planes of w x h (row major) into their transposes (h x w), through a padded shared tile.
__global__ void k_transpose2(const float* __restrict__ a, const float* __restrict__ b, float* __restrict__ at,
                             float* __restrict__ bt, int w, int h) {
    __shared__ float ta[32][33], tb[32][33];
    int x0 = blockIdx.x * 32, y0 = blockIdx.y * 32;
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        int x = x0 + threadIdx.x, y = y0 + r;
        if (x < w && y < h) {
            ta[r][threadIdx.x] = a[(long)y * w + x];
            tb[r][threadIdx.x] = b[(long)y * w + x];
        }
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        int y = y0 + threadIdx.x, x = x0 + r;
        if (x < w && y < h) {
            at[(long)x * h + y] = ta[threadIdx.x][r];
            bt[(long)x * h + y] = tb[threadIdx.x][r];
        }
    }
}

// The row sweeps of rows 1..h-2 of the field f, the result into the transposed field ft (element (x,
// y) at [x * h + y]) at the interior of those rows
__global__ void __launch_bounds__(BM_MAX_THREADS) k_bm_rows(const float* __restrict__ A, const float* __restrict__ B, const float2* __restrict__ f, int w,
                          int h, float2* __restrict__ ft, float z) {
    int y = blockIdx.x + 1;  // rows 1..h-2
    if (y > h - 2) return;
    bm_line<false>(A, B, f, nullptr, ft, w, h, y, z, nullptr);
}

// The column sweeps of columns 1..w-2 from the transposed field ft that k_bm_rows wrote, the end rows 0
// and h-1 from f; the result into f at rows 1..h-2 of those columns; any (may be null): the level's range flag
__global__ void __launch_bounds__(BM_MAX_THREADS) k_bm_cols(const float* __restrict__ AT, const float* __restrict__ BT, const float2* __restrict__ ft, int w,
                          int h, float2* f, float z, int* any) {
    int x = blockIdx.x + 1;  // columns 1..w-2
    if (x > w - 2) return;
    bm_line<true>(AT, BT, ft, f, f, w, h, x, z, any);
}

TW_VARIANT_END
}  // namespace tw
