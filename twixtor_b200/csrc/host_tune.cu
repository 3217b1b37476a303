// The autotuner: per level size of a solve, the launch shapes of the solver iteration (tile shape
// and block size) and of block matching (block size per line), measured on the device and kept in
// the context's table, with a JSON file as its persistent cache. Every shape computes the same
// bytes (each element keeps the reference's operation order whatever the tiling), so the table
// changes only the time.
#include "runtime.h"

namespace tw {

// Deterministic stand-in data for the timings: planes of band-like values (a hash of the index,
// centred on 0, amplitude `amp`) and a small flow.
__global__ void k_tune_fill(float* p, long n, uint32_t seed, float amp) {
    long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t x = (uint32_t)i * 2654435761u ^ seed;
    x ^= x >> 15;
    x *= 2246822519u;
    x ^= x >> 13;
    p[i] = ((float)(x & 0xffffff) / 16777216.0f - 0.5f) * amp;
}

uint64_t key(int w, int h) { return ((uint64_t)(uint32_t)w << 32) | (uint32_t)h; }
bool valid_threads(int t, int max) { return t >= 32 && t <= max && t % 32 == 0; }

namespace {

const char* const TILE_NAMES[] = {"32x32", "64x32", "64x64", "16x16", "32x64"};  // by LEVEL_TILE_*
const char* tile_name(int t) { return TILE_NAMES[t]; }

// The table as JSON: the device's name, then one entry per level size.
std::string table_json(tw_ctx* ctx) {
    cudaDeviceProp prop{};
    cudaGetDeviceProperties(&prop, ctx->device);
    std::string out = "{\n  \"device\": \"";
    out += prop.name;
    out += "\",\n  \"levels\": {\n";
    size_t k = 0;
    char line[256];
    for (auto& kv : ctx->tune_table) {
        int w = (int)(kv.first >> 32), h = (int)(kv.first & 0xffffffffu);
        const LevelTune& t = kv.second;
        snprintf(line, sizeof line,
                 "    \"%dx%d\": {\"iter_tile\": \"%s\", \"iter_threads\": %d, \"bm_rows_threads\": %d, "
                 "\"bm_cols_threads\": %d}%s\n",
                 w, h, tile_name(t.iter_tile), t.iter_threads, t.bm_rows_threads, t.bm_cols_threads,
                 ++k < ctx->tune_table.size() ? "," : "");
        out += line;
    }
    out += "  }\n}\n";
    return out;
}

// Reads the entries of a table this library wrote for the same device; other lines are ignored.
void load_table(tw_ctx* ctx, const char* path) {
    FILE* f = fopen(path, "r");
    if (!f) return;
    cudaDeviceProp prop{};
    cudaGetDeviceProperties(&prop, ctx->device);
    char line[512];
    bool same_device = false;
    while (fgets(line, sizeof line, f)) {
        char dev[256];
        if (sscanf(line, " \"device\": \"%255[^\"]\"", dev) == 1) same_device = std::strcmp(dev, prop.name) == 0;
        int w, h, it, rt, ct;
        char tile[16];
        if (same_device &&
            sscanf(line, " \"%dx%d\": {\"iter_tile\": \"%15[0-9x]\", \"iter_threads\": %d, \"bm_rows_threads\": %d, "
                         "\"bm_cols_threads\": %d}",
                   &w, &h, tile, &it, &rt, &ct) == 6) {
            int t = LEVEL_TILE_32x32;
            for (int k = 0; k < 5; k++)
                if (std::strcmp(tile, TILE_NAMES[k]) == 0) t = k;
            if (w > 0 && h > 0 && valid_threads(it, LEVEL_ITER_MAX_THREADS) && valid_threads(rt, 1024) &&
                valid_threads(ct, 1024))
                ctx->tune_table[key(w, h)] = LevelTune{t, it, rt, ct};
        }
    }
    fclose(f);
}

}  // namespace
}  // namespace tw

extern "C" {

int tw_autotune(tw_ctx* ctx, const tw_flow_settings* s, int32_t width, int32_t height, const char* path,
                int32_t* measured) {
    if (!ctx) return TW_ERR_BAD_PARAM;
    std::lock_guard<std::mutex> lk(ctx->mu);
    ctx->cur = ctx->stream;
    if (measured) *measured = 0;
    if (!s || width <= 0 || height <= 0) return ctx->fail(TW_ERR_BAD_PARAM, "autotune: bad argument");
    Geo g;
    CHECK(geometry(*s, width, height, &g, &ctx->err));
    if (path) load_table(ctx, path);
    std::vector<int> todo;
    for (int l = 0; l < g.levels; l++)
        if (!ctx->tune_table.count(key(g.sizes[l][0], g.sizes[l][1]))) todo.push_back(l);
    if (!todo.empty()) {
        // stand-in planes of the largest level: the bands and their transposes, the gradient, the tensor,
        // the flow, its output, its transpose and a copy that block matching updates in place, and two B
        // planes of an even pitch, 16-byte aligned
        const size_t n0 = (size_t)g.w * g.h, bplane = (size_t)((g.w + 1) & ~1) * g.h;
        DevBuf buf;
        size_t held = 0;
        cudaError_t e = buf.ensure((n0 * (4 + 5 * 2 + 4) + 2 * 2 * bplane) * sizeof(float), &held);
        if (e != cudaSuccess) return ctx->cuda(e, "autotune buffers");
        float4* tensor = buf.as<float4>();
        float2 *bin = (float2*)(tensor + n0), *bout = bin + bplane, *grad = bout + bplane, *f = grad + n0, *fn = f + n0,
               *ft = fn + n0, *fsave = ft + n0;
        float *A = (float*)(fsave + n0), *Bp = A + n0, *AT = Bp + n0, *BT = AT + n0;
        uint32_t seed = 0;
        auto fill = [&](void* p, size_t floats, float amp) {
            k_tune_fill<<<grid1((long)floats), TB, 0, ctx->stream>>>((float*)p, (long)floats, 0x9e3779b9u * ++seed, amp);
            ctx->launches++;
        };
        fill(tensor, 4 * n0, 60.f);
        fill(bin, 2 * bplane, 50.f);
        fill(grad, 2 * n0, 8.f);
        fill(f, 2 * n0, 3.f);
        for (float* p : {A, Bp, AT, BT}) fill(p, n0, 40.f);
        cudaEvent_t e0 = nullptr, e1 = nullptr;
        cudaEventCreate(&e0);
        cudaEventCreate(&e1);
        auto timed = [&](auto&& run) -> float {  // the best of three after a warm-up launch
            run();
            float best = 1e30f;
            for (int r = 0; r < 3; r++) {
                cudaEventRecord(e0, ctx->stream);
                run();
                cudaEventRecord(e1, ctx->stream);
                cudaEventSynchronize(e1);
                float ms = 0.0f;
                cudaEventElapsedTime(&ms, e0, e1);
                best = std::min(best, ms);
            }
            return best;
        };
        bool af = s->taps_above_first != 0;
        for (int l : todo) {
            int w = g.sizes[l][0], h = g.sizes[l][1];
            LevelTune best = default_tune(w, h);
            // the solver iteration: every tile shape with 256 and 512 threads (64 x 64 with 512)
            const LevelTune iter_cands[9] = {{LEVEL_TILE_16x16, 256, 0, 0}, {LEVEL_TILE_16x16, 512, 0, 0},
                                             {LEVEL_TILE_32x32, 256, 0, 0}, {LEVEL_TILE_32x32, 512, 0, 0},
                                             {LEVEL_TILE_32x64, 256, 0, 0}, {LEVEL_TILE_32x64, 512, 0, 0},
                                             {LEVEL_TILE_64x32, 256, 0, 0}, {LEVEL_TILE_64x32, 512, 0, 0},
                                             {LEVEL_TILE_64x64, 512, 0, 0}};
            LevelIterArgs P;
            std::memset(&P, 0, sizeof P);
            P.b_in = bin;
            P.i1 = A;
            P.i0 = Bp;
            P.grad = grad;
            P.tensor = tensor;
            P.f = f;
            P.f_out = fn;
            P.b_out = bout;
            P.w = w;
            P.h = h;
            P.bp = (w + 1) & ~1;
            P.af = af;
            P.g7 = ctx->g7;
            P.g5 = ctx->g5;
            float bt = 1e30f;
            for (const LevelTune& c : iter_cands) {
                float ms = timed([&] { level_iter(ctx, c, P, false); });
                if (ms < bt) {
                    bt = ms;
                    best.iter_tile = c.iter_tile;
                    best.iter_threads = c.iter_threads;
                }
            }
            // block matching: the row and the column kernel, 128 to 512 threads per line (each one's
            // input field restored before every launch)
            if (w >= 4 && h >= 4) {
                const size_t fbytes = (size_t)w * h * sizeof(float2);
                cudaMemcpyAsync(fsave, f, fbytes, cudaMemcpyDeviceToDevice, ctx->stream);
                float br = 1e30f, bc = 1e30f;
                for (int th : {128, 256, 512}) {
                    float ms = timed([&] {
                        cudaMemcpyAsync(f, fsave, fbytes, cudaMemcpyDeviceToDevice, ctx->stream);
                        LAUNCH(ctx, k_bm_rows, h - 2, th, bm_smem_bytes(w), A, Bp, f, w, h, ft, ctx->g7.z);
                    });
                    if (ms < br) { br = ms; best.bm_rows_threads = th; }
                    ms = timed([&] {
                        cudaMemcpyAsync(ft, fsave, fbytes, cudaMemcpyDeviceToDevice, ctx->stream);
                        LAUNCH(ctx, k_bm_cols, w - 2, th, bm_smem_bytes(h), AT, BT, ft, w, h, f, ctx->g7.z, (int*)nullptr);
                    });
                    if (ms < bc) { bc = ms; best.bm_cols_threads = th; }
                }
            }
            ctx->tune_table[key(w, h)] = best;
            if (measured) (*measured)++;
        }
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        e = cudaStreamSynchronize(ctx->stream);
        if (e == cudaSuccess) e = cudaGetLastError();
        buf.release(&held);
        if (e != cudaSuccess) return ctx->cuda(e, "autotune");
    }
    if (path) {
        FILE* f = fopen(path, "w");
        if (!f) return ctx->fail(TW_ERR_BAD_PARAM, "autotune: cannot write %s", path);
        std::string js = table_json(ctx);
        fwrite(js.data(), 1, js.size(), f);
        fclose(f);
    }
    return TW_OK;
}

size_t tw_tuning_table(tw_ctx* ctx, char* buf, size_t cap) {
    if (!ctx) return 0;
    std::lock_guard<std::mutex> lk(ctx->mu);
    std::string js = table_json(ctx);
    if (buf && cap) {
        size_t m = std::min(js.size(), cap - 1);
        std::memcpy(buf, js.data(), m);
        buf[m] = 0;
    }
    return js.size();
}

int tw_tuning_clear(tw_ctx* ctx) {
    if (!ctx) return TW_ERR_BAD_PARAM;
    std::lock_guard<std::mutex> lk(ctx->mu);
    ctx->tune_table.clear();
    return TW_OK;
}

}  // extern "C"

extern "C" int tw_tuning_set(tw_ctx* ctx, int32_t width, int32_t height, int32_t iter_tile, int32_t iter_threads,
                             int32_t bm_rows_threads, int32_t bm_cols_threads) {
    if (!ctx) return TW_ERR_BAD_PARAM;
    std::lock_guard<std::mutex> lk(ctx->mu);
    if (width <= 0 || height <= 0 || iter_tile < 0 || iter_tile >= LEVEL_TILE_COUNT ||
        !tw::valid_threads(iter_threads, LEVEL_ITER_MAX_THREADS) || !tw::valid_threads(bm_rows_threads, 1024) ||
        !tw::valid_threads(bm_cols_threads, 1024))
        return ctx->fail(TW_ERR_BAD_PARAM, "tuning entry: tile %d, threads %d / %d / %d", iter_tile, iter_threads,
                         bm_rows_threads, bm_cols_threads);
    ctx->tune_table[tw::key(width, height)] = LevelTune{iter_tile, iter_threads, bm_rows_threads, bm_cols_threads};
    return TW_OK;
}
