// Tests of the host driver (the C ABI without its kernels) over the CPU runtime of fake_cuda.h.  The kernel
// launches are recorded or do nothing.  Usage: driver_test <name>; exit status 0 when it holds.
#include <cstdio>
#include <cstring>
#include <map>
#include <string>
#include <vector>

#include "../../seesharp_gb300/csrc/sst_host.h"
#include "fake_cuda.h"

#define EXPECT(c)                                                             \
    do {                                                                      \
        if (!(c)) {                                                           \
            std::printf("%s:%d: %s does not hold\n", __FILE__, __LINE__, #c); \
            return 1;                                                         \
        }                                                                     \
    } while (0)

// ---- kernel launches --------------------------------------------------------------------------
struct Query {
    const float4* rays;
    const int* occl;
    DevScene scene;  // the job table's record, as the kernel finds it
    std::vector<char> read;  // the rays, as the kernel finds them
};
static std::vector<Query> g_queries;

namespace sst {
size_t lbvhScratchBytes(int) { return 256; }
size_t bvh4ScratchBytes(int) { return 256; }
size_t bvh8ScratchBytes(int) { return 256; }
int buildLbvh(const float4*, int, float4*, int*, void*, size_t, int* nodes, int* depth, cudaStream_t, int) { return *nodes = 1, *depth = 0, 0; }
int buildBvh4(const float4*, int, float4*, void*, int* nodes, int* depth, cudaStream_t) { return *nodes = 1, *depth = 1, 0; }
int buildBvh8(const float4*, int, float4*, void*, int* nodes, int* depth, cudaStream_t) { return *nodes = 1, *depth = 1, 0; }
void launch_leaf_gather(const int*, int, const float4*, const float4*, const int4*, const int4*, float4*, float4*, int4*, int4*, cudaStream_t) {}
void launch_env_build(const float4*, int, int, float*, float*, int*, float*, cudaStream_t) {}
void launch_camera(const DevJob*, const WaveChunk*, const WaveDesc*, const int*, const PathBuf&, int*, int, cudaStream_t) {}
void launch_light_start(const DevJob*, const LightParams&, const LightPathBuf&, int*, const LightVerts&, int*, cudaStream_t) {}
void launch_light_walk(const DevJob*, const LightParams&, const LightPathBuf&, const LightPathBuf&, const float4*, const int*, int*, const LightVerts&, int*,
                       int, cudaStream_t) {}
void launch_error_trim(const float*, int, int, int, double*, cudaStream_t) {}
void launch_variance_finish(const float*, const float*, int, int, float*, double*, cudaStream_t) {}
void launch_film_fold(const DevJob*, const WaveChunk*, const WaveDesc*, int*, const float*, DevStats*, int, int, cudaStream_t) {}
bool traceTuningValid(const TraceTuning&) { return true; }
int traceGrid(const TraceTuning&) { return 152; }
int traceMaxBlocksPerSM(const TraceTuning&) { return 1; }
void launch_trace_closest(const TraceTuning&, const DevJob*, const uint32_t*, const float4*, const float4*, const int*, int*, float4*, DevStats*,
                          cudaStream_t) {}
void launch_trace_shadow(const TraceTuning&, const DevJob*, const uint32_t*, const float4*, const float4*, const int*, const int*, int*, float4*, DevStats*,
                         cudaStream_t) {}
void launch_trace_query(const TraceTuning&, const DevJob* jobs, const float4* rays, int n, int*, float4*, int* occl, DevStats*, bool any, cudaStream_t) {
    fake::enqueue([=] {
        Query q{rays, occl, jobs[0].sc, {}};
        const char* r = reinterpret_cast<const char*>(rays);
        q.read.assign(r, r + size_t(n) * sizeof(SstRay));
        if (any) std::fill(occl, occl + n, 1);
        g_queries.push_back(q);
    });
}
void launch_wave_advance(int*, int, cudaStream_t) {}
void launch_partition(bool, const uint32_t*, const float4*, const int*, int*, int*, int, cudaStream_t) {}
bool shadeBlocksValid(int) { return true; }
void launch_shade(int, bool, bool, int, const DevJob*, const PathBuf&, const PathBuf&, const float4*, float4*, float4*, int, float4*, float4*, int*,
                  uint32_t*, const int*, int*, int*, float*, DevStats*, int, cudaStream_t) {}
void launch_shade_pyramid(int, const DevJob*, const PathBuf&, const PathBuf&, const float4*, float4*, int, float4*, float4*, int*, uint32_t*, const int*,
                          int*, int*, float*, DevStats*, const PyrArgs&, int, cudaStream_t) {}
void launch_hit_expand(const DevScene&, const float4*, int, SstHitDev*, cudaStream_t) {}
void launch_debug_material_eval(const DevScene&, int, int, const float*, const float*, const float*, float*, float*, cudaStream_t) {}
void launch_debug_material_sample(const DevScene&, int, int, const float*, const float*, const float*, float*, float*, float*, cudaStream_t) {}
void launch_debug_env(const DevScene&, int, const float*, float*, float*, float*, const float*, float*, float*, cudaStream_t) {}
void launch_debug_rng(uint32_t, uint32_t, int, const uint32_t*, int, uint32_t*, cudaStream_t) {}
void launch_debug_camera(const DevScene&, int, const float*, float*, float*, cudaStream_t) {}
}  // namespace sst

// ---- a scene of one emissive triangle ------------------------------------------------------------
static sst_scene* makeScene(sst_ctx* ctx) {
    sst_scene* s = nullptr;
    if (sst_scene_create(ctx, &s) != SST_OK) return nullptr;
    const float base[3] = {0.5f, 0.5f, 0.5f}, V[9] = {0, 0, 0, 1, 0, 0, 0, 1, 0}, rad[3] = {1, 1, 1};
    const float w2c[16] = {1, 0, 0, 0, 0, 1, 0, 0, 0, 0, 1, 0, 0, 0, -5, 1};
    const int32_t I[3] = {0, 1, 2};
    int32_t id = 0, first = 0, count = 0;
    if (sst_scene_add_material_diffuse(s, base, -1, 0, &id) != SST_OK) return nullptr;
    if (sst_scene_add_mesh(s, V, 3, I, 1, nullptr, nullptr, id, &id) != SST_OK) return nullptr;
    if (sst_scene_add_emitters(s, id, nullptr, 0, rad, -1.0f, &first, &count) != SST_OK) return nullptr;
    if (sst_scene_set_camera(s, w2c, 40.0f) != SST_OK) return nullptr;
    return s;
}

// ---- the tests --------------------------------------------------------------------------------------
// The job table that queries keep is read from memory that is still there, also when it is uploaded
// again because a query has built the 8-wide BVH.
static int queryJob(sst_ctx* ctx) {
    SstTuning t;
    EXPECT(sst_get_tuning(ctx, &t) == SST_OK);
    sst_scene* s = makeScene(ctx);
    EXPECT(s && sst_scene_commit(s, 8, 8) == SST_OK);
    SstRay ray{};
    ray.tmax = 1.0f;
    int32_t occ = -1;
    for (int width : {4, 8, 8}) {
        t.traceBvhWidth = width;
        EXPECT(sst_set_tuning(ctx, &t) == SST_OK);
        EXPECT(sst_occluded(s, &ray, 1, &occ, SST_MEM_HOST) == SST_OK && occ == 1);
        const DevScene& got = g_queries.back().scene;
        EXPECT(got.triv == s->triv.as<float4>() && got.nodes4 == s->nodes4.as<float4>() && got.nNodes4 == 1 && got.nTri == 1);
        EXPECT(got.nNodes8 == (width == 8 ? 1 : 0) && got.nodes8 == (width == 8 ? s->nodes8.as<float4>() : nullptr));
    }
    return sst_scene_destroy(s);
}

// Device results that overlay the rays are written only once the rays have been read.
static int overlay(sst_ctx* ctx) {
    sst_scene* s = makeScene(ctx);
    EXPECT(s && sst_scene_commit(s, 8, 8) == SST_OK);
    const int n = 100;
    SstRay* rays = nullptr;
    EXPECT(cudaMalloc(reinterpret_cast<void**>(&rays), n * sizeof(SstRay)) == cudaSuccess);
    for (int k = 0; k < n; ++k) rays[k] = SstRay{{float(k), 0, 0}, 0, {0, 0, 1}, 1};
    const std::vector<SstRay> before(rays, rays + n);
    int32_t* const at[] = {reinterpret_cast<int32_t*>(rays), reinterpret_cast<int32_t*>(rays + n / 2), reinterpret_cast<int32_t*>(rays + n) - 1};
    const int count[] = {n, 60, 1};
    for (int k = 0; k < 3; ++k) {
        std::copy(before.begin(), before.end(), rays);
        EXPECT(sst_occluded(s, rays, count[k], at[k], SST_MEM_DEVICE) == SST_OK);
        const Query& q = g_queries.back();
        const char *r0 = reinterpret_cast<const char*>(q.rays), *r1 = r0 + count[k] * sizeof(SstRay);
        const char *o0 = reinterpret_cast<const char*>(q.occl), *o1 = o0 + count[k] * sizeof(int32_t);
        EXPECT(q.occl == at[k] && (o1 <= r0 || r1 <= o0));
        EXPECT(std::memcmp(q.read.data(), before.data(), q.read.size()) == 0);
    }
    // apart: read where they are
    int32_t* occ = nullptr;
    EXPECT(cudaMalloc(reinterpret_cast<void**>(&occ), n * sizeof(int32_t)) == cudaSuccess);
    EXPECT(sst_occluded(s, rays, n, occ, SST_MEM_DEVICE) == SST_OK && g_queries.back().rays == reinterpret_cast<const float4*>(rays));
    cudaFree(occ);
    cudaFree(rays);
    return sst_scene_destroy(s);
}

static SstPathTracerParams params(int spp) {
    SstPathTracerParams p{};
    p.width = p.height = 8;
    p.totalSpp = spp;
    p.maxDepth = 3;
    p.numShadowRays = 1;
    return p;
}

// Output pages are populated by helper threads; a process that can start no more threads renders all the same.
static int threads(sst_ctx* ctx) {
    sst_scene* s = makeScene(ctx);
    EXPECT(s && sst_scene_commit(s, 8, 8) == SST_OK);
    const SstPathTracerParams p = params(2);
    std::vector<float> film(3 * 64);
    std::vector<SstPathVertex> v(10 * 4);
    std::vector<int32_t> len(10);
    fake::threadsFail = true;
    EXPECT(sst_render(s, &p, film.data(), SST_MEM_HOST, nullptr) == SST_OK);
    EXPECT(sst_trace_light_paths(s, 1, 0, 10, 3, v.data(), len.data(), SST_MEM_HOST, nullptr) == SST_OK);
    fake::threadsFail = false;
    return sst_scene_destroy(s);
}

// A render that fails midway has waited for what it launched: nothing runs on after it returns.
static int failedRender(sst_ctx* ctx) {
    sst_scene* s = makeScene(ctx);
    EXPECT(s && sst_scene_commit(s, 8, 8) == SST_OK);
    const SstPathTracerParams p = params(2);
    std::vector<float> film(3 * 64);
    bool failed = true;
    for (int k = 1; failed; ++k) {
        fake::failingRecord = k;
        failed = sst_render(s, &p, film.data(), SST_MEM_HOST, nullptr) != SST_OK;
        EXPECT(fake::pending() == 0);
        EXPECT(k > 2 || failed);
    }
    fake::failingRecord = 0;
    return sst_scene_destroy(s);
}

// Memory that a pool holds unused does not make another allocation fail, in or outside the pool, nor
// leave an error behind.
static int outOfMemory(sst_ctx* ctx) {
    const size_t MB = size_t(1) << 20;
    const size_t own = fake::used();
    fake::budget = own + 512 * MB;
    {
        DevBuf a, b, c, d;
        for (DevBuf* x : {&a, &b, &c}) x->pool = &ctx->scenePool;
        a.ensure(200 * MB);
        b.ensure(200 * MB);
        EXPECT(cudaStreamSynchronize(ctx->stream) == cudaSuccess);
        a.release();
        d.ensure(300 * MB);  // the context's own: 200 MB are in use and 200 MB held
        EXPECT(d.p && cudaGetLastError() == cudaSuccess);
        d.release();
        a.ensure(200 * MB);
        a.release();
        c.ensure(256 * MB);
        EXPECT(c.p && cudaGetLastError() == cudaSuccess);
        bool refused = false;
        try {
            d.ensure(300 * MB);
        } catch (const SstException& e) {
            refused = e.code == SST_ERR_OUT_OF_MEMORY;
        }
        EXPECT(refused && !d.p && d.bytes == 0 && cudaGetLastError() == cudaSuccess);
    }
    return 0;
}

// What is kept of a destroyed scene does not depend on how much memory other scenes use.
static int severalScenes(sst_ctx* ctx) {
    const size_t MB = size_t(1) << 20;
    sst_scene *a = makeScene(ctx), *b = makeScene(ctx);
    EXPECT(a && b && sst_scene_commit(a, 8, 8) == SST_OK && sst_scene_commit(b, 8, 8) == SST_OK);
    for (DevBuf* x : {&a->record, &a->gTex, &a->dLdI}) x->ensure(200 * MB);
    b->record.ensure(100 * MB);
    const size_t both = fake::used();
    EXPECT(sst_scene_destroy(b) == SST_OK);
    EXPECT(fake::used() >= both - 2 * MB && fake::used() <= both);
    for (DevBuf* x : {&a->record, &a->gTex}) x->release();
    EXPECT(sst_scene_commit(a, 8, 8) == SST_OK && fake::used() <= both - (500 - 256) * MB);
    return sst_scene_destroy(a);
}

// A destroyed scene leaves at most the pool's bound behind, without another call.
static int scenePool(sst_ctx* ctx) {
    const size_t MB = size_t(1) << 20, own = fake::used();
    const char* env = getenv("SST_SCENE_POOL_MB");
    const size_t bound = env ? size_t(atoi(env)) * MB : 256 * MB;
    sst_scene* s = makeScene(ctx);
    EXPECT(s && sst_scene_commit(s, 8, 8) == SST_OK);
    const size_t context = fake::used();  // the commit's scratch stays with the context
    for (DevBuf* b : {&s->record, &s->gTex, &s->dLdI}) b->ensure(200 * MB);
    EXPECT(fake::used() >= own + 600 * MB);
    EXPECT(sst_scene_destroy(s) == SST_OK);
    EXPECT(fake::pending() == 0 && fake::used() <= context + bound);
    EXPECT(bound == 0 || fake::used() >= own + bound);
    return 0;
}

// The films that a batch stages on the device go back with the call when they are large.
static int batchFilms(sst_ctx* ctx) {
    const int W = 4096, H = 2048;
    sst_scene *small = makeScene(ctx), *large = makeScene(ctx);
    EXPECT(small && large && sst_scene_commit(small, 8, 8) == SST_OK && sst_scene_commit(large, W, H) == SST_OK);
    std::vector<float> film(3 * size_t(W) * H), few(3 * 64);
    SstRenderJob jobs[2] = {};
    jobs[0].scene = large;
    jobs[0].params = params(1);
    jobs[0].params.width = W;
    jobs[0].params.height = H;
    jobs[0].film = film.data();
    jobs[1].scene = small;
    jobs[1].params = params(1);
    jobs[1].film = few.data();
    EXPECT(sst_render_batch(ctx, jobs + 1, 1, nullptr) == SST_OK);
    EXPECT(ctx->batchFilm.bytes > 0 && ctx->batchFilm.bytes < 4096);
    const void* kept = ctx->batchFilm.p;
    EXPECT(sst_render_batch(ctx, jobs + 1, 1, nullptr) == SST_OK && ctx->batchFilm.p == kept);
    EXPECT(sst_render_batch(ctx, jobs, 2, nullptr) == SST_OK);
    EXPECT(ctx->batchFilm.bytes <= (size_t(64) << 20));
    EXPECT(sst_forward_batch(ctx, jobs, 2, nullptr) == SST_OK);
    EXPECT(ctx->batchFilm.bytes <= (size_t(64) << 20));
    return sst_scene_destroy(small) + sst_scene_destroy(large);
}

int main(int argc, char** argv) {
    const std::map<std::string, int (*)(sst_ctx*)> tests = {{"query_job", queryJob}, {"overlay", overlay}, {"threads", threads}, {"failed_render", failedRender}, {"out_of_memory", outOfMemory}, {"scene_pool", scenePool}, {"several_scenes", severalScenes}, {"batch_films", batchFilms}};
    const auto it = argc > 1 ? tests.find(argv[1]) : tests.end();
    sst_ctx* ctx = nullptr;
    EXPECT(it != tests.end() && sst_create(0, &ctx) == SST_OK);
    const int rc = it->second(ctx);
    return rc ? rc : sst_destroy(ctx);
}
