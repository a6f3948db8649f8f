// Ray queries, the TinyEmbree Raytracer.Trace / IsOccluded drop-ins (Integrators/PathTracer.cs:319,467),
// their allocation-free form, and the light-path random walk (LightPathCache.TraceAllPaths).
#include "sst_host.h"

// The scene's one-entry job table (for the ray-query entry points), uploaded whenever its record
// changes: at a commit and when the 8-wide BVH is built.  Its source stays in the scene, as the copy may
// read it after this returns.
void uploadQueryJob(sst_scene* s) {
    s->queryJobHost = DevJob{};
    s->queryJobHost.sc = s->dev;
    s->queryJob.ensure(sizeof(DevJob));
    CUDA_CHECK(cudaMemcpyAsync(s->queryJob.p, &s->queryJobHost, sizeof(DevJob), cudaMemcpyHostToDevice, s->ctx->stream));
}

// Queries of up to this many rays between host arrays go through page-locked memory that the kernels
// read and write in place, instead of two copies.  In us, in place / copied, on the Cornell box, 205K and 1M
// triangles: closest hits of 97 rays 33 / 38, 48 / 53, 72 / 84, of 2048 rays 43 / 52, 67 / 76, 95 / 102, of 4096
// 52 / 53, 82 / 85, 114 / 122, of 8192 71 / 59, 109 / 102, 137 / 127 (the 48-byte records make the link the
// bound); occlusion of 97 rays 26 / 34, 37 / 45, 54 / 60, of 8192 37 / 44, 74 / 80, 93 / 104, of 16384 50 / 46,
// 78 / 82, 117 / 119, of 32768 87 / 51, 128 / 99, 143 / 111.  The lines lie where every scene gains.
constexpr int kTraceInPlace = 2048, kOcclInPlace = 8192;

// Trace / IsOccluded over n rays.  The traversal reads the SstRay records where they are (device
// arrays on a 16-byte boundary, apart from the results) or from one copy of them; sst_trace's SstHit
// records are expanded on the device from the traversal's (t, u, v, triangle) records.  The buffers are
// the context's and only grow, so repeated queries of the same size allocate nothing.
static void runQuery(sst_scene* s, const SstRay* rays, int n, SstHit* hits, int32_t* occl, int memory, bool anyHit) {
    static_assert(sizeof(SstHit) == sizeof(SstHitDev), "hit layout");
    static_assert(sizeof(SstRay) == 2 * sizeof(float4), "ray layout");
    if (!s || (n > 0 && !rays) || n < 0) fail(SST_ERR_INVALID_ARGUMENT, "invalid query");
    if (memory != SST_MEM_HOST && memory != SST_MEM_DEVICE) fail(SST_ERR_INVALID_ARGUMENT, "memory must be SST_MEM_HOST or SST_MEM_DEVICE");
    if (!s->committed) fail(SST_ERR_NOT_COMMITTED, "scene is not committed");
    if (n == 0) return;
    sst_ctx* c = s->ctx;
    CUDA_CHECK(cudaSetDevice(c->device));
    cudaStream_t st = c->stream;
    const bool device = memory == SST_MEM_DEVICE, inPlace = !device && n <= (anyHit ? kOcclInPlace : kTraceInPlace);
    const size_t rayBytes = size_t(n) * sizeof(SstRay), outBytes = size_t(n) * (anyHit ? sizeof(int32_t) : sizeof(SstHitDev));
    void* const userOut = anyHit ? static_cast<void*>(occl) : static_cast<void*>(hits);
    const TraceTuning tt = traceForBuilding(c, &s, 1);
    // page-locked: the overflow flag's record, then the rays and results of an in-place query
    c->queryStage.ensure(256 + size_t(kOcclInPlace) * (sizeof(SstRay) + sizeof(int32_t)));
    static_assert(size_t(kTraceInPlace) * (sizeof(SstRay) + sizeof(SstHitDev)) <= size_t(kOcclInPlace) * (sizeof(SstRay) + sizeof(int32_t)), "stage size");
    char* const stage = c->queryStage.as<char>();
    DevStats* const stats = reinterpret_cast<DevStats*>(stage);
    static_assert(sizeof(DevStats) <= 256, "query stage layout");
    std::memset(stats, 0, sizeof(DevStats));
    const void* dRays = rays;
    void* dOut = userOut;
    if (inPlace) {
        std::memcpy(stage + 256, rays, rayBytes);
        dRays = stage + 256;
        dOut = stage + 256 + rayBytes;
    } else {
        // device rays that the results overlay are copied too: a ray's flag may be written before another ray is read
        const char *r = reinterpret_cast<const char*>(rays), *o = static_cast<const char*>(userOut);
        const bool overlaid = o < r + rayBytes && r < o + outBytes;
        if (!device || overlaid || (reinterpret_cast<uintptr_t>(rays) & 15u)) {
            c->qRays.ensure(rayBytes);
            CUDA_CHECK(cudaMemcpyAsync(c->qRays.p, rays, rayBytes, device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice, st));
            dRays = c->qRays.p;
        }
        if (!device) {
            c->qOut.ensure(outBytes);
            dOut = c->qOut.p;
        }
    }
    c->qCnt.ensure(sizeof(int));
    CUDA_CHECK(cudaMemsetAsync(c->qCnt.p, 0, sizeof(int), st));
    if (!anyHit) c->qHits.ensure(size_t(n) * 16);
    launch_trace_query(tt, s->queryJob.as<DevJob>(), static_cast<const float4*>(dRays), n, c->qCnt.as<int>(), c->qHits.as<float4>(),
                       static_cast<int*>(dOut), stats, anyHit, st);
    if (!anyHit) launch_hit_expand(s->dev, c->qHits.as<float4>(), n, static_cast<SstHitDev*>(dOut), st);
    CUDA_CHECK(cudaGetLastError());
    if (!device && !inPlace) CUDA_CHECK(cudaMemcpyAsync(userOut, dOut, outBytes, cudaMemcpyDeviceToHost, st));
    CUDA_CHECK(cudaStreamSynchronize(st));
    if (stats->errorFlags & 1) fail(SST_ERR_DEVICE_LIMIT, "BVH traversal stack overflow");
    if (inPlace) std::memcpy(userOut, dOut, outBytes);
}

static LightPathBuf bindLight(DevBuf* b, size_t cap) {
    const size_t sz[9] = {4, 4, 4, 16, 16, 16, 16, 16, 16};
    for (int k = 0; k < 9; ++k) b[k].ensure(cap * sz[k]);
    LightPathBuf l;
    l.path = b[0].as<uint32_t>();
    l.rng = b[1].as<uint32_t>();
    l.depth = b[2].as<uint32_t>();
    l.prefix = b[3].as<float4>();
    l.approx = b[4].as<float4>();
    l.prevP = b[5].as<float4>();
    l.prevN = b[6].as<float4>();
    l.ro = b[7].as<float4>();
    l.rd = b[8].as<float4>();
    return l;
}

extern "C" {

int sst_trace(sst_scene* s, const SstRay* rays, int32_t n, SstHit* hits, int32_t memory) {
    return guarded([&] {
        if (!hits && n > 0) fail(SST_ERR_INVALID_ARGUMENT, "hits is NULL");
        runQuery(s, rays, n, hits, nullptr, memory, false);
    });
}

int sst_occluded(sst_scene* s, const SstRay* rays, int32_t n, int32_t* occluded, int32_t memory) {
    return guarded([&] {
        if (!occluded && n > 0) fail(SST_ERR_INVALID_ARGUMENT, "occluded is NULL");
        runQuery(s, rays, n, nullptr, occluded, memory, true);
    });
}


int sst_trace_light_paths(sst_scene* s, uint32_t seed, uint32_t iteration, int32_t numPaths, int32_t maxDepth, SstPathVertex* vertices,
                          int32_t* lengths, int32_t memory, SstRenderStats* stats) {
    static_assert(sizeof(SstPathVertex) == sizeof(SstPathVertexDev), "path vertex layout");
    return guarded([&] {
        if (!s || numPaths < 0 || numPaths > (1 << 24) || maxDepth < 1 || maxDepth > kMaxPathDepth || (numPaths > 0 && (!vertices || !lengths)))
            fail(SST_ERR_INVALID_ARGUMENT, "invalid light-path query");
        if (!s->committed) fail(SST_ERR_NOT_COMMITTED, "scene is not committed");
        SstRenderStats local = emptyStats();
        if (numPaths == 0) { if (stats) *stats = local; return; }
        sst_ctx* c = s->ctx;
        cudaStream_t st = c->stream;
        CUDA_CHECK(cudaSetDevice(c->device));
        const size_t n = size_t(numPaths), stride = size_t(maxDepth) + 1;
        LightPathBuf A = bindLight(c->lightA, n), B = bindLight(c->lightB, n);
        c->lightHits.ensure(n * 16);
        const size_t words = n * stride * (sizeof(SstPathVertexDev) / 4);
        float* dv = reinterpret_cast<float*>(vertices);
        int* dl = lengths;
        if (memory != SST_MEM_DEVICE) {
            c->lightVerts.ensure(words * 4);
            c->lightLengths.ensure(n * 4);
            dv = c->lightVerts.as<float>();
            dl = c->lightLengths.as<int>();
        }
        const LightVerts lv = memory == SST_MEM_HOST_PLANES ? LightVerts{dv, reinterpret_cast<int*>(dv + n * stride * 16), 16, 6}
                                                            : LightVerts{dv, reinterpret_cast<int*>(dv + 16), 22, 22};
        CUDA_CHECK(cudaMemsetAsync(dv, 0, words * 4, st));
        HostPrefault prefault;
        if (memory != SST_MEM_DEVICE) {
            prefault.add(vertices, words * 4);
            prefault.add(lengths, n * 4);
        }
        c->lightCnt.ensure(sizeof(int) * 2 * (size_t(maxDepth) + 3));
        int* cnt = c->lightCnt.as<int>();
        CUDA_CHECK(cudaMemsetAsync(cnt, 0, sizeof(int) * 2 * (size_t(maxDepth) + 3), st));
        c->stats.ensure(sizeof(DevStats));
        CUDA_CHECK(cudaMemsetAsync(c->stats.p, 0, sizeof(DevStats), st));
        const TraceTuning tt = traceForBuilding(c, &s, 1);
        const DevJob* job = s->queryJob.as<DevJob>();
        LightParams P{numPaths, maxDepth, seed, iteration};
        CUDA_CHECK(cudaEventRecord(c->ev0, st));
        launch_light_start(job, P, A, cnt, lv, dl, st);
        CUDA_CHECK(cudaGetLastError());
        prefault.start();
        int items = 0;
        CUDA_CHECK(cudaMemcpyAsync(&items, cnt, sizeof(int), cudaMemcpyDeviceToHost, st));
        CUDA_CHECK(cudaStreamSynchronize(st));
        // each step: closest hit, then one walk step (a path reaches at most maxDepth + 1 hits)
        for (int d = 0; d <= maxDepth && items > 0; ++d) {
            int* qIn = cnt + d;
            int* qOut = cnt + d + 1;
            int* work = cnt + (maxDepth + 2) + d;
            launch_trace_closest(tt, job, nullptr, A.ro, A.rd, qIn, work, c->lightHits.as<float4>(), c->stats.as<DevStats>(), st);
            launch_light_walk(job, P, A, B, c->lightHits.as<float4>(), qIn, qOut, lv, dl, items, st);
            CUDA_CHECK(cudaGetLastError());
            std::swap(A, B);
            CUDA_CHECK(cudaMemcpyAsync(&items, qOut, sizeof(int), cudaMemcpyDeviceToHost, st));
            CUDA_CHECK(cudaStreamSynchronize(st));
        }
        CUDA_CHECK(cudaEventRecord(c->ev1, st));
        prefault.finish();
        if (memory != SST_MEM_DEVICE) {
            CUDA_CHECK(cudaMemcpyAsync(vertices, dv, words * 4, cudaMemcpyDeviceToHost, st));
            CUDA_CHECK(cudaMemcpyAsync(lengths, dl, n * 4, cudaMemcpyDeviceToHost, st));
        }
        DevStats hs;
        CUDA_CHECK(cudaMemcpyAsync(&hs, c->stats.p, sizeof(DevStats), cudaMemcpyDeviceToHost, st));
        CUDA_CHECK(cudaStreamSynchronize(st));
        if (hs.errorFlags & 1) fail(SST_ERR_DEVICE_LIMIT, "BVH traversal stack overflow");
        float ms = 0.f;
        CUDA_CHECK(cudaEventElapsedTime(&ms, c->ev0, c->ev1));
        local.renderTimeMs = ms;
        local.numRays = hs.rays;
        if (stats) *stats = local;
    });
}

}  // extern "C"

// ---------------------------------------------------------------------------------------------
// Allocation-free occlusion query (sst_occluded_noalloc).  Its scratch is one array of fixed size
// in this library's device image, laid out as
//   [0, 256)      work counter of the traversal kernel
//   [256, 512)    DevStats (ray counts)
//   [512, 2048)   DevJob (the scene record the traversal kernel reads)
//   then          rays (two float4 x max rays), occlusion flags (int x max rays).
// ---------------------------------------------------------------------------------------------
namespace {
constexpr size_t kNaCounters = 0, kNaStats = 256, kNaJob = 512, kNaHeader = 2048;
constexpr size_t kNaMaxRays = SST_NOALLOC_MAX_RAYS;
constexpr size_t kNaBytes = kNaHeader + 2 * 16 * kNaMaxRays + 4 * kNaMaxRays;
static_assert(kNaBytes == 2361344, "the header states the scratch size");
static_assert(sizeof(DevStats) <= kNaJob - kNaStats && sizeof(DevJob) <= kNaHeader - kNaJob, "scratch header too small");
static_assert(alignof(DevJob) <= 256 && alignof(DevStats) <= 256, "scratch header alignment");
constexpr int kNaMaxDevices = 64;
}  // namespace

static __device__ __align__(256) unsigned char g_noallocScratch[kNaBytes];
static std::mutex g_noallocLock;
static void* g_noallocAddr[kNaMaxDevices] = {};

// Device address of the scratch array on `device` (the current device).  Looked up on the first
// call for each device and kept; the caller holds g_noallocLock.
static unsigned char* noallocScratch(int device) {
    if (device < 0 || device >= kNaMaxDevices) fail(SST_ERR_INVALID_ARGUMENT, "device ordinal beyond the allocation-free query's table");
    if (!g_noallocAddr[device]) {
        void* ptr = nullptr;
        cudaError_t e = cudaGetSymbolAddress((void**)&ptr, g_noallocScratch);
        if (e != cudaSuccess || !ptr) fail(SST_ERR_CUDA, std::string("cudaGetSymbolAddress(scratch): ") + cudaGetErrorString(e));
        g_noallocAddr[device] = ptr;
    }
    return static_cast<unsigned char*>(g_noallocAddr[device]);
}

extern "C" int sst_occluded_noalloc(sst_scene* s, const SstRay* rays, int32_t n, int32_t* occluded, int32_t memory) {
    return guarded([&] {
        if (!s || n < 0 || (n > 0 && (!rays || !occluded))) fail(SST_ERR_INVALID_ARGUMENT, "invalid query");
        if (memory != SST_MEM_HOST && memory != SST_MEM_DEVICE) fail(SST_ERR_INVALID_ARGUMENT, "memory must be SST_MEM_HOST or SST_MEM_DEVICE");
        if (size_t(n) > kNaMaxRays)
            fail(SST_ERR_INVALID_ARGUMENT, "sst_occluded_noalloc: " + std::to_string(n) + " rays exceed the limit of " + std::to_string(kNaMaxRays) +
                                               " rays per call (SST_NOALLOC_MAX_RAYS)");
        if (!s->committed) fail(SST_ERR_NOT_COMMITTED, "scene is not committed");
        if (n == 0) return;
        std::lock_guard<std::mutex> lock(g_noallocLock);
        sst_ctx* c = s->ctx;
        CUDA_CHECK(cudaSetDevice(c->device));
        unsigned char* base = noallocScratch(c->device);
        cudaStream_t st = c->stream;
        int* cnt = reinterpret_cast<int*>(base + kNaCounters);
        DevStats* stats = reinterpret_cast<DevStats*>(base + kNaStats);
        DevJob* job = reinterpret_cast<DevJob*>(base + kNaJob);
        float4* dRays = reinterpret_cast<float4*>(base + kNaHeader);
        int* occ = reinterpret_cast<int*>(dRays + 2 * kNaMaxRays);
        const cudaMemcpyKind in = memory == SST_MEM_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice;
        const cudaMemcpyKind out = memory == SST_MEM_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost;
        CUDA_CHECK(cudaMemcpyAsync(dRays, rays, size_t(n) * sizeof(SstRay), in, st));
        // set every call: the work counter and the statistics (zero), the job
        CUDA_CHECK(cudaMemsetAsync(base, 0, kNaJob, st));
        DevJob j{};
        j.sc = s->dev;
        CUDA_CHECK(cudaMemcpyAsync(job, &j, sizeof(DevJob), cudaMemcpyHostToDevice, st));
        launch_trace_query(traceFor(c, &s, 1), job, dRays, n, cnt, nullptr, occ, stats, true, st);
        CUDA_CHECK(cudaGetLastError());
        CUDA_CHECK(cudaMemcpyAsync(occluded, occ, size_t(n) * 4, out, st));
        CUDA_CHECK(cudaStreamSynchronize(st));
    });
}

