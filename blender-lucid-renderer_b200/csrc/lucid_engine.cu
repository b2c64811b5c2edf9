// lucid_engine.cu — B200 path tracer: device BVH build, wavefront and
// whole-path kernels, film; host orchestration.
//
// A wave is a block of (pixel, sample) paths, sample-major.  Waves of at most
// 2^17 paths run in k_paths alone; larger ones start in the wavefront
// (wave_plan):
//   k_trace_primary               seed PCG32 per (x, y, sample), jitter, camera ray
//                                 and its closest hit
//   per depth:
//     k_trace_lb  (persistent)    closest BVH hit of the extension rays
//     k_trace_post                volume boundaries, triangles kept out of the
//                                 BVH, native lights, the shading bin
//     k_bin_scatter               the queue in bin order
//     k_shade     (persistent)    volume / emission / NEE / BSDF -> next queue,
//                                 shadow queue
//     k_shadow_pre                what of a shadow ray needs no BVH
//     k_shadow_lb (persistent)    any hit, adds unoccluded NEE
//   k_paths                       the paths left when a queue is short, each
//                                 followed to its end
// and then
//   k_film_output (k_film)        per-pixel sum in sample order (deterministic)
// Path state, hits and shadow rays are records of 64, 32 and 48 bytes; queues
// are compacted with warp ballots + one atomic per warp.  Work counts stay on
// the device; the host enqueues a whole wave without synchronising.
#include <cooperative_groups.h>
#include <cooperative_groups/scan.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <chrono>
#include <condition_variable>
#include <future>
#include <cub/cub.cuh>
#include <thrust/iterator/counting_iterator.h>
#include <array>
#include <map>
#include <mutex>
#include <thread>
#include <string>
#include <vector>

#include "lucid_diag.h"
#include "lucid_engine.h"
#include "lucid_guide.cuh"
#include "lucid_guide_host.h"
#include "lucid_kernels.cuh"

namespace lucid {
namespace cg = cooperative_groups;

#define CK(call)                                                                              \
    do {                                                                                      \
        cudaError_t e_ = (call);                                                              \
        if (e_ != cudaSuccess) return fail(e_ == cudaErrorMemoryAllocation ? LUCID_ERR_OOM     \
                                                                           : LUCID_ERR_CUDA,  \
                                           std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)

// ---------------------------------------------------------------- buffers
template <class T>
struct DBuf {
    T* p = nullptr;
    size_t n = 0;
    DBuf() = default;
    DBuf(const DBuf&) = delete;
    DBuf& operator=(const DBuf&) = delete;
    ~DBuf() { release(); }
    cudaError_t alloc(size_t count) {
        release();
        if (count == 0) count = 1;
        cudaError_t e = cudaMalloc(&p, count * sizeof(T));
        if (e == cudaSuccess) n = count; else p = nullptr;
        return e;
    }
    // As alloc, keeping an allocation that holds `count` and is at most about
    // twice as large (contents undefined either way).
    cudaError_t fit(size_t count) {
        if (p && n >= count && n <= 2 * count + 4096) return cudaSuccess;
        return alloc(count);
    }
    void release() { if (p) cudaFree(p); p = nullptr; n = 0; }
};

// One device allocation handed out in pieces: the temporaries of a BVH build
// (some thirty arrays; allocating and freeing each took 3 ms a build).
struct DeviceArena {
    unsigned char* p = nullptr;
    size_t used = 0, cap = 0;
    DeviceArena() = default;
    DeviceArena(const DeviceArena&) = delete;
    DeviceArena& operator=(const DeviceArena&) = delete;
    ~DeviceArena() { if (p) cudaFree(p); }
    static size_t round(size_t b) { return (b + 255) & ~(size_t)255; }
    cudaError_t reserve(size_t bytes) {
        cudaError_t e = cudaMalloc((void**)&p, bytes);
        if (e == cudaSuccess) cap = bytes; else p = nullptr;
        return e;
    }
    // null, now and from then on, when the arena is exhausted
    template <class T>
    T* take(size_t n) {
        const size_t b = round(std::max<size_t>(1, n) * sizeof(T));
        if (used + b > cap) {
            cap = 0;
            return nullptr;
        }
        T* q = reinterpret_cast<T*>(p + used);
        used += b;
        return q;
    }
};

// Pinned host memory for what a call reads back (a few kilobytes a context):
// page-locking a block takes about a millisecond, so up to kPinnedKept blocks
// that closed contexts gave back are kept for the next ones.
constexpr size_t kPinnedBytes = 48 << 10;
constexpr size_t kPinnedKept = 16;
namespace {
std::mutex g_pinned_mu;
std::vector<void*>& pinned_blocks() {
    static std::vector<void*>* v = new std::vector<void*>();   // (no CUDA call from a static destructor)
    return *v;
}
cudaError_t pinned_take(void** p) {
    {
        std::lock_guard<std::mutex> lk(g_pinned_mu);
        std::vector<void*>& v = pinned_blocks();
        if (!v.empty()) {
            *p = v.back();
            v.pop_back();
            return cudaSuccess;
        }
    }
    return cudaHostAlloc(p, kPinnedBytes, cudaHostAllocPortable);
}
void pinned_give(void* p) {
    {
        std::lock_guard<std::mutex> lk(g_pinned_mu);
        std::vector<void*>& v = pinned_blocks();
        if (v.size() < kPinnedKept) {
            v.push_back(p);
            return;
        }
    }
    cudaFreeHost(p);
}
}  // namespace

struct DeviceScene {
    DBuf<float4> bvh_tris, bnd_tris, bnd_box, big_tris, prim_fn, prim_vn, light_bsph;
    DBuf<int4> prim_info;
    DBuf<unsigned char> prim_cls;
    DBuf<int> guide;
    DBuf<DevNode4> nodes;
    DBuf<DevNode> nodes2;
    DBuf<DevMaterial> materials;
    DBuf<float4> tex_ops, prim_uv;
    DBuf<DevLight> lights;
    DBuf<float> cdf, grid;
    DBuf<DevVolume> volumes;
    DevScene view{};
    // an edited version (Engine::update_scene) owns only its material, light
    // and class arrays and keeps the version whose geometry it renders alive
    std::shared_ptr<DeviceScene> base;
    void release() {
        base.reset();
        bvh_tris.release(); bnd_tris.release(); bnd_box.release(); light_bsph.release(); big_tris.release(); prim_fn.release(); prim_vn.release(); prim_info.release();
        prim_cls.release(); nodes.release(); nodes2.release(); guide.release(); materials.release(); tex_ops.release(); prim_uv.release(); lights.release(); cdf.release(); grid.release(); volumes.release();
    }
};

// Per-path state, indexed by path id (sample-major within a wave), and the
// queues.  The queues visit paths in bin order, so a path's state is reached
// by scattered accesses: what one kernel reads or writes together lies in one
// 64- or 32-byte record, so that every 32-byte sector moved is used whole
// (one array per field moved 32 bytes for each 16 or 8 used: the 1M-triangle
// 1080p frame shades in 43.1 ms that way).
struct alignas(64) PathState {
    float4 ray_o;      // origin, tMin
    float4 ray_d;      // direction, depth (int bits)
    float4 thr;        // throughput rgb, pdf of the sampler that chose the ray
    ulonglong2 rng;    // PCG state, increment
};
struct alignas(32) PathHit {
    float4 hit;        // t, u, v, prim (int bits, -1 = miss)
    float4 light;      // native light index (int bits, -1 = none), t
};
// A queued light sample, stored at its place in the shadow queue.
struct ShadowRec {
    float4 o;          // origin, length
    float4 d;          // direction, guide slot to credit first (int bits)
    float4 c;          // radiance added when unoccluded, path id (int bits)
};
struct PathView {
    PathState* st;
    PathHit* hit;
    float4* rad;       // accumulated radiance
    ShadowRec* sh;     // the shadow queue
    int* q0;
    int* q1;
    int* qb;           // shading queue binned by event / material class
    unsigned short* cls;  // shading bin of each queue entry's pending event
    int* counters;     // per depth: [0] active, [1] shadow, [2..4] fetch cursors, [5] shadow rays to trace,
                       // [8, 8 + kBins) bin counts, then kBins bin cursors
    int* errors;       // [0] traversal stack overflow, from [4] on k_paths' PathsCount
    int2* rec_prim;
    int4* rec_cnt;     // bounces, nee tests, nee occluded
    unsigned long long* rec_hash;
    // path guiding (null when off)
    float* gmix;       // compact guide mixture per path (k_guide_infer, kGMixFloats)
    int4* gslot;       // training records of the path's 3 latest guided vertices (-1: none)
    float4* ginv;      // 3 per path: 1 / throughput after each of those vertices
    GuideRec* grec;    // training records of this wave
    int* gcount;       // [0] records written, [1] guided vertices
    int gcap;
    unsigned gkeep;    // a guided vertex is recorded when its hash < gkeep
    int gdepth;        // vertices at path depth < gdepth are guided
    float glo[3], gscale[3];   // scene box -> [0,1]^3
    // batched jobs (null otherwise): the device table of the batch's scenes
    // and each path's index into it, set with its camera ray
    const DevScene* scenes;
    unsigned short* sid;
};
// Shading bins: the event / material class (bin_class, 16 values) times
// the cell of the hit point in a 4 x 4 x 4 grid over the scene box.
constexpr int kClassBins = 16;
constexpr int kCellBits = 2;                       // per axis
constexpr int kCellDim = 1 << kCellBits;
constexpr int kCells = 1 << (3 * kCellBits);
constexpr int kBins = kClassBins * kCells;
constexpr int kCountersPerDepth = 8 + 2 * kBins;
constexpr int kMaxDepth = 1024;
constexpr int kErrorInts = 16;   // PathView::errors

struct PathPool {
    long long cap = 0;
    bool records = false;
    DBuf<PathState> st;
    DBuf<PathHit> hit;
    DBuf<ShadowRec> sh;
    DBuf<float4> rad;
    DBuf<int> q0, q1, qb, counters, errors;
    DBuf<unsigned short> cls;
    DBuf<int2> rec_prim;
    DBuf<int4> rec_cnt;
    DBuf<unsigned long long> rec_hash;
    DBuf<float4> film;
    DBuf<float4> out;
    size_t film_n = 0;
    DBuf<double> film64, out64;   // FP64 accumulation (converged references)
    size_t film64_n = 0;
    DBuf<unsigned short> sid;     // batched jobs: scene index per path (render_batch)
    DBuf<unsigned char> btab;     // batched jobs: the scene table, then a wave's job table
    PathView view{};
    void release() {
        sid.release();
        btab.release();
        st.release(); hit.release(); sh.release(); rad.release(); q0.release(); q1.release();
        qb.release(); cls.release();
        counters.release(); errors.release(); rec_prim.release(); rec_cnt.release(); rec_hash.release();
        film.release(); out.release(); film64.release(); out64.release();
        film_n = 0;
        film64_n = 0;
        cap = 0;
    }
};

// Path guiding: the network and the per-path / per-wave buffers.
constexpr int kGuideBatch = 1 << 18;   // training records per step
constexpr long long kGuideWave = 1LL << 24;
struct GuideState {
    GuideNet net;
    DBuf<float> gmix;
    DBuf<int4> gslot;
    DBuf<float4> ginv;
    DBuf<GuideRec> recs;
    DBuf<int> count;
    long long cap = 0;
    float keep = 1.0f;
    float lr = 1e-2f;
    int steps = 2;   // Adam steps per wave, each on its own batch of records
    int max_depth = 1;   // vertices at path depth < max_depth are guided (camera hits: depth 0)
    bool on = false;
};

// Completed-path records of the path diagnostics (compact form: 16-B units
// and an index of each record's first unit) and their counts.
struct DiagDevice {
    DBuf<uint4> units;
    DBuf<uint32_t> index;
    DBuf<unsigned long long> count;   // [0] records, [1] units
    // pinned host copies of a band's records, two of them: the host replays
    // one band while the device renders the next into the other (kept
    // between calls: page-locked copies run at full link speed and the
    // buffers are not zero-filled)
    uint8_t* host_units[2] = {nullptr, nullptr};
    uint32_t* host_index[2] = {nullptr, nullptr};
    size_t host_units_cap[2] = {0, 0}, host_index_cap[2] = {0, 0};
    ~DiagDevice() {
        for (int b = 0; b < 2; ++b) {
            if (host_units[b]) cudaFreeHost(host_units[b]);
            if (host_index[b]) cudaFreeHost(host_index[b]);
        }
    }
    // grows a pinned buffer of `elem`-byte entries to hold n, keeping the first `keep`
    template <typename T>
    static cudaError_t grow(T*& buf, size_t& cap, size_t n, size_t keep, size_t elem) {
        if (n <= cap) return cudaSuccess;
        const size_t c = n + n / 4;
        T* h = nullptr;
        cudaError_t e = cudaHostAlloc(reinterpret_cast<void**>(&h), c * elem, cudaHostAllocDefault);
        if (e != cudaSuccess) return e;
        if (buf && keep) std::memcpy(h, buf, keep * elem);
        if (buf) cudaFreeHost(buf);
        buf = h;
        cap = c;
        return cudaSuccess;
    }
    cudaError_t reserve_host(int b, size_t n_rec, size_t keep_rec, size_t n_units, size_t keep_units) {
        cudaError_t e = grow(host_index[b], host_index_cap[b], n_rec, keep_rec, sizeof(uint32_t));
        if (e != cudaSuccess) return e;
        return grow(host_units[b], host_units_cap[b], n_units, keep_units, kDiagUnitBytes);
    }
};

struct FrameParams {
    float pos[3], fwd[3], right[3], up[3];
    float aspect, scale;
    int tile_x, tile_y, tile_w, tile_h, full_w, full_h;
    int samples, sample_offset, max_depth, algo;
    int npix;
    int s0;          // first sample (within the call) of this wave
    int n_wave;      // paths in this wave
    int records;
    int jitter;      // jitter camera rays even when `samples` is 1 (progressive jobs)
    const int* dyn;  // when set, dyn[0] replaces sample_offset (graph-replayed iterations)
};

// ---------------------------------------------------------------- warp helpers
LD unsigned lane_id() { return threadIdx.x & 31u; }

// Warp-aggregated append: one atomic per warp, ranks from the ballot.
// Returns the lane's place in the queue (meaningful where pred holds).
LD int warp_append(int* counter, bool pred) {
    unsigned mask = __ballot_sync(0xffffffffu, pred);
    if (mask == 0) return 0;
    int leader = __ffs(mask) - 1;
    int base = 0;
    if ((int)lane_id() == leader) base = atomicAdd(counter, __popc(mask));
    base = __shfl_sync(0xffffffffu, base, leader);
    return base + __popc(mask & ((1u << lane_id()) - 1u));
}

// Persistent-thread work fetch: a warp claims 32 consecutive items.
LD int warp_fetch(int* cursor) {
    int base = 0;
    if (lane_id() == 0) base = atomicAdd(cursor, 32);
    return __shfl_sync(0xffffffffu, base, 0);
}

// ---------------------------------------------------------------- raygen
LD V3 primary_dir(const FrameParams& f, float nx, float ny) {
    V3 v = v3(f.fwd[0] + f.right[0] * (nx * f.scale) + f.up[0] * (ny * f.scale),
              f.fwd[1] + f.right[1] * (nx * f.scale) + f.up[1] * (ny * f.scale),
              f.fwd[2] + f.right[2] * (nx * f.scale) + f.up[2] * (ny * f.scale));
    return make_dir_or(v, v3(f.fwd[0], f.fwd[1], f.fwd[2]));
}

// Primary ray of path `local` of the frame (pybind_renderer.hpp:250-293):
// NDC, seed (x, y, offset + s), two jitter draws when the call has more than
// one sample; returns the direction (the origin is the camera position, tMin
// 0) and the path's RNG stream.
LD V3 camera_dir(const FrameParams& f, int local, Rng& rng) {
    int p = local % f.npix, sl = local / f.npix;
    int gx = f.tile_x + p % f.tile_w, gy = f.tile_y + p / f.tile_w;
    float nx = (2.0f * ((float)gx + 0.5f) / (float)f.full_w - 1.0f) * f.aspect;
    float ny = 1.0f - 2.0f * ((float)gy + 0.5f) / (float)f.full_h;
    const int offset = f.dyn ? f.dyn[0] : f.sample_offset;
    rng = seed_xyz((uint32_t)gx, (uint32_t)gy, (uint32_t)(offset + f.s0 + sl));
    if (f.samples > 1 || f.jitter) {
        float jx = (randf(rng) - 0.5f) / (float)f.full_w;
        float jy = (randf(rng) - 0.5f) / (float)f.full_h;
        return primary_dir(f, nx + jx, ny + jy);
    }
    return primary_dir(f, nx, ny);
}

LD void records_begin(const PathView& pv, int id) {
    pv.rec_prim[id] = make_int2(-1, -1);
    pv.rec_cnt[id] = make_int4(0, 0, 0, 0);
    pv.rec_hash[id] = 1469598103934665603ULL;
}

// The primary ray of path `local` of the frame `f` stored as wave path `id`
// (a batched job's paths start at its base in the wave) with the path's
// initial state.
LD V3 camera_ray_at(const FrameParams& f, const PathView& pv, int local, int id) {
    Rng rng;
    const V3 d = camera_dir(f, local, rng);
    PathState& st = pv.st[id];
    st.ray_o = make_float4(f.pos[0], f.pos[1], f.pos[2], 0.0f);
    st.ray_d = make_float4(d.x, d.y, d.z, __int_as_float(0));
    st.thr = make_float4(1.0f, 1.0f, 1.0f, 0.0f);
    st.rng = make_ulonglong2(rng.state, rng.inc);
    pv.rad[id] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (f.records) records_begin(pv, id);
    return d;
}
LD V3 camera_ray(const FrameParams& f, const PathView& pv, int id) { return camera_ray_at(f, pv, id, id); }

// Primary rays alone, for the passes that do not trace them at once.
__global__ void k_raygen(FrameParams f, PathView pv) {
    int id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id == 0) pv.counters[0] = f.n_wave;
    if (id >= f.n_wave) return;
    camera_ray(f, pv, id);
}

// ---------------------------------------------------------------- trace
// Idle lanes of a warp that make it fetch new rays (1M-triangle frame, closest
// hit + shadow rays: 8 -> 78.1 ms, 16 -> 77.2 ms, 20 -> 77.7 ms).
constexpr int kRefill = 16;

LD unsigned lanemask_lt() { return (1u << lane_id()) - 1u; }

// Claims a queue index for each lane of `idle` (one atomic per warp); every
// lane calls it.  `exhausted` is set for the warp once the queue is drained.
LD int warp_refill(int* cursor, int n, unsigned idle, bool& exhausted) {
    const int leader = __ffs(idle) - 1, want = __popc(idle);
    int base = 0;
    if ((int)lane_id() == leader) base = atomicAdd(cursor, want);
    base = __shfl_sync(0xffffffffu, base, leader);
    exhausted = base + want >= n;
    const int r = base + __popc(idle & lanemask_lt());
    return ((idle >> lane_id()) & 1u) && r < n ? r : -1;
}

// Per-lane dynamic refill: lanes without a ray claim new ones together (one
// atomic per warp per round); `exhausted` stops claiming once the queue is
// drained.  Returns the claimed index or -1.
LD int refill(int* cursor, int n, bool need, bool& exhausted) {
    unsigned m = __ballot_sync(0xffffffffu, need && !exhausted);
    if (m == 0) return -1;
    int leader = __ffs(m) - 1;
    int base = 0;
    if ((int)lane_id() == leader) base = atomicAdd(cursor, __popc(m));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (!(need && !exhausted)) return -1;
    int r = base + __popc(m & lanemask_lt());
    if (r >= n) { exhausted = true; return -1; }
    return r;
}

// ---------------------------------------------------------------- shading bins
// The shading kernel is limited by instruction fetch: divergent warps run
// different parts of it (light/environment hits, emitters, glass, near-delta
// metal, general Principled lobes, volume delta tracking).  Before each
// shading launch the queue is binned by that class — a counting sort whose
// histogram the trace kernels build as each ray finishes (the hit, the
// native-light hit and the ray are still in registers there) and whose
// scatter pass is k_bin_scatter — so neighbouring warps shade the same kind
// of event.  The order of paths in a queue does not change any result.
LD int bin_class(const DevScene& sc, int prim, float t, int li, float lt, V3 o, V3 d, bool vol) {
    // 0: light or environment reached; else the prim's material class
    // (emitter, glass, near-delta metal, metal, dielectric), set at upload
    int c = (prim >= 0 && !(li >= 0 && lt < t)) ? (int)__ldg(sc.prim_cls + prim) : 0;
    if (vol && sc.num_volumes > 0) {
        float ts = 1e6f;
        if (prim >= 0) ts = smin(ts, t);
        if (li >= 0) ts = smin(ts, lt);
        for (int k = 0; k < sc.num_volumes && k < 4; ++k) {
            float te, tx;
            if (ray_aabb_segment(o, d, ts, sc.volumes[k], te, tx)) { c += 8; break; }
        }
    }
    return c;
}

// Cell of a surface hit point: its Morton index in the kCellDim^3 grid over
// the scene box, so that neighbouring bins hold neighbouring cells.  Paths
// shaded in bin order hand the trace and shadow kernels rays whose origins
// lie close together (neighbouring lanes then walk similar BVH nodes).
LD int bin_cell(const DevScene& sc, V3 p) {
    const float c[3] = {p.x, p.y, p.z};
    int m = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        int q = (int)((c[a] - sc.bin_lo[a]) * sc.bin_scale[a]);
        q = min(max(q, 0), kCellDim - 1);
#pragma unroll
        for (int b = 0; b < kCellBits; ++b) m |= ((q >> b) & 1) << (3 * b + a);
    }
    return m;
}

// Per-block histogram of the shading bins of the rays a trace kernel
// finished, flushed to the depth's bin counters when the block ends.  bins
// < 0: no binning; else a set of kBin* flags: the volume bit of the class,
// and the hit-point cell (without it every ray of a class takes cell 0).
// The cells pay off on large waves only: each block flushes up to kBins
// counters, which a small wave (a few thousand rays per block) does not
// amortise (a 256x256 16-spp Cornell render: 546 M samples/s without the
// cells, 478 M with them; the 1M-triangle 1080p frame gains 1.5 % with
// them).
constexpr int kBinVolume = 1, kBinCells = 2;
constexpr long long kCellBinPaths = 1LL << 24;   // waves from this size on use the cells
struct BinHist {
    int* h;
    LD void clear() {
        for (int i = threadIdx.x; i < kBins; i += blockDim.x) h[i] = 0;
        __syncthreads();
    }
    // `at`: the ray's place in the queue
    LD void add(const DevScene& sc, const PathView& pv, int at, int bins, int prim, float t, int li, float lt, V3 o,
                V3 d) {
        const int c = bin_class(sc, prim, t, li, lt, o, d, (bins & kBinVolume) != 0);
        const int key = c * kCells + ((bins & kBinCells) && (c & 7) != 0 ? bin_cell(sc, o + d * t) : 0);
        pv.cls[at] = (unsigned short)key;
        atomicAdd(&h[key], 1);
    }
    LD void flush(int* cnt) {
        __syncthreads();
        for (int i = threadIdx.x; i < kBins; i += blockDim.x)
            if (h[i]) atomicAdd(&cnt[8 + i], h[i]);
    }
};

// Camera rays, generated and traced in one pass: neighbouring pixels trace
// similar paths, so a warp claims 32 consecutive rays at a time and keeps
// them together.  Also publishes the wave's path count as the depth-0 queue
// length for the kernels after it.
template <bool FMA>
__global__ void __launch_bounds__(128) k_trace_primary_t(DevScene sc, FrameParams f, PathView pv, int* cnt,
                                                       int records, int bins) {
    __shared__ int hist[kBins];
    BinHist bh{hist};
    bh.clear();
    const int n = f.n_wave;
    if (blockIdx.x == 0 && threadIdx.x == 0) cnt[0] = n;
    const V3 o = v3(f.pos[0], f.pos[1], f.pos[2]);
    // a warp traces the 8 x 4 pixels of one screen tile (one sample each):
    // a compact footprint keeps its lanes on the same BVH nodes longer than
    // a 32-pixel row.  Slots run over the tiles of the first sample, then of
    // the next; lanes past the tile's edge idle.
    const int tiles_x = (f.tile_w + 7) / 8, tiles_y = (f.tile_h + 3) / 4;
    const long long per_sample = (long long)tiles_x * tiles_y * 32;
    const long long slots = per_sample * (long long)(n / max(f.npix, 1));
    const int lane = (int)lane_id();
    bool ok = true;
    for (;;) {
        const int base = warp_fetch(&cnt[2]);
        if (base >= slots) break;
        const long long slot = (long long)base + lane;
        const int sl = (int)(slot / per_sample), tile = (int)((slot % per_sample) >> 5);
        const int px = (tile % tiles_x) * 8 + (lane & 7), py = (tile / tiles_x) * 4 + (lane >> 3);
        if (slot >= slots || px >= f.tile_w || py >= f.tile_h) continue;
        const int id = sl * f.npix + py * f.tile_w + px;
        const V3 d = camera_ray(f, pv, id);
        HitRec h = closest_skip_boundaries<FMA>(sc, o, d, 0.0f, ok);
        if (h.prim < 0) { h.t = 1e30f; h.u = 0.0f; h.v = 0.0f; }
        pv.hit[id].hit = make_float4(h.t, h.u, h.v, __int_as_float(h.prim));
        pv.hit[id].light = make_float4(__int_as_float(-1), 1e30f, 0.f, 0.f);   // lights are invisible to camera rays
        bh.add(sc, pv, id, bins, h.prim, h.t, -1, 1e30f, o, d);
        if (records) {
            int4 pi = h.prim >= 0 ? sc.prim_info[h.prim] : make_int4(-1, -1, -1, 0);
            pv.rec_prim[id] = make_int2(pi.x, pi.y);
            pv.rec_cnt[id].x += 1;
            unsigned long long hs = pv.rec_hash[id];
            hs = hpush(hs, (uint32_t)pi.x);
            hs = hpush(hs, (uint32_t)pi.y);
            hs = hpush(hs, 0xffffffffu);
            pv.rec_hash[id] = hs;
        }
    }
    bh.flush(cnt);
    if (!ok) atomicAdd(&pv.errors[0], 1);
}

// Camera rays take the FMA slab test when the camera lies within the
// scene's coordinate bound (its error analysis then holds as for secondary
// rays), else the subtraction form.
using PrimaryKernel = void (*)(DevScene, FrameParams, PathView, int*, int, int);
static PrimaryKernel k_trace_primary_for(const DevScene& sc, const float pos[3]) {
    const float m = std::max(std::fabs(pos[0]), std::max(std::fabs(pos[1]), std::fabs(pos[2])));
    return m <= sc.coord_bound ? k_trace_primary_t<true> : k_trace_primary_t<false>;
}

// ---------------------------------------------------------------- batched jobs
// One entry of the device job table of a batch wave: a piece of one job (a
// range of its samples) with its camera and image (f: s0 = the piece's first
// sample, n_wave = its paths), the scene it renders (index into the wave's
// scene table), where its paths start in the wave, and where its camera-ray
// slots start (each piece has whole warps of slots: 8 x 4 pixel tiles per
// sample).
struct BatchJob {
    FrameParams f;
    int sid;
    int path_base;
    int slot_base;
    int pad;
};
constexpr int kMaxBatchPieces = 1024;

// Camera rays of a batch wave, generated and traced in one pass over every
// piece: a warp's 32 slots lie in one piece (found by binary search over the
// slot bases, staged in shared memory), whose camera and sample range give
// the rays and whose scene the rays are traced in.  Each path's scene index
// is stored for the kernels after this one.  The subtraction form of the
// slab test is used throughout (the FMA form's error bound needs the camera
// inside its scene's coordinate bound, which varies from job to job); both
// give the same hits.
__global__ void __launch_bounds__(128) k_trace_primary_batch(PathView pv, const BatchJob* jobs, int njobs, int slots,
                                                           int n, int* cnt, int bins) {
    __shared__ int hist[kBins];
    __shared__ int sbase[kMaxBatchPieces];
    for (int i = threadIdx.x; i < njobs; i += blockDim.x) sbase[i] = jobs[i].slot_base;
    BinHist bh{hist};
    bh.clear();   // ends with a block barrier, which also publishes sbase
    if (blockIdx.x == 0 && threadIdx.x == 0) cnt[0] = n;
    const int lane = (int)lane_id();
    bool ok = true;
    for (;;) {
        const int base = warp_fetch(&cnt[2]);
        if (base >= slots) break;
        int lo = 0, hi = njobs - 1;   // the last piece whose slots start at or before base
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (sbase[mid] <= base) lo = mid; else hi = mid - 1;
        }
        const BatchJob& J = jobs[lo];
        const FrameParams& f = J.f;
        const int tw = f.tile_w, th = f.tile_h;
        const int tiles_x = (tw + 7) / 8, tiles_y = (th + 3) / 4;
        const int per_sample = tiles_x * tiles_y * 32;
        const int slot = base - sbase[lo] + lane;
        const int sl = slot / per_sample, tile = (slot % per_sample) >> 5;
        const int px = (tile % tiles_x) * 8 + (lane & 7), py = (tile / tiles_x) * 4 + (lane >> 3);
        if (px >= tw || py >= th) continue;
        const int local = sl * f.npix + py * tw + px;
        const int id = J.path_base + local;
        const int sid = J.sid;
        const DevScene& sc = pv.scenes[sid];
        const V3 d = camera_ray_at(f, pv, local, id);
        const V3 o = v3(f.pos[0], f.pos[1], f.pos[2]);
        pv.sid[id] = (unsigned short)sid;
        HitRec h = closest_skip_boundaries<false>(sc, o, d, 0.0f, ok);
        if (h.prim < 0) { h.t = 1e30f; h.u = 0.0f; h.v = 0.0f; }
        pv.hit[id].hit = make_float4(h.t, h.u, h.v, __int_as_float(h.prim));
        pv.hit[id].light = make_float4(__int_as_float(-1), 1e30f, 0.f, 0.f);   // lights are invisible to camera rays
        bh.add(sc, pv, id, bins, h.prim, h.t, -1, 1e30f, o, d);
    }
    bh.flush(cnt);
    if (!ok) atomicAdd(&pv.errors[0], 1);
}

// The scene of path `id`: the kernel's scene, or in a batch wave the entry
// of the wave's scene table the path's camera ray chose.
template <bool MULTI>
LD const DevScene& path_scene(const DevScene& sc, const PathView& pv, int id) {
    if constexpr (MULTI) return pv.scenes[id >= 0 ? pv.sid[id] : 0];
    else return sc;
}

// Closest BVH hit of extension rays (persistent, dynamic refill).  A round
// ends with few of a warp's rays done (two lanes of 32 on the 1M-triangle
// scene), so nothing but the traversal happens here: what a finished ray
// needs besides — the triangles kept out of the BVH, volume boundaries,
// native lights, its shading bin — is k_trace_post's, with every lane at
// work.  (All of it at the end of a ray, in here: 65.6 ms a frame on that
// scene.)
template <int MINB, bool MULTI = false>
__global__ void __launch_bounds__(128, MINB) k_trace_lb(DevScene sc0, PathView pv, int* cnt, int stop) {
    const int n = *(volatile int*)&cnt[0];
    if (n <= stop) return;   // left to k_paths (see WavePlan)
    const int* q = pv.q0;
    int2 stack[kStack];
    Trav s;
    trav_none(s);
    bool exhausted = false, ok = true;
    int id = -1, sid = 0;
    // the lane's scene: the kernel's, or in a batch wave its ray's entry of
    // the wave's scene table (kept in a register between refills)
    auto scene = [&]() -> const DevScene& {
        if constexpr (MULTI) return pv.scenes[sid];
        else return sc0;
    };
    for (;;) {
        const unsigned idle = __ballot_sync(0xffffffffu, id < 0);
        if (__popc(idle) >= kRefill && !exhausted) {
            const int r = warp_refill(&cnt[2], n, idle, exhausted);
            if (r >= 0) {
                id = q[r];
                if constexpr (MULTI) sid = pv.sid[id];
                const float4 ro = pv.st[id].ray_o, rd = pv.st[id].ray_d;
                trav_begin<false, false>(s, scene(), f3(ro), f3(rd), ro.w, 1e30f);
            }
        } else if (idle == 0xffffffffu) {
            break;
        }
        warp_step(s, __popc(__ballot_sync(0xffffffffu, id >= 0)), stack, scene(), ok);
        if (id >= 0 && trav_done(s)) {
            pv.hit[id].hit = make_float4(s.h.t, s.h.u, s.h.v, __int_as_float(s.h.prim));
            id = -1;
        }
    }
    if (!ok) atomicAdd(&pv.errors[0], 1);
}

// The rest of a closest-hit query, one ray a lane in queue order: from the
// closest BVH hit to the hit beyond the volume boundaries
// (path_tracer.hpp:82-95), the native light in front of it, the shading bin
// and the block's bin histogram.  `traced` 0: the scene has no BVH and
// k_trace_lb did not run.
constexpr int kPostThreads = 256;
template <bool MULTI>
__global__ void __launch_bounds__(kPostThreads) k_trace_post(DevScene sc0, PathView pv, int* cnt, int stop, int traced,
                                                             int records, int bins) {
    __shared__ int hist[kBins];
    const int n = *(volatile int*)&cnt[0];
    if (n <= stop) return;
    BinHist bh{hist};
    bh.clear();
    bool ok = true;
    for (int i = blockIdx.x * kPostThreads + threadIdx.x; i < n; i += gridDim.x * kPostThreads) {
        const int id = pv.q0[i];
        const DevScene& sc = path_scene<MULTI>(sc0, pv, id);
        const float4 ro = pv.st[id].ray_o, rd = pv.st[id].ray_d;
        const V3 o = f3(ro), d = f3(rd);
        HitRec real;
        real.t = 1e30f; real.u = real.v = 0.0f; real.prim = -1;
        if (traced) {
            const float4 h = pv.hit[id].hit;
            real.t = h.x; real.u = h.y; real.v = h.z; real.prim = __float_as_int(h.w);
        }
        if (sc.num_big_tris) list_closest(sc.big_tris, sc.num_big_tris, o, d, ro.w, real);
        HitRec res = real;
        if (sc.num_bnd_tris) {
            const V3 inv = v3(1.0f / d.x, 1.0f / d.y, 1.0f / d.z);
            float search = ro.w;
            for (int peek = 0;;) {
                HitRec b = real;
                if (real.prim < 0) b.t = 1e30f;
                boundary_closest<true>(sc, o, d, inv, search, b);
                if (b.prim < 0) { res.prim = -1; break; }
                if (b.prim == real.prim) { res = real; break; }
                search = b.t + 1e-3f;
                if (++peek == 8) { res.prim = -1; break; }
                if (real.prim >= 0 && real.t < search) {
                    // the surface lies within the skipped millimetre: look again behind it
                    real.t = 1e30f; real.u = real.v = 0.0f; real.prim = -1;
                    ok &= bvh_closest<true>(sc, o, d, search, real);
                }
            }
        }
        if (res.prim < 0) { res.t = 1e30f; res.u = 0.0f; res.v = 0.0f; }
        float lt = 1e30f;
        // a native light counts only in front of the surface hit (the shading
        // kernel's `lh.y < hh.x`): lights beyond it are not tested
        const int li = native_lights_closest(sc, o, d, res.t, lt);
        pv.hit[id].hit = make_float4(res.t, res.u, res.v, __int_as_float(res.prim));
        pv.hit[id].light = make_float4(__int_as_float(li), lt, 0.f, 0.f);
        bh.add(sc, pv, i, bins, res.prim, res.t, li, lt, o, d);
        if (records) {
            const int4 pi = res.prim >= 0 ? sc.prim_info[res.prim] : make_int4(-1, -1, -1, 0);
            pv.rec_cnt[id].x += 1;
            unsigned long long hs = pv.rec_hash[id];
            hs = hpush(hs, (uint32_t)pi.x);
            hs = hpush(hs, (uint32_t)pi.y);
            hs = hpush(hs, (uint32_t)li);
            pv.rec_hash[id] = hs;
        }
    }
    bh.flush(cnt);
    if (!ok) atomicAdd(&pv.errors[0], 1);
}

// ---------------------------------------------------------------- shade
// Adds a radiance contribution c (already weighted by the path throughput)
// to the training records of the path's guided vertices from slot `from` on
// (c / throughput-after-vertex = radiance that arrived along its sample).
LD void guide_credit(const PathView& pv, int id, RGB c, int from) {
    int4 s = pv.gslot[id];
    const int r[3] = {s.x, s.y, s.z};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        if (k < from || r[k] < 0) continue;
        float4 iv = pv.ginv[3 * id + k];
        GuideRec& g = pv.grec[r[k]];
        g.L[0] += c.r * iv.x; g.L[1] += c.g * iv.y; g.L[2] += c.b * iv.z;
    }
}

// Hit UV (bvh.hpp:67-72): the triangle's UVs at the hit's barycentrics,
// (0, 0) when it has none.
LD void hit_uv(const DevScene& sc, int prim, float bu, float bv, float& su, float& sv) {
    su = 0.0f;
    sv = 0.0f;
    if (!sc.prim_uv) return;
    const float4 a = sc.prim_uv[2 * prim], b = sc.prim_uv[2 * prim + 1];
    if (b.z == 0.0f) return;
    const float w = 1.0f - bu - bv;
    su = a.x * w + a.z * bu + b.x * bv;
    sv = a.y * w + a.w * bu + b.y * bv;
}

// A material node program (the loader's folding, lucid_nodes.cpp, in the
// same float operations) at (u, v).  Out of line: only textured materials
// run it, and its step array stays out of the shading kernels' frames.
static __device__ __noinline__ RGB tex_eval(const float4* ops, int start, int n, float u, float v) {
    float val[kTexMaxOps][3];
    n = min(n, kTexMaxOps);
    for (int i = 0; i < n; ++i) {
        const float4 s0 = ops[2 * (start + i)], s1 = ops[2 * (start + i) + 1];
        const int kind = __float_as_int(s0.x), a = __float_as_int(s0.y), b = __float_as_int(s0.z);
        const float k = s0.w;
        if (kind == TEX_CONST) {
            val[i][0] = s1.x; val[i][1] = s1.y; val[i][2] = s1.z;
        } else if (kind == TEX_CHECKER) {   // node_evaluator.cpp:385-396
            int cu = (int)floorf(u * k) % 2, cv = (int)floorf(v * k) % 2;
            if (cu < 0) cu += 2;
            if (cv < 0) cv += 2;
            const int src = (cu + cv) % 2 == 0 ? a : b;
            for (int c = 0; c < 3; ++c) val[i][c] = val[src][c];
        } else if (kind == TEX_MIX) {
            for (int c = 0; c < 3; ++c) val[i][c] = val[a][c] * (1.0f - k) + val[b][c] * k;
        } else {
            for (int c = 0; c < 3; ++c) val[i][c] = val[a][c] * k;
        }
    }
    return n > 0 ? rgb(val[n - 1][0], val[n - 1][1], val[n - 1][2]) : rgb(0.0f, 0.0f, 0.0f);
}

// Albedo and emission of a textured material at the hit (getMaterialParams
// / getEmission, integrator/path_tracer.hpp:45-72); the other parameters
// are constants of the material.
LD void apply_textures(const DevScene& sc, const DevMaterial& dm, int prim, float bu, float bv, RGB& albedo, RGB& em,
                       bool& has_em) {
    if (!(__float_as_int(dm.rough_trans_ior_flags.w) & MAT_TEXTURED)) return;
    float u, v;
    hit_uv(sc, prim, bu, bv, u, v);
    if (dm.program.y > 0) albedo = tex_eval(sc.tex_ops, dm.program.x, dm.program.y, u, v);
    if (dm.program.w > 0) {
        em = tex_eval(sc.tex_ops, dm.program.z, dm.program.w, u, v);
        has_em = (0.2126f * em.r + 0.7152f * em.g + 0.0722f * em.b) > 1e-6f;
    }
}

// A surface the guide may sample: no transmission lobe and not the
// near-delta metal that sample_bsdf weights in closed form.
LD bool guide_eligible(const DevMaterial& dm) {
    float rough = smax(dm.rough_trans_ior_flags.x, MIN_ROUGHNESS);
    return dm.rough_trans_ior_flags.y == 0.0f && !(rough < 0.05f && dm.albedo_metallic.w > 0.5f);
}

// A path between two segments: the ray to trace next (its depth counts the
// segments before it), throughput, pdf of the sampler that chose the ray and
// the RNG stream.
struct PathRegs {
    V3 o, d;
    RGB T;
    float last_pdf;
    int depth;
    Rng rng;
};
// A light sample waiting for its shadow ray.
struct ShadowRay {
    V3 o, d;
    float len;
    RGB inc;
    int pushed;   // the first guide slot the contribution credits (a vertex's
                  // own light sample did not arrive along its sampled direction)
};
struct ShadeResult {
    bool cont, shadow;
    RGB add;      // radiance of the event (zero: none)
};
struct BlockSync {
    LD void operator()() const { __syncthreads(); }
};

// One path segment on a path held in registers: the closest hit hh = (t, u,
// v, prim) and the native-light hit lh = (index, t) of its ray give the
// radiance of this event (add), the light sample (sr, when `shadow` is set)
// and, when `cont` is set, the next ray (o, d, depth) of the path.
//
// The segment runs in phases — medium, hit and emission, light sample,
// direction sample — with `sync` between them, which every lane reaches
// whatever became of its path (`live`: the lane has one).  k_shade passes a
// block barrier: the code of a segment is far larger than an SM's
// instruction caches near the schedulers, and warps that march through it
// together share every fetched line.  Events of one phase share code where
// they do the same operations on the same operands (the light sample of a
// medium scatter and of a surface, the two reflection lobes' directions,
// values and pdfs), which shortens the code and keeps more lanes together.
template <int ALGO, bool GUIDE, class Sync>
LD ShadeResult shade_segment(const DevScene& sc, bool live, int max_depth, bool records, const PathView& pv, int id,
                             PathRegs& ps, const float4 hh, const float2 lh, ShadowRay& sr, Sync sync) {
    constexpr int algo = ALGO;
    constexpr bool nee = algo == ALGO_NEE || algo == ALGO_MIS || algo == ALGO_VOLUME_MIS;
    constexpr bool mis = algo == ALGO_MIS || algo == ALGO_VOLUME_MIS;
    ShadeResult out;
    out.cont = false;
    out.shadow = false;
    out.add = rgb(0.f, 0.f, 0.f);
    const int depth = ps.depth;
    const int prim = __float_as_int(hh.w), lidx = __float_as_int(lh.x);
    const bool has_hit = prim >= 0, has_lh = lidx >= 0;
    RGB T = ps.T;
    float last_pdf = ps.last_pdf;
    const V3 wo = -ps.d;
    V3 p = ps.o;
    int vi = -1;   // the volume the path scatters in before its hit

    // ---- medium
    if (algo == ALGO_VOLUME_SIMPLE && live) {
        float ts = 1e6f;
        if (has_hit) ts = smin(ts, hh.x);
        if (has_lh) ts = smin(ts, lh.y);
        T = mul(T, volume_transmittance(sc, ps.o, ps.d, ts, false));
    }
    if (algo == ALGO_VOLUME_MIS && live) {
        float ts = 1e6f;
        if (has_hit) ts = smin(ts, hh.x);
        if (has_lh) ts = smin(ts, lh.y);
        float vt = 0.0f;
        vi = sample_volume_distance(sc, ps.o, ps.d, ts, ps.rng, vt);
        if (records) pv.rec_hash[id] = hpush(pv.rec_hash[id], vi >= 0 ? 1u : 0u);
        if (vi >= 0) {
            // scatter event (path_tracer.hpp:616-700)
            const DevVolume& v = sc.volumes[vi];
            T = mul(T, rgb(v.color[0] / (1.0f + v.absorption[0]), v.color[1] / (1.0f + v.absorption[1]),
                           v.color[2] / (1.0f + v.absorption[2])));
            p = ps.o + ps.d * vt;
        }
    }
    sync();

    // ---- hit and emission
    const bool scat = algo == ALGO_VOLUME_MIS && vi >= 0;
    bool surf = false, has_em = false, guided = false;
    V3 n = wo, sn = wo;
    Mat m;
    m.albedo = rgb(0.f, 0.f, 0.f);
    m.metallic = m.transmission = 0.0f;
    m.roughness = m.ior = 1.0f;
    if (live && !scat) {
        if (has_lh && (!has_hit || lh.y < hh.x)) {
            // native light hit (path_tracer.hpp:429-452)
            const DevLight& L = sc.lights[sc.native_start + lidx];
            RGB em = c3(L.emission_radius);
            if (mis) {
                float lpdf = 0.0f;
                if (sc.num_lights > 0) {
                    float sp = area_ratio(L.normal_area.w, sc.total_light_area);
                    if (sp > 0.0f) {
                        V3 lp = ps.o + ps.d * lh.y;
                        V3 ln = (__float_as_int(L.pos_type.w) == LIGHT_POINT) ? normalize_nz(lp - f3(L.pos_type))
                                                                              : f3(L.normal_area);
                        lpdf = pdf_light(L.normal_area.w, ps.o, lp, ln) * sp;
                    }
                }
                float mw = (last_pdf > MIN_PDF && lpdf > MIN_PDF) ? mis_power(last_pdf, lpdf) : 1.0f;
                out.add = mul(T, em) * mw;
            } else {
                out.add = mul(T, em);
            }
            if (GUIDE) guide_credit(pv, id, out.add, 0);
        } else if (!has_hit) {
            out.add = mul(T, rgb(sc.env[0], sc.env[1], sc.env[2]));
            if (GUIDE) guide_credit(pv, id, out.add, 0);
        } else {
            // surface hit: point and normal from (t, u, v, prim) as in bvh.hpp:108-128
            surf = true;
            p = ps.o + ps.d * hh.x;
            int4 pi = sc.prim_info[prim];
            V3 fn = f3(sc.prim_fn[prim]);
            n = fn;
            if (pi.w) {
                float u = hh.y, v = hh.z;
                float w = 1.0f - u - v;
                V3 ni = f3(sc.prim_vn[3 * prim]) * w + f3(sc.prim_vn[3 * prim + 1]) * u + f3(sc.prim_vn[3 * prim + 2]) * v;
                n = make_dir_or(ni, fn);
            }
            const DevMaterial& dm = sc.materials[pi.x];
            m.albedo = c3(dm.albedo_metallic);
            m.metallic = dm.albedo_metallic.w;
            m.roughness = smax(dm.rough_trans_ior_flags.x, MIN_ROUGHNESS);
            m.transmission = dm.rough_trans_ior_flags.y;
            m.ior = dm.rough_trans_ior_flags.z;
            RGB em = c3(dm.emission);
            has_em = dm.emission.w != 0.0f;
            apply_textures(sc, dm, prim, hh.y, hh.z, m.albedo, em, has_em);
            sn = n;
            if (m.transmission < 0.5f && !(dot(wo, n) > 0)) sn = -n;
            if (!nee) {
                out.add = mul(T, em);
            } else if (!mis) {
                if (has_em && depth == 0) out.add = mul(T, em);
            } else if (has_em) {
                float mw = 1.0f;
                if (sc.num_lights > 0 && last_pdf > MIN_PDF && pi.z >= 0) {
                    const DevLight& L = sc.lights[pi.z];
                    float sp = area_ratio(L.normal_area.w, sc.total_light_area);
                    if (sp > 0.0f) {
                        float lpdf = pdf_light(L.normal_area.w, ps.o, p, n) * sp;
                        if (lpdf > MIN_PDF) mw = mis_power(last_pdf, lpdf);
                    }
                }
                out.add = mul(T, em) * mw;
                if (GUIDE) guide_credit(pv, id, out.add, 0);
            }
            guided = GUIDE && depth < pv.gdepth && guide_eligible(dm);
        }
    }
    sync();

    // ---- light sample, at a surface or at a scatter point
    const float* gm = GUIDE ? pv.gmix + (size_t)id * kGMixFloats : nullptr;
    if (nee && sc.num_lights > 0 && (scat || (surf && !has_em && !(m.transmission > 0.5f)))) {
        float usel = randf(ps.rng);
        const DevLight& L = sc.lights[select_light(sc, usel)];
        float lsp = area_ratio(L.normal_area.w, sc.total_light_area);
        if (lsp > 1e-6f) {
            float u1 = randf(ps.rng), u2 = randf(ps.rng);
            LightSample ls = sample_light(L, p, u1, u2);
            if (ls.pdf > MIN_PDF) {
                const float pl = ls.pdf * lsp;
                float nl = 1.0f, pb = 0.0f;
                RGB fb = rgb(0.f, 0.f, 0.f);
                if (scat) {
                    pb = hg_eval(sc.volumes[vi].anisotropy, dot(wo, ls.dir));
                    fb = rgb(pb, pb, pb);
                } else {
                    nl = dot(sn, ls.dir);
                    if (nl > 1e-6f) fb = eval_bsdf<mis>(m, wo, ls.dir, sn, nl, pb);
                }
                if (nl > 1e-6f) {
                    RGB c = bsdf_weight(fb, nl, pl);
                    if (mis) {
                        if (guided) pb = 0.5f * pb + 0.5f * guide_pdf_c(gm, ls.dir);
                        c = c * mis_power(pl, pb);
                    }
                    if (algo == ALGO_VOLUME_MIS) {
                        RGB Tsh = volume_transmittance(sc, p, ls.dir, ls.dist, true);
                        c = mul(c, mul(Tsh, ls.emission));
                    } else {
                        c = mul(c, ls.emission);
                    }
                    sr.inc = mul(T, c);
                    sr.o = p;
                    sr.d = ls.dir;
                    sr.len = ls.dist;
                    out.shadow = true;
                }
            }
        }
    }
    sync();

    // ---- next direction
    V3 wi = wo;
    float gpdf = 0.0f;
    if (scat) {
        float u1 = randf(ps.rng), u2 = randf(ps.rng);
        wi = hg_sample(sc.volumes[vi].anisotropy, wo, u1, u2, last_pdf);
        out.cont = true;
    } else if (surf) {
        const V3 smp_n = (m.transmission > 0.5f) ? n : sn;
        float usel = 0.0f;
        if (guided) usel = randf(ps.rng);
        float u1 = randf(ps.rng), u2 = randf(ps.rng), u3 = randf(ps.rng);
        if (guided) {
            // one-sample MIS of BSDF and guide sampling, 1/2 each (balance heuristic)
            if (usel < 0.5f) wi = sample_bsdf(m, wo, smp_n, u1, u2, u3, ps.rng).wi;
            else wi = guide_sample_c(gm, u1, u2, u3);
            float c = dot(smp_n, wi);
            if (!(c <= 1e-6f)) {
                float pb;
                RGB f = eval_bsdf<true>(m, wo, wi, smp_n, c, pb);
                gpdf = 0.5f * pb + 0.5f * guide_pdf_c(gm, wi);
                if (gpdf > MIN_PDF) {
                    T = mul(T, bsdf_weight(f, c, gpdf));
                    last_pdf = gpdf;
                    out.cont = true;
                }
            }
        } else {
            BsdfSample bs = sample_bsdf(m, wo, smp_n, u1, u2, u3, ps.rng);
            RGB w = bs.f;
            out.cont = true;
            if (bs.kind != BS_PRECOMP) {
                float c = fabsf(dot(smp_n, bs.wi));
                if (!(bs.pdf > MIN_PDF) || c <= 1e-6f) out.cont = false;
                else w = bsdf_weight(bs.f, c, bs.pdf);
            }
            T = mul(T, w);
            if (mis) last_pdf = (bs.kind == BS_EVAL) ? bs.pdf : 0.0f;
            wi = bs.wi;
        }
    }
    if (out.cont && depth >= 3) {
        float rr = smin(smax3(T.r, T.g, T.b), 0.95f);
        if (randf(ps.rng) > rr) out.cont = false;
        else T = T * (1.0f / rr);
    }
    if (!rgb_valid(T)) out.cont = false;
    int pushed = 0;
    if (GUIDE && guided && out.cont) {
        // warp-aggregated counters: guided vertices, then record slots
        unsigned am = __activemask();
        int leader = __ffs(am) - 1;
        if ((int)lane_id() == leader) atomicAdd(&pv.gcount[1], __popc(am));
        unsigned hsh = murmur3_finalize((unsigned)id * 0x9E3779B9u ^ (unsigned)(depth + 1) * 0x85EBCA6Bu);
        if (hsh < pv.gkeep) {
            unsigned km = __activemask();
            int kl = __ffs(km) - 1, rb = 0;
            if ((int)lane_id() == kl) rb = atomicAdd(&pv.gcount[0], __popc(km));
            int r = __shfl_sync(km, rb, kl) + __popc(km & lanemask_lt());
            if (r < pv.gcap) {
                GuideRec g;
                g.p[0] = (p.x - pv.glo[0]) * pv.gscale[0];
                g.p[1] = (p.y - pv.glo[1]) * pv.gscale[1];
                g.p[2] = (p.z - pv.glo[2]) * pv.gscale[2];
                g.n[0] = n.x; g.n[1] = n.y; g.n[2] = n.z;
                g.wo[0] = wo.x; g.wo[1] = wo.y; g.wo[2] = wo.z;
                g.wi[0] = wi.x; g.wi[1] = wi.y; g.wi[2] = wi.z;
                g.pdf = gpdf;
                g.L[0] = g.L[1] = g.L[2] = 0.0f;
                pv.grec[r] = g;
                int4 sl = pv.gslot[id];
                pv.gslot[id] = make_int4(r, sl.x, sl.y, -1);
                pv.ginv[3 * id + 2] = pv.ginv[3 * id + 1];
                pv.ginv[3 * id + 1] = pv.ginv[3 * id];
                pv.ginv[3 * id] = make_float4(T.r > 0.0f ? 1.0f / T.r : 0.0f, T.g > 0.0f ? 1.0f / T.g : 0.0f,
                                              T.b > 0.0f ? 1.0f / T.b : 0.0f, 0.0f);
                pushed = 1;
            }
        }
    }
    sr.pushed = pushed;
    if (depth + 1 >= max_depth) out.cont = false;
    if (out.cont) {
        ps.T = T;
        ps.last_pdf = last_pdf;
        ps.o = p;
        ps.d = wi;
        ps.depth = depth + 1;
    }
    return out;
}

// The same on the wavefront's path state: reads path `id` (-1: the lane has
// none), shades it, writes back what changed and queues its shadow ray.
template <int ALGO, bool GUIDE>
LD ShadeResult shade_path(const DevScene& sc, const FrameParams& f, const PathView& pv, int id, int* nshadow) {
    const bool live = id >= 0;
    PathRegs ps;
    ps.o = ps.d = v3(0.f, 0.f, 1.f);
    ps.T = rgb(0.f, 0.f, 0.f);
    ps.last_pdf = 0.0f;
    ps.depth = 0;
    ps.rng.state = ps.rng.inc = 0;
    float4 hh = make_float4(0.f, 0.f, 0.f, __int_as_float(-1));
    float2 lh = make_float2(__int_as_float(-1), 0.f);
    if (live) {
        const PathState& st = pv.st[id];
        ps.o = f3(st.ray_o);
        const float4 rd = st.ray_d;
        ps.d = f3(rd);
        ps.depth = __float_as_int(rd.w);
        const float4 th = st.thr;
        ps.T = c3(th);
        ps.last_pdf = th.w;
        const ulonglong2 rs = st.rng;
        ps.rng.state = rs.x;
        ps.rng.inc = rs.y;
        hh = pv.hit[id].hit;
        const float4 l = pv.hit[id].light;
        lh = make_float2(l.x, l.y);
    }
    ShadowRay sr;
    const ShadeResult out =
        shade_segment<ALGO, GUIDE>(sc, live, f.max_depth, f.records != 0, pv, id, ps, hh, lh, sr, BlockSync());
    if (out.add.r != 0.0f || out.add.g != 0.0f || out.add.b != 0.0f) {
        const float4 ra = pv.rad[id];
        pv.rad[id] = make_float4(ra.x + out.add.r, ra.y + out.add.g, ra.z + out.add.b, 0.0f);
    }
    if (out.cont) {
        PathState& st = pv.st[id];
        st.ray_o = make_float4(ps.o.x, ps.o.y, ps.o.z, RAY_T_MIN);
        st.ray_d = make_float4(ps.d.x, ps.d.y, ps.d.z, __int_as_float(ps.depth));
        st.thr = make_float4(ps.T.r, ps.T.g, ps.T.b, ps.last_pdf);
        st.rng = make_ulonglong2(ps.rng.state, ps.rng.inc);
    }
    const int at = warp_append(nshadow, out.shadow);
    if (out.shadow) {
        ShadowRec& q = pv.sh[at];
        q.o = make_float4(sr.o.x, sr.o.y, sr.o.z, sr.len);
        q.d = make_float4(sr.d.x, sr.d.y, sr.d.z, __int_as_float(sr.pushed));
        q.c = make_float4(sr.inc.r, sr.inc.g, sr.inc.b, __int_as_float(id));
    }
    return out;
}

// A block takes 256 queue entries at a time and its eight warps go through
// shade_segment's phases together.  What bounds the kernel is instruction
// fetch (a segment runs some 2,800 warp instructions of straight-line code);
// in phase, eight warps share each fetched line.  The bench frame (1M
// triangles, 1080p, 64 spp, volume_mis, 265 M segments) shades in 43.1 ms,
// against 61.3 ms with warps fetching on their own and each event's code
// written out; 128 threads 45.5, 512 42.1, 1,024 46.7 ms.  Small waves lose
// from 512 threads on (an 800x600 1-spp frame: 307, 310, 327, 377 us for
// 128, 256, 512, 1,024; 403 us before), so every wave takes 256.
// MINB is the register cap: 128 * MINB threads per SM (8: 64 registers).
constexpr int kShadeThreads = 256;
template <int ALGO, bool GUIDE = false, int MINB = 8, bool MULTI = false>
__global__ void __launch_bounds__(kShadeThreads, MINB / 2) k_shade(DevScene sc, FrameParams f, PathView pv, int* cnt,
                                                         int* cnt_next, int stop, const int* qin, int* qout) {
    __shared__ int s_base[2];
    const int n = *(volatile int*)&cnt[0];
    if (n <= stop) return;
    for (int it = 0;; it ^= 1) {
        if (threadIdx.x == 0) s_base[it] = atomicAdd(&cnt[3], (int)blockDim.x);
        __syncthreads();
        const int base = s_base[it];
        if (base >= n) break;
        const int i = base + (int)threadIdx.x;
        const int id = i < n ? qin[i] : -1;
        const ShadeResult r = shade_path<ALGO, GUIDE>(path_scene<MULTI>(sc, pv, id), f, pv, id, &cnt[1]);
        const int at = warp_append(&cnt_next[0], r.cont);
        if (r.cont) qout[at] = id;
    }
}

using ShadeKernel = void (*)(DevScene, FrameParams, PathView, int*, int*, int, const int*, int*);
template <int MINB>
static ShadeKernel shade_kernel_lb(int algo, bool guide) {
    if (guide && algo == ALGO_MIS) return k_shade<ALGO_MIS, true, MINB>;
    switch (algo) {
        case ALGO_SIMPLE: return k_shade<ALGO_SIMPLE, false, MINB>;
        case ALGO_MIS: return k_shade<ALGO_MIS, false, MINB>;
        case ALGO_VOLUME_SIMPLE: return k_shade<ALGO_VOLUME_SIMPLE, false, MINB>;
        case ALGO_VOLUME_MIS: return k_shade<ALGO_VOLUME_MIS, false, MINB>;
        default: return k_shade<ALGO_NEE, false, MINB>;
    }
}
// Batch waves (unguided): each path shaded in its own job's scene.
static ShadeKernel shade_kernel_batch(int algo) {
    switch (algo) {
        case ALGO_SIMPLE: return k_shade<ALGO_SIMPLE, false, 8, true>;
        case ALGO_MIS: return k_shade<ALGO_MIS, false, 8, true>;
        case ALGO_VOLUME_SIMPLE: return k_shade<ALGO_VOLUME_SIMPLE, false, 8, true>;
        case ALGO_VOLUME_MIS: return k_shade<ALGO_VOLUME_MIS, false, 8, true>;
        default: return k_shade<ALGO_NEE, false, 8, true>;
    }
}

// ---------------------------------------------------------------- shading bins
// The scatter half of the counting sort whose histogram the trace kernels
// build (bin_class): paths of a bin are kept together so neighbouring warps
// shade the same kind of event.  A block takes kBinTile entries at a time,
// ranks them within their bins in shared memory and claims each bin's places
// with one global atomic; with one per bin and warp the few counters most
// paths go to were what the pass waited for (5.3 ms of the 1M-triangle
// 1920x1080, 64 spp frame, 1.4 ms this way).
constexpr int kBinThreads = 256, kBinItems = 8, kBinTile = kBinThreads * kBinItems;
static_assert(kBins % kBinThreads == 0, "bins per scatter thread");
__global__ void __launch_bounds__(kBinThreads) k_bin_scatter(PathView pv, int* cnt, int identity, int stop,
                                                             const int* qin, int* qb) {
    __shared__ int base[kBins];
    __shared__ int wsum[kBinThreads / 32];
    const int n = *(volatile int*)&cnt[0];
    if (n <= stop) return;
    {
        // exclusive prefix sum of the bin counts: kPer bins per thread, then a
        // block scan of the per-thread sums
        constexpr int kPer = kBins / kBinThreads;
        int loc[kPer], sum = 0;
#pragma unroll
        for (int j = 0; j < kPer; ++j) { loc[j] = sum; sum += cnt[8 + threadIdx.x * kPer + j]; }
        const int lane = (int)(threadIdx.x & 31), w = (int)(threadIdx.x >> 5);
        int x = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) wsum[w] = x;
        __syncthreads();
        int before = 0;
        for (int k = 0; k < w; ++k) before += wsum[k];
        const int excl = before + x - sum;
#pragma unroll
        for (int j = 0; j < kPer; ++j) base[threadIdx.x * kPer + j] = excl + loc[j];
    }
    __syncthreads();
    __shared__ int h[kBins];
    for (int i0 = blockIdx.x * kBinTile; i0 < n; i0 += gridDim.x * kBinTile) {
        for (int b = threadIdx.x; b < kBins; b += kBinThreads) h[b] = 0;
        __syncthreads();
        int id[kBinItems], key[kBinItems], rank[kBinItems];
#pragma unroll
        for (int j = 0; j < kBinItems; ++j) {
            const int i = i0 + j * kBinThreads + (int)threadIdx.x;
            key[j] = i < n ? (int)pv.cls[i] : -1;
            id[j] = i < n && !identity ? qin[i] : i;
        }
#pragma unroll
        for (int j = 0; j < kBinItems; ++j)
            if (key[j] >= 0) rank[j] = atomicAdd(&h[key[j]], 1);
        __syncthreads();
        for (int b = threadIdx.x; b < kBins; b += kBinThreads)
            if (h[b]) h[b] = base[b] + atomicAdd(&cnt[8 + kBins + b], h[b]);
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kBinItems; ++j)
            if (key[j] >= 0) qb[h[key[j]] + rank[j]] = id[j];
        __syncthreads();
    }
}

// ---------------------------------------------------------------- guide inference
// Raw guide outputs for every queued path whose next event is a guidable
// surface hit: 16 paths per warp-tile through the BF16 tensor-core MLP
// (16 warps per block, one block per SM), the weights staged once per block
// in shared memory.  Two lanes encode each path (lanes r and r + 16, half of
// the features each).
constexpr int kInferWarps = 16;
constexpr size_t kInferSmem = sizeof(GuideSmemW) + kInferWarps * sizeof(GuideLeanTile);

__global__ void __launch_bounds__(32 * kInferWarps, 1) k_guide_infer(DevScene sc, PathView pv, int* cnt, int identity,
                                                                     const int* qin, const __nv_bfloat16* wq,
                                                                     const float* master) {
    extern __shared__ __align__(16) unsigned char smem[];
    GuideSmemW& W = *reinterpret_cast<GuideSmemW*>(smem);
    GuideLeanTile* tiles = reinterpret_cast<GuideLeanTile*>(smem + sizeof(GuideSmemW));
    guide_load_weights(W, wq, master);
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rl = lane & 15, half = lane >> 4;
    GuideLeanTile& T = tiles[warp];
    const int n = *(volatile int*)&cnt[0];
    const int ntiles = (n + 15) / 16;
    for (int tile = blockIdx.x * kInferWarps + warp; tile < ntiles; tile += gridDim.x * kInferWarps) {
        int id = -1;
        bool elig = false;
        __nv_bfloat16* row = T.x + rl * kLdIn;
        const int i = tile * 16 + rl;
        if (i < n) {
            id = identity ? i : qin[i];
            float4 hh = pv.hit[id].hit;
            int prim = __float_as_int(hh.w);
            float4 lh = pv.hit[id].light;
            int li = __float_as_int(lh.x);
            if (prim >= 0 && !(li >= 0 && lh.y < hh.x)) {
                int4 pi = sc.prim_info[prim];
                elig = guide_eligible(sc.materials[pi.x]);
                if (elig) {
                    float4 ro = pv.st[id].ray_o, rd = pv.st[id].ray_d;
                    V3 o = f3(ro), d = f3(rd);
                    V3 p = o + d * hh.x;
                    V3 p01 = v3((p.x - pv.glo[0]) * pv.gscale[0], (p.y - pv.glo[1]) * pv.gscale[1],
                                (p.z - pv.glo[2]) * pv.gscale[2]);
                    V3 fn = f3(sc.prim_fn[prim]);
                    V3 nn = fn;
                    if (pi.w) {
                        float w = 1.0f - hh.y - hh.z;
                        V3 ni = f3(sc.prim_vn[3 * prim]) * w + f3(sc.prim_vn[3 * prim + 1]) * hh.y +
                                f3(sc.prim_vn[3 * prim + 2]) * hh.z;
                        nn = make_dir_or(ni, fn);
                    }
                    guide_encode_half(p01, nn, -d, half, [&](int k, float v) { row[k] = __float2bfloat16(v); });
                }
            }
        }
        if (!elig)
            for (int k = half * 88; k < half * 88 + 88; ++k) row[k] = __float2bfloat16(0.0f);
        __syncwarp();
        guide_forward_lean(W, T);
        // the compact mixture of each path, half by each of its two lanes
        if (elig) {
            float4 o[5];
            guide_compact_half(T.raw() + rl * kGOut, half, o);
            float4* dst = reinterpret_cast<float4*>(pv.gmix + (size_t)id * kGMixFloats);
#pragma unroll
            for (int k = 0; k < 4; ++k) dst[4 * half + k] = o[k];
            dst[8 + half] = o[4];
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------- shadow
// A shadow ray's verdict (is_shadowed_skipping_volume_boundaries,
// path_tracer.hpp:103-119): adds the light sample when unoccluded.
LD void shadow_done(const PathView& pv, int at, bool occ, int records) {
    if (!occ) {
        const float4 c = pv.sh[at].c;
        const int id = __float_as_int(c.w);
        const float4 ra = pv.rad[id];
        pv.rad[id] = make_float4(ra.x + c.x, ra.y + c.y, ra.z + c.z, 0.0f);
        if (pv.grec) guide_credit(pv, id, rgb(c.x, c.y, c.z), __float_as_int(pv.sh[at].d.w));
    }
    if (records) {
        const int id = __float_as_int(pv.sh[at].c.w);
        int4 rc = pv.rec_cnt[id];
        rc.y += 1;
        rc.z += occ ? 1 : 0;
        pv.rec_cnt[id] = rc;
        pv.rec_hash[id] = hpush(pv.rec_hash[id], 0x5EED0000u | (occ ? 1u : 0u));
    }
}

// What of a shadow ray needs no BVH, one ray a lane: the end of its first
// segment at the nearest volume boundary and the triangles kept out of the
// BVH.  Rays decided here are done; a ray that would add nothing (a spot
// light outside its cone) is dropped, unless per-sample records count it.  On
// the 1M-triangle 960x540 frame the two full-lane passes take 98 us (this)
// and 180 us (k_trace_post) of the 1.0 and 1.0 ms of shadow rays and closest
// hits.
// The others go to k_shadow_lb's queue (pv.q0, whose depth is shaded by now)
// with their segment's end (in the hit records, which are free until the
// next trace).
template <bool MULTI>
__global__ void __launch_bounds__(kPostThreads) k_shadow_pre(DevScene sc0, PathView pv, int* cnt, int records) {
    const int n = *(volatile int*)&cnt[1];
    float* const seg_end = reinterpret_cast<float*>(pv.hit);
    for (int i0 = blockIdx.x * kPostThreads; i0 < n; i0 += gridDim.x * kPostThreads) {
        const int at = i0 + (int)threadIdx.x;
        bool trace = false;
        float bt = -1.0f;
        if (at < n) {
            const float4 so = pv.sh[at].o, sd = pv.sh[at].d, c = pv.sh[at].c;
            const DevScene& sc = path_scene<MULTI>(sc0, pv, __float_as_int(c.w));
            if (records || c.x != 0.0f || c.y != 0.0f || c.z != 0.0f) {
                const V3 o = f3(so), d = f3(sd);
                const float rem = so.w;
                bool done = true, occ = false;
                if (!(rem <= 0.0f)) {
                    if (sc.num_bnd_tris) {
                        HitRec b; b.t = rem; b.u = 0.f; b.v = 0.f; b.prim = -1;
                        boundary_closest_all(sc, o, d, RAY_T_MIN, b);
                        if (b.prim >= 0) bt = b.t;
                    }
                    if (sc.num_big_tris)
                        occ = list_any(sc.big_tris, sc.num_big_tris, o, d, RAY_T_MIN, bt >= 0.0f ? bt : rem);
                    done = occ || (sc.num_bvh_tris == 0 && bt < 0.0f);
                }
                if (done) shadow_done(pv, at, occ, records);
                trace = !done;
            }
        }
        const int j = warp_append(&cnt[5], trace);
        if (trace) {
            pv.q0[j] = at;
            seg_end[j] = bt;
        }
    }
}

// Shadow rays over the BVH (persistent, dynamic refill); a segment ends at
// the nearest boundary-only hit, past which the probe advances 1 mm.  As for
// k_trace_lb, few lanes start or finish a ray at a time, so a ray's first
// segment is prepared by k_shadow_pre (in here: 46.9 ms a frame on the
// 1M-triangle scene).
template <int MINB, bool MULTI = false>
__global__ void __launch_bounds__(128, MINB) k_shadow_lb(DevScene sc0, PathView pv, int* cnt, int records) {
    const int n = *(volatile int*)&cnt[5];
    if (n == 0) return;
    const float* const seg_end = reinterpret_cast<const float*>(pv.hit);
    int stack[kStack];
    Trav s;
    trav_none(s);
    bool exhausted = false, ok = true;
    int at = -1, peek = 0, sid = 0;
    float tmax = 0.0f, off = 0.0f, bt = -1.0f;
    // the lane's scene (a batch wave: its ray's entry of the scene table)
    auto scene = [&]() -> const DevScene& {
        if constexpr (MULTI) return pv.scenes[sid];
        else return sc0;
    };
    for (;;) {
        const unsigned idle = __ballot_sync(0xffffffffu, at < 0);
        if (__popc(idle) >= kRefill && !exhausted) {
            const int r = warp_refill(&cnt[4], n, idle, exhausted);
            if (r >= 0) {
                at = pv.q0[r];
                bt = seg_end[r];
                if constexpr (MULTI) sid = pv.sid[__float_as_int(pv.sh[at].c.w)];
                const float4 so = pv.sh[at].o, sd = pv.sh[at].d;
                tmax = so.w; off = 0.0f; peek = 0;
                trav_begin<true, false>(s, scene(), f3(so), f3(sd), RAY_T_MIN, bt >= 0.0f ? bt : tmax);
            }
        } else if (idle == 0xffffffffu) {
            break;
        }
        warp_step_any(s, __popc(__ballot_sync(0xffffffffu, at >= 0)), stack, scene(), ok);
        if (at >= 0 && trav_done(s)) {
            const DevScene& sc = scene();
            bool occ = s.any_hit, next = false;
            if (!occ && bt >= 0.0f) {
                // skip past the boundary hit and start the next segment
                const float skip = bt + 1e-3f;
                off += skip;
                const V3 po = s.o + s.d * skip, d = s.d;
                const float rem = tmax - off;
                if (++peek < 8 && !(rem <= 0.0f)) {
                    bt = -1.0f;
                    HitRec b; b.t = rem; b.u = 0.f; b.v = 0.f; b.prim = -1;
                    boundary_closest_all(sc, po, d, RAY_T_MIN, b);
                    if (b.prim >= 0) bt = b.t;
                    trav_begin<true>(s, sc, po, d, RAY_T_MIN, bt >= 0.0f ? bt : rem);
                    occ = s.any_hit;
                    next = !occ;
                }
            }
            if (!next) {
                shadow_done(pv, at, occ, records);
                trav_none(s);
                at = -1;
            }
        }
        __syncwarp();
    }
    if (!ok) atomicAdd(&pv.errors[0], 1);
}

// ---------------------------------------------------------------- whole paths
// A lane follows one path to its end with all its state in registers, then
// takes the next: the camera paths of a small wave (depths 0; slots as in
// k_trace_primary_t, or k_trace_primary_batch's in a batch wave), or the
// paths at which the wavefront stopped (see WavePlan).  Every query and
// float operation is the wavefront kernels' own, in a path's own order, so
// the image does not depend on which of them ran.
//
// What bounds it is the latency of one warp's dependent instructions (a few
// warps per scheduler, each waiting for its slowest lane), not throughput:
// 128 registers and four resident blocks per SM (80 registers 5 % slower),
// the warps of a block in phase as in k_shade (volume 333x207: 625 -> 430 us,
// 800x600: 477 -> 430 us in here), at least eight lanes a warp (1M-triangle
// 960x540 frame, the last paths: 1,026 us with all 32, 895 us with 16, 897 us
// with 4).  96x64 1 spp takes 169 us on the device, against 580 us for the 34
// launches of a wavefront.
struct PathsCount {
    int cursor;
    int pad[3];
    unsigned long long segments, shadows;
};

constexpr int kPathsThreads = 128, kMinLanes = 8;
template <int ALGO, bool MULTI>
__global__ void __launch_bounds__(kPathsThreads, 512 / kPathsThreads) k_paths(DevScene sc0, FrameParams f0, PathView pv, const BatchJob* jobs,
                                                   int njobs, int slots, int fma0, int depths, int stop,
                                                   PathsCount* cnt) {
    __shared__ int sbase[MULTI ? kMaxBatchPieces : 1];
    if constexpr (MULTI) {
        for (int i = threadIdx.x; i < njobs; i += blockDim.x) sbase[i] = jobs[i].slot_base;
        __syncthreads();
    }
    const int* q = nullptr;
    if (depths > 0) {
        // the depth at which the wavefront left its paths
        int d = 1;
        for (;; ++d) {
            slots = *(volatile const int*)&pv.counters[kCountersPerDepth * d];
            if (slots <= stop || d == depths) break;
        }
        q = (d & 1) ? pv.q1 : pv.q0;
    }
    if (slots == 0) return;
    int2 stack[kStack];
    Trav s;
    // few paths are spread over the warps there are: each then waits for fewer
    // lanes and runs fewer kinds of event
    const int warps = (int)(gridDim.x * blockDim.x) / 32, lanes = min(32, max(kMinLanes, (slots + warps - 1) / warps));
    bool active = false, exhausted = (int)lane_id() >= lanes, ok = true;
    int id = 0, sid = 0;
    unsigned nseg = 0, nsh = 0;
    PathRegs ps;
    RGB result = rgb(0.f, 0.f, 0.f);
    auto scene = [&]() -> const DevScene& {
        if constexpr (MULTI) return pv.scenes[sid];
        else return sc0;
    };
    for (;;) {
        const int slot0 = refill(&cnt->cursor, slots, !active, exhausted);
        if (slot0 >= 0) {
            if (q) {
                id = q[slot0];
                if constexpr (MULTI) sid = pv.sid[id];
                const PathState& st = pv.st[id];
                ps.o = f3(st.ray_o);
                const float4 rd = st.ray_d, th = st.thr;
                ps.d = f3(rd);
                ps.depth = __float_as_int(rd.w);
                ps.T = c3(th);
                ps.last_pdf = th.w;
                const ulonglong2 rs = st.rng;
                ps.rng.state = rs.x;
                ps.rng.inc = rs.y;
                result = c3(pv.rad[id]);
                active = true;
            } else {
                int slot = slot0, base = 0;
                const FrameParams* f = &f0;
                if constexpr (MULTI) {
                    int lo = 0, hi = njobs - 1;   // the last piece whose slots start at or before the slot
                    while (lo < hi) {
                        const int mid = (lo + hi + 1) >> 1;
                        if (sbase[mid] <= slot) lo = mid; else hi = mid - 1;
                    }
                    f = &jobs[lo].f;
                    base = jobs[lo].path_base;
                    sid = jobs[lo].sid;
                    slot -= sbase[lo];
                }
                const int tw = f->tile_w, tiles_x = (tw + 7) / 8, per_sample = tiles_x * ((f->tile_h + 3) / 4) * 32;
                const int sl = slot / per_sample, in = slot - sl * per_sample, tile = in >> 5;
                const int px = (tile % tiles_x) * 8 + (in & 7), py = (tile / tiles_x) * 4 + ((in >> 3) & 3);
                if (px < tw && py < f->tile_h) {
                    const int local = sl * f->npix + py * tw + px;
                    id = base + local;
                    ps.d = camera_dir(*f, local, ps.rng);
                    ps.o = v3(f->pos[0], f->pos[1], f->pos[2]);
                    ps.T = rgb(1.0f, 1.0f, 1.0f);
                    result = rgb(0.0f, 0.0f, 0.0f);
                    ps.last_pdf = 0.0f;
                    ps.depth = 0;
                    if (!MULTI && f0.records) records_begin(pv, id);
                    active = true;
                }
            }
        }
        if (__syncthreads_or(active || !exhausted) == 0) break;
        const DevScene& sc = scene();
        HitRec h;
        h.t = 1e30f; h.u = h.v = 0.0f; h.prim = -1;
        float lt = 1e30f;
        int li = -1;
        const bool records = !MULTI && f0.records != 0;
        // closest hit beyond the volume boundaries (k_trace_lb, k_trace_post)
        const bool fma = ps.depth != 0 || fma0;
        const V3 sub = fma ? v3(0.f, 0.f, 0.f) : ps.o;
        float search = ps.depth == 0 ? 0.0f : RAY_T_MIN;
        auto begin = [&] {
            trav_begin<false>(s, sc, ps.o, ps.d, search, 1e30f);
            if (!fma) s.ooi = v3(0.f, 0.f, 0.f);
        };
        trav_none(s);
        if (active) begin();
        bool query = active;   // looking for the closest hit from `search` on
        int peek = 0;
        while (__ballot_sync(0xffffffffu, query) != 0) {
            for (unsigned m; (m = __ballot_sync(0xffffffffu, !trav_done(s))) != 0;)
                warp_step<true>(s, __popc(m), stack, sc, ok, sub);
            if (query) {
                query = false;
                h = s.h;
                while (sc.num_bnd_tris) {
                    HitRec b = s.h;
                    if (b.prim < 0) b.t = 1e30f;
                    boundary_closest<true>(sc, s.o, s.d, s.inv, search, b);
                    if (b.prim < 0) { h.prim = -1; break; }
                    if (b.prim == s.h.prim) break;
                    search = b.t + 1e-3f;
                    if (++peek == 8) { h.prim = -1; break; }
                    if (s.h.prim >= 0 && s.h.t < search) {
                        begin();
                        query = true;
                        break;
                    }
                }
            }
            __syncwarp();
        }
        if (active) {
            if (h.prim < 0) { h.t = 1e30f; h.u = 0.0f; h.v = 0.0f; }
            li = ps.depth == 0 ? -1 : native_lights_closest(sc, ps.o, ps.d, h.t, lt);
            ++nseg;
            if (records) {
                const int4 pi = h.prim >= 0 ? sc.prim_info[h.prim] : make_int4(-1, -1, -1, 0);
                if (ps.depth == 0) pv.rec_prim[id] = make_int2(pi.x, pi.y);
                pv.rec_cnt[id].x += 1;
                unsigned long long hs = pv.rec_hash[id];
                hs = hpush(hs, (uint32_t)pi.x);
                hs = hpush(hs, (uint32_t)pi.y);
                hs = hpush(hs, (uint32_t)li);
                pv.rec_hash[id] = hs;
            }
        }
        __syncwarp();
        ShadowRay sr;
        const ShadeResult r =
            shade_segment<ALGO, false>(sc, active, f0.max_depth, records, pv, id, ps,
                                       make_float4(h.t, h.u, h.v, __int_as_float(h.prim)),
                                       make_float2(__int_as_float(li), lt), sr, BlockSync());
        result = result + r.add;
        __syncwarp();
        if (r.shadow) {
            // (a sample that would add nothing is traced only to be counted)
            const bool adds = records || sr.inc.r != 0.0f || sr.inc.g != 0.0f || sr.inc.b != 0.0f;
            const bool occ = adds && shadowed_skip_boundaries<true>(sc, sr.o, sr.d, sr.len, ok);
            if (!occ) result = result + sr.inc;
            ++nsh;
            if (records) {
                int4 rc = pv.rec_cnt[id];
                rc.y += 1;
                rc.z += occ ? 1 : 0;
                pv.rec_cnt[id] = rc;
                pv.rec_hash[id] = hpush(pv.rec_hash[id], 0x5EED0000u | (occ ? 1u : 0u));
            }
        }
        if (active && !r.cont) {
            pv.rad[id] = make_float4(result.r, result.g, result.b, 0.0f);
            active = false;
        }
        __syncwarp();
    }
    nseg = __reduce_add_sync(0xffffffffu, nseg);
    nsh = __reduce_add_sync(0xffffffffu, nsh);
    if (lane_id() == 0 && nseg) {
        atomicAdd(&cnt->segments, (unsigned long long)nseg);
        atomicAdd(&cnt->shadows, (unsigned long long)nsh);
    }
    if (!ok) atomicAdd(&pv.errors[0], 1);
}
using PathsKernel = void (*)(DevScene, FrameParams, PathView, const BatchJob*, int, int, int, int, int, PathsCount*);
template <bool MULTI>
static PathsKernel paths_kernel(int algo) {
    switch (algo) {
        case ALGO_SIMPLE: return k_paths<ALGO_SIMPLE, MULTI>;
        case ALGO_MIS: return k_paths<ALGO_MIS, MULTI>;
        case ALGO_VOLUME_SIMPLE: return k_paths<ALGO_VOLUME_SIMPLE, MULTI>;
        case ALGO_VOLUME_MIS: return k_paths<ALGO_VOLUME_MIS, MULTI>;
        default: return k_paths<ALGO_NEE, MULTI>;
    }
}

// ---------------------------------------------------------------- launch profiles
// Resident CTAs per SM of the wavefront kernels (their register caps):
// profile 0 is the measured optimum on the 1M-triangle scene (closest hit 9,
// shading 8, shadow 9); profile 1 gives each kernel more registers and fewer
// spills (8, 6, 8), which scenes with short paths or few triangles can
// prefer.  The request loop's autotuner picks per job shape.
using TraceKernel = void (*)(DevScene, PathView, int*, int);
using ShadowKernel = void (*)(DevScene, PathView, int*, int);
struct LaunchSet {
    TraceKernel trace;
    ShadeKernel shade;
    ShadowKernel shadow;
};
constexpr int kLaunchProfiles = 2;
static LaunchSet launch_set(int algo, bool guide, int profile) {
    if (profile == 1) return {k_trace_lb<8>, shade_kernel_lb<6>(algo, guide), k_shadow_lb<8>};
    return {k_trace_lb<9>, shade_kernel_lb<8>(algo, guide), k_shadow_lb<9>};
}
// Batch waves: the same kernels reading each path's scene from the wave's
// scene table (profile 0's resident CTAs).
static LaunchSet launch_set_batch(int algo) {
    return {k_trace_lb<9, true>, shade_kernel_batch(algo), k_shadow_lb<9, true>};
}

// ---------------------------------------------------------------- film
// Per-pixel radiance sum in sample order: film += rad(s0), rad(s0+1), ...
// (the reference's `radiance = radiance + sample_radiance`, :318-327).
__global__ void k_film(int npix, int spw, const float4* rad, float4* film) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= npix) return;
    float4 a = film[p];
    for (int s = 0; s < spw; ++s) {
        float4 r = rad[(size_t)s * npix + p];
        a.x = a.x + r.x; a.y = a.y + r.y; a.z = a.z + r.z;
    }
    film[p] = a;
}

// FP64 accumulation for converged references: the same per-sample FP32
// radiance, summed per pixel in double in sample order.
__global__ void k_film_f64(int npix, int spw, const float4* rad, double* film) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= npix) return;
    double a0 = film[3 * (size_t)p], a1 = film[3 * (size_t)p + 1], a2 = film[3 * (size_t)p + 2];
    for (int s = 0; s < spw; ++s) {
        float4 r = rad[(size_t)s * npix + p];
        a0 += (double)r.x; a1 += (double)r.y; a2 += (double)r.z;
    }
    film[3 * (size_t)p] = a0; film[3 * (size_t)p + 1] = a1; film[3 * (size_t)p + 2] = a2;
}
__global__ void k_output_f64(int tw, int th, const double* film, double* out) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= tw * th) return;
    int x = p % tw, y = p / tw;
    double* o = out + ((size_t)(th - 1 - y) * tw + x) * 4;
    for (int c = 0; c < 3; ++c) {
        double v = film[3 * (size_t)p + c];
        o[c] = (v < 0.0) ? 0.0 : v;
    }
    o[3] = 1.0;
}

// Camera sensitivity (EV 0 => 1), clamp >= 0 keeping NaN, alpha 1, Y flip
// (pybind_renderer.hpp:330-360).
__global__ void k_output(int tw, int th, const float4* film, float4* out) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= tw * th) return;
    int x = p % tw, y = p / tw;
    float4 a = film[p];
    float r = a.x * 1.0f, g = a.y * 1.0f, b = a.z * 1.0f;
    out[(size_t)(th - 1 - y) * tw + x] = make_float4(smax(r, 0.0f), smax(g, 0.0f), smax(b, 0.0f), 1.0f);
}

// Film sum and output in one pass, for a call whose samples are one wave.  A
// pixel's sum is one chain in sample order, and with few pixels nothing else
// hides its loads: a group of kFilmGroup is loaded while the one before it is
// summed (1 pixel x 300,000 samples 20.5 -> 15.8 ms, 3 x 3 x 65,536 6.3 -> 4.5
// ms; 65,536 pixels x 32 and 2 M x 64 at the memory's rate either way).
constexpr int kFilmGroup = 8;
__global__ void __launch_bounds__(128) k_film_output(int tw, int th, int spw, const float4* rad, float4* out) {
    const int npix = tw * th;
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= npix) return;
    int x = p % tw, y = p / tw;
    float r = 0.0f, g = 0.0f, b = 0.0f;
    const int whole = spw / kFilmGroup * kFilmGroup;
    if (whole > 0) {
        float4 v[kFilmGroup];
#pragma unroll
        for (int j = 0; j < kFilmGroup; ++j) v[j] = rad[(size_t)j * npix + p];
        for (int s = 0; s < whole; s += kFilmGroup) {
            float4 next[kFilmGroup];
            const int n = s + kFilmGroup < whole ? s + kFilmGroup : s;   // (the last group's are not used)
#pragma unroll
            for (int j = 0; j < kFilmGroup; ++j) next[j] = rad[(size_t)(n + j) * npix + p];
#pragma unroll
            for (int j = 0; j < kFilmGroup; ++j) { r = r + v[j].x; g = g + v[j].y; b = b + v[j].z; }
#pragma unroll
            for (int j = 0; j < kFilmGroup; ++j) v[j] = next[j];
        }
    }
    for (int s = whole; s < spw; ++s) {
        const float4 v = rad[(size_t)s * npix + p];
        r = r + v.x; g = g + v.y; b = b + v.z;
    }
    r = r * 1.0f; g = g * 1.0f; b = b * 1.0f;
    out[(size_t)(th - 1 - y) * tw + x] = make_float4(smax(r, 0.0f), smax(g, 0.0f), smax(b, 0.0f), 1.0f);
}

__global__ void k_records(FrameParams f, PathView pv, LucidSampleRecord* out) {
    int id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= f.n_wave) return;
    int p = id % f.npix, sl = id / f.npix;
    LucidSampleRecord r;
    float4 ra = pv.rad[id];
    r.rgb[0] = ra.x; r.rgb[1] = ra.y; r.rgb[2] = ra.z;
    int2 pp = pv.rec_prim[id];
    int4 c = pv.rec_cnt[id];
    r.primary_mesh = pp.x; r.primary_tri = pp.y;
    r.bounces = (uint32_t)c.x; r.nee_tests = (uint32_t)c.y; r.nee_occluded = (uint32_t)c.z;
    r.hash = pv.rec_hash[id];
    out[(size_t)p * f.samples + f.s0 + sl] = r;
}

// ---------------------------------------------------------------- path diagnostics
// trace{Simple,NEE,MIS}WithDiagnostics (integrator/path_tracer.hpp:880-1514)
// with the PathDiagnosticRecorder (diagnostics/diagnostic_integrator.hpp:
// 87-389): one thread follows one (pixel, sample) path through every bounce;
// intersectScene covers every triangle (no volume-boundary skipping), shadow
// rays are any-hit queries over every triangle, volumes are ignored.  Each
// completed path (light, environment or emitter reached) is appended to the
// record buffer; the host replays the records into the DiagnosticFilm.
enum DiagBsdf { DB_DIFFUSE = 0, DB_GLOSSY = 1, DB_MIRROR = 2, DB_GLASS = 3, DB_EMISSION = 4 };
enum DiagLight { DL_UNKNOWN = 0, DL_POINT = 1, DL_AREA = 2, DL_DIRECTIONAL = 3, DL_SPOT = 4, DL_ENV = 5, DL_EMISSIVE = 6 };
enum DiagStrategy { DS_BSDF = 0, DS_NEE = 1, DS_MIS_BSDF = 2, DS_MIS_NEE = 3 };

LD uint8_t diag_light_type(int type) {   // to_light_source_type (diagnostics/path_types.hpp)
    switch (type) {
        case LIGHT_EMISSIVE: return DL_AREA;
        case LIGHT_POINT: return DL_POINT;
        case LIGHT_SUN: return DL_DIRECTIONAL;
        case LIGHT_SPOT: return DL_SPOT;
        case LIGHT_AREA: return DL_AREA;
    }
    return DL_UNKNOWN;
}

struct DiagPath {   // the recorder's current PathTrace
    int depth;
    int32_t obj[kDiagMaxDepth];
    uint8_t bsdf[kDiagMaxDepth], flags[kDiagMaxDepth];
    V3 pos[kDiagMaxDepth], nrm[kDiagMaxDepth];
};

struct DiagOut {
    uint4* units;
    uint32_t* index;
    unsigned long long* count;   // [0] records, [1] units
    long long cap, cap_units;
    uint32_t unit_base;          // the band's units before this wave (index entries are band offsets)
};

LD void diag_vertex(DiagPath& P, int32_t obj, uint8_t type, bool delta, V3 p, V3 n) {
    if (P.depth >= kDiagMaxDepth) return;
    P.obj[P.depth] = obj; P.bsdf[P.depth] = type; P.flags[P.depth] = delta ? 1 : 0;
    P.pos[P.depth] = p; P.nrm[P.depth] = n;
    ++P.depth;
}

// record_completed_path_with_geometry (diagnostic_integrator.hpp:349-389):
// the path plus a final Emission vertex (object -1 for the environment, else
// -(light + 2)) when there is room, in the compact form (lucid_diag.h).
// A record slot and its units per calling thread with one atomic each per
// group of converged lanes (the lanes that complete a path at the same point
// of the loop; the units by an exclusive scan of the record sizes); each
// thread's slots still increase in its own program order, which the host's
// sort uses to keep records of one (pixel, sample, bounce) in order.
LD void diag_vertex_store(uint4* u, int32_t obj, uint32_t bsdf, uint32_t flags, V3 p, V3 n) {
    u[0] = make_uint4((uint32_t)obj, bsdf | (flags << 8), __float_as_uint(p.x), __float_as_uint(p.y));
    u[1] = make_uint4(__float_as_uint(p.z), __float_as_uint(n.x), __float_as_uint(n.y), __float_as_uint(n.z));
}

LD void diag_complete(const DiagOut& o, const DiagPath& P, uint32_t pixel, uint32_t sample, uint32_t seq,
                      uint8_t strategy, int light_id, uint8_t ltype, RGB c, V3 lpos) {
    const int d = P.depth;
    const bool emission = d < kDiagMaxDepth;
    const int dv = d + (emission ? 1 : 0);
    const unsigned size = 2u + 2u * (unsigned)dv;
    cg::coalesced_group g = cg::coalesced_threads();
    const unsigned before = cg::exclusive_scan(g, size);
    const unsigned total = g.shfl(before + size, g.size() - 1);
    unsigned long long rb = 0, ub = 0;
    if (g.thread_rank() == 0) {
        rb = atomicAdd(&o.count[0], (unsigned long long)g.size());
        ub = atomicAdd(&o.count[1], (unsigned long long)total);
    }
    const unsigned long long slot = g.shfl(rb, 0) + g.thread_rank();
    const unsigned long long uoff = g.shfl(ub, 0) + before;
    // past either capacity the host grows the buffers and runs the wave again
    if ((long long)slot >= o.cap || (long long)(uoff + size) > o.cap_units) return;
    o.index[slot] = o.unit_base + (uint32_t)uoff;
    uint4* u = o.units + uoff;
    u[0] = make_uint4(pixel, sample, seq, (uint32_t)strategy | ((uint32_t)ltype << 8) | ((uint32_t)dv << 16));
    u[1] = make_uint4(__float_as_uint(c.r), __float_as_uint(c.g), __float_as_uint(c.b), 0u);
    for (int k = 0; k < d; ++k) diag_vertex_store(u + 2 + 2 * k, P.obj[k], P.bsdf[k], P.flags[k], P.pos[k], P.nrm[k]);
    if (emission)
        diag_vertex_store(u + 2 + 2 * d, (ltype == DL_ENV) ? -1 : -(light_id + 2), DB_EMISSION, 0u, lpos,
                          v3(0.0f, 0.0f, 0.0f));
}

__global__ void __launch_bounds__(128) k_diag_paths(DevScene sc, FrameParams f, PathView pv, DiagOut out,
                                                    int pixel_base) {
    int id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= f.n_wave) return;
    const int algo = f.algo;   // ALGO_SIMPLE, ALGO_MIS, else NEE (pybind_renderer.hpp:300-309)
    const bool simple = algo == ALGO_SIMPLE, mis = algo == ALGO_MIS, nee_only = !simple && !mis;
    const uint32_t pixel = (uint32_t)(pixel_base + id % f.npix);
    const uint32_t sample = (uint32_t)(f.s0 + id / f.npix);
    ulonglong2 rs = pv.st[id].rng;
    Rng rng;
    rng.state = rs.x;
    rng.inc = rs.y;
    float4 ro = pv.st[id].ray_o, rd = pv.st[id].ray_d;
    V3 o = f3(ro), d = f3(rd);
    float tmin = 0.0f;
    RGB result = rgb(0.f, 0.f, 0.f), T = rgb(1.f, 1.f, 1.f);
    float last_pdf = 0.0f;
    bool ok = true;
    DiagPath P;
    P.depth = 0;
    for (int depth = 0; depth < f.max_depth; ++depth) {
        const uint32_t seq = (uint32_t)depth * 2u;
        HitRec h = scene_closest(sc, o, d, tmin, 1e30f, ok);
        float lt = 1e30f;
        int li = (depth == 0) ? -1 : native_lights_closest(sc, o, d, h.prim >= 0 ? h.t : 1e30f, lt);
        if (li >= 0) {   // in front of the surface hit (the bound above)
            if (!nee_only || depth == 0) {
                const DevLight& L = sc.lights[sc.native_start + li];
                uint8_t ltype = diag_light_type(__float_as_int(L.pos_type.w));
                V3 lp = o + d * lt;
                float mw = 1.0f;
                if (mis) {
                    float lpdf = 0.0f;
                    if (sc.num_lights > 0) {
                        float sp = area_ratio(L.normal_area.w, sc.total_light_area);
                        if (sp > 0.0f) {
                            V3 ln = (__float_as_int(L.pos_type.w) == LIGHT_POINT) ? normalize_nz(lp - f3(L.pos_type))
                                                                                  : f3(L.normal_area);
                            lpdf = pdf_light(L.normal_area.w, o, lp, ln) * sp;
                        }
                    }
                    mw = (last_pdf > MIN_PDF && lpdf > MIN_PDF) ? mis_power(last_pdf, lpdf) : 1.0f;
                }
                RGB em = c3(L.emission_radius);
                RGB pc = mis ? mul(T, em) * mw : mul(T, em);
                diag_complete(out, P, pixel, sample, seq, mis ? DS_MIS_BSDF : DS_BSDF, li, ltype, pc, lp);
                result = result + pc;
            }
            break;
        }
        if (h.prim < 0) {
            if (!nee_only || depth == 0) {
                RGB env = mul(T, rgb(sc.env[0], sc.env[1], sc.env[2]));
                diag_complete(out, P, pixel, sample, seq, mis ? DS_MIS_BSDF : DS_BSDF, -1, DL_ENV, env,
                              o + d * 1000.0f);
                result = result + env;
            }
            break;
        }
        V3 p = o + d * h.t;
        int4 pi = sc.prim_info[h.prim];
        V3 fn = f3(sc.prim_fn[h.prim]);
        V3 n = fn;
        if (pi.w) {
            float w = 1.0f - h.u - h.v;
            V3 ni = f3(sc.prim_vn[3 * h.prim]) * w + f3(sc.prim_vn[3 * h.prim + 1]) * h.u +
                    f3(sc.prim_vn[3 * h.prim + 2]) * h.v;
            n = make_dir_or(ni, fn);
        }
        const DevMaterial& dm = sc.materials[pi.x];
        Mat m;
        m.albedo = c3(dm.albedo_metallic);
        m.metallic = dm.albedo_metallic.w;
        m.roughness = smax(dm.rough_trans_ior_flags.x, MIN_ROUGHNESS);
        m.transmission = dm.rough_trans_ior_flags.y;
        m.ior = dm.rough_trans_ior_flags.z;
        RGB em = c3(dm.emission);
        bool has_em = dm.emission.w != 0.0f;
        apply_textures(sc, dm, h.prim, h.u, h.v, m.albedo, em, has_em);
        // classify_bsdf / is_delta_bsdf (diagnostic_integrator.hpp:25-60)
        uint8_t bt = m.transmission > 0.5f                       ? DB_GLASS
                     : (m.roughness < 0.01f && m.metallic > 0.5f) ? DB_MIRROR
                     : (m.metallic > 0.5f || m.roughness < 0.5f)  ? DB_GLOSSY
                                                                  : DB_DIFFUSE;
        bool delta = (m.transmission > 0.5f && m.roughness < 0.01f) || (m.metallic > 0.5f && m.roughness < 0.01f);
        V3 wo = -d;
        bool front = dot(wo, n) > 0;
        V3 sn = n;
        if (m.transmission < 0.5f && !front) sn = -n;
        if (simple) {
            if (has_em) {
                RGB ec = mul(T, em);
                diag_complete(out, P, pixel, sample, seq, DS_BSDF, pi.x, DL_EMISSIVE, ec, p);
                result = result + ec;
                break;
            }
            diag_vertex(P, pi.x, bt, delta, p, n);
        } else {
            bool do_nee = false;
            if (has_em && (mis || depth == 0)) {
                float mw = 1.0f;
                if (mis && sc.num_lights > 0 && last_pdf > MIN_PDF && pi.z >= 0) {
                    const DevLight& L = sc.lights[pi.z];
                    float sp = area_ratio(L.normal_area.w, sc.total_light_area);
                    if (sp > 0.0f) {
                        float lpdf = pdf_light(L.normal_area.w, o, p, n) * sp;
                        if (lpdf > MIN_PDF) mw = mis_power(last_pdf, lpdf);
                    }
                }
                RGB ec = mis ? mul(T, em) * mw : mul(T, em);
                diag_complete(out, P, pixel, sample, seq, mis ? DS_MIS_BSDF : DS_BSDF, pi.x, DL_EMISSIVE, ec, p);
                result = result + ec;
            } else if (!has_em) {
                diag_vertex(P, pi.x, bt, delta, p, n);
                do_nee = true;
            }
            const bool transmissive = m.transmission > 0.5f;
            if (do_nee && sc.num_lights > 0 && !transmissive) {
                float usel = randf(rng);
                int sli = select_light(sc, usel);
                const DevLight& L = sc.lights[sli];
                float lsp = area_ratio(L.normal_area.w, sc.total_light_area);
                if (lsp > 1e-6f) {
                    float u1 = randf(rng), u2 = randf(rng);
                    LightSample ls = sample_light(L, p, u1, u2);
                    if (ls.pdf > MIN_PDF) {
                        float nl = dot(sn, ls.dir);
                        if (nl > 1e-6f) {
                            bool occ = bvh_any(sc, p, ls.dir, RAY_T_MIN, ls.dist, ok) ||
                                       (sc.num_bnd_tris &&
                                        list_any(sc.bnd_tris, sc.num_bnd_tris, p, ls.dir, RAY_T_MIN, ls.dist));
                            if (!occ) {
                                float pb;
                                RGB fb = eval_bsdf<true>(m, wo, ls.dir, sn, nl, pb);
                                float pl = ls.pdf * lsp;
                                RGB nr;
                                if (mis) {
                                    float mw = mis_power(pl, pb);
                                    nr = mul(bsdf_weight(fb, nl, pl) * mw, ls.emission);
                                } else {
                                    nr = mul(bsdf_weight(fb, nl, pl), ls.emission);
                                }
                                RGB tot = mul(T, nr);
                                diag_complete(out, P, pixel, sample, seq + 1u, mis ? DS_MIS_NEE : DS_NEE,
                                              sli - sc.native_start, diag_light_type(__float_as_int(L.pos_type.w)),
                                              tot, ls.pos);
                                result = result + tot;
                            }
                        }
                    }
                }
            }
        }
        V3 smp_n = (m.transmission > 0.5f) ? n : sn;
        float u1 = randf(rng), u2 = randf(rng), u3 = randf(rng);
        BsdfSample bs = sample_bsdf(m, wo, smp_n, u1, u2, u3, rng);
        if (!(bs.kind == BS_PRECOMP || bs.pdf > MIN_PDF)) break;
        RGB w;
        if (bs.kind == BS_PRECOMP) {
            w = bs.f;
        } else {
            float c = fabsf(dot(smp_n, bs.wi));
            if (c <= 1e-6f || bs.pdf < MIN_PDF) break;
            w = bsdf_weight(bs.f, c, bs.pdf);
        }
        T = mul(T, w);
        if (mis) last_pdf = (bs.kind == BS_EVAL) ? bs.pdf : 0.0f;
        if (depth >= 3) {
            float rr = smin(smax3(T.r, T.g, T.b), 0.95f);
            if (randf(rng) > rr) break;
            T = T * (1.0f / rr);
        }
        if (!rgb_valid(T)) break;
        o = p;
        d = bs.wi;
        tmin = RAY_T_MIN;
    }
    pv.rad[id] = make_float4(result.r, result.g, result.b, 0.0f);
    if (!ok) atomicAdd(&pv.errors[0], 1);
}

// ---------------------------------------------------------------- debug passes
// render_debug (renderer.hpp:59-93): intersectScene from t = 0 over every
// triangle (boundary meshes included), no jitter.
__global__ void k_debug(DevScene sc, FrameParams f, int mode, float4* out, int* errors) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= f.npix) return;
    int px = p % f.tile_w, py = p / f.tile_w;
    int gx = f.tile_x + px, gy = f.tile_y + py;
    float nx = (2.0f * ((float)gx + 0.5f) / (float)f.full_w - 1.0f) * f.aspect;
    float ny = 1.0f - 2.0f * ((float)gy + 0.5f) / (float)f.full_h;
    V3 d = primary_dir(f, nx, ny);
    bool ok = true;
    HitRec h = scene_closest(sc, v3(f.pos[0], f.pos[1], f.pos[2]), d, 0.0f, 1e30f, ok);
    if (!ok) atomicAdd(&errors[0], 1);
    // a miss is black, except in the normal pass, which maps its colour to
    // 0..1 after the lookup (pybind_renderer.hpp:412-415): grey
    float4 c = mode == 0 ? make_float4(0.5f, 0.5f, 0.5f, 1.f) : make_float4(0.f, 0.f, 0.f, 1.f);
    if (h.prim >= 0) {
        int4 pi = sc.prim_info[h.prim];
        V3 fn = f3(sc.prim_fn[h.prim]);
        V3 n = fn;
        if (pi.w) {
            float w = 1.0f - h.u - h.v;
            V3 ni = f3(sc.prim_vn[3 * h.prim]) * w + f3(sc.prim_vn[3 * h.prim + 1]) * h.u +
                    f3(sc.prim_vn[3 * h.prim + 2]) * h.v;
            n = make_dir_or(ni, fn);
        }
        const DevMaterial& dm = sc.materials[pi.x];
        RGB alb = c3(dm.albedo_metallic), em = c3(dm.emission);
        bool has_em = false;
        apply_textures(sc, dm, h.prim, h.u, h.v, alb, em, has_em);
        if (mode == 0) c = make_float4(n.x * 0.5f + 0.5f, n.y * 0.5f + 0.5f, n.z * 0.5f + 0.5f, 1.0f);
        else if (mode == 1) c = make_float4(alb.r, alb.g, alb.b, 1.0f);
        else c = make_float4(em.r * 1.0f, em.g * 1.0f, em.b * 1.0f, 1.0f);
    }
    out[(size_t)(f.tile_h - 1 - py) * f.tile_w + px] = c;
}

// ---------------------------------------------------------------- LBVH build
// Karras 2012 ("Maximizing parallelism in the construction of BVHs"):
// 63-bit Morton codes of triangle centroids, radix sort, one thread per
// internal node, bottom-up refit with arrival counters; subtrees of at most
// four triangles are collapsed into leaves when the nodes are flattened.
__host__ __device__ __forceinline__ int ord_f(float f) {
    int i;
    memcpy(&i, &f, 4);
    return i >= 0 ? i : i ^ 0x7fffffff;
}
__host__ __device__ __forceinline__ float unord_f(int i) {
    i = i >= 0 ? i : i ^ 0x7fffffff;
    float f;
    memcpy(&f, &i, 4);
    return f;
}
LD V3 centroid(const float4* verts, int prim) {
    V3 a = f3(verts[3 * prim]), b = f3(verts[3 * prim + 1]), c = f3(verts[3 * prim + 2]);
    return (a + b + c) * (1.0f / 3.0f);
}

__global__ void k_centroid_bounds(const float4* verts, const int* ids, int n, int* bounds) {
    __shared__ int s[6][128];
    int t = threadIdx.x;
    int mn[3] = {0x7fffffff, 0x7fffffff, 0x7fffffff}, mx[3] = {(int)0x80000000, (int)0x80000000, (int)0x80000000};
    for (int i = blockIdx.x * blockDim.x + t; i < n; i += gridDim.x * blockDim.x) {
        V3 c = centroid(verts, ids[i]);
        int o[3] = {ord_f(c.x), ord_f(c.y), ord_f(c.z)};
        for (int k = 0; k < 3; ++k) { mn[k] = min(mn[k], o[k]); mx[k] = max(mx[k], o[k]); }
    }
    for (int k = 0; k < 3; ++k) { s[k][t] = mn[k]; s[3 + k][t] = mx[k]; }
    __syncthreads();
    for (int w = 64; w > 0; w >>= 1) {
        if (t < w)
            for (int k = 0; k < 3; ++k) {
                s[k][t] = min(s[k][t], s[k][t + w]);
                s[3 + k][t] = max(s[3 + k][t], s[3 + k][t + w]);
            }
        __syncthreads();
    }
    if (t == 0)
        for (int k = 0; k < 3; ++k) { atomicMin(&bounds[k], s[k][0]); atomicMax(&bounds[3 + k], s[3 + k][0]); }
}

LD unsigned long long expand21(unsigned long long v) {
    v &= 0x1fffffULL;
    v = (v | v << 32) & 0x1f00000000ffffULL;
    v = (v | v << 16) & 0x1f0000ff0000ffULL;
    v = (v | v << 8) & 0x100f00f00f00f00fULL;
    v = (v | v << 4) & 0x10c30c30c30c30c3ULL;
    v = (v | v << 2) & 0x1249249249249249ULL;
    return v;
}

__global__ void k_morton(const float4* verts, const int* ids, int n, const int* bounds, unsigned long long* keys,
                         int* vals) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    V3 c = centroid(verts, ids[i]);
    float lo[3] = {unord_f(bounds[0]), unord_f(bounds[1]), unord_f(bounds[2])};
    float hi[3] = {unord_f(bounds[3]), unord_f(bounds[4]), unord_f(bounds[5])};
    float cc[3] = {c.x, c.y, c.z};
    unsigned long long code = 0;
    for (int k = 0; k < 3; ++k) {
        float ext = hi[k] - lo[k];
        float u = ext > 0.0f ? (cc[k] - lo[k]) / ext : 0.5f;
        unsigned long long q = (unsigned long long)fminf(fmaxf(u * 2097152.0f, 0.0f), 2097151.0f);
        code |= expand21(q) << (2 - k);
    }
    keys[i] = code;
    vals[i] = ids[i];
}

LD int delta_k(const unsigned long long* keys, int n, int i, int j) {
    if (j < 0 || j >= n) return -1;
    unsigned long long a = keys[i], b = keys[j];
    if (a == b) return 64 + __clz(i ^ j);
    return __clzll(a ^ b);
}

// children: code >= 0 internal node, < 0 ~leaf index
__global__ void k_karras(const unsigned long long* keys, int n, int2* child, int* parent, int* leaf_parent,
                         int2* range) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n - 1) return;
    int d = (delta_k(keys, n, i, i + 1) - delta_k(keys, n, i, i - 1)) >= 0 ? 1 : -1;
    int dmin = delta_k(keys, n, i, i - d);
    int lmax = 2;
    while (delta_k(keys, n, i, i + lmax * d) > dmin) lmax <<= 1;
    int l = 0;
    for (int t = lmax >> 1; t >= 1; t >>= 1)
        if (delta_k(keys, n, i, i + (l + t) * d) > dmin) l += t;
    int j = i + l * d;
    int dnode = delta_k(keys, n, i, j);
    int s = 0, t = l;
    do {
        t = (t + 1) >> 1;
        if (delta_k(keys, n, i, i + (s + t) * d) > dnode) s += t;
    } while (t > 1);
    int gamma = i + s * d + min(d, 0);
    int first = min(i, j), last = max(i, j);
    int cl = (first == gamma) ? ~gamma : gamma;
    int cr = (last == gamma + 1) ? ~(gamma + 1) : gamma + 1;
    child[i] = make_int2(cl, cr);
    range[i] = make_int2(first, last);
    if (cl >= 0) parent[cl] = i; else leaf_parent[~cl] = i;
    if (cr >= 0) parent[cr] = i; else leaf_parent[~cr] = i;
}

LD void leaf_box(const float4* verts, int prim, float* b) {
    V3 a = f3(verts[3 * prim]), c = f3(verts[3 * prim + 1]), e = f3(verts[3 * prim + 2]);
    b[0] = fminf(fminf(a.x, c.x), e.x); b[1] = fminf(fminf(a.y, c.y), e.y); b[2] = fminf(fminf(a.z, c.z), e.z);
    b[3] = fmaxf(fmaxf(a.x, c.x), e.x); b[4] = fmaxf(fmaxf(a.y, c.y), e.y); b[5] = fmaxf(fmaxf(a.z, c.z), e.z);
}

__global__ void k_refit(const float4* verts, const int* sorted_ids, int n, const int2* child, const int* parent,
                        const int* leaf_parent, int* arrive, float* nbox) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    int node = leaf_parent[k];
    // A Karras tree is at most 64 + log2(n) levels deep; the bound only
    // guards against a malformed hierarchy.
    for (int level = 0; node >= 0 && level < 256; ++level) {
        __threadfence();
        if (atomicAdd(&arrive[node], 1) == 0) return;   // the sibling subtree finishes this node
        __threadfence();
        int2 c = child[node];
        float b[6], bb[6];
        if (c.x < 0) leaf_box(verts, sorted_ids[~c.x], b);
        else for (int q = 0; q < 6; ++q) b[q] = __ldcg(&nbox[6 * c.x + q]);
        if (c.y < 0) leaf_box(verts, sorted_ids[~c.y], bb);
        else for (int q = 0; q < 6; ++q) bb[q] = __ldcg(&nbox[6 * c.y + q]);
        for (int q = 0; q < 3; ++q) {
            __stcg(&nbox[6 * node + q], fminf(b[q], bb[q]));
            __stcg(&nbox[6 * node + 3 + q], fmaxf(b[3 + q], bb[3 + q]));
        }
        node = parent[node];
    }
}

__host__ __device__ __forceinline__ int leaf_code(int start, int count) { return ~((start << 3) | (count - 1)); }

__global__ void k_flatten(const float4* verts, const int* sorted_ids, int n, const int2* child, const int2* range,
                          const float* nbox, float pad, DevNode* nodes) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n - 1) return;
    int2 c = child[i];
    int cc[2] = {c.x, c.y};
    float bx[2][6];
    int code[2];
    for (int s = 0; s < 2; ++s) {
        int ch = cc[s];
        if (ch < 0) {
            leaf_box(verts, sorted_ids[~ch], bx[s]);
            code[s] = leaf_code(~ch, 1);
        } else {
            for (int q = 0; q < 6; ++q) bx[s][q] = nbox[6 * ch + q];
            int2 r = range[ch];
            int cnt = r.y - r.x + 1;
            code[s] = cnt <= 4 ? leaf_code(r.x, cnt) : ch;
        }
        for (int q = 0; q < 3; ++q) { bx[s][q] -= pad; bx[s][3 + q] += pad; }
    }
    DevNode nd;
    nd.lmin_lc = make_float4(bx[0][0], bx[0][1], bx[0][2], __int_as_float(code[0]));
    nd.lmax_rc = make_float4(bx[0][3], bx[0][4], bx[0][5], __int_as_float(code[1]));
    nd.rmin = make_float4(bx[1][0], bx[1][1], bx[1][2], 0.0f);
    nd.rmax = make_float4(bx[1][3], bx[1][4], bx[1][5], 0.0f);
    nodes[i] = nd;
}

// ---------------------------------------------------------------- PLOC build
// Parallel locally-ordered clustering (Meister & Bittner, "Parallel Locally-
// Ordered Clustering for Bounding Volume Hierarchy Construction", IEEE TVCG
// 2018): clusters start as the Morton-sorted triangles; each round every
// cluster finds the neighbour within +-kPlocRadius positions whose merged box
// has the smallest surface area, mutual nearest neighbours merge into a new
// node, and the cluster array is compacted in order.  Candidate pairs are
// totally ordered (area, then a tie key of the pair), so the best pair of a
// round is always mutual and every round merges at least one pair.  Node ids follow
// creation order (root last); a top-down pass then gives every subtree a
// contiguous range of triangle slots so that k_flatten can collapse small
// subtrees into leaves exactly as for the Karras tree.
constexpr int kPlocRadius = 32;
constexpr int kPlocBlock = 256;

struct PlocBox { float lo[3], hi[3]; };

LD float ploc_area(const float* a, const float* b) {
    float dx = fmaxf(a[3], b[3]) - fminf(a[0], b[0]);
    float dy = fmaxf(a[4], b[4]) - fminf(a[1], b[1]);
    float dz = fmaxf(a[5], b[5]) - fminf(a[2], b[2]);
    return dx * dy + dy * dz + dz * dx;
}

// Initial clusters: leaf i (Morton order) with its triangle's box.
__global__ void k_ploc_init(const float4* verts, const int* sorted_ids, int n, int* cl, float* cbox, int* cnt_leaf) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    cl[i] = ~i;
    leaf_box(verts, sorted_ids[i], cbox + 6 * (size_t)i);
    cnt_leaf[i] = 1;
}

// Nearest neighbour of every cluster within the window (boxes staged in
// shared memory with a halo of kPlocRadius on both sides).
__global__ void __launch_bounds__(kPlocBlock) k_ploc_nn(const float* cbox, int count, int* nn) {
    __shared__ float sb[(kPlocBlock + 2 * kPlocRadius) * 6];
    const int b0 = blockIdx.x * kPlocBlock;
    for (int t = threadIdx.x; t < (kPlocBlock + 2 * kPlocRadius) * 6; t += kPlocBlock) {
        int j = b0 - kPlocRadius + t / 6;
        sb[t] = (j >= 0 && j < count) ? cbox[6 * (size_t)j + t % 6] : 0.0f;
    }
    __syncthreads();
    int i = b0 + threadIdx.x;
    if (i >= count) return;
    const float* bi = sb + 6 * (threadIdx.x + kPlocRadius);
    float best = 3.0e38f;
    int bj = -1, bgap = 0, ba = 0;
    int lo = max(0, i - kPlocRadius), hi = min(count - 1, i + kPlocRadius);
    for (int j = lo; j <= hi; ++j) {
        if (j == i) continue;
        float d = ploc_area(bi, sb + 6 * (j - b0 + kPlocRadius));
        // pair key (area, index gap, parity of the lower index, lower index):
        // it depends on the pair only, so the best pair is mutual; on equal
        // areas neighbours pair up (0,1), (2,3), ... instead of chaining
        int a = min(i, j), gap = abs(i - j);
        bool better = bj < 0 || d < best ||
                      (d == best && (gap < bgap || (gap == bgap && ((a & 1) < (ba & 1) ||
                                                                    ((a & 1) == (ba & 1) && a < ba)))));
        if (better) { best = d; bj = j; bgap = gap; ba = a; }
    }
    nn[i] = bj;
}

// flags[i]: high word 1 = creates a node (mutual pair, lower index), low word
// 1 = the cluster survives (unmerged, or the lower index of a merged pair);
// one scan sums both.
__global__ void k_ploc_flags(const int* nn, int count, unsigned long long* flags) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    int j = nn[i];
    bool mutual = j >= 0 && nn[j] == i;
    flags[i] = ((mutual && i < j) ? 1ull << 32 : 0ull) | ((!mutual || i < j) ? 1ull : 0ull);
}

// Merges (node id = base + exclusive scan of create) and compacts the
// clusters (position = exclusive scan of keep) into the other buffers.
// totals: the nodes created (high word) and the clusters that survive.
__global__ void k_ploc_merge(const int* cl, const float* cbox, const int* nn, const unsigned long long* flags,
                             const unsigned long long* pos, int count, int base, int2* child, float* nbox,
                             int* cnt_node, const int* cnt_leaf, int* cl_out, float* cbox_out,
                             unsigned long long* totals) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    if (i == count - 1) *totals = pos[i] + flags[i];
    if (!(flags[i] & 0xffffffffull)) return;
    int o = (int)(pos[i] & 0xffffffffull);
    if (!(flags[i] >> 32)) {
        cl_out[o] = cl[i];
        for (int q = 0; q < 6; ++q) cbox_out[6 * (size_t)o + q] = cbox[6 * (size_t)i + q];
        return;
    }
    int j = nn[i];
    int id = base + (int)(pos[i] >> 32);
    int a = cl[i], b = cl[j];
    child[id] = make_int2(a, b);
    float m[6];
    for (int q = 0; q < 3; ++q) {
        m[q] = fminf(cbox[6 * (size_t)i + q], cbox[6 * (size_t)j + q]);
        m[3 + q] = fmaxf(cbox[6 * (size_t)i + 3 + q], cbox[6 * (size_t)j + 3 + q]);
    }
    for (int q = 0; q < 6; ++q) { nbox[6 * (size_t)id + q] = m[q]; cbox_out[6 * (size_t)o + q] = m[q]; }
    cnt_node[id] = (a >= 0 ? cnt_node[a] : cnt_leaf[~a]) + (b >= 0 ? cnt_node[b] : cnt_leaf[~b]);
    cl_out[o] = id;
}

// Top-down slot assignment for the nodes created in one round (processed in
// reverse creation order, so a node's own offset is already known).
__global__ void k_ploc_offsets(const int2* child, const int* cnt_node, int base, int m, int* off_node, int* leaf_pos) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= m) return;
    int id = base + k;
    int2 c = child[id];
    int o = off_node[id];
    int ca = c.x >= 0 ? cnt_node[c.x] : 1;
    if (c.x >= 0) off_node[c.x] = o; else leaf_pos[~c.x] = o;
    if (c.y >= 0) off_node[c.y] = o + ca; else leaf_pos[~c.y] = o + ca;
}

// Children re-coded to triangle slots, subtree slot ranges, triangle ids in
// slot order.
__global__ void k_ploc_finish(const int* sorted_ids, const int* leaf_pos, int n, int2* child, const int* off_node,
                              const int* cnt_node, int2* range, int* slot_ids) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) slot_ids[leaf_pos[i]] = sorted_ids[i];
    if (i < n - 1) {
        int2 c = child[i];
        if (c.x < 0) c.x = ~leaf_pos[~c.x];
        if (c.y < 0) c.y = ~leaf_pos[~c.y];
        child[i] = c;
        range[i] = make_int2(off_node[i], off_node[i] + cnt_node[i] - 1);
    }
}

// Triangle k of the BVH order: v0 | prim, v1 - v0, v2 - v0.
__global__ void k_gather_tris(const float4* verts, const int* sorted_ids, int n, float4* out) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int prim = sorted_ids[k];
    const float4 a = verts[3 * (size_t)prim], b = verts[3 * (size_t)prim + 1], c = verts[3 * (size_t)prim + 2];
    out[4 * (size_t)k] = make_float4(a.x, a.y, a.z, __int_as_float(prim));
    out[4 * (size_t)k + 1] = make_float4(b.x - a.x, b.y - a.y, b.z - a.z, 0.0f);
    out[4 * (size_t)k + 2] = make_float4(c.x - a.x, c.y - a.y, c.z - a.z, 0.0f);
    out[4 * (size_t)k + 3] = make_float4(0.f, 0.f, 0.f, 0.f);
}

// ---- per-prim values the upload leaves to the device ----
// Face normals as the scene assembly computes them (the same float
// operations), and each prim's shading class from its mesh's.
__global__ void k_prim_values(const float4* verts, const int4* info, const unsigned char* mesh_cls, int n, float4* fn,
                              unsigned char* cls) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const V3 a = f3(verts[3 * (size_t)p]), b = f3(verts[3 * (size_t)p + 1]), c = f3(verts[3 * (size_t)p + 2]);
    const V3 f = make_dir_or(cross(b - a, c - a), v3(0.f, 1.f, 0.f));
    fn[p] = make_float4(f.x, f.y, f.z, 0.0f);
    cls[p] = mesh_cls[info[p].x];
}
// Bounds of the prims in the BVH or its list, and the largest coordinate
// magnitude of all (ordered-int form, starting from +-1e30 and 0).
struct PrimBounds {
    int lo[3], hi[3], maxabs;
    int big;   // candidates found by k_big_candidates
};
__global__ void __launch_bounds__(256) k_prim_bounds(const float4* verts, const unsigned char* boundary, int n,
                                                     PrimBounds* out) {
    float lo[3] = {1e30f, 1e30f, 1e30f}, hi[3] = {-1e30f, -1e30f, -1e30f}, m = 0.0f;
    for (int p = blockIdx.x * 256 + (int)threadIdx.x; p < n; p += gridDim.x * 256) {
        const bool in = !boundary[p];
        for (int k = 0; k < 3; ++k) {
            const float4 q = verts[3 * (size_t)p + k];
            const float c[3] = {q.x, q.y, q.z};
            for (int a = 0; a < 3; ++a) {
                m = fmaxf(m, fabsf(c[a]));
                if (in) { lo[a] = fminf(lo[a], c[a]); hi[a] = fmaxf(hi[a], c[a]); }
            }
        }
    }
    for (int a = 0; a < 3; ++a) {
        const int l = __reduce_min_sync(0xffffffffu, ord_f(lo[a])), h = __reduce_max_sync(0xffffffffu, ord_f(hi[a]));
        if (lane_id() == 0) {
            atomicMin(&out->lo[a], l);
            atomicMax(&out->hi[a], h);
        }
    }
    const int mm = __reduce_max_sync(0xffffffffu, ord_f(m));
    if (lane_id() == 0) atomicMax(&out->maxabs, mm);
}
// Prims whose bounding-box diagonal exceeds `thr`: (prim, diagonal), at most
// cap of them in any order, and how many there are.
__global__ void k_big_candidates(const float4* verts, const unsigned char* boundary, int n, float thr, int cap,
                                 PrimBounds* b, int2* out) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n || boundary[p]) return;
    float lo[3] = {1e30f, 1e30f, 1e30f}, hi[3] = {-1e30f, -1e30f, -1e30f};
    for (int k = 0; k < 3; ++k) {
        const float4 q = verts[3 * (size_t)p + k];
        const float c[3] = {q.x, q.y, q.z};
        for (int a = 0; a < 3; ++a) { lo[a] = fminf(lo[a], c[a]); hi[a] = fmaxf(hi[a], c[a]); }
    }
    const float d = sqrtf((hi[0] - lo[0]) * (hi[0] - lo[0]) + (hi[1] - lo[1]) * (hi[1] - lo[1]) +
                          (hi[2] - lo[2]) * (hi[2] - lo[2]));
    if (!(d > thr)) return;
    const int at = atomicAdd(&b->big, 1);
    if (at < cap) out[at] = make_int2(p, __float_as_int(d));
}
// Prims of the BVH: neither boundary-only nor in the list of large ones.
constexpr int kMaxBig = 32;
struct InBvh {
    const unsigned char* boundary;
    int big[kMaxBig];
    int nbig;
    __device__ bool operator()(int p) const {
        if (boundary[p]) return false;
        for (int k = 0; k < nbig; ++k)
            if (big[k] == p) return false;
        return true;
    }
};

// ---- the flattened tree's levels, order and 4-wide collapse ----
constexpr int kTreeLevels = kStack;   // levels of internal nodes a traversal stack allows for
struct TreeCounts {
    int error, leaves, leaf_tris, pad;
    // level l: list[first[l] .. first[l] + count[l]); the same for the 4-wide tree
    int first[kTreeLevels + 1], count[kTreeLevels + 1];
    int wide_first[kTreeLevels + 1], wide_count[kTreeLevels + 1];
};

LD void node_codes(const DevNode& nd, int c[2]) {
    c[0] = __float_as_int(nd.lmin_lc.w);
    c[1] = __float_as_int(nd.lmax_rc.w);
}

__global__ void k_tree_root(int root, int n, int* list, int* seen, TreeCounts* tc) {
    if (root < 0 || root >= n - 1) { tc->error = 1; return; }
    list[0] = root;
    seen[root] = 0;
    tc->count[0] = 1;
}

// Appends the internal children of level l's nodes as level l + 1.  `seen`
// is -1 for nodes not reached yet.
__global__ void __launch_bounds__(256) k_tree_level(const DevNode* nodes, int n, int l, int* list, int* seen,
                                                    TreeCounts* tc) {
    const int begin = tc->first[l], end = begin + tc->count[l];
    if (blockIdx.x == 0 && threadIdx.x == 0) tc->first[l + 1] = end;
    int leaves = 0, tris = 0;
    for (int i0 = begin + blockIdx.x * 256; i0 < end; i0 += gridDim.x * 256) {
        const int i = i0 + (int)threadIdx.x;
        for (int s = 0; s < 2; ++s) {
            int c = -1;
            bool inner = false;
            if (i < end) {
                int cc[2];
                node_codes(nodes[list[i]], cc);
                c = cc[s];
                if (c < 0) {
                    const int start = ~c >> 3, count = (~c & 7) + 1;
                    if (start < 0 || start + count > n) tc->error = 1;
                    ++leaves;
                    tris += count;
                } else if (c >= n - 1 || atomicExch(&seen[c], 0) != -1) {
                    tc->error = 1;
                } else {
                    inner = true;
                }
            }
            const int at = warp_append(&tc->count[l + 1], inner);
            if (inner) list[end + at] = c;   // each node is reached once: below n - 1
        }
    }
    leaves = __reduce_add_sync(0xffffffffu, leaves);
    tris = __reduce_add_sync(0xffffffffu, tris);
    if (lane_id() == 0 && leaves) {
        atomicAdd(&tc->leaves, leaves);
        atomicAdd(&tc->leaf_tris, tris);
    }
}

// Internal nodes of each subtree, level by level from the last.
__global__ void __launch_bounds__(256) k_tree_inner(const DevNode* nodes, int l, const int* list, const TreeCounts* tc,
                                                    int* inner) {
    const int end = tc->first[l] + tc->count[l];
    for (int i = tc->first[l] + blockIdx.x * 256 + (int)threadIdx.x; i < end; i += gridDim.x * 256) {
        int c[2];
        node_codes(nodes[list[i]], c);
        inner[list[i]] = 1 + (c[0] >= 0 ? inner[c[0]] : 0) + (c[1] >= 0 ? inner[c[1]] : 0);
    }
}

// Depth-first places from the root down, and the nodes written there.
__global__ void __launch_bounds__(256) k_tree_place(const DevNode* nodes, int l, const int* list, const TreeCounts* tc,
                                                    const int* inner, int* place, DevNode* out) {
    const int end = tc->first[l] + tc->count[l];
    for (int i = tc->first[l] + blockIdx.x * 256 + (int)threadIdx.x; i < end; i += gridDim.x * 256) {
        DevNode nd = nodes[list[i]];
        const int p = l == 0 ? 0 : place[list[i]];
        int c[2];
        node_codes(nd, c);
        if (c[0] >= 0) {
            place[c[0]] = p + 1;
            nd.lmin_lc.w = __int_as_float(p + 1);
        }
        if (c[1] >= 0) {
            const int q = p + 1 + (c[0] >= 0 ? inner[c[0]] : 0);
            place[c[1]] = q;
            nd.lmax_rc.w = __int_as_float(q);
        }
        out[p] = nd;
    }
}

__global__ void k_wide_root(int root, int* list, TreeCounts* tc) {
    list[0] = root;
    tc->wide_count[0] = 1;
}

// One level of the 4-wide collapse: starting from a node's two children, the
// internal child with the largest box is replaced by its own two children
// until there are four (or only leaves).
__global__ void __launch_bounds__(256) k_wide_level(const DevNode* nodes, int l, int* list, TreeCounts* tc,
                                                    DevNode4* out) {
    const int begin = tc->wide_first[l], end = begin + tc->wide_count[l];
    if (blockIdx.x == 0 && threadIdx.x == 0) tc->wide_first[l + 1] = end;
    for (int i0 = begin + blockIdx.x * 256; i0 < end; i0 += gridDim.x * 256) {
        const int i = i0 + (int)threadIdx.x;
        float4 lo[4], hi[4];
        int code[4], cnt = 0, inner = 0;
        if (i < end) {
            const DevNode nd = nodes[list[i]];
            int c[2];
            node_codes(nd, c);
            lo[0] = nd.lmin_lc; hi[0] = nd.lmax_rc; code[0] = c[0];
            lo[1] = nd.rmin; hi[1] = nd.rmax; code[1] = c[1];
            cnt = 2;
            while (cnt < 4) {
                int best = -1;
                double ba = -1.0;
                for (int k = 0; k < cnt; ++k) {
                    if (code[k] < 0) continue;
                    const double dx = (double)hi[k].x - lo[k].x, dy = (double)hi[k].y - lo[k].y,
                                 dz = (double)hi[k].z - lo[k].z;
                    const double a = dx * dy + dy * dz + dz * dx;
                    if (a > ba) { ba = a; best = k; }
                }
                if (best < 0) break;
                const DevNode ch = nodes[code[best]];
                node_codes(ch, c);
                lo[best] = ch.lmin_lc; hi[best] = ch.lmax_rc; code[best] = c[0];
                lo[cnt] = ch.rmin; hi[cnt] = ch.rmax; code[cnt] = c[1];
                ++cnt;
            }
            for (int k = 0; k < cnt; ++k) inner += code[k] >= 0;
        }
        // one place range per node, siblings together
        int before = inner;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, before, o);
            if ((int)lane_id() >= o) before += y;
        }
        const int total = __shfl_sync(0xffffffffu, before, 31);
        int base = 0;
        if (lane_id() == 0 && total) base = atomicAdd(&tc->wide_count[l + 1], total);
        int at = end + __shfl_sync(0xffffffffu, base, 0) + before - inner;
        if (i >= end) continue;
        DevNode4 q;
        float* f[6] = {&q.xmin.x, &q.xmax.x, &q.ymin.x, &q.ymax.x, &q.zmin.x, &q.zmax.x};
        int out_code[4];
        for (int k = 0; k < 4; ++k) {
            const bool used = k < cnt;
            f[0][k] = used ? lo[k].x : 0.0f; f[1][k] = used ? hi[k].x : 0.0f;
            f[2][k] = used ? lo[k].y : 0.0f; f[3][k] = used ? hi[k].y : 0.0f;
            f[4][k] = used ? lo[k].z : 0.0f; f[5][k] = used ? hi[k].z : 0.0f;
            out_code[k] = !used ? kEmptyChild : code[k];
            if (used && code[k] >= 0) {
                list[at] = code[k];
                out_code[k] = at++;
            }
        }
        q.child = make_int4(out_code[0], out_code[1], out_code[2], out_code[3]);
        q.pad = make_int4(0, 0, 0, 0);
        out[i] = q;
    }
}

// ---------------------------------------------------------------- Engine
static inline cudaStream_t S(void* s) { return (cudaStream_t)s; }

Engine::Engine(int device) : device_(device) {
    ds_ = std::make_shared<DeviceScene>();
    pool_ = new PathPool();
}

Engine::~Engine() {
    async_stop();
    cudaSetDevice(device_);
    if (async_acc_) cudaFree(async_acc_);
    if (async_pinned_) cudaFreeHost(async_pinned_);
    if (jacc_) cudaFree(jacc_);
    job_end();
    delete guide_;
    ds_.reset();   // the device scene is freed with its last sharing engine
    if (pool_) { pool_->release(); delete pool_; }
    delete diag_dev_;
    for (void* e : render_ev_)
        if (e) cudaEventDestroy((cudaEvent_t)e);
    if (host_block_) pinned_give(host_block_);
    if (stream_) cudaStreamDestroy(S(stream_));
}

int Engine::device_info(char* buf, size_t cap) const {
    cudaDeviceProp prop;
    if (cudaGetDeviceProperties(&prop, device_) != cudaSuccess) return LUCID_ERR_CUDA;
    snprintf(buf, cap, "%s (sm_%d%d, %d SMs)", prop.name, prop.major, prop.minor, prop.multiProcessorCount);
    return LUCID_OK;
}

int Engine::set_camera(float px, float py, float pz, float dx, float dy, float dz, float ux, float uy, float uz,
                       float fov_deg) {
    GpuLock gl(*this);
    make_camera(cam_, px, py, pz, dx, dy, dz, ux, uy, uz, fov_deg);
    const float raw[10] = {px, py, pz, dx, dy, dz, ux, uy, uz, fov_deg};
    std::memcpy(cam_raw_, raw, sizeof(cam_raw_));
    camera_set_ = true;
    return LUCID_OK;
}

int Engine::set_algorithm(const char* name) {
    GpuLock gl(*this);
    std::string a = name ? name : "";
    if (a == "simple") algo_ = ALGO_SIMPLE;
    else if (a == "mis") algo_ = ALGO_MIS;
    else if (a == "volume_simple") algo_ = ALGO_VOLUME_SIMPLE;
    else if (a == "volume_mis") algo_ = ALGO_VOLUME_MIS;
    else algo_ = ALGO_NEE;   // the reference's dispatch falls through to traceNEE
    return LUCID_OK;
}

int Engine::set_wave_capacity(long long paths) {
    if (paths < 0) return fail(LUCID_ERR_INVALID, "wave capacity must be >= 0");
    wave_cap_ = paths;
    return LUCID_OK;
}

int Engine::scene_stats(int out8[8]) const {
    if (!scene_loaded_) return LUCID_ERR_NO_SCENE;
    scene_stats_locked(out8);
    return LUCID_OK;
}

void Engine::scene_stats_locked(int out8[8]) const {
    if (shared_) { std::memcpy(out8, shared_stats_, 8 * sizeof(int)); return; }
    int nvol = (int)host_.volumes.size();
    out8[0] = host_.num_meshes; out8[1] = host_.num_prims; out8[2] = host_.num_native;
    out8[3] = (int)host_.lights.size(); out8[4] = host_.num_boundary_meshes; out8[5] = nvol;
    out8[6] = bvh_nodes_; out8[7] = bvh_leaves_;
}

int Engine::stats(LucidRenderStats* out) const { *out = stats_; return LUCID_OK; }

// The next scene's arrays take the place of the last one's (allocating and
// freeing some twenty of them took 4 ms a load) unless another engine still
// uses it or it is an edited version of one (see upload_scene for a scene
// that does not fit beside them).
void Engine::free_scene() {
    if (ds_.use_count() > 1 || ds_->base) ds_ = std::make_shared<DeviceScene>();
    scene_loaded_ = false;
}

int Engine::ensure_stream() {
    if (stream_) return LUCID_OK;
    cudaStream_t s;
    CK(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    stream_ = s;
    cudaDeviceProp prop;
    CK(cudaGetDeviceProperties(&prop, device_));
    num_sms_ = prop.multiProcessorCount;
    return LUCID_OK;
}

int Engine::share_scene(Engine& owner) {
    SceneSnapshot snap;
    int rc = owner.snapshot_scene(snap);
    if (rc != LUCID_OK) return fail(rc, owner.last_error());
    return use_snapshot(snap);
}

int Engine::snapshot_scene(SceneSnapshot& out) {
    GpuLock gl(*this);
    if (!scene_loaded_) return fail(LUCID_ERR_NO_SCENE, "the sharing source has no scene");
    out.ds = ds_;
    scene_stats_locked(out.stats);
    for (int k = 0; k < 3; ++k) { out.lo[k] = scene_lo_[k]; out.hi[k] = scene_hi_[k]; }
    return LUCID_OK;
}

int Engine::use_snapshot(const SceneSnapshot& snap) {
    if (!snap.ds) return fail(LUCID_ERR_NO_SCENE, "empty scene snapshot");
    GpuLock gl(*this);
    CK(cudaSetDevice(device_));
    int rc = ensure_stream();
    if (rc != LUCID_OK) return rc;
    ds_ = snap.ds;
    std::memcpy(shared_stats_, snap.stats, sizeof(shared_stats_));
    for (int k = 0; k < 3; ++k) { scene_lo_[k] = snap.lo[k]; scene_hi_[k] = snap.hi[k]; }
    shared_ = true;
    scene_loaded_ = true;
    return LUCID_OK;
}

// A new scene version: the edited materials, lights, light CDF and guide,
// and per-prim shading classes in buffers of its own; the BVH, triangles and
// everything else are the current version's, which it keeps alive.  Engines
// rendering the current version keep it until they take the new one.
int Engine::update_scene(const LucidSceneEdit* edits, int count) {
    GpuLock gl(*this);
    if (!scene_loaded_) return fail(LUCID_ERR_NO_SCENE, "no scene loaded");
    if (shared_) return fail(LUCID_ERR_INVALID, "this context renders a scene it does not own; edit the owner");
    CK(cudaSetDevice(device_));
    std::string err;
    if (!apply_scene_edits(host_, edits, count, err)) return fail(LUCID_ERR_INVALID, err);
    const HostScene& H = host_;
    std::vector<unsigned char> cls(H.prim_info.size());
    for (size_t p = 0; p < cls.size(); ++p) cls[p] = prim_shading_class(H.materials[H.prim_info[p].x]);
    auto nv = std::make_shared<DeviceScene>();
    cudaStream_t st = S(stream_);
    auto up = [&](auto& buf, const auto& vec) -> cudaError_t {
        cudaError_t e = buf.alloc(vec.size());
        if (e != cudaSuccess || vec.empty()) return e;
        return cudaMemcpyAsync(buf.p, vec.data(), vec.size() * sizeof(vec[0]), cudaMemcpyHostToDevice, st);
    };
    CK(up(nv->materials, H.materials));
    CK(up(nv->lights, H.lights));
    CK(up(nv->light_bsph, native_light_bounds(H)));
    CK(up(nv->cdf, H.cdf));
    CK(up(nv->guide, H.light_guide));
    CK(up(nv->prim_cls, cls));
    CK(cudaStreamSynchronize(st));   // complete before any other stream reads the version
    nv->view = ds_->view;
    nv->view.materials = nv->materials.p;
    nv->view.lights = nv->lights.p;
    nv->view.light_bsph = H.num_native > 0 ? nv->light_bsph.p : nullptr;
    nv->view.light_cdf = nv->cdf.p;
    nv->view.light_guide = nv->guide.p;
    nv->view.prim_cls = nv->prim_cls.p;
    nv->view.total_light_area = H.total_light_area;
    nv->base = ds_;
    ds_ = nv;
    return LUCID_OK;
}

int Engine::load_scene_json(const char* json, size_t len) {
    GpuLock gl(*this);
    CK(cudaSetDevice(device_));
    {
        int rc = ensure_stream();
        if (rc != LUCID_OK) return rc;
    }
    shared_ = false;
    HostScene hs;
    std::string err;
    free_scene();
    if (!parse_scene_json(json, len, hs, err)) {
        ds_->release();
        return fail(LUCID_ERR_INVALID, err);
    }
    return upload_scene(std::move(hs));
}

int Engine::load_scene_arrays(const LucidSceneDesc& desc) {
    GpuLock gl(*this);
    CK(cudaSetDevice(device_));
    {
        int rc = ensure_stream();
        if (rc != LUCID_OK) return rc;
    }
    shared_ = false;
    HostScene hs;
    std::string err;
    free_scene();
    if (!build_scene_arrays(desc, hs, err)) {
        ds_->release();
        return fail(LUCID_ERR_INVALID, err);
    }
    return upload_scene(std::move(hs));
}

// Uploads a flattened scene and builds its BVH (the caller holds the GPU
// lock with the device current and the stream created).  Where the last
// scene's arrays leave too little memory the upload starts again without
// them, and a load that fails keeps none.
int Engine::upload_scene(HostScene&& hs) {
    host_ = std::move(hs);
    int rc = upload_host_scene();
    if (rc == LUCID_ERR_OOM) {
        cudaGetLastError();   // the failed allocation's, which the next launch check would take for its own
        ds_->release();
        rc = upload_host_scene();
    }
    if (rc != LUCID_OK) {
        cudaGetLastError();
        ds_->release();
    }
    return rc;
}

// What a no-allocation render launches, launched once per device with nothing
// to do: the first launch of a kernel loads its code, and the first with a
// larger stack than any before it makes the driver allocate local memory for
// every thread the device can hold (120 MB for k_paths).  Both would be device
// allocations of the first render_noalloc call (and fail it where another
// allocator holds the rest).  Without the memory the load succeeds all the
// same: a render may find more of it.
static void reserve_kernel_memory(int device, cudaStream_t st) {
    static std::mutex mu;
    static bool done[64] = {};
    std::lock_guard<std::mutex> lk(mu);
    if (device < 0 || device >= 64 || done[device]) return;
    for (int algo = 0; algo < 5; ++algo)
        paths_kernel<false>(algo)<<<1, kPathsThreads, 0, st>>>(DevScene{}, FrameParams{}, PathView{}, nullptr, 0, 0, 0, 0,
                                                               -1, nullptr);
    k_film<<<1, 32, 0, st>>>(0, 0, nullptr, nullptr);
    k_output<<<1, 32, 0, st>>>(0, 0, nullptr, nullptr);
    done[device] = cudaGetLastError() == cudaSuccess;
}

// The first boundary-only prim from p on; num_prims when there is none.
static int next_boundary(const HostScene& H, int p) {
    if (H.num_boundary_meshes == 0 || p >= H.num_prims) return H.num_prims;
    const unsigned char* const b = H.prim_boundary.data();
    const void* q = std::memchr(b + p, 1, (size_t)(H.num_prims - p));
    return q ? (int)(static_cast<const unsigned char*>(q) - b) : H.num_prims;
}

int Engine::upload_host_scene() {
    DeviceScene& D = *ds_;
    const HostScene& H = host_;
    // boundary triangles (brute force list) and per-prim shading data
    std::vector<float4> bnd;
    for (int p = next_boundary(H, 0); p < H.num_prims; p = next_boundary(H, p + 1))
        for (int k = 0; k < 3; ++k) bnd.push_back(H.tri[3 * p + k]);
    auto up = [&](auto& buf, const auto& vec) -> cudaError_t {
        cudaError_t e = buf.fit(vec.size());
        if (e != cudaSuccess) return e;
        if (vec.empty()) return cudaSuccess;
        return cudaMemcpyAsync(buf.p, vec.data(), vec.size() * sizeof(vec[0]), cudaMemcpyHostToDevice, S(stream_));
    };
    CK(up(D.bnd_tris, bnd));
    CK(up(D.prim_info, H.prim_info));
    CK(up(D.prim_vn, H.prim_vn));
    CK(D.prim_fn.fit(H.prim_fn.size()));       // k_prim_values
    CK(D.prim_cls.fit(H.prim_info.size()));
    CK(up(D.materials, H.materials));
    CK(up(D.tex_ops, H.tex_ops));
    CK(up(D.prim_uv, H.prim_uv));
    CK(up(D.lights, H.lights));
    CK(up(D.light_bsph, native_light_bounds(H)));
    CK(up(D.cdf, H.cdf));
    CK(up(D.guide, H.light_guide));
    CK(up(D.volumes, H.volumes));
    CK(up(D.grid, H.grid));
    DevScene& v = D.view;
    v = DevScene{};
    v.bnd_tris = D.bnd_tris.p;
    v.num_bnd_tris = (int)(bnd.size() / 3);
    v.prim_info = D.prim_info.p;
    v.prim_cls = D.prim_cls.p;
    v.prim_fn = D.prim_fn.p;
    v.prim_vn = D.prim_vn.p;
    v.materials = D.materials.p;
    v.tex_ops = H.tex_ops.empty() ? nullptr : D.tex_ops.p;
    v.prim_uv = H.prim_uv.empty() ? nullptr : D.prim_uv.p;
    v.lights = D.lights.p;
    v.light_cdf = D.cdf.p;
    v.light_guide = D.guide.p;
    v.num_lights = (int)H.lights.size();
    v.native_start = H.native_start;
    v.num_native = H.num_native;
    v.light_bsph = H.num_native > 0 ? D.light_bsph.p : nullptr;
    v.total_light_area = H.total_light_area;
    for (int k = 0; k < 3; ++k) v.env[k] = H.env[k];
    v.volumes = D.volumes.p;
    v.num_volumes = (int)H.volumes.size();
    v.grid = D.grid.p;
    v.has_boundary = v.num_bnd_tris > 0;
    int rc = build_bvh();
    if (rc != LUCID_OK) return rc;
    reserve_kernel_memory(device_, S(stream_));
    CK(cudaStreamSynchronize(S(stream_)));
    scene_loaded_ = true;
    return LUCID_OK;
}

// PLOC rounds on the device; the host reads one word per round to know the
// surviving cluster count.  Returns LUCID_OK with root = -1 when the
// clustering needs more than kPlocMaxRounds rounds (the caller then builds
// the Karras tree instead).
int Engine::build_ploc(void* arena, const float4* verts, const int* sorted_ids, int n, int2* child, int2* range,
                       float* nbox, int* slot_ids, int& root) {
    DeviceArena& A = *static_cast<DeviceArena*>(arena);
    constexpr int kPlocMaxRounds = 4096;
    cudaStream_t st = S(stream_);
    root = -1;
    int* cl[2] = {A.take<int>(n), A.take<int>(n)};
    float* cb[2] = {A.take<float>((size_t)6 * n), A.take<float>((size_t)6 * n)};
    int *nn = A.take<int>(n), *cnt_leaf = A.take<int>(n), *cnt_node = A.take<int>(n), *off_node = A.take<int>(n),
        *leaf_pos = A.take<int>(n);
    unsigned long long *flags = A.take<unsigned long long>(n), *pos = A.take<unsigned long long>(n),
                       *d_totals = A.take<unsigned long long>(1);
    size_t temp = 0;
    CK(cub::DeviceScan::ExclusiveSum(nullptr, temp, flags, pos, n, st));
    unsigned char* d_temp = A.take<unsigned char>(temp);
    if (!d_temp) return fail(LUCID_ERR_OOM, "BVH build: temporaries exceed their estimate");
    k_ploc_init<<<(n + 255) / 256, 256, 0, st>>>(verts, sorted_ids, n, cl[0], cb[0], cnt_leaf);
    int cur = 0, count = n, base = 0;
    std::vector<std::pair<int, int>> rounds;
    while (count > 1) {
        if ((int)rounds.size() >= kPlocMaxRounds) return LUCID_OK;
        k_ploc_nn<<<(count + kPlocBlock - 1) / kPlocBlock, kPlocBlock, 0, st>>>(cb[cur], count, nn);
        k_ploc_flags<<<(count + 255) / 256, 256, 0, st>>>(nn, count, flags);
        size_t t1 = temp;
        CK(cub::DeviceScan::ExclusiveSum(d_temp, t1, flags, pos, count, st));
        k_ploc_merge<<<(count + 255) / 256, 256, 0, st>>>(cl[cur], cb[cur], nn, flags, pos, count, base, child, nbox,
                                                         cnt_node, cnt_leaf, cl[cur ^ 1], cb[cur ^ 1], d_totals);
        CK(cudaGetLastError());
        unsigned long long* const word = static_cast<unsigned long long*>(host_block_);
        CK(cudaMemcpyAsync(word, d_totals, sizeof(unsigned long long), cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        const int m = (int)(*word >> 32), survivors = (int)(*word & 0xffffffffull);
        if (m <= 0 || survivors != count - m) return fail(LUCID_ERR_CUDA, "BVH clustering made no progress");
        rounds.push_back({base, m});
        base += m;
        count = survivors;
        cur ^= 1;
    }
    if (base != n - 1) return fail(LUCID_ERR_CUDA, "BVH clustering produced a wrong node count");
    const int r = n - 2;   // the last node created is the root
    CK(cudaMemsetAsync(off_node + r, 0, sizeof(int), st));
    for (auto it = rounds.rbegin(); it != rounds.rend(); ++it)
        k_ploc_offsets<<<(it->second + 255) / 256, 256, 0, st>>>(child, cnt_node, it->first, it->second, off_node,
                                                                 leaf_pos);
    k_ploc_finish<<<(n + 255) / 256, 256, 0, st>>>(sorted_ids, leaf_pos, n, child, off_node, cnt_node, range, slot_ids);
    CK(cudaGetLastError());
    ploc_rounds_ = (int)rounds.size();
    root = r;
    return LUCID_OK;
}

int Engine::build_bvh() {
    DeviceScene& D = *ds_;
    const HostScene& H = host_;
    cudaStream_t st = S(stream_);
    const int np = H.num_prims;
    static_assert(sizeof(TreeCounts) <= kPinnedBytes, "what a build reads back");
    if (!host_block_) CK(pinned_take(&host_block_));
    size_t sort_temp = 0, scan_temp = 0, select_temp = 0;
    CK(cub::DeviceRadixSort::SortPairs(nullptr, sort_temp, (unsigned long long*)nullptr, (unsigned long long*)nullptr,
                                       (int*)nullptr, (int*)nullptr, np, 0, 63, st));
    CK(cub::DeviceScan::ExclusiveSum(nullptr, scan_temp, (unsigned long long*)nullptr, (unsigned long long*)nullptr, np, st));
    CK(cub::DeviceSelect::If(nullptr, select_temp, thrust::make_counting_iterator(0), (int*)nullptr, (int*)nullptr, np,
                             InBvh{}, st));
    // per triangle: vertices 48, ids, keys, values and flags 29, children,
    // ranges, boxes and slots 44, clustering 92, flattened nodes, levels,
    // subtree sizes and places 76, the Karras fallback's 12; each array
    // rounded to 256 bytes
    constexpr int kCandidates = 4096;
    DeviceArena A;
    CK(A.reserve((size_t)np * 301 + sort_temp + scan_temp + select_temp + H.materials.size() + (128 << 10)));
    float4* d_verts = A.take<float4>((size_t)3 * np);
    unsigned char *d_boundary = A.take<unsigned char>(np), *d_mesh_cls = A.take<unsigned char>(H.materials.size());
    PrimBounds* d_pb = A.take<PrimBounds>(1);
    int2* d_cand = A.take<int2>(kCandidates);
    if (!d_cand) return fail(LUCID_ERR_OOM, "BVH build: temporaries exceed their estimate");
    CK(cudaMemcpyAsync(d_verts, H.verts.data(), H.verts.size() * sizeof(float4), cudaMemcpyHostToDevice, st));
    CK(cudaMemcpyAsync(d_boundary, H.prim_boundary.data(), (size_t)np, cudaMemcpyHostToDevice, st));
    // Scene bounds, then split off the largest triangles: at most kMaxBig
    // whose bounding-box diagonal exceeds a quarter of the scene's.
    float lo[3] = {1e30f, 1e30f, 1e30f}, hi[3] = {-1e30f, -1e30f, -1e30f};
    float maxabs = 0.0f;
    PrimBounds* const pb = static_cast<PrimBounds*>(host_block_);
    if (np > 0) {
        // each prim's shading class for a surface hit (the material part of
        // bin_class) is decided once here instead of per hit
        std::vector<unsigned char> mesh_cls(H.materials.size());
        for (size_t k = 0; k < mesh_cls.size(); ++k) mesh_cls[k] = prim_shading_class(H.materials[k]);
        CK(cudaMemcpyAsync(d_mesh_cls, mesh_cls.data(), mesh_cls.size(), cudaMemcpyHostToDevice, st));
        k_prim_values<<<(np + 255) / 256, 256, 0, st>>>(d_verts, D.prim_info.p, d_mesh_cls, np, D.prim_fn.p, D.prim_cls.p);
        for (int a = 0; a < 3; ++a) { pb->lo[a] = ord_f(lo[a]); pb->hi[a] = ord_f(hi[a]); }
        pb->maxabs = ord_f(0.0f);
        pb->big = 0;
        CK(cudaMemcpyAsync(d_pb, pb, sizeof(PrimBounds), cudaMemcpyHostToDevice, st));
        k_prim_bounds<<<std::min(4 * num_sms_, (np + 255) / 256), 256, 0, st>>>(d_verts, d_boundary, np, d_pb);
        CK(cudaMemcpyAsync(pb, d_pb, sizeof(PrimBounds), cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        for (int a = 0; a < 3; ++a) { lo[a] = unord_f(pb->lo[a]); hi[a] = unord_f(pb->hi[a]); }
        maxabs = unord_f(pb->maxabs);
    }
    // secondary-ray origins lie on triangles (boundary ones included) or
    // inside volume boxes: all of them bound the FMA slab test's error
    for (const DevVolume& vol : H.volumes)
        for (int a = 0; a < 3; ++a)
            maxabs = std::max(maxabs, std::max(std::fabs(vol.wmin[a]), std::fabs(vol.wmax[a])));
    for (int a = 0; a < 3; ++a) { scene_lo_[a] = lo[a]; scene_hi_[a] = hi[a]; }
    {
        // boundary-only triangles grouped by mesh (they are stored in prim
        // order), each group with its bounding box padded as the BVH's boxes
        std::vector<float4> boxes;
        const float bpad = maxabs * 9.5367431640625e-07f + 1e-30f;
        int k = 0;
        for (int p = next_boundary(H, 0); p < np; p = next_boundary(H, p + 1)) {
            const int mesh = H.prim_info[(size_t)p].x;
            bool fresh = boxes.empty();
            if (!fresh) {
                int last_mesh;
                std::memcpy(&last_mesh, &boxes[boxes.size() - 1].w, 4);   // scratch: mesh id of the open group
                fresh = last_mesh != mesh;
            }
            if (fresh) {
                float first;
                std::memcpy(&first, &k, 4);
                float m;
                std::memcpy(&m, &mesh, 4);
                boxes.push_back(make_float4(1e30f, 1e30f, 1e30f, first));
                boxes.push_back(make_float4(-1e30f, -1e30f, -1e30f, m));
            }
            float4& blo = boxes[boxes.size() - 2];
            float4& bhi = boxes[boxes.size() - 1];
            for (int c = 0; c < 3; ++c) {
                const float4& q = H.verts[3 * p + c];
                blo.x = std::min(blo.x, q.x); blo.y = std::min(blo.y, q.y); blo.z = std::min(blo.z, q.z);
                bhi.x = std::max(bhi.x, q.x); bhi.y = std::max(bhi.y, q.y); bhi.z = std::max(bhi.z, q.z);
            }
            ++k;
        }
        // close the groups: pad the boxes, replace the mesh id by the count
        for (size_t g = 0; g < boxes.size(); g += 2) {
            int first, next;
            std::memcpy(&first, &boxes[g].w, 4);
            if (g + 2 < boxes.size()) std::memcpy(&next, &boxes[g + 2].w, 4);
            else next = k;
            const int count = next - first;
            boxes[g].x -= bpad; boxes[g].y -= bpad; boxes[g].z -= bpad;
            boxes[g + 1].x += bpad; boxes[g + 1].y += bpad; boxes[g + 1].z += bpad;
            std::memcpy(&boxes[g + 1].w, &count, 4);
        }
        DeviceScene& Db = D;
        cudaError_t e = Db.bnd_box.fit(std::max<size_t>(1, boxes.size()));
        if (e != cudaSuccess) return fail(LUCID_ERR_OOM, "boundary box allocation failed");
        if (!boxes.empty())
            CK(cudaMemcpyAsync(Db.bnd_box.p, boxes.data(), boxes.size() * sizeof(float4), cudaMemcpyHostToDevice,
                               S(stream_)));
        Db.view.bnd_box = boxes.empty() ? nullptr : Db.bnd_box.p;
        Db.view.num_bnd_groups = (int)(boxes.size() / 2);
        if (k != Db.view.num_bnd_tris) return fail(LUCID_ERR_CUDA, "boundary triangle groups do not cover the list");
    }
    float sdiag = std::sqrt((hi[0] - lo[0]) * (hi[0] - lo[0]) + (hi[1] - lo[1]) * (hi[1] - lo[1]) +
                            (hi[2] - lo[2]) * (hi[2] - lo[2]));
    const int nonbnd = np - D.view.num_bnd_tris;
    std::vector<std::pair<float, int>> cand;   // (diagonal, prim)
    if (np > 0) {
        k_big_candidates<<<(np + 255) / 256, 256, 0, st>>>(d_verts, d_boundary, np, 0.25f * sdiag, kCandidates, d_pb, d_cand);
        std::vector<int2> found(kCandidates);
        CK(cudaMemcpyAsync(pb, d_pb, sizeof(PrimBounds), cudaMemcpyDeviceToHost, st));
        CK(cudaMemcpyAsync(found.data(), d_cand, kCandidates * sizeof(int2), cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        if (pb->big <= kCandidates) {
            for (int k = 0; k < pb->big; ++k) {
                float d;
                std::memcpy(&d, &found[(size_t)k].y, 4);
                cand.push_back({d, found[(size_t)k].x});
            }
        } else {   // more than the list holds: all of them, on the host
            for (int p = 0; p < np; ++p) {
                if (H.prim_boundary[p]) continue;
                float pl[3] = {1e30f, 1e30f, 1e30f}, ph[3] = {-1e30f, -1e30f, -1e30f};
                for (int k = 0; k < 3; ++k) {
                    const float4& q = H.verts[3 * (size_t)p + k];
                    const float c[3] = {q.x, q.y, q.z};
                    for (int a = 0; a < 3; ++a) { pl[a] = std::min(pl[a], c[a]); ph[a] = std::max(ph[a], c[a]); }
                }
                const float d = std::sqrt((ph[0] - pl[0]) * (ph[0] - pl[0]) + (ph[1] - pl[1]) * (ph[1] - pl[1]) +
                                          (ph[2] - pl[2]) * (ph[2] - pl[2]));
                if (d > 0.25f * sdiag) cand.push_back({d, p});
            }
        }
    }
    std::sort(cand.begin(), cand.end(), [](const auto& a, const auto& b) {
        return a.first > b.first || (a.first == b.first && a.second < b.second);
    });
    if ((int)cand.size() > kMaxBig) cand.resize(kMaxBig);
    // keep at least one triangle in the BVH so tiny scenes still build one
    if ((int)cand.size() == nonbnd) cand.clear();
    std::vector<int> bigc;
    for (const auto& c : cand) bigc.push_back(c.second);
    std::sort(bigc.begin(), bigc.end());
    std::vector<float4> big;
    for (int p : bigc)
        for (int k = 0; k < 3; ++k) big.push_back(H.tri[3 * (size_t)p + k]);
    const int n = nonbnd - (int)bigc.size();
    DevScene& v = D.view;
    v.coord_bound = maxabs;
    for (int a = 0; a < 3; ++a) {
        const float ext = hi[a] - lo[a];
        v.bin_lo[a] = ext > 0.0f ? lo[a] : 0.0f;
        v.bin_scale[a] = ext > 0.0f ? (float)kCellDim / ext : 0.0f;
    }
    {
        cudaError_t e = D.big_tris.fit(big.size());
        if (e != cudaSuccess) return fail(LUCID_ERR_OOM, "big triangle list allocation failed");
        if (!big.empty())
            CK(cudaMemcpyAsync(D.big_tris.p, big.data(), big.size() * sizeof(float4), cudaMemcpyHostToDevice, S(stream_)));
        v.big_tris = D.big_tris.p;
        v.num_big_tris = (int)(big.size() / 3);
        num_big_ = v.num_big_tris;
    }
    v.num_bvh_tris = n;
    bvh_nodes_ = 0; bvh_leaves_ = 0; bvh_depth_ = 0;
    if (n == 0) { v.root = v.root2 = 0; v.nodes = nullptr; v.nodes2 = nullptr; v.bvh_tris = nullptr; return LUCID_OK; }
    int *d_ids = A.take<int>(n), *d_vals = A.take<int>(n), *d_vals_sorted = A.take<int>(n), *d_bounds = A.take<int>(6),
        *d_num = A.take<int>(1);
    unsigned long long *d_keys = A.take<unsigned long long>(n), *d_keys_sorted = A.take<unsigned long long>(n);
    unsigned char *d_temp = A.take<unsigned char>(sort_temp), *d_select = A.take<unsigned char>(select_temp);
    if (!d_select) return fail(LUCID_ERR_OOM, "BVH build: temporaries exceed their estimate");
    InBvh in_bvh{};
    in_bvh.boundary = d_boundary;
    in_bvh.nbig = (int)bigc.size();
    for (size_t k = 0; k < bigc.size(); ++k) in_bvh.big[k] = bigc[k];
    CK(cub::DeviceSelect::If(d_select, select_temp, thrust::make_counting_iterator(0), d_ids, d_num, np, in_bvh, st));
    int init[6] = {0x7fffffff, 0x7fffffff, 0x7fffffff, (int)0x80000000, (int)0x80000000, (int)0x80000000};
    CK(cudaMemcpyAsync(d_bounds, init, sizeof(init), cudaMemcpyHostToDevice, st));
    k_centroid_bounds<<<std::max(1, std::min(4 * num_sms_, (n + 127) / 128)), 128, 0, st>>>(d_verts, d_ids, n, d_bounds);
    k_morton<<<(n + 255) / 256, 256, 0, st>>>(d_verts, d_ids, n, d_bounds, d_keys, d_vals);
    CK(cub::DeviceRadixSort::SortPairs(d_temp, sort_temp, d_keys, d_keys_sorted, d_vals, d_vals_sorted, n, 0, 63, st));
    CK(D.bvh_tris.fit((size_t)4 * n));
    v.bvh_tris = D.bvh_tris.p;
    if (n <= 4) {
        k_gather_tris<<<(n + 255) / 256, 256, 0, st>>>(d_verts, d_vals_sorted, n, D.bvh_tris.p);
        v.root = leaf_code(0, n);
        v.root2 = v.root;
        v.nodes = nullptr;
        v.nodes2 = nullptr;
        bvh_leaves_ = 1;
        CK(cudaGetLastError());
        CK(cudaStreamSynchronize(st));
        return LUCID_OK;
    }
    int2 *d_child = A.take<int2>(n), *d_range = A.take<int2>(n);
    float* d_nbox = A.take<float>((size_t)6 * n);
    int* d_slot = A.take<int>(n);
    int root = -1;
    int rc = build_ploc(&A, d_verts, d_vals_sorted, n, d_child, d_range, d_nbox, d_slot, root);
    if (rc != LUCID_OK) return rc;
    const bool ploc = root >= 0;
    const int* slot_ids = ploc ? d_slot : d_vals_sorted;
    if (!ploc) {   // Karras LBVH: the fallback when clustering does not converge
        int *d_parent = A.take<int>(n), *d_leaf_parent = A.take<int>(n), *d_arrive = A.take<int>(n);
        if (!d_arrive) return fail(LUCID_ERR_OOM, "BVH build: temporaries exceed their estimate");
        CK(cudaMemsetAsync(d_parent, 0xff, (n - 1) * sizeof(int), st));   // root's parent = -1
        CK(cudaMemsetAsync(d_arrive, 0, (n - 1) * sizeof(int), st));
        k_karras<<<(n - 1 + 255) / 256, 256, 0, st>>>(d_keys_sorted, n, d_child, d_parent, d_leaf_parent, d_range);
        k_refit<<<(n + 255) / 256, 256, 0, st>>>(d_verts, d_vals_sorted, n, d_child, d_parent, d_leaf_parent, d_arrive,
                                                d_nbox);
        root = 0;
    }
    k_gather_tris<<<(n + 255) / 256, 256, 0, st>>>(d_verts, slot_ids, n, D.bvh_tris.p);
    const float pad = maxabs * 9.5367431640625e-07f + 1e-30f;   // 2^-20 of the scene's coordinate magnitude
    DevNode* d_flat = A.take<DevNode>(n);
    int *d_list = A.take<int>(n), *d_inner = A.take<int>(n), *d_place = A.take<int>(n);
    TreeCounts* d_tc = A.take<TreeCounts>(1);
    if (!d_tc) return fail(LUCID_ERR_OOM, "BVH build: temporaries exceed their estimate");
    k_flatten<<<(n - 1 + 255) / 256, 256, 0, st>>>(d_verts, slot_ids, n, d_child, d_range, d_nbox, pad, d_flat);

    // Levels of the flattened tree from the root.  The walk also validates
    // the hierarchy before any traversal kernel uses it: child indices in
    // range, leaf ranges inside the triangle array, no node reached twice,
    // every triangle in one leaf.  d_inner (subtree sizes) marks the nodes
    // reached until it is filled.
    TreeCounts* const tc = static_cast<TreeCounts*>(host_block_);
    CK(cudaMemsetAsync(d_inner, 0xff, (size_t)n * sizeof(int), st));
    CK(cudaMemsetAsync(d_tc, 0, sizeof(TreeCounts), st));
    k_tree_root<<<1, 1, 0, st>>>(root, n, d_list, d_inner, d_tc);
    const int g = num_sms_ * 2;
    int levels = 0;
    for (int l = 0; levels == 0 && l < kTreeLevels;) {
        for (const int end = std::min(kTreeLevels, l + 32); l < end; ++l)   // (levels past the last are empty)
            k_tree_level<<<g, 256, 0, st>>>(d_flat, n, l, d_list, d_inner, d_tc);
        CK(cudaGetLastError());
        CK(cudaMemcpyAsync(tc, d_tc, sizeof(TreeCounts), cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        if (tc->error) return fail(LUCID_ERR_CUDA, "BVH build produced an invalid hierarchy");
        while (levels < l && tc->count[levels] > 0) ++levels;
        if (levels == l) levels = 0;   // more to come
    }
    if (levels == 0 || levels + 1 >= kStack)
        return fail(LUCID_ERR_OVERFLOW, "BVH depth " + std::to_string(levels + 1) + " exceeds the traversal stack");
    if (tc->leaf_tris != n) return fail(LUCID_ERR_CUDA, "BVH leaves do not cover every triangle");
    const int nodes = tc->first[levels - 1] + tc->count[levels - 1], leaves = tc->leaves, depth = levels + 1;
    // Binary nodes in depth-first order (a node, its left subtree, its right
    // subtree; root first): a ray's descent then reads nearby lines, and the
    // top of the tree shares a few cache lines.  Subtree sizes from the last
    // level up, places from the root down.
    CK(D.nodes2.fit((size_t)nodes));
    for (int l = levels - 1; l >= 0; --l) k_tree_inner<<<g, 256, 0, st>>>(d_flat, l, d_list, d_tc, d_inner);
    for (int l = 0; l < levels; ++l) k_tree_place<<<g, 256, 0, st>>>(d_flat, l, d_list, d_tc, d_inner, d_place, D.nodes2.p);
    // 4-wide collapse, a level at a time: node i of the collapse stands for
    // binary node d_list[i] (the levels' list is done with).  A 4-wide node with
    // inner children takes in three binary nodes and has at most four of them,
    // one without takes in one at least: (2 nodes + 1) / 3 at most (the
    // 1M-triangle scene has 159,152 for 320,882 binary nodes).
    CK(D.nodes.fit(((size_t)nodes * 2 + 1) / 3));
    k_wide_root<<<1, 1, 0, st>>>(root, d_list, d_tc);
    for (int l = 0; l < levels; ++l) k_wide_level<<<g, 256, 0, st>>>(d_flat, l, d_list, d_tc, D.nodes.p);
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(tc, d_tc, sizeof(TreeCounts), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    int levels4 = 0;
    while (levels4 < levels && tc->wide_count[levels4] > 0) ++levels4;
    const int nodes4 = tc->wide_first[levels4 - 1] + tc->wide_count[levels4 - 1], depth4 = levels4 + 1;
    v.nodes = D.nodes.p;
    v.root = 0;
    v.nodes2 = D.nodes2.p;
    v.root2 = 0;
    bvh_nodes_ = nodes4; bvh_leaves_ = leaves; bvh_depth_ = depth4;
    if (std::getenv("LUCID_VERBOSE"))
        std::fprintf(stderr, "[lucid] BVH %s (%d rounds): %d binary nodes, %d leaves, depth %d; %d 4-wide nodes, depth %d\n",
                     ploc ? "ploc" : "lbvh", ploc ? ploc_rounds_ : 0, nodes, leaves, depth, nodes4, depth4);
    if (3 * (depth4 - 1) >= kStack)
        return fail(LUCID_ERR_OVERFLOW, "BVH depth " + std::to_string(depth) + " exceeds the traversal stack");
    return LUCID_OK;
}

int Engine::ensure_pool(long long paths, bool records) {
    PathPool& P = *pool_;
    if (P.cap >= paths && (!records || P.records)) return LUCID_OK;
    long long cap = std::max(paths, P.cap);
    P.release();
    CK(P.st.alloc(cap)); CK(P.hit.alloc(cap)); CK(P.sh.alloc(cap)); CK(P.rad.alloc(cap));
    CK(P.q0.alloc(cap)); CK(P.q1.alloc(cap)); CK(P.qb.alloc(cap)); CK(P.cls.alloc(cap));
    CK(P.counters.alloc((size_t)kCountersPerDepth * (kMaxDepth + 1)));
    CK(P.errors.alloc(kErrorInts));
    if (records) { CK(P.rec_prim.alloc(cap)); CK(P.rec_cnt.alloc(cap)); CK(P.rec_hash.alloc(cap)); }
    P.cap = cap;
    P.records = records;
    PathView& v = P.view;
    v.st = P.st.p; v.hit = P.hit.p; v.sh = P.sh.p; v.rad = P.rad.p; v.q0 = P.q0.p; v.q1 = P.q1.p;
    v.qb = P.qb.p; v.cls = P.cls.p; v.counters = P.counters.p; v.errors = P.errors.p;
    v.rec_prim = P.rec_prim.p; v.rec_cnt = P.rec_cnt.p; v.rec_hash = P.rec_hash.p;
    return LUCID_OK;
}

namespace {
// Algorithmic bytes per unit of work (compulsory path traffic: the fields a
// kernel needs, not the whole 32-byte sectors of their records; BVH node and
// triangle fetches are scene-dependent and excluded):
//   trace : ray 32 + queue id 4 + hit 16 + light hit 8
//           + the hit prim's class 1 and the shading bin 2 (binning)   = 63 / ray
//   shade : queue 4 + hit 24 + ray 32 + throughput 16 + radiance 16 + rng 16
//           + prim info/normal 32 + material 48  (reads)
//           + rng 16 + radiance 16 + throughput 16 + ray 32 + queue 4
//           + shadow record 48, path id inside  (writes)            = 336 / path
//   shadow: shadow record 48 + queue 4 (first segment to traversal)
//           + radiance 16 read + 16 write                            = 84 / ray
//   raygen: rng 16 + ray 32 + throughput 16 + radiance 16            = 80 / path
//   camera trace (generates its rays): the raygen writes 80 + hit 16
//           + light hit 8 + prim class 1 + shading bin 2               = 107 / ray
//   film  : radiance 16 / path + film 32 / pixel
//   bin   : queue id 4 + shading bin 2 + binned id 4 (scatter)       = 10 / path
constexpr double kBytesTrace0 = 107, kBytesTrace = 63, kBytesShade = 336, kBytesShadow = 84, kBytesRaygen = 80, kBytesFilm = 16,
                 kBytesBin = 10, kBytesPaths = 80;
//   paths : prim info/normal 32 + material 48 per segment (the state stays in registers)
//   guide : queue 4 + hit 24 + ray 32 + raw outputs 160 w              = 220 / path
//   train : one record 64 / record (weights are read from shared memory)
enum Kind { K_RAYGEN, K_TRACE0, K_TRACE, K_SHADE, K_SHADOW, K_FILM, K_BIN, K_GUIDE, K_TRAIN, K_PATHS, K_NUM };
const char* kKindNames[K_NUM] = {"k_raygen", "k_trace_primary", "k_trace", "k_shade", "k_shadow", "k_film", "k_bin",
                                 "k_guide_infer", "k_guide_train", "k_paths"};
const double kKindBytes[K_NUM] = {kBytesRaygen, kBytesTrace0, kBytesTrace, kBytesShade, kBytesShadow, kBytesFilm,
                                  kBytesBin, 220, 64, kBytesPaths};
static_assert(K_NUM <= LUCID_MAX_KERNEL_KINDS, "kernel kinds");
}  // namespace

// ---------------------------------------------------------------- waves
// One wave: the wavefront kernels of `depths` depths (camera rays, then per
// depth trace, bin, shade, shadow), then k_paths for what is left of the
// paths.  A depth > 0 whose queue holds at most `stop` paths leaves them to
// k_paths at once: the remaining launches of the wave return on reading the
// queue length.  depths 0: every path runs in k_paths from its camera ray.
// stop < 0: no k_paths (guided renders; a single depth).
//
// Four launches of a depth take 65-80 us however few paths are queued (each
// waits for its slowest ray), so small queues are better followed to the end
// by one kernel.  The line is 2^17 paths, two thirds of what k_paths keeps
// resident: a 26k- and a 77k-path wave of the all-lights scene take 582 us
// in k_paths and 798 us with the wavefront first; the 480k paths of an
// 800x600 frame 887 us in k_paths alone against 787 us; of `stop` = 2^15,
// 2^16, 2^17, 2^18, 2^19 the volume frame (333x207, 5 spp, depth 16) takes
// 1.05, 1.06, 1.06, 1.40, 1.39 ms and the 1M-triangle frame (960x540, 4 spp,
// depth 16) 5.34, 5.08, 5.12, 5.08, 5.36 ms (2.09 and 7.3 ms with every
// depth launched).  `depths` bounds the launches of a wave whose queue
// shrinks as usual (two depths, and one more for each doubling from 2^19
// paths on); where it shrinks more slowly k_paths takes a longer queue.  Of
// such waves closed rooms with walls of albedo 0.95 and 0.99 (26 and
// 43,214 triangles, `simple` and `mis`) were measured at depths 8, 16, 32 and 64
// and 2^20, 2^22 and 2^23 paths: 1.15 to 2.4 times as fast as the kernels before
// k_paths with every depth launched (the tessellated room, `mis`, depth 64,
// 2^23 paths: 37.9 against 52.3 ms).
constexpr long long kPathsWave = Engine::kPathsWave;
struct WavePlan {
    LaunchSet ks;
    PathsKernel paths;
    int g_trace0 = 1, g_trace = 1, g_shade = 1, g_shadow = 1, g_bin = 1, g_paths = 1, g_post = 1;   // blocks
    int depths = 0, stop = -1;
    int bins = 0;    // shading bins (BinHist)
};
static WavePlan wave_plan(int device, int sms, int algo, bool guide, int profile, bool batch, long long paths,
                          int max_depth) {
    WavePlan w;
    w.ks = batch ? launch_set_batch(algo) : launch_set(algo, guide, profile);
    w.paths = batch ? paths_kernel<true>(algo) : paths_kernel<false>(algo);
    // the kernels' resident blocks per SM, queried once per device and set
    static std::mutex mu;
    static std::map<int, std::array<int, 5>>* occ = new std::map<int, std::array<int, 5>>();
    {
        std::lock_guard<std::mutex> lk(mu);
        std::array<int, 5>& o = (*occ)[((device * 8 + algo) * 2 + (guide ? 1 : 0)) * 4 + profile * 2 + (batch ? 1 : 0)];
        if (o[0] == 0) {
            auto query = [&](auto kernel, int threads) {
                int n = 1;
                cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, 0);
                return std::max(1, n);
            };
            o[1] = query(w.ks.trace, 128);
            o[2] = query(w.ks.shade, kShadeThreads);
            o[3] = query(w.ks.shadow, 128);
            o[4] = query(w.paths, kPathsThreads);
            o[0] = batch ? query(k_trace_primary_batch, 128) : query(k_trace_primary_t<false>, 128);
        }
        w.g_trace0 = sms * o[0];
        w.g_trace = sms * o[1];
        w.g_shade = sms * o[2];
        w.g_shadow = sms * o[3];
        w.g_paths = sms * o[4];
    }
    w.g_bin = sms * 8;
    w.g_post = sms * 4;
    w.bins = ((algo == ALGO_VOLUME_MIS || algo == ALGO_VOLUME_SIMPLE) ? kBinVolume : 0) |
             (paths >= kCellBinPaths ? kBinCells : 0);
    w.depths = std::max(0, max_depth);
    if (guide || max_depth < 1) return w;
    if (paths <= kPathsWave) {
        w.depths = 0;
    } else {
        int d = 2;
        for (long long p = paths >> 19; p > 0; p >>= 1) ++d;
        w.depths = std::min(max_depth, d);
        if (max_depth > 1) w.stop = (int)kPathsWave;
    }
    return w;
}

// k_paths for what the wavefront leaves of a wave (all of it where depths is 0).
template <class Mark>
static void enqueue_paths(const WavePlan& w, const DevScene& sc, const FrameParams& f, const PathView& base,
                          cudaStream_t st, Mark mark, const BatchJob* jobs, int njobs, int slots) {
    PathsCount* pc = reinterpret_cast<PathsCount*>(base.errors + 4);
    int grid = w.g_paths, fma0 = 0;
    if (!jobs) {
        const float m = std::max(std::fabs(f.pos[0]), std::max(std::fabs(f.pos[1]), std::fabs(f.pos[2])));
        fma0 = m <= sc.coord_bound;
        if (w.depths == 0)
            slots = ((f.tile_w + 7) / 8) * ((f.tile_h + 3) / 4) * 32 * (f.n_wave / std::max(f.npix, 1));
    }
    constexpr int kBlockLanes = kMinLanes * kPathsThreads / 32;
    if (w.depths == 0) grid = std::min(grid, (slots + kBlockLanes - 1) / kBlockLanes);
    cudaMemsetAsync(pc, 0, sizeof(PathsCount), st);
    mark(K_PATHS, w.depths, 1, [&] {
        w.paths<<<grid, kPathsThreads, 0, st>>>(sc, f, base, jobs, njobs, slots, fma0, w.depths, w.stop, pc);
    });
}

// Launches one wave.  primary(pv, cnt): the camera-ray kernel; infer(depth,
// pv, cnt, queue): guide inference before a depth's shading; mark(kind,
// depth, kernels, launch): runs a step's launches (inside profiling events).
template <class Primary, class Infer, class Mark>
static void enqueue_wave(const WavePlan& w, const DevScene& sc, const FrameParams& f, const PathView& base, int* qb,
                         int max_depth, cudaStream_t st, Primary primary, Infer infer, Mark mark,
                         const BatchJob* jobs = nullptr, int njobs = 0, int slots = 0) {
    for (int depth = 0; depth < w.depths; ++depth) {
        int* cnt = base.counters + kCountersPerDepth * depth;
        int* cnt_next = base.counters + kCountersPerDepth * (depth + 1);
        PathView pv = base;
        // queue ping-pong: depth d reads q[d & 1] and writes q[(d + 1) & 1]
        int* qin = (depth & 1) ? base.q1 : base.q0;
        int* qout = (depth & 1) ? base.q0 : base.q1;
        pv.q0 = qin;
        const int stop = depth == 0 ? -1 : w.stop;
        const bool traced = jobs || sc.num_bvh_tris > 0;
        if (depth == 0)
            mark(K_TRACE0, depth, 1, [&] { primary(pv, cnt); });
        else
            mark(K_TRACE, depth, 1 + traced, [&] {
                if (traced) w.ks.trace<<<w.g_trace, 128, 0, st>>>(sc, pv, cnt, stop);
                const auto post = jobs ? k_trace_post<true> : k_trace_post<false>;
                post<<<w.g_post, kPostThreads, 0, st>>>(sc, pv, cnt, stop, traced, f.records, w.bins);
            });
        infer(depth, pv, cnt, qin);
        mark(K_BIN, depth, 1, [&] { k_bin_scatter<<<w.g_bin, kBinThreads, 0, st>>>(pv, cnt, depth == 0, stop, qin, qb); });
        mark(K_SHADE, depth, 1, [&] {
            w.ks.shade<<<w.g_shade, kShadeThreads, 0, st>>>(sc, f, pv, cnt, cnt_next, stop, qb, qout);
        });
        const bool any_bvh = jobs || sc.num_bvh_tris > 0 || sc.num_bnd_tris > 0;
        mark(K_SHADOW, depth, 1 + any_bvh, [&] {
            const auto pre = jobs ? k_shadow_pre<true> : k_shadow_pre<false>;
            pre<<<w.g_post, kPostThreads, 0, st>>>(sc, pv, cnt, f.records);
            if (any_bvh)
                w.ks.shadow<<<w.g_shadow, 128, 0, st>>>(sc, pv, cnt, f.records);
        });
    }
    if (max_depth < 1 || (w.depths == max_depth && w.stop < 0)) return;
    enqueue_paths(w, sc, f, base, st, mark, jobs, njobs, slots);
}

// Adds up the segments and shadow rays of a wave whose first eight counters
// of each depth 0 .. depths are in `c` and whose k_paths totals are `pc`.
static void wave_totals(const WavePlan& w, const int* c, const PathsCount& pc, double& seg, double& shadows) {
    for (int d = 0; d < w.depths; ++d) {
        if (d > 0 && c[8 * d] <= w.stop) break;
        seg += c[8 * d];
        shadows += c[8 * d + 1];
    }
    seg += (double)pc.segments;
    shadows += (double)pc.shadows;
}

// Default paths per wave: large waves keep every depth's launches full and
// amortise each persistent kernel's tail (measured on the 1M-triangle
// frame, samples/s: 4 Mi paths 287 M, 16 Mi 390 M, 64 Mi 429 M, the whole
// 133 M-path frame 435 M; with the current kernels 64 Mi 608 M against 622 M
// for the whole frame), so up to 256 Mi paths (47 GB of path state), bounded
// to a fifth of the free device memory (about 174 bytes per path).
long long Engine::default_wave_paths(bool records) const {
    constexpr long long kMaxWave = 1LL << 28;
    // path state 64, hit 32, shadow record 48, radiance 16, three int queues
    // 12 and the shading bin 2 = 174 B (+ 32 B of records)
    const long long per_path = 174 + (records ? 32 : 0);
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) return 1LL << 22;
    long long fit = (long long)(free_b / 5) / per_path;
    return std::max(1LL << 20, std::min(kMaxWave, fit));
}

int Engine::render(const LucidRenderParams& p, float* out_host, LucidSampleRecord* recs, float* out_device) {
    GpuLock gl(*this);
    if (diag_enabled_) {
        if (recs) return fail(LUCID_ERR_INVALID, "per-sample records are not produced while diagnostics are enabled");
        return render_diag_impl(p, out_host, out_device);
    }
    const long long paths = (long long)std::max(0, p.tile_w) * std::max(0, p.tile_h) * std::max(0, p.samples);
    if (combine_ && out_host && !recs && !out_device && !(guide_ && guide_->on) && scene_loaded_ && camera_set_ &&
        paths > 0 && paths <= kCombinePaths && p.full_w > 0 && p.full_h > 0 && p.max_depth >= 1 &&
        p.max_depth <= kMaxDepth)
        return render_combined(p, out_host);
    return render_impl(p, out_host, recs, out_device, nullptr, false);
}

// ---------------------------------------------------------------- combining concurrent small renders
// Concurrent sessions (the add-on's viewport, material previews and F12
// renders each own a Renderer) meet on one device.  Small render calls
// (at most kCombinePaths paths, image to host memory, no records,
// diagnostics or guiding) pass through a process-wide combiner per device:
// a call that finds no other small call running renders on its own
// context exactly as without the combiner; calls that arrive while one
// runs wait, and the first of them to find the device free renders every
// waiting call with the same integrator and depth as one batch
// (render_batch on the combiner's own engine), each call's image bit for
// bit its own render.  Large calls never wait here: they overlap on their
// own streams as before.
namespace {
const char* const kAlgoNames[5] = {"simple", "nee", "mis", "volume_simple", "volume_mis"};
struct CombineReq {
    Engine* e;
    Engine::BatchItem item;
    int algo;
    int rc = LUCID_OK;
    bool done = false;
    std::string err;
    LucidRenderStats stats{};
};
struct Combiner {
    std::mutex mu;
    std::condition_variable cv;
    bool busy = false;
    std::vector<CombineReq*> pending;
    std::unique_ptr<Engine> runner;   // renders the batches (its own stream and path pool)
    long long batches = 0, calls = 0;
};
// One per device for the life of the process (never destroyed, so no CUDA
// call runs from a static destructor at exit).
Combiner& combiner_for(int device) {
    static std::mutex mu;
    static std::map<int, Combiner*>* all = new std::map<int, Combiner*>();
    std::lock_guard<std::mutex> lk(mu);
    Combiner*& c = (*all)[device];
    if (!c) c = new Combiner();
    return *c;
}
}  // namespace

int Engine::render_combined(const LucidRenderParams& p, float* out_host) {
    reset_cancel();
    Combiner& C = combiner_for(device_);
    CombineReq r;
    r.e = this;
    r.item.scene = ds_.get();
    std::memcpy(r.item.camera, cam_raw_, sizeof(cam_raw_));
    r.item.p = p;
    r.item.p.flags = 0;
    r.item.out_host = out_host;
    r.algo = algo_;
    std::shared_ptr<DeviceScene> keep = ds_;   // this call's scene version, whoever renders it
    std::unique_lock<std::mutex> lk(C.mu);
    C.pending.push_back(&r);
    while (!r.done) {
        if (C.busy) {
            C.cv.wait(lk);
            continue;
        }
        // lead: every waiting call with this call's integrator and depth
        C.busy = true;
        std::vector<CombineReq*> group;
        for (auto it = C.pending.begin(); it != C.pending.end();) {
            CombineReq* q = *it;
            if (q->algo == r.algo && q->item.p.max_depth == r.item.p.max_depth && group.size() < 256) {
                group.push_back(q);
                it = C.pending.erase(it);
            } else {
                ++it;
            }
        }
        lk.unlock();
        if (group.size() == 1) {
            // alone: this context's own render, as without the combiner
            r.rc = render_impl(p, out_host, nullptr, nullptr, nullptr, false);
            if (r.rc != LUCID_OK) r.err = err_;
            r.stats = stats_;
        } else {
            int rc = LUCID_OK;
            if (!C.runner) C.runner.reset(new Engine(device_));
            std::vector<BatchItem> items;
            items.reserve(group.size());
            for (CombineReq* q : group) items.push_back(q->item);
            rc = C.runner->render_batch(items.data(), (int)items.size(), kAlgoNames[r.algo], kCombinePaths * 8);
            LucidRenderStats bst{};
            C.runner->stats(&bst);
            for (CombineReq* q : group) {
                q->rc = rc;
                if (rc != LUCID_OK) q->err = C.runner->last_error();
                q->stats = bst;
                q->stats.paths = (double)q->item.p.tile_w * q->item.p.tile_h * q->item.p.samples;
            }
        }
        lk.lock();
        for (CombineReq* q : group) q->done = true;
        if (group.size() > 1) {
            ++C.batches;
            C.calls += (long long)group.size();
        }
        C.busy = false;
        C.cv.notify_all();
    }
    lk.unlock();
    stats_ = r.stats;
    if (r.rc == LUCID_OK && is_cancelled()) return fail(LUCID_ERR_CANCELLED, "render cancelled");
    if (r.rc != LUCID_OK) return fail(r.rc, r.err);
    return LUCID_OK;
}

void Engine::combine_stats(int device, long long* batches, long long* calls) {
    Combiner& C = combiner_for(device);
    std::lock_guard<std::mutex> lk(C.mu);
    if (batches) *batches = C.batches;
    if (calls) *calls = C.calls;
}

int Engine::render_f64(const LucidRenderParams& p, double* out_host) {
    GpuLock gl(*this);
    if (diag_enabled_) return fail(LUCID_ERR_INVALID, "FP64 references are not rendered while diagnostics are enabled");
    return render_impl(p, nullptr, nullptr, nullptr, nullptr, false, out_host);
}

// ---------------------------------------------------------------- path diagnostics (host)
constexpr long long kDiagWavePaths = 1LL << 20;   // paths per diagnostic wave

// render_tile with diagnostics enabled (pybind_renderer.hpp:205-316): a
// fresh DiagnosticFilm per call.  The tile is processed in bands of whole
// 8-row micro-tile rows, so replaying each band's records (sorted into the
// reference's loop order) band after band gives the order of the whole tile.
int Engine::render_diag_impl(const LucidRenderParams& p, float* out_host, float* out_device) {
    reset_cancel();
    if (p.tile_w <= 0 || p.tile_h <= 0 || p.full_w <= 0 || p.full_h <= 0)
        return fail(LUCID_ERR_INVALID, "tile and image sizes must be positive");
    const size_t np = (size_t)p.tile_w * p.tile_h;
    if (out_host) std::fill(out_host, out_host + np * 4, 0.0f);
    if (!scene_loaded_ || !camera_set_) return fail(LUCID_ERR_NO_SCENE, "scene or camera not set");
    CK(cudaSetDevice(device_));
    if (p.samples <= 0) return fail(LUCID_ERR_INVALID, "samples must be >= 1");
    if (p.max_depth > kMaxDepth) return fail(LUCID_ERR_INVALID, "max_depth too large");
    if (np > (size_t)0x7fffffff / 2) return fail(LUCID_ERR_INVALID, "tile too large");
    diag_film_.init(p.tile_w, p.tile_h, diag_cfg_.subsample_factor);
    diag_film_.set_limits(diag_cfg_.max_groups_per_pixel, diag_cfg_.max_outliers_per_pixel);
    cudaStream_t st = S(stream_);
    const long long wave = wave_cap_ > 0 ? std::min(wave_cap_, kDiagWavePaths) : kDiagWavePaths;
    const long long row_paths = (long long)p.tile_w * p.samples;
    int band_rows = 8 * (int)std::max<long long>(1, wave / (8 * row_paths));
    band_rows = std::min(band_rows, (p.tile_h + 7) / 8 * 8);
    const long long band_np = (long long)band_rows * p.tile_w;
    const int spw = (int)std::max<long long>(1, std::min<long long>(p.samples, wave / band_np));
    int rc = ensure_pool((long long)spw * band_np, false);
    if (rc != LUCID_OK) return rc;
    PathPool& P = *pool_;
    if (P.film_n < np) {
        CK(P.film.alloc(np));
        CK(P.out.alloc(np));
        P.film_n = np;
    }
    if (!diag_dev_) diag_dev_ = new DiagDevice();
    DiagDevice& D = *diag_dev_;
    const long long want = diag_cfg_.record_capacity > 0 ? diag_cfg_.record_capacity : (1LL << 20);
    if ((long long)D.index.n < want) CK(D.index.alloc((size_t)want));
    if ((long long)D.units.n < 8 * want) CK(D.units.alloc((size_t)(8 * want)));   // a few bounces per record
    if (!D.count.p) CK(D.count.alloc(2));
    CK(cudaMemsetAsync(P.film.p, 0, np * sizeof(float4), st));
    CK(cudaMemsetAsync(P.errors.p, 0, kErrorInts * sizeof(int), st));

    FrameParams f{};
    for (int k = 0; k < 3; ++k) { f.pos[k] = cam_.pos[k]; f.fwd[k] = cam_.forward[k]; f.right[k] = cam_.right[k]; f.up[k] = cam_.up[k]; }
    f.aspect = (float)p.full_w / (float)p.full_h;
    f.scale = std::tan(cam_.fov * 0.5f);
    f.tile_x = p.tile_x; f.tile_w = p.tile_w; f.full_w = p.full_w; f.full_h = p.full_h;
    f.samples = p.samples; f.sample_offset = p.sample_offset; f.max_depth = p.max_depth; f.algo = algo_;
    f.records = 0;

    stats_ = LucidRenderStats{};
    struct Events {   // destroyed on every return
        cudaEvent_t e[6] = {};
        Events() { for (cudaEvent_t& x : e) cudaEventCreate(&x); }
        ~Events() { for (cudaEvent_t x : e) if (x) cudaEventDestroy(x); }
    } events;
    const cudaEvent_t t0 = events.e[0], t1 = events.e[1], ka = events.e[2], kb = events.e[3], ca = events.e[4],
                      cb = events.e[5];
    cudaEventRecord(t0, st);
    int status = LUCID_OK;
    int waves = 0;
    double kernel_ms = 0.0, copy_ms = 0.0, replay_ms = 0.0, records_total = 0.0, record_bytes = 0.0;
    size_t band_n = 0, band_units = 0;
    // the host replays band k (in band order) while the device renders band
    // k + 1 into the other pinned buffer; the film is touched by the replay
    // alone.  A pending replay is waited for before the next starts, and on
    // every return (the future's destructor).
    int hb = 0;
    std::future<double> replay;
    for (int y0 = 0; y0 < p.tile_h && status == LUCID_OK; y0 += band_rows) {
        const int bh = std::min(band_rows, p.tile_h - y0);
        f.tile_y = p.tile_y + y0;
        f.tile_h = bh;
        f.npix = bh * p.tile_w;
        band_n = 0;
        band_units = 0;
        for (int s0 = 0; s0 < p.samples; s0 += spw) {
            if (is_cancelled()) { status = LUCID_ERR_CANCELLED; break; }
            const int this_spw = std::min(spw, p.samples - s0);
            f.s0 = s0;
            f.n_wave = this_spw * f.npix;
            unsigned long long produced[2] = {0, 0};
            for (;;) {
                CK(cudaMemsetAsync(D.count.p, 0, 2 * sizeof(unsigned long long), st));
                cudaEventRecord(ka, st);
                k_raygen<<<(f.n_wave + 255) / 256, 256, 0, st>>>(f, P.view);
                DiagOut o{D.units.p, D.index.p, D.count.p, (long long)D.index.n, (long long)D.units.n,
                          (uint32_t)band_units};
                k_diag_paths<<<(f.n_wave + 127) / 128, 128, 0, st>>>(ds_->view, f, P.view, o, y0 * p.tile_w);
                cudaEventRecord(kb, st);
                CK(cudaGetLastError());
                CK(cudaMemcpyAsync(produced, D.count.p, sizeof(produced), cudaMemcpyDeviceToHost, st));
                CK(cudaStreamSynchronize(st));
                float kms = 0.0f;
                cudaEventElapsedTime(&kms, ka, kb);
                kernel_ms += kms;
                if (band_units + produced[1] >= (1ULL << 32))
                    return fail(LUCID_ERR_OVERFLOW, "path diagnostics: a band's records exceed 64 GB");
                if (produced[0] <= (unsigned long long)D.index.n && produced[1] <= (unsigned long long)D.units.n) break;
                // the wave is deterministic: grow the buffers and run it again
                if (produced[0] > (unsigned long long)D.index.n) CK(D.index.alloc((size_t)(produced[0] + produced[0] / 4)));
                if (produced[1] > (unsigned long long)D.units.n) CK(D.units.alloc((size_t)(produced[1] + produced[1] / 4)));
            }
            k_film<<<(f.npix + 255) / 256, 256, 0, st>>>(f.npix, this_spw, P.rad.p, P.film.p + (size_t)y0 * p.tile_w);
            CK(D.reserve_host(hb, band_n + (size_t)produced[0], band_n, band_units + (size_t)produced[1], band_units));
            cudaEventRecord(ca, st);
            if (produced[0]) {
                CK(cudaMemcpyAsync(D.host_index[hb] + band_n, D.index.p, (size_t)produced[0] * sizeof(uint32_t),
                                   cudaMemcpyDeviceToHost, st));
                CK(cudaMemcpyAsync(D.host_units[hb] + band_units * kDiagUnitBytes, D.units.p,
                                   (size_t)produced[1] * kDiagUnitBytes, cudaMemcpyDeviceToHost, st));
            }
            band_n += (size_t)produced[0];
            band_units += (size_t)produced[1];
            record_bytes += (double)produced[0] * sizeof(uint32_t) + (double)produced[1] * kDiagUnitBytes;
            cudaEventRecord(cb, st);
            CK(cudaStreamSynchronize(st));
            float cms = 0.0f;
            cudaEventElapsedTime(&cms, ca, cb);
            copy_ms += cms;
            records_total += (double)produced[0];
            ++waves;
        }
        if (status == LUCID_OK) {
            if (replay.valid()) replay_ms += replay.get();
            const uint8_t* units = D.host_units[hb];
            const uint32_t* index = D.host_index[hb];
            const size_t n_rec = band_n;
            const int tw = p.tile_w;
            const bool last = y0 + band_rows >= p.tile_h;
            // while the device renders the next band, this thread waits on it:
            // the replay leaves it a core
            const unsigned hw = std::max(1u, std::thread::hardware_concurrency());
            const unsigned nt = last ? hw : std::max(1u, hw - 1);
            auto run = [this, units, index, n_rec, tw, nt]() {
                const auto h0 = std::chrono::steady_clock::now();
                diag_film_.replay(units, index, n_rec, tw, nt);
                return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - h0).count();
            };
            if (last) replay_ms += run();   // the last band: nothing left to overlap
            else replay = std::async(std::launch::async, run);
            hb ^= 1;
        }
    }
    if (replay.valid()) replay_ms += replay.get();
    // where a diagnostic render's time goes: the path kernel (raygen
    // included), the record copies to the host, and the host replay
    const char* names[3] = {"k_diag_paths", "diag_record_copy", "diag_replay_host"};
    const double ms3[3] = {kernel_ms, copy_ms, replay_ms};
    stats_.num_kinds = 3;
    for (int k = 0; k < 3; ++k) {
        std::snprintf(stats_.kinds[k].name, sizeof(stats_.kinds[k].name), "%s", names[k]);
        stats_.kinds[k].launches = waves;
        stats_.kinds[k].total_ms = ms3[k];
        stats_.kinds[k].units = k == 0 ? (double)np * p.samples : records_total;
        stats_.kinds[k].algo_bytes = k == 1 ? record_bytes : 0.0;
    }
    const int np_i = (int)np;
    k_output<<<(np_i + 255) / 256, 256, 0, st>>>(p.tile_w, p.tile_h, P.film.p, out_device ? (float4*)out_device : P.out.p);
    CK(cudaGetLastError());
    cudaEventRecord(t1, st);
    int herr[4] = {0, 0, 0, 0};
    CK(cudaMemcpyAsync(herr, P.errors.p, sizeof(herr), cudaMemcpyDeviceToHost, st));
    if (out_host && !out_device)
        CK(cudaMemcpyAsync(out_host, P.out.p, np * sizeof(float4), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    float tot = 0.0f;
    cudaEventElapsedTime(&tot, t0, t1);
    stats_.total_ms = tot;
    stats_.paths = (double)np * p.samples;
    stats_.waves = waves;
    if (herr[0] != 0) return fail(LUCID_ERR_OVERFLOW, "BVH traversal stack overflow");
    if (status == LUCID_ERR_CANCELLED) return fail(LUCID_ERR_CANCELLED, "render cancelled");
    return LUCID_OK;
}

// PathRecordingConfig::standard() (diagnostics/path_stats_config.hpp).
int Engine::diag_enable(const LucidDiagConfig* cfg) {
    GpuLock gl(*this);
    LucidDiagConfig c{2, 16, 4, 16, 0.001f, 3.0f, 0};
    if (cfg) c = *cfg;
    if (c.subsample_factor < 1) return fail(LUCID_ERR_INVALID, "subsample_factor must be >= 1");
    diag_cfg_ = c;
    diag_enabled_ = true;
    diag_film_.reset();
    return LUCID_OK;
}
int Engine::diag_disable() {
    GpuLock gl(*this);
    diag_enabled_ = false;
    diag_film_.reset();
    if (diag_dev_) { delete diag_dev_; diag_dev_ = nullptr; }
    return LUCID_OK;
}
int Engine::diag_clear() {
    GpuLock gl(*this);
    if (diag_film_.valid()) diag_film_.clear();
    return LUCID_OK;
}
int Engine::diag_stats(LucidDiagStats* out) {
    GpuLock gl(*this);
    std::memset(out, 0, sizeof(*out));
    if (diag_film_.valid()) diag_film_.stats(out);
    return LUCID_OK;
}
int Engine::diag_pixel(int x, int y, bool by_mean, LucidDiagPixel* info, LucidDiagGroup* groups, int cap) {
    GpuLock gl(*this);
    std::memset(info, 0, sizeof(*info));
    if (!diag_film_.valid()) return 0;
    return diag_film_.export_pixel(x, y, by_mean, info, groups, groups ? cap : 0);
}
int Engine::diag_variance_map(float* out, size_t cap) {
    GpuLock gl(*this);
    if (!diag_film_.valid()) return 0;
    size_t n = (size_t)diag_film_.width() * diag_film_.height();
    if (cap < n) return fail(LUCID_ERR_INVALID, "variance map buffer too small");
    diag_film_.variance_map(out);
    return (int)n;
}
int Engine::diag_top(int n, bool by_mean, LucidDiagGroup* groups, int32_t* xy, int cap) {
    GpuLock gl(*this);
    if (!diag_film_.valid()) return 0;
    return diag_film_.export_top(n, by_mean, groups, xy, groups ? cap : 0);
}

int Engine::diag_coarse(LucidDiagCoarse* out) {
    GpuLock gl(*this);
    if (!diag_film_.valid()) {
        DiagFilm empty;
        empty.coarse_export(out);
        return 8;
    }
    diag_film_.coarse_export(out);
    return 8;
}
int Engine::diag_suggestions(LucidDiagSuggestion* out, int cap) {
    GpuLock gl(*this);
    if (!diag_film_.valid()) return 0;
    return diag_film_.suggestions(out, out ? cap : 0);
}
long long Engine::diag_export_binary(uint8_t* out, size_t cap) {
    GpuLock gl(*this);
    const std::vector<uint8_t> b = diag_film_.export_binary();
    if (out) std::memcpy(out, b.data(), std::min(cap, b.size()));
    return (long long)b.size();
}
long long Engine::diag_metadata_json(char* out, size_t cap) {
    GpuLock gl(*this);
    const std::string m = diag_film_.metadata_json();
    if (out && cap > 0) {
        const size_t n = std::min(cap - 1, m.size());
        std::memcpy(out, m.data(), n);
        out[n] = 0;
    }
    return (long long)m.size();
}

// Adds one render's film into the async accumulator (float4 sum per pixel).
__global__ void k_accumulate(int npix, const float4* film, float4* acc) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= npix) return;
    float4 a = acc[p], f = film[p];
    acc[p] = make_float4(a.x + f.x, a.y + f.y, a.z + f.z, 0.0f);
}

int Engine::render_impl(const LucidRenderParams& p, float* out_host, LucidSampleRecord* recs, float* out_device,
                        void* accumulate, bool from_async, double* out_f64) {
    if (!from_async) reset_cancel();
    if (p.tile_w <= 0 || p.tile_h <= 0 || p.full_w <= 0 || p.full_h <= 0)
        return fail(LUCID_ERR_INVALID, "tile and image sizes must be positive");
    size_t np = (size_t)p.tile_w * p.tile_h;
    // A call that returns before its image is copied out leaves a zero image
    // (the reference's empty result); a finished copy is not written twice,
    // which at 1920x1080 saves a 33 MB host fill per call.
    struct ZeroUnlessCopied {
        float* f;
        double* d;
        size_t n;
        bool copied = false;
        ~ZeroUnlessCopied() {
            if (copied) return;
            if (f) std::fill(f, f + n * 4, 0.0f);
            if (d) std::fill(d, d + n * 4, 0.0);
        }
    } host_image{out_host, out_f64, np};
    if (!scene_loaded_ || !camera_set_) return fail(LUCID_ERR_NO_SCENE, "scene or camera not set");
    CK(cudaSetDevice(device_));
    if (p.samples <= 0) return fail(LUCID_ERR_INVALID, "samples must be >= 1");
    if (p.max_depth > kMaxDepth) return fail(LUCID_ERR_INVALID, "max_depth too large");
    if (np > (size_t)0x7fffffff / 2) return fail(LUCID_ERR_INVALID, "tile too large");
    cudaStream_t st = S(stream_);
    const bool profile = (p.flags & LUCID_RENDER_PROFILE) != 0;
    const bool records = recs != nullptr;
    const bool guide = guide_ && guide_->on && algo_ == ALGO_MIS && !from_async;
    // The wave cap needs a device memory query (a driver call that other
    // processes' driver traffic can hold up for tens of milliseconds); a
    // call that fits the path pool it already has skips it.
    const PathPool& P0 = *pool_;
    long long cap;
    if (wave_cap_ > 0)
        cap = wave_cap_;
    else if (P0.cap >= (long long)p.samples * (long long)np && (!records || P0.records))
        cap = P0.cap;
    else
        cap = default_wave_paths(records);
    if (guide) cap = std::min(cap, kGuideWave);
    int spw = (int)std::max<long long>(1, std::min<long long>(p.samples, cap / (long long)np));
    long long wave_paths = (long long)spw * (long long)np;
    // A progressive caller (the add-on's F12 loop: 4, 8, 16, 32, then 64
    // samples per call) grows the wave call by call; reserving 64 samples
    // per pixel of the tile (within the cap) at the first multi-sample call
    // keeps the later calls from reallocating the pool (50-60 ms each at
    // 1920x1080).  Async dispatches (1 sample each) keep their small pool.
    long long reserve = wave_paths;
    if (!from_async && !records && p.samples > 1)
        reserve = std::max(wave_paths, std::min(cap, 64LL * (long long)np));
    int rc = ensure_pool(reserve, records);
    if (rc != LUCID_OK) return rc;
    PathPool& P = *pool_;
    if (P.film_n < np) {
        CK(P.film.alloc(np));
        CK(P.out.alloc(np));
        P.film_n = np;
    }
    if (spw < p.samples || accumulate || guide) CK(cudaMemsetAsync(P.film.p, 0, np * sizeof(float4), st));
    CK(cudaMemsetAsync(P.errors.p, 0, kErrorInts * sizeof(int), st));
    if (out_f64) {
        if (P.film64_n < np) {
            CK(P.film64.alloc(np * 3));
            CK(P.out64.alloc(np * 4));
            P.film64_n = np;
        }
        CK(cudaMemsetAsync(P.film64.p, 0, np * 3 * sizeof(double), st));
    }
    DBuf<LucidSampleRecord> d_recs;
    if (records) CK(d_recs.alloc(np * (size_t)p.samples));

    FrameParams f{};
    for (int k = 0; k < 3; ++k) { f.pos[k] = cam_.pos[k]; f.fwd[k] = cam_.forward[k]; f.right[k] = cam_.right[k]; f.up[k] = cam_.up[k]; }
    f.aspect = (float)p.full_w / (float)p.full_h;
    f.scale = std::tan(cam_.fov * 0.5f);
    f.tile_x = p.tile_x; f.tile_y = p.tile_y; f.tile_w = p.tile_w; f.tile_h = p.tile_h;
    f.full_w = p.full_w; f.full_h = p.full_h;
    f.samples = p.samples; f.sample_offset = p.sample_offset; f.max_depth = p.max_depth; f.algo = algo_;
    f.npix = (int)np;
    f.records = records ? 1 : 0;

    const WavePlan w = wave_plan(device_, num_sms_, algo_, guide, launch_profile_, false, wave_paths, p.max_depth);
    PathView gv = P.view;   // the path view with the guide's buffers when guiding
    if (guide) {
        int rc2 = guide_buffers(wave_paths);
        if (rc2 != LUCID_OK) return rc2;
        GuideState& G = *guide_;
        gv.gmix = G.gmix.p; gv.gslot = G.gslot.p; gv.ginv = G.ginv.p; gv.grec = G.recs.p; gv.gcount = G.count.p;
        gv.gcap = G.steps * kGuideBatch;
        gv.gdepth = G.max_depth;
        for (int k = 0; k < 3; ++k) {
            gv.glo[k] = scene_lo_[k];
            float ext = scene_hi_[k] - scene_lo_[k];
            gv.gscale[k] = ext > 0.0f ? 1.0f / ext : 0.0f;
        }
        static bool attr = false;
        if (!attr) {
            CK(cudaFuncSetAttribute(k_guide_infer, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kInferSmem));
            attr = true;
        }
    }
    struct Launch { int kind; cudaEvent_t a, b; int depth; int kernels = 1; };
    std::vector<Launch> launches;
    auto ev_begin = [&](int kind, int depth) -> int {
        if (!profile) return -1;
        Launch l{kind, nullptr, nullptr, depth};
        cudaEventCreate(&l.a);
        cudaEventCreate(&l.b);
        cudaEventRecord(l.a, st);
        launches.push_back(l);
        return (int)launches.size() - 1;
    };
    auto ev_end = [&](int idx) { if (idx >= 0) cudaEventRecord(launches[idx].b, st); };

    stats_ = LucidRenderStats{};
    double seg = 0, shadows = 0;
    // pinned: the first eight counters of each depth, then the error words
    static_assert(sizeof(int) * (8 * (kMaxDepth + 1) + kErrorInts) <= kPinnedBytes, "a call's counters");
    if (!host_block_) CK(pinned_take(&host_block_));
    int* const hcnt = static_cast<int*>(host_block_);
    int* const herr = hcnt + 8 * (kMaxDepth + 1);
    const bool one_wave = spw >= p.samples;
    std::vector<double> kind_units(K_NUM, 0.0);
    if (!render_ev_[0]) { CK(cudaEventCreate((cudaEvent_t*)&render_ev_[0])); CK(cudaEventCreate((cudaEvent_t*)&render_ev_[1])); }
    const cudaEvent_t t0 = (cudaEvent_t)render_ev_[0], t1 = (cudaEvent_t)render_ev_[1];
    cudaEventRecord(t0, st);
    int status = LUCID_OK;
    int waves = 0;
    // a wave's counts, once its copies have arrived
    auto add_totals = [&]() {
        PathsCount pc;
        std::memcpy(&pc, herr + 4, sizeof(pc));
        if (w.depths >= p.max_depth && w.stop < 0) pc.segments = pc.shadows = 0;   // k_paths did not run
        wave_totals(w, hcnt, pc, seg, shadows);
        if (!profile) return;
        kind_units[K_FILM] += f.n_wave;
        for (int d = 0; d < w.depths; ++d) {
            if (d > 0 && hcnt[8 * d] <= w.stop) break;
            const double n = hcnt[8 * d];
            kind_units[d == 0 ? K_TRACE0 : K_TRACE] += n;
            kind_units[K_SHADE] += n;
            kind_units[K_BIN] += n;
            if (guide) kind_units[K_GUIDE] += n;
            kind_units[K_SHADOW] += hcnt[8 * d + 1];
        }
        kind_units[K_PATHS] += (double)pc.segments;
    };
    auto fetch_counts = [&]() -> cudaError_t {
        cudaError_t e = cudaSuccess;
        if (w.depths > 0)
            e = cudaMemcpy2DAsync(hcnt, 32, P.counters.p, sizeof(int) * kCountersPerDepth, 32, (size_t)w.depths,
                                  cudaMemcpyDeviceToHost, st);
        if (e != cudaSuccess) return e;
        return cudaMemcpyAsync(herr, P.errors.p, kErrorInts * sizeof(int), cudaMemcpyDeviceToHost, st);
    };
    for (int s0 = 0; s0 < p.samples; s0 += spw) {
        if (!from_async && is_cancelled()) { status = LUCID_ERR_CANCELLED; break; }
        int this_spw = std::min(spw, p.samples - s0);
        f.s0 = s0;
        f.n_wave = (int)((long long)this_spw * (long long)np);
        if (p.max_depth < 1) CK(cudaMemsetAsync(P.rad.p, 0, (size_t)f.n_wave * sizeof(float4), st));   // no segment at all
        if (w.depths > 0) CK(cudaMemsetAsync(P.counters.p, 0, sizeof(int) * kCountersPerDepth * (w.depths + 1), st));
        if (guide) {
            GuideState& G = *guide_;
            gv.gkeep = (unsigned)std::min(4294967295.0, (double)G.keep * 4294967296.0);
            CK(cudaMemsetAsync(G.gslot.p, 0xff, (size_t)f.n_wave * sizeof(int4), st));
            CK(cudaMemsetAsync(G.count.p, 0, 2 * sizeof(int), st));
        }
        int e = 0;
        enqueue_wave(w, ds_->view, f, gv, P.qb.p, p.max_depth, st, [&](const PathView& pv, int* cnt) {
            k_trace_primary_for(ds_->view, f.pos)<<<w.g_trace0, 128, 0, st>>>(ds_->view, f, pv, cnt, f.records, w.bins);
        }, [&](int depth, const PathView& pv, int* cnt, const int* qin) {
            if (!guide || depth >= guide_->max_depth) return;
            const int k = ev_begin(K_GUIDE, depth);
            k_guide_infer<<<num_sms_, 32 * kInferWarps, kInferSmem, st>>>(
                ds_->view, pv, cnt, depth == 0, qin, static_cast<const __nv_bfloat16*>(guide_->net.weights_bf16()),
                guide_->net.master());
            ev_end(k);
        }, [&](int kind, int depth, int kernels, auto&& launch) {
            const int k = ev_begin(kind, depth);
            if (k >= 0) launches[(size_t)k].kernels = kernels;
            launch();
            ev_end(k);
        });
        if (records) k_records<<<(f.n_wave + 255) / 256, 256, 0, st>>>(f, P.view, d_recs.p);
        ++waves;
        if (one_wave && !out_f64 && !accumulate && !guide) break;   // summed straight into the output image below
        e = ev_begin(K_FILM, 0);
        if (out_f64)
            k_film_f64<<<(f.npix + 255) / 256, 256, 0, st>>>(f.npix, this_spw, P.rad.p, P.film64.p);
        else
            k_film<<<(f.npix + 255) / 256, 256, 0, st>>>(f.npix, this_spw, P.rad.p, P.film.p);
        ev_end(e);
        CK(cudaGetLastError());
        if (one_wave && !guide) break;   // the counts come with the image
        CK(fetch_counts());
        int gcnt[2] = {0, 0};
        if (guide) CK(cudaMemcpyAsync(gcnt, guide_->count.p, sizeof(gcnt), cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        if (guide) {
            // Adam steps on this wave's records, one batch each; the next
            // wave's sampling rate aims at 90 % of the batches
            GuideState& G = *guide_;
            int nrec = std::min(gcnt[0], G.steps * kGuideBatch);
            e = ev_begin(K_TRAIN, 0);
            for (int b = 0; b * kGuideBatch < nrec; ++b)
                if (G.net.train_step(G.recs.p + (size_t)b * kGuideBatch, std::min(kGuideBatch, nrec - b * kGuideBatch),
                                     st, G.lr) != 0)
                    return fail(LUCID_ERR_CUDA, "guide training: " + G.net.error());
            ev_end(e);
            if (profile) kind_units[K_TRAIN] += nrec;
            G.keep = (float)std::min(1.0, 0.9 * G.steps * kGuideBatch / std::max(1.0, (double)gcnt[1]));
        }
        add_totals();
    }
    const int np_i = (int)np;
    if (one_wave && waves == 0) CK(cudaMemsetAsync(P.film.p, 0, np * sizeof(float4), st));   // cancelled at once
    if (accumulate) {
        k_accumulate<<<(np_i + 255) / 256, 256, 0, st>>>(np_i, P.film.p, (float4*)accumulate);
    } else if (out_f64) {
        k_output_f64<<<(np_i + 255) / 256, 256, 0, st>>>(p.tile_w, p.tile_h, P.film64.p, P.out64.p);
    } else {
        float4* const out = out_device ? (float4*)out_device : P.out.p;
        if (one_wave && !guide && waves == 1) {
            const int e = ev_begin(K_FILM, 0);
            k_film_output<<<(np_i + 127) / 128, 128, 0, st>>>(p.tile_w, p.tile_h, p.samples, P.rad.p, out);
            ev_end(e);
        } else {
            k_output<<<(np_i + 255) / 256, 256, 0, st>>>(p.tile_w, p.tile_h, P.film.p, out);
        }
    }
    cudaEventRecord(t1, st);
    CK(cudaGetLastError());
    CK(fetch_counts());
    if (out_host && !out_device)
        CK(cudaMemcpyAsync(out_host, P.out.p, np * sizeof(float4), cudaMemcpyDeviceToHost, st));
    if (out_f64)
        CK(cudaMemcpyAsync(out_f64, P.out64.p, np * 4 * sizeof(double), cudaMemcpyDeviceToHost, st));
    if (records)
        CK(cudaMemcpyAsync(recs, d_recs.p, np * (size_t)p.samples * sizeof(LucidSampleRecord), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    host_image.copied = true;
    if (one_wave && !guide && waves == 1) add_totals();
    if (guide && guide_->net.failed(st) != 0) return fail(LUCID_ERR_TIMEOUT, guide_->net.error());
    float tot = 0.0f;
    cudaEventElapsedTime(&tot, t0, t1);
    stats_.total_ms = tot;
    stats_.paths = (double)np * p.samples;
    stats_.segments = seg;
    stats_.shadow_rays = shadows;
    stats_.waves = waves;
    if (profile) {
        stats_.num_kinds = K_NUM;
        for (int k = 0; k < K_NUM; ++k) {
            std::snprintf(stats_.kinds[k].name, sizeof(stats_.kinds[k].name), "%s", kKindNames[k]);
            stats_.kinds[k].units = kind_units[k];
            stats_.kinds[k].algo_bytes = kind_units[k] * kKindBytes[k];
        }
        for (auto& l : launches) {
            float ms = 0.0f;
            cudaEventElapsedTime(&ms, l.a, l.b);
            stats_.kinds[l.kind].launches += l.kernels;
            stats_.kinds[l.kind].total_ms += ms;
            cudaEventDestroy(l.a);
            cudaEventDestroy(l.b);
        }
        stats_.kinds[K_FILM].algo_bytes += (double)np * 32.0 * waves;
    }
    if (herr[0] != 0) return fail(LUCID_ERR_OVERFLOW, "BVH traversal stack overflow");
    if (status == LUCID_ERR_CANCELLED) return fail(LUCID_ERR_CANCELLED, "render cancelled");
    return LUCID_OK;
}

// ---------------------------------------------------------------- batched jobs (host)
static int algo_from_name(const char* name) {
    std::string a = name ? name : "";
    if (a == "simple") return ALGO_SIMPLE;
    if (a == "mis") return ALGO_MIS;
    if (a == "volume_simple") return ALGO_VOLUME_SIMPLE;
    if (a == "volume_mis") return ALGO_VOLUME_MIS;
    return ALGO_NEE;   // the reference's dispatch falls through to traceNEE
}

long long Engine::batch_bytes(long long pixels, long long wave_paths) {
    // path state (174 B) and scene index (2 B) per path with slack, film and
    // output per pixel, the job and scene tables
    return wave_paths * 178 + pixels * 32 + (2 << 20);
}

// Jobs on different scenes (and cameras, image sizes, sample counts) in one
// set of wavefront launches: the jobs' samples are cut into pieces that fill
// waves of up to `wave_paths` paths in job order (a job larger than a wave
// continues in the next one, in sample order); a wave's device job table
// gives the camera-ray kernel each piece's camera, image, sample range,
// scene and first path, and every later kernel reads a path's scene from the
// wave's scene table.  Each job's film sums its samples in sample order, so
// its image is the one lucid_cuda_render gives for the same call on its own
// scene, bit for bit.
int Engine::render_batch(const BatchItem* items, int n, const char* algorithm, long long wave_paths) {
    GpuLock gl(*this);
    reset_cancel();
    if (n <= 0 || !items) return fail(LUCID_ERR_INVALID, "batch: no jobs");
    // a call that returns before the images are copied out leaves every
    // job's image zero, as a single render call does
    struct ZeroUnlessCopied {
        const BatchItem* it;
        int n;
        bool copied = false;
        ~ZeroUnlessCopied() {
            if (copied) return;
            for (int j = 0; j < n; ++j)
                if (it[j].out_host && it[j].p.tile_w > 0 && it[j].p.tile_h > 0)
                    std::fill(it[j].out_host, it[j].out_host + (size_t)it[j].p.tile_w * it[j].p.tile_h * 4, 0.0f);
        }
    } host_images{items, n};
    const int algo = algo_from_name(algorithm);
    const int depth = items[0].p.max_depth;
    if (depth < 1 || depth > kMaxDepth) return fail(LUCID_ERR_INVALID, "batch: max_depth must be 1..1024");
    std::vector<const DeviceScene*> scenes;
    std::vector<int> job_sid((size_t)n);
    std::vector<size_t> film_off((size_t)n + 1, 0);
    long long total_paths = 0, max_np = 1;
    for (int j = 0; j < n; ++j) {
        const LucidRenderParams& p = items[j].p;
        if (!items[j].scene || !items[j].out_host) return fail(LUCID_ERR_INVALID, "batch: a job has no scene or output");
        if (p.tile_w <= 0 || p.tile_h <= 0 || p.full_w <= 0 || p.full_h <= 0)
            return fail(LUCID_ERR_INVALID, "batch: tile and image sizes must be positive");
        if (p.samples <= 0) return fail(LUCID_ERR_INVALID, "batch: samples must be >= 1");
        if (p.max_depth != depth) return fail(LUCID_ERR_INVALID, "batch: every job needs the same max_depth");
        const long long np = (long long)p.tile_w * p.tile_h;
        if (np > (1LL << 28)) return fail(LUCID_ERR_INVALID, "batch: tile too large");
        const DeviceScene* ds = static_cast<const DeviceScene*>(items[j].scene);
        int k = 0;
        while (k < (int)scenes.size() && scenes[k] != ds) ++k;
        if (k == (int)scenes.size()) {
            if (scenes.size() >= 65535) return fail(LUCID_ERR_INVALID, "batch: more than 65535 scenes");
            scenes.push_back(ds);
        }
        job_sid[j] = k;
        film_off[j + 1] = film_off[j] + (size_t)np;
        total_paths += np * p.samples;
        max_np = std::max(max_np, np);
    }
    CK(cudaSetDevice(device_));
    int rc = ensure_stream();
    if (rc != LUCID_OK) return rc;
    cudaStream_t st = S(stream_);
    long long cap = wave_paths > 0 ? wave_paths : wave_cap_;
    if (cap <= 0) cap = pool_->cap >= total_paths ? pool_->cap : default_wave_paths(false);
    cap = std::max(cap, max_np);                 // one sample of the largest tile per wave at least
    cap = std::min(cap, std::max(total_paths, max_np));
    if (cap >= (1LL << 31) - 64) return fail(LUCID_ERR_INVALID, "batch: wave too large");
    rc = ensure_pool(cap, false);
    if (rc != LUCID_OK) return rc;
    PathPool& P = *pool_;
    if (P.sid.n < (size_t)P.cap) CK(P.sid.alloc((size_t)P.cap));
    const size_t npix_all = film_off[(size_t)n];
    if (P.film_n < npix_all) {
        CK(P.film.alloc(npix_all));
        CK(P.out.alloc(npix_all));
        P.film_n = npix_all;
    }
    CK(cudaMemsetAsync(P.film.p, 0, npix_all * sizeof(float4), st));
    CK(cudaMemsetAsync(P.errors.p, 0, kErrorInts * sizeof(int), st));

    // the scene table, then room for the largest wave's job table
    std::vector<DevScene> scene_tab(scenes.size());
    for (size_t k = 0; k < scenes.size(); ++k) scene_tab[k] = scenes[k]->view;
    const size_t tab_off = (scene_tab.size() * sizeof(DevScene) + 255) & ~(size_t)255;
    const size_t tab_bytes = tab_off + (size_t)kMaxBatchPieces * sizeof(BatchJob);
    if (P.btab.n < tab_bytes) CK(P.btab.alloc(tab_bytes));
    CK(cudaMemcpyAsync(P.btab.p, scene_tab.data(), scene_tab.size() * sizeof(DevScene), cudaMemcpyHostToDevice, st));
    const DevScene* d_scenes = reinterpret_cast<const DevScene*>(P.btab.p);
    const BatchJob* d_jobs = reinterpret_cast<const BatchJob*>(P.btab.p + tab_off);

    std::vector<HostCamera> cams((size_t)n);
    for (int j = 0; j < n; ++j) {
        const float* c = items[j].camera;
        make_camera(cams[j], c[0], c[1], c[2], c[3], c[4], c[5], c[6], c[7], c[8], c[9]);
    }
    auto frame_of = [&](int j, int s0, int spw) {
        const LucidRenderParams& p = items[j].p;
        const HostCamera& cam = cams[j];
        FrameParams f{};
        for (int k = 0; k < 3; ++k) { f.pos[k] = cam.pos[k]; f.fwd[k] = cam.forward[k]; f.right[k] = cam.right[k]; f.up[k] = cam.up[k]; }
        f.aspect = (float)p.full_w / (float)p.full_h;
        f.scale = std::tan(cam.fov * 0.5f);
        f.tile_x = p.tile_x; f.tile_y = p.tile_y; f.tile_w = p.tile_w; f.tile_h = p.tile_h;
        f.full_w = p.full_w; f.full_h = p.full_h;
        f.samples = p.samples; f.sample_offset = p.sample_offset; f.max_depth = depth; f.algo = algo;
        f.npix = p.tile_w * p.tile_h;
        f.s0 = s0;
        f.n_wave = spw * f.npix;
        return f;
    };

    FrameParams fshade{};
    fshade.max_depth = depth;
    fshade.algo = algo;

    stats_ = LucidRenderStats{};
    double seg = 0, shadows = 0;
    std::vector<int> hcnt((size_t)8 * (depth + 1));
    cudaEvent_t t0, t1;
    cudaEventCreate(&t0);
    cudaEventCreate(&t1);
    cudaEventRecord(t0, st);
    int waves = 0, status = LUCID_OK;
    std::vector<BatchJob> tab;
    struct PieceFilm { int job, spw, path_base; };
    std::vector<PieceFilm> films;
    int j = 0, s = 0;   // next sample s of job j still to render
    while (j < n) {
        if (is_cancelled()) { status = LUCID_ERR_CANCELLED; break; }
        // fill one wave with pieces, in job order
        tab.clear();
        films.clear();
        long long used = 0, slots = 0;
        while (j < n && (int)tab.size() < kMaxBatchPieces) {
            const LucidRenderParams& p = items[j].p;
            const long long np = (long long)p.tile_w * p.tile_h;
            const int take = (int)std::min<long long>(p.samples - s, (cap - used) / np);
            if (take < 1) break;
            const long long per_sample = (long long)((p.tile_w + 7) / 8) * ((p.tile_h + 3) / 4) * 32;
            if (slots + per_sample * take >= (1LL << 31) - 64) break;
            BatchJob b{};
            b.f = frame_of(j, s, take);
            b.sid = job_sid[j];
            b.path_base = (int)used;
            b.slot_base = (int)slots;
            tab.push_back(b);
            films.push_back({j, take, (int)used});
            used += np * take;
            slots += per_sample * take;
            s += take;
            if (s >= p.samples) { ++j; s = 0; }
        }
        if (tab.empty()) return fail(LUCID_ERR_INVALID, "batch: a job piece does not fit a wave");
        CK(cudaMemcpyAsync(const_cast<BatchJob*>(d_jobs), tab.data(), tab.size() * sizeof(BatchJob),
                           cudaMemcpyHostToDevice, st));
        const int n_wave = (int)used;
        const WavePlan w = wave_plan(device_, num_sms_, algo, false, 0, true, n_wave, depth);
        if (w.depths > 0) CK(cudaMemsetAsync(P.counters.p, 0, sizeof(int) * kCountersPerDepth * (w.depths + 1), st));
        PathView pv = P.view;
        pv.scenes = d_scenes;
        pv.sid = P.sid.p;
        enqueue_wave(w, scene_tab[0], fshade, pv, P.qb.p, depth, st, [&](const PathView& v, int* cnt) {
            k_trace_primary_batch<<<w.g_trace0, 128, 0, st>>>(v, d_jobs, (int)tab.size(), (int)slots, n_wave, cnt, w.bins);
        }, [](int, const PathView&, int*, const int*) {}, [](int, int, int, auto&& launch) { launch(); },
        d_jobs, (int)tab.size(), (int)slots);
        for (const PieceFilm& pf : films) {
            const int np_j = (int)(film_off[(size_t)pf.job + 1] - film_off[(size_t)pf.job]);
            k_film<<<(np_j + 255) / 256, 256, 0, st>>>(np_j, pf.spw, P.rad.p + pf.path_base, P.film.p + film_off[pf.job]);
        }
        CK(cudaGetLastError());
        PathsCount pc{};
        if (w.depths > 0)
            CK(cudaMemcpy2DAsync(hcnt.data(), 32, P.counters.p, sizeof(int) * kCountersPerDepth, 32, (size_t)w.depths,
                                 cudaMemcpyDeviceToHost, st));
        if (w.depths < depth || w.stop >= 0)
            CK(cudaMemcpyAsync(&pc, P.errors.p + 4, sizeof(pc), cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        wave_totals(w, hcnt.data(), pc, seg, shadows);
        ++waves;
    }
    for (int k = 0; k < n && status == LUCID_OK; ++k) {
        const LucidRenderParams& p = items[k].p;
        const int np_k = p.tile_w * p.tile_h;
        k_output<<<(np_k + 255) / 256, 256, 0, st>>>(p.tile_w, p.tile_h, P.film.p + film_off[k], P.out.p + film_off[k]);
    }
    cudaEventRecord(t1, st);
    int herr[4] = {0, 0, 0, 0};
    CK(cudaMemcpyAsync(herr, P.errors.p, sizeof(herr), cudaMemcpyDeviceToHost, st));
    if (status == LUCID_OK)
        for (int k = 0; k < n; ++k)
            CK(cudaMemcpyAsync(items[k].out_host, P.out.p + film_off[k],
                               (film_off[(size_t)k + 1] - film_off[k]) * sizeof(float4), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    host_images.copied = status == LUCID_OK;
    float tot = 0.0f;
    cudaEventElapsedTime(&tot, t0, t1);
    cudaEventDestroy(t0);
    cudaEventDestroy(t1);
    stats_.total_ms = tot;
    stats_.paths = (double)total_paths;
    stats_.segments = seg;
    stats_.shadow_rays = shadows;
    stats_.waves = waves;
    if (herr[0] != 0) return fail(LUCID_ERR_OVERFLOW, "BVH traversal stack overflow");
    if (status == LUCID_ERR_CANCELLED) return fail(LUCID_ERR_CANCELLED, "render cancelled");
    return LUCID_OK;
}

// ---------------------------------------------------------------- path guiding (host)
int Engine::guide_buffers(long long paths) {
    GuideState& G = *guide_;
    if (G.cap < paths) {
        CK(G.gmix.alloc((size_t)paths * kGMixFloats));
        CK(G.gslot.alloc((size_t)paths));
        CK(G.ginv.alloc((size_t)paths * 3));
        G.cap = paths;
    }
    if ((long long)G.recs.n < (long long)G.steps * kGuideBatch) CK(G.recs.alloc((size_t)G.steps * kGuideBatch));
    if (!G.count.p) CK(G.count.alloc(2));
    return LUCID_OK;
}

int Engine::guide_enable(bool on, int seed) {
    GpuLock gl(*this);
    CK(cudaSetDevice(device_));
    if (!on) {
        if (guide_) guide_->on = false;
        return LUCID_OK;
    }
    int rc = ensure_stream();
    if (rc != LUCID_OK) return rc;
    if (!guide_) guide_ = new GuideState();
    if (guide_->net.init(seed, S(stream_)) != 0) return fail(LUCID_ERR_CUDA, "guide init: " + guide_->net.error());
    CK(cudaStreamSynchronize(S(stream_)));
    guide_->keep = 1.0f;
    guide_->on = true;
    return LUCID_OK;
}

int Engine::guide_steps() const { return guide_ ? guide_->net.steps() : 0; }

int Engine::guide_params(float* out, size_t cap, float* box6) {
    GpuLock gl(*this);
    if (!guide_) return fail(LUCID_ERR_INVALID, "guide: not enabled on this context");
    if (cap < (size_t)kGuideParams) return fail(LUCID_ERR_INVALID, "guide: output buffer too small");
    CK(cudaSetDevice(device_));
    if (guide_->net.get_params(out, S(stream_)) != 0) return fail(LUCID_ERR_CUDA, guide_->net.error());
    if (box6)
        for (int k = 0; k < 3; ++k) { box6[k] = scene_lo_[k]; box6[3 + k] = scene_hi_[k]; }
    return kGuideParams;
}

int Engine::guide_config(int steps_per_wave, float lr) {
    GpuLock gl(*this);
    if (steps_per_wave < 1 || steps_per_wave > 64 || !(lr > 0.0f)) return fail(LUCID_ERR_INVALID, "guide: bad config");
    if (!guide_) guide_ = new GuideState();
    guide_->steps = steps_per_wave;
    guide_->lr = lr;
    return LUCID_OK;
}

int Engine::guide_max_depth(int max_depth) {
    GpuLock gl(*this);
    if (max_depth < 1 || max_depth > kMaxDepth) return fail(LUCID_ERR_INVALID, "guide: bad guided depth");
    if (!guide_) guide_ = new GuideState();
    guide_->max_depth = max_depth;
    return LUCID_OK;
}

// ---------------------------------------------------------------- progressive jobs
// A job renders one image progressively: each iteration adds n samples to a
// film that keeps its sum across iterations, pixel by pixel in sample order,
// so a job's image is bit-identical to one render call with all its samples
// (camera rays are jittered whenever the job has more than one sample, as in
// that call).  Iterations of `chunk` samples are captured once into a CUDA
// graph and replayed; the sample offset comes from a device integer that a
// one-thread kernel sets before each replay.  Nothing in an iteration waits
// for the host, so iterations of jobs on different engines (streams) overlap
// on the device.
__global__ void k_set_int(int* p, int v) { *p = v; }

struct JobState {
    int w = 0, h = 0, spp = 0, depth = 8, chunk = 1;
    bool active = false;
    cudaGraphExec_t graph = nullptr;
    cudaEvent_t ev[2] = {nullptr, nullptr};   // iteration k records ev[k & 1]
    long long issued = 0;
    DBuf<int> dyn;
    FrameParams f{};
    int profile = 0;   // launch profile of the job's kernels
};

long long Engine::job_bytes(int w, int h, int chunk) {
    const long long np = (long long)w * h;
    return (long long)chunk * np * 176 + np * 32 + (1 << 20);   // path state (174 B) with slack
}

void Engine::enqueue_iteration(void* fp, int n) {
    JobState& J = *job_;
    FrameParams f = *static_cast<const FrameParams*>(fp);
    PathPool& P = *pool_;
    cudaStream_t st = S(stream_);
    f.s0 = 0;
    f.samples = n;
    f.n_wave = n * f.npix;
    const WavePlan w = wave_plan(device_, num_sms_, algo_, false, J.profile, false, f.n_wave, J.depth);
    if (w.depths > 0) cudaMemsetAsync(P.counters.p, 0, sizeof(int) * kCountersPerDepth * (w.depths + 1), st);
    enqueue_wave(w, ds_->view, f, P.view, P.qb.p, J.depth, st, [&](const PathView& pv, int* cnt) {
        k_trace_primary_for(ds_->view, f.pos)<<<w.g_trace0, 128, 0, st>>>(ds_->view, f, pv, cnt, 0, w.bins);
    }, [](int, const PathView&, int*, const int*) {}, [](int, int, int, auto&& launch) { launch(); });
    k_film<<<(f.npix + 255) / 256, 256, 0, st>>>(f.npix, n, P.rad.p, P.film.p);
}

int Engine::job_begin(int w, int h, int spp, int max_depth, int chunk, bool use_graph) {
    GpuLock gl(*this);
    if (w <= 0 || h <= 0 || spp <= 0 || chunk <= 0) return fail(LUCID_ERR_INVALID, "job: sizes must be positive");
    if (max_depth <= 0 || max_depth > kMaxDepth) return fail(LUCID_ERR_INVALID, "job: bad max_depth");
    if (!scene_loaded_ || !camera_set_) return fail(LUCID_ERR_NO_SCENE, "scene or camera not set");
    if ((long long)w * h * chunk > 0x7fffffffLL) return fail(LUCID_ERR_INVALID, "job: chunk too large");
    CK(cudaSetDevice(device_));
    job_end_locked();
    if (!job_) job_ = new JobState();
    JobState& J = *job_;
    J.w = w; J.h = h; J.spp = spp; J.depth = max_depth; J.chunk = std::min(chunk, spp);
    const size_t np = (size_t)w * h;
    int rc = ensure_pool((long long)J.chunk * (long long)np, false);
    if (rc != LUCID_OK) return rc;
    PathPool& P = *pool_;
    if (P.film_n < np) {
        CK(P.film.alloc(np));
        CK(P.out.alloc(np));
        P.film_n = np;
    }
    cudaStream_t st = S(stream_);
    CK(cudaMemsetAsync(P.film.p, 0, np * sizeof(float4), st));
    CK(cudaMemsetAsync(P.errors.p, 0, kErrorInts * sizeof(int), st));
    if (!J.dyn.p) CK(J.dyn.alloc(1));
    FrameParams& f = J.f;
    f = FrameParams{};
    for (int k = 0; k < 3; ++k) { f.pos[k] = cam_.pos[k]; f.fwd[k] = cam_.forward[k]; f.right[k] = cam_.right[k]; f.up[k] = cam_.up[k]; }
    f.aspect = (float)w / (float)h;
    f.scale = std::tan(cam_.fov * 0.5f);
    f.tile_w = w; f.tile_h = h; f.full_w = w; f.full_h = h;
    f.max_depth = max_depth; f.algo = algo_;
    f.npix = (int)np;
    f.jitter = spp > 1 ? 1 : 0;
    J.profile = launch_profile_;
    for (int k = 0; k < 2; ++k)
        if (!J.ev[k]) CK(cudaEventCreateWithFlags(&J.ev[k], cudaEventDisableTiming));
    J.issued = 0;
    J.active = true;
    return use_graph ? capture_locked(J.chunk) : LUCID_OK;
}

// Captures one iteration of `chunk` samples into a graph (chunk <= the
// chunk the job's path state was sized for).
int Engine::capture_locked(int chunk) {
    JobState& J = *job_;
    cudaStream_t st = S(stream_);
    if (J.graph) { cudaGraphExecDestroy(J.graph); J.graph = nullptr; }
    FrameParams fg = J.f;
    fg.dyn = J.dyn.p;
    cudaGraph_t graph = nullptr;
    CK(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    enqueue_iteration(&fg, chunk);
    cudaError_t e = cudaStreamEndCapture(st, &graph);
    if (e != cudaSuccess) return fail(LUCID_ERR_CUDA, std::string("graph capture: ") + cudaGetErrorString(e));
    e = cudaGraphInstantiate(&J.graph, graph, 0);
    cudaGraphDestroy(graph);
    if (e != cudaSuccess) { J.graph = nullptr; return fail(LUCID_ERR_CUDA, std::string("graph instantiate: ") + cudaGetErrorString(e)); }
    J.chunk = chunk;
    return LUCID_OK;
}

int Engine::set_launch_profile(int profile) {
    GpuLock gl(*this);
    if (profile < 0 || profile >= kLaunchProfiles) return fail(LUCID_ERR_INVALID, "unknown launch profile");
    launch_profile_ = profile;
    return LUCID_OK;
}

int Engine::job_set_profile(int profile, bool use_graph) {
    GpuLock gl(*this);
    if (!job_ || !job_->active) return fail(LUCID_ERR_INVALID, "no job");
    if (profile < 0 || profile >= kLaunchProfiles) return fail(LUCID_ERR_INVALID, "unknown launch profile");
    CK(cudaSetDevice(device_));
    // iterations in flight were enqueued with the old grids; they finish first
    CK(cudaStreamSynchronize(S(stream_)));
    job_->profile = profile;
    if (use_graph) return capture_locked(job_->chunk);
    if (job_->graph) { cudaGraphExecDestroy(job_->graph); job_->graph = nullptr; }
    return LUCID_OK;
}

int Engine::job_set_chunk(int chunk, bool use_graph) {
    GpuLock gl(*this);
    if (!job_ || !job_->active) return fail(LUCID_ERR_INVALID, "no job");
    if (chunk <= 0 || (long long)chunk * job_->w * job_->h > pool_->cap)
        return fail(LUCID_ERR_INVALID, "job: chunk exceeds the job's path state");
    CK(cudaSetDevice(device_));
    if (use_graph) return capture_locked(chunk);
    if (job_->graph) { cudaGraphExecDestroy(job_->graph); job_->graph = nullptr; }
    job_->chunk = chunk;
    return LUCID_OK;
}

int Engine::job_iterate(int sample_offset, int n) {
    GpuLock gl(*this);
    if (!job_ || !job_->active) return fail(LUCID_ERR_INVALID, "no job");
    JobState& J = *job_;
    if (n <= 0 || n > J.chunk) return fail(LUCID_ERR_INVALID, "job: iteration size must be in [1, chunk]");
    CK(cudaSetDevice(device_));
    cudaStream_t st = S(stream_);
    // at most two iterations in flight per job: wait for iteration k - 2
    if (J.issued >= 2) CK(cudaEventSynchronize(J.ev[J.issued & 1]));
    if (J.graph && n == J.chunk) {
        k_set_int<<<1, 1, 0, st>>>(J.dyn.p, sample_offset);
        CK(cudaGraphLaunch(J.graph, st));
    } else {
        FrameParams f = J.f;
        f.sample_offset = sample_offset;
        enqueue_iteration(&f, n);
    }
    CK(cudaGetLastError());
    CK(cudaEventRecord(J.ev[J.issued & 1], st));
    ++J.issued;
    return LUCID_OK;
}

int Engine::job_wait() {
    GpuLock gl(*this);
    CK(cudaSetDevice(device_));
    CK(cudaStreamSynchronize(S(stream_)));
    int herr[4] = {0, 0, 0, 0};
    CK(cudaMemcpy(herr, pool_->errors.p, sizeof(herr), cudaMemcpyDeviceToHost));
    if (herr[0] != 0) return fail(LUCID_ERR_OVERFLOW, "BVH traversal stack overflow");
    return LUCID_OK;
}

int Engine::job_output(float* out_host) {
    GpuLock gl(*this);
    if (!job_ || !job_->active) return fail(LUCID_ERR_INVALID, "no job");
    JobState& J = *job_;
    CK(cudaSetDevice(device_));
    cudaStream_t st = S(stream_);
    const int np = J.w * J.h;
    k_output<<<(np + 255) / 256, 256, 0, st>>>(J.w, J.h, pool_->film.p, pool_->out.p);
    CK(cudaMemcpyAsync(out_host, pool_->out.p, (size_t)np * sizeof(float4), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    return LUCID_OK;
}

long long Engine::guide_job_bytes(long long paths) {
    // per path: compact mixture (40 floats), slot and inverse-throughput
    // entries; fixed: two batches of records, the feature-major training
    // workspace and the per-block partial gradients
    return paths * (kGMixFloats * 4 + 16 + 48) + 2LL * kGuideBatch * (long long)sizeof(GuideRec) +
           608LL * kGuideBatch * 2 + 148LL * 51200 * 4 + (1 << 20);
}

int Engine::accum_begin(int w, int h) {
    GpuLock gl(*this);
    if (w <= 0 || h <= 0) return fail(LUCID_ERR_INVALID, "accumulator: sizes must be positive");
    CK(cudaSetDevice(device_));
    int rc = ensure_stream();
    if (rc != LUCID_OK) return rc;
    const size_t np = (size_t)w * h;
    if (jacc_n_ < np) {
        if (jacc_) cudaFree(jacc_);
        jacc_ = nullptr;
        jacc_n_ = 0;
        CK(cudaMalloc(&jacc_, np * sizeof(float4)));
        jacc_n_ = np;
    }
    jacc_w_ = w;
    jacc_h_ = h;
    CK(cudaMemsetAsync(jacc_, 0, np * sizeof(float4), S(stream_)));
    return LUCID_OK;
}

int Engine::render_accumulate(const LucidRenderParams& p) {
    GpuLock gl(*this);
    if (!jacc_ || p.tile_w != jacc_w_ || p.tile_h != jacc_h_) return fail(LUCID_ERR_INVALID, "accumulator size mismatch");
    return render_impl(p, nullptr, nullptr, nullptr, jacc_, false);
}

int Engine::accum_output(float* out_host) {
    GpuLock gl(*this);
    if (!jacc_) return fail(LUCID_ERR_INVALID, "no accumulator");
    CK(cudaSetDevice(device_));
    cudaStream_t st = S(stream_);
    const int np = jacc_w_ * jacc_h_;
    PathPool& P = *pool_;
    if (P.film_n < (size_t)np) { CK(P.film.alloc(np)); CK(P.out.alloc(np)); P.film_n = np; }
    k_output<<<(np + 255) / 256, 256, 0, st>>>(jacc_w_, jacc_h_, (const float4*)jacc_, P.out.p);
    CK(cudaMemcpyAsync(out_host, P.out.p, (size_t)np * sizeof(float4), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    return LUCID_OK;
}

void Engine::accum_end() {
    GpuLock gl(*this);
    if (!jacc_) return;
    cudaSetDevice(device_);
    if (stream_) cudaStreamSynchronize(S(stream_));
    cudaFree(jacc_);
    jacc_ = nullptr;
    jacc_n_ = 0;
}

void Engine::guide_free() {
    GpuLock gl(*this);
    if (!guide_) return;
    cudaSetDevice(device_);
    if (stream_) cudaStreamSynchronize(S(stream_));
    delete guide_;
    guide_ = nullptr;
}

void Engine::job_end_locked() {
    if (!job_) return;
    if (stream_) cudaStreamSynchronize(S(stream_));
    if (job_->graph) { cudaGraphExecDestroy(job_->graph); job_->graph = nullptr; }
    job_->active = false;
}

void Engine::job_end() {
    GpuLock gl(*this);
    cudaSetDevice(device_);
    job_end_locked();
    if (job_)
        for (int k = 0; k < 2; ++k)
            if (job_->ev[k]) cudaEventDestroy(job_->ev[k]);
    delete job_;
    job_ = nullptr;
}

void Engine::release_pool() {
    GpuLock gl(*this);
    cudaSetDevice(device_);
    if (stream_) cudaStreamSynchronize(S(stream_));
    pool_->release();
}

// ---------------------------------------------------------------- async accumulator
// The viewport's progressive mode (PyRenderer::render_start_async ..
// render_stop_async, pybind_renderer.hpp:689-856; the Dawn worker it drives,
// gpu/path_tracer.cpp:838-1090): a worker thread adds one 1-spp render per
// iteration (sample offset n, so iteration n seeds (x, y, n)) into a device
// accumulator and publishes an averaged snapshot after 1, 2, 4, 8 and then
// every 16 samples.  reset() wipes the accumulator without stopping.
int Engine::async_start(int w, int h, int max_depth) {
    async_stop();
    if (w <= 0 || h <= 0) return fail(LUCID_ERR_INVALID, "async: size must be positive");
    if (!scene_loaded_ || !camera_set_) return fail(LUCID_ERR_NO_SCENE, "scene or camera not set");
    {
        GpuLock gl(*this);
        CK(cudaSetDevice(device_));
        size_t n = (size_t)w * h;
        if (async_acc_n_ < n) {
            if (async_acc_) cudaFree(async_acc_);
            if (async_pinned_) cudaFreeHost(async_pinned_);
            async_acc_ = nullptr;
            async_pinned_ = nullptr;
            async_acc_n_ = 0;
            CK(cudaMalloc(&async_acc_, n * sizeof(float4)));
            CK(cudaMallocHost((void**)&async_pinned_, n * sizeof(float4)));
            async_acc_n_ = n;
        }
        CK(cudaMemset(async_acc_, 0, n * sizeof(float4)));
        async_w_ = w; async_h_ = h; async_depth_ = std::max(1, max_depth);
    }
    {
        std::lock_guard<std::mutex> sl(snap_mu_);
        snap_.clear();
        snap_samples_ = 0;
    }
    async_reset_ = false;
    async_run_ = true;
    async_thread_ = std::thread([this] { async_worker(); });
    return LUCID_OK;
}

int Engine::async_reset(int w, int h, int max_depth) {
    if (!async_run_) return LUCID_OK;
    if ((size_t)w * h > async_acc_n_ || w <= 0 || h <= 0)
        return fail(LUCID_ERR_INVALID, "async reset: a larger resolution needs stop + start");
    {
        GpuLock gl(*this);
        async_w_ = w; async_h_ = h; async_depth_ = std::max(1, max_depth);
    }
    async_reset_ = true;
    return LUCID_OK;
}

int Engine::async_stop() {
    async_run_ = false;
    if (async_thread_.joinable()) async_thread_.join();
    return LUCID_OK;
}

int Engine::async_poll(int* samples, float* out, size_t cap_floats) {
    std::lock_guard<std::mutex> sl(snap_mu_);
    *samples = snap_samples_;
    if (snap_samples_ == 0) return LUCID_OK;
    if (!out || cap_floats < snap_.size()) return fail(LUCID_ERR_INVALID, "async poll: output buffer too small");
    std::copy(snap_.begin(), snap_.end(), out);
    return LUCID_OK;
}

void Engine::async_worker() {
    cudaSetDevice(device_);
    long long n = 0;
    int w = 0, h = 0, depth = 8;
    while (async_run_) {
        bool wipe = async_reset_.exchange(false);
        // std::mutex is not fair: back off while an API call waits for the
        // GPU, or a set_camera / reset from the UI thread could wait for
        // minutes behind the worker's back-to-back iterations
        while (gpu_waiters_.load() > 0 && async_run_) std::this_thread::sleep_for(std::chrono::microseconds(100));
        {
            std::lock_guard<std::mutex> gl(gpu_mu_);
            if (wipe || w != async_w_ || h != async_h_) {
                w = async_w_; h = async_h_;
                cudaMemsetAsync(async_acc_, 0, (size_t)w * h * sizeof(float4), S(stream_));
                n = 0;
            }
            depth = async_depth_;
            LucidRenderParams p{0, 0, w, h, w, h, 1, (int)n, depth, 0};
            int rc = render_impl(p, nullptr, nullptr, nullptr, async_acc_, true);
            if (rc != LUCID_OK) {
                async_err_ = err_;
            } else {
                ++n;
                if (n <= 8 ? ((n & (n - 1)) == 0) : (n % 16 == 0)) {
                    size_t np = (size_t)w * h;
                    cudaMemcpyAsync(async_pinned_, async_acc_, np * sizeof(float4), cudaMemcpyDeviceToHost, S(stream_));
                    cudaStreamSynchronize(S(stream_));
                    // average, camera sensitivity (EV 0 -> 1), clamp >= 0, alpha 1, Y flip
                    std::vector<float> img(np * 4);
                    const float inv = (float)n;
                    for (int y = 0; y < h; ++y)
                        for (int x = 0; x < w; ++x) {
                            const float* a = async_pinned_ + 4 * ((size_t)y * w + x);
                            float* o = img.data() + 4 * ((size_t)(h - 1 - y) * w + x);
                            for (int c = 0; c < 3; ++c) {
                                float v = (a[c] / inv) * 1.0f;
                                o[c] = (v < 0.0f) ? 0.0f : v;
                            }
                            o[3] = 1.0f;
                        }
                    std::lock_guard<std::mutex> sl(snap_mu_);
                    snap_.swap(img);
                    snap_samples_ = (int)n;
                    async_revision_.fetch_add(1);
                }
            }
        }
        if (async_err_.size()) {
            std::this_thread::sleep_for(std::chrono::milliseconds(2));   // the reference backs off 2 ms
            async_err_.clear();
        }
    }
}

// ---------------------------------------------------------------- no-allocation render
// Some callers cannot allocate device memory when they render: a host whose
// device memory is owned by another allocator (a framework's caching pool
// that hands out every byte), or a latency-critical thread such as a
// viewport draw callback that must not call cudaMalloc/cudaFree because
// those calls can synchronise the whole device.  lucid_cuda_render_noalloc
// serves them with the whole-path kernel of lucid_cuda_render_device, but its
// working memory (a wave's radiance, the error words, the film) lives in the
// fixed-size device array below, which every GPU that loads this library
// holds until the process exits.  The scene itself was allocated earlier by
// lucid_cuda_load_scene_json.
constexpr int kNoAllocPaths = 65536;              // paths per wave
constexpr int kNoAllocPixels = 65536;             // tile pixels (e.g. 256 x 256)
constexpr int kNoAllocMaxDepth = 64;
static_assert(kNoAllocPaths <= kPathsWave, "its waves run in k_paths, which keeps a path's state in registers");
constexpr size_t kNoAllocAlign = 256;
constexpr size_t na_round(size_t b) { return (b + kNoAllocAlign - 1) / kNoAllocAlign * kNoAllocAlign; }
constexpr size_t kNaRad = na_round(sizeof(float4) * kNoAllocPaths);
constexpr size_t kNaErr = na_round(sizeof(int) * kErrorInts);
constexpr size_t kNaFilm = na_round(sizeof(float4) * kNoAllocPixels);
constexpr size_t kNoAllocBytes = kNaRad + kNaErr + kNaFilm;   // 2 MB

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

namespace {
// Device address of g_noalloc_scratch per device, looked up once with that
// device current (a host-side reference to the array is not a device
// address).
std::mutex g_noalloc_mu;
unsigned char* g_noalloc_addr[64] = {};
// Calls on one device, whichever context they are made on, take turns with the
// array: held until the call's work on it is done.
std::mutex g_noalloc_turn[64];
struct NoAllocTurn {
    std::unique_lock<std::mutex> lk;
    cudaStream_t st;
    bool done = false;   // the stream has been waited for
    NoAllocTurn(int device, cudaStream_t s) : lk(g_noalloc_turn[device]), st(s) {}
    ~NoAllocTurn() { if (!done) cudaStreamSynchronize(st); }   // (then lk is released)
};
}  // namespace

int Engine::render_noalloc(const LucidRenderParams& p, float* d_out) {
    GpuLock gl(*this);
    reset_cancel();
    if (!d_out) return fail(LUCID_ERR_INVALID, "output pointer is null");
    if (p.tile_w <= 0 || p.tile_h <= 0 || p.full_w <= 0 || p.full_h <= 0)
        return fail(LUCID_ERR_INVALID, "tile and image sizes must be positive");
    if (!scene_loaded_ || !camera_set_) return fail(LUCID_ERR_NO_SCENE, "scene or camera not set");
    long long np = (long long)p.tile_w * p.tile_h;
    if (np > kNoAllocPixels)
        return fail(LUCID_ERR_INVALID, "render_noalloc: tile of " + std::to_string(np) + " pixels exceeds the " +
                                           std::to_string(kNoAllocPixels) + "-pixel limit of its fixed scratch");
    if (p.max_depth < 1 || p.max_depth > kNoAllocMaxDepth)
        return fail(LUCID_ERR_INVALID, "render_noalloc: max_depth must be in [1, " + std::to_string(kNoAllocMaxDepth) + "]");
    if (p.samples <= 0) return fail(LUCID_ERR_INVALID, "samples must be >= 1");
    if (device_ < 0 || device_ >= 64) return fail(LUCID_ERR_INVALID, "device index out of range");
    if (algo_ < 0 || algo_ > 4) return fail(LUCID_ERR_INVALID, "unknown integrator");
    // Diagnostics and path guiding keep per-render buffers that this entry
    // point cannot allocate; rendering without them would give a different
    // image than lucid_cuda_render_device, so refuse instead.
    if (diag_enabled_)
        return fail(LUCID_ERR_INVALID, "render_noalloc: path diagnostics are enabled; they need allocated record "
                                       "buffers (disable them or use lucid_cuda_render_device)");
    if (guide_ && guide_->on && algo_ == ALGO_MIS)
        return fail(LUCID_ERR_INVALID, "render_noalloc: path guiding is on; it needs allocated training and "
                                       "inference buffers (turn it off or use lucid_cuda_render_device)");
    CK(cudaSetDevice(device_));
    unsigned char* base;
    {
        std::lock_guard<std::mutex> lk(g_noalloc_mu);
        if (!g_noalloc_addr[device_]) {
            void* ptr = nullptr;
            cudaError_t e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
            if (e != cudaSuccess || !ptr)
                return fail(LUCID_ERR_CUDA, std::string("cudaGetSymbolAddress(g_noalloc_scratch): ") + cudaGetErrorString(e));
            g_noalloc_addr[device_] = (unsigned char*)ptr;
        }
        base = g_noalloc_addr[device_];
    }
    PathView v{};
    v.rad = (float4*)base;
    v.errors = (int*)(base + kNaRad);
    float4* film = (float4*)(base + kNaRad + kNaErr);

    cudaStream_t st = S(stream_);
    NoAllocTurn turn(device_, st);
    // the array keeps the previous call's contents: clear what starts at zero
    CK(cudaMemsetAsync(film, 0, sizeof(float4) * np, st));
    CK(cudaMemsetAsync(v.errors, 0, sizeof(int) * kErrorInts, st));
    FrameParams f{};
    for (int k = 0; k < 3; ++k) { f.pos[k] = cam_.pos[k]; f.fwd[k] = cam_.forward[k]; f.right[k] = cam_.right[k]; f.up[k] = cam_.up[k]; }
    f.aspect = (float)p.full_w / (float)p.full_h;
    f.scale = std::tan(cam_.fov * 0.5f);
    f.tile_x = p.tile_x; f.tile_y = p.tile_y; f.tile_w = p.tile_w; f.tile_h = p.tile_h;
    f.full_w = p.full_w; f.full_h = p.full_h;
    f.samples = p.samples; f.sample_offset = p.sample_offset; f.max_depth = p.max_depth; f.algo = algo_;
    f.npix = (int)np;
    f.records = 0;
    const int spw = (int)std::max<long long>(1, std::min<long long>(p.samples, kNoAllocPaths / np));
    int status = LUCID_OK;
    for (int s0 = 0; s0 < p.samples; s0 += spw) {
        if (is_cancelled()) { status = LUCID_ERR_CANCELLED; break; }
        int this_spw = std::min(spw, p.samples - s0);
        f.s0 = s0;
        f.n_wave = (int)(this_spw * np);
        const WavePlan w = wave_plan(device_, num_sms_, algo_, false, 0, false, f.n_wave, p.max_depth);
        enqueue_paths(w, ds_->view, f, v, st, [](int, int, int, auto&& launch) { launch(); }, nullptr, 0, 0);
        k_film<<<(f.npix + 255) / 256, 256, 0, st>>>(f.npix, this_spw, v.rad, film);
        CK(cudaGetLastError());
        // no wait here: stream order keeps the next wave behind this film sum
    }
    k_output<<<(f.npix + 255) / 256, 256, 0, st>>>(p.tile_w, p.tile_h, film, (float4*)d_out);
    int herr[4] = {0, 0, 0, 0};
    CK(cudaMemcpyAsync(herr, v.errors, sizeof(herr), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    turn.done = true;
    if (herr[0] != 0) return fail(LUCID_ERR_OVERFLOW, "BVH traversal stack overflow");
    if (status == LUCID_ERR_CANCELLED) return fail(LUCID_ERR_CANCELLED, "render cancelled");
    return LUCID_OK;
}

int Engine::render_debug(int tx, int ty, int tw, int th, int fw, int fh, const char* mode, float* out_host) {
    GpuLock gl(*this);
    reset_cancel();
    if (tw <= 0 || th <= 0 || fw <= 0 || fh <= 0) return fail(LUCID_ERR_INVALID, "tile and image sizes must be positive");
    size_t np = (size_t)tw * th;
    std::fill(out_host, out_host + np * 4, 0.0f);
    if (!scene_loaded_ || !camera_set_) return fail(LUCID_ERR_NO_SCENE, "scene or camera not set");
    std::string m = mode ? mode : "";
    int md;
    if (m == "normal") md = 0;
    else if (m == "albedo") md = 1;
    else if (m == "emission") md = 2;
    else {
        // unknown mode: magenta, as render_debug does (pybind_renderer.hpp:420-422)
        for (size_t i = 0; i < np; ++i) { out_host[4 * i] = 1.0f; out_host[4 * i + 1] = 0.0f; out_host[4 * i + 2] = 1.0f; out_host[4 * i + 3] = 1.0f; }
        return LUCID_OK;
    }
    CK(cudaSetDevice(device_));
    cudaStream_t st = S(stream_);
    PathPool& P = *pool_;
    if (P.film_n < np) { CK(P.film.alloc(np)); CK(P.out.alloc(np)); P.film_n = np; }
    if (!P.errors.p) CK(P.errors.alloc(kErrorInts));
    CK(cudaMemsetAsync(P.errors.p, 0, kErrorInts * sizeof(int), st));
    FrameParams f{};
    for (int k = 0; k < 3; ++k) { f.pos[k] = cam_.pos[k]; f.fwd[k] = cam_.forward[k]; f.right[k] = cam_.right[k]; f.up[k] = cam_.up[k]; }
    f.aspect = (float)fw / (float)fh;
    f.scale = std::tan(cam_.fov * 0.5f);
    f.tile_x = tx; f.tile_y = ty; f.tile_w = tw; f.tile_h = th; f.full_w = fw; f.full_h = fh; f.npix = (int)np;
    k_debug<<<((int)np + 255) / 256, 256, 0, st>>>(ds_->view, f, md, P.out.p, P.errors.p);
    CK(cudaGetLastError());
    int herr[4];
    CK(cudaMemcpyAsync(herr, P.errors.p, sizeof(herr), cudaMemcpyDeviceToHost, st));
    CK(cudaMemcpyAsync(out_host, P.out.p, np * sizeof(float4), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    if (herr[0]) return fail(LUCID_ERR_OVERFLOW, "BVH traversal stack overflow");
    return LUCID_OK;
}

}  // namespace lucid
