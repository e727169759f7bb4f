// C ABI of the cloth solver: handle lifetime, validation, colour batches,
// AoS <-> SoA conversion at the boundary, and the cooperative launch.
//
// Replaces the reference Metal host runGPU (tools/cloth_bag_metal.mm:4010-4760):
// buffer allocation (:4091-4202), per-substep encoding (:4211-4709), commit
// and readback (:4710-4757), and the colouring check verifyColoring
// (tools/cloth_bag_metal.mm:1705-1819).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <initializer_list>
#include <memory>
#include <mutex>
#include <new>
#include <queue>
#include <system_error>
#include <thread>
#include <utility>
#include <vector>

#include "cloth_frame.cuh"
#include "cloth_adjoint.cuh"
#include "numi_cloth.h"

static_assert(sizeof(NumiClothConfig) == 224, "Config layout");
static_assert(sizeof(NumiClothParticle) == 48, "Particle layout");
static_assert(sizeof(NumiClothDistance) == 32, "Distance layout");
static_assert(sizeof(NumiClothGrip) == 48, "Grip layout");
static_assert(sizeof(NumiClothKnot) == 48, "Knot layout");
static_assert(sizeof(NumiClothBend) == 32, "Bend layout");
static_assert(sizeof(NumiClothFruit) == 96, "Fruit layout");
static_assert(sizeof(NumiClothFruitPair) == 32, "FruitPair layout");
static_assert(sizeof(NumiClothBatch) == 16, "Batch layout");
static_assert(offsetof(NumiClothConfig, gravityAndTimestep) == 48, "Config offsets");
static_assert(offsetof(NumiClothConfig, mouthMaterial) == 208, "Config offsets");
static_assert(sizeof(DeviceCloth) % 4u == 0u, "DeviceCloth is copied as 32-bit words");

__global__ void __launch_bounds__(NC_THREADS) numi_cloth_residual_kernel(DeviceCloth d, NumiClothConfig cfg) {
    Schedule s{};
    nc::Ctx ctx{d, s};
    ctx.gx = d.x;
    ctx.gv = d.v;
    ctx.c = nc::load_cfg(&cfg);
    ctx.tid = blockIdx.x * blockDim.x + threadIdx.x;
    ctx.nthreads = gridDim.x * blockDim.x;
    ctx.rank = blockIdx.x;
    ctx.ranks = gridDim.x;
    nc::residual_partials(ctx, d.red);
}

namespace {

constexpr uint32_t kSnapshotSlots = 8;
constexpr uint32_t kTuneSlot = kSnapshotSlots;   // snapshot slot of the launch-shape tuners
constexpr uint32_t kResidentChunk = 4096;   // particles a CTA holds in resident mode
constexpr uint32_t kResidentClusterChunk = 256;   // default chunk of a small resident cloth
constexpr uint32_t kBarrierWords = 48;   // barrier counter, abort, release and fruit flags: three 128-byte lines

struct Snapshot {
    bool valid = false;
    void* mem = nullptr;
    size_t bytes = 0;
    std::vector<float> grip_compliance;   // the grips' at the snapshot
};

bool env_u32(const char* name, uint32_t& out) {
    const char* v = std::getenv(name);
    if (v == nullptr || *v == 0) return false;
    out = static_cast<uint32_t>(std::strtoul(v, nullptr, 10));
    return true;
}

}  // namespace

// Typed pieces of one allocation, 256-byte aligned (with a null base the
// walk only measures).
struct Carver {
    char* base;
    size_t used = 0;
    template <class T>
    T* get(size_t count) {
        T* p = reinterpret_cast<T*>(base + used);
        used += (count * sizeof(T) + 255u) & ~size_t(255u);
        return p;
    }
};

cudaError_t device_malloc(void** p, size_t bytes);

// Device memory of the rollout gradients of one handle or batch: kept from
// call to call (an allocation and its release cost more than a small
// rollout) as long as all that the process keeps so takes no more than a
// sixteenth of the device's memory, else given back at the call's end.  It is
// freed with its owner, and when another allocation of the library finds no
// room.
struct Workspace {
    void* mem = nullptr;
    size_t bytes = 0, most = 0;   // most: what may be kept on its device
    int device = -1;
    bool busy = false;   // a call uses it
    Workspace* next = nullptr;   // every workspace of the process
    Workspace() {
        std::lock_guard<std::mutex> lock(mutex());
        next = std::exchange(first(), this);
    }
    Workspace(const Workspace&) = delete;
    Workspace& operator=(const Workspace&) = delete;
    ~Workspace() {
        std::lock_guard<std::mutex> lock(mutex());
        Workspace** at = &first();
        while (*at != this) at = &(*at)->next;
        *at = next;
        release();
    }
    void release() {
        if (mem != nullptr) cudaFree(mem);
        mem = nullptr;
        bytes = 0;
    }
    static std::mutex& mutex() {
        static std::mutex m;
        return m;
    }
    static Workspace*& first() {
        static Workspace* head = nullptr;
        return head;
    }
    // Gives back what no call uses on the device; false where that is nothing.
    static bool reclaim(int device) {
        std::lock_guard<std::mutex> lock(mutex());
        bool any = false;
        for (Workspace* w = first(); w != nullptr; w = w->next)
            if (!w->busy && w->mem != nullptr && w->device == device) {
                w->release();
                any = true;
            }
        return any;
    }
    // One call's use of it, on the current device.
    struct Lease {
        Workspace& w;
        cudaStream_t stream;
        Lease(Workspace& space, cudaStream_t s) : w(space), stream(s) {
            std::lock_guard<std::mutex> lock(mutex());
            w.busy = true;
            cudaGetDevice(&w.device);
        }
        ~Lease() {
            std::unique_lock<std::mutex> lock(mutex());
            size_t kept = 0;
            for (const Workspace* o = first(); o != nullptr; o = o->next)
                if (o->device == w.device) kept += o->bytes;
            if (kept > w.most) {
                lock.unlock();
                cudaStreamSynchronize(stream);
                lock.lock();
                w.release();
            }
            w.busy = false;
        }
        void hold(void* p, size_t bytes, size_t most) {
            std::lock_guard<std::mutex> lock(mutex());
            w.release();
            w.mem = p;
            w.bytes = bytes;
            w.most = most;
        }
        // False where the device has no room for the pieces; with `quarter`
        // also where they would take more than a quarter of what is free.
        template <class F>
        bool layout(F&& pieces, bool quarter = false) {
            Carver measure{nullptr};
            pieces(measure);
            if (measure.used > w.bytes) {
                size_t room = 0, total = 0;
                if (cudaMemGetInfo(&room, &total) != cudaSuccess) return false;
                if (quarter && measure.used > (room + w.bytes) / 4u) return false;
                // whatever ran on the old memory has ended
                if (w.mem != nullptr && cudaStreamSynchronize(stream) != cudaSuccess) return false;
                hold(nullptr, 0, 0);
                void* p = nullptr;
                if (device_malloc(&p, measure.used) != cudaSuccess) return false;
                hold(p, measure.used, total / 16u);
            }
            Carver c{static_cast<char*>(w.mem)};
            pieces(c);
            return true;
        }
    };
};

// cudaMalloc on the current device, which takes back idle workspaces where
// there is no room.
cudaError_t device_malloc(void** p, size_t bytes) {
    int device = 0;
    cudaGetDevice(&device);
    cudaError_t e = cudaMalloc(p, bytes);
    if (e == cudaErrorMemoryAllocation && Workspace::reclaim(device)) {
        cudaGetLastError();
        e = cudaMalloc(p, bytes);
    }
    if (e != cudaSuccess) cudaGetLastError();
    return e;
}

struct DeviceBuffers {
    std::vector<void*> owned;
    // Zeroed on the stream that uses it first (the default stream does not
    // order a non-blocking one's work).
    template <class T>
    T* alloc(size_t count, cudaStream_t stream = nullptr) {
        if (count == 0) count = 1;
        void* p = nullptr;
        if (device_malloc(&p, count * sizeof(T)) != cudaSuccess) return nullptr;
        cudaMemsetAsync(p, 0, count * sizeof(T), stream);
        owned.push_back(p);
        return static_cast<T*>(p);
    }
    ~DeviceBuffers() {
        for (void* p : owned) cudaFree(p);
    }
};

// What the tile plans of a cloth are made from: its colours, grid width and
// particles, the ends of its records, and the shape of the tile launch.
struct TileSource {
    DeviceCloth d;
    uint32_t grid = 0;   // CTAs of the tile launch
    size_t smem_budget = 0;
    std::vector<uint2> distances, bends;
};

// A plan on the device, with the buffers that a tile launch alternates to;
// one allocation.
struct TileBlock {
    void* mem = nullptr;
    uint32_t* words = nullptr;
    uint32_t* off = nullptr;
    uint32_t* owner = nullptr;
    float4 *x_alt = nullptr, *v_alt = nullptr;
    bool stream = false;
    size_t smem = 0;
    TileBlock() = default;
    TileBlock(const TileBlock&) = delete;
    TileBlock& operator=(const TileBlock&) = delete;
    TileBlock& operator=(TileBlock&& o) noexcept {
        if (mem != nullptr) cudaFree(mem);
        mem = std::exchange(o.mem, nullptr);
        words = o.words;
        off = o.off;
        owner = o.owner;
        x_alt = o.x_alt;
        v_alt = o.v_alt;
        stream = o.stream;
        smem = o.smem;
        return *this;
    }
    ~TileBlock() {
        if (mem != nullptr) cudaFree(mem);
    }
};

struct TileJob {
    TileSource source;
    int device = 0;
    TileBlock block;   // no memory where the plan did not fit
    enum { kQueued, kRunning, kDone } state = kQueued;
};

struct numi_cloth {
    int device = 0;
    cudaStream_t stream = nullptr;
    DeviceBuffers buf;
    DeviceCloth d{};
    NumiClothConfig base{};
    NumiClothConfig* d_cfg = nullptr;
    uint32_t cfg_capacity = 0;
    uint32_t epoch = 1;
    uint32_t host_failure = 0;
    bool poisoned = false;
    bool self_exact = false;   // point self contact in the reference's order (NUMI_CLOTH_SELF_ORDER=reference)
    uint32_t grid = 1;
    uint32_t block = NC_THREADS;
    uint32_t cluster = 0;   // > 0: the grid is one cluster of this many CTAs
    size_t smem = nc_resident_offset();   // dynamic shared memory of a frame launch
    uint32_t launches = 0;
    uint32_t trace_capacity = 0;   // substeps the trace buffer holds
    uint32_t trace_ctas = 0;       // CTAs its per-CTA part holds
    uint32_t last_substeps = 0;
    float yarn_rest_median = 0.0f;   // median yarn segment rest length
    bool neighbours = false;         // neighbour-sync tables built for the cooperative grid
    size_t nbr_smem = 0;             // dynamic shared memory of a frame launch with them
    // tile mode (cloth_tile.cuh): plan, launch shape and shared memory of a
    // tile launch
    bool tiles = false;
    TileBlock plan;
    uint32_t tile_grid = 0, tile_block = 0;
    size_t tile_smem = 0;
    // a small cloth that will have a plan: what it is made from until the
    // build is under way, and the substeps it has stepped (or is about to)
    // that a plan covers
    std::unique_ptr<TileSource> tile_source;
    std::shared_ptr<TileJob> tile_job;
    uint32_t tile_substeps = 0;
    uint32_t last_grid = 0, last_block = 0;
    bool last_tiles = false;
    // host copies for the edge/edge local lists, built with the edge buffers
    std::vector<uint2> host_yarn;
    std::vector<uint32_t> host_local_off, host_local_idx;
    Snapshot snaps[kSnapshotSlots + 1u];   // the callers' slots, then the tuners' own
    // Host copy of what the compliance groups are made of: per family
    // (distance, knot, bend) the distinct values, ascending, and every
    // record's index among them (read from the device when first asked for,
    // then kept in step by numi_cloth_replace_compliance, the only writer);
    // and every grip's compliance, which a restore brings back with the grips.
    // What a graph replays the host does not see: once a change was captured,
    // both are read from the device every time.
    bool compliance_known = false;
    bool compliance_captured = false;
    std::vector<float> compliance[3];
    std::vector<uint8_t> compliance_id[3];
    std::vector<float> grip_compliance;
    // dynamic state regions copied by snapshot/restore
    struct Region {
        void* ptr;
        size_t bytes;
    };
    std::vector<Region> dynamic;
    // device staging of particle records for the host copies (one transfer
    // each way, transposed to and from the state arrays on the device)
    NumiClothParticle* io = nullptr;
    Workspace grad;   // rollout gradients
    bool rollout_touched = false;   // a fruit touched the cloth in the last rollout
};

namespace {

// cudaFuncAttributeMaxDynamicSharedMemorySize is per function, not per
// launch, and cloths with different launch modes share the frame kernel: only
// ever raise it, so that creating one cloth never breaks another's launch.
// The frame and batch kernels come in two builds: without and with the
// edge/edge yarn self-collision phases (primitiveSelf).
// A third pair resolves point self contact in the reference's Gauss-Seidel
// order (NUMI_CLOTH_SELF_ORDER=reference at create).
const void* frame_fn(bool edge, bool exact = false) {
    if (exact)
        return edge ? reinterpret_cast<const void*>(numi_cloth_frame_edge_exact_kernel)
                    : reinterpret_cast<const void*>(numi_cloth_frame_exact_kernel);
    return edge ? reinterpret_cast<const void*>(numi_cloth_frame_edge_kernel)
                : reinterpret_cast<const void*>(numi_cloth_frame_kernel);
}
const void* batch_fn(bool edge) {
    return edge ? reinterpret_cast<const void*>(numi_cloth_batch_edge_kernel)
                : reinterpret_cast<const void*>(numi_cloth_batch_kernel);
}

const void* batch_cluster_fn() { return reinterpret_cast<const void*>(numi_cloth_batch_cluster_kernel); }
// The kernels of rollout gradients (for handles of either self-contact order:
// their schedules have none).
const void* frame_tape_fn() { return reinterpret_cast<const void*>(numi_cloth_frame_tape_kernel); }
const void* batch_tape_fn(bool cluster) {
    return cluster ? reinterpret_cast<const void*>(numi_cloth_batch_cluster_tape_kernel)
                   : reinterpret_cast<const void*>(numi_cloth_batch_tape_kernel);
}
const std::initializer_list<const void*> kFrameKernels = {frame_fn(false), frame_fn(true), frame_fn(false, true),
                                                          frame_fn(true, true), frame_tape_fn()};

cudaError_t raise_smem(const void* fn, size_t bytes) {
    cudaFuncAttributes fa{};
    cudaError_t e = cudaFuncGetAttributes(&fa, fn);
    if (e != cudaSuccess) return e;
    if (static_cast<size_t>(fa.maxDynamicSharedSizeBytes) >= bytes) return cudaSuccess;
    return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
}
cudaError_t raise_frame_smem(size_t bytes) {
    cudaError_t e = cudaSuccess;
    for (const void* fn : kFrameKernels)
        if (e == cudaSuccess) e = raise_smem(fn, bytes);
    return e;
}
void allow_large_clusters() {
    for (const void* fn : kFrameKernels) cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
}
// Clusters of cfg's shape that every frame kernel can place at once.
int frame_clusters(const cudaLaunchConfig_t& cfg) {
    int lo = 1 << 30;
    for (const void* fn : kFrameKernels) {
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, fn, &cfg) != cudaSuccess) return 0;
        lo = std::min(lo, clusters);
    }
    return lo;
}
// Shared memory of its own the larger of a handle's tile-mode kernels has.
size_t tile_static_smem(const numi_cloth* h) {
    cudaFuncAttributes fa{}, ft{};
    cudaFuncGetAttributes(&fa, frame_fn(false, h->self_exact));
    cudaFuncGetAttributes(&ft, frame_tape_fn());
    return std::max(fa.sharedSizeBytes, ft.sharedSizeBytes);
}
// Whether the device holds the handle's tile launch co-resident.
bool tiles_fit(const numi_cloth* h) {
    int sms = 0, lo = 1 << 30;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, h->device);
    if (raise_frame_smem(h->tile_smem) != cudaSuccess) return false;
    for (const void* fn : {frame_fn(false, h->self_exact), frame_tape_fn()}) {
        int k = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&k, fn, NC_BLOCK_MAX, h->tile_smem) != cudaSuccess) return false;
        lo = std::min(lo, k);
    }
    return static_cast<uint64_t>(lo) * static_cast<uint64_t>(sms) >= h->tile_grid;
}

bool finite4(const numi_float4& v) {
    return std::isfinite(v.x) && std::isfinite(v.y) && std::isfinite(v.z) && std::isfinite(v.w);
}

// Host twin of the reference validConfig (ClothBag.metal:16-55).
uint32_t validate_config(const NumiClothConfig& c, const NumiClothConfig& base) {
    if (c.control.x != NUMI_CLOTH_ABI_VERSION) return NUMI_CLOTH_FAILURE_ABI;
    if (c.control.y != base.control.y || c.control.z != base.control.z || c.control.w != base.control.w ||
        c.constraintCounts.x != base.constraintCounts.x || c.constraintCounts.y != base.constraintCounts.y ||
        c.constraintCounts.w != base.constraintCounts.w || c.contactCounts.x != base.contactCounts.x)
        return NUMI_CLOTH_FAILURE_RANGE;
    const float dt = c.gravityAndTimestep.w;
    bool ok = dt > 0.0f && std::isfinite(dt) && finite4(c.gravityAndTimestep) && finite4(c.gripTargetAndActive) &&
              finite4(c.gripOrientation) && finite4(c.gripMaterial) && finite4(c.clothMaterial) &&
              finite4(c.fruitMaterial) && finite4(c.airVelocityAndDensity) && finite4(c.aerodynamicCoefficients) &&
              finite4(c.mouthMaterial) && c.clothMaterial.x >= 0.0f && c.airVelocityAndDensity.w >= 0.0f &&
              c.aerodynamicCoefficients.x >= 0.0f && c.aerodynamicCoefficients.y >= 0.0f &&
              c.aerodynamicCoefficients.z >= 0.0f && c.aerodynamicCoefficients.w >= 0.0f &&
              c.gripMaterial.x >= 0.0f && c.gripControl.y <= 1u && c.mouthMaterial.x >= 0.0f &&
              c.mouthControl.x <= NUMI_CLOTH_MOUTH_RIM_CAPACITY;
    if (ok && c.gripTargetAndActive.w > 0.0f) {
        const numi_float4& q = c.gripOrientation;
        const float len = std::sqrt(q.x * q.x + q.y * q.y + q.z * q.z + q.w * q.w);
        ok = std::fabs(len - 1.0f) <= 1.0e-4f && c.gripControl.x != 0u && c.gripMaterial.x > 0.0f;
    }
    if (ok && c.gripControl.y == 1u) {
        ok = c.gripControl.z >= 2u * c.gripControl.w + 1u && c.gripControl.z <= NUMI_CLOTH_MOUTH_RIM_CAPACITY &&
             c.gripControl.w <= 16u && c.control.w == 2u * (2u * c.gripControl.w + 1u);
    }
    return ok ? 0u : NUMI_CLOTH_FAILURE_NONFINITE;
}

// Colour runs -> batches; checks contiguity and one writer per particle.
template <class Rec, class ColourFn, class WritersFn, class YarnFn, class LimitFn>
int make_batches(const Rec* recs, uint32_t count, uint32_t n_targets, ColourFn colour, WritersFn writers,
                 YarnFn yarn, LimitFn limited, Batch* out, uint32_t& n_out) {
    n_out = 0;
    std::vector<uint32_t> stamp(n_targets, 0xffffffffu);
    std::vector<uint32_t> seen_colours;
    uint32_t k = 0;
    while (k < count) {
        const uint32_t col = colour(recs[k]);
        if (std::find(seen_colours.begin(), seen_colours.end(), col) != seen_colours.end()) return NUMI_CLOTH_EBATCH;
        seen_colours.push_back(col);
        if (n_out >= NC_MAX_BATCHES) return NUMI_CLOTH_EINVAL;
        Batch b{k, 0, 0, 0};
        bool yarn_open = true;
        while (k < count && colour(recs[k]) == col) {
            uint32_t w[4];
            const int nw = writers(recs[k], w);
            if (nw < 0) return NUMI_CLOTH_EINVAL;
            for (int e = 0; e < nw; ++e) {
                if (w[e] >= n_targets) return NUMI_CLOTH_EINVAL;
                if (stamp[w[e]] == n_out) return NUMI_CLOTH_EBATCH;
                stamp[w[e]] = n_out;
            }
            if (yarn(recs[k])) {
                if (!yarn_open) return NUMI_CLOTH_EINVAL;   // yarn segments lead their colour
                b.yarn = k - b.first + 1u;
            } else {
                yarn_open = false;
            }
            if (limited(recs[k])) b.limited = k - b.first + 1u;
            ++k;
        }
        b.count = k - b.first;
        out[n_out++] = b;
    }
    return NUMI_CLOTH_OK;
}

// Neighbour syncs of the cooperative grid.  CTA r takes, in every colour
// batch, the items whose lowest particle lies in its equal share
// [r n / R, (r + 1) n / R) of the particle range (a list of batch-relative
// indices per colour, staged in its shared memory); its neighbours are the
// CTAs whose items share a particle with its own in any colour (reads
// included: a bend's middle particle).  Built when no CTA has more than
// NC_NBR_MAX neighbours, its lists fit NC_NBR_WORDS words, and the grid
// stays co-resident with them; otherwise every colour ends with the grid
// barrier.  NUMI_CLOTH_NEIGHBOUR_SYNC=0 keeps the grid barrier.
#define NC_NBR_WORDS 4096u
bool prepare_neighbours(numi_cloth* h, const NumiClothScene* scene) {
    DeviceCloth& d = h->d;
    const uint32_t R = h->grid, n = d.n;
    const uint32_t slots = d.n_dist_batches + d.n_knot_batches + d.n_bend_batches;
    uint32_t want = 1;
    env_u32("NUMI_CLOTH_NEIGHBOUR_SYNC", want);
    if (want == 0u || R < 2u || h->cluster != 0u || d.resident != 0u || n == 0u || slots == 0u ||
        slots > 3u * NC_MAX_BATCHES)
        return false;
    auto cta_of = [&](uint32_t p) { return static_cast<uint32_t>(static_cast<uint64_t>(p) * R / n); };
    // lists[r][slot]: CTA r's items of the colour, ascending
    std::vector<std::vector<std::vector<uint32_t>>> lists(R, std::vector<std::vector<uint32_t>>(slots));
    std::vector<std::vector<uint32_t>> touch(n);   // CTAs touching each particle
    auto batch = [&](uint32_t slot, const Batch& bt, auto parts) {
        for (uint32_t k = 0; k < bt.count; ++k) {
            uint32_t p[4];
            const int np = parts(bt.first + k, p);
            uint32_t lowest = p[0];
            for (int e = 1; e < np; ++e) lowest = std::min(lowest, p[e]);
            const uint32_t c = cta_of(lowest);
            lists[c][slot].push_back(k);
            for (int e = 0; e < np; ++e) {
                std::vector<uint32_t>& t = touch[p[e]];
                if (std::find(t.begin(), t.end(), c) == t.end()) t.push_back(c);
            }
        }
    };
    for (uint32_t b = 0; b < d.n_dist_batches; ++b)
        batch(b, d.dist_batches[b], [&](uint32_t i, uint32_t* p) {
            p[0] = scene->distances[i].particlesAndColor.x;
            p[1] = scene->distances[i].particlesAndColor.y;
            return 2;
        });
    for (uint32_t b = 0; b < d.n_knot_batches; ++b)
        batch(d.n_dist_batches + b, d.knot_batches[b], [&](uint32_t i, uint32_t* p) {
            const NumiClothKnot& r = scene->knots[i];
            p[0] = r.particles.x;
            p[1] = r.particles.y;
            p[2] = r.particles.z;
            p[3] = r.particles.w;
            return 4;
        });
    for (uint32_t b = 0; b < d.n_bend_batches; ++b)
        batch(d.n_dist_batches + d.n_knot_batches + b, d.bend_batches[b], [&](uint32_t i, uint32_t* p) {
            p[0] = scene->bends[i].particlesAndColor.x;
            p[1] = scene->bends[i].particlesAndColor.y;
            p[2] = scene->bends[i].particlesAndColor.z;
            return 3;
        });
    std::vector<std::vector<uint32_t>> nbr(R);
    for (const std::vector<uint32_t>& t : touch)
        for (uint32_t c : t)
            for (uint32_t o : t)
                if (o != c && std::find(nbr[c].begin(), nbr[c].end(), o) == nbr[c].end()) {
                    if (nbr[c].size() >= NC_NBR_MAX) return false;
                    nbr[c].push_back(o);
                }
    std::vector<uint32_t> off(R + 1u, 0u), idx, block(R + 1u, 0u), items;
    uint32_t widest = 0;
    for (uint32_t r = 0; r < R; ++r) {
        std::sort(nbr[r].begin(), nbr[r].end());
        idx.insert(idx.end(), nbr[r].begin(), nbr[r].end());
        off[r + 1u] = static_cast<uint32_t>(idx.size());
        // the CTA's block: slot offsets, then the items
        uint32_t at = 0;
        for (uint32_t b = 0; b < slots; ++b) {
            items.push_back(at);
            at += static_cast<uint32_t>(lists[r][b].size());
        }
        items.push_back(at);
        for (uint32_t b = 0; b < slots; ++b) items.insert(items.end(), lists[r][b].begin(), lists[r][b].end());
        block[r + 1u] = static_cast<uint32_t>(items.size());
        widest = std::max(widest, block[r + 1u] - block[r]);
    }
    if (widest > NC_NBR_WORDS) return false;
    const size_t smem = nc_resident_offset() + static_cast<size_t>(widest) * sizeof(uint32_t);
    int per_sm = 0;
    if (raise_frame_smem(smem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, frame_fn(false, h->self_exact), static_cast<int>(h->block), smem) !=
            cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, h->device);
    if (static_cast<uint64_t>(per_sm) * static_cast<uint64_t>(sms) < R) return false;   // must stay co-resident
    uint32_t* d_block = h->buf.alloc<uint32_t>(block.size());
    uint32_t* d_items = h->buf.alloc<uint32_t>(items.size());
    uint32_t* d_off = h->buf.alloc<uint32_t>(off.size());
    uint32_t* d_idx = h->buf.alloc<uint32_t>(std::max<size_t>(idx.size(), 1));
    unsigned int* d_flag = h->buf.alloc<unsigned int>(static_cast<size_t>(NC_NBR_FLAG_STRIDE) * R);
    if (!d_block || !d_items || !d_off || !d_idx || !d_flag) return false;
    if (cudaMemcpy(d_block, block.data(), block.size() * sizeof(uint32_t), cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(d_items, items.data(), items.size() * sizeof(uint32_t), cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(d_off, off.data(), off.size() * sizeof(uint32_t), cudaMemcpyHostToDevice) != cudaSuccess ||
        (!idx.empty() &&
         cudaMemcpy(d_idx, idx.data(), idx.size() * sizeof(uint32_t), cudaMemcpyHostToDevice) != cudaSuccess))
        return false;
    d.colour_slots = slots;
    d.nbr_block = d_block;
    d.nbr_items = d_items;
    d.nbr_off = d_off;
    d.nbr_idx = d_idx;
    d.nbr_flag = d_flag;
    h->nbr_smem = smem;
    return true;
}

// Tile plans of the cooperative grid (cloth_tile.cuh).  CTA t < T owns a
// tile: for a row-major grid cloth a block of a x b particles (the shape
// with the fewest estimated closure particles among those giving at most T
// tiles), else an index strip; the last CTA is the fruit CTA and owns none.
// For each chain of colours the closure of a tile is found backwards: the
// items of the last colour touching an owned particle, then those of the
// colour before touching an owned particle or a particle of an item found,
// and so on.  Local particles are ordered own, then the fruit/yarn and
// strain chains' other particles, then the constraint chain's, so every
// chain reads a prefix.  Returns false (tile mode off) when a plan's
// particles would not fit the shared memory of one CTA per SM or a closure
// holds 65,536 particles or more.
struct TileColour {
    uint32_t family, first, count, batch;
};

struct TilePlan {
    std::vector<uint32_t> words, off, owner;
    bool stream = false;
    size_t smem = 0;
};

bool build_tiles(const TileSource& src, TilePlan& plan) {
    const DeviceCloth& d = src.d;
    const uint32_t n = d.n, grid_width = d.grid_width, R = src.grid, T = R - 1u;
    if (R < 3u || n == 0u) return false;
    // tiles
    std::vector<uint32_t> tile_of(n);
    uint32_t tiles = 0;
    if (grid_width > 0u && n % grid_width == 0u) {
        const uint32_t W = grid_width, H = n / grid_width;
        uint32_t best_a = 0, best_b = 0;
        uint64_t best = ~0ull;
        for (uint32_t a = 1; a <= std::min(H, 512u); ++a)
            for (uint32_t b = 1; b <= std::min(W, 512u); ++b) {
                const uint64_t count = static_cast<uint64_t>((H + a - 1u) / a) * ((W + b - 1u) / b);
                if (count > T) continue;
                const uint64_t cost = static_cast<uint64_t>(a + 12u) * (b + 12u);
                if (cost < best) {
                    best = cost;
                    best_a = a;
                    best_b = b;
                }
            }
        if (best_a == 0u) return false;
        const uint32_t across = (W + best_b - 1u) / best_b;
        for (uint32_t i = 0; i < n; ++i) tile_of[i] = (i / W / best_a) * across + (i % W) / best_b;
        tiles = ((H + best_a - 1u) / best_a) * across;
    } else {
        for (uint32_t i = 0; i < n; ++i) tile_of[i] = static_cast<uint32_t>(static_cast<uint64_t>(i) * T / n);
        tiles = T;
    }
    // chains
    std::vector<std::vector<TileColour>> chains(NC_TILE_CHAINS);
    for (uint32_t b = 0; b < d.n_dist_batches; ++b) {
        const Batch& bt = d.dist_batches[b];
        chains[NC_TILE_CONSTRAINTS].push_back({NC_TILE_DISTANCE, bt.first, bt.count, b});
        if (bt.yarn) chains[NC_TILE_YARN].push_back({NC_TILE_SEGMENT, bt.first, bt.yarn, b});
        if (bt.limited) chains[NC_TILE_STRAIN].push_back({NC_TILE_LIMIT, bt.first, bt.limited, b});
    }
    for (uint32_t b = 0; b < d.n_bend_batches; ++b)
        chains[NC_TILE_CONSTRAINTS].push_back({NC_TILE_BEND, d.bend_batches[b].first, d.bend_batches[b].count, b});
    // the record of every particle in each colour (a colour's records share
    // none)
    constexpr uint32_t kNone = ~0u;
    std::vector<uint32_t> dist_of(static_cast<size_t>(d.n_dist_batches) * n, kNone);
    std::vector<uint32_t> bend_of(static_cast<size_t>(d.n_bend_batches) * n, kNone);
    for (uint32_t b = 0; b < d.n_dist_batches; ++b)
        for (uint32_t k = 0; k < d.dist_batches[b].count; ++k) {
            const uint32_t rec = d.dist_batches[b].first + k;
            const uint2 e = src.distances[rec];
            dist_of[static_cast<size_t>(b) * n + e.x] = dist_of[static_cast<size_t>(b) * n + e.y] = rec;
        }
    for (uint32_t b = 0; b < d.n_bend_batches; ++b)
        for (uint32_t k = 0; k < d.bend_batches[b].count; ++k) {
            const uint32_t rec = d.bend_batches[b].first + k;
            const uint2 e = src.bends[rec];
            bend_of[static_cast<size_t>(b) * n + e.x] = bend_of[static_cast<size_t>(b) * n + e.y] = rec;
        }
    auto ends = [&](uint32_t family, uint32_t rec) {
        return family == NC_TILE_BEND ? src.bends[rec] : src.distances[rec];
    };
    std::vector<uint32_t> owner(n, 0u), local_of(n, 0u);
    std::vector<uint32_t> need_stamp(n, 0u), item_stamp_d(d.d_count, 0u), item_stamp_b(d.b_count, 0u);
    std::vector<int32_t> lidx(n, -1);
    uint32_t stamp = 0;
    std::vector<std::vector<uint32_t>> plans(R);
    size_t widest = 0, widest_stream = 0;   // bytes of a plan and its particles, without and with streamed items
    std::vector<std::vector<uint32_t>> own_of(tiles);
    for (uint32_t i = 0; i < n; ++i) own_of[tile_of[i]].push_back(i);
    for (uint32_t t = 0; t < R; ++t) {
        const std::vector<uint32_t> none;
        const std::vector<uint32_t>& own = t < tiles ? own_of[t] : none;
        // closures: per chain, the items of every colour and the particles
        std::vector<std::vector<std::vector<uint32_t>>> items(NC_TILE_CHAINS);
        std::vector<std::vector<uint32_t>> parts(NC_TILE_CHAINS);
        for (uint32_t k = 0; k < NC_TILE_CHAINS; ++k) {
            const uint32_t g = ++stamp;
            std::vector<uint32_t> cur(own.begin(), own.end());
            for (uint32_t p : cur) need_stamp[p] = g;
            items[k].resize(chains[k].size());
            for (size_t c = chains[k].size(); c-- > 0;) {
                const TileColour& col = chains[k][c];
                const uint32_t cs = ++stamp;
                std::vector<uint32_t>& its = items[k][c];
                const uint32_t* record_of =
                    (col.family == NC_TILE_BEND ? bend_of.data() : dist_of.data()) + static_cast<size_t>(col.batch) * n;
                std::vector<uint32_t>& ist = col.family == NC_TILE_BEND ? item_stamp_b : item_stamp_d;
                const size_t upto = cur.size();
                for (size_t q = 0; q < upto; ++q) {
                    const uint32_t p = cur[q];
                    const uint32_t rec = record_of[p];
                    if (rec >= col.first + col.count || ist[rec] == cs) continue;   // (kNone is past any colour)
                    ist[rec] = cs;
                    its.push_back(rec);
                    const uint2 pe = ends(col.family, rec);
                    for (uint32_t v : {pe.x, pe.y})
                        if (need_stamp[v] != g) {
                            need_stamp[v] = g;
                            cur.push_back(v);
                        }
                }
                std::sort(its.begin(), its.end());
            }
            parts[k] = cur;
        }
        // local order: own, then the yarn and strain chains' others, then
        // the constraint chain's
        std::vector<uint32_t> local(own.begin(), own.end());
        for (uint32_t p : own) lidx[p] = 0;
        auto add = [&](std::initializer_list<uint32_t> ks) {
            std::vector<uint32_t> extra;
            for (uint32_t k : ks)
                for (uint32_t p : parts[k])
                    if (lidx[p] < 0) {
                        lidx[p] = 0;
                        extra.push_back(p);
                    }
            std::sort(extra.begin(), extra.end());
            local.insert(local.end(), extra.begin(), extra.end());
        };
        add({NC_TILE_YARN, NC_TILE_STRAIN});
        const uint32_t small = static_cast<uint32_t>(local.size());
        add({NC_TILE_CONSTRAINTS});
        for (uint32_t l = 0; l < local.size(); ++l) lidx[local[l]] = static_cast<int32_t>(l);
        if (local.size() >= 65536u) return false;
        for (uint32_t l = 0; l < own.size(); ++l) {
            owner[own[l]] = t;
            local_of[own[l]] = l;
        }
        // plan words
        uint32_t colours = 0, nitems = 0;
        for (uint32_t k = 0; k < NC_TILE_CHAINS; ++k) {
            colours += static_cast<uint32_t>(chains[k].size());
            for (const auto& its : items[k]) nitems += static_cast<uint32_t>(its.size());
        }
        std::vector<uint32_t>& w = plans[t];
        const uint32_t table_at = NC_TILE_HEADER;
        const uint32_t list_at = table_at + 2u * colours;
        const uint32_t items_at = (list_at + static_cast<uint32_t>(local.size()) + 3u) & ~3u;
        w.assign(items_at + 4u * nitems, 0u);
        w[0] = static_cast<uint32_t>(local.size());
        w[1] = static_cast<uint32_t>(own.size());
        w[2] = list_at;
        w[3] = items_at;
        w[4u + NC_TILE_CONSTRAINTS] = static_cast<uint32_t>(local.size());
        w[4u + NC_TILE_YARN] = small;
        w[4u + NC_TILE_STRAIN] = small;
        uint32_t tat = table_at, item = 0;
        for (uint32_t k = 0; k < NC_TILE_CHAINS; ++k) {
            w[8u + 2u * k] = tat;
            w[9u + 2u * k] = static_cast<uint32_t>(chains[k].size());
            for (size_t c = 0; c < chains[k].size(); ++c) {
                const TileColour& col = chains[k][c];
                const std::vector<uint32_t>& its = items[k][c];
                w[tat++] = item;
                w[tat++] = static_cast<uint32_t>(its.size()) | (col.family << 28);
                for (uint32_t rec : its) {
                    const uint2 pe = ends(col.family, rec);
                    uint32_t* o = w.data() + items_at + 4u * item++;
                    o[0] = static_cast<uint32_t>(lidx[pe.x]) | (static_cast<uint32_t>(lidx[pe.y]) << 16);
                    o[1] = rec | ((t < tiles && tile_of[pe.x] == t) ? 0x80000000u : 0u);
                }
            }
        }
        for (uint32_t l = 0; l < local.size(); ++l) w[list_at + l] = local[l];
        for (uint32_t p : local) lidx[p] = -1;
        widest = std::max(widest, w.size() * 4u + local.size() * sizeof(float4));
        widest_stream = std::max(widest_stream, items_at * 4u + local.size() * sizeof(float4));
    }
    // the fruit CTA holds its fruit state and the staged friction sweep.
    // Plans that do not fit keep their items in global memory: the
    // 512 x 512 cloth's are 25,000 items a CTA, 59 MB in all, which the L2
    // holds (a substep 158 us colour by colour, 101 with streamed items).
    const size_t fruit = nc_resident_offset() + sizeof(FrictionStage);
    const bool stream = std::max(fruit, nc_fruit_offset() + widest) > src.smem_budget;
    const size_t smem = std::max(fruit, nc_fruit_offset() + (stream ? widest_stream : widest));
    if (smem > src.smem_budget) return false;
    plan.off.assign(R + 1u, 0u);
    for (uint32_t t = 0; t < R; ++t) {
        plan.words.insert(plan.words.end(), plans[t].begin(), plans[t].end());
        plan.off[t + 1u] = static_cast<uint32_t>(plan.words.size());
    }
    plan.owner.resize(n);
    for (uint32_t i = 0; i < n; ++i) plan.owner[i] = (owner[i] << 16) | local_of[i];
    plan.stream = stream;
    plan.smem = smem;
    return true;
}

// While one lives, the calls of this thread are none that another stream's
// capture forbids.
struct RelaxedCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

// A plan of `src` on the current device, on a stream of its own: no other
// stream is waited for.  False where it does not fit.
bool make_tiles(const TileSource& src, TileBlock& out) {
    TilePlan plan;
    if (!build_tiles(src, plan)) return false;
    RelaxedCapture relaxed;
    TileBlock block;
    auto pieces = [&](Carver& c) {
        block.words = c.get<uint32_t>(plan.words.size());
        block.off = c.get<uint32_t>(plan.off.size());
        block.owner = c.get<uint32_t>(plan.owner.size());
        block.x_alt = c.get<float4>(src.d.n);
        block.v_alt = c.get<float4>(src.d.n);
    };
    Carver measure{nullptr};
    pieces(measure);
    cudaStream_t stream = nullptr;
    cudaError_t e = device_malloc(&block.mem, measure.used);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking);
    Carver carver{static_cast<char*>(block.mem)};
    pieces(carver);
    auto up = [&](uint32_t* dst, const std::vector<uint32_t>& v) {
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(dst, v.data(), v.size() * sizeof(uint32_t), cudaMemcpyHostToDevice, stream);
    };
    up(block.words, plan.words);
    up(block.off, plan.off);
    up(block.owner, plan.owner);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    if (stream != nullptr) cudaStreamDestroy(stream);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    block.stream = plan.stream;
    block.smem = plan.smem;
    out = std::move(block);
    return true;
}

// The materials of a plan's items from the records (a plan is built without
// them, and written again where they change).  A CTA per CTA of the plan.
__global__ void numi_cloth_tile_materials_kernel(DeviceCloth d) {
    uint32_t* plan = const_cast<uint32_t*>(d.tile_words) + d.tile_off[blockIdx.x];
    for (uint32_t chain = 0; chain < NC_TILE_CHAINS; ++chain) {
        const uint32_t* table = plan + plan[8u + 2u * chain];
        for (uint32_t c = 0; c < plan[9u + 2u * chain]; ++c) {
            uint4* items = reinterpret_cast<uint4*>(plan + plan[3]) + table[2u * c];
            const uint32_t count = table[2u * c + 1u] & 0x0fffffffu, family = table[2u * c + 1u] >> 28;
            if (family == NC_TILE_SEGMENT) continue;
            for (uint32_t k = threadIdx.x; k < count; k += blockDim.x) {
                const uint32_t rec = items[k].y & 0x7fffffffu;
                float2 m;
                if (family == NC_TILE_BEND) {
                    m = d.b_mat[rec];
                } else {
                    const float4 v = d.d_mat[rec];
                    m = make_float2(v.x, family == NC_TILE_DISTANCE ? v.y : v.w);
                }
                items[k].z = __float_as_uint(m.x);
                items[k].w = __float_as_uint(m.y);
            }
        }
    }
}

cudaError_t tile_materials(numi_cloth* h) {
    numi_cloth_tile_materials_kernel<<<h->tile_grid, 256, 0, h->stream>>>(h->d);
    return cudaGetLastError();
}

// Tile mode with this plan from the next launch on, where the device holds
// the tile launch.  The plan it replaces is no longer in use.
void adopt_tiles(numi_cloth* h, TileBlock&& block) {
    h->plan = std::move(block);
    DeviceCloth& d = h->d;
    d.tile_words = h->plan.words;
    d.tile_off = h->plan.off;
    d.tile_owner = h->plan.owner;
    d.tile_stream = h->plan.stream ? 1u : 0u;
    d.x_alt = h->plan.x_alt;
    d.v_alt = h->plan.v_alt;
    h->tile_smem = h->plan.smem;
    h->tiles = h->plan.mem != nullptr && tiles_fit(h) && tile_materials(h) == cudaSuccess;
    cudaGetLastError();
}

// Source of a handle's plans, without the ends of its records.
TileSource tile_source(const numi_cloth* h) {
    int max_optin = 0;
    cudaDeviceGetAttribute(&max_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, h->device);
    TileSource src;
    src.d = h->d;
    src.grid = h->tile_grid;
    src.smem_budget = static_cast<size_t>(max_optin) - tile_static_smem(h);
    return src;
}

// One thread of the process that builds small cloths' plans beside the
// threads that step them: started with the first build, ended with the
// process.  A build is a few milliseconds of host work at most.
class TileBuilder {
  public:
    static TileBuilder& get() {
        static TileBuilder builder;
        return builder;
    }
    void submit(const std::shared_ptr<TileJob>& job) {
        std::lock_guard<std::mutex> lock(mutex_);
        queue_.push_back(job);
        if (!thread_.joinable()) {
            try {
                thread_ = std::thread([this] { run(); });
            } catch (const std::system_error&) {   // no thread: finish() builds
            }
        }
        wake_.notify_all();
    }
    // The job done: by the thread, or here where it had not begun.
    void finish(const std::shared_ptr<TileJob>& job) {
        std::unique_lock<std::mutex> lock(mutex_);
        if (take(job)) {
            lock.unlock();
            build(*job);
            lock.lock();
            job->state = TileJob::kDone;
        }
        wake_.wait(lock, [&] { return job->state == TileJob::kDone; });
    }
    // The job not done, or over.
    void abandon(const std::shared_ptr<TileJob>& job) {
        std::unique_lock<std::mutex> lock(mutex_);
        if (take(job)) return;
        wake_.wait(lock, [&] { return job->state != TileJob::kRunning; });
    }

  private:
    ~TileBuilder() {
        {
            std::lock_guard<std::mutex> lock(mutex_);
            stop_ = true;
        }
        wake_.notify_all();
        if (thread_.joinable()) thread_.join();
    }
    bool take(const std::shared_ptr<TileJob>& job) {
        const auto at = std::find(queue_.begin(), queue_.end(), job);
        if (at == queue_.end()) return false;
        queue_.erase(at);
        return true;
    }
    static void build(TileJob& job) {
        cudaSetDevice(job.device);
        try {
            make_tiles(job.source, job.block);
        } catch (const std::bad_alloc&) {   // no plan: the cloth stays on its cluster
        }
    }
    void run() {
        RelaxedCapture relaxed;   // also where the thread is the last to drop a job
        std::unique_lock<std::mutex> lock(mutex_);
        for (;;) {
            wake_.wait(lock, [&] { return stop_ || !queue_.empty(); });
            if (stop_) return;
            const std::shared_ptr<TileJob> job = queue_.front();
            queue_.pop_front();
            job->state = TileJob::kRunning;
            lock.unlock();
            build(*job);
            lock.lock();
            job->state = TileJob::kDone;
            wake_.notify_all();
        }
    }
    std::mutex mutex_;
    std::condition_variable wake_;
    std::deque<std::shared_ptr<TileJob>> queue_;
    std::thread thread_;
    bool stop_ = false;
};

// A launch runs in tile mode when the cloth has tile plans and the
// schedule is one the tile substep covers.
bool tile_covers(const Schedule& s) {
    return s.iterations == 1u && s.aerodynamics == 0u && s.swept_fruit_yarn == 0u &&
           s.primitive_self == 0u && s.reconcile_passes == 0u && s.final_passes == 0u && s.certificate_passes == 0u;
}
bool tile_schedule(const numi_cloth* h, const Schedule& s) { return h->tiles && tile_covers(s); }

// A small cloth's plan is built from its kTileBuildSubsteps'th covered
// substep on, beside the stepping thread, and taken up at its
// kTilePlanSubsteps'th: a build takes 0.4 (24 x 24) to 3 ms (61 x 61) of
// another core, and the substeps between are 5 to 7 ms of the GPU's time, so
// the launch that takes it up finds it done unless launches are issued far
// ahead of the GPU.  A cloth that only joins batches never needs one.
constexpr uint32_t kTileBuildSubsteps = 32, kTilePlanSubsteps = 128;
void prepare_small_tiles(numi_cloth* h, uint32_t substeps) {
    h->tile_substeps += std::min(substeps, kTilePlanSubsteps - std::min(h->tile_substeps, kTilePlanSubsteps));
    if (h->tile_source != nullptr) {
        if (h->tile_substeps < kTileBuildSubsteps) return;
        h->tile_job = std::make_shared<TileJob>();
        h->tile_job->source = std::move(*h->tile_source);
        h->tile_job->device = h->device;
        h->tile_source.reset();
        TileBuilder::get().submit(h->tile_job);
        return;   // for a later launch
    }
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    if (h->tile_substeps < kTilePlanSubsteps || cudaStreamIsCapturing(h->stream, &capturing) != cudaSuccess ||
        capturing != cudaStreamCaptureStatusNone)
        return;
    TileBuilder::get().finish(h->tile_job);
    adopt_tiles(h, std::move(h->tile_job->block));
    h->tile_job.reset();
}

// Adjoint tape of a launch: [substep][slots][n] positions, [substep][n]
// velocities, [substep][grips] grips.
struct Tape {
    float4* x = nullptr;      // null: the launch is not taped
    float4* v = nullptr;
    NumiClothGrip* grip = nullptr;
    uint32_t slots = 0;
    uint32_t first = 0;       // substep of the tape the launch starts at
    uint32_t* touched = nullptr;   // set where a fruit touched the cloth
};

cudaError_t launch(numi_cloth* h, uint32_t substeps, const Schedule& s, uint32_t cfg_offset = 0,
                   const Tape& tape = {}) {
    if ((h->tile_source != nullptr || h->tile_job != nullptr) && tile_covers(s)) {
        try {
            prepare_small_tiles(h, substeps);
        } catch (const std::bad_alloc&) {   // it stays on its cluster
            h->tile_source.reset();
            if (h->tile_job) TileBuilder::get().abandon(h->tile_job);
            h->tile_job.reset();
        }
    }
    DeviceCloth d = h->d;
    d.cfg = h->d_cfg + cfg_offset;
    d.epoch_base = h->epoch;
    const bool taped = tape.x != nullptr;
    const bool rollout = taped || tape.touched != nullptr;
    d.yarn_touched = tape.touched;
    if (taped) {
        d.tape = tape.x;
        d.tape_v = tape.v;
        d.tape_grip = tape.grip;
        d.tape_slots = tape.slots;
        d.trace = nullptr;
    }
    Schedule sc = s;
    sc.substeps = substeps;
    sc.tape_first = tape.first;
    void* args[] = {&d, &sc};
    const bool edge = sc.primitive_self != 0u && d.edge_count != nullptr;
    const void* fn = rollout ? frame_tape_fn() : frame_fn(edge, h->self_exact);
    if (d.trace != nullptr && substeps > h->trace_capacity) d.trace = nullptr;
    if (d.trace == nullptr) d.trace_cta = nullptr;
    cudaError_t e = cudaMemsetAsync(h->d.bar_count, 0, kBarrierWords * sizeof(unsigned long long), h->stream);
    if (e != cudaSuccess) return e;
    h->last_substeps = substeps;
    size_t smem = h->smem;
    uint32_t grid = h->grid;
    const bool tiled = tile_schedule(h, sc);
    if (edge) {
        // the edge/edge phases' box tree after the launch's own shared memory,
        // where the device has room and the cloth is of a size that has one
        int max_optin = 0;
        cudaDeviceGetAttribute(&max_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, h->device);
        cudaFuncAttributes fe{};
        cudaFuncGetAttributes(&fe, frame_fn(true, h->self_exact));
        const size_t at = nc_round256(smem);
        const size_t bytes = at + edge_tree_bytes(d.y_count, true);
        if (d.y_count <= NC_EDGE_TREE_MAX && bytes + fe.sharedSizeBytes <= static_cast<size_t>(max_optin) &&
            raise_smem(frame_fn(true, h->self_exact), bytes) == cudaSuccess) {
            sc.tree_keys = static_cast<uint32_t>(at);
            sc.tree_lists = 1u;
            smem = bytes;
        }
        // the tree can cost a cooperative grid its second CTA on an SM: as
        // many as are co-resident (the bits are those of any grid)
        int k = 0, sms = 0;
        if (h->cluster == 0u && grid > 1u &&
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&k, fn, static_cast<int>(h->block), smem) == cudaSuccess &&
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, h->device) == cudaSuccess && k > 0)
            grid = std::min(grid, static_cast<uint32_t>(k * sms));
        cudaGetLastError();
    }
    if (h->cluster > 0 && !tiled) {
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(h->cluster);
        cfg.blockDim = dim3(h->block);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = h->stream;
        cudaLaunchAttribute attr{};
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = h->cluster;
        attr.val.clusterDim.y = 1;
        attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        d.cluster_barrier = 1u;
        e = cudaLaunchKernelExC(&cfg, fn, args);
    } else if (h->grid == 1 && !tiled) {
        e = cudaLaunchKernel(fn, dim3(1), dim3(h->block), args, smem, h->stream);
    } else if (tiled) {
        sc.tiles = 1u;
        d.resident = 0u;   // a small cloth's other launches keep it in a cluster's shared memory
        if (h->tile_grid > h->trace_ctas) d.trace_cta = nullptr;
        e = raise_frame_smem(h->tile_smem);
        if (e == cudaSuccess)
            e = cudaLaunchCooperativeKernel(fn, dim3(h->tile_grid), dim3(h->tile_block), args, h->tile_smem, h->stream);
        h->last_grid = h->tile_grid;
        h->last_block = h->tile_block;
        h->last_tiles = true;
        if (e == cudaSuccess) ++h->launches;
        return e;
    } else {
        // neighbour syncs between colours (the kernel without the edge/edge
        // phases; its flags start at zero in every launch)
        if (h->neighbours && !edge && !rollout) {
            d.nbr_on = 1u;
            e = cudaMemsetAsync(d.nbr_flag, 0, NC_NBR_FLAG_STRIDE * h->grid * sizeof(unsigned int), h->stream);
            if (e != cudaSuccess) return e;
        }
        e = cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(h->block), args, d.nbr_on ? h->nbr_smem : smem, h->stream);
    }
    h->last_grid = h->cluster > 0 ? h->cluster : grid;
    h->last_block = h->block;
    h->last_tiles = false;
    if (e == cudaSuccess) ++h->launches;
    return e;
}

Schedule device_schedule(const NumiClothSchedule& schedule) {
    Schedule s{};
    s.iterations = schedule.iterations;
    s.strain_sweeps = schedule.strainSweeps;
    s.reconcile_passes = schedule.reconcilePasses;
    s.final_passes = schedule.finalPasses;
    s.certificate_passes = schedule.certificatePasses;
    s.early_exit = schedule.earlyExit;
    s.self_collision = schedule.selfCollision;
    s.aerodynamics = schedule.aerodynamics;
    s.swept_ground = schedule.sweptGround;
    s.swept_fruit_yarn = schedule.sweptFruitYarn;
    s.frictions = schedule.frictions;
    s.release = schedule.release;
    s.damping = schedule.damping;
    s.primitive_self = schedule.primitiveSelf;
    return s;
}

// Point self-contact grid of a cloth, allocated on first use (about four
// buckets per particle, of which a cloth in an axis plane uses half); the bucket heads are cleared when the 26-bit
// substep part of their tags wraps within the next `substeps`.
int prepare_self_grid(numi_cloth* h, bool self_collision, uint32_t substeps, cudaStream_t stream) {
    if (self_collision && h->d.hash_head == nullptr) {
        uint32_t buckets = 1024u;
        while (buckets < 4u * h->d.n) buckets <<= 1;
        DeviceCloth& d = h->d;
        d.hash_head = h->buf.alloc<unsigned long long>(buckets, stream);
        d.hash_over_head = h->buf.alloc<unsigned long long>(1, stream);
        d.hash_over = h->buf.alloc<HashSlot>(h->d.n, stream);
        d.hash = h->buf.alloc<HashSlot>(static_cast<size_t>(buckets) * NC_HASH_CAP, stream);
        d.self_stats = h->buf.alloc<unsigned long long>(8, stream);
        // the ordered pass's list: room for three pairs per particle (a
        // power of two, at least 4,096); scratch of three words per listed
        // pair (sort keys, or the wavefront form's keys, predecessors and
        // waves) plus one turn's partners
        uint32_t list_cap = 4096u;
        while (list_cap < 3u * h->d.n) list_cap <<= 1;
        bool order_ok = true;
        if (h->self_exact) {
            d.self_list = h->buf.alloc<float4>(2u * static_cast<size_t>(list_cap), stream);
            d.self_list_head = h->buf.alloc<unsigned long long>(1, stream);
            d.self_pass_stats = h->buf.alloc<unsigned long long>(2, stream);
            d.self_keys = h->buf.alloc<unsigned long long>(3u * static_cast<size_t>(list_cap) + NC_SELF_GROUP, stream);
            d.self_mark = h->buf.alloc<unsigned long long>(h->d.n, stream);
            d.self_x0 = h->buf.alloc<float4>(h->d.n, stream);
            d.self_disp = h->buf.alloc<float>(h->d.n, stream);
            order_ok = d.self_list != nullptr && d.self_list_head != nullptr && d.self_pass_stats != nullptr &&
                       d.self_keys != nullptr && d.self_mark != nullptr && d.self_x0 != nullptr &&
                       d.self_disp != nullptr;
        }
        if (d.hash_head == nullptr || d.hash == nullptr || d.self_stats == nullptr || d.hash_over_head == nullptr ||
            d.hash_over == nullptr || !order_ok) {
            d.hash_head = nullptr;
            return NUMI_CLOTH_ENOMEM;
        }
        d.self_list_cap = list_cap;
        d.self_key_cap = list_cap;
        d.hash_mask = buckets - 1u;
    }
    if (h->d.hash_head != nullptr && ((h->epoch + substeps) >> 26) != (h->epoch >> 26)) {
        if (cudaMemsetAsync(h->d.hash_head, 0, (static_cast<size_t>(h->d.hash_mask) + 1u) * sizeof(unsigned long long),
                            stream) != cudaSuccess ||
            cudaMemsetAsync(h->d.hash_over_head, 0, sizeof(unsigned long long), stream) != cudaSuccess ||
            (h->self_exact &&
             (cudaMemsetAsync(h->d.self_list_head, 0, sizeof(unsigned long long), stream) != cudaSuccess ||
              cudaMemsetAsync(h->d.self_mark, 0, static_cast<size_t>(h->d.n) * sizeof(unsigned long long),
                              stream) != cudaSuccess)))
            return NUMI_CLOTH_ECUDA;
    }
    return NUMI_CLOTH_OK;
}

// Edge/edge buffers of a cloth, allocated on first use: a build grid of
// about four buckets per yarn segment with room for 27 cells per segment, 32
// listed pairs and 16 candidate pairs per segment.  The build cell is a
// median yarn segment plus the yarn diameter and skin (three diameters), so
// that a typical segment's grown box spans at most two cells a side.
// Every yarn segment's local segments of higher index, ascending: the pairs
// the edge/edge family skips (edgePairLocal, tools/cloth_bag.cpp:2740-2749:
// some endpoint of one is local to some endpoint of the other, by the 2-hop
// topology list or, on a row-major grid cloth, the 5 x 5 block).
bool build_local_lists(const numi_cloth* h, std::vector<uint32_t>& off, std::vector<uint32_t>& idx) {
    const DeviceCloth& d = h->d;
    const std::vector<uint2>& y = h->host_yarn;
    const bool csr = !h->host_local_off.empty();
    auto local = [&](uint32_t a, uint32_t b) {
        if (csr) {
            const uint32_t* lo = h->host_local_idx.data() + h->host_local_off[a];
            const uint32_t* hi = h->host_local_idx.data() + h->host_local_off[a + 1u];
            return std::binary_search(lo, hi, b);
        }
        if (d.grid_width == 0u) return a == b;
        const int ra = static_cast<int>(a / d.grid_width), ca = static_cast<int>(a % d.grid_width);
        const int rb = static_cast<int>(b / d.grid_width), cb = static_cast<int>(b % d.grid_width);
        return std::abs(ra - rb) <= 2 && std::abs(ca - cb) <= 2;
    };
    // segments at each particle
    std::vector<uint32_t> at_off(d.n + 1u, 0u), at(2u * y.size());
    for (const uint2& s : y) {
        ++at_off[s.x + 1u];
        ++at_off[s.y + 1u];
    }
    for (uint32_t p = 0; p < d.n; ++p) at_off[p + 1u] += at_off[p];
    std::vector<uint32_t> fill(at_off.begin(), at_off.end() - 1);
    for (uint32_t k = 0; k < y.size(); ++k) {
        at[fill[y[k].x]++] = k;
        at[fill[y[k].y]++] = k;
    }
    // the particles an endpoint can be local to
    std::vector<uint32_t> near;
    auto gather = [&](uint32_t a) {
        near.push_back(a);
        if (csr) {
            near.insert(near.end(), h->host_local_idx.begin() + h->host_local_off[a],
                        h->host_local_idx.begin() + h->host_local_off[a + 1u]);
        } else if (d.grid_width != 0u) {
            const int w = static_cast<int>(d.grid_width), rows = static_cast<int>((d.n + d.grid_width - 1u) / d.grid_width);
            const int ra = static_cast<int>(a / d.grid_width), ca = static_cast<int>(a % d.grid_width);
            for (int r = std::max(ra - 2, 0); r <= std::min(ra + 2, rows - 1); ++r)
                for (int c = std::max(ca - 2, 0); c <= std::min(ca + 2, w - 1); ++c) {
                    const uint32_t q = static_cast<uint32_t>(r * w + c);
                    if (q < d.n) near.push_back(q);
                }
        }
    };
    off.assign(y.size() + 1u, 0u);
    idx.clear();
    std::vector<uint32_t> cand;
    for (uint32_t i = 0; i < y.size(); ++i) {
        near.clear();
        gather(y[i].x);
        gather(y[i].y);
        cand.clear();
        for (uint32_t q : near)
            for (uint32_t k = at_off[q]; k < at_off[q + 1u]; ++k)
                if (at[k] > i) cand.push_back(at[k]);
        std::sort(cand.begin(), cand.end());
        cand.erase(std::unique(cand.begin(), cand.end()), cand.end());
        for (uint32_t j : cand)
            if (local(y[i].x, y[j].x) || local(y[i].x, y[j].y) || local(y[i].y, y[j].x) || local(y[i].y, y[j].y))
                idx.push_back(j);
        off[i + 1u] = static_cast<uint32_t>(idx.size());
    }
    return true;
}

int prepare_edge_grid(numi_cloth* h, bool primitive, uint32_t substeps, float radius, cudaStream_t stream) {
    (void)substeps;
    DeviceCloth& d = h->d;
    if (primitive && d.edge_count == nullptr && d.y_count > 0u) {
        uint32_t buckets = 1024u;
        while (buckets < 4u * d.y_count) buckets <<= 1;
        const uint32_t cap = std::max(1024u, 16u * d.y_count);
        const uint32_t list_cap = std::max(2048u, 32u * d.y_count);
        const uint32_t ctas = std::max<uint32_t>(h->grid, 1u);
        DeviceCloth e = d;
        e.edge_count = h->buf.alloc<uint32_t>(buckets, stream);
        e.edge_offs = h->buf.alloc<uint32_t>(buckets, stream);
        e.edge_chunk_total = h->buf.alloc<uint32_t>(ctas, stream);
        e.edge_entries = h->buf.alloc<float4>(static_cast<size_t>(54u) * d.y_count, stream);
        e.edge_giant = h->buf.alloc<uint32_t>(d.y_count, stream);
        e.edge_bbox = h->buf.alloc<float4>(2u * d.y_count, stream);
        std::vector<uint32_t> loc_off, loc_idx;
        build_local_lists(h, loc_off, loc_idx);
        uint32_t* d_loc_off = h->buf.alloc<uint32_t>(loc_off.size());
        uint32_t* d_loc_idx = h->buf.alloc<uint32_t>(std::max<size_t>(loc_idx.size(), 1));
        if (d_loc_off != nullptr && d_loc_idx != nullptr &&
            (cudaMemcpy(d_loc_off, loc_off.data(), loc_off.size() * sizeof(uint32_t), cudaMemcpyHostToDevice) !=
                 cudaSuccess ||
             (!loc_idx.empty() && cudaMemcpy(d_loc_idx, loc_idx.data(), loc_idx.size() * sizeof(uint32_t),
                                             cudaMemcpyHostToDevice) != cudaSuccess)))
            d_loc_off = nullptr;
        e.edge_loc_off = d_loc_off;
        e.edge_loc_idx = d_loc_idx;
        e.edge_pairs = h->buf.alloc<uint2>(list_cap, stream);
        e.edge_xb = h->buf.alloc<float4>(d.n, stream);
        e.edge_pb = h->buf.alloc<float4>(d.n, stream);
        e.edge_built_radius = h->buf.alloc<float>(1, stream);
        e.edge_sph = h->buf.alloc<float4>(d.y_count, stream);
        e.edge_x0 = h->buf.alloc<float4>(d.n, stream);
        e.edge_path = h->buf.alloc<float>(d.n, stream);
        e.edge_cand = h->buf.alloc<uint4>(cap, stream);
        e.edge_order = h->buf.alloc<unsigned long long>(cap, stream);
        e.edge_sorted = h->buf.alloc<unsigned long long>(cap, stream);
        e.edge_new = h->buf.alloc<EdgeRecord>(cap, stream);
        e.edge_done = h->buf.alloc<uint32_t>(cap, stream);
        e.edge_lv = h->buf.alloc<uint32_t>(cap, stream);
        e.edge_level = h->buf.alloc<uint32_t>(d.n, stream);
        e.edge_qbox_raw = h->buf.alloc<float>(6u * d.y_count, stream);
        e.edge_tree = h->buf.alloc<uint32_t>(static_cast<size_t>(NC_EDGE_TREE_WORDS) * d.y_count + NC_EDGE_TREE_HEAD, stream);
        e.edge_centre = h->buf.alloc<float4>(2u * static_cast<size_t>(d.y_count), stream);   // centres, last build's
        e.edge_rec = h->buf.alloc<EdgeRecord>(cap, stream);
        e.edge_ctl = h->buf.alloc<uint32_t>(8, stream);
        e.edge_stats = h->buf.alloc<unsigned long long>(2, stream);
        e.edge_red = h->buf.alloc<double>(3u * ctas, stream);
        if (!e.edge_count || !e.edge_offs || !e.edge_chunk_total || !e.edge_entries || !e.edge_giant ||
            !e.edge_pairs || !e.edge_xb || !e.edge_pb || !e.edge_built_radius || !e.edge_sph || !e.edge_x0 ||
            !e.edge_path || !e.edge_cand || !e.edge_order || !e.edge_sorted || !e.edge_new || !e.edge_done || !e.edge_rec ||
            !e.edge_ctl || !e.edge_stats || !e.edge_red || !e.edge_lv || !e.edge_level || !e.edge_qbox_raw || !e.edge_bbox ||
            !e.edge_tree || !e.edge_centre ||
            !e.edge_loc_off || !e.edge_loc_idx)
            return NUMI_CLOTH_ENOMEM;
        e.edge_mask = buckets - 1u;
        e.edge_cap = cap;
        e.edge_list_cap = list_cap;
        d = e;
    }
    if (d.edge_count != nullptr) {
        d.edge_cell = h->yarn_rest_median + 3.0f * (2.0f * radius);
        if (const char* v = std::getenv("NUMI_CLOTH_EDGE_CELL")) {
            const float cell = std::strtof(v, nullptr);   // test hook: force long segments or crowded cells
            if (cell > 0.0f) d.edge_cell = cell;
        }
    }
    return NUMI_CLOTH_OK;
}

}  // namespace

extern "C" {

const char* numi_cloth_version(void) { return "numi-cloth-b200 0.1 (sm_100a, ABI 13)"; }

int numi_cloth_create(const NumiClothScene* scene, numi_cloth_t** out) {
    if (scene == nullptr || out == nullptr || scene->config == nullptr || scene->particles == nullptr)
        return NUMI_CLOTH_EINVAL;
    *out = nullptr;
    const NumiClothConfig& cfg = *scene->config;
    if (cfg.control.x != NUMI_CLOTH_ABI_VERSION) return NUMI_CLOTH_EINVAL;
    const uint32_t n = cfg.control.y, D = cfg.control.z, G = cfg.control.w;
    const uint32_t K = cfg.constraintCounts.x, B = cfg.constraintCounts.y, F = cfg.constraintCounts.w;
    const uint32_t P = cfg.contactCounts.x;
    if (n == 0 || F > NC_MAX_FRUITS || G > NC_MAX_GRIPS || P > NC_MAX_PAIRS) return NUMI_CLOTH_EINVAL;
    if ((D && !scene->distances) || (K && !scene->knots) || (B && !scene->bends) || (G && !scene->grips) ||
        (F && !scene->fruits) || (P && !scene->fruitPairs))
        return NUMI_CLOTH_EINVAL;
    if (validate_config(cfg, cfg) != 0u) return NUMI_CLOTH_EINVAL;
    if (cfg.gripControl.y == 1u && scene->cuffParticles == nullptr) return NUMI_CLOTH_EINVAL;

    numi_cloth* h = new (std::nothrow) numi_cloth();
    if (h == nullptr) return NUMI_CLOTH_ENOMEM;
    cudaGetDevice(&h->device);
    h->base = cfg;

    // Batches.
    int rc = make_batches(
        scene->distances, D, n, [](const NumiClothDistance& r) { return r.particlesAndColor.z; },
        [](const NumiClothDistance& r, uint32_t* w) {
            w[0] = r.particlesAndColor.x;
            w[1] = r.particlesAndColor.y;
            return w[0] == w[1] ? -1 : 2;
        },
        [](const NumiClothDistance& r) { return r.particlesAndColor.w != 3u; },
        [](const NumiClothDistance& r) { return r.material.w > 0.0f; }, h->d.dist_batches, h->d.n_dist_batches);
    if (rc == NUMI_CLOTH_OK)
        rc = make_batches(
            scene->knots, K, n, [](const NumiClothKnot& r) { return r.control.x; },
            [](const NumiClothKnot& r, uint32_t* w) {
                w[0] = r.particles.x;
                w[1] = r.particles.y;
                w[2] = r.particles.z;
                w[3] = r.particles.w;
                return 4;
            },
            [](const NumiClothKnot&) { return false; }, [](const NumiClothKnot&) { return false; },
            h->d.knot_batches, h->d.n_knot_batches);
    if (rc == NUMI_CLOTH_OK)
        rc = make_batches(
            scene->bends, B, n, [](const NumiClothBend& r) { return r.particlesAndColor.w; },
            [](const NumiClothBend& r, uint32_t* w) {
                w[0] = r.particlesAndColor.x;
                w[1] = r.particlesAndColor.z;
                return w[0] == w[1] ? -1 : 2;
            },
            [](const NumiClothBend&) { return false; }, [](const NumiClothBend&) { return false; },
            h->d.bend_batches, h->d.n_bend_batches);
    if (rc == NUMI_CLOTH_OK)
        rc = make_batches(
            scene->fruitPairs, P, F, [](const NumiClothFruitPair& r) { return r.fruitsAndColor.z; },
            [](const NumiClothFruitPair& r, uint32_t* w) {
                w[0] = r.fruitsAndColor.x;
                w[1] = r.fruitsAndColor.y;
                return w[0] == w[1] ? -1 : 2;
            },
            [](const NumiClothFruitPair&) { return false; }, [](const NumiClothFruitPair&) { return false; },
            h->d.pair_batches, h->d.n_pair_batches);
    // the middle particle of a bend is read-only but must still exist
    for (uint32_t k = 0; rc == NUMI_CLOTH_OK && k < B; ++k)
        if (scene->bends[k].particlesAndColor.y >= n) rc = NUMI_CLOTH_EINVAL;
    for (uint32_t g = 0; rc == NUMI_CLOTH_OK && g < G; ++g) {
        if (scene->grips[g].particle.x >= n) rc = NUMI_CLOTH_EINVAL;
        for (uint32_t e = 0; e < g && rc == NUMI_CLOTH_OK; ++e)
            if (scene->grips[e].particle.x == scene->grips[g].particle.x) rc = NUMI_CLOTH_EBATCH;
    }
    if (rc == NUMI_CLOTH_OK && cfg.gripControl.y == 1u)
        for (uint32_t k = 0; k < 2u * cfg.gripControl.z; ++k)
            if (scene->cuffParticles[k] >= n) rc = NUMI_CLOTH_EINVAL;
    if (rc != NUMI_CLOTH_OK) {
        delete h;
        return rc;
    }

    // Device buffers.
    DeviceCloth& d = h->d;
    d.n = n;
    d.d_count = D;
    d.k_count = K;
    d.b_count = B;
    d.g_count = G;
    d.f_count = F;
    d.p_count = P;
    d.grid_width = scene->gridWidth;
    d.damping = -1.0f;
    d.x = h->buf.alloc<float4>(n);
    d.xp = h->buf.alloc<float4>(n);
    d.v = h->buf.alloc<float4>(n);
    float4* rest = h->buf.alloc<float4>(n);
    d.rest = rest;
    uint2* d_ij = h->buf.alloc<uint2>(D);
    float4* d_mat = h->buf.alloc<float4>(D);
    d.d_ij = d_ij;
    d.d_mat = d_mat;
    d.d_lambda = h->buf.alloc<float>(D);
    uint4* k_ij = h->buf.alloc<uint4>(K);
    float2* k_mat = h->buf.alloc<float2>(K);
    d.k_ij = k_ij;
    d.k_mat = k_mat;
    d.k_lambda = h->buf.alloc<float>(K);
    uint4* b_ij = h->buf.alloc<uint4>(B);
    float2* b_mat = h->buf.alloc<float2>(B);
    d.b_ij = b_ij;
    d.b_mat = b_mat;
    d.b_lambda = h->buf.alloc<float>(B);
    d.grips = h->buf.alloc<NumiClothGrip>(G);
    d.fruits = h->buf.alloc<NumiClothFruit>(F);
    d.pairs = h->buf.alloc<NumiClothFruitPair>(P);
    uint32_t* cuff = h->buf.alloc<uint32_t>(cfg.gripControl.y == 1u ? 2u * cfg.gripControl.z : 1u);
    d.cuff = cuff;
    const uint32_t rim_count = scene->mouthRim != nullptr ? cfg.mouthControl.x : 0u;
    uint32_t* rim = h->buf.alloc<uint32_t>(rim_count);
    d.rim = rim_count >= 3u ? rim : nullptr;
    d.release = h->buf.alloc<uint32_t>(2);
    d.yarn_slot_a = h->buf.alloc<float4>(static_cast<size_t>(F ? D : 1) * NC_YARN_SLOTS);
    d.yarn_slot_b = h->buf.alloc<float4>(static_cast<size_t>(F ? D : 1) * NC_YARN_SLOTS);
    d.yarn_live = h->buf.alloc<uint32_t>(F ? D : 1);
    d.yarn_list = h->buf.alloc<uint32_t>(F ? D : 1);
    d.yarn_list_n = h->buf.alloc<uint32_t>(1);
    d.force = h->buf.alloc<float4>(n);
    d.fruit_partial = h->buf.alloc<float4>(NC_MAX_FRUITS * 9u / 2u + 1u);
    d.failure = h->buf.alloc<unsigned int>(1);
    // barrier counter (u64) and abort flag share one 16-byte block so one
    // memset resets both before a launch
    d.bar_count = h->buf.alloc<unsigned long long>(kBarrierWords);
    d.abort_flag = reinterpret_cast<unsigned int*>(d.bar_count + 1);
    d.bar_flag = d.bar_count + 16;     // 128 bytes away from the arrival counter
    d.fruit_flag = d.bar_count + 32;   // and 128 more
    d.stats = h->buf.alloc<uint32_t>(4);

    // Point self contact in the reference's Gauss-Seidel order
    // (NUMI_CLOTH_SELF_ORDER=reference): the frame kernels of
    // cloth_self_order_kernels.cu; else the batched (Jacobi) order.
    if (const char* order = std::getenv("NUMI_CLOTH_SELF_ORDER")) h->self_exact = std::strcmp(order, "reference") == 0;

    // Launch geometry: one resident CTA for a small cloth, else a full
    // cooperative grid (as many CTAs as can be co-resident).
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, h->device);
    int per_sm = 0;
    raise_frame_smem(nc_resident_offset());
    // NUMI_CLOTH_BLOCK=512 runs the cooperative grid with 512-thread CTAs
    // (one per SM) instead of 256 (two per SM); NUMI_CLOTH_BLOCK=256 runs a
    // one-CTA cloth with 256 threads instead of 512.
    uint32_t block = NC_THREADS;
    const bool forced_block = env_u32("NUMI_CLOTH_BLOCK", block);
    if (forced_block && block != NC_BLOCK_MAX) block = NC_THREADS;
    h->block = block;
    per_sm = 1 << 30;
    for (const void* fn : {frame_fn(false, h->self_exact), frame_fn(true, h->self_exact), frame_tape_fn()}) {
        int k = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&k, fn, static_cast<int>(block), nc_resident_offset());
        per_sm = std::min(per_sm, k);
    }
    uint32_t work = std::max({n, D, K, B});
    uint32_t grid = (work <= 8192u) ? 1u : std::min<uint32_t>(sms * std::max(per_sm, 1), (work + block - 1u) / block);
    uint32_t forced = 0;
    if (env_u32("NUMI_CLOTH_GRID", forced) && forced > 0) grid = std::min<uint32_t>(forced, sms * std::max(per_sm, 1));
    h->grid = std::max(grid, 1u);
    // one CTA holds the whole cloth: every phase is latency-bound on one SM,
    // so it runs with the most threads (16 warps instead of 8: 20 % less
    // time per frame on the produce bag)
    if (h->grid == 1u && !forced_block) h->block = NC_BLOCK_MAX;
    // NUMI_CLOTH_CLUSTER=8 or =16 runs a large cloth as one thread-block
    // cluster (hardware cluster barrier) when the device can place it; the
    // default is the cooperative grid.
    uint32_t want_cluster = 0;
    env_u32("NUMI_CLOTH_CLUSTER", want_cluster);
    // Resident mode: particle positions and velocities stay in the shared
    // memory of one CTA (n <= 4096, the default) or, with
    // NUMI_CLOTH_RESIDENT=2, of one thread-block cluster of up to 16 CTAs
    // holding 4096 particles each (n <= 65536) for the whole frame, where
    // accesses to another CTA's particles go through distributed shared
    // memory.  NUMI_CLOTH_RESIDENT=0 keeps them in global memory.  The
    // cluster form is off by default: 16 CTAs leave too few threads to hide
    // the latency of a 65,536-particle cloth's colour batches, and it
    // measured slower than the cooperative grid.
    uint32_t want_resident = 1;
    env_u32("NUMI_CLOTH_RESIDENT", want_resident);
    const uint32_t resident_limit = want_resident >= 2u ? 16u * kResidentChunk : kResidentChunk;
    // Particles each CTA of a resident cluster holds: a cloth of up to
    // 4096 particles runs on a cluster of ceil(n / 256) CTAs (up to 16),
    // which measured 1.3-1.5x faster on the 1,400-particle bag than one CTA
    // holding it all (more threads per colour batch, the same bits); with
    // NUMI_CLOTH_RESIDENT=2 each CTA holds 4096.  NUMI_CLOTH_RESIDENT_CHUNK
    // (a power of two, 64 to 4096) overrides it.
    uint32_t chunk = want_resident >= 2u ? kResidentChunk : kResidentClusterChunk;
    env_u32("NUMI_CLOTH_RESIDENT_CHUNK", chunk);
    if (chunk < 64u || chunk > kResidentChunk || (chunk & (chunk - 1u)) != 0u) chunk = kResidentChunk;
    if (want_resident != 0u && forced == 0 && n > 0u && n <= resident_limit && (n + chunk - 1u) / chunk <= 16u) {
        uint32_t shift = 4u;
        while ((1u << shift) < std::min(n, chunk)) ++shift;
        const uint32_t ranks = (n + (1u << shift) - 1u) >> shift;
        const size_t smem = nc_resident_offset() + 2u * (static_cast<size_t>(1u) << shift) * sizeof(float4);
        int max_optin = 0;
        cudaDeviceGetAttribute(&max_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, h->device);
        cudaFuncAttributes fa{}, fe{};
        cudaFuncGetAttributes(&fa, frame_fn(false, h->self_exact));
        cudaFuncGetAttributes(&fe, frame_fn(true, h->self_exact));
        bool ok = smem + std::max(fa.sharedSizeBytes, fe.sharedSizeBytes) <= static_cast<size_t>(max_optin) &&
                  raise_frame_smem(smem) == cudaSuccess;
        if (ok && ranks > 1u) {
            allow_large_clusters();
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3(ranks);
            cfg.blockDim = dim3(NC_BLOCK_MAX);
            cfg.dynamicSmemBytes = smem;
            cudaLaunchAttribute attr{};
            attr.id = cudaLaunchAttributeClusterDimension;
            attr.val.clusterDim.x = ranks;
            attr.val.clusterDim.y = 1;
            attr.val.clusterDim.z = 1;
            cfg.attrs = &attr;
            cfg.numAttrs = 1;
            ok = frame_clusters(cfg) >= 1;
        }
        cudaGetLastError();
        if (ok) {
            d.resident = 1u;
            d.resident_shift = shift;
            h->smem = smem;
            h->grid = ranks;
            if (ranks > 1u) {
                h->cluster = ranks;
                h->block = NC_BLOCK_MAX;
            }
            want_cluster = 0;
        }
    }
    if (h->grid > 1 && want_cluster > 0 && forced == 0) {
        allow_large_clusters();
        for (uint32_t c : {want_cluster, 8u}) {
            if (c > 16u || c < 2u) continue;
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3(c);
            cfg.blockDim = dim3(NC_BLOCK_MAX);
            cfg.dynamicSmemBytes = nc_resident_offset();
            cudaLaunchAttribute attr{};
            attr.id = cudaLaunchAttributeClusterDimension;
            attr.val.clusterDim.x = c;
            attr.val.clusterDim.y = 1;
            attr.val.clusterDim.z = 1;
            cfg.attrs = &attr;
            cfg.numAttrs = 1;
            if (frame_clusters(cfg) >= 1) {
                h->cluster = c;
                h->grid = c;
                h->block = NC_BLOCK_MAX;
                break;
            }
        }
        cudaGetLastError();
    }
    // Bounded waits: NUMI_CLOTH_WAIT_LIMIT sets the polls a barrier or
    // neighbour wait makes before it raises TIMEOUT (default 2^22, a few
    // seconds).  NUMI_CLOTH_TEST_MISSING_CTA=1 is a failure-path test hook:
    // every grid barrier of the cooperative grid also waits for a CTA that
    // does not exist, so the first wait runs out and the launch ends with
    // TIMEOUT.
    env_u32("NUMI_CLOTH_WAIT_LIMIT", d.spin_limit);
    env_u32("NUMI_CLOTH_TEST_MISSING_CTA", d.bar_phantom);
    if (d.bar_phantom > 1u) d.bar_phantom = 1u;
    uint32_t trace_substeps = 0;
    if (env_u32("NUMI_CLOTH_TRACE", trace_substeps) && trace_substeps > 0) {
        d.trace = h->buf.alloc<unsigned long long>(static_cast<size_t>(trace_substeps) * NC_TRACE_SLOTS);
        h->trace_capacity = d.trace ? trace_substeps : 0u;
        uint32_t per_cta = 0;
        if (env_u32("NUMI_CLOTH_TRACE_CTA", per_cta) && per_cta > 0) {
            h->trace_ctas = h->grid + 1u;   // a small cloth's tile launch has one more than its cluster
            d.trace_cta = h->buf.alloc<unsigned long long>(static_cast<size_t>(trace_substeps) * NC_TRACE_SLOTS *
                                                           h->trace_ctas);
        }
    }
    const uint32_t chunks = (n + NC_THREADS - 1u) / NC_THREADS;
    d.red = h->buf.alloc<double>(std::max<size_t>(3u * 4096u, 2u * chunks + 8u));

    bool ok = d.x && d.xp && d.v && rest && d_ij && d_mat && d.d_lambda && k_ij && k_mat && d.k_lambda && b_ij &&
              b_mat && d.b_lambda && d.grips && d.fruits && d.pairs && cuff && d.yarn_slot_a && d.yarn_slot_b && d.yarn_live && d.yarn_list && d.yarn_list_n &&
              d.force && d.fruit_partial && d.failure && d.bar_count && d.abort_flag && d.stats && d.red && rim &&
              d.release;
    if (!ok) {
        delete h;
        return NUMI_CLOTH_ENOMEM;
    }

    // AoS -> SoA.
    std::vector<float4> hx(n), hxp(n), hv(n), hr(n);
    for (uint32_t i = 0; i < n; ++i) {
        const NumiClothParticle& p = scene->particles[i];
        hx[i] = make_float4(p.positionAndInverseMass.x, p.positionAndInverseMass.y, p.positionAndInverseMass.z,
                            p.positionAndInverseMass.w);
        hxp[i] = make_float4(p.previousAndMass.x, p.previousAndMass.y, p.previousAndMass.z, p.previousAndMass.w);
        hv[i] = make_float4(p.velocity.x, p.velocity.y, p.velocity.z, p.velocity.w);
        if (scene->restPositions != nullptr)
            hr[i] = make_float4(scene->restPositions[i].x, scene->restPositions[i].y, scene->restPositions[i].z, 0.0f);
        else
            hr[i] = make_float4(hx[i].x, hx[i].y, hx[i].z, 0.0f);
    }
    std::vector<uint2> hij(D);
    std::vector<float4> hdm(D);
    std::vector<float> hdl(D);
    for (uint32_t k = 0; k < D; ++k) {
        const NumiClothDistance& r = scene->distances[k];
        hij[k] = make_uint2(r.particlesAndColor.x, r.particlesAndColor.y);
        hdm[k] = make_float4(r.material.x, r.material.y, 0.0f, r.material.w);
        hdl[k] = r.material.z;
    }
    std::vector<uint4> hkij(K);
    std::vector<float2> hkm(K);
    std::vector<float> hkl(K);
    for (uint32_t k = 0; k < K; ++k) {
        const NumiClothKnot& r = scene->knots[k];
        hkij[k] = make_uint4(r.particles.x, r.particles.y, r.particles.z, r.particles.w);
        hkm[k] = make_float2(r.material.x, r.material.y);
        hkl[k] = r.material.z;
    }
    std::vector<uint4> hbij(B);
    std::vector<float2> hbm(B);
    std::vector<float> hbl(B);
    for (uint32_t k = 0; k < B; ++k) {
        const NumiClothBend& r = scene->bends[k];
        hbij[k] = make_uint4(r.particlesAndColor.x, r.particlesAndColor.y, r.particlesAndColor.z, 0u);
        hbm[k] = make_float2(r.material.x, r.material.z);
        hbl[k] = r.material.w;
    }
    cudaError_t e = cudaSuccess;
    auto up = [&](void* dst, const void* src, size_t bytes) {
        if (e == cudaSuccess && bytes) e = cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice);
    };
    up(d.x, hx.data(), n * sizeof(float4));
    up(d.xp, hxp.data(), n * sizeof(float4));
    up(d.v, hv.data(), n * sizeof(float4));
    up(rest, hr.data(), n * sizeof(float4));
    up(d_ij, hij.data(), D * sizeof(uint2));
    {
        // yarn segments: the distances that are not shear diagonals, in array order
        std::vector<uint2> hy;
        std::vector<float> rest_lengths;
        for (uint32_t k = 0; k < D; ++k) {
            const NumiClothDistance& r = scene->distances[k];
            if (r.particlesAndColor.w == 3u) continue;
            hy.push_back(make_uint2(r.particlesAndColor.x, r.particlesAndColor.y));
            rest_lengths.push_back(r.material.x);
        }
        if (!rest_lengths.empty()) {
            std::nth_element(rest_lengths.begin(), rest_lengths.begin() + rest_lengths.size() / 2, rest_lengths.end());
            h->yarn_rest_median = rest_lengths[rest_lengths.size() / 2];
        }
        uint2* y_ij = h->buf.alloc<uint2>(hy.size());
        if (y_ij == nullptr && e == cudaSuccess) e = cudaErrorMemoryAllocation;
        d.y_ij = y_ij;
        d.y_count = static_cast<uint32_t>(hy.size());
        up(y_ij, hy.data(), hy.size() * sizeof(uint2));
        h->host_yarn = hy;
    }
    up(d_mat, hdm.data(), D * sizeof(float4));
    up(d.d_lambda, hdl.data(), D * sizeof(float));
    up(k_ij, hkij.data(), K * sizeof(uint4));
    up(k_mat, hkm.data(), K * sizeof(float2));
    up(d.k_lambda, hkl.data(), K * sizeof(float));
    up(b_ij, hbij.data(), B * sizeof(uint4));
    up(b_mat, hbm.data(), B * sizeof(float2));
    up(d.b_lambda, hbl.data(), B * sizeof(float));
    up(d.grips, scene->grips, G * sizeof(NumiClothGrip));
    up(d.fruits, scene->fruits, F * sizeof(NumiClothFruit));
    up(d.pairs, scene->fruitPairs, P * sizeof(NumiClothFruitPair));
    if (cfg.gripControl.y == 1u) up(cuff, scene->cuffParticles, 2u * cfg.gripControl.z * sizeof(uint32_t));
    if (rim_count > 0u) up(rim, scene->mouthRim, rim_count * sizeof(uint32_t));
    if (scene->localOffsets != nullptr && scene->localIndices != nullptr) {
        // 2-hop topology CSR of the point self-contact exclusion
        const uint32_t entries = scene->localOffsets[n];
        uint32_t* off = h->buf.alloc<uint32_t>(n + 1u);
        uint32_t* idx = h->buf.alloc<uint32_t>(entries);
        if (off == nullptr || idx == nullptr) {
            delete h;
            return NUMI_CLOTH_ENOMEM;
        }
        up(off, scene->localOffsets, (n + 1u) * sizeof(uint32_t));
        up(idx, scene->localIndices, entries * sizeof(uint32_t));
        h->host_local_off.assign(scene->localOffsets, scene->localOffsets + n + 1u);
        h->host_local_idx.assign(scene->localIndices, scene->localIndices + entries);
        d.local_off = off;
        d.local_idx = idx;
    }
    if (e != cudaSuccess) {
        delete h;
        return NUMI_CLOTH_ECUDA;
    }
    h->neighbours = prepare_neighbours(h, scene);
    // Tile mode of the cooperative grid (cloth_tile.cuh): one 512-thread CTA
    // per SM, used by the launches whose schedule it covers;
    // on by default; NUMI_CLOTH_TILES=0 keeps the colour-by-colour schedule.
    uint32_t want_tiles = 1;
    env_u32("NUMI_CLOTH_TILES", want_tiles);
    // A small cloth that runs resident on a cluster of its own choice takes
    // tile mode too, on as many CTAs as the cluster has and one for the
    // fruits (the same share of the GPU when several cloths step at once):
    // five grid barriers a substep instead of 26 cluster barriers (a frame of
    // a 61 x 61 cloth: 3.6 -> 2.1 ms), once it has stepped a little
    // (prepare_small_tiles).  The
    // reference-order kernels stay on the cluster, whose barrier has no bound
    // for the ordered pass's serial fallback to outlast.
    if (want_tiles != 0u && h->cluster > 1u && d.resident != 0u && K == 0u && !h->self_exact && forced == 0u &&
        !forced_block && std::getenv("NUMI_CLOTH_CLUSTER") == nullptr && std::getenv("NUMI_CLOTH_RESIDENT") == nullptr &&
        std::getenv("NUMI_CLOTH_RESIDENT_CHUNK") == nullptr) {
        h->tile_grid = std::max(h->cluster + 1u, 3u);
        h->tile_block = NC_BLOCK_MAX;
        h->tile_source = std::make_unique<TileSource>(tile_source(h));
        h->tile_source->distances = hij;
        for (const uint4& q : hbij) h->tile_source->bends.push_back(make_uint2(q.x, q.z));
    }
    if (want_tiles != 0u && h->grid > 1u && h->cluster == 0u && d.resident == 0u && K == 0u) {
        uint32_t tgrid = static_cast<uint32_t>(sms);
        env_u32("NUMI_CLOTH_TILE_GRID", tgrid);
        h->tile_grid = std::max(tgrid, 3u);
        h->tile_block = NC_BLOCK_MAX;
        TileSource src = tile_source(h);
        src.distances = hij;
        for (const uint4& q : hbij) src.bends.push_back(make_uint2(q.x, q.z));
        TileBlock block;
        if (make_tiles(src, block)) adopt_tiles(h, std::move(block));
    }
    for (uint32_t g = 0; g < G; ++g) h->grip_compliance.push_back(scene->grips[g].targetOffsetAndCompliance.w);
    h->dynamic = {{d.x, n * sizeof(float4)},
                  {d.xp, n * sizeof(float4)},
                  {d.v, n * sizeof(float4)},
                  {d.d_lambda, std::max<size_t>(D, 1) * sizeof(float)},
                  {d.k_lambda, std::max<size_t>(K, 1) * sizeof(float)},
                  {d.b_lambda, std::max<size_t>(B, 1) * sizeof(float)},
                  {d.grips, std::max<size_t>(G, 1) * sizeof(NumiClothGrip)},
                  {d.fruits, std::max<size_t>(F, 1) * sizeof(NumiClothFruit)},
                  {d.pairs, std::max<size_t>(P, 1) * sizeof(NumiClothFruitPair)},
                  {d.release, 2u * sizeof(uint32_t)}};
    *out = h;
    return NUMI_CLOTH_OK;
}

void numi_cloth_destroy(numi_cloth_t* h) {
    if (h == nullptr) return;
    cudaSetDevice(h->device);
    if (h->tile_job) TileBuilder::get().abandon(h->tile_job);
    if (h->stream) cudaStreamSynchronize(h->stream);
    for (auto& s : h->snaps)
        if (s.mem) cudaFree(s.mem);
    cudaFree(h->d_cfg);
    delete h;
}

int numi_cloth_set_damping(numi_cloth_t* h, float damping) {
    if (h == nullptr || !std::isfinite(damping)) return NUMI_CLOTH_EINVAL;
    h->d.damping = damping < 0.0f ? -1.0f : damping;
    return NUMI_CLOTH_OK;
}

int numi_cloth_set_stream(numi_cloth_t* h, void* stream) {
    if (h == nullptr) return NUMI_CLOTH_EINVAL;
    h->stream = static_cast<cudaStream_t>(stream);
    return NUMI_CLOTH_OK;
}

int numi_cloth_step(numi_cloth_t* h, const NumiClothConfig* configs, uint32_t count,
                    const NumiClothSchedule* schedule) {
    if (h == nullptr || configs == nullptr || schedule == nullptr || count == 0) return NUMI_CLOTH_EINVAL;
    if (h->poisoned) return NUMI_CLOTH_ESTATE;
    cudaSetDevice(h->device);
    for (uint32_t k = 0; k < count; ++k) {
        const uint32_t bad = validate_config(configs[k], h->base);
        if (bad) {
            h->host_failure |= bad;
            return NUMI_CLOTH_OK;   // the failure word reports it; nothing ran
        }
    }
    if (count > h->cfg_capacity) {
        cudaFree(h->d_cfg);
        h->d_cfg = nullptr;
        h->cfg_capacity = 0;
        if (device_malloc(reinterpret_cast<void**>(&h->d_cfg), count * sizeof(NumiClothConfig)) != cudaSuccess)
            return NUMI_CLOTH_ECUDA;
        h->cfg_capacity = count;
    }
    if (cudaMemcpyAsync(h->d_cfg, configs, count * sizeof(NumiClothConfig), cudaMemcpyHostToDevice, h->stream) !=
        cudaSuccess)
        return NUMI_CLOTH_ECUDA;
    const Schedule s = device_schedule(*schedule);
    int rc = prepare_self_grid(h, s.self_collision != 0u, count, h->stream);
    if (rc == NUMI_CLOTH_OK) rc = prepare_edge_grid(h, s.primitive_self != 0u, count, configs[0].clothMaterial.x, h->stream);
    if (rc != NUMI_CLOTH_OK) return rc;
    const cudaError_t e = launch(h, count, s);
    h->epoch += count;
    if (e != cudaSuccess) {
        h->poisoned = true;
        return NUMI_CLOTH_ECUDA;
    }
    return NUMI_CLOTH_OK;
}

uint32_t numi_cloth_failure(numi_cloth_t* h) {
    if (h == nullptr) return NUMI_CLOTH_FAILURE_RANGE;
    cudaSetDevice(h->device);
    uint32_t f = 0;
    if (cudaStreamSynchronize(h->stream) != cudaSuccess ||
        cudaMemcpy(&f, h->d.failure, sizeof(f), cudaMemcpyDeviceToHost) != cudaSuccess) {
        h->poisoned = true;
        return h->host_failure | NUMI_CLOTH_FAILURE_RANGE;
    }
    return f | h->host_failure;
}

// Particle records <-> the state arrays (x, previous, v), one thread per
// particle: coalesced 16-byte loads and stores on both sides.
__global__ void numi_cloth_unpack_particles_kernel(const NumiClothParticle* in, float4* x, float4* xp, float4* v,
                                                   uint32_t n) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4* r = reinterpret_cast<const float4*>(in + i);
        x[i] = __ldcs(r);
        xp[i] = __ldcs(r + 1);
        v[i] = __ldcs(r + 2);
    }
}

__global__ void numi_cloth_pack_particles_kernel(const float4* x, const float4* xp, const float4* v,
                                                 NumiClothParticle* out, uint32_t n) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float4* r = reinterpret_cast<float4*>(out + i);
        __stcs(r, x[i]);
        __stcs(r + 1, xp[i]);
        __stcs(r + 2, v[i]);
    }
}

static_assert(sizeof(NumiClothParticle) == 3u * sizeof(float4), "particle record: three float4 words");

// The handle's staging buffer for particle records, allocated on first use.
static NumiClothParticle* particle_io(numi_cloth_t* h) {
    if (h->io == nullptr) h->io = h->buf.alloc<NumiClothParticle>(h->d.n, h->stream);
    return h->io;
}

int numi_cloth_read_particles(numi_cloth_t* h, NumiClothParticle* out, uint32_t count) {
    if (h == nullptr || out == nullptr || count != h->d.n) return NUMI_CLOTH_EINVAL;
    cudaSetDevice(h->device);
    NumiClothParticle* io = particle_io(h);
    if (io == nullptr) return NUMI_CLOTH_ECUDA;
    const uint32_t blocks = std::min<uint32_t>((count + 255u) / 256u, 1184u);
    numi_cloth_pack_particles_kernel<<<blocks, 256, 0, h->stream>>>(h->d.x, h->d.xp, h->d.v, io, count);
    if (cudaGetLastError() != cudaSuccess ||
        cudaMemcpyAsync(out, io, count * sizeof(NumiClothParticle), cudaMemcpyDeviceToHost, h->stream) !=
            cudaSuccess ||
        cudaStreamSynchronize(h->stream) != cudaSuccess)
        return NUMI_CLOTH_ECUDA;
    return NUMI_CLOTH_OK;
}

int numi_cloth_write_particles(numi_cloth_t* h, const NumiClothParticle* in, uint32_t count) {
    if (h == nullptr || in == nullptr || count != h->d.n) return NUMI_CLOTH_EINVAL;
    cudaSetDevice(h->device);
    NumiClothParticle* io = particle_io(h);
    if (io == nullptr) return NUMI_CLOTH_ECUDA;
    const uint32_t blocks = std::min<uint32_t>((count + 255u) / 256u, 1184u);
    if (cudaMemcpyAsync(io, in, count * sizeof(NumiClothParticle), cudaMemcpyHostToDevice, h->stream) !=
        cudaSuccess)
        return NUMI_CLOTH_ECUDA;
    numi_cloth_unpack_particles_kernel<<<blocks, 256, 0, h->stream>>>(io, h->d.x, h->d.xp, h->d.v, count);
    // synchronous: the caller may reuse its buffer on return
    if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(h->stream) != cudaSuccess)
        return NUMI_CLOTH_ECUDA;
    return NUMI_CLOTH_OK;
}

static int copy_records(numi_cloth_t* h, void* dst, const void* src, size_t bytes, cudaMemcpyKind kind) {
    cudaSetDevice(h->device);
    if (cudaStreamSynchronize(h->stream) != cudaSuccess) return NUMI_CLOTH_ECUDA;
    if (bytes && cudaMemcpy(dst, src, bytes, kind) != cudaSuccess) return NUMI_CLOTH_ECUDA;
    return NUMI_CLOTH_OK;
}

int numi_cloth_read_fruits(numi_cloth_t* h, NumiClothFruit* out, uint32_t count) {
    if (h == nullptr || (out == nullptr && count) || count != h->d.f_count) return NUMI_CLOTH_EINVAL;
    return copy_records(h, out, h->d.fruits, count * sizeof(NumiClothFruit), cudaMemcpyDeviceToHost);
}

int numi_cloth_write_fruits(numi_cloth_t* h, const NumiClothFruit* in, uint32_t count) {
    if (h == nullptr || (in == nullptr && count) || count != h->d.f_count) return NUMI_CLOTH_EINVAL;
    return copy_records(h, h->d.fruits, in, count * sizeof(NumiClothFruit), cudaMemcpyHostToDevice);
}

int numi_cloth_read_grips(numi_cloth_t* h, NumiClothGrip* out, uint32_t count) {
    if (h == nullptr || (out == nullptr && count) || count != h->d.g_count) return NUMI_CLOTH_EINVAL;
    return copy_records(h, out, h->d.grips, count * sizeof(NumiClothGrip), cudaMemcpyDeviceToHost);
}

int numi_cloth_read_distances(numi_cloth_t* h, NumiClothDistance* out, uint32_t count) {
    if (h == nullptr || out == nullptr || count != h->d.d_count) return NUMI_CLOTH_EINVAL;
    std::vector<uint2> ij(count);
    std::vector<float4> m(count);
    std::vector<float> l(count);
    int rc = copy_records(h, ij.data(), h->d.d_ij, count * sizeof(uint2), cudaMemcpyDeviceToHost);
    if (rc == NUMI_CLOTH_OK) rc = copy_records(h, m.data(), h->d.d_mat, count * sizeof(float4), cudaMemcpyDeviceToHost);
    if (rc == NUMI_CLOTH_OK) rc = copy_records(h, l.data(), h->d.d_lambda, count * sizeof(float), cudaMemcpyDeviceToHost);
    if (rc != NUMI_CLOTH_OK) return rc;
    for (uint32_t k = 0; k < count; ++k) {
        out[k].particlesAndColor.x = ij[k].x;
        out[k].particlesAndColor.y = ij[k].y;
        out[k].material = {m[k].x, m[k].y, l[k], m[k].w};
    }
    return NUMI_CLOTH_OK;
}

int numi_cloth_residuals(numi_cloth_t* h, double out[4]) {
    if (h == nullptr || out == nullptr) return NUMI_CLOTH_EINVAL;
    cudaSetDevice(h->device);
    const uint32_t grid = std::max<uint32_t>(1u, std::min<uint32_t>(h->grid, 4096u));
    DeviceCloth d = h->d;
    NumiClothConfig cfg = h->base;
    numi_cloth_residual_kernel<<<grid, NC_THREADS, 0, h->stream>>>(d, cfg);
    std::vector<double> r(3u * grid);
    if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(h->stream) != cudaSuccess ||
        cudaMemcpy(r.data(), d.red, r.size() * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess)
        return NUMI_CLOTH_ECUDA;
    out[0] = out[1] = out[2] = out[3] = 0.0;
    for (uint32_t b = 0; b < grid; ++b)
        for (int e = 0; e < 3; ++e) out[e] = std::max(out[e], r[3u * b + e]);
    return NUMI_CLOTH_OK;
}

int numi_cloth_self_contacts(numi_cloth_t* h, unsigned long long* contacts, double* max_penetration) {
    if (h == nullptr || contacts == nullptr || max_penetration == nullptr) return NUMI_CLOTH_EINVAL;
    *contacts = 0ull;
    *max_penetration = 0.0;
    if (h->d.self_stats == nullptr) return NUMI_CLOTH_OK;
    cudaSetDevice(h->device);
    unsigned long long st[2] = {0ull, 0ull};
    if (cudaStreamSynchronize(h->stream) != cudaSuccess ||
        cudaMemcpy(st, h->d.self_stats, sizeof(st), cudaMemcpyDeviceToHost) != cudaSuccess)
        return NUMI_CLOTH_ECUDA;
    *contacts = st[0];
    float pen = 0.0f;
    const uint32_t bits = static_cast<uint32_t>(st[1]);
    std::memcpy(&pen, &bits, sizeof(pen));
    *max_penetration = pen;
    return NUMI_CLOTH_OK;
}

int numi_cloth_self_order_stats(numi_cloth_t* h, unsigned long long out[4]) {
    if (h == nullptr || out == nullptr) return NUMI_CLOTH_EINVAL;
    for (int k = 0; k < 4; ++k) out[k] = 0ull;
    if (h->d.self_stats == nullptr) return NUMI_CLOTH_OK;
    cudaSetDevice(h->device);
    if (cudaStreamSynchronize(h->stream) != cudaSuccess ||
        cudaMemcpy(out, h->d.self_stats + 2, 4 * sizeof(unsigned long long), cudaMemcpyDeviceToHost) != cudaSuccess)
        return NUMI_CLOTH_ECUDA;
    return NUMI_CLOTH_OK;
}

int numi_cloth_edge_contacts(numi_cloth_t* h, unsigned long long out[2]) {
    if (h == nullptr || out == nullptr) return NUMI_CLOTH_EINVAL;
    out[0] = out[1] = 0ull;
    if (h->d.edge_stats == nullptr) return NUMI_CLOTH_OK;
    cudaSetDevice(h->device);
    if (cudaStreamSynchronize(h->stream) != cudaSuccess ||
        cudaMemcpy(out, h->d.edge_stats, 2u * sizeof(unsigned long long), cudaMemcpyDeviceToHost) != cudaSuccess)
        return NUMI_CLOTH_ECUDA;
    return NUMI_CLOTH_OK;
}

int numi_cloth_release_masks(numi_cloth_t* h, uint32_t out[2]) {
    if (h == nullptr || out == nullptr) return NUMI_CLOTH_EINVAL;
    out[0] = out[1] = 0u;
    cudaSetDevice(h->device);
    if (cudaStreamSynchronize(h->stream) != cudaSuccess ||
        cudaMemcpy(out, h->d.release, 2u * sizeof(uint32_t), cudaMemcpyDeviceToHost) != cudaSuccess)
        return NUMI_CLOTH_ECUDA;
    return NUMI_CLOTH_OK;
}

namespace {
int snapshot_slot(numi_cloth_t* h, uint32_t slot);
int restore_slot(numi_cloth_t* h, uint32_t slot);
}  // namespace

int numi_cloth_snapshot(numi_cloth_t* h, uint32_t slot) {
    if (h == nullptr || slot >= kSnapshotSlots) return NUMI_CLOTH_EINVAL;
    return snapshot_slot(h, slot);
}

int numi_cloth_restore(numi_cloth_t* h, uint32_t slot) {
    if (h == nullptr || slot >= kSnapshotSlots || !h->snaps[slot].valid) return NUMI_CLOTH_EINVAL;
    return restore_slot(h, slot);
}

}  // extern "C"

namespace {

void note_capture(numi_cloth* h) {
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(h->stream, &capturing) == cudaSuccess && capturing != cudaStreamCaptureStatusNone)
        h->compliance_captured = true;
}

// The dynamic state's regions (each a whole number of 4-byte words, 16-byte
// aligned) to or from one block, every region at a multiple of 256 bytes:
// one launch in place of ten copies of 2 us of host time each.
constexpr uint32_t kStateRegions = 16;
struct StateCopy {
    struct Op {
        const char* src;
        char* dst;
        uint32_t words;
    } op[kStateRegions];
};

__global__ void numi_cloth_state_copy_kernel(StateCopy c) {
    const StateCopy::Op op = c.op[blockIdx.y];
    const uint32_t quads = op.words / 4u;
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < quads; k += gridDim.x * blockDim.x)
        reinterpret_cast<uint4*>(op.dst)[k] = __ldcg(reinterpret_cast<const uint4*>(op.src) + k);
    if (blockIdx.x == 0u && threadIdx.x < op.words % 4u) {
        const uint32_t k = 4u * quads + threadIdx.x;
        reinterpret_cast<uint32_t*>(op.dst)[k] = __ldcg(reinterpret_cast<const uint32_t*>(op.src) + k);
    }
}

cudaError_t copy_state(numi_cloth* h, char* block, bool save) {
    StateCopy c{};
    uint32_t regions = 0, most = 0;
    for (const auto& r : h->dynamic) {
        if (regions == kStateRegions || r.bytes % 4u != 0u || r.bytes / 4u > 0xffffffffull) return cudaErrorInvalidValue;
        char* live = static_cast<char*>(r.ptr);
        const uint32_t words = static_cast<uint32_t>(r.bytes / 4u);
        c.op[regions++] = {save ? live : block, save ? block : live, words};
        most = std::max(most, words);
        block += (r.bytes + 255u) & ~size_t(255u);
    }
    const uint32_t blocks = std::max(1u, std::min(most / 4u / 256u, 148u));
    numi_cloth_state_copy_kernel<<<dim3(blocks, regions), 256, 0, h->stream>>>(c);
    return cudaGetLastError();
}

int snapshot_slot(numi_cloth_t* h, uint32_t slot) {
    cudaSetDevice(h->device);
    size_t total = 0;
    for (const auto& r : h->dynamic) total += (r.bytes + 255u) & ~size_t(255u);
    Snapshot& s = h->snaps[slot];
    if (s.mem == nullptr) {
        if (device_malloc(&s.mem, total) != cudaSuccess) return NUMI_CLOTH_ENOMEM;
        s.bytes = total;
    }
    if (copy_state(h, static_cast<char*>(s.mem), true) != cudaSuccess) return NUMI_CLOTH_ECUDA;
    s.grip_compliance = h->grip_compliance;
    note_capture(h);
    s.valid = true;
    return NUMI_CLOTH_OK;
}

int restore_slot(numi_cloth_t* h, uint32_t slot) {
    cudaSetDevice(h->device);
    if (copy_state(h, static_cast<char*>(h->snaps[slot].mem), false) != cudaSuccess) return NUMI_CLOTH_ECUDA;
    h->grip_compliance = h->snaps[slot].grip_compliance;
    note_capture(h);
    return NUMI_CLOTH_OK;
}
}  // namespace

extern "C" {

int numi_cloth_trace(numi_cloth_t* h, unsigned long long* out, uint32_t substeps, uint32_t slots) {
    if (h == nullptr || out == nullptr || slots != NC_TRACE_SLOTS) return NUMI_CLOTH_EINVAL;
    if (h->d.trace == nullptr || substeps > h->trace_capacity) return NUMI_CLOTH_ESTATE;
    cudaSetDevice(h->device);
    if (cudaStreamSynchronize(h->stream) != cudaSuccess ||
        cudaMemcpy(out, h->d.trace, static_cast<size_t>(substeps) * NC_TRACE_SLOTS * sizeof(unsigned long long),
                   cudaMemcpyDeviceToHost) != cudaSuccess)
        return NUMI_CLOTH_ECUDA;
    return NUMI_CLOTH_OK;
}

int numi_cloth_trace_cta(numi_cloth_t* h, unsigned long long* out, uint32_t substeps) {
    if (h == nullptr || out == nullptr) return NUMI_CLOTH_EINVAL;
    if (h->d.trace_cta == nullptr || substeps > h->trace_capacity) return NUMI_CLOTH_ESTATE;
    cudaSetDevice(h->device);
    // the last launch's CTAs (a tile launch may use fewer than the grid)
    const uint32_t grid = h->last_grid != 0u ? h->last_grid : h->grid;
    if (grid > h->trace_ctas) return NUMI_CLOTH_ESTATE;   // not traced per CTA
    if (cudaStreamSynchronize(h->stream) != cudaSuccess ||
        cudaMemcpy(out, h->d.trace_cta,
                   static_cast<size_t>(substeps) * NC_TRACE_SLOTS * grid * sizeof(unsigned long long),
                   cudaMemcpyDeviceToHost) != cudaSuccess)
        return NUMI_CLOTH_ECUDA;
    return NUMI_CLOTH_OK;
}

int numi_cloth_pass_counts(numi_cloth_t* h, uint32_t out[3]) {
    if (h == nullptr || out == nullptr) return NUMI_CLOTH_EINVAL;
    cudaSetDevice(h->device);
    uint32_t stats[4] = {0, 0, 0, 0};
    if (cudaStreamSynchronize(h->stream) != cudaSuccess ||
        cudaMemcpy(stats, h->d.stats, sizeof(stats), cudaMemcpyDeviceToHost) != cudaSuccess)
        return NUMI_CLOTH_ECUDA;
    out[0] = stats[0];
    out[1] = stats[1];
    out[2] = stats[2];
    return NUMI_CLOTH_OK;
}

}  // extern "C"

namespace {

// Tile plans for a tile launch of `grid` CTAs; false where the device does
// not hold that grid co-resident with their shared memory.
bool configure_tiles(numi_cloth* h, uint32_t grid) {
    const DeviceCloth& d = h->d;
    h->tile_grid = grid;
    h->tiles = false;
    TileSource src = tile_source(h);
    src.distances.resize(d.d_count);
    std::vector<uint4> bends(d.b_count);
    if (cudaStreamSynchronize(h->stream) != cudaSuccess ||
        (d.d_count &&
         cudaMemcpy(src.distances.data(), d.d_ij, d.d_count * sizeof(uint2), cudaMemcpyDeviceToHost) != cudaSuccess) ||
        (d.b_count && cudaMemcpy(bends.data(), d.b_ij, d.b_count * sizeof(uint4), cudaMemcpyDeviceToHost) != cudaSuccess))
        return false;
    for (const uint4& q : bends) src.bends.push_back(make_uint2(q.x, q.z));
    TileBlock block;
    if (make_tiles(src, block)) adopt_tiles(h, std::move(block));
    return h->tiles;
}

}  // namespace

extern "C" int numi_cloth_tune(numi_cloth_t* h, const NumiClothConfig* configs, uint32_t count,
                               const NumiClothSchedule* schedule, uint32_t out[4]) {
    if (h == nullptr || configs == nullptr || schedule == nullptr || count == 0 || out == nullptr)
        return NUMI_CLOTH_EINVAL;
    if (h->poisoned) return NUMI_CLOTH_ESTATE;
    cudaSetDevice(h->device);
    if (numi_cloth_failure(h) != 0u) return NUMI_CLOTH_ESTATE;   // a failed cloth is not timed
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, h->device);
    const Schedule sched = device_schedule(*schedule);
    const uint32_t colours = h->d.n_dist_batches + h->d.n_bend_batches;
    // the candidates: one colour per synchronisation (the colour-by-colour
    // launch), and tile mode at three CTA counts
    struct Shape {
        bool tiles;
        uint32_t grid;
    };
    std::vector<Shape> shapes;
    const bool had_tiles = h->tiles;
    const uint32_t had_grid = h->tile_grid;
    const bool tile_capable = h->tile_block != 0u && h->grid > 1u && h->cluster == 0u && h->d.resident == 0u;
    if (h->grid > 1u) shapes.push_back({false, h->grid});
    if (tile_capable) {
        h->tiles = true;   // tile_schedule asks only whether the schedule is covered
        const bool covered = tile_schedule(h, sched);
        h->tiles = had_tiles;
        if (covered)
            for (uint32_t g : {static_cast<uint32_t>(sms), static_cast<uint32_t>(3 * sms / 4), static_cast<uint32_t>(sms / 2)})
                shapes.push_back({true, std::max(g, 3u)});
    }
    auto report = [&](float us) {
        out[0] = h->tiles ? colours : 1u;
        out[1] = h->tiles ? h->tile_grid : h->grid;
        out[2] = h->tiles ? h->tile_block : h->block;
        out[3] = static_cast<uint32_t>(us);
    };
    if (shapes.size() < 2u) {
        report(0.0f);
        return NUMI_CLOTH_OK;
    }
    int rc = snapshot_slot(h, kTuneSlot);
    if (rc != NUMI_CLOTH_OK) return rc;
    cudaEvent_t t0, t1;
    cudaEventCreate(&t0);
    cudaEventCreate(&t1);
    float best_ms = INFINITY;
    size_t best = shapes.size();
    for (size_t k = 0; k < shapes.size() && rc == NUMI_CLOTH_OK; ++k) {
        if (shapes[k].tiles) {
            if (!configure_tiles(h, shapes[k].grid)) continue;
        } else {
            h->tiles = false;
        }
        float ms = 0.0f;
        for (int rep = 0; rep < 2 && rc == NUMI_CLOTH_OK; ++rep) {   // a warm-up run, then the timed one
            rc = restore_slot(h, kTuneSlot);
            if (rc == NUMI_CLOTH_OK) cudaEventRecord(t0, h->stream);
            if (rc == NUMI_CLOTH_OK) rc = numi_cloth_step(h, configs, count, schedule);
            if (rc == NUMI_CLOTH_OK) {
                cudaEventRecord(t1, h->stream);
                if (cudaEventSynchronize(t1) != cudaSuccess) rc = NUMI_CLOTH_ECUDA;
            }
        }
        if (rc != NUMI_CLOTH_OK) break;
        cudaEventElapsedTime(&ms, t0, t1);
        if (numi_cloth_failure(h) != 0u || h->host_failure != 0u) {
            // this shape failed (the caller's state comes back below)
            cudaMemsetAsync(h->d.failure, 0, sizeof(uint32_t), h->stream);
            h->host_failure = 0u;
            continue;
        }
        if (ms < best_ms) {
            best_ms = ms;
            best = k;
        }
    }
    cudaEventDestroy(t0);
    cudaEventDestroy(t1);
    // keep the fastest shape (else the one the cloth had) and its state
    if (best < shapes.size() && shapes[best].tiles) {
        if (!configure_tiles(h, shapes[best].grid)) best = shapes.size();
    } else if (best < shapes.size()) {
        h->tiles = false;
    }
    if (best == shapes.size()) {
        if (had_tiles)
            configure_tiles(h, had_grid);
        else
            h->tiles = false;
    }
    const int rrc = restore_slot(h, kTuneSlot);
    if (rc == NUMI_CLOTH_OK) rc = rrc;
    if (rc == NUMI_CLOTH_OK && cudaStreamSynchronize(h->stream) != cudaSuccess) rc = NUMI_CLOTH_ECUDA;
    report(best < shapes.size() ? 1000.0f * best_ms : 0.0f);
    return rc;
}

extern "C" {

int numi_cloth_launch_info(numi_cloth_t* h, uint32_t out[6]) {
    if (h == nullptr || out == nullptr) return NUMI_CLOTH_EINVAL;
    cudaSetDevice(h->device);
    uint32_t stats[4] = {0, 0, 0, 0};
    if (cudaStreamSynchronize(h->stream) != cudaSuccess ||
        cudaMemcpy(stats, h->d.stats, sizeof(stats), cudaMemcpyDeviceToHost) != cudaSuccess)
        return NUMI_CLOTH_ECUDA;
    // the shape of the last launch (tile mode has its own), else the default
    out[0] = h->last_grid != 0u ? h->last_grid : h->grid;
    out[1] = h->last_block != 0u ? h->last_block : h->block;
    out[2] = stats[0];
    out[3] = h->launches;
    out[4] = h->cluster;
    out[5] = h->d.resident | (h->neighbours ? 2u : 0u) | (h->tiles ? 4u : 0u) | (h->last_tiles ? 8u : 0u) |
             (h->self_exact ? 16u : 0u);
    return NUMI_CLOTH_OK;
}

}  // extern "C"

// ------------------------------------------------------------------------
// Allocation-free stepping (numi_cloth_step_noalloc in numi_cloth.h).  The
// array below is the only device memory this path uses besides the
// caller's buffers: contact records, air forces, fixed-point fruit sums,
// reduction partials and the substep Configs of one call.
namespace {

struct NoAllocScratch {
    float4 slot_a[NUMI_CLOTH_NOALLOC_MAX_DISTANCES * NC_YARN_SLOTS];
    float4 slot_b[NUMI_CLOTH_NOALLOC_MAX_DISTANCES * NC_YARN_SLOTS];
    uint32_t live[NUMI_CLOTH_NOALLOC_MAX_DISTANCES];
    uint32_t list[NUMI_CLOTH_NOALLOC_MAX_DISTANCES];
    uint32_t list_n[4];
    float4 force[NUMI_CLOTH_NOALLOC_MAX_PARTICLES];
    unsigned long long fruit_sums[9u * NC_MAX_FRUITS + 8u];
    double red[256];
    uint32_t stamp[NUMI_CLOTH_NOALLOC_MAX_PARTICLES + NC_MAX_FRUITS];
    NumiClothConfig configs[NUMI_CLOTH_NOALLOC_MAX_SUBSTEPS];
    unsigned long long barrier[32];
    uint32_t stats[4];
};

// File-scope device array.  In host code this name is only a stand-in for
// the symbol, never a device address; the address comes from
// cudaGetSymbolAddress, once per device.
static __device__ __align__(256) unsigned char g_noalloc_scratch[sizeof(NoAllocScratch)];

// The scratch array's device address on each device, looked up on the
// first call with that device current and kept for the process (stale after
// a cudaDeviceReset of the device).  The lookup runs under a mutex, so two
// host threads making their first calls on one device at once agree.
constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mutex;
NoAllocScratch* g_noalloc_ptr[kMaxDevices] = {};

NoAllocScratch* noalloc_scratch(int device) {
    if (device < 0 || device >= kMaxDevices) return nullptr;
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (g_noalloc_ptr[device] == nullptr) {
        void* ptr = nullptr;
        if (cudaGetSymbolAddress(&ptr, g_noalloc_scratch) != cudaSuccess || ptr == nullptr) return nullptr;
        g_noalloc_ptr[device] = static_cast<NoAllocScratch*>(ptr);
    }
    return g_noalloc_ptr[device];
}

int noalloc_reject(const char* what) {
    std::fprintf(stderr, "numi_cloth_step_noalloc: %s\n", what);
    return NUMI_CLOTH_EINVAL;
}

}  // namespace

extern "C" int numi_cloth_step_noalloc(const NumiClothConfig* base, const NumiClothDeviceState* st,
                                       const NumiClothBatch* batches, const uint32_t batchCounts[4],
                                       const NumiClothConfig* configs, uint32_t count,
                                       const NumiClothSchedule* schedule, void* stream_ptr) {
    if (base == nullptr || st == nullptr || configs == nullptr || schedule == nullptr || batchCounts == nullptr ||
        count == 0)
        return noalloc_reject("null argument or zero substeps");
    const uint32_t n = base->control.y, D = base->control.z, G = base->control.w;
    const uint32_t K = base->constraintCounts.x, B = base->constraintCounts.y, F = base->constraintCounts.w;
    const uint32_t P = base->contactCounts.x;
    if (n == 0 || n > NUMI_CLOTH_NOALLOC_MAX_PARTICLES)
        return noalloc_reject("particle count is zero or above NUMI_CLOTH_NOALLOC_MAX_PARTICLES (4096)");
    if (D > NUMI_CLOTH_NOALLOC_MAX_DISTANCES)
        return noalloc_reject("distance count above NUMI_CLOTH_NOALLOC_MAX_DISTANCES (8192)");
    if (count > NUMI_CLOTH_NOALLOC_MAX_SUBSTEPS)
        return noalloc_reject("substeps per call above NUMI_CLOTH_NOALLOC_MAX_SUBSTEPS (256)");
    if (F > NC_MAX_FRUITS || G > NC_MAX_GRIPS || P > NC_MAX_PAIRS)
        return noalloc_reject("fruit, grip or fruit-pair count above its limit");
    for (int k = 0; k < 4; ++k)
        if (batchCounts[k] > NC_MAX_BATCHES) return noalloc_reject("more than 64 colour runs in one family");
    if ((batchCounts[0] + batchCounts[1] + batchCounts[2] + batchCounts[3]) != 0u && batches == nullptr)
        return noalloc_reject("null batches");
    {
        // every colour run stays inside its family's records, and a distance
        // run's yarn and strain-limited prefixes inside the run
        const uint32_t records[4] = {D, K, B, P};
        const NumiClothBatch* run = batches;
        for (int fam = 0; fam < 4; ++fam)
            for (uint32_t k = 0; k < batchCounts[fam]; ++k, ++run) {
                const uint64_t first = run->control.x, cnt = run->control.y;
                if (first + cnt > records[fam]) return noalloc_reject("a colour run reaches past its family's records");
                if (fam == 0 && ((run->control.w & 0xffffu) > cnt || (run->control.w >> 16) > cnt))
                    return noalloc_reject("a distance run's yarn or strain-limited prefix is longer than the run");
            }
    }
    if (schedule->selfCollision)
        return noalloc_reject("selfCollision needs the point self-contact hash grid, which this path does not hold");
    if (schedule->release)
        return noalloc_reject("release needs the mouth rim, which NumiClothDeviceState does not carry");
    if (schedule->primitiveSelf)
        return noalloc_reject("primitiveSelf needs the edge/edge pass buffers, which this path does not hold");
    if (!st->positions || !st->previous || !st->velocities || !st->rest || !st->failure ||
        (D && (!st->distanceIJ || !st->distanceMaterial || !st->distanceLambda)) ||
        (K && (!st->knotIJ || !st->knotMaterial || !st->knotLambda)) ||
        (B && (!st->bendIJ || !st->bendMaterial || !st->bendLambda)) || (G && !st->grips) || (F && !st->fruits) ||
        (P && !st->fruitPairs) || (base->gripControl.y == 1u && !st->cuffParticles))
        return noalloc_reject("null device buffer");
    uint32_t bad = 0;
    for (uint32_t k = 0; k < count && bad == 0u; ++k) bad = validate_config(configs[k], *base);
    if (bad != 0u) return static_cast<int>(bad);
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) return NUMI_CLOTH_ECUDA;
    NoAllocScratch* scratch = noalloc_scratch(device);
    if (scratch == nullptr) return NUMI_CLOTH_ECUDA;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);

    DeviceCloth d{};
    d.x = reinterpret_cast<float4*>(st->positions);
    d.xp = reinterpret_cast<float4*>(st->previous);
    d.v = reinterpret_cast<float4*>(st->velocities);
    d.rest = reinterpret_cast<const float4*>(st->rest);
    d.n = n;
    d.d_ij = reinterpret_cast<const uint2*>(st->distanceIJ);
    d.d_mat = reinterpret_cast<const float4*>(st->distanceMaterial);
    d.d_lambda = st->distanceLambda;
    d.d_count = D;
    d.k_ij = reinterpret_cast<const uint4*>(st->knotIJ);
    d.k_mat = reinterpret_cast<const float2*>(st->knotMaterial);
    d.k_lambda = st->knotLambda;
    d.k_count = K;
    d.b_ij = reinterpret_cast<const uint4*>(st->bendIJ);
    d.b_mat = reinterpret_cast<const float2*>(st->bendMaterial);
    d.b_lambda = st->bendLambda;
    d.b_count = B;
    d.grips = st->grips;
    d.g_count = G;
    d.fruits = st->fruits;
    d.f_count = F;
    d.pairs = st->fruitPairs;
    d.p_count = P;
    d.cuff = st->cuffParticles;
    d.failure = st->failure;
    d.yarn_slot_a = scratch->slot_a;
    d.yarn_slot_b = scratch->slot_b;
    d.yarn_live = scratch->live;
    d.yarn_list = scratch->list;
    d.yarn_list_n = scratch->list_n;
    d.force = scratch->force;
    d.fruit_partial = reinterpret_cast<float4*>(scratch->fruit_sums);
    d.red = scratch->red;
    d.bar_count = scratch->barrier;
    d.abort_flag = reinterpret_cast<unsigned int*>(scratch->barrier + 1);
    d.bar_flag = scratch->barrier + 16;
    d.stats = scratch->stats;
    d.cfg = scratch->configs;
    d.epoch_base = 1u;   // contact records are cleared below, so epochs restart at 1
    d.damping = -1.0f;   // the schedule's damping applies (as on the handle path)
    d.check_stamp = scratch->stamp;   // the kernel checks the caller's records first
    Batch* families[4] = {d.dist_batches, d.knot_batches, d.bend_batches, d.pair_batches};
    uint32_t* family_counts[4] = {&d.n_dist_batches, &d.n_knot_batches, &d.n_bend_batches, &d.n_pair_batches};
    const NumiClothBatch* b = batches;
    for (int fam = 0; fam < 4; ++fam) {
        *family_counts[fam] = batchCounts[fam];
        for (uint32_t k = 0; k < batchCounts[fam]; ++k, ++b) {
            Batch& o = families[fam][k];
            o.first = b->control.x;
            o.count = b->control.y;
            o.yarn = fam == 0 ? (b->control.w & 0xffffu) : 0u;
            o.limited = fam == 0 ? (b->control.w >> 16) : 0u;
        }
    }
    // Every call shares the scratch: clear what must start at zero (contact
    // records and their live epochs, fixed-point fruit sums, barrier words,
    // stats) and the caller's failure word.
    cudaError_t e = cudaMemsetAsync(scratch->slot_b, 0, sizeof(scratch->slot_b), stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(scratch->live, 0, sizeof(scratch->live), stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(scratch->fruit_sums, 0, sizeof(scratch->fruit_sums), stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(scratch->barrier, 0, sizeof(scratch->barrier), stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(scratch->stats, 0, sizeof(scratch->stats), stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(st->failure, 0, sizeof(uint32_t), stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(scratch->configs, configs, count * sizeof(NumiClothConfig), cudaMemcpyHostToDevice,
                            stream);
    if (e != cudaSuccess) return NUMI_CLOTH_ECUDA;
    Schedule s{};
    s.iterations = schedule->iterations;
    s.strain_sweeps = schedule->strainSweeps;
    s.reconcile_passes = schedule->reconcilePasses;
    s.final_passes = schedule->finalPasses;
    s.certificate_passes = schedule->certificatePasses;
    s.early_exit = schedule->earlyExit;
    s.self_collision = schedule->selfCollision;
    s.aerodynamics = schedule->aerodynamics;
    s.swept_ground = schedule->sweptGround;
    s.swept_fruit_yarn = schedule->sweptFruitYarn;
    s.frictions = schedule->frictions;
    s.release = schedule->release;
    s.damping = schedule->damping;
    s.substeps = count;
    void* args[] = {&d, &s};
    e = raise_frame_smem(nc_resident_offset());
    if (e == cudaSuccess)
        e = cudaLaunchKernel(reinterpret_cast<const void*>(numi_cloth_frame_kernel), dim3(1), dim3(NC_THREADS), args,
                             nc_resident_offset(), stream);
    return e == cudaSuccess ? NUMI_CLOTH_OK : NUMI_CLOTH_ECUDA;
}

// ------------------------------------------------------------------------
// Batched stepping (numi_cloth_batch_* in numi_cloth.h): many independent
// cloths in one persistent launch.  Each CTA takes the next cloth from a
// device work queue (largest cloths first, so the last wave is short) and
// runs its whole frame alone with CTA barriers; the cloths' device state is
// their handles' own, so every per-handle read/write call still works.

struct numi_cloth_batch {
    int device = 0;
    cudaStream_t stream = nullptr;
    std::vector<numi_cloth*> cloths;   // caller order
    std::vector<uint32_t> order;       // launch position -> caller index
    DeviceBuffers buf;
    DeviceCloth* d_cloths = nullptr;   // launch order
    std::vector<DeviceCloth> host_cloths;   // the same on the host, as last laid out
    NumiClothConfig* d_cfg = nullptr;  // caller order, cloth-major
    uint32_t cfg_capacity = 0;         // substeps per cloth d_cfg holds
    uint32_t layout_substeps = 0;      // substeps the uploaded descriptors assume
    bool layout_valid = false;
    unsigned int* queue = nullptr;
    uint32_t* epoch = nullptr;         // device substep counter
    uint32_t epoch_host = 1;
    uint32_t block = NC_THREADS;
    uint32_t chunk = 0;                // resident particle chunk (0: none)
    bool edge_room = true;             // the shape leaves room for the box tree
    bool edge_lists = true;            // and for its lists
    uint32_t tree_segments = 0;        // of the largest member that has one
    uint32_t ctas = 0;
    size_t smem = 0;
    // the default shape (batch_fit): residency cloth by cloth, a cluster of
    // `ranks` CTAs per cloth; its launches with the edge/edge family run one
    // CTA per cloth
    bool fitted = false;
    uint32_t per_sm = 1;               // CTAs per SM of its launches without the edge/edge family
    size_t room = 0;                   // shared memory a CTA of those has for particles
    uint32_t fit_chunk = 0, fit_block = 0;   // the chunk and threads that shape reports
    uint32_t ranks = 1;
    uint32_t edge_ctas = 0;
    size_t edge_smem = 0;
    bool layout_edge = false;          // which of the two the descriptors are laid out for
    Workspace grad;   // rollout gradients
    bool rollout_touched = false;   // a fruit touched a cloth in the last rollout
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    void* graph_mem = nullptr;   // the captured launch's own descriptors and Configs
    const NumiClothConfig* graph_cfg = nullptr;
    uint32_t graph_substeps = 0;
};

namespace {

uint32_t log2_pow2(uint32_t v) {
    uint32_t s = 0;
    while ((1u << s) < v) ++s;
    return s;
}

// Shared memory of an edge/edge launch whose particles and fruits take `smem`.
size_t batch_edge_smem(const numi_cloth_batch* b, size_t smem, bool lists) {
    return nc_round256(smem) + edge_tree_bytes(b->tree_segments, lists);
}

// Launch shape: resident chunk (0 or a power of two), threads per CTA, and
// as many CTAs as fit on the device (never more than the cloths).
int batch_shape(numi_cloth_batch* b, uint32_t chunk, uint32_t block) {
    const size_t smem = nc_resident_offset() + (chunk ? 2u * static_cast<size_t>(chunk) * sizeof(float4) : 0u);
    int optin = 0, sms = 0;
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, b->device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, b->device);
    int per_sm = 1 << 30;
    bool edge_room = false, edge_lists = false;
    for (bool edge : {false, true}) {
        // the edge/edge kernel also holds the box tree's sort keys, and its
        // lists where an SM then holds as many CTAs as without; a shape
        // without room for the keys serves only schedules without that family
        cudaFuncAttributes fa{};
        if (cudaFuncGetAttributes(&fa, batch_fn(edge)) != cudaSuccess) return NUMI_CLOTH_ECUDA;
        int most = 0;
        for (bool lists : {false, true}) {
            if (lists && !edge) break;
            const size_t bytes = edge ? batch_edge_smem(b, smem, lists) : smem;
            int k = 0;
            if (bytes + fa.sharedSizeBytes > static_cast<size_t>(optin)) break;
            if (raise_smem(batch_fn(edge), bytes) != cudaSuccess) return NUMI_CLOTH_ECUDA;
            if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&k, batch_fn(edge), static_cast<int>(block), bytes) !=
                cudaSuccess)
                return NUMI_CLOTH_EINVAL;
            if (edge) {
                edge_room = true;
                edge_lists = lists && k >= most;
            } else {
                per_sm = k;
            }
            most = k;
        }
        if (!edge && most == 0) return NUMI_CLOTH_EINVAL;
    }
    b->edge_room = edge_room;
    b->edge_lists = edge_lists;
    b->chunk = chunk;
    b->block = block;
    b->smem = smem;
    b->ctas = std::min<uint32_t>(static_cast<uint32_t>(b->cloths.size()), static_cast<uint32_t>(sms * per_sm));
    b->fitted = false;
    b->ranks = 1u;
    b->layout_valid = false;
    return NUMI_CLOTH_OK;
}

// How a cloth of n particles lives in `room` bytes of the shared memory of
// each of its cluster's CTAs: positions and velocities where both fit (1),
// else the positions (2: every colour gathers them, velocities are read
// twice a substep), else neither (0).
struct Residency {
    uint32_t mode = 0, shift = 0;
    size_t bytes = 0;
};

Residency batch_residency(uint32_t n, uint32_t ranks, size_t room) {
    Residency r;
    r.shift = 4u;
    while ((static_cast<uint64_t>(ranks) << r.shift) < n) ++r.shift;
    const size_t one = std::min<size_t>(static_cast<size_t>(1) << r.shift, n) * sizeof(float4);
    r.mode = 2u * one <= room ? 1u : one <= room ? 2u : 0u;
    r.bytes = r.mode == 1u ? 2u * one : r.mode == 2u ? one : 0u;
    return r;
}

// Shared memory a CTA of the batch kernel has left for particles, where an
// SM holds `per_sm` of them.
size_t batch_room(const numi_cloth_batch* b, bool edge, uint32_t per_sm) {
    int optin = 0;
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, b->device);
    if (per_sm > 1u) {
        int sm = 0, reserved = 0;
        cudaDeviceGetAttribute(&sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, b->device);
        cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, b->device);
        optin = std::min(optin, sm / static_cast<int>(per_sm) - reserved);
    }
    cudaFuncAttributes fa{};
    if (cudaFuncGetAttributes(&fa, batch_fn(edge)) != cudaSuccess) return 0;
    cudaFuncAttributes ft = fa;
    if (!edge && cudaFuncGetAttributes(&ft, batch_tape_fn(false)) != cudaSuccess) return 0;
    const size_t fixed = nc_resident_offset() + std::max(fa.sharedSizeBytes, ft.sharedSizeBytes) + 256u +
                         (edge ? edge_tree_bytes(b->tree_segments, true) : 0u);
    return static_cast<size_t>(optin) > fixed ? static_cast<size_t>(optin) - fixed : 0u;
}

// Time until a queue of cloths (largest first) is empty, `workers` taking the
// next one when they are free.
template <class F>
double queue_time(const std::vector<uint32_t>& particles, size_t workers, F&& time) {
    std::priority_queue<double, std::vector<double>, std::greater<double>> free;
    double end = 0.0;
    for (uint32_t n : particles) {
        double at = 0.0;
        if (free.size() == workers) {
            at = free.top();
            free.pop();
        }
        at += time(n);
        free.push(at);
        end = std::max(end, at);
    }
    return end;
}

// CTAs per SM of a batch with a CTA per cloth: one of 512 threads, which
// ends a cloth's frame soonest (a frame is latency-bound on its SM), or two
// of 256, which end two cloths in less than twice that time.  24 substeps of
// cloths of 100, 576, 1,024, 1,600, 3,136 and 5,184 particles take 970, 1,130,
// 1,360, 1,630, 2,270 and 3,760 us alone on an SM with 512 threads, two of
// them with 256 threads each 990, 1,450, 1,640, 2,070, 4,050 and 6,210 (from some
// 2,700 on nothing of a cloth fits in half an SM's shared memory).  It is
// the queue that decides: 160 cloths of 576 take 2,117 us by ones and 1,446 by
// twos, 148 take 1,133 and 1,279, 300 cloths of 3,136 take 6,169 and 7,250,
// 400 square cloths of 24 to 64 particles a side 5.14 ms and 4.85, and 512 of
// 16 to 96, whose largest have 9,216 particles, 9.5 and 10.8.  The lines below
// are these times, which are off by some per cent.
uint32_t batch_per_sm(const numi_cloth_batch* b, size_t sms) {
    if (b->cloths.size() <= sms) return 1u;
    std::vector<uint32_t> particles;
    for (numi_cloth* h : b->cloths) particles.push_back(h->d.n);
    std::sort(particles.begin(), particles.end(), std::greater<uint32_t>());
    const double ones =
        queue_time(particles, sms, [](double n) { return n <= 4400.0 ? 900.0 + 0.46 * n : 900.0 + 0.55 * n; });
    const double twos =
        queue_time(particles, 2u * sms, [](double n) { return n <= 2700.0 ? 1000.0 + 0.68 * n : 430.0 + 1.13 * n; });
    return twos < 0.98 * ones ? 2u : 1u;
}

// The default launch shape: one or two CTAs per SM, particles in shared
// memory as far as they fit, and where there are SMs to spare a cluster of up
// to 8 CTAs per cloth, until each CTA holds 256 particles (the single cloth's
// resident cluster).  Launches with the edge/edge family, whose box tree takes
// most of an SM's shared memory, run one CTA of 512 threads per cloth.
int batch_fit(numi_cloth_batch* b) {
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, b->device);
    const uint32_t count = static_cast<uint32_t>(b->cloths.size());
    uint32_t largest = 0;
    for (numi_cloth* h : b->cloths) largest = std::max(largest, h->d.n);
    b->per_sm = batch_per_sm(b, static_cast<size_t>(std::max(sms, 1)));
    b->block = NC_BLOCK_MAX / b->per_sm;
    uint32_t ranks = 1;
    while (ranks < 8u && static_cast<uint64_t>(count) * 2u * ranks <= static_cast<uint64_t>(std::max(sms, 1)) &&
           256u * ranks < largest)
        ranks *= 2u;
    for (bool edge : {false, true}) {
        size_t room = batch_room(b, edge, edge ? 1u : b->per_sm);
        // two to an SM, particles in shared memory only where every cloth's
        // are: the others read theirs through the L1, which has what shared
        // memory leaves (400 cloths of 24 to 64 a side: 4.84 ms, 5.48 with
        // those in shared memory that fit)
        if (!edge && b->per_sm > 1u && batch_residency(largest, 1u, room).mode == 0u) room = 0u;
        if (!edge) b->room = room;
        const uint32_t block = edge ? NC_BLOCK_MAX : b->block;
        for (;;) {
            const uint32_t r = edge ? 1u : ranks;
            size_t bytes = 0;
            b->chunk = edge ? b->chunk : 0u;
            for (numi_cloth* h : b->cloths) {
                const Residency res = batch_residency(h->d.n, r, room);
                bytes = std::max(bytes, res.bytes);
                if (!edge && res.mode != 0u) b->chunk = std::max(b->chunk, h->d.n);
            }
            const size_t smem = nc_resident_offset() + bytes;
            const size_t launch = edge ? batch_edge_smem(b, smem, true) : smem;
            const void* fn = r > 1u ? batch_cluster_fn() : batch_fn(edge);
            if (raise_smem(fn, launch) != cudaSuccess) return NUMI_CLOTH_ECUDA;
            int fit = 0;
            if (r > 1u) {
                cudaLaunchAttribute attr{};
                attr.id = cudaLaunchAttributeClusterDimension;
                attr.val.clusterDim.x = r;
                attr.val.clusterDim.y = 1;
                attr.val.clusterDim.z = 1;
                cudaLaunchConfig_t cfg{};
                cfg.gridDim = dim3(r);
                cfg.blockDim = dim3(block);
                cfg.dynamicSmemBytes = launch;
                cfg.attrs = &attr;
                cfg.numAttrs = 1;
                if (cudaOccupancyMaxActiveClusters(&fit, fn, &cfg) != cudaSuccess ||
                    static_cast<uint32_t>(std::max(fit, 0)) < count) {
                    // not every cloth would have a cluster: fewer CTAs each
                    cudaGetLastError();
                    ranks /= 2u;
                    continue;
                }
            } else {
                int k = 0;
                if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&k, fn, static_cast<int>(block), launch) !=
                        cudaSuccess ||
                    k < 1)
                    return NUMI_CLOTH_EINVAL;
                fit = k * sms;
            }
            const uint32_t ctas = r * std::min<uint32_t>(count, static_cast<uint32_t>(fit));
            if (edge) {
                b->edge_smem = smem;
                b->edge_ctas = ctas;
            } else {
                b->smem = smem;
                b->ctas = ctas;
            }
            break;
        }
    }
    b->ranks = ranks;
    b->fitted = true;
    b->fit_chunk = b->chunk;
    b->fit_block = b->block;
    b->edge_room = b->edge_lists = true;
    b->layout_valid = false;
    return NUMI_CLOTH_OK;
}

// Launch of the batch kernel (of rollout gradients with `rollout`) over
// `cloths` (launch order) in the batch's shape; the work queue starts at
// zero.
cudaError_t batch_kernel(numi_cloth_batch* b, const DeviceCloth* cloths, const Schedule& s, bool rollout = false) {
    const bool edge = s.primitive_self != 0u;
    const bool fit_edge = b->fitted && edge;
    uint32_t ranks = fit_edge ? 1u : b->ranks;
    uint32_t count = static_cast<uint32_t>(b->cloths.size());
    Schedule sc = s;
    size_t smem = fit_edge ? b->edge_smem : b->smem;
    if (edge) {   // the box tree (the shape has room for it)
        sc.tree_keys = static_cast<uint32_t>(nc_round256(smem));
        sc.tree_lists = b->edge_lists ? 1u : 0u;
        smem = batch_edge_smem(b, smem, b->edge_lists);
    }
    cudaError_t e = cudaMemsetAsync(b->queue, 0, sizeof(unsigned int), b->stream);
    if (e != cudaSuccess) return e;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = ranks;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(fit_edge ? b->edge_ctas : b->ctas);
    cfg.blockDim = dim3(fit_edge ? NC_BLOCK_MAX : b->block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = b->stream;
    cfg.attrs = &attr;
    cfg.numAttrs = ranks > 1u ? 1u : 0u;
    unsigned int* queue = b->queue;
    void* args[] = {&cloths, &count, &sc, &queue, &ranks};
    const void* fn = rollout ? batch_tape_fn(ranks > 1u) : ranks > 1u ? batch_cluster_fn() : batch_fn(edge);
    if (rollout) e = raise_smem(fn, smem);
    return e == cudaSuccess ? cudaLaunchKernelExC(&cfg, fn, args) : e;
}

// Descriptors of every cloth for a launch of `substeps` Configs each.
int batch_layout(numi_cloth_batch* b, uint32_t substeps, bool edge) {
    if (b->layout_valid && b->layout_substeps == substeps && (!b->fitted || b->layout_edge == edge))
        return NUMI_CLOTH_OK;
    const uint32_t ranks = b->fitted && !edge ? b->ranks : 1u;
    const size_t room = !b->fitted ? 0u : edge ? batch_room(b, true, 1u) : b->room;
    const uint32_t count = static_cast<uint32_t>(b->cloths.size());
    std::vector<DeviceCloth>& host = b->host_cloths;
    host.resize(count);
    for (uint32_t j = 0; j < count; ++j) {
        const uint32_t k = b->order[j];
        DeviceCloth d = b->cloths[k]->d;
        d.cfg = b->d_cfg + static_cast<size_t>(k) * substeps;
        d.trace = nullptr;
        d.trace_cta = nullptr;
        d.cluster_barrier = ranks > 1u ? 1u : 0u;
        d.resident = (b->chunk != 0u && d.n <= b->chunk) ? 1u : 0u;
        d.resident_shift = b->chunk ? log2_pow2(b->chunk) : 0u;
        if (b->fitted) {
            const Residency res = batch_residency(d.n, ranks, room);
            d.resident = res.mode;
            d.resident_shift = res.shift;
        }
        host[j] = d;
    }
    if (cudaMemcpyAsync(b->d_cloths, host.data(), count * sizeof(DeviceCloth), cudaMemcpyHostToDevice, b->stream) !=
        cudaSuccess)
        return NUMI_CLOTH_ECUDA;
    if (cudaStreamSynchronize(b->stream) != cudaSuccess) return NUMI_CLOTH_ECUDA;
    b->layout_substeps = substeps;
    b->layout_edge = edge;
    b->layout_valid = true;
    return NUMI_CLOTH_OK;
}

// Validate and stage one launch: Configs, self-contact grids, descriptors.
int batch_prepare(numi_cloth_batch* b, const NumiClothConfig* configs, uint32_t substeps, const NumiClothSchedule& sched) {
    if (sched.primitiveSelf != 0u && !b->edge_room) return NUMI_CLOTH_EINVAL;   // set a smaller shape first
    const uint32_t count = static_cast<uint32_t>(b->cloths.size());
    for (uint32_t k = 0; k < count; ++k) {
        numi_cloth* h = b->cloths[k];
        if (h->poisoned) return NUMI_CLOTH_ESTATE;
        for (uint32_t q = 0; q < substeps; ++q) {
            const uint32_t bad = validate_config(configs[static_cast<size_t>(k) * substeps + q], h->base);
            if (bad) {
                h->host_failure |= bad;
                return static_cast<int>(bad);
            }
        }
    }
    if (substeps > b->cfg_capacity) {
        NumiClothConfig* cfg = b->buf.alloc<NumiClothConfig>(static_cast<size_t>(count) * substeps);
        if (cfg == nullptr) return NUMI_CLOTH_ENOMEM;
        b->d_cfg = cfg;
        b->cfg_capacity = substeps;
        b->layout_valid = false;
    }
    for (size_t k = 0; k < b->cloths.size(); ++k) {
        numi_cloth* h = b->cloths[k];
        void* before = h->d.hash_head;
        void* edge_before = h->d.edge_count;
        const float cell_before = h->d.edge_cell;
        h->epoch = b->epoch_host;
        int rc = prepare_self_grid(h, sched.selfCollision != 0u, substeps, b->stream);
        if (rc == NUMI_CLOTH_OK)
            rc = prepare_edge_grid(h, sched.primitiveSelf != 0u, substeps,
                                   configs[k * substeps].clothMaterial.x, b->stream);
        if (rc != NUMI_CLOTH_OK) return rc;
        if (h->d.hash_head != before || h->d.edge_count != edge_before || h->d.edge_cell != cell_before)
            b->layout_valid = false;
        if (h->stream != b->stream && h->stream != nullptr && cudaStreamSynchronize(h->stream) != cudaSuccess)
            return NUMI_CLOTH_ECUDA;
    }
    return batch_layout(b, substeps, sched.primitiveSelf != 0u);
}

// One step over `cloths` (launch order), whose Configs are d_cfg.
cudaError_t batch_launch(numi_cloth_batch* b, const DeviceCloth* cloths, NumiClothConfig* d_cfg,
                         const NumiClothConfig* configs, uint32_t substeps, const Schedule& s) {
    const uint32_t count = static_cast<uint32_t>(b->cloths.size());
    cudaError_t e = cudaMemcpyAsync(d_cfg, configs, static_cast<size_t>(count) * substeps * sizeof(NumiClothConfig),
                                    cudaMemcpyHostToDevice, b->stream);
    Schedule sc = s;
    sc.substeps = substeps;
    sc.epoch_ptr = b->epoch;
    if (e == cudaSuccess) e = batch_kernel(b, cloths, sc);
    if (e != cudaSuccess) return e;
    numi_cloth_epoch_kernel<<<1, 1, 0, b->stream>>>(b->epoch, substeps);
    return cudaGetLastError();
}

void batch_advance(numi_cloth_batch* b, uint32_t substeps) {
    b->epoch_host += substeps;
    for (numi_cloth* h : b->cloths) {
        h->epoch = b->epoch_host;
        h->last_substeps = substeps;
        ++h->launches;
    }
}

void batch_drop_graph(numi_cloth_batch* b) {
    if (b->exec) cudaGraphExecDestroy(b->exec);
    if (b->graph) cudaGraphDestroy(b->graph);
    cudaFree(b->graph_mem);   // (a launch in flight ends first)
    b->exec = nullptr;
    b->graph = nullptr;
    b->graph_mem = nullptr;
    b->graph_cfg = nullptr;
}

}  // namespace

extern "C" {

int numi_cloth_batch_create(numi_cloth_t* const* cloths, uint32_t count, numi_cloth_batch_t** out) {
    if (cloths == nullptr || out == nullptr || count == 0) return NUMI_CLOTH_EINVAL;
    *out = nullptr;
    auto* b = new numi_cloth_batch();
    b->device = cloths[0] ? cloths[0]->device : 0;
    for (uint32_t k = 0; k < count; ++k) {
        if (cloths[k] == nullptr || cloths[k]->device != b->device) {
            delete b;
            return NUMI_CLOTH_EINVAL;
        }
        for (uint32_t j = 0; j < k; ++j)
            if (cloths[j] == cloths[k]) {
                delete b;
                return NUMI_CLOTH_EINVAL;
            }
        b->cloths.push_back(cloths[k]);
        if (cloths[k]->d.y_count <= NC_EDGE_TREE_MAX)
            b->tree_segments = std::max(b->tree_segments, cloths[k]->d.y_count);
        b->epoch_host = std::max(b->epoch_host, cloths[k]->epoch);
    }
    cudaSetDevice(b->device);
    // largest work first: particles plus constraints
    b->order.resize(count);
    for (uint32_t k = 0; k < count; ++k) b->order[k] = k;
    auto work = [&](uint32_t k) {
        const DeviceCloth& d = b->cloths[k]->d;
        return static_cast<uint64_t>(d.n) + d.d_count + d.k_count + d.b_count;
    };
    std::stable_sort(b->order.begin(), b->order.end(), [&](uint32_t a, uint32_t c) { return work(a) > work(c); });
    b->d_cloths = b->buf.alloc<DeviceCloth>(count);
    b->queue = b->buf.alloc<unsigned int>(1);
    b->epoch = b->buf.alloc<uint32_t>(1);
    if (!b->d_cloths || !b->queue || !b->epoch ||
        cudaMemcpy(b->epoch, &b->epoch_host, sizeof(uint32_t), cudaMemcpyHostToDevice) != cudaSuccess) {
        delete b;
        return NUMI_CLOTH_ENOMEM;
    }
    const int rc = batch_fit(b);
    if (rc != NUMI_CLOTH_OK) {
        delete b;
        return rc;
    }
    *out = b;
    return NUMI_CLOTH_OK;
}

void numi_cloth_batch_destroy(numi_cloth_batch_t* b) {
    if (b == nullptr) return;
    cudaSetDevice(b->device);
    cudaStreamSynchronize(b->stream);
    batch_drop_graph(b);
    delete b;
}

int numi_cloth_batch_set_stream(numi_cloth_batch_t* b, void* stream) {
    if (b == nullptr) return NUMI_CLOTH_EINVAL;
    b->stream = static_cast<cudaStream_t>(stream);
    batch_drop_graph(b);
    return NUMI_CLOTH_OK;
}

int numi_cloth_batch_set_shape(numi_cloth_batch_t* b, uint32_t resident_chunk, uint32_t threads) {
    if (b == nullptr || (threads != NC_THREADS && threads != NC_BLOCK_MAX)) return NUMI_CLOTH_EINVAL;
    const bool power = (resident_chunk & (resident_chunk - 1u)) == 0u && resident_chunk <= 4096u;
    // what batch_shape or the tuner reported of the default shape
    const bool fit = !power && resident_chunk == b->fit_chunk && threads == b->fit_block;
    if (!power && !fit) return NUMI_CLOTH_EINVAL;
    cudaSetDevice(b->device);
    batch_drop_graph(b);
    return fit ? batch_fit(b) : batch_shape(b, resident_chunk, threads);
}

int numi_cloth_batch_shape(numi_cloth_batch_t* b, uint32_t out[3]) {
    if (b == nullptr || out == nullptr) return NUMI_CLOTH_EINVAL;
    out[0] = b->chunk;
    out[1] = b->block;
    out[2] = b->ctas;
    return NUMI_CLOTH_OK;
}

int numi_cloth_batch_step(numi_cloth_batch_t* b, const NumiClothConfig* configs, uint32_t substeps,
                          const NumiClothSchedule* schedule) {
    if (b == nullptr || configs == nullptr || schedule == nullptr || substeps == 0) return NUMI_CLOTH_EINVAL;
    cudaSetDevice(b->device);
    const int rc = batch_prepare(b, configs, substeps, *schedule);
    if (rc > 0) return NUMI_CLOTH_OK;   // a rejected Config: its cloth's failure word reports it
    if (rc != NUMI_CLOTH_OK) return rc;
    const cudaError_t e = batch_launch(b, b->d_cloths, b->d_cfg, configs, substeps, device_schedule(*schedule));
    batch_advance(b, substeps);
    if (e != cudaSuccess) {
        for (numi_cloth* h : b->cloths) h->poisoned = true;
        return NUMI_CLOTH_ECUDA;
    }
    return NUMI_CLOTH_OK;
}

int numi_cloth_batch_tune(numi_cloth_batch_t* b, const NumiClothConfig* configs, uint32_t substeps,
                          const NumiClothSchedule* schedule, uint32_t out[3]) {
    if (b == nullptr || configs == nullptr || schedule == nullptr || substeps == 0) return NUMI_CLOTH_EINVAL;
    cudaSetDevice(b->device);
    batch_drop_graph(b);
    uint32_t largest = 0;
    for (numi_cloth* h : b->cloths) largest = std::max(largest, h->d.n);
    const uint32_t slot = kTuneSlot;
    for (numi_cloth* h : b->cloths) {
        const int rc = snapshot_slot(h, slot);
        if (rc != NUMI_CLOTH_OK) return rc;
        if (h->stream && cudaStreamSynchronize(h->stream) != cudaSuccess) return NUMI_CLOTH_ECUDA;
    }
    if (cudaDeviceSynchronize() != cudaSuccess) return NUMI_CLOTH_ECUDA;
    cudaEvent_t t0, t1;
    cudaEventCreate(&t0);
    cudaEventCreate(&t1);
    float best_ms = INFINITY;
    constexpr uint32_t kFit = ~0u;   // the default shape
    uint32_t best_chunk = kFit, best_block = NC_BLOCK_MAX;
    auto shape = [&](uint32_t chunk, uint32_t block) { return chunk == kFit ? batch_fit(b) : batch_shape(b, chunk, block); };
    const uint32_t chunks[] = {kFit, 0u, 256u, 512u, 1024u, 2048u, 4096u};
    const uint32_t blocks[] = {NC_THREADS, NC_BLOCK_MAX};
    const Schedule s = device_schedule(*schedule);
    int rc = NUMI_CLOTH_OK;
    for (uint32_t chunk : chunks) {
        if (chunk != kFit && chunk > 0u && chunk / 2u >= largest) continue;   // same as a smaller chunk
        for (uint32_t block : blocks) {
            if (chunk == kFit && block != NC_BLOCK_MAX) continue;   // it has its own
            if (shape(chunk, block) != NUMI_CLOTH_OK) continue;
            if (schedule->primitiveSelf != 0u && !b->edge_room) continue;
            rc = batch_prepare(b, configs, substeps, *schedule);
            if (rc != NUMI_CLOTH_OK) break;
            cudaEventRecord(t0, b->stream);
            const cudaError_t e = batch_launch(b, b->d_cloths, b->d_cfg, configs, substeps, s);
            cudaEventRecord(t1, b->stream);
            if (e != cudaSuccess || cudaEventSynchronize(t1) != cudaSuccess) {
                rc = NUMI_CLOTH_ECUDA;
                break;
            }
            float ms = 0.0f;
            cudaEventElapsedTime(&ms, t0, t1);
            batch_advance(b, substeps);
            if (ms < best_ms) {
                best_ms = ms;
                best_chunk = chunk;
                best_block = block;
            }
            for (numi_cloth* h : b->cloths) restore_slot(h, slot);
            if (cudaDeviceSynchronize() != cudaSuccess) {
                rc = NUMI_CLOTH_ECUDA;
                break;
            }
        }
        if (rc != NUMI_CLOTH_OK) break;
    }
    cudaEventDestroy(t0);
    cudaEventDestroy(t1);
    if (rc != NUMI_CLOTH_OK) return rc;
    rc = shape(best_chunk, best_block);
    if (rc == NUMI_CLOTH_OK && out != nullptr) numi_cloth_batch_shape(b, out);
    return rc;
}

int numi_cloth_batch_capture(numi_cloth_batch_t* b, const NumiClothConfig* configs, uint32_t substeps,
                             const NumiClothSchedule* schedule) {
    if (b == nullptr || configs == nullptr || schedule == nullptr || substeps == 0) return NUMI_CLOTH_EINVAL;
    cudaSetDevice(b->device);
    batch_drop_graph(b);
    int rc = batch_prepare(b, configs, substeps, *schedule);
    if (rc > 0) return NUMI_CLOTH_EINVAL;
    if (rc != NUMI_CLOTH_OK) return rc;
    // the graph has descriptors and Configs of its own: a step with the other
    // kernel family (another residency and barrier) or another substep count
    // lays the batch's out anew in place
    const size_t count = b->cloths.size();
    DeviceCloth* cloths = nullptr;
    NumiClothConfig* d_cfg = nullptr;
    auto pieces = [&](Carver& c) {
        cloths = c.get<DeviceCloth>(count);
        d_cfg = c.get<NumiClothConfig>(count * substeps);
    };
    Carver measure{nullptr};
    pieces(measure);
    if (device_malloc(&b->graph_mem, measure.used) != cudaSuccess) {
        b->graph_mem = nullptr;
        return NUMI_CLOTH_ENOMEM;
    }
    Carver carver{static_cast<char*>(b->graph_mem)};
    pieces(carver);
    std::vector<DeviceCloth> host = b->host_cloths;
    for (size_t j = 0; j < count; ++j) host[j].cfg = d_cfg + static_cast<size_t>(b->order[j]) * substeps;
    if (cudaMemcpy(cloths, host.data(), count * sizeof(DeviceCloth), cudaMemcpyHostToDevice) != cudaSuccess) {
        batch_drop_graph(b);
        return NUMI_CLOTH_ECUDA;
    }
    cudaStream_t cap = nullptr;
    if (cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking) != cudaSuccess) {
        batch_drop_graph(b);
        return NUMI_CLOTH_ECUDA;
    }
    cudaStream_t saved = b->stream;
    b->stream = cap;
    cudaError_t e = cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
        const cudaError_t le = batch_launch(b, cloths, d_cfg, configs, substeps, device_schedule(*schedule));
        e = cudaStreamEndCapture(cap, &b->graph);
        if (le != cudaSuccess) e = le;
    }
    b->stream = saved;
    cudaStreamDestroy(cap);
    if (e == cudaSuccess) e = cudaGraphInstantiate(&b->exec, b->graph, 0);
    if (e != cudaSuccess) {
        batch_drop_graph(b);
        cudaGetLastError();
        return NUMI_CLOTH_ECUDA;
    }
    b->graph_cfg = configs;
    b->graph_substeps = substeps;
    return NUMI_CLOTH_OK;
}

int numi_cloth_batch_replay(numi_cloth_batch_t* b) {
    if (b == nullptr || b->exec == nullptr) return NUMI_CLOTH_ESTATE;
    cudaSetDevice(b->device);
    const uint32_t count = static_cast<uint32_t>(b->cloths.size());
    for (uint32_t k = 0; k < count; ++k) {
        numi_cloth* h = b->cloths[k];
        if (h->poisoned) return NUMI_CLOTH_ESTATE;
        for (uint32_t q = 0; q < b->graph_substeps; ++q) {
            const uint32_t bad = validate_config(b->graph_cfg[static_cast<size_t>(k) * b->graph_substeps + q], h->base);
            if (bad) {
                h->host_failure |= bad;
                return NUMI_CLOTH_OK;
            }
        }
        if (h->d.hash_head != nullptr && ((b->epoch_host + b->graph_substeps) >> 26) != (b->epoch_host >> 26))
            return NUMI_CLOTH_ESTATE;   // tag wrap: capture again after a plain step
    }
    const cudaError_t e = cudaGraphLaunch(b->exec, b->stream);
    batch_advance(b, b->graph_substeps);
    if (e != cudaSuccess) {
        for (numi_cloth* h : b->cloths) h->poisoned = true;
        return NUMI_CLOTH_ECUDA;
    }
    return NUMI_CLOTH_OK;
}

}  // extern "C"

// ------------------------------------------------------------------------
// Reverse-mode gradients of a rollout (numi_cloth_rollout_grad).

namespace {

// Substeps a rollout tapes at once: all of them where the tape fits
// kTapeBytes, which needs no replay; else as many whole checkpoint intervals
// as fit, at least one.
//
// Where a fruit touches the cloth, the gradient is taken along replays from
// checkpoints at the caller's interval, as it has always been: a replay meets
// the forward's contact records of the same substeps and resolves the fruits'
// friction by them, so its trajectory, and the loss and gradient on it, are
// not quite the forward's.  Whether one touches shows only as the forward
// runs.  So a cloth with fruits is taped and checkpointed, and the tape is
// used where nothing was recorded; a rollout after one that did record does
// not tape.
//
// However it is taped, a rollout's gradients are summed checkpoint interval
// by interval (AdjointArgs::interval): equal calls give equal bits.
// NUMI_CLOTH_TAPE_BYTES is a test hook: a smaller limit gives small rollouts
// several segments.
constexpr size_t kTapeBytes = size_t(8) << 30;
uint32_t taped_substeps(uint32_t substeps, uint32_t checkpoint_every, size_t bytes_per_substep) {
    uint32_t limit = 0;
    const size_t bytes = env_u32("NUMI_CLOTH_TAPE_BYTES", limit) ? limit : kTapeBytes;
    const size_t fit = bytes / std::max<size_t>(bytes_per_substep, 1u);
    if (substeps <= fit) return substeps;
    const size_t whole = std::max<size_t>(fit / checkpoint_every, 1u) * checkpoint_every;
    return static_cast<uint32_t>(std::min<size_t>(whole, substeps));
}

// Barrier sequence of one substep for the schedules the adjoint supports
// (one iteration, no reconciliation / final / certificate passes, no air
// load, no self contact): mirrors nc::substep.
std::vector<uint4> adjoint_phases(const DeviceCloth& d, const Schedule& s) {
    std::vector<uint4> ph;
    auto add = [&](uint32_t type, uint32_t first, uint32_t count) { ph.push_back(make_uint4(type, first, count, 0u)); };
    add(ADJ_BEGIN, 0u, 0u);
    for (uint32_t b = 0; b < d.n_dist_batches; ++b) add(ADJ_DIST, d.dist_batches[b].first, d.dist_batches[b].count);
    for (uint32_t b = 0; b < d.n_knot_batches; ++b) add(ADJ_KNOT, d.knot_batches[b].first, d.knot_batches[b].count);
    for (uint32_t b = 0; b < d.n_bend_batches; ++b) add(ADJ_BEND, d.bend_batches[b].first, d.bend_batches[b].count);
    add(ADJ_GRIP, 0u, 0u);
    if (d.f_count > 0u)
        for (uint32_t b = 0; b < d.n_dist_batches; ++b)
            if (d.dist_batches[b].yarn != 0u) add(ADJ_YARN, 0u, 0u);
    add(ADJ_GROUND, 0u, 0u);
    for (uint32_t sw = 0; sw < s.strain_sweeps; ++sw)
        for (uint32_t b = 0; b < d.n_dist_batches; ++b)
            if (d.dist_batches[b].limited != 0u)
                add(ADJ_STRAIN, d.dist_batches[b].first, d.dist_batches[b].limited);
    add(ADJ_FINAL, 0u, 0u);
    // fruit/yarn friction and the fruit tail share the substep's last phase
    add(ADJ_TAIL, 0u, 0u);
    return ph;
}

// Launch shape of the reverse sweep of `count` cloths: a cluster of `ranks`
// CTAs per cloth.  More CTAs shorten a phase until each of its items has a
// thread of its own (256 items a CTA leave half of its threads for the FP64
// units to switch between), as long as all clusters run at once: one
// 64 x 64 cloth takes 8, 96 bags one each.
struct AdjointShape {
    uint32_t ranks = 1;
    bool shared = true;
    size_t smem = 0;
};

uint32_t adjoint_shift(uint32_t n, uint32_t ranks) {
    uint32_t shift = 0;
    while ((static_cast<uint64_t>(ranks) << shift) < n) ++shift;
    return shift;
}

int adjoint_shape(int device, const std::vector<const DeviceCloth*>& cloths, AdjointShape& out) {
    int optin = 0, sms = 0;
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    uint32_t items = 0;
    for (const DeviceCloth* d : cloths) {
        for (uint32_t b = 0; b < d->n_dist_batches; ++b) items = std::max(items, d->dist_batches[b].count);
        for (uint32_t b = 0; b < d->n_knot_batches; ++b) items = std::max(items, d->knot_batches[b].count);
        for (uint32_t b = 0; b < d->n_bend_batches; ++b) items = std::max(items, d->bend_batches[b].count);
    }
    uint32_t ranks = 1;
    while (ranks < ADJ_CLUSTER_MAX && 256u * ranks < items &&
           cloths.size() * 2u * ranks <= static_cast<size_t>(std::max(sms, 1)))
        ranks *= 2u;
    const void* fns[2] = {reinterpret_cast<const void*>(numi_cloth_adjoint_kernel<true>),
                          reinterpret_cast<const void*>(numi_cloth_adjoint_kernel<false>)};
    for (;; ranks /= 2u) {
        size_t smem = 0;
        for (const DeviceCloth* d : cloths) {
            const size_t chunk = static_cast<size_t>(1) << adjoint_shift(d->n, ranks);
            smem = std::max(smem, std::min<size_t>(chunk, d->n) * 3u * sizeof(double));
        }
        cudaFuncAttributes fa{};
        if (cudaFuncGetAttributes(&fa, fns[0]) != cudaSuccess) return NUMI_CLOTH_ECUDA;
        out.ranks = ranks;
        out.shared = smem + fa.sharedSizeBytes <= static_cast<size_t>(optin);
        out.smem = out.shared ? smem : 0u;
        const void* fn = fns[out.shared ? 0 : 1];
        if (out.shared && raise_smem(fn, smem) != cudaSuccess) return NUMI_CLOTH_ECUDA;
        if (ranks == 1u) return NUMI_CLOTH_OK;
        cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        cudaLaunchAttribute attr{};
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = ranks;
        attr.val.clusterDim.y = 1;
        attr.val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(ranks);
        cfg.blockDim = dim3(ADJ_THREADS);
        cfg.dynamicSmemBytes = out.smem;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        // every cloth's cluster at once: sixteen clusters of 8 take two
        // turns where the GPU's partitions hold fifteen
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, fn, &cfg) == cudaSuccess &&
            static_cast<size_t>(std::max(clusters, 0)) >= cloths.size())
            return NUMI_CLOTH_OK;
        cudaGetLastError();
    }
}

cudaError_t adjoint_launch(const AdjointShape& shape, const AdjointArgs* args, uint32_t count, cudaStream_t stream) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = shape.ranks;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(count * shape.ranks);
    cfg.blockDim = dim3(ADJ_THREADS);
    cfg.dynamicSmemBytes = shape.smem;
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = shape.ranks > 1u ? 1u : 0u;
    return shape.shared ? cudaLaunchKernelEx(&cfg, numi_cloth_adjoint_kernel<true>, args, shape.ranks)
                        : cudaLaunchKernelEx(&cfg, numi_cloth_adjoint_kernel<false>, args, shape.ranks);
}

// Compliance groups: the distinct compliance values of each constraint
// family (distance, knot, bend, grip), ascending, numbered family by family.
struct Groups {
    std::vector<uint32_t> family;
    std::vector<float> value;
    std::vector<uint8_t> d, k, b, g;   // per record
};

// Distinct values, ascending, and every value's index among them.
void distinct_values(const std::vector<float>& values, std::vector<float>& distinct, std::vector<uint8_t>& ids) {
    distinct = values;
    std::sort(distinct.begin(), distinct.end());
    distinct.erase(std::unique(distinct.begin(), distinct.end()), distinct.end());
    ids.resize(values.size());
    for (size_t r = 0; r < values.size(); ++r)
        ids[r] = static_cast<uint8_t>(std::lower_bound(distinct.begin(), distinct.end(), values[r]) - distinct.begin());
}

int read_compliance(numi_cloth* h) {
    if (h->compliance_known && !h->compliance_captured) return NUMI_CLOTH_OK;
    const DeviceCloth& d = h->d;
    std::vector<float4> dm(d.d_count);
    std::vector<float2> km(d.k_count), bm(d.b_count);
    cudaError_t e = cudaStreamSynchronize(h->stream);
    if (e == cudaSuccess && d.d_count) e = cudaMemcpy(dm.data(), d.d_mat, d.d_count * sizeof(float4), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && d.k_count) e = cudaMemcpy(km.data(), d.k_mat, d.k_count * sizeof(float2), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && d.b_count) e = cudaMemcpy(bm.data(), d.b_mat, d.b_count * sizeof(float2), cudaMemcpyDeviceToHost);
    std::vector<NumiClothGrip> grips(h->compliance_captured ? d.g_count : 0u);
    if (e == cudaSuccess && !grips.empty())
        e = cudaMemcpy(grips.data(), d.grips, grips.size() * sizeof(NumiClothGrip), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return NUMI_CLOTH_ECUDA;
    for (size_t g = 0; g < grips.size(); ++g) h->grip_compliance[g] = grips[g].targetOffsetAndCompliance.w;
    std::vector<float> v;
    for (const float4& m : dm) v.push_back(m.y);
    distinct_values(v, h->compliance[0], h->compliance_id[0]);
    v.clear();
    for (const float2& m : km) v.push_back(m.y);
    distinct_values(v, h->compliance[1], h->compliance_id[1]);
    v.clear();
    for (const float2& m : bm) v.push_back(m.y);
    distinct_values(v, h->compliance[2], h->compliance_id[2]);
    // more values than groups can be: read again when asked again
    h->compliance_known = h->compliance[0].size() + h->compliance[1].size() + h->compliance[2].size() <= NUMI_CLOTH_MAX_GROUPS;
    return NUMI_CLOTH_OK;
}

int compliance_groups(numi_cloth* h, Groups& out) {
    const int rc = read_compliance(h);
    if (rc != NUMI_CLOTH_OK) return rc;
    auto assign = [&](uint32_t family, const std::vector<float>& distinct, const std::vector<uint8_t>& id,
                      std::vector<uint8_t>& ids) {
        const uint32_t base = static_cast<uint32_t>(out.value.size());
        for (float v : distinct) {
            out.family.push_back(family);
            out.value.push_back(v);
        }
        ids.resize(id.size());
        for (size_t r = 0; r < id.size(); ++r) ids[r] = static_cast<uint8_t>(base + id[r]);
    };
    std::vector<float> grip;
    std::vector<uint8_t> grip_id;
    distinct_values(h->grip_compliance, grip, grip_id);
    assign(0u, h->compliance[0], h->compliance_id[0], out.d);
    assign(1u, h->compliance[1], h->compliance_id[1], out.k);
    assign(2u, h->compliance[2], h->compliance_id[2], out.b);
    assign(3u, grip, grip_id, out.g);
    return out.value.size() <= NUMI_CLOTH_MAX_GROUPS ? NUMI_CLOTH_OK : NUMI_CLOTH_EINVAL;
}

// The host copy after every record of `family` with compliance `from` took
// `to`: the values stay distinct and ascending.
void replaced_compliance(numi_cloth* h, uint32_t family, float from, float to) {
    if (family == 3u) {
        for (float& v : h->grip_compliance)
            if (v == from) v = to;
        return;
    }
    if (!h->compliance_known) return;
    std::vector<float>& values = h->compliance[family];
    std::vector<float> moved = values, distinct;
    for (float& v : moved)
        if (v == from) v = to;
    std::vector<uint8_t> at;   // old index -> new index
    distinct_values(moved, distinct, at);
    for (uint8_t& id : h->compliance_id[family]) id = at[id];
    values = distinct;
}

__global__ void numi_cloth_replace_compliance_kernel(DeviceCloth d, uint32_t family, float from, float to) {
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;; k += stride) {
        bool any = false;
        if (family == 0u && k < d.d_count) {
            any = true;
            float4* m = const_cast<float4*>(d.d_mat) + k;
            if (m->y == from) m->y = to;
        }
        if (family == 1u && k < d.k_count) {
            any = true;
            float2* m = const_cast<float2*>(d.k_mat) + k;
            if (m->y == from) m->y = to;
        }
        if (family == 2u && k < d.b_count) {
            any = true;
            float2* m = const_cast<float2*>(d.b_mat) + k;
            if (m->y == from) m->y = to;
        }
        if (family == 3u && k < d.g_count) {
            any = true;
            if (d.grips[k].targetOffsetAndCompliance.w == from) d.grips[k].targetOffsetAndCompliance.w = to;
        }
        if (!any) break;
    }
}

}  // namespace

extern "C" int numi_cloth_compliance_groups(numi_cloth_t* h, uint32_t family[NUMI_CLOTH_MAX_GROUPS],
                                            float compliance[NUMI_CLOTH_MAX_GROUPS], uint32_t* count) {
    if (h == nullptr || family == nullptr || compliance == nullptr || count == nullptr) return NUMI_CLOTH_EINVAL;
    cudaSetDevice(h->device);
    Groups g;
    const int rc = compliance_groups(h, g);
    if (rc != NUMI_CLOTH_OK) return rc;
    *count = static_cast<uint32_t>(g.value.size());
    for (size_t k = 0; k < g.value.size(); ++k) {
        family[k] = g.family[k];
        compliance[k] = g.value[k];
    }
    return NUMI_CLOTH_OK;
}

extern "C" int numi_cloth_replace_compliance(numi_cloth_t* h, uint32_t family, float from, float to) {
    if (h == nullptr || family > 3u || !(to >= 0.0f) || !std::isfinite(to)) return NUMI_CLOTH_EINVAL;
    cudaSetDevice(h->device);
    numi_cloth_replace_compliance_kernel<<<64, 256, 0, h->stream>>>(h->d, family, from, to);
    if (cudaGetLastError() != cudaSuccess) return NUMI_CLOTH_ECUDA;
    // a tile plan's items carry the materials
    if (h->tiles && (family == 0u || family == 2u) && tile_materials(h) != cudaSuccess) return NUMI_CLOTH_ECUDA;
    replaced_compliance(h, family, from, to);
    note_capture(h);
    return NUMI_CLOTH_OK;
}

extern "C" int numi_cloth_rollout_grad(numi_cloth_t* h, const NumiClothConfig* configs, uint32_t substeps,
                                       const NumiClothSchedule* schedule, uint32_t checkpoint_every,
                                       const uint32_t* tracked, uint32_t n_tracked, const double* targets,
                                       uint32_t loss_every, double* loss, double* grads, double* grip_grads,
                                       uint32_t* nonsmooth) {
    if (h == nullptr || configs == nullptr || schedule == nullptr || substeps == 0 || checkpoint_every == 0 ||
        loss == nullptr || grads == nullptr || (n_tracked > 0 && (tracked == nullptr || targets == nullptr)) ||
        loss_every == 0)
        return NUMI_CLOTH_EINVAL;
    if (h->poisoned) return NUMI_CLOTH_ESTATE;
    const NumiClothSchedule& sc = *schedule;
    if (sc.iterations != 1u || sc.reconcilePasses != 0u || sc.finalPasses != 0u || sc.certificatePasses != 0u ||
        sc.aerodynamics != 0u || sc.selfCollision != 0u || sc.primitiveSelf != 0u)
        return NUMI_CLOTH_EINVAL;
    for (uint32_t t = 0; t < n_tracked; ++t)
        if (tracked[t] >= h->d.n) return NUMI_CLOTH_EINVAL;
    cudaSetDevice(h->device);
    for (uint32_t k = 0; k < substeps; ++k) {
        const uint32_t bad = validate_config(configs[k], h->base);
        if (bad) {
            h->host_failure |= bad;
            return static_cast<int>(bad);
        }
    }
    if (substeps > h->cfg_capacity) {
        cudaFree(h->d_cfg);
        h->d_cfg = nullptr;
        h->cfg_capacity = 0;
        if (device_malloc(reinterpret_cast<void**>(&h->d_cfg), substeps * sizeof(NumiClothConfig)) != cudaSuccess)
            return NUMI_CLOTH_ECUDA;
        h->cfg_capacity = substeps;
    }
    if (cudaMemcpyAsync(h->d_cfg, configs, substeps * sizeof(NumiClothConfig), cudaMemcpyHostToDevice, h->stream) !=
        cudaSuccess)
        return NUMI_CLOTH_ECUDA;
    const Schedule s = device_schedule(sc);
    const std::vector<uint4> phases = adjoint_phases(h->d, s);
    const uint32_t slots = static_cast<uint32_t>(phases.size()) + 1u;
    const uint32_t n = h->d.n;
    const uint32_t losses = substeps / loss_every;

    Groups groups;
    {
        const int rc = compliance_groups(h, groups);
        if (rc != NUMI_CLOTH_OK) return rc;
    }
    const uint32_t ngroups = static_cast<uint32_t>(groups.value.size());
    size_t state_bytes = 0;
    for (const auto& r : h->dynamic) state_bytes += (r.bytes + 255u) & ~size_t(255u);
    // the taped segment, and without a tape of the whole rollout the
    // checkpoints of the segments before it
    const size_t tape_step = static_cast<size_t>(slots + 1u) * n * sizeof(float4) + h->d.g_count * sizeof(NumiClothGrip);
    uint32_t every = taped_substeps(substeps, checkpoint_every, tape_step);   // substeps on the tape
    const bool fruits = h->d.f_count > 0u;
    const uint32_t interval = std::min(checkpoint_every, substeps);
    if (fruits && (h->rollout_touched || every < substeps)) every = interval;
    uint32_t seg = 0, segs = 0;   // substeps of a forward launch, their number
    float4 *tape_x = nullptr, *tape_v = nullptr;
    NumiClothGrip* tape_grip = nullptr;
    char* ckpt = nullptr;
    uint4* d_phases = nullptr;
    DeviceCloth* d_cloth = nullptr;
    AdjointArgs* d_args = nullptr;
    uint32_t* d_tracked = nullptr;
    double* d_targets = nullptr;
    double4 *gx = nullptr, *gv = nullptr, *gprev = nullptr;
    double *d_out = nullptr, *d_grip = nullptr;   // d_out: group gradients, damping, loss
    uint8_t *gd = nullptr, *gk = nullptr, *gb = nullptr, *gg = nullptr;
    unsigned int* d_rough = nullptr;
    uint32_t* d_touched = nullptr;
    char* zero_end = nullptr;
    auto layout = [&](Carver& c) {
        seg = fruits ? interval : every;
        segs = (substeps + seg - 1u) / seg;
        // zeroed
        gx = c.get<double4>(n);
        gv = c.get<double4>(n);
        gprev = c.get<double4>(n);
        d_out = c.get<double>(ngroups + 2u);
        d_grip = c.get<double>(static_cast<size_t>(substeps) * 6u);
        d_rough = c.get<unsigned int>(1);
        d_touched = c.get<uint32_t>(1);
        zero_end = c.get<char>(0);
        // written before they are read
        d_phases = c.get<uint4>(phases.size());
        d_cloth = c.get<DeviceCloth>(1);
        d_args = c.get<AdjointArgs>(1);
        d_tracked = c.get<uint32_t>(n_tracked);
        d_targets = c.get<double>(static_cast<size_t>(losses) * n_tracked * 3u);
        gd = c.get<uint8_t>(groups.d.size());
        gk = c.get<uint8_t>(groups.k.size());
        gb = c.get<uint8_t>(groups.b.size());
        gg = c.get<uint8_t>(groups.g.size());
        tape_x = c.get<float4>(static_cast<size_t>(every) * slots * n);
        tape_v = c.get<float4>(static_cast<size_t>(every) * n);
        tape_grip = c.get<NumiClothGrip>(static_cast<size_t>(every) * h->d.g_count);
        if (fruits || segs > 1u) ckpt = c.get<char>((segs + 1u) * state_bytes);
    };
    Workspace::Lease mem(h->grad, h->stream);
    if (!mem.layout(layout, every > checkpoint_every)) {
        every = interval;
        if (!mem.layout(layout)) return NUMI_CLOTH_ENOMEM;
    }
    if (cudaMemsetAsync(gx, 0, static_cast<size_t>(zero_end - reinterpret_cast<char*>(gx)), h->stream) != cudaSuccess)
        return NUMI_CLOTH_ECUDA;
    // the whole rollout on the tape (with fruits only while none touched)
    bool whole = every == substeps && !(fruits && h->rollout_touched);
    cudaError_t e = cudaMemcpyAsync(d_phases, phases.data(), phases.size() * sizeof(uint4), cudaMemcpyHostToDevice,
                                    h->stream);
    if (e == cudaSuccess && n_tracked)
        e = cudaMemcpyAsync(d_tracked, tracked, n_tracked * sizeof(uint32_t), cudaMemcpyHostToDevice, h->stream);
    if (e == cudaSuccess && n_tracked && losses)
        e = cudaMemcpyAsync(d_targets, targets, static_cast<size_t>(losses) * n_tracked * 3u * sizeof(double),
                            cudaMemcpyHostToDevice, h->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_cloth, &h->d, sizeof(DeviceCloth), cudaMemcpyHostToDevice, h->stream);
    const std::vector<uint8_t>* lists[4] = {&groups.d, &groups.k, &groups.b, &groups.g};
    uint8_t* dst[4] = {gd, gk, gb, gg};
    for (int f = 0; f < 4 && e == cudaSuccess; ++f)
        if (!lists[f]->empty())
            e = cudaMemcpyAsync(dst[f], lists[f]->data(), lists[f]->size(), cudaMemcpyHostToDevice, h->stream);
    if (e != cudaSuccess) return NUMI_CLOTH_ECUDA;

    auto save = [&](uint32_t slot) { return copy_state(h, ckpt + slot * state_bytes, true) == cudaSuccess; };
    auto load = [&](uint32_t slot) { return copy_state(h, ckpt + slot * state_bytes, false) == cudaSuccess; };

    // forward in the handle's own launch shape: taped where the tape holds
    // it, else checkpointed (the last segment of a cloth without fruits is
    // taped as it runs)
    std::vector<uint32_t> seg_epoch(segs);
    auto last_taped = [&](uint32_t g) { return whole || (!fruits && g + 1u == segs); };
    for (uint32_t g = 0; g < segs; ++g) {
        const uint32_t first = g * seg;
        const uint32_t count = std::min(seg, substeps - first);
        seg_epoch[g] = h->epoch;
        if ((fruits || g + 1u < segs) && !save(g)) return NUMI_CLOTH_ECUDA;
        Tape tape;
        if (last_taped(g)) tape = Tape{tape_x, tape_v, tape_grip, slots, whole ? first : 0u};
        tape.touched = d_touched;
        e = launch(h, count, s, first, tape);
        h->epoch += count;
        if (e != cudaSuccess) {
            h->poisoned = true;
            return NUMI_CLOTH_ECUDA;
        }
    }
    const uint32_t end_epoch = h->epoch;
    if ((fruits || segs > 1u) && !save(segs)) return NUMI_CLOTH_ECUDA;
    if (fruits) {
        uint32_t touched = 0u;
        if (cudaMemcpyAsync(&touched, d_touched, sizeof(touched), cudaMemcpyDeviceToHost, h->stream) != cudaSuccess ||
            cudaStreamSynchronize(h->stream) != cudaSuccess) {
            h->poisoned = true;
            return NUMI_CLOTH_ECUDA;
        }
        h->rollout_touched = touched != 0u;
        if (touched != 0u) whole = false;
    }
    // backward: reverse the tape, or segment by segment after a taped replay
    // from its checkpoint
    const float damping = h->d.damping >= 0.0f ? h->d.damping : s.damping;
    const uint32_t launches = h->launches;
    AdjointShape shape;
    {
        const int rc = adjoint_shape(h->device, {&h->d}, shape);
        if (rc != NUMI_CLOTH_OK) return rc;
    }
    bool replayed = false;
    for (uint32_t g = whole ? 1u : segs; g-- > 0u;) {
        const uint32_t first = g * seg;
        const uint32_t count = whole ? substeps : std::min(seg, substeps - first);
        if (!last_taped(g)) {
            replayed = true;
            if (!load(g)) return NUMI_CLOTH_ECUDA;
            h->epoch = seg_epoch[g];
            e = launch(h, count, s, first, Tape{tape_x, tape_v, tape_grip, slots});
            h->epoch = end_epoch;
            if (e != cudaSuccess) {
                h->poisoned = true;
                return NUMI_CLOTH_ECUDA;
            }
        }
        AdjointArgs A{};
        A.cloth = d_cloth;
        A.cfg = h->d_cfg + first;
        A.tape = tape_x;
        A.tape_v = tape_v;
        A.tape_grip = tape_grip;
        A.phases = d_phases;
        A.slots = slots;
        A.shift = adjoint_shift(n, shape.ranks);
        A.substeps = count;
        A.first_substep = first;
        A.interval = checkpoint_every;
        A.damping = damping;
        A.frictions = s.frictions;
        A.tracked = d_tracked;
        A.n_tracked = n_tracked;
        A.targets = d_targets;
        A.loss_every = loss_every;
        A.gx = gx;
        A.gv = gv;
        A.gprev = gprev;
        A.d_group = gd;
        A.k_group = gk;
        A.b_group = gb;
        A.g_group = gg;
        A.groups = ngroups;
        A.grads = d_out;
        A.loss = d_out + ngroups + 1u;
        A.grip_grads = d_grip;
        A.nonsmooth = d_rough;
        e = cudaMemcpyAsync(d_args, &A, sizeof(A), cudaMemcpyHostToDevice, h->stream);
        if (e == cudaSuccess) e = adjoint_launch(shape, d_args, 1u, h->stream);
        if (e != cudaSuccess || cudaGetLastError() != cudaSuccess) {
            h->poisoned = true;
            return NUMI_CLOTH_ECUDA;
        }
    }
    if (replayed && !load(segs)) return NUMI_CLOTH_ECUDA;
    h->epoch = end_epoch;
    h->launches = launches;
    h->last_substeps = substeps;
    uint32_t barriers = 0;
    if (cudaMemcpyAsync(&barriers, h->d.stats, sizeof(uint32_t), cudaMemcpyDeviceToHost, h->stream) != cudaSuccess ||
        cudaStreamSynchronize(h->stream) != cudaSuccess) {
        h->poisoned = true;
        return NUMI_CLOTH_ECUDA;
    }
    // the phase list does not match the kernel's barriers (the last launch
    // was taped; in tile mode it counts its slots)
    if (barriers + 1u != slots) return NUMI_CLOTH_ESTATE;
    std::vector<double> out(ngroups + 2u);
    unsigned int rough = 0;
    e = cudaMemcpyAsync(out.data(), d_out, out.size() * sizeof(double), cudaMemcpyDeviceToHost, h->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(&rough, d_rough, sizeof(rough), cudaMemcpyDeviceToHost, h->stream);
    if (e == cudaSuccess && grip_grads)
        e = cudaMemcpyAsync(grip_grads, d_grip, static_cast<size_t>(substeps) * 6u * sizeof(double),
                            cudaMemcpyDeviceToHost, h->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
    if (e != cudaSuccess) {
        h->poisoned = true;
        return NUMI_CLOTH_ECUDA;
    }
    for (uint32_t k = 0; k <= ngroups; ++k) grads[k] = out[k];
    *loss = out[ngroups + 1u];
    if (nonsmooth) *nonsmooth = rough;
    return NUMI_CLOTH_OK;
}

// ------------------------------------------------------------------------
// Batched rollout gradients (numi_cloth_batch_rollout_grad): the forward of
// every cloth in one persistent launch per segment, the taped replays in one
// launch per segment, and the adjoint of every cloth's segment in one grid
// (a cluster per cloth).  Checkpoints are moved by one copy kernel per segment.

constexpr size_t kGripFloat4s = sizeof(NumiClothGrip) / sizeof(float4);   // a grip's room on the tape

extern "C" int numi_cloth_batch_rollout_grad(numi_cloth_batch_t* b, const NumiClothConfig* configs, uint32_t substeps,
                                             const NumiClothSchedule* schedule, uint32_t checkpoint_every,
                                             const uint32_t* tracked, uint32_t n_tracked, const double* targets,
                                             uint32_t loss_every, double* loss, double* grads, uint32_t* groups_out,
                                             uint32_t* nonsmooth) {
    if (b == nullptr || configs == nullptr || schedule == nullptr || substeps == 0 || checkpoint_every == 0 ||
        loss == nullptr || grads == nullptr || loss_every == 0 || (n_tracked > 0 && (tracked == nullptr || targets == nullptr)))
        return NUMI_CLOTH_EINVAL;
    const NumiClothSchedule& sc = *schedule;
    if (sc.iterations != 1u || sc.reconcilePasses != 0u || sc.finalPasses != 0u || sc.certificatePasses != 0u ||
        sc.aerodynamics != 0u || sc.selfCollision != 0u || sc.primitiveSelf != 0u)
        return NUMI_CLOTH_EINVAL;
    cudaSetDevice(b->device);
    batch_drop_graph(b);
    const uint32_t count = static_cast<uint32_t>(b->cloths.size());
    for (numi_cloth* h : b->cloths)
        for (uint32_t t = 0; t < n_tracked; ++t)
            if (tracked[t] >= h->d.n) return NUMI_CLOTH_EINVAL;
    // Configs, descriptors (always rebuilt: damping and compliances may have
    // changed since the last launch)
    b->layout_valid = false;
    {
        const int rc = batch_prepare(b, configs, substeps, sc);
        if (rc > 0) return rc;
        if (rc != NUMI_CLOTH_OK) return rc;
    }
    cudaError_t e = cudaMemcpyAsync(b->d_cfg, configs, static_cast<size_t>(count) * substeps * sizeof(NumiClothConfig),
                                    cudaMemcpyHostToDevice, b->stream);
    if (e != cudaSuccess) return NUMI_CLOTH_ECUDA;
    const Schedule s = device_schedule(sc);
    const uint32_t losses = substeps / loss_every;

    // per cloth: groups, phase list, tape, checkpoints, adjoint arrays
    std::vector<Groups> groups(count);
    std::vector<std::vector<uint4>> phases(count);
    AdjointShape shape;
    {
        std::vector<const DeviceCloth*> all;
        for (numi_cloth* h : b->cloths) all.push_back(&h->d);
        const int rc = adjoint_shape(b->device, all, shape);
        if (rc != NUMI_CLOTH_OK) return rc;
    }
    std::vector<size_t> state_bytes(count);
    size_t tape_step = 0, state_total = 0;   // float4s a substep tapes, bytes of a checkpoint
    uint32_t regions = 0;
    for (uint32_t k = 0; k < count; ++k) {
        numi_cloth* h = b->cloths[k];
        const int rc = compliance_groups(h, groups[k]);
        if (rc != NUMI_CLOTH_OK) return rc;
        phases[k] = adjoint_phases(h->d, s);
        tape_step += (phases[k].size() + 2u) * h->d.n + kGripFloat4s * h->d.g_count;   // positions, velocities, grips
        for (const auto& r : h->dynamic) state_bytes[k] += (r.bytes + 255u) & ~size_t(255u);
        state_total += state_bytes[k];
        regions += static_cast<uint32_t>(h->dynamic.size());
    }
    uint32_t every = taped_substeps(substeps, checkpoint_every, tape_step * sizeof(float4));   // substeps on the tape
    bool fruits = false;
    for (numi_cloth* h : b->cloths) fruits = fruits || h->d.f_count > 0u;
    const uint32_t interval = std::min(checkpoint_every, substeps);
    if (fruits && (b->rollout_touched || every < substeps)) every = interval;
    uint32_t seg = 0, segs = 0;   // substeps of a forward launch, their number
    uint32_t* d_touched = nullptr;
    float4* tape = nullptr;
    char *ckpt = nullptr, *arena = nullptr, *zero = nullptr, *zero_end = nullptr;
    uint32_t* d_tracked = nullptr;
    double *d_targets = nullptr, *d_out = nullptr;
    unsigned int* d_rough = nullptr;
    DeviceCloth *d_replay = nullptr, *d_plain = nullptr;   // launch order with the tape; caller order for the adjoint
    AdjointArgs* d_args = nullptr;
    CopyOp* d_ops = nullptr;
    std::vector<double4*> adjoint(count);   // a cloth's gx, gv and gprev
    // one arena for every cloth's phase list and group ids
    auto round256 = [](size_t v) { return (v + 255u) & ~size_t(255u); };
    size_t arena_bytes = 0;
    for (uint32_t k = 0; k < count; ++k)
        arena_bytes += round256(phases[k].size() * sizeof(uint4)) + round256(groups[k].d.size() + 1u) +
                       round256(groups[k].k.size() + 1u) + round256(groups[k].b.size() + 1u) +
                       round256(groups[k].g.size() + 1u);
    auto layout = [&](Carver& c) {
        seg = fruits ? interval : every;
        segs = (substeps + seg - 1u) / seg;
        // zeroed
        zero = c.get<char>(0);
        for (uint32_t k = 0; k < count; ++k) adjoint[k] = c.get<double4>(3u * static_cast<size_t>(b->cloths[k]->d.n));
        d_out = c.get<double>(static_cast<size_t>(count) * (NUMI_CLOTH_MAX_GROUPS + 2u));
        d_rough = c.get<unsigned int>(count);
        d_touched = c.get<uint32_t>(1);
        zero_end = c.get<char>(0);
        // written before they are read
        arena = c.get<char>(arena_bytes);
        d_tracked = c.get<uint32_t>(n_tracked);
        d_targets = c.get<double>(static_cast<size_t>(count) * losses * n_tracked * 3u);
        d_replay = c.get<DeviceCloth>(count);
        d_plain = c.get<DeviceCloth>(count);
        d_args = c.get<AdjointArgs>(count);
        tape = c.get<float4>(tape_step * every);
        if (fruits || segs > 1u) {
            d_ops = c.get<CopyOp>(2u * static_cast<size_t>(segs + 1u) * regions);
            ckpt = c.get<char>((segs + 1u) * state_total);
        }
    };
    Workspace::Lease mem(b->grad, b->stream);
    if (!mem.layout(layout, every > checkpoint_every)) {
        every = interval;
        if (!mem.layout(layout)) return NUMI_CLOTH_ENOMEM;
    }
    // the whole rollout on the tape (with fruits only while none touched)
    bool whole = every == substeps && !(fruits && b->rollout_touched);
    if (cudaMemsetAsync(zero, 0, static_cast<size_t>(zero_end - zero), b->stream) != cudaSuccess)
        return NUMI_CLOTH_ECUDA;
    std::vector<AdjointArgs> args(count);
    std::vector<DeviceCloth> replay(count), plain(count);
    std::vector<char> host_arena(arena_bytes);   // filled cloth by cloth, uploaded once
    size_t cursor = 0;
    float4* tape_at = tape;
    auto carve = [&](const void* from, size_t bytes, size_t room) {
        char* p = arena + cursor;
        if (bytes != 0u) std::memcpy(host_arena.data() + cursor, from, bytes);
        cursor += round256(room);
        return p;
    };
    for (uint32_t k = 0; k < count; ++k) {
        numi_cloth* h = b->cloths[k];
        const uint32_t n = h->d.n;
        const uint32_t slots = static_cast<uint32_t>(phases[k].size()) + 1u;
        double4* gx = adjoint[k];
        const size_t ph_bytes = phases[k].size() * sizeof(uint4);
        const uint4* ph = reinterpret_cast<const uint4*>(carve(phases[k].data(), ph_bytes, ph_bytes));
        auto ids = [&](const std::vector<uint8_t>& list) {
            return reinterpret_cast<const uint8_t*>(carve(list.data(), list.size(), list.size() + 1u));
        };
        const uint8_t* gd = ids(groups[k].d);
        const uint8_t* gk = ids(groups[k].k);
        const uint8_t* gb = ids(groups[k].b);
        const uint8_t* gg = ids(groups[k].g);
        plain[k] = h->d;
        AdjointArgs& A = args[k];
        A.cloth = d_plain + k;
        A.tape = tape_at;
        A.tape_v = A.tape + static_cast<size_t>(every) * slots * n;
        tape_at += static_cast<size_t>(every) * (slots + 1u) * n;
        A.tape_grip = reinterpret_cast<const NumiClothGrip*>(tape_at);
        tape_at += static_cast<size_t>(every) * kGripFloat4s * h->d.g_count;
        A.phases = ph;
        A.slots = slots;
        A.shift = adjoint_shift(n, shape.ranks);
        A.interval = checkpoint_every;
        A.damping = h->d.damping >= 0.0f ? h->d.damping : s.damping;
        A.frictions = s.frictions;
        A.tracked = d_tracked;
        A.n_tracked = n_tracked;
        A.targets = d_targets + static_cast<size_t>(k) * losses * n_tracked * 3u;
        A.loss_every = loss_every;
        A.gx = gx;
        A.gv = gx + n;
        A.gprev = gx + 2u * static_cast<size_t>(n);
        A.d_group = gd;
        A.k_group = gk;
        A.b_group = gb;
        A.g_group = gg;
        A.groups = static_cast<uint32_t>(groups[k].value.size());
        A.grads = d_out + static_cast<size_t>(k) * (NUMI_CLOTH_MAX_GROUPS + 2u);
        A.loss = A.grads + NUMI_CLOTH_MAX_GROUPS + 1u;
        A.grip_grads = nullptr;
        A.nonsmooth = d_rough + k;
    }
    // replay descriptors: the batch's launch-order descriptors with tapes
    for (uint32_t j = 0; j < count; ++j) {
        const uint32_t k = b->order[j];
        replay[j] = b->host_cloths[j];
        replay[j].tape = const_cast<float4*>(args[k].tape);
        replay[j].tape_v = const_cast<float4*>(args[k].tape_v);
        replay[j].tape_grip = const_cast<NumiClothGrip*>(args[k].tape_grip);
        replay[j].tape_slots = args[k].slots;
        replay[j].yarn_touched = d_touched;
    }
    e = cudaMemcpyAsync(arena, host_arena.data(), arena_bytes, cudaMemcpyHostToDevice, b->stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(d_replay, replay.data(), count * sizeof(DeviceCloth), cudaMemcpyHostToDevice, b->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_plain, plain.data(), count * sizeof(DeviceCloth), cudaMemcpyHostToDevice, b->stream);
    if (e == cudaSuccess && n_tracked)
        e = cudaMemcpyAsync(d_tracked, tracked, n_tracked * sizeof(uint32_t), cudaMemcpyHostToDevice, b->stream);
    if (e == cudaSuccess && n_tracked && losses)
        e = cudaMemcpyAsync(d_targets, targets, static_cast<size_t>(count) * losses * n_tracked * 3u * sizeof(double),
                            cudaMemcpyHostToDevice, b->stream);
    if (e != cudaSuccess) return NUMI_CLOTH_ECUDA;

    // one copy kernel per checkpoint move: op tables for save (state ->
    // checkpoint) and load (checkpoint -> state) of every slot
    std::vector<CopyOp> save_ops, load_ops;
    const bool checkpoints = fruits || segs > 1u;
    for (uint32_t g = 0; checkpoints && g <= segs; ++g) {
        char* slot = ckpt + g * state_total;
        for (numi_cloth* h : b->cloths)
            for (const auto& r : h->dynamic) {
                save_ops.push_back(CopyOp{r.ptr, slot, r.bytes});
                load_ops.push_back(CopyOp{slot, r.ptr, r.bytes});
                slot += (r.bytes + 255u) & ~size_t(255u);
            }
    }
    if (checkpoints) e = cudaMemcpyAsync(d_ops, save_ops.data(), save_ops.size() * sizeof(CopyOp), cudaMemcpyHostToDevice, b->stream);
    if (checkpoints && e == cudaSuccess)
        e = cudaMemcpyAsync(d_ops + save_ops.size(), load_ops.data(), load_ops.size() * sizeof(CopyOp),
                            cudaMemcpyHostToDevice, b->stream);
    if (e != cudaSuccess) return NUMI_CLOTH_ECUDA;
    auto move = [&](bool save, uint32_t g) {
        const CopyOp* ops = d_ops + (save ? 0u : save_ops.size()) + static_cast<size_t>(g) * regions;
        numi_cloth_copy_kernel<<<regions, 256, 0, b->stream>>>(ops);
    };
    auto set_epoch = [&](uint32_t value) {
        return cudaMemcpyAsync(b->epoch, &value, sizeof(uint32_t), cudaMemcpyHostToDevice, b->stream) == cudaSuccess &&
               cudaStreamSynchronize(b->stream) == cudaSuccess;
    };

    // one segment of every cloth, taped (from tape_first on) or not
    auto step = [&](uint32_t g, bool taped, uint32_t tape_first) {
        const uint32_t first = g * seg;
        Schedule st = s;
        st.substeps = std::min(seg, substeps - first);
        st.cfg_offset = first;
        st.epoch_ptr = b->epoch;
        st.tape_first = tape_first;
        return batch_kernel(b, taped ? d_replay : b->d_cloths, st, true) == cudaSuccess;
    };
    // forward: taped where the tape holds it, else checkpointed (the last
    // segment of cloths without fruits is taped as it runs)
    const uint32_t epoch0 = b->epoch_host;
    if (!set_epoch(epoch0)) return NUMI_CLOTH_ECUDA;
    auto last_taped = [&](uint32_t g) { return whole || (!fruits && g + 1u == segs); };
    for (uint32_t g = 0; g < segs; ++g) {
        if (fruits || g + 1u < segs) move(true, g);
        if (!step(g, last_taped(g), whole ? g * seg : 0u)) return NUMI_CLOTH_ECUDA;
        numi_cloth_epoch_kernel<<<1, 1, 0, b->stream>>>(b->epoch, std::min(seg, substeps - g * seg));
    }
    if (checkpoints) move(true, segs);
    if (fruits && whole) {
        uint32_t touched = 0u;
        if (cudaMemcpyAsync(&touched, d_touched, sizeof(touched), cudaMemcpyDeviceToHost, b->stream) != cudaSuccess ||
            cudaStreamSynchronize(b->stream) != cudaSuccess) {
            for (numi_cloth* h : b->cloths) h->poisoned = true;
            return NUMI_CLOTH_ECUDA;
        }
        b->rollout_touched = touched != 0u;
        if (touched != 0u) whole = false;
    }
    // backward: reverse the tape, or segment by segment after a taped replay
    // from its checkpoint
    bool replayed = false;
    for (uint32_t g = whole ? 1u : segs; g-- > 0u;) {
        const uint32_t first = g * seg;
        const uint32_t cnt = whole ? substeps : std::min(seg, substeps - first);
        if (!last_taped(g)) {
            replayed = true;
            move(false, g);
            if (!set_epoch(epoch0 + first) || !step(g, true, 0u)) return NUMI_CLOTH_ECUDA;
        }
        for (uint32_t k = 0; k < count; ++k) {
            args[k].cfg = b->d_cfg + static_cast<size_t>(k) * substeps + first;
            args[k].substeps = cnt;
            args[k].first_substep = first;
        }
        e = cudaMemcpyAsync(d_args, args.data(), count * sizeof(AdjointArgs), cudaMemcpyHostToDevice, b->stream);
        if (e != cudaSuccess) return NUMI_CLOTH_ECUDA;
        if (adjoint_launch(shape, d_args, count, b->stream) != cudaSuccess) return NUMI_CLOTH_ECUDA;
        // args is rewritten next segment: wait for this copy to be consumed
        if (cudaStreamSynchronize(b->stream) != cudaSuccess) {
            for (numi_cloth* h : b->cloths) h->poisoned = true;
            return NUMI_CLOTH_ECUDA;
        }
    }
    if (replayed) move(false, segs);
    const uint32_t end_epoch = epoch0 + substeps;
    if (!set_epoch(end_epoch)) return NUMI_CLOTH_ECUDA;
    b->epoch_host = end_epoch;
    for (numi_cloth* h : b->cloths) {
        h->epoch = end_epoch;
        h->last_substeps = substeps;
    }
    std::vector<double> out(static_cast<size_t>(count) * (NUMI_CLOTH_MAX_GROUPS + 2u));
    std::vector<unsigned int> rough(count);
    uint32_t touched = 0u;
    e = cudaMemcpyAsync(&touched, d_touched, sizeof(touched), cudaMemcpyDeviceToHost, b->stream);
    if (e != cudaSuccess) return NUMI_CLOTH_ECUDA;
    e = cudaMemcpyAsync(out.data(), d_out, out.size() * sizeof(double), cudaMemcpyDeviceToHost, b->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(rough.data(), d_rough, count * sizeof(unsigned int), cudaMemcpyDeviceToHost, b->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(b->stream);
    if (e != cudaSuccess) {
        for (numi_cloth* h : b->cloths) h->poisoned = true;
        return NUMI_CLOTH_ECUDA;
    }
    b->rollout_touched = touched != 0u;   // (replays see the forward's contacts too)
    for (uint32_t k = 0; k < count; ++k) {
        const double* o = out.data() + static_cast<size_t>(k) * (NUMI_CLOTH_MAX_GROUPS + 2u);
        for (uint32_t q = 0; q <= NUMI_CLOTH_MAX_GROUPS; ++q) grads[static_cast<size_t>(k) * (NUMI_CLOTH_MAX_GROUPS + 1u) + q] = o[q];
        loss[k] = o[NUMI_CLOTH_MAX_GROUPS + 1u];
        if (groups_out) groups_out[k] = static_cast<uint32_t>(groups[k].value.size());
        if (nonsmooth) nonsmooth[k] = rough[k];
    }
    return NUMI_CLOTH_OK;
}
