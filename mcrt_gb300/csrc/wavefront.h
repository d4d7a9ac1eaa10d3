// Wavefront state shared by the render entry points (kernels.cu, noalloc.cu): the control
// block, the SoA layout of the queues, and the host helpers that lay it out and enqueue
// iterations of stage kernels.
//
// Path state travels with its ray through the queues (no per-path slots): every stage
// reads and writes its items by queue position, so all per-path traffic is coalesced.
// One iteration (parity p = iteration & 1):
//   k_admit, k_start    admit new paths and start their camera rays: the queue is topped up to
//                 its capacity from the path counter, bounded by the admission limit.  Only
//                 while paths wait to be admitted: a render whose paths fit one queue, and a
//                 wave, admit all of them before their first iteration
//   k_extend      closest hit of every ray of queue p
//   k_shade       one vertex per ray: continuing paths to queue p ^ 1, ended paths to
//                 the finished list p ^ 1, next-event rays to the next-event queues
//   k_shadow, k_connect   trace the next-event rays (environment, area lights); each result
//                 goes to the slot its path will read next (queue p ^ 1 position or
//                 finished-list position)
//   k_finish      finish the paths that ended: radiance into the ring, pixel resolved in
//                 sample order when its last path finished
// The last two need only what k_shade wrote, and nothing before the next iteration's k_shade
// needs them: mcrt_render runs them on a second stream beside the next iteration's k_extend
// (IterStreams).  Counters are kept per parity and cleared by the next kernel that may.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <string>

#include "../../include/mcrt_gb300.h"
#include "layout.h"

namespace mcrt {

constexpr int kTraceBlock = 128;
constexpr int kStack = 64;
// the smaller traversal stack, used when the tree is shallow enough (MCRT_VARIANT_STACK32)
constexpr int kSmallStack = 32;
// Blocks of kTraceBlock threads per SM that the traversal kernels' registers are capped for
// under MCRT_VARIANT_REGCAP.  Outdoor frame (1.3 M triangles, 67 M paths), extension /
// next-event ms: extension rays at 9 blocks (56 registers) 38.9, at 8 (64, no spills) 37.7,
// at 7 39.9; next-event rays to the environment at 12 (40 registers, spills) 27.6, at 10 (48)
// 23.3, at 9 23.5.  With the lanes refilled (trace_stream) more warps than this no longer help.
// Next-event rays to area lights: 7 blocks (72 registers) 0.68 ms per Cornell frame, 8 0.72.
constexpr int kTraceMinBlocks = 8;
// The adjoint's build: 9 (56 registers).  It adds each ray's emission derivative to its block's
// sums, lanes of one emitter one after the other, and more warps hide that: the gradients of a
// 512x512 Cornell box with a mirror 22.2 ms forward and adjoint, at 7 22.6.  More blocks also
// mean shorter float sums, and the sum's rounding shows in the gradient: between 7 and 9 blocks
// dL/dE differs by 2e-5 to 4e-5 relative, between runs of one build by 5e-6.
constexpr int kConnectMinBlocks = 7;
constexpr int kConnectAdjMinBlocks = 9;
constexpr int kAnyHitMinBlocks = 10;
constexpr int kMaxDepth = 62;
constexpr int64_t kMaxQueue = int64_t(1) << 27;     // rays per queue (result indices stay in int)
// Streaming schedule default: 64 M rays (45 GB of queues).  Per cfg1 frame (67 M paths):
// 0.5 / 1 / 2 / 4 / 8 / 16 / 32 / 64 M rays 172 / 124 / 99.5 / 86.6 / 81.1 / 78.8 / 77.6 /
// 78.1 ms -- fewer, longer launches amortise each launch's ramp and tail.  If its
// allocation fails the default halves itself, down to kMinDefaultQueue.
constexpr int64_t kDefaultQueue = int64_t(1) << 26;
constexpr int64_t kMinDefaultQueue = int64_t(1) << 20;

// Counters of one render.  Cleared by: k_extend of parity p lists[p ^ 1], k_shade of parity p
// the scount and fetch of p ^ 1 (each after their last reader, before their next writer, also
// with k_shadow / k_connect / k_finish beside the next k_extend).
// Every block of k_shade takes places in the ray queue and the finished list, every warp in the
// next-event queues, and waits for the old counts; the L2 answers about one atomic per ns on one
// line (with an atomic per warp and list, a million of them per 8 M rays).  So the ray queue and
// the finished list share one 64-bit counter (one atomic for both), and the counters that are not
// added to together have lines of their own: Cornell box with a mirror, 8 M rays per launch,
// k_shade 926 -> 765 and 1100 -> 910 us (first and second vertex).
struct Ctrl
{
    struct alignas(256) Count
    {
        int n[2];  // by parity
    };
    alignas(256) unsigned long long lists[2];  // by parity: ray queue (low half), finished paths (high half)
    Count              scount[2];  // next-event queues, any-hit and closest-hit
    Count              fetch[3];   // rays taken by k_extend, k_shadow, k_connect
    int                new_base;      // admitted paths to start: first queue position
    int                new_count;     //   and how many
    int                chunk;         // wave schedule: index of the current wave
    unsigned long long next;          // index of the next path to admit
    unsigned long long limit;         // admission limit (exclusive)
    unsigned long long new_g;         // index of the first path to start
    unsigned long long finished;      // paths whose radiance reached the ring
};

__host__ __device__ inline int queue_count(unsigned long long lists) { return static_cast<int>(lists & 0xffffffffu); }
__host__ __device__ inline int done_count(unsigned long long lists) { return static_cast<int>(lists >> 32); }
__host__ __device__ inline unsigned long long list_counts(int queue, int done)
{
    return static_cast<unsigned long long>(queue) | static_cast<unsigned long long>(done) << 32;
}

// device pointers of one render's state (SoA, `capacity` rays per queue)
struct WaveArgs
{
    Ctrl*          ctrl;
    const int64_t* chunk_table;  // wave schedule: wave boundaries (path indices)
    const JobGPU*  jobs;
    int            num_jobs;
    int64_t        capacity;
    // ray queues by parity.  o.w = job index, d.w = pixel index (int bits; extension rays
    // always span [kEpsRay, inf)); thr.w = flags | vertex << 8 | pending mask << 16;
    // rad.w = sample index (int bits)
    float4*   qo[2];
    float4*   qd[2];
    float4*   qthr[2];
    float4*   qrad[2];
    uint64_t* qrng[2];
    float4*   hits;  // by position of the current queue
    // finished paths by parity: radiance (w = sample), {pixel, job, pending mask, 0}
    float4* drad[2];
    int4*   dmeta[2];
    // next-event results by parity, s of 2 ^ nev_log2 slots: [(i << nev_log2) + s] for queue
    // position i, [((capacity + j) << nev_log2) + s] for finished-list position j
    float4* nev[2];
    int     nev_log2;  // 2 with both kinds of light, else 1 (set with the shading build)
    // next-event queues; tmin is kEpsRay for all.
    // [0] any-hit: origin + result index, direction + job (int bits); the value an unoccluded
    //     ray adds is already in its result slot
    // [1] closest-hit: origin + stop distance (a nearer hit ends the ray, emitter_span),
    //     direction + tmax, value, meta = {result index, type | light << 2, pixel, job}
    float4* so[2];
    float4* sd[2];
    float4* sv;
    int4*   sm;
    int64_t shadow_cap;
    // per-path radiance of path g at g % ring_size until its pixel resolves; per pixel
    // (at its first path's ring index) the count of its finished paths
    float4*             ring;
    int*                ring_cnt;
    int64_t             ring_size;
    unsigned long long* stats;  // [0] extension rays, [1] next-event rays, [2..5] work counters
    int*                err;
    // traversal kernels: each warp takes the next 32 queue entries from a counter until the
    // queue is empty (1), or every thread strides over the queue by the grid size (0)
    int batch_fetch;
    // adjoint (paths replayed through the same queues, JobGPU::image = dL/dimage): the
    // material ids of a path's parameterised Lambert vertices, 16 bits each, at most
    // kAdjLog per path (thr.w bits 20.. hold the count), two uint4 per queue position and
    // per finished-list position; gradients (in shared memory per block when grad_shared)
    uint4* qlog[2];
    uint4* dlog[2];
    float* g_albedo;
    float* g_emis;
    int    n_albedo;
    int    n_emis;
    int    grad_shared;
};

constexpr int kAdjLog = 16;

struct LaunchShape
{
    int grid_trace, grid_any, grid_connect, grid_shade, grid_regen, grid_small, block;  // grid_any: k_shadow; grid_regen: k_start, k_finish
    bool fast_only = false;  // every job traverses in FAST mode: kernels built without the REF traversal
    int  lights = 3;         // light kinds of the jobs (1 environment, 2 area, 3 both): the k_shade build
};

// sub-array allocator: consecutive 256-B aligned pieces of one block
struct Carver
{
    char* p;
    void* take(size_t n)
    {
        size_t off = (reinterpret_cast<uintptr_t>(p) + 255) & ~static_cast<uintptr_t>(255);
        char*  r = reinterpret_cast<char*>(off);
        p = r + n;
        return r;
    }
};

// bytes of the queues for `capacity` rays (256-B aligned sub-arrays)
size_t queue_bytes(int64_t capacity);
// lays the queues out in [base, base + queue_bytes(capacity))
void carve_queues(WaveArgs& a, void* base, int64_t capacity);
// bytes of a ring of `entries` paths (radiance + per-pixel counts)
size_t ring_bytes(int64_t entries);
void   carve_ring(WaveArgs& a, void* base, int64_t entries);
// ring entries the streaming schedule needs: paths admitted during the lifetime of one
// path (a path is finished at most max_depth + 2 iterations after admission, at most
// `capacity` paths are admitted per iteration) plus one pixel's samples
int64_t stream_ring_entries(int64_t capacity, int max_depth, int64_t max_spp, int64_t total);
// iterations of one wave of the wave schedule (even, so every wave starts on parity 0)
int wave_iterations(int max_depth);
// persistent grid sizes from the SM count and occupancy (queries only, no allocation)
LaunchShape launch_shape();
LaunchShape launch_shape_variant(bool stack32, bool regcap, bool fast_only = false, int lights = 3);
// starts a render: zeroes the counters and sets the admission limit (`limit`; with `waves`
// nothing is admitted until the first wave's k_wave_next) -- one kernel, so it may run
// inside a stream capture; the per-pixel counts of the ring must be zero
void enqueue_render_begin(const WaveArgs& a, bool waves, int64_t limit, cudaStream_t st);
// one wave of the wave schedule with the plain kernels (no counters, 64-entry stacks)
void enqueue_wave_plain(const WaveArgs& a, int max_depth, const LaunchShape& ls, cudaStream_t st);
// Camera::Camera in float with the reference's operation order
CameraGPU make_camera(const mcrt_camera& c);
// argument checks shared by the render entry points; sets the last error
int validate_job(const mcrt_scene* s, const mcrt_camera* c, const mcrt_render_params* p);
// Device memory of one host thread on one device, kept for the thread's life: small requests of
// calls that return only when their work is done (host-buffer traces, film sums) pay no
// cudaMalloc / cudaFree (which synchronises the device).  Null when `bytes` is over the limit
// or the device index past the table (allocate instead), or when its allocation failed.
constexpr size_t kThreadScratchMax = size_t(1) << 20;
void* thread_scratch(int device, size_t bytes, bool& failed);
// records the calling thread's last error message and returns `code`
int set_error(int code, const std::string& msg);
// read-only facts about a scene handle
const SceneView& scene_view(const mcrt_scene* s);
int              scene_device(const mcrt_scene* s);
int              scene_stack_depth(const mcrt_scene* s, int traverse);  // see the stack checks

}  // namespace mcrt
