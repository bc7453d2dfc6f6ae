// Persistent tracker with its paths in shared memory: the slots of a CTA hold the state of its
// paths, and work queues (rings of slot numbers) say what each needs next: a segment to track,
// a collision (roulette, light sample, shadow segment), the end of a shadow segment (NEE
// contribution, phase sample, next segment), or the end of a path (accumulation, next work item,
// camera ray). A warp takes up to 32 slots of one kind at a time. Scenes with triangle meshes have
// two more kinds: a vertex on a triangle and the end of its shadow segment. Whichever batch starts a
// segment there, all its lanes search the closest hit (and test the light's visibility) together.
//
// * Events: one kind per batch, so that the long event code (environment sampling, phase function,
//   camera ray, segment set-up) runs with nearly full warps. The segments that a batch starts are
//   tracked by the same warp at once.
// * Tracking: each lane advances its segment by free-flight draws and density lookups (delta
//   tracking of primary segments, ratio tracking of shadow segments); lanes whose segment ended are
//   handed to the event queues and filled with other segments kRefill at a time.
//
// What bounded the form that keeps a path in each lane was divergence: its warps ran every event
// for the few lanes that happened to have it (5.4 threads per warp instruction on the sparse
// 512^3 scene, here 13.8; 27 of 32 lanes hold work in a tracking step and 25 to 28 in an event batch
// while there is any, and diverge inside it). CTA barriers between a tracking and an event phase (17 barrier stalls per issue), one
// queue per CTA of 128 or of 768 threads, and 4 CTAs per SM at 64 registers were all slower. ms per
// launch, lane-per-path form against this one, both with the stencil copy and one seed's clouds (another
// seed's or another GPU's sparse launch takes 15.5 to 20.7): 1024^2 x 16 spp sparse 512^3 23.6 -> 16.0, 2048^2 x
// 4 spp 1024^3 17.4 -> 11.9, dense 64^3 at 256^2 x 16 spp 0.89 -> 0.74 and x 1 spp 0.53 -> 0.45,
// reference rules 256^2 x 8 spp 4.2 -> 2.9, a radiance-cache frame 4.27 -> 2.99. With meshes, 512^2 x
// 4 spp: the room 23.9 -> 6.7, with two spheres through the BVH 30.5 -> 10.2 (bound by instruction
// fetch: a third to a half of the issue slots). Of a warp's cycles, clock64 gives on the dense / sparse
// launch: tracking 32 / 62%, choosing, handing over and taking work 24 / 12%, collisions 8 / 10% (the
// sparse scene's sky has 11 mip levels), the other events 10 / 5%, loading segments 8 / 6%, idle 10-18
// / 4%.
//
// Each path draws its random numbers in its own order whichever lane works on it, so its samples
// are those of the other forms to the bit. The reference is the plain and radiance-cache ray-
// generation programs (renderer/gpu_kernels/optix_pathtracing_kernels.cu:31-434).
#include "vpt_ctx.h"
#include "vpt_track.cuh"

namespace vpt {
namespace {

enum : uint32_t {
    RS_DONE = 0,    // no path and no item left
    RS_TRACK,       // the segment is being tracked
    RS_VERTEX,      // primary collision: roulette, light sample, shadow segment
    RS_NEE_DONE,    // shadow segment over: NEE contribution, phase sample, next segment
    RS_ESCAPE,      // primary segment left the grid
    RS_END,         // the path ended otherwise
    RS_FETCH,       // a slot without a path
    RS_SURFACE,     // scenes with meshes: primary segment ended on a triangle
    RS_NEE_SURF,    // shadow segment of a surface vertex over
};
constexpr uint32_t kStateMask = 15u;
constexpr uint32_t kShadow = 1u << 4;      // the tracked segment is a shadow segment
constexpr uint32_t kPickSun = 1u << 5;     // the light sample is the sun
constexpr uint32_t kTrain = 1u << 6;       // the item is a training pixel
constexpr uint32_t kUnbiased = 1u << 7;    // its suffix is an unbiased one
constexpr uint32_t kTermDone = 1u << 8;    // its terminal record is written
constexpr int kSetShift = 9;               // training set (2 bits)
constexpr int kEndShift = 11;              // end code (3 bits)
constexpr uint32_t kEndMask = 7u << kEndShift;
constexpr uint32_t kHit = 1u << 14;        // the primary segment ends on a triangle
constexpr uint32_t kAtSurface = 1u << 15;  // the current vertex is on a triangle
constexpr uint32_t kItemBits = kTrain | kUnbiased | (3u << kSetShift);  // kept over the whole path

// Words of a slot. The stride is odd, so that consecutive slots lie in different banks.
enum : int {
    W_ST = 0,
    W_RNG,                 // 2 words
    W_PIXEL = W_RNG + 2,
    W_SAMPLE,              // sample of the pixel, or the RNG state index of a training pixel
    W_ORG,
    W_DIR = W_ORG + 3,
    W_DPDF = W_DIR + 3,
    W_INIT,                // luminance of the camera weight
    W_TP,                  // throughput: the three channels are equal in a medium
    W_CON,
    W_LEN = W_CON + 3,
    W_LDIR,
    W_EMI = W_LDIR + 3,    // emittance of an environment sample (the sun's is a parameter)
    W_APDF = W_EMI + 3,
    W_VIS,
    W_T,                   // segment: position, end, lookups so far
    W_T1,
    W_STEPS,
    W_DDA,                 // cell, crossings left per axis, next boundaries
    W_DDA_END = W_DDA + 7,
};
constexpr int kNrcWords = 4;      // primary spread, root of the path spread, last density, previous vertex
constexpr int kPixelWords = 9;    // per-pixel streams: sums (3 doubles), running mean
constexpr int kLogWords = 2;      // primary and shadow lookups of the sample
// Scenes with meshes: throughput g and b, the segment's triangle and its barycentrics, the shadow
// ray's origin, the light-side cosine over the distance and the squared distance of its sample.
constexpr int kSurfaceWords = 10;
constexpr int queue_words(bool grid_majorant, bool log, bool nrc, bool per_pixel, bool surfaces) {
    return ((grid_majorant ? W_DDA_END : W_DDA) + (nrc ? kNrcWords : 0) + (per_pixel ? kPixelWords : 0) +
            (log ? kLogWords : 0) + (surfaces ? kSurfaceWords : 0)) | 1;
}

// Slots of a CTA: half as many again as lanes, so that work waits in the queues for full batches
// (a quarter more: sparse 512^3 16.0 -> 16.7 ms; twice as many do not leave room for the L1).
// Scenes with meshes have more kinds of work and fewer CTAs: three quarters more (room / with spheres
// through the BVH, ms per 4 spp at 512^2: a half 6.9 / 10.25, three quarters 6.7 / 10.15).
__host__ __device__ constexpr uint32_t queue_slots(uint32_t threads, bool surfaces) {
    return threads + (surfaces ? threads * 3 / 4 : threads / 2);
}
__host__ __device__ constexpr uint32_t queue_ring(uint32_t threads) {
    uint32_t n = 64;
    while (n < queue_slots(threads, true)) n *= 2;
    return n;
}
// Tuned together on the sparse 512^3 launch / the radiance-cache frame (ms): cells per step 1 / 2 /
// 3 / 4 -> 17.4 / 16.3 / 16.2 / 16.7 and 3.46 / 3.25 / 3.21 / 3.21; refill at 4 / 8 / 12 / 16 / 20
// idle lanes -> 17.2 / 16.3 / 16.0 / 16.2 / 16.7 and 3.30 / 3.25 / 3.23 / 3.16 / 3.12; event batch 24
// / 32 / 48 / 64 / 96 -> 16.5 / 16.3 / 16.2 / 16.5 / 18.7 and 3.34 / 3.25 / 3.06 / 3.05 / 3.13.
constexpr int kCellSteps = 3;               // majorant cells a tracking step crosses at most
constexpr uint32_t kEventBatch = 48;        // slots of one event kind that call a tracking warp away
constexpr int kRefill = 14;                 // idle lanes of a tracking warp that are filled together

// Work queues of a CTA: rings of slots per kind of work.
enum : uint32_t { Q_VERTEX = 0, Q_NEE_DONE, Q_END, Q_TRACK, Q_SURFACE, Q_NEE_SURF };
constexpr uint32_t queue_count(bool surfaces) { return surfaces ? 6u : 4u; }
constexpr uint32_t kEmpty = 0xffffu;
constexpr uint32_t kSpinLimit = 1u << 20;   // polls of a ring entry before the CTA gives up
constexpr uint32_t kIdleSleep = 400;        // ns between polls without work
constexpr uint32_t kIdleLimit = 1u << 22;   // such polls before a warp leaves the rest to the others

// Orders the slots' words and the ring entries between the warps of a CTA.
__device__ __forceinline__ void fence_cta() { asm volatile("fence.acq_rel.cta;" ::: "memory"); }

template <bool kGridMajorant, bool kLog, int kMode, int kStreams, bool kStencil, bool kSurfaces>
__global__ void __launch_bounds__(kQueueThreads, kSurfaces ? kQueueMeshCtasPerSm : kQueueCtasPerSm) queue_trace_kernel(const __grid_constant__ TraceParams P) {
    constexpr uint32_t kQueues = queue_count(kSurfaces);
    constexpr bool kNrc = kMode != kModePlain;
    constexpr bool kCombo = kMode == kModeComboNrc;
    constexpr bool kMayTrain = kMode == kModeTrainNrc || kCombo;
    constexpr bool kMayPerPixel = !kNrc && kStreams == kStreamsPerPixel;
    constexpr int kW = queue_words(kGridMajorant, kLog, kNrc, kMayPerPixel, kSurfaces);
    constexpr int kBase = kGridMajorant ? W_DDA_END : W_DDA;
    constexpr int W_PSPREAD = kBase, W_SSPREAD = kBase + 1, W_LDENS = kBase + 2, W_PREV = kBase + 3;
    constexpr int W_SUM = kBase, W_MEAN = kBase + 6;
    constexpr int W_REC = kBase + (kNrc ? kNrcWords : 0) + (kMayPerPixel ? kPixelWords : 0);
    constexpr int W_TPGB = W_REC + (kLog ? kLogWords : 0), W_HIT = W_TPGB + 2, W_EYE = W_HIT + 3, W_LPCOS = W_EYE + 3;
    constexpr uint32_t kKept = kItemBits | kPickSun | (kSurfaces ? kHit | kAtSurface : 0u);  // bits a segment's end leaves
    const bool sample_parallel = kStreams == kStreamsRuntime ? P.stream_mode == 1 : kStreams == kStreamsSampleParallel;

    extern __shared__ __align__(16) uint32_t s_mem[];
    const uint32_t slots = queue_slots(blockDim.x, kSurfaces), ring = queue_ring(blockDim.x);
    uint32_t* const s_queue = s_mem;                 // per queue: tail << 16 | head
    uint32_t* const s_live = s_mem + kQueues;        // slots with a path or an item to fetch
    uint32_t* const s_abort = s_mem + kQueues + 1;
    uint32_t* const s_slots = s_mem + 8;
    volatile uint16_t* const s_ring = reinterpret_cast<volatile uint16_t*>(s_slots + slots * kW);
    float* const s_maj = reinterpret_cast<float*>(s_slots + slots * kW + kQueues * ring / 2);

    const Grid& g = P.grid;
    const float* maj_grid = g.maj;
    if constexpr (kGridMajorant) {
        if (P.maj_in_smem) {
            const int cells = g.mx * g.my * g.mz;
            for (int i = threadIdx.x; i < cells; i += blockDim.x) s_maj[i] = g.maj[i];
            maj_grid = s_maj;
        }
    }
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t num_pixels = static_cast<uint32_t>(P.width) * static_cast<uint32_t>(P.height);
    const float global_maj = P.density_coeff * g.global_majorant;
    const uint32_t step_cap = P.max_steps > 0 ? static_cast<uint32_t>(P.max_steps) : kHardStepCap;
    const V3 bmin = v3(g.bbox_min[0], g.bbox_min[1], g.bbox_min[2]);
    const V3 bmax = v3(g.bbox_max[0], g.bbox_max[1], g.bbox_max[2]);
    const float trace_len = 2 * P.world_radius;
    // Radiance queries locate positions in the world box, the volume's box unless there are meshes.
    const V3 wmin = kSurfaces ? v3(P.world_min[0], P.world_min[1], P.world_min[2]) : bmin;
    const V3 wmax = kSurfaces ? v3(P.world_max[0], P.world_max[1], P.world_max[2]) : bmax;
    uint32_t n_lookups = 0, n_vertices = 0, n_samples = 0, n_cells = 0;
    unsigned int err = 0;

    // Training images of the radiance-cache passes (adaptive sizes prepared on the device).
    auto set_buf = [&](uint32_t k) -> uint32_t { return (P.train_bufs >> k) & 1u; };
    auto set_w = [&](uint32_t k) -> uint32_t {
        if constexpr (kCombo)
            return min(P.train_sets[k].counters[2 + 2 * set_buf(k)], static_cast<uint32_t>(P.width));
        else
            return min(P.nrc.counters[2 + 2 * P.nrc_buf], static_cast<uint32_t>(P.width));
    };
    auto set_h = [&](uint32_t k) -> uint32_t {
        if constexpr (kCombo)
            return min(P.train_sets[k].counters[3 + 2 * set_buf(k)], static_cast<uint32_t>(P.height));
        else
            return min(P.nrc.counters[3 + 2 * P.nrc_buf], static_cast<uint32_t>(P.height));
    };
    uint32_t num_train = 0;
    if constexpr (kMayTrain) {
        const uint32_t sets = kCombo ? P.num_train_sets : 1u;
        for (uint32_t k = 0; k < sets; ++k) num_train += min(set_w(k) * set_h(k), num_pixels);
    }
    auto tr_set = [&](uint32_t st) -> uint32_t { return (st >> kSetShift) & 3u; };
    auto tr_counters = [&](uint32_t st) -> uint32_t* {
        if constexpr (kCombo) return P.train_sets[tr_set(st)].counters;
        else return P.nrc.counters;
    };
    auto tr_buf = [&](uint32_t st) -> uint32_t {
        if constexpr (kCombo) return set_buf(tr_set(st));
        else return P.nrc_buf;
    };
    auto tr_vertex = [&](uint32_t st) -> TrainVertexInfo* {
        if constexpr (kCombo) return P.train_sets[tr_set(st)].vertex;
        else return P.nrc.train_vertex;
    };
    auto tr_query0 = [&](uint32_t st) -> float* {
        if constexpr (kCombo) return P.train_sets[tr_set(st)].query0;
        else return P.nrc.train_query[0];
    };
    auto tr_target0 = [&](uint32_t st) -> float* {
        if constexpr (kCombo) return P.train_sets[tr_set(st)].target0;
        else return P.nrc.train_target[0];
    };
    auto tr_end_query = [&](uint32_t st) -> float* {
        if constexpr (kCombo) return P.train_sets[tr_set(st)].end_query;
        else return P.nrc.train_end_query;
    };
    auto tr_suffix = [&](uint32_t st) -> uint32_t* {
        if constexpr (kCombo) return P.train_sets[tr_set(st)].suffix;
        else return P.nrc.train_suffix;
    };
    const float term_factor = P.nrc_termination > 0 ? P.nrc_termination : kPathTerminationFactor;
    const float train_term_factor = P.nrc_train_termination > 0 ? P.nrc_train_termination : 2 * term_factor;

    uint64_t num_items = num_pixels;
    if constexpr (kMode == kModeTrainNrc) {
        num_items = num_train;
    } else {
        if (sample_parallel) num_items = static_cast<uint64_t>(num_pixels) * P.spp;
        if constexpr (kCombo) num_items += num_train;
    }

    auto slot_ptr = [&](uint32_t slot) -> uint32_t* { return s_slots + slot * kW; };
    auto ldf = [](const uint32_t* q, int w) -> float { return __uint_as_float(q[w]); };
    auto stf = [](uint32_t* q, int w, float v) { q[w] = __float_as_uint(v); };
    auto ld3 = [](const uint32_t* q, int w) -> V3 {
        return v3(__uint_as_float(q[w]), __uint_as_float(q[w + 1]), __uint_as_float(q[w + 2]));
    };
    auto st3 = [](uint32_t* q, int w, V3 v) {
        q[w] = __float_as_uint(v.x);
        q[w + 1] = __float_as_uint(v.y);
        q[w + 2] = __float_as_uint(v.z);
    };
    auto ld_rng = [](const uint32_t* q) -> Pcg32 {
        return Pcg32{static_cast<uint64_t>(q[W_RNG]) | (static_cast<uint64_t>(q[W_RNG + 1]) << 32)};
    };
    auto st_rng = [](uint32_t* q, const Pcg32& r) {
        q[W_RNG] = static_cast<uint32_t>(r.state);
        q[W_RNG + 1] = static_cast<uint32_t>(r.state >> 32);
    };
    // The three channels of a throughput are equal in a medium; meshes have coloured ones.
    auto ld_tp = [&](const uint32_t* q) -> RGB {
        const float r = __uint_as_float(q[W_TP]);
        if constexpr (kSurfaces) return rgb(r, __uint_as_float(q[W_TPGB]), __uint_as_float(q[W_TPGB + 1]));
        return rgb(r, r, r);
    };
    auto st_tp = [&](uint32_t* q, RGB tp) {
        q[W_TP] = __float_as_uint(tp.r);
        if constexpr (kSurfaces) {
            q[W_TPGB] = __float_as_uint(tp.g);
            q[W_TPGB + 1] = __float_as_uint(tp.b);
        }
    };
    auto nee_state = [&](uint32_t st) -> uint32_t {
        return kSurfaces && (st & kAtSurface) ? RS_NEE_SURF : RS_NEE_DONE;
    };
    auto is_train = [&](uint32_t st) -> bool { return kMode == kModeTrainNrc || (kCombo && (st & kTrain)); };
    // Record index of an item in the pass buffers.
    auto record_of = [&](const uint32_t* q, uint32_t st) -> uint32_t {
        if (is_train(st) || !sample_parallel) return q[W_PIXEL];
        return q[W_SAMPLE] * num_pixels + q[W_PIXEL];
    };

    // The path ends at a vertex whose cache query was just written (optix_pathtracing_kernels.cu
    // :307-330): the training suffix's terminal record, or the render path's terminal info and,
    // when the render queries are listed, its record in the inference list.
    auto end_with_query = [&](const uint32_t* q, uint32_t s, uint32_t rec, uint32_t path_length, RGB tp) {
        if (is_train(s)) {
            tr_suffix(s)[rec] = pack_suffix(q[W_PREV], 1, path_length, s & kUnbiased ? 1 : 0);
            return;
        }
        TerminalInfo ti;
        ti.tp[0] = tp.r;
        ti.tp[1] = tp.g;
        ti.tp[2] = tp.b;
        ti.bits = 1u | ((path_length & 0xFFu) << 1);
        P.nrc.infer_terminal[rec] = ti;
        if (P.nrc.infer_index) {
            // One atomic per converged group.
            const uint32_t m = __activemask();
            const int leader = __ffs(m) - 1;
            uint32_t base = 0;
            if (static_cast<int>(lane) == leader) base = atomicAdd(P.nrc.counters + 8, __popc(m));
            base = __shfl_sync(m, base, leader);
            P.nrc.infer_index[base + __popc(m & ((1u << lane) - 1u))] = rec;
        }
    };

    // Segment set-up at the clip box: false when the ray misses it.
    auto start_segment = [&](uint32_t* q, V3 eye, V3 dir, float tmax) -> bool {
        float a, b;
        if (!clip_ray(bmin, bmax, eye, dir, 0.0f, tmax, &a, &b)) return false;
        const float t = fmaxf(0.0f, a);
        stf(q, W_T, t);
        stf(q, W_T1, b);
        q[W_STEPS] = 0;
        if constexpr (kGridMajorant) {
            DdaState dda;
            dda_init(g, eye, dir, t, &dda);
            const int cdim[3] = {g.mx, g.my, g.mz};
            q[W_DDA] = static_cast<uint32_t>((dda.cell[0] * g.my + dda.cell[1]) * g.mz + dda.cell[2]);
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                q[W_DDA + 1 + i] = static_cast<uint32_t>(dda.step[i] > 0 ? cdim[i] - 1 - dda.cell[i] : dda.cell[i]);
                stf(q, W_DDA + 4 + i, dda.tnext[i]);
            }
        }
        return true;
    };

    // ---------------------------------------------------------------- work queues
    // Entries are published with the state of their slot: the producer fences its stores, reserves
    // ring positions with one atomic per warp and writes the slots; a consumer claims positions and
    // takes each entry once it is there (the wait for an entry being written is bounded).
    auto push_states = [&](bool pred, uint32_t slot, uint32_t st) {
        const uint32_t s = st & kStateMask;
        uint32_t queue = s == RS_TRACK ? Q_TRACK : (s == RS_VERTEX ? Q_VERTEX : (s == RS_NEE_DONE ? Q_NEE_DONE : Q_END));
        if constexpr (kSurfaces) queue = s == RS_SURFACE ? Q_SURFACE : (s == RS_NEE_SURF ? Q_NEE_SURF : queue);
        fence_cta();
        // Lane k reserves the positions of queue k; lane kQueues takes ended slots off the live count.
        const bool put = pred && s != RS_DONE;
        uint32_t mine = 0, add = 0;
        // (Rolled in the larger kernels, which wait for instructions: spheres 11.2 -> 10.25 ms, cache
        // frame 2.82 -> 2.79; the plain volume kernels are 1-2% faster unrolled.)
#pragma unroll (kSurfaces || kNrc ? 1 : 4)
        for (uint32_t k = 0; k < kQueues; ++k) {
            const uint32_t m = __ballot_sync(0xffffffffu, put && queue == k);
            if (queue == k) mine = m;
            if (lane == k) add = static_cast<uint32_t>(__popc(m)) << 16;
        }
        const uint32_t done = __ballot_sync(0xffffffffu, pred && s == RS_DONE);
        if (lane == kQueues) add = 0u - static_cast<uint32_t>(__popc(done));
        uint32_t base = 0;
        if (add) base = atomicAdd(s_mem + lane, add) >> 16;
        base = __shfl_sync(0xffffffffu, base, queue);
        if (put) {
            volatile uint16_t* e = s_ring + queue * ring + ((base + __popc(mine & ((1u << lane) - 1u))) & (ring - 1));
            uint32_t spin = 0;
            while (*e != kEmpty && ++spin < kSpinLimit) {}
            if (spin >= kSpinLimit) *s_abort = 1;
            *e = static_cast<uint16_t>(slot);
        }
    };
    // Up to popc(want) slots of a queue, one to each lane in `want`; kEmpty where there is none.
    auto pop = [&](uint32_t queue, uint32_t want) -> uint32_t {
        uint32_t head = 0, n = 0;
        if (lane == 0) {
            const uint32_t most = __popc(want);
            uint32_t w = *static_cast<volatile uint32_t*>(s_queue + queue);
            for (int tries = 0; tries < 64; ++tries) {
                n = min(((w >> 16) - w) & 0xffffu, most);
                if (n == 0) break;
                head = w & 0xffffu;
                const uint32_t old = atomicCAS(s_queue + queue, w, (w & 0xffff0000u) | ((w + n) & 0xffffu));
                if (old == w) break;
                w = old;
                n = 0;
            }
        }
        head = __shfl_sync(0xffffffffu, head, 0);
        n = __shfl_sync(0xffffffffu, n, 0);
        const uint32_t rank = __popc(want & ((1u << lane) - 1u));
        uint32_t slot = kEmpty;
        if (((want >> lane) & 1u) && rank < n) {
            volatile uint16_t* e = s_ring + queue * ring + ((head + rank) & (ring - 1));
            uint32_t spin = 0;
            while ((slot = *e) == kEmpty && ++spin < kSpinLimit) {}
            if (slot == kEmpty) *s_abort = 1;
            *e = static_cast<uint16_t>(kEmpty);
        }
        fence_cta();
        __syncwarp();
        return slot;
    };
    auto count_of = [](uint32_t w) -> uint32_t { return ((w >> 16) - w) & 0xffffu; };

    // Slots start without a path. A launch with fewer items than slots spreads them over the CTAs.
    {
        const uint64_t quota = (num_items + gridDim.x - 1) / gridDim.x;
        const uint32_t live = quota < slots ? static_cast<uint32_t>(quota) : slots;
        for (uint32_t i = threadIdx.x; i < kQueues * ring; i += blockDim.x) s_ring[i] = kEmpty;
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < live; i += blockDim.x) {
            slot_ptr(i)[W_ST] = RS_FETCH;
            s_ring[Q_END * ring + i] = static_cast<uint16_t>(i);
        }
        if (threadIdx.x < kQueues) s_queue[threadIdx.x] = threadIdx.x == Q_END ? live << 16 : 0u;
        if (threadIdx.x == 0) {
            *s_live = live;
            *s_abort = 0;
        }
    }
    __syncthreads();

    // The warp's lanes hold the segments they track (slot, act) from one turn to the next; `give`
    // marks the lanes whose slot goes back to the queues with the state `st`.
    uint32_t idle = 0, slot = kEmpty, st = 0, next = 0, steps = 0, steps0 = 0;
    bool act = false, give = false;
    Pcg32 rng{0};
    float t = 0, t1 = 0, vis = 0, maj = global_maj, texit = 0.0f, last = 0.0f;
    V3 dir = v3(0, 0, 1), eye = v3(0, 0, 0);
    int lin = 0, rem0 = 0, rem1 = 0, rem2 = 0;
    float tn0 = 0, tn1 = 0, tn2 = 0, td0 = 0, td1 = 0, td2 = 0;
    LeafCache leaf_cache;
    while (true) {
        if (__any_sync(0xffffffffu, give)) {
            push_states(give, slot, st);
            if (give) slot = kEmpty;
            give = false;
        }
        // Full event batches first, then tracking, then what there is.
        const uint32_t active = __ballot_sync(0xffffffffu, act);
        const volatile uint32_t* sv = s_mem;
        uint32_t w0, w1, w2, w3, w4, w5, w6, w7;  // the queues, then the live count and the abort flag
        asm volatile("ld.volatile.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(w0), "=r"(w1), "=r"(w2), "=r"(w3)
                     : "r"(smem_addr32(s_mem)));
        asm volatile("ld.volatile.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(w4), "=r"(w5), "=r"(w6), "=r"(w7)
                     : "r"(smem_addr32(s_mem + 4)));
        const uint32_t c0 = count_of(w0), c1 = count_of(w1), c2 = count_of(w2), c3 = count_of(w3);
        uint32_t most = max(c0, max(c1, c2));
        uint32_t kind = c0 == most ? 0u : (c1 == most ? 1u : 2u);
        if constexpr (kSurfaces) {
            const uint32_t c4 = count_of(w4), c5 = count_of(w5);
            if (max(c4, c5) > most) {
                kind = c4 >= c5 ? Q_SURFACE : Q_NEE_SURF;
                most = max(c4, c5);
            }
        }
        if (active || (most < kEventBatch && c3 > 0 && (c3 >= 32 || c3 >= most))) kind = Q_TRACK;
        if ((kSurfaces ? w6 : w4) == 0 || (kSurfaces ? w7 : w5) != 0) kind = kQueues;
        kind = __shfl_sync(0xffffffffu, kind, 0);
        if (kind == kQueues) break;
        uint32_t got = pop(kind, ~active);
        if (!(active | __ballot_sync(0xffffffffu, got != kEmpty))) {
            if (++idle > kIdleLimit) break;  // the other warps go on
            __nanosleep(kIdleSleep);
            continue;
        }
        idle = 0;
        if (kind != Q_TRACK) {
            slot = got;
            // The segment that the event starts: its eye, direction and length, and the state
            // that follows when it misses the box.
            bool segment = false;
            V3 seg_eye = v3(0, 0, 0), seg_dir = v3(0, 0, 1);
            float seg_max = 1e10f;
            bool light = false;  // scenes with meshes: a light sample for the vertex at seg_eye
            Pcg32 rng{0};
            st = RS_DONE;
            if (kind == Q_VERTEX) {
                // Primary collision (optix_pathtracing_kernels.cu:176-182, 254-268, 282-332) and
                // light sample (renderer_kernel_common.h:297-358).
                if (slot != kEmpty) {
                    uint32_t* q = slot_ptr(slot);
                    uint32_t s = q[W_ST] & kItemBits;
                    rng = ld_rng(q);
                    const V3 seg_origin = ld3(q, W_ORG), dir = ld3(q, W_DIR);
                    const V3 origin = seg_origin + ldf(q, W_T) * dir;
                    st3(q, W_ORG, origin);
                    const uint32_t path_length = q[W_LEN];
                    RGB tp = ld_tp(q);
                    float primary_spread = 0.0f, sqrt_spread = 0.0f;
                    if constexpr (kNrc) {
                        primary_spread = ldf(q, W_PSPREAD);
                        sqrt_spread = ldf(q, W_SSPREAD);
                        V3 dv = seg_origin - origin;
                        float dist2 = dv.x * dv.x + dv.y * dv.y + dv.z * dv.z;
                        if (path_length == 1) {
                            primary_spread = dist2 / (4 * kPi * 1.0f);
                            stf(q, W_PSPREAD, primary_spread);
                        } else {
                            sqrt_spread += sqrtf(dist2 / (ldf(q, W_DPDF) * 1.0f));
                            stf(q, W_SSPREAD, sqrt_spread);
                        }
                    }
                    float continue_prob = 1.0f;
                    bool rr_kill = false;
                    const int32_t rr_from = is_train(s) ? max(P.rr_start, 3) : P.rr_start;
                    if (static_cast<int32_t>(path_length) >= rr_from) {
                        continue_prob = fminf(luminance(tp) / ldf(q, W_INIT), 1.0f);
                        if (rng.uniform() >= continue_prob) rr_kill = true;
                    }
                    bool over = false;
                    if constexpr (!kNrc) {
                        if (rr_kill) {
                            s |= RS_END | (END_RR << kEndShift);
                            over = true;
                        }
                    } else {
                        bool ends_with_cache = rr_kill;
                        const float spread2 = sqrt_spread * sqrt_spread;
                        if (is_train(s)) {
                            if (!(s & kUnbiased)) ends_with_cache |= spread2 > train_term_factor * primary_spread;
                        } else {
                            ends_with_cache |= spread2 > term_factor * primary_spread;
                        }
                        if (ends_with_cache) {
                            const float rough =
                                P.nrc_density_query && P.density_coeff > 0 ? ldf(q, W_LDENS) / P.density_coeff : 0.0f;
                            const uint32_t rec = record_of(q, s);
                            float* qdst = is_train(s) ? tr_end_query(s) : P.nrc.infer_query;
                            write_query(qdst + kQueryFloats * static_cast<size_t>(rec), origin, -dir, rough, P.albedo, wmin,
                                        wmax);
                            end_with_query(q, s, rec, path_length, tp);
                            s |= RS_END | kTermDone | (END_CACHE << kEndShift);
                            over = true;
                        }
                    }
                    if (!over) {
                        tp = rdiv(tp, continue_prob);
                        st_tp(q, tp);
                    }
                    if (kSurfaces && !over) {
                        light = true;
                        seg_eye = origin;
                    } else if (!over) {
                        const float u_light = rng.uniform();
                        const float u0 = rng.uniform();
                        const float u1 = rng.uniform();
                        bool pick_sun = false;
                        float light_prob = 1.0f;
                        bool have_light = true;
                        if (P.sun.enabled && P.env_enabled) {
                            if (u_light < P.sun.select_prob) {
                                pick_sun = true;
                                light_prob = P.sun.select_prob;
                            } else {
                                light_prob = 1.0f - P.sun.select_prob;
                            }
                        } else if (P.sun.enabled) {
                            pick_sun = true;
                        } else if (!P.env_enabled) {
                            have_light = false;
                        }
                        V3 light_dir = v3(0, 1, 0);
                        if (have_light) {
                            if (pick_sun) {
                                light_dir = v3(P.sun.dir[0], P.sun.dir[1], P.sun.dir[2]);
                                stf(q, W_APDF, light_prob);
                                s |= kPickSun;
                            } else {
                                float pdf;
                                const RGB radiance = env_sample(P.env, u0, u1, &light_dir, &pdf);
                                const RGB emittance = kPi * radiance;
                                st3(q, W_EMI, v3(emittance.r, emittance.g, emittance.b));
                                if (pdf == 0.0f) have_light = false;
                                stf(q, W_APDF, pdf * light_prob);
                            }
                        }
                        if (have_light) {
                            const V3 sdir = -light_dir;
                            const float lp_cos = dot(sdir, -light_dir);
                            if (lp_cos <= 0.0f) have_light = false;
                        }
                        st3(q, W_LDIR, light_dir);
                        stf(q, W_VIS, have_light ? 1.0f : 0.0f);
                        s |= RS_NEE_DONE;
                        if (have_light) {
                            segment = true;
                            seg_eye = origin + trace_len * light_dir;
                            seg_dir = -light_dir;
                            seg_max = trace_len;
                        }
                    }
                    st_rng(q, rng);
                    st = s;
                }
            } else if (kSurfaces && kind == Q_SURFACE) {
                // A triangle hit (optix_pathtracing_kernels.cu:176-239, 254-330): the surface point, its
                // emission weighted against area-light sampling, roulette, light sample.
                if (slot != kEmpty) {
                    uint32_t* q = slot_ptr(slot);
                    uint32_t s = (q[W_ST] & kItemBits) | kAtSurface;
                    rng = ld_rng(q);
                    const SurfPoint sp = surface_point(P.surf, q[W_HIT], ldf(q, W_HIT + 1), ldf(q, W_HIT + 2), P.env_enabled != 0);
                    const V3 ray_origin = ld3(q, W_ORG), dir = ld3(q, W_DIR), origin = sp.pos;
                    st3(q, W_ORG, origin);
                    const float dir_pdf = ldf(q, W_DPDF);
                    const uint32_t path_length = q[W_LEN];
                    RGB tp = ld_tp(q);
                    const V3 vout_local = to_local(sp.sf, -dir);
                    const SurfMaterial& mt = P.surf.mats[sp.material];
                    float primary_spread = 0.0f, sqrt_spread = 0.0f;
                    if constexpr (kNrc) {
                        // :200-210: path spread, |cos| against the geometric normal.
                        primary_spread = ldf(q, W_PSPREAD);
                        sqrt_spread = ldf(q, W_SSPREAD);
                        const V3 dv = ray_origin - origin;
                        const float dist2 = dv.x * dv.x + dv.y * dv.y + dv.z * dv.z;
                        const float abs_dot = fabsf(dot(dir, sp.gn));
                        if (path_length == 1) {
                            primary_spread = dist2 / (4 * kPi * abs_dot);
                            stf(q, W_PSPREAD, primary_spread);
                        } else {
                            sqrt_spread += sqrtf(dist2 / (dir_pdf * abs_dot));
                            stf(q, W_SSPREAD, sqrt_spread);
                        }
                    }
                    if (vout_local.z > 0 && mt.emissive) {
                        const RGB em = rgb(mt.emittance[0], mt.emittance[1], mt.emittance[2]);
                        float mis = 1.0f;
                        if (path_length > 1) {
                            const V3 dv = ray_origin - origin;
                            const float dist2 = dot(dv, dv);
                            const float light_pdf = sp.hyp_area_pdf * dist2 / vout_local.z;
                            const float bsdf_pdf = dir_pdf;
                            mis = (bsdf_pdf * bsdf_pdf) / ((bsdf_pdf * bsdf_pdf) + (light_pdf * light_pdf));
                        }
                        const RGB implicit = em * (mis / kPi);
                        if (!is_train(s)) {
                            const V3 c = ld3(q, W_CON);
                            const RGB add = tp * implicit;
                            st3(q, W_CON, v3(c.x + add.r, c.y + add.g, c.z + add.b));
                        } else if (q[W_PREV] != kInvalidVertex) {
                            // :231-237: the emission completes the previous vertex's target.
                            const TrainVertexInfo& pv = tr_vertex(s)[q[W_PREV]];
                            float* tg = tr_target0(s) + 3 * static_cast<size_t>(q[W_PREV]);
                            const RGB add = rgb(pv.local_tp[0], pv.local_tp[1], pv.local_tp[2]) * implicit;
                            tg[0] += add.r;
                            tg[1] += add.g;
                            tg[2] += add.b;
                        }
                    }
                    float continue_prob = 1.0f;
                    bool rr_kill = false;
                    const int32_t rr_from = is_train(s) ? max(P.rr_start, 3) : P.rr_start;
                    if (static_cast<int32_t>(path_length) >= rr_from) {
                        continue_prob = fminf(luminance(tp) / ldf(q, W_INIT), 1.0f);
                        if (rng.uniform() >= continue_prob) rr_kill = true;
                    }
                    bool over = false;
                    if constexpr (!kNrc) {
                        if (rr_kill) {
                            s |= RS_END | (END_RR << kEndShift);
                            over = true;
                        }
                    } else {
                        // :282-330 at a surface: the query holds the shading normal and the material's
                        // reflectances and roughness.
                        bool ends_with_cache = rr_kill;
                        const float spread2 = sqrt_spread * sqrt_spread;
                        if (is_train(s)) {
                            if (!(s & kUnbiased)) ends_with_cache |= spread2 > train_term_factor * primary_spread;
                        } else {
                            ends_with_cache |= spread2 > term_factor * primary_spread;
                        }
                        if (ends_with_cache) {
                            const uint32_t rec = record_of(q, s);
                            float* qdst = is_train(s) ? tr_end_query(s) : P.nrc.infer_query;
                            write_query_surface(qdst + kQueryFloats * static_cast<size_t>(rec), origin, sp.sf.n, -dir, mt, wmin,
                                                wmax);
                            end_with_query(q, s, rec, path_length, tp);
                            s |= RS_END | kTermDone | (END_CACHE << kEndShift);
                            over = true;
                        }
                    }
                    if (!over) {
                        tp = rdiv(tp, continue_prob);
                        st_tp(q, tp);
                        light = true;
                        seg_eye = origin;
                    }
                    st_rng(q, rng);
                    st = s;
                }
            } else if (kSurfaces && kind == Q_NEE_SURF) {
                // NEE contribution with the surface's BSDF (renderer_kernel_common.h:385-402), BSDF
                // sample, offset origin of the next ray (optix_pathtracing_kernels.cu:340-409).
                if (slot != kEmpty) {
                    uint32_t* q = slot_ptr(slot);
                    const uint32_t s_in = q[W_ST];
                    uint32_t s = s_in & kItemBits;
                    rng = ld_rng(q);
                    const V3 old_dir = ld3(q, W_DIR);
                    RGB tp = ld_tp(q);
                    const SurfPoint sp = surface_point(P.surf, q[W_HIT], ldf(q, W_HIT + 1), ldf(q, W_HIT + 2), P.env_enabled != 0);
                    const SurfMaterial& mt = P.surf.mats[sp.material];
                    const Bsdf f = make_bsdf(mt);
                    const V3 vq = to_local(sp.sf, -old_dir);
                    RGB nee_value = rgb(0, 0, 0);
                    const float vis = ldf(q, W_VIS);
                    if (vis > 0.0f) {
                        const V3 light_dir = ld3(q, W_LDIR);
                        const float area_pdf = ldf(q, W_APDF);
                        const float nee_lp_cos = ldf(q, W_LPCOS), nee_dist2 = ldf(q, W_LPCOS + 1);
                        const V3 sdir = -light_dir;
                        const V3 vin = to_local(sp.sf, -sdir);
                        float bpdf0;
                        const RGB fs = bsdf_eval_pdf(f, vq, vin, &bpdf0);
                        const float sp_cos = fabsf(dot(sdir, sp.gn));
                        RGB nee;
                        if (s_in & kPickSun) {
                            const RGB emittance = rgb(P.sun.irradiance[0], P.sun.irradiance[1], P.sun.irradiance[2]);
                            nee = fs * emittance * (vis * sp_cos / area_pdf);
                        } else {
                            const V3 e = ld3(q, W_EMI);
                            const RGB emittance = rgb(e.x, e.y, e.z);
                            float bpdf = bpdf0 * nee_lp_cos / nee_dist2;
                            if (!isfinite(bpdf)) bpdf = 0.0f;
                            const float light_pdf = area_pdf;
                            const float mis = (light_pdf * light_pdf) / ((bpdf * bpdf) + (light_pdf * light_pdf));
                            const RGB le = rdiv(emittance, kPi);
                            const float gterm = nee_lp_cos * sp_cos / nee_dist2;
                            nee = fs * le * (vis * mis * gterm / area_pdf);
                        }
                        if (!is_train(s)) {
                            const V3 c = ld3(q, W_CON);
                            const RGB add = tp * nee;
                            st3(q, W_CON, v3(c.x + add.r, c.y + add.g, c.z + add.b));
                        }
                        nee_value = nee;
                    }
                    uint32_t path_length = q[W_LEN];
                    bool over = false;
                    if (P.max_bounces > 0 && static_cast<int32_t>(path_length) >= P.max_bounces) {
                        s |= RS_END | (END_MAX_BOUNCES << kEndShift);
                        over = true;
                    }
                    if (!over) {
                        const float u0 = rng.uniform();
                        const float u1 = rng.uniform();
                        V3 local;
                        float pdf;
                        const RGB fs = bsdf_sample(f, vq, u0, u1, &local, &pdf);
                        if (pdf == 0.0f) {
                            s |= RS_END | (END_PDF_ZERO << kEndShift);
                            over = true;
                        } else {
                            const V3 dir = from_local(sp.sf, local);
                            const float dot_sgn = dot(dir, sp.gn);
                            const RGB local_tp = fs * (fabsf(dot_sgn) / pdf);
                            tp = tp * local_tp;
                            st_tp(q, tp);
                            const V3 origin = offset_ray_origin(sp.pos, (dot_sgn > 0.0f ? 1.0f : -1.0f) * sp.gn);
                            st3(q, W_ORG, origin);
                            st3(q, W_DIR, dir);
                            stf(q, W_DPDF, pdf);
                            if (is_train(s)) {
                                // :358-409 at a surface vertex: the query at the surface point (not the offset
                                // origin), the BSDF's local throughput, the NEE target.
                                const uint32_t prev = q[W_PREV];
                                const uint32_t idx = atomicAdd(tr_counters(s) + tr_buf(s), 1u);
                                if (idx < kTrainBufferSize) {
                                    write_query_surface(tr_query0(s) + kQueryFloats * static_cast<size_t>(idx), sp.pos, sp.sf.n,
                                                        -old_dir, mt, wmin, wmax);
                                    TrainVertexInfo vi;
                                    vi.local_tp[0] = local_tp.r;
                                    vi.local_tp[1] = local_tp.g;
                                    vi.local_tp[2] = local_tp.b;
                                    vi.bits = (prev & kInvalidVertex) | ((path_length & 0xFFu) << 22) |
                                              ((s & kUnbiased ? 1u : 0u) << 30);
                                    tr_vertex(s)[idx] = vi;
                                    float* tg = tr_target0(s) + 3 * static_cast<size_t>(idx);
                                    tg[0] = nee_value.r;
                                    tg[1] = nee_value.g;
                                    tg[2] = nee_value.b;
                                    q[W_PREV] = idx;
                                } else {
                                    const uint32_t rec = record_of(q, s);
                                    write_query_surface(tr_end_query(s) + kQueryFloats * static_cast<size_t>(rec), sp.pos,
                                                        sp.sf.n, -old_dir, mt, wmin, wmax);
                                    tr_suffix(s)[rec] = pack_suffix(prev, 1, path_length, s & kUnbiased ? 1 : 0);
                                    err |= VPT_DEVERR_TRAIN_FULL;
                                    s |= RS_END | kTermDone | (END_TRAIN_FULL << kEndShift);
                                    over = true;
                                }
                            }
                            seg_eye = origin;
                            seg_dir = dir;
                        }
                    }
                    if (!over) {
                        ++path_length;
                        ++n_vertices;
                        q[W_LEN] = path_length;
                        s |= path_length > kHardVertexCap ? RS_END | (END_MAX_BOUNCES << kEndShift) : RS_ESCAPE;
                        segment = path_length <= kHardVertexCap;
                    }
                    st_rng(q, rng);
                    st = s;
                }
            } else if (kind == Q_NEE_DONE) {
                // NEE contribution (renderer_kernel_common.h:385-402), phase sample and next
                // segment (optix_pathtracing_kernels.cu:341-409).
                if (slot != kEmpty) {
                    uint32_t* q = slot_ptr(slot);
                    const uint32_t s_in = q[W_ST];
                    uint32_t s = s_in & kItemBits;
                    rng = ld_rng(q);
                    const V3 old_dir = ld3(q, W_DIR);
                    RGB tp = ld_tp(q);
                    RGB nee_value = rgb(0, 0, 0);
                    const float vis = ldf(q, W_VIS);
                    if (vis > 0.0f) {
                        const V3 light_dir = ld3(q, W_LDIR);
                        const float area_pdf = ldf(q, W_APDF);
                        V3 sdir = -light_dir;
                        Frame fr = make_frame(-old_dir);
                        V3 v_in_local = to_local(fr, -sdir);
                        float pf = phase_pdf(P.phase_kind, P.phase_param, v_in_local);
                        RGB fs = rgb(P.albedo, P.albedo, P.albedo) * pf;
                        RGB nee;
                        if (s_in & kPickSun) {
                            const RGB emittance = rgb(P.sun.irradiance[0], P.sun.irradiance[1], P.sun.irradiance[2]);
                            nee = fs * emittance * (vis / area_pdf);
                        } else {
                            const V3 e = ld3(q, W_EMI);
                            const RGB emittance = rgb(e.x, e.y, e.z);
                            // Scenes with meshes keep the light-side cosine over the distance and the
                            // squared distance of an area-light sample (1 for the environment).
                            float lp_cos = kSurfaces ? ldf(q, W_LPCOS) : dot(sdir, -light_dir);
                            const float dist2 = kSurfaces ? ldf(q, W_LPCOS + 1) : 1.0f;
                            float bsdf_pdf = pf * lp_cos / dist2;
                            if (!isfinite(bsdf_pdf)) bsdf_pdf = 0.0f;
                            float light_pdf = area_pdf;
                            float mis = (light_pdf * light_pdf) / ((bsdf_pdf * bsdf_pdf) + (light_pdf * light_pdf));
                            RGB le = rdiv(emittance, kPi);
                            float gterm = lp_cos * 1.0f / dist2;
                            nee = fs * le * (vis * mis * gterm / area_pdf);
                        }
                        if (!is_train(s)) {
                            const V3 c = ld3(q, W_CON);
                            const RGB add = tp * nee;
                            st3(q, W_CON, v3(c.x + add.r, c.y + add.g, c.z + add.b));
                        }
                        nee_value = nee;
                    }
                    uint32_t path_length = q[W_LEN];
                    bool over = false;
                    if (P.max_bounces > 0 && static_cast<int32_t>(path_length) >= P.max_bounces) {
                        s |= RS_END | (END_MAX_BOUNCES << kEndShift);
                        over = true;
                    }
                    V3 dir = old_dir;
                    if (!over) {
                        Frame fr = make_frame(-old_dir);
                        float u0 = rng.uniform();
                        float u1 = rng.uniform();
                        V3 local;
                        float pdf = phase_sample(P.phase_kind, P.phase_param, u0, u1, &local);
                        if (pdf == 0.0f) {
                            s |= RS_END | (END_PDF_ZERO << kEndShift);
                            over = true;
                        } else {
                            RGB fs = rgb(P.albedo, P.albedo, P.albedo) * pdf;
                            dir = from_local(fr, local);
                            RGB local_tp = fs * (fabsf(1.0f) / pdf);
                            tp = tp * local_tp;
                            st_tp(q, tp);
                            st3(q, W_DIR, dir);
                            stf(q, W_DPDF, pdf);
                            if (is_train(s)) {
                                const uint32_t prev = q[W_PREV];
                                const uint32_t idx = atomicAdd(tr_counters(s) + tr_buf(s), 1u);
                                const float rough =
                                    P.nrc_density_query && P.density_coeff > 0 ? ldf(q, W_LDENS) / P.density_coeff : 0.0f;
                                const V3 origin = ld3(q, W_ORG);
                                if (idx < kTrainBufferSize) {
                                    write_query(tr_query0(s) + kQueryFloats * static_cast<size_t>(idx), origin, -old_dir,
                                                rough, P.albedo, wmin, wmax);
                                    TrainVertexInfo vi;
                                    vi.local_tp[0] = local_tp.r;
                                    vi.local_tp[1] = local_tp.g;
                                    vi.local_tp[2] = local_tp.b;
                                    vi.bits = (prev & kInvalidVertex) | ((path_length & 0xFFu) << 22) |
                                              ((s & kUnbiased ? 1u : 0u) << 30);
                                    tr_vertex(s)[idx] = vi;
                                    float* tg = tr_target0(s) + 3 * static_cast<size_t>(idx);
                                    tg[0] = nee_value.r;
                                    tg[1] = nee_value.g;
                                    tg[2] = nee_value.b;
                                    q[W_PREV] = idx;
                                } else {
                                    const uint32_t rec = record_of(q, s);
                                    write_query(tr_end_query(s) + kQueryFloats * static_cast<size_t>(rec), origin, -old_dir,
                                                rough, P.albedo, wmin, wmax);
                                    tr_suffix(s)[rec] = pack_suffix(prev, 1, path_length, s & kUnbiased ? 1 : 0);
                                    err |= VPT_DEVERR_TRAIN_FULL;
                                    s |= RS_END | kTermDone | (END_TRAIN_FULL << kEndShift);
                                    over = true;
                                }
                            }
                        }
                    }
                    if (!over) {
                        ++path_length;
                        ++n_vertices;
                        q[W_LEN] = path_length;
                        if (path_length > kHardVertexCap)
                            s |= RS_END | (END_MAX_BOUNCES << kEndShift);
                        else
                            s |= RS_ESCAPE;
                        segment = path_length <= kHardVertexCap;
                        seg_eye = ld3(q, W_ORG);
                        seg_dir = dir;
                    }
                    st_rng(q, rng);
                    st = s;
                }
            } else {
                // End of a path (optix_pathtracing_kernels.cu:130-174, 413-432), next work item,
                // camera ray (:43-81) and first segment. A camera ray that misses the box comes back
                // here as an escaped path.
                if (slot != kEmpty) {
                    uint32_t* q = slot_ptr(slot);
                    uint32_t s = q[W_ST];
                    V3 dir = ld3(q, W_DIR);
                    do {
                        bool same_pixel = false;
                        if ((s & kStateMask) != RS_FETCH) {
                            const V3 c0 = ld3(q, W_CON);
                            RGB contribution = rgb(c0.x, c0.y, c0.z);
                            const RGB tp = ld_tp(q);
                            const uint32_t path_length = q[W_LEN];
                            uint32_t end_code = (s & kEndMask) >> kEndShift;
                            if ((s & kStateMask) == RS_ESCAPE) {
                                if (P.env_enabled) {
                                    float hyp_pdf;
                                    const RGB radiance = env_evaluate<true>(P.env, dir, &hyp_pdf);
                                    float mis = 1.0f;
                                    if (path_length > 1) {
                                        float sel = P.sun.enabled ? (1.0f - P.sun.select_prob) : 1.0f;
                                        // :140-142: with emitting triangles the environment is picked with
                                        // probToSampleEnvLight.
                                        if constexpr (kSurfaces) {
                                            if (P.surf.inst_integral > 0.0f)
                                                sel = P.sun.enabled ? kProbEnvLight * sel : kProbEnvLight;
                                        }
                                        float light_pdf = sel * hyp_pdf;
                                        float bsdf_pdf = ldf(q, W_DPDF);
                                        mis = (bsdf_pdf * bsdf_pdf) / ((bsdf_pdf * bsdf_pdf) + (light_pdf * light_pdf));
                                    }
                                    const RGB implicit = radiance * mis;
                                    if (!is_train(s)) contribution = contribution + tp * implicit;
                                    if (is_train(s)) {
                                        const uint32_t prev = q[W_PREV];
                                        if (prev != kInvalidVertex) {
                                            const TrainVertexInfo& pv = tr_vertex(s)[prev];
                                            float* tg = tr_target0(s) + 3 * static_cast<size_t>(prev);
                                            RGB add = rgb(pv.local_tp[0], pv.local_tp[1], pv.local_tp[2]) * implicit;
                                            tg[0] += add.r;
                                            tg[1] += add.g;
                                            tg[2] += add.b;
                                        }
                                    }
                                }
                                end_code = END_ESCAPE;
                            }
                            // End of the sample: non-finite contributions are dropped and flagged.
                            ++n_samples;
                            const uint32_t pixel = q[W_PIXEL];
                            if constexpr (kNrc) {
                                const uint32_t rec = record_of(q, s);
                                if (is_train(s)) {
                                    if (!(s & kTermDone))
                                        tr_suffix(s)[rec] = pack_suffix(q[W_PREV], 0, path_length, s & kUnbiased ? 1 : 0);
                                } else {
                                    if (!(s & kTermDone)) {
                                        TerminalInfo ti;
                                        ti.tp[0] = tp.r;
                                        ti.tp[1] = tp.g;
                                        ti.tp[2] = tp.b;
                                        ti.bits = (path_length & 0xFFu) << 1;
                                        P.nrc.infer_terminal[rec] = ti;
                                    }
                                    RGB c = contribution;
                                    if (!all_nonneg_finite(c)) {
                                        err |= VPT_DEVERR_NONFINITE;
                                        c = rgb(0, 0, 0);
                                    }
                                    float* fc = P.nrc.frame_contribution + 3 * static_cast<size_t>(rec);
                                    fc[0] = c.r;
                                    fc[1] = c.g;
                                    fc[2] = c.b;
                                }
                                if (is_train(s))
                                    (kCombo ? P.train_sets[tr_set(s)].rng : P.rng)[q[W_SAMPLE]] = ld_rng(q).state;
                                else if (!sample_parallel)
                                    P.rng[pixel] = ld_rng(q).state;
                            } else {
                                if constexpr (kLog) {
                                    reinterpret_cast<uint4*>(P.dlog)[static_cast<uint64_t>(pixel) * P.spp + q[W_SAMPLE]] =
                                        make_uint4(path_length, q[W_REC], q[W_REC + 1], end_code);
                                }
                                const bool fine = all_nonneg_finite(contribution);
                                if (!fine) err |= VPT_DEVERR_NONFINITE;
                                if (sample_parallel) {
                                    if (fine) {
                                        atomicAdd(P.sum_rgb + 3 * pixel, static_cast<double>(contribution.r));
                                        atomicAdd(P.sum_rgb + 3 * pixel + 1, static_cast<double>(contribution.g));
                                        atomicAdd(P.sum_rgb + 3 * pixel + 2, static_cast<double>(contribution.b));
                                    }
                                } else if constexpr (kMayPerPixel) {
                                    // The pixel's sums of this launch and its running mean.
                                    const uint32_t smp = q[W_SAMPLE];
                                    auto sum_of = [&](int c) -> double {
                                        return __hiloint2double(static_cast<int>(q[W_SUM + 2 * c + 1]),
                                                                static_cast<int>(q[W_SUM + 2 * c]));
                                    };
                                    auto set_sum = [&](int c, double v) {
                                        q[W_SUM + 2 * c] = static_cast<uint32_t>(__double2loint(v));
                                        q[W_SUM + 2 * c + 1] = static_cast<uint32_t>(__double2hiint(v));
                                    };
                                    const V3 m3 = ld3(q, W_MEAN);
                                    RGB mean = rgb(m3.x, m3.y, m3.z);
                                    if (fine) {
                                        set_sum(0, sum_of(0) + contribution.r);
                                        set_sum(1, sum_of(1) + contribution.g);
                                        set_sum(2, sum_of(2) + contribution.b);
                                        uint32_t n = P.accum_base + smp;
                                        RGB prev = n > 0 ? mean : rgb(0, 0, 0);
                                        float w = 1.0f / (n + 1);
                                        mean = (1 - w) * prev + w * contribution;
                                        st3(q, W_MEAN, v3(mean.r, mean.g, mean.b));
                                    }
                                    if (smp + 1 < P.spp) {
                                        q[W_SAMPLE] = smp + 1;
                                        same_pixel = true;
                                    } else {
                                        P.rng[pixel] = ld_rng(q).state;
                                        P.sum_rgb[3 * pixel] += sum_of(0);
                                        P.sum_rgb[3 * pixel + 1] += sum_of(1);
                                        P.sum_rgb[3 * pixel + 2] += sum_of(2);
                                        P.mean_rgb[3 * pixel] = mean.r;
                                        P.mean_rgb[3 * pixel + 1] = mean.g;
                                        P.mean_rgb[3 * pixel + 2] = mean.b;
                                    }
                                }
                            }
                        }
                        s = 0;
                        uint32_t pixel, img_w = static_cast<uint32_t>(P.width), img_h = static_cast<uint32_t>(P.height);
                        if (kMayPerPixel && same_pixel) {
                            rng = ld_rng(q);
                            pixel = q[W_PIXEL];
                        } else {
                            // One atomic for all lanes of the warp that need an item now.
                            const uint32_t need = __activemask();
                            const int leader = __ffs(need) - 1;
                            uint32_t base = 0;
                            if (static_cast<int>(lane) == leader) base = atomicAdd(P.work_counter, __popc(need));
                            base = __shfl_sync(need, base, leader);
                            const uint32_t item = base + __popc(need & ((1u << lane) - 1u));
                            if (item >= num_items) {
                                break;  // st stays RS_DONE
                            }
                            if (kMayTrain && (kMode == kModeTrainNrc || item < num_train)) {
                                uint32_t px, py, local = item, tset = 0;
                                if constexpr (kCombo) {
                                    while (tset + 1 < P.num_train_sets) {
                                        const uint32_t n = min(set_w(tset) * set_h(tset), num_pixels);
                                        if (local < n) break;
                                        local -= n;
                                        ++tset;
                                    }
                                    s |= kTrain | (tset << kSetShift);
                                }
                                img_w = set_w(tset);
                                img_h = set_h(tset);
                                const uint32_t offset = tr_counters(s)[6];
                                train_item_to_pixel(local, img_w, img_h, offset, &px, &py);
                                pixel = py * img_w + px;  // linear index in the training image
                                const uint32_t rng_index = py * static_cast<uint32_t>(P.width) + px;
                                if constexpr (kCombo)
                                    rng.state = P.train_sets[tset].rng[rng_index];
                                else
                                    rng.state = P.rng[rng_index];
                                // optix_pathtracing_kernels.cu:60-66: one unbiased suffix per 4x4 tile.
                                const uint32_t tile_index = (py % 4) * 4 + (px % 4);
                                if ((tile_index + offset) % 16 == 0) s |= kUnbiased;
                                q[W_SAMPLE] = rng_index;
                            } else if (sample_parallel) {
                                // The samples of a pixel are consecutive items: they trace the same
                                // primary rays through the same leaves.
                                const uint32_t r = kCombo ? item - num_train : item;
                                pixel = r / P.spp;
                                const uint32_t smp = r % P.spp;
                                const ulonglong2 jump = P.sample_jumps[smp];
                                rng.state = jump.x * P.rng[pixel] + jump.y;
                                q[W_SAMPLE] = smp;
                            } else {
                                pixel = kCombo ? item - num_train : item;
                                rng.state = P.rng[pixel];
                                q[W_SAMPLE] = 0;
                                if constexpr (kMayPerPixel) {
#pragma unroll
                                    for (int c = 0; c < 6; ++c) q[W_SUM + c] = 0;
#pragma unroll
                                    for (int c = 0; c < 3; ++c)
                                        stf(q, W_MEAN + c, P.accum_base > 0 ? P.mean_rgb[3 * pixel + c] : 0.0f);
                                }
                            }
                            q[W_PIXEL] = pixel;
                        }
                        const uint32_t px = pixel % img_w;
                        const uint32_t py = pixel / img_w;
                        float ux = rng.uniform();
                        float fx = (px + ux) / static_cast<float>(img_w);
                        float uy = rng.uniform();
                        float fy = (py + uy) / static_cast<float>(img_h);
                        const float cam_vh = 2 * tanf(P.cam_fovy * 0.5f);
                        const float cam_vw = P.cam_aspect * cam_vh;
                        const float sensor_area = cam_vw * cam_vh;
                        const V3 origin = v3(P.cam_pos[0], P.cam_pos[1], P.cam_pos[2]);
                        V3 local = normalize(v3(cam_vw * (-0.5f + fx), cam_vh * (0.5f - fy), -1));
                        dir = normalize(mul(quat_to_m3(P.cam_quat[0], P.cam_quat[1], P.cam_quat[2], P.cam_quat[3]), local));
                        float az = fabsf(local.z);
                        const float dir_pdf = 1 / (az * az * az * sensor_area);
                        const float inv = 1.0f / dir_pdf;
                        const RGB tp = rgb(1, 1, 1) * inv;
                        st_rng(q, rng);
                        st3(q, W_ORG, origin);
                        st3(q, W_DIR, dir);
                        stf(q, W_DPDF, dir_pdf);
                        st_tp(q, tp);
                        stf(q, W_INIT, luminance(tp));
                        st3(q, W_CON, v3(0, 0, 0));
                        q[W_LEN] = 1;
                        if constexpr (kNrc) {
                            stf(q, W_SSPREAD, 0.0f);
                            stf(q, W_LDENS, 0.0f);
                            q[W_PREV] = kInvalidVertex;
                        }
                        if constexpr (kLog) q[W_REC] = q[W_REC + 1] = 0;
                        ++n_vertices;
                        st = s | RS_ESCAPE;
                        segment = true;
                        seg_eye = origin;
                        seg_dir = dir;
                    } while (false);
                }
            }
            if constexpr (kSurfaces) {
                bool overflow = false;
                if (segment) {
                    // A primary segment ends at its closest triangle (optix_pathtracing_kernels.cu:84-96).
                    uint32_t* q = slot_ptr(slot);
                    const SurfHit h = bvh_closest(P.surf, seg_eye, seg_dir, 0.0f, 1e10f, &overflow);
                    if (h.tri != ~0u) {
                        q[W_HIT] = h.tri;
                        stf(q, W_HIT + 1, h.b1);
                        stf(q, W_HIT + 2, h.b2);
                        seg_max = h.t;
                        st = (st & ~kStateMask) | RS_SURFACE | kHit;
                    }
                    segment = P.volume_enabled != 0;
                }
                if (light) {
                    // Light sample (renderer_kernel_common.h:297-358): the environment group (image or
                    // sky, and the sun) against the emitting triangles with probToSampleEnvLight, the
                    // triangles' visibility test from the light towards the vertex, then the shadow
                    // segment through the volume.
                    uint32_t* q = slot_ptr(slot);
                    const V3 origin = seg_eye;
                    float u_light = rng.uniform();
                    const float u0 = rng.uniform();
                    const float u1 = rng.uniform();
                    const bool areas = P.surf.inst_integral > 0.0f;
                    const bool env_group = P.env_enabled || P.sun.enabled;
                    bool select_env = false, pick_sun = false;
                    float type_prob = 1.0f;
                    if (env_group) {
                        if (areas) {
                            if (u_light < kProbEnvLight) {
                                type_prob = kProbEnvLight;
                                u_light /= type_prob;
                                select_env = true;
                            } else {
                                type_prob = 1.0f - kProbEnvLight;
                                u_light = (u_light - kProbEnvLight) / type_prob;
                            }
                        } else {
                            select_env = true;
                        }
                    }
                    float nee_lp_cos = 1.0f, nee_dist2 = 1.0f, area_pdf = 1.0f;
                    bool have_light = env_group || areas;
                    V3 sdir = v3(0, 0, 1), light_dir = v3(0, 1, 0), shadow_eye = v3(0, 0, 0);
                    RGB emittance = rgb(0, 0, 0);
                    float trace_length = trace_len;
                    if (have_light && select_env) {
                        float light_prob = 1.0f;
                        if (P.sun.enabled && P.env_enabled) {
                            if (u_light < P.sun.select_prob) {
                                pick_sun = true;
                                light_prob = P.sun.select_prob;
                            } else {
                                light_prob = 1.0f - P.sun.select_prob;
                            }
                        } else if (P.sun.enabled) {
                            pick_sun = true;
                        }
                        if (pick_sun) {
                            light_dir = v3(P.sun.dir[0], P.sun.dir[1], P.sun.dir[2]);
                            area_pdf = light_prob;
                        } else {
                            float pdf;
                            const RGB radiance = env_sample(P.env, u0, u1, &light_dir, &pdf);
                            emittance = kPi * radiance;
                            area_pdf = pdf;
                            if (area_pdf == 0.0f) have_light = false;
                            area_pdf *= light_prob;
                        }
                        if (have_light) {
                            area_pdf *= type_prob;
                            sdir = -light_dir;
                            nee_lp_cos = dot(sdir, -light_dir);
                            if (nee_lp_cos <= 0.0f) have_light = false;
                            shadow_eye = origin + trace_len * light_dir;
                        }
                    } else if (have_light) {
                        const AreaSample as = sample_area_light(P.surf, u_light, u0, u1);
                        if (as.area_pdf == 0.0f) {
                            have_light = false;
                        } else {
                            area_pdf = as.area_pdf * type_prob;
                            emittance = as.emittance;
                            sdir = origin - as.pos;
                            const float lp_cos = dot(sdir, as.normal);
                            if (lp_cos <= 0.0f) {
                                have_light = false;
                            } else {
                                shadow_eye = offset_ray_origin(as.pos, as.normal);
                                sdir = origin - shadow_eye;
                                nee_dist2 = dot(sdir, sdir);
                                trace_length = sqrtf(nee_dist2);
                                sdir = sdir * (1.0f / trace_length);
                                nee_lp_cos = lp_cos / trace_length;
                                light_dir = -sdir;
                            }
                        }
                    }
                    if (have_light && bvh_any(P.surf, shadow_eye, sdir, 0.0f, trace_length * 0.9999f, &overflow))
                        have_light = false;
                    st3(q, W_LDIR, light_dir);
                    st3(q, W_EMI, v3(emittance.r, emittance.g, emittance.b));
                    stf(q, W_APDF, area_pdf);
                    stf(q, W_LPCOS, nee_lp_cos);
                    stf(q, W_LPCOS + 1, nee_dist2);
                    st3(q, W_EYE, shadow_eye);
                    stf(q, W_VIS, have_light ? 1.0f : 0.0f);
                    st_rng(q, rng);
                    st |= nee_state(st) | (pick_sun ? kPickSun : 0u);
                    segment = have_light && P.volume_enabled;
                    seg_eye = shadow_eye;
                    seg_dir = sdir;
                    seg_max = trace_length;
                }
                if (overflow) err |= VPT_DEVERR_BVH_STACK;
            }
            if (slot != kEmpty) {
                uint32_t* q = slot_ptr(slot);
                if (segment && start_segment(q, seg_eye, seg_dir, seg_max))
                    st = (st & ~kStateMask) | RS_TRACK | (kind == Q_VERTEX || (kSurfaces && kind == Q_SURFACE) ? kShadow : 0u);
                q[W_ST] = st;
                // The segments that start here are tracked by this warp at once.
                give = (st & kStateMask) != RS_TRACK;
                if (give) got = kEmpty;
            }
        }

        // ---------------------------------------------------------------- tracking
        // Lanes whose segment ended are handed to the event queues and filled with other segments
        // once kRefill lanes are idle, so that the steps run with nearly full warps.
        if (got != kEmpty) {
            slot = got;
            const uint32_t* q = slot_ptr(slot);
            st = q[W_ST];
            act = true;
            next = st & (kStateMask | kShadow);
            rng = ld_rng(q);
            t = ldf(q, W_T);
            t1 = ldf(q, W_T1);
            vis = ldf(q, W_VIS);
            dir = ld3(q, W_DIR);
            eye = ld3(q, W_ORG);
            if (st & kShadow) {
                const V3 light_dir = ld3(q, W_LDIR);
                if constexpr (kSurfaces)
                    eye = ld3(q, W_EYE);
                else
                    eye = eye + trace_len * light_dir;
                dir = -light_dir;
            }
            steps = steps0 = q[W_STEPS];
            if constexpr (kGridMajorant) {
                lin = static_cast<int>(q[W_DDA]);
                rem0 = static_cast<int>(q[W_DDA + 1]);
                rem1 = static_cast<int>(q[W_DDA + 2]);
                rem2 = static_cast<int>(q[W_DDA + 3]);
                tn0 = ldf(q, W_DDA + 4);
                tn1 = ldf(q, W_DDA + 5);
                tn2 = ldf(q, W_DDA + 6);
                const float size = static_cast<float>(1 << g.maj_shift);
                td0 = dda_delta(size, dir.x * g.inv_voxel_size);
                td1 = dda_delta(size, dir.y * g.inv_voxel_size);
                td2 = dda_delta(size, dir.z * g.inv_voxel_size);
                texit = fminf(fminf(tn0, tn1), fminf(tn2, t1));
                maj = P.density_coeff * maj_grid[lin];
            }
        }
        while (true) {
            bool lookup = false;
            if (act) {
                if constexpr (!kGridMajorant) {
                    t += -logf(1.0f - rng.uniform()) / maj;
                    lookup = t <= t1;
                    act = lookup;
                } else {
                    // A free-flight distance within the current cell; an overshoot of the cell's
                    // exit restarts at the exit (memoryless), empty cells are crossed without draws.
#pragma unroll 1
                    for (int c = 0; c < kCellSteps; ++c) {
                        if (maj > 0) {
                            const float tt = t + -logf(1.0f - rng.uniform()) / maj;
                            if (tt < texit) {
                                t = tt;
                                lookup = true;
                                break;
                            }
                        }
                        t = texit;
                        if (texit >= t1) {
                            act = false;
                            break;
                        }
                        // Along the axis whose boundary comes first (x, then y, then z on ties).
                        const bool ax0 = tn0 <= tn1 && tn0 <= tn2;
                        const bool ax1 = !ax0 && tn1 <= tn2;
                        const int rem = ax0 ? rem0 : (ax1 ? rem1 : rem2);
                        ++n_cells;
                        if (rem == 0) {
                            t = t1;
                            act = false;
                            break;
                        }
                        const float d = ax0 ? dir.x : (ax1 ? dir.y : dir.z);
                        const int stride = ax0 ? g.my * g.mz : (ax1 ? g.mz : 1);
                        lin += d > 0 ? stride : -stride;
                        if (ax0) {
                            tn0 += td0;
                            --rem0;
                        } else if (ax1) {
                            tn1 += td1;
                            --rem1;
                        } else {
                            tn2 += td2;
                            --rem2;
                        }
                        texit = fminf(fminf(tn0, tn1), fminf(tn2, t1));
                        maj = P.density_coeff * maj_grid[lin];
                    }
                }
                if constexpr (kSurfaces) {
                    if (!act) next = st & kShadow ? nee_state(st) : (st & kHit ? RS_SURFACE : RS_ESCAPE);
                } else {
                    if (!act) next = st & kShadow ? RS_NEE_DONE : RS_ESCAPE;
                }
            }
            if (lookup) {
                const V3 xyz = world_to_index(g, eye + dir * t);
                float density;
                if constexpr (kStencil)
                    density = P.density_coeff * sample_stencil(g, xyz, leaf_cache);
                else
                    density = P.density_coeff * sample_trilinear(g, xyz, leaf_cache);
                ++steps;
                if (st & kShadow) {
                    vis *= (1 - density / maj);
                    // Roulette on the remaining visibility; training suffixes keep plain ratio tracking.
                    const float rr_thr = is_train(st) ? 0.0f : P.shadow_rr;
                    if (vis < rr_thr) {
                        const float p = vis / rr_thr;
                        if (rng.uniform() >= p) {
                            vis = 0.0f;
                            act = false;
                            if constexpr (kSurfaces)
                                next = nee_state(st);
                            else
                                next = RS_NEE_DONE;
                        } else {
                            vis = rr_thr;
                        }
                    }
                } else if (rng.uniform() < density / maj) {
                    act = false;
                    next = RS_VERTEX;
                    last = density;
                }
                if (act && steps >= step_cap) {
                    err |= VPT_DEVERR_STEP_CAP;
                    act = false;
                    next = RS_END | (END_STEP_CAP << kEndShift);
                }
            }
            // On while enough lanes track, or none has ended and there is no segment to take.
            const uint32_t on = __ballot_sync(0xffffffffu, act);
            if (__popc(on) > 32 - kRefill) continue;
            if (on == 0 || __any_sync(0xffffffffu, slot != kEmpty && !act) ||
                __shfl_sync(0xffffffffu, count_of(sv[Q_TRACK]), 0) != 0)
                break;
        }
        // Hand over the ended segments; all of them when a full event batch waits.
        bool leave = max(count_of(sv[Q_VERTEX]), max(count_of(sv[Q_NEE_DONE]), count_of(sv[Q_END]))) >= kEventBatch;
        if (kSurfaces) leave = leave || max(count_of(sv[Q_SURFACE]), count_of(sv[Q_NEE_SURF])) >= kEventBatch;
        const bool all = __shfl_sync(0xffffffffu, leave, 0);
        if (slot != kEmpty && !give && (!act || all)) {
            uint32_t* q = slot_ptr(slot);
            n_lookups += steps - steps0;
            if constexpr (kLog) q[W_REC + (st & kShadow ? 1 : 0)] += steps - steps0;
            st = (st & kKept) | next;
            q[W_ST] = st;
            st_rng(q, rng);
            stf(q, W_T, t);
            stf(q, W_VIS, vis);
            q[W_STEPS] = steps;
            if constexpr (kNrc) {
                if ((next & kStateMask) == RS_VERTEX) stf(q, W_LDENS, last);
            }
            if (kGridMajorant && act) {
                q[W_DDA] = static_cast<uint32_t>(lin);
                q[W_DDA + 1] = static_cast<uint32_t>(rem0);
                q[W_DDA + 2] = static_cast<uint32_t>(rem1);
                q[W_DDA + 3] = static_cast<uint32_t>(rem2);
                stf(q, W_DDA + 4, tn0);
                stf(q, W_DDA + 5, tn1);
                stf(q, W_DDA + 6, tn2);
            }
            give = true;
            act = false;
        }
    }
    if (*static_cast<volatile uint32_t*>(s_abort) != 0) err |= VPT_DEVERR_QUEUE_TIMEOUT;

    // warp-reduce the work counters
    unsigned long long c_lookups = n_lookups, c_vertices = n_vertices, c_samples = n_samples, c_cells = n_cells;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        c_lookups += __shfl_down_sync(0xffffffffu, c_lookups, o);
        c_vertices += __shfl_down_sync(0xffffffffu, c_vertices, o);
        c_samples += __shfl_down_sync(0xffffffffu, c_samples, o);
        c_cells += __shfl_down_sync(0xffffffffu, c_cells, o);
    }
    err = __reduce_or_sync(0xffffffffu, err);
    if (lane == 0) {
        atomicAdd(P.counters + 0, c_lookups);
        atomicAdd(P.counters + 1, c_vertices);
        atomicAdd(P.counters + 2, c_samples);
        atomicAdd(P.counters + 3, c_cells);
        if (err) atomicOr(P.error_flags, err);
    }
}

template <bool kGridMajorant, bool kLog, int kMode, int kStreams, bool kSurfaces>
const void* kernel_of(bool stencil) {
    return stencil ? reinterpret_cast<const void*>(queue_trace_kernel<kGridMajorant, kLog, kMode, kStreams, true, kSurfaces>)
                   : reinterpret_cast<const void*>(queue_trace_kernel<kGridMajorant, kLog, kMode, kStreams, false, kSurfaces>);
}
template <bool kLog, int kMode, int kStreams, bool kSurfaces>
const void* kernel_of(bool grid_majorant, bool stencil) {
    return grid_majorant ? kernel_of<true, kLog, kMode, kStreams, kSurfaces>(stencil)
                         : kernel_of<false, kLog, kMode, kStreams, kSurfaces>(stencil);
}

template <bool kSurfaces>
const void* kernel_ptr(int mode, bool grid_majorant, bool logged, bool sample_parallel, bool stencil) {
    if (mode == kModeTrainNrc) return kernel_of<false, kModeTrainNrc, kStreamsRuntime, kSurfaces>(grid_majorant, stencil);
    if (mode == kModeComboNrc) return kernel_of<false, kModeComboNrc, kStreamsRuntime, kSurfaces>(grid_majorant, stencil);
    if (mode == kModeRenderNrc) return kernel_of<false, kModeRenderNrc, kStreamsRuntime, kSurfaces>(grid_majorant, stencil);
    if (logged)
        return sample_parallel ? kernel_of<true, kModePlain, kStreamsSampleParallel, kSurfaces>(grid_majorant, stencil)
                               : kernel_of<true, kModePlain, kStreamsPerPixel, kSurfaces>(grid_majorant, stencil);
    return sample_parallel ? kernel_of<false, kModePlain, kStreamsSampleParallel, kSurfaces>(grid_majorant, stencil)
                           : kernel_of<false, kModePlain, kStreamsPerPixel, kSurfaces>(grid_majorant, stencil);
}

}  // namespace

cudaError_t launch_queues(TraceParams& p, int mode, bool grid_majorant, int threads, int ctas_per_sm, int sms,
                          cudaStream_t s) {
    const bool logged = p.dlog != nullptr, sample_parallel = p.stream_mode == 1, nrc = mode != kModePlain;
    const bool surfaces = p.surf.enabled != 0, stencil = p.grid.st_values != nullptr;
    const int cells = grid_majorant ? p.grid.mx * p.grid.my * p.grid.mz : 0;
    p.maj_in_smem = cells > 0 && cells <= kQueueMajCells;
    const void* kernel = surfaces ? kernel_ptr<true>(mode, grid_majorant, logged, sample_parallel, stencil)
                                  : kernel_ptr<false>(mode, grid_majorant, logged, sample_parallel, stencil);
    const size_t words = queue_words(grid_majorant, logged, nrc, !nrc && !sample_parallel, surfaces);
    auto bytes = [&](int n, int maj_cells) -> size_t {
        return 32 + queue_slots(n, surfaces) * words * 4 + queue_count(surfaces) * queue_ring(n) * 2 + maj_cells * sizeof(float);
    };
    const size_t smem = bytes(threads, p.maj_in_smem ? cells : 0);
    // The limit is the kernel's largest launch, not this one's: threads with contexts of different
    // shapes may launch the same kernel at once.
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(bytes(kQueueThreads, kQueueMajCells)));
    if (e != cudaSuccess) return e;
    if (ctas_per_sm <= 0 &&
        (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ctas_per_sm, kernel, threads, smem) != cudaSuccess ||
         ctas_per_sm <= 0))
        ctas_per_sm = 1;
    void* args[] = {&p};
    return cudaLaunchKernel(kernel, dim3(sms * ctas_per_sm), dim3(threads), args, smem, s);
}

}  // namespace vpt
