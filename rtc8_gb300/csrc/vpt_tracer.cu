// Leaf-staging form of the plain volume tracer (vpt_set_leaf_staging): one path per lane, each warp
// keeping one 8^3 leaf of the grid in shared memory. Without leaf staging the tracker with work
// queues (vpt_queues.cu) runs, which gives the same paths. The reference is the pathTrace
// ray-generation program (renderer/gpu_kernels/optix_pathtracing_kernels.cu:31-434). Beside it, the
// small kernels of a launch: jump tables, mean image, frame counters, pooled majorants.
//
// One resident set of CTAs per SM pulls work items from a global counter (path regeneration: a
// lane that finishes a path starts the next one at once). A work item is a pixel (reference
// streams, logged launches only) or one (pixel, sample) pair (sample-parallel streams). Each loop
// iteration first lets every lane run its cheap, divergent event logic until it needs a density
// value, then all lanes perform their grid lookups together, so that lanes in one leaf can share it.
#include "vpt_ctx.h"
#include "vpt_track.cuh"

namespace vpt {
namespace {

enum : uint32_t {
    ST_FETCH = 0,    // get the next work item
    ST_CAMERA,       // start a sample: camera ray
    ST_SEGMENT,      // start a primary segment: ++pathLength, clip
    ST_STEP,         // advance the current segment to its next lookup
    ST_VERTEX,       // primary collision: RR, NEE set-up
    ST_NEE_DONE,     // shadow segment finished: NEE contribution, phase sampling
    ST_ESCAPE,       // primary segment left the grid
    ST_END_SAMPLE,   // accumulate, next sample or next item
    ST_DONE,
};

// Majorant-grid cells a lane crosses per tracking iteration before yielding to the warp, parked
// lanes of a warp that trigger a joint event phase, and resident CTAs of 128 threads per SM the
// register allocation is bounded for.
constexpr int kStageCellSteps = 8;
constexpr int kStageParkThreshold = 16;
constexpr int kStageCtasPerSm = 5;

enum : int { PASS_LOOKUP = 0, PASS_YIELD = 1, PASS_END = 2 };

// One tracking pass of a segment from (t, texit, maj, dda): a free-flight distance
// (optix_pathtracing_kernels.cu:113-118 / renderer_kernel_common.h:374-378), with the majorant
// grid sampled within the current cell, where an overshoot of the cell's exit restarts at the
// exit (memoryless) and empty cells are crossed without draws, at most kStageCellSteps crossings per
// pass. PASS_LOOKUP leaves t at the tentative collision; PASS_END means the segment
// is over (also on a NaN distance); PASS_YIELD means the pass crossed its cells without one.
__device__ __forceinline__ int track_pass(const Grid& g, const float* maj_grid, float density_coeff, float t1, V3 dir,
                                          Pcg32& rng, float& t, float& texit, float& maj, DdaState& dda,
                                          uint32_t& n_cells) {
    for (int c = 0; c < kStageCellSteps; ++c) {
        if (maj > 0) {
            const float tt = t + -logf(1.0f - rng.uniform()) / maj;
            if (tt < texit) {
                t = tt;
                return PASS_LOOKUP;
            }
        }
        t = texit;
        if (texit >= t1) return PASS_END;
        // Advance along the axis whose boundary comes first (x, then y, then z on ties);
        // written with selects so the DDA state stays in registers.
        const bool ax0 = dda.tnext[0] <= dda.tnext[1] && dda.tnext[0] <= dda.tnext[2];
        const bool ax1 = !ax0 && dda.tnext[1] <= dda.tnext[2];
        const bool ax2 = !ax0 && !ax1;
        if (ax0) dda.cell[0] += step_of(dir.x);
        if (ax1) dda.cell[1] += step_of(dir.y);
        if (ax2) dda.cell[2] += step_of(dir.z);
        ++n_cells;
        if (dda.cell[0] < 0 || dda.cell[0] >= g.mx || dda.cell[1] < 0 || dda.cell[1] >= g.my || dda.cell[2] < 0 ||
            dda.cell[2] >= g.mz) {
            t = t1;
            return PASS_END;
        }
        if (ax0) dda.tnext[0] += dda.tdelta[0];
        if (ax1) dda.tnext[1] += dda.tdelta[1];
        if (ax2) dda.tnext[2] += dda.tdelta[2];
        texit = fminf(fminf(dda.tnext[0], dda.tnext[1]), fminf(dda.tnext[2], t1));
        maj = density_coeff * cell_maj(maj_grid, g, dda);
    }
    return PASS_YIELD;
}

template <bool kLog>
__global__ void __launch_bounds__(128, kStageCtasPerSm) staged_trace_kernel(const TraceParams P) {
    const bool sample_parallel = kLog ? P.stream_mode == 1 : true;
    extern __shared__ __align__(128) float s_maj[];
    const Grid& g = P.grid;
    const float* maj_grid = g.maj;
    if (P.maj_in_smem) {
        const int cells = g.mx * g.my * g.mz;
        for (int i = threadIdx.x; i < cells; i += blockDim.x) s_maj[i] = g.maj[i];
        __syncthreads();
        maj_grid = s_maj;
    }
    // After the staged majorant grid: the warps' leaf buffers, then their mbarriers.
    LeafStage stage{nullptr, nullptr, -1, -1, 0u};
    bool stage_timed_out = false;
    {
        const size_t maj_bytes = P.maj_in_smem ? static_cast<size_t>(g.mx) * g.my * g.mz * sizeof(float) : 0;
        unsigned char* area = reinterpret_cast<unsigned char*>(s_maj) + (maj_bytes + 127) / 128 * 128;
        const int warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
        stage.values = reinterpret_cast<float*>(area + static_cast<size_t>(warp) * kLeafBytes);
        stage.bar = reinterpret_cast<uint64_t*>(area + static_cast<size_t>(warps) * kLeafBytes) + warp;
        if ((threadIdx.x & 31) == 0) stage_bar_init(stage.bar);
        __syncwarp();
    }
    const uint32_t num_pixels = static_cast<uint32_t>(P.width) * static_cast<uint32_t>(P.height);
    const uint32_t step_cap = P.max_steps > 0 ? static_cast<uint32_t>(P.max_steps) : kHardStepCap;
    const int park_threshold = P.park_threshold > 0 ? P.park_threshold : kStageParkThreshold;
    const V3 bmin = v3(g.bbox_min[0], g.bbox_min[1], g.bbox_min[2]);
    const V3 bmax = v3(g.bbox_max[0], g.bbox_max[1], g.bbox_max[2]);
    // Sensor height of the launch's camera (optix_pathtracing_kernels.cu:43-55).
    const float cam_vh = 2 * tanf(P.cam_fovy * 0.5f);

    uint32_t st = ST_FETCH;
    uint32_t pixel = 0, sample = 0;
    Pcg32 rng{0};
    double sum_r = 0, sum_g = 0, sum_b = 0;
    RGB mean = rgb(0, 0, 0);

    // per-sample state
    V3 origin = v3(0, 0, 0), dir = v3(0, 0, 1);
    float dir_pdf = 1.0f, init_importance = 1.0f;
    RGB throughput = rgb(0, 0, 0), contribution = rgb(0, 0, 0);
    uint32_t path_length = 0, end_code = 0;
    uint32_t rec_primary = 0, rec_shadow = 0;

    // The current segment: a primary segment starts at the path's origin along its direction, a
    // shadow segment at origin + trace_len * light_dir towards -light_dir.
    bool shadow = false;
    const float trace_len = 2 * P.world_radius;
    float t = 0, t1 = 0, maj = 0, texit = 0;
    uint32_t seg_steps = 0;
    DdaState dda;

    // NEE in flight
    V3 light_dir = v3(0, 1, 0);
    RGB emittance = rgb(0, 0, 0);
    float area_pdf = 1.0f, vis = 1.0f;
    bool pick_sun = false;

    // Per-lane work counters, summed over the warp in 64 bits at the end.
    uint32_t n_lookups = 0, n_vertices = 0, n_samples = 0, n_cells = 0;
    unsigned int err = 0;
    LeafCache leaf_cache;

    while (true) {
        // Warp-level event batching: lanes whose path reached an event (segment end, collision,
        // new sample) park until at least park_threshold lanes of the warp are parked, or no lane
        // is tracking any more; then all parked lanes run their event logic together. In between,
        // the tracking lanes advance one step per iteration.
        const bool tracking = st == ST_STEP;
        const uint32_t ev_mask = __ballot_sync(0xffffffffu, !tracking && st != ST_DONE);
        const uint32_t tr_mask = __ballot_sync(0xffffffffu, tracking);
        if ((ev_mask | tr_mask) == 0) break;
        const bool event_phase = ev_mask != 0 && (tr_mask == 0 || __popc(ev_mask) >= park_threshold);
        bool need_lookup = false, yield = false;
        V3 lookup_pos = v3(0, 0, 0);
        while (!need_lookup && !yield && st != ST_DONE && (event_phase ? st != ST_STEP : st == ST_STEP)) {
            switch (st) {
            case ST_FETCH: {
                // Warp-aggregated fetch: one atomic for all lanes of the warp that need work now.
                const uint32_t need = __activemask();
                const int leader = __ffs(need) - 1;
                const uint32_t lane = threadIdx.x & 31;
                uint32_t base = 0;
                if (static_cast<int>(lane) == leader) base = atomicAdd(P.work_counter, __popc(need));
                base = __shfl_sync(need, base, leader);
                const uint32_t item = base + __popc(need & ((1u << lane) - 1u));
                if (item >= (sample_parallel ? num_pixels * P.spp : num_pixels)) {
                    st = ST_DONE;
                    break;
                }
                st = ST_CAMERA;
                if (sample_parallel) {
                    // One (pixel, sample) per work item, the spp samples of a pixel consecutive. Sample
                    // (stream_base + sample) starts (stream_base + sample) * 2^40 draws into the
                    // pixel's stream: state = A * seed + C with the launch's jump table.
                    pixel = item / P.spp;
                    sample = item % P.spp;
                    const ulonglong2 jump = P.sample_jumps[sample];
                    rng.state = jump.x * P.rng[pixel] + jump.y;
                    break;
                }
                pixel = item;
                rng.state = P.rng[pixel];
                sum_r = sum_g = sum_b = 0;
                if (P.accum_base > 0) {
                    mean = rgb(P.mean_rgb[3 * pixel], P.mean_rgb[3 * pixel + 1], P.mean_rgb[3 * pixel + 2]);
                } else {
                    mean = rgb(0, 0, 0);
                }
                sample = 0;
                break;
            }
            case ST_CAMERA: {
                // optix_pathtracing_kernels.cu:43-55, 76-81.
                uint32_t img_w = static_cast<uint32_t>(P.width), img_h = static_cast<uint32_t>(P.height);
                uint32_t px = pixel % img_w;
                uint32_t py = pixel / img_w;
                float ux = rng.uniform();
                float fx = (px + ux) / static_cast<float>(img_w);
                float uy = rng.uniform();
                float fy = (py + uy) / static_cast<float>(img_h);
                const float cam_vw = P.cam_aspect * cam_vh;
                const float sensor_area = cam_vw * cam_vh;
                origin = v3(P.cam_pos[0], P.cam_pos[1], P.cam_pos[2]);
                V3 local = normalize(v3(cam_vw * (-0.5f + fx), cam_vh * (0.5f - fy), -1));
                dir = normalize(mul(quat_to_m3(P.cam_quat[0], P.cam_quat[1], P.cam_quat[2], P.cam_quat[3]), local));
                float az = fabsf(local.z);
                dir_pdf = 1 / (az * az * az * sensor_area);
                float inv = 1.0f / dir_pdf;
                throughput = rgb(1, 1, 1) * inv;
                init_importance = luminance(throughput);
                contribution = rgb(0, 0, 0);
                path_length = 0;
                end_code = 0;
                rec_primary = rec_shadow = 0;
                st = ST_SEGMENT;
                break;
            }
            case ST_SEGMENT: {
                ++path_length;
                ++n_vertices;
                if (path_length > kHardVertexCap) {
                    end_code = END_MAX_BOUNCES;
                    st = ST_END_SAMPLE;
                    break;
                }
                float a, b;
                if (clip_ray(bmin, bmax, origin, dir, 0.0f, 1e10f, &a, &b)) {
                    shadow = false;
                    t = fmaxf(0.0f, a);
                    t1 = b;
                    seg_steps = 0;
                    dda_init(g, origin, dir, t, &dda);
                    texit = fminf(fminf(dda.tnext[0], dda.tnext[1]), fminf(dda.tnext[2], t1));
                    maj = P.density_coeff * cell_maj(maj_grid, g, dda);
                    st = ST_STEP;
                } else {
                    st = ST_ESCAPE;
                }
                break;
            }
            case ST_STEP: {
                const V3 seg_dir = shadow ? -light_dir : dir;
                const int r = track_pass(g, maj_grid, P.density_coeff, t1, seg_dir, rng, t, texit, maj, dda, n_cells);
                if (r == PASS_LOOKUP) {
                    const V3 seg_eye = shadow ? origin + trace_len * light_dir : origin;
                    lookup_pos = seg_eye + seg_dir * t;
                    need_lookup = true;
                } else if (r == PASS_END) {
                    st = shadow ? ST_NEE_DONE : ST_ESCAPE;
                } else {
                    yield = true;  // let the warp's lookups run before crossing more cells
                }
                break;
            }
            case ST_ESCAPE: {
                // optix_pathtracing_kernels.cu:130-174.
                if (P.env_enabled) {
                    float hyp_pdf;
                    RGB radiance = env_evaluate(P.env, dir, &hyp_pdf);
                    float mis = 1.0f;
                    if (path_length > 1) {
                        float sel = P.sun.enabled ? (1.0f - P.sun.select_prob) : 1.0f;
                        float light_pdf = sel * hyp_pdf;
                        float bsdf_pdf = dir_pdf;
                        mis = (bsdf_pdf * bsdf_pdf) / ((bsdf_pdf * bsdf_pdf) + (light_pdf * light_pdf));
                    }
                    contribution = contribution + throughput * (radiance * mis);
                }
                end_code = END_ESCAPE;
                st = ST_END_SAMPLE;
                break;
            }
            case ST_VERTEX: {
                // In-medium vertex (:176-182), Russian roulette (:254-268, 332), NEE set-up
                // (renderer_kernel_common.h:297-358).
                origin = origin + t * dir;
                float continue_prob = 1.0f;
                if (static_cast<int32_t>(path_length) >= P.rr_start) {
                    continue_prob = fminf(luminance(throughput) / init_importance, 1.0f);
                    if (rng.uniform() >= continue_prob) {
                        end_code = END_RR;
                        st = ST_END_SAMPLE;
                        break;
                    }
                }
                throughput = rdiv(throughput, continue_prob);

                float u_light = rng.uniform();
                float u0 = rng.uniform();
                float u1 = rng.uniform();
                pick_sun = false;
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
                vis = 0.0f;
                if (have_light) {
                    if (pick_sun) {
                        light_dir = v3(P.sun.dir[0], P.sun.dir[1], P.sun.dir[2]);
                        emittance = rgb(P.sun.irradiance[0], P.sun.irradiance[1], P.sun.irradiance[2]);
                        area_pdf = light_prob;
                    } else {
                        float pdf;
                        RGB radiance = env_sample(P.env, u0, u1, &light_dir, &pdf);
                        emittance = kPi * radiance;
                        area_pdf = pdf;
                        if (area_pdf == 0.0f) have_light = false;
                        area_pdf *= light_prob;
                    }
                }
                if (have_light) {
                    V3 sdir = -light_dir;
                    float lp_cos = dot(sdir, -light_dir);
                    if (lp_cos <= 0.0f) have_light = false;
                }
                if (!have_light) {
                    st = ST_NEE_DONE;  // vis = 0: no contribution
                    break;
                }
                vis = 1.0f;
                const V3 seg_dir = -light_dir;
                const V3 seg_eye = origin + trace_len * light_dir;
                float a, b;
                if (clip_ray(bmin, bmax, seg_eye, seg_dir, 0.0f, trace_len, &a, &b)) {
                    shadow = true;
                    t = fmaxf(0.0f, a);
                    t1 = b;
                    seg_steps = 0;
                    dda_init(g, seg_eye, seg_dir, t, &dda);
                    texit = fminf(fminf(dda.tnext[0], dda.tnext[1]), fminf(dda.tnext[2], t1));
                    maj = P.density_coeff * cell_maj(maj_grid, g, dda);
                    st = ST_STEP;
                } else {
                    st = ST_NEE_DONE;
                }
                break;
            }
            case ST_NEE_DONE: {
                // renderer_kernel_common.h:385-402, then phase sampling (:341-356).
                if (vis > 0.0f) {
                    V3 sdir = -light_dir;
                    Frame fr = make_frame(-dir);
                    V3 v_in_local = to_local(fr, -sdir);
                    float pf = phase_pdf(P.phase_kind, P.phase_param, v_in_local);
                    RGB fs = rgb(P.albedo, P.albedo, P.albedo) * pf;
                    RGB nee;
                    if (pick_sun) {
                        nee = fs * emittance * (vis / area_pdf);
                    } else {
                        float lp_cos = dot(sdir, -light_dir);
                        const float dist2 = 1.0f;
                        float bsdf_pdf = pf * lp_cos / dist2;
                        if (!isfinite(bsdf_pdf)) bsdf_pdf = 0.0f;
                        float light_pdf = area_pdf;
                        float mis = (light_pdf * light_pdf) / ((bsdf_pdf * bsdf_pdf) + (light_pdf * light_pdf));
                        RGB le = rdiv(emittance, kPi);
                        float gterm = lp_cos * 1.0f / dist2;
                        nee = fs * le * (vis * mis * gterm / area_pdf);
                    }
                    contribution = contribution + throughput * nee;
                }
                if (P.max_bounces > 0 && static_cast<int32_t>(path_length) >= P.max_bounces) {
                    end_code = END_MAX_BOUNCES;
                    st = ST_END_SAMPLE;
                    break;
                }
                Frame fr = make_frame(-dir);
                float u0 = rng.uniform();
                float u1 = rng.uniform();
                V3 local;
                float pdf = phase_sample(P.phase_kind, P.phase_param, u0, u1, &local);
                if (pdf == 0.0f) {
                    end_code = END_PDF_ZERO;
                    st = ST_END_SAMPLE;
                    break;
                }
                RGB fs = rgb(P.albedo, P.albedo, P.albedo) * pdf;
                dir = from_local(fr, local);
                RGB local_tp = fs * (fabsf(1.0f) / pdf);
                throughput = throughput * local_tp;
                dir_pdf = pdf;
                st = ST_SEGMENT;
                break;
            }
            case ST_END_SAMPLE: {
                // optix_pathtracing_kernels.cu:413-432 (non-finite samples are dropped).
                ++n_samples;
                if constexpr (kLog) {
                    uint4 rec = make_uint4(path_length, rec_primary, rec_shadow, end_code);
                    reinterpret_cast<uint4*>(P.dlog)[static_cast<uint64_t>(pixel) * P.spp + sample] = rec;
                }
                if (sample_parallel) {
                    if (all_nonneg_finite(contribution)) {
                        atomicAdd(P.sum_rgb + 3 * pixel, static_cast<double>(contribution.r));
                        atomicAdd(P.sum_rgb + 3 * pixel + 1, static_cast<double>(contribution.g));
                        atomicAdd(P.sum_rgb + 3 * pixel + 2, static_cast<double>(contribution.b));
                    } else {
                        err |= VPT_DEVERR_NONFINITE;
                    }
                    st = ST_FETCH;
                    break;
                }
                if (all_nonneg_finite(contribution)) {
                    sum_r += contribution.r;
                    sum_g += contribution.g;
                    sum_b += contribution.b;
                    uint32_t n = P.accum_base + sample;
                    RGB prev = n > 0 ? mean : rgb(0, 0, 0);
                    float w = 1.0f / (n + 1);
                    mean = (1 - w) * prev + w * contribution;
                } else {
                    err |= VPT_DEVERR_NONFINITE;
                }
                ++sample;
                if (sample < P.spp) {
                    st = ST_CAMERA;
                } else {
                    P.rng[pixel] = rng.state;
                    P.sum_rgb[3 * pixel] += sum_r;
                    P.sum_rgb[3 * pixel + 1] += sum_g;
                    P.sum_rgb[3 * pixel + 2] += sum_b;
                    P.mean_rgb[3 * pixel] = mean.r;
                    P.mean_rgb[3 * pixel + 1] = mean.g;
                    P.mean_rgb[3 * pixel + 2] = mean.b;
                    st = ST_FETCH;
                }
                break;
            }
            default:
                st = ST_DONE;
                break;
            }
        }

        if (event_phase || !__any_sync(0xffffffffu, need_lookup)) continue;

        // ---------------------------------------------------------------- converged lookups
        const float density = P.density_coeff * sample_trilinear_staged(g, need_lookup, world_to_index(g, lookup_pos),
                                                                        leaf_cache, stage, P.leaf_stage_min, stage_timed_out);
        if (!need_lookup) continue;
        ++n_lookups;
        ++seg_steps;
        if (shadow) {
            ++rec_shadow;
            vis *= (1 - density / maj);
            // Russian roulette on the remaining visibility (configuration mode).
            if (vis < P.shadow_rr) {
                const float q = vis / P.shadow_rr;
                if (rng.uniform() >= q) {
                    vis = 0.0f;
                    st = ST_NEE_DONE;
                } else {
                    vis = P.shadow_rr;
                }
            }
        } else {
            ++rec_primary;
            if (rng.uniform() < density / maj) st = ST_VERTEX;
        }
        if (st == ST_STEP && seg_steps >= step_cap) {
            err |= VPT_DEVERR_STEP_CAP;
            end_code = END_STEP_CAP;
            st = ST_END_SAMPLE;
        }
    }

    if (stage_timed_out) {
        // A copy that did not complete may still land in this warp's buffer: wait for it
        // (again bounded) before the CTA's shared memory is released.
        err |= VPT_DEVERR_STAGE_TIMEOUT;
        stage_wait(stage.bar, stage.phase ^ 1u);
    }

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
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(P.counters + 0, c_lookups);
        atomicAdd(P.counters + 1, c_vertices);
        atomicAdd(P.counters + 2, c_samples);
        atomicAdd(P.counters + 3, c_cells);
        if (err) atomicOr(P.error_flags, err);
    }
}

// Mean image of the sample-parallel mode: FP64 sums over the samples accumulated so far.
__global__ void finalize_mean_kernel(const double* __restrict__ sum, float* __restrict__ mean, uint32_t n,
                                     double inv_samples) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        mean[i] = static_cast<float>(sum[i] * inv_samples);
}

// Majorant grid of 2^shift-voxel cells from the 8^3-voxel cells (max-pooling by 2^(shift-3)).
__global__ void pool_majorants_kernel(const float* __restrict__ fine, int lx, int ly, int lz, float* __restrict__ out,
                                      int mx, int my, int mz, int factor) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= mx * my * mz) return;
    int cz = i % mz, cy = (i / mz) % my, cx = i / (mz * my);
    float m = 0.0f;
    for (int x = cx * factor; x < min((cx + 1) * factor, lx); ++x)
        for (int y = cy * factor; y < min((cy + 1) * factor, ly); ++y)
            for (int z = cz * factor; z < min((cz + 1) * factor, lz); ++z)
                m = fmaxf(m, fine[(static_cast<int64_t>(x) * ly + y) * lz + z]);
    out[i] = m;
}

// Entry i: LCG jump (multiplier, increment) advancing a pixel's seed state by (first + i) * 2^40
// draws, the start of that sample's stream (O(log) jump-ahead, Brown 1994).
__global__ void sample_jump_table_kernel(ulonglong2* out, uint32_t first, uint32_t count) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    uint64_t delta = static_cast<uint64_t>(first + i) << kSampleStreamShift;
    uint64_t cur_mult = 6364136223846793005ULL, cur_plus = 1ULL, acc_mult = 1ULL, acc_plus = 0ULL;
    while (delta > 0) {
        if (delta & 1ULL) {
            acc_mult *= cur_mult;
            acc_plus = acc_plus * cur_mult + cur_plus;
        }
        cur_plus = (cur_mult + 1ULL) * cur_plus;
        cur_mult *= cur_mult;
        delta >>= 1;
    }
    out[i] = make_ulonglong2(acc_mult, acc_plus);
}

// As sample_jump_table_kernel, with the first sample index read from the context's device
// frame counters (so that a launch captured in a CUDA graph continues the streams on replay).
__global__ void sample_jump_table_dev_kernel(ulonglong2* out, const uint32_t* __restrict__ frame, uint32_t count) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    uint64_t delta = static_cast<uint64_t>(frame[0] + i) << kSampleStreamShift;
    uint64_t cur_mult = 6364136223846793005ULL, cur_plus = 1ULL, acc_mult = 1ULL, acc_plus = 0ULL;
    while (delta > 0) {
        if (delta & 1ULL) {
            acc_mult *= cur_mult;
            acc_plus = acc_plus * cur_mult + cur_plus;
        }
        cur_plus = (cur_mult + 1ULL) * cur_plus;
        cur_mult *= cur_mult;
        delta >>= 1;
    }
    out[i] = make_ulonglong2(acc_mult, acc_plus);
}

// mean = sum / (accumulated samples + spp), the count read from the device frame counters.
__global__ void finalize_mean_dev_kernel(const double* __restrict__ sum, float* __restrict__ mean, uint32_t n,
                                         const uint32_t* __restrict__ frame, uint32_t spp) {
    const double inv = 1.0 / (static_cast<double>(frame[1]) + spp);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        mean[i] = static_cast<float>(sum[i] * inv);
}

// frame[0] += add_stream; frame[1] = set ? value : frame[1] + value.
__global__ void frame_update_kernel(uint32_t* frame, uint32_t add_stream, int set_accum, uint32_t value) {
    frame[0] += add_stream;
    frame[1] = set_accum ? value : frame[1] + value;
}

}  // namespace

void launch_sample_jump_table_dev(ulonglong2* out, const uint32_t* frame, uint32_t count, cudaStream_t s) {
    sample_jump_table_dev_kernel<<<(count + 127) / 128, 128, 0, s>>>(out, frame, count);
}
void launch_finalize_mean_dev(const double* sum, float* mean, uint32_t n_values, const uint32_t* frame, uint32_t spp,
                              cudaStream_t s) {
    finalize_mean_dev_kernel<<<(n_values + 255) / 256, 256, 0, s>>>(sum, mean, n_values, frame, spp);
}
void launch_frame_update(uint32_t* frame, uint32_t add_stream, bool set_accum, uint32_t value, cudaStream_t s) {
    frame_update_kernel<<<1, 1, 0, s>>>(frame, add_stream, set_accum ? 1 : 0, value);
}

void launch_sample_jump_table(ulonglong2* out, uint32_t first, uint32_t count, cudaStream_t s) {
    sample_jump_table_kernel<<<(count + 127) / 128, 128, 0, s>>>(out, first, count);
}

void launch_finalize_mean(const double* sum, float* mean, uint32_t n_values, uint32_t samples, cudaStream_t s) {
    finalize_mean_kernel<<<(n_values + 255) / 256, 256, 0, s>>>(sum, mean, n_values, 1.0 / samples);
}

void pool_majorants(const float* fine, int lx, int ly, int lz, float* out, int mx, int my, int mz, int factor,
                    cudaStream_t s) {
    int n = mx * my * mz;
    pool_majorants_kernel<<<(n + 255) / 256, 256, 0, s>>>(fine, lx, ly, lz, out, mx, my, mz, factor);
}

size_t stage_smem_bytes(size_t maj_bytes, int threads) {
    const size_t warps = static_cast<size_t>(threads) / 32;
    return (maj_bytes + 127) / 128 * 128 + warps * (kLeafBytes + sizeof(uint64_t));
}

const void* stage_kernel_ptr(bool logged) {
    return logged ? reinterpret_cast<const void*>(staged_trace_kernel<true>)
                  : reinterpret_cast<const void*>(staged_trace_kernel<false>);
}

void launch_stage(const TraceParams& p, int grid_ctas, int threads, size_t smem, cudaStream_t s) {
    if (p.dlog)
        staged_trace_kernel<true><<<grid_ctas, threads, smem, s>>>(p);
    else
        staged_trace_kernel<false><<<grid_ctas, threads, smem, s>>>(p);
}

}  // namespace vpt
