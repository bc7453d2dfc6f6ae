// Building blocks shared by the forms of the persistent tracker: end codes and caps, the
// majorant-grid DDA, the records of the radiance-cache passes.
#pragma once

#include "vpt_tracer.cuh"

namespace vpt {
namespace {

enum : uint32_t {
    END_ESCAPE = 1,
    END_RR = 2,
    END_PDF_ZERO = 3,
    END_MAX_BOUNCES = 4,
    END_STEP_CAP = 5,
    END_CACHE = 6,       // radiance-cache passes: ended with a cache query
    END_TRAIN_FULL = 7,  // training pass: the training-vertex buffer was full
};

// Limits that apply even when the caller disables the configurable caps, so that no input
// (zero or non-finite majorants, albedo 1 in a huge medium) can keep a launch running forever.
constexpr uint32_t kHardStepCap = 1u << 24;
constexpr uint32_t kHardVertexCap = 1u << 16;
// RNG stream layout a kernel is compiled for; kStreamsRuntime follows TraceParams::stream_mode.
constexpr int kStreamsPerPixel = 0, kStreamsSampleParallel = 1, kStreamsRuntime = 2;

struct DdaState {
    int cell[3];
    int step[3];
    float tnext[3], tdelta[3];
};

// Majorant-grid DDA in index space. Cells are 2^maj_shift voxels wide; shared definition with
// the oracle's restatement (overshooting a cell's exit restarts sampling at the exit).
__device__ __forceinline__ void dda_init(const Grid& g, V3 eye, V3 dir, float t, DdaState* d) {
    float o[3] = {(eye.x - g.origin[0]) * g.inv_voxel_size, (eye.y - g.origin[1]) * g.inv_voxel_size,
                  (eye.z - g.origin[2]) * g.inv_voxel_size};
    float dd[3] = {dir.x * g.inv_voxel_size, dir.y * g.inv_voxel_size, dir.z * g.inv_voxel_size};
    int cdim[3] = {g.mx, g.my, g.mz};
    const float size = static_cast<float>(1 << g.maj_shift);
    const float inv_size = 1.0f / size;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        float p = o[a] + dd[a] * t;
        int c = static_cast<int>(floorf(p * inv_size));
        c = min(max(c, 0), cdim[a] - 1);
        d->cell[a] = c;
        if (dd[a] > 0) {
            d->step[a] = 1;
            d->tnext[a] = ((c + 1) * size - o[a]) / dd[a];
            d->tdelta[a] = size / dd[a];
        } else if (dd[a] < 0) {
            d->step[a] = -1;
            d->tnext[a] = (c * size - o[a]) / dd[a];
            d->tdelta[a] = -size / dd[a];
        } else {
            d->step[a] = 0;
            d->tnext[a] = INFINITY;
            d->tdelta[a] = INFINITY;
        }
    }
}

// tdelta of one axis (dda_init), from the index-space direction component.
__device__ __forceinline__ float dda_delta(float size, float d) {
    return d > 0 ? size / d : (d < 0 ? -size / d : INFINITY);
}

__device__ __forceinline__ float cell_maj(const float* maj, const Grid& g, const DdaState& d) {
    return maj[(d.cell[0] * g.my + d.cell[1]) * g.mz + d.cell[2]];
}

// The sign of a direction component: the DDA step along that axis (dda_init derives it from the
// same sign, the index-space direction being the world direction times a positive scale).
__device__ __forceinline__ int step_of(float d) { return d > 0 ? 1 : (d < 0 ? -1 : 0); }

// createRadianceQuery (optix_pathtracing_kernels.cu:14-29) for an in-medium vertex: position in
// the world box (basic_types.h:2835-2838), normal = vOut as toPolarYUp outputs (the first slot
// holds acos(y), the second the azimuth), roughness, diffuse = albedo, specular = 0.
__device__ __forceinline__ void write_query(float* q, V3 pos, V3 vout, float roughness, float albedo, V3 wmin, V3 wmax) {
    V3 d = wmax - wmin, r = pos - wmin;
    float a, b;
    to_polar_yup_sel(vout, &a, &b);
    float2* p = reinterpret_cast<float2*>(q);
    p[0] = make_float2(d.x != 0 ? r.x / d.x : 0.0f, d.y != 0 ? r.y / d.y : 0.0f);
    p[1] = make_float2(d.z != 0 ? r.z / d.z : 0.0f, a);
    p[2] = make_float2(b, a);
    p[3] = make_float2(b, roughness);
    p[4] = make_float2(albedo, albedo);
    p[5] = make_float2(albedo, 0.0f);
    p[6] = make_float2(0.0f, 0.0f);
}

// RadianceQuery of a surface vertex (optix_pathtracing_kernels.cu:14-29 with the BSDF's
// getSurfaceParameters, common_renderer_types.h:1491-1496 Lambert, 1671-1677 dichromatic):
// position in the world box, the shading normal and vOut as toPolarYUp outputs, roughness,
// diffuse and specular reflectance of the material.
__device__ __forceinline__ void write_query_surface(float* q, V3 pos, V3 normal, V3 vout, const SurfMaterial& m, V3 wmin,
                                                    V3 wmax) {
    V3 d = wmax - wmin, r = pos - wmin;
    float na, nb, va, vb;
    to_polar_yup_sel(normal, &na, &nb);
    to_polar_yup_sel(vout, &va, &vb);
    float2* p = reinterpret_cast<float2*>(q);
    p[0] = make_float2(d.x != 0 ? r.x / d.x : 0.0f, d.y != 0 ? r.y / d.y : 0.0f);
    p[1] = make_float2(d.z != 0 ? r.z / d.z : 0.0f, na);
    p[2] = make_float2(nb, va);
    p[3] = make_float2(vb, m.roughness);
    p[4] = make_float2(m.diffuse[0], m.diffuse[1]);
    p[5] = make_float2(m.diffuse[2], m.specular[0]);
    p[6] = make_float2(m.specular[1], m.specular[2]);
}

// Work order of the training pass: item -> pixel of the training image, class by class, where
// the class of a pixel is (its position in the 4x4 tile + offset) % 16 and class 0 holds the
// unbiased suffixes (optix_pathtracing_kernels.cu:60-66). The long unbiased paths thus gather in
// the first warps and CTAs, and the CTAs of the short biased suffixes retire early, freeing their
// SM slots for the render pass that runs concurrently. Records stay at the reference's pixel
// index; only the order in which the pixels are traced changes.
__device__ __forceinline__ void train_item_to_pixel(uint32_t item, uint32_t w, uint32_t h, uint32_t offset,
                                                    uint32_t* px, uint32_t* py) {
    const uint32_t off = offset % 16;
    for (uint32_t k = 0; k < 16; ++k) {
        const uint32_t p = (k + 16 - off) % 16;  // tile position with (p + offset) % 16 == k
        const uint32_t a = p % 4, b = p / 4;
        const uint32_t cx = w > a ? (w - a + 3) / 4 : 0, cy = h > b ? (h - b + 3) / 4 : 0;
        const uint32_t n = cx * cy;
        if (item < n) {
            *px = a + 4 * (item % cx);
            *py = b + 4 * (item / cx);
            return;
        }
        item -= n;
    }
    *px = 0;  // not reached for item < w * h
    *py = 0;
}

}  // namespace
}  // namespace vpt
