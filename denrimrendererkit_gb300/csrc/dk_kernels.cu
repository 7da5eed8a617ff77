// Wavefront kernels of the sm_103a progressive path tracer.
//
// The reference runs the whole path of a pixel-sample in one thread
// (pathTraceKernel, Sources/DenrimRendererKit/Resources/Shaders/
// PathTrace.metal:5167-5586).  Here one batch of paths (tile pixels x several
// sample indices) advances bounce by bounce through four stages over SoA path
// state in HBM:
//   k_generate  camera rays + RNG seeds              (:5204-5225)
//   k_extend    closest hit of every active ray      (intersectScene, :3294-3421)
//   k_shade     the bounce body: misses, materials, random walks, emission,
//               NEE ray generation, BSDF sampling, Russian roulette  (:5252-5518)
//   k_shadow    the NEE shadow queries and the clamped direct-light sum
//               (sampleDirectLighting, :4407-4585; shadowOccluded, :4196-4274)
//   k_finalize  Kahan-compensated accumulation + last-sample AOVs (:5520-5585)
// Surviving paths are compacted into the next queue with warp-ballot appends.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <type_traits>

#include "dk_kernels.h"
#include "dk_sdf.cuh"
#include "dk_shade.cuh"

namespace dk {

__device__ __forceinline__ uint32_t laneId() { return threadIdx.x & 31u; }

// Warp-aggregated append: one atomic per warp, order-stable within the warp.
__device__ __forceinline__ uint32_t warpAppend(uint32_t* counter, bool pred) {
    unsigned active = __activemask();
    unsigned ballot = __ballot_sync(active, pred);
    if (ballot == 0u) return 0u;
    int leader = __ffs(ballot) - 1;
    uint32_t base = 0;
    if ((int)laneId() == leader) base = atomicAdd(counter, (uint32_t)__popc(ballot));
    base = __shfl_sync(active, base, leader);
    unsigned lower = ballot & ((1u << laneId()) - 1u);
    return base + (uint32_t)__popc(lower);
}

// makeCameraRay (PathTrace.metal:4056-4091); pinhole arithmetic in exact ops.
__device__ Ray makeCameraRay(const dk_camera& cam, uint32_t width, uint32_t height, uint32_t gx, uint32_t gy, float jx,
                             float jy, float lx, float ly) {
    float u = ex::div(ex::add((float)gx, jx), (float)width);
    float v = ex::sub(1.0f, ex::div(ex::add((float)gy, jy), (float)height));
    float3 ll = f3(cam.lower_left.x, cam.lower_left.y, cam.lower_left.z);
    float3 hz = f3(cam.horizontal.x, cam.horizontal.y, cam.horizontal.z);
    float3 vt = f3(cam.vertical.x, cam.vertical.y, cam.vertical.z);
    float3 planePoint = ex::add(ex::add(ll, ex::mul(u, hz)), ex::mul(v, vt));
    Ray ray;
    if (cam.origin.w > 0.5f) {
        ray.origin = planePoint;
        ray.direction = ex::normalize(ex::cross(vt, hz));
    } else {
        ray.origin = f3(cam.origin.x, cam.origin.y, cam.origin.z);
        ray.direction = ex::normalize(ex::sub(planePoint, ray.origin));
    }
    float aperture = fmaxf(cam.lens.x, 0.0f);
    if (cam.origin.w <= 0.5f && aperture > 0.0f) {
        float3 forward = normalize(cross(vt, hz));
        float focus = fmaxf(cam.lens.y, 0.0001f);
        float focalT = focus / fmaxf(dot(ray.direction, forward), 0.0001f);
        float3 focal = ray.origin + ray.direction * focalT;
        float2 disk = uniformDisk(lx, ly);
        disk.x *= aperture;
        disk.y *= aperture;
        ray.origin += normalize(hz) * disk.x + normalize(vt) * disk.y;
        ray.direction = normalize(focal - ray.origin);
    }
    return ray;
}

// applyNormalMap (PathTrace.metal:4021-4054).
__device__ Hit applyNormalMap(const DevScene& S, Hit h, uint32_t idx, float3 rayDir) {
    float3 mapped = xyz(sampleTexture(S, idx, h.uv, make_float4(0.5f, 0.5f, 1.0f, 1.0f)));
    mapped = ex::normalize(ex::sub(ex::mul(mapped, 2.0f), f3(1.0f)));
    float3 t = ex::sub(h.tangent, ex::mul(h.normal, ex::dot(h.tangent, h.normal)));
    if (__fsqrt_rn(ex::dot(t, t)) <= 1e-5f) {
        float3 helper = fabsf(h.normal.y) < 0.999f ? f3(0, 1, 0) : f3(1, 0, 0);
        t = ex::cross(helper, h.normal);
    }
    t = ex::normalize(t);
    float3 b = ex::sub(h.bitangent, ex::mul(h.normal, ex::dot(h.bitangent, h.normal)));
    if (__fsqrt_rn(ex::dot(b, b)) <= 1e-5f) b = ex::cross(h.normal, t);
    b = ex::normalize(b);
    h.normal = ex::normalize(ex::add(ex::add(ex::mul(mapped.x, t), ex::mul(mapped.y, b)), ex::mul(mapped.z, h.normal)));
    if (ex::dot(h.normal, rayDir) > 0.0f) h.normal = -h.normal;
    return h;
}

__device__ __forceinline__ float4 exMix4(float4 a, float4 b, float t) {
    return make_float4(exMix(a.x, b.x, t), exMix(a.y, b.y, t), exMix(a.z, b.z, t), exMix(a.w, b.w, t));
}

// blendMaterials (:527-547): m = mix(m, materials[b], t) field by field.
__device__ __noinline__ void blendMaterialInto(Material& m, const dk_material* mats, uint32_t b, float t) {
    const float4* p = reinterpret_cast<const float4*>(mats + b);
    float4* f = reinterpret_cast<float4*>(&m);
#pragma unroll 1
    for (int k = 0; k < 17; ++k) f[k] = exMix4(f[k], __ldg(p + k), t);
}

// A render's material table: S.mats[base, base + count).
struct MatTable {
    uint32_t base, count;
};

__device__ __forceinline__ MatTable matTable(const DevJob& J) {
    return MatTable{__ldg(&J.mat_base), __ldg(&J.mat_count)};
}

// materialForHit (:1096-1121); the material-program VM and the field
// overrides are no-ops here (no programs, no material-field samples).
__device__ __forceinline__ Material materialForHit(const DevScene& S, MatTable mt, const Hit& h) {
    Material m = loadMaterial(S.mats, mt.base + min(h.materialID, mt.count - 1u));
    if (h.materialBlend > 0.0f)
        blendMaterialInto(m, S.mats, mt.base + min(h.materialID2, mt.count - 1u), clampf(h.materialBlend, 0.0f, 1.0f));
    return m;
}

__device__ __forceinline__ VolumeScene volumeScene(const DevScene& S) {
    VolumeScene V;
    V.volumes = S.volumes;
    V.bricks = S.bricks;
    V.samples = S.brick_samples;
    V.dist = DistSrc{S.brick_dist, S.brick_dist16};
    V.grids = S.brick_grids;
    V.gridIndices = S.brick_grid_indices;
    V.sampleCount = S.brick_sample_count;
    V.gridIndexCount = S.brick_grid_index_count;
    V.volumeCount = S.volume_count;
    V.brickCount = S.brick_count;
    V.gridCount = S.brick_grid_count;
    return V;
}

// Hit attributes of a distance-field hit at (t, brick): the tail of
// intersectVolumeBrickPrepared (PathTrace.metal:2741-2802).
__device__ __noinline__ Hit makeVolumeHit(const DevScene& S, const Ray& ray, float t, uint32_t brickIndex) {
    VolumeScene V = volumeScene(S);
    const dk_volume_brick_descriptor& brick = V.bricks[brickIndex];
    uint32_t vi = __ldg(&brick.grid_origin_and_volume.w);
    if (vi >= V.volumeCount) vi = 0;
    const dk_volume_descriptor& vol = V.volumes[vi];
    VolumeRay vr = volumeRay(vol, ray.origin, ray.direction);
    BrickCtx c = makeBrickCtx(brick, V.sampleCount);
    float3 rp = ex::add(vr.lo, ex::mul(vr.ld, t));
    bool cubic = vr.cellSize <= 0.03f;
    Hit h;
    h.t = t;
    h.position = ex::add(ray.origin, ex::mul(ray.direction, t));
    float3 n = brickNormal(V, vol, c, rp, cubic, !cubic);
    h.frontFacing = ex::dot(n, ray.direction) <= 0.0f;
    if (!h.frontFacing) n = -n;
    h.normal = n;
    h.uv = make_float2(0.0f, 0.0f);
    h.tangent = ex::normalize(ex::cross(fabsf(n.y) < 0.999f ? f3(0, 1, 0) : f3(1, 0, 0), n));
    h.bitangent = ex::normalize(ex::cross(n, h.tangent));
    // sampleVolumeBrickMaterial: nearest stored sample (:2319-2372)
    float3 uvw = clamp3(exDiv(ex::sub(rp, c.sampleMin), c.sampleExtent), f3(0.0f), f3(1.0f));
    uint32_t nx = min((uint32_t)roundf(ex::mul(uvw.x, (float)(c.dims[0] - 1u))), c.dims[0] - 1u);
    uint32_t ny = min((uint32_t)roundf(ex::mul(uvw.y, (float)(c.dims[1] - 1u))), c.dims[1] - 1u);
    uint32_t nz = min((uint32_t)roundf(ex::mul(uvw.z, (float)(c.dims[2] - 1u))), c.dims[2] - 1u);
    uint4 ms = __ldg(reinterpret_cast<const uint4*>(V.samples + c.sampleOffset + nx + ny * c.strideY + nz * c.strideZ));
    h.materialID = ms.y;
    h.materialID2 = ms.z;
    h.materialBlend = clampf(__uint_as_float(ms.w), 0.0f, 1.0f);
    h.objectID = __ldg(&vol.metadata.y);
    h.primitiveID = __ldg(&vol.metadata.z);
    return h;
}

__device__ __forceinline__ Hit makeHitAny(const DevScene& S, const Ray& ray, const HitRec& r) {
    if (r.tri == kVolumeHit) return makeVolumeHit(S, ray, r.t, __float_as_uint(r.u));
    return makeHit(S, ray, r);
}

// intersectScene (:3294-3421): triangles, then the sparse volumes with the
// triangle distance as the bound.  traceSceneCounting also counts the volume
// walk's events into the session's SDF traversal counters when it has them;
// the subsurface walk inside the shading kernel takes the plain form, which
// keeps that kernel's registers (its walk steps still count as scene queries).
__device__ __noinline__ HitRec traceScene(const DevScene& S, float3 o, float3 d) {
    HitRec r = S.wide8 ? traceClosest8(S, o, d) : traceClosest(S, o, d);
    if (S.volume_count) {
        VolumeHitRec vh;
        if (closestVolumeHit(volumeScene(S), o, d, r.t, vh)) {
            r.t = vh.t;
            r.tri = kVolumeHit;
            r.u = __uint_as_float(vh.brick);
            r.v = 0.0f;
        }
    }
    return r;
}
__device__ __noinline__ HitRec traceSceneCounting(const DevScene& S, float3 o, float3 d) {
    HitRec r = S.wide8 ? traceClosest8(S, o, d) : traceClosest(S, o, d);
    if (S.volume_count) {
        VolumeHitRec vh;
        if (closestVolumeHitAny(volumeScene(S), o, d, r.t, vh, S.sdf_counters)) {
            r.t = vh.t;
            r.tri = kVolumeHit;
            r.u = __uint_as_float(vh.brick);
            r.v = 0.0f;
        }
    }
    return r;
}

// The closest hit nearer than `tmax`; a record with t >= tmax is as good as a
// miss.  Scenes with volumes and the 8-wide tree take the unbounded query.
__device__ __noinline__ HitRec traceSceneWithin(const DevScene& S, float3 o, float3 d, float tmax) {
    if (S.wide8 || S.volume_count) return traceSceneCounting(S, o, d);
    return traceClosest(S, o, d, tmax);
}

// Subsurface walk helpers (PathTrace.metal:3490-3523).
__device__ __forceinline__ float sampleSubsurfaceFreeFlight(float3 sigmaT, float ux, float uy) {
    float sigma = sigmaT.z;
    if (ux < 0.33333333333f) sigma = sigmaT.x;
    else if (ux < 0.66666666667f) sigma = sigmaT.y;
    return -logf(fmaxf(1.0f - uy, 1e-6f)) / fmaxf(sigma, 1e-4f);
}
__device__ __forceinline__ float subsurfaceCollisionPDF(float3 s, float d) {
    float3 tr = exp3((-s) * d);
    return fmaxf((s.x * tr.x + s.y * tr.y + s.z * tr.z) * 0.33333333333f, 1e-6f);
}
__device__ __forceinline__ float subsurfaceBoundaryPDF(float3 s, float d) {
    float3 tr = exp3((-s) * d);
    return fmaxf((tr.x + tr.y + tr.z) * 0.33333333333f, 1e-6f);
}

// continueSubsurfaceRandomWalk (PathTrace.metal:3525-3621) inside the shading
// kernel, for scenes with volumes and the 8-wide tree; the others run
// k_subsurface_walk before shading.
__device__ bool continueSubsurfaceRandomWalk(const DevScene& S, const Hit& entry, const Material& m, Ray& ray,
                                             float3& tp, float& prevPdf, uint32_t& state) {
    if (materialSubsurface(m) <= 0.0f || !entry.frontFacing) return false;
    float e0 = randomFloat(state);
    float e1 = randomFloat(state);
    float3 entryDir = orientHemisphere(cosineHemisphere(e0, e1), -entry.normal);
    Ray medium{entry.position + entryDir * 0.001f, entryDir};
    float3 sigmaT = 1.0f / mx(xyz(m.subsurfaceRadius) * fmaxf(m.subsurfaceRadius.w, 0.0f), f3(1e-4f));
    float3 albedo = clamp3(xyz(m.subsurfaceColor), f3(0.0f), f3(0.999f));
    float anisotropy = clampf(m.subsurfaceParameters.x, -0.95f, 0.95f);
    for (uint32_t step = 0u; step < 8u; ++step) {
        sdfCount(S.sdf_counters, kSdfBounceSceneQueries);
        HitRec r = traceScene(S, medium.origin, medium.direction);
        if (r.tri == kNoHit) return false;
        float f0 = randomFloat(state);
        float f1 = randomFloat(state);
        float freeFlight = sampleSubsurfaceFreeFlight(sigmaT, f0, f1);
        if (freeFlight < r.t) {
            medium.origin += medium.direction * freeFlight;
            float h0 = randomFloat(state);
            float h1 = randomFloat(state);
            medium.direction = sampleHenyeyGreenstein(h0, h1, medium.direction, anisotropy);
            float3 tr = exp3((-sigmaT) * freeFlight);
            tp *= albedo * sigmaT * tr / subsurfaceCollisionPDF(sigmaT, freeFlight);
            if (maxComponent(tp) <= 1e-4f) return false;
            continue;
        }
        Hit b = makeHitAny(S, medium, r);
        float3 exitNormal = normalize(b.frontFacing ? b.normal : -b.normal);
        float x0 = randomFloat(state);
        float x1 = randomFloat(state);
        ray.direction = orientHemisphere(cosineHemisphere(x0, x1), exitNormal);
        ray.origin = b.position + exitNormal * 0.001f;
        float3 tr = exp3((-sigmaT) * r.t);
        tp *= tr / subsurfaceBoundaryPDF(sigmaT, r.t);
        prevPdf = fmaxf(dot(exitNormal, ray.direction), 0.0f) * 0.31830988618f;
        return true;
    }
    return false;
}

// continueTransmissionVolumeRandomWalk (PathTrace.metal:3685-3721).
__device__ bool continueTransmissionVolumeRandomWalk(const Hit& b, const Material& m, Ray& ray, float3& tp,
                                                     float& prevPdf, uint32_t& state) {
    if (b.frontFacing || !materialHasVolumeScattering(m)) return false;
    float3 sigmaT = materialVolumeSigmaT(m);
    float3 sigmaS = materialVolumeSigmaS(m);
    if (maxComponent(sigmaT) <= 1e-5f || maxComponent(sigmaS) <= 1e-5f) return false;
    float f0 = randomFloat(state);
    float f1 = randomFloat(state);
    float freeFlight = sampleSubsurfaceFreeFlight(sigmaT, f0, f1);
    if (freeFlight >= b.t) {
        tp *= exp3((-sigmaT) * b.t) / subsurfaceBoundaryPDF(sigmaT, b.t);
        return false;
    }
    float3 tr = exp3((-sigmaT) * freeFlight);
    tp *= sigmaS * tr / subsurfaceCollisionPDF(sigmaT, freeFlight);
    ray.origin += ray.direction * freeFlight;
    float h0 = randomFloat(state);
    float h1 = randomFloat(state);
    ray.direction = sampleHenyeyGreenstein(h0, h1, ray.direction, clampf(m.volumeParameters.y, -0.95f, 0.95f));
    ray.origin += ray.direction * 0.001f;
    prevPdf = 0.0f;
    return maxComponent(tp) > 1e-4f;
}

// continueTransmissiveSurface (PathTrace.metal:1723-1799).
__device__ bool continueTransmissiveSurface(const Hit& h, const Material& m, Ray& ray, float3& tp, float& prevPdf,
                                            uint32_t& state) {
    float transmission = materialTransmission(m);
    if (transmission <= 0.0f || randomFloat(state) > transmission) return false;
    float3 incoming = ray.direction;
    float3 view = -incoming;
    float roughness = clampf(m.parameters3.y, 0.001f, 1.0f);
    float ior = fmaxf(m.parameters3.z, 1.0001f);
    float3 micro = h.normal;
    if (roughness > 0.01f) {
        float a = randomFloat(state);
        float b = randomFloat(state);
        micro = sampleGGXHalfVector(a, b, h.normal, roughness);
        if (dot(micro, incoming) > 0.0f) micro = -micro;
    }
    float etaI = h.frontFacing ? 1.0f : ior;
    float etaT = h.frontFacing ? ior : 1.0f;
    float eta = etaI / etaT;
    float cosI = fmaxf(dot(view, micro), 0.0f);
    float fresnel = dielectricFresnel(cosI, etaI, etaT);
    if (materialThinWalled(m)) {
        fresnel = dielectricFresnel(cosI, 1.0f, ior);
        float rp = clampf(fresnel, 0.02f, 0.98f);
        if (randomFloat(state) < rp) {
            ray.direction = normalize(reflect(incoming, micro));
            ray.origin = h.position + micro * 0.001f;
            tp *= fresnel / fmaxf(rp, 1e-5f);
        } else {
            ray.direction = incoming;
            ray.origin = h.position + ray.direction * 0.001f;
            float grazing = 1.0f - fabsf(dot(view, h.normal));
            float tint = mixf(0.35f, 0.95f, grazing * grazing);
            tp *= materialTransmissionTint(m, tint) * ((1.0f - fresnel) / fmaxf(1.0f - rp, 1e-5f));
        }
        prevPdf = 0.0f;
        return true;
    }
    float3 refracted = refract(incoming, micro, eta);
    bool tir = dot(refracted, refracted) <= 1e-7f;
    float rp = tir ? 1.0f : clampf(fresnel, 0.02f, 0.98f);
    if (randomFloat(state) < rp) {
        ray.direction = normalize(reflect(incoming, micro));
        ray.origin = h.position + micro * 0.001f;
        tp *= tir ? 1.0f : fresnel / fmaxf(rp, 1e-5f);
    } else {
        ray.direction = normalize(refracted);
        ray.origin = h.position + ray.direction * 0.001f;
        float grazing = 1.0f - fabsf(dot(view, h.normal));
        float tint = mixf(0.35f, 0.95f, grazing * grazing);
        float w = (1.0f - fresnel) / fmaxf(1.0f - rp, 1e-5f);
        float3 absorption = materialTransmissionAbsorption(m, h.t, !h.frontFacing && !materialHasVolumeScattering(m));
        tp *= materialTransmissionTint(m, tint) * absorption * w;
    }
    prevPdf = 0.0f;
    return true;
}

// ================================================================ kernels ==

__device__ __forceinline__ uint32_t gridStride() { return gridDim.x * blockDim.x; }
__device__ __forceinline__ uint32_t globalId() { return blockIdx.x * blockDim.x + threadIdx.x; }

// The job whose [begin, next begin) range holds `i` (the last job whose
// begin <= i), by binary search over the wave's ascending job table.
__device__ __forceinline__ uint32_t jobOfPath(const Wave& W, uint32_t i) {
    uint32_t lo = 0, hi = W.job_count - 1u;
    while (lo < hi) {
        uint32_t mid = (lo + hi + 1u) >> 1;
        if (__ldg(&W.jobs[mid].path_begin) <= i) lo = mid; else hi = mid - 1u;
    }
    return lo;
}
__device__ __forceinline__ uint32_t jobOfPixel(const Wave& W, uint32_t i) {
    uint32_t lo = 0, hi = W.job_count - 1u;
    while (lo < hi) {
        uint32_t mid = (lo + hi + 1u) >> 1;
        if (__ldg(&W.jobs[mid].pixel_begin) <= i) lo = mid; else hi = mid - 1u;
    }
    return lo;
}
__device__ __forceinline__ uint32_t jobOf(const Wave& W, uint32_t p) { return W.rng[p].y >> 8; }

__device__ __forceinline__ void writeAovMiss(float4* aov, uint32_t local, uint32_t tileN) {
    aov[0 * (size_t)tileN + local] = make_float4(0.0f, 0.0f, 0.0f, __uint_as_float(0u));  // t, -, -, hasHit
    aov[1 * (size_t)tileN + local] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    aov[2 * (size_t)tileN + local] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    aov[3 * (size_t)tileN + local] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
}
__device__ __forceinline__ void writeAovHit(float4* aov, uint32_t local, uint32_t tileN, const Hit& h, float4 albedo) {
    aov[0 * (size_t)tileN + local] = make_float4(h.t, __uint_as_float(h.materialID), __uint_as_float(h.objectID), __uint_as_float(1u));
    aov[1 * (size_t)tileN + local] = make_float4(h.normal.x, h.normal.y, h.normal.z, 0.0f);
    aov[2 * (size_t)tileN + local] = albedo;
    aov[3 * (size_t)tileN + local] = make_float4(h.position.x, h.position.y, h.position.z, 0.0f);
}

__global__ void __launch_bounds__(256) k_generate(DevScene S, Wave W) {
    for (uint32_t p = globalId(); p < W.path_count; p += gridStride()) {
        uint32_t j = jobOfPath(W, p);
        const DevJob& J = W.jobs[j];
        const DevParams& P = J.P;
        const uint32_t tileN = P.tile_w * P.tile_h;
        uint32_t rel = p - J.path_begin;
        uint32_t slice = rel / tileN, local = rel - slice * tileN;
        uint32_t px = P.tile_x + local % P.tile_w, py = P.tile_y + local / P.tile_w;
        uint32_t sample = P.sample_begin + slice;
        uint32_t state = P.frame_seed ^ hash_u32(px + py * P.width) ^ hash_u32(sample + 1u);
        float j0 = randomFloat(state);
        float j1 = randomFloat(state);
        float j2 = randomFloat(state);
        float j3 = randomFloat(state);
        Ray ray = makeCameraRay(P.cam, P.width, P.height, px, py, j0, j1, j2, j3);
        W.ray_o[p] = make_float4(ray.origin.x, ray.origin.y, ray.origin.z, 0.0f);
        W.ray_d[p] = make_float4(ray.direction.x, ray.direction.y, ray.direction.z, 0.0f);
        W.tp[p] = make_float4(1.0f, 1.0f, 1.0f, 0.0f);
        W.rad[p] = make_float4(0.0f, 0.0f, 0.0f, 1.0f);
        W.rng[p] = make_uint2(state, j << 8);
        W.q[0][p] = p;
        if (slice == P.samples_in_batch - 1u) writeAovMiss(W.aov, J.pixel_begin + local, W.aov_stride);
    }
    if (globalId() == 0) {
        W.counts[0] = W.path_count;
        for (int k = 1; k < 8; ++k) W.counts[k] = 0u;
    }
}

constexpr uint32_t kNoWork = 0xffffffffu;
#ifndef DK_STEP_BUDGET
#define DK_STEP_BUDGET 16
#endif
constexpr int kStepBudget = DK_STEP_BUDGET;  // the 8-wide tree's visits between refills
// Idle lanes are refilled when fewer than this many of a warp's are running
// (8 / 12 / 16 / 24 / 28: 58.6 / 57.7 / 57.5 / 61.1 / 63.6 ms a frame, large
// scene at 16 spp).
#ifndef DK_REFILL_BELOW
#define DK_REFILL_BELOW 16
#endif
constexpr int kRefillBelow = DK_REFILL_BELOW;

// Refills the lanes that asked for work with consecutive items of a queue of
// length `n` through one atomic per warp; returns this lane's item or kNoWork.
__device__ __forceinline__ uint32_t warpFetch(uint32_t* counter, uint32_t n, bool need, bool& exhausted) {
    unsigned m = __ballot_sync(0xffffffffu, need);
    if (m == 0u) return kNoWork;
    int leader = __ffs(m) - 1;
    uint32_t base = 0;
    if ((int)laneId() == leader) base = atomicAdd(counter, (uint32_t)__popc(m));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (!need) return kNoWork;
    uint32_t idx = base + (uint32_t)__popc(m & ((1u << laneId()) - 1u));
    if (idx >= n) {
        exhausted = true;
        return kNoWork;
    }
    return idx;
}

// Closest hit for every ray of the input queue (intersectScene), persistent
// threads with per-lane refill.  W.counts[4] is the work cursor (zeroed by the
// kernel that runs before).
template <bool kWide8>
__global__ void __launch_bounds__(128) k_extend(DevScene S, Wave W, uint32_t sel, uint32_t bounce) {
    const uint32_t* q = W.q[sel];
    const uint32_t n = W.counts[sel];
    if (blockIdx.x == 0)
        for (uint32_t b = threadIdx.x; b < 2u * kSortBins; b += blockDim.x) W.bins[b] = 0u;
    if (globalId() == 0) {
        // one scene query per active path and bounce (PathTrace.metal:5252-5256)
        if (S.sdf_counters && n)
            atomicAdd(S.sdf_counters + (bounce == 0u ? kSdfPrimarySceneQueries : kSdfBounceSceneQueries),
                      (unsigned long long)n);
        W.counts[sel ^ 1u] = 0u;
        W.counts[2] = 0u;
        W.counts[3] = 0u;
        W.counts[5] = 0u;
        W.counts[6] = 0u;
        W.counts[7] = 0u;
        W.counts[8] = 0u;
    }
    if (S.node_count == 0) {  // no triangles: a volume-only scene
        for (uint32_t i = globalId(); i < n; i += gridStride())
            W.hit[q[i]] = make_float4(INFINITY, __uint_as_float(kNoHit), 0.0f, 0.0f);
        return;
    }
    // The stacks stay separate objects from the scalar state, so that only
    // they live in local memory.
    int stackNode[kWide8 ? 1 : kStackSize];
    float stackT[kWide8 ? 1 : kStackSize];
    uint2 stack8[kWide8 ? kTraversalStack : 1];
    std::conditional_t<kWide8, Closest8, ClosestState> st;
    uint32_t p = kNoWork;
    bool exhausted = false;
    for (;;) {
        uint32_t idx = warpFetch(&W.counts[4], n, p == kNoWork && !exhausted, exhausted);
        if (idx != kNoWork) {
            p = q[idx];
            float4 o = W.ray_o[p], d = W.ray_d[p];
            closestInit(st, xyz(o), xyz(d));
        }
        if (__all_sync(0xffffffffu, p == kNoWork && exhausted)) break;
        if constexpr (kWide8) {
            if (p != kNoWork && closestSteps(S, st, stack8, kStepBudget)) {
                W.hit[p] = make_float4(st.bestT, __uint_as_float(st.bestTri), st.bu, st.bv);
                p = kNoWork;
            }
        } else {
            const int least = __any_sync(0xffffffffu, exhausted) ? 1 : kRefillBelow;
            for (;;) {
                int running;
                const bool nodes = majorityStep(p != kNoWork, st.node, running);
                if (running < least) break;
                const bool leaf = (st.node & kLeafBit) != 0u;
                if (p == kNoWork || nodes == leaf) continue;
                if (!(leaf ? closestTriStep(S, st, stackNode, stackT) : closestNodeStep(S, st, stackNode, stackT))) {
                    W.hit[p] = make_float4(st.bestT, __uint_as_float(st.bestTri), st.bu, st.bv);
                    p = kNoWork;
                }
            }
        }
    }
}

// ------------------------------------------------ material ordering ----
// The active queue is reordered by material before shading (a counting sort
// on the hit's material ID), so the paths of a warp take the same BSDF
// branches and read the same material record.  The order of paths does not
// change any result: every path carries its own RNG state and pixel samples
// are accumulated in sample order.
// Keys: 0 a miss, 1 + material ID (at most kSortBins - 3), kSortBins - 2 a
// material with a subsurface weight (where k_subsurface_walk begins),
// kSortBins - 1 a distance-volume hit.
constexpr uint32_t kSubsurfaceKey = kSortBins - 2u;
__device__ __forceinline__ uint32_t shadeKey(const DevScene& S, const Wave& W, uint32_t p) {
    uint32_t tri = __float_as_uint(W.hit[p].y);
    if (tri == kNoHit) return 0u;
    if (tri >= S.tri_count) return kSortBins - 1u;  // distance-volume hits
    const uint32_t id = __ldg(&S.tris[tri].material_id);
    // the material the shading kernel loads, and materialSubsurface's own test
    const MatTable mt = matTable(W.jobs[W.rng[p].y >> 8]);
    const float4* q = reinterpret_cast<const float4*>(S.mats + mt.base + min(id, mt.count - 1u));
    Material m;
    m.emission = __ldg(q + 1);
    m.parameters = __ldg(q + 2);
    m.subsurfaceColor = __ldg(q + 12);
    if (materialSubsurface(m) > 0.0f) return kSubsurfaceKey;
    return 1u + min(id, kSortBins - 3u);
}

// Exclusive scan of one value per thread over a block of 256, and the sum.
__device__ __forceinline__ uint32_t blockExclusiveScan256(uint32_t v, uint32_t& total) {
    __shared__ uint32_t warpSums[8];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (uint32_t o = 1; o < 32u; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31u) warpSums[warp] = x;
    __syncthreads();
    uint32_t before = 0u;
    total = 0u;
#pragma unroll
    for (uint32_t w = 0; w < 8u; ++w) {
        const uint32_t c = warpSums[w];
        if (w < warp) before += c;
        total += c;
    }
    __syncthreads();
    return before + x - v;
}

__global__ void __launch_bounds__(256) k_sort_count(DevScene S, Wave W, uint32_t sel) {
    __shared__ uint32_t hist[kSortBins];
    for (uint32_t b = threadIdx.x; b < kSortBins; b += blockDim.x) hist[b] = 0u;
    __syncthreads();
    const uint32_t* q = W.q[sel];
    const uint32_t n = W.counts[sel];
    for (uint32_t i = globalId(); i < n; i += gridStride()) {
        uint32_t k = shadeKey(S, W, q[i]);
        W.keys[i] = k;
        atomicAdd(&hist[k], 1u);
    }
    __syncthreads();
    for (uint32_t b = threadIdx.x; b < kSortBins; b += blockDim.x)
        if (hist[b]) atomicAdd(&W.bins[b], hist[b]);
}

// Block b places its kItems x 256 queue entries stably: an entry's
// rank among the block's entries of its key follows queue order (in-warp
// ranks from __match_any_sync, warp offsets per key scanned in shared memory,
// kItems rounds of 256 entries in order), and one global reservation per
// (block, key) places the block's run.  The queue is in path order, so every
// run of a key holds increasing path indices -- neighbouring lanes of the
// shading kernel read neighbouring path state.  Every block scans the histogram
// itself: 256 counts cost less than a launch of one block that leaves the other
// SMs idle.
// kItems: 8 in large waves; 2 in waves of less than kSortSmall paths, whose few
// blocks would spend their time in the rounds.
constexpr uint32_t kSortSmall = 1u << 22;
template <uint32_t kItems>
__global__ void __launch_bounds__(256) k_sort_scatter(Wave W, uint32_t sel) {
    __shared__ uint32_t cnt[kSortBins];
    __shared__ uint32_t base[kSortBins];
    __shared__ uint32_t warpCnt[8][kSortBins];
    const uint32_t* q = W.q[sel];
    const uint32_t n = W.counts[sel];
    const uint32_t start = blockIdx.x * 256u * kItems;
    if (start >= n) return;  // uniform over the block
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t lanesBelow = (1u << lane) - 1u;
    cnt[tid] = 0u;  // kSortBins == blockDim.x
    uint32_t entries;
    const uint32_t first = blockExclusiveScan256(W.bins[tid], entries);  // of key `tid` in shading order
    if (blockIdx.x == 0u && tid == kSubsurfaceKey) W.counts[7] = first;
    uint32_t key[kItems], rank[kItems];
#pragma unroll
    for (uint32_t k = 0; k < kItems; ++k) {
#pragma unroll
        for (uint32_t w = 0; w < 8u; ++w) warpCnt[w][tid] = 0u;
        __syncthreads();
        const uint32_t i = start + k * 256u + tid;
        const bool valid = i < n;
        key[k] = valid ? W.keys[i] : kSortBins - 1u;
        const uint32_t peers = __match_any_sync(0xffffffffu, valid ? key[k] : 0xffffffffu);
        const uint32_t inWarp = __popc(peers & lanesBelow);
        if (valid && inWarp == 0u) warpCnt[warp][key[k]] = __popc(peers);
        __syncthreads();
        {  // thread `tid` scans key `tid` over the warps, after the earlier rounds
            uint32_t run = cnt[tid];
#pragma unroll
            for (uint32_t w = 0; w < 8u; ++w) {
                const uint32_t c = warpCnt[w][tid];
                warpCnt[w][tid] = run;
                run += c;
            }
            cnt[tid] = run;
        }
        __syncthreads();
        rank[k] = valid ? warpCnt[warp][key[k]] + inWarp : 0u;
        __syncthreads();
    }
    if (cnt[tid]) base[tid] = first + atomicAdd(&W.bins[kSortBins + tid], cnt[tid]);
    __syncthreads();
#pragma unroll
    for (uint32_t k = 0; k < kItems; ++k) {
        uint32_t i = start + k * 256u + tid;
        if (i < n) W.qsorted[base[key[k]] + rank[k]] = q[i];
    }
}

// ------------------------------------------ survivors in path order ----
// Shading writes a flag per path; the next bounce's queue is the flagged
// paths in increasing path order: a count per block of kLiveBlock paths, and a
// scatter of each block's paths after those of the blocks before it.  Every
// block adds up the counts before it itself, which saves a launch of one block
// while the others wait; the sums grow with the square of the blocks, so waves
// of more than kLiveDirect blocks (33.5 M paths) run that block's scan: 0.3 % of
// a frame of 268 M paths, nothing at 34 and 134 M, and bounded at the 537 M that
// a wave may have.  Path order keeps the extension stage's and (through the
// stable material sort) the shading stage's path-state accesses coalesced.
constexpr uint32_t kLiveDirect = 8192u;
inline uint32_t liveBlocks(const Wave& W) { return (W.path_count + kLiveBlock - 1u) / kLiveBlock; }
__device__ __forceinline__ uint32_t liveCount16(const Wave& W, uint32_t first, uint32_t n, uint32_t& bits) {
    bits = 0u;
    if (first + 16u <= n) {
        const uint4 v = *reinterpret_cast<const uint4*>(W.live + first);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (uint32_t j = 0; j < 4u; ++j)
#pragma unroll
            for (uint32_t b = 0; b < 4u; ++b) bits |= (((w[j] >> (8u * b)) & 0xffu) ? 1u : 0u) << (4u * j + b);
    } else {
        for (uint32_t j = 0; j < 16u && first + j < n; ++j) bits |= (W.live[first + j] ? 1u : 0u) << j;
    }
    return __popc(bits);
}

__global__ void __launch_bounds__(256) k_live_count(Wave W) {
    const uint32_t n = W.path_count;
    const uint32_t first = blockIdx.x * kLiveBlock + threadIdx.x * 16u;
    uint32_t bits, total;
    const uint32_t c = first < n ? liveCount16(W, first, n, bits) : 0u;
    blockExclusiveScan256(c, total);
    if (threadIdx.x == 0) W.scan[blockIdx.x] = total;
}

// Exclusive scan of the block counts (one block).
__global__ void __launch_bounds__(256) k_live_scan(Wave W, uint32_t blocks) {
    const uint32_t per = (blocks + 255u) / 256u, begin = threadIdx.x * per, end = min(begin + per, blocks);
    uint32_t sum = 0u, total;
    for (uint32_t b = begin; b < end; ++b) sum += W.scan[b];
    uint32_t before = blockExclusiveScan256(sum, total);
    for (uint32_t b = begin; b < end; ++b) {
        const uint32_t c = W.scan[b];
        W.scan[b] = before;
        before += c;
    }
}

__global__ void __launch_bounds__(256) k_live_scatter(Wave W, uint32_t sel) {
    const uint32_t n = W.path_count;
    const uint32_t first = blockIdx.x * kLiveBlock + threadIdx.x * 16u;
    uint32_t bits = 0u, total;
    const uint32_t c = first < n ? liveCount16(W, first, n, bits) : 0u;
    uint32_t sum = 0u, before;
    if (gridDim.x <= kLiveDirect) {
        for (uint32_t b = threadIdx.x; b < blockIdx.x; b += 256u) sum += W.scan[b];
        blockExclusiveScan256(sum, before);
    } else {
        before = W.scan[blockIdx.x];
    }
    uint32_t slot = before + blockExclusiveScan256(c, total);
    if (blockIdx.x == gridDim.x - 1u && threadIdx.x == 0u) W.counts[sel ^ 1u] = before + total;  // the next queue's length
    uint32_t* qNext = W.q[sel ^ 1u];
    while (bits) {
        const uint32_t j = __ffs(bits) - 1u;
        bits &= bits - 1u;
        qNext[slot++] = first + j;
    }
}

// ------------------------------------------------ subsurface walk ----
// continueSubsurfaceRandomWalk (PathTrace.metal:3525-3621) for the paths whose
// material has a subsurface weight, ahead of the shading kernel: up to eight
// rays inside the surface per path.  Persistent threads with per-lane refill,
// like k_extend: a warp advances its rays by majority steps, and a lane whose
// ray is done scatters, leaves or fetches the next path with the others that
// wait.  Inside the shading kernel the same walks kept 5.8 of a
// warp's 32 lanes busy and took 102 of the 159 ms of a 20-job serving mix whose
// largest image has such a material; with this kernel the mix takes 67 ms.
// The outcome goes to the path's NEE slots, which shading reads before it
// fills them: origin and outcome, direction and RNG state, throughput and pdf.
constexpr uint32_t kWalkNone = 0u;  // not entered: the weight's draw decided against it, or a back face
constexpr uint32_t kWalkExit = 1u;  // left the surface: the path goes on from there
constexpr uint32_t kWalkLost = 2u;  // absorbed, or no surface found: shading goes on with the state so far
__global__ void __launch_bounds__(128) k_subsurface_walk(DevScene S, Wave W, uint32_t sel, uint32_t sorted) {
    const uint32_t* q = sorted ? W.qsorted : W.q[sel];
    const uint32_t begin = sorted ? W.counts[7] : 0u, n = W.counts[sel] - begin;
    int stackNode[kStackSize];
    float stackT[kStackSize];
    ClosestState st;
    uint32_t i = kNoWork, state = 0u, mat = 0u, step = 0u;
    float3 tp = f3(0.0f);
    bool exhausted = false;
    for (;;) {
        uint32_t idx = warpFetch(&W.counts[8], n, i == kNoWork && !exhausted, exhausted);
        if (idx != kNoWork) {
            const uint32_t at = begin + idx, p = q[at];
            const float4 hr = W.hit[p];
            const uint32_t tri = __float_as_uint(hr.y);
            if (tri != kNoHit) {
                const uint2 rs = W.rng[p];
                const MatTable mt = matTable(W.jobs[rs.y >> 8]);
                const float4 ro = W.ray_o[p], rd = W.ray_d[p];
                const Ray ray{xyz(ro), xyz(rd)};
                Hit h = makeHit(S, ray, HitRec{hr.x, tri, hr.z, hr.w});
                mat = mt.base + min(h.materialID, mt.count - 1u);
                const Material m = loadMaterial(S.mats, mat);
                const float subsurface = materialSubsurface(m);
                if (subsurface > 0.0f) {
                    const uint32_t nIdx = (uint32_t)m.parameters.w, bIdx = (uint32_t)m.parameters.z;
                    if (nIdx != 0u) h = applyNormalMap(S, h, nIdx, ray.direction);
                    float alpha = m.baseColor.w;
                    if (bIdx != 0u)
                        alpha = ex::mul(alpha, sampleTexture(S, bIdx, h.uv, make_float4(1.0f, 1.0f, 1.0f, 1.0f)).w);
                    state = rs.x;
                    if (alpha <= 0.001f || !h.frontFacing || !(randomFloat(state) < subsurface)) {
                        W.nee_o[at] = make_float4(0.0f, 0.0f, 0.0f, __uint_as_float(kWalkNone));
                    } else {
                        float e0 = randomFloat(state);
                        float e1 = randomFloat(state);
                        float3 entryDir = orientHemisphere(cosineHemisphere(e0, e1), -h.normal);
                        closestInit(st, h.position + entryDir * 0.001f, entryDir);
                        tp = xyz(W.tp[p]);
                        step = 0u;
                        i = at;
                        sdfCount(S.sdf_counters, kSdfBounceSceneQueries);
                    }
                }
            }
        }
        if (__all_sync(0xffffffffu, i == kNoWork && exhausted)) break;
        // Advance the rays until as many lanes wait (for their event or for a new
        // path) as run, and to the last one once no new paths are left: events are
        // long code, worth sharing (the material scene, 1024 x 1024 x 1 spp, whose
        // paths are all fetched at once: 3.82 -> 3.73 ms a frame with the second).
        bool running = i != kNoWork;
        const bool last = __any_sync(0xffffffffu, exhausted);
        for (;;) {
            int count;
            const bool nodes = majorityStep(running, st.node, count);
            const int waiting = __popc(__ballot_sync(0xffffffffu, !running && !(i == kNoWork && exhausted)));
            if (last ? count == 0 : waiting >= count) break;
            const bool leaf = (st.node & kLeafBit) != 0u;
            if (!running || nodes == leaf) continue;
            running = leaf ? closestTriStep(S, st, stackNode, stackT) : closestNodeStep(S, st, stackNode, stackT);
        }
        if (i == kNoWork || running) continue;
        uint32_t outcome = kWalkLost;
        float3 origin = st.o, direction = st.d;
        float pdf = 0.0f;
        bool again = false;
        if (st.bestTri != kNoHit) {
            const float4* mp = reinterpret_cast<const float4*>(S.mats + mat);
            Material m;
            m.subsurfaceColor = __ldg(mp + 12);
            m.subsurfaceRadius = __ldg(mp + 13);
            m.subsurfaceParameters = __ldg(mp + 14);
            float3 sigmaT = 1.0f / mx(xyz(m.subsurfaceRadius) * fmaxf(m.subsurfaceRadius.w, 0.0f), f3(1e-4f));
            float f0 = randomFloat(state);
            float f1 = randomFloat(state);
            float freeFlight = sampleSubsurfaceFreeFlight(sigmaT, f0, f1);
            if (freeFlight < st.bestT) {
                float3 albedo = clamp3(xyz(m.subsurfaceColor), f3(0.0f), f3(0.999f));
                origin += direction * freeFlight;
                float h0 = randomFloat(state);
                float h1 = randomFloat(state);
                direction = sampleHenyeyGreenstein(h0, h1, direction, clampf(m.subsurfaceParameters.x, -0.95f, 0.95f));
                float3 tr = exp3((-sigmaT) * freeFlight);
                tp *= albedo * sigmaT * tr / subsurfaceCollisionPDF(sigmaT, freeFlight);
                again = !(maxComponent(tp) <= 1e-4f) && ++step < 8u;
            } else {
                Hit b = makeHit(S, Ray{origin, direction}, HitRec{st.bestT, st.bestTri, st.bu, st.bv});
                float3 exitNormal = normalize(b.frontFacing ? b.normal : -b.normal);
                float x0 = randomFloat(state);
                float x1 = randomFloat(state);
                float bt = st.bestT;
                direction = orientHemisphere(cosineHemisphere(x0, x1), exitNormal);
                origin = b.position + exitNormal * 0.001f;
                float3 tr = exp3((-sigmaT) * bt);
                tp *= tr / subsurfaceBoundaryPDF(sigmaT, bt);
                pdf = fmaxf(dot(exitNormal, direction), 0.0f) * 0.31830988618f;
                outcome = kWalkExit;
            }
        }
        if (again) {
            closestInit(st, origin, direction);
            sdfCount(S.sdf_counters, kSdfBounceSceneQueries);
            continue;
        }
        W.nee_o[i] = make_float4(origin.x, origin.y, origin.z, __uint_as_float(outcome));
        W.nee_d[i] = make_float4(direction.x, direction.y, direction.z, __uint_as_float(state));
        W.nee_c[i] = make_float4(tp.x, tp.y, tp.z, pdf);
        i = kNoWork;
    }
}

struct ShadeOut { bool survive; uint32_t neeMask; uint32_t maxBounces; };

// The body of the reference bounce loop (PathTrace.metal:5252-5518) for one
// path whose closest hit is already in W.hit.
// kVolumes: with the subsurface random walk; without, k_subsurface_walk has
// left its outcome in the path's NEE slots.
template <bool kVolumes>
__device__ ShadeOut shadePath(const DevScene& S, const Wave& W, uint32_t p, uint32_t i, uint32_t bounce) {
    float4 ro = W.ray_o[p], rd = W.ray_d[p], tpw = W.tp[p], radw = W.rad[p], hr = W.hit[p];
    uint2 rs = W.rng[p];
    const DevJob& J = W.jobs[rs.y >> 8];
    const DevParams& P = J.P;
    ShadeOut out{false, 0u, P.max_bounces};
    Ray ray{xyz(ro), xyz(rd)};
    float3 tp = xyz(tpw);
    float prevPdf = tpw.w;
    float3 rad = xyz(radw);
    float alpha = radw.w;
    uint32_t state = rs.x, flags = rs.y;
    bool primaryFound = (flags & 1u) != 0u;
    uint32_t tri = __float_as_uint(hr.y);

    if (tri == kNoHit) {  // :5279-5305
        if (P.transparent_background != 0u && !primaryFound) {
            alpha = 0.0f;
        } else if (P.shows_env_bg == 0u && !primaryFound) {
            alpha = 1.0f;
            rad += mx(f3(P.bg[0], P.bg[1], P.bg[2]), f3(0.0f));
        } else {
            float envWeight = 1.0f;
            if (bounce > 0u && prevPdf > 0.0f) envWeight = powerHeuristic(prevPdf, environmentPDF(S, ray.direction));
            rad += clampSampleContribution(tp * sampleEnvironment(S, ray.direction) * envWeight, P.clamp);
        }
        W.rad[p] = make_float4(rad.x, rad.y, rad.z, alpha);
        return out;
    }
    HitRec rec{hr.x, tri, hr.z, hr.w};
    Hit h = kVolumes ? makeHitAny(S, ray, rec) : makeHit(S, ray, rec);
    const MatTable mt = matTable(J);
    Material m = kVolumes ? materialForHit(S, mt, h) : loadMaterial(S.mats, mt.base + min(h.materialID, mt.count - 1u));
    uint32_t nIdx = (uint32_t)m.parameters.w;
    if (nIdx != 0u) h = applyNormalMap(S, h, nIdx, ray.direction);
    uint32_t bIdx = (uint32_t)m.parameters.z;
    if (bIdx != 0u) {
        float4 texel = sampleTexture(S, bIdx, h.uv, make_float4(1.0f, 1.0f, 1.0f, 1.0f));
        m.baseColor = make_float4(ex::mul(m.baseColor.x, texel.x), ex::mul(m.baseColor.y, texel.y),
                                  ex::mul(m.baseColor.z, texel.z), ex::mul(m.baseColor.w, texel.w));
    }
    if (m.baseColor.w <= 0.001f) {  // cut-out: pass through (:5318-5321)
        ray.origin = ex::add(h.position, ex::mul(ray.direction, 0.001f));
        W.ray_o[p] = make_float4(ray.origin.x, ray.origin.y, ray.origin.z, 0.0f);
        out.survive = true;
        return out;
    }
    if (!primaryFound) {
        flags |= 1u;
        const uint32_t tileN = P.tile_w * P.tile_h;
        uint32_t rel = p - J.path_begin;
        uint32_t slice = rel / tileN;
        if (slice == P.samples_in_batch - 1u && P.denoiser == 0u)
            writeAovHit(W.aov, J.pixel_begin + (rel - slice * tileN), W.aov_stride, h, m.baseColor);
    }

    bool continued = false;
    if (continueTransmissionVolumeRandomWalk(h, m, ray, tp, prevPdf, state)) {
        continued = true;
    } else {
        float subsurface = materialSubsurface(m);
        if constexpr (kVolumes) {
            continued = subsurface > 0.0f && randomFloat(state) < subsurface &&
                        continueSubsurfaceRandomWalk(S, h, m, ray, tp, prevPdf, state);
        } else if (subsurface > 0.0f) {
            const float4 wo = W.nee_o[i];
            const uint32_t walk = __float_as_uint(wo.w);
            if (walk == kWalkNone) {
                randomFloat(state);  // the draw that decided against the walk
            } else {
                const float4 wd = W.nee_d[i], wt = W.nee_c[i];
                state = __float_as_uint(wd.w);
                tp = xyz(wt);
                if (walk == kWalkExit) {
                    ray.origin = xyz(wo);
                    ray.direction = xyz(wd);
                    prevPdf = wt.w;
                    continued = true;
                }
            }
        }
        if (!continued) continued = continueTransmissiveSurface(h, m, ray, tp, prevPdf, state);
    }
    if (continued) {
        bool dead = terminatePathWithRussianRoulette(bounce, tp, state);
        W.ray_o[p] = make_float4(ray.origin.x, ray.origin.y, ray.origin.z, 0.0f);
        W.ray_d[p] = make_float4(ray.direction.x, ray.direction.y, ray.direction.z, 0.0f);
        W.tp[p] = make_float4(tp.x, tp.y, tp.z, prevPdf);
        W.rng[p] = make_uint2(state, flags);
        out.survive = !dead;
        return out;
    }

    float3 emission = xyz(m.emission);
    if (maxComponent(emission) > 0.0f) {  // :5376-5392
        float w = 1.0f;
        if (bounce > 0u && prevPdf > 0.0f) w = powerHeuristic(prevPdf, lightPDFForHit(S, h, ray.direction));
        rad += clampSampleContribution(tp * emission * w, P.clamp);
        W.rad[p] = make_float4(rad.x, rad.y, rad.z, alpha);
        return out;
    }

    // ------------------------------------ NEE (sampleDirectLighting) ------
    float3 view = -ray.direction;
    ShadePoint sp;
    makeShadePoint(sp, m, h.normal, h.tangent, h.bitangent, view);
    float3 shadowOrigin = h.position + h.normal * 0.001f;
    const size_t cap = W.cap;
    // NEE slots are indexed by shading order `i` (coalesced); the slot's
    // direction.w carries the path's job, nee_tp.w the slot mask | path << 3.
    const float jobBits = __uint_as_float(rs.y >> 8);
    if (S.light_count > 0u) {
        uint32_t index = selectLightIndex(S, randomFloat(state));
        const dk_light_record& L = S.lights[index];
        float selPdf = lightSelectionPDF(S, index);
        uint32_t lti = __ldg(&L.triangle_index);
        if (lti < S.tri_count && selPdf > 0.0f) {
            uint32_t lmi = min(__ldg(&L.material_index), S.mat_count - 1u);
            float3 le = xyz(__ldg(reinterpret_cast<const float4*>(S.mats + lmi) + 1));
            float area = __ldg(&L.area);
            if (area > 0.0f) {
                float r0 = randomFloat(state);
                float r1 = randomFloat(state);
                float3 lp = sampleTriangle(S.tris[lti], r0, r1);
                float3 toL = lp - h.position;
                float d2 = dot(toL, toL);
                float dist = sqrtf(d2);
                float3 ld = toL / dist;
                float cosS = fmaxf(0.0f, dot(h.normal, ld));
                float cosL = fmaxf(0.0f, dot(xyz(__ldg(reinterpret_cast<const float4*>(&L.normal))), -ld));
                if (cosS > 0.0f && cosL > 0.0f) {
                    float lightPdf = selPdf * (d2 / fmaxf(cosL * area, 1e-6f));
                    float bsdfPdf = bsdfPDF(sp, ld);
                    float mis = powerHeuristic(lightPdf, bsdfPdf);
                    float G = cosS * cosL * area / fmaxf(d2, 1e-6f);
                    float3 c = evalBRDF(m, sp, ld) * le * G * mis;
                    if (!(c.x == 0.0f && c.y == 0.0f && c.z == 0.0f)) {
                        W.nee_o[i] = make_float4(shadowOrigin.x, shadowOrigin.y, shadowOrigin.z, dist - 0.002f);
                        W.nee_d[i] = make_float4(ld.x, ld.y, ld.z, jobBits);
                        W.nee_c[i] = make_float4(c.x, c.y, c.z, selPdf);
                        out.neeMask |= 1u;
                    }
                }
            }
        }
    }
#pragma unroll 1
    for (uint32_t e = 0u; e < 2u; ++e) {
        float a = randomFloat(state);
        float b = randomFloat(state);
        float cdf = randomFloat(state);
        float envPdf;
        float3 dir = sampleEnvironmentDirection(S, a, b, cdf, envPdf);
        float cosS = fmaxf(0.0f, dot(h.normal, dir));
        if (envPdf > 0.0f && cosS > 0.0f) {
            float bsdfPdf = bsdfPDF(sp, dir);
            float mis = powerHeuristic(envPdf, bsdfPdf);
            float3 c = evalBRDF(m, sp, dir) * sampleEnvironment(S, dir) * cosS * mis;
            if (!(c.x == 0.0f && c.y == 0.0f && c.z == 0.0f)) {
                size_t slot = (size_t)(1u + e) * cap + i;
                W.nee_o[slot] = make_float4(shadowOrigin.x, shadowOrigin.y, shadowOrigin.z, 1.0e20f);
                W.nee_d[slot] = make_float4(dir.x, dir.y, dir.z, jobBits);
                W.nee_c[slot] = make_float4(c.x, c.y, c.z, envPdf * 2.0f);
                out.neeMask |= 2u << e;
            }
        }
    }
    if (out.neeMask) W.nee_tp[i] = make_float4(tp.x, tp.y, tp.z, __uint_as_float(out.neeMask | (p << 3)));

    // --------------------------------------------- BSDF sampling ----------
    float c0 = randomFloat(state);
    float c1 = randomFloat(state);
    float3 diffuseDir = orientHemisphere(cosineHemisphere(c0, c1), h.normal);
    float lobe = randomFloat(state);
    float3 next;
    if (lobe < sp.cP) {
        float a = randomFloat(state);
        float b = randomFloat(state);
        float3 hv = sampleVNDF(sp, a, b, sp.ccAlpha);
        next = normalize(reflect(ray.direction, hv));
        if (dot(next, h.normal) <= 0.0f) {
            next = diffuseDir;
            tp *= diffuseBounceWeight(m, sp, next) / fmaxf(sp.dP, 1e-5f);
        } else {
            float nDotL = fmaxf(dot(h.normal, next), 1e-5f);
            float vDotH = fmaxf(dot(view, hv), 1e-5f);
            tp *= sp.clearcoat * fresnelSchlickThinFilm(vDotH, sp.ccF0, m) * geometrySmithG1GGX(nDotL, sp.ccR) /
                  fmaxf(sp.cP, 1e-5f);
        }
    } else if (lobe < sp.cP + sp.sP) {
        float a = randomFloat(state);
        float b = randomFloat(state);
        float3 hv = sampleVNDF(sp, a, b, sp.specAlpha);
        next = normalize(reflect(ray.direction, hv));
        if (dot(next, h.normal) <= 0.0f) {
            next = diffuseDir;
            tp *= diffuseBounceWeight(m, sp, next) / fmaxf(sp.dP, 1e-5f);
        } else {
            float vDotH = fmaxf(dot(view, hv), 1e-5f);
            float3 fres = fresnelSchlickThinFilm(vDotH, sp.f0, m);
            float3 cca = materialClearcoatAttenuationForDirection(m, h.normal, view, next);
            // The reference passes the raw tangent / bitangent here (PathTrace.metal:5486-5493).
            tp *= cca * fres *
                  geometrySmithG1GGXAnisotropic(next, h.normal, h.tangent, h.bitangent, sp.roughness, sp.anisotropy) /
                  fmaxf(sp.sP, 1e-5f);
        }
    } else {
        next = diffuseDir;
        tp *= diffuseBounceWeight(m, sp, next) / fmaxf(sp.dP, 1e-5f);
    }
    prevPdf = bsdfPDF(sp, next);
    ray.origin = shadowOrigin;
    ray.direction = next;
    bool dead = terminatePathWithRussianRoulette(bounce, tp, state);
    W.ray_o[p] = make_float4(ray.origin.x, ray.origin.y, ray.origin.z, 0.0f);
    W.ray_d[p] = make_float4(ray.direction.x, ray.direction.y, ray.direction.z, 0.0f);
    W.tp[p] = make_float4(tp.x, tp.y, tp.z, prevPdf);
    W.rng[p] = make_uint2(state, flags);
    out.survive = !dead;
    return out;
}

// Shading is bound by load latency and, at 200 to 500 KB of code, by
// instruction fetch.  A barrier per path keeps a block's warps near each other
// in the code, so that a fetched line serves all of them: on the large scene
// 66.4 -> 62.4 ms a frame (1920 x 1080, 16 spp) with blocks of 128 or 256
// threads, 63.8 with 512; without the barrier block size makes no difference.
// The kernel for volumes and the 8-wide tree, whose paths differ more (it
// traces rays), has 128 threads and no barrier (24.4 -> 25.1 ms a frame with
// it).
#ifndef DK_SHADE_BLOCK
#define DK_SHADE_BLOCK 256
#endif
#ifndef DK_SHADE_WARPS
#define DK_SHADE_WARPS 16
#endif
template <bool kVolumes>
constexpr int shadeBlock() { return kVolumes ? 128 : DK_SHADE_BLOCK; }
template <bool kVolumes>
__global__ void __launch_bounds__(shadeBlock<kVolumes>(), DK_SHADE_WARPS * 32 / shadeBlock<kVolumes>())
    k_shade(DevScene S, Wave W, uint32_t bounce, uint32_t sel, uint32_t sorted) {
    const uint32_t* q = sorted ? W.qsorted : W.q[sel];
    const uint32_t n = W.counts[sel];
    if (globalId() == 0) W.counts[4] = 0u;  // extend cursor of the next bounce
    for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += gridStride()) {
        const uint32_t i = base + threadIdx.x;
        if (!kVolumes) __syncthreads();
        if (i >= n) continue;
        uint32_t p = q[i];
        ShadeOut o = shadePath<kVolumes>(S, W, p, i, bounce);
        bool keep = o.survive && bounce + 1u < o.maxBounces;
        W.live[p] = keep ? 1u : 0u;  // the next queue is built from these flags in path order
        bool sh = o.neeMask != 0u;
        uint32_t sslot = warpAppend(&W.counts[2], sh);
        if (sh) W.qs[sslot] = i;
        for (uint32_t k = 0; k < 3u; ++k) {
            bool has = (o.neeMask >> k) & 1u;
            uint32_t r = warpAppend(&W.counts[3], has);
            if (has) W.qr[r] = (i << 2) | k;
        }
    }
}

// The ordered walk of shadowOccluded (PathTrace.metal:4196-4274) over layers
// collected in (distance, reference slot) order -- the order the reference's
// repeated closest-hit queries meet them: restart 0.001 past each layer,
// transmittance below 0.02 occludes.
__device__ __noinline__ bool walkLayers(const DevScene& S, MatTable mt, float3 o, float3 d, const float* lt,
                                        const uint32_t* ltri, const float* lu, const float* lv, int count, float3& T) {
    float prev = 0.0f;
    bool started = false;
    Ray ray{o, d};
    for (int i = 0; i < count; ++i) {
        float a = lt[i];
        if (started && a <= prev + 0.0015f) continue;  // inside the 0.001 restart gap + 0.0005 epsilon
        float trel = started ? a - (prev + 0.001f) : a;
        HitRec r{a, ltri[i], lu[i], lv[i]};
        Hit h = makeHit(S, ray, r);
        Material sm = materialForHit(S, mt, h);
        prev = a;
        started = true;
        if (sm.baseColor.w <= 0.001f) continue;
        float transmission = materialTransmission(sm);
        bool insideSolid = !h.frontFacing && !materialThinWalled(sm);
        float3 medium = (materialHasVolumeScattering(sm) && insideSolid)
                            ? exp3((-materialVolumeSigmaT(sm)) * trel)
                            : materialTransmissionAbsorption(sm, trel, insideSolid);
        T *= materialTransmissionTint(sm, 0.35f) * medium * transmission;
        if (maxComponent(T) < 0.02f) return true;
    }
    return false;
}

// Inserts a layer into (t, slot) order.
__device__ __forceinline__ void insertLayer(float* lt, uint32_t* ltri, uint32_t* lslot, float* lu, float* lv,
                                            int& count, float t, uint32_t tri, uint32_t slot, float u, float v) {
    int j = count++;
    while (j > 0 && (lt[j - 1] > t || (lt[j - 1] == t && lslot[j - 1] > slot))) {
        lt[j] = lt[j - 1];
        ltri[j] = ltri[j - 1];
        lslot[j] = lslot[j - 1];
        lu[j] = lu[j - 1];
        lv[j] = lv[j - 1];
        --j;
    }
    lt[j] = t;
    ltri[j] = tri;
    lslot[j] = slot;
    lu[j] = u;
    lv[j] = v;
}

// shadowOccluded for scenes with cut-out or transmissive triangles, in one
// traversal: an opaque blocker anywhere in (0.0005, maxDistance) occludes;
// otherwise the non-opaque layers are collected and walked.
// The same collecting traversal over the 8-wide tree.
__device__ __noinline__ bool shadowLayers8(const DevScene& S, MatTable mt, uint32_t opaqueMask, float3 o, float3 d,
                                           float tmax, float3& T) {
    constexpr int kMaxLayers = 8;
    float lt[kMaxLayers];
    uint32_t ltri[kMaxLayers], lslot[kMaxLayers];
    float lu[kMaxLayers], lv[kMaxLayers];
    int count = 0;
    if (S.node_count == 0) return false;
    Trav tr;
    uint2 stack[kTraversalStack];
    travInit(tr, o, d);
    float tm = tmax;
    int r = travSteps(S, tr, stack, tm, 1 << 30, [&](uint32_t i, float&) {
        const float4* q = S.isect + 3 * (size_t)i;
        const float4 a = __ldg(q + 0), b = __ldg(q + 1), c = __ldg(q + 2);
        float t, u, v;
        if (!triTest(S, o, d, a, b, c, t, u, v) || !(t < tmax)) return false;
        if (blocksShadow(__float_as_uint(c.w), opaqueMask)) return true;  // opaque blocker
        if (count == kMaxLayers - 1) return true;                        // an 8th layer: the walk ends occluded
        insertLayer(lt, ltri, lslot, lu, lv, count, t, __float_as_uint(b.w), __float_as_uint(a.w), u, v);
        return false;
    });
    if (r == 2) return true;
    return walkLayers(S, mt, o, d, lt, ltri, lu, lv, count, T);
}

__device__ bool shadowLayers(const DevScene& S, MatTable mt, uint32_t opaqueMask, float3 o, float3 d, float tmax,
                             float3& T) {
    if (S.wide8) return shadowLayers8(S, mt, opaqueMask, o, d, tmax, T);
    constexpr int kMaxLayers = 8;
    float lt[kMaxLayers];
    uint32_t ltri[kMaxLayers], lslot[kMaxLayers];
    float lu[kMaxLayers], lv[kMaxLayers];
    int count = 0;
    float3 inv = rcp3(d);
    int stackNode[kStackSize];
    int sp = 0;
    uint32_t node = 0;
    if (S.node_count == 0) return false;
    for (;;) {
        if ((node & kLeafBit) == 0) {
            Wide w;
            int k = wideVisit(S, node, o, inv, tmax, w);
            if (k > 0) {
                if (k > 3) stackNode[sp++] = (int)w.c3;
                if (k > 2) stackNode[sp++] = (int)w.c2;
                if (k > 1) stackNode[sp++] = (int)w.c1;
                node = w.c0;
                continue;
            }
        } else {
            uint32_t first = (node & ~kLeafBit) >> 3;
            uint32_t cnt = (node & 7u) + 1u;
            for (uint32_t i = first; i < first + cnt; ++i) {
                const float4* q = S.isect + 3 * (size_t)i;
                float4 a = __ldg(q + 0), b = __ldg(q + 1), c = __ldg(q + 2);
                float t, u, v;
                if (!triTest(S, o, d, a, b, c, t, u, v) || !(t < tmax)) continue;
                if (blocksShadow(__float_as_uint(c.w), opaqueMask)) return true;  // opaque blocker
                if (count == kMaxLayers - 1) return true;    // an 8th layer: the walk ends occluded
                insertLayer(lt, ltri, lslot, lu, lv, count, t, __float_as_uint(b.w), __float_as_uint(a.w), u, v);
            }
        }
        if (sp == 0) break;
        node = (uint32_t)stackNode[--sp];
    }
    return walkLayers(S, mt, o, d, lt, ltri, lu, lv, count, T);
}

// The same walk over the (at most kRecLayers) layers the any-hit pass
// recorded: each recorded triangle slot is intersected again with the same
// arithmetic, which reproduces its (t, u, v).
__device__ bool recordedLayers(const DevScene& S, MatTable mt, float3 o, float3 d, const uint2* rec, uint32_t n,
                               float3& T) {
    float lt[kRecLayers];
    uint32_t ltri[kRecLayers], lslot[kRecLayers];
    float lu[kRecLayers], lv[kRecLayers];
    int count = 0;
    for (uint32_t k = 0; k < n && k < kRecLayers; ++k) {
        const float4* q = S.isect + 3 * (size_t)rec[k].y;
        float4 a = __ldg(q + 0), b = __ldg(q + 1), c = __ldg(q + 2);
        float t, u, v;
        if (!triTest(S, o, d, a, b, c, t, u, v)) continue;
        insertLayer(lt, ltri, lslot, lu, lv, count, t, __float_as_uint(b.w), __float_as_uint(a.w), u, v);
    }
    return walkLayers(S, mt, o, d, lt, ltri, lu, lv, count, T);
}

// shadowOccluded (PathTrace.metal:4196-4274) exactly as the reference walks
// it — closest hit per layer, including distance-field hits — for scenes with
// sparse volumes whose layers the single-pass collection does not model.
__device__ bool shadowWalk(const DevScene& S, MatTable mt, float3 o, float3 d, float maxDistance, float3& T) {
    float traveled = 0.0f;
    for (uint32_t step = 0; step < 8u; ++step) {
        sdfCount(S.sdf_counters, kSdfShadowSceneQueries);
        HitRec r = traceSceneCounting(S, o, d);
        if (r.tri == kNoHit || traveled + r.t >= maxDistance) return false;
        Ray ray{o, d};
        Hit h = makeHitAny(S, ray, r);
        Material sm = materialForHit(S, mt, h);
        if (sm.baseColor.w <= 0.001f) {
            traveled += r.t;
            o = h.position + d * 0.001f;
            continue;
        }
        float transmission = materialTransmission(sm);
        if (transmission <= 0.001f) return true;
        bool insideSolid = !h.frontFacing && !materialThinWalled(sm);
        float3 medium = (materialHasVolumeScattering(sm) && insideSolid)
                            ? exp3((-materialVolumeSigmaT(sm)) * r.t)
                            : materialTransmissionAbsorption(sm, r.t, insideSolid);
        T *= materialTransmissionTint(sm, 0.35f) * medium * transmission;
        if (maxComponent(T) < 0.02f) return true;
        traveled += r.t;
        o = h.position + d * 0.001f;
    }
    return true;
}

// Distance-volume closest hit for every ray of the queue, bounded by the
// triangle hit k_extend found (the volume half of intersectScene): the general
// form, one ray per thread over the scene's volumes.  With the session's
// traversal counters (kStats) a single volume is walked by persistent threads
// with per-lane refill, `kCountedCells` cells at a time (W.counts[8] is the
// cursor); without them it runs k_volume_march.
constexpr int kCountedCells = 256;
template <bool kStats>
__global__ void __launch_bounds__(128, 4) k_extend_volume(DevScene S, Wave W, uint32_t sel) {
    const uint32_t* q = W.q[sel];
    const uint32_t n = W.counts[sel];
    VolumeScene V = volumeScene(S);
    DDAGrid g;
    if (!kStats || !(V.volumeCount == 1u && V.gridCount != 0u && V.gridIndexCount != 0u &&
                     V.volumes[0].metadata.w == 1u && ddaGrid(V, 0u, g))) {
        for (uint32_t i = globalId(); i < n; i += gridStride()) {
            uint32_t p = q[i];
            float4 o = W.ray_o[p], d = W.ray_d[p];
            float4 h = W.hit[p];
            VolumeHitRec vh;
            if (kStats ? closestVolumeHitCounted(V, xyz(o), xyz(d), h.x, vh, S.sdf_counters)
                       : closestVolumeHit(V, xyz(o), xyz(d), h.x, vh))
                W.hit[p] = make_float4(vh.t, __uint_as_float(kVolumeHit), __uint_as_float(vh.brick), 0.0f);
        }
        return;
    }
    DDAState st;
    float closestT = 0.0f;
    uint32_t p = kNoWork;
    bool exhausted = false;
    for (;;) {
        uint32_t idx = warpFetch(&W.counts[8], n, p == kNoWork && !exhausted, exhausted);
        if (idx != kNoWork) {
            p = q[idx];
            float4 o = W.ray_o[p], d = W.ray_d[p];
            closestT = W.hit[p].x;
            if (!ddaBegin(g, xyz(o), xyz(d), closestT, st)) p = kNoWork;  // misses the volume's bounds
        }
        if (__all_sync(0xffffffffu, p == kNoWork && exhausted)) break;
        if (p != kNoWork && ddaStepsCounted(V, g, st, kCountedCells, S.sdf_counters)) {
            if (st.found && st.out.t < closestT)
                W.hit[p] = make_float4(st.out.t, __uint_as_float(kVolumeHit), __uint_as_float(st.out.brick), 0.0f);
            p = kNoWork;
        }
    }
}

// The same for a scene with one sparse volume, as persistent threads with
// per-lane refill.  A ray's walk (ddaSteps and intersectBrickT, the same
// operations in the same order) is cut into steps of three kinds: a cell of
// the brick grid, a distance sample with the decision that follows from it
// (brick entry, backward search, march, bisection: all the same trilinear
// sample at another t), and a Newton step of the cubic polish.  A warp takes
// the kind that most of its lanes wait for, as in the triangle traversal; as
// nested loops the lanes of a warp waited for its longest march in every
// brick (16 of 32 busy on camera rays, 8 after the first bounce).  The sample
// divides by the brick's extents through their reciprocals (divBy).
// A camera ray visits 26 cells, 21 of them skipped macro cells, and takes a
// few samples: the walk's arithmetic bounds it (issue 0.66 of the slots), so
// it too divides through reciprocals, and the entry's constants are computed
// once per block.  Sparse-SDF configuration, 1024 x 1024 at 16 spp, whole
// frame: 23.3 ms as nested loops; 21.4 as steps, 19.6 with the divisions
// through reciprocals, 18.2 with the block's constants.  Blocks per SM 5 / 6 / 7 /
// 8: 19.2 / 18.2 / 17.7 / 17.3 ms.
// W.counts[8] is the work cursor (zeroed by k_extend).
constexpr int kVolumeMinBlocks = 8;
constexpr int kWalkCells = 2;  // cells a lane may walk per step (1 / 2 / 4 / 16: 20.2 / 19.6 / 19.7 / 21.7 ms)
enum MarchPhase : uint32_t { kMarchIdle, kMarchWalk, kMarchEntry, kMarchBack, kMarchStep, kMarchBisect, kMarchPolish };

// a / b rounded to nearest, from y = RN(1 / b): two residual corrections of a * y, the last of
// which rounds correctly (P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", 1990) where no residual underflows.  b is a length of at least 1e-6 and a
// a coordinate difference or a distance.
__device__ __forceinline__ float divBy(float a, float b, float y) {
    float q = ex::mul(a, y);
    q = __fmaf_rn(__fmaf_rn(-b, q, a), y, q);
    return __fmaf_rn(__fmaf_rn(-b, q, a), y, q);
}

// The same for a finite distance a >= 0, which may be as large as FP32 goes: where the quotient leaves its
// range the corrections give no number, and it is infinite.
__device__ __forceinline__ float divDistance(float a, float b, float y) { return fminf(divBy(a, b, y), INFINITY); }

// The volume's constants of a ray's entry (ddaBegin), computed once per block.
struct MarchVolume {
    float3 worldMin, worldMax, localMin, extent, rExtent, sampleDen, brick, rBrick;
    float cellSize;
};
__device__ __forceinline__ void marchVolume(const DDAGrid& g, MarchVolume& v) {
    const dk_volume_descriptor& vol = *g.vol;
    v.worldMin = ld3f(vol.world_bounds_min);
    v.worldMax = ld3f(vol.world_bounds_max);
    v.localMin = ld3f(vol.local_bounds_min);
    v.extent = mx(ex::sub(ld3f(vol.local_bounds_max), v.localMin), f3(1e-6f));
    v.rExtent = rcp3(v.extent);
    v.sampleDen = mx(ex::sub(f3((float)vol.dimensions.x, (float)vol.dimensions.y, (float)vol.dimensions.z), f3(1.0f)), f3(1.0f));
    v.brick = mx(f3((float)g.bsz[0], (float)g.bsz[1], (float)g.bsz[2]), f3(1.0f));
    v.rBrick = rcp3(v.brick);
    v.cellSize = cellSizeOf(vol);
}

// One ray's constants: 1 / va of the walk (with whether divBy may use them: no
// component so small or large that a residual could leave the normal range),
// 1 / units per world unit, and the shortest march step.
struct MarchRay {
    float rva[3], rUpw, minimumStep;
    bool byReciprocal;
};

// ddaBegin with the block's constants; a component of the local direction too
// small for divBy's residuals takes the divisions themselves.
__device__ __forceinline__ bool marchEnter(const DDAGrid& g, const MarchVolume& v, float3 o, float3 d, float closestT,
                                           DDAState& s, MarchRay& r) {
    if (!intersectAABB(o, d, v.worldMin, v.worldMax, closestT, s.tNear, s.tFar)) return false;
    s.vr.lo = mulColumns(g.vol->world_to_local, o, 1.0f);
    s.vr.ld = mulColumns(g.vol->world_to_local, d, 0.0f);
    s.vr.upw = fmaxf(exLength(s.vr.ld), 1e-6f);
    s.vr.cellSize = v.cellSize;
    s.t = s.tNear;
    const float3 lp = ex::sub(ex::add(s.vr.lo, ex::mul(s.vr.ld, s.t)), v.localMin);
    const float from[3] = {lp.x, lp.y, lp.z}, dir[3] = {s.vr.ld.x, s.vr.ld.y, s.vr.ld.z};
    const float ext[3] = {v.extent.x, v.extent.y, v.extent.z}, rExt[3] = {v.rExtent.x, v.rExtent.y, v.rExtent.z};
    const float den[3] = {v.sampleDen.x, v.sampleDen.y, v.sampleDen.z};
    const float bsf[3] = {v.brick.x, v.brick.y, v.brick.z}, rBsf[3] = {v.rBrick.x, v.rBrick.y, v.rBrick.z};
    r.byReciprocal = true;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float sp = ex::mul(divBy(from[a], ext[a], rExt[a]), den[a]);
        s.bpa[a] = divBy(ex::add(sp, 0.5f), bsf[a], rBsf[a]);
        const bool plain = !(dir[a] == 0.0f || fabsf(dir[a]) >= 1e-12f);
        const float vel = ex::mul(plain ? ex::div(dir[a], ext[a]) : divBy(dir[a], ext[a], rExt[a]), den[a]);
        s.va[a] = plain ? ex::div(vel, bsf[a]) : divBy(vel, bsf[a], rBsf[a]);
        const float va = fabsf(s.va[a]);
        r.rva[a] = ex::rcp(s.va[a]);
        if (!(va == 0.0f || (va >= 1e-12f && va <= 1e12f))) r.byReciprocal = false;  // (no division by a zero component)
        s.cell[a] = (int)clampf(floorf(s.bpa[a]), 0.0f, ex::sub((float)g.gd[a], 1.0f));
        s.stepDir[a] = s.va[a] > 0.0f ? 1 : (s.va[a] < 0.0f ? -1 : 0);
        const float nb = s.stepDir[a] > 0 ? ex::add((float)s.cell[a], 1.0f) : (float)s.cell[a];
        const float x = ex::sub(nb, s.bpa[a]);
        s.tMax[a] = s.stepDir[a] == 0
                        ? INFINITY
                        : ex::add(s.t, va >= 1e-12f && va <= 1e12f ? divBy(x, s.va[a], r.rva[a]) : ex::div(x, s.va[a]));
        s.tDelta[a] = s.stepDir[a] == 0 ? INFINITY : fabsf(r.rva[a]);  // RN(1 / va)
    }
    s.step = 0u;
    s.found = false;
    s.closest = closestT;
    r.rUpw = ex::rcp(s.vr.upw);
    r.minimumStep = fmaxf(divBy(ex::mul(s.vr.cellSize, 0.10f), s.vr.upw, r.rUpw), 0.0005f);
    return true;
}
// The distance to the plane `to` of axis `a` from `from`, in walk units.
__device__ __forceinline__ float marchPlane(const DDAState& s, const MarchRay& r, int a, float to, float from) {
    const float x = ex::sub(to, from);
    return r.byReciprocal ? divBy(x, s.va[a], r.rva[a]) : ex::div(x, s.va[a]);
}

struct MarchState {
    uint32_t phase, brick, count;
    uint32_t dims[3], offset;               // of the brick's samples
    float3 lo, ext, inv;                    // sample bounds: minimum, extent, 1 / extent
    float t, lowT, lowD, highT, tFar, entryT;
};

template <class D>
__device__ __forceinline__ float marchSample(const D& dist, const MarchState& m, float3 p) {
    const float u[3] = {divBy(ex::sub(p.x, m.lo.x), m.ext.x, m.inv.x), divBy(ex::sub(p.y, m.lo.y), m.ext.y, m.inv.y),
                        divBy(ex::sub(p.z, m.lo.z), m.ext.z, m.inv.z)};
    uint32_t b[3], n[3];
    float f[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float g = ex::mul(clampf(u[a], 0.0f, 1.0f), (float)(m.dims[a] - 1u));
        b[a] = (uint32_t)floorf(g);
        n[a] = min(b[a] + 1u, m.dims[a] - 1u);
        f[a] = ex::sub(g, (float)b[a]);
    }
    const uint32_t strideZ = m.dims[0] * m.dims[1];
    const uint32_t y0 = b[1] * m.dims[0], y1 = n[1] * m.dims[0];
    const uint32_t z0 = m.offset + b[2] * strideZ, z1 = m.offset + n[2] * strideZ;
    const float c00 = exMix(dist.at(z0 + y0 + b[0]), dist.at(z0 + y0 + n[0]), f[0]);
    const float c10 = exMix(dist.at(z0 + y1 + b[0]), dist.at(z0 + y1 + n[0]), f[0]);
    const float c01 = exMix(dist.at(z1 + y0 + b[0]), dist.at(z1 + y0 + n[0]), f[0]);
    const float c11 = exMix(dist.at(z1 + y1 + b[0]), dist.at(z1 + y1 + n[0]), f[0]);
    return exMix(exMix(c00, c10, f[1]), exMix(c01, c11, f[1]), f[2]);
}

// The walk leaves its cell: false when the ray is finished.
__device__ __forceinline__ bool marchNextCell(DDAState& s) {
    const float nextT = fminf(s.tMax[0], fminf(s.tMax[1], s.tMax[2]));
    if (s.found && s.closest <= ex::add(nextT, 0.0005f)) return false;
    if (nextT > s.tFar || nextT >= s.closest) return false;
    if (s.tMax[0] <= s.tMax[1] && s.tMax[0] <= s.tMax[2]) {
        s.cell[0] += s.stepDir[0];
        s.t = s.tMax[0];
        s.tMax[0] = ex::add(s.tMax[0], s.tDelta[0]);
    } else if (s.tMax[1] <= s.tMax[2]) {
        s.cell[1] += s.stepDir[1];
        s.t = s.tMax[1];
        s.tMax[1] = ex::add(s.tMax[1], s.tDelta[1]);
    } else {
        s.cell[2] += s.stepDir[2];
        s.t = s.tMax[2];
        s.tMax[2] = ex::add(s.tMax[2], s.tDelta[2]);
    }
    ++s.step;
    return true;
}

// One cell of the walk: the lane stays in kMarchWalk, enters a brick
// (kMarchEntry) or is finished (kMarchIdle).
__device__ __forceinline__ void marchWalk(const VolumeScene& V, const DDAGrid& g, const uint32_t* macroShift,
                                          DDAState& s, const MarchRay& ray, MarchState& m) {
    m.phase = kMarchIdle;
    if (!(s.step < g.maxSteps && s.t <= s.tFar && s.t < s.closest)) return;
    if (s.cell[0] < 0 || s.cell[1] < 0 || s.cell[2] < 0 || s.cell[0] >= (int)g.gd[0] || s.cell[1] >= (int)g.gd[1] ||
        s.cell[2] >= (int)g.gd[2])
        return;
    if (g.hasMacro) {
        uint32_t mc[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const uint32_t c = (uint32_t)s.cell[a];
            mc[a] = min(macroShift[a] < 32u ? c >> macroShift[a] : c / g.msz[a], g.md[a] - 1u);
        }
        const uint64_t macroSlot = (uint64_t)g.macroOffset + mc[0] + mc[1] * g.md[0] + mc[2] * g.md[0] * g.md[1];
        if (macroSlot < V.gridIndexCount && __ldg(V.gridIndices + macroSlot) == 0u) {
            const float dt = ex::sub(s.t, s.tNear);
            float mt[3];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const float cb = ex::add(s.bpa[a], ex::mul(s.va[a], dt));
                const float mb = s.stepDir[a] > 0 ? (float)min((mc[a] + 1u) * g.msz[a], g.gd[a]) : (float)(mc[a] * g.msz[a]);
                mt[a] = s.stepDir[a] == 0 ? INFINITY : ex::add(s.t, marchPlane(s, ray, a, mb, cb));
            }
            const float macroNextT = fminf(mt[0], fminf(mt[1], mt[2]));
            if (macroNextT > ex::add(s.t, 1e-6f)) {
                if (macroNextT > s.tFar || macroNextT >= s.closest) return;
                s.t = ex::add(macroNextT, 1e-5f);
                const float dt2 = ex::sub(s.t, s.tNear);
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    const float c2 = ex::add(s.bpa[a], ex::mul(s.va[a], dt2));
                    s.cell[a] = (int)clampf(floorf(c2), 0.0f, ex::sub((float)g.gd[a], 1.0f));
                    const float nb = s.stepDir[a] > 0 ? ex::add((float)s.cell[a], 1.0f) : (float)s.cell[a];
                    s.tMax[a] = s.stepDir[a] == 0 ? INFINITY : ex::add(s.t, marchPlane(s, ray, a, nb, c2));
                }
                ++s.step;
                m.phase = kMarchWalk;
                return;
            }
        }
    }
    const uint64_t slot = (uint64_t)g.gridOffset + (uint32_t)s.cell[0] + (uint32_t)s.cell[1] * g.gd[0] +
                          (uint32_t)s.cell[2] * g.gd[0] * g.gd[1];
    if (slot < V.gridIndexCount) {
        const uint32_t bi = __ldg(V.gridIndices + slot);
        if (bi != 0xffffffffu && bi < V.brickCount) {
            const dk_volume_brick_descriptor& brick = V.bricks[bi];
            float tNear, tFar;
            if (intersectAABB(s.vr.lo, s.vr.ld, ld3f(brick.local_bounds_min), ld3f(brick.local_bounds_max), s.closest,
                              tNear, tFar)) {
                const BrickCtx c = makeBrickCtx(brick, V.sampleCount);
                if (c.valid && !(__ldg(&brick.sample_bounds_min.w) > 0.0f || __ldg(&brick.sample_bounds_max.w) < 0.0f)) {
                    m.brick = bi;
#pragma unroll
                    for (int a = 0; a < 3; ++a) m.dims[a] = c.dims[a];
                    m.offset = c.sampleOffset;
                    m.lo = c.sampleMin;
                    m.ext = c.sampleExtent;
                    m.inv = rcp3(c.sampleExtent);
                    m.tFar = tFar;
                    m.t = m.entryT = tNear;
                    m.phase = kMarchEntry;
                    return;
                }
            }
        }
    }
    if (marchNextCell(s)) m.phase = kMarchWalk;
}

// The march from the brick's entry (or the point the backward search found):
// kMarchStep at its first t, or the brick is left without a hit.
__device__ __forceinline__ bool marchBegin(MarchState& m, float closest, float upw, float rUpw, float minimumStep) {
    m.t = fmaxf(m.entryT, ex::add(m.lowT, fmaxf(ex::mul(divDistance(fabsf(m.lowD), upw, rUpw), 0.9f), minimumStep)));
    m.count = 0u;
    m.phase = kMarchStep;
    return m.t <= m.tFar && m.t < closest;
}

template <class D>
__global__ void __launch_bounds__(128, kVolumeMinBlocks) k_volume_march(DevScene S, Wave W, uint32_t sel, D dist) {
    const uint32_t* q = W.q[sel];
    const uint32_t n = W.counts[sel];
    const VolumeScene V = volumeScene(S);
    DDAGrid g;
    if (V.gridCount == 0u || V.gridIndexCount == 0u || V.volumes[0].metadata.w != 1u || !ddaGrid(V, 0u, g)) return;
    __shared__ MarchVolume vol;
    if (threadIdx.x == 0) marchVolume(g, vol);
    __syncthreads();
    uint32_t macroShift[3];  // of the macro size where it is a power of two, else 32
#pragma unroll
    for (int a = 0; a < 3; ++a) macroShift[a] = (g.msz[a] & (g.msz[a] - 1u)) ? 32u : 31u - __clz(g.msz[a]);
    DDAState s;
    MarchState m;
    MarchRay ray = {};
    m.phase = kMarchIdle;
    uint32_t p = kNoWork;
    bool exhausted = false;
    for (;;) {
        uint32_t idx = warpFetch(&W.counts[8], n, p == kNoWork && !exhausted, exhausted);
        if (idx != kNoWork) {
            p = q[idx];
            float4 o = W.ray_o[p], d = W.ray_d[p];
            if (marchEnter(g, vol, xyz(o), xyz(d), W.hit[p].x, s, ray))
                m.phase = kMarchWalk;
            else
                p = kNoWork;  // misses the volume's bounds
        }
        if (__all_sync(0xffffffffu, p == kNoWork && exhausted)) break;
        const int least = __any_sync(0xffffffffu, exhausted) ? 1 : kRefillBelow;
        for (;;) {
            const unsigned walkers = __ballot_sync(0xffffffffu, m.phase == kMarchWalk);
            const unsigned samplers = __ballot_sync(0xffffffffu, m.phase >= kMarchEntry && m.phase <= kMarchBisect);
            const unsigned polishers = __ballot_sync(0xffffffffu, m.phase == kMarchPolish);
            const int nw = __popc(walkers), ns = __popc(samplers), np = __popc(polishers);
            if (nw + ns + np < least) break;
            if (np > max(nw, ns)) {
                if (m.phase != kMarchPolish) continue;
                // Two Newton steps on the cubic interpolant: lowT, highT the bracket, t the refined distance.
                BrickCtx c;
#pragma unroll
                for (int a = 0; a < 3; ++a) c.dims[a] = m.dims[a];
                c.sampleOffset = m.offset;
                c.strideY = m.dims[0];
                c.strideZ = m.dims[0] * m.dims[1];
                c.sampleMin = m.lo;
                c.sampleExtent = m.ext;
                c.valid = true;
                const DistGrad pg = brickDistGradCubic(dist, c, ex::add(s.vr.lo, ex::mul(s.vr.ld, m.t)));
                const float slope = ex::dot(pg.gradient, s.vr.ld);
                bool more = isfinite(pg.distance) && !(fabsf(slope) <= 1e-6f);
                if (more) {
                    const float projected = ex::sub(m.t, ex::div(pg.distance, slope));
                    more = !(projected <= m.lowT || projected >= m.highT);
                    if (more) m.t = projected;
                }
                if (more && ++m.count < 2u) continue;
            } else if (ns >= nw) {
                if (m.phase < kMarchEntry || m.phase > kMarchBisect) continue;
                const float dd = marchSample(dist, m, ex::add(s.vr.lo, ex::mul(s.vr.ld, m.t)));
                const bool finite = isfinite(dd);
                bool miss = false;
                if (m.phase == kMarchBisect) {
                    if ((m.lowD > 0.0f && dd > 0.0f) || (m.lowD < 0.0f && dd < 0.0f)) {
                        m.lowT = m.t;
                        m.lowD = dd;
                    } else {
                        m.highT = m.t;
                    }
                    m.t = ex::mul(0.5f, ex::add(m.lowT, m.highT));
                    if (++m.count < 8u) continue;
                    if (s.vr.cellSize <= 0.03f) {
                        m.phase = kMarchPolish;
                        m.count = 0u;
                        continue;
                    }
                } else {
                    if (m.phase == kMarchStep) {
                        if (!finite) {
                            miss = true;
                        } else if ((m.lowD > 0.0f && dd <= 0.0f) || (m.lowD < 0.0f && dd >= 0.0f)) {
                            m.highT = m.t;
                            m.t = ex::mul(0.5f, ex::add(m.lowT, m.highT));
                            m.count = 0u;
                            m.phase = kMarchBisect;
                            continue;
                        } else {
                            m.lowT = m.t;
                            m.lowD = dd;
                            m.t = ex::add(m.t,
                                          fmaxf(ex::mul(divDistance(fabsf(dd), s.vr.upw, ray.rUpw), 0.8f), ray.minimumStep));
                            miss = !(++m.count < 192u && m.t <= m.tFar && m.t < s.closest);
                        }
                    } else if (m.phase == kMarchEntry) {
                        m.lowT = m.t;
                        m.lowD = dd;
                        if (!finite) {
                            miss = true;
                        } else if (dd <= 0.0f) {
                            m.phase = kMarchBack;
                            m.count = 0u;
                        } else {
                            miss = !marchBegin(m, s.closest, s.vr.upw, ray.rUpw, ray.minimumStep);
                        }
                    } else {  // kMarchBack
                        if (finite && dd > 0.0f) {
                            m.lowT = m.t;
                            m.lowD = dd;
                        }
                        if (!finite || dd > 0.0f || m.t <= 0.0005f || ++m.count == 12u)
                            miss = !marchBegin(m, s.closest, s.vr.upw, ray.rUpw, ray.minimumStep);
                    }
                    if (!miss) {
                        if (m.phase == kMarchBack)
                            m.t = fmaxf(ex::sub(m.t, fmaxf(ex::mul(ex::div(s.vr.cellSize, s.vr.upw), 0.5f), ray.minimumStep)),
                                        0.0005f);
                        continue;
                    }
                }
                if (miss) {  // the brick is left without a hit
                    m.phase = marchNextCell(s) ? kMarchWalk : kMarchIdle;
                    if (m.phase == kMarchWalk) continue;
                }
            } else {
                if (m.phase != kMarchWalk) continue;
#pragma unroll 1
                for (int k = 0; k < kWalkCells && m.phase == kMarchWalk; ++k) marchWalk(V, g, macroShift, s, ray, m);
                if (m.phase != kMarchIdle) continue;
            }
            // Here: a hit at m.t (phase bisect or polish), or the ray is finished (idle).
            if (m.phase != kMarchIdle) {
                if (m.t < s.closest) {
                    s.closest = m.t;
                    s.out.t = m.t;
                    s.out.brick = m.brick;
                    s.found = true;
                }
                m.phase = marchNextCell(s) ? kMarchWalk : kMarchIdle;
                if (m.phase == kMarchWalk) continue;
            }
            if (s.found) W.hit[p] = make_float4(s.out.t, __uint_as_float(kVolumeHit), __uint_as_float(s.out.brick), 0.0f);
            p = kNoWork;
        }
    }
}

// Shadow rays, persistent threads with per-lane refill: an any-hit query for
// an opaque blocker replaces the slot's unshadowed contribution by its
// shadowed value (contribution / pdf divisor, or 0).  Rays that crossed a
// cut-out or transmissive triangle without meeting an opaque one go to a
// second queue for the layer walk (W.counts[6]).  W.counts[5] is the cursor.
template <bool kWide8>
__global__ void __launch_bounds__(128) k_shadow_rays(DevScene S, Wave W) {
    const uint32_t n = W.counts[3];
    const size_t cap = W.cap;
    // Triangle-only scenes: one scene query per shadow ray (the reference steps through
    // transmissive layers one closest hit at a time; scenes with volumes count the walk's steps).
    if (S.sdf_counters && S.volume_count == 0u && globalId() == 0 && n)
        atomicAdd(S.sdf_counters + kSdfShadowSceneQueries, (unsigned long long)n);
    int stackNode[kWide8 ? 1 : kStackSize];
    uint2 stack8[kWide8 ? kTraversalStack : 1];
    std::conditional_t<kWide8, Any8, AnyState> st;
    uint32_t e = kNoWork;
    bool exhausted = false;
    for (;;) {
        uint32_t idx = warpFetch(&W.counts[5], n, e == kNoWork && !exhausted, exhausted);
        if (idx != kNoWork) {
            e = W.qr[idx];
            size_t slot = (size_t)(e & 3u) * cap + (e >> 2);
            float4 o = W.nee_o[slot], d = W.nee_d[slot];
            anyInit(st, xyz(o), xyz(d), o.w, __ldg(&W.jobs[__float_as_uint(d.w)].opaque_mask),
                    S.volume_count ? nullptr : W.layer_hits + slot * kRecLayers);
        }
        if (__all_sync(0xffffffffu, e == kNoWork && exhausted)) break;
        auto settle = [&](int r) {  // 1: no opaque blocker, 2: occluded
            size_t slot = (size_t)(e & 3u) * cap + (e >> 2);
            if (r == 1 && S.volume_count) st.sawNonOpaque = true;  // distance volumes: the walk decides
            if (r == 2) {
                W.nee_c[slot] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            } else if (st.sawNonOpaque) {
                W.layer_count[slot] = st.recCount | (st.recOverflow ? 0x80000000u : 0u);
                W.qr2[atomicAdd(&W.counts[6], 1u)] = e;
            } else {
                float4 c = W.nee_c[slot];
                W.nee_c[slot] = make_float4(c.x / c.w, c.y / c.w, c.z / c.w, 0.0f);
            }
            e = kNoWork;
        };
        if (S.node_count == 0) {
            if (e != kNoWork) settle(1);
        } else if constexpr (kWide8) {
            if (e != kNoWork)
                if (int r = anySteps(S, st, stack8, kStepBudget)) settle(r);
        } else {
            const int least = __any_sync(0xffffffffu, exhausted) ? 1 : kRefillBelow;
            for (;;) {
                int running;
                const bool nodes = majorityStep(e != kNoWork, st.node, running);
                if (running < least) break;
                const bool leaf = (st.node & kLeafBit) != 0u;
                if (e == kNoWork || nodes == leaf) continue;
                if (int r = leaf ? anyTriStep(S, st, stackNode) : anyNodeStep(S, st, stackNode)) settle(r);
            }
        }
    }
}

// The layer walk for the rays the any-hit pass could not settle: from the
// layers it recorded, or by a collecting traversal when it crossed more.
#ifndef DK_LAYERS_MIN_BLOCKS
#define DK_LAYERS_MIN_BLOCKS 4
#endif
// kVolumes: scenes with sparse volumes walk every shadow ray the reference's
// way (shadowWalk); the others take the recorded layers, or the collecting
// traversal when more were crossed -- two kernels, so that neither carries the
// other's code.
template <bool kVolumes>
__global__ void __launch_bounds__(128, DK_LAYERS_MIN_BLOCKS) k_shadow_layers(DevScene S, Wave W) {
    const uint32_t n = W.counts[6];
    const size_t cap = W.cap;
    for (uint32_t i = globalId(); i < n; i += gridStride()) {
        uint32_t e = W.qr2[i];
        size_t slot = (size_t)(e & 3u) * cap + (e >> 2);
        float4 o = W.nee_o[slot], d = W.nee_d[slot], c = W.nee_c[slot];
        float3 T = f3(1.0f);
        const DevJob& J = W.jobs[__float_as_uint(d.w)];
        const MatTable mt = matTable(J);
        bool occluded;
        if (kVolumes) {
            occluded = shadowWalk(S, mt, xyz(o), xyz(d), o.w, T);
        } else {
            uint32_t lc = W.layer_count[slot];
            occluded = (lc & 0x80000000u)
                           ? shadowLayers(S, mt, __ldg(&J.opaque_mask), xyz(o), xyz(d), o.w, T)
                           : recordedLayers(S, mt, xyz(o), xyz(d), W.layer_hits + slot * kRecLayers, lc, T);
        }
        float3 v = occluded ? f3(0.0f) : xyz(c) * T / c.w;
        W.nee_c[slot] = make_float4(v.x, v.y, v.z, 0.0f);
    }
}

// `radiance += clampSampleContribution(throughput * direct)` with direct the
// sum of the path's shadowed NEE terms in the reference's order (light, env 0,
// env 1; PathTrace.metal:4437-4584, 5396-5421).
__global__ void __launch_bounds__(256) k_resolve(Wave W) {
    const uint32_t n = W.counts[2];
    const size_t cap = W.cap;
    for (uint32_t i = globalId(); i < n; i += gridStride()) {
        uint32_t si = W.qs[i];
        float4 tpw = W.nee_tp[si];
        uint32_t bits = __float_as_uint(tpw.w);
        uint32_t mask = bits & 7u, p = bits >> 3;
        float3 direct = f3(0.0f);
        for (uint32_t k = 0; k < 3u; ++k)
            if (mask & (1u << k)) direct += xyz(W.nee_c[k * cap + si]);
        float4 r = W.rad[p];
        float3 add = clampSampleContribution(xyz(tpw) * direct, __ldg(&W.jobs[jobOf(W, p)].P.clamp));
        W.rad[p] = make_float4(r.x + add.x, r.y + add.y, r.z + add.z, r.w);
    }
}

// tracePrimaryAOV (PathTrace.metal:4093-4159) for the denoiser's unjittered AOV ray.
__global__ void __launch_bounds__(128) k_aov_primary(DevScene S, Wave W) {
    for (uint32_t i = globalId(); i < W.pixel_count; i += gridStride()) {
        const DevJob& J = W.jobs[jobOfPixel(W, i)];
        const DevParams& P = J.P;
        if (P.denoiser == 0u) continue;
        const MatTable mt = matTable(J);
        uint32_t local = i - J.pixel_begin;
        uint32_t px = P.tile_x + local % P.tile_w, py = P.tile_y + local / P.tile_w;
        Ray ray = makeCameraRay(P.cam, P.width, P.height, px, py, 0.5f, 0.5f, 0.0f, 0.0f);
        writeAovMiss(W.aov, i, W.aov_stride);
        for (uint32_t pass = 0; pass < 32u; ++pass) {
            sdfCount(S.sdf_counters, kSdfPrimarySceneQueries);
            HitRec r = traceSceneCounting(S, ray.origin, ray.direction);
            if (r.tri == kNoHit) break;
            Hit h = makeHitAny(S, ray, r);
            Material m = materialForHit(S, mt, h);
            uint32_t nIdx = (uint32_t)m.parameters.w;
            if (nIdx != 0u) h = applyNormalMap(S, h, nIdx, ray.direction);
            uint32_t bIdx = (uint32_t)m.parameters.z;
            if (bIdx != 0u) {
                float4 t = sampleTexture(S, bIdx, h.uv, make_float4(1.0f, 1.0f, 1.0f, 1.0f));
                m.baseColor = make_float4(ex::mul(m.baseColor.x, t.x), ex::mul(m.baseColor.y, t.y),
                                          ex::mul(m.baseColor.z, t.z), ex::mul(m.baseColor.w, t.w));
            }
            if (m.baseColor.w <= 0.001f) {
                ray.origin = ex::add(h.position, ex::mul(ray.direction, 0.001f));
                continue;
            }
            writeAovHit(W.aov, i, W.aov_stride, h, m.baseColor);
            break;
        }
    }
}

// projectToScreen (PathTrace.metal:1662-1697), exact ops.
__device__ bool projectToScreen(const dk_camera& cam, float3 w, uint32_t width, uint32_t height, float2& s) {
    float3 hz = f3(cam.horizontal.x, cam.horizontal.y, cam.horizontal.z);
    float3 vt = f3(cam.vertical.x, cam.vertical.y, cam.vertical.z);
    float3 ll = f3(cam.lower_left.x, cam.lower_left.y, cam.lower_left.z);
    float3 org = f3(cam.origin.x, cam.origin.y, cam.origin.z);
    float3 forward = ex::normalize(ex::cross(vt, hz));
    float3 center = ex::add(ex::add(ll, ex::mul(hz, 0.5f)), ex::mul(vt, 0.5f));
    float3 planePoint;
    if (cam.origin.w > 0.5f) {
        planePoint = ex::sub(w, ex::mul(forward, ex::dot(ex::sub(w, center), forward)));
    } else {
        float3 toPoint = ex::sub(w, org);
        float den = ex::dot(toPoint, forward);
        if (fabsf(den) <= 1e-5f) return false;
        float planeT = ex::div(ex::dot(ex::sub(center, org), forward), den);
        if (planeT <= 0.0f) return false;
        planePoint = ex::add(org, ex::mul(toPoint, planeT));
    }
    float3 rel = ex::sub(planePoint, ll);
    float u = ex::div(ex::dot(rel, hz), fmaxf(ex::dot(hz, hz), 1e-5f));
    float v = ex::div(ex::dot(rel, vt), fmaxf(ex::dot(vt, vt), 1e-5f));
    s = make_float2(ex::mul(u, (float)width), ex::mul(ex::sub(1.0f, v), (float)height));
    return true;
}

// ------------------------------------------- preview and interactive ----
// flatPreviewKernel (PathTrace.metal:4728-4868) and interactiveMaterialKernel
// (:4870-5165), the kernels of RenderQuality.preview and .interactive
// (DenrimRenderer.primaryPipeline, DenrimRenderer.swift:197-214): one camera
// ray through each pixel centre, shaded without path tracing.  Like the
// reference they overwrite the beauty and the AOV planes on every sample
// (the result does not depend on the sample index); the beauty goes into the
// accumulation as one sample.
__device__ __forceinline__ float smoothstepf(float e0, float e1, float x) {  // Metal smoothstep
    float t = clampf((x - e0) / (e1 - e0), 0.0f, 1.0f);
    return t * t * (3.0f - 2.0f * t);
}

// The preview kernels call one copy of the environment lookup: inlined at each
// of its dozen uses it made them stall on instruction fetch (see k_preview).
__device__ __noinline__ float3 sampleEnvironmentCall(const DevScene& S, float3 d) { return sampleEnvironment(S, d); }

// The environment along the six axis directions sampleInteractiveDiffuse-
// Environment blends: the same for every pixel, so a block samples them once.
__device__ __forceinline__ void loadAxisEnvironment(const DevScene& S, float3* axis) {
    if (threadIdx.x < 6u) {
        const float s = (threadIdx.x & 1u) ? -1.0f : 1.0f;
        const uint32_t a = threadIdx.x >> 1;
        axis[threadIdx.x] = sampleEnvironmentCall(S, f3(a == 1u ? s : 0.0f, a == 0u ? s : 0.0f, a == 2u ? s : 0.0f));
    }
    __syncthreads();
}

// sampleInteractiveDiffuseEnvironment (:3805-3823)
__device__ float3 interactiveDiffuseEnv(const float3* axis, float3 n) {
    float3 up = axis[0];
    float3 down = axis[1];
    float3 side = (axis[2] + axis[3] + axis[4] + axis[5]) * 0.25f;
    float upW = smoothstepf(-0.15f, 0.85f, n.y);
    float downW = smoothstepf(0.15f, -0.85f, n.y);
    float sideW = fmaxf(0.0f, 1.0f - upW - downW);
    return up * upW + down * downW + side * sideW;
}

// interactiveHemisphereDirection (:3825-3831)
__device__ __forceinline__ float3 interactiveHemisphere(float3 d, float3 n) {
    float nd = dot(n, d);
    if (nd < 0.0f) d = d - n * (2.0f * nd);
    return normalize(d);
}

// sampleInteractiveSpecularEnvironment (:3833-3880); `diffuse` is
// interactiveDiffuseEnv at the same normal.
__device__ __noinline__ float3 interactiveSpecularEnv(const DevScene& S, float3 r, float3 n, float roughness, float3 diffuse) {
    r = interactiveHemisphere(normalize(r), n);
    roughness = clampf(roughness, 0.0f, 1.0f);
    float spread = roughness * roughness;
    float3 helper = fabsf(r.y) < 0.999f ? f3(0.0f, 1.0f, 0.0f) : f3(1.0f, 0.0f, 0.0f);
    float3 t = normalize(cross(helper, r));
    float3 b = cross(r, t);
    float3 cone = sampleEnvironmentCall(S, r) * 0.42f;
    cone += sampleEnvironmentCall(S, interactiveHemisphere(r + t * spread * 0.95f + n * spread * 0.18f, n)) * 0.145f;
    cone += sampleEnvironmentCall(S, interactiveHemisphere(r - t * spread * 0.95f + n * spread * 0.18f, n)) * 0.145f;
    cone += sampleEnvironmentCall(S, interactiveHemisphere(r + b * spread * 0.95f + n * spread * 0.18f, n)) * 0.145f;
    cone += sampleEnvironmentCall(S, interactiveHemisphere(r - b * spread * 0.95f + n * spread * 0.18f, n)) * 0.145f;
    return mix3(cone, diffuse, smoothstepf(0.62f, 0.95f, roughness));
}

// interactiveContactAmbientOcclusion (:4276-4360): four short probes around
// the normal, each nearby occluder weighted by its opacity and proximity.
// Called by every thread of the block (`hit`: this thread has a surface).
__device__ __forceinline__ float interactiveContactAO(const DevScene& S, MatTable mt, bool hit, const Hit& h,
                                                      const Material& m, float3 n) {
    constexpr float kRadius = 0.34f;
    TangentFrame frame = makeTangentFrame(n, h.tangent, h.bitangent);
    const float3 local[4] = {f3(0.000f, 0.000f, 1.000f), f3(0.780f, 0.180f, 0.600f), f3(-0.420f, 0.720f, 0.552f),
                             f3(-0.620f, -0.520f, 0.587f)};
    float occlusion = 0.0f;
#pragma unroll 1
    for (int k = 0; k < 4; ++k) {
        __syncthreads();
        if (!hit) continue;
        float3 l = normalize(local[k]);
        float3 dir = normalize(l.x * frame.tangent + l.y * frame.bitangent + l.z * n);
        Ray ray{h.position + n * 0.003f, dir};
        sdfCount(S.sdf_counters, kSdfShadowSceneQueries);
        HitRec r = traceSceneWithin(S, ray.origin, ray.direction, kRadius);
        if (r.tri == kNoHit || !(r.t < kRadius)) continue;
        Hit oh = makeHitAny(S, ray, r);
        Material om = materialForHit(S, mt, oh);
        float blocker = clampf(om.baseColor.w, 0.0f, 1.0f) * (1.0f - materialTransmission(om) * 0.72f);
        occlusion += blocker * (1.0f - smoothstepf(0.0f, kRadius, r.t));
    }
    float strength = 0.72f + (0.36f - 0.72f) * materialTransmission(m);  // mix(0.72, 0.36, transmission)
    return 1.0f - clampf((occlusion / 4.0f) * strength, 0.0f, 0.72f);
}

__device__ __forceinline__ void storePreview(const Accum& A, size_t pix, float4 beauty) {
    A.sum[pix] = beauty;
    A.comp[pix] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    A.resolved[pix] = D4{0.0, 0.0, 0.0, 0.0};
    A.count[pix] = 1u;
}

// One thread per pixel.  The kernel is bound by
// instruction fetch: some 400 KB of code, of which every warp runs a large
// part once, so warps at different places evict each other's instructions (a
// version without barriers spent 31 of 36 cycles between a warp's issues
// waiting for an instruction, whatever its occupancy).  Hence large blocks
// whose warps go through the phases -- primary ray, each light, environment,
// each occlusion probe -- together, with a barrier between phases, so that one
// fetch serves 16 warps; threads without a hit go along with a neighbour's.
// Interactive 1280 x 720 of the material scene, whole frame with its display
// encoding: 7.56 ms as a grid-stride loop with everything inlined; 4.0 with the
// axis directions of the environment sampled once per block and the occlusion
// probes bounded by their radius; 2.7 with the environment lookup called;
// 0.78 with the phases.  Blocks x minimum residency 128 x 4 / 256 x 2 / 512 x 1 /
// 512 x 2 / 1024 x 1: 1.22 / 0.99 / 1.03 / 0.78 / 0.82 ms.
// Frames that do not fill the SMs with such blocks, and volume walks, whose
// lanes differ too much to wait for each other, lose by it: they run in blocks
// of 128 threads, or of one warp (launchPreview), with 128 registers or more.
// A warp has 8 x 4 pixels, in blocks of one warp 32 in a row, which spread a
// surface's expensive pixels over more warps.
// The interactive kernels stay within 128 registers: with more, a product is
// fused differently and the last bits of a frame change.
constexpr uint32_t kPreviewLarge = 512u, kPreviewMid = 128u, kPreviewSmall = 32u;
template <bool kInteractive, uint32_t kBlock>
constexpr uint32_t previewResidency() {
    return kBlock == kPreviewLarge ? 2u : kInteractive || kBlock == kPreviewMid ? 512u / kBlock : 1u;
}
template <bool kInteractive, uint32_t kBlock>
__global__ void __launch_bounds__(kBlock, previewResidency<kInteractive, kBlock>())
    k_preview(const __grid_constant__ DevScene S, const __grid_constant__ DevParams P, Accum A, MatTable mt,
              uint32_t opaqueMask) {
    const size_t plane = (size_t)P.width * P.height;
    uint32_t lx, ly;
    if constexpr (kBlock == kPreviewSmall) {
        const uint32_t i = blockIdx.x * kBlock + threadIdx.x;
        lx = i % P.tile_w;
        ly = i / P.tile_w;
    } else {
        const uint32_t lane = laneId(), warp = (blockIdx.x * kBlock + threadIdx.x) >> 5;
        const uint32_t tilesX = (P.tile_w + 7u) / 8u;
        lx = (warp % tilesX) * 8u + (lane & 7u);
        ly = (warp / tilesX) * 4u + (lane >> 3);
    }
    const bool valid = lx < P.tile_w && ly < P.tile_h;
    // Threads outside the tile, and later those whose ray missed, run the block's
    // phases on a neighbour's pixel or hit and store nothing of them.
    const uint32_t px = P.tile_x + min(lx, P.tile_w - 1u), py = P.tile_y + min(ly, P.tile_h - 1u);
    const size_t pix = (size_t)py * P.width + px;
    Ray ray = makeCameraRay(P.cam, P.width, P.height, px, py, 0.5f, 0.5f, 0.0f, 0.0f);
    HitRec rec;
    rec.tri = kNoHit;
    if (valid) {
        sdfCount(S.sdf_counters, kSdfPrimarySceneQueries);
        rec = traceSceneCounting(S, ray.origin, ray.direction);
    }
    const bool hit = rec.tri != kNoHit;
    __shared__ uint32_t firstHit;
    __shared__ HitRec sharedHit;
    if (threadIdx.x == 0) firstHit = 0xffffffffu;
    __syncthreads();
    if (hit) atomicMin(&firstHit, threadIdx.x);
    __syncthreads();
    if (threadIdx.x == firstHit) sharedHit = rec;
    __syncthreads();
    if (valid && !hit) {
        float alpha = P.transparent_background ? 0.0f : 1.0f;
        float3 color = mx(f3(P.bg[0], P.bg[1], P.bg[2]), f3(0.0f));
        if (!P.transparent_background && P.shows_env_bg) color = sampleEnvironmentCall(S, ray.direction);
        A.aov[0 * plane + pix] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        A.aov[1 * plane + pix] = make_float4(0.5f, 0.5f, 0.5f, 0.0f);
        for (int k = 2; k < 6; ++k) A.aov[k * plane + pix] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        storePreview(A, pix, make_float4(color.x, color.y, color.z, alpha));
    }
    if (firstHit == 0xffffffffu) return;
    if (!hit) rec = sharedHit;
    __shared__ float3 axisEnv[6];
    if (kInteractive) loadAxisEnvironment(S, axisEnv);

    Hit h = makeHitAny(S, ray, rec);
    Material m = materialForHit(S, mt, h);
    float4 beauty, albedo;
    float3 color;
    uint32_t nIdx = (uint32_t)m.parameters.w;
    if (nIdx != 0u) h = applyNormalMap(S, h, nIdx, ray.direction);
    uint32_t bIdx = (uint32_t)m.parameters.z;
    if (bIdx != 0u) {  // applyBaseColorTexture
        float4 t = sampleTexture(S, bIdx, h.uv, make_float4(1.0f, 1.0f, 1.0f, 1.0f));
        m.baseColor = make_float4(ex::mul(m.baseColor.x, t.x), ex::mul(m.baseColor.y, t.y),
                                  ex::mul(m.baseColor.z, t.z), ex::mul(m.baseColor.w, t.w));
    }
    const float3 n = ex::normalize(h.normal);
    const float3 view = ex::normalize(-ray.direction);
    if constexpr (!kInteractive) {  // :4824-4834
        const float3 key = ex::normalize(f3(0.35f, 0.72f, 0.58f));
        float lambert = fmaxf(ex::dot(n, key), 0.0f);
        float facing = fmaxf(ex::dot(n, view), 0.0f);
        float rim = ex::mul(powf(ex::sub(1.0f, facing), 2.0f), 0.08f);
        float shade = ex::add(ex::add(0.32f, ex::mul(0.68f, lambert)), rim);
        color = ex::add(ex::mul(mx(xyz(m.baseColor), f3(0.0f)), shade), mx(xyz(m.emission), f3(0.0f)));
        beauty = make_float4(color.x, color.y, color.z,
                             P.transparent_background ? clampf(m.baseColor.w, 0.0f, 1.0f) : 1.0f);
        albedo = m.baseColor;
    } else {  // :4961-5133
        const float roughness = clampf(m.parameters.x, 0.02f, 1.0f);
        const float metallic = clampf(m.parameters.y, 0.0f, 1.0f);
        const float opacity = clampf(m.baseColor.w, 0.0f, 1.0f);
        const float3 base = mx(xyz(m.baseColor), f3(0.0f));
        color = mx(xyz(m.emission), f3(0.0f));
        ShadePoint sp;
        makeShadePoint(sp, m, n, h.tangent, h.bitangent, view);
        const uint32_t nl = min(S.light_count, 12u);
#pragma unroll 1
        for (uint32_t l = 0; l < nl; ++l) {
            __syncthreads();
            const dk_light_record& L = S.lights[l];
            if (L.triangle_index >= S.tri_count || L.material_index >= S.mat_count) continue;
            const dk_triangle& lt = S.tris[L.triangle_index];
            float3 emission = mx(xyz(__ldg(reinterpret_cast<const float4*>(S.mats + L.material_index) + 1)), f3(0.0f));
            if (!hit || maxComponent(emission) <= 0.0f || L.area <= 0.0f) continue;
            float3 lp = (f3(lt.v0.x, lt.v0.y, lt.v0.z) + f3(lt.v1.x, lt.v1.y, lt.v1.z) +
                         f3(lt.v2.x, lt.v2.y, lt.v2.z)) / 3.0f;
            float3 toL = lp - h.position;
            float d2 = fmaxf(dot(toL, toL), 1e-5f);
            float dist = sqrtf(d2);
            float3 ld = toL / dist;
            float cosS = fmaxf(dot(n, ld), 0.0f);
            float cosL = fmaxf(dot(f3(L.normal.x, L.normal.y, L.normal.z), -ld), 0.0f);
            if (cosS <= 0.0f || cosL <= 0.0f) continue;
            float3 T = f3(1.0f);
            float3 so = h.position + n * 0.001f;
            if (!S.volume_count) sdfCount(S.sdf_counters, kSdfShadowSceneQueries);
            bool occluded = S.volume_count ? shadowWalk(S, mt, so, ld, dist - 0.002f, T)
                                           : shadowLayers(S, mt, opaqueMask, so, ld, dist - 0.002f, T);
            if (occluded) continue;
            float3 brdf = evalBRDF(m, sp, ld);
            float ccGloss = materialClearcoat(m) * powf(1.0f - materialClearcoatRoughness(m), 2.0f);
            float glossW = clampf(metallic + ccGloss +
                                      (1.0f - metallic) * powf(1.0f - roughness, 4.0f) *
                                          clampf(m.parameters2.x, 0.0f, 1.0f),
                                  0.0f, 1.0f);
            float3 f0 = materialF0(m);
            float3 diffuseOnly = (1.0f - metallic) * base * mx(f3(0.0f), f3(1.0f) - f0) * 0.31830988618f;
            brdf = mix3(diffuseOnly, brdf, glossW);
            float G = cosS * cosL * L.area / d2;
            color += brdf * emission * G * T;
        }
        __syncthreads();
        float3 envDiffuse = interactiveDiffuseEnv(axisEnv, n);
        float3 refl = normalize(reflect(-view, n));
        float3 baseRefl = interactiveSpecularEnv(S, refl, n, roughness, envDiffuse);
        float ccRough = materialClearcoatRoughness(m);
        float3 ccRefl = interactiveSpecularEnv(S, refl, n, ccRough, envDiffuse);
        float nDotV = fmaxf(dot(n, view), 0.0f);
        float3 fresnel = fresnelSchlickThinFilm(nDotV, materialF0(m), m);
        float glossy = powf(1.0f - roughness, 4.0f);
        float metalW = metallic * powf(1.0f - roughness, 2.0f);
        float ccW = materialClearcoat(m) * powf(1.0f - ccRough, 3.0f);
        float dielectricW = (1.0f - metallic) * glossy * clampf(m.parameters2.x, 0.0f, 1.0f);
        float3 roughFresnel = mix3(fresnel, materialF0(m), smoothstepf(0.45f, 0.95f, roughness));
        float3 ccFresnel = fresnelSchlickThinFilm(nDotV, materialClearcoatF0Color(m), m);
        float horizon = 0.58f + 0.42f * clampf(n.y * 0.5f + 0.5f, 0.0f, 1.0f);
        float contact = interactiveContactAO(S, mt, hit, h, m, n);
        float diffuseStrength = 0.58f * (1.0f - metallic) * (horizon * contact);
        float baseReflStrength = metalW * 1.05f + dielectricW * 0.32f;
        color += base * envDiffuse * diffuseStrength;
        color += baseRefl * roughFresnel * baseReflStrength;
        color += ccRefl * ccFresnel * ccW * 0.42f;
        const float3 key = normalize(f3(-0.32f, 0.78f, 0.52f));
        color += base * (1.0f - metallic) * fmaxf(dot(n, key), 0.0f) * 0.16f * contact;
        float subsurface = materialSubsurface(m);
        if (subsurface > 0.0f) {
            float wrap = powf(1.0f - nDotV, 2.0f);
            color += clamp3(xyz(m.subsurfaceColor), f3(0.0f), f3(0.999f)) * base * envDiffuse * subsurface *
                     (0.12f + 0.22f * wrap) * contact;
        }
        float transmission = materialTransmission(m);
        if (transmission > 0.0f) {
            float3 transmitted = sampleEnvironmentCall(S, ray.direction);
            color = mix3(color, transmitted * materialTransmissionTint(m, 0.65f), transmission * 0.55f);
            color += baseRefl * fresnel * transmission * 0.35f;
        }
        color = clamp3(color, f3(0.0f), f3(fmaxf(P.clamp, 1.0f)));
        beauty = make_float4(color.x, color.y, color.z, P.transparent_background ? opacity : 1.0f);
        albedo = make_float4(base.x, base.y, base.z, opacity);
    }
    if (!hit) return;
    const float3 enc = ex::add(ex::mul(n, 0.5f), f3(0.5f));
    const float mid = (float)(h.materialID + 1u), oid = (float)(h.objectID + 1u);
    A.aov[0 * plane + pix] = make_float4(h.t, h.t, h.t, 1.0f);
    A.aov[1 * plane + pix] = make_float4(enc.x, enc.y, enc.z, 1.0f);
    A.aov[2 * plane + pix] = albedo;
    A.aov[3 * plane + pix] = make_float4(mid, mid, mid, 1.0f);
    A.aov[4 * plane + pix] = make_float4(oid, oid, oid, 1.0f);
    float2 cur, prev;
    if (projectToScreen(P.cam, h.position, P.width, P.height, cur) &&
        projectToScreen(P.prev_cam, h.position, P.width, P.height, prev))
        A.aov[5 * plane + pix] = make_float4(ex::sub(prev.x, cur.x), ex::sub(prev.y, cur.y), 0.0f, 1.0f);
    else
        A.aov[5 * plane + pix] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    storePreview(A, pix, beauty);
}

// Kahan-compensated accumulation of every path of the batch into its pixel,
// in sample order, plus the AOV block (PathTrace.metal:5559-5585) from the
// batch's last sample.  After every 4096th sample of a pixel the FP32 sum is
// folded into an FP64 resolve buffer, so the result does not depend on how the
// samples were split into batches.
__global__ void __launch_bounds__(256) k_finalize(Wave W) {
    for (uint32_t i = globalId(); i < W.pixel_count; i += gridStride()) {
        const DevJob& J = W.jobs[jobOfPixel(W, i)];
        const DevParams& P = J.P;
        const Accum A = J.A;
        const uint32_t tileN = P.tile_w * P.tile_h;
        uint32_t local = i - J.pixel_begin;
        const float4* rad = W.rad + J.path_begin;
        uint32_t px = P.tile_x + local % P.tile_w, py = P.tile_y + local / P.tile_w;
        size_t pix = (size_t)py * P.width + px;
        float4 s = A.sum[pix], c = A.comp[pix];
        uint32_t count = A.count[pix];
        for (uint32_t k = 0; k < P.samples_in_batch; ++k) {
            float4 r = rad[(size_t)k * tileN + local];
            float y, t;
            y = r.x - c.x; t = s.x + y; c.x = (t - s.x) - y; s.x = t;
            y = r.y - c.y; t = s.y + y; c.y = (t - s.y) - y; s.y = t;
            y = r.z - c.z; t = s.z + y; c.z = (t - s.z) - y; s.z = t;
            y = r.w - c.w; t = s.w + y; c.w = (t - s.w) - y; s.w = t;
            if (((count + k + 1u) & 4095u) == 0u) {  // a 4096-sample block is complete: fold it in FP64
                D4 R = A.resolved[pix];
                R.x += (double)s.x - (double)c.x;
                R.y += (double)s.y - (double)c.y;
                R.z += (double)s.z - (double)c.z;
                R.w += (double)s.w - (double)c.w;
                A.resolved[pix] = R;
                s = make_float4(0, 0, 0, 0);
                c = make_float4(0, 0, 0, 0);
            }
        }
        uint32_t newCount = count + P.samples_in_batch;
        A.sum[pix] = s;
        A.comp[pix] = c;
        A.count[pix] = newCount;
        const size_t st = W.aov_stride;
        float4 a0 = W.aov[i], a1 = W.aov[st + i], a2 = W.aov[2 * st + i], a3 = W.aov[3 * st + i];
        size_t plane = (size_t)P.width * P.height;
        if (__float_as_uint(a0.w) != 0u) {
            float t = a0.x;
            float3 n = f3(a1.x, a1.y, a1.z);
            float3 enc = ex::add(ex::mul(n, 0.5f), f3(0.5f));
            float mid = (float)(__float_as_uint(a0.y) + 1u), oid = (float)(__float_as_uint(a0.z) + 1u);
            A.aov[0 * plane + pix] = make_float4(t, t, t, 1.0f);
            A.aov[1 * plane + pix] = make_float4(enc.x, enc.y, enc.z, 1.0f);
            A.aov[2 * plane + pix] = a2;
            A.aov[3 * plane + pix] = make_float4(mid, mid, mid, 1.0f);
            A.aov[4 * plane + pix] = make_float4(oid, oid, oid, 1.0f);
            float2 cur, prev;
            float3 pos = f3(a3.x, a3.y, a3.z);
            if (projectToScreen(P.cam, pos, P.width, P.height, cur) &&
                projectToScreen(P.prev_cam, pos, P.width, P.height, prev)) {
                A.aov[5 * plane + pix] = make_float4(ex::sub(prev.x, cur.x), ex::sub(prev.y, cur.y), 0.0f, 1.0f);
            } else {
                A.aov[5 * plane + pix] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
        } else {
            A.aov[0 * plane + pix] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            A.aov[1 * plane + pix] = make_float4(0.5f, 0.5f, 0.5f, 0.0f);
            A.aov[2 * plane + pix] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            A.aov[3 * plane + pix] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            A.aov[4 * plane + pix] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            A.aov[5 * plane + pix] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    }
}

// Beauty resolve for readback: (FP64 resolve + FP32 Kahan sum) / samples.
__global__ void k_resolve_beauty(Accum A, uint32_t pixels, float4* out) {
    for (uint32_t i = globalId(); i < pixels; i += gridStride()) {
        uint32_t n = A.count[i];
        if (n == 0u) {
            out[i] = make_float4(0, 0, 0, 0);
            continue;
        }
        D4 R = A.resolved[i];
        float4 s = A.sum[i], c = A.comp[i];
        double inv = 1.0 / (double)n;
        out[i] = make_float4((float)((R.x + ((double)s.x - (double)c.x)) * inv), (float)((R.y + ((double)s.y - (double)c.y)) * inv),
                             (float)((R.z + ((double)s.z - (double)c.z)) * inv), (float)((R.w + ((double)s.w - (double)c.w)) * inv));
    }
}

// ------------------------------------------ environment importance table --
// environmentSamples (Acceleration/LightingGPUEncoding.swift:66-119) with an
// FP64 weight and prefix sum; stored as FP32 {cdf, pdfSolidAngle}.
__global__ void k_env_weights(const float4* px, uint32_t w, uint32_t h, float intensity, float maxR, double* weights) {
    uint32_t n = w * h;
    double dTheta = 3.141592653589793 / (double)h, dPhi = 2.0 * 3.141592653589793 / (double)w;
    for (uint32_t i = globalId(); i < n; i += gridStride()) {
        uint32_t y = i / w;
        double theta = ((double)y + 0.5) * dTheta;
        double solid = fmax(sin(theta) * dTheta * dPhi, 1e-8);
        float4 t = px[i];
        double r = (double)t.x * intensity, g = (double)t.y * intensity, b = (double)t.z * intensity;
        if (maxR > 0.0f) {
            r = fmin(r, (double)maxR);
            g = fmin(g, (double)maxR);
            b = fmin(b, (double)maxR);
        }
        double lum = r * 0.2126 + g * 0.7152 + b * 0.0722;
        weights[i] = fmax(lum, 0.0) * solid;
    }
}

// Block-local inclusive scan (FP64) of 1024 elements per block; block totals out.
__global__ void __launch_bounds__(1024) k_scan_block(double* data, uint32_t n, double* blockSums) {
    __shared__ double warpSums[32];
    uint32_t i = blockIdx.x * 1024u + threadIdx.x;
    double v = i < n ? data[i] : 0.0;
    for (int o = 1; o < 32; o <<= 1) {
        double u = __shfl_up_sync(0xffffffffu, v, o);
        if ((int)laneId() >= o) v += u;
    }
    if (laneId() == 31u) warpSums[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x < 32u) {
        double ws = warpSums[threadIdx.x];
        for (int o = 1; o < 32; o <<= 1) {
            double u = __shfl_up_sync(0xffffffffu, ws, o);
            if ((int)threadIdx.x >= o) ws += u;
        }
        warpSums[threadIdx.x] = ws;
    }
    __syncthreads();
    if ((threadIdx.x >> 5) > 0u) v += warpSums[(threadIdx.x >> 5) - 1u];
    if (i < n) data[i] = v;
    if (threadIdx.x == 1023u) blockSums[blockIdx.x] = v;
}

// Sequential scan of the (few thousand) block totals, then the finished table.
__global__ void k_scan_totals(double* blockSums, uint32_t nb) {
    if (globalId() != 0) return;
    double acc = 0.0;
    for (uint32_t b = 0; b < nb; ++b) {
        double t = blockSums[b];
        blockSums[b] = acc;
        acc += t;
    }
    blockSums[nb] = acc;
}

__global__ void k_env_finish(const double* prefix, const double* blockSums, const double* weights, uint32_t w,
                             uint32_t h, uint32_t nb, float2* out) {
    uint32_t n = w * h;
    double total = blockSums[nb];
    double dTheta = 3.141592653589793 / (double)h, dPhi = 2.0 * 3.141592653589793 / (double)w;
    for (uint32_t i = globalId(); i < n; i += gridStride()) {
        double cum = prefix[i] + blockSums[i >> 10];
        uint32_t y = i / w;
        double theta = ((double)y + 0.5) * dTheta;
        double solid = fmax(sin(theta) * dTheta * dPhi, 1e-8);
        double prob = weights[i] / total;
        out[i] = make_float2((float)fmin(cum / total, 1.0), (float)(prob / solid));
    }
}

}  // namespace dk

// =========================================================== launchers =====
namespace dk {

int kernelGrid(int which, int smCount) {
    int perSM = 1;
    switch (which) {
        case 0: cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, k_generate, 256, 0); break;
        case 1: cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, k_extend<false>, 128, 0); break;
        case 2:
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, k_shade<false>, shadeBlock<false>(), 0);
            break;
        case 3: cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, k_shadow_rays<false>, 128, 0); break;
        case 5: cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, k_extend<true>, 128, 0); break;
        case 6: cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, k_shadow_rays<true>, 128, 0); break;
        case 7: cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, k_volume_march<DistF16>, 128, 0); break;
        case 8: cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, k_subsurface_walk, 128, 0); break;
        default: cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, k_finalize, 256, 0); break;
    }
    return (perSM < 1 ? 1 : perSM) * smCount;
}

cudaError_t launchGenerate(const DevScene& S, const Wave& W, int grid, cudaStream_t st) {
    k_generate<<<grid, 256, 0, st>>>(S, W);
    return cudaGetLastError();
}
cudaError_t launchExtend(const DevScene& S, const Wave& W, uint32_t sel, uint32_t bounce, int grid, int volumeGrid,
                         cudaStream_t st) {
    if (S.wide8)
        k_extend<true><<<grid, 128, 0, st>>>(S, W, sel, bounce);
    else
        k_extend<false><<<grid, 128, 0, st>>>(S, W, sel, bounce);
    if (S.volume_count) {
        if (S.volume_count > 1u || S.sdf_counters) {
            if (S.sdf_counters)  // the counting instantiation only when the session collects them
                k_extend_volume<true><<<volumeGrid, 128, 0, st>>>(S, W, sel);
            else
                k_extend_volume<false><<<volumeGrid, 128, 0, st>>>(S, W, sel);
        } else if (S.brick_dist16) {
            k_volume_march<<<volumeGrid, 128, 0, st>>>(S, W, sel, DistF16{S.brick_dist16});
        } else {
            k_volume_march<<<volumeGrid, 128, 0, st>>>(S, W, sel, DistF32{S.brick_dist});
        }
    }
    return cudaGetLastError();
}
// The environment rotation's sine and cosine with the device's sincosf, the
// values every environment lookup of the reference computes per call.
__global__ void k_env_rotation(float radians, float* out) {
    float sn, cs;
    sincosf(radians, &sn, &cs);
    out[0] = sn;
    out[1] = cs;
}

cudaError_t envRotation(float radians, float* sinCos, cudaStream_t st) {
    k_env_rotation<<<1, 1, 0, st>>>(radians, sinCos);
    return cudaGetLastError();
}

int g_sortMaterials = -1;  // -1: from DK_SORT_MATERIALS (default on)

// Kernels one bounce launches (extend, shade, shadow, resolve stages).
uint32_t bounceLaunches(const DevScene& S, const Wave& W) {
    if (g_sortMaterials < 0) {
        const char* e = getenv("DK_SORT_MATERIALS");
        g_sortMaterials = (e && e[0] == '0') ? 0 : 1;
    }
    uint32_t n = 1u + (S.volume_count ? 1u : 0u);                  // extend
    n += (g_sortMaterials ? 2u : 0u) + (S.has_subsurface && !S.volume_count && !S.wide8 ? 2u : 1u) + 2u;  // sort, (walk,) shade, survivors
    n += liveBlocks(W) > kLiveDirect ? 1u : 0u;
    n += 1u + ((!S.all_shadow_opaque || S.volume_count) ? 1u : 0u);  // shadow
    return n + 1u;                                                   // resolve
}

cudaError_t launchShade(const DevScene& S, const Wave& W, uint32_t bounce, uint32_t sel, int grid, int walkGrid,
                        cudaStream_t st) {
    if (g_sortMaterials < 0) {
        const char* e = getenv("DK_SORT_MATERIALS");
        g_sortMaterials = (e && e[0] == '0') ? 0 : 1;
    }
    uint32_t sorted = (uint32_t)g_sortMaterials;
    if (sorted) {
        const bool small = W.path_count < kSortSmall;
        const uint32_t perBlock = 256u * (small ? 2u : 8u), sortBlocks = (W.path_count + perBlock - 1u) / perBlock;
        // A gather of hits and materials, bound by latency: eight blocks per SM, four times shading's two
        // (with those 65 us a launch under ncu at 16.6 M paths; the frame takes 1.6 % less).
        k_sort_count<<<std::min(4u * (uint32_t)grid, sortBlocks), 256, 0, st>>>(S, W, sel);
        if (small)
            k_sort_scatter<2><<<sortBlocks, 256, 0, st>>>(W, sel);
        else
            k_sort_scatter<8><<<sortBlocks, 256, 0, st>>>(W, sel);
    }
    // The general shading kernel (volume hits, random walks through
    // traceScene) also serves the 8-wide tree, keeping the layout switch out
    // of the triangle-only kernels.
    if (S.volume_count || S.wide8) {
        k_shade<true><<<std::max(1, grid * shadeBlock<false>() / shadeBlock<true>()), shadeBlock<true>(), 0, st>>>(
            S, W, bounce, sel, sorted);
    } else {
        if (S.has_subsurface) k_subsurface_walk<<<walkGrid, 128, 0, st>>>(S, W, sel, sorted);
        k_shade<false><<<grid, shadeBlock<false>(), 0, st>>>(S, W, bounce, sel, sorted);
    }
    // The survivors, in path order, are the next bounce's queue.
    const uint32_t blocks = liveBlocks(W);
    if (blocks) {
        k_live_count<<<blocks, 256, 0, st>>>(W);
        if (blocks > kLiveDirect) k_live_scan<<<1, 256, 0, st>>>(W, blocks);
        k_live_scatter<<<blocks, 256, 0, st>>>(W, sel);
    }
    return cudaGetLastError();
}
cudaError_t launchShadow(const DevScene& S, const Wave& W, int grid, cudaStream_t st) {
    if (S.wide8)
        k_shadow_rays<true><<<grid, 128, 0, st>>>(S, W);
    else
        k_shadow_rays<false><<<grid, 128, 0, st>>>(S, W);
    if (S.volume_count)
        k_shadow_layers<true><<<grid, 128, 0, st>>>(S, W);
    else if (!S.all_shadow_opaque)
        k_shadow_layers<false><<<grid, 128, 0, st>>>(S, W);
    return cudaGetLastError();
}
cudaError_t launchResolve(const Wave& W, int grid, cudaStream_t st) {
    k_resolve<<<grid, 256, 0, st>>>(W);
    return cudaGetLastError();
}
cudaError_t launchAovPrimary(const DevScene& S, const Wave& W, int grid, cudaStream_t st) {
    k_aov_primary<<<grid, 128, 0, st>>>(S, W);
    return cudaGetLastError();
}
cudaError_t launchPreview(const DevScene& S, const DevParams& P, const Accum& A, uint32_t matCount,
                          uint32_t opaqueMask, bool interactive, cudaStream_t st) {
    const MatTable mt{0u, matCount};
    const uint64_t pixels = (uint64_t)P.tile_w * P.tile_h;
    if (!pixels) return cudaSuccess;
    // us a frame, blocks of 32 / 128 / 512 threads (a general loop of 128 before them all), interactive quality:
    // material scene 200 x 150 173 / 177 / 223 (269), 400 x 300 282 / 208 / 232 (605), 640 x 360 450 / 302 / 247;
    // 82,000 triangles 64 x 64 631 / 707 / 972 (658), 400 x 300 1015 / 967 / 1214, 640 x 360 1614 / 1333 / 1188;
    // 768^3 volume 200 x 150 831 / 1095 / 1717 (882), 1280 x 720 2449 / 1856 / 2754.  Preview quality likewise.
    const uint64_t small = S.volume_count ? 150000u : 40000u;
    const uint32_t block = pixels < small ? kPreviewSmall
                           : S.volume_count || pixels < 200000u ? kPreviewMid : kPreviewLarge;
    const uint64_t warps = block == kPreviewSmall ? (pixels + 31u) / 32u
                                                  : (uint64_t)((P.tile_w + 7u) / 8u) * ((P.tile_h + 3u) / 4u);
    const uint32_t grid = (uint32_t)((warps * 32u + block - 1u) / block);
    auto kernel = block == kPreviewLarge ? (interactive ? k_preview<true, kPreviewLarge> : k_preview<false, kPreviewLarge>)
                  : block == kPreviewMid ? (interactive ? k_preview<true, kPreviewMid> : k_preview<false, kPreviewMid>)
                                         : (interactive ? k_preview<true, kPreviewSmall> : k_preview<false, kPreviewSmall>);
    kernel<<<grid, block, 0, st>>>(S, P, A, mt, opaqueMask);
    return cudaGetLastError();
}
cudaError_t launchFinalize(const Wave& W, int grid, cudaStream_t st) {
    k_finalize<<<grid, 256, 0, st>>>(W);
    return cudaGetLastError();
}
cudaError_t launchResolveBeauty(const Accum& A, uint32_t pixels, float4* out, int grid, cudaStream_t st) {
    k_resolve_beauty<<<grid, 256, 0, st>>>(A, pixels, out);
    return cudaGetLastError();
}
cudaError_t buildEnvironmentTable(const float4* dPixels, uint32_t w, uint32_t h, float intensity, float maxR,
                                  double* dWeights, double* dPrefix, double* dBlockSums, float2* dOut, int grid,
                                  cudaStream_t st, double* hostTotal) {
    uint32_t n = w * h;
    uint32_t nb = (n + 1023u) / 1024u;
    k_env_weights<<<grid, 256, 0, st>>>(dPixels, w, h, intensity, maxR, dWeights);
    cudaError_t e = cudaMemcpyAsync(dPrefix, dWeights, sizeof(double) * n, cudaMemcpyDeviceToDevice, st);
    if (e != cudaSuccess) return e;
    k_scan_block<<<nb, 1024, 0, st>>>(dPrefix, n, dBlockSums);
    k_scan_totals<<<1, 32, 0, st>>>(dBlockSums, nb);
    e = cudaMemcpyAsync(hostTotal, dBlockSums + nb, sizeof(double), cudaMemcpyDeviceToHost, st);
    if (e != cudaSuccess) return e;
    e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return e;
    if (!(*hostTotal > 0.0)) return cudaSuccess;
    k_env_finish<<<grid, 256, 0, st>>>(dPrefix, dBlockSums, dWeights, w, h, nb, dOut);
    return cudaGetLastError();
}

}  // namespace dk
