// seis3d_views.cuh - display extraction of the 3-D solver (extractViews3D, reference
// cuda/Cuda_Seis3D.cu:334-418,627-646) without a graphics stack: three packed physical
// slices (XZ at y = sy, YZ at x = sx, XY at z = sz, each including the visible CPML) and an
// optional bounded volume resampled trilinearly at cell centres, written as interleaved
// (wave value, material value) pairs into a caller-owned device buffer, with the reference's
// colour statistics (largest |value|, material range, largest velocity magnitude).
//
// The per-sample arithmetic is the reference's (collocated face velocities, material
// transforms, trilinear weights), read from this solver's pitched volumes.  Output samples are
// independent; the grid strides over them.
#pragma once

#include "../../include/seis3d_capi.h"

#include <cstdint>

namespace seis3d {

struct ViewArgs {
    const float* v[3];      // vx, vy, vz
    const float* s[3];      // sxx, syy, szz
    const float* invRho;
    const float* lambda;
    const float* mu;
    int64_t pitch, plane;
    int ox, oy, oz;         // physical origin inside the padded volume
    int nx, ny, nz;         // physical size
    seis3d_view_layout layout;
    int sx, sy, sz;
    int includeBoundary;
    float* out;
    unsigned* stats;        // [0] |value| max, [2] material min, [3] material max, [4] |v| max
    unsigned* nonFinite;    // the session's non-finite flag
};

// One sample: the displayed wave value, the velocity magnitude and the material value.
struct ViewSample { float value, magnitude, material; };

// sampleScalar3D (cuda/Cuda_Seis3D.cu:335-352) at the cell with offset i.  Components: 0 vz, 1 vx,
// 2 vy, 3 |v|, 4 pressure, 5 vp, 6 vs, 7 rho; the magnitude is 0 where a material is the wave.
template <int kMaterial> __device__ __forceinline__ float viewMaterial(const ViewArgs& a, int64_t i) {
    if (kMaterial == 5) return sqrtf((a.lambda[i] + 2 * a.mu[i]) * a.invRho[i]);
    if (kMaterial == 6) return sqrtf(a.mu[i] * a.invRho[i]);
    return 1 / a.invRho[i];
}

template <int kWave, int kMaterial> __device__ __forceinline__ ViewSample viewCell(const ViewArgs& a, int64_t i) {
    ViewSample s;
    s.material = viewMaterial<kMaterial>(a, i);
    if (kWave >= 5) {
        s.value = viewMaterial<kWave>(a, i);
        s.magnitude = 0;
        return s;
    }
    const float vx = 0.5f * (a.v[0][i] + a.v[0][i - 1]);
    const float vy = 0.5f * (a.v[1][i] + a.v[1][i - a.pitch]);
    const float vz = 0.5f * (a.v[2][i] + a.v[2][i - a.plane]);
    s.magnitude = sqrtf(vx * vx + vy * vy + vz * vz);
    if (kWave == 4) s.value = -(a.s[0][i] + a.s[1][i] + a.s[2][i]) / 3;
    else s.value = kWave == 0 ? vz : kWave == 1 ? vx : kWave == 2 ? vy : s.magnitude;
    return s;
}

// resampleScalar3D (:355-367): trilinear over the 8 cells around (x, y, z); cells of weight 0 are
// not read.  The corners are unrolled, so the loads of all of them are in flight together.
template <int kWave, int kMaterial>
__device__ __forceinline__ ViewSample viewResample(const ViewArgs& a, float x, float y, float z) {
    const int ix = int(floorf(x)), iy = int(floorf(y)), iz = int(floorf(z));
    const float fraction[3] = {x - ix, y - iy, z - iz};
    const int64_t origin = int64_t(iz + a.oz) * a.plane + int64_t(iy + a.oy) * a.pitch + (ix + a.ox);
    ViewSample corner[8];
    float weight[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int dx = k & 1, dy = (k >> 1) & 1, dz = k >> 2;
        weight[k] = (dx ? fraction[0] : 1 - fraction[0]) * (dy ? fraction[1] : 1 - fraction[1]) *
                    (dz ? fraction[2] : 1 - fraction[2]);
        corner[k] = ViewSample{0.0f, 0.0f, 0.0f};
        if (weight[k] > 0) corner[k] = viewCell<kWave, kMaterial>(a, origin + dz * a.plane + dy * a.pitch + dx);
    }
    ViewSample s{0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int k = 0; k < 8; ++k)
        if (weight[k] > 0) {
            s.value += weight[k] * corner[k].value;
            s.magnitude += weight[k] * corner[k].magnitude;
            s.material += weight[k] * corner[k].material;
        }
    return s;
}

// Extremes of a thread's samples, then of the block's.
struct ViewExtremes { float wave, velocity, low, high; };

__device__ __forceinline__ void reduceExtremes(ViewExtremes& e) {
#pragma unroll
    for (int offset = 16; offset > 0; offset /= 2) {
        e.wave = fmaxf(e.wave, __shfl_down_sync(0xffffffffu, e.wave, offset));
        e.velocity = fmaxf(e.velocity, __shfl_down_sync(0xffffffffu, e.velocity, offset));
        e.low = fminf(e.low, __shfl_down_sync(0xffffffffu, e.low, offset));
        e.high = fmaxf(e.high, __shfl_down_sync(0xffffffffu, e.high, offset));
    }
}

constexpr int kViewThreads = 256;

// The grid strides over the samples (at most 2^24 of the volume and three slices, so 32-bit
// indices serve), and a block reduces its statistics before its four atomics: one set per
// warp of samples meant 600,000 atomics on four words for the 324x74x312 domain, which
// serialised in L2 and were most of the kernel's 435 us (136 us now; 33 us at the copy rate).
template <int kWave, int kMaterial>
__global__ void __launch_bounds__(kViewThreads) extractViews(const __grid_constant__ ViewArgs a, unsigned limit) {
    const seis3d_view_layout& L = a.layout;
    const unsigned nx = L.domainSize3D[0], ny = L.domainSize3D[1];
    const int ox = L.domainOrigin3D[0], oy = L.domainOrigin3D[1], oz = L.domainOrigin3D[2];
    const unsigned slice1 = unsigned(L.sliceOffset3D[1]), slice2 = unsigned(L.sliceOffset3D[2]);
    const unsigned volume = unsigned(L.volumeOffset3D);
    const unsigned VX = L.volumeX3D, VY = L.volumeY3D;
    const bool paired = reinterpret_cast<uintptr_t>(a.out) % 8 == 0;   // the output may start at any float
    ViewExtremes e{0.0f, 0.0f, 3.402823466e38f, 0.0f};
    bool bad = false;
    for (unsigned i = blockIdx.x * kViewThreads + threadIdx.x; i < limit; i += gridDim.x * kViewThreads) {
        int x, y, z;
        ViewSample s;
        if (i < volume) {
            if (i < slice1) {
                x = int(i % nx) + ox; y = a.sy; z = int(i / nx) + oz;
            } else if (i < slice2) {
                const unsigned j = i - slice1;
                x = a.sx; y = int(j % ny) + oy; z = int(j / ny) + oz;
            } else {
                const unsigned j = i - slice2;
                x = int(j % nx) + ox; y = int(j / nx) + oy; z = a.sz;
            }
            s = viewCell<kWave, kMaterial>(a, int64_t(z + a.oz) * a.plane + int64_t(y + a.oy) * a.pitch + (x + a.ox));
        } else {
            const unsigned j = i - volume;
            const float fx = (float(j % VX) + .5f) * float(nx) / VX - .5f + ox;
            const float fy = (float((j / VX) % VY) + .5f) * float(ny) / VY - .5f + oy;
            const float fz = (float(j / (VX * VY)) + .5f) * float(L.domainSize3D[2]) / L.volumeZ3D - .5f + oz;
            x = int(floorf(fx)); y = int(floorf(fy)); z = int(floorf(fz));
            s = viewResample<kWave, kMaterial>(a, fx, fy, fz);
        }
        const bool waveFinite = isfinite(s.value), materialFinite = isfinite(s.material), speedFinite = isfinite(s.magnitude);
        const float wave = waveFinite ? s.value : 0, material = materialFinite ? s.material : 0;
        if (paired) {
            reinterpret_cast<float2*>(a.out)[i] = make_float2(wave, material);
        } else {
            a.out[2 * i] = wave;
            a.out[2 * i + 1] = material;
        }
        bad |= !waveFinite || !materialFinite || !speedFinite || s.material < 0;
        const bool physical = x >= 0 && x < a.nx && y >= 0 && y < a.ny && z >= 0 && z < a.nz;
        if ((physical || a.includeBoundary) && waveFinite) e.wave = fmaxf(e.wave, fabsf(s.value));
        if ((physical || a.includeBoundary) && speedFinite) e.velocity = fmaxf(e.velocity, s.magnitude);
        if (physical && materialFinite) {
            e.low = fminf(e.low, s.material);
            e.high = fmaxf(e.high, s.material);
        }
    }
    if (bad) atomicExch(a.nonFinite, 1u);
    reduceExtremes(e);
    __shared__ ViewExtremes warps[kViewThreads / 32];
    if ((threadIdx.x & 31) == 0) warps[threadIdx.x / 32] = e;
    __syncthreads();
    if (threadIdx.x >= 32) return;
    if (threadIdx.x < kViewThreads / 32) e = warps[threadIdx.x];
    reduceExtremes(e);
    if (threadIdx.x == 0) {
        // Non-negative floats order like their bit patterns.
        atomicMax(a.stats, __float_as_uint(e.wave));
        atomicMin(a.stats + 2, __float_as_uint(e.low));
        atomicMax(a.stats + 3, __float_as_uint(e.high));
        atomicMax(a.stats + 4, __float_as_uint(e.velocity));
    }
}

}  // namespace seis3d
