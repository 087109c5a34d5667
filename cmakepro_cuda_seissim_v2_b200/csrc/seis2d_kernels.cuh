// seis2d_kernels.cuh - sm_100a kernels of the 2-D P-SV velocity-stress solver.
//
// The reference runs four to five launches per step (CUDA_Kernels/Cuda_Check.cu:1027-1085):
// stress, free-surface mirror, velocity, a one-thread source injection and an edge clear,
// each thread re-reading both halves of every split field from global memory for each of
// its sixteen stencil taps.  Here one step is two kernels:
//
//   stressStep   - stress update of all three schemes; the free-surface mirror is written by
//                  the threads that own the mirrored rows; the stress-type point source of the
//                  previous step is folded into the old value it would have been added to;
//                  an extra row of blocks samples the receivers of the previous step.
//   velocityStep - velocity update; air rows cleared; the force-type point source of this
//                  step is added by the thread that owns the source cell; the outer ring of
//                  velocities is cleared by the threads that own it.
//
// plus, at the end of a batch, finishBatch (stress-type source and receivers of the last
// step) so that the field state between API calls is the reference's.  Threads own columns and
// keep the rows around theirs in register windows (see "strips").  Each expression keeps the
// reference's operand order ((a1 + a2 - b1 - b2) per tap, the same tap order and the same
// averaging order) and the arithmetic matches the reference kernels operation for operation.
// Grids that fit on the chip run many steps in one launch instead (seis2d_resident.cuh), with
// the same cell updates and so the same bits.
// The translation unit is compiled with --use_fast_math, the flag the reference builds its
// 2-D solver with (CMakeLists.txt:128-135).
//
// The grid is at most INT_MAX cells (checkedGridElementCount), so 32-bit indices suffice.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

#include "../../include/seis2d_capi.h"

namespace seis2d {

// Programmatic dependent launch: a step kernel may become resident once every block of the one
// before it has called launchDependents, and waits in waitForPrevious until that one has
// completed.  Both are no-ops in an ordinary launch.
__device__ __forceinline__ void launchDependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void waitForPrevious() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

constexpr int kThreads = 128;         // columns a block loads, one per thread
constexpr int kHalo = 4;              // stencil radius (kStencilRadius, SolverNumerics.h:9)
constexpr int kCols = kThreads - 2 * kHalo;   // columns a block updates

// Rows a thread updates.  More rows mean fewer halo rows read per cell (R + 7 for R), fewer rows more
// blocks and a shorter chain in each: us a step of 1 / 2 / 3 / 4 rows on 120x100 4.1 / 4.9 / 5.2 /
// 5.8, 250x220 5.6 / 5.7 / 5.6 / 6.1, 250x300 6.1 / 5.8 / 6.0 / 6.3, 400x350 8.3 / 7.3 / 7.4 / 7.4,
// 440x420 9.3 / 8.5 / 7.6 / 7.5, 1601x1203 78 / 67 / 63 / 60 (split halves), 250x300 5.5 / 5.3 / 5.7
// / 6.2, 1601x1203 46 / 40 / 38 / 37 (hybrid).
__host__ __device__ __forceinline__ int stripRows(int cells) { return cells <= 55000 ? 1 : cells <= 150000 ? 2 : 4; }

// Scheme ids of the kernels (flag_type, with flag 3 and upFlag off run as flag 1;
// Cuda_Check.cu:1038-1046).
enum Scheme { kSplit = 1, kHybrid = 2, kFree = 3 };

struct Grid2D {
    int NX, NZ, total;
    int npml, fs;
    float dt, inv_dt;
    float c1, c2, c3, c4;
};

// Device buffers of a session (GPUSimData, Cuda_Check.cuh:68-121).
struct Fields2D {
    float *vx1, *vx2, *vz1, *vz2, *sxx1, *sxx2, *szz1, *szz2, *sxz1, *sxz2;
    float *vx, *vz, *sxx, *szz, *sxz;
    const float *rho, *mu, *lambda, *l2m;
    const float *muX, *lambdaX, *l2mX, *muZ, *rhoXZ, *rhoOrig;
    const float *dx, *dxh, *dz, *dzh, *dp;
};

// Per-run control block in device memory, written by configureRun before the steps of a
// run so that one captured graph serves every start step, source and receiver set.
struct Control2D {
    int base;            // step index of graph slot 0; finishBatch advances it
    int srcSingle;       // 1: the context's point source (num_active_sources < 0)
    int srcIdx;          // flat source index after the free-surface clamp
    int srcValid;        // the index passes applyPointSource's bounds checks
    int srcType;
    int srcLength;       // steps that have a wavelet sample: min(nt, wavelet size)
    float srcAngle;
    int multiCount;      // active sources injected after each velocity update
    int multiAdvance;    // advance the active sources' time by dt before each step
    int rcvCount;        // receivers sampled into the gather
    int gatherOn;
    int gatherStart, gatherStride, gatherSamples;
    const float* series; // wavelet * src_amp * 1e7 per step (computed on the host like the reference)
    const int* rcvIdx;
    float* gatherVx;
    float* gatherVz;
    seis2d_source* sources;
};

// ---- strips ------------------------------------------------------------------------------
//
// A block updates R rows of kCols columns (stripRows).  A thread owns one column: it loads the rows its
// z derivatives span straight into registers (R + 7 per array) and shares only its own rows
// through shared memory for its neighbours' x derivatives; the first and last four threads only
// share.  All loads (the cells' own values and materials too) are issued before the one
// barrier, so a block waits for memory once.

// Offsets of rows row-4 .. row+R+3 of a thread's column, formed once for all arrays: with an index, a
// test and a 64-bit address for each load a hybrid cell took 270 instructions.  Rows past
// the grid, in its last strip, repeat the last one: only cells that are not updated read them.
template <int R> struct Rows {
    unsigned o[R + 8];
    __device__ __forceinline__ Rows(const Grid2D& g, int row, int j) {
#pragma unroll
        for (int k = 0; k < R + 8; ++k) o[k] = unsigned(min(row - 4 + k, g.NZ - 1)) * unsigned(g.NX) + unsigned(j);
    }
    __device__ __forceinline__ unsigned own(int r) const { return o[4 + r]; }
};

// One array of a strip as its thread holds it: R + 7 rows of its column, from `before` rows above its own.
template <int R> struct Column {
    float v[R + 7];
    __device__ __forceinline__ void load(const float* f, const Rows<R>& rows, int before) {
        // L2-only loads: the next kernel rewrites these fields, and L1 keeps what is read again
        // (materials, damping).
#pragma unroll
        for (int k = 0; k < R + 7; ++k) v[k] = __ldcg(f + rows.o[4 - before + k]);
    }
    // The thread's own rows only, where they stand in a column that starts `before` rows earlier.
    __device__ __forceinline__ void loadOwn(const float* f, const Rows<R>& rows, int before) {
#pragma unroll
        for (int r = 0; r < R; ++r) v[before + r] = __ldcg(f + rows.own(r));
    }
};

using Shared = float[kThreads];   // one row of one array across the block

// Weighted sum of four taps, in the reference's order.  The roundings that the compiler's
// contraction gives the reference's expression are written out, here and in advance, so that
// the results do not depend on how the surrounding code is arranged.
__device__ __forceinline__ float weigh(const Grid2D& g, float t1, float t2, float t3, float t4) {
    return __fmaf_rn(g.c4, t4, __fmaf_rn(g.c3, t3, __fmaf_rn(g.c1, t1, __fmul_rn(g.c2, t2))));
}

struct Damp;
// Damping of the thread's column and rows, loaded with everything else: between the rows' stores
// each of these loads would wait for memory on its own.
template <int R> struct Damping {
    float x, xh, z[R], zh[R];
    __device__ __forceinline__ void load(const Grid2D& g, const Fields2D& f, int row, int j) {
        x = f.dx[j]; xh = f.dxh[j];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int i = min(row + r, g.NZ - 1);
            z[r] = f.dz[i]; zh[r] = f.dzh[i];
        }
    }
    // Of own row r; `undamped` rows near a free surface have no damping along z.
    __device__ __forceinline__ Damp at(int r, bool undamped) const;
};

// One split half: (old (1/dt - d) + m D) / (1/dt + d).
__device__ __forceinline__ float advance(const Grid2D& g, float old, float d, float m, float derivative) {
    return __fmaf_rn(old, g.inv_dt - d, __fmul_rn(m, derivative)) / (g.inv_dt + d);
}

// Split-field first derivatives (Cuda_Check.cu:236-254, 283-304, 434-486, 530-559): each tap is the
// two halves of the upper sample minus the two halves of the lower sample, in that order, so the
// sum of the upper halves is formed once per sample and shared by the taps it is in.
struct SplitRow {
    const float *a, *b, *s;   // halves and their sum across the block, at the thread's column
    __device__ __forceinline__ float tap(int u, int l) const { return s[u] - a[l] - b[l]; }
};
__device__ __forceinline__ float dxForward(const Grid2D& g, const SplitRow& f) {
    return weigh(g, f.tap(1, 0), f.tap(2, -1), f.tap(3, -2), f.tap(4, -3));
}
__device__ __forceinline__ float dxBackward(const Grid2D& g, const SplitRow& f) {
    return weigh(g, f.tap(0, -1), f.tap(1, -2), f.tap(2, -3), f.tap(3, -4));
}
template <int R> struct SplitColumn {
    Column<R> a, b;
    float s[R + 7];
    __device__ __forceinline__ void sum() {
#pragma unroll
        for (int k = 0; k < R + 7; ++k) s[k] = a.v[k] + b.v[k];
    }
    __device__ __forceinline__ float tap(int u, int l) const { return s[u] - a.v[l] - b.v[l]; }
    // z derivative of own row r: 8 rows from r, both directions (the column starts 3 rows above the
    // strip for the forward one, 4 for the backward one).
    __device__ __forceinline__ float dz(const Grid2D& g, int r) const {
        return weigh(g, tap(r + 4, r + 3), tap(r + 5, r + 2), tap(r + 6, r + 1), tap(r + 7, r));
    }
};

// Total-field derivatives of the hybrid scheme (Cuda_Check.cu:324-334, 377-387).
__device__ __forceinline__ float dxForward(const Grid2D& g, const float* f) {
    return weigh(g, f[1] - f[0], f[2] - f[-1], f[3] - f[-2], f[4] - f[-3]);
}
__device__ __forceinline__ float dxBackward(const Grid2D& g, const float* f) {
    return weigh(g, f[0] - f[-1], f[1] - f[-2], f[2] - f[-3], f[3] - f[-4]);
}
template <int R> __device__ __forceinline__ float dzAt(const Grid2D& g, const Column<R>& c, int r) {
    return weigh(g, c.v[r + 4] - c.v[r + 3], c.v[r + 5] - c.v[r + 2], c.v[r + 6] - c.v[r + 1], c.v[r + 7] - c.v[r]);
}

// The same with the term as it is.
__device__ __forceinline__ float advanceBy(const Grid2D& g, float old, float d, float term) {
    return __fmaf_rn(old, g.inv_dt - d, term) / (g.inv_dt + d);
}

// ---- cell updates --------------------------------------------------------------------------

struct Damp { float x, xh, z, zh; };   // of one cell, whole and half node, along x and z

template <int R> __device__ __forceinline__ Damp Damping<R>::at(int r, bool undamped) const {
    return Damp{x, xh, undamped ? 0.0f : z[r], undamped ? 0.0f : zh[r]};
}

// Hybrid stresses (Cuda_Check.cu:315-364): totals inside, sums of damped halves in the layer.
// h: sxz1, sxz2, sxx1, szz1, sxx2, szz2.
__device__ __forceinline__ void hybridStress(const Grid2D& g, bool pml, const Damp& d, float muZ, float l2mX, float lambdaX,
                                             float dvz_dx, float dvx_dz, float dvx_dx, float dvz_dz, float& sxz, float& sxx,
                                             float& szz, float (&h)[6]) {
    if (!pml) {
        sxz = __fmaf_rn(g.dt * muZ, dvz_dx + dvx_dz, sxz);
        sxx = __fmaf_rn(g.dt, __fmaf_rn(l2mX, dvx_dx, __fmul_rn(lambdaX, dvz_dz)), sxx);
        szz = __fmaf_rn(g.dt, __fmaf_rn(lambdaX, dvx_dx, __fmul_rn(l2mX, dvz_dz)), szz);
        return;
    }
    h[0] = advance(g, h[0], d.x, muZ, dvz_dx);
    h[1] = advance(g, h[1], d.zh, muZ, dvx_dz);
    h[2] = advance(g, h[2], d.xh, l2mX, dvx_dx);
    h[3] = advance(g, h[3], d.xh, lambdaX, dvx_dx);
    h[4] = advance(g, h[4], d.z, lambdaX, dvz_dz);
    h[5] = advance(g, h[5], d.z, l2mX, dvz_dz);
    sxz = h[0] + h[1];
    sxx = h[2] + h[4];
    szz = h[3] + h[5];
}

// Hybrid velocities (Cuda_Check.cu:368-412).  h: vz1, vz2, vx1, vx2.
__device__ __forceinline__ void hybridVelocity(const Grid2D& g, bool pml, const Damp& d, float rhoXZ, float rho,
                                               float dsigxz_dx, float dsigzz_dz, float dsigxx_dx, float dsigxz_dz, float& vx,
                                               float& vz, float (&h)[4]) {
    if (!pml) {
        vz = __fmaf_rn(g.dt * (dsigxz_dx + dsigzz_dz), __fdividef(1.0f, rhoXZ), vz);
        vx = __fmaf_rn(g.dt * (dsigxx_dx + dsigxz_dz), __fdividef(1.0f, rho), vx);
        return;
    }
    h[0] = advanceBy(g, h[0], d.xh, dsigxz_dx / rhoXZ);
    h[1] = advanceBy(g, h[1], d.zh, dsigzz_dz / rhoXZ);
    h[2] = advanceBy(g, h[2], d.x, dsigxx_dx / rho);
    h[3] = advanceBy(g, h[3], d.z, dsigxz_dz / rho);
    vx = h[2] + h[3];
    vz = h[0] + h[1];
}

// The stress-type point source, half of it into each split half.
__device__ __forceinline__ void addSplitSource(const Control2D& c, float w, float (&s)[6]) {
    const float half = w * 0.5f;
    if (c.srcType == SEIS2D_EXPLOSIVE) {
#pragma unroll
        for (int h = 0; h < 4; ++h) s[h] = __fadd_rn(s[h], half);
    } else {
        s[4] = __fadd_rn(s[4], half); s[5] = __fadd_rn(s[5], half);
    }
}

// Split-field stresses (Cuda_Check.cu:224-266, 453-487).  s: sxx1, sxx2, szz1, szz2, sxz1, sxz2.
__device__ __forceinline__ void splitStress(const Grid2D& g, const Damp& d, float mu, float l2m, float lambda, float dvx_dx,
                                            float dvz_dz, float dvz_dx, float dvx_dz, float (&s)[6]) {
    s[0] = advance(g, s[0], d.xh, l2m, dvx_dx);
    s[1] = advance(g, s[1], d.z, lambda, dvz_dz);
    s[2] = advance(g, s[2], d.xh, lambda, dvx_dx);
    s[3] = advance(g, s[3], d.z, l2m, dvz_dz);
    s[4] = advance(g, s[4], d.x, mu, dvz_dx);
    s[5] = advance(g, s[5], d.zh, mu, dvx_dz);
}

// The traction-free row (Cuda_Check.cu:431-452); the shear derivatives take two taps there.
__device__ __forceinline__ void freeRowStress(const Grid2D& g, const Damp& d, float mu, float dp, float dvx_dx, float dvz_dx,
                                              float dvx_dz, float (&s)[6]) {
    s[0] = advance(g, s[0], d.xh, dp, dvx_dx);
    s[1] = s[2] = s[3] = 0.0f;
    s[4] = advance(g, s[4], d.x, mu, dvz_dx);
    s[5] = advance(g, s[5], d.zh, mu, dvx_dz);
}
__device__ __forceinline__ float weigh2(const Grid2D& g, float t1, float t2) { return __fmaf_rn(g.c1, t1, __fmul_rn(g.c2, t2)); }

// Split-field velocities (Cuda_Check.cu:270-311, 512-563).  v: vx1, vx2, vz1, vz2.
__device__ __forceinline__ void splitVelocity(const Grid2D& g, const Damp& d, float rho, float rhoMean, float dsigxx_dx,
                                              float dsigxz_dz, float dsigxz_dx, float dsigzz_dz, float (&v)[4]) {
    v[0] = advanceBy(g, v[0], d.x, dsigxx_dx / rho);
    v[1] = advanceBy(g, v[1], d.z, dsigxz_dz / rho);
    v[2] = advanceBy(g, v[2], d.xh, dsigxz_dx / rhoMean);
    v[3] = advanceBy(g, v[3], d.zh, dsigzz_dz / rhoMean);
}

// The hybrid scheme's absorbing cells, whose totals are the sums of their halves.
__device__ __forceinline__ bool inPml(const Grid2D& g, int i, int j) {
    return i < g.npml || i >= g.NZ - g.npml || j < g.npml || j >= g.NX - g.npml;
}

// Rows of shared memory a strip needs: the arrays with x derivatives (halves and sum).
template <int S> constexpr int kSharedArrays = S == kHybrid ? 2 : 6;

// R rows of one array at the thread's column (own values and materials).
template <int R> __device__ __forceinline__ void loadRows(float (&v)[R], const float* f, const Rows<R>& rows) {
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = __ldcg(f + rows.own(r));
}

// Receiver sample of the current state (extractReceiverSamplesKernel, Cuda_Check.cu:793-818).
template <int S>
__device__ __forceinline__ void sampleReceiver(const Grid2D& g, const Fields2D& f, int k, float& vx, float& vz) {
    if (k < 0 || k >= g.total) { vx = 0.0f; vz = 0.0f; return; }
    if (S == kHybrid) { vx = __ldcg(f.vx + k); vz = __ldcg(f.vz + k); }
    else { vx = __ldcg(f.vx1 + k) + __ldcg(f.vx2 + k); vz = __ldcg(f.vz1 + k) + __ldcg(f.vz2 + k); }
}

// Gather row of step `step` (the recording rule of src/Seis2D/Workflow2D.inc:320-345).
template <int S>
__device__ void recordStep(const Grid2D& g, const Fields2D& f, const Control2D& c, int step, int tid, int nthreads) {
    if (!c.gatherOn) return;
    const int rs = step - c.gatherStart;
    if (rs < 0 || rs % c.gatherStride != 0) return;
    const int sample = rs / c.gatherStride;
    if (sample >= c.gatherSamples) return;
    for (int r = tid; r < c.rcvCount; r += nthreads) {
        float vx, vz;
        sampleReceiver<S>(g, f, c.rcvIdx[r], vx, vz);
        c.gatherVx[std::size_t(r) * c.gatherSamples + sample] = vx;
        c.gatherVz[std::size_t(r) * c.gatherSamples + sample] = vz;
    }
}

// Stress-type point-source value of `step` (applyPointSource types 2 and 3,
// Cuda_Check.cu:602-621); 0 when that step injects nothing.
__device__ __forceinline__ bool stressSource(const Control2D& c, int step, float& w) {
    if (!c.srcSingle || !c.srcValid || (c.srcType != SEIS2D_EXPLOSIVE && c.srcType != SEIS2D_SHEAR)) return false;
    if (step < 0 || step >= c.srcLength) return false;
    w = c.series[step];
    return isfinite(w);
}

// ---- launch shapes -------------------------------------------------------------------------

// Strips of a grid: across, and down for the stresses and the velocities.
__host__ __device__ __forceinline__ int stripsAcross(const Grid2D& g) { return (g.NX - 8 + kCols - 1) / kCols; }
// Threads of a strip's block: a grid narrower than one strip has no columns for the last warps, whose
// registers would only keep other strips off the SM.  us per step with 128 threads and with these: 12x60000
// split 94.6 / 45.9, 12x200000 hybrid 273.8 / 115.2, 40x50000 split 118.1 / 80.9 and with a free surface
// 123.0 / 83.9, 60x20000 hybrid 43.9 / 33.5.
inline int stripThreads(const Grid2D& g) { return g.NX < kThreads ? (g.NX + 31) / 32 * 32 : kThreads; }
__host__ __device__ __forceinline__ int stressStrips(const Grid2D& g, int scheme, int rows) {
    return (g.NZ - 4 - (scheme == kFree ? g.fs : 4) + rows - 1) / rows;
}
__host__ __device__ __forceinline__ int velocityStrips(const Grid2D& g, int rows) { return (g.NZ - 8 + rows - 1) / rows; }
// Place of a block among the strips down the grid.  They are numbered along y and go on along z: a
// grid of a few columns can have more strips than the 65,535 blocks that y takes.
__device__ __forceinline__ int stripRow() { return int(blockIdx.z * gridDim.y + blockIdx.y); }

// ---- stress ----------------------------------------------------------------------------

// Whether a strip of R rows has cells in the hybrid scheme's layer.  Strips without them run a body
// without its halves, damping and tests.  With the shared offsets (Rows), at three rows: 1601x1203
// cells with a 30-cell layer 44.8 -> 38.5 us a step, where the instructions issued (270 a cell, 0.7
// of the issue slots) were the bound; split halves there 71.1 -> 64.0 by the offsets alone.
template <int R> __device__ __forceinline__ bool touchesLayer(const Grid2D& g, int row, int bx) {
    const int first = bx * kCols + kHalo;
    return inPml(g, row, first) || inPml(g, row + R - 1, min(first + kCols, g.NX) - 1);
}

template <int R, bool kLayer>
__device__ __forceinline__ void hybridStressStrip(const Grid2D& g, const Fields2D& f, const Control2D& c, int step, bool pendingOk,
                                                  int row, int j, Shared* sh) {
    const int tid = threadIdx.x;
    const bool inside = j < g.NX;
    const bool own = tid >= kHalo && tid < kThreads - kHalo && j < g.NX - 4;
    const Rows<R> rows(g, row, j);
    // vx forward in x and z, vz backward in both.
    Column<R> vx, vz;
    float muZ[R], l2mX[R], lambdaX[R], sxz[R], sxx[R], szz[R], half[R][6];
    Damping<R> d;
    if (own) {
        const float* const halves[6] = {f.sxz1, f.sxz2, f.sxx1, f.szz1, f.sxx2, f.szz2};
        if (kLayer) d.load(g, f, row, j);
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (kLayer && inPml(g, row + r, j))
#pragma unroll
                for (int h = 0; h < 6; ++h) half[r][h] = __ldcg(halves[h] + rows.own(r));
        vx.load(f.vx, rows, 3);
        vz.load(f.vz, rows, 4);
        loadRows(muZ, f.muZ, rows);
        loadRows(l2mX, f.l2mX, rows);
        loadRows(lambdaX, f.lambdaX, rows);
        loadRows(sxz, f.sxz, rows);
        loadRows(sxx, f.sxx, rows);
        loadRows(szz, f.szz, rows);
    } else if (inside) {
        vx.loadOwn(f.vx, rows, 3);
        vz.loadOwn(f.vz, rows, 4);
    }
    if (inside) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            sh[2 * r][tid] = vx.v[r + 3];
            sh[2 * r + 1][tid] = vz.v[r + 4];
        }
    }
    __syncthreads();
    if (!own) return;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int i = row + r;
        if (i >= g.NZ - 4) break;
        const unsigned k = rows.own(r);
        const float dvz_dx = dxBackward(g, &sh[2 * r + 1][tid]);
        const float dvx_dz = dzAt(g, vx, r);
        const float dvx_dx = dxForward(g, &sh[2 * r][tid]);
        const float dvz_dz = dzAt(g, vz, r);
        const bool pml = kLayer && inPml(g, i, j);
        float w = 0.0f;
        if (!pml && pendingOk && int(k) == c.srcIdx && stressSource(c, step - 1, w)) {
            if (c.srcType == SEIS2D_EXPLOSIVE) { sxx[r] = __fadd_rn(sxx[r], w); szz[r] = __fadd_rn(szz[r], w); }
            else sxz[r] = __fadd_rn(sxz[r], w);
        }
        hybridStress(g, pml, d.at(r, false), muZ[r], l2mX[r], lambdaX[r], dvz_dx, dvx_dz, dvx_dx, dvz_dz, sxz[r], sxx[r],
                     szz[r], half[r]);
        if (pml) {
            f.sxz1[k] = half[r][0]; f.sxz2[k] = half[r][1]; f.sxx1[k] = half[r][2];
            f.szz1[k] = half[r][3]; f.sxx2[k] = half[r][4]; f.szz2[k] = half[r][5];
        }
        f.sxz[k] = sxz[r]; f.sxx[k] = sxx[r]; f.szz[k] = szz[r];
    }
}

// Stress update of strip (bx, by) at `step`, all three schemes (Cuda_Check.cu:224-266, 315-364,
// 416-487) with the free-surface mirror of :491-508 written by the owners of the mirrored rows;
// `pendingOk` allows folding in the stress-type source of step-1 (false for the first step of
// a batch, whose source the batch end applied).  All threads of the block call it.
template <int S, int R>
__device__ __forceinline__ void stressStrip(const Grid2D& g, const Fields2D& f, const Control2D& c, int step, bool pendingOk,
                                            int bx, int by, Shared* sh) {
    const int tid = threadIdx.x, j = bx * kCols + tid;
    const int row = (S == kFree ? g.fs : 4) + by * R;
    const bool inside = j < g.NX;
    const bool own = tid >= kHalo && tid < kThreads - kHalo && j < g.NX - 4;   // j >= 4 by tid >= kHalo
    const Rows<R> rows(g, row, j);

    if constexpr (S == kHybrid) {
        if (touchesLayer<R>(g, row, bx)) hybridStressStrip<R, true>(g, f, c, step, pendingOk, row, j, sh);
        else hybridStressStrip<R, false>(g, f, c, step, pendingOk, row, j, sh);
        return;
    }

    SplitColumn<R> vx, vz;
    float t[R][6];   // sxx1, sxx2, szz1, szz2, sxz1, sxz2
    float mu[R + 1], l2m[R], l2mRight[R], lambda[R], lambdaRight[R];
    Damping<R> d;
    if (own) {
        d.load(g, f, row, j);
        vx.a.load(f.vx1, rows, 3);
        vx.b.load(f.vx2, rows, 3);
        vz.a.load(f.vz1, rows, 4);
        vz.b.load(f.vz2, rows, 4);
        const float* const stresses[6] = {f.sxx1, f.sxx2, f.szz1, f.szz2, f.sxz1, f.sxz2};
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int h = 0; h < 6; ++h) t[r][h] = __ldcg(stresses[h] + rows.own(r));
        loadRows(l2m, f.l2m, rows);
        loadRows(l2mRight, f.l2m + 1, rows);
        loadRows(lambda, f.lambda, rows);
        loadRows(lambdaRight, f.lambda + 1, rows);
#pragma unroll
        for (int r = 0; r <= R; ++r) mu[r] = __ldcg(f.mu + rows.own(r));
    } else if (inside) {
        vx.a.loadOwn(f.vx1, rows, 3);
        vx.b.loadOwn(f.vx2, rows, 3);
        vz.a.loadOwn(f.vz1, rows, 4);
        vz.b.loadOwn(f.vz2, rows, 4);
    }
    if (inside) {
        vx.sum();
        vz.sum();
#pragma unroll
        for (int r = 0; r < R; ++r) {
            sh[6 * r][tid] = vx.a.v[r + 3]; sh[6 * r + 1][tid] = vx.b.v[r + 3]; sh[6 * r + 2][tid] = vx.s[r + 3];
            sh[6 * r + 3][tid] = vz.a.v[r + 4]; sh[6 * r + 4][tid] = vz.b.v[r + 4]; sh[6 * r + 5][tid] = vz.s[r + 4];
        }
    }
    __syncthreads();
    if (!own) return;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int i = row + r;
        if (i >= g.NZ - 4) break;
        const unsigned k = rows.own(r);
        const SplitRow rvx{&sh[6 * r][tid], &sh[6 * r + 1][tid], &sh[6 * r + 2][tid]};
        const SplitRow rvz{&sh[6 * r + 3][tid], &sh[6 * r + 4][tid], &sh[6 * r + 5][tid]};
        const Damp damp = d.at(r, S == kFree && i <= g.fs + 5);
        float w = 0.0f;
        if (pendingOk && int(k) == c.srcIdx && stressSource(c, step - 1, w)) addSplitSource(c, w, t[r]);
        const float muAvg = 0.5f * (mu[r] + mu[r + 1]);
        const float dvx_dx = dxForward(g, rvx);
        if (S == kFree && r == 0 && i == g.fs) {
            freeRowStress(g, damp, muAvg, f.dp[j], dvx_dx, weigh2(g, rvz.tap(0, -1), rvz.tap(1, -2)),
                          weigh2(g, vx.tap(r + 4, r + 3), vx.tap(r + 5, r + 2)), t[r]);
        } else {
            splitStress(g, damp, muAvg, 0.5f * (l2m[r] + l2mRight[r]), 0.5f * (lambda[r] + lambdaRight[r]), dvx_dx, vz.dz(g, r),
                        dxBackward(g, rvz), vx.dz(g, r), t[r]);
        }
        f.sxx1[k] = t[r][0]; f.sxx2[k] = t[r][1]; f.szz1[k] = t[r][2];
        f.szz2[k] = t[r][3]; f.sxz1[k] = t[r][4]; f.sxz2[k] = t[r][5];
        if (S == kFree) {
            // Odd images above the free surface (Cuda_Check.cu:491-508): szz of row fs+l into
            // row fs-l, sxz of row fs+l-1 into row fs-l, l = 1..4.
            const int l = i - g.fs;
            if (l >= 1 && l <= 4) {
                const int above = (g.fs - l) * g.NX + j;
                f.szz1[above] = -t[r][2]; f.szz2[above] = -t[r][3];
            }
            if (l <= 3) {
                const int above = (g.fs - l - 1) * g.NX + j;
                f.sxz1[above] = -t[r][4]; f.sxz2[above] = -t[r][5];
            }
        }
    }
}

// kTall: the strips go on along gridDim.z (stripRow).  Grids that do not need that have kernels without it: with
// it in theirs, 1601x1203 cells in the hybrid scheme took 36.5 us a step instead of 35.8 and 250x300 5.9
// instead of 5.7.
template <int S, int R, bool kTall>
__global__ void __launch_bounds__(kThreads) stressStep(Grid2D g, Fields2D f, const Control2D* __restrict__ ctl, int slot) {
    __shared__ Shared sh[kSharedArrays<S> * R];
    waitForPrevious();
    const Control2D c = *ctl;
    const int step = c.base + slot;
    const bool receivers = kTall ? stripRow() >= stressStrips(g, S, R) : blockIdx.y == gridDim.y - 1;
    if (receivers) {
        // Receiver row: the velocities of step-1 are final while the stresses update.
        if (slot > 0 && (!kTall || stripRow() == stressStrips(g, S, R)))
            recordStep<S>(g, f, c, step - 1, blockIdx.x * blockDim.x + threadIdx.x, blockDim.x * gridDim.x);
        return;
    }
    stressStrip<S, R>(g, f, c, step, slot > 0, blockIdx.x, kTall ? stripRow() : blockIdx.y, sh);
    launchDependents();
}

// ---- velocity --------------------------------------------------------------------------

// Force-type point source of `step` added by the owner of the source cell after its update
// (applyPointSource types 0, 1, 4, Cuda_Check.cu:578-600, 622-633).
template <int S>
__device__ __forceinline__ void forceSource(const Grid2D& g, const Fields2D& f, const Control2D& c, int step, int k,
                                            float& vxOut, float& vzOut) {
    if (!c.srcSingle || !c.srcValid || k != c.srcIdx || step < 0 || step >= c.srcLength) return;
    if (c.srcType != SEIS2D_VERTICAL_FORCE && c.srcType != SEIS2D_HORIZONTAL_FORCE && c.srcType != SEIS2D_ROTATED_FORCE)
        return;
    const float w = c.series[step];
    if (!isfinite(w)) return;
    float force_x = w, force_z = w;
    if (c.srcType == SEIS2D_ROTATED_FORCE) {
        // M_PI is a double in the host headers the reference compiles against.
        force_x = sinf(c.srcAngle * 3.14159265358979323846 / 180.0f) * w;
        force_z = cosf(c.srcAngle * 3.14159265358979323846 / 180.0f) * w;
    }
    // The reference adds the force in a separate kernel after the update has been stored, so
    // the sum is rounded on its own: __fadd_rn keeps it from being fused into the update.
    if (S == kHybrid) {
        if (c.srcType != SEIS2D_VERTICAL_FORCE) vxOut = __fadd_rn(vxOut, force_x * g.dt / f.rhoOrig[k]);
        if (c.srcType != SEIS2D_HORIZONTAL_FORCE) vzOut = __fadd_rn(vzOut, force_z * g.dt / f.rhoXZ[k]);
    } else {
        if (c.srcType != SEIS2D_VERTICAL_FORCE) vxOut = __fadd_rn(vxOut, force_x * g.dt / f.rho[k]);
        if (c.srcType != SEIS2D_HORIZONTAL_FORCE) {
            const float rho_avg = 0.25f * (f.rho[k] + f.rho[k + 1] + f.rho[k + g.NX] + f.rho[k + g.NX + 1]);
            vzOut = __fadd_rn(vzOut, force_z * g.dt / rho_avg);
        }
    }
}

// The outer ring of velocities that zeroBoundaryKernel clears (Cuda_Check.cu:643-667): the first and
// last column along the strip's rows, and with the first and last strip the rows beyond them.
template <int S, int R> __device__ __forceinline__ void clearRing(const Grid2D& g, const Fields2D& f, int row, int j, bool last) {
    if (j >= g.NX) return;
    auto clear = [&](int i) {
        const int k = i * g.NX + j;
        if (S == kHybrid) { f.vx[k] = 0.0f; f.vz[k] = 0.0f; }
        else { f.vx1[k] = 0.0f; f.vx2[k] = 0.0f; f.vz1[k] = 0.0f; f.vz2[k] = 0.0f; }
    };
    const bool edge = j == 0 || j == g.NX - 1;
    const int from = row == 4 ? 0 : row, to = last ? g.NZ : row + R;
    if (edge)
        for (int i = from; i < to; ++i) clear(i);
    else {
        if (row == 4) clear(0);
        if (last) clear(g.NZ - 1);
    }
}

template <int R, bool kLayer>
__device__ __forceinline__ void hybridVelocityStrip(const Grid2D& g, const Fields2D& f, const Control2D& c, int step, int row,
                                                    int j, bool lastStrip, Shared* sh) {
    const int tid = threadIdx.x;
    const bool inside = j < g.NX;
    const bool own = tid >= kHalo && tid < kThreads - kHalo && j < g.NX - 4;
    const Rows<R> rows(g, row, j);
    // sxx backward in x, szz forward in z, sxz forward in x and backward in z.
    Column<R> szz, sxz;
    float sxx[R], vx[R], vz[R], rhoXZ[R], rho[R], half[R][4];
    Damping<R> d;
    if (own) {
        const float* const halves[4] = {f.vz1, f.vz2, f.vx1, f.vx2};
        if (kLayer) d.load(g, f, row, j);
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (kLayer && inPml(g, row + r, j))
#pragma unroll
                for (int h = 0; h < 4; ++h) half[r][h] = __ldcg(halves[h] + rows.own(r));
        szz.load(f.szz, rows, 3);
        sxz.load(f.sxz, rows, 4);
        loadRows(vx, f.vx, rows);
        loadRows(vz, f.vz, rows);
        loadRows(rhoXZ, f.rhoXZ, rows);
        loadRows(rho, f.rhoOrig, rows);
    } else if (inside) {
        sxz.loadOwn(f.sxz, rows, 4);
    }
    if (inside) {
        loadRows(sxx, f.sxx, rows);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            sh[2 * r][tid] = sxx[r];
            sh[2 * r + 1][tid] = sxz.v[r + 4];
        }
    }
    __syncthreads();
    clearRing<kHybrid, R>(g, f, row, j, lastStrip);
    if (!own) return;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int i = row + r;
        if (i >= g.NZ - 4) break;
        const unsigned k = rows.own(r);
        const float dsigxz_dx = dxForward(g, &sh[2 * r + 1][tid]);
        const float dsigzz_dz = dzAt(g, szz, r);
        const float dsigxx_dx = dxBackward(g, &sh[2 * r][tid]);
        const float dsigxz_dz = dzAt(g, sxz, r);
        const bool pml = kLayer && inPml(g, i, j);
        hybridVelocity(g, pml, d.at(r, false), rhoXZ[r], rho[r], dsigxz_dx, dsigzz_dz, dsigxx_dx, dsigxz_dz, vx[r], vz[r],
                       half[r]);
        if (pml) { f.vz1[k] = half[r][0]; f.vz2[k] = half[r][1]; f.vx1[k] = half[r][2]; f.vx2[k] = half[r][3]; }
        forceSource<kHybrid>(g, f, c, step, k, vx[r], vz[r]);
        f.vx[k] = vx[r]; f.vz[k] = vz[r];
    }
}

// Velocity update of strip (bx, by), all three schemes (Cuda_Check.cu:270-311, 368-412, 512-563);
// rows start at 4, so that the free surface's air rows are cleared too.
template <int S, int R>
__device__ __forceinline__ void velocityStrip(const Grid2D& g, const Fields2D& f, const Control2D& c, int step, int bx, int by,
                                              bool lastStrip, Shared* sh) {
    const int tid = threadIdx.x, j = bx * kCols + tid;
    const int row = 4 + by * R;
    const bool inside = j < g.NX;
    const bool own = tid >= kHalo && tid < kThreads - kHalo && j < g.NX - 4;
    const Rows<R> rows(g, row, j);

    if constexpr (S == kHybrid) {
        if (touchesLayer<R>(g, row, bx)) hybridVelocityStrip<R, true>(g, f, c, step, row, j, lastStrip, sh);
        else hybridVelocityStrip<R, false>(g, f, c, step, row, j, lastStrip, sh);
        return;
    }

    SplitColumn<R> szz, sxz;
    float sxx1[R], sxx2[R], v[R][4];   // vx1, vx2, vz1, vz2
    float rho[R + 1], rhoRight[R + 1];
    Damping<R> d;
    if (own) {
        d.load(g, f, row, j);
        szz.a.load(f.szz1, rows, 3);
        szz.b.load(f.szz2, rows, 3);
        sxz.a.load(f.sxz1, rows, 4);
        sxz.b.load(f.sxz2, rows, 4);
        const float* const velocities[4] = {f.vx1, f.vx2, f.vz1, f.vz2};
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int h = 0; h < 4; ++h) v[r][h] = __ldcg(velocities[h] + rows.own(r));
#pragma unroll
        for (int r = 0; r <= R; ++r) {
            rho[r] = __ldcg(f.rho + rows.own(r));
            rhoRight[r] = __ldcg(f.rho + 1 + rows.own(r));
        }
    } else if (inside) {
        sxz.a.loadOwn(f.sxz1, rows, 4);
        sxz.b.loadOwn(f.sxz2, rows, 4);
    }
    if (inside) {
        loadRows(sxx1, f.sxx1, rows);
        loadRows(sxx2, f.sxx2, rows);
        szz.sum();
        sxz.sum();
#pragma unroll
        for (int r = 0; r < R; ++r) {
            sh[6 * r][tid] = sxx1[r]; sh[6 * r + 1][tid] = sxx2[r]; sh[6 * r + 2][tid] = sxx1[r] + sxx2[r];
            sh[6 * r + 3][tid] = sxz.a.v[r + 4]; sh[6 * r + 4][tid] = sxz.b.v[r + 4]; sh[6 * r + 5][tid] = sxz.s[r + 4];
        }
    }
    __syncthreads();
    clearRing<S, R>(g, f, row, j, lastStrip);
    if (!own) return;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int i = row + r;
        if (i >= g.NZ - 4) break;
        const unsigned k = rows.own(r);
        if (S == kFree && i < g.fs) {
            f.vx1[k] = 0.0f; f.vx2[k] = 0.0f; f.vz1[k] = 0.0f; f.vz2[k] = 0.0f;
            continue;
        }
        const SplitRow rxx{&sh[6 * r][tid], &sh[6 * r + 1][tid], &sh[6 * r + 2][tid]};
        const SplitRow rxz{&sh[6 * r + 3][tid], &sh[6 * r + 4][tid], &sh[6 * r + 5][tid]};
        const float rhoMean = 0.25f * (rho[r] + rhoRight[r] + rho[r + 1] + rhoRight[r + 1]);
        splitVelocity(g, d.at(r, S == kFree && i <= g.fs + 5), rho[r], rhoMean, dxBackward(g, rxx), sxz.dz(g, r),
                      dxForward(g, rxz), szz.dz(g, r), v[r]);
        forceSource<S>(g, f, c, step, k, v[r][0], v[r][2]);
        f.vx1[k] = v[r][0]; f.vx2[k] = v[r][1]; f.vz1[k] = v[r][2]; f.vz2[k] = v[r][3];
    }
}

template <int S, int R, bool kTall>
__global__ void __launch_bounds__(kThreads) velocityStep(Grid2D g, Fields2D f, const Control2D* __restrict__ ctl, int slot) {
    __shared__ Shared sh[kSharedArrays<S> * R];
    waitForPrevious();
    if (kTall && stripRow() >= velocityStrips(g, R)) return;
    const Control2D c = *ctl;
    const bool last = kTall ? stripRow() == velocityStrips(g, R) - 1 : blockIdx.y == gridDim.y - 1;
    velocityStrip<S, R>(g, f, c, c.base + slot, blockIdx.x, kTall ? stripRow() : blockIdx.y, last, sh);
    launchDependents();
}

// ---- multi-source injection (injectMultipleSourcesKernel, Cuda_Check.cu:822-834) ---------

// Adds one source value through the field the reference's applyPointSource picks
// (Cuda_Check.cu:567-634), with atomics because sources may overlap.
template <int S>
__device__ void applySource(const Grid2D& g, const Fields2D& f, int type, float angle, float w, int idx) {
    if (idx < 0 || idx >= g.total || !isfinite(w)) return;
    const int x = idx % g.NX, z = idx / g.NX;
    if (x < 4 || x >= g.NX - 4 || z < 4 || z >= g.NZ - 4 || (S == kFree && z <= g.fs)) return;
    if (type == SEIS2D_VERTICAL_FORCE || type == SEIS2D_HORIZONTAL_FORCE || type == SEIS2D_ROTATED_FORCE) {
        float force_x = w, force_z = w;
        if (type == SEIS2D_ROTATED_FORCE) {
            force_x = sinf(angle * 3.14159265358979323846 / 180.0f) * w;
            force_z = cosf(angle * 3.14159265358979323846 / 180.0f) * w;
        }
        if (S == kHybrid) {
            if (type != SEIS2D_VERTICAL_FORCE) atomicAdd(&f.vx[idx], force_x * g.dt / f.rhoOrig[idx]);
            if (type != SEIS2D_HORIZONTAL_FORCE) atomicAdd(&f.vz[idx], force_z * g.dt / f.rhoXZ[idx]);
        } else {
            if (type != SEIS2D_VERTICAL_FORCE) atomicAdd(&f.vx1[idx], force_x * g.dt / f.rho[idx]);
            if (type != SEIS2D_HORIZONTAL_FORCE) {
                const float rho_avg = 0.25f * (f.rho[idx] + f.rho[idx + 1] + f.rho[idx + g.NX] + f.rho[idx + g.NX + 1]);
                atomicAdd(&f.vz1[idx], force_z * g.dt / rho_avg);
            }
        }
    } else if (type == SEIS2D_EXPLOSIVE) {
        if (S == kHybrid) { atomicAdd(&f.sxx[idx], w); atomicAdd(&f.szz[idx], w); }
        else {
            atomicAdd(&f.sxx1[idx], w * 0.5f); atomicAdd(&f.sxx2[idx], w * 0.5f);
            atomicAdd(&f.szz1[idx], w * 0.5f); atomicAdd(&f.szz2[idx], w * 0.5f);
        }
    } else if (type == SEIS2D_SHEAR) {
        if (S == kHybrid) atomicAdd(&f.sxz[idx], w);
        else { atomicAdd(&f.sxz1[idx], w * 0.5f); atomicAdd(&f.sxz2[idx], w * 0.5f); }
    }
}

// Index written over an active source that has expired during an advancing run.
constexpr int kDroppedSource = INT32_MIN;

// One thread per active source.  With multiAdvance the source time moves by dt first and a
// source past 2.5 / f_peak is dropped, as the reference host loop does before each step
// (src/Seis2D/Workflow2D.inc:300-312); host arithmetic there, so the expiry test uses a
// correctly rounded division.
template <int S>
__global__ void injectSources(Grid2D g, Fields2D f, const Control2D* __restrict__ ctl) {
    const Control2D c = *ctl;
    const int r = threadIdx.x;
    if (r >= c.multiCount) return;
    seis2d_source src = c.sources[r];
    if (c.multiAdvance) {
        if (src.idx == kDroppedSource) return;  // expired earlier
        src.t = src.t + g.dt;
        c.sources[r].t = src.t;
        const float t_peak_host = __fdiv_rn(1.0f, src.f_peak);
        if (src.t > 2.5f * t_peak_host) { c.sources[r].idx = kDroppedSource; return; }
    }
    if (!isfinite(src.f_peak) || src.f_peak <= 0.0f || !isfinite(src.t)) return;
    const float t_peak = 1.0f / src.f_peak;
    const float x = 3.14159265358979323846 * src.f_peak * (src.t - t_peak);
    const float val = src.amp * (1.0f - 2.0f * x * x) * expf(-x * x);
    applySource<S>(g, f, c.srcType, c.srcAngle, val * SEIS2D_SOURCE_INJECTION_SCALE, src.idx);
}

// ---- batch boundaries ------------------------------------------------------------------

// State of the persistent runs (seis2d_resident.cuh).
struct GridSync {
    unsigned failed;    // a wait of a run gave up and no synchronising call has said so yet
    unsigned first;     // number of the exchange before the run's first
    unsigned last;      // number of the run's last exchange
    unsigned pad;
};

// Prepares the steps that follow in the stream.  A persistent run's exchanges are numbered here
// and not by the host, so that a replay of a captured run has numbers of its own too.  The failure of an
// earlier run stays until the host has read it: cleared here, a run enqueued before the next
// synchronising call would hide it and go on from the broken state.
__global__ void configureRun(Control2D* ctl, Control2D value, GridSync* gs, unsigned exchanges) {
    *ctl = value;
    if (exchanges) *gs = GridSync{gs->failed, gs->last, gs->last + exchanges, 0};
}

// Completes the last step of a batch: its stress-type point source and its receivers, then
// advances the clock by the batch length.
template <int S>
__device__ void finishStep(const Grid2D& g, const Fields2D& f, const Control2D& c, int step, int tid, int nthreads) {
    recordStep<S>(g, f, c, step, tid, nthreads);
    if (tid == 0) {
        float w;
        if (stressSource(c, step, w)) {
            const int k = c.srcIdx;
            if (S == kHybrid) {
                if (c.srcType == SEIS2D_EXPLOSIVE) { f.sxx[k] += w; f.szz[k] += w; }
                else f.sxz[k] += w;
            } else if (c.srcType == SEIS2D_EXPLOSIVE) {
                f.sxx1[k] += w * 0.5f; f.sxx2[k] += w * 0.5f; f.szz1[k] += w * 0.5f; f.szz2[k] += w * 0.5f;
            } else {
                f.sxz1[k] += w * 0.5f; f.sxz2[k] += w * 0.5f;
            }
        }
    }
}

template <int S>
__global__ void finishBatch(Grid2D g, Fields2D f, Control2D* ctl, int slot, int batch) {
    const Control2D c = *ctl;
    finishStep<S>(g, f, c, c.base + slot, threadIdx.x, blockDim.x);
    __syncthreads();
    if (threadIdx.x == 0) ctl->base = c.base + batch;
}

// ---- waits of a persistent run --------------------------------------------------------------

// Default bound of one wait in SM clock cycles (about two seconds): the launch is cooperative,
// so every block is resident and a normal wait ends in microseconds.
constexpr long long kBarrierCycles = 4000000000LL;

// Bound of the waits and the withheld-block test hook of one persistent run.
struct BarrierLimits {
    long long cycles;     // bound of every wait
    int withheldBlock;    // test hook: this block sends nothing in its first exchange; -1 in use
};

// recordReceiverStepOnGpu / copyReceiverRecordsFromGpu sample (Cuda_Check.cu:793-818).
template <int S>
__global__ void extractReceivers(Grid2D g, Fields2D f, const int* __restrict__ idx, int count, float* outVx, float* outVz) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= count) return;
    float vx, vz;
    sampleReceiver<S>(g, f, idx[r], vx, vz);
    outVx[r] = vx;
    outVz[r] = vz;
}

// generateColorMapKernel (Cuda_Check.cu:700-790) behind generateWavefieldTextureOnGpu
// (:1136-1141): one RGBA pixel per grid cell, red for positive and blue for negative values of
// the selected component times scale and the component's balance factor.  `split` selects the
// split-field halves (flag_type 1 and 3) or the total fields (flag_type 2); any other scheme id
// reads the totals and shows no stress, as the reference's branches do.  The expressions keep
// the reference's operand order and its float-to-byte truncations.
struct ColorFields {
    const float *vx1, *vx2, *vz1, *vz2, *sxx1, *sxx2, *szz1, *szz2, *sxz1, *sxz2;
    const float *vx, *vz, *sxx, *szz, *sxz;
    const float *mu, *l2m;
};

__device__ __forceinline__ float colorVx(const ColorFields& f, int NX, int NZ, bool split, int i, int j) {
    const int r = i < 0 ? 0 : (i > NZ - 1 ? NZ - 1 : i);
    const int c = j < 0 ? 0 : (j > NX - 1 ? NX - 1 : j);
    const int k = r * NX + c;
    return split ? f.vx1[k] + f.vx2[k] : f.vx[k];
}

__device__ __forceinline__ float colorVz(const ColorFields& f, int NX, int NZ, bool split, int i, int j) {
    const int r = i < 0 ? 0 : (i > NZ - 1 ? NZ - 1 : i);
    const int c = j < 0 ? 0 : (j > NX - 1 ? NX - 1 : j);
    const int k = r * NX + c;
    return split ? f.vz1[k] + f.vz2[k] : f.vz[k];
}

__global__ void __launch_bounds__(256) colorMap(ColorFields f, int NX, int NZ, int flag, uchar4* out, float scale,
                                                int component) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= NZ || j >= NX) return;
    const int k = i * NX + j;
    const bool split = flag == 1 || flag == 3;
    float val = 0.0f, balance = 1.0f;
    if (component == 0) {
        const float vx = colorVx(f, NX, NZ, split, i, j), vz = colorVz(f, NX, NZ, split, i, j);
        val = sqrtf(vx * vx + vz * vz);
    } else if (component == 1) {
        val = colorVx(f, NX, NZ, split, i, j);
    } else if (component == 2) {
        val = colorVz(f, NX, NZ, split, i, j);
    } else if (component == 3) {
        // Normal stress scaled to a strain by lambda + 2 mu.
        float stress = 0.0f;
        if (split) stress = f.sxx1[k] + f.sxx2[k] + f.szz1[k] + f.szz2[k];
        else if (flag == 2) stress = f.sxx[k] + f.szz[k];
        const float l2m = f.l2m[k];
        val = l2m > 1000.0f ? stress / l2m : stress;
        val *= 1000;
        balance = 2.0f;
    } else if (component == 4) {
        // Shear stress scaled by mu.
        float shear = 0.0f;
        if (split) shear = f.sxz1[k] + f.sxz2[k];
        else if (flag == 2) shear = f.sxz[k];
        const float mu = f.mu[k];
        val = mu > 1000.0f ? shear / mu : shear;
        val *= 1000;
        balance = 3.0f;
    } else if (component == 5) {
        // Divergence (P waves).
        const float dvxdx = colorVx(f, NX, NZ, split, i, j) - colorVx(f, NX, NZ, split, i, j - 1);
        const float dvzdz = colorVz(f, NX, NZ, split, i, j) - colorVz(f, NX, NZ, split, i - 1, j);
        val = dvxdx + dvzdz;
        balance = 8.0f;
    } else if (component == 6) {
        // Curl (S waves).
        const float dvzdx = colorVz(f, NX, NZ, split, i, j) - colorVz(f, NX, NZ, split, i, j - 1);
        const float dvxdz = colorVx(f, NX, NZ, split, i, j) - colorVx(f, NX, NZ, split, i - 1, j);
        val = dvzdx - dvxdz;
        balance = 8.0f;
    }
    float norm = val * scale * balance;
    if (norm > 1.0f) norm = 1.0f;
    if (norm < -1.0f) norm = -1.0f;
    unsigned char r = 255, g = 255, b = 255;
    if (norm > 0.0f) {
        g = static_cast<unsigned char>(255.0f * (1.0f - norm));
        b = static_cast<unsigned char>(255.0f * (1.0f - norm));
    } else {
        r = static_cast<unsigned char>(255.0f * (1.0f + norm));
        g = static_cast<unsigned char>(255.0f * (1.0f + norm));
    }
    out[k] = make_uchar4(r, g, b, 255);
}

}  // namespace seis2d
