// seis3d_tma.cuh - Tensor Memory Accelerator staging for the z-marching passes (sm_100a).
//
// Each CTA streams the planes of its column tile through a ring of kStages shared-memory
// stages.  One elected thread fills a stage with cp.async.bulk.tensor tile copies whose
// completion is tracked by the stage's mbarrier (expect-tx bytes); every thread waits on
// that mbarrier before reading the stage.  Waits are bounded: a stage that does not
// arrive within the session's wait limit (~2 s of SM clock by default) sets a stall flag
// that the host reports, and the CTA drains its in-flight copies (again bounded) and
// exits.  No cluster multicast is used.
#pragma once

#include <cuda.h>
#include <cstdint>

namespace seis3d {
namespace tma {

constexpr int kStages = 3;

constexpr long long kWaitCycles = 4000000000LL;   // default wait limit, ~2 s at 1.9 GHz

// Tensor-map table, kept in global memory.  The twelve volumes of a session are equally spaced in
// one allocation, so a four-dimensional map {x, y, z, volume} brings the tiles of several
// fields (and, with a box two planes deep, of two planes) in one copy: 7 and 6 copies per stage
// instead of 13 and 15, which the one issuing thread has to get out between two planes.
enum MapIndex : int {
    kSxxSxz = 0,         // sigma_xx and sigma_xz, (32+8) x TY (x halo)
    kSxy = 1,            // sigma_xy, (32+8) x (TY+8)
    kSyySyz = 2,         // sigma_yy and sigma_yz, 32 x (TY+8)
    kRhoTwo = 3,         // 1/rho, 36 x (TY+1) x 2 planes
    kVelocity = 4,       // vx, vy, vz, 32 x TY
    kSyzSxzCentre = 5,   // sigma_yz and sigma_xz, 32 x TY
    kSzzCentre = 6,      // sigma_zz, 32 x TY
    kVelocityHalo = 7,   // vx, vy, vz, (32+8) x (TY+8)
    kMuTwo = 8,          // mu, 36 x (TY+1) x 2 planes
    kLambda = 9,         // lambda, 32 x TY
    kStress = 10,        // the six stresses, 32 x TY
    kVxVyCentre = 11,    // vx and vy, 32 x TY
    kVzCentre = 12,      // vz, 32 x TY
    kMapCount = 13
};

__device__ __forceinline__ uint32_t smemAddress(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void barrierInit(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smemAddress(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void barrierInitFence() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void arriveExpectTx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smemAddress(bar)), "r"(bytes)
                 : "memory");
}

// Test the phase; if it is incomplete the thread may be suspended for a short,
// system-defined time before the instruction returns.  (A long explicit suspend-time hint
// measured 30 % slower on B200: suspended warps resume late after the phase completes.)
__device__ __forceinline__ bool tryWait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smemAddress(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Wait of at most `limit` SM cycles on one stage; returns false when it timed out.
__device__ __forceinline__ bool waitStage(uint64_t* bar, uint32_t parity, long long limit) {
    if (tryWait(bar, parity)) return true;
    const long long start = clock64();
    while (!tryWait(bar, parity))
        if (clock64() - start > limit) return false;
    return true;
}

// Programmatic dependent launch: the next kernel of the stream may become resident as soon as
// every CTA has called launchDependents, and waits in waitForPrevious until this one has
// completed and its writes are visible.  Both are no-ops in an ordinary launch.  A CTA calls
// the first after its last plane: with the call at its start, the next pass's CTAs sat waiting
// in the slots beside it, and the 40x32x36 step took 33.9 us instead of 28.6 (30.8 without
// programmatic launch).
__device__ __forceinline__ void launchDependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void waitForPrevious() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Order this thread's earlier generic-proxy shared-memory accesses before its later
// async-proxy (TMA) accesses.
__device__ __forceinline__ void fenceProxyAsync() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// One tile copy global -> shared from {x, y, z, first volume of the map}, completing on `bar`.
__device__ __forceinline__ void load4d(void* dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
        ::"r"(smemAddress(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(0), "r"(smemAddress(bar))
        : "memory");
}

}  // namespace tma
}  // namespace seis3d
