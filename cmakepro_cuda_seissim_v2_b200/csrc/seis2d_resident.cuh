// seis2d_resident.cuh - many steps of the 2-D solver in one cooperative launch, the whole state
// on the chip.
//
// The grid is cut into at most one tile per SM.  The stresses and velocities of a tile stand in its
// CTA's shared memory with a 4-cell halo for the whole run; materials, damping and the hybrid
// layer's halves stand in the registers of the threads that own the cells (R rows of one column
// each).  So a step moves nothing through L2 but the halos.  Neighbours exchange those twice a
// step, after the velocities and after the stresses, through mailboxes in global memory: 16-byte
// words of two values and the exchange's number, each written and read by one access, so a word
// that carries the number is complete and no flag, fence or grid barrier is needed.  A mailbox
// word is rewritten only after its reader has sent the words that the writer waited for in
// between.
//
// What bounds it: with one row per thread mostly the exchange (a store, its visibility in L2 and the
// load that sees it, twice a step), with more rows the instructions of the cells: hybrid tiles of
// 1 / 2 / 3 rows take 2.7 / 3.9 / 5.9 us a step, split ones 3.1 / 6.0 / 7.7.  us per
// step, graph replay of the step kernels against this: split 120x100 4.1/3.1, 300x240 5.8/5.2,
// 440x420 7.5/7.7; free surface 97x93 3.9/3.2, 250x300 6.0/5.1, 440x420 7.9/8.1; hybrid 128x250
// 3.9/2.7, 250x300 5.2/3.9, 440x420 7.4/6.0.  Two grid barriers per step and the state in L2 took
// 6.4 to 21 us.
//
// All waits are bounded (BarrierLimits): a CTA that gives up sets the failure flag, which the
// others see in their own waits, and every CTA leaves the run.  The flag stands until a
// synchronising call has reported it, and runs that find it set do nothing.
#pragma once

#include "seis2d_kernels.cuh"

namespace seis2d {

constexpr int kResidentThreads = 512;      // most threads of a tile
// Shared-memory arrays of one fixed shape, so that a thread addresses its cells in all of them, and
// the rows around them, by constant offsets from one register (with the shape in registers a
// cell took 807 instructions a step).
constexpr int kPitch = 72, kTileWidth = kPitch - 2 * kHalo;       // floats per row
constexpr int kTileRows = 55, kArea = kPitch * kTileRows + 8;     // floats per array
__host__ __device__ constexpr int tileHeight(int rows) { return kTileRows - 2 * kHalo - rows; }   // windows reach past the tile
constexpr int kHaloWords = 4;              // mailbox words a thread collects per exchange, at most
constexpr int kResidentReceivers = 1024;   // most receivers of a run's gather

struct ResidentPlan {
    int px, pz;        // tiles across and down
    int longest;       // longest side of a tile
    int side;          // mailbox words per side of a tile and kind of exchange
    uint4* mail;
};

// Arrays in shared memory.  The split schemes keep the sums of the halves whose x derivatives are
// taken (SplitRow).
enum SplitArray { aVx1, aVx2, aVxS, aVz1, aVz2, aVzS, aSxx1, aSxx2, aSxxS, aSzz1, aSzz2, aSxz1, aSxz2, aSxzS, kSplitArrays };
enum HybridArray { aVx, aVz, aSxx, aSzz, aSxz, kHybridArrays };
template <int S> constexpr int residentArrays = S == kHybrid ? int(kHybridArrays) : int(kSplitArrays);
template <int S> constexpr int cellWords = S == kHybrid ? 1 : 2;   // mailbox words per halo cell

__device__ __forceinline__ void sendWord(uint4* p, float a, float b, unsigned epoch) {
    const unsigned long long lo = (unsigned long long)__float_as_uint(a) | ((unsigned long long)__float_as_uint(b) << 32);
    asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p), "l"(lo),
                 "l"((unsigned long long)epoch)
                 : "memory");
}
__device__ __forceinline__ bool receiveWord(const uint4* p, unsigned epoch, float& a, float& b) {
    unsigned long long lo, hi;
    asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
                 : "=l"(lo), "=l"(hi)
                 : "l"(p)
                 : "memory");
    a = __uint_as_float(unsigned(lo));
    b = __uint_as_float(unsigned(lo >> 32));
    return unsigned(hi) == epoch;
}

// One tile of a resident run.
template <int S> struct Tile {
    const Grid2D& g;
    const ResidentPlan& P;
    float* sm;
    int tx, tz, left, top, width, height;   // place among the tiles, first cell, size
    bool surface;                           // the tile or its halo holds rows that take part in images

    __device__ __forceinline__ Tile(const Grid2D& grid, const ResidentPlan& plan, float* shared) : g(grid), P(plan), sm(shared) {
        tx = int(blockIdx.x) % P.px; tz = int(blockIdx.x) / P.px;
        left = int((long long)tx * g.NX / P.px); width = int((long long)(tx + 1) * g.NX / P.px) - left;
        top = int((long long)tz * g.NZ / P.pz); height = int((long long)(tz + 1) * g.NZ / P.pz) - top;
        surface = S == kFree && top - kHalo <= g.fs + 4 && top + height + kHalo > g.fs - 4;
    }
    __device__ __forceinline__ int cell(int row, int col) const { return (row + kHalo) * kPitch + col + kHalo; }
    __device__ __forceinline__ float* array(int a) const { return sm + a * kArea; }
    __device__ __forceinline__ void put(int a, int at, float v) const { sm[a * kArea + at] = v; }
    __device__ __forceinline__ float get(int a, int at) const { return sm[a * kArea + at]; }
    // Both halves of an array group, and their sum where one is kept.
    __device__ __forceinline__ void putHalves(int a, int at, float v1, float v2, bool sum) const {
        put(a, at, v1); put(a + 1, at, v2);
        if (sum) put(a + 2, at, v1 + v2);
    }

    // The images of a free surface (Cuda_Check.cu:491-508) in the rows that the tile and its halo
    // hold: szz of row fs+l into row fs-l, sxz of row fs+l-1 into row fs-l, l = 1..4.  A pass of its
    // own over the eight rows: tested for by every cell's update it cost the whole tile more.
    __device__ __forceinline__ void images() const {
        for (int n = threadIdx.x; n < 8 * width; n += blockDim.x) {
            const int col = n % width, l = n / width % 4 + 1;
            const bool second = n >= 4 * width;
            const int from = g.fs + l - (second ? 1 : 0) - top, to = g.fs - l - top;
            if (left + col < 4 || left + col >= g.NX - 4 || !holds(from) || !holds(to)) continue;
            const int a = second ? aSxz1 : aSzz1;
            putHalves(a, cell(to, col), -get(a, cell(from, col)), -get(a + 1, cell(from, col)), false);
        }
    }
    __device__ __forceinline__ bool holds(int row) const { return row >= -kHalo && row < height + kHalo; }
};

// The halo words that a thread sends and collects: the same ones in every exchange.  Sending has
// threads of its own choice read the border cells from shared memory, after a barrier: sent by
// the threads that compute the cells, each word's address cost every warp of the tile its
// instructions, since columns of the left and right borders are in all of them.
template <int S> struct HaloWords {
    int count = 0;
    int mail[kHaloWords];    // word offset from the tile's mailboxes of one kind
    int place[kHaloWords];   // halo cell in shared memory; bitwise complement above and below
    int out[kHaloWords];     // word offset of the border cell's word in the neighbour's mailboxes
    int from[kHaloWords];    // border cell in shared memory

    __device__ __forceinline__ void init(const Tile<S>& T) {
        const bool beside[4] = {T.tx > 0, T.tx + 1 < T.P.px, T.tz > 0, T.tz + 1 < T.P.pz};   // left, right, above, below
        const int step[4] = {-1, 1, -T.P.px, T.P.px};
#pragma unroll
        for (int h = 0; h < kHaloWords; ++h) {
            int n = threadIdx.x + h * blockDim.x;
            mail[h] = place[h] = out[h] = from[h] = 0;
#pragma unroll
            for (int side = 0; side < 4; ++side) {
                const int length = side < 2 ? T.height : T.width, words = beside[side] ? kHalo * length * cellWords<S> : 0;
                if (n >= 0 && n < words) {
                    const int w = n % cellWords<S>, pos = (n / cellWords<S>) % length, layer = n / (cellWords<S> * length);
                    const int word = (layer * T.P.longest + pos) * cellWords<S> + w;
                    mail[h] = side * T.P.side + word;
                    // What this tile collects on one side its neighbour there sends from the opposite border.
                    out[h] = step[side] * 8 * T.P.side + (side ^ 1) * T.P.side + word;
                    const int halo = side == 0 || side == 2 ? layer - kHalo : side == 1 ? T.width + layer : T.height + layer;
                    const int border = side == 0 || side == 2 ? layer : side == 1 ? T.width - kHalo + layer : T.height - kHalo + layer;
                    place[h] = side < 2 ? T.cell(pos, halo) : ~T.cell(halo, pos);
                    from[h] = side < 2 ? T.cell(pos, border) : T.cell(border, pos);
                    count = h + 1;
                }
                n -= words;   // negative once found, and from then on
            }
        }
    }

    // Sends the words of one exchange (kind 0 velocities, 1 stresses).
    __device__ __forceinline__ void send(const Tile<S>& T, int kind, unsigned epoch) const {
        uint4* box = T.P.mail + (int(blockIdx.x) * 2 + kind) * 4 * T.P.side;
#pragma unroll
        for (int h = 0; h < kHaloWords; ++h) {
            if (h >= count) break;
            const bool vertical = place[h] < 0;
            int a, b;
            if constexpr (S == kHybrid) {
                a = kind == 0 ? aVx : vertical ? aSzz : aSxx;
                b = kind == 0 ? aVz : aSxz;
            } else {
                const bool second = (mail[h] & 1) != 0;
                a = kind == 0 ? (second ? aVz1 : aVx1) : second ? aSxz1 : vertical ? aSzz1 : aSxx1;
                b = a + 1;
            }
            sendWord(box + out[h], T.get(a, from[h]), T.get(b, from[h]), epoch);
        }
    }

    // Puts one received word in its place.
    __device__ __forceinline__ void deliver(const Tile<S>& T, int kind, int h, float a, float b) const {
        const bool vertical = place[h] < 0;
        const int at = vertical ? ~place[h] : place[h];
        if constexpr (S == kHybrid) {
            if (kind == 0) { T.put(aVx, at, a); T.put(aVz, at, b); }
            else { T.put(vertical ? aSzz : aSxx, at, a); T.put(aSxz, at, b); }
        } else {
            const bool second = (mail[h] & 1) != 0;
            if (kind == 0) {
                T.putHalves(second ? aVz1 : aVx1, at, a, b, true);
            } else if (!vertical) {
                T.putHalves(second ? aSxz1 : aSxx1, at, a, b, true);
            } else {
                if (second) T.putHalves(aSxz1, at, a, b, true);
                else T.putHalves(aSzz1, at, a, b, false);
            }
        }
    }

    // Waits (bounded) for the words of one exchange; false when it gave up.
    __device__ __forceinline__ bool collect(const Tile<S>& T, int kind, unsigned epoch, GridSync* gs,
                                            const BarrierLimits& lim) const {
        const uint4* box = T.P.mail + (int(blockIdx.x) * 2 + kind) * 4 * T.P.side;
        unsigned waiting = (1u << count) - 1;
        long long start = 0;
        for (unsigned turn = 0; waiting; ++turn) {
            float a[kHaloWords], b[kHaloWords];
            bool here[kHaloWords];
#pragma unroll
            for (int h = 0; h < kHaloWords; ++h) here[h] = (waiting >> h & 1) && receiveWord(box + mail[h], epoch, a[h], b[h]);
#pragma unroll
            for (int h = 0; h < kHaloWords; ++h)
                if (here[h]) {
                    deliver(T, kind, h, a[h], b[h]);
                    waiting &= ~(1u << h);
                }
            if (!waiting || (turn & 63) != 63) continue;
            if (start == 0) start = clock64();
            if (*reinterpret_cast<volatile unsigned*>(&gs->failed)) return false;
            if (clock64() - start > lim.cycles) {
                atomicExch(&gs->failed, 1u);
                return false;
            }
        }
        return true;
    }
};

// `count` steps from ctl->base; single-source runs only.  The control block is only read: the mailboxes
// order neighbours, not a block that starts late against one that has finished, so a block that
// moved `base` past the run could give a late one the wrong first step.  Every run has a
// configureRun of its own, so nothing wants it moved.
template <int S, int R>
__global__ void __launch_bounds__(kResidentThreads, 1) residentRun(Grid2D g, Fields2D f, const Control2D* ctl, GridSync* gs,
                                                                   int count, BarrierLimits lim, ResidentPlan P) {
    extern __shared__ float sm[];
    __shared__ int listed;
    __shared__ unsigned failed;
    __shared__ Control2D c;
    const Tile<S> T(g, P, sm);
    int2* list = reinterpret_cast<int2*>(sm + residentArrays<S> * kArea);   // {receiver, cell} of the tile's receivers
    const int tid = threadIdx.x;
    if (tid == 0) {
        listed = 0;
        c = *ctl;
        failed = *reinterpret_cast<volatile unsigned*>(&gs->failed);
    }

    // Every array with its halo.
    const int loadWidth = T.width + 2 * kHalo, loadCells = loadWidth * (T.height + 2 * kHalo);
    for (int n = tid; n < loadCells; n += blockDim.x) {
        const int row = n / loadWidth - kHalo, col = n % loadWidth - kHalo;
        const int i = T.top + row, j = T.left + col, k = i * g.NX + j, at = T.cell(row, col);
        const bool in = i >= 0 && i < g.NZ && j >= 0 && j < g.NX;
        auto read = [&](const float* p) { return in ? __ldcg(p + k) : 0.0f; };
        if constexpr (S == kHybrid) {
            T.put(aVx, at, read(f.vx)); T.put(aVz, at, read(f.vz));
            T.put(aSxx, at, read(f.sxx)); T.put(aSzz, at, read(f.szz)); T.put(aSxz, at, read(f.sxz));
        } else {
            T.putHalves(aVx1, at, read(f.vx1), read(f.vx2), true);
            T.putHalves(aVz1, at, read(f.vz1), read(f.vz2), true);
            T.putHalves(aSxx1, at, read(f.sxx1), read(f.sxx2), true);
            T.putHalves(aSzz1, at, read(f.szz1), read(f.szz2), false);
            T.putHalves(aSxz1, at, read(f.sxz1), read(f.sxz2), true);
        }
    }

    // The thread's cells.
    const int col = tid % T.width, row = tid / T.width * R, j = T.left + col, i0 = T.top + row;
    const int rows = min(R, T.height - row);            // <= 0: no cells
    const bool columnIn = j >= 4 && j < g.NX - 4;
    const int firstRow = S == kFree ? g.fs : 4;
    // Stresses and velocities stand in the arrays; the hybrid layer's halves in registers.
    float hs[S == kHybrid ? R : 1][6], hv[S == kHybrid ? R : 1][4];
    float m[R][5];   // hybrid: muZ, l2mX, lambdaX, rhoXZ, rho; split: mu, l2m, lambda, rho, mean rho
    Damping<R> d;
    if (rows > 0) {
        d.load(g, f, i0, j);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (r >= rows) break;
            const int i = i0 + r, k = i * g.NX + j;
            if (S == kFree && i <= g.fs + 5) d.z[r] = d.zh[r] = 0.0f;
            if (!(columnIn && i >= 4 && i < g.NZ - 4)) continue;
            auto at = [&](const float* p) { return __ldcg(p + k); };
            if constexpr (S == kHybrid) {
                m[r][0] = at(f.muZ); m[r][1] = at(f.l2mX); m[r][2] = at(f.lambdaX); m[r][3] = at(f.rhoXZ); m[r][4] = at(f.rhoOrig);
                if (inPml(g, i, j)) {
                    hs[r][0] = at(f.sxz1); hs[r][1] = at(f.sxz2); hs[r][2] = at(f.sxx1);
                    hs[r][3] = at(f.szz1); hs[r][4] = at(f.sxx2); hs[r][5] = at(f.szz2);
                    hv[r][0] = at(f.vz1); hv[r][1] = at(f.vz2); hv[r][2] = at(f.vx1); hv[r][3] = at(f.vx2);
                }
            } else {
                m[r][0] = 0.5f * (at(f.mu) + at(f.mu + g.NX));
                m[r][1] = 0.5f * (at(f.l2m) + at(f.l2m + 1));
                m[r][2] = 0.5f * (at(f.lambda) + at(f.lambda + 1));
                m[r][3] = at(f.rho);
                m[r][4] = 0.25f * (at(f.rho) + at(f.rho + 1) + at(f.rho + g.NX) + at(f.rho + g.NX + 1));
            }
        }
    }
    HaloWords<S> halo;
    halo.init(T);
    __syncthreads();   // `listed` is 0, `c` and `failed` are there
    if (failed) return;   // an earlier run left the state half way, or this one has already
    if (c.gatherOn)
        for (int r = tid; r < c.rcvCount; r += blockDim.x) {
            const int k = c.rcvIdx[r], i = k / g.NX - T.top, jr = k % g.NX - T.left;
            if (i >= 0 && i < T.height && jr >= 0 && jr < T.width) list[atomicAdd(&listed, 1)] = make_int2(r, T.cell(i, jr));
        }
    // Gather row of step `step` (recordStep), from the tile's final velocities.
    auto record = [&](int step) {
        const int rs = step - c.gatherStart;
        if (!c.gatherOn || rs < 0 || rs % c.gatherStride != 0 || rs / c.gatherStride >= c.gatherSamples) return;
        const int sample = rs / c.gatherStride;
        for (int n = tid; n < listed; n += blockDim.x) {
            const int2 e = list[n];
            c.gatherVx[std::size_t(e.x) * c.gatherSamples + sample] = T.array(S == kHybrid ? int(aVx) : int(aVxS))[e.y];
            c.gatherVz[std::size_t(e.x) * c.gatherSamples + sample] = T.array(S == kHybrid ? int(aVz) : int(aVzS))[e.y];
        }
    };
    // A column window of an array, `before` rows above the thread's first.
    auto window = [&](Column<R>& w, int a, int before) {
        const float* p = T.array(a) + T.cell(row - before, col);
#pragma unroll
        for (int k = 0; k < R + 7; ++k) w.v[k] = p[k * kPitch];
    };

    const unsigned firstEpoch = gs->first;
    bool bad = false;
    for (int q = 0; q < count; ++q) {
        const int step = c.base + q;
        unsigned epoch = firstEpoch + 2 * unsigned(q);
        if (q > 0) bad = !halo.collect(T, 0, epoch, gs, lim);
        if (__syncthreads_or(bad)) return;

        // Stresses.
        ++epoch;
        if (rows > 0) {
            if constexpr (S == kHybrid) {
                Column<R> vx, vz;
                window(vx, aVx, 3);
                window(vz, aVz, 4);
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    if (r >= rows) break;
                    const int i = i0 + r, k = i * g.NX + j, at = T.cell(row + r, col);
                    float sxz = T.get(aSxz, at), sxx = T.get(aSxx, at), szz = T.get(aSzz, at);
                    if (columnIn && i >= 4 && i < g.NZ - 4) {
                        const bool pml = inPml(g, i, j);
                        float w = 0.0f;
                        if (!pml && q > 0 && k == c.srcIdx && stressSource(c, step - 1, w)) {
                            if (c.srcType == SEIS2D_EXPLOSIVE) { sxx = __fadd_rn(sxx, w); szz = __fadd_rn(szz, w); }
                            else sxz = __fadd_rn(sxz, w);
                        }
                        hybridStress(g, pml, d.at(r, false), m[r][0], m[r][1], m[r][2], dxBackward(g, T.array(aVz) + at),
                                     dzAt(g, vx, r), dxForward(g, T.array(aVx) + at), dzAt(g, vz, r), sxz, sxx, szz, hs[r]);
                        T.put(aSxz, at, sxz); T.put(aSxx, at, sxx); T.put(aSzz, at, szz);
                    }
                }
            } else {
                SplitColumn<R> vx, vz;
                window(vx.a, aVx1, 3); window(vx.b, aVx2, 3);
                window(vz.a, aVz1, 4); window(vz.b, aVz2, 4);
                vx.sum();
                vz.sum();
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    if (r >= rows) break;
                    const int i = i0 + r, k = i * g.NX + j, at = T.cell(row + r, col);
                    float t[6] = {T.get(aSxx1, at), T.get(aSxx2, at), T.get(aSzz1, at),
                                  T.get(aSzz2, at), T.get(aSxz1, at), T.get(aSxz2, at)};
                    if (columnIn && i >= firstRow && i < g.NZ - 4) {
                        const SplitRow rvx{T.array(aVx1) + at, T.array(aVx2) + at, T.array(aVxS) + at};
                        const SplitRow rvz{T.array(aVz1) + at, T.array(aVz2) + at, T.array(aVzS) + at};
                        const Damp damp = d.at(r, false);
                        float w = 0.0f;
                        if (q > 0 && k == c.srcIdx && stressSource(c, step - 1, w)) addSplitSource(c, w, t);
                        const float dvx_dx = dxForward(g, rvx);
                        if (S == kFree && i == g.fs)
                            freeRowStress(g, damp, m[r][0], f.dp[j], dvx_dx, weigh2(g, rvz.tap(0, -1), rvz.tap(1, -2)),
                                          weigh2(g, vx.tap(r + 4, r + 3), vx.tap(r + 5, r + 2)), t);
                        else
                            splitStress(g, damp, m[r][0], m[r][1], m[r][2], dvx_dx, vz.dz(g, r), dxBackward(g, rvz), vx.dz(g, r), t);
                        T.putHalves(aSxx1, at, t[0], t[1], true);
                        T.putHalves(aSzz1, at, t[2], t[3], false);
                        T.putHalves(aSxz1, at, t[4], t[5], true);
                    }
                }
            }
        }
        if (q > 0) record(step - 1);   // the velocities of the step before, still in place
        __syncthreads();
        if (!(q == 0 && int(blockIdx.x) == lim.withheldBlock)) halo.send(T, 1, epoch);   // (test hook)
        bad = !halo.collect(T, 1, epoch, gs, lim);
        if (__syncthreads_or(bad)) return;
        if (S == kFree && T.surface) {
            T.images();
            __syncthreads();
        }

        // Velocities.
        ++epoch;
        if (rows > 0) {
            if constexpr (S == kHybrid) {
                Column<R> szz, sxz;
                window(szz, aSzz, 3);
                window(sxz, aSxz, 4);
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    if (r >= rows) break;
                    const int i = i0 + r, k = i * g.NX + j, at = T.cell(row + r, col);
                    float vx = T.get(aVx, at), vz = T.get(aVz, at);
                    if (i == 0 || i == g.NZ - 1 || j == 0 || j == g.NX - 1) {
                        vx = vz = 0.0f;
                    } else if (columnIn && i >= 4 && i < g.NZ - 4) {
                        hybridVelocity(g, inPml(g, i, j), d.at(r, false), m[r][3], m[r][4], dxForward(g, T.array(aSxz) + at),
                                       dzAt(g, szz, r), dxBackward(g, T.array(aSxx) + at), dzAt(g, sxz, r), vx, vz, hv[r]);
                        forceSource<S>(g, f, c, step, k, vx, vz);
                    }
                    T.put(aVx, at, vx); T.put(aVz, at, vz);
                }
            } else {
                SplitColumn<R> szz, sxz;
                window(szz.a, aSzz1, 3); window(szz.b, aSzz2, 3);
                window(sxz.a, aSxz1, 4); window(sxz.b, aSxz2, 4);
                szz.sum();
                sxz.sum();
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    if (r >= rows) break;
                    const int i = i0 + r, k = i * g.NX + j, at = T.cell(row + r, col);
                    float u[4] = {T.get(aVx1, at), T.get(aVx2, at), T.get(aVz1, at), T.get(aVz2, at)};
                    const bool inside = columnIn && i >= 4 && i < g.NZ - 4;
                    if (i == 0 || i == g.NZ - 1 || j == 0 || j == g.NX - 1 || (S == kFree && inside && i < g.fs)) {
                        u[0] = u[1] = u[2] = u[3] = 0.0f;
                    } else if (inside) {
                        const SplitRow rxx{T.array(aSxx1) + at, T.array(aSxx2) + at, T.array(aSxxS) + at};
                        const SplitRow rxz{T.array(aSxz1) + at, T.array(aSxz2) + at, T.array(aSxzS) + at};
                        splitVelocity(g, d.at(r, false), m[r][3], m[r][4], dxBackward(g, rxx), sxz.dz(g, r),
                                      dxForward(g, rxz), szz.dz(g, r), u);
                        forceSource<S>(g, f, c, step, k, u[0], u[2]);
                    }
                    T.putHalves(aVx1, at, u[0], u[1], true);
                    T.putHalves(aVz1, at, u[2], u[3], true);
                }
            }
        }
        __syncthreads();
        if (q + 1 < count) halo.send(T, 0, epoch);
    }

    // The last step's receivers and stress-type source, and the state back to memory.
    const int last = c.base + count - 1;
    record(last);
#pragma unroll
    for (int r = 0; r < R; ++r) {
        if (r >= rows) break;
        const int i = i0 + r, k = i * g.NX + j, at = T.cell(row + r, col);
        const bool updated = columnIn && i >= firstRow && i < g.NZ - 4;
        float w = 0.0f;
        const bool source = updated && k == c.srcIdx && stressSource(c, last, w);
        if constexpr (S == kHybrid) {
            f.vx[k] = T.get(aVx, at); f.vz[k] = T.get(aVz, at);
            if (!updated) continue;
            float sxz = T.get(aSxz, at), sxx = T.get(aSxx, at), szz = T.get(aSzz, at);
            if (source) {
                if (c.srcType == SEIS2D_EXPLOSIVE) { sxx += w; szz += w; }
                else sxz += w;
            }
            f.sxz[k] = sxz; f.sxx[k] = sxx; f.szz[k] = szz;
            if (inPml(g, i, j)) {
                f.sxz1[k] = hs[r][0]; f.sxz2[k] = hs[r][1]; f.sxx1[k] = hs[r][2];
                f.szz1[k] = hs[r][3]; f.sxx2[k] = hs[r][4]; f.szz2[k] = hs[r][5];
                f.vz1[k] = hv[r][0]; f.vz2[k] = hv[r][1]; f.vx1[k] = hv[r][2]; f.vx2[k] = hv[r][3];
            }
        } else {
            f.vx1[k] = T.get(aVx1, at); f.vx2[k] = T.get(aVx2, at); f.vz1[k] = T.get(aVz1, at); f.vz2[k] = T.get(aVz2, at);
            if (!updated) continue;
            float t[6] = {T.get(aSxx1, at), T.get(aSxx2, at), T.get(aSzz1, at),
                          T.get(aSzz2, at), T.get(aSxz1, at), T.get(aSxz2, at)};
            if (S == kFree) {
                const int l = i - g.fs;
                if (l >= 1 && l <= 4) { f.szz1[k - 2 * l * g.NX] = -t[2]; f.szz2[k - 2 * l * g.NX] = -t[3]; }
                if (l <= 3) { f.sxz1[k - (2 * l + 1) * g.NX] = -t[4]; f.sxz2[k - (2 * l + 1) * g.NX] = -t[5]; }
            }
            if (source) addSplitSource(c, w, t);
            f.sxx1[k] = t[0]; f.sxx2[k] = t[1]; f.szz1[k] = t[2]; f.szz2[k] = t[3]; f.sxz1[k] = t[4]; f.sxz2[k] = t[5];
        }
    }
}

}  // namespace seis2d
