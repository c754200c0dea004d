// Kernels of the step: the phases of phys/step_phases.h on the device.
//
// A block of the ray, drive, pair and finish kernels serves 32 arenas, one warp per car or body: lanes
// run over arenas, so every record word is read and written coalesced, and the bodies of an
// arena exchange what the reference's order needs through shared memory.  The queue kernels
// (heavy rays, contacts, islands) run one queued item per thread; their counts are known on the
// device only, so their grids loop.
#pragma once
#include "phys/step_phases.h"

namespace rsb {

// Adds a thread's counters to the handle's statistics: one atomic per block and counter.
RSB_D void blockStats(const EngineView& D, const PhaseStats& st) {
    __shared__ uint32_t sum[4];
    if (threadIdx.x < 4) sum[threadIdx.x] = 0;
    __syncthreads();
    const uint32_t v[4] = {st.nStatic, st.nCulled, st.nMissed, st.nRows};
    for (int k = 0; k < 4; k++) {
        const uint32_t w = __reduce_add_sync(0xffffffffu, v[k]);
        if ((threadIdx.x & 31) == 0 && w) atomicAdd(&sum[k], w);
    }
    __syncthreads();
    if (threadIdx.x < 4 && sum[threadIdx.x] && D.counters)
        atomicAdd(&D.counters[threadIdx.x], (unsigned long long)sum[threadIdx.x]);
}

// Places for n items of this thread in a queue: one atomic per warp.  Called by whole warps.
RSB_D uint32_t queueAlloc(uint32_t* counter, uint32_t n) {
    const int lane = threadIdx.x & 31;
    uint32_t incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    uint32_t base = 0;
    if (lane == 31 && incl) base = atomicAdd(counter, incl);
    base = __shfl_sync(0xffffffffu, base, 31);
    return base + incl - n;
}

// Warps per SM that a queue kernel spreads its items over before a warp takes more than one of
// them, up to 32.  Items' paths differ, so few items spread wide finish in the time of the longest
// one; but a thread's local memory shares its cache lines with its warp's other lanes, so the
// kernels that use much of it lose by spreading when the queues are long.  Measured with 4 / 8 /
// 16 / 32 / 64, us per tick, 3v3 x 65,536 after 17 env steps: heavy rays 180 / 125 / 111 / 104 /
// 149 (2v2 x 8,192: 49 / 42 / 52 / 61 / 83), triangles 116 / 79 / 64 / 95 / 145 (44 / 33 / 46 /
// 61 / 74); find 202 with 32 items to every warp and 107 with 64, deep 214 and 141, combine 113 and 102, whole-arena
// islands 234 and 886 (64).
constexpr int kMeshRayWarps = 32, kBodyRayWarps = 16, kTriangleWarps = 12, kPairWarps = 12, kCombineWarps = 16,
              kBodyWarps = 8;

// Items of several queues, fn(queue, item): a warp takes items of one queue at a time, as few as
// it takes to give each of spread[queue] warps some.
template <int NQ, class F>
RSB_D void forItems(const uint32_t (&n)[NQ], const uint32_t (&spread)[NQ], F&& fn) {
    const uint32_t warps = gridDim.x * (blockDim.x >> 5), lane = threadIdx.x & 31u;
    uint32_t width[NQ], tiles[NQ], total = 0;
#pragma unroll
    for (int k = 0; k < NQ; k++) {
        width[k] = max(1u, min(32u, (n[k] + spread[k] - 1u) / spread[k]));
        tiles[k] = (n[k] + width[k] - 1u) / width[k];
        total += tiles[k];
    }
    for (uint32_t tile = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); tile < total; tile += warps) {
        uint32_t q = tile;
#pragma unroll
        for (int k = 0; k < NQ; k++) {
            if (q < tiles[k]) {
                const uint32_t i = q * width[k] + lane;
                if (lane < width[k] && i < n[k]) fn(k, i);
                break;
            }
            q -= tiles[k];
        }
    }
}

constexpr int BODY_THREADS = MAX_BODIES * PHASE_ARENAS;
constexpr int CAR_THREADS = MAX_CARS * PHASE_ARENAS;

RSB_D size_t rayPlaces(const EngineView& D) { return (size_t)4 * MAX_CARS * D.N; }

__global__ void __launch_bounds__(CAR_THREADS) rayKernel(const __grid_constant__ EngineView D,
                                                         const __grid_constant__ StepTemp T) {
    __shared__ uint32_t cell[MAX_BODIES][PHASE_ARENAS];
    const int lane = threadIdx.x & 31, s = threadIdx.x >> 5;
    const int a = blockIdx.x * PHASE_ARENAS + lane;
    const int nb = a < D.N ? arenaBodies(D, a) : 0;
    for (int b = s; b < MAX_BODIES; b += blockDim.x >> 5)
        if (b < nb) cell[b][lane] = bodyCellWord(D, a, b);
    __syncthreads();
    PhaseStats st{0, 0, 0, 0};
    Xf xf;
    bool culled = false;
    const bool live = 1 + s < nb && rayCar(D, a, s, xf, culled);
    auto near = [&](uint32_t at) {
        uint32_t n = 0;
        for (int b = 0; b < nb; b++) n |= cellsNear(at, cell[b][lane]) ? 1u << b : 0u;
        return n;
    };
#pragma unroll 1
    for (int w = 0; w < 4; w++) {
        const RayClass c = live ? rayPhase(D, T, a, s, w, xf, culled, near, st) : RAY_DONE;
        const uint32_t m = queueAlloc(&T.count[QC_RAY], c == RAY_MESHES ? 1u : 0u);
        const uint32_t o = queueAlloc(&T.count[QC_BODYRAY], c == RAY_BODIES ? 1u : 0u);
        if (c == RAY_MESHES) T.rayQ[m] = (uint32_t)rayIdx(D, a, s, w);
        else if (c == RAY_BODIES) T.rayQ[rayPlaces(D) + o] = (uint32_t)rayIdx(D, a, s, w);
    }
    blockStats(D, st);
}

// Rays near meshes: few registers, so that many warps wait for triangles at once (in one kernel
// with the convex casts, at 232 registers, 295 us per tick at 3v3 x 65,536).
constexpr int MESHRAY_THREADS = 128;
__global__ void __launch_bounds__(MESHRAY_THREADS) meshRayKernel(const __grid_constant__ EngineView D,
                                                                 const __grid_constant__ StepTemp T) {
    const uint32_t n[1] = {T.count[QC_RAY]};
    PhaseStats st{0, 0, 0, 0};
    const uint32_t w[1] = {kMeshRayWarps * T.sms};
    forItems(n, w, [&](int, uint32_t i) {
        const uint32_t r = T.rayQ[i];
        if (meshRayPhase(D, T, r, st)) T.rayQ[rayPlaces(D) + atomicAdd(&T.count[QC_BODYRAY], 1u)] = r;
    });
    blockStats(D, st);
}

template <int MINB>
__global__ void __launch_bounds__(128, MINB) bodyRayKernel(const __grid_constant__ EngineView D,
                                                           const __grid_constant__ StepTemp T) {
    const uint32_t n[1] = {T.count[QC_BODYRAY]};
    PhaseStats st{0, 0, 0, 0};
    const uint32_t w[1] = {kBodyRayWarps * T.sms};
    forItems(n, w, [&](int, uint32_t i) { bodyRayPhase(D, T, T.rayQ[rayPlaces(D) + i], st); });
    blockStats(D, st);
}

// The car's state and its four wheels fill about 250 registers; held to 168, two blocks share an
// SM at the price of some spills: 183 us against 265 at 3v3 x 65,536.
__global__ void __launch_bounds__(CAR_THREADS, 2) driveKernel(const __grid_constant__ EngineView D,
                                                           const __grid_constant__ StepTemp T) {
    __shared__ DriveShared sh;
    const int lane = threadIdx.x & 31;
    DriveThread t;
    t.s = threadIdx.x >> 5;
    t.la = lane;
    t.a = blockIdx.x * PHASE_ARENAS + lane;
    t.finished = true;
    t.deps = 0;
    const bool valid = t.a < D.N && 1 + t.s < arenaBodies(D, t.a);
    if (blockIdx.x == 0 && threadIdx.x == 0) T.count[QC_RAY] = T.count[QC_BODYRAY] = 0;  // the queued rays are cast
    if (threadIdx.x < PHASE_ARENAS) sh.done[lane] = 0;
    if (valid) driveLoad(D, T, t, sh);
    __syncthreads();
    if (valid && t.finished) atomicOr(&sh.done[lane], 1u << t.s);
    __syncthreads();
    // a car waits only for cars of higher slots, so every round finishes the highest one left
    for (int round = 0; round <= MAX_CARS; round++) {
        const bool ready = !t.finished && !(t.deps & ~sh.done[lane]);
        if (ready) driveRun(t, sh);
        const int all = __syncthreads_and(t.finished);
        if (all) break;
        if (ready) atomicOr(&sh.done[lane], 1u << t.s);
        __syncthreads();
    }
    if (valid) driveStore(D, T, t);
}

__global__ void __launch_bounds__(BODY_THREADS) pairKernel(const __grid_constant__ EngineView D,
                                                           const __grid_constant__ StepTemp T, bool firstTick) {
    __shared__ PairShared sh;
    const int lane = threadIdx.x & 31;
    PairThread t;
    t.b = threadIdx.x >> 5;
    t.la = lane;
    t.a = blockIdx.x * PHASE_ARENAS + lane;
    t.nb = t.a < D.N ? arenaBodies(D, t.a) : 0;
    const bool valid = t.b < t.nb;
    if (threadIdx.x < PHASE_ARENAS) sh.need[lane] = 0;
    if (valid) pairLoad(D, T, t, sh, firstTick);
    __syncthreads();
    if (valid) pairPick(D, t, sh);
    __syncthreads();
    PhaseStats st{0, 0, 0, 0};
    BodyStatics o;
    o.meshes = o.planes = 0;
    uint32_t dyn = 0;
    if (valid) {
        o = pairStatics(D, t, st);
        dyn = pairDynamics(D, t, sh);
    }
    const uint32_t m0 = queueAlloc(&T.count[t.b == 0 ? QC_BALLMESH : QC_CARMESH], (uint32_t)__popc(o.meshes));
    const uint32_t p0 = queueAlloc(&T.count[QC_PLANE], (uint32_t)__popc(o.planes));
    const uint32_t d0 = queueAlloc(&T.count[t.b == 0 ? QC_CARBALL : QC_CARCAR], (uint32_t)__popc(dyn));
    if (valid) {
        pairStore(D, T, t, o, dyn, m0, p0, d0);
        pairNeed(t, o, sh);
    }
    __syncthreads();
    const uint32_t need = sh.need[lane];
    if (valid) pairStoreHead(D, T, t, o, need);
    if (threadIdx.x < PHASE_ARENAS) {
        const bool whole = arenaHasContacts(need) && !arenaByBodies(need);
        const uint32_t as = queueAlloc(&T.count[QC_SOLVE], whole ? 1u : 0u);
        if (whole) T.solveQ[as] = (uint32_t)t.a;
    }
    blockStats(D, st);
}

// The candidates of mesh pairs, eight lanes to a pair: the subtrees' headers and then the leaves of
// those that overlap, eight at a time, so that the loads of a pair do not wait for one another as
// those of a walk do.  The four pairs of a warp step together (their lanes meet in the ballots).
constexpr int FIND_LANES = 8, FIND_GROUPS = 32 / FIND_LANES, FIND_HEADERS = 64;
// `list`: PAIR_CANDIDATES places for each of the warp's groups.  The pairs are nCar car pairs from
// place car0 of their queue on, then those of the ball up to `total`, from ball0 on.
RSB_D void findPairs(const EngineView& D, const StepTemp& T, int16_t (*list)[PAIR_CANDIDATES], uint32_t car0,
                     uint32_t nCar, uint32_t ball0, uint32_t total, uint32_t warp, uint32_t warps) {
    const int lane = threadIdx.x & 31, g = lane / FIND_LANES, l = lane % FIND_LANES;
    const uint32_t groupBits = (1u << FIND_LANES) - 1u, all = 0xffffffffu;
    int16_t* mine = list[g];
    const ArenaStatic& S = D.S;
    for (uint32_t p0 = warp * FIND_GROUPS; p0 < total; p0 += warps * FIND_GROUPS) {
        const uint32_t p = p0 + g;
        bool has = p < total;
        uint32_t res = 0, n = 0;
        int mesh = 0, subCount = 0, subOff = 0;
        FindBody f;
        uint16_t qmn[3], qmx[3];
        if (has) {
            res = p < nCar ? (uint32_t)resultBase(QC_CARMESH) * (uint32_t)D.N + car0 + p
                           : (uint32_t)resultBase(QC_BALLMESH) * (uint32_t)D.N + ball0 + (p - nCar);
            const PairTask k = T.tasks[res];
            mesh = k.o0;
            findBody(D, (int)k.a, k.o1 - OBJ_BALL, f);
            const MeshDesc& m = S.meshes[mesh];
            bvhQuantizeClamp(m, f.amn, 0, qmn);
            bvhQuantizeClamp(m, f.amx, 1, qmx);
            subCount = m.subCount;
            subOff = m.subOff;
        }
        if (has && subCount > FIND_HEADERS) {
            // more subtrees than a group's mask holds
            if (l == 0) findPhase(D, T, res);
            has = false;
            subCount = 0;
        }
        unsigned long long mask = 0;
        const int rounds = (__reduce_max_sync(all, subCount) + FIND_LANES - 1) / FIND_LANES;
        for (int r = 0; r < rounds; r++) {
            const int h = r * FIND_LANES + l;
            bool ov = false;
            if (h < subCount) {
                const BvhSubtree& st = S.subs[subOff + h];
                ov = qOverlap(qmn, qmx, st.qmin, st.qmax);
            }
            const uint32_t bal = __ballot_sync(all, ov);
            mask |= (unsigned long long)((bal >> (g * FIND_LANES)) & groupBits) << (r * FIND_LANES);
        }
        int pos = 0, end = 0;
        while (__any_sync(all, mask != 0 || pos < end)) {
            if (pos >= end && mask) {
                const SubtreeLeaves sl = S.subLeaves[subOff + __ffsll((long long)mask) - 1];
                mask &= mask - 1ull;
                pos = sl.off;
                end = sl.off + sl.count;
            }
            bool ok = pos + l < end;
            int tri = 0;
            if (ok) {
                const BvhNode nd = S.leaves[pos + l];
                tri = nd.data;
                ok = qOverlap(qmn, qmx, nd.qmin, nd.qmax) && findTest(D, f, triData(S, mesh, tri));
            }
            const uint32_t bits = (__ballot_sync(all, ok) >> (g * FIND_LANES)) & groupBits;
            const uint32_t at = n + (uint32_t)__popc(bits & ((1u << l) - 1u));
            if (ok && at < (uint32_t)PAIR_CANDIDATES) mine[at] = (int16_t)tri;
            n += (uint32_t)__popc(bits);
            pos += FIND_LANES;
        }
        __syncwarp();
        // places for the warp's candidates, then its pairs' places in the queues
        const uint32_t cnt = has && l == 0 && n <= (uint32_t)PAIR_CANDIDATES ? n : 0u;
        const uint32_t first = __shfl_sync(all, queueAlloc(&T.count[QC_TRI], cnt), g * FIND_LANES);
        if (has && n <= (uint32_t)PAIR_CANDIDATES)
            for (uint32_t i = l; i < n; i += FIND_LANES) putCandidate(T, first + i, res, mine[i]);
        const bool combine = has && l == 0 && findStore(T, res, first, n);
        const uint32_t at = queueAlloc(&T.count[QC_COMBINE], combine ? 1u : 0u);
        if (combine) T.combineQ[at] = res;
        __syncwarp();
    }
}

constexpr int FIND_THREADS = 128;
__global__ void __launch_bounds__(FIND_THREADS) findKernel(const __grid_constant__ EngineView D,
                                                           const __grid_constant__ StepTemp T) {
    __shared__ int16_t list[FIND_THREADS / FIND_LANES][PAIR_CANDIDATES];
    const uint32_t nCar = T.count[QC_CARMESH], total = nCar + T.count[QC_BALLMESH], nBall = T.count[QC_CARBALL];
    const uint32_t warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    findPairs(D, T, list + warp * FIND_GROUPS, 0u, nCar, 0u, total, blockIdx.x * warps + warp, gridDim.x * warps);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nBall; i += gridDim.x * blockDim.x)
        findPhase(D, T, (uint32_t)resultBase(QC_CARBALL) * (uint32_t)D.N + i);
}

template <int MINB>
__global__ void __launch_bounds__(128, MINB) triangleKernel(const __grid_constant__ EngineView D,
                                                            const __grid_constant__ StepTemp T) {
    PhaseStats st{0, 0, 0, 0};
    const uint32_t n[3] = {min(T.count[QC_TRI], T.candCap), T.count[QC_CARCAR], T.count[QC_PLANE]};
    const uint32_t w[3] = {kTriangleWarps * T.sms, kPairWarps * T.sms, kPairWarps * T.sms};
    forItems(n, w, [&](int k, uint32_t i) {
        if (k == 0) trianglePhase(D, T, i);
        else if (k == 1) carCarPhase(D, T, (uint32_t)resultBase(QC_CARCAR) * (uint32_t)D.N + i);
        else planePhase(D, T, (uint32_t)resultBase(QC_PLANE) * (uint32_t)D.N + i, st);
    });
    blockStats(D, st);
}

// The penetration solver, one item to a warp with the solver's 12 KB of faces and support points
// in shared memory.  The items are few (about one in forty arenas) and each is a serial chain
// through that memory; as thread-local memory every word of it took a sector of its own, since
// one lane was active, and a tick waited 140 us for the longest item at 3v3 x 65,536.
__global__ void __launch_bounds__(32, 1) deepKernel(const __grid_constant__ EngineView D,
                                                 const __grid_constant__ StepTemp T) {
    __shared__ EpaWork epa;
    PhaseStats st{0, 0, 0, 0};
    const uint32_t n = T.count[QC_DEEP];
    if (threadIdx.x == 0)
        for (uint32_t i = blockIdx.x; i < n; i += gridDim.x) deepPhase(D, T, T.deepQ[i], &epa, st);
    __syncwarp();
    blockStats(D, st);
}

__global__ void __launch_bounds__(128) combineKernel(const __grid_constant__ EngineView D,
                                                     const __grid_constant__ StepTemp T) {
    PhaseStats st{0, 0, 0, 0};
    const uint32_t n[1] = {T.count[QC_COMBINE]};
    const uint32_t w[1] = {kCombineWarps * T.sms};
    forItems(n, w, [&](int, uint32_t i) { combinePhase(D, T, T.combineQ[i], st); });
    blockStats(D, st);
}

struct WarpLanes {
    int lane = (int)(threadIdx.x & 31), count = 32;
    RSB_D void sync() const { __syncwarp(); }
};

// Arenas with pairs of bodies, one to a warp with its solver in shared memory: bodies are loaded
// and rows set up a lane each, the iterations run on one.  These arenas are few (one in fifty),
// and a tick waits for the one with the most rows.
__global__ void __launch_bounds__(32, 1) solveKernel(const __grid_constant__ EngineView D,
                                                     const __grid_constant__ StepTemp T) {
    __shared__ SolveShared sh;
    const uint32_t n = T.count[QC_SOLVE];
    PhaseStats st{0, 0, 0, 0};
    for (uint32_t i = blockIdx.x; i < n; i += gridDim.x) solvePhase(D, T, (int)T.solveQ[i], sh, WarpLanes{}, st);
    blockStats(D, st);
}

constexpr int SOLVEBODY_THREADS = 64;
__global__ void __launch_bounds__(SOLVEBODY_THREADS) solveBodyKernel(const __grid_constant__ EngineView D,
                                                                     const __grid_constant__ StepTemp T) {
    const uint32_t n[1] = {T.count[QC_BODY]}, w[1] = {kBodyWarps * T.sms};
    PhaseStats st{0, 0, 0, 0};
    forItems(n, w, [&](int, uint32_t i) { bodyPhase(D, T, T.bodyQ[i], st); });
    blockStats(D, st);
}

__global__ void __launch_bounds__(BODY_THREADS) finishKernel(const __grid_constant__ EngineView D,
                                                             const __grid_constant__ StepTemp T) {
    __shared__ FinishShared sh;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    FinishThread t;
    t.body = warp;
    t.la = lane;
    t.a = blockIdx.x * PHASE_ARENAS + lane;
    t.nb = t.a < D.N ? arenaBodies(D, t.a) : 0;
    const bool valid = t.body < t.nb, pads = t.nb > 1;
    if (blockIdx.x == 0 && threadIdx.x >= QC_CARMESH && threadIdx.x < QC_WORDS) T.count[threadIdx.x] = 0;
    if (pads)
        for (int p = warp; p < NUM_PADS; p += warps) padLoad(D, t.a, lane, p, sh);
    if (warp > 0) sh.picked[warp - 1][lane] = 0;
    else sh.touched[lane] = 0;
    __syncthreads();
    if (valid) {
        finishBody(D, T, t, sh);
        if (t.body > 0) finishPads(D, t, sh);
    }
    __syncthreads();
    if (pads)
        for (int p = warp; p < NUM_PADS; p += warps) finishPad(D, t.a, lane, p, sh);
    __syncthreads();
    if (!valid) return;
    if (t.body > 0) finishBoost(D, t, sh);
    else finishArena(D, t, sh);
}

// ------------------------------------------------------------------ small batches

// All phases of all ticks in one launch, for batches that do not fill the GPU: a block owns up to
// 32 arenas and runs the phases in turn with barriers between them, its queues in its arenas'
// share of the batch's.  Arenas are independent, so nothing crosses blocks.  What a batch of this
// size waits for otherwise is twelve launches a tick, each with a handful of items to it.
constexpr int BLOCK_WARPS = 8, BLOCK_THREADS = 32 * BLOCK_WARPS;
static_assert(MAX_BODIES * PHASE_ARENAS <= BLOCK_THREADS, "one thread per body");
struct BlockShared {
    union {
        PairShared pair;
        DriveShared drive;
        FinishShared finish;
        int16_t list[BLOCK_WARPS * FIND_GROUPS][PAIR_CANDIDATES];
        EpaWork epa[BLOCK_WARPS];
        SolveShared solve[BLOCK_WARPS];
    };
    RSB_D BlockShared() {}
};

__global__ void __launch_bounds__(BLOCK_THREADS, 1) stepBlockKernel(const __grid_constant__ EngineView D,
                                                                    const __grid_constant__ StepTemp T0, int ticks,
                                                                    int perBlock, int maxCars) {
    extern __shared__ __align__(16) unsigned char blockSmem[];
    BlockShared& sh = *reinterpret_cast<BlockShared*>(blockSmem);
    __shared__ uint32_t count[QC_WORDS], base[QC_WORDS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int a0 = blockIdx.x * perBlock, n = min(perBlock, D.N - a0);
    const size_t rays = rayPlaces(D);
    // this block's share of every queue
    StepTemp T = T0;
    T.count = count;
    T.candCap = (uint32_t)(CAP_CANDIDATES * (a0 + n));
    T.blockCap = T.arenaBlocks * (uint32_t)(a0 + n);
    if (tid == 0) {
        base[QC_RAY] = base[QC_BODYRAY] = (uint32_t)(4 * MAX_CARS * a0);
        base[QC_CARMESH] = (uint32_t)(CAP_CARMESH * a0);
        base[QC_BALLMESH] = (uint32_t)(CAP_BALLMESH * a0);
        base[QC_CARBALL] = (uint32_t)(CAP_CARBALL * a0);
        base[QC_CARCAR] = (uint32_t)(CAP_CARCAR * a0);
        base[QC_PLANE] = (uint32_t)(CAP_PLANE * a0);
        base[QC_BLOCK] = T.arenaBlocks * (uint32_t)a0;
        base[QC_SOLVE] = (uint32_t)a0;
        base[QC_BODY] = (uint32_t)(MAX_BODIES * a0);
        base[QC_TRI] = (uint32_t)(CAP_CANDIDATES * a0);
        base[QC_DEEP] = (uint32_t)((CAP_RESULTS + CAP_CANDIDATES) * a0);
        base[QC_COMBINE] = (uint32_t)(CAP_RESULTS * a0);
    }
    __syncthreads();
    if (tid < QC_WORDS) count[tid] = base[tid];
    __syncthreads();
    // items go to warps in turn, so that few items have a warp each
    const int first = lane * BLOCK_WARPS + warp;
    auto each = [&](int items, auto&& fn) {
        for (int i = first; i < items; i += BLOCK_THREADS) fn(i);
    };
    auto queue = [&](int q, auto&& fn) {
        const uint32_t b = base[q], e = count[q];
        for (uint32_t i = b + first; i < e; i += BLOCK_THREADS) fn(i);
    };
    auto place = [&](int q, uint32_t res0) { return (uint32_t)resultBase(q) * (uint32_t)D.N + res0; };
    PhaseStats st{0, 0, 0, 0};
    const int bodies = 1 + maxCars;
    // this thread's car and body
    const int la = first % n, slot = first / n, a = a0 + la;
    const int nb = arenaBodies(D, a);
    const bool hasCar = slot < maxCars && 1 + slot < nb, hasBody = slot < bodies && slot < nb;
#pragma unroll 1
    for (int tick = 0; tick < ticks; tick++) {
        // rays
        if (hasBody) sh.pair.cell[slot][la] = bodyCellWord(D, a, slot);
        __syncthreads();
        each(4 * maxCars * n, [&](int i) {
            const int l = i % n, q = i / n, s = q % maxCars, w = q / maxCars, ar = a0 + l, nbr = arenaBodies(D, ar);
            Xf xf;
            bool culled;
            if (1 + s >= nbr || !rayCar(D, ar, s, xf, culled)) return;
            const RayClass c = rayPhase(D, T, ar, s, w, xf, culled, [&](uint32_t at) {
                uint32_t m = 0;
                for (int b = 0; b < nbr; b++) m |= cellsNear(at, sh.pair.cell[b][l]) ? 1u << b : 0u;
                return m;
            }, st);
            if (c == RAY_MESHES) T.rayQ[atomicAdd(&count[QC_RAY], 1u)] = (uint32_t)rayIdx(D, ar, s, w);
            else if (c == RAY_BODIES) T.rayQ[rays + atomicAdd(&count[QC_BODYRAY], 1u)] = (uint32_t)rayIdx(D, ar, s, w);
        });
        __syncthreads();
        queue(QC_RAY, [&](uint32_t i) {
            const uint32_t r = T.rayQ[i];
            if (meshRayPhase(D, T, r, st)) T.rayQ[rays + atomicAdd(&count[QC_BODYRAY], 1u)] = r;
        });
        __syncthreads();
        queue(QC_BODYRAY, [&](uint32_t i) { bodyRayPhase(D, T, T.rayQ[rays + i], st); });
        __syncthreads();
        // cars
        if (maxCars > 0) {
            DriveShared& ds = sh.drive;
            DriveThread t;
            t.s = slot;
            t.la = la;
            t.a = a;
            t.finished = true;
            t.deps = 0;
            if (tid < PHASE_ARENAS) ds.done[tid] = 0;
            if (hasCar) driveLoad(D, T, t, ds);
            __syncthreads();
            if (hasCar && t.finished) atomicOr(&ds.done[la], 1u << slot);
            __syncthreads();
            for (int round = 0; round <= MAX_CARS; round++) {
                const bool ready = !t.finished && !(t.deps & ~ds.done[la]);
                if (ready) driveRun(t, ds);
                const int all = __syncthreads_and(t.finished);
                if (all) break;
                if (ready) atomicOr(&ds.done[la], 1u << slot);
                __syncthreads();
            }
            if (hasCar) driveStore(D, T, t);
            __syncthreads();
        }
        // pairs
        {
            PairShared& ps = sh.pair;
            PairThread t;
            t.b = slot;
            t.la = la;
            t.a = a;
            t.nb = nb;
            if (tid < PHASE_ARENAS) ps.need[tid] = 0;
            if (hasBody) pairLoad(D, T, t, ps, tick == 0);
            __syncthreads();
            if (hasBody) pairPick(D, t, ps);
            __syncthreads();
            BodyStatics o;
            if (hasBody) {
                o = pairStatics(D, t, st);
                const uint32_t dyn = pairDynamics(D, t, ps);
                const uint32_t m0 = atomicAdd(&count[slot == 0 ? QC_BALLMESH : QC_CARMESH], (uint32_t)__popc(o.meshes));
                const uint32_t p0 = atomicAdd(&count[QC_PLANE], (uint32_t)__popc(o.planes));
                const uint32_t d0 = atomicAdd(&count[slot == 0 ? QC_CARBALL : QC_CARCAR], (uint32_t)__popc(dyn));
                pairStore(D, T, t, o, dyn, m0, p0, d0);
                pairNeed(t, o, ps);
            }
            __syncthreads();
            if (hasBody) {
                const uint32_t need = ps.need[la];
                pairStoreHead(D, T, t, o, need);
                if (slot == 0 && arenaHasContacts(need) && !arenaByBodies(need))
                    T.solveQ[atomicAdd(&count[QC_SOLVE], 1u)] = (uint32_t)a;
            }
            __syncthreads();
        }
        // contacts
        {
            const uint32_t c0 = base[QC_CARMESH], b0 = base[QC_BALLMESH], nCar = count[QC_CARMESH] - c0;
            findPairs(D, T, sh.list + warp * FIND_GROUPS, c0, nCar, b0, nCar + count[QC_BALLMESH] - b0, (uint32_t)warp,
                      (uint32_t)BLOCK_WARPS);
            queue(QC_CARBALL, [&](uint32_t i) { findPhase(D, T, place(QC_CARBALL, i)); });
        }
        __syncthreads();
        if (tid == 0) count[QC_TRI] = min(count[QC_TRI], T.candCap);
        __syncthreads();
        queue(QC_TRI, [&](uint32_t i) { trianglePhase(D, T, i); });
        queue(QC_CARCAR, [&](uint32_t i) { carCarPhase(D, T, place(QC_CARCAR, i)); });
        queue(QC_PLANE, [&](uint32_t i) { planePhase(D, T, place(QC_PLANE, i), st); });
        __syncthreads();
        for (uint32_t i = base[QC_DEEP] + warp, e = count[QC_DEEP]; i < e; i += BLOCK_WARPS)
            if (lane == 0) deepPhase(D, T, T.deepQ[i], &sh.epa[warp], st);
        __syncthreads();
        queue(QC_COMBINE, [&](uint32_t i) { combinePhase(D, T, T.combineQ[i], st); });
        __syncthreads();
        // islands
        for (uint32_t i = base[QC_SOLVE] + warp, e = count[QC_SOLVE]; i < e; i += BLOCK_WARPS)
            solvePhase(D, T, (int)T.solveQ[i], sh.solve[warp], WarpLanes{}, st);
        queue(QC_BODY, [&](uint32_t i) { bodyPhase(D, T, T.bodyQ[i], st); });
        __syncthreads();
        // finish
        {
            FinishShared& fs = sh.finish;
            FinishThread t;
            t.body = slot;
            t.la = la;
            t.a = a;
            t.nb = nb;
            if (tid < QC_WORDS) count[tid] = base[tid];
            each(NUM_PADS * n, [&](int i) {
                if (arenaBodies(D, a0 + i % n) > 1) padLoad(D, a0 + i % n, i % n, i / n, fs);
            });
            if (hasCar) fs.picked[slot][la] = 0;
            if (slot == 0) fs.touched[la] = 0;
            __syncthreads();
            if (hasBody) {
                finishBody(D, T, t, fs);
                if (slot > 0) finishPads(D, t, fs);
            }
            __syncthreads();
            each(NUM_PADS * n, [&](int i) {
                if (arenaBodies(D, a0 + i % n) > 1) finishPad(D, a0 + i % n, i % n, i / n, fs);
            });
            __syncthreads();
            if (hasBody) {
                if (slot > 0) finishBoost(D, t, fs);
                else finishArena(D, t, fs);
            }
            __syncthreads();
        }
    }
    blockStats(D, st);
}

}  // namespace rsb
