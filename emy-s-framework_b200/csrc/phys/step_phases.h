// One physics tick of the whole batch as a sequence of phases.
//
// stepArena() (engine_core.h) runs a tick of one arena from start to end on one thread.  Here
// the same computation is cut where the work changes shape, so that each phase runs on the
// threads that fit it: a thread per wheel ray, per body, per contact pair, per arena with
// contacts.  Rare and expensive work (rays near meshes or other bodies, box-mesh and
// convex-convex contacts, islands to solve) goes through queues, so that a warp holds 32 items
// of it instead of the few that 32 arenas happen to have at the same time.
//
//   rays ....... every wheel ray of every car: the planes here, the rest into the ray queue
//   mesh rays .. the queued rays near meshes: meshes, planes
//   body rays .. the queued rays near other bodies: what the mesh rays left, then the bodies
//   drive ...... respawns and the vehicle update of every car
//   pairs ...... predicted motion of every body, broadphase pairs; queues the pairs that can be in
//                contact and the arenas that have any
//   find ....... queued mesh pairs: the triangles whose boxes and planes the body's box meets
//                (candidates, in walk order)
//   triangles .. one candidate per thread: box-triangle and box-sphere GJK; box-box and plane pairs
//   deep ....... the candidates whose GJK needs the penetration solver
//   combine .... one pair per thread: its candidates' contacts into the manifold, in walk order
//   islands .... bodies whose contacts are all with static objects, one per thread; the arenas
//                with pairs of bodies: contact callbacks, islands, solver (solveIslands)
//   finish ..... integration, post-tick updates, boost pads, goal and tick counters
//
// Between the phases a tick lives in the persistent records (state.h) and in StepTemp.  What
// orders the reference's results is kept: rays of a car see the cars that pre-tick before it
// (higher slots) as those left them and the others as the last tick left them; manifolds,
// callbacks and solver rows follow the pair order of computePairs.  Every operation on a value
// is the one stepArena applies, in the same order, so the results are the same bit for bit.
#pragma once
#include <stddef.h>

#include "engine_core.h"

namespace rsb {

// Words of the body information planes ([word][MAX_BODIES][N]).
enum : int {
    BI_PAIRS = 0,   // static pairs (20 bits) | activation << 20 | BI_* flags
    BI_MANI,        // static pairs that have a manifold (20 bits)
    BI_TASKS,       // meshes with a queued contact pair (16 bits) | planes with a contact << 16
    BI_MESHRES,     // result of the first queued mesh pair (the others follow)
    BI_PLANERES,    // result of the first plane contact (the others follow)
    BI_DYN,         // dynamic pairs in visiting order, 3 bits each, count << 24
    BI_DYNMANI,     // bodies of higher index with which this body has a manifold (7 bits)
    BI_WORDS
};
constexpr int BI_ACT_SHIFT = 20;
constexpr uint32_t BI_ACT_MASK = 7u << BI_ACT_SHIFT;
constexpr uint32_t BI_SOLVED = 1u << 24;    // velocities and transform were written by the islands phase
constexpr uint32_t BI_CACHE = 1u << 25;     // the body's velocity cache holds an impulse
constexpr uint32_t BI_RESPONDS = 1u << 26;  // contact response on (cars)
constexpr uint32_t BI_ALONE = 1u << 27;     // every island of the arena is one body
constexpr uint32_t BI_CONTACT = 1u << 28;   // a contact of the body was found (and its place in bodyQ taken)

// Dynamic pairs (lo < hi) of seven bodies.
constexpr int NUM_DYN_PAIRS = MAX_BODIES * (MAX_BODIES - 1) / 2;
RSB_HD int dynPair(int lo, int hi) { return lo * (2 * MAX_BODIES - lo - 1) / 2 + (hi - lo - 1); }

// Queue counters.
enum : int {
    QC_RAY = 0, QC_BODYRAY, QC_CARMESH, QC_BALLMESH, QC_CARBALL, QC_CARCAR, QC_PLANE, QC_BLOCK, QC_SOLVE, QC_BODY, QC_TRI, QC_DEEP, QC_COMBINE,
    QC_WORDS
};
constexpr int NUM_TASK_TYPES = 4;  // QC_CARMESH .. QC_CARCAR
// The most pairs of each type that an arena can have.
constexpr int CAP_CARMESH = MAX_CARS * MAX_MESHES, CAP_BALLMESH = MAX_MESHES, CAP_CARBALL = MAX_CARS,
              CAP_CARCAR = MAX_CARS * (MAX_CARS - 1) / 2, CAP_PLANE = MAX_BODIES * NUM_PLANES;
constexpr int CAP_RESULTS = CAP_CARMESH + CAP_BALLMESH + CAP_CARBALL + CAP_CARCAR + CAP_PLANE;
RSB_HD int resultBase(int type) {  // per arena: first result of the type
    return type == QC_CARMESH ? 0
         : type == QC_BALLMESH ? CAP_CARMESH
         : type == QC_CARBALL ? CAP_CARMESH + CAP_BALLMESH
         : type == QC_CARCAR ? CAP_CARMESH + CAP_BALLMESH + CAP_CARBALL
                             : CAP_CARMESH + CAP_BALLMESH + CAP_CARBALL + CAP_CARCAR;
}
// ... and the most that can hold contacts in one tick, where a broadphase cell has at most
// `cellStatics` static objects: a body's pairs with static objects are those of one cell.  The point
// pool has a place for each.  Of an arena's manifolds with contacts the first MAX_BLOCKS in dispatch
// order keep them (solveCallbacks, as the one-thread tick), but the points are stored as the pairs
// finish, in any order and side by side with other arenas'.
RSB_HD int contactPairs(int cars, int cellStatics) { return (1 + cars) * cellStatics + cars * (cars + 1) / 2; }

struct PairTask {
    uint32_t a;
    uint16_t o0, o1;
};

// Outcome of one contact pair.
struct PairResult {
    int32_t n;        // points left in the manifold
    uint32_t flags;   // PR_*
    uint32_t block;   // its points (when PR_BLOCK is set)
    float normal[3];  // normal of the last world contact reported to the car
};
enum : uint32_t {
    PR_BLOCK = 1u,  // a contact was added, so the manifold owns a point block
    PR_WORLD = 2u   // ... and the car-world callback saw it
};

// One triangle (tri < 0: the ball) that a queued pair may touch; a pair's candidates lie one
// after another in the order in which the reference visits them.
struct Candidate {
    uint32_t res;   // the pair's place in the task and result arrays
    int32_t tri;
};
// What GJK found for a candidate; between the triangles and the deep phase, its state.
struct CandidateOut {
    uint32_t flags;  // CO_*
    float normal[3], point[3], dist;
};
enum : uint32_t { CO_HAS = 1u, CO_VALID = 2u };
// Candidates per arena that the batch has room for, and per pair.  Pairs with more of them, and
// pairs that find no room left, are taken triangle by triangle on one thread (the deep queue
// holds them as DEEP_PAIR | result).
constexpr int CAP_CANDIDATES = 64, PAIR_CANDIDATES = 32;
constexpr uint32_t DEEP_PAIR = 1u << 31;

struct StepTemp {
    // wheel rays, [4][MAX_CARS][N]: object hit (-1 none), fraction, normal (3 planes)
    int32_t* rayObj;
    float* rayFrac;
    float* rayN;
    uint32_t* info;      // BI_WORDS planes of [MAX_BODIES][N]
    float* force;        // force, torque of the tick: 6 planes of [MAX_BODIES][N]
    float* box;          // broadphase AABB: 6 planes of [MAX_BODIES][N]
    float* cache;        // velocity impulse caches: 3 planes of [MAX_BODIES][N]
    uint32_t* dynRes;    // result of each dynamic pair: [NUM_DYN_PAIRS][N]
    uint32_t* count;     // QC_WORDS counters
    uint32_t* rayQ;      // rays near meshes [4 * MAX_CARS * N], then as many places for the others
    PairTask* tasks;     // per type, [cap * N], at resultBase(type) * N
    PairResult* results;
    MPoint* blocks;      // [blockCap][MAX_POINTS]
    uint32_t blockCap, arenaBlocks;  // places in all, and to an arena
    uint32_t* solveQ;    // arenas with pairs of bodies [N]
    uint32_t* bodyQ;     // bodies with contacts in the others, b * N + a [MAX_BODIES * N]
    uint32_t* first;     // first candidate of each pair and their number << 26, as results
    Candidate* cand;     // [candCap]
    CandidateOut* out;   // [candCap]
    uint32_t candCap;
    uint32_t* deepQ;     // [CAP_RESULTS * N + candCap]
    uint32_t* combineQ;  // [CAP_RESULTS * N]
    uint32_t sms;        // multiprocessors of the device
};

// Static-test counters of one thread (rsb_stats).
struct PhaseStats {
    uint32_t nStatic, nCulled, nMissed, nRows;
};

RSB_HD uint32_t phaseAtomicAdd(uint32_t* p, uint32_t v) {
#if defined(__CUDA_ARCH__)
    return atomicAdd(p, v);
#else
    const uint32_t o = *p;
    *p += v;
    return o;
#endif
}
RSB_HD uint32_t phaseAtomicOr(uint32_t* p, uint32_t v) {
#if defined(__CUDA_ARCH__)
    return atomicOr(p, v);
#else
    const uint32_t o = *p;
    *p |= v;
    return o;
#endif
}
RSB_HD void phaseAtomicAnd(uint32_t* p, uint32_t v) {
#if defined(__CUDA_ARCH__)
    atomicAnd(p, v);
#else
    *p &= v;
#endif
}

#define RSB_PW(T, f) ((int)(offsetof(T, f) / 4))

// ------------------------------------------------------------------ record access

RSB_HD uint32_t ballWord(const EngineView& D, int a, int w) { return D.ball[(size_t)w * D.N + a]; }
RSB_HD uint32_t carWord(const EngineView& D, int a, int s, int w) { return D.car[((size_t)w * MAX_CARS + s) * D.N + a]; }
RSB_HD float carFloat(const EngineView& D, int a, int s, int w) { return u2f(carWord(D, a, s, w)); }
RSB_HD void putCarWord(const EngineView& D, int a, int s, int w, uint32_t v) {
    D.car[((size_t)w * MAX_CARS + s) * D.N + a] = v;
}
RSB_HD void putCarFloat(const EngineView& D, int a, int s, int w, float v) { putCarWord(D, a, s, w, f2u(v)); }
RSB_HD V3 carV3(const EngineView& D, int a, int s, int w) {
    return V3{carFloat(D, a, s, w), carFloat(D, a, s, w + 1), carFloat(D, a, s, w + 2)};
}
RSB_HD void putCarV3(const EngineView& D, int a, int s, int w, V3 v) {
    putCarFloat(D, a, s, w, v.x);
    putCarFloat(D, a, s, w + 1, v.y);
    putCarFloat(D, a, s, w + 2, v.z);
}
RSB_HD uint32_t arenaWord(const EngineView& D, int a, int w) { return D.arena[(size_t)w * D.N + a]; }
RSB_HD uint64_t arenaTickCount(const EngineView& D, int a) {
    return (uint64_t)arenaWord(D, a, RSB_PW(ArenaP, tick)) | ((uint64_t)arenaWord(D, a, RSB_PW(ArenaP, tick) + 1) << 32);
}
RSB_HD uint32_t* arenaStatus(const EngineView& D, int a) { return D.arena + (size_t)RSB_PW(ArenaP, status) * D.N + a; }

// Pose and velocity words lie at the same offsets in the ball and the car records.
static_assert(offsetof(BallP, ang) == offsetof(CarP, ang) && offsetof(BallP, regStamp) == offsetof(CarP, regStamp),
              "common head of the body records");
RSB_HD uint32_t bodyWord(const EngineView& D, int a, int b, int w) {
    return b == 0 ? ballWord(D, a, w) : carWord(D, a, b - 1, w);
}
RSB_HD float bodyFloat(const EngineView& D, int a, int b, int w) { return u2f(bodyWord(D, a, b, w)); }
RSB_HD void putBodyWord(const EngineView& D, int a, int b, int w, uint32_t v) {
    if (b == 0) D.ball[(size_t)w * D.N + a] = v;
    else putCarWord(D, a, b - 1, w, v);
}
RSB_HD V3 bodyV3(const EngineView& D, int a, int b, int w) {
    return V3{bodyFloat(D, a, b, w), bodyFloat(D, a, b, w + 1), bodyFloat(D, a, b, w + 2)};
}
RSB_HD void putBodyV3(const EngineView& D, int a, int b, int w, V3 v) {
    putBodyWord(D, a, b, w, f2u(v.x));
    putBodyWord(D, a, b, w + 1, f2u(v.y));
    putBodyWord(D, a, b, w + 2, f2u(v.z));
}
RSB_HD Xf bodyXf(const EngineView& D, int a, int b) {
    Xf x;
    x.o = bodyV3(D, a, b, RSB_PW(CarP, pos));
    for (int r = 0; r < 3; r++) x.b.r[r] = bodyV3(D, a, b, RSB_PW(CarP, rot) + 3 * r);
    return x;
}
RSB_HD void putBodyXf(const EngineView& D, int a, int b, const Xf& x) {
    putBodyV3(D, a, b, RSB_PW(CarP, pos), x.o);
    for (int r = 0; r < 3; r++) putBodyV3(D, a, b, RSB_PW(CarP, rot) + 3 * r, x.b.r[r]);
}

RSB_HD size_t bodyIdx(const EngineView& D, int a, int b) { return (size_t)b * D.N + a; }
RSB_HD uint32_t& infoWord(const EngineView& D, const StepTemp& T, int a, int b, int w) {
    return T.info[(size_t)w * MAX_BODIES * D.N + bodyIdx(D, a, b)];
}
RSB_HD V3 tempV3(const EngineView& D, const float* p, int a, int b, int k) {
    const size_t st = (size_t)MAX_BODIES * D.N, i = (size_t)k * st + bodyIdx(D, a, b);
    return V3{p[i], p[i + st], p[i + 2 * st]};
}
RSB_HD void putTempV3(const EngineView& D, float* p, int a, int b, int k, V3 v) {
    const size_t st = (size_t)MAX_BODIES * D.N, i = (size_t)k * st + bodyIdx(D, a, b);
    p[i] = v.x;
    p[i + st] = v.y;
    p[i + 2 * st] = v.z;
}

// Constants of a body at transform x (the pose-independent part of loadBall / loadCar).
RSB_HD void bodyConstants(const EngineView& D, int b, Body& o) {
    initBodyCommon(o);
    if (b == 0) {
        o.invMass = D.P.ballInvMass;
        o.grav = D.P.ballGrav;
        o.invIl = D.P.ballInvInertia;
        o.linDampFactor = D.P.ballLinDampFactor;
        o.friction = D.P.ballFriction;
        o.restitution = D.P.ballRestitution;
    } else {
        o.invMass = D.P.car.invMass;
        o.grav = D.P.car.grav;
        o.invIl = D.P.car.invInertiaLocal;
        o.linDampFactor = 1.f;
        o.friction = CAR_COLLISION_FRICTION;
        o.restitution = CAR_COLLISION_RESTITUTION;
    }
}

RSB_HD int arenaBodies(const EngineView& D, int a) { return 1 + 2 * D.teamSize[a]; }
RSB_HD int respawnPick(const EngineView& D, int a, uint64_t tick, int ci) {
    return (int)(mixHash(mixHash(D.seed, (uint32_t)a, 0x5EEDu), (uint32_t)tick, (uint32_t)ci) & 3u);
}
// Whether car s, demoed before the tick, respawns in it.
RSB_HD bool respawns(const EngineView& D, int a, int s) {
    return fmax_(carFloat(D, a, s, RSB_PW(CarP, demoRespawnTimer)) - D.P.dt, 0) == 0;
}
RSB_HD Xf respawnXf(const EngineView& D, int a, int s, uint32_t flags, uint64_t tick) {
    V3 pos;
    M3 rot;
    respawnPlacement((flags & CF_TEAM_ORANGE) ? 1 : 0, respawnPick(D, a, tick, s), pos, rot);
    return Xf{rot, pos * kUuToBt};
}

// A broadphase cell's indices in one word (they are below 256, as every registration is in the
// grid), and whether two cells are neighbours or the same (inRegNeighbourhood).
RSB_HD uint32_t cellWord(int i, int j, int k) { return (uint32_t)i | ((uint32_t)j << 8) | ((uint32_t)k << 16); }
RSB_HD bool cellsNear(uint32_t p, uint32_t q) {
#if defined(__CUDA_ARCH__)
    return (__vabsdiffu4(p, q) & 0x00fefefeu) == 0;
#else
    for (int s = 0; s < 24; s += 8) {
        const int d = (int)((p >> s) & 255u) - (int)((q >> s) & 255u);
        if (d < -1 || d > 1) return false;
    }
    return true;
#endif
}
RSB_HD uint32_t bodyCellWord(const EngineView& D, int a, int b) {
    return cellWord((int)bodyWord(D, a, b, RSB_PW(CarP, ci)), (int)bodyWord(D, a, b, RSB_PW(CarP, cj)),
                    (int)bodyWord(D, a, b, RSB_PW(CarP, ck)));
}

// ------------------------------------------------------------------ wheel rays

// What castRay reads of the world, for the rays of car `viewer`, from the records as the last
// tick left them.  Cars of higher slots have pre-ticked before the viewer's rays are cast: a
// respawning one stands at its spawn, and a demoed one has no contact response.
struct RayBody {
    Xf xf;
    int noResp;
};
struct RayWorld;
struct RayBodies {
    const EngineView* D;
    int a, viewer;
    uint64_t tick;
    RSB_HD RayBody operator[](int b) const {
        RayBody r;
        r.noResp = 0;
        if (b > 0) {
            const int s = b - 1;
            const uint32_t f = carWord(*D, a, s, RSB_PW(CarP, flags));
            if (s > viewer) {
                r.noResp = (f & CF_DEMOED) ? 1 : 0;
                if ((f & CF_DEMOED) && respawns(*D, a, s)) {
                    r.xf = respawnXf(*D, a, s, f, tick);
                    return r;
                }
            } else {
                r.noResp = (f & CF_NO_RESPONSE) ? 1 : 0;
            }
        }
        r.xf = rsb::bodyXf(*D, a, b);
        return r;
    }
};
struct RayWorld {
    const ArenaStatic* S;
    const WorldParams* P;
    RayBodies b;
    int nb;
    uint32_t cull;
    int32_t cullAudit;
    mutable uint32_t nStatic, nCulled, nMissed, cullMissed;
    RegOrder reg;
};

// Registration order of the arena's bodies from their records (buildRegOrder).
template <class StampF, class CellF>
RSB_HD void regOrderOf(RegOrder& R, int nb, StampF&& stamp, CellF&& cell) {
    R.n = 0;
    for (int e = 0; e < nb; e++) {
        const int32_t st = stamp(e);
        int i, j, k;
        cell(e, i, j, k);
        int r = R.n++;
        while (r > 0 && R.stamp[r - 1] > (uint32_t)st) {
            R.body[r] = R.body[r - 1];
            R.stamp[r] = R.stamp[r - 1];
            R.ci[r] = R.ci[r - 1];
            R.cj[r] = R.cj[r - 1];
            R.ck[r] = R.ck[r - 1];
            r--;
        }
        R.body[r] = (int8_t)e;
        R.stamp[r] = (uint32_t)st;
        R.ci[r] = (int16_t)i;
        R.cj[r] = (int16_t)j;
        R.ck[r] = (int16_t)k;
    }
}

RSB_HD size_t rayIdx(const EngineView& D, int a, int s, int w) { return ((size_t)w * MAX_CARS + s) * D.N + a; }
RSB_HD void storeRay(const EngineView& D, const StepTemp& T, size_t r, int obj, float frac, V3 n) {
    T.rayObj[r] = obj;
    if (obj < 0) return;
    const size_t st = (size_t)4 * MAX_CARS * D.N;
    T.rayFrac[r] = frac;
    T.rayN[r] = n.x;
    T.rayN[r + st] = n.y;
    T.rayN[r + 2 * st] = n.z;
}

// The casting car at the start of its pre-tick: false when it stays demoed (casts no rays).
RSB_HD bool rayCar(const EngineView& D, int a, int s, Xf& xf, bool& culled) {
    const uint32_t f = carWord(D, a, s, RSB_PW(CarP, flags));
    culled = D.cull && ((D.cull[a] >> (1 + s)) & 1u);
    if (f & CF_DEMOED) {
        if (!respawns(D, a, s)) return false;
        xf = respawnXf(D, a, s, f, arenaTickCount(D, a));
        culled = false;
    } else {
        xf = bodyXf(D, a, 1 + s);
    }
    return true;
}

// What the ray phase leaves in rayObj of a queued ray: the meshes near it (16 bits), the bodies
// registered around its cell (7 bits), or RAY_ANY for one that castRay takes as a whole.
constexpr int RAY_BODIES_SHIFT = MAX_MESHES;
constexpr uint32_t RAY_ANY = 1u << 30;
enum RayClass : int { RAY_DONE = 0, RAY_MESHES, RAY_BODIES };

// Wheel w of car s: casts the ray if only planes can be near, else says which queue it goes to.
// `near(cell)`: the bodies registered around that cell, the car itself among them.
template <class NearF>
RSB_HD RayClass rayPhase(const EngineView& D, const StepTemp& T, int a, int s, int w, const Xf& xf, bool culled,
                         NearF&& near, PhaseStats& st) {
    const ArenaStatic& S = D.S;
    Body cb;
    WheelTick wt;
    V3 from, to;
    cb.xf = xf;
    wheelSegment(D.P.car, cb, wt, w, from, to);
    const size_t r = rayIdx(D, a, s, w);
    if (culled || !(dist2(from, to) < S.bp.cellSize * S.bp.cellSize)) {
        T.rayObj[r] = (int32_t)RAY_ANY;
        return RAY_BODIES;
    }
    int i, j, k;
    bpCellIndices(S.bp, from, i, j, k);
    uint32_t mask = S.bpCells[i * S.bp.cellsY * S.bp.cellsZ + j * S.bp.cellsZ + k];
    const uint32_t bodies = near(cellWord(i, j, k)), kMeshBits = (1u << MAX_MESHES) - 1u;
    uint32_t meshes = mask & kMeshBits;
    if (meshes) {
        const V3 tolv{kOccTol, kOccTol, kOccTol};
        meshes &= occMask(S, vmin(from, to) - tolv, vmax(from, to) + tolv);
    }
    if (meshes || (bodies & ~(2u << s))) {
        T.rayObj[r] = (int32_t)(meshes | (bodies << RAY_BODIES_SHIFT));
        return meshes ? RAY_MESHES : RAY_BODIES;
    }
    RayHit hit;
    hit.fraction = 1.f;
    hit.obj = -1;
    hit.normal = v3zero();
    for (mask >>= MAX_MESHES; mask; mask &= mask - 1u) {
        if (hit.fraction == 0.f) break;
        st.nStatic++;
        rayVsPlane(S, MAX_MESHES + lowestBit(mask), from, to, hit);
    }
    storeRay(D, T, r, hit.obj, hit.fraction, hit.obj >= 0 ? normalized(hit.normal) : hit.normal);
    return RAY_DONE;
}

// A ray of any kind, by castRay itself: culled bodies, and segments that are longer than a
// broadphase cell or not finite.
RSB_HD_COLD int anyRay(const EngineView& D, int a, int s, bool culled, V3 from, V3 to, V3& hn, float& frac,
                       PhaseStats& st) {
    RayWorld W;
    W.S = &D.S;
    W.P = &D.P;
    W.nb = arenaBodies(D, a);
    W.b.D = &D;
    W.b.a = a;
    W.b.viewer = s;
    W.b.tick = arenaTickCount(D, a);
    W.cull = culled ? 1u << (1 + s) : 0u;
    W.cullAudit = D.cullAudit;
    W.nStatic = W.nCulled = W.nMissed = W.cullMissed = 0;
    regOrderOf(W.reg, W.nb, [&](int e) { return (int32_t)bodyWord(D, a, e, RSB_PW(CarP, regStamp)); },
               [&](int e, int& i, int& j, int& k) {
                   i = (int)bodyWord(D, a, e, RSB_PW(CarP, ci));
                   j = (int)bodyWord(D, a, e, RSB_PW(CarP, cj));
                   k = (int)bodyWord(D, a, e, RSB_PW(CarP, ck));
               });
    V3 hp;
    const int obj = castRay(W, from, to, OBJ_CAR0 + s, hp, hn, frac);
    st.nStatic += W.nStatic;
    st.nCulled += W.nCulled;
    st.nMissed += W.nMissed;
    if (W.cullMissed) phaseAtomicOr(arenaStatus(D, a), W.cullMissed);
    return obj;
}

// Bodies of `cand` in registration order, one call after another: a proxy whose stamp equals
// the one just visited is passed over (the broadphase's rule).  -1 at the end.
struct RegWalk {
    uint32_t cand, last;
    bool first;
    template <class StampF>
    RSB_HD int next(StampF&& stamp) {
        while (cand) {
            int pick = -1;
            uint32_t ps = 0;
            for (uint32_t m = cand; m; m &= m - 1u) {
                const int e = lowestBit(m);
                const uint32_t s = stamp(e);
                if (pick < 0 || s < ps) {
                    pick = e;
                    ps = s;
                }
            }
            cand &= ~(1u << pick);
            if (!first && ps <= last) continue;
            first = false;
            last = ps;
            return pick;
        }
        return -1;
    }
};

// The planes registered in the cell of a ray's start, in their order.
RSB_HD void rayPlanes(const ArenaStatic& S, V3 from, V3 to, RayHit& hit, PhaseStats& st) {
    int i, j, k;
    bpCellIndices(S.bp, from, i, j, k);
    for (uint32_t m = S.bpCells[i * S.bp.cellsY * S.bp.cellsZ + j * S.bp.cellsZ + k] >> MAX_MESHES; m; m &= m - 1u) {
        if (hit.fraction == 0.f) break;
        st.nStatic++;
        rayVsPlane(S, MAX_MESHES + lowestBit(m), from, to, hit);
    }
}
struct RayItem {
    int a, s;
    V3 from, to;
};
RSB_HD bool rayItem(const EngineView& D, uint32_t r, RayItem& o, bool& culled) {
    const int q = (int)(r / (uint32_t)D.N), w = q / MAX_CARS;
    o.a = (int)(r % (uint32_t)D.N);
    o.s = q % MAX_CARS;
    Xf xf;
    if (!rayCar(D, o.a, o.s, xf, culled)) return false;  // never queued
    Body cb;
    WheelTick wt;
    cb.xf = xf;
    wheelSegment(D.P.car, cb, wt, w, o.from, o.to);
    return true;
}

// A queued ray near meshes: these, then the planes.  Returns true when it goes on to the body
// queue: with what was hit so far (RAY_PART), or as a whole.
constexpr uint32_t RAY_PART = 1u << 29;
RSB_HD bool meshRayPhase(const EngineView& D, const StepTemp& T, uint32_t r, PhaseStats& st) {
    RayItem q;
    bool culled;
    if (!rayItem(D, r, q, culled)) return false;
    const uint32_t code = (uint32_t)T.rayObj[r], meshes = code & ((1u << MAX_MESHES) - 1u);
    RayHit hit;
    hit.fraction = 1.f;
    hit.obj = -1;
    hit.normal = v3zero();
    if (!rayVsMeshesNearest(D.S, meshes, q.from, q.to, kOccTol, hit)) {
        T.rayObj[r] = (int32_t)RAY_ANY;
        return true;
    }
    st.nStatic += (uint32_t)bitCount(meshes);
    rayPlanes(D.S, q.from, q.to, hit, st);
    if ((code >> RAY_BODIES_SHIFT) & ~(2u << q.s)) {
        storeRay(D, T, r, 0, hit.fraction, hit.normal);
        T.rayObj[r] = (int32_t)(RAY_PART | (uint32_t)(hit.obj & 31) | (code >> RAY_BODIES_SHIFT << RAY_BODIES_SHIFT));
        return true;
    }
    storeRay(D, T, r, hit.obj, hit.fraction, hit.obj >= 0 ? normalized(hit.normal) : hit.normal);
    return false;
}

// A queued ray near other bodies, these in registration order, as castRay tests them.
RSB_HD void bodyRayPhase(const EngineView& D, const StepTemp& T, uint32_t r, PhaseStats& st) {
    RayItem q;
    bool culled;
    if (!rayItem(D, r, q, culled)) return;
    const uint32_t code = (uint32_t)T.rayObj[r];
    if (code == RAY_ANY) {
        V3 hn = v3zero();
        float frac = 1.f;
        const int obj = anyRay(D, q.a, q.s, culled, q.from, q.to, hn, frac, st);
        storeRay(D, T, r, obj, frac, hn);
        return;
    }
    RayHit hit;
    hit.fraction = 1.f;
    hit.obj = -1;
    hit.normal = v3zero();
    if (code & RAY_PART) {
        const size_t rst = (size_t)4 * MAX_CARS * D.N;
        if ((code & 31u) != 31u) hit.obj = (int)(code & 31u);
        hit.fraction = T.rayFrac[r];
        hit.normal = V3{T.rayN[r], T.rayN[r + rst], T.rayN[r + 2 * rst]};
    } else {
        rayPlanes(D.S, q.from, q.to, hit, st);
    }
    RegWalk walk{(code >> RAY_BODIES_SHIFT) & ((1u << MAX_BODIES) - 1u), 0u, true};
    const RayBodies bodies{&D, q.a, q.s, arenaTickCount(D, q.a)};
    while (true) {
        const int b = walk.next([&](int e) { return bodyWord(D, q.a, e, RSB_PW(CarP, regStamp)); });
        if (b < 0) break;
        if (b == 1 + q.s) continue;
        const Xf bx = bodies[b].xf;
        const ConvexShape sh = b == 0 ? makeSphere(D.P.ballRadius) : carBoxShape(D.P.car);
        float frac;
        V3 n;
        if (subsimplexCast(q.from, q.to, sh, b == 0 ? bx : carChildXf(D.P.car, bx), frac, n) && length2(n) > 0.0001f &&
            frac < hit.fraction) {
            hit.fraction = frac;
            hit.obj = OBJ_BALL + b;
            hit.normal = normalized(n);
        }
    }
    if (hit.obj >= OBJ_BALL && bodies[hit.obj - OBJ_BALL].noResp) hit.obj = -1;
    storeRay(D, T, r, hit.obj, hit.fraction, hit.obj >= 0 ? normalized(hit.normal) : hit.normal);
}

// ------------------------------------------------------------------ bodies

// What the threads of one arena's cars exchange during the drive phase, one column per arena.
constexpr int PHASE_ARENAS = 32;
struct DriveShared {
    float pre[MAX_CARS][6][PHASE_ARENAS];   // linear and angular velocity before the car's pre-tick
    float post[MAX_CARS][6][PHASE_ARENAS];  // ... and after it
    uint32_t done[PHASE_ARENAS];            // cars whose pre-tick is finished
};
// ... and the threads of its bodies during the pairs phase.
struct PairShared {
    float box[MAX_BODIES][6][PHASE_ARENAS];
    uint32_t cell[MAX_BODIES][PHASE_ARENAS];  // cellWord of the registration
    uint32_t stamp[MAX_BODIES][PHASE_ARENAS];
    uint32_t pick[MAX_BODIES][PHASE_ARENAS];  // BI_DYN word of each body
    uint32_t live[MAX_BODIES][PHASE_ARENAS];  // 1: active (objActive)
    uint32_t need[PHASE_ARENAS];              // PN_* sums over the arena's bodies
};

struct OneBody {
    Body v;
    RSB_HD Body& operator[](int) { return v; }
    RSB_HD const Body& operator[](int) const { return v; }
};
struct OneCar {
    CarSim v;
    RSB_HD CarSim& operator[](int) { return v; }
    RSB_HD const CarSim& operator[](int) const { return v; }
};

// One car's view of the world in its pre-tick.
struct CarWorld {
    const ArenaStatic* S;
    const WorldParams* P;
    uint64_t tick;
    uint32_t cull;
    OneBody b;
    OneCar c;
    const EngineView* D;
    const DriveShared* sh;
    int a, la, ci;
};

// A dynamic ground object of a wheel: cars of higher slots have finished their pre-tick.
RSB_HD GroundRef groundRef(const CarWorld& W, int o) {
    GroundRef g;
    g.body = nullptr;
    if (o < OBJ_BALL) {
        g.com = o < MAX_MESHES ? v3zero() : W.S->planeOrigin[o - MAX_MESHES];
        g.lin = g.ang = v3zero();
        g.basis = m3identity();
        g.invInertiaLocal = v3zero();
        g.invMass = 0.f;
        return g;
    }
    const int b = o - OBJ_BALL;
    const Xf x = bodyXf(*W.D, W.a, b);
    g.com = x.o;
    g.basis = x.b;
    if (b == 0) {
        g.lin = bodyV3(*W.D, W.a, 0, RSB_PW(BallP, lin));
        g.ang = bodyV3(*W.D, W.a, 0, RSB_PW(BallP, ang));
        g.invInertiaLocal = W.P->ballInvInertia;
        g.invMass = W.P->ballInvMass;
    } else {
        const float(*v)[PHASE_ARENAS] = (b - 1 > W.ci) ? W.sh->post[b - 1] : W.sh->pre[b - 1];
        g.lin = V3{v[0][W.la], v[1][W.la], v[2][W.la]};
        g.ang = V3{v[3][W.la], v[4][W.la], v[5][W.la]};
        g.invInertiaLocal = W.P->car.invInertiaLocal;
        g.invMass = W.P->car.invMass;
    }
    return g;
}

// Sums over an arena's bodies: pairs that can be in contact (8 bits), static pairs (8 bits), and
// whether any pair of bodies exists.  Without such pairs every island is one body, solved by
// itself, unless the arena's contacts might not fit its pools, whose limits run over all bodies.
constexpr uint32_t PN_PAIR = 1u << 8, PN_DYN = 1u << 24;
constexpr int BODY_MAX_TASKS = 14;  // MAX_BLOCKS blocks, and MAX_CONTACT_ROWS rows with the special rows
RSB_HD bool arenaHasContacts(uint32_t need) { return (need & 255u) != 0 || need >= PN_DYN; }
RSB_HD bool arenaByBodies(uint32_t need) {
    return need < PN_DYN && (need & 255u) <= (uint32_t)BODY_MAX_TASKS && ((need >> 8) & 255u) <= (uint32_t)MAX_PAIRS;
}

// One car's thread of the drive phase.
struct DriveThread {
    int a, la, s;
    bool live;          // the vehicle update runs (the car is not demoed)
    bool respawned, finished;
    uint32_t deps;      // cars whose finished pre-tick this one waits for
    CarWorld W;
};

RSB_HD void publishVel(float (*v)[PHASE_ARENAS], int la, const Body& b) {
    v[0][la] = b.lin.x; v[1][la] = b.lin.y; v[2][la] = b.lin.z;
    v[3][la] = b.ang.x; v[4][la] = b.ang.y; v[5][la] = b.ang.z;
}

// Loads the car, runs its status update and takes up its rays' results.  Nothing is written to
// the records before every thread of the arena has published what others read.
RSB_HD void driveLoad(const EngineView& D, const StepTemp& T, DriveThread& t, DriveShared& sh) {
    CarWorld& W = t.W;
    Body& b = W.b.v;
    CarSim& c = W.c.v;
    const int a = t.a, s = t.s;
    W.S = &D.S;
    W.P = &D.P;
    W.D = &D;
    W.sh = &sh;
    W.a = a;
    W.la = t.la;
    W.ci = s;
    W.tick = arenaTickCount(D, a);
    W.cull = 0;
    t.deps = 0;
    bodyConstants(D, 1 + s, b);
    b.xf = bodyXf(D, a, 1 + s);
    b.lin = bodyV3(D, a, 1 + s, RSB_PW(CarP, lin));
    b.ang = bodyV3(D, a, 1 + s, RSB_PW(CarP, ang));
    updateInertia(b);
    publishVel(sh.pre[s], t.la, b);
    c.flags = carWord(D, a, s, RSB_PW(CarP, flags));
    c.team = (c.flags & CF_TEAM_ORANGE) ? 1 : 0;
    c.id = (uint32_t)s + 1u;
    c.boost = carFloat(D, a, s, RSB_PW(CarP, boost));
    c.timeSpentBoosting = carFloat(D, a, s, RSB_PW(CarP, timeSpentBoosting));
    c.jumpTime = carFloat(D, a, s, RSB_PW(CarP, jumpTime));
    c.flipTime = carFloat(D, a, s, RSB_PW(CarP, flipTime));
    c.airTime = carFloat(D, a, s, RSB_PW(CarP, airTime));
    c.airTimeSinceJump = carFloat(D, a, s, RSB_PW(CarP, airTimeSinceJump));
    c.handbrakeVal = carFloat(D, a, s, RSB_PW(CarP, handbrakeVal));
    c.autoFlipTimer = carFloat(D, a, s, RSB_PW(CarP, autoFlipTimer));
    c.autoFlipTorqueScale = carFloat(D, a, s, RSB_PW(CarP, autoFlipTorqueScale));
    c.demoRespawnTimer = carFloat(D, a, s, RSB_PW(CarP, demoRespawnTimer));
    c.flipRelTorque = carV3(D, a, s, RSB_PW(CarP, flipRelTorque));
    c.worldContactNormal = carV3(D, a, s, RSB_PW(CarP, worldContactNormal));
#pragma unroll
    for (int r = 0; r < 3; r++) c.rotMat.r[r] = carV3(D, a, s, RSB_PW(CarP, rotMat) + 3 * r);
    c.lastCtlBits = carWord(D, a, s, RSB_PW(CarP, lastCtlBits));
    c.steerAngle = carFloat(D, a, s, RSB_PW(CarP, steerAngle));
    c.engineForce = carFloat(D, a, s, RSB_PW(CarP, engineForce));
    c.brake = carFloat(D, a, s, RSB_PW(CarP, brake));
#pragma unroll
    for (int i = 0; i < 4; i++) {
        c.latF[i] = carFloat(D, a, s, RSB_PW(CarP, latFriction) + i);
        c.longF[i] = carFloat(D, a, s, RSB_PW(CarP, longFriction) + i);
        c.extraPush[i] = carFloat(D, a, s, RSB_PW(CarP, extraPushback) + i);
    }
    const CtlRec& ctl = D.controls[D.carOffset[a] + s];
#pragma unroll
    for (int k = 0; k < 5; k++) c.ctl[k] = ctl.v[k];
    c.ctlBits = (ctl.jump ? 1u : 0u) | (ctl.boost ? 2u : 0u) | (ctl.handbrake ? 4u : 0u);
    const bool wasDemoed = (c.flags & CF_DEMOED) != 0;
    t.live = carPreTickStatus(W, s, mixHash(mixHash(D.seed, (uint32_t)a, 0x5EEDu), (uint32_t)W.tick, (uint32_t)s));
    t.respawned = wasDemoed && t.live;
    t.finished = !t.live;
    if (t.finished) publishVel(sh.post[s], t.la, b);
    if (t.respawned && D.cull) phaseAtomicAnd(const_cast<uint32_t*>(D.cull) + a, ~(2u << s));
    if (!t.live) return;
    // wheels: the steering basis (the same for both wheels of an axle) and the rays' results
    wheelTransform(D.P.car, b, c.w[0], 0, c.steerAngle);
    wheelTransform(D.P.car, b, c.w[2], 2, 0.f);
    c.w[1].basis = c.w[0].basis;
    c.w[3].basis = c.w[2].basis;
    const size_t rst = (size_t)4 * MAX_CARS * D.N;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        V3 from, to, hp = v3zero(), hn = v3zero();
        wheelSegment(D.P.car, b, c.w[i], i, from, to);
        const size_t r = rayIdx(D, a, s, i);
        const int obj = T.rayObj[r];
        if (obj >= 0) {
            const float f = T.rayFrac[r], f1 = 1.f - f;
            hp = from * f1 + to * f;
            hn = V3{T.rayN[r], T.rayN[r + rst], T.rayN[r + 2 * rst]};
            if (obj > OBJ_CAR0 + s) t.deps |= 1u << (obj - OBJ_CAR0);
        }
        wheelFromHit(W, s, i, to, obj, hp, hn);
    }
}

// The vehicle update, once the cars it stands on have finished theirs.
RSB_HD void driveRun(DriveThread& t, DriveShared& sh) {
    carDrive(t.W, t.s);
    publishVel(sh.post[t.s], t.la, t.W.b.v);
    t.finished = true;
}

// Gravity; writes the record.
RSB_HD void driveStore(const EngineView& D, const StepTemp& T, DriveThread& t) {
    Body& b = t.W.b.v;
    const CarSim& c = t.W.c.v;
    const int a = t.a, s = t.s;
    if (b.act != ACT_SLEEPING && b.act != ACT_DISABLE_SIM) b.force = b.force + b.grav;
    putTempV3(D, T.force, a, 1 + s, 0, b.force);
    putTempV3(D, T.force, a, 1 + s, 3, b.torque);
    putCarWord(D, a, s, RSB_PW(CarP, flags), (c.flags & ~CF_NO_RESPONSE) | (b.noResp ? CF_NO_RESPONSE : 0u));
    putCarFloat(D, a, s, RSB_PW(CarP, demoRespawnTimer), c.demoRespawnTimer);
    if (!t.live) return;
    putBodyV3(D, a, 1 + s, RSB_PW(CarP, lin), b.lin);
    putBodyV3(D, a, 1 + s, RSB_PW(CarP, ang), b.ang);
    putCarFloat(D, a, s, RSB_PW(CarP, boost), c.boost);
    putCarFloat(D, a, s, RSB_PW(CarP, timeSpentBoosting), c.timeSpentBoosting);
    putCarFloat(D, a, s, RSB_PW(CarP, jumpTime), c.jumpTime);
    putCarFloat(D, a, s, RSB_PW(CarP, flipTime), c.flipTime);
    putCarFloat(D, a, s, RSB_PW(CarP, airTime), c.airTime);
    putCarFloat(D, a, s, RSB_PW(CarP, airTimeSinceJump), c.airTimeSinceJump);
    putCarFloat(D, a, s, RSB_PW(CarP, handbrakeVal), c.handbrakeVal);
    putCarFloat(D, a, s, RSB_PW(CarP, autoFlipTimer), c.autoFlipTimer);
    putCarFloat(D, a, s, RSB_PW(CarP, autoFlipTorqueScale), c.autoFlipTorqueScale);
    putCarV3(D, a, s, RSB_PW(CarP, flipRelTorque), c.flipRelTorque);
    putCarFloat(D, a, s, RSB_PW(CarP, steerAngle), c.steerAngle);
    putCarFloat(D, a, s, RSB_PW(CarP, engineForce), c.engineForce);
    putCarFloat(D, a, s, RSB_PW(CarP, brake), c.brake);
#pragma unroll
    for (int i = 0; i < 4; i++) {
        putCarFloat(D, a, s, RSB_PW(CarP, latFriction) + i, c.latF[i]);
        putCarFloat(D, a, s, RSB_PW(CarP, longFriction) + i, c.longF[i]);
        putCarFloat(D, a, s, RSB_PW(CarP, extraPushback) + i, c.extraPush[i]);
    }
    if (!t.respawned) return;
    // Car::SetState of the spawn: the rest of the record
    putBodyXf(D, a, 1 + s, b.xf);
    putCarFloat(D, a, s, RSB_PW(CarP, supersonicTime), 0.f);
    putCarFloat(D, a, s, RSB_PW(CarP, carContactCooldown), 0.f);
    putCarV3(D, a, s, RSB_PW(CarP, worldContactNormal), v3zero());
    putCarWord(D, a, s, RSB_PW(CarP, carContactOtherId), 0u);
    for (int k = 0; k < 2; k++) {
        putCarWord(D, a, s, RSB_PW(CarP, ballHitTick) + k, ~0u);
        putCarWord(D, a, s, RSB_PW(CarP, ballHitExtraTick) + k, ~0u);
    }
    putCarV3(D, a, s, RSB_PW(CarP, ballHitRelPos), v3zero());
    putCarV3(D, a, s, RSB_PW(CarP, ballHitBallPos), v3zero());
    putCarV3(D, a, s, RSB_PW(CarP, ballHitExtraVel), v3zero());
    for (int r = 0; r < 3; r++) putCarV3(D, a, s, RSB_PW(CarP, rotMat) + 3 * r, c.rotMat.r[r]);
}

// One body's thread of the pairs phase.
struct PairThread {
    int a, la, b, nb;   // b < nb when there is such a body
    uint32_t dyn;       // BI_DYN word
    OneBody body;
};
// The body as updateBodyAabb sees it.
struct BoxWorld {
    const ArenaStatic* S;
    const WorldParams* P;
    int nb;
    uint32_t stampBase, status;
    OneBody& b;
};

// Predicted motion, broadphase box and registration.
RSB_HD void pairLoad(const EngineView& D, const StepTemp& T, PairThread& t, PairShared& sh, bool firstTick) {
    Body& b = t.body.v;
    const int a = t.a, la = t.la;
    const float dt = D.P.dt;
    bodyConstants(D, t.b, b);
    b.xf = bodyXf(D, a, t.b);
    b.lin = bodyV3(D, a, t.b, RSB_PW(CarP, lin));
    b.ang = bodyV3(D, a, t.b, RSB_PW(CarP, ang));
    b.cell = (int32_t)bodyWord(D, a, t.b, RSB_PW(CarP, cell));
    b.ci = (int32_t)bodyWord(D, a, t.b, RSB_PW(CarP, ci));
    b.cj = (int32_t)bodyWord(D, a, t.b, RSB_PW(CarP, cj));
    b.ck = (int32_t)bodyWord(D, a, t.b, RSB_PW(CarP, ck));
    b.regStamp = (int32_t)bodyWord(D, a, t.b, RSB_PW(CarP, regStamp));
    if (t.b == 0) {
        // ball zero-velocity sleeping (Arena.cpp:721-727)
        b.act = (length2(b.lin) == 0.f && length2(b.ang) == 0.f) ? ACT_SLEEPING : ACT_ACTIVE;
        if (b.act != ACT_SLEEPING) b.force = b.force + b.grav;
        putTempV3(D, T.force, a, 0, 0, b.force);
        putTempV3(D, T.force, a, 0, 3, b.torque);
        b.lin = b.lin * b.linDampFactor;
        putBodyV3(D, a, 0, RSB_PW(BallP, lin), b.lin);
        b.ixf = integrateTransformNoRot(b.xf, b.lin, dt);
    } else {
        // a car without contact response is out of the simulation, and no other is
        b.noResp = carWord(D, a, t.b - 1, RSB_PW(CarP, flags)) & CF_NO_RESPONSE ? 1 : 0;
        b.act = b.noResp ? ACT_DISABLE_SIM : ACT_ACTIVE;
        b.ixf = integrateTransform(b.xf, b.lin, b.ang, dt);
    }
    // the box of the last tick stays when this one's is not finite
    b.bpMin = b.bpMax = b.xf.o;
    const int32_t cell0 = b.cell, stamp0 = b.regStamp;
    BoxWorld M{&D.S, &D.P, t.nb, (uint32_t)((arenaTickCount(D, a) + 1) * 8u), 0u, t.body};
    updateBodyAabb(M, t.b);
    if (M.status) {
        phaseAtomicOr(arenaStatus(D, a), M.status);
        if (!firstTick) {
            b.bpMin = tempV3(D, T.box, a, t.b, 0);
            b.bpMax = tempV3(D, T.box, a, t.b, 3);
        }
    }
    putTempV3(D, T.box, a, t.b, 0, b.bpMin);
    putTempV3(D, T.box, a, t.b, 3, b.bpMax);
    const float bx[6] = {b.bpMin.x, b.bpMin.y, b.bpMin.z, b.bpMax.x, b.bpMax.y, b.bpMax.z};
#pragma unroll
    for (int k = 0; k < 6; k++) sh.box[t.b][k][la] = bx[k];
    sh.cell[t.b][la] = cellWord(b.ci, b.cj, b.ck);
    sh.stamp[t.b][la] = (uint32_t)b.regStamp;
    sh.live[t.b][la] = (b.act != ACT_SLEEPING && b.act != ACT_DISABLE_SIM) ? 1u : 0u;
    if (b.cell != cell0) putBodyWord(D, a, t.b, RSB_PW(CarP, cell), (uint32_t)b.cell);
    if (b.regStamp != stamp0) {
        putBodyWord(D, a, t.b, RSB_PW(CarP, ci), (uint32_t)b.ci);
        putBodyWord(D, a, t.b, RSB_PW(CarP, cj), (uint32_t)b.cj);
        putBodyWord(D, a, t.b, RSB_PW(CarP, ck), (uint32_t)b.ck);
        putBodyWord(D, a, t.b, RSB_PW(CarP, regStamp), (uint32_t)b.regStamp);
    }
}

RSB_HD V3 sharedV3(const float (*v)[PHASE_ARENAS], int k, int la) { return V3{v[k][la], v[k + 1][la], v[k + 2][la]}; }

// The dynamic pairs of this body in visiting order (the second half of computePairs).
RSB_HD void pairPick(const EngineView& D, PairThread& t, PairShared& sh) {
    const Body& b = t.body.v;
    const BpGrid& g = D.S.bp;
    const int la = t.la;
    t.dyn = 0;
    if (t.nb > 1) {
        const uint32_t own = cellWord(b.cell / (g.cellsY * g.cellsZ), (b.cell / g.cellsZ) % g.cellsY, b.cell % g.cellsZ);
        uint32_t cand = 0, n = 0;
        for (int e = 0; e < t.nb; e++) cand |= cellsNear(own, sh.cell[e][la]) ? 1u << e : 0u;
        if (cand & (cand - 1u)) {
            RegWalk walk{cand, 0u, true};
            while (true) {
                const int e = walk.next([&](int x) { return sh.stamp[x][la]; });
                if (e < 0) break;
                if (e != t.b && aabbOverlap(b.bpMin, b.bpMax, sharedV3(sh.box[e], 0, la), sharedV3(sh.box[e], 3, la)))
                    t.dyn |= (uint32_t)e << (3 * n++);
            }
            t.dyn |= n << 24;
        }
    }
    sh.pick[t.b][la] = t.dyn;
}

// Contact world of one pair: at most two bodies.
struct LocalPool {
    int32_t n;
    uint32_t* status;  // only written when more than MAX_BLOCKS manifolds share the pool; one does here
    MPoint pts[MAX_POINTS];
};
struct PairBodies {
    Body v0, v1;
    int i0;
    RSB_HD Body& operator[](int i) { return i == i0 ? v0 : v1; }
    RSB_HD const Body& operator[](int i) const { return i == i0 ? v0 : v1; }
};
template <class BodiesT>
struct PairWorldT {
    const ArenaStatic* S;
    const WorldParams* P;
    BodiesT b;
    OneCar c;
    LocalPool* pool;  // apart, so that the points' indexing leaves the rest in registers
    uint32_t status;
    EpaWork* epa;
    uint32_t cull;
    int32_t cullAudit;
    mutable uint32_t nStatic, nCulled, nMissed, cullMissed;
};
template <class BodiesT>
RSB_HD LocalPool& poolOf(PairWorldT<BodiesT>& W) { return *W.pool; }
template <class WT>
RSB_HD void pairWorldInit(const EngineView& D, WT& W, LocalPool& pool, EpaWork* epa, uint32_t cull) {
    W.S = &D.S;
    W.P = &D.P;
    W.pool = &pool;
    pool.n = 0;
    pool.status = 0;
    W.status = 0;
    W.epa = epa;
    W.cull = cull;
    W.cullAudit = D.cullAudit;
    W.nStatic = W.nCulled = W.nMissed = W.cullMissed = 0;
    W.c.v.flags = 0;
    W.c.v.worldContactNormal = v3zero();
}
RSB_HD void pairManifold(Manifold& m, int o0, int o1, float cbt) {
    m.o0 = o0;
    m.o1 = o1;
    m.cbt = cbt;
    m.n = 0;
    m.pt = nullptr;
}
template <class WT>
RSB_HD void storePair(const EngineView& D, const StepTemp& T, int a, WT& W, const Manifold& m, uint32_t res) {
    PairResult r;
    r.n = m.n;
    r.flags = (m.pt ? PR_BLOCK : 0u) | ((W.c.v.flags & CF_WORLD_CONTACT) ? PR_WORLD : 0u);
    r.block = 0;
    r.normal[0] = W.c.v.worldContactNormal.x;
    r.normal[1] = W.c.v.worldContactNormal.y;
    r.normal[2] = W.c.v.worldContactNormal.z;
    if (m.n > 0) {
        r.block = phaseAtomicAdd(&T.count[QC_BLOCK], 1u);
        if (r.block < T.blockCap) {
            MPoint* dst = T.blocks + (size_t)MAX_POINTS * r.block;
            for (int k = 0; k < m.n; k++) dst[k] = m.pt[k];
        } else {
            r.n = 0;  // out of range: the pool has a place for every pair
            r.block = r.flags = 0;
            W.status |= WS_OVERFLOW;
        }
    }
    T.results[res] = r;
    if (W.status | W.cullMissed) phaseAtomicOr(arenaStatus(D, a), W.status | W.cullMissed);
    // the first contact of a body that is an island by itself queues the body
    const int b = imax_(m.o0, m.o1) - OBJ_BALL;
    if (r.flags && !(infoWord(D, T, a, b, BI_PAIRS) & BI_CONTACT) && (infoWord(D, T, a, b, BI_PAIRS) & BI_ALONE) &&
        !(phaseAtomicOr(&infoWord(D, T, a, b, BI_PAIRS), BI_CONTACT) & BI_CONTACT))
        T.bodyQ[phaseAtomicAdd(&T.count[QC_BODY], 1u)] = (uint32_t)bodyIdx(D, a, b);
}

// Static pairs: all of them, those with a manifold, and those that can be in contact (the
// caller allocates the queue places of these, and pairStore fills them).
struct BodyStatics {
    uint32_t pairs, mani, meshes, planes;
};
RSB_HD BodyStatics pairStatics(const EngineView& D, PairThread& t, PhaseStats& st) {
    BodyStatics o;
    o.pairs = o.mani = o.meshes = o.planes = 0;
    const ArenaStatic& S = D.S;
    const Body& b = t.body.v;
    const CarParams& C = D.P.car;
    const bool active = b.act != ACT_SLEEPING && b.act != ACT_DISABLE_SIM;
    const bool culled = D.cull && ((D.cull[t.a] >> t.b) & 1u);
    // the box the narrowphase tests: the ball's, or the hitbox at its place in the car
    const Xf childXf = t.b == 0 ? b.xf : carChildXf(C, b.xf);
    V3 bmn, bmx;
    if (t.b == 0) ballAabb(D.P, b.xf, bmn, bmx);
    else carBoxAabb(C, childXf, bmn, bmx);
    uint32_t occ = 0;
    bool occKnown = false;
    for (uint32_t mask = S.bpCells[b.cell]; mask; mask &= mask - 1u) {
        const int s = lowestBit(mask);
        V3 smn, smx;
        if (s < MAX_MESHES) { smn = S.meshes[s].bpMin; smx = S.meshes[s].bpMax; }
        else { smn = S.planeBpMin[s - MAX_MESHES]; smx = S.planeBpMax[s - MAX_MESHES]; }
        if (!aabbOverlap(b.bpMin, b.bpMax, smn, smx)) continue;
        o.pairs |= 1u << s;
        if (!active) continue;
        if (t.b != 0) {
            if (s < MAX_MESHES) { smn = S.meshes[s].shapeMin; smx = S.meshes[s].shapeMax; }
            else { smn = S.planeShapeMin[s - MAX_MESHES]; smx = S.planeShapeMax[s - MAX_MESHES]; }
            if (!aabbOverlap(bmn, bmx, smn, smx)) continue;  // its manifold is released again
        }
        o.mani |= 1u << s;
        // cullSkip's bookkeeping, then the rejects of the tests themselves
        if (culled) {
            st.nCulled++;
            if (!D.cullAudit) continue;
        }
        st.nStatic++;
        if (s < MAX_MESHES) {
            if (!occKnown) {
                const V3 tolv{kOccTol, kOccTol, kOccTol};
                occ = occMask(S, bmn - tolv, bmx + tolv);
                occKnown = true;
            }
            if ((occ >> s) & 1u) o.meshes |= 1u << s;
        } else {
            V3 vip;
            const bool near = t.b == 0 ? ballPlaneDistance(S, D.P, s, b.xf, vip) < D.P.ballCbt + 0.f
                                       : boxPlaneDistance(S, C, s, childXf, vip) < C.cbt + 0.f;
            if (near) o.planes |= 1u << (s - MAX_MESHES);
        }
    }
    return o;
}

// The dynamic pairs (b, hi > b) that have a manifold: bit hi.
RSB_HD uint32_t pairDynamics(const EngineView& D, const PairThread& t, const PairShared& sh) {
    const CarParams& C = D.P.car;
    const Body& b = t.body.v;
    uint32_t m = 0;
    auto picked = [&](int x, int y) {
        const uint32_t d = sh.pick[x][t.la];
        for (uint32_t k = 0; k < (d >> 24); k++)
            if (((d >> (3 * k)) & 7u) == (uint32_t)y) return true;
        return false;
    };
    for (int hi = t.b + 1; hi < t.nb; hi++) {
        if (!picked(t.b, hi) && !picked(hi, t.b)) continue;
        if (!sh.live[t.b][t.la] && !sh.live[hi][t.la]) continue;
        const Xf hx = bodyXf(D, t.a, hi);
        V3 mn, mx, mn2, mx2;
        if (t.b == 0) {
            carBoxAabb(C, carChildXf(C, hx), mn, mx);
            ballAabb(D.P, b.xf, mn2, mx2);
            if (aabbOverlap(mn, mx, mn2, mx2)) m |= 1u << hi;
        } else {
            // car a = lower slot, car b = higher slot (collideCarCar)
            carBoxAabb(C, carChildXf(C, b.xf), mn, mx);
            carCompoundAabb(C, hx, mn2, mx2);
            if (!aabbOverlap(mn, mx, mn2, mx2)) continue;
            carBoxAabb(C, carChildXf(C, hx), mn2, mx2);
            if (aabbOverlap(mn2, mx2, mn, mx)) m |= 1u << hi;
        }
    }
    return m;
}

// Stores the body's pair information and fills its queue places: `mesh0` the first of its mesh
// pairs in their queue, `plane0` of its plane contacts, `dyn0` of its dynamic pairs.
RSB_HD void pairStore(const EngineView& D, const StepTemp& T, const PairThread& t, const BodyStatics& o,
                      uint32_t dynMani, uint32_t mesh0, uint32_t plane0, uint32_t dyn0) {
    const int a = t.a;
    const Body& b = t.body.v;
    const int meshType = t.b == 0 ? QC_BALLMESH : QC_CARMESH, dynType = t.b == 0 ? QC_CARBALL : QC_CARCAR;
    infoWord(D, T, a, t.b, BI_DYN) = t.dyn;
    if (o.pairs | t.dyn | dynMani) {
        infoWord(D, T, a, t.b, BI_MANI) = o.mani;
        infoWord(D, T, a, t.b, BI_TASKS) = o.meshes | (o.planes << 16);
        infoWord(D, T, a, t.b, BI_DYNMANI) = dynMani;
    }
    uint32_t k = (uint32_t)resultBase(meshType) * (uint32_t)D.N + mesh0;
    if (o.meshes) infoWord(D, T, a, t.b, BI_MESHRES) = k;
    for (uint32_t m = o.meshes; m; m &= m - 1u, k++)
        T.tasks[k] = PairTask{(uint32_t)a, (uint16_t)lowestBit(m), (uint16_t)(OBJ_BALL + t.b)};
    k = (uint32_t)resultBase(QC_PLANE) * (uint32_t)D.N + plane0;
    if (o.planes) infoWord(D, T, a, t.b, BI_PLANERES) = k;
    for (uint32_t m = o.planes; m; m &= m - 1u, k++)
        T.tasks[k] = PairTask{(uint32_t)a, (uint16_t)(MAX_MESHES + lowestBit(m)), (uint16_t)(OBJ_BALL + t.b)};
    k = (uint32_t)resultBase(dynType) * (uint32_t)D.N + dyn0;
    for (uint32_t m = dynMani; m; m &= m - 1u, k++) {
        const int hi = lowestBit(m);
        T.tasks[k] = PairTask{(uint32_t)a, (uint16_t)(OBJ_BALL + t.b), (uint16_t)(OBJ_BALL + hi)};
        T.dynRes[(size_t)dynPair(t.b, hi) * D.N + a] = k;
    }
}

// The body's first word, once the sums over the arena's bodies are known.
RSB_HD void pairStoreHead(const EngineView& D, const StepTemp& T, const PairThread& t, const BodyStatics& o,
                          uint32_t need) {
    const Body& b = t.body.v;
    infoWord(D, T, t.a, t.b, BI_PAIRS) = o.pairs | ((uint32_t)b.act << BI_ACT_SHIFT) | (b.noResp ? 0u : BI_RESPONDS) |
                                         (arenaByBodies(need) ? BI_ALONE : 0u);
}

RSB_HD void pairNeed(const PairThread& t, const BodyStatics& o, PairShared& sh) {
    const uint32_t v = (uint32_t)bitCount(o.meshes) + (uint32_t)bitCount(o.planes) +
                       PN_PAIR * (uint32_t)bitCount(o.pairs) + (t.dyn ? PN_DYN : 0u);
    if (v) phaseAtomicAdd(&sh.need[t.la], v);
}

// ------------------------------------------------------------------ contacts

RSB_HD void pairBody(const EngineView& D, int a, int b, Body& o) {
    bodyConstants(D, b, o);
    o.xf = bodyXf(D, a, b);
    o.noResp = b > 0 && (carWord(D, a, b - 1, RSB_PW(CarP, flags)) & CF_NO_RESPONSE) ? 1 : 0;
}

// A whole mesh pair on one thread; `res` is its place in the task and result arrays.
RSB_HD void carMeshPhase(const EngineView& D, const StepTemp& T, uint32_t res, EpaWork* epa, PhaseStats& st) {
    const PairTask k = T.tasks[res];
    const int a = (int)k.a, b = k.o1 - OBJ_BALL;
    PairWorldT<OneBody> W;
    LocalPool pool;
    pairWorldInit(D, W, pool, epa, D.cull ? (D.cull[a] & (1u << b)) : 0u);
    pairBody(D, a, b, W.b.v);
    Manifold m;
    pairManifold(m, k.o1, k.o0, D.P.car.cbt);
    collideBoxMesh(W, k.o0, b - 1, carChildXf(D.P.car, W.b.v.xf), m);
    st.nMissed += W.nMissed;
    storePair(D, T, a, W, m, res);
}
RSB_HD void ballMeshPhase(const EngineView& D, const StepTemp& T, uint32_t res, PhaseStats& st) {
    const PairTask k = T.tasks[res];
    const int a = (int)k.a;
    PairWorldT<OneBody> W;
    LocalPool pool;
    pairWorldInit(D, W, pool, nullptr, D.cull ? (D.cull[a] & 1u) : 0u);
    pairBody(D, a, 0, W.b.v);
    Manifold m;
    pairManifold(m, OBJ_BALL, k.o0, D.P.ballCbt);
    collideBallMesh(W, k.o0, m);
    st.nMissed += W.nMissed;
    storePair(D, T, a, W, m, res);
}

// What a mesh pair's body tests triangles with.
struct FindBody {
    Xf xf;      // the ball's transform, the hitbox's otherwise
    M3 invB;
    V3 amn, amx;
    bool ball;
};
RSB_HD void findBody(const EngineView& D, int a, int b, FindBody& f) {
    f.ball = b == 0;
    f.xf = bodyXf(D, a, b);
    if (f.ball) {
        ballAabb(D.P, f.xf, f.amn, f.amx);
    } else {
        f.xf = carChildXf(D.P.car, f.xf);
        carBoxAabb(D.P.car, f.xf, f.amn, f.amx);
    }
    f.invB = inverse(f.xf.b);
}
RSB_HD bool findTest(const EngineView& D, const FindBody& f, const TriData& t) {
    if (!triBoxOverlap(t, f.amn, f.amx)) return false;
    return f.ball ? ballTriPlanes(D.P, f.xf, f.invB, D.P.ballCbt, t.unit, t.unitDist)
                  : boxTriPlanes(carBoxShape(D.P.car), f.xf, f.invB, D.P.car.cbt, t.unit, t.unitDist);
}
// A pair whose n candidates begin at `first`: nothing to combine, too many, or to combine (the
// return value; the caller queues the pair).
constexpr int CANDIDATE_SHIFT = 26;
RSB_HD bool findStore(const StepTemp& T, uint32_t res, uint32_t first, uint32_t n) {
    if (n == 0) {
        T.results[res] = PairResult{0, 0u, 0u, {0.f, 0.f, 0.f}};
        return false;
    }
    if (n > (uint32_t)PAIR_CANDIDATES || first + n > T.candCap || first >= (1u << CANDIDATE_SHIFT)) {
        T.deepQ[phaseAtomicAdd(&T.count[QC_DEEP], 1u)] = DEEP_PAIR | res;
        return false;
    }
    T.first[res] = first | (n << CANDIDATE_SHIFT);
    return true;
}
RSB_HD void putCandidate(const StepTemp& T, uint32_t at, uint32_t res, int tri) {
    if (at < T.candCap) T.cand[at] = Candidate{res, tri};
}

// A pair on one thread.
RSB_HD void findPhase(const EngineView& D, const StepTemp& T, uint32_t res) {
    const PairTask k = T.tasks[res];
    uint32_t n = 0, first = 0;
    if (k.o0 == OBJ_BALL) {
        first = phaseAtomicAdd(&T.count[QC_TRI], 1u);
        n = 1;
        putCandidate(T, first, res, -1);
    } else {
        int16_t tri[PAIR_CANDIDATES];
        FindBody f;
        findBody(D, (int)k.a, k.o1 - OBJ_BALL, f);
        bvhQueryLeaves(D.S, k.o0, f.amn, f.amx, [&](int t) {
            if (!findTest(D, f, triData(D.S, k.o0, t))) return true;
            if (n < (uint32_t)PAIR_CANDIDATES) tri[n] = (int16_t)t;
            return ++n <= (uint32_t)PAIR_CANDIDATES;
        });
        if (n > 0 && n <= (uint32_t)PAIR_CANDIDATES) {
            first = phaseAtomicAdd(&T.count[QC_TRI], n);
            for (uint32_t i = 0; i < n; i++) putCandidate(T, first + i, res, tri[i]);
        }
    }
    if (findStore(T, res, first, n)) T.combineQ[phaseAtomicAdd(&T.count[QC_COMBINE], 1u)] = res;
}

// The two shapes of a box candidate.
struct CandidateShapes {
    ConvexShape box, other;
    Xf boxXf, otherXf;
    float maxDist2;
};
RSB_HD bool candidateShapes(const EngineView& D, const StepTemp& T, const Candidate& c, CandidateShapes& o, int& a) {
    const PairTask k = T.tasks[c.res];
    const CarParams& C = D.P.car;
    a = (int)k.a;
    const int b = k.o1 - OBJ_BALL;
    if (b == 0) return false;  // the ball's triangles are tested by the combine phase
    o.box = carBoxShape(C);
    o.boxXf = carChildXf(C, bodyXf(D, a, b));
    if (c.tri < 0) {
        o.other = makeSphere(D.P.ballRadius);
        o.otherXf = bodyXf(D, a, 0);
        o.maxDist2 = sq((C.boxMargin + D.P.ballMargin) + fmin_(C.cbt, D.P.ballCbt));
        return true;
    }
    V3 v[3];
    triVerts(D.S, k.o0, c.tri, v);
    o.other = makeTri(v, 0.f);
    o.otherXf = xfIdentity();
    o.maxDist2 = boxMeshMaxDist2(C, C.cbt);
    return true;
}
RSB_HD void storeCandidate(CandidateOut& o, uint32_t flags, V3 n, V3 p, float d) {
    o.flags = flags;
    o.normal[0] = n.x; o.normal[1] = n.y; o.normal[2] = n.z;
    o.point[0] = p.x; o.point[1] = p.y; o.point[2] = p.z;
    o.dist = d;
}

RSB_HD void trianglePhase(const EngineView& D, const StepTemp& T, uint32_t i) {
    const Candidate c = T.cand[i];
    CandidateShapes s;
    int a;
    if (!candidateShapes(D, T, c, s, a)) return;
    T.out[i].flags = 0;
    if (c.tri >= 0 && boxTriApart(D.P.car, s.box, s.boxXf, D.P.car.cbt, s.other.v)) return;
    GjkState g;
    gjkIterate(s.box, s.boxXf, s.other, s.otherXf, s.maxDist2, g);
    if (g.needEpa) {
        storeCandidate(T.out[i], g.isValid ? CO_VALID : 0u, g.normalInB, g.pointOnB, g.distance);
        T.deepQ[phaseAtomicAdd(&T.count[QC_DEEP], 1u)] = i;
        return;
    }
    const GjkOut o = gjkFinish(s.box, s.other, g, s.maxDist2);
    if (o.has) storeCandidate(T.out[i], CO_HAS, o.normal, o.point, o.dist);
}

RSB_HD void deepPhase(const EngineView& D, const StepTemp& T, uint32_t e, EpaWork* epa, PhaseStats& st) {
    if (e & DEEP_PAIR) {
        const uint32_t res = e & ~DEEP_PAIR;
        const PairTask k = T.tasks[res];
        if (k.o1 == OBJ_BALL) {
            ballMeshPhase(D, T, res, st);
        } else if (k.o0 == OBJ_BALL) {
            PairWorldT<PairBodies> W;
            LocalPool pool;
            pairWorldInit(D, W, pool, epa, 0u);
            W.b.i0 = 0;
            pairBody(D, (int)k.a, 0, W.b.v0);
            pairBody(D, (int)k.a, k.o1 - OBJ_BALL, W.b.v1);
            Manifold m;
            pairManifold(m, k.o1, OBJ_BALL, fmin_(D.P.car.cbt, D.P.ballCbt));
            carBallContact(W, k.o1 - OBJ_CAR0, carChildXf(D.P.car, W.b.v1.xf), m);
            storePair(D, T, (int)k.a, W, m, res);
        } else {
            carMeshPhase(D, T, res, epa, st);
        }
        return;
    }
    CandidateOut& o = T.out[e];
    CandidateShapes s;
    int a;
    candidateShapes(D, T, T.cand[e], s, a);
    GjkState g;
    gjkFrames(s.boxXf, s.otherXf, g);
    g.isValid = (o.flags & CO_VALID) != 0;
    g.normalInB = V3{o.normal[0], o.normal[1], o.normal[2]};
    g.pointOnB = V3{o.point[0], o.point[1], o.point[2]};
    g.distance = o.dist;
    o.flags = 0;
    if (gjkPenetrate(epa, s.box, s.other, g)) {
        phaseAtomicOr(arenaStatus(D, a), WS_EPA_OVERFLOW);
        return;
    }
    const GjkOut r = gjkFinish(s.box, s.other, g, s.maxDist2);
    if (r.has) storeCandidate(o, CO_HAS, r.normal, r.point, r.dist);
}

// A pair's contacts in the order of its candidates.  Pairs of two bodies keep their points as
// added: the islands phase runs the callbacks on them before refreshContactPoints.
RSB_HD void combinePhase(const EngineView& D, const StepTemp& T, uint32_t res, PhaseStats& st) {
    const PairTask k = T.tasks[res];
    const int a = (int)k.a, b = k.o1 - OBJ_BALL;
    if (k.o0 == OBJ_BALL) {
        const CandidateOut& o = T.out[T.first[res] & ((1u << CANDIDATE_SHIFT) - 1u)];
        PairWorldT<PairBodies> W;
        LocalPool pool;
        pairWorldInit(D, W, pool, nullptr, 0u);
        W.b.i0 = 0;
        pairBody(D, a, 0, W.b.v0);
        pairBody(D, a, b, W.b.v1);
        Manifold m;
        pairManifold(m, k.o1, OBJ_BALL, fmin_(D.P.car.cbt, D.P.ballCbt));
        if (o.flags & CO_HAS)
            addContact(m, pool, OBJ_BALL, objRef(W, OBJ_BALL), k.o1, objRef(W, k.o1),
                       V3{o.normal[0], o.normal[1], o.normal[2]}, V3{o.point[0], o.point[1], o.point[2]}, o.dist);
        storePair(D, T, a, W, m, res);
        return;
    }
    PairWorldT<OneBody> W;
    LocalPool pool;
    pairWorldInit(D, W, pool, nullptr, D.cull ? (D.cull[a] & (1u << b)) : 0u);
    pairBody(D, a, b, W.b.v);
    Manifold m;
    pairManifold(m, k.o1, k.o0, b == 0 ? D.P.ballCbt : D.P.car.cbt);
    bool found = false;
    const uint32_t f = T.first[res], c0 = f & ((1u << CANDIDATE_SHIFT) - 1u);
    for (uint32_t c = c0; c < c0 + (f >> CANDIDATE_SHIFT); c++) {
        const Candidate cd = T.cand[c];
        V3 v[3], n, p;
        float d;
        bool has;
        if (b == 0) {
            triVerts(D.S, k.o0, cd.tri, v);
            has = sphereTriCollide(v, W.b.v.xf.o, D.P.ballRadius, m.cbt, p, n, d);
        } else {
            const CandidateOut& o = T.out[c];
            has = (o.flags & CO_HAS) != 0;
            if (has) {
                triVerts(D.S, k.o0, cd.tri, v);
                n = V3{o.normal[0], o.normal[1], o.normal[2]};
                p = V3{o.point[0], o.point[1], o.point[2]};
                d = o.dist;
            }
        }
        if (has) {
            found = true;
            if (b == 0) addBallTriContact(W, k.o0, cd.tri, v, n, p, d, m);
            else addBoxTriContact(W, k.o0, b - 1, cd.tri, v, n, p, d, m);
        }
    }
    cullCheck(W, b, found);
    if (m.n) refreshContactPoints(m, W.b.v.xf, xfIdentity());
    st.nMissed += W.nMissed;
    storePair(D, T, a, W, m, res);
}

// A plane pair whose test found it in contact.
RSB_HD void planePhase(const EngineView& D, const StepTemp& T, uint32_t res, PhaseStats& st) {
    const PairTask k = T.tasks[res];
    const int a = (int)k.a, b = k.o1 - OBJ_BALL;
    PairWorldT<OneBody> W;
    LocalPool pool;
    pairWorldInit(D, W, pool, nullptr, D.cull ? (D.cull[a] & (1u << b)) : 0u);
    pairBody(D, a, b, W.b.v);
    Manifold m;
    pairManifold(m, k.o1, k.o0, b == 0 ? D.P.ballCbt : D.P.car.cbt);
    if (b == 0) collideBallPlane(W, k.o0, m);
    else collideBoxPlane(W, k.o0, b - 1, carChildXf(D.P.car, W.b.v.xf), m);
    st.nMissed += W.nMissed;
    storePair(D, T, a, W, m, res);
}

RSB_HD void carCarPhase(const EngineView& D, const StepTemp& T, uint32_t res) {
    const PairTask k = T.tasks[res];
    const int a = (int)k.a, ba = k.o0 - OBJ_BALL, bb = k.o1 - OBJ_BALL;
    PairWorldT<PairBodies> W;
    LocalPool pool;
    pairWorldInit(D, W, pool, nullptr, 0u);
    W.b.i0 = ba;
    pairBody(D, a, ba, W.b.v0);
    pairBody(D, a, bb, W.b.v1);
    Manifold m;
    pairManifold(m, k.o1, k.o0, D.P.car.cbt);
    BoxContacts bc;
    carCarContacts(W, ba - 1, bb - 1, bc);
    ObjRef rA = objRef(W, k.o0), rB = objRef(W, k.o1);
    for (int c = 0; c < bc.n; c++)
        addContact(m, pool, k.o0, rA, k.o1, rB, bc.c[c].normalOnB, bc.c[c].point, bc.c[c].depth);
    storePair(D, T, a, W, m, res);
}

// ------------------------------------------------------------------ islands of one body

// Rows of a body against the fixed body: the general rows (SRow) without the fixed side, whose
// vectors are zero, and without the constants (cfm = 0 * jacInv, limits).
struct ContactRow1 {
    V3 n, rc, ang;
    float rhs, rhsPen, jacInv, friction, applied, push;
    int32_t special;
};
struct FrictionRow1 {
    V3 n, rc, ang;
    float rhs, jacInv, applied;
    int32_t contact;
};
constexpr int MAX_ROWS1 = BODY_MAX_TASKS * MAX_POINTS + 1;

struct Solver1State {
    V3 lin, ang, extF, extT;   // the solver body's velocities and external impulses
    V3 dLin, dAng, push, turn;
    V3 invMassV;
};
struct Solver1 : Solver1State {
    int nc, nf;
    ContactRow1 c[MAX_ROWS1];
    FrictionRow1 f[MAX_ROWS1];
};
// setupContactConstraint and convertContactInner's friction row for one contact of the body.
RSB_HD void makeRows1(const Solver1State& S, const Body& b, V3 normal, float dist, float fric, float rest, V3 rel, float dt,
                      int special, ContactRow1& r, FrictionRow1& fr) {
    const float invDt = 1.f / dt;
    const V3 torqueAxis = cross(rel, normal);
    const V3 angA = b.invIw * torqueAxis;
    const float denom0 = b.invMass + dot(normal, cross(angA, rel));
    const float jacInv = 1.f / (denom0 + 0.f + 0.f);
    const V3 vel = b.lin + cross(b.ang, rel);
    const float relVel = dot(normal, vel - v3zero());
    float restitution = restitutionCurve(relVel, rest);
    if (restitution <= 0.f) restitution = 0.f;
    const float v1 = dot(normal, S.lin + S.extF) + dot(torqueAxis, S.ang + S.extT);
    const float rel1 = v1 + 0.f;
    const float velErr = restitution - rel1;
    const float penetration = dist + 0.f;
    const float posErr = (penetration > 0) ? 0.f : -penetration * kErp2 * invDt;
    r.n = normal;
    r.rc = torqueAxis;
    r.ang = angA;
    r.rhsPen = posErr * jacInv;
    r.rhs = velErr * jacInv;
    r.jacInv = jacInv;
    r.friction = fric;
    r.applied = r.push = 0.f;
    r.special = special;
    // friction along the lateral velocity
    const V3 v = (S.lin + S.extF + cross(S.ang + S.extT, rel)) - v3zero();
    const float rv = dot(normal, v);
    V3 lat = v - normal * rv;
    const float latRel = length2(lat);
    if (latRel > kEpsilon) {
        lat *= 1.f / fsqrt(latRel);
    } else {
        V3 lat2;
        planeSpace1(normal, lat, lat2);
    }
    fr.n = lat;
    fr.rc = cross(rel, lat);
    fr.ang = b.invIw * fr.rc;
    const float d0 = b.invMass + dot(lat, cross(fr.ang, rel));
    fr.jacInv = 1.f / (d0 + 0.f);
    const float fv1 = dot(lat, S.lin + S.extF) + dot(fr.rc, S.ang);
    const float fvelErr = 0.f - (fv1 + 0.f);
    fr.rhs = 0.f + fvelErr * fr.jacInv;
    fr.applied = 0.f;
}
RSB_HD void addRows1(Solver1& S, const Body& b, V3 normal, float dist, float fric, float rest, V3 rel, float dt,
                     int special) {
    makeRows1(S, b, normal, dist, fric, rest, rel, dt, special, S.c[S.nc], S.f[S.nf]);
    S.f[S.nf].contact = S.nc;
    S.nc++;
    S.nf++;
}

// resolveSingleConstraintRow* against the fixed body; returns the impulse.
RSB_HD float solveRow1(Solver1State& S, V3 n, V3 rc, V3 ang, float rhs, float cfm, float jacInv, float lo, float hi,
                       bool generic, float& applied) {
    const float applied0 = applied;
    float delta = rhs - applied0 * cfm;
    const float d1 = dot_simd(n, S.dLin) + dot_simd(rc, S.dAng);
    delta = delta - d1 * jacInv;
    delta = delta - 0.f * jacInv;
    const float sum = applied0 + delta;
    const bool lowerLess = sum < lo;
    delta = lowerLess ? (lo - applied0) : delta;
    applied = lowerLess ? lo : sum;
    if (generic) {
        const bool upperLess = sum < hi;
        delta = upperLess ? delta : (hi - applied0);
        applied = upperLess ? applied : hi;
    }
    S.dLin = S.dLin + (n * S.invMassV) * delta;
    S.dAng = S.dAng + ang * delta;
    return delta;
}
// One pass of the split impulse's row; whether it changed anything.
template <class RowT>
RSB_HD bool pushRow1(Solver1State& S, RowT& c) {
    if (c.rhsPen == 0.f) return false;
    const float applied0 = c.push;
    float delta = c.rhsPen - applied0 * (0.f * c.jacInv);
    const float d1 = dot_simd(c.n, S.push) + dot_simd(c.rc, S.turn);
    delta = delta - d1 * c.jacInv;
    delta = delta - 0.f * c.jacInv;
    const float sum = applied0 + delta;
    const bool lowerLess = sum < 0.f;
    delta = lowerLess ? (0.f - applied0) : delta;
    c.push = lowerLess ? 0.f : sum;
    S.push = S.push + (c.n * S.invMassV) * delta;
    S.turn = S.turn + c.ang * delta;
    return delta != 0.f;
}
RSB_HD void iterate1(Solver1& S) {
    for (int it = 0; it < kNumIterations; it++) {
        bool any = false;
        for (int j = 0; j < S.nc; j++) any |= pushRow1(S, S.c[j]);
        if (!any) break;
    }
    for (int it = 0; it < kNumIterations; it++) {
        for (int j = 0; j < S.nc; j++) {
            ContactRow1& c = S.c[j];
            if (c.special) continue;
            solveRow1(S, c.n, c.rc, c.ang, c.rhs, 0.f * c.jacInv, c.jacInv, 0.f, 1e10f, false, c.applied);
        }
        for (int j = 0; j < S.nf; j++) {
            FrictionRow1& fr = S.f[j];
            const ContactRow1& c = S.c[fr.contact];
            const float total = c.applied;
            if (total > 0.f)
                solveRow1(S, fr.n, fr.rc, fr.ang, fr.rhs, 0.f, fr.jacInv, -(c.friction * total), c.friction * total, true,
                          fr.applied);
        }
    }
}

// The place of body i's k-th manifold (in dispatch order) among its island's manifolds in the
// order solveIslands takes them: its unstable sort of the arena's manifolds by island, here one
// island per body, permutes manifolds of one island too.
struct ManifoldOrder {
    int32_t key[MAX_MANIFOLDS], idx[MAX_MANIFOLDS];
    int n;
};
RSB_HD void manifoldOrder(const EngineView& D, const StepTemp& T, int a, int nb, ManifoldOrder& o) {
    o.n = 0;
    for (int i = 0; i < nb; i++) {
        const uint32_t p = infoWord(D, T, a, i, BI_PAIRS);
        const uint32_t act = (p & BI_ACT_MASK) >> BI_ACT_SHIFT;
        // manifolds of sleeping and of non-responding bodies are not in the list
        if (!(p & ((1u << NUM_STATICS) - 1u)) || act == ACT_SLEEPING || !(p & BI_RESPONDS)) continue;
        const int cnt = bitCount(infoWord(D, T, a, i, BI_MANI));
        for (int k = 0; k < cnt; k++) {
            o.key[o.n] = i;
            o.idx[o.n] = k;
            o.n++;
        }
    }
    uint32_t status = 0;
    if (o.n > 1) quickSortKV(o.key, o.idx, 0, o.n - 1, status);
}

// Callbacks and solver of one body that touches static objects only.
RSB_HD void bodyPhase(const EngineView& D, const StepTemp& T, uint32_t e, PhaseStats& st) {
    const int a = (int)(e % (uint32_t)D.N), i = (int)(e / (uint32_t)D.N);
    const float dt = D.P.dt;
    const uint32_t info = infoWord(D, T, a, i, BI_PAIRS), mani = infoWord(D, T, a, i, BI_MANI),
                   tasks = infoWord(D, T, a, i, BI_TASKS);
    // the results of the body's manifolds, in dispatch order
    const uint32_t mesh0 = (tasks & ((1u << MAX_MESHES) - 1u)) ? infoWord(D, T, a, i, BI_MESHRES) : 0u;
    const uint32_t plane0 = (tasks >> MAX_MESHES) ? infoWord(D, T, a, i, BI_PLANERES) : 0u;
    auto resultOf = [&](int s) -> const PairResult& {
        return s < MAX_MESHES
                   ? T.results[mesh0 + bitCount(tasks & ((1u << s) - 1u))]
                   : T.results[plane0 + bitCount((tasks >> MAX_MESHES) & ((1u << (s - MAX_MESHES)) - 1u))];
    };
    uint32_t with = 0;  // manifolds that hold points
    bool world = false;
    V3 worldNormal = v3zero();
    for (uint32_t m = tasks; m; m &= m - 1u) {
        const int s = lowestBit(m);
        const PairResult& r = resultOf(s);
        if (r.n > 0) with |= 1u << s;
        if (r.flags & PR_WORLD) {
            world = true;
            worldNormal = V3{r.normal[0], r.normal[1], r.normal[2]};
        }
    }
    if (world) {
        // onCarWorld's state; its material is in the points already
        putCarV3(D, a, i - 1, RSB_PW(CarP, worldContactNormal), worldNormal);
        putCarWord(D, a, i - 1, RSB_PW(CarP, flags), carWord(D, a, i - 1, RSB_PW(CarP, flags)) | CF_WORLD_CONTACT);
    }
    if (!with) return;  // the finish phase adds the external impulses
    Body b;
    bodyConstants(D, i, b);
    b.xf = bodyXf(D, a, i);
    b.lin = bodyV3(D, a, i, RSB_PW(CarP, lin));
    b.ang = bodyV3(D, a, i, RSB_PW(CarP, ang));
    updateInertia(b);
    Solver1 S;
    S.lin = b.lin;
    S.ang = b.ang;
    S.extF = (tempV3(D, T.force, a, i, 0) * b.invMass) * dt;
    S.extT = tmul(tempV3(D, T.force, a, i, 3), b.invIw) * dt;
    S.dLin = S.dAng = S.push = S.turn = v3zero();
    S.invMassV = V3{b.invMass, b.invMass, b.invMass};
    S.nc = S.nf = 0;
    int spCount = 0;
    float spFric = 0.f, spRest = 0.f, spDist = 0.f;
    V3 spNormal = v3zero();
    auto addManifold = [&](int s) {
        const PairResult& r = resultOf(s);
        const MPoint* pt = T.blocks + (size_t)MAX_POINTS * r.block;
        for (int j = 0; j < r.n; j++) {
            const MPoint& cp = pt[j];
            const V3 rel = cp.posA - b.xf.o, normal = cp.normal;
            if (cp.special) {
                spCount++;
                spFric = cp.fric;
                spRest = cp.rest;
                spNormal = spNormal + normal;
                spDist = spDist + length(rel);
            }
            addRows1(S, b, normal, cp.dist, cp.fric, cp.rest, rel, dt, cp.special);
        }
    };
    if (!(with & (with - 1u))) {
        addManifold(lowestBit(with));
    } else {
        ManifoldOrder o;
        manifoldOrder(D, T, a, arenaBodies(D, a), o);
        for (int k = 0; k < o.n; k++) {
            if (o.key[k] != i) continue;
            uint32_t m = mani;
            for (int q = 0; q < o.idx[k]; q++) m &= m - 1u;
            const int s = lowestBit(m);
            if ((with >> s) & 1u) addManifold(s);
        }
    }
    if (spCount > 0) {
        // convertContactSpecial
        const float distance = spDist / (float)spCount;
        const V3 normal = bdiv(spNormal, (float)spCount);
        addRows1(S, b, normal, distance, spFric, spRest, normal * -distance, dt, 0);
    }
    st.nRows += (uint32_t)(S.nc + S.nf);
    iterate1(S);
    // writeBackBodies
    S.lin = S.lin + S.dLin;
    S.ang = S.ang + S.dAng;
    if (S.push.x != 0.f || S.push.y != 0 || S.push.z != 0 || S.turn.x != 0.f || S.turn.y != 0 || S.turn.z != 0) {
        if (i == 0) b.xf = integrateTransformNoRot(b.xf, S.push, dt);
        else b.xf = integrateTransform(b.xf, S.push, S.turn * kSplitTurnErp, dt);
        putBodyXf(D, a, i, b.xf);
    }
    putBodyV3(D, a, i, RSB_PW(CarP, lin), S.lin + S.extF);
    putBodyV3(D, a, i, RSB_PW(CarP, ang), S.ang + S.extT);
    infoWord(D, T, a, i, BI_PAIRS) = info | BI_SOLVED;
}

// ------------------------------------------------------------------ islands

struct SolveCars {
    CarSim v[2];
    int i0;
    RSB_HD CarSim& operator[](int i) { return v[i == i0 ? 0 : 1]; }
    RSB_HD const CarSim& operator[](int i) const { return v[i == i0 ? 0 : 1]; }
};
// The arena as the contact callbacks and solveIslands see it.
struct SolveWorld {
    const ArenaStatic* S;
    const WorldParams* P;
    int nb;
    Body b[MAX_BODIES];
    int noRot[MAX_BODIES];
    int np;
    int16_t po0[MAX_PAIRS], po1[MAX_PAIRS];
    int nm;
    Manifold m[MAX_MANIFOLDS];
    uint32_t status;
    SolveCars c;
    uint64_t tick;
    V3 ballVelCache;
    uint32_t nRows;
};

// The car fields that the car-ball and car-car callbacks read and write.
RSB_HD void loadContactCar(const EngineView& D, int a, int s, CarSim& c, V3 velCache) {
    c.flags = carWord(D, a, s, RSB_PW(CarP, flags));
    c.team = (c.flags & CF_TEAM_ORANGE) ? 1 : 0;
    c.id = (uint32_t)s + 1u;
    c.carContactOtherId = carWord(D, a, s, RSB_PW(CarP, carContactOtherId));
    c.carContactCooldown = carFloat(D, a, s, RSB_PW(CarP, carContactCooldown));
    c.demoRespawnTimer = carFloat(D, a, s, RSB_PW(CarP, demoRespawnTimer));
    c.ballHitExtraTick = (uint64_t)carWord(D, a, s, RSB_PW(CarP, ballHitExtraTick)) |
                         ((uint64_t)carWord(D, a, s, RSB_PW(CarP, ballHitExtraTick) + 1) << 32);
    for (int r = 0; r < 3; r++) c.rotMat.r[r] = carV3(D, a, s, RSB_PW(CarP, rotMat) + 3 * r);
    c.velCache = velCache;
}

// One arena's solver as its lanes share it.
struct SolveShared {
    SolveWorld W;
    IslandWork I;
    uint32_t actBits[MAX_BODIES], cached;
};

// Pairs, manifolds and contact callbacks of one arena, in dispatch order.
RSB_HD void solveCallbacks(const EngineView& D, const StepTemp& T, int a, SolveShared& sh) {
    SolveWorld& W = sh.W;
    const uint32_t* actBits = sh.actBits;
    uint32_t cached = 0, dynDone = 0;
    int blocks = 0;
    auto addPairTo = [&](int lo, int hi) -> bool {
        if (W.np >= MAX_PAIRS) {
            W.status |= WS_OVERFLOW;
            return false;
        }
        W.po0[W.np] = (int16_t)lo;
        W.po1[W.np] = (int16_t)hi;
        W.np++;
        return true;
    };
    auto active = [&](int i) { return W.b[i].act != ACT_SLEEPING && W.b[i].act != ACT_DISABLE_SIM; };
    // a manifold in dispatch order, with the points of its result (null: none)
    auto addManifold = [&](int o0, int o1, float cbt, const PairResult* r) -> Manifold* {
        if (W.nm >= MAX_MANIFOLDS) {
            W.status |= WS_OVERFLOW;
            return nullptr;
        }
        Manifold& m = W.m[W.nm++];
        pairManifold(m, o0, o1, cbt);
        if (r && (r->flags & PR_BLOCK)) {
            if (blocks >= MAX_BLOCKS) {
                W.status |= WS_OVERFLOW;
                return nullptr;
            }
            blocks++;
            m.n = r->n;
            m.pt = T.blocks + (size_t)MAX_POINTS * r->block;
            return &m;
        }
        return nullptr;
    };
    for (int i = 0; i < W.nb; i++) {
        const uint32_t pairs = actBits[i] & ((1u << NUM_STATICS) - 1u), dyn = infoWord(D, T, a, i, BI_DYN);
        const uint32_t mani = pairs ? infoWord(D, T, a, i, BI_MANI) : 0u;
        const uint32_t tasks = pairs ? infoWord(D, T, a, i, BI_TASKS) : 0u;
        for (uint32_t k = pairs; k; k &= k - 1u) {
            const int s = lowestBit(k);
            if (!addPairTo(s, OBJ_BALL + i)) continue;
            if (!((mani >> s) & 1u)) continue;
            const PairResult* r = nullptr;
            if (s < MAX_MESHES) {
                if ((tasks >> s) & 1u)
                    r = T.results + infoWord(D, T, a, i, BI_MESHRES) + bitCount(tasks & ((1u << s) - 1u));
            } else if ((tasks >> s) & 1u) {
                r = T.results + infoWord(D, T, a, i, BI_PLANERES) +
                    bitCount((tasks >> MAX_MESHES) & ((1u << (s - MAX_MESHES)) - 1u));
            }
            if (addManifold(OBJ_BALL + i, s, i == 0 ? D.P.ballCbt : D.P.car.cbt, r) && (r->flags & PR_WORLD)) {
                // onCarWorld's state; its material is in the points already
                putCarV3(D, a, i - 1, RSB_PW(CarP, worldContactNormal), V3{r->normal[0], r->normal[1], r->normal[2]});
                putCarWord(D, a, i - 1, RSB_PW(CarP, flags), carWord(D, a, i - 1, RSB_PW(CarP, flags)) | CF_WORLD_CONTACT);
            }
        }
        for (uint32_t q = 0; q < (dyn >> 24); q++) {
            const int j = (int)((dyn >> (3 * q)) & 7u), lo = imin_(i, j), hi = imax_(i, j);
            const uint32_t bit = 1u << dynPair(lo, hi);
            if (dynDone & bit) continue;
            if (!addPairTo(OBJ_BALL + lo, OBJ_BALL + hi)) continue;
            dynDone |= bit;
            if (!active(lo) && !active(hi)) continue;
            if (!((infoWord(D, T, a, lo, BI_DYNMANI) >> hi) & 1u)) continue;
            const PairResult* r = T.results + T.dynRes[(size_t)dynPair(lo, hi) * D.N + a];
            if (lo == 0) {
                Manifold* m = addManifold(OBJ_BALL + hi, OBJ_BALL, fmin_(D.P.car.cbt, D.P.ballCbt), r);
                if (!m) continue;
                if (!W.b[hi].noResp) {
                    W.c.i0 = hi - 1;
                    CarSim& c = W.c.v[0];
                    loadContactCar(D, a, hi - 1, c, v3zero());
                    c.ballHitExtraVel = v3zero();
                    onCarBall(W, hi - 1, m->pt[0], false);
                    putCarWord(D, a, hi - 1, RSB_PW(CarP, flags), c.flags);
                    putCarV3(D, a, hi - 1, RSB_PW(CarP, ballHitRelPos), c.ballHitRelPos);
                    putCarWord(D, a, hi - 1, RSB_PW(CarP, ballHitTick), (uint32_t)c.ballHitTick);
                    putCarWord(D, a, hi - 1, RSB_PW(CarP, ballHitTick) + 1, (uint32_t)(c.ballHitTick >> 32));
                    putCarV3(D, a, hi - 1, RSB_PW(CarP, ballHitBallPos), c.ballHitBallPos);
                    putCarV3(D, a, hi - 1, RSB_PW(CarP, ballHitExtraVel), c.ballHitExtraVel);
                    putCarWord(D, a, hi - 1, RSB_PW(CarP, ballHitExtraTick), (uint32_t)c.ballHitExtraTick);
                    putCarWord(D, a, hi - 1, RSB_PW(CarP, ballHitExtraTick) + 1, (uint32_t)(c.ballHitExtraTick >> 32));
                    cached |= 1u;
                }
                if (m->n) refreshContactPoints(*m, W.b[hi].xf, W.b[0].xf);
            } else {
                Manifold* m = addManifold(OBJ_BALL + hi, OBJ_BALL + lo, D.P.car.cbt, r);
                if (!m) continue;
                const int ca = lo - 1, cb = hi - 1;
                if (!W.b[lo].noResp && !W.b[hi].noResp) {
                    W.c.i0 = ca;
                    loadContactCar(D, a, ca, W.c.v[0], (cached >> lo) & 1u ? tempV3(D, T.cache, a, lo, 0) : v3zero());
                    loadContactCar(D, a, cb, W.c.v[1], (cached >> hi) & 1u ? tempV3(D, T.cache, a, hi, 0) : v3zero());
                    for (int k = 0; k < m->n; k++) onCarCar(W, cb, ca, m->pt[k]);
                    for (int e = 0; e < 2; e++) {
                        const int s = e ? cb : ca;
                        const CarSim& c = W.c.v[e];
                        putCarWord(D, a, s, RSB_PW(CarP, flags), c.flags);
                        putCarFloat(D, a, s, RSB_PW(CarP, demoRespawnTimer), c.demoRespawnTimer);
                        putCarWord(D, a, s, RSB_PW(CarP, carContactOtherId), c.carContactOtherId);
                        putCarFloat(D, a, s, RSB_PW(CarP, carContactCooldown), c.carContactCooldown);
                        putTempV3(D, T.cache, a, 1 + s, 0, c.velCache);
                        cached |= 2u << s;
                    }
                }
                if (m->n) refreshContactPoints(*m, W.b[hi].xf, W.b[lo].xf);
            }
        }
    }
    sh.cached = cached;
}

// Callbacks, islands and solver of one arena.
template <class LanesT>
RSB_HD void solvePhase(const EngineView& D, const StepTemp& T, int a, SolveShared& sh, const LanesT& L, PhaseStats& st) {
    SolveWorld& W = sh.W;
    if (L.lane == 0) {
        W.S = &D.S;
        W.P = &D.P;
        W.nb = arenaBodies(D, a);
        W.status = 0;
        W.nRows = 0;
        W.tick = arenaTickCount(D, a);
        W.ballVelCache = v3zero();
        W.np = W.nm = 0;
    }
    const int nb = arenaBodies(D, a);
    for (int i = L.lane; i < nb; i += L.count) {
        Body& b = W.b[i];
        bodyConstants(D, i, b);
        const uint32_t p = infoWord(D, T, a, i, BI_PAIRS);
        sh.actBits[i] = p;
        b.act = (int32_t)((p & BI_ACT_MASK) >> BI_ACT_SHIFT);
        b.noResp = i > 0 && !(p & BI_RESPONDS) ? 1 : 0;
        b.xf = bodyXf(D, a, i);
        b.lin = bodyV3(D, a, i, RSB_PW(CarP, lin));
        b.ang = bodyV3(D, a, i, RSB_PW(CarP, ang));
        b.force = tempV3(D, T.force, a, i, 0);
        b.torque = tempV3(D, T.force, a, i, 3);
        updateInertia(b);
        W.noRot[i] = i == 0 ? 1 : 0;
    }
    L.sync();
    if (L.lane == 0) {
        solveCallbacks(D, T, a, sh);
        islandLists(W, sh.I);
    }
    L.sync();
    solveLists(W, sh.I, L);
    for (int i = L.lane; i < nb; i += L.count) {
        const Body& b = W.b[i];
        putBodyXf(D, a, i, b.xf);
        putBodyV3(D, a, i, RSB_PW(CarP, lin), b.lin);
        putBodyV3(D, a, i, RSB_PW(CarP, ang), b.ang);
        infoWord(D, T, a, i, BI_PAIRS) = (sh.actBits[i] & ~BI_ACT_MASK) | ((uint32_t)b.act << BI_ACT_SHIFT) | BI_SOLVED |
                                         ((sh.cached >> i) & 1u ? BI_CACHE : 0u);
    }
    if (L.lane == 0) {
        if (sh.cached & 1u) putTempV3(D, T.cache, a, 0, 0, W.ballVelCache);
        st.nRows += W.nRows;
        if (W.status) phaseAtomicOr(arenaStatus(D, a), W.status);
    }
    L.sync();
}

// ------------------------------------------------------------------ finish

struct FinishShared {
    int32_t locked[NUM_PADS][PHASE_ARENAS];        // car that locked the pad this tick, MAX_CARS none
    uint32_t prevLocked[NUM_PADS][PHASE_ARENAS];   // car id of the last tick
    uint32_t picked[MAX_CARS][PHASE_ARENAS];       // pads taken: small | big << 16
    uint32_t touched[PHASE_ARENAS];
};

RSB_HD void padLoad(const EngineView& D, int a, int la, int p, FinishShared& sh) {
    sh.locked[p][la] = MAX_CARS;
    sh.prevLocked[p][la] = D.pad[((size_t)RSB_PW(PadP, bits) * NUM_PADS + p) * D.N + a] >> 8;
}

struct FinishThread {
    const WorldParams* P;
    OneBody b;
    OneCar c;
    int a, la, body, nb;
    uint64_t tick;
    bool pads;  // the car may collide with pads
};

// Integration and post-tick of one body (integrateBodies, updateActivation, carPostTick,
// ballFinishTick).
RSB_HD void finishBody(const EngineView& D, const StepTemp& T, FinishThread& t, FinishShared& sh) {
    Body& b = t.b.v;
    CarSim& c = t.c.v;
    const int a = t.a, i = t.body, s = i - 1;
    const float dt = D.P.dt;
    const uint32_t info = infoWord(D, T, a, i, BI_PAIRS);
    t.P = &D.P;
    t.tick = arenaTickCount(D, a);
    t.pads = false;
    bodyConstants(D, i, b);
    b.act = (int32_t)((info & BI_ACT_MASK) >> BI_ACT_SHIFT);
    b.xf = bodyXf(D, a, i);
    b.lin = bodyV3(D, a, i, RSB_PW(CarP, lin));
    b.ang = bodyV3(D, a, i, RSB_PW(CarP, ang));
    const bool moves = b.act != ACT_SLEEPING && b.act != ACT_DISABLE_SIM;
    if (!(info & BI_SOLVED) && moves) {
        // an island of one body without contacts: the solver adds the external impulses only
        updateInertia(b);
        b.force = tempV3(D, T.force, a, i, 0);
        b.torque = tempV3(D, T.force, a, i, 3);
        const V3 extF = (b.force * b.invMass) * dt, extT = tmul(b.torque, b.invIw) * dt;
        b.lin = (b.lin + v3zero()) + extF;
        b.ang = (b.ang + v3zero()) + extT;
    }
    if (moves) b.xf = i == 0 ? integrateTransformNoRot(b.xf, b.lin, dt) : integrateTransform(b.xf, b.lin, b.ang, dt);
    if (b.act == ACT_SLEEPING) b.lin = b.ang = v3zero();
    if (moves) {
        putBodyV3(D, a, i, RSB_PW(CarP, pos), b.xf.o);
        if (i != 0)
#pragma unroll
            for (int r = 0; r < 3; r++) putBodyV3(D, a, i, RSB_PW(CarP, rot) + 3 * r, b.xf.b.r[r]);
    }
    if (i == 0) {
        ballFinishTick(t, (info & BI_CACHE) ? tempV3(D, T.cache, a, 0, 0) : v3zero());
        putBodyV3(D, a, 0, RSB_PW(BallP, lin), b.lin);
        putBodyV3(D, a, 0, RSB_PW(BallP, ang), b.ang);
        return;
    }
    c.flags = carWord(D, a, s, RSB_PW(CarP, flags));
    if (!(c.flags & CF_DEMOED)) {
        const uint32_t flags0 = c.flags;
        c.boost = carFloat(D, a, s, RSB_PW(CarP, boost));
        c.supersonicTime = carFloat(D, a, s, RSB_PW(CarP, supersonicTime));
        c.carContactCooldown = carFloat(D, a, s, RSB_PW(CarP, carContactCooldown));
        const float supersonic0 = c.supersonicTime, cooldown0 = c.carContactCooldown;
        const CtlRec& ctl = D.controls[D.carOffset[a] + s];
#pragma unroll
        for (int k = 0; k < 5; k++) c.ctl[k] = clampf(ctl.v[k], -1, 1);
        c.ctlBits = (ctl.jump ? 1u : 0u) | (ctl.boost ? 2u : 0u) | (ctl.handbrake ? 4u : 0u);
        c.velCache = (info & BI_CACHE) ? tempV3(D, T.cache, a, i, 0) : v3zero();
        carPostTick(t, s);
        putBodyV3(D, a, i, RSB_PW(CarP, lin), b.lin);
        putBodyV3(D, a, i, RSB_PW(CarP, ang), b.ang);
#pragma unroll
        for (int r = 0; r < 3; r++) putCarV3(D, a, s, RSB_PW(CarP, rotMat) + 3 * r, c.rotMat.r[r]);
        if (c.flags != flags0) putCarWord(D, a, s, RSB_PW(CarP, flags), c.flags);
        if (f2u(c.supersonicTime) != f2u(supersonic0)) putCarFloat(D, a, s, RSB_PW(CarP, supersonicTime), c.supersonicTime);
        if (f2u(c.carContactCooldown) != f2u(cooldown0))
            putCarFloat(D, a, s, RSB_PW(CarP, carContactCooldown), c.carContactCooldown);
#pragma unroll
        for (int k = 0; k < 5; k++) putCarFloat(D, a, s, RSB_PW(CarP, lastCtl) + k, c.lastCtl[k]);
        putCarWord(D, a, s, RSB_PW(CarP, lastCtlBits), c.lastCtlBits);
        t.pads = c.boost < 100;
    } else if (moves) {
        // demoed in this tick: integrated, then left alone
        putBodyV3(D, a, i, RSB_PW(CarP, lin), b.lin);
        putBodyV3(D, a, i, RSB_PW(CarP, ang), b.ang);
    }
    const uint64_t hit = (uint64_t)carWord(D, a, s, RSB_PW(CarP, ballHitTick)) |
                         ((uint64_t)carWord(D, a, s, RSB_PW(CarP, ballHitTick) + 1) << 32);
    if (hit == t.tick) phaseAtomicOr(&sh.touched[t.la], 1u << s);
}

// BoostPadGrid::CheckCollision of one car: the pads it locks (the lowest slot wins a pad, as
// the last writer of the reference's loop over the cars in reverse creation order).
RSB_HD void finishPads(const EngineView& D, FinishThread& t, FinishShared& sh) {
    if (!t.pads) return;
    const V3 carPos = t.b.v.xf.o * kBtToUu;
    if (carPos.z > PAD_CYL_HEIGHT + 250.f) return;
    const int ix = (int)(carPos.x / 1024.f + 4.f), iy = (int)(carPos.y / 1024.f + 5.f);
    for (int i = imax_(ix - 1, 0); i <= imin_(ix + 1, 7); i++)
        for (int j = imax_(iy - 1, 0); j <= imin_(iy + 1, 9); j++) {
            const int p = D.P.padGrid[i * 10 + j];
            if (p < 0) continue;
            if (padCollides(D.P, p, t.b.v.xf, sh.prevLocked[p][t.la] == (uint32_t)t.body)) {
#if defined(__CUDA_ARCH__)
                atomicMin(&sh.locked[p][t.la], t.body - 1);
#else
                sh.locked[p][t.la] = imin_(sh.locked[p][t.la], t.body - 1);
#endif
            }
        }
}

// One pad's cooldown and pickup.
RSB_HD void finishPad(const EngineView& D, int a, int la, int p, FinishShared& sh) {
    uint32_t* cool = D.pad + ((size_t)RSB_PW(PadP, cooldown) * NUM_PADS + p) * D.N + a;
    uint32_t* bits = D.pad + ((size_t)RSB_PW(PadP, bits) * NUM_PADS + p) * D.N + a;
    const uint32_t cool0 = *cool;
    float cd = u2f(cool0);
    if (cd > 0) cd = fmax_(cd - D.P.dt, 0);
    uint32_t isActive = cd == 0 ? 1u : 0u, locked = 0;
    const int car = sh.locked[p][la];
    if (car < MAX_CARS) {
        locked = (uint32_t)car + 1u;
        if (isActive) {
            phaseAtomicAdd(&sh.picked[car][la], p < NUM_BIG_PADS ? 0x10000u : 1u);
            isActive = 0;
            cd = p < NUM_BIG_PADS ? D.P.car.padCooldownBig : D.P.car.padCooldownSmall;
        }
    }
    if (f2u(cd) != cool0) *cool = f2u(cd);
    *bits = isActive | (locked << 8);
}

// The boost of the pads a car took.  The amounts are added one by one and clamped, so their
// order does not matter: equal amounts commute, and a big pad fills the tank.
RSB_HD void finishBoost(const EngineView& D, const FinishThread& t, const FinishShared& sh) {
    const int s = t.body - 1;
    const uint32_t n = sh.picked[s][t.la];
    if (!n) return;
    float boost = t.c.v.boost;
    for (uint32_t k = 0; k < (n & 0xffffu); k++) boost = fmin_(boost + PAD_BOOST_AMOUNT_SMALL, BOOST_MAX);
    for (uint32_t k = 0; k < (n >> 16); k++) boost = fmin_(boost + PAD_BOOST_AMOUNT_BIG, BOOST_MAX);
    putCarFloat(D, t.a, s, RSB_PW(CarP, boost), boost);
}

// Arena counters, by the ball's thread.
RSB_HD void finishArena(const EngineView& D, const FinishThread& t, const FinishShared& sh) {
    const int a = t.a;
    const bool scored = ballScored(t, D.P.goalBaseY, D.P.ballRadiusUu);
    const int side = t.b.v.xf.o.y > 0 ? 0 : 1;
    auto put = [&](int w, uint32_t v) { D.arena[(size_t)w * D.N + a] = v; };
    if (scored && (int32_t)arenaWord(D, a, RSB_PW(ArenaP, goalTeam)) < 0) put(RSB_PW(ArenaP, goalTeam), (uint32_t)side);
    put(RSB_PW(ArenaP, scored), scored ? (side == 0 ? 1u : 2u) : 0u);
    const uint64_t tk = t.tick + 1;
    put(RSB_PW(ArenaP, tick), (uint32_t)tk);
    put(RSB_PW(ArenaP, tick) + 1, (uint32_t)(tk >> 32));
    put(RSB_PW(ArenaP, episodeTicks), arenaWord(D, a, RSB_PW(ArenaP, episodeTicks)) + 1u);
    const uint32_t touched = sh.touched[t.la];
    if (touched) put(RSB_PW(ArenaP, touchedMask), arenaWord(D, a, RSB_PW(ArenaP, touchedMask)) | touched);
}

#undef RSB_PW

}  // namespace rsb
