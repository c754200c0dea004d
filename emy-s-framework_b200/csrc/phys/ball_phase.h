// Ticks of a world that holds the ball alone (ball prediction).
//
// The tick is arenaTick() for an arena without cars, kept in registers: gravity, predicted
// motion, static pairs, sphere-plane and sphere-triangle contacts, the solver for one body
// (Solver1), integration and speed limits.  The ball never rotates (btRigidBody m_noRot).
// Triangles near the ball are listed once for a box BALL_MARGIN larger than the ball's and
// tested from the list while the ball stays within the margin: a triangle whose box overlaps the
// ball's is in the list, the list keeps the order of the mesh queries, and every listed triangle
// goes through the query's own tests, so the contacts are those of the query.  Until the ball has
// come as near to where the nearest listed triangle can be as a contact needs, none is tested.
#pragma once
#include "step_phases.h"

namespace rsb {

constexpr int BALL_LIST = 96;          // triangles a list holds
constexpr int BALL_LIST_NONE = -1;     // not made yet
constexpr int BALL_LIST_OVER = -2;     // more triangles than it holds: the meshes are queried
constexpr float BALL_MARGIN = 2.f;      // Bullet units (100 uu: two ticks of flight at the top speed)
constexpr float BALL_LIST_SLACK = 1e-2f;

struct BallSim {
    Xf xf;
    V3 lin, ang;
    M3 invIw;
    int32_t cell;
    V3 bpMin, bpMax;
    int act;
    uint32_t pairs;   // static pairs of the tick
    V3 listAt;        // where the list was made
    int listN;
    float listClear;  // no listed triangle is nearer to listAt
};

RSB_HD uint16_t ballListKey(int mesh, int tri) { return (uint16_t)((mesh << 10) | tri); }

RSB_HD void ballSimInit(const EngineView& D, const BallP& p, BallSim& s) {
    Body b;
    ballBodyOf(D, p, b);
    s.xf = b.xf;
    s.lin = b.lin;
    s.ang = b.ang;
    s.invIw = b.invIw;
    s.cell = b.cell;
    s.bpMin = s.bpMax = b.xf.o;
    s.listN = BALL_LIST_NONE;
    s.listClear = 0.f;
    s.listAt = b.xf.o;
}

// The box that a list made at `at` covers.
RSB_HD void ballListBox(const WorldParams& P, V3 at, V3& mn, V3& mx) {
    const float e = P.ballAabbExt + BALL_MARGIN + BALL_LIST_SLACK;
    mn = at - V3{e, e, e};
    mx = at + V3{e, e, e};
}

// The tick up to the static pairs.  Returns true when the ball needs a new list.
RSB_HD bool ballTickPairs(const EngineView& D, BallSim& s) {
    const ArenaStatic& S = D.S;
    const WorldParams& P = D.P;
    s.act = (length2(s.lin) == 0.f && length2(s.ang) == 0.f) ? ACT_SLEEPING : ACT_ACTIVE;
    s.lin = s.lin * P.ballLinDampFactor;
    // btCollisionWorld::updateSingleAabb over the transform and the predicted one
    const Xf ixf = integrateTransformNoRot(s.xf, s.lin, P.dt);
    const V3 thr{0.02f, 0.02f, 0.02f};
    V3 mn, mx, mn2, mx2;
    ballAabb(P, s.xf, mn, mx);
    ballAabb(P, ixf, mn2, mx2);
    mn = vmin(mn - thr, mn2 - thr);
    mx = vmax(mx + thr, mx2 + thr);
    if (!(length2(mx - mn) < 1e12f)) {
        s.act = ACT_DISABLE_SIM;
    } else {
        s.bpMin = mn;
        s.bpMax = mx;
        int i, j, k;
        bpCellIndices(S.bp, mn, i, j, k);
        s.cell = i * S.bp.cellsY * S.bp.cellsZ + j * S.bp.cellsZ + k;
    }
    s.pairs = 0;
    for (uint32_t m = S.bpCells[s.cell]; m; m &= m - 1u) {
        const int o = lowestBit(m);
        V3 smn, smx;
        if (o < MAX_MESHES) { smn = S.meshes[o].bpMin; smx = S.meshes[o].bpMax; }
        else { smn = S.planeBpMin[o - MAX_MESHES]; smx = S.planeBpMax[o - MAX_MESHES]; }
        if (aabbOverlap(s.bpMin, s.bpMax, smn, smx)) s.pairs |= 1u << o;
    }
    if (s.act != ACT_ACTIVE || !(s.pairs & ((1u << MAX_MESHES) - 1u))) return false;
    const V3 d = s.xf.o - s.listAt;
    if (s.listN != BALL_LIST_NONE && fabsf(d.x) <= BALL_MARGIN && fabsf(d.y) <= BALL_MARGIN && fabsf(d.z) <= BALL_MARGIN)
        return false;
    // far from every mesh: an empty list, by the voxel's distance bound (uu) against the half
    // diagonal of the list's box
    s.listAt = s.xf.o;
    s.listN = 0;
    const int x = (int)floorf((s.xf.o.x - S.occMin.x) * S.occInvCell), y = (int)floorf((s.xf.o.y - S.occMin.y) * S.occInvCell),
              z = (int)floorf((s.xf.o.z - S.occMin.z) * S.occInvCell);
    if (x >= 0 && y >= 0 && z >= 0 && x < S.occX && y < S.occY && z < S.occZ) {
        const float clear = (float)S.occDist[(x * S.occY + y) * S.occZ + z] * kUuToBt;
        if (clear > 1.7321f * (P.ballAabbExt + BALL_MARGIN + 2 * BALL_LIST_SLACK)) return false;
    }
    return true;
}

// The tests that every triangle of the tick's mesh queries passes before its contact is computed.
struct BallBox {
    V3 mn, mx;
    M3 invB;
};
RSB_HD void ballBoxOf(const WorldParams& P, const Xf& xf, BallBox& x) {
    ballAabb(P, xf, x.mn, x.mx);
    x.invB = inverse(xf.b);
}
RSB_HD bool ballNear(const EngineView& D, const Xf& xf, const BallBox& x, int mesh, int tri) {
    const TriData& td = triData(D.S, mesh, tri);
    return triBoxOverlap(td, x.mn, x.mx) && ballTriPlanes(D.P, xf, x.invB, D.P.ballCbt, td.unit, td.unitDist);
}
// Whether the tick's contacts read triangles.
RSB_HD bool ballReadsList(const WorldParams& P, const BallSim& s) {
    return s.act == ACT_ACTIVE && (s.pairs & ((1u << MAX_MESHES) - 1u)) && s.listN != 0 &&
           !(s.listClear - length(s.xf.o - s.listAt) > P.ballRadius + P.ballCbt + BALL_LIST_SLACK);
}
// A point's distance from a triangle's box, which bounds its distance from the triangle.
RSB_HD float triBoxDistance(const TriData& t, V3 o) {
    const V3 d = vmax(vmax(t.lo - o, o - t.hi), v3zero());
    return length(d);
}

// The list on one thread.
RSB_HD void ballListMake(const EngineView& D, BallSim& s, uint16_t* list) {
    V3 mn, mx;
    ballListBox(D.P, s.listAt, mn, mx);
    int n = 0;
    s.listClear = 1e30f;
    for (int m = 0; m < D.S.numMeshes; m++) {
        if (!aabbOverlap(mn, mx, D.S.meshes[m].shapeMin, D.S.meshes[m].shapeMax)) continue;
        bvhQueryLeaves(D.S, m, mn, mx, [&](int tri) {
            const TriData& td = triData(D.S, m, tri);
            if (!triBoxOverlap(td, mn, mx)) return true;
            s.listClear = fmin_(s.listClear, triBoxDistance(td, s.listAt));
            if (n < BALL_LIST) list[n] = ballListKey(m, tri);
            n++;
            return true;
        });
    }
    s.listN = n <= BALL_LIST ? n : BALL_LIST_OVER;
}

// Contacts of one tick: the points of the manifolds that hold any, as the solver reads them.  Their
// friction and restitution are the same for every static object.
struct BallPoint {
    V3 pos, normal;  // posA, on the ball
    float dist;
};
struct BallContacts {
    int blocks;
    uint8_t of[MAX_BLOCKS], n[MAX_BLOCKS];  // place of the manifold among the tick's, and its points
    BallPoint pts[MAX_BLOCKS][MAX_POINTS];
};

// collideBallPlane for a ball whose deepest point is vip, `distance` from the plane: addContact and
// refreshContactPoints on a manifold of one point.  Returns its points, none or one.
RSB_HD int ballPlanePoint(const EngineView& D, int plane, const Xf& xf, V3 vip, float distance, BallPoint& q) {
    const Xf planeXf{m3identity(), D.S.planeOrigin[plane - MAX_MESHES]};
    const V3 pn = D.S.planeNormal[plane - MAX_MESHES];
    const V3 proj = vip - pn * distance;
    const V3 world = xfPoint(planeXf, proj);
    const V3 nb = planeXf.b * pn;
    const V3 localA = xfInvPoint(xf, world + nb * distance), localB = xfInvPoint(planeXf, world);
    q.pos = xfPoint(xf, localA);
    const V3 posB = xfPoint(planeXf, localB);
    q.normal = nb;
    q.dist = dot(q.pos - posB, nb);
    if (!(q.dist <= D.P.ballCbt)) return 0;
    const V3 diff = posB - (q.pos - nb * q.dist);
    return dot(diff, diff) > D.P.ballCbt * D.P.ballCbt ? 0 : 1;
}

// The solver's rows for a ball that touches static objects only.  Every point's row is special
// (Arena.cpp:264-271): it takes part in the split impulse only, and its friction, whose limit is the
// row's impulse of zero, never acts.  The velocities are those of one aggregated row.  The first
// row is kept apart, in registers: a ball mostly touches one point.
struct BallRow {
    V3 n, rc, ang;
    float rhsPen, jacInv, push;
};
struct BallRows {
    int n;  // rows that push, after the first
    BallRow r[MAX_CONTACT_ROWS];
};
RSB_HD BallRow ballRowOf(const ContactRow1& c) { return BallRow{c.n, c.rc, c.ang, c.rhsPen, c.jacInv, 0.f}; }

// The rest of the tick: contacts, solver, integration, speed limits.  list holds the listN triangles
// that may touch the ball, in query order (BALL_LIST_OVER: the meshes are queried).
RSB_HD void ballTickSolve(const EngineView& D, BallSim& s, const uint16_t* list, int listN, BallContacts& C, BallRows& R) {
    const ArenaStatic& S = D.S;
    const WorldParams& P = D.P;
    const float dt = P.dt;
    if (s.act == ACT_ACTIVE) {
        // dispatchAllCollisionPairs: every pair of an active ball has a manifold
        C.blocks = 0;
        int place = 0, at = 0, points = 0;
        BallPoint one;  // the first block's first point, in registers
        LocalPool pool;
        PairWorldT<OneBody> W;
        bool inited = false;
        for (uint32_t m = s.pairs; m; m &= m - 1u, place++) {
            const int o = lowestBit(m);
            Manifold man;
            auto begin = [&]() {
                if (inited) return;
                pairWorldInit(D, W, pool, nullptr, 0u);
                bodyConstants(D, 0, W.b.v);
                W.b.v.xf = s.xf;
                inited = true;
            };
            pool.n = 0;
            pairManifold(man, OBJ_BALL, o, P.ballCbt);
            if (o < MAX_MESHES) {
                if (listN == 0) continue;
                BallBox box;
                ballBoxOf(P, s.xf, box);
                auto test = [&](int tri) {
                    if (!ballNear(D, s.xf, box, o, tri)) return true;
                    V3 v[3], p, n;
                    float d;
                    triVerts(S, o, tri, v);
                    if (sphereTriCollide(v, s.xf.o, P.ballRadius, P.ballCbt, p, n, d)) {
                        begin();
                        addBallTriContact(W, o, tri, v, n, p, d, man);
                    }
                    return true;
                };
                if (listN == BALL_LIST_OVER) {
                    bvhQueryAabb(S, o, box.mn, box.mx, test);
                } else {
                    while (at < listN && (int)(list[at] >> 10) < o) at++;
                    for (; at < listN && (int)(list[at] >> 10) == o; at++) test((int)(list[at] & 1023u));
                }
                if (man.n) refreshContactPoints(man, s.xf, xfIdentity());
            } else {
                V3 vip;
                const float distance = ballPlaneDistance(S, P, o, s.xf, vip);
                if (!(distance < P.ballCbt + 0.f)) continue;
                if (C.blocks >= MAX_BLOCKS) continue;
                BallPoint q;
                const int n = ballPlanePoint(D, o, s.xf, vip, distance, q);
                if (C.blocks == 0) one = q;
                C.of[C.blocks] = (uint8_t)place;
                C.n[C.blocks] = (uint8_t)n;
                C.pts[C.blocks++][0] = q;
                points += n;
                continue;
            }
            // a manifold takes a block with its first contact, while there are blocks
            if (!man.pt || C.blocks >= MAX_BLOCKS) continue;
            C.of[C.blocks] = (uint8_t)place;
            C.n[C.blocks] = (uint8_t)man.n;
            for (int k = 0; k < man.n; k++) {
                const BallPoint q{man.pt[k].posA, man.pt[k].normal, man.pt[k].dist};
                if (C.blocks == 0 && k == 0) one = q;
                C.pts[C.blocks][k] = q;
            }
            points += man.n;
            C.blocks++;
        }
        Body b;
        bodyConstants(D, 0, b);
        b.force = b.force + b.grav;
        const V3 extF = (b.force * b.invMass) * dt, extT = tmul(b.torque, s.invIw) * dt;
        if (points == 0) {
            s.lin = (s.lin + v3zero()) + extF;
            s.ang = (s.ang + v3zero()) + extT;
        } else {
            b.xf = s.xf;
            b.lin = s.lin;
            b.ang = s.ang;
            b.invIw = s.invIw;
            Solver1State S1;
            S1.lin = s.lin;
            S1.ang = s.ang;
            S1.extF = extF;
            S1.extT = extT;
            S1.dLin = S1.dAng = S1.push = S1.turn = v3zero();
            S1.invMassV = V3{b.invMass, b.invMass, b.invMass};
            R.n = 0;
            ContactRow1 c;
            FrictionRow1 f;
            BallRow first;
            first.rhsPen = 0.f;
            int spCount = 0;
            float spDist = 0.f;
            const float fric = STATIC_FRICTION < b.friction ? STATIC_FRICTION : b.friction,
                        rest = STATIC_RESTITUTION > b.restitution ? STATIC_RESTITUTION : b.restitution;
            V3 spNormal = v3zero();
            // the island's manifolds after its unstable sort (all of one island)
            const bool sorted = C.blocks > 1;
            int32_t idx[MAX_MANIFOLDS];
            if (sorted) {
                int32_t key[MAX_MANIFOLDS];
                for (int k = 0; k < place; k++) {
                    key[k] = 0;
                    idx[k] = k;
                }
                uint32_t status = 0;
                quickSortKV(key, idx, 0, place - 1, status);
            }
            for (int q = 0; q < (sorted ? place : 1); q++) {
                int k = 0;
                if (sorted)
                    while (k < C.blocks && C.of[k] != idx[q]) k++;
                if (k == C.blocks) continue;
                for (int j = 0; j < C.n[k] && spCount < MAX_CONTACT_ROWS; j++) {
                    const BallPoint cp = (k | j) ? C.pts[k][j] : one;
                    const V3 rel = cp.pos - s.xf.o;
                    spCount++;
                    spNormal = spNormal + cp.normal;
                    spDist = spDist + length(rel);
                    makeRows1(S1, b, cp.normal, cp.dist, fric, rest, rel, dt, 1, c, f);
                    if (c.rhsPen == 0.f) continue;
                    if (first.rhsPen == 0.f) first = ballRowOf(c);
                    else R.r[R.n++] = ballRowOf(c);
                }
            }
            const bool solved = spCount < MAX_CONTACT_ROWS;
            BallRow last;
            last.rhsPen = 0.f;
            if (solved) {
                const float distance = spDist / (float)spCount;
                const V3 normal = bdiv(spNormal, (float)spCount);
                makeRows1(S1, b, normal, distance, fric, rest, normal * -distance, dt, 0, c, f);
                last = ballRowOf(c);
            }
            for (int it = 0; it < kNumIterations; it++) {
                bool any = pushRow1(S1, first);
                for (int j = 0; j < R.n; j++) any |= pushRow1(S1, R.r[j]);
                any |= pushRow1(S1, last);
                if (!any) break;
            }
            for (int it = 0; solved && it < kNumIterations; it++) {
                solveRow1(S1, c.n, c.rc, c.ang, c.rhs, 0.f * c.jacInv, c.jacInv, 0.f, 1e10f, false, c.applied);
                const float total = c.applied;
                if (total > 0.f)
                    solveRow1(S1, f.n, f.rc, f.ang, f.rhs, 0.f, f.jacInv, -(c.friction * total), c.friction * total, true,
                              f.applied);
            }
            const V3 push = S1.push, turn = S1.turn;
            if (push.x != 0.f || push.y != 0 || push.z != 0 || turn.x != 0.f || turn.y != 0 || turn.z != 0)
                s.xf = integrateTransformNoRot(s.xf, push, dt);
            s.lin = (S1.lin + S1.dLin) + extF;
            s.ang = (S1.ang + S1.dAng) + extT;
        }
        s.xf = integrateTransformNoRot(s.xf, s.lin, dt);
    } else if (s.act == ACT_SLEEPING) {
        s.lin = s.ang = v3zero();
    }
    // ballFinishTick without a velocity cache
    const float ms = P.ballMaxSpeedBt;
    if (length2(s.lin) > ms * ms) s.lin = normalized(s.lin) * ms;
    if (length2(s.ang) > BALL_MAX_ANG_SPEED * BALL_MAX_ANG_SPEED) s.ang = normalized(s.ang) * BALL_MAX_ANG_SPEED;
}

// The ball as a record (for the public state).
RSB_HD BallP ballSimRecord(const BallP& from, const BallSim& s) {
    BallP p = from;
    xfToP(s.xf, p.pos, p.rot);
    putV3(p.lin, s.lin);
    putV3(p.ang, s.ang);
    return p;
}

}  // namespace rsb
