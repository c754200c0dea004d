// Host run of the step's phases (emy-s-framework_b200/csrc/phys/step_phases.h) beside the
// one-thread tick of the host engine, for the CPU test that compares the two byte by byte.
// The loops below stand for the kernels of step_kernels.cuh: blocks of 32 arenas with one
// thread per body, queues taken from the back so that nothing depends on their order.
#include "host_engine.cpp"

#include "phys/ball_phase.h"
#include "phys/step_phases.h"

extern "C" {

// `ticks` ticks of the handle's arenas through the phases.  cull: a body mask per arena, or null;
// cand_cap: room for triangle candidates (-1: as the engine has); by_bodies 0: every arena with
// contacts is solved as a whole.
// Returns the number of items that went through each queue in counts[QC_WORDS].
int32_t rsb_host_step_phases(rsb_handle* h, int32_t ticks, uint32_t* cull, int32_t cand_cap, int32_t by_bodies,
                             int64_t* counts,
                             uint64_t* stats) {
    const size_t N = h->N, B = MAX_BODIES * N, R = (size_t)4 * MAX_CARS * N;
    EngineView D;
    D.S = h->S.view;
    D.P = h->P;
    D.N = h->N;
    D.teamSize = h->teamSize.data();
    D.carOffset = h->carOffset.data();
    D.ball = h->ball.data();
    D.car = h->car.data();
    D.pad = h->pad.data();
    D.arena = h->arena.data();
    D.controls = reinterpret_cast<const CtlRec*>(h->controls.data());
    D.seed = (uint32_t)(h->seed ^ (h->seed >> 32));
    D.cull = cull;
    D.cullAudit = 0;
    D.counters = nullptr;
    D.work = nullptr;
    std::vector<int32_t> rayObj(R);
    std::vector<float> rayFrac(R), rayN(3 * R), force(6 * B), box(6 * B), cache(3 * B);
    std::vector<uint32_t> info(BI_WORDS * B, 0xdeadbeefu), dynRes(NUM_DYN_PAIRS * N), count(QC_WORDS, 0u), rayQ(2 * R), solveQ(N), bodyQ(B);
    std::vector<BodyStatics> statics(MAX_BODIES * PHASE_ARENAS);
    std::vector<PairTask> tasks(CAP_RESULTS * N);
    std::vector<PairResult> results(CAP_RESULTS * N);
    std::vector<MPoint> blocks(MAX_BLOCKS * N * MAX_POINTS);
    StepTemp T;
    T.rayObj = rayObj.data();
    T.rayFrac = rayFrac.data();
    T.rayN = rayN.data();
    T.info = info.data();
    T.force = force.data();
    T.box = box.data();
    T.cache = cache.data();
    T.dynRes = dynRes.data();
    T.count = count.data();
    T.rayQ = rayQ.data();
    T.tasks = tasks.data();
    T.results = results.data();
    T.blocks = blocks.data();
    T.blockCap = (uint32_t)(MAX_BLOCKS * N);
    T.solveQ = solveQ.data();
    T.bodyQ = bodyQ.data();
    T.candCap = cand_cap < 0 ? (uint32_t)(CAP_CANDIDATES * N) : (uint32_t)cand_cap;
    std::vector<uint32_t> first(CAP_RESULTS * N), deepQ(CAP_RESULTS * N + T.candCap), combineQ(CAP_RESULTS * N);
    std::vector<Candidate> cand(T.candCap);
    std::vector<CandidateOut> candOut(T.candCap);
    T.first = first.data();
    T.cand = cand.data();
    T.out = candOut.data();
    T.deepQ = deepQ.data();
    T.combineQ = combineQ.data();
    T.sms = 1;
    std::unique_ptr<EpaWork> epa(new EpaWork());
    std::unique_ptr<DriveShared> ds(new DriveShared());
    std::unique_ptr<PairShared> sh(new PairShared());
    std::unique_ptr<SolveShared> ss(new SolveShared());
    std::unique_ptr<FinishShared> fs(new FinishShared());
    std::vector<DriveThread> dt(MAX_CARS * PHASE_ARENAS);
    std::vector<PairThread> bt(MAX_BODIES * PHASE_ARENAS);
    std::vector<FinishThread> ft(MAX_BODIES * PHASE_ARENAS);
    PhaseStats st{0, 0, 0, 0};
    for (int tick = 0; tick < ticks; tick++) {
        // rays
        for (int a = 0; a < h->N; a++)
            for (int s = 0; s < 2 * h->teamSize[a]; s++) {
                Xf xf;
                bool culled;
                if (!rayCar(D, a, s, xf, culled)) continue;
                auto near = [&](uint32_t at) {
                    uint32_t n = 0;
                    for (int b = 0; b < arenaBodies(D, a); b++) n |= cellsNear(at, bodyCellWord(D, a, b)) ? 1u << b : 0u;
                    return n;
                };
                for (int w = 0; w < 4; w++) {
                    const RayClass c = rayPhase(D, T, a, s, w, xf, culled, near, st);
                    if (c == RAY_MESHES) T.rayQ[T.count[QC_RAY]++] = (uint32_t)rayIdx(D, a, s, w);
                    else if (c == RAY_BODIES) T.rayQ[R + T.count[QC_BODYRAY]++] = (uint32_t)rayIdx(D, a, s, w);
                }
            }
        counts[QC_RAY] += T.count[QC_RAY];
        while (T.count[QC_RAY] > 0) {
            const uint32_t r = T.rayQ[--T.count[QC_RAY]];
            if (meshRayPhase(D, T, r, st)) T.rayQ[R + T.count[QC_BODYRAY]++] = r;
        }
        counts[QC_BODYRAY] += T.count[QC_BODYRAY];
        while (T.count[QC_BODYRAY] > 0) bodyRayPhase(D, T, T.rayQ[R + --T.count[QC_BODYRAY]], st);
        // cars
        for (int g = 0; g < h->N; g += PHASE_ARENAS) {
            auto each = [&](auto&& fn) {
                for (int s = MAX_CARS - 1; s >= 0; s--)
                    for (int la = 0; la < PHASE_ARENAS && g + la < h->N; la++)
                        if (1 + s < arenaBodies(D, g + la)) fn(dt[s * PHASE_ARENAS + la], s, la);
            };
            std::memset(ds->done, 0, sizeof ds->done);
            each([&](DriveThread& t, int s, int la) {
                t.s = s;
                t.la = la;
                t.a = g + la;
                driveLoad(D, T, t, *ds);
                if (t.finished) ds->done[la] |= 1u << s;
            });
            for (bool all = false; !all;) {
                std::vector<DriveThread*> ran;
                all = true;
                each([&](DriveThread& t, int, int la) {
                    if (!t.finished && !(t.deps & ~ds->done[la])) {
                        driveRun(t, *ds);
                        ran.push_back(&t);
                    }
                });
                for (DriveThread* t : ran) ds->done[t->la] |= 1u << t->s;
                each([&](DriveThread& t, int, int) { all &= t.finished; });
                if (!all && ran.empty()) return -1;
            }
            each([&](DriveThread& t, int, int) { driveStore(D, T, t); });
        }
        // pairs
        for (int g = 0; g < h->N; g += PHASE_ARENAS) {
            auto each = [&](auto&& fn) {
                for (int b = MAX_BODIES - 1; b >= 0; b--)
                    for (int la = 0; la < PHASE_ARENAS && g + la < h->N; la++)
                        if (b < arenaBodies(D, g + la)) fn(bt[b * PHASE_ARENAS + la], b, la);
            };
            std::memset(sh->need, 0, sizeof sh->need);
            each([&](PairThread& t, int b, int la) {
                t.b = b;
                t.la = la;
                t.a = g + la;
                t.nb = arenaBodies(D, t.a);
                pairLoad(D, T, t, *sh, tick == 0);
            });
            each([&](PairThread& t, int, int) { pairPick(D, t, *sh); });
            each([&](PairThread& t, int b, int) {
                const BodyStatics o = pairStatics(D, t, st);
                const uint32_t dyn = pairDynamics(D, t, *sh);
                const uint32_t m0 = phaseAtomicAdd(&T.count[b == 0 ? QC_BALLMESH : QC_CARMESH], (uint32_t)bitCount(o.meshes));
                const uint32_t p0 = phaseAtomicAdd(&T.count[QC_PLANE], (uint32_t)bitCount(o.planes));
                const uint32_t d0 = phaseAtomicAdd(&T.count[b == 0 ? QC_CARBALL : QC_CARCAR], (uint32_t)bitCount(dyn));
                pairStore(D, T, t, o, dyn, m0, p0, d0);
                pairNeed(t, o, *sh);
                statics[b * PHASE_ARENAS + t.la] = o;
            });
            each([&](PairThread& t, int b, int la) {
                pairStoreHead(D, T, t, statics[b * PHASE_ARENAS + la], by_bodies ? sh->need[la] : sh->need[la] | PN_DYN);
            });
            for (int la = 0; la < PHASE_ARENAS; la++)
                if (arenaHasContacts(sh->need[la]) && !(arenaByBodies(sh->need[la]) && by_bodies))
                    T.solveQ[T.count[QC_SOLVE]++] = (uint32_t)(g + la);
        }
        // contacts, islands
        for (int k = 0; k < NUM_TASK_TYPES; k++) {
            const int type = QC_CARMESH + k;
            for (uint32_t i = T.count[type]; i-- > 0;) {
                const uint32_t res = (uint32_t)resultBase(type) * (uint32_t)D.N + i;
                if (type == QC_CARCAR) carCarPhase(D, T, res);
                else findPhase(D, T, res);
            }
        }
        for (uint32_t i = std::min(T.count[QC_TRI], T.candCap); i-- > 0;) trianglePhase(D, T, i);
        for (uint32_t i = T.count[QC_PLANE]; i-- > 0;) planePhase(D, T, (uint32_t)resultBase(QC_PLANE) * (uint32_t)D.N + i, st);
        for (uint32_t i = T.count[QC_DEEP]; i-- > 0;) deepPhase(D, T, T.deepQ[i], epa.get(), st);
        for (uint32_t i = T.count[QC_COMBINE]; i-- > 0;) combinePhase(D, T, T.combineQ[i], st);
        for (uint32_t i = T.count[QC_SOLVE]; i-- > 0;) solvePhase(D, T, (int)T.solveQ[i], *ss, OneLane{}, st);
        for (uint32_t i = T.count[QC_BODY]; i-- > 0;) bodyPhase(D, T, T.bodyQ[i], st);
        // finish
        for (int g = 0; g < h->N; g += PHASE_ARENAS) {
            auto each = [&](auto&& fn) {
                for (int b = 0; b < MAX_BODIES; b++)
                    for (int la = 0; la < PHASE_ARENAS && g + la < h->N; la++)
                        if (b < arenaBodies(D, g + la)) fn(ft[b * PHASE_ARENAS + la], b, la);
            };
            auto eachPad = [&](auto&& fn) {
                for (int p = 0; p < NUM_PADS; p++)
                    for (int la = 0; la < PHASE_ARENAS && g + la < h->N; la++)
                        if (arenaBodies(D, g + la) > 1) fn(p, la);
            };
            eachPad([&](int p, int la) { padLoad(D, g + la, la, p, *fs); });
            std::memset(fs->picked, 0, sizeof fs->picked);
            std::memset(fs->touched, 0, sizeof fs->touched);
            each([&](FinishThread& t, int b, int la) {
                t.body = b;
                t.la = la;
                t.a = g + la;
                t.nb = arenaBodies(D, t.a);
                finishBody(D, T, t, *fs);
                if (b > 0) finishPads(D, t, *fs);
            });
            eachPad([&](int p, int la) { finishPad(D, g + la, la, p, *fs); });
            each([&](FinishThread& t, int b, int) {
                if (b > 0) finishBoost(D, t, *fs);
                else finishArena(D, t, *fs);
            });
        }
        for (int k = QC_CARMESH; k < QC_WORDS; k++) {
            counts[k] += T.count[k];
            T.count[k] = 0;
        }
    }
    stats[0] += st.nStatic;
    stats[1] += st.nCulled;
    stats[2] += st.nMissed;
    stats[3] += st.nRows;
    return RSB_OK;
}

// `ticks` ticks of every arena's ball in a world without cars, by arenaTick (ref) and by the
// ball's own tick: the number of (arena, tick) pairs whose records differ, and in seen[] how many
// ticks had a list made, contacts, more than one manifold with contacts, and an overflowed list.
int64_t rsb_host_ball_ticks_differ(rsb_handle* h, int32_t ticks, int64_t* seen) {
    EngineView D;
    std::memset(&D, 0, sizeof D);
    D.S = h->S.view;
    D.P = h->P;
    D.N = h->N;
    std::unique_ptr<ArenaSim> A(new ArenaSim());
    std::unique_ptr<EpaWork> epa(new EpaWork());
    std::unique_ptr<BallContacts> C(new BallContacts());
    std::unique_ptr<BallRows> R(new BallRows());
    int64_t bad = 0;
    for (int a = 0; a < h->N; a++) {
        World& W = A->W;
        W.epa = epa.get();
        W.S = &D.S;
        W.P = &D.P;
        A->teamSize = A->numCars = 0;
        W.nc = 0;
        W.nb = 1;
        W.status = 0;
        W.noRot[0] = 1;
        BallP p;
        loadPlanes(p, h->ball.data(), a, h->N);
        applyBallState(p, ballStateOf(p));
        ballBodyOf(D, p, W.b[0]);
        BallSim s;
        ballSimInit(D, p, s);
        A->tickCount = 0;
        A->status = 0;
        A->goalTeam = -1;
        A->touchedMask = 0;
        A->rngKey = 0;
        W.cull = 0;
        W.cullAudit = 0;
        W.nStatic = W.nCulled = W.nMissed = 0;
        W.cullMissed = 0;
        W.nRows = 0;
        uint16_t list[BALL_LIST], hits[BALL_LIST];
        BallBox box;
        for (int t = 0; t < ticks; t++) {
            arenaTick(*A);
            if (ballTickPairs(D, s)) {
                ballListMake(D, s, list);
                seen[0]++;
                seen[3] += s.listN == BALL_LIST_OVER;
            }
            C->blocks = 0;
            ballBoxOf(D.P, s.xf, box);
            // every other tick the triangles that pass the first tests only, as the kernel takes them
            int n = s.listN;
            if (t & 1) {
                n = ballReadsList(D.P, s) ? s.listN : 0;
                const int all = n;
                if (n > 0) n = 0;
                for (int k = 0; k < all; k++)
                    if (ballNear(D, s.xf, box, list[k] >> 10, list[k] & 1023)) hits[n++] = list[k];
            }
            ballTickSolve(D, s, t & 1 ? hits : list, n, *C, *R);
            seen[1] += C->blocks > 0;
            seen[2] += C->blocks > 1;
            const rsb_ball_state x = ballStateOf(ballRecordOf(W.b[0])), y = ballStateOf(ballSimRecord(p, s));
            if (std::memcmp(&x, &y, sizeof x) != 0) {
                bad++;
                break;
            }
        }
    }
    return bad;
}

// The first word at which the records of two handles differ, as plane * 2^40 + index, or -1.
int64_t rsb_host_records_differ(const rsb_handle* x, const rsb_handle* y) {
    const std::vector<uint32_t>* p[4] = {&x->ball, &x->car, &x->pad, &x->arena};
    const std::vector<uint32_t>* q[4] = {&y->ball, &y->car, &y->pad, &y->arena};
    for (int k = 0; k < 4; k++)
        for (size_t i = 0; i < p[k]->size(); i++)
            if ((*p[k])[i] != (*q[k])[i]) return ((int64_t)k << 40) + (int64_t)i;
    return -1;
}

}  // extern "C"
