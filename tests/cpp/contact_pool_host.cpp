// step_phases_host.cpp with the engine's pool of contact points, whose size that file writes as
// MAX_BLOCKS places for each arena (`h` is the handle there).
#include <algorithm>

#include "arena_build.h"
#include "engine_host.h"
#include "phys/ball_phase.h"
#include "phys/step_phases.h"

#define MAX_BLOCKS (size_t)std::max(1, contactPairs(h->maxCars, h->S.cellStatics))
#include "step_phases_host.cpp"
