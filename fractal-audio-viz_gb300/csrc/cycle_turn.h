// When an alternate-formula pixel's cycle test is due.
#pragma once

#include "scaled.h"

namespace fx {

// Whether the step that arrives at iteration `it` is followed by a cycle test
// (every 32nd from 2,048 on).
FX_HD bool cycle_turn(bool cycle, int it) { return cycle && it >= 2048 && (it & 31) == 0; }

// Whether a pixel at `it` may take its next turn before it is listed: a list
// entry has no room for what a cycle test begins (the value and the counts it
// compares with later), so a pixel whose next step ends with one waits for
// its lane.
FX_HD bool turn_before_listing(bool cycle, int it) { return !cycle_turn(cycle, it + 1); }

}  // namespace fx
