// pd_slots.h -- index arithmetic of the serial block-per-slice kernels
// (device) and its check (host).
//
// A slice walks its slots for all 32 lanes, whether a lane uses a slot or
// not: padding lanes have none, and a stencil slot that only other lanes use
// names an arbitrary record of the environment -- padding (type -1), or a
// particle of a neighbouring block, whose types are numbered differently.
#pragma once

#include "pd_ieee.h"

namespace pd {

// Pair parameters of a slot: those of types (tp, tq) where the lane has the
// bond, otherwise the block's first pair.
PD_HD int32_t slot_pair(int32_t pair_base, int32_t nt, int32_t tp, int32_t tinfo_q, bool live) {
    return live ? pair_base + tp + (tinfo_q & 255) * nt : pair_base;
}

}  // namespace pd
