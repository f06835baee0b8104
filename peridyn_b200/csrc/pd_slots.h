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

// Record a slot's evaluation reads: its neighbour where the lane has the
// bond (entry: the stencil offset, or the index of an explicit slice),
// otherwise the lane's own, so that a block's evaluation reads the records
// of that block only -- callers may hold no others -- and none for nothing.
PD_HD int32_t slot_record(bool stencil, int32_t own, int32_t entry, bool live) {
    return !live ? own : stencil ? own + entry : entry;
}

// Record a lane stands for: its particle's, or for a padding lane that of
// the slice's first particle (every slice has one).
PD_HD int32_t lane_record(int32_t p, int32_t tinfo) { return tinfo >= 0 ? p : p & ~31; }

// Pair parameters of a slot: those of types (tp, tq) where the lane has the
// bond, otherwise the block's first pair.
PD_HD int32_t slot_pair(int32_t pair_base, int32_t nt, int32_t tp, int32_t tinfo_q, bool live) {
    return live ? pair_base + tp + (tinfo_q & 255) * nt : pair_base;
}

}  // namespace pd
