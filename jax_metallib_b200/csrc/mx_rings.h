// The rings of mx_prefill_kernel, in plain C++: a host program can check what its waits rely on.
//
// A wait names a phase of a slot by its parity, so that it also passes while the phase before is still on its way, unless that
// one is known to be complete.  A group of converters takes every kGroups-th stage and therefore does not see every phase of
// every slot.  For stage c it waits, in this order, for the raw weights of its box, for stage c - slots to have retired (where
// there is one), and for its activations.
#pragma once

namespace qmm {
namespace mxp {

constexpr int kStageK = 128;     // k per stage: waits and arrivals cost a warp some 100 clocks each, a stage of 64 k was bound by them
constexpr int kGroups = 2;       // warpgroups of converters
constexpr int kConsumed = 8;     // stages whose retirement can be asked for

struct Rings {
  int slots;            // stages of converted weights in TMEM
  int x_stages;         // stages of activations in shared memory
  int raw_boxes;        // boxes of raw weights: 128 bytes of each column
  int stages_per_box;
};

// bits: of a code; rows: of a tile for each promoter thread, at most (32, 64 or 96)
constexpr Rings rings(int bits, int rows) {
  // activations and raw weights in flight: a copy takes about 1 us from request to arrival, a stage's MMAs 0.1 - 0.4 us
  return {rows == 96 ? 2 : 4, rows == 96 ? 3 : (rows == 64 ? 4 : (bits == 8 ? 6 : 8)), rows == 32 && bits == 8 ? 6 : 4,
          128 * 8 / bits / kStageK};
}

// Activations: a group sees every phase of a slot, or the stage before in the slot has retired when the group comes to its wait.
// Boxes of two stages: both groups see every box, but for the last one of a tile with an odd number of stages; of five and more,
// the last stage of the box before in its slot has retired then, one and three leave each group slots of its own.
constexpr bool sound(const Rings& r) {
  return (r.x_stages % kGroups == 0 || r.slots <= r.x_stages) && r.raw_boxes % kGroups == 0 &&
         (r.stages_per_box == 1 || (r.raw_boxes == 4 && r.slots <= 4)) && r.slots <= kConsumed && r.x_stages <= kConsumed;
}

}  // namespace mxp
}  // namespace qmm
