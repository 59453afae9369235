// The schedule of the pair kernel (pair.cuh): the sizes of its rings, the heights of its tiles and the order in which its
// decode warps fill slots and drain accumulators. Plain C++, so that a model of the kernel's waits can be built from it
// without a GPU.
#pragma once

#ifdef __CUDACC__
#define MSK_HOST_DEVICE __host__ __device__
#else
#define MSK_HOST_DEVICE
#endif

namespace msk {

constexpr int PAIR_BH = 128;             // most token rows a CTA holds of a tile; columns of an accumulator buffer
constexpr int PAIR_SLOT_K = 128;         // K of an A / B slot
constexpr int PAIR_NSLOT = 4;            // A slots; places of token rows, each PAIR_SLOT_K of PAIR_BH rows in either CTA
constexpr int PAIR_MARKS = 2 * PAIR_NSLOT;   // slots whose MMAs have their own barrier
constexpr int PAIR_GROUPS = 4;           // of decode warps: group g fills the slots g, g + PAIR_GROUPS, ... of the list of all slots
constexpr int PAIR_NST = 5;              // weight stages
constexpr int PAIR_UNITS = 4;            // units handed out ahead of their use

// Rows of each tile of an expert with c rows in n tiles: even shares, in steps of 32 (the last tile has the rest, which
// is never empty: a share is below its limit only while the limit exceeds c / n by more than the rounding).
MSK_HOST_DEVICE inline int pair_tile_rows(int c, int n) { return ((c + n - 1) / n + 31) & ~31; }

// Columns of the MMAs of a tile with `rows` rows, half of them (eight at the least) from either CTA.
MSK_HOST_DEVICE inline int pair_cols(int rows) { return (rows + 15) & ~15; }

// Token rows come a K stage at a time: the two slots 2 * stage and 2 * stage + 1, numbered through all units. Where a stage lies: a tile of more than
// PAIR_BH columns takes two places, this one and the next; a narrower one (half of its rows are PAIR_BH / 2 at the most) takes one, in
// turn with the other of the pair, so that its rows are fetched four stages ahead instead of two.
MSK_HOST_DEVICE inline unsigned pair_b_place(unsigned stage, int cols) {
  return (stage & 1u) * 2u + (cols > PAIR_BH ? 0u : (stage >> 1) & 1u);
}

// The slot whose MMAs have to be done before the rows of a stage are copied: the second one of the last stage that used any of its bytes
// (MMAs are done in order). `wide_end`: the number behind the last stage of a tile of more than PAIR_BH columns.
MSK_HOST_DEVICE inline unsigned pair_b_waits_for(unsigned stage, int cols, unsigned wide_end) {
  return 2u * (cols <= PAIR_BH && stage >= wide_end + 2u ? stage - 4u : stage - 2u) + 1u;
}

// Slots of its next unit that a decode warp fills before it drains the unit it owes (phase 0 gate/up, 1 down; cols: columns
// of the accumulators). A group's next slot is free once the MMAs have read the slot it filled before, so the first slot of a
// unit waits for MMAs of the owed unit at the latest, the second one for the unit's own first MMAs. Those need
//  - the accumulators that the owed unit holds, if either of the two is wider than a buffer;
//  - for a down unit the gate/up units of its token tile, which the owed one may be among, or the owed one of a cluster
//    that waits in the same way: nobody would move any more.
// In both cases the drain comes behind the first slot, otherwise behind the second.
MSK_HOST_DEVICE inline int pair_slots_before_drain(int owed_phase, int owed_cols, int phase, int cols) {
  return owed_phase < phase || cols > PAIR_BH || owed_cols > PAIR_BH ? 1 : 2;
}

}  // namespace msk
