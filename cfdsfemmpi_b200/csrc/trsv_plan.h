// Schedule of a block triangular solve for the persistent kernel ilu_trsv
// (ilu_kernels.cuh), built on the host from the factor pattern.
#pragma once
#include <cstdint>
#include <vector>

#include "setup.h"

namespace cfdgpu {

constexpr int TRSV_STRANDS = 4;         // strands of rows that a CTA solves side by side
constexpr int TRSV_WARPS = 16;          // its solving warps: four per strand, taking its rows in turn
constexpr int TRSV_LOADERS = 3;         // warps of a CTA that fetch inputs of other groups
// blocks per piece, and rows (own + inputs) that a group may hold in shared
// memory: what the pieces in flight leave of it
constexpr int trsv_cap(int nb) { return nb == 4 ? 16 : 24; }
constexpr int trsv_max_slots(int nb) { return nb == 4 ? 2600 : 4200; }
// slot entries of a piece's record: a lane of the kernel reads four at once
// (block 4 p + s of 4x4 blocks, 8 p + s of 3x3 blocks, is entry 4 s + p)
constexpr int trsv_slots(int nb) { return nb == 4 ? 16 : 32; }
// How rows are put into groups and given to a group's warps (build_trsv_plan):
// Short strands (a strand is a run of rows each depending on the one before):
// on a mesh numbered without locality rows depend on rows far away, so groups
// are taken from the level order, where their inputs are long done.
constexpr int TRSV_SHORT_STRAND = 8;    // mean rows per strand below which this holds
constexpr int TRSV_LEVEL_ROWS = 128;    // rows of such a group, at most
// Otherwise groups are runs of consecutive rows, TRSV_STRANDS strands each.  When
// a row has more off-diagonal blocks than this, its own work outweighs handing
// the previous row's value on, and its rows go to all warps in turn.
constexpr int TRSV_CYCLIC_BLOCKS = 32;
// A single row with more inputs than a group may hold reads them from memory.

// One warp's unit of work: up to `cap` consecutive blocks of one row.
struct TrsvPiece {
  int32_t q0;       // first block in the factor values
  int32_t n;        // blocks | TRSV_FIRST | TRSV_LAST | TRSV_DIRECT | low bits of q0 << TRSV_Q0_SHIFT
  int32_t desc;     // its record, in units of 16 bytes
  int32_t at;       // where the row's right-hand side lies: node (lower solve) or factor row (upper)
};
constexpr int32_t TRSV_FIRST = 1 << 16, TRSV_LAST = 1 << 17, TRSV_DIRECT = 1 << 20;
constexpr int TRSV_Q0_SHIFT = 18;       // two bits: where the blocks start within 16 bytes

// Groups are listed in an order in which every input of a group belongs to the
// group itself or to an earlier one.  Slots 0..rows-1 are the group's own rows,
// slots rows..rows+next-1 its inputs ext[ext0..ext0+next) from other groups.
// The group starts once input `gate` is there: the last one that its lowest row needs.
struct TrsvGroup {
  int32_t rows, ext0, next, gate;
};

struct TrsvPlan {
  int max_slots = 0;                 // largest rows + next
  std::vector<TrsvGroup> groups;
  std::vector<int32_t> wptr;         // groups x (TRSV_WARPS + 1): pieces of each warp
  std::vector<TrsvPiece> pieces;
  // record of every piece: factor row, node, n, the row's own slot | the slot of
  // the block nearest the diagonal << 16 (counted in doubles), and the byte
  // offsets of the slots of its blocks as trsv_slots says; entries past its
  // blocks name the slot after the largest group's, which holds zero.  With
  // TRSV_DIRECT, the blocks' entries are positions in the source vector instead.
  std::vector<uint32_t> desc;
  std::vector<int32_t> ext;          // factor rows, in the order in which the group's rows come to need them
};

// Builds the plan of the lower (upper = false) or upper solve for nb x nb blocks.
void build_trsv_plan(const IluPattern &f, int nb, bool upper, TrsvPlan &p);

}  // namespace cfdgpu
