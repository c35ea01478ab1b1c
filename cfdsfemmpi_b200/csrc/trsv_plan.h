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
//
// When the chains of rows are the better schedule (ilu_trsv_chains, no groups).
// P = rows / dependency levels is how many rows can be solved at once.  Groups pay
// for bringing their inputs into shared memory, chains for a trip through L2 at
// every level.  Times of a solve in us, groups / chains:
//  - level order: a group's inputs are nearly all from elsewhere (12 to 17 a row), a
//    load after another for each lane, and a level cannot start before its groups
//    have them.  256^2 quads in random order, ILU(0), P = 3,476: 225 / 98; ILU(3),
//    734: 2,718 / 161; hex8 40^3 in random order, ILU(0), 1,276: 742 / 154; O-grid in
//    Cuthill-McKee order, ILU(3), 25.8: 2,115 / 1,842; 24^2 quads, ILU(1), 22.3: 46 / 39;
//    the other way at 21.4 (hex8 8^3, ILU(0)): 52 / 62; at 15.2 (200^2 quads in random
//    runs of 8, ILU(3)): 2,503 / 4,079.  Long rows move the line, by the blocks of P
//    rows: hex8 12^3, ILU(1), 14.0 rows of 33.5: 391 / 318; 8^3, ILU(1), 6.6 of 29.6:
//    131 / 251.
constexpr double TRSV_LEVEL_P = 22.0, TRSV_LEVEL_BLOCKS = 300.0;
//  - rows to all warps in turn: a group solves its rows one after another, whatever P
//    is.  hex8, ILU(2), 500 to 750 rows a group, 40^3 / 48^3 / 56^3 (P = 82, 117, 157):
//    5,508 / 6,746, 9,544 / 8,121, 14,974 / 9,679; with 31 to 120 rows a group and
//    P = 177 (hex8 30^3 in random runs of 32 and 256, ILU(1)): 290 / 1,113, 391 / 1,105.
constexpr double TRSV_CYCLIC_P = 100.0;
constexpr int TRSV_CYCLIC_ROWS = 256;
//  - strands: a group takes about 8.5 us from its ticket to its end and an SM has one
//    at a time; a level takes a chain 0.9 us and 0.09 (3x3) or 0.14 (4x4) a block of a
//    row.  200^2 quads in random runs of 12, 16 and 32, ILU(0): 164 / 110, 157 / 135,
//    149 / 209; hex8 30^3 in runs of 12: 170 / 211.
constexpr double TRSV_GROUP_US = 8.5, TRSV_LEVEL_US = 0.9;
constexpr double trsv_block_us(int nb) { return nb == 4 ? 0.14 : 0.09; }

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
  bool chains = false;               // chains of rows are the better schedule (above)
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

// Builds the plan of the lower (upper = false) or upper solve for nb x nb blocks;
// with `choose`, no groups where chains are better.
void build_trsv_plan(const IluPattern &f, int nb, bool upper, TrsvPlan &p, bool choose = false);

}  // namespace cfdgpu
