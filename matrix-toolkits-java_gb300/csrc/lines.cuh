// lines.cuh -- triangular solves by tiles of lines (lines.cu): the plan of a
// factor's two sweeps and its entry points.
#pragma once

#include "internal.h"

namespace mtjg {

// A triangular operator's rows: entries [rp[i], rp[i+1]) (range 0), below (1)
// or above (2) the diagonal; desc: a row reads rows of larger index.  mode:
// the sweep's MODE (precond.cu).
struct TriOp {
    int mode, n, desc, range;
    const int *rp, *ci, *diag;
};

// Where each row of a factor sits: part (CTA), step and lane.  A vector in
// plan order has the rows of one step of one part next to each other:
// position (first step of the part + step) * lanes + lane.
struct TilePlan {
    int n = 0, kmax = 0;      // rows, entries of the longest row of either triangle
    int parts = 0, lanes = 0;
    int steps = 0;            // steps of all parts
    // one device allocation, at b64:
    double *b64 = nullptr, *y64 = nullptr, *x64 = nullptr;  // vectors in plan order
    int *row = nullptr;       // [steps * lanes]: row at each position, -1 for none
    int *pos = nullptr;       // [n]: position of each row
    int *part_step = nullptr; // [parts + 1]: first step of each part
    float *b32 = nullptr, *y32 = nullptr, *x32 = nullptr;
};

// One sweep over a plan.  A step's record: entry values [kmax][lanes],
// diagonals [lanes] and their reciprocals [lanes] (value type V), and four
// entry codes (int) per lane.  rem: what each step reads from other parts (or
// from too long ago for the ring), rem_max places a step: the entry's
// position and its place k * lanes + lane, or -1.
struct TileOp {
    int mode = 0;
    unsigned char *rec64 = nullptr, *rec32 = nullptr;
    int *rem = nullptr;       // [steps][rem_max][2]
    int rem_max = 0;
};

// The first (ascending) and second (descending) sweep of an apply.
struct TilePair {
    TilePlan *plan = nullptr;
    bool owns_plan = true;
    unsigned char *mem = nullptr;  // device: both ops' rec64 and rem
    TileOp op[2];
};

// Whether the pivots' sweep (tile_ilu) may take a plan of this many positions:
// its vector holds two values a position, indexed by int.  (The plans' own
// positions always fit one: with lines of 4 rows and mirrored triangles 2^31
// entries are at most 859 million rows, and a plan has at most twice the rows
// and 65536 positions.)
constexpr bool pivot_pairs_fit(int64_t positions) { return 2 * positions <= 0x7fffffff; }

// Plans the two sweeps; *out stays null when the rows do not form lines (see
// the rule at tile_plan) and the caller keeps the level schedules.  `plan`:
// an existing plan of the same factor to use (its transposed sweeps), or null.
int tile_pair(mtjg_ctx *ctx, const TriOp &lo, const TriOp &up, TilePlan *plan, TilePair **out);
// A sweep's values into its records.
int tile_values(mtjg_ctx *ctx, TilePair *tp, int which, const TriOp &op, const double *v, const double *diagv);
int tile_values(mtjg_ctx *ctx, TilePair *tp, int which, const TriOp &op, const float *v, const float *diagv);
// ILU(0) of `data` (the matrix's values, lo its lower triangle) in place,
// where its elimination changes only the pivots; else *factored is false and
// data as it was.
int tile_ilu(mtjg_ctx *ctx, TilePair *tp, const TriOp &lo, double *data, bool *factored);
void free_tiles_of(TilePair *&tp);
void tile_drop32(TilePair *tp);  // the FP32 records and vectors go
// x = (second) \ ((first) \ b); x may be b.
cudaError_t tile_apply(mtjg_ctx *ctx, const TilePair *tp, bool strict, const double *b, double *x, const int *status,
                       int spin);
cudaError_t tile_apply(mtjg_ctx *ctx, const TilePair *tp, bool strict, const float *b, float *x, const int *status,
                       int spin);

}  // namespace mtjg
