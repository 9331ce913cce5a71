// cg_group.cuh -- the persistent Jacobi-PCG: interface of cg_group.cu.
#pragma once

#include <vector>

#include "nb2_internal.cuh"

namespace nb2 {

// Where the scalars of the systems ("jobs") live: entry j of every array belongs to job j.  Both
// the single solve (CgScalars, one job) and the batch (structure of arrays) point in here.
struct GroupScalars {
    double *thr, *absnew, *beta, *rr, *rrcap;
    int *iters, *done, *status, *maxit;
};

// One turn of a CTA: it works on part `part` (member `rank` of m1 x m2) of `job`; the group's
// exchange slots (16 bytes each) start at `slot0`.
struct GroupTurn {
    int job, part, rank, m1, m2, slot0;
};

// The matrix of one or several independent systems in tiles of 8 rows x 4 lanes (a warp): step s
// of a tile holds, for lane 4 i + l, the 3x3 block 4 s + l of the tile's row i, every component
// contiguous over the 32 lanes.  Rows shorter than the tile's
// longest are padded with zeros.  A system's tiles are cut into as many parts as CTAs work on it;
// columns are indices into the part's halo, the sorted list of all rows it reads (its own among
// them).  Built once per sparsity pattern; the values are copied in at the start of a solve.
struct SellPlan {
    long long steps = 0;
    int ntiles = 0, nparts = 0;
    std::vector<int> offsets;        // first row of every job, and the number of rows
    std::vector<int> job_tile;       // first tile of every job, and the number of tiles
    std::vector<int> job_part;       // first part of every job, and the number of parts
    std::vector<int> job_m1;         // a job's parts are m1 x m2 CTAs
    int *tile_row = nullptr, *tile_end = nullptr;  // [ntiles] first row, end of the rows
    int* tile_off = nullptr;         // [ntiles + 1] first step
    int* part_tile = nullptr;        // [nparts + 1] first tile
    int* halo_ptr = nullptr;         // [nparts + 1]
    int* halo = nullptr;             // rows of every part's halo
    int* own0 = nullptr;             // [nparts] halo position of the part's first own row
    unsigned short* col = nullptr;   // [steps][32]
    void* val[2] = {nullptr, nullptr};  // [steps][9][32]: double, float
    double* z = nullptr;             // the exchanged vector {value, tag}, 3 per row
    double* s = nullptr;             // K p of parts whose vectors do not fit in shared memory
    double* slots = nullptr;
    GroupTurn* turns = nullptr;      // device copy of the schedule
    int* turn_ptr = nullptr;
    std::vector<GroupTurn> h_turns, sent_turns;  // the schedule, and the one on the device
    std::vector<int> h_turn_ptr, sent_turn_ptr;
    int turns_cap = 0, nslots = 0, slots_cap = 0;
};

void sell_release(SellPlan* p);

// The plan of the block pattern cut into systems at `offsets` (block rows, first 0, last N), cached
// in the context; *out stays null where the persistent solver does not apply: no cooperative
// launch, no room, too much padding, or a halo that does not fit in shared memory.  value_bytes: of
// the values it will mostly hold (it decides how many CTAs share a system, nothing else).
int sell_plan(nb2_ctx* c, const std::vector<int>& offsets, int value_bytes, SellPlan** out);

// Copy the values in, rows of masked unknowns as zeros; then iterate every active job whose `done`
// is 0 until it stops by itself or has made its iterations of one launch (all of them when `active`
// is empty).  Nothing is waited for.  Once the stream is idle and the CG scalars are on the host
// (wait_scalars): a job that is not done takes another launch, unless group_failed says that a wait
// of the launch ran out, which leaves x undefined.
template <typename V>
int sell_fill(nb2_ctx* c, SellPlan* P, const V* K, const unsigned char* mask);
template <typename V, typename X>
int group_cg(nb2_ctx* c, SellPlan* P, GroupScalars S, const std::vector<int>& active, X* x, X* r,
             X* p, X* q, const X* inv, const float* dc);
bool group_failed(const nb2_ctx* c);

}  // namespace nb2
