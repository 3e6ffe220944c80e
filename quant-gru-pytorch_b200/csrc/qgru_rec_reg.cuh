// qgru_rec_reg.cuh - plan and launch interface of the register-resident recurrence (qgru_rec_reg.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "qgru_internal.h"

struct qgru_handle;

namespace qgru {

// Clusters of P CTAs own Bt batch rows, each CTA U hidden units (a multiple of 16) as U / 16 unit groups; KS warps
// share a unit group, each multiplying KST * 32 of the K (= H) inputs.
struct RecRegPlan {
    int H = 0, B = 0, sms = 0, ih_bytes = 0, cell = 0, n_table = 0;      // what the plan was made for
    bool ok = false;
    int KST = 2, KS = 1, U = 16, P = 1, Bt = 1, G = 1, D = 2;
    bool few = false;      // tiles of two to four rows take one row a thread
    size_t smem = 0;
    // W*x + bw is stored as [P][T*B][3][U]: what a CTA needs of its rows in one step is one contiguous block
    size_t ih_elements(long long N) const { return (size_t)N * 3 * P * U; }
};

// The training cells keep the gate buffer and the packed clamp masks; their W*x + bw comes clamped to one step
// beyond the operator's range on either side, so that it still tells what the clamp changed.
enum RecCell { CELL_INT_FAST = 0, CELL_INT_FAST_NOTIE = 1, CELL_INT_GENERIC = 2, CELL_FS = 3, CELL_INT_TRAIN = 4, CELL_FS_TRAIN = 5 };

struct RecRegArgs {
    int T, B, H, Hpad, reverse;
    const int8_t *r8;             // [3H][Hpad]
    const void *ih;               // [P][T*B][3][U]: W*x + bw as the cell takes it
    const uint8_t *h8;            // [B][Hpad] initial state
    OutView out;
    LinearConsts lc;              // R*h + br epilogue
    const int32_t *tables;
    int n_table;
    const float *fs_chan;         // float-storage cell: [3][C] offset, bias term, scale ratio of R*h + br
    FsConsts fs;
    // training cells: all states [(T+1)][B][H] or null, gate buffer [T*B][4H], clamp masks [T*B][H] (PM_* bits)
    float *h_all, *v;
    uint16_t *pm;
    FsTrainConsts tc;
    int U, P, Bt, NT, D, vec2;       // set by the launcher
    int *abort_flag;
    bool pdl;                     // launched beside the product before it (programmatic dependent launch)
    unsigned long long *stamp;    // start time, or null
};

typedef void (*RegKernel)(const GateConsts, const RecRegArgs);
RegKernel rec_reg_float_kernel(RecCell cell, int ih_bytes, int kst, int ks, bool hu, bool few);   // qgru_rec_reg_float.cu

// False where the form does not exist (H > 1024, no shared memory left).
bool rec_reg_plan(qgru_handle *h, int B, int sms, int ih_bytes, RecCell cell, int n_table, RecRegPlan *pl);
int rec_reg_launch(qgru_handle *h, const RecRegPlan &pl, RecRegArgs a, RecCell cell, int ih_bytes, cudaStream_t st);

}  // namespace qgru
