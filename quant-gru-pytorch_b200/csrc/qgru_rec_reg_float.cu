// qgru_rec_reg_float.cu - instantiations of the register-resident recurrence (qgru_rec_reg.cu) for the float-storage cell
// and the training cells.
#include "qgru_rec_reg_kernel.cuh"

namespace qgru {

RegKernel rec_reg_float_kernel(RecCell cell, int ih_bytes, int kst, int ks, bool hu, bool few) {
    switch (cell) {
        case CELL_INT_TRAIN: return ih_bytes == 2 ? pick<int16_t, CELL_INT_TRAIN>(kst, ks, hu, few) : pick<int32_t, CELL_INT_TRAIN>(kst, ks, hu, few);
        case CELL_FS_TRAIN: return ih_bytes == 2 ? pick<int16_t, CELL_FS_TRAIN>(kst, ks, hu, few) : pick<int32_t, CELL_FS_TRAIN>(kst, ks, hu, few);
        default: return ih_bytes == 1 ? pick<int8_t, CELL_FS>(kst, ks, hu, few) : pick<int16_t, CELL_FS>(kst, ks, hu, few);
    }
}

}  // namespace qgru
