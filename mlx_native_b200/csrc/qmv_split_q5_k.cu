// Q5_K instances of the split mat-vec (qmv_split.cuh); one file per block type so that they compile side by side.
#include "qmv_split.cuh"

namespace mlxn {
template cudaError_t sp_run<GT_Q5_K>(const QmvArgs *, int, int, uint8_t *, int *, cudaStream_t);
}
