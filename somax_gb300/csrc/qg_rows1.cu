// Kernels of the FP32 row engine with 1 column of a transform per lane.
#include "qg_rows.cuh"

namespace qg {
extern const RowsTable kRowsTable1;
QG_ROWS_TABLE(1)
}  // namespace qg
