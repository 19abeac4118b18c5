// Kernels of the FP32 row engine with 4 columns of a transform per lane.
#include "qg_rows.cuh"

namespace qg {
extern const RowsTable kRowsTable4;
QG_ROWS_TABLE(4)
}  // namespace qg
