// Kernels of the FP32 row engine with 3 columns of a transform per lane.
#include "qg_rows.cuh"

namespace qg {
extern const RowsTable kRowsTable3;
QG_ROWS_TABLE(3)
}  // namespace qg
