// Kernels of the FP32 row engine with 5 columns of a transform per lane.
#include "qg_rows.cuh"

namespace qg {
extern const RowsTable kRowsTable5;
QG_ROWS_TABLE(5)
}  // namespace qg
