// Kernels of the FP32 row engine with 2 columns of a transform per lane.
#include "qg_rows.cuh"

namespace qg {
extern const RowsTable kRowsTable2;
QG_ROWS_TABLE(2)
}  // namespace qg
