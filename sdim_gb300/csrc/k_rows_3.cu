// Row form of the x / z pass for d = 3.
#include "rows_kernels.cuh"

namespace sdim {

const RowOps& row_ops_3() {
  static const RowOps ops = row_ops<3>();
  return ops;
}

}  // namespace sdim
