// Row form of the x / z pass for d = 2.
#include "rows_kernels.cuh"

namespace sdim {

const RowOps& row_ops_2() {
  static const RowOps ops = row_ops<2>();
  return ops;
}

}  // namespace sdim
