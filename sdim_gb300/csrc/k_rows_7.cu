// Row form of the x / z pass for d = 7.
#include "rows_kernels.cuh"

namespace sdim {

const RowOps& row_ops_7() {
  static const RowOps ops = row_ops<7>();
  return ops;
}

}  // namespace sdim
