// Row form of the x / z pass for d = 5.
#include "rows_kernels.cuh"

namespace sdim {

const RowOps& row_ops_5() {
  static const RowOps ops = row_ops<5>();
  return ops;
}

}  // namespace sdim
