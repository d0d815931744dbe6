// Batch-union iteration (strip_union.cuh) for batches of up to
// 96 rows x 40 columns: boxes of up to 96 rows with rows of up to 39 pixels.
#include "strip_union.cuh"

namespace jpet {

const UnionOps& union_ops_96x40() {
  static const UnionOps ops = UnionHost<UShape<12, 8, 5, 1, 1>>::ops();
  return ops;
}

}  // namespace jpet
