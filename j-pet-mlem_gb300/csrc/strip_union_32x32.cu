// Batch-union iteration (strip_union.cuh) for batches of up to
// 32 rows x 32 columns: boxes of up to 30 rows with rows of up to 28 pixels.
#include "strip_union.cuh"

namespace jpet {

const UnionOps& union_ops_32x32() {
  static const UnionOps ops = UnionHost<UShape<4, 8, 4, 1, 4>>::ops();
  return ops;
}

}  // namespace jpet
