// Batch-union iteration (strip_union.cuh) for batches of up to
// 32 rows x 16 columns: boxes of up to 30 rows with rows of up to about 11 pixels.
#include "strip_union.cuh"

namespace jpet {

const UnionOps& union_ops_32x16() {
  static const UnionOps ops = UnionHost<UShape<4, 16, 2, 1, 4>>::ops();
  return ops;
}

}  // namespace jpet
