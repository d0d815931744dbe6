// Batch-union iteration (strip_union.cuh) for batches of up to
// 64 rows x 16 columns: boxes of up to 64 rows with rows of up to about 9 pixels.
#include "strip_union.cuh"

namespace jpet {

const UnionOps& union_ops_64x16() {
  static const UnionOps ops = UnionHost<UShape<8, 16, 2, 1, 2>>::ops();
  return ops;
}

}  // namespace jpet
