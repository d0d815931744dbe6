// Batch-union iteration (strip_union.cuh) for batches of up to
// 64 rows x 32 columns in 128-thread CTAs (batches of 4 events): on request only.
#include "strip_union.cuh"

namespace jpet {

const UnionOps& union_ops_64x32n4() {
  static const UnionOps ops = UnionHost<UShape<4, 4, 4, 2, 4>>::ops();
  return ops;
}

}  // namespace jpet
