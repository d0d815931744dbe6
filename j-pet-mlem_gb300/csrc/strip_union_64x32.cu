// Batch-union iteration (strip_union.cuh) for batches of up to
// 64 rows x 32 columns, 256 threads: boxes of up to 64 rows with rows of up to 28
// pixels, and events that no batch takes.
#include "strip_union.cuh"

namespace jpet {

const UnionOps& union_ops_64x32() {
  static const UnionOps ops = UnionHost<UShape<8, 8, 4, 1, 2>>::ops();
  return ops;
}

}  // namespace jpet
