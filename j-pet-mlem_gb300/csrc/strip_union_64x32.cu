// Batch-union iteration (strip_union.cuh) for batches of up to
// 64 rows x 32 columns, 256 threads: 2 mm pixels at sigma 10 / 42, 1 mm at 5 / 20.
#include "strip_union.cuh"

namespace jpet {

const UnionOps& union_ops_64x32() {
  static const UnionOps ops = UnionHost<UShape<8, 8, 4, 1, 2>>::ops();
  return ops;
}

}  // namespace jpet
