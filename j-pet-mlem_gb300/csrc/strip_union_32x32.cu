// Batch-union iteration (strip_union.cuh) for batches of up to
// 32 rows x 32 columns: wide rows of short boxes (4 mm pixels at sigma_z 14).
#include "strip_union.cuh"

namespace jpet {

const UnionOps& union_ops_32x32() {
  static const UnionOps ops = UnionHost<UShape<4, 8, 4, 1, 4>>::ops();
  return ops;
}

}  // namespace jpet
