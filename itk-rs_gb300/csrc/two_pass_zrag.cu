// The z kernels of the two-pass 3-D forward for f32 rows that end in a partial
// quad (k_z_pass<R, REF, kStoreF32Ragged>).
#include "two_pass.cuh"

namespace itkg {
namespace twopass {
namespace {
const ZFn kFma[kMaxR] = ITKG_Z_ROW(false, kStoreF32Ragged);
const ZFn kRef[kMaxR] = ITKG_Z_ROW(true, kStoreF32Ragged);
}  // namespace
const ZFn* z_row_fma_f32rag() { return kFma; }
const ZFn* z_row_ref_f32rag() { return kRef; }
}  // namespace twopass
}  // namespace itkg
