// Dispatch of the Family M kernels (fm_inst.cu) by precision, form and length.
#include "fft_common.hpp"
#include "launch.hpp"
#include "mixed_plan.hpp"

namespace b200fft {

#define FM_DECLARE(p, f)                                                       \
  MixedKernel fm_##p##_##f##_0(int L, int kind);                               \
  MixedKernel fm_##p##_##f##_1(int L, int kind);                               \
  MixedKernel fm_##p##_##f##_2(int L, int kind);                               \
  MixedKernel fm_##p##_##f##_3(int L, int kind);                               \
  MixedKernel fm_##p##_##f##_4(int L, int kind);                               \
  MixedKernel fm_##p##_##f##_5(int L, int kind);                               \
  static MixedKernel find_##p##_##f(int L, int kind) {                         \
    return L < kMixedCut[0]   ? fm_##p##_##f##_0(L, kind)                      \
           : L < kMixedCut[1] ? fm_##p##_##f##_1(L, kind)                      \
           : L < kMixedCut[2] ? fm_##p##_##f##_2(L, kind)                      \
           : L < kMixedCut[3] ? fm_##p##_##f##_3(L, kind)                      \
           : L < kMixedCut[4] ? fm_##p##_##f##_4(L, kind)                      \
                              : fm_##p##_##f##_5(L, kind);                     \
  }
// ranges of lengths of the compilation units (FM_LO / FM_HI in build.py)
static constexpr int kMixedCut[5] = {136, 351, 801, 1201, 2049};
FM_DECLARE(32, 0)
FM_DECLARE(32, 1)
FM_DECLARE(32, 2)
FM_DECLARE(64, 0)
FM_DECLARE(64, 1)
FM_DECLARE(64, 2)

// L: complex points of the stage loop (n/2 for an even real length n, else n).
MixedKernel mixed_kernel(bool f64, int kind, bool odd, bool col, int L) {
  if (kind != KIND_C2C && col)
    return MixedKernel{};
  if (!mixed_length_ok(L, col) &&
      (col || !mixed_pow2_row(L, f64 ? 16 : 8, kind)))
    return MixedKernel{};
  if (kind == KIND_C2C)
    return f64 ? (col ? find_64_0(L, kind) : find_64_1(L, kind))
               : (col ? find_32_0(L, kind) : find_32_1(L, kind));
  const int k = kind | (odd ? 4 : 0);
  return f64 ? find_64_2(L, k) : find_32_2(L, k);
}

} // namespace b200fft
