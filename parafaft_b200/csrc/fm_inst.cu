// Instantiations of the Family M kernels. The build compiles this file once
// per precision, form and range of lengths (FM_PREC 32/64, FM_FORM 0 columns,
// 1 rows, 2 real rows; FM_LO <= L < FM_HI), so that the set compiles in
// parallel; FM_NAME is the unit's lookup function.
#include <atomic>
#include <climits>
#include <utility>

#include "fft_mixed.cuh"
#include "launch.hpp"

namespace b200fft {
namespace {

#if FM_PREC == 64
using Real = double;
#else
using Real = float;
#endif

// Opt in to more than 48 KiB of shared memory, once per kernel and device.
template <size_t SMEM, class Kern> cudaError_t configure(Kern kern, std::atomic<int> &mask) {
  if constexpr (SMEM > 48 * 1024) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 31 || !(mask.load() & (1 << dev))) {
      const cudaError_t e = cudaFuncSetAttribute(
          kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(SMEM));
      if (e != cudaSuccess)
        return e;
      if (dev >= 0 && dev < 31)
        mask.fetch_or(1 << dev);
    }
  }
  return cudaSuccess;
}

template <int L, int KIND, bool ODD, bool COL>
cudaError_t launch_one(const PassArgs &a, unsigned flip, cudaStream_t st) {
  using K = KM<Real, L, KIND, ODD, COL>;
  static std::atomic<int> mask{0};
  const cudaError_t e = configure<K::smem_bytes()>(fft_mixed_kernel<K>, mask);
  if (e != cudaSuccess)
    return e;
  const long long grid = (a.total + K::TB - 1) / K::TB;
  if (grid <= 0)
    return cudaSuccess;
  if (grid > INT_MAX)
    return cudaErrorInvalidConfiguration;
  return launch_chained(a.chained != 0, fft_mixed_kernel<K>, static_cast<unsigned>(grid), K::NT,
                        K::smem_bytes(), st, a, flip);
}

template <int L, int KIND, bool ODD, bool COL>
cudaError_t launch_group(const PassArgs *items, const int2 *map, long long ntiles, unsigned flip,
                         cudaStream_t st) {
  using K = KM<Real, L, KIND, ODD, COL>;
  static std::atomic<int> mask{0};
  const cudaError_t e = configure<K::smem_bytes()>(fft_mixed_group_kernel<K>, mask);
  if (e != cudaSuccess)
    return e;
  if (ntiles <= 0)
    return cudaSuccess;
  if (ntiles > INT_MAX)
    return cudaErrorInvalidConfiguration;
  fft_mixed_group_kernel<K>
      <<<static_cast<unsigned>(ntiles), K::NT, K::smem_bytes(), st>>>(items, map, flip);
  return cudaGetLastError();
}

template <int L, int KIND, bool ODD, bool COL> constexpr MixedKernel kernel() {
  return MixedKernel{&launch_one<L, KIND, ODD, COL>, &launch_group<L, KIND, ODD, COL>,
                     KM<Real, L, KIND, ODD, COL>::TB};
}

// KINDX: KIND_C2C; KIND_R2C or KIND_C2R of real length 2L, or of odd length L (| 4).
template <int L, int KINDX> constexpr MixedKernel entry() {
#if FM_FORM == 0
  if constexpr (mixed_length_ok(L, true))
    return kernel<L, KIND_C2C, false, true>();
#elif FM_FORM == 1
  if constexpr (mixed_length_ok(L, false) || mixed_pow2_row(L, 2 * sizeof(Real), KIND_C2C))
    return kernel<L, KIND_C2C, false, false>();
#else
  if constexpr (mixed_length_ok(L, false) || mixed_pow2_row(L, 2 * sizeof(Real), KINDX & 3)) {
    if constexpr ((KINDX & 4) == 0)
      return kernel<L, KINDX, false, false>();
    else if constexpr (L % 2 == 1)
      return kernel<L, KINDX & 3, true, false>();
  }
#endif
  return MixedKernel{};
}

template <int KINDX, int... I>
const MixedKernel *table(std::integer_sequence<int, I...>) {
  static const MixedKernel t[] = {entry<FM_LO + I, KINDX>()...};
  return t;
}
template <int KINDX> MixedKernel find(int L) {
  return table<KINDX>(std::make_integer_sequence<int, FM_HI - FM_LO>{})[L - FM_LO];
}

} // namespace

MixedKernel FM_NAME(int L, int kind) {
  if (L < FM_LO || L >= FM_HI)
    return MixedKernel{};
#if FM_FORM == 2
  switch (kind) {
  case KIND_R2C: return find<KIND_R2C>(L);
  case KIND_C2R: return find<KIND_C2R>(L);
  case KIND_R2C | 4: return find<(KIND_R2C | 4)>(L);
  case KIND_C2R | 4: return find<(KIND_C2R | 4)>(L);
  default: return MixedKernel{};
  }
#else
  (void)kind;
  return find<KIND_C2C>(L);
#endif
}

} // namespace b200fft
