// Family M plans: the radices, threads per transform and transforms per CTA of
// the kernels compiled for lengths with odd prime factors (fft_mixed.cuh).
// Everything is constexpr: the kernels are instantiated from it and the
// planner describes them with it.
#pragma once

#include "fft_common.hpp"

namespace b200fft {

struct MixedPlan {
  int nst = 0;                  // radix stages
  int rad[4] = {1, 1, 1, 1};
  int P = 1;                    // threads per transform
  int TB = 1;                   // transforms per CTA
  int NT = 1;                   // threads per CTA
  int minb = 1;                 // CTAs per SM the registers are bounded for
  long long score = 0;
};

// Lengths with a compiled plan: 6..2048 (columns also 3 and 5) of factors 2, 3,
// 5, 7 and at most one 11 or 13, other than powers of two. Rows of one prime
// stage would read a whole transform per lane, so prime rows stay generic.
constexpr int kMixedMaxL = 2048;
constexpr bool mixed_factors_ok(int L) {
  int m = L;
  for (int p = 2; p <= 7; ++p)
    while (m % p == 0)
      m /= p;
  return m == 1 || m == 11 || m == 13;
}
constexpr bool mixed_length_ok(int L, bool col) {
  if (L < 3 || L > kMixedMaxL || is_pow2(L) || !mixed_factors_ok(L))
    return false;
  return col || !(L == 3 || L == 5 || L == 7 || L == 11 || L == 13);
}

// Power-of-two rows that take a compiled plan too (R2C/C2R rows by their half
// length): fewer points per thread and more CTAs per SM than the row tiles of
// cfg_static, and short rows read as runs of 2 to 4 lanes instead of a row per
// lane. 400 MB passes, row tile -> compiled plan, TB/s:
//   C2C FP32: 8 points 3.2 -> 5.6, 16 3.2 -> 5.5, 32 5.1 -> 5.5, 64 6.0 -> 6.4,
//     128 5.9 -> 6.3, 256 5.8 -> 6.4, 512 5.7 -> 6.0, 2048 4.3 -> 4.8,
//     4096 4.2 -> 4.6 (1024 points 5.4 -> 5.3 stay);
//   C2C FP64: 8 3.5 -> 5.6, 16 5.5 -> 6.5, 128 5.7 -> 6.2, 256 6.3 -> 6.4,
//     2048 5.0 -> 5.2 (32, 64, 512, 1024 and 4096 stay: 6.5, 6.4, 6.2 -> 5.7, 5.1,
//     5.5 -> 4.8);
//   R2C FP32 of 2 x 8 3.4 -> 5.5, 2 x 16 4.1 -> 4.5, 2 x 64 5.6 -> 5.7, 2 x 128 5.4 ->
//     5.8 (2 x 256 stays; 2 x 1024 5.5 -> 5.4 and 2 x 2048 4.2 -> 4.1 stay);
//   R2C FP64 of 2 x 8 4.7 -> 5.3, 2 x 16 4.7 -> 5.7, 2 x 64 5.8 -> 6.3, 2 x 128 5.2 ->
//     5.6, 2 x 256 5.3 -> 5.5, 2 x 1024 3.9 -> 4.5, 2 x 2048 3.8 -> 4.3 (2 x 512 stays);
//   C2R FP32 of 2 x 16 3.5 -> 4.4, 2 x 128 5.4 -> 5.6, 2 x 1024 4.3 -> 5.1,
//     2 x 2048 2.0 -> 3.8 (2 x 256 5.8 -> 5.6 stays);
//   C2R FP64 of 2 x 16 4.5 -> 5.7, 2 x 64 5.7 -> 5.9, 2 x 1024 2.8 -> 4.0,
//     2 x 2048 2.8 -> 4.1 (2 x 512 4.8 -> 4.3 stays).
constexpr bool mixed_pow2_row(int L, int es, int kind) {
  if (L < 8 || !is_pow2(L))
    return false;
  if (kind == KIND_R2C && es == 8 && L >= 1024)
    return false;
  if (kind != KIND_C2C)
    return L <= 2048 && !(es == 8 && L == 256) && !(es == 16 && L == 512);
  return es == 8 ? L <= 4096 && L != 1024
                 : L <= 2048 && L != 32 && L != 64 && L != 512 && L != 1024;
}

constexpr int ce_div_up(int a, int b) { return (a + b - 1) / b; }

// Rows whose P threads fill a warp to 7/8 or more (32 / P transforms each, the
// lanes left over repeat the first ones) stay within their warps and exchange
// with warp barriers; other rows and all columns pack P x TB threads. (R2C rows
// of 2 x 120 points on 8 threads 5.1 TB/s; with P = 20 or 25 the repeated lanes
// cost more than the block barriers: 500-point rows 4.3 against 4.7.)
constexpr bool mixed_warped(bool col, int P) { return !col && P <= 32 && 32 / P * P >= 28; }
constexpr int mixed_threads(bool col, int P, int TB) {
  return mixed_warped(col, P) ? ce_div_up(TB, 32 / P) * 32 : P * TB;
}

// Registers that hold E points per thread and their butterflies with few spills
// (from the sweep below).
constexpr int mixed_regs(int es, int E) {
  if (es == 8)
    return E <= 6 ? 32 : E <= 8 ? 40 : E <= 15 ? 48 : E <= 16 ? 56 : E <= 20 ? 64
           : E <= 27 ? 72 : 96;
  return E <= 6 ? 56 : E <= 10 ? 64 : E <= 14 ? 80 : E <= 16 ? 96 : E <= 20 ? 104
         : E <= 22 ? 112 : 128;
}

// Score of one plan (higher is better; -1: does not fit). It models what the
// sweep over about 1500 plans (17 lengths of 36..1000 points, both layouts and
// precisions, 400 MB passes) showed:
//  * CTAs per SM: one resident CTA runs its load, exchange and store phases
//    one after another (3.5-3.8 TB/s), 2 reach 4.4-5.2, 4 and more 5.4-6.3;
//  * points in flight: about 100 KB per SM are wanted;
//  * one more stage is one more exchange (15x15 against 9x5x5 points:
//    FP32 5.7 against 5.3 TB/s, 15x20 against 5x6x10: 5.4 against 4.6);
//  * idle slots: butterflies that do not fill the P threads;
//  * uneven radices and more than 24 points per thread cost registers;
//  * column segments of 64 bytes (`half`) instead of 128: FP32 300 points 3.4
//    TB/s against 5.4; they pay where whole tiles leave one CTA per SM (900
//    points 3.9 against 3.2);
//  * rows whose lanes read runs of under 64 bytes, and several
//    butterflies per thread (175-point FP64 columns as 5x5x7 on 18 threads 2.9,
//    on 35 threads 5.2; 640-point FP32 columns as 8x8x10 on 22 threads 2.8, as
//    20x32 on 32 threads 4.4).
constexpr long long mixed_score(int L, int es, bool col, int n, const int *rad, int P,
                                bool half, MixedPlan *out) {
  int E = 0, slot = 0, kmax = 1, rmin = 1 << 20, rmax = 0;
  for (int s = 0; s < n; ++s) {
    const int B = L / rad[s], K = ce_div_up(B, P);
    E = ce_max(E, K * rad[s]);
    kmax = ce_max(kmax, K);
    slot += K * P * 1000 / B;
    rmin = ce_min(rmin, rad[s]);
    rmax = ce_max(rmax, rad[s]);
  }
  slot /= n;
  if (E > (es == 8 ? 32 : 25))
    return -1;
  const int regs = mixed_regs(es, E);
  int TB = 1;
  if (col) {
    TB = 128 / es;
    while (TB * P < 96 && TB < 64)
      TB *= 2;
    if (half)
      TB = 64 / es;
  } else {
    TB = mixed_warped(col, P) ? 4 * (32 / P) : ce_max(1, (128 + P / 2) / P);
  }
  const int NT = mixed_threads(col, P, TB), NTr = ce_div_up(NT, 32) * 32;
  if (NT > 1024)
    return -1;
  const int pitch = L + ((rad[0] % 2 == 0 && !col) ? L / rad[0] : 0);
  const long long smem = n > 1 ? static_cast<long long>(TB) * pitch * es : 0;
  int occ = ce_min(65536 / (NTr * regs), 2048 / NTr);
  if (smem > 0)
    occ = ce_min(occ, static_cast<int>(233472 / (smem + 1024)));
  occ = ce_min(occ, 32);
  if (occ < 1)
    return -1;
  const long long flight = static_cast<long long>(occ) * TB * L * es / 1024;
  long long sc = 1000000000ll * occ / (10 * occ + 6) * 10;      // occ / (occ + 0.6)
  sc = sc / (flight + 15) * flight;
  long long cost = 1000 + 400 * (n - 2) + (slot - 1000) / 4 +
                   60 * (rmax - rmin) / rmin + (E > 24 ? 50 : 0);
  cost += 50 * (kmax - 1) + (kmax > 2 ? 100 * (kmax - 2) : 0) + (n > 3 ? 150 : 0);
  if (!col && P * es < 64)
    cost += P * es < 32 ? 300 : 150;
  if (half)
    cost += 200;
  sc = sc / cost;
  if (sc > out->score) {
    out->score = sc;
    out->nst = n;
    for (int s = 0; s < 4; ++s)
      out->rad[s] = s < n ? rad[s] : 1;
    out->P = P;
    out->TB = TB;
    out->NT = NT;
    out->minb = occ;
  }
  return sc;
}

// Every thread count that makes some stage come out even.
constexpr void mixed_try(int L, int es, bool col, int n, const int *asc, MixedPlan *out) {
  int rad[4] = {1, 1, 1, 1}; // columns: smaller radices first; rows: larger first
  for (int s = 0; s < n; ++s)
    rad[s] = col ? asc[s] : asc[n - 1 - s];
  for (int s = 0; s < n; ++s)
    for (int k = 1; k <= 4; ++k)
      for (int half = 0; half < (col && L > 256 ? 2 : 1); ++half)
        mixed_score(L, es, col, n, rad, ce_div_up(L / rad[s], k), half != 0, out);
}

constexpr MixedPlan mixed_plan(int L, int es, bool col) {
  MixedPlan best;
  const int rm = es == 8 ? 32 : 25; // radix-32 (25) butterflies still fit the registers
  int r[4] = {1, 1, 1, 1};
  if (col && L <= rm) { // one thread per transform, no exchange
    r[0] = L;
    mixed_try(L, es, col, 1, r, &best);
  }
  for (int a = 2; a * a <= L; ++a) {
    if (L % a != 0)
      continue;
    const int La = L / a;
    if (a <= rm && La <= rm) {
      r[0] = a;
      r[1] = La;
      mixed_try(L, es, col, 2, r, &best);
    }
    for (int b = a; a <= rm && b * b <= La; ++b) {
      if (La % b != 0)
        continue;
      const int Lb = La / b;
      if (b <= rm && Lb <= rm) {
        r[0] = a;
        r[1] = b;
        r[2] = Lb;
        mixed_try(L, es, col, 3, r, &best);
      }
      for (int c = b; L > 512 && b <= rm && c * c <= Lb; ++c)
        if (Lb % c == 0 && Lb / c <= rm) {
          r[0] = a;
          r[1] = b;
          r[2] = c;
          r[3] = Lb / c;
          mixed_try(L, es, col, 4, r, &best);
          r[3] = 1;
        }
      r[2] = 1;
    }
  }
  return best;
}

} // namespace b200fft
