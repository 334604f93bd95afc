// Family M: specialised kernels for lengths with odd prime factors.
//
// The Stockham stages of fft_device.cuh with a compile-time plan per length
// (mixed_plan.hpp): radices R0 x R1 (x R2 x R3) of up to 32 points, any product
// of 2, 3, 5, 7, 11 and 13 being one register butterfly, P threads per transform
// and TB transforms per CTA. Neither P nor TB x P has to be a power of two, so a
// length gets few and even stages: 300 = 20 x 15 on 20 threads, one
// shared-memory exchange, where the runtime schedule (fft_generic_kernel) takes
// 4 x 5 x 5 x 3 with an integer division per butterfly and two tile buffers.
//
// What bounds them: HBM first, then how many CTAs an SM holds (each runs its
// load, exchange and store phases one after another). Passes of 400 MB,
// forward, back to back, runtime schedule -> here, TB/s:
//   points           FP32 rows    FP32 columns  FP64 rows    FP64 columns
//   36               2.9 -> 6.0   2.8 -> 5.8    2.8 -> 6.7   2.8 -> 6.0
//   100              2.7 -> 6.4   2.4 -> 6.1    2.7 -> 6.1   2.7 -> 6.3
//   225              2.2 -> 6.3   2.1 -> 5.8    2.2 -> 6.6   2.2 -> 5.8
//   300              2.2 -> 5.7   1.9 -> 5.4    2.4 -> 6.7   2.4 -> 5.7
//   500              2.2 -> 5.3   1.8 -> 4.8    2.4 -> 6.3   2.2 -> 5.6
//   1000             2.1 -> 4.4   1.5 -> 3.5    2.1 -> 5.0   1.6 -> 3.9
//   1225             0.8 -> 4.0   0.6 -> 2.9    1.1 -> 5.1   0.9 -> 3.3
// Long columns stay behind because a tile of 128-byte segments leaves one or
// two CTAs per SM. R2C/C2R rows pair Z[k] with Z[L-k] through one more exchange
// (2.7-5.4 TB/s). Their error is at most 1.04 of the runtime schedule's at any
// length, 0.94 of it on average.
#pragma once

#include "fft_device.cuh"
#include "mixed_plan.hpp"

namespace b200fft {

#define BF_HD __host__ __device__

// ---- butterflies of the odd primes above 5 and of their products -----------
// DFT of an odd prime p: with a_m = x_m + x_{p-m} and b_m = x_m - x_{p-m},
//   X_k, X_{p-k} = x_0 + sum_m a_m cos(2 pi k m / p) -+ i sum_m b_m sin(2 pi k m / p)
template <int p, bool FWD, typename V> struct PrimeDft {
  using T = decltype(V().x);
  static constexpr int H = (p - 1) / 2;
  template <int k, int m> static BF_D void acc(const V *a, const V *b, V &c, V &s) {
    if constexpr (m <= H) {
      constexpr T co = T(TwC<(k * m) % p, p>::c), si = T(TwC<(k * m) % p, p>::s);
      c.x += co * a[m - 1].x;
      c.y += co * a[m - 1].y;
      s.x += si * b[m - 1].x;
      s.y += si * b[m - 1].y;
      acc<k, m + 1>(a, b, c, s);
    }
  }
  template <int k> static BF_D void outs(V x0, const V *a, const V *b, V *v) {
    if constexpr (k <= H) {
      V c = x0, s = czero<V>();
      acc<k, 1>(a, b, c, s);
      const V r = rot<FWD>(s); // -i*s forward, +i*s backward
      v[k] = cadd(c, r);
      v[p - k] = csub(c, r);
      outs<k + 1>(x0, a, b, v);
    }
  }
  static BF_D void run(V *v) {
    V a[H], b[H];
    V sum = v[0];
#pragma unroll
    for (int m = 1; m <= H; ++m) {
      a[m - 1] = cadd(v[m], v[p - m]);
      b[m - 1] = csub(v[m], v[p - m]);
      sum = cadd(sum, a[m - 1]);
    }
    const V x0 = v[0];
    v[0] = sum;
    outs<1>(x0, a, b, v);
  }
};

// Outer factor N1 of a composite radix (the N1-point butterflies run first): the
// power of 2 (of odd radices the power of 3) in it, whose cofactor then has no
// factor in common with it; of a prime power 4, 3 or 5.
BF_HD constexpr int mixed_outer(int R) {
  for (int p = 2; p <= 3; ++p) {
    int q = 1;
    while (R % (p * q) == 0)
      q *= p;
    if (q > 1 && q < R)
      return q;
  }
  return R % 4 == 0 ? 4 : R % 3 == 0 ? 3 : 5;
}
BF_HD constexpr int ce_gcd(int a, int b) { return b == 0 ? a : ce_gcd(b, a % b); }
BF_HD constexpr int inverse_mod(int a, int m) { // x with x * a = 1 (mod m)
  for (int x = 1; x < m; ++x)
    if (a * x % m == 1)
      return x;
  return 1;
}

// v with the sign of its imaginary part flipped where `flip` is 0x80000000
BF_D float2 conj_if(float2 v, unsigned flip) {
  v.y = __uint_as_float(__float_as_uint(v.y) ^ flip);
  return v;
}
BF_D double2 conj_if(double2 v, unsigned flip) {
  v.y = __hiloint2double(__double2hiint(v.y) ^ static_cast<int>(flip), __double2loint(v.y));
  return v;
}

template <int R, bool FWD, typename V> BF_D void dft_mixed(V *v);

// CompositeDft of fft_device.cuh over the butterflies of this file (prime powers).
template <int N1, int N2, bool FWD, typename V> struct MixedComposite {
  static constexpr int N = N1 * N2;
  template <int n2, int k1> static BF_D void twiddle_into(const V *u, V *t) {
    if constexpr (k1 < N1) {
      t[k1 * N2 + n2] = twk<n2 * k1, N, FWD>(u[k1]);
      twiddle_into<n2, k1 + 1>(u, t);
    }
  }
  template <int n2> static BF_D void inner(const V *v, V *t) {
    if constexpr (n2 < N2) {
      V u[N1];
#pragma unroll
      for (int n1 = 0; n1 < N1; ++n1)
        u[n1] = v[N2 * n1 + n2];
      dft_mixed<N1, FWD>(u);
      twiddle_into<n2, 0>(u, t);
      inner<n2 + 1>(v, t);
    }
  }
  static BF_D void run(V *v) {
    V t[N];
    inner<0>(v, t);
#pragma unroll
    for (int k1 = 0; k1 < N1; ++k1) {
      dft_mixed<N2, FWD>(&t[k1 * N2]);
#pragma unroll
      for (int k2 = 0; k2 < N2; ++k2)
        v[k1 + N1 * k2] = t[k1 * N2 + k2];
    }
  }
};

// N = N1*N2 points, N1 and N2 without a common factor (Good's prime-factor map):
// with n = N2*n1 + N1*n2 and k = N2*(1/N2 mod N1)*k1 + N1*(1/N1 mod N2)*k2 (mod N),
//   w_N^(n k) = w_N1^(n1 k1) w_N2^(n2 k2),
// so no twiddles stand between the N1- and the N2-point butterflies: fewer
// roundings (FP64 points of 2^a 3^b 5^c lengths had up to 12% more error than the
// runtime-generic kernel's with inner twiddles at 6, 10, 12, 15, 18, 20, 24 and 30
// points) and no constants to hold.
template <int N1, int N2, bool FWD, typename V> struct CoprimeDft {
  static constexpr int N = N1 * N2;
  static constexpr int U1 = N2 * inverse_mod(N2 % N1, N1), U2 = N1 * inverse_mod(N1 % N2, N2);
  static BF_D void run(V *v) {
    V t[N];
#pragma unroll
    for (int n2 = 0; n2 < N2; ++n2) {
      V u[N1];
#pragma unroll
      for (int n1 = 0; n1 < N1; ++n1)
        u[n1] = v[(N2 * n1 + N1 * n2) % N];
      dft_mixed<N1, FWD>(u);
#pragma unroll
      for (int k1 = 0; k1 < N1; ++k1)
        t[k1 * N2 + n2] = u[k1];
    }
#pragma unroll
    for (int k1 = 0; k1 < N1; ++k1) {
      dft_mixed<N2, FWD>(&t[k1 * N2]);
#pragma unroll
      for (int k2 = 0; k2 < N2; ++k2)
        v[(U1 * k1 + U2 * k2) % N] = t[k1 * N2 + k2];
    }
  }
};

template <int R, bool FWD, typename V> BF_D void dft_mixed(V *v) {
  if constexpr (R <= 5 || R == 8)
    dft<R, FWD>(v);
  else if constexpr (R == 7 || R == 11 || R == 13)
    PrimeDft<R, FWD, V>::run(v);
  else if constexpr (ce_gcd(mixed_outer(R), R / mixed_outer(R)) == 1)
    CoprimeDft<mixed_outer(R), R / mixed_outer(R), FWD, V>::run(v);
  else
    MixedComposite<mixed_outer(R), R / mixed_outer(R), FWD, V>::run(v);
}

// v[r] *= w^r, w^r = tw[r * base] of the flat table (conjugated when CONJ). A
// power formed as a product carries more roundings than a loaded one, so radices
// up to 5, in columns (whose lanes mostly share an address) up to 9, load every
// power. Longer radices load w, w^2 and every w^(4a) and form w^(4a+1) and
// w^(4a+2) from the entry before. w^(4a+3) is w^(4a+4) conj(w) in FP32, one
// product; FP64 has no registers for the entry ahead and takes w^(4a) w^3 (1125-
// and 1701-point rows spill 108 and 316 bytes otherwise, 36 and 252 so: C2R rows
// of 1125 reals 205 -> 219 us). Three or four powers are live at a time (a chain
// over powers of two keeps half of all powers live). Loading all powers of radices
// 8 and 9 too took FP64 rows of 768 to 1008 points 30% longer, all powers of any
// radix FP64 columns 2% longer on average and of 490, 550, 720 and 1280 points
// 13-16%.
template <int R, bool CONJ, bool COL, typename V>
BF_D void apply_twiddles_mixed(V *v, const V *tw, int base) {
  if constexpr (R <= (COL ? 9 : 5)) {
#pragma unroll
    for (int r = 1; r < R; ++r)
      v[r] = cmulw<CONJ>(v[r], ldtw(tw, r * base));
  } else {
    constexpr bool AHEAD = sizeof(V) == 8;
    const V w1 = ldtw(tw, base), w2 = ldtw(tw, 2 * base);
    V wa = ldtw(tw, 4 * base), w3;
    if constexpr (AHEAD)
      w3 = cmulw<true>(wa, w1);
    else
      w3 = cmulw<false>(w1, w2);
    v[1] = cmulw<CONJ>(v[1], w1);
    v[2] = cmulw<CONJ>(v[2], w2);
    v[3] = cmulw<CONJ>(v[3], w3);
#pragma unroll
    for (int a = 4; a < R; a += 4) {
      v[a] = cmulw<CONJ>(v[a], wa);
      if (a + 1 < R)
        v[a + 1] = cmulw<CONJ>(v[a + 1], cmulw<false>(wa, w1));
      if (a + 2 < R)
        v[a + 2] = cmulw<CONJ>(v[a + 2], cmulw<false>(wa, w2));
      const V here = wa;
      if (a + 4 < R)
        wa = ldtw(tw, (a + 4) * base);
      if (a + 3 < R)
        v[a + 3] = cmulw<CONJ>(v[a + 3], AHEAD && a + 4 < R ? cmulw<true>(wa, w1)
                                                            : cmulw<false>(here, w3));
    }
  }
}

// One pass of a mixed length. C2C kernels transform forward; a backward pass
// conjugates its points on the way in and out (conj F conj = F^-1 up to scale):
// `flip` is XORed into the sign of the imaginary parts, one integer
// instruction per load and store, exact, and half the kernels to compile.
template <int L, int ES, bool COL> struct MixedPlanOf {
  static constexpr MixedPlan value = mixed_plan(L, ES, COL);
};
template <typename T, int L, int KIND, bool ODD, bool COL,
          class PlanT = MixedPlanOf<L, int(sizeof(cvec<T>)), COL>>
struct KM {
  using V = cvec<T>;
  static constexpr bool FWD = KIND != KIND_C2R;
  static constexpr MixedPlan PL = PlanT::value;
  static constexpr int NST = PL.nst, P = PL.P, TB = PL.TB, NT = mixed_threads(COL, P, TB);
  static BF_HD constexpr int rad(int s) { return PL.rad[s]; }
  static BF_HD constexpr int ns(int s) { // product of the radices before stage s
    int p = 1;
    for (int i = 0; i < s; ++i)
      p *= PL.rad[i];
    return p;
  }
  static_assert(ns(NST) == L, "radices must multiply to the length");
  static BF_HD constexpr int bfl(int s) { return L / rad(s); }              // butterflies
  static BF_HD constexpr int per(int s) { return (bfl(s) + P - 1) / P; }    // per thread
  static constexpr int emax() {
    int e = 1;
    for (int s = 0; s < NST; ++s)
      if (per(s) * rad(s) > e)
        e = per(s) * rad(s);
    return e;
  }
  static constexpr int EMAX = emax();
  // Rows of TPW transforms per warp, each within its warp: exchanges need warp
  // barriers only. The 32 - TPW*P lanes left over do lanes 0, 1, ... over again
  // (same addresses, same values).
  static constexpr bool WARP_SYNC = mixed_warped(COL, P);
  static constexpr int TPW = WARP_SYNC ? 32 / P : 1;
  // Rows keep one pad element after every R0 points when R0 is even: the
  // first stage's writes then have the odd stride R0 + 1 across lanes (every
  // bank once); odd R0 needs none. The other stages' accesses stay affine in
  // j and r because R0 divides L/R_s and Ns for s >= 1.
  static constexpr int PADE = (!COL && rad(0) % 2 == 0) ? rad(0) : 0;
  static BF_HD constexpr int padded(int n) { return PADE ? n + n / PADE : n; }
  // Lane `l` of warp 0: thread of its transform and transform of the tile.
  static constexpr int lane_g(int l) { return WARP_SYNC ? l % (TPW * P) % P : l % P; }
  static constexpr int lane_tb(int l) { return WARP_SYNC ? l % (TPW * P) / P : l / P; }
  // Shared-memory wavefronts of one access of warp 0 where the lane's thread g
  // of transform tb is at tb * lp + a*g + b (8-byte points: half a warp over
  // 16 bank pairs, 16-byte points: a quarter over 8 bank quads; equal
  // addresses broadcast).
  static constexpr int fronts(int lp, int kind, int s) {
    constexpr int NB = 128 / int(sizeof(V));
    int cost = 0;
    for (int l0 = 0; l0 < 32; l0 += NB) {
      int at_bank[NB] = {}, addr[NB][NB] = {};
      int mx = 0;
      for (int l = l0; l < l0 + NB; ++l) {
        const int g = lane_g(l);
        int n = g; // reads of a stage, pairs k
        if (kind == 1) // writes of stage s
          n = s == 0 ? g * padded(rad(0))
                     : g / ns(s) * padded(ns(s) * rad(s)) + padded(g % ns(s));
        else if (kind == 2) // pairs L - k
          n = padded(L - g);
        else
          n = padded(g);
        const int ad = lane_tb(l) * lp + n, bk = ad % NB;
        bool seen = false;
        for (int q = 0; q < at_bank[bk]; ++q)
          seen = seen || addr[bk][q] == ad;
        if (!seen)
          addr[bk][at_bank[bk]++] = ad;
        mx = at_bank[bk] > mx ? at_bank[bk] : mx;
      }
      cost += mx;
    }
    return cost;
  }
  // Row pitch with the fewest wavefronts over a row's exchanges: neighbouring
  // transforms share a warp when P does not divide 32, and the pitch decides
  // whether their lanes meet in one bank.
  static constexpr int row_pitch() {
    const int base = padded(L - 1) + 1;
    if (COL)
      return base;
    int best = base, bc = 1 << 30;
    for (int lp = base; lp < base + 128 / int(sizeof(V)); ++lp) {
      int c = 0;
      for (int s = 0; s < NST; ++s) {
        if (s > 0 || (KIND == KIND_C2R && !ODD))
          c += fronts(lp, 0, s); // about L reads
        if (s < NST - 1)
          c += fronts(lp, 1, s); // and L writes
      }
      if (REAL && !ODD) // pairs: half the points ascending, half descending, and
        c += fronts(lp, 0, 0) + (fronts(lp, 0, 0) + fronts(lp, 2, 0)) / 2; // R2C's writes
      if (c < bc) {
        bc = c;
        best = lp;
      }
    }
    return best;
  }
  static constexpr bool REAL = KIND != KIND_C2C;
  static constexpr int LP = row_pitch();
  static constexpr bool STAGE_IN = KIND == KIND_C2R && !ODD; // points arrive in shared memory
  static_assert(COL || NST > 1, "rows of one stage are not compiled");
  static_assert(!WARP_SYNC || TB % TPW == 0, "warps of whole transforms");
  static constexpr int TSC = (REAL && !ODD) ? 2 : 1; // table of 2L entries for even real
  static constexpr size_t smem_bytes() {
    return (NST > 1 || STAGE_IN || (KIND == KIND_R2C && !ODD))
               ? static_cast<size_t>(TB) * LP * sizeof(V) : 0;
  }

  struct Ctx {
    int g, tb;
    bool act;
    const void *in; // first point of the transform
    void *out;
    const V *tw;
    long long ist, ost;
    unsigned flip;
    V *sm; // this transform's shared memory (rows) or the tile + tb (columns)
  };
  static BF_D void bar() {
    if constexpr (WARP_SYNC)
      __syncwarp();
    else
      __syncthreads();
  }
  static BF_D V &at(const Ctx &c, int m) { return c.sm[COL ? m * TB : m]; }

  // point n of the transform
  static BF_D V load(const Ctx &c, int n) {
    const V *in = static_cast<const V *>(c.in);
    if constexpr (KIND == KIND_C2C) {
      return conj_if(in[(long long)n * c.ist], c.flip);
    } else if constexpr (KIND == KIND_R2C && !ODD) {
      return in[n];
    } else if constexpr (KIND == KIND_R2C) {
      return cmake(static_cast<const T *>(c.in)[n], T(0));
    } else { // C2R of odd length: Hermitian extension
      if (n <= L / 2) {
        V x = in[n];
        if (n == 0)
          x.y = T(0);
        return x;
      }
      return cconj(in[L - n]);
    }
  }
  static BF_D void store(const Ctx &c, int k, V z) {
    V *out = static_cast<V *>(c.out);
    if constexpr (KIND == KIND_C2C)
      out[(long long)k * c.ost] = conj_if(z, c.flip);
    else if constexpr (KIND == KIND_C2R && !ODD)
      out[k] = z;
    else if constexpr (KIND == KIND_C2R)
      static_cast<T *>(c.out)[k] = z.x;
    else if (k <= L / 2) // R2C of odd length
      out[k] = z;
  }

  template <int s> static BF_D void run(const Ctx &c, V (&v)[EMAX]) {
    constexpr int R = rad(s), Ns = ns(s), B = bfl(s), K = per(s);
    constexpr bool FULL = B % P == 0;
    const V *tw = c.tw;
#pragma unroll
    for (int i = 0; i < K; ++i) {
      const int j = c.g + P * i;
      // (several butterflies per thread: the last one's idle threads compute
      // along, which keeps the code of all of them in one block)
      if (FULL || K > 1 || j < B) {
        if constexpr (s > 0)
          apply_twiddles_mixed<R, !FWD, COL>(&v[i * R], tw, (j % Ns) * (TSC * L / (Ns * R)));
        dft_mixed<R, FWD>(&v[i * R]);
      }
    }
    if constexpr (s == NST - 1) {
      if constexpr (KIND == KIND_R2C && !ODD) {
        if constexpr (s > 0 || STAGE_IN)
          bar();
#pragma unroll
        for (int i = 0; i < K; ++i) {
          const int j = c.g + P * i;
          if (FULL || j < B) {
            const int m = PADE > 0 ? j + j / (PADE > 0 ? PADE : 1) : j;
#pragma unroll
            for (int r = 0; r < R; ++r)
              at(c, m + padded(r * B)) = v[i * R + r];
          }
        }
        bar();
        r2c_out(c);
      } else {
        if (c.act) {
#pragma unroll
          for (int i = 0; i < K; ++i) {
            const int j = c.g + P * i;
            if (FULL || j < B) {
#pragma unroll
              for (int r = 0; r < R; ++r)
                store(c, j + r * B, v[i * R + r]);
            }
          }
        }
      }
    } else {
      if constexpr (s > 0 || STAGE_IN)
        bar();
#pragma unroll
      for (int i = 0; i < K; ++i) {
        const int j = c.g + P * i;
        if (FULL || j < B) {
          // (j/Ns)*Ns*R + j%Ns + r*Ns; every term but j%Ns a multiple of R0
          const int q = j / Ns, k = j - q * Ns;
          int m = s == 0 ? q * padded(R) : q * padded(Ns * R) + k;
          if constexpr (s > 0 && PADE > 0)
            m += k / PADE;
#pragma unroll
          for (int r = 0; r < R; ++r)
            at(c, m + (s == 0 ? r : padded(r * Ns))) = v[i * R + r];
        }
      }
      bar();
      read_stage<s + 1>(c, v);
      run<s + 1>(c, v);
    }
  }
  template <int s> static BF_D void read_stage(const Ctx &c, V (&v)[EMAX]) {
    constexpr int R = rad(s), B = bfl(s), K = per(s);
    constexpr bool FULL = B % P == 0;
#pragma unroll
    for (int i = 0; i < K; ++i) {
      const int j = c.g + P * i;
      if (FULL || j < B) {
        int m = j;
        if constexpr (PADE > 0)
          m += j / PADE;
#pragma unroll
        for (int r = 0; r < R; ++r) // R0 | B unless s == 0 (then the sum is folded below)
          v[i * R + r] = s == 0 ? at(c, padded(j + r * B)) : at(c, m + padded(r * B));
      }
    }
  }

  // R2C of even length 2L: X[k] and X[L-k] from Z[k], Z[L-k] in shared memory.
  static BF_D void r2c_out(const Ctx &c) {
    const V *tw = c.tw;
    V *X = static_cast<V *>(c.out);
    constexpr int H = L / 2; // pairs k = 0..H
    constexpr int KO = (H + 1 + P - 1) / P;
    if (!c.act)
      return;
#pragma unroll
    for (int i = 0; i < KO; ++i) {
      const int k = c.g + P * i;
      if (k <= H) {
        const V za = at(c, padded(k));
        const V zb = cconj(at(c, padded(k == 0 ? 0 : L - k)));
        const V e = cmake(T(0.5) * (za.x + zb.x), T(0.5) * (za.y + zb.y));
        const V d = csub(za, zb);
        const V o = cmulw<false>(cmake(T(0.5) * d.y, T(-0.5) * d.x), ldtw(tw, k));
        X[k] = cadd(e, o);
        if (2 * k != L)
          X[L - k] = cconj(csub(e, o));
      }
    }
  }
  // C2R of even length 2L: Z[k] and Z[L-k] from X[k], X[L-k] into shared memory.
  static BF_D void c2r_in(const Ctx &c) {
    const V *tw = c.tw;
    const V *X = static_cast<const V *>(c.in);
    constexpr int H = L / 2;
    constexpr int KO = (H + 1 + P - 1) / P;
    V xa[KO], xb[KO];
#pragma unroll
    for (int i = 0; i < KO; ++i) {
      const int k = c.g + P * i;
      if (c.act && k <= H) {
        xa[i] = X[k];
        xb[i] = X[L - k];
      }
    }
#pragma unroll
    for (int i = 0; i < KO; ++i) {
      const int k = c.g + P * i;
      if (c.act && k <= H) {
        if (k == 0) { // Im of DC and Nyquist are ignored
          xa[i].y = T(0);
          xb[i].y = T(0);
        }
        const V b = cconj(xb[i]);
        const V e = cadd(xa[i], b);
        const V o = cmulw<true>(csub(xa[i], b), ldtw(tw, k));
        at(c, padded(k)) = cmake(e.x - o.y, e.y + o.x); // e + i o
        if (k != 0 && 2 * k != L) // Z[L-k] = conj(e) + i conj(o) = conj(e - i o)
          at(c, padded(L - k)) = cmake(e.x + o.y, o.x - e.y);
      }
    }
  }

  static BF_D void entry(const PassArgs &a, unsigned flip, V *sm, long long tile) {
    Ctx c;
    const int tid = threadIdx.x;
    if constexpr (WARP_SYNC) {
      const int lane = (tid & 31) % (TPW * P);
      c.g = lane % P;
      c.tb = (tid >> 5) * TPW + lane / P;
    } else {
      c.g = COL ? tid / TB : tid % P;
      c.tb = COL ? tid % TB : tid / P;
    }
    const long long b = tile * TB + c.tb;
    c.act = b < a.total;
    long long io = 0, oo = 0;
    if (c.act) {
      long long sl, w;
      slab_of(a, b, sl, w);
      io = sl * a.islab + w * a.idist;
      oo = sl * a.oslab + w * a.odist;
    }
    // offsets count the kernel's units: reals on the real side of an odd length
    c.in = static_cast<const char *>(a.in) +
           io * static_cast<long long>(KIND == KIND_R2C && ODD ? sizeof(T) : sizeof(V));
    c.out = static_cast<char *>(a.out) +
            oo * static_cast<long long>(KIND == KIND_C2R && ODD ? sizeof(T) : sizeof(V));
    c.tw = static_cast<const V *>(a.tw);
    c.ist = a.istride;
    c.ost = a.ostride;
    c.flip = flip;
    c.sm = sm + (COL ? c.tb : c.tb * LP);
    pass_begin(a);
    V v[EMAX];
    if constexpr (KIND == KIND_C2R && !ODD) {
      c2r_in(c);
      bar();
      read_stage<0>(c, v);
    } else {
      constexpr int R = rad(0), B = bfl(0), K = per(0);
      constexpr bool FULL = B % P == 0;
#pragma unroll
      for (int i = 0; i < K; ++i) {
        const int j = c.g + P * i;
        const bool ok = c.act && (FULL || j < B);
#pragma unroll
        for (int r = 0; r < R; ++r)
          v[i * R + r] = ok ? load(c, j + r * B) : czero<V>();
      }
    }
    run<0>(c, v);
  }
};

template <class K>
__global__ void __launch_bounds__(K::NT, K::PL.minb)
    fft_mixed_kernel(const PassArgs a, const unsigned flip) {
  extern __shared__ __align__(16) unsigned char smraw[];
  K::entry(a, flip, reinterpret_cast<typename K::V *>(smraw), blockIdx.x);
}

// The passes of one length of many grids: CTA t runs tile map[t].y of
// items[map[t].x]. A kernel of its own: one that takes either form keeps the
// pass arguments in registers and ran 2-4% slower on single passes.
template <class K>
__global__ void __launch_bounds__(K::NT, K::PL.minb)
    fft_mixed_group_kernel(const PassArgs *__restrict__ items, const int2 *__restrict__ map,
                           const unsigned flip) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const int2 t = map[blockIdx.x];
  const PassArgs a = items[t.x];
  K::entry(a, flip, reinterpret_cast<typename K::V *>(smraw), t.y);
}

} // namespace b200fft
