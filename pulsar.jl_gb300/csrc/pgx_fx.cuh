// Block fixed-point complex matrices on the tensor cores: the products of the
// FP64 path at D = 8, 16 and 32, and of the mixed path's propagators and
// prefixes at D = 16 and 32.
//
// GB300 issues 1.8 FP64 FMAs per clock and SM (measured), so a 16 x 16 complex
// FP64 product takes 9,100 SM cycles.  Here a matrix is 64-bit integers with
// one exponent, value = x 2^(E - 56), |x| < 0.75 2^56 (the FP64 gate chains: all
// 64 bits, "full" below), and a product is a sum of exact integer products (the
// Ozaki scheme): each factor is cut into up to seven (full: eight) balanced 8-bit
// digits held as FP16, every pair of digit matrices is
// one real-arithmetic complex product of mma.sync.m16n8k16, and the pairs
// (i, j) of one level i + j accumulate exactly in FP32.  All seven levels of a
// 16 x 16 product are 224 MMAs = 448 SM cycles (measured: one m16n8k16 takes 2
// SM cycles).  mma.sync and not tcgen05: a 16 x 16 unit would fill an M = 128
// tile only together with seven others whose cross products are thrown away,
// and its accumulators would have to come back through TMEM between every two
// products; a warp keeps a whole unit in registers.
//
// Exactness.  |digit| <= 128, the leading one <= 192; at K = 32 real terms a
// level's sum (eight pairs at most) stays within 2^22, so an accumulator started at 1.5 2^23 holds
// 2^23 + integer with unit spacing: its bits minus those of 1.5 2^23 are the
// integer.  Two levels then join in one 32-bit integer, the pairs in one
// 64-bit integer.  Only the levels left out round: level n's largest
// neglected sum is about 2^(0.5 - 8 n) of the factors' scale (rms).
//
// Every product of an exponential or a series keeps the levels that hold its
// absolute error near 2^-57 (state targets 2^-59, df 2^-51) of the result it
// enters, so small terms (the inner Horner steps) take few.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace pgx {
namespace fx {

constexpr int kFrac = 56;      // fractional bits of a normalised matrix
constexpr int kSlices = 7;     // 8-bit digits of a factor
constexpr int kFullSlices = 8; // digits of a full matrix (below)
constexpr int kMaxLevels = 8;  // levels 0..7 of digit pairs

// A team of W warps owns one D x D matrix; a warp owns RT-th rows x NTW 8-column
// tiles.  Lane (g, t) = (lane / 4, lane % 4) holds, of each real plane, the
// accumulator fragments of m16n8k16: rows 16 rt + g + 8 i, columns 8 (nt of the
// warp) + 2 t + {0, 1}.  Value index v = part NV / 2 + 4 nt + 2 i + h.  D = 8
// (W = 1) is one MMA with the real and imaginary part stacked in its 16 rows.
//
// A digit plane is 8 x 8 blocks of FP16, block (rb, cb) at (cb D / 8 + rb) 128
// bytes, rows of 16 bytes: every ldmatrix reads, and every lane-private store
// writes, whole conflict-free 128-byte lines.
template <int D, int W> struct Geo {
  static constexpr int RT = D >= 16 ? D / 16 : 1;      // 16-row tiles
  static constexpr int CG = W / RT;                    // column groups
  static constexpr int NTW = D / 8 / CG;               // 8-column tiles of a warp
  static constexpr int NI = D >= 16 ? 2 : 1;           // 8-row blocks of a warp's tile
  static constexpr int NV = 4 * NTW * NI;              // real values of a lane
  static constexpr int KT = RT;                        // 16-deep steps of a product
  static constexpr int PLANE = D * D * 2;              // bytes of one digit plane
  static constexpr int PLANES = kSlices * 2 * PLANE;   // digit planes of a matrix
  static constexpr int PLANES_FULL = kFullSlices * 2 * PLANE;
  static constexpr int INTS = 2 * D * D * 8;           // 64-bit values of a matrix
  static_assert(NV * 32 * W == 2 * D * D, "a team covers the matrix");
};

template <int D, int W> struct Tm {
  using G = Geo<D, W>;
  int lane, w, bar;     // bar: the team's hardware barrier (W > 1)
  uint32_t* red;        // 3 W words of shared memory (W > 1)
  __device__ __forceinline__ int rt() const { return W == 1 ? 0 : w % G::RT; }
  __device__ __forceinline__ int nt0() const { return W == 1 ? 0 : w / G::RT * G::NTW; }
  // coordinates of the lane's values (nt, i, h)
  __device__ __forceinline__ int row(int i) const { return 16 * rt() + (lane >> 2) + 8 * i; }
  __device__ __forceinline__ int col(int nt, int h) const { return 8 * (nt0() + nt) + 2 * (lane & 3) + h; }
  __device__ __forceinline__ void sync() const {
    if constexpr (W == 1) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(32 * W) : "memory");
  }
  // largest x of the team's lanes; between two calls with one slot the team
  // has to sync
  __device__ __forceinline__ uint32_t max(uint32_t x, int slot) const {
    x = __reduce_max_sync(0xffffffffu, x);
    if constexpr (W > 1) {
      volatile uint32_t* r = red + slot * W;
      if (lane == 0) r[w] = x;
      sync();
#pragma unroll
      for (int i = 0; i < W; ++i) x = ::max(x, r[i]);
    }
    return x;
  }
  __device__ __forceinline__ longlong2* mine(longlong2* s) const { return s + (size_t)w * (G::NV / 2) * 32 + lane; }
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void ldsm4(uint32_t* r, uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t* r, uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ldsm2(uint32_t* r, uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ldsm2t(uint32_t* r, uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];"
               : "=r"(r[0]), "=r"(r[1]) : "r"(a) : "memory");
}
__device__ __forceinline__ void mma(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                    uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// One digit of the left factor: the warp's rows, columns 16 kt ..
template <int D, int W> struct Left {
  using G = Geo<D, W>;
  static constexpr uint32_t KSTEP = 2 * (D / 8) * 128;  // bytes of a 16-deep step
  uint32_t f[D >= 16 ? 8 : 2];  // re, im
  // the lane's row address of digit 0, step 0
  __device__ __forceinline__ static uint32_t at(const Tm<D, W>& tm, uint32_t planes) {
    const int l = tm.lane;
    if constexpr (D >= 16)
      return planes + ((l >> 4) * (D / 8) + 2 * tm.rt() + ((l >> 3) & 1)) * 128 + (l & 7) * 16;
    else
      return planes + ((l >> 3) & 1) * G::PLANE + (l & 7) * 16;
  }
  __device__ __forceinline__ void load(uint32_t a) {
    if constexpr (D >= 16) {
      ldsm4(f, a);
      ldsm4(f + 4, a + G::PLANE);
    } else {
      ldsm2(f, a);
    }
  }
};
// The same of the conjugate transpose of the matrix in the planes (D >= 16).
template <int D, int W> struct LeftH {
  using G = Geo<D, W>;
  static constexpr uint32_t KSTEP = 2 * 128;
  uint32_t f[8];
  __device__ __forceinline__ static uint32_t at(const Tm<D, W>& tm, uint32_t planes) {
    const int l = tm.lane;
    return planes + ((2 * tm.rt() + ((l >> 3) & 1)) * (D / 8) + (l >> 4)) * 128 + (l & 7) * 16;
  }
  __device__ __forceinline__ void load(uint32_t a) {
    ldsm4t(f, a);
    ldsm4t(f + 4, a + G::PLANE);
#pragma unroll
    for (int i = 4; i < 8; ++i) f[i] ^= 0x80008000u;
  }
};
// One digit of the right factor: rows 16 kt .., the warp's columns.
template <int D, int W> struct Right {
  using G = Geo<D, W>;
  uint32_t f[D >= 16 ? 4 * G::NTW : 2];    // per 8-column tile: re (2), im (2)
  uint32_t neg[D >= 16 ? 2 * G::NTW : 1];  // -im
  __device__ __forceinline__ static uint32_t at(const Tm<D, W>& tm, uint32_t planes) {
    const int l = tm.lane;
    if constexpr (D >= 16)
      return planes + (l >> 4) * G::PLANE + (tm.nt0() * (D / 8) + ((l >> 3) & 1)) * 128 + (l & 7) * 16;
    else
      return planes + ((l >> 3) & 1) * G::PLANE + (l & 7) * 16;
  }
  __device__ __forceinline__ void load(uint32_t a) {
    if constexpr (D >= 16) {
#pragma unroll
      for (int j = 0; j < G::NTW; ++j) {
        ldsm4t(f + 4 * j, a + j * (D / 8) * 128);
        neg[2 * j] = f[4 * j + 2] ^ 0x80008000u;
        neg[2 * j + 1] = f[4 * j + 3] ^ 0x80008000u;
      }
    } else {
      ldsm2t(f, a);
    }
  }
};

constexpr float kMagic = 12582912.0f;  // 1.5 2^23

// acc += a b (complex), one digit pair, one 16-deep step.
template <int D, int W, class LeftT>
__device__ __forceinline__ void mma_pair(float (&acc)[Geo<D, W>::NV], const LeftT& a, const Right<D, W>& b) {
  if constexpr (D >= 16) {
    constexpr int NTW = Geo<D, W>::NTW;
    const uint32_t* x = a.f;
    const uint32_t* y = a.f + 4;
#pragma unroll
    for (int j = 0; j < NTW; ++j) {
      mma(acc + 4 * j, x[0], x[1], x[2], x[3], b.f[4 * j], b.f[4 * j + 1]);
      mma(acc + 4 * (NTW + j), x[0], x[1], x[2], x[3], b.f[4 * j + 2], b.f[4 * j + 3]);
    }
#pragma unroll
    for (int j = 0; j < NTW; ++j) {
      mma(acc + 4 * j, y[0], y[1], y[2], y[3], b.neg[2 * j], b.neg[2 * j + 1]);
      mma(acc + 4 * (NTW + j), y[0], y[1], y[2], y[3], b.f[4 * j], b.f[4 * j + 1]);
    }
  } else {  // [Re; Im] = [Ar -Ai; Ai Ar] [Br; Bi] in one MMA
    mma(acc, a.f[0], a.f[1], a.f[1] ^ 0x80008000u, a.f[0], b.f[0], b.f[1]);
  }
}

constexpr uint32_t kPairBias = (0x4B400000u << 8) + 0x4B400000u;  // two magic starts joined (mod 2^32)

// Levels (L, L + 1) of A B, L even, level L + 1 only if TWO: (level L) 2^8 +
// (level L + 1), summed over the 16-deep steps.  The two levels share every
// left digit, and the right digit of level L + 1 is the one level L uses next.
// All digit loops are unrolled: as rolled loops the products of the d = 8 and
// d = 16 chains took 1.5 and 1.25 times as long.
template <int D, int W, int L, bool TWO, class LeftT = Left<D, W>, int S = kSlices>
__device__ __forceinline__ void level_pair(uint32_t la, uint32_t rb, uint32_t (&t)[Geo<D, W>::NV]) {
  using G = Geo<D, W>;
  constexpr int NV = G::NV;
  constexpr uint32_t kDigit = 2 * G::PLANE;
#pragma unroll 1
  for (int kt = 0; kt < G::KT; ++kt) {
    float a0[NV], a1[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) a0[v] = a1[v] = kMagic;
    const uint32_t pl = la + kt * LeftT::KSTEP, pr = rb + kt * 2 * 128;
    Right<D, W> b[2];
    if (TWO && L + 1 < S) b[1].load(pr + (L + 1) * kDigit);
#pragma unroll
    for (int i = 0; i < S; ++i) {
      if (i > L + (TWO ? 1 : 0)) break;
      LeftT a;
      a.load(pl + i * kDigit);
      if (i <= L) b[i & 1].load(pr + (L - i) * kDigit);  // b[(i + 1) & 1] holds B_{L + 1 - i}
      if (TWO && L + 1 - i < S) mma_pair<D, W>(a1, a, b[(i + 1) & 1]);
      if (i <= L) mma_pair<D, W>(a0, a, b[i & 1]);
    }
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const uint32_t x = (__float_as_uint(a0[v]) << 8) + __float_as_uint(a1[v]) - kPairBias;
      t[v] = kt == 0 ? x : t[v] + x;
    }
  }
}

// r <- r 2^-16 + t 2^32: needs no carries, because a level pair only touches
// the high word.
template <int NV> __device__ __forceinline__ void join_pair(long long (&r)[NV], const uint32_t (&t)[NV], int L) {
  if (L == 0) {  // to nearest: a floor's bias adds up over a chain of products
#pragma unroll
    for (int v = 0; v < NV; ++v) r[v] += 0x8000;
  }
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int hi = (int)(r[v] >> 32);
    const uint32_t lo = __funnelshift_r((uint32_t)r[v], (uint32_t)hi, 16);
    r[v] = (long long)((unsigned long long)(t[v] + (uint32_t)(hi >> 16)) << 32 | lo);
  }
}

// r = A B with N levels, as value 2^(EA + EB - 56): pa, pb address the factors'
// digit planes.  The lowest two levels first, which keeps 32 bits below the
// last one.
template <int D, int W, int N, class LeftT, int L = (N - 1) & ~1>
__device__ __forceinline__ void mul_levels(uint32_t la, uint32_t rb, long long (&r)[Geo<D, W>::NV]) {
  uint32_t t[Geo<D, W>::NV];
  level_pair<D, W, L, (L + 1 < N), LeftT>(la, rb, t);
  join_pair<Geo<D, W>::NV>(r, t, L);
  if constexpr (L > 0) mul_levels<D, W, N, LeftT, L - 2>(la, rb, r);
}
template <int D, int W, int N, class LeftT = Left<D, W>>
__device__ __forceinline__ void mul_fixed(const Tm<D, W>& tm, uint32_t pa, uint32_t pb, long long (&r)[Geo<D, W>::NV]) {
#pragma unroll
  for (int v = 0; v < Geo<D, W>::NV; ++v) r[v] = 0;
  mul_levels<D, W, N, LeftT>(LeftT::at(tm, pa), Right<D, W>::at(tm, pb), r);
}

// A full matrix: value x 2^(E - 64), |x| < 127/128 2^63, its eight digits the
// bytes of the 64-bit integer (a digit counts 2^(E - 8 (i + 1)) in either
// format, so full factors and others mix).  The FP64 gate chains use it: their
// factors are near the identity or the target, and the generator's trace reads
// the entries far below the largest, which FP64 keeps to their own 53 bits.
// With 56 bits under one exponent and products rounded at 2^-56 of the factors'
// scales, the gradients of two-qubit Lindblad pulses below 100 slices were 2.4
// times further off than FP64's (geometric mean of 40 draws); see k_fx_grad.
//
// Largest |high word| -> shift that brings |x| just below 127/128 2^63.
__device__ __forceinline__ int full_shift(uint32_t M) {
  const uint32_t m = M + 1;
  const int lz = __clz(m);
  return lz - 1 - ((m << lz) >= 0xFE000000u ? 1 : 0);
}
template <int D, int W, int N, class LeftT, int S, int L = (N - 1) & ~1>
__device__ __forceinline__ void mul_low_levels(uint32_t la, uint32_t rb, long long (&r)[Geo<D, W>::NV]) {
  if constexpr (L > 0) {
    uint32_t t[Geo<D, W>::NV];
    level_pair<D, W, L, (L + 1 < N), LeftT, S>(la, rb, t);
    join_pair<Geo<D, W>::NV>(r, t, L);
    mul_low_levels<D, W, N, LeftT, S, L - 2>(la, rb, r);
  }
}
// (x, E) <- A B, full and normalised, from S digits of each factor, E the sum
// of their exponents.  The levels below the leading pair stay 64 bits wide, t
// 2^48 + r in units of 2^(E - 72), so nothing is rounded before the shift.
template <int D, int W, int S, int N = kMaxLevels>
__device__ __forceinline__ void mul_full(const Tm<D, W>& tm, uint32_t pa, uint32_t pb, long long (&x)[Geo<D, W>::NV], int& E) {
  constexpr int NV = Geo<D, W>::NV;
  const uint32_t la = Left<D, W>::at(tm, pa), rb = Right<D, W>::at(tm, pb);
#pragma unroll
  for (int v = 0; v < NV; ++v) x[v] = 0;
  mul_low_levels<D, W, N, Left<D, W>, S>(la, rb, x);
  uint32_t t[NV];
  level_pair<D, W, 0, (N > 1), Left<D, W>, S>(la, rb, t);
  uint32_t M = 0;
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    t[v] += (uint32_t)((int)(x[v] >> 32) >> 16);
    M = max(M, (uint32_t)abs((int)t[v]));
  }
  const int sh = full_shift(tm.max(M, 0));  // 0 .. 30
#pragma unroll
  for (int v = 0; v < NV; ++v) {  // the 96 bits t, x's low 48, 0 moved up, upper 64 kept
    const uint32_t mid = (uint32_t)(x[v] >> 16), lo = (uint32_t)x[v] << 16;
    x[v] = (long long)((unsigned long long)__funnelshift_l(mid, t[v], sh) << 32 | __funnelshift_l(lo, mid, sh));
  }
  E = max(E + 8 - sh, -(1 << 20));
}

// Level pair (L, L + 1) with L and `two` chosen by the data: rolled digit loops
// (eight unrolled forms behind a switch were as fast at D = 16 and a fifth
// slower at D = 8).
template <int D, int W>
__device__ __forceinline__ void any_level_pair(uint32_t la, uint32_t rb, int L, bool two, uint32_t (&t)[Geo<D, W>::NV]) {
  using G = Geo<D, W>;
  constexpr int NV = G::NV;
  constexpr uint32_t kDigit = 2 * G::PLANE;
#pragma unroll 1
  for (int kt = 0; kt < G::KT; ++kt) {
    float a0[NV], a1[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) a0[v] = a1[v] = kMagic;
    Left<D, W> a;
    Right<D, W> b0, b1;
    uint32_t pl = la + kt * 2 * (D / 8) * 128, pr = rb + kt * 2 * 128 + L * kDigit;  // A_0, B_L
    a.load(pl);
    b0.load(pr);
    mma_pair<D, W>(a0, a, b0);
    if (two) {
      if (L + 1 < kSlices) {
        b1.load(pr + kDigit);
        mma_pair<D, W>(a1, a, b1);
      }
#pragma unroll 1
      for (int i = 0; i < L; i += 2) {
        a.load(pl + kDigit);
        b1.load(pr - kDigit);
        mma_pair<D, W>(a1, a, b0);
        mma_pair<D, W>(a0, a, b1);
        pl += 2 * kDigit;
        pr -= 2 * kDigit;
        a.load(pl);
        b0.load(pr);
        mma_pair<D, W>(a1, a, b1);
        mma_pair<D, W>(a0, a, b0);
      }
      if (L + 1 < kSlices) {
        a.load(pl + kDigit);
        mma_pair<D, W>(a1, a, b0);
      }
    } else {
#pragma unroll 1
      for (int i = 0; i < L; i += 2) {
        a.load(pl + kDigit);
        b1.load(pr - kDigit);
        mma_pair<D, W>(a0, a, b1);
        pl += 2 * kDigit;
        pr -= 2 * kDigit;
        a.load(pl);
        b0.load(pr);
        mma_pair<D, W>(a0, a, b0);
      }
    }
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const uint32_t x = (__float_as_uint(a0[v]) << 8) + __float_as_uint(a1[v]) - kPairBias;
      t[v] = kt == 0 ? x : t[v] + x;
    }
  }
}

// r = A B with `nlev` levels.
template <int D, int W>
__device__ __forceinline__ void mul(const Tm<D, W>& tm, uint32_t pa, uint32_t pb, int nlev,
                                    long long (&r)[Geo<D, W>::NV]) {
  const uint32_t la = Left<D, W>::at(tm, pa), rb = Right<D, W>::at(tm, pb);
#pragma unroll
  for (int v = 0; v < Geo<D, W>::NV; ++v) r[v] = 0;
#pragma unroll 1
  for (int L = (nlev - 1) & ~1; L >= 0; L -= 2) {
    uint32_t t[Geo<D, W>::NV];
    any_level_pair<D, W>(la, rb, L, L + 1 < nlev, t);
    join_pair<Geo<D, W>::NV>(r, t, L);
  }
}

// r = A B - B A.  Up to D = 16 the level pairs (at most 2^29.9 each with both
// factors below 2^55) are subtracted before they join; at D = 32 their
// difference could pass 2^31, so the products join first.
template <int D, int W>
__device__ __forceinline__ void commutator(const Tm<D, W>& tm, uint32_t pa, uint32_t pb, int nlev,
                                           long long (&r)[Geo<D, W>::NV]) {
  constexpr int NV = Geo<D, W>::NV;
  if constexpr (Geo<D, W>::KT > 1) {
    long long s[NV];
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
      mul<D, W>(tm, h ? pa : pb, h ? pb : pa, nlev, r);
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        if (h) r[v] -= s[v];
        else s[v] = r[v];
      }
    }
  } else {
    const uint32_t la = Left<D, W>::at(tm, pa), rb = Right<D, W>::at(tm, pb);
    const uint32_t lb = Left<D, W>::at(tm, pb), ra = Right<D, W>::at(tm, pa);
#pragma unroll
    for (int v = 0; v < NV; ++v) r[v] = 0;
#pragma unroll 1
    for (int L = (nlev - 1) & ~1; L >= 0; L -= 2) {
      uint32_t t[NV], s[NV];
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {
        any_level_pair<D, W>(h ? la : lb, h ? rb : ra, L, L + 1 < nlev, t);
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          if (h) t[v] -= s[v];
          else s[v] = t[v];
        }
      }
      join_pair<NV>(r, t, L);
    }
  }
}

// Shift that brings max |r| just below 0.75 2^56 (positive = left), or below
// 2^55 with HALF; M = the largest |high word|, so max |r| < (M + 1) 2^32.  HALF
// bounds every digit by 128: two level pairs then add up within 32 bits (the
// 16-deep steps of D = 32, commutators).
template <bool HALF> __device__ __forceinline__ int norm_shift(uint32_t M) {
  const uint32_t m = M + 1;
  const int lz = __clz(m);
  return lz - 8 - (HALF || (m << lz) >= 0xBF000000u ? 1 : 0);
}
__device__ __forceinline__ long long shift_round(long long v, int right) {  // v >> right, to nearest; right in [1, 63]
  return (v + (1ll << (right - 1))) >> right;
}

// r 2^(e - 56) -> x 2^(E - 56), normalised; returns E.
template <int D, int W, bool HALF = (Geo<D, W>::KT > 1)> __device__ __forceinline__ int normalize(const Tm<D, W>& tm, long long (&r)[Geo<D, W>::NV], int e,
                                                                        int slot = 0) {
  constexpr int NV = Geo<D, W>::NV;
  uint32_t M = 0;
#pragma unroll
  for (int v = 0; v < NV; ++v) M = max(M, (uint32_t)abs((int)(r[v] >> 32)));
  const int sh = norm_shift<HALF>(tm.max(M, slot));
  if (sh >= 0) {
#pragma unroll
    for (int v = 0; v < NV; ++v) r[v] <<= sh;
  } else {
#pragma unroll
    for (int v = 0; v < NV; ++v) r[v] = shift_round(r[v], -sh);
  }
  return max(e - sh, -(1 << 20));
}

// The leading `ns` digit planes of a normalised matrix into shared memory.
template <int D, int W>
__device__ __forceinline__ void store_planes(const Tm<D, W>& tm, uint32_t base, const long long (&x)[Geo<D, W>::NV],
                                             int ns) {
  using G = Geo<D, W>;
  constexpr int NV = G::NV;
  // balanced digits: 128 in every byte below the top; the top digit (|.| <=
  // 192) is read as the 16 bits above bit 48, offset by 512 to stay positive
  constexpr unsigned long long kBias = 0x0080808080808080ull + (512ull << 48);
  uint32_t lo[NV], hi[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const unsigned long long a = (unsigned long long)x[v] + kBias;
    lo[v] = (uint32_t)a;
    hi[v] = (uint32_t)(a >> 32);
  }
  const uint32_t at = base + (tm.nt0() * (D / 8) + 2 * tm.rt()) * 128 + tm.lane * 4;
#pragma unroll
  for (int s = 0; s < kSlices; ++s) {
    if (s >= ns) break;
    const int byte = 6 - s;  // of the 64-bit value
#pragma unroll
    for (int b = 0; b < NV / 2; ++b) {  // columns 2 t, 2 t + 1 of one 8 x 8 block
      const int part = b / (NV / 4), nt = b % (NV / 4) / G::NI, i = b % G::NI;
      uint32_t t, d;
      if (s == 0) {
        t = __byte_perm(hi[2 * b], hi[2 * b + 1], 0x7632) | 0x64006400u;  // FP16 1024 + byte
      } else {
        const uint32_t wa = byte >= 4 ? hi[2 * b] : lo[2 * b], wb = byte >= 4 ? hi[2 * b + 1] : lo[2 * b + 1];
        t = (__byte_perm(wa, wb, (unsigned)((byte & 3) | (4 + (byte & 3)) << 8)) & 0x00ff00ffu) | 0x64006400u;
      }
      // minus 1024 + 512 + 128, minus 1024 + 128
      asm("sub.f16x2 %0, %1, %2;" : "=r"(d) : "r"(t), "r"(s == 0 ? 0x66806680u : 0x64806480u));
      asm volatile("st.shared.b32 [%0], %1;" ::"r"(at + (2 * s + part) * G::PLANE + (nt * (D / 8) + i) * 128), "r"(d)
                   : "memory");
    }
  }
}

// r 2^(e - 64) -> full, normalised (r != -2^63); returns its exponent.
template <int D, int W>
__device__ __forceinline__ int normalize_full(const Tm<D, W>& tm, long long (&r)[Geo<D, W>::NV], int e, int slot = 0) {
  constexpr int NV = Geo<D, W>::NV;
  uint32_t M = 0;
#pragma unroll
  for (int v = 0; v < NV; ++v) M = max(M, (uint32_t)abs((int)(r[v] >> 32)));
  const int sh = full_shift(tm.max(M, slot));
  if (sh >= 0) {
#pragma unroll
    for (int v = 0; v < NV; ++v) r[v] <<= sh;
  } else {
#pragma unroll
    for (int v = 0; v < NV; ++v) r[v] = shift_round(r[v], -sh);
  }
  return max(e - sh, -(1 << 20));
}
// The leading S digit planes of a full matrix into shared memory.
template <int D, int W, int S>
__device__ __forceinline__ void store_full(const Tm<D, W>& tm, uint32_t base, const long long (&x)[Geo<D, W>::NV]) {
  using G = Geo<D, W>;
  constexpr int NV = G::NV;
  uint32_t lo[NV], hi[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) {  // balanced digits: 128 in every byte
    const unsigned long long a = (unsigned long long)x[v] + 0x8080808080808080ull;
    lo[v] = (uint32_t)a;
    hi[v] = (uint32_t)(a >> 32);
  }
  const uint32_t at = base + (tm.nt0() * (D / 8) + 2 * tm.rt()) * 128 + tm.lane * 4;
#pragma unroll
  for (int s = 0; s < S; ++s) {
    const int byte = 7 - s;
#pragma unroll
    for (int b = 0; b < NV / 2; ++b) {  // columns 2 t, 2 t + 1 of one 8 x 8 block
      const int part = b / (NV / 4), nt = b % (NV / 4) / G::NI, i = b % G::NI;
      const uint32_t wa = byte >= 4 ? hi[2 * b] : lo[2 * b], wb = byte >= 4 ? hi[2 * b + 1] : lo[2 * b + 1];
      const uint32_t t =  // FP16 1024 + byte
          (__byte_perm(wa, wb, (unsigned)((byte & 3) | (4 + (byte & 3)) << 8)) & 0x00ff00ffu) | 0x64006400u;
      uint32_t d;
      asm("sub.f16x2 %0, %1, %2;" : "=r"(d) : "r"(t), "r"(0x64806480u));  // minus 1024 + 128
      asm volatile("st.shared.b32 [%0], %1;" ::"r"(at + (2 * s + part) * G::PLANE + (nt * (D / 8) + i) * 128), "r"(d)
                   : "memory");
    }
  }
}

// 64-bit values of a matrix, lane-private (16-byte accesses; s = tm.mine()).
template <int NV> __device__ __forceinline__ void put_ints(longlong2* s, const long long (&x)[NV]) {
#pragma unroll
  for (int v = 0; v < NV; v += 2) s[(v / 2) * 32] = make_longlong2(x[v], x[v + 1]);
}
template <int NV> __device__ __forceinline__ void get_ints(const longlong2* s, long long (&x)[NV]) {
#pragma unroll
  for (int v = 0; v < NV; v += 2) {
    const longlong2 a = s[(v / 2) * 32];
    x[v] = a.x;
    x[v + 1] = a.y;
  }
}

// The levels that keep a product's neglected part near 2^-(bits2 - 1)/2 when
// its result is weighted by 2^w: e = the factors' exponents + w.
__device__ __forceinline__ int levels(int bits2, int e) {
  return min(kMaxLevels, max(1, (bits2 + 2 * e + 15) >> 4));
}

__device__ __forceinline__ unsigned long long shr64(unsigned long long v, int s) {  // 0 from s = 64 on
  unsigned long long r;
  asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(s));
  return r;
}

// Largest biased exponent of the team's doubles (0x7ff = not finite).
template <int D, int W> __device__ __forceinline__ int max_exponent(const Tm<D, W>& tm, const double (&x)[Geo<D, W>::NV]) {
  uint32_t M = 0;
#pragma unroll
  for (int v = 0; v < Geo<D, W>::NV; ++v) M = max(M, (uint32_t)__double2hiint(x[v]) & 0x7ff00000u);
  return (int)(tm.max(M, 2) >> 20);
}
// Double -> integer d 2^(1075 + guard - EX), EX the matrix's largest biased
// exponent: |result| < 2^(53 + guard).  guard = 2: the format above with
// E = EX - 1021.
__device__ __forceinline__ long long from_double(double d, int EX, int guard) {
  const uint32_t hi = (uint32_t)__double2hiint(d);
  const int ex = (int)((hi >> 20) & 0x7ff);
  unsigned long long m = ((unsigned long long)((hi & 0xfffffu) | 0x100000u) << 32) | (uint32_t)__double2loint(d);
  m = shr64(m << guard, EX - ex);  // denormals are far below the last bit, or the matrix is zero
  if (ex == 0) m = 0;
  const long long s = (long long)(int)hi >> 31;
  return ((long long)m ^ s) - s;
}
// r 2^k -> double, to nearest.
__device__ __forceinline__ double to_double(long long r, int k) {
  const unsigned long long u = (unsigned long long)(r < 0 ? -r : r);
  const int lz = __clzll((long long)u);
  // bit 52 set (or 53 after a carry).  Ties to even: r often has a few low zero
  // bits, and ties away from zero then raised the norm of U by 3e-17 a slice at d = 32
  const unsigned long long v = u << (lz - 1), m = (v + 0x1ff + (v >> 10 & 1)) >> 10;
  const int be = 63 - lz + k + 1022;                             // biased exponent - 1
  unsigned long long b = m + ((unsigned long long)be << 52);
  if (be > 2045) b = 0x7ff0000000000000ull;
  if (be < 0 || r == 0) b = 0;
  return __longlong_as_double((long long)(b | ((unsigned long long)r & 0x8000000000000000ull)));
}

// c = mant 2^(exp - 61) with mant < 2^61: Taylor coefficients 1/k!.
struct Coef {
  unsigned long long mant;
  int exp;
};

// A coefficient aligned to a frame: r += c x, x 2^(E - 62) the matrix kept by
// put_ints and r an integer with F <= 60 fractional bits in frame fr (value
// r 2^(fr - F), fr >= E + c.exp).  The product's high 64 bits without its low
// quarter: one multiply-add into r and the high word of the two mixed terms.
struct Scaled {
  int m1, m0;  // m = m1 2^32 + m0, m0 balanced
  __device__ __forceinline__ Scaled(Coef c, int E, int fr, int F) {
    const unsigned long long m = shr64(c.mant << 1, min(fr - E - c.exp + 60 - F, 63));
    m0 = (int)(uint32_t)m;
    m1 = (int)((m + 0x80000000ull) >> 32);
  }
  __device__ __forceinline__ long long operator()(long long x, long long r) const {
    const int b1 = (int)(x >> 32);
    const long long mid = (long long)((unsigned long long)(uint32_t)x * (uint32_t)m1) + 0x80000000ll + (long long)b1 * m0;
    return r + (long long)b1 * m1 + (long long)(int)(mid >> 32);
  }
};
template <int NV>
__device__ __forceinline__ void add_scaled(long long (&r)[NV], const longlong2* xs, const Scaled& sc) {
#pragma unroll
  for (int v = 0; v < NV; v += 2) {
    const longlong2 a = xs[(v / 2) * 32];
    r[v] = sc(a.x, r[v]);
    r[v + 1] = sc(a.y, r[v + 1]);
  }
}
// r (56 fractional bits at e) -> F fractional bits in frame fr.
template <int NV> __device__ __forceinline__ void to_frame(long long (&r)[NV], int e, int fr, int F) {
  const int sh = fr - e + kFrac - F;
  if (sh > 0) {
#pragma unroll
    for (int v = 0; v < NV; ++v) r[v] = shift_round(r[v], min(sh, 63));
  } else {
#pragma unroll
    for (int v = 0; v < NV; ++v) r[v] <<= -sh;
  }
}
// r += c I with F fractional bits in frame fr.
template <int D, int W>
__device__ __forceinline__ void add_diag(const Tm<D, W>& tm, long long (&r)[Geo<D, W>::NV], Coef c, int fr, int F) {
  using G = Geo<D, W>;
  const long long d = (long long)shr64(c.mant, min(fr - c.exp + 61 - F, 63));
#pragma unroll
  for (int b = 0; b < G::NV / 2; ++b)
    if (tm.row(b / 2 % G::NI) == tm.col(b / 2 / G::NI, b % 2)) r[b] += d;
}

// A double matrix in the team's order, and back.
template <int D, int W>
__device__ __forceinline__ void load_mat(const Tm<D, W>& tm, const double2* A, double (&x)[Geo<D, W>::NV]) {
  using G = Geo<D, W>;
#pragma unroll
  for (int b = 0; b < G::NV / 2; ++b) {
    const double2 a = A[tm.row(b / 2 % G::NI) + D * tm.col(b / 2 / G::NI, b % 2)];
    x[b] = a.x;
    x[G::NV / 2 + b] = a.y;
  }
}
// r 2^k -> df pair, |r| < 2^60: three exact float pieces (24, 24 and 12 bits)
// joined by a fast two-sum.
__device__ __forceinline__ float2 to_df(long long r, float scale) {
  const float a = (float)(int)(r >> 36), b = (float)((uint32_t)(r >> 12) & 0xffffffu), c = (float)((uint32_t)r & 0xfffu);
  const float x = a * 68719476736.f, y = b * 4096.f;  // 2^36, 2^12
  const float hi = x + y;
  return make_float2(hi * scale, ((y - (hi - x)) + c) * scale);
}
// Float of a matrix whose largest biased exponent is EX -> integer below 2^55,
// value x 2^(E - 56) with E = EX - 125.
__device__ __forceinline__ long long from_float(float f, int EX) {
  const uint32_t u = __float_as_uint(f);
  const int ex = (int)((u >> 23) & 0xff);
  unsigned long long m = (unsigned long long)((u & 0x7fffffu) | 0x800000u) << 31;
  m = ex == 0 ? 0 : shr64(m, EX - ex);
  const long long s = (long long)((int)u >> 31);
  return ((long long)m ^ s) - s;
}

// A full matrix in global memory, lane-private: bit i of its exponent is the
// lowest bit of lane i's first value (2^-64 of the scale; each warp its own copy).
constexpr int kExpBias = 1 << 20;
constexpr int kNotFinite = kExpBias - 1;  // the exponent of a matrix with no finite value
template <int D, int W>
__device__ __forceinline__ void put_packed(const Tm<D, W>& tm, longlong2* s, const long long (&x)[Geo<D, W>::NV], int E) {
  constexpr int NV = Geo<D, W>::NV;
  const int e = max(min(E, kNotFinite), -kExpBias) + kExpBias;
  long long y[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) y[v] = x[v];
  y[0] = (y[0] & ~1ll) | ((e >> tm.lane) & 1);
  put_ints<NV>(s, y);
}
template <int NV> __device__ __forceinline__ int unpack(const long long (&x)[NV]) {  // the whole warp together
  return (int)__ballot_sync(0xffffffffu, (int)x[0] & 1) - kExpBias;
}

// U = r 2^ex
template <int D, int W>
__device__ __forceinline__ void store_mat(const Tm<D, W>& tm, double2* U, const long long (&r)[Geo<D, W>::NV], int ex) {
  using G = Geo<D, W>;
#pragma unroll
  for (int b = 0; b < G::NV / 2; ++b)
    U[tm.row(b / 2 % G::NI) + D * tm.col(b / 2 / G::NI, b % 2)] =
        make_double2(to_double(r[b], ex), to_double(r[G::NV / 2 + b], ex));
}
template <int D, int W> __device__ __forceinline__ void store_nan(const Tm<D, W>& tm, double2* U) {
  using G = Geo<D, W>;
  const double nan = __longlong_as_double(0x7ff8000000000000ll);
#pragma unroll
  for (int b = 0; b < G::NV / 2; ++b)
    U[tm.row(b / 2 % G::NI) + D * tm.col(b / 2 / G::NI, b % 2)] = make_double2(nan, nan);
}

}  // namespace fx
}  // namespace pgx
