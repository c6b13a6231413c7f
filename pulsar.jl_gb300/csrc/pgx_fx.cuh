// Block fixed-point complex matrices on the tensor cores: the products of the
// FP64 path at D = 8 and 16.
//
// GB300 issues 1.8 FP64 FMAs per clock and SM (measured), so a 16 x 16 complex
// FP64 product takes 9,100 SM cycles.  Here a matrix is 64-bit integers with
// one exponent, value = x 2^(E - 56), |x| < 0.75 2^56, and a product is a sum
// of exact integer products (the Ozaki scheme): each factor is cut into up to
// seven balanced 8-bit digits held as FP16, every pair of digit matrices is
// one real-arithmetic complex product of mma.sync.m16n8k16, and the pairs
// (i, j) of one level i + j accumulate exactly in FP32.  All seven levels of a
// 16 x 16 product are 224 MMAs = 448 SM cycles (measured: one m16n8k16 takes 2
// SM cycles).  mma.sync and not tcgen05: a 16 x 16 unit would fill an M = 128
// tile only together with seven others whose cross products are thrown away,
// and its accumulators would have to come back through TMEM between every two
// products; a warp keeps a whole unit in registers.
//
// Exactness.  |digit| <= 128, the leading one <= 192; at K = 32 real terms a
// level's sum stays within 2^22, so an accumulator started at 1.5 2^23 holds
// 2^23 + integer with unit spacing: its bits minus those of 1.5 2^23 are the
// integer.  Two levels then join in one 32-bit integer, the pairs in one
// 64-bit integer.  Only the levels left out round: level n's largest
// neglected sum is about 2^(0.5 - 8 n) of the factors' scale (rms).
//
// Every product keeps the levels that hold its absolute error near 2^-57 of
// the result it enters, so small terms (the inner Horner steps) take few.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace pgx {
namespace fx {

constexpr int kFrac = 56;      // fractional bits of a normalised matrix
constexpr int kSlices = 7;     // 8-bit digits of a factor
constexpr int kMaxLevels = 8;  // levels 0..7 of digit pairs

// One warp owns one D x D matrix.  Lane (g, t) = (lane / 4, lane % 4) holds,
// of each real plane, the 8 x 8 blocks q: row g + 8 (q & 1), columns
// 2 t + {0, 1} + 8 (q >> 1) -- the accumulator and left-factor fragments of
// m16n8k16.  Value index v = part * NV / 2 + 2 q + h.
template <int D> struct Geo {
  static constexpr int NQ = D >= 16 ? 4 : 1;         // 8 x 8 blocks per plane
  static constexpr int NV = 4 * NQ;                  // real values of a lane
  static constexpr int PLANE = NQ * 128;             // bytes of one digit plane
  static constexpr int PLANES = kSlices * 2 * PLANE; // digit planes of a matrix
  static constexpr int INTS = NV * 32 * 8;           // 64-bit values of a matrix
  __device__ __forceinline__ static int row(int lane, int q) { return (lane >> 2) + 8 * (q & 1); }
  __device__ __forceinline__ static int col(int lane, int q, int h) { return 2 * (lane & 3) + h + 8 * (q >> 1); }
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ldsm2(uint32_t& r0, uint32_t& r1, uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];" : "=r"(r0), "=r"(r1) : "r"(a) : "memory");
}
__device__ __forceinline__ void ldsm2t(uint32_t& r0, uint32_t& r1, uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];"
               : "=r"(r0), "=r"(r1) : "r"(a) : "memory");
}
__device__ __forceinline__ void mma(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                    uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// One digit (re, im) of a factor: the left or the right operand's fragments.
template <int D> struct Frag {
  uint32_t re[Geo<D>::NQ], im[Geo<D>::NQ];
  __device__ __forceinline__ void left(uint32_t base, int s, int lane) {
    if constexpr (D >= 16) {
      ldsm4(re, base + (2 * s) * Geo<D>::PLANE + lane * 16);
      ldsm4(im, base + (2 * s + 1) * Geo<D>::PLANE + lane * 16);
    } else {
      ldsm2(re[0], im[0], base + 2 * s * Geo<D>::PLANE + (lane & 15) * 16);
    }
  }
  __device__ __forceinline__ void right(uint32_t base, int s, int lane) {
    if constexpr (D >= 16) {
      ldsm4t(re, base + (2 * s) * Geo<D>::PLANE + lane * 16);
      ldsm4t(im, base + (2 * s + 1) * Geo<D>::PLANE + lane * 16);
    } else {
      ldsm2t(re[0], im[0], base + 2 * s * Geo<D>::PLANE + (lane & 15) * 16);
    }
  }
};

// acc += a b (complex), one digit pair.
template <int D> __device__ __forceinline__ void mma_pair(float (&acc)[Geo<D>::NV], const Frag<D>& a, const Frag<D>& b) {
  if constexpr (D >= 16) {
    uint32_t n[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) n[i] = a.im[i] ^ 0x80008000u;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      mma(acc + 4 * j, a.re[0], a.re[1], a.re[2], a.re[3], b.re[2 * j], b.re[2 * j + 1]);
      mma(acc + 8 + 4 * j, a.re[0], a.re[1], a.re[2], a.re[3], b.im[2 * j], b.im[2 * j + 1]);
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      mma(acc + 4 * j, n[0], n[1], n[2], n[3], b.im[2 * j], b.im[2 * j + 1]);
      mma(acc + 8 + 4 * j, a.im[0], a.im[1], a.im[2], a.im[3], b.re[2 * j], b.re[2 * j + 1]);
    }
  } else {  // [Re; Im] = [Ar -Ai; Ai Ar] [Br; Bi] in one MMA
    mma(acc, a.re[0], a.im[0], a.im[0] ^ 0x80008000u, a.re[0], b.re[0], b.im[0]);
  }
}

constexpr float kMagic = 12582912.0f;  // 1.5 2^23
constexpr uint32_t kPairBias = (0x4B400000u << 8) + 0x4B400000u;  // two magic starts joined (mod 2^32)

// r += the two levels (2 P, 2 P + 1) held in a0, a1: 56 fractional bits.
template <int D>
__device__ __forceinline__ void join_levels(long long (&r)[Geo<D>::NV], const float (&a0)[Geo<D>::NV],
                                            const float (&a1)[Geo<D>::NV], int P) {
  const uint32_t bias = P == 3 ? 0x8000u - kPairBias : 0u - kPairBias;  // P = 3 rounds its 16 lost bits
#pragma unroll
  for (int v = 0; v < Geo<D>::NV; ++v) {
    const uint32_t t = (__float_as_uint(a0[v]) << 8) + __float_as_uint(a1[v]) + bias;
    r[v] += (long long)((unsigned long long)t << 32) >> (16 * P);
  }
}

// r = A B with `nlev` levels, as value 2^(EA + EB - 56): pa, pb address the
// factors' digit planes.  The two levels of a pass share every left digit;
// the right digit of level 2 P + 1 is the one level 2 P used before.
template <int D>
__device__ __forceinline__ void mul(int lane, uint32_t pa, uint32_t pb, int nlev, long long (&r)[Geo<D>::NV]) {
  constexpr int NV = Geo<D>::NV;
#pragma unroll
  for (int v = 0; v < NV; ++v) r[v] = 0;
#pragma unroll 1
  for (int P = 0; 2 * P < nlev; ++P) {
    const int L = 2 * P;
    const bool two = L + 1 < nlev;
    float a0[NV], a1[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) a0[v] = a1[v] = kMagic;
    const int last = two ? min(L + 1, kSlices - 1) : L;
    Frag<D> bc, bn;
    if (two && L + 1 < kSlices) bc.right(pb, L + 1, lane);
#pragma unroll 1
    for (int i = 0; i <= last; ++i) {
      Frag<D> a;
      a.left(pa, i, lane);
      if (i <= L) bn.right(pb, L - i, lane);
      if (two && L + 1 - i < kSlices) mma_pair<D>(a1, a, bc);
      if (i <= L) mma_pair<D>(a0, a, bn);
      bc = bn;
    }
    join_levels<D>(r, a0, a1, P);
  }
}

// Shift that brings max |r| just below 0.75 2^56 (positive = left); M = the
// largest |high word|, so max |r| < (M + 1) 2^32.
__device__ __forceinline__ int norm_shift(uint32_t M) {
  const uint32_t m = M + 1;
  const int lz = __clz(m);
  return lz - 8 - ((m << lz) >= 0xBF000000u ? 1 : 0);
}
__device__ __forceinline__ long long shift_round(long long v, int right) {  // v >> right, to nearest; right in [1, 63]
  return (v + (1ll << (right - 1))) >> right;
}

// r 2^(e - 56) -> x 2^(E - 56) with 0.37 2^56 < max |x| < 0.75 2^56; returns E.
template <int NV> __device__ __forceinline__ int normalize(long long (&r)[NV], int e) {
  uint32_t M = 0;
#pragma unroll
  for (int v = 0; v < NV; ++v) M = max(M, (uint32_t)abs((int)(r[v] >> 32)));
  M = __reduce_max_sync(0xffffffffu, M);
  const int sh = norm_shift(M);
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
template <int D>
__device__ __forceinline__ void store_planes(int lane, uint32_t base, const long long (&x)[Geo<D>::NV], int ns) {
  constexpr int NQ = Geo<D>::NQ;
  // balanced digits: 128 in every byte below the top; the top digit (|.| <=
  // 192) is read as the 16 bits above bit 48, offset by 512 to stay positive
  constexpr unsigned long long kBias = 0x0080808080808080ull + (512ull << 48);
#pragma unroll
  for (int p = 0; p < 2; ++p)
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const unsigned long long a = (unsigned long long)x[p * 2 * NQ + 2 * q] + kBias;
      const unsigned long long b = (unsigned long long)x[p * 2 * NQ + 2 * q + 1] + kBias;
      const uint32_t al = (uint32_t)a, ah = (uint32_t)(a >> 32), bl = (uint32_t)b, bh = (uint32_t)(b >> 32);
      const uint32_t at = base + p * Geo<D>::PLANE + q * 128 + lane * 4;
#pragma unroll
      for (int s = 0; s < kSlices; ++s) {
        uint32_t t, off;
        if (s == 0) {
          t = __byte_perm(ah, bh, 0x7632) | 0x64006400u;
          off = 0x66806680u;  // 1024 + 512 + 128
        } else {
          const int byte = 6 - s;  // of the 64-bit value
          const uint32_t wa = byte >= 4 ? ah : al, wb = byte >= 4 ? bh : bl;
          const int k = byte & 3;
          t = (__byte_perm(wa, wb, (unsigned)(k | (4 + k) << 8)) & 0x00ff00ffu) | 0x64006400u;
          off = 0x64806480u;  // 1024 + 128
        }
        uint32_t d;
        asm("sub.f16x2 %0, %1, %2;" : "=r"(d) : "r"(t), "r"(off));
        if (s < ns) asm volatile("st.shared.b32 [%0], %1;" ::"r"(at + s * 2 * Geo<D>::PLANE), "r"(d) : "memory");
      }
    }
}

// 64-bit values of a matrix, lane-private in shared memory (16-byte accesses).
template <int NV> __device__ __forceinline__ void put_ints(longlong2* s, int lane, const long long (&x)[NV]) {
#pragma unroll
  for (int v = 0; v < NV; v += 2) s[(v / 2) * 32 + lane] = make_longlong2(x[v], x[v + 1]);
}
template <int NV> __device__ __forceinline__ void get_ints(const longlong2* s, int lane, long long (&x)[NV]) {
#pragma unroll
  for (int v = 0; v < NV; v += 2) {
    const longlong2 a = s[(v / 2) * 32 + lane];
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

// Largest biased exponent of the warp's doubles (0x7ff = not finite).
template <int N> __device__ __forceinline__ int max_exponent(const double (&x)[N]) {
  uint32_t M = 0;
#pragma unroll
  for (int v = 0; v < N; ++v) M = max(M, (uint32_t)__double2hiint(x[v]) & 0x7ff00000u);
  return (int)(__reduce_max_sync(0xffffffffu, M) >> 20);
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
  const unsigned long long m = ((u << (lz - 1)) + 0x200) >> 10;  // bit 52 set (or 53 after a carry)
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

// A coefficient aligned to a frame: c x (x 2^(E - 56)) with 60 fractional bits
// in frame fr is x m 2^-57; the 64-bit product's low quarter is left out (its
// part of the result is below 2^-64 of the frame).
struct Scaled {
  int m1, m0;  // m = m1 2^32 + m0, m0 balanced
  __device__ __forceinline__ Scaled(Coef c, int E, int fr) {
    const unsigned long long m = shr64(c.mant, min(fr - E - c.exp, 63));
    m0 = (int)(uint32_t)m;
    m1 = (int)((m + 0x80000000ull) >> 32);
  }
  __device__ __forceinline__ long long operator()(long long x) const {
    const int b1 = (int)(x >> 32);
    const long long mid = (long long)((unsigned long long)(uint32_t)x * (uint32_t)m1) + (long long)b1 * m0;
    return ((long long)b1 * m1 << 7) + (mid >> 25);
  }
};
// r (60 fractional bits in frame fr) += c x, x 2^(E - 56) normalised.
template <int NV>
__device__ __forceinline__ void add_scaled(long long (&r)[NV], const longlong2* xs, int lane, int E, Coef c, int fr) {
  const Scaled sc(c, E, fr);
#pragma unroll
  for (int v = 0; v < NV; v += 2) {
    const longlong2 a = xs[(v / 2) * 32 + lane];
    r[v] += sc(a.x);
    r[v + 1] += sc(a.y);
  }
}
// r (56 fractional bits at e) -> 60 fractional bits in frame fr >= e + 6.
template <int NV> __device__ __forceinline__ void to_frame(long long (&r)[NV], int e, int fr) {
  const int sh = min(fr - e - 4, 63);
#pragma unroll
  for (int v = 0; v < NV; ++v) r[v] = shift_round(r[v], sh);
}
// r += c I in frame fr.
template <int D> __device__ __forceinline__ void add_diag(long long (&r)[Geo<D>::NV], int lane, Coef c, int fr) {
  const long long d = (long long)shr64(c.mant >> 1, min(fr - c.exp, 63));
#pragma unroll
  for (int q = 0; q < Geo<D>::NQ; ++q)
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (Geo<D>::row(lane, q) == Geo<D>::col(lane, q, h)) r[2 * q + h] += d;
}

}  // namespace fx
}  // namespace pgx
