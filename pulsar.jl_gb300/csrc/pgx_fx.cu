// FP64-class kernels on block fixed-point tensor-core products (pgx_fx.cuh).
#include "pgx.h"
#include "pgx_fx.cuh"
#include "pgx_stages.cuh"

namespace pgx {
namespace fx {

static __constant__ float c_log2theta[2][PGX_N_FXDEGREES] = {PGX_LOG2_THETA64_EVEN_INIT, PGX_LOG2_THETADF_EVEN_INIT};
static __constant__ Coef c_coef[PGX_N_INVFACT] = PGX_INVFACT_FX_INIT;

constexpr int kMaxTerms = 24;       // generator terms: drift, controls, ramp
constexpr int kMaxTerms32 = 7;      // at D = 32: 16 KB of shared memory each beside two teams
// Absolute error of a slice propagator's products: 2^-57 for the FP64 gate
// chains; 2^-59 for the state chains, whose overlaps can be as small as 1e-4 (at
// 2^-57 the gradients of four-spin transfers below 100 slices were 0.9, at 2^-59
// 0.6 of FP64's error, for 3 % of this kernel); 2^-51 on the mixed path, whose df
// pairs hold 2^-48 of an element (with 2^-48 U_total's defect over 1000 slices
// stayed 2.5 times larger).
template <bool DF> __device__ __forceinline__ int bits2_of(const ProbDev& p) {
  return 2 * (DF ? 51 : p.target == TGT_GATE ? 57 : 59) + 1;
}
constexpr int kNever = 1 << 20;     // an exponent no finite entry reaches
constexpr int kPrefixLevels = 7;  // the mixed path's prefixes, rounded to df pairs or FP32 afterwards

// The constant matrices of the generator, A_mk = c sum_j alpha_j K_j with
// alpha = dt_k {1, scale u_1k, ..., tau_k} and K = {drift_m + off_m O, C_1,
// ..., R_m}, as 64-bit integers K = (b1 2^32 + b0) 2^(E - 60), b0 balanced, in
// the lanes' own order: 3 integer multiply-adds per real value and term in
// place of one FP64 FMA, which is 18 times slower.
template <int D, int W> struct Terms {
  using G = Geo<D, W>;
  int4* k;        // [n][W][NV / 2][32] (b0, b1, b0', b1')
  int* e;         // [n] exponents; kNever: not finite
  int n;
  __host__ __device__ __forceinline__ static size_t bytes(int n) { return (size_t)n * G::INTS + (kMaxTerms + 8) * sizeof(int); }
  __device__ __forceinline__ int4* at(const Tm<D, W>& tm, int j) const {
    return k + ((size_t)j * W + tm.w) * (G::NV / 2) * 32 + tm.lane;
  }
};

// A team converts a matrix (doubles in the lanes' order) into term j.
template <int D, int W>
__device__ __forceinline__ void put_term(const Terms<D, W>& T, int j, const Tm<D, W>& tm, const double (&x)[Geo<D, W>::NV]) {
  constexpr int NV = Geo<D, W>::NV;
  const int EX = max_exponent<D, W>(tm, x);
  int4* dst = T.at(tm, j);
#pragma unroll
  for (int v = 0; v < NV; v += 2) {
    const long long a = from_double(x[v], EX, 6), b = from_double(x[v + 1], EX, 6);
    dst[(v / 2) * 32] = make_int4((int)a, (int)((a + 0x80000000ll) >> 32), (int)b, (int)((b + 0x80000000ll) >> 32));
  }
  if (tm.lane == 0 && tm.w == 0) T.e[j] = EX == 0x7ff ? kNever : EX - 1021;
  tm.sync();
}

// Member m's own terms: drift + offset, and its ramp operator.
template <int D, int W>
__device__ __forceinline__ void put_member_terms(const Terms<D, W>& T, const ProbDev& p, int m, const Tm<D, W>& tm) {
  constexpr int NV = Geo<D, W>::NV;
  double x[NV], o[NV];
  load_mat<D, W>(tm, p.drifts + (size_t)p.m_drift[m] * D * D, x);
  load_mat<D, W>(tm, p.offset_op, o);
  const double off = p.m_offset[m];
#pragma unroll
  for (int v = 0; v < NV; ++v) x[v] = fma(off, o[v], x[v]);
  put_term<D, W>(T, 0, tm, x);
  if (p.n_ramp) {
    const int ro = p.m_ramp[m];
    if (ro >= 0) load_mat<D, W>(tm, p.ramp_ops + (size_t)ro * D * D, x);
#pragma unroll
    for (int v = 0; v < NV; ++v)
      if (ro < 0) x[v] = 0.0;
    put_term<D, W>(T, p.n_c + 1, tm, x);
  }
}

// A = c sum_j alpha_j K_j, 62 fractional bits in the frame returned; a frame
// above kNever / 2 means a term is not finite.  |b1| <= 2^27, |a0| <= 2^31 and
// sum |a1| <= 2^30 keep 24 terms' mixed products inside 63 bits; the products of
// the low halves are left out (at most 2^-60 of the frame a term).  (The frame
// holds the sum of the terms' bounds, up to 2^6 times A's largest entry, so
// 58 bits rounded A more coarsely than doubles do.)
template <int D, int W>
__device__ __forceinline__ int assemble(const Terms<D, W>& T, const ProbDev& p, const double* u, int m, int k,
                                        const Tm<D, W>& tm, long long (&A)[Geo<D, W>::NV]) {
  constexpr int NV = Geo<D, W>::NV;
  const int lane = tm.lane;
  double al = 0.0;
  if (lane < T.n) {
    const double dt = p.dt[k];
    al = lane == 0 ? dt : lane <= p.n_c ? dt * (p.m_scale[m] * u[(size_t)k * p.n_c + lane - 1]) : dt * p.tau[k];
  }
  const uint32_t hi = (uint32_t)__double2hiint(al);
  const int ex = (int)((hi >> 20) & 0x7ff);
  int te = -kNever;
  if (ex == 0x7ff) te = kNever;
  else if (ex > 0) te = ex - 1022 + T.e[lane];  // ex > 0 only below T.n
  const int EA = __reduce_max_sync(0xffffffffu, te) + (32 - __clz(T.n - 1));
  // |alpha_j| 2^(E_j - EA) <= 1 / n in 62 fractional bits
  const int s = te == -kNever ? -64 : te - EA + 9;
  unsigned long long am = ((unsigned long long)((hi & 0xfffffu) | 0x100000u) << 32) | (uint32_t)__double2loint(al);
  am = s >= 0 ? am << min(s, 9) : shr64(am, min(-s, 64));
  const long long sg = (long long)(int)hi >> 31;
  const long long a = ((long long)am ^ sg) - sg;
  const int my0 = (int)a, my1 = (int)((a + 0x80000000ll) >> 32);
  long long main[NV], mid[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    main[v] = 0;
    mid[v] = 1ll << 27;  // to nearest
  }
#pragma unroll 1
  for (int j = 0; j < T.n; ++j) {
    const int a0 = __shfl_sync(0xffffffffu, my0, j), a1 = __shfl_sync(0xffffffffu, my1, j);
    const int4* kp = T.at(tm, j);
#pragma unroll
    for (int v = 0; v < NV; v += 2) {
      const int4 b = kp[(v / 2) * 32];
      main[v] += (long long)b.y * a1;
      mid[v] += (long long)b.y * a0;
      mid[v] += (long long)b.x * a1;
      main[v + 1] += (long long)b.w * a1;
      mid[v + 1] += (long long)b.w * a0;
      mid[v + 1] += (long long)b.z * a1;
    }
  }
  // times c: -i for a Hermitian generator, 1 for a Liouvillian
#pragma unroll
  for (int v = 0; v < NV; ++v) main[v] = (main[v] << 4) + (mid[v] >> 28);
#pragma unroll
  for (int v = 0; v < NV / 2; ++v) {
    A[v] = p.gen == GEN_HERM ? main[NV / 2 + v] : main[v];
    A[NV / 2 + v] = p.gen == GEN_HERM ? -main[v] : main[NV / 2 + v];
  }
  return EA;
}

// log2 of a bound of ||A||_1 (F fractional bits in frame EA): the largest
// column sum, from D = 32 on over each warp's rows and then added up.
template <int D, int W> __device__ __forceinline__ float log2_norm1(const Tm<D, W>& tm, const long long (&A)[Geo<D, W>::NV], int EA,
                                                                                 int F = 62) {
  using G = Geo<D, W>;
  float best = 0.f;
#pragma unroll
  for (int nt = 0; nt < G::NTW; ++nt)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float s = 0.f;
#pragma unroll
      for (int i = 0; i < G::NI; ++i) {
        const int b = 2 * (nt * G::NI + i) + h;
        const float x = (float)(int)(A[b] >> 32), y = (float)(int)(A[G::NV / 2 + b] >> 32);
        s += __fsqrt_rn(fmaf(x, x, y * y));
      }
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      best = fmaxf(best, s);
    }
  if constexpr (G::RT == 1) {
    best = __uint_as_float(tm.max(__float_as_uint(best), 1));
  } else {
    best = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(best)));
    volatile uint32_t* part = tm.red + W;  // slot 1
    if (tm.lane == 0) part[tm.w] = __float_as_uint(best);
    tm.sync();
    best = 0.f;
#pragma unroll
    for (int c = 0; c < G::CG; ++c) {
      float s = 0.f;
#pragma unroll
      for (int i = 0; i < G::RT; ++i) s += __uint_as_float(part[c * G::RT + i]);
      best = fmaxf(best, s);
    }
  }
  return __log2f(fmaf(best, 1.00001f, 2.f * D)) + (float)(EA + 32 - F) + 1e-5f;
}

// Degree 2 L and squarings s that minimise the products L + s (squarings last:
// they double the error), from l1 = log2 of a bound of ||A||_1 and lb = half of
// log2 of a bound of ||A^2||_1 (l1 when A^2 is not known; lb <= l1).  The tail
// of T_m is at most that of a scalar of norm 2^lb (2^(l1 - lb))^(1 / (m + 1)):
// ||A^k|| <= ||A^2||^(k / 2), times ||A|| for odd k.  At d = 32 a random
// generator's 2^lb is 0.4 of its 1-norm, which saves two products.
template <bool DF> __device__ __forceinline__ void choose_degree2(float l1, float lb, int lane, int& L, int& s) {
  uint32_t key = 0xffffffffu;
  if (lane < PGX_N_FXDEGREES) {
    const float x = lb + (l1 - lb) * (1.f / (2 * lane + 5)) - c_log2theta[DF][lane];
    const int si = (int)fmaxf(ceilf(x), 0.f);
    if (si < 64) key = (uint32_t)((2 + lane + si) << 16 | si << 8 | lane);
  }
  key = __reduce_min_sync(0xffffffffu, key);
  s = (int)((key >> 8) & 0xff);
  L = 2 + (int)(key & 0xff);
}

// Warps of a matrix: eight columns each (and, at D = 32, sixteen rows).
template <int D> constexpr int kWarps = D >= 32 ? 8 : D >= 16 ? 2 : 1;
constexpr int kRed = 128;  // bytes of a team's maxima

// U = r 2^ex in df pairs (float4), |r| < 2^60; ex = 0x7ff: not finite.
template <int D, int W>
__device__ __forceinline__ void store_df(const Tm<D, W>& tm, float4* U, const long long (&r)[Geo<D, W>::NV], int ex) {
  using G = Geo<D, W>;
  const float sc = ex == 0x7ff ? __int_as_float(0x7fc00000) : ldexpf(1.f, ex);
#pragma unroll
  for (int b = 0; b < G::NV / 2; ++b) {
    const float2 x = to_df(r[b], sc), y = to_df(r[G::NV / 2 + b], sc);
    U[tm.row(b / 2 % G::NI) + D * tm.col(b / 2 / G::NI, b % 2)] = make_float4(x.x, y.x, x.y, y.y);
  }
}

template <int D> struct ExpmCfg {
  static constexpr int W = kWarps<D>;
  static constexpr int TEAMS = D >= 32 ? 2 : D >= 16 ? 10 : 12;  // slices in flight per CTA, at most
  static constexpr bool REG_B = D >= 32;                         // B stays in registers
  // planes of X, of Y; B; maxima
  static constexpr int TEAM_BYTES = 2 * Geo<D, W>::PLANES + (REG_B ? 0 : Geo<D, W>::INTS) + kRed;
};

// U_mk = exp(A_mk), one team per slice: T_2L(A / 2^s) in the q = 2
// Paterson-Stockmeyer form (X = B^2, Horner in X), then s squarings.  A CTA
// walks runs of `run` slices of one member.
//
// Bound: instruction issue (digits of each factor, joining the levels,
// rescaling), then the tensor pipe (about 64 digit pairs of 16 SM cycles at
// D = 16).  A slice's planes and integers take 18 KB of shared memory, so an SM
// holds ten; two warps share one, each with half the columns.
// DF: the mixed path's propagators, df pairs with 2^-51 products.
// 231,000 slices at d = 16: 42.5 ms as FP64 FMA products, 3.4 here (issue 59 %,
// tensor pipe 33 %); as df products on the FP32 pipe 6.4 ms, 2.8 here (60 and
// 28 %).  32,000 at d = 32 in df: 8.1 and 3.5 ms.
template <int D, bool DF>
__global__ void __launch_bounds__(32 * ExpmCfg<D>::TEAMS * ExpmCfg<D>::W) k_fx_expm(ProbDev p, WorkDev w, int run) {
  using C = ExpmCfg<D>;
  constexpr int W = C::W;
  using G = Geo<D, W>;
  constexpr int NV = G::NV;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int team = threadIdx.x / (32 * W), nt = blockDim.x / (32 * W);
  Terms<D, W> T;
  T.n = p.n_c + 1 + (p.n_ramp ? 1 : 0);
  T.k = reinterpret_cast<int4*>(smem_raw);
  T.e = reinterpret_cast<int*>(smem_raw + (size_t)T.n * G::INTS);
  unsigned char* mine = smem_raw + Terms<D, W>::bytes(T.n) + (size_t)team * C::TEAM_BYTES;
  const uint32_t px = smem_u32(mine), py = px + G::PLANES;
  const Tm<D, W> tm{(int)(threadIdx.x & 31), (int)(threadIdx.x >> 5) % W, 1 + team,
                    reinterpret_cast<uint32_t*>(mine + C::TEAM_BYTES - kRed)};
  longlong2* Bs = tm.mine(reinterpret_cast<longlong2*>(mine + 2 * G::PLANES));
  long long bx[C::REG_B ? NV : 1];
  for (int j = team; j < p.n_c; j += nt) {
    double x[NV];
    load_mat<D, W>(tm, p.ctrls + (size_t)j * D * D, x);
    put_term<D, W>(T, j + 1, tm, x);
  }
  const int runs = (p.n_t + run - 1) / run;
  int cur = -1;
  for (long c = blockIdx.x; c < (long)p.n_members * runs; c += gridDim.x) {
    const int m = (int)(c / runs), k0 = (int)(c % runs) * run;
    if (m != cur) {
      __syncthreads();
      if (team == 0) put_member_terms<D, W>(T, p, m, tm);
      __syncthreads();
      cur = m;
    }
    const int k1 = min(p.n_t, k0 + run);
#pragma unroll 1
    for (int k = k0 + team; k < k1; k += nt) {
      long long r[NV];
      const int EA = assemble<D, W>(T, p, w.u, m, k, tm, r);
      const float l1 = log2_norm1<D, W>(tm, r, EA);
      double2* out = w.U + ((size_t)m * p.n_t + k) * D * D;
      const bool packed = !DF && p.target == TGT_GATE;  // the FP64 gate chains' own format
      const int bits2 = bits2_of<DF>(p);
      // Squares keep an odd number of levels: the first one left out then has no
      // pair of equal digits, whose squares a (skew-)Hermitian matrix sums into
      // its diagonal with one sign.  Six levels of df propagators raised a state's
      // norm by 9e-16 a slice at d = 32 (df products on the FP32 pipe: -5e-16;
      // seven: 2e-17).  Not for unitary gates of the mixed path, whose U_total is
      // projected onto the unitary matrices before its overlap: 4 % of this kernel.
      const int odd = DF && p.target == TGT_GATE && p.gen == GEN_HERM ? 0 : 1;
      int ex;  // U = r 2^ex
      if (EA > kNever / 2 || l1 > 60.f) {
        if constexpr (DF) {
          store_df<D, W>(tm, (float4*)out, r, 0x7ff);
          if (tm.lane == 0 && tm.w == 0) *w.norm_flag = 1;
        } else if (packed) {
          put_packed<D, W>(tm, tm.mine((longlong2*)out), r, kNotFinite);
        } else {
          store_nan<D, W>(tm, out);
        }
        tm.sync();  // the maxima are read
        continue;
      }
      // B = A and X = B B before the degree is known: scaling by 2^-s only moves
      // exponents
      int EB = normalize<D, W>(tm, r, EA - 6), EX = 0, EY = EB, F = 60, L = 2, s = 0, g = 1, lx = 0;
      uint32_t pa = py;
      // step 0: X = B B; L - 1 Horner steps Y <- X Y + c_{2i+1} B + c_2i I,
      // whose error later meets X^i; s squarings.  One product in the loop
      // body keeps the kernel inside the instruction cache.
#pragma unroll 1
      for (int st = 0; st < L + s; ++st) {
        int n;
        if (st == 0) n = min(levels(bits2, 2 * (EB - (int)fmaxf(l1, 0.f))) | odd, kMaxLevels);
        else if (st < L) n = levels(bits2, EX + EY + (L - 1 - st) * lx);
        else n = min(levels(bits2, 2 * EY) | odd, kMaxLevels);
        tm.sync();
        if (st == 0) {
          long long x6[NV];
#pragma unroll
          for (int v = 0; v < NV; ++v) x6[v] = r[v] << 6;
          if constexpr (C::REG_B) {
#pragma unroll
            for (int v = 0; v < NV; ++v) bx[v] = x6[v];
          } else {
            put_ints<NV>(Bs, x6);
          }
        }
        store_planes<D, W>(tm, py, r, n);
        tm.sync();
        mul<D, W>(tm, pa, py, n, r);
        if (st == 0) {
          EX = normalize<D, W>(tm, r, 2 * EB);
          // below 2^-2.6 the 1-norm's own degree is within a product of the best
          const float l2 = l1 > -2.6f ? log2_norm1<D, W>(tm, r, EX, kFrac) : 2.f * l1, lb = fminf(l1, 0.5f * l2);
          choose_degree2<DF>(l1, lb, tm.lane, L, s);
          if (DF && lb > 0.f && tm.lane == 0 && tm.w == 0) *w.norm_flag = 1;  // beyond the gradient's series
          EB -= s;
          EX -= 2 * s;
          // |X| <= 2^lx, and |Y_i| <= c_2i e^nu, nu = 2^(lb - s) -- for a matrix
          // that is not normal, times ||B|| / nu -- so Y_i keeps the fixed
          // frame c_2i.exp + g: e^nu <= 0.75 2^g
          lx = min(0, (int)ceilf(l2 - 2.f * s));
          const float nu = exp2f(lb - (float)s) * 1.4426951f + (p.gen == GEN_HERM ? 0.f : l1 - lb);
          g = max(max(1, EB + 1), (int)ceilf(nu + 0.4151f));
          store_planes<D, W>(tm, px, r, kSlices);
          pa = px;
        }
        if (st < L) {
          const int i = L - 1 - st;
          const bool final = !DF && i == 0 && s == 0;  // |U| <= e^nu <= 0.75 2^g
          const int fr = final ? g : c_coef[2 * i].exp + g;
          F = st > 0 && i == 0 ? 60 : kFrac;
          if (st == 0) {
            // Y = c_2L X + c_{2L-1} B + c_{2L-2} I
            const Scaled sx(c_coef[2 * L], EX, fr, F);
#pragma unroll
            for (int v = 0; v < NV; ++v) r[v] = sx(r[v] << 6, 0);
          } else {
            to_frame<NV>(r, EX + EY, fr, F);
          }
          const Scaled sb(c_coef[2 * i + 1], EB, fr, F);
          if constexpr (C::REG_B) {
#pragma unroll
            for (int v = 0; v < NV; ++v) r[v] = sb(bx[v], r[v]);
          } else {
            add_scaled<NV>(r, Bs, sb);
          }
          add_diag<D, W>(tm, r, c_coef[2 * i], fr, F);
          EY = fr;
          if (i == 0) {
            ex = fr - 60;
            if (s > 0) EY = normalize<D, W>(tm, r, fr - 4);
            pa = py;
          }
        } else {
          ex = 2 * EY - kFrac;
          if (packed || st + 1 < L + s) EY = normalize<D, W>(tm, r, 2 * EY);
        }
      }
      if constexpr (DF) {
        store_df<D, W>(tm, (float4*)out, r, ex);
        continue;
      }
      if (packed) {  // from 60 fractional bits of frame EY, 56 after squarings
#pragma unroll
        for (int v = 0; v < NV; ++v) r[v] <<= s == 0 ? 3 : 7;
        put_packed<D, W>(tm, tm.mine((longlong2*)out), r, EY + 1);
      } else {
        store_mat<D, W>(tm, out, r, ex);
      }
    }
  }
}

// sum_s psi_s[k] lambda_s[kl]' of a state target in the team's order: M_k (kl =
// k + 1) or N_k = M_k U_k (kl = k).
template <int D, int W>
__device__ __forceinline__ void load_M(const Tm<D, W>& tm, const ProbDev& p, const WorkDev& w, int m, int k, int kl,
                                       double (&x)[Geo<D, W>::NV]) {
  using G = Geo<D, W>;
  const int np = p.n_pairs;
  const double2* psi = w.psi + ((size_t)m * (p.n_t + 1) + k) * np * D;
  const double2* lam = w.lam + ((size_t)m * (p.n_t + 1) + kl) * np * D;
#pragma unroll
  for (int v = 0; v < G::NV; ++v) x[v] = 0.0;
  for (int s = 0; s < np; ++s)
#pragma unroll
    for (int b = 0; b < G::NV / 2; ++b) {
      double2 y = psi[s * D + tm.row(b / 2 % G::NI)];
      const double2 l = lam[s * D + tm.col(b / 2 / G::NI, b % 2)];
      if (lam_unscaled(p, D)) y = cmul(w.kap[(size_t)m * np + s], y);
      const double2 acc = cmac(make_double2(x[b], x[G::NV / 2 + b]), y, make_double2(l.x, -l.y));
      x[b] = acc.x;
      x[G::NV / 2 + b] = acc.y;
    }
}

// t = Tr(X K_j), its real (im = 0) or imaginary part, as an integer sum over
// the team: the lanes' X (58 fractional bits) against the transposed term (60).
// A lane's 2 D D / (32 W) products sum below 2^57 in units of 2^-54; its lowest
// PS bits join the next 24 in a second word, so the warp's sum stays inside 63
// bits and no low part is rounded by itself (gradients much smaller than |X|
// |K| would lose bits).
struct Trace {
  long long hi;  // units of 2^(PS - 54)
  uint32_t lo;   // units of 2^(PS - 78)
};
template <int D> constexpr int kTraceShift = D >= 32 ? 4 : 2;
template <int D, int W>
__device__ __forceinline__ Trace trace_term(const Terms<D, W>& T, const Tm<D, W>& tm, int j, int im,
                                            const long long (&x)[Geo<D, W>::NV]) {
  using G = Geo<D, W>;
  constexpr int PS = kTraceShift<D>;
  const int2* kp = reinterpret_cast<const int2*>(T.k + (size_t)j * W * (G::NV / 2) * 32);
  long long main = 0, mid = 0;
#pragma unroll
  for (int b = 0; b < G::NV / 2; ++b) {
    // element (row', col') = (col, row) of the term in the team's layout
    const int r = tm.col(b / 2 / G::NI, b % 2), c = tm.row(b / 2 % G::NI);
    const int nt = c / 8 % G::NTW, wt = c / 8 / G::NTW * G::RT + (D >= 16 ? r / 16 : 0);
    const int v = 2 * (nt * G::NI + r / 8 % G::NI) + c % 2;
    const int2* e = kp + ((size_t)(wt * (G::NV / 2) + v / 2) * 32 + (r % 8) * 4 + c % 8 / 2) * 2 + v % 2;
    const int2 cr = e[0], ci = e[(G::NV / 4) * 64];
    // re: xr cr - xi ci, im: xr ci + xi cr
    const long long xr = x[b], xi = im ? x[G::NV / 2 + b] : -x[G::NV / 2 + b];
    const int xr0 = (int)xr, xr1 = (int)((xr + 0x80000000ll) >> 32);
    const int xi0 = (int)xi, xi1 = (int)((xi + 0x80000000ll) >> 32);
    const int2 p = im ? ci : cr, q = im ? cr : ci;
    main += (long long)xr1 * p.y;
    main += (long long)xi1 * q.y;
    mid += (long long)xr1 * p.x;
    mid += (long long)xr0 * p.y;
    mid += (long long)xi1 * q.x;
    mid += (long long)xi0 * q.y;
  }
  const long long sum = main + (mid >> 32);
  Trace t;
  t.hi = sum >> PS;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t.hi += __shfl_xor_sync(0xffffffffu, t.hi, o);
  t.lo = __reduce_add_sync(0xffffffffu, ((uint32_t)sum & ((1u << PS) - 1)) << (24 - PS) | (uint32_t)mid >> (8 + PS));
  return t;
}

constexpr int kGradBits2 = 2 * 56 + 1;
constexpr unsigned long long kTodo = 0x7ff8dead00000001ull;  // a slice left to k_fx_grad_norm (a NaN no sum produces)

template <int D> constexpr int kTraces = D >= 32 ? kMaxTerms32 + 1 : kMaxTerms;
// Digits of R_k and V_k in the gradient's product: all, but seven at D = 32,
// where two teams of eight beside seven terms pass the shared memory.
template <int D> constexpr int kPrefixDigits = D >= 32 ? kSlices : kFullSlices;
template <int D, int PLANE_BYTES, int MAX_TEAMS> struct GradCfg {
  static constexpr int W = kWarps<D>;
  static constexpr int TEAMS = MAX_TEAMS;
  static constexpr int TRACES = W > 1 ? W * kTraces<D> * 12 : 0;  // the warps' traces, hi and lo
  static constexpr int TEAM_BYTES = PLANE_BYTES + kRed + TRACES;
  static_assert(TEAM_BYTES % 16 == 0, "teams' planes are 16-byte aligned");
};
template <int D> constexpr int kPrefixPlane = kPrefixDigits<D> * 2 * Geo<D, kWarps<D>>::PLANE;  // bytes of one factor
template <int D> using SeriesCfg = GradCfg<D, 2 * kPrefixPlane<D>, (D >= 32 ? 2 : D >= 16 ? 10 : 12)>;
template <int D> using NormCfg = GradCfg<D, 4 * Geo<D, kWarps<D>>::PLANES, (D >= 32 ? 1 : D >= 16 ? 7 : 12)>;

// g_jk = cds {Re, Im} Tr(X C_j), X 2^(E - 58) the team's: integer traces, lane
// j keeps control j's.  `traces` is free again after the team's next sync.
template <int D, int W>
__device__ __forceinline__ void put_traces(const Terms<D, W>& T, const Tm<D, W>& tm, const ProbDev& p, const WorkDev& w,
                                           int m, int k, const long long (&x)[Geo<D, W>::NV], int E, long long* traces) {
  uint32_t* low = reinterpret_cast<uint32_t*>(traces + W * kTraces<D>);
  Trace keep{0, 0};
#pragma unroll 1
  for (int j = 0; j < p.n_c; ++j) {
    const Trace t = trace_term<D, W>(T, tm, j + 1, p.gen == GEN_HERM ? 1 : 0, x);
    if constexpr (W > 1) {
      if (tm.lane == 0) {
        traces[tm.w * kTraces<D> + j] = t.hi;
        low[tm.w * kTraces<D> + j] = t.lo;
      }
    }
    if (tm.lane == j) keep = t;
  }
  if constexpr (W > 1) tm.sync();
  if (tm.w == 0 && tm.lane < p.n_c) {
    if constexpr (W > 1) {
#pragma unroll
      for (int i = 1; i < W; ++i) {
        keep.hi += traces[i * kTraces<D> + tm.lane];
        keep.lo += low[i * kTraces<D> + tm.lane];
      }
    }
    const int e = E + T.e[tm.lane + 1] - 54 + kTraceShift<D>;
    w.Gm[((size_t)m * p.n_t + k) * p.n_c + tm.lane] =
        p.dt[k] * p.m_scale[m] * (to_double(keep.hi, e) + to_double(keep.lo, e - 24));
  }
}
template <int D, int W>
__device__ __forceinline__ void put_grad_value(const Tm<D, W>& tm, const ProbDev& p, const WorkDev& w, int m, int k,
                                               unsigned long long bits) {
  if (tm.w == 0 && tm.lane < p.n_c)
    w.Gm[((size_t)m * p.n_t + k) * p.n_c + tm.lane] = __longlong_as_double((long long)bits);
}

template <int D, int W> __device__ __forceinline__ longlong2* slot(const Tm<D, W>& tm, double2* stack, size_t i) {
  return tm.mine(reinterpret_cast<longlong2*>(stack + i * D * D));
}

// (x, E) <- R_k x, full, with the product before slice k inside its block (the
// identity at its start); x's digits go to pr, R_k's to pl.
template <int D, int W>
__device__ __forceinline__ void times_prefix(const Tm<D, W>& tm, const ProbDev& p, const WorkDev& w, int m, int k, int len,
                                             uint32_t pl, uint32_t pr, long long (&x)[Geo<D, W>::NV], int& E) {
  if (k % len == 0) return;
  constexpr int S = kPrefixDigits<D>;
  long long r[Geo<D, W>::NV];
  get_ints<Geo<D, W>::NV>(slot(tm, w.P, (size_t)m * p.n_t + k), r);
  const int ER = unpack(r);
  tm.sync();  // the last slice's products have read their planes
  store_full<D, W, S>(tm, pr, x);
  store_full<D, W, S>(tm, pl, r);
  tm.sync();
  const bool bad = max(E, ER) == kNotFinite;
  E += ER;
  mul_full<D, W, S>(tm, pl, pr, x, E);
  if (bad) E = kNotFinite;
}

// The gradient of gate targets in any mode, and of exact state targets without
// tracking (whose co-state lambda_k holds more than U_k' lambda_{k+1}).  One
// team per slice: g_jk = Re(c dt scale Tr(X C_j)).
//
// Exact: X = L_exp(A, M) = sum_n ad_A^n(N) / (n + 1)!, N = M e^A = P_k
// Lambda_{k-1} (ad_A X = A X - X A commutes with the factor e^A).  Two products
// and one matrix a term, each term in block fixed point with the levels its
// size asks for, until it is below 2^-56 of N: about ten terms at ||A|| = 0.15.
// The Paterson-Stockmeyer derivative takes as many digit products, but four
// matrices' planes where this takes two, so half as many slices an SM.  Where
// the terms grow (norms above 2 or so), cancellation would cost bits: such
// slices are left to k_fx_grad_norm.
// First order: X = M_k = R_k V_k, or with the costate that includes U_k.
//
// Bound: instruction issue (60 %), then the tensor pipe (36 %).  231,000 slices
// at d = 16: 109.7 ms as a Frechet form of FP64 FMA products, 11.7 as that form
// in block fixed point, 9.3 here.
//
// Accuracy against long double, as a part of the FMA kernels' (whose doubles keep
// every entry to 53 bits of itself), geometric means over 50 to 200 draws each of
// 20 to 2000 slices: four-spin gates 0.11, random gates 0.18 to 0.28 (d = 20
// 0.5), two-qubit Lindblad gates 0.25 (below 100 slices 0.4), four-spin transfers
// 0.45 (0.6), random transfers 0.25 to 0.5.
template <int D>
__global__ void __launch_bounds__(32 * SeriesCfg<D>::TEAMS * SeriesCfg<D>::W)
k_fx_grad(ProbDev p, WorkDev w, int run, int len) {
  using C = SeriesCfg<D>;
  constexpr int W = C::W;
  using G = Geo<D, W>;
  constexpr int NV = G::NV;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int team = threadIdx.x / (32 * W), nt = blockDim.x / (32 * W);
  Terms<D, W> T;
  T.n = p.n_c + 1 + (p.n_ramp ? 1 : 0);
  T.k = reinterpret_cast<int4*>(smem_raw);
  T.e = reinterpret_cast<int*>(smem_raw + (size_t)T.n * G::INTS);
  unsigned char* mine = smem_raw + Terms<D, W>::bytes(T.n) + (size_t)team * C::TEAM_BYTES;
  const uint32_t pa = smem_u32(mine), pd = pa + kPrefixPlane<D>;
  const Tm<D, W> tm{(int)(threadIdx.x & 31), (int)(threadIdx.x >> 5) % W, 1 + team,
                    reinterpret_cast<uint32_t*>(mine + 2 * kPrefixPlane<D>)};
  long long* traces = reinterpret_cast<long long*>(mine + 2 * kPrefixPlane<D> + kRed);
  for (int j = team; j < p.n_c; j += nt) {
    double x[NV];
    load_mat<D, W>(tm, p.ctrls + (size_t)j * D * D, x);
    put_term<D, W>(T, j + 1, tm, x);
  }
  const int runs = (p.n_t + run - 1) / run;
  int cur = -1;
  for (long c = blockIdx.x; c < (long)p.n_members * runs; c += gridDim.x) {
    const int m = (int)(c / runs), k0 = (int)(c % runs) * run;
    if (m != cur) {
      __syncthreads();
      if (team == 0) put_member_terms<D, W>(T, p, m, tm);
      __syncthreads();
      cur = m;
    }
    const int k1 = min(p.n_t, k0 + run);
#pragma unroll 1
    for (int k = k0 + team; k < k1; k += nt) {
      long long x[NV];
      int E;  // N (exact) or M = x 2^(E - 64)
      if (p.target == TGT_GATE) {
        // slot k holds V_k U_k = Lambda_{k-1} up to the block's prefix; V_k is
        // the next slice's, or W_b at the end of the block
        if (p.grad_mode != GRAD_REF_MR) get_ints<NV>(slot(tm, w.U, (size_t)m * p.n_t + k), x);
        else if ((k + 1) % len != 0 && k + 1 < p.n_t) get_ints<NV>(slot(tm, w.U, (size_t)m * p.n_t + k + 1), x);
        else get_ints<NV>(slot(tm, w.P, (size_t)m * p.n_t + k / len * len), x);
        E = unpack(x);
        times_prefix<D, W>(tm, p, w, m, k, len, pa, pd, x, E);
      } else {
        double d[NV];
        load_M<D, W>(tm, p, w, m, k, k, d);
        const int EXd = max_exponent<D, W>(tm, d);
#pragma unroll
        for (int v = 0; v < NV; ++v) x[v] = from_double(d[v], EXd, 10);
        E = EXd == 0x7ff ? kNotFinite : EXd - 1021;
      }
      tm.sync();
      if (p.grad_mode == GRAD_EXACT && E != kNotFinite) {
        long long r[NV];
        const int EA = assemble<D, W>(T, p, w.u, m, k, tm, r);
        const float l2 = log2_norm1<D, W>(tm, r, EA);
        bool todo = l2 > 1.3f;
        if (EA > kNever / 2) E = kNotFinite;
        else if (!todo) {
          const int EB = normalize<D, W, true>(tm, r, EA - 6);
          store_planes<D, W>(tm, pa, r, kSlices);
          const int EN = E;
#pragma unroll
          for (int v = 0; v < NV; ++v) r[v] = shift_round(x[v], 8);  // 56 fractional bits, below 2^55
          // x becomes the sum, 60 fractional bits in frame EN + h: h = 0 where
          // the first term is below half of N (so the entries of N keep 2^-60 of
          // the largest's scale), else 3
          int Er = EN, h = -4;  // (no term: x as it is)
          float size = 1.f;  // of the terms, in units of N: below 7 the sum stays inside its frame
          todo = true;
#pragma unroll 1
          for (int n = 1; n < PGX_N_INVFACT - 1; ++n) {
            const Coef cf = c_coef[n + 1];
            const int lev = (kGradBits2 + 2 * (EB + Er + cf.exp - EN) + 15) >> 4;
            if (lev <= 0) {
              todo = false;
              break;
            }
            tm.sync();
            store_planes<D, W>(tm, pd, r, min(lev, kSlices));
            tm.sync();
            commutator<D, W>(tm, pa, pd, min(lev, kMaxLevels), r);
            Er = normalize<D, W, true>(tm, r, EB + Er);
            const int et = Er + cf.exp - EN;  // the term is below 2^(et - 1) N's scale
            if (n == 1) {
              h = et <= -1 ? 0 : 3;
#pragma unroll
              for (int v = 0; v < NV; ++v) x[v] = shift_round(x[v], h + 4);
            }
            size += exp2f((float)et);
            if (size > 7.f || et > h) break;
            const Scaled sc(cf, Er, EN + h, 60);
#pragma unroll
            for (int v = 0; v < NV; ++v) x[v] = sc(r[v] << 6, x[v]);
          }
          tm.sync();
          E = normalize_full<D, W>(tm, x, EN + h + 4);
        }
        if (todo && E != kNotFinite) {
          put_grad_value<D, W>(tm, p, w, m, k, kTodo);
          tm.sync();
          continue;
        }
      }
      if (E == kNotFinite) {
        put_grad_value<D, W>(tm, p, w, m, k, 0x7ff8000000000000ull);
        tm.sync();
      } else {
#pragma unroll
        for (int v = 0; v < NV; ++v) x[v] = shift_round(x[v], 6);
        put_traces<D, W>(T, tm, p, w, m, k, x, E, traces);
        tm.sync();  // the maxima and the traces are read
      }
    }
  }
}

// The slices k_fx_grad left (kTodo): large norms.  X = L_f(A_k, M_k), the
// Frechet derivative of f = T_2L(A / 2^s)^(2^s) in the q = 2 form (three
// products a step).  The derivative's matrices keep an exponent of their own,
// so any magnitude of M_k does.  Runs with no such slice cost one pass over
// their flags.
template <int D>
__global__ void __launch_bounds__(32 * NormCfg<D>::TEAMS * NormCfg<D>::W)
k_fx_grad_norm(ProbDev p, WorkDev w, int run, int len) {
  using C = NormCfg<D>;
  constexpr int W = C::W;
  using G = Geo<D, W>;
  constexpr int NV = G::NV;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int team = threadIdx.x / (32 * W), nt = blockDim.x / (32 * W);
  Terms<D, W> T;
  T.n = p.n_c + 1 + (p.n_ramp ? 1 : 0);
  T.k = reinterpret_cast<int4*>(smem_raw);
  T.e = reinterpret_cast<int*>(smem_raw + (size_t)T.n * G::INTS);
  unsigned char* mine = smem_raw + Terms<D, W>::bytes(T.n) + (size_t)team * C::TEAM_BYTES;
  const uint32_t px = smem_u32(mine), pdx = px + G::PLANES, py = px + 2 * G::PLANES, pdy = px + 3 * G::PLANES;
  const Tm<D, W> tm{(int)(threadIdx.x & 31), (int)(threadIdx.x >> 5) % W, 1 + team,
                    reinterpret_cast<uint32_t*>(mine + 4 * G::PLANES)};
  long long* traces = reinterpret_cast<long long*>(mine + 4 * G::PLANES + kRed);
  const int runs = (p.n_t + run - 1) / run;
  int cur = -1;
  for (long c = blockIdx.x; c < (long)p.n_members * runs; c += gridDim.x) {
    const int m = (int)(c / runs), k0 = (int)(c % runs) * run, k1 = min(p.n_t, k0 + run);
    bool any = false;
    for (int k = k0 + (int)threadIdx.x; k < k1; k += blockDim.x)
      any |= (unsigned long long)__double_as_longlong(w.Gm[((size_t)m * p.n_t + k) * p.n_c]) == kTodo;
    if (!__syncthreads_or(any)) continue;
    if (cur < 0)
      for (int j = team; j < p.n_c; j += nt) {
        double x[NV];
        load_mat<D, W>(tm, p.ctrls + (size_t)j * D * D, x);
        put_term<D, W>(T, j + 1, tm, x);
      }
    if (m != cur) {
      if (team == 0) put_member_terms<D, W>(T, p, m, tm);
      cur = m;
    }
    __syncthreads();
#pragma unroll 1
    for (int k = k0 + team; k < k1; k += nt) {
      if ((unsigned long long)__double_as_longlong(w.Gm[((size_t)m * p.n_t + k) * p.n_c]) != kTodo) continue;
      long long b[NV], db[NV], r[NV], q[NV];
      int EM;  // M_k = db 2^(EM - 56)
      if (p.target == TGT_GATE) {
        if ((k + 1) % len != 0 && k + 1 < p.n_t) get_ints<NV>(slot(tm, w.U, (size_t)m * p.n_t + k + 1), db);
        else get_ints<NV>(slot(tm, w.P, (size_t)m * p.n_t + k / len * len), db);
        EM = unpack(db);
        // two full factors in the four sets of planes
        times_prefix<D, W>(tm, p, w, m, k, len, px, py, db, EM);
#pragma unroll
        for (int v = 0; v < NV; ++v) db[v] = shift_round(db[v], 8);
      } else {
        double x[NV];
        load_M<D, W>(tm, p, w, m, k, k + 1, x);
        const int EXd = max_exponent<D, W>(tm, x);
#pragma unroll
        for (int v = 0; v < NV; ++v) db[v] = from_double(x[v], EXd, 2);
        EM = EXd - 1021;
      }
      tm.sync();  // every lane has read the flag
      const int EA = assemble<D, W>(T, p, w.u, m, k, tm, b);
      const float l2 = log2_norm1<D, W>(tm, b, EA);
      int L, s;
      choose_degree2<false>(l2, l2, tm.lane, L, s);
      if (s > 60) {
        put_grad_value<D, W>(tm, p, w, m, k, 0x7ff8000000000000ull);
        tm.sync();
        continue;
      }
      const int ED = EM - s;  // dB = M / 2^s
      const float nu2 = l2 - (float)s;
      const int lx = min(0, 2 * (int)ceilf(nu2));
      const int g = nu2 <= -1.33f ? 1 : 3;
      const int EB = normalize<D, W>(tm, b, EA - 6 - s);
      tm.sync();
      store_planes<D, W>(tm, py, b, kSlices);
      store_planes<D, W>(tm, pdy, db, kSlices);
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        b[v] <<= 6;
        db[v] <<= 6;
      }
      int EX = EB, EdX = ED, EY = EB, EdY = ED;  // step 0: (X, dX) <- (B B, dB B + B dB)
      uint32_t pl = py, pdl = pdy;
#pragma unroll 1
      for (int st = 0; st < L + s; ++st) {
        const int i = L - 1 - st;
        const bool last = st + 1 == L + s;
        const int fq = max(EdX + EY, EX + EdY) + 6;
        tm.sync();
#pragma unroll 1
        for (int h = 0; h < (last ? 2 : 3); ++h) {
          const int ea = h == 0 ? EdX : EX, eb = h == 1 ? EdY : EY;
          // relative to dB for the derivative, to I for Y; the error of step i
          // meets X^i later, and Y only acts through dX Y
          const int e = ea + eb + (st > 0 && st < L ? (h == 2 ? max(i - 1, 0) : i) * lx : 0) - (h == 2 ? 0 : ED);
          mul<D, W>(tm, h == 0 ? pdl : pl, h == 1 ? pdy : py, levels(kGradBits2, e), r);
          if (h < 2) {
            to_frame<NV>(r, ea + eb, fq, 60);
#pragma unroll
            for (int v = 0; v < NV; ++v) q[v] = h == 0 ? r[v] : q[v] + r[v];
          }
        }
        // derivative
        if (st < L) {
          if (st == 0) {
            EdX = normalize<D, W>(tm, q, fq - 4);
            EX = normalize<D, W>(tm, r, 2 * EB, 1);
            store_planes<D, W>(tm, pdx, q, kSlices);
            store_planes<D, W>(tm, px, r, kSlices);
            const int fr = c_coef[2 * i].exp + g, fd = max(EdX + c_coef[2 * L].exp, ED + c_coef[2 * i + 1].exp) + 1;
            const Scaled sx(c_coef[2 * L], EX, fr, kFrac), sdx(c_coef[2 * L], EdX, fd, 60);
#pragma unroll
            for (int v = 0; v < NV; ++v) {
              r[v] = sx(r[v] << 6, 0);
              q[v] = sdx(q[v] << 6, 0);
            }
            const Scaled sb(c_coef[2 * i + 1], EB, fr, kFrac), sdb(c_coef[2 * i + 1], ED, fd, 60);
#pragma unroll
            for (int v = 0; v < NV; ++v) {
              r[v] = sb(b[v], r[v]);
              q[v] = sdb(db[v], q[v]);
            }
            add_diag<D, W>(tm, r, c_coef[2 * i], fr, kFrac);
            EY = fr;
            tm.sync();  // the maxima are read
            EdY = normalize<D, W>(tm, q, fd - 4);
            pl = px;
            pdl = pdx;
          } else {
            const int fd = max(fq, ED + c_coef[2 * i + 1].exp + 1) + 1;
            const Scaled sdb(c_coef[2 * i + 1], ED, fd, 60);
#pragma unroll
            for (int v = 0; v < NV; ++v) q[v] = sdb(db[v], q[v] >> min(fd - fq, 63));
            const int eq = normalize<D, W>(tm, q, fd - 4);
            if (!last) {
              const int fr = c_coef[2 * i].exp + g, F = i > 0 ? kFrac : 60;
              to_frame<NV>(r, EX + EY, fr, F);
              const Scaled sb(c_coef[2 * i + 1], EB, fr, F);
#pragma unroll
              for (int v = 0; v < NV; ++v) r[v] = sb(b[v], r[v]);
              add_diag<D, W>(tm, r, c_coef[2 * i], fr, F);
              EY = fr;
              if (i == 0) {
                tm.sync();
                EY = normalize<D, W>(tm, r, fr - 4);
              }
            }
            EdY = eq;
          }
        } else {
          const int eq = normalize<D, W>(tm, q, fq - 4);
          if (!last) {
            tm.sync();
            EY = normalize<D, W>(tm, r, 2 * EY);
          }
          EdY = eq;
        }
        if (!last) {
          tm.sync();  // every product of this step has read its planes
          store_planes<D, W>(tm, py, r, kSlices);
          store_planes<D, W>(tm, pdy, q, kSlices);
          if (i <= 0) {  // squarings: both factors are Y
            pl = py;
            pdl = pdy;
            EX = EY;
            EdX = EdY;
          }
        }
      }
#pragma unroll
      for (int v = 0; v < NV; ++v) q[v] <<= 2;
      put_traces<D, W>(T, tm, p, w, m, k, q, EdY, traces);
      tm.sync();  // the maxima and the traces are read
    }
  }
}

// Gate chains, parallel in time over blocks of `len` slices (identical launches
// read them as one shape, chain_shape):
//   k_fx_chain_fwd      per (member, block): R_k = U_{k-1} ... U_{k0} into the P
//                       slots (R_{k0} = I is implied) and the block product
//                       into the block's first P slot (F only: U slot)
//   k_fx_chain_combine  per member: T_b = the product before block b, z, f,
//                       kappa; Lambda_b = T' (product after block b); W_b =
//                       kappa T_b Lambda_b into the block's first P slot
//   k_fx_chain_bwd      per (member, block): V_k U_k = W_b U_{k1-1} ... U_k
//                       into the U slots, so P_k Lambda_{k-1} = R_k V_k U_k and
//                       M_k = P_k Lambda_k = R_k V_k with V_k = V_{k+1} U_{k+1}
// A block product is a chain of its own, so short pulses of few members fill
// the chip too; the forward, backward and gradient products are one each.
// Bound: the latency of a product, a few chains deep per SM (issue 42 %, tensor
// pipe 60 % with eight of them).  231 members of 1000 slices at d = 16: 8.1 + 16.6
// ms as one FP64 chain per member, 0.75 + 0.75 here; 32 members of 500 slices 2.1
// + 4.4 ms, 0.12 + 0.08.
template <int D> struct ChainCfg {
  static constexpr int W = kWarps<D>;
  static constexpr int TEAMS = D >= 32 ? 1 : 4;                // (member, block) chains of a CTA, mixed path
  // of the full chains: one at D = 16, where a CTA of four held 174 registers a
  // thread and left an SM with four chains (231 members of 1000 slices: forward
  // and backward 0.98 + 1.14 ms; eight chains, alone or in fours, 0.75 + 0.75
  // and 0.79 + 0.76)
  static constexpr int FULL_TEAMS = D >= 16 ? 1 : 8;
  static constexpr int PER_SM = D >= 32 ? 3 : D >= 16 ? 8 : 24;  // full chains an SM holds
  static constexpr int MIN_CTAS = D >= 32 ? 2 : D >= 16 ? 8 : 3;
  static constexpr int COMBINE = D >= 32 ? 2 : D >= 16 ? 4 : 8;  // teams of a member's combine
  static constexpr int TEAM_BYTES = 2 * Geo<D, W>::PLANES + kRed;            // the mixed path's chains
  static constexpr int FULL_BYTES = 2 * Geo<D, W>::PLANES_FULL + kRed;
  // T_b (b > 0) and Lambda_b of a member in shared memory
  static constexpr int MAX_BLOCKS = D >= 32 ? 3 : D >= 16 ? 20 : 96;
};

template <int D, int W, int S> struct ChainTeam {
  static constexpr int SET = S * 2 * Geo<D, W>::PLANE;
  Tm<D, W> tm;
  uint32_t pl, pr;  // planes of the left and the right factor
  __device__ __forceinline__ ChainTeam(unsigned char* smem, int team)
      : tm{(int)(threadIdx.x & 31), (int)(threadIdx.x >> 5) % W, 1 + team, reinterpret_cast<uint32_t*>(smem + 2 * SET)},
        pl(smem_u32(smem)), pr(pl + SET) {}
  // (r, E) <- left (r, E); an operand that is not finite stays so.  Full
  // matrices with S = 8, else 56 fractional bits and LEVELS levels.
  template <bool R_IS_LEFT, int LEVELS = kMaxLevels>
  __device__ __forceinline__ void step(long long (&r)[Geo<D, W>::NV], int& E, const long long (&x)[Geo<D, W>::NV], int Ex) {
    const uint32_t at_r = R_IS_LEFT ? pl : pr, at_x = R_IS_LEFT ? pr : pl;
    const bool bad = max(E, Ex) == kNotFinite;
    tm.sync();  // the last product has read its planes
    if constexpr (S == kFullSlices) {
      store_full<D, W, S>(tm, at_r, r);
      store_full<D, W, S>(tm, at_x, x);
      tm.sync();
      E += Ex;
      mul_full<D, W, S, LEVELS>(tm, pl, pr, r, E);
    } else {
      store_planes<D, W>(tm, at_r, r, kSlices);
      store_planes<D, W>(tm, at_x, x, kSlices);
      tm.sync();
      mul_fixed<D, W, LEVELS>(tm, pl, pr, r);
      E = normalize<D, W>(tm, r, E + Ex);
    }
    if (bad) E = kNotFinite;
  }
};

template <int D>
__global__ void __launch_bounds__(32 * ChainCfg<D>::W * ChainCfg<D>::FULL_TEAMS, ChainCfg<D>::MIN_CTAS)
k_fx_chain_fwd(ProbDev p, WorkDev w, int blocks, int len, int store) {
  using C = ChainCfg<D>;
  constexpr int W = C::W, NV = Geo<D, W>::NV;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int team = threadIdx.x / (32 * W);
  ChainTeam<D, W, kFullSlices> ct(smem_raw + (size_t)team * C::FULL_BYTES, team);
  const long item = (long)blockIdx.x * C::FULL_TEAMS + team;
  if (item >= (long)p.n_members * blocks) return;  // whole teams
  const int m = (int)(item / blocks), k0 = (int)(item % blocks) * len, k1 = min(p.n_t, k0 + len);
  const size_t base = (size_t)m * p.n_t;
  long long r[NV], x[NV];
  get_ints<NV>(slot(ct.tm, w.U, base + k0), r);
  int E = unpack(r);
  if (k0 + 1 < k1) get_ints<NV>(slot(ct.tm, w.U, base + k0 + 1), x);
#pragma unroll 1
  for (int k = k0 + 1; k < k1; ++k) {
    long long u[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) u[v] = x[v];
    const int Eu = unpack(u);
    if (k + 1 < k1) get_ints<NV>(slot(ct.tm, w.U, base + k + 1), x);  // while this product runs
    if (store) put_packed<D, W>(ct.tm, slot(ct.tm, w.P, base + k), r, E);
    ct.template step<false>(r, E, u, Eu);
  }
  put_packed<D, W>(ct.tm, slot(ct.tm, store ? w.P : w.U, base + k0), r, E);
}

template <int D>
__global__ void __launch_bounds__(32 * ChainCfg<D>::W * ChainCfg<D>::FULL_TEAMS, ChainCfg<D>::MIN_CTAS)
k_fx_chain_bwd(ProbDev p, WorkDev w, int blocks, int len) {
  using C = ChainCfg<D>;
  constexpr int W = C::W, NV = Geo<D, W>::NV;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int team = threadIdx.x / (32 * W);
  ChainTeam<D, W, kFullSlices> ct(smem_raw + (size_t)team * C::FULL_BYTES, team);
  const long item = (long)blockIdx.x * C::FULL_TEAMS + team;
  if (item >= (long)p.n_members * blocks) return;
  const int m = (int)(item / blocks), k0 = (int)(item % blocks) * len, k1 = min(p.n_t, k0 + len);
  const size_t base = (size_t)m * p.n_t;
  long long r[NV], x[NV];
  get_ints<NV>(slot(ct.tm, w.P, base + k0), r);
  int E = unpack(r);
  get_ints<NV>(slot(ct.tm, w.U, base + k1 - 1), x);
#pragma unroll 1
  for (int k = k1 - 1; k >= k0; --k) {
    long long u[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) u[v] = x[v];
    const int Eu = unpack(u);
    if (k > k0) get_ints<NV>(slot(ct.tm, w.U, base + k - 1), x);
    ct.template step<true>(r, E, u, Eu);
    put_packed<D, W>(ct.tm, slot(ct.tm, w.U, base + k), r, E);
  }
}

// A df matrix (the lanes' entries) in block fixed point; returns its exponent.
template <int D, int W>
__device__ __forceinline__ int from_df(const Tm<D, W>& tm, const float4 (&f)[Geo<D, W>::NV / 2], long long (&u)[Geo<D, W>::NV]) {
  constexpr int H = Geo<D, W>::NV / 2;
  uint32_t M = 0;
#pragma unroll
  for (int b = 0; b < H; ++b) M = max(M, max(__float_as_uint(f[b].x) & 0x7f800000u, __float_as_uint(f[b].y) & 0x7f800000u));
  const int EX = (int)(tm.max(M, 2) >> 23);
#pragma unroll
  for (int b = 0; b < H; ++b) {
    u[b] = from_float(f[b].x, EX) + from_float(f[b].z, EX);
    u[H + b] = from_float(f[b].y, EX) + from_float(f[b].w, EX);
  }
  return EX == 0xff ? kNotFinite : EX - 125;
}

// The mixed path's in-block prefixes: U_k as df pairs, R_k rounded to float2
// for the FP32 fix-up, block products as df pairs.  Seven levels: with six
// (2^-47.5 of the factors' scale) the defect of U_total, 4.8e-12 after 1000
// slices, passed that of the df products (9.6e-13); seven leave 1e-13.

template <int D>
__global__ void __launch_bounds__(32 * ChainCfg<D>::W * ChainCfg<D>::TEAMS, 2) k_fx_prefix_df(ProbDev p, WorkDev w, int store) {
  using C = ChainCfg<D>;
  constexpr int W = C::W, H = Geo<D, W>::NV / 2;
  using G = Geo<D, W>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int team = threadIdx.x / (32 * W);
  ChainTeam<D, W, kSlices> ct(smem_raw + (size_t)team * C::TEAM_BYTES, team);
  const Tm<D, W>& tm = ct.tm;
  const long item = (long)blockIdx.x * C::TEAMS + team;
  if (item >= (long)p.n_members * w.pit_blocks) return;  // whole teams
  const int m = (int)(item / w.pit_blocks), k0 = (int)(item % w.pit_blocks) * w.pit_len, k1 = min(p.n_t, k0 + w.pit_len);
  const float4* Um = reinterpret_cast<const float4*>(w.U) + (size_t)m * p.n_t * D * D;
  float2* Pm = reinterpret_cast<float2*>(w.P) + (size_t)m * p.n_t * D * D;
  int at[H];
#pragma unroll
  for (int b = 0; b < H; ++b) at[b] = tm.row(b / 2 % G::NI) + D * tm.col(b / 2 / G::NI, b % 2);
  long long r[2 * H];
  int E = 0;
  float4 f[H];
#pragma unroll
  for (int b = 0; b < H; ++b) {
    f[b] = Um[(size_t)k0 * D * D + at[b]];
    if (store) Pm[(size_t)k0 * D * D + at[b]] = make_float2(at[b] % D == at[b] / D ? 1.f : 0.f, 0.f);
  }
#pragma unroll 1
  for (int k = k0; k < k1; ++k) {
    long long u[2 * H];
    const int Eu = from_df<D, W>(tm, f, u);
    if (k + 1 < k1) {
#pragma unroll
      for (int b = 0; b < H; ++b) f[b] = Um[(size_t)(k + 1) * D * D + at[b]];  // while this product runs
    }
    if (k == k0) {
#pragma unroll
      for (int v = 0; v < 2 * H; ++v) r[v] = u[v];
      E = Eu;
      tm.sync();  // the maxima are read
    } else {
      ct.template step<false, kPrefixLevels>(r, E, u, Eu);
    }
    if (store && k + 1 < k1) {
      const float sc = E == kNotFinite ? __int_as_float(0x7fc00000) : ldexpf(1.f, E - kFrac);
#pragma unroll
      for (int b = 0; b < H; ++b)
        Pm[(size_t)(k + 1) * D * D + at[b]] = make_float2(to_df(r[b], sc).x, to_df(r[H + b], sc).x);
    }
  }
  store_df<D, W>(tm, w.pit_tot + (size_t)item * D * D, r, E == kNotFinite ? 0x7ff : E - kFrac);
}

// x -> kappa x, both full: each part times a double, in a common frame; returns
// its exponent.
template <int D, int W>
__device__ __forceinline__ int scale_complex(const Tm<D, W>& tm, long long (&x)[Geo<D, W>::NV], int E, double2 kap) {
  constexpr int H = Geo<D, W>::NV / 2;
  const int ex = max((int)((uint32_t)__double2hiint(kap.x) >> 20 & 0x7ff), (int)((uint32_t)__double2hiint(kap.y) >> 20 & 0x7ff));
  if (ex == 0x7ff) return kNotFinite;
  // parts below 2^(ex - 1022) in 61 fractional bits, x in 61
  const long long a = from_double(kap.x, ex, 8), b = from_double(kap.y, ex, 8);
  const int a0 = (int)a, a1 = (int)((a + 0x80000000ll) >> 32), b0 = (int)b, b1 = (int)((b + 0x80000000ll) >> 32);
#pragma unroll
  for (int v = 0; v < H; ++v) {
    const long long re = shift_round(x[v], 3), im = shift_round(x[H + v], 3);
    const int r0 = (int)re, r1 = (int)((re + 0x80000000ll) >> 32);
    const int i0 = (int)im, i1 = (int)((im + 0x80000000ll) >> 32);
    const long long mr = (long long)r1 * a0 + (long long)r0 * a1 - (long long)i1 * b0 - (long long)i0 * b1;
    const long long mi = (long long)r1 * b0 + (long long)r0 * b1 + (long long)i1 * a0 + (long long)i0 * a1;
    x[v] = (((long long)r1 * a1 - (long long)i1 * b1) << 3) + shift_round(mr, 29);
    x[H + v] = (((long long)r1 * b1 + (long long)i1 * a1) << 3) + shift_round(mi, 29);
  }
  const int e = normalize_full<D, W>(tm, x, E + ex - 1024 + 5, 1);
  return E == kNotFinite ? kNotFinite : e;
}

// U_total of a member, r with FRAC fractional bits.
template <int D, int W, int FRAC>
__device__ __forceinline__ void put_total(const Tm<D, W>& tm, const WorkDev& w, int m, const long long (&r)[Geo<D, W>::NV], int E) {
  double2* Ut = w.Utot + (size_t)m * D * D;
  if (E == kNotFinite) store_nan<D, W>(tm, Ut);
  else store_mat<D, W>(tm, Ut, r, E - FRAC);
}
// z = Tr(T' U) / D, f and the weighted kappa of a member from U, the team's
// (r, E), FRAC fractional bits; the team is threads 0 .. 32 W - 1 of the block.
template <int D, int W, int FRAC>
__device__ __forceinline__ void finish_gate(const Tm<D, W>& tm, const ProbDev& p, const WorkDev& w, int m,
                                            const long long (&r)[Geo<D, W>::NV], int E, double2* s_red, double2* s_kap) {
  using G = Geo<D, W>;
  constexpr int NV = G::NV;
  double2 acc = make_double2(0.0, 0.0);
#pragma unroll
  for (int b = 0; b < NV / 2; ++b) {
    double2 v = make_double2(to_double(r[b], E - FRAC), to_double(r[NV / 2 + b], E - FRAC));
    if (E == kNotFinite) v.x = v.y = __longlong_as_double(0x7ff8000000000000ll);
    acc = cmac_cj(acc, p.target_op[tm.row(b / 2 % G::NI) + D * tm.col(b / 2 / G::NI, b % 2)], v);
  }
  s_red[threadIdx.x] = acc;
  tm.sync();
  for (int h = 16 * W; h > 0; h >>= 1) {
    if ((int)threadIdx.x < h) s_red[threadIdx.x] = cadd(s_red[threadIdx.x], s_red[threadIdx.x + h]);
    tm.sync();
  }
  if (threadIdx.x == 0) {
    double2 z = s_red[0], kap;
    z.x /= p.D;
    z.y /= p.D;
    double f;
    fid_kappa(z, p.fid, p.grad_mode, f, kap);
    const double sc = p.m_weight[m] / p.D;
    kap = make_double2(kap.x * sc, kap.y * sc);
    w.z[m] = z;
    w.kap[m] = kap;
    w.Fm[m] = f;
    *s_kap = kap;
  }
}

// Per member, the mixed path's block products in order (T_b in df pairs, the
// prefixes before each block rounded to float2): a latency-bound chain of one
// team, whose product takes about 1.5 us at D = 16 and 3 us at D = 32 where the
// CUDA-core df product of the same chain took 2.2 and 10.
template <int D>
__global__ void __launch_bounds__(32 * ChainCfg<D>::W) k_fx_combine_df(ProbDev p, WorkDev w, int store) {
  using C = ChainCfg<D>;
  constexpr int W = C::W, H = Geo<D, W>::NV / 2;
  using G = Geo<D, W>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double2 s_red[32 * W];
  __shared__ double2 s_kap;
  ChainTeam<D, W, kSlices> ct(smem_raw, 0);
  const Tm<D, W>& tm = ct.tm;
  const int m = blockIdx.x;
  int at[H];
#pragma unroll
  for (int b = 0; b < H; ++b) at[b] = tm.row(b / 2 % G::NI) + D * tm.col(b / 2 / G::NI, b % 2);
  long long r[2 * H];
  int E = 0;
  float4 f[H];
#pragma unroll
  for (int b = 0; b < H; ++b) f[b] = w.pit_tot[(size_t)m * w.pit_blocks * D * D + at[b]];
#pragma unroll 1
  for (int b = 0; b < w.pit_blocks; ++b) {
    const size_t blk = ((size_t)m * w.pit_blocks + b) * D * D;
    if (store) {
      const float sc = E == kNotFinite ? __int_as_float(0x7fc00000) : ldexpf(1.f, E - kFrac);
#pragma unroll
      for (int i = 0; i < H; ++i)
        w.pit_pre[blk + at[i]] = b == 0 ? make_float2(at[i] % D == at[i] / D ? 1.f : 0.f, 0.f)
                                        : make_float2(to_df(r[i], sc).x, to_df(r[H + i], sc).x);
    }
    long long u[2 * H];
    const int Eu = from_df<D, W>(tm, f, u);
    if (b + 1 < w.pit_blocks) {
#pragma unroll
      for (int i = 0; i < H; ++i) f[i] = w.pit_tot[blk + D * D + at[i]];
    }
    if (b == 0) {
#pragma unroll
      for (int v = 0; v < 2 * H; ++v) r[v] = u[v];
      E = Eu;
      tm.sync();  // the maxima are read
    } else {
      ct.template step<false, kPrefixLevels>(r, E, u, Eu);
    }
  }
  put_total<D, W, kFrac>(tm, w, m, r, E);
  if (p.gen == GEN_HERM && E != kNotFinite) {
    // one Newton-Schulz step of the polar decomposition, U (3I - U'U) / 2,
    // before the overlap (k_refine_unitary_mx, which takes 10 us at D = 16
    // and 76 us at D = 32 on the FP64 pipe)
    tm.sync();
    store_planes<D, W>(tm, ct.pl, r, kSlices);
    tm.sync();
    long long s[2 * H];
    mul_fixed<D, W, kMaxLevels, LeftH<D, W>>(tm, ct.pl, ct.pl, s);
    to_frame<2 * H>(s, 2 * E, 3, kFrac);
#pragma unroll
    for (int v = 0; v < 2 * H; ++v) s[v] = -s[v];
#pragma unroll
    for (int i = 0; i < H; ++i)
      if (at[i] % D == at[i] / D) s[i] += 3ll << (kFrac - 3);
    store_planes<D, W>(tm, ct.pr, s, kSlices);
    tm.sync();
    mul_fixed<D, W, kMaxLevels>(tm, ct.pl, ct.pr, r);
    E += 2;  // frame 3, halved
  }
  finish_gate<D, W, kFrac>(tm, p, w, m, r, E, s_red, &s_kap);
}

template <int D>
__global__ void __launch_bounds__(32 * ChainCfg<D>::W * ChainCfg<D>::COMBINE)
k_fx_chain_combine(ProbDev p, WorkDev w, int blocks, int len, int want_grad) {
  using C = ChainCfg<D>;
  constexpr int W = C::W;
  using G = Geo<D, W>;
  constexpr int NV = G::NV, TEAMS = C::COMBINE;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double2 s_red[32 * W];
  __shared__ double2 s_kap;
  const int team = threadIdx.x / (32 * W);
  ChainTeam<D, W, kFullSlices> ct(smem_raw + (size_t)team * C::FULL_BYTES, team);
  const Tm<D, W>& tm = ct.tm;
  longlong2* Ls = reinterpret_cast<longlong2*>(smem_raw + (size_t)TEAMS * C::FULL_BYTES);
  longlong2* Ts = Ls + (size_t)(blocks - 1) * (G::INTS / 16);  // T_b at b, b > 0: after Lambda's last
  const int m = blockIdx.x;
  const size_t base = (size_t)m * p.n_t;
  double2* tot = want_grad ? w.P : w.U;  // where k_fx_chain_fwd left the block products
  long long r[NV], x[NV];
  if (team == 0) {  // T_1 = Tot_0, T_{b+1} = Tot_b T_b
    get_ints<NV>(slot(tm, tot, base), r);
    int E = unpack(r);
#pragma unroll 1
    for (int b = 1; b < blocks; ++b) {
      if (want_grad) put_packed<D, W>(tm, tm.mine(Ts + (size_t)b * (G::INTS / 16)), r, E);
      get_ints<NV>(slot(tm, tot, base + (size_t)b * len), x);
      const int Ex = unpack(x);
      ct.template step<false>(r, E, x, Ex);
    }
    put_total<D, W, 64>(tm, w, m, r, E);
    finish_gate<D, W, 64>(tm, p, w, m, r, E, s_red, &s_kap);
  } else if (team == 1 && want_grad) {  // Lambda_B = T', Lambda_{b-1} = Lambda_b Tot_b
    double t[NV];
#pragma unroll
    for (int b = 0; b < NV / 2; ++b) {
      const double2 v = p.target_op[tm.col(b / 2 / G::NI, b % 2) + D * tm.row(b / 2 % G::NI)];
      t[b] = v.x;
      t[NV / 2 + b] = -v.y;
    }
    const int EX = max_exponent<D, W>(tm, t);
#pragma unroll
    for (int v = 0; v < NV; ++v) r[v] = from_double(t[v], EX, 9);
    int E = EX - 1020;
#pragma unroll 1
    for (int b = blocks - 1;; --b) {
      put_packed<D, W>(tm, tm.mine(Ls + (size_t)b * (G::INTS / 16)), r, E);
      if (b == 0) break;
      get_ints<NV>(slot(tm, tot, base + (size_t)b * len), x);
      const int Ex = unpack(x);
      ct.template step<true>(r, E, x, Ex);
    }
  }
  if (!want_grad) return;
  __syncthreads();
  const double2 kap = s_kap;
  for (int b = team; b < blocks; b += TEAMS) {  // W_b = kappa T_b Lambda_b
    get_ints<NV>(tm.mine(Ls + (size_t)b * (G::INTS / 16)), r);
    int E = unpack(r);
    if (b > 0) {
      get_ints<NV>(tm.mine(Ts + (size_t)b * (G::INTS / 16)), x);
      const int Ex = unpack(x);
      ct.template step<false>(r, E, x, Ex);
    }
    E = scale_complex<D, W>(tm, r, E, kap);
    put_packed<D, W>(tm, slot(tm, w.P, base + (size_t)b * len), r, E);
  }
}

// State chains, forward and backward together: one warp per (member, pair,
// direction) applies the slices to its vector in 64-bit integers.
//   forward   psi_{k+1} = U_k psi_k, z_s, f, kappa
//   backward  lambda_k = U_k' lambda_{k+1} from lambda_n = t_s, stored without
//             the factor conj(kappa_s) (the gradient applies it), so it does not
//             wait for the forward chain
//
// Bound: the latency of one step, n_t times.  A warp's FP64 FMA takes 70 cycles
// of its scheduler's pipe, so FP64 chains spent 1,500 (D = 2) to 3,000 cycles a
// slice; a complex multiply-add is 12 integer ones here.  Only the multiply-
// adds, their sum over the lanes of a row and the hand-over of the vector are
// left on the chain: eight helper warps load and convert the next chunk of
// slices and write the last chunk's vectors out meanwhile.  (With the
// conversions in the chain's own warp a D = 2 step took 1,070 cycles.)
//
// Vectors are x 2^(E - 57) with one exponent, U_k's entries u 2^-G, both in two
// balanced halves of 30 bits; y = x u 2^-G takes all four partial products, so
// a step only rounds its result.  (Without the low one, overlaps of 1e-3 lost
// five bits against FP64, which keeps small amplitudes to their own scale.)
//   Hermitian generators keep the vector's norm, so its exponent never moves:
//   ||x|| <= 2^60.5 from the start (which leaves a basis state's small
//   amplitudes 2^-60 of its norm), so a component's high half stays below 2^31,
//   and G = 60 with ||u|| <= 2^60 in every row: high sums stay below 2^61, the
//   mixed ones of eight columns below 2^62.3 (Cauchy-Schwarz).
//   Others: the larger scale of |x| < 2^57 (2^56 at D = 32) and sum |x| < 2^60
//   over both parts of all components (near a basis state, whose small
//   components it leaves three more bits), renewed every step; |u| < 2^G of
//   U_k's largest entry, G = 60 up to D = 8, where a lane has one or two columns,
//   and 59 above: a row's sum is below 2^62 either way, the mixed sums of eight
//   columns below 2^62.4.
// At D = 32 a lane sums its row in four parts, so the mixed and low sums stay
// inside 63 bits as at D = 16 (200 slices of 8 members and two pairs at d = 24:
// 1.01 + 1.12 ms in FP64 on shared memory, 0.55 ms here).
template <int D> struct StCfg {
  static constexpr int QS = 32 / D < D ? 32 / D : D;  // lanes that share a row
  static constexpr int QN = D / QS;                   // columns of a lane
  static constexpr int ACTIVE = D * QS;               // the other lanes repeat their work
  static constexpr int CH = D >= 32 ? 1 : D >= 16 ? 2 : D >= 8 ? 8 : 128 / D;  // slices of a chunk
  static constexpr int QB = QN < 8 ? QN : 8;          // columns summed at a time
  static constexpr int GUARD = D >= 32 ? 1 : 0;       // one bit less of a vector that may grow (below)
  __host__ __device__ static constexpr int ubits(bool herm) { return herm || D <= 8 ? 60 : 59; }  // G below
  static constexpr int HELPERS = 8;
  static constexpr int NPT = 2 * CH * D * D / (32 * HELPERS);  // entries of a helper lane and chunk, both directions
  static constexpr int RING = 2 * CH * D * D;         // entries of one chunk
  __host__ __device__ static constexpr size_t smem(int chains) {
    return (size_t)16 * (2 * RING + 2 * chains * CH * D) + sizeof(int) * (2 * 2 * CH + 2 * chains * CH);
  }
};

__device__ __forceinline__ int4 split2(long long re, long long im) {  // x = hi 2^30 + lo, |lo| <= 2^29
  const int r0 = (int)((uint32_t)re << 2) >> 2, i0 = (int)((uint32_t)im << 2) >> 2;
  return make_int4(r0, (int)((re - r0) >> 30), i0, (int)((im - i0) >> 30));
}
__device__ __forceinline__ long long join2(int lo, int hi) { return ((long long)hi << 30) + lo; }

template <int D, bool HERM>
__global__ void __launch_bounds__(32 * (16 + StCfg<D>::HELPERS)) k_fx_states(ProbDev p, WorkDev w, int store) {
  using C = StCfg<D>;
  constexpr int QN = C::QN, QS = C::QS, QB = C::QB, CH = C::CH, NPT = C::NPT;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double s_f[8];
  __shared__ int s_bad;
  const int np = p.n_pairs, chains = store ? 2 * np : np, m = blockIdx.x;
  int4* ring = reinterpret_cast<int4*>(smem_raw);      // [2][direction][CH][D D]
  int4* hist = ring + 2 * C::RING;                     // [2][chain][CH][D] the chunk's vectors
  int* s_eu = reinterpret_cast<int*>(hist + 2 * chains * CH * D);  // [2][direction][CH] biased exponents
  int* s_ev = s_eu + 2 * 2 * CH;                       // [2][chain][CH]
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const double2* Um = w.U + (size_t)m * p.n_t * D * D;
  const size_t pan = (size_t)np * D;
  const int chunks = (p.n_t + CH - 1) / CH;
  // entry (i, c) of a slice at column c, row i ^ (c mod 8): rows and columns
  // both read without bank conflicts
  auto swz = [](int i, int c) { return c * D + (i ^ (c & (D < 8 ? D - 1 : 7))); };
  if (threadIdx.x == 0) s_bad = 0;
  if (!HERM)
    for (int i = threadIdx.x; i < 2 * 2 * CH; i += blockDim.x) s_eu[i] = 0;
  __syncthreads();

  if (wid >= chains) {  // helpers
    const int h = threadIdx.x - 32 * chains;
    double2 raw[NPT];
    auto where = [&](int c, int i, int& dir, int& sl, int& e) {  // entry i of chunk c: its slice, or -1
      const int x = i * 32 * C::HELPERS + h;
      dir = x / (CH * D * D);
      sl = x / (D * D) % CH;
      e = x % (D * D);
      const int st = c * CH + sl;
      return st < p.n_t && (dir == 0 || store) ? (dir == 0 ? st : p.n_t - 1 - st) : -1;
    };
    auto fetch = [&](int c) {
      if (c >= chunks) return;
#pragma unroll
      for (int i = 0; i < NPT; ++i) {
        int dir, sl, e;
        const int k = where(c, i, dir, sl, e);
        raw[i] = k >= 0 ? Um[(size_t)k * D * D + e] : make_double2(0.0, 0.0);
      }
    };
    auto convert = [&](int c) {
      if (c >= chunks) return;
      const int buf = c & 1;
      int dir, sl, e;
      bool bad = false;
#pragma unroll
      for (int i = 0; i < NPT; ++i) {
        where(c, i, dir, sl, e);
        const int ex = (int)(max((uint32_t)__double2hiint(raw[i].x) & 0x7ff00000u,
                                 (uint32_t)__double2hiint(raw[i].y) & 0x7ff00000u) >> 20);
        bad |= ex >= (HERM ? 1024 : 0x7ff);  // a unitary's entries stay below 2
        if (!HERM) atomicMax(&s_eu[(buf * 2 + dir) * CH + sl], ex);
      }
      if (bad) s_bad = 1;
      if (!HERM) asm volatile("bar.sync 1, %0;" ::"n"(32 * C::HELPERS) : "memory");
#pragma unroll
      for (int i = 0; i < NPT; ++i) {
        where(c, i, dir, sl, e);
        const int EX = HERM ? 1023 : s_eu[(buf * 2 + dir) * CH + sl];
        constexpr int guard = C::ubits(HERM) - (HERM ? 52 : 53);
        ring[(size_t)(buf * 2 + dir) * CH * D * D + sl * D * D + swz(e % D, e / D)] =
            split2(from_double(raw[i].x, EX, guard), from_double(raw[i].y, EX, guard));
      }
    };
    auto put = [&](int c) {  // the vectors of chunk c
      if (!store) return;
      const int buf = c & 1;
      for (int x = h; x < chains * CH * D; x += 32 * C::HELPERS) {
        const int ch = x / (CH * D), sl = x / D % CH, r = x % D, st = c * CH + sl;
        if (st >= p.n_t) continue;
        const int4 v = hist[(size_t)(buf * chains + ch) * CH * D + sl * D + r];
        const int E = s_ev[(buf * chains + ch) * CH + sl];
        double2* out = (ch < np ? w.psi : w.lam) + ((size_t)m * (p.n_t + 1) + (ch < np ? st + 1 : p.n_t - 1 - st)) * pan;
        double2 d = make_double2(to_double(join2(v.x, v.y), E - 57), to_double(join2(v.z, v.w), E - 57));
        if (E == kNotFinite) d.x = d.y = __longlong_as_double(0x7ff8000000000000ll);
        out[(size_t)(ch % np) * D + r] = d;
      }
    };
    fetch(0);
    convert(0);
    fetch(1);
    if (store)
      for (int x = h; x < chains * D; x += 32 * C::HELPERS) {  // both ends
        const int ch = x / D, r = x % D;
        const size_t at = (size_t)(ch % np) * D + r;
        if (ch < np) w.psi[(size_t)m * (p.n_t + 1) * pan + at] = p.psi_init[at];
        else w.lam[((size_t)m * (p.n_t + 1) + p.n_t) * pan + at] = p.psi_targ[at];
      }
    __syncthreads();
#pragma unroll 1
    for (int c = 0; c < chunks; ++c) {
      if (!HERM) {  // the exponents of the chunk before last are read
        for (int i = h; i < 2 * CH; i += 32 * C::HELPERS) s_eu[((c + 1) & 1) * 2 * CH + i] = 0;
        asm volatile("bar.sync 1, %0;" ::"n"(32 * C::HELPERS) : "memory");
      }
      convert(c + 1);
      fetch(c + 2);
      if (c > 0) put(c - 1);
      __syncthreads();
    }
    put(chunks - 1);
    __syncthreads();
    return;
  }

  const bool fwd = wid < np;
  const int s = wid % np, dir = fwd ? 0 : 1;
  const int al = lane & (C::ACTIVE - 1), r = al % D, q0 = al / D * QN;
  int E;
  bool bad;
  int4 first;  // the start vector, of row `r`
  {
    const double2 v0 = (fwd ? p.psi_init : p.psi_targ)[s * D + r];
    const int EX = (int)(__reduce_max_sync(0xffffffffu, max((uint32_t)__double2hiint(v0.x) & 0x7ff00000u,
                                                            (uint32_t)__double2hiint(v0.y) & 0x7ff00000u)) >> 20);
    bad = EX == 0x7ff;
    // from the norm, ||x|| <= 2^60.5, or the sum of the parts, below 2^60, in
    // units of 2^(EX - 1022)
    const float re = (float)scalbn(v0.x, 1022 - EX), im = (float)scalbn(v0.y, 1022 - EX);
    float sum = HERM ? fmaf(re, re, im * im) : fabsf(re) + fabsf(im);
#pragma unroll
    for (int o = 1; o < D; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const int guard = HERM ? min(max((int)floorf(7.499f - 0.5f * __log2f(sum)), 0), 8)
                           : min(max((int)floorf(6.999f - __log2f(sum)), 4 - C::GUARD), 7);
    first = split2(from_double(v0.x, EX, guard), from_double(v0.y, EX, guard));
    E = EX - 1018 - guard;  // x 2^(EX - 1075 - guard)
  }
  // the start vector goes where chunk -1 would have left its last one
  int4* mine = hist + (size_t)wid * CH * D;
  const size_t other = (size_t)chains * CH * D;
  if (lane < D) mine[other + (CH - 1) * D + r] = first;
  int4 last = first;
  __syncthreads();
#pragma unroll 1
  for (int c = 0; c < chunks; ++c) {
    const int buf = c & 1, n = min(CH, p.n_t - c * CH);
    const int4* U = ring + (size_t)(buf * 2 + dir) * CH * D * D;
    const int4* prev = mine + (buf ? 0 : other) + (CH - 1) * D;
    int4* cur = mine + (buf ? other : 0);
    // U_k's entries of columns q0 + b QB and on (rows in the backward chain)
    int4 u[QB];
    auto load = [&](const int4* V, int b) {
#pragma unroll
      for (int i = 0; i < QB; ++i) {
        const int q = q0 + b * QB + i;
        u[i] = V[fwd ? swz(r, q) : swz(q, r)];
      }
    };
    load(U, 0);
#pragma unroll 1
    for (int sl = 0; sl < n; ++sl) {
      const int EX = HERM ? 0 : s_eu[(buf * 2 + dir) * CH + sl];
      long long yr = 0, yi = 0;
#pragma unroll 1
      for (int b = 0; b < QN / QB; ++b) {
        // re = sum ur xr -+ ui xi, im = sum ur xi +- ui xr (backward: conj(U))
        // high, mixed and low partial products of the four sums
        long long pr = 0, pi = 0, nr = 0, ni = 0, mpr = 0, mpi = 0, mnr = 0, mni = 0, lpr = 0, lpi = 0, lnr = 0, lni = 0;
#pragma unroll
        for (int i = 0; i < QB; ++i) {
          const int4 x = prev[q0 + b * QB + i];
          pr += (long long)u[i].y * x.y;
          mpr += (long long)u[i].y * x.x + (long long)u[i].x * x.y;
          lpr += (long long)u[i].x * x.x;
          nr += (long long)u[i].w * x.w;
          mnr += (long long)u[i].w * x.z + (long long)u[i].z * x.w;
          lnr += (long long)u[i].z * x.z;
          pi += (long long)u[i].y * x.w;
          mpi += (long long)u[i].y * x.z + (long long)u[i].x * x.w;
          lpi += (long long)u[i].x * x.z;
          ni += (long long)u[i].w * x.y;
          mni += (long long)u[i].w * x.x + (long long)u[i].z * x.y;
          lni += (long long)u[i].z * x.x;
        }
        if (b + 1 < QN / QB) load(U + sl * D * D, b + 1);
        else if (sl + 1 < n) load(U + (sl + 1) * D * D, 0);
        constexpr int SH = 60 - C::ubits(HERM);
        const long long mr = (fwd ? mpr - mnr : mpr + mnr) + ((fwd ? lpr - lnr : lpr + lnr) >> 30);
        const long long mi = (fwd ? mpi + mni : mpi - mni) + ((fwd ? lpi + lni : lpi - lni) >> 30);
        yr += ((fwd ? pr - nr : pr + nr) << SH) + shift_round(mr, 30 - SH);
        yi += ((fwd ? pi + ni : pi - ni) << SH) + shift_round(mi, 30 - SH);
      }
#pragma unroll
      for (int o = D; o < D * QS; o <<= 1) {
        yr += __shfl_xor_sync(0xffffffffu, yr, o);
        yi += __shfl_xor_sync(0xffffffffu, yi, o);
      }
      if (!HERM) {
        const uint32_t top = __reduce_max_sync(0xffffffffu, max((uint32_t)abs((int)(yr >> 32)), (uint32_t)abs((int)(yi >> 32))));
        // the sum of all rows' parts is below part 2^36 (the lanes hold 32 / D copies)
        const uint32_t part = (__reduce_add_sync(0xffffffffu, ((uint32_t)abs((int)(yr >> 32)) + (uint32_t)abs((int)(yi >> 32))) >> 4) / (32 / D)) + 4 * D;
        const int sh = max(__clz(top + 1) - 7 - C::GUARD, __clz(part) - 8);
        yr = sh >= 0 ? yr << sh : shift_round(yr, -sh);
        yi = sh >= 0 ? yi << sh : shift_round(yi, -sh);
        E = max(E + EX - 1022 - sh, -(1 << 20));
      }
      last = split2(yr, yi);
      if (lane < D) cur[sl * D + r] = last;
      if (lane == 0) s_ev[(buf * chains + wid) * CH + sl] = bad ? kNotFinite : E;
      __syncwarp();
      prev = cur + sl * D;
    }
    __syncthreads();
  }
  if (fwd) {
    double2 d = make_double2(to_double(join2(last.x, last.y), E - 57), to_double(join2(last.z, last.w), E - 57));
    if (bad || s_bad) d.x = d.y = __longlong_as_double(0x7ff8000000000000ll);
    double2 z = make_double2(0.0, 0.0);
    if (lane < D) z = cmac_cj(z, p.psi_targ[s * D + r], d);
#pragma unroll
    for (int o = D / 2; o > 0; o >>= 1) {
      z.x += __shfl_xor_sync(0xffffffffu, z.x, o);
      z.y += __shfl_xor_sync(0xffffffffu, z.y, o);
    }
    if (lane == 0) {
      double f;
      double2 kap;
      fid_kappa(z, p.fid, p.grad_mode, f, kap);
      const double wgt = p.m_weight[m];
      w.z[(size_t)m * np + s] = z;
      w.kap[(size_t)m * np + s] = make_double2(kap.x * wgt, kap.y * wgt);
      s_f[s] = f;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double Fm = 0.0;
    for (int i = 0; i < np; ++i) Fm += s_f[i];
    w.Fm[m] = Fm;
  }
}

// ---- the mixed path's exact gradient ---------------------------------------------
// The commutator series of k_fx_grad in FP32 class: X = sum ad_A^n(N) / (n + 1)!
// until a term is below 2^-27 of N, six or so at ||A|| = 0.15, each one
// A D - D A in 3xFP16 (x = hi + lo in FP16, 22 bits; lo hi + hi lo + hi hi
// accumulated in FP32).  N and every term are scaled by a power of two to a
// largest entry in [1/2, 1), so FP16's range covers 2^-25 of it.
//
// The CUDA-core Frechet derivative (k_grad_gate_mx) executes 15 FP32 products
// bound by shared-memory operand loads; here A's fragments stay in registers
// and a term is 24 MMAs a warp and one pass of D through shared memory.
//
// The series needs ||A|| up to about 1: the propagator kernel raises
// w.norm_flag for an evaluation that has larger slices, which then runs the
// CUDA-core gradient (and its chains' pairing M_k instead of N_k).
//
// Gradients against long double over the same draws, as a part of the FP32
// kernels' error: gates 0.4 to 0.6 at d = 9 to 32 (Lindblad 0.37), four-spin
// transfers 0.45, random transfers 0.99 to 1.00 (their FP32 vectors set it).
template <int D> struct TfCfg {
  static constexpr int W = kWarps<D>;
  static constexpr int TEAMS = D >= 32 ? 1 : 4;
  static constexpr int MIN_CTAS = D >= 32 ? 2 : 3;
  static constexpr int SPLIT = 4 * Geo<D, W>::PLANE;  // bytes of a hi, lo pair of matrices
  static constexpr int TRACE = 32;                    // controls of one pass over the traces
  static constexpr int TEAM_BYTES = 2 * SPLIT + W * TRACE * 4 + kRed;
};

// x -> hi, lo planes (FP16).
template <int D, int W>
__device__ __forceinline__ void store_split(const Tm<D, W>& tm, uint32_t base, const float (&x)[Geo<D, W>::NV]) {
  using G = Geo<D, W>;
  constexpr int NV = G::NV;
  const uint32_t at = base + (tm.nt0() * (D / 8) + 2 * tm.rt()) * 128 + tm.lane * 4;
#pragma unroll
  for (int b = 0; b < NV / 2; ++b) {
    const int part = b / (NV / 4), nt = b % (NV / 4) / G::NI, i = b % G::NI;
    const float u = x[2 * b], v = x[2 * b + 1];
    uint32_t h, l;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(h) : "f"(v), "f"(u));
    float hu, hv;
    asm("{.reg .f16 a, b; mov.b32 {a, b}, %2; cvt.f32.f16 %0, a; cvt.f32.f16 %1, b;}" : "=f"(hu), "=f"(hv) : "r"(h));
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(l) : "f"(v - hv), "f"(u - hu));
    const uint32_t to = at + part * G::PLANE + (nt * (D / 8) + i) * 128;
    asm volatile("st.shared.b32 [%0], %1;" ::"r"(to), "r"(h) : "memory");
    asm volatile("st.shared.b32 [%0], %1;" ::"r"(to + 2 * G::PLANE), "r"(l) : "memory");
  }
}

// 2^-e with the team's largest |x| in [1/2, 1) after scaling by it (1 when all
// are zero or not finite).
template <int D, int W>
__device__ __forceinline__ float unit_scale(const Tm<D, W>& tm, const float (&x)[Geo<D, W>::NV], int slot) {
  uint32_t M = 0;
#pragma unroll
  for (int v = 0; v < Geo<D, W>::NV; ++v) M = max(M, __float_as_uint(x[v]) & 0x7fffffffu);
  const int ex = (int)(tm.max(M, slot) >> 23);
  return ex == 0 || ex >= 253 ? 1.f : __uint_as_float((uint32_t)(252 - ex + 1) << 23);  // 2^(126 - ex)
}

// A = c dt_k (drift + off O + tau_k R + scale sum_j u_jk C_j) in FP32.
template <int D, int W>
__device__ __forceinline__ void assemble32(const Tm<D, W>& tm, const ProbDev& p, const WorkDev& w, int m, int k,
                                           const int (&at)[Geo<D, W>::NV / 2], float (&A)[Geo<D, W>::NV]) {
  constexpr int H = Geo<D, W>::NV / 2;
  const float dt = p.dt_df[k].x, sc = p.m_scale_df[m].x, off = p.m_offset_df[m].x;
  const float2* Gd = p.drifts_f32 + (size_t)p.m_drift[m] * D * D;
  const float2* uk = w.u_df + (size_t)k * p.n_c;
  const int ro = p.n_ramp ? p.m_ramp[m] : -1;
  float2 v[H];
#pragma unroll
  for (int b = 0; b < H; ++b) {
    const float2 g = Gd[at[b]], o = p.offset_f32[at[b]];
    v[b] = make_float2(fmaf(off, o.x, g.x), fmaf(off, o.y, g.y));
  }
  if (ro >= 0) {
    const float4* Rm = p.ramp_ops_df + (size_t)ro * D * D;
    const float tk = p.tau_df[k].x;
#pragma unroll
    for (int b = 0; b < H; ++b) v[b] = make_float2(fmaf(tk, Rm[at[b]].x, v[b].x), fmaf(tk, Rm[at[b]].y, v[b].y));
  }
#pragma unroll 1
  for (int j = 0; j < p.n_c; ++j) {
    const float a = sc * uk[j].x;
    const float2* Cj = p.ctrls_f32 + (size_t)j * D * D;
#pragma unroll
    for (int b = 0; b < H; ++b) {
      const float2 c = Cj[at[b]];
      v[b] = make_float2(fmaf(a, c.x, v[b].x), fmaf(a, c.y, v[b].y));
    }
  }
#pragma unroll
  for (int b = 0; b < H; ++b) {
    A[b] = dt * (p.gen == GEN_HERM ? v[b].y : v[b].x);
    A[H + b] = dt * (p.gen == GEN_HERM ? -v[b].x : v[b].y);
  }
}

template <int D>
__global__ void __launch_bounds__(32 * TfCfg<D>::W * TfCfg<D>::TEAMS, TfCfg<D>::MIN_CTAS) k_tf_grad(ProbDev p, WorkDev w) {
  using C = TfCfg<D>;
  constexpr int W = C::W;
  using G = Geo<D, W>;
  constexpr int NV = G::NV, H = NV / 2, KT = G::KT;
  if (*w.norm_flag) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int team = threadIdx.x / (32 * W);
  unsigned char* mine = smem_raw + (size_t)team * C::TEAM_BYTES;
  const uint32_t pa = smem_u32(mine), pd = pa + C::SPLIT;
  float* traces = reinterpret_cast<float*>(mine + 2 * C::SPLIT);  // [W][TRACE]
  const Tm<D, W> tm{(int)(threadIdx.x & 31), (int)(threadIdx.x >> 5) % W, 1 + team,
                    reinterpret_cast<uint32_t*>(mine + C::TEAM_BYTES - kRed)};
  int at[H], tr[H];  // the lane's entries, and their transposes
#pragma unroll
  for (int b = 0; b < H; ++b) {
    const int r = tm.row(b / 2 % G::NI), c = tm.col(b / 2 / G::NI, b % 2);
    at[b] = r + D * c;
    tr[b] = c + D * r;
  }
  const uint32_t dl = Left<D, W>::at(tm, pd), dr = Right<D, W>::at(tm, pd);
  const long items = (long)p.n_members * p.n_t;
#pragma unroll 1
  for (long it = (long)blockIdx.x * C::TEAMS + team; it < items; it += (long)gridDim.x * C::TEAMS) {
    const int m = (int)(it / p.n_t), k = (int)(it % p.n_t);
    float x[NV], sum[NV];
    assemble32<D, W>(tm, p, w, m, k, at, x);
    const float sa = unit_scale<D, W>(tm, x, 0);
#pragma unroll
    for (int v = 0; v < NV; ++v) x[v] *= sa;
    store_split<D, W>(tm, pa, x);
    // N = P_k Lambda_{k-1}
    if (p.target == TGT_GATE) {
      const float2* N = reinterpret_cast<const float2*>(w.P) + (size_t)it * D * D;
#pragma unroll
      for (int b = 0; b < H; ++b) {
        const float2 v = N[at[b]];
        x[b] = v.x;
        x[H + b] = v.y;
      }
    } else {
      const int np = p.n_pairs, pan = np * D;
      const float2* ps = reinterpret_cast<const float2*>(w.psi) + ((size_t)m * (p.n_t + 1) + k) * pan;
      const float2* ls = reinterpret_cast<const float2*>(w.lam) + ((size_t)m * (p.n_t + 1) + k) * pan;
#pragma unroll
      for (int b = 0; b < H; ++b) {
        float2 acc = make_float2(0.f, 0.f);
        for (int s = 0; s < np; ++s) {
          const float2 l = ls[s * D + at[b] / D];
          acc = cmac(acc, ps[s * D + at[b] % D], make_float2(l.x, -l.y));
        }
        x[b] = acc.x;
        x[H + b] = acc.y;
      }
    }
    const float sn = unit_scale<D, W>(tm, x, 1);
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      x[v] *= sn;
      sum[v] = x[v];
    }
    store_split<D, W>(tm, pd, x);
    tm.sync();
    // A's fragments, those of the right operand negated
    Left<D, W> al[2][KT];
    Right<D, W> ar[2][KT];
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll
      for (int kt = 0; kt < KT; ++kt) {
        al[s][kt].load(Left<D, W>::at(tm, pa) + 2 * s * G::PLANE + kt * 2 * (D / 8) * 128);
        ar[s][kt].load(Right<D, W>::at(tm, pa) + 2 * s * G::PLANE + kt * 2 * 128);
#pragma unroll
        for (int i = 0; i < 4 * G::NTW; ++i) ar[s][kt].f[i] ^= 0x80008000u;
#pragma unroll
        for (int i = 0; i < 2 * G::NTW; ++i) ar[s][kt].neg[i] ^= 0x80008000u;
      }
    float sig = 1.f;  // the term is sig x
#pragma unroll 1
    for (int n = 1; n < 40; ++n) {
      float acc[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) acc[v] = 0.f;
#pragma unroll
      for (int kt = 0; kt < KT; ++kt) {
        Left<D, W> l[2];
        Right<D, W> r[2];
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          l[s].load(dl + 2 * s * G::PLANE + kt * 2 * (D / 8) * 128);
          r[s].load(dr + 2 * s * G::PLANE + kt * 2 * 128);
        }
        mma_pair<D, W>(acc, al[1][kt], r[0]);
        mma_pair<D, W>(acc, l[1], ar[0][kt]);
        mma_pair<D, W>(acc, al[0][kt], r[1]);
        mma_pair<D, W>(acc, l[0], ar[1][kt]);
        mma_pair<D, W>(acc, al[0][kt], r[0]);
        mma_pair<D, W>(acc, l[0], ar[0][kt]);
      }
      sig *= __fdividef(1.f, sa * (float)(n + 1));  // sa is a power of two
      const float su = unit_scale<D, W>(tm, acc, n & 1);  // (the sync inside: every product has read D)
#pragma unroll
      for (int v = 0; v < NV; ++v) sum[v] = fmaf(sig, acc[v], sum[v]);
      sig /= su;
      if (!(sig >= 7.4505806e-9f)) break;  // 2^-27
#pragma unroll
      for (int v = 0; v < NV; ++v) x[v] = acc[v] * su;
      if constexpr (W == 1) __syncwarp();
      store_split<D, W>(tm, pd, x);
      tm.sync();
    }
    // traces
    const float inv = 1.f / sn;
    for (int j0 = 0; j0 < p.n_c; j0 += C::TRACE) {
      const int nj = min(C::TRACE, p.n_c - j0);
      float keep = 0.f;
#pragma unroll 1
      for (int j = 0; j < nj; ++j) {
        const float2* Cj = p.ctrls_f32 + (size_t)(j0 + j) * D * D;
        float t = 0.f;
#pragma unroll
        for (int b = 0; b < H; ++b) {
          const float2 c = Cj[tr[b]];
          t = p.gen == GEN_HERM ? fmaf(sum[b], c.y, fmaf(sum[H + b], c.x, t)) : fmaf(sum[b], c.x, fmaf(-sum[H + b], c.y, t));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (W > 1 && tm.lane == 0) traces[tm.w * C::TRACE + j] = t;
        if (tm.lane == j) keep = t;
      }
      tm.sync();
      if (tm.w == 0 && tm.lane < nj) {
#pragma unroll
        for (int i = 1; i < W; ++i) keep += traces[i * C::TRACE + tm.lane];
        w.Gm[(size_t)it * p.n_c + j0 + tm.lane] = p.dt[k] * p.m_scale[m] * (double)(keep * inv);
      }
      tm.sync();
    }
  }
}

constexpr size_t kSmemMax = 232448;  // dynamic shared memory of a CTA

// Launches a slice-parallel kernel of configuration C (dimension D): as many
// teams as the shared memory beside the generator's terms holds.
template <class C, int D, class... A>
static cudaError_t launch_slices(void (*kernel)(ProbDev, WorkDev, int, A...), const ProbDev& p, const WorkDev& w,
                                 const LaunchInfo& li, A... more) {
  const int n = p.n_c + 1 + (p.n_ramp ? 1 : 0);
  const size_t consts = Terms<D, C::W>::bytes(n);
  const int fit = (int)((kSmemMax - consts) / C::TEAM_BYTES);
  // fewer teams where every SM still gets its share of the slices: ten slices of
  // one SM wait for each other, and one or two alone set the generator's terms up
  // longer (d = 16, one member of 20 slices, F only: mixed states 73 us with ten
  // teams, 60 with two; df products on the CUDA cores 64.  FP64 72 and 60)
  constexpr long few = D >= 32 ? 1 : D >= 16 ? 2 : 4;
  const long share = ((long)p.n_members * p.n_t + li.num_sms - 1) / li.num_sms;
  int nt = fit < C::TEAMS ? fit : C::TEAMS;
  if (share < nt) nt = (int)(share > few ? share : few < nt ? few : nt);
  const int threads = 32 * C::W * nt;
  const size_t smem = consts + (size_t)nt * C::TEAM_BYTES;
  set_smem_once((const void*)kernel, smem);
  int per_sm = 1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
  if (per_sm < 1) per_sm = 1;
  // Runs long enough to amortise the member's own terms, short enough that
  // every CTA gets several.
  const long items = (long)p.n_members * p.n_t, ctas = (long)li.num_sms * per_sm;
  long rounds = items / (ctas * nt * 4);
  if (rounds < 1) rounds = 1;
  if (rounds > 8) rounds = 8;
  const int run = (int)rounds * nt;
  long grid = (long)p.n_members * ((p.n_t + run - 1) / run);
  if (grid > ctas) grid = ctas;
  kernel<<<(int)grid, threads, smem, li.stream>>>(p, w, run, more...);
  ++*li.launches;
  return cudaGetLastError();
}

// Blocks of the gate chains.  Chains run in two dependent passes of `len`
// products with one of `blocks` between: more blocks than sqrt(2 n_t) only
// lengthen the sum, and more (member, block) chains than the SMs hold (3 of 66 KB
// at D = 32, 8 of 16 KB at D = 16, 24 of 4 KB at D = 8) run as a second wave.
template <int D> static void chain_shape(const ProbDev& p, int num_sms, int* blocks, int* len) {
  const long chains = (long)num_sms * ChainCfg<D>::PER_SM;
  long b = chains / p.n_members;
  long most = 1;
  while (most < ChainCfg<D>::MAX_BLOCKS && (most + 1) * (most + 1) <= 2L * p.n_t) ++most;
  if (b > most) b = most;
  if (b < 1) b = 1;
  *len = (int)((p.n_t + b - 1) / b);
  *blocks = (p.n_t + *len - 1) / *len;
}

template <int D> static cudaError_t do_chain_fwd(const ProbDev& p, const WorkDev& w, const LaunchInfo& li, bool store) {
  using C = ChainCfg<D>;
  int blocks, len;
  chain_shape<D>(p, li.num_sms, &blocks, &len);
  const size_t smem = (size_t)C::FULL_TEAMS * C::FULL_BYTES;
  const int threads = 32 * C::W * C::FULL_TEAMS;
  set_smem_once((const void*)k_fx_chain_fwd<D>, smem);
  const long items = (long)p.n_members * blocks;
  k_fx_chain_fwd<D><<<(int)((items + C::FULL_TEAMS - 1) / C::FULL_TEAMS), threads, smem, li.stream>>>(p, w, blocks, len, store ? 1 : 0);
  const size_t smem2 = (size_t)C::COMBINE * C::FULL_BYTES + (store ? (size_t)(2 * blocks - 1) * Geo<D, C::W>::INTS : 0);
  set_smem_once((const void*)k_fx_chain_combine<D>, smem2);
  k_fx_chain_combine<D><<<p.n_members, 32 * C::W * C::COMBINE, smem2, li.stream>>>(p, w, blocks, len, store ? 1 : 0);
  *li.launches += 2;
  return cudaGetLastError();
}

template <int D> static cudaError_t do_chain_bwd(const ProbDev& p, const WorkDev& w, const LaunchInfo& li) {
  using C = ChainCfg<D>;
  int blocks, len;
  chain_shape<D>(p, li.num_sms, &blocks, &len);
  const size_t smem = (size_t)C::FULL_TEAMS * C::FULL_BYTES;
  set_smem_once((const void*)k_fx_chain_bwd<D>, smem);
  const long items = (long)p.n_members * blocks;
  k_fx_chain_bwd<D><<<(int)((items + C::FULL_TEAMS - 1) / C::FULL_TEAMS), 32 * C::W * C::FULL_TEAMS, smem, li.stream>>>(p, w, blocks, len);
  ++*li.launches;
  return cudaGetLastError();
}

template <int D> static cudaError_t do_grad(const ProbDev& p, const WorkDev& w, const LaunchInfo& li) {
  int blocks, len;
  chain_shape<D>(p, li.num_sms, &blocks, &len);
  const cudaError_t e = launch_slices<SeriesCfg<D>, D>(k_fx_grad<D>, p, w, li, len);
  if (e != cudaSuccess || p.grad_mode != GRAD_EXACT) return e;
  return launch_slices<NormCfg<D>, D>(k_fx_grad_norm<D>, p, w, li, len);
}

template <int D> static cudaError_t do_prefix_df(const ProbDev& p, const WorkDev& w, const LaunchInfo& li, bool store) {
  using C = ChainCfg<D>;
  const size_t smem = (size_t)C::TEAMS * C::TEAM_BYTES;
  set_smem_once((const void*)k_fx_prefix_df<D>, smem);
  const long items = (long)p.n_members * w.pit_blocks;
  k_fx_prefix_df<D><<<(int)((items + C::TEAMS - 1) / C::TEAMS), 32 * C::W * C::TEAMS, smem, li.stream>>>(p, w, store ? 1 : 0);
  ++*li.launches;
  return cudaGetLastError();
}

template <int D> static cudaError_t do_combine_df(const ProbDev& p, const WorkDev& w, const LaunchInfo& li, bool store) {
  using C = ChainCfg<D>;
  set_smem_once((const void*)k_fx_combine_df<D>, C::TEAM_BYTES);
  k_fx_combine_df<D><<<p.n_members, 32 * C::W, C::TEAM_BYTES, li.stream>>>(p, w, store ? 1 : 0);
  ++*li.launches;
  return cudaGetLastError();
}

template <int D> static long prefix_capacity() {
  using C = ChainCfg<D>;
  const size_t smem = (size_t)C::TEAMS * C::TEAM_BYTES;
  set_smem_once((const void*)k_fx_prefix_df<D>, smem);
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_fx_prefix_df<D>, 32 * C::W * C::TEAMS, smem);
  return (long)per_sm * C::TEAMS;
}

template <int D> static cudaError_t do_states(const ProbDev& p, const WorkDev& w, const LaunchInfo& li, bool store) {
  using C = StCfg<D>;
  const int chains = p.n_pairs * (store ? 2 : 1);
  const size_t smem = C::smem(chains);
  auto kernel = p.gen == GEN_HERM ? k_fx_states<D, true> : k_fx_states<D, false>;
  set_smem_once((const void*)kernel, smem);
  kernel<<<p.n_members, 32 * (chains + C::HELPERS), smem, li.stream>>>(p, w, store ? 1 : 0);
  ++*li.launches;
  return cudaGetLastError();
}

template <int D> static cudaError_t do_tf_grad(const ProbDev& p, const WorkDev& w, const LaunchInfo& li) {
  using C = TfCfg<D>;
  const size_t smem = (size_t)C::TEAMS * C::TEAM_BYTES;
  const int threads = 32 * C::W * C::TEAMS;
  set_smem_once((const void*)k_tf_grad<D>, smem);
  int per_sm = 1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_tf_grad<D>, threads, smem);
  const long need = ((long)p.n_members * p.n_t + C::TEAMS - 1) / C::TEAMS, most = (long)li.num_sms * (per_sm < 1 ? 1 : per_sm);
  k_tf_grad<D><<<(int)(need < most ? need : most), threads, smem, li.stream>>>(p, w);
  ++*li.launches;
  return cudaGetLastError();
}

}  // namespace fx

bool fx_applies(const ProbDev& p) {
  const int n = p.n_c + 1 + (p.n_ramp ? 1 : 0);
  return ((p.Dp == 8 || p.Dp == 16) && n <= fx::kMaxTerms) || (p.Dp == 32 && n <= fx::kMaxTerms32);
}

#define PGX_FX_DISPATCH(CALL)                          \
  switch (p.Dp) {                                      \
    case 8: { constexpr int D_ = 8; return CALL; }     \
    case 16: { constexpr int D_ = 16; return CALL; }   \
    case 32: { constexpr int D_ = 32; return CALL; }   \
    default: return cudaErrorInvalidValue;             \
  }
// the mixed path's dimensions
#define PGX_FX_DISPATCH_DF(CALL)                         \
  switch (p.Dp) {                                        \
    case 16: { constexpr int D_ = 16; return CALL; }     \
    case 32: { constexpr int D_ = 32; return CALL; }     \
    default: return cudaErrorInvalidValue;               \
  }

cudaError_t launch_fx_expm(const ProbDev& p, const WorkDev& w, const LaunchInfo& li) {
  PGX_FX_DISPATCH((fx::launch_slices<fx::ExpmCfg<D_>, D_>(fx::k_fx_expm<D_, false>, p, w, li)));
}
cudaError_t launch_fx_expm_df(const ProbDev& p, const WorkDev& w, const LaunchInfo& li) {
  PGX_FX_DISPATCH_DF((fx::launch_slices<fx::ExpmCfg<D_>, D_>(fx::k_fx_expm<D_, true>, p, w, li)));
}
cudaError_t launch_fx_prefix_df(const ProbDev& p, const WorkDev& w, const LaunchInfo& li, bool store) {
  PGX_FX_DISPATCH_DF(fx::do_prefix_df<D_>(p, w, li, store));
}
cudaError_t launch_tf_grad(const ProbDev& p, const WorkDev& w, const LaunchInfo& li) {
  return p.Dp == 16 ? fx::do_tf_grad<16>(p, w, li) : fx::do_tf_grad<32>(p, w, li);
}
cudaError_t launch_fx_states(const ProbDev& p, const WorkDev& w, const LaunchInfo& li, bool store) {
  switch (p.Dp) {
    case 2: return fx::do_states<2>(p, w, li, store);
    case 4: return fx::do_states<4>(p, w, li, store);
    case 8: return fx::do_states<8>(p, w, li, store);
    case 16: return fx::do_states<16>(p, w, li, store);
    case 32: return fx::do_states<32>(p, w, li, store);
    default: return cudaErrorInvalidValue;
  }
}
cudaError_t launch_fx_combine_df(const ProbDev& p, const WorkDev& w, const LaunchInfo& li, bool store) {
  PGX_FX_DISPATCH_DF(fx::do_combine_df<D_>(p, w, li, store));
}
// At D = 32 an SM holds two chains of 57 KB, and is given twice as many: the FP32
// suffixes beside them gain from more blocks than the prefixes lose by queueing,
// and from 153 to 304 members the chains stay cut at all.  Evaluations of 500
// slices (60 from 153 members on) in ms with one, two and three times what it
// holds, in brackets F alone: 16 members 1.57 (0.99), 1.62 (1.08), 1.62 (1.08);
// 64: 5.42 (3.42), 5.27 (3.33), 5.27 (3.34); 128: 10.85 (6.84), 10.69 (6.81),
// 10.71 (6.81); 153: 2.61 (1.94), 1.72 (1.16), 1.72 (1.16); 304: 3.71 (2.64),
// 3.11 (1.99), 3.11 (1.99); 305: 4.46 (3.33) with any.  The same grid on the
// FP32 pipe's df kernels: never faster.
constexpr long kPrefixWaves32 = 2;
long fx_prefix_capacity(int Dp) {
  switch (Dp) {
    case 16: return fx::prefix_capacity<16>();
    case 32: return kPrefixWaves32 * fx::prefix_capacity<32>();
    default: return 0;
  }
}
cudaError_t launch_fx_chain_fwd(const ProbDev& p, const WorkDev& w, const LaunchInfo& li, bool store) {
  PGX_FX_DISPATCH(fx::do_chain_fwd<D_>(p, w, li, store));
}
cudaError_t launch_fx_chain_bwd(const ProbDev& p, const WorkDev& w, const LaunchInfo& li) {
  PGX_FX_DISPATCH(fx::do_chain_bwd<D_>(p, w, li));
}
cudaError_t launch_fx_grad(const ProbDev& p, const WorkDev& w, const LaunchInfo& li) {
  PGX_FX_DISPATCH(fx::do_grad<D_>(p, w, li));
}

}  // namespace pgx
