// FP64-class kernels on block fixed-point tensor-core products (pgx_fx.cuh).
#include "pgx.h"
#include "pgx_fx.cuh"
#include "pgx_stages.cuh"

namespace pgx {
namespace fx {

static __constant__ float c_log2theta[PGX_N_FXDEGREES] = PGX_LOG2_THETA64_EVEN_INIT;
static __constant__ Coef c_coef[PGX_N_INVFACT] = PGX_INVFACT_FX_INIT;

constexpr int kMaxTerms = 24;       // generator terms: drift, controls, ramp
constexpr int kBits = 57;           // absolute error of a slice propagator: 2^-57 per product
constexpr int kBits2 = 2 * kBits + 1;
constexpr int kNever = 1 << 20;     // an exponent no finite entry reaches

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

// A = c sum_j alpha_j K_j, 58 fractional bits in the frame returned; a frame
// above kNever / 2 means a term is not finite.  |b1| <= 2^27, |a0| <= 2^31 and
// sum |a1| <= 2^30 keep 24 terms' mixed products inside 63 bits.
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
  for (int v = 0; v < NV; ++v) main[v] = mid[v] = 0;
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
  for (int v = 0; v < NV; ++v) main[v] += (long long)(int)(mid[v] >> 32);
#pragma unroll
  for (int v = 0; v < NV / 2; ++v) {
    A[v] = p.gen == GEN_HERM ? main[NV / 2 + v] : main[v];
    A[NV / 2 + v] = p.gen == GEN_HERM ? -main[v] : main[NV / 2 + v];
  }
  return EA;
}

// log2 of a bound of ||A||_1 (58 fractional bits in frame EA), D <= 16.
template <int D, int W> __device__ __forceinline__ float log2_norm1(const Tm<D, W>& tm, const long long (&A)[Geo<D, W>::NV], int EA) {
  using G = Geo<D, W>;
  static_assert(G::RT == 1, "a column's rows belong to one warp");
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
  best = __uint_as_float(tm.max(__float_as_uint(best), 1));
  return __log2f(fmaf(best, 1.00001f, 2.f * D)) + (float)(EA - 26) + 1e-5f;
}

// Degree 2 L and squarings s with ||A||_1 / 2^s <= theta_2L that minimise the
// products L + s (squarings last: they double the error).
__device__ __forceinline__ void choose_degree2(float l2, int lane, int& L, int& s) {
  uint32_t key = 0xffffffffu;
  if (lane < PGX_N_FXDEGREES) {
    const int si = (int)fmaxf(ceilf(l2 - c_log2theta[lane]), 0.f);
    if (si < 64) key = (uint32_t)((2 + lane + si) << 16 | si << 8 | lane);
  }
  key = __reduce_min_sync(0xffffffffu, key);
  s = (int)((key >> 8) & 0xff);
  L = 2 + (int)(key & 0xff);
}

template <int D> struct ExpmCfg {
  static constexpr int W = D >= 16 ? 2 : 1;             // warps of a slice
  static constexpr int TEAMS = D >= 16 ? 10 : 12;       // slices in flight per CTA, at most
  static constexpr int TEAM_BYTES = 2 * Geo<D, W>::PLANES + Geo<D, W>::INTS + 64;  // planes of X, of Y; B; maxima
};

// U_mk = exp(A_mk), one team per slice: T_2L(A / 2^s) in the q = 2
// Paterson-Stockmeyer form (X = B^2, Horner in X), then s squarings.  A CTA
// walks runs of `run` slices of one member.
//
// Bound: instruction issue (digits of each factor, joining the levels,
// rescaling), then the tensor pipe (about 64 digit pairs of 16 SM cycles at
// D = 16).  A slice's planes and integers take 18 KB of shared memory, so an SM
// holds ten; two warps share one, each with half the columns.
template <int D>
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
                    reinterpret_cast<uint32_t*>(mine + 2 * G::PLANES + G::INTS)};
  longlong2* Bs = tm.mine(reinterpret_cast<longlong2*>(mine + 2 * G::PLANES));
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
      const float l2 = log2_norm1<D, W>(tm, r, EA);
      int L, s;
      choose_degree2(l2, tm.lane, L, s);
      double2* out = w.U + ((size_t)m * p.n_t + k) * D * D;
      int ex;  // U = r 2^ex
      if (EA > kNever / 2 || s > 60) {
        store_nan<D, W>(tm, out);
        tm.sync();  // the maxima are read
        continue;
      }
      // bounds: |X| <= nu^2 (nu = the scaled norm), and |Y_i| <= c_2i e^nu, so
      // Y_i keeps the fixed frame c_2i.exp + g
      const float nu2 = l2 - (float)s;
      const int lx = min(0, 2 * (int)ceilf(nu2));
      const int g = nu2 <= -1.33f ? 1 : 3;  // e^nu <= 0.75 2^g, nu <= 0.397 or 1.51
      const int EB = normalize<D, W>(tm, r, EA - 2 - s);
      int EX = 0, EY = EB, n = kSlices, F = 60;
      uint32_t pa = py;
      // step 0: X = B B; L - 1 Horner steps Y <- X Y + c_{2i+1} B + c_2i I,
      // whose error later meets X^i; s squarings.  One product in the loop
      // body keeps the kernel inside the instruction cache.
#pragma unroll 1
      for (int st = 0; st < L + s; ++st) {
        const int i = L - 1 - st;
        if (st == 0) n = levels(kBits2, 2 * EB);
        else if (st < L) n = levels(kBits2, EX + EY + i * lx);
        else n = levels(kBits2, 2 * EY);
        tm.sync();
        if (st == 0) {
          long long x6[NV];
#pragma unroll
          for (int v = 0; v < NV; ++v) x6[v] = r[v] << 6;
          put_ints<NV>(Bs, x6);
        }
        store_planes<D, W>(tm, py, r, n);
        tm.sync();
        mul<D, W>(tm, pa, py, n, r);
        if (st < L) {
          const int fr = c_coef[2 * i].exp + g;
          if (st == 0) {
            // Y = c_2L X + c_{2L-1} B + c_{2L-2} I
            EX = normalize<D, W>(tm, r, 2 * EB);
            store_planes<D, W>(tm, px, r, kSlices);
            pa = px;
            F = kFrac;
            const Scaled sx(c_coef[2 * L], EX, fr, F);
#pragma unroll
            for (int v = 0; v < NV; ++v) r[v] = sx(r[v] << 6, 0);
          } else {
            F = i > 0 ? kFrac : 60;
            to_frame<NV>(r, EX + EY, fr, F);
          }
          add_scaled<NV>(r, Bs, Scaled(c_coef[2 * i + 1], EB, fr, F));
          add_diag<D, W>(tm, r, c_coef[2 * i], fr, F);
          EY = fr;
          if (i == 0) {
            ex = fr - 60;
            if (s > 0) EY = normalize<D, W>(tm, r, fr - 4);
            pa = py;
          }
        } else {
          ex = 2 * EY - kFrac;
          if (st + 1 < L + s) EY = normalize<D, W>(tm, r, 2 * EY);
        }
      }
      store_mat<D, W>(tm, out, r, ex);
    }
  }
}

constexpr size_t kSmemMax = 232448;  // dynamic shared memory of a CTA

template <int D> static cudaError_t do_expm(const ProbDev& p, const WorkDev& w, const LaunchInfo& li) {
  using C = ExpmCfg<D>;
  const int n = p.n_c + 1 + (p.n_ramp ? 1 : 0);
  const size_t consts = Terms<D, C::W>::bytes(n);
  const int fit = (int)((kSmemMax - consts) / C::TEAM_BYTES);
  const int nt = fit < C::TEAMS ? fit : C::TEAMS, threads = 32 * C::W * nt;
  const size_t smem = consts + (size_t)nt * C::TEAM_BYTES;
  set_smem_once((const void*)k_fx_expm<D>, smem);
  int per_sm = 1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_fx_expm<D>, threads, smem);
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
  k_fx_expm<D><<<(int)grid, threads, smem, li.stream>>>(p, w, run);
  ++*li.launches;
  return cudaGetLastError();
}

}  // namespace fx

bool fx_expm_applies(const ProbDev& p) {
  return (p.Dp == 8 || p.Dp == 16) && p.n_c + 1 + (p.n_ramp ? 1 : 0) <= fx::kMaxTerms;
}
cudaError_t launch_fx_expm(const ProbDev& p, const WorkDev& w, const LaunchInfo& li) {
  return p.Dp == 8 ? fx::do_expm<8>(p, w, li) : fx::do_expm<16>(p, w, li);
}

}  // namespace pgx
