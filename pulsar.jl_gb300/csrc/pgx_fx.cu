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
// ..., R_m}, as 64-bit integers K = (b1 2^32 + b0) 2^(E - 58), b0 balanced, in
// the lanes' own order: 3 integer multiply-adds per real value and term in
// place of one FP64 FMA, which is 18 times slower.
template <int D> struct Terms {
  int4* k;        // [n][NV / 2][32] (b0, b1, b0', b1')
  int* e;         // [n] exponents; kNever: not finite
  int n;
  __device__ __forceinline__ static size_t bytes(int n) { return (size_t)n * Geo<D>::INTS + (kMaxTerms + 8) * sizeof(int); }
};

// One warp converts a matrix (doubles in the lanes' order) into term j.
template <int D>
__device__ __forceinline__ void put_term(const Terms<D>& T, int j, int lane, const double (&x)[Geo<D>::NV]) {
  constexpr int NV = Geo<D>::NV;
  const int EX = max_exponent<NV>(x);
  int4* dst = T.k + (size_t)j * (NV / 2) * 32;
#pragma unroll
  for (int v = 0; v < NV; v += 2) {
    const long long a = from_double(x[v], EX, 4), b = from_double(x[v + 1], EX, 4);
    dst[(v / 2) * 32 + lane] = make_int4((int)a, (int)((a + 0x80000000ll) >> 32), (int)b, (int)((b + 0x80000000ll) >> 32));
  }
  if (lane == 0) T.e[j] = EX == 0x7ff ? kNever : EX - 1021;
}

template <int D>
__device__ __forceinline__ void load_mat(const double2* A, int lane, double (&x)[Geo<D>::NV]) {
  using G = Geo<D>;
#pragma unroll
  for (int q = 0; q < G::NQ; ++q)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const double2 a = A[G::row(lane, q) + D * G::col(lane, q, h)];
      x[2 * q + h] = a.x;
      x[G::NV / 2 + 2 * q + h] = a.y;
    }
}

// Member m's own terms: drift + offset, and its ramp operator.
template <int D>
__device__ __forceinline__ void put_member_terms(const Terms<D>& T, const ProbDev& p, int m, int lane) {
  constexpr int NV = Geo<D>::NV;
  double x[NV], o[NV];
  load_mat<D>(p.drifts + (size_t)p.m_drift[m] * D * D, lane, x);
  load_mat<D>(p.offset_op, lane, o);
  const double off = p.m_offset[m];
#pragma unroll
  for (int v = 0; v < NV; ++v) x[v] = fma(off, o[v], x[v]);
  put_term<D>(T, 0, lane, x);
  if (p.n_ramp) {
    const int ro = p.m_ramp[m];
    if (ro >= 0) load_mat<D>(p.ramp_ops + (size_t)ro * D * D, lane, x);
#pragma unroll
    for (int v = 0; v < NV; ++v)
      if (ro < 0) x[v] = 0.0;
    put_term<D>(T, p.n_c + 1, lane, x);
  }
}

// A = c sum_j alpha_j K_j, 60 fractional bits in the frame returned; a frame
// above kNever / 2 means a term is not finite.
template <int D>
__device__ __forceinline__ int assemble(const Terms<D>& T, const ProbDev& p, const double* u, int m, int k, int lane,
                                        long long (&A)[Geo<D>::NV]) {
  constexpr int NV = Geo<D>::NV;
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
  // |alpha_j| 2^(E_j - EA) <= 1 / n in 61 fractional bits
  const int s = te == -kNever ? -64 : te - EA + 8;
  unsigned long long am = ((unsigned long long)((hi & 0xfffffu) | 0x100000u) << 32) | (uint32_t)__double2loint(al);
  am = s >= 0 ? am << min(s, 8) : shr64(am, min(-s, 64));
  const long long sg = (long long)(int)hi >> 31;
  const long long a = ((long long)am ^ sg) - sg;
  const int my0 = (int)a, my1 = (int)((a + 0x80000000ll) >> 32);
  long long main[NV], mid[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) main[v] = mid[v] = 0;
  const int4* kp = T.k + lane;
#pragma unroll 1
  for (int j = 0; j < T.n; ++j) {
    const int a0 = __shfl_sync(0xffffffffu, my0, j), a1 = __shfl_sync(0xffffffffu, my1, j);
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
    kp += (NV / 2) * 32;
  }
  // times c: -i for a Hermitian generator, 1 for a Liouvillian
#pragma unroll
  for (int v = 0; v < NV; ++v) main[v] = (main[v] << 5) + (mid[v] >> 27);
#pragma unroll
  for (int v = 0; v < NV / 2; ++v) {
    A[v] = p.gen == GEN_HERM ? main[NV / 2 + v] : main[v];
    A[NV / 2 + v] = p.gen == GEN_HERM ? -main[v] : main[NV / 2 + v];
  }
  return EA;
}

// log2 of a bound of ||A||_1 (60 fractional bits in frame EA).
template <int D> __device__ __forceinline__ float log2_norm1(const long long (&A)[Geo<D>::NV], int EA) {
  constexpr int NQ = Geo<D>::NQ, NV = Geo<D>::NV;
  float best = 0.f;
#pragma unroll
  for (int cb = 0; cb < (NQ + 1) / 2; ++cb)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float s = 0.f;
#pragma unroll
      for (int rb = 0; rb < (NQ + 1) / 2; ++rb) {
        const int v = 2 * (2 * cb + rb) + h;
        const float x = (float)(int)(A[v] >> 32), y = (float)(int)(A[NV / 2 + v] >> 32);
        s += __fsqrt_rn(fmaf(x, x, y * y));
      }
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      best = fmaxf(best, s);
    }
  best = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(best)));
  return __log2f(fmaf(best, 1.00001f, 2.f * D)) + (float)(EA - 28) + 1e-5f;
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
  static constexpr int WARP_BYTES = 2 * Geo<D>::PLANES + Geo<D>::INTS;  // planes of X, of Y; B
  static constexpr int MAX_WARPS = D >= 16 ? 10 : 12;
};

// U_mk = exp(A_mk), one warp per slice: T_2L(A / 2^s) in the q = 2
// Paterson-Stockmeyer form (X = B^2, Horner in X), then s squarings.  A CTA
// walks runs of `run` slices of one member.
//
// Bound: the tensor pipe (about 64 digit pairs of 16 SM cycles at D = 16) and,
// as much again, the integer work around it: digits of each factor, joining
// the levels, rescaling.  A unit's planes and integers take 18 KB of shared
// memory, so an SM holds ten warps; the FP64 form kept the FP64 pipe busy for
// 41,000 cycles a slice.
template <int D>
__global__ void __launch_bounds__(32 * ExpmCfg<D>::MAX_WARPS) k_fx_expm(ProbDev p, WorkDev w, int run) {
  using G = Geo<D>;
  constexpr int NV = G::NV;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  Terms<D> T;
  T.n = p.n_c + 1 + (p.n_ramp ? 1 : 0);
  T.k = reinterpret_cast<int4*>(smem_raw);
  T.e = reinterpret_cast<int*>(smem_raw + (size_t)T.n * G::INTS);
  unsigned char* mine = smem_raw + Terms<D>::bytes(T.n) + (size_t)wid * ExpmCfg<D>::WARP_BYTES;
  const uint32_t px = smem_u32(mine), py = px + G::PLANES;
  longlong2* Bs = reinterpret_cast<longlong2*>(mine + 2 * G::PLANES);
  for (int j = wid; j < p.n_c; j += nw) {
    double x[NV];
    load_mat<D>(p.ctrls + (size_t)j * D * D, lane, x);
    put_term<D>(T, j + 1, lane, x);
  }
  const int runs = (p.n_t + run - 1) / run;
  int cur = -1;
  for (long c = blockIdx.x; c < (long)p.n_members * runs; c += gridDim.x) {
    const int m = (int)(c / runs), k0 = (int)(c % runs) * run;
    if (m != cur) {
      __syncthreads();
      if (wid == 0) put_member_terms<D>(T, p, m, lane);
      __syncthreads();
      cur = m;
    }
    const int k1 = min(p.n_t, k0 + run);
#pragma unroll 1
    for (int k = k0 + wid; k < k1; k += nw) {
      long long r[NV];
      const int EA = assemble<D>(T, p, w.u, m, k, lane, r);
      const float l2 = log2_norm1<D>(r, EA);
      int L, s;
      choose_degree2(l2, lane, L, s);
      double2* out = w.U + ((size_t)m * p.n_t + k) * D * D;
      int ex;  // U = r 2^ex
      if (EA > kNever / 2 || s > 60) {
#pragma unroll
        for (int q = 0; q < G::NQ; ++q)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const double nan = __longlong_as_double(0x7ff8000000000000ll);
            out[G::row(lane, q) + D * G::col(lane, q, h)] = make_double2(nan, nan);
          }
        continue;
      }
      const int lx = min(0, 2 * (int)ceilf(l2 - (float)s));  // log2 of a bound of ||X||
      const int EB = normalize<NV>(r, EA - 4 - s);
      __syncwarp();
      put_ints<NV>(Bs, lane, r);
      store_planes<D>(lane, py, r, kSlices);
      __syncwarp();
      mul<D>(lane, py, py, levels(kBits2, 2 * EB), r);
      const int EX = normalize<NV>(r, 2 * EB);
      store_planes<D>(lane, px, r, kSlices);
      // Y = c_2L X + c_{2L-1} B + c_{2L-2} I
      int fr = max(max(EX + c_coef[2 * L].exp, EB + c_coef[2 * L - 1].exp), c_coef[2 * L - 2].exp) + 1;
      const Scaled sx(c_coef[2 * L], EX, fr);
#pragma unroll
      for (int v = 0; v < NV; ++v) r[v] = sx(r[v]);
      add_scaled<NV>(r, Bs, lane, EB, c_coef[2 * L - 1], fr);
      add_diag<D>(r, lane, c_coef[2 * L - 2], fr);
      int EY = normalize<NV>(r, fr - 4);
#pragma unroll 1
      for (int i = L - 2; i >= 0; --i) {  // Y <- X Y + c_{2i+1} B + c_2i I, whose error later meets X^i
        const int n = levels(kBits2, EX + EY + i * lx);
        __syncwarp();
        store_planes<D>(lane, py, r, n);
        __syncwarp();
        mul<D>(lane, px, py, n, r);
        fr = max(max(EX + EY + 5, EB + c_coef[2 * i + 1].exp), c_coef[2 * i].exp) + 1;
        to_frame<NV>(r, EX + EY, fr);
        add_scaled<NV>(r, Bs, lane, EB, c_coef[2 * i + 1], fr);
        add_diag<D>(r, lane, c_coef[2 * i], fr);
        if (i > 0 || s > 0) EY = normalize<NV>(r, fr - 4);
      }
      ex = fr - 60;
#pragma unroll 1
      for (int q = 0; q < s; ++q) {
        __syncwarp();
        store_planes<D>(lane, py, r, kSlices);
        __syncwarp();
        mul<D>(lane, py, py, levels(kBits2, 2 * EY), r);
        ex = 2 * EY - kFrac;
        if (q + 1 < s) EY = normalize<NV>(r, 2 * EY);
      }
#pragma unroll
      for (int q = 0; q < G::NQ; ++q)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          out[G::row(lane, q) + D * G::col(lane, q, h)] =
              make_double2(to_double(r[2 * q + h], ex), to_double(r[NV / 2 + 2 * q + h], ex));
    }
  }
}

constexpr size_t kSmemMax = 232448;  // dynamic shared memory of a CTA

template <int D> static cudaError_t do_expm(const ProbDev& p, const WorkDev& w, const LaunchInfo& li) {
  const int n = p.n_c + 1 + (p.n_ramp ? 1 : 0);
  const size_t consts = (size_t)n * Geo<D>::INTS + (kMaxTerms + 8) * sizeof(int);
  const int fit = (int)((kSmemMax - consts) / ExpmCfg<D>::WARP_BYTES);
  const int nw = fit < ExpmCfg<D>::MAX_WARPS ? fit : ExpmCfg<D>::MAX_WARPS;
  const size_t smem = consts + (size_t)nw * ExpmCfg<D>::WARP_BYTES;
  set_smem_once((const void*)k_fx_expm<D>, smem);
  int per_sm = 1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_fx_expm<D>, 32 * nw, smem);
  if (per_sm < 1) per_sm = 1;
  // Runs long enough to amortise the member's own terms, short enough that
  // every CTA gets several.
  const long items = (long)p.n_members * p.n_t, ctas = (long)li.num_sms * per_sm;
  long rounds = items / (ctas * nw * 4);
  if (rounds < 1) rounds = 1;
  if (rounds > 8) rounds = 8;
  const int run = (int)rounds * nw;
  long grid = (long)p.n_members * ((p.n_t + run - 1) / run);
  if (grid > ctas) grid = ctas;
  k_fx_expm<D><<<(int)grid, 32 * nw, smem, li.stream>>>(p, w, run);
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
