// FP64 gate chains of small systems (padded dimension 2 or 4), parallel in
// time over blocks of `len` slices:
//   k_small_chain_fwd      per (member, block): R_k = U_{k-1} ... U_{k0} into
//                          the P slots (R_{k0} = I is implied) and the block
//                          product into the block's first P slot (F only: U slot)
//   k_small_chain_combine  per member: T_b = the product before block b, z, f,
//                          kappa; Lambda_b = T' (product after block b); W_b =
//                          kappa T_b Lambda_b into the block's first P slot
//   k_small_chain_bwd      per (member, block): V = W_b U_{k1-1} ... , and
//                          M_k = R_k V, which is P_k Lambda_k (or P_k Lambda_{k-1}
//                          in the GRAPE form), into the P slots
// D D lanes hold a matrix, one entry each, and a product takes its row and
// column from them by shuffles.
//
// Bound: a warp's FP64 FMA takes 16 cycles of an SM's pipe, so a D = 4 product
// of 16 of them costs about 300 cycles however many lanes are in use, and a
// serial chain is one such latency per slice (with the shared-memory round
// trips of a team 0.6 us, and 1.5 us for the two products and loads of a
// backward step).  Blocks divide it by their number until the SMs are full:
// D = 3, 200 slices of 8 members, forward and backward 124 + 295 us as serial
// chains, 33 + 16 us in blocks.
#pragma once
#include "pgx_stages.cuh"

namespace pgx {
namespace small {

template <int D> struct Geo {
  static constexpr int L = D * D;               // lanes of a matrix
  static constexpr int PER_WARP = 32 / L;       // matrices of a warp
  static constexpr int MAX_BLOCKS = 64;         // T_b and Lambda_b of a member in shared memory
  static constexpr int COMBINE_WARPS = 4;
};

// This lane's matrix of its warp and its entry (row i, column j) there.
template <int D> struct Lane {
  int g, e, i, j, first;
  __device__ __forceinline__ Lane()
      : g((int)(threadIdx.x & 31) / Geo<D>::L), e((int)threadIdx.x % Geo<D>::L), i(e % D), j(e / D), first(g * Geo<D>::L) {}
  __device__ __forceinline__ double2 one() const { return make_double2(i == j ? 1.0 : 0.0, 0.0); }
};
__device__ __forceinline__ double2 shfl2(double2 v, int src) {
  return make_double2(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}
// Entry of A B from the lanes' entries (the whole warp together).
template <int D> __device__ __forceinline__ double2 mul(const Lane<D>& l, double2 a, double2 b) {
  double2 s = make_double2(0.0, 0.0);
#pragma unroll
  for (int k = 0; k < D; ++k) s = cmac(s, shfl2(a, l.first + l.i + D * k), shfl2(b, l.first + k + D * l.j));
  return s;
}

template <int D>
__global__ void __launch_bounds__(32) k_small_chain_fwd(ProbDev p, WorkDev w, int blocks, int len, int store) {
  const Lane<D> l;
  const long item = (long)blockIdx.x * Geo<D>::PER_WARP + l.g;
  const bool valid = item < (long)p.n_members * blocks;
  const int m = valid ? (int)(item / blocks) : 0, k0 = (int)(item % blocks) * len;
  const int n = valid ? min(p.n_t - k0, len) : 0;
  const size_t at = ((size_t)m * p.n_t + k0) * Geo<D>::L + l.e;
  const double2* U = w.U + at;
  const double2 z = make_double2(0.0, 0.0);
  double2 r = 0 < n ? U[0] : z;
  double2 x1 = 1 < n ? U[Geo<D>::L] : z, x2 = 2 < n ? U[2 * Geo<D>::L] : z;
#pragma unroll 1
  for (int s = 1; s < len; ++s) {
    const double2 u = x1;
    x1 = x2;
    if (s + 2 < n) x2 = U[(size_t)(s + 2) * Geo<D>::L];  // two products ahead
    if (store && s < n) w.P[at + (size_t)s * Geo<D>::L] = r;
    const double2 y = mul<D>(l, u, r);
    if (s < n) r = y;
  }
  if (valid) (store ? w.P : w.U)[at] = r;
}

template <int D>
__global__ void __launch_bounds__(32) k_small_chain_bwd(ProbDev p, WorkDev w, int blocks, int len) {
  const Lane<D> l;
  const long item = (long)blockIdx.x * Geo<D>::PER_WARP + l.g;
  const bool valid = item < (long)p.n_members * blocks;
  const int m = valid ? (int)(item / blocks) : 0, k0 = (int)(item % blocks) * len;
  const int n = valid ? min(p.n_t - k0, len) : 0;
  const bool grape = p.grad_mode == GRAD_REF_GRAPE;  // the costate includes the slice's own U_k
  const size_t at = ((size_t)m * p.n_t + k0) * Geo<D>::L + l.e;
  const double2* U = w.U + at;
  double2* P = w.P + at;
  const double2 z = make_double2(0.0, 0.0);
  double2 v = valid ? P[0] : z;
  auto u_of = [&](int s) { return s >= 0 ? U[(size_t)s * Geo<D>::L] : z; };
  auto r_of = [&](int s) { return s > 0 ? P[(size_t)s * Geo<D>::L] : l.one(); };
  double2 u1 = u_of(n - 1), u2 = u_of(n - 2), r1 = r_of(n - 1), r2 = r_of(n - 2);
#pragma unroll 1
  for (int d = 1; d <= len; ++d) {
    const int s = n - d;
    const double2 u = u1, r = r1;
    u1 = u2;
    r1 = r2;
    u2 = u_of(s - 2);
    r2 = r_of(s - 2);
    const double2 vu = mul<D>(l, v, u);
    const double2 M = mul<D>(l, r, grape ? vu : v);
    v = vu;
    if (s >= 0) P[(size_t)s * Geo<D>::L] = M;
  }
}

template <int D>
__global__ void __launch_bounds__(32 * Geo<D>::COMBINE_WARPS)
k_small_chain_combine(ProbDev p, WorkDev w, int blocks, int len, int want_grad) {
  using G = Geo<D>;
  __shared__ double2 s_T[G::MAX_BLOCKS][G::L], s_L[G::MAX_BLOCKS][G::L];
  __shared__ double2 s_kap;
  const Lane<D> l;
  const int warp = threadIdx.x >> 5, m = blockIdx.x;
  const size_t base = (size_t)m * p.n_t * G::L + l.e, step = (size_t)len * G::L;
  const double2* tot = (want_grad ? w.P : w.U) + base;  // where k_small_chain_fwd left the block products
  const double2 z0 = make_double2(0.0, 0.0);
  if (warp == 0) {  // T_0 = I, T_{b+1} = Tot_b T_b (every group of the warp alike)
    double2 r = tot[0];
    double2 x1 = 1 < blocks ? tot[step] : z0, x2 = 2 < blocks ? tot[2 * step] : z0;
    if (l.g == 0) s_T[0][l.e] = l.one();
#pragma unroll 1
    for (int b = 1; b < blocks; ++b) {
      if (l.g == 0) s_T[b][l.e] = r;
      const double2 x = x1;
      x1 = x2;
      if (b + 2 < blocks) x2 = tot[(size_t)(b + 2) * step];
      r = mul<D>(l, x, r);
    }
    if (l.g == 0) w.Utot[(size_t)m * G::L + l.e] = r;
    double2 z = cmac_cj(z0, p.target_op[l.e], r);
#pragma unroll
    for (int o = G::L / 2; o > 0; o >>= 1) {
      z.x += __shfl_xor_sync(0xffffffffu, z.x, o);
      z.y += __shfl_xor_sync(0xffffffffu, z.y, o);
    }
    if (threadIdx.x == 0) {
      z.x /= p.D;
      z.y /= p.D;
      double f;
      double2 kap;
      fid_kappa(z, p.fid, p.grad_mode, f, kap);
      const double sc = p.m_weight[m] / p.D;
      kap = make_double2(kap.x * sc, kap.y * sc);
      w.z[m] = z;
      w.kap[m] = kap;
      w.Fm[m] = f;
      s_kap = kap;
    }
  } else if (warp == 1 && want_grad) {  // Lambda_B = T', Lambda_{b-1} = Lambda_b Tot_b
    const double2 t = p.target_op[l.j + D * l.i];
    double2 r = make_double2(t.x, -t.y);
    auto tot_of = [&](int b) { return b > 0 ? tot[(size_t)b * step] : z0; };
    double2 x1 = tot_of(blocks - 1), x2 = tot_of(blocks - 2);
#pragma unroll 1
    for (int b = blocks - 1; b >= 0; --b) {
      if (l.g == 0) s_L[b][l.e] = r;
      const double2 x = x1;
      x1 = x2;
      x2 = tot_of(b - 2);
      if (b > 0) r = mul<D>(l, r, x);
    }
  }
  if (!want_grad) return;
  __syncthreads();
  const double2 kap = s_kap;
  constexpr int STRIDE = G::COMBINE_WARPS * G::PER_WARP;
#pragma unroll 1
  for (int b0 = 0; b0 < blocks; b0 += STRIDE) {  // W_b = kappa T_b Lambda_b
    const int b = b0 + warp * G::PER_WARP + l.g, c = min(b, blocks - 1);
    const double2 x = cmul(kap, mul<D>(l, s_T[c][l.e], s_L[c][l.e]));
    if (b < blocks) w.P[base + (size_t)b * step] = x;
  }
}

// Blocks of a member's chain: a chain of b blocks takes about 3 n_t / b steps
// inside them and b across, so b b <= 3 n_t; and no more (member, block) pairs
// than four warps per SM hold, which keep its FP64 pipe busy.
template <int D> inline void chain_shape(const ProbDev& p, int num_sms, int* blocks, int* len) {
  long b = (long)num_sms * 4 * Geo<D>::PER_WARP / p.n_members, most = 1;
  while (most < Geo<D>::MAX_BLOCKS && (most + 1) * (most + 1) <= 3L * p.n_t) ++most;
  if (b > most) b = most;
  if (b < 1) b = 1;
  *len = (int)((p.n_t + b - 1) / b);
  *blocks = (p.n_t + *len - 1) / *len;
}

template <int D> inline cudaError_t launch_fwd(const ProbDev& p, const WorkDev& w, const LaunchInfo& li, bool store) {
  int blocks, len;
  chain_shape<D>(p, li.num_sms, &blocks, &len);
  const long items = (long)p.n_members * blocks;
  k_small_chain_fwd<D><<<(int)((items + Geo<D>::PER_WARP - 1) / Geo<D>::PER_WARP), 32, 0, li.stream>>>(p, w, blocks, len, store ? 1 : 0);
  k_small_chain_combine<D><<<p.n_members, 32 * Geo<D>::COMBINE_WARPS, 0, li.stream>>>(p, w, blocks, len, store ? 1 : 0);
  *li.launches += 2;
  return cudaGetLastError();
}
template <int D> inline cudaError_t launch_bwd(const ProbDev& p, const WorkDev& w, const LaunchInfo& li) {
  int blocks, len;
  chain_shape<D>(p, li.num_sms, &blocks, &len);
  const long items = (long)p.n_members * blocks;
  k_small_chain_bwd<D><<<(int)((items + Geo<D>::PER_WARP - 1) / Geo<D>::PER_WARP), 32, 0, li.stream>>>(p, w, blocks, len);
  ++*li.launches;
  return cudaGetLastError();
}

}  // namespace small
}  // namespace pgx
