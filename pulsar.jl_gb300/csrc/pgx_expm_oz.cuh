// The D = 64 df expm with every product on the tensor cores (the sliced bf16
// engine of pgx_oz.cuh, levels 0..6).
//
// The scheme is the CUDA-core kernel's: A_k = c dt_k (...) in df, the degree
// m = q L, block size q and squarings s from the FP32 1-norm and the df theta
// table, B = A / 2^s, the powers B^2 .. B^q, the Paterson-Stockmeyer Horner
// steps Y <- Y B^q + C_i (Y and B^q are polynomials in B and commute), then s
// squarings.  Every product is a full one (no triangular or half-column
// forms: the tensor-core product costs the same either way).
//
// What bounds it: the workers' instructions (slicing, level sums, Horner
// blocks) and the latencies between a product's phases; the MMAs take about a
// fifth of the time.  Measured on the three-qubit Lindblad gate (16,000
// generators of 1-norm 0.13, four products each), prologue and kernel: 10.0 ms
// with 256 workers, 26 slice pairs in every product, rintf slicing and one
// thread issuing from a divergent branch; 6.5 ms now.
//
// One CTA per SM: 512 worker threads and one issuing warp.
//   - Worker (TMEM lane L, column quarter) owns entries (L mod 64, c0 ..
//     c0+15) of the real (L < 64) or imaginary part of every matrix: exactly
//     the values it stages into both operands of a sliced product and the
//     values it reads back from the accumulators.  So a product's result feeds
//     the next product from registers.  (256 workers of 32 values leave two
//     warps per SM sub-partition to hide each other's latencies: 9.6 against
//     8.1 ms, all else equal.)
//   - The workers cut the left factor's slices into two alternating buffers;
//     after each slice every warp arrives on the buffer's "full" barrier.  The
//     issuing warp waits there, issues the slice's pairs and commits them to
//     the buffer's "empty" barrier, which the workers wait on before they
//     reuse the buffer.  The workers never wait for the issue itself, so the
//     Horner block of a step is formed, in registers, while its MMAs run.
//   - A product takes as many levels (4 to 7, and as many slices, at most 6)
//     as its entries' share of exp(A) needs: levels_of.
//   - A prologue kernel assembles every unit's generator, takes its 1-norm
//     and degree, and leaves B = A / 2^s in the unit's U slot.  B arrives in
//     shared memory by TMA bulk copies while the previous unit ends.
//   - The slab (the per-CTA global workspace of the CUDA-core kernel) keeps
//     B^2 and B^3 as every worker's own values, thread-major, for the Horner
//     blocks C_i = sum_j c_{qi+j} B^j: each worker reads back only what it
//     wrote.
#pragma once
#include "pgx_oz.cuh"

namespace pgx {
namespace oz {

constexpr int kExpmLevels = 7;
constexpr int kExpmBits = 54;
constexpr int kWorkers = 512;
constexpr int kCols = 8192 / kWorkers;  // values of a matrix that one worker holds
constexpr int kExpmThreads = kWorkers + 32;
constexpr uint32_t kCiBytes = 8192u * 8u;  // kCols df values per worker
constexpr size_t kExpmSmem = (size_t)kSlices * kBSlice + 2 * kASlice + kCiBytes + tc::kSmemAlign;

// A worker's place: TMEM lane (row of the stacked [re; im] matrix) and its
// columns c0 .. c0 + kCols - 1.
__device__ __forceinline__ Lane worker_lane() {
  Lane l = tc::lane_of();
  l.c0 = kCols * (int)(threadIdx.x >> 7);
  return l;
}

// Barrier 1 of the workers (the issuing warp never joins it).
__device__ __forceinline__ void wsync() { asm volatile("bar.sync 1, %0;" ::"n"(kWorkers) : "memory"); }
// The same, returning whether any worker's pred was true.
__device__ __forceinline__ bool wsync_or(bool pred) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred pi, po;\n\tsetp.ne.u32 pi, %1, 0;\n\t"
      "bar.red.or.pred po, 1, %2, pi;\n\tselp.u32 %0, 1, 0, po;\n\t}"
      : "=r"(r)
      : "r"((uint32_t)pred), "n"(kWorkers)
      : "memory");
  return r != 0;
}
__device__ __forceinline__ void mbar_arrive(uint32_t mbar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(mbar) : "memory");
}
__device__ __forceinline__ void mbar_init_n(uint32_t mbar, int n) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mbar), "r"(n) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

struct Engine {
  uint8_t* bsl;       // kSlices right-operand slices
  uint8_t* abuf;      // two left-operand slice buffers
  float2* ci;         // 64 KB: the expm's B (workers' own values), the chains' next left factor
  float* red;         // [2][kWorkers / 32] block-maximum scratch, used alternately
  volatile int* cmd;  // [2] the slice behind each "full" phase: index | levels << 8 (-1: stop)
  uint32_t tmem;
  uint32_t bar;       // barriers at bar + 8 b: 0, 1 "full" of the two buffers, 2, 3 "empty"
  uint32_t eph;       // bit b: parity of buffer b's next "empty" phase to wait for
  uint32_t pend;      // byte b: slices committed on buffer b and not yet waited for
  int par;
  int seq;  // slices handed to the issuer so far (their buffer alternates)
  bool abort;
};

// Exponent of the scale of a matrix given by every worker's 32 leading parts.
__device__ __forceinline__ int block_exp(Engine& g, const float (&h)[kCols]) {
  float mx = 0.f;
#pragma unroll
  for (int c = 0; c < kCols; ++c) mx = fmaxf(mx, fabsf(h[c]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  float* r = g.red + kWorkers / 32 * g.par;  // alternate: a slow reader of the previous call is past a barrier
  g.par ^= 1;
  if ((threadIdx.x & 31) == 0) r[threadIdx.x >> 5] = mx;
  wsync();
  mx = 0.f;
#pragma unroll
  for (int w = 0; w < kWorkers / 32; ++w) mx = fmaxf(mx, r[w]);
  return scale_exp(mx);
}

// Stages the six right-operand slices of the matrix whose values this worker
// holds in (h, lo) (unchanged); returns its scale exponent.  No MMA may be
// reading the slices (every product waits for its MMAs before it returns).
__device__ __forceinline__ int stage_right(Engine& g, const Lane& l, const float (&h)[kCols], const float (&lo)[kCols]) {
  const int e = block_exp(g, h);
  const float sc = ldexpf(1.f, -e);
  float hh[kCols], ll[kCols];
#pragma unroll
  for (int c = 0; c < kCols; ++c) {
    hh[c] = h[c] * sc;
    ll[c] = lo[c] * sc;
  }
#pragma unroll 1
  for (int j = 0; j < kSlices; ++j) {
    float s[kCols];
#pragma unroll
    for (int c = 0; c < kCols; ++c) s[c] = next_slice(hh[c], ll[c], j);
    stage_B(g.bsl + j * kBSlice, l, s);
  }
  return e;
}

// Waits for the MMAs still reading buffer b.  Returns false on timeout.
__device__ __forceinline__ bool drain(Engine& g, int b) {
  if (((g.pend >> (8 * b)) & 255u) == 0) return true;
  if (!tc::mbar_wait(g.bar + 16u + 8u * (uint32_t)b, (g.eph >> b) & 1u)) return false;
  g.eph ^= 1u << b;
  g.pend -= 1u << (8 * b);
  return true;
}

// Hands a command (a staged slice, or -1 to stop) to the issuing warp on the
// next buffer: every worker calls it once its part of the slice is staged; the
// "full" barrier counts one arrival per warp.
__device__ __forceinline__ void hand_over(Engine& g, int cmd) {
  const int b = g.seq & 1;
  if (threadIdx.x == 0) g.cmd[b] = cmd;  // its last reader has committed the buffer's previous slice
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive(g.bar + 8u * (uint32_t)b);
}

// This worker's values of sum_l 2^(-8 l) L_l, scaled by sc, from the first
// LEVELS level accumulators; with `add` plus the pairs in (h, lo).
template <int LEVELS>
__device__ __forceinline__ void read_levels(const Engine& g, const Lane& l, float (&h)[kCols], float (&lo)[kCols], float sc,
                                            bool add) {
#pragma unroll
  for (int q = 0; q < kCols / 8; ++q) {
    float Lv[LEVELS][8];
    tmem_ld8xn<LEVELS>(g.tmem + l.lane_addr + (uint32_t)(l.c0 + 8 * q), Lv);
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      float L[LEVELS];
#pragma unroll
      for (int lv = 0; lv < LEVELS; ++lv) L[lv] = Lv[lv][c];
      float hi, lw;
      combine_levels<LEVELS>(L, hi, lw);
      df v{hi * sc, lw * sc};
      if (add) {
        v = df_add(v, df{h[8 * q + c], lo[8 * q + c]});
      }
      h[8 * q + c] = v.hi;
      lo[8 * q + c] = v.lo;
    }
  }
}

// The levels of a product whose entries may be off by 2^-need: levels beyond
// n leave about 2^(1 - 8 n) of the operands' scales 2^eX 2^eR (six or so slice
// pairs of 128 products of two digits each, added with random signs).
constexpr int kAllLevels = 1 << 16;  // need of a product with every level
__device__ __forceinline__ int levels_of(int eX, int eR, int need) {
  const int n = (eX + eR + need + 8) >> 3;
  return n < 4 ? 4 : n > kExpmLevels ? kExpmLevels : n;
}

// (h, lo) <- this worker's values of X R in df: X given by this worker's
// values (h, lo), R by the staged right-operand slices (exponent eR), entries
// to about 2^-need.  `during(h, lo)` runs while the last slices' MMAs execute
// (X is staged by then); with `add` the pairs it left in (h, lo) are added to
// the product.  Returns false (g.abort set) when a wait gave up.
template <class During>
__device__ __forceinline__ bool product(Engine& g, const Lane& l, float (&h)[kCols], float (&lo)[kCols], int eR,
                                        int need, bool add, During during) {
  const int eX = block_exp(g, h);
  const int levels = levels_of(eX, eR, need);
  const int n_slices = min(levels, kSlices);
  {
    const float sc = ldexpf(1.f, -eX);
#pragma unroll
    for (int c = 0; c < kCols; ++c) {
      h[c] *= sc;
      lo[c] *= sc;
    }
  }
  if (levels > kSlices) zero_level6<kCols>(g.tmem, l);  // this worker read it in the previous product's combine
  bool ok = true;
#pragma unroll 1
  for (int i = 0; i < n_slices; ++i) {
    const int b = g.seq & 1;
    ok &= drain(g, b);  // the pairs of slice i - 2 have read buffer b
    float s[kCols];
#pragma unroll
    for (int c = 0; c < kCols; ++c) s[c] = next_slice(h[c], lo[c], i);
    stage_A(g.abuf + b * kASlice, l, s);
    tc::fence_smem_to_async();
    tc::fence_before_sync();
    hand_over(g, i | levels << 8);
    g.pend += 1u << (8 * b);
    ++g.seq;
  }
  during(h, lo);
  ok &= drain(g, 0) & drain(g, 1);
  if (wsync_or(!ok)) {
    g.abort = true;
    return false;
  }
  tc::fence_after_sync();
  const float sc = ldexpf(1.f, eX + eR - 16);
  switch (levels) {
    case 4: read_levels<4>(g, l, h, lo, sc, add); break;
    case 5: read_levels<5>(g, l, h, lo, sc, add); break;
    case 6: read_levels<6>(g, l, h, lo, sc, add); break;
    default: read_levels<7>(g, l, h, lo, sc, add); break;
  }
  tc::fence_before_sync();  // accumulators read before the next product's MMAs
  return true;
}

// The issuing warp: waits for each staged slice in turn, issues its pairs and
// commits them to the buffer's "empty" barrier, until a stop command.  Every
// wait is bounded; a timeout stops it (the workers' own bounded waits then
// fail too).
// What the issue needs is kept provably warp-uniform (votes and reductions
// write uniform registers), so the descriptors are formed there.
__device__ __forceinline__ void issue_loop(const Engine& g) {
  constexpr uint32_t kAll = 0xffffffffu;
  const uint32_t bar = g.bar, abuf = tc::smem_u32(g.abuf), bsl = tc::smem_u32(g.bsl);
  const uint32_t tmem = __reduce_or_sync(kAll, g.tmem);
  const bool leader = (threadIdx.x & 31) == 0;
  uint32_t fph = 0;
#pragma unroll 1
  for (uint32_t n = 0;; ++n) {
    const uint32_t b = n & 1u;
    if (__any_sync(kAll, !tc::mbar_wait(bar + 8u * b, (fph >> b) & 1u))) return;
    fph ^= 1u << b;
    const int cmd = (int)__reduce_or_sync(kAll, (unsigned)g.cmd[b]);
    if (cmd < 0) return;
    tc::fence_after_sync();
    issue_slice(tmem, abuf + b * kASlice, bsl, cmd & 255, cmd >> 8);
    if (leader) tc::commit(bar + 16u + 8u * b);
    __syncwarp();
  }
}

// v <- a c and v <- v + a c as an unevaluated pair: the leading parts' sum
// and product errors are kept exactly in .lo, which is not folded into .hi.
__device__ __forceinline__ void df_scale(df a, df c, df& v) {
  v.hi = a.hi * c.hi;
  v.lo = fmaf(a.lo, c.hi, fmaf(a.hi, c.lo, fmaf(a.hi, c.hi, -v.hi)));
}
__device__ __forceinline__ void df_fma(df a, df c, df& v) {
  df p;
  df_scale(a, c, p);
  float e;
  two_sum(v.hi, p.hi, v.hi, e);
  v.lo += p.lo + e;
}

// (h, lo) <- this worker's values of the Horner block C_i = sum_{j<q}
// c_{qi+j} B^j (B^0 = I) as unevaluated pairs, with FROM_X plus c_{q(i+1)}
// times the values (h, lo) came with, then folded.  B comes from shared memory
// (g.ci), B^2 and B^3 from this worker's copies in the slab, whose loads are
// issued together: one trip to L2 instead of one per entry pair.
template <bool FROM_X>
__device__ __forceinline__ void horner_block(const Engine& g, int i, int q, const Lane& l, const float4* own,
                                             float (&h)[kCols], float (&lo)[kCols]) {
  const int o = q * i;
  const float4* B = reinterpret_cast<const float4*>(g.ci);
  const auto add = [&](const float4& b, df c, int cp) {
    df v0{h[2 * cp], lo[2 * cp]}, v1{h[2 * cp + 1], lo[2 * cp + 1]};
    df_fma(df{b.x, b.y}, c, v0);
    df_fma(df{b.z, b.w}, c, v1);
    h[2 * cp] = v0.hi;
    lo[2 * cp] = v0.lo;
    h[2 * cp + 1] = v1.hi;
    lo[2 * cp + 1] = v1.lo;
  };
  if constexpr (FROM_X) {
#pragma unroll
    for (int c = 0; c < kCols; ++c) {
      df v;
      df_scale(df{h[c], lo[c]}, c_dfcoef[o + q], v);
      h[c] = v.hi;
      lo[c] = v.lo;
    }
  } else {
#pragma unroll
    for (int c = 0; c < kCols; ++c) h[c] = lo[c] = 0.f;
  }
#pragma unroll 1
  for (int j = q - 1; j >= 2; --j) {
    float4 b[kCols / 2];
#pragma unroll
    for (int cp = 0; cp < kCols / 2; ++cp) b[cp] = __ldcg(own + (kCols / 2 * (j - 2) + cp) * kWorkers + threadIdx.x);
#pragma unroll
    for (int cp = 0; cp < kCols / 2; ++cp) add(b[cp], c_dfcoef[o + j], cp);
  }
#pragma unroll
  for (int cp = 0; cp < kCols / 2; ++cp) add(B[cp * kWorkers + threadIdx.x], c_dfcoef[o + 1], cp);
#pragma unroll
  for (int c = 0; c < kCols; ++c) {
    if (l.im == 0 && l.i == l.c0 + c) {
      const df v = df_add(df{h[c], lo[c]}, c_dfcoef[o]);
      h[c] = v.hi;
      lo[c] = v.lo;
    }
    if constexpr (FROM_X) fast_two_sum(h[c], lo[c], h[c], lo[c]);
  }
}

// Writes this worker's values as matrix `mat` (0: B^2, 1: B^3) of the
// own-value copies: thread-major float4 {hi, lo, hi, lo} per entry pair, so a
// warp's loads are 512 contiguous bytes.
__device__ __forceinline__ void store_own(float4* own, int mat, const float (&h)[kCols], const float (&lo)[kCols]) {
#pragma unroll
  for (int cp = 0; cp < kCols / 2; ++cp)
    own[(kCols / 2 * mat + cp) * kWorkers + threadIdx.x] =
        make_float4(h[2 * cp], lo[2 * cp], h[2 * cp + 1], lo[2 * cp + 1]);
}

// Index, in float4 {hi, lo, hi, lo} pairs, of row i, columns 2 cc and 2 cc + 1
// of the real (im = 0) or imaginary part in a matrix stored as the workers'
// own values.
__device__ __forceinline__ int own_pair(int i, int cc, int im) {
  return (cc % (kCols / 2)) * kWorkers + (cc / (kCols / 2)) * 128 + 64 * im + i;
}

// Shared-memory carve-up, TMEM, barriers and the engine state of a CTA of the
// sliced engine's kernels (kExpmThreads threads, kExpmSmem dynamic bytes).
struct CtaStatic {
  uint32_t tmem;
  uint64_t bar[5];  // full[2], empty[2], and the chain kernels' operand copies
  float red[2 * kWorkers / 32];
  int cmd[2];
};
__device__ __forceinline__ void engine_setup(Engine& g, uint8_t* smem_raw, CtaStatic& st) {
  const uint32_t pad = (tc::kSmemAlign - (tc::smem_u32(smem_raw) & (tc::kSmemAlign - 1))) & (tc::kSmemAlign - 1);
  g.bsl = smem_raw + pad;
  g.abuf = g.bsl + kSlices * kBSlice;
  g.ci = reinterpret_cast<float2*>(g.abuf + 2 * kASlice);
  g.red = st.red;
  g.cmd = st.cmd;
  g.par = 0;
  g.seq = 0;
  g.abort = false;
  g.eph = 0;
  g.pend = 0;
  g.bar = tc::smem_u32(&st.bar[0]);
  if (threadIdx.x < 32) tc::tmem_alloc(&st.tmem, tc::kTmemCols);
  if (threadIdx.x == 0)
    for (int b = 0; b < 5; ++b) mbar_init_n(tc::smem_u32(&st.bar[b]), b < 2 ? kWorkers / 32 : 1);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  g.tmem = st.tmem;
}

// The chain kernels' next left factor (one 64 KB df matrix, contiguous in
// HBM) into g.ci by two bulk copies (TMA) on barrier `mbar`; issued by worker
// 0 once every worker has read the previous one.
__device__ __forceinline__ void fetch_left(Engine& g, uint32_t mbar, const float4* src) {
  tc::mbar_expect_tx(mbar, 65536u);
  tc::tma_bulk_copy(tc::smem_u32(g.ci), src, 32768u, mbar);
  tc::tma_bulk_copy(tc::smem_u32(g.ci) + 32768u, reinterpret_cast<const uint8_t*>(src) + 32768, 32768u, mbar);
}
// This worker's values of the fetched matrix (after waiting for the copy).
__device__ __forceinline__ void read_left(const Engine& g, const Lane& l, float (&h)[kCols], float (&lo)[kCols]) {
  const float4* M = reinterpret_cast<const float4*>(g.ci);
#pragma unroll
  for (int c = 0; c < kCols; ++c) {
    const float4 v = M[l.i + 64 * (l.c0 + c)];
    h[c] = l.im ? v.y : v.x;
    lo[c] = l.im ? v.w : v.z;
  }
}
// Workers: stop the issuer, then (bounded) let the groups in flight finish.
__device__ __forceinline__ void workers_finish(Engine& g) {
  hand_over(g, -1);
  drain(g, 0);
  drain(g, 1);
}
// Every thread: frees TMEM once workers and issuer are done.
__device__ __forceinline__ void engine_teardown(Engine& g) {
  tc::fence_before_sync();
  __syncthreads();
  if (threadIdx.x < 32) {
    tc::fence_after_sync();
    tc::tmem_dealloc(g.tmem, tc::kTmemCols);
  }
}

}  // namespace oz

// Flag of the tensor-core expm: a completion wait gave up (its units are
// NaN-poisoned).
__device__ int g_expm_tc_timeout;

// Prologue of the tensor-core expm, per unit (member, slice): the generator
// A_k in df, its FP32 1-norm and the degree, block size and squarings (the
// CUDA-core kernel's choice, without the triangular costs).  A_k stays in the
// unit's U slot as the expm workers' own values (the expm scales it by 2^-s
// and overwrites the slot with exp(A_k) at the end).  Work for many warps,
// kept out of the one-CTA-per-SM tensor-core kernel.
//
// A CTA assembles NS consecutive slices of one member, so the operators (64 KB
// each) are read from L2 once for NS units, and thread t holds the pair
// (i, 2 cc), (i, 2 cc + 1) of each.  At 500 slices of 32 members and six
// controls 1.29 ms with one slice per CTA and renormalised sums; NS = 4 takes
// 0.75 ms.  Fewer slices than that many CTAs fill the SMs with: NS = 1.

// FP32 1-norm of a 64 x 64 matrix of moduli (column pitch kMagPitch) by all
// 256 threads (x 1.00001, as norm1f): thread t sums rows 16 (t % 4) .. + 15 of
// column t / 4, the four partial sums of a column meet by two xor shuffles
// (every lane of the four ends with the same sum), and the largest column
// comes from warp and block maxima.  red: 8 floats.
constexpr int kMagPitch = 65;
__device__ __forceinline__ float prep_norm1_64(const float* mag, float* red) {
  const int t = threadIdx.x, c = t >> 2, r0 = (t & 3) * 16;
  float s = 0.f;
#pragma unroll 4
  for (int r = r0; r < r0 + 16; ++r) s += mag[r + kMagPitch * c];
  s += __shfl_xor_sync(0xffffffffu, s, 1);
  s += __shfl_xor_sync(0xffffffffu, s, 2);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s = fmaxf(s, __shfl_xor_sync(0xffffffffu, s, o));
  if ((t & 31) == 0) red[t >> 5] = s;
  __syncthreads();
  float best = red[0];
#pragma unroll
  for (int i = 1; i < 8; ++i) best = fmaxf(best, red[i]);
  __syncthreads();  // red is the degree choice's scratch next
  return best * 1.00001f;
}

template <int NS>
__global__ void __launch_bounds__(256) k_expm_prep_oz64(ProbDev p, WorkDev w) {
  using oz::df_fma;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float* mag = reinterpret_cast<float*>(smem_raw);  // [NS][64 * kMagPitch] moduli
  float* red = mag + NS * 64 * kMagPitch;
  const Team<256> tm{(int)threadIdx.x};
  const int per = (p.n_t + NS - 1) / NS;
  const long items = (long)p.n_members * per;
  for (long it = blockIdx.x; it < items; it += gridDim.x) {
    const int m = (int)(it / per), k0 = (int)(it % per) * NS, n = min(NS, p.n_t - k0);
    const df sc = df_ld(p.m_scale_df[m]), off = df_ld(p.m_offset_df[m]);
    const float4* Gd = p.drifts_df + (size_t)p.m_drift[m] * 4096;
    const int ro = p.n_ramp ? p.m_ramp[m] : -1;
    const size_t unit = (size_t)m * p.n_t + k0;
#pragma unroll 1
    for (int e = tm.lane; e < 2048; e += 256) {
      const int i = e % 64, cc = e / 64, q0 = i + 128 * cc, q1 = q0 + 64;
      dfc v[NS][2];
      // v[s][.] += c[s] M, as pairs folded at the end
      const auto add = [&](const float4* M, auto coef) {
        const dfc a = dfc_load(M[q0]), b = dfc_load(M[q1]);
#pragma unroll
        for (int s = 0; s < NS; ++s) {
          const df c = coef(min(k0 + s, p.n_t - 1));
          df_fma(a.re, c, v[s][0].re);
          df_fma(a.im, c, v[s][0].im);
          df_fma(b.re, c, v[s][1].re);
          df_fma(b.im, c, v[s][1].im);
        }
      };
      {
        const dfc a = dfc_load(Gd[q0]), b = dfc_load(Gd[q1]);
#pragma unroll
        for (int s = 0; s < NS; ++s) {
          v[s][0] = a;
          v[s][1] = b;
        }
      }
      if (off.hi != 0.f) add(p.offset_df, [&](int) { return off; });
      if (ro >= 0) add(p.ramp_ops_df + (size_t)ro * 4096, [&](int k) { return df_ld(p.tau_df[k]); });
#pragma unroll 1
      for (int j = 0; j < p.n_c; ++j)
        add(p.ctrls_df + (size_t)j * 4096, [&](int k) { return df_mul(sc, df_ld(w.u_df[(size_t)k * p.n_c + j])); });
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        const df dt = df_ld(p.dt_df[min(k0 + s, p.n_t - 1)]);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          dfc& x = v[s][h];
          fast_two_sum(x.re.hi, x.re.lo, x.re.hi, x.re.lo);
          fast_two_sum(x.im.hi, x.im.lo, x.im.hi, x.im.lo);
          x = dfc_scale(x, dt);
          if (p.gen == GEN_HERM) x = {x.im, df_neg(x.re)};  // times -i
          mag[s * 64 * kMagPitch + i + kMagPitch * (2 * cc + h)] = sqrtf(fmaf(x.re.hi, x.re.hi, x.im.hi * x.im.hi));
        }
        if (s < n) {
          float4* out = reinterpret_cast<float4*>(w.U) + (unit + s) * 4096;
          const dfc x = v[s][0], y = v[s][1];
          // read once, by the expm
          __stcs(out + oz::own_pair(i, cc, 0), make_float4(x.re.hi, x.re.lo, y.re.hi, y.re.lo));
          __stcs(out + oz::own_pair(i, cc, 1), make_float4(x.im.hi, x.im.lo, y.im.hi, y.im.lo));
        }
      }
    }
    tm.sync();
    for (int s = 0; s < n; ++s) {
      const float nrm = prep_norm1_64(mag + s * 64 * kMagPitch, red);
      const int pk = choose_expm_df<256>(tm, nrm, 64, false, reinterpret_cast<int*>(red));
      if (tm.lane == 0) {  // and the exponent of a bound of ||B||: ||B||_1 < 2^x, -31 <= x <= 31
        int x;
        frexpf(ldexpf(nrm, -((pk >> 8) & 63)), &x);
        w.expm_plan[unit + s] = pk | (max(-31, min(31, x)) + 32) << 21;
      }
    }
    tm.sync();  // mag is rewritten by the next units
  }
}
constexpr size_t expm_prep_smem(int ns) { return (size_t)(ns * 64 * kMagPitch + 64) * sizeof(float); }

// 544 threads: an SM sub-partition hosts five of the 17 warps, so at most 96
// registers per thread.
__global__ void __launch_bounds__(oz::kExpmThreads, 1) k_expm_oz64(ProbDev p, WorkDev w) {
  using namespace oz;
  extern __shared__ uint8_t smem_raw[];
  __shared__ CtaStatic st;
  Engine g;
  engine_setup(g, smem_raw, st);
  if (threadIdx.x >= kWorkers) {  // the issuing warp
    issue_loop(g);
    __syncwarp();
  } else {
    const Lane l = worker_lane();
    float4* own = reinterpret_cast<float4*>(w.slab) + (size_t)blockIdx.x * 3 * (kCols / 2) * kWorkers;  // B^2, B^3
    const uint32_t tbar = tc::smem_u32(&st.bar[4]);
    uint32_t tph = 0;
    int tpend = 0;  // copies of B issued and not yet waited for
    const auto fetch = [&](long unit) {  // B of `unit` into g.ci: every worker has read the last one
      if (threadIdx.x == 0) fetch_left(g, tbar, reinterpret_cast<const float4*>(w.U) + (size_t)unit * 4096);
      ++tpend;
    };
    const long items = (long)p.n_members * p.n_t;
    long it = blockIdx.x;
    if (it < items) fetch(it);
    for (; it < items; it += gridDim.x) {
      const int m = (int)(it / p.n_t), k = (int)(it % p.n_t);
      const int pk = w.expm_plan[it];
      const int deg = pk & 31, q = (pk >> 5) & 7, s = (pk >> 8) & 63, nL = deg / q;
      const int nx = ((pk >> 21) & 63) - 32;  // ||B|| < 2^nx
      // x: the values this worker holds of the matrix in hand, first B
      float xh[kCols], xl[kCols];
      {
        const bool got = tc::mbar_wait(tbar, tph);
        if (wsync_or(!got)) {
          g.abort = true;
          break;
        }
        tph ^= 1;
        --tpend;
        float4* Bs = reinterpret_cast<float4*>(g.ci);
        const float sc = ldexpf(1.f, -s);
#pragma unroll
        for (int cp = 0; cp < kCols / 2; ++cp) {
          float4 v = Bs[cp * kWorkers + threadIdx.x];
          v = make_float4(v.x * sc, v.y * sc, v.z * sc, v.w * sc);
          if (s > 0) Bs[cp * kWorkers + threadIdx.x] = v;
          xh[2 * cp] = v.x;
          xl[2 * cp] = v.y;
          xh[2 * cp + 1] = v.z;
          xl[2 * cp + 1] = v.w;
        }
      }
      // The products of the unit, at one call site (one copy of the
      // product's code), in place on x:
      //   powers:  B^2 = B B (st 0), B^3 = B^2 B (st 1), B^4 = B^2 B^2 (st 2);
      //   then x = B^q becomes the right factor and Y = C_{L-1} + c_m B^q;
      //   Horner:  Y <- Y B^q + C_i, i = L-2 .. 0;
      //   squarings: Y <- Y Y.
      const int n_pow = q - 1, n_hor = nL - 1, n_steps = n_pow + n_hor + s;
      int eR = 0;
      bool ok = true;
#pragma unroll 1
      for (int st = 0; st <= n_steps && ok; ++st) {
        if (st == 1 && q >= 3) store_own(own, 0, xh, xl);
        if (st == 2 && q == 4) {  // B^4 = B^2 B^2
          store_own(own, 1, xh, xl);
#pragma unroll
          for (int cp = 0; cp < kCols / 2; ++cp) {
            const float4 v = own[cp * kWorkers + threadIdx.x];
            xh[2 * cp] = v.x;
            xl[2 * cp] = v.y;
            xh[2 * cp + 1] = v.z;
            xl[2 * cp + 1] = v.w;
          }
          eR = stage_right(g, l, xh, xl);
        }
        if (st == n_pow) {  // x = B^q
          if (n_hor > 0) eR = stage_right(g, l, xh, xl);
          horner_block<true>(g, nL - 1, q, l, own, xh, xl);
        }
        if (st == n_steps) break;
        if (st == 0 || st >= n_pow + n_hor) eR = stage_right(g, l, xh, xl);  // B; or a squaring's Y
        // The entries of exp(A) are wanted to 2^-kExpmBits: an error of Y after
        // Horner step i reaches exp(B) times B^{q i}, an error of a power as it
        // is (its coefficients are at most 1/2), and exp(B)'s grows by 2^s in
        // the squarings.
        const bool horner = st >= n_pow && st < n_pow + n_hor;
        const int i = n_pow + n_hor - 1 - st;
        const int need = st >= n_pow + n_hor ? kAllLevels : kExpmBits + s + (horner ? q * i * nx : 0);
        ok = product(g, l, xh, xl, eR, need, horner, [&](float (&h)[kCols], float (&lo)[kCols]) {
          if (horner) horner_block<false>(g, i, q, l, own, h, lo);
        });
      }
      if (!ok) break;
      if (s > 0) tc::fence_smem_to_async();  // this worker's scaled B, before the next copy into its place
      wsync();  // every worker is done with B
      if (it + gridDim.x < items) fetch(it + gridDim.x);
      // U: the stack streams out (gigabytes, read back from DRAM by the chains)
      float* out = reinterpret_cast<float*>(w.U) + ((size_t)m * p.n_t + k) * 64 * 64 * 4;
#pragma unroll
      for (int c = 0; c < kCols; ++c) {
        const size_t e = (size_t)(l.i + 64 * (l.c0 + c)) * 4;
        __stcs(out + e + l.im, xh[c]);
        __stcs(out + e + 2 + l.im, xl[c]);
      }
    }
    if (g.abort) {
      // units from the one that failed on: NaN, so no stale propagator is used
      const float nan = __int_as_float(0x7fffffff);
      for (; it < items; it += gridDim.x) {
        float* out = reinterpret_cast<float*>(w.U) + (size_t)it * 64 * 64 * 4;
        for (int e = threadIdx.x; e < 64 * 64 * 4; e += kWorkers) out[e] = nan;
      }
      if (threadIdx.x == 0) atomicOr(&g_expm_tc_timeout, 1);
      if (tpend > 0) tc::mbar_wait(tbar, tph);  // bounded: the copy in flight lands before the CTA ends
    }
    workers_finish(g);
  }
  engine_teardown(g);
}

// The parallel-in-time forward chain's in-block prefix products at D = 64 on
// the same engine: per (member m, block b of slices k0 .. k1-1) P_k0 = I,
// P_{k+1} = U_k P_k in df; with `store` the FP32 rounding of every P_k
// (k0 <= k < k1) for the gradient; the block product P_k1 into pit_tot.
// P_{k0+1} = U_k0 is taken as is.  Each step stages P_k as the right factor
// and multiplies U_k (left, this worker's values) into it; U_{k+1} arrives in
// shared memory by TMA bulk copies while the step's MMAs run.  Same CTA shape, barriers and
// bounded waits as k_expm_oz64; a CTA that gives up NaN-poisons the block
// products of its remaining items.
__global__ void __launch_bounds__(oz::kExpmThreads, 1) k_chainf_local_oz64(ProbDev p, WorkDev w, int store) {
  using namespace oz;
  extern __shared__ uint8_t smem_raw[];
  __shared__ CtaStatic st;
  Engine g;
  engine_setup(g, smem_raw, st);  // g.ci receives U_{k+1}
  if (threadIdx.x >= kWorkers) {
    issue_loop(g);
    __syncwarp();
  } else {
    const Lane l = worker_lane();
    const long items = (long)p.n_members * w.pit_blocks;
    const uint32_t tbar = tc::smem_u32(&st.bar[4]);
    uint32_t tph = 0;
    int tpend = 0;  // operand copies issued and not yet waited for
    // this worker's entries e = i + 64 c of a 4096-entry matrix
    const auto entry = [&](int c) { return (size_t)(l.i + 64 * (l.c0 + c)); };
    long it = blockIdx.x;
    for (; it < items; it += gridDim.x) {
      const int m = (int)(it / w.pit_blocks), b = (int)(it % w.pit_blocks);
      const int k0 = b * w.pit_len, k1 = min(p.n_t, k0 + w.pit_len);
      const float4* Um = reinterpret_cast<const float4*>(w.U) + (size_t)m * p.n_t * 4096;
      float* Pst = reinterpret_cast<float*>(w.P) + (size_t)m * p.n_t * 4096 * 2;  // float2 {re, im} per entry
      float xh[kCols], xl[kCols], uh[kCols], ul[kCols];
      if (store) {  // P_k0 = I
#pragma unroll
        for (int c = 0; c < kCols; ++c)
          Pst[((size_t)k0 * 4096 + entry(c)) * 2 + l.im] = (l.im == 0 && l.i == l.c0 + c) ? 1.f : 0.f;
      }
#pragma unroll
      for (int c = 0; c < kCols; ++c) {  // x = P_{k0+1} = U_k0
        const float4 v = Um[(size_t)k0 * 4096 + entry(c)];
        xh[c] = l.im ? v.y : v.x;
        xl[c] = l.im ? v.w : v.z;
      }
      bool ok = true;
      if (k0 + 1 < k1) {  // U_{k0+1} by TMA
        if (threadIdx.x == 0) fetch_left(g, tbar, Um + (size_t)(k0 + 1) * 4096);
        ++tpend;
      }
#pragma unroll 1
      for (int k = k0 + 1; k <= k1 && ok; ++k) {  // x holds P_k
        if (store && k < k1)
#pragma unroll
          for (int c = 0; c < kCols; ++c) Pst[((size_t)k * 4096 + entry(c)) * 2 + l.im] = xh[c];
        if (k == k1) break;
        const int eR = stage_right(g, l, xh, xl);  // P_k
        const bool got = tc::mbar_wait(tbar, tph);  // U_k in shared memory
        if (wsync_or(!got)) {
          g.abort = true;
          ok = false;
          break;
        }
        tph ^= 1;
        --tpend;
        read_left(g, l, uh, ul);
        const auto prefetch = [&](float (&)[kCols], float (&)[kCols]) {  // U_{k+1} while the MMAs run: every worker has read U_k
          if (k + 1 < k1) {
            if (threadIdx.x == 0) fetch_left(g, tbar, Um + (size_t)(k + 1) * 4096);
            ++tpend;
          }
        };
        ok = product(g, l, uh, ul, eR, kAllLevels, false, prefetch);  // U_k P_k
#pragma unroll
        for (int c = 0; c < kCols; ++c) {
          xh[c] = uh[c];
          xl[c] = ul[c];
        }
      }
      if (!ok) break;
      float* tot = reinterpret_cast<float*>(w.pit_tot + ((size_t)m * w.pit_blocks + b) * 4096);
#pragma unroll
      for (int c = 0; c < kCols; ++c) {
        tot[entry(c) * 4 + l.im] = xh[c];
        tot[entry(c) * 4 + 2 + l.im] = xl[c];
      }
    }
    if (g.abort) {
      const float nan = __int_as_float(0x7fffffff);
      for (; it < items; it += gridDim.x) {
        float* tot = reinterpret_cast<float*>(w.pit_tot + (size_t)it * 4096);
        for (int e = threadIdx.x; e < 4096 * 4; e += kWorkers) tot[e] = nan;
      }
      if (threadIdx.x == 0) atomicOr(&g_expm_tc_timeout, 1);
      if (tpend > 0) tc::mbar_wait(tbar, tph);  // bounded: the copy in flight lands before the CTA ends
    }
    workers_finish(g);
  }
  engine_teardown(g);
}

// The parallel-in-time forward chain's combine at D = 64 on the same engine:
// per member P = I, then for each block b in order pit_pre[b] = P (FP32, when
// `store`) and P <- T_b P in df (T_0 I = T_0 as is; T_{b+1} arrives by TMA
// bulk copies while step b's MMAs run); then the CUDA-core
// kernel's epilogue (U_total in FP64, the overlap, f and the chain-rule
// coefficient) on P copied into shared memory.  A CTA that gives up
// NaN-poisons the objective of its remaining members.
__global__ void __launch_bounds__(oz::kExpmThreads, 1) k_chainf_combine_oz64(ProbDev p, WorkDev w, int store) {
  using namespace oz;
  extern __shared__ uint8_t smem_raw[];
  __shared__ CtaStatic st;
  Engine g;
  engine_setup(g, smem_raw, st);
  if (threadIdx.x >= kWorkers) {
    issue_loop(g);
    __syncwarp();
  } else {
    const Lane l = worker_lane();
    const Team<kWorkers> tm{(int)threadIdx.x, 1};           // the workers' barrier
    float4* Pc = reinterpret_cast<float4*>(g.ci);       // 64 KB: P for the epilogue
    double2* red = reinterpret_cast<double2*>(g.abuf);  // the epilogue's scratch (idle slice buffers)
    const auto entry = [&](int c) { return (size_t)(l.i + 64 * (l.c0 + c)); };
    const uint32_t tbar = tc::smem_u32(&st.bar[4]);
    uint32_t tph = 0;
    int tpend = 0;  // operand copies issued and not yet waited for
    int m = blockIdx.x;
    for (; m < p.n_members; m += gridDim.x) {
      float xh[kCols], xl[kCols], uh[kCols], ul[kCols];
#pragma unroll
      for (int c = 0; c < kCols; ++c) {  // P = I
        xh[c] = (l.im == 0 && l.i == l.c0 + c) ? 1.f : 0.f;
        xl[c] = 0.f;
      }
      bool ok = true;
      const float4* Tm = w.pit_tot + (size_t)m * w.pit_blocks * 4096;
      if (store) {  // pit_pre[0] = I
        float* pre = reinterpret_cast<float*>(w.pit_pre + (size_t)m * w.pit_blocks * 4096);
#pragma unroll
        for (int c = 0; c < kCols; ++c) pre[entry(c) * 2 + l.im] = xh[c];
      }
#pragma unroll
      for (int c = 0; c < kCols; ++c) {  // P = T_0 I = T_0
        const float4 v = Tm[entry(c)];
        xh[c] = l.im ? v.y : v.x;
        xl[c] = l.im ? v.w : v.z;
      }
      if (w.pit_blocks > 1) {  // T_1 by TMA
        if (threadIdx.x == 0) fetch_left(g, tbar, Tm + 4096);
        ++tpend;
      }
#pragma unroll 1
      for (int b = 1; b < w.pit_blocks && ok; ++b) {
        if (store) {
          float* pre = reinterpret_cast<float*>(w.pit_pre + ((size_t)m * w.pit_blocks + b) * 4096);
#pragma unroll
          for (int c = 0; c < kCols; ++c) pre[entry(c) * 2 + l.im] = xh[c];
        }
        const int eR = stage_right(g, l, xh, xl);  // P
        const bool got = tc::mbar_wait(tbar, tph);  // T_b in shared memory
        if (wsync_or(!got)) {
          g.abort = true;
          ok = false;
          break;
        }
        tph ^= 1;
        --tpend;
        read_left(g, l, uh, ul);
        const auto prefetch = [&](float (&)[kCols], float (&)[kCols]) {  // T_{b+1} while the MMAs run: every worker has read T_b
          if (b + 1 < w.pit_blocks) {
            if (threadIdx.x == 0) fetch_left(g, tbar, Tm + (size_t)(b + 1) * 4096);
            ++tpend;
          }
        };
        ok = product(g, l, uh, ul, eR, kAllLevels, false, prefetch);  // T_b P
#pragma unroll
        for (int c = 0; c < kCols; ++c) {
          xh[c] = uh[c];
          xl[c] = ul[c];
        }
      }
      if (!ok) break;
#pragma unroll
      for (int c = 0; c < kCols; ++c) {
        float* f = reinterpret_cast<float*>(Pc + entry(c));
        f[l.im] = xh[c];
        f[2 + l.im] = xl[c];
      }
      wsync();
      chain_epilogue_mx<64, kWorkers>(tm, p, w, m, Pc, red);
      tc::fence_smem_to_async();  // these writes to g.ci before the next member's copies into it
      wsync();  // P and the scratch are read before the next member reuses them
    }
    if (g.abort && threadIdx.x == 0) {
      for (; m < p.n_members; m += gridDim.x) w.Fm[m] = __longlong_as_double(0x7ff8000000000000LL);
      atomicOr(&g_expm_tc_timeout, 1);
    }
    if (g.abort && tpend > 0) tc::mbar_wait(tbar, tph);  // bounded: the copy in flight lands first
    workers_finish(g);
  }
  engine_teardown(g);
}

}  // namespace pgx
