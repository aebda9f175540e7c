// te_resident.cu -- all three-term Lanczos iterations of a Krylov step in one
// cooperative launch with the recurrence's rows in registers.
//
// Replaces, for matrices whose rows fit (te_resident_fits), the loop of
// arnoldiAlgorithm (core/krylovTimeEvolver.cpp:523-571).  What bounds an
// iteration of such a matrix is not bandwidth but the chain apply -> <u_j, w'>
// over all rows -> update -> all rows visible -> next apply, so the kernel is
// laid out for the length of that chain:
//  * one block per SM; a warp owns CPW chunks of 32 rows for the whole step
//    and keeps u_j, u_{j-1} and w' of its rows in registers.  Only the vector
//    that other SMs gather (u_j, or its fixed-point copy X_j) goes through
//    memory, and the matrix slots are read through L1, which holds a block's
//    share of a small matrix from one iteration to the next;
//  * chunk c belongs to block c mod gridDim.x: rows are sorted by length, so
//    every block gets the same mix of lengths;
//  * the two grid-wide sums are exact integers (as on the per-pass
//    fixed-point path): each warp adds its lanes' values as 24-bit limbs
//    (redux.sync), each block its warps', and one lane per limb adds the
//    block's sum to a 64-bit word whose upper 16 bits count the blocks.  A
//    reader knows from the word itself that its sum is complete, so the sum
//    is its own barrier: no separate arrival counter, and no FP64 reduction
//    tree (a warp-wide FP64 instruction costs 64 cycles here);
//  * maxima (the fixed-point scale, as tight as the passes': the scale costs
//    u_{j+1} a bit per factor of two) go out as one tagged word per block and
//    are read once a sum is complete, when they have nearly always arrived:
//    max|w'| while alpha_j / e is formed, max|u_{j+1}| while the others gather.
//    (Polled together with the sums they took the L2 slices' time, see below;
//    counted by exponent inside a sum's line, below a bound known beforehand,
//    they cost ten and more bits where ||H|| is far above what the state
//    reaches: energies of 1e4 and more in rows that no other row couples to.)
//  * every scalar of the recurrence is a product of ||u_j||^2 and its
//    reciprocal: c_w = (beta_j / e)^2 = S_{j-1} ||u_j||^2, alpha_j / e =
//    S_j <u_j, w'> with S_j = s_j^2 = 1 / ||u_j||^2, so the chain holds no
//    square root and no division: one spare warp computes S_j, beta_j and s_j
//    while the others gather.
//
// Times on GB300, per iteration: Bose-Hubbard L=10 (dim 92 378) 31 us as two
// passes, 11.4 us here; an exchange takes 2 to 4 thousand cycles, the gathers
// 6 700, the rows' FP64 recurrence 4 100 of an iteration's 23 000.  With the
// rows' sums of all 152 blocks in tagged words instead (one line per 16
// blocks) the polls themselves took the L2 slices' time: 16 us.
#include <algorithm>
#include <cmath>

#include "te_fixed.cuh"
#include "te_internal.cuh"

namespace {

constexpr int kResWarps = 19;     // worker warps per block at most
constexpr int kResMaxCpw = 4;     // chunks per worker warp at most
constexpr int kMaxPerLane = 5;    // blocks whose maximum a lane reads
constexpr int kResMaxBlocks = 32 * kMaxPerLane;
static_assert(sizeof(TeResidentSync::wmax) == 2 * kResMaxBlocks * sizeof(unsigned long long), "a word per block");
constexpr int kStreamMaxWarps = 31;        // worker warps per block of the streaming kernel at most
// Its dynamic shared memory at most.  The L1 has the rest of the SM's 256 KB, and
// the gathers in flight need it: us per iteration, passes / streamed, random
// rows of up to 64 and 256 (complex): 1.2 M 167 / 137 and 350 / 253, 1.5 M (158
// KB) 202 / 189 and 421 / 350, 1.9 M (196 KB) 245 / 517 and 481 / 966.
constexpr size_t kStreamSmem = 160 << 10;
// Worker warps and slots in flight per lane by format (0 real limbs, 1 value
// dictionary, 2 complex limbs): more warps leave fewer registers for slots in
// flight.  Measured per iteration on GB300, dictionary (Bose-Hubbard L=12): 31
// warps of 2 / 4 / 6 slots 79 / 66 / 63 us, 27 of 6 68, 23 of 8 71; complex
// (dim 1 000 003, 49 M entries): 31 of 6 235 us, 27 of 6 222, 23 of 8 216.
template <int FMT>
constexpr int kStreamWarps = FMT == 1 ? 31 : FMT == 2 ? 23 : 27;
template <int FMT>
constexpr int kStreamSlots = FMT == 2 ? 8 : 6;
constexpr int kLimbs = 5;                // of 24 bits each
constexpr int kAlphaWords = 2 * kLimbs;  // <u_j, w'>: re, im
constexpr int kNormWords = kLimbs;       // ||u_{j+1}||^2
constexpr unsigned int kNonFinite = 0x7ff00000u;  // high word of an infinity, the least of a non-finite value
constexpr int kCountShift = 48;   // blocks counted in bits 48..63 of a word
constexpr unsigned long long kTopBias = 1ull << 34;  // per block, keeps a signed top limb's sum positive

// exponent x with |v| < 2^x (from the high word; zero and subnormals give -1022)
__device__ __forceinline__ int exp_above(unsigned int hiword) { return (int)((hiword >> 20) & 0x7ffu) - 1022; }
__device__ __forceinline__ int exp_above(double v) { return exp_above(te_fix_hiword(v)); }

struct ResShared {
  int part[kStreamMaxWarps][kAlphaWords];  // per-warp limb sums
  unsigned int pmax[kStreamMaxWarps];
  double cw, gr, gi;
  int k1, k2, xs;  // units of the two sums, fixed-point scale of u_{j+1}
  int go;          // 1 continue, 0 leave (a wait gave up)
  int go_start;    // 1 continue, 0 lucky breakdown, -1 a wait gave up
  double norm2[TE_MMAX + 1], cws[TE_MMAX + 1];  // ||u_j||^2 and (beta_j / e)^2 of the step
};

// A warp's sum of limbs (24 bits each); lane l < N keeps limb l.
template <int N>
__device__ __forceinline__ void warp_limbs(const int (&limb)[N], int* out) {
  const int lane = threadIdx.x & 31;
  int mine = 0;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int s = __reduce_add_sync(0xffffffffu, limb[i]);
    if (lane == i) mine = s;
  }
  if (lane < N) out[lane] = mine;
}

// A warp's sum of the lanes' x in units of 2^-k, as limbs (the top one signed).
// The caller's units keep a top limb below 2^23; an x beyond (not finite, or a
// matrix whose norm is beyond the units' range) counts as zero here and as
// non-finite in mx, so that no limb runs into the count of blocks.
__device__ __forceinline__ void warp_limbs_signed(double x, int k, int* out, unsigned int& mx) {
  unsigned long long lo = 0ull, hi = 0ull;
  const unsigned int h = te_fix_hiword(x);
  if (h >= kNonFinite || (h >= 0x100000u && exp_above(h) + k >= 24 * kLimbs))
    mx = kNonFinite;
  else
    te_fix_encode128(x, k, lo, hi);  // 0 for a zero and subnormals
  const int limb[kLimbs] = {(int)(lo & 0xffffffull), (int)((lo >> 24) & 0xffffffull),
                            (int)(((lo >> 48) | (hi << 16)) & 0xffffffull), (int)((hi >> 8) & 0xffffffull),
                            (int)(hi >> 32)};
  warp_limbs<kLimbs>(limb, out);
}

// Sum over limb words (weights 2^24i, the top one biased) as a 128-bit integer.
template <int N>
__device__ __forceinline__ void limbs_join(const unsigned long long (&t)[N], unsigned long long bias,
                                           unsigned long long& lo, unsigned long long& hi) {
  const unsigned long long mask = (1ull << kCountShift) - 1;
  lo = hi = 0;
#pragma unroll
  for (int i = N - 1; i >= 0; --i) {
    // {hi, lo} = {hi, lo} << 24 + t_i
    hi = (hi << 24) | (lo >> 40);
    lo <<= 24;
    const long long v = (long long)(t[i] & mask) - (i == N - 1 ? (long long)bias : 0ll);
    const unsigned long long add = (unsigned long long)v;
    lo += add;
    hi += (v < 0 ? ~0ull : 0ull) + (lo < add ? 1ull : 0ull);
  }
}

__device__ __forceinline__ unsigned long long ld_relaxed(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void red_add(unsigned long long* p, unsigned long long v) {
  asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ void st_relaxed(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

}  // namespace

struct TeResidentArgs {
  int64_t n;
  int n_chunks, n_workers, m;
  const int64_t* chunk_off;
  const int32_t* col;
  const double* val;   // FP64 slots
  const int2* hv;      // fixed point: real limbs
  const int4* hv4;     // fixed point: complex limbs
  const uint32_t* pk;  // fixed point: value dictionary
  const int2* table;
  int nvals, cbits, sh;
  int r_exp;           // ||H|| < 2^r_exp
  int n_exp;           // 2 n < 2^n_exp
  int4* X;             // fixed point: copies of the basis (m x n)
  TeResidentSync* sync;
  int parity;         // which half of sync this launch uses
  unsigned int tag0;  // tags of this launch's maxima: tag0 + j
  unsigned int spin_limit, arrivals;
  double2* u[TE_MMAX];
};

// One lane's row of chunk slots [s, e) times the gathered vector, by format:
// 0 fixed real limbs, 1 fixed value dictionary, 2 fixed complex limbs,
// 3 FP64 real, 4 FP64 complex.  UNR slots in flight per lane: registers are
// plentiful at one block per SM, and the gathers' latency is the chain.
template <int FMT, int UNR>
__device__ __forceinline__ double2 res_row(const TeResidentArgs& a, const int2* tab, int s, int e, const void* x,
                                           int shift) {
  if (FMT >= 3) {
    const double2* xv = static_cast<const double2*>(x);
    double re = 0.0, im = 0.0;
#pragma unroll UNR
    for (; s < e; s += 32) {
      const double2 v = __ldca(xv + __ldg(a.col + s));
      if (FMT == 3) {
        const double h = __ldg(a.val + s);
        re = fma(h, v.x, re);
        im = fma(h, v.y, im);
      } else {
        const double2 h = __ldg(reinterpret_cast<const double2*>(a.val) + s);
        re = fma(h.x, v.x, re);
        re = fma(-h.y, v.y, re);
        im = fma(h.x, v.y, im);
        im = fma(h.y, v.x, im);
      }
    }
    return make_double2(re, im);
  }
  const int4* xv = static_cast<const int4*>(x);
  int64_t sr = 0, si = 0;
  if (FMT == 1) {
    const uint32_t cmask = (1u << a.cbits) - 1u;
#pragma unroll UNR
    for (; s < e; s += 32) {
      const uint32_t wd = __ldg(a.pk + s);
      te_fix_mac(tab[wd >> a.cbits], __ldca(xv + (wd & cmask)), sr, si);
    }
  } else if (FMT == 0) {
#pragma unroll UNR
    for (; s < e; s += 32) te_fix_mac(__ldg(a.hv + s), __ldca(xv + __ldg(a.col + s)), sr, si);
  } else {
#pragma unroll UNR
    for (; s < e; s += 32) {
      const int4 h = __ldg(a.hv4 + s);
      const int4 v = __ldca(xv + __ldg(a.col + s));
      sr += te_fix_prod(h.x, h.y, v.x, v.y) - te_fix_prod(h.z, h.w, v.z, v.w);
      si += te_fix_prod(h.x, h.y, v.z, v.w) + te_fix_prod(h.z, h.w, v.x, v.y);
    }
  }
  return make_double2(te_i64_to_double(sr, 62 - shift), te_i64_to_double(si, 62 - shift));
}

// The spare warp sends this block's words: its warps' limb sums (the signed top
// limbs biased), and its maximum, tagged.
template <int N>
__device__ __forceinline__ void res_send(const TeResidentArgs& a, const ResShared& S, unsigned long long* words,
                                         unsigned long long* maxima, unsigned int tag) {
  const int lane = threadIdx.x & 31, l = lane & 15;
  unsigned long long v = 0;
  unsigned int mx = 0;
  for (int w = 0; w < a.n_workers; ++w) {
    if (l < N) v += (unsigned long long)(long long)S.part[w][l];
    mx = max(mx, S.pmax[w]);
  }
  if (lane == 31) st_relaxed(maxima + blockIdx.x, ((unsigned long long)tag << 32) | mx);
  if (l % kLimbs == kLimbs - 1) v += kTopBias;
  v += 1ull << kCountShift;
  if (lane < N) red_add(words + lane, v);
}

// The grid's words on lanes 0..N-1 (spare warp); false when the wait gave up.
template <int N>
__device__ __forceinline__ bool res_receive(const TeResidentArgs& a, const unsigned long long* words,
                                            unsigned long long& word, TeDevState* ds) {
  const int lane = threadIdx.x & 31;
  word = 0;
  unsigned int spins = 0;
  while (true) {
    bool ok = true;
    if (lane < N) {
      word = ld_relaxed(words + lane);
      ok = (unsigned int)(word >> kCountShift) == a.arrivals;
    }
    if (__all_sync(0xffffffffu, ok)) return true;
    if (++spins > a.spin_limit) {
      if (lane == 0) atomicExch(&ds->fatal, TE_ERR_DEVICE_TIMEOUT);
      return false;
    }
  }
}

// The blocks' tagged maxima, kMaxPerLane per lane: fetched first, then waited
// for until every tag has arrived (false: gave up).
struct ResMaxima {
  unsigned long long t[kMaxPerLane];
};
__device__ __forceinline__ ResMaxima res_fetch(const unsigned long long* maxima) {
  ResMaxima r;
#pragma unroll
  for (int k = 0; k < kMaxPerLane; ++k) {
    const int b = (threadIdx.x & 31) + 32 * k;
    r.t[k] = b < (int)gridDim.x ? ld_relaxed(maxima + b) : 0ull;
  }
  return r;
}
__device__ __forceinline__ bool res_max(const TeResidentArgs& a, const unsigned long long* maxima, unsigned int tag,
                                        ResMaxima r, unsigned int& hiword, TeDevState* ds) {
  const int lane = threadIdx.x & 31;
  unsigned int spins = 0;
  while (true) {
    bool ok = (unsigned int)gridDim.x == a.arrivals;
    unsigned int m = 0;
#pragma unroll
    for (int k = 0; k < kMaxPerLane; ++k) {
      if (lane + 32 * k < (int)gridDim.x) ok = ok && (unsigned int)(r.t[k] >> 32) == tag;
      m = max(m, (unsigned int)r.t[k]);
    }
    if (__all_sync(0xffffffffu, ok)) {
      hiword = __reduce_max_sync(0xffffffffu, m);
      return true;
    }
    if (++spins > a.spin_limit) {
      if (lane == 0) atomicExch(&ds->fatal, TE_ERR_DEVICE_TIMEOUT);
      return false;
    }
    r = res_fetch(maxima);
  }
}

// The same as a call, from the fetch on.
__device__ __noinline__ bool res_max_call(const TeResidentArgs& a, const unsigned long long* maxima, unsigned int tag,
                                          unsigned int& hiword, TeDevState* ds) {
  return res_max(a, maxima, tag, res_fetch(maxima), hiword, ds);
}
template <bool CALL>
__device__ __forceinline__ bool res_grid_max(const TeResidentArgs& a, const unsigned long long* maxima,
                                             unsigned int tag, unsigned int& hiword, TeDevState* ds) {
  if constexpr (CALL)
    return res_max_call(a, maxima, tag, hiword, ds);
  else
    return res_max(a, maxima, tag, res_fetch(maxima), hiword, ds);
}

// Spare warp, from the grid's words of <u_j, w'> and its maxima: alpha_j / e =
// S_j <u_j, w'>, the fixed-point scale of u_{j+1} from B = (W + (|Re| + |Im|)
// (alpha_j / e) U)(1 + 1e-12) (W >= max|w'|, U >= max|u_j|, as in
// lanczos_update_kernel), and the units of its norm.  False: the wait for the
// maxima gave up.  EARLY: the maxima are on their way while alpha_j is formed.
template <bool EARLY, bool CALL>
__device__ __forceinline__ bool res_alpha(const TeResidentArgs& a, ResShared& S, unsigned long long word, double Sj,
                                          unsigned int umax, const unsigned long long* maxima, unsigned int tag,
                                          double e, int j, bool leader, int G, TeDevState* ds) {
  ResMaxima r{};
  if constexpr (EARLY) r = res_fetch(maxima);
  // the even lanes join re, the odd lanes im
  const int lane = threadIdx.x & 31, im = lane & 1;
  unsigned long long t[kLimbs], lo, hi;
#pragma unroll
  for (int i = 0; i < kLimbs; ++i) t[i] = __shfl_sync(0xffffffffu, word, i + kLimbs * im);
  limbs_join<kLimbs>(t, (unsigned long long)G * kTopBias, lo, hi);
  double g = Sj * te_i128_to_double(lo, hi, -S.k1);
  unsigned int wmax = 0;
  if (!(EARLY ? res_max(a, maxima, tag, r, wmax, ds) : res_grid_max<CALL>(a, maxima, tag, wmax, ds))) return false;
  const double go = __shfl_xor_sync(0xffffffffu, g, 1);
  const double B = fma(fabs(g) + fabs(go), te_fix_upper(umax), te_fix_upper(wmax)) * (1.0 + 1e-12);
  const int xs = te_fix_scale(B);
  // beyond the scale's range (or not finite): no coefficients rather than wrong ones
  const double nan = __longlong_as_double(0x7ff8000000000000ll);
  const bool fits = max(wmax, umax) < kNonFinite && B < 1e300;
  g = fits ? g : nan;
  if (lane == 0) {
    S.gr = g;
    S.gi = fits ? go : nan;
    S.xs = xs;
    S.k2 = a.X ? 2 * xs - 62 : 117 - (2 * exp_above(B) + a.n_exp);
    if (leader) {
      ds->alpha[j] = make_double2(S.gr * e, S.gi * e);
      if (a.X) ds->fx_xs[j + 1] = xs;
    }
  }
  __syncwarp();
  return true;
}

// ||u_{j+1}||^2 from the grid's words.
__device__ __forceinline__ double res_norm(const ResShared& S, unsigned long long word, int G) {
  unsigned long long t[kLimbs], lo, hi;
#pragma unroll
  for (int i = 0; i < kLimbs; ++i) t[i] = __shfl_sync(0xffffffffu, word, i);
  limbs_join<kLimbs>(t, (unsigned long long)G * kTopBias, lo, hi);
  return te_u128_to_double(hi, lo, -S.k2);
}

// Start of iteration j on the spare warp, while the others gather: max|u_j|,
// then the scalars that the rows and the sum of <u_j, w'> need.  umax: the
// high word of max|u_j|, known at j = 0 on the fixed-point path.
template <bool CALL>
__device__ __forceinline__ void res_start(const TeResidentArgs& a, ResShared& S, int j, bool leader, double bd2,
                                          unsigned int& umax, double& Sj, double& norm2, TeDevState* ds) {
  const int lane = threadIdx.x & 31;
  bool ok = true;
  if (j > 0 || !a.X) {
    const unsigned long long* maxima = a.sync->umax[j & 1];
    ok = res_grid_max<CALL>(a, maxima, a.tag0 + j, umax, ds);
    if (umax >= kNonFinite) norm2 = __longlong_as_double(0x7ff8000000000000ll);
  }
  const double cw = j > 0 ? Sj * norm2 : 0.0;  // (beta_j / e)^2
  const bool go = !(cw < bd2) || j == 0;       // else the lucky breakdown (:551-555)
  if (lane == 0) {
    S.cw = cw;
    S.go_start = !ok ? -1 : go ? 1 : 0;
    // units 2^-k1 of <u_j, w'>: |<u_j, w'>| <= ||u_j||^2 (||H|| + beta_j / e),
    // 12 bits to spare (||H|| in the 2-norm is below the 1-norm, sqrt(n) of it
    // for an H that is not Hermitian).  ||u_0|| is only bounded through max|u_0|
    const int ex = j == 0 ? 2 * exp_above(umax) + a.n_exp : exp_above(norm2);
    S.k1 = 24 * kLimbs - 14 - ex - max(a.r_exp, j > 0 ? (exp_above(cw) + 2) / 2 : -2000);
    if (leader && j > 0) {
      S.norm2[j] = norm2;
      S.cws[j] = cw;
    }
  }
  if (j > 0) Sj = 1.0 / norm2;
}
// The same as a call.
__device__ __noinline__ void res_start_call(const TeResidentArgs& a, ResShared& S, int j, bool leader, double bd2,
                                            unsigned int& umax, double& Sj, double& norm2, TeDevState* ds) {
  res_start<false>(a, S, j, leader, bd2, umax, Sj, norm2, ds);
}

// The spare warp's registers come out of the others' loads in flight, so where its
// code is a call and when it fetches the maxima was measured per format and chunks
// per warp.  us per iteration, all inlined and early / with this choice / (before
// the maxima were exchanged, the fewest registers): start as a call, 90 000 rows of
// up to 256 real 38.6 / 36.5 / (37.1), 150 000 complex 122 / 103 / (122), 220 000
// complex 143 / 119 / (145), streamed complex 1 000 003 225 / 214 / (217); inlined
// for the dictionary, Bose-Hubbard L=10 11.3 (a call 11.7) / (11.5); 4 chunks:
// maxima as a call, 369 000 complex 163 / 154 / (160); late, 369 000 real FP64 53.0 /
// 51.9 / (51.9).
template <int FMT, int CPW>
constexpr bool kStartCall = CPW == 4 ? FMT == 1 || FMT == 4 : FMT != 1;
template <int FMT, int CPW>
constexpr bool kMaxCall = CPW == 4 && FMT == 2;
template <int FMT, int CPW>
constexpr bool kEarly = CPW < 4 || FMT == 1 || FMT == 4;

// End of a launch, first block: the step's coefficients beta_j = |e| sqrt((beta_j
// / e)^2), s_j = +-1 / ||u_j|| (s_j = e s_{j-1} / beta_j); the last one is h, or
// the breakdown's.
__device__ void res_coefficients(const ResShared& S, int last_j, bool broke, double bd2, double e, TeDevState* ds) {
  for (int j = 1 + (int)threadIdx.x; j <= last_j; j += blockDim.x) {
    const double b = fabs(e) * sqrt(S.cws[j]);
    if (j < last_j) {
      const double sn = 1.0 / sqrt(S.norm2[j]);
      ds->beta[j] = b;
      ds->s[j] = e < 0.0 && (j & 1) ? -sn : sn;
    } else {
      ds->h = b;
      ds->m_eff = j;
      if (broke || S.cws[j] < bd2) ds->breakdown = 1;
    }
  }
}

template <int FMT, int CPW>
__global__ void __launch_bounds__((kResWarps + 1) * 32, 1) lanczos_resident_kernel(TeResidentArgs a, TeDevState* ds) {
  constexpr bool FIX = FMT < 3;
  __shared__ ResShared S;
  extern __shared__ int2 tab[];  // FMT 1: the value table
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int G = gridDim.x;
  const bool leader = blockIdx.x == 0;
  TeResidentSync& sy = *a.sync;
  if (leader)  // the other half, for the next launch (no launch in flight uses it)
    for (int i = threadIdx.x; i < TE_MMAX * 32; i += blockDim.x) (&sy.words[a.parity ^ 1][0][0])[i] = 0ull;
  if (ds->fatal != 0 || ds->done != 0 || ds->breakdown != 0) return;
  if (FMT == 1)
    for (int i = threadIdx.x; i < a.nvals; i += blockDim.x) tab[i] = a.table[i];
  const int m = min(a.m, ds->m_cur);
  const double e = ds->exp_factor;
  const bool spare = warp == a.n_workers;
  // this lane's rows: chunks blockIdx.x + (warp + i n_workers) G
  int s0[CPW], s1[CPW];
  int row[CPW];
  double2 u[CPW], up[CPW], w[CPW];
  unsigned int mx = 0;
#pragma unroll
  for (int i = 0; i < CPW; ++i) {
    const int64_t c = blockIdx.x + (int64_t)(warp + i * a.n_workers) * G;
    const bool have = !spare && c < a.n_chunks;
    s0[i] = have ? (int)__ldg(a.chunk_off + c) + lane : 0;
    s1[i] = have ? (int)__ldg(a.chunk_off + c + 1) : 0;
    const int64_t r = c * 32 + lane;
    row[i] = have && r < a.n ? (int)r : -1;
    u[i] = row[i] >= 0 ? a.u[0][row[i]] : make_double2(0.0, 0.0);
    up[i] = make_double2(0.0, 0.0);
    if (!FIX) mx = max(mx, max(te_fix_hiword(u[i].x), te_fix_hiword(u[i].y)));
  }
  // scalars of the spare warp (the same in every block): S_j = s_j^2 and
  // ||u_j||^2, the high word of max|u_j|
  double Sj = 1.0, norm2 = 1.0;
  unsigned int umax = FIX ? ds->fx_umax[0] : 0u;
  int xs = FIX ? ds->fx_xs[0] : 0;
  const double bd2 = (ds->tol_rate / e) * (ds->tol_rate / e);
  int last_j = m;
  bool broke = false;
  if (!FIX) {
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (!spare && lane == 0) S.pmax[warp] = mx;
  }
  __syncthreads();  // the value table, or the maxima of u_0
  if (!FIX && spare) {
    mx = 0;
    for (int w = 0; w < a.n_workers; ++w) mx = max(mx, S.pmax[w]);
    if (lane == 0) st_relaxed(sy.umax[0] + blockIdx.x, ((unsigned long long)a.tag0 << 32) | mx);
  }
  for (int j = 0; j < m; ++j) {
    unsigned long long* words = sy.words[a.parity][j];
    // apply: y = H u_j for the workers; the spare warp finishes the previous
    // norm meanwhile
    if (!spare) {
      const void* x = FIX ? (const void*)(a.X + (int64_t)j * a.n) : (const void*)a.u[j];
#pragma unroll
      for (int i = 0; i < CPW; ++i) w[i] = res_row<FMT, CPW == 1 ? 8 : 4>(a, tab, s0[i], s1[i], x, a.sh + xs);
    } else {
      if constexpr (kStartCall<FMT, CPW>)
        res_start_call(a, S, j, leader, bd2, umax, Sj, norm2, ds);
      else
        res_start<kMaxCall<FMT, CPW>>(a, S, j, leader, bd2, umax, Sj, norm2, ds);
    }
    __syncthreads();
    if (S.go_start < 0) return;
    if (S.go_start == 0) {
      last_j = j;
      broke = true;
      break;
    }
    if (!spare) {
      const double cw = S.cw;
      double dr = 0.0, di = 0.0;
      mx = 0;
#pragma unroll
      for (int i = 0; i < CPW; ++i) {
        if (row[i] >= 0) {
          // w' = -i H u_j + c_w u_{j-1}; <u_j, w'> += conj(u_j) w'
          const double2 y = w[i];
          if (j > 0) {
            w[i].x = fma(cw, up[i].x, y.y);
            w[i].y = fma(cw, up[i].y, -y.x);
          } else {
            w[i] = make_double2(y.y, -y.x);
          }
          dr = fma(u[i].x, w[i].x, fma(u[i].y, w[i].y, dr));
          di = fma(u[i].x, w[i].y, fma(-u[i].y, w[i].x, di));
          mx = max(mx, max(te_fix_hiword(w[i].x), te_fix_hiword(w[i].y)));
        }
      }
      warp_limbs_signed(dr, S.k1, S.part[warp], mx);
      warp_limbs_signed(di, S.k1, S.part[warp] + kLimbs, mx);
      mx = __reduce_max_sync(0xffffffffu, mx);
      if (lane == 0) S.pmax[warp] = mx;
    }
    __syncthreads();
    if (spare) {
      unsigned long long *maxima = sy.wmax[j & 1], word;
      res_send<kAlphaWords>(a, S, words, maxima, a.tag0 + j);
      const bool ok = res_receive<kAlphaWords>(a, words, word, ds) &&
                      res_alpha<kEarly<FMT, CPW>, kMaxCall<FMT, CPW>>(a, S, word, Sj, umax, maxima, a.tag0 + j, e, j,
                                                                      leader, G, ds);
      if (lane == 0) S.go = ok ? 1 : 0;
    }
    __syncthreads();
    if (!S.go) return;
    xs = S.xs;
    if (!spare) {
      // update: u_{j+1} = w' - (alpha_j / e) u_j
      const double gr = S.gr, gi = S.gi;
      unsigned long long lo = 0, hi = 0;
      double nr = 0.0;
      mx = 0;
#pragma unroll
      for (int i = 0; i < CPW; ++i) {
        if (row[i] >= 0) {
          double2 o;
          o.x = fma(-gr, u[i].x, fma(gi, u[i].y, w[i].x));
          o.y = fma(-gr, u[i].y, fma(-gi, u[i].x, w[i].y));
          up[i] = u[i];
          u[i] = o;
          mx = max(mx, max(te_fix_hiword(o.x), te_fix_hiword(o.y)));
          if (FIX) {
            const int64_t er = te_fix_encode(o.x, xs), ei = te_fix_encode(o.y, xs);
            if (j + 1 < m) {
              const int2 p = te_fix_split(er), q = te_fix_split(ei);
              a.X[(int64_t)(j + 1) * a.n + row[i]] = make_int4(p.x, p.y, q.x, q.y);
            }
            const unsigned long long sq = te_fix_sq(er) + te_fix_sq(ei);
            lo += sq;
            hi += lo < sq ? 1ull : 0ull;
          } else {
            if (j + 1 < m) a.u[j + 1][row[i]] = o;
            nr = fma(o.x, o.x, fma(o.y, o.y, nr));
          }
        }
      }
      if (!FIX) {
        te_fix_encode128(nr, S.k2, lo, hi);
        if (te_fix_hiword(nr) >= kNonFinite) mx = kNonFinite;
      }
      int limb[kNormWords];
      limb[0] = (int)(lo & 0xffffffull);
      limb[1] = (int)((lo >> 24) & 0xffffffull);
      limb[2] = (int)(((lo >> 48) | (hi << 16)) & 0xffffffull);
      limb[3] = (int)((hi >> 8) & 0xffffffull);
      limb[4] = (int)((hi >> 32) & 0xffffffull);
      warp_limbs<kNormWords>(limb, S.part[warp]);
      mx = __reduce_max_sync(0xffffffffu, mx);
      if (lane == 0) S.pmax[warp] = mx;
    }
    __syncthreads();
    const bool last = j + 1 == m;
    if (spare) {
      fence_gpu();  // the rows this block stored, before its sums
      unsigned long long *maxima = sy.umax[(j + 1) & 1], word;
      res_send<kNormWords>(a, S, words + 16, maxima, a.tag0 + j + 1);
      bool ok = true;
      if (!last || leader) {
        ok = res_receive<kNormWords>(a, words + 16, word, ds);
        fence_gpu();  // the other blocks' rows, after their sums
        if (ok) norm2 = res_norm(S, word, G);
      }
      if (last && leader && ok) {
        ok = res_grid_max<kMaxCall<FMT, CPW>>(a, maxima, a.tag0 + m, umax, ds);
        if (umax >= kNonFinite) norm2 = __longlong_as_double(0x7ff8000000000000ll);
        if (lane == 0) {
          S.cws[m] = Sj * norm2;
          S.norm2[m] = norm2;
        }
      }
      if (lane == 0) S.go = ok ? 1 : 0;
    }
    __syncthreads();
    if (!S.go) return;
  }
  if (leader) res_coefficients(S, last_j, broke, bd2, e, ds);
}

// --------------------------------------------------------------------------
// The same iterations for rows that do not fit the registers (fixed point
// only): chunk c belongs to block c mod gridDim.x, the block's warps take its
// chunks in turn (the same ones in every iteration), w' of its rows stays in
// shared memory, u_j and u_{j-1} are read back. Against the two passes an
// iteration saves w' through memory, two launches and the serial FP64 start of
// every block (square root and divisions on the spare warp here).  No unit is
// full (L1 data pipe 51%, integer multiplies 40%, FP64 39%, issue 36% of their
// cycles): what bounds it is a warp's own chain per chunk (offsets, words, gathers,
// products, rows: 9 000 cycles) at 31 warps an SM; the slot loop has no predicates (groups of U, then 4, 2, 1) and
// 32-bit counters, since predicated groups with the next words fetched ahead
// doubled the instructions (95 us).  Gathers made coalesced, or all from L1,
// change nothing (61.4, 59.4 us), nor does a value table per lane (62.1).
// Measured on GB300 per iteration: Bose-Hubbard L=12 (dim 1 352 078, 113 values)
// 85.6 us in two passes, 61.1 us here; complex, dim 1 000 003, 49 M entries: 293
// -> 214 us.  In the L=12 iteration's 124 000 cycles the row sums take 85 000,
// the update 22 000, the two exchanges with their scalars 16 000.
template <int FMT, int U>
__device__ __forceinline__ void stream_slots(const TeResidentArgs& a, const int2* tab, int s, const int4* X,
                                             int64_t& sr, int64_t& si) {
  int4 x[U];
  if (FMT == 1) {
    const uint32_t cmask = (1u << a.cbits) - 1u;
    uint32_t wd[U];
#pragma unroll
    for (int q = 0; q < U; ++q) wd[q] = __ldcs(a.pk + s + 32 * q);
#pragma unroll
    for (int q = 0; q < U; ++q) x[q] = __ldca(X + (wd[q] & cmask));
#pragma unroll
    for (int q = 0; q < U; ++q) te_fix_mac(tab[wd[q] >> a.cbits], x[q], sr, si);
  } else if (FMT == 0) {
    int2 h[U];
#pragma unroll
    for (int q = 0; q < U; ++q) {
      h[q] = __ldcs(a.hv + s + 32 * q);
      x[q] = __ldca(X + (uint32_t)__ldcs(a.col + s + 32 * q));
    }
#pragma unroll
    for (int q = 0; q < U; ++q) te_fix_mac(h[q], x[q], sr, si);
  } else {
    int4 h[U];
#pragma unroll
    for (int q = 0; q < U; ++q) {
      h[q] = __ldcs(a.hv4 + s + 32 * q);
      x[q] = __ldca(X + (uint32_t)__ldcs(a.col + s + 32 * q));
    }
#pragma unroll
    for (int q = 0; q < U; ++q) {
      sr += te_fix_prod(h[q].x, h[q].y, x[q].x, x[q].y) - te_fix_prod(h[q].z, h[q].w, x[q].z, x[q].w);
      si += te_fix_prod(h[q].x, h[q].y, x[q].z, x[q].w) + te_fix_prod(h[q].z, h[q].w, x[q].x, x[q].y);
    }
  }
}

template <int FMT>
__global__ void __launch_bounds__((kStreamWarps<FMT> + 1) * 32, 1)
    lanczos_stream_kernel(TeResidentArgs a, TeDevState* ds) {
  constexpr int W = kStreamWarps<FMT>, U = kStreamSlots<FMT>;
  __shared__ ResShared S;
  extern __shared__ __align__(16) unsigned char dyn[];  // w' of the block's rows; FMT 1: the value table
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int G = gridDim.x;
  const bool leader = blockIdx.x == 0;
  TeResidentSync& sy = *a.sync;
  if (leader)  // the other half, for the next launch (no launch in flight uses it)
    for (int i = threadIdx.x; i < TE_MMAX * 32; i += blockDim.x) (&sy.words[a.parity ^ 1][0][0])[i] = 0ull;
  if (ds->fatal != 0 || ds->done != 0 || ds->breakdown != 0) return;
  // chunks blockIdx.x + i G, i < nc; warp w takes i = w, w + W, ...
  const int nc = (a.n_chunks - (int)blockIdx.x + G - 1) / G;
  double2* ws = reinterpret_cast<double2*>(dyn);
  int2* tab = reinterpret_cast<int2*>(ws + nc * 32);
  if (FMT == 1)
    for (int i = threadIdx.x; i < a.nvals; i += blockDim.x) tab[i] = a.table[i];
  const int m = min(a.m, ds->m_cur);
  const double e = ds->exp_factor;
  const bool spare = warp == W;
  const uint32_t n32 = (uint32_t)a.n;
  double Sj = 1.0, norm2 = 1.0;  // the spare warp's, as in the resident kernel
  unsigned int umax = ds->fx_umax[0];
  int xs = ds->fx_xs[0];
  const double bd2 = (ds->tol_rate / e) * (ds->tol_rate / e);
  int last_j = m;
  bool broke = false;
  __syncthreads();  // the value table
  for (int j = 0; j < m; ++j) {
    unsigned long long* words = sy.words[a.parity][j];
    const int4* X = a.X + (int64_t)j * a.n;
    const double2 *uj = a.u[j], *up = a.u[j > 0 ? j - 1 : 0];
    double dr = 0.0, di = 0.0;
    unsigned int mx = 0;
    if (spare) res_start_call(a, S, j, leader, bd2, umax, Sj, norm2, ds);
    // apply; the first chunk's row sums before the scalars are needed
    bool first = true;
    double cw = 0.0;
    if (!spare) {
      const int shift = a.sh + xs;
      for (int i = warp; i < nc; i += W) {
        const int c = (int)blockIdx.x + i * G;
        int s = (int)__ldg(a.chunk_off + c);
        int len = ((int)__ldg(a.chunk_off + c + 1) - s) >> 5;
        s += lane;
        const uint32_t r = (uint32_t)c * 32u + lane;
        const bool live = r < n32;
        int64_t sr = 0, si = 0;
        for (; len >= U; len -= U, s += 32 * U) stream_slots<FMT, U>(a, tab, s, X, sr, si);
        if (len >= 4) {
          stream_slots<FMT, 4>(a, tab, s, X, sr, si);
          s += 128;
          len -= 4;
        }
        if (len >= 2) {
          stream_slots<FMT, 2>(a, tab, s, X, sr, si);
          s += 64;
          len -= 2;
        }
        if (len) stream_slots<FMT, 1>(a, tab, s, X, sr, si);
        const double yr = te_i64_to_double(sr, 62 - shift), yi = te_i64_to_double(si, 62 - shift);
        if (first) {  // the spare warp's scalars
          asm volatile("bar.sync 1, %0;" ::"r"((W + 1) * 32) : "memory");
          first = false;
          if (S.go_start != 1) break;
          cw = S.cw;
        }
        if (live) {
          // w' = -i H u_j + c_w u_{j-1}; <u_j, w'> += conj(u_j) w'
          const double2 u = __ldca(uj + r);
          double2 w = make_double2(yi, -yr);
          if (j > 0) {
            const double2 v = __ldca(up + r);
            w.x = fma(cw, v.x, yi);
            w.y = fma(cw, v.y, -yr);
          }
          ws[i * 32 + lane] = w;
          dr = fma(u.x, w.x, fma(u.y, w.y, dr));
          di = fma(u.x, w.y, fma(-u.y, w.x, di));
          mx = max(mx, max(te_fix_hiword(w.x), te_fix_hiword(w.y)));
        }
      }
    }
    if (first) asm volatile("bar.sync 1, %0;" ::"r"((W + 1) * 32) : "memory");
    if (S.go_start < 0) return;
    if (S.go_start == 0) {
      last_j = j;
      broke = true;
      break;
    }
    if (!spare) {
      warp_limbs_signed(dr, S.k1, S.part[warp], mx);
      warp_limbs_signed(di, S.k1, S.part[warp] + kLimbs, mx);
      mx = __reduce_max_sync(0xffffffffu, mx);
      if (lane == 0) S.pmax[warp] = mx;
    }
    __syncthreads();
    if (spare) {
      unsigned long long *maxima = sy.wmax[j & 1], word;
      res_send<kAlphaWords>(a, S, words, maxima, a.tag0 + j);
      const bool ok = res_receive<kAlphaWords>(a, words, word, ds) &&
                      res_alpha<true, false>(a, S, word, Sj, umax, maxima, a.tag0 + j, e, j, leader, G, ds);
      if (lane == 0) S.go = ok ? 1 : 0;
    }
    __syncthreads();
    if (!S.go) return;
    xs = S.xs;
    if (!spare) {
      // update: u_{j+1} = w' - (alpha_j / e) u_j
      const double gr = S.gr, gi = S.gi;
      unsigned long long lo = 0, hi = 0;
      mx = 0;
      int4* Xn = a.X + (int64_t)(j + 1) * a.n;
      double2* un = a.u[j + 1 < m ? j + 1 : j];
#pragma unroll 2
      for (int i = warp; i < nc; i += W) {
        const uint32_t r = ((uint32_t)blockIdx.x + (uint32_t)i * G) * 32u + lane;
        if (r < n32) {
          const double2 w = ws[i * 32 + lane], u = __ldca(uj + r);
          double2 o;
          o.x = fma(-gr, u.x, fma(gi, u.y, w.x));
          o.y = fma(-gr, u.y, fma(-gi, u.x, w.y));
          mx = max(mx, max(te_fix_hiword(o.x), te_fix_hiword(o.y)));
          const int64_t er = te_fix_encode(o.x, xs), ei = te_fix_encode(o.y, xs);
          if (j + 1 < m) {
            const int2 p = te_fix_split(er), q = te_fix_split(ei);
            Xn[r] = make_int4(p.x, p.y, q.x, q.y);
            un[r] = o;
          }
          const unsigned long long sq = te_fix_sq(er) + te_fix_sq(ei);
          lo += sq;
          hi += lo < sq ? 1ull : 0ull;
        }
      }
      int limb[kNormWords];
      limb[0] = (int)(lo & 0xffffffull);
      limb[1] = (int)((lo >> 24) & 0xffffffull);
      limb[2] = (int)(((lo >> 48) | (hi << 16)) & 0xffffffull);
      limb[3] = (int)((hi >> 8) & 0xffffffull);
      limb[4] = (int)((hi >> 32) & 0xffffffull);
      warp_limbs<kNormWords>(limb, S.part[warp]);
      mx = __reduce_max_sync(0xffffffffu, mx);
      if (lane == 0) S.pmax[warp] = mx;
    }
    __syncthreads();
    const bool last = j + 1 == m;
    if (spare) {
      fence_gpu();  // the rows this block stored, before its sums
      unsigned long long *maxima = sy.umax[(j + 1) & 1], word;
      res_send<kNormWords>(a, S, words + 16, maxima, a.tag0 + j + 1);
      bool ok = true;
      if (!last || leader) {
        ok = res_receive<kNormWords>(a, words + 16, word, ds);
        fence_gpu();  // the other blocks' rows, after their sums
        if (ok) norm2 = res_norm(S, word, G);
      }
      if (last && leader && ok) {
        ok = res_grid_max<false>(a, maxima, a.tag0 + m, umax, ds);
        if (umax >= kNonFinite) norm2 = __longlong_as_double(0x7ff8000000000000ll);
        if (lane == 0) {
          S.cws[m] = Sj * norm2;
          S.norm2[m] = norm2;
        }
      }
      if (lane == 0) S.go = ok ? 1 : 0;
    }
    __syncthreads();
    if (!S.go) return;
  }
  if (leader) res_coefficients(S, last_j, broke, bd2, e, ds);
}

namespace {

using ResKernel = void (*)(TeResidentArgs, TeDevState*);

template <int FMT>
ResKernel res_kernel_cpw(int cpw) {
  switch (cpw) {
    case 1: return lanczos_resident_kernel<FMT, 1>;
    case 2: return lanczos_resident_kernel<FMT, 2>;
    case 3: return lanczos_resident_kernel<FMT, 3>;
    default: return lanczos_resident_kernel<FMT, 4>;
  }
}

ResKernel res_kernel(int fmt, int cpw) {
  switch (fmt) {
    case 0: return res_kernel_cpw<0>(cpw);
    case 1: return res_kernel_cpw<1>(cpw);
    case 2: return res_kernel_cpw<2>(cpw);
    case 3: return res_kernel_cpw<3>(cpw);
    default: return res_kernel_cpw<4>(cpw);
  }
}

}  // namespace

// w' of a block's rows and the value table fit its shared memory (1.55 million
// rows on 152 SMs), fixed-point form built.
bool te_stream_fits(const TeSell& A) {
  if (A.n_long > 0 || A.fix_nblk > 0 || te_num_sms() > kResMaxBlocks || A.slots >= ((int64_t)1 << 31) - 256) return false;
  const int64_t most = (A.n_chunks + te_num_sms() - 1) / te_num_sms();
  return (size_t)most * 512 + sizeof(int2) * A.fix_nvals <= kStreamSmem;
}

// Rows that fit the registers of one block per SM: kResWarps warps of
// kResMaxCpw chunks (369 664 rows on 152 SMs).
bool te_resident_fits(const TeSell& A, bool fixed) {
  if (A.n_long > 0 || A.n < 1 || (fixed && A.fix_nblk > 0) || te_num_sms() > kResMaxBlocks) return false;
  if (A.slots >= ((int64_t)1 << 31) - 256) return false;  // 32-bit slot counters
  return A.n_chunks <= (int64_t)te_num_sms() * kResWarps * kResMaxCpw;
}

bool te_launch_lanczos_resident(const TeSell& A, bool is_real, bool fixed, double norm1, double2* const* cols, int m,
                                int4* X, TeDevState* ds, TeResidentSync* sync, unsigned int launch, cudaStream_t st,
                                unsigned int spin_limit, unsigned int extra_arrivals) {
  const bool stream = !te_resident_fits(A, fixed);
  if (m < 1 || m > TE_MMAX || (stream && !(fixed && te_stream_fits(A)))) return false;
  const int G = stream ? te_num_sms() : (int)std::min<int64_t>(te_num_sms(), A.n_chunks);
  const int per_block = (int)((A.n_chunks + G - 1) / G);
  const int cpw = (per_block + kResWarps - 1) / kResWarps;
  TeResidentArgs a{};
  a.n = A.n;
  a.n_chunks = (int)A.n_chunks;
  a.m = m;
  a.chunk_off = A.chunk_off;
  a.col = A.col;
  a.val = A.val;
  a.hv = A.fix_val;
  a.hv4 = A.fix_val4;
  a.pk = A.fix_pk;
  a.table = A.fix_table;
  a.nvals = A.fix_nvals;
  a.cbits = A.fix_cbits;
  a.sh = A.fix_sh;
  int ex = 0;
  std::frexp(norm1 > 0.0 && norm1 < 1e300 ? norm1 : 1.0, &ex);
  if (fixed) ex = std::max(ex, 61 - A.fix_sh);  // ||H||_inf < 2^(61 - sh)
  a.r_exp = ex;
  a.n_exp = 2;
  while (((int64_t)1 << (a.n_exp - 2)) < A.n) ++a.n_exp;
  a.X = fixed ? X : nullptr;
  a.sync = sync;
  a.parity = (int)(launch & 1u);
  a.tag0 = (launch + 1u) * 128u;
  a.spin_limit = spin_limit;
  a.arrivals = (unsigned int)G + extra_arrivals;
  for (int j = 0; j < TE_MMAX; ++j) a.u[j] = j < m ? cols[j] : nullptr;
  const int fmt = fixed ? (A.fix_val4 ? 2 : (A.fix_pk ? 1 : 0)) : (is_real ? 3 : 4);
  a.n_workers = !stream    ? (per_block + cpw - 1) / cpw
                : fmt == 1 ? kStreamWarps<1>
                : fmt == 2 ? kStreamWarps<2>
                           : kStreamWarps<0>;
  const ResKernel k = !stream    ? res_kernel(fmt, cpw)
                      : fmt == 2 ? lanczos_stream_kernel<2>
                      : fmt == 1 ? lanczos_stream_kernel<1>
                                 : lanczos_stream_kernel<0>;
  size_t smem = fmt == 1 ? sizeof(int2) * A.fix_nvals : 0;
  if (stream) {
    smem += (size_t)per_block * 512;
    if (cudaFuncSetAttribute((const void*)k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kStreamSmem) !=
        cudaSuccess) {
      cudaGetLastError();
      return false;
    }
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(G);
  cfg.blockDim = dim3((a.n_workers + 1) * 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, k, a, ds) != cudaSuccess) {
    cudaGetLastError();  // a refused launch is not an error of the evolution: the caller falls back
    return false;
  }
  return true;
}
