// te_lanczos.cu -- one Lanczos iteration of arnoldiAlgorithm
// (core/krylovTimeEvolver.cpp:523-571) as two grid passes.
//
// The basis is kept unnormalised: u_0 = currentVec, v_j = s_j u_j with
// s_j = 1/beta_j.  Iteration j:
//   pass 1 (apply):  w = A v_j + beta_j v_{j-1}       (A = -i expFactor H; the
//                    reference subtracts H[j-1,j] = -beta_j, :537-541)
//                    alpha_j = <v_j, w>                (:542-543)
//   pass 2 (update): u_{j+1} = w - alpha_j v_j         (:544-546)
//                    beta_{j+1} = ||u_{j+1}||          (:548)
//                    lucky breakdown if beta_{j+1} < tolRate (:551-555)
// The 1/beta scaling of :558-565 is deferred into s_{j+1}, so no pass rewrites
// a vector.  The Krylov coefficients never leave the device.  On the FP64
// path each pass finishes its reduction in the last block to complete (fixed
// order).  On the fixed-point path alpha_j and ||u_{j+1}||^2 are summed exactly
// as 128-bit integers with per-block atomics, and the pass after each sum
// finishes it (no block waits for the others; the total does not depend on
// the order of the atomics).  Pass 1 runs on the SELL-32 layout: a warp owns
// 32 equal-length rows.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "te_internal.cuh"
#include "te_reduce.cuh"
#include "te_sell.cuh"
#include "te_fixed.cuh"

__device__ __forceinline__ bool te_step_inactive(const TeDevState* ds) {
  return ds->fatal != 0 || ds->done != 0 || ds->breakdown != 0;
}

// The recurrence epilogue of one row r (A u_j row sum y): writes w (or the
// folded w') and accumulates conj(u_j) w.
template <bool HAS_PREV, bool FOLD>
__device__ __forceinline__ double2 apply_row_epilogue(int64_t r, double2 y, double g, double cw,
                                                   const double2* __restrict__ u_j,
                                                   const double2* __restrict__ u_jm1, double2* __restrict__ w,
                                                   double (&acc)[2]) {
  double2 wr;
  if (FOLD) {
    if (HAS_PREV) {
      double2 up = u_jm1[r];
      wr.x = fma(cw, up.x, y.y);
      wr.y = fma(cw, up.y, -y.x);
    } else {
      wr.x = y.y;
      wr.y = -y.x;
    }
  } else if (HAS_PREV) {
    double2 up = u_jm1[r];
    wr.x = fma(cw, up.x, g * y.y);
    wr.y = fma(cw, up.y, -g * y.x);
  } else {
    wr.x = g * y.y;
    wr.y = -g * y.x;
  }
  w[r] = wr;
  double2 uj = u_j[r];
  // conj(u_j) * w
  acc[0] = fma(uj.x, wr.x, fma(uj.y, wr.y, acc[0]));
  acc[1] = fma(uj.x, wr.y, fma(-uj.y, wr.x, acc[1]));
  return wr;
}

// 6 (real H: at most 40 registers) or 5 (complex H, or K > 1) resident blocks
// of 256; the static chunk schedule of the matrix assumes the whole grid is
// resident.
//
// FOLD (three-term mode, expFactor != 0): with g = expFactor s_j the kernel
// stores w' = w / g = -i H u_j + (beta_j s_{j-1} / g) u_{j-1}, which saves the
// two multiplications by g per row (FP64 issue is the bound); alpha_j is
// still the reference's <v_j, w> = s_j g <u_j, w'>.
//
// K lanes per row: K = 1 walks the matrix's static chunk schedule; K = 2, 4
// (small matrices, chosen by te_tune_sell_lanes) give each warp 32/K rows and
// stride over (chunk, part) units.
// LONG: the matrix has long rows (merge-path segments).  Matrices without
// them take the instantiation without that loop, whose registers otherwise
// spill from the slot loop.
template <bool REAL, bool HAS_PREV, bool FOLD, int K, bool LONG = true>
__global__ void __launch_bounds__(TE_THREADS, (REAL && K == 1) ? 6 : 5) lanczos_apply_kernel(
    int64_t n, int64_t n_chunks, const int32_t* __restrict__ warp_chunk, const int64_t* __restrict__ chunk_off,
    const int32_t* __restrict__ col, const double* __restrict__ val, TeLongRows L, const double2* __restrict__ u_j,
    const double2* __restrict__ u_jm1, double2* __restrict__ w, TeDevState* ds, double* partials, int j) {
  __shared__ double scratch[2 * 32];
  __shared__ double wide[2 * TE_THREADS];
  te_pdl_trigger();
  te_pdl_wait();
  if (te_step_inactive(ds)) return;
  const int lane = threadIdx.x & 31;
  const double sj = ds->s[j];
  const double g = ds->exp_factor * sj;  // A v_j = -i g H u_j
  // the u_{j-1} term: beta_j s_{j-1}, divided by g when folded; the folded
  // update sets s_j = expFactor s_{j-1} / beta_j, so that is beta_j^2 / expFactor^2
  double cw = 0.0;
  if (HAS_PREV) {
    const double bj = ds->beta[j];
    const double ie = ds->inv_exp_factor;
    cw = FOLD ? (bj * ie) * (bj * ie) : bj * ds->s[j - 1];
  }
  double acc[2] = {0.0, 0.0};
  const int64_t wid = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (K == 1) {
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    // long rows (sorted rows 0..L.n-1) by merge-path segments, one warp each
    for (int64_t sg = wid; LONG && sg < L.n_seg; sg += warps) {
      int64_t lr;
      double2 y;
      const int done = te_long_segment<REAL>(L, sg, u_j, lane, &lr, &y);
      if (done == 1 && lane == 0) apply_row_epilogue<HAS_PREV, FOLD>(lr, y, g, cw, u_j, u_jm1, w, acc);
      if (done == 2 && lane == 0) {  // a split row: its terms join the final sum in row order
        double a2[2] = {0.0, 0.0};
        apply_row_epilogue<HAS_PREV, FOLD>(lr, y, g, cw, u_j, u_jm1, w, a2);
        te_split_row_publish(L, lr, a2);
      }
    }
    // 32-bit chunk counter and an unsigned live-row test (rows < 2^31): fewer
    // registers across the slot loop
    const int c_end = warp_chunk[wid + 1];
    const uint32_t live_lo = (uint32_t)L.n, live_cnt = (uint32_t)(n - L.n);
    for (int c = warp_chunk[wid]; c < c_end; ++c) {
      const double2 y = te_sell_row<REAL>(chunk_off, col, val, u_j, c, lane);
      const int64_t r = (int64_t)c * 32 + lane;
      if ((uint32_t)r - live_lo < live_cnt) apply_row_epilogue<HAS_PREV, FOLD>(r, y, g, cw, u_j, u_jm1, w, acc);
    }
  } else {
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t u = wid; u < n_chunks * K; u += warps) {
      const int64_t c = u / K;
      const int part = (int)(u - c * K);
      const double2 y = te_sell_row_k<REAL, K>(chunk_off, col, val, u_j, c, part, lane);
      const int64_t r = c * 32 + part * (32 / K) + lane / K;
      if (lane % K == 0 && r < n) apply_row_epilogue<HAS_PREV, FOLD>(r, y, g, cw, u_j, u_jm1, w, acc);
    }
  }
  te_block_sum_wide<2>(acc, wide);
  if (te_publish_partials<2>(acc, partials, &ds->counter[0])) {
    double tot[2];
    te_final_sum<2>(tot, partials, &ds->counter[0], scratch, [&](double (&o)[2]) { te_split_rows_add(o, L); });
    const double f = FOLD ? sj * g : sj;
    if (threadIdx.x == 0) {
      const double2 alpha = make_double2(f * tot[0], f * tot[1]);
      ds->alpha[j] = alpha;
      const double q = FOLD ? ds->inv_exp_factor : sj;  // alpha_j s_j / g = alpha_j / expFactor when folded
      ds->upd_gr = alpha.x * q;
      ds->upd_gi = alpha.y * q;
    }
  }
}

// Block maximum of a per-thread unsigned value, folded into *dst with one
// atomicMax by thread 0.  Call between the warp loop and a block-wide
// synchronisation that precedes thread 0's read (slots: one per warp).
__device__ __forceinline__ void te_warp_max_to_smem(unsigned int v, unsigned int* slots) {
  v = __reduce_max_sync(0xffffffffu, v);
  if ((threadIdx.x & 31) == 0) slots[threadIdx.x >> 5] = v;
}
__device__ __forceinline__ unsigned int te_block_max_from_smem(const unsigned int* slots) {
  unsigned int m = 0;
  for (int i = 0; i < (int)(blockDim.x >> 5); ++i) m = max(m, slots[i]);
  return m;
}

// Start of a fixed-point apply pass j, by thread 0 of every block (a square
// root and divisions are long FP64 sequences on GB300), shared through sh[3]:
// for j > 0, beta_j = |e s_{j-1}| ||u'_j|| from the exact norm that update
// pass j - 1 accumulated, s_j = e s_{j-1} / beta_j, or the lucky breakdown
// (:551-555; false is returned and the pass does nothing); then the units
// 2^-k of the exact <u_j, w'> sum, from the bound
// |<u_j, w'>| <= ||u_j|| (R ||u_j|| + c_w ||u_{j-1}||) with ||u_i|| = 1/|s_i|,
// R < 2^(61 - sh) the matrix's row-norm bound, doubled for rounding, below
// 2^(124 - k).  Block 0 records beta_j, s_j and k.
template <bool HAS_PREV>
__device__ __forceinline__ bool fix_apply_prologue(TeDevState* ds, int j, int msh, double* sh, double& sj, double& bj,
                                                   int& k) {
  if (threadIdx.x == 0) {
    double s0 = ds->s[j], b = 0.0;
    bool ok = true;
    if (HAS_PREV) {
      const unsigned long long lo = ds->fx_nrm[j][0], hi = ds->fx_nrm[j][1];
      const double gp = ds->exp_factor * ds->s[j - 1];
      b = fabs(gp) * sqrt(te_u128_to_double(hi, lo, 62 - 2 * ds->fx_xs[j]));
      if (b < ds->tol_rate) {
        ok = false;
        if (blockIdx.x == 0) {
          ds->breakdown = 1;
          ds->m_eff = j;
          ds->h = b;
        }
      } else {
        s0 = gp / b;
      }
    }
    int kk = 0;
    if (ok) {
      const double ie = ds->inv_exp_factor;
      const double nu = 1.0 / fabs(s0);
      const double cw = HAS_PREV ? (b * ie) * (b * ie) : 0.0;
      const double nprev = HAS_PREV ? 1.0 / fabs(ds->s[j - 1]) : 0.0;
      const double B = 2.0 * nu * (ldexp(1.0, 61 - msh) * nu + cw * nprev);
      if (B > 0.0 && B < 1e300) {
        int E;
        frexp(B, &E);  // B < 2^E
        kk = 124 - E;
      }
      if (blockIdx.x == 0) {
        if (HAS_PREV) {
          ds->beta[j] = b;
          ds->s[j] = s0;
        }
        ds->fx_ak[j] = kk;
      }
    }
    sh[0] = b;
    sh[1] = ok ? s0 : 0.0;
    sh[2] = (double)kk;
  }
  __syncthreads();
  bj = sh[0];
  sj = sh[1];
  k = (int)sh[2];
  return sj != 0.0;
}

// <u_j, w'> terms (re, im) added exactly to the pass's accumulator in units
// of 2^-k (one thread).
__device__ __forceinline__ void fix_alpha_add(TeDevState* ds, int j, int k, double re, double im) {
  unsigned long long lo, hi;
  te_fix_encode128(re, k, lo, hi);
  te_atomic_add128(&ds->fx_alpha[j][0], lo, hi);
  te_fix_encode128(im, k, lo, hi);
  te_atomic_add128(&ds->fx_alpha[j][2], lo, hi);
}

// End of a fixed-point apply pass: the block's <u_j, w'> sums into the exact
// accumulator and its max|w'| into fx_wmaxj[j].  No last-block reduction: the
// update pass finishes alpha_j, its coefficient and xs_{j+1} from them.
__device__ __forceinline__ void fix_apply_publish(double (&acc)[2], unsigned int wmax, TeDevState* ds, int j, int k,
                                                  double* wide, unsigned int* wmax_w) {
  te_warp_max_to_smem(wmax, wmax_w);
  te_block_sum_wide<2>(acc, wide);
  if (threadIdx.x == 0) {
    atomicMax(&ds->fx_wmaxj[j], te_block_max_from_smem(wmax_w));
    fix_alpha_add(ds, j, k, acc[0], acc[1]);
  }
}

// Folded three-term apply pass with the fixed-point SpMV (te_fixed.cuh):
// w' = -i H u_j + (beta_j / e)^2 u_{j-1}, alpha_j = s_j g <u_j, w'> as in
// lanczos_apply_kernel<REAL, HAS_PREV, FOLD = true, K = 1>, with H u_j of the
// chunk rows from the integer pipes (X = round(u_j 2^xs_j)); long rows stay
// FP64.  Also bounds the next vector: with W >= max|w'| (block maxima) and
// U >= max|u_j|, u'_{j+1} = w' - (alpha_j / e) u_j has components below
// B = W + (|Re| + |Im|)(alpha_j / e) U, which fixes xs_{j+1} for the update.
// Resident blocks per SM of the fixed-point apply kernel (40 registers).
// Measured on the L=12 Bose-Hubbard matrix (us per launch, with the slots per
// lane in flight of te_sell_row_fix): 4 blocks 113 (4 slots) / 128 (2 slots);
// 5 blocks 76; 6 blocks 72 (2 slots) / 117 (1 slot); 8 blocks 74.  The spill
// of the 6-block build (a few words outside the slot loop) costs less than
// the latency hiding it buys.
#ifndef TE_FIX_MIN_BLOCKS
#define TE_FIX_MIN_BLOCKS 6
#endif
// The matrix side of the fixed-point apply, by format FMT: 0 real limbs per
// slot (col, hv), 1 real packed slots with a value table (pk, table, nvals,
// cbits), 2 complex limbs per slot (col, hv4).
struct TeFixMatrix {
  const int32_t* col;
  const int2* hv;
  const int4* hv4;
  const uint32_t* pk;
  const int2* table;
  int nvals, cbits, sh;
};

template <bool HAS_PREV, int FMT, bool LONG = true>  // LONG: as for lanczos_apply_kernel
__global__ void __launch_bounds__(TE_THREADS, TE_FIX_MIN_BLOCKS) lanczos_apply_fix_kernel(
    int64_t n, const int32_t* __restrict__ warp_chunk, const int64_t* __restrict__ chunk_off, TeFixMatrix M,
    TeLongRows L, const int4* __restrict__ X, const double2* __restrict__ u_j, const double2* __restrict__ u_jm1,
    double2* __restrict__ w, TeDevState* ds, double* partials, int j) {
  __shared__ double scratch[2 * 32];
  __shared__ double wide[2 * TE_THREADS];
  __shared__ unsigned int wmax_w[TE_THREADS / 32];
  extern __shared__ int2 tab[];  // FMT 1: the value table (constant across launches)
  if (FMT == 1) {
    for (int i = threadIdx.x; i < M.nvals; i += blockDim.x) tab[i] = M.table[i];
    __syncthreads();
  }
  te_pdl_trigger();
  te_pdl_wait();
  if (te_step_inactive(ds)) return;
  const int lane = threadIdx.x & 31;
  double sj, bj;
  int ak;
  if (!fix_apply_prologue<HAS_PREV>(ds, j, M.sh, scratch, sj, bj, ak)) return;
  const double g = ds->exp_factor * sj;
  const double ie = ds->inv_exp_factor;
  double cw = 0.0;
  if (HAS_PREV) cw = (bj * ie) * (bj * ie);
  const int shift = M.sh + ds->fx_xs[j];
  double acc[2] = {0.0, 0.0};
  unsigned int wmax = 0;
  const int64_t wid = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t sg = wid; LONG && sg < L.n_seg; sg += warps) {  // long rows: merge-path segments, FP64
    int64_t lr;
    double2 y;
    const int done = te_long_segment<FMT != 2>(L, sg, u_j, lane, &lr, &y);
    if (done && lane == 0) {
      // a split row's terms go to the exact accumulator on their own, so that
      // no block's FP64 sum depends on which warp completed the row
      double a2[2] = {0.0, 0.0};
      const double2 wr = apply_row_epilogue<HAS_PREV, true>(lr, y, g, cw, u_j, u_jm1, w, done == 1 ? acc : a2);
      if (done == 2) fix_alpha_add(ds, j, ak, a2[0], a2[1]);
      wmax = max(wmax, max(te_fix_hiword(wr.x), te_fix_hiword(wr.y)));
    }
  }
  // the warp's chunk offsets in one coalesced load (lane k holds the offset
  // of chunk c_begin + k) when its range has at most 31 chunks.  Chunk and
  // row counters are 32-bit (rows < 2^31), and a row is live when r - L.n is
  // below n - L.n as unsigned: fewer registers across the slot loop
  const int c_begin = warp_chunk[wid], c_end = warp_chunk[wid + 1];
  const bool offs_in_regs = c_end - c_begin <= 31;
  const int64_t my_off = (offs_in_regs && c_begin + lane <= c_end) ? __ldg(chunk_off + c_begin + lane) : 0;
  const uint32_t live_lo = (uint32_t)L.n, live_cnt = (uint32_t)(n - L.n);
  for (int c = c_begin; c < c_end; ++c) {
    const int k = c - c_begin;
    int64_t s0, s1;
    if (offs_in_regs) {
      s0 = __shfl_sync(0xffffffffu, my_off, k);
      s1 = __shfl_sync(0xffffffffu, my_off, k + 1);
    } else {
      s0 = __ldg(chunk_off + c);
      s1 = __ldg(chunk_off + c + 1);
    }
    const int64_t r = (int64_t)c * 32 + lane;
    const bool live = (uint32_t)r - live_lo < live_cnt;
    const double2 y = FMT == 1   ? te_sell_row_fix_packed(s0 + lane, s1, M.pk, tab, M.cbits, X, shift)
                      : FMT == 2 ? te_sell_row_fix_c(s0 + lane, s1, M.col, M.hv4, X, shift)
                                 : te_sell_row_fix(s0 + lane, s1, M.col, M.hv, X, shift);
    if (live) {
      const double2 wr = apply_row_epilogue<HAS_PREV, true>(r, y, g, cw, u_j, u_jm1, w, acc);
      wmax = max(wmax, max(te_fix_hiword(wr.x), te_fix_hiword(wr.y)));
    }
  }
  fix_apply_publish(acc, wmax, ds, j, (int)scratch[2], wide, wmax_w);  // k from the prologue's broadcast
}

// One column block of the fixed-point SpMV: for block row i (main row
// row[i]) the exact int64 sums S over the block's entries are added into
// acc[row[i]] (written when first != 0; block 0 covers every row).
template <bool REAL>
__global__ void __launch_bounds__(TE_THREADS, TE_FIX_MIN_BLOCKS) fix_block_kernel(
    int64_t n_rows, const int32_t* __restrict__ warp_chunk, const int64_t* __restrict__ chunk_off,
    const int32_t* __restrict__ row, const int32_t* __restrict__ col, const int2* __restrict__ hv,
    const int4* __restrict__ hv4, const int4* __restrict__ X, longlong2* __restrict__ acc, int first,
    const TeDevState* ds) {
  te_pdl_trigger();
  te_pdl_wait();
  if (te_step_inactive(ds)) return;
  const int lane = threadIdx.x & 31;
  const int64_t wid = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int64_t c_begin = warp_chunk[wid], c_end = warp_chunk[wid + 1];
  for (int64_t c = c_begin; c < c_end; ++c) {
    const int64_t s0 = __ldg(chunk_off + c), s1 = __ldg(chunk_off + c + 1);
    longlong2 S = REAL ? te_sell_row_fix_sum<kTeFixBlockUnroll>(s0 + lane, s1, col, hv, X)
                       : te_sell_row_fix_c_sum<kTeFixBlockUnroll>(s0 + lane, s1, col, hv4, X);
    const int64_t i = c * 32 + lane;
    if (i < n_rows) {
      const int32_t r = __ldg(row + i);
      if (!first) {
        const longlong2 a = acc[r];
        S.x += a.x;
        S.y += a.y;
      }
      acc[r] = S;
    }
  }
}

// Epilogue pass of the column-blocked apply: y from the accumulated sums,
// then as lanczos_apply_fix_kernel (w', <u_j, w'>, max|w'|, alpha_j, xs_{j+1}).
template <bool HAS_PREV>
__global__ void __launch_bounds__(TE_THREADS) fix_epilogue_kernel(int64_t n, const longlong2* __restrict__ acc_in,
                                                                  int sh, const double2* __restrict__ u_j,
                                                                  const double2* __restrict__ u_jm1,
                                                                  double2* __restrict__ w, TeDevState* ds,
                                                                  double* partials, int j) {
  __shared__ double scratch[2 * 32];
  __shared__ double wide[2 * TE_THREADS];
  __shared__ unsigned int wmax_w[TE_THREADS / 32];
  te_pdl_trigger();
  te_pdl_wait();
  if (te_step_inactive(ds)) return;
  double sj, bj;
  int ak;
  if (!fix_apply_prologue<HAS_PREV>(ds, j, sh, scratch, sj, bj, ak)) return;
  const double g = ds->exp_factor * sj;
  const double ie = ds->inv_exp_factor;
  double cw = 0.0;
  if (HAS_PREV) cw = (bj * ie) * (bj * ie);
  const int shift = sh + ds->fx_xs[j];
  double acc[2] = {0.0, 0.0};
  unsigned int wmax = 0;
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
    const double2 wr = apply_row_epilogue<HAS_PREV, true>(r, te_fix_to_double(acc_in[r], shift), g, cw, u_j, u_jm1, w,
                                                          acc);
    wmax = max(wmax, max(te_fix_hiword(wr.x), te_fix_hiword(wr.y)));
  }
  fix_apply_publish(acc, wmax, ds, j, ak, wide, wmax_w);
}

// Start of a Krylov step on the fixed-point path, two passes over u_0:
// per-block maxima of |u_0| (high words) into partials, then every block of
// the encode pass reduces those maxima itself (same value everywhere), sets
// xs_0 and writes X = round(u_0 2^xs_0); block 0 records xs_0 and the bound.
__global__ void __launch_bounds__(TE_THREADS) fix_start_max_kernel(int64_t n, const double2* __restrict__ u,
                                                                   const TeDevState* ds, unsigned int* bmax) {
  __shared__ unsigned int slots[TE_THREADS / 32];
  if (ds->fatal != 0 || ds->done != 0) return;
  unsigned int m = 0;
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
    const double2 v = u[r];
    m = max(m, max(te_fix_hiword(v.x), te_fix_hiword(v.y)));
  }
  te_warp_max_to_smem(m, slots);
  __syncthreads();
  if (threadIdx.x == 0) bmax[blockIdx.x] = te_block_max_from_smem(slots);
}

__global__ void __launch_bounds__(TE_THREADS) fix_start_encode_kernel(int64_t n, const double2* __restrict__ u,
                                                                      int4* __restrict__ X, TeDevState* ds,
                                                                      const unsigned int* __restrict__ bmax,
                                                                      int n_bmax) {
  __shared__ unsigned int slots[TE_THREADS / 32];
  __shared__ int xs_s;
  if (ds->fatal != 0 || ds->done != 0) return;
  unsigned int m = 0;
  for (int i = threadIdx.x; i < n_bmax; i += blockDim.x) m = max(m, bmax[i]);
  te_warp_max_to_smem(m, slots);
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned int um = te_block_max_from_smem(slots);
    xs_s = te_fix_scale(te_fix_upper(um));
    if (blockIdx.x == 0) {
      ds->fx_xs[0] = xs_s;
      ds->fx_umax[0] = um;
      ds->fx_wmax = 0u;
    }
  }
  if (blockIdx.x == 0) {  // the exact accumulators of this Krylov step's passes
    for (int i = threadIdx.x; i < TE_MMAX; i += blockDim.x) {
      ds->fx_alpha[i][0] = ds->fx_alpha[i][1] = ds->fx_alpha[i][2] = ds->fx_alpha[i][3] = 0ull;
      ds->fx_wmaxj[i] = 0u;
      ds->fx_nrm[i + 1][0] = ds->fx_nrm[i + 1][1] = 0ull;
      ds->fx_umax[i + 1] = 0u;
    }
  }
  __syncthreads();
  const int xs = xs_s;
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
    const double2 v = u[r];
    const int2 a = te_fix_split(te_fix_encode(v.x, xs)), b = te_fix_split(te_fix_encode(v.y, xs));
    X[r] = make_int4(a.x, a.y, b.x, b.y);
  }
}

// u_{j+1} = w - alpha_j v_j and beta_{j+1} = ||u_{j+1}||.  With a folded w'
// (fold != 0) the kernel forms u'_{j+1} = w' - (alpha_j s_j / g) u_j = u_{j+1} / g
// and keeps the factor in the scale: beta_{j+1} = |g| ||u'||, s_{j+1} = g / beta_{j+1}.
// FIX: also writes X = round(u'_{j+1} 2^xs_{j+1}) (the fixed-point copy read
// by the next apply pass) and folds max |u'_{j+1}| into fx_umax[j + 1].
// ACC (fixed-point path): alpha_j = s_j g <u_j, w'> from the apply pass's
// exact accumulator, its coefficient alpha_j / e and xs_{j+1} from
// B = (W + (|Re| + |Im|)(alpha_j / e) U)(1 + 1e-12) (W >= max|w'|, U >=
// max|u_j|), computed by thread 0 of every block; block 0 records them.
template <bool STORE, bool FIX, bool ACC>
__global__ void __launch_bounds__(TE_THREADS) lanczos_update_kernel(int64_t n, const double2* __restrict__ w,
                                                                    const double2* __restrict__ u_j,
                                                                    double2* __restrict__ u_jp1, TeDevState* ds,
                                                                    double* partials, int j, int fold,
                                                                    int4* __restrict__ X) {
  __shared__ double scratch[32];
  __shared__ double wide[TE_THREADS];
  __shared__ unsigned int umax_w[TE_THREADS / 32];
  te_pdl_trigger();
  te_pdl_wait();
  if (te_step_inactive(ds)) return;
  double gr, gi;  // alpha_j s_j / g
  int xs;
  if (ACC) {
    if (threadIdx.x == 0) {
      const int k = ds->fx_ak[j];
      const double re = te_i128_to_double(ds->fx_alpha[j][0], ds->fx_alpha[j][1], -k);
      const double im = te_i128_to_double(ds->fx_alpha[j][2], ds->fx_alpha[j][3], -k);
      const double sj = ds->s[j];
      const double f = sj * (ds->exp_factor * sj);
      const double ie = ds->inv_exp_factor;
      const double2 alpha = make_double2(f * re, f * im);
      const double W = te_fix_upper(ds->fx_wmaxj[j]);
      const double U = te_fix_upper(ds->fx_umax[j]);
      const double B = (W + (fabs(alpha.x * ie) + fabs(alpha.y * ie)) * U) * (1.0 + 1e-12);
      const int x = te_fix_scale(B);
      // beyond the scale's range (or not finite): no coefficients rather than wrong ones
      const double one = B < 1e300 ? 1.0 : __longlong_as_double(0x7ff8000000000000ll);
      scratch[0] = alpha.x * ie;
      scratch[1] = alpha.y * ie;
      scratch[2] = (double)x;
      if (blockIdx.x == 0) {
        ds->alpha[j] = make_double2(one * alpha.x, one * alpha.y);
        ds->upd_gr = alpha.x * ie;
        ds->upd_gi = alpha.y * ie;
        ds->fx_xs[j + 1] = x;
      }
    }
    __syncthreads();
    gr = scratch[0];
    gi = scratch[1];
    xs = FIX ? (int)scratch[2] : 0;
    __syncthreads();
  } else {
    gr = ds->upd_gr;
    gi = ds->upd_gi;
    xs = FIX ? ds->fx_xs[j + 1] : 0;
  }
  double acc[1] = {0.0};
  unsigned int umax = 0;
  unsigned long long sq_lo = 0, sq_hi = 0;  // FIX: sum |X|^2 / 2^62 in 128 bits
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
    double2 wv = w[r];
    double2 u = u_j[r];
    double2 o;
    o.x = fma(-gr, u.x, fma(gi, u.y, wv.x));
    o.y = fma(-gr, u.y, fma(-gi, u.x, wv.y));
    if (STORE) u_jp1[r] = o;
    if (FIX) {
      const int64_t er = te_fix_encode(o.x, xs), ei = te_fix_encode(o.y, xs);
      const int2 p = te_fix_split(er), q2 = te_fix_split(ei);
      X[r] = make_int4(p.x, p.y, q2.x, q2.y);
      umax = max(umax, max(te_fix_hiword(o.x), te_fix_hiword(o.y)));
      // ||u'||^2 from the integer copy, off the FP64 pipe
      const unsigned long long sq = te_fix_sq(er) + te_fix_sq(ei);
      asm("add.cc.u64 %0, %0, %2;\n\taddc.u64 %1, %1, 0;" : "+l"(sq_lo), "+l"(sq_hi) : "l"(sq));
    } else {
      acc[0] = fma(o.x, o.x, fma(o.y, o.y, acc[0]));
    }
  }
  if (FIX) {
    // ||u'||^2 exactly: 128-bit sums per warp and block, then two atomics into
    // fx_nrm[j + 1]; the next apply pass takes beta_{j+1} from it (no
    // last-block reduction, and the total does not depend on the order)
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long l2 = __shfl_xor_sync(0xffffffffu, sq_lo, o);
      const unsigned long long h2 = __shfl_xor_sync(0xffffffffu, sq_hi, o);
      sq_lo += l2;
      sq_hi += h2 + (sq_lo < l2 ? 1ull : 0ull);
    }
    te_warp_max_to_smem(umax, umax_w);
    unsigned long long* wsum = reinterpret_cast<unsigned long long*>(wide);  // 2 words per warp
    if ((threadIdx.x & 31) == 0) {
      wsum[2 * (threadIdx.x >> 5)] = sq_lo;
      wsum[2 * (threadIdx.x >> 5) + 1] = sq_hi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned long long lo = 0, hi = 0;
      for (int k = 0; k < (int)(blockDim.x >> 5); ++k) {
        lo += wsum[2 * k];
        hi += wsum[2 * k + 1] + (lo < wsum[2 * k] ? 1ull : 0ull);
      }
      const unsigned long long old = atomicAdd(&ds->fx_nrm[j + 1][0], lo);
      atomicAdd(&ds->fx_nrm[j + 1][1], hi + (old + lo < old ? 1ull : 0ull));
      atomicMax(&ds->fx_umax[j + 1], te_block_max_from_smem(umax_w));
    }
    return;
  }
  te_block_sum_wide<1>(acc, wide);
  if (te_publish_partials<1>(acc, partials, &ds->counter[1])) {
    double tot[1];
    te_final_sum<1>(tot, partials, &ds->counter[1], scratch);
    if (threadIdx.x == 0) {
      const double g = fold ? ds->exp_factor * ds->s[j] : 1.0;
      const double beta = fabs(g) * sqrt(tot[0]);
      const int m = ds->m_cur;
      if (beta < ds->tol_rate) {  // lucky breakdown (:551-555)
        ds->breakdown = 1;
        ds->m_eff = j + 1;
        ds->h = beta;
      } else if (j + 1 != m) {
        ds->beta[j + 1] = beta;
        ds->s[j + 1] = g / beta;
      } else {
        ds->h = beta;
        ds->m_eff = m;
      }
    }
  }
}

// --------------------------------------------------------------------------
// Reorthogonalising mode: classical Gram-Schmidt with one reorthogonalisation
// pass (CGS2) against all previous basis vectors.  Iteration j, after
// w = A v_j (apply kernel without the three-term term):
//   project:          p1_i = <v_i, w>                         i = 0..j
//   update + project: w' = w - sum_i p1_i v_i,  p2_i = <v_i, w'>
//   update + norm:    u_{j+1} = w' - sum_i p2_i v_i, beta_{j+1} = ||u_{j+1}||
// alpha_j = p1_j + p2_j; the tridiagonal Krylov matrix keeps alpha and beta
// (the remaining projections vanish up to rounding for an anti-Hermitian A).
// A block owns TE_GS_ROWS consecutive rows and keeps its slice of w in shared
// memory; each warp accumulates the projections of its share of the basis
// vectors over the block's rows (coalesced reads of every u_i).

__device__ __forceinline__ int gs_row_begin(int64_t n) {
  return (int)min((int64_t)blockIdx.x * TE_GS_ROWS, n);
}

// Per-warp projections <u_i, w_s> over the block's rows, i = warp, warp + 8, ...;
// partial sums (re, im) of vector i go to partials[(2 i + c) * gridDim.x + block].
__device__ void gs_block_projections(int rows, int64_t r0, const double2* const* u_s, int nvec,
                                     const double2* w_s, double* partials) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int i = warp; i < nvec; i += nw) {
    const double2* __restrict__ u = u_s[i] + r0;
    double re = 0.0, im = 0.0;
    for (int r = lane; r < rows; r += 32) {
      const double2 a = u[r], b = w_s[r];
      re = fma(a.x, b.x, fma(a.y, b.y, re));
      im = fma(a.x, b.y, fma(-a.y, b.x, im));
    }
    re = te_warp_sum(re);
    im = te_warp_sum(im);
    if (lane == 0) {
      partials[(2 * i) * gridDim.x + blockIdx.x] = re;
      partials[(2 * i + 1) * gridDim.x + blockIdx.x] = im;
      __threadfence();
    }
  }
}

// Last block: proj[i] = s_i * sum over blocks (fixed order), i < nvec.
__device__ void gs_finish(int nvec, const double* partials, double2* proj, const TeDevState* ds) {
  __shared__ double red[2][TE_MMAX];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int v = warp; v < 2 * nvec; v += nw) {
    double s = 0.0;
    for (int b = lane; b < (int)gridDim.x; b += 32) s += __ldcg(partials + (int64_t)v * gridDim.x + b);
    s = te_warp_sum(s);
    if (lane == 0) red[v & 1][v >> 1] = s;
  }
  __syncthreads();
  if ((int)threadIdx.x < nvec) {
    const double si = ds->s[threadIdx.x];
    proj[threadIdx.x] = make_double2(si * red[0][threadIdx.x], si * red[1][threadIdx.x]);
  }
}

__device__ __forceinline__ bool gs_last_block(unsigned int* counter) {
  __shared__ bool is_last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    is_last = (atomicAdd(counter, 1u) == gridDim.x - 1);
  }
  __syncthreads();
  if (is_last) __threadfence();
  return is_last;
}

__global__ void __launch_bounds__(TE_THREADS) gs_project_kernel(int64_t n, TeBasisPtrs V, int nvec,
                                                                const double2* __restrict__ w, TeDevState* ds,
                                                                double* partials) {
  __shared__ double2 w_s[TE_GS_ROWS];
  __shared__ const double2* u_s[TE_MMAX];
  if (te_step_inactive(ds)) return;
  if ((int)threadIdx.x < nvec) u_s[threadIdx.x] = V.u[threadIdx.x];
  const int64_t r0 = gs_row_begin(n);
  const int rows = (int)min((int64_t)TE_GS_ROWS, n - r0);
  for (int r = threadIdx.x; r < rows; r += blockDim.x) w_s[r] = w[r0 + r];
  __syncthreads();
  gs_block_projections(rows, r0, u_s, nvec, w_s, partials);
  if (gs_last_block(&ds->counter[0])) {
    gs_finish(nvec, partials, ds->proj1, ds);
    if (threadIdx.x == 0) ds->counter[0] = 0u;
  }
}

__global__ void __launch_bounds__(TE_THREADS) gs_update_project_kernel(int64_t n, TeBasisPtrs V, int nvec,
                                                                       double2* __restrict__ w, TeDevState* ds,
                                                                       double* partials) {
  __shared__ double2 w_s[TE_GS_ROWS];
  __shared__ double2 c_s[TE_MMAX];
  __shared__ const double2* u_s[TE_MMAX];
  if (te_step_inactive(ds)) return;
  if ((int)threadIdx.x < nvec) {
    const double si = ds->s[threadIdx.x];
    const double2 p = ds->proj1[threadIdx.x];
    c_s[threadIdx.x] = make_double2(p.x * si, p.y * si);  // w -= p1_i v_i = (p1_i s_i) u_i
    u_s[threadIdx.x] = V.u[threadIdx.x];
  }
  __syncthreads();
  const int64_t r0 = gs_row_begin(n);
  const int rows = (int)min((int64_t)TE_GS_ROWS, n - r0);
  for (int r = threadIdx.x; r < rows; r += blockDim.x) {
    double2 x = w[r0 + r];
    for (int i = 0; i < nvec; ++i) {
      const double2 u = u_s[i][r0 + r], c = c_s[i];
      x.x = fma(-c.x, u.x, fma(c.y, u.y, x.x));
      x.y = fma(-c.x, u.y, fma(-c.y, u.x, x.y));
    }
    w_s[r] = x;
    w[r0 + r] = x;
  }
  __syncthreads();
  gs_block_projections(rows, r0, u_s, nvec, w_s, partials);
  if (gs_last_block(&ds->counter[0])) {
    gs_finish(nvec, partials, ds->proj2, ds);
    if (threadIdx.x == 0) ds->counter[0] = 0u;
  }
}

__global__ void __launch_bounds__(TE_THREADS) gs_update_norm_kernel(int64_t n, TeBasisPtrs V, int nvec,
                                                                    const double2* __restrict__ w,
                                                                    double2* __restrict__ u_next, TeDevState* ds,
                                                                    double* partials, int j) {
  __shared__ double2 c_s[TE_MMAX];
  __shared__ const double2* u_s[TE_MMAX];
  __shared__ double scratch[32];
  if (te_step_inactive(ds)) return;
  if ((int)threadIdx.x < nvec) {
    const double si = ds->s[threadIdx.x];
    const double2 p = ds->proj2[threadIdx.x];
    c_s[threadIdx.x] = make_double2(p.x * si, p.y * si);
    u_s[threadIdx.x] = V.u[threadIdx.x];
  }
  __syncthreads();
  double acc[1] = {0.0};
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
    double2 x = w[r];
    for (int i = 0; i < nvec; ++i) {
      const double2 u = u_s[i][r], c = c_s[i];
      x.x = fma(-c.x, u.x, fma(c.y, u.y, x.x));
      x.y = fma(-c.x, u.y, fma(-c.y, u.x, x.y));
    }
    if (u_next) u_next[r] = x;
    acc[0] = fma(x.x, x.x, fma(x.y, x.y, acc[0]));
  }
  te_block_sum<1>(acc, scratch);
  if (te_publish_partials<1>(acc, partials, &ds->counter[1])) {
    double tot[1];
    te_final_sum<1>(tot, partials, &ds->counter[1], scratch);
    if (threadIdx.x == 0) {
      const double2 a1 = ds->proj1[j], a2 = ds->proj2[j];
      ds->alpha[j] = make_double2(a1.x + a2.x, a1.y + a2.y);
      const double beta = sqrt(tot[0]);
      const int m = ds->m_cur;
      if (beta < ds->tol_rate) {
        ds->breakdown = 1;
        ds->m_eff = j + 1;
        ds->h = beta;
      } else if (j + 1 != m) {
        ds->beta[j + 1] = beta;
        ds->s[j + 1] = 1.0 / beta;
      } else {
        ds->h = beta;
        ds->m_eff = m;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// The same three passes for dimensions that give TE_GS_ROWS-row blocks to fewer
// than every SM (n < 311 296 on 152 SMs), one block per SM at most.
//  * Both phases are bound by FP64 issue (64 cycles per warp instruction and
//    scheduler), so a block's 8 warps share its chunks and, while it has fewer
//    than 8, the basis vectors too (update).  A projection gives a lane one
//    component of one <u_i, w> and walks the rows: no shuffle trees, which
//    would cost more than the products on so few rows.
//  * The projections are summed exactly, as 128-bit integers added atomically
//    (units from ||u_i|| = 1 / s_i and ||w|| <= |e| ||H||, 24 bits to spare; for
//    u_0 from its norm): no block sums another's partials, and the total does
//    not depend on the order.  The next pass converts them.
// Measured on GB300, dim 12 870, per iteration: project 71 -> 13 us, update and
// project 113 -> 15 us, update and norm 16 us as before.
struct TeGsSmall {
  int64_t n;
  int chunks;  // of 32 rows per block
  int r_exp;   // ||H|| < 2^r_exp
  unsigned long long* acc1;  // [2 i + c][2]: sums of the first projection, zero before it
  unsigned long long* acc2;  // of the second
  unsigned long long* bad;   // non-zero when a sum was not finite
};

// units 2^-k of <u_i, w> in iteration j
__device__ __forceinline__ int gs_units(const TeGsSmall& a, const TeDevState* ds, int i, int j) {
  auto ex = [](double v) { return (int)((te_fix_hiword(v) >> 20) & 0x7ffu) - 1022; };  // |v| < 2^ex
  const int e0 = (ex(ds->norm2_final) + 2) / 2;  // ||u_0|| < 2^e0 (set at the start of the step)
  const int eu = i == 0 ? e0 : 2 - ex(ds->s[i]);
  return 101 - (eu + a.r_exp + ex(ds->exp_factor) + (j == 0 ? e0 : 0));
}

// MODE 0: acc1 += <u_i, w>; 1: w -= sum p1_i v_i, acc2 += <u_i, w>;
// 2: u_next = w - sum p2_i v_i, its norm, alpha_j, beta_{j+1}, s_{j+1}.
template <int MODE>
__global__ void __launch_bounds__(TE_THREADS) gs_small_kernel(TeGsSmall a, TeBasisPtrs V, int nvec,
                                                              double2* __restrict__ w, double2* __restrict__ u_next,
                                                              TeDevState* ds, double* partials, int j) {
  constexpr int kWarps = TE_THREADS / 32;
  __shared__ double2 w_s[TE_GS_ROWS];
  __shared__ double2 part[TE_THREADS];
  __shared__ double2 c_s[TE_MMAX];
  __shared__ const double2* u_s[TE_MMAX];
  __shared__ double scratch[32];
  if (te_step_inactive(ds)) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if ((int)threadIdx.x < nvec) {
    const int i = threadIdx.x;
    u_s[i] = V.u[i];
    if (MODE > 0) {  // w -= p_i v_i = (s_i <u_i, w>) s_i u_i
      const unsigned long long* q = (MODE == 1 ? a.acc1 : a.acc2) + 4 * i;
      const int k = gs_units(a, ds, i, j);
      const double si = ds->s[i], s2 = si * si;
      c_s[i] = make_double2(s2 * te_i128_to_double(__ldcg(q), __ldcg(q + 1), -k),
                            s2 * te_i128_to_double(__ldcg(q + 2), __ldcg(q + 3), -k));
      if (__ldcg(a.bad)) c_s[i].x = c_s[i].y = __longlong_as_double(0x7ff8000000000000ll);
    }
  }
  const int64_t r0 = blockIdx.x * (int64_t)a.chunks * 32;
  const int rows = (int)min((int64_t)a.chunks * 32, a.n - r0);
  __syncthreads();
  // update: chunks over the warps, the vectors split g ways between them
  const int cc = min(a.chunks, kWarps), g = MODE > 0 ? kWarps / cc : 1, split = warp / cc;
  double acc[1] = {0.0};
  for (int ch = warp % cc; ch < a.chunks; ch += cc) {
    const int r = ch * 32 + lane;
    const bool live = r < rows && split < g;
    double2 x = make_double2(0.0, 0.0);
    if (live && split == 0) x = w[r0 + r];
    if (MODE > 0 && live) {
#pragma unroll 4
      for (int i = split; i < nvec; i += g) {
        const double2 u = u_s[i][r0 + r], c = c_s[i];
        x.x = fma(-c.x, u.x, fma(c.y, u.y, x.x));
        x.y = fma(-c.x, u.y, fma(-c.y, u.x, x.y));
      }
    }
    if (g > 1) {  // one chunk per warp: the shares of its vectors
      part[threadIdx.x] = x;
      __syncthreads();
      if (split == 0)
        for (int q = 1; q < g; ++q) {
          const double2 y = part[(q * cc + ch) * 32 + lane];
          x.x += y.x;
          x.y += y.y;
        }
    }
    if (live && split == 0) {
      w_s[r] = x;
      if (MODE == 1) w[r0 + r] = x;
      if (MODE == 2 && u_next) u_next[r0 + r] = x;
      if (MODE == 2) acc[0] = fma(x.x, x.x, fma(x.y, x.y, acc[0]));
    }
  }
  __syncthreads();
  if (MODE < 2) {
    // project: lane = (vector, component) of a group of 16 vectors, the rows
    // split between the warps of a group
    const int groups = (nvec + 15) / 16, share = kWarps / groups, gi = warp % groups, sh = warp / groups;
    const int i = gi * 16 + (lane >> 1), c = lane & 1;
    double d = 0.0;
    if (sh < share && i < nvec) {
      const double2* __restrict__ u = u_s[i] + r0;
      const int b = rows * sh / share, e = rows * (sh + 1) / share;
      // c = 0: Re conj(u) w = u.x w.x + u.y w.y; c = 1: Im = u.x w.y - u.y w.x
#pragma unroll 8
      for (int r = b; r < e; ++r) {
        const double2 q = u[r], x = w_s[r];
        d = fma(q.x, c ? x.y : x.x, fma(c ? -q.y : q.y, c ? x.x : x.y, d));
      }
    }
    double* sums = reinterpret_cast<double*>(part);
    sums[threadIdx.x] = d;
    __syncthreads();
    if (warp < groups && i < nvec) {
      for (int q = 1; q < share; ++q) d += sums[(q * groups + gi) * 32 + lane];
      unsigned long long lo, hi;
      te_fix_encode128(d, gs_units(a, ds, i, j), lo, hi);
      if (te_fix_hiword(d) >= 0x7ff00000u) {
        atomicExch(a.bad, 1ull);
        lo = hi = 0ull;
      }
      te_atomic_add128((MODE == 0 ? a.acc1 : a.acc2) + 4 * i + 2 * c, lo, hi);
    }
    return;
  }
  te_block_sum<1>(acc, scratch);
  if (te_publish_partials<1>(acc, partials, &ds->counter[1])) {
    double tot[1];
    te_final_sum<1>(tot, partials, &ds->counter[1], scratch);
    if (threadIdx.x == 0) {
      // alpha_j = s_j (<u_j, w> + <u_j, w'>), the sums in their integer form
      const unsigned long long *p = a.acc1 + 4 * j, *q = a.acc2 + 4 * j;
      const int k = gs_units(a, ds, j, j);
      const double sj = ds->s[j];
      const double re = sj * te_i128_to_double(__ldcg(p), __ldcg(p + 1), -k),
                   im = sj * te_i128_to_double(__ldcg(p + 2), __ldcg(p + 3), -k);
      ds->alpha[j] = make_double2(re + sj * te_i128_to_double(__ldcg(q), __ldcg(q + 1), -k),
                                  im + sj * te_i128_to_double(__ldcg(q + 2), __ldcg(q + 3), -k));
      const double beta = sqrt(tot[0]);
      const int m = ds->m_cur;
      if (beta < ds->tol_rate) {
        ds->breakdown = 1;
        ds->m_eff = j + 1;
        ds->h = beta;
      } else if (j + 1 != m) {
        ds->beta[j + 1] = beta;
        ds->s[j + 1] = 1.0 / beta;
      } else {
        ds->h = beta;
        ds->m_eff = m;
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 4 * TE_MMAX; i += blockDim.x) a.acc1[i] = a.acc2[i] = 0ull;
  }
}

bool te_launch_gs_small(int64_t n, const TeBasisPtrs& V, int nvec, double2* w, double2* u_next, TeDevState* ds,
                        double* partials, unsigned long long* acc, double norm1, int j, cudaStream_t st) {
  const int64_t chunks = (n + 31) / 32;
  if (n >= (int64_t)TE_GS_ROWS * te_num_sms()) return false;
  TeGsSmall a;
  a.n = n;
  a.chunks = (int)((chunks + te_num_sms() - 1) / te_num_sms());
  const int grid = (int)((chunks + a.chunks - 1) / a.chunks);
  std::frexp(norm1 > 0.0 && norm1 < 1e300 ? norm1 : 1.0, &a.r_exp);
  a.acc1 = acc;
  a.acc2 = acc + 4 * TE_MMAX;
  a.bad = acc + 8 * TE_MMAX;
  gs_small_kernel<0><<<grid, TE_THREADS, 0, st>>>(a, V, nvec, w, nullptr, ds, partials, j);
  gs_small_kernel<1><<<grid, TE_THREADS, 0, st>>>(a, V, nvec, w, nullptr, ds, partials, j);
  gs_small_kernel<2><<<grid, TE_THREADS, 0, st>>>(a, V, nvec, w, u_next, ds, partials, j);
  return true;
}

static int gs_grid(int64_t n) { return (int)std::max<int64_t>(1, (n + TE_GS_ROWS - 1) / TE_GS_ROWS); }

void te_launch_gs_project(int64_t n, const TeBasisPtrs& V, int nvec, const double2* w, TeDevState* ds,
                          double* partials, cudaStream_t st) {
  gs_project_kernel<<<gs_grid(n), TE_THREADS, 0, st>>>(n, V, nvec, w, ds, partials);
}

void te_launch_gs_update_project(int64_t n, const TeBasisPtrs& V, int nvec, double2* w, TeDevState* ds,
                                 double* partials, cudaStream_t st) {
  gs_update_project_kernel<<<gs_grid(n), TE_THREADS, 0, st>>>(n, V, nvec, w, ds, partials);
}

void te_launch_gs_update_norm(int64_t n, const TeBasisPtrs& V, int nvec, const double2* w, double2* u_next,
                              TeDevState* ds, double* partials, int j, cudaStream_t st) {
  gs_update_norm_kernel<<<te_grid_for(n, TE_THREADS, 8), TE_THREADS, 0, st>>>(n, V, nvec, w, u_next, ds, partials,
                                                                                j);
}

namespace {

using ApplyKernel = void (*)(int64_t, int64_t, const int32_t*, const int64_t*, const int32_t*, const double*,
                             TeLongRows, const double2*, const double2*, double2*, TeDevState*, double*, int);

template <int K, bool LONG>
ApplyKernel apply_kernel_for(bool is_real, bool has_prev, bool fold) {
  static const ApplyKernel table[2][2][2] = {
      {{lanczos_apply_kernel<false, false, false, K, LONG>, lanczos_apply_kernel<false, false, true, K, LONG>},
       {lanczos_apply_kernel<false, true, false, K, LONG>, lanczos_apply_kernel<false, true, true, K, LONG>}},
      {{lanczos_apply_kernel<true, false, false, K, LONG>, lanczos_apply_kernel<true, false, true, K, LONG>},
       {lanczos_apply_kernel<true, true, false, K, LONG>, lanczos_apply_kernel<true, true, true, K, LONG>}}};
  return table[is_real ? 1 : 0][has_prev ? 1 : 0][fold ? 1 : 0];
}

// K > 1 never has long rows (te_matrix_set_spmv_lanes refuses them).
ApplyKernel apply_kernel(int lanes, bool is_real, bool has_prev, bool fold, bool has_long = true) {
  switch (lanes) {
    case 2: return apply_kernel_for<2, false>(is_real, has_prev, fold);
    case 4: return apply_kernel_for<4, false>(is_real, has_prev, fold);
    default:
      return has_long ? apply_kernel_for<1, true>(is_real, has_prev, fold)
                      : apply_kernel_for<1, false>(is_real, has_prev, fold);
  }
}

// Blocks of the apply kernel for K > 1: one warp per (chunk, part) unit, at
// most one resident wave.
int apply_grid_k(const TeSell& A, int lanes, ApplyKernel k) {
  const int64_t units = A.n_chunks * lanes;
  const int64_t cap = (int64_t)te_num_sms() * te_kernel_blocks_per_sm((const void*)k, TE_THREADS, 0);
  return (int)std::max<int64_t>(1, std::min<int64_t>((units + 7) / 8, cap));
}

}  // namespace

int te_sell_blocks_per_sm(bool is_real) {
  int b = 8;
  for (int hp = 0; hp < 2; ++hp)
    for (int f = 0; f < 2; ++f)
      b = std::min(b, te_kernel_blocks_per_sm((const void*)apply_kernel(1, is_real, hp, f), TE_THREADS, 0));
  return b;
}

void te_launch_lanczos_apply(const TeSell& A, bool is_real, const double2* u_j, const double2* u_jm1, double2* w,
                             TeDevState* ds, double* partials, int j, bool fold, cudaStream_t st,
                             const TeSegCarry* carry) {
  const int lanes = A.lanes;
  const ApplyKernel k = apply_kernel(lanes, is_real, u_jm1 != nullptr, fold, A.n_seg > 0);
  const int grid = lanes == 1 ? A.grid : apply_grid_k(A, lanes, k);
  te_launch_pdl(lanes == 1 && A.saturated, k, grid, TE_THREADS, st, A.n, A.n_chunks, A.warp_chunk, A.chunk_off,
                A.col, A.val, te_long_rows(A, carry), u_j, u_jm1, w, ds, partials, j);
}

// Lanes per row of the FP64 passes (the fixed-point passes always use one
// lane per row), chosen from the matrix's shape so that the same matrix always
// gets the same K -- K changes the rounding of the row sums.  Two lanes per
// row when the chunks are fewer than the resident warps (with one lane some
// warps would have no chunk), else one.  Timed on GB300 (apply pass per
// launch, K = 1 / 2 / 4): L=10 (2 887 chunks, 7 296 resident warps) 24.1 /
// 22.1 / 26.8 us; L=11 (11 011 chunks) 38 / 41 / 61 us; L=12 97 / 122 / 197
// us; four lanes never won where this choice applies.  Matrices of fewer than
// 2048 chunks run their Lanczos iterations in one launch (te_step.cu, K = 1);
// matrices with long rows keep K = 1.  te_matrix_set_spmv_lanes overrides.
//
// The autotuner proper (te_matrix_set_spmv_lanes(A, -1)): time the
// three-term apply pass (the dominant kernel) for K = 1, 2, 4 on the matrix
// itself, with scratch vectors and a scratch state, and keep K > 1 only when
// it is more than 10% faster.  It follows the GPU it runs on, but two copies
// of one matrix near that margin can be tuned differently.
static int tune_lanes_timed(te_matrix_s* A) {
  TeSell& S = A->sell;
  const int64_t resident_warps = (int64_t)te_num_sms() * te_sell_blocks_per_sm(A->is_real) * (TE_THREADS / 32);
  S.lanes = 1;
  if (S.n_chunks >= 8 * resident_warps || S.n_chunks < 2048 || S.n_long > 0) {
    S.lanes_fixed = true;
    return TE_OK;
  }
  const int64_t n = S.n;
  double2 *x = nullptr, *xp = nullptr, *w = nullptr;
  double* partials = nullptr;
  TeDevState* ds = nullptr;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  auto cleanup = [&]() {
    te_free(x);
    te_free(xp);
    te_free(w);
    te_free(partials);
    te_free(ds);
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
  };
  int rc = TE_OK;
  if ((rc = te_cuda_check(te_malloc(&x, sizeof(double2) * n), "tune")) == TE_OK &&
      (rc = te_cuda_check(te_malloc(&xp, sizeof(double2) * n), "tune")) == TE_OK &&
      (rc = te_cuda_check(te_malloc(&w, sizeof(double2) * n), "tune")) == TE_OK &&
      (rc = te_cuda_check(te_malloc(&partials, sizeof(double) * 2 * 8 * 4096), "tune")) == TE_OK &&
      (rc = te_cuda_check(te_malloc(&ds, sizeof(TeDevState)), "tune")) == TE_OK &&
      (rc = te_cuda_check(cudaEventCreate(&e0), "tune")) == TE_OK &&
      (rc = te_cuda_check(cudaEventCreate(&e1), "tune")) == TE_OK) {
    TeDevState* hs = new TeDevState();
    std::memset(hs, 0, sizeof(TeDevState));
    hs->exp_factor = 1.0;
    hs->inv_exp_factor = 1.0;
    hs->m_cur = 2;
    hs->s[0] = hs->s[1] = 1.0;
    hs->beta[1] = 1.0;
    rc = te_cuda_check(cudaMemcpy(ds, hs, sizeof(TeDevState), cudaMemcpyHostToDevice), "tune");
    delete hs;
    if (rc == TE_OK) rc = te_cuda_check(cudaMemset(x, 0, sizeof(double2) * n), "tune");
    if (rc == TE_OK) rc = te_cuda_check(cudaMemset(xp, 0, sizeof(double2) * n), "tune");
  }
  float best[3] = {0, 0, 0};
  const int cand[3] = {1, 2, 4};
  for (int v = 0; v < 3 && rc == TE_OK; ++v) {
    S.lanes = cand[v];
    float t_min = 1e30f;
    for (int rep = 0; rep < 6 && rc == TE_OK; ++rep) {
      cudaEventRecord(e0, 0);
      te_launch_lanczos_apply(S, A->is_real, x, xp, w, ds, partials, 1, true, 0);
      cudaEventRecord(e1, 0);
      rc = te_cuda_check(cudaEventSynchronize(e1), "tune");
      float ms = 0.0f;
      cudaEventElapsedTime(&ms, e0, e1);
      if (rep > 0) t_min = std::min(t_min, ms);  // the first launch warms the caches
    }
    best[v] = t_min;
  }
  cleanup();
  S.lanes = 1;
  if (rc != TE_OK) return rc;
  int pick = 0;
  for (int v = 1; v < 3; ++v)
    if (best[v] < best[pick]) pick = v;
  if (pick != 0 && best[pick] > 0.9f * best[0]) pick = 0;
  S.lanes = cand[pick];
  S.lanes_fixed = true;
  return TE_OK;
}

int te_tune_sell_lanes(te_matrix_s* A) {
  TeSell& S = A->sell;
  if (S.lanes_fixed) return TE_OK;
  if (S.lanes_timed) return tune_lanes_timed(A);
  const int64_t resident_warps = (int64_t)te_num_sms() * te_sell_blocks_per_sm(A->is_real) * (TE_THREADS / 32);
  S.lanes = (S.n_chunks >= 2048 && S.n_chunks < resident_warps && S.n_long == 0) ? 2 : 1;
  S.lanes_fixed = true;
  return TE_OK;
}

void te_launch_lanczos_update(int64_t n, const double2* w, const double2* u_j, double2* u_jp1, TeDevState* ds,
                              double* partials, int j, bool fold, cudaStream_t st, int4* X_out, bool alpha_acc) {
  const bool fix = u_jp1 && X_out;
  const auto k = fix ? lanczos_update_kernel<true, true, true>
                     : (alpha_acc ? lanczos_update_kernel<false, false, true>
                                  : (u_jp1 ? lanczos_update_kernel<true, false, false>
                                           : lanczos_update_kernel<false, false, false>));
  const void* kk = (const void*)k;
  const int grid = te_grid_fit(kk, n, TE_THREADS);
  te_launch_pdl(te_grid_saturated(kk, n, TE_THREADS), k, grid, TE_THREADS, st, n, w, u_j, u_jp1, ds, partials, j,
                (int)fold, fix ? X_out : nullptr);
}

void te_launch_fix_start(int64_t n, const double2* u_0, int4* X, TeDevState* ds, double* partials, cudaStream_t st) {
  unsigned int* bmax = reinterpret_cast<unsigned int*>(partials);
  const int g1 = te_grid_fit((const void*)fix_start_max_kernel, n, TE_THREADS);
  fix_start_max_kernel<<<g1, TE_THREADS, 0, st>>>(n, u_0, ds, bmax);
  const int g2 = te_grid_fit((const void*)fix_start_encode_kernel, n, TE_THREADS);
  fix_start_encode_kernel<<<g2, TE_THREADS, 0, st>>>(n, u_0, X, ds, bmax, g1);
}

namespace {

using ApplyFixKernel = void (*)(int64_t, const int32_t*, const int64_t*, TeFixMatrix, TeLongRows, const int4*,
                                const double2*, const double2*, double2*, TeDevState*, double*, int);

ApplyFixKernel apply_fix_kernel(int fmt, bool has_prev, bool has_long = true) {
  static const ApplyFixKernel table[2][3][2] = {
      {{lanczos_apply_fix_kernel<false, 0, false>, lanczos_apply_fix_kernel<true, 0, false>},
       {lanczos_apply_fix_kernel<false, 1, false>, lanczos_apply_fix_kernel<true, 1, false>},
       {lanczos_apply_fix_kernel<false, 2, false>, lanczos_apply_fix_kernel<true, 2, false>}},
      {{lanczos_apply_fix_kernel<false, 0, true>, lanczos_apply_fix_kernel<true, 0, true>},
       {lanczos_apply_fix_kernel<false, 1, true>, lanczos_apply_fix_kernel<true, 1, true>},
       {lanczos_apply_fix_kernel<false, 2, true>, lanczos_apply_fix_kernel<true, 2, true>}}};
  return table[has_long ? 1 : 0][fmt][has_prev ? 1 : 0];
}

}  // namespace

int te_fix_block_blocks_per_sm(bool is_real) {
  return te_kernel_blocks_per_sm(is_real ? (const void*)fix_block_kernel<true> : (const void*)fix_block_kernel<false>,
                                 TE_THREADS, 0);
}

void te_launch_lanczos_apply_fix_blocked(const TeSell& A, bool is_real, const int4* X, longlong2* acc,
                                         const double2* u_j, const double2* u_jm1, double2* w, TeDevState* ds,
                                         double* partials, int j, cudaStream_t st) {
  for (int b = 0; b < A.fix_nblk; ++b) {
    const TeSell::Block& B = A.fix_blk[b];
    te_launch_pdl(B.saturated, is_real ? fix_block_kernel<true> : fix_block_kernel<false>, B.grid, TE_THREADS, st,
                  B.n_rows, (const int32_t*)B.warp_chunk, (const int64_t*)B.chunk_off, (const int32_t*)B.row,
                  (const int32_t*)B.col, (const int2*)B.hv, (const int4*)B.hv4, X, acc, b == 0 ? 1 : 0,
                  (const TeDevState*)ds);
  }
  const auto k = u_jm1 ? fix_epilogue_kernel<true> : fix_epilogue_kernel<false>;
  const void* kk = (const void*)k;
  te_launch_pdl(te_grid_saturated(kk, A.n, TE_THREADS), k, te_grid_fit(kk, A.n, TE_THREADS), TE_THREADS, st, A.n,
                (const longlong2*)acc, A.fix_sh, u_j, u_jm1, w, ds, partials, j);
}

int te_apply_fix_blocks_per_sm(int fmt, size_t dyn_smem) {
  return std::min(te_kernel_blocks_per_sm((const void*)apply_fix_kernel(fmt, true), TE_THREADS, dyn_smem),
                  te_kernel_blocks_per_sm((const void*)apply_fix_kernel(fmt, false), TE_THREADS, dyn_smem));
}

void te_launch_lanczos_apply_fix(const TeSell& A, const int4* X, const double2* u_j, const double2* u_jm1,
                                 double2* w, TeDevState* ds, double* partials, int j, cudaStream_t st,
                                 const TeSegCarry* carry) {
  const int fmt = A.fix_val4 ? 2 : (A.fix_pk ? 1 : 0);
  const TeFixMatrix M{A.col, A.fix_val, A.fix_val4, A.fix_pk, A.fix_table, A.fix_nvals, A.fix_cbits, A.fix_sh};
  const size_t smem = fmt == 1 ? sizeof(int2) * A.fix_nvals : 0;
  te_launch_pdl_smem(A.fix_saturated, apply_fix_kernel(fmt, u_jm1 != nullptr, A.n_seg > 0), A.fix_grid, TE_THREADS,
                     smem, st, A.n,
                     A.fix_warp_chunk, A.chunk_off, M, te_long_rows(A, carry), X, u_j, u_jm1, w, ds, partials, j);
}



