// te_sample.cu -- states and observables from the Krylov basis.
//
// Replaces, in krylovTimeEvolver::timeEvolve (core/krylovTimeEvolver.cpp):
//   currentVec = V w                 (:382, cblas_zgemv n x m)
//   sampledState = V y(t_sampling)   (:409-421)
//   sample() -> observable->expectation (:120-126, krylovObservables.cpp:173-236)
//   the final norm check            (:446-452, cblas_dznrm2)
// One pass over the m basis columns produces every output of a batch (the
// next start vector and the batch's samples), so V is read once per batch;
// diagonal and vector observables are reduced in one further pass over the
// batch.  All reductions finish in the last block to complete, in a fixed
// order.
#include <algorithm>

#include "te_fixed.cuh"
#include "te_internal.cuh"
#include "te_reduce.cuh"

#define TE_COMBINE_GROUP 4

// Rows of G outputs: psi_o[r] = sum_j u_j[r] ys[o][j].  G is a compile-time
// count: on GB300 a predicated-off FP64 instruction still occupies the FP64
// pipe, so every output slot that exists in the code must be a real output.
template <int G>
__device__ __forceinline__ void combine_rows(const TeCombineArgs& a, const double2* const* cols, int m,
                                             const double2 (*ys)[TE_MMAX], const int* slot_s, int S,
                                             double2* last_out, double2* store, int64_t store_ld, int base) {
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < a.n; r += (int64_t)gridDim.x * blockDim.x) {
    double2 acc[G];
#pragma unroll
    for (int o = 0; o < G; ++o) acc[o] = make_double2(0.0, 0.0);
    for (int j = 0; j < m; ++j) {
      const double2 u = cols[j][r];
#pragma unroll
      for (int o = 0; o < G; ++o) {
        const double2 y = ys[o][j];
        acc[o].x = fma(u.x, y.x, fma(-u.y, y.y, acc[o].x));
        acc[o].y = fma(u.x, y.y, fma(u.y, y.x, acc[o].y));
      }
    }
#pragma unroll
    for (int o = 0; o < G; ++o) {
      const int slot = slot_s[o];
      if (slot == 0) {
        a.w_out[r] = acc[o];
      } else {
        a.sample_out[(int64_t)(slot - 1) * a.n + r] = acc[o];
        if (slot == S) last_out[r] = acc[o];
        if (store) store[(int64_t)(base + slot - 1) * store_ld + r] = acc[o];
      }
    }
  }
}

// Basis vectors of a row in flight per thread in the fixed-point combine: 8
// measured 10.4 ms per L=12 solve against 11.2 (4) and 13.4 (1).
constexpr int kCombineUnroll = 8;

// The same outputs from the fixed-point copies X_j = round(u_j 2^xs_j) of the
// basis (te_fixed.cuh), on the integer pipes: with c_oj = Y[slot_o][j] 2^-xs_j
// (so that c_oj X_j = Y[slot_o][j] u_j) quantised per output as
// C_oj = round(c_oj 2^sc_o), sc_o putting sum_j (|Re c_oj| + |Im c_oj|) below
// 2^61, psi_o = 2^(62 - sc_o) sum_j C_oj X_j with the limb products of
// te_fix_mac (complex: Re = Cr Xr - Ci Xi, Im = Cr Xi + Ci Xr).  Error per
// component below 4 m 1.25 2^-56 + (m + 1) 2^-61 of sum_j |Y_oj| max|u_j|.
template <int G>
__device__ __forceinline__ void combine_rows_fix(const TeCombineArgs& a, int m, const int4 (*C)[TE_MMAX],
                                                 const int* sc, const int* slot_s, int S, double2* last_out,
                                                 double2* store, int64_t store_ld, int base) {
  const int64_t n = a.n;
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
    int64_t sr[G], si[G];
#pragma unroll
    for (int o = 0; o < G; ++o) sr[o] = si[o] = 0;
#pragma unroll(kCombineUnroll)
    for (int j = 0; j < m; ++j) {
      const int4 x = __ldcs(a.fx + (int64_t)j * n + r);  // {re0, re1, im0, im1}
#pragma unroll
      for (int o = 0; o < G; ++o) {
        const int4 c = C[o][j];  // {re0, re1, im0, im1}
        sr[o] += te_fix_prod(c.x, c.y, x.x, x.y) - te_fix_prod(c.z, c.w, x.z, x.w);
        si[o] += te_fix_prod(c.x, c.y, x.z, x.w) + te_fix_prod(c.z, c.w, x.x, x.y);
      }
    }
#pragma unroll
    for (int o = 0; o < G; ++o) {
      const double2 v = make_double2(te_i64_to_double(sr[o], 62 - sc[o]), te_i64_to_double(si[o], 62 - sc[o]));
      const int slot = slot_s[o];
      if (slot == 0) {
        a.w_out[r] = v;
      } else {
        a.sample_out[(int64_t)(slot - 1) * n + r] = v;
        if (slot == S) last_out[r] = v;
        if (store) store[(int64_t)(base + slot - 1) * store_ld + r] = v;
      }
    }
  }
}

// psi_o = sum_j u_j Y[slot_o][j] for the outputs of this batch (the step's
// next start vector w, then its samples), one pass over V per group of up to
// four outputs.
__global__ void __launch_bounds__(TE_THREADS) combine_kernel(TeCombineArgs a, TeDevState* ds, double2* last_out) {
  __shared__ double2 ys[TE_COMBINE_GROUP][TE_MMAX];
  __shared__ int4 cfix[TE_COMBINE_GROUP][TE_MMAX];  // fixed-point coefficients (a.fx)
  __shared__ int sc_s[TE_COMBINE_GROUP];
  __shared__ int slot_s[TE_COMBINE_GROUP];
  __shared__ const double2* cols[TE_MMAX];
  if (ds->fatal != 0) return;
  const int want_w = ds->want_w;
  const int S = ds->samples_in_batch;
  const int nout = want_w + S;
  const int m = min(a.m, ds->m_eff);  // a lucky breakdown shrinks the basis of this step
  if (threadIdx.x < TE_MMAX) cols[threadIdx.x] = threadIdx.x < m ? a.cols[threadIdx.x] : nullptr;
  for (int g0 = 0; g0 < nout; g0 += TE_COMBINE_GROUP) {
    const int G = min(TE_COMBINE_GROUP, nout - g0);
    __syncthreads();
    if (threadIdx.x < TE_COMBINE_GROUP) {
      const int o = g0 + threadIdx.x;
      slot_s[threadIdx.x] = want_w ? o : o + 1;  // slot 0 = w, slots 1.. = samples
    }
    __syncthreads();
    for (int i = threadIdx.x; i < G * TE_MMAX; i += blockDim.x) {
      const int o = i / TE_MMAX, j = i % TE_MMAX;
      ys[o][j] = j < m ? ds->Y[slot_s[o] * TE_MMAX + j] : make_double2(0.0, 0.0);
    }
    __syncthreads();
    double2* store = ds->state_store;
    const int64_t sld = ds->store_ld;
    const int base = ds->sample_base;
    if (a.fx) {
      // coefficients c_oj = Y_oj 2^-xs_j in fixed point, per output scale
      if (threadIdx.x < G) {
        double b = 0.0;
        for (int j = 0; j < m; ++j) {
          const int xs = ds->fx_xs[j];
          b += ldexp(fabs(ys[threadIdx.x][j].x), -xs) + ldexp(fabs(ys[threadIdx.x][j].y), -xs);
        }
        sc_s[threadIdx.x] = te_fix_scale(b * (1.0 + 1e-12));
      }
      __syncthreads();
      for (int i = threadIdx.x; i < G * TE_MMAX; i += blockDim.x) {
        const int o = i / TE_MMAX, j = i % TE_MMAX;
        int4 c = make_int4(0, 0, 0, 0);
        if (j < m) {
          const int xs = ds->fx_xs[j];
          const int2 cr = te_fix_split(te_fix_encode(ldexp(ys[o][j].x, -xs), sc_s[o]));
          const int2 ci = te_fix_split(te_fix_encode(ldexp(ys[o][j].y, -xs), sc_s[o]));
          c = make_int4(cr.x, cr.y, ci.x, ci.y);
        }
        cfix[o][j] = c;
      }
      __syncthreads();
      switch (G) {
        case 1: combine_rows_fix<1>(a, m, cfix, sc_s, slot_s, S, last_out, store, sld, base); break;
        case 2: combine_rows_fix<2>(a, m, cfix, sc_s, slot_s, S, last_out, store, sld, base); break;
        case 3: combine_rows_fix<3>(a, m, cfix, sc_s, slot_s, S, last_out, store, sld, base); break;
        default: combine_rows_fix<4>(a, m, cfix, sc_s, slot_s, S, last_out, store, sld, base); break;
      }
      continue;
    }
    switch (G) {
      case 1: combine_rows<1>(a, cols, m, ys, slot_s, S, last_out, store, sld, base); break;
      case 2: combine_rows<2>(a, cols, m, ys, slot_s, S, last_out, store, sld, base); break;
      case 3: combine_rows<3>(a, cols, m, ys, slot_s, S, last_out, store, sld, base); break;
      default: combine_rows<4>(a, cols, m, ys, slot_s, S, last_out, store, sld, base); break;
    }
  }
}

// The FP64 outputs of a small basis, one (4 chunks of 32 rows, output) per
// block of 4 warps.  The pass is bound by FP64 issue (4 m per row and output),
// so what counts is how many SMs share it: combine_kernel gives 256 rows and
// every output to one block, 2 SMs at dim 462.  Each output's sum is the same
// bit for bit.  Measured on GB300 (m = 30..40, 9 outputs): dim 462 79 -> 13 us,
// dim 6 435 80 -> 23 us; from 2048 chunks on both fill the GPU and sharing the
// basis reads between outputs pays.
__global__ void __launch_bounds__(128) combine_small_kernel(TeCombineArgs a, TeDevState* ds, double2* last_out) {
  __shared__ double2 y[TE_MMAX];
  if (ds->fatal != 0) return;
  const int want_w = ds->want_w, S = ds->samples_in_batch;
  if ((int)blockIdx.y >= want_w + S) return;
  const int slot = want_w ? blockIdx.y : blockIdx.y + 1;  // slot 0 = w, slots 1.. = samples
  const int m = min(a.m, ds->m_eff);
  if ((int)threadIdx.x < m) y[threadIdx.x] = ds->Y[slot * TE_MMAX + threadIdx.x];
  __syncthreads();
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (r >= a.n) return;
  double2 acc = make_double2(0.0, 0.0);
#pragma unroll 8
  for (int j = 0; j < m; ++j) {
    const double2 u = a.cols[j][r], c = y[j];
    acc.x = fma(u.x, c.x, fma(-u.y, c.y, acc.x));
    acc.y = fma(u.x, c.y, fma(u.y, c.x, acc.y));
  }
  if (slot == 0) {
    a.w_out[r] = acc;
  } else {
    a.sample_out[(int64_t)(slot - 1) * a.n + r] = acc;
    if (slot == S) last_out[r] = acc;
    if (ds->state_store) ds->state_store[(int64_t)(ds->sample_base + slot - 1) * ds->store_ld + r] = acc;
  }
}

void te_launch_combine(const TeCombineArgs& a, TeDevState* ds, double2* last_out, cudaStream_t st) {
  if (!a.fx && a.n < 2048 * 32) {
    combine_small_kernel<<<dim3((unsigned)((a.n + 127) / 128), TE_SCAP + 1), 128, 0, st>>>(a, ds, last_out);
    return;
  }
  combine_kernel<<<te_grid_fit((const void*)combine_kernel, a.n, TE_THREADS), TE_THREADS, 0, st>>>(a, ds, last_out);
}

// Block sums of V values per thread, one warp per value (wide: V * blockDim.x
// doubles; a warp adds blockDim.x / 32 values per lane, then a shuffle tree);
// warp v's lane 0 stores value v's sum at dst[v * stride].
template <int V>
__device__ __forceinline__ void obs_block_sums(const double (&acc)[V], double* wide, double* dst, int64_t stride) {
  const int B = blockDim.x, lane = threadIdx.x & 31;
  __syncthreads();
#pragma unroll
  for (int v = 0; v < V; ++v) wide[v * B + threadIdx.x] = acc[v];
  __syncthreads();
  for (int v = threadIdx.x >> 5; v < V; v += B >> 5) {
    double s = wide[v * B + lane];
    for (int i = lane + 32; i < B; i += 32) s += wide[v * B + i];
    s = te_warp_sum(s);
    if (lane == 0) dst[v * stride] = s;
  }
}

// Blocks that work on a batch of S samples over gridDim.y; the last of them to
// arrive returns true (and resets the counter).
__device__ __forceinline__ bool obs_last_block(unsigned int* counter, int S) {
  __shared__ bool is_last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned int all = gridDim.x * (unsigned int)min((int)gridDim.y, S);
    is_last = atomicAdd(counter, 1u) == all - 1;
    if (is_last) *counter = 0u;
  }
  __syncthreads();
  if (is_last) __threadfence();
  return is_last;
}

// One warp's sum of the row blocks' partials of one value (lane 0).
__device__ __forceinline__ double obs_partial_sum(const double* p) {
  double s = 0.0;
  for (int b = threadIdx.x & 31; b < (int)gridDim.x; b += 32) s += __ldcg(p + b);
  return te_warp_sum(s);
}

// Rows and samples of a batch over the grid: row blocks in x; a small dimension
// takes a block of its own per sample in y (up to TE_SCAP), a large one loops
// over the samples.  Measured on GB300 (8 occupations, batches of 7 samples):
// dim 6 435 48 -> 15 us per launch, and half the launches.
static dim3 obs_grid(int64_t n, const void* kernel) {
  const int64_t blocks = (n + TE_THREADS - 1) / TE_THREADS;
  if (blocks * TE_SCAP <= 8 * (int64_t)te_num_sms() || blocks <= 64) return dim3((unsigned)std::max<int64_t>(blocks, 1), TE_SCAP);
  return dim3((unsigned)te_grid_fit(kernel, n, TE_THREADS));
}

// Diagonal observables: Re sum_i O_ii |psi_i|^2 (= Re zdotc(psi, O psi) for a
// diagonal O); vector observables: |sum_i conj(psi_i) o_i|^2.  ND diagonal and
// NV vector observables per launch, compile-time counts (no predicated FP64).
template <int ND, int NV>
__global__ void __launch_bounds__(TE_THREADS) fused_obs_kernel(int64_t n, const double2* __restrict__ psi_base,
                                                               TeFusedObs f, TeDevState* ds, double* partials,
                                                               double* results, int n_samples_total) {
  constexpr int V = ND + 2 * NV;
  __shared__ double wide[V * TE_THREADS];
  if (ds->fatal != 0) return;
  const int S = ds->samples_in_batch;
  const int base = ds->sample_base;
  if ((int)blockIdx.y >= S) return;
  for (int s = blockIdx.y; s < S; s += gridDim.y) {
    const double2* __restrict__ psi = psi_base + (int64_t)s * n;
    double acc[V];
#pragma unroll
    for (int v = 0; v < V; ++v) acc[v] = 0.0;
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
      const double2 p = psi[r];
      if (ND > 0) {
        const double p2 = fma(p.x, p.x, p.y * p.y);
#pragma unroll
        for (int v = 0; v < ND; ++v) acc[v] = fma(__ldg(f.diag[v] + r), p2, acc[v]);
      }
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        const double2 o = __ldg(f.vec[v] + r);
        // conj(psi) * o
        acc[ND + 2 * v] = fma(p.x, o.x, fma(p.y, o.y, acc[ND + 2 * v]));
        acc[ND + 2 * v + 1] = fma(p.x, o.y, fma(-p.y, o.x, acc[ND + 2 * v + 1]));
      }
    }
    obs_block_sums<V>(acc, wide, partials + (int64_t)s * V * gridDim.x + blockIdx.x, gridDim.x);
  }
  if (!obs_last_block(&ds->counter[2], S)) return;
  const int lane = threadIdx.x & 31;
  for (int q = threadIdx.x >> 5; q < S * (ND + NV); q += blockDim.x >> 5) {
    const int s = q / (ND + NV), v = q % (ND + NV);
    const double* p = partials + (int64_t)s * V * gridDim.x;
    if (v < ND) {
      const double t = obs_partial_sum(p + (int64_t)v * gridDim.x);
      if (lane == 0) results[(int64_t)f.row_diag[v] * n_samples_total + base + s] = t;
    } else {
      const int w = v - ND;
      const double re = obs_partial_sum(p + (int64_t)(ND + 2 * w) * gridDim.x);
      const double im = obs_partial_sum(p + (int64_t)(ND + 2 * w + 1) * gridDim.x);
      if (lane == 0) results[(int64_t)f.row_vec[w] * n_samples_total + base + s] = re * re + im * im;
    }
  }
}

template <int ND, int NV>
static void launch_fused(int64_t n, const double2* psi, const TeFusedObs& f, TeDevState* ds, double* partials,
                         double* results, int n_samples_total, cudaStream_t st) {
  fused_obs_kernel<ND, NV><<<obs_grid(n, (const void*)fused_obs_kernel<ND, NV>), TE_THREADS, 0, st>>>(
      n, psi, f, ds, partials, results, n_samples_total);
}

void te_launch_fused_obs(int64_t n, const double2* psi, const TeFusedObs& f, TeDevState* ds, double* partials,
                         double* results, int n_samples_total, cudaStream_t st) {
  typedef void (*L)(int64_t, const double2*, const TeFusedObs&, TeDevState*, double*, double*, int, cudaStream_t);
  static const L table[TE_FUSED_DIAG + 1][TE_FUSED_VEC + 1] = {
      {nullptr, launch_fused<0, 1>, launch_fused<0, 2>},
      {launch_fused<1, 0>, launch_fused<1, 1>, launch_fused<1, 2>},
      {launch_fused<2, 0>, launch_fused<2, 1>, launch_fused<2, 2>},
      {launch_fused<3, 0>, launch_fused<3, 1>, launch_fused<3, 2>},
      {launch_fused<4, 0>, launch_fused<4, 1>, launch_fused<4, 2>},
      {launch_fused<5, 0>, launch_fused<5, 1>, launch_fused<5, 2>},
      {launch_fused<6, 0>, launch_fused<6, 1>, launch_fused<6, 2>},
      {launch_fused<7, 0>, launch_fused<7, 1>, launch_fused<7, 2>},
      {launch_fused<8, 0>, launch_fused<8, 1>, launch_fused<8, 2>}};
  L fn = table[f.n_diag][f.n_vec];
  if (fn) fn(n, psi, f, ds, partials, results, n_samples_total, st);
}

// General sparse observable: Re sum_i conj(psi_i) (O psi)_i
// (krylovObservables.cpp:187-189) of every sample of the batch, on O's original
// CSR: psi is in the evolver's row order, so original row i is read at
// iperm[i].  Results go to results_row[base + s].
template <bool REAL>
__global__ void __launch_bounds__(TE_THREADS) general_obs_kernel(int64_t n, const int32_t* __restrict__ row_ptr,
                                                                 const int32_t* __restrict__ col,
                                                                 const double* __restrict__ val,
                                                                 const int32_t* __restrict__ iperm,
                                                                 const double2* __restrict__ psi_base,
                                                                 TeDevState* ds, double* partials,
                                                                 double* results_row) {
  __shared__ double wide[TE_THREADS];
  if (ds->fatal != 0) return;
  const int S = ds->samples_in_batch;
  if ((int)blockIdx.y >= S) return;
  for (int s = blockIdx.y; s < S; s += gridDim.y) {
    const double2* __restrict__ psi = psi_base + (int64_t)s * n;
    double acc[1] = {0.0};
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
      const int32_t b = __ldg(row_ptr + r), e = __ldg(row_ptr + r + 1);
      if (b == e) continue;
      double re = 0.0, im = 0.0;
#pragma unroll 4
      for (int32_t q = b; q < e; ++q) {
        const double2 x = __ldg(psi + __ldg(iperm + __ldg(col + q)));
        if (REAL) {
          const double h = __ldg(val + q);
          re = fma(h, x.x, re);
          im = fma(h, x.y, im);
        } else {
          const double2 h = __ldg(reinterpret_cast<const double2*>(val) + q);
          re = fma(h.x, x.x, re);
          re = fma(-h.y, x.y, re);
          im = fma(h.x, x.y, im);
          im = fma(h.y, x.x, im);
        }
      }
      const double2 p = __ldg(psi + __ldg(iperm + r));
      acc[0] = fma(p.x, re, fma(p.y, im, acc[0]));
    }
    obs_block_sums<1>(acc, wide, partials + (int64_t)s * gridDim.x + blockIdx.x, 1);
  }
  if (!obs_last_block(&ds->counter[3], S)) return;
  for (int s = threadIdx.x >> 5; s < S; s += blockDim.x >> 5) {
    const double t = obs_partial_sum(partials + (int64_t)s * gridDim.x);
    if ((threadIdx.x & 31) == 0) results_row[ds->sample_base + s] = t;
  }
}

void te_launch_general_obs(const te_matrix_s& O, const int32_t* iperm, const double2* psi, TeDevState* ds,
                           double* partials, double* results_row, cudaStream_t st) {
  if (O.is_real)
    general_obs_kernel<true><<<obs_grid(O.n_rows, (const void*)general_obs_kernel<true>), TE_THREADS, 0, st>>>(
        O.n_rows, O.row_ptr, O.col, O.val, iperm, psi, ds, partials, results_row);
  else
    general_obs_kernel<false><<<obs_grid(O.n_rows, (const void*)general_obs_kernel<false>), TE_THREADS, 0, st>>>(
        O.n_rows, O.row_ptr, O.col, O.val, iperm, psi, ds, partials, results_row);
}

// Dense observable: Re sum_i conj(psi_i) (O psi)_i for a column-major complex O
// (original ordering; psi read through iperm) of every sample of the batch (the
// zgemv + zdotc of krylovObservables.cpp:119-138).  One thread per row
// (column-major: a warp reads 32 consecutive entries of a column); psi is
// staged through shared memory in tiles.
#define TE_DENSE_TILE 1024
__global__ void __launch_bounds__(TE_THREADS) dense_obs_kernel(int64_t n, const double2* __restrict__ O,
                                                               const int32_t* __restrict__ iperm,
                                                               const double2* __restrict__ psi_base, TeDevState* ds,
                                                               double* partials, double* results_row) {
  __shared__ double2 tile[TE_DENSE_TILE];
  __shared__ double wide[TE_THREADS];
  if (ds->fatal != 0) return;
  const int S = ds->samples_in_batch;
  if ((int)blockIdx.y >= S) return;
  for (int s = blockIdx.y; s < S; s += gridDim.y) {
    const double2* __restrict__ psi = psi_base + (int64_t)s * n;
    double acc[1] = {0.0};
    const int64_t rows_per_pass = (int64_t)gridDim.x * blockDim.x;
    for (int64_t r0 = (int64_t)blockIdx.x * blockDim.x; r0 < n; r0 += rows_per_pass) {
      const int64_t r = r0 + threadIdx.x;
      double yr = 0.0, yi = 0.0;
      for (int64_t j0 = 0; j0 < n; j0 += TE_DENSE_TILE) {
        const int64_t jn = min((int64_t)TE_DENSE_TILE, n - j0);
        __syncthreads();
        for (int64_t k = threadIdx.x; k < jn; k += blockDim.x) tile[k] = psi[iperm[j0 + k]];
        __syncthreads();
        if (r < n) {
          const double2* __restrict__ col = O + j0 * n + r;
          for (int64_t k = 0; k < jn; ++k) {
            const double2 a = col[k * n];
            const double2 x = tile[k];
            yr = fma(a.x, x.x, fma(-a.y, x.y, yr));
            yi = fma(a.x, x.y, fma(a.y, x.x, yi));
          }
        }
      }
      if (r < n) {
        const double2 p = psi[iperm[r]];
        acc[0] = fma(p.x, yr, fma(p.y, yi, acc[0]));
      }
    }
    obs_block_sums<1>(acc, wide, partials + (int64_t)s * gridDim.x + blockIdx.x, 1);
  }
  if (!obs_last_block(&ds->counter[3], S)) return;
  for (int s = threadIdx.x >> 5; s < S; s += blockDim.x >> 5) {
    const double t = obs_partial_sum(partials + (int64_t)s * gridDim.x);
    if ((threadIdx.x & 31) == 0) results_row[ds->sample_base + s] = t;
  }
}

void te_launch_dense_obs(int64_t n, const double2* O, const int32_t* iperm, const double2* psi, TeDevState* ds,
                         double* partials, double* results_row, cudaStream_t st) {
  dense_obs_kernel<<<obs_grid(n, (const void*)dense_obs_kernel), TE_THREADS, 0, st>>>(n, O, iperm, psi, ds, partials,
                                                                                      results_row);
}

__global__ void stop_check_kernel(TeStopConds c, const double* __restrict__ results, int n_samples_total,
                                  TeDevState* ds) {
  if (threadIdx.x != 0 || ds->fatal != 0 || ds->stop_flag != 0) return;
  const int S = ds->samples_in_batch, base = ds->sample_base;
  for (int s = 0; s < S; ++s)
    for (int k = 0; k < c.count; ++k) {
      const double v = results[(int64_t)c.obs[k] * n_samples_total + base + s];
      if (c.direction[k] > 0 ? v >= c.threshold[k] : v <= c.threshold[k]) {
        ds->stop_flag = s + 1;
        return;
      }
    }
}

void te_launch_stop_check(const TeStopConds& c, const double* results, int n_samples_total, TeDevState* ds,
                          cudaStream_t st) {
  stop_check_kernel<<<1, 32, 0, st>>>(c, results, n_samples_total, ds);
}

// ||x||^2 into ds->norm2_final (cblas_dznrm2 of :446).
__global__ void __launch_bounds__(TE_THREADS) norm2_kernel(int64_t n, const double2* __restrict__ x, TeDevState* ds,
                                                           double* partials) {
  __shared__ double scratch[32];
  double acc[1] = {0.0};
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
    const double2 p = x[r];
    acc[0] = fma(p.x, p.x, fma(p.y, p.y, acc[0]));
  }
  te_block_sum<1>(acc, scratch);
  if (te_publish_partials<1>(acc, partials, &ds->counter[3])) {
    double tot[1];
    te_final_sum<1>(tot, partials, &ds->counter[3], scratch);
    if (threadIdx.x == 0) ds->norm2_final = tot[0];
  }
}

void te_launch_norm2(int64_t n, const double2* x, double* partials, TeDevState* ds, cudaStream_t st) {
  norm2_kernel<<<te_grid_fit((const void*)norm2_kernel, n, TE_THREADS), TE_THREADS, 0, st>>>(n, x, ds, partials);
}
