// te_step.cu -- all three-term Lanczos iterations of a Krylov step in one
// cooperative launch, for matrices of fewer than 2048 chunks.
//
// Replaces the loop of arnoldiAlgorithm (core/krylovTimeEvolver.cpp:523-571).
// On the matrix's static schedule (8 warps per block), per iteration:
//   apply: w' = -i H u_j + (beta_j / e)^2 u_{j-1} for the warp's rows, the
//     block's <u_j, w'> -> published; every block reads all blocks' sums and
//     adds them in one fixed order, so alpha_j is the same in every block;
//   update: u'_{j+1} = w' - (alpha_j / e) u_j of the same rows, the block's
//     ||u'_{j+1}||^2 -> published and read the same way; the breakdown test.
// At these sizes an iteration is a chain of latencies, not work: one wave of
// FP64 instructions (64 cycles each per warp), gathers from L2, and two
// exchanges between all blocks.  Hence:
//  * an exchange is one store and one poll: a block's partial sum goes out as
//    tagged words (32 bits of the double, 32 bits of tag), and a reader's lane
//    polls one block's words, so arriving and reading are the same access (no
//    counter, no second round trip for the sums);
//  * rows stay in registers (u_j, u_{j-1}, w'; CPW chunks per warp at most),
//    the block's matrix slots in shared memory, so an apply waits for one
//    round of gathers and a store of u_{j+1} is the only other vector access;
//  * a ninth warp computes beta_j, s_j and the breakdown test (square root and
//    division: long FP64 sequences) while the others gather, and nothing but
//    the two products alpha_j = f <u_j, w'>, gamma = alpha_j / e follows a sum;
//  * the FP64 adds of a block's sum run on two warps (re, im) at once.
// The sums keep the order of the per-iteration version (lane by lane over the
// 8 warps, a shuffle tree, then trees over blocks of 32 partials), so the
// coefficients do not depend on how the blocks are spread.
//
// Times on GB300, per iteration: Bose-Hubbard L=6 (dim 462, 2 blocks) 12.7 us
// and L=8 (dim 6 435, 26 blocks) 16.4 us with one counter barrier per sum, the
// sums read after it and rows re-read from L2; 7.0 and 9.9 us here, with the
// same coefficients bit for bit.  What is left (cycles of an L=8 iteration of
// 19 700): apply 5 600 (30 dependent FP64 instructions on 2 warps per
// scheduler), the two exchanges 4 200 and 7 000 (with the fences that order
// the rows), the FP64 sums 2 200, the rows' recurrence 1 500.
#include <cmath>

#include "te_internal.cuh"
#include "te_reduce.cuh"

namespace {

constexpr int kWorkers = TE_THREADS / 32;           // worker warps: the schedule's 8 per block
constexpr int kStepThreads = TE_THREADS + 32;       // and one for the scalars
constexpr size_t kStepSlotBytes = 200 << 10;        // shared memory for a block's slots at most

struct TeStepArgs {
  int64_t n;
  const int32_t* warp_chunk;
  const int64_t* chunk_off;
  const int32_t* col;
  const double* val;
  double2* w;        // generic variant: w' of the step's rows
  TeStepSync* sync;
  int m;
  int slots_in_smem;        // most slots of a block when they are staged, else 0
  unsigned int tag0;        // tags of this launch: tag0 + 2 j (+ 1)
  unsigned int spin_limit;  // polls before an exchange gives up
  unsigned int blocks;      // blocks to wait for (gridDim.x; more only to test the timeout)
  double2* u[TE_MMAX];
};

struct StepShared {
  double wide[2][TE_THREADS];  // the block's per-thread sums (re, im)
  double group[2][kWorkers];   // sums of 32 blocks each
  double cw, f, gamma[2];
  int fail, breakdown;
};

__device__ __forceinline__ ulonglong2 tagged(double v, unsigned int tag) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v), t = (unsigned long long)tag << 32;
  return make_ulonglong2(t | (b & 0xffffffffull), t | (b >> 32));
}
__device__ __forceinline__ void put(ulonglong2* p, ulonglong2 v) {
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(v.x), "l"(v.y) : "memory");
}
// The double behind a tagged pair, if both words carry the tag.
__device__ __forceinline__ bool get(const ulonglong2* p, unsigned int tag, double& v) {
  ulonglong2 t;
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(t.x), "=l"(t.y) : "l"(p) : "memory");
  v = __longlong_as_double((long long)((t.y << 32) | (t.x & 0xffffffffull)));
  return (unsigned int)(t.x >> 32) == tag && (unsigned int)(t.y >> 32) == tag;
}

// Warp `q`'s share of an exchange: the sums of blocks 32 q .. 32 q + 31 (NV
// tagged pairs per block) when all of them have arrived, added by a shuffle
// tree into group[v][q].  False when the wait gave up.
template <int NV>
__device__ __forceinline__ bool step_collect(const ulonglong2* recs, unsigned int tag, const TeStepArgs& a,
                                             StepShared& S, int q, TeDevState* ds) {
  const int lane = threadIdx.x & 31;
  const unsigned int b = 32u * q + lane;
  const bool mine = b < a.blocks;
  double v[NV];
  unsigned int spins = 0;
  while (true) {
    bool ok = true;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      v[k] = 0.0;
      if (mine) ok = get(recs + (size_t)b * NV + k, tag, v[k]) && ok;
    }
    if (__all_sync(0xffffffffu, ok)) break;
    if (++spins > a.spin_limit) {
      if (lane == 0) {
        S.fail = 1;
        atomicExch(&ds->fatal, TE_ERR_DEVICE_TIMEOUT);
      }
      return false;
    }
  }
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    v[k] = te_warp_sum(v[k]);
    if (lane == 0) S.group[k][q] = v[k];
  }
  return true;
}

// The sum of the groups in the order of a shuffle tree over 8 lanes.
__device__ __forceinline__ double step_total(const double* g, int groups) {
  if (groups == 1) return g[0];
  auto at = [&](int i) { return i < groups ? g[i] : 0.0; };
  return ((at(0) + at(4)) + (at(2) + at(6))) + ((at(1) + at(5)) + (at(3) + at(7)));
}

// One block sum: lane by lane over the 8 warps, then a shuffle tree (lane 0).
__device__ __forceinline__ double step_block_sum(const double* wide) {
  const int lane = threadIdx.x & 31;
  double s = wide[lane];
#pragma unroll
  for (int i = 1; i < kWorkers; ++i) s += wide[32 * i + lane];
  return te_warp_sum(s);
}

// One lane's row, slots [s, e), entries in order (staged slots: cs, vs).
template <bool REAL, int UNR>
__device__ __forceinline__ double2 step_row(int s, int e, const int32_t* cs, const double* vs,
                                            const double2* __restrict__ x) {
  double re = 0.0, im = 0.0;
  if (REAL) {
#pragma unroll UNR
    for (; s < e; s += 32) {
      const double2 v = __ldca(x + cs[s]);
      const double h = vs[s];
      re = fma(h, v.x, re);
      im = fma(h, v.y, im);
    }
  } else {
    const double2* __restrict__ v2 = reinterpret_cast<const double2*>(vs);
#pragma unroll UNR
    for (; s < e; s += 32) {
      const double2 v = __ldca(x + cs[s]);
      const double2 h = v2[s];
      re = fma(h.x, v.x, re);
      re = fma(-h.y, v.y, re);
      im = fma(h.x, v.y, im);
      im = fma(h.y, v.x, im);
    }
  }
  return make_double2(re, im);
}

// CPW chunks per warp in registers; 0: any number, rows re-read from memory.
template <bool REAL, int CPW>
__global__ void __launch_bounds__(kStepThreads, 2) lanczos_step_kernel(TeStepArgs a, TeDevState* ds) {
  constexpr int NR = CPW > 0 ? CPW : 1;
  __shared__ StepShared S;
  extern __shared__ __align__(16) unsigned char slot_mem[];
  if (ds->fatal != 0 || ds->done != 0 || ds->breakdown != 0) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool worker = warp < kWorkers;
  const int64_t wid = (int64_t)blockIdx.x * kWorkers + warp;
  const int c_begin = worker ? a.warp_chunk[wid] : 0, c_end = worker ? a.warp_chunk[wid + 1] : 0;
  const int groups = ((int)a.blocks + 31) / 32;
  const bool leader = blockIdx.x == 0;
  if (threadIdx.x == 0) S.fail = S.breakdown = 0;
  // the block's slots, contiguous in the schedule, into shared memory
  const int32_t* cs = a.col;
  const double* vs = a.val;
  int64_t base = 0;
  if (a.slots_in_smem) {
    base = a.chunk_off[a.warp_chunk[(int64_t)blockIdx.x * kWorkers]];
    const int cnt = (int)(a.chunk_off[a.warp_chunk[(int64_t)(blockIdx.x + 1) * kWorkers]] - base);
    double* sv = reinterpret_cast<double*>(slot_mem);
    int32_t* sc = reinterpret_cast<int32_t*>(sv + (REAL ? 1 : 2) * (size_t)a.slots_in_smem);
    for (int i = threadIdx.x; i < cnt; i += kStepThreads) sc[i] = a.col[base + i];
    for (int i = threadIdx.x; i < (REAL ? 1 : 2) * cnt; i += kStepThreads)
      sv[i] = a.val[(REAL ? 1 : 2) * base + i];
    cs = sc;
    vs = sv;
  }
  int s0[NR], s1[NR], row[NR];
  double2 u[NR], up[NR], w[NR];
  if (CPW > 0) {
#pragma unroll
    for (int i = 0; i < NR; ++i) {
      const int c = c_begin + i;
      const bool have = c < c_end;
      s0[i] = have ? (int)(a.chunk_off[c] - base) + lane : 0;
      s1[i] = have ? (int)(a.chunk_off[c + 1] - base) : 0;
      const int64_t r = (int64_t)c * 32 + lane;
      row[i] = have && r < a.n ? (int)r : -1;
      u[i] = row[i] >= 0 ? a.u[0][row[i]] : make_double2(0.0, 0.0);
      up[i] = make_double2(0.0, 0.0);
    }
  }
  __syncthreads();
  const double e = ds->exp_factor, ie = ds->inv_exp_factor, tol_rate = ds->tol_rate;
  const int m = min(a.m, ds->m_cur);
  double sj = ds->s[0], g = e * sj;  // the scalar warp's
  for (int j = 0; j < m; ++j) {
    // apply; the scalar warp turns the previous norm into beta_j and s_j
    const double2* uj = a.u[j];
    if (worker) {
      if (CPW > 0) {
#pragma unroll
        for (int i = 0; i < NR; ++i)
          if (CPW == 1 || c_begin + i < c_end) w[i] = step_row<REAL, 8>(s0[i], s1[i], cs, vs, uj);
      }
    } else {
      double cw = 0.0;
      if (j > 0) {
        const double beta = fabs(g) * sqrt(step_total(S.group[0], groups));
        if (beta < tol_rate) {  // lucky breakdown (:551-555)
          if (lane == 0) S.breakdown = 1;
          if (leader && lane == 0) {
            ds->breakdown = 1;
            ds->m_eff = j;
            ds->h = beta;
          }
        } else {
          sj = g / beta;
          g = e * sj;
          cw = (beta * ie) * (beta * ie);
          if (leader && lane == 0) {
            ds->beta[j] = beta;
            ds->s[j] = sj;
          }
        }
      }
      if (lane == 0) {
        S.cw = cw;
        S.f = sj * g;
      }
    }
    __syncthreads();
    if (S.breakdown) return;
    if (worker) {
      const double cw = S.cw;
      double dr = 0.0, di = 0.0;
      auto epilogue = [&](double2 y, double2 uu, double2 pp) {
        double2 wr;
        if (j > 0) {
          wr.x = fma(cw, pp.x, y.y);
          wr.y = fma(cw, pp.y, -y.x);
        } else {
          wr.x = y.y;
          wr.y = -y.x;
        }
        dr = fma(uu.x, wr.x, fma(uu.y, wr.y, dr));
        di = fma(uu.x, wr.y, fma(-uu.y, wr.x, di));
        return wr;
      };
      if (CPW > 0) {
#pragma unroll
        for (int i = 0; i < NR; ++i)
          if (row[i] >= 0) w[i] = epilogue(w[i], u[i], up[i]);
      } else {
        for (int c = c_begin; c < c_end; ++c) {
          const double2 y = step_row<REAL, 4>((int)(a.chunk_off[c] - base) + lane, (int)(a.chunk_off[c + 1] - base), cs,
                                              vs, uj);
          const int64_t r = (int64_t)c * 32 + lane;
          if (r < a.n) a.w[r] = epilogue(y, __ldca(uj + r), j > 0 ? __ldca(a.u[j - 1] + r) : make_double2(0.0, 0.0));
        }
      }
      S.wide[0][threadIdx.x] = dr;
      S.wide[1][threadIdx.x] = di;
    }
    __syncthreads();
    const unsigned int tag = a.tag0 + 2u * j;
    if (warp < 2) {
      const double s = step_block_sum(S.wide[warp]);
      if (lane == 0) put(&a.sync->alpha[blockIdx.x][warp], tagged(s, tag));
    }
    if (warp < groups) step_collect<2>(&a.sync->alpha[0][0], tag, a, S, warp, ds);
    if (groups > 1) __syncthreads();
    if (warp == 0) {  // lane 0: re, lane 1: im
      __syncwarp();
      const double al = S.f * step_total(S.group[lane & 1], groups);
      const double ga = al * ie;  // gamma = alpha_j / e
      if (lane < 2) {
        S.gamma[lane] = ga;
        if (leader) reinterpret_cast<double*>(&ds->alpha[j])[lane] = al;
      }
    }
    __syncthreads();
    if (S.fail) return;
    const double gr = S.gamma[0], gi = S.gamma[1];
    // update of this warp's rows: u'_{j+1} = w' - gamma u_j
    if (worker) {
      double2* ujp1 = j + 1 < m ? a.u[j + 1] : nullptr;
      double nr = 0.0;
      auto update = [&](double2 wv, double2 uu) {
        double2 o;
        o.x = fma(-gr, uu.x, fma(gi, uu.y, wv.x));
        o.y = fma(-gr, uu.y, fma(-gi, uu.x, wv.y));
        nr = fma(o.x, o.x, fma(o.y, o.y, nr));
        return o;
      };
      if (CPW > 0) {
#pragma unroll
        for (int i = 0; i < NR; ++i) {
          if (row[i] >= 0) {
            const double2 o = update(w[i], u[i]);
            if (ujp1) ujp1[row[i]] = o;
            up[i] = u[i];
            u[i] = o;
          }
        }
      } else {
        for (int c = c_begin; c < c_end; ++c) {
          const int64_t r = (int64_t)c * 32 + lane;
          if (r < a.n) {
            const double2 o = update(__ldca(a.w + r), __ldca(uj + r));
            if (ujp1) ujp1[r] = o;
          }
        }
      }
      S.wide[0][threadIdx.x] = nr;
    }
    __syncthreads();
    if (warp == 0) {
      const double s = step_block_sum(S.wide[0]);
      asm volatile("fence.acq_rel.gpu;" ::: "memory");  // the rows this block stored, before its sum
      if (lane == 0) put(&a.sync->norm[blockIdx.x], tagged(s, tag + 1));
    }
    const bool last = j + 1 == m;
    if (last && !leader) return;
    if (warp < groups) {
      step_collect<1>(&a.sync->norm[0], tag + 1, a, S, warp, ds);
      asm volatile("fence.acq_rel.gpu;" ::: "memory");  // the other blocks' rows, after their sums
    }
    __syncthreads();
    if (S.fail) return;
    if (last && threadIdx.x == TE_THREADS) {
      const double beta = fabs(g) * sqrt(step_total(S.group[0], groups));
      if (beta < tol_rate) {
        ds->breakdown = 1;
        ds->m_eff = j + 1;
      } else {
        ds->m_eff = m;
      }
      ds->h = beta;
    }
  }
}

using StepKernel = void (*)(TeStepArgs, TeDevState*);

template <bool REAL>
StepKernel step_kernel(int chunks) {
  if (chunks <= 1) return lanczos_step_kernel<REAL, 1>;
  if (chunks <= 2) return lanczos_step_kernel<REAL, 2>;
  if (chunks <= 4) return lanczos_step_kernel<REAL, 4>;
  return lanczos_step_kernel<REAL, 0>;
}

}  // namespace

bool te_launch_lanczos_step(const TeSell& A, bool is_real, double2* const* cols, int m, double2* w, TeDevState* ds,
                            TeStepSync* sync, unsigned int launch, cudaStream_t st, unsigned int spin_limit,
                            unsigned int extra_arrivals) {
  if (A.n_long > 0 || m < 1 || m > TE_MMAX || A.grid + (int)extra_arrivals > TE_STEP_BLOCKS || A.n_chunks < 1 ||
      A.slots >= ((int64_t)1 << 31) - 256)
    return false;
  static const int coop = [] {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrCooperativeLaunch, dev);
    return v;
  }();
  if (!coop) return false;
  const StepKernel k = is_real ? step_kernel<true>(A.warp_chunks) : step_kernel<false>(A.warp_chunks);
  TeStepArgs a{};
  size_t smem = (size_t)A.block_slots * (is_real ? 12 : 20);
  // one block per SM is enough up to 152 blocks; beyond that two share an SM
  const size_t cap = A.grid > te_num_sms() ? kStepSlotBytes / 2 : kStepSlotBytes;
  if (smem > cap) smem = 0;
  if (smem > 0 &&
      cudaFuncSetAttribute((const void*)k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kStepSlotBytes) !=
          cudaSuccess) {
    cudaGetLastError();
    smem = 0;
  }
  a.slots_in_smem = smem ? (int)A.block_slots : 0;
  a.n = A.n;
  a.warp_chunk = A.warp_chunk;
  a.chunk_off = A.chunk_off;
  a.col = A.col;
  a.val = A.val;
  a.w = w;
  a.sync = sync;
  a.m = m;
  a.tag0 = (launch + 1u) * 256u;
  a.spin_limit = spin_limit;
  a.blocks = (unsigned int)A.grid + extra_arrivals;
  for (int j = 0; j < TE_MMAX; ++j) a.u[j] = j < m ? cols[j] : nullptr;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(A.grid);
  cfg.blockDim = dim3(kStepThreads);
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
