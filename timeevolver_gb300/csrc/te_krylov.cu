// te_krylov.cu -- the Krylov-space part of one time step, on one cluster of blocks.
//
// Replaces, per Krylov step of krylovTimeEvolver::timeEvolve
// (core/krylovTimeEvolver.cpp:261-512):
//   LAPACKE_zhseqr on the m x m Krylov matrix (:365, matrixDataTypes.h:135-156),
//   expKrylov (:685-702), integrateError (:584-618),
//   findMaximalStepSize (:153-254), and the sampling schedule of :405-421.
//
// Krylov matrix.  Lanczos on A = -i expFactor H gives H_k with diagonal
// alpha_j (imaginary up to rounding) and off-diagonals +-beta_j.  With
// D = diag(i^j), H_k = D (-i T) D^{-1} where T is the real symmetric
// tridiagonal matrix with T_jj = -Im(alpha_j), T_{j,j+1} = beta_{j+1}; so
// exp(x H_k) e_1 = D exp(-i x T) e_1 (the rounding-level real parts of
// alpha_j are dropped).
//
// Exponential.  On GB300 FP64 issue is the scarce resource (a warp FP64
// instruction costs the same with 1 or 32 lanes active), so the dense
// eigensolve of the reference is replaced on the hot path by the
// Chebyshev-Bessel (Jacobi-Anger) expansion
//   exp(-i x T) e_1 = e^{-ixc} sum_n eps_n (-i)^n J_n(x rho) t_n,
//   t_n = T_n((T - c)/rho) e_1,   [c - rho, c + rho] = Gershgorin interval,
// with the vectors t_n built once per step by the three-term recurrence and
// the Bessel values J_n by Miller's backward recurrence (one lane per
// abscissa, all lanes busy).  The error integrand h |e_m^T exp(-ixT) e_1|
// only involves n >= m-1 (t_n has support 0..n), so it is evaluated without
// the cancellation of the eigenvector form.  Arguments x rho beyond the
// stored degree (lucky-breakdown steps that jump to the final time, very long
// step candidates) use the eigen-decomposition T = Q diag(lam) Q^T computed
// by implicit symmetric QR with Wilkinson shifts on one warp.
//
// Quadrature.  Tanh-sinh with the level rule shared with the CPU oracle
// (nodes t in [-3, 3], level k adds odd multiples of 2^-k, stop at the first
// level k >= 2 with |I_k - I_{k-1}| <= 1e-3 L1_k, at most level 8); levels
// 0..3 are evaluated together (49 abscissae; the integrand rises like x^(m-1)
// and stops there).  Gauss-Legendre 15/7 for fastIntegration.
//
// Layout.  A step is a chain of short FP64 sequences, and a warp issues one
// FP64 instruction per 64 cycles however many lanes it uses (one warp per
// scheduler: 4 warps a block).  So the work is spread for latency:
//  * a cluster of blocks runs the reference's step-size search (all blocks and
//    threads follow the same branches): the integral asked for and the ones
//    the search is likely to ask for next (the following substeps, the next
//    halvings or doublings) are evaluated at the same time, one per block, and
//    exchanged through distributed shared memory.  The search takes the
//    results it needs from that list and starts another round when one is
//    missing, so its decisions and values are those of the serial search;
//  * the outputs of a step (next start vector, samples) are spread over the
//    blocks as well;
//  * two warps share the Bessel recurrence of 32 abscissae, one running J_k and
//    its factor, the other the sums, 16 steps behind through shared memory.
//    (Two lanes sharing it, one FP64 instruction for both, is slower: a value
//    that leaves the FP64 pipe for a shuffle or a select takes ~150 cycles,
//    one that stays in it 65.)
// Measured on GB300 per Krylov step, against one block of 256 threads with the
// integrals in sequence, results the same bit for bit: Bose-Hubbard L=6 170 ->
// 69 us, L=8 (9 integrals a step) 294 -> 88 us, L=10 219 -> 108 us, L=12 169
// -> 83 us.
#include <cfloat>
#include <cmath>
#include <vector>

#include "te_batch.cuh"
#include "te_internal.cuh"

__constant__ TeQuadTables c_quad;
// The abscissae and weights again in global memory: lanes read different nodes
// at once, which constant memory serves one by one.
__device__ TeQuadTables g_quad;
constexpr int kTsFirst = 3;        // tanh-sinh levels evaluated at once
constexpr int kTsFirstNodes = 25;  // their nodes

#define TE_KBUF 8  // outputs per coefficient group
#define TE_KTHREADS 128  // threads per block: one warp per scheduler
#define TE_KCLUSTER 8    // blocks of a cluster at most

// One integral of the search: its interval and rule (method < 0: none), the
// same in every block, and what the block that evaluated it found.
struct KIntegral {
  double a, b;
  int method;
  int K;  // series length at the interval's end
};
struct KValue {
  double value;
  int state;  // 4 round + 1, or + 3 when the quadrature missed its accuracy
};

struct KSmem {
  double tc[(TE_NCHEB + 1) * TE_MMAX];  // Chebyshev vectors, row n
  double fp[TE_TS_NODES], fm[TE_TS_NODES];
  double Q[TE_MMAX * TE_MMAX];          // eigenvectors (col-major), fallback path
  union {
    double J[TE_SCAP + 1][TE_NCHEB + 8];  // Bessel values per output
    struct {  // integrals: J_k between the two warps of an argument set (2 blocks of 16 steps, J_0)
      double ring[2][2][17][32];
      int rescaled[2][2][4][32];  // after every fourth step of a block
    };
  };
  double lam[TE_MMAX];
  double d[TE_MMAX], e[TE_MMAX], dd[TE_MMAX], ee[TE_MMAX];
  double gs[TE_NCHEB + 8];              // signed, doubled last components of t_n
  double s[TE_MMAX];                    // column scales
  double tsu[kTsFirstNodes], tsw[kTsFirstNodes];  // tanh-sinh nodes and weights of the first levels
  double rc[TE_MMAX], rs[TE_MMAX];      // rotations of one QR sweep
  double lev[TE_TS_KMAX + 1][2];        // level sums of the tanh-sinh rule
  int bad[TE_TS_KMAX + 1];
  double bc[16];
  int ibc[16];
  KIntegral spec[TE_KCLUSTER];          // the last round of integrals (this block's copy)
  KValue found[2][TE_KCLUSTER];         // their values, by round parity, stored by the blocks that evaluated them
  double dts[TE_SCAP + 1];              // times of this launch's outputs
  double trig[TE_SCAP + 1][2];
  double inv[TE_SCAP + 1];              // 1 / normalisation of the tables
  int outK[3];                          // series lengths: start vector, samples 0..7, samples 8..15
};

static_assert(sizeof(KSmem) + 4096 <= 232448, "Krylov kernel shared memory exceeds the per-block limit");

__device__ __forceinline__ double warp_sum_all(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Miller start index (multiple of 4) for accurate J_n(z), n <= max(m, z).
__device__ __forceinline__ int bessel_start(double z, int m) {
  double a = fmax((double)m, z);
  double k0 = a + 25.0 + 2.0 * sqrt(a);
  if (!(k0 < 1e6)) return 1 << 30;
  return 4 * (int)ceil(k0 * 0.25);
}

__device__ __forceinline__ bool needs_rescale(double v) {
  int hi = __double2hiint(v);
  return ((hi >> 20) & 0x7ff) > 1023 + 600;
}

struct KCtx {
  TeDevState* ds;
  KSmem* sm;
  int rank, size;  // block of the cluster; rank 0 writes the state
  int round;       // rounds of integrals so far
  int n_integrals;
  int ts_kmax;     // deepest tanh-sinh level
  int m;
  double h, rho, c;
  int cheb_n;     // Chebyshev vectors available up to this degree
  bool eig_ok;    // eigen-decomposition available
  int fatal;
};

// ------------------------------------------------------------ Chebyshev

// Extend t_n (and the signed last components gs) up to degree K
// (block-cooperative; K >= 2).
__device__ void ensure_cheb(KCtx& C, int K) {
  if (K <= C.cheb_n) return;
  KSmem* S = C.sm;
  const int m = C.m;
  const int j = threadIdx.x;
  const int old = C.cheb_n;
  int n0 = old;
  if (old < 0) {
    if (j < TE_MMAX) S->tc[j] = (j == 0) ? 1.0 : 0.0;
    __syncthreads();
    if (j < TE_MMAX) {
      double v = 0.0;
      if (j < m) {
        v = 0.5 * S->dd[j] * S->tc[j];
        if (j > 0) v = fma(0.5 * S->ee[j - 1], S->tc[j - 1], v);
        if (j + 1 < m) v = fma(0.5 * S->ee[j], S->tc[j + 1], v);
      }
      S->tc[TE_MMAX + j] = v;
    }
    __syncthreads();
    n0 = 1;
  }
  for (int n = n0; n < K; ++n) {
    if (j < TE_MMAX) {
      const double* tn = S->tc + n * TE_MMAX;
      const double* tp = S->tc + (n - 1) * TE_MMAX;
      double v = 0.0;
      if (j < m) {
        v = fma(S->dd[j], tn[j], -tp[j]);
        if (j > 0) v = fma(S->ee[j - 1], tn[j - 1], v);
        if (j + 1 < m) v = fma(S->ee[j], tn[j + 1], v);
      }
      S->tc[(n + 1) * TE_MMAX + j] = v;
    }
    __syncthreads();
  }
  // signed doubled last components: R uses even n, I odd n
  for (int n = old + 1 + threadIdx.x; n <= K; n += blockDim.x) {
    const double g = S->tc[n * TE_MMAX + (m - 1)];
    const int r = n & 3;
    S->gs[n] = (n == 0) ? g : ((r == 0 || r == 3) ? 2.0 * g : -2.0 * g);
  }
  C.cheb_n = K;
  __syncthreads();
}

// Integrand h |e_m^T exp(-i x T) e_1| by Chebyshev-Bessel, K iterations (a
// multiple of 4), at nev arguments x = arg(e), results through put(e, value)
// (block-cooperative).  Warps 0..3 form two sets of 32 arguments: the even warp
// of a set runs J_{k-1} = f_k J_k - J_{k+1}, f_{k-1} = f_k - 2 / z, the odd one
// the sums of the signed components and the normalisation.
template <class Arg, class Put>
__device__ void integrand_series(const KCtx& C, int nev, int K, Arg arg, Put put) {
  KSmem* S = C.sm;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, set = warp >> 1;
  if (warp < 4) {
    // named barriers of the set: ring block b full / empty again
    auto sync = [&](int id) { asm volatile("bar.sync %0, 64;" ::"r"(id + 4 * set) : "memory"); };
    auto arrive = [&](int id) { asm volatile("bar.arrive %0, 64;" ::"r"(id + 4 * set) : "memory"); };
    const int blocks = (K + 15) / 16;
    for (int e0 = 32 * set; e0 < nev; e0 += 64) {
      const double x = arg(min(e0 + lane, nev - 1));
      double z = x * C.rho;
      const bool tiny = !(z > 1e-200);
      if (tiny) z = 1.0;
      if ((warp & 1) == 0) {
        const double inv2z = 2.0 / z;
        double jp1 = 0.0, jk = 1e-200, f = (double)K * inv2z;
        for (int b = 0; b < blocks; ++b) {
          if (b >= 2) sync(3 + (b & 1));
          double(*J)[32] = S->ring[set][b & 1];
          const int steps = min(16, K - 16 * b);
          for (int q4 = 0; q4 < steps; q4 += 4) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              J[q4 + q][lane] = jk;
              const double jm = fma(f, jk, -jp1);
              f -= inv2z;
              jp1 = jk;
              jk = jm;
            }
            const bool big = needs_rescale(jk);
            S->rescaled[set][b & 1][q4 >> 2][lane] = big;
            if (big) {
              jk *= 0x1p-600;
              jp1 *= 0x1p-600;
            }
          }
          J[16][lane] = jk;  // J_0 in the last block
          arrive(1 + (b & 1));
        }
      } else {
        const double* gs = S->gs;
        double R = 0.0, I = 0.0, nrm = 0.0;
        for (int b = 0; b < blocks; ++b) {
          sync(1 + (b & 1));
          double(*J)[32] = S->ring[set][b & 1];
          const int steps = min(16, K - 16 * b);
          for (int q4 = 0; q4 < steps; q4 += 4) {
            const int k = K - 16 * b - q4;
            const double j0 = J[q4][lane], j2 = J[q4 + 2][lane];
            R = fma(gs[k], j0, R);
            nrm = fma(2.0, j0, nrm);
            I = fma(gs[k - 1], J[q4 + 1][lane], I);
            R = fma(gs[k - 2], j2, R);
            nrm = fma(2.0, j2, nrm);
            I = fma(gs[k - 3], J[q4 + 3][lane], I);
            if (S->rescaled[set][b & 1][q4 >> 2][lane]) {
              R *= 0x1p-600;
              I *= 0x1p-600;
              nrm *= 0x1p-600;
            }
          }
          if (b + 1 == blocks) {
            const double j0 = J[16][lane];  // unnormalised
            nrm += j0;
            R = fma(gs[0], j0, R);
          }
          if (b + 2 < blocks) arrive(3 + (b & 1));
        }
        const double v = tiny ? ((C.m == 1) ? C.h * fabs(gs[0]) : 0.0) : C.h * hypot(R, I) / fabs(nrm);
        if (e0 + lane < nev) put(e0 + lane, v);
      }
      sync(3);  // the ring is free for the next arguments
    }
  }
  __syncthreads();
}

// Bessel values J_0..J_K(z), unnormalised, into out[] (one thread); returns
// their normalisation.
__device__ double bessel_table(double z, int K, double* out) {
  if (!(z > 1e-200)) {
    for (int k = 0; k <= K; ++k) out[k] = (k == 0) ? 1.0 : 0.0;
    return 1.0;
  }
  const double inv2z = 2.0 / z;
  double jp1 = 0.0, jk = 1e-200, nrm = 0.0;
  double f = (double)K * inv2z;
  out[K] = jk;
  for (int k = K; k >= 1; --k) {
    if ((k & 1) == 0) nrm = fma(2.0, jk, nrm);
    double jm = fma(f, jk, -jp1);
    f -= inv2z;
    jp1 = jk;
    jk = jm;
    out[k - 1] = jk;
    if (needs_rescale(jk)) {
      const double sc = 0x1p-600;
      for (int q = k - 1; q <= K; ++q) out[q] *= sc;
      jk = out[k - 1];
      jp1 *= sc;
      nrm *= sc;
    }
  }
  return nrm + jk;
}

// ------------------------------------------------------------ eigen path

// Implicit symmetric tridiagonal QR with Wilkinson shifts, warp 0 only.
// Q (col-major, ld TE_MMAX) must hold the identity on entry.  Returns 0 on
// success, 1 if the sweep limit was reached.
__device__ int tridiag_qr_warp(int m, double* d, double* e, double* Q, double* rc, double* rs, int max_sweeps) {
  const int lane = threadIdx.x & 31;
  int q = m - 1;
  int sweeps = 0;
  while (true) {
    int p_out = 0, q_out = 0;
    if (lane == 0) {
      for (int i = 0; i < q; ++i)
        if (fabs(e[i]) <= DBL_EPSILON * (fabs(d[i]) + fabs(d[i + 1]))) e[i] = 0.0;
      while (q > 0 && e[q - 1] == 0.0) --q;
      int p = q;
      if (q > 0) {
        p = q - 1;
        while (p > 0 && e[p - 1] != 0.0) --p;
        // Wilkinson shift from the trailing 2x2 block
        double dl = d[q - 1], dq = d[q], eq = e[q - 1];
        double delta = 0.5 * (dl - dq);
        double rr = hypot(delta, eq);
        double den = delta + (delta >= 0.0 ? rr : -rr);
        double mu = (den != 0.0) ? dq - eq * eq / den : dq - fabs(eq);
        double x = d[p] - mu, zz = e[p];
        for (int k = p; k < q; ++k) {
          double r = hypot(x, zz);
          double cs = 1.0, sn = 0.0;
          if (r != 0.0) {
            cs = x / r;
            sn = zz / r;
          }
          if (k > p) e[k - 1] = r;
          double a = d[k], b = e[k], dd2 = d[k + 1];
          double cc = cs * cs, ss = sn * sn, csn = cs * sn;
          d[k] = cc * a + 2.0 * csn * b + ss * dd2;
          d[k + 1] = ss * a - 2.0 * csn * b + cc * dd2;
          e[k] = csn * (dd2 - a) + (cc - ss) * b;
          if (k + 1 < q) {
            double bulge = sn * e[k + 1];
            e[k + 1] = cs * e[k + 1];
            x = e[k];
            zz = bulge;
          }
          rc[k] = cs;
          rs[k] = sn;
        }
      }
      p_out = p;
      q_out = q;
    }
    q = __shfl_sync(0xffffffffu, q_out, 0);
    int p = __shfl_sync(0xffffffffu, p_out, 0);
    if (q == 0) break;
    __syncwarp();
    for (int row = lane; row < m; row += 32) {
      double a = Q[p * TE_MMAX + row];
      for (int k = p; k < q; ++k) {
        double b = Q[(k + 1) * TE_MMAX + row];
        double cs = rc[k], sn = rs[k];
        Q[k * TE_MMAX + row] = cs * a + sn * b;
        a = -sn * a + cs * b;
      }
      Q[q * TE_MMAX + row] = a;
    }
    __syncwarp();
    if (++sweeps > max_sweeps) return 1;
  }
  return 0;
}

// Eigen-decomposition of T into sm->lam / sm->Q (block-cooperative call).
__device__ void ensure_eig(KCtx& C) {
  if (C.eig_ok) return;
  KSmem* S = C.sm;
  __shared__ double dtmp[TE_MMAX], etmp[TE_MMAX];
  const int m = C.m;
  for (int i = threadIdx.x; i < TE_MMAX * TE_MMAX; i += blockDim.x) {
    int r = i % TE_MMAX, c = i / TE_MMAX;
    S->Q[i] = (r == c) ? 1.0 : 0.0;
  }
  if (threadIdx.x < TE_MMAX) {
    dtmp[threadIdx.x] = threadIdx.x < m ? S->d[threadIdx.x] : 0.0;
    etmp[threadIdx.x] = threadIdx.x + 1 < m ? S->e[threadIdx.x] : 0.0;
  }
  __syncthreads();
  int fail = 0;
  const int max_sweeps = C.ds->qr_sweeps > 0 ? C.ds->qr_sweeps : 40 * m + 40;
  if (threadIdx.x < 32) fail = tridiag_qr_warp(m, dtmp, etmp, S->Q, S->rc, S->rs, max_sweeps);
  if (threadIdx.x == 0) S->ibc[0] = fail;
  __syncthreads();
  if (S->ibc[0] && threadIdx.x == 0) C.ds->fatal = TE_ERR_EIGEN;
  if (threadIdx.x < m) S->lam[threadIdx.x] = dtmp[threadIdx.x];
  C.eig_ok = true;
  __syncthreads();
}

__device__ double integrand_eig(const KCtx& C, double x) {
  const KSmem* S = C.sm;
  const int m = C.m;
  double re = 0.0, im = 0.0;
  for (int k = 0; k < m; ++k) {
    double ck = S->Q[k * TE_MMAX + (m - 1)] * S->Q[k * TE_MMAX];
    double sn, cs;
    sincos(x * S->lam[k], &sn, &cs);
    re = fma(ck, cs, re);
    im = fma(-ck, sn, im);
  }
  return C.h * hypot(re, im);
}

// ------------------------------------------------------------ quadrature

struct IntResult {
  double value, err;
  bool nonfinite;
};

// Evaluate the integrand at the abscissae of nodes [n0, n1) of the tanh-sinh
// table on [a, b] into sm->fp / sm->fm (block-cooperative); t = 0 once.
__device__ void eval_ts_nodes(KCtx& C, double a, double b, int n0, int n1, bool use_eig, int K) {
  KSmem* S = C.sm;
  const double c = 0.5 * (a + b), d = 0.5 * (b - a);
  const int skip = n0 == 0 ? 1 : 0;  // node 0 has no minus side
  const int nev = 2 * (n1 - n0) - skip;
  auto node = [&](int e) { return n0 + ((e + skip) >> 1); };
  auto minus = [&](int e) { return ((e + skip) & 1) != 0 && node(e) != 0; };
  auto arg = [&](int e) {
    const int i = node(e);
    const double u = i < kTsFirstNodes ? S->tsu[i] : g_quad.ts_u[i];
    return minus(e) ? c - d * u : c + d * u;
  };
  auto put = [&](int e, double f) { (minus(e) ? S->fm : S->fp)[node(e)] = f; };
  if (!use_eig) {
    integrand_series(C, nev, K, arg, put);
    return;
  }
  for (int e = threadIdx.x; e < nev; e += blockDim.x) put(e, integrand_eig(C, arg(e)));
  __syncthreads();
}

// The level's weighted sums on one warp.
__device__ void ts_level_sum(KCtx& C, int k) {
  KSmem* S = C.sm;
  const int* lb = c_quad.ts_level_begin;
  double s = 0.0, sa = 0.0;
  bool bad = false;
  for (int node = lb[k] + (int)(threadIdx.x & 31); node < lb[k + 1]; node += 32) {
    const double w = node < kTsFirstNodes ? S->tsw[node] : g_quad.ts_w[node];
    if (node == 0) {
      double fv = S->fp[0];
      s = fma(w, fv, s);
      sa = fma(w, fabs(fv), sa);
      bad |= !isfinite(fv);
    } else {
      double f1 = S->fp[node], f2 = S->fm[node];
      s = fma(w, f1 + f2, s);
      sa = fma(w, fabs(f1) + fabs(f2), sa);
      bad |= !isfinite(f1) || !isfinite(f2);
    }
  }
  s = warp_sum_all(s);
  sa = warp_sum_all(sa);
  bad = __any_sync(0xffffffffu, bad);
  if ((threadIdx.x & 31) == 0) {
    S->lev[k][0] = s;
    S->lev[k][1] = sa;
    S->bad[k] = bad ? 1 : 0;
  }
}

// Tanh-sinh integral of the error integrand on [a, b].
__device__ IntResult ts_integrate(KCtx& C, double a, double b, int K, bool use_eig) {
  KSmem* S = C.sm;
  IntResult res = {0.0, 0.0, false};
  if (!(b > a)) return res;
  if (use_eig)
    ensure_eig(C);
  else
    ensure_cheb(C, K);
  const double d = 0.5 * (b - a);
  const int* lb = c_quad.ts_level_begin;
  eval_ts_nodes(C, a, b, 0, kTsFirstNodes, use_eig, K);
  const int warp = threadIdx.x >> 5;
  if (warp <= kTsFirst) ts_level_sum(C, warp);
  __syncthreads();
  double sum = 0.0, sum_abs = 0.0, prev = 0.0;
  bool nonfinite = false;
  const int kmax = C.ts_kmax;
  // levels 0..3 side by side: lane k of every warp holds the sums up to level
  // k (added in order), so their estimates take one round of FP64 instructions
  const int lane = threadIdx.x & 31, kl = min(lane, kTsFirst);
  double s = 0.0, sa = 0.0;
#pragma unroll
  for (int k = 0; k <= kTsFirst; ++k) {
    const double ns = s + S->lev[k][0], nsa = sa + S->lev[k][1];
    if (k <= kl) s = ns, sa = nsa;
  }
  {
    const double hk = __hiloint2double((1023 - kl) << 20, 0);  // 2^-k
    const double Ik = d * hk * s, L1 = d * hk * sa;
    const double err = fabs(Ik - __shfl_up_sync(0xffffffffu, Ik, 1));
    const bool stop = kl >= TE_TS_KMIN && err <= 1e-3 * L1;
    const unsigned int done = __ballot_sync(0xffffffffu, (stop || kl == kmax) && lane <= kTsFirst);
    const int k = done ? __ffs(done) - 1 : kTsFirst;
    res.value = __shfl_sync(0xffffffffu, Ik, k);
    res.err = __shfl_sync(0xffffffffu, err, k);
    for (int i = 0; i <= k; ++i) nonfinite |= S->bad[i] != 0;
    sum = __shfl_sync(0xffffffffu, s, k);
    sum_abs = __shfl_sync(0xffffffffu, sa, k);
    prev = res.value;
    if (done) {
      res.nonfinite = nonfinite;
      __syncthreads();
      return res;
    }
  }
  for (int k = kTsFirst + 1; k <= kmax; ++k) {
    eval_ts_nodes(C, a, b, lb[k], lb[k + 1], use_eig, K);
    if (warp == 0) ts_level_sum(C, k);
    __syncthreads();
    sum += S->lev[k][0];
    sum_abs += S->lev[k][1];
    nonfinite |= S->bad[k] != 0;
    const double hk = __hiloint2double((1023 - k) << 20, 0);  // 2^-k
    const double Ik = d * hk * sum;
    const double L1 = d * hk * sum_abs;
    res.value = Ik;
    res.err = fabs(Ik - prev);
    if (res.err <= 1e-3 * L1) break;
    prev = Ik;
  }
  res.nonfinite = nonfinite;
  __syncthreads();
  return res;
}

__device__ double gauss_integrate(KCtx& C, double a, double b, int npts, int K, bool use_eig) {
  KSmem* S = C.sm;
  const double* xs = npts == 15 ? c_quad.g15_x : c_quad.g7_x;
  const double* ws = npts == 15 ? c_quad.g15_w : c_quad.g7_w;
  const double c = 0.5 * (a + b), d = 0.5 * (b - a);
  if (use_eig)
    ensure_eig(C);
  else
    ensure_cheb(C, K);
  auto arg = [&](int e) { return c + d * xs[e]; };
  if (use_eig) {
    if ((int)threadIdx.x < npts) S->fp[threadIdx.x] = integrand_eig(C, arg(threadIdx.x));
    __syncthreads();
  } else {
    integrand_series(C, npts, K, arg, [&](int e, double f) { S->fp[e] = f; });
  }
  if (threadIdx.x < 32) {
    double s = (int)threadIdx.x < npts ? ws[threadIdx.x] * S->fp[threadIdx.x] : 0.0;
    s = warp_sum_all(s);
    if (threadIdx.x == 0) S->bc[0] = s;
  }
  __syncthreads();
  double r = d * S->bc[0];
  __syncthreads();
  return r;
}

// One integral of the search on this block (integrateError,
// core/krylovTimeEvolver.cpp:584-618); only the block that runs the
// eigen-decomposition path (rank 0) evaluates arguments beyond the series.
// Returns whether the quadrature was accurate.
__device__ bool eval_integral(KCtx& C, const KIntegral& q, double tolRate, double& ret) {
  TeDevState* ds = C.ds;
  const double a = q.a, b = q.b;
  const int K = q.K;
  const bool use_eig = K > TE_NCHEB;
  double error = 0.0;
  if (q.method == 0) {
    ret = gauss_integrate(C, a, b, 15, K, use_eig);
  } else if (q.method == 1) {
    ret = gauss_integrate(C, a, b, 7, K, use_eig);
  } else {
    IntResult r = ts_integrate(C, a, b, K, use_eig);
    if (r.nonfinite) {
      ret = ds->tol * 10.0;  // the reference's response to a failed quadrature (:601-605)
    } else {
      ret = r.value;
      error = r.err;
    }
  }
  return !(q.method == 2 && error / ret > 1e-3 && ret > 1e-3 * (b - a) * tolRate);
}

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ unsigned int cluster_addr(const void* p, int rank) {
  unsigned int a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((unsigned int)__cvta_generic_to_shared(p)), "r"(rank));
  return a;
}

// What the search may ask for next, after [0, t] (from = 0: and the doublings
// or the halvings and substeps that follow) or substep n of t.
struct KNext {
  double t, t_max;
  int n_substeps;
  int n;        // 0: an interval [0, t]; else substep n
  bool doubling;
  int method_long, method_short;
};

// The value of one integral the search asks for: from the last round when it
// is there, else a new round with it and the likely next ones, one per block.
__device__ double integrate_error(KCtx& C, double a, double b, int method, double tolRate, bool& successful,
                                  const KNext& nx) {
  KSmem* S = C.sm;
  ++C.n_integrals;
  int hit = -1;
  for (int i = 0; i < C.size; ++i) {
    const KIntegral& q = S->spec[i];
    if (q.method == method && __double_as_longlong(q.a) == __double_as_longlong(a) &&
        __double_as_longlong(q.b) == __double_as_longlong(b) && (S->found[C.round & 1][i].state >> 2) == C.round) {
      hit = i;
      break;
    }
  }
  if (hit < 0) {
    ++C.round;
    __syncthreads();
    if ((int)threadIdx.x < C.size) {
      const int i = threadIdx.x;
      KIntegral q{a, b, method, 0};
      bool use = true;
      if (i > 0) {
        int n = nx.n + i;  // substeps after substep n
        if (nx.n == 0 && nx.doubling) {
          n = 0;
          double t = nx.t;
          for (int k = 0; k < i; ++k) t *= 2;
          // the doubling loop stops at t_max: only its first clipped value counts
          use = t < 2 * nx.t_max;
          q.a = 0.0;
          q.b = t > nx.t_max ? nx.t_max : t;
        } else if (nx.n == 0) {
          n = i - 1;
          if (i == 1) {
            q.a = 0.0;
            q.b = nx.t / 2.0;
          }
          use = i == 1 || nx.t < nx.t_max;
        }
        if (n > 0) {
          const double s = nx.t / nx.n_substeps;
          q.a = nx.t + (n - 1) * s;
          q.b = nx.t + n * s;
          q.method = nx.method_short;
        }
      }
      q.K = bessel_start(fmax(fabs(q.a), fabs(q.b)) * C.rho, C.m);
      // arguments beyond the series take the eigen-decomposition: only when asked for
      if (!use || (i > 0 && q.K > TE_NCHEB)) q.method = -1;
      S->spec[i] = q;
    }
    __syncthreads();
    const KIntegral mine = S->spec[C.rank];
    if (mine.method >= 0) {
      double v;
      const bool good = eval_integral(C, mine, tolRate, v);
      if ((int)threadIdx.x < C.size) {
        KValue* f = &S->found[C.round & 1][C.rank];
        const int st = 4 * C.round + (good ? 1 : 3);
        if (C.size > 1) {
          asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(cluster_addr(&f->value, threadIdx.x)), "d"(v) : "memory");
          asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(cluster_addr(&f->state, threadIdx.x)), "r"(st)
                       : "memory");
        } else {
          f->value = v;
          f->state = st;
        }
      }
    }
    if (C.size > 1)
      cluster_barrier();
    else
      __syncthreads();
    hit = 0;
  }
  const KValue& f = S->found[C.round & 1][hit];
  if ((f.state & 2) != 0) successful = false;
  return f.value;
}

// findMaximalStepSize (core/krylovTimeEvolver.cpp:153-254).  Returns the
// code (0/1/20/21) or -1 when 20 halvings did not suffice.
__device__ int find_step(KCtx& C, double tolRate, double t_stepSuggestion, double t_step_max, int n_substeps,
                         double numericalErrorEstimate, bool increaseStep, double* t_stepRet, double* err_stepRet) {
  TeDevState* ds = C.ds;
  const int mlong = ds->integ_long, mshort = ds->integ_short;
  const unsigned GO_MAX = 20;
  unsigned nbReductions = 0;
  double t_step = t_stepSuggestion;
  int code = 0;
  bool ok = true;
  bool skipSubsteps = false;
  if (t_step > t_step_max) {
    t_step = t_step_max;
    skipSubsteps = true;
  }
  // candidates for the other blocks: what follows an interval [0, t] or substep n
  auto next = [&](double t, int n, bool doubling) {
    return KNext{t, t_step_max, n_substeps, n, doubling, mlong, mshort};
  };
  double err_step =
      integrate_error(C, 0.0, t_step, mlong, tolRate, ok, next(t_step, 0, increaseStep && !skipSubsteps));
  if (increaseStep && !skipSubsteps) {
    double err_new = err_step, t_new = t_step;
    int guard = 0;
    while (err_new < tolRate * t_new && t_step < t_step_max && guard++ < 4096) {
      t_step = t_new;
      err_step = err_new;
      if (t_step >= t_step_max) {
        skipSubsteps = true;
        break;
      }
      t_new *= 2;
      if (t_new > t_step_max) t_new = t_step_max;
      err_new = integrate_error(C, 0.0, t_new, mlong, tolRate, ok, next(t_new, 0, true));
    }
  }
  while (err_step > tolRate * t_step) {
    nbReductions++;
    t_step = t_step / 2.0;
    err_step = integrate_error(C, 0.0, t_step, mlong, tolRate, ok, next(t_step, 0, false));
    if (nbReductions == GO_MAX) return -1;
    skipSubsteps = false;
  }
  const double s = t_step / n_substeps;
  int n_s = 0;
  double deltaError = 0.0;
  if (!skipSubsteps) {
    while (err_step + deltaError < tolRate * (t_step + n_s * s)) {
      err_step += deltaError;
      n_s++;
      if (t_step + (n_s - 1) * s >= t_step_max) break;
      if (n_s > (1 << 22)) return -2;
      deltaError =
          integrate_error(C, t_step + (n_s - 1) * s, t_step + n_s * s, mshort, tolRate, ok, next(t_step, n_s, false));
    }
    t_step += (n_s - 1) * s;
  }
  if (err_step < numericalErrorEstimate) {
    if (!skipSubsteps || err_step > 0.1 * tolRate * t_step) code += 1;
  }
  if (!ok) code += 20;
  *t_stepRet = t_step;
  *err_stepRet = err_step;
  return code;
}

// ------------------------------------------------------- coefficient vectors

// Y[slot] = s_j i^j [exp(-i dt T) e_1]_j for the outputs of a launch: S->dts[0]
// (slot 0) when want_w, and the samples S->dts[1..cnt] (slot = index).  The
// start vector and each group of TE_KBUF samples share a series length.  The
// start vector goes to the last block of the cluster, samples round the blocks;
// each block runs all its tables at once (a warp per group).
__device__ void output_coefficients(KCtx& C, bool want_w, int cnt) {
  KSmem* S = C.sm;
  TeDevState* ds = C.ds;
  const int m = C.m;
  if (threadIdx.x < 3) {
    const int q = threadIdx.x, o0 = q == 0 ? 0 : 1 + (q - 1) * TE_KBUF;
    const int o1 = q == 0 ? (want_w ? 1 : 0) : min(o0 + TE_KBUF, cnt + 1);
    double zmax = 0.0;
    for (int o = o0; o < o1; ++o) zmax = fmax(zmax, fabs(S->dts[o]) * C.rho);
    S->outK[q] = o1 > o0 ? bessel_start(zmax, m) : 0;
  }
  __syncthreads();
  auto group = [](int o) { return o == 0 ? 0 : 1 + (o - 1) / TE_KBUF; };
  // own outputs: o = first, first + size, ...; the start vector on the last block
  const bool own_w = want_w && C.rank == C.size - 1;
  const int first = 1 + C.rank;
  const int own = (own_w ? 1 : 0) + (first <= cnt ? (cnt - first) / C.size + 1 : 0);
  auto output = [&](int i) { return own_w ? (i == 0 ? 0 : first + (i - 1) * C.size) : first + i * C.size; };
  int K = 0;
  bool eig = false;
  for (int q = 0; q < 3; ++q) {
    if (S->outK[q] > TE_NCHEB)
      eig = true;
    else
      K = max(K, S->outK[q]);
  }
  if (eig && C.rank == 0) {  // one eigen-decomposition, on rank 0, for whole groups
    ensure_eig(C);
    for (int o = want_w ? 0 : 1; o <= cnt; ++o) {
      if (S->outK[group(o)] <= TE_NCHEB) continue;
      for (int j = threadIdx.x; j < m; j += blockDim.x) {
        const double dt = S->dts[o];
        double re = 0.0, im = 0.0;
        for (int k = 0; k < m; ++k) {
          double q = S->Q[k * TE_MMAX + j] * S->Q[k * TE_MMAX];
          double sn, cs;
          sincos(dt * S->lam[k], &sn, &cs);
          re = fma(q, cs, re);
          im = fma(-q, sn, im);
        }
        double yr, yi;
        switch (j & 3) {
          case 0: yr = re; yi = im; break;
          case 1: yr = -im; yi = re; break;
          case 2: yr = -re; yi = -im; break;
          default: yr = im; yi = -re; break;
        }
        const double sj = S->s[j];
        ds->Y[o * TE_MMAX + j] = make_double2(yr * sj, yi * sj);
      }
    }
  }
  if (own == 0 || K == 0) {
    __syncthreads();
    return;
  }
  ensure_cheb(C, K);
  // tables: a warp per group, a lane per output; the phases on the last warp
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp < 3) {
    if (lane < own && group(output(lane)) == warp && S->outK[warp] <= TE_NCHEB)
      S->inv[lane] = 1.0 / bessel_table(S->dts[output(lane)] * C.rho, S->outK[warp], S->J[lane]);
  } else if (warp == 3 && lane < own) {
    sincos(S->dts[output(lane)] * C.c, &S->trig[lane][0], &S->trig[lane][1]);
  }
  __syncthreads();
  // signed coefficients eps_n sigma_n J_n (sigma: + for n%4 in {0,3}, - otherwise)
  for (int i = threadIdx.x; i < own * (K + 1); i += blockDim.x) {
    const int o = i / (K + 1), n = i % (K + 1);
    if (n > S->outK[group(output(o))]) continue;
    const double sg = ((n & 3) == 0 || (n & 3) == 3) ? 1.0 : -1.0;
    S->J[o][n] = (S->J[o][n] * S->inv[o]) * ((n == 0) ? 1.0 : 2.0 * sg);
  }
  __syncthreads();
  // the even terms (re) and the odd ones (im) of a component on their own
  // lanes, then times e^{-i dt c}
  for (int i0 = 0; i0 < 2 * own * m; i0 += blockDim.x) {
    const int i = min(i0 + (int)threadIdx.x, 2 * own * m - 1);
    const int c = i & 1, o = (i >> 1) / m, j = (i >> 1) % m;
    const int out = output(o), Ko = S->outK[group(out)];
    const bool live = i0 + (int)threadIdx.x < 2 * own * m && Ko <= TE_NCHEB;
    const double* a = S->J[o];
    double v = 0.0;
    if (live) {
#pragma unroll 4
      for (int n = c; n <= Ko; n += 2) v = fma(a[n], S->tc[n * TE_MMAX + j], v);
    }
    const double w = __shfl_xor_sync(0xffffffffu, v, 1);
    const double sn = S->trig[o][0], cs = S->trig[o][1];
    // re' = re cs + im sn, im' = im cs - re sn
    const double x = v * cs, y = w * sn;
    const double t = c == 0 ? x + y : x - y;
    // times i^j, then the column scale s_j of the unnormalised basis
    const double other = __shfl_xor_sync(0xffffffffu, t, 1);
    const double re = c == 0 ? t : other, im = c == 0 ? other : t;
    double yv;
    switch (j & 3) {
      case 0: yv = c == 0 ? re : im; break;
      case 1: yv = c == 0 ? -im : re; break;
      case 2: yv = c == 0 ? -re : -im; break;
      default: yv = c == 0 ? im : -re; break;
    }
    if (live) reinterpret_cast<double*>(&ds->Y[out * TE_MMAX + j])[c] = yv * S->s[j];
  }
  __syncthreads();
}

// Schedule the next batch of samples of the current Krylov space (the
// while-condition of :405) and compute their coefficients, with the step's
// next start vector (want_w: at t_step) before them.  When the batch exhausts
// the step, advance t_now and err (:440-441) and open the next step.
__device__ void schedule_batch(KCtx& C, double t_step, bool want_w) {
  TeDevState* ds = C.ds;
  KSmem* S = C.sm;
  // every block finds the batch's times; rank 0 alone writes the state, once
  // all have read it
  int idx = ds->index_samples, cnt = 0;
  double ts = ds->t_sampling;
  const int base = idx;
  const double t = ds->t, ss = ds->sampling_step, t_now = ds->t_now;
  const double t_end = t_now + t_step;
  const int ns = ds->n_samples, max_batch = ds->max_batch;
  const double* times = ds->sample_times;
  auto cond = [&](int i, double tsv) {
    if (i >= ns) return false;
    const double next = times ? times[i] : tsv + ss;
    return next <= t_end || (i == ns - 1 && fabs(t_end - t) <= DBL_EPSILON);
  };
  while (cnt < max_batch && cond(idx, ts)) {
    ts = times ? times[idx] : ts + ss;
    if (threadIdx.x == 0) S->dts[1 + cnt] = ts - t_now;
    ++cnt;
    ++idx;
  }
  const bool pending = cond(idx, ts);
  if (threadIdx.x == 0) S->dts[0] = t_step;
  __syncthreads();
  if (C.size > 1) cluster_barrier();
  if (C.rank == 0 && threadIdx.x == 0) {
    ds->sample_base = base;
    ds->t_sampling = ts;
    ds->index_samples = idx;
    ds->samples_in_batch = cnt;
    ds->samples_pending = pending ? 1 : 0;
    if (!pending) {
      ds->t_now += ds->t_step;
      ds->err += ds->err_step;
      if (idx < ns) {
        ds->n_steps++;
        ds->breakdown = 0;
      } else {
        ds->done = 1;
      }
    }
  }
  output_coefficients(C, want_w, cnt);
}

// Load T from the Lanczos coefficients and set up the Chebyshev data.
__device__ void setup_krylov_matrix(KCtx& C) {
  TeDevState* ds = C.ds;
  KSmem* S = C.sm;
  const int m = C.m;
  if ((int)threadIdx.x >= TE_MMAX && (int)threadIdx.x < TE_MMAX + kTsFirstNodes) {
    const int i = threadIdx.x - TE_MMAX;
    S->tsu[i] = g_quad.ts_u[i];
    S->tsw[i] = g_quad.ts_w[i];
  }
  if (threadIdx.x < TE_MMAX) {
    int j = threadIdx.x;
    S->d[j] = j < m ? -ds->alpha[j].y : 0.0;
    S->e[j] = j + 1 < m ? ds->beta[j + 1] : 0.0;
    if (C.rank == 0) {
      ds->d[j] = S->d[j];
      ds->e[j] = S->e[j];
    }
  }
  __syncthreads();
  // Gershgorin interval on warp 0
  if (threadIdx.x < 32) {
    double lo = INFINITY, hi = -INFINITY;
    for (int j = threadIdx.x; j < m; j += 32) {
      double r = fabs(S->e[j]) + (j > 0 ? fabs(S->e[j - 1]) : 0.0);
      lo = fmin(lo, S->d[j] - r);
      hi = fmax(hi, S->d[j] + r);
    }
    // as integers of the same order: minima and maxima off the FP64 pipe
    auto key = [](double v) {
      const long long b = __double_as_longlong(v);
      return b < 0 ? b ^ 0x7fffffffffffffffll : b;
    };
    long long klo = key(lo), khi = key(hi);
    for (int o = 16; o > 0; o >>= 1) {
      klo = min(klo, __shfl_xor_sync(0xffffffffu, klo, o));
      khi = max(khi, __shfl_xor_sync(0xffffffffu, khi, o));
    }
    lo = __longlong_as_double(klo < 0 ? klo ^ 0x7fffffffffffffffll : klo);
    hi = __longlong_as_double(khi < 0 ? khi ^ 0x7fffffffffffffffll : khi);
    if (threadIdx.x == 0) {
      double c = 0.5 * (hi + lo), rho = 0.5 * (hi - lo);
      if (!(rho > 1e-300 * fmax(1.0, fabs(c)))) rho = 1.0;
      S->bc[2] = c;
      S->bc[3] = rho;
    }
  }
  __syncthreads();
  C.c = S->bc[2];
  C.rho = S->bc[3];
  if (threadIdx.x < TE_MMAX) {
    int j = threadIdx.x;
    S->dd[j] = j < m ? 2.0 * (S->d[j] - C.c) / C.rho : 0.0;
    S->ee[j] = j + 1 < m ? 2.0 * S->e[j] / C.rho : 0.0;
  }
  __syncthreads();
  C.cheb_n = -1;
  C.eig_ok = false;
}

// Persist Chebyshev / eigen data for the later batch launches.
__device__ void save_krylov_data(KCtx& C, bool pending) {
  TeDevState* ds = C.ds;
  KSmem* S = C.sm;
  if (pending)  // only a further batch of samples reads them
    for (int i = threadIdx.x; i < (C.cheb_n + 1) * TE_MMAX; i += blockDim.x) ds->cheb_t[i] = S->tc[i];
  if (C.eig_ok) {
    for (int i = threadIdx.x; i < TE_MMAX * TE_MMAX; i += blockDim.x) ds->eig_Q[i] = S->Q[i];
    if (threadIdx.x < TE_MMAX) ds->eig_lam[threadIdx.x] = S->lam[threadIdx.x];
  }
  if (threadIdx.x == 0) {
    ds->cheb_c = C.c;
    ds->cheb_rho = C.rho;
    ds->cheb_n = C.cheb_n;
    ds->eig_valid = C.eig_ok ? 1 : 0;
  }
  __syncthreads();
}

__device__ void load_krylov_data(KCtx& C) {
  TeDevState* ds = C.ds;
  KSmem* S = C.sm;
  C.c = ds->cheb_c;
  C.rho = ds->cheb_rho;
  C.cheb_n = ds->cheb_n;
  C.eig_ok = ds->eig_valid != 0;
  if (threadIdx.x < TE_MMAX) {
    S->d[threadIdx.x] = ds->d[threadIdx.x];
    S->e[threadIdx.x] = ds->e[threadIdx.x];
    S->dd[threadIdx.x] = threadIdx.x < C.m ? 2.0 * (S->d[threadIdx.x] - C.c) / C.rho : 0.0;
    S->ee[threadIdx.x] = threadIdx.x + 1 < C.m ? 2.0 * S->e[threadIdx.x] / C.rho : 0.0;
    if (C.eig_ok) S->lam[threadIdx.x] = ds->eig_lam[threadIdx.x];
  }
  for (int i = threadIdx.x; i < (C.cheb_n + 1) * TE_MMAX; i += blockDim.x) S->tc[i] = ds->cheb_t[i];
  if (C.eig_ok)
    for (int i = threadIdx.x; i < TE_MMAX * TE_MMAX; i += blockDim.x) S->Q[i] = ds->eig_Q[i];
  __syncthreads();
  if (C.cheb_n >= 0) {
    // rebuild the signed last components
    const int K = C.cheb_n;
    for (int n = threadIdx.x; n <= K; n += blockDim.x) {
      const double g = S->tc[n * TE_MMAX + (C.m - 1)];
      const int r = n & 3;
      S->gs[n] = (n == 0) ? g : ((r == 0 || r == 3) ? 2.0 * g : -2.0 * g);
    }
  }
  __syncthreads();
}

// One Krylov-space step of one evolution, by the blocks of a cluster (rank,
// size; size 1: one block of any size).
// mode 0: full step (matrix setup, step search, w, first sample batch);
// mode 1: next sample batch of the same Krylov space.
__device__ void krylov_step_body(TeDevState* ds, int mode, KSmem* S, int rank, int size) {
  if (ds->fatal != 0) return;
  if ((mode == 0 && ds->done != 0) || (mode == 1 && ds->samples_pending == 0)) {
    // nothing to do for this evolution: make the combine/observable passes skip it
    if (size > 1) cluster_barrier();  // all blocks have read the state
    if (threadIdx.x == 0 && rank == 0) {
      ds->samples_in_batch = 0;
      ds->want_w = 0;
    }
    return;
  }
  KCtx C;
  C.ds = ds;
  C.sm = S;
  C.rank = rank;
  C.size = size;
  C.round = 0;
  C.n_integrals = 0;
  if ((int)threadIdx.x < TE_KCLUSTER) {
    S->spec[threadIdx.x].method = -1;
    S->found[0][threadIdx.x].state = S->found[1][threadIdx.x].state = 0;
  }
  // what the step reads of the state, all loads in flight at once
  const double t_end = ds->t, t_now = ds->t_now, t_last = ds->t_step, tol_rate = ds->tol_rate, est = ds->num_err_est;
  const int m_eff = ds->m_eff, bd = ds->breakdown, kmax = ds->ts_kmax;
  const double h = ds->h;
  if ((int)threadIdx.x < TE_MMAX) S->s[threadIdx.x] = ds->s[threadIdx.x];
  // every block runs, and has read the state, before any stores into the
  // others' shared memory or writes the state
  if (size > 1)
    cluster_barrier();
  else
    __syncthreads();
  C.m = m_eff;
  C.h = h;
  C.ts_kmax = kmax >= TE_TS_KMIN && kmax < TE_TS_KMAX ? kmax : TE_TS_KMAX;
  C.fatal = 0;
  const bool writer = rank == 0 && threadIdx.x == 0;
  if (mode == 1) {
    load_krylov_data(C);
    schedule_batch(C, t_last, false);
    if (rank == 0) {
      if (threadIdx.x == 0) ds->want_w = 0;
      __syncthreads();
      save_krylov_data(C, ds->samples_pending != 0);
    }
    if (size > 1) cluster_barrier();
    return;
  }
  const bool hbd = bd != 0;
  double t_step = 0.0;
  int code = 0;
  setup_krylov_matrix(C);
  if (hbd) {
    // lucky breakdown (:342-363): the remaining time in one step, m reduced for good
    t_step = t_end - t_now;
    if (size > 1) cluster_barrier();
    if (writer) {
      ds->t_step = t_step;
      ds->err_step = 0.0;
      ds->m_cur = C.m;
      ds->status = TE_STATUS_LUCKY_BREAKDOWN;
      ds->want_w = 0;
      ds->new_start = 0;
    }
  } else {
    const double s0 = 0.97 * t_last;
    double err_step = 0.0;
    code = find_step(C, tol_rate, s0, t_end - t_now, 50, est, t_now == 0.0, &t_step, &err_step);
    if (size > 1) cluster_barrier();
    if (code < 0) {
      if (writer) ds->fatal = code == -1 ? TE_ERR_NO_STEP : TE_ERR_UNSUPPORTED;
      return;
    }
    if (writer) {
      ds->t_step = t_step;
      ds->err_step = err_step;
      ds->err_code_find = code;
      ds->want_w = 1;
      ds->new_start = 1;
    }
  }
  if (writer) {
    ds->n_integrals = C.n_integrals;
    switch (ds->err_code_find) {  // :386-399 (a breakdown step re-counts the previous code)
      case 1: ds->nb_err_roundoff++; break;
      case 20: ds->nb_err_int++; break;
      case 21:
        ds->nb_err_int++;
        ds->nb_err_roundoff++;
        break;
      default: break;
    }
  }
  __syncthreads();
  schedule_batch(C, t_step, !hbd);
  if (rank == 0) {
    __syncthreads();
    save_krylov_data(C, ds->samples_pending != 0);
  }
  if (size > 1) cluster_barrier();  // no block leaves while others may store into its shared memory
}

// One block (one per SM at most: the shared memory of KSmem), so the whole
// register file is available; at the default budget of 64 registers the
// kernel spilled 260 bytes.
__global__ void __launch_bounds__(TE_KTHREADS, 1) krylov_kernel(TeDevState* ds, int mode) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  krylov_step_body(ds, mode, reinterpret_cast<KSmem*>(smem_raw), blockIdx.x, gridDim.x);
}

// Batched evolutions: cluster b (of `size` blocks) runs the step of instance b.
__global__ void __launch_bounds__(TE_KTHREADS, 1) krylov_batch_kernel(TeDevState* states, int mode, int size) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  krylov_step_body(states + blockIdx.x / size, mode, reinterpret_cast<KSmem*>(smem_raw), blockIdx.x % size, size);
}

// ---------------------------------------------------------------------------
// Batched evolutions in one persistent launch: the whole run of a batch (every
// global step: active list, new start vectors, schedule, the m Lanczos
// iterations, the Krylov-space step of every instance, combine, observables,
// extra sample batches, and the final norms) in one cooperative kernel of one
// 1024-thread block per SM, the passes separated by bounded grid barriers.
// The passes are the device bodies of te_batch.cuh, called with the same
// logical schedule warps as the per-pass kernels (hardware warps loop over
// them) and with 256-thread groups for the per-instance reductions, so the
// results equal the graph path's bit for bit; the host waits once per run
// instead of once per global step.
__device__ __forceinline__ void batch_flags_all(const TeDevState* states, int n_inst, int& pending, int& all_done,
                                                int& fatal) {
  int p = 0, d = 1, f = 0;
  for (int i = threadIdx.x; i < n_inst; i += blockDim.x) {
    const int fl = batch_flag(states[i]);
    p |= (fl & 2) != 0;
    d &= (fl & 1) != 0;
    f |= (fl & 4) != 0;
  }
  pending = __syncthreads_or(p);
  all_done = __syncthreads_and(d);
  fatal = __syncthreads_or(f);
}

template <bool REAL>
__global__ void __launch_bounds__(TE_BATCH_PTHREADS, 1) batch_persistent_kernel(TeBatchPersist a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  KSmem* S = reinterpret_cast<KSmem*>(smem_raw);
  // outside the Krylov phase the shared memory serves the group reductions and
  // the schedule
  static_assert(sizeof(KSmem) >= TE_BATCH_TILE * sizeof(double), "the schedule's tile");
  const int ngrp = blockDim.x / TE_THREADS, grp = threadIdx.x / TE_THREADS, gtid = threadIdx.x % TE_THREADS;
  double* gscratch = reinterpret_cast<double*>(smem_raw) + grp * (TE_BATCH_MAX_OBS * 32);
  auto gsync = [grp]() { asm volatile("bar.sync %0, %1;" ::"r"(grp + 1), "r"(TE_THREADS) : "memory"); };
  const int G = gridDim.x;
  auto bar = [&]() { return te_grid_barrier(a.bar_count, a.bar_gen, a.err, a.spin_limit, a.arrivals); };
  const int64_t wpb = blockDim.x >> 5;
  const int64_t pw = (int64_t)blockIdx.x * wpb + (threadIdx.x >> 5), PW = (int64_t)G * wpb;
  const int64_t tg = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, TG = (int64_t)G * blockDim.x;
  const int n_inst = a.n_inst;
  for (int64_t step = 0; step < a.max_global_steps; ++step) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *a.active_count = 0;
    if (!bar()) return;
    batch_active_body(a.g.n_chunks, a.g.chunk_inst, a.states, a.active, a.active_count, tg, TG);
    if (!bar()) return;
    batch_new_start_body<true>(a.g, a.V, a.spare, a.states, pw, PW);
    if (!bar()) return;
    for (int64_t i = tg; i < n_inst; i += TG) a.states[i].new_start = 0;
    if (blockIdx.x == 0)
      batch_cost_body(a.g, a.states, n_inst, a.w_slot, a.inst_cost, reinterpret_cast<double*>(smem_raw));
    if (!bar()) return;
    batch_boundaries_body(a.g, n_inst, a.n_warps, a.w_slot, a.inst_cost, a.warp_begin, tg, TG);
    if (!bar()) return;
    if (blockIdx.x == 0)
      batch_segments_body(a.g, a.states, n_inst, a.n_warps, a.warp_begin, a.inst_w0, a.inst_nseg, a.seg_base,
                          a.next_run, a.inst_nwrite,
                          (a.n_warps + 1) * sizeof(int32_t) <= sizeof(KSmem) ? reinterpret_cast<int32_t*>(smem_raw)
                                                                             : nullptr);
    if (!bar()) return;
    for (int j = 0; j < a.m_max; ++j) {
      for (int64_t vw = pw; vw < a.n_warps; vw += PW) {
        if (j > 0)
          batch_apply_warp<REAL, true, true>(a.g, a.sc, a.V, a.w, a.states, a.seg_partials, j, (int)vw);
        else
          batch_apply_warp<REAL, false, true>(a.g, a.sc, a.V, a.w, a.states, a.seg_partials, j, (int)vw);
      }
      if (!bar()) return;
      for (int64_t vw = pw; vw < a.n_warps; vw += PW)
        batch_update_warp<true>(a.g, a.sc, a.V, a.w, a.states, a.seg_partials, j, (int)vw);
      if (!bar()) return;
    }
    int pending, all_done, fatal;
    for (int mode = 0;; mode = 1) {
      for (int i = blockIdx.x; i < n_inst; i += G) krylov_step_body(a.states + i, mode, S, 0, 1);
      if (!bar()) return;
      batch_combine_body<true>(a.g, a.V, a.spare, a.sampled, a.states, 0, pw, PW);
      if (!bar()) return;
      for (int i = blockIdx.x * ngrp + grp; i < n_inst; i += G * ngrp)
        batch_obs_inst<true>(a.g, a.sampled, a.diag, a.n_obs, a.result_off, a.results, a.states, i, gtid,
                             TE_THREADS, gscratch, gsync);
      if (!bar()) return;
      batch_flags_all(a.states, n_inst, pending, all_done, fatal);
      if (!pending || fatal) break;
    }
    if (threadIdx.x == 0 && blockIdx.x == 0) *a.steps_done = step + 1;
    if (fatal || all_done) break;
  }
  for (int i = blockIdx.x * ngrp + grp; i < n_inst; i += G * ngrp)
    batch_norm_inst<true>(a.g, a.sampled, a.states, i, gtid, TE_THREADS, gscratch, gsync);
}

// ---------------------------------------------------------------- host side

static bool g_tables_uploaded = false;
static int g_cluster = 1;  // blocks per cluster of the Krylov kernels (te_upload_quad_tables)

int te_upload_quad_tables() {
  if (g_tables_uploaded) return TE_OK;
  TeQuadTables T;
  const double half_pi = 1.5707963267948966;
  int idx = 0;
  for (int k = 0; k <= TE_TS_KMAX; ++k) {
    T.ts_level_begin[k] = idx;
    auto add = [&](double tt) {
      double s = half_pi * std::sinh(tt);
      double cs = std::cosh(s);
      T.ts_t[idx] = tt;
      T.ts_u[idx] = std::tanh(s);
      T.ts_w[idx] = half_pi * std::cosh(tt) / (cs * cs);
      ++idx;
    };
    if (k == 0) {
      for (int i = 0; i <= 3; ++i) add((double)i);
    } else {
      double h = std::ldexp(1.0, -k);
      for (int i = 0;; ++i) {
        double tt = (2 * i + 1) * h;
        if (tt > 3.0) break;
        add(tt);
      }
    }
  }
  T.ts_level_begin[TE_TS_KMAX + 1] = idx;
  if (idx != TE_TS_NODES) {
    te_set_error("tanh-sinh table size mismatch (%d)", idx);
    return TE_ERR_UNSUPPORTED;
  }
  auto gauss = [](int n, double* x, double* w) {
    for (int i = 0; i < n; ++i) {
      double z = std::cos(M_PI * (i + 0.75) / (n + 0.5));
      for (int it = 0; it < 100; ++it) {
        double p0 = 1.0, p1 = z;
        for (int k = 2; k <= n; ++k) {
          double p2 = ((2.0 * k - 1.0) * z * p1 - (k - 1.0) * p0) / k;
          p0 = p1;
          p1 = p2;
        }
        double pp = n * (z * p1 - p0) / (z * z - 1.0);
        double dz = p1 / pp;
        z -= dz;
        if (std::fabs(dz) < 1e-17) break;
      }
      double p0 = 1.0, p1 = z;
      for (int k = 2; k <= n; ++k) {
        double p2 = ((2.0 * k - 1.0) * z * p1 - (k - 1.0) * p0) / k;
        p0 = p1;
        p1 = p2;
      }
      double pp = n * (z * p1 - p0) / (z * z - 1.0);
      x[i] = z;
      w[i] = 2.0 / ((1.0 - z * z) * pp * pp);
    }
  };
  gauss(15, T.g15_x, T.g15_w);
  gauss(7, T.g7_x, T.g7_w);
  if (T.ts_level_begin[kTsFirst + 1] != kTsFirstNodes) {
    te_set_error("tanh-sinh table: unexpected first levels");
    return TE_ERR_UNSUPPORTED;
  }
  TE_CUDA(cudaMemcpyToSymbol(c_quad, &T, sizeof(T)));
  TE_CUDA(cudaMemcpyToSymbol(g_quad, &T, sizeof(T)));
  TE_CUDA(cudaFuncSetAttribute(krylov_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(KSmem)));
  TE_CUDA(cudaFuncSetAttribute(krylov_batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(KSmem)));
  // the largest cluster whose blocks (one per SM: their shared memory) can run together
  for (int size = TE_KCLUSTER; size > 1; size /= 2) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(size);
    cfg.blockDim = dim3(TE_KTHREADS);
    cfg.dynamicSmemBytes = sizeof(KSmem);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = size;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, krylov_kernel, &cfg) != cudaSuccess) cudaGetLastError();
    if (clusters >= 1) {
      g_cluster = size;
      break;
    }
  }
  g_tables_uploaded = true;
  return TE_OK;
}

template <typename... KArgs, typename... Args>
static void launch_clusters(void (*kernel)(KArgs...), int clusters, int size, cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(clusters * size);
  cfg.blockDim = dim3(TE_KTHREADS);
  cfg.dynamicSmemBytes = sizeof(KSmem);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = size;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

void te_launch_krylov_step(TeDevState* ds, cudaStream_t st) { launch_clusters(krylov_kernel, 1, g_cluster, st, ds, 0); }

void te_launch_schedule_samples(TeDevState* ds, cudaStream_t st) {
  launch_clusters(krylov_kernel, 1, g_cluster, st, ds, 1);
}

// Blocks per instance: as many as leave all clusters resident at once (a
// block takes a whole SM's shared memory); finished instances leave at once.
void te_launch_krylov_batch(TeDevState* states, int n_instances, int mode, cudaStream_t st) {
  int size = g_cluster;
  while (size > 1 && n_instances * size > te_num_sms()) size /= 2;
  launch_clusters(krylov_batch_kernel, n_instances, size, st, states, mode, size);
}

int te_batch_persistent_grid(bool is_real) {
  const void* k = is_real ? (const void*)batch_persistent_kernel<true> : (const void*)batch_persistent_kernel<false>;
  int dev = 0, coop = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop) return 0;
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(KSmem)) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, TE_BATCH_PTHREADS, sizeof(KSmem)) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return per_sm >= 1 ? te_num_sms() : 0;  // one block per SM
}

int te_launch_batch_persistent(const TeBatchPersist& a, int grid, cudaStream_t st) {
  void* k = a.is_real ? (void*)batch_persistent_kernel<true> : (void*)batch_persistent_kernel<false>;
  TeBatchPersist arg = a;
  void* params[] = {&arg};
  return te_cuda_check(cudaLaunchCooperativeKernel(k, dim3(grid), dim3(TE_BATCH_PTHREADS), params, sizeof(KSmem), st),
                       "persistent batch launch");
}
