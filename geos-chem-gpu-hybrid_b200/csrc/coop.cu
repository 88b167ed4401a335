/*
 * coop.cu -- the cooperative Rodas3 kernel: one thread block per cell, the
 * whole cell state in shared memory.
 *
 * The one-thread-per-cell kernels stream every cell's workspace (the LU
 * factors, the Jacobian, the stage vectors) through HBM, because 256 cells
 * per SM cannot keep 50-125 KB each on chip.  Here a block of 128 or 256
 * threads owns one cell at a time and keeps its factors G (NNZ doubles), the
 * state and stage vectors, the rate constants and a scratch array in shared
 * memory (69 KB for the 120-species synthetic mechanism, 94 KB for
 * fullchem), so the solve reads HBM only to load a cell and store its
 * result.  The block drains the same cost-ordered work queue as the
 * persistent kernel: thread 0 takes the next queue position, and the block
 * solves that cell to the end (with the in-place retry), then takes the next.
 *
 * Parallelism inside a cell comes from tables generated from the mechanism
 * (coop.inc, mechanism/coop.py):
 *   Fun      rates A(j) one per thread, then P_VAR/D_VAR/Vdot one species per
 *            thread (gckpp_Function.F90:2170-5060 expressions, same rounding);
 *   Jac      partials B(m), then entries JVS(k), written straight into the
 *            factor array as -JVS (+ 1/(H*gamma) on the diagonal); the
 *            Jacobian is recomputed at every attempt instead of being stored
 *            (Y is unchanged after a rejection, so it is the same Jacobian);
 *   KppDecomp right-looking: step j forms column j's multipliers, then
 *            applies pivot row j to every row below it at once; each entry
 *            gets its updates in the reference's order
 *            (gckpp_LinearAlgebra.F90:46-84), so the factors are identical;
 *   KppSolve forward sweep by columns, each row's terms in the reference's
 *            order (:645-2311); backward sweep by levels of rows in the
 *            reference's order (--fmad=false build), or by columns (FMA
 *            build: 120 parallel steps instead of a chain of every row's
 *            terms, the per-row order reversed).
 * Step-size control, counters, options and the retry protocol are the
 * arithmetic of Integrate_Cell_S (gckpp_BatchIntegrator.F90:408-707) and of
 * the model's retry (fullchem_mod.F90:2436-2520), computed redundantly by
 * every thread of the block so that every branch is block-uniform; the one
 * sequential sum (the error norm, in species order) is taken by thread 0.
 *
 * Built with --fmad=false this kernel reproduces the CPU oracle bit for bit,
 * as the one-thread-per-cell kernels do; the FMA build contracts into FMA
 * and forms the multipliers and the backward quotients from one reciprocal
 * per pivot (GC_IRECIP).
 *
 * Every __syncthreads() is reached by all threads of the block: loop bounds
 * come from the tables, and every branch around a barrier depends only on
 * values all threads hold identically (shared-memory words read after a
 * barrier, or scalars computed redundantly from them).  Nothing waits on
 * another block.
 */
#include <cuda_runtime.h>
#include <float.h>
#include <limits.h>
#include "rodas3_device.cuh"
#include "gc_pow.h"
#include "rodas3_kernels.h"
/* sums may be split over lanes where the build need not round like the
   reference */
#define COOP_SPLIT GC_IRECIP
#include "coop.inc"

#if MECH_COOP

#if !COOP_SPLIT
static __constant__ int coop_diag_c[NVAR] = MECH_LU_DIAG_INIT;
#endif

/* shared-memory layout of one cell (in doubles).  Y0 and Y1 carry the fixed
   species and the constants of the rate tables behind the NVAR species.
   The rates A and partials B live in areas that are dead at that time:
   A of the step's first Fun and B in K1..K3 and S (the stages start later),
   A of the stages' Fun in S and FCN0 (Fcn0 is read by stages 1 and 2 only;
   it is formed again at every attempt). */
#define COOP_MAX2(a, b) ((a) > (b) ? (a) : (b))
#define COOP_NS COOP_MAX2(COOP_MAX2(NREACT - NVAR, COOP_NBP - 3 * NVAR), 1)
#define SO_G     0
#define SO_Y0    (SO_G + NNZ)
#define SO_Y1    (SO_Y0 + COOP_NX)
#define SO_K     (SO_Y1 + COOP_NX)
#define SO_S     (SO_K + 3 * NVAR)
#define SO_FCN0  (SO_S + COOP_NS)
#define SO_K4    (SO_FCN0 + NVAR)
#define SO_DFDT  SO_K4              /* read by stages 1 and 2, K4 is written by stage 4 */
#define SO_R     (SO_K4 + NVAR)
#define SO_EXTRA (SO_R + NVAR)
#define SO_END   (SO_EXTRA + COOP_NEXTRA + 1)
#define COOP_NO  0xFFFFFFFFu
#define COOP_BARRIER 1
#define COOP_CHAIN 2
#define COOP_PW  8                  /* product words of a lane fetched one round ahead */

extern __shared__ double sm[];

struct CoopArgs {
  int ncell;
  double tstart, tend;
  double* C;
  const double* RCONST;
  const double* ATOL;
  const double* RTOL;
  const int* ICNTRL;
  const double* RCNTRL;
  const int* order;
  int* ISTAT;
  double* RSTAT;
  int* IERR;
  unsigned int* qhead;
  int* nfail;
  const double* ATOLr;
  const double* RTOLr;
  double* ckpt;            /* adjoint checkpoints (y_n, h_n) per accepted step, or NULL */
  int ckpt_max;
};

/* the cell's integrator state; every thread of the block holds the same */
struct CoopCell {
  long col;
  CellOpts o;
  CellStat st;
  double T, H;
  int nsteps, ncons, rej_last, rej_more, newstep, ierr, ysel, attempt;
};

/* ---- rounds --------------------------------------------------------------
   A program (dest, prod, jvs, lu, fwd, bwd; see mechanism/coop.py) is a list
   of rounds of at most 256 lanes.  What bounds a round is latency: table
   words from L2, shared-memory operands, the sum's dependent FMAs, the
   exchanges and the barrier.  The words of the next round are therefore
   fetched into registers before the current one runs, and all operands of a
   lane are loaded before its first FMA. */
enum { P_DEST, P_PROD, P_JVS, P_LU, P_FWD, P_BWD };

template <int NT>
struct CoopWords {
  unsigned int h[256 / NT];
  unsigned int w[256 / NT][COOP_PW];
};

template <int NT>
__device__ __forceinline__ void coop_fetch(CoopWords<NT>& q, int2 r,
                                           const unsigned int* __restrict__ tab) {
  const int nl = r.y & 0x3FF, k = (r.y >> 10) & 0x3FF;
#pragma unroll
  for (int f = 0; f < 256 / NT; ++f) {
    const int v = threadIdx.x + f * NT;
    const bool in = v < nl;
    q.h[f] = in ? __ldg(tab + r.x + v) : COOP_NO;
#pragma unroll
    for (int t = 0; t < COOP_PW; ++t)
      q.w[f][t] = (in && t < k) ? __ldg(tab + r.x + nl * (1 + t) + v) : COOP_NO;
  }
}

/* KK products of a lane: operands first, then the sum in order.  off: the
   vector operand's place (V for dest, rates or partials for prod and jvs, the
   solution for the sweeps); rc: the cell's rate constants */
template <int PROG, int KK>
__device__ __forceinline__ double coop_products(double acc, const unsigned int* w, int off,
                                                const double* __restrict__ rc) {
  double a[KK], b[KK];
#pragma unroll
  for (int t = 0; t < KK; ++t) {
    const unsigned int x = w[t] == COOP_NO ? 0u : w[t];
    if (PROG == P_DEST) {
      const int f0 = x & 0x7FF, f2 = x >> 21;
      a[t] = f0 < NREACT ? __ldg(rc + f0) : sm[SO_EXTRA + f0 - NREACT];
      b[t] = sm[off + ((x >> 11) & 0x3FF)];
      if (f2 != NVAR + NFIX) { a[t] = a[t] * b[t]; b[t] = sm[off + f2]; }
    } else if (PROG == P_PROD || PROG == P_JVS) {
      a[t] = __ldg(coop_coef + (x & 0xFFFF));
      b[t] = sm[off + (x >> 16)];
    } else {
      a[t] = sm[SO_G + (x & 0xFFFF)];
      b[t] = sm[(PROG == P_LU ? SO_G : off) + (x >> 16)];
    }
  }
#pragma unroll
  for (int t = 0; t < KK; ++t) {
    if (w[t] != COOP_NO) {
      if (PROG == P_DEST || PROG == P_PROD || PROG == P_JVS) acc = acc + a[t] * b[t];
      else acc = acc - a[t] * b[t];
    }
  }
  return acc;
}

/* what a program leaves behind: out is the result vector of dest and prod
   and the place of the solution in the sweeps, v the state of Fun */
struct CoopOut {
  int out, v;
  double ghinv;
  int* ising;
};

template <int PROG>
__device__ __forceinline__ void coop_finish(unsigned int h, double acc, const CoopOut& o) {
  const int d = h & 0x1FFF;
  if (PROG == P_DEST) {
    sm[o.out + d] = acc;
  } else if (PROG == P_PROD) {
    sm[o.out + d] = acc - sm[o.out + d] * sm[o.v + d];
  } else if (PROG == P_JVS) {
    const int row = (int)((h >> 16) & 0xFFF) - 1;
    if (row >= 0) {
      acc = acc + o.ghinv;
      if (fabs(acc) < DBL_MIN) atomicMin(o.ising, row + 1);
#if COOP_SPLIT
      if (h >> 28) sm[SO_R + row] = 1.0 / acc;
#endif
    }
    sm[SO_G + d] = acc;
  } else if (PROG == P_LU) {
    const int c = (h >> 16) & 0xFFF;
#if COOP_SPLIT
    if (h & (1u << 28)) acc = acc * sm[SO_R + c];
    if (h & (1u << 29)) sm[SO_R + c] = 1.0 / acc;
#else
    if (h & (1u << 28)) acc = acc / sm[SO_G + coop_diag_c[c]];
#endif
    sm[SO_G + d] = acc;
  } else if (PROG == P_FWD) {
    sm[o.out + d] = acc;
  } else {
#if COOP_SPLIT
    if (!(h >> 28)) acc = acc * sm[SO_R + d];
#else
    acc = acc / sm[SO_G + coop_diag_c[d]];
#endif
    sm[o.out + d] = acc;
  }
}

#if COOP_SPLIT
/* A warp chain: up to 32 rows that depend on one another in turn, one per
   lane.  The factors are loaded ahead; a step is one exchange and one FMA. */
template <int PROG>
__device__ __forceinline__ void coop_chain(int m, const unsigned int* __restrict__ tab, int x) {
  const int lane = threadIdx.x & 31;
  const int row = (int)__ldg(tab + lane);
  const unsigned int mask = __ldg(tab + 32 + lane);
  unsigned int pos[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) pos[j] = (2 * j < m) ? __ldg(tab + 64 + 32 * j + lane) : 0u;
  double acc = (lane < m) ? sm[x + row] : 0.0;
  const double rr = (PROG == P_BWD && lane < m) ? sm[SO_R + row] : 1.0;
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    if (16 * c < m) {
      double l[16];
#pragma unroll
      for (int j = 0; j < 16; ++j)
        l[j] = sm[SO_G + ((pos[8 * c + j / 2] >> (16 * (j & 1))) & 0xFFFF)];
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        if (16 * c + j < m) {
          const double xj = __shfl_sync(0xFFFFFFFFu, PROG == P_BWD ? acc * rr : acc, 16 * c + j);
          if (mask >> (16 * c + j) & 1u) acc = acc - l[j] * xj;
        }
      }
    }
  }
  if (lane < m) sm[x + row] = PROG == P_BWD ? acc * rr : acc;
}
#endif

template <int PROG, int NT>
__device__ __forceinline__ void coop_rounds(int r0, int r1, const unsigned int* __restrict__ tab,
                                            int off, const double* __restrict__ rc,
                                            const CoopOut& o) {
  CoopWords<NT> nxt;
  int2 rn = coop_round[r0];
  coop_fetch<NT>(nxt, rn, tab);
  for (int r = r0; r < r1; ++r) {
    const CoopWords<NT> cur = nxt;
    const int2 rd = rn;
    if (r + 1 < r1) {
      rn = coop_round[r + 1];
      coop_fetch<NT>(nxt, rn, tab);
    }
    const int nl = rd.y & 0x3FF, k = (rd.y >> 10) & 0x3FF, s = (rd.y >> 20) & 0xF,
              flags = rd.y >> 24;
#if COOP_SPLIT
    if ((PROG == P_FWD || PROG == P_BWD) && (flags & COOP_CHAIN)) {
      if (threadIdx.x < 32) coop_chain<PROG>(k, tab + rd.x, o.out);
    } else
#endif
    {
#pragma unroll
      for (int f = 0; f < 256 / NT; ++f) {
        const int v = threadIdx.x + f * NT;
        if (v < nl) {                       /* whole warps: nl is a multiple of 32 */
          const unsigned int h = cur.h[f];
          const int lg = (h >> 13) & 7;
          const bool lead = h != COOP_NO && (v & ((1 << lg) - 1)) == 0;
          double acc = 0.0;
          if (PROG == P_LU && lead) acc = sm[SO_G + (h & 0x1FFF)];
          if ((PROG == P_FWD || PROG == P_BWD) && lead) acc = sm[o.out + (h & 0x1FFF)];
          if (k > 4) acc = coop_products<PROG, 8>(acc, cur.w[f], off, rc);
          else if (k > 2) acc = coop_products<PROG, 4>(acc, cur.w[f], off, rc);
          else if (k > 0) acc = coop_products<PROG, 2>(acc, cur.w[f], off, rc);
          for (int t0 = COOP_PW; t0 < k; t0 += 4) {
            unsigned int w[4];
#pragma unroll
            for (int t = 0; t < 4; ++t)
              w[t] = t0 + t < k ? __ldg(tab + rd.x + nl * (1 + t0 + t) + v) : COOP_NO;
            acc = coop_products<PROG, 4>(acc, w, off, rc);
          }
          for (int e = 0; e < s; ++e) {
            const double y = __shfl_xor_sync(0xFFFFFFFFu, acc, 1 << e);
            if (e < lg) acc = acc + y;
          }
          if (lead) coop_finish<PROG>(h, acc, o);
        }
      }
    }
    if (flags & COOP_BARRIER) __syncthreads();
  }
}

/* products of four factors (rates A, partials B), one per thread and pass:
   ((f0*f1)*f2)*f3, absent factors being the constant 1 */
template <int NT, int N>
__device__ __forceinline__ void coop_rates(const unsigned short* __restrict__ rec, int v, int out,
                                           const double* __restrict__ rc) {
  const ushort4* r4 = reinterpret_cast<const ushort4*>(rec);
#pragma unroll 4
  for (int j = threadIdx.x; j < N; j += NT) {
    const ushort4 f = __ldg(r4 + j);
    double x = f.x < NREACT ? __ldg(rc + f.x) : sm[SO_EXTRA + f.x - NREACT];
    x = (x * sm[v + f.y]) * sm[v + f.z];
    if (f.w != NVAR + NFIX) x = x * sm[v + f.w];
    sm[out + j] = x;
  }
}

/* Fun_SPLIT: out = P_VAR - D_VAR*V, rates A at `area`.  The destruction
   sums need no rates, so they run before the barrier that publishes A. */
template <int NT>
__device__ __noinline__ void coop_fun(int v, int out, int area, const double* __restrict__ rc) {
  CoopOut o;
  o.out = out; o.v = v; o.ghinv = 0.0; o.ising = nullptr;
  coop_rates<NT, NREACT>(coop_rate, v, area, rc);
  coop_rounds<P_DEST, NT>(COOP_R0_DEST, COOP_R1_DEST, coop_w_dest, v, rc, o);
  __syncthreads();
  coop_rounds<P_PROD, NT>(COOP_R0_PROD, COOP_R1_PROD, coop_w_prod, area, rc, o);
}

/* Jac_SP straight into ros_PrepareMatrix's form: G = -JVS, plus ghinv on
   the diagonal.  KppDecomp's singularity test reads each prepared diagonal
   before its row is eliminated, so it is taken here: *ising becomes the
   lowest failing row + 1 (it holds INT_MAX on entry). */
template <int NT>
__device__ __forceinline__ void coop_jac_prep(int v, const double* __restrict__ rc, double ghinv,
                                              int* ising) {
  CoopOut o;
  o.out = 0; o.v = v; o.ghinv = ghinv; o.ising = ising;
  coop_rates<NT, COOP_NBP>(coop_bpart, v, SO_K, rc);
  __syncthreads();
  coop_rounds<P_JVS, NT>(COOP_R0_JVS, COOP_R1_JVS, coop_w_jvs, SO_K, rc, o);
}

/* KppDecomp entry by entry, in levels: G(i,c) - sum L(i,j) U(j,c), times
   1/U(c,c) (R, FMA build) or over U(c,c) left of the diagonal */
template <int NT>
__device__ __forceinline__ void coop_decomp() {
  CoopOut o;
  o.out = 0; o.v = 0; o.ghinv = 0.0; o.ising = nullptr;
  coop_rounds<P_LU, NT>(COOP_R0_LU, COOP_R1_LU, coop_w_lu, SO_G, nullptr, o);
}

/* KppSolve in place on the vector at x (the caller has synchronised after
   writing it) */
template <int NT>
__device__ __forceinline__ void coop_solve(int x) {
  CoopOut o;
  o.out = x; o.v = 0; o.ghinv = 0.0; o.ising = nullptr;
  coop_rounds<P_FWD, NT>(COOP_R0_FWD, COOP_R1_FWD, coop_w_fwd, x, nullptr, o);
  coop_rounds<P_BWD, NT>(COOP_R0_BWD, COOP_R1_BWD, coop_w_bwd, x, nullptr, o);
}

/* load the cell's column and set the integrator state (lane_start of the
   one-thread-per-cell kernels); attempt 1 is the retry: Hstart taken as 0
   and the retry tolerances */
__device__ __forceinline__ void coop_start(CoopCell& c, const CoopArgs& a, long col,
                                           int attempt) {
  c.col = col;
  c.attempt = attempt;
  const double* cc = a.C + col * NSPEC;
  const double* rr = a.RCONST + col * NREACT;
  for (int i = threadIdx.x; i < COOP_NX; i += blockDim.x) {
    const double y = i < NSPEC ? cc[i] : coop_ext[i - NSPEC];
    sm[SO_Y0 + i] = y;
    if (i >= NVAR) sm[SO_Y1 + i] = y;
  }
  for (int i = threadIdx.x; i < COOP_NEXTRA; i += blockDim.x) {
    const int j = coop_extra_src[i];
    sm[SO_EXTRA + i] = j >= 0 ? rr[j] * coop_extra_val[i] : coop_extra_val[i];
  }
  c.o = decode_options(a.ICNTRL + col * 20, a.RCNTRL + col * 20, a.tstart, a.tend, attempt);
  c.st.nfun = c.st.njac = c.st.nstp = c.st.nacc = 0;
  c.st.nrej = c.st.ndec = c.st.nsol = c.st.nsng = 0;
  c.st.texit = c.st.hexit = c.st.hnew = 0.0;
  c.ierr = c.o.ierr_early;
  c.T = a.tstart;
  double H = fminF(fmaxF(fabs(c.o.hmin), fabs(c.o.hstart)), fabs(c.o.hmax));
  if (fabs(H) <= 10.0 * ROUNDOFF) H = DELTAMIN;
  const double dir = (a.tend >= a.tstart) ? 1.0 : -1.0;
  c.H = dir * H;
  c.nsteps = 0;
  c.ncons = 0;
  c.rej_last = c.rej_more = 0;
  c.newstep = 1;
  c.ysel = 0;
  __syncthreads();
}

__device__ __forceinline__ void coop_store_istat(const CoopCell& c, const CoopArgs& a, int add) {
  int* is = a.ISTAT + c.col * 8;
  const int v[8] = {c.st.nfun, c.st.njac, c.st.nstp, c.st.nacc,
                    c.st.nrej, c.st.ndec, c.st.nsol, c.st.nsng};
#pragma unroll
  for (int k = 0; k < 8; ++k) is[k] = add ? is[k] + v[k] : v[k];
}

/* the end of a solve (lane_end / lane_finish of the other kernels): with the
   retry protocol on, a failed first solve stores its counters and restarts
   from the untouched input column; returns 1 when the cell is finished */
__device__ __forceinline__ int coop_end(CoopCell& c, const CoopArgs& a) {
  if (a.nfail && c.attempt == 0 && c.ierr < 0) {
    if (threadIdx.x == 0) {
      coop_store_istat(c, a, 0);
      atomicAdd(&a.nfail[0], 1);
    }
    __syncthreads();
    coop_start(c, a, c.col, 1);
    if (c.ierr == 0) return 0;
  }
  if (c.o.ierr_early == 0) {
    const double* Y = sm + (c.ysel ? SO_Y1 : SO_Y0);
    double* cc = a.C + c.col * NSPEC;
    for (int i = threadIdx.x; i < NVAR; i += blockDim.x) cc[i] = Y[i];
  }
  if (threadIdx.x == 0) {
    coop_store_istat(c, a, c.attempt);
    if (c.attempt && c.ierr < 0) atomicAdd(&a.nfail[1], 1);
    double* rs = a.RSTAT + c.col * 3;
    rs[0] = c.st.texit; rs[1] = c.st.hexit; rs[2] = c.st.hnew;
    a.IERR[c.col] = c.ierr;
  }
  return 1;
}

/* err**(1/3) of the step-size factor.  gc_pow's double-double series is a
   chain of ~1,000 dependent operations, a fifth of an attempt here.  The
   production build starts from cbrt and adds the residual of one
   double-double cube and the difference between the double 1/3 and 1/3
   (x**(1/3 - d) = x**(1/3) (1 - d ln x), d = 1.850371707708594e-17); the one
   rounding left is the last addition, as in gc_pow. */
__device__ __forceinline__ double coop_root(double x) {
#if COOP_SPLIT
  if (x < 1.0e300) {
    const double c = cbrt(x);
    const double p = c * c, pl = __fma_rn(c, c, -p);
    const double q = p * c, ql = __fma_rn(p, c, -q) + pl * c;
    const double r = (x - q) - ql;
    return c + (r / (3.0 * p) - c * (1.850371707708594e-17 * log(x)));
  }
#endif
  return gc_pow(x, 1.0 / ROS_ELO);
}

/* One pass of TimeLoop/UntilAccepted (gckpp_BatchIntegrator.F90:535-704)
   for the block's cell; returns 1 when the cell is finished (c.ierr holds
   IERR).  The statement-level arithmetic is that of step_begin,
   step_prologue, step_factor and step_stages in rodas3_kernels.cu. */
template <int NT>
__device__ __forceinline__ int coop_attempt(CoopCell& c, const CoopArgs& a, int* s_ising,
                                            double* s_err) {
  const int tid = threadIdx.x;
  const double Tend = a.tend;
  const double dir = (Tend >= a.tstart) ? 1.0 : -1.0;
  const int y = c.ysel ? SO_Y1 : SO_Y0, ynew = c.ysel ? SO_Y0 : SO_Y1;
  const double* __restrict__ rc = a.RCONST + c.col * NREACT;

  if (c.newstep) {
    /* TimeLoop exit tests and the H clamp */
    const int direction = (Tend >= a.tstart) ? 1 : -1;
    const bool running = (direction > 0 && ((c.T - Tend) + ROUNDOFF <= 0.0)) ||
                         (direction < 0 && ((Tend - c.T) + ROUNDOFF <= 0.0));
    if (!running) { c.ierr = 1; return 1; }
    if (c.nsteps > c.o.max_steps) { c.ierr = -6; return 1; }
    if (((c.T + 0.1 * c.H) == c.T) || (c.H <= ROUNDOFF)) { c.ierr = -7; return 1; }
    c.H = fminF(c.H, fabs(Tend - c.T));
    c.st.nfun += c.o.autonomous ? 1 : 2;
    c.st.njac += 1;
    c.newstep = 0;
    c.ncons = 0;
  }

  /* Fcn0 [, dFdT] and the Jacobian.  A retried attempt forms them again from
     the unchanged state (the same values; the counters move once per step):
     their shared memory holds the stages' rates meanwhile. */
  coop_fun<NT>(y, SO_FCN0, SO_K, rc);
  if (!c.o.autonomous) {
    const double delta = sqrt(ROUNDOFF) * fmaxF(1.0e-6, fabs(c.T));
    coop_fun<NT>(y, SO_DFDT, SO_K, rc);
    for (int k = tid; k < NVAR; k += NT)
      sm[SO_DFDT + k] = (sm[SO_DFDT + k] - sm[SO_FCN0 + k]) / delta;
  }

  /* ros_PrepareMatrix + KppDecomp */
  const double ghinv = 1.0 / ((dir * c.H) * 0.5);
  if (tid == 0) *s_ising = INT_MAX;
  coop_jac_prep<NT>(y, rc, ghinv, s_ising);
  const int ising = (*s_ising == INT_MAX) ? 0 : *s_ising;
  if (ising == 0) coop_decomp<NT>();
  c.st.ndec += 1;
  if (ising != 0) {
    c.st.nsng += 1;
    c.ncons += 1;
    __syncthreads();      /* every thread has read *s_ising */
    if (c.ncons <= 5) { c.H = c.H * 0.5; return 0; }
    c.ierr = -8;
    return 1;
  }

  /* the four stages (per-element operation order of :595-632) */
  const double dH = dir * c.H;
  const double hc1 = 1.0 / dH, hc2 = -1.0 / dH, hc3 = -(8.0 / 3.0) / dH, hc21 = 4.0 / dH;
  for (int s = 0; s < 4; ++s) {
    const int x = s < 3 ? SO_K + s * NVAR : SO_K4;
    if (s >= 2) {
      /* Ynew = (Y + 2 K1) + 0 K2, then + 1 K3 for stage 4 (Ynew still holds
         stage 3's value, rounded as the reference's expression rounds it) */
      for (int k = tid; k < NVAR; k += NT)
        sm[ynew + k] = s == 2 ? (sm[y + k] + 2.0 * sm[SO_K + k]) + 0.0 * sm[SO_K + NVAR + k]
                              : sm[ynew + k] + 1.0 * sm[SO_K + 2 * NVAR + k];
      __syncthreads();
      coop_fun<NT>(ynew, x, SO_S, rc);
      c.st.nfun += 1;
    }
    for (int k = tid; k < NVAR; k += NT) {
      double v;
      if (s == 0) {
        v = sm[SO_FCN0 + k];
        if (!c.o.autonomous) v = v + (dH * 0.5) * sm[SO_DFDT + k];
      } else if (s == 1) {
        v = sm[SO_FCN0 + k] + hc21 * sm[SO_K + k];
        if (!c.o.autonomous) v = v + (dH * 1.5) * sm[SO_DFDT + k];
      } else {
        v = (sm[x + k] + hc1 * sm[SO_K + k]) + hc2 * sm[SO_K + NVAR + k];
        if (s == 3) v = v + hc3 * sm[SO_K + 2 * NVAR + k];
      }
      sm[x + k] = v;
    }
    __syncthreads();
    coop_solve<NT>(x);
    c.st.nsol += 1;
  }

  /* Ynew, Yerr and the scaled error terms in parallel; the WRMS sum over
     warps, or in species order by thread 0 where the build rounds like the
     reference */
  const double* atol = c.attempt ? a.ATOLr : a.ATOL;
  const double* rtol = c.attempt ? a.RTOLr : a.RTOL;
  double err = 0.0;
  for (int i = tid; i < NVAR; i += NT) {
    const double yi = sm[y + i];
    const double k1 = sm[SO_K + i], k2 = sm[SO_K + NVAR + i], k3 = sm[SO_K + 2 * NVAR + i],
                 k4 = sm[SO_K4 + i];
    const double yn = (((yi + 2.0 * k1) + 0.0 * k2) + 1.0 * k3) + 1.0 * k4;
    sm[ynew + i] = yn;
    const double ye = (((0.0 + 0.0 * k1) + 0.0 * k2) + 0.0 * k3) + 1.0 * k4;
    const double ymax = fmaxF(fabs(yi), fabs(yn));
    const double scal = c.o.vectortol ? (__ldg(atol + i) + __ldg(rtol + i) * ymax)
                                      : (__ldg(atol) + __ldg(rtol) * ymax);
    const double q = ye / scal;
#if COOP_SPLIT
    err = err + q * q;
#else
    sm[SO_FCN0 + i] = q;
#endif
  }
#if COOP_SPLIT
#pragma unroll
  for (int e = 16; e > 0; e >>= 1) err = err + __shfl_xor_sync(0xFFFFFFFFu, err, e);
  if ((tid & 31) == 0) s_err[tid >> 5] = err;
  __syncthreads();
  err = 0.0;
#pragma unroll
  for (int w = 0; w < NT / 32; ++w) err = err + s_err[w];
#else
  __syncthreads();
  if (tid == 0) {
    for (int i = 0; i < NVAR; ++i) {
      const double q = sm[SO_FCN0 + i];
      err = err + q * q;
    }
    s_err[0] = err;
  }
  __syncthreads();
  err = s_err[0];
#endif
  err = sqrt(err / (double)NVAR);
  err = fmaxF(err, 1.0e-10);
  const double fac = fminF(c.o.facmax,
                           fmaxF(c.o.facmin, c.o.facsafe / coop_root(err)));
  double hnew = c.H * fac;

  c.nsteps += 1;
  c.st.nstp += 1;
  if ((err <= 1.0) || (c.H <= c.o.hmin)) {
    c.st.nacc += 1;
    if (a.ckpt && c.st.nacc <= a.ckpt_max) {
      /* checkpoint for the adjoint: the step's starting state and its size */
      double* ck = a.ckpt + (c.col * a.ckpt_max + (c.st.nacc - 1)) * (NVAR + 1);
      for (int k = tid; k < NVAR; k += NT) ck[k] = sm[y + k];
      if (tid == 0) ck[NVAR] = c.H;
    }
    if (c.o.clamp) {
      for (int k = tid; k < NVAR; k += NT) sm[ynew + k] = fmaxF(sm[ynew + k], 0.0);
    }
    c.ysel ^= 1;              /* Y = Ynew: the arrays swap roles */
    c.T = c.T + dir * c.H;
    hnew = fmaxF(c.o.hmin, fminF(hnew, c.o.hmax));
    if (c.rej_last) hnew = fminF(hnew, c.H);
    c.st.hexit = c.H;
    c.st.hnew = hnew;
    c.st.texit = c.T;
    c.rej_last = 0;
    c.rej_more = 0;
    c.H = hnew;
    c.newstep = 1;
  } else {
    if (c.rej_more) hnew = c.H * c.o.facrej;
    c.rej_more = c.rej_last;
    c.rej_last = 1;
    c.H = hnew;
    if (c.st.nacc >= 1) c.st.nrej += 1;
    c.ncons = 0;
  }
  __syncthreads();            /* s_err read by all; the clamp is complete */
  return 0;
}
template <int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) rodas3_coop(CoopArgs a) {
  __shared__ unsigned int s_pos;
  __shared__ int s_ising;
  __shared__ double s_err[NT / 32];
  for (;;) {
    if (threadIdx.x == 0) s_pos = atomicAdd(a.qhead, 1u);
    __syncthreads();
    const unsigned int p = s_pos;
    __syncthreads();          /* s_pos read by all before thread 0 rewrites it */
    if (p >= (unsigned int)a.ncell) break;
    CoopCell c;
    coop_start(c, a, (long)a.order[p], 0);
    do {
      if (c.ierr == 0) {
        while (!coop_attempt<NT>(c, a, &s_ising, s_err)) {}
      }
    } while (!coop_end(c, a));
    __syncthreads();          /* the result is stored before the next cell loads */
  }
}

static size_t coop_smem_bytes(void) { return (size_t)SO_END * sizeof(double); }

/* the kernel instance for a block size (128 or 256 threads) */
static const void* coop_kernel(int threads) {
  if (threads == 128) return (const void*)rodas3_coop<128, 3>;
  if (threads == 256) return (const void*)rodas3_coop<256, 2>;
  return nullptr;
}

static cudaError_t coop_attr(int threads) {
  const void* k = coop_kernel(threads);
  if (!k) return cudaErrorInvalidValue;
  return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)coop_smem_bytes());
}

extern "C" int rodas3_coop_ok(void) {
  return coop_smem_bytes() <= 227 * 1024 ? 1 : 0;
}

extern "C" size_t rodas3_coop_smem_bytes(void) { return coop_smem_bytes(); }

extern "C" int rodas3_coop_blocks_per_sm(int threads) {
  if (!rodas3_coop_ok() || coop_attr(threads) != cudaSuccess) return 0;
  int nb = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, coop_kernel(threads), threads,
                                                    coop_smem_bytes()) != cudaSuccess)
    return 0;
  return nb;
}

/* blocks: resident blocks of the launch (the caller's SM count x blocks per
   SM, at most one per cell) */
extern "C" cudaError_t rodas3_coop_launch(const Rodas3Launch* L, int blocks, cudaStream_t s) {
  if (!rodas3_coop_ok()) return cudaErrorInvalidValue;
  const int threads = L->threads;
  const cudaError_t ea = coop_attr(threads);
  if (ea != cudaSuccess) return ea;
  if (blocks > L->ncell) blocks = L->ncell;
  if (blocks <= 0) return cudaSuccess;
  CoopArgs a;
  a.ncell = L->ncell; a.tstart = L->tstart; a.tend = L->tend;
  a.C = L->C; a.RCONST = L->RCONST; a.ATOL = L->ATOL; a.RTOL = L->RTOL;
  a.ICNTRL = L->ICNTRL; a.RCNTRL = L->RCNTRL; a.order = L->order;
  a.ISTAT = L->ISTAT; a.RSTAT = L->RSTAT; a.IERR = L->IERR;
  a.qhead = L->qhead; a.nfail = L->nfail; a.ATOLr = L->ATOLr; a.RTOLr = L->RTOLr;
  a.ckpt = L->ckpt; a.ckpt_max = L->ckpt_max;
  cudaMemsetAsync(L->qhead, 0, sizeof(unsigned int), s);
  const size_t smem = coop_smem_bytes();
  if (threads == 128)
    rodas3_coop<128, 3><<<blocks, 128, smem, s>>>(a);
  else
    rodas3_coop<256, 2><<<blocks, 256, smem, s>>>(a);
  return cudaGetLastError();
}

#else  /* no tables for this mechanism */

extern "C" int rodas3_coop_ok(void) { return 0; }
extern "C" size_t rodas3_coop_smem_bytes(void) { return 0; }
extern "C" int rodas3_coop_blocks_per_sm(int) { return 0; }
extern "C" cudaError_t rodas3_coop_launch(const Rodas3Launch*, int, cudaStream_t) {
  return cudaErrorInvalidValue;
}

#endif
