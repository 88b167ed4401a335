/*
 * coop.cu -- the cooperative Rodas3 kernel: one thread block per cell, the
 * whole cell state on chip.
 *
 * One thread per cell is right when hundreds of thousands of cells hide the
 * latency of each other's workspace accesses.  A small batch cannot: a thread
 * needs 2.5-4 ms for one attempt of a step (B200, fullchem, any batch of up to
 * a few thousand cells), whatever the GPU has idle.  Here a group of 128 or 256
 * threads owns one cell: the factors, the vectors, the rate constants and the
 * rates are in shared memory (110 KB for fullchem), the state and the stage
 * vectors in registers, so a solve reads HBM only to load a cell and store its
 * result, and an attempt takes 72 us.  A block holds one cell, or two when
 * there are more cells than one-cell blocks fit on the GPU (two per SM for both
 * shipped mechanisms: 296 cells on 148 SMs).  The groups drain the same cost-ordered queue
 * as the persistent kernel.
 *
 * Parallelism inside a cell comes from the instruction streams that
 * mechanism/coop.py generates (coop.inc), one list of operations per warp:
 *   Fun      rates A(j), then the destruction and production sums, each in the
 *            reference's order in one lane (gckpp_Function.F90:2170-5060); the
 *            few long ones from a buffer of their products;
 *   Jac      partials B(m), then the entries, straight into the factor array
 *            as -JVS, + 1/(H*gamma) on the diagonal; formed again at every
 *            attempt instead of stored (Y is unchanged after a rejection);
 *   KppDecomp by dependency levels: an entry's updates, in the reference's
 *            order (gckpp_LinearAlgebra.F90:46-84), as soon as their factors
 *            are final;
 *   KppSolve by levels of rows (:645-2311).
 * The FMA build (COOP_SPLIT) may round differently: there sums other than
 * Fun's are split over lanes, quotients become products with one reciprocal
 * per pivot (GC_IRECIP), the last rows are inverted as a block (coop_tail) and
 * the sweeps use inverses of their diagonal blocks, 22 levels in place of 130.
 * Built with --fmad=false the kernel reproduces the CPU oracle bit for bit.
 *
 * Step-size control, counters, options and the retry protocol are the
 * arithmetic of Integrate_Cell_S (gckpp_BatchIntegrator.F90:408-707) and of
 * the model's retry (fullchem_mod.F90:2436-2520), computed redundantly by
 * every thread of the cell so that every branch is uniform.
 *
 * Every barrier of a cell is reached by all threads of its group: the streams
 * of all warps hold the same number of barriers between two phases (checked by
 * the generator's test), and every branch around a barrier depends only on
 * values all threads hold identically (shared-memory words read after a
 * barrier, or scalars computed redundantly from them).  Nothing waits on
 * another block, nor on the block's other cell.
 */
#include <cuda_runtime.h>
#include <float.h>
#include <limits.h>
#include "rodas3_device.cuh"
#include "gc_root.h"
#include "rodas3_kernels.h"
/* sums may be split over lanes where the build need not round like the
   reference */
#define COOP_SPLIT GC_IRECIP
#include "coop.inc"

#if MECH_COOP

/* shared memory: the coefficients of the sums, shared by the block's cells,
   then each cell (in doubles).  G holds the factors, the tail block, the
   inverses of the sweeps' parts, -1/U(i,i), -1 and 0 (see mechanism/coop.py); V the state that
   Fun and Jac read, with the fixed species and the constants of the rate
   tables behind it; A the rates, or the Jacobian partials of a part of the
   columns; X [vector | 0 | second place].  The state and the stage vectors
   live in registers (thread t of the cell owns species t, t + NT, ..).  A and
   RX end in a 0, the operand of missing products.  B is 16-byte aligned (as the
   cells and COOP_NCOEF are even), for loads of two products. */
template <int NT>
struct CoopAt {
  static constexpr int ZERO = NT == 128 ? COOP_NG4 : COOP_NG8;   /* index of 0 in G */
  static constexpr int RECIP = ZERO - 1 - NVAR;                  /* of -1/U(0,0) */
  static constexpr int G = 0;
  static constexpr int V = G + ZERO + 1;
  static constexpr int X = V + COOP_NX;
  static constexpr int A = X + 2 * NVAR + 2;
  static constexpr int RX = A + NREACT + 1;
  static constexpr int B = (RX + NREACT + COOP_NEXTRA + 2) / 2 * 2;   /* products of the long sums */
  static constexpr int RED = B + COOP_BUFFER;   /* error sums of up to 8 warps, two ints */
  static constexpr int CELL = (RED + 10) / 2 * 2;
};
extern __shared__ __align__(16) unsigned char coop_smem[];
/* the generator fits the cell into shared memory by the same sum */
static_assert(CoopAt<128>::CELL == COOP_CELL4 && CoopAt<256>::CELL == COOP_CELL8, "layout of a cell");
/* offsets in the streams: bytes (COOP_UNIT 8), or doubles where an array is
   beyond the 64 KB that 16 bits reach (COOP_UNIT 1; then a multiplication more
   for each).  An element's offset is its index times COOP_UNIT. */
#define COOP_BYTES (8 / COOP_UNIT)

/* control bits of the streams (mechanism/coop.py) */
#define CL_LEAD   1u
#define CL_FIRST  2u
#define CL_END    4u
#define CL_START  8u
#define CL_DIAG   16u
#define CL_SCALED 32u
#define CL_DIAGS  (1u << 15)       /* some lane of the warp has CL_DIAG */
#define CL_UNIFORM (CL_FIRST | CL_END | ~0u << 9)   /* alike in all lanes */

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
  int nsteps, ncons, rej_last, rej_more, newstep, ierr, attempt;
};

/* ---- warp streams ---------------------------------------------------------
   What bounds a cell is the instruction stream of its busiest warp: a level
   takes as long as one warp needs for its operations (~100 instructions of ~6
   cycles each: ALU latencies, shared memory, exchanges).  Every warp therefore
   executes its own list of operations (mechanism/coop.py), whose words hold
   offsets that need no tests, and fetches them COOP_DEPTH operations ahead into
   registers, across the phases of the attempt (L2 answers after ~320 cycles);
   and the programs have few levels.  One cell, fullchem, time of an attempt on
   a B200: rounds of the whole block with words loaded one round ahead 185 us;
   streams 118 us; with inverses of the sweeps' parts and of the tail block
   (13 + 9 levels instead of 61 + 69) 86 us; with byte offsets, six products to
   an operation of Fun and a buffer without bank conflicts 72 us (137,000 cycles:
   ~85,000 warp instructions in four warps, 6-7 cycles each; the FP64 pipe is
   used at 3%).  Two cells in a block share the schedulers' gaps: 290 cells take
   78 us per attempt, 16,000 cells 3.4 M attempts per second. */
struct CoopFetch {
  uint4 q[COOP_DEPTH][2];
};

template <bool kShare>
__device__ __forceinline__ uint4 coop_ld(const uint4* p) {
  uint4 v;
  if (kShare)   /* the other cells of the block read the same words soon */
    asm("ld.global.nc.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  else
    asm("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
        : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

template <int NT>
__device__ __forceinline__ int2 coop_segment(int seg) {
  const int k = seg * (NT / 32) + ((threadIdx.x % NT) >> 5);
  return NT == 128 ? coop_seg4[k] : coop_seg8[k];
}

template <int NT>
__device__ __forceinline__ const uint4* coop_stream(int2 sg) {
  return reinterpret_cast<const uint4*>(NT == 128 ? coop_words4 : coop_words8) + sg.x +
         (threadIdx.x & 31);
}

/* barrier of one cell's threads */
template <int NT, int NG>
__device__ __forceinline__ void coop_sync(void) {
  if (NG == 1) __syncthreads();
  else asm volatile("bar.sync %0, %1;" :: "r"(1 + (int)threadIdx.x / NT), "n"(NT) : "memory");
}

/* Shared-memory access by 32-bit address: `cell` is the address of the cell's
   first array, SO a compile-time place, off an offset from a stream. */
template <int SO>
__device__ __forceinline__ double coop_get(unsigned int cell, unsigned int off) {
  double x;
  asm volatile("ld.shared.f64 %0, [%1+%2];" : "=d"(x) : "r"(cell + off * COOP_BYTES), "n"(SO * 8));
  return x;
}
template <int SO>
__device__ __forceinline__ void coop_put(unsigned int cell, unsigned int off, double x) {
  asm volatile("st.shared.f64 [%0+%1], %2;" :: "r"(cell + off * COOP_BYTES), "n"(SO * 8), "d"(x) : "memory");
}
template <int SO>
__device__ __forceinline__ void coop_put_if(bool p, unsigned int cell, unsigned int off, double x) {
  asm volatile("{ .reg .pred q; setp.ne.u32 q, %3, 0; @q st.shared.f64 [%0+%1], %2; }"
               :: "r"(cell + off * COOP_BYTES), "n"(SO * 8), "d"(x), "r"((unsigned int)p) : "memory");
}

/* a word that all lanes of the warp hold, as a warp-uniform value: branches on
   it need no convergence bookkeeping */
__device__ __forceinline__ unsigned int coop_uniform(unsigned int x) {
  return __reduce_or_sync(0xFFFFFFFFu, x);
}

enum { P_RATE, P_BUFD, P_DEST, P_PROD, P_BUFP, P_JVS, P_ONE, P_LU, P_SWEEP };

/* sum over the lane groups of a warp: the s exchanges that its largest group
   needs, kept by the lanes whose group is that large (ctl) */
template <int K>
__device__ __forceinline__ double coop_exchange(double acc, unsigned int lg) {
  const double y = __shfl_xor_sync(0xFFFFFFFFu, acc, 1 << K);
  asm("{ .reg .pred q; setp.gt.u32 q, %1, %2; @q add.f64 %0, %0, %3; }"
      : "+d"(acc) : "r"(lg), "n"(K), "d"(y));
  return acc;
}
__device__ __forceinline__ double coop_fold(double acc, unsigned int ctl, unsigned int s) {
  const unsigned int lg = (ctl >> 6) & 7u;
  if (s > 0) {
    acc = coop_exchange<0>(acc, lg);
    if (s > 1) {
      acc = coop_exchange<1>(acc, lg);
      if (s > 2) {
        acc = coop_exchange<2>(acc, lg);
        if (s > 3) {
          acc = coop_exchange<3>(acc, lg);
          if (s > 4) acc = coop_exchange<4>(acc, lg);
        }
      }
    }
  }
  return acc;
}

/* four products ((f0*f1)*f2)*f3 */
template <int NT, int OUT>
__device__ __forceinline__ void coop_rate_op(unsigned int cell, uint4 a, uint4 b, int j, int step,
                                             int n) {
  const unsigned int w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  double f[4][4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    f[k][0] = coop_get<CoopAt<NT>::RX>(cell, w[2 * k] & 0xFFFFu);
    f[k][1] = coop_get<CoopAt<NT>::V>(cell, w[2 * k] >> 16);
    f[k][2] = coop_get<CoopAt<NT>::V>(cell, w[2 * k + 1] & 0xFFFFu);
    f[k][3] = coop_get<CoopAt<NT>::V>(cell, w[2 * k + 1] >> 16);
  }
#pragma unroll
  for (int k = 0; k < 4; ++k)
    coop_put_if<OUT>(j + k * step < n, cell, COOP_UNIT * (j + k * step),
                      ((f[k][0] * f[k][1]) * f[k][2]) * f[k][3]);
}

/* six products of a sum that one lane adds up in order (dest, prod) */
template <int PROG, int NT>
__device__ __forceinline__ double coop_line_op(unsigned int cell, unsigned int coef, double acc,
                                               uint4 qa, uint4 qb) {
  using L = CoopAt<NT>;
  const unsigned int w[6] = {qa.z, qa.w, qb.x, qb.y, qb.z, qb.w}, u = coop_uniform(qa.y & CL_UNIFORM);
  double a[6], b[6];
#pragma unroll
  for (int t = 0; t < 6; ++t) {
    a[t] = PROG == P_DEST ? coop_get<L::RX>(cell, w[t] & 0xFFFFu) : coop_get<0>(coef, w[t] & 0xFFFFu);
    b[t] = coop_get<PROG == P_DEST ? L::V : L::A>(cell, w[t] >> 16);
  }
  if (u & CL_FIRST) acc = 0.0;
#pragma unroll
  for (int t = 0; t < 6; ++t) acc = acc + a[t] * b[t];
  if (u & CL_END) {
    const unsigned int d = qa.x & 0xFFFFu;
    double x = acc;
    if (PROG == P_PROD) x = acc - coop_get<L::X>(cell, d) * coop_get<L::V>(cell, d);
    coop_put_if<L::X>(qa.y & CL_LEAD, cell, d, x);
  }
  return acc;
}

/* half of a sum operation: three products, then perhaps the entry's end */
template <int NT>
__device__ __forceinline__ double coop_sum_half(unsigned int cell, unsigned int coef, double acc,
                                                uint4 q) {
  const unsigned int w[3] = {q.y, q.z, q.w}, ctl = q.x >> 16, d = q.x & 0xFFFFu;
  const unsigned int u = coop_uniform(ctl & CL_UNIFORM);
  double a[3], b[3];
#pragma unroll
  for (int t = 0; t < 3; ++t) {
    a[t] = coop_get<0>(coef, w[t] & 0xFFFFu);
    b[t] = coop_get<CoopAt<NT>::A>(cell, w[t] >> 16);
  }
  if (u & CL_FIRST) acc = 0.0;
#pragma unroll
  for (int t = 0; t < 3; ++t) acc = acc + a[t] * b[t];
  if (u & CL_END) {
    acc = coop_fold(acc, ctl, (u >> 9) & 7u);
    coop_put_if<CoopAt<NT>::G>(ctl & CL_LEAD, cell, d, acc);
  }
  return acc;
}

/* four entries of one product */
template <int NT, int OUT>
__device__ __forceinline__ void coop_one_op(unsigned int cell, unsigned int coef, uint4 a, uint4 b) {
  const unsigned int w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  double f[4], g[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    f[k] = coop_get<0>(coef, w[2 * k] >> 16);
    g[k] = coop_get<CoopAt<NT>::A>(cell, w[2 * k + 1]);
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const unsigned int d = w[2 * k] & 0xFFFFu;
    coop_put_if<OUT>(d != 0xFFFFu, cell, d, f[k] * g[k]);
  }
}

/* level operation of the factorisation (P_LU) or a sweep */
template <int PROG, int NT, int NG>
__device__ __forceinline__ double coop_level_op(unsigned int cell, double acc, uint4 qa, uint4 qb) {
  using L = CoopAt<NT>;
  constexpr int BASE = PROG == P_LU ? L::G : L::X;
  const unsigned int ctl = qa.y, d = qa.x & 0xFFFFu, e = qa.x >> 16;
  const unsigned int u = coop_uniform(ctl & CL_UNIFORM);
  const unsigned int w[6] = {qa.z, qa.w, qb.x, qb.y, qb.z, qb.w};
  double a[6], b[6];
#pragma unroll
  for (int t = 0; t < 3; ++t) {
    a[t] = coop_get<L::G>(cell, w[t] & 0xFFFFu);
    b[t] = coop_get<BASE>(cell, w[t] >> 16);
  }
  if (u & CL_FIRST) {
    acc = 0.0;
    asm volatile("{ .reg .pred q; setp.ne.u32 q, %2, 0; @q ld.shared.f64 %0, [%1+%3]; }"
                 : "+d"(acc) : "r"(cell + d * COOP_BYTES), "r"(ctl & CL_START), "n"(BASE * 8));
  }
  if (u & (4u << 12)) {                    /* more than three products */
#pragma unroll
    for (int t = 3; t < 6; ++t) {
      a[t] = coop_get<L::G>(cell, w[t] & 0xFFFFu);
      b[t] = coop_get<BASE>(cell, w[t] >> 16);
    }
#pragma unroll
    for (int t = 0; t < 6; ++t) acc = acc - a[t] * b[t];
  } else {
#pragma unroll
    for (int t = 0; t < 3; ++t) acc = acc - a[t] * b[t];
  }
  if (u & CL_END) {
    acc = coop_fold(acc, ctl, (u >> 9) & 7u);
#if COOP_SPLIT
    if (PROG == P_LU) {
      const double r = coop_get<L::G>(cell, e);   /* -1/U, or -1 */
      if ((u & CL_DIAGS) && (ctl & (CL_LEAD | CL_DIAG)) == (CL_LEAD | CL_DIAG))
        coop_put<L::G>(cell, e, -1.0 / acc);
      if (!(ctl & CL_DIAG)) acc = -(acc * r);
    }
#else
    if ((ctl & (CL_LEAD | CL_SCALED)) == (CL_LEAD | CL_SCALED)) acc = acc / coop_get<L::G>(cell, e);
#endif
    coop_put_if<BASE>(ctl & CL_LEAD, cell, d, acc);
  }
  if (u >> 20) {
    for (unsigned int k = u >> 20; k > 0; --k) coop_sync<NT, NG>();
  }
  return acc;
}

/* fetch the first operations of a segment */
template <int NT, int NG>
__device__ __forceinline__ void coop_prime(CoopFetch& f, int seg) {
  const uint4* p = coop_stream<NT>(coop_segment<NT>(seg));
#pragma unroll
  for (int d = 0; d < COOP_DEPTH; ++d) {
    f.q[d][0] = coop_ld<(NG > 1)>(p + d * 64);
    f.q[d][1] = coop_ld<(NG > 1)>(p + d * 64 + 32);
  }
}

/* run a segment; the fetches of its last operations belong to `next`.
   n: number of products (rates) */
template <int PROG, int NT, int NG>
__device__ __forceinline__ void coop_run(unsigned int cell, CoopFetch& f, int seg, int next,
                                         int n = 0) {
  const int2 sg = coop_segment<NT>(seg);
  const uint4* cur = coop_stream<NT>(sg);
  const uint4* nxt = coop_stream<NT>(coop_segment<NT>(next));
  const unsigned int coef = (unsigned int)__cvta_generic_to_shared(coop_smem);
  double acc = 0.0;
  int j = threadIdx.x % NT;                    /* rates: number of the first product */
#pragma unroll 1
  for (int i = COOP_DEPTH; i <= sg.y; i += COOP_DEPTH) {
    const uint4* p = i < sg.y ? cur + i * 64 : nxt;
#pragma unroll
    for (int d = 0; d < COOP_DEPTH; ++d) {
      const uint4 a = f.q[d][0], b = f.q[d][1];
      if (PROG == P_RATE || PROG == P_BUFD) {
        coop_rate_op<NT, PROG == P_RATE ? CoopAt<NT>::A : CoopAt<NT>::B>(cell, a, b, j, NT, n);
        j += 4 * NT;
      } else if (PROG == P_ONE || PROG == P_BUFP) {
        coop_one_op<NT, PROG == P_ONE ? CoopAt<NT>::G : CoopAt<NT>::B>(cell, coef, a, b);
      } else if (PROG == P_DEST || PROG == P_PROD) {
        acc = coop_line_op<PROG, NT>(cell, coef, acc, a, b);
      } else if (PROG == P_LU || PROG == P_SWEEP) {
        acc = coop_level_op<PROG, NT, NG>(cell, acc, a, b);
      } else {
        acc = coop_sum_half<NT>(cell, coef, acc, a);
        acc = coop_sum_half<NT>(cell, coef, acc, b);
      }
      /* into the registers just read: a load into others would be copied at
         the end of the loop, and the copy would wait for it */
      f.q[d][0] = coop_ld<(NG > 1)>(p + d * 64);
      f.q[d][1] = coop_ld<(NG > 1)>(p + d * 64 + 32);
    }
  }
}

/* Fun's long sums (a lane per sum: species, first product, blocks): the
   products wait in B, so a term costs a load and an addition, in order. */
template <int NT>
__device__ __forceinline__ double coop_chain(const double* sm, int first, int blocks) {
  const double2* b = reinterpret_cast<const double2*>(sm + CoopAt<NT>::B + first);
  double s = 0.0;
  const int most = __reduce_max_sync(0xFFFFFFFFu, blocks), last = blocks > 0 ? blocks - 1 : 0;
  double2 v[4];
#pragma unroll
  for (int t = 0; t < 4; ++t) v[t] = b[t];
#pragma unroll 2
  for (int k = 0; k < most; ++k) {
    /* the next block's loads run during this one's additions */
    const double2* nb = b + 4 * (k < last ? k + 1 : last);
    double2 u[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) u[t] = nb[t];
    double x = s;
#pragma unroll
    for (int t = 0; t < 4; ++t) x = (x + v[t].x) + v[t].y;
    s = k < blocks ? x : s;
#pragma unroll
    for (int t = 0; t < 4; ++t) v[t] = u[t];
  }
  return s;
}

#if COOP_TAIL
/* The tail block's Schur complement becomes its negative inverse: Gauss-Jordan
   elimination in place without pivoting (the factorisation has none), rows over
   the warps, columns over the lanes.  A step scales the pivot row in its warp,
   hands it over through A (free here; two rows in turn, so that one barrier per
   step is enough) and updates the other rows, their factors coming from the
   pivot column's lane.  ~250 cycles a step; the 61-level program that walked
   these pivots took 49 of its levels, ~1,000 cycles each, for them. */
template <int NT, int NG>
__device__ __forceinline__ void coop_tail(double* sm) {
  using L = CoopAt<NT>;
  constexpr int M = COOP_TAIL, W = NT / 32, R = M / W, C = M / 32;
  const int lane = threadIdx.x & 31, warp = (threadIdx.x % NT) >> 5;
  double* D = sm + L::G + COOP_BLOCK;
  double* buf = sm + L::A;
  double a[R][C];
#pragma unroll
  for (int q = 0; q < R; ++q)
#pragma unroll
    for (int c = 0; c < C; ++c) a[q][c] = D[(warp * R + q) * M + c * 32 + lane];
#pragma unroll 1
  for (int w = 0; w < W; ++w) {
    const int kc = w * R / 32;                /* the pivots' column block */
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int kl = (w * R + r) & 31;
      double row[C];
      if (warp == w) {
        const double piv = __shfl_sync(0xFFFFFFFFu, C == 1 || kc == 0 ? a[r][0] : a[r][C - 1], kl);
        const double inv = 1.0 / piv;
#pragma unroll
        for (int c = 0; c < C; ++c) {
          row[c] = lane == kl && c == kc ? inv : a[r][c] * inv;
          a[r][c] = row[c];
          buf[(r & 1) * M + c * 32 + lane] = row[c];
        }
      }
      coop_sync<NT, NG>();
      if (warp != w) {
#pragma unroll
        for (int c = 0; c < C; ++c) row[c] = buf[(r & 1) * M + c * 32 + lane];
      }
#pragma unroll
      for (int q = 0; q < R; ++q) {
        if (q != r || warp != w) {
          const double f = __shfl_sync(0xFFFFFFFFu, C == 1 || kc == 0 ? a[q][0] : a[q][C - 1], kl);
#pragma unroll
          for (int c = 0; c < C; ++c)
            a[q][c] = (lane == kl && c == kc ? 0.0 : a[q][c]) - f * row[c];
        }
      }
    }
  }
#pragma unroll
  for (int q = 0; q < R; ++q)
#pragma unroll
    for (int c = 0; c < C; ++c) D[(warp * R + q) * M + c * 32 + lane] = -a[q][c];
  coop_sync<NT, NG>();
}
#endif

/* a thread's long sum of round r (32 sums each): the first warp's are
   productions, the last's destructions */
template <int NT>
__device__ __forceinline__ void coop_chain_load(int* chain, int r = 0) {
  const int tid = threadIdx.x % NT, k = 3 * (32 * r + (tid & 31) + (tid < 32 ? 32 * COOP_CHAINS : 0));
#pragma unroll
  for (int t = 0; t < 3; ++t) chain[t] = coop_chain_of[k + t];
}

/* the warp's long sums, finish(species, sum); the first round's are kept in
   registers over the solve (`chain`), further ones are rare */
template <int NT, class F>
__device__ __forceinline__ void coop_chains(const double* sm, const int* chain, F finish) {
  int c[3] = {chain[0], chain[1], chain[2]};
#pragma unroll 1
  for (int r = 0;;) {
    const double x = coop_chain<NT>(sm, c[1], c[2]);
    if (c[0] >= 0) finish(c[0], x);
    if (++r == COOP_CHAINS) break;
    coop_chain_load<NT>(c, r);
  }
}

/* Fun_SPLIT of the state in V into X; `after`: the segment that follows */
template <int NT, int NG>
__device__ __forceinline__ void coop_fun(unsigned int cell, CoopFetch& f, double* sm,
                                         const int* chain, int after) {
  using L = CoopAt<NT>;
  const int tid = threadIdx.x % NT;
  (void)sm; (void)tid; (void)chain;
  /* Fun_SPLIT: X = P_VAR - D_VAR*V; the destruction sums need no rates,
     so they run before the barrier that publishes A */
  coop_run<P_RATE, NT, NG>(cell, f, COOP_SEG_RATE, COOP_SEG_DEST, NREACT);
#if COOP_BUFFER
  coop_run<P_DEST, NT, NG>(cell, f, COOP_SEG_DEST, COOP_SEG_BUFD);
  coop_run<P_BUFD, NT, NG>(cell, f, COOP_SEG_BUFD, COOP_SEG_PROD, COOP_NBUFD);
  coop_sync<NT, NG>();
  /* the last warp adds up the long destruction sums, then the first the
     long production sums, which wait for all products */
  if (tid >= NT - 32)
    coop_chains<NT>(sm, chain, [sm](int i, double d) { sm[L::X + i] = d; });
  coop_run<P_PROD, NT, NG>(cell, f, COOP_SEG_PROD, COOP_SEG_BUFP);
  coop_run<P_BUFP, NT, NG>(cell, f, COOP_SEG_BUFP, after);
  coop_sync<NT, NG>();
  if (tid < 32)
    coop_chains<NT>(sm, chain, [sm](int i, double p) { sm[L::X + i] = p - sm[L::X + i] * sm[L::V + i]; });
#else
  coop_run<P_DEST, NT, NG>(cell, f, COOP_SEG_DEST, COOP_SEG_PROD);
  coop_sync<NT, NG>();
  coop_run<P_PROD, NT, NG>(cell, f, COOP_SEG_PROD, after);
#endif
  coop_sync<NT, NG>();
}

/* -Jac0 + ghinv on the diagonal, into G; *ising (INT_MAX before) */
template <int NT, int NG>
__device__ __forceinline__ void coop_jacobian(unsigned int cell, CoopFetch& f, double* sm,
                                              double ghinv, int* s_ising) {
  using L = CoopAt<NT>;
  constexpr int NE = (NVAR + NT - 1) / NT;
  const int tid = threadIdx.x % NT;
  /* Jac_SP straight into ros_PrepareMatrix's form: G = -JVS, a part of
     the columns at a time, then ghinv on the diagonal.  KppDecomp's
     singularity test reads each prepared diagonal before its row is
     eliminated, so it is taken here: *ising becomes the lowest failing
     row + 1.  Diagonals without updates are final: their reciprocals. */
#pragma unroll 1
  for (int q = 0; q < COOP_PARTS; ++q) {
    const int seg = COOP_SEG_BPART0 + 3 * q;
    coop_run<P_RATE, NT, NG>(cell, f, seg, seg + 1, COOP_NBP(q));
    coop_sync<NT, NG>();
    coop_run<P_JVS, NT, NG>(cell, f, seg + 1, seg + 2);
    coop_run<P_ONE, NT, NG>(cell, f, seg + 2, q + 1 < COOP_PARTS ? seg + 3 : COOP_SEG_LU);
    coop_sync<NT, NG>();
  }
#pragma unroll
  for (int m = 0; m < NE; ++m) {
    const int k = tid + m * NT;
    if (k < NVAR) {
      const int o = __ldg(coop_diag + k);
      const double g = sm[L::G + (o >> 1)] + ghinv;
      if (fabs(g) < DBL_MIN) atomicMin(s_ising, k + 1);
      sm[L::G + (o >> 1)] = g;
#if COOP_SPLIT
      if (o & 1) sm[L::G + L::RECIP + k] = -1.0 / g;
#endif
    }
  }
  coop_sync<NT, NG>();
}

template <int NT, int NG>
__device__ __forceinline__ void coop_factor(unsigned int cell, CoopFetch& f, double* sm) {
  /* KppDecomp entry by entry, in levels */
  coop_run<P_LU, NT, NG>(cell, f, COOP_SEG_LU, COOP_SEG_SWEEP);
#if COOP_TAIL
  coop_tail<NT, NG>(sm);
#endif
}

/* load the cell's column and set the integrator state (lane_start of the
   one-thread-per-cell kernels); attempt 1 is the retry: Hstart taken as 0
   and the retry tolerances */
template <int NT, int NG>
__device__ __forceinline__ void coop_start(CoopCell& c, const CoopArgs& a, double* sm, double* y,
                                           long col, int attempt) {
  using L = CoopAt<NT>;
  const int tid = threadIdx.x % NT;
  c.col = col;
  c.attempt = attempt;
  const double* cc = a.C + col * NSPEC;
  const double* rr = a.RCONST + col * NREACT;
#pragma unroll
  for (int m = 0; m < (NVAR + NT - 1) / NT; ++m) y[m] = tid + m * NT < NVAR ? cc[tid + m * NT] : 0.0;
  for (int i = NVAR + tid; i < COOP_NX; i += NT) sm[L::V + i] = i < NSPEC ? cc[i] : coop_ext[i - NSPEC];
  for (int j = tid; j < NREACT; j += NT) sm[L::RX + j] = rr[j];
  for (int i = tid; i < COOP_NEXTRA; i += NT) {
    const int j = coop_extra_src[i];
    sm[L::RX + NREACT + i] = j >= 0 ? rr[j] * coop_extra_val[i] : coop_extra_val[i];
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
  coop_sync<NT, NG>();
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
template <int NT, int NG>
__device__ __forceinline__ int coop_end(CoopCell& c, const CoopArgs& a, double* sm, double* y) {
  const int tid = threadIdx.x % NT;
  if (a.nfail && c.attempt == 0 && c.ierr < 0) {
    if (tid == 0) {
      coop_store_istat(c, a, 0);
      atomicAdd(&a.nfail[0], 1);
    }
    coop_sync<NT, NG>();
    coop_start<NT, NG>(c, a, sm, y, c.col, 1);
    if (c.ierr == 0) return 0;
  }
  if (c.o.ierr_early == 0) {
    double* cc = a.C + c.col * NSPEC;
#pragma unroll
    for (int m = 0; m < (NVAR + NT - 1) / NT; ++m)
      if (tid + m * NT < NVAR) cc[tid + m * NT] = y[m];
  }
  if (tid == 0) {
    coop_store_istat(c, a, c.attempt);
    if (c.attempt && c.ierr < 0) atomicAdd(&a.nfail[1], 1);
    double* rs = a.RSTAT + c.col * 3;
    rs[0] = c.st.texit; rs[1] = c.st.hexit; rs[2] = c.st.hnew;
    a.IERR[c.col] = c.ierr;
  }
  return 1;
}

/* err**(1/3) of the step-size factor */
__device__ __forceinline__ double coop_root(double x) {
#if COOP_SPLIT
  if (x < 1.0e300) return gc_root3(x);
#endif
  return gc_pow(x, 1.0 / ROS_ELO);
}

/* One pass of TimeLoop/UntilAccepted (gckpp_BatchIntegrator.F90:535-704)
   for the block's cell; returns 1 when the cell is finished (c.ierr holds
   IERR).  The statement-level arithmetic is that of step_begin,
   step_prologue, step_factor and step_stages in rodas3_kernels.cu. */
template <int NT, int NG>
__device__ __forceinline__ int coop_attempt(CoopCell& c, const CoopArgs& a, CoopFetch& f,
                                            unsigned int cell, double* sm, double* y, const int* place,
                                            const int* chain) {
  using L = CoopAt<NT>;
  const int tid = threadIdx.x % NT;
  constexpr int NE = (NVAR + NT - 1) / NT;      /* species of a thread */
  const double Tend = a.tend;
  const double dir = (Tend >= a.tstart) ? 1.0 : -1.0;
  double* s_err = sm + L::RED;
  int* s_ising = reinterpret_cast<int*>(sm + L::RED + 8);

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

  const double dH = dir * c.H;
  const double hc1 = 1.0 / dH, hc2 = -1.0 / dH, hc3 = -(8.0 / 3.0) / dH, hc21 = 4.0 / dH;
  const double ghinv = 1.0 / (dH * 0.5);
  if (tid == 0) *s_ising = INT_MAX;
  double f0[NE], k1[NE], k2[NE], k3[NE], yn[NE];

  /* s = -1: Fcn0, the Jacobian and its factorisation.  A retried attempt
     forms Fcn0 and the Jacobian again from the unchanged state (the same
     values; the counters move once per step), so neither is stored.
     s = 0..3: the stages (per-element operation order of :595-632). */
#pragma unroll 1
  for (int s = -1; s < 4; ++s) {
    if (s == -1 || s >= 2) {
      /* the state that Fun reads: Y, then Ynew = (Y + 2 K1) + 0 K2, then
         + 1 K3 (yn still holds stage 3's value, rounded as the reference's
         expression rounds it) */
#pragma unroll
      for (int m = 0; m < NE; ++m) {
        const int k = tid + m * NT;
        if (s == -1) yn[m] = y[m];
        else if (s == 2) yn[m] = (y[m] + 2.0 * k1[m]) + 0.0 * k2[m];
        else yn[m] = yn[m] + 1.0 * k3[m];
        if (k < NVAR) sm[L::V + k] = yn[m];
      }
      if (s >= 2) c.st.nfun += 1;
      coop_sync<NT, NG>();
      coop_fun<NT, NG>(cell, f, sm, chain, s == -1 ? COOP_SEG_BPART0 : COOP_SEG_SWEEP);
    }
    if (s == -1) {
#pragma unroll
      for (int m = 0; m < NE; ++m) f0[m] = tid + m * NT < NVAR ? sm[L::X + tid + m * NT] : 0.0;
      coop_jacobian<NT, NG>(cell, f, sm, ghinv, s_ising);
      c.st.ndec += 1;
      if (*s_ising != INT_MAX) {
        c.st.nsng += 1;
        c.ncons += 1;
        coop_prime<NT, NG>(f, COOP_SEG_RATE);
        coop_sync<NT, NG>();      /* every thread has read *s_ising */
        if (c.ncons <= 5) { c.H = c.H * 0.5; return 0; }
        c.ierr = -8;
        return 1;
      }
      coop_factor<NT, NG>(cell, f, sm);
      continue;
    }
#pragma unroll
    for (int m = 0; m < NE; ++m) {
      const int k = tid + m * NT;
      if (k < NVAR) {
        double v;
        if (s < 2) {
          v = f0[m];
          if (s == 1) v = v + hc21 * k1[m];
          if (!c.o.autonomous) {
            /* dFdT = (Fun(Y) - Fcn0)/delta: Fun has no explicit time here, so
               its second evaluation is Fcn0 itself */
            const double dfdt = (f0[m] - f0[m]) / (sqrt(ROUNDOFF) * fmaxF(1.0e-6, fabs(c.T)));
            v = v + (s == 0 ? dH * 0.5 : dH * 1.5) * dfdt;
          }
        } else {
          v = (sm[L::X + k] + hc1 * k1[m]) + hc2 * k2[m];
          if (s == 3) v = v + hc3 * k3[m];
        }
        sm[L::X + k] = v;
      }
    }
    coop_sync<NT, NG>();
    coop_run<P_SWEEP, NT, NG>(cell, f, COOP_SEG_SWEEP, s == 0 ? COOP_SEG_SWEEP : COOP_SEG_RATE);
    c.st.nsol += 1;
    if (s < 3) {
#pragma unroll
      for (int m = 0; m < NE; ++m) {
        const double v = sm[L::X + place[m]];
        if (s == 0) k1[m] = v;
        else if (s == 1) k2[m] = v;
        else k3[m] = v;
      }
    }
  }

  /* Ynew, Yerr and the scaled error terms in parallel; the WRMS sum over
     warps, or in species order by one thread where the build rounds like the
     reference */
  const double* atol = c.attempt ? a.ATOLr : a.ATOL;
  const double* rtol = c.attempt ? a.RTOLr : a.RTOL;
  double err = 0.0;
#pragma unroll
  for (int m = 0; m < NE; ++m) {
    const int i = tid + m * NT;
    if (i < NVAR) {
      const double yi = y[m];
      const double k4 = sm[L::X + place[m]];
      yn[m] = (((yi + 2.0 * k1[m]) + 0.0 * k2[m]) + 1.0 * k3[m]) + 1.0 * k4;
      const double ye = (((0.0 + 0.0 * k1[m]) + 0.0 * k2[m]) + 0.0 * k3[m]) + 1.0 * k4;
      const double ymax = fmaxF(fabs(yi), fabs(yn[m]));
      const double scal = c.o.vectortol ? (__ldg(atol + i) + __ldg(rtol + i) * ymax)
                                        : (__ldg(atol) + __ldg(rtol) * ymax);
      const double q = ye / scal;
#if COOP_SPLIT
      err = err + q * q;
#else
      sm[L::X + i] = q;
#endif
    }
  }
#if COOP_SPLIT
#pragma unroll
  for (int k = 16; k > 0; k >>= 1) err = err + __shfl_xor_sync(0xFFFFFFFFu, err, k);
  if ((tid & 31) == 0) s_err[tid >> 5] = err;
  coop_sync<NT, NG>();
  err = 0.0;
#pragma unroll
  for (int w = 0; w < NT / 32; ++w) err = err + s_err[w];
#else
  coop_sync<NT, NG>();
  if (tid == 0) {
    for (int i = 0; i < NVAR; ++i) {
      const double q = sm[L::X + i];
      err = err + q * q;
    }
    s_err[0] = err;
  }
  coop_sync<NT, NG>();
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
#pragma unroll
      for (int m = 0; m < NE; ++m)
        if (tid + m * NT < NVAR) ck[tid + m * NT] = y[m];
      if (tid == 0) ck[NVAR] = c.H;
    }
#pragma unroll
    for (int m = 0; m < NE; ++m) y[m] = c.o.clamp ? fmaxF(yn[m], 0.0) : yn[m];
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
  coop_sync<NT, NG>();        /* s_err read by all */
  return 0;
}

/* NG cells per block, each with NT threads and its own part of the shared
   memory.  The cells of a block meet at every attempt, so that they read the
   same stream words at about the same time and share them through L1; in
   between each synchronises on its own barrier. */
template <int NT, int NG>
__global__ void __launch_bounds__(NT * NG, NG > 1 ? 1 : 2) rodas3_coop(CoopArgs a) {
  __shared__ unsigned int s_pos[NG];
  const int g = NG == 1 ? 0 : threadIdx.x / NT, tid = threadIdx.x % NT;
  double* sm = reinterpret_cast<double*>(coop_smem) + COOP_NCOEF + g * CoopAt<NT>::CELL;
  /* warp-uniform, so that it is added by the load itself */
  const unsigned int cell = __reduce_max_sync(0xFFFFFFFFu, (unsigned int)__cvta_generic_to_shared(sm));
  for (int i = threadIdx.x; i < COOP_NCOEF; i += NT * NG)
    reinterpret_cast<double*>(coop_smem)[i] = coop_coef[i];
  if (tid == 0) {
    using L = CoopAt<NT>;
    sm[L::G + L::ZERO] = sm[L::X + NVAR] = sm[L::A + NREACT] = sm[L::RX + NREACT + COOP_NEXTRA] = 0.0;
    sm[L::G + L::ZERO - 1] = -1.0;
  }
  __syncthreads();
  CoopFetch f;
  coop_prime<NT, NG>(f, COOP_SEG_RATE);
  CoopCell c;
  constexpr int NE = (NVAR + NT - 1) / NT;
  double y[NE];
  int place[NE];              /* where the sweeps leave the thread's species */
#pragma unroll
  for (int m = 0; m < NE; ++m)
    place[m] = tid + m * NT < NVAR ? (NT == 128 ? coop_place4 : coop_place8)[tid + m * NT] : NVAR;
  int chain[3];
  coop_chain_load<NT>(chain);
  int have = 0, drained = 0;
  for (;;) {
    while (!have && !drained) {
      if (tid == 0) s_pos[g] = atomicAdd(a.qhead, 1u);
      coop_sync<NT, NG>();
      const unsigned int p = s_pos[g];
      coop_sync<NT, NG>();    /* s_pos read by all before it is written again */
      if (p >= (unsigned int)a.ncell) {
        drained = 1;
      } else {
        coop_start<NT, NG>(c, a, sm, y, (long)a.order[p], 0);
        have = c.ierr == 0 || !coop_end<NT, NG>(c, a, sm, y);
      }
    }
    if (NG > 1) {
      if (!__syncthreads_or(have)) break;
    } else if (!have) {
      break;
    }
    if (have && coop_attempt<NT, NG>(c, a, f, cell, sm, y, place, chain)) {
      have = !coop_end<NT, NG>(c, a, sm, y);
      coop_sync<NT, NG>();    /* the result is stored before the next cell loads */
    }
  }
}

#if COOP_SPLIT
#include "coop_adjoint.cuh"
#else
extern "C" int rodas3_coop_adjoint_ok(void) { return 0; }
extern "C" cudaError_t rodas3_coop_adjoint_launch(int, const double*, const double*, const int*,
                                                  const double*, int, const double*, double*,
                                                  double*, int*, const int*, int, cudaStream_t) {
  return cudaErrorInvalidValue;
}
#endif

static size_t coop_smem_bytes(int threads, int cells) {
  const int cell = threads == 128 ? CoopAt<128>::CELL : CoopAt<256>::CELL;
  return ((size_t)cells * cell + COOP_NCOEF) * sizeof(double);
}

/* cells per block of the shared form: fullchem's shared memory (110 KB a cell)
   and both mechanisms' registers (228 and 254 per thread) hold no third */
#define COOP_NG 2

/* the kernel instances: threads per cell (128 or 256), cells per block */
static const void* coop_kernel(int threads, int cells) {
  if (threads == 128) return cells == 1 ? (const void*)rodas3_coop<128, 1> : (const void*)rodas3_coop<128, COOP_NG>;
  if (threads == 256) return cells == 1 ? (const void*)rodas3_coop<256, 1> : (const void*)rodas3_coop<256, COOP_NG>;
  return nullptr;
}

static cudaError_t coop_attr(int threads, int cells) {
  const void* k = coop_kernel(threads, cells);
  if (!k) return cudaErrorInvalidValue;
  return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)coop_smem_bytes(threads, cells));
}

extern "C" int rodas3_coop_ok(void) {
  return coop_smem_bytes(128, 1) <= 227 * 1024 && coop_smem_bytes(256, 1) <= 227 * 1024 ? 1 : 0;
}

extern "C" size_t rodas3_coop_smem_bytes(void) { return coop_smem_bytes(128, 1); }

extern "C" int rodas3_coop_blocks_per_sm(int threads) {
  if (!rodas3_coop_ok() || coop_attr(threads, 1) != cudaSuccess) return 0;
  int nb = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, coop_kernel(threads, 1), threads,
                                                    coop_smem_bytes(threads, 1)) != cudaSuccess)
    return 0;
  return nb;
}

/* bps: blocks per SM that the caller allows (0: as many as fit) */
extern "C" cudaError_t rodas3_coop_launch(const Rodas3Launch* L, int sms, int bps,
                                          cudaStream_t s) {
  if (!rodas3_coop_ok()) return cudaErrorInvalidValue;
  const int threads = L->threads;
  const int occ = rodas3_coop_blocks_per_sm(threads);
  if (occ <= 0) return cudaErrorInvalidValue;
  int cells = 1, blocks = sms * (bps > 0 && bps < occ ? bps : occ);
  if (bps <= 0 && L->ncell > blocks && coop_smem_bytes(threads, COOP_NG) <= 227 * 1024) {
    cells = COOP_NG;
    blocks = sms;
  }
  const cudaError_t ea = coop_attr(threads, cells);
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
  void* args[] = {&a};
  const cudaError_t el = cudaLaunchKernel(coop_kernel(threads, cells), dim3(blocks), dim3(threads * cells),
                                          args, coop_smem_bytes(threads, cells), s);
  if (el != cudaSuccess) return el;
  return cudaGetLastError();
}

#else  /* no tables for this mechanism */

extern "C" int rodas3_coop_ok(void) { return 0; }
extern "C" size_t rodas3_coop_smem_bytes(void) { return 0; }
extern "C" int rodas3_coop_blocks_per_sm(int) { return 0; }
extern "C" int rodas3_coop_adjoint_ok(void) { return 0; }
extern "C" cudaError_t rodas3_coop_adjoint_launch(int, const double*, const double*, const int*,
                                                  const double*, int, const double*, double*,
                                                  double*, int*, const int*, int, cudaStream_t) {
  return cudaErrorInvalidValue;
}
extern "C" cudaError_t rodas3_coop_launch(const Rodas3Launch*, int, int, cudaStream_t) {
  return cudaErrorInvalidValue;
}

#endif
