/*
 * coop_adjoint.cuh -- discrete adjoint of the Rodas3 solve, one thread block
 * per cell (included by coop.cu; production build).
 *
 * The same adjoint as adjoint.cu (see there for the equations): backward over
 * the checkpoints, each step recomputes the Jacobian, the factors and the four
 * stages, then applies the transposed stage equations.  One thread per cell
 * walks ~100,000 dependent loads per step, 10-15 ms for any small batch; here a
 * step runs on the streams of the forward kernel (coop.cu) plus four more:
 *
 *   sweept   the solve with the transposed matrix on the same factors and
 *            inverses, parts in reverse
 *   tj       t_j = S_j . u for every reaction
 *   apart    the partials dA(j)/dV(i) at the stage's state, and in a second
 *            run their derivative along the stage vector at the step's start
 *   vthl     per species  VT = J^T u  and the Hessian term, sums of t_j times
 *            these
 *
 * and the rates' stream once more for the gradient with respect to ln k_j.
 */

struct CoopAdjAt : CoopAt<128> {
  static constexpr int YB = CELL;                    /* [y | FIX | constants] at the step's start */
  static constexpr int KX = YB + COOP_NX;            /* [stage vector | 0 ..] */
  static constexpr int UX = KX + COOP_NX;            /* [u | 0] */
  static constexpr int T = UX + NVAR + 1;            /* [t_j | 0] */
  static constexpr int BM = T + NREACT + 1;          /* [partials | 0] */
  static constexpr int DM = BM + COOP_NAPART + 1;    /* [their derivatives | 0] */
  static constexpr int MU = DM + COOP_NAPART + 1;    /* dL/d ln k_j */
  static constexpr int VT = MU + NREACT;
  static constexpr int HL = VT + NVAR;
  static constexpr int SC = HL + NVAR;               /* stoichiometric coefficients */
  static constexpr int END = SC + COOP_NSCOEF;
};

enum { A_TJ, A_PART, A_DUAL, A_VTHL, A_MU };

/* half of t_j's sums */
__device__ __forceinline__ double adj_tj_half(unsigned int cell, double acc, uint4 q) {
  using L = CoopAdjAt;
  const unsigned int w[3] = {q.y, q.z, q.w}, ctl = q.x >> 16, d = q.x & 0xFFFFu;
  const unsigned int u = coop_uniform(ctl & CL_UNIFORM);
  if (u & CL_FIRST) acc = 0.0;
#pragma unroll
  for (int t = 0; t < 3; ++t)
    acc = acc + coop_get<L::SC>(cell, w[t] & 0xFFFFu) * coop_get<L::UX>(cell, w[t] >> 16);
  if (u & CL_END) {
    acc = coop_fold(acc, ctl, (u >> 9) & 7u);
    coop_put_if<L::T>(ctl & CL_LEAD, cell, d, acc);
  }
  return acc;
}

/* half of the species' two sums */
__device__ __forceinline__ void adj_vthl_half(unsigned int cell, double& v, double& h, uint4 q) {
  using L = CoopAdjAt;
  const unsigned int w[3] = {q.y, q.z, q.w}, ctl = q.x >> 16, d = q.x & 0xFFFFu;
  const unsigned int u = coop_uniform(ctl & CL_UNIFORM);
  if (u & CL_FIRST) v = h = 0.0;
#pragma unroll
  for (int t = 0; t < 3; ++t) {
    const double tj = coop_get<L::T>(cell, w[t] & 0xFFFFu);
    v = v + tj * coop_get<L::BM>(cell, w[t] >> 16);
    h = h + tj * coop_get<L::DM>(cell, w[t] >> 16);
  }
  if (u & CL_END) {
    v = coop_fold(v, ctl, (u >> 9) & 7u);
    h = coop_fold(h, ctl, (u >> 9) & 7u);
    coop_put_if<L::VT>(ctl & CL_LEAD, cell, d, v);
    coop_put_if<L::HL>(ctl & CL_LEAD, cell, d, h);
  }
}

/* derivative of four partials f0*z1*z2 along the stage vector; the third
   factor of a partial is always the constant 1 */
__device__ __forceinline__ void adj_dual_op(unsigned int cell, uint4 a, uint4 b, int j) {
  using L = CoopAdjAt;
  const unsigned int w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const unsigned int o0 = w[2 * k] & 0xFFFFu, o1 = w[2 * k] >> 16, o2 = w[2 * k + 1] & 0xFFFFu;
    const double z1 = coop_get<L::YB>(cell, o1), z2 = coop_get<L::YB>(cell, o2);
    const double k1 = coop_get<L::KX>(cell, o1), k2 = coop_get<L::KX>(cell, o2);
    coop_put_if<L::DM>(j + k * 128 < COOP_NAPART, cell, COOP_UNIT * (j + k * 128),
                       coop_get<L::RX>(cell, o0) * (k1 * z2 + z1 * k2));
  }
}

/* MU(j) += t_j (A_j at the stage's state + dA_j along the stage vector) */
__device__ __forceinline__ void adj_mu_op(unsigned int cell, uint4 a, uint4 b, int j0) {
  using L = CoopAdjAt;
  const unsigned int w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int j = j0 + k * 128;
    if (j < NREACT && coop_has_k[j]) {
      const unsigned int o[3] = {w[2 * k] >> 16, w[2 * k + 1] & 0xFFFFu, w[2 * k + 1] >> 16};
      const double c = coop_get<L::RX>(cell, w[2 * k] & 0xFFFFu);
      const double ea = coop_get<L::V>(cell, o[0]), eb = coop_get<L::V>(cell, o[1]),
                   ec = coop_get<L::V>(cell, o[2]);
      const double za = coop_get<L::YB>(cell, o[0]), zb = coop_get<L::YB>(cell, o[1]),
                   zc = coop_get<L::YB>(cell, o[2]);
      const double ka = coop_get<L::KX>(cell, o[0]), kb = coop_get<L::KX>(cell, o[1]),
                   kc = coop_get<L::KX>(cell, o[2]);
      const double dak = c * (ka * zb * zc + kb * za * zc + kc * za * zb);
      const double x = coop_get<L::MU>(cell, COOP_UNIT * j) +
                       coop_get<L::T>(cell, COOP_UNIT * j) * (((c * ea) * eb) * ec + dak);
      coop_put<L::MU>(cell, COOP_UNIT * j, x);
    }
  }
}

template <int PROG>
__device__ __forceinline__ void adj_run(unsigned int cell, CoopFetch& f, int seg, int next) {
  const int2 sg = coop_segment<128>(seg);
  const uint4* cur = coop_stream<128>(sg);
  const uint4* nxt = coop_stream<128>(coop_segment<128>(next));
  double v = 0.0, h = 0.0;
  int j = threadIdx.x;
#pragma unroll 1
  for (int i = COOP_DEPTH; i <= sg.y; i += COOP_DEPTH) {
    const uint4* p = i < sg.y ? cur + i * 64 : nxt;
#pragma unroll
    for (int d = 0; d < COOP_DEPTH; ++d) {
      const uint4 a = f.q[d][0], b = f.q[d][1];
      if (PROG == A_TJ) {
        v = adj_tj_half(cell, v, a);
        v = adj_tj_half(cell, v, b);
      } else if (PROG == A_VTHL) {
        adj_vthl_half(cell, v, h, a);
        adj_vthl_half(cell, v, h, b);
      } else {
        if (PROG == A_PART) coop_rate_op<128, CoopAdjAt::BM>(cell, a, b, j, 128, COOP_NAPART);
        else if (PROG == A_DUAL) adj_dual_op(cell, a, b, j);
        else adj_mu_op(cell, a, b, j);
        j += 4 * 128;
      }
      f.q[d][0] = coop_ld<false>(p + d * 64);
      f.q[d][1] = coop_ld<false>(p + d * 64 + 32);
    }
  }
}

struct CoopAdjArgs {
  int ncell;
  const double* C0;
  const double* RCONST;
  const int* ISTAT;
  const double* ckpt;
  int ckpt_max;
  const double* lam;
  double* gC0;
  double* gK;
  int* ierr;
  const int* order;
};

__global__ void __launch_bounds__(128, 1) rodas3_coop_adjoint(CoopAdjArgs a) {
  using L = CoopAdjAt;
  constexpr int NT = 128, NE = (NVAR + NT - 1) / NT;
  const int tid = threadIdx.x;
  double* sm = reinterpret_cast<double*>(coop_smem) + COOP_NCOEF;
  const unsigned int cell = __reduce_max_sync(0xFFFFFFFFu, (unsigned int)__cvta_generic_to_shared(sm));
  int* s_ising = reinterpret_cast<int*>(sm + L::RED + 8);
  for (int i = tid; i < COOP_NCOEF; i += NT) reinterpret_cast<double*>(coop_smem)[i] = coop_coef[i];
  for (int i = tid; i < COOP_NSCOEF; i += NT) sm[L::SC + i] = coop_scoef[i];
  for (int i = tid; i < COOP_NX; i += NT) sm[L::KX + i] = 0.0;
  if (tid == 0) {
    sm[L::G + L::ZERO] = sm[L::X + NVAR] = sm[L::A + NREACT] = sm[L::RX + NREACT + COOP_NEXTRA] = 0.0;
    sm[L::G + L::ZERO - 1] = -1.0;
    sm[L::UX + NVAR] = sm[L::T + NREACT] = sm[L::BM + COOP_NAPART] = sm[L::DM + COOP_NAPART] = 0.0;
  }
  int place[NE], place_t[NE];
#pragma unroll
  for (int m = 0; m < NE; ++m) {
    place[m] = tid + m * NT < NVAR ? coop_place4[tid + m * NT] : NVAR;
    place_t[m] = tid + m * NT < NVAR ? coop_place_t4[tid + m * NT] : NVAR;
  }
  int chain[3];
  coop_chain_load<NT>(chain);
  CoopFetch f;
  coop_prime<NT, 1>(f, COOP_SEG_RATE);
  for (int q = blockIdx.x; q < a.ncell; q += gridDim.x) {
    const long col = a.order ? a.order[q] : q;
    const double* c0 = a.C0 + col * NSPEC;
    const double* rr = a.RCONST + col * NREACT;
    __syncthreads();                       /* the previous cell's results are out */
    for (int i = NVAR + tid; i < COOP_NX; i += NT)
      sm[L::V + i] = sm[L::YB + i] = i < NSPEC ? c0[i] : coop_ext[i - NSPEC];
    for (int j = tid; j < NREACT; j += NT) { sm[L::RX + j] = rr[j]; sm[L::MU + j] = 0.0; }
    for (int i = tid; i < COOP_NEXTRA; i += NT) {
      const int j = coop_extra_src[i];
      sm[L::RX + NREACT + i] = j >= 0 ? rr[j] * coop_extra_val[i] : coop_extra_val[i];
    }
    double lam[NE];
#pragma unroll
    for (int m = 0; m < NE; ++m)
      lam[m] = tid + m * NT < NVAR ? a.lam[col * NSPEC + tid + m * NT] : 0.0;
    const int nacc = a.ISTAT[col * 8 + 3];
    int ierr = nacc > a.ckpt_max ? -101 : 1;
    for (int n = ierr == 1 ? nacc - 1 : -1; n >= 0; --n) {
      const double* ck = a.ckpt + (col * a.ckpt_max + n) * (NVAR + 1);
      const double h = ck[NVAR];
      const double hc21 = 4.0 / h, hc1 = 1.0 / h, hc2 = -1.0 / h, hc3 = -(8.0 / 3.0) / h;
      double y[NE], ys[NE], f0[NE], k[4][NE];
      if (tid == 0) *s_ising = INT_MAX;
#pragma unroll
      for (int m = 0; m < NE; ++m) {
        y[m] = tid + m * NT < NVAR ? ck[tid + m * NT] : 0.0;
        if (tid + m * NT < NVAR) sm[L::YB + tid + m * NT] = y[m];
      }
      /* the accepted step's stages, as the forward kernel forms them */
      int singular = 0;
#pragma unroll 1
      for (int s = -1; s < 4 && !singular; ++s) {
        if (s == -1 || s >= 2) {
#pragma unroll
          for (int m = 0; m < NE; ++m) {
            ys[m] = s == -1 ? y[m] : s == 2 ? (y[m] + 2.0 * k[0][m]) + 0.0 * k[1][m] : ys[m] + 1.0 * k[2][m];
            if (tid + m * NT < NVAR) sm[L::V + tid + m * NT] = ys[m];
          }
          __syncthreads();
          coop_fun<NT, 1>(cell, f, sm, chain, s == -1 ? COOP_SEG_BPART0 : COOP_SEG_SWEEP);
        }
        if (s == -1) {
#pragma unroll
          for (int m = 0; m < NE; ++m) f0[m] = tid + m * NT < NVAR ? sm[L::X + tid + m * NT] : 0.0;
          coop_jacobian<NT, 1>(cell, f, sm, 1.0 / (h * 0.5), s_ising);
          singular = *s_ising != INT_MAX;
          if (!singular) coop_factor<NT, 1>(cell, f, sm);
          continue;
        }
#pragma unroll
        for (int m = 0; m < NE; ++m) {
          const int i = tid + m * NT;
          if (i < NVAR) {
            double v = s < 2 ? f0[m] : (sm[L::X + i] + hc1 * k[0][m]) + hc2 * k[1][m];
            if (s == 1) v = v + hc21 * k[0][m];
            if (s == 3) v = v + hc3 * k[2][m];
            sm[L::X + i] = v;
          }
        }
        __syncthreads();
        coop_run<P_SWEEP, NT, 1>(cell, f, COOP_SEG_SWEEP,
                                 s == 0 ? COOP_SEG_SWEEP : s < 3 ? COOP_SEG_RATE : COOP_SEG_SWEEPT);
#pragma unroll
        for (int m = 0; m < NE; ++m) {
          const double v = sm[L::X + place[m]];
          if (s == 0) k[0][m] = v;
          else if (s == 1) k[1][m] = v;
          else if (s == 2) k[2][m] = v;
          else k[3][m] = v;
        }
      }
      if (singular) {
        ierr = -8;
        coop_prime<NT, 1>(f, COOP_SEG_RATE);
        break;
      }
      /* adjoint of the step: W_s = m_s lambda, m = (2, 0, 1, 1) */
      double lamn[NE], w1[NE], w2[NE], w3[NE];
#pragma unroll
      for (int m = 0; m < NE; ++m) {
        lamn[m] = lam[m];
        w1[m] = 2.0 * lam[m];
        w2[m] = 0.0;
        w3[m] = lam[m];
      }
#pragma unroll 1
      for (int s = 3; s >= 0; --s) {
        __syncthreads();                   /* X, V, KX and UX are free again */
#pragma unroll
        for (int m = 0; m < NE; ++m) {
          const int i = tid + m * NT;
          if (s == 2) ys[m] = (y[m] + 2.0 * k[0][m]) + 0.0 * k[1][m];
          if (s == 1) ys[m] = y[m];
          if (i < NVAR) {
            sm[L::X + i] = s == 3 ? lam[m] : s == 2 ? w3[m] : s == 1 ? w2[m] : w1[m];
            sm[L::V + i] = ys[m];
            sm[L::KX + i] = s == 3 ? k[3][m] : s == 2 ? k[2][m] : s == 1 ? k[1][m] : k[0][m];
          }
        }
        __syncthreads();
        coop_run<P_SWEEP, NT, 1>(cell, f, COOP_SEG_SWEEPT, COOP_SEG_TJ);
        double u[NE];
#pragma unroll
        for (int m = 0; m < NE; ++m) {
          u[m] = sm[L::X + place_t[m]];
          if (tid + m * NT < NVAR) sm[L::UX + tid + m * NT] = u[m];
        }
        __syncthreads();
        adj_run<A_TJ>(cell, f, COOP_SEG_TJ, COOP_SEG_APART);
        adj_run<A_PART>(cell, f, COOP_SEG_APART, COOP_SEG_APART);
        adj_run<A_DUAL>(cell, f, COOP_SEG_APART, COOP_SEG_VTHL);
        __syncthreads();
        adj_run<A_VTHL>(cell, f, COOP_SEG_VTHL, COOP_SEG_RATE);
        adj_run<A_MU>(cell, f, COOP_SEG_RATE, s > 0 ? COOP_SEG_SWEEPT : COOP_SEG_RATE);
        __syncthreads();
#pragma unroll
        for (int m = 0; m < NE; ++m) {
          const int i = tid + m * NT < NVAR ? tid + m * NT : 0;
          const double v = sm[L::VT + i], hl = sm[L::HL + i];
          lamn[m] += hl;
          if (s > 0) lamn[m] += v;
          if (s == 3) {
            w1[m] += 2.0 * v + hc1 * u[m];
            w2[m] += hc2 * u[m];
            w3[m] += v + hc3 * u[m];
          } else if (s == 2) {
            w1[m] += 2.0 * v + hc1 * u[m];
            w2[m] += hc2 * u[m];
          } else if (s == 1) {
            w1[m] += hc21 * u[m];
          } else {
            lam[m] = lamn[m] + v;
          }
        }
      }
    }
    __syncthreads();
    double* g = a.gC0 + col * NSPEC;
#pragma unroll
    for (int m = 0; m < NE; ++m)
      if (tid + m * NT < NVAR) g[tid + m * NT] = ierr == 1 ? lam[m] : NAN;
    for (int i = NVAR + tid; i < NSPEC; i += NT) g[i] = 0.0;
    for (int j = tid; j < NREACT; j += NT) a.gK[col * NREACT + j] = ierr == 1 ? sm[L::MU + j] : NAN;
    if (tid == 0) a.ierr[col] = ierr;
  }
}

static size_t coop_adjoint_smem(void) {
  return ((size_t)CoopAdjAt::END + COOP_NCOEF) * sizeof(double);
}

extern "C" int rodas3_coop_adjoint_ok(void) { return coop_adjoint_smem() <= 227 * 1024 ? 1 : 0; }

extern "C" cudaError_t rodas3_coop_adjoint_launch(int ncell, const double* C0, const double* RCONST,
                                                  const int* ISTAT, const double* ckpt, int ckpt_max,
                                                  const double* lam, double* gC0, double* gK,
                                                  int* ierr, const int* order, int sms,
                                                  cudaStream_t s) {
  const cudaError_t e = cudaFuncSetAttribute(rodas3_coop_adjoint,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)coop_adjoint_smem());
  if (e != cudaSuccess) return e;
  const CoopAdjArgs a = {ncell, C0, RCONST, ISTAT, ckpt, ckpt_max, lam, gC0, gK, ierr, order};
  rodas3_coop_adjoint<<<ncell < sms ? ncell : sms, 128, coop_adjoint_smem(), s>>>(a);
  return cudaGetLastError();
}
