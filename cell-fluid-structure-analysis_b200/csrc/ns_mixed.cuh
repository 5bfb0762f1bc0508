// Mixed-precision momentum solve: one batched BiCGSTAB sequence in FP32 with reliable updates
// of the solution and the residual in FP64 (residual replacement: van der Vorst & Ye, SIAM J. Sci.
// Comput. 22(5), 2000; group-wise solution updates: Sleijpen & van der Vorst, Computing 56, 1996;
// their mixed-precision GPU form: Clark et al., Comput. Phys. Commun. 181, 2010).
//
//   FP64: b, x (solution), xs = diag(A) x; the true residual is formed and rounded to r in one pass
//   FP32: r, r0, p, v, s, t (Krylov vectors), dx (correction accumulated since the last update)
//   every iteration (FP32 operator At32 = FP32 copy of A D^-1, FP64 dot products and scalars):
//     p = r + beta (p - omega v); v = At32 p; alpha = rho / (r0.v); s = r - alpha v;
//     t = At32 s; omega = (t.s) / (t.t); dx += alpha D^-1 p + omega D^-1 s; r = s - omega t
//   reliable update of component c when its iterated residual has dropped below delta times the
//   largest one since its last update, meets the tolerance, hits the iteration cap or nears a
//   breakdown:  x += dx; dx = 0; r64 = b - A x (FP64 operator); r = (float) r64
// The Krylov space is kept across updates (p, r0 and the scalars carry on), so the iteration
// count stays that of the FP64 solve instead of restarting with every correction. Convergence is
// decided on the FP64 true residual only, with the FP64 solve's criterion. The iterations and
// updates run in k_mp_solve (ns_resident.cuh); this file holds the state, the initialisation and the
// check. The penalty rows (diagonal 1e10) have unit diagonal in A D^-1, so
// FP32 holds them without overflow or loss. Components are independent (per-component scalars,
// masks and updates).
#pragma once

#include "ns_kernels.cuh"

namespace cfsa {

constexpr double kMixedDrift2 = 100.0;  // true / iterated residual (squared) that restarts the space

struct MixedState {
  double bnorm2[3], tol2[3], rnorm2[3];  // FP64 criterion; rnorm2: true residual at the last update
  double rho[3], alpha[3], omega[3], beta[3], r0norm2[3];
  double rin2[3];   // iterated FP32 residual, same norm
  double rmax2[3];  // largest iterated residual since the last update
  int iters[3], status[3], updates[3];
  int active;   // components iterating
  int upd;      // components updated at the end of this iteration
  int restart;  // components whose Krylov space restarts at that update (near-breakdown)
  int restart_next;  // components restarting at the next iteration (the FP32 recurrence drifted)
  int force;         // components whose r0 . v vanished: update and restart at this iteration's end
  int maxit;
  double delta2;  // update trigger: rin2 < delta2 * rmax2
  int restarts[3];  // Krylov-space restarts (drift or a growing true residual)
};

struct MixedArgs {
  SellView S;
  const float *At32;
  const double *At64, *diagA, *invA;
  const float *invA32;
  const double *b;
  double *x, *xs;  // FP64 solution, scaled solution D x
  float *r, *r0, *p, *v, *s, *t, *dx;
  int n;
  MixedState *ms;
  DevStatus *st;
  Reduce red;
  const double *cw;   // convergence-norm weights (diag(A)^-1), nullptr: unscaled ||r||
  const float *cw32;  // the same for the FP32 residual
};

// Init (after k_momentum_rhs wrote b and x = 0): r = r0 = (float) b, p = v = dx = 0;
// FP64 ||b|| in the convergence norm, rho = r0 . r.
__global__ void k_mp_init(MixedArgs A, double tol, int maxit, double delta) {
  if (A.st->halt) return;
  const int64_t n = A.n;
  __shared__ WarpSums<6> S;
  const int nblk = (A.n + kBlock - 1) / kBlock;
  int slot = 0;
  for (int bk = blockIdx.x; bk < nblk; bk += gridDim.x, ++slot) {
    const int i = bk * kBlock + threadIdx.x;
    double part[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    if (i < A.n) {
      const double w = A.cw ? A.cw[i] : 1.0;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const int64_t o = c * n + i;
        const double bi = A.b[o];
        const float ri = (float)bi;
        A.r[o] = ri;
        A.r0[o] = ri;
        A.p[o] = 0.f;
        A.v[o] = 0.f;
        A.dx[o] = 0.f;
        part[c] = (bi * bi) * w;
        part[3 + c] = (double)ri * (double)ri;
      }
    }
    warp_partial<6>(part, S, slot);
  }
  double tot[6];
  if (grid_reduce_strided<6>(S, slot, nblk, A.red, tot) && threadIdx.x == 0) {
    MixedState *m = A.ms;
    m->active = 0;
    m->upd = 0;
    m->restart = 0;
    m->restart_next = 0;
    m->force = 0;
    m->maxit = maxit;
    m->delta2 = delta * delta;
    for (int c = 0; c < 3; ++c) {
      m->bnorm2[c] = tot[c];
      m->rnorm2[c] = tot[c];
      m->rin2[c] = tot[c];
      m->rmax2[c] = tot[c];
      m->tol2[c] = tol * tol * tot[c];
      m->rho[c] = tot[3 + c];
      m->r0norm2[c] = tot[3 + c];
      m->alpha[c] = m->omega[c] = 1.0;
      m->beta[c] = 0.0;
      m->iters[c] = 0;
      m->updates[c] = 0;
      m->restarts[c] = 0;
      if (isnan(tot[c]) || isnan(tot[3 + c])) {
        m->status[c] = KS_BREAKDOWN;
      } else if (tot[c] == 0.0 || tot[c] <= m->tol2[c]) {
        m->status[c] = KS_CONVERGED;
      } else {
        m->status[c] = KS_RUNNING;
        m->active |= 1 << c;
      }
    }
  }
}

__global__ void k_mp_check(const MixedState *__restrict__ m, DevStatus *st, const int *__restrict__ barrier_err) {
  if (st->halt) return;
  int code = *barrier_err ? 4 : 0, it = 0;  // 4: the solve gave up waiting at a grid barrier
  for (int c = 0; c < 3; ++c) {
    it = max(it, m->iters[c]);
    if (m->status[c] == KS_MAXIT && code == 0) code = 1;
    if (m->status[c] == KS_BREAKDOWN && code == 0) code = 2;
  }
  st->iters[0] += (unsigned long long)it;
  if (code) {
    st->code = code;
    st->halt = 1;
  }
}

// ------------------------------------------------------------------------------------------
// Mixed-precision momentum CG (the CFSA_KRYLOV_CG momentum method with a mixed precision): one
// batched Jacobi CG sequence in FP32 with FP64 reliable updates, the scheme of the BiCGSTAB above
// applied to CG (residual replacement with group-wise solution updates, van der Vorst & Ye 2000).
//   FP64: b, x (solution), r64 (true residual); FP32: r, p, q, dx; FP32 copy A32 of A
//   every iteration (FP64 dot products and scalars):
//     q = A32 p; alpha = rho / (p.q); dx += alpha p; r -= alpha q; z = D^-1 r; rho' = r.z
//   reliable update of component c when its iterated residual has dropped below delta times the
//   largest one since its last update, meets the tolerance or hits the cap:
//     x += dx; dx = 0; r64 = b - A x (FP64 operator); r = (float) r64; rho' = r.z
//   then p = z + (rho'/rho) p: the search direction carries on across updates. Convergence is
//   decided on the FP64 true residual with the FP64 solve's criterion. An update that finds the
//   true residual more than 10x the iterated one, or larger than at the previous update, restarts
//   the direction (p = z).

// Init (after k_momentum_rhs wrote b and x = 0): r = (float) b, p = z = D^-1 r, dx = 0; the FP64
// ||b|| in the convergence norm and rho = r.z.
__global__ void k_mpc_init(MixedArgs A, double tol, int maxit, double delta) {
  if (A.st->halt) return;
  const int64_t n = A.n;
  __shared__ WarpSums<6> S;
  const int nblk = (A.n + kBlock - 1) / kBlock;
  int slot = 0;
  for (int bk = blockIdx.x; bk < nblk; bk += gridDim.x, ++slot) {
    const int i = bk * kBlock + threadIdx.x;
    double part[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    if (i < A.n) {
      const double w = A.cw ? A.cw[i] : 1.0;
      const float dinv = A.invA32[i];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const int64_t o = c * n + i;
        const double bi = A.b[o];
        const float ri = (float)bi;
        const float zi = dinv * ri;
        A.r[o] = ri;
        A.p[o] = zi;
        A.dx[o] = 0.f;
        part[c] = (bi * bi) * w;
        part[3 + c] = (double)ri * (double)zi;
      }
    }
    warp_partial<6>(part, S, slot);
  }
  double tot[6];
  if (grid_reduce_strided<6>(S, slot, nblk, A.red, tot) && threadIdx.x == 0) {
    MixedState *m = A.ms;
    m->active = 0;
    m->upd = 0;
    m->restart = 0;
    m->restart_next = 0;
    m->force = 0;
    m->maxit = maxit;
    m->delta2 = delta * delta;
    for (int c = 0; c < 3; ++c) {
      m->bnorm2[c] = tot[c];
      m->rnorm2[c] = tot[c];
      m->rin2[c] = tot[c];
      m->rmax2[c] = tot[c];
      m->tol2[c] = tol * tol * tot[c];
      m->rho[c] = tot[3 + c];
      m->alpha[c] = 0.0;
      m->beta[c] = 0.0;
      m->iters[c] = 0;
      m->updates[c] = 0;
      m->restarts[c] = 0;
      if (isnan(tot[c]) || isnan(tot[3 + c])) {
        m->status[c] = KS_BREAKDOWN;
      } else if (tot[c] == 0.0 || tot[c] <= m->tol2[c]) {
        m->status[c] = KS_CONVERGED;
      } else {
        m->status[c] = KS_RUNNING;
        m->active |= 1 << c;
      }
    }
  }
}

// ------------------------------------------------------------------------------------------
// Mixed-precision pressure solve: FP64 defect correction around the two-level CG with float
// storage (k_cg2l_resident<float>: operator values, inverse diagonal and Krylov vectors in float,
// arithmetic and reductions in FP64).
//   x = 0, r = b                                  (FP64, from k_pressure_rhs)
//   while ||r|| > tol ||b|| (the FP64 solve's criterion, on the FP64 true residual):
//     solve Lbc d = r in float to tol_in relative  (k_cg2l_resident<float>, one cooperative launch)
//     x += d;  r = b - Lbc x                       (FP64)
// The operator is L2-resident at the benchmark sizes and the solve is bound by the latency of its
// grid barriers, so float storage shortens the body of an iteration (half the bytes gathered per
// entry) but not its barrier; the sweeps add one FP64 product each.
struct PMixState {
  double bnorm2, tol2, rnorm2;  // outer criterion on the FP64 true residual
  int sweeps, status, active;
  int iters;       // inner iterations over all sweeps
  int bar_failed;  // an inner solve gave up at a grid barrier
  int max_sweeps;
  double tol_in;
};

struct PMixArgs {
  SellView S;
  const double *Ls, *invL;  // FP64 penalised operator (SELL) and its inverse diagonal
  const float *invL32;
  const double *b;
  double *x, *r;            // FP64 solution and true residual (x = 0, r = b on entry)
  float *r32, *x32, *p32, *s32;  // inner right-hand side, solution, and the two zero-on-entry vectors
  int n, scaled, maxit;
  CgState *cs;     // the FP64 solve's state (criterion of b from k_pressure_rhs; totals at the end)
  CgState *cs_in;  // the inner float solve
  PMixState *pm;
  DevStatus *st;
  Reduce red;
  const int *bar_err;
  cudaGraphConditionalHandle cond;
  int use_cond;
};

__global__ void k_pmx_init(PMixArgs A, double tol_in, int max_sweeps) {
  PMixState *m = A.pm;
  const bool halted = A.st && A.st->halt;
  m->bnorm2 = A.cs->bnorm2;
  m->tol2 = A.cs->tol2;
  m->rnorm2 = A.cs->bnorm2;
  m->sweeps = 0;
  m->iters = 0;
  m->bar_failed = 0;
  m->status = A.cs->status;
  m->active = halted ? 0 : A.cs->active;
  m->max_sweeps = max_sweeps;
  m->tol_in = tol_in;
}

// Sweep start: inner right-hand side r32 = (float) r, x32 = p32 = s32 = 0, inner criterion.
__global__ void k_pmx_prep(PMixArgs A) {
  if (!A.pm->active) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      A.cs_in->active = 0;
      if (A.use_cond) cudaGraphSetConditional(A.cond, 0);
    }
    return;
  }
  __shared__ WarpSums<2> S;
  const int nblk = (A.n + kBlock - 1) / kBlock;
  int slot = 0;
  for (int bk = blockIdx.x; bk < nblk; bk += gridDim.x, ++slot) {
    const int i = bk * kBlock + threadIdx.x;
    double part[2] = {0.0, 0.0};
    if (i < A.n) {
      const float rf = (float)A.r[i];
      A.r32[i] = rf;
      A.x32[i] = 0.f;
      A.p32[i] = 0.f;
      A.s32[i] = 0.f;
      const double rd = (double)rf;
      part[0] = rd * rd;
      part[1] = A.scaled ? rd * ((double)A.invL32[i] * rd) : rd * rd;
    }
    warp_partial<2>(part, S, slot);
  }
  double tot[2];
  if (grid_reduce_strided<2>(S, slot, nblk, A.red, tot) && threadIdx.x == 0) {
    CgState *c = A.cs_in;
    c->bb = tot[0];
    c->bnorm2 = tot[1];
    c->rnorm2 = tot[1];
    c->tol2 = A.pm->tol_in * A.pm->tol_in * tot[1];
    c->iters = 0;
    c->maxit = A.maxit;
    const bool run = tot[1] > 0.0 && !isnan(tot[1]);
    c->status = run ? KS_RUNNING : KS_BREAKDOWN;
    c->active = run ? 1 : 0;
  }
}

// x += d (FP64)
__global__ void k_pmx_xupdate(PMixArgs A) {
  if (!A.pm->active) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < A.n) A.x[i] += (double)A.x32[i];
}

// r = b - Lbc x (FP64 true residual, rows in SELL order, one thread per row); outer criterion,
// sweep count and loop condition.
__global__ void k_pmx_residual(PMixArgs A) {
  if (!A.pm->active) {
    if (A.use_cond && blockIdx.x == 0 && threadIdx.x == 0) cudaGraphSetConditional(A.cond, 0);
    return;
  }
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = (r < A.S.nrows_pad) ? A.S.perm[r] : -1;
  double part[1] = {0.0};
  if (i >= 0) {
    const int base = A.S.sptr[r >> 5] + (r & 31), len = A.S.len[r];
    double acc = 0.0;
    for (int k = 0; k < len; ++k) {
      const int pos = base + k * kSellC;
      acc += A.Ls[pos] * A.x[A.S.col[pos]];
    }
    const double ri = A.b[i] - acc;
    A.r[i] = ri;
    part[0] = A.scaled ? ri * (A.invL[i] * ri) : ri * ri;
  }
  double tot[1];
  if (grid_reduce<1>(part, A.red, tot) && threadIdx.x == 0) {
    PMixState *m = A.pm;
    m->sweeps += 1;
    m->iters += A.cs_in->iters;
    m->rnorm2 = tot[0];
    if (A.bar_err && *A.bar_err) {
      m->bar_failed = 1;
      m->status = KS_BREAKDOWN;
      m->active = 0;
    } else if (isnan(tot[0])) {
      m->status = KS_BREAKDOWN;
      m->active = 0;
    } else if (tot[0] <= m->tol2) {
      m->status = KS_CONVERGED;
      m->active = 0;
    } else if (A.cs_in->status == KS_BREAKDOWN) {
      m->status = KS_BREAKDOWN;
      m->active = 0;
    } else if (m->sweeps >= m->max_sweeps) {
      m->status = KS_MAXIT;
      m->active = 0;
    }
    if (A.use_cond) cudaGraphSetConditional(A.cond, m->active ? 1u : 0u);
  }
}

// After the sweeps: totals into the FP64 solve's state (for the statistics) and, on failure, the
// step's status word (as k_check_cg does for the FP64 solve).
__global__ void k_pmx_check(PMixArgs A, DevStatus *st) {
  const PMixState *m = A.pm;
  if (st->halt) return;
  A.cs->iters = m->iters;
  A.cs->rnorm2 = m->rnorm2;
  A.cs->status = m->status;
  A.cs->active = 0;
  st->iters[1] += (unsigned long long)m->iters;
  int code = 0;
  if (m->status == KS_MAXIT) code = 1;
  if (m->status == KS_BREAKDOWN) code = 2;
  if (m->bar_failed) code = 4;
  if (code) {
    st->code = code;
    st->halt = 1;
  }
}

__global__ void k_to_f32(int64_t n, const double *__restrict__ src, float *__restrict__ dst) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) dst[k] = (float)src[k];
}

}  // namespace cfsa
