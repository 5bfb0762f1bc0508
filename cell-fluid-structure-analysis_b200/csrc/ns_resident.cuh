// Resident Krylov solves: one cooperative launch of one CTA per SM runs a whole momentum solve (CG or
// BiCGSTAB, FP64 or FP32 with FP64 reliable updates) or the whole pressure BiCGSTAB.
//
// What bounds them: the momentum product (the operator's stream and the gathers of x) on large meshes,
// the latency of a phase (barrier, block partials, one chain of row loads) on small ones. As separate
// kernels inside a conditional graph node an iteration paid three to five launches and the node's own
// turn-around: 39 us per CG iteration at 32k tets where the work is 5 us.
//
// An iteration is a sequence of phases; each phase runs over 32-position chunks, and a grid barrier
// separates phases that read what other CTAs wrote:
//   * a row phase walks the CTA's two runs of SELL slices (SellView::rfirst: one of vertex rows, one of
//     edge rows, which are shorter), warps taking slices from a shared counter;
//   * a vector phase walks a contiguous range of 256-position blocks of the natural order, so a CTA
//     meets the same entries in every vector phase.
// Dot products keep the tree of grid_reduce: warp sums per chunk, 8 chunks in order per block partial,
// 256 accumulators over the block partials, warp butterflies and an in-order sum of 8. The chunk sums
// stay in shared memory, the block partials go to global memory ([value][block], so that a warp reads 32
// neighbouring blocks of a value at once), and after the barrier every CTA forms the totals itself and
// takes the same decisions: the bits do not depend on the number of CTAs, and no CTA waits for another
// one's scalars. Scalars live in a shared-memory copy of the solver state; CTA 0 writes it back.
// Vectors are read with plain loads: the barrier's acquire orders them after the other CTAs' stores.
// Consecutive phases walk their range in opposite directions, so the entries a phase touched last, which
// L2 still holds, are the next one's first.
#pragma once

#include "ns_kernels.cuh"
#include "ns_mixed.cuh"

namespace cfsa {


struct ResidentArgs {
  GridBarrier bar;
  double *part;   // block partials [2][kMaxRed][stride]
  int stride;
  double *slots;  // chunk sums in global memory, slots_per_cta doubles per CTA; nullptr: in shared memory
  int slots_per_cta;
};

template <int T>  // threads per CTA
struct Resident {
  static constexpr int kWarps = T / 32;
  const ResidentArgs &R;
  double *s_slots;  // dynamic shared memory (chunk sums)
  unsigned int phase = 0;
  bool rev = false;  // direction of the next phase
  int buf = 0;       // partials buffer of the next reduction: a CTA may write the next phase's partials
                     // while another still reads this one's
  // The CTA's chunks in the current phase: na from a0 on, then nc from c0 on (both on block
  // boundaries); all chunks of the phase's order.
  int a0 = 0, na = 0, c0 = 0, nc = 0, nchunk = 0;

  __device__ Resident(const ResidentArgs &r, double *dyn) : R(r), s_slots(dyn) {}

  __device__ __forceinline__ bool sync() { return grid_sync(R.bar, phase); }
  __device__ __forceinline__ double *slots() const {
    return R.slots ? R.slots + (size_t)blockIdx.x * R.slots_per_cta : s_slots;
  }
  // The q-th chunk of the phase: the first range before the second, each in the phase's direction.
  __device__ __forceinline__ int chunk(int q, int &slot) const {
    const bool second = q >= na;
    const int k = second ? q - na : q, n = second ? nc : na, l = rev ? n - 1 - k : k;
    slot = second ? na + l : l;
    return (second ? c0 : a0) + l;
  }

  template <int NV>
  __device__ __forceinline__ void chunk_sums(const double (&v)[NV], int slot) const {
    double *sl = slots() + (size_t)slot * NV;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const double w = warp_sum(v[j]);
      if ((threadIdx.x & 31) == 0) sl[j] = w;
    }
  }

  // The CTA's runs of slices and the counter its warps take further slices from.
  __device__ __forceinline__ int *begin_rows(const SellView &S) {
    __shared__ int s_next;
    const int *f = S.rfirst + blockIdx.x, *f2 = f + gridDim.x + 1;
    a0 = f[0];
    na = f[1] - a0;
    c0 = f2[0];
    nc = f2[1] - c0;
    nchunk = S.nrows_pad / kSellC;
    if (threadIdx.x == 0) s_next = kWarps;
    __syncthreads();
    return &s_next;
  }

  // f(r, i, part) for every row i (SELL position r) of the CTA's runs.
  template <int NV, class F>
  __device__ __forceinline__ void rows(const SellView &S, F &&f) {
    int *next = begin_rows(S);
    for (int q = threadIdx.x >> 5; q < na + nc; q = run_next_slice(next)) {
      int slot;
      const int r = chunk(q, slot) * kSellC + (int)(threadIdx.x & 31);
      const int i = S.perm[r];
      double part[NV];
#pragma unroll
      for (int j = 0; j < NV; ++j) part[j] = 0.0;
      if (i >= 0) f(r, i, part);
      chunk_sums<NV>(part, slot);
    }
    rev = !rev;
  }

  // Row products of the CTA's run against NC right-hand sides: finish(i, acc, own, part) for every row
  // i, with acc[c] the row's product, own[c] = own(c, i) and part its NV sums. One thread per row adds
  // its entries in ascending column order (as sell_spmv_row), in chunks of U: indices and values, then
  // the gathers, then the sums. Bound: L1 serves the gathers, about six cycles of the SM for 32 lanes
  // spread over eleven lines (under ncu at 415k tets 73% of its peak, DRAM 0.57 of the copy rate). With one
  // or two FP64 components, and in the 256-thread form, the next chunk's indices and values are requested
  // along with the gathers; with three, or in FP32, the registers that holds are worth more to longer
  // chunks: three components at 1M tets 118 against 139 us (577 MB, 4.9 TB/s), FP32 81 against 98 us; two
  // components 95 against 100 us.
  // load(c, j) reads entry j of x_c with a plain load, since other CTAs rewrite x between the phases of
  // a launch.
  template <int NV, int NC, int U, int MASK, class TV, class TA, class L, class O, class F>
  __device__ __forceinline__ void products(const SellView &S, const TV *val, TA, L &&load, O &&own, F &&finish) {
    int *next = begin_rows(S);
    constexpr bool kAhead = T <= 256 || (sizeof(TV) == 8 && !(NC == 3 && MASK == 7));
    const int lane = threadIdx.x & 31;
    for (int q = threadIdx.x >> 5; q < na + nc; q = run_next_slice(next)) {
      int slot;
      const int sl = chunk(q, slot);
      const int i = S.perm[sl * kSellC + lane], len = S.len[sl * kSellC + lane], base = S.sptr[sl] + lane;
      double part[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) part[v] = 0.0;
      if (i >= 0) {
        TA acc[NC], ov[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) acc[c] = TA(0);
        int j[U];
        TV a[U];
        auto fetch = [&](int k, int (&jj)[U], TV (&aa)[U]) {
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const bool in = k + u < len;
            jj[u] = in ? __ldcs(S.col + base + (k + u) * kSellC) : 0;
            aa[u] = in ? __ldcs(val + base + (k + u) * kSellC) : TV(0);
          }
        };
        fetch(0, j, a);
        for (int k = 0; k < len; k += U) {
          TA xv[U][NC];
#pragma unroll
          for (int u = 0; u < U; ++u)
#pragma unroll
            for (int c = 0; c < NC; ++c)
              if ((MASK >> c) & 1) xv[u][c] = (k + u < len) ? load(c, j[u]) : TA(0);
          int jn[U];
          TV an[U];
          if constexpr (kAhead) fetch(k + U, jn, an);
#pragma unroll
          for (int u = 0; u < U; ++u)
#pragma unroll
            for (int c = 0; c < NC; ++c)
              if (((MASK >> c) & 1) && k + u < len) acc[c] += a[u] * xv[u][c];
          if constexpr (kAhead) {
#pragma unroll
            for (int u = 0; u < U; ++u) j[u] = jn[u], a[u] = an[u];
          } else if (k + U < len) {
            fetch(k + U, j, a);
          }
        }
#pragma unroll
        for (int c = 0; c < NC; ++c) ov[c] = ((MASK >> c) & 1) ? own(c, i) : TA(0);
        finish(i, acc, ov, part);
      }
      chunk_sums<NV>(part, slot);
    }
    rev = !rev;
  }

  // The CTA's natural blocks.
  __device__ __forceinline__ void begin_entries(int n) {
    nchunk = (n + 31) / 32;
    const int nblk = (n + kBlock - 1) / kBlock;
    a0 = kSlicesPerBlock * (int)((int64_t)nblk * blockIdx.x / gridDim.x);
    na = min(kSlicesPerBlock * (int)((int64_t)nblk * (blockIdx.x + 1) / gridDim.x), nchunk) - a0;
    nc = 0;
  }

  // Vector phase: apply(c, i, common(i), load(c, i), scalar(c), part) for every entry i < n of the CTA's
  // natural blocks and every component c in `mask`, the loads ahead of the stores; value 3 v + c of the phase
  // sums part[v] (NV = 0: no sums). With 1024 threads the components follow one another and two chunks' loads
  // are in flight, which leaves the 64 registers of a thread room (FP64 BiCGSTAB spills 36 bytes, the other
  // solves none) where all components of one entry at a time did not (momentum CG iteration at 1M tets
  // 180 -> 161 us); with fewer threads there is room for all components at once, and short ranges want the
  // latency paid once (512 threads at 250k tets 54 against 57 us).
  template <int NV, class S, class C, class L, class F>
  __device__ __forceinline__ void vector(int n, int mask, S &&scalar, C &&common, L &&load, F &&apply) {
    using V = decltype(load(0, 0));
    using W = decltype(common(0));
    begin_entries(n);
    const int lane = threadIdx.x & 31;
    if constexpr (T >= 1024) {
      constexpr int K = 2;
      for (int q = K * (int)(threadIdx.x >> 5); q < na; q += K * kWarps) {
        W w[K];
        int slot;
#pragma unroll
        for (int u = 0; u < K; ++u) w[u] = common(min(32 * chunk(min(q + u, na - 1), slot) + lane, n - 1));
#pragma unroll 1
        for (int c = 0; c < 3; ++c) {
          if (!((mask >> c) & 1)) continue;
          const auto sc = scalar(c);
          V v[K];
#pragma unroll
          for (int u = 0; u < K; ++u) v[u] = load(c, min(32 * chunk(min(q + u, na - 1), slot) + lane, n - 1));
#pragma unroll
          for (int u = 0; u < K; ++u) {
            if (q + u >= na) break;
            const int i = 32 * chunk(q + u, slot) + lane;
            double part[NV > 0 ? NV : 1] = {};
            if (i < n) apply(c, i, w[u], v[u], sc, part);
            if constexpr (NV > 0) {
              double *sl = slots() + (size_t)slot * 3 * NV + c;
#pragma unroll
              for (int j = 0; j < NV; ++j) {
                const double t = warp_sum(part[j]);
                if (lane == 0) sl[3 * j] = t;
              }
            }
          }
        }
      }
    } else {
      constexpr int K = (T <= 256 && NV == 0) ? 2 : 1;
      const decltype(scalar(0)) sc[3] = {scalar(0), scalar(1), scalar(2)};
      for (int q = threadIdx.x >> 5; q < na; q += K * kWarps) {
        V v[K][3];
        W w[K];
        int i[K], slot[K];
#pragma unroll
        for (int u = 0; u < K; ++u) {
          const int k = q + u * kWarps;
          i[u] = (u == 0 || k < na) ? 32 * chunk(k, slot[u]) + lane : n;
          const int il = min(i[u], n - 1);  // past the end: loads that are not used, no divergence
          w[u] = common(il);
#pragma unroll
          for (int c = 0; c < 3; ++c)
            if ((mask >> c) & 1) v[u][c] = load(c, il);
        }
#pragma unroll
        for (int u = 0; u < K; ++u) {
          double sum[NV > 0 ? 3 * NV : 1] = {};
          if (i[u] < n) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
              if (!((mask >> c) & 1)) continue;
              double part[NV > 0 ? NV : 1] = {};
              apply(c, i[u], w[u], v[u][c], sc[c], part);
#pragma unroll
              for (int j = 0; j < NV; ++j) sum[3 * j + c] = part[j];
            }
          }
          if constexpr (NV > 0) chunk_sums<3 * NV>(sum, slot[u]);
        }
      }
    }
    rev = !rev;
  }

  // Totals of the sums of the phase just run, in every thread of warp 0; false: a barrier wait ran out.
  template <int NV>
  __device__ __forceinline__ bool reduce(double (&tot)[NV]) {
    __shared__ double s_tree[kMaxRed][kBlock / 32];
    double *part = R.part + (size_t)buf * kMaxRed * R.stride;
    buf ^= 1;
    __syncthreads();  // chunk sums
    const double *sl = slots();
    const int ba = (na + kSlicesPerBlock - 1) / kSlicesPerBlock, bc = (nc + kSlicesPerBlock - 1) / kSlicesPerBlock;
    for (int t = threadIdx.x; t < (ba + bc) * NV; t += T) {
      const int l = t / NV, j = t % NV;
      const bool second = l >= ba;
      const int b = second ? c0 / kSlicesPerBlock + l - ba : a0 / kSlicesPerBlock + l;
      const int q0 = second ? na + kSlicesPerBlock * (l - ba) : kSlicesPerBlock * l, q1 = second ? na + nc : na;
      double s = 0.0;
#pragma unroll
      for (int w = 0; w < kSlicesPerBlock; ++w)
        if (q0 + w < q1) s += sl[(size_t)(q0 + w) * NV + j];
      __stcg(part + (size_t)j * R.stride + b, s);
    }
    if (!sync()) return false;
    const int nblk = (nchunk + kSlicesPerBlock - 1) / kSlicesPerBlock;
    for (int t = threadIdx.x; t < NV * kBlock; t += T) {  // accumulator a of value j
      const int j = t / kBlock, a = t & (kBlock - 1);
      const double *pj = part + (size_t)j * R.stride;
      constexpr int kB = 8;  // block partials in flight per thread
      double s = 0.0;
      for (int b = a; b < nblk; b += kB * kBlock) {
        double v[kB];
#pragma unroll
        for (int q = 0; q < kB; ++q) v[q] = (b + q * kBlock < nblk) ? __ldcg(pj + b + q * kBlock) : 0.0;
#pragma unroll
        for (int q = 0; q < kB; ++q)
          if (b + q * kBlock < nblk) s += v[q];
      }
      s = warp_sum(s);
      if ((t & 31) == 0) s_tree[j][a >> 5] = s;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
#pragma unroll
      for (int j = 0; j < NV; ++j) {
        double s = 0.0;
#pragma unroll
        for (int w = 0; w < kBlock / 32; ++w) s += s_tree[j][w];
        tot[j] = s;
      }
    }
    return true;
  }
};

// Scalar step of each running component: lane c of warp 0 runs f(c), which says whether component c
// runs on; the new mask goes to *mask in shared memory and to every thread.
template <int NC, class F>
__device__ __forceinline__ int each_component(int active, int *mask, F &&f) {
  if (threadIdx.x < 32) {
    const int c = threadIdx.x;
    bool on = c < NC && ((active >> c) & 1);
    if (on) on = f(c);
    const unsigned int m = __ballot_sync(0xffffffffu, on);
    if (c == 0) *mask = (int)m;
  }
  __syncthreads();
  return *mask;
}

// tot[c] for a run-time c without indexing registers
template <int NC, int NV>
__device__ __forceinline__ double pick(const double (&tot)[NV], int c, int first = 0) {
  double v = 0.0;
#pragma unroll
  for (int k = 0; k < NC; ++k)
    if (c == k) v = tot[first + k];
  return v;
}

// ------------------------------------------------------------------------------------------
// Batched momentum CG (recurrences and stopping rule: k_mcg_init's comment).
template <int T, int U>
__global__ void __launch_bounds__(T, 1) k_mcg_solve(BicgArgs A, ResidentArgs R) {
  extern __shared__ double s_slots[];
  __shared__ BicgState s;
  if (A.st && A.st->halt) return;
  if (threadIdx.x == 0) s = *A.bs;
  if (blockIdx.x == 0 && threadIdx.x == 0 && A.st) A.st->body_runs[A.slot] += 1;
  __syncthreads();
  Resident<T> G(R, s_slots);
  const int64_t n = A.n;
  int active = s.active;
  while (active) {
    // q = A p, alpha = absnew / (p . q)
    with_mask<3>(active, [&](auto mk) {
      constexpr int MASK = decltype(mk)::value;
      const auto pk = [&](int c, int j) { return A.pk[c * n + j]; };
      G.template products<3, 3, U, MASK>(A.S, A.At, double(), pk, pk,
                                         [&](int i, const double *acc, const double *own, double (&part)[3]) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          if (!((MASK >> c) & 1)) continue;
          A.v[c * n + i] = acc[c];
          part[c] = own[c] * acc[c];
        }
      });
    });
    double pq[3];
    if (!G.template reduce<3>(pq)) return;
    active = each_component<3>(active, &s.active, [&](int c) {
      const double d = pick<3>(pq, c);
      if (d == 0.0) {
        s.status[c] = KS_BREAKDOWN;
        return false;
      }
      s.alpha[c] = s.rho[c] / d;
      return true;
    });
    if (!active) break;
    // x += alpha p, r -= alpha q, z = D^-1 r; r.r and r.z; convergence and next beta
    {
      struct V {
        double x, p, r, q;
      };
      G.template vector<2>(
          A.n, active, [&](int c) { return s.alpha[c]; }, [&](int i) { return A.invA[i]; },
          [&](int c, int i) {
            const int64_t o = c * n + i;
            return V{A.x[o], A.pk[o], A.r[o], A.v[o]};
          },
          [&](int c, int i, double dinv, const V &v, double al, double (&part)[2]) {
            const int64_t o = c * n + i;
            A.x[o] = v.x + al * v.p;
            const double ri = v.r - al * v.q;
            A.r[o] = ri;
            const double zi = dinv * ri;
            part[0] = ri * ri;
            part[1] = ri * zi;
          });
    }
    double t[6];
    if (!G.template reduce<6>(t)) return;
    active = each_component<3>(active, &s.active, [&](int c) {
      const double rr = pick<3>(t, c), rz = pick<3>(t, c, 3), crit = A.cw ? rz : rr;
      s.iters[c] += 1;
      s.rnorm2[c] = crit;
      if (isnan(rr) || isnan(rz)) {
        s.status[c] = KS_BREAKDOWN;
        return false;
      }
      if (crit <= s.tol2[c]) {
        s.status[c] = KS_CONVERGED;
        return false;
      }
      if (s.iters[c] >= s.maxit) {
        s.status[c] = KS_MAXIT;
        return false;
      }
      s.beta[c] = rz / s.rho[c];
      s.rho[c] = rz;
      return true;
    });
    if (!active) break;
    // p = z + beta p
    {
      struct V {
        double r, p;
      };
      G.template vector<0>(
          A.n, active, [&](int c) { return s.beta[c]; }, [&](int i) { return A.invA[i]; },
          [&](int c, int i) { return V{A.r[c * n + i], A.pk[c * n + i]}; },
          [&](int c, int i, double dinv, const V &v, double be, double (&)[1]) {
            A.pk[c * n + i] = dinv * v.r + be * v.p;
          });
    }
    if (!G.sync()) return;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *A.bs = s;
}

// ------------------------------------------------------------------------------------------
// Scalar steps of BiCGSTAB, shared by the batched momentum solve and the pressure solve.
__device__ __forceinline__ bool bicg_after_v(BicgState &s, int c, double r0v) {
  if (r0v == 0.0) {
    s.status[c] = KS_BREAKDOWN;
    return false;
  }
  s.alpha[c] = s.rho[c] / r0v;
  return true;
}
__device__ __forceinline__ bool bicg_after_t(BicgState &s, int c, double tt, double ts) {
  s.omega[c] = (tt > 0.0) ? ts / tt : 0.0;
  return true;
}
__device__ __forceinline__ bool bicg_after_xr(BicgState &s, int c, double rr, double rho_new) {
  const double eps = 2.220446049250313e-16;
  s.iters[c] += 1;
  s.rnorm2[c] = rr;
  if (isnan(rr) || isnan(rho_new)) {
    s.status[c] = KS_BREAKDOWN;
    return false;
  }
  if (rr <= s.tol2[c]) {
    s.status[c] = KS_CONVERGED;
    return false;
  }
  if (s.iters[c] >= s.maxit) {
    s.status[c] = KS_MAXIT;
    return false;
  }
  if (s.omega[c] == 0.0) {
    s.status[c] = KS_BREAKDOWN;
    return false;
  }
  if (fabs(rho_new) < eps * eps * s.r0norm2[c]) {
    atomicOr(&s.restart, 1 << c);
  } else {
    s.beta[c] = (rho_new / s.rho[c]) * (s.alpha[c] / s.omega[c]);
    s.rho[c] = rho_new;
  }
  return true;
}

// Restart of component c at row i: r = b - A x, r0 = p = r; returns |r_i|^2.
__device__ __forceinline__ double bicg_restart_row(const BicgArgs &A, double *p, int c, int r, int i) {
  const int64_t n = A.n;
  const int base = A.S.sptr[r >> 5] + (r & 31), len = A.S.len[r];
  double acc = 0.0;
  for (int k = 0; k < len; ++k) {
    const int pos = base + k * kSellC;
    const int j = A.S.col[pos];
    acc += A.At[pos] * (A.diagA[j] * A.x[c * n + j]);
  }
  const int64_t o = c * n + i;
  const double ri = A.b[o] - acc;
  A.r[o] = ri;
  A.r0[o] = ri;
  p[o] = ri;
  return ri * ri;
}

// Batched right-preconditioned momentum BiCGSTAB on At = A D^-1 (the reference's method).
template <int T, int U>
__global__ void __launch_bounds__(T, 1) k_bicg_solve3(BicgArgs A, ResidentArgs R) {
  extern __shared__ double s_slots[];
  __shared__ BicgState s;
  if (A.st && A.st->halt) return;
  if (threadIdx.x == 0) s = *A.bs;
  if (blockIdx.x == 0 && threadIdx.x == 0 && A.st) A.st->body_runs[A.slot] += 1;
  __syncthreads();
  Resident<T> G(R, s_slots);
  const int64_t n = A.n;
  int active = s.active;
  while (active) {
    const int restart = s.restart & active;
    // p = r + beta (p - omega v)
    {
      struct V {
        double r, p, v;
      };
      G.template vector<0>(
          A.n, active & ~restart, [&](int c) { return make_double2(s.beta[c], s.omega[c]); },
          [](int) { return 0; },
          [&](int c, int i) {
            const int64_t o = c * n + i;
            return V{A.r[o], A.pk[o], A.v[o]};
          },
          [&](int c, int i, int, const V &x, double2 k, double (&)[1]) {  // k: beta, omega
            A.pk[c * n + i] = x.r + k.x * (x.p - k.y * x.v);
          });
    }
    if (restart) {
      G.template rows<3>(A.S, [&](int r, int i, double (&part)[3]) {
#pragma unroll
        for (int c = 0; c < 3; ++c)
          if ((restart >> c) & 1) part[c] = bicg_restart_row(A, A.pk, c, r, i);
      });
      double t[3];
      if (!G.template reduce<3>(t)) return;
      each_component<3>(active, &s.active, [&](int c) {
        if ((restart >> c) & 1) s.rho[c] = s.r0norm2[c] = pick<3>(t, c);
        return true;
      });
      if (threadIdx.x == 0) s.restart = 0;
      __syncthreads();
    } else if (!G.sync()) {
      return;
    }
    // v = At p, alpha = rho / (r0 . v)
    with_mask<3>(active, [&](auto mk) {
      constexpr int MASK = decltype(mk)::value;
      G.template products<3, 3, U, MASK>(A.S, A.At, double(), [&](int c, int j) { return A.pk[c * n + j]; },
                                         [&](int c, int i) { return A.r0[c * n + i]; },
                                         [&](int i, const double *acc, const double *own, double (&part)[3]) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          if (!((MASK >> c) & 1)) continue;
          A.v[c * n + i] = acc[c];
          part[c] = own[c] * acc[c];
        }
      });
    });
    {
      double t[3];
      if (!G.template reduce<3>(t)) return;
      active = each_component<3>(active, &s.active, [&](int c) { return bicg_after_v(s, c, pick<3>(t, c)); });
    }
    if (!active) break;
    // s = r - alpha v
    {
      struct V {
        double r, v;
      };
      G.template vector<0>(
          A.n, active, [&](int c) { return s.alpha[c]; }, [](int) { return 0; },
          [&](int c, int i) { return V{A.r[c * n + i], A.v[c * n + i]}; },
          [&](int c, int i, int, const V &x, double al, double (&)[1]) { A.s[c * n + i] = x.r - al * x.v; });
    }
    if (!G.sync()) return;
    // t = At s, omega = (t . s) / (t . t)
    with_mask<3>(active, [&](auto mk) {
      constexpr int MASK = decltype(mk)::value;
      const auto sv = [&](int c, int j) { return A.s[c * n + j]; };
      G.template products<6, 3, U, MASK>(A.S, A.At, double(), sv, sv,
                                         [&](int i, const double *acc, const double *own, double (&part)[6]) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          if (!((MASK >> c) & 1)) continue;
          A.t[c * n + i] = acc[c];
          part[c] = acc[c] * acc[c];
          part[3 + c] = acc[c] * own[c];
        }
      });
    });
    {
      double t[6];
      if (!G.template reduce<6>(t)) return;
      each_component<3>(active, &s.active, [&](int c) { return bicg_after_t(s, c, pick<3>(t, c), pick<3>(t, c, 3)); });
    }
    // x += alpha D^-1 p + omega D^-1 s, r = s - omega t; convergence test and next beta
    {
      struct V {
        double p, s, t, x, r0;
      };
      G.template vector<2>(
          A.n, active, [&](int c) { return make_double2(s.alpha[c], s.omega[c]); },
          [&](int i) { return make_double2(A.invA[i], A.cw ? A.cw[i] : 1.0); },
          [&](int c, int i) {
            const int64_t o = c * n + i;
            return V{A.pk[o], A.s[o], A.t[o], A.x[o], A.r0[o]};
          },
          [&](int c, int i, double2 d, const V &v, double2 k, double (&part)[2]) {  // k: alpha, omega
            const int64_t o = c * n + i;
            const double y = d.x * v.p;
            const double z = d.x * v.s;
            A.x[o] = v.x + (k.x * y + k.y * z);
            const double ri = v.s - k.y * v.t;
            A.r[o] = ri;
            part[0] = (ri * ri) * d.y;
            part[1] = v.r0 * ri;
          });
    }
    double t[6];
    if (!G.template reduce<6>(t)) return;
    active = each_component<3>(active, &s.active, [&](int c) { return bicg_after_xr(s, c, pick<3>(t, c), pick<3>(t, c, 3)); });
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *A.bs = s;
}

// Pressure BiCGSTAB, one right-hand side, on the rows and windows of the resident CG kernels. The
// operator and the vectors are L2-resident and an SM owns only a few rows per thread, so a barrier costs
// more than reading a vector twice: p and s are not stored before the products but formed from r, p, v
// (r, v) where a product reads them, with the owner's expression, which leaves three barriers per
// iteration. p and v are double-buffered, since neighbours still read the old ones while a row writes
// its new ones; the block partials alternate between two buffers.
struct PBicgArgs {
  BicgArgs B;
  CgResidentArgs R;
  double *p2, *v2;  // second buffers of p and v
};

// Without windows p and s are stored once per row before the products (one more barrier each) instead of
// being evaluated per entry from three and two vectors: 158 -> 97 us per iteration on a 4M-tet bifurcation.
template <bool WIN>
__global__ void __launch_bounds__(kCgResThreads<WIN>, 1) k_bicg_resident(PBicgArgs P) {
  extern __shared__ double s_dbl[];
  __shared__ double s_grp[kCgResGroups<WIN>][2][kBlock / 32];
  __shared__ double s_tree[2][kBlock / 32];
  __shared__ BicgState s;
  const BicgArgs &A = P.B;
  const CgPersistentArgs &C = P.R.P;
  if (A.st && A.st->halt) return;
  if (threadIdx.x == 0) s = *A.bs;
  if (blockIdx.x == 0 && threadIdx.x == 0 && A.st) A.st->body_runs[A.slot] += 1;
  __syncthreads();
  if (!s.active) return;
  unsigned int phase = 0, nred = 0;
  const int g = threadIdx.x / kBlock, lt = threadIdx.x & (kBlock - 1);
  ResidentRows<double, WIN> rows(P.R, A.At, reinterpret_cast<char *>(s_dbl));
  const int c0 = min(C.nblk_nat, (int)blockIdx.x * P.R.bpc_nat), c1 = min(C.nblk_nat, c0 + P.R.bpc_nat);
  int active = s.active, cur = 0;
  while (active) {
    const double *po = cur ? P.p2 : A.pk, *vo = cur ? P.v2 : A.v;
    double *pn = cur ? A.pk : P.p2, *vn = cur ? A.v : P.v2;
    const bool restart = s.restart != 0;
    if (restart) {
      double *part = (nred++ & 1) ? C.part_b : C.part_a;
      for (int b = rows.b0 + g; b < rows.b1; b += kCgResGroups<WIN>) {
        const int lp = (b - rows.b0) * kBlock + lt, i = rows.row_of(lp);
        double v[1] = {0.0};
        if (i >= 0) v[0] = bicg_restart_row(A, pn, 0, rows.b0 * kBlock + lp, i);
        group_partial<1>(v, part, b, g, s_grp);
      }
      if (!grid_sync(C.bar, phase)) return;
      double t[1];
      tree_total_cta<1, WIN>(part, C.nblk_sell, t, s_tree);
      if (threadIdx.x == 0) {
        s.rho[0] = s.r0norm2[0] = t[0];
        s.restart = 0;
      }
      __syncthreads();
    }
    // p = r + beta (p - omega v), v = At p, alpha = rho / (r0 . v)
    const double be = s.beta[0], om0 = s.omega[0];
    {
      double *part = (nred++ & 1) ? C.part_b : C.part_a;
      const auto pnew = [&](int j) { return A.r[j] + be * (po[j] - om0 * vo[j]); };
      if (!WIN && !restart) {
        for (int i = c0 * kBlock + (int)threadIdx.x; i < min(A.n, c1 * kBlock); i += kCgResThreads<WIN>) pn[i] = pnew(i);
        if (!grid_sync(C.bar, phase)) return;
      }
      const auto pj = [&](int j) { return (!WIN || restart) ? pn[j] : pnew(j); };
      rows.fill(pj);
      for (int b = rows.b0 + g; b < rows.b1; b += kCgResGroups<WIN>) {
        const int lp = (b - rows.b0) * kBlock + lt, i = rows.row_of(lp);
        double v[1] = {0.0};
        if (i >= 0) {
          const double acc = rows.product(b, lp, pj);
          if (WIN && !restart) pn[i] = pj(i);
          vn[i] = acc;
          v[0] = A.r0[i] * acc;
        }
        group_partial<1>(v, part, b, g, s_grp);
      }
      if (!grid_sync(C.bar, phase)) return;
      double t[1];
      tree_total_cta<1, WIN>(part, C.nblk_sell, t, s_tree);
      active = each_component<1>(active, &s.active, [&](int) { return bicg_after_v(s, 0, t[0]); });
    }
    if (!active) break;
    // s = r - alpha v, t = At s, omega = (t . s) / (t . t)
    const double al = s.alpha[0];
    {
      double *part = (nred++ & 1) ? C.part_b : C.part_a;
      const auto snew = [&](int j) { return A.r[j] - al * vn[j]; };
      if (!WIN) {
        for (int i = c0 * kBlock + (int)threadIdx.x; i < min(A.n, c1 * kBlock); i += kCgResThreads<WIN>) A.s[i] = snew(i);
        if (!grid_sync(C.bar, phase)) return;
      }
      const auto sj = [&](int j) { return WIN ? snew(j) : A.s[j]; };
      rows.fill(sj);
      for (int b = rows.b0 + g; b < rows.b1; b += kCgResGroups<WIN>) {
        const int lp = (b - rows.b0) * kBlock + lt, i = rows.row_of(lp);
        double v[2] = {0.0, 0.0};
        if (i >= 0) {
          const double acc = rows.product(b, lp, sj);
          A.t[i] = acc;
          v[0] = acc * acc;
          v[1] = acc * sj(i);
        }
        group_partial<2>(v, part, b, g, s_grp);
      }
      if (!grid_sync(C.bar, phase)) return;
      double t[2];
      tree_total_cta<2, WIN>(part, C.nblk_sell, t, s_tree);
      each_component<1>(active, &s.active, [&](int) { return bicg_after_t(s, 0, t[0], t[1]); });
    }
    // x += alpha D^-1 p + omega D^-1 s, r = s - omega t; convergence test and next beta
    const double om = s.omega[0];
    double *part = (nred++ & 1) ? C.part_b : C.part_a;
    for (int b = c0 + g; b < c1; b += kCgResGroups<WIN>) {
      const int i = b * kBlock + lt;
      double v[2] = {0.0, 0.0};
      if (i < A.n) {
        const double dinv = A.invA[i];
        const double w = A.cw ? A.cw[i] : 1.0;
        const double si = A.r[i] - al * vn[i];
        const double y = dinv * pn[i];
        const double z = dinv * si;
        A.x[i] = A.x[i] + (al * y + om * z);
        const double ri = si - om * A.t[i];
        A.r[i] = ri;
        v[0] = (ri * ri) * w;
        v[1] = A.r0[i] * ri;
      }
      group_partial<2>(v, part, b, g, s_grp);
    }
    if (!grid_sync(C.bar, phase)) return;
    double t[2];
    tree_total_cta<2, WIN>(part, C.nblk_nat, t, s_tree);
    active = each_component<1>(active, &s.active, [&](int) { return bicg_after_xr(s, 0, t[0], t[1]); });
    cur ^= 1;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *A.bs = s;
}

// ------------------------------------------------------------------------------------------
// FP32 CG with FP64 reliable updates (scheme: k_mpc_init's comment).
template <int T, int U, int UF>
__global__ void __launch_bounds__(T, 1) k_mpc_solve(MixedArgs A, ResidentArgs R) {
  extern __shared__ double s_slots[];
  __shared__ MixedState s;
  if (A.st && A.st->halt) return;
  if (threadIdx.x == 0) s = *A.ms;
  if (blockIdx.x == 0 && threadIdx.x == 0 && A.st) A.st->body_runs[0] += 1;
  __syncthreads();
  Resident<T> G(R, s_slots);
  const int64_t n = A.n;
  int active = s.active;
  while (active) {
    // q = A32 p, alpha = rho / (p . q)
    with_mask<3>(active, [&](auto mk) {
      constexpr int MASK = decltype(mk)::value;
      const auto pv = [&](int c, int j) { return A.p[c * n + j]; };
      G.template products<3, 3, UF, MASK>(A.S, A.At32, float(), pv, pv,
                                             [&](int i, const float *acc, const float *own, double (&part)[3]) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          if (!((MASK >> c) & 1)) continue;
          A.v[c * n + i] = acc[c];
          part[c] = (double)own[c] * (double)acc[c];
        }
      });
    });
    {
      double t[3];
      if (!G.template reduce<3>(t)) return;
      active = each_component<3>(active, &s.active, [&](int c) {
        const double pq = pick<3>(t, c);
        if (isnan(pq) || pq == 0.0) {
          s.status[c] = KS_BREAKDOWN;
          return false;
        }
        s.alpha[c] = s.rho[c] / pq;
        return true;
      });
    }
    if (!active) break;
    // dx += alpha p, r -= alpha q, z = D^-1 r; the iterated residual and r.z; which components take
    // a reliable update, next beta for the others
    {
      struct V {
        float p, q, r, dx;
      };
      G.template vector<2>(
          A.n, active, [&](int c) { return (float)s.alpha[c]; },
          [&](int i) { return make_float2(A.invA32[i], A.cw32 ? A.cw32[i] : 1.f); },
          [&](int c, int i) {
            const int64_t o = c * n + i;
            return V{A.p[o], A.v[o], A.r[o], A.dx[o]};
          },
          [&](int c, int i, float2 d, const V &v, float al, double (&part)[2]) {
            const int64_t o = c * n + i;
            A.dx[o] = v.dx + al * v.p;
            const float ri = v.r - al * v.q;
            A.r[o] = ri;
            const float zi = d.x * ri;
            part[0] = ((double)ri * (double)ri) * (double)d.y;
            part[1] = (double)ri * (double)zi;
          });
    }
    {
      double t[6];
      if (!G.template reduce<6>(t)) return;
      active = each_component<3>(active, &s.active, [&](int c) {
        const double rr = pick<3>(t, c), rz = pick<3>(t, c, 3);
        s.iters[c] += 1;
        s.rin2[c] = rr;
        if (isnan(rr) || isnan(rz)) {
          s.status[c] = KS_BREAKDOWN;
          return false;
        }
        if (rr <= s.tol2[c] || s.iters[c] >= s.maxit || rr < s.delta2 * s.rmax2[c]) {
          atomicOr(&s.upd, 1 << c);  // the update replaces rho and beta from the true residual
        } else {
          s.beta[c] = rz / s.rho[c];
          s.rho[c] = rz;
          s.rmax2[c] = fmax(s.rmax2[c], rr);
        }
        return true;
      });
    }
    const int upd = s.upd;
    if (upd) {
      // x += dx (FP64), dx = 0
      struct X {
        double x;
        float dx;
      };
      G.template vector<0>(
          A.n, upd, [](int) { return 0; }, [](int) { return 0; },
          [&](int c, int i) { return X{A.x[c * n + i], A.dx[c * n + i]}; },
          [&](int c, int i, int, const X &v, int, double (&)[1]) {
            const int64_t o = c * n + i;
            A.x[o] = v.x + (double)v.dx;
            A.dx[o] = 0.f;
          });
      if (!G.sync()) return;
      // r64 = b - A x (FP64 operator), r = (float) r64; convergence on the true residual
      with_mask<3>(upd, [&](auto mk) {
        constexpr int MASK = decltype(mk)::value;
        G.template products<6, 3, U, MASK>(A.S, A.At64, double(), [&](int c, int j) { return A.x[c * n + j]; },
                                           [&](int c, int i) { return A.b[c * n + i]; },
                                           [&](int i, const double *acc, const double *own, double (&part)[6]) {
          const double w = A.cw ? A.cw[i] : 1.0;
          const float dinv = A.invA32[i];
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            if (!((MASK >> c) & 1)) continue;
            const int64_t o = c * n + i;
            const double ri = own[c] - acc[c];
            const float rf = (float)ri;
            A.r[o] = rf;
            part[c] = (ri * ri) * w;
            part[3 + c] = (double)rf * (double)(dinv * rf);
          }
        });
      });
      double t[6];
      if (!G.template reduce<6>(t)) return;
      active = each_component<3>(active, &s.active, [&](int c) {
        if (!((upd >> c) & 1)) return true;
        const double rr = pick<3>(t, c), rz = pick<3>(t, c, 3);
        s.updates[c] += 1;
        const double prev2 = s.rnorm2[c];  // true residual at the previous update
        s.rnorm2[c] = rr;
        if (isnan(rr) || isnan(rz)) {
          s.status[c] = KS_BREAKDOWN;
          return false;
        }
        if (rr <= s.tol2[c]) {
          s.status[c] = KS_CONVERGED;
          return false;
        }
        if (s.iters[c] >= s.maxit) {
          s.status[c] = KS_MAXIT;
          return false;
        }
        // the FP32 recurrence drifted from the true residual, or convergence turned erratic: restart
        // the direction from the replaced residual
        const bool restart = rr > kMixedDrift2 * s.rin2[c] || rr > prev2;
        s.beta[c] = restart ? 0.0 : rz / s.rho[c];
        if (restart) s.restarts[c] += 1;
        s.rho[c] = rz;
        s.rin2[c] = rr;
        s.rmax2[c] = rr;
        return true;
      });
      if (threadIdx.x == 0) s.upd = 0;
    }
    if (!active) break;
    // p = z + beta p with z = D^-1 r
    {
      struct V {
        float r, p;
      };
      G.template vector<0>(
          A.n, active, [&](int c) { return (float)s.beta[c]; }, [&](int i) { return A.invA32[i]; },
          [&](int c, int i) { return V{A.r[c * n + i], A.p[c * n + i]}; },
          [&](int c, int i, float dinv, const V &v, float be, double (&)[1]) {
            A.p[c * n + i] = dinv * v.r + be * v.p;
          });
    }
    if (!G.sync()) return;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *A.ms = s;
}

// FP32 BiCGSTAB with FP64 reliable updates (scheme: top of ns_mixed.cuh). Components update on their
// own triggers only: replacing a residual before it has dropped by delta perturbs BiCGSTAB's
// recurrences, and on the 4M-tet Y-bifurcation updates brought forward to share one FP64 product made
// the iteration erratic until it hit the cap.
template <int T, int U, int UF>
__global__ void __launch_bounds__(T, 1) k_mp_solve(MixedArgs A, ResidentArgs R) {
  extern __shared__ double s_slots[];
  __shared__ MixedState s;
  if (A.st && A.st->halt) return;
  if (threadIdx.x == 0) s = *A.ms;
  if (blockIdx.x == 0 && threadIdx.x == 0 && A.st) A.st->body_runs[0] += 1;
  __syncthreads();
  Resident<T> G(R, s_slots);
  const int64_t n = A.n;
  int active = s.active;
  while (active) {
    // p = r + beta (p - omega v); components whose FP32 recurrence drifted restart here instead:
    // r0 = p = r and rho = r0 . r
    const int rs = s.restart_next & active;
    {
      struct V {
        float r, p, v;
      };
      const auto load = [&](int c, int i) {
        const int64_t o = c * n + i;
        return V{A.r[o], A.p[o], A.v[o]};
      };
      const auto scalar = [&](int c) { return make_float2((float)s.beta[c], (float)s.omega[c]); };
      const auto none = [](int) { return 0; };
      if (rs) {
        G.template vector<1>(A.n, active, scalar, none, load, [&](int c, int i, int, const V &x, float2 k, double (&part)[1]) {
          const int64_t o = c * n + i;
          if ((rs >> c) & 1) {
            A.p[o] = x.r;
            A.r0[o] = x.r;
            part[0] = (double)x.r * (double)x.r;
          } else {
            A.p[o] = x.r + k.x * (x.p - k.y * x.v);
          }
        });
        double t[3];
        if (!G.template reduce<3>(t)) return;
        each_component<3>(active, &s.active, [&](int c) {
          if ((rs >> c) & 1) {
            s.rho[c] = s.r0norm2[c] = pick<3>(t, c);
            s.restarts[c] += 1;
          }
          return true;
        });
        if (threadIdx.x == 0) s.restart_next = 0;
      } else {
        G.template vector<0>(A.n, active, scalar, none, load, [&](int c, int i, int, const V &x, float2 k, double (&)[1]) {
          A.p[c * n + i] = x.r + k.x * (x.p - k.y * x.v);
        });
        if (!G.sync()) return;
      }
    }
    // v = At32 p, alpha = rho / (r0 . v)
    with_mask<3>(active, [&](auto mk) {
      constexpr int MASK = decltype(mk)::value;
      G.template products<3, 3, UF, MASK>(A.S, A.At32, float(), [&](int c, int j) { return A.p[c * n + j]; },
                                             [&](int c, int i) { return A.r0[c * n + i]; },
                                             [&](int i, const float *acc, const float *own, double (&part)[3]) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          if (!((MASK >> c) & 1)) continue;
          A.v[c * n + i] = acc[c];
          part[c] = (double)own[c] * (double)acc[c];
        }
      });
    });
    {
      double t[3];
      if (!G.template reduce<3>(t)) return;
      active = each_component<3>(active, &s.active, [&](int c) {
        const double d = pick<3>(t, c);
        if (isnan(d)) {
          s.status[c] = KS_BREAKDOWN;
          return false;
        }
        if (d == 0.0) {  // no step along p; the iteration ends in an update and a restart
          s.alpha[c] = 0.0;
          atomicOr(&s.force, 1 << c);
        } else {
          s.alpha[c] = s.rho[c] / d;
        }
        return true;
      });
    }
    if (!active) break;
    // s = r - alpha v
    {
      struct V {
        float r, v;
      };
      G.template vector<0>(
          A.n, active, [&](int c) { return (float)s.alpha[c]; }, [](int) { return 0; },
          [&](int c, int i) { return V{A.r[c * n + i], A.v[c * n + i]}; },
          [&](int c, int i, int, const V &x, float al, double (&)[1]) { A.s[c * n + i] = x.r - al * x.v; });
    }
    if (!G.sync()) return;
    // t = At32 s, omega = (t . s) / (t . t)
    with_mask<3>(active, [&](auto mk) {
      constexpr int MASK = decltype(mk)::value;
      const auto sv = [&](int c, int j) { return A.s[c * n + j]; };
      G.template products<6, 3, UF, MASK>(A.S, A.At32, float(), sv, sv,
                                             [&](int i, const float *acc, const float *own, double (&part)[6]) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          if (!((MASK >> c) & 1)) continue;
          A.t[c * n + i] = acc[c];
          part[c] = (double)acc[c] * (double)acc[c];
          part[3 + c] = (double)acc[c] * (double)own[c];
        }
      });
    });
    {
      double t[6];
      if (!G.template reduce<6>(t)) return;
      each_component<3>(active, &s.active, [&](int c) {
        const double tt = pick<3>(t, c);
        s.omega[c] = (tt > 0.0) ? pick<3>(t, c, 3) / tt : 0.0;
        return true;
      });
    }
    // dx += alpha D^-1 p + omega D^-1 s, r = s - omega t; ||r||, r0 . r; which components take a
    // reliable update, next beta for the others
    {
      struct V {
        float p, s, t, dx, r0;
      };
      G.template vector<2>(
          A.n, active, [&](int c) { return make_float2((float)s.alpha[c], (float)s.omega[c]); },
          [&](int i) { return make_float2(A.invA32[i], A.cw32 ? A.cw32[i] : 1.f); },
          [&](int c, int i) {
            const int64_t o = c * n + i;
            return V{A.p[o], A.s[o], A.t[o], A.dx[o], A.r0[o]};
          },
          [&](int c, int i, float2 d, const V &v, float2 k, double (&part)[2]) {  // k: alpha, omega
            const int64_t o = c * n + i;
            A.dx[o] = v.dx + (k.x * (d.x * v.p) + k.y * (d.x * v.s));
            const float ri = v.s - k.y * v.t;
            A.r[o] = ri;
            part[0] = ((double)ri * (double)ri) * (double)d.y;
            part[1] = (double)v.r0 * (double)ri;
          });
    }
    {
      double t[6];
      if (!G.template reduce<6>(t)) return;
      active = each_component<3>(active, &s.active, [&](int c) {
        const double eps = 2.220446049250313e-16;
        const double rr = pick<3>(t, c), rho_new = pick<3>(t, c, 3);
        s.iters[c] += 1;
        s.rin2[c] = rr;
        if (isnan(rr) || isnan(rho_new)) {
          s.status[c] = KS_BREAKDOWN;
          return false;
        }
        // near-breakdown, a vanished omega or r0 . v: the FP32 space is exhausted; the update
        // replaces the residual and the Krylov space restarts from it
        const bool restart =
            fabs(rho_new) < eps * eps * s.r0norm2[c] || s.omega[c] == 0.0 || ((s.force >> c) & 1);
        if (rr <= s.tol2[c] || s.iters[c] >= s.maxit || rr < s.delta2 * s.rmax2[c] || restart) {
          atomicOr(&s.upd, 1 << c);
          if (restart) atomicOr(&s.restart, 1 << c);
        } else {
          s.beta[c] = (rho_new / s.rho[c]) * (s.alpha[c] / s.omega[c]);
          s.rho[c] = rho_new;
          s.rmax2[c] = fmax(s.rmax2[c], rr);
        }
        return true;
      });
    }
    const int upd = s.upd, rst = s.restart;
    if (upd) {
      // x += dx (FP64), dx = 0, xs = diag(A) x
      struct X {
        double x;
        float dx;
      };
      G.template vector<0>(
          A.n, upd, [](int) { return 0; }, [&](int i) { return A.diagA[i]; },
          [&](int c, int i) { return X{A.x[c * n + i], A.dx[c * n + i]}; },
          [&](int c, int i, double d, const X &v, int, double (&)[1]) {
            const int64_t o = c * n + i;
            const double xi = v.x + (double)v.dx;
            A.x[o] = xi;
            A.dx[o] = 0.f;
            A.xs[o] = d * xi;
          });
      if (!G.sync()) return;
      // r64 = b - At64 (D x), r = (float) r64 (and r0 = r for a restart); convergence on the true
      // residual, next beta from the replaced one
      with_mask<3>(upd, [&](auto mk) {
        constexpr int MASK = decltype(mk)::value;
        G.template products<6, 3, U, MASK>(A.S, A.At64, double(), [&](int c, int j) { return A.xs[c * n + j]; },
                                           [&](int c, int i) { return A.b[c * n + i]; },
                                           [&](int i, const double *acc, const double *own, double (&part)[6]) {
          const double w = A.cw ? A.cw[i] : 1.0;
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            if (!((MASK >> c) & 1)) continue;
            const int64_t o = c * n + i;
            const double ri = own[c] - acc[c];
            const float rf = (float)ri;
            A.r[o] = rf;
            float r0 = A.r0[o];
            if ((rst >> c) & 1) {
              r0 = rf;
              A.r0[o] = rf;
            }
            part[c] = (ri * ri) * w;
            part[3 + c] = (double)r0 * (double)rf;
          }
        });
      });
      double t[6];
      if (!G.template reduce<6>(t)) return;
      active = each_component<3>(active, &s.active, [&](int c) {
        if (!((upd >> c) & 1)) return true;
        const double rr = pick<3>(t, c), rho_new = pick<3>(t, c, 3);
        s.updates[c] += 1;
        const double prev2 = s.rnorm2[c];  // true residual at the previous update
        s.rnorm2[c] = rr;
        if (isnan(rr) || isnan(rho_new)) {
          s.status[c] = KS_BREAKDOWN;
          return false;
        }
        if (rr <= s.tol2[c]) {
          s.status[c] = KS_CONVERGED;
          return false;
        }
        if (s.iters[c] >= s.maxit) {
          s.status[c] = KS_MAXIT;
          return false;
        }
        if ((rst >> c) & 1) {
          s.r0norm2[c] = rho_new;
          s.beta[c] = 0.0;
        } else {
          s.beta[c] = (rho_new / s.rho[c]) * (s.alpha[c] / s.omega[c]);
          // the true residual is more than 10x (in norm) the FP32 recurrence's (its Krylov space has
          // drifted), or it grew since the previous update (erratic convergence): the next iteration
          // restarts the space from the replaced residual
          if (rr > kMixedDrift2 * s.rin2[c] || rr > prev2) atomicOr(&s.restart_next, 1 << c);
        }
        s.rho[c] = rho_new;
        s.rin2[c] = rr;
        s.rmax2[c] = rr;
        return true;
      });
    }
    if (threadIdx.x == 0) s.upd = s.restart = s.force = 0;
    __syncthreads();
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *A.ms = s;
}

// The product phase alone, `iters` times in one launch on unchanging input (kernel timing): products,
// dot partials, barrier and totals, as in the solves.
struct MomentumProductArgs {
  BicgArgs B;
  int iters;
};
struct MixedProductArgs {
  MixedArgs M;
  int iters;
};

template <int T, int U>
__global__ void __launch_bounds__(T, 1) k_momentum_product(MomentumProductArgs P, ResidentArgs R) {
  extern __shared__ double s_slots[];
  const BicgArgs &A = P.B;
  Resident<T> G(R, s_slots);
  const int64_t n = A.n;
  for (int k = 0; k < P.iters; ++k) {
    G.template products<3, 3, U, 7>(A.S, A.At, double(), [&](int c, int j) { return A.pk[c * n + j]; },
                                    [&](int c, int i) { return A.r0[c * n + i]; },
                                    [&](int i, const double *acc, const double *own, double (&part)[3]) {
#pragma unroll
      for (int c = 0; c < 3; ++c) A.v[c * n + i] = acc[c], part[c] = own[c] * acc[c];
    });
    double t[3];
    if (!G.template reduce<3>(t)) return;
    if (blockIdx.x == 0 && threadIdx.x < 3) A.bs->alpha[threadIdx.x] = pick<3>(t, threadIdx.x);
  }
}

template <int T, int U, int UF>
__global__ void __launch_bounds__(T, 1) k_mixed_product(MixedProductArgs P, ResidentArgs R) {
  extern __shared__ double s_slots[];
  const MixedArgs &A = P.M;
  Resident<T> G(R, s_slots);
  const int64_t n = A.n;
  for (int k = 0; k < P.iters; ++k) {
    G.template products<3, 3, UF, 7>(A.S, A.At32, float(), [&](int c, int j) { return A.p[c * n + j]; },
                                        [&](int c, int i) { return A.r0[c * n + i]; },
                                        [&](int i, const float *acc, const float *own, double (&part)[3]) {
#pragma unroll
      for (int c = 0; c < 3; ++c) A.v[c * n + i] = acc[c], part[c] = (double)own[c] * (double)acc[c];
    });
    double t[3];
    if (!G.template reduce<3>(t)) return;
    if (blockIdx.x == 0 && threadIdx.x < 3) A.ms->alpha[threadIdx.x] = pick<3>(t, threadIdx.x);
  }
}

}  // namespace cfsa
