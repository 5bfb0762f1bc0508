// Coarse space of the two-level pressure preconditioner (k_cg2l_resident), built on the device whenever
// the Poisson operator changes: the aggregates (boxes of a uniform grid over the vertices without a
// penalty row, numbered by first vertex), A_c = P^T L P, its inverse Z by Cholesky, and each CTA's lists.
// Every sum keeps a fixed order (rows and entries ascending, k ascending in the factorisation), so Z is
// the same to the bit as the sequential construction's, which the oracle restates.
//
// What bounds it: chains of dependent steps (432 aggregates at 1M tets: 432 columns to eliminate and to
// invert), not work (2e8 operations). The host's sequential form took 27 ms of an 86k-tet moving-mesh
// step and 0.1 s at 1M tets; here the factorisation advances 32 columns per pair of launches and the
// columns of the inverse run side by side, one CTA each.
#pragma once

#include "ns_kernels.cuh"

namespace cfsa {

struct BoxArgs {
  int n, outlet_type, ref_node;
  const double *xyz;      // [n][3]
  const signed char *bc;  // outlet vertices carry the penalty with a Dirichlet outlet
  double lo[3], h;
  unsigned long long *key;  // hash table of occupied boxes (kBoxEmpty: free), size mask + 1
  unsigned int mask;
  int *first;   // [table] lowest vertex of the box
  int *slot;    // [n] table slot of the vertex's box, -1: penalised
  int *count;   // occupied boxes
};
constexpr unsigned long long kBoxEmpty = ~0ull;

__device__ __forceinline__ bool box_penalised(const BoxArgs &A, int i) {
  return A.outlet_type == 1 ? i == A.ref_node : A.outlet_type == 0 && A.bc[i] == BC_OUTLET;
}

// Bounding box of the unpenalised vertices: per-CTA minima and maxima [gridDim][6].
__global__ void k_box_bounds(BoxArgs A, double *__restrict__ out) {
  __shared__ double sm[6][kBlock / 32];
  double v[6];
  for (int d = 0; d < 3; ++d) v[d] = 1.7976931348623157e308, v[3 + d] = -1.7976931348623157e308;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < A.n; i += gridDim.x * blockDim.x) {
    if (box_penalised(A, i)) continue;
    for (int d = 0; d < 3; ++d) {
      const double x = A.xyz[3 * (int64_t)i + d];
      v[d] = fmin(v[d], x);
      v[3 + d] = fmax(v[3 + d], x);
    }
  }
  for (int d = 0; d < 6; ++d) {
    for (int o = 16; o > 0; o >>= 1) {
      const double w = __shfl_xor_sync(0xffffffffu, v[d], o);
      v[d] = d < 3 ? fmin(v[d], w) : fmax(v[d], w);
    }
    if ((threadIdx.x & 31) == 0) sm[d][threadIdx.x >> 5] = v[d];
  }
  __syncthreads();
  if (threadIdx.x < 6) {
    double r = sm[threadIdx.x][0];
    for (int w = 1; w < kBlock / 32; ++w) r = threadIdx.x < 3 ? fmin(r, sm[threadIdx.x][w]) : fmax(r, sm[threadIdx.x][w]);
    out[6 * blockIdx.x + threadIdx.x] = r;
  }
}

// Enters every unpenalised vertex's box into the table; counts the boxes. The table holds more slots than
// there are vertices, so a probe always ends at the box or at a free slot.
__global__ void k_box_insert(BoxArgs A) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= A.n) return;
  if (box_penalised(A, i)) {
    A.slot[i] = -1;
    return;
  }
  long long q[3];
  for (int d = 0; d < 3; ++d) q[d] = (long long)floor((A.xyz[3 * (int64_t)i + d] - A.lo[d]) / A.h);
  const unsigned long long key = (unsigned long long)((q[0] * 2097152 + q[1]) * 2097152 + q[2]);
  unsigned int s = (unsigned int)((key * 0x9E3779B97F4A7C15ull) >> 32) & A.mask;
  for (unsigned int probe = 0; probe <= A.mask; ++probe, s = (s + 1) & A.mask) {
    const unsigned long long old = atomicCAS(A.key + s, kBoxEmpty, key);
    if (old == kBoxEmpty) atomicAdd(A.count, 1);
    if (old == kBoxEmpty || old == key) break;
  }
  A.slot[i] = (int)s;
  atomicMin(A.first + s, i);
}

// The first vertices of the boxes, in no particular order ...
__global__ void k_box_collect(int n, const int *__restrict__ slot, const int *__restrict__ first, int *count,
                              int *__restrict__ list) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && slot[i] >= 0 && first[slot[i]] == i) list[atomicAdd(count, 1)] = i;
}
// ... their ranks number the boxes ...
__global__ void k_box_number(int nc, const int *__restrict__ list, const int *__restrict__ slot, int *__restrict__ id) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nc) return;
  const int f = list[i];
  int r = 0;
  for (int j = 0; j < nc; ++j) r += list[j] < f;
  id[slot[f]] = r;
}
// ... and every vertex takes its box's number (nc: no aggregate).
__global__ void k_box_assign(int n, int nc, const int *__restrict__ slot, const int *__restrict__ id,
                             int *__restrict__ agg, int *count) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int a = slot[i] < 0 ? nc : id[slot[i]];
  agg[i] = a;
  if (a < nc) atomicAdd(count + a, 1);
}
// Exclusive prefix sums of count[0..n) into ptr[0..n] (one warp).
__global__ void k_prefix(int n, const int *__restrict__ count, int *__restrict__ ptr) {
  int total = 0;
  for (int k0 = 0; k0 < n; k0 += 32) {
    const int k = k0 + (int)threadIdx.x, v = (k < n) ? count[k] : 0;
    int s = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, s, o);
      if ((int)threadIdx.x >= o) s += u;
    }
    if (k < n) ptr[k] = total + s - v;
    total += __shfl_sync(0xffffffffu, s, 31);
  }
  if (threadIdx.x == 0) ptr[n] = total;
}
// The rows of each aggregate in ascending order: one CTA per aggregate scans all rows.
__global__ void k_agg_rows(int n, const int *__restrict__ agg, const int *__restrict__ ptr, int *__restrict__ rows) {
  __shared__ int s_cnt[kBlock / 32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int at = ptr[blockIdx.x];
  for (int i0 = 0; i0 < n; i0 += kBlock) {
    const int i = i0 + (int)threadIdx.x;
    const bool mine = i < n && agg[i] == (int)blockIdx.x;
    const unsigned int m = __ballot_sync(0xffffffffu, mine);
    if (lane == 0) s_cnt[warp] = __popc(m);
    __syncthreads();
    int before = 0, all = 0;
    for (int w = 0; w < kBlock / 32; ++w) {
      if (w < warp) before += s_cnt[w];
      all += s_cnt[w];
    }
    if (mine) rows[at + before + __popc(m & ((1u << lane) - 1u))] = i;
    at += all;
    __syncthreads();
  }
}

// Row a of A_c = P^T L P (one CTA per aggregate a): entry b adds the entries of a's rows whose column lies
// in b, rows ascending and columns ascending within a row. Tiles of up to kTileRows rows are staged in
// shared memory; thread b walks the staged entries in order.
constexpr int kTileRows = 64, kTileEntries = 2048;
__global__ void k_coarse_matrix(int nc, const int *__restrict__ ptr, const int *__restrict__ rows,
                                const int *__restrict__ rp, const int *__restrict__ ci, const double *__restrict__ L,
                                const int *__restrict__ agg, double *__restrict__ Ac) {
  __shared__ double s_v[kTileEntries];
  __shared__ int s_a[kTileEntries], s_off[kTileRows + 1], s_n;
  const int r0 = ptr[blockIdx.x], r1 = ptr[blockIdx.x + 1];
  for (int b0 = 0; b0 < nc; b0 += blockDim.x) {
    const int b = b0 + (int)threadIdx.x;
    double acc = 0.0;
    for (int r = r0; r < r1;) {
      __syncthreads();
      if (threadIdx.x < kTileRows) {
        const int q = r + (int)threadIdx.x;
        s_off[threadIdx.x + 1] = (q < r1) ? rp[rows[q] + 1] - rp[rows[q]] : 0;
      }
      __syncthreads();
      if (threadIdx.x == 0) {  // as many rows as the tile holds (a row has at most kPatternCap entries)
        s_off[0] = 0;
        int k = 0;
        for (; k < kTileRows && r + k < r1 && s_off[k] + s_off[k + 1] <= kTileEntries; ++k) s_off[k + 1] += s_off[k];
        s_n = k;
      }
      __syncthreads();
      const int nr = s_n;
      for (int k = threadIdx.x >> 5; k < nr; k += blockDim.x >> 5) {
        const int e0 = rp[rows[r + k]], len = s_off[k + 1] - s_off[k];
        for (int e = threadIdx.x & 31; e < len; e += 32) {
          s_a[s_off[k] + e] = agg[ci[e0 + e]];
          s_v[s_off[k] + e] = L[e0 + e];
        }
      }
      __syncthreads();
      for (int e = 0; e < s_off[nr]; ++e)
        if (s_a[e] == b) acc = acc + s_v[e];
      r += nr;
    }
    if (b < nc) Ac[(size_t)blockIdx.x * nc + b] = acc;
  }
}

// Cholesky A_c = G G^T in panels of kPanel columns, G over the lower triangle of the matrix A. Element
// (i, j) subtracts G(i,k) G(j,k) for k = 0, 1, ... in order: first the columns before the panel
// (k_chol_update), then those inside it (k_chol_panel). The factored diagonal blocks go to `diag`
// ([n][kPanel]) and not back to A: the CTAs of a panel launch are not ordered, and one that starts late
// must still find the unfactored block there. Later panels read rows below the block only.
constexpr int kPanel = 32;

__global__ void k_chol_update(int n, int j0, double *__restrict__ A) {
  __shared__ double s_i[kPanel][kPanel + 1], s_j[kPanel][kPanel + 1];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 32 threads: column j0 + tx, row i0 + ty
  const int i = j0 + kPanel * blockIdx.x + ty, j = j0 + tx;
  double sum = (i < n && j <= i) ? A[(size_t)i * n + j] : 0.0;
  for (int k0 = 0; k0 < j0; k0 += kPanel) {
    s_i[ty][tx] = (i < n) ? A[(size_t)i * n + k0 + tx] : 0.0;
    s_j[ty][tx] = (j0 + ty < n) ? A[(size_t)(j0 + ty) * n + k0 + tx] : 0.0;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kPanel; ++k) sum = sum - s_i[ty][k] * s_j[tx][k];
    __syncthreads();
  }
  if (i < n && j <= i) A[(size_t)i * n + j] = sum;
}

// One warp per CTA: every CTA factors the diagonal block (lane = row), then takes its 32 rows below it
// (CTA 0 writes the factored block to `diag` instead). A pivot that is not positive clears *spd.
__global__ void k_chol_panel(int n, int j0, double *__restrict__ A, double *__restrict__ diag, int *spd) {
  __shared__ double s_g[kPanel][kPanel + 1];
  const int lane = threadIdx.x, w = min(kPanel, n - j0);
  double a[kPanel];
#pragma unroll
  for (int k = 0; k < kPanel; ++k) a[k] = (lane < w && k <= lane && k < w) ? A[(size_t)(j0 + lane) * n + j0 + k] : 0.0;
  bool ok = true;
#pragma unroll
  for (int j = 0; j < kPanel; ++j) {
    if (j >= w) break;
    const double piv = __shfl_sync(0xffffffffu, a[j], j);
    ok = ok && piv > 0.0;
    const double d = sqrt(piv), g = (lane == j) ? d : a[j] / d;
    a[j] = g;
    s_g[lane][j] = g;
    __syncwarp();
#pragma unroll
    for (int k = j + 1; k < kPanel; ++k)
      if (k < w) a[k] = a[k] - g * s_g[k][j];
  }
  __syncwarp();
  if (blockIdx.x == 0) {
    for (int k = 0; k <= lane && lane < w; ++k) diag[(size_t)(j0 + lane) * kPanel + k] = s_g[lane][k];
    if (lane == 0 && !ok) *spd = 0;
    return;
  }
  const int i = j0 + kPanel * blockIdx.x + lane;
  if (i >= n) return;
#pragma unroll
  for (int k = 0; k < kPanel; ++k) a[k] = A[(size_t)i * n + j0 + k];
#pragma unroll
  for (int j = 0; j < kPanel; ++j) {
    a[j] = a[j] / s_g[j][j];
#pragma unroll
    for (int k = j + 1; k < kPanel; ++k) a[k] = a[k] - a[j] * s_g[k][j];
  }
#pragma unroll
  for (int k = 0; k < kPanel; ++k) A[(size_t)i * n + j0 + k] = a[k];
}

// T = G transposed: the lower triangle of A with the diagonal blocks from `diag` (tiles are panels).
__global__ void k_transpose(int n, const double *__restrict__ A, const double *__restrict__ diag,
                            double *__restrict__ T) {
  static_assert(kPanel == 32, "a tile of the transposition is a panel");
  __shared__ double s[32][33];
  const int x = 32 * blockIdx.x + (threadIdx.x & 31), y0 = 32 * blockIdx.y;
  for (int r = threadIdx.x >> 5; r < 32; r += blockDim.x >> 5)
    if (x <= y0 + r && y0 + r < n)
      s[r][threadIdx.x & 31] = (blockIdx.x == blockIdx.y) ? diag[(size_t)(y0 + r) * kPanel + (threadIdx.x & 31)]
                                                          : A[(size_t)(y0 + r) * n + x];
    else
      s[r][threadIdx.x & 31] = 0.0;  // above the diagonal
  __syncthreads();
  const int tx = y0 + (int)(threadIdx.x & 31);
  for (int r = threadIdx.x >> 5; r < 32; r += blockDim.x >> 5)
    if (tx < n && 32 * (int)blockIdx.x + r < n) T[(size_t)(32 * blockIdx.x + r) * n + tx] = s[threadIdx.x & 31][r];
}

// Column j of G^-1 (one CTA per column): entry k is sum_k / G(k,k) with sum_k = 0 - G(k,j) Gi(j,j) - ...
// in ascending order; every known entry is subtracted from all later sums at once (GT = G transposed, so
// that the threads read neighbouring values, one step ahead).
__global__ void k_coarse_inverse(int n, const double *__restrict__ GT, double *__restrict__ Gi) {
  extern __shared__ double s_sum[];
  const int j = blockIdx.x;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s_sum[i] = 0.0;
  const int i0 = threadIdx.x;
  double d = GT[(size_t)j * n + j], g = (i0 > j && i0 < n) ? GT[(size_t)j * n + i0] : 0.0;
  __syncthreads();
  for (int k = j; k < n; ++k) {
    const double x = (k == j) ? 1.0 / d : s_sum[k] / d;
    if (threadIdx.x == 0) Gi[(size_t)k * n + j] = x;
    const double gk = g;
    if (k + 1 < n) {
      d = GT[(size_t)(k + 1) * n + k + 1];
      g = (i0 > k + 1 && i0 < n) ? GT[(size_t)(k + 1) * n + i0] : 0.0;
    }
    if (i0 > k && i0 < n) s_sum[i0] = s_sum[i0] - gk * x;
    for (int i = i0 + blockDim.x; i < n; i += blockDim.x)
      if (i > k) s_sum[i] = s_sum[i] - GT[(size_t)k * n + i] * x;
    __syncthreads();
  }
}

// Z = G^-T G^-1: entry (m, k) adds Gi(q,m) Gi(q,k) for q = max(m,k), ... in order.
__global__ void k_coarse_z(int n, const double *__restrict__ Gi, double *__restrict__ Z) {
  const int k = 32 * blockIdx.x + (threadIdx.x & 31), m = 8 * blockIdx.y + (threadIdx.x >> 5);
  if (k >= n || m >= n) return;
  double sum = 0.0;
#pragma unroll 8
  for (int q = max(m, k); q < n; ++q) sum = sum + Gi[(size_t)q * n + m] * Gi[(size_t)q * n + k];
  Z[(size_t)m * n + k] = sum;
}

// The lists of one CTA of the resident solve (its rows are the natural rows of its blocks): staging
// positions of the rows sorted by (aggregate, row), the pieces of the aggregates' segments, and the
// aggregates of its rows and of their columns.
struct CoarseListArgs {
  int n, nc, bpc;
  const int *rp, *ci, *agg;
  int *row_pos;
  int4 *pieces;
  int *npieces, piece_stride;
  int *need, *nneed, need_stride;
};

__global__ void k_coarse_lists(CoarseListArgs A) {
  extern __shared__ int s_int[];
  const int rows = A.bpc * kBlock, words = (A.nc + 31) / 32;
  int *s_agg = s_int, *s_cnt = s_agg + rows, *s_lo = s_cnt + A.nc;
  unsigned int *s_need = reinterpret_cast<unsigned int *>(s_lo + A.nc);
  const int r0 = (int)min((int64_t)A.n, (int64_t)rows * blockIdx.x), r1 = min(A.n, r0 + rows);
  for (int a = threadIdx.x; a < A.nc; a += blockDim.x) s_cnt[a] = 0;
  for (int w = threadIdx.x; w < words; w += blockDim.x) s_need[w] = 0u;
  __syncthreads();
  for (int i = r0 + (int)threadIdx.x; i < r1; i += blockDim.x) {
    const int a = A.agg[i];
    s_agg[i - r0] = a;
    if (a < A.nc) {
      atomicAdd(s_cnt + a, 1);
      atomicOr(s_need + (a >> 5), 1u << (a & 31));
    }
    for (int k = A.rp[i]; k < A.rp[i + 1]; ++k) {
      const int b = A.agg[A.ci[k]];
      if (b < A.nc && !(s_need[b >> 5] >> (b & 31) & 1u)) atomicOr(s_need + (b >> 5), 1u << (b & 31));
    }
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    int rows_before = 0, pieces_before = 0, need_before = 0;
    for (int a0 = 0; a0 < A.nc; a0 += 32) {
      const int a = a0 + lane, cnt = (a < A.nc) ? s_cnt[a] : 0, np = (cnt + kSegPiece - 1) / kSegPiece;
      int sr = cnt, sp = np;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, sr, o), v = __shfl_up_sync(0xffffffffu, sp, o);
        if (lane >= o) sr += u, sp += v;
      }
      const int lo = rows_before + sr - cnt;
      if (a < A.nc) s_lo[a] = lo;
      for (int p = 0; p < np; ++p)
        A.pieces[(size_t)blockIdx.x * A.piece_stride + pieces_before + sp - np + p] =
            make_int4(lo + p * kSegPiece, min(lo + cnt, lo + (p + 1) * kSegPiece), a, 0);
      const unsigned int m = s_need[a0 >> 5];
      if (m >> lane & 1u)
        A.need[(size_t)blockIdx.x * A.need_stride + need_before + __popc(m & ((1u << lane) - 1u))] = a;
      rows_before += __shfl_sync(0xffffffffu, sr, 31);
      pieces_before += __shfl_sync(0xffffffffu, sp, 31);
      need_before += __popc(m);
    }
    if (lane == 0) {
      A.npieces[blockIdx.x] = pieces_before;
      A.nneed[blockIdx.x] = need_before;
    }
  }
  __syncthreads();
  for (int i = r0 + (int)threadIdx.x; i < r1; i += blockDim.x) {
    const int a = s_agg[i - r0];
    int p = -1;
    if (a < A.nc) {
      p = s_lo[a];
      for (int q = 0; q < i - r0; ++q) p += s_agg[q] == a;
    }
    A.row_pos[i] = p;
  }
}

}  // namespace cfsa
