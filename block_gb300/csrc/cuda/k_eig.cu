// Batched dense symmetric eigensolver (FP64); see k_eig.cuh for the layout.
//
// Householder step k (0 <= k <= n-3) of A = A^(0), lower triangle:
//   x = A^(k)[k+1:n, k],  beta = -sign(x_0) |x|,  tau = (beta - x_0) / beta,
//   v = (0..0, 1, x_1.. / (x_0 - beta)),  p = tau A^(k) v,
//   w = p - (tau / 2)(p . v) v,  A^(k+1) = A^(k) - v w^T - w v^T
// (Golub & Van Loan, Matrix Computations, 4th ed., sections 5.1 and 8.3.1).
// The trailing update of step k-1 and the product A^(k) v_k of step k share
// one pass over the matrix: column k of A^(k) is formed lazily from the
// stored column (still A^(k-1)) and the rank-2 correction of step k-1.
//
// The tridiagonal eigenproblem is solved by divide and conquer (k_dc.cu);
// its leaves use the implicit QL iteration with the Wilkinson shift of the
// leading 2 x 2 block (Bowdler, Martin, Reinsch and Wilkinson, "The QR and
// QL algorithms for symmetric matrices", Numer. Math. 11 (1968) 293-306).
#include <algorithm>
#include <cmath>
#include <vector>

#include "k_eig.cuh"

namespace bgpu {
namespace dev {
namespace {

constexpr int kHouseThreads = 256;
constexpr int kUpdThreads = 256;
constexpr int kBtThreads = 32 * kEigBtCols;

__device__ __forceinline__ double warp_sum(double x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// deterministic block sum (every thread gets the result)
template <int NT>
__device__ double block_sum(double x, double* red) {
  x = warp_sum(x);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) red[warp] = x;
  __syncthreads();
  double s = 0.0;
#pragma unroll
  for (int i = 0; i < NT / 32; ++i) s += red[i];
  return s;
}

struct Scal {
  double *d, *e, *tau, *eu, *wr, *prow, *pcol;
};
__device__ __forceinline__ Scal scal(const EigBufs& b, const EigJob& J) {
  Scal s;
  s.d = b.work + J.s_off;
  s.e = s.d + J.n;
  s.tau = s.e + J.n;
  s.eu = s.tau + J.n;
  s.wr = s.eu + J.n;  // two vectors of n: slot (k & 1)
  s.prow = s.wr + 2 * (int64_t)J.n;
  s.pcol = s.prow + (int64_t)J.nt * J.n;
  return s;
}

// One CTA per job: reduces the partial products of step k-1 into w_{k-1},
// forms column k of A^(k) and the reflector of step k (or, at k = n-2, the
// last 2 x 2 block of the tridiagonal matrix).
__global__ void __launch_bounds__(kHouseThreads) eig_house(EigBufs b, const EigJob* __restrict__ jobs, int k) {
  __shared__ double red[kHouseThreads / 32];
  const EigJob J = jobs[blockIdx.x];
  const int n = J.n, tid = threadIdx.x;
  const Scal S = scal(b, J);
  const double* __restrict__ A = b.a + J.a_off;
  double* __restrict__ V = b.work + J.v_off;
  if (n == 1) {
    if (k == 0 && tid == 0) {
      S.d[0] = A[0];
      S.e[0] = 0.0;
    }
    return;
  }
  if (k > n - 2) return;
  const double* vp = V + (int64_t)(k >= 1 ? k - 1 : 0) * n;  // v_{k-1} (read for k >= 1)
  double* wp = S.wr + (int64_t)((k + 1) & 1) * n;            // w_{k-1}
  double* col = S.wr + (int64_t)(k & 1) * n;
  if (k >= 1) {
    const int nt = J.nt, j0 = k / kEigTile;
    const double t = S.tau[k - 1];
    double pv = 0.0;
    for (int i = k + tid; i < n; i += kHouseThreads) {
      const int ti = i / kEigTile;
      double s = 0.0;
      for (int jt = j0; jt <= ti; ++jt) s += S.prow[(int64_t)jt * n + i];
      for (int it = ti + 1; it < nt; ++it) s += S.pcol[(int64_t)it * n + i];
      s *= t;
      wp[i] = s;
      pv += s * vp[i];
    }
    const double K = 0.5 * t * block_sum<kHouseThreads>(pv, red);
    for (int i = k + tid; i < n; i += kHouseThreads) wp[i] -= K * vp[i];
    __syncthreads();
  }
  // column k of A^(k), rows k..n-1
  const double wk = k >= 1 ? wp[k] : 0.0, vk = k >= 1 ? vp[k] : 0.0;
  double ss = 0.0;
  for (int i = k + tid; i < n; i += kHouseThreads) {
    double c = A[(int64_t)i * n + k];
    if (k >= 1) c -= vp[i] * wk + wp[i] * vk;
    col[i] = c;
    if (i >= k + 2) ss += c * c;
  }
  ss = block_sum<kHouseThreads>(ss, red);  // also orders the writes of col
  if (k == n - 2) {
    if (tid == 0) {
      S.d[k] = col[k];
      S.e[k] = col[k + 1];
      double dd = A[(int64_t)(k + 1) * n + k + 1];
      if (k >= 1) dd -= 2.0 * vp[k + 1] * wp[k + 1];
      S.d[k + 1] = dd;
      S.e[k + 1] = 0.0;
      S.tau[k] = 0.0;
    }
    return;
  }
  const double alpha = col[k + 1];
  const double xn = sqrt(ss + alpha * alpha);
  double beta = 0.0, t = 0.0, scale = 0.0, lead = 0.0;
  if (xn != 0.0) {
    beta = -copysign(xn, alpha);
    t = (beta - alpha) / beta;
    scale = 1.0 / (alpha - beta);
    lead = 1.0;
  }
  double* vk_row = V + (int64_t)k * n;
  for (int i = tid; i < n; i += kHouseThreads) vk_row[i] = i <= k ? 0.0 : (i == k + 1 ? lead : col[i] * scale);
  if (tid == 0) {
    S.d[k] = col[k];
    S.e[k] = beta;
    S.tau[k] = t;
  }
}

__device__ __forceinline__ int find_job(const EigJob* jobs, int njobs, int bid, int which) {
  int j = 0;
  for (int q = 1; q < njobs; ++q) {
    const int first = which == 0 ? jobs[q].tile0 : jobs[q].bt0;
    if (first <= bid) j = q;
  }
  return j;
}

// One CTA per 64 x 64 tile (I >= J) of a job's lower triangle: applies the
// rank-2 update of step k-1 to the tile's part of rows / columns >= k+1 and
// writes the tile's partial sums of A^(k) v_k: row sums to prow[J][rows of
// I], column sums (off-diagonal tiles) to pcol[I][columns of J]; a diagonal
// tile writes the sum of both to prow[I].
__global__ void __launch_bounds__(kUpdThreads) eig_update(EigBufs b, const EigJob* __restrict__ jobs, int njobs,
                                                          int k) {
  __shared__ double vr[kEigTile], vc[kEigTile], pvr[kEigTile], pwr[kEigTile], pvc[kEigTile], pwc[kEigTile];
  __shared__ double rows[kEigTile], colred[kUpdThreads / 32][kEigTile];
  const int bid = blockIdx.x;
  const EigJob J = jobs[find_job(jobs, njobs, bid, 0)];
  const int n = J.n;
  if (k > n - 3) return;
  const int t = bid - J.tile0;
  int I = (int)((sqrt(8.0 * t + 1.0) - 1.0) * 0.5);
  while ((I + 1) * (I + 2) / 2 <= t) ++I;
  while (I * (I + 1) / 2 > t) --I;
  const int JJ = t - I * (I + 1) / 2;
  if (I >= J.nt || JJ * kEigTile + kEigTile - 1 < k + 1) return;  // no active column
  const Scal S = scal(b, J);
  double* __restrict__ A = b.a + J.a_off;
  const double* __restrict__ V = b.work + J.v_off;
  const double* v = V + (int64_t)k * n;
  const double* vp = V + (int64_t)(k >= 1 ? k - 1 : 0) * n;
  const double* wp = S.wr + (int64_t)((k + 1) & 1) * n;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int r0 = I * kEigTile, c0 = JJ * kEigTile;
  if (tid < kEigTile) {
    const int i = r0 + tid, j = c0 + tid;
    vr[tid] = i < n ? v[i] : 0.0;
    vc[tid] = j < n ? v[j] : 0.0;
    pvr[tid] = (k >= 1 && i < n) ? vp[i] : 0.0;
    pwr[tid] = (k >= 1 && i < n) ? wp[i] : 0.0;
    pvc[tid] = (k >= 1 && j < n) ? vp[j] : 0.0;
    pwc[tid] = (k >= 1 && j < n) ? wp[j] : 0.0;
  }
  __syncthreads();
  double cacc[2] = {0.0, 0.0};
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int r = warp * 8 + q, i = r0 + r;
    double racc = 0.0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int c = lane + 32 * h, j = c0 + c;
      if (i < n && j < n && j >= k + 1 && i >= j) {
        double* pa = A + (int64_t)i * n + j;
        double a = *pa;
        if (k >= 1) {
          a -= pvr[r] * pwc[c] + pwr[r] * pvc[c];
          *pa = a;
        }
        racc += a * vc[c];
        if (i != j) cacc[h] += a * vr[r];
      }
    }
    racc = warp_sum(racc);
    if (lane == 0) rows[r] = racc;
  }
  colred[warp][lane] = cacc[0];
  colred[warp][lane + 32] = cacc[1];
  __syncthreads();
  if (tid < kEigTile) {
    double cs = 0.0;
#pragma unroll
    for (int w = 0; w < kUpdThreads / 32; ++w) cs += colred[w][tid];
    if (I == JJ) {
      if (r0 + tid < n) S.prow[(int64_t)JJ * n + r0 + tid] = rows[tid] + cs;
    } else {
      if (r0 + tid < n) S.prow[(int64_t)JJ * n + r0 + tid] = rows[tid];
      if (c0 + tid < n) S.pcol[(int64_t)I * n + c0 + tid] = cs;
    }
  }
}

// Back-transformation V = H_0 H_1 ... H_{n-3} Z, one eigenvector per warp in
// shared memory, written at the rank of its eigenvalue (ascending; ties in
// index order).  Four warps a block, one per quarter of the SM, since a
// warp's FP64 operations issue every 63 clocks; the next reflector is copied
// while the present one is applied.  12 matrices up to order 400: 1000 ->
// 846 us (eight warps and two barriers a reflector: fewer, longer blocks).
__global__ void __launch_bounds__(kBtThreads) eig_backtransform(EigBufs b, const EigJob* __restrict__ jobs,
                                                                int njobs, int max_n) {
  extern __shared__ double sm[];
  const int bid = blockIdx.x;
  const int jidx = find_job(jobs, njobs, bid, 2);
  const EigJob J = jobs[jidx];
  const int n = J.n, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const Scal S = scal(b, J);
  const double* __restrict__ V = b.work + J.v_off;
  const double* __restrict__ Q = b.work + J.q_off;
  double* zc = sm + (2 + warp) * (int64_t)max_n;
  const int j = (bid - J.bt0) * kEigBtCols + warp;
  const bool mine = j < n;
  if (mine)
    for (int i = lane; i < n; i += 32) zc[i] = Q[(int64_t)j * n + i];
  auto fetch = [&](int k) {  // reflector k into its buffer
    double* dst = sm + (k & 1) * (int64_t)max_n;
    for (int i = k + 1 + tid; i < n; i += kBtThreads)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst + i)),
                   "l"(V + (int64_t)k * n + i)
                   : "memory");
  };
  if (n >= 3) fetch(n - 3);
  for (int k = n - 3; k >= 0; --k) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();  // reflector k is here, k + 1 is no longer read
    if (k > 0) fetch(k - 1);
    if (!mine) continue;
    const double* vs = sm + (k & 1) * (int64_t)max_n;
    const double tau = S.tau[k];
    double dot = 0.0;
    for (int i = k + 1 + lane; i < n; i += 32) dot = fma(vs[i], zc[i], dot);
    dot = -tau * warp_sum(dot);
    for (int i = k + 1 + lane; i < n; i += 32) zc[i] = fma(dot, vs[i], zc[i]);
  }
  if (!mine) return;
  const double lam = S.eu[j];
  int rank = 0;
  for (int i = lane; i < n; i += 32) {
    const double x = S.eu[i];
    rank += (x < lam || (x == lam && i < j)) ? 1 : 0;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) rank += __shfl_xor_sync(0xffffffffu, rank, o);
  __syncwarp();
  double* out = b.z + J.z_off + (int64_t)rank * n;
  for (int i = lane; i < n; i += 32) out[i] = zc[i];
  if (lane == 0) b.w[J.w_off + rank] = lam;
}

// ---------------------------------------------------------------- clusters
//
// The same reduction with the matrix held in the shared memory of one
// thread-block cluster per job (full symmetric storage, row i in block
// i mod C), all columns in one launch.  Per column k:
//   col   every block corrects column k in its rows (the lazy rank-2 update
//         of step k-1) and stores it into all blocks' shared memory;
//   upd   while that exchange is under way, the rank-2 update of the block's
//         trailing rows (it does not need the new reflector);
//   house every block forms the whole reflector from the exchanged column;
//   mul   p = A v for the block's rows, stored into all blocks;
//   w     every block forms w from p.
// Two cluster barriers a column replace two launches of the whole grid.
// Bound by the FP64 pipe (3 n^3 / 3 FMAs at 1.7 a clock and SM over C SMs)
// and, per column, by about 40 dependent FP64 operations of 63 clocks each:
// sums therefore use four warps (one per quarter of the SM), four rows share
// a warp's reduction, and the scalars are formed by one warp.  12 matrices up
// to order 400 in clusters of 16: 2950 us, against 11.7 ms for the tiled
// launches (17 + 12 us a column).
constexpr int kClThreads = 512, kClWarps = kClThreads / 32;
constexpr int kClSumWarps = 4;

// (.aligned: every lane of a warp executes them together, also behind a loop that
// the lanes leave after different numbers of turns)
__device__ __forceinline__ void cl_arrive() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cl_wait() {
  __syncwarp();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cl_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cl_size() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
// x into block `rank`'s copy of the shared-memory variable at p
__device__ __forceinline__ void cl_store(double* p, uint32_t rank, double x) {
  uint32_t a = (uint32_t)__cvta_generic_to_shared(p), m;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(m) : "r"(a), "r"(rank));
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(m), "d"(x) : "memory");
}

// row stride of the shared matrix: odd, so that a column's rows fall into
// different banks
__host__ __device__ inline int cl_ld(int n) { return n | 1; }

__global__ void __launch_bounds__(kClThreads, 1) eig_tridiag_cluster(EigBufs b, const EigJob* __restrict__ jobs) {
  extern __shared__ double sm[];
  __shared__ double red[kClSumWarps], sc[4];  // sc: scale, lead, tau, K
  const uint32_t C = cl_size(), rank = cl_rank();
  const EigJob J = jobs[blockIdx.x / C];
  const int n = J.n, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const Scal S = scal(b, J);
  const double* __restrict__ A = b.a + J.a_off;
  double* __restrict__ V = b.work + J.v_off;
  if (n == 1) {  // the whole cluster
    if (rank == 0 && tid == 0) {
      S.d[0] = A[0];
      S.e[0] = 0.0;
    }
    return;
  }
  const int ld = cl_ld(n), rows = (n - (int)rank + (int)C - 1) / (int)C;  // rows rank, rank + C, ..
  double *v = sm, *w = sm + n, *col = sm + 2 * n, *p = sm + 3 * n, *a = sm + 4 * n;
  for (int r = warp; r < rows; r += kClWarps) {
    const int i = r * (int)C + (int)rank;
    for (int j = lane; j < n; j += 32) a[r * ld + j] = j <= i ? A[(int64_t)i * n + j] : A[(int64_t)j * n + i];
  }
  for (int i = tid; i < n; i += kClThreads) v[i] = w[i] = 0.0;  // step 0 has no update behind it
  cl_arrive();
  cl_wait();  // every block runs before its shared memory is written
  // first local row of global row i or above
  auto first = [&](int i) { return max(0, (i - (int)rank + (int)C - 1) / (int)C); };
  for (int k = 0; k <= n - 2; ++k) {
    // column k of A^(k), rows k..n-1
    const int rk = first(k);
    if (tid < rows - rk) {
      const int r = rk + tid, i = r * (int)C + (int)rank;
      double c = a[r * ld + k];
      c -= v[i] * w[k] + w[i] * v[k];
      for (uint32_t q = 0; q < C; ++q) cl_store(col + i, q, c);
    }
    cl_arrive();
    // rank-2 update of the trailing rows and columns k+1..
    const int r1 = first(k + 1);
    if (k > 0) {
      for (int r = r1 + warp; r < rows; r += kClWarps) {
        const int i = r * (int)C + (int)rank;
        const double vi = v[i], wi = w[i];
        double* row = a + r * ld;
        for (int j = k + 1 + lane; j < n; j += 32) row[j] = fma(-wi, v[j], fma(-vi, w[j], row[j]));
      }
    }
    cl_wait();
    if (k == n - 2) break;
    // reflector
    if (warp < kClSumWarps) {
      double ss = 0.0;
      for (int i = k + 2 + tid; i < n; i += 32 * kClSumWarps) ss = fma(col[i], col[i], ss);
      ss = warp_sum(ss);
      if (lane == 0) red[warp] = ss;
    }
    __syncthreads();
    if (warp == 0) {
      const double ss = (red[0] + red[1]) + (red[2] + red[3]);
      const double alpha = col[k + 1];
      const double xn = sqrt(fma(alpha, alpha, ss));
      const double beta = -copysign(xn, alpha);
      // lane 0: tau = (beta - alpha) / beta, lane 1: scale = 1 / (alpha - beta)
      const double num = lane == 0 ? beta - alpha : 1.0, den = lane == 0 ? beta : alpha - beta;
      const double q = xn != 0.0 ? num / den : 0.0;
      if (lane == 0) {
        sc[2] = q;
        sc[1] = xn != 0.0 ? 1.0 : 0.0;
        if (rank == 0) {
          S.d[k] = col[k];
          S.e[k] = xn != 0.0 ? beta : 0.0;
          S.tau[k] = q;
        }
      } else if (lane == 1) {
        sc[0] = q;
      }
    }
    __syncthreads();
    for (int i = k + 1 + tid; i < n; i += kClThreads) {
      const double x = i == k + 1 ? sc[1] : col[i] * sc[0];
      v[i] = x;
      if ((uint32_t)i % C == rank) V[(int64_t)k * n + i] = x;
    }
    __syncthreads();
    // p = A v, the block's rows: eight lanes per row, so that four rows share
    // a reduction of three steps
    for (int g = r1 + 4 * warp; g < rows; g += 4 * kClWarps) {
      const int r = g + (lane >> 3);
      const bool mine = r < rows;
      const double* row = a + (mine ? r : g) * ld;
      double x = 0.0;
      for (int j = k + 1 + (lane & 7); j < n; j += 8) x = fma(row[j], v[j], x);
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
      if (mine)
        for (uint32_t q = lane & 7; q < C; q += 8) cl_store(p + r * (int)C + (int)rank, q, x);
    }
    cl_arrive();
    cl_wait();
    // w = tau p - (tau / 2) (tau p . v) v
    const double t = sc[2];
    if (warp < kClSumWarps) {
      double pv = 0.0;
      for (int i = k + 1 + tid; i < n; i += 32 * kClSumWarps) pv = fma(p[i], v[i], pv);
      pv = warp_sum(pv);
      if (lane == 0) red[warp] = pv;
    }
    __syncthreads();
    if (warp == 0) {
      const double pv = (red[0] + red[1]) + (red[2] + red[3]);
      if (lane == 0) sc[3] = 0.5 * t * (t * pv);
    }
    __syncthreads();
    const double K = sc[3];
    for (int i = k + 1 + tid; i < n; i += kClThreads) w[i] = fma(-K, v[i], t * p[i]);
    __syncthreads();
  }
  // last 2 x 2 block (the update of step n-3 has been applied to its rows)
  if (tid == 0 && (uint32_t)(n - 1) % C == rank) {
    S.d[n - 2] = col[n - 2];
    S.e[n - 2] = col[n - 1];
    S.d[n - 1] = a[(rows - 1) * ld + n - 1];
    S.e[n - 1] = 0.0;
    S.tau[n - 2] = 0.0;
  }
}

}  // namespace

// One CTA per matrix, one warp per eigenvector: the vector's largest
// component (the first of equal ones) made positive.
__global__ void __launch_bounds__(256) canon_signs_kernel(double* V, const int64_t* __restrict__ off,
                                                          const int* __restrict__ dims, const int* __restrict__ colmajor) {
  const int q = blockIdx.x, n = dims[q];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double* v = V + off[q];
  const bool cm = colmajor[q] != 0;
  for (int j = warp + 8 * blockIdx.y; j < n; j += 8 * gridDim.y) {
    double best = -1.0, val = 0.0;
    int bi = n;
    for (int i = lane; i < n; i += 32) {
      const double x = cm ? v[(int64_t)j * n + i] : v[(int64_t)i * n + j];
      if (fabs(x) > best) {
        best = fabs(x);
        bi = i;
        val = x;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double b2 = __shfl_xor_sync(0xffffffffu, best, o);
      const int i2 = __shfl_xor_sync(0xffffffffu, bi, o);
      const double v2 = __shfl_xor_sync(0xffffffffu, val, o);
      if (b2 > best || (b2 == best && i2 < bi)) {
        best = b2;
        bi = i2;
        val = v2;
      }
    }
    if (val < 0.0)
      for (int i = lane; i < n; i += 32) {
        double& x = cm ? v[(int64_t)j * n + i] : v[(int64_t)i * n + j];
        x = -x;
      }
  }
}

// Square matrices transposed, 32 x 32 tiles through shared memory.
__global__ void __launch_bounds__(256) transpose_kernel(const double* __restrict__ a, double* __restrict__ t,
                                                        const int64_t* __restrict__ off, const int* __restrict__ dims) {
  __shared__ double tile[32][33];
  const int n = dims[blockIdx.x], nt = (n + 31) / 32, x = threadIdx.x & 31, y = threadIdx.x >> 5;
  const double* src = a + off[blockIdx.x];
  double* dst = t + off[blockIdx.x];
  for (int b = blockIdx.y; b < nt * nt; b += gridDim.y) {
    const int r0 = 32 * (b / nt), c0 = 32 * (b % nt);
    for (int i = y; i < 32; i += 8)
      if (r0 + i < n && c0 + x < n) tile[i][x] = src[(int64_t)(r0 + i) * n + c0 + x];
    __syncthreads();
    for (int i = y; i < 32; i += 8)
      if (c0 + i < n && r0 + x < n) dst[(int64_t)(c0 + i) * n + r0 + x] = tile[x][i];
    __syncthreads();
  }
}

cudaError_t launch_transpose(const double* a, double* t, const int64_t* off, const int* dims, int nmat,
                             cudaStream_t s) {
  if (nmat > 0) transpose_kernel<<<dim3(nmat, 32), 256, 0, s>>>(a, t, off, dims);
  return cudaGetLastError();
}

cudaError_t launch_canon_signs(double* V, const int64_t* off, const int* dims, const int* colmajor, int nmat,
                               cudaStream_t s) {
  if (nmat > 0) canon_signs_kernel<<<dim3(nmat, 8), 256, 0, s>>>(V, off, dims, colmajor);
  return cudaGetLastError();
}

cudaError_t launch_eig_tridiag(const EigBufs& b, const EigJob* jobs, int njobs, int max_n, int tiles,
                               cudaStream_t s) {
  if (njobs <= 0) return cudaSuccess;
  if (max_n < 1 || max_n > kEigMaxN) return cudaErrorInvalidValue;
  for (int k = 0; k <= max_n - 2 || k == 0; ++k) {
    eig_house<<<njobs, kHouseThreads, 0, s>>>(b, jobs, k);
    if (k <= max_n - 3 && tiles > 0) eig_update<<<tiles, kUpdThreads, 0, s>>>(b, jobs, njobs, k);
    if (max_n < 2) break;
  }
  return cudaGetLastError();
}

namespace {
size_t cl_smem(int n, int c) { return ((size_t)4 * n + (size_t)((n + c - 1) / c) * cl_ld(n)) * sizeof(double); }
constexpr size_t kClSmemMax = 226 * 1024;
}  // namespace

// largest order that clusters of 1 << k blocks hold
static int eig_cluster_order(int k) {
  int n = 1;
  while (cl_smem(n + 1, 1 << k) <= kClSmemMax) ++n;
  return n;
}

static cudaError_t eig_cluster_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute& attr, int c, int nclusters,
                                      size_t smem, cudaStream_t s) {
  // the kernel's limits are always set to the same values: another context's thread
  // may set them between here and the launch
  cudaError_t e =
      cudaFuncSetAttribute(eig_tridiag_cluster, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kClSmemMax);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(eig_tridiag_cluster, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e != cudaSuccess) return e;
  cfg = {};
  cfg.gridDim = dim3((unsigned)(c * nclusters));
  cfg.blockDim = dim3(kClThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  attr = {};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = (unsigned)c;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaSuccess;
}

cudaError_t eig_clusters(EigClusters& ec) {
  for (int k = 0; k < kEigClusterSizes; ++k) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr;
    const cudaError_t e = eig_cluster_config(cfg, attr, 1 << k, 1, kClSmemMax, nullptr);
    if (e != cudaSuccess) return e;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, eig_tridiag_cluster, &cfg) != cudaSuccess) {
      cudaGetLastError();  // no cluster of this size
      n = 0;
    }
    ec.resident[k] = n;
    ec.order[k] = n > 0 ? eig_cluster_order(k) : 0;
  }
  return cudaSuccess;
}

int eig_cluster_max_n(const EigClusters& ec) { return *std::max_element(ec.order, ec.order + kEigClusterSizes); }

// Orders fall into classes by the smallest clusters that hold them; runs of
// neighbouring classes share a launch, and each launch takes the cluster size
// with which it ends first: small clusters for many matrices (400 of order 100:
// 2.1 ms with one block each, 11.9 with 8, 7.0 with the tiled launches), large
// ones for few (12 up to order 400: 2.9 ms with 16 blocks, 3.8 with 8).  A job
// takes n^3 / 1.7 C clocks of FMAs and 7400 + 90 C a column for the exchanges and
// scalars (fitted to orders 100 to 640).  The jobs of a launch, in descending
// order, run as clusters become free: their time lies between their sum over
// the resident clusters and that of rounds of the largest jobs.  The launches run
// one after the other.
std::vector<EigClass> eig_cluster_classes(const EigClusters& ec, const int* dims, int njobs) {
  if (njobs <= 0) return {};
  std::vector<int> at{0};  // first jobs of the classes
  auto needs = [&](int n) {
    int k = 0;
    while (k < kEigClusterSizes && ec.order[k] < n) ++k;
    return k;
  };
  std::vector<double> s1(njobs + 1, 0.0), s3(njobs + 1, 0.0);
  for (int j = 0; j < njobs; ++j) {
    const double n = dims[j];
    s1[j + 1] = s1[j] + n;
    s3[j + 1] = s3[j] + n * n * n;
    if (j > 0 && needs(dims[j]) != needs(dims[j - 1])) at.push_back(j);
  }
  at.push_back(njobs);
  const int nc = (int)at.size() - 1;
  std::vector<double> best(nc + 1, 1e300);
  std::vector<EigClass> last(nc + 1);
  best[0] = 0.0;
  for (int i = 0; i < nc; ++i)
    for (int k = 0; k < kEigClusterSizes; ++k) {
      if (ec.order[k] < dims[at[i]]) continue;
      const double fma = 1.0 / (1.7 * (1 << k)), col = 7400.0 + 90.0 * (1 << k);
      for (int e = i + 1; e <= nc; ++e) {
        double rounds = 0.0;
        for (int j = at[i]; j < at[e]; j += ec.resident[k]) {
          const double n = dims[j];
          rounds += n * n * n * fma + n * col;
        }
        const double n0 = dims[at[i]], one = n0 * n0 * n0 * fma + n0 * col;
        const double even = ((s3[at[e]] - s3[at[i]]) * fma + (s1[at[e]] - s1[at[i]]) * col) / ec.resident[k];
        const double t = best[i] + 0.5 * (rounds + std::max(one, even));
        if (t < best[e]) {
          best[e] = t;
          last[e] = {at[e] - at[i], k};
        }
      }
    }
  std::vector<EigClass> out;
  for (int e = nc; e > 0;) {
    out.push_back(last[e]);
    const int first = at[e] - last[e].jobs;
    while (at[e] != first) --e;
  }
  std::reverse(out.begin(), out.end());
  return out;
}

cudaError_t launch_eig_tridiag_cluster(const EigBufs& b, const EigJob* jobs, int max_n, const EigClass& cl,
                                       cudaStream_t s) {
  if (cl.jobs <= 0) return cudaSuccess;
  if (cl.k < 0 || cl.k >= kEigClusterSizes || max_n < 1 || cl_smem(max_n, 1 << cl.k) > kClSmemMax)
    return cudaErrorInvalidValue;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr;
  cudaError_t e = eig_cluster_config(cfg, attr, 1 << cl.k, cl.jobs, cl_smem(max_n, 1 << cl.k), s);
  if (e != cudaSuccess) return e;
  e = cudaLaunchKernelEx(&cfg, eig_tridiag_cluster, b, jobs);
  if (e != cudaSuccess) return e;
  return cudaGetLastError();
}

cudaError_t launch_eig_backtransform(const EigBufs& b, const EigJob* jobs, int njobs, int max_n, int bt_ctas,
                                     cudaStream_t s) {
  if (njobs <= 0) return cudaSuccess;
  if (max_n < 1 || max_n > kEigMaxN) return cudaErrorInvalidValue;
  constexpr size_t per_row = (2 + kEigBtCols) * sizeof(double);
  const size_t smem = per_row * max_n;
  cudaError_t e = cudaFuncSetAttribute(eig_backtransform, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)(per_row * kEigMaxN));  // the same for every call, as above
  if (e != cudaSuccess) return e;
  eig_backtransform<<<bt_ctas, kBtThreads, smem, s>>>(b, jobs, njobs, max_n);
  return cudaGetLastError();
}

}  // namespace dev
}  // namespace bgpu
