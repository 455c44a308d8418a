// FP64 dense building blocks on the library's own kernels: batched LU
// (qbg_linalg.cu), explicit inverses, and the smallest singular value of A(k): by
// subspace iteration on A(k)^{-1} (the inverses' entry and the Newton step), and by
// a Lanczos iteration on the LU factors (namespace lz below; the sweeps).
//
// sigma_min (the reference: svdvals(A)[end], macros.jl:159-161): with
// C = A^{-1} = V S^{-1} U^H, sigma_min(A) = 1 / sigma_max(C). A block X of
// DENSE_P orthonormal columns is iterated X <- orth(C^H C X); after W = C X,
// the Rayleigh-Ritz value lambda_max(W^H W) approaches sigma_max(C)^2 from
// below, and W z (z the top Ritz vector) approaches v_min / sigma_min, the
// right singular vector of A. Convergence per step goes like
// (sigma_1 / sigma_{DENSE_P + 1})^2 of A; the iteration stops when
// 1 / sqrt(lambda_max) changes by less than tol relative.
#include <algorithm>
#include <cmath>
#include <cooperative_groups.h>
#include <vector>

#include "qbg_dense.cuh"

namespace qbg {

namespace {

constexpr int SP = DENSE_P;
constexpr int KC = 128;  // rows of X staged per chunk of the product C X

// every thread receives the block total of v[0..NV) (256 threads)
template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV], double* sh) {
#pragma unroll
  for (int i = 0; i < NV; ++i)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0)
#pragma unroll
    for (int i = 0; i < NV; ++i) sh[wid * NV + i] = v[i];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    double t = 0.0;
#pragma unroll
    for (int w = 0; w < 8; ++w) t += sh[w * NV + i];
    v[i] = t;
  }
}

// deterministic fill value in [-1, 1) for (row, column, salt)
__device__ __forceinline__ double fillv(int r, int c, int salt) {
  unsigned long long x = 0x9E3779B97F4A7C15ull * (unsigned long long)(r + 1) + 0xBF58476D1CE4E5B9ull * (c + 7) +
                         0x94D049BB133111EBull * (salt + 3);
  x ^= x >> 31;
  x *= 0xD6E8FEB86659FD93ull;
  x ^= x >> 29;
  return (double)(x >> 11) * (2.0 / 9007199254740992.0) - 1.0;
}

// orthonormal columns of Q (n x SP, column-major) in place: classical
// Gram-Schmidt applied twice per column; a column that vanishes against the
// earlier ones (below 1e-14 of its length) is refilled and orthogonalised again
__device__ void orth_cgs2(cxd* Q, int n, double* sh, int salt) {
  const int tid = threadIdx.x;
  for (int j = 0; j < SP; ++j) {
    cxd* qj = Q + (size_t)j * n;
    for (int attempt = 0; attempt < 3; ++attempt) {
      double v0[1] = {0.0};
      for (int r = tid; r < n; r += 256) v0[0] += cabs2(qj[r]);
      block_sum<1>(v0, sh);
      const double n0 = sqrt(v0[0]);
      for (int pass = 0; pass < 2 && j > 0; ++pass) {
        double c[2 * SP];
#pragma unroll
        for (int i = 0; i < 2 * SP; ++i) c[i] = 0.0;
        for (int r = tid; r < n; r += 256) {
          const cxd y = qj[r];
#pragma unroll
          for (int i = 0; i < SP; ++i)
            if (i < j) {
              const cxd qi = Q[(size_t)i * n + r];
              c[2 * i] += qi.re * y.re + qi.im * y.im;  // conj(qi) y
              c[2 * i + 1] += qi.re * y.im - qi.im * y.re;
            }
        }
        block_sum<2 * SP>(c, sh);
        for (int r = tid; r < n; r += 256) {
          cxd y = qj[r];
#pragma unroll
          for (int i = 0; i < SP; ++i)
            if (i < j) cfms(y, Q[(size_t)i * n + r], cxd(c[2 * i], c[2 * i + 1]));
          qj[r] = y;
        }
      }
      double v1[1] = {0.0};
      for (int r = tid; r < n; r += 256) v1[0] += cabs2(qj[r]);
      block_sum<1>(v1, sh);
      const double n1 = sqrt(v1[0]);
      if (n1 > 1e-14 * n0 && n1 > 1e-300 && isfinite(n1)) {
        const double s = 1.0 / n1;
        for (int r = tid; r < n; r += 256) qj[r] = qj[r] * s;
        break;
      }
      for (int r = tid; r < n; r += 256) qj[r] = cxd(fillv(r, j, salt + attempt), fillv(r, j + SP, salt + attempt));
      __syncthreads();
    }
  }
  __syncthreads();
}

// largest eigenvalue and its eigenvector of the Hermitian SP x SP matrix G
// (column-major, complex, exactly Hermitian) by cyclic Jacobi on its real
// 2SP x 2SP embedding [[Re G, -Im G], [Im G, Re G]], run by one whole warp on
// the shared scratch wk (2 (2SP)^2 doubles): for each rotation every lane
// derives the same (c, s) from the pivot entries, then lane k < 2SP rotates
// column k's pair (p, q) and row k's pair of the matrix, lanes 2SP.. the
// eigenvector columns. Lane 0 writes lam and z (SP complex). A one-thread
// version on thread-local 16 x 16 arrays lost the symmetry of the matrix
// after its first sweep when built with device optimisation for sm_103a
// (correct at -G and on the host), hence the shared-memory form.
__device__ void herm_top(const double* G, double* lam, double* z, double* wk) {
  constexpr int M2 = 2 * SP;
  const int lane = threadIdx.x & 31;
  double* a = wk;
  double* v = wk + M2 * M2;
  for (int e = lane; e < M2 * M2; e += 32) {
    const int r = e / M2, c = e % M2, gr = r % SP, gc = c % SP;
    const double re = G[2 * (gc * SP + gr)], im = G[2 * (gc * SP + gr) + 1];
    a[e] = (r < SP) == (c < SP) ? re : (r >= SP ? im : -im);
    v[e] = r == c ? 1.0 : 0.0;
  }
  __syncwarp();
  for (int sweep = 0; sweep < 40; ++sweep) {
    double off = 0.0, dia = 0.0;
    for (int e = lane; e < M2 * M2; e += 32) {
      const double t = a[e] * a[e];
      if (e / M2 == e % M2)
        dia += t;
      else
        off += t;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      off += __shfl_xor_sync(0xffffffffu, off, o);
      dia += __shfl_xor_sync(0xffffffffu, dia, o);
    }
    // lane 0's sums decide for the whole warp (the butterfly may round per lane).
    // Converged at an off-diagonal norm of 1e-15 of the diagonal's: rounding
    // keeps every rotated pair at ~eps of its entries, so a tighter stop is
    // never met and the sweeps would run to their limit.
    off = __shfl_sync(0xffffffffu, off, 0);
    dia = __shfl_sync(0xffffffffu, dia, 0);
    if (!(off > 1e-30 * dia)) break;
    for (int p = 0; p < M2 - 1; ++p)
      for (int q = p + 1; q < M2; ++q) {
        const double apq = a[p * M2 + q];
        // an entry at rounding level of its diagonal pair needs no rotation
        if (fabs(apq) < 1e-300 || fabs(apq) <= 1e-17 * sqrt(fabs(a[p * M2 + p] * a[q * M2 + q]))) continue;
        const double th = (a[q * M2 + q] - a[p * M2 + p]) / (2.0 * apq);
        const double t = (th >= 0.0 ? 1.0 : -1.0) / (fabs(th) + sqrt(th * th + 1.0));
        const double c = 1.0 / sqrt(t * t + 1.0), s = t * c;
        __syncwarp();
        if (lane < M2) {
          const double akp = a[lane * M2 + p], akq = a[lane * M2 + q];
          a[lane * M2 + p] = c * akp - s * akq;
          a[lane * M2 + q] = s * akp + c * akq;
        } else {
          const int k = lane - M2;
          const double vkp = v[k * M2 + p], vkq = v[k * M2 + q];
          v[k * M2 + p] = c * vkp - s * vkq;
          v[k * M2 + q] = s * vkp + c * vkq;
        }
        __syncwarp();
        if (lane < M2) {
          const double apk = a[p * M2 + lane], aqk = a[q * M2 + lane];
          a[p * M2 + lane] = c * apk - s * aqk;
          a[q * M2 + lane] = s * apk + c * aqk;
        }
        __syncwarp();
      }
  }
  if (lane == 0) {
    int best = 0;
    for (int i = 1; i < M2; ++i)
      if (a[i * M2 + i] > a[best * M2 + best]) best = i;
    *lam = a[best * M2 + best];
    double nrm = 0.0;
    for (int i = 0; i < SP; ++i) {
      z[2 * i] = v[i * M2 + best];
      z[2 * i + 1] = v[(i + SP) * M2 + best];
      nrm += z[2 * i] * z[2 * i] + z[2 * i + 1] * z[2 * i + 1];
    }
    nrm = nrm > 0.0 ? 1.0 / sqrt(nrm) : 0.0;
    for (int i = 0; i < 2 * SP; ++i) z[i] *= nrm;
  }
  __syncwarp();
}

// One CTA per matrix: the subspace iteration on C_b = A_b^{-1} (n x n,
// column-major, stride n^2). X0: the shared n x SP start block; work: per
// matrix 3 n SP elements. sig[b] = sigma_min(A_b); iters[b] = steps taken;
// vec (optional): the unit right singular vector of A_b (n per matrix).
__global__ void __launch_bounds__(256) k_sigma_iter(const cxd* __restrict__ Cb, int n, const cxd* __restrict__ X0,
                                                    cxd* work, int maxit, double tol, double* sig, int* iters,
                                                    cxd* vec) {
  const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const cxd* C = Cb + (size_t)b * n * n;
  cxd* X = work + (size_t)b * 3 * n * SP;
  cxd* W = X + (size_t)n * SP;
  cxd* Y = W + (size_t)n * SP;
  __shared__ double sh[8 * SP * (SP + 1)];
  __shared__ cxd xs[KC][SP];
  __shared__ double Gs[2 * SP * SP];
  __shared__ double zs[2 * SP];
  __shared__ double lam_s;
  __shared__ double hw[2 * 4 * SP * SP];
  for (size_t e = tid; e < (size_t)n * SP; e += 256) X[e] = X0[e];
  __syncthreads();
  orth_cgs2(X, n, sh, 0);
  double est = -1.0;
  int it = 0;
  for (; it < maxit; ++it) {
    // W = C X
    for (int r0 = 0; r0 < n; r0 += 256) {
      const int r = r0 + tid;
      cxd acc[SP];
#pragma unroll
      for (int q = 0; q < SP; ++q) acc[q] = cxd(0.0, 0.0);
      for (int k0 = 0; k0 < n; k0 += KC) {
        __syncthreads();
        for (int e = tid; e < KC * SP; e += 256) {
          const int kk = e % KC, q = e / KC;
          xs[kk][q] = (k0 + kk < n) ? X[(size_t)q * n + k0 + kk] : cxd(0.0, 0.0);
        }
        __syncthreads();
        if (r < n) {
          const int kmax = min(KC, n - k0);
          const cxd* cp = C + r + (size_t)k0 * n;
          for (int kk = 0; kk < kmax; ++kk) {
            const cxd c = cp[(size_t)kk * n];
#pragma unroll
            for (int q = 0; q < SP; ++q) cfma(acc[q], c, xs[kk][q]);
          }
        }
      }
      if (r < n)
#pragma unroll
        for (int q = 0; q < SP; ++q) W[(size_t)q * n + r] = acc[q];
    }
    __syncthreads();
    // G = W^H W (upper triangle, then mirrored)
    {
      double g[SP * (SP + 1)];
#pragma unroll
      for (int i = 0; i < SP * (SP + 1); ++i) g[i] = 0.0;
      for (int r = tid; r < n; r += 256) {
        cxd w[SP];
#pragma unroll
        for (int q = 0; q < SP; ++q) w[q] = W[(size_t)q * n + r];
        int e = 0;
#pragma unroll
        for (int j = 0; j < SP; ++j)
#pragma unroll
          for (int i = 0; i <= j; ++i, e += 2) {
            g[e] += w[i].re * w[j].re + w[i].im * w[j].im;
            g[e + 1] += w[i].re * w[j].im - w[i].im * w[j].re;
          }
      }
      block_sum<SP * (SP + 1)>(g, sh);
      if (wid == 0) {
        if (lane == 0) {
          int e = 0;
          for (int j = 0; j < SP; ++j)
            for (int i = 0; i <= j; ++i, e += 2) {
              // exactly Hermitian: the diagonal of W^H W is real, the summed
              // products only leave a rounding residue there
              const double im = (i == j) ? 0.0 : g[e + 1];
              Gs[2 * (j * SP + i)] = g[e];
              Gs[2 * (j * SP + i) + 1] = im;
              Gs[2 * (i * SP + j)] = g[e];
              Gs[2 * (i * SP + j) + 1] = -im;
            }
        }
        __syncwarp();
        herm_top(Gs, &lam_s, zs, hw);
      }
      __syncthreads();
    }
    const double lam = lam_s;
    const double cur = (lam > 0.0 && isfinite(lam)) ? 1.0 / sqrt(lam) : 0.0;
    const bool done = (it > 0 && fabs(cur - est) <= tol * cur) || !(lam > 0.0 && isfinite(lam));
    est = cur;
    if (done || it + 1 == maxit) {
      ++it;
      break;
    }
    // Y = C^H W, one warp per column of C
    for (int r = wid; r < n; r += 8) {
      double acc[2 * SP];
#pragma unroll
      for (int i = 0; i < 2 * SP; ++i) acc[i] = 0.0;
      const cxd* cc = C + (size_t)r * n;
      for (int k = lane; k < n; k += 32) {
        const cxd c = conj(cc[k]);
#pragma unroll
        for (int q = 0; q < SP; ++q) {
          const cxd w = W[(size_t)q * n + k];
          acc[2 * q] += c.re * w.re - c.im * w.im;
          acc[2 * q + 1] += c.re * w.im + c.im * w.re;
        }
      }
#pragma unroll
      for (int i = 0; i < 2 * SP; ++i)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], o);
      if (lane == 0)
#pragma unroll
        for (int q = 0; q < SP; ++q) Y[(size_t)q * n + r] = cxd(acc[2 * q], acc[2 * q + 1]);
    }
    __syncthreads();
    orth_cgs2(Y, n, sh, 8 * (it + 1));
    cxd* t = X;  // X <- Y (Y is the old X's storage from now on)
    X = Y;
    Y = t;
  }
  if (tid == 0) {
    sig[b] = est;
    if (iters) iters[b] = it;
  }
  if (vec) {
    // W z / |W z|
    double nv[1] = {0.0};
    for (int r = tid; r < n; r += 256) {
      cxd v(0.0, 0.0);
#pragma unroll
      for (int q = 0; q < SP; ++q) cfma(v, W[(size_t)q * n + r], cxd(zs[2 * q], zs[2 * q + 1]));
      vec[(size_t)b * n + r] = v;
      nv[0] += cabs2(v);
    }
    block_sum<1>(nv, sh);
    const double s = nv[0] > 0.0 ? 1.0 / sqrt(nv[0]) : 0.0;
    for (int r = tid; r < n; r += 256) vec[(size_t)b * n + r] = vec[(size_t)b * n + r] * s;
  }
}

// One-matrix steps of the same iteration for callers that spread the products
// over the whole GPU (split-k GEMMs between these launches), one CTA each:
// k_rr_step: G = W^H W, its top eigenpair (lambda, z), est = 1/sqrt(lambda)
// and the convergence flag against the previous estimate (state: est, done,
// z[2 SP]); k_orth8: orthonormal columns of Y in place; k_topvec: x = W z / |W z|.
__global__ void __launch_bounds__(256) k_rr_step(const cxd* __restrict__ W, int n, double tol, double* state) {
  __shared__ double sh[8 * SP * (SP + 1)];
  __shared__ double Gs[2 * SP * SP];
  __shared__ double hw[2 * 4 * SP * SP];
  __shared__ double lam_s;
  const int tid = threadIdx.x;
  double g[SP * (SP + 1)];
#pragma unroll
  for (int i = 0; i < SP * (SP + 1); ++i) g[i] = 0.0;
  for (int r = tid; r < n; r += 256) {
    cxd w[SP];
#pragma unroll
    for (int q = 0; q < SP; ++q) w[q] = W[(size_t)q * n + r];
    int e = 0;
#pragma unroll
    for (int j = 0; j < SP; ++j)
#pragma unroll
      for (int i = 0; i <= j; ++i, e += 2) {
        g[e] += w[i].re * w[j].re + w[i].im * w[j].im;
        g[e + 1] += w[i].re * w[j].im - w[i].im * w[j].re;
      }
  }
  block_sum<SP * (SP + 1)>(g, sh);
  if (tid >= 32) return;
  if (tid == 0) {
    int e = 0;
    for (int j = 0; j < SP; ++j)
      for (int i = 0; i <= j; ++i, e += 2) {
        const double im = (i == j) ? 0.0 : g[e + 1];  // real diagonal (see k_sigma_iter)
        Gs[2 * (j * SP + i)] = g[e];
        Gs[2 * (j * SP + i) + 1] = im;
        Gs[2 * (i * SP + j)] = g[e];
        Gs[2 * (i * SP + j) + 1] = -im;
      }
  }
  __syncwarp();
  herm_top(Gs, &lam_s, state + 2, hw);
  if (tid == 0) {
    const double lam = lam_s;
    const bool ok = lam > 0.0 && isfinite(lam);
    const double cur = ok ? 1.0 / sqrt(lam) : 0.0;
    const double prev = state[0];
    state[1] = (prev >= 0.0 && fabs(cur - prev) <= tol * cur) || !ok ? 1.0 : 0.0;
    state[0] = cur;
  }
}

__global__ void __launch_bounds__(256) k_orth8(cxd* Y, int n, int salt) {
  __shared__ double sh[8 * 2 * SP];
  orth_cgs2(Y, n, sh, salt);
}

__global__ void __launch_bounds__(256) k_topvec(const cxd* __restrict__ W, const double* __restrict__ state, int n,
                                                cxd* __restrict__ x) {
  __shared__ double sh[8];
  const int tid = threadIdx.x;
  double nv[1] = {0.0};
  for (int r = tid; r < n; r += 256) {
    cxd v(0.0, 0.0);
#pragma unroll
    for (int q = 0; q < SP; ++q) cfma(v, W[(size_t)q * n + r], cxd(state[2 + 2 * q], state[3 + 2 * q]));
    x[r] = v;
    nv[0] += cabs2(v);
  }
  block_sum<1>(nv, sh);
  const double s = nv[0] > 0.0 ? 1.0 / sqrt(nv[0]) : 0.0;
  for (int r = tid; r < n; r += 256) x[r] = x[r] * s;
}

// M = G - lam I + mu x x^H (n x n, column-major)
__global__ void k_deflate_shift(const cxd* __restrict__ G, const cxd* __restrict__ x, int n, double lam, double mu,
                                cxd* __restrict__ M) {
  const size_t count = (size_t)n * n;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < count; e += (size_t)gridDim.x * blockDim.x) {
    const int r = (int)(e % n), c = (int)(e / n);
    cxd v = G[e];
    if (r == c) v.re -= lam;
    const cxd xr = x[r], xc = x[c];
    v.re += mu * (xr.re * xc.re + xr.im * xc.im);
    v.im += mu * (xr.im * xc.re - xr.re * xc.im);
    M[e] = v;
  }
}

// ---------------------------------------------------------------------------
// sigma_min of many operators from their LU factors, without the inverses:
// Lanczos with full reorthogonalisation on (A A^H)^{-1}, one cluster of CTAs
// per operator and one launch for the whole iteration.
//
// Each step applies A^{-1} and A^{-H} to one vector by the four triangular
// sweeps of P A = L U (the nb x nb inverses of the diagonal blocks stand in
// for the triangular solves inside a block), orthogonalises against all
// earlier vectors (classical Gram-Schmidt, twice) and every third step takes
// the largest eigenvalue theta of the tridiagonal matrix (Laguerre from
// above); the iteration stops when the Ritz residual beta |s_k| is below
// 1e-12 theta. sigma_min = theta^{-1/2}.
//
// Bound by FP64 issue: 2 n^2 complex products a step, against 16 n^2 a step
// for the eight-column subspace iteration on the explicit inverse and the
// 8/3 n^3 of that inverse. Block r of a vector belongs to CTA r mod CS;
// in step s of a sweep the owner of the next block updates it first, forms
// its part of the solution and arrives at the cluster barrier before its
// other blocks, so that the chain of nblk blocks runs ahead of the updates.
// Measured, the whole sweep: 200 k at n = 512 476 -> 81 ms, 16 k at n = 1130
// 470 -> 78 ms (inverse and subspace iteration before).
// ---------------------------------------------------------------------------
namespace lz {

constexpr int NB = 64, T = 256, KMAX = 96;

struct Op {
  const cxd *A, *Linv, *Uinv;
  const int* perm;
  int n, nblk, rank, cs;
};

// red[64] = rows of a 64 x 64 block times xs: M (ADJ 0) or M^H (ADJ 1), M = m
// with leading dimension ld, rows (of the result) < nr, columns < nc.
template <bool ADJ>
__device__ __forceinline__ cxd block_times(const cxd* m, long long ld, int nr, int nc, const cxd* xs, cxd* red) {
  const int tid = threadIdx.x;
  cxd acc(0.0, 0.0);
  if (!ADJ) {  // thread = row, a quarter of the columns each
    const int i = tid & 63, kq = (tid >> 6) * 16;
    if (i < nr) {
      const cxd* p = m + i + (long long)kq * ld;
      const int ke = min(16, nc - kq);
      if (ke == 16) {
        cxd v[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) v[q] = p[(long long)q * ld];
#pragma unroll
        for (int q = 0; q < 16; ++q) cfma(acc, v[q], xs[kq + q]);
      } else {
        for (int q = 0; q < ke; ++q) cfma(acc, p[(long long)q * ld], xs[kq + q]);
      }
    }
    if (tid >= 64) red[tid - 64] = acc;
    __syncthreads();
    if (tid < 64) acc = ((acc + red[tid]) + red[64 + tid]) + red[128 + tid];
  } else {  // four lanes per column of M
    const int j = tid >> 2, l = tid & 3;
    if (j < nr) {
      const cxd* p = m + (long long)j * ld + l;
      cxd v[16];
#pragma unroll
      for (int q = 0; q < 16; ++q) v[q] = (4 * q + l < nc) ? p[4 * q] : cxd(0.0, 0.0);
#pragma unroll
      for (int q = 0; q < 16; ++q) cfma(acc, conj(v[q]), xs[4 * q + l]);
    }
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
      acc.re += __shfl_xor_sync(0xffffffffu, acc.re, o);
      acc.im += __shfl_xor_sync(0xffffffffu, acc.im, o);
    }
    if (l == 0) red[j] = acc;
    __syncthreads();
    if (tid < 64) acc = red[tid];
  }
  return acc;  // threads 0..63: the result's rows
}

// One triangular sweep in place on z: MODE 0 L, 1 U, 2 U^H, 3 L^H. z is
// complete and visible to the whole cluster afterwards.
template <int MODE>
__device__ void sweep(const Op& o, cxd* z, cxd* xs, cxd* red) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  constexpr bool FWD = MODE == 0 || MODE == 2, ADJ = MODE >= 2;
  const cxd* inv = (MODE == 0 || MODE == 3) ? o.Linv : o.Uinv;
  const int tid = threadIdx.x;
  auto blk = [&](int s) { return FWD ? s : o.nblk - 1 - s; };
  auto size = [&](int b) { return min(NB, o.n - b * NB); };
  auto solve = [&](int b) {  // z_b = inv_b z_b
    const int w = size(b);
    if (tid < 64) xs[tid] = tid < w ? z[b * NB + tid] : cxd(0.0, 0.0);
    __syncthreads();
    const cxd v = block_times<ADJ>(inv + (long long)b * NB * NB, NB, w, w, xs, red);
    if (tid < w) z[b * NB + tid] = v;
    __syncthreads();
  };
  auto update = [&](int r, int b, const cxd* x) {  // z_r -= M(r, b) x
    const int wr = size(r), wb = size(b);
    const cxd* m = ADJ ? o.A + (long long)b * NB + (long long)r * NB * o.n : o.A + (long long)r * NB + (long long)b * NB * o.n;
    const cxd v = block_times<ADJ>(m, o.n, wr, wb, x, red);
    if (tid < wr) z[r * NB + tid] = z[r * NB + tid] - v;
    __syncthreads();
  };
  cxd* x2 = xs + 64;
  if (blk(0) % o.cs == o.rank) solve(blk(0));
  cl.barrier_arrive();
  for (int s = 0; s < o.nblk; ++s) {
    const int b = blk(s);
    cl.barrier_wait();
    if (tid < 64) x2[tid] = tid < size(b) ? z[b * NB + tid] : cxd(0.0, 0.0);
    __syncthreads();
    if (s + 1 == o.nblk) break;
    const int nx = blk(s + 1);
    if (nx % o.cs == o.rank) {
      update(nx, b, x2);
      solve(nx);
    }
    cl.barrier_arrive();
    for (int t = s + 2; t < o.nblk; ++t)
      if (blk(t) % o.cs == o.rank) update(blk(t), b, x2);
    __syncthreads();
  }
}

// largest eigenvalue of the k x k tridiagonal (al, be) and the last component
// of its unit eigenvector; one thread. Laguerre's iteration from the
// Gershgorin bound decreases monotonically to the largest root.
__device__ void tridiag_top(const double* al, const double* be, int k, double* theta, double* last) {
  double bound = 0.0;
  for (int j = 0; j < k; ++j) bound = fmax(bound, al[j] + (j > 0 ? be[j - 1] : 0.0) + (j + 1 < k ? be[j] : 0.0));
  const double sc = 1.0 / bound;  // scaled matrix: spectrum in [0, 1]
  double x = 1.0;
  for (int it = 0; it < 60 && k > 1; ++it) {
    double p0 = 1.0, q0 = 0.0, h0 = 0.0;  // p, p', p'' of the leading minors
    double p1 = x - al[0] * sc, q1 = 1.0, h1 = 0.0;
    for (int j = 1; j < k; ++j) {
      const double d = x - al[j] * sc, b = be[j - 1] * sc, b2 = b * b;
      const double p = fma(d, p1, -b2 * p0), q = fma(d, q1, fma(-b2, q0, p1)), h = fma(d, h1, fma(-b2, h0, 2.0 * q1));
      p0 = p1; q0 = q1; h0 = h1;
      p1 = p; q1 = q; h1 = h;
      if (fabs(q1) < 1e-100) {
        p0 *= 1e100; q0 *= 1e100; h0 *= 1e100;
        p1 *= 1e100; q1 *= 1e100; h1 *= 1e100;
      }
    }
    if (!(p1 > 0.0)) break;  // at the root to rounding
    const double g = q1 / p1, hh = g * g - h1 / p1;
    const double rad = (double)(k - 1) * ((double)k * hh - g * g);
    const double dx = (double)k / (g + sqrt(fmax(rad, 0.0)));
    x -= dx;
    if (!(dx > 2e-16 * x)) break;
  }
  const double th = k > 1 ? x * bound : al[0];
  // eigenvector from its last component upwards (growing, hence stable)
  double s1 = 1.0, s2 = 0.0, nrm = 1.0;
  for (int j = k - 1; j > 0; --j) {
    const double s = ((th - al[j]) * s1 - (j + 1 < k ? be[j] * s2 : 0.0)) / be[j - 1];
    s2 = s1;
    s1 = s;
    nrm = fma(s, s, nrm);
    if (nrm > 1e200) break;  // the last component is below 1e-100
  }
  *theta = th;
  *last = rsqrt(nrm);
}

// per operator: V (n x (KMAX + 1)), z, w (n), coef (2 KMAX), part (cs)
__global__ void __launch_bounds__(T, 2) k_lanczos_sigma(const cxd* LU, const cxd* Linv, const cxd* Uinv, const int* perm,
                                                        const int* info, int n, int nblk, cxd* work, size_t per,
                                                        double tol, double* sig) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  __shared__ cxd xs[128], red[192];
  __shared__ double al[KMAX], be[KMAX], nr[T / 32], sres[2];
  Op o;
  o.cs = (int)cl.num_blocks();
  o.rank = (int)cl.block_rank();
  const int mat = blockIdx.x / o.cs;
  o.A = LU + (size_t)mat * n * n;
  o.Linv = Linv + (size_t)mat * nblk * NB * NB;
  o.Uinv = Uinv + (size_t)mat * nblk * NB * NB;
  o.perm = perm + (size_t)mat * n;
  o.n = n;
  o.nblk = nblk;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  if (info[mat] > 0) {  // no pivot (the whole cluster leaves): sigma_min = 0 at an exact zero, else the column is NaN
    const cxd u = o.A[(size_t)(info[mat] - 1) * (n + 1)];
    if (o.rank == 0 && tid == 0)
      sig[mat] = u.re == 0.0 && u.im == 0.0 ? 0.0 : __longlong_as_double(0x7FF8000000000000ll);
    return;
  }
  cxd* V = work + (size_t)mat * per;
  cxd* z = V + (size_t)n * (KMAX + 1);
  cxd* w = z + n;
  cxd* coef = w + n;
  double* part = reinterpret_cast<double*>(coef + 2 * KMAX);
  // the rows this CTA owns in the vector operations
  const int per_cta = (n + o.cs - 1) / o.cs, r0 = min(n, o.rank * per_cta), r1 = min(n, r0 + per_cta);
  // |u|^2 over the cluster, u given by rows r0 .. r1 - 1
  auto norm2 = [&](const cxd* u) {
    double s = 0.0;
    for (int r = r0 + tid; r < r1; r += T) s += cabs2(u[r]);
#pragma unroll
    for (int q = 16; q > 0; q >>= 1) s += __shfl_xor_sync(0xffffffffu, s, q);
    if (lane == 0) nr[wid] = s;
    __syncthreads();
    if (tid == 0) {
      double t = 0.0;
      for (int q = 0; q < T / 32; ++q) t += nr[q];
      part[o.rank] = t;
    }
    cl.sync();
    double t = 0.0;
    for (int q = 0; q < o.cs; ++q) t += part[q];
    return t;
  };
  for (int r = r0 + tid; r < r1; r += T) w[r] = cxd(fillv(r, 0, 11), fillv(r, 1, 11));
  __syncthreads();
  double beta = sqrt(norm2(w)), theta = 0.0;
  const int kmax = min(KMAX, n);
  for (int k = 0; k < kmax; ++k) {
    cxd* v = V + (size_t)k * n;
    const double ib = 1.0 / beta;
    for (int r = r0 + tid; r < r1; r += T) v[r] = w[r] * ib;
    cl.sync();
    for (int r = r0 + tid; r < r1; r += T) z[r] = v[o.perm[r]];  // P v
    cl.sync();
    sweep<0>(o, z, xs, red);
    sweep<1>(o, z, xs, red);
    sweep<2>(o, z, xs, red);
    sweep<3>(o, z, xs, red);
    for (int r = r0 + tid; r < r1; r += T) w[o.perm[r]] = z[r];  // P^T z
    cl.sync();
    // w -= V (V^H w), twice; alpha = v^H w
    double alpha = 0.0;
    for (int pass = 0; pass < 2; ++pass) {
      cxd* cf = coef + pass * KMAX;
      for (int q = o.rank * (T / 32) + wid; q <= k; q += o.cs * (T / 32)) {
        const cxd* vq = V + (size_t)q * n;
        cxd s(0.0, 0.0);
        for (int r = lane; r < n; r += 32) cfma(s, conj(vq[r]), w[r]);
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
          s.re += __shfl_xor_sync(0xffffffffu, s.re, d);
          s.im += __shfl_xor_sync(0xffffffffu, s.im, d);
        }
        if (lane == 0) cf[q] = s;
      }
      cl.sync();
      alpha += cf[k].re;
      for (int r = r0 + tid; r < r1; r += T) {
        cxd y = w[r];
        for (int q = 0; q <= k; ++q) cfms(y, V[(size_t)q * n + r], cf[q]);
        w[r] = y;
      }
      cl.sync();
    }
    beta = sqrt(norm2(w));
    if (tid == 0) {
      al[k] = alpha;
      be[k] = beta;
    }
    __syncthreads();
    const bool end = k + 1 == kmax || !(beta > 0.0) || !isfinite(alpha) || !isfinite(beta);
    if (end || k % 3 == 2) {
      if (tid == 0) tridiag_top(al, be, k + 1, &sres[0], &sres[1]);
      __syncthreads();
      theta = sres[0];
      // every CTA of the cluster holds the same al, be and takes the same exit
      if (end || !(beta * sres[1] > tol * theta)) break;
    }
  }
  // a NaN here (an infinite entry of A) stays one: 0 is the answer of a singular operator
  if (o.rank == 0 && tid == 0) sig[mat] = 1.0 / sqrt(theta);
}

}  // namespace lz

}  // namespace

int Dense64::create(int n_, int batch_, cudaStream_t st_) {
  cxd* A = nullptr;
  st = st_;
  QBG_TRY(alloc(&A, sizeof(cxd) * (size_t)n_ * n_ * batch_));
  return bind(A, n_, batch_, st_);
}

int Dense64::bind(cxd* A, int n_, int batch_, cudaStream_t st_) {
  n = n_;
  batch = batch_;
  st = st_;
  f = LUBatch<double>();
  f.n = n;
  f.batch = batch;
  f.nb = 64;
  f.nblk = (n + f.nb - 1) / f.nb;
  f.stride = (long long)n * n;
  f.A = A;
  QBG_TRY(alloc(&f.ipiv, sizeof(int) * (size_t)n * batch));
  QBG_TRY(alloc(&f.perm, sizeof(int) * (size_t)n * batch));
  QBG_TRY(alloc(&f.info, sizeof(int) * batch));
  QBG_TRY(alloc(&f.Linv, sizeof(cxd) * (size_t)f.nblk * f.nb * f.nb * batch));
  QBG_TRY(alloc(&f.Uinv, sizeof(cxd) * (size_t)f.nblk * f.nb * f.nb * batch));
  return QBG_OK;
}

int Dense64::factor(std::vector<int>* info_host) {
  QBG_TRY(lu_factor<double>(f, st));
  if (!info_host) return QBG_OK;
  info_host->assign(batch, 0);
  QBG_CUDA(cudaMemcpyAsync(info_host->data(), f.info, sizeof(int) * batch, cudaMemcpyDeviceToHost, st));
  return tc_check(st);  // waits for the stream; a product that gave up left its output unwritten
}

void Dense64::release() {
  if (st && !mem.empty()) cudaStreamSynchronize(st);
  for (void* q : mem) dfree(q, st);
  mem.clear();
}

Dense64::~Dense64() { release(); }

namespace {
// one CTA: modified Gram-Schmidt, each column projected twice against the
// earlier ones; a column that vanishes (below 1e-14 of its length) is refilled
__global__ void __launch_bounds__(256) k_orth_mgs2(cxd* Q, int n, int p) {
  __shared__ double sh[8 * 2];
  const int tid = threadIdx.x;
  for (int j = 0; j < p; ++j) {
    cxd* qj = Q + (size_t)j * n;
    for (int attempt = 0; attempt < 3; ++attempt) {
      double v0[1] = {0.0};
      for (int r = tid; r < n; r += 256) v0[0] += cabs2(qj[r]);
      block_sum<1>(v0, sh);
      for (int pass = 0; pass < 2; ++pass)
        for (int i = 0; i < j; ++i) {
          const cxd* qi = Q + (size_t)i * n;
          double c[2] = {0.0, 0.0};
          for (int r = tid; r < n; r += 256) {
            const cxd a = qi[r], y = qj[r];
            c[0] += a.re * y.re + a.im * y.im;
            c[1] += a.re * y.im - a.im * y.re;
          }
          block_sum<2>(c, sh);
          for (int r = tid; r < n; r += 256) {
            cxd y = qj[r];
            cfms(y, qi[r], cxd(c[0], c[1]));
            qj[r] = y;
          }
        }
      double v1[1] = {0.0};
      for (int r = tid; r < n; r += 256) v1[0] += cabs2(qj[r]);
      block_sum<1>(v1, sh);
      const double n1 = sqrt(v1[0]);
      if (n1 > 1e-14 * sqrt(v0[0]) && n1 > 1e-300 && isfinite(n1)) {
        const double s = 1.0 / n1;
        for (int r = tid; r < n; r += 256) qj[r] = qj[r] * s;
        break;
      }
      for (int r = tid; r < n; r += 256) qj[r] = cxd(fillv(r, j, 97 + attempt), fillv(r, j + p, 97 + attempt));
      __syncthreads();
    }
    __syncthreads();
  }
}
}  // namespace

int orth_columns(cxd* Q, int n, int p, cudaStream_t st) {
  k_orth_mgs2<<<1, 256, 0, st>>>(Q, n, p);
  QBG_LAUNCH_CHECK("k_orth_mgs2");
  return QBG_OK;
}

int sigma_iterate(const cxd* Cinv, int n, int batch, const cxd* X0, cxd* work, int maxit, double tol, double* sig,
                  int* iters, cxd* vec, cudaStream_t st) {
  if (batch < 1) return QBG_OK;
  k_sigma_iter<<<batch, 256, 0, st>>>(Cinv, n, X0, work, maxit, tol, sig, iters, vec);
  QBG_LAUNCH_CHECK("k_sigma_iter");
  return QBG_OK;
}

size_t sigma_lu_work(int n) {
  // V, z, w, coefficients and the partial norms of one operator, in complex words
  return ((size_t)n * (lz::KMAX + 3) + 2 * lz::KMAX + 8 + 15) / 16 * 16;
}

int sigma_lu(const LUBatch<double>& f, cxd* work, double tol, double* sig, cudaStream_t st) {
  if (f.batch < 1) return QBG_OK;
  if (f.nb != lz::NB || f.levels != 0) {
    set_error("sigma_lu: needs 64-row diagonal blocks");
    return QBG_EINVAL;
  }
  // CTAs per operator: about two per SM over the batch, at most one per block
  // row. The sweeps' block chains shorten little beyond that, while every step
  // is a cluster barrier. 8 is the portable limit.
  int cs = 1;
  while (cs < 8 && (long long)f.batch * cs < 304 && cs < f.nblk) cs *= 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(f.batch * cs), 1, 1);
  cfg.blockDim = dim3(lz::T, 1, 1);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = cs;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  QBG_CUDA(cudaLaunchKernelEx(&cfg, lz::k_lanczos_sigma, (const cxd*)f.A, (const cxd*)f.Linv, (const cxd*)f.Uinv,
                              (const int*)f.perm, (const int*)f.info, f.n, f.nblk, work, sigma_lu_work(f.n), tol, sig));
  QBG_LAUNCH_CHECK("k_lanczos_sigma");
  return QBG_OK;
}

void dense_start_block(int n, std::vector<cxd>& hx) {
  // fixed (reproducible) start block: entries of a 64-bit LCG in [-1, 1)
  hx.resize((size_t)n * DENSE_P);
  unsigned long long lcg = 0x9E3779B97F4A7C15ull;
  auto nxt = [&]() {
    lcg = lcg * 6364136223846793005ull + 1442695040888963407ull;
    return (double)(lcg >> 11) * (2.0 / 9007199254740992.0) - 1.0;
  };
  for (auto& v : hx) {
    v.re = nxt();
    v.im = nxt();
  }
}

int rr_step(const cxd* W, int n, double tol, double* state, cudaStream_t st) {
  k_rr_step<<<1, 256, 0, st>>>(W, n, tol, state);
  QBG_LAUNCH_CHECK("k_rr_step");
  return QBG_OK;
}

int orth8(cxd* Y, int n, int salt, cudaStream_t st) {
  k_orth8<<<1, 256, 0, st>>>(Y, n, salt);
  QBG_LAUNCH_CHECK("k_orth8");
  return QBG_OK;
}

int topvec(const cxd* W, const double* state, int n, cxd* x, cudaStream_t st) {
  k_topvec<<<1, 256, 0, st>>>(W, state, n, x);
  QBG_LAUNCH_CHECK("k_topvec");
  return QBG_OK;
}

int sigma_single(const cxd* Cinv, cxd* CH, int n, const cxd* X0, cxd* X, cxd* W, cxd* Y, cxd* P, double* state,
                 int maxit, double tol, double* sig, cxd* x_out, cudaStream_t st) {
  QBG_TRY(conj_transpose(Cinv, CH, n, st));
  QBG_CUDA(cudaMemcpyAsync(X, X0, sizeof(cxd) * (size_t)n * DENSE_P, cudaMemcpyDeviceToDevice, st));
  QBG_TRY(orth8(X, n, 0, st));
  static const double init[2] = {-1.0, 0.0};
  QBG_CUDA(cudaMemcpyAsync(state, init, sizeof(init), cudaMemcpyHostToDevice, st));
  double h[2] = {0.0, 0.0};
  for (int it = 0; it < maxit; ++it) {
    QBG_TRY(gemm_tall(Cinv, X, W, n, DENSE_P, P, st));
    // the Rayleigh-Ritz step only tests convergence (the iteration itself is
    // X <- orth(C^H C X)): every fourth step, always before the host reads the
    // state, so the estimate and the Ritz vector belong to the last W
    const bool check = (it % 8 == 7) || it + 1 == maxit;
    if (check || it % 4 == 3) QBG_TRY(rr_step(W, n, tol, state, st));
    if (check) {
      QBG_CUDA(cudaMemcpyAsync(h, state, sizeof(h), cudaMemcpyDeviceToHost, st));
      QBG_CUDA(cudaStreamSynchronize(st));
      if (h[1] != 0.0 || it + 1 == maxit) break;
    }
    QBG_TRY(gemm_tall(CH, W, Y, n, DENSE_P, P, st));
    QBG_TRY(orth8(Y, n, 8 * (it + 1), st));
    cxd* t = X;
    X = Y;
    Y = t;
  }
  *sig = h[0];
  if (x_out) QBG_TRY(topvec(W, state, n, x_out, st));
  return QBG_OK;
}

int deflate_shift(const cxd* G, const cxd* x, int n, double lam, double mu, cxd* M, cudaStream_t st) {
  k_deflate_shift<<<2048, 256, 0, st>>>(G, x, n, lam, mu, M);
  QBG_LAUNCH_CHECK("k_deflate_shift");
  return QBG_OK;
}

}  // namespace qbg
