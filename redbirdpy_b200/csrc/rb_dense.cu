// Dense FP64 pieces of the Gauss-Newton step (reginvunder,
// redbirdpy/recon.py:429-509 and _normalize_diag, recon.py:784-789):
//   H += lambda I, di = 1/sqrt(|diag H| + 1e-16), H <- di H di     (prepare)
//   H = L L^T, blocked right-looking Cholesky (64-wide panels; the
//   inverse of each diagonal block kept in its strict upper triangle)  (cholesky)
//   L L^T x = b                                                    (chol_solve)
//   out = alpha * J^T y   (J FP32 M x K rows, y FP64)              (gemv_t)
//   sum(J^2)              (Frobenius block scaling, recon.py:235)   (sumsq)
#include <algorithm>
#include <mutex>

#include <cuda_bf16.h>

#include "rb_common.cuh"
#include "rb_tc.cuh"

namespace rb {

constexpr int kNB = 64;  // panel width

__global__ void prep_diag_kernel(double* __restrict__ H, int64_t M, int64_t ldh, double lam, double* __restrict__ di) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= M) return;
  const double d = H[i * ldh + i] + lam;
  H[i * ldh + i] = d;
  di[i] = 1.0 / sqrt(fabs(d) + 1e-16);
}

__global__ void prep_scale_kernel(double* __restrict__ H, int64_t M, int64_t ldh, const double* __restrict__ di) {
  const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t i = blockIdx.y;
  if (j >= M) return;
  H[i * ldh + j] *= di[i] * di[j];
}

// Factor the nb x nb diagonal block at (j0, j0) (lower, L11) and form its
// inverse X = L11^-1, stored transposed in the block's strict upper triangle:
// H[j0 + j][j0 + i] = X[i][j], i > j (the diagonal of X is 1 / L[i][i]).  The
// panel solve and rb_chol_solve then apply X as a product.
//
// One block of 256 threads; the bound is the chain of 64 pivots.  It runs in
// four steps of 16 columns, so that only a 16 x 16 block's pivots are serial:
// one warp factors it in registers (lane = row; a pivot's reciprocal root and
// one row exchange per column, no barrier) and inverts it, then all threads
// apply that inverse to the rows below (16-term products) and update the rest
// of the triangle (16-term products, 2 x 2 entries per thread).  X is put
// together from the four 16 x 16 inverses by block products.  Rows beyond nb
// are padded with the identity.  (Two columns per barrier pair over the whole
// block, and the inverse by a chain of 64 substitution steps, took 63.6 us per
// block in an M = 8192 factorisation, now 38, 24 where no update shares its SM;
// 128 of them are on the critical path.)
constexpr int kPB = 16;
__global__ void __launch_bounds__(256) potrf_diag_kernel(double* __restrict__ H, int64_t ldh, int64_t j0, int nb,
                                                         int* __restrict__ err) {
  __shared__ double Ls[kNB][kNB + 1];  // the block, then L
  extern __shared__ double psm[];
  double(*Xs)[kNB + 1] = reinterpret_cast<double(*)[kNB + 1]>(psm);           // X (lower)
  double(*Ts)[kPB + 1] = reinterpret_cast<double(*)[kPB + 1]>(psm + kNB * (kNB + 1));  // 3 x 16 x 16 products
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  double in[kNB * kNB / 256];  // every load under way before the first is used
#pragma unroll
  for (int v = 0; v < kNB * kNB / 256; ++v) {
    const int i = (tid + 256 * v) / kNB, j = tid % kNB;
    in[v] = (i < nb && j <= i) ? H[(j0 + i) * ldh + j0 + j] : (i == j ? 1.0 : 0.0);
  }
#pragma unroll
  for (int v = 0; v < kNB * kNB / 256; ++v) {
    const int i = (tid + 256 * v) / kNB, j = tid % kNB;
    Ls[i][j] = in[v];
    Xs[i][j] = 0.0;
  }
  __syncthreads();
#pragma unroll 1
  for (int kb = 0; kb < kNB; kb += kPB) {
    if (w == 0) {  // lanes 16..31 repeat lanes 0..15
      const int l = lane & (kPB - 1);
      double r[kPB], x[kPB], ri = 1.0;
#pragma unroll
      for (int c = 0; c < kPB; ++c) r[c] = Ls[kb + l][kb + c];
#pragma unroll
      for (int c = 0; c < kPB; ++c) {
        const double d = __shfl_sync(0xffffffffu, r[c], c);
        const bool ok = d > 0.0 && isfinite(d);
        const double rp = ok ? rsqrt(d) : 1.0;
        if (lane == 0 && !ok && kb + c < nb) atomicCAS(err, 0, (int)(j0 + kb + c) + 1);
        const double lc = l == c ? (ok ? d * rp : 1.0) : r[c] * rp;
        r[c] = lc;
#pragma unroll
        for (int j = c + 1; j < kPB; ++j) r[j] = fma(-lc, __shfl_sync(0xffffffffu, lc, j), r[j]);
      }
      if (lane < kPB) {
#pragma unroll
        for (int c = 0; c < kPB; ++c)
          if (c <= l) Ls[kb + l][kb + c] = r[c];
      }
      // column l of the inverse by substitution; 1 / L[i][i] = ri of lane i
#pragma unroll
      for (int c = 0; c < kPB; ++c)
        if (c == l) ri = r[c];
      ri = 1.0 / ri;
#pragma unroll
      for (int i = 0; i < kPB; ++i) {
        double s0 = 0.0, s1 = 0.0;
#pragma unroll
        for (int k = 0; k < i; ++k) {
          const double lik = __shfl_sync(0xffffffffu, r[k], i);
          if (k & 1) s1 = fma(lik, x[k], s1);
          else s0 = fma(lik, x[k], s0);
        }
        const double rii = __shfl_sync(0xffffffffu, ri, i);
        x[i] = i < l ? 0.0 : i == l ? rii : -(s0 + s1) * rii;
      }
      if (lane < kPB) {
#pragma unroll
        for (int i = 0; i < kPB; ++i) Xs[kb + i][kb + l] = x[i];
      }
    }
    __syncthreads();
    const int m0 = kb + kPB, mr = kNB - m0;  // rows below
    // L21 = A21 X11^T: thread = (row, 4 columns)
    for (int e = tid; e < mr * 4; e += 256) {
      const int i = m0 + (e >> 2), c0 = (e & 3) * 4;
      double a[kPB], o[4];
#pragma unroll
      for (int t = 0; t < kPB; ++t) a[t] = Ls[i][kb + t];
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        double s0 = 0.0, s1 = 0.0;
#pragma unroll
        for (int t = 0; t < kPB; t += 2) {
          s0 = fma(a[t], Xs[kb + c0 + v][kb + t], s0);
          s1 = fma(a[t + 1], Xs[kb + c0 + v][kb + t + 1], s1);
        }
        o[v] = s0 + s1;
      }
      __syncwarp();  // the four threads of a row have read it (whole warps: mr * 4 is a multiple of 32)
#pragma unroll
      for (int v = 0; v < 4; ++v) Ls[i][kb + c0 + v] = o[v];
    }
    __syncthreads();
    // the rest of the triangle, 2 x 2 entries per thread
    const int h = mr / 2;
    for (int e = tid; e < h * (h + 1) / 2; e += 256) {
      int bi = (int)((sqrtf(8.f * (float)e + 1.f) - 1.f) * 0.5f);
      while (bi * (bi + 1) / 2 > e) --bi;
      while ((bi + 1) * (bi + 2) / 2 <= e) ++bi;
      const int i = m0 + 2 * bi, j = m0 + 2 * (e - bi * (bi + 1) / 2);
      double s00 = Ls[i][j], s01 = Ls[i][j + 1], s10 = Ls[i + 1][j], s11 = Ls[i + 1][j + 1];
#pragma unroll
      for (int t = 0; t < kPB; ++t) {
        const double a0 = Ls[i][kb + t], a1 = Ls[i + 1][kb + t], b0 = Ls[j][kb + t], b1 = Ls[j + 1][kb + t];
        s00 = fma(-a0, b0, s00);
        s01 = fma(-a0, b1, s01);
        s10 = fma(-a1, b0, s10);
        s11 = fma(-a1, b1, s11);
      }
      Ls[i][j] = s00;
      if (j + 1 <= i) Ls[i][j + 1] = s01;
      Ls[i + 1][j] = s10;
      Ls[i + 1][j + 1] = s11;
    }
    __syncthreads();
  }
  for (int e = tid; e < kNB * kNB; e += 256) {
    const int i = e / kNB, j = e % kNB;
    if (i < nb && j <= i) H[(j0 + i) * ldh + j0 + j] = Ls[i][j];
  }
  // X below its diagonal blocks, one block diagonal after the other:
  // X_pq = -X_pp sum_{q <= k < p} L_pk X_kq; thread = one entry of a block
  const int bi = tid >> 4, bj = tid & 15;
#pragma unroll 1
  for (int dgl = 1; dgl < kNB / kPB; ++dgl) {
    for (int q = 0; q + dgl < kNB / kPB; ++q) {
      const int p = q + dgl;
      double s0 = 0.0, s1 = 0.0;
      for (int k = q; k < p; ++k)
#pragma unroll
        for (int t = 0; t < kPB; t += 2) {
          s0 = fma(Ls[p * kPB + bi][k * kPB + t], Xs[k * kPB + t][q * kPB + bj], s0);
          s1 = fma(Ls[p * kPB + bi][k * kPB + t + 1], Xs[k * kPB + t + 1][q * kPB + bj], s1);
        }
      Ts[q * kPB + bi][bj] = s0 + s1;
    }
    __syncthreads();
    for (int q = 0; q + dgl < kNB / kPB; ++q) {
      const int p = q + dgl;
      double s0 = 0.0, s1 = 0.0;
#pragma unroll
      for (int t = 0; t < kPB; t += 2) {
        s0 = fma(Xs[p * kPB + bi][p * kPB + t], Ts[q * kPB + t][bj], s0);
        s1 = fma(Xs[p * kPB + bi][p * kPB + t + 1], Ts[q * kPB + t + 1][bj], s1);
      }
      Xs[p * kPB + bi][q * kPB + bj] = -(s0 + s1);
    }
    __syncthreads();
  }
  for (int e = tid; e < kNB * kNB; e += 256) {
    const int j = e / kNB, i = e % kNB;
    if (i > j && i < nb) H[(j0 + j) * ldh + j0 + i] = Xs[i][j];
  }
}
constexpr int kPotrfSmem = (kNB * (kNB + 1) + 3 * kPB * (kPB + 1)) * (int)sizeof(double);

// X^T of a factored diagonal block in shared memory: Xt[t][c] = X[c][t]
// (t <= c; H's strict upper triangle of the block, 1 / L[c][c] on the
// diagonal, zero below)
__device__ __forceinline__ void load_inv_t(const double* __restrict__ H, int64_t ldh, int64_t j0, int nb,
                                           double (*Xt)[kNB + 1]) {
  for (int e = threadIdx.x; e < kNB * kNB; e += blockDim.x) {
    const int t = e / kNB, c = e % kNB;
    double v = 0.0;
    if (t < nb && c < nb) {
      if (c > t) v = H[(j0 + t) * ldh + j0 + c];
      else if (c == t) v = 1.0 / H[(j0 + t) * ldh + j0 + t];
    }
    Xt[t][c] = v;
  }
}

// L21 = A21 L11^-T = A21 X^T for the rows below the panel: a CTA takes 64
// rows (4 x 4 outputs per thread), sums t = 0..c in order, and writes its
// rows back in place
constexpr int kTrsmSmem = 2 * kNB * (kNB + 1) * (int)sizeof(double);  // dynamic: above the 48 KB static limit
__global__ void __launch_bounds__(256) trsm_panel_kernel(double* __restrict__ H, int64_t ldh, int64_t M, int64_t j0,
                                                         int nb) {
  extern __shared__ double tsm[];
  double(*Xt)[kNB + 1] = reinterpret_cast<double(*)[kNB + 1]>(tsm);
  double(*As)[kNB + 1] = Xt + kNB;
  const int tid = threadIdx.x;
  const int64_t r0 = j0 + nb + blockIdx.x * (int64_t)kNB;
  load_inv_t(H, ldh, j0, nb, Xt);
  for (int e = tid; e < kNB * kNB; e += blockDim.x) {
    const int i = e / kNB, t = e % kNB;
    As[i][t] = (r0 + i < M && t < nb) ? H[(r0 + i) * ldh + j0 + t] : 0.0;
  }
  __syncthreads();
  const int tr = (tid >> 4) * 4, tc = (tid & 15) * 4;
  double acc[4][4];
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int v = 0; v < 4; ++v) acc[u][v] = 0.0;
  const int tmax = min(nb, tc + 4);
  for (int t = 0; t < tmax; ++t) {
    double xa[4], xb[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) xa[u] = As[tr + u][t];
#pragma unroll
    for (int v = 0; v < 4; ++v) xb[v] = Xt[t][tc + v];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int v = 0; v < 4; ++v) acc[u][v] = fma(xa[u], xb[v], acc[u][v]);
  }
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const int64_t r = r0 + tr + u;
      const int c = tc + v;
      if (r < M && c < nb) H[r * ldh + j0 + c] = acc[u][v];
    }
}

// trailing update A22 -= L21 L21^T on 64 x 64 tiles of the lower triangle,
// on the FP64 tensor cores (mma.sync m8n8k4 .f64: D = A B + C, every
// product and sum in FP64).  128 threads: warp w owns the 32 x 32 quarter
// (w / 2, w % 2) of the tile as 4 x 4 MMA tiles of 8 x 8.  The panel's rows
// stream through shared memory in 32-column stages, double-buffered with
// cp.async (16-byte copies when every row start is 16-byte aligned, else
// 8-byte copies), rows kept k-contiguous with a stride of 36 doubles so that
// the fragment loads (8 rows x 4 k per warp) take the minimum two
// wavefronts.  Rows past M are zero-filled by the copy (source size 0).
// The panel is columns j0 .. j0 + nb; the tiles start at row and column s0
// and reach columns below c_end only.  With tri = 0 (a band of columns) the
// grid is 2-D, x the row tile and y the column tile, and tiles above the
// diagonal return at once; with tri = 1 (a whole trailing triangle)
// blockIdx.x enumerates the lower tiles.
constexpr int kSyrkThreads = 128;
constexpr int kSyK = 32;             // panel columns per stage
constexpr int kSyLd = kSyK + 4;      // shared row stride (doubles)
constexpr int kSyrkSmem = 2 * 2 * kNB * kSyLd * (int)sizeof(double);  // 2 stages x (A, B): 73,728 bytes

__device__ __forceinline__ void cp_async_f64(uint32_t dst, const double* src, int bytes, int src_bytes) {
  if (bytes == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ void dmma_8x8x4(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

// one stage of the panel: rows r0.. (A) and c0.. (B), columns kk.. of the
// panel (kc of them), into the shared buffers
template <int CH>
__device__ __forceinline__ void syrk_stage(const double* __restrict__ H, int64_t ldh, int64_t M, int64_t r0,
                                           int64_t c0, int64_t kcol, int kc, double* As, double* Bs) {
  constexpr int PER = kSyK * (int)sizeof(double) / CH;  // copies per row
  for (int e = threadIdx.x; e < 2 * kNB * PER; e += kSyrkThreads) {
    const int m = e / (kNB * PER), rem = e % (kNB * PER);
    const int i = rem / PER, kq = (rem % PER) * (CH / (int)sizeof(double));
    const int64_t row = (m == 0 ? r0 : c0) + i;
    const bool in = row < M && kq < kc;
    const double* src = in ? H + row * ldh + kcol + kq : H;
    double* dst = (m == 0 ? As : Bs) + i * kSyLd + kq;
    cp_async_f64(smem_u32(dst), src, CH, in ? min(CH, (kc - kq) * (int)sizeof(double)) : 0);
  }
}

template <int CH>
__global__ void __launch_bounds__(kSyrkThreads) syrk_update_kernel(double* __restrict__ H, int64_t ldh, int64_t M,
                                                                   int64_t j0, int nb, int64_t s0, int64_t c_end,
                                                                   int tri) {
  extern __shared__ __align__(16) double sy[];
  int64_t ti, tj;  // tile (ti, tj) covers rows s0 + 64 ti .., columns s0 + 64 tj ..
  if (!tri) {
    ti = blockIdx.x;
    tj = blockIdx.y;
    if (tj > ti) return;
  } else {
    // blockIdx.x enumerates lower tiles (ti >= tj) in row-major order
    int64_t t = blockIdx.x;
    ti = 0;
    while (t > ti) {
      t -= ti + 1;
      ++ti;
    }
    tj = t;
  }
  const int64_t r0 = s0 + ti * kNB, c0 = s0 + tj * kNB;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int wm = (w >> 1) * 32, wn = (w & 1) * 32;
  const int g = lane >> 2, t4 = lane & 3;
  double acc[4][4][2];
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int n = 0; n < 4; ++n) acc[m][n][0] = acc[m][n][1] = 0.0;
  const int nst = (nb + kSyK - 1) / kSyK;
  auto bufA = [&](int s) { return sy + (s & 1) * 2 * kNB * kSyLd; };
  auto bufB = [&](int s) { return sy + (s & 1) * 2 * kNB * kSyLd + kNB * kSyLd; };
  syrk_stage<CH>(H, ldh, M, r0, c0, j0, min(kSyK, nb), bufA(0), bufB(0));
  cp_async_commit();
  for (int s = 0; s < nst; ++s) {
    if (s + 1 < nst) {
      syrk_stage<CH>(H, ldh, M, r0, c0, j0 + (int64_t)(s + 1) * kSyK, min(kSyK, nb - (s + 1) * kSyK), bufA(s + 1),
                     bufB(s + 1));
      cp_async_commit();
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    const double* A = bufA(s) + (wm + g) * kSyLd + t4;
    const double* B = bufB(s) + (wn + g) * kSyLd + t4;
#pragma unroll
    for (int ks = 0; ks < kSyK; ks += 4) {
      double a[4], b[4];
#pragma unroll
      for (int m = 0; m < 4; ++m) a[m] = A[m * 8 * kSyLd + ks];
#pragma unroll
      for (int n = 0; n < 4; ++n) b[n] = B[n * 8 * kSyLd + ks];
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int n = 0; n < 4; ++n) dmma_8x8x4(acc[m][n][0], acc[m][n][1], a[m], b[n]);
    }
    __syncthreads();  // the buffer is refilled by the stage after next
  }
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int64_t i = r0 + wm + m * 8 + g, j = c0 + wn + n * 8 + 2 * t4 + h;
        if (i < M && j < c_end && j <= i) H[i * ldh + j] -= acc[m][n][h];
      }
}

// L L^T x = b in one launch: a block of threads per 64-row block row (block
// rows dealt round robin when there are more than resident blocks), forward in
// ascending and then backward in descending order, so that every block only
// waits for block rows that come earlier in its own order.  A solved segment
// is handed on through global memory: its words start as kEmpty and a reader
// polls the values themselves (one round trip through L2 instead of a flag and
// then the data; a computed NaN is stored with another payload).  A thread
// loads the next tile of L before it waits for the segment that multiplies it,
// so per 64 rows the chain is one hand-over, a 64-term product, a quad
// reduction and the product with the block's inverse.  One launch per block
// row and direction before: 1024 launches of 8-11 us for the four solves of a
// refined M = 8192 step, 2.36 ms per solve, now 0.43 ms (M = 8192).  Waits are bounded;
// one that gives up ends its block with NaN in its segment and sets the word
// that rb_chol_solve_status reads.
constexpr unsigned long long kEmpty = ~0ull;
constexpr int kTrsvSpins = 1 << 20;  // about a second
__device__ int g_trsv_err;

__device__ __forceinline__ double2 ld_seg(const double* p) {
  double2 v;
  asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_seg(double* p, double v) {
  if (isnan(v)) v = __longlong_as_double(0x7ff8000000000000LL);
  asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}
__device__ __forceinline__ bool seg_empty(double v) { return (unsigned long long)__double_as_longlong(v) == kEmpty; }

// 8 pairs of a segment at p + stride u; false when they do not arrive
template <int STRIDE>
__device__ __forceinline__ bool wait_seg(const double* p, double2 (&v)[8], const volatile int& bad) {
  for (int spin = 0; spin < kTrsvSpins; ++spin) {
    bool ok = true;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      v[u] = ld_seg(p + STRIDE * u);
      ok = ok && !seg_empty(v[u].x) && !seg_empty(v[u].y);
    }
    if (ok) return true;
    if (spin > 256) {
      if (bad) return false;  // (the block has given up already)
      __nanosleep(64);
    }
  }
  return false;
}

// y, x: segments of ceil(M / 64) x 64 words, all kEmpty at launch; xio: b on
// entry, the solution on return
__global__ void __launch_bounds__(256, 1) chol_solve_kernel(const double* __restrict__ L, int64_t ldh, int64_t M,
                                                            double* __restrict__ xio, double* __restrict__ y,
                                                            double* __restrict__ x) {
  __shared__ double t[kNB], part[4][kNB];
  __shared__ int bad;
  const int tid = threadIdx.x;
  const int64_t nblk = (M + kNB - 1) / kNB;
  if (tid == 0) bad = 0;
  __syncthreads();
  // ---- L y = b: thread (r, q) sums columns 8 u + 2 q, + 1 of row r
  {
    const int r = tid >> 2, q = tid & 3;
    for (int64_t j = blockIdx.x; j < nblk; j += gridDim.x) {
      const int64_t j0 = j * kNB, row = j0 + r;
      const int nb = (int)min((int64_t)kNB, M - j0);
      const bool on = r < nb;
      // the inverse's row r: X[r][c] at (c, r), c < r; 1 / L[r][r]
      double xi[16];
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        const int c = 8 * (u >> 1) + 2 * q + (u & 1);
        xi[u] = !on || c > r ? 0.0 : c == r ? 1.0 / L[row * ldh + row] : L[(j0 + c) * ldh + row];
      }
      const double* Lr = L + (on ? row : j0) * ldh + 2 * q;
      double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0, lt[16];
      auto tile = [&](int64_t i) {
#pragma unroll
        for (int u = 0; u < 16; ++u) lt[u] = Lr[i * kNB + 8 * (u >> 1) + (u & 1)];
      };
      if (j > 0) tile(0);
      for (int64_t i = 0; i < j; ++i) {
        double c[16];
#pragma unroll
        for (int u = 0; u < 16; ++u) c[u] = lt[u];
        if (i + 1 < j) tile(i + 1);
        double2 v[8];
        if (!wait_seg<8>(y + i * kNB + 2 * q, v, bad)) bad = 1;
#pragma unroll
        for (int u = 0; u < 8; u += 2) {
          a0 = fma(c[2 * u], v[u].x, a0);
          a1 = fma(c[2 * u + 1], v[u].y, a1);
          a2 = fma(c[2 * u + 2], v[u + 1].x, a2);
          a3 = fma(c[2 * u + 3], v[u + 1].y, a3);
        }
      }
      double s = (a0 + a1) + (a2 + a3);
      s += __shfl_xor_sync(0xffffffffu, s, 1);
      s += __shfl_xor_sync(0xffffffffu, s, 2);
      if (q == 0) t[r] = on ? xio[row] - s : 0.0;
      __syncthreads();
      double z0 = 0.0, z1 = 0.0;
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        z0 = fma(xi[2 * u], t[8 * u + 2 * q], z0);
        z1 = fma(xi[2 * u + 1], t[8 * u + 2 * q + 1], z1);
      }
      double z = z0 + z1;
      z += __shfl_xor_sync(0xffffffffu, z, 1);
      z += __shfl_xor_sync(0xffffffffu, z, 2);
      if (q == 0) st_seg(y + j0 + r, bad ? __longlong_as_double(0x7ff8000000000000LL) : z);
      __syncthreads();
    }
  }
  // ---- L^T x = y: thread (c, g) sums rows 16 g .. + 15 of column c
  {
    const int c = tid & 63, g = tid >> 6;
    const int64_t last = (nblk - 1 - blockIdx.x) / gridDim.x * gridDim.x + blockIdx.x;  // the block's last block row
    for (int64_t j = blockIdx.x < nblk ? last : -1; j >= 0; j -= gridDim.x) {
      const int64_t j0 = j * kNB;
      const int nb = (int)min((int64_t)kNB, M - j0);
      const bool on = c < nb;
      // column c of the inverse: X[r][c] at (c, r), r > c; 1 / L[c][c]
      double xi[16];
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        const int r = 16 * g + u;
        xi[u] = !on || r < c || r >= nb ? 0.0 : r == c ? 1.0 / L[(j0 + c) * ldh + j0 + c] : L[(j0 + c) * ldh + j0 + r];
      }
      const double* Lc = L + j0 + (on ? c : 0);
      double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0, lt[16];
      auto tile = [&](int64_t i) {
#pragma unroll
        for (int u = 0; u < 16; ++u) {
          const int64_t r = i * kNB + 16 * g + u;
          lt[u] = r < M ? Lc[r * ldh] : 0.0;
        }
      };
      if (j + 1 < nblk) tile(nblk - 1);
      for (int64_t i = nblk - 1; i > j; --i) {
        double l[16];
#pragma unroll
        for (int u = 0; u < 16; ++u) l[u] = lt[u];
        if (i - 1 > j) tile(i - 1);
        double2 v[8];
        if (!wait_seg<2>(x + i * kNB + 16 * g, v, bad)) bad = 1;
#pragma unroll
        for (int u = 0; u < 8; u += 2) {
          a0 = fma(l[2 * u], v[u].x, a0);
          a1 = fma(l[2 * u + 1], v[u].y, a1);
          a2 = fma(l[2 * u + 2], v[u + 1].x, a2);
          a3 = fma(l[2 * u + 3], v[u + 1].y, a3);
        }
      }
      part[g][c] = (a0 + a1) + (a2 + a3);
      __syncthreads();
      if (tid < kNB) {
        // this block row's own y (the same block solved it)
        const double yv = ld_seg(y + j0 + (tid & ~1)).x, yw = ld_seg(y + j0 + (tid & ~1)).y;
        const double s = (part[0][tid] + part[1][tid]) + (part[2][tid] + part[3][tid]);
        t[tid] = tid < nb ? ((tid & 1) ? yw : yv) - s : 0.0;
      }
      __syncthreads();
      double z0 = 0.0, z1 = 0.0;
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        z0 = fma(xi[2 * u], t[16 * g + 2 * u], z0);
        z1 = fma(xi[2 * u + 1], t[16 * g + 2 * u + 1], z1);
      }
      part[g][c] = z0 + z1;
      __syncthreads();
      if (tid < kNB) {
        double z = (part[0][tid] + part[1][tid]) + (part[2][tid] + part[3][tid]);
        if (bad) z = __longlong_as_double(0x7ff8000000000000LL);
        st_seg(x + j0 + tid, z);
        if (tid < nb) xio[j0 + tid] = z;
      }
      __syncthreads();
    }
  }
  if (tid == 0 && bad) atomicExch(&g_trsv_err, 1);
}

constexpr int kGemvSlabs = 16;

__device__ __forceinline__ double jval(float v) { return v; }
__device__ __forceinline__ double jval(__nv_bfloat16 v) { return __bfloat162float(v); }

// four consecutive entries of a row (16-byte FP32 / 8-byte BF16 loads)
__device__ __forceinline__ void ld4(const float* p, double (&v)[4]) {
  const float4 x = __ldcs(reinterpret_cast<const float4*>(p));
  v[0] = x.x;
  v[1] = x.y;
  v[2] = x.z;
  v[3] = x.w;
}
__device__ __forceinline__ void ld4(const __nv_bfloat16* p, double (&v)[4]) {
  const uint2 x = __ldcs(reinterpret_cast<const uint2*>(p));
  const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&x.x);
  const __nv_bfloat162 b = *reinterpret_cast<const __nv_bfloat162*>(&x.y);
  v[0] = __bfloat162float(a.x);
  v[1] = __bfloat162float(a.y);
  v[2] = __bfloat162float(b.x);
  v[3] = __bfloat162float(b.y);
}

// four consecutive entries of a row as FP32 (BF16 widened exactly)
__device__ __forceinline__ float4 ld4f(const float* p) { return __ldcs(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ float4 ld4f(const __nv_bfloat16* p) {
  const uint2 x = __ldcs(reinterpret_cast<const uint2*>(p));
  const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&x.x);
  const __nv_bfloat162 b = *reinterpret_cast<const __nv_bfloat162*>(&x.y);
  return make_float4(__bfloat162float(a.x), __bfloat162float(a.y), __bfloat162float(b.x), __bfloat162float(b.y));
}

// J stored as FP32 or BF16 (JT).  A thread owns 4 consecutive columns (one
// vector load per row; ldj % 4 == 0 keeps it aligned and inside the padded
// row) and sums its slab's rows in 4 interleaved partial sums per column
// (rows m = 0, 1, 2, 3 mod 4), added as (s0 + s1) + (s2 + s3).
template <typename JT>
__global__ void gemv_t_part_kernel(const JT* __restrict__ J, int64_t M, int64_t K, int64_t ldj,
                                   const double* __restrict__ y, double* __restrict__ part) {
  const int64_t k = 4 * (blockIdx.x * (int64_t)blockDim.x + threadIdx.x);
  if (k >= K) return;
  const int64_t rows = (M + gridDim.y - 1) / gridDim.y;
  const int64_t m0 = blockIdx.y * rows, m1 = min(M, m0 + rows);
  double s[4][4];
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int u = 0; u < 4; ++u) s[j][u] = 0.0;
  int64_t m = m0;
  for (; m + 3 < m1; m += 4) {
    double v[4][4];
#pragma unroll
    for (int u = 0; u < 4; ++u) ld4(J + (m + u) * ldj + k, v[u]);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const double ym = y[m + u];
#pragma unroll
      for (int j = 0; j < 4; ++j) s[j][u] = fma(v[u][j], ym, s[j][u]);
    }
  }
  for (; m < m1; ++m) {
    double v[4];
    ld4(J + m * ldj + k, v);
    const double ym = y[m];
#pragma unroll
    for (int j = 0; j < 4; ++j) s[j][0] = fma(v[j], ym, s[j][0]);
  }
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if (k + j < K) part[blockIdx.y * K + k + j] = (s[j][0] + s[j][1]) + (s[j][2] + s[j][3]);
}

__global__ void gemv_t_sum_kernel(const double* __restrict__ part, int slabs, int64_t K, double alpha, double beta,
                                  double* __restrict__ out) {
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k >= K) return;
  double s = 0.0;
  for (int b = 0; b < slabs; ++b) s += part[b * K + k];
  out[k] = alpha * s + (beta != 0.0 ? beta * out[k] : 0.0);
}

// out[m] = alpha sum_k J[m][k] x[k] + beta out[m] in two passes.  Block
// (cx, ry) takes the 1024 columns [1024 cx, 1024 cx + 1024) (4 per thread,
// one vector load per row) of kGemvNRows rows, so a warp reads whole 512-byte
// row segments and the block's rows stream side by side; each row's block
// sum (fixed-order warp and block reduction) goes to part[m][cx], and
// gemv_n_sum_kernel adds a row's parts (lane-strided, then a warp sum).
// The result is the same bits on every run.
constexpr int kGemvNRows = 16;
constexpr int kGemvNCols = 1024;
template <typename JT>
__global__ void __launch_bounds__(256) gemv_n_part_kernel(const JT* __restrict__ J, int64_t M, int64_t K, int64_t ldj,
                                                          const double* __restrict__ x, double* __restrict__ part,
                                                          int64_t nchunk) {
  __shared__ double red[kGemvNRows][8];
  const int64_t k = (int64_t)blockIdx.x * kGemvNCols + 4 * threadIdx.x;
  const int64_t m0 = (int64_t)blockIdx.y * kGemvNRows;
  double xv[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) xv[j] = (k + j < K) ? x[k + j] : 0.0;
  // every row's load is issued before the first product
  float4 v[kGemvNRows];
#pragma unroll
  for (int r = 0; r < kGemvNRows; ++r)
    v[r] = (k < K && m0 + r < M) ? ld4f(J + (m0 + r) * ldj + k) : make_float4(0.f, 0.f, 0.f, 0.f);
  if (k + 3 >= K) {  // the padded row's entries past K are dropped (they may hold anything)
#pragma unroll
    for (int r = 0; r < kGemvNRows; ++r) {
      if (k + 1 >= K) v[r].y = 0.f;
      if (k + 2 >= K) v[r].z = 0.f;
      if (k + 3 >= K) v[r].w = 0.f;
    }
  }
  double s[kGemvNRows];
#pragma unroll
  for (int r = 0; r < kGemvNRows; ++r) {
    s[r] = fma((double)v[r].x, xv[0], 0.0);
    s[r] = fma((double)v[r].y, xv[1], s[r]);
    s[r] = fma((double)v[r].z, xv[2], s[r]);
    s[r] = fma((double)v[r].w, xv[3], s[r]);
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int r = 0; r < kGemvNRows; ++r) {
    const double t = warp_sum(s[r]);
    if (lane == 0) red[r][w] = t;
  }
  __syncthreads();
  if (threadIdx.x < kGemvNRows && m0 + threadIdx.x < M) {
    double t = 0.0;
#pragma unroll
    for (int q = 0; q < 8; ++q) t += red[threadIdx.x][q];
    part[(m0 + threadIdx.x) * nchunk + blockIdx.x] = t;
  }
}

// a warp per row: out[m] = alpha sum_c part[m][c] + beta out[m]
__global__ void gemv_n_sum_kernel(const double* __restrict__ part, int64_t nchunk, int64_t M, double alpha,
                                  double beta, double* __restrict__ out) {
  const int64_t m = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5);
  if (m >= M) return;
  const int lane = threadIdx.x & 31;
  double s = 0.0;
  for (int64_t c = lane; c < nchunk; c += 32) s += part[m * nchunk + c];
  s = warp_sum(s);
  if (lane == 0) out[m] = alpha * s + (beta != 0.0 ? beta * out[m] : 0.0);
}

// per-block partial sums of x . y (FP64), fixed order
__global__ void dot_part_kernel(int64_t n, const double* __restrict__ x, const double* __restrict__ y,
                                double* __restrict__ part) {
  __shared__ double red[32];
  double s = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    s = fma(x[i], y[i], s);
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    double t = (threadIdx.x < (blockDim.x >> 5)) ? red[threadIdx.x] : 0.0;
    t = warp_sum(t);
    if (threadIdx.x == 0) part[blockIdx.x] = t;
  }
}

__global__ void axpby_kernel(int64_t n, double a, const double* __restrict__ x, double b, double* __restrict__ y) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) y[i] = a * x[i] + (b != 0.0 ? b * y[i] : 0.0);
}

// per-block partial sums of J^2
template <typename JT>
__global__ void sumsq_kernel(const JT* __restrict__ J, int64_t M, int64_t K, int64_t ldj,
                             double* __restrict__ part) {
  __shared__ double red[32];
  double s = 0.0;
  for (int64_t m = blockIdx.x; m < M; m += gridDim.x)
    for (int64_t k = threadIdx.x; k < K; k += blockDim.x) {
      const double v = jval(J[m * ldj + k]);
      s += v * v;
    }
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    double t = (threadIdx.x < (blockDim.x >> 5)) ? red[threadIdx.x] : 0.0;
    t = warp_sum(t);
    if (threadIdx.x == 0) part[blockIdx.x] = t;
  }
}

// out[m] = sum_k J[m][k]^2 in FP64: a block per row, a fixed-order
// reduction (the diagonal of J J^T without the tensor cores' input rounding)
// With bf != NULL the pass also writes the rows rounded to BF16 (row stride
// ldb, the padding columns K..ldb-1 zeroed): the operand of a BF16 product
// whose refinement runs over the FP32 rows.
template <typename JT, bool VEC>
__global__ void row_sumsq_kernel(const JT* __restrict__ J, int64_t M, int64_t K, int64_t ldj,
                                 double* __restrict__ out, __nv_bfloat16* __restrict__ bf, int64_t ldb) {
  __shared__ double red[32];
  for (int64_t m = blockIdx.x; m < M; m += gridDim.x) {
    double s = 0.0;
    int64_t kpad = K;  // first column of the BF16 row's zero padding
    if constexpr (VEC) {
      // 4 columns per thread and chunk: one 16-byte (BF16: 8-byte) load and
      // one 8-byte store; four chunks' loads are issued before their sums
      kpad = (K + 3) / 4 * 4;
      constexpr int U = 4;
      const int64_t step = 4 * (int64_t)blockDim.x;
      for (int64_t k0 = 4 * (int64_t)threadIdx.x; k0 < K; k0 += U * step) {
        float4 v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int64_t k = k0 + u * step;
          v[u] = k < K ? ld4f(J + m * ldj + k) : make_float4(0.f, 0.f, 0.f, 0.f);  // inside the row (ldj % 4 == 0)
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int64_t k = k0 + u * step;
          if (k >= K) break;
          if (k + 1 >= K) v[u].y = 0.f;  // entries past K are dropped
          if (k + 2 >= K) v[u].z = 0.f;
          if (k + 3 >= K) v[u].w = 0.f;
          s = fma((double)v[u].x, (double)v[u].x, s);
          s = fma((double)v[u].y, (double)v[u].y, s);
          s = fma((double)v[u].z, (double)v[u].z, s);
          s = fma((double)v[u].w, (double)v[u].w, s);
          if (bf) {
            __nv_bfloat162 lo = __floats2bfloat162_rn(v[u].x, v[u].y), hi = __floats2bfloat162_rn(v[u].z, v[u].w);
            uint2 w;
            w.x = *reinterpret_cast<uint32_t*>(&lo);
            w.y = *reinterpret_cast<uint32_t*>(&hi);
            *reinterpret_cast<uint2*>(bf + m * ldb + k) = w;
          }
        }
      }
    } else {
      for (int64_t k = threadIdx.x; k < K; k += blockDim.x) {
        const double v = jval(J[m * ldj + k]);
        s = fma(v, v, s);
        if (bf) bf[m * ldb + k] = __float2bfloat16_rn((float)v);
      }
    }
    if (bf)
      for (int64_t k = kpad + threadIdx.x; k < ldb; k += blockDim.x) bf[m * ldb + k] = __float2bfloat16_rn(0.f);
    s = warp_sum(s);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
      double t = (threadIdx.x < (blockDim.x >> 5)) ? red[threadIdx.x] : 0.0;
      t = warp_sum(t);
      if (threadIdx.x == 0) out[m] = t;
    }
    __syncthreads();
  }
}

// H[i][i] = alpha d[i]
__global__ void set_diag_kernel(double* __restrict__ H, int64_t M, int64_t ldh, const double* __restrict__ d,
                                double alpha) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < M) H[i * ldh + i] = alpha * d[i];
}

__global__ void sum_parts_kernel(const double* __restrict__ part, int n, double* __restrict__ out) {
  __shared__ double red[32];
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s += part[i];
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    double t = (threadIdx.x < (blockDim.x >> 5)) ? red[threadIdx.x] : 0.0;
    t = warp_sum(t);
    if (threadIdx.x == 0) *out = t;
  }
}

__global__ void vec_mul_kernel(const double* __restrict__ a, const double* __restrict__ b, double* __restrict__ out,
                               int64_t n) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) out[i] = a[i] * b[i];
}

// hi = tf32(J) rounded to nearest (in place), lo = J - hi
__global__ void split_tf32_kernel(float* __restrict__ J, float* __restrict__ lo, int64_t M, int64_t K, int64_t ldj) {
  for (int64_t m = blockIdx.y; m < M; m += gridDim.y)
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < K; k += (int64_t)gridDim.x * blockDim.x) {
      const float v = J[m * ldj + k];
      uint32_t h;
      asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(h) : "f"(v));
      const float hv = __uint_as_float(h);
      J[m * ldj + k] = hv;
      lo[m * ldj + k] = v - hv;
    }
}

// The two streams of rb_cholesky's look-ahead, per device, created once:
// the panel stream at the device's highest priority, the bulk-update stream
// at the default one; both non-blocking.
struct CholStreams {
  cudaStream_t panel = nullptr, rest = nullptr;
};
static int chol_streams(CholStreams* out) {
  static std::mutex mu;
  static CholStreams per_dev[64];
  int dev = 0;
  RB_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return fail(RB_ESIZE, "rb_cholesky: device index %d out of range", dev);
  std::lock_guard<std::mutex> lock(mu);
  CholStreams& c = per_dev[dev];
  if (!c.panel) {
    int least = 0, greatest = 0;
    RB_CUDA_TRY(cudaDeviceGetStreamPriorityRange(&least, &greatest));
    RB_CUDA_TRY(cudaStreamCreateWithPriority(&c.panel, cudaStreamNonBlocking, greatest));
    RB_CUDA_TRY(cudaStreamCreateWithPriority(&c.rest, cudaStreamNonBlocking, least));
  }
  *out = c;
  return RB_OK;
}

// events without timing, destroyed with the set
struct EventSet {
  cudaEvent_t e[4] = {nullptr, nullptr, nullptr, nullptr};
  int n = 0;
  int make(int k) {
    for (; n < k; ++n) RB_CUDA_TRY(cudaEventCreateWithFlags(&e[n], cudaEventDisableTiming));
    return RB_OK;
  }
  ~EventSet() {
    for (int i = 0; i < n; ++i) cudaEventDestroy(e[i]);
  }
};

}  // namespace rb

using namespace rb;

extern "C" {

int rb_reginv_prepare(double* H, int64_t M, int64_t ldh, double lambda, double* di, void* stream) {
  if (!H || !di || M < 1 || ldh < M) return fail(RB_EARG, "rb_reginv_prepare: bad arguments");
  if (M > 65535) return fail(RB_ESIZE, "rb_reginv_prepare: at most 65535 rows");
  cudaStream_t st = as_stream(stream);
  prep_diag_kernel<<<(unsigned)ceil_div(M, 256), 256, 0, st>>>(H, M, ldh, lambda, di);
  RB_LAUNCH_CHECK();
  prep_scale_kernel<<<dim3((unsigned)ceil_div(M, 256), (unsigned)M), 256, 0, st>>>(H, M, ldh, di);
  RB_LAUNCH_CHECK();
  return RB_OK;
}

size_t rb_cholesky_work_bytes(void) { return 256; }

int rb_cholesky(double* H, int64_t M, int64_t ldh, void* work, size_t work_bytes, void* stream) {
  if (!H || !work || M < 1 || ldh < M) return fail(RB_EARG, "rb_cholesky: bad arguments");
  if (work_bytes < rb_cholesky_work_bytes()) return fail(RB_EARG, "rb_cholesky: workspace too small");
  if (M > 65535 * 32) return fail(RB_ESIZE, "rb_cholesky: matrix too large");
  cudaStream_t st = as_stream(stream);
  RB_CUDA_TRY(cudaFuncSetAttribute(potrf_diag_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPotrfSmem));
  int* err = reinterpret_cast<int*>(work);
  RB_CUDA_TRY(cudaMemsetAsync(err, 0, sizeof(int), st));
  RB_CUDA_TRY(cudaFuncSetAttribute(trsm_panel_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTrsmSmem));
  // 16-byte panel copies when every row of H starts on a 16-byte boundary
  const bool ch16 = (reinterpret_cast<uintptr_t>(H) % 16 == 0) && (ldh % 2 == 0);
  auto syrk = ch16 ? syrk_update_kernel<16> : syrk_update_kernel<8>;
  RB_CUDA_TRY(cudaFuncSetAttribute(syrk, cudaFuncAttributeMaxDynamicSharedMemorySize, kSyrkSmem));
  // Right-looking in outer blocks of kOuter columns: inside a block each
  // 64-wide panel is factored (diagonal block, panel solve) and updates only
  // the rest of the block's columns; the trailing matrix then takes one
  // update of depth kOuter per outer block.  Look-ahead: that update is
  // split into the next block's column band (on the panel stream, so the
  // next block can start at once) and the rest of the trailing triangle (on
  // a second stream, overlapping the next block's serial panel work).  The
  // panel stream has the higher priority, so its small launches take SMs as
  // the bulk update's CTAs retire.  Ordering: the rest update of block b
  // waits for block b's panels (event ev_p); the band update of block b + 1,
  // which writes tiles the rest update of block b also writes, waits for it
  // (event ev_r).  Both streams fork from and join back into the caller's.
  CholStreams cs;
  RB_TRY(chol_streams(&cs));
  cudaStream_t sp = cs.panel, sr = cs.rest;
  EventSet ev;
  RB_TRY(ev.make(4));
  cudaEvent_t ev_in = ev.e[0], ev_p = ev.e[1], ev_r = ev.e[2], ev_out = ev.e[3];
  RB_CUDA_TRY(cudaEventRecord(ev_in, st));
  RB_CUDA_TRY(cudaStreamWaitEvent(sp, ev_in, 0));
  RB_CUDA_TRY(cudaStreamWaitEvent(sr, ev_in, 0));
  bool rest_queued = false;
  constexpr int64_t kOuter = 4 * kNB;
  for (int64_t J0 = 0; J0 < M; J0 += kOuter) {
    const int64_t bend = std::min<int64_t>(J0 + kOuter, M);
    for (int64_t j0 = J0; j0 < bend; j0 += kNB) {
      const int nb = (int)std::min<int64_t>(kNB, M - j0);
      potrf_diag_kernel<<<1, 256, kPotrfSmem, sp>>>(H, ldh, j0, nb, err);
      RB_LAUNCH_CHECK();
      const int64_t rest = M - j0 - nb;
      if (rest <= 0) break;
      trsm_panel_kernel<<<(unsigned)ceil_div(rest, kNB), 256, kTrsmSmem, sp>>>(H, ldh, M, j0, nb);
      RB_LAUNCH_CHECK();
      if (j0 + nb < bend) {  // the block's later panels
        const int64_t T = ceil_div(rest, kNB), Tc = ceil_div(bend - (j0 + nb), kNB);
        syrk<<<dim3((unsigned)T, (unsigned)Tc), kSyrkThreads, kSyrkSmem, sp>>>(H, ldh, M, j0, nb, j0 + nb, bend, 0);
        RB_LAUNCH_CHECK();
      }
    }
    const int64_t rest = M - bend;
    if (rest <= 0) break;
    const int depth = (int)(bend - J0);
    const int64_t band_end = std::min<int64_t>(bend + kOuter, M);
    RB_CUDA_TRY(cudaEventRecord(ev_p, sp));  // block J0's panels are final
    if (rest_queued) RB_CUDA_TRY(cudaStreamWaitEvent(sp, ev_r, 0));
    {  // the next block's columns [bend, band_end), all rows below bend
      const int64_t T = ceil_div(rest, kNB), Tc = ceil_div(band_end - bend, kNB);
      syrk<<<dim3((unsigned)T, (unsigned)Tc), kSyrkThreads, kSyrkSmem, sp>>>(H, ldh, M, J0, depth, bend, band_end,
                                                                              0);
      RB_LAUNCH_CHECK();
    }
    if (band_end < M) {  // the trailing triangle right of the band
      const int64_t T = ceil_div(M - band_end, kNB);
      RB_CUDA_TRY(cudaStreamWaitEvent(sr, ev_p, 0));
      syrk<<<(unsigned)(T * (T + 1) / 2), kSyrkThreads, kSyrkSmem, sr>>>(H, ldh, M, J0, depth, band_end, M, 1);
      RB_LAUNCH_CHECK();
      RB_CUDA_TRY(cudaEventRecord(ev_r, sr));
      rest_queued = true;
    }
  }
  RB_CUDA_TRY(cudaEventRecord(ev_out, sr));
  RB_CUDA_TRY(cudaStreamWaitEvent(st, ev_out, 0));
  RB_CUDA_TRY(cudaEventRecord(ev_out, sp));
  RB_CUDA_TRY(cudaStreamWaitEvent(st, ev_out, 0));
  int herr = 0;
  RB_CUDA_TRY(cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, st));
  RB_CUDA_TRY(cudaStreamSynchronize(st));
  if (herr) return fail(RB_ENOTSPD, "rb_cholesky: non-positive pivot at row %d", herr - 1);
  return RB_OK;
}

// the segments of y and x, whole blocks of 64
size_t rb_chol_solve_work_bytes(int64_t M) {
  return 2 * (size_t)ceil_div(std::max<int64_t>(M, 1), kNB) * kNB * sizeof(double) + 16;
}

int rb_chol_solve(const double* L, int64_t M, int64_t ldh, double* x, void* work, size_t work_bytes, void* stream) {
  if (!L || !x || !work || M < 1 || ldh < M) return fail(RB_EARG, "rb_chol_solve: bad arguments");
  if (work_bytes < (size_t)M * sizeof(double)) return fail(RB_EARG, "rb_chol_solve: workspace too small");
  cudaStream_t st = as_stream(stream);
  const int64_t nblk = ceil_div(M, kNB);
  // a workspace of M doubles is taken as well: the segments come from the pool
  void* own = nullptr;
  if (work_bytes < rb_chol_solve_work_bytes(M)) {
    RB_CUDA_TRY(cudaMallocAsync(&own, rb_chol_solve_work_bytes(M), st));
    work = own;
  }
  double* ys = reinterpret_cast<double*>((reinterpret_cast<uintptr_t>(work) + 15) & ~uintptr_t(15));
  double* xs = ys + nblk * kNB;
  cudaError_t e = cudaMemsetAsync(ys, 0xff, 2 * (size_t)nblk * kNB * sizeof(double), st);
  // the blocks wait for one another: a cooperative launch, at most one per SM
  int dev = 0, sms = 1;
  if (e == cudaSuccess) e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess) {
    void* args[] = {(void*)&L, (void*)&ldh, (void*)&M, (void*)&x, (void*)&ys, (void*)&xs};
    e = cudaLaunchCooperativeKernel((const void*)chol_solve_kernel, dim3((unsigned)std::min<int64_t>(nblk, sms)),
                                    dim3(256), args, 0, st);
  }
  if (own) {
    const cudaError_t f = cudaFreeAsync(own, st);
    if (e == cudaSuccess) e = f;
  }
  RB_CUDA_TRY(e);
  return RB_OK;
}

int rb_chol_solve_status(void* stream) {
  RB_CUDA_TRY(cudaStreamSynchronize(as_stream(stream)));
  int h = 0;
  RB_CUDA_TRY(cudaMemcpyFromSymbol(&h, g_trsv_err, sizeof(int)));
  if (h) {
    const int zero = 0;
    RB_CUDA_TRY(cudaMemcpyToSymbol(g_trsv_err, &zero, sizeof(int)));
    return fail(RB_ECUDA, "rb_chol_solve: a wait for another block row gave up; the solution is not valid");
  }
  return RB_OK;
}

size_t rb_gemv_t_work_bytes(int64_t K) { return (size_t)kGemvSlabs * K * sizeof(double) + 256; }

}  // extern "C"

template <typename JT>
static int gemv_t_run(const JT* J, int64_t M, int64_t K, int64_t ldj, const double* y, double alpha, double beta,
                      double* out, void* work, size_t work_bytes, void* stream) {
  if (!J || !y || !out || !work || M < 1 || K < 1 || ldj < K) return fail(RB_EARG, "rb_gemv_t: bad arguments");
  if (work_bytes < rb_gemv_t_work_bytes(K)) return fail(RB_EARG, "rb_gemv_t: workspace too small");
  if ((reinterpret_cast<uintptr_t>(J) & (4 * sizeof(JT) - 1)) || (ldj % 4))
    return fail(RB_EARG, "rb_gemv_t: J rows must start on %d-byte boundaries (aligned J, ldj %% 4 == 0)",
                (int)(4 * sizeof(JT)));
  cudaStream_t st = as_stream(stream);
  const int slabs = (int)std::min<int64_t>(kGemvSlabs, M);
  double* part = reinterpret_cast<double*>(work);
  gemv_t_part_kernel<JT><<<dim3((unsigned)ceil_div(K, 4 * 256), (unsigned)slabs), 256, 0, st>>>(J, M, K, ldj, y,
                                                                                                part);
  RB_LAUNCH_CHECK();
  gemv_t_sum_kernel<<<(unsigned)ceil_div(K, 256), 256, 0, st>>>(part, slabs, K, alpha, beta, out);
  RB_LAUNCH_CHECK();
  return RB_OK;
}

template <typename JT>
static int gemv_n_run(const JT* J, int64_t M, int64_t K, int64_t ldj, const double* x, double alpha, double beta,
                      double* out, void* work, size_t work_bytes, void* stream) {
  if (!J || !x || !out || M < 1 || K < 1 || ldj < K) return fail(RB_EARG, "rb_gemv_n: bad arguments");
  if ((reinterpret_cast<uintptr_t>(J) & (4 * sizeof(JT) - 1)) || (ldj % 4) || ldj < ceil_div(K, 4) * 4)
    return fail(RB_EARG, "rb_gemv_n: J rows must start on %d-byte boundaries and hold K rounded up to 4 entries",
                (int)(4 * sizeof(JT)));
  if (ceil_div(M, kGemvNRows) > 65535) return fail(RB_ESIZE, "rb_gemv_n: too many rows");
  if (!work || work_bytes < rb_gemv_n_work_bytes(M, K)) return fail(RB_EARG, "rb_gemv_n: workspace too small");
  cudaStream_t st = as_stream(stream);
  const int64_t nchunk = ceil_div(K, kGemvNCols);
  double* part = reinterpret_cast<double*>(work);  // M x nchunk row parts
  gemv_n_part_kernel<JT><<<dim3((unsigned)nchunk, (unsigned)ceil_div(M, kGemvNRows)), 256, 0, st>>>(J, M, K, ldj, x,
                                                                                                   part, nchunk);
  RB_LAUNCH_CHECK();
  gemv_n_sum_kernel<<<(unsigned)ceil_div(M, 8), 256, 0, st>>>(part, nchunk, M, alpha, beta, out);
  RB_LAUNCH_CHECK();
  return RB_OK;
}

extern "C" {

size_t rb_gemv_n_work_bytes(int64_t M, int64_t K) {
  return (size_t)std::max<int64_t>(M, 1) * (size_t)std::max<int64_t>(ceil_div(K, kGemvNCols), 1) * sizeof(double);
}

int rb_gemv_n(const float* J, int64_t M, int64_t K, int64_t ldj, const double* x, double alpha, double beta,
              double* out, void* work, size_t work_bytes, void* stream) {
  return gemv_n_run(J, M, K, ldj, x, alpha, beta, out, work, work_bytes, stream);
}

int rb_gemv_n_bf16(const void* J, int64_t M, int64_t K, int64_t ldj, const double* x, double alpha, double beta,
                   double* out, void* work, size_t work_bytes, void* stream) {
  return gemv_n_run(reinterpret_cast<const __nv_bfloat16*>(J), M, K, ldj, x, alpha, beta, out, work, work_bytes,
                    stream);
}

size_t rb_dot_work_bytes(void) { return 64 * sizeof(double) + 256; }

int rb_dot(int64_t n, const double* x, const double* y, double* out, void* work, size_t work_bytes, void* stream) {
  if (!x || !y || !out || !work || n < 1) return fail(RB_EARG, "rb_dot: bad arguments");
  if (work_bytes < rb_dot_work_bytes()) return fail(RB_EARG, "rb_dot: workspace too small");
  cudaStream_t st = as_stream(stream);
  const int blocks = (int)std::min<int64_t>(64, ceil_div(n, 256));
  double* part = reinterpret_cast<double*>(work);
  dot_part_kernel<<<blocks, 256, 0, st>>>(n, x, y, part);
  RB_LAUNCH_CHECK();
  sum_parts_kernel<<<1, 64, 0, st>>>(part, blocks, out);
  RB_LAUNCH_CHECK();
  return RB_OK;
}

int rb_axpby(int64_t n, double a, const double* x, double b, double* y, void* stream) {
  if (!x || !y || n < 0) return fail(RB_EARG, "rb_axpby: bad arguments");
  if (n == 0) return RB_OK;
  axpby_kernel<<<(unsigned)ceil_div(n, 256), 256, 0, as_stream(stream)>>>(n, a, x, b, y);
  RB_LAUNCH_CHECK();
  return RB_OK;
}

int rb_gemv_t(const float* J, int64_t M, int64_t K, int64_t ldj, const double* y, double alpha, double beta,
              double* out, void* work, size_t work_bytes, void* stream) {
  return gemv_t_run(J, M, K, ldj, y, alpha, beta, out, work, work_bytes, stream);
}

int rb_gemv_t_bf16(const void* J, int64_t M, int64_t K, int64_t ldj, const double* y, double alpha, double beta,
                   double* out, void* work, size_t work_bytes, void* stream) {
  return gemv_t_run(reinterpret_cast<const __nv_bfloat16*>(J), M, K, ldj, y, alpha, beta, out, work, work_bytes,
                    stream);
}

int rb_vec_mul(const double* a, const double* b, double* out, int64_t n, void* stream) {
  if (!a || !b || !out || n < 0) return fail(RB_EARG, "rb_vec_mul: bad arguments");
  if (n == 0) return RB_OK;
  vec_mul_kernel<<<(unsigned)ceil_div(n, 256), 256, 0, as_stream(stream)>>>(a, b, out, n);
  RB_LAUNCH_CHECK();
  return RB_OK;
}

int rb_split_tf32(float* J, float* lo, int64_t M, int64_t K, int64_t ldj, void* stream) {
  if (!J || !lo || M < 1 || K < 1 || ldj < K) return fail(RB_EARG, "rb_split_tf32: bad arguments");
  dim3 g((unsigned)std::min<int64_t>(ceil_div(K, 256), 64), (unsigned)std::min<int64_t>(M, 4096));
  split_tf32_kernel<<<g, 256, 0, as_stream(stream)>>>(J, lo, M, K, ldj);
  RB_LAUNCH_CHECK();
  return RB_OK;
}

size_t rb_sumsq_work_bytes(void) { return 148 * 8 * sizeof(double) + 256; }

}  // extern "C"

template <typename JT>
static int sumsq_run(const JT* J, int64_t M, int64_t K, int64_t ldj, double* out, void* work, size_t work_bytes,
                     void* stream) {
  if (!J || !out || !work || M < 1 || K < 1 || ldj < K) return fail(RB_EARG, "rb_sumsq: bad arguments");
  if (work_bytes < rb_sumsq_work_bytes()) return fail(RB_EARG, "rb_sumsq: workspace too small");
  cudaStream_t st = as_stream(stream);
  const int nb = 148 * 8;
  double* part = reinterpret_cast<double*>(work);
  sumsq_kernel<JT><<<nb, 256, 0, st>>>(J, M, K, ldj, part);
  RB_LAUNCH_CHECK();
  sum_parts_kernel<<<1, 1024, 0, st>>>(part, nb, out);
  RB_LAUNCH_CHECK();
  return RB_OK;
}

extern "C" {


int rb_sumsq(const float* J, int64_t M, int64_t K, int64_t ldj, double* out, void* work, size_t work_bytes,
             void* stream) {
  return sumsq_run(J, M, K, ldj, out, work, work_bytes, stream);
}

int rb_sumsq_bf16(const void* J, int64_t M, int64_t K, int64_t ldj, double* out, void* work, size_t work_bytes,
                  void* stream) {
  return sumsq_run(reinterpret_cast<const __nv_bfloat16*>(J), M, K, ldj, out, work, work_bytes, stream);
}

}  // extern "C"

template <typename JT>
static int row_sumsq_run(const JT* J, int64_t M, int64_t K, int64_t ldj, double* rows, double* total, void* stream,
                         __nv_bfloat16* bf = nullptr, int64_t ldb = 0) {
  if (!J || !rows || M < 1 || K < 1 || ldj < K || M > INT32_MAX) return fail(RB_EARG, "rb_row_sumsq: bad arguments");
  if (bf && (ldb < K || ldb % 8)) return fail(RB_EARG, "rb_row_sumsq_to_bf16: ldb must be >= K and a multiple of 8");
  cudaStream_t st = as_stream(stream);
  const unsigned nb = (unsigned)std::min<int64_t>(M, 148 * 16);
  // vector path: rows start on 4-entry boundaries (and, for the copy, the BF16 rows on 8-byte ones)
  const bool vec = (reinterpret_cast<uintptr_t>(J) % (4 * sizeof(JT)) == 0) && ldj % 4 == 0 &&
                   (!bf || reinterpret_cast<uintptr_t>(bf) % 8 == 0);
  if (vec)
    row_sumsq_kernel<JT, true><<<nb, 256, 0, st>>>(J, M, K, ldj, rows, bf, ldb);
  else
    row_sumsq_kernel<JT, false><<<nb, 256, 0, st>>>(J, M, K, ldj, rows, bf, ldb);
  RB_LAUNCH_CHECK();
  if (total) {
    sum_parts_kernel<<<1, 1024, 0, st>>>(rows, (int)M, total);
    RB_LAUNCH_CHECK();
  }
  return RB_OK;
}

extern "C" {

int rb_row_sumsq(const float* J, int64_t M, int64_t K, int64_t ldj, double* rows, double* total, void* stream) {
  return row_sumsq_run(J, M, K, ldj, rows, total, stream);
}

int rb_row_sumsq_bf16(const void* J, int64_t M, int64_t K, int64_t ldj, double* rows, double* total,
                      void* stream) {
  return row_sumsq_run(reinterpret_cast<const __nv_bfloat16*>(J), M, K, ldj, rows, total, stream);
}

int rb_row_sumsq_to_bf16(const float* J, int64_t M, int64_t K, int64_t ldj, double* rows, double* total, void* bf,
                         int64_t ldb, void* stream) {
  if (!bf) return fail(RB_EARG, "rb_row_sumsq_to_bf16: null output");
  return row_sumsq_run(J, M, K, ldj, rows, total, stream, reinterpret_cast<__nv_bfloat16*>(bf), ldb);
}

int rb_set_diag(double* H, int64_t M, int64_t ldh, const double* d, double alpha, void* stream) {
  if (!H || !d || M < 1 || ldh < M) return fail(RB_EARG, "rb_set_diag: bad arguments");
  set_diag_kernel<<<(unsigned)ceil_div(M, 256), 256, 0, as_stream(stream)>>>(H, M, ldh, d, alpha);
  RB_LAUNCH_CHECK();
  return RB_OK;
}

}  // extern "C"
