// Three-level V-cycle preconditioner of the mixed-precision block CG / COCG
// (included by rb_krylov.cu), for meshes large enough to need a coarse space.
//
// Levels: the mesh nodes (n rows); the spatial row groups of the blocked SpMM
// (up to 8 neighbouring nodes each, P1 their 0/1 membership); aggregates of
// the groups (P2, at most kCoarseMax), whose operator is inverted densely.
// Every level is scaled to a unit diagonal, A^ = S A S with S = D^-1/2, so the
// Jacobi smoother is a number: with w = 1.7 / (Gershgorin bound of D^-1 A),
// below 2 / lambda_max, so that the cycle stays positive definite (real) or
// symmetric (complex), one application of the symmetric cycle to r^ is
//   t = A^ r^,  f = P1^T S^-1 (r^ - w t),  e = M1 f,
//   z = 2 w r^ - w^2 t + S^-1 P1 e - w S A P1 e,
// the pre-smoothed, coarse-corrected, post-smoothed vector written out, and
//   (r^, z) = 2 w (r^, r^) - w^2 (r^, t) + (e, f).
// z is never stored: the p-update forms it from r, t and the few e rows that
// a group's neighbours share (A P1 has about two entries per row).  M1 is one
// cycle of the same kind on the group level (degree-2 Chebyshev smoothing
// there, an eighth of the rows) around the dense inverse.
//
// Why: an iteration of the two-level form (Jacobi plus coarse correction) is
// bound by its 10 vector passes over HBM, and 33-43 of them were needed per
// 1e-5 sweep on the 520k-node box; the cycle costs one more product (t) and
// one more pass, about 1.6 times the bytes, and needs 12-14.  The products run
// over the row groups: each x row is gathered once per group, and P1^T of a
// product is the sum of the rows the same warp has in registers.
// Measured (whole forward, two-level -> this): 520k nodes x 128 columns 96.3 ->
// 49.9 ms (130 -> 34 iterations), complex 224.6 -> 116.3 (160 -> 34); 43k x 37
// 9.9 -> 4.7 (100 -> 25); gradient at 68k x 64 11.9 -> 5.4 (90 -> 25); batch of 64
// boxes 48.6 (Jacobi) -> 23.8.  The kernels of an iteration are launched early
// (launch_early): a gap of a microsecond before each of 16 kernels was an eighth
// of the middle sizes' time (43k x 37 5.42 -> 4.75).
#pragma once

namespace rb {

// lanes per group task, columns per lane, column slices: 16 bytes per lane
struct GShape {
  int L, V, S;
};
template <typename T>
static GShape vc_shape(int64_t k) {
  constexpr int V = 16 / (int)sizeof(T);
  GShape s{32, V, 1};
  while (s.L > 4 && (int64_t)(s.L / 2) * V >= k) s.L /= 2;
  if ((int64_t)s.L * V < k) s.S = 2;
  return s;
}
// columns a cycle solve runs on: whole lanes of 4 columns
static int64_t vc_cols(int64_t k) { return ceil_div(k, 4) * 4; }

#define RB_DISPATCH_G(sh, FN)                                              \
  switch (sh.L * 4 + sh.S) {                                               \
    case 4 * 4 + 1: FN(4, 1); break;                                       \
    case 8 * 4 + 1: FN(8, 1); break;                                       \
    case 16 * 4 + 1: FN(16, 1); break;                                     \
    case 32 * 4 + 1: FN(32, 1); break;                                     \
    case 32 * 4 + 2: if constexpr (sizeof(T) == 8) { FN(32, 2); } break;   \
    default: return fail(RB_EARG, "bad group shape");                      \
  }

// cycle parameters on the device (from the Gershgorin bounds)
struct VcPar {
  uint32_t g[2];            // bits of the bounds of the two levels (positive floats)
  float w, w2;              // fine smoother: w, w^2
  float one, mone;
  float a, b, na, nb;       // group smoother q(A^) = a - b A^ and the negatives
};

template <typename T>
struct VcOp {
  RowGroupsDev rg;          // coef: scaled matrix, 8 values per union entry
  int64_t ng = 0;
  const int32_t *mptr = nullptr, *mcol = nullptr;  // group-level pattern
  T* cm = nullptr;          // nnz1 x 8: S A P1, the group's 8 rows per entry
  T* v1 = nullptr;          // nnz1: scaled group-level matrix
  T *s = nullptr, *is = nullptr;    // n: S and S^-1
  T *s1 = nullptr, *is1 = nullptr;  // ng: the same of the group level
  T* vs = nullptr;          // nnz: scaled CSR values (row-pair SpMM of complex solves)
  T* t = nullptr;           // n x k
  T *f = nullptr, *x2 = nullptr, *w = nullptr, *e = nullptr;  // ng x k
  VcPar* par = nullptr;
  void* part_c = nullptr;   // kGridMax x k acc: (e, f)
  CoarseOp<T> co;           // over the groups
};

template <typename T64, typename T>
struct VcBufs {
  VcOp<T> op;
  CoarseBufs<T64, T> cb;
  T64 *s64 = nullptr, *s64_1 = nullptr, *d64_1 = nullptr, *val1 = nullptr;
  int64_t nnz1 = 0;
};

template <typename T64, typename T>
static size_t vc_carve(Carver& cv, VcBufs<T64, T>& b, int64_t n, int64_t nnz, int64_t ng, int64_t nu, int64_t nnz1,
                       int64_t nc, int64_t k) {
  b.nnz1 = nnz1;
  b.op.ng = ng;
  b.s64 = cv.take<T64>(n);
  b.s64_1 = cv.take<T64>(ng);
  b.d64_1 = cv.take<T64>(ng);
  b.val1 = cv.take<T64>(nnz1);
  b.op.rg.coef = cv.take<T>(nu * kRG);
  b.op.cm = cv.take<T>(nnz1 * kRG);
  b.op.v1 = cv.take<T>(nnz1);
  b.op.s = cv.take<T>(n);
  b.op.is = cv.take<T>(n);
  b.op.s1 = cv.take<T>(ng);
  b.op.is1 = cv.take<T>(ng);
  b.op.vs = cv.take<T>(std::max<int64_t>(nnz, 1));
  b.op.t = cv.take<T>(n * k);
  b.op.f = cv.take<T>(ng * k);
  b.op.x2 = cv.take<T>(ng * k);
  b.op.w = cv.take<T>(ng * k);
  b.op.e = cv.take<T>(ng * k);
  b.op.par = cv.take<VcPar>(1);
  b.op.part_c = cv.take<cdouble>((size_t)kGridMax * k);
  return coarse_carve(cv, b.cb, nc, k);
}

// ----------------------------------------------------------------- setup
__device__ __forceinline__ double c_abs(double v) { return fabs(v); }
__device__ __forceinline__ double c_abs(cdouble v) { return sqrt(v.x * v.x + v.y * v.y); }
__device__ __forceinline__ double c_sqrt(double v) { return sqrt(v); }
__device__ __forceinline__ cdouble c_sqrt(cdouble v) {  // principal root
  const double m = c_abs(v), x = sqrt(0.5 * (m + v.x));
  return make_double2(x, x > 0.0 ? 0.5 * v.y / x : 0.0);
}
__device__ __forceinline__ double c_inv(double v) { return 1.0 / v; }
__device__ __forceinline__ cdouble c_inv(cdouble v) {
  const double d = v.x * v.x + v.y * v.y;
  return make_double2(v.x / d, -v.y / d);
}
__device__ __forceinline__ float r_mul(float r, float v) { return r * v; }
__device__ __forceinline__ cfloat r_mul(float r, cfloat v) { return make_float2(r * v.x, r * v.y); }
__device__ __forceinline__ double r_mul(double r, double v) { return r * v; }
__device__ __forceinline__ cdouble r_mul(double r, cdouble v) { return make_double2(r * v.x, r * v.y); }
__device__ __forceinline__ double cs_mul(double s, double v) { return s * v; }
__device__ __forceinline__ cdouble cs_mul(cdouble s, double v) { return make_double2(s.x * v, s.y * v); }
__device__ __forceinline__ cdouble cs_mul(cdouble s, cdouble v) { return s_mul(s, v); }
__device__ __forceinline__ double widen(float v) { return v; }
__device__ __forceinline__ cdouble widen(cfloat v) { return make_double2(v.x, v.y); }
template <typename T> __device__ __forceinline__ T narrow_to(double v) { return (T)v; }
template <typename T> __device__ __forceinline__ T narrow_to(cdouble v) { return T{(float)v.x, (float)v.y}; }

// S = D^-1/2 and its inverse from the reciprocal diagonal
template <typename T64, typename T>
__global__ void vc_scale_kernel(int64_t n, const T64* __restrict__ dinv, T64* __restrict__ s64, T* __restrict__ s,
                                T* __restrict__ is) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const T64 r = c_sqrt(dinv[i]);
    s64[i] = r;
    s[i] = narrow_to<T>(r);
    is[i] = narrow_to<T>(c_inv(r));
  }
}

// scaled values S A S and the Gershgorin bound of D^-1 A; 16 lanes per row
template <typename T64, typename T>
__global__ void __launch_bounds__(256)
vc_values_kernel(int64_t n, const int32_t* __restrict__ indptr, const int32_t* __restrict__ indices,
                 const T64* __restrict__ val, const T64* __restrict__ dinv, const T64* __restrict__ s64,
                 T* __restrict__ vs, uint32_t* __restrict__ bound) {
  const int l = threadIdx.x & 15;
  float top = 0.f;
  for (int64_t i = blockIdx.x * (int64_t)16 + (threadIdx.x >> 4); i < n; i += (int64_t)gridDim.x * 16) {
    const T64 si = s64[i];
    double a = 0.0;
    for (int32_t p = indptr[i] + l; p < indptr[i + 1]; p += 16) {
      const T64 v = val[p];
      vs[p] = narrow_to<T>(s_mul(s_mul(v, si), s64[indices[p]]));
      a += c_abs(v);
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffu << (threadIdx.x & 16), a, o);
    top = fmaxf(top, (float)(a * c_abs(dinv[i]) * (1.0 + 1e-6)));
  }
  const uint32_t m = __reduce_max_sync(0xffffffffu, __float_as_uint(top));
  if ((threadIdx.x & 31) == 0) atomicMax(bound, m);
}

// smoother parameters from the bounds g: fine w = 1.7 / g; group level the
// degree-2 Chebyshev polynomial of [g / 16, g] (Saad, Iterative Methods for
// Sparse Linear Systems, section 12.3) written as a - b A^.  Iterations at
// w g / (bound over lower end) 1.6 / 8, 1.7 / 16, 1.9 / 16: regular boxes, whose
// bound is tight, 24, 22, 36 (43k nodes) and 32, 30, 39 (520k); displaced
// nodes, whose bound is a fifth too large, 26, 25, 24 and 41, 38, 38.
__global__ void vc_param_kernel(VcPar* __restrict__ p) {
  const float g0 = __uint_as_float(p->g[0]), g1 = __uint_as_float(p->g[1]);
  p->w = 1.7f / g0;
  p->w2 = p->w * p->w;
  p->one = 1.f;
  p->mone = -1.f;
  const double hi = g1, lo = hi / 16.0, th = 0.5 * (hi + lo), de = 0.5 * (hi - lo), sg = th / de;
  const double r0 = 1.0 / sg, r1 = 1.0 / (2.0 * sg - r0);
  p->a = (float)((1.0 + r1 * r0) / th + 2.0 * r1 / de);
  p->b = (float)(2.0 * r1 / (de * th));
  p->na = -p->a;
  p->nb = -p->b;
}

constexpr int kMidMax = 64;  // neighbour groups of a group at most (else no group level)
constexpr int kMidWarps = 4;

// A P1 of a group's 8 rows and the group-level matrix P1^T A P1: a warp per
// group, lane r < 8 adds row r's entries into its own column of the table
// (ascending columns: the same sums on every run)
template <typename T64, typename T>
__global__ void __launch_bounds__(kMidWarps * 32)
vc_mid_kernel(int64_t ng, const int32_t* __restrict__ rows, const int32_t* __restrict__ indptr,
              const int32_t* __restrict__ indices, const T64* __restrict__ val, const int32_t* __restrict__ grp,
              const int32_t* __restrict__ mptr, const int32_t* __restrict__ mcol, const T64* __restrict__ s64,
              T64* __restrict__ val1, T* __restrict__ cm) {
  __shared__ T64 sc[kMidWarps][kMidMax][kRG];
  __shared__ int32_t sh[kMidWarps][kMidMax];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int64_t g = blockIdx.x * (int64_t)kMidWarps + w; g < ng; g += (int64_t)gridDim.x * kMidWarps) {
    const int32_t m0 = mptr[g], nm = min(mptr[g + 1] - m0, kMidMax);
    for (int j = lane; j < nm; j += 32) sh[w][j] = mcol[m0 + j];
    for (int j = lane; j < nm * kRG; j += 32) sc[w][j / kRG][j % kRG] = s_zero(T64());
    __syncwarp();
    const int32_t row = lane < kRG ? rows[g * kRG + lane] : -1;
    if (row >= 0) {
      for (int32_t p = indptr[row]; p < indptr[row + 1]; ++p) {
        const int32_t h = grp[indices[p]];
        int lo = 0, hi = nm - 1;  // mcol ascending
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (sh[w][mid] < h) lo = mid + 1;
          else hi = mid;
        }
        sc[w][lo][lane] = s_add(sc[w][lo][lane], val[p]);
      }
    }
    __syncwarp();
    const T64 sr = row >= 0 ? s64[row] : s_zero(T64());
    for (int j = lane; j < nm; j += 32) {
      T64 a = s_zero(T64());
#pragma unroll
      for (int r = 0; r < kRG; ++r) a = s_add(a, sc[w][j][r]);
      val1[m0 + j] = a;
    }
    if (lane < kRG)
      for (int j = 0; j < nm; ++j) cm[(int64_t)(m0 + j) * kRG + lane] = narrow_to<T>(s_mul(sc[w][j][lane], sr));
    __syncwarp();
  }
}

// ------------------------------------------------- products over row groups
// accumulators of NR of a group's rows x V columns and one entry's update;
// m: a bit per row that holds the entry
template <typename T, int V, int NR> struct GAcc;
template <int V, int NR> struct GAcc<float, V, NR> {
  float2 y[NR / 2][V];  // rows 2p, 2p + 1
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int p = 0; p < NR / 2; ++p)
#pragma unroll
      for (int q = 0; q < V; ++q) y[p][q] = make_float2(0.f, 0.f);
  }
  __device__ __forceinline__ void add(const float* cf, const float (&x)[V], uint32_t m) {
    alignas(16) float2 a[NR / 2];
    ldv_s<float2, NR / 2>(reinterpret_cast<const float2*>(cf), a);
#pragma unroll
    for (int p = 0; p < NR / 2; ++p)
      if (m & (3u << (2 * p))) {
#pragma unroll
        for (int q = 0; q < V; ++q) y[p][q] = __ffma2_rn(a[p], make_float2(x[q], x[q]), y[p][q]);
      }
  }
  __device__ __forceinline__ float get(int r, int q) const { return (r & 1) ? y[r / 2][q].y : y[r / 2][q].x; }
};
template <int V, int NR> struct GAcc<cfloat, V, NR> {
  cfloat y[NR][V];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int r = 0; r < NR; ++r)
#pragma unroll
      for (int q = 0; q < V; ++q) y[r][q] = make_float2(0.f, 0.f);
  }
  __device__ __forceinline__ void add(const cfloat* cf, const cfloat (&x)[V], uint32_t) {
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      const cfloat a = cf[r];
#pragma unroll
      for (int q = 0; q < V; ++q)
        y[r][q] = __ffma2_rn(make_float2(a.x, a.x), x[q],
                             __ffma2_rn(make_float2(-a.y, a.y), make_float2(x[q].y, x[q].x), y[r][q]));
    }
  }
  __device__ __forceinline__ cfloat get(int r, int q) const { return y[r][q]; }
};

// the entries ub..ue of one group task against X rows col[u]: L lanes stage
// L entries at a time (offset, mask, the NR rows' coefficients of kRG) and
// gather 4 at once
template <typename T, int L, int V, int NR, bool MASK>
__device__ __forceinline__ void g_walk(GAcc<T, V, NR>& acc, int32_t ub, int32_t ue, const int32_t* __restrict__ col,
                                       const uint8_t* __restrict__ mask, const T* __restrict__ coef, int64_t k,
                                       const T* xl, bool on, int32_t* s_off, uint8_t* s_m, T* s_cf, int li,
                                       unsigned sub) {
  constexpr int U = 4;
  for (int32_t u0 = ub; u0 < ue; u0 += L) {
    const int cnt = min(L, ue - u0);
    const int cntp = (cnt + U - 1) / U * U;
    if (li < cntp) {  // padding repeats the last offset at coefficient 0 with an empty mask
      const int32_t u = u0 + min(li, cnt - 1);
      s_off[li] = col[u] * (int32_t)k;
      s_m[li] = li < cnt ? (MASK ? mask[u] : (uint8_t)0xff) : (uint8_t)0;
      alignas(16) T a[NR];
      if (li < cnt) {
        ldv<T, NR>(coef + (int64_t)u * kRG, a);
      } else {
#pragma unroll
        for (int r = 0; r < NR; ++r) a[r] = s_zero(T());
      }
      stv<T, NR>(s_cf + li * NR, a);
    }
    __syncwarp(sub);
    for (int j = 0; j < cntp; j += U) {
      alignas(16) int32_t oo[U];
      ldv_s<int32_t, U>(s_off + j, oo);
      const uint32_t m4 = *reinterpret_cast<const uint32_t*>(s_m + j);
      if (on) {
        alignas(16) T xv[U][V];
#pragma unroll
        for (int u = 0; u < U; ++u) ldv_w<T, V>(xl + (uint32_t)oo[u], xv[u]);
#pragma unroll
        for (int u = 0; u < U; ++u) acc.add(s_cf + (j + u) * NR, xv[u], (m4 >> (8 * u)) & 0xffu);
      }
    }
    __syncwarp(sub);
  }
}

#define RB_G_TASK(T, L, V, S)                                                                       \
  __shared__ __align__(16) int32_t s_off_[kBlk];                                                    \
  __shared__ __align__(16) uint8_t s_m_[kBlk];                                                      \
  __shared__ __align__(16) T s_cf_[kBlk * kRG];                                                     \
  const int li = threadIdx.x % L, sg = threadIdx.x / L;                                             \
  const unsigned sub = L == 32 ? 0xffffffffu : ((1u << (L & 31)) - 1u) << ((threadIdx.x & 31) / L * L); \
  int32_t* const s_off = s_off_ + sg * L;                                                           \
  uint8_t* const s_m = s_m_ + sg * L;                                                               \
  T* const s_cf = s_cf_ + sg * L * kRG;                                                             \
  const int64_t task0 = blockIdx.x * (int64_t)(kBlk / L) + sg, tasks = (int64_t)gridDim.x * (kBlk / L); \
  const int64_t c0 = (task0 % S) * (int64_t)(L * V) + (int64_t)li * V;                              \
  const bool on = c0 < k

// y = A^ x over the row groups, y stored, part += x.y (real, 65..128 columns;
// other layouts walk the scaled CSR rows).  MID also gives the group-level
// right-hand side f^ = S1 P1^T S^-1 (x - w y) from the rows in registers.
template <bool MID>
__global__ void __launch_bounds__(kBlk, 3)
vc_spmm_kernel(int64_t k, VcOp<float> o, const float* X, float* __restrict__ Y,
               double* __restrict__ part, const int32_t* live) {
  chain_wait();
  if (chain_dead(live)) return;
  constexpr int V = 4, L = 32;
  __shared__ double sm[kBlk * V];
  RB_G_TASK(float, L, V, 1);
  const float* const coef = reinterpret_cast<const float*>(o.rg.coef);
  const float w = MID ? o.par->w : 0.f;
  alignas(16) double acc[V];
#pragma unroll
  for (int q = 0; q < V; ++q) acc[q] = 0.0;
  for (int64_t g = task0; g < o.ng; g += tasks) {
    GAcc<float, V, kRG> y;
    y.clear();
    g_walk<float, L, V, kRG, true>(y, o.rg.uptr[g], o.rg.uptr[g + 1], o.rg.ucol, o.rg.umask, coef, k, X + c0, on,
                                   s_off, s_m, s_cf, li, sub);
    if (!on) continue;
    float fs[V];
#pragma unroll
    for (int q = 0; q < V; ++q) fs[q] = 0.f;
#pragma unroll
    for (int r = 0; r < kRG; ++r) {
      const int32_t row = o.rg.rows[g * kRG + r];
      if (row < 0) continue;
      alignas(16) float xv[V], yv[V];
      ldv_w<float, V>(X + (int64_t)row * k + c0, xv);
      const float is = MID ? o.is[row] : 0.f;
#pragma unroll
      for (int q = 0; q < V; ++q) {
        yv[q] = y.get(r, q);
        acc[q] = acc_fma(xv[q], yv[q], acc[q]);
        if (MID) fs[q] = fmaf(is, fmaf(-w, yv[q], xv[q]), fs[q]);
      }
      stv<float, V>(Y + (int64_t)row * k + c0, yv);
    }
    if (MID) {
      const float s1 = o.s1[g];
      alignas(16) float fv[V];
#pragma unroll
      for (int q = 0; q < V; ++q) fv[q] = s1 * fs[q];
      stv<float, V>(o.f + g * k + c0, fv);
    }
  }
  block_colreduce<double, L, V, 1>(acc, part, k, sm);
}

// f^ = S1 P1^T S^-1 (r - w t), a group per lane group (after a row-wise t)
template <typename T, int L, int S>
__global__ void __launch_bounds__(kBlk)
vc_restrict_kernel(int64_t k, VcOp<T> o, const T* R, const int32_t* live) {
  chain_wait();
  if (chain_dead(live)) return;
  constexpr int V = 16 / (int)sizeof(T);
  const int li = threadIdx.x % L;
  const int64_t task0 = blockIdx.x * (int64_t)(kBlk / L) + threadIdx.x / L, tasks = (int64_t)gridDim.x * (kBlk / L);
  const int64_t c0 = (task0 % S) * (int64_t)(L * V) + (int64_t)li * V;
  if (c0 >= k) return;
  const float w = o.par->w;
  for (int64_t task = task0; task < o.ng * S; task += tasks) {
    const int64_t g = task / S;
    const int32_t row0 = max(o.rg.rows[g * kRG], 0);  // (a group has at least one row, and its rows come first)
    alignas(16) T f[V];
#pragma unroll
    for (int q = 0; q < V; ++q) f[q] = s_zero(T());
#pragma unroll
    for (int h = 0; h < kRG; h += 4) {
      alignas(16) T rv[4][V], tv[4][V];
      T is[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int32_t row = o.rg.rows[g * kRG + h + r];
        // an empty slot repeats the group's first row at coefficient 0
        const int64_t at = (int64_t)(row >= 0 ? row : row0) * k + c0;
        ldv_w<T, V>(R + at, rv[r]);
        ldv_w<T, V>(o.t + at, tv[r]);
        const T s = o.is[row >= 0 ? row : row0];
        is[r] = row >= 0 ? s : s_zero(T());
      }
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int q = 0; q < V; ++q) f[q] = s_fma(is[r], s_sub(rv[r][q], r_mul(w, tv[r][q])), f[q]);
    }
    const T s1 = o.s1[g];
#pragma unroll
    for (int q = 0; q < V; ++q) f[q] = s_mul(s1, f[q]);
    stv<T, V>(o.f + g * k + c0, f);
  }
}

// x += alpha p, p = z + beta p with z = 2 w r - w^2 t + S^-1 P1 e - w S A P1 e
// (bound: HBM, six vector passes).  A lane group takes half a group: the four
// rows' r, t, p and x are all loaded before the walk over the neighbour
// groups' e rows (L2), 16 loads of 16 bytes in flight per lane.  With whole
// groups and the rows loaded one after another after the walk it took 0.327
// ms (real) and 0.881 ms (complex) at 520k nodes x 128 columns, now 0.323 (81%
// of the HBM rate) and 0.67.
constexpr int kPupRows = 4;
template <typename T, int L, int S>
__global__ void __launch_bounds__(kBlk, 2)
vc_pupdate_kernel(int64_t k, VcOp<T> o, const ColState* cs, const T* R, T* P, T* Xs) {
  chain_wait();
  constexpr int V = 16 / (int)sizeof(T), NR = kPupRows, H = kRG / NR;
  RB_G_TASK(T, L, V, S);
  T al[V], be[V];
  bool act[V], upd[V];
  int any = 0;
#pragma unroll
  for (int q = 0; q < V; ++q) {
    act[q] = on && cs[c0 + q].active;
    upd[q] = on && cs[c0 + q].upd;
    al[q] = upd[q] ? from_c<T>(cs[c0 + q].alpha) : s_zero(T());
    be[q] = act[q] ? from_c<T>(cs[c0 + q].beta) : s_zero(T());
    any |= (act[q] ? 1 : 0) | (upd[q] ? 2 : 0);
  }
  any = __reduce_or_sync(sub, any);  // of the lane group
  if (!any) return;
  const float w = o.par->w, w2 = o.par->w2;
  for (int64_t task = task0; task < o.ng * (H * S); task += tasks) {
    const int64_t gh = task / S, g = gh / H;
    const int h = (int)(gh - g * H) * NR;
    int32_t row[NR];
    alignas(16) T p[NR][V], x[NR][V], rv[NR][V], tv[NR][V], eg[V];
#pragma unroll
    for (int r = 0; r < NR; ++r) row[r] = o.rg.rows[g * kRG + h + r];
    if (row[0] < 0) continue;  // (rows of a short group come first)
    if (on) {
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        const int64_t at = (int64_t)max(row[r], 0) * k + c0;
        ldv_w<T, V>(P + at, p[r]);
        if (any & 2) ldv_w<T, V>(Xs + at, x[r]);
        if (any & 1) {
          ldv_w<T, V>(R + at, rv[r]);
          ldv_w<T, V>(o.t + at, tv[r]);
        }
      }
      if (any & 1) ldv_w<T, V>(o.e + g * k + c0, eg);
    }
    GAcc<T, V, NR> a;
    a.clear();
    if (any & 1)
      g_walk<T, L, V, NR, false>(a, o.mptr[g], o.mptr[g + 1], o.mcol, nullptr, o.cm + h, k, o.e + c0, on, s_off, s_m,
                                 s_cf, li, sub);
    if (!on) continue;
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      if (row[r] < 0) continue;
      const int64_t at = (int64_t)row[r] * k + c0;
      if (any & 2) {
#pragma unroll
        for (int q = 0; q < V; ++q)
          if (upd[q]) x[r][q] = s_fma(al[q], p[r][q], x[r][q]);
        stv<T, V>(Xs + at, x[r]);
      }
      if (any & 1) {
        const T is = o.is[row[r]];
#pragma unroll
        for (int q = 0; q < V; ++q)
          if (act[q]) {
            T z = s_sub(r_mul(2.f * w, rv[r][q]), r_mul(w2, tv[r][q]));
            z = s_fma(is, eg[q], s_sub(z, r_mul(w, a.get(r, q))));
            p[r][q] = s_fma(be[q], p[r][q], z);
          }
        stv<T, V>(P + at, p[r]);
      }
    }
  }
}

// r -= alpha q, part += |r|^2 and, for complex r, part_u += r.r unconjugated
// (INIT: the sums alone); rows in order
template <typename T, int L, int S, bool INIT>
__global__ void __launch_bounds__(kBlk, 4)
vc_update_kernel(int64_t n, int64_t k, const ColState* cs, T* R, const T* Q, double* __restrict__ part,
                 cdouble* __restrict__ part_u, const int32_t* live) {
  chain_wait();
  if (chain_dead(live)) return;
  constexpr int V = 16 / (int)sizeof(T);
  constexpr bool CX = Scalar<T>::is_complex;
  __shared__ double sm[kBlk * V];
  __shared__ cdouble smu[CX ? kBlk * V : 1];
  const int li = threadIdx.x % L;
  const int64_t task0 = blockIdx.x * (int64_t)(kBlk / L) + threadIdx.x / L, tasks = (int64_t)gridDim.x * (kBlk / L);
  const int64_t c0 = (task0 % S) * (int64_t)(L * V) + (int64_t)li * V;
  const bool on = c0 < k;
  T al[V];
  bool act[V];
#pragma unroll
  for (int q = 0; q < V; ++q) {
    act[q] = !INIT && on && cs[c0 + q].active;
    al[q] = act[q] ? from_c<T>(cs[c0 + q].alpha) : s_zero(T());
  }
  alignas(16) double acc[V];
  alignas(16) cdouble acu[V];
#pragma unroll
  for (int q = 0; q < V; ++q) {
    acc[q] = 0.0;
    acu[q] = make_double2(0.0, 0.0);
  }
  if (on) {
    // two rows at a time, all their loads before the first store
    for (int64_t task = task0; task < n * S; task += 2 * tasks) {
      const bool two = task + tasks < n * S;
      alignas(16) T r[2][V], q_[2][V];
#pragma unroll
      for (int u = 0; u < 2; ++u)
        if (u == 0 || two) {
          const int64_t at = (task + u * tasks) / S * k + c0;
          ldv_w<T, V>(R + at, r[u]);
          if (!INIT) ldv_w<T, V>(Q + at, q_[u]);
        }
#pragma unroll
      for (int u = 0; u < 2; ++u)
        if (u == 0 || two) {
          if (!INIT) {
#pragma unroll
            for (int q = 0; q < V; ++q)
              if (act[q]) r[u][q] = s_sub(r[u][q], s_mul(al[q], q_[u][q]));
            stv<T, V>(R + (task + u * tasks) / S * k + c0, r[u]);
          }
#pragma unroll
          for (int q = 0; q < V; ++q) {
            acc[q] += s_abs2(r[u][q]);
            if constexpr (CX) acu[q] = acc_fma(r[u][q], r[u][q], acu[q]);
          }
        }
    }
  }
  block_colreduce<double, L, V, S>(acc, part, k, sm);
  if constexpr (CX) block_colreduce<cdouble, L, V, S>(acu, part_u, k, smu);
}

// --------------------------------------------------------- the group level
// out = rowscale (cu U + cv W + cg A1^ G) on ng x k rows; DOT: part += (row
// before the scale) . F
template <typename T, int L, int S, bool DOT>
__global__ void __launch_bounds__(kBlk, 4)
vc_mid_spmm_kernel(int64_t k, VcOp<T> o, const T* U, const float* __restrict__ cu, const T* W,
                   const float* __restrict__ cw, const T* G, const float* __restrict__ cg,
                   const T* __restrict__ rowscale, T* __restrict__ out,
                   typename Scalar<T>::acc* __restrict__ part, const int32_t* live) {
  chain_wait();
  if (chain_dead(live)) return;
  constexpr int V = 16 / (int)sizeof(T);
  typedef typename Scalar<T>::acc A;
  __shared__ A sm[DOT ? kBlk * V : 1];
  const int li = threadIdx.x % L;
  const int64_t task0 = blockIdx.x * (int64_t)(kBlk / L) + threadIdx.x / L, tasks = (int64_t)gridDim.x * (kBlk / L);
  const int64_t c0 = (task0 % S) * (int64_t)(L * V) + (int64_t)li * V;
  const bool on = c0 < k;
  const float fu = *cu, fw = W ? *cw : 0.f, fg = *cg;
  alignas(16) A acc[V];
#pragma unroll
  for (int q = 0; q < V; ++q) acc[q] = acc_zero<A>();
  if (on) {
    for (int64_t task = task0; task < o.ng * S; task += tasks) {
      const int64_t g = task / S;
      const int32_t b = o.mptr[g], e = o.mptr[g + 1];
      alignas(16) T y[V], u[V];
#pragma unroll
      for (int q = 0; q < V; ++q) y[q] = s_zero(T());
      ldv_w<T, V>(U + g * k + c0, u);
#pragma unroll 4
      for (int32_t p = b; p < e; ++p) {
        const T a = o.v1[p];
        alignas(16) T x[V];
        ldv_w<T, V>(G + (int64_t)o.mcol[p] * k + c0, x);
#pragma unroll
        for (int q = 0; q < V; ++q) y[q] = s_fma(a, x[q], y[q]);
      }
#pragma unroll
      for (int q = 0; q < V; ++q) y[q] = s_add(r_mul(fg, y[q]), r_mul(fu, u[q]));
      if (W) {
        alignas(16) T v[V];
        ldv_w<T, V>(W + g * k + c0, v);
#pragma unroll
        for (int q = 0; q < V; ++q) y[q] = s_add(y[q], r_mul(fw, v[q]));
      }
      if (DOT) {
        alignas(16) T f[V];
        ldv_w<T, V>(o.f + g * k + c0, f);
#pragma unroll
        for (int q = 0; q < V; ++q) acc[q] = acc_fma(y[q], f[q], acc[q]);
      }
      if (rowscale) {
        const T s = rowscale[g];
#pragma unroll
        for (int q = 0; q < V; ++q) y[q] = s_mul(s, y[q]);
      }
      stv<T, V>(out + g * k + c0, y);
    }
  }
  if (DOT) block_colreduce<A, L, V, S>(acc, part, k, sm);
}

// x2 += S1^-1 P2 ec
template <typename T>
__global__ void vc_prolong_kernel(int64_t ng, int64_t k, const int32_t* __restrict__ agg, const T* ec,
                                  const T* __restrict__ is1, T* x2, const int32_t* live) {
  chain_wait();
  if (chain_dead(live)) return;
  constexpr int V = 16 / (int)sizeof(T);
  const int64_t kv = k / V;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < ng * kv; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t g = i / kv, c = (i - g * kv) * V;
    const T s = is1[g];
    alignas(16) T x[V], e[V];
    ldv_w<T, V>(x2 + g * k + c, x);
    ldv_w<T, V>(ec + (int64_t)agg[g] * k + c, e);
#pragma unroll
    for (int q = 0; q < V; ++q) x[q] = s_fma(s, e[q], x[q]);
    stv<T, V>(x2 + g * k + c, x);
  }
}

// ------------------------------------------------------------- finalizers
// after the update: ||r||^2, convergence; counts the columns that go on.
// ColState::pq keeps (r, r) unconjugated for the cycle's (r, z).
template <bool CX>
__device__ __forceinline__ cdouble vc_rru(int nb, const double* part, const cdouble* part_u, int64_t k, int64_t c,
                                          double& rr) {
  rr = block_sum_part<double>(part, nb, k, c).x;
  if constexpr (CX) return block_sum_part<cdouble>(part_u, nb, k, c);
  return make_double2(rr, 0.0);
}

// A column whose residual has grown to 1e8 of its start is beyond what FP32
// brings back: COCG can diverge on meshes with slivers (32,640 nodes x 128, tets
// of 1e-6 of the cube: 2000 iterations of one column up to 1e27 before the solve
// was handed to the two-level form).
constexpr double kVcDiverged = 1e16;  // of squared norms
template <bool CX>
__global__ void __launch_bounds__(kFinThreads)
vc_rr_kernel(int64_t k, int nb, const double* part, const cdouble* part_u, ColState* cs, double tol2,
             int32_t* nactive) {
  chain_wait();
  const int64_t c = blockIdx.x;
  if (c >= k || !cs[c].active) return;  // uniform over the block
  double rr;
  const cdouble u = vc_rru<CX>(nb, part, part_u, k, c, rr);
  if (threadIdx.x) return;
  ColState s = cs[c];
  s.iters += 1;
  s.rr = rr;
  s.pq = u;
  if (!(rr <= kVcDiverged * s.rr0)) {  // (or not finite)
    s.active = 0;
    s.status = 2;
  } else if (rr <= (s.tol2 >= 0.0 ? s.tol2 : tol2) * s.rr0) {
    s.active = 0;
  }
  cs[c] = s;
  if (s.active) atomicAdd(nactive, 1);
}

// before the first iteration of a sweep
template <bool CX>
__global__ void __launch_bounds__(kFinThreads)
vc_start_kernel(int64_t k, int nb, const double* part, const cdouble* part_u, ColState* cs,
                const OuterState* __restrict__ os, int32_t* nactive) {
  chain_wait();
  const int64_t c = blockIdx.x;
  if (c >= k) return;
  double rr;
  const cdouble u = vc_rru<CX>(nb, part, part_u, k, c, rr);
  if (threadIdx.x) return;
  ColState s = cs[c];
  s.rr = s.rr0 = rr;
  s.pq = u;
  s.rz = s.alpha = s.beta = make_double2(0, 0);
  s.active = rr > 0.0;
  s.status = 0;
  s.iters = 0;
  s.upd = 0;
  s.tol2 = os[c].itol2;
  cs[c] = s;
  if (s.active) atomicAdd(nactive, 1);
}

// (r, z) = 2 w (r, r) - w^2 (r, t) + (e, f) and beta (first: no beta)
template <typename A>
__global__ void __launch_bounds__(kFinThreads)
vc_beta_kernel(int64_t k, int nbt, const A* part_t, int nbe, const A* part_e, const VcPar* __restrict__ par,
               ColState* cs, int first, int32_t* nactive) {
  chain_wait();
  const int64_t c = blockIdx.x;
  if (c >= k || !cs[c].active) return;  // uniform over the block
  const cdouble rt = block_sum_part<A>(part_t, nbt, k, c), ef = block_sum_part<A>(part_e, nbe, k, c);
  if (threadIdx.x) return;
  ColState s = cs[c];
  const double w = par->w, w2 = par->w2;
  const cdouble rz = make_double2(2.0 * w * s.pq.x - w2 * rt.x + ef.x, 2.0 * w * s.pq.y - w2 * rt.y + ef.y);
  if (!finite_c(rz) || (!first && s.rz.x == 0.0 && s.rz.y == 0.0)) {
    s.active = 0;
    s.status = 2;
    atomicSub(nactive, 1);
  } else {
    if (!first) s.beta = cdiv(rz, s.rz);
    s.rz = rz;
  }
  cs[c] = s;
}

// ------------------------------------------------ scaled residual, correction
// Column factors: scale or its reciprocal, 0 where not active (one division
// per block and column instead of one per entry).  With stacked instances
// they are per (instance, column), read from a table made for the sweep.
template <bool INV>
__device__ __forceinline__ double vc_factor(const OuterState& o) { return o.active ? (INV ? 1.0 / o.scale : o.scale) : 0.0; }
template <bool INV>
__device__ __forceinline__ void vc_factors(int64_t k, const OuterState* __restrict__ os, double* f) {
  for (int c = threadIdx.x; c < k; c += blockDim.x) f[c] = vc_factor<INV>(os[c]);
  __syncthreads();
}

// factors of every (instance, column): fac[j] the scale, fac[m + j] its reciprocal
__global__ void vc_seg_factor_kernel(int64_t m, const OuterState* __restrict__ seg, double* __restrict__ fac) {
  const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (j >= m) return;
  fac[j] = vc_factor<false>(seg[j]);
  fac[m + j] = vc_factor<true>(seg[j]);
}

// r^ = T(S R64 scale) for active columns, 0 elsewhere; x = p = 0.  RT: the
// residual's type (double for the right-hand side of a first sweep from 0,
// the caller's array: read in 16-byte loads only where it lies on 16 bytes);
// rinst / segf: the rows' instances and their factors, or NULL
template <typename T64, typename RT, typename T>
__global__ void __launch_bounds__(256)
vc_cast_kernel(int64_t n, int64_t k, const RT* __restrict__ R64, const T64* __restrict__ s64,
               const OuterState* __restrict__ os, const int32_t* __restrict__ rinst, const double* __restrict__ segf,
               T* __restrict__ R, T* __restrict__ P, T* __restrict__ Xs) {
  constexpr int V = 16 / (int)sizeof(T);
  __shared__ double fac[kMaxCols];
  if (!rinst) vc_factors<false>(k, os, fac);
  const bool wide = (reinterpret_cast<uintptr_t>(R64) & 15) == 0;
  const int64_t kv = k / V;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n * kv; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t row = i / kv, c = (i - row * kv) * V;
    const double* f = rinst ? segf + (int64_t)rinst[row] * k + c : fac + c;
    const T64 s = s64[row];
    alignas(16) RT v[V];
    alignas(16) T o[V], z[V];
    if (wide) {
      ldv<RT, V>(R64 + row * k + c, v);
    } else {
#pragma unroll
      for (int q = 0; q < V; ++q) v[q] = R64[row * k + c + q];
    }
#pragma unroll
    for (int q = 0; q < V; ++q) {
      const double fq = f[q];  // (a done column's residual may be non-finite: 0, not 0 x it)
      o[q] = fq != 0.0 ? narrow_to<T>(r_mul(fq, cs_mul(s, v[q]))) : s_zero(T());
      z[q] = s_zero(T());
    }
    stv<T, V>(R + row * k + c, o);
    stv<T, V>(P + row * k + c, z);
    stv<T, V>(Xs + row * k + c, z);
  }
}

// X64 += S x^ / scale for active columns
template <typename T64, typename T>
__global__ void __launch_bounds__(256)
vc_correct_kernel(int64_t n, int64_t k, const T* __restrict__ D, const T64* __restrict__ s64,
                  const OuterState* __restrict__ os, const int32_t* __restrict__ rinst,
                  const double* __restrict__ segf, T64* __restrict__ X) {
  constexpr int V = 16 / (int)sizeof(T);
  __shared__ double fac[kMaxCols];
  if (!rinst) vc_factors<true>(k, os, fac);
  const int64_t kv = k / V;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n * kv; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t row = i / kv, c = (i - row * kv) * V;
    const double* f = rinst ? segf + (int64_t)rinst[row] * k + c : fac + c;
    const T64 s = s64[row];
    alignas(16) T64 x[V];
    alignas(16) T d[V];
    T64* const xp = X + row * k + c;
#pragma unroll
    for (int q = 0; q < V; ++q) x[q] = xp[q];
    ldv<T, V>(D + row * k + c, d);
#pragma unroll
    for (int q = 0; q < V; ++q) {
      const double fq = f[q];
      if (fq != 0.0) x[q] = s_add(x[q], r_mul(fq, s_mul(s, widen(d[q]))));
    }
    stv<T64, V>(xp, x);
  }
}

// ------------------------------------------------------------- host side
struct VcGrids {
  GShape sh;
  unsigned grp, half, row, mid, pro;  // blocks of the group, half-group, row and group-row kernels
};
template <typename T>
static VcGrids vc_grids(int64_t n, int64_t ng, int64_t k) {
  VcGrids g;
  g.sh = vc_shape<T>(k);
  const int64_t per = kBlk / g.sh.L;
  auto cap = [&](int64_t rows, int64_t bps) {
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>({num_sms() * bps, ceil_div(rows * g.sh.S, per), kGridMax}));
  };
  g.grp = cap(ng, 3);
  g.half = cap(ng * (kRG / kPupRows), 2);
  g.row = cap(n, 4);
  g.mid = cap(ng, 4);
  g.pro = (unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(ng * k * (int64_t)sizeof(T) / 16, 256), 148 * 16));
  return g;
}

// the matrix-dependent part: scaled values, group-level matrix, its dense inverse
template <typename T64, typename T>
static int vc_setup(const rb_csr& A, const rb_midlevel& mid, VcBufs<T64, T>& b, bool groups, cudaStream_t st) {
  VcOp<T>& o = b.op;
  const T64* val = (const T64*)A.val64;
  const T64* dinv = (const T64*)A.dinv64;
  const unsigned gn = (unsigned)std::min<int64_t>(ceil_div(A.n, 256), 148 * 16);
  const unsigned gg = (unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(o.ng, 256), 148 * 16));
  RB_CUDA_TRY(cudaMemsetAsync(o.par, 0, sizeof(VcPar), st));
  vc_scale_kernel<T64, T><<<gn, 256, 0, st>>>(A.n, dinv, b.s64, o.s, o.is);
  vc_values_kernel<T64, T><<<(unsigned)std::min<int64_t>(ceil_div(A.n, 16), 148 * 32), 256, 0, st>>>(
      A.n, A.indptr, A.indices, val, dinv, b.s64, o.vs, &o.par->g[0]);
  RB_LAUNCH_CHECK();
  if (groups) RB_TRY(rg_fill_coef<T>(A, o.vs, o.rg, st));  // (read by vc_spmm_kernel alone)
  vc_mid_kernel<T64, T><<<(unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(o.ng, kMidWarps), 148 * 64)),
                          kMidWarps * 32, 0, st>>>(o.ng, o.rg.rows, A.indptr, A.indices, val, mid.grp, o.mptr, o.mcol,
                                                   b.s64, b.val1, o.cm);
  csr_prepare_kernel<T64, T><<<gg, 256, 0, st>>>(o.ng, o.mptr, o.mcol, b.val1, (T*)nullptr, b.d64_1, (T*)nullptr);
  vc_scale_kernel<T64, T><<<gg, 256, 0, st>>>(o.ng, b.d64_1, b.s64_1, o.s1, o.is1);
  vc_values_kernel<T64, T><<<(unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(o.ng, 16), 148 * 32)), 256, 0, st>>>(
      o.ng, o.mptr, o.mcol, b.val1, b.d64_1, b.s64_1, o.v1, &o.par->g[1]);
  vc_param_kernel<<<1, 1, 0, st>>>(o.par);
  RB_LAUNCH_CHECK();
  rb_csr A1 = A;
  A1.n = o.ng;
  A1.nnz = b.nnz1;
  A1.indptr = o.mptr;
  A1.indices = o.mcol;
  A1.val64 = b.val1;
  A1.val32 = nullptr;
  A1.dinv64 = A1.dinv32 = nullptr;
  RB_TRY((coarse_setup<T64, T>(A1, b.cb, st)));
  o.co = b.cb.op;
  return RB_OK;
}

// The product of a cycle solve: y = A^ x, part = x.y.  Real solves of 65-128
// columns walk the row groups (0.200 against 0.229 ms for row pairs at 520k
// nodes x 128).  Narrower ones walk rows: a group is one long chain of gathers
// and there are too few of them (67,626 nodes x 64: 20.2 against 15.8 us).
// Complex ones walk row pairs (128 columns) or rows: a complex group's
// products are bound by their instructions (0.97 against 0.50 ms).
template <typename T>
static bool vc_groups(const VcGrids& g) { return std::is_same<T, float>::value && g.sh.L == 32; }
template <typename T>
static int vc_spmm(const rb_csr& A, const VcOp<T>& o, const VcGrids& g, const GroupPlan* gp, bool mid, const T* X, T* Y,
                   void* part, int64_t k, unsigned* nb, cudaStream_t st, const int32_t* live) {
  if constexpr (std::is_same<T, float>::value) {
    if (vc_groups<T>(g)) {
      *nb = g.grp;
      if (mid) RB_CUDA_TRY(launch_early(true, vc_spmm_kernel<true>, dim3(g.grp), dim3(kBlk), st, k, o, X, Y, (double*)part, live));
      else RB_CUDA_TRY(launch_early(true, vc_spmm_kernel<false>, dim3(g.grp), dim3(kBlk), st, k, o, X, Y, (double*)part, live));
      return RB_OK;
    }
  }
  if (gp) return spmm_pair<T, EPI_PQDOT>(A, o.vs, *gp, X, Y, part, k, nb, st, live, true);
  const Shape sh = pick_spmm_shape<T>(A.n, k);
  *nb = sh.grid;
  return spmm_t<T, EPI_PQDOT>(A, o.vs, X, Y, nullptr, part, k, sh, st, live, true);
}

// t = A^ r, f, then e = M1 f with (e, f): all but the p-update of one cycle
template <typename T>
static int vc_apply(const rb_csr& A, const VcOp<T>& o, const VcGrids& g, const GroupPlan* gp, const T* R, void* part_t,
                    int64_t k, unsigned* nbt, cudaStream_t st, const int32_t* live, int* launches) {
  typedef typename Scalar<T>::acc Acc;
  const VcPar* p = o.par;
  RB_TRY(vc_spmm<T>(A, o, g, gp, true, R, o.t, part_t, k, nbt, st, live));
  if (!vc_groups<T>(g)) {
#define RB_VR(L_, S_) \
  RB_CUDA_TRY(launch_early(true, vc_restrict_kernel<T, L_, S_>, dim3(g.mid), dim3(kBlk), st, k, o, R, live))
    RB_DISPATCH_G(g.sh, RB_VR);
#undef RB_VR
    *launches += 1;
  }
#define RB_VM1(L_, S_, DOT_, ...) \
  RB_CUDA_TRY(launch_early(true, vc_mid_spmm_kernel<T, L_, S_, DOT_>, dim3(g.mid), dim3(kBlk), st, k, o, __VA_ARGS__, live))
#define RB_VM(L_, S_)                                                                                              \
  RB_VM1(L_, S_, false, o.f, &p->a, nullptr, nullptr, o.f, &p->nb, nullptr, o.x2, nullptr);                        \
  RB_VM1(L_, S_, false, o.f, &p->one, nullptr, nullptr, o.x2, &p->mone, o.is1, o.w, nullptr)
  RB_DISPATCH_G(g.sh, RB_VM);
#undef RB_VM
  RB_TRY(coarse_apply<T>(o.co, o.w, k, st, live, true));
  RB_CUDA_TRY(launch_early(true, vc_prolong_kernel<T>, dim3(g.pro), dim3(256), st, o.ng, k, o.co.agg, o.co.ec, o.is1,
                           o.x2, live));
#define RB_VM(L_, S_)                                                                                              \
  RB_VM1(L_, S_, false, o.f, &p->one, nullptr, nullptr, o.x2, &p->mone, nullptr, o.w, nullptr);                    \
  RB_VM1(L_, S_, true, o.x2, &p->one, o.w, &p->a, o.w, &p->nb, o.s1, o.e, (Acc*)o.part_c)
  RB_DISPATCH_G(g.sh, RB_VM);
#undef RB_VM
#undef RB_VM1
  *launches += 9;
  return RB_OK;
}

// One correction sweep: x^ (Xs) from the scaled residual in R.
template <typename T64, typename T>
static int vc_inner(const rb_csr& A, const VcOp<T>& o, int64_t k, void* part_a, double* part_b, T* Xs, T* R, T* P,
                    T* Q, ColState* cs, const OuterState* os, int32_t* counter, double tol, int maxiter,
                    const GroupPlan* gp, int* iters_out, int* launches, KernelTimer& tm, cudaStream_t st) {
  typedef typename Scalar<T>::acc Acc;
  constexpr bool CX = Scalar<T>::is_complex;
  const VcGrids g = vc_grids<T>(A.n, o.ng, k);
  // live counts, one of four words per iteration: iteration i fills word i % 4,
  // which iteration i + 1 reads and iteration i + 4 clears
  int32_t* const slot = counter + 4;
  RB_CUDA_TRY(cudaMemsetAsync(slot + 3, 0, sizeof(int32_t), st));
#define RB_VU(L_, S_)                                                                                                vc_update_kernel<T, L_, S_, true><<<g.row, kBlk, 0, st>>>(A.n, k, cs, R, Q, part_b, (cdouble*)part_a, nullptr)
  RB_DISPATCH_G(g.sh, RB_VU);
#undef RB_VU
  vc_start_kernel<CX><<<(unsigned)k, kFinThreads, 0, st>>>(k, (int)g.row, part_b, (cdouble*)part_a, cs, os, slot + 3);
  RB_LAUNCH_CHECK();
  auto precondition = [&](int first, int32_t* live) -> int {
    unsigned nbt = 0;
    RB_TRY(vc_apply<T>(A, o, g, gp, R, part_a, k, &nbt, st, live, launches));
    RB_CUDA_TRY(launch_early(true, vc_beta_kernel<Acc>, dim3((unsigned)k), dim3(kFinThreads), st, k, (int)nbt,
                             (const Acc*)part_a, (int)g.mid, (const Acc*)o.part_c, o.par, cs, first, live));
#define RB_VP(L_, S_) \
  RB_CUDA_TRY(launch_early(true, vc_pupdate_kernel<T, L_, S_>, dim3(g.half), dim3(kBlk), st, k, o, cs, R, P, Xs))
    RB_DISPATCH_G(g.sh, RB_VP);
#undef RB_VP
    *launches += 2;
    return RB_OK;
  };
  RB_TRY(precondition(1, slot + 3));
  *launches += 2;
  // Every iteration is a handful of launches, so the host looks at the live
  // count of each, one iteration behind the one it has queued (BurstSync).
  BurstSync bs;
  RB_TRY(bs.init());
  int it = 0;
  while (it < maxiter) {
    const int32_t* live = slot + ((it + 3) & 3);
    int32_t* next = slot + (it & 3);
    RB_TRY(tm.record(st));
    unsigned nb = 0;
    RB_TRY(vc_spmm<T>(A, o, g, gp, false, P, Q, part_a, k, &nb, st, live));
    RB_TRY(tm.record(st));
    RB_CUDA_TRY(launch_early(true, fin_alpha_kernel<Acc>, dim3((unsigned)k), dim3(kFinThreads), st, k, (int)nb,
                             (const Acc*)part_a, cs, next));
#define RB_VU(L_, S_)                                                                                        \
  RB_CUDA_TRY(launch_early(true, vc_update_kernel<T, L_, S_, false>, dim3(g.row), dim3(kBlk), st, A.n, k, cs, R, Q, \
                           part_b, (cdouble*)part_a, live))
    RB_DISPATCH_G(g.sh, RB_VU);
#undef RB_VU
    RB_TRY(tm.record(st));
    RB_CUDA_TRY(launch_early(true, vc_rr_kernel<CX>, dim3((unsigned)k), dim3(kFinThreads), st, k, (int)g.row,
                             (const double*)part_b, (const cdouble*)part_a, cs, tol * tol, next));
    RB_TRY(precondition(0, next));
    RB_TRY(tm.record(st));
    *launches += 4;
    RB_CUDA_TRY(cudaEventRecord(bs.ev[it & 1], st));
    // (BurstSync::read takes a base that its event's number is added to)
    auto count = [&](int i, int32_t* v) { return bs.read(i & 1, slot + (i & 3) - (i & 1), v); };
    int32_t v = 1;
    ++it;
    if (tm.on) {
      RB_TRY(count(it - 1, &v));
      RB_TRY(tm.harvest());
      if (v == 0) break;
      continue;
    }
    if (it > 1) {
      RB_TRY(count(it - 2, &v));
      if (v == 0) {
        --it;  // the iteration queued after the last one was a no-op
        break;
      }
    }
  }
  *iters_out = it;
  return RB_OK;
}

}  // namespace rb
