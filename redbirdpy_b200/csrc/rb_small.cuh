// Whole mixed-precision solve of a small system in one launch (included by
// rb_krylov.cu): FP64 refinement around FP32 (complex64) Jacobi CG / COCG,
// the same rules as solve_block, with every decision taken on the device.
//
// The columns of a block solve are independent Krylov problems, so a cluster
// of CL blocks takes V columns from the right-hand side to the solution and
// never talks to another cluster.  Block r of a cluster owns a run of nr rows:
// their matrix entries stay in its shared memory for the whole solve (what
// does not fit is streamed from L2), the vector entries in its registers (a
// thread owns RPT rows), and z, the vector that the product gathers, in
// shared memory, read by the other blocks through distributed shared memory.
//
// What bounds a small solve is neither bytes nor flops but the steps that
// wait for one another: as separate kernels an iteration was five launches of
// 2-3 us (12 us of GPU time at 1-12k nodes) and the host's launch rate on
// top.  Here it is two cluster barriers: the recurrence takes both products
// of an iteration ((r, z) and (A z, z)) in one reduction (Chronopoulos and
// Gear, J. Comput. Appl. Math. 25, 1989):
//   z = D^-1 r; w = A z; g = (r, z), d = (w, z); beta = g / g_old;
//   alpha = g / (d - beta g / alpha_old); p = z + beta p; s = w + beta s;
//   x += alpha p; r -= alpha s.
// Measured (solve alone, separate kernels -> this): 1,183 nodes x 3 columns
// 2.57 -> 0.30 ms; 3,927 x 12 complex 4.93 -> 0.58; 11,284 x 24 5.48 -> 1.29;
// 12,555 x 22 complex (its matrix 1.4 times the shared memory of 8 blocks)
// 6.07 -> 2.58.  An iteration of the smallest is 3.5 us, nearly all of it the
// two barriers, the reduction and the scalars.
#pragma once

#include <atomic>

namespace rb {

constexpr int kSmThreads = 512;
constexpr int kSmWarps = kSmThreads / 32;
constexpr int kSmMaxCl = 16;
constexpr int kSmLocalBits = 12;  // an entry's column: rank << 12 | row within the rank's run

struct SmallOut {  // per column
  double relres;
  int32_t done;    // OuterState::done
  int32_t status;  // ColState::status of the last sweep
  int32_t outer, iters, sweep_max;
  int32_t pad;
};

template <typename T64, typename T>
struct SmallArgs {
  int32_t n, k, nr, cap;  // rows, columns, rows per block, entries that fit a block's shared memory
  const int32_t* indptr;
  const int32_t* indices;
  const T64* val64;
  const T* val;
  const T* dinv;
  const int32_t* soff;  // sliced matrix (small_slice_kernel): per rank kSmWarps * rpt + 1 slice offsets
  const T* sval;        // entries, slots per rank
  const uint16_t* scol;
  int32_t slots;
  const double* B;
  T64* X;
  double tol, inner_tol, itol_min, stall;
  int32_t maxiter, max_outer, use_x0;
  int32_t itcap;  // iterations of a column in all
  SmallOut* out;
};
// Complex columns stop after this many iterations (boxes and well-shaped
// unstructured meshes take 100 to 350).  On meshes with slivers the one-reduction
// COCG in FP32 needs up to ten times the iterations of the two-reduction form:
// 12,672 nodes x 16 (Delaunay, tets of 1e-6 of the cube) ended unconverged after
// 211 ms where the separate kernels take 90; real CG needs as many as theirs.
constexpr int kSmComplexCap = 600;

__device__ __forceinline__ uint32_t cl_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ uint32_t cl_size() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ uint32_t cl_id() { uint32_t r; asm volatile("mov.u32 %0, %%clusterid.x;" : "=r"(r)); return r; }
// all threads of all blocks of the cluster; orders shared and global writes
// before it with reads after it, cluster-wide
__device__ __forceinline__ void cl_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cl_map(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cl_st(uint32_t addr, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}
// NB bytes (4, 8, 16 or 32) from distributed shared memory
template <int NB>
__device__ __forceinline__ void cl_ld(uint32_t addr, void* o_) {
  uint32_t* o = reinterpret_cast<uint32_t*>(o_);
  if constexpr (NB == 4) {
    asm volatile("ld.shared::cluster.b32 %0, [%1];" : "=r"(o[0]) : "r"(addr) : "memory");
  } else if constexpr (NB == 8) {
    asm volatile("ld.shared::cluster.v2.b32 {%0, %1}, [%2];" : "=r"(o[0]), "=r"(o[1]) : "r"(addr) : "memory");
  } else {
#pragma unroll
    for (int j = 0; j < NB / 16; ++j)
      asm volatile("ld.shared::cluster.v4.b32 {%0, %1, %2, %3}, [%4];"
                   : "=r"(o[4 * j]), "=r"(o[4 * j + 1]), "=r"(o[4 * j + 2]), "=r"(o[4 * j + 3])
                   : "r"(addr + 16 * j)
                   : "memory");
  }
}

// the same from the block's own shared memory
template <int NB>
__device__ __forceinline__ void sm_ld(uint32_t addr, void* o_) {
  uint32_t* o = reinterpret_cast<uint32_t*>(o_);
  if constexpr (NB == 4) {
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(o[0]) : "r"(addr) : "memory");
  } else if constexpr (NB == 8) {
    asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(o[0]), "=r"(o[1]) : "r"(addr) : "memory");
  } else {
#pragma unroll
    for (int j = 0; j < NB / 16; ++j)
      asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                   : "=r"(o[4 * j]), "=r"(o[4 * j + 1]), "=r"(o[4 * j + 2]), "=r"(o[4 * j + 3])
                   : "r"(addr + 16 * j)
                   : "memory");
  }
}

// Sum of each of the lanes' N values over the warp: the exchange halves the
// values a lane carries at each of the first log2(N) steps (N shuffles in all
// instead of 5 N); value i ends in every lane l with (l >> (5 - log2 N)) == i.
template <int N>
__device__ __forceinline__ double warp_sum_n(double (&v)[N]) {
  const int lane = threadIdx.x & 31;
  int o = 16;
#pragma unroll
  for (int h = N / 2; h > 0; h >>= 1, o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < h; ++i) {
      const double send = up ? v[i] : v[i + h], keep = up ? v[i + h] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  double s = v[0];
  for (; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

constexpr int sm_pow2(int n) { return n <= 1 ? 1 : n <= 2 ? 2 : n <= 4 ? 4 : n <= 8 ? 8 : n <= 16 ? 16 : 32; }

// values of one cluster reduction: per column (r, z), (w, z) and ||r||^2
template <typename T> constexpr int sm_nval(int V) { return V * (Scalar<T>::is_complex ? 5 : 3); }

template <int NV>
struct SmRed {
  double warp[kSmWarps][NV];
  double slot[2][kSmMaxCl][NV];  // by parity of the reduction and rank
  double tot[NV];
};

// Cluster-wide sums of NV values per thread; tot is valid in every thread
// after it (ends with a block barrier).  Every block adds the same partials in
// the same order, so all blocks hold the same bits and decide alike.
template <int NV>
__device__ __forceinline__ void sm_reduce(const double (&v)[NV], SmRed<NV>& red, int& par, uint32_t rank,
                                          uint32_t cl) {
  constexpr int P = sm_pow2(NV), SH = 5 - (P == 1 ? 0 : P == 2 ? 1 : P == 4 ? 2 : P == 8 ? 3 : P == 16 ? 4 : 5);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  double t[P];
#pragma unroll
  for (int i = 0; i < P; ++i) t[i] = i < NV ? v[i] : 0.0;
  const double s = warp_sum_n<P>(t);
  const int i = lane >> SH;
  if ((lane & ((1 << SH) - 1)) == 0 && i < NV) red.warp[w][i] = s;
  __syncthreads();
  for (int q = threadIdx.x; q < NV * (int)cl; q += kSmThreads) {
    const int j = q % NV, dst = q / NV;
    double a = 0.0;
#pragma unroll
    for (int x = 0; x < kSmWarps; ++x) a += red.warp[x][j];
    cl_st(cl_map(smem_u32(&red.slot[par][rank][j]), dst), a);
  }
  cl_sync();
  if (threadIdx.x < NV) {
    double a = 0.0;
    for (uint32_t r = 0; r < cl; ++r) a += red.slot[par][r][threadIdx.x];
    red.tot[threadIdx.x] = a;
  }
  __syncthreads();
  par ^= 1;
}

__device__ __forceinline__ cdouble cmul(cdouble a, cdouble b) { return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
template <typename T> __device__ __forceinline__ T ldcg_t(const T* p) { return __ldcg(p); }

// per-column scalars of a cluster, the same in each of its blocks
template <typename T>
struct SmCol {
  double bnorm, relres, prev, scale, itol2, rr0;
  cdouble g, den;         // (r, z) and its alpha's divisor
  cdouble igam, ialpha;   // 1 / (r, z) and 1 / alpha = den / (r, z) of the last iteration
  T be, al;        // of the current iteration
  int32_t open;    // refinement goes on
  int32_t active;  // inner sweep goes on
  int32_t done, status, iters, outer, sweep_max, it_sweep;
};

// The matrix in slices of 32 rows, entry-major, one run per rank of a cluster:
// rank r's thread t owns the rows r nr + s kSmThreads + t, slice q = s
// kSmWarps + w is warp w's 32 rows of pass s, entry j of a row at soff[q] +
// 32 j + lane (a warp's reads are contiguous).  Short rows are padded with
// their own column at coefficient 0.  A column is stored as rank << 12 | row
// within the rank's run.  Slices that do not fit the rank's slots are left out
// (their offset ends beyond `slots`) and read from the CSR arrays.
template <typename T>
__global__ void __launch_bounds__(kSmThreads)
small_slice_kernel(int32_t n, int32_t nr, int32_t rpt, int32_t slots, const int32_t* __restrict__ indptr,
                   const int32_t* __restrict__ indices, const T* __restrict__ val, int32_t* __restrict__ soff,
                   T* __restrict__ sval, uint16_t* __restrict__ scol) {
  __shared__ int32_t off[kSmWarps * 4 + 1];
  const int rank = blockIdx.x, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int row0 = min(n, rank * nr), rows = min(n, row0 + nr) - row0, ns = kSmWarps * rpt;
  for (int s = 0; s < rpt; ++s) {
    const int i = s * kSmThreads + tid;
    const int len = i < rows ? indptr[row0 + i + 1] - indptr[row0 + i] : 0;
    const int m = __reduce_max_sync(0xffffffffu, len);
    if (lane == 0) off[s * kSmWarps + w + 1] = m;
  }
  if (tid == 0) off[0] = 0;
  __syncthreads();
  if (tid == 0)
    for (int q = 0; q < ns; ++q) off[q + 1] = min(slots + 1 - off[q], 32 * off[q + 1]) + off[q];  // no overflow
  __syncthreads();
  for (int q = tid; q <= ns; q += kSmThreads) soff[rank * (ns + 1) + q] = off[q];
  sval += (int64_t)rank * slots;
  scol += (int64_t)rank * slots;
  for (int s = 0; s < rpt; ++s) {
    const int i = s * kSmThreads + tid, q = s * kSmWarps + w;
    if (off[q + 1] > slots) continue;
    const int beg = i < rows ? indptr[row0 + i] : 0, len = i < rows ? indptr[row0 + i + 1] - beg : 0;
    const int o = off[q], m = (off[q + 1] - o) / 32;
    for (int j = 0; j < m; ++j) {
      T v = s_zero(T());
      uint32_t c = ((uint32_t)rank << kSmLocalBits) | (uint32_t)min(i, nr - 1);
      if (j < len) {
        v = val[beg + j];
        const int g = indices[beg + j], rk = g / nr;
        c = ((uint32_t)rk << kSmLocalBits) | (uint32_t)(g - rk * nr);
      }
      sval[o + 32 * j + lane] = v;
      scol[o + 32 * j + lane] = (uint16_t)c;
    }
  }
}

template <typename T64, typename T, int V, int RPT>
__global__ void __launch_bounds__(kSmThreads, 1) small_solve_kernel(SmallArgs<T64, T> a) {
  constexpr bool CX = Scalar<T>::is_complex;
  constexpr int NV = sm_nval<T>(V);
  typedef typename Scalar<T>::acc Acc;
  extern __shared__ __align__(16) unsigned char sm_raw[];
  __shared__ SmRed<NV> red;
  __shared__ SmCol<T> col[V];
  __shared__ int32_t s_off[kSmWarps * RPT + 1];  // entry offset of each 32-row slice
  __shared__ int32_t s_run, s_any;
  const uint32_t rank = cl_rank(), cl = cl_size();
  const int c0 = (int)cl_id() * V;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int n = a.n, nr = a.nr, k = a.k;
  const int row0 = min(n, (int)rank * nr), rows = min(n, row0 + nr) - row0;
  T* const z = reinterpret_cast<T*>(sm_raw);  // nr x V
  T* const ev = reinterpret_cast<T*>(sm_raw + ((size_t)nr * V * sizeof(T) + 15) / 16 * 16);
  uint16_t* const ec = reinterpret_cast<uint16_t*>(ev + a.cap);
  const uint32_t zaddr = smem_u32(z);
  int par = 0;

  // ---- the block's rows: the first slices into shared memory, as many as fit
  int32_t len[RPT], beg[RPT];
  T dinv[RPT];
#pragma unroll
  for (int s = 0; s < RPT; ++s) {
    const int i = s * kSmThreads + tid;
    beg[s] = i < rows ? a.indptr[row0 + i] : 0;
    len[s] = i < rows ? a.indptr[row0 + i + 1] - beg[s] : 0;
    dinv[s] = i < rows ? a.dinv[row0 + i] : s_zero(T());
  }
  for (int q = tid; q <= kSmWarps * RPT; q += kSmThreads) s_off[q] = a.soff[rank * (kSmWarps * RPT + 1) + q];
  __syncthreads();
  const T* const gv = a.sval + (int64_t)rank * a.slots;
  const uint16_t* const gc = a.scol + (int64_t)rank * a.slots;
  {
    int q = kSmWarps * RPT;
    while (q > 0 && s_off[q] > min(a.cap, a.slots)) --q;
    for (int j = tid; j < s_off[q]; j += kSmThreads) {
      ev[j] = gv[j];
      ec[j] = gc[j];
    }
  }

  // ---- ||b|| and the starting state
  double v[NV];
#pragma unroll
  for (int j = 0; j < NV; ++j) v[j] = 0.0;
#pragma unroll
  for (int s = 0; s < RPT; ++s) {
    const int i = s * kSmThreads + tid;
    if (i < rows)
#pragma unroll
      for (int q = 0; q < V; ++q)
        if (c0 + q < k) {
          const double b = a.B[(int64_t)(row0 + i) * k + c0 + q];
          v[q] += b * b;
          if (!a.use_x0) a.X[(int64_t)(row0 + i) * k + c0 + q] = s_zero(T64());
        }
  }
  cl_sync();  // every block of the cluster runs before its shared memory is written
  sm_reduce<NV>(v, red, par, rank, cl);
  if (tid < V) {
    const OuterState o = outer_start(red.tot[tid]);
    SmCol<T>& c = col[tid];
    c.bnorm = o.bnorm;
    c.relres = o.relres;
    c.prev = o.prev;
    c.scale = 0.0;
    c.itol2 = -1.0;
    c.open = o.active && c0 + tid < k;
    c.done = o.done;
    c.status = 0;
    c.iters = c.outer = c.sweep_max = 0;
  }
  __syncthreads();

  T r[RPT][V], x[RPT][V], p[RPT][V], sv[RPT][V];
  for (int outer = 0; outer <= a.max_outer; ++outer) {
    // ---- R = B - A X in FP64 (X of the other blocks through L2)
    T64 rd[RPT][V];
#pragma unroll
    for (int j = 0; j < NV; ++j) v[j] = 0.0;
#pragma unroll
    for (int s = 0; s < RPT; ++s) {
      const int i = s * kSmThreads + tid;
#pragma unroll
      for (int q = 0; q < V; ++q) rd[s][q] = s_zero(T64());
      for (int j = 0; j < len[s]; ++j) {
        const T64 av = a.val64[beg[s] + j];
        const int64_t g = (int64_t)a.indices[beg[s] + j] * k + c0;
#pragma unroll
        for (int q = 0; q < V; ++q)
          if (c0 + q < k) rd[s][q] = s_fma(av, ldcg_t(a.X + g + q), rd[s][q]);
      }
      if (i < rows)
#pragma unroll
        for (int q = 0; q < V; ++q)
          if (c0 + q < k) {
            const double b = a.B[(int64_t)(row0 + i) * k + c0 + q];
            if constexpr (CX) rd[s][q] = make_double2(b - rd[s][q].x, -rd[s][q].y);
            else rd[s][q] = b - rd[s][q];
            v[q] += s_abs2(rd[s][q]);
          }
    }
    if (tid == 0) s_run = 0;
    sm_reduce<NV>(v, red, par, rank, cl);
    if (tid < V) {  // the rules of fin_outer_kernel
      SmCol<T>& c = col[tid];
      c.active = 0;
      c.it_sweep = 0;
      if (c.open) {
        const double s2 = red.tot[tid], rel = sqrt(s2) / c.bnorm;
        c.prev = c.relres;
        c.relres = rel;
        if (!isfinite(rel)) {
          c.open = 0;
          c.done = 3;
        } else if (!(rel > a.tol)) {
          c.open = 0;
          c.done = 1;
        } else if (rel > a.stall * c.prev) {
          c.open = 0;
          c.done = 2;
        } else {
          c.scale = 1.0 / sqrt(s2);
          double it = a.inner_tol;
          if (rel * a.inner_tol < 10.0 * a.tol) it = fmax(fmin(a.inner_tol, 1e-2 * a.tol / rel), a.itol_min);
          c.itol2 = it * it;
        }
      }
      if (c.open && outer < a.max_outer && c.iters < a.itcap) {
        c.active = 1;
        c.status = 0;
        c.outer += 1;
        s_run = 1;
      }
    }
    __syncthreads();
    if (!s_run) break;  // the same in every block of the cluster

    // ---- inner sweep on the scaled residual
#pragma unroll
    for (int s = 0; s < RPT; ++s) {
      const int i = s * kSmThreads + tid;
#pragma unroll
      for (int q = 0; q < V; ++q) {
        const double sc = col[q].active ? col[q].scale : 0.0;
        if constexpr (CX) r[s][q] = T{(float)(rd[s][q].x * sc), (float)(rd[s][q].y * sc)};
        else r[s][q] = (T)(rd[s][q] * sc);
        x[s][q] = p[s][q] = sv[s][q] = s_zero(T());
        if (i < rows) z[i * V + q] = s_mul(dinv[s], r[s][q]);
      }
    }
    for (int it = 0; it <= a.maxiter; ++it) {
      cl_sync();  // z of all blocks is written
      T wv[RPT][V];
#pragma unroll
      for (int j = 0; j < NV; ++j) v[j] = 0.0;
#pragma unroll
      for (int s = 0; s < RPT; ++s) {
        const int i = s * kSmThreads + tid, sl = s * kSmWarps + w;
#pragma unroll
        for (int q = 0; q < V; ++q) wv[s][q] = s_zero(T());
        const int o = s_off[sl], e = s_off[sl + 1];
        if (e <= a.slots) {
          const bool here = e <= a.cap;
          const T* const pv = here ? ev : gv;
          const uint16_t* const pc = here ? ec : gc;
#pragma unroll 5
          for (int j = o + lane; j < e; j += 32) {
            const uint32_t c = pc[j];
            const T av = pv[j];
            alignas(16) T zv[V];
            const uint32_t at = zaddr + (c & ((1u << kSmLocalBits) - 1u)) * (uint32_t)(V * sizeof(T));
            const uint32_t rk = c >> kSmLocalBits;
            if (rk == rank) sm_ld<V * (int)sizeof(T)>(at, zv);
            else cl_ld<V * (int)sizeof(T)>(cl_map(at, rk), zv);
#pragma unroll
            for (int q = 0; q < V; ++q) wv[s][q] = s_fma(av, zv[q], wv[s][q]);
          }
        } else {
          for (int j = 0; j < len[s]; ++j) {
            const int g = a.indices[beg[s] + j], rk = g / nr;
            const T av = a.val[beg[s] + j];
            alignas(16) T zv[V];
            cl_ld<V * (int)sizeof(T)>(cl_map(zaddr + (uint32_t)((g - rk * nr) * V * (int)sizeof(T)), rk), zv);
#pragma unroll
            for (int q = 0; q < V; ++q) wv[s][q] = s_fma(av, zv[q], wv[s][q]);
          }
        }
        if (i < rows) {
#pragma unroll
          for (int q = 0; q < V; ++q) {
            const T zo = s_mul(dinv[s], r[s][q]);
            v[q] += s_abs2(r[s][q]);
            if constexpr (CX) {
              const Acc g = acc_fma(r[s][q], zo, acc_zero<Acc>()), d = acc_fma(wv[s][q], zo, acc_zero<Acc>());
              v[V + q] += g.x;
              v[2 * V + q] += g.y;
              v[3 * V + q] += d.x;
              v[4 * V + q] += d.y;
            } else {
              v[V + q] = acc_fma(r[s][q], zo, v[V + q]);
              v[2 * V + q] = acc_fma(wv[s][q], zo, v[2 * V + q]);
            }
          }
        }
      }
      if (tid == 0) s_any = 0;
      sm_reduce<NV>(v, red, par, rank, cl);
      if (tid < V) {
        SmCol<T>& c = col[tid];
        const double rr = red.tot[tid];
        cdouble g, d;
        if constexpr (CX) {
          g = make_double2(red.tot[V + tid], red.tot[2 * V + tid]);
          d = make_double2(red.tot[3 * V + tid], red.tot[4 * V + tid]);
        } else {
          g = make_double2(red.tot[V + tid], 0.0);
          d = make_double2(red.tot[2 * V + tid], 0.0);
        }
        c.be = c.al = s_zero(T());
        if (c.active) {
          if (it == 0) c.rr0 = rr;
          if (!isfinite(rr) || !finite_c(g)) {
            c.active = 0;
            c.status = 2;
          } else if (rr == 0.0 || (it > 0 && rr <= c.itol2 * c.rr0) || it == a.maxiter || c.iters + it >= a.itcap) {
            c.active = 0;
          } else {
            cdouble be = make_double2(0.0, 0.0), den = d;
            if (it > 0) {
              be = cmul(g, c.igam);
              den = make_double2(d.x, d.y);
              const cdouble t = cmul(cmul(be, c.ialpha), g);  // beta g / alpha_old
              den.x -= t.x;
              den.y -= t.y;
            }
            const cdouble al = cdiv(g, den);
            if (!finite_c(al) || (g.x == 0.0 && g.y == 0.0)) {  // breakdown
              c.active = 0;
              c.status = 2;
            } else {
              c.g = g;
              c.den = den;
              c.be = from_c<T>(be);
              c.al = from_c<T>(al);
              c.it_sweep += 1;
              s_any = 1;
            }
          }
        }
      }
      __syncthreads();
      if (!s_any) break;  // the same in every block of the cluster
      if (tid < V && col[tid].active) {  // for the next iteration, off the path of this one
        SmCol<T>& c = col[tid];
        c.igam = cdiv(make_double2(1.0, 0.0), c.g);
        c.ialpha = cmul(c.den, c.igam);
      }
#pragma unroll
      for (int s = 0; s < RPT; ++s) {
        const int i = s * kSmThreads + tid;
#pragma unroll
        for (int q = 0; q < V; ++q)
          if (col[q].active) {
            const T be = col[q].be, al = col[q].al;
            p[s][q] = s_fma(be, p[s][q], s_mul(dinv[s], r[s][q]));
            sv[s][q] = s_fma(be, sv[s][q], wv[s][q]);
            x[s][q] = s_fma(al, p[s][q], x[s][q]);
            r[s][q] = s_sub(r[s][q], s_mul(al, sv[s][q]));
            if (i < rows) z[i * V + q] = s_mul(dinv[s], r[s][q]);
          }
      }
    }
    if (tid < V) {
      SmCol<T>& c = col[tid];
      c.iters += c.it_sweep;
      c.sweep_max = max(c.sweep_max, c.it_sweep);
    }
    // ---- X += x / scale
#pragma unroll
    for (int s = 0; s < RPT; ++s) {
      const int i = s * kSmThreads + tid;
      if (i < rows)
#pragma unroll
        for (int q = 0; q < V; ++q)
          if (c0 + q < k && col[q].open) {
            const double inv = 1.0 / col[q].scale;
            T64* X = a.X + (int64_t)(row0 + i) * k + c0 + q;
            T64 t = ldcg_t(X);
            if constexpr (CX) {
              t.x += (double)x[s][q].x * inv;
              t.y += (double)x[s][q].y * inv;
            } else {
              t += (double)x[s][q] * inv;
            }
            __stcg(X, t);
          }
    }
    cl_sync();  // X of all blocks before the next residual
  }
  if (rank == 0 && tid < V && c0 + tid < k) {
    const SmCol<T>& c = col[tid];
    SmallOut& o = a.out[c0 + tid];
    o.relres = c.relres;
    o.done = c.done;
    o.status = c.status;
    o.outer = c.outer;
    o.iters = c.iters;
    o.sweep_max = c.sweep_max;
  }
  cl_sync();  // no block leaves while another may still read its shared memory
}

// X[:, c] = 0 for the columns of the mask
template <typename T64>
__global__ void small_reset_kernel(int64_t n, int64_t k, uint64_t lo, uint64_t hi, T64* __restrict__ X) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n * k; i += (int64_t)gridDim.x * blockDim.x) {
    const int c = (int)(i % k);
    if (((c < 64 ? lo >> c : hi >> (c - 64)) & 1) != 0) X[i] = s_zero(T64());
  }
}

// Model time of an iteration in microseconds (fit to the measurements above):
// barriers, reductions and scalars, then a thread's entries, each a gather
// and V products.
template <typename T>
static double small_time(int64_t nnz, int cl, int V, double waves) {
  const double e = (double)nnz / cl / kSmThreads;
  return waves * (3.0 + 0.3 * V + e * (0.03 + (Scalar<T>::is_complex ? 0.08 : 0.055) * V));
}

// The launch of a small solve: cluster size, columns per cluster and rows per
// thread; ok is false when the system does not fit.  The line lies where the
// clusters of one wave hold all columns: more blocks per cluster shorten a
// thread's entries but fewer clusters run at once (33 of 4 blocks, 15 of 8, 7
// of 16 on a B200), more columns per cluster share an entry's read but not
// its products.  Measured at 12,555 x 22 complex: 8 blocks x 2 columns 2.58
// ms, 16 x 2 (two waves) 2.63, 8 x 1 (two waves) 3.13, 16 x 1 3.67; at 11,284
// x 24 real 8 x 2 1.29, 16 x 4 1.39, 16 x 2 1.93, 8 x 1 2.01.  Complex solves
// take at most 2 columns (4 spill: 3.75 ms).
struct SmallPlan {
  bool ok = false;
  int cl = 0, V = 0, rpt = 0, nr = 0, cap = 0, slots = 0;
  size_t smem = 0;
  double us = 0.0;  // model time of an iteration (small_time)
};
constexpr size_t kSmBytes = 227 * 1024 - 12 * 1024;  // dynamic shared memory beside the static arrays

// clusters of size cl that run at once (0: this device cannot hold one)
template <typename T64, typename T, int V, int RPT>
static int small_fit_t(int cl) {
  static std::atomic<int> known[kSmMaxCl + 1];
  int v = known[cl].load(std::memory_order_relaxed);
  if (v) return v - 1;
  auto kern = small_solve_kernel<T64, T, V, RPT>;
  int m = 0;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)cl;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)cl);
  cfg.blockDim = dim3(kSmThreads);
  cfg.dynamicSmemBytes = kSmBytes;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmBytes) != cudaSuccess ||
      cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&m, kern, &cfg) != cudaSuccess) {
    cudaGetLastError();
    m = 0;
  }
  known[cl].store(m + 1, std::memory_order_relaxed);
  return m;
}

template <typename T64, typename T>
static int small_fit(int V, int rpt, int cl) {
  switch (V * 8 + rpt) {
    case 1 * 8 + 1: return small_fit_t<T64, T, 1, 1>(cl);
    case 1 * 8 + 2: return small_fit_t<T64, T, 1, 2>(cl);
    case 1 * 8 + 4: return small_fit_t<T64, T, 1, 4>(cl);
    case 2 * 8 + 1: return small_fit_t<T64, T, 2, 1>(cl);
    case 2 * 8 + 2: return small_fit_t<T64, T, 2, 2>(cl);
    case 2 * 8 + 4: return small_fit_t<T64, T, 2, 4>(cl);
  }
  if constexpr (!Scalar<T>::is_complex) {
    if (V * 8 + rpt == 4 * 8 + 1) return small_fit_t<T64, T, 4, 1>(cl);
    if (V * 8 + rpt == 4 * 8 + 2) return small_fit_t<T64, T, 4, 2>(cl);
  }
  return 0;
}

constexpr int64_t kSmMaxRows = 16 * 2048;
// entry slots of a rank: slices padded to their longest row take about a tenth
// more than nnz / cl entries on a mesh
static int64_t small_slots(int64_t nnz, int cl) { return (nnz * 6 / 5 / cl + 2048) / 32 * 32; }
static int64_t small_soff(int cl, int rpt) { return (int64_t)cl * (kSmWarps * rpt + 1); }
// bytes of the sliced matrix for any plan
template <typename T>
static size_t small_bytes(int64_t n, int64_t nnz) {
  if (n > kSmMaxRows) return 0;
  return (size_t)(small_slots(nnz, 1) + 2048 * kSmMaxCl) * (sizeof(T) + 2) + small_soff(kSmMaxCl, 4) * 4 + 1024;
}

template <typename T64, typename T>
static SmallPlan small_plan(int64_t n, int64_t nnz, int64_t k) {
  SmallPlan p;
  if (n < 1 || n > kSmMaxRows || nnz >= (int64_t(1) << 30)) return p;
  double best = 0.0;
  for (int cl : {4, 8, 16}) {
    const int nr = (int)ceil_div(n, cl);
    if (nr > 2048) continue;
    const int rpt = nr <= kSmThreads ? 1 : nr <= 2 * kSmThreads ? 2 : 4;
    const int64_t slots = small_slots(nnz, cl);
    for (int V : {1, 2, 4}) {
      if (V * rpt > 8 || (Scalar<T>::is_complex && V > 2)) continue;
      const size_t zb = ((size_t)nr * V * sizeof(T) + 15) / 16 * 16;
      if (zb > kSmBytes) continue;
      const int cap = (int)std::min<int64_t>(slots, (int64_t)((kSmBytes - zb) / (sizeof(T) + 2)) / 32 * 32);
      const int fit = small_fit<T64, T>(V, rpt, cl);
      if (fit < 1) continue;
      const double waves = (double)ceil_div(ceil_div(k, V), fit);
      const double t = small_time<T>(nnz, cl, V, waves);
      if (!p.ok || t < best) {
        best = t;
        p.ok = true;
        p.us = t;
        p.cl = cl;
        p.V = V;
        p.rpt = rpt;
        p.nr = nr;
        p.cap = cap;
        p.slots = (int)slots;
        p.smem = zb + (size_t)cap * (sizeof(T) + 2);
      }
    }
  }
  return p;
}

// Whether a solve goes faster in one launch than by the separate kernels.
// Their iteration takes about 28 us of launches and read-backs and, streaming
// all columns in one wave, a time per row and column (half of it the product's:
// per entry); the one launch's waves grow with the columns.  Fit on boxes of
// 1,210 to 32,736 nodes x 1 to 128 columns; the separate kernels stop at their
// next host check (15% more iterations) and the model above is a third low for
// complex columns, four rows a thread.  Separate kernels / one launch, ms: real 9,261
// x 128 7.5 / 5.3, 16,900 x 64 7.4 / 6.0, x 96 8.0 / 8.4, x 128 8.4 / 11.8, 24,273 x
// 64 8.1 / 6.8, x 96 9.4 / 9.6, 32,736 x 48 8.8 / 7.5, x 64 9.3 / 9.1, x 128 11.8 /
// 18.3; complex 9,261 x 96 8.1 / 7.2, x 128 8.9 / 8.8, 16,900 x 48 8.5 / 8.4, x 64
// 9.3 / 10.4, x 128 12.0 / 20.5, 24,273 x 32 8.8 / 7.4, x 48 9.6 / 10.0, 32,736 x 32
// 9.5 / 9.2, x 48 11.6 / 12.4, x 128 20.5 / 30.5.
template <typename T>
static bool small_wins(const SmallPlan& p, int64_t n, int64_t nnz, int64_t k) {
  constexpr bool CX = Scalar<T>::is_complex;
  const double work = 0.5 * (double)(n + nnz / 14.4) * (double)k;  // (14.4 entries per row of those boxes)
  const double sep = CX ? 29.8 + 0.03 * k + 16.7e-6 * work : 28.4 + 0.05 * k + 6.3e-6 * work;
  return p.ok && (CX ? 1.3 : 1.0) * p.us < 1.15 * sep;
}

template <typename T64, typename T, int V, int RPT>
static int small_launch_t(const SmallArgs<T64, T>& a, const SmallPlan& p, cudaStream_t st) {
  auto kern = small_solve_kernel<T64, T, V, RPT>;
  // the bound is the same for every plan: it belongs to the function, not to
  // the launch, and another thread's smaller plan must not lower it in between
  RB_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmBytes));
  RB_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(ceil_div(a.k, V) * p.cl));
  cfg.blockDim = dim3(kSmThreads);
  cfg.dynamicSmemBytes = p.smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)p.cl;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  small_slice_kernel<T><<<p.cl, kSmThreads, 0, st>>>(a.n, p.nr, p.rpt, p.slots, a.indptr, a.indices, a.val,
                                                     const_cast<int32_t*>(a.soff), const_cast<T*>(a.sval),
                                                     const_cast<uint16_t*>(a.scol));
  RB_LAUNCH_CHECK();
  RB_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, a));
  return RB_OK;
}

template <typename T64, typename T>
static int small_launch(const SmallArgs<T64, T>& a, const SmallPlan& p, cudaStream_t st) {
  switch (p.V * 8 + p.rpt) {
    case 1 * 8 + 1: return small_launch_t<T64, T, 1, 1>(a, p, st);
    case 1 * 8 + 2: return small_launch_t<T64, T, 1, 2>(a, p, st);
    case 1 * 8 + 4: return small_launch_t<T64, T, 1, 4>(a, p, st);
    case 2 * 8 + 1: return small_launch_t<T64, T, 2, 1>(a, p, st);
    case 2 * 8 + 2: return small_launch_t<T64, T, 2, 2>(a, p, st);
    case 2 * 8 + 4: return small_launch_t<T64, T, 2, 4>(a, p, st);
  }
  if constexpr (!Scalar<T>::is_complex) {
    if (p.V * 8 + p.rpt == 4 * 8 + 1) return small_launch_t<T64, T, 4, 1>(a, p, st);
    if (p.V * 8 + p.rpt == 4 * 8 + 2) return small_launch_t<T64, T, 4, 2>(a, p, st);
  }
  return fail(RB_EARG, "small solve: bad plan");
}

}  // namespace rb
