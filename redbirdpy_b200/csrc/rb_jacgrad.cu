// Adjoint gradient of the node-based model in one pass over the tets:
//   gm[n] = Re sum_s phi_s^T (-dA/dmua_n) lam_s   (mua at fixed D),
//   gd[n] = Re sum_s phi_s^T (-dA/dD_n) lam_s,
// the column sums of rb_jac's 'mua_nodal' and 'D' rows for the pairs
// (s, lam_s) without forming a row (dA/dp as femlhs's node-based weights,
// redbirdpy/forward.py:177-228).  Per tet, with G_ij = sum_s phi_i[s] lam_j[s]
// over its four nodes, U_n = sum_j (G_nj + G_jn), V_n = G_nn:
//   to gm[n]: -V_e/120 (1/2 sum U + sum V + U_n + 2 V_n),
//   to gd[n]: -1/4 sum_ij ddd_ij G_ij   (the same for the four nodes).
// What bounds it: the reads of phi and lam (8 rows of ns values per tet; a
// node's rows are shared by its ~24 tets, which are close in tet order, so
// most of them hit L1/L2).  L lanes own a tet and stride over the columns, so
// a row is read in whole sectors and nine partial sums are reduced over L
// lanes only; 32 / L tets per warp keep 8 x 32 independent loads in flight.
// A second kernel adds each node's tet terms in ascending tet order: no
// atomics, the same bits on every run.  The row kernel it replaces on this
// path staged every node's neighbourhood in shared memory to write ns x nn
// rows that were then summed.  Measured, both parameters (rows and their sum
// before, this after): 67,626 nodes / 375,000 tets, 32 real columns: 1.75 ->
// 0.16 ms; 64 instances of 3.6M tets in all, 16 columns: 18.7 -> 1.2 ms.
#include <algorithm>

#include "rb_common.cuh"

namespace rb {

constexpr int kGradThreads = 256;

__device__ __forceinline__ double re_mul(double a, double b) { return a * b; }
__device__ __forceinline__ double re_mul(cdouble a, cdouble b) { return a.x * b.x - a.y * b.y; }
__device__ __forceinline__ double re_fma(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ double re_fma(cdouble a, cdouble b, double c) { return fma(a.x, b.x, fma(-a.y, b.y, c)); }
__device__ __forceinline__ double r_scale(double r, double v) { return r * v; }
__device__ __forceinline__ cdouble r_scale(double r, cdouble v) { return make_double2(r * v.x, r * v.y); }

template <typename T, int L>
__global__ void __launch_bounds__(kGradThreads)
tet_grad_kernel(int64_t ne, const int4* __restrict__ elem, const double* __restrict__ evol,
                const double* __restrict__ ddd, const T* __restrict__ phi, int64_t ldp, const T* __restrict__ lam,
                int64_t ldl, int ns, double* __restrict__ tm, double* __restrict__ td) {
  const int lane = threadIdx.x % L;
  const int64_t groups = (int64_t)gridDim.x * (kGradThreads / L);
  // every lane group of a warp makes the same number of rounds (full-warp shuffles)
  const int64_t rounds = (ne + groups - 1) / groups;
  for (int64_t it = 0; it < rounds; ++it) {
    const int64_t e = it * groups + blockIdx.x * (int64_t)(kGradThreads / L) + threadIdx.x / L;
    const bool on = e < ne;
    double u[4] = {0, 0, 0, 0}, v[4] = {0, 0, 0, 0}, g = 0.0;
    if (on) {
      const int4 en = elem[e];
      const int32_t nd[4] = {en.x, en.y, en.z, en.w};
      double k[10];
      if (td) {
#pragma unroll
        for (int j = 0; j < 10; ++j) k[j] = ddd[10 * e + j];
      }
      for (int c = lane; c < ns; c += L) {
        T p[4], q[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          p[i] = phi[(int64_t)nd[i] * ldp + c];
          q[i] = lam[(int64_t)nd[i] * ldl + c];
        }
        if (tm) {
          const T sp = s_add(s_add(p[0], p[1]), s_add(p[2], p[3]));
          const T sq = s_add(s_add(q[0], q[1]), s_add(q[2], q[3]));
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            u[i] = re_fma(p[i], sq, re_fma(q[i], sp, u[i]));
            v[i] = re_fma(p[i], q[i], v[i]);
          }
        }
        if (td) {
          // row i of the symmetric ddd against q: columns of (0..3, 4..6, 7..8, 9)
          const T r0 = s_add(s_add(r_scale(k[0], q[0]), r_scale(k[1], q[1])), s_add(r_scale(k[2], q[2]), r_scale(k[3], q[3])));
          const T r1 = s_add(s_add(r_scale(k[1], q[0]), r_scale(k[4], q[1])), s_add(r_scale(k[5], q[2]), r_scale(k[6], q[3])));
          const T r2 = s_add(s_add(r_scale(k[2], q[0]), r_scale(k[5], q[1])), s_add(r_scale(k[7], q[2]), r_scale(k[8], q[3])));
          const T r3 = s_add(s_add(r_scale(k[3], q[0]), r_scale(k[6], q[1])), s_add(r_scale(k[8], q[2]), r_scale(k[9], q[3])));
          g = re_fma(p[0], r0, re_fma(p[1], r1, re_fma(p[2], r2, re_fma(p[3], r3, g))));
        }
      }
    }
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        u[i] += __shfl_xor_sync(0xffffffffu, u[i], o);
        v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
      }
      g += __shfl_xor_sync(0xffffffffu, g, o);
    }
    if (on && lane == 0) {
      if (tm) {
        const double w = -evol[e] / 120.0;
        const double t = 0.5 * ((u[0] + u[1]) + (u[2] + u[3])) + ((v[0] + v[1]) + (v[2] + v[3]));
        double2* o = reinterpret_cast<double2*>(tm + 4 * e);
        o[0] = make_double2(w * (t + u[0] + 2.0 * v[0]), w * (t + u[1] + 2.0 * v[1]));
        o[1] = make_double2(w * (t + u[2] + 2.0 * v[2]), w * (t + u[3] + 2.0 * v[3]));
      }
      if (td) td[e] = -0.25 * g;
    }
  }
}

// a node's tet terms in ascending tet order
__global__ void node_grad_kernel(int64_t nn, const int32_t* __restrict__ eptr, const int32_t* __restrict__ elist,
                                 const int4* __restrict__ elem, const double* __restrict__ tm,
                                 const double* __restrict__ td, double* __restrict__ gm, double* __restrict__ gd) {
  for (int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; n < nn; n += (int64_t)gridDim.x * blockDim.x) {
    double a = 0.0, d = 0.0;
    const int32_t q1 = eptr[n + 1];
#pragma unroll 4
    for (int32_t q = eptr[n]; q < q1; ++q) {
      const int32_t e = elist[q];
      if (gm) {
        const int4 en = elem[e];
        const int i = en.y == n ? 1 : en.z == n ? 2 : en.w == n ? 3 : 0;
        a += tm[4 * (int64_t)e + i];
      }
      if (gd) d += td[e];
    }
    if (gm) gm[n] = a;
    if (gd) gd[n] = d;
  }
}

template <typename T>
static int grad_run(const rb_mesh& m, const T* phi, int64_t ldp, const T* lam, int64_t ldl, int64_t ns,
                    const double* evol, const double* ddd, double* gm, double* gd, double* work, cudaStream_t st) {
  double* tm = gm ? work : nullptr;
  double* td = gd ? work + 4 * m.ne : nullptr;
  const int4* elem = reinterpret_cast<const int4*>(m.elem);
  // lanes per tet: enough for the columns, at most 8 (a lane then takes
  // several columns: fewer shuffles per product and more tets per warp)
  const int L = ns <= 2 ? 2 : ns <= 4 ? 4 : 8;
  const unsigned g = (unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(m.ne * L, kGradThreads), 148 * 32));
  if (m.ne > 0) {
    switch (L) {
      case 2: tet_grad_kernel<T, 2><<<g, kGradThreads, 0, st>>>(m.ne, elem, evol, ddd, phi, ldp, lam, ldl, (int)ns, tm, td); break;
      case 4: tet_grad_kernel<T, 4><<<g, kGradThreads, 0, st>>>(m.ne, elem, evol, ddd, phi, ldp, lam, ldl, (int)ns, tm, td); break;
      default: tet_grad_kernel<T, 8><<<g, kGradThreads, 0, st>>>(m.ne, elem, evol, ddd, phi, ldp, lam, ldl, (int)ns, tm, td); break;
    }
    RB_LAUNCH_CHECK();
  }
  const unsigned gn = (unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(m.nn, 128), 148 * 16));
  node_grad_kernel<<<gn, 128, 0, st>>>(m.nn, m.node_eptr, m.node_elist, elem, tm, td, gm, gd);
  RB_LAUNCH_CHECK();
  return RB_OK;
}

}  // namespace rb

using namespace rb;

extern "C" {

size_t rb_jac_grad_work_bytes(int64_t ne) { return (size_t)std::max<int64_t>(ne, 1) * 5 * sizeof(double) + 16; }

int rb_jac_grad(const rb_mesh* mesh, const void* phi, int64_t ldp, const void* lam, int64_t ldl, int64_t ns,
                int32_t kind, const double* evol, const double* ddd, double* gm, double* gd, void* work,
                size_t work_bytes, void* stream) {
  if (!mesh || !phi || !lam || !evol || !work || ns < 1 || ldp < ns || ldl < ns)
    return fail(RB_EARG, "rb_jac_grad: bad arguments");
  if (gd && !ddd) return fail(RB_EARG, "rb_jac_grad: the D gradient needs deldotdel");
  if (kind != RB_F64 && kind != RB_C128) return fail(RB_EARG, "rb_jac_grad: kind must be RB_F64 or RB_C128");
  if (work_bytes < rb_jac_grad_work_bytes(mesh->ne) || (reinterpret_cast<uintptr_t>(work) & 15))
    return fail(RB_EARG, "rb_jac_grad: workspace too small or unaligned");
  if ((!gm && !gd) || mesh->nn == 0) return RB_OK;
  cudaStream_t st = as_stream(stream);
  if (kind == RB_F64)
    return grad_run<double>(*mesh, (const double*)phi, ldp, (const double*)lam, ldl, ns, evol, ddd, gm, gd,
                            (double*)work, st);
  return grad_run<cdouble>(*mesh, (const cdouble*)phi, ldp, (const cdouble*)lam, ldl, ns, evol, ddd, gm, gd,
                           (double*)work, st);
}

}  // extern "C"
