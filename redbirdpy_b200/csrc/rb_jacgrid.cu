// Jacobian rows of the full (source x detector) grid, products formed in FP64
// and stored as FP32 rows (the Gauss-Newton step's J).
//
//   J_p[k = (d, s)][n] = sum_a phi_s[a] C_p,n[a][d],
//   C_p,n[a][d] = sum_b B_p,n[a][b] phi_d[b],
// a, b over the CSR row of node n and B_p,n the small matrix that rb_jac.cu's
// jac_stage builds (same coefficients, same order of every sum: the rows equal
// jac_kernel's bit for bit).
//
// What bounded jac_kernel: its staging and its stores.  A block of two nodes
// went through six barrier-separated steps of dependent loads (row -> tets ->
// nodes -> search) with two blocks per SM, 42 us per two nodes against 4 us of
// FP64 products; and a J row got 8 bytes at a time.  A store's cost on this
// chip is its segment, and more so where it covers part of a 32-byte sector:
// 2.2 GB of 8192 rows took 6.1 ms in 8-byte segments, 4.5 in 16-byte, 1.4 in
// aligned 32-byte ones, 3.2 in 32-byte ones off the sector grid.  Here
//  - jac_b_kernel builds the B matrices of a chunk of nodes, a warp per node,
//    into a workspace that stays in L2;
//  - jac_grid_kernel is persistent: 4 warps bring the next item's fields and B
//    into the other half of the shared memory while 8 warps form the products:
//    by bulk copies of a row's column range where sources and detectors are two
//    ranges on 16 bytes (5.6 ms at the size below), else by cp.async (6.1; with
//    the computing warps fetching as well the two did not overlap: 6.9; with 2
//    fetching warps 8.9); the neighbour lists that this needs are loaded two
//    items ahead;
//  - a thread takes 4 sources x 4 detectors of one node; 8 neighbouring lanes
//    take 8 neighbouring nodes whose J columns are one aligned sector (blocks
//    of nodes start where the quantity's J column is a multiple of 8), and a
//    thread's sources lie NSB apart, so that its reads of phi are free of bank
//    conflicts;
//  - C replaces phi_d in place (a thread owns half of a column, the lane next
//    to it the other half), which is what lets two buffers of 8 nodes fit.
// Measured at 67,626 nodes, 64 x 64 complex pairs, two quantities (4.4 GB of
// rows): 9.9 ms before, 6.2 now, of which 0.6 the B matrices.  Shared memory
// bounds it now: the products' reads take about as long as their FP64 work (2.1
// ms at the full rate), the C matrices' two thirds of that again, with two warps
// per scheduler to overlap them.  (The fetching warps forming C as well: 5.61
// ms against 5.56.)
#include <algorithm>

#include "rb_common.cuh"
#include "rb_tc.cuh"

namespace rb {

int* jac_err_word();  // rb_jac.cu: what rb_jac_status reads
int jac_resident(bool cx, bool grid, int rmax, int nc, int ndet, int emax);  // rb_jac.cu

enum { JG_MUA_REF = 0, JG_MUA_NODAL = 1, JG_D = 2 };
constexpr int kJgThreads = 256;    // threads that compute
constexpr int kJgProducers = 128;  // threads that fetch
constexpr int kJgMaxE = 64;   // incident tets of a node at most
constexpr size_t kJgSmem = 226 * 1024;

struct JgArgs {
  const int32_t *indptr, *indices, *eptr, *elist;
  const int4* elem;
  const double *evol, *ddd;
  const int32_t* cols;  // phi columns: sources (0 .. nsu - 1) and detectors (det0 ..)
  int32_t nsu, det0, nd, rmax, what;
  int64_t ld, ldj, nsd, col0;           // col0: J column of the range's first node
  int64_t node0, chunk0, chunk1, blk0;  // range start, nodes of this launch, first node block's start (<= chunk0)
};

// B of the nodes chunk0 .. chunk1 - 1: out[(n - chunk0) rmax RM + a RM + b]
template <int RM> constexpr int jg_bwarps() { return RM == 16 ? 4 : 2; }  // static shared memory
template <int RM>
__global__ void __launch_bounds__(jg_bwarps<RM>() * 32) jac_b_kernel(JgArgs a, double* __restrict__ out) {
  constexpr int kJgBWarps = jg_bwarps<RM>();
  __shared__ int32_t s_nb[kJgBWarps][RM];
  __shared__ double s_vol[kJgBWarps][kJgMaxE], s_dd[kJgBWarps][kJgMaxE][10];
  __shared__ int8_t s_lp[kJgBWarps][kJgMaxE][4];
  __shared__ int8_t s_li[kJgBWarps][kJgMaxE];
  __shared__ double s_B[kJgBWarps][RM * (RM + 1)];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int rmax = a.rmax;
  for (int64_t n = a.chunk0 + blockIdx.x * (int64_t)kJgBWarps + w; n < a.chunk1; n += (int64_t)gridDim.x * kJgBWarps) {
    const int32_t rb = a.indptr[n], rn = a.indptr[n + 1] - rb;
    const int32_t eb = a.eptr[n], ek = a.eptr[n + 1] - eb;
    if (lane < RM) s_nb[w][lane] = lane < rn ? a.indices[rb + lane] : -1;
    __syncwarp();
    for (int q = lane; q < ek; q += 32) {
      const int32_t e = a.elist[eb + q];
      const int4 en = a.elem[e];
      const int32_t nd4[4] = {en.x, en.y, en.z, en.w};
      s_vol[w][q] = a.evol[e];
      if (a.ddd)
        for (int j = 0; j < 10; ++j) s_dd[w][q][j] = a.ddd[10 * (int64_t)e + j];
      int li = 0;
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        int pos = -1;
        for (int b = 0; b < rn; ++b)
          if (s_nb[w][b] == nd4[m]) pos = b;
        s_lp[w][q][m] = (int8_t)pos;
        if (nd4[m] == n) li |= 1 << m;
      }
      s_li[w][q] = (int8_t)li;
    }
    __syncwarp();
    double* const B = s_B[w];
    const int what = a.what;
    if (lane < RM) {  // lane = row: its tets in ascending order
      double* const Brow = B + lane * (RM + 1);
      for (int b = 0; b < RM; ++b) Brow[b] = 0.0;
      if (lane < rn)
        for (int q = 0; q < ek; ++q) {
          const int8_t* lp = s_lp[w][q];
          int pa = -1;
#pragma unroll
          for (int m = 0; m < 4; ++m)
            if (lp[m] == lane) pa = m;
          if (pa < 0) continue;
          const double vol = s_vol[w][q];
          const int li = s_li[w][q];
#pragma unroll
          for (int m = 0; m < 4; ++m) {
            double wv;
            if (what == JG_MUA_REF) {
              wv = -0.0125 * vol * (m == pa ? 2.0 : 1.0);
            } else if (what == JG_MUA_NODAL) {
              const double f = 1.0 + ((li >> pa) & 1) + ((li >> m) & 1);
              wv = -vol / 120.0 * f * (m == pa ? 2.0 : 1.0);
            } else {
              const int lo = min(pa, m), hi = max(pa, m);
              wv = -0.25 * s_dd[w][q][lo * 4 - lo * (lo - 1) / 2 + (hi - lo)];
            }
            if (lp[m] >= 0) Brow[lp[m]] += wv;
          }
        }
    }
    __syncwarp();
    double* o = out + (n - a.chunk0) * (int64_t)(rmax * RM);
    for (int i = lane; i < rmax * RM; i += 32) o[i] = B[i / RM * (RM + 1) + i % RM];
    __syncwarp();
  }
}

__device__ __forceinline__ uint32_t jg_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
template <int NB>
__device__ __forceinline__ void jg_cp(void* dst, const void* src) {
  if constexpr (NB == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(jg_u32(dst)), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(jg_u32(dst)), "l"(src) : "memory");
}

__device__ __forceinline__ void b_fma(double& acc, double b, double v) { acc = fma(b, v, acc); }
__device__ __forceinline__ void b_fma(cdouble& acc, double b, cdouble v) {
  acc.x = fma(b, v.x, acc.x);
  acc.y = fma(b, v.y, acc.y);
}

// a copy of the asynchronous engine, completed on a barrier (16-byte aligned, whole 16 bytes)
__device__ __forceinline__ void jg_bulk(void* dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(jg_u32(dst)),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

// shared memory, per buffer: phi_s [TN][SP], phi_d (then C) [TN][SD], B
// [TN][rmax RM]; then the neighbour lists of three items and the column map
struct JgLayout {
  int SP, SD, DT, ST, NSB, NDB, nst, ndt;  // strides (elements), tile sizes, 4-wide groups of a tile, tiles
  size_t phis, phid, b, buf, nb, total;
};
template <typename C, int TN, int RM>
__host__ __device__ inline JgLayout jg_layout(int rmax, int nsu, int nd, int nbuf) {
  JgLayout L;
  constexpr int E = 128 / (int)sizeof(C);  // elements per bank row
  L.nst = (nsu + 31) / 32;
  L.NSB = (nsu + 4 * L.nst - 1) / (4 * L.nst);
  L.ST = 4 * L.NSB;
  L.NDB = kJgThreads / (TN * L.NSB);
  if (L.NDB > 8) L.NDB = 8;  // (phi_d: at most 32 columns)
  if (TN * L.NSB * L.NDB > 128 && TN < 8) L.NDB = 128 / (TN * L.NSB);
  if (L.NDB > 4 && L.NSB > 4) L.NDB = 4;
  if (L.NDB > (nd + 3) / 4) L.NDB = (nd + 3) / 4;
  L.DT = 4 * L.NDB;
  L.ndt = (nd + L.DT - 1) / L.DT;
  // the TN lanes of a group lie E / TN elements apart in the banks
  L.SP = (rmax * L.ST + E - 1) / E * E + (E >= TN ? E / TN : 1);
  L.SD = (rmax * L.DT + E - 1) / E * E + (E >= TN ? E / TN : 1);
  L.phis = 0;
  L.phid = ((size_t)TN * L.SP * sizeof(C) + 15) / 16 * 16;
  L.b = L.phid + ((size_t)TN * L.SD * sizeof(C) + 15) / 16 * 16;
  L.buf = L.b + (size_t)TN * rmax * RM * sizeof(double);
  L.nb = L.buf * nbuf;
  L.total = L.nb + (size_t)3 * TN * (RM + 1) * sizeof(int32_t) + 128 * sizeof(int32_t);
  return L;
}

// TN = 8 nodes per item and rows of at most 16 neighbours (a Kuhn box has 15),
// or TN = 4 and at most 32
template <typename C, bool SPLIT, int RM, int TN, int NBUF>
__global__ void __launch_bounds__(kJgThreads + kJgProducers, 1)
jac_grid_kernel(JgArgs a, const C* __restrict__ phi, const double* __restrict__ Bg, float* __restrict__ J,
                int32_t items, int* __restrict__ err) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ __align__(8) uint64_t full[2];
  __shared__ int s_bad;
  constexpr int NT = kJgThreads;
  static_assert(TN * RM <= NT, "a thread loads one neighbour at most");
  const int rmax = a.rmax, nsu = a.nsu, nd = a.nd;
  const JgLayout L = jg_layout<C, TN, RM>(rmax, nsu, nd, NBUF);
  int32_t* const snb = reinterpret_cast<int32_t*>(smem + L.nb);  // [3][TN][RM + 1]: row length, neighbours
  int32_t* const scol = snb + 3 * TN * (RM + 1);
  const int tid = threadIdx.x, lane = tid & 31;
  const int NSB = L.NSB, DT = L.DT, ST = L.ST, ntile = L.nst * L.ndt;
  for (int c = tid; c < nsu + nd && c < 128; c += NT + kJgProducers) scol[c] = a.cols[c < nsu ? c : a.det0 + c - nsu];

  // Neighbour lists: thread i < TN RM holds neighbour q = i % RM of node i / RM.
  // Its loads are spread over the items (row bounds, then the neighbour, then
  // the store into shared memory), so that none is waited for.
  const int lt = tid / RM, lq = tid % RM;
  const bool lon = tid < TN * RM;
  auto bounds = [&](int32_t item, int32_t& b, int32_t& e) {
    b = e = 0;
    const int64_t n = a.blk0 + (int64_t)(item / ntile) * TN + lt;
    if (lon && item < items && n >= a.chunk0 && n < a.chunk1) {
      b = a.indptr[n];
      e = a.indptr[n + 1];
    }
  };
  auto neighbour = [&](int32_t b, int32_t e) { return lon && b + lq < e ? a.indices[b + lq] : -1; };
  auto keep = [&](int slot, int32_t rn, int32_t m) {
    if (!lon) return;
    int32_t* o = snb + (slot * TN + lt) * (RM + 1);
    if (lq == 0) o[0] = rn;
    o[1 + lq] = m;
  };
  // the item's fields and B on their way into buffer buf: a warp per (node,
  // neighbour), lanes over columns (at most 32 of each)
  auto fetch = [&](int32_t item, int slot, int buf) {
    const int32_t nb = item / ntile, tile = item - nb * ntile;
    const int s0 = tile / L.ndt * ST, d0 = tile % L.ndt * DT;
    const int64_t n0 = a.blk0 + (int64_t)nb * TN;
    unsigned char* const base = smem + (size_t)buf * L.buf;
    C* const ps = reinterpret_cast<C*>(base + L.phis) + lane;
    C* const pd = reinterpret_cast<C*>(base + L.phid) + lane;
    double* const pb = reinterpret_cast<double*>(base + L.b);
    const int cs = lane < ST && s0 + lane < nsu ? scol[s0 + lane] : -1;
    const int cd = lane < DT && d0 + lane < nd ? scol[nsu + d0 + lane] : -1;
#pragma unroll 5
    for (int r = (tid - NT) >> 5; r < TN * rmax; r += kJgProducers / 32) {
      const int t = r / rmax, q = r - t * rmax;
      const int32_t m = snb[(slot * TN + t) * (RM + 1) + 1 + q];
      if (m < 0) continue;
      const C* src = phi + (int64_t)m * a.ld;
      if (cs >= 0) jg_cp<sizeof(C)>(ps + t * L.SP + q * ST, src + cs);
      if (cd >= 0) jg_cp<sizeof(C)>(pd + t * L.SD + q * DT, src + cd);
    }
    // B of the block's nodes within the launch's range
    const int t0 = (int)max((int64_t)0, a.chunk0 - n0), t1 = (int)min((int64_t)TN, a.chunk1 - n0);
    const int per = rmax * (RM / 2);  // 16-byte pieces of a node
    const double* bs = Bg + (n0 - a.chunk0) * (int64_t)(rmax * RM);
    for (int i = t0 * per + tid - NT; i < t1 * per; i += kJgProducers) jg_cp<16>(pb + 2 * i, bs + 2 * i);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  // the same by bulk copies, a row and column range each: where the sources'
  // and the detectors' columns are two ranges that start on 16 bytes
  auto fetch_bulk = [&](int32_t item, int slot, int buf) {
    const int32_t nb = item / ntile, tile = item - nb * ntile;
    const int s0 = tile / L.ndt * ST, d0 = tile % L.ndt * DT;
    const int64_t n0 = a.blk0 + (int64_t)nb * TN;
    unsigned char* const base = smem + (size_t)buf * L.buf;
    const uint32_t bar = smem_u32(&full[buf]);
    const int r = tid - NT, t = r / rmax, q = r - t * rmax;
    const int32_t m = r < TN * rmax ? snb[(slot * TN + t) * (RM + 1) + 1 + q] : -1;
    const uint32_t sbytes = (uint32_t)(min(ST, nsu - s0) * (int)sizeof(C));
    const uint32_t dbytes = (uint32_t)(min(DT, nd - d0) * (int)sizeof(C));
    uint32_t bytes = m >= 0 ? sbytes + dbytes : 0u, bbytes = 0u;
    const int t0 = (int)max((int64_t)0, a.chunk0 - n0), t1 = (int)min((int64_t)TN, a.chunk1 - n0);
    if (r == 0 && t1 > t0) bbytes = (uint32_t)((t1 - t0) * rmax * RM * (int)sizeof(double));
    mbar_expect_tx(bar, bytes + bbytes);  // (arrives for this thread)
    if (m >= 0) {
      const C* src = phi + (int64_t)m * a.ld;
      jg_bulk(reinterpret_cast<C*>(base + L.phis) + t * L.SP + q * ST, src + scol[s0], sbytes, bar);
      jg_bulk(reinterpret_cast<C*>(base + L.phid) + t * L.SD + q * DT, src + scol[nsu + d0], dbytes, bar);
    }
    if (bbytes)
      jg_bulk(reinterpret_cast<double*>(base + L.b) + (size_t)t0 * rmax * RM,
              Bg + (n0 + t0 - a.chunk0) * (int64_t)(rmax * RM), bbytes, bar);
  };

  const int32_t step = gridDim.x;
  int32_t item = blockIdx.x;
  if (item >= items) return;
  if (tid == 0) {
    s_bad = 0;
    mbar_init(smem_u32(&full[0]), kJgProducers);
    mbar_init(smem_u32(&full[1]), kJgProducers);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  int32_t lb, le, mb, me, mm;  // row bounds of the item three ahead; bounds and neighbour of the one two ahead
  bounds(item, lb, le);
  keep(0, le - lb, neighbour(lb, le));
  bounds(item + step, lb, le);
  keep(1, le - lb, neighbour(lb, le));
  bounds(item + 2 * step, lb, le);
  __syncthreads();
  bool range = ((reinterpret_cast<uintptr_t>(phi + scol[0]) | reinterpret_cast<uintptr_t>(phi + scol[nsu])) & 15) == 0 &&
               (a.ld * (int64_t)sizeof(C)) % 16 == 0 && (nsu * sizeof(C)) % 16 == 0 && (nd * sizeof(C)) % 16 == 0;
  if (tid < nsu) range = range && scol[tid] == scol[0] + tid;
  if (tid < nd) range = range && scol[nsu + tid] == scol[nsu] + tid;
  const bool bulk = __syncthreads_and(range);
  const bool producer = tid >= NT;
  if (producer) {
    if (bulk) fetch_bulk(item, 0, 0);
    else fetch(item, 0, 0);
  }
  const int t = tid % TN, g = tid / TN, sb = g % NSB, db = g / NSB;
  int slot = 0;
  for (int it = 0; item < items; item += step, ++it) {
    const int buf = NBUF == 2 ? it & 1 : 0;
    const int next = slot == 2 ? 0 : slot + 1, after = next == 2 ? 0 : next + 1;
    if (bulk) {
      if (!producer && !mbar_wait(smem_u32(&full[buf]), (NBUF == 2 ? it >> 1 : it) & 1, err, 64)) s_bad = 1;
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    if (bulk && *reinterpret_cast<volatile int*>(&s_bad)) {  // (reported by rb_jac_status)
      mbar_wait(smem_u32(&full[buf]), (NBUF == 2 ? it >> 1 : it) & 1, err, 64);  // its own copies, again with a limit
      return;
    }
    mb = lb;
    me = le;
    mm = neighbour(mb, me);
    bounds(item + 3 * step, lb, le);
    if (NBUF == 2 && producer && item + step < items) {
      if (bulk) fetch_bulk(item + step, next, buf ^ 1);
      else fetch(item + step, next, buf ^ 1);
    }
    unsigned char* const base = smem + (size_t)buf * L.buf;
    const C* const ps = reinterpret_cast<const C*>(base + L.phis);
    C* const pd = reinterpret_cast<C*>(base + L.phid);
    const double* const pb = reinterpret_cast<const double*>(base + L.b);
    const int32_t nbk = item / ntile, tile = item - nbk * ntile;
    const int s0 = tile / L.ndt * ST, d0 = tile % L.ndt * DT;
    const int32_t* const rn_ = snb + slot * TN * (RM + 1);
    // C over phi_d: a thread takes two detectors of a node and half of the
    // rows (adjacent lanes the two halves, so that both have read the columns
    // before either writes); B is symmetric: its row b holds the coefficients
    // of phi_d[b] in every C[a]
    constexpr int RH = RM / 2;
    const int nci = (2 * TN * DT + 31) / 32 * 32;
    for (int i = tid; i < nci && !producer; i += NT) {
      const int h = i & 1, j = i >> 1, d = j % DT, tt = j / DT;
      const bool con = tt < TN;
      const int rn = con ? rn_[tt * (RM + 1)] : 0;
      C* const col = pd + (con ? tt : 0) * L.SD + d;
      const double2* B2 = reinterpret_cast<const double2*>(pb + (size_t)(con ? tt : 0) * rmax * RM + h * RH);
      C c0[RH];
#pragma unroll
      for (int q = 0; q < RH; ++q) c0[q] = s_zero(C());
#pragma unroll 2
      for (int b = 0; b < rn; ++b) {
        const C v0 = col[b * DT];
#pragma unroll
        for (int q = 0; q < RH / 2; ++q) {
          const double2 bb = B2[b * (RM / 2) + q];
          b_fma(c0[2 * q], bb.x, v0);
          b_fma(c0[2 * q + 1], bb.y, v0);
        }
      }
      __syncwarp();
#pragma unroll
      for (int q = 0; q < RH; ++q)
        if (h * RH + q < rn) col[(h * RH + q) * DT] = c0[q];
    }
    if (!producer) asm volatile("bar.sync 1, 256;" ::: "memory");  // (kJgThreads)
    const int64_t n = a.blk0 + (int64_t)nbk * TN + t;
    if (!producer && db < L.NDB && n >= a.chunk0 && n < a.chunk1) {
      const int rn = rn_[t * (RM + 1)];
      const C* P = ps + t * L.SP + sb;
      const C* Cn = pd + t * L.SD + db * 4;
      C acc[4][4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) acc[u][v] = s_zero(C());
#pragma unroll 2
      for (int q = 0; q < rn; ++q) {
        C pv[4], cv[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          pv[u] = P[q * ST + u * NSB];
          cv[u] = Cn[q * DT + u];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int v = 0; v < 4; ++v) acc[u][v] = s_fma(pv[u], cv[v], acc[u][v]);
      }
      float* const Jn = J + (n - a.node0) + a.col0;
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const int d = d0 + db * 4 + v;
        if (d >= nd) break;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int s = s0 + sb + u * NSB;
          if (s >= nsu || sb + u * NSB >= ST) break;
          float* const o = Jn + ((int64_t)d * nsu + s) * a.ldj;
          if constexpr (SPLIT) {
            o[0] = (float)acc[u][v].x;
            o[a.nsd * a.ldj] = (float)acc[u][v].y;
          } else {
            o[0] = (float)acc[u][v];
          }
        }
      }
    }
    keep(after, me - mb, mm);  // (that slot's item is done with)
    // the buffer's reads and writes come before the copies that refill it
    if (bulk) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (NBUF == 1 && item + step < items) {
      __syncthreads();
      if (producer) {
        if (bulk) fetch_bulk(item + step, next, 0);
        else fetch(item + step, next, 0);
      }
    }
    slot = next;
  }
}

// nodes per launch: B of a chunk stays in L2
static int64_t jg_chunk(int rmax, int RM) {
  const int64_t per = (int64_t)rmax * RM * 8;
  return std::max<int64_t>(1024, (int64_t(48) << 20) / per / 8 * 8);
}
static int jg_rm(int rmax) { return rmax <= 16 ? 16 : 32; }
// the fraction of the tiles' pairs that exist
template <typename C>
static double jg_fill(int rmax, int nsu, int nd) {
  const JgLayout L = rmax <= 16 ? jg_layout<C, 8, 16>(rmax, nsu, nd, 2) : jg_layout<C, 4, 32>(rmax, nsu, nd, 2);
  return (double)nsu * nd / ((double)L.nst * L.ST * L.ndt * L.DT);
}

template <typename C, bool SPLIT, int RM, int TN>
static int jg_run(JgArgs a, int64_t node1, const C* phi, float* J, double* work, bool* done, cudaStream_t st) {
  int* const err = jac_err_word();
  if (!err) return fail(RB_ECUDA, "rb_jac_multi: no error word");
  int nbuf = 2;
  JgLayout L = jg_layout<C, TN, RM>(a.rmax, a.nsu, a.nd, 2);
  if (L.total > kJgSmem) {
    nbuf = 1;
    L = jg_layout<C, TN, RM>(a.rmax, a.nsu, a.nd, 1);
    if (L.total > kJgSmem) return RB_OK;
  }
  auto kern = nbuf == 2 ? jac_grid_kernel<C, SPLIT, RM, TN, 2> : jac_grid_kernel<C, SPLIT, RM, TN, 1>;
  RB_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kJgSmem));
  const int ntile = L.nst * L.ndt;
  const int64_t chunk = jg_chunk(a.rmax, RM);
  // node blocks start where the J column is a multiple of the block: the row's
  // sectors are then written whole (rows are 32-byte aligned when ldj % 8 == 0)
  const int64_t shift = (a.col0 + (int64_t)((reinterpret_cast<uintptr_t>(J) / 4) % TN)) % TN;
  for (int64_t c = a.node0; c < node1; c = a.chunk1) {
    a.chunk0 = c;
    a.blk0 = c - (c - a.node0 + shift) % TN;
    a.chunk1 = std::min(node1, a.blk0 + chunk);  // the next launch starts on a block
    constexpr int bw = jg_bwarps<RM>();
    jac_b_kernel<RM><<<(unsigned)std::min<int64_t>(ceil_div(a.chunk1 - c, bw), 148 * 64), bw * 32, 0, st>>>(a, work);
    RB_LAUNCH_CHECK();
    const int64_t items = ceil_div(a.chunk1 - a.blk0, TN) * ntile;
    kern<<<(unsigned)std::min<int64_t>(items, 148), kJgThreads + kJgProducers, L.total, st>>>(a, phi, work, J, (int32_t)items, err);
    RB_LAUNCH_CHECK();
  }
  *done = true;
  return RB_OK;
}

template <typename C, bool SPLIT>
static int jg_pick(const JgArgs& a, int64_t node1, const C* phi, float* J, double* work, bool* done, cudaStream_t st) {
  if (a.rmax <= 16) return jg_run<C, SPLIT, 16, 8>(a, node1, phi, J, work, done, st);
  return jg_run<C, SPLIT, 32, 4>(a, node1, phi, J, work, done, st);
}

}  // namespace rb

using namespace rb;

extern "C" {

size_t rb_jac_multi_work_bytes(int32_t rmax, int32_t nsu, int32_t ndet, int32_t is_complex) {
  if (rmax < 1 || rmax > 32 || nsu < 1 || ndet < 1) return 0;
  // the tiles must be filled: seven tenths of them with real fields, four with
  // complex ones.  16,926 nodes x 2 quantities, jac_kernel / this, ms: real
  // 1 x 1 pairs (1/16 filled) 0.37 / 0.43, 2 x 3 (3/8) 0.37 / 0.43, 33 x 17 (0.44)
  // 0.83 / 0.90, 5 x 7 (0.55) 0.43 / 0.43, 11 x 13 (0.74) 0.57 / 0.44; complex 1 x 1
  // 0.38 / 0.40, 2 x 3 0.44 / 0.41, 33 x 17 1.12 / 1.01, 11 x 13 0.61 / 0.45, 61 x 64
  // 3.80 / 1.82
  const double fill = is_complex ? jg_fill<cdouble>(rmax, nsu, ndet) : jg_fill<double>(rmax, nsu, ndet);
  if (fill < (is_complex ? 0.4 : 0.7)) return 0;
  const int RM = jg_rm(rmax);
  return (size_t)jg_chunk(rmax, RM) * rmax * RM * sizeof(double) + 256;
}

// Where the pipelined kernel is the faster one.  Rows of at most 16 neighbours:
// wherever its tiles are filled, but real 3 x 4 pairs (8,400 nodes x 2 quantities,
// jac_kernel / this, ms: 0.25 / 0.29; 4 x 4 0.30 / 0.27).
// Longer rows: an item has four nodes and half of the threads' columns, a
// store half a sector, so it depends on the other side, which is as fast as it
// has nodes at work on an SM (R).  Meshes of Delaunay tets, rmax 24 to 32, ms:
// R >= 12 (small rows and few columns) goes to jac_kernel: 12,000 nodes real 8 x 8
// 0.51 / 0.50, 60,480 nodes 4 x 4 1.92 / 2.11, 12 x 12 2.00 / 2.11, complex 5 x 7 at
// 9,196 0.44 / 0.49.  Complex below that comes here: 60,480 nodes 16 x 16 4.43 /
// 2.45, 64 x 64 17.4 / 11.0, 61 x 64 19.3 / 11.0, rmax 32 18.3 / 13.8; real counts off
// 4 as well: 61 x 64 11.5 / 8.3.  Real blocked pairs: a fit to 30 counts, us per
// node; 60,480 nodes 16 x 16 2.74 / 2.09, 32 x 64 5.83 / 4.49, 64 x 48 6.84 / 6.03 here,
// 40 x 40 4.27 / 6.12, 56 x 56 6.99 / 7.71, 64 x 64 6.91 / 7.66 there (at rmax 29 R falls
// to 3: 20,160 nodes 3.20 / 2.85).
int rb_jac_multi_wins(int32_t rmax, int32_t emax, int32_t nsu, int32_t ndet, int32_t is_complex) {
  if (emax < 1 || emax > kJgMaxE || !rb_jac_multi_work_bytes(rmax, nsu, ndet, is_complex)) return 0;
  const double pairs = (double)nsu * ndet;
  if (rmax <= 16) return is_complex || pairs >= 16.0;
  const bool blocked = nsu % 4 == 0 && ndet % 4 == 0;
  const int R = jac_resident(is_complex != 0, blocked, rmax, nsu + ndet, ndet, emax);
  if (R >= 12) return 0;
  if (is_complex || !blocked || R < 4 || R >= 8) return 1;
  const JgLayout L = jg_layout<double, 4, 32>(rmax, nsu, ndet, 2);
  const double general = R >= 6 ? 0.053 + 1.2e-5 * pairs : 0.075 + 1.35e-5 * pairs;
  return 0.025 + 0.0137 * L.nst * L.ndt < general;
}

int rb_jac_multi(const rb_mesh* mesh, int32_t nparam, const int32_t* what, const int64_t* col0, const void* phi,
                 int32_t phi_kind, int64_t ld, const int32_t* cols, int32_t nc, int32_t det0, int32_t ndet,
                 const int32_t* pair_src, const int32_t* pair_det, int64_t nsd, void* J, int64_t ldj, int32_t out_kind,
                 int32_t rmax, int32_t emax, const double* evol, const double* ddd, int64_t node0, int64_t count,
                 void* work, size_t work_bytes, void* stream) {
  if (!mesh || !what || !col0 || nparam < 1) return fail(RB_EARG, "rb_jac_multi: bad arguments");
  bool done = false;
  // the full grid (nsd < 0) of FP64 fields into FP32 rows formed in FP64, where
  // the staging fits; everything else through rb_jac_range
  const bool cx = phi_kind == RB_C128 && out_kind == RB_JAC_SPLIT_F32_ACC64;
  const bool re = phi_kind == RB_F64 && out_kind == RB_JAC_F32_ACC64;
  const size_t need = rb_jac_multi_work_bytes(rmax, det0, ndet, cx);
  if (nsd < 0 && (cx || re) && need && work && work_bytes >= need && (reinterpret_cast<uintptr_t>(work) & 15) == 0 &&
      emax <= kJgMaxE && phi && cols && pair_src && pair_det && J && evol && nc >= 1 && ndet >= 1 && det0 >= 1 &&
      det0 + ndet <= nc && det0 + ndet <= 128 && det0 <= 64 && -nsd == (int64_t)det0 * ndet && node0 >= 0 && count > 0 && node0 + count <= mesh->nn && ldj >= count) {
    bool ok = (reinterpret_cast<uintptr_t>(phi) & (cx ? 15 : 7)) == 0;
    for (int p = 0; p < nparam; ++p) ok = ok && what[p] >= JG_MUA_REF && what[p] <= JG_D && (what[p] != JG_D || ddd);
    if (ok) {
      JgArgs a{};
      a.indptr = mesh->indptr;
      a.indices = mesh->indices;
      a.eptr = mesh->node_eptr;
      a.elist = mesh->node_elist;
      a.elem = reinterpret_cast<const int4*>(mesh->elem);
      a.evol = evol;
      a.ddd = ddd;
      a.cols = cols;
      a.nsu = det0;
      a.det0 = det0;
      a.nd = ndet;
      a.rmax = rmax;
      a.ld = ld;
      a.ldj = ldj;
      a.nsd = -nsd;
      a.node0 = node0;
      cudaStream_t st = as_stream(stream);
      for (int p = 0; p < nparam; ++p) {
        a.what = what[p];
        a.col0 = col0[p];
        done = false;
        if (cx) RB_TRY((jg_pick<cdouble, true>(a, node0 + count, (const cdouble*)phi, (float*)J, (double*)work, &done, st)));
        else RB_TRY((jg_pick<double, false>(a, node0 + count, (const double*)phi, (float*)J, (double*)work, &done, st)));
        if (!done) break;  // (the staging's size does not depend on the quantity)
      }
    }
  }
  if (done) return RB_OK;
  if (nsd < 0 && (det0 % 4 || ndet % 4)) nsd = -nsd;  // (rb_jac's grid form takes multiples of 4)
  const int esz = out_kind == RB_JAC_SPLIT_BF16 || out_kind == RB_JAC_BF16 ? 2
                  : out_kind == RB_F64 || out_kind == RB_C64 || out_kind == RB_JAC_SPLIT_F64 ? 8
                  : out_kind == RB_C128 ? 16 : 4;
  for (int p = 0; p < nparam; ++p)
    RB_TRY(rb_jac_range(mesh, what[p], phi, phi_kind, ld, cols, nc, det0, ndet, pair_src, pair_det, nsd,
                        J ? (char*)J + col0[p] * esz : nullptr, ldj, out_kind, rmax, emax, evol,
                        what[p] == JG_D ? ddd : nullptr, node0, count, stream));
  return RB_OK;
}

}  // extern "C"
