// Batched right-hand sides: up to kMaxRhs sources solved together on one set
// of subdomain factors (the reference solves one source per HDDM run,
// hddm_solver.h:25-183; several sources are several runs of the same loop).
//
// Every vector is stored right-hand-side minor, [row][kMaxRhs], so that the
// 16 values of one DOF are one 256-byte (FP64) line.  The subdomain phase of
// an iteration is three launches, as in the single-source staged path:
//   multi_rhs_kernel     f_I - A_IG v for every (interior row, two sources),
//   multi_sweep_kernel   the envelope sweeps, one CTA per subdomain and
//                        kRS sources; the factor entries come from the
//                        TMA-staged row blocks as shared-memory broadcasts,
//                        so one staged block serves kRS sources,
//   multi_iface_kernel   q = A_G.[x; v] (- f_G) for every (slot, two sources).
// The COCG kernels keep one set of scalars and a stopping status per source
// (ITERATION_S, hddm_solver_s.h:260-400, per source); a finished source
// keeps its vectors while the others go on.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdint>
#include <type_traits>

#include "fw_device.cuh"
#include "fw_kernels.cuh"
#include "fw_launch.cuh"

namespace fw {

namespace {

using namespace dev;

constexpr int kR = kMaxRhs;
constexpr int kMT = 256;  // reduction blocks: 16 DOFs x 16 sources
enum { kMPqRe = 0, kMPqIm, kMMax, kMRzRe, kMRzIm, kML2, kMFields };

__device__ __forceinline__ bool multi_stopped(const MultiProblem &m, int mode) {
  return mode == kModeIter && m.ms->all_status != 0;
}

// ---- grid-wide products, one thread per (row, two sources) -------------------
// A row's entries and columns are the same for its 16 sources: with two of
// them per thread half as many threads load and decode them.

struct Pair {
  double2 a, b;
};
__device__ __forceinline__ Pair load_pair(const double2 *p) { return {p[0], p[1]}; }

__global__ void multi_rhs_kernel(MultiProblem m, int mode, double2 *__restrict__ out) {
  chain_begin();
  if (multi_stopped(m, mode)) return;
  const DevProblem &p = m.p;
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int r = 2 * (int)(t % (kR / 2));
  const int64_t i = t / (kR / 2);
  if (i >= p.n_interior) return;
  const int64_t row = p.row0 + i;
  Pair acc = {cz(), cz()};
  if (mode != kModeFirst) {
    const int64_t q1 = p.cpl_rowptr[row + 1];
#pragma unroll 4
    for (int64_t q = p.cpl_rowptr[row]; q < q1; q++) {
      const double2 v = p.cpl_val[q];
      const Pair x = load_pair(m.P + (int64_t)p.cpl_gcol[q] * kR + r);
      acc.a = cadd(acc.a, cmul(v, x.a));
      acc.b = cadd(acc.b, cmul(v, x.b));
    }
  }
  const Pair f = mode != kModeIter ? load_pair(m.fI + row * kR + r) : Pair{cz(), cz()};
  out[row * kR + r] = csub(f.a, acc.a);
  out[row * kR + r + 1] = csub(f.b, acc.b);
}

__global__ void multi_iface_kernel(MultiProblem m, int mode) {
  chain_begin();
  if (multi_stopped(m, mode)) return;
  const DevProblem &p = m.p;
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int r = 2 * (int)(t % (kR / 2));
  const int64_t i = t / (kR / 2);
  if (i >= p.n_slots) return;
  const int64_t slot = p.slot0 + i;
  const bool with_bc = mode != kModeFirst;
  Pair acc = {cz(), cz()};
  const int64_t q1 = p.ifr_rowptr[slot + 1];
#pragma unroll 4
  for (int64_t q = p.ifr_rowptr[slot]; q < q1; q++) {
    const int64_t g = p.ifr_gcol[q];
    const double2 v = p.ifr_val[q];
    const Pair x = g >= 0 ? load_pair(m.Y + g * kR + r) : (with_bc ? load_pair(m.P + (-g - 1) * kR + r) : Pair{cz(), cz()});
    acc.a = cadd(acc.a, cmul(v, x.a));
    acc.b = cadd(acc.b, cmul(v, x.b));
  }
  if (mode != kModeIter) {
    const Pair f = load_pair(m.fG + slot * kR + r);
    acc.a = csub(acc.a, f.a);
    acc.b = csub(acc.b, f.b);
  }
  m.qloc[slot * kR + r] = acc.a;
  m.qloc[slot * kR + r + 1] = acc.b;
  if (mode == kModeLast) {
    const Pair v = with_bc ? load_pair(m.P + (int64_t)p.if_ln[slot] * kR + r) : Pair{cz(), cz()};
    m.V[slot * kR + r] = v.a;
    m.V[slot * kR + r + 1] = v.b;
  }
}

__global__ void multi_residual_kernel(MultiProblem m, int mode) {
  if (multi_stopped(m, mode)) return;
  const DevProblem &p = m.p;
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int r = 2 * (int)(t % (kR / 2));
  const int64_t i = t / (kR / 2);
  if (i >= p.n_interior) return;
  const int64_t row = p.row0 + i;
  Pair acc = {cz(), cz()};
  const int64_t q1 = p.aii_rowptr[row + 1];
#pragma unroll 4
  for (int64_t q = p.aii_rowptr[row]; q < q1; q++) {
    const double2 v = p.aii_val[q];
    const Pair x = load_pair(m.Y + (int64_t)p.aii_gcol[q] * kR + r);
    acc.a = cadd(acc.a, cmul(v, x.a));
    acc.b = cadd(acc.b, cmul(v, x.b));
  }
  const Pair f = load_pair(m.B + row * kR + r);
  m.Rres[row * kR + r] = csub(f.a, acc.a);
  m.Rres[row * kR + r + 1] = csub(f.b, acc.b);
}

// ---- the sweeps --------------------------------------------------------------

constexpr int kRS = 8;             // sources of one CTA
constexpr int kSweepThreads = 32 * kMultiSweepWarps;  // 32 rows (or columns) x kRS sources at a time

struct MultiLayout {
  size_t y, buf0, buf1, dinv, meta, rect, bar, blk, total;
  int tight;  // one row table, no 1/d in shared memory
};

inline MultiLayout multi_layout(int max_interior, int max_blocks, int cap, bool fp32) {
  const size_t es = fp32 ? 8 : 16;
  MultiLayout l;
  // the largest subdomains (FP64: interiors over about 1,330 DOFs, up to
  // about 1,500) leave no room for the pivots and a second row table: their
  // sweeps read the pivots again from the factor and wait for each block's
  // table
  for (l.tight = 0; l.tight < 2; l.tight++) {
    size_t o = 0;
    l.y = o;
    o += a16((size_t)max_interior * kRS * es);
    l.buf0 = o;
    o += a16((size_t)cap * es);
    l.buf1 = o;
    o += a16((size_t)cap * es);
    l.dinv = o;
    if (!l.tight) o += a16((size_t)max_interior * es);
    l.meta = o;
    o += (l.tight ? 1 : 2) * 32 * 8;
    l.rect = o;
    o += a16((size_t)32 * kRS * es);
    l.bar = o;
    o += 16;
    l.blk = o;
    o += a16(((size_t)max_blocks + 1) * 8);
    l.total = o;
    if (l.tight || o <= 227 * 1024) break;
  }
  return l;
}

// One CTA per (subdomain, kRS sources); the sources' vectors stay in shared
// memory, y[row][kRS].  Per staged block of rows r0 .. r0+nb-1:
//   forward  - the entries left of the block: thread (row, source) sums the
//              row's entries in order, even and odd ones apart;
//              then the triangle: one warp per source, lane t holding row t.
//              A row's sum over the block's columns is split into kQ strands
//              (column k0 + h, k0 + h + kQ, ...) of two alternating sums each,
//              added pairwise: lane t keeps all 2 kQ of them and takes column
//              j as soon as row j is final, so the strands cost no shuffle;
//   backward - the triangle from the last row, one warp per source with lanes
//              over columns; then the columns left of the block: thread
//              (column, source) applies the block's rows from the last to the
//              first in place.
// The order of every sum is that of a row taken by kQ lane groups (FP64: 4,
// FP32: 2), whatever the number of warps.  One warp for all the sources of a
// subdomain, as before, left each row a chain of shuffles on one warp per
// scheduler (16 sources on 551 subdomains of up to 600 elements: 1.96 ms per
// iteration, 0.73 so; FP32+IR on 123 of up to 1,000: 8.26 and 0.93 ms).
template <typename T>
__global__ void __launch_bounds__(kSweepThreads, 2) multi_sweep_kernel(MultiProblem m, int mode, const double2 *rhs,
                                                                   double2 *xout, int accumulate, MultiLayout lay,
                                                                   int first) {
  constexpr int kQ = sizeof(T) == 8 ? 2 : 4;
  constexpr int kParts = kR / kRS;
  constexpr int nt = kSweepThreads, nw = nt / 32;
  if (multi_stopped(m, mode)) return;
  const DevProblem &p = m.p;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int part = blockIdx.x % kParts;  // which kRS sources
  const int s = p.sub_order[first + blockIdx.x / kParts];
  const int64_t io = p.int_off[s];
  const int nI = (int)(p.int_off[s + 1] - io);
  const int b0 = p.blk_off[s];
  const int nblk = p.blk_off[s + 1] - b0 - 1;
  if (nI == 0 || nblk <= 0) return;
  T *__restrict__ y = (T *)(smem_raw + lay.y);
  T *__restrict__ dinv = (T *)(smem_raw + lay.dinv);
  int2 *rows = (int2 *)(smem_raw + lay.meta);
  const int tabs = lay.tight ? 0 : 1;  // mask of the row tables
  T *__restrict__ rect = (T *)(smem_raw + lay.rect);
  int2 *blk = (int2 *)(smem_raw + lay.blk);
  Stage<T> st;
  st.buf0 = (T *)(smem_raw + lay.buf0);
  st.buf1 = (T *)(smem_raw + lay.buf1);
  st.bar = (uint64_t *)(smem_raw + lay.bar);
  st.blk = blk;
  stage_init(st, &m.ms->err, 0);
  const int64_t base = p.env_ptr[io];
  st.L = (sizeof(T) == 8 ? (const T *)(const void *)p.L32 : (const T *)(const void *)p.L64) + base;
  for (int b = tid; b <= nblk; b += nt) blk[b] = p.blk_tab[b0 + b];
  if (tid == 0) {
    mbar_init(&st.bar[0], 1);
    mbar_init(&st.bar[1], 1);
    fence_mbar_init();
  }
  // global vectors are [row][16]; this CTA's sources are kRS*part ..
  const int64_t g0 = io * kR + part * kRS;
  for (int e = tid; e < nI * kRS; e += nt) y[e] = from_d2<T>(rhs[g0 + (int64_t)(e / kRS) * kR + (e % kRS)]);
  __syncthreads();
  const int2 *rows_g = p.row_tab + io;
  const int r = tid % kRS, row = tid / kRS;  // of the (row, source) passes
  constexpr int kRows = nt / kRS;

  // forward
  bool ok = true;
  stage_issue(st, 0, tid);
  if (warp == 0) rows_issue(st, rows_g, rows, 0, lane);
  for (int b = 0; b < nblk; b++) {
    const int r0 = blk[b].x, nb = blk[b + 1].x - r0;
    const int2 *meta = rows + (b & tabs) * 32;
    const bool next = b + 1 < nblk;
    if (next) stage_issue(st, b + 1, tid);
    if (warp == 0) rows_wait();
    const bool late = !stage_wait(st, b);
    if (__syncthreads_or(late)) {
      ok = false;
      break;
    }
    if (warp == 0 && next && tabs) rows_issue(st, rows_g, rows + ((b + 1) & tabs) * 32, b + 1, lane);
    const T *S = ((b & 1) ? st.buf1 : st.buf0) - stage_a0(st, b);
    const int my_lo = meta[lane].x, my_pr = meta[lane].y;
    // entries left of the block
    for (int t = row; t < nb; t += kRows) {
      const int2 mt = meta[t];
      const int len = max(0, r0 - mt.x);
      const T *__restrict__ rw = S + mt.y;
      const T *__restrict__ yk = y + mt.x * kRS + r;
      T a0 = czero<T>(), a1 = czero<T>();
      int k = 0;
      for (; k + 3 < len; k += 4) {
        T w[4], v[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
          w[u] = rw[k + u];
          v[u] = yk[(k + u) * kRS];
        }
        a0 = cmac(a0, w[0], v[0]);
        a1 = cmac(a1, w[1], v[1]);
        a0 = cmac(a0, w[2], v[2]);
        a1 = cmac(a1, w[3], v[3]);
      }
      for (; k < len; k += 2) {
        a0 = cmac(a0, rw[k], yk[k * kRS]);
        if (k + 1 < len) a1 = cmac(a1, rw[k + 1], yk[(k + 1) * kRS]);
      }
      rect[t * kRS + r] = cadd(a0, a1);
    }
    __syncthreads();
    // the triangle
    for (int q = warp; q < kRS; q += nw) {
      const bool in = lane < nb;
      const T rc = in ? rect[lane * kRS + q] : czero<T>();
      const T yv = in ? y[(r0 + lane) * kRS + q] : czero<T>();
      const T *mine = S + my_pr - my_lo + r0;  // mine[j]: this lane's row at the block's column j
      const int s0 = max(0, my_lo - r0);       // its first column in the block
      // strand of column j: (j - s0) mod 2 kQ.  The sums are kept at j mod
      // 2 kQ; which two strands are added first then depends on s0's parity
      T a[2 * kQ], h[kQ];  // strands, and each pair's sum
#pragma unroll
      for (int u = 0; u < 2 * kQ; u++) a[u] = czero<T>();
#pragma unroll
      for (int u = 0; u < kQ; u++) h[u] = czero<T>();
      T e0 = czero<T>(), e1 = czero<T>();  // the two pairs of pairs (kQ = 4): {0, 1} and {2, 3}, or {0, 3} and {2, 1}
      const bool odd = s0 & 1;
      T val = czero<T>();
      for (int j0 = 0; j0 < nb; j0 += 2 * kQ) {
        T op[2 * kQ];
#pragma unroll
        for (int u = 0; u < 2 * kQ; u++) op[u] = lane > j0 + u && in && j0 + u >= s0 ? mine[j0 + u] : czero<T>();
#pragma unroll
        for (int u = 0; u < 2 * kQ; u++) {
          const int j = j0 + u;
          if (j < nb) {
            const T tot = kQ == 2 ? cadd(h[0], h[1]) : cadd(e0, e1);
            const T fin = csub(yv, cadd(rc, tot));
            if (lane == j) val = fin;
            const T yj = shfl_idx(fin, j);
            if (lane > j && j >= s0) {
              a[u] = cmac(a[u], op[u], yj);
              constexpr int kH = kQ - 1;
              h[u & kH] = cadd(a[u & kH], a[(u & kH) + kQ]);
              if (kQ == 4) {
                // only the sum that holds this strand changes
                if ((u & kH) == 0) e0 = cadd(h[0], odd ? h[kQ - 1] : h[1]);
                if ((u & kH) == 1) {
                  const T v = cadd(h[1], odd ? h[2 % kQ] : h[0]);
                  if (odd)
                    e1 = v;
                  else
                    e0 = v;
                }
                if ((u & kH) == 2) e1 = cadd(h[2 % kQ], odd ? h[1] : h[kQ - 1]);
                if ((u & kH) == 3) {
                  const T v = cadd(h[kQ - 1], odd ? h[0] : h[2 % kQ]);
                  if (odd)
                    e0 = v;
                  else
                    e1 = v;
                }
              }
            }
          }
        }
      }
      if (in) {
        y[(r0 + lane) * kRS + q] = val;
        if (q == 0 && tabs) dinv[r0 + lane] = mine[lane];  // 1/d on the diagonal
      }
    }
    __syncthreads();
    if (warp == 0 && next && !tabs) rows_issue(st, rows_g, rows, b + 1, lane);
  }
  if (ok) {
    if (tabs) {
      for (int e = tid; e < nI * kRS; e += nt) y[e] = cmul_rn(dinv[e / kRS], y[e]);
    } else {
      for (int e = tid; e < nI * kRS; e += nt) {
        const int i = e / kRS;
        const int2 t = rows_g[i];
        y[e] = cmul_rn(st.L[t.y + i - t.x], y[e]);
      }
    }
    __syncthreads();
  }

  // backward
  for (int b = nblk - 1; b >= 0 && ok; b--) {
    const int r0 = blk[b].x, nb = blk[b + 1].x - r0;
    const int2 *meta = rows + (b & tabs) * 32;
    // the forward sweep left blocks nblk-1 and nblk-2 in the buffers, and their row tables
    const bool next = b >= 1 && b - 1 < nblk - 2;
    if (next) stage_issue(st, b - 1, tid);
    if (warp == 0) rows_wait();
    const bool late = !stage_wait(st, b);
    if (__syncthreads_or(late)) {
      ok = false;
      break;
    }
    if (warp == 0 && next && tabs) rows_issue(st, rows_g, rows + ((b - 1) & tabs) * 32, b - 1, lane);
    const int my_lo = meta[lane].x;
    const int bmin = __reduce_min_sync(0xffffffffu, lane < nb ? my_lo : INT_MAX);
    const T *S = ((b & 1) ? st.buf1 : st.buf0) - stage_a0(st, b);
    // the triangle from the last row, lanes over the block's columns
    for (int q = warp; q < kRS; q += nw) {
      T val = lane < nb ? y[(r0 + lane) * kRS + q] : czero<T>();
      const int col = r0 + lane;
      for (int i0 = nb - 1; i0 >= 1; i0 -= 4) {
        T op[4];
        bool act[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const int i = i0 - u;
          const int2 mt = meta[max(i, 0)];
          act[u] = i >= 1 && lane < i && col >= mt.x;
          op[u] = act[u] ? S[mt.y + col - mt.x] : czero<T>();
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const T xi = shfl_idx(val, max(i0 - u, 0));
          if (act[u]) val = cmsub(val, op[u], xi);
        }
      }
      if (lane < nb) y[(r0 + lane) * kRS + q] = val;
    }
    __syncthreads();
    // the columns left of the block: a warp's four columns take the rows that
    // reach them, from the last
    for (int cb = bmin + warp * (32 / kRS); cb < r0; cb += kRows) {
      const int c = cb + lane / kRS;
      uint32_t rows = __ballot_sync(0xffffffffu, lane < nb && my_lo < cb + 32 / kRS);
      const bool in = c < r0;
      T yc = in ? y[c * kRS + r] : czero<T>();
      while (rows) {
        T w[4], x[4];
        bool act[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const int t = rows ? 31 - __clz(rows) : 0;
          const int2 mt = meta[t];
          act[u] = rows && in && c >= mt.x;
          w[u] = act[u] ? S[mt.y + c - mt.x] : czero<T>();
          x[u] = y[(r0 + t) * kRS + r];
          rows &= ~(1u << t);
        }
#pragma unroll
        for (int u = 0; u < 4; u++)
          if (act[u]) yc = cmsub(yc, w[u], x[u]);
      }
      if (in) y[c * kRS + r] = yc;
    }
    __syncthreads();
    if (warp == 0 && b >= 1 && !tabs) rows_issue(st, rows_g, rows, b - 1, lane);
  }
  // every copy issued into this CTA's shared memory has landed before it exits
  stage_drain(st);
  if (!ok) return;
  for (int e = tid; e < nI * kRS; e += nt) {
    const int64_t ge = g0 + (int64_t)(e / kRS) * kR + (e % kRS);
    double2 x = make_double2((double)y[e].x, (double)y[e].y);
    if (accumulate) x = cadd(xout[ge], x);
    xout[ge] = x;
  }
}

// ---- COCG, one set of scalars per source ------------------------------------

// per-source block reductions of N fields (field f a maximum where bit f of
// kMax is set): thread (gi, r) = (threadIdx.x >> 4, & 15) brings source r's
// values; field gi's result is valid in the threads gi < N.  sh: N (kMT +
// kMT / kR) doubles.
template <int N, unsigned kMax>
__device__ __forceinline__ double block_reduce_r(const double (&v)[N], double *sh) {
  constexpr int kW = kMT / kR * (kR + 1);
  const int r = threadIdx.x & (kR - 1), gi = threadIdx.x >> 4;
  __syncthreads();
#pragma unroll
  for (int f = 0; f < N; f++) sh[f * kW + gi * (kR + 1) + r] = v[f];
  __syncthreads();
  double a = 0.0;
  if (gi < N) {
    const bool is_max = kMax >> gi & 1;
    for (int j = 0; j < kMT / kR; j++) {
      const double x = sh[gi * kW + j * (kR + 1) + r];
      a = is_max ? fmax(a, x) : a + x;
    }
  }
  return a;
}

// this CTA's partials of fields f0 .. f0 + N - 1
template <int N, unsigned kMax>
__device__ __forceinline__ void write_parts(const MultiProblem &m, int f0, const double (&v)[N], double *sh) {
  const double a = block_reduce_r<N, kMax>(v, sh);
  const int gi = threadIdx.x >> 4;
  if (gi < N) m.part[((int64_t)(f0 + gi) * m.p.n_part_blocks + blockIdx.x) * kR + (threadIdx.x & (kR - 1))] = a;
}

// the last CTA: the fields of source r over all blocks, blocks split over the
// 16 thread groups and combined in group order (fixed order); out[] in every thread
template <int N, unsigned kMax>
__device__ __forceinline__ void reduce_parts(const MultiProblem &m, int f0, double *sh, double (&out)[N]) {
  const int r = threadIdx.x & (kR - 1), gi = threadIdx.x >> 4;
  const int nb = m.p.n_part_blocks;
  double a[N];
#pragma unroll
  for (int f = 0; f < N; f++) a[f] = 0.0;
  for (int j = gi; j < nb; j += kMT / kR) {
#pragma unroll
    for (int f = 0; f < N; f++) {
      const double x = __ldcg(m.part + ((int64_t)(f0 + f) * nb + j) * kR + r);
      a[f] = (kMax >> f & 1) ? fmax(a[f], x) : a[f] + x;
    }
  }
  const double t = block_reduce_r<N, kMax>(a, sh);
  __syncthreads();
  if (gi < N) sh[gi * kR + r] = t;
  __syncthreads();
#pragma unroll
  for (int f = 0; f < N; f++) out[f] = sh[f * kR + r];
}

__device__ __forceinline__ double2 gather_slots_r(const DevProblem &p, const double2 *v, int g, int r) {
  double2 q = cz();
  for (int t = p.gq_ptr[g]; t < p.gq_ptr[g + 1]; t++) q = cadd(q, v[p.gq_slot[t] * kR + r]);
  return q;
}

__global__ void multi_set_status_kernel(MultiScalars *ms, double eps, int32_t max_loop) {
  for (int r = 0; r < kR; r++) {
    ms->s[r].eps = eps;
    ms->s[r].max_loop = max_loop;
    ms->s[r].status = 0;
    ms->s[r].converged = 0;
    ms->s[r].nonfinite = 0;
  }
  ms->all_status = 0;
  for (int i = 0; i < 4; i++) ms->ticket[i] = 0;
}

// first step of every source (hddm_solver_s.h:158-256): Q, PC, r = q, z, p, max|r|, (r, z)
__global__ void multi_first_kernel(MultiProblem m, const double2 *__restrict__ pcloc) {
  __shared__ double sh[4 * (kMT + kMT / kR)];
  const DevProblem &p = m.p;
  const int r = threadIdx.x & (kR - 1), gi = threadIdx.x >> 4;
  double mx = 0.0, rzr = 0.0, rzi = 0.0, l2 = 0.0;
  for (int g = blockIdx.x * (kMT / kR) + gi; g < p.nfree; g += gridDim.x * (kMT / kR)) {
    const double2 q = gather_slots_r(p, m.qloc, g, r);
    double2 pc = cz();
    for (int t = p.gq_ptr[g]; t < p.gq_ptr[g + 1]; t++) pc = cadd(pc, pcloc[p.gq_slot[t]]);
    pc = ciszero(pc) ? make_double2(1.0, 0.0) : cdiv_ref(make_double2(1.0, 0.0), pc);
    if (r == 0) m.PC[g] = pc;
    const int64_t e = (int64_t)g * kR + r;
    m.Q[e] = q;
    m.R[e] = q;
    const double2 z = cmul(q, pc);
    m.Z[e] = z;
    m.P[e] = z;
    m.U[e] = cz();
    mx = fmax(mx, cabs_ref(q));
    const double2 rz = cmul(q, z);
    rzr += rz.x;
    rzi += rz.y;
    l2 += q.x * q.x + q.y * q.y;
  }
  const double part[4] = {mx, rzr, rzi, l2};
  write_parts<4, 1>(m, kMMax, part, sh);
  if (!last_cta(&m.ms->ticket[0])) return;
  double all[4];
  reduce_parts<4, 1>(m, kMMax, sh, all);
  const double vmx = all[0], vrr = all[1], vri = all[2], vl2 = all[3];
  if (gi == 0) {
    CocgScalars &c = m.ms->s[r];
    c.norm0 = vmx;
    c.l2_0 = sqrt(vl2);
    c.r0inv = vmx > 0.0 ? 1.0 / vmx : 0.0;
    c.rz = make_double2(vrr, vri);
    c.resi = 1.0;
    c.resi_l2 = 1.0;
    c.loop = 1;
    const bool bad = !isfinite(vmx) || !isfinite(vl2) || !isfinite(vrr) || !isfinite(vri);
    c.status = (bad || vmx < kNearlyZero) ? 1 : 0;
    c.converged = (!bad && vmx < kNearlyZero) ? 1 : 0;
    c.nonfinite = bad ? 1 : 0;
  }
  if (threadIdx.x == 0) m.ms->ticket[0] = 0;
}

// Q and (p, q); last CTA: -alpha per iterating source
__global__ void multi_pq_kernel(MultiProblem m) {
  chain_begin();
  if (m.ms->all_status != 0) return;
  __shared__ double sh[2 * (kMT + kMT / kR)];
  const DevProblem &p = m.p;
  const int r = threadIdx.x & (kR - 1), gi = threadIdx.x >> 4;
  double re = 0.0, im = 0.0;
  for (int g = blockIdx.x * (kMT / kR) + gi; g < p.nfree; g += gridDim.x * (kMT / kR)) {
    const int64_t e = (int64_t)g * kR + r;
    const double2 q = gather_slots_r(p, m.qloc, g, r);
    m.Q[e] = q;
    const double2 t = cmul(m.P[e], q);
    re += t.x;
    im += t.y;
  }
  const double part[2] = {re, im};
  write_parts<2, 0>(m, kMPqRe, part, sh);
  if (!last_cta(&m.ms->ticket[1])) return;
  double all[2];
  reduce_parts<2, 0>(m, kMPqRe, sh, all);
  const double pr = all[0], pi = all[1];
  if (gi == 0) {
    CocgScalars &c = m.ms->s[r];
    if (c.status == 0) {
      const double2 pq = make_double2(pr, pi);
      c.malpha = (cabs_ref(c.rz) < kNearlyZero && cabs_ref(pq) < kNearlyZero) ? cz() : csub(cz(), cdiv_ref(c.rz, pq));
    }
  }
  if (threadIdx.x == 0) m.ms->ticket[1] = 0;
}

// u += -alpha p, r += -alpha q, z, max|r|, (r, z); last CTA: resi, beta, stopping
__global__ void multi_update_kernel(MultiProblem m) {
  chain_begin();
  if (m.ms->all_status != 0) return;
  __shared__ double sh[4 * (kMT + kMT / kR)];
  const DevProblem &p = m.p;
  const int r = threadIdx.x & (kR - 1), gi = threadIdx.x >> 4;
  const bool live = m.ms->s[r].status == 0;
  const double2 ma = m.ms->s[r].malpha;
  double mx = 0.0, rzr = 0.0, rzi = 0.0, l2 = 0.0;
  if (live) {
    for (int g = blockIdx.x * (kMT / kR) + gi; g < p.nfree; g += gridDim.x * (kMT / kR)) {
      const int64_t e = (int64_t)g * kR + r;
      m.U[e] = cadd(m.U[e], cmul(ma, m.P[e]));
      const double2 rv = cadd(m.R[e], cmul(ma, m.Q[e]));
      m.R[e] = rv;
      mx = fmax(mx, cabs_ref(rv));
      const double2 z = cmul(rv, m.PC[g]);
      m.Z[e] = z;
      const double2 rz = cmul(rv, z);
      rzr += rz.x;
      rzi += rz.y;
      l2 += rv.x * rv.x + rv.y * rv.y;
    }
  }
  const double part[4] = {mx, rzr, rzi, l2};
  write_parts<4, 1>(m, kMMax, part, sh);
  if (!last_cta(&m.ms->ticket[2])) return;
  double all[4];
  reduce_parts<4, 1>(m, kMMax, sh, all);
  const double vmx = all[0], vrr = all[1], vri = all[2], vl2 = all[3];
  if (gi == 0) {
    CocgScalars &c = m.ms->s[r];
    if (c.status == 0) {
      const double resi = vmx * c.r0inv;
      c.resi = resi;
      c.resi_l2 = c.l2_0 > 0.0 ? sqrt(vl2) / c.l2_0 : 0.0;
      const double2 rz = make_double2(vrr, vri);
      c.beta = (cabs_ref(rz) < kNearlyZero && cabs_ref(c.rz) < kNearlyZero) ? cz() : cdiv_ref(rz, c.rz);
      c.rz = rz;
      if (!isfinite(vl2) || !isfinite(vrr) || !isfinite(vri)) {
        c.status = 1;
        c.nonfinite = 1;
      } else if (resi < c.eps) {
        c.status = 1;
        c.converged = 1;
      } else if (c.loop >= c.max_loop) {
        c.status = 1;
      }
      c.loop += 1;
    }
  }
  if (threadIdx.x == 0) m.ms->ticket[2] = 0;
}

// p = z + beta p, or p = u for a source that just stopped; last CTA marks
// stopped sources finished and the batch finished when all are
__global__ void multi_pupdate_kernel(MultiProblem m) {
  chain_begin();
  if (m.ms->all_status != 0) return;
  const DevProblem &p = m.p;
  const int r = threadIdx.x & (kR - 1), gi = threadIdx.x >> 4;
  const int st = m.ms->s[r].status;
  const double2 be = m.ms->s[r].beta;
  if (st != 2) {
    for (int g = blockIdx.x * (kMT / kR) + gi; g < p.nfree; g += gridDim.x * (kMT / kR)) {
      const int64_t e = (int64_t)g * kR + r;
      m.P[e] = st == 1 ? m.U[e] : cadd(m.Z[e], cmul(be, m.P[e]));
    }
  }
  if (!last_cta(&m.ms->ticket[3])) return;
  if (threadIdx.x == 0) {
    int all = 2;
    for (int k = 0; k < kR; k++) {
      if (m.ms->s[k].status == 1) m.ms->s[k].status = 2;
      if (m.ms->s[k].status != 2) all = 0;
    }
    m.ms->all_status = all;
    m.ms->ticket[3] = 0;
  }
}

__global__ void multi_edge_solution_kernel(int64_t ne, int k, const int64_t *__restrict__ src,
                                           const double2 *__restrict__ Y, const double2 *__restrict__ V,
                                           double2 *__restrict__ x) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= ne) return;
  const int64_t s = src[e];
  x[e] = s >= 0 ? Y[s * kR + k] : (s < -1 ? V[(-s - 2) * kR + k] : make_double2(0.0, 0.0));
}

__global__ void multi_put_kernel(int64_t n, int k, const double2 *__restrict__ src, double2 *__restrict__ dst) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i * kR + k] = src[i];
}

unsigned grid_for(int64_t n, int threads) { return n > 0 ? (unsigned)((n + threads - 1) / threads) : 1u; }

}  // namespace

size_t multi_smem_bytes(int max_interior, int max_blocks, int cap, bool fp32) {
  return multi_layout(max_interior, max_blocks, cap, fp32).total;
}

int multi_ctas_per_sm(size_t smem) { return (int)std::min<size_t>(2, (227 * 1024) / (smem + 1024)); }

int configure_multi(size_t smem, bool fp32) {
  return fp32 ? raise_smem_limit((const void *)multi_sweep_kernel<float2>, kSlotMulti32, smem)
              : raise_smem_limit((const void *)multi_sweep_kernel<double2>, kSlotMulti64, smem);
}

// The sweep, one launch per size bucket, each with the shared memory of its
// largest subdomain (a single bucket of every subdomain when none are set).
template <typename T>
static void launch_multi_sweep(const MultiProblem &m, int mode, bool fp32, const double2 *rhs, double2 *xout,
                               int accumulate, cudaStream_t stream) {
  const DevProblem &p = m.p;
  const int nb = m.n_buckets > 0 ? m.n_buckets : 1;
  for (int k = 0; k < nb; k++) {
    const int first = m.n_buckets > 0 ? m.bucket_first[k] : 0;
    const int count = m.n_buckets > 0 ? m.bucket_count[k] : p.nsub;
    const int mi = m.n_buckets > 0 ? m.bucket_max_interior[k] : p.max_interior;
    const int mb = m.n_buckets > 0 ? m.bucket_max_blocks[k] : p.max_blocks;
    if (count <= 0) continue;
    const MultiLayout lay = multi_layout(mi, mb, p.stage_cap, fp32);
    multi_sweep_kernel<T><<<(unsigned)count * (kR / kRS), kSweepThreads, lay.total, stream>>>(m, mode, rhs, xout,
                                                                                             accumulate, lay, first);
  }
}

void launch_multi_subsolve(const MultiProblem &m, int mode, bool fp32, cudaStream_t stream) {
  const DevProblem &p = m.p;
  const unsigned gi = grid_for(p.n_interior * kR / 2, 256), gs = grid_for(p.n_slots * kR / 2, 256);
  double2 *rhs = fp32 ? m.B : m.Y;
  launch_chained(multi_rhs_kernel, gi, 256, 0, stream, m, mode, rhs);
  if (fp32) {
    launch_multi_sweep<float2>(m, mode, true, m.B, m.Y, 0, stream);
    for (int k = 0; k < p.ir_steps; k++) {
      multi_residual_kernel<<<gi, 256, 0, stream>>>(m, mode);
      launch_multi_sweep<float2>(m, mode, true, m.Rres, m.Y, 1, stream);
    }
  } else {
    launch_multi_sweep<double2>(m, mode, false, m.Y, m.Y, 0, stream);
  }
  multi_iface_kernel<<<gs, 256, 0, stream>>>(m, mode);
}

int multi_iteration_launches(bool fp32, int ir_steps, int n_buckets) {
  const int nb = n_buckets > 0 ? n_buckets : 1;
  return 2 + nb * (fp32 ? 1 + ir_steps : 1) + (fp32 ? ir_steps : 0) + 3;
}

void launch_multi_set_status(MultiScalars *ms, double eps, int32_t max_loop, cudaStream_t stream) {
  multi_set_status_kernel<<<1, 1, 0, stream>>>(ms, eps, max_loop);
}

void launch_multi_first(const MultiProblem &m, const double2 *pcloc, cudaStream_t stream) {
  multi_first_kernel<<<m.p.n_part_blocks, kMT, 0, stream>>>(m, pcloc);
}

void launch_multi_iteration(const MultiProblem &m, bool fp32, cudaStream_t stream) {
  launch_multi_subsolve(m, kModeIter, fp32, stream);
  launch_chained(multi_pq_kernel, m.p.n_part_blocks, kMT, 0, stream, m);
  launch_chained(multi_update_kernel, m.p.n_part_blocks, kMT, 0, stream, m);
  launch_chained(multi_pupdate_kernel, m.p.n_part_blocks, kMT, 0, stream, m);
}

void launch_multi_put(int64_t n, int k, const double2 *src, double2 *dst, cudaStream_t stream) {
  if (n <= 0) return;
  multi_put_kernel<<<grid_for(n, 256), 256, 0, stream>>>(n, k, src, dst);
}

void launch_multi_edge_solution(const MultiProblem &m, int k, int64_t ne, const int64_t *edge_src, double2 *x,
                                cudaStream_t stream) {
  if (ne <= 0) return;
  multi_edge_solution_kernel<<<grid_for(ne, 256), 256, 0, stream>>>(ne, k, edge_src, m.Y, m.V, x);
}

}  // namespace fw
