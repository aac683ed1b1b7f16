// Triangular solves with the dense trailing block, every vector of the batch, in one launch.
//
// L then U of the block (or U^T then L^T) in row blocks of 64, as a dataflow among the CTAs of one
// cooperative launch: the CTAs of a unit (an instance and up to NV of its right-hand sides) own
// its row blocks in turn; a CTA subtracts the products with the blocks solved before from its own,
// tile by tile as they become known, solves its 64 x 64 triangle and publishes the 64 values.  The
// tiles do not depend on the solution, so they are fetched ahead of it, and the chain through the
// block is, per 64 rows, one hand-over between CTAs, one tile product and one triangle.
//
// The solved values themselves are the signal: they go to a buffer that launch_solve_permute_in
// has filled with kUnsolved, a NaN of a payload that no arithmetic produces, and a reader polls
// the value it needs.  One 8-byte relaxed load that is not kUnsolved is the value, so a hand-over
// needs neither a fence nor a flag behind the data.
//
// Bound by latency with few vectors (a hand-over and 64 dependent pivots per 64 rows), by HBM with
// many.  Measured, L and U of n = 20,000's block (69 blocks of rows, 156 MB read): 0.38 ms for one
// vector and 0.50 ms for 32, where a triangle launch and a push launch per block took 1.65 and
// 2.36 ms; 256 x n = 2,000 0.13 ms, one CTA per vector with barriers between the steps 0.26 ms.
// U is divided row by row by its diagonal while the CTA waits (one more rounding of each entry, a
// division less on the chain of pivots: 0.94 -> 0.38 ms together with the polled values, against
// progress counters that needed a fence and a second look).  Where that rounding has no bound or
// something overflows, the rows are solved undivided (solve_block; the look costs 5 us of 480 of a
// solve at n = 20,000).
//
// It replaces the reference's dense part of Symbolic_Matrix::solve (src/symbolic.cc:221-236).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <map>
#include <mutex>
#include <utility>

#include "glu_b200.h"
#include "kernels.cuh"
#include "quotient.cuh"
#include "wait.cuh"

namespace glu {

namespace {

constexpr int kWarp = 32;
constexpr int kB = 64;               // rows of a block
constexpr int kDs = 66;              // column stride of a staged triangle: rows by lane, 2-way at most

template <int NV>
constexpr int flow_smem() {
  return (kB * kDs + 2 * kB * NV + 4 * NV * kB + kB) * 8;
}

// The 64 x 64 triangle at T (T[i + kDs * j]) for one vector, rows lane and lane + 32 in r0 and r1.
// which: 0 = L (unit lower, forward), 1 = U (backward), 2 = U^T (forward), 3 = L^T (backward).
// Each solved value is broadcast and pushed into the remaining rows.  DIV: divide by the diagonal
// (which 1, 2) with its reciprocals rc; otherwise the rows were divided by it beforehand.
template <int WHICH, bool DIV>
__device__ __forceinline__ void triangle(const double* __restrict__ T,
                                         const double* __restrict__ rc, int lane, double& r0,
                                         double& r1) {
  constexpr bool fwd = WHICH == 0 || WHICH == 2;
  constexpr int si = WHICH < 2 ? 1 : kDs, sj = WHICH < 2 ? kDs : 1;   // M(i, j) = T[i si + j sj]
  const double* __restrict__ c0 = T + lane * si;
  const double* __restrict__ c1 = T + (lane + 32) * si;
#pragma unroll
  for (int h = 0; h < 2; ++h) {               // the half of the rows that pivots lie in
    const bool lo = fwd ? h == 0 : h == 1;
#pragma unroll 8
    for (int q = 0; q < 32; ++q) {
      const int p = fwd ? q : 31 - q;         // lane of the pivot
      const int j = lo ? p : p + 32;
      double x = lo ? r0 : r1;
      if (DIV) x = quotient(x, T[j * (kDs + 1)], rc[j]);
      const double xj = __shfl_sync(0xffffffffu, x, p);
      if (DIV && lane == p) (lo ? r0 : r1) = xj;
      const bool rest = fwd ? lane > p : lane < p;
      if (lo) {
        if (rest) r0 -= c0[j * sj] * xj;
        if (fwd) r1 -= c1[j * sj] * xj;
      } else {
        if (rest) r1 -= c1[j * sj] * xj;
        if (!fwd) r0 -= c0[j * sj] * xj;
      }
    }
  }
}

// A diagonal block where it lies: entry (i, j), i, j < m, at A[i + j ld], or, if lp is not null (a front,
// lp from its first column on, and the block at its row and column b), at A[lp[b + j] - j + i].
struct DiagBlock {
  const double* A;
  int64_t ld;
  const uint32_t* lp;
  int b, m;
  __device__ __forceinline__ double operator()(int i, int j) const {
    if (i >= m || j >= m) return i == j ? 1.0 : 0.0;
    return lp ? A[(int64_t)lp[b + j] - j + i] : A[i + j * ld];
  }
};

// The same solve for which 1 and 2 from where the block lies, with a division per pivot, for the
// vectors that the divided rows do not serve (see solve_block).
template <int WHICH>
__device__ __forceinline__ double2 triangle_divide(DiagBlock M, double r0, double r1) {
  static_assert(WHICH == 1 || WHICH == 2, "");
  const int lane = threadIdx.x % kWarp;
#pragma unroll 1
  for (int q = 0; q < kB; ++q) {
    const int j = WHICH == 2 ? q : kB - 1 - q;
    const double m0 = WHICH == 2 ? M(j, lane) : M(lane, j);
    const double m1 = WHICH == 2 ? M(j, lane + 32) : M(lane + 32, j);
    const double xj = __shfl_sync(0xffffffffu, j < 32 ? r0 : r1, j % 32) / M(j, j);
    if (j == lane) r0 = xj;
    else if (WHICH == 2 ? lane > j : lane < j) r0 -= m0 * xj;
    if (j == lane + 32) r1 = xj;
    else if (WHICH == 2 ? lane + 32 > j : lane + 32 < j) r1 -= m1 * xj;
  }
  return make_double2(r0, r1);
}

// Rows of the staged triangle divided by their diagonal (U: row i; U^T: column i of U), its
// reciprocals in rc: the division leaves the chain of pivots for one more rounding of each entry.
// Where a quotient by more than 2^64 drops below the normal range, and with it the rounding's bound,
// the first row to be solved is made NaN, which solve_block takes up.  (By less, the entry was
// below 2^-958, as some fill of large blocks is, and is off by 2^-1011 at most.)
template <bool TRANS>
__device__ __forceinline__ void divide_rows(double* Ds, double* rc) {
  bool low = false;
  for (int e = threadIdx.x; e < kB * kB; e += 256) {
    const int i = e % kB, j = e / kB, d = TRANS ? j : i;
    if (i < j) {
      const double v = Ds[i + j * kDs], dd = Ds[d * (kDs + 1)], q = quotient(v, dd, rc[d]);
      Ds[i + j * kDs] = q;
      low |= (__double2hiint(q) & 0x7ff00000) == 0 && v != 0.0 && fabs(dd) > 0x1p64;
    }
  }
  if (low) rc[TRANS ? 0 : kB - 1] = __longlong_as_double(kNaN);
}

// Rows not finite, a bit each.
__device__ __forceinline__ unsigned long long bad_rows(double r0, double r1) {
  return __ballot_sync(0xffffffffu, !finite_bits(r0)) |
         (unsigned long long)__ballot_sync(0xffffffffu, !finite_bits(r1)) << 32;
}

// One vector's rows of the block, staged at Ds (diagonal's reciprocals rc), divided by the diagonal
// if its exponents are ordinary (`plain`).  That serves unless something is not finite on the way
// that would be with a division at the end: a quotient overflows where the undivided sum does not
// (U(i, j) / d or y / d with d of 2^-900), a reciprocal is infinite.  It shows as the first value
// that is not finite lying before the first such row of the right-hand side; the rows are then
// solved again from where they lie.
template <int WHICH>
__device__ __forceinline__ void solve_block(const double* Ds, const double* rc, int lane,
                                            bool plain, const DiagBlock& M, double& y0,
                                            double& y1) {
  if (WHICH == 0 || WHICH == 3) {
    triangle<WHICH, false>(Ds, rc, lane, y0, y1);
    return;
  }
  const double w0 = y0, w1 = y1;
  if (plain) {
    y0 = quotient(y0, Ds[lane * (kDs + 1)], rc[lane]);
    y1 = quotient(y1, Ds[(lane + 32) * (kDs + 1)], rc[lane + 32]);
    triangle<WHICH, false>(Ds, rc, lane, y0, y1);
    if (!__any_sync(0xffffffffu, !finite_bits(y0) || !finite_bits(y1))) return;
  } else {
    triangle<WHICH, true>(Ds, rc, lane, y0, y1);
  }
  if (__any_sync(0xffffffffu, !finite_bits(y0) || !finite_bits(y1))) {
    const unsigned long long in = bad_rows(w0, w1), out = bad_rows(y0, y1);
    if (WHICH == 2 ? (unsigned)__ffsll(out) - 1u < (unsigned)__ffsll(in) - 1u
                   : __clzll(out) < __clzll(in)) {
      const double2 x = triangle_divide<WHICH == 2 ? 2 : 1>(M, w0, w1);
      y0 = x.x;
      y1 = x.y;
    }
  }
}

__device__ __forceinline__ double ld_relaxed(const double* p) {
  double v;
  asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed(double* p, double v) {
  asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}
__device__ __forceinline__ bool unsolved(double v) {
  return __double_as_longlong(v) == kUnsolved;
}

// The value at p, the first look at which gave v, once it is solved.  Bounded: after `budget_ns`
// (recorded in *err), or once another CTA has recorded a failure there, *fail is set.
__device__ __forceinline__ double wait_value(const double* p, double v, int* err,
                                             unsigned long long budget_ns, int* fail) {
  if (!unsolved(v)) return v;
  const unsigned long long t0 = global_ns();
  for (int spin = 1; unsolved(v = ld_relaxed(p)); ++spin) {
    if (spin % 64) continue;
    if (*(volatile int*)err) {
      *fail = 1;
      break;
    }
    if (global_ns() - t0 > budget_ns) {
      atomicExch(err, 1);
      *fail = 1;
      break;
    }
  }
  return v;
}

// The end of a CTA whose wait gave up: its own copies have landed before it returns.
__device__ __forceinline__ bool gave_up() {
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  return false;
}

// One phase (WHICH as in triangle) of a unit (an instance's nv vectors) for CTA r of G.  rhs: the
// block's right-hand side, to be waited for if `wait_rhs`; xb: the solved values (vectors xl
// apart), also written to yd (vectors yl apart) if not null.  Returns false if a wait gave up.
template <int NV, int WHICH>
__device__ bool flow_phase(const double* __restrict__ D, int64_t ld, int nblk, const double* rhs,
                           int64_t rl, bool wait_rhs, double* xb, int64_t xl, double* yd,
                           int64_t yl, int nv, int r, int G, int* err,
                           unsigned long long budget_ns, double* sm) {
  constexpr bool fwd = WHICH == 0 || WHICH == 2;
  constexpr bool trans = WHICH >= 2;
  constexpr bool diag = WHICH == 1 || WHICH == 2;
  constexpr int NX = (kB * NV + 255) / 256;   // values of a solved block per thread
  double* Ds = sm;
  double* xs = Ds + kB * kDs;                 // [2][kB][NV]
  double* red = xs + 2 * kB * NV;             // [4][NV][kB]
  double* rc = red + 4 * NV * kB;
  const int tid = threadIdx.x, lane = tid % kWarp, warp = tid / kWarp;
  const int vec = warp % NV;                  // the vector whose triangle this warp solves
  for (int o = r; o < nblk; o += G) {
    const int b = (fwd ? o : nblk - 1 - o) * kB;
    // the diagonal block, the first tile and the right-hand side are on their way meanwhile
    for (int e = tid; e < kB * kB / 2; e += 256) {
      const int i = (e % 32) * 2, j = e / 32;
      const unsigned dst = (unsigned)__cvta_generic_to_shared(Ds + i + j * kDs);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst),
                   "l"(D + b + i + (int64_t)(b + j) * ld));
    }
    asm volatile("cp.async.commit_group;\n" ::);
    // a thread's 16 entries of the tile against block k: !trans, row tid % 64 of 16 columns;
    // trans, two rows (of the solved block) of 8 columns
    double m[16], xn[NX];
    auto fetch = [&](int k, double (&t)[16]) {
      const int kb = (fwd ? k : nblk - 1 - k) * kB;
      if (!trans) {
        const double* __restrict__ p = D + b + (tid & 63) + (int64_t)(kb + (tid >> 6) * 16) * ld;
#pragma unroll
        for (int q = 0; q < 16; ++q, p += ld) t[q] = *p;
      } else {
        const double* __restrict__ p = D + kb + 2 * lane + (int64_t)(b + warp * 8) * ld;
#pragma unroll
        for (int q = 0; q < 8; ++q, p += ld) {
          const double2 v = *reinterpret_cast<const double2*>(p);
          t[2 * q] = v.x;
          t[2 * q + 1] = v.y;
        }
      }
    };
    // the address of value e (row e % 64 of vector e / 64) of solved block k; vectors past nv
    // repeat the last one
    auto xaddr = [&](int k, int e) {
      return xb + (int64_t)min(e / kB, nv - 1) * xl + (fwd ? k : nblk - 1 - k) * kB + e % kB;
    };
    if (o > 0) {
      fetch(0, m);
#pragma unroll
      for (int h = 0; h < NX; ++h)
        if (tid + h * 256 < kB * NV) xn[h] = ld_relaxed(xaddr(0, tid + h * 256));
    }
    const double* ry = rhs + (int64_t)min(vec, nv - 1) * rl + b + lane;
    double y0 = ld_relaxed(ry), y1 = ld_relaxed(ry + 32);
    double acc[trans ? 8 * NV : NV];
#pragma unroll
    for (int i = 0; i < (trans ? 8 * NV : NV); ++i) acc[i] = 0.0;
    int fail = 0;
    bool plain = true;                        // the diagonal's exponents are ordinary
    auto finish_stage = [&]() {
      asm volatile("cp.async.wait_group 0;\n" ::);
      __syncthreads();
      if (diag) {
        bool odd = false;
        if (tid < kB) {
          const double d = Ds[tid * (kDs + 1)];
          rc[tid] = 1.0 / d;
          const int ex = (__double2hiint(d) >> 20) & 0x7ff;
          odd = ex < 64 || ex > 0x7ff - 64;
        }
        plain = !__syncthreads_or(odd);
        if (plain) divide_rows<trans>(Ds, rc);
      }
    };
    for (int k = 0; k < o; ++k) {
      if (k == o - 1) finish_stage();         // before waiting for the last block
      double* x = xs + (k & 1) * kB * NV;
#pragma unroll
      for (int h = 0; h < NX; ++h) {
        const int e = tid + h * 256;
        if (e < kB * NV)
          x[(e % kB) * NV + e / kB] = wait_value(xaddr(k, e), xn[h], err, budget_ns, &fail);
      }
      if (__syncthreads_or(fail)) return gave_up();
      if (k + 1 < o) {
#pragma unroll
        for (int h = 0; h < NX; ++h)
          if (tid + h * 256 < kB * NV) xn[h] = ld_relaxed(xaddr(k + 1, tid + h * 256));
      }
      if (!trans) {
#pragma unroll
        for (int q = 0; q < 16; ++q)
#pragma unroll
          for (int v = 0; v < NV; ++v) acc[v] += m[q] * x[((tid >> 6) * 16 + q) * NV + v];
      } else {
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          const double x0 = x[2 * lane * NV + v], x1 = x[(2 * lane + 1) * NV + v];
#pragma unroll
          for (int q = 0; q < 8; ++q) acc[q * NV + v] += m[2 * q] * x0 + m[2 * q + 1] * x1;
        }
      }
      if (k + 1 < o) fetch(k + 1, m);         // on its way while block k + 1 is waited for
    }
    if (o == 0) finish_stage();
    if (!trans) {
#pragma unroll
      for (int v = 0; v < NV; ++v) red[((tid >> 6) * NV + v) * kB + (tid & 63)] = acc[v];
    } else {
#pragma unroll
      for (int i = 0; i < 8 * NV; ++i) {
        double t = acc[i];
        for (int d = 16; d > 0; d >>= 1) t += __shfl_xor_sync(0xffffffffu, t, d);
        if (lane == 0) red[(i % NV) * kB + warp * 8 + i / NV] = t;
      }
    }
    if (wait_rhs) {
      y0 = wait_value(ry, y0, err, budget_ns, &fail);
      y1 = wait_value(ry + 32, y1, err, budget_ns, &fail);
    }
    if (__syncthreads_or(fail)) return gave_up();  // sums, triangle and reciprocals are there too
    double s0 = 0.0, s1 = 0.0;
#pragma unroll
    for (int q = 0; q < (trans ? 1 : 4); ++q) {
      s0 += red[(q * NV + vec) * kB + lane];
      s1 += red[(q * NV + vec) * kB + lane + 32];
    }
    y0 -= s0;
    y1 -= s1;
    // every warp solves (NV < 8: some the same vector), so that no branch holds the shuffles
    solve_block<WHICH>(Ds, rc, lane, plain, DiagBlock{D + b + b * ld, ld, nullptr, 0, kB}, y0, y1);
    if (warp < nv) {
      double* xo = xb + vec * xl + b + lane;
      st_relaxed(xo, unsolved(y0) ? __longlong_as_double(kNaN) : y0);
      st_relaxed(xo + 32, unsolved(y1) ? __longlong_as_double(kNaN) : y1);
      if (yd) {
        yd[vec * yl + b + lane] = y0;
        yd[vec * yl + b + lane + 32] = y1;
      }
    }
    __syncthreads();                          // smem reuse by the next block
  }
  return true;
}

// Grid: groups of G CTAs; group g takes units g, g + groups, ...  xbuf: solve_buffer values a
// vector, the dense block's first.
template <int NV, bool TRANS>
__global__ void __launch_bounds__(256, NV * (TRANS ? 2 : 1) >= 8 ? 1 : 2)
    k_dense_flow(PlanDev P, const double* vals, int count, int nrhs, double* y, int64_t ylen,
                 int G, double* xbuf, int* err, int32_t* status, unsigned long long budget_ns) {
  extern __shared__ double sm[];
  const int chunks = (nrhs + NV - 1) / NV;
  const int units = count * chunks, groups = gridDim.x / G;
  const int r = blockIdx.x % G, nblk = (int)(P.ntp / kB);
  const int64_t xl = solve_buffer(P);
  for (int u = blockIdx.x / G; u < units; u += groups) {
    const int inst = u / chunks, v0 = (u % chunks) * NV;
    const int nv = min(NV, nrhs - v0);
    const int64_t vec = (int64_t)inst * nrhs + v0;
    const double* D = vals + (int64_t)inst * P.blob + P.dbase;
    double* yd = y + vec * ylen + P.t;
    double* x1 = xbuf + vec * xl;
    double* x2 = x1 + P.ntp;
    const bool ok =
        flow_phase<NV, TRANS ? 2 : 0>(D, P.ntp, nblk, yd, ylen, false, x1, xl, nullptr, 0, nv, r, G,
                                      err, budget_ns, sm) &&
        flow_phase<NV, TRANS ? 3 : 1>(D, P.ntp, nblk, x1, xl, true, x2, xl, yd, ylen, nv, r, G, err,
                                      budget_ns, sm);
    if (!ok) {                                // a wait gave up: this unit and the rest are void
      if (threadIdx.x == 0)
        for (int w = u; w < units; w += groups) atomicOr(status + w / chunks, kSolveGaveUp);
      return;
    }
  }
}

// CTAs of a kernel that fit on the current device at once (cached per kernel and device).
int flow_capacity(const void* kern, size_t smem) {
  static std::mutex mu;
  static std::map<std::pair<const void*, int>, int> known;
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lock(mu);
  int& cap = known[{kern, dev}];
  if (cap == 0) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 256, smem) != cudaSuccess)
      cudaGetLastError();
    cap = std::max(1, per_sm) * sm_count();
  }
  return cap;
}

template <int NV, bool TRANS>
void flow_launch(const PlanDev& P, const double* vals, int count, int nrhs, double* y, int64_t ylen,
                 double* xbuf, int* err, int32_t* status, double budget_ms, cudaStream_t s,
                 LaunchCounter& lc) {
  const auto kern = k_dense_flow<NV, TRANS>;
  ensure_smem_limit((const void*)kern, flow_smem<NV>());
  const int cap = flow_capacity((const void*)kern, flow_smem<NV>()), nblk = (int)(P.ntp / kB);
  // the vectors' units share the CTAs that fit on the device: all of a block's rows in flight for
  // a few vectors, down to one CTA walking the blocks of each of many
  const int64_t units = (int64_t)count * ((nrhs + NV - 1) / NV);
  const int G = (int)std::max<int64_t>(1, std::min<int64_t>(nblk, cap / units));
  const int64_t groups = std::min<int64_t>(units, cap / G);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(groups * G));
  cfg.blockDim = dim3(256);
  cfg.dynamicSmemBytes = flow_smem<NV>();
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;      // every CTA resident at once
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kern, P, vals, count, nrhs, y, ylen, G, xbuf, err, status,
                     (unsigned long long)(budget_ms * 1e6));
  lc.n++;
}

// ---------------------------------------------------------------------------------------------
// fronts
// ---------------------------------------------------------------------------------------------

// Row block `o` (in the order of the phase) of front f for nv vectors: the body of flow_phase with
// the front's own columns, whose rows lie contiguously in the value slots (row i of column x at
// lp[s0 + x] - x + i), and bounds for a last block that is not full.
template <int NV, int WHICH>
__device__ bool front_block(const PlanDev& P, const double* __restrict__ V, int f, int o, double* y,
                            int64_t yl, double* xb, int64_t xl, int nv, int* err,
                            unsigned long long budget_ns, double* sm) {
  constexpr bool fwd = WHICH == 0 || WHICH == 2;
  constexpr bool trans = WHICH >= 2;
  constexpr bool diag = WHICH == 1 || WHICH == 2;
  constexpr int NX = (kB * NV + 255) / 256;
  double* Ds = sm;
  double* xs = Ds + kB * kDs;                 // [2][kB][NV]
  double* red = xs + 2 * kB * NV;             // [4][NV][kB]
  double* rc = red + 4 * NV * kB;
  const int tid = threadIdx.x, lane = tid % kWarp, warp = tid / kWarp;
  const int vec = warp % NV;
  const int s0 = P.fs0[f], w = P.fw[f], nblk = (w + kB - 1) / kB;
  const int b = (fwd ? o : nblk - 1 - o) * kB;
  const uint32_t* __restrict__ lp = P.lp + s0;
  auto at = [&](int i, int x) { return V + ((int64_t)lp[x] - x + i); };
  for (int e = tid; e < kB * kB; e += 256) {
    const int i = b + e % kB, j = b + e / kB;
    const bool ok = i < w && j < w;
    const unsigned dst = (unsigned)__cvta_generic_to_shared(Ds + e % kB + (e / kB) * kDs);
    const double* src = ok ? at(i, j) : V;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(dst), "l"(src),
                 "r"(ok ? 8 : 0));
  }
  asm volatile("cp.async.commit_group;\n" ::);
  double m[16], xn[NX];
  auto fetch = [&](int k) {
    const int kb = (fwd ? k : nblk - 1 - k) * kB;
    if (!trans) {
      const int i = b + (tid & 63);
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        const int x = kb + (tid >> 6) * 16 + q;
        m[q] = i < w && x < w ? *at(i, x) : 0.0;
      }
    } else {
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int x = b + warp * 8 + q;
        m[2 * q] = x < w && kb + lane < w ? *at(kb + lane, x) : 0.0;
        m[2 * q + 1] = x < w && kb + lane + 32 < w ? *at(kb + lane + 32, x) : 0.0;
      }
    }
  };
  // the place of value e of solved block k in the front's values, -1 past them
  auto place = [&](int k, int e) {
    const int i = (fwd ? k : nblk - 1 - k) * kB + e % kB;
    return i < w ? i : -1;
  };
  auto look = [&](int k) {
#pragma unroll
    for (int h = 0; h < NX; ++h) {
      const int e = tid + h * 256, i = e < kB * NV ? place(k, e) : -1;
      xn[h] = i >= 0 ? ld_relaxed(xb + (int64_t)min(e / kB, nv - 1) * xl + i) : 0.0;
    }
  };
  if (o > 0) {
    fetch(0);
    look(0);
  }
  double* yv = y + (int64_t)min(vec, nv - 1) * yl + s0;
  double y0 = b + lane < w ? yv[b + lane] : 0.0;
  double y1 = b + lane + 32 < w ? yv[b + lane + 32] : 0.0;
  double acc[trans ? 8 * NV : NV];
#pragma unroll
  for (int i = 0; i < (trans ? 8 * NV : NV); ++i) acc[i] = 0.0;
  int fail = 0;
  bool plain = true;
  auto finish_stage = [&]() {
    asm volatile("cp.async.wait_group 0;\n" ::);
    __syncthreads();
    bool odd = false;
    if (tid < kB) {
      if (b + tid >= w) Ds[tid * (kDs + 1)] = 1.0;   // padding: identity
      const double d = Ds[tid * (kDs + 1)];
      if (diag) rc[tid] = 1.0 / d;
      const int ex = (__double2hiint(d) >> 20) & 0x7ff;
      odd = ex < 64 || ex > 0x7ff - 64;
    }
    if (diag) {
      plain = !__syncthreads_or(odd);
      if (plain) divide_rows<trans>(Ds, rc);
    }
  };
  for (int k = 0; k < o; ++k) {
    if (k == o - 1) finish_stage();
    double* x = xs + (k & 1) * kB * NV;
#pragma unroll
    for (int h = 0; h < NX; ++h) {
      const int e = tid + h * 256;
      if (e < kB * NV) {
        const int i = place(k, e);
        x[(e % kB) * NV + e / kB] =
            i < 0 ? 0.0
                  : wait_value(xb + (int64_t)min(e / kB, nv - 1) * xl + i, xn[h], err, budget_ns,
                               &fail);
      }
    }
    if (__syncthreads_or(fail)) return gave_up();
    if (k + 1 < o) look(k + 1);
    if (!trans) {
#pragma unroll
      for (int q = 0; q < 16; ++q)
#pragma unroll
        for (int v = 0; v < NV; ++v) acc[v] += m[q] * x[((tid >> 6) * 16 + q) * NV + v];
    } else {
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        const double x0 = x[lane * NV + v], x1 = x[(lane + 32) * NV + v];
#pragma unroll
        for (int q = 0; q < 8; ++q) acc[q * NV + v] += m[2 * q] * x0 + m[2 * q + 1] * x1;
      }
    }
    if (k + 1 < o) fetch(k + 1);
  }
  if (o == 0) finish_stage();
  if (!trans) {
#pragma unroll
    for (int v = 0; v < NV; ++v) red[((tid >> 6) * NV + v) * kB + (tid & 63)] = acc[v];
  } else {
#pragma unroll
    for (int i = 0; i < 8 * NV; ++i) {
      double t = acc[i];
      for (int d = 16; d > 0; d >>= 1) t += __shfl_xor_sync(0xffffffffu, t, d);
      if (lane == 0) red[(i % NV) * kB + warp * 8 + i / NV] = t;
    }
  }
  __syncthreads();
  double t0 = 0.0, t1 = 0.0;
#pragma unroll
  for (int q = 0; q < (trans ? 1 : 4); ++q) {
    t0 += red[(q * NV + vec) * kB + lane];
    t1 += red[(q * NV + vec) * kB + lane + 32];
  }
  y0 -= t0;
  y1 -= t1;
  solve_block<WHICH>(Ds, rc, lane, plain, DiagBlock{V, 0, lp, b, min(kB, w - b)}, y0, y1);
  if (warp < nv) {
    double* xo = xb + vec * xl + b;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int i = lane + 32 * h;
      const double v = h ? y1 : y0;
      if (b + i < w) {
        if (o + 1 < nblk) st_relaxed(xo + i, unsolved(v) ? __longlong_as_double(kNaN) : v);
        yv[b + i] = v;
      }
    }
  }
  __syncthreads();                            // smem reuse by the next block
  return true;
}

// The rows of a level's fronts among themselves: items {front, order of the row block}, every
// front's earlier blocks before its later ones, each for every unit (an instance and up to NV of
// its right-hand sides).  A CTA takes items in increasing order, and an item waits only for lower
// ones, so with every CTA resident (a cooperative launch wherever a front has two blocks) the
// lowest unfinished item can always go on.
// Bound by latency as the dense block's solve.  Measured, 512 x 512 x 2 nodes, 4 vectors: 11 us per L
// level and 17 us per U level (wider fronts), where one CTA per front took 30 us a level and a
// cluster of eight 116 us for the wide ones.
template <int NV, int WHICH>
__global__ void __launch_bounds__(256, NV * (WHICH >= 2 ? 2 : 1) >= 8 ? 1 : 2)
    k_front_flow(PlanDev P, const double* vals, int count, int nrhs, double* y, int64_t ylen,
                 const int2* __restrict__ items, int nitems, double* xbuf, int* err,
                 int32_t* status, unsigned long long budget_ns) {
  extern __shared__ double sm[];
  const int chunks = (nrhs + NV - 1) / NV;
  const int64_t units = (int64_t)count * chunks;
  const int64_t xl = solve_buffer(P);
  double* xf = xbuf + 2 * (int64_t)P.ntp + (WHICH == 1 || WHICH == 3 ? P.fx_len : 0);
  after_previous();
  for (int64_t it = blockIdx.x; it < nitems * units; it += gridDim.x) {
    const int2 item = items[it / units];
    const int u = (int)(it % units), inst = u / chunks, v0 = (u % chunks) * NV;
    const int64_t vec = (int64_t)inst * nrhs + v0;
    if (!front_block<NV, WHICH>(P, vals + (int64_t)inst * P.blob, item.x, item.y, y + vec * ylen,
                                ylen, xf + vec * xl + P.fx0[item.x], xl, min(NV, nrhs - v0), err,
                                budget_ns, sm)) {
      // a wait gave up: this item and the CTA's later ones are void, and the last block of a front
      // has nobody waiting for it who would notice
      if (threadIdx.x == 0)
        for (; it < nitems * units; it += gridDim.x)
          atomicOr(status + (int)(it % units) / chunks, kSolveGaveUp);
      return;
    }
  }
}

template <int NV, int WHICH>
void front_launch(const PlanDev& P, const double* vals, int count, int nrhs, double* y,
                  int64_t ylen, const FrontLevelSolve& L, double* xbuf, int* err, int32_t* status,
                  double budget_ms, cudaStream_t s, LaunchCounter& lc) {
  const auto kern = k_front_flow<NV, WHICH>;
  ensure_smem_limit((const void*)kern, flow_smem<NV>());
  const int64_t total = (int64_t)L.nflow * count * ((nrhs + NV - 1) / NV);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  cfg.gridDim = dim3((unsigned)total);
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // as launch_next
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (L.nflow > L.nfronts) {                  // some front has blocks that wait
    const int cap = flow_capacity((const void*)kern, flow_smem<NV>());
    cfg.gridDim = dim3((unsigned)std::min<int64_t>(total, std::max(cap, 1)));
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
  }
  cfg.blockDim = dim3(256);
  cfg.dynamicSmemBytes = flow_smem<NV>();
  cfg.stream = s;
  cudaLaunchKernelEx(&cfg, kern, P, vals, count, nrhs, y, ylen,
                     reinterpret_cast<const int2*>(L.flow), L.nflow, xbuf, err, status,
                     (unsigned long long)(budget_ms * 1e6));
  lc.n++;
}

// ---------------------------------------------------------------------------------------------
// sparse columns
// ---------------------------------------------------------------------------------------------

// A phase of the sparse columns' solves (WHICH 0: L by rows, with the rows of L21; 1: U by rows, the
// entries left of t; 2: U^T, 3: L^T by columns, the entries above t) for plans without fronts: a
// warp per row and unit (an instance and up to NV of its right-hand sides) polls the values its
// entries need, sums and publishes its own.  Rows come in the order of the levels, a warp takes
// them in increasing order and every CTA is resident, so the first unfinished row can always go on.
// The sums have a fixed order.
// A launch per level costs some 3 us a level; here the chain is a hand-over per level.
// Measured: adjoint solve at n = 20,000 (30 + 29 levels) 0.72 -> 0.56 ms, 4 x n = 4,960 deterministic
// pass (16 + 17 levels, two solves) 1.37 -> 1.20 ms, n = 2,000 pass (14 + 14 levels) 405 -> 385 us.
template <int NV, int WHICH>
__global__ void __launch_bounds__(256) k_sparse_flow(PlanDev P, const double* vals, int count,
                                                     int nrhs, double* y, int64_t ylen,
                                                     const int32_t* __restrict__ items, int G,
                                                     double* xbuf, int* err, int32_t* status,
                                                     unsigned long long budget_ns) {
  const int chunks = (nrhs + NV - 1) / NV;
  const int units = count * chunks, groups = gridDim.x / G;
  const int lane = threadIdx.x % kWarp;
  const int wi = (int)(blockIdx.x % G) * 8 + (int)(threadIdx.x / kWarp), W = G * 8;
  const int t = (int)P.t, total = WHICH == 0 ? (int)P.n : t;
  const int64_t xl = solve_buffer(P);
  for (int u = blockIdx.x / G; u < units; u += groups) {
    const int inst = u / chunks, v0 = (u % chunks) * NV;
    const int nv = min(NV, nrhs - v0);
    const int64_t vec = (int64_t)inst * nrhs + v0;
    const double* __restrict__ V = vals + (int64_t)inst * P.blob;
    double* y0 = y + vec * ylen;
    double* xb = xbuf + vec * xl + 2 * (int64_t)P.ntp + (WHICH == 1 || WHICH == 3 ? P.fx_len : 0);
    for (int i = wi; i < total; i += W) {
      const int c = i < t ? items[WHICH < 2 ? i : t - 1 - i] : i;
      int64_t e0, e1;
      if (WHICH == 0) e0 = P.lr_ptr[c], e1 = P.lr_ptr[c + 1];
      if (WHICH == 1) e0 = P.ur_ptr[c], e1 = e0 + P.ur_split[c];
      if (WHICH == 2) e0 = P.cp[c], e1 = P.lp[c];
      if (WHICH == 3) e0 = (int64_t)P.lp[c] + 1, e1 = e0 + P.lsplit[c];
      const double d = WHICH == 1 || WHICH == 2 ? V[P.lp[c]] : 1.0;
      const double yc = lane < nv ? y0[lane * ylen + c] : 0.0;
      double sum[NV];
#pragma unroll
      for (int k = 0; k < NV; ++k) sum[k] = 0.0;
      int fail = 0;
      for (int64_t e = e0; e < e1; e += kWarp) {
        const bool mine = e + lane < e1;
        int32_t j = 0;
        double m = 0.0;
        if (mine) {
          j = WHICH == 0 ? P.lr_col[e + lane] : WHICH == 1 ? P.ur_col[e + lane]
                                                           : (int32_t)P.ri[e + lane];
          m = WHICH == 0 ? V[P.lr_slot[e + lane]] : WHICH == 1 ? V[P.ur_slot[e + lane]]
                                                               : V[e + lane];
        }
        double x[NV];
#pragma unroll
        for (int k = 0; k < NV; ++k) x[k] = mine && k < nv ? ld_relaxed(xb + k * xl + j) : 0.0;
#pragma unroll
        for (int k = 0; k < NV; ++k) {
          if (mine && k < nv) x[k] = wait_value(xb + k * xl + j, x[k], err, budget_ns, &fail);
          sum[k] += m * x[k];
        }
      }
      if (__any_sync(0xffffffffu, fail)) {    // a wait gave up: this unit and the rest are void
        if (lane == 0)
          for (int w = u; w < units; w += groups) atomicOr(status + w / chunks, kSolveGaveUp);
        return;
      }
      double s = 0.0;
#pragma unroll
      for (int k = 0; k < NV; ++k) {
        for (int o = 16; o > 0; o >>= 1) sum[k] += __shfl_xor_sync(0xffffffffu, sum[k], o);
        if (lane == k) s = sum[k];
      }
      if (lane < nv) {
        const double v = WHICH == 1 || WHICH == 2 ? (yc - s) / d : yc - s;
        if (i < t) st_relaxed(xb + lane * xl + c, unsolved(v) ? __longlong_as_double(kNaN) : v);
        y0[lane * ylen + c] = v;
      }
    }
  }
}

template <int NV, int WHICH>
void sparse_launch(const PlanDev& P, const double* vals, int count, int nrhs, double* y,
                   int64_t ylen, const int32_t* items, double* xbuf, int* err, int32_t* status,
                   double budget_ms, cudaStream_t s, LaunchCounter& lc) {
  const auto kern = k_sparse_flow<NV, WHICH>;
  const int64_t units = (int64_t)count * ((nrhs + NV - 1) / NV);
  const int cap = flow_capacity((const void*)kern, 0);
  const int rows = (int)(WHICH == 0 ? P.n : P.t);
  const int G = (int)std::max<int64_t>(1, std::min<int64_t>((rows + 7) / 8, cap / units));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(std::min<int64_t>(units, cap / G) * G));
  cfg.blockDim = dim3(256);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;      // every CTA resident at once
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kern, P, vals, count, nrhs, y, ylen, items, G, xbuf, err, status,
                     (unsigned long long)(budget_ms * 1e6));
  lc.n++;
}

}  // namespace

void launch_dense_solve(const PlanDev& P, const double* vals, int count, int nrhs, double* y,
                        int64_t ylen, bool transpose, double* xbuf, int* err, int32_t* status,
                        double budget_ms, cudaStream_t s, LaunchCounter& lc) {
  if (P.ntp == 0) return;
#define GLU_FLOW(NV, T)                                                                        \
  flow_launch<NV, T>(P, vals, count, nrhs, y, ylen, xbuf, err, status, budget_ms, s, lc)
  if (!transpose) {
    if (nrhs == 1) GLU_FLOW(1, false);
    else if (nrhs == 2) GLU_FLOW(2, false);
    else if (nrhs <= 4) GLU_FLOW(4, false);
    else GLU_FLOW(8, false);
  } else {
    if (nrhs == 1) GLU_FLOW(1, true);
    else if (nrhs == 2) GLU_FLOW(2, true);
    else GLU_FLOW(4, true);
  }
#undef GLU_FLOW
}

void launch_front_flow(const PlanDev& P, const double* vals, int count, int nrhs, double* y,
                       int64_t ylen, const FrontLevelSolve& L, int which, double* xbuf, int* err,
                       int32_t* status, double budget_ms, cudaStream_t s, LaunchCounter& lc) {
  if (L.nflow == 0) return;
#define GLU_FRONT(NV, W) \
  front_launch<NV, W>(P, vals, count, nrhs, y, ylen, L, xbuf, err, status, budget_ms, s, lc)
#define GLU_FRONT_NV(W)                      \
  if (nrhs == 1) GLU_FRONT(1, W);            \
  else if (nrhs == 2) GLU_FRONT(2, W);       \
  else GLU_FRONT(4, W);
  switch (which) {
    case 0: GLU_FRONT_NV(0) break;
    case 1: GLU_FRONT_NV(1) break;
    case 2: GLU_FRONT_NV(2) break;
    default: GLU_FRONT_NV(3) break;
  }
#undef GLU_FRONT_NV
#undef GLU_FRONT
}

// Few rows in all: with many, every warp walks hundreds of rows, each a hand-over long, and the
// launches per level, whose many warps hide their loads, win.  Measured, dataflow against levels,
// whole passes (rows, groups of right-hand sides counted): n = 2,000 385 / 405 us (1,562),
// 64 x n = 2,000 0.993 / 1.003 ms (99,968), 8 groups at n = 20,000 0.798 / 0.884 ms (124,928),
// 10 groups transposed 1.055 / 1.276 ms (156,160), 256 x n = 2,000 3.01 / 2.92 ms (399,872).
int64_t sparse_flow_vectors(const PlanDev& P, int count) {
  return P.t > 0 ? 200000 / ((int64_t)count * P.t) * 4 * count : 0;
}
bool sparse_solve_flows(const PlanDev& P, int count, int nrhs) {
  return (int64_t)count * nrhs <= sparse_flow_vectors(P, count);
}

void launch_sparse_flow(const PlanDev& P, const double* vals, int count, int nrhs, double* y,
                        int64_t ylen, const int32_t* items, int which, double* xbuf, int* err,
                        int32_t* status, double budget_ms, cudaStream_t s, LaunchCounter& lc) {
#define GLU_SPARSE(NV, W) \
  sparse_launch<NV, W>(P, vals, count, nrhs, y, ylen, items, xbuf, err, status, budget_ms, s, lc)
#define GLU_SPARSE_NV(W)                   \
  if (nrhs == 1) GLU_SPARSE(1, W);         \
  else GLU_SPARSE(4, W);
  switch (which) {
    case 0: GLU_SPARSE_NV(0) break;
    case 1: GLU_SPARSE_NV(1) break;
    case 2: GLU_SPARSE_NV(2) break;
    default: GLU_SPARSE_NV(3) break;
  }
#undef GLU_SPARSE_NV
#undef GLU_SPARSE
}

}  // namespace glu
