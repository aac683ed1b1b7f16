// Device body of the residual check r = b - op(A) x on the user's ORIGINAL matrix, shared by
// the kernel behind glu_residual / glu_refine (kernels.cu) and the one behind
// glu_residual_noalloc (noalloc.cu), so both entry points run the same arithmetic.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "plan.h"

namespace glu {

// Rows chunk * blockDim.x + threadIdx.x (blockDim.x a multiple of 32), stepping by
// nchunks * blockDim.x, of vector v
// (= instance * nrhs + rhs): r = b - op(A) x is written to R (if not null), and the infinity
// norms ||r||, ||x||, ||b||, ||A|| of the vector are folded into norms[4 v .. 4 v + 4) with
// atomicMax on their bit patterns (non-negative doubles order like their bits).  A NaN residual
// counts as infinite.  The whole warp must call this (it reduces with shuffles).
__device__ __forceinline__ void residual_rows(const PlanDev& P, int nrhs,
                                              const double* a,
                                              const double* X,
                                              const double* Bm,
                                              double* R, unsigned long long* norms,
                                              int transpose, int64_t v, int64_t chunk,
                                              int64_t nchunks) {
  const int64_t inst = v / nrhs;
  const double* av = a + inst * P.nnz_g;
  const double* xv = X + v * P.n;
  const double* bv = Bm + v * P.n;
  const int64_t* ptr = transpose ? P.o_col_ptr : P.o_row_ptr;
  const int64_t* ent = transpose ? P.o_col_e : P.o_row_e;
  const uint32_t* other = transpose ? P.g_row : P.g_col;
  double mr = 0.0, mx = 0.0, mb = 0.0, ma = 0.0;
  // A row per lane; rows of more than kLongRow entries (a grid's rail nodes have thousands) are summed
  // by the whole warp, four loads a lane in flight: on 512 x 512 x 2 nodes one thread walking 2,600
  // entries set the kernel's time, 1.10 ms of a pass.
  constexpr int kLongRow = 64;
  const int lane = threadIdx.x % 32;
  for (int64_t i0 = chunk * blockDim.x + (threadIdx.x - lane); i0 < P.n;
       i0 += nchunks * blockDim.x) {
    const int64_t i = i0 + lane;
    const int64_t q0 = i < P.n ? ptr[i] : 0, q1 = i < P.n ? ptr[i + 1] : 0;
    double s = 0.0, arow = 0.0;
    const bool is_long = q1 - q0 > kLongRow;
    if (!is_long)
      for (int64_t q = q0; q < q1; ++q) {
        const int64_t e = ent[q];
        s += av[e] * xv[other[e]];
        arow += fabs(av[e]);
      }
    for (unsigned m = __ballot_sync(0xffffffffu, is_long); m; m &= m - 1) {
      const int owner = __ffs(m) - 1;
      const int64_t f0 = __shfl_sync(0xffffffffu, q0, owner);
      const int64_t f1 = __shfl_sync(0xffffffffu, q1, owner);
      double t = 0.0, at = 0.0;
      for (int64_t q = f0 + lane; q < f1; q += 128) {
        double val[4], x[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int64_t e = q + 32 * u < f1 ? ent[q + 32 * u] : -1;
          val[u] = e >= 0 ? av[e] : 0.0;
          x[u] = e >= 0 ? xv[other[e]] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          t += val[u] * x[u];
          at += fabs(val[u]);
        }
      }
      for (int o = 16; o > 0; o >>= 1) {
        t += __shfl_xor_sync(0xffffffffu, t, o);
        at += __shfl_xor_sync(0xffffffffu, at, o);
      }
      if (lane == owner) {
        s = t;
        arow = at;
      }
    }
    if (i >= P.n) continue;
    const double r = bv[i] - s;
    if (R) R[v * P.n + i] = r;
    mr = fmax(mr, fabs(r));
    if (!(r == r)) mr = __longlong_as_double(0x7ff0000000000000LL);   // NaN -> inf
    mx = fmax(mx, fabs(xv[i]));
    mb = fmax(mb, fabs(bv[i]));
    ma = fmax(ma, arow);
  }
  for (int o = 16; o > 0; o >>= 1) {
    mr = fmax(mr, __shfl_xor_sync(0xffffffffu, mr, o));
    mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    mb = fmax(mb, __shfl_xor_sync(0xffffffffu, mb, o));
    ma = fmax(ma, __shfl_xor_sync(0xffffffffu, ma, o));
  }
  if ((threadIdx.x % 32) == 0) {
    unsigned long long* nv = norms + 4 * v;
    atomicMax(nv + 0, (unsigned long long)__double_as_longlong(mr));
    atomicMax(nv + 1, (unsigned long long)__double_as_longlong(mx));
    atomicMax(nv + 2, (unsigned long long)__double_as_longlong(mb));
    atomicMax(nv + 3, (unsigned long long)__double_as_longlong(ma));
  }
}

// ||r|| / (||A|| ||x|| + ||b||) from the four norms of one vector (||r|| when the denominator
// is zero).
__device__ __forceinline__ double residual_ratio(const unsigned long long* nv) {
  const double r = __longlong_as_double((long long)nv[0]);
  const double x = __longlong_as_double((long long)nv[1]);
  const double b = __longlong_as_double((long long)nv[2]);
  const double A = __longlong_as_double((long long)nv[3]);
  const double den = A * x + b;
  return den > 0.0 ? r / den : r;
}

}  // namespace glu
