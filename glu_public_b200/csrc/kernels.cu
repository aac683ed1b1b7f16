// Device kernels of the GLU numeric phase for sm_100a (FP64 throughout).
//
// Factorization = sparse phase + dense phase:
//  * sparse phase: one launch per level of the reference's level sets restricted to the
//    columns before the dense trailing block (src/symbolic.cc:106-151 builds those levels).  A
//    warp (narrow levels: a CTA) owns one column c: it divides L(:,c) by the pivot
//    (src/numeric.cu:37-47) and then, for every U(c,j) != 0, subtracts L(:,c)*U(c,j) from
//    column j (src/numeric.cu:51-89).  The target slots come from the precomputed position map
//    instead of the reference's scan of the whole of column j, so each update costs one load of
//    the map entry.  Columns of one level may hit the same target, so updates are FP64 atomics,
//    as in the reference.  Targets inside the dense block are left to dense.cu.
//  * dense phase (dense.cu): right-looking blocked LU without pivoting of the trailing block that
//    fill has made dense, with FP64 DMMA tensor-core trailing updates.
//
// Every kernel takes the instance index from blockIdx.y / blockIdx.z, so one launch covers a
// whole batch of value sets of the same pattern.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "glu_b200.h"
#include "kernels.cuh"
#include "residual.cuh"
#include "wait.cuh"

namespace glu {

namespace {

constexpr int kWarp = 32;

__device__ __forceinline__ void set_flag(int32_t* status, int b, int32_t f) {
  atomicOr(status + b, f);
}

__device__ __forceinline__ void pivot_flags(int32_t* status, int b, double d, bool perturbed) {
  if (d == 0.0) set_flag(status, b, GLU_INST_ZERO_PIVOT);
  else if (!(fabs(d) <= 1.79769313486231570e308)) set_flag(status, b, GLU_INST_NAN_PIVOT);
  if (perturbed) set_flag(status, b, GLU_INST_PERTURBED);
}

// ---------------------------------------------------------------------------------------------
// value handling
// ---------------------------------------------------------------------------------------------

__global__ void k_pad_identity(PlanDev P, double* vals, int first) {
  double* D = vals + (int64_t)(first + blockIdx.y) * P.blob + P.dbase;
  for (uint32_t i = P.nt + blockIdx.x * blockDim.x + threadIdx.x; i < P.ntp;
       i += gridDim.x * blockDim.x)
    D[(int64_t)i * P.ntp + i] = 1.0;
}

__global__ void k_zero_slots(PlanDev P, double* vals, int first) {
  after_previous();
  double* V = vals + (int64_t)(first + blockIdx.y) * P.blob;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < P.nasm_zero;
       e += (int64_t)gridDim.x * blockDim.x)
    V[P.asm_zero[e]] = 0.0;
}

__global__ void k_ingest(PlanDev P, double* vals, int first, const double* a) {
  after_previous();
  const int b = blockIdx.y;
  double* V = vals + (int64_t)(first + b) * P.blob;
  const double* ab = a + (int64_t)b * P.nnz_a;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < P.nnz_a;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t s = P.ing_slot[e];
    if (s >= 0) V[s] = P.ing_scale ? ab[e] * P.ing_scale[e] : ab[e];
  }
}

__global__ void k_load_lu(PlanDev P, double* vals, int first, const double* val) {
  after_previous();
  const int b = blockIdx.y;
  double* V = vals + (int64_t)(first + b) * P.blob;
  const double* vb = val + (int64_t)b * P.nnz;
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < P.nnz;
       p += (int64_t)gridDim.x * blockDim.x)
    V[P.pos2slot[p]] = vb[p];
}

__global__ void k_export_lu(PlanDev P, const double* vals, int inst, double* __restrict__ val) {
  after_previous();
  const double* V = vals + (int64_t)inst * P.blob;
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < P.nnz;
       p += (int64_t)gridDim.x * blockDim.x)
    val[p] = V[P.pos2slot[p]];
}

// 1-norm of every instance (max column abs sum over the filled pattern, src/numeric.cu:405-417),
// accumulated as the bit pattern of a non-negative double so atomicMax orders it correctly.
__global__ void k_norm1(PlanDev P, const double* vals, unsigned long long* norm_bits) {
  const int b = blockIdx.y;
  const double* V = vals + (int64_t)b * P.blob;
  const int lane = threadIdx.x % kWarp;
  const int warps = blockDim.x / kWarp;
  for (uint32_t j = blockIdx.x * warps + threadIdx.x / kWarp; j < P.n; j += gridDim.x * warps) {
    double s = 0.0;
    for (uint32_t p = P.cp[j] + lane; p < P.cp[j + 1]; p += kWarp) s += fabs(V[P.pos2slot[p]]);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) atomicMax(norm_bits + b, (unsigned long long)__double_as_longlong(s));
  }
}

__global__ void k_pert_finish(int count, const unsigned long long* norm_bits, double* pert) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b < count) pert[b] = 3.45e-4 * __longlong_as_double((long long)norm_bits[b]);
}

__global__ void k_fill(int count, double v, double* out) {
  after_previous();
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b < count) out[b] = v;
}

// ---------------------------------------------------------------------------------------------
// sparse phase: one level
// ---------------------------------------------------------------------------------------------

// The threads that share one column: `gsize` threads (whole warps) of which this is thread
// `gtid` in warp `wig` of `nwg`; `bar` says how they synchronise: 0 one warp (__syncwarp), -1 the
// whole CTA (__syncthreads), k > 0 the named barrier k (several warps of a larger CTA).
// `ilane` / `istride`: the lane and lane count that walk one pair's L rows (the whole warp, or the
// group's own lanes when a group is a fraction of a warp); `mask`: those lanes when bar == 0.
struct ColGroup {
  int gtid, gsize, wig, nwg, bar, ilane, istride;
  unsigned mask;
};

__device__ __forceinline__ void group_sync(const ColGroup& g) {
  if (g.bar == 0) __syncwarp(g.mask);
  else if (g.bar < 0) __syncthreads();
  else asm volatile("bar.sync %0, %1;" ::"r"(g.bar), "r"(g.gsize) : "memory");
}

__device__ __forceinline__ ColGroup warp_group() {
  const int lane = threadIdx.x % kWarp;
  return ColGroup{lane, kWarp, 0, 1, 0, lane, kWarp, 0xffffffffu};
}

__device__ __forceinline__ ColGroup cta_group() {
  return ColGroup{(int)threadIdx.x, (int)blockDim.x, (int)(threadIdx.x / kWarp),
                  (int)(blockDim.x / kWarp), -1, (int)(threadIdx.x % kWarp), kWarp, 0xffffffffu};
}

// The pairs (c, j) of one column applied by group w of W groups of `width` lanes (8, 16 or 32;
// `mask`) of which this is lane `il`: column j of each pair takes -L(:,c) * U(c,j) through the
// position map (src/numeric.cu:51-89); rows >= t of a tail column j belong to the dense block and
// are applied afterwards by the hub GEMM and the per-column pull, so a pair with j >= t has only
// nsplit updates and one with j < t has nL.
// What bounds this is the latency of dependent loads (pair, then U value and map entry, then the
// atomic) and, in the columns next to the dense block, a few pairs of thousands of updates among
// thousands of a dozen.  So fewer long pairs than groups are shared in pieces of 4 * width updates;
// of the others the lanes fetch the data `width` pairs at a time and the map entries of four pairs are in
// flight together, with one load of the L value for the four.
// Measured, sparse levels of one refactorization: n = 20,000 1.13 -> 0.39 ms (a few pairs of 2,860
// updates in columns of 2,850 pairs), 512 x 512 x 2 nodes 9.4 -> 6.8 ms, 64 x n = 20,000 5.6 -> 3.0 ms;
// sharing long pairs in pieces wherever there are fewer than groups, not a quarter as many: 128 x 128
// x 2 nodes 2.15 ms against 1.88.  A pair that a group has to itself goes four rows at a time, or the
// long columns of a plan without a dense block (up to a thousand pairs of a thousand updates, a pair
// a warp) have one load in flight: one n = 4,960 17.3 -> 10.3 ms, four of them 16.8 -> 10.4 (15.0 with
// a loop over the pairs alone), eight 16.4 -> 15.2, 128 x 128 x 2 nodes 4.09 -> 3.91 ms a pass;
// 64 x n = 2,000 without a dense block 8.5 -> 6.1 ms before that.
__device__ __forceinline__ void apply_pairs(const PlanDev& P, double* __restrict__ V, uint32_t c,
                                            const double* __restrict__ Lc, uint32_t nL, int64_t w,
                                            int64_t W, int il, int width, unsigned mask) {
  const uint32_t nsplit = P.lsplit[c];
  int64_t q0 = P.pair_ptr[c];
  const int64_t q1 = P.pair_ptr[c + 1];
  const int64_t na = P.usplit[c];              // pairs with j < t, the first ones
  if (4 * na < W && nL > 2 * (uint32_t)width) {  // they would leave most groups without one
    const uint32_t piece = 4 * width, np = (nL + piece - 1) / piece;
    for (int64_t e = w; e < na * np; e += W) {
      const int64_t q = q0 + e / np;
      const uint32_t k0 = (uint32_t)(e % np) * piece + il;
      const int32_t* __restrict__ tm = P.tmap + P.pair_moff[q];
      const double u = V[P.pair_uslot[q]];
      int32_t t[4];
      double l[4];
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const uint32_t k = k0 + h * width;
        t[h] = k < nL ? tm[k] : -1;
        l[h] = k < nL ? Lc[k] : 0.0;
      }
#pragma unroll
      for (int h = 0; h < 4; ++h)
        if (t[h] >= 0) atomicAdd(V + t[h], -(l[h] * u));
    }
    q0 += na;
  }
  for (int64_t q = q0 + w; q < q1; q += W * width) {
    const int64_t mine = q + W * il;
    uint32_t nsp = 0;
    int64_t mo = 0;
    double u = 0.0;
    if (mine < q1) {
      nsp = (uint32_t)P.pair_j[mine] < P.t ? nL : nsplit;
      mo = P.pair_moff[mine];
      u = V[P.pair_uslot[mine]];
    }
    const int n = (int)min((int64_t)width, (q1 - q + W - 1) / W);
    if (n == 1) {                              // a pair by itself: four of its rows in flight
      const uint32_t ns = __shfl_sync(mask, nsp, 0, width);
      const int32_t* tm = P.tmap + __shfl_sync(mask, mo, 0, width);
      const double us = __shfl_sync(mask, u, 0, width);
      for (uint32_t k0 = il; k0 < ns; k0 += 4 * width) {
        int32_t t[4];
        double l[4];
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          const uint32_t k = k0 + h * width;
          t[h] = k < ns ? tm[k] : -1;
          l[h] = k < ns ? Lc[k] : 0.0;
        }
#pragma unroll
        for (int h = 0; h < 4; ++h)
          if (t[h] >= 0) atomicAdd(V + t[h], -(l[h] * us));
      }
      continue;
    }
    for (int i = 0; i < n; i += 4) {
      const int32_t* tm[4];
      uint32_t ns[4], most = 0;
      double us[4];
#pragma unroll
      for (int h = 0; h < 4; ++h) {            // lanes past n hold nsp = 0
        const int src = min(i + h, width - 1);
        ns[h] = i + h < n ? __shfl_sync(mask, nsp, src, width) : 0u;
        tm[h] = P.tmap + __shfl_sync(mask, mo, src, width);
        us[h] = __shfl_sync(mask, u, src, width);
        most = max(most, ns[h]);
      }
      for (uint32_t k = il; k < most; k += width) {
        const double l = Lc[k];
        int32_t t[4];
#pragma unroll
        for (int h = 0; h < 4; ++h) t[h] = k < ns[h] ? tm[h][k] : -1;
#pragma unroll
        for (int h = 0; h < 4; ++h)
          if (t[h] >= 0) atomicAdd(V + t[h], -(l * us[h]));
      }
    }
  }
}

// One column c of a sparse level for instance b, by the threads of group g (their warps split the
// U(c,:) pairs): pivot (perturbed if |d| < pert and the column has an L part,
// src/numeric.cu:139-140), L(:,c) /= d (src/numeric.cu:37-47), then for every U(c,j) != 0 the
// targets of column j take -L(:,c) * U(c,j) through the position map (src/numeric.cu:51-89).
// Columns of one level may hit the same target, hence the FP64 atomics (as in the reference).
// SCALE_ONLY: pivot and scaling only (the updates are applied by sparse_split_part or, in the
// deterministic mode, by k_sparse_pull).
// Ls (optional, |L(:,c)| doubles of shared memory, whole-CTA groups only): the scaled L(:,c) is
// also kept there and the updates read it from there instead of from global memory.
template <bool SCALE_ONLY>
__device__ __forceinline__ void sparse_column(const PlanDev& P, double* __restrict__ V, double pv,
                                              int32_t* status, int b, uint32_t c,
                                              const ColGroup& g, double* Ls = nullptr) {
  const uint32_t dslot = P.lp[c];
  const uint32_t l0 = dslot + 1;
  const uint32_t nL = P.cp[c + 1] - l0;
  const double d0 = V[dslot];
  double d = d0;
  const bool perturbed = pv > 0.0 && nL > 0 && fabs(d0) < pv;   // numeric.cu:139-140
  if (perturbed) d = pv;
  group_sync(g);
  if (g.gtid == 0) {
    if (perturbed) V[dslot] = d;
    pivot_flags(status, b, d, perturbed);
  }
  for (uint32_t k = g.gtid; k < nL; k += g.gsize) {
    const double l = V[l0 + k] / d;
    V[l0 + k] = l;
    if (Ls) Ls[k] = l;
  }
  group_sync(g);

  if (SCALE_ONLY) return;
  const double* __restrict__ Lc = Ls ? Ls : V + l0;
  apply_pairs(P, V, c, Lc, nL, g.wig, g.nwg, g.ilane, g.istride, g.mask);
}

// Part `part` of `splits` of column c's pairs (c, j), by the whole CTA: L(:,c) = A(:,c) / d is
// formed in shared memory (Ls, |L(:,c)| doubles; the pivot perturbed as in sparse_column) and
// the part's pairs are applied from there; the column itself is scaled afterwards by
// sparse_column<true>, so no CTA writes what another reads.  Each update is the same L * u
// product as in sparse_column, from the same rounded L.
__device__ __forceinline__ void sparse_split_part(const PlanDev& P, double* __restrict__ V,
                                                  double pv, uint32_t c, int part, int splits,
                                                  double* Ls) {
  const int lane = threadIdx.x % kWarp, wig = threadIdx.x / kWarp, nwg = blockDim.x / kWarp;
  const uint32_t dslot = P.lp[c];
  const uint32_t l0 = dslot + 1;
  const uint32_t nL = P.cp[c + 1] - l0;
  const double d0 = V[dslot];
  const double d = (pv > 0.0 && nL > 0 && fabs(d0) < pv) ? pv : d0;   // numeric.cu:139-140
  __syncthreads();                             // Ls may still be read by the previous item
  for (uint32_t k = threadIdx.x; k < nL; k += 4 * blockDim.x) {
    double a[4];                               // four loads in flight
#pragma unroll
    for (int h = 0; h < 4; ++h)
      a[h] = k + h * blockDim.x < nL ? V[l0 + k + h * blockDim.x] : 0.0;
#pragma unroll
    for (int h = 0; h < 4; ++h)
      if (k + h * blockDim.x < nL) Ls[k + h * blockDim.x] = a[h] / d;
  }
  __syncthreads();
  apply_pairs(P, V, c, Ls, nL, part * nwg + wig, (int64_t)splits * nwg, lane, kWarp, 0xffffffffu);
}

// One launch per sparse level: groups of `wpc` warps share a column (wpc = 1: a warp per
// column; wpc = blockDim/32: the whole CTA), or, with wpc = 1 and lanes < 32, groups of `lanes`
// lanes of a warp (8 or 16: columns whose L parts are that short leave most of a warp idle);
// each group takes `cpw` consecutive columns of the level in turn.  Grid
// (ceil(ncols / (groups per CTA * cpw)), count).  stage: whole-CTA groups keep the scaled L(:,c)
// in dynamic shared memory (the launch sizes it for the level's longest L part) and every warp's
// updates read it from there.
__global__ void __launch_bounds__(256) k_sparse_level(PlanDev P, double* vals,
                                                      const double* pert,
                                                      int32_t* status, int begin, int ncols,
                                                      int wpc, int cpw, int stage, int lanes) {
  after_previous();
  extern __shared__ double Lsm[];
  const int b = blockIdx.y;
  const int gsz = wpc == 1 ? lanes : kWarp * wpc;
  const int groups = blockDim.x / gsz;
  const int gi = threadIdx.x / gsz;
  const int gtid = (int)(threadIdx.x % gsz);
  const unsigned sub = gsz >= kWarp ? 0xffffffffu
                                    : (((1u << gsz) - 1u) << ((threadIdx.x % kWarp) / gsz * gsz));
  const ColGroup g{gtid, gsz, wpc == 1 ? 0 : (int)((threadIdx.x / kWarp) % wpc), wpc,
                   wpc == 1 ? 0 : (groups == 1 ? -1 : 1 + gi),
                   gsz >= kWarp ? (int)(threadIdx.x % kWarp) : gtid, gsz >= kWarp ? kWarp : gsz,
                   sub};
  double* V = vals + (int64_t)b * P.blob;
  const int first = (blockIdx.x * groups + gi) * cpw;
  for (int k = 0; k < cpw; ++k) {
    const int col = first + k;
    if (col >= ncols) break;                   // the same for every thread of the group
    sparse_column<false>(P, V, pert[b], status, b, (uint32_t)P.scols[begin + col], g,
                         stage ? Lsm : nullptr);
  }
}

// Pivot and scaling of a level's columns (a CTA per column): after k_sparse_split, and in the
// deterministic mode before k_sparse_pull.
__global__ void __launch_bounds__(256) k_sparse_scale(PlanDev P, double* vals,
                                                      const double* pert,
                                                      int32_t* status, int begin) {
  after_previous();
  const int b = blockIdx.y;
  sparse_column<true>(P, vals + (int64_t)b * P.blob, pert[b], status, b,
                      (uint32_t)P.scols[begin + blockIdx.x], cta_group());
}

// A narrow level's columns with their updates split over `splits` CTAs each (grid
// (ncols * splits, count)); k_sparse_scale scales the columns afterwards.
__global__ void __launch_bounds__(256) k_sparse_split(PlanDev P, double* vals,
                                                      const double* pert, int begin,
                                                      int splits) {
  after_previous();
  extern __shared__ double Ls[];
  const int b = blockIdx.y;
  const int col = blockIdx.x / splits, part = blockIdx.x % splits;
  sparse_split_part(P, vals + (int64_t)b * P.blob, pert[b], (uint32_t)P.scols[begin + col], part,
                    splits, Ls);
}

// Deterministic level, after k_sparse_scale: one warp per target column j of the level applies
// the level's pairs (c, j) in the level's column order, -L(:,c) * U(c,j) into column j's slots,
// without atomics: the rows of one L(:,c) are distinct, the pairs of one target follow each
// other, and no two warps share a target column.  Same products and sums as sparse_column, in a
// fixed order.  Grid (ceil(targets / 8), count), targets [t0, t0 + ntargets) of det_tptr.
__global__ void __launch_bounds__(256) k_sparse_pull(PlanDev P, double* vals, int64_t t0,
                                                     int64_t ntargets) {
  after_previous();
  const int64_t w = (int64_t)blockIdx.x * (blockDim.x / kWarp) + threadIdx.x / kWarp;
  if (w >= ntargets) return;
  const int lane = threadIdx.x % kWarp;
  double* __restrict__ V = vals + (int64_t)blockIdx.y * P.blob;
  const int64_t e1 = P.det_tptr[t0 + w + 1];
  for (int64_t e = P.det_tptr[t0 + w]; e < e1; ++e) {
    const int64_t q = P.det_q[e];
    const uint32_t c = (uint32_t)P.det_c[e];
    const uint32_t j = (uint32_t)P.pair_j[q];
    const uint32_t l0 = P.lp[c] + 1;
    const uint32_t nL = P.cp[c + 1] - l0;
    const double u = V[P.pair_uslot[q]];
    const int32_t* __restrict__ tm = P.tmap + P.pair_moff[q];
    const uint32_t nsp = j < P.t ? nL : P.lsplit[c];
    for (uint32_t k = lane; k < nsp; k += kWarp) V[tm[k]] += -(V[l0 + k] * u);
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------------------------
// sparse phase: a run of consecutive levels in ONE cooperative launch
// ---------------------------------------------------------------------------------------------

// Barrier among the CTAs of one group: every CTA adds one arrival to the group's counter and
// waits until it reaches `target`.  The wait is bounded: after `budget_ns` of waiting, or as soon
// as another CTA has reported a failure in *err, it gives up, records the failure in *err and
// returns false.  All threads of the CTA must call it.
__device__ bool group_barrier(unsigned* ctr, int* err, unsigned target,
                              unsigned long long budget_ns) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    int ok = 1;
    __threadfence();                           // this CTA's writes before its arrival
    atomicAdd(ctr, 1u);
    const unsigned long long t0 = global_ns();
    while (ld_acquire_u32(ctr) < target) {
      if (*(volatile int*)err) {
        ok = 0;
        break;
      }
      if (global_ns() - t0 > budget_ns) {
        atomicExch(err, 1);
        ok = 0;
        break;
      }
      __nanosleep(64);
    }
    __threadfence();
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// A run of consecutive sparse levels (no fronts among them) for every instance, in one
// cooperative launch: the grid is split into `count` groups of gridDim.x / count CTAs (or, with
// more instances than CTAs, every CTA is a group of one and walks its instances b, b + gridDim.x,
// ... one after another).  A group walks the levels of its instance in order; per level its CTAs
// share the level's columns in the mode the plan chose (desc[l] = {begin, ncols, mode, splits}:
// mode 0 a warp per column, 1 a CTA per column, 3 the column's pairs split over `splits` CTA
// items, then scaled by a CTA each after the level's barrier), with the same per-column code as
// the per-level kernels.  Between levels the group's CTAs meet at a device-side barrier (a
// group of one CTA needs only __syncthreads); instances never depend on each other, so no
// barrier spans groups.  Every wait is bounded (group_barrier): on expiry the CTA marks its
// instances GLU_INST_TIMEOUT, *err becomes non-zero, and every CTA returns.  `extra` arrivals are
// added to every barrier target (0 in use; a test sets 1 to make the first barrier unreachable).
__global__ void __launch_bounds__(256) k_sparse_persistent(PlanDev P, double* vals,
                                                           const double* pert,
                                                           int32_t* status,
                                                           const int4* __restrict__ desc,
                                                           int nlev, int count, unsigned* bar,
                                                           int* err, unsigned long long budget_ns,
                                                           int extra) {
  extern __shared__ double Ls[];
  __shared__ int s_abort;
  const int G = count < (int)gridDim.x ? count : (int)gridDim.x;
  const int cpg = gridDim.x / G;               // CTAs per group
  const int g = blockIdx.x / cpg;
  if (g >= G) return;                          // CTAs beyond G * cpg have no group
  const int r = blockIdx.x % cpg;
  const int warp = threadIdx.x / kWarp, nw = blockDim.x / kWarp;
  unsigned epoch = 0;
  for (int b = g; b < count; b += G) {
    double* V = vals + (int64_t)b * P.blob;
    const double pv = pert[b];
    int4 pending = make_int4(0, 0, -1, 0);     // a split level whose columns still need scaling
    for (int l = 0; l < nlev; ++l) {
      if (threadIdx.x == 0) s_abort = *(volatile int*)err;   // another group gave up
      __syncthreads();
      if (s_abort) {
        if (threadIdx.x == 0 && r == 0)
          for (int bb = b; bb < count; bb += G) atomicOr(status + bb, GLU_INST_TIMEOUT);
        return;
      }
      if (pending.z == 3) {                    // scale the previous split level's columns: no
        for (int col = r; col < pending.y; col += cpg)   // later level reads or writes them
          sparse_column<true>(P, V, pv, status, b, (uint32_t)P.scols[pending.x + col],
                              cta_group());
        pending.z = -1;
      }
      const int4 d = desc[l];
      if (d.z == 0) {
        for (int col = r * nw + warp; col < d.y; col += cpg * nw)
          sparse_column<false>(P, V, pv, status, b, (uint32_t)P.scols[d.x + col], warp_group());
      } else if (d.z == 1) {
        for (int col = r; col < d.y; col += cpg)
          sparse_column<false>(P, V, pv, status, b, (uint32_t)P.scols[d.x + col], cta_group());
      } else {
        for (int it = r; it < d.y * d.w; it += cpg)
          sparse_split_part(P, V, pv, (uint32_t)P.scols[d.x + it / d.w], it % d.w, d.w, Ls);
        pending = d;
      }
      if (cpg > 1) {
        ++epoch;
        if (!group_barrier(bar + g, err, epoch * (unsigned)cpg + (unsigned)extra, budget_ns)) {
          if (threadIdx.x == 0)
            for (int bb = b; bb < count; bb += G) atomicOr(status + bb, GLU_INST_TIMEOUT);
          return;
        }
      } else {
        __syncthreads();
        if (extra > 0) {                       // a group of one CTA has no barrier to miss: the
          if (threadIdx.x == 0) {              // unreachable-target test times out here instead
            const unsigned long long t0 = global_ns();
            while (global_ns() - t0 <= budget_ns && !*(volatile int*)err) __nanosleep(1000);
            atomicExch(err, 1);
            for (int bb = b; bb < count; bb += G) atomicOr(status + bb, GLU_INST_TIMEOUT);
          }
          return;
        }
      }
    }
    if (pending.z == 3) {
      for (int col = r; col < pending.y; col += cpg)
        sparse_column<true>(P, V, pv, status, b, (uint32_t)P.scols[pending.x + col], cta_group());
    }
    if (cpg == 1) __syncthreads();             // Ls and V reuse by the next instance
  }
}

// ---------------------------------------------------------------------------------------------
// solves
// ---------------------------------------------------------------------------------------------

// Also marks the vector's values of the dataflow solves unsolved and clears their failure word and,
// if `fresh`, the instances' kSolveGaveUp.
__global__ void k_permute_in(PlanDev P, int nrhs, const double* Bm, double* y,
                             int64_t ylen, int transpose, double* xbuf, int* err, int32_t* status,
                             int fresh) {
  after_previous();
  const int64_t v = blockIdx.y;                 // instance * nrhs + rhs
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (v == 0) *err = 0;
    if (fresh && v % nrhs == 0) atomicAnd(status + v / nrhs, ~kSolveGaveUp);
  }
  const int64_t nx = solve_buffer(P);
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < nx;
       k += (int64_t)gridDim.x * blockDim.x)
    xbuf[v * nx + k] = __longlong_as_double(kUnsolved);
  const double* bv = Bm + v * P.n;
  double* yv = y + v * ylen;
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < ylen;
       k += (int64_t)gridDim.x * blockDim.x) {
    double out = 0.0;
    if (k < P.n) {
      if (!transpose) {          // symbolic.cc:211-219 with pivot = identity
        const uint32_t src = P.col_perm[k];
        out = P.col_scale_perm ? bv[src] * P.col_scale_perm[k] : bv[src];
      } else {                   // g'[i] = row_scale[row_perm[i]] * g[row_perm[i]]
        const uint32_t src = P.row_perm[k];
        out = P.row_scale ? P.row_scale[src] * bv[src] : bv[src];
      }
    }
    yv[k] = out;
  }
}

__global__ void k_permute_out(PlanDev P, int nrhs, const double* y, double* X,
                              int64_t ylen, int transpose, const int32_t* status) {
  after_previous();
  const int64_t v = blockIdx.y;
  const double* yv = y + v * ylen;
  double* xv = X + v * P.n;
  const bool gave_up = status[v / nrhs] & kSolveGaveUp;   // not a solution
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < P.n;
       k += (int64_t)gridDim.x * blockDim.x) {
    if (!transpose) {            // symbolic.cc:238-245
      double b = yv[P.row_perm_inv[k]];
      b = P.row_scale ? b * P.row_scale[k] : b;
      xv[k] = gave_up ? __longlong_as_double(kNaN) : b;
    } else {                     // lambda[col_perm[k]] = col_scale_perm[k] * w[k]
      const double w = P.col_scale_perm ? P.col_scale_perm[k] * yv[k] : yv[k];
      xv[P.col_perm[k]] = gave_up ? __longlong_as_double(kNaN) : w;
    }
  }
}

// Right-hand sides handled together in the push-form sparse solves: a column's indices and values
// are loaded once for all of them.
constexpr int kSolveVecs = 4;

// The threads that share one column of a sparse solve level: kSolveLong or more entries take a CTA
// of their own (the level's first nlong columns, one per CTA), else a warp each, eight columns
// per CTA; i = the column's place in the level, -1 past its end.  Loads of kSolveUnroll entries
// are in flight per thread: what bounds these kernels is the latency of the loads, a wide level's
// columns being short and a few columns of the netlists (next to the dense block) thousands of
// entries long.  Measured at n = 20,000, one vector: 30 L levels 0.93 -> 0.12 ms, 30 L^T levels
// 0.70 -> 0.17 ms (before: one warp per column, one load in flight); 256 x n = 2,000, 14 L + 14 U
// levels 0.253 -> 0.204 ms (a form of the kernels for one vector, no unrolling of short columns).
constexpr int kSolveUnroll = 4;

struct SolveShare {
  int i, first, step;          // place in the level; first entry and stride of this thread
  bool cta;
};

__device__ __forceinline__ SolveShare solve_share(int ncols, int nlong) {
  if ((int)blockIdx.x < nlong)
    return SolveShare{(int)blockIdx.x, (int)threadIdx.x, (int)blockDim.x, true};
  const int i = nlong + ((int)blockIdx.x - nlong) * (int)(blockDim.x / kWarp) +
                (int)(threadIdx.x / kWarp);
  return SolveShare{i < ncols ? i : -1, (int)(threadIdx.x % kWarp), kWarp, false};
}

// Entries [p0, p1) of a column pushed into nk vectors: y(ri[p]) -= V[p] xc; r0 = ri of the thread's
// first entry.
template <int NV>
__device__ __forceinline__ void solve_push(const PlanDev& P, const double* __restrict__ V,
                                           double* y0, int64_t ylen, int nk,
                                           const double (&xc)[NV], uint32_t p0, uint32_t p1,
                                           uint32_t r0, const SolveShare& sh) {
  uint32_t p = p0 + sh.first;
  if (p1 - p0 <= 2 * (uint32_t)sh.step) {      // short columns: most of them, in a netlist
    for (uint32_t q = p; q < p1; q += sh.step) {
      const uint32_t r = q == p ? r0 : P.ri[q];
      const double m = V[q];
#pragma unroll
      for (int k = 0; k < NV; ++k)
        if (k < nk) atomicAdd(y0 + k * ylen + r, -(m * xc[k]));
    }
    return;
  }
  for (; p < p1; p += kSolveUnroll * sh.step) {
    uint32_t r[kSolveUnroll];
    double m[kSolveUnroll];
#pragma unroll
    for (int u = 0; u < kSolveUnroll; ++u) {
      const uint32_t q = p + u * sh.step;
      r[u] = q < p1 ? P.ri[q] : 0xffffffffu;
      m[u] = q < p1 ? V[q] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < kSolveUnroll; ++u) {
      if (r[u] == 0xffffffffu) break;
#pragma unroll
      for (int k = 0; k < NV; ++k)
        if (k < nk) atomicAdd(y0 + k * ylen + r[u], -(m[u] * xc[k]));
    }
  }
}

// L solve, column oriented with unit diagonal (symbolic.cc:221-226), up to NV (1 or kSolveVecs)
// right-hand sides of one instance together (grid.y = instance * groups + group).
template <int NV>
__global__ void __launch_bounds__(256) k_sparse_lsolve(PlanDev P, const double* vals, int nrhs,
                                                       double* y, int64_t ylen,
                                                       const int32_t* __restrict__ cols, int begin,
                                                       int ncols, int nlong) {
  const SolveShare sh = solve_share(ncols, nlong);
  const uint32_t c = sh.i < 0 ? 0 : (uint32_t)cols[begin + sh.i];
  const uint32_t p0 = P.lp[c] + 1, p1 = P.cp[c + 1];
  const uint32_t r0 = sh.i >= 0 && p0 + sh.first < p1 ? P.ri[p0 + sh.first] : 0;
  after_previous();
  if (sh.i < 0) return;
  const int groups = (nrhs + NV - 1) / NV;
  const int64_t inst = blockIdx.y / groups;
  const int k0 = (blockIdx.y % groups) * NV;
  const int nk = min(NV, nrhs - k0);
  double* y0 = y + (inst * nrhs + k0) * ylen;
  double yc[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) yc[k] = k < nk ? y0[k * ylen + c] : 0.0;
  solve_push(P, vals + inst * P.blob, y0, ylen, nk, yc, p0, p1, r0, sh);
}

// U solve (symbolic.cc:228-236).
template <int NV>
__global__ void __launch_bounds__(256) k_sparse_usolve(PlanDev P, const double* vals, int nrhs,
                                                       double* y, int64_t ylen,
                                                       const int32_t* __restrict__ cols, int begin,
                                                       int ncols, int nlong) {
  const SolveShare sh = solve_share(ncols, nlong);
  const uint32_t c = sh.i < 0 ? 0 : (uint32_t)cols[begin + sh.i];
  const uint32_t p0 = P.cp[c], p1 = P.lp[c];
  const uint32_t r0 = sh.i >= 0 && p0 + sh.first < p1 ? P.ri[p0 + sh.first] : 0;
  after_previous();
  if (sh.i < 0) return;
  const int groups = (nrhs + NV - 1) / NV;
  const int64_t inst = blockIdx.y / groups;
  const int k0 = (blockIdx.y % groups) * NV;
  const int nk = min(NV, nrhs - k0);
  const double* V = vals + inst * P.blob;
  double* y0 = y + (inst * nrhs + k0) * ylen;
  const double d = V[p1];
  double xc[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) xc[k] = k < nk ? y0[k * ylen + c] / d : 0.0;
  if (sh.cta) __syncthreads(); else __syncwarp();   // every thread has read y_c
  if (sh.first < nk) {                         // thread k stores x_c of right-hand side k
    double xv = xc[0];
#pragma unroll
    for (int k = 1; k < NV; ++k)
      if (sh.first == k) xv = xc[k];
    y0[sh.first * ylen + c] = xv;
  }
  solve_push(P, V, y0, ylen, nk, xc, p0, p1, r0, sh);
}

// Sum of V[p] y(ri[p]) over the entries [p0, p1) of a column, in every thread of a warp share, in
// thread 0 of a CTA share; the same order of additions in every run.
__device__ __forceinline__ double solve_pull(const PlanDev& P, const double* __restrict__ V,
                                             const double* yv, uint32_t p0, uint32_t p1,
                                             const SolveShare& sh) {
  __shared__ double part[8];
  double s = 0.0;
  uint32_t p = p0 + sh.first;
  if (p1 - p0 <= 2 * (uint32_t)sh.step)
    for (; p < p1; p += sh.step) s += V[p] * yv[P.ri[p]];
  for (; p < p1; p += kSolveUnroll * sh.step) {
    double m[kSolveUnroll], x[kSolveUnroll];
#pragma unroll
    for (int u = 0; u < kSolveUnroll; ++u) {
      const uint32_t q = p + u * sh.step;
      m[u] = q < p1 ? V[q] : 0.0;
      x[u] = q < p1 ? yv[P.ri[q]] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < kSolveUnroll; ++u) s += m[u] * x[u];
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (sh.cta) {                                // the same for the whole CTA
    if (threadIdx.x % kWarp == 0) part[threadIdx.x / kWarp] = s;
    __syncthreads();
    s = 0.0;
    for (int w = 0; w < (int)(blockDim.x / kWarp); ++w) s += part[w];
  }
  return s;
}

// U^T solve (row j of U^T = column j of U), pull form.
__global__ void __launch_bounds__(256) k_sparse_utsolve(PlanDev P, const double* vals, int nrhs,
                                                        double* y, int64_t ylen,
                                                        const int32_t* __restrict__ cols,
                                                        int begin, int ncols, int nlong) {
  const SolveShare sh = solve_share(ncols, nlong);
  const uint32_t j = sh.i < 0 ? 0 : (uint32_t)cols[begin + sh.i];
  const uint32_t p0 = P.cp[j], p1 = P.lp[j];
  after_previous();
  if (sh.i < 0) return;
  const int64_t v = blockIdx.y;
  const double* V = vals + (v / nrhs) * P.blob;
  double* yv = y + v * ylen;
  const double s = solve_pull(P, V, yv, p0, p1, sh);
  if (sh.first == 0) yv[j] = (yv[j] - s) / V[P.lp[j]];
}

// L^T solve (row j of L^T = column j of L), pull form, unit diagonal.
__global__ void __launch_bounds__(256) k_sparse_ltsolve(PlanDev P, const double* vals, int nrhs,
                                                        double* y, int64_t ylen,
                                                        const int32_t* __restrict__ cols,
                                                        int begin, int ncols, int nlong) {
  const SolveShare sh = solve_share(ncols, nlong);
  const uint32_t j = sh.i < 0 ? 0 : (uint32_t)cols[begin + sh.i];
  const uint32_t p0 = P.lp[j] + 1, p1 = P.cp[j + 1];
  after_previous();
  if (sh.i < 0) return;
  const int64_t v = blockIdx.y;
  const double* V = vals + (v / nrhs) * P.blob;
  double* yv = y + v * ylen;
  const double s = solve_pull(P, V, yv, p0, p1, sh);
  if (sh.first == 0) yv[j] = yv[j] - s;
}

// One level of a phase of the solves of a plan with fronts (WHICH 0: L, 1: U, 2: U^T, 3: L^T), its
// single columns and the products of its fronts with what lies outside them, up to NV right-hand
// sides of one instance together (grid.y = instance * groups + group).  CTAs [0, ncb): columns as
// in the kernels above; U by rows (all entries right of the diagonal pulled), so that the entries
// above a front's rows need no atomics of their own.  The other CTAs take the pieces ext[..]:
//   WHICH 0 / 1, 64 rows by up to 256 columns of L(R, S) or U(S, J), whose columns hold the rows
//   contiguously: y_R -= L(R, S) x_S (after the level's launch_front_flow), y_S -= U(S, J) x_J
//   (before it), a sum per row in registers and one atomic;
//   WHICH 2 / 3, a warp per column: y_x -= U(. < s0, x) . y or L(R, x) . y (before it).
// Bound by the latency of loads on most levels (a few columns and fronts), by HBM on none: the
// grid of 512 x 512 x 2 nodes with 4 vectors reads 0.59 GB a solve.
// Measured on that grid, per solve of 4 vectors: 169 L levels 1.38 ms, 169 U levels 1.17 ms and the
// fronts' own rows (launch_front_flow) 1.55 ms, where pushed columns, one atomic per entry above a
// front and one CTA or cluster per front took 11.6 ms; 128 x 128 x 2, one vector: 1.28 / 1.63 ms.
template <int NV, int WHICH>
__global__ void __launch_bounds__(256) k_solve_level(PlanDev P, const double* vals, int nrhs,
                                                     double* y, int64_t ylen,
                                                     const int32_t* __restrict__ cols, int begin,
                                                     int ncols, int nlong, int ncb,
                                                     const int4* __restrict__ ext) {
  __shared__ double xs[256 * NV];
  __shared__ double red[4 * NV * 64];
  __shared__ uint32_t bs[256];
  const int groups = (nrhs + NV - 1) / NV;
  const int64_t inst = blockIdx.y / groups;
  const int k0 = (blockIdx.y % groups) * NV;
  const int nk = min(NV, nrhs - k0);
  const double* __restrict__ V = vals + inst * P.blob;
  double* y0 = y + (inst * nrhs + k0) * ylen;
  const int tid = threadIdx.x, lane = tid % kWarp, warp = tid / kWarp;
  if ((int)blockIdx.x < ncb) {
    const SolveShare sh = solve_share(ncols, nlong);
    const uint32_t c = sh.i < 0 ? 0 : (uint32_t)cols[begin + sh.i];
    const uint32_t dc = P.lp[c], p0 = dc + 1, p1 = P.cp[c + 1];
    const uint32_t r0 = WHICH == 0 && sh.i >= 0 && p0 + sh.first < p1 ? P.ri[p0 + sh.first] : 0;
    const int64_t e0 = WHICH == 1 ? P.ur_ptr[c] : 0, e1 = WHICH == 1 ? P.ur_ptr[c + 1] : 0;
    after_previous();
    if (sh.i < 0) return;
    if (WHICH == 0) {
      double yc[NV];
#pragma unroll
      for (int k = 0; k < NV; ++k) yc[k] = k < nk ? y0[k * ylen + c] : 0.0;
      solve_push(P, V, y0, ylen, nk, yc, p0, p1, r0, sh);
    } else if (WHICH == 1) {
      double sum[NV];
#pragma unroll
      for (int k = 0; k < NV; ++k) sum[k] = 0.0;
      // the diagonal and the running value are on their way while the row is summed
      const double d = V[dc];
      const double yc = sh.first < nk ? y0[sh.first * ylen + c] : 0.0;
      int64_t e = e0 + sh.first;
      if (e1 - e0 <= 2 * sh.step) {
        for (; e < e1; e += sh.step) {
          const int32_t j = P.ur_col[e];
          const double m = V[P.ur_slot[e]];
#pragma unroll
          for (int k = 0; k < NV; ++k) sum[k] += m * (k < nk ? y0[k * ylen + j] : 0.0);
        }
      }
      for (; e < e1; e += kSolveUnroll * sh.step) {
        int32_t j[kSolveUnroll];
        double m[kSolveUnroll];
#pragma unroll
        for (int u = 0; u < kSolveUnroll; ++u) {
          const int64_t q = e + u * sh.step;
          j[u] = q < e1 ? P.ur_col[q] : -1;
          m[u] = q < e1 ? V[P.ur_slot[q]] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < kSolveUnroll; ++u) {
          if (j[u] < 0) break;
#pragma unroll
          for (int k = 0; k < NV; ++k) sum[k] += m[u] * (k < nk ? y0[k * ylen + j[u]] : 0.0);
        }
      }
#pragma unroll
      for (int k = 0; k < NV; ++k) {
        for (int o = 16; o > 0; o >>= 1) sum[k] += __shfl_xor_sync(0xffffffffu, sum[k], o);
        if (sh.cta && lane == 0) red[k * 8 + warp] = sum[k];
      }
      if (sh.cta) __syncthreads();
      if (sh.first < nk) {                     // thread k finishes right-hand side k
        double t = 0.0;
#pragma unroll
        for (int k = 0; k < NV; ++k)
          if (sh.first == k) t = sum[k];
        if (sh.cta) {
          t = 0.0;
          for (int w = 0; w < 8; ++w) t += red[sh.first * 8 + w];
        }
        y0[sh.first * ylen + c] = (yc - t) / d;
      }
    } else {
      const double t = WHICH == 2 ? solve_pull(P, V, y0, P.cp[c], dc, sh)
                                  : solve_pull(P, V, y0, p0, p1, sh);
      if (sh.first == 0) y0[c] = WHICH == 2 ? (y0[c] - t) / V[dc] : y0[c] - t;
    }
    return;
  }
  const int4 it = ext[blockIdx.x - ncb];
  const int f = it.x, s0 = P.fs0[f], w = P.fw[f];
  after_previous();
  if (WHICH >= 2) {
    const int x = it.y + warp;
    if (x >= w) return;
    const uint32_t d = P.lp[s0 + x];           // rows s0 .. of column s0 + x start at d - x
    const SolveShare sh{x, lane, kWarp, false};
    const double t = WHICH == 2 ? solve_pull(P, V, y0, P.cp[s0 + x], d - x, sh)
                                : solve_pull(P, V, y0, d - x + w, P.cp[s0 + x + 1], sh);
    if (lane == 0) y0[s0 + x] -= t;
    return;
  }
  const int r0 = it.y, c0 = it.z;
  const uint32_t q0 = P.lp[s0] + w;            // rows R in column s0
  const int64_t j0 = WHICH == 1 ? P.uj_ptr[f] + c0 : 0;
  const int rows = WHICH == 0 ? (int)(P.cp[s0 + 1] - q0) : w;
  const int nc = WHICH == 0 ? min(256, w - c0) : (int)min((int64_t)256, P.uj_ptr[f + 1] - j0);
  if (tid < nc) {
    const int32_t j = WHICH == 0 ? s0 + c0 + tid : P.uj_col[j0 + tid];
    bs[tid] = (WHICH == 0 ? P.lp[j] - (c0 + tid) + w : (uint32_t)P.uj_slot[j0 + tid]) + r0;
#pragma unroll
    for (int k = 0; k < NV; ++k) xs[tid * NV + k] = k < nk ? y0[k * ylen + j] : 0.0;
  }
  __syncthreads();
  const int r = tid & 63, seg = tid >> 6;
  double acc[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) acc[k] = 0.0;
  if (r0 + r < rows) {
    int i = seg;
    for (; i + 28 < nc; i += 32) {             // 8 columns of this quarter in flight
      double m[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) m[u] = V[bs[i + 4 * u] + r];
#pragma unroll
      for (int u = 0; u < 8; ++u)
#pragma unroll
        for (int k = 0; k < NV; ++k) acc[k] += m[u] * xs[(i + 4 * u) * NV + k];
    }
    for (; i < nc; i += 4) {
      const double m = V[bs[i] + r];
#pragma unroll
      for (int k = 0; k < NV; ++k) acc[k] += m * xs[i * NV + k];
    }
  }
#pragma unroll
  for (int k = 0; k < NV; ++k) red[(seg * NV + k) * 64 + r] = acc[k];
  __syncthreads();
  for (int e = tid; e < 64 * nk; e += 256) {
    const int row = e % 64, k = e / 64;
    if (r0 + row >= rows) continue;
    double t = 0.0;
#pragma unroll
    for (int g = 0; g < 4; ++g) t += red[(g * NV + k) * 64 + row];
    const uint32_t target = WHICH == 0 ? P.ri[q0 + r0 + row] : (uint32_t)(s0 + r0 + row);
    atomicAdd(y0 + k * ylen + target, -t);
  }
}

// Sums of solved values from the dense block taken off sparse rows (WHICH 1: the entries of U right
// of t) or columns (3: the entries of L below t), up to NV right-hand sides of one instance
// together; the long ones take a CTA.  No atomics, the same order of additions in every run.
template <int NV, int WHICH>
__global__ void __launch_bounds__(256) k_outer_rows(PlanDev P, const double* vals, int nrhs,
                                                    double* y, int64_t ylen, int nrows, int nlong) {
  __shared__ double red[NV * 8];
  const SolveShare sh = solve_share(nrows, nlong);
  const int32_t c = sh.i < 0 ? 0 : (WHICH == 1 ? P.br_rows : P.lc_cols)[sh.i];
  const int64_t e0 = WHICH == 1 ? P.ur_ptr[c] + P.ur_split[c] : (int64_t)P.lp[c] + 1 + P.lsplit[c];
  const int64_t e1 = WHICH == 1 ? P.ur_ptr[c + 1] : (int64_t)P.cp[c + 1];
  after_previous();
  if (sh.i < 0) return;
  const int groups = (nrhs + NV - 1) / NV;
  const int64_t inst = blockIdx.y / groups;
  const int k0 = (blockIdx.y % groups) * NV;
  const int nk = min(NV, nrhs - k0);
  const double* __restrict__ V = vals + inst * P.blob;
  double* y0 = y + (inst * nrhs + k0) * ylen;
  double sum[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) sum[k] = 0.0;
  for (int64_t e = e0 + sh.first; e < e1; e += kSolveUnroll * sh.step) {
    int32_t j[kSolveUnroll];
    double m[kSolveUnroll];
#pragma unroll
    for (int u = 0; u < kSolveUnroll; ++u) {
      const int64_t q = e + u * sh.step;
      j[u] = q < e1 ? (WHICH == 1 ? P.ur_col[q] : (int32_t)P.ri[q]) : -1;
      m[u] = q < e1 ? (WHICH == 1 ? V[P.ur_slot[q]] : V[q]) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < kSolveUnroll; ++u) {
      if (j[u] < 0) break;
#pragma unroll
      for (int k = 0; k < NV; ++k) sum[k] += m[u] * (k < nk ? y0[k * ylen + j[u]] : 0.0);
    }
  }
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    for (int o = 16; o > 0; o >>= 1) sum[k] += __shfl_xor_sync(0xffffffffu, sum[k], o);
    if (sh.cta && threadIdx.x % kWarp == 0) red[k * 8 + threadIdx.x / kWarp] = sum[k];
  }
  if (sh.cta) __syncthreads();
  if (sh.first < nk) {
    double t = 0.0;
#pragma unroll
    for (int k = 0; k < NV; ++k)
      if (sh.first == k) t = sum[k];
    if (sh.cta) {
      t = 0.0;
      for (int w = 0; w < 8; ++w) t += red[sh.first * 8 + w];
    }
    y0[sh.first * ylen + c] -= t;
  }
}

// Row-wise (pull) forward solves of the deterministic mode, one warp per row; each sum is
// formed lane by lane over the row's entries and reduced by shuffles, in a fixed order.
// which 0 (L, unit diagonal): y_r -= sum L(r, c) y_c over the row's entries with c < min(r, t);
// which 1 (U): y_c = (y_c - sum_{j > c} U(c, j) y_j) / U(c, c), the border columns j >= t
// included.  rows: a level's rows rows[begin .. begin + nrows), or nullptr for rows
// begin .. begin + nrows - 1.
__global__ void __launch_bounds__(256) k_rows_solve(PlanDev P, const double* vals, int nrhs,
                                                    double* y, int64_t ylen,
                                                    const int32_t* __restrict__ rows, int begin,
                                                    int nrows, int which) {
  after_previous();
  const int w = blockIdx.x * (blockDim.x / kWarp) + threadIdx.x / kWarp;
  if (w >= nrows) return;
  const int lane = threadIdx.x % kWarp;
  const int64_t v = blockIdx.y;
  const double* __restrict__ V = vals + (v / nrhs) * P.blob;
  double* yv = y + v * ylen;
  const uint32_t r = rows ? (uint32_t)rows[begin + w] : (uint32_t)(begin + w);
  double s = 0.0;
  if (which == 0) {
    for (uint32_t q = P.rp[r] + lane; q < P.dp[r]; q += kWarp) {
      const uint32_t c = P.ci[q];
      if (c < P.t) s += V[P.csr_slot[q]] * yv[c];
    }
  } else {
    for (uint32_t q = P.dp[r] + 1 + lane; q < P.rp[r + 1]; q += kWarp)
      s += V[P.csr_slot[q]] * yv[P.ci[q]];
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) yv[r] = which == 0 ? yv[r] - s : (yv[r] - s) / V[P.lp[r]];
}

// Border U(r < t, j >= t): push x_j into rows r (solve) or pull w_r into w_j (transpose).
__global__ void k_border(PlanDev P, const double* vals, int nrhs, double* y, int64_t ylen,
                         int transpose) {
  after_previous();
  const int jt = blockIdx.x * (blockDim.x / kWarp) + threadIdx.x / kWarp;
  if (jt >= (int)P.nt) return;
  const int lane = threadIdx.x % kWarp;
  const int64_t v = blockIdx.y;
  const double* V = vals + (v / nrhs) * P.blob;
  double* yv = y + v * ylen;
  const int64_t e0 = P.bord_ptr[jt], e1 = P.bord_ptr[jt + 1];
  if (!transpose) {
    const double xj = yv[P.t + jt];
    for (int64_t e = e0 + lane; e < e1; e += kWarp)
      atomicAdd(yv + P.bord_row[e], -(V[P.bord_slot[e]] * xj));
  } else {
    double s = 0.0;
    for (int64_t e = e0 + lane; e < e1; e += kWarp) s += V[P.bord_slot[e]] * yv[P.bord_row[e]];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) yv[P.t + jt] -= s;
  }
}

// The forward solve's border y_r -= U(r, j) x_j (r < t <= j) in chunks of at most 1024 entries
// of one tail column, a warp per chunk and up to NV right-hand sides of an instance (grid
// (ceil(chunks / 8), instances * groups)), so the long border columns of a mesh's top separator
// are shared by many warps and their entries are loaded once per group.
template <int NV>
__global__ void __launch_bounds__(256) k_border_chunks(PlanDev P, const double* vals, int nrhs,
                                                       double* y, int64_t ylen) {
  after_previous();
  const int64_t c = (int64_t)blockIdx.x * (blockDim.x / kWarp) + threadIdx.x / kWarp;
  if (c >= P.nbordck) return;
  const int lane = threadIdx.x % kWarp;
  const int jt = P.bord_ckcol[c];
  const int groups = (nrhs + NV - 1) / NV;
  const int64_t inst = blockIdx.y / groups;
  const int k0 = (blockIdx.y % groups) * NV;
  const int nk = min(NV, nrhs - k0);
  const double* V = vals + inst * P.blob;
  double* y0 = y + (inst * nrhs + k0) * ylen;
  const int64_t e0 = P.bord_ck0[c], e1 = min(e0 + 1024, P.bord_ptr[jt + 1]);
  double xj[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) xj[k] = k < nk ? y0[k * ylen + P.t + jt] : 0.0;
  int64_t e = e0 + lane;
  if (e1 - e0 <= 2 * kWarp) {
    for (; e < e1; e += kWarp) {
      const int32_t r = P.bord_row[e];
      const double m = V[P.bord_slot[e]];
#pragma unroll
      for (int k = 0; k < NV; ++k)
        if (k < nk) atomicAdd(y0 + k * ylen + r, -(m * xj[k]));
    }
    return;
  }
  for (; e < e1; e += kSolveUnroll * kWarp) {
    int32_t r[kSolveUnroll];
    double m[kSolveUnroll];
#pragma unroll
    for (int u = 0; u < kSolveUnroll; ++u) {
      const int64_t q = e + u * kWarp;
      r[u] = q < e1 ? P.bord_row[q] : -1;
      m[u] = q < e1 ? V[P.bord_slot[q]] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < kSolveUnroll; ++u) {
      if (r[u] < 0) break;
#pragma unroll
      for (int k = 0; k < NV; ++k)
        if (k < nk) atomicAdd(y0 + k * ylen + r[u], -(m[u] * xj[k]));
    }
  }
}

__global__ void k_grad(PlanDev P, int nrhs, const double* __restrict__ lambda,
                       const double* __restrict__ x, double* __restrict__ ga) {
  const int64_t b = blockIdx.y;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < P.nnz_g;
       e += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t r = P.g_row[e], c = P.g_col[e];
    double s = 0.0;
    for (int k = 0; k < nrhs; ++k) {
      const int64_t v = (b * nrhs + k) * P.n;
      s += lambda[v + r] * x[v + c];
    }
    ga[b * P.nnz_g + e] = -s;
  }
}

// r = b - A x (or b - A^T x) for every (instance, rhs) vector on the ORIGINAL matrix, and the
// infinity norms ||r||, ||x||, ||b||, ||A|| of each vector (as non-negative double bits) for
// ||r|| / (||A|| ||x|| + ||b||), the acceptance test of the solves.  Grid (chunks, vectors).
__global__ void k_residual(PlanDev P, int nrhs, const double* a,
                           const double* X, const double* Bm,
                           double* R, unsigned long long* norms, int transpose) {
  after_previous();
  residual_rows(P, nrhs, a, X, Bm, R, norms, transpose, blockIdx.y, blockIdx.x, gridDim.x);
}

__global__ void k_resid_finish(int64_t nv, const unsigned long long* norms, double* out) {
  const int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (v < nv) out[v] = residual_ratio(norms + 4 * v);
}

__global__ void k_axpy(int64_t n, const double* dx, double* x) {
  after_previous();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    x[i] += dx[i];
}

inline int grid1(int64_t work, int threads, int cap = 148 * 16) {
  int64_t g = (work + threads - 1) / threads;
  if (g < 1) g = 1;
  if (g > cap) g = cap;
  return (int)g;
}

}  // namespace

// ---------------------------------------------------------------------------------------------
// launch wrappers
// ---------------------------------------------------------------------------------------------

void launch_prepare_blob(const PlanDev& P, double* vals, int first, int count, bool assemble,
                         cudaStream_t s, LaunchCounter& lc) {
  if (assemble) {
    if (P.dbase > 0)
      cudaMemset2DAsync(vals + (int64_t)first * P.blob, sizeof(double) * P.blob, 0,
                        sizeof(double) * P.dbase, count, s);
    if (P.nasm_zero > 0) {
      launch_next(k_zero_slots, dim3(grid1(P.nasm_zero, 256, 256), count), 256, 0, s, P, vals,
                  first);
      lc.n++;
    }
    return;
  }
  cudaMemsetAsync(vals + (int64_t)first * P.blob, 0, sizeof(double) * P.blob * count, s);
  if (P.ntp > P.nt) {
    k_pad_identity<<<dim3(1, count), 64, 0, s>>>(P, vals, first);
    lc.n++;
  }
}

void launch_ingest(const PlanDev& P, double* vals, int first, int count, const double* a,
                   cudaStream_t s, LaunchCounter& lc) {
  launch_next(k_ingest, dim3(grid1(P.nnz_a, 256, 1024), count), 256, 0, s, P, vals, first, a);
  lc.n++;
}

void launch_load_lu(const PlanDev& P, double* vals, int first, int count, const double* val,
                    cudaStream_t s, LaunchCounter& lc) {
  launch_next(k_load_lu, dim3(grid1(P.nnz, 256, 1024), count), 256, 0, s, P, vals, first, val);
  lc.n++;
}

void launch_export_lu(const PlanDev& P, const double* vals, int inst, double* val, cudaStream_t s,
                      LaunchCounter& lc) {
  launch_next(k_export_lu, dim3(grid1(P.nnz, 256)), 256, 0, s, P, vals, inst, val);
  lc.n++;
}

void launch_pert(const PlanDev& P, const double* vals, int count, double pert, double* pert_dev,
                 cudaStream_t s, LaunchCounter& lc) {
  if (pert >= 0.0) {
    launch_next(k_fill, dim3((count + 127) / 128), 128, 0, s, count, pert, pert_dev);
    lc.n++;
    return;
  }
  // pert_dev doubles as the bit accumulator (non-negative doubles order like their bits)
  unsigned long long* bits = reinterpret_cast<unsigned long long*>(pert_dev);
  cudaMemsetAsync(bits, 0, sizeof(double) * count, s);
  k_norm1<<<dim3(grid1(P.n, 8, 512), count), 256, 0, s>>>(P, vals, bits);
  k_pert_finish<<<(count + 127) / 128, 128, 0, s>>>(count, bits, pert_dev);
  lc.n += 2;
}

void launch_sparse_level(const PlanDev& P, double* vals, int count, const double* pert,
                         int32_t* status, int begin, int ncols, int wpc, int max_nl,
                         int max_pairs, int block, int cpw, int lanes, int grow, int occ,
                         cudaStream_t s, LaunchCounter& lc) {
  // a wide level of heavy columns whose columns of the batch are fewer than half the warps the
  // GPU should hold (occ per SM): 2, 4 or 8 warps per column, so the pairs of each column are
  // shared instead of walked by one warp
  const int64_t want = (int64_t)occ * sm_count();
  if (grow && occ > 0 && wpc == 1)
    while (wpc < 8 && (int64_t)ncols * count * wpc * 2 <= want && max_pairs > 4 * wpc) wpc *= 2;
  // a level whose CTA-per-column grid covers fewer CTAs than the GPU should hold (occ warps per
  // SM, two CTAs per SM when occ = 0) and whose columns have more pairs than one CTA's warps:
  // split each column's pairs over several CTAs
  constexpr int kSplitMaxL = 6144;               // L(:,c) staged in 48 KB of shared memory
  const int64_t ctas = (int64_t)ncols * count;
  const int64_t target = occ > 0 ? std::max<int64_t>(want / 8, 2 * (int64_t)sm_count())
                                 : 2 * (int64_t)sm_count();
  if (wpc > 1 && ctas < target && max_pairs > 16 && max_nl <= kSplitMaxL) {
    int splits = (int)std::min<int64_t>((target + ctas - 1) / ctas, (max_pairs + 7) / 8);
    launch_next(k_sparse_split, dim3(ncols * splits, count), 256, sizeof(double) * std::max(max_nl,
                1), s, P, vals, pert, begin, splits);
    launch_next(k_sparse_scale, dim3(ncols, count), 256, 0, s, P, vals, pert, status, begin);
    lc.n += 2;
    return;
  }
  if (block != 128) block = 256;
  wpc = std::max(1, std::min(wpc, block / kWarp));
  if (wpc > 1 || (lanes != 8 && lanes != 16)) lanes = kWarp;
  const int groups = block / (wpc == 1 ? lanes : kWarp * wpc);
  const int per_cta = groups * std::max(1, cpw);
  // a CTA per column: its L(:,c) staged in shared memory when eight CTAs of it still fit on an
  // SM (at most 24 KB each), so the staging costs no occupancy
  constexpr int kStageMaxL = 3072;
  const bool stage = groups == 1 && max_nl > 0 && max_nl <= kStageMaxL;
  const size_t smem = stage ? sizeof(double) * max_nl : 0;
  launch_next(k_sparse_level, dim3((ncols + per_cta - 1) / per_cta, count), block, smem, s, P, vals,
              pert, status, begin, ncols, wpc, std::max(1, cpw), stage ? 1 : 0, lanes);
  lc.n++;
}

void launch_sparse_level_det(const PlanDev& P, double* vals, int count, const double* pert,
                             int32_t* status, int begin, int ncols, int64_t t0, int64_t t1,
                             cudaStream_t s, LaunchCounter& lc) {
  launch_next(k_sparse_scale, dim3(ncols, count), 256, 0, s, P, vals, pert, status, begin);
  lc.n++;
  const int64_t nt = t1 - t0;
  if (nt > 0) {
    launch_next(k_sparse_pull, dim3((unsigned)((nt + 7) / 8), count), 256, 0, s, P, vals, t0, nt);
    lc.n++;
  }
}

void launch_rows_solve(const PlanDev& P, const double* vals, int count, int nrhs, double* y,
                       int64_t ylen, const int32_t* rows, int begin, int nrows, int which,
                       cudaStream_t s, LaunchCounter& lc) {
  if (nrows <= 0) return;
  launch_next(k_rows_solve, dim3((nrows + 7) / 8, count * nrhs), 256, 0, s, P, vals, nrhs, y, ylen,
              rows, begin, nrows, which);
  lc.n++;
}

int persistent_grid(size_t smem) {
  int dev = 0, per_sm = 0;
  cudaGetDevice(&dev);
  ensure_smem_limit((const void*)k_sparse_persistent, smem);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_sparse_persistent, 256, smem) !=
          cudaSuccess ||
      per_sm < 1) {
    cudaGetLastError();
    return 0;
  }
  return per_sm * sm_count();
}

void launch_sparse_persistent(const PlanDev& P, double* vals, int count, const double* pert,
                              int32_t* status, const int4* desc, int nlev, unsigned* bar,
                              int groups, int* err, double budget_ms, int extra, int grid,
                              size_t smem, cudaStream_t s, LaunchCounter& lc) {
  cudaMemsetAsync(bar, 0, sizeof(unsigned) * groups, s);
  cudaMemsetAsync(err, 0, sizeof(int), s);
  ensure_smem_limit((const void*)k_sparse_persistent, smem);
  const unsigned long long budget = (unsigned long long)(budget_ms * 1e6);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(256);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;      // every CTA resident at once
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, k_sparse_persistent, P, vals, pert, status, desc, nlev, count, bar, err,
                     budget, extra);
  lc.n++;
}

void launch_solve_permute_in(const PlanDev& P, int count, int nrhs, const double* B, double* y,
                             int64_t ylen, int transpose, double* xbuf, int* err, int32_t* status,
                             bool fresh, cudaStream_t s, LaunchCounter& lc) {
  launch_next(k_permute_in, dim3(grid1(ylen, 256, 256), count * nrhs), 256, 0, s, P, nrhs, B, y,
              ylen, transpose, xbuf, err, status, fresh ? 1 : 0);
  lc.n++;
}

void launch_solve_permute_out(const PlanDev& P, int count, int nrhs, const double* y, double* X,
                              int64_t ylen, int transpose, const int32_t* status, cudaStream_t s,
                              LaunchCounter& lc) {
  launch_next(k_permute_out, dim3(grid1(P.n, 256, 256), count * nrhs), 256, 0, s, P, nrhs, y, X,
              ylen, transpose, status);
  lc.n++;
}

void launch_sparse_lsolve(const PlanDev& P, const double* vals, int count, int nrhs, double* y,
                          int64_t ylen, const int32_t* cols, int begin, int ncols, int nlong,
                          cudaStream_t s, LaunchCounter& lc) {
  const unsigned gx = nlong + (ncols - nlong + 7) / 8;
  if (nrhs == 1)
    launch_next(k_sparse_lsolve<1>, dim3(gx, count), 256, 0, s, P, vals, nrhs, y, ylen, cols, begin,
                ncols, nlong);
  else
    launch_next(k_sparse_lsolve<kSolveVecs>, dim3(gx,
                count * ((nrhs + kSolveVecs - 1) / kSolveVecs)), 256, 0, s, P, vals, nrhs, y, ylen,
                cols, begin, ncols, nlong);
  lc.n++;
}
void launch_sparse_usolve(const PlanDev& P, const double* vals, int count, int nrhs, double* y,
                          int64_t ylen, const int32_t* cols, int begin, int ncols, int nlong,
                          cudaStream_t s, LaunchCounter& lc) {
  const unsigned gx = nlong + (ncols - nlong + 7) / 8;
  if (nrhs == 1)
    launch_next(k_sparse_usolve<1>, dim3(gx, count), 256, 0, s, P, vals, nrhs, y, ylen, cols, begin,
                ncols, nlong);
  else
    launch_next(k_sparse_usolve<kSolveVecs>, dim3(gx,
                count * ((nrhs + kSolveVecs - 1) / kSolveVecs)), 256, 0, s, P, vals, nrhs, y, ylen,
                cols, begin, ncols, nlong);
  lc.n++;
}
void launch_sparse_utsolve(const PlanDev& P, const double* vals, int count, int nrhs, double* y,
                           int64_t ylen, const int32_t* cols, int begin, int ncols, int nlong,
                           cudaStream_t s, LaunchCounter& lc) {
  launch_next(k_sparse_utsolve, dim3(nlong + (ncols - nlong + 7) / 8, count * nrhs), 256, 0, s, P,
              vals, nrhs, y, ylen, cols, begin, ncols, nlong);
  lc.n++;
}
void launch_sparse_ltsolve(const PlanDev& P, const double* vals, int count, int nrhs, double* y,
                           int64_t ylen, const int32_t* cols, int begin, int ncols, int nlong,
                           cudaStream_t s, LaunchCounter& lc) {
  launch_next(k_sparse_ltsolve, dim3(nlong + (ncols - nlong + 7) / 8, count * nrhs), 256, 0, s, P,
              vals, nrhs, y, ylen, cols, begin, ncols, nlong);
  lc.n++;
}

void launch_solve_level(const PlanDev& P, const double* vals, int count, int nrhs, double* y,
                        int64_t ylen, const int32_t* cols, int begin, int ncols, int nlong,
                        const FrontLevelSolve& L, int which, cudaStream_t s, LaunchCounter& lc) {
  const int ncb = nlong + (ncols - nlong + 7) / 8;
  if (ncb + L.next == 0) return;
  const int4* ext = reinterpret_cast<const int4*>(L.ext);
  const auto launch = [&](auto kern, int nv) {
    launch_next(kern, dim3(ncb + L.next, count * ((nrhs + nv - 1) / nv)), 256, 0, s, P, vals, nrhs,
                y, ylen, cols, begin, ncols, nlong, ncb, ext);
    lc.n++;
  };
  if (which == 0) nrhs == 1 ? launch(k_solve_level<1, 0>, 1) : launch(k_solve_level<kSolveVecs, 0>, kSolveVecs);
  if (which == 1) nrhs == 1 ? launch(k_solve_level<1, 1>, 1) : launch(k_solve_level<kSolveVecs, 1>, kSolveVecs);
  if (which == 2) launch(k_solve_level<1, 2>, 1);
  if (which == 3) launch(k_solve_level<1, 3>, 1);
}

void launch_outer_rows(const PlanDev& P, const double* vals, int count, int nrhs, double* y,
                       int64_t ylen, int nrows, int nlong, int which, cudaStream_t s,
                       LaunchCounter& lc) {
  if (nrows == 0) return;
  const unsigned gx = nlong + (nrows - nlong + 7) / 8;
  const auto launch = [&](auto kern, int nv) {
    launch_next(kern, dim3(gx, count * ((nrhs + nv - 1) / nv)), 256, 0, s, P, vals, nrhs, y, ylen,
                nrows, nlong);
    lc.n++;
  };
  if (which == 1 && nrhs == 1) launch(k_outer_rows<1, 1>, 1);
  else if (which == 1) launch(k_outer_rows<kSolveVecs, 1>, kSolveVecs);
  else if (nrhs == 1) launch(k_outer_rows<1, 3>, 1);
  else launch(k_outer_rows<kSolveVecs, 3>, kSolveVecs);
}

void launch_border(const PlanDev& P, const double* vals, int count, int nrhs, double* y,
                   int64_t ylen, int transpose, cudaStream_t s, LaunchCounter& lc) {
  if (P.nt == 0) return;
  const unsigned gx = (unsigned)((P.nbordck + 7) / 8);
  if (!transpose && P.nbordck > 0 && nrhs == 1)
    launch_next(k_border_chunks<1>, dim3(gx, count), 256, 0, s, P, vals, nrhs, y, ylen);
  else if (!transpose && P.nbordck > 0)
    launch_next(k_border_chunks<kSolveVecs>, dim3(gx,
                count * ((nrhs + kSolveVecs - 1) / kSolveVecs)), 256, 0, s, P, vals, nrhs, y, ylen);
  else
    launch_next(k_border, dim3((P.nt + 7) / 8, count * nrhs), 256, 0, s, P, vals, nrhs, y, ylen,
                transpose);
  lc.n++;
}

void launch_residual(const PlanDev& P, int count, int nrhs, const double* a, const double* X,
                     const double* B, double* R, unsigned long long* norms, double* resid,
                     int transpose, cudaStream_t s, LaunchCounter& lc) {
  const int64_t nv = (int64_t)count * nrhs;
  cudaMemsetAsync(norms, 0, sizeof(unsigned long long) * 4 * nv, s);
  launch_next(k_residual, dim3(grid1(P.n, 256, 64), (unsigned)nv), 256, 0, s, P, nrhs, a, X, B, R,
              norms, transpose);
  lc.n++;
  if (resid) {
    k_resid_finish<<<(unsigned)((nv + 127) / 128), 128, 0, s>>>(nv, norms, resid);
    lc.n++;
  }
}

void launch_axpy(int64_t n, const double* dx, double* x, cudaStream_t s, LaunchCounter& lc) {
  launch_next(k_axpy, dim3(grid1(n, 256, 4096)), 256, 0, s, n, dx, x);
  lc.n++;
}

void launch_grad(const PlanDev& P, int count, int nrhs, const double* lambda, const double* x,
                 double* ga, cudaStream_t s, LaunchCounter& lc) {
  k_grad<<<dim3(grid1(P.nnz_g, 256, 1024), count), 256, 0, s>>>(P, nrhs, lambda, x, ga);
  lc.n++;
}

}  // namespace glu
