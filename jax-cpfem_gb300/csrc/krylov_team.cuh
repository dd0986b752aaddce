// The persistent BiCGSTAB of one system, or of a batch of systems by teams of blocks: the
// kernel of the point preconditioners (krylov_point.cu) and of the multigrid V-cycle
// (krylov_mg.cu).
//
// What bounds an iteration at these sizes is latency: five dependencies that cross the grid,
// and FP64 instructions, which GB300 issues at one warp instruction per 64 cycles and
// sub-partition, with 65 cycles of latency (a division takes 550).  So
//  * the nodes are spread over all SMs, one block each, in equal contiguous ranges.  A warp
//    takes one of the three rows of 32 / QL consecutive nodes, and QL lanes share a row's
//    neighbour slots.  With one thread per node a 10^3 mesh ran on 6 SMs.
//  * every vector but the two that neighbours gather lives in the block's shared memory, and
//    so do, where they fit, the block's matrix rows and column indices (up to ~21^3 cells),
//    copied once per solve.  A transposed solve copies the transposed rows, so its product
//    reads shared memory in order like any other.
//  * FP64 instructions are spent where there is data: one lane computes the scalars, one
//    warp adds a sum, comparisons of non-negative numbers are integer ones.
// us per Jacobi iteration on one GB300, one thread per node on n / 256 blocks -> this kernel:
// 1 cell 30 -> 17, 10^3 57 -> 19, 16^3 60 -> 20, 24^3 60 -> 33, 32^3 61 -> 51, 40^3 116 -> 87.
// Every sum has a fixed order, so a solve is bitwise reproducible, and all blocks of a team
// hold the same scalars and take the same branch.  Polls are bounded: a block that waits too
// long sets the error flag, on which all waits end, and the solve returns CPFEM_ERR_SOLVE.
#pragma once

#include <type_traits>

#include "krylov_point.cuh"
#include "reduce.cuh"

namespace cpfem {

constexpr int kPtMaxThreads = 768;
constexpr int kMgThreads = 256;                      // the V-cycle's kernel: 255 registers a thread
constexpr int kPtMaxWidth = 27;                      // slots per row the plan counts on
constexpr int kPtSmemBytes = 206 * 1024;             // dynamic shared memory of a block, at most
constexpr int kPtSpinLimit = 1 << 22;                 // polls of ~0.4 us each: a second or two

// Diagonal (precond 1) or inverted 3x3 diagonal block (precond 2) per node.
template <bool TRANS>
__global__ void k_precond_setup(const cpfem_sell_t L, const double* __restrict__ vals, int precond,
                                double* __restrict__ minv) {
  const int64_t a = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= L.num_nodes) return;
  const double* v0 = vals + 9 * L.group_off[a >> 5] + (a & 31) + 288 * (int64_t)L.diag_slot[a];
  double blk[9];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const double v = v0[32 * (3 * i + k)];
      if (TRANS) blk[3 * k + i] = v; else blk[3 * i + k] = v;
    }
  if (precond == 1) {
#pragma unroll
    for (int i = 0; i < 3; ++i) minv[3 * a + i] = 1.0 / blk[4 * i];
  } else {
    double bi[9];
    inv3(blk, bi);
#pragma unroll
    for (int c = 0; c < 9; ++c) minv[9 * a + c] = bi[c];
  }
}

struct PtTeam {
  int first, nb, id;
  unsigned int seq;   // barriers crossed
};

struct PtShared {
  double part[kPointMaxValues][kPtMaxThreads];     // the threads' partial sums
  double sum[kPointMaxValues];
  double alpha, omega, beta;
  double rho, rho_new, rs, atol2, cap, drift;      // thread 0's
  int bad, steps, k, go, early, restart;           // bad: a wait of this block ran out
  int lb;                                          // multigrid: mg_dense_from
};

// One warp adds v[0 .. n) in a fixed order; the result is valid in lane 0.
__device__ __forceinline__ double pt_warp_total(const double* v, int n) {
  const int lane = threadIdx.x & 31;
  double a0 = 0.0, a1 = 0.0;
  int i = lane;
  for (; i + 32 < n; i += 64) {
    a0 += v[i];
    a1 += v[i + 32];
  }
  if (i < n) a0 += v[i];
  double acc[1] = {n > 32 ? a0 + a1 : a0};
  warp_sum<1>(acc);
  return acc[0];
}

// Team-wide sums of NV values, left in sh.sum (NV = 0: a barrier); also publishes every global
// write the block made before.  The threads below `active` hold partial sums.  The block's
// total of value k is warp k's work, as is the team's, whose partials every block adds in
// block order, so all hold the same bits.  The FP64 pipe is why: a warp instruction takes it
// 64 cycles, and a shuffle tree in all 16 warps costs more of it than the vector work it sums.
// The barrier is a counter that only grows (zeroed before the launch): one arrival per block,
// one polling warp per value.  Every 64th poll looks at the error word too, so once a block has
// waited too long all other waits, and its own later ones in the iteration, end within
// microseconds.  (Testing sh.bad here instead cost the multigrid kernel 2 to 5 %.)
template <int NV>
__device__ __forceinline__ void pt_reduce(const double* v, int active, PtTeam& tm, const PointArgs& a, PtShared& sh) {
  constexpr int NC = NV > 0 ? NV : 1;
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if constexpr (NV > 0) {
    if ((int)threadIdx.x < active)
#pragma unroll
      for (int k = 0; k < NC; ++k) sh.part[k][threadIdx.x] = v[k];
    __syncthreads();
  }
  double* const cells = a.cells + (size_t)(tm.seq & 1) * kPointMaxValues * kPointMaxBlocks;
  tm.seq += 1;
  if constexpr (NV > 0) {
    if (wid < NC) {
      const double tot = pt_warp_total(sh.part[wid], active);
      if (lane == 0) {
        if (tm.nb == 1) sh.sum[wid] = tot;
        else __stcg(cells + wid * kPointMaxBlocks + blockIdx.x, tot);
      }
    }
  }
  __syncthreads();
  if (tm.nb == 1) return;
  if (wid < NC) {
    unsigned int* const count = a.counters + 32 * tm.id;
    const unsigned int target = tm.seq * (unsigned)tm.nb;
    if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(count), "r"(1u) : "memory");
    if (lane == 0) {
      unsigned int c;
      int spins = 0;
      for (;;) {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(count) : "memory");
        if (c >= target) break;
        if ((++spins & 63) == 0 && (spins >= a.polls || *(volatile int*)a.error != 0)) break;
      }
      if (c < target) {
        atomicExch(a.error, 1);
        sh.bad = 1;
      }
    }
    __syncwarp();
    if constexpr (NV > 0) {
      const double* p = cells + wid * kPointMaxBlocks + tm.first;
      constexpr int kPer = (kPointMaxBlocks + 31) / 32;
      double c[kPer];
#pragma unroll
      for (int i = 0; i < kPer; ++i) c[i] = (lane + 32 * i < tm.nb) ? __ldcg(p + lane + 32 * i) : 0.0;
      double acc[1] = {c[0]};
#pragma unroll
      for (int i = 1; i < kPer; ++i)
        if (32 * i < tm.nb) acc[0] += c[i];
      warp_sum<1>(acc);
      if (lane == 0) sh.sum[wid] = acc[0];
    }
  }
  __syncthreads();
}

__device__ __forceinline__ double mad(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float mad(float a, float b, float c) { return fmaf(a, b, c); }

// An operator value in the precision R of the product.  FP64 -> FP32 by integer operations on
// the two words of the double (exponent re-bias, mantissa truncated to 23 bits, magnitudes
// below FP32's normal range flushed to zero), so the FP32 V-cycle can read the resident FP64
// operator without a conversion instruction per value on GB300's narrow FP64 pipe.  The
// truncation error (< 2^-23 relative) is below what an FP32 preconditioner resolves.
template <typename R>
__device__ __forceinline__ R opval(double v);
template <>
__device__ __forceinline__ double opval<double>(double v) { return v; }
template <>
__device__ __forceinline__ float opval<float>(double v) {
  const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
  const int e = (int)((hi >> 20) & 0x7FFu) - 1023 + 127;
  const unsigned bits = (e <= 0) ? (hi & 0x80000000u)
                                 : ((hi & 0x80000000u) | ((unsigned)e << 23) | ((hi & 0xFFFFFu) << 3) | (lo >> 29));
  return __uint_as_float(bits);
}

// a > b, and a <= b, for a, b that are sums of squares or NaN of either sign (CUDA's own has it set;
// then false), and v == 0, without the FP64 pipe.
__device__ __forceinline__ long long pt_bits(double v) { return __double_as_longlong(v) & 0x7FFFFFFFFFFFFFFFll; }
__device__ __forceinline__ bool pt_greater(double a, double b) {
  const long long x = pt_bits(a), y = pt_bits(b);
  return x > y && x <= 0x7FF0000000000000ll;    // b NaN: no x that is none lies above it
}
__device__ __forceinline__ bool pt_at_most(double a, double b) {
  const long long x = pt_bits(a), y = pt_bits(b);
  return x <= y && y <= 0x7FF0000000000000ll;
}
__device__ __forceinline__ bool pt_zero(double v) { return (__double_as_longlong(v) << 1) == 0ll; }

// The block's share of the system and where its copies live.
struct PtLocal {
  int64_t n0;        // first node
  int nn;            // nodes
  int units;         // groups of 32 / QL nodes
  int steps;         // slots per lane, at most
  bool staged;
  double* mat;       // [unit][row][step][3][32]
  int* cols;         // [unit][step][32], 3 * node
};

// The 3x3 block of node nd's slot (of A^T when TRANS): row i, column c at [stride_i i + stride_c c].
template <bool TRANS>
__device__ __forceinline__ const double* pt_block(const PointArgs& a, int64_t nd, int64_t goff, int slot) {
  const int l = (int)(nd & 31);
  if (!TRANS) return a.vals + 9 * goff + l + 288 * (int64_t)slot;
  const int64_t col = __ldg(&a.L.cols[goff + 32 * slot + l]);
  return a.vals + 9 * __ldg(&a.L.group_off[col >> 5]) + (col & 31) + 288 * (int64_t)__ldg(&a.L.tpos[goff + 32 * slot + l]);
}

// One row of 32 / QL nodes of A x (A^T x): this warp's task, x gathered from global memory.
// Plain loads: what other blocks wrote is ordered by the reduction's acquire, and a node's
// neighbours share most of each other's values, which L1 then serves.  Two chains: a row's
// FMAs are latency where few warps are at work.  In FP64, or in FP32 on values truncated in
// registers (a V-cycle's sweeps).  Returns the sum in every lane of the node.
template <bool TRANS, int QL, bool STAGED, typename R>   // STAGED: the rows are
__device__ __forceinline__ R pt_row(const PointArgs& a, const PtLocal& B, const R* x, int unit, int row) {
  constexpr int NPW = 32 / QL;
  constexpr int RS = TRANS ? 32 : 96, CS = TRANS ? 96 : 32;   // strides of a block's row, column
  const int lane = threadIdx.x & 31;
  const int node = lane % NPW, q = lane / NPW;
  R acc = R(0), acc2 = R(0);
  if (STAGED || B.staged) {
    const double* m = B.mat + ((size_t)(3 * unit + row) * B.steps) * 96 + lane;
    const int* c = B.cols + (size_t)unit * B.steps * 32 + lane;
    int j = 0;
#pragma unroll 2
    for (; j + 1 < B.steps; j += 2) {
      const R *xb = x + c[32 * j], *xc = x + c[32 * j + 32];
      const R x0 = xb[0], x1 = xb[1], x2 = xb[2], y0 = xc[0], y1 = xc[1], y2 = xc[2];
      acc = mad(opval<R>(m[96 * j]), x0, mad(opval<R>(m[96 * j + 32]), x1, mad(opval<R>(m[96 * j + 64]), x2, acc)));
      acc2 = mad(opval<R>(m[96 * j + 96]), y0, mad(opval<R>(m[96 * j + 128]), y1, mad(opval<R>(m[96 * j + 160]), y2, acc2)));
    }
    if (j < B.steps) {
      const R* xb = x + c[32 * j];
      acc = mad(opval<R>(m[96 * j]), xb[0], mad(opval<R>(m[96 * j + 32]), xb[1], mad(opval<R>(m[96 * j + 64]), xb[2], acc)));
    }
  } else if (unit * NPW + node < B.nn) {
    const int64_t nd = B.n0 + (int64_t)(unit * NPW + node);
    const int64_t goff = a.L.group_off[nd >> 5];
    const int32_t* cols = a.L.cols + goff + (nd & 31);
    const int w = a.L.group_width[nd >> 5];
    int j = q;
#pragma unroll 2
    for (; j + QL < w; j += 2 * QL) {
      const double *vb = pt_block<TRANS>(a, nd, goff, j) + RS * row, *vc = pt_block<TRANS>(a, nd, goff, j + QL) + RS * row;
      const R *xb = x + 3 * (int64_t)__ldg(&cols[32 * j]), *xc = x + 3 * (int64_t)__ldg(&cols[32 * (j + QL)]);
      const double a0 = __ldg(&vb[0]), a1 = __ldg(&vb[CS]), a2 = __ldg(&vb[2 * CS]);
      const double b0 = __ldg(&vc[0]), b1 = __ldg(&vc[CS]), b2 = __ldg(&vc[2 * CS]);
      const R x0 = xb[0], x1 = xb[1], x2 = xb[2], y0 = xc[0], y1 = xc[1], y2 = xc[2];
      acc = mad(opval<R>(a0), x0, mad(opval<R>(a1), x1, mad(opval<R>(a2), x2, acc)));
      acc2 = mad(opval<R>(b0), y0, mad(opval<R>(b1), y1, mad(opval<R>(b2), y2, acc2)));
    }
    if (j < w) {
      const double* vb = pt_block<TRANS>(a, nd, goff, j) + RS * row;
      const R* xb = x + 3 * (int64_t)__ldg(&cols[32 * j]);
      acc = mad(opval<R>(__ldg(&vb[0])), xb[0], mad(opval<R>(__ldg(&vb[CS])), xb[1], mad(opval<R>(__ldg(&vb[2 * CS])), xb[2], acc)));
    }
  }
  __syncwarp();
  acc += acc2;
#pragma unroll
  for (int o = NPW; o < 32; o <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  return acc;
}

// The three rows of 32 / QL nodes of A x by one warp, from global memory: a slot's column and x
// are read once for its nine values (half the loads of three row tasks, a third where a
// transposed block has to be found first), so it streams large systems better; it needs the
// registers of a kernel with few warps to keep its loads in flight.
template <bool TRANS, int QL, typename R>
__device__ __forceinline__ void pt_nodes(const PointArgs& a, const PtLocal& B, const R* x, int unit, R* y) {
  constexpr int NPW = 32 / QL;
  constexpr int RS = TRANS ? 32 : 96, CS = TRANS ? 96 : 32;
  const int lane = threadIdx.x & 31, q = lane / NPW;
  const int k = unit * NPW + lane % NPW;
  R e[3] = {R(0), R(0), R(0)}, o[3] = {R(0), R(0), R(0)};   // even and odd slots: independent chains
  if (k < B.nn) {
    const int64_t nd = B.n0 + k, goff = a.L.group_off[nd >> 5];
    const int32_t* cols = a.L.cols + goff + (nd & 31);
    const int w = a.L.group_width[nd >> 5];
    auto slot = [&](int j, R (&s)[3]) {
      const R* xb = x + 3 * (int64_t)__ldg(&cols[32 * j]);
      const double* vb = pt_block<TRANS>(a, nd, goff, j);
      const R x0 = xb[0], x1 = xb[1], x2 = xb[2];
#pragma unroll
      for (int i = 0; i < 3; ++i)
        s[i] = mad(opval<R>(__ldg(&vb[RS * i])), x0,
                   mad(opval<R>(__ldg(&vb[RS * i + CS])), x1, mad(opval<R>(__ldg(&vb[RS * i + 2 * CS])), x2, s[i])));
    };
    int j = q;
#pragma unroll 2
    for (; j + QL < w; j += 2 * QL) {
      slot(j, e);
      slot(j + QL, o);
    }
    if (j < w) slot(j, e);
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    e[i] += o[i];
#pragma unroll
    for (int off = NPW; off < 32; off <<= 1) e[i] += __shfl_xor_sync(0xffffffffu, e[i], off);
    if (lane < NPW && k < B.nn) y[3 * k + i] = e[i];
  }
}

// y = A x for the block's rows in precision R, x complete in global memory; ends with every y
// visible to the block.  NODES: rows that are not staged by pt_nodes.
template <bool TRANS, int QL, bool NODES, typename R>
__device__ __forceinline__ void pt_product(const PointArgs& a, const PtLocal& B, const R* x, R* y) {
  constexpr int NPW = 32 / QL;
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = (int)(blockDim.x >> 5);
  if (NODES && !B.staged) {
    // whole rounds of the warps; a last round of a few units is shared out in halves or quarters
    // (at 48^3 a block has 25 units for its 8 warps)
    const int whole = B.units / warps * warps, rest = B.units - whole;
    const int split = QL <= 2 && 4 * rest <= warps ? 4 : 2 * rest <= warps ? 2 : 1;
    for (int u = wid; u < (split > 1 ? whole : B.units); u += warps) pt_nodes<TRANS, QL, R>(a, B, x, u, y);
    if (split == 2 && wid < 2 * rest) pt_nodes<TRANS, 2 * QL, R>(a, B, x, 2 * whole + wid, y);
    if constexpr (QL <= 2)
      if (split == 4 && wid < 4 * rest) pt_nodes<TRANS, 4 * QL, R>(a, B, x, 4 * whole + wid, y);
  } else {
    for (int task = wid; task < 3 * B.units; task += warps) {
      const int u = task / 3, row = task - 3 * u;
      const R acc = pt_row<TRANS, QL, NODES, R>(a, B, x, u, row);
      const int k = u * NPW + lane;
      if (lane < NPW && k < B.nn) y[3 * k + row] = acc;
    }
  }
  __syncthreads();
}

// ... out of line, where the V-cycle calls it from a dozen places.
template <bool TRANS, int QL, typename R>
__device__ __noinline__ void pt_product_call(const PointArgs& a, const PtLocal B, const R* x, R* y) {
  pt_product<TRANS, QL, true, R>(a, B, x, y);
}

// The multigrid V-cycle in precision R (krylov_mg.cuh).
template <bool TRANS, int QL, typename R>
__device__ __noinline__ void mg_vcycle(const PointArgs& a, const cpfem_mg_t& mg, const PtLocal& B, const double* v, double* hat,
                          double* out, R* y, PtTeam& tm, PtShared& sh);
template <typename R>
__device__ __forceinline__ int mg_dense_from(const cpfem_mg_t& mg);

struct NoMg {};   // the preconditioner argument of the point kernel

// MR: void for a point preconditioner (a.precond), or the V-cycle's precision.
template <bool TRANS, int QL, typename MR, typename MG>
__global__ void __launch_bounds__(std::is_void<MR>::value ? kPtMaxThreads : kMgThreads, 1) k_bicgstab_team(
    const __grid_constant__ PointArgs a, const __grid_constant__ MG mg) {
  constexpr bool kMg = !std::is_void<MR>::value;
  constexpr int NPW = 32 / QL;
  constexpr int RS = TRANS ? 32 : 96, CS = TRANS ? 96 : 32;
  extern __shared__ __align__(16) unsigned char pt_smem[];
  __shared__ PtShared sh;
  const int threads = (int)blockDim.x;
  PtTeam tm{0, (int)gridDim.x, 0, 0u};
  int64_t t0 = 0, t1 = a.L.num_nodes;
  int job = 0;
  if (a.teams != nullptr) {
    tm.id = a.team_of_block[blockIdx.x];
    const PointTeam t = a.teams[tm.id];
    tm.first = t.first; tm.nb = t.nb; t0 = t.n0; t1 = t.n1; job = t.job;
  }
  // this block's units of NPW nodes: an equal share of the team's
  const int64_t tu = (t1 - t0 + NPW - 1) / NPW;
  const int64_t rank = (int)blockIdx.x - tm.first;
  const int64_t u0 = tu * rank / tm.nb, u1 = tu * (rank + 1) / tm.nb;
  PtLocal B;
  B.n0 = t0 + u0 * NPW;
  B.units = (int)(u1 - u0);
  B.nn = u1 > u0 ? (int)(min(t0 + u1 * NPW, t1) - B.n0) : 0;
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nn = B.nn, nd = 3 * nn;
  const int mw = a.precond == 2 ? 9 : (a.precond == 1 ? 3 : 0);
  double* r = reinterpret_cast<double*>(pt_smem);
  double *rhat = r + nd, *p = rhat + nd, *q = p + nd, *t = q + nd, *xs = t + nd, *ph = xs + nd, *sh_ = ph + nd;
  double* minv = sh_ + nd;
  if (threadIdx.x == 0) {
    sh.bad = 0;
    sh.steps = 0;
    if constexpr (kMg) sh.lb = mg_dense_from<MR>(mg);
  }
  __syncthreads();
  // slots per lane, and whether the block's rows fit beside the vectors
  for (int k = threadIdx.x; k < nn; k += threads)
    atomicMax(&sh.steps, (a.L.group_width[(B.n0 + k) >> 5] + QL - 1) / QL);
  __syncthreads();
  B.steps = sh.steps;
  const size_t vec_bytes = sizeof(double) * (8 * (size_t)nd + (size_t)mw * nn);
  const size_t items = (size_t)B.units * B.steps * 32;
  B.staged = vec_bytes + items * (9 * sizeof(double) + sizeof(int)) <= (size_t)a.smem_bytes;
  B.mat = reinterpret_cast<double*>(pt_smem + vec_bytes);
  B.cols = reinterpret_cast<int*>(B.mat + 9 * items);
  if (B.staged)
    for (int it = threadIdx.x; it < (int)items; it += threads) {
      const int ln = it & 31, us = it >> 5, u = us / B.steps, j = us - u * B.steps;
      const int k = u * NPW + ln % NPW, slot = ln / NPW + QL * j;
      const int64_t node = B.n0 + min(k, nn - 1);    // a lane past the end repeats the last node, with zeros
      const int64_t goff = a.L.group_off[node >> 5];
      int64_t col = node;
      double v[9] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
      if (k < nn && slot < a.L.group_width[node >> 5]) {
        col = a.L.cols[goff + 32 * slot + (node & 31)];
        const double* vb = pt_block<TRANS>(a, node, goff, slot);
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int c = 0; c < 3; ++c) v[3 * i + c] = __ldg(&vb[RS * i + CS * c]);
      }
      B.cols[it] = (int)(3 * col);
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int c = 0; c < 3; ++c) B.mat[((size_t)(3 * u + i) * B.steps + j) * 96 + 32 * c + ln] = v[3 * i + c];
    }
  // the preconditioner of the block's nodes, and x
  for (int k = threadIdx.x; k < nn; k += threads) {
    const int64_t node = B.n0 + k;
    if (mw) {
      const double* v0 = a.vals + 9 * a.L.group_off[node >> 5] + (node & 31) + 288 * (int64_t)a.L.diag_slot[node];
      if (mw == 3) {
#pragma unroll
        for (int i = 0; i < 3; ++i) minv[3 * k + i] = 1.0 / v0[32 * 4 * i];
      } else {
        double blk[9], bi[9];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int c = 0; c < 3; ++c) blk[TRANS ? 3 * c + i : 3 * i + c] = v0[32 * (3 * i + c)];
        inv3(blk, bi);
#pragma unroll
        for (int c = 0; c < 9; ++c) minv[9 * k + c] = bi[c];
      }
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) xs[3 * k + i] = a.x[3 * node + i];
  }
  __syncthreads();

  const int active = min(nd, threads);       // threads with a dof in the vector phases
  auto product = [&](const double* x, double* y) {
    if constexpr (kMg) pt_product_call<TRANS, QL, double>(a, B, x, y);
    else pt_product<TRANS, QL, false, double>(a, B, x, y);
  };
  // out = M v at the block's dofs, in global memory (for the neighbours) and in hat
  auto precond = [&](const double* v, double* hat, double* out) {
    if constexpr (kMg) {
      // t is free until the next product: the V-cycle's row sums
      __syncthreads();
      mg_vcycle<TRANS, QL, MR>(a, mg, B, v, hat, out, reinterpret_cast<MR*>(t), tm, sh);
      return;
    }
    if (mw == 9) __syncthreads();
    for (int d = threadIdx.x; d < nd; d += threads) {
      double o;
      if (mw == 0) o = v[d];
      else if (mw == 3) o = v[d] * minv[d];
      else {
        const int n = d / 3;
        o = fma(minv[3 * d], v[3 * n], fma(minv[3 * d + 1], v[3 * n + 1], minv[3 * d + 2] * v[3 * n + 2]));
      }
      hat[d] = o;
      out[3 * B.n0 + d] = o;
    }
  };
  // r = b - A x; rhat = p = q = r
  auto start = [&]() {
    product(a.x, t);
    double v2[2] = {0.0, 0.0};
    for (int d = threadIdx.x; d < nd; d += threads) {
      const double bv = a.b[3 * B.n0 + d];
      const double rv = bv - t[d];
      r[d] = rhat[d] = p[d] = q[d] = rv;
      v2[0] = fma(bv, bv, v2[0]);
      v2[1] = fma(rv, rv, v2[1]);
    }
    pt_reduce<2>(v2, active, tm, a, sh);   // b.b, r.r
  };
  // The scalars of the recurrence, its tests and its stop decision are thread 0's work, the
  // others read what they need from shared memory: a division in all 16 warps takes the FP64
  // pipe 1.1 us, a comparison 0.13 us.
  start();
  int restarts = 0;
  if (threadIdx.x == 0) {
    sh.atol2 = fmax(a.tol * a.tol * sh.sum[0], a.atol * a.atol);
    if (a.out != nullptr && (int)blockIdx.x == tm.first) a.out->bb = sh.sum[0];
    sh.rs = sh.rho_new = sh.beta = sh.sum[1];
    sh.rho = sh.alpha = sh.omega = 1.0;
    sh.k = 0;
    sh.go = pt_greater(sh.rs, sh.atol2) && a.maxiter > 0;
    sh.cap = 1e16 * fmax(sh.rs, sh.atol2);
    sh.drift = __longlong_as_double(0x7FF0000000000000ll);
  }
  __syncthreads();

  // restart at the x in global memory: rhat = p = q = r = b - A x
  auto restart = [&]() {
    ++restarts;
    start();
    if (threadIdx.x == 0) {
      sh.rs = sh.rho_new = sh.beta = sh.sum[1];
      sh.rho = sh.alpha = sh.omega = 1.0;
      sh.go = pt_greater(sh.rs, sh.atol2) && sh.k < a.maxiter;
    }
    __syncthreads();
  };

  double true_rs = -1.0;
  for (;;) {
    while (!sh.bad && sh.go) {
      {
        const double beta = sh.beta, omega = sh.omega;
        for (int d = threadIdx.x; d < nd; d += threads) p[d] = r[d] + beta * (p[d] - omega * q[d]);
      }
      precond(p, ph, a.phat);
      pt_reduce<0>(nullptr, active, tm, a, sh);
      product(a.phat, q);
      double v1[1] = {0.0};
      for (int d = threadIdx.x; d < nd; d += threads) v1[0] = fma(rhat[d], q[d], v1[0]);
      pt_reduce<1>(v1, active, tm, a, sh);
      if (threadIdx.x == 0) sh.alpha = sh.rho_new / sh.sum[0];
      __syncthreads();
      const double alpha = sh.alpha;
      // s = r - alpha q, kept in r; s.s joins the next sums
      double vt[3] = {0.0, 0.0, 0.0};
      for (int d = threadIdx.x; d < nd; d += threads) {
        const double sv = r[d] - alpha * q[d];
        r[d] = sv;
        vt[2] = fma(sv, sv, vt[2]);
      }
      precond(r, sh_, a.shat);
      pt_reduce<0>(nullptr, active, tm, a, sh);
      product(a.shat, t);
      for (int d = threadIdx.x; d < nd; d += threads) {
        vt[0] = fma(t[d], r[d], vt[0]);
        vt[1] = fma(t[d], t[d], vt[1]);
      }
      pt_reduce<3>(vt, active, tm, a, sh);
      if (threadIdx.x == 0) {
        sh.omega = sh.sum[0] / sh.sum[1];
        sh.early = pt_greater(sh.atol2, sh.sum[2]);
      }
      __syncthreads();
      const bool early = sh.early != 0;
      const double omega = sh.omega;
      double vr[2] = {0.0, 0.0};
      for (int d = threadIdx.x; d < nd; d += threads) {
        double rv;
        if (early) {
          xs[d] = xs[d] + alpha * ph[d];
          rv = r[d];
        } else {
          xs[d] = xs[d] + (alpha * ph[d] + omega * sh_[d]);
          rv = r[d] - omega * t[d];
        }
        r[d] = rv;
        vr[0] = fma(rv, rv, vr[0]);
        vr[1] = fma(rhat[d], rv, vr[1]);
      }
      pt_reduce<2>(vr, active, tm, a, sh);
      if (wid == 0) {
        // beta = rho_new / rho * alpha / omega, both quotients at once
        const double num = lane == 1 ? alpha : sh.sum[1], den = lane == 1 ? omega : sh.rho_new;
        const double f = num / den;
        const double g = __shfl_sync(0xffffffffu, f, 1);
        if (lane == 0) {
          int kn = (pt_zero(omega) || pt_zero(alpha)) ? -11 : sh.k + 1;
          if (pt_zero(sh.rho_new)) kn = -10;
          // an FP32 V-cycle cannot resolve the near-null modes of a near-singular system (its
          // rounding, amplified by the condition number, swamps them); a residual that grew by
          // 1e8 or went non-finite ends the solve with -12 so the caller can re-solve in FP64
          if (std::is_same<MR, float>::value && !pt_at_most(sh.sum[0], sh.cap)) kn = -12;
          sh.rho = sh.rho_new;
          sh.rs = sh.sum[0];
          sh.rho_new = sh.sum[1];
          sh.beta = f * g;
          const bool left = pt_greater(sh.rs, sh.atol2);
          sh.restart = kn < 0 && kn != -12 && restarts < a.max_restarts && left;
          sh.k = sh.restart ? sh.k + 1 : kn;
          sh.go = left && sh.k < a.maxiter && sh.k >= 0;
        }
      }
      __syncthreads();
      if (sh.restart && !sh.bad) {
        for (int d = threadIdx.x; d < nd; d += threads) a.x[3 * B.n0 + d] = xs[d];
        pt_reduce<0>(nullptr, active, tm, a, sh);
        restart();
      }
    }
    for (int d = threadIdx.x; d < nd; d += threads) a.x[3 * B.n0 + d] = xs[d];
    if (!(a.true_res || a.max_restarts > 0) || sh.bad) break;
    double vt[1] = {0.0};
    pt_reduce<0>(nullptr, active, tm, a, sh);
    product(a.x, t);
    for (int d = threadIdx.x; d < nd; d += threads) {
      const double rv = a.b[3 * B.n0 + d] - t[d];
      vt[0] = fma(rv, rv, vt[0]);
    }
    pt_reduce<1>(vt, active, tm, a, sh);
    true_rs = sh.sum[0];
    // Where restarts are allowed, a recursive residual that met the stop rule while the true one
    // is ten times above it (a near-singular system drives it through values so large that it
    // drifts from b - A x) is a breakdown too, as long as each such restart halves the true one:
    // below FP64's reach of the system they would go on to max_restarts for nothing (12^3 cells at
    // 1e-14: 428 iterations, 184 without).
    if (threadIdx.x == 0) {
      sh.restart = restarts < a.max_restarts && sh.k >= 0 && sh.k < a.maxiter && !pt_greater(sh.rs, sh.atol2) &&
                   pt_greater(true_rs, 100.0 * sh.atol2) && pt_greater(sh.drift, 4.0 * true_rs);
      sh.drift = true_rs;
    }
    __syncthreads();
    if (!sh.restart || sh.bad) break;
    restart();
  }
  if ((int)blockIdx.x == tm.first && threadIdx.x == 0) {
    if (a.out != nullptr) {
      a.out->true_rs = a.true_res ? true_rs : -1.0;
      a.out->restarts = restarts;
      a.out->k = sh.k;
      a.out->rs = sh.rs;
      a.out->atol2 = sh.atol2;
      a.out->rho = sh.rho;
      a.out->alpha = sh.alpha;
      a.out->omega = sh.omega;
    }
    if (a.info != nullptr) {
      a.info[2 * job] = sh.k;
      a.info[2 * job + 1] = (sh.rs <= sh.atol2) ? 1 : 0;
    }
  }
}

}  // namespace cpfem
