// Geometric multigrid V-cycle of the persistent BiCGSTAB (precond 3), in FP64 or FP32.
//
// Level 0 uses the Krylov kernel's own layout (rows by warps, own nodes in order), the coarser
// levels a quad of lanes per node spread over all blocks.  The coarse levels that are small
// enough (at most 256 nodes) are not smoothed during a solve at all: their whole part of the
// cycle -- down sweeps, coarsest sweeps, up sweeps, transfers among them -- is a linear map of
// their right-hand side, formed once per set-up as a dense operator and applied by all blocks
// in one phase.  (Smoothed inside one block they took 18-24 us of a 220 us iteration at
// 32^3, twice, and 21 us of 103 at 16^3; the dense phase takes 4.)
#pragma once

#include "krylov_team.cuh"

namespace cpfem {

// ---- geometric multigrid (precond 3) ------------------------------------------------
// Levels of a structured box of nodes, x fastest.  Fine node i of level l and coarse node
// I of level l+1 are linked when i is within one fine node of 2I in every direction, with
// the trilinear weight prod_d (1 if i_d = 2 I_d else 1/2).

__device__ __forceinline__ void mg_xyz(int64_t a, const int32_t* dims, int& x, int& y, int& z) {
  // node counts fit 32 bits (cpfem_sell_t.num_nodes is int32): 32-bit divisions
  const unsigned ua = (unsigned)a, d0 = (unsigned)dims[0], d1 = (unsigned)dims[1];
  const unsigned q = ua / d0;
  x = (int)(ua - q * d0);
  z = (int)(q / d1);
  y = (int)(q - (unsigned)z * d1);
}

// z = D^-1 v with the stored inverse diagonal block; TRANS uses its transpose, which is
// the inverse of the diagonal block of A^T.
template <bool TRANS, typename R>
__device__ __forceinline__ void mg_apply_minv(const R* __restrict__ minv, int64_t a, const R* v, R* out) {
  const R* bi = minv + 9 * a;
  if (TRANS) {
#pragma unroll
    for (int i = 0; i < 3; ++i) out[i] = mad(bi[i], v[0], mad(bi[3 + i], v[1], bi[6 + i] * v[2]));
  } else {
#pragma unroll
    for (int i = 0; i < 3; ++i) out[i] = mad(bi[3 * i], v[0], mad(bi[3 * i + 1], v[1], bi[3 * i + 2] * v[2]));
  }
}

// Rows of node a of A x (A^T x when TRANS) restricted to the slots j = q (mod 4) (one lane of
// a quad).  x by plain loads: shared memory, or global memory whose writers the grid's last
// barrier ordered (neighbours share values, which L1 then serves).
template <bool TRANS, typename R>
__device__ __forceinline__ void sell_rows_quad(const cpfem_sell_t& L, const R* __restrict__ vals, const R* x,
                                               int64_t a, int q, R* acc) {
  const int64_t g = a >> 5;
  const int lane = (int)(a & 31);
  const int64_t c0 = L.group_off[g] + lane;
  const R* v0 = vals + 9 * L.group_off[g] + lane;
  const int w = L.group_width[g];
  R a0 = R(0), a1 = R(0), a2 = R(0);
#pragma unroll 2
  for (int j = q; j < w; j += 4) {
    const int64_t b = __ldg(&L.cols[c0 + 32 * j]);
    const R x0 = x[3 * b], x1 = x[3 * b + 1], x2 = x[3 * b + 2];
    if (!TRANS) {
      const R* vb = v0 + 288 * j;
      a0 = mad(__ldg(&vb[0]), x0, mad(__ldg(&vb[32]), x1, mad(__ldg(&vb[64]), x2, a0)));
      a1 = mad(__ldg(&vb[96]), x0, mad(__ldg(&vb[128]), x1, mad(__ldg(&vb[160]), x2, a1)));
      a2 = mad(__ldg(&vb[192]), x0, mad(__ldg(&vb[224]), x1, mad(__ldg(&vb[256]), x2, a2)));
    } else {
      const int64_t tp = __ldg(&L.tpos[c0 + 32 * j]);
      const R* vb = vals + 9 * L.group_off[b >> 5] + (b & 31) + 288 * tp;
      a0 = mad(__ldg(&vb[0]), x0, mad(__ldg(&vb[96]), x1, mad(__ldg(&vb[192]), x2, a0)));
      a1 = mad(__ldg(&vb[32]), x0, mad(__ldg(&vb[128]), x1, mad(__ldg(&vb[224]), x2, a1)));
      a2 = mad(__ldg(&vb[64]), x0, mad(__ldg(&vb[160]), x1, mad(__ldg(&vb[256]), x2, a2)));
    }
  }
  acc[0] = a0;
  acc[1] = a1;
  acc[2] = a2;
}

constexpr int kMgMaxWidth = 27;                 // neighbour slots of a structured-box node

// Staged (shared-memory) copies of a block-local level are skewed: the four lanes of a
// node's quad read four consecutive slots, whose sliced-ELL rows (288 values, or 32 index
// entries) start in the same bank, so every slot row is followed by 8 unused words.  Lanes
// (node k, slot phase q) of a warp then read bank k + 8q: no bank conflicts.
constexpr int64_t kStSkew = 8;
__host__ __device__ constexpr int64_t st_val_index(int64_t i) { return i + kStSkew * (i / 288); }
__host__ __device__ constexpr int64_t st_idx_index(int64_t i) { return i + kStSkew * (i >> 5); }
constexpr int64_t kStValRow = 288 + kStSkew, kStIdxRow = 32 + kStSkew;

// sell_rows_quad on a level staged in shared memory: values, x and the index tables
// (group offsets, widths and columns as int32, mg_stage) all there, the values and the columns in
// the skewed order above (group offsets are multiples of 32 slots, so a group's rows start at a
// whole skewed row).
template <typename R>
__device__ __forceinline__ void sell_rows_quad_st(const int* ix, int ng, const R* vals, const R* x, int64_t a,
                                                  int q, R* acc) {
  const int* goff = ix;
  const int* gw = ix + ng + 1;
  const int* cols = gw + ng;
  const int g = (int)(a >> 5);
  const int lane = (int)(a & 31);
  const int gs = goff[g];
  const int c0 = gs + (int)kStSkew * (gs >> 5) + lane;               // st_idx_index(gs + lane)
  const R* v0 = vals + 9 * gs + (int)kStSkew * (gs >> 5) + lane;     // st_val_index(9 gs + lane)
  const int w = gw[g];
  R a0 = R(0), a1 = R(0), a2 = R(0);
#pragma unroll 2
  for (int j = q; j < w; j += 4) {
    const int b = cols[c0 + (int)kStIdxRow * j];
    const R x0 = x[3 * b], x1 = x[3 * b + 1], x2 = x[3 * b + 2];
    const R* vb = v0 + kStValRow * j;
    a0 = mad(vb[0], x0, mad(vb[32], x1, mad(vb[64], x2, a0)));
    a1 = mad(vb[96], x0, mad(vb[128], x1, mad(vb[160], x2, a1)));
    a2 = mad(vb[192], x0, mad(vb[224], x1, mad(vb[256], x2, a2)));
  }
  acc[0] = a0;
  acc[1] = a1;
  acc[2] = a2;
}

// The arrays of a V-cycle in precision R: FP64 uses the hierarchy's own operators (level
// 0: the system's values), FP32 the single-precision copies cpfem_mg_setup makes.
template <typename R>
struct MgArrays;
template <>
struct MgArrays<double> {
  const cpfem_mg_t& m;
  const double* v0;
  __device__ __forceinline__ const double* values(int l) const { return l == 0 ? v0 : m.values[l]; }
  __device__ __forceinline__ const double* minv(int l) const { return m.minv[l]; }
  __device__ __forceinline__ double* x(int l) const { return m.x[l]; }
  __device__ __forceinline__ double* t(int l) const { return m.t[l]; }
  __device__ __forceinline__ double* r(int l) const { return m.r[l]; }
  __device__ __forceinline__ double* b(int l) const { return m.b[l]; }
};
template <>
struct MgArrays<float> {
  const cpfem_mg_t& m;
  const double* v0;
  __device__ __forceinline__ const float* values(int l) const { return m.values32[l]; }
  __device__ __forceinline__ const float* minv(int l) const { return m.minv32[l]; }
  __device__ __forceinline__ float* x(int l) const { return m.x32[l]; }
  __device__ __forceinline__ float* t(int l) const { return m.t32[l]; }
  __device__ __forceinline__ float* r(int l) const { return m.r32[l]; }
  __device__ __forceinline__ float* b(int l) const { return m.b32[l]; }
};

template <typename R>
__device__ __forceinline__ void quad_sum3(R* v) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    v[i] += __shfl_xor_sync(0xffffffffu, v[i], 1);
    v[i] += __shfl_xor_sync(0xffffffffu, v[i], 2);
  }
}

// Level operations of the V-cycle on a coarse level (l >= 1), one quad of lanes per node:
// nodes a = tq, tq + sq, ... (tq = this lane's quad, sq = the quads taking part; a warp
// holds 8 consecutive quads and runs the padded loops in lockstep, so the shuffles always
// see the whole warp); lane 0 of a node's quad owns its writes.  The level's vectors are
// passed explicitly: global arrays in a solve, shared memory in mg_dense_setup.
template <bool TRANS, typename R>
__device__ __forceinline__ void mgq_first_sweep(const cpfem_mg_t& mg, const R* Mi, int l, R* X, const R* B,
                                                int64_t tq, int64_t sq, int q) {
  if (q != 0) return;
  const R om = (R)mg.omega;
  for (int64_t a = tq; a < mg.sell[l].num_nodes; a += sq) {
    R v[3] = {B[3 * a], B[3 * a + 1], B[3 * a + 2]}, z[3];
    mg_apply_minv<TRANS>(Mi, a, v, z);
#pragma unroll
    for (int i = 0; i < 3; ++i) X[3 * a + i] = om * z[i];
  }
}

// T = X + omega Minv (B - A X)  (residual = false)  or  T = B - A X  (residual = true)
template <bool TRANS, bool SHV = false, typename R>
__device__ __forceinline__ void mgq_apply(const cpfem_mg_t& mg, const R* V, const R* Mi, int l, const R* X, R* T,
                                          const R* B, bool residual, int64_t tq, int64_t sq, int q,
                                          const int* sidx = nullptr) {
  const cpfem_sell_t& S = mg.sell[l];
  const R om = (R)mg.omega;
  const int64_t n = S.num_nodes, npad = (n + 7) / 8 * 8;
  for (int64_t a = tq; a < npad; a += sq) {
    R acc[3] = {R(0), R(0), R(0)};
    if (a < n) {
      if constexpr (SHV) sell_rows_quad_st(sidx, S.num_groups, V, X, a, q, acc);
      else sell_rows_quad<TRANS, R>(S, V, X, a, q, acc);
    }
    quad_sum3(acc);
    if (a < n && q == 0) {
      R r[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) r[i] = B[3 * a + i] - acc[i];
      if (residual) {
#pragma unroll
        for (int i = 0; i < 3; ++i) T[3 * a + i] = r[i];
      } else {
        R z[3];
        mg_apply_minv<TRANS>(Mi, a, r, z);
#pragma unroll
        for (int i = 0; i < 3; ++i) T[3 * a + i] = mad(om, z[i], X[3 * a + i]);
      }
    }
  }
}

// Bc = P^T Res_l (the level l+1 right-hand side): the 27 fine nodes of a coarse node
// split over its quad.
template <typename R>
__device__ __forceinline__ void mgq_restrict(const cpfem_mg_t& mg, int l, const R* Res, R* Bc, int64_t tq,
                                             int64_t sq, int q) {
  const int32_t* df = mg.dims[l];
  const int32_t* dc = mg.dims[l + 1];
  const int64_t nc = mg.sell[l + 1].num_nodes, ncpad = (nc + 7) / 8 * 8;
  for (int64_t I = tq; I < ncpad; I += sq) {
    R acc[3] = {R(0), R(0), R(0)};
    if (I < nc) {
      int cx, cy, cz;
      mg_xyz(I, dc, cx, cy, cz);
      // the lane's fine neighbours k = q, q+4, ... < 27, unrolled and predicated (an absent
      // neighbour reads node 0 with weight 0), so all their loads are in flight together
#pragma unroll
      for (int kk = 0; kk < 7; ++kk) {
        const int k = q + 4 * kk;
        const int dz = k / 9 - 1, dy = (k / 3) % 3 - 1, dx = k % 3 - 1;
        const int ix = 2 * cx + dx, iy = 2 * cy + dy, iz = 2 * cz + dz;
        const bool in = k < 27 && ix >= 0 && ix < df[0] && iy >= 0 && iy < df[1] && iz >= 0 && iz < df[2];
        const R w = in ? (dx ? R(0.5) : R(1)) * (dy ? R(0.5) : R(1)) * (dz ? R(0.5) : R(1)) : R(0);
        const int64_t i = in ? ix + (int64_t)df[0] * (iy + (int64_t)df[1] * iz) : 0;
#pragma unroll
        for (int c = 0; c < 3; ++c) acc[c] = mad(w, Res[3 * i + c], acc[c]);
      }
    }
    quad_sum3(acc);
    if (I < nc && q == 0)
#pragma unroll
      for (int c = 0; c < 3; ++c) Bc[3 * I + c] = acc[c];
  }
}

// X_l += P X_{l+1} at the nodes a = first, first + step, ... < end (masked on Dirichlet dofs of
// level 0).
template <typename R>
__device__ __forceinline__ void mg_prolong(const cpfem_mg_t& mg, int l, R* X, const R* Xc, int64_t first,
                                           int64_t step, int64_t end) {
  const int32_t* df = mg.dims[l];
  const int32_t* dc = mg.dims[l + 1];
  for (int64_t a = first; a < end; a += step) {
    int ix, iy, iz;
    mg_xyz(a, df, ix, iy, iz);
    const int cx0 = ix >> 1, cy0 = iy >> 1, cz0 = iz >> 1;
    const int nxc = (ix & 1) + 1, nyc = (iy & 1) + 1, nzc = (iz & 1) + 1;
    const R w = ((ix & 1) ? R(0.5) : R(1)) * ((iy & 1) ? R(0.5) : R(1)) * ((iz & 1) ? R(0.5) : R(1));
    R acc[3] = {R(0), R(0), R(0)};
    // the 1, 2, 4 or 8 coarse parents, unrolled over 2x2x2 and predicated (an absent one
    // reads its first parent with weight 0), so all their loads are in flight together
#pragma unroll
    for (int kz = 0; kz < 2; ++kz)
#pragma unroll
      for (int ky = 0; ky < 2; ++ky)
#pragma unroll
        for (int kx = 0; kx < 2; ++kx) {
          const bool in = kx < nxc && ky < nyc && kz < nzc;
          const int64_t I = (cx0 + (in ? kx : 0)) +
                            (int64_t)dc[0] * ((cy0 + (in ? ky : 0)) + (int64_t)dc[1] * (cz0 + (in ? kz : 0)));
          const R wk = in ? w : R(0);
#pragma unroll
          for (int c = 0; c < 3; ++c) acc[c] = mad(wk, Xc[3 * I + c], acc[c]);
        }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const bool fixed = (l == 0 && mg.free_dof != nullptr && mg.free_dof[3 * a + c] == 0);
      if (!fixed) X[3 * a + c] += acc[c];
    }
  }
}

constexpr int kMgDenseNodes = 256;   // largest level that becomes a dense operator

// What the dense operator in scratch[0] belongs to and was formed with: written in front of it by
// the set-up, checked by a solve, which smooths the levels itself where it does not match (the
// smoother's settings may change between set-up and solve: those levels then follow them as the
// others do).  The Galerkin passes of
// every set-up write scratch[0] from its first element on, so a set-up of any size that uses the
// same scratch, one that forms no dense operator too, takes the tag of the one before away.
struct MgTag {
  unsigned long long magic;
  const void* minv;
  long long omega;       // its bits
  int levels, level, nodes, real_bytes, pre_sweeps, post_sweeps, coarse_sweeps, pad;
};
constexpr unsigned long long kMgTagMagic = 0x6D67636F61727365ull;
constexpr size_t kMgTagBytes = 64;
static_assert(sizeof(MgTag) <= kMgTagBytes, "the tag fits in front of the operator");

// The first level of the dense part (num_levels: none): the coarsest levels, from level 1 on,
// with at most local_nodes (0: 256, and never more than 256) nodes, whose operator and tag fit
// in scratch[0].
__host__ __device__ inline int mg_dense_level(const cpfem_mg_t& mg, size_t real_bytes) {
  const int64_t most = mg.local_nodes > 0 && mg.local_nodes < kMgDenseNodes ? mg.local_nodes : kMgDenseNodes;
  int lb = mg.num_levels;
  for (int l = mg.num_levels - 1; l >= 1 && mg.sell[l].num_nodes <= most; --l) {
    const size_t n = 3 * (size_t)mg.sell[l].num_nodes;
    if (n * n * real_bytes + kMgTagBytes > sizeof(double) * 243 * (size_t)mg.scratch_nodes) break;
    lb = l;
  }
  return lb;
}

template <typename R>
__host__ __device__ inline R* mg_dense(const cpfem_mg_t& mg) {
  return reinterpret_cast<R*>(reinterpret_cast<char*>(mg.scratch[0]) + kMgTagBytes);
}
__host__ __device__ inline MgTag* mg_tag(const cpfem_mg_t& mg) { return reinterpret_cast<MgTag*>(mg.scratch[0]); }
template <typename R>
__device__ __forceinline__ MgTag mg_tag_of(const cpfem_mg_t& mg, const R* minv, int lb) {
  return MgTag{kMgTagMagic, minv, __double_as_longlong(mg.omega), mg.num_levels, lb, (int)mg.sell[lb].num_nodes, (int)sizeof(R),
               mg.pre_sweeps, mg.post_sweeps, mg.coarse_sweeps, 0};
}
__device__ __forceinline__ bool mg_tag_same(const MgTag& a, const MgTag& b) {
  // no short circuits: the loads together
  return (a.magic == b.magic) & (a.minv == b.minv) & (a.omega == b.omega) & (a.levels == b.levels) &
         (a.level == b.level) & (a.nodes == b.nodes) & (a.real_bytes == b.real_bytes) & (a.pre_sweeps == b.pre_sweeps) &
         (a.post_sweeps == b.post_sweeps) & (a.coarse_sweeps == b.coarse_sweeps);
}

// The first level that this solve applies as the dense operator (num_levels: none is there for it).
template <typename R>
__device__ __forceinline__ int mg_dense_from(const cpfem_mg_t& mg) {
  const int lb = mg_dense_level(mg, sizeof(R));
  if (lb >= mg.num_levels) return mg.num_levels;
  return mg_tag_same(*mg_tag(mg), mg_tag_of<R>(mg, MgArrays<R>{mg, nullptr}.minv(lb), lb)) ? lb : mg.num_levels;
}

constexpr size_t kMgStageBytes = 220 * 1024;    // shared memory of a dense set-up's block, at most

// Shared memory of the levels lb .. L-1, in elements of R: x, t, r, b of each level (3
// values per node) and, when everything fits in kMgStageBytes and the V-cycle is FP32, the
// levels' operators (sliced-ELL, at most kMgMaxWidth slots per node) and inverse diagonal
// blocks, staged once per launch.  Host and device derive the same layout.
struct MgShared {
  size_t vec[CPFEM_MG_MAX_LEVELS];
  size_t val[CPFEM_MG_MAX_LEVELS];
  size_t minv[CPFEM_MG_MAX_LEVELS];
  size_t idx[CPFEM_MG_MAX_LEVELS];   // int32: group offsets, group widths, columns
  size_t total;
  bool staged;
};

// int32 entries of a staged level's layout: ng+1 group offsets, ng widths, and the columns of
// 32 * kMgMaxWidth slots per group (skewed: kStIdxRow words per slot row)
__host__ __device__ inline size_t mg_idx_words(int32_t ng) {
  return 2 * (size_t)ng + 1 + (size_t)kStIdxRow * (size_t)kMgMaxWidth * ng;
}

__host__ __device__ inline MgShared mg_shared_layout(const cpfem_mg_t& mg, int lb, size_t real_bytes) {
  MgShared s{};
  size_t off = 0;
  for (int m = lb; m < mg.num_levels; ++m) {
    s.vec[m] = off;
    off += 12 * (size_t)mg.sell[m].num_nodes;
  }
  size_t off_v = off;
  for (int m = lb; m < mg.num_levels; ++m) {
    s.val[m] = off_v;
    off_v += (size_t)kStValRow * (size_t)kMgMaxWidth * (size_t)mg.sell[m].num_groups;
    s.minv[m] = off_v;
    off_v += 9 * (size_t)mg.sell[m].num_nodes;
    s.idx[m] = off_v;   // in 4-byte words, which the staged (FP32) layout's elements are
    off_v += mg_idx_words(mg.sell[m].num_groups);
  }
  s.staged = real_bytes == sizeof(float) && lb < mg.num_levels && off_v * real_bytes <= kMgStageBytes;
  s.total = (s.staged ? off_v : off) * real_bytes;
  return s;
}

extern __shared__ __align__(16) unsigned char mg_shared[];

// Once per block: the levels' operators and inverse diagonal blocks to shared memory (when the
// layout stages them).
// Returns whether they were staged (every level within kMgMaxWidth slots per node).
template <typename R>
__device__ bool mg_stage(const cpfem_mg_t& mg, int lb, const MgArrays<R>& A, const MgShared& lay) {
  if (!lay.staged) return false;
  for (int m = lb; m < mg.num_levels; ++m)
    if (mg.sell[m].group_off[mg.sell[m].num_groups] > 32 * (int64_t)kMgMaxWidth * mg.sell[m].num_groups) return false;
  R* sh = reinterpret_cast<R*>(mg_shared);
  for (int m = lb; m < mg.num_levels; ++m) {
    const cpfem_sell_t& S = mg.sell[m];
    const int64_t nv = 9 * S.group_off[S.num_groups];
    const R* V = A.values(m);
    const R* Mi = A.minv(m);
    for (int64_t i = threadIdx.x; i < nv; i += blockDim.x) sh[lay.val[m] + st_val_index(i)] = V[i];
    for (int64_t i = threadIdx.x; i < 9 * (int64_t)S.num_nodes; i += blockDim.x) sh[lay.minv[m] + i] = Mi[i];
    int* ix = reinterpret_cast<int*>(sh + lay.idx[m]);
    const int ng = S.num_groups;
    const int64_t ns = S.group_off[ng];
    int* cols = ix + 2 * ng + 1;
    for (int64_t i = threadIdx.x; i <= ng; i += blockDim.x) ix[i] = (int)S.group_off[i];
    for (int64_t i = threadIdx.x; i < ng; i += blockDim.x) ix[ng + 1 + i] = S.group_width[i];
    for (int64_t i = threadIdx.x; i < ns; i += blockDim.x) cols[st_idx_index(i)] = S.cols[i];
  }
  __syncthreads();
  return true;
}

// The levels lb .. L-1 of one block on its shared memory: vec(lb, 3) holds level lb's
// right-hand side; returns where its iterate ends up.  SHV: the operators were staged.
template <bool SHV, typename R>
__device__ R* mg_local_cycle(const cpfem_mg_t& mg, const MgArrays<R>& A, const MgShared& lay, int lb) {
  const int L = mg.num_levels, q = (int)(threadIdx.x & 3);
  const int64_t tqb = threadIdx.x >> 2, sqb = blockDim.x >> 2;   // block-local quads
  R* sh = reinterpret_cast<R*>(mg_shared);
  auto vec = [&](int m, int k) { return sh + lay.vec[m] + (size_t)k * 3 * mg.sell[m].num_nodes; };  // x t r b
  auto V = [&](int m) { return SHV ? (const R*)(sh + lay.val[m]) : A.values(m); };
  auto Mi = [&](int m) { return SHV ? (const R*)(sh + lay.minv[m]) : A.minv(m); };
  auto Ix = [&](int m) { return SHV ? reinterpret_cast<const int*>(sh + lay.idx[m]) : (const int*)nullptr; };
  R* at[CPFEM_MG_MAX_LEVELS];
  for (int m = lb; m < L; ++m) {
    R* Xm = vec(m, 0);
    R* Tm = vec(m, 1);
    mgq_first_sweep<false>(mg, Mi(m), m, Xm, vec(m, 3), tqb, sqb, q);
    const int nsw = (m == L - 1) ? mg.coarse_sweeps : mg.pre_sweeps;
    for (int k = 1; k < nsw; ++k) {
      __syncthreads();
      mgq_apply<false, SHV>(mg, V(m), Mi(m), m, Xm, Tm, vec(m, 3), false, tqb, sqb, q, Ix(m));
      R* tmp = Xm; Xm = Tm; Tm = tmp;
    }
    at[m] = Xm;
    if (m == L - 1) break;
    __syncthreads();
    mgq_apply<false, SHV>(mg, V(m), Mi(m), m, Xm, vec(m, 2), vec(m, 3), true, tqb, sqb, q, Ix(m));
    __syncthreads();
    mgq_restrict(mg, m, vec(m, 2), vec(m + 1, 3), tqb, sqb, q);
  }
  for (int m = L - 2; m >= lb; --m) {
    R* Xm = at[m];
    R* Tm = (Xm == vec(m, 0)) ? vec(m, 1) : vec(m, 0);
    __syncthreads();
    if (q == 0) mg_prolong(mg, m, Xm, (const R*)at[m + 1], tqb, sqb, mg.sell[m].num_nodes);
    for (int k = 0; k < mg.post_sweeps; ++k) {
      __syncthreads();
      mgq_apply<false, SHV>(mg, V(m), Mi(m), m, Xm, Tm, vec(m, 3), false, tqb, sqb, q, Ix(m));
      R* tmp = Xm; Xm = Tm; Tm = tmp;
    }
    at[m] = Xm;
  }
  __syncthreads();
  return at[lb];
}

// Levels 1 .. L-1 of a V-cycle.  Level 0's residual is complete in A.r(0); the iterate of level 1
// that is returned is complete after the caller's next barrier.  tq, sq, q as in mgq_apply; rank of
// nb blocks; b: room for 3 kMgDenseNodes values in shared memory.
template <bool TRANS, typename R, class Barrier>
__device__ __forceinline__ const R* mg_coarse_levels(const cpfem_mg_t& mg, const MgArrays<R>& A, int lb, int64_t tq,
                                                     int64_t sq, int q, int rank, int nb, R* b, Barrier barrier) {
  const int L = mg.num_levels;
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = (int)blockDim.x >> 5;
  R* at[CPFEM_MG_MAX_LEVELS];
  // ---- levels 1 .. lb-1, down
  for (int l = 1; l < lb; ++l) {
    const R* V = A.values(l);
    const R* Mi = A.minv(l);
    R *X = A.x(l), *T = A.t(l);
    mgq_restrict(mg, l - 1, (const R*)A.r(l - 1), A.b(l), tq, sq, q);
    mgq_first_sweep<TRANS>(mg, Mi, l, X, (const R*)A.b(l), tq, sq, q);
    const int nsw = (l == L - 1) ? mg.coarse_sweeps : mg.pre_sweeps;
    for (int k = 1; k < nsw; ++k) {
      barrier();
      mgq_apply<TRANS>(mg, V, Mi, l, (const R*)X, T, (const R*)A.b(l), false, tq, sq, q);
      R* tmp = X; X = T; T = tmp;
    }
    at[l] = X;
    if (l == L - 1) break;
    barrier();
    mgq_apply<TRANS>(mg, V, Mi, l, (const R*)X, A.r(l), (const R*)A.b(l), true, tq, sq, q);
    barrier();
  }
  // ---- levels lb .. L-1: the dense operator.  Every block restricts the whole right-hand side
  // (a few KB of residual, L1's work) rather than wait for its parts; a warp per row.
  if (lb < L) {
    mgq_restrict(mg, lb - 1, (const R*)A.r(lb - 1), b, threadIdx.x >> 2, blockDim.x >> 2, q);
    __syncthreads();
    const int N = 3 * (int)mg.sell[lb].num_nodes;
    const R* K = mg_dense<R>(mg);
    R* X = A.x(lb);
    const int r1 = (int)((int64_t)N * (rank + 1) / nb);
    for (int row = (int)((int64_t)N * rank / nb) + wid; row < r1; row += warps) {
      R acc = R(0);
#pragma unroll 4
      for (int c = lane; c < N; c += 32)
        acc = mad(TRANS ? __ldg(&K[(size_t)c * N + row]) : __ldg(&K[(size_t)row * N + c]), b[c], acc);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (lane == 0) X[row] = acc;
    }
    at[lb] = X;
  }
  // ---- levels below the coarsest, up
  for (int l = (lb < L ? lb : L - 1) - 1; l >= 1; --l) {
    const R* V = A.values(l);
    const R* Mi = A.minv(l);
    R* X = at[l];
    R* T = (X == A.x(l)) ? A.t(l) : A.x(l);
    barrier();
    if (q == 0) mg_prolong(mg, l, X, (const R*)at[l + 1], tq, sq, mg.sell[l].num_nodes);
    for (int k = 0; k < mg.post_sweeps; ++k) {
      barrier();
      mgq_apply<TRANS>(mg, V, Mi, l, (const R*)X, T, (const R*)A.b(l), false, tq, sq, q);
      R* tmp = X; X = T; T = tmp;
    }
    at[l] = X;
  }
  return at[1];
}

// One V-cycle hat = out = M^-1 v: v and hat are the block's dofs of FP64 vectors, out the global
// vector that neighbours gather, y room for the block's row sums.
template <bool TRANS, int QL, typename R>
__device__ __noinline__ void mg_vcycle(const PointArgs& a, const cpfem_mg_t& mg, const PtLocal& B, const double* v, double* hat,
                          double* out, R* y, PtTeam& tm, PtShared& sh) {
  const MgArrays<R> A{mg, a.vals};
  const R om = (R)mg.omega;
  const int threads = (int)blockDim.x, wid = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = threads >> 5;
  const int rank = (int)blockIdx.x - tm.first, nn = B.nn;
  const int64_t n0 = B.n0;
  // the coarse levels' nodes go to the warps of all blocks in turn, eight to a warp
  const int q = lane & 3;
  const int64_t tq = 8 * ((int64_t)wid * tm.nb + rank) + (lane >> 2), sq = 8 * (int64_t)warps * tm.nb;
  auto barrier = [&]() { pt_reduce<0>(nullptr, 0, tm, a, sh); };
  const R* Mi0 = A.minv(0);
  // one sweep of level 0 after its row sums: f(node, X + om D^-1 (v - A X))
  auto sweep0 = [&](const R* X, auto&& f) {
    pt_product_call<TRANS, QL, R>(a, B, X, y);
    for (int n = threadIdx.x; n < nn; n += threads) {
      R r[3], z[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) r[i] = to_prec<R>(v[3 * n + i]) - y[3 * n + i];
      mg_apply_minv<TRANS>(Mi0, n0 + n, r, z);
#pragma unroll
      for (int i = 0; i < 3; ++i) z[i] = mad(om, z[i], X[3 * (n0 + n) + i]);
      f(n, z);
    }
  };
  R* at0;
  // ---- level 0, down
  {
    R *X = A.x(0), *T = A.t(0);
    for (int n = threadIdx.x; n < nn; n += threads) {
      R r[3], z[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) r[i] = to_prec<R>(v[3 * n + i]);
      mg_apply_minv<TRANS>(Mi0, n0 + n, r, z);
#pragma unroll
      for (int i = 0; i < 3; ++i) X[3 * (n0 + n) + i] = om * z[i];
    }
    for (int k = 1; k < mg.pre_sweeps; ++k) {
      barrier();
      sweep0(X, [&](int n, const R* z) {
#pragma unroll
        for (int i = 0; i < 3; ++i) T[3 * (n0 + n) + i] = z[i];
      });
      R* tmp = X; X = T; T = tmp;
    }
    barrier();
    pt_product_call<TRANS, QL, R>(a, B, X, y);
    R* Res = A.r(0);
    for (int d = threadIdx.x; d < 3 * nn; d += threads) {
      const R rv = to_prec<R>(v[d]) - y[d];
      Res[3 * n0 + d] = (mg.free_dof != nullptr && mg.free_dof[3 * n0 + d] == 0) ? R(0) : rv;
    }
    barrier();
    at0 = X;
  }
  static_assert(sizeof(sh.part) >= sizeof(double) * 3 * kMgDenseNodes, "the dense right-hand side fits");
  const R* X1 = mg_coarse_levels<TRANS, R>(mg, A, sh.lb, tq, sq, q, rank, tm.nb, reinterpret_cast<R*>(sh.part), barrier);
  // ---- level 0, up
  {
    R* X = at0;
    R* T = (X == A.x(0)) ? A.t(0) : A.x(0);
    barrier();
    mg_prolong(mg, 0, X, X1, n0 + threadIdx.x, threads, n0 + nn);
    auto finish = [&](int n, const R* z) {
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const double o = to_f64(z[i]);
        hat[3 * n + i] = o;
        out[3 * (n0 + n) + i] = o;
      }
    };
    for (int k = 0; k < mg.post_sweeps; ++k) {
      barrier();
      if (k + 1 < mg.post_sweeps) {
        sweep0(X, [&](int n, const R* z) {
#pragma unroll
          for (int i = 0; i < 3; ++i) T[3 * (n0 + n) + i] = z[i];
        });
        R* tmp = X; X = T; T = tmp;
      } else {
        sweep0(X, finish);
      }
    }
    if (mg.post_sweeps == 0)
      for (int n = threadIdx.x; n < nn; n += threads) finish(n, X + 3 * (n0 + n));
  }
}

}  // namespace cpfem
