// sm_100a kernels of the supernodal left-looking Bunch-Kaufman LDL^T factor.
//
// Data layout in HBM (one pool per factor handle, offsets fixed at analysis):
//   panel[s]  : nrow_s x ncol_s column-major (stride nrow_s) at poff[s]; after
//               the factor rows/cols are in the panel's pivot order, the
//               strictly-lower part holds L (zero at a 2x2's coupling entry,
//               whose d21 is in dsub), the diagonal holds D.
//   e-indexed : d[n], dsub[n], kind[n] (0 = 1x1, 1/2 = first/second column of
//               a 2x2 block), lperm[n] (pivot position -> pre-pivot local
//               column) — e = first_col(s) + pivot position.
// Kernels (one level of the assembly tree per launch group):
//   k_assemble      scatter-add of the equilibrated A (precomputed targets)
//   k_cmod          tile-owner gather of every descendant update (deterministic
//                   updater order, no atomics) — ll_factor_node cmod
//   k_getf2, k_deep (panel.cuh)  panel-bounded BK on one nb-wide block and its
//                   deep rows — ll_cdiv_emit getf2, apply_bk_panel_trailing
//   k_schur         deferred in-panel Schur update of the remaining columns
// Reference: src/numeric/multifrontal_ldlt.rs:2400-3256, 1347-1408.
#pragma once

#include "async_copy.cuh"
#include "scalar.cuh"

namespace rsd {

constexpr int TILE = 64;      // output tile edge of the GEMM-class kernels
constexpr int TPB = 256;      // threads per CTA of the GEMM-class kernels
// Deep rows that getf2 solves itself, for blocks of at most FUSE_PW columns:
// two passes of its eight warps (10 us) against a launch of k_deep (about 8 us
// with the launch); 192 rows took six.  A pass over 128 columns takes 45 us
// (c32), so wider blocks always leave them to k_deep.  On the two warps of the
// narrow instance the same rows are eight passes (32 columns, f64: 14 to 18
// us), which counts only where its launch has few blocks; launches that fill
// the GPU with narrow blocks save the second reading of L.
constexpr int FUSE_DEEP_ROWS = 64, FUSE_PW = 64;
constexpr int EA_ROWS = 1024;        // front rows per extend-add task
struct FactorArgs {
  // structure (device)
  const int* sn_first;
  const int* sn_ncol;
  const int* sn_nrow;
  const long long* sn_poff;
  const long long* sn_rsoff;
  const int* rs;
  const int* upd_ptr;
  const int* upd_k;
  const int* upd_p0;
  const int* upd_p1;
  // numeric state
  void* panel;
  void* d;
  void* dsub;
  unsigned char* kind;
  int* lperm;
  int* status;          // [0] = error code, [1] = first failing supernode, [2] = n_perturbed
  double perturb_floor; // < 0: exact mode
  void* gpool;          // G_k = L21_k D_k, (nrow_k - ncol_k) x ncol_k at goff[k] (tensor-core cmod)
  const long long* goff;
  const double* floor_dev;  // non-null: static-pivot floor computed on the device (force-accept)
  // Multifrontal variant: the contribution blocks of the fronts, supernode
  // s's (nrow - ncol)^2 column-major block at cb_off[s].
  void* cbpool;
  const long long* cb_off;
  // Pivot record (e-indexed, block-local): kp for a 1x1 step at e, -(kp + 1)
  // for a 2x2 step starting at e.  Written by every factor that searches; when
  // *pivot_reuse is set, getf2 replays the recorded steps instead of searching
  // (static pivot reuse across a value sweep of one pattern).
  int* pivrec;
  const int* pivot_reuse;
};

// ---------------------------------------------------------------------------
// Equilibration + assembly.
// ---------------------------------------------------------------------------

// Row maxima of |A| over the stored lower triangle, both triangles counted
// (onepass_scale, src/numeric/sparse_solver.rs:399-421).  Non-negative
// doubles order like their bit patterns, so atomicMax on the bits is exact
// and order independent.
template <typename T>
__global__ void k_rowmax(long long nnz, const int* __restrict__ row, const int* __restrict__ col,
                         const T* __restrict__ val, unsigned long long* __restrict__ rmax) {
  long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (k >= nnz) return;
  double m = Field<T>::mag(val[k]);
  unsigned long long b = __double_as_longlong(m);
  int i = row[k], j = col[k];
  atomicMax(&rmax[i], b);
  if (i != j) atomicMax(&rmax[j], b);
}

// s_i = 1/sqrt(rowmax_i), guarded (src/scaling/mod.rs:85-96).
__global__ void k_scale_from_rowmax(int n, const unsigned long long* __restrict__ rmax, double* __restrict__ s) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double m = __longlong_as_double(rmax[i]);
  double r = 1.0;
  if (m > 0.0) {
    double c = 1.0 / sqrt(m);
    if (isfinite(c) && c > 0.0) r = c;
  }
  s[i] = r;
}

// panel[dst[k]] = A_k * s_i * s_j.  Every stored entry has its own target
// (the permutation is a bijection), so this is a plain scatter.
template <typename T>
__global__ void k_assemble(long long nnz, const int* __restrict__ row, const int* __restrict__ col,
                           const T* __restrict__ val, const double* __restrict__ s,
                           const long long* __restrict__ dst, T* __restrict__ panel) {
  long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (k >= nnz) return;
  int i = row[k], j = col[k];
  panel[dst[k]] = Field<T>::scale(val[k], s[i] * s[j]);
}

// Demote a high-precision value array to the low-precision field.
template <typename Hi, typename Lo>
__global__ void k_demote(long long nnz, const Hi* __restrict__ a, Lo* __restrict__ b);

template <>
__global__ void k_demote<double, float>(long long nnz, const double* __restrict__ a, float* __restrict__ b) {
  long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (k < nnz) b[k] = (float)a[k];
}
template <>
__global__ void k_demote<c64, c32>(long long nnz, const c64* __restrict__ a, c32* __restrict__ b) {
  long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (k < nnz) b[k] = c32{(float)a[k].re, (float)a[k].im};
}

// ---------------------------------------------------------------------------
// Shared GEMM-class tile engine: acc[i][j] = sum_t A(i,t) * G(j,t), G = L*D,
// i, j < 64, computed by 256 threads as 4x4 register micro-tiles
// (rows ty + 16*ii, cols tx + 16*jj).
// ---------------------------------------------------------------------------

// Inner-dimension chunk of the tile engine (elements of T per A/B row).
template <typename T> struct KChunk { static constexpr int v = 32; };
template <> struct KChunk<c64> { static constexpr int v = 16; };

// G(j, t) for column t of a factored panel with block-diagonal D.
template <typename T>
__device__ __forceinline__ T ld_G(const T* __restrict__ L, long long ld, int j, int t, const T* __restrict__ d,
                                  const T* __restrict__ dsub, const unsigned char* __restrict__ kind) {
  using F = Field<T>;
  unsigned char kd = kind[t];
  T a = L[j + (long long)t * ld];
  if (kd == 0) return F::mul(a, d[t]);
  if (kd == 1) {
    T b = L[j + (long long)(t + 1) * ld];
    return F::add(F::mul(d[t], a), F::mul(dsub[t], b));
  }
  T p = L[j + (long long)(t - 1) * ld];
  return F::add(F::mul(dsub[t - 1], p), F::mul(d[t], a));
}

// acc[i][j] = sum_t A(i,t) * B(j,t) over t in [0, kdim) for i, j < 64.
// A rows  : L_A + i (i < arows), column t at stride lda
// B rows  : L_B + j (j < brows), column t at stride ldb
// D (indexed by t) multiplies the B operand (D_ON_A = false: the cmod form
// U = L_k G^T, G = L_k D) or the A operand (D_ON_A = true: the deferred
// panel Schur tmp = (L21 D) L21^T).  Accumulation is one explicit FMA per t in
// ascending t, the same order as the oracle.  256 threads, 4x4 register
// micro-tiles (rows ty + 16*ii, cols tx + 16*jj); the next chunk is fetched
// into registers while the current one is multiplied out of shared memory.
template <typename T, bool D_ON_A = false>
__device__ void tile_product(T (&acc)[4][4], const T* __restrict__ LA, long long lda, int arows,
                             const T* __restrict__ LB, long long ldb, int brows, int kdim,
                             const T* __restrict__ d, const T* __restrict__ dsub,
                             const unsigned char* __restrict__ kind, T* As, T* Bs) {
  using F = Field<T>;
  constexpr int KT = KChunk<T>::v;
  constexpr int PER = KT * TILE / TPB;  // elements of each operand staged per thread
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = F::zero();
  T ra[PER], rb[PER];
  auto fetch = [&](int t0) {
    const int kt = min(KT, kdim - t0);
#pragma unroll
    for (int q = 0; q < PER; ++q) {
      const int e = tid + q * TPB;
      const int t = e / TILE, r = e % TILE;
      T av = F::zero(), bv = F::zero();
      if (t < kt) {
        if constexpr (D_ON_A) {
          if (r < arows) av = ld_G(LA, lda, r, t0 + t, d, dsub, kind);
          if (r < brows) bv = LB[r + (long long)(t0 + t) * ldb];
        } else {
          if (r < arows) av = LA[r + (long long)(t0 + t) * lda];
          if (r < brows) bv = ld_G(LB, ldb, r, t0 + t, d, dsub, kind);
        }
      }
      ra[q] = av;
      rb[q] = bv;
    }
  };
  if (kdim > 0) fetch(0);
  for (int t0 = 0; t0 < kdim; t0 += KT) {
    const int kt = min(KT, kdim - t0);
#pragma unroll
    for (int q = 0; q < PER; ++q) {
      const int e = tid + q * TPB;
      As[e] = ra[q];
      Bs[e] = rb[q];
    }
    __syncthreads();
    if (t0 + KT < kdim) fetch(t0 + KT);
    if (kt == KT) {
#pragma unroll 8
      for (int t = 0; t < KT; ++t) {
        T a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = As[t * TILE + ty + 16 * i];
#pragma unroll
        for (int j = 0; j < 4; ++j) b[j] = Bs[t * TILE + tx + 16 * j];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = F::fma_(a[i], b[j], acc[i][j]);
      }
    } else {
      for (int t = 0; t < kt; ++t) {
        T a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = As[t * TILE + ty + 16 * i];
#pragma unroll
        for (int j = 0; j < 4; ++j) b[j] = Bs[t * TILE + tx + 16 * j];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = F::fma_(a[i], b[j], acc[i][j]);
      }
    }
    __syncthreads();
  }
}

__device__ __forceinline__ int lower_bound_i(const int* __restrict__ a, int lo, int hi, int key) {
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    if (a[mid] < key)
      lo = mid + 1;
    else
      hi = mid;
  }
  return lo;
}

// ---------------------------------------------------------------------------
// cmod: task = (s, (r0/64) << 16 | (c0/64), pair_begin, pair_end): tile rows
// [r0, r0+64) x cols [c0, c0+64) of s's panel.  The pairs, precomputed at
// analysis, list in update-list order every descendant k whose update lands
// in the tile: (k, a, q0, nr << 16 | nc) = k's off-diagonal rows [a, a+nr)
// times its rows [q0, q0+nc) (the tile's columns).  No searches at run time
// beyond the tile-local row positions.
//
// Per pair the product U = L_k[a.., :] G_k[q0.., :]^T (G_k = L21_k D_k,
// formed once per updater by k_make_g with ld_G's arithmetic) runs in the
// updater's row space: operands are contiguous column runs of k's panel and
// of G_k, staged by cp.async in shared memory (the next chunks, possibly of
// the next pairs, load while the current one is multiplied).
// 128 threads, warp w owns rows 16w..16w+15 of the pair, each thread an 8 x 4
// register micro-tile (8 consecutive rows, columns cx + 16 j: conflict-free
// shared-memory reads); warps whose rows lie past nr skip the arithmetic.
// Every product is one explicit FMA per column t in ascending t, then
// subtracted from the tile held in shared memory through the pair's row /
// column maps (rows r >= column c in k's ordering only): the same operations
// in the same order as the oracle, so the result is bit-identical to it.
//
// This engine runs the small factors, where a tile has tens of pairs of a few
// columns each: bound by the latency of a pair, not by its arithmetic.  So
// the descriptors of CM_PB pairs are fetched together (their panel offsets
// hang off two dependent loads), and CM_STAGES operand chunks, with the pairs'
// row indices, are in flight by cp.async; and a pair of at most CM_SMALL
// outputs (most of a 2D grid's) is formed one output per thread: the micro-tile
// would run 32 products a column for a handful, and 32 scatter tests.
// 480-unknown 2D grid: 0.264 ms in five launches with descriptors read per
// pair, one chunk ahead and micro-tiles only (0.253 with the first two alone),
// 0.150 now; a KKT factor of 1,866 unknowns 0.407 -> 0.325.
// ---------------------------------------------------------------------------
constexpr int CM_NT = 128;
constexpr int CM_PB = 32;  // pair descriptors per shared-memory batch
constexpr int CM_SMALL = 4 * CM_NT;  // outputs of a pair up to which every thread owns single outputs
template <typename T> struct CmChunk { static constexpr int v = 16, stages = 4; };
template <> struct CmChunk<c64> { static constexpr int v = 8, stages = 2; };  // two CTAs per SM

struct CmPair {
  long long a_off, b_off, r_off;  // L21 rows of the pair, G rows, first off-diagonal row index
  int lda, ldb, nck, a, q0, nr, nc;
};

// Shared memory of k_cmod: the tile, the operand stages with their row and
// column indices, the row / column maps, the tile's row structure and the
// pair descriptors.
template <typename T>
__host__ __device__ constexpr size_t smem_cmod_bytes() {
  return (size_t)TILE * TILE * sizeof(T) +
         CmChunk<T>::stages * (2 * (size_t)CmChunk<T>::v * TILE * sizeof(T) + 2 * TILE * 4) + 3 * TILE * 4 +
         CM_PB * sizeof(CmPair) + 16;
}

template <typename T>
__global__ void __launch_bounds__(CM_NT, 2) k_cmod(FactorArgs fa, const int4* __restrict__ tasks,
                                                   const int4* __restrict__ pairs) {
  using F = Field<T>;
  constexpr int KC = CmChunk<T>::v, NST = CmChunk<T>::stages;
  constexpr int STAGE = 2 * KC * TILE;  // A chunk [t][64 rows] then B chunk [t][64 cols]
  if (factor_failed(fa.status)) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* acc_s = reinterpret_cast<T*>(smem_raw);  // [64 cols][64 rows]
  T* stg = acc_s + TILE * TILE;               // NST stages
  CmPair* prs = reinterpret_cast<CmPair*>(stg + NST * STAGE);
  int* ids = reinterpret_cast<int*>(prs + CM_PB);  // per stage: 64 row and 64 column indices
  int* rs_tile = ids + NST * 2 * TILE;             // 64
  int* rowmap = rs_tile + TILE;                    // 64
  int* colmap = rowmap + TILE;                     // 64

  const int4 tk = tasks[blockIdx.x];
  const int s = tk.x, r0 = (tk.y >> 16) * TILE, c0 = (tk.y & 0xffff) * TILE;
  const int first = fa.sn_first[s], ncol = fa.sn_ncol[s], nrow = fa.sn_nrow[s];
  const int rows_here = min(TILE, nrow - r0), cols_here = min(TILE, ncol - c0);
  T* panel = reinterpret_cast<T*>(fa.panel) + fa.sn_poff[s];
  const int* rss = fa.rs + fa.sn_rsoff[s];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int e = tid; e < TILE * TILE; e += CM_NT) {
    const int c = e / TILE, r = e % TILE;
    T v = F::zero();
    if (r < rows_here && c < cols_here) v = panel[(r0 + r) + (long long)(c0 + c) * nrow];
    acc_s[e] = v;
  }
  if (tid < TILE) rs_tile[tid] = tid < rows_here ? rss[r0 + tid] : INT_MAX;
  const T* pall = reinterpret_cast<const T*>(fa.panel);
  const T* gall = reinterpret_cast<const T*>(fa.gpool);

  // chunk stream over (pair u of the batch, columns [t0, t0 + KC) of its updater)
  struct Cur {
    int u, t0;
  };
  auto issue = [&](Cur x, int st) {
    const CmPair& p = prs[x.u];
    const T* A = pall + p.a_off;
    const T* B = gall + p.b_off;
    T* As = stg + st * STAGE;
    T* Bs = As + KC * TILE;
    const int nr = p.nr, nc = p.nc, kt = p.nck - x.t0;
    const int r = tid % TILE, tb = tid / TILE;
    const T* Ar = A + r + (long long)(x.t0 + tb) * p.lda;
    const T* Br = B + r + (long long)(x.t0 + tb) * p.ldb;
    const long long sa = (CM_NT / TILE) * (long long)p.lda, sb = (CM_NT / TILE) * (long long)p.ldb;
#pragma unroll
    for (int q = 0; q < KC * TILE / CM_NT; ++q) {
      const bool in_t = tb + q * (CM_NT / TILE) < kt;
      const int e = tid + q * CM_NT;
      cp_async_zfill<(int)sizeof(T)>(As + e, in_t && r < nr ? Ar + q * sa : A, in_t && r < nr);
      cp_async_zfill<(int)sizeof(T)>(Bs + e, in_t && r < nc ? Br + q * sb : B, in_t && r < nc);
    }
    if (x.t0 == 0) {
      const int* ok = fa.rs + p.r_off + (tid < TILE ? p.a : p.q0);
      const int i = tid & (TILE - 1);
      if (i < (tid < TILE ? nr : nc)) cp_async_zfill<4>(ids + st * 2 * TILE + tid, ok + i, true);
    }
  };
  auto advance = [&](Cur x) -> Cur {
    x.t0 += KC;
    if (x.t0 >= prs[x.u].nck) {
      x.u += 1;
      x.t0 = 0;
    }
    return x;
  };

  const int ry = lane >> 4, cx = lane & 15;
  const int rb = 16 * warp + 8 * ry;  // this thread's rows rb..rb+7, columns cx + 16 j
  T acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = F::zero();

  for (int u0 = tk.z; u0 < tk.w; u0 += CM_PB) {
    const int np = min(CM_PB, tk.w - u0);
    __syncthreads();  // the previous batch's descriptors and stages are free (first: the tile is written)
    for (int e = tid; e < np; e += CM_NT) {
      const int4 pr = pairs[u0 + e];
      const int k = pr.x, nck = fa.sn_ncol[k], nrk = fa.sn_nrow[k];
      prs[e] = CmPair{fa.sn_poff[k] + nck + pr.y, fa.goff[k] + pr.z, fa.sn_rsoff[k] + nck, nrk, nrk - nck, nck,
                      pr.y, pr.z, pr.w >> 16, pr.w & 0xffff};
    }
    __syncthreads();
    Cur cur{0, 0}, nxt{0, 0};
    int si = 0, sc = 0;  // issue / compute stage
#pragma unroll 1
    for (int q = 0; q < NST - 1; ++q) {
      if (nxt.u < np) {
        issue(nxt, si);
        nxt = advance(nxt);
        si = si + 1 == NST ? 0 : si + 1;
      }
      cp_async_commit();
    }
    while (cur.u < np) {
      if (nxt.u < np) {
        issue(nxt, si);
        nxt = advance(nxt);
        si = si + 1 == NST ? 0 : si + 1;
      }
      cp_async_commit();
      cp_async_wait<NST - 1>();
      __syncthreads();  // the chunk landed everywhere; the last pair's scatter is done
      const CmPair& p = prs[cur.u];
      const int nr = p.nr, nc = p.nc, a = p.a, q0 = p.q0;
      if (cur.t0 == 0) {
        // the tile positions of this pair's rows and columns (read at the
        // pair's scatter, after the next barrier)
        const int* id = ids + sc * 2 * TILE;
        if (tid < nr) rowmap[tid] = lower_bound_i(rs_tile, 0, rows_here, id[tid]);
        if (tid >= TILE && tid - TILE < nc) colmap[tid - TILE] = id[tid] - first - c0;
      }
      const T* As = stg + sc * STAGE;
      const T* Bs = As + KC * TILE;
      const int kt = min(KC, p.nck - cur.t0);
      // a pair of at most CM_SMALL outputs: one output per thread and pass
      // instead of a mostly empty micro-tile (its results in acc[0][.])
      const bool small = nr * nc <= CM_SMALL;
      if (small) {
#pragma unroll
        for (int z = 0; z < CM_SMALL / CM_NT; ++z) {
          const int o = tid + z * CM_NT;
          if (o < nr * nc) {
            const int cj = o / nr, ri = o - cj * nr;
            T v = acc[0][z];
#pragma unroll 4
            for (int t = 0; t < kt; ++t) v = F::fma_(As[t * TILE + ri], Bs[t * TILE + cj], v);
            acc[0][z] = v;
          }
        }
      } else if (rb - 8 * ry < nr) {  // the warp has rows of this pair
        if (kt == KC) {
#pragma unroll 2
          for (int t = 0; t < KC; ++t) {
            T av[8], bv[4];
            lds_row<T, 8>(As + t * TILE + rb, av);
#pragma unroll
            for (int j = 0; j < 4; ++j) bv[j] = Bs[t * TILE + cx + 16 * j];
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
              for (int j = 0; j < 4; ++j) acc[i][j] = F::fma_(av[i], bv[j], acc[i][j]);
          }
        } else {
          for (int t = 0; t < kt; ++t) {
            T av[8], bv[4];
            lds_row<T, 8>(As + t * TILE + rb, av);
#pragma unroll
            for (int j = 0; j < 4; ++j) bv[j] = Bs[t * TILE + cx + 16 * j];
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
              for (int j = 0; j < 4; ++j) acc[i][j] = F::fma_(av[i], bv[j], acc[i][j]);
          }
        }
      }
      const Cur after = advance(cur);
      __syncthreads();  // the stage is free for the next issue; the maps are written
      if (after.u != cur.u && small) {
#pragma unroll
        for (int z = 0; z < CM_SMALL / CM_NT; ++z) {
          const int o = tid + z * CM_NT;
          const int cj = o / nr, ri = o - cj * nr;
          if (o < nr * nc && a + ri >= q0 + cj) {
            const int e = colmap[cj] * TILE + rowmap[ri];
            acc_s[e] = F::sub(acc_s[e], acc[0][z]);
          }
          acc[0][z] = F::zero();
        }
      } else if (after.u != cur.u) {
        // the pair is complete: subtract it from the tile, reset the registers
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int ri = rb + i;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int cj = cx + 16 * j;
            if (ri < nr && cj < nc && a + ri >= q0 + cj) {
              const int e = colmap[cj] * TILE + rowmap[ri];
              acc_s[e] = F::sub(acc_s[e], acc[i][j]);
            }
            acc[i][j] = F::zero();
          }
        }
      }
      sc = sc + 1 == NST ? 0 : sc + 1;
      cur = after;
    }
  }
  cp_async_wait<0>();
  __syncthreads();
  for (int e = tid; e < TILE * TILE; e += CM_NT) {
    const int c = e / TILE, r = e % TILE;
    if (r < rows_here && c < cols_here && r0 + r >= c0 + c) panel[(r0 + r) + (long long)(c0 + c) * nrow] = acc_s[e];
  }
}

// ---------------------------------------------------------------------------
// Deferred in-panel Schur: task = (s, kb, r0, c0) with tile rows [ke+r0, ...)
// and cols [ke+c0, ...): panel -= L21 D L21^T on rows >= cols.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(TPB) k_schur(FactorArgs fa, const int4* __restrict__ tasks, int nb_small,
                                               int nb_big) {
  using F = Field<T>;
  if (factor_failed(fa.status)) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* As = reinterpret_cast<T*>(smem_raw);
  T* Bs = As + KChunk<T>::v * TILE;
  const int4 tk = tasks[blockIdx.x];
  const int s = tk.x, kb = tk.y, r0 = tk.z, c0 = tk.w;
  const int first = fa.sn_first[s], ncol = fa.sn_ncol[s], nrow = fa.sn_nrow[s];
  const int nb = ncol >= 512 ? nb_big : nb_small;
  const int ke = min(kb + nb, ncol);
  const int pw = ke - kb, mt = nrow - ke, cw = ncol - ke;
  T* panel = reinterpret_cast<T*>(fa.panel) + fa.sn_poff[s];
  const int rows_here = min(TILE, mt - r0), cols_here = min(TILE, cw - c0);
  const T* L21 = panel + ke + (long long)kb * nrow;
  T acc[4][4];
  tile_product<T, true>(acc, L21 + r0, nrow, rows_here, L21 + c0, nrow, cols_here, pw,
                  reinterpret_cast<const T*>(fa.d) + first + kb, reinterpret_cast<const T*>(fa.dsub) + first + kb,
                  fa.kind + first + kb, As, Bs);
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  // every load before the first store (distinct targets)
  T old[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int rr = r0 + ty + 16 * i, cc = c0 + tx + 16 * j;
      const bool in = ty + 16 * i < rows_here && tx + 16 * j < cols_here && rr >= cc;
      old[i][j] = in ? panel[(ke + rr) + (long long)(ke + cc) * nrow] : F::zero();
    }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int rr = r0 + ty + 16 * i, cc = c0 + tx + 16 * j;
      if (ty + 16 * i < rows_here && tx + 16 * j < cols_here && rr >= cc)
        panel[(ke + rr) + (long long)(ke + cc) * nrow] = F::sub(old[i][j], acc[i][j]);
    }
}

// ---------------------------------------------------------------------------
// Multifrontal variant (factor_front + extend-add, multifrontal_ldlt.rs:901,
// 1494-1510).  A front of supernode s is its panel (nrow x ncol, the
// fully-summed columns) plus its contribution block CB_s (m x m, m = nrow -
// ncol, the trailing rows and columns, lower part).
//
// k_extend_add: task (s, ct, pair_begin, pair_end): front columns [64 ct,
// 64 ct + 64) of s, front rows of one chunk of EA_ROWS; pair (c, ja, jb):
// child c's contribution-block columns [ja, jb) land there, its rows
// [i0, i1) (the pair's row range) in the chunk.  Children are added in order (a block barrier between
// them), each entry (i, j), i >= j, of a child's block into the front entry
// (map[i], map[j]) (the child's rows' positions in the front): the panel
// when map[j] < ncol, CB_s otherwise.  Deterministic; no atomics.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) k_extend_add(FactorArgs fa, const int4* __restrict__ tasks,
                                                    const int4* __restrict__ pairs, const int2* __restrict__ prow,
                                                    const int* __restrict__ emap,
                                                    const long long* __restrict__ emoff) {
  using F = Field<T>;
  if (factor_failed(fa.status)) return;
  const int4 tk = tasks[blockIdx.x];
  const int s = tk.x, ncol = fa.sn_ncol[s], nrow = fa.sn_nrow[s], ms = nrow - ncol;
  T* panel = reinterpret_cast<T*>(fa.panel) + fa.sn_poff[s];
  T* cbs = reinterpret_cast<T*>(fa.cbpool) + fa.cb_off[s];
  constexpr int EB = 8;  // entries per thread per batch: every load of a batch before its stores
  for (int u = tk.z; u < tk.w; ++u) {
    const int4 pr = pairs[u];
    const int c = pr.x, mc = fa.sn_nrow[c] - fa.sn_ncol[c];
    const T* cbc = reinterpret_cast<const T*>(fa.cbpool) + fa.cb_off[c];
    const int* map = emap + emoff[c];
    // the child's columns [ja, jb) x rows [i0, i1) (the rows landing in this
    // task's row chunk) as one index space (rows fastest: coalesced reads of
    // the child's block), entries above the diagonal skipped; the targets of
    // one child are distinct
    const int2 rr = prow[u];
    const int len = rr.y - rr.x;
    const int tot = (pr.z - pr.y) * len;  // at most 64 columns x EA_ROWS rows
    for (int e0 = 0; e0 < tot; e0 += EB * 256) {
      T* tp[EB];
      T v[EB], old[EB];
#pragma unroll
      for (int q = 0; q < EB; ++q) {
        const int e = e0 + (int)threadIdx.x + q * 256;
        tp[q] = nullptr;
        if (e < tot) {
          const int j = pr.y + e / len, i = rr.x + e % len;
          if (i >= j) {
            const int li = map[i], lj = map[j];
            tp[q] = lj < ncol ? panel + li + (long long)lj * nrow : cbs + (li - ncol) + (long long)(lj - ncol) * ms;
            v[q] = cbc[i + (long long)j * mc];
          }
        }
      }
#pragma unroll
      for (int q = 0; q < EB; ++q) old[q] = tp[q] ? *tp[q] : F::zero();
#pragma unroll
      for (int q = 0; q < EB; ++q)
        if (tp[q]) *tp[q] = F::add(old[q], v[q]);
    }
    __syncthreads();  // the next child's additions follow this one's
  }
}

// k_front_cb: task (s, r0, c0, 0): CB_s rows [r0, r0 + 64) x columns [c0,
// c0 + 64), r0 >= c0, minus (L21 D L21^T) over all of s's columns (the
// tile engine with D on the row operand, as the in-panel Schur update), on
// its lower part.
template <typename T>
__global__ void __launch_bounds__(TPB) k_front_cb(FactorArgs fa, const int4* __restrict__ tasks) {
  using F = Field<T>;
  if (factor_failed(fa.status)) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* As = reinterpret_cast<T*>(smem_raw);
  T* Bs = As + KChunk<T>::v * TILE;
  const int4 tk = tasks[blockIdx.x];
  const int s = tk.x, r0 = tk.y, c0 = tk.z;
  const int first = fa.sn_first[s], ncol = fa.sn_ncol[s], nrow = fa.sn_nrow[s], m = nrow - ncol;
  const T* L21 = reinterpret_cast<const T*>(fa.panel) + fa.sn_poff[s] + ncol;
  T* cb = reinterpret_cast<T*>(fa.cbpool) + fa.cb_off[s];
  const int rows_here = min(TILE, m - r0), cols_here = min(TILE, m - c0);
  T acc[4][4];
  tile_product<T, true>(acc, L21 + r0, nrow, rows_here, L21 + c0, nrow, cols_here, ncol,
                        reinterpret_cast<const T*>(fa.d) + first, reinterpret_cast<const T*>(fa.dsub) + first,
                        fa.kind + first, As, Bs);
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  // every load before the first store (distinct targets)
  T old[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int rr = r0 + ty + 16 * i, cc = c0 + tx + 16 * j;
      const bool in = ty + 16 * i < rows_here && tx + 16 * j < cols_here && rr >= cc;
      old[i][j] = in ? cb[rr + (long long)cc * m] : F::zero();
    }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int rr = r0 + ty + 16 * i, cc = c0 + tx + 16 * j;
      if (ty + 16 * i < rows_here && tx + 16 * j < cols_here && rr >= cc)
        cb[rr + (long long)cc * m] = F::sub(old[i][j], acc[i][j]);
    }
}

// ---------------------------------------------------------------------------
// Block reductions for the pivot search: max of a non-negative double with
// the lowest index on ties (the reference's strict `>` scan).
// ---------------------------------------------------------------------------
// Warp-wide arg-max of every lane's (v, i), v >= 0 or -1 (none): largest v,
// then smallest i, from three warp reductions on an
// order-preserving key (bits of v + 1; 0 for none), instead of a shuffle tree.
__device__ __forceinline__ void warp_argmax(double& v, int& i) {
  const unsigned long long key = v >= 0.0 ? (unsigned long long)__double_as_longlong(v) + 1ull : 0ull;
  const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
  const unsigned mhi = __reduce_max_sync(0xffffffffu, hi);
  const unsigned mlo = __reduce_max_sync(0xffffffffu, hi == mhi ? lo : 0u);
  const bool win = hi == mhi && lo == mlo;
  const int mi = (int)__reduce_min_sync(0xffffffffu, win ? (unsigned)i : 0xffffffffu);
  const unsigned long long mk = ((unsigned long long)mhi << 32) | mlo;
  v = mk == 0ull ? -1.0 : __longlong_as_double((long long)(mk - 1ull));
  i = mk == 0ull ? INT_MAX : mi;
}

template <typename T>
__device__ __forceinline__ T shfl_t(T v, int src) {
  if constexpr (Field<T>::complex) {
    T r;
    r.re = __shfl_sync(0xffffffffu, v.re, src);
    r.im = __shfl_sync(0xffffffffu, v.im, src);
    return r;
  } else {
    return __shfl_sync(0xffffffffu, v, src);
  }
}

// ---------------------------------------------------------------------------
// Force-accept floor: max(max_ij |A_scaled ij|, 1) * eps over the assembled
// panels (every stored entry of the equilibrated matrix lands in exactly one
// slot; the other slots are zero).
// ---------------------------------------------------------------------------
template <typename T>
__global__ void k_panel_absmax(long long m, const T* __restrict__ panel, unsigned long long* __restrict__ out) {
  double v = 0.0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < m; i += (long long)gridDim.x * blockDim.x)
    v = fmax(v, Field<T>::mag(panel[i]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  if ((threadIdx.x & 31) == 0) atomicMax(out, __double_as_longlong(v));
}

__global__ void k_force_floor(const unsigned long long* __restrict__ amax, double* __restrict__ floor_out) {
  const double a = __longlong_as_double(*amax);
  *floor_out = fmax(a, 1.0) * 2.220446049250313e-16;
}

// ---------------------------------------------------------------------------
// Incomplete factor (drop_tol): per pivot column p of every panel, drop the
// multipliers below tau * max |L_ip| (rows below the pivot, the 2x2 coupling
// slot excluded) — ldlt_emit_and_free, src/numeric/multifrontal_ldlt.rs:2359.
// One CTA per supernode, one warp per column.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void k_drop_tol(FactorArgs fa, double tau) {
  using F = Field<T>;
  if (factor_failed(fa.status)) return;
  const int s = blockIdx.x;
  const int first = fa.sn_first[s], ncol = fa.sn_ncol[s], nrow = fa.sn_nrow[s];
  T* panel = reinterpret_cast<T*>(fa.panel) + fa.sn_poff[s];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int p = warp; p < ncol; p += nw) {
    const int i0 = p + (fa.kind[first + p] == 1 ? 2 : 1);
    T* col = panel + (long long)p * nrow;
    double cm = 0.0;
    for (int i = i0 + lane; i < nrow; i += 32) cm = fmax(cm, F::mag(col[i]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) cm = fmax(cm, __shfl_xor_sync(0xffffffffu, cm, o));
    const double thresh = tau * cm;
    for (int i = i0 + lane; i < nrow; i += 32)
      if (F::mag(col[i]) < thresh) col[i] = F::zero();
  }
}

}  // namespace rsd
