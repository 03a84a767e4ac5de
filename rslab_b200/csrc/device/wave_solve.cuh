// Triangular-solve kernels of the supernodal solve that stream the panels
// at memory bandwidth, and the dependency-chain solve of the wide
// supernodes' diagonal blocks.
//
// Streaming (k_stream): the forward push U_s = L21_s z_s and the backward
// off-diagonal dots L21_s^T x_anc.  An item owns 64 outputs and loops over
// 32-wide reduction units; each unit's 2048-element panel tile and its 32
// right-hand-side rows are copied global -> shared with cp.async (zero
// filled outside the panel), `st_stages<T>(NR)` units in flight, one CTA
// barrier per unit.  Tile layouts keep every lane on consecutive or odd
// strided shared memory:
//   forward  : 64 output rows x 32 reduction columns, S[q * 65 + r]
//   backward : 32 reduction rows x 64 output columns, S[p * 33 + r]
// Thread (x = tid & 63, g = tid >> 6) owns output x and the reduction slice
// [8g, 8g + 8) of every unit; the four slice partials are added in order
// g = 0..3 at the end, so results are deterministic.  The right-hand sides
// read here are final before the launch (forward: z of this level, solved
// by an earlier launch; backward: the ancestors' x, each unit's 32 rows
// read through the supernode's row structure).
//
// Chain (k_chain): every supernode is cut into TB = 64 column blocks whose
// solves form a chain (forward: block i needs z of blocks j < i; backward:
// x of blocks j > i).  One CTA per block and group of at most CH_NR
// right-hand-side columns (the columns' chains are independent):
//   forward : z_i = Linv_i (y_i - sum_{j<i} L_ij z_j)
//   backward: x_i = Linv_i^T (w_i - W_i - sum_{j>i, descending} L_ji^T x_j)
// with Linv_i the precomputed inverse of the unit-lower diagonal block and
// W_i the off-diagonal dots.  The 64 x 64 tiles stream through shared
// memory ahead of the chain.  Items are handed out in ticket order (an
// atomic counter per launch, not blockIdx) and every item waits only on items
// with smaller tickets, whose CTAs have therefore started, so the chain
// progresses whatever the number of resident CTAs.  A block's values are
// their own flags: the vector starts out as a bit pattern that no result has
// (all ones; a NaN result is stored as the quiet NaN), every value is stored
// with a gpu-scope relaxed store, and a waiting thread polls the values it
// needs (relaxed loads of the same width).  One round trip through L2 per
// block, against three (release fence, flag, value) with a flag per block:
// 64^3 root, 64 blocks, 231 us with flags.  Polls are bounded; on a
// timeout the thread raises the launch-wide abort word and a sticky status
// that the host reads after the solve.
// Reference: the column-block substitution of solve_ldlt_block
// (src/dense/ldlt_generic.rs:618-714), reorganised as a dependency chain.
#pragma once

#include "async_copy.cuh"
#include "solve_kernels.cuh"

namespace rsd {

constexpr int WV_NT = 256;
constexpr long WV_POLL_LIMIT = 1L << 21;  // polls before a wait gives up
constexpr int ST_UNIT = 2112;             // streamed tile elements (max of 32 x 65 and 64 x 33)
constexpr int CH_UNIT = 64 * 65;          // chain tile elements
// Units (32 x 64 panel tiles) that a streamed item takes one after another: a
// level's units over ST_ITEMS items (four per SM: the kernel runs one to three
// CTAs on an SM, see st_minb), within these bounds.  Fixed items of 16 units left the upper levels with 20 to 300 items
// of 30 to 50 us each.
constexpr int ST_ITEMS = 4 * 148, ST_UNITS_MIN = 2, ST_UNITS_MAX = 16;
// The right-hand sides of a pass are solved as CH_GROUPS independent chains
// of at most CH_NR columns (more CTAs, shorter per-block products).
constexpr int CH_NR = 4;
constexpr int CH_GROUPS = RHS_MAX / CH_NR;
// blocks in a level from which its chains take every column of a pass
constexpr int CH_WIDE_ITEMS = 600;

// CTAs per SM of the streamed kernel, and with them its stages and the columns
// whose slice partials are exchanged at a time.  Instances of one and four
// columns: three CTAs, four stages (three for 16-byte elements).  Sixteen
// columns in the single-precision fields: two stages (the next unit loads while one is
// multiplied) and partials by halves, so that three CTAs fit instead of two
// (64^3 mixed step 54.9 -> 52.6 ms; f32, 40 columns on 37 x 40 x 33: 3.53 ->
// 3.39).  In double precision that costs more than it gives: f64 has three
// stages and whole partials on two CTAs (40 columns on 24 x 25 x 23: 1.49 ms
// with three CTAs and more spills, 1.44 so; on 150 x 140 1.13 and 1.07), c64
// the same on one (two: 0.7% slower).
template <typename T>
__host__ __device__ constexpr bool st_three(int nr) {
  return nr < 16 || sizeof(typename Field<T>::Real) == 4;
}
template <typename T>
__host__ __device__ constexpr int st_stages(int nr) {
  return nr >= 16 && st_three<T>(nr) ? 2 : nr >= 16 || sizeof(T) >= 16 ? 3 : 4;
}
template <typename T>
__host__ __device__ constexpr int st_red_cols(int nr) {
  return nr >= 16 && st_three<T>(nr) ? 8 : nr;
}
template <typename T>
__host__ __device__ constexpr int st_minb(int nr) {
  return st_three<T>(nr) ? 3 : sizeof(T) >= 16 ? 1 : 2;
}

// Right-hand-side buffers are sized by the pass's column count nr (<=
// RHS_MAX), so a one-column solve keeps several CTAs resident per SM; the
// kernels are instantiated for NR = 1, 4 and 16 register columns (the
// smallest NR >= nr runs) so the inner loops carry no dead columns.
// Streaming: stages of (tile + 32 x nr right-hand sides), then the slice
// partials (4 x st_red_cols x 65).
template <typename T>
__host__ __device__ constexpr size_t st_stage_elems(int nr) {
  return (size_t)ST_UNIT + 32 * nr;
}
template <typename T>
__host__ __device__ constexpr size_t st_smem_bytes(int nr) {
  return ((size_t)st_stages<T>(nr) * st_stage_elems<T>(nr) + 4 * 65 * st_red_cols<T>(nr)) * sizeof(T) + 16;
}
// Chain: one tile slot (its copy overlaps the wait for the dependency's
// values; after the chain it holds the slice partials), the inverse block,
// right-hand sides (64 x nr) and the block vector (64 x nr).
template <typename T>
__host__ __device__ constexpr size_t ch_smem_bytes(int nr) {
  return ((size_t)2 * CH_UNIT + 64 * nr + 64 * nr) * sizeof(T) + 16;
}

// Wave state (ints): [0] sticky status (nonzero after a timed-out wait;
// cleared by the host when read), then the per-pass region cleared before
// every pass: [1] abort word, [2, 2 + nchain) ticket counters.
constexpr int WV_STATE_ABORT = 1;
constexpr int WV_STATE_CTR = 2;

// Published values: relaxed gpu-scope stores and loads of one word per
// component group (c32 as one 8-byte word, c64 as two); false from
// ld_published while the value is still the initial pattern.
__device__ __forceinline__ void st_word(unsigned* p, unsigned v) {
  asm volatile("st.relaxed.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void st_word(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned ld_word(const unsigned* p) {
  unsigned v;
  asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned long long ld_word(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned quiet_bits(float v) { return v != v ? 0x7fc00000u : __float_as_uint(v); }
__device__ __forceinline__ unsigned long long quiet_bits(double v) {
  return v != v ? 0x7ff8000000000000ull : (unsigned long long)__double_as_longlong(v);
}
__device__ __forceinline__ void st_published(float* p, float v) { st_word(reinterpret_cast<unsigned*>(p), quiet_bits(v)); }
__device__ __forceinline__ void st_published(double* p, double v) {
  st_word(reinterpret_cast<unsigned long long*>(p), quiet_bits(v));
}
__device__ __forceinline__ void st_published(c32* p, c32 v) {
  st_word(reinterpret_cast<unsigned long long*>(p),
          (unsigned long long)quiet_bits(v.im) << 32 | quiet_bits(v.re));
}
__device__ __forceinline__ void st_published(c64* p, c64 v) {
  st_published(&p->re, v.re);
  st_published(&p->im, v.im);
}
__device__ __forceinline__ bool ld_published(const float* p, float& v) {
  const unsigned w = ld_word(reinterpret_cast<const unsigned*>(p));
  v = __uint_as_float(w);
  return w != ~0u;
}
__device__ __forceinline__ bool ld_published(const double* p, double& v) {
  const unsigned long long w = ld_word(reinterpret_cast<const unsigned long long*>(p));
  v = __longlong_as_double((long long)w);
  return w != ~0ull;
}
__device__ __forceinline__ bool ld_published(const c32* p, c32& v) {
  const unsigned long long w = ld_word(reinterpret_cast<const unsigned long long*>(p));
  v = c32{__uint_as_float((unsigned)w), __uint_as_float((unsigned)(w >> 32))};
  return w != ~0ull;
}
__device__ __forceinline__ bool ld_published(const c64* p, c64& v) {
  const bool a = ld_published(&p->re, v.re), b = ld_published(&p->im, v.im);
  return a && b;
}
__device__ __forceinline__ int ld_volatile(const int* p) { return *reinterpret_cast<const volatile int*>(p); }

// Slice partials live at red[(g * NR + c) * 65 + x] (lanes over x write
// consecutive words).  The sum over g = 0..3 in order:
template <typename T, int NR>
__device__ __forceinline__ T slice_sum(const T* red, int x, int c) {
  using F = Field<T>;
  T s = red[c * 65 + x];
  s = F::add(s, red[(NR + c) * 65 + x]);
  s = F::add(s, red[(2 * NR + c) * 65 + x]);
  return F::add(s, red[(3 * NR + c) * 65 + x]);
}
template <typename T, int NR>
__device__ __forceinline__ void store_partials(T* red, const T (&acc)[NR], int x, int g) {
#pragma unroll
  for (int c = 0; c < NR; ++c) red[(g * NR + c) * 65 + x] = acc[c];
}

// ---------------------------------------------------------------------------
// Streaming items.  Forward push (s, r0, nrb): U rows [r0, r0 + 64 nrb) of s
// = L[ncol + r, :] z_s, one 64-row block after another (narrow supernodes
// take several blocks per item so an item streams a few units at least).
// Backward dots (s, i, r0, slot): for the columns of block i, sum over
// the off-diagonal rows from ncol + r0 on (32 per unit) of L[r, p] x_anc[r];
// slot < 0 (the only chunk) writes Wb, else partial sums go to slot `slot`
// (64 x ld each), which the backward chain item of block i adds up in chunk
// order.
// ---------------------------------------------------------------------------
template <typename T, bool FWD>
struct StItem {
  const T* L;
  long long ld;       // panel leading dimension (nrow)
  int r0, rlim;       // tile rows
  int c0, clim;       // tile columns
  const T* V;         // right-hand-side row 0 of the item (row stride a.ld); backward: x in g order
  const int* vrows;   // backward: g of each of the item's rows (x is read through it)
  int vlim;           // right-hand-side rows valid < vlim (relative)
  int cu;             // forward: column units per 64-row block (of this item's column chunk)
  int cb0;            // forward: first column unit of the item
  int nunits;
};

template <typename T, bool FWD>
__device__ __forceinline__ StItem<T, FWD> st_item(const SolveArgs& a, int4 tk) {
  const int s = tk.x;
  const int first = a.sn_first[s], ncol = a.sn_ncol[s], nrow = a.sn_nrow[s];
  StItem<T, FWD> it;
  it.L = reinterpret_cast<const T*>(a.panel) + a.sn_poff[s];
  it.ld = nrow;
  if (FWD) {
    it.r0 = ncol + tk.y; it.rlim = nrow;
    it.c0 = 0; it.clim = ncol;
    it.V = reinterpret_cast<const T*>(a.Ze) + a.c0 + (long long)first * a.ld;
    it.vlim = ncol;
    if (tk.w < 0) {  // z = row blocks
      it.cb0 = 0;
      it.cu = (ncol + 31) / 32;
      it.nunits = min(tk.z, (nrow - it.r0 + 63) / 64) * it.cu;
    } else {  // z = 1 | column units << 3 | first column unit << 8 (partial sums to slot w)
      it.cb0 = tk.z >> 8;
      it.cu = min((tk.z >> 3) & 31, (ncol + 31) / 32 - it.cb0);
      it.nunits = it.cu;
    }
  } else {
    it.r0 = ncol + tk.z; it.rlim = min(nrow, it.r0 + 32 * (tk.y >> 24));  // y = block | units << 24
    it.c0 = (tk.y & 0xffffff) * TB; it.clim = ncol;
    // the ancestors' x straight from the solution vector: row r of the item
    // is g = rs[ncol + r0 + r] (no gathered copy)
    it.V = reinterpret_cast<const T*>(a.Xg) + a.c0;
    it.vrows = a.rs + a.sn_rsoff[s] + ncol + tk.z;
    it.vlim = it.rlim - it.r0;
    it.cu = 1;
    it.cb0 = 0;
    it.nunits = (it.vlim + 31) / 32;
  }
  return it;
}

template <typename T, bool FWD, int NR>
__device__ __forceinline__ void st_issue(T* S, T* Vs, const StItem<T, FWD>& it, int u, int ld, int nr) {
  int rr0, cc0, vr0;
  if constexpr (FWD) {
    const int rb = u / it.cu, cb = it.cb0 + u - rb * it.cu;
    rr0 = it.r0 + 64 * rb; cc0 = 32 * cb; vr0 = 32 * cb;
  } else {
    rr0 = it.r0 + 32 * u; cc0 = it.c0; vr0 = 32 * u;
  }
#pragma unroll
  for (int m = 0; m < 2048 / WV_NT; ++m) {
    const int e = threadIdx.x + WV_NT * m;
    int r, c, dst;
    if constexpr (FWD) {
      r = rr0 + (e & 63); c = cc0 + (e >> 6); dst = (e >> 6) * 65 + (e & 63);
    } else {
      r = rr0 + (e & 31); c = cc0 + (e >> 5); dst = (e >> 5) * 33 + (e & 31);
    }
    // forward: columns past the block are not reduced over (nothing to fill);
    // backward: the same for rows
    const bool ok = r < it.rlim && c < it.clim;
    if (FWD ? c >= it.clim : r >= it.rlim) continue;
    const T* g = ok ? it.L + r + (long long)c * it.ld : it.L;
    cp_async_zfill<sizeof(T)>(S + dst, g, ok);
  }
  for (int e = threadIdx.x; e < 32 * nr; e += WV_NT) {
    const int k = e / nr, c = e - k * nr, row = vr0 + k;
    if (row >= it.vlim) break;
    const long long vr = FWD ? row : it.vrows[row];
    cp_async_zfill<sizeof(T)>(Vs + k * NR + c, it.V + vr * ld + c, true);
  }
}

template <typename T, bool FWD, int NR>
__global__ void __launch_bounds__(WV_NT, st_minb<T>(NR)) k_stream(SolveArgs a, const int4* __restrict__ tasks) {
  using F = Field<T>;
  constexpr int NST = st_stages<T>(NR), RC = st_red_cols<T>(NR);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nr = a.nrhs, ld = a.ld;
  constexpr int SE = (int)st_stage_elems<T>(NR);
  T* stages = reinterpret_cast<T*>(smem_raw);  // NST x (tile, V rows of stride NR)
  T* red = stages + NST * SE;                  // slice partials, 4 x RC x 65
  const int4 tk = tasks[blockIdx.x];
  const int s = tk.x;
  const StItem<T, FWD> it = st_item<T, FWD>(a, tk);
  const int tid = threadIdx.x, x = tid & 63, g = tid >> 6;
  T acc[NR];
#pragma unroll
  for (int c = 0; c < NR; ++c) acc[c] = F::zero();
  // slice partials of the finished output block -> U (forward) / Wb / slot
  auto flush = [&](int rb) {
#pragma unroll
    for (int h = 0; h < NR; h += RC) {
      if (h > 0) {
        if (h >= nr) break;
        __syncthreads();  // the columns before are summed
      }
#pragma unroll
      for (int c = 0; c < RC; ++c) red[(g * RC + c) * 65 + x] = acc[h + c];
      __syncthreads();
      const int nc = min(RC, nr - h);
      for (int e = tid; e < 64 * nc; e += WV_NT) {
        const int r = e / nc, c = e - r * nc;
        const T v = slice_sum<T, RC>(red, r, c);
        T* out = nullptr;
        if (FWD) {
          const int row = it.r0 + 64 * rb + r;
          if (row < it.rlim && tk.w < 0)
            out = reinterpret_cast<T*>(a.U) + a.c0 + (a.uoff[s] + row - a.sn_ncol[s]) * (long long)ld;
          else if (row < it.rlim)
            out = reinterpret_cast<T*>(a.Wp) + ((long long)tk.w * 64 + r) * ld;
        } else if (it.c0 + r < it.clim) {
          if (tk.w < 0)
            out = reinterpret_cast<T*>(a.Wb) + a.c0 + (long long)(a.sn_first[s] + it.c0 + r) * ld;
          else
            out = reinterpret_cast<T*>(a.Wp) + ((long long)tk.w * 64 + r) * ld;
        }
        if (out) out[h + c] = v;
      }
    }
#pragma unroll
    for (int c = 0; c < NR; ++c) acc[c] = F::zero();
  };
#pragma unroll 1
  for (int u = 0; u < NST - 1; ++u) {
    T* S = stages + u * SE;
    if (u < it.nunits) st_issue<T, FWD, NR>(S, S + ST_UNIT, it, u, ld, nr);
    cp_async_commit();
  }
#pragma unroll 1
  for (int u = 0; u < it.nunits; ++u) {
    if (FWD && u > 0 && u % it.cu == 0) flush(u / it.cu - 1);
    cp_async_wait<NST - 2>();
    __syncthreads();  // unit u landed everywhere; unit u - 1's stage and the partials are free
    {
      const int un = u + NST - 1;
      T* Sn = stages + (un % NST) * SE;
      if (un < it.nunits) st_issue<T, FWD, NR>(Sn, Sn + ST_UNIT, it, un, ld, nr);
      cp_async_commit();
    }
    const T* S = stages + (u % NST) * SE;
    const T* V = S + ST_UNIT;
    auto term = [&](int q) {
      const T l = FWD ? S[q * 65 + x] : S[x * 33 + q];
      T v[NR];
      lds_row<T, NR>(V + q * NR, v);
#pragma unroll
      for (int c = 0; c < NR; ++c) acc[c] = F::fma_(l, v[c], acc[c]);
    };
    // reduction entries of the unit: columns (forward) or rows of the block
    const int nq = it.vlim - 32 * (FWD ? it.cb0 + u % it.cu : u);
    if (nq >= 32) {
#pragma unroll
      for (int k = 0; k < 8; ++k) term(8 * g + k);
    } else {
      const int qe = min(8 * g + 8, nq);
      for (int q = 8 * g; q < qe; ++q) term(q);
    }
  }
  cp_async_wait<0>();
  if (it.nunits > 0) flush(FWD ? (it.nunits - 1) / it.cu : 0);
}

// Forward: sum the column-chunk partials of (s, 64-row block r0) in chunk
// order into U.  Task (s, r0, slot0, nchunks).
template <typename T>
__global__ void __launch_bounds__(WV_NT) k_push_reduce(SolveArgs a, const int4* __restrict__ tasks) {
  using F = Field<T>;
  const int4 tk = tasks[blockIdx.x];
  const int s = tk.x, r0 = tk.y, slot0 = tk.z, nch = tk.w;
  const int off = a.sn_nrow[s] - a.sn_ncol[s];
  const int ld = a.ld, nr = a.nrhs;
  const T* part = reinterpret_cast<const T*>(a.Wp) + (long long)slot0 * 64 * ld;
  T* Us = reinterpret_cast<T*>(a.U) + a.c0 + a.uoff[s] * ld;
  for (int e = threadIdx.x; e < 64 * nr; e += WV_NT) {
    const int r = e / nr, c = e - r * nr;
    if (r0 + r >= off) continue;
    T v = part[(long long)r * ld + c];
#pragma unroll 8
    for (int k = 1; k < nch; ++k) v = F::add(v, part[((long long)k * 64 + r) * ld + c]);
    Us[(long long)(r0 + r) * ld + c] = v;
  }
}

// ---------------------------------------------------------------------------
// Chain items (s, direction | 2 column group, block i, -); direction 0 = forward, 1 = backward.
// ---------------------------------------------------------------------------

// Wait until *p is published; false on timeout or abort.
template <typename T>
__device__ __forceinline__ bool wv_wait(const T* p, T& v, int* state) {
  for (long it = 0; it < WV_POLL_LIMIT; ++it) {
    if (ld_published(p, v)) return true;
    if ((it & 15) == 15 && ld_volatile(state + WV_STATE_ABORT) != 0) return false;
  }
  atomicExch(state + WV_STATE_ABORT, 1);
  atomicExch(state, 1);
  return false;
}

// Copy the 64 x 64 tile at (r0, c0) of a column-major source (rows < rlim,
// columns < clim, zero elsewhere) into S[c * 65 + r].
template <typename T>
__device__ __forceinline__ void ch_issue(T* S, const T* src, long long ld, int r0, int rlim, int c0, int clim) {
#pragma unroll
  for (int m = 0; m < 4096 / WV_NT; ++m) {
    const int e = threadIdx.x + WV_NT * m;
    const int r = e & 63, c = e >> 6;
    if (c0 + c >= clim) break;  // (the same for a warp's lanes; columns past the block are not used)
    const bool ok = r0 + r < rlim;
    const T* g = ok ? src + (r0 + r) + (long long)(c0 + c) * ld : src;
    cp_async_zfill<sizeof(T)>(S + c * 65 + r, g, ok);
  }
}

// acc[c] += sum over the thread's 16 reduction entries of the 64 x 64 tile
// S (forward: S[q * 65 + x] = A[x, q]; backward: S[x * 65 + q] = A[q, x])
// times V[q * nr + c], q < nq.
template <typename T, bool FWD, int NR>
__device__ __forceinline__ void ch_tile_mv(T (&acc)[NR], const T* S, const T* V, int x, int g, int nq) {
  using F = Field<T>;
  auto term = [&](int q) {
    const T l = FWD ? S[q * 65 + x] : S[x * 65 + q];
    T v[NR];
    lds_row<T, NR>(V + q * NR, v);
#pragma unroll
    for (int c = 0; c < NR; ++c) acc[c] = F::fma_(l, v[c], acc[c]);
  };
  if (nq >= TB) {
#pragma unroll
    for (int k = 0; k < 16; ++k) term(16 * g + k);
  } else {  // a narrow block (most leaves have one to a few columns)
    const int qe = min(16 * g + 16, nq);
    for (int q = 16 * g; q < qe; ++q) term(q);
  }
}

// gw: right-hand-side columns per chain group (CH_NR, or every column of the
// pass for the levels whose items already fill the GPU: one CTA per block
// then reads the block's inverse and dependency tiles once).
template <typename T, bool FWD, int NR>
__global__ void __launch_bounds__(WV_NT) k_chain(SolveArgs a, const int4* __restrict__ tasks, int ctr, int gw) {
  using F = Field<T>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int sh_t;
  const int ld = a.ld;
  T* S = reinterpret_cast<T*>(smem_raw);  // dependency tile; later the slice partials (4 x NR x 65)
  T* red = S;
  T* Lv = S + CH_UNIT;                    // the inverse block
  T* Vs = Lv + CH_UNIT;                   // 64 x NR
  T* wv = Vs + 64 * NR;                   // 64 x NR
  const int tid = threadIdx.x, x = tid & 63, g = tid >> 6;
  if (tid == 0) sh_t = atomicAdd(a.wstate + WV_STATE_CTR + ctr, 1);
  __syncthreads();
  if (ld_volatile(a.wstate + WV_STATE_ABORT) != 0) return;
  const int4 tk = tasks[sh_t];
  const int s = tk.x, i = tk.z;
  // column group: columns [cg0, cg0 + nr) of the pass; a group with no
  // columns in this pass has nothing to do (its dependents are in the same
  // group)
  const int cg0 = gw * (tk.y >> 1);
  const int nr = min(gw, a.nrhs - cg0);
  if (nr <= 0) return;
  const int first = a.sn_first[s], ncol = a.sn_ncol[s], nrow = a.sn_nrow[s];
  const int nblk = (ncol + TB - 1) / TB, nb = min(TB, ncol - i * TB);
  const T* L = reinterpret_cast<const T*>(a.panel) + a.sn_poff[s];
  const T* Li = reinterpret_cast<const T*>(a.linv) + a.linv_off[s] + (long long)i * TB * TB;
  T* Ze = reinterpret_cast<T*>(a.Ze) + a.c0 + cg0 + (long long)first * ld;
  // dependency blocks in chain order: step u is block dep(u)
  const int nd = FWD ? i : nblk - 1 - i;
  auto dep = [&](int u) { return FWD ? u : nblk - 1 - u; };
  auto issue = [&](int u) {
    const int j = dep(u);
    if (FWD) ch_issue<T>(S, L, nrow, i * TB, ncol, j * TB, ncol);
    else ch_issue<T>(S, L, nrow, j * TB, ncol, i * TB, ncol);
    // the tile after it into L2 (one tile fits in shared memory)
    if (u + 1 < nd) {
      const int jn = dep(u + 1);
      const int pr = FWD ? i * TB : jn * TB, pc = FWD ? jn * TB : i * TB;
      constexpr int LPC = TB * (int)sizeof(T) / 128;  // cache lines of a tile column
      for (int e = tid; e < TB * LPC; e += WV_NT) {
        const int c = pc + e / LPC, r = pr + (e % LPC) * (128 / (int)sizeof(T));
        if (c < ncol && r < ncol)
          asm volatile("prefetch.global.L2 [%0];" ::"l"(L + r + (long long)c * nrow));
      }
    }
  };
  ch_issue<T>(Lv, Li, ncol <= TB ? ncol : TB, 0, nb, 0, nb);
  if (nd > 0) issue(0);
  cp_async_commit();
  // block vector.  Forward: y_i, gathered here — the right-hand side at
  // g = first + lperm[p] minus every push that lands on g, in update-list
  // order (the pull list of g, built at analysis; the pushes are final
  // before this launch), so no separate gather pass.  Backward: w_i - W_i
  // (W_i = off-diagonal dots; for a supernode whose dots were split into
  // row chunks, the chunk partials summed here in chunk order).
  const T* Wb = (!FWD && nrow > ncol) ? reinterpret_cast<const T*>(a.Wb) + a.c0 + cg0 + (long long)first * ld : nullptr;
  const T* Wd = reinterpret_cast<const T*>(a.Yg) + a.c0 + cg0 + (long long)first * ld;  // backward: D^-1 z
  const int2 dred = FWD ? make_int2(0, 0) : a.dots_red[s];
  const T* Wpart = reinterpret_cast<const T*>(a.Wp) + (long long)(dred.x + i * dred.y) * 64 * ld + cg0;
  for (int e = tid; e < 64 * NR; e += WV_NT) {
    const int r = e / NR, c = e % NR;
    T v = F::zero();
    if (r < nb && c < nr) {
      if constexpr (FWD) {
        const int gg = first + a.lperm[first + i * TB + r];
        const T* Uc = reinterpret_cast<const T*>(a.U) + a.c0 + cg0 + c;
        v = reinterpret_cast<const T*>(a.Yg)[a.c0 + cg0 + (long long)gg * ld + c];
        const int t0 = a.pull_ptr[gg], t1 = a.pull_ptr[gg + 1];
#pragma unroll 8
        for (int t = t0; t < t1; ++t) v = F::sub(v, Uc[(long long)a.pull_src[t] * ld]);
      } else {
        v = Wd[(long long)(i * TB + r) * ld + c];
        if (dred.y > 1) {
          T w = Wpart[(long long)r * ld + c];
#pragma unroll 8
          for (int q = 1; q < dred.y; ++q) w = F::add(w, Wpart[((long long)q * 64 + r) * ld + c]);
          v = F::sub(v, w);
        } else if (Wb) {
          v = F::sub(v, Wb[(long long)(i * TB + r) * ld + c]);
        }
      }
    }
    wv[e] = v;
  }
  T acc[NR];
#pragma unroll
  for (int c = 0; c < NR; ++c) acc[c] = F::zero();
#pragma unroll 1
  for (int u = 0; u < nd; ++u) {
    const int j = dep(u);
    bool bad = false;
    if (nd - u > 2) {
      // not next in line: one thread waits, so that the blocks far behind
      // leave the values' cache lines to the ones about to use them
      T v;
      if (tid == 0) bad = !wv_wait(Ze + (long long)(min((j + 1) * TB, ncol) - 1) * ld, v, a.wstate);
      if (__syncthreads_or(bad)) return;
    }
    for (int e = tid; e < 64 * NR; e += WV_NT) {
      const int r = e / NR, c = e % NR;
      T v = F::zero();
      if (!bad && c < nr && j * TB + r < ncol) bad = !wv_wait(Ze + (long long)(j * TB + r) * ld + c, v, a.wstate);
      Vs[e] = v;
    }
    cp_async_wait<0>();
    if (__syncthreads_or(bad)) return;  // tile u and block j are here
    ch_tile_mv<T, FWD, NR>(acc, S, Vs, x, g, min(TB, ncol - j * TB));
    __syncthreads();  // tile and right-hand sides consumed
    if (u + 1 < nd) issue(u + 1);
    cp_async_commit();
  }
  cp_async_wait<0>();
  // wv -= sum of the slice partials, then the inverse block
  store_partials<T, NR>(red, acc, x, g);
#pragma unroll
  for (int c = 0; c < NR; ++c) acc[c] = F::zero();
  __syncthreads();
  for (int e = tid; e < 64 * NR; e += WV_NT) {
    const int r = e / NR, c = e % NR;
    wv[e] = (r < nb && c < nr) ? F::sub(wv[e], slice_sum<T, NR>(red, r, c)) : F::zero();
  }
  __syncthreads();
  ch_tile_mv<T, FWD, NR>(acc, Lv, wv, x, g, nb);
  store_partials<T, NR>(red, acc, x, g);
  __syncthreads();
  for (int e = tid; e < 64 * nr; e += WV_NT) {
    const int r = e / nr, c = e - r * nr;
    if (r >= nb) continue;
    const T v = slice_sum<T, NR>(red, r, c);
    st_published(Ze + (long long)(i * TB + r) * ld + c, v);
    if (!FWD) {
      T* Xw = reinterpret_cast<T*>(a.Xg) + a.c0 + cg0;
      Xw[(long long)(first + a.lperm[first + i * TB + r]) * ld + c] = v;
    }
  }
}

}  // namespace rsd
