// Bunch-Kaufman factorization of one panel block and its deep rows.
//
//   k_getf2  one CTA per block: unblocked BK over panel columns [kb, ke),
//            every pivot candidate, update and interchange bounded to rows
//            < ke (ll_cdiv_emit getf2);
//   k_deep   the block's pivot steps on the rows below it
//            (apply_bk_panel_trailing), as a triangular solve.
//
// k_getf2.  A step of the factorization is a short dependent chain (column,
// pivot test, reciprocal, multipliers), so the block lives in REGISTERS and
// the chain is kept to one shared-memory round trip and one block barrier:
// G x G threads own the lower triangle cyclically (thread (tx, ty) holds the
// entries (ty + G ii, tx + G jj), slots ii >= jj).  The warp that owns column
// k + 1 updates it first, in its registers, tests step k + 1 (vote on the
// squared moduli against alpha^2 |a_kk|^2, with a margin far above rounding;
// the reciprocal overlaps the vote), and publishes the column and its
// multipliers; then it applies the rest of step k like every other warp.
// Steps that the margin does not decide are decided by warp 0 with the
// reference's expressions; those that need the row maximum (and so possibly
// an interchange or a 2x2 pivot) have the candidate column and column k + 1
// written to shared memory, warp 0 composes the post-interchange columns, and
// the owners of the interchanged row and column reload them.  Every entry
// sees the operations of the reference in its order, so with EXACT (the FMA
// engine) the factor is the oracle's bit for bit in every field; the tensor
// engine, whose products are summed in tiles anyway, takes fused updates and
// one division per complex reciprocal, except in real f64 (see minus_prod and
// kSumUpdates for how its updates round).  The finished columns collect in
// shared memory (packed lower triangle).
// Measured (B200), a diagonally dominant block on one CTA, FMA engine / fused:
// 64 columns of f64 31 / 27 us, f32 28 / 25, c64 61 / 41, c32 43 / 35; 128
// columns of f64 49 / 41, f32 40 / 35, c64 111 / 80, c32 62 / 52 (0.4 to 0.7 us
// a step; an indefinite block of random entries twice that).  A shared-memory
// block with per-step trailing updates took 2.4 us a step.  All panel launches
// of a refactor: 128^2 f64 4.65 -> 1.70 ms, 64^3 c32 20.3 -> 10.1 ms.
//
// k_deep.  The interchanges of a block permute its columns before any step
// touches a deep row, so the replay is X = (X P) L^-T D^-1 with the final L:
// no step-by-step interchange is left.  Eight lanes hold one row (column t +
// 8 s in slot s); a step is one shuffle of x_k and one multiply-subtract per
// later slot, L read from shared memory.  Bound by that chain (64 steps); it
// needs no separate block transform: deep rows of a 64^3 c32 refactor 11.1 ->
// 5.6 ms in 169 launches instead of 334.
// Reference: src/numeric/multifrontal_ldlt.rs:2400-3256.
#pragma once

#include <type_traits>
#include <utility>

#include "factor_kernels.cuh"

namespace rsd {

// Thread grids and slot counts of the k_getf2 instances: blocks of at most
// 32 columns on 64 threads (many CTAs per SM), at most 64 and at most 128
// columns on 256 threads.
constexpr int GF_NARROW_G = 8, GF_G = 16;
constexpr int GF_NARROW_PW = 32, GF_MID_PW = 64, GF_WIDE_PW = 128;
constexpr int GF_NARROW_MIN = 2 * 148;  // narrow blocks of a level that get a launch of their own

// CTAs per SM that the instances are compiled for.
__host__ __device__ constexpr int getf2_minb(int g, int ns, size_t es) {
  return g == GF_NARROW_G ? (es >= 16 ? 6 : 8) : (ns <= 4 && es < 16) ? 2 : 1;
}

__host__ __device__ constexpr size_t gf_align16(size_t b) { return (b + 15) & ~size_t(15); }

// Shared memory of k_getf2 for blocks of at most pwm columns: the packed L
// (padded: the triangular solve reads up to 8 entries past a column), two
// sets of published columns (u1, u2), the candidate columns (v2, v3)
// and the replaced column, D, the inverse pivots, the control words and the
// interchange bookkeeping.
__host__ __device__ constexpr size_t gf_packed(int pwm) { return (size_t)pwm * (pwm + 1) / 2 + 16; }
__host__ __device__ constexpr size_t smem_getf2(size_t es, int pwm) {
  return gf_align16(gf_packed(pwm) * es) + ((size_t)(4 + 3 + 3) * pwm + 4) * es + 64 + 4 * (size_t)pwm * 4 + pwm + 16;
}
// Shared memory of k_deep: the packed L, D, dsub, the inverse pivots, the
// column permutation and the pivot kinds.
__host__ __device__ constexpr size_t smem_deep(size_t es, int pwm) {
  return gf_align16(gf_packed(pwm) * es) + (size_t)3 * pwm * es + (size_t)pwm * 4 + pwm + 16;
}

// Packed start of column j minus j: entry (i, j), i >= j, at pk_col(j, pw) + i.
__device__ __forceinline__ int pk_col(int j, int pw) { return j * pw - (j * (j - 1)) / 2 - j; }

// c ? x : y as a value (a conditional on array elements is a conditional on
// their addresses, which would put a register array into local memory).
template <typename T>
__device__ __forceinline__ T sel(bool c, T x, T y) {
  if constexpr (Field<T>::complex)
    return T{c ? x.re : y.re, c ? x.im : y.im};
  else
    return c ? x : y;
}

// fn(0), fn(1), ... with the index as a compile-time constant.
template <typename Fn, int... J>
__device__ __forceinline__ void for_each_int(Fn&& fn, std::integer_sequence<int, J...>) {
  (fn(std::integral_constant<int, J>{}), ...);
}

// The panel kernel's quick tests compare squared moduli formed with fused
// operations in the field's own precision; a relative margin far above the
// rounding (of the squares and of the reference's moduli) separates sure
// outcomes from the ones left to the reference's expressions.
template <typename R> struct QuickTest;
template <> struct QuickTest<double> {
  static constexpr double margin = 1e-9, lo = 1e-140, hi = 1e140;
};
template <> struct QuickTest<float> {
  static constexpr float margin = 1e-4f, lo = 1e-15f, hi = 1e15f;
};
template <typename T>
__device__ __forceinline__ typename Field<T>::Real quick2(T x) {
  if constexpr (Field<T>::complex)
    return fma(x.re, x.re, x.im * x.im);
  else
    return x * x;
}
// 1 / a, correctly rounded (Field::recip's value, without the general division).
__device__ __forceinline__ double panel_recip(double a) { return __drcp_rn(a); }
__device__ __forceinline__ float panel_recip(float a) { return __frcp_rn(a); }
template <typename R>
__device__ __forceinline__ cplx<R> panel_recip(cplx<R> a) {
  return Field<cplx<R>>::recip(a);
}

// u w, rounded at its own magnitude (one rounding in a component's first
// product, one in the sum).
template <typename T>
__device__ __forceinline__ T product(T u, T w) {
  if constexpr (Field<T>::complex)
    return T{fma(-u.im, w.im, u.re * w.re), fma(u.re, w.im, u.im * w.re)};
  else
    return u * w;
}
// e - u w: the reference's multiply and subtract, each rounded (zero
// multipliers skipped, as there), or fused.  The fused complex form rounds e
// once: two fused operations in a row on e round it twice, which lost 1.3 to
// 2.2 times the reference's accuracy on a dominant block.
template <typename T, bool EXACT>
__device__ __forceinline__ T minus_prod(T e, T u, T w) {
  using F = Field<T>;
  if constexpr (EXACT)
    return sel(F::is_zero(w), e, F::sub(e, F::mul(u, w)));
  else if constexpr (F::complex)
    return F::sub(e, product(u, w));
  else
    return F::fnma(u, w, e);
}
// Whether the updates of an entry are summed by themselves and subtracted from
// it once, when its column is due, instead of one after another: the c32
// instances of the tensor engine.  A sum of updates is smaller than the entry
// of a dominant matrix and so are its roundings: residual of a 64-column block
// a fifth, error of the refined 27-point sweep (24^3, lowest frequency) 5.8e-14
// -> 5.1e-14, for 34.1 -> 34.7 ms a 64^3 factor.  The other fields reach the
// accuracy of their sequential reference without it.
template <typename T, bool EXACT>
inline constexpr bool kSumUpdates = !EXACT && std::is_same_v<T, c32>;
// 1 / a for the multipliers of every 1x1 step, whichever path decides it (a
// replay takes a recorded step in place on the quick path even where the
// search needed the row maximum): the reference's two divisions of a complex
// reciprocal, or one reciprocal of |a|^2.
template <typename T, bool EXACT>
__device__ __forceinline__ T step_recip(T a) {
  if constexpr (EXACT || !Field<T>::complex) {
    return panel_recip(a);
  } else {
    const auto r = panel_recip(quick2(a));
    return T{a.re * r, -a.im * r};
  }
}

// Inverse of the pivot block that starts at position k (1x1: 1 / d; 2x2:
// 1 / (d11 d22 - d21^2); zero for the second position of a 2x2).
template <typename T>
__device__ __forceinline__ T pivot_inverse(unsigned char kd, T d, T ds, T dn) {
  using F = Field<T>;
  if (kd == 0) return panel_recip(d);
  if (kd == 1) return panel_recip(F::sub(F::mul(d, dn), F::mul(ds, ds)));
  return F::zero();
}

// Deep rows [r_begin, r_end) of panel columns [kb, kb + pw): X := (X P) L^-T
// D^-1.  Lp = the block's packed L (shared memory), src = the composed column
// permutation (block-local), inv / dd / ds / kd the pivots.  Warps of the CTA
// take 4 rows each in turn; NSL = column slots (8 NSL >= pw).  EXACT: the
// reference's multiply and subtract, each rounded (zero multipliers skipped,
// as there); otherwise fused.
template <typename T, int NSL, bool EXACT>
__device__ __forceinline__ void deep_rows(T* panel, long long nrow, int kb, int pw, int r_begin, int r_end,
                                          const T* Lp, const int* src, const T* inv, const T* dd, const T* ds,
                                          const unsigned char* kd, bool any2) {
  using F = Field<T>;
  constexpr bool SUM = kSumUpdates<T, EXACT>;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int t = lane >> 2, r = lane & 3;
  for (int r0 = r_begin + 4 * warp; r0 < r_end; r0 += 4 * nw) {
    const int row = r0 + r;
    const bool live = row < r_end;
    auto entry = [&](int s) -> T {
      const int col = t + 8 * s;
      return (live && col < pw) ? panel[row + (long long)(kb + src[col]) * nrow] : F::zero();
    };
    T x[NSL];  // the row, or the sums of its updates until a slot's columns are due
#pragma unroll
    for (int s = 0; s < NSL; ++s) x[s] = SUM ? F::zero() : entry(s);
    T due = SUM ? entry(0) : F::zero();
#pragma unroll
    for (int s0 = 0; s0 < NSL; ++s0) {
      if (8 * s0 >= pw) break;
      if constexpr (SUM) {
        x[s0] = F::sub(due, x[s0]);
        if (s0 + 1 < NSL) due = entry(s0 + 1);
      }
      const int te = min(8, pw - 8 * s0);
      // (columns past pw read what follows in L's allocation and are not used)
#pragma unroll 2
      for (int t0 = 0; t0 < te; ++t0) {
        const T* Lk = Lp + pk_col(8 * s0 + t0, pw) + t;
        const T xk = shfl_t(x[s0], 4 * t0 + r);
#pragma unroll
        for (int s = s0; s < NSL; ++s) {
          const T l0 = Lk[8 * s];
          const T l = s > s0 ? l0 : sel(t > t0, l0, F::zero());
          x[s] = SUM && s > s0 ? F::add(x[s], product(xk, l)) : minus_prod<T, EXACT>(x[s], xk, l);
        }
      }
    }
    if (!any2) {
#pragma unroll
      for (int s = 0; s < NSL; ++s) {
        const int col = t + 8 * s;
        if (live && col < pw) panel[row + (long long)(kb + col) * nrow] = F::mul(x[s], inv[col]);
      }
    } else {
#pragma unroll
      for (int s = 0; s < NSL; ++s) {
        const int col = t + 8 * s;
        // the neighbours' values (columns col + 1 and col - 1)
        T nx = shfl_t(x[s], (lane + 4) & 31), pv = shfl_t(x[s], (lane - 4) & 31);
        const T nxw = s + 1 < NSL ? shfl_t(x[s + 1 < NSL ? s + 1 : s], r) : F::zero();
        const T pvw = s > 0 ? shfl_t(x[s > 0 ? s - 1 : 0], 28 + r) : F::zero();
        if (t == 7) nx = nxw;
        if (t == 0) pv = pvw;
        if (live && col < pw) {
          const unsigned char k = kd[col];
          T y;
          if (k == 0)
            y = F::mul(x[s], inv[col]);
          else if (k == 1)
            y = F::mul(F::sub(F::mul(dd[col + 1], x[s]), F::mul(ds[col], nx)), inv[col]);
          else
            y = F::mul(F::sub(F::mul(dd[col - 1], x[s]), F::mul(ds[col - 1], pv)), inv[col - 1]);
          panel[row + (long long)(kb + col) * nrow] = y;
        }
      }
    }
  }
}

// The instance for the block's width (NSL: the widest the caller may pass).
template <typename T, int NSL, bool EXACT, typename... A>
__device__ __forceinline__ void deep_rows_for(T* panel, long long nrow, int kb, int pw, A... rest) {
  if constexpr (NSL > 4) {
    if (pw <= 4 * NSL) {
      deep_rows_for<T, NSL / 2, EXACT>(panel, nrow, kb, pw, rest...);
      return;
    }
  }
  deep_rows<T, NSL, EXACT>(panel, nrow, kb, pw, rest...);
}

// ---------------------------------------------------------------------------
// getf2: task (s, kb, -, fuse).
// ---------------------------------------------------------------------------
template <typename T, int G, int NS, bool EXACT>
__global__ void __launch_bounds__(G * G, getf2_minb(G, NS, sizeof(T)))
    k_getf2(FactorArgs fa, const int4* __restrict__ tasks, int nb_small, int nb_big) {
  using F = Field<T>;
  constexpr int NT = G * G, NW = NT / 32, PWM = G * NS, PWS = PWM + 1;
  constexpr int NE = NS * (NS + 1) / 2;
  if (factor_failed(fa.status)) return;
  const double pfloor = fa.floor_dev ? *fa.floor_dev : fa.perturb_floor;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int4 tk = tasks[blockIdx.x];
  const int s = tk.x, kb = tk.y, fuse = tk.w;
  const int first = fa.sn_first[s], ncol = fa.sn_ncol[s], nrow = fa.sn_nrow[s];
  const int nb = ncol >= 512 ? nb_big : nb_small;
  const int ke = min(kb + nb, ncol), pw = ke - kb;
  T* panel = reinterpret_cast<T*>(fa.panel) + fa.sn_poff[s];
  const bool reuse = fa.pivot_reuse && fa.pivrec && *fa.pivot_reuse != 0;
  int* prec = fa.pivrec ? fa.pivrec + first + kb : nullptr;  // no record without a handle

  T* Lp = reinterpret_cast<T*>(smem_raw);  // packed lower pw x pw: L, the diagonal holds D
  T* pub = reinterpret_cast<T*>(smem_raw + gf_align16(gf_packed(PWM) * sizeof(T)));
  T* v2 = pub + 4 * PWS;   // candidate column
  T* v3 = v2 + PWM;        // column k + 1
  T* rep = v3 + PWM;       // the interchanged position's new row / column
  T* d_s = rep + PWM;
  T* ds_s = d_s + PWM;
  T* inv_s = ds_s + PWM;
  // control words: slow steps: [9] accepted width, [10] candidate, [11]
  // recorded width, then [4] width, [5] [7] interchange; [6] perturbed pivots,
  // [8] any 2x2, [1] moved rows
  int* ctl = reinterpret_cast<int*>(inv_s + PWM);
  double* mod_s = reinterpret_cast<double*>(ctl + 12);  // the undecided test's |a_kk| and column maximum
  int* lp_s = ctl + 16;       // the block's slice of lperm
  int* rec_s = lp_s + PWM;    // replayed pivot record
  int* supp = rec_s + PWM;    // rows moved by the interchanges
  int* src_s = supp + PWM;    // block-local lperm
  unsigned char* kd_s = reinterpret_cast<unsigned char*>(src_s + PWM);

  const int npk = pw * (pw + 1) / 2;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ty = tid % G, tx = tid / G;
  auto ix = [](int ii, int jj) constexpr { return jj * NS - jj * (jj - 1) / 2 + (ii - jj); };
  // SUM: a[] holds the sum of an entry's updates, the entry itself waits in its
  // place of the packed L, which only its thread reads or writes until its
  // column is due
  constexpr bool SUM = kSumUpdates<T, EXACT>;
  T a[NE];
#pragma unroll
  for (int jj = 0; jj < NS; ++jj)
#pragma unroll
    for (int ii = jj; ii < NS; ++ii) {
      const int i = ty + G * ii, j = tx + G * jj;
      const bool in = i < pw && i >= j;
      const T e = in ? panel[(kb + i) + (long long)(kb + j) * nrow] : F::zero();
      a[ix(ii, jj)] = SUM ? F::zero() : e;
      if (SUM && in) Lp[pk_col(j, pw) + i] = e;
    }
  if (kb == 0)
    for (int p = tid; p < ncol; p += NT) fa.lperm[first + p] = p;
  for (int i = tid; i < pw; i += NT) {
    lp_s[i] = kb + i;  // interchanges never leave a block
    ds_s[i] = F::zero();
    d_s[i] = F::zero();
    kd_s[i] = 0;
    if (reuse) {
      // (a block that no factor has finished yet may have no record, or part
      // of one: a step that reaches outside the block's remaining rows is
      // taken in place)
      const int code = prec[i], q = code < 0 ? -code - 1 : code;
      rec_s[i] = q < pw && q >= i + (code < 0) ? code : i;
    } else if (prec)
      prec[i] = i;  // a 1x1 step in place, unless slow_step records another
  }
  if (tid < 16) ctl[tid] = 0;
  __syncthreads();

  using R = typename F::Real;
  using Q = QuickTest<R>;
  const double alpha = (1.0 + sqrt(17.0)) / 8.0;
  // A quick test is only taken where the squares neither under- nor overflow,
  // and above the static-pivot floor (a floor past the range leaves no step to
  // the quick test).
  const R a2m = (R)(alpha * alpha * (1.0 + (double)Q::margin));
  const double fl2 = pfloor > 0.0 ? pfloor * pfloor * (1.0 + (double)Q::margin) : 0.0;
  const R lo2 = (R)fmin(fmax((double)Q::lo, fl2), 2.0 * (double)Q::hi);
  // x >= y for non-negative x, y: 1 / 0 where the margin decides it, -1 where
  // it does not (or a value may have under- or overflowed).
  auto quick_ge = [](double x, double y) -> int {
    if (!(x >= 1e-280 && x <= 1e280) || !(y <= 1e280)) return -1;
    return x >= y * (1.0 + 1e-9) ? 1 : x <= y * (1.0 - 1e-9) ? 0 : -1;
  };
  // The static-pivot rule of a 1x1 pivot; false = zero pivot in exact mode.
  auto perturb1 = [&](T& dk, bool count) -> bool {
    if (pfloor >= 0.0) {
      const double m = F::mag(dk);
      if (m < pfloor) {
        dk = m == 0.0 ? F::from_real(pfloor) : F::scale(dk, pfloor / m);
        if (count) ++ctl[6];
      }
      return true;
    }
    return !F::is_zero(dk);
  };
  // Slot (ii, jj) holds rows off + ty + G ii, columns off + tx + G jj: once a
  // slot column is finished the registers move one slot up, so the current
  // column is always in slot column 0 and one copy of the step's code serves
  // every step (a copy per slot column measured 1.3x slower: a block is
  // short, and each copy is fetched anew).
  int off = 0, nact = (pw + G - 1) / G;
  // SUM: the entries of column c, which will be column cx of slot column 0
  // (read ahead of the column's last update; in decide: 35.2 ms).
  auto due_entries = [&](int c, int cx, T (&e)[NS]) __attribute__((always_inline)) {
    const int lc = pk_col(c, pw);
#pragma unroll
    for (int ii = 0; ii < NS; ++ii) {
      const int r = ty + G * ii - cx;
      e[ii] = Lp[(tx == cx) & (r >= 0) & (r < pw - c) ? lc + c + r : npk];
    }
  };
  // The warp that owns column c: publish it (set `par`) with the multipliers
  // of a 1x1 pivot in place, which go straight into L.  Returns true in a lane
  // whose entries leave |a_cc| >= alpha max_i |a_ic| in doubt; such a step
  // (the block barrier collects the lanes' answers) is redone by slow_step.
  // Branch-free: lanes without a part in the column store into the padding.
  auto decide = [&](int c, int par, const T (&e)[NS]) __attribute__((always_inline)) -> bool {
    T* u1 = pub + 2 * par * PWS;
    const int cx = c - off;
    T cv[NS];  // the column
#pragma unroll
    for (int ii = 0; ii < NS; ++ii) cv[ii] = SUM ? F::sub(e[ii], a[ix(ii, 0)]) : a[ix(ii, 0)];
    const T akk = shfl_t(cv[0], (cx * G + cx) & 31);
    const R akk2 = quick2(akk);
    const T dinv = step_recip<T, EXACT>(akk);
    const int rem = pw - c, lc = pk_col(c, pw);
    bool doubt = !((akk2 >= lo2) & (akk2 <= Q::hi));
    if (reuse) doubt = doubt | (rec_s[c] != c);
#pragma unroll
    for (int ii = 0; ii < NS; ++ii) {
      const int r = ty + G * ii - cx;  // row - c
      const bool mine = (tx == cx) & (r >= 0) & (r < rem);
      const T col = cv[ii], w = F::mul(col, dinv);
      // true for NaN
      const bool big = !(quick2(col) * a2m <= akk2);
      doubt = doubt | (big & mine & (r != 0) & !reuse);
      u1[mine ? c + r : PWM] = col;
      Lp[mine ? lc + c + r : npk] = sel(r == 0, akk, w);
    }
    return doubt;
  };
  // Column q of the active block (rows >= its first active row) into v.
  // (Value selects over the slots: a branch per slot would put the register
  // array into local memory.)
  auto write_col = [&](int q, T* v) {
    const int qs = (q - off) / G, qx = (q - off) % G;
#pragma unroll
    for (int ii = 0; ii < NS; ++ii) {
      T c = a[ix(ii, 0)], r = a[ix(NS - 1, ii)];  // column slot qs, row slot qs
#pragma unroll
      for (int z = 1; z <= ii; ++z) c = sel(z == qs, a[ix(ii, z)], c);
#pragma unroll
      for (int z = ii; z < NS - 1; ++z) r = sel(z == qs, a[ix(z, ii)], r);
      const int i = off + ty + G * ii, j = off + tx + G * ii;
      if (ii < nact && tx == qx && (ii > qs || (ii == qs && ty >= tx)) && (!SUM || i < pw))
        v[i] = SUM ? F::sub(Lp[pk_col(q, pw) + i], c) : c;
      if (ty == qx && (ii < qs || (ii == qs && tx < ty))) v[j] = SUM ? F::sub(Lp[pk_col(j, pw) + q], r) : r;
    }
  };
  // Row / column q of the registers := v, from position p + 1 on.
  auto read_col = [&](int q, const T* v, int p) {
    const int qs = (q - off) / G, qx = (q - off) % G;
#pragma unroll
    for (int jj = 0; jj < NS; ++jj)
#pragma unroll
      for (int ii = jj; ii < NS; ++ii) {
        T e = a[ix(ii, jj)];
        const T vc = v[min(off + ty + G * ii, PWM - 1)], vr = v[min(off + tx + G * jj, PWM - 1)];
        const bool inc = tx == qx && jj == qs && (ii > jj || ty >= tx);
        const bool inr = ty == qx && ii == qs && (ii > jj || tx < ty);
        if constexpr (SUM) {
          const int i = off + ty + G * ii, j = off + tx + G * jj;
          a[ix(ii, jj)] = sel(inc || inr, F::zero(), e);
          if ((inc || inr) && i < pw && j > p) Lp[pk_col(j, pw) + i] = inr ? vr : vc;
        } else {
          e = sel(inc, vc, e);
          a[ix(ii, jj)] = sel(inr, vr, e);
        }
      }
  };
  // Step c by the reference's expressions: warp 0 tests the published column;
  // a step that needs the row maximum of candidate row q (or replays a
  // recorded interchange / 2x2 step) has columns q and c + 1 written out first,
  // then warp 0 decides and composes the post-interchange columns.  Returns
  // the step's width, 0 on a failed pivot.  Every thread calls it.
  auto slow_step = [&](int c, int par) __attribute__((always_inline)) -> int {
    T *u1 = pub + 2 * par * PWS, *u2 = u1 + PWS;
    T *w1 = Lp + pk_col(c, pw), *w2 = Lp + pk_col(c + 1, pw);
    if (warp == 0) {
      const T akk = u1[c];
      bool err = false, accept;
      int cand = c, forced = 0;
      if (reuse) {
        // the recorded step: no search (a zero pivot is still caught below)
        const int code = rec_s[c];
        cand = code < 0 ? -code - 1 : code;
        forced = code < 0 ? 2 : 1;
        accept = forced == 1 && cand == c;
      } else {
        double v = -1.0;
        int idx = INT_MAX;
#pragma unroll
        for (int z = 0; z < (PWM + 31) / 32; ++z) {
          const int i = c + 1 + lane + 32 * z;
          const double m = F::mag2(u1[min(i, pw - 1)]);
          if ((i < pw) & (m > v)) {
            v = m;
            idx = i;
          }
        }
        warp_argmax(v, idx);
        cand = v > 0.0 ? idx : c;
        const double akk2 = F::mag2(akk);
        const int t = quick_ge(akk2, alpha * alpha * v);
        if (t >= 0) {
          accept = t != 0;
        } else {
          const double absakk = F::mag(akk), colmax = sqrt(v > 0.0 ? v : 0.0);
          if (fmax(absakk, colmax) == 0.0) {
            err = pfloor < 0.0;
            accept = true;
          } else {
            accept = absakk >= alpha * colmax;
          }
        }
        if (lane == 0) {
          mod_s[0] = akk2;
          mod_s[1] = v;
        }
      }
      if (accept) {
        T dk = akk;
        if (!err) err = !perturb1(dk, lane == 0);
        const T dinv = step_recip<T, EXACT>(dk);
        for (int i = c + 1 + lane; i < pw; i += 32) w1[i] = F::mul(u1[i], dinv);
        if (lane == 0) w1[c] = dk;
      }
      if (lane == 0) {
        ctl[9] = accept ? (err ? 0 : 1) : -1;
        ctl[10] = cand;
        ctl[11] = forced;
      }
    }
    __syncthreads();
    if (ctl[9] >= 0) return ctl[9];
    const int q = ctl[10], forced = ctl[11];
    write_col(q, v2);
    if (q != c + 1) write_col(c + 1, v3);
    __syncthreads();
    if (warp == 0) {
      constexpr int NZ = (PWM + 31) / 32;  // rows per lane
      int kstep = 1, kp = c;
      bool err = false;
      if (forced) {
        kstep = forced;
        kp = q;
      } else {
        double rmx = -1.0;
        int idx = 0;
#pragma unroll
        for (int z = 0; z < NZ; ++z) {
          const int i = c + lane + 32 * z;
          const double m = F::mag2(i == c ? u1[q] : v2[min(i, pw - 1)]);  // (column c is published, not written out)
          if ((i < pw) & (i != q) & (m > rmx)) rmx = m;
        }
        warp_argmax(rmx, idx);
        const double akk2 = mod_s[0], v = mod_s[1], aqq2 = F::mag2(v2[q]);
        // |a_cc| >= alpha colmax (colmax / rowmax), |a_qq| >= alpha rowmax
        int t1 = quick_ge(akk2 * rmx, alpha * alpha * v * v), t2 = quick_ge(aqq2, alpha * alpha * rmx);
        if (t1 < 0 || (t1 == 0 && t2 < 0)) {
          const double rowmax = sqrt(fmax(rmx, 0.0)), colmax = sqrt(v > 0.0 ? v : 0.0);
          t1 = F::mag(u1[c]) >= alpha * colmax * (colmax / rowmax);
          t2 = F::mag(v2[q]) >= alpha * rowmax;
        }
        kstep = (t1 | t2) ? 1 : 2;
        kp = t1 ? c : q;
        if (lane == 0 && prec) prec[c] = kstep == 2 ? -kp - 1 : kp;  // (1x1 in place is the default record)
      }
      const int p = kstep == 1 ? c : c + 1;
      const T v1c = u1[c], v1q = u1[q], v1p = u1[min(p, pw - 1)], v2p = v2[min(p, pw - 1)], v2q = v2[q];
      const T v3p = q != c + 1 ? v3[min(p, pw - 1)] : F::zero();
      __syncwarp();
      if (kstep == 1) {
        T dk = kp == c ? v1c : v2q;
        err = !perturb1(dk, lane == 0);
        const T dinv = step_recip<T, EXACT>(dk);
#pragma unroll
        for (int z = 0; z < NZ; ++z) {
          const int i = c + 1 + lane + 32 * z;
          if (i < pw) {
            const T o = u1[i], t = v2[i];
            const T u = sel(kp == c, o, sel(i == q, v1q, t));
            rep[i] = sel(i == q, v1c, o);
            u1[i] = u;
            w1[i] = F::mul(u, dinv);
          }
        }
        if (lane == 0) w1[c] = dk;
      } else {
        const bool sw = kp != p;
        const T a11 = v1c, d21 = sw ? v1q : v1p, a22 = v2q;
        T d11 = a11, d22 = a22;
        T det = F::sub(F::mul(d11, d22), F::mul(d21, d21));
        const double scale2 = fmax(fmax(F::mag2(d11), F::mag2(d22)), F::mag2(d21));
        const double fl0 = fmax(pfloor, 0.0) * fmax(pfloor, 0.0);
        if (quick_ge(F::mag2(det), fmax(1e-28 * scale2 * scale2, fl0 * fl0)) == 1) {
          // well above the growth and static floors
        } else {
        const double scale = fmax(fmax(F::mag(d11), F::mag(d22)), F::mag(d21));
        const double growth_floor = 1e-14 * scale * scale;
        if (pfloor >= 0.0) {
          const double fl = fmax(pfloor * pfloor, growth_floor);
          if (F::mag(det) < fl) {
            const double lift = fmax(pfloor, scale * sqrt(1e-14));
            d11 = F::add(d11, F::from_real(lift));
            d22 = F::add(d22, F::from_real(lift));
            det = F::sub(F::mul(d11, d22), F::mul(d21, d21));
            if (F::mag(det) < fl) det = F::add(det, F::from_real(fl));
            if (lane == 0) ++ctl[6];
          }
        } else if (F::mag(det) <= growth_floor) {
          err = true;
        }
        }
        const T detinv = panel_recip(det);
#pragma unroll
        for (int z = 0; z < NZ; ++z) {
          const int i = c + 2 + lane + 32 * z;
          if (i < pw) {
            const T x1 = sel(sw && i == q, v1p, u1[i]), x2 = sel(sw && i == q, v2p, v2[i]);
            rep[i] = sel(i == q, v3p, v3[i]);
            u1[i] = x1;
            u2[i] = x2;
            w1[i] = F::mul(F::sub(F::mul(d22, x1), F::mul(d21, x2)), detinv);
            w2[i] = F::mul(F::sub(F::mul(d11, x2), F::mul(d21, x1)), detinv);
          }
        }
        if (lane == 0) {
          w1[c] = a11;
          w1[c + 1] = F::zero();  // the coupling lives in dsub only
          w2[c + 1] = a22;
          d_s[c] = d11;
          ds_s[c] = d21;
          d_s[c + 1] = d22;
          kd_s[c] = 1;
          kd_s[c + 1] = 2;
          ctl[8] = 1;
        }
      }
      if (lane == 0) {
        if (kp != p) {
          const int lpv = lp_s[p];
          lp_s[p] = lp_s[q];
          lp_s[q] = lpv;
        }
        ctl[4] = err ? 0 : kstep;
        ctl[5] = p;
        ctl[7] = kp;
      }
    }
    __syncthreads();
    const int kstep = ctl[4], p = ctl[5], kp = ctl[7];
    if (kp != p) {
      read_col(kp, rep, p);
      // rows p, kp of the finished columns (one warp throughout, so the
      // interchanges stay ordered)
      if (warp == NW - 1)
        for (int jj = lane; jj < c; jj += 32) {
          const int b = pk_col(jj, pw);
          const T t = Lp[b + p];
          Lp[b + p] = Lp[b + kp];
          Lp[b + kp] = t;
        }
    }
    return kstep;
  };

  // One step's update of an entry (of its sum).
  auto step_update = [](T e, T u, T w) -> T { return SUM ? F::fma_(u, w, e) : minus_prod<T, EXACT>(e, u, w); };
  bool failed = false;
  auto shift = [&]() __attribute__((always_inline)) {
#pragma unroll
    for (int jj = 0; jj + 1 < NS; ++jj)
#pragma unroll
      for (int ii = jj; ii + 1 < NS; ++ii) a[ix(ii, jj)] = a[ix(ii + 1, jj + 1)];
    off += G;
    --nact;
  };
  for (int k = -1, par = 1;;) {
    // the first column, or a step by the reference's expressions
    int kn = 0;
    if (k >= 0) {
      const int kstep = slow_step(k, par);
      if (kstep == 0) {
        failed = true;
        break;
      }
      kn = k + kstep;
      const T *u1 = pub + 2 * par * PWS, *u2 = u1 + PWS;
      const T *w1 = Lp + pk_col(k, pw), *w2 = Lp + pk_col(k + 1, pw);
#pragma unroll
      for (int ii = 0; ii < NS; ++ii)
        if (ii < nact) {
          const T x = u1[off + ty + G * ii], x2 = u2[off + ty + G * ii];
#pragma unroll
          for (int jj = 0; jj < NS; ++jj)
            if (jj <= ii) {
              const T e = a[ix(ii, jj)], w = w1[off + tx + G * jj], wb = w2[off + tx + G * jj];
              const T v = step_update(e, x, w);
              const T vb = EXACT ? F::sub(F::sub(e, F::mul(x, w)), F::mul(x2, wb)) : step_update(v, x2, wb);
              a[ix(ii, jj)] = sel(kstep == 2, vb, v);
            }
        }
    }
    if (kn >= pw) break;
    if (kn - off >= G) shift();
    bool doubt = false;
    T due[NS] = {};
    if (warp == ((kn - off) * G) >> 5) {
      if constexpr (SUM) due_entries(kn, kn - off, due);
      doubt = decide(kn, par ^ 1, due);
    }
    par ^= 1;
    k = kn;
    // runs of 1x1 pivots in place
    bool slow = __syncthreads_or(doubt) != 0;
    while (!slow) {
      if (++k >= pw) break;
      // (slots past the block read whatever follows in shared memory and
      // update entries that nothing reads)
      const T* u1 = pub + 2 * par * PWS + off + ty;
      const T* w1 = Lp + pk_col(k - 1, pw) + off + tx;
      const bool bnd = k - off == G;  // slot column 0 is finished
      const int cx = bnd ? 0 : k - off;
      const bool owner = warp == (cx * G) >> 5;
      if constexpr (SUM)
        if (owner) due_entries(k, cx, due);
      T ur[NS], wc[NS];
#pragma unroll
      for (int ii = 0; ii < NS; ++ii) {
        ur[ii] = u1[G * ii];
        wc[ii] = w1[G * ii];
      }
      auto upd = [&](int ii, int jj) __attribute__((always_inline)) {
        a[ix(ii, jj)] = step_update(a[ix(ii, jj)], ur[ii], wc[jj]);
      };
      // the columns beyond slot column 0 (rows past the block are skipped
      // where that saves more than the branch)
      auto upd_rest = [&]() __attribute__((always_inline)) {
#pragma unroll
        for (int ii = 1; ii < NS; ++ii)
          if ((NS <= 4 && sizeof(T) < 16) || ii < nact) {
#pragma unroll
            for (int jj = 1; jj < NS; ++jj)
              if (jj <= ii) upd(ii, jj);
          }
      };
#pragma unroll
      for (int ii = 0; ii < NS; ++ii) upd(ii, 0);
      par ^= 1;
      if (bnd) {
        upd_rest();
        shift();
      }
      doubt = false;
      if (owner) doubt = decide(k, par, due);
      if (!bnd) upd_rest();
      slow = __syncthreads_or(doubt) != 0;
    }
    if (!slow) break;
  }
  __syncthreads();

  // D, kinds and the pivot order
  for (int i = tid; i < pw; i += NT) {
    if (kd_s[i] == 0) d_s[i] = Lp[pk_col(i, pw) + i];
    // (the deep rows' inverse of a 2x2 block is that of the stored D)
    inv_s[i] = pivot_inverse<T>(kd_s[i], d_s[i], ds_s[i], kd_s[i] == 1 ? d_s[i + 1] : F::zero());
    reinterpret_cast<T*>(fa.d)[first + kb + i] = d_s[i];
    reinterpret_cast<T*>(fa.dsub)[first + kb + i] = ds_s[i];
    fa.kind[first + kb + i] = kd_s[i];
    fa.lperm[first + kb + i] = lp_s[i];
    src_s[i] = lp_s[i] - kb;
  }
  if (failed) {
    if (tid == 0 && atomicCAS(&fa.status[0], 0, 1) == 0) fa.status[1] = s;
    return;
  }
  if (tid == 0 && ctl[6]) atomicAdd(&fa.status[2], ctl[6]);
  for (int j = warp; j < pw; j += NW) {
    const T* Lj = Lp + pk_col(j, pw);
    for (int i = j + lane; i < pw; i += 32) panel[(kb + i) + (long long)(kb + j) * nrow] = Lj[i];
  }
  // rows moved by the interchanges, in order (warp 0)
  if (warp == 0) {
    int m = 0;
    for (int b = 0; b < pw; b += 32) {
      const bool mv = b + lane < pw && lp_s[b + lane] != kb + b + lane;
      const unsigned bal = __ballot_sync(0xffffffffu, mv);
      if (mv) supp[m + __popc(bal & ((1u << lane) - 1u))] = b + lane;
      m += __popc(bal);
    }
    if (lane == 0) ctl[1] = m;
  }
  __syncthreads();
  // The interchanges on the rows' left segments (columns [0, kb)): only the
  // moved rows are copied, in column chunks whose loads are all in flight
  // before the barrier that precedes the stores.
  const int nmv = ctl[1];
  if (nmv > 0 && kb > 0) {
    constexpr int PER = 8;  // elements per thread per chunk
    const int cols = max(1, (NT * PER) / nmv);
    for (int j0 = 0; j0 < kb; j0 += cols) {
      const int jn = min(cols, kb - j0);
      T v[PER];
#pragma unroll
      for (int u = 0; u < PER; ++u) {
        const int idx = tid + u * NT;
        if (idx < nmv * jn) {
          const int r = supp[idx % nmv], j = j0 + idx / nmv;
          v[u] = panel[(kb + src_s[r]) + (long long)j * nrow];
        }
      }
      __syncthreads();
#pragma unroll
      for (int u = 0; u < PER; ++u) {
        const int idx = tid + u * NT;
        if (idx < nmv * jn) {
          const int r = supp[idx % nmv], j = j0 + idx / nmv;
          panel[(kb + r) + (long long)j * nrow] = v[u];
        }
      }
      __syncthreads();
    }
  }
  if constexpr (PWM <= GF_MID_PW)  // (no launch with a wider block has fused tasks)
    if (fuse && nrow > ke)
      deep_rows_for<T, PWM / 8, EXACT>(panel, nrow, kb, pw, ke, nrow, Lp, src_s, inv_s, d_s, ds_s, kd_s, ctl[8] != 0);
}

// ---------------------------------------------------------------------------
// Deep rows of a taller panel: task (s, kb, -, r0), DEEP_R rows per task.
// ---------------------------------------------------------------------------
constexpr int DEEP_R = 32, DEEP_NT = 256;

template <typename T, int NSL, bool EXACT>
__global__ void __launch_bounds__(DEEP_NT) k_deep(FactorArgs fa, const int4* __restrict__ tasks, int nb_small,
                                                  int nb_big) {
  using F = Field<T>;
  constexpr int PWM = 8 * NSL;
  if (factor_failed(fa.status)) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int4 tk = tasks[blockIdx.x];
  const int s = tk.x, kb = tk.y, r0 = tk.w;
  const int first = fa.sn_first[s], ncol = fa.sn_ncol[s], nrow = fa.sn_nrow[s];
  const int nb = ncol >= 512 ? nb_big : nb_small;
  const int ke = min(kb + nb, ncol), pw = ke - kb;
  T* panel = reinterpret_cast<T*>(fa.panel) + fa.sn_poff[s];
  T* Lp = reinterpret_cast<T*>(smem_raw);
  T* dd = reinterpret_cast<T*>(smem_raw + gf_align16(gf_packed(PWM) * sizeof(T)));
  T* ds = dd + PWM;
  T* inv = ds + PWM;
  int* src = reinterpret_cast<int*>(inv + PWM);
  unsigned char* kd = reinterpret_cast<unsigned char*>(src + PWM);
  const int tid = threadIdx.x;
  // strictly lower L (rows fastest), every copy in flight
  for (int j = tid >> 5; j < pw; j += DEEP_NT / 32) {
    const T* g = panel + (kb) + (long long)(kb + j) * nrow;
    T* d = Lp + pk_col(j, pw);
    for (int i = j + 1 + (tid & 31); i < pw; i += 32) cp_async_zfill<sizeof(T)>(d + i, g + i, true);
  }
  cp_async_commit();
  bool two = false;
  for (int k = tid; k < pw; k += DEEP_NT) {
    const unsigned char kk = fa.kind[first + kb + k];
    const T dk = reinterpret_cast<const T*>(fa.d)[first + kb + k];
    const T dsk = reinterpret_cast<const T*>(fa.dsub)[first + kb + k];
    const T dn = kk == 1 ? reinterpret_cast<const T*>(fa.d)[first + kb + k + 1] : F::zero();
    dd[k] = dk;
    ds[k] = dsk;
    kd[k] = kk;
    src[k] = fa.lperm[first + kb + k] - kb;
    inv[k] = pivot_inverse<T>(kk, dk, dsk, dn);
    two = two || kk != 0;
  }
  cp_async_wait<0>();
  const bool any2 = __syncthreads_or(two) != 0;
  deep_rows_for<T, NSL, EXACT>(panel, nrow, kb, pw, r0, min(r0 + DEEP_R, nrow), Lp, src, inv, dd, ds, kd, any2);
}

}  // namespace rsd
