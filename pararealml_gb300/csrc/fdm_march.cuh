/*
 * Marching step kernels on 2D meshes: a warp owns a strip of columns and
 * walks it down row by row, every integrator stage (or, for single-stage
 * steps, every one of several consecutive time steps) following one row
 * behind its predecessor.
 *
 * Why: the staged kernels (fdm_step.cuh) recompute the halo of every tile
 * (four vertices on every side for RK4), move every stage value through
 * shared memory to its readers, and spend as many instructions on tile and
 * ring indexes as on the equation.  Here a stage value lives in the
 * registers of the thread that owns its column: the rows above and below
 * are the thread's own, the columns left and right come from the
 * neighbouring lanes by shuffle, there is no shared memory and no barrier,
 * and only a strip's side columns and a chunk's first rows are computed
 * twice.
 *
 * A job is one strip (U = 32 VW - 2 HL VW output columns of VW per lane, HL
 * halo lanes on each side) of one chunk of rows of one instance.  An
 * iteration reads input row i; stage s = 1 .. NP then evaluates row
 * i - s from the last three rows of stage s - 1's values.  The host sizes the chunks so
 * that the jobs fill the resident warps a whole number of times (every warp
 * of a wave then ends at the same time; see engine.StencilPlan.march_rows).
 *
 * float64 results equal the staged kernels' bit for bit (the same operations
 * in the same order).  Pairs of float32 columns in packed two-wide
 * instructions were slower (the column shifts become register moves):
 * 3.3 ms against 2.4 ms on the 64 x 257^2 case below.
 */
#pragma once

namespace prml {

template <typename T>
__device__ __forceinline__ T free_value() {
  if constexpr (sizeof(T) == 4) return __int_as_float(0x7fc00000);
  else return __hiloint2double(0x7ff80000, 0);
}

/* VW consecutive elements read through L2 only (see ld16), or stored */
template <typename T, int VW>
__device__ __forceinline__ void ld_vec(const T* a, T* d) {
  constexpr int per = 16 / (int)sizeof(T);
  if constexpr (VW % per == 0) {
#pragma unroll
    for (int q = 0; q < VW / per; ++q) ld16(a + q * per, d + q * per);
  } else if constexpr (VW == 2 && sizeof(T) == 4) {
    const float2 v = __ldcg(reinterpret_cast<const float2*>(a));
    d[0] = v.x;
    d[1] = v.y;
  } else {
#pragma unroll
    for (int q = 0; q < VW; ++q) d[q] = __ldcg(a + q);
  }
}
template <typename T, int VW>
__device__ __forceinline__ void st_vec(T* a, const T* d) {
  constexpr int per = 16 / (int)sizeof(T);
  if constexpr (VW % per == 0) {
#pragma unroll
    for (int q = 0; q < VW / per; ++q) st16(a + q * per, d + q * per);
  } else if constexpr (VW == 2 && sizeof(T) == 4) {
    *reinterpret_cast<float2*>(a) = make_float2(d[0], d[1]);
  } else {
#pragma unroll
    for (int q = 0; q < VW; ++q) a[q] = d[q];
  }
}

/* A vertex of a marching window, with the stencil operators the generated
 * right-hand sides call (Point's, operation for operation).  ER / EC: the row
 * (a column) may lie on a face of kernel axis 0 / 1.  Face values are read
 * and selected, never branched on: a branch at every face, component and
 * stage would split the warp and expose the load's latency each time. */
template <typename T, class Eq, int VW, bool ER, bool EC>
struct MarchPoint {
  using real = T;
  static constexpr int C = Eq::C;

  const T (*mid)[VW]; /* [C][VW]: row gi, gi - 1 and gi + 1 */
  const T (*up)[VW];
  const T (*dn)[VW];
  const T (*left)[3][VW];  /* [C][row]: one column to the left of row gi (row 1); rows 0 and 2 */
  const T (*right)[3][VW]; /* (gi - 1, gi + 1) only where a mixed derivative reads them */
  const T* col_neu;        /* [C]: column-face values at row gi (Eq::PRE) */
  const T* col_dir;
  const MeshC<T>* m;
  double time;
  int h;  /* column of the lane */
  int gi; /* row; inside the mesh */
  int gj; /* column; may lie outside the mesh where EC */

  __device__ __forceinline__ T v(int c, int di, int dj) const {
    if (dj < 0) return left[c][di + 1][h];
    if (dj > 0) return right[c][di + 1][h];
    return di < 0 ? up[c][h] : (di > 0 ? dn[c][h] : mid[c][h]);
  }
  template <int c> __device__ __forceinline__ T val() const { return mid[c][h]; }
  __device__ __forceinline__ T t() const { return T(time); }
  __device__ __forceinline__ int col() const { return EC ? min(max(gj, 0), m->ny - 1) : gj; }
  template <int ka> __device__ __forceinline__ T x() const {
    if constexpr (sizeof(T) == 4) return ka == 0 ? m->c0f[gi] : m->c1f[col()];
    else return ka == 0 ? T(m->c0[gi]) : T(m->c1[col()]);
  }

  static __device__ __forceinline__ constexpr bool bit(unsigned long long mask, int f, int c) {
    return (f < 2 ? ER : EC) && ((mask >> (f * C + c)) & 1ull);
  }
  /* whether the vertex, offset by (di, dj), lies on face f; the lower column
   * face only ever meets the first column of a lane */
  template <int f> __device__ __forceinline__ bool at_face(int di, int dj) const {
    if (f < 2) return gi + di == (f ? m->nx - 1 : 0);
    return (f == 2 && dj == 0) ? (h == 0 && gj == 0) : gj + dj == (f == 3 ? m->ny - 1 : 0);
  }
  /* entry of a face table at the vertex offset by (di, dj) */
  template <int f> __device__ __forceinline__ T entry(const T* tab, int c, int di, int dj) const {
    const int k = f < 2 ? min(max(gj + dj, 0), m->ny - 1) : min(max(gi + di, 0), m->nx - 1);
    return __ldg(tab + (f * C + c) * m->flen + k);
  }
  /* face f's Neumann value for component c, and whether it applies */
  template <int f, int c> __device__ __forceinline__ bool neu(int di, int dj, T& g) const {
    if (!bit(Eq::NEU_MASK, f, c)) return false;
    if constexpr (Eq::PRE && f >= 2) g = col_neu[c];
    else g = entry<f>(m->neu, c, di, dj);
    return at_face<f>(di, dj) && is_value(g);
  }

  /* constrained first derivative along kernel axis ka at the vertex offset
   * by (di, dj); zero outside the mesh when CHECK */
  template <int c, int ka, bool CHECK> __device__ __forceinline__ T grad_at(int di, int dj) const {
    T r = ka == 0 ? (v(c, di + 1, dj) - v(c, di - 1, dj)) * m->inv2d0
                  : (v(c, di, dj + 1) - v(c, di, dj - 1)) * m->inv2d1;
    T g;
    if (neu<2 * ka + 1, c>(di, dj, g)) r = g;
    if (neu<2 * ka, c>(di, dj, g)) r = g;
    if (CHECK && ((ER && (gi + di < 0 || gi + di >= m->nx)) || (EC && (gj + dj < 0 || gj + dj >= m->ny)))) r = T(0);
    return r;
  }
  template <int c, int ka> __device__ __forceinline__ T grad() const { return grad_at<c, ka, false>(0, 0); }

  /* neighbours along one axis, with the Neumann ghost vertices */
  template <int c, int ka> __device__ __forceinline__ void ends(T& prev, T& next) const {
    const int di = ka == 0 ? 1 : 0, dj = ka == 0 ? 0 : 1;
    const T lo = v(c, -di, -dj), hi = v(c, di, dj);
    const T twod = ka == 0 ? m->twod0 : m->twod1;
    prev = lo;
    next = hi;
    T g;
    if (neu<2 * ka, c>(0, 0, g)) prev = hi - twod * g;
    if (neu<2 * ka + 1, c>(0, 0, g)) next = lo + twod * g;
  }
  template <int c, int ka> __device__ __forceinline__ T sd() const {
    T prev, next;
    ends<c, ka>(prev, next);
    return ((next - T(2) * mid[c][h]) + prev) * (ka == 0 ? m->invdd0 : m->invdd1);
  }
  template <int c> __device__ __forceinline__ T lap() const {
    T p0, n0, p1, n1;
    ends<c, 0>(p0, n0);
    ends<c, 1>(p1, n1);
    if constexpr (Eq::EQUAL_DX) return fmaT(T(-4), mid[c][h], (n0 + p0) + (n1 + p1)) * m->invdd0;
    else
      return fmaT(fmaT(T(-2), mid[c][h], n0 + p0), m->invdd0,
                  fmaT(T(-2), mid[c][h], n1 + p1) * m->invdd1);
  }
  template <int c> __device__ __forceinline__ T lapr() const {
    T p0, n0, p1, n1;
    ends<c, 0>(p0, n0);
    ends<c, 1>(p1, n1);
    return fmaT(T(-4), mid[c][h], (n0 + p0) + (n1 + p1));
  }
  __device__ __forceinline__ T inv_dd() const { return m->invdd0; }
  template <int c, int a1, int a2> __device__ __forceinline__ T hess() const {
    if constexpr (a1 == a2) return sd<c, a1>();
    else if constexpr (a2 == 0)
      return (grad_at<c, a1, true>(1, 0) - grad_at<c, a1, true>(-1, 0)) * m->inv2d0;
    else
      return (grad_at<c, a1, true>(0, 1) - grad_at<c, a1, true>(0, -1)) * m->inv2d1;
  }

  /* Dirichlet re-imposition (tables `d`) with the reference's face precedence */
  template <int f> __device__ __forceinline__ void fix(T& r, int c, const MeshC<T>& d) const {
    if (!bit(Eq::DIR_MASK, f, c)) return;
    T g;
    if constexpr (Eq::PRE && f >= 2) g = col_dir[c];
    else g = entry<f>(d.dir, c, 0, 0);
    if (at_face<f>(0, 0) && is_value(g)) r = g;
  }
  __device__ __forceinline__ T dirichlet(T r, int c, const MeshC<T>& d) const {
    fix<0>(r, c, d);
    fix<1>(r, c, d);
    fix<2>(r, c, d);
    fix<3>(r, c, d);
    return r;
  }
};

/* What bounds it: instruction issue and latency (float32: 226 warp instructions
 * per row of a strip for the four stages of RK4 diffusion with the face strips
 * and a chunk's first rows counted in, 55 % of the issue slots while SMs are
 * active) and the float64 pipe (82 % busy).  Measured, per 100
 * RK4 steps: 64 x 257^2 diffusion in float32 4.60 -> 2.43 ms, 16 x 257^2 in
 * float64 12.5 -> 9.1 ms (staged kernel before); 200 Cahn-Hilliard steps at
 * 1025^2 in float32 1.24 -> 0.95 ms with two steps per launch.  Three coupled
 * components in float32 run as fast staged (2.80 against 2.90 ms for 32 shallow
 * water steps at 16 x 513^2: the windows take 168 registers), so the
 * autotuner times both families.  Starting each stage two rows behind its
 * predecessor, which makes the stages of an iteration independent, cost more
 * registers than it hid latency (3.1 ms in the first case).
 *
 * NP = pipeline depth: the stages of one multi-stage step, or the most time
 * steps of one launch for single-stage steps. */
template <typename T, class Eq, int INTEG, int VW, int NP>
struct March {
  static constexpr int C = Eq::C;
  static constexpr int ND = Eq::ND;
  static constexpr int NDA = ND > 0 ? ND : 1;
  static constexpr bool MULTI = !(Eq::STAGE_INVARIANT || INTEG == FORWARD_EULER);
  static constexpr int HL = (NP + VW - 1) / VW;
  static constexpr int COLS = 32 * VW;
  static constexpr int U = COLS - 2 * HL * VW;
  /* rows read ahead: several where that is cheap in registers (short
   * iterations, whose arithmetic does not cover a load's latency) */
  static constexpr int PF = C * VW * (int)sizeof(T) <= 16 ? 3 : (C * VW * (int)sizeof(T) <= 32 ? 2 : 1);
  static_assert(!MULTI || (NP == INTEG && Eq::NYC == 0), "multi-stage marching needs dy/dt rows only");
  static constexpr int NOLD = MULTI && NP > 2 ? NP - 2 : 1;
  static_assert(!MULTI || NP <= 4, "the slopes' schedule is RK4's at most");

  const prml_step_params& p;
  const MeshC<T>& m;
  const T* in;
  T* out;
  T win[NP][C][3][VW]; /* [stage]: the last three rows, oldest first */
  T old[C][NOLD][VW];  /* the input's rows before win[0]: i - 3, .., i - NP */
  T acc[NP][NDA][VW];  /* slope sums of each stage's latest row */
  T pf[PF][C][VW];
  /* Eq::PRE: values of the column face the lane touches (NaN: none or free)
   * at rows i + 1 (read ahead), i, i - 1, .., i - NP */
  T cn[NP + 2][C], cd[NP + 2][C];
  int col_face; /* 2 / 3: the lane's columns reach the lower / upper face; 0 */
  int b, r0, r1, gj0, nsteps, slot0;
  double t0;
  T dt, acc_scale;
  bool owner; /* the lane's columns are output columns */

  __device__ __forceinline__ March(const prml_step_params& p_, const MeshC<T>& m_) : p(p_), m(m_) {}

  __device__ __forceinline__ void load_row(int i, T (&d)[C][VW]) const {
    /* a vector that starts inside the mesh stays inside the row pitch */
    const bool ok = i >= 0 && i < p.nx && i < r1 + NP && gj0 >= 0 && gj0 < p.ny;
#pragma unroll
    for (int c = 0; c < C; ++c) {
#pragma unroll
      for (int h = 0; h < VW; ++h) d[c][h] = T(0);
      if (ok) ld_vec<T, VW>(in + c * p.cstride + (long long)i * p.pitch + gj0, d[c]);
    }
  }

  static __device__ __forceinline__ constexpr bool col_bit(unsigned long long mask, int c) {
    return ((mask >> (2 * C + c)) & 1ull) || ((mask >> (3 * C + c)) & 1ull);
  }
  __device__ __forceinline__ void load_faces(int i) {
    const bool ok = col_face && i >= 0 && i < p.nx;
#pragma unroll
    for (int c = 0; c < C; ++c) {
      if (col_bit(Eq::NEU_MASK, c)) cn[0][c] = ok ? __ldg(m.neu + (col_face * C + c) * m.flen + i) : free_value<T>();
      if (col_bit(Eq::DIR_MASK, c)) cd[0][c] = ok ? __ldg(m.dir + (col_face * C + c) * m.flen + i) : free_value<T>();
    }
  }

  /* the newest row of stage s (s = 0: the input) */
  __device__ __forceinline__ void push(int s, const T (&row)[C][VW]) {
#pragma unroll
    for (int c = 0; c < C; ++c)
#pragma unroll
      for (int h = 0; h < VW; ++h) {
        win[s][c][0][h] = win[s][c][1][h];
        win[s][c][1][h] = win[s][c][2][h];
        win[s][c][2][h] = row[c][h];
      }
  }

  /* One iteration: input row i.  EDGE: some row computed here may lie on or
   * outside a face, or some stage has no valid (or no needed) row at this end
   * of the chunk; EC: columns may lie on or outside a face. */
  template <bool EDGE, bool EC>
  __device__ __forceinline__ void iterate(int i) {
    if constexpr (MULTI && NP > 2) {
#pragma unroll
      for (int c = 0; c < C; ++c)
#pragma unroll
        for (int h = 0; h < VW; ++h) {
#pragma unroll
          for (int r = NOLD - 1; r > 0; --r) old[c][r][h] = old[c][r - 1][h];
          old[c][0][h] = win[0][c][0][h];
        }
    }
    T row[C][VW];
#pragma unroll
    for (int c = 0; c < C; ++c)
#pragma unroll
      for (int h = 0; h < VW; ++h) {
        /* columns past the mesh are the reference's zero halo (the row
         * padding holds no state) */
        row[c][h] = EC && gj0 + h >= p.ny ? T(0) : pf[0][c][h];
#pragma unroll
        for (int q = 0; q + 1 < PF; ++q) pf[q][c][h] = pf[q + 1][c][h];
      }
    push(0, row);
    load_row(i + PF, pf[PF - 1]);
    if constexpr (EC && Eq::PRE) {
#pragma unroll
      for (int r = NP + 1; r > 0; --r)
#pragma unroll
        for (int c = 0; c < C; ++c) {
          if (col_bit(Eq::NEU_MASK, c)) cn[r][c] = cn[r - 1][c];
          if (col_bit(Eq::DIR_MASK, c)) cd[r][c] = cd[r - 1][c];
        }
      load_faces(i + 1);
    }

    T carry[NDA][VW]; /* the predecessor's slope sums of this row, from the iteration before */
#pragma unroll
    for (int s = 1; s <= NP; ++s) {
      T next[NDA][VW];
      if constexpr (MULTI) {
#pragma unroll
        for (int d = 0; d < ND; ++d)
#pragma unroll
          for (int h = 0; h < VW; ++h) next[d][h] = acc[s - 1][d][h];
      }
      const int q = i - s;
      T res[C][VW];
      if constexpr (!EDGE) {
        if (MULTI || s <= nsteps) stage<false, EC>(s, q, carry, res);
      } else {
        /* rows outside the mesh: the zero halo of the next stage */
#pragma unroll
        for (int c = 0; c < C; ++c)
#pragma unroll
          for (int h = 0; h < VW; ++h) res[c][h] = T(0);
        /* face rows; a mixed derivative reaches a row further */
        constexpr int X = Eq::CORNERS ? 1 : 0;
        if ((MULTI || s <= nsteps) && q >= max(0, r0 - NP + s) && q < min(p.nx, r1 + NP - s)) {
          if (q <= X || q >= p.nx - 1 - X) stage<true, true>(s, q, carry, res);
          else stage<false, EC>(s, q, carry, res);
        }
      }
      if (s < NP) push(s, res);
      if constexpr (MULTI) {
#pragma unroll
        for (int d = 0; d < ND; ++d)
#pragma unroll
          for (int h = 0; h < VW; ++h) carry[d][h] = next[d][h];
      }
    }
  }

  /* The columns left and right of a row's, from the neighbouring lanes at the
   * lane's ends. */
  static __device__ __forceinline__ void sides(const T (&row)[VW], T (&l)[VW], T (&r)[VW]) {
    l[0] = __shfl_up_sync(0xffffffffu, row[VW - 1], 1);
    r[VW - 1] = __shfl_down_sync(0xffffffffu, row[0], 1);
#pragma unroll
    for (int h = 1; h < VW; ++h) {
      l[h] = row[h - 1];
      r[h - 1] = row[h];
    }
  }

  /* Stage (or step) s on row q. */
  template <bool ER, bool EC>
  __device__ __forceinline__ void stage(int s, int q, const T (&carry)[NDA][VW], T (&res)[C][VW]) {
    using P = MarchPoint<T, Eq, VW, ER, EC>;
    const bool last = MULTI ? s == NP : s == nsteps;
    T up[C][VW], mid[C][VW], dn[C][VW], left[C][3][VW], right[C][3][VW];
#pragma unroll
    for (int c = 0; c < C; ++c) {
#pragma unroll
      for (int h = 0; h < VW; ++h) {
        up[c][h] = win[s - 1][c][0][h];
        mid[c][h] = win[s - 1][c][1][h];
        dn[c][h] = win[s - 1][c][2][h];
      }
      if ((Eq::HMASK >> c) & 1u) {
        sides(mid[c], left[c][1], right[c][1]);
        if constexpr (Eq::CORNERS) {
          sides(up[c], left[c][0], right[c][0]);
          sides(dn[c], left[c][2], right[c][2]);
        }
      }
    }

    const int h0 = MULTI ? stage_half<INTEG>(s - 1) : 2 * (s - 1);
    const int h1 = last ? (MULTI ? 2 : 2 * s) : (MULTI ? stage_half<INTEG>(s) : 2 * s);
    const MeshC<T> ms = Eq::DYNAMIC ? mesh_at(m, p, slot0 + h0) : m;
    const MeshC<T> me = Eq::DYNAMIC ? mesh_at(m, p, slot0 + h1) : m;
    const double ts = Eq::USES_T ? t0 + (MULTI ? stage_time<INTEG>(s - 1) : (double)(s - 1)) * p.dt : 0.0;

#pragma unroll
    for (int h = 0; h < VW; ++h) {
      P pt;
      pt.mid = mid;
      pt.up = up;
      pt.dn = dn;
      pt.left = left;
      pt.right = right;
      pt.col_neu = cn[s + 1];
      pt.col_dir = cd[s + 1];
      pt.m = &ms;
      pt.time = ts;
      pt.h = h;
      pt.gi = q;
      pt.gj = gj0 + h;
      T f[NDA];
      if constexpr (MULTI) {
        Eq::rhs_dt(pt, f);
#pragma unroll
        for (int d = 0; d < ND; ++d) {
          const int c = Eq::dcomp(d);
          const T y = s == 1 ? win[0][c][1][h] : (s == 2 ? win[0][c][0][h] : old[c][s - 3][h]);
          T a = s == 1 ? T(0) : carry[d][h];
          stage_accumulate<T, Eq, INTEG>(a, f[d], dt, s - 1);
          acc[s - 1][d][h] = a;
          const T v = last ? step_result<T, Eq, INTEG>(y, a, acc_scale) : stage_input<T, Eq, INTEG>(y, f[d], dt, s - 1);
          res[c][h] = pt.dirichlet(v, c, me);
        }
      } else {
        T fk[NDA];
        if constexpr (ND > 0) {
          if constexpr (Eq::FAST) {
            Eq::rhs_dt_split(pt, f, fk);
          } else {
            Eq::rhs_dt(pt, f);
          }
        }
        T yrhs[Eq::NYC > 0 ? Eq::NYC : 1];
        if constexpr (Eq::NYC > 0) Eq::rhs_y(pt, yrhs);
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const T y = mid[c][h];
          T hi = y;
#pragma unroll
          for (int d = 0; d < ND; ++d) {
            if (Eq::dcomp(d) == c) {
              if constexpr (Eq::FAST) {
                hi = fmaT(dt * fk[d], f[d], y);
              } else {
                const T kk = dt * f[d];
                hi = y + ((INTEG == RK4) ? div6(((kk + T(2) * kk) + T(2) * kk) + kk) : kk);
              }
            }
          }
#pragma unroll
          for (int d = 0; d < Eq::NYC; ++d)
            if (Eq::ycomp(d) == c) hi = yrhs[d];
          res[c][h] = pt.dirichlet(hi, c, me);
        }
      }
      /* columns outside the mesh stay zero */
      if (EC && (gj0 + h < 0 || gj0 + h >= p.ny)) {
#pragma unroll
        for (int c = 0; c < C; ++c) res[c][h] = T(0);
      }
    }

    if ((MULTI ? s == NP : true) && q >= r0 && q < r1 && owner) {
      T* dst = last ? out : (p.tb_out[s - 1] ? static_cast<T*>(p.tb_out[s - 1]) + (long long)b * p.tb_bstride : nullptr);
      if (dst) {
        dst += (long long)q * p.pitch + gj0;
#pragma unroll
        for (int c = 0; c < C; ++c) {
          if (!EC || gj0 + VW <= p.ny) {
            st_vec<T, VW>(dst + c * p.cstride, res[c]);
          } else {
#pragma unroll
            for (int h = 0; h < VW; ++h)
              if (gj0 + h < p.ny) dst[c * p.cstride + h] = res[c][h];
          }
        }
      }
    }
  }

  __device__ __forceinline__ void run(int b_, int r0_, int c0, int rows) {
    b = b_;
    r0 = r0_;
    r1 = r0 + rows < p.nx ? r0 + rows : p.nx;
    const int lane = threadIdx.x & 31;
    gj0 = c0 + lane * VW;
    owner = lane >= HL && lane < 32 - HL && gj0 < p.ny;
    in = static_cast<const T*>(p.in) + (long long)b * p.in_bstride;
    out = static_cast<T*>(p.out) + (long long)b * p.out_bstride;
    nsteps = MULTI ? NP : (p.tb_steps < 1 ? 1 : (p.tb_steps > NP ? NP : p.tb_steps));
    slot0 = bc_slot(p, b);
    t0 = Eq::USES_T ? p.t + (p.t_offset ? p.t_offset[b] : 0.0) : 0.0;
    dt = step_dt<T>(p);
    acc_scale = INTEG == RK4 ? dt * T(1.0 / 6.0) : dt;
    const T zero = T(0);
#pragma unroll
    for (int h = 0; h < VW; ++h) {
#pragma unroll
      for (int s = 0; s < NP; ++s) {
#pragma unroll
        for (int c = 0; c < C; ++c) win[s][c][0][h] = win[s][c][1][h] = win[s][c][2][h] = zero;
#pragma unroll
        for (int d = 0; d < ND; ++d) acc[s][d][h] = zero;
      }
#pragma unroll
      for (int c = 0; c < C; ++c)
#pragma unroll
        for (int r = 0; r < NOLD; ++r) old[c][r][h] = zero;
    }
    /* rows above the mesh are zeros, as the windows start */
    const int i0 = r0 > NP ? r0 - NP : 0;
#pragma unroll
    for (int q = 0; q < PF; ++q) load_row(i0 + q, pf[q]);
    col_face = gj0 == 0 ? 2 : (gj0 >= 0 && gj0 < p.ny && gj0 + VW >= p.ny ? 3 : 0);
    if constexpr (Eq::PRE) {
#pragma unroll
      for (int r = 0; r < NP + 2; ++r)
#pragma unroll
        for (int c = 0; c < C; ++c) cn[r][c] = cd[r][c] = free_value<T>();
      load_faces(i0);
    }
    const bool ec = c0 < 2 || c0 + COLS > p.ny - 2;
    const int end = r1 + NP;
#pragma unroll 1
    for (int i = i0; i < end; ++i) {
      /* rows i - NP .. i - 1 are computed; a mixed derivative reaches one more */
      if (i - NP <= 1 || i >= p.nx - 1 || i < r0 + NP) iterate<true, true>(i);
      else if (ec) iterate<false, true>(i);
      else iterate<false, false>(i);
    }
  }
};

/* Kernel body.  The jobs of an instance: its first and last strips (which
 * touch the column faces and cost more per row) in chunks of p.edge_rows
 * rows, then the strips between in chunks of p.tile_z rows.  The warps of the
 * grid take the jobs of all instances with a stride of all warps, the edge
 * strips of every instance first. */
template <typename T, class Eq, int INTEG, int VW, int NP, int NT>
__device__ __forceinline__ void march_body(const prml_step_params& p) {
  using M = March<T, Eq, INTEG, VW, NP>;
  const int strips = (p.ny + M::U - 1) / M::U;
  const int edges = strips < 2 ? strips : 2;
  const int e_chunks = (p.nx + p.edge_rows - 1) / p.edge_rows, chunks = (p.nx + p.tile_z - 1) / p.tile_z;
  const int e_inst = edges * e_chunks, i_inst = (strips - edges) * chunks;
  const int e_jobs = e_inst * p.batch;
  const int jobs = e_jobs + i_inst * p.batch; /* the host keeps this below 2^31 */
  const MeshC<T> m = make_mesh<T>(p);
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  for (int job = blockIdx.x * (NT / 32) + (threadIdx.x >> 5); job < jobs; job += gridDim.x * (NT / 32)) {
    int b, chunk, strip, rows;
    if (job < e_jobs) {
      b = job / e_inst;
      const int r = job - b * e_inst;
      chunk = r / edges;
      strip = r - chunk * edges ? strips - 1 : 0;
      rows = p.edge_rows;
    } else {
      const int j = job - e_jobs;
      b = j / i_inst;
      const int r = j - b * i_inst;
      chunk = r / (strips - edges);
      strip = 1 + r - chunk * (strips - edges);
      rows = p.tile_z;
    }
    M k(p, m);
    k.run(b, chunk * rows, strip * M::U - M::HL * VW, rows);
  }
}

}  // namespace prml
