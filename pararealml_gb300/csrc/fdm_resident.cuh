/*
 * Every step of a small 2D mesh in one launch: one thread-block cluster per
 * instance holds the state in shared memory, each CTA a band of rows.
 *
 * Why: a launch per step costs 2.4 us on GB300 however small the mesh (the
 * chain of dependent launches and a round trip through L2), which is all of a
 * 65^2 step.  Here a stage is: the warps with the band's two boundary rows
 * wait for the neighbour CTAs' rows (st.async into this CTA's halo rows,
 * counted on one mbarrier per buffer), evaluate theirs and send them on; the
 * other warps evaluate the rows between meanwhile; one barrier.  The two buffers alternate: a
 * neighbour overwrites a halo row only after it has received the row next to
 * it, which is the only one that reads that halo.  Saved states are plain
 * stores that nothing waits for.
 * GB300, us per step of one instance, the best other kernel against this:
 * 65^2 forward Euler diffusion 2.4 -> 1.5 in float64 and 1.6 -> 0.74 in
 * float32, Cahn-Hilliard 4.6 -> 2.8 and 2.1 -> 1.0, RK4 shallow water 34 ->
 * 20 in float64; 16 instances of 33^2 RK4 diffusion 13.7 -> 5.7.  What bounds
 * it: in float32 the exchange between CTAs (0.7 us a stage), in float64 also
 * the pipe of the 16 SMs a cluster has (its dependent chain at the smallest
 * sizes).
 *
 * Results equal the other step kernels' (the same operations in the same
 * order; bit for bit in float64).
 */
#pragma once

namespace prml {

__device__ __forceinline__ unsigned resident_remote(const void* p, unsigned rank) {
  unsigned a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_addr(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ void resident_send(unsigned a, float v, unsigned bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];" ::"r"(a), "f"(v), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void resident_send(unsigned a, double v, unsigned bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];" ::"r"(a), "d"(v), "r"(bar)
               : "memory");
}
__device__ __forceinline__ bool resident_landed(const unsigned long long* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ void resident_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <typename T, class Eq, int INTEG, int NT>
__device__ __forceinline__ void resident_body(const prml_step_params& p, const prml_resident_params& rp) {
  constexpr int C = Eq::C;
  constexpr int ND = Eq::ND;
  constexpr int NSTAGE = Eq::STAGE_INVARIANT ? 1 : INTEG;
  using P = Point<T, Eq, 0, 0>;
  extern __shared__ __align__(128) unsigned char prml_smem[];
  __shared__ unsigned long long bars[2]; /* halo rows of buffer w have landed */

  unsigned nc, rank;
  asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(nc));
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int b = (int)(blockIdx.x / nc);
  const int r0 = (int)rank * rp.band;
  const int rows = p.nx - r0 < rp.band ? p.nx - r0 : rp.band; /* >= 1: the host leaves no CTA without rows */
  const bool up = rank > 0, down = rank + 1 < nc;
  const int S = rp.spitch, SC = rp.scomp, BUF = C * SC;
  T* buf = reinterpret_cast<T*>(prml_smem); /* two buffers, then (several stages) the step start and the sums */
  T* ystart = buf + 2 * BUF;
  T* sums = ystart + BUF;

  const MeshC<T> m = make_mesh<T>(p);
  const unsigned halo_bytes = (unsigned)((int)up + (int)down) * (unsigned)(C * p.ny * (int)sizeof(T));
  if (threadIdx.x == 0) {
    mbar_init(&bars[0], 1);
    mbar_init(&bars[1], 1);
    fence_barrier_init();
  }
  for (int e = threadIdx.x; e < 2 * BUF; e += NT) buf[e] = T(0); /* zero outside the mesh */
  __syncthreads();
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const T* in = static_cast<const T*>(p.in) + (long long)b * p.in_bstride;
  for (int e = threadIdx.x; e < (rows + 2) * p.ny; e += NT) {
    const int r = e / p.ny, j = e - r * p.ny, gi = r0 + r - 1;
    if (gi < 0 || gi >= p.nx) continue;
#pragma unroll
    for (int c = 0; c < C; ++c) buf[c * SC + r * S + 1 + j] = __ldcg(in + c * p.cstride + (long long)gi * p.pitch + j);
  }
  resident_cluster_sync();

  /* the neighbours' buffers: row band of the CTA above, row -1 of the one below */
  const unsigned above = up ? resident_remote(buf + (rp.band + 1) * S + 1, rank - 1) : 0u;
  const unsigned below = down ? resident_remote(buf + 1, rank + 1) : 0u;
  const unsigned bar_above = up ? resident_remote(bars, rank - 1) : 0u;
  const unsigned bar_below = down ? resident_remote(bars, rank + 1) : 0u;
  const unsigned long long wait_ns = p.wait_limit_ns ? p.wait_limit_ns : kWaitLimitNs;
  const T dt = step_dt<T>(p);
  const T acc_scale = INTEG == RK4 ? dt * T(1.0 / 6.0) : dt;
  (void)acc_scale;
  const int slot_in = bc_slot(p, b);
  const double t_in = Eq::USES_T ? p.t + (p.t_offset ? p.t_offset[b] : 0.0) : 0.0;
  T* out = static_cast<T*>(p.out) + (long long)b * p.out_bstride + (long long)r0 * p.pitch;
  const int total = rows * p.ny;
  /* this thread's first vertex, and the step to its next one, in the order
   * first row, last row, rows between */
  const int q0 = (int)threadIdx.x / p.ny, j0 = (int)threadIdx.x - q0 * p.ny;
  const int dq = NT / p.ny, dj = NT - dq * p.ny;

  /* only warps with vertices of the band's first or last row read the halo:
   * the others go on while it travels */
  const bool boundary = (int)(threadIdx.x & ~31u) < 2 * p.ny;

  int until = rp.save_every;
  bool ok = true;
  unsigned g = 0; /* stages done */
  for (long long step = 0; step < rp.n_steps && ok; ++step) {
    const int slot0 = slot_in + (int)(2 * step);
    const bool save = --until == 0;
#pragma unroll 1
    for (int s = 0; s < NSTAGE; ++s, ++g) {
      const unsigned w = (g + 1) & 1u;
      const T* cur = buf + (g & 1u) * BUF;
      T* nxt = buf + w * BUF;
      const bool last = s == NSTAGE - 1, end = last && step + 1 == rp.n_steps;
      if (threadIdx.x == 0 && !end) mbar_expect_tx(&bars[w], halo_bytes);
      if (g > 0 && boundary) {
        const unsigned parity = ((g - 1) >> 1) & 1u;
        if (!resident_landed(&bars[g & 1u], parity)) {
          const unsigned long long t0 = global_ns();
          while (ok && !resident_landed(&bars[g & 1u], parity)) ok = global_ns() - t0 <= wait_ns;
        }
      }
      const double ts = Eq::USES_T ? __dadd_rn(t_in, __dmul_rn((double)step, p.dt)) + stage_time<INTEG>(s) * p.dt : 0.0;
      const MeshR<T> ms{mesh_at(m, p, slot0 + stage_half<INTEG>(s)), S, SC};
      const MeshC<T> me = mesh_at(m, p, slot0 + (last ? 2 : stage_half<INTEG>(s + 1)));
      const unsigned shift = (unsigned)(w * BUF) * (unsigned)sizeof(T);
      int q = q0, j = j0;
      for (int v = threadIdx.x; v < total && ok; v += NT) {
        const int r = q == 0 ? 0 : (q == 1 ? rows - 1 : q - 1);
        const int l = (r + 1) * S + 1 + j;
        const int gi = r0 + r;
        P pt{cur, l, gi, j, &ms, ts};
        T f[ND > 0 ? ND : 1], fk[ND > 0 ? ND : 1];
        if constexpr (ND > 0) {
          if constexpr (Eq::FAST && NSTAGE == 1) {
            Eq::rhs_dt_split(pt, f, fk);
          } else {
            Eq::rhs_dt(pt, f);
          }
        }
        T yrhs[Eq::NYC > 0 ? Eq::NYC : 1];
        if (Eq::NYC > 0 && s == 0) Eq::rhs_y(pt, yrhs);
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const T here = cur[c * SC + l];
          T y = here, res = here;
          if constexpr (NSTAGE > 1) {
            if (s == 0) ystart[c * SC + l] = here;
            else y = ystart[c * SC + l];
            res = y;
          }
#pragma unroll
          for (int i = 0; i < ND; ++i) {
            if (Eq::dcomp(i) != c) continue;
            if constexpr (NSTAGE > 1) {
              T a = s == 0 ? T(0) : sums[c * SC + l];
              stage_accumulate<T, Eq, INTEG>(a, f[i], dt, s);
              if (!last) sums[c * SC + l] = a;
              res = last ? step_result<T, Eq, INTEG>(y, a, acc_scale) : stage_input<T, Eq, INTEG>(y, f[i], dt, s);
            } else if constexpr (Eq::FAST) {
              res = fmaT(dt * fk[i], f[i], y);
            } else {
              const T kk = dt * f[i];
              res = y + ((INTEG == RK4) ? div6(((kk + T(2) * kk) + T(2) * kk) + kk) : kk);
            }
          }
          /* LHS.Y rows: their value at the step start, kept in the sums' plane */
#pragma unroll
          for (int i = 0; i < Eq::NYC; ++i) {
            if (Eq::ycomp(i) != c) continue;
            if constexpr (NSTAGE > 1) {
              if (s == 0) sums[c * SC + l] = yrhs[i];
              if (last) res = sums[c * SC + l];
            } else {
              res = yrhs[i];
            }
          }
          res = dirichlet<T, Eq, true, false>(res, c, gi, j, me);
          nxt[c * SC + l] = res;
          if (!end) {
            const unsigned off = shift + (unsigned)(c * SC + j) * (unsigned)sizeof(T);
            if (r == 0 && up) resident_send(above + off, res, bar_above + 8u * w);
            if (r == rows - 1 && down) resident_send(below + off, res, bar_below + 8u * w);
          }
          if (last && save) out[c * p.cstride + (long long)r * p.pitch + j] = res;
        }
        q += dq;
        j += dj;
        if (j >= p.ny) {
          j -= p.ny;
          ++q;
        }
      }
      ok = !__syncthreads_or(!ok);
      if (!ok) break;
    }
    if (save) {
      until = rp.save_every;
      out += rp.step_stride;
    }
  }
  /* a neighbour that stopped coming: report; every wait above is bounded, so
   * every CTA of the cluster gets here */
  if (!ok && threadIdx.x == 0 && p.status) atomicExch(p.status, 1);
  resident_cluster_sync();
}

}  // namespace prml
