// agx_plain.cu -- FP64 kernels of the DE timestep (plain form, bit-exact).
//
// Compiled with --fmad=false: every floating-point operation is rounded on its
// own, as in the reference built without contraction, so results match the
// reference's FP64 path bit for bit (Manning's pow excepted: CUDA's and the C
// library's pow may differ in the last place).
//
// One timestep is a fixed sequence of kernels (DE1 = RK2 shown):
//   prep(backup) -> extrap -> flux -> accum (last block: timestep) -> update+prep
//   -> extrap -> flux -> accum -> update(saxpy; last block: clock)
// (DE2 = RK3 adds a third stage: generic_domain.py:2053-2172; with operators
// they and a clock kernel follow).  The flux kernel forms the boundary values
// of its own edges.  All state stays in device memory; the clock decides on
// the device whether another step is needed and sets the graph's while
// condition.
#include "agx_internal.cuh"
#include "inlet.cuh"
#include <cuda_runtime.h>

namespace agx {

// Threads per block of the elementwise and per-edge kernels: 128, so that the
// blocks of a mesh of some tens of thousands of cells spread evenly over the
// 152 SMs (40,000 cells: 157 blocks of 256 gave five SMs twice the work).
constexpr int TPB = 128;
// resident blocks of 128 per SM asked of the compiler (register budgets),
// measured on the 4.0M-triangle DE1 run: extrapolation 8 (6: +2%, 10: the
// same and +4% at 40,000 cells), flux 7 (8: +0.5%), update 10 (8: +1%, 12: the
// same), accumulation 8 on large meshes (5: +0.5%)
#ifndef AGX_MINB_EXTRAP
#define AGX_MINB_EXTRAP 8
#endif
#ifndef AGX_MINB_FLUX
#define AGX_MINB_FLUX 7
#endif
#ifndef AGX_MINB_UPDATE
#define AGX_MINB_UPDATE 10
#endif

__device__ __forceinline__ double warp_sum(double x) {
  for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
  return x;
}
__device__ __forceinline__ unsigned long long warp_max_u64(unsigned long long x) {
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long y = __shfl_down_sync(0xffffffffu, x, o);
    x = y > x ? y : x;
  }
  return x;
}

// Block-wide sum, result valid in thread 0.
__device__ double block_sum(double x) {
  __shared__ double part[TPB / 32];
  x = warp_sum(x);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) part[wid] = x;
  __syncthreads();
  double r = 0.0;
  if (wid == 0) {
    r = lane < (int)(blockDim.x >> 5) ? part[lane] : 0.0;
    r = warp_sum(r);
  }
  __syncthreads();
  return r;
}

__device__ unsigned long long block_max_u64(unsigned long long x) {
  __shared__ unsigned long long part[TPB / 32];
  x = warp_max_u64(x);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) part[wid] = x;
  __syncthreads();
  unsigned long long r = 0;
  if (wid == 0) {
    r = lane < (int)(blockDim.x >> 5) ? part[lane] : 0ull;
    r = warp_max_u64(r);
  }
  __syncthreads();
  return r;
}

// The last block of a kernel to finish does the work that used to take a
// one-thread kernel after it (about 2 us a launch inside the step graph):
// thread 0 of each block counts itself once everything its block wrote is
// visible (the block's barrier, then a device fence); true for the last.
__device__ __forceinline__ bool last_to_finish(Clock* c) {
  __syncthreads();
  if (threadIdx.x != 0) return false;
  __threadfence();
  return atomicAdd(&c->blocks_done, 1u) == gridDim.x - 1;
}

// After the accumulation: the stage's boundary flux sum, and at a step's
// first stage its timestep.
__device__ __noinline__ void finish_accum(Clock* c, int substep, int timestep) {
  __threadfence();
  clock_refresh(c);
  c->bfs[substep] = c->bfs_acc;
  if (timestep) timestep_logic(c);
  c->blocks_done = 0u;
}

// After the step's last update: the clock and the graph's while condition.
__device__ __noinline__ void finish_step(Clock* c, cudaGraphConditionalHandle handle, int set_cond) {
  __threadfence();
  clock_refresh(c);
  const int reason = clock_logic(c);
  c->blocks_done = 0u;
  if (set_cond) cudaGraphSetConditional(handle, reason == 0 ? 1u : 0u);
}

// ---------------------------------------------------------------------------
// mode bit 0: backup, bit 1: skip protect, bit 2: protect only
__global__ void k_prep(Dev d, int mode) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  double added = 0.0;
  if (k < d.N) {
    if (mode & 1) {
      d.w0[k] = d.w[k];
      d.uh0[k] = d.uh[k];
      d.vh0[k] = d.vh[k];
    }
    added = prep_cell(d.P, k, d.w, d.uh, d.vh, d.z, d.areas, d.h, d.u, d.v, (mode & 2) == 0,
                      (mode & 4) == 0);
  }
  const int any = __syncthreads_or(added != 0.0);
  if (any) {
    const double s = block_sum(added);
    if (threadIdx.x == 0) atomicAdd(&d.clock->mass_added, s);
  }
}

// Extrapolation (:1418-1896): a block takes XCELLS cells, one per lane, and
// each of its four warps reconstructs one quantity of them (stage, depth, x
// and y velocity).  The height warp forms the wet/dry factor the others'
// limiters need while they form their jumps, and hands over its edge depths
// for the bed (w - h) and the momenta (u h).  The FP64 pipe bounds it on large
// meshes (per launch of a 4.0M-triangle DE1 step 1.00 -> 0.98 ms against one
// thread per cell) and the chain of one thread's operations on small ones,
// which is a quarter as long this way: 26 -> 7.4 us on 396 cells, 41 -> 26 us
// on 40,000 (DE0), 96 -> 70 us on 250,000 (DE1).
// Cells are visited as stored: with one quantity to a warp, grouping the cells
// of the wet/dry fronts (a counting sort a step) no longer pays for its three
// launches (a 4.0M-triangle DE1 step 5.70 ms with it, 5.62 without; 250,000
// 465 and 439 us).
constexpr int XCELLS = 32;
constexpr int XTPB = 4 * XCELLS;
template <bool VERT, bool IM>
__global__ void __launch_bounds__(XTPB, AGX_MINB_EXTRAP) k_extrap(Dev d) {
  __shared__ double s_factor[XCELLS];
  __shared__ double s_h[3][XCELLS];
  const int lane = threadIdx.x & 31, q = threadIdx.x >> 5;
  const int at = blockIdx.x * XCELLS + lane;
  const bool in = at < d.N;
  const int k = in ? at : d.N - 1;
  const Params& P = d.P;
  const int4 s = d.surr[k];
  const int meta = d.conn[k].w;
  const int nb = meta_nb(meta);
  const double* A = q == 0 ? d.w : q == 1 ? d.h : q == 2 ? d.u : d.v;
  const double beta0 = q < 2 ? P.beta_w : q == 2 ? P.beta_uh : P.beta_vh;
  const double beta0_dry = q < 2 ? P.beta_w_dry : q == 2 ? P.beta_uh_dry : P.beta_vh_dry;
  double qc = A[k], q0 = A[s.x], q1 = A[s.y], q2 = A[s.z];
  const double hk = d.h[k], h0 = d.h[s.x], h1 = d.h[s.y], h2 = d.h[s.z];
  const bool sdry = (dlt(h0, P.hmin) | (s.x == k)) & (dlt(h1, P.hmin) | (s.y == k)) & (dlt(h2, P.hmin) | (s.z == k));
  const bool dry = dlt(hk, P.hmin);
  if (q >= 2) {
    if (sdry) qc = 0.0;
    // Neighbour velocities can be stale-zeroed only for a dry cell (a wet
    // neighbour rules out "surrounded by dry"); they matter only if the dry
    // reconstruction has a positive beta (the factor of a dry cell is 0), or
    // towards the one neighbour of a cell with two boundary edges.
    if (nb == 2 || (nb <= 1 && dry && (dgt0(P.beta_uh_dry) || dgt0(P.beta_vh_dry)))) {
      const int sv[3] = {s.x, s.y, s.z};
      double* qv[3] = {&q0, &q1, &q2};
#pragma unroll
      for (int i = 0; i < 3; i++) {
        double us, vs;
        if (sv[i] != k) {
          neighbour_uv(P, sv[i], meta_before(meta, i) != 0, d.surr, d.h, d.u, d.v, us, vs);
          *qv[i] = q == 2 ? us : vs;
        }
      }
    }
    if (s.x == k) q0 = qc;
    if (s.y == k) q1 = qc;
    if (s.z == k) q2 = qc;
  }
  // The factor is 0 where a depth around the cell is at most hmin (its third
  // term is 0 over a positive number): with a dry beta of 0 the edges then
  // take the cell's value and no gradient is needed.
  const double hlo = dmin(dmin(h0, dmin(h1, h2)), hk);
  const bool factor0 = dgt0(P.hmin) && dle(hlo, P.hmin);
  const bool grad = nb <= 1 && (dgt0(beta0_dry) || (dgt0(beta0) && !factor0));
  double G[GEO_STRIDE];
  double jump[3], lo = 0.0, hi = 0.0, E[3];
  if (grad || nb == 2) {
#pragma unroll
    for (int i = 0; i < GEO_STRIDE; i++) G[i] = d.geo[(size_t)i * d.N + k];
  }
  if (q == 1 && nb <= 1) {
    double f = 0.0;
    if (!factor0) f = wet_dry_factor(P, hk, hlo, dmax(dmax(h0, dmax(h1, h2)), hk));
    s_factor[lane] = f;
  }
  if (grad) edge_jumps<IM>(qc, q0, q1, q2, G, jump, lo, hi);
  __syncthreads();
  E[0] = E[1] = E[2] = qc;
  if (grad) {
    const double f = s_factor[lane];
    // at factor 1 the betas and their reciprocals are the precomputed ones
    const bool one = dbits(f) == dbits(1.0);
    const double beta1 = q < 2 ? P.beta_w1 : q == 2 ? P.beta_uh1 : P.beta_vh1;
    const double inv1 = q < 2 ? P.inv_beta_w1 : q == 2 ? P.inv_beta_uh1 : P.inv_beta_vh1;
    const double beta = one ? beta1 : beta0_dry + (beta0 - beta0_dry) * f;
    if (dgt0(beta)) limited_edges(qc, jump, limiter_phi(jump, lo, hi, beta, one ? inv1 : 0.0), E);
  } else if (nb == 2) {
    const double qn = s.x != k ? q0 : (s.y != k ? q1 : q2);
    reconstruct_towards(P.beta_w, P.inv_beta_w, qc, qn, G, E);
  }
  if (q == 1) {
#pragma unroll
    for (int i = 0; i < 3; i++) s_h[i][lane] = E[i];
  }
  __syncthreads();
  if (!in) return;
  const size_t b = 3 * (size_t)k;
  if (q >= 2 && P.velocity_extrapolation) {
#pragma unroll
    for (int i = 0; i < 3; i++) E[i] = imul<IM>(E[i], s_h[i][lane]);
  }
  double* const out = q == 0 ? d.we : q == 1 ? d.he : q == 2 ? d.uhe : d.vhe;
#pragma unroll
  for (int i = 0; i < 3; i++) out[b + i] = E[i];
  if (q >= 2 && sdry) (q == 2 ? d.uh : d.vh)[k] = 0.0;
  double vx[3];
  if (VERT) {
    double* const vert = q == 0 ? d.wv : q == 1 ? d.hv : q == 2 ? d.uhv : d.vhv;
    vertex_from_edges(E, vx);
    for (int i = 0; i < 3; i++) vert[b + i] = vx[i];
  }
  if (q == 0) {
#pragma unroll
    for (int i = 0; i < 3; i++) {
      E[i] = E[i] - s_h[i][lane];
      d.ze[b + i] = E[i];
    }
    if (VERT || P.sloped_mannings) {       // sloped friction reads the bed vertex values
      vertex_from_edges(E, vx);
      for (int i = 0; i < 3; i++) d.zv[b + i] = vx[i];
    }
  }
}

// The extrapolation geometry from the caller's rows [N][GEO_STRIDE] to one
// array per coefficient, so that the lanes of a warp read it contiguously.
__global__ void k_geo_transpose(double* out, const double* rows, int N) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= N) return;
#pragma unroll
  for (int i = 0; i < GEO_STRIDE; i++) out[(size_t)i * N + k] = rows[(size_t)GEO_STRIDE * k + i];
}

__device__ void series_value(const double* rows, int n, double t, double out[3]) {
  if (n <= 0) { out[0] = out[1] = out[2] = 0.0; return; }
  if (t <= rows[0]) { out[0] = rows[1]; out[1] = rows[2]; out[2] = rows[3]; return; }
  if (t >= rows[4 * (n - 1)]) {
    const double* r = rows + 4 * (n - 1);
    out[0] = r[1]; out[1] = r[2]; out[2] = r[3];
    return;
  }
  int lo = 0, hi = n - 1;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (rows[4 * mid] <= t) lo = mid; else hi = mid;
  }
  const double* a = rows + 4 * lo;
  const double* c = rows + 4 * hi;
  const double ratio = (t - a[0]) / (c[0] - a[0]);
  for (int q = 0; q < 3; q++) out[q] = a[1 + q] + ratio * (c[1 + q] - a[1 + q]);
}

// Boundary values of segment m; a time series is read at t_override, or (NaN)
// at the clock's time + frac * timestep (the stage's time: frac 0, 1 or 0.5).
__device__ __forceinline__ void boundary_segment(const Dev& d, int m, double t_override, double frac) {
  const int kind = d.bkind[m];
  if (kind == BK_NONE) return;
  const int s = d.bslot[m];
  const int k = s / 3;
  double tv[3];
  const double* val = d.bval + 3 * (size_t)m;
  if (kind == BK_TIME_SERIES) {
    double t = t_override;
    if (t != t) t = d.clock->time + frac * d.clock->timestep;  // NaN: use the clock
    series_value(d.bseries, d.nseries, t, tv);
    val = tv;
  }
  double wb, uhb, vhb;
  boundary_value(kind, d.normals[2 * s], d.normals[2 * s + 1], d.we[s], d.uhe[s], d.vhe[s], d.ze[s], d.w[k],
                 d.uh[k], d.vh[k], d.z[k], d.P.g, val, wb, uhb, vhb);
  d.wb[m] = wb;
  d.uhb[m] = uhb;
  d.vhb[m] = vhb;
}

__global__ void k_bc(Dev d, double t_override) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m < d.B) boundary_segment(d, m, t_override, 0.0);
}

// The same for the one thread of the flux kernel that needs the segment, out
// of line: the boundary kinds' registers stay out of the edge loop.
__device__ __noinline__ void stage_boundary(const Dev& d, int m, double frac) {
  boundary_segment(d, m, __longlong_as_double(0x7ff8000000000000ll), frac);
}

// Edge fluxes.  BC: in the step loop each boundary edge's values are formed
// by the thread that reads them.  The first thread clears the accumulators
// of the accumulation that follows.
template <bool BC, bool IM>
__global__ void __launch_bounds__(TPB, AGX_MINB_FLUX) k_flux(const __grid_constant__ Dev d, double frac) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e == 0) {
    d.clock->dt_key = 0ull;
    d.clock->bfs_acc = 0.0;
  }
  if (e >= d.E) return;
  const int s = d.edge_slot[e];
  const int k = s / 3, i = s - 3 * k;
  const int4 cn = d.conn[k];
  if (BC) {
    const int n = i == 0 ? cn.x : i == 1 ? cn.y : cn.z;
    if (n < 0) stage_boundary(d, -n - 1, frac);
  }
  const Riverwall RW = {d.rw_counter, d.rw_elev, d.rw_row, d.rw_hyd, d.rw_ncol};
  SlotResult R;
  double hr;
  slot_flux<IM>(d.P, k, i, cn, d.we, d.uhe, d.vhe, d.ze, d.he, d.wb, d.uhb, d.vhb, d.normals, d.w,
            d.h, d.z, RW, R, hr);
  // the contributions -f * length of the edge's two cells (opposite but for
  // the length, which a table could hold differently for the two sides)
  const double len = d.lengths[s];
  const double e0 = imul<IM>(dneg(R.f[0]), len), e1 = imul<IM>(dneg(R.f[1]), len),
               e2 = imul<IM>(dneg(R.f[2]), len);
  d.sl0[s] = e0;
  d.sl1[s] = e1;
  d.sl2[s] = e2;
  d.slsp[s] = R.speed;
  d.slpf[s] = R.pflux;
  d.slhl[s] = R.hleft;
  const int o = d.edge_opp[e];
  if (o >= 0) {
    const double len_o = d.lengths[o];
    const bool same = dbits(len_o) == dbits(len);
    d.sl0[o] = same ? dneg(e0) : R.f[0] * len_o;
    d.sl1[o] = same ? dneg(e1) : R.f[1] * len_o;
    d.sl2[o] = same ? dneg(e2) : R.f[2] * len_o;
    d.slsp[o] = R.speed;
    d.slpf[o] = R.pflux;
    d.slhl[o] = hr;
  }
}

// timestep: form the step's timestep once every block is done.
template <bool IM>
__global__ void __launch_bounds__(TPB, IM ? 8 : 5) k_accum(Dev d, int substep, int timestep) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned long long key = 0ull;
  double bflux = 0.0;
  if (k < d.N) {
    const int4 c = d.conn[k];
    SlotResult R[3];
    int fn[3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
      const size_t s = 3 * (size_t)k + i;
      R[i].f[0] = d.sl0[s];
      R[i].f[1] = d.sl1[s];
      R[i].f[2] = d.sl2[s];
      R[i].speed = d.slsp[s];
      R[i].pflux = d.slpf[s];
      R[i].hleft = d.slhl[s];
      const int n = i == 0 ? c.x : i == 1 ? c.y : c.z;
      fn[i] = n >= 0 ? meta_full(d.conn[n].w) : 1;
    }
    // A dry cell whose three slots carry a zero flux, no speed, a +0 pressure
    // flux and zero depths on both sides: every term of accum_cell is then
    // a zero, its sums and the pressure terms come out +0 (the pressure
    // bracket is +0 - +0 - (+0 * dz) = +0 whatever the sign of dz), so the
    // FP64 arithmetic is skipped with the same bits.
    bool dry = !dnz(d.h[k]);
#pragma unroll
    for (int i = 0; i < 3; i++)
      dry = dry && !dnz(R[i].f[0]) && !dnz(R[i].f[1]) && !dnz(R[i].f[2]) && dbits(R[i].pflux) == 0 &&
            !dnz(R[i].hleft) && !dnz(d.he[3 * (size_t)k + i]) && !dgt(R[i].speed, d.P.epsilon);
    CellFlux F;
    if (dry) {
      F.ew = F.euh = F.evh = 0.0 * d.inv_area[k];     // +0 * (1/area), as the sums' scaling
      F.smax = 0.0;
      F.bflux = 0.0;
    } else {
      accum_cell<true, IM>(d.P, k, c, R, d.he, d.ze, d.h, d.z, d.normals, d.lengths, d.inv_area[k], fn, F);
    }
    d.xw[k] = F.ew;
    d.xuh[k] = F.euh;
    d.xvh[k] = F.evh;
    bflux = F.bflux;
    if (substep == 0) {
      d.max_speed[k] = F.smax;
      if (F.smax > 0.0) {
        const double dt = ddiv(d.radii[k] * 1.0, F.smax);
        key = ~(unsigned long long)__double_as_longlong(dt);
      }
    }
  }
  if (substep == 0) {
    const unsigned long long bk = block_max_u64(key);
    if (threadIdx.x == 0 && bk != 0ull && bk > __ldcg(&d.clock->dt_key)) atomicMax(&d.clock->dt_key, bk);
  }
  const int any = __syncthreads_or(bflux != 0.0);
  if (any) {
    const double bs = block_sum(bflux);
    if (threadIdx.x == 0) atomicAdd(&d.clock->bfs_acc, bs);
  }
  if (last_to_finish(d.clock)) finish_accum(d.clock, substep, timestep);
}

// saxpy: 0 none; 1 RK2 combine 0.5 Q + 0.5 Q0; 2 RK3 second stage
// 0.25 Q + 0.75 Q0; 3 RK3 last stage (2 Q + Q0) / 3 (generic_domain.py:2126, 2160-2166).
// PREP: followed by the preparation of the next stage (k_prep on the values in
// registers).  clock: the step ends here (the last block runs its clock).
template <bool PREP>
__global__ void __launch_bounds__(TPB, AGX_MINB_UPDATE) k_update(Dev d, int stage, int use_clock_dt, double dt_arg, int saxpy, int clock,
                         cudaGraphConditionalHandle handle, int set_cond) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  int bad = 0, neg = 0, nf = 0;
  double added = 0.0;
  if (k < d.N) {
    const double dt = use_clock_dt ? d.clock->timestep : dt_arg;
    double w = d.w[k], uh = d.uh[k], vh = d.vh[k];
    const double z = d.z[k];
    double sw = d.sw[k], suh = d.suh[k], svh = d.svh[k];
    if (stage >= 0) {   // forcing terms: manning_friction_implicit
      double S;
      if (d.P.sloped_mannings) S = manning_S_sloped(d.P, w, d.zv + 3 * (size_t)k, d.vcoord + 6 * (size_t)k, uh, vh, d.eta[k]);
      else S = manning_S(d.P, w, z, uh, vh, d.eta[k]);
      suh = dnz(suh) ? suh + S * uh : S * uh;     // 0 + x: a zero's sign plays no part in the update
      svh = dnz(svh) ? svh + S * vh : S * vh;
    }
    if (!update_quantity(w, d.xw[k], sw, dt)) bad = 1;
    if (!update_quantity(uh, d.xuh[k], suh, dt)) bad = 1;
    if (!update_quantity(vh, d.xvh[k], svh, dt)) bad = 1;
    if ((dkey(w - z) < -1) & (meta_full(d.conn[k].w) > 0)) {     // w - z < 0
      neg = 1;
      w = z;
      uh = 0.0;
      vh = 0.0;
    }
    if (saxpy == 1) {
      w = dhalf_sum(w, d.w0[k]);
      uh = dhalf_sum(uh, d.uh0[k]);
      vh = dhalf_sum(vh, d.vh0[k]);
    } else if (saxpy) {
      const double a = saxpy == 2 ? 0.25 : 2.0;
      const double b = saxpy == 2 ? 0.75 : 1.0;
      w = a * w + b * d.w0[k];
      uh = a * uh + b * d.uh0[k];
      vh = a * vh + b * d.vh0[k];
      if (saxpy == 3) {
        w = ddiv(w, 3.0);
        uh = ddiv(uh, 3.0);
        vh = ddiv(vh, 3.0);
      }
    }
    // a NaN or an infinity in the conserved state stops the step loop (the
    // CFL minimum would otherwise skip the cell and let it spread)
    nf = nonfinite64(w) | nonfinite64(uh) | nonfinite64(vh);
    if (PREP) {
      double h, u, v;
      added = prep_values(d.P, w, uh, vh, z, d.areas + k, h, u, v);
      d.h[k] = h;
      d.u[k] = u;
      d.v[k] = v;
    }
    d.w[k] = w;
    d.uh[k] = uh;
    d.vh[k] = vh;
    d.sw[k] = sw;
    d.suh[k] = suh;
    d.svh[k] = svh;
  }
  if (__syncthreads_or(neg | bad | nf | (PREP && added != 0.0))) {
    const int nneg = __syncthreads_count(neg);
    const int anybad = __syncthreads_or(bad);
    const int nnf = __syncthreads_count(nf);
    const double mass = PREP ? block_sum(added) : 0.0;
    if (threadIdx.x == 0) {
      if (nneg) atomicAdd((unsigned long long*)&d.clock->negative_cells, (unsigned long long)nneg);
      if (anybad) atomicOr(&d.clock->error, (int)ERR_NUMERIC);
      if (nnf) {
        atomicAdd((unsigned long long*)&d.clock->nonfinite_cells, (unsigned long long)nnf);
        atomicOr(&d.clock->error, (int)ERR_NONFINITE);
      }
      if (mass != 0.0) atomicAdd(&d.clock->mass_added, mass);
    }
  }
  if (clock && last_to_finish(d.clock)) finish_step(d.clock, handle, set_cond);
}

// Forcing only (per-phase API): accumulate Manning into semi_implicit_update.
__global__ void k_forcing(Dev d) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= d.N) return;
  const double w = d.w[k], uh = d.uh[k], vh = d.vh[k];
  double S;
  if (d.P.sloped_mannings) S = manning_S_sloped(d.P, w, d.zv + 3 * (size_t)k, d.vcoord + 6 * (size_t)k, uh, vh, d.eta[k]);
  else S = manning_S(d.P, w, d.z[k], uh, vh, d.eta[k]);
  d.suh[k] += S * uh;
  d.svh[k] += S * vh;
}

__global__ void k_backup(Dev d) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= d.N) return;
  d.w0[k] = d.w[k];
  d.uh0[k] = d.uh[k];
  d.vh0[k] = d.vh[k];
}

// Conserved centroid values divided by `divisor` (the last RK3 stage's
// Q / 3.0, generic_domain.py:2163-2166).
__global__ void k_divide(Dev d, double divisor) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= d.N) return;
  d.w[k] = ddiv(d.w[k], divisor);
  d.uh[k] = ddiv(d.uh[k], divisor);
  d.vh[k] = ddiv(d.vh[k], divisor);
}

__global__ void k_saxpy(Dev d, double a, double b) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= d.N) return;
  d.w[k] = a * d.w[k] + b * d.w0[k];
  d.uh[k] = a * d.uh[k] + b * d.uh0[k];
  d.vh[k] = a * d.vh[k] + b * d.vh0[k];
}

// Rate_operator with a constant non-negative or negative rate.
// dt_arg < 0: the step's timestep from the device clock (the step loop);
// otherwise the timestep the host gives (operators applied from the host).
__global__ void k_rate(Dev d, const int* idx, int n, double rate, double factor, int op, double dt_arg) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  double influx = 0.0;
  if (j < n) {
    const int k = idx ? idx[j] : j;
    const double dt = dt_arg >= 0.0 ? dt_arg : d.clock->timestep;
    if (rate >= 0.0) {
      const double local = factor * dt * rate;
      d.w[k] = d.w[k] + local;
      influx = local * d.areas[k];
    } else {
      const double height = d.w[k] - d.z[k];
      const double local = fmax(factor * dt * rate, -height);
      const double f = local < 0.0 ? (local + height) / (height + 1.0e-10) : 1.0;
      d.w[k] = d.w[k] + local;
      d.uh[k] = d.uh[k] * f;
      d.vh[k] = d.vh[k] * f;
      influx = local * d.areas[k];
    }
  }
  const int any = __syncthreads_or(influx != 0.0);
  if (any) {
    const double s = block_sum(influx);
    if (threadIdx.x == 0 && op < MAX_OPS) atomicAdd(&d.clock->op_influx[op], s);
  }
}

// Inlet_operator (structures/inlet_operator.py:75-165, inlet.py:107-226) on
// the scenario's stage-stored state; the steps are in inlet.cuh.  The
// discharge is Q = 0.5 (q1 + q2) over the timestep (dt_arg < 0: the step's
// timestep from the clock).
struct PlainInletCells {
  Dev d;
  __device__ int cell(int a) const { return d_idx[a]; }
  __device__ double stage(int k) const { return d.w[k]; }
  __device__ double height(int k) const { return d.w[k] - d.z[k]; }
  __device__ double area(int k) const { return d.areas[k]; }
  __device__ double uh(int k) const { return d.uh[k]; }
  __device__ double vh(int k) const { return d.vh[k]; }
  __device__ void set_level(int k, double level) { d.w[k] = level; }
  __device__ void set_depth(int k, double depth) { d.w[k] = d.z[k] + depth; }
  __device__ void empty(int k) {
    d.w[k] = d.z[k];
    d.uh[k] = 0.0;
    d.vh[k] = 0.0;
  }
  __device__ void set_momenta(int k, double mx, double my) {
    d.uh[k] = mx;
    d.vh[k] = my;
  }
  const int* d_idx;
};

__global__ void __launch_bounds__(INLET_TPB) k_inlet(Dev d, RateOp op, int slot, double q1, double q2, double dt_arg) {
  const double dt = dt_arg >= 0.0 ? dt_arg : d.clock->timestep;
  const double volume = 0.5 * (q1 + q2) * dt;
  PlainInletCells c{d, op.idx};
  const double applied = inlet_apply(c, op.n, op.flags, op.vu, op.vv, op.area, volume);
  if (threadIdx.x == 0 && slot < MAX_OPS) d.clock->op_influx[slot] += applied;
}

// One sww frame (file/sww.py:352-410 store_timestep, smoothed node values):
// per node the mean over its vertex slots in the order the caller gives (the
// reference's vertex_value_indices, summed and divided as quantity.c:823-915
// do, total / k) of the centroid values of the slots' triangles
// (centroid_avg: the DE algorithms' centroid averaging,
// shallow_water_domain.py:596) or of the slots' vertex values; a node is
// storable when its mean stage minus its mean bed is at least
// minimum_storable_height: otherwise the stage stored is the bed and the
// momenta are zero.  Centroid values are stored as they are.  All as float.
__global__ void k_sww_nodes(Dev d, int P, const int* off, const int* slot, double msh, int centroid_avg, float* out) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= P) return;
  double aw = 0.0, az = 0.0, au = 0.0, av = 0.0;
  const int a = off[p], b = off[p + 1];
  for (int q = a; q < b; q++) {
    const int s = slot[q];
    if (centroid_avg) {
      const int k = s / 3;
      aw += d.w[k];
      az += d.z[k];
      au += d.uh[k];
      av += d.vh[k];
    } else {
      aw += d.wv[s];
      az += d.zv[s];
      au += d.uhv[s];
      av += d.vhv[s];
    }
  }
  if (b > a) {
    const double k = (double)(b - a);
    aw = aw / k;
    az = az / k;
    au = au / k;
    av = av / k;
  }
  const bool storable = aw - az >= msh;
  out[p] = (float)(storable ? aw : az);
  out[P + p] = storable ? (float)au : 0.0f;
  out[2 * P + p] = storable ? (float)av : 0.0f;
}

__global__ void k_sww_cells(Dev d, float* out) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= d.N) return;
  out[k] = (float)d.w[k];
  out[d.N + k] = (float)d.uh[k];
  out[2 * d.N + k] = (float)d.vh[k];
}


// The clock of a step that ends with operators.
__global__ void k_clock(Dev d, cudaGraphConditionalHandle handle, int set_cond) {
  const int reason = clock_logic(d.clock);
  if (set_cond) cudaGraphSetConditional(handle, reason == 0 ? 1u : 0u);
}

// ---------------------------------------------------------------------------
static inline int nblk(int n) { return (n + TPB - 1) / TPB; }
// Meshes from here on take the integer products (see imul).  us a step with
// them and without, two scenes in DE0 and DE1 (dam DE0, inflow DE0, dam DE1,
// inflow DE1):
//    4,900 cells   41.3/39.1   42.4/39.6   69.9/65.1   74.2/67.4
//   14,900         43.9/43.7   43.6/40.9   75.7/73.0   78.3/72.4
//   20,200         46.9/45.4   46.9/45.5   79.1/81.0   81.6/79.3
//   30,300         51.8/54.8   50.2/50.3   88.8/92.9   86.5/85.7
//   40,000         58.5/62.9   54.1/55.6  101.7/109.6  97.2/99.0
//  160,000        137.6/154.9 119.2/129.0 249.4/282.7 214.7/236.4
// With few warps a scheduler the longer chain of an integer product shows, with
// many the FP64 pipe is full.  They cross between 20,000 and 30,000 cells, the
// extrapolation first, the accumulation last; the difference there is within 4%
// either way.
constexpr int IMUL_MIN_CELLS = 20000;
static inline int xblk(int n) { return (n + XCELLS - 1) / XCELLS; }

#define LAUNCHK(cat, ...)                  \
  do {                                     \
    __VA_ARGS__;                           \
    count_launch();                        \
    cudaError_t _e = cudaGetLastError();   \
    if (_e != cudaSuccess) return _e;      \
    phase_mark(st, cat);                   \
  } while (0)
#define LAUNCH(...) LAUNCHK(PH_SMALL, __VA_ARGS__)

template <bool VERT>
static cudaError_t launch_extrap(const Dev& d, cudaStream_t st) {
  if (d.N < IMUL_MIN_CELLS) LAUNCHK(PH_EXTRAP, k_extrap<VERT, false><<<xblk(d.N), XTPB, 0, st>>>(d));
  else LAUNCHK(PH_EXTRAP, k_extrap<VERT, true><<<xblk(d.N), XTPB, 0, st>>>(d));
  return cudaSuccess;
}
template <bool BC>
static cudaError_t launch_flux(const Dev& d, cudaStream_t st, double frac) {
  if (d.N < IMUL_MIN_CELLS) LAUNCHK(PH_FLUX, k_flux<BC, false><<<nblk(d.E), TPB, 0, st>>>(d, frac));
  else LAUNCHK(PH_FLUX, k_flux<BC, true><<<nblk(d.E), TPB, 0, st>>>(d, frac));
  return cudaSuccess;
}
static cudaError_t launch_accum(const Dev& d, cudaStream_t st, int substep, int timestep) {
  if (d.N < IMUL_MIN_CELLS) LAUNCHK(PH_ACCUM, k_accum<false><<<nblk(d.N), TPB, 0, st>>>(d, substep, timestep));
  else LAUNCHK(PH_ACCUM, k_accum<true><<<nblk(d.N), TPB, 0, st>>>(d, substep, timestep));
  return cudaSuccess;
}

cudaError_t enqueue_distribute(Scenario* s, cudaStream_t st, bool with_protect, bool vertices) {
  const Dev& d = s->d;
  if (d.N == 0) return cudaSuccess;
  LAUNCHK(PH_PREP, k_prep<<<nblk(d.N), TPB, 0, st>>>(d, with_protect ? 0 : 2));
  if (vertices) return launch_extrap<true>(d, st);
  return launch_extrap<false>(d, st);
}

cudaError_t enqueue_protect(Scenario* s, cudaStream_t st) {
  if (s->d.N == 0) return cudaSuccess;
  LAUNCHK(PH_PREP, k_prep<<<nblk(s->d.N), TPB, 0, st>>>(s->d, 4));
  return cudaSuccess;
}

cudaError_t enqueue_boundary(Scenario* s, cudaStream_t st, double t_override) {
  const Dev& d = s->d;
  if (d.B == 0) return cudaSuccess;
  LAUNCHK(PH_BC, k_bc<<<nblk(d.B), TPB, 0, st>>>(d, t_override));
  return cudaSuccess;
}

cudaError_t enqueue_fluxes(Scenario* s, cudaStream_t st, int substep) {
  const Dev& d = s->d;
  if (d.N == 0) return cudaSuccess;
  if (cudaError_t e = launch_flux<false>(d, st, 0.0)) return e;
  return launch_accum(d, st, substep, 0);
}

cudaError_t enqueue_forcing(Scenario* s, cudaStream_t st) {
  const Dev& d = s->d;
  if (d.N == 0) return cudaSuccess;
  LAUNCHK(PH_UPDATE, k_forcing<<<nblk(d.N), TPB, 0, st>>>(d));
  return cudaSuccess;
}

cudaError_t enqueue_update(Scenario* s, cudaStream_t st, int stage, bool use_clock_dt, double dt) {
  const Dev& d = s->d;
  if (d.N == 0) return cudaSuccess;
  // stage < 0: forcing already accumulated (per-phase API)
  LAUNCHK(PH_UPDATE, k_update<false><<<nblk(d.N), TPB, 0, st>>>(d, stage, use_clock_dt ? 1 : 0, dt, 0, 0, 0, 0));
  return cudaSuccess;
}

cudaError_t enqueue_backup(Scenario* s, cudaStream_t st) {
  if (s->d.N == 0) return cudaSuccess;
  LAUNCH(k_backup<<<nblk(s->d.N), TPB, 0, st>>>(s->d));
  return cudaSuccess;
}

cudaError_t enqueue_divide(Scenario* s, cudaStream_t st, double divisor) {
  if (s->d.N == 0) return cudaSuccess;
  LAUNCH(k_divide<<<nblk(s->d.N), TPB, 0, st>>>(s->d, divisor));
  return cudaSuccess;
}

cudaError_t enqueue_saxpy(Scenario* s, cudaStream_t st, double a, double b) {
  if (s->d.N == 0) return cudaSuccess;
  LAUNCH(k_saxpy<<<nblk(s->d.N), TPB, 0, st>>>(s->d, a, b));
  return cudaSuccess;
}

cudaError_t enqueue_geo_transpose(Scenario* s, cudaStream_t st, const double* rows) {
  if (s->d.N == 0) return cudaSuccess;
  LAUNCH(k_geo_transpose<<<nblk(s->d.N), TPB, 0, st>>>((double*)s->d.geo, rows, s->d.N));
  return cudaSuccess;
}

// One full timestep (Euler, RK2 or RK3), ending with the clock.  Fused so that
// a DE1 step takes 9 launches instead of 20 (DE0: 5 instead of 12).
cudaError_t enqueue_step(Scenario* s, cudaStream_t st, unsigned long long cond_handle, bool set_cond) {
  const Dev& d = s->d;
  const int nb = nblk(d.N);
  const int stages = s->prm.timestepping_method;
  // times of the stages within the step (of time series) and how each
  // stage's update combines with the step's start (k_update's saxpy)
  const double frac[3] = {0.0, 1.0, 0.5};
  const int combine[3] = {0, stages == 2 ? 1 : 2, 3};
  const cudaGraphConditionalHandle h = (cudaGraphConditionalHandle)cond_handle;
  const int sc = set_cond ? 1 : 0;
  LAUNCHK(PH_PREP, k_prep<<<nb, TPB, 0, st>>>(d, stages > 1 ? 1 : 0));
  for (int i = 0; i < stages; i++) {
    const bool last = i == stages - 1;
    if (cudaError_t e = launch_extrap<false>(d, st)) return e;
    if (cudaError_t e = launch_flux<true>(d, st, frac[i])) return e;
    if (cudaError_t e = launch_accum(d, st, i, i == 0 ? 1 : 0)) return e;
    if (!last) LAUNCHK(PH_UPDATE, k_update<true><<<nb, TPB, 0, st>>>(d, 1, 1, 0.0, combine[i], 0, h, sc));
    else LAUNCHK(PH_UPDATE, k_update<false><<<nb, TPB, 0, st>>>(d, 1, 1, 0.0, combine[i], s->ops.empty() ? 1 : 0, h, sc));
  }
  for (size_t i = 0; i < s->ops.size(); i++) {
    const RateOp& op = s->ops[i];
    if (op.kind == 1) {
      LAUNCHK(PH_RATE, k_inlet<<<1, INLET_TPB, 0, st>>>(d, op, (int)i, op.rate, op.rate, -1.0));
    } else {
      LAUNCHK(PH_RATE, k_rate<<<nblk(op.n), TPB, 0, st>>>(d, op.idx, op.n, op.rate, op.factor, (int)i, -1.0));
    }
  }
  if (!s->ops.empty()) LAUNCH(k_clock<<<1, 1, 0, st>>>(d, h, sc));
  return cudaSuccess;
}

cudaError_t enqueue_rate_once(Scenario* s, cudaStream_t st, int i, double rate, double factor, double dt) {
  const Dev& d = s->d;
  const RateOp& op = s->ops[i];
  if (op.n == 0) return cudaSuccess;
  if (op.kind == 1) {
    LAUNCHK(PH_RATE, k_inlet<<<1, INLET_TPB, 0, st>>>(d, op, i, rate, factor, dt));
  } else {
    LAUNCHK(PH_RATE, k_rate<<<nblk(op.n), TPB, 0, st>>>(d, op.idx, op.n, rate, factor, i, dt));
  }
  return cudaSuccess;
}

cudaError_t enqueue_sww_frame(Scenario* s, cudaStream_t st, double msh, int centroid_avg) {
  const Dev& d = s->d;
  if (s->P > 0)
    LAUNCH(k_sww_nodes<<<nblk(s->P), TPB, 0, st>>>(d, s->P, s->node_off, s->node_slot, msh, centroid_avg, s->frame));
  if (d.N > 0) LAUNCH(k_sww_cells<<<nblk(d.N), TPB, 0, st>>>(d, s->frame + 3 * (size_t)s->P));
  return cudaSuccess;
}

}  // namespace agx
