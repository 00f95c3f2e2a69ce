// qas_stage1d.cuh -- one SSP-RK stage of the 1D step in one kernel (MHD1D::ideal,
// 1D/SERIAL/shock/mhd1d_solve.cpp:3-124, with the ghost fill and exec_'s loop test folded in).
//
// A 1D grid has some thousand cells: a stage in five launches is five launch latencies and five
// trips through L2 for a few microseconds of dependent arithmetic (Brio-Wu 1024: 62.7 us a step, 22.6 us
// this way, most of it the dependent FP64 chain of one cell's states and flux).  Here a block takes TC cells and the
// four on either side that their update reads, and keeps primitives, face states and fluxes in shared
// memory; cells past the ends are gathered through the ghost map, so no stage waits for a fill.
// Thread t works on cell s - 4 + t: primitives for all, face states for t in [2, NT - 2), the flux at the
// cell's left face for t in [3, NT - 2), the update for t in [4, NT - 4).
#pragma once

#include "qas_kernels.cuh"

namespace qas {

constexpr int S1_NT = 64;             // threads of a block
constexpr int S1_TC = S1_NT - 2 * GH;  // cells a block updates

// P(f, m) on the block's primitives
struct Stencil1 {
  const double (*q)[S1_NT];
  int t;
  __device__ __forceinline__ double operator()(int f, int m) const { return q[f][t + m - 2]; }
};
// the states of a thread's cell into shared memory; beyond the fast interpolation's range the
// reference's divisions, out of line
template <int ODR>
__device__ __noinline__ void states1_again(const double (*q)[S1_NT], int t, double bn, double gam, double *l, double *r)
{
  double vl[7], vr[7];
  face_states_of<ODR>(Stencil1{q, t}, bn, gam, vl, vr);
  for (int m = 0; m < 7; m++) {
    l[m * S1_NT] = vl[m];
    r[m * S1_NT] = vr[m];
  }
}
template <int ODR>
struct States1 {
  double *l, *r;
  __device__ __forceinline__ void operator()(int m, double lv, double rv) const
  {
    l[m * S1_NT] = lv;
    r[m * S1_NT] = rv;
  }
  __device__ __forceinline__ void again(const Stencil1 &P, double bn, double gam) const
  {
    states1_again<ODR>(P.q, P.t, bn, gam, l, r);
  }
};

// last: the step's last stage, whose last block to finish advances exec_'s counters
template <int ODR, int RMN>
__global__ void __launch_bounds__(S1_NT) k_stage1(const __grid_constant__ View v, double c0, double c1, int check_tim,
                                                  int last)
{
  pdl_begin();
  Ctl *ctl = v.ctl;
  if (ctl->done) return;
  const bool go = run_goes_on(ctl, check_tim);
  __shared__ double q[7][S1_NT], sl[7][S1_NT], sr[7][S1_NT];
  const Geo &g = v.g;
  const int t = threadIdx.x;
  const int i = GH + blockIdx.x * S1_TC - GH + t;  // padded index; the last block may run past the grid
  if (go) {
    const double dtdx = ctl->dt / v.dx;
    const bool in = i < g.nx;
    double u[8], ut[8];
    if (in) {
#pragma unroll
      for (int m = 0; m < 8; m++) {
        const int s = map_src(v.maps, 0, m, 0, i);
        const double x = v.u[m][s];
        u[m] = s == i ? x : map_fac(v.maps, 0, m, 0, i) * x;
      }
    } else {
#pragma unroll
      for (int m = 0; m < 8; m++) u[m] = m == 0 || m == 7 ? 1.0 : 0.0;  // a state to compute on, never used
    }
    const bool mine = t >= GH && t < S1_NT - GH && i < g.nx - GH;
    if (mine) {
#pragma unroll
      for (int m = 0; m < 8; m++) ut[m] = c0 == 0.0 ? u[m] : v.u0[m][i];
    }
    {
      const double ro = u[0], iro = 1.0 / ro;
      const double vx = u[1] * iro, vy = u[2] * iro, vz = u[3] * iro;
      const double v2 = vx * vx + vy * vy + vz * vz;
      const double b2 = u[4] * u[4] + u[5] * u[5] + u[6] * u[6];
      const double pr = (v.gam - 1) * (u[7] - 0.5 * (ro * v2 + b2));
      q[0][t] = ro;
      q[1][t] = vx;
      q[2][t] = vy;
      q[3][t] = vz;
      q[4][t] = u[5];
      q[5][t] = u[6];
      q[6][t] = pr;
      if (mine && !(ro > 0.0 && pr > 0.0 && isfinite(vx) && isfinite(vy) && isfinite(vz))) atomicOr(&ctl->err, 1);
    }
    __syncthreads();
    if (t >= 2 && t < S1_NT - 2) {
      const Stencil1 st{q, t};
      if (v.recon == 1) {
        double vl[7], vr[7];
        face_states_prim<ODR>(st, vl, vr);
#pragma unroll
        for (int m = 0; m < 7; m++) {
          sl[m][t] = vl[m];
          sr[m][t] = vr[m];
        }
      } else {
        face_states_emit<ODR>(st, u[4], v.gam, States1<ODR>{&sl[0][t], &sr[0][t]});
      }
    }
    __syncthreads();
    double F[7];
    if (t >= 3 && t < S1_NT - 2) {
      double L[7], R[7];
#pragma unroll
      for (int m = 0; m < 7; m++) {
        L[m] = sl[m][t - 1];
        R[m] = sr[m][t];
      }
      riemann<RMN>(L, R, u[4], v.gam, v.gm1i, RMN >= 2 ? q[1][t] - q[1][t - 1] : 0.0, 0.0, F);
    }
    __syncthreads();
    if (t >= 3 && t < S1_NT - 2) {
#pragma unroll
      for (int m = 0; m < 7; m++) sl[m][t] = F[m];
    }
    __syncthreads();
    if (mine) {
      const int to[7] = {0, 1, 2, 3, 5, 6, 7};
#pragma unroll
      for (int m = 0; m < 7; m++) {
        const double du = -dtdx * dfc<ODR>(sl[m][t - 1], sl[m][t], sl[m][t + 1], sl[m][t + 2]);
        v.uo[to[m]][i] = rk_combine(u[to[m]], ut[to[m]], du, c0, c1);
      }
    }
  }
  if (!last || t != 0) return;
  // every block has read the counters when the last one comes here
  if (atomicAdd(&ctl->ticket, 1u) == gridDim.x - 1) {
    ctl->ticket = 0;
    begin_body(v, check_tim);
  }
}

// the ghost fill at the end of a call whose steps ran by k_stage1 (which neither reads nor writes ghosts)
static __global__ void k_bound_end(View v, int n0)
{
  pdl_begin();
  if (v.ctl->n == n0) return;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= shell_cells(v.g)) return;
  int i, j, k;
  shell_cell(v.g, t, i, j, k);
  bound_body(v, i, j, k);
}

// the stage kernel (qas_stage1d.cu) of an order (2 or 4) and solver
using Stage1Fn = void (*)(const View, double, double, int, int);
Stage1Fn stage1_kernel(int odr, int rmn);

}  // namespace qas
