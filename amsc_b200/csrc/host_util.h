// host_util.h -- host-side helpers shared by the single-scenario and batch
// boundaries: device geometry and physics from the C-ABI structs.
#pragma once
#include <cmath>

#include "../../include/dampm_cuda.h"
#include "dampm_kernels.h"

namespace dampm {

// grid.set_sizes(Ney, Nex, hx, hy) (main/optim_par.cpp:136): rows = Ney.
inline Geom make_geom(const dampm_grid& g) {
  Geom G{};
  G.nrows = g.Ney;
  G.ncols = g.Nex;
  G.hx = g.hx;
  G.hy = g.hy;
  G.Lx = g.Nex * g.hx;
  G.Ly = g.Ney * g.hy;
  int e;
  G.hx_pow2 = std::frexp(g.hx, &e) == 0.5 ? 1 : 0;
  G.hy_pow2 = std::frexp(g.hy, &e) == 0.5 ? 1 : 0;
  G.ihx = 1.0 / g.hx;
  G.ihy = 1.0 / g.hy;
  int L = 0;
  while ((1LL << L) < g.Ney) ++L;
  G.rshift = 31 + L;
  G.rmul = unsigned((1ULL << G.rshift) / unsigned(g.Ney) + 1);
  set_pieces(G, 0);
  G.pc_lo = 0;
  G.pc_hi = g.Nex;
  G.nc_lo = 0;
  G.nc_hi = g.Nex;
  return G;
}

inline Phys make_phys(const dampm_params& d) {
  Phys P{};
  P.g = d.g;
  P.rho = d.rho;
  P.mu = d.mu;
  P.tauy = d.tauy;
  P.xi = d.xi;
  const double fric_ang = d.phi * M_PI / 180.;  // main/optim_par.cpp:193
  P.tan_fa = std::tan(fric_ang);
  P.BING = d.BINGHAM_ON;
  P.FON = d.FRICTION_ON;
  P.CFL = d.CFL;
  P.eq_level = d.eq_level;
  P.DT_FIXED = d.DT_FIXED;
  P.T = d.T;
  P.BC = d.BC_FLAG;
  P.NSTEPS = d.NSTEPS;
  P.fixed = d.DT_FIXED > 0.0 ? 1 : 0;
  return P;
}

// The condition a pass's sort runs on (Gate): begun != 0 where the step has
// begun before it.
inline Gate make_gate(const Phys& P, int begun) {
  return Gate{begun, P.fixed, P.NSTEPS, P.T};
}

inline int grid_blocks(long long n, int threads) {
  long long b = (n + threads - 1) / threads;
  if (b < 1) b = 1;
  if (b > 148 * 16) b = 148 * 16;
  return int(b);
}

// Host halves (a, b) of n pairs into a pair array: one linear copy each into
// the scratch arrays ta and tb, joined on the device.  (As two strided copies
// into the pairs, 8 bytes a row, 4M pairs took 13 ms instead of 1.3.)
inline cudaError_t upload_pair(double2* dst, const double* a, const double* b, long long n,
                               double* ta, double* tb, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  cudaError_t e = cudaMemcpyAsync(ta, a, sizeof(double) * size_t(n), cudaMemcpyHostToDevice, st);
  if (e != cudaSuccess) return e;
  e = cudaMemcpyAsync(tb, b, sizeof(double) * size_t(n), cudaMemcpyHostToDevice, st);
  if (e != cudaSuccess) return e;
  k_pair_join<<<grid_blocks(n, 256), 256, 0, st>>>(ta, tb, dst, n);
  return cudaGetLastError();
}

// Half `half` (0: first, 1: second) of n pairs to the host, through scratch t.
inline cudaError_t download_pair_half(double* out, const double2* src, int half, long long n,
                                      double* t, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  k_pair_half<<<grid_blocks(n, 256), 256, 0, st>>>(src, half, t, n);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  return cudaMemcpyAsync(out, t, sizeof(double) * size_t(n), cudaMemcpyDeviceToHost, st);
}

}  // namespace dampm
