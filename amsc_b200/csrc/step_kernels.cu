// step_kernels.cu -- the FP64 MPM time step on sm_100a.
//
// One pass of the loop body of main/optim_par.cpp:281-668 is
//   SORT        : scan -> scatter -> per-cell order (G2P counted the keys; a1);
//                 the last kernel also cuts P2G's work list, ends the step before
//                 (t += dt) and begins this one -- dt (fixed or CFL from the
//                 previous G2P's max-reductions), it++
//   P2G+NODAL   : per-node sequential chains over the sorted particles of the
//                 node's 4 cells, nodal momentum/velocity/BC  (a2-a7, a10, a14)
//   G2P         : velocity, advection, gradients, height, Bingham stress,
//                 next cell key, CFL max-reductions  (a8, a9, a11, a13); one
//                 block of its own sums the ledger
// The loop state lives on the device: no host synchronisation in a pass.
#include <cstdio>

#include "dampm_device.cuh"
#include "dampm_kernels.h"

namespace dampm {

// ---------------------------------------------------------------------------
// loop control
// ---------------------------------------------------------------------------
// The end of the step that G2P left pending.
__device__ __forceinline__ void step_end_one(Scalars* S) {
  if (!S->pending) return;
  S->pending = 0;
  S->t += S->dt;
  S->fresh = 0;
  S->red_cur[0] = S->red_next[0];
  S->red_cur[1] = S->red_next[1];
  S->red_cur[2] = S->red_next[2];
}

// One scenario's pass start, after the end of the one before: the loop
// condition, dt, it++ (device side).
__device__ __forceinline__ void step_begin_one(Scalars* S, const Geom& G,
                                               const Phys& P) {
  step_end_one(S);
  const bool cond = P.fixed ? (S->it < P.NSTEPS) : (S->t < P.T);
  if (!cond || S->status != 0) {
    S->active = 0;
    return;
  }
  S->active = 1;
  double dt;
  if (P.fixed) {
    dt = P.DT_FIXED;
  } else {
    // main/optim_par.cpp:289-304; first pass: 1e-3 (main/gpu_offload.cpp:255)
    dt = 1.0e-3;
    if (S->it > 0) {
      const double mvx = ordered_value(S->red_cur[0]);
      const double mvy = ordered_value(S->red_cur[1]);
      const double hmean = ordered_value(S->red_cur[2]);
      const double a = sqrt(P.g * hmean) + mvx;
      const double b = sqrt(P.g * hmean) + mvy;
      const double max_vel = (a < b) ? b : a;  // std::max
      const double cel = fabs(max_vel);
      const double hmin = (G.hy < G.hx) ? G.hy : G.hx;  // std::min
      dt = P.CFL * hmin / (1e-2 + cel);
    }
  }
  S->dt = dt;
  S->it += 1;
  S->red_next[0] = S->red_next[1] = S->red_next[2] = 0ull;
}

// The last of n blocks to call it (counted in *arrived, which it resets): all
// its threads get true.  What thread 0 of a block did before (its stores, its
// atomics) is visible to the last block past L1.
__device__ __forceinline__ bool last_block(int* arrived, int n) {
  __shared__ int last;
  __syncthreads();  // every thread has done its part (and left a call before)
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(arrived, 1) == n - 1;
    if (last) *arrived = 0;
    __threadfence();
  }
  __syncthreads();
  return last;
}

// The pass start as a launch of its own: a merge/split at the cadence comes
// between it and the sort.
__global__ void k_step_begin(Scalars* S, Geom G, Phys P) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  step_begin_one(S, G, P);
}

// The step end as a launch of its own, after the last pass of a call: the
// state is complete when the host reads it.
__global__ void k_step_end(Scalars* S) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  step_end_one(S);
  // slab mode: the neighbour's column copies were read by P2G only; G2P
  // wrote the slab's own particles
  S->np -= S->nghost;
  S->nghost = 0;
}

// ---------------------------------------------------------------------------
// initialisation after upload: main/optim_par.cpp:239-264
// ---------------------------------------------------------------------------
template <class R>
__global__ void k_init_particles(ParticlesT<R> p, const double* __restrict__ Z,
                                 const double* __restrict__ dZdx,
                                 const double* __restrict__ dZdy, Geom G,
                                 Phys P, Scalars* S, int np, int key_off) {
  __shared__ unsigned long long red[3];
  if (threadIdx.x < 3) red[threadIdx.x] = 0ull;
  __syncthreads();
  unsigned long long m0 = 0, m1 = 0, m2 = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < np;
       i += gridDim.x * blockDim.x) {
    const double x = p.x[i], y = p.y[i];
    const int r = cell_row(y, G), c = cell_col(x, G);
    p.key[i] = r + c * G.nrows + key_off;
    p.idx[i] = i;
    p.label[i] = i;
    p.level[i] = 0;
    double xi, eta;
    local_xy(x, y, c, r, G.hx, G.hy, xi, eta);
    double zp = 0.0, dzx = 0.0, dzy = 0.0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const double N = shp(xi, eta, k);
      const int n = node_of(k, c, r, G.nrows);
      zp += N * Z[n];
      dzx += N * dZdx[n];
      dzy += N * dZdy[n];
    }
    const double hp = p.hp[i];
    const double diff = P.eq_level - zp;
    const double H = (P.eq_level > 0 && diff > 0) ? diff : 0.0;
    p.H[i] = H;
    const double h_corr = hp > 1e-10 ? hp - (H * H) / hp : 0.0;
    const double f = -.5 * P.rho * P.g * h_corr;
    p.F11[i] = f;
    p.F12[i] = 0.0;
    p.F22[i] = f;
    p.Fbx[i] = 0.0;
    p.Fby[i] = 0.0;
    if (p.Zp) {
      p.Zp[i] = zp;
      p.hpZ[i] = hp + zp;
      p.dZxp[i] = dzx;
      p.dZyp[i] = dzy;
    }
    m0 = max(m0, ordered_key(fabs(p.vpx[i])));
    m1 = max(m1, ordered_key(fabs(p.vpy[i])));
    m2 = max(m2, ordered_key(hp));
  }
  atomicMax(&red[0], m0);
  atomicMax(&red[1], m1);
  atomicMax(&red[2], m2);
  __syncthreads();
  if (threadIdx.x == 0) {
    atomicMax(&S->red_cur[0], red[0]);
    atomicMax(&S->red_cur[1], red[1]);
    atomicMax(&S->red_cur[2], red[2]);
  }
}

// Recomputes the cell key of every particle after a merge/split emit (which
// wrote idx) or a state upload (slots in reference order: set_idx sets
// idx = slot); the next sort scans every cell.
__global__ void k_keys(Particles p, Geom G, Scalars* S, int set_idx) {
  const int np = S->np;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < np;
       i += gridDim.x * blockDim.x) {
    const int r = cell_row(p.y[i], G);
    const int c = cell_col(p.x[i], G);
    p.key[i] = r + c * G.nrows;
    if (set_idx) p.idx[i] = i;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    S->knext[0] = 0;
    S->knext[1] = G.nrows * G.ncols - 1;
  }
}

// Max-reductions of the current state (for the next CFL dt).
__global__ void k_reduce_state(Particles p, Scalars* S) {
  __shared__ unsigned long long red[3];
  if (threadIdx.x < 3) red[threadIdx.x] = 0ull;
  __syncthreads();
  unsigned long long m0 = 0, m1 = 0, m2 = 0;
  const int np = S->np;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < np;
       i += gridDim.x * blockDim.x) {
    m0 = max(m0, ordered_key(fabs(p.vpx[i])));
    m1 = max(m1, ordered_key(fabs(p.vpy[i])));
    m2 = max(m2, ordered_key(p.hp[i]));
  }
  atomicMax(&red[0], m0);
  atomicMax(&red[1], m1);
  atomicMax(&red[2], m2);
  __syncthreads();
  if (threadIdx.x == 0) {
    atomicMax(&S->red_cur[0], red[0]);
    atomicMax(&S->red_cur[1], red[1]);
    atomicMax(&S->red_cur[2], red[2]);
  }
}

template <class R>
struct ShapeT {
  R ihx, mihx, ihy, mihy;
};
// 1/h, -1/h: in FP64 the geometry's (the host's quotient is the same value)
template <class R>
__device__ __forceinline__ ShapeT<R> shape_of(const Geom& G) {
  if constexpr (sizeof(R) == 8) {
    return ShapeT<R>{G.ihx, -G.ihx, G.ihy, -G.ihy};
  } else {
    const R ihx = R(1) / R(G.hx), ihy = R(1) / R(G.hy);
    return ShapeT<R>{ihx, -ihx, ihy, -ihy};
  }
}
using Shape = ShapeT<double>;

// Record of the next P2G for every particle (see Particles): from the stored
// Ap/Fb/mom (derive == 0: after an upload or a merge/split) or from the state
// alone (derive != 0), exactly as the reference computes these values
// (main/optim_par.cpp:387,447-459,600-626).
// The terrain gradient and the well-balanced factor 1 - H/hp are evaluated
// in FP64 whatever R is (the bed slope and the near-cancelling free-surface
// difference).
template <class R>
__device__ __forceinline__ void next_record(const Geom& G, const Phys& P,
                                            const double* __restrict__ Z, R x,
                                            R y, R hp, R H, R Vp, R& xi, R& eta,
                                            R& gx, R& gy) {
  const int r = cell_row(double(y), G);
  const int c = cell_col(double(x), G);
  const ShapeT<R> sh = shape_of<R>(G);
  local_xy_g(x, y, c, r, G, sh.ihx, sh.ihy, xi, eta);
  // g2pd Z -> dZxp, dZyp (main/optim_par.cpp:387)
  const double dihx = G.ihx, dmihx = -G.ihx;
  const double dihy = G.ihy, dmihy = -G.ihy;
  const double dxi = xi, deta = eta;
  double dzx = 0.0, dzy = 0.0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const double zn = Z[node_of(k, c, r, G.nrows)];
    dzx += shg_x(deta, k, dihx, dmihx) * zn;
    dzy += shg_y(dxi, k, dihy, dmihy) * zn;
  }
  // gravity along the bed, well balanced (main/optim_par.cpp:447-454)
  const double hpd = hp, Hd = H, Vpd = Vp;
  // H/hp is +0 when H == 0 (no still-water level): 1 - 0 is 1
  const double wb = (hpd > 1e-10 && Hd != 0.0) ? 1.0 - (Hd / hpd) : 1.0;
  gx = R(-P.g * Vpd * P.rho * dzx * wb);
  gy = R(-P.g * Vpd * P.rho * dzy * wb);
}

template <class R>
__global__ void k_prep(ParticlesT<R> p, const double* __restrict__ Z, Geom G,
                       Phys P, const Scalars* S, int derive) {
  const int np = S->np;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < np;
       i += gridDim.x * blockDim.x) {
    const R hp = p.hp[i];
    R Ap, fbx, fby;
    if (derive) {
      Ap = hp > R(1.e-2) ? p.Vp[i] / hp : R(0);
      rheology_friction<R>(P, p.vpx[i], p.vpy[i], hp, fbx, fby);
      p.mp[i] = V2<R>{p.vpx[i] * p.Mp[i], p.vpy[i] * p.Mp[i]};
    } else {  // the stored values, in reference order
      const int r = p.idx[i];
      Ap = p.Ap[r];
      fbx = p.Fbx[r];
      fby = p.Fby[r];
    }
    p.qf[i] = V2<R>{Ap * fbx, Ap * fby};
    R xi, eta, gx, gy;
    next_record<R>(G, P, Z, p.x[i], p.y[i], hp, p.H[i], p.Vp[i], xi, eta, gx, gy);
    p.xe[i] = V2<R>{xi, eta};
    p.qg[i] = V2<R>{gx, gy};
  }
}

// ---------------------------------------------------------------------------
// SORT: stable counting sort by cell, (cell, particle index) order
// (init_particle_mesh + cell_start/cell_ptcls, main/gpu_offload.cpp:243-249)
// ---------------------------------------------------------------------------
// The counting sort's first step, done where the keys are made (G2P; k_count
// after an upload or a merge/split): a particle of cell k takes a slot among its
// cell's particles, one atomic per cell and warp (the lanes that share a cell
// take consecutive slots), and its tile of kScanTile cells counts it, mostly
// with one more atomic per warp, whose result nobody waits for: the scan needs
// no pass of its own over the counts for the tile totals (a launch of 7 us at 4M
// particles, 3 at 0.25M, 8 for 96 scenarios).
// tile_sum may be null (a grid that k_scan_scatter takes).  All 32 lanes call
// it; ok == false lanes take part without a particle.
__device__ __forceinline__ void count_key(int k, bool ok, int* __restrict__ count,
                                          int* __restrict__ tile_sum,
                                          int* __restrict__ slot_out) {
  const int lane = threadIdx.x & 31;
  const int kk = ok ? k : -1;
  const unsigned peers = __match_any_sync(0xffffffffu, kk);
  const int leader = __ffs(peers) - 1;
  int base = 0;
  if (ok && lane == leader) base = atomicAdd(&count[kk], __popc(peers));
  if (tile_sum) {
    const unsigned who = __ballot_sync(0xffffffffu, ok);
    const int first = __ffs(who) - 1, t = kk / kScanTile;
    const int t0 = __shfl_sync(0xffffffffu, t, first & 31);
    if (__all_sync(0xffffffffu, !ok || t == t0)) {
      if (lane == first) atomicAdd(&tile_sum[t * kTileStride], __popc(who));
    } else if (ok && lane == leader) {
      atomicAdd(&tile_sum[t * kTileStride], __popc(peers));
    }
  }
  base = __shfl_sync(0xffffffffu, base, leader);
  if (ok) *slot_out = base + __popc(peers & ((1u << lane) - 1u));
}

// Slots and counts of the keys [0, n).
__device__ __forceinline__ void count_keys(const int* __restrict__ key, int* __restrict__ count,
                                           int* __restrict__ tile_sum, int* __restrict__ slot,
                                           int n) {
  const int lane = threadIdx.x & 31;
  const int stride = gridDim.x * blockDim.x;
  for (int i0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31); i0 < n; i0 += stride) {
    const int i = i0 + lane;
    const bool ok = i < n;
    count_key(ok ? key[i] : -1, ok, count, tile_sum, slot + (ok ? i : 0));
  }
}
__global__ void k_count(const int* __restrict__ key, int* __restrict__ count,
                        int* __restrict__ tile_sum, int* __restrict__ slot, const Scalars* S) {
  if (S->active) count_keys(key, count, tile_sum, slot, S->np);
}
__global__ void k_count_n(const int* __restrict__ key, int* __restrict__ count,
                          int* __restrict__ tile_sum, int* __restrict__ slot, int n) {
  count_keys(key, count, tile_sum, slot, n);
}

// Cells of more than kCrowded particles are ordered by a block each (see
// order_crowded).
constexpr int kCrowded = 256;
constexpr int kBigRun = 8192;  // entries of a sorted run (two buffers: 128 KB of shared memory)
constexpr unsigned long long kNoEntry = ~0ull;

// Exclusive scan of count[0..n) into start[0..n], restricted to the tiles of
// kScanTile = 4 x kScanThreads cells (each thread one int4) that meet the key
// range [L, H] = krange U knext: the keys the starts describe and the keys
// G2P produced since.  Outside that range no cell's count changed and every
// start is either 0 (below every key) or np (above), as before, so the old
// values stand.  k_scan_apply adds, per tile, the totals of the preceding
// tiles in the range (count_key's, or k_scan_sums') to a block scan.
// count is zeroed on the way (ready for the next step's atomics).  With
// tile flags (batches) only the flagged tiles are scanned: the others hold
// no particle of any scenario, now or at the last sort, so their totals are
// zero and their starts stand.  The crowded cells are listed.
__device__ __forceinline__ int block_incl_scan(int v, int* wsum) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) wsum[w] = incl;
  __syncthreads();
  if (w == 0) {
    const int nw = blockDim.x >> 5;
    int ws = (lane < nw) ? wsum[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, ws, o);
      if (lane >= o) ws += t;
    }
    if (lane < nw) wsum[lane] = ws;  // inclusive warp totals
  }
  __syncthreads();
  return incl + (w > 0 ? wsum[w - 1] : 0);
}

__device__ __forceinline__ int block_sum(int v, int* wsum) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5] = v;
  __syncthreads();
  int t = 0;
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += wsum[w];
  __syncthreads();
  return t;
}

__device__ __forceinline__ int4 load_count4(const int* count, int i0, int n) {
  if (i0 + 3 < n && (i0 & 3) == 0) return *reinterpret_cast<const int4*>(count + i0);
  int4 c;
  c.x = (i0 < n) ? count[i0] : 0;
  c.y = (i0 + 1 < n) ? count[i0 + 1] : 0;
  c.z = (i0 + 2 < n) ? count[i0 + 2] : 0;
  c.w = (i0 + 3 < n) ? count[i0 + 3] : 0;
  return c;
}

// tiles [t0, t1] meet the scan range (t0 > t1: none); ranged == 0: all
__device__ __forceinline__ void scan_tiles_of(const Scalars* S, int n, int ranged, int& t0,
                                              int& t1) {
  if (!ranged) {
    t0 = 0;
    t1 = (n - 1) / kScanTile;
    return;
  }
  int L = min(S->krange[0], S->knext[0]);
  int H = max(S->krange[1], S->knext[1]);
  L = max(L, 0);
  H = min(H, n - 1);
  if (H < L) {
    t0 = 1;
    t1 = 0;
    return;
  }
  t0 = L / kScanTile;
  t1 = H / kScanTile;
}

__global__ void __launch_bounds__(kScanThreads)
    k_scan_sums(const int* __restrict__ count, int n, int* __restrict__ tile_sum,
                const Scalars* S) {
  if (!S->active) return;
  const int t = blockIdx.x;
  __shared__ int wsum[32];
  const int4 c = load_count4(count, t * kScanTile + threadIdx.x * 4, n);
  const int tot = block_sum(c.x + c.y + c.z + c.w, wsum);
  if (threadIdx.x == 0) tile_sum[t * kTileStride] = tot;
}

// Appends a thread's crowded cells among i0 .. i0+3 (of cv particles) to `big`.
__device__ __forceinline__ void list_crowded(const int (&cv)[4], int i0, int* __restrict__ big,
                                             int* __restrict__ big_n) {
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (cv[k] > kCrowded) big[atomicAdd(big_n, 1)] = i0 + k;
}

// A block per tile, its threads four cells in each of kApplyRows rows: one barrier
// between the loads and the stores, and eight blocks per SM.
// (one block of 1024 threads per tile, five barriers: 9.7 us at 4M particles, 12 for
// 96 scenarios; this way 6.3 and 7.7; 12 B a cell in range, which take 3 at 4M)
__global__ void __launch_bounds__(kApplyThreads)
    k_scan_apply(int* __restrict__ count, int n, const int* __restrict__ tile_sum,
                 int* __restrict__ start, int* __restrict__ big, int* __restrict__ list_n,
                 const Scalars* S, Gate gate, int ranged,
                 const unsigned char* __restrict__ tflag) {
  if (!gate_open(S, gate)) return;
  int t0, t1;
  scan_tiles_of(S, n, ranged, t0, t1);
  const int t = blockIdx.x;
  if (t < t0 || t > t1) return;  // block-uniform
  if (tflag && !tflag[t]) return;  // its starts stand (see k_b_step_begin)
  constexpr int kWarps = kApplyThreads / 32;
  static_assert(kApplyRows * kWarps == 32, "one total per lane");
  __shared__ int wsum[32], wpre[kWarps];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int4 c[kApplyRows];
  int v[kApplyRows], incl[kApplyRows];
#pragma unroll
  for (int k = 0; k < kApplyRows; ++k)
    c[k] = load_count4(count, t * kScanTile + (k * kApplyThreads + int(threadIdx.x)) * 4, n);
  // particles in the range's tiles before this one
  int pre = 0;
  for (int q = t0 + threadIdx.x; q < t; q += kApplyThreads) pre += tile_sum[q * kTileStride];
  pre = __reduce_add_sync(0xffffffffu, pre);
#pragma unroll
  for (int k = 0; k < kApplyRows; ++k) {
    v[k] = c[k].x + c[k].y + c[k].z + c[k].w;
    incl[k] = v[k];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, incl[k], o);
      if (lane >= o) incl[k] += u;
    }
    if (lane == 31) wsum[k * kWarps + w] = incl[k];
  }
  if (lane == 0) wpre[w] = pre;
  __syncthreads();
  int tot = wsum[lane];
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, tot, o);
    if (lane >= o) tot += u;
  }
  pre = 0;
#pragma unroll
  for (int k = 0; k < kWarps; ++k) pre += wpre[k];
#pragma unroll
  for (int k = 0; k < kApplyRows; ++k) {
    const int before = __shfl_sync(0xffffffffu, tot, (k * kWarps + w + 31) & 31);
    const int i0 = t * kScanTile + (k * kApplyThreads + int(threadIdx.x)) * 4;
    int4 o;
    o.x = pre + (k + w > 0 ? before : 0) + incl[k] - v[k];
    o.y = o.x + c[k].x;
    o.z = o.y + c[k].y;
    o.w = o.z + c[k].z;
    if (i0 + 3 < n) {
      *reinterpret_cast<int4*>(start + i0) = o;
      *reinterpret_cast<int4*>(count + i0) = make_int4(0, 0, 0, 0);
    } else {
      const int ov[4] = {o.x, o.y, o.z, o.w};
      for (int q = 0; q < 4; ++q)
        if (i0 + q < n) {
          start[i0 + q] = ov[q];
          count[i0 + q] = 0;
        }
    }
    if (big) {
      const int cv[4] = {c[k].x, c[k].y, c[k].z, c[k].w};
      list_crowded(cv, i0, big, list_n);
    }
  }
  // start[n]: the total (with a key range: every particle, unchanged by a
  // step; written whenever the range reaches the last tile)
  if (t == (n - 1) / kScanTile && threadIdx.x == 31) start[n] = pre + tot;
}

// The starts now describe the keys the last G2P made, and the next G2P starts
// an empty range.
__device__ __forceinline__ void roll_keys(Scalars* S) {
  S->krange[0] = S->knext[0];
  S->krange[1] = S->knext[1];
  S->knext[0] = 0x7fffffff;
  S->knext[1] = -1;
}

// Sorted position start[key] + slot takes the storage slot, the reference index
// and the key (the cell of each sorted position, which G2P reads without waiting
// for perm); inside a cell they lie as the count's atomics came.
// kScatterPer particles per thread and trip: their loads, and then those of
// their starts, are on the way together (4M particles: 21 us, one at a time 27; 24 B
// a particle and the starts, which take 16).
constexpr int kScatterPer = 4;
__device__ __forceinline__ void scatter(const Binning& n, const int* start, int np) {
  const int stride = gridDim.x * blockDim.x;
  for (int i0 = blockIdx.x * blockDim.x + threadIdx.x; i0 < np; i0 += kScatterPer * stride) {
    int key[kScatterPer], slot[kScatterPer], idx[kScatterPer];
#pragma unroll
    for (int u = 0; u < kScatterPer; ++u) {
      const long long i = i0 + (long long)u * stride;
      key[u] = -1;
      if (i < np) {
        key[u] = n.key[i];
        slot[u] = n.slot[i];
        idx[u] = n.idx[i];
      }
    }
#pragma unroll
    for (int u = 0; u < kScatterPer; ++u)
      if (key[u] >= 0) slot[u] += start[key[u]];
#pragma unroll
    for (int u = 0; u < kScatterPer; ++u)
      if (key[u] >= 0) {
        n.sslot[slot[u]] = i0 + u * stride;
        n.sidx[slot[u]] = idx[u];
        n.skey[slot[u]] = key[u];
      }
  }
}

// Empties P2G's unit list for the planner that comes after (whether or not a G2P
// followed the last one: half a step, then another upload).
__device__ __forceinline__ void empty_units(int* ucount) {
  if (blockIdx.x == 0 && threadIdx.x < kUnitCounts) ucount[kUnitsPlain + threadIdx.x] = 0;
}

// Also zeroes the tile totals (the scan has used them); block 0 rolls the key
// ranges over.
__global__ void k_scatter(Binning n, const int* __restrict__ start, int* __restrict__ tile_sum,
                          int ntiles, int* __restrict__ ucount, Scalars* S, Gate gate) {
  if (!gate_open(S, gate)) return;
  scatter(n, start, S->np);
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < ntiles; t += gridDim.x * blockDim.x)
    tile_sum[t * kTileStride] = 0;
  empty_units(ucount);
  if (blockIdx.x == 0 && threadIdx.x == 0) roll_keys(S);
}

// The scan and the scatter of a small grid (up to kSmallCells cells) in one
// launch: every block scans all the counts into its shared memory, then
// scatters its share of the particles; block 0 writes the starts and the list
// of crowded cells.  The counts are zeroed by the kernel after (k_order_units):
// blocks that start later still read them.
// At 4096 particles on 64 x 64 cells the launches it replaces (tile totals, scan,
// scatter) took 8.7 us, this one 4.2.  The line lies where a block's share of the
// work, 64 KB of counts from L2, costs what the launches did.
__global__ void __launch_bounds__(kScanThreads)
    k_scan_scatter(const int* __restrict__ count, int ncell, int* __restrict__ start,
                   int* __restrict__ big, int* __restrict__ ucount, Binning n, Scalars* S,
                   Gate gate) {
  if (!gate_open(S, gate)) return;
  extern __shared__ int sstart[];  // ncell
  __shared__ int wsum[32];
  const bool writes = blockIdx.x == 0;
  int carry = 0;
  for (int t = 0; t * kScanTile < ncell; ++t) {
    const int i0 = t * kScanTile + threadIdx.x * 4;
    const int4 c = load_count4(count, i0, ncell);
    const int v = c.x + c.y + c.z + c.w;
    const int incl = block_incl_scan(v, wsum);
    const int total = wsum[(kScanThreads >> 5) - 1];
    const int cv[4] = {c.x, c.y, c.z, c.w};
    int e = carry + incl - v;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (i0 + k < ncell) {
        sstart[i0 + k] = e;
        if (writes) start[i0 + k] = e;
      }
      e += cv[k];
    }
    if (writes) list_crowded(cv, i0, big, ucount);
    carry += total;
    __syncthreads();  // wsum is free again; the starts are in place
  }
  scatter(n, sstart, S->np);
  empty_units(ucount);
  if (writes && threadIdx.x == 0) {
    start[ncell] = carry;
    roll_keys(S);
  }
}

// The order inside the cells, by the particles' reference index (the atomics of
// the count hand out a cell's places in arbitrary order): a position's particle
// goes to the place its index has among those of its cell, counted over the
// cell's indices.  The indices are unique -- two particles with the same one
// would take the same place, and the place behind it none -- except in a slab,
// whose caller numbers the particles: there (kRepeats) equal indices follow in
// the order of their storage slots, as in order_crowded.
// A warp takes tiles of kOrderPer positions per lane, with the indices of all
// their cells in its part `win` of the shared memory (no more than kCrowded
// before and behind the tile): the lanes lie in a
// few cells and mostly read the same word, and no warp waits for another.
// Warp w of nw takes every nw-th tile.
// Before, a lane sorted a cell of up to 16 particles in registers and a warp a
// larger one, from lists of cells: reads of 32 cells by 32 lanes, and at 16
// particles per cell half of the cells in the warps' share.  Counting over the
// indices in global memory is bound by L1's tag lookups, with a block's tile in
// shared memory by the block's barriers (k_order_units 66 and 60 us at 4M
// particles, this way 42, and 36 with the planning warps in blocks of their own,
// below; 16 B a particle, which take 10 us).
constexpr int kOrderPer = 4;
constexpr int kOrderWin = 32 * kOrderPer + 2 * kCrowded;
template <bool kRepeats>
__device__ __forceinline__ void order_cells(const CellOrder& o, int np, int w, int nw,
                                            unsigned* win) {
  const int lane = threadIdx.x & 31;
  const int per = max(1, min(kOrderPer, np / (32 * nw)));
  const int tile = 32 * per;
  const int tiles = (np - 1) / tile + 1;
  int key[kOrderPer];
  const auto load_keys = [&](int t) {
#pragma unroll
    for (int u = 0; u < kOrderPer; ++u) {
      const int p = t * tile + u * 32 + lane;
      key[u] = t < tiles && u < per && p < np ? o.n.skey[p] : -1;
    }
  };
  if (np <= 0) return;
  load_keys(w);
  for (int t = w; t < tiles; t += nw) {
    const int p0 = t * tile + lane;
    int b[kOrderPer], e[kOrderPer], slot[kOrderPer];
    int lo = 0x7fffffff, hi = 0;  // the cells' positions (crowded ones left out)
#pragma unroll
    for (int u = 0; u < kOrderPer; ++u) {
      b[u] = e[u] = slot[u] = 0;
      if (key[u] >= 0) {
        b[u] = o.start[key[u]];
        e[u] = o.start[key[u] + 1];
        slot[u] = o.n.sslot[p0 + u * 32];
      }
    }
#pragma unroll
    for (int u = 0; u < kOrderPer; ++u) {
      if (e[u] - b[u] > kCrowded) e[u] = b[u];  // order_crowded's
      if (e[u] > b[u]) {
        lo = min(lo, b[u]);
        hi = max(hi, e[u]);
      }
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if (lo < hi)  // (else crowded cells only: lo + lane would overflow)
      for (int i = lo + lane; i < hi; i += 32) win[i - lo] = unsigned(o.n.sidx[i]);
    load_keys(t + nw < tiles ? t + nw : tiles);
    __syncwarp();  // the window is filled
#pragma unroll
    for (int u = 0; u < kOrderPer; ++u) {
      const int n = e[u] - b[u];
      if (n == 0) continue;
      // (unsigned, as the entries of order_crowded compare: a slab's indices may
      // have the top bit set)
      const unsigned mine = win[p0 + u * 32 - lo];
      const unsigned* v = win + (b[u] - lo);
      int rank = 0;
      if constexpr (kRepeats) {  // by index, then by storage slot
        const int* s = o.n.sslot + b[u];
        for (int i = 0; i < n; ++i)
          rank += v[i] < mine || (v[i] == mine && s[i] < slot[u]) ? 1 : 0;
      } else {
#pragma unroll 4
        for (int i = 0; i < n; ++i) rank += v[i] < mine ? 1 : 0;
      }
      o.perm[b[u] + rank] = slot[u];
    }
    __syncwarp();  // the window is free
  }
}

// the 32 values of a warp (one per lane) in ascending order across the lanes
__device__ __forceinline__ unsigned long long warp_bitonic32(unsigned long long v, int lane) {
#pragma unroll
  for (int k = 2; k <= 32; k <<= 1) {
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
      const unsigned long long o = __shfl_xor_sync(0xffffffffu, v, j);
      const bool up = ((lane & k) == 0);
      const bool lower = ((lane & j) == 0);
      // keep the min in the lower lane of an ascending pair
      v = (lower == up) ? min(v, o) : max(v, o);
    }
  }
  return v;
}

// One level of a merge sort along the merge path: src holds sorted runs of w
// entries over [0, len) (the last one shorter), dst receives runs of 2w.
// Each thread writes a contiguous piece of the output: it finds where the
// piece starts in the two runs by a binary search, then merges sequentially
// (again after a search where the piece enters the next pair of runs).
__device__ __forceinline__ void merge_level(const unsigned long long* src,
                                            unsigned long long* dst, int len, int w) {
  const int per = (len + int(blockDim.x) - 1) / int(blockDim.x);
  int k = min(int(threadIdx.x) * per, len);
  const int k1 = min(k + per, len);
  while (k < k1) {
    const int lo = (k / (2 * w)) * (2 * w);
    const int la = min(w, len - lo), lb = max(0, min(w, len - lo - la));
    const unsigned long long* A = src + lo;
    const unsigned long long* B = A + la;
    const int kk = k - lo;
    int i0 = max(0, kk - lb), i1 = min(kk, la);  // output kk takes i of A, kk - i of B
    while (i0 < i1) {
      const int mid = (i0 + i1) >> 1;
      if (A[mid] < B[kk - mid - 1]) i0 = mid + 1; else i1 = mid;
    }
    int i = i0, j = kk - i0;
    const int kend = min(k1, lo + la + lb);
    for (; k < kend; ++k) {
      // i + j < la + lb, so j >= lb leaves i < la
      const bool take_a = j >= lb || (i < la && A[i] < B[j]);
      dst[k] = take_a ? A[i++] : B[j++];
    }
  }
}

// All blocks of the kernel call it, with `sv` = two buffers of kBigRun entries
// in shared memory: zeroes the counts and orders the crowded cells by the
// entries idx << 32 | slot.  Runs of up to kBigRun of them are sorted in
// shared memory -- groups of 32 by a bitonic network in each warp's registers,
// then merged level by level along the merge path between two buffers -- and
// written to pk[b, b+m); longer cells then merge the sorted runs pairwise,
// ping-ponging between pk[b, b+m) and pk[cap + b, cap + b + m): each thread finds where its
// piece of the output starts by a binary search along the merge path, then
// merges the piece sequentially.  The slots go back to perm.
__device__ __forceinline__ void order_crowded(const CellOrder& o, unsigned long long* sv) {
  const int lane = threadIdx.x & 31;
  const int* __restrict__ start = o.start;
  int* __restrict__ perm = o.perm;
  const int nb = o.list_n[0];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < o.n_count; i += gridDim.x * blockDim.x)
    o.count[i] = 0;
  for (int q = blockIdx.x; q < nb; q += gridDim.x) {
    unsigned long long* tmp = o.pk;
    const int c = o.big[q];
    const int b = start[c], m = start[c + 1] - b;
    for (int r0 = 0; r0 < m; r0 += kBigRun) {
      const int len = min(kBigRun, m - r0);
      unsigned long long* A = sv;
      unsigned long long* B = sv + kBigRun;
      // groups of 32 sorted in registers, one warp each, then merged level
      // by level between the two buffers
      const int bw = blockDim.x >> 5;
      for (int g = threadIdx.x >> 5; g * 32 < len; g += bw) {
        const int q = g * 32 + lane;
        const int p = b + r0 + q;
        const unsigned long long v = warp_bitonic32(
            q < len ? ((unsigned long long)(unsigned)o.n.sidx[p] << 32) | (unsigned)o.n.sslot[p]
                    : kNoEntry,
            lane);
        if (q < len) A[q] = v;
      }
      __syncthreads();
      for (int w = 32; w < len; w <<= 1) {
        merge_level(A, B, len, w);
        __syncthreads();
        unsigned long long* t = A;
        A = B;
        B = t;
      }
      for (int i = threadIdx.x; i < len; i += blockDim.x) tmp[b + r0 + i] = A[i];
      __syncthreads();
    }
    unsigned long long* src = tmp + b;
    unsigned long long* dst = tmp + o.cap + b;
    for (int w = kBigRun; w < m; w <<= 1) {
      for (int lo = 0; lo < m; lo += 2 * w) {  // runs [lo, lo+w) and [lo+w, lo+2w)
        const int la = min(w, m - lo), lb = max(0, min(w, m - lo - la));
        const int tot = la + lb;
        const unsigned long long* A = src + lo;
        const unsigned long long* B = A + la;
        const int per = (tot + int(blockDim.x) - 1) / int(blockDim.x);
        const int k0 = min(int(threadIdx.x) * per, tot), k1 = min(k0 + per, tot);
        if (k0 >= k1) continue;
        // output k0 takes i of A and k0 - i of B
        int i0 = max(0, k0 - lb), i1 = min(k0, la);
        while (i0 < i1) {
          const int mid = (i0 + i1) >> 1;
          if (A[mid] < B[k0 - mid - 1]) i0 = mid + 1; else i1 = mid;
        }
        int i = i0, j = k0 - i0;
        for (int k = k0; k < k1; ++k) {
          // i + j == k < tot, so j >= lb leaves i < la
          const bool take_a = j >= lb || (i < la && A[i] < B[j]);
          dst[lo + k] = take_a ? A[i++] : B[j++];
        }
      }
      __syncthreads();
      unsigned long long* t = src;
      src = dst;
      dst = t;
    }
    for (int i = threadIdx.x; i < m; i += blockDim.x) perm[b + i] = int(unsigned(src[i]));
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// P2G + NODAL
//
// Work unit: node rows [r0, r0+kTR) of one strip x node columns [cA, cB); the
// unit walks the cell columns cA-1 .. cB-1.  For cell column cc the particles
// of cells (rlo..rhi, cc) are one contiguous range of the sorted order,
// processed in batches of at most kCap particles.  Each particle's record
// (local coordinates and the nine transferred quantities, built by the
// previous step's G2P) is copied with cp.async into shared memory: the four
// record pairs (xi, eta), (mom_x, mom_y), gravity and friction force with
// one 16-byte copy each, Mp, F11, F12, F22 and Vp with one 8-byte copy each.
// The sorted indices of the next batch are loaded while the copies fly.
// Four CTAs share an SM, so one CTA's copies overlap the others' transfers.
//
// Node row r is served by lane r of four warps, one per quantity group
// (warp-uniform code) g0 {Mv, mom_x, mom_y}, g1 {FPx, FPy, Fric_x, Fric_y},
// g2 {Fint_x}, g3 {Fint_y}; each lane carries two chains per quantity:
//   fin   node (r, cc)   -- local node 1 of cell (r-1,cc), then 0 of (r,cc);
//         it already holds cells (r-1,cc-1), (r,cc-1);
//   start node (r, cc+1) -- local node 3 of cell (r-1,cc), then 2 of (r,cc).
// That is each node's contributions in quadgrid's cell-sweep order, so every
// nodal sum equals the reference's sequential sum bit for bit.  At the end of
// a column the finished sums go through shared memory to warp kNodalWarp,
// which applies the nodal update to node column cc, and each lane's started
// chains become its finishing ones.  Records are stored SoA with an XOR
// swizzle of the low index bits so that lanes of consecutive rows (records
// ~ppc apart) hit distinct banks.
// ---------------------------------------------------------------------------
namespace {

constexpr int kPf = (kCap + kP2GThreads - 1) / kP2GThreads;

// The staged records of one batch: the four record pairs and five single
// values of each particle (13 values of R).
template <class R>
struct P2GSmemT {
  V2<R> pr[4][kCap];  // xe, mp, qg, qf
  R sg[5][kCap];      // Mp, F11, F12, F22, Vp
  R xch[9][kTR];      // finished sums per quantity
  double led[6][kP2GThreads / 32];
  int rowstart[3][kTR + 2];
};
using P2GSmem = P2GSmemT<double>;

// Slot of batch position j: an XOR of the bank-selecting low bits by the
// next ones, so that lanes reading cells 16 records apart hit distinct banks
// (8 sixteen-byte, 16 eight-byte or 32 four-byte slots span the 32 banks).
template <class R>
__device__ __forceinline__ int swz_pair(int j) {
  return sizeof(R) == 8 ? (j ^ ((j >> 4) & 7)) : (j ^ ((j >> 4) & 15));
}
template <class R>
__device__ __forceinline__ int swz_one(int j) {
  return sizeof(R) == 8 ? (j ^ ((j >> 4) & 15)) : (j ^ ((j >> 5) & 31));
}

template <int kBytes>
__device__ __forceinline__ void cp_async(void* dst, const void* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  if (kBytes == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
  else if (kBytes == 8)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}

struct Batch {
  int cc, bb, be;
  bool valid;
};

// the batch after b: the rest of its column, else the start of the next one
template <class R>
__device__ __forceinline__ Batch next_batch(const Batch& b, const P2GSmemT<R>& s,
                                            int nrs, int ccLast) {
  Batch n{0, 0, 0, false};
  if (!b.valid) return n;
  const int seg1 = s.rowstart[b.cc % 3][nrs - 1];
  if (b.be < seg1) return Batch{b.cc, b.be, min(b.be + kCap, seg1), true};
  if (b.cc + 1 > ccLast) return n;
  const int s0 = s.rowstart[(b.cc + 1) % 3][0];
  const int s1 = s.rowstart[(b.cc + 1) % 3][nrs - 1];
  return Batch{b.cc + 1, s0, min(s0 + kCap, s1), true};
}

__device__ __forceinline__ void load_perm(int (&pf)[kPf],
                                          const int* __restrict__ perm,
                                          const Batch& b) {
#pragma unroll
  for (int u = 0; u < kPf; ++u) {
    const int j = b.bb + threadIdx.x + u * kP2GThreads;
    pf[u] = (b.valid && j < b.be) ? perm[j] : 0;
  }
}

template <class R>
__device__ __forceinline__ void issue_gather(P2GSmemT<R>& s, const ParticlesT<R>& p,
                                             const int (&pf)[kPf],
                                             const Batch& b) {
  constexpr int kB = sizeof(R), kB2 = sizeof(V2<R>);
#pragma unroll
  for (int u = 0; u < kPf; ++u) {
    const int j = b.bb + threadIdx.x + u * kP2GThreads;
    if (j >= b.be) break;
    const int i = pf[u];
    const int l2 = swz_pair<R>(j - b.bb), l1 = swz_one<R>(j - b.bb);
    cp_async<kB2>(&s.pr[0][l2], p.xe + i);
    cp_async<kB2>(&s.pr[1][l2], p.mp + i);
    cp_async<kB2>(&s.pr[2][l2], p.qg + i);
    cp_async<kB2>(&s.pr[3][l2], p.qf + i);
    cp_async<kB>(&s.sg[0][l1], p.Mp + i);
    cp_async<kB>(&s.sg[1][l1], p.F11 + i);
    cp_async<kB>(&s.sg[2][l1], p.F12 + i);
    cp_async<kB>(&s.sg[3][l1], p.F22 + i);
    cp_async<kB>(&s.sg[4][l1], p.Vp + i);
  }
  cp_async_commit();
}

// Nodal momentum, velocity and wall conditions of node (r, nc) from its nine
// P2G sums (main/optim_par.cpp:467-529); also accumulates the node ledger.
template <class R>
__device__ __forceinline__ void nodal_update(
    R Mv, R momx, R momy, R FPx, R FPy, R Frx, R Fry, R Fix, R Fiy, int r, int nc,
    const Geom& G, const Phys& P, double dtd, const NodesT<R>& nodes, int record,
    double& ln0, double& ln1, double& ln2) {
  if (nc < G.nc_lo || nc > G.nc_hi) return;  // a slab's neighbour writes this column
  const int nrows = G.nrows, ncols = G.ncols;
  const int n = r + nc * (nrows + 1);
  const R dt = R(dtd);
  const R Fextx = FPx + Frx;
  const R Fexty = FPy + Fry;
  const R Ftx = Fextx - Fix;
  const R Fty = Fexty - Fiy;
  ln0 += Mv;
  ln1 += momx;
  ln2 += momy;
  momx = dt * Ftx + momx;
  momy = dt * Fty + momy;
  const bool act = Mv > R(1.e-2);
  R avx = act ? Ftx / Mv : R(0);
  R avy = act ? Fty / Mv : R(0);
  R vvx = act ? momx / Mv : R(0);
  R vvy = act ? momy / Mv : R(0);
  R vvxL = dt * avx + vvx;
  R vvyL = dt * avy + vvy;
  if (P.BC) {  // cells on the walls zero their 4 nodes (main/optim_par.cpp:503-529)
    if (nc == 0 || nc == 1 || nc == ncols - 1 || nc == ncols) {
      avx = R(0); vvx = R(0); vvxL = R(0); momx = R(0);
    }
    if (r == 0 || r == 1 || r == nrows - 1 || r == nrows) {
      avy = R(0); vvy = R(0); vvyL = R(0); momy = R(0);
    }
  }
  nodes.vvL[n] = V2<R>{vvxL, vvyL};
  if (record) {
    nodes.Mv[n] = Mv;
    nodes.mvx[n] = momx;
    nodes.mvy[n] = momy;
    nodes.avx[n] = avx;
    nodes.avy[n] = avy;
    nodes.vvx[n] = vvx;
    nodes.vvy[n] = vvy;
    nodes.FPxv[n] = FPx;
    nodes.FPyv[n] = FPy;
    nodes.Fricx[n] = Frx;
    nodes.Fricy[n] = Fry;
    nodes.Fintx[n] = Fix;
    nodes.Finty[n] = Fiy;
  }
}

// s += v.  The FP32 chains are compensated (Kahan): c carries the part of
// the running sum that the last rounding lost, so a chain of thousands of
// contributions keeps FP32 precision.  The FP64 chains are the reference's
// plain sums.
template <class R>
__device__ __forceinline__ void acc_add(R& s, R& c, R v) {
  if constexpr (sizeof(R) == 4) {
    const R y = v - c;
    const R t = s + y;
    c = (t - s) - y;
    s = t;
  } else {
    s += v;
  }
}

// a chain's value: the FP32 sum with its carried correction
template <class R>
__device__ __forceinline__ R acc_value(R s, R c) {
  if constexpr (sizeof(R) == 4) return s - c;
  return s;
}

// Running sums of one lane: finishing (f) and starting (s) chains, with
// their compensations (FP32 only).  Quantity groups (one warp each):
//   0: Mv, mom_x, mom_y         1: FPx, FPy, Fric_x, Fric_y
//   2: F_int_x                   3: F_int_y
// about the same FP64 work per particle in each; the lightest (3) also runs
// the nodal update.
constexpr int kMaxQ = 4;
constexpr int kNodalWarp = 3;
template <class R>
struct Chains {
  R f[kMaxQ], fc[kMaxQ], s[kMaxQ], sc[kMaxQ];
};

// One particle's contributions to the chains of quantity group kG: kUpper
// selects the cell (r-1: local nodes 1 (fin) and 3 (start); r: local nodes 0
// and 2).  With fb = eta or (1-eta):
//   fin   N = (1-xi)*fb, Nx = mihx*fb, Ny = (1-xi)*(ihy or mihy)
//   start N = xi*fb,     Nx = ihx*fb,  Ny = xi*(ihy or mihy)
// -- shp/shg of main/gpu_kernels.cpp:33-59 for those local nodes.  kFin off
// runs the started chains alone (a unit's leading column).  Group 0 also
// adds Mp and the momentum to the particle ledger (`led`, once per particle).
template <class R, int kG, bool kFin, bool kUpper>
__device__ __forceinline__ void chain_step(Chains<R>& a, const P2GSmemT<R>& s, int j,
                                           const ShapeT<R>& sh, bool led,
                                           double& lp0, double& lp1, double& lp2) {
  const int l2 = swz_pair<R>(j), l1 = swz_one<R>(j);
  const V2<R> xe = s.pr[0][l2];
  const R xi = xe.x, eta = xe.y;
  const R fa = R(1) - xi;
  const R fb = kUpper ? eta : (R(1) - eta);
  if constexpr (kG == 0 || kG == 1) {
    constexpr int nq = kG == 0 ? 3 : 4;
    const R Nf = fa * fb;
    const R Ns = xi * fb;
    R q[nq];
    if constexpr (kG == 0) {
      const V2<R> m = s.pr[1][l2];
      q[0] = s.sg[0][l1];
      q[1] = m.x;
      q[2] = m.y;
      if (led) {
        lp0 += q[0];
        lp1 += q[1];
        lp2 += q[2];
      }
    } else {
      const V2<R> g = s.pr[2][l2], f = s.pr[3][l2];
      q[0] = g.x;
      q[1] = g.y;
      q[2] = f.x;
      q[3] = f.y;
    }
    if (kFin) {
#pragma unroll
      for (int k = 0; k < nq; ++k) acc_add(a.f[k], a.fc[k], Nf * q[k]);
    }
#pragma unroll
    for (int k = 0; k < nq; ++k) acc_add(a.s[k], a.sc[k], Ns * q[k]);
  } else {
    const R hy = kUpper ? sh.ihy : sh.mihy;
    const R Nxs = sh.ihx * fb, Nys = xi * hy;
    const R f12 = s.sg[2][l1], vp = s.sg[4][l1];
    const R fo = kG == 2 ? s.sg[1][l1] : s.sg[3][l1];  // F11 or F22
    // F_int_x: (Nx*F11 + Ny*F12)*Vp;  F_int_y: (Nx*F12 + Ny*F22)*Vp
    if (kFin) {
      const R Nxf = sh.mihx * fb, Nyf = fa * hy;
      const R v = kG == 2 ? (Nxf * fo + Nyf * f12) : (Nxf * f12 + Nyf * fo);
      acc_add(a.f[0], a.fc[0], v * vp);
    }
    const R v = kG == 2 ? (Nxs * fo + Nys * f12) : (Nxs * f12 + Nys * fo);
    acc_add(a.s[0], a.sc[0], v * vp);
  }
}

// The particles of cells (r-1, cc) and (r, cc) are the adjacent ranges
// [a0, a1) and [a1, b1) of the sorted order, walked in order: the first
// with the upper cell's shape factors, the second with the lower cell's
// (whose particles the lane's own row counts into the particle ledger).
template <class R, int kG, bool kFin, int kUnroll>
__device__ __forceinline__ void chain_range(Chains<R>& a, const P2GSmemT<R>& s, int a0,
                                            int a1, int b1, int bb, int be,
                                            const ShapeT<R>& sh, bool own,
                                            double& lp0, double& lp1, double& lp2) {
  const int u1 = min(a1, be);
  int j = max(a0, bb);
#pragma unroll kUnroll
  for (; j < u1; ++j) chain_step<R, kG, kFin, true>(a, s, j - bb, sh, false, lp0, lp1, lp2);
  const int j1 = min(b1, be);
  const bool led = kG == 0 && own;
  j = max(a1, bb);
#pragma unroll kUnroll
  for (; j < j1; ++j) chain_step<R, kG, kFin, false>(a, s, j - bb, sh, led, lp0, lp1, lp2);
}

template <class R, int kG, int kUnroll>
__device__ __forceinline__ void chain_group(Chains<R>& a, const P2GSmemT<R>& s, bool lead,
                                            int a0, int a1, int b1, int bb, int be,
                                            const ShapeT<R>& sh, bool own, double& lp0,
                                            double& lp1, double& lp2) {
  if (lead)
    chain_range<R, kG, false, kUnroll>(a, s, a0, a1, b1, bb, be, sh, own, lp0, lp1, lp2);
  else
    chain_range<R, kG, true, kUnroll>(a, s, a0, a1, b1, bb, be, sh, own, lp0, lp1, lp2);
}

// ---- a batch inside one crowded cell ---------------------------------------
// When a whole batch lies in one cell (rc, cc), only two lanes of each warp
// have work in it: lane rc+1 (the cell is its cell r-1: local nodes 1 and 3)
// and lane rc (its cell r: local nodes 0 and 2), each walking the batch's
// records one after another for its 2 to 8 chains.  Those chains -- 9
// quantities at each of the 4 nodes, the fin chains only outside a lead
// column -- and the cell's 3 ledger sums go through shared memory to one
// thread each, which walks the records with the operations of chain_step in
// the same order (so every sum is the same, bit for bit), and come back.
// A thread's chains are one kind per warp (warp 0: N * value, warp 1: the
// internal forces, warp 2: the ledger), so a warp's threads run the same
// instructions on different operands.
constexpr int kSoloMin = 32;  // records of a batch worth handing over

// The row of the cell that holds all of [bb, be), or -1, from the lanes'
// ranges of their two cells ([a0, a1): cell r-1, [a1, b1): cell r): every
// warp holds the same ranges, so each finds the same row without a barrier.
__device__ __forceinline__ int solo_row(int a0, int a1, int b1, int bb, int be, int r0) {
  if (be - bb < kSoloMin) return -1;
  const unsigned lo = __ballot_sync(0xffffffffu, b1 > a1 && a1 <= bb && be <= b1);
  if (lo) return r0 + __ffs(lo) - 1;
  const unsigned up = __ballot_sync(0xffffffffu, a1 > a0 && a0 <= bb && be <= a1);
  if (up) return r0 + __ffs(up) - 2;
  return -1;
}

// All threads of the block call it.  rc: the cell's row; chain (role, fs, q)
// sits at X[2 id] with its compensation at X[2 id + 1], id = (2 role + fs) 9 + q,
// role 0 for lane rc+1 and 1 for lane rc, fs 0 for the fin chains, 1 for the
// started ones, q the quantity (0-2 group 0, 3-6 group 1, 7 and 8 groups 2, 3).
template <class R>
__device__ __forceinline__ void solo_batch(Chains<R>& a, P2GSmemT<R>& s, int rc, int r0,
                                           int nrows, int grp, int slot0, int nq, bool lead,
                                           bool own, int n, const ShapeT<R>& sh,
                                           double& lp0, double& lp1, double& lp2) {
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int lup = rc + 1 - r0, llo = rc - r0;
  const bool pup = lup >= 0 && lup < kTR && rc + 1 <= nrows;
  const bool plo = llo >= 0 && llo < kTR && rc <= nrows;
  R* X = &s.xch[0][0];
  const int mine = (pup && lane == lup) ? 0 : ((plo && lane == llo) ? 1 : -1);
  if (mine >= 0) {
#pragma unroll
    for (int k = 0; k < kMaxQ; ++k) {
      if (k < nq) {
        const int idf = (2 * mine) * 9 + slot0 + k, ids = idf + 9;
        X[2 * idf] = a.f[k];
        X[2 * idf + 1] = a.fc[k];
        X[2 * ids] = a.s[k];
        X[2 * ids + 1] = a.sc[k];
      }
    }
    if (grp == 0 && mine == 1) {
      s.led[0][0] = lp0;
      s.led[1][0] = lp1;
      s.led[2][0] = lp2;
    }
  }
  __syncthreads();
  if (w == 0 && lane < 28) {  // Mv, mom_x, mom_y, FPx, FPy, Fric_x, Fric_y
    const int q = lane % 7, rf = lane / 7;
    const int role = rf >> 1, fs = rf & 1;
    if ((role == 0 ? pup : plo) && (fs == 1 || !lead)) {
      const int id = rf * 9 + q;
      R v = X[2 * id], c = X[2 * id + 1];
      const bool single = q == 0;
      const R* pb = reinterpret_cast<const R*>(s.pr[single ? 1 : (q + 1) >> 1]);
      const int half = (q + 1) & 1;
      for (int j = 0; j < n; ++j) {
        const int l2 = swz_pair<R>(j), l1 = swz_one<R>(j);
        const V2<R> xe = s.pr[0][l2];
        const R xi = xe.x, eta = xe.y;
        const R fa = R(1) - xi;
        const R fb = role == 0 ? eta : (R(1) - eta);
        const R N = (fs == 0 ? fa : xi) * fb;
        const R val = single ? s.sg[0][l1] : pb[2 * l2 + half];
        acc_add(v, c, N * val);
      }
      X[2 * id] = v;
      X[2 * id + 1] = c;
    }
  } else if (w == 1 && lane < 8) {  // F_int_x, F_int_y
    const int qb = lane & 1, rf = lane >> 1;
    const int role = rf >> 1, fs = rf & 1;
    if ((role == 0 ? pup : plo) && (fs == 1 || !lead)) {
      const int id = rf * 9 + 7 + qb;
      R v = X[2 * id], c = X[2 * id + 1];
      const R hy = role == 0 ? sh.ihy : sh.mihy;
      const R hxs = fs == 0 ? sh.mihx : sh.ihx;
      const R* P1 = s.sg[qb == 0 ? 1 : 2];  // F11 or F12
      const R* P2 = s.sg[qb == 0 ? 2 : 3];  // F12 or F22
      for (int j = 0; j < n; ++j) {
        const int l2 = swz_pair<R>(j), l1 = swz_one<R>(j);
        const V2<R> xe = s.pr[0][l2];
        const R xi = xe.x, eta = xe.y;
        const R fa = R(1) - xi;
        const R fb = role == 0 ? eta : (R(1) - eta);
        const R Nx = hxs * fb;
        const R Ny = (fs == 0 ? fa : xi) * hy;
        const R vv = Nx * P1[l1] + Ny * P2[l1];
        acc_add(v, c, vv * s.sg[4][l1]);
      }
      X[2 * id] = v;
      X[2 * id + 1] = c;
    }
  } else if (w == 2 && lane < 3) {  // the particle ledger of lane rc (Mp, mom)
    if (plo && own) {
      double lp = s.led[lane][0];
      const R* pb = reinterpret_cast<const R*>(s.pr[1]);
      for (int j = 0; j < n; ++j) {
        const int l2 = swz_pair<R>(j), l1 = swz_one<R>(j);
        lp += lane == 0 ? s.sg[0][l1] : pb[2 * l2 + (lane - 1)];
      }
      s.led[lane][0] = lp;
    }
  }
  __syncthreads();
  if (mine >= 0) {
#pragma unroll
    for (int k = 0; k < kMaxQ; ++k) {
      if (k < nq) {
        const int idf = (2 * mine) * 9 + slot0 + k, ids = idf + 9;
        a.f[k] = X[2 * idf];
        a.fc[k] = X[2 * idf + 1];
        a.s[k] = X[2 * ids];
        a.sc[k] = X[2 * ids + 1];
      }
    }
    if (grp == 0 && mine == 1) {
      lp0 = s.led[0][0];
      lp1 = s.led[1][0];
      lp2 = s.led[2][0];
    }
  }
  __syncthreads();  // the exchange space is free again
}

}  // namespace

// ---- P2G work units -------------------------------------------------------
// A unit is node rows [r0, r0+kTR) of one strip x node columns [cA, cB); it
// walks cell columns cA-1 .. cB-1.  Units are cut per strip so that each
// carries about the same weight -- its particles plus kColWeight per column
// -- whatever the local particle density: P2G takes them from a shared
// cursor, so its time is the average load rather than the heaviest fixed
// block.  The list is in no particular order; the ledger partials of the units
// of a piece sit in order from the slot of its first column on, so the ledger
// reduction order is fixed.
namespace {

__device__ __forceinline__ int column_count(const int* __restrict__ cstart,
                                            int rlo, int rhi, int cc, int nrows) {
  return cstart[rhi + cc * nrows + 1] - cstart[rlo + cc * nrows];
}

}  // namespace

// Cuts node columns [c_lo, c_hi] of strip `strip` of one grid (cstart of that
// grid's cells) into units of weight about T and appends those with particles
// (including the particles of the leading column cA-1, which feed node column
// cA) to P2G's list as make(cA, cB), with the ledger slot slot0 + n of the n-th
// of them; units of more than twice the target weight (a crowded column) go to
// the half of the list that P2G takes first.  Returns the number of units.  Node column nc (< ncols) weighs the particles of cell column
// nc in the strip's cell rows plus col_weight; nc starts a unit where
// floor(exclusive prefix / T) changes.
// One warp cuts a strip (or a piece of one), 32 columns at a time, and needs no barrier: a lane
// whose column starts a unit emits the one that ends there.  The units wait in
// `buf` (kUnitBuf entries of shared memory) and are appended together, so that
// nothing has to wait for all the strips.  With one block per strip, scans over
// the block and a flat list by the last block, this took 8 us at 4096 particles,
// 12 at 4M and 30 for the 800 strips of a batch of 96 scenarios, all of it on the
// way to P2G; by warps it runs beside the ordering (below).
constexpr int kUnitBuf = int(2 * sizeof(unsigned long long) * kBigRun / sizeof(int4)) /
                         (kOrderThreads / 32);

template <class Make>
__device__ __forceinline__ void flush_units(const UnitPlan& u, const int4* buf, int n, int heavies,
                                            int slot, Make make) {
  const int lane = threadIdx.x & 31;
  int at = 0;  // lane 0: the plain units' place, lane 1: the heavy ones'
  if (lane == 0 && n > heavies) at = atomicAdd(u.ucount + kUnitsPlain, n - heavies);
  if (lane == 1 && heavies > 0) at = u.cap + atomicAdd(u.ucount + kUnitsHeavy, heavies);
  __syncwarp();  // the buffer is written
  int plain = __shfl_sync(0xffffffffu, at, 0), heavy = __shfl_sync(0xffffffffu, at, 1);
  for (int i0 = 0; i0 < n; i0 += 32) {
    const int i = i0 + lane;
    int4 e = make_int4(0, 0, 0, 0);
    if (i < n) e = buf[i];
    const unsigned below = (1u << lane) - 1u;
    const unsigned mh = __ballot_sync(0xffffffffu, i < n && e.z);
    const unsigned mp = __ballot_sync(0xffffffffu, i < n && !e.z);
    if (i < n) {
      const int f = e.z ? heavy + __popc(mh & below) : plain + __popc(mp & below);
      u.ulist[f] = make(e.x, e.y);
      u.uslot[f] = slot + i;
    }
    plain += __popc(mp);
    heavy += __popc(mh);
  }
  __syncwarp();  // the buffer is free
}

template <class Make>
__device__ __forceinline__ int plan_columns(const int* __restrict__ cstart, const Geom& G,
                                            long long T, int strip, int4* buf, const UnitPlan& u,
                                            int slot0, int col_weight, int c_lo, int c_hi,
                                            Make make) {
  col_weight = min(col_weight, 1 << 25);
  const int nrows = G.nrows, ncols = G.ncols;
  const int r0 = strip * kTR;
  const int rlo = max(r0 - 1, 0), rhi = min(r0 + kTR - 1, nrows - 1);
  const int lane = threadIdx.x & 31;
  const unsigned T32 = unsigned(T);
  const long long heavy_from = 2 * max(T, (long long)kUnitMinWeight);
  // floor(p / T): in 32 bits where p allows it (T always does)
  const auto part = [&](long long p) {
    return (unsigned long long)p >> 32 ? p / T : (long long)(unsigned(p) / T32);
  };
  const auto column = [&](int nc) {
    return nc <= c_hi && nc < ncols ? column_count(cstart, rlo, rhi, nc, nrows) : 0;
  };
  int J = 0, n = 0, heavies = 0;  // units flushed, in the buffer, heavy ones among them
  const auto emit = [&](bool ends, int cA, int cB, long long p0, long long p1, int prev) {
    const long long np = p1 - p0 - (long long)col_weight * (min(cB, ncols) - cA) + prev;
    const bool keep = ends && np > 0, heavy = np > heavy_from;
    const unsigned m = __ballot_sync(0xffffffffu, keep);
    if (keep) buf[n + __popc(m & ((1u << lane) - 1u))] = make_int4(cA, cB, heavy ? 1 : 0, 0);
    n += __popc(m);
    heavies += __popc(__ballot_sync(0xffffffffu, keep && heavy));
    if (n > kUnitBuf - 32) {
      flush_units(u, buf, n, heavies, slot0 + J, make);
      J += n;
      n = heavies = 0;
    }
  };
  // the open unit: its first column, the prefix there, the column before it
  int oA = c_lo, oV = c_lo > 0 ? column_count(cstart, rlo, rhi, c_lo - 1, nrows) : 0;
  long long oP = 0, carry = 0;
  int last = oV;  // particles of the column before the tile
  // counts of the tiles to come, on the way
  int n0 = column(c_lo + lane), n1 = column(c_lo + 32 + lane), n2 = column(c_lo + 64 + lane);
  long long last_id = 0;  // part() of the column before the tile
  for (int base = c_lo; base <= c_hi; base += 32) {
    const int nc = base + lane;
    const int cnt = n0;
    n0 = n1;
    n1 = n2;
    n2 = column(nc + 96);
    // (32 bits hold a tile: fewer than 2^31 particles and 32 bounded weights)
    const unsigned w = nc <= c_hi && nc < ncols ? unsigned(cnt) + col_weight : 0;
    unsigned incl = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    const long long pex = carry + incl - w;
    int prev = __shfl_up_sync(0xffffffffu, cnt, 1);
    const long long id = part(pex);
    long long id_prev = __shfl_up_sync(0xffffffffu, id, 1);
    if (lane == 0) {
      prev = last;
      id_prev = last_id;
    }
    const bool starts = nc > c_lo && nc <= c_hi && nc < ncols && id != id_prev;
    const unsigned m = __ballot_sync(0xffffffffu, starts);
    if (m) {
      const unsigned below = m & ((1u << lane) - 1u);
      const int src = below ? 31 - __clz(below) : lane;
      const long long sp = __shfl_sync(0xffffffffu, pex, src);
      const int sv = __shfl_sync(0xffffffffu, prev, src);
      emit(starts, below ? base + src : oA, nc, below ? sp : oP, pex, below ? sv : oV);
      const int l = 31 - __clz(m);
      oA = base + l;
      oP = __shfl_sync(0xffffffffu, pex, l);
      oV = __shfl_sync(0xffffffffu, prev, l);
    }
    carry += __shfl_sync(0xffffffffu, incl, 31);
    last = __shfl_sync(0xffffffffu, cnt, 31);
    last_id = __shfl_sync(0xffffffffu, id, 31);
  }
  emit(lane == 0, oA, c_hi + 1, oP, carry, oV);
  if (n > 0) flush_units(u, buf, n, heavies, slot0 + J, make);
  return J + n;
}

__device__ __forceinline__ long long unit_weight(const Scalars* S,
                                                 const UnitPlan& u) {
  const long long T = (long long)S->np / max(u.target_units, 1);
  return T < u.min_weight ? u.min_weight : T;
}

// Piece q of a grid: its strip, its first ledger slot (of the grid's; seg to a
// strip), and its share of node columns [c_lo, c_hi].
__device__ __forceinline__ void piece_of(const Geom& G, int q, int seg, int& strip, int& slot,
                                         int& c_lo, int& c_hi) {
  strip = q;
  slot = q * seg;
  if (G.pieces > 1) {
    strip = q / G.pieces;
    const int k = q - strip * G.pieces, first = k * G.plan_cols;
    slot = strip * seg + first;
    c_lo = max(c_lo, first);
    if (k + 1 < G.pieces) c_hi = min(c_hi, first + G.plan_cols - 1);
  }
}

// Who plans and who orders: the first plan_blocks() blocks plan, four warps each,
// and the others order -- beside the ordering's busy warps a planning warp got an
// eighth of its scheduler's issue slots and was the last to finish (a step of the
// 4096-particle dam break 0.6 us longer, of 4M particles 4).  Where that would take
// more than one block in kPlanShare (a batch of many scenarios, or a grid of few
// blocks) the pieces are spread over the blocks, warp 0 of each, then warp 1 ...,
// and the other warps order (everyone where that leaves fewer than half): 12.5 us
// against 15 with the 800 strips of 96 scenarios.
constexpr int kPlanShare = 4;
__device__ __forceinline__ int plan_blocks(int pieces) {
  const int nb = (pieces + 3) / 4;
  return nb <= int(gridDim.x) / kPlanShare ? nb : 0;
}
// this warp's first piece and the step to its next one
__device__ __forceinline__ int2 plan_share(int pieces) {
  const int nb = plan_blocks(pieces), w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int over = nb ? nb : gridDim.x;
  return make_int2(int(blockIdx.x) < over ? w * over + int(blockIdx.x) : pieces, over * nw);
}
template <bool kRepeats>
__device__ __forceinline__ void order_share(const CellOrder& o, int np, int pieces,
                                            unsigned long long* sv) {
  static_assert(kOrderWin * sizeof(unsigned) <= kUnitBuf * sizeof(int4), "");
  unsigned* win =
      reinterpret_cast<unsigned*>(reinterpret_cast<int4*>(sv) + (threadIdx.x >> 5) * kUnitBuf);
  const int nb = plan_blocks(pieces), w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  int first, all;  // this warp's place among those that order
  if (nb > 0) {
    first = (int(blockIdx.x) - nb) * nw + w;
    all = (int(gridDim.x) - nb) * nw;
  } else {
    all = int(gridDim.x) * nw;
    const int planners = 2 * pieces <= all ? pieces : 0;
    first = w * int(gridDim.x) + int(blockIdx.x) - planners;
    all -= planners;
  }
  if (first >= 0) order_cells<kRepeats>(o, np, first, all, win);
}
__device__ __forceinline__ int4* unit_buf(unsigned long long* sv) {
  return reinterpret_cast<int4*>(sv) + (threadIdx.x >> 5) * kUnitBuf;
}

// The last kernel of a sort: P2G's work list, which needs the cell starts only,
// and the order inside the cells.  The last block to finish ends the step before
// and begins this one unless it has begun (a merge/split came before the sort):
// no block still reads the loop condition then.
// The planner and the order of the smaller and of the larger cells were launches
// of their own: 46 us in all at 4M particles, 20 at 0.25M, 13 at 4096 and 53 in a
// batch of 96 scenarios; together 36, 11.5, 6 and 12.5.
// The begin sits here and not at the end of G2P, where every block would have
// to wait for its stores before it counts itself done (7 us at 0.25M and 4M
// particles).
// pieces: of all strips; 0: the sort alone (before a merge/split); seg: unit slots
// per strip
template <bool kRepeats>
__global__ void __launch_bounds__(kOrderThreads, 1)
    k_order_units(CellOrder o, UnitPlan u, Geom G, Phys P, Scalars* S, int pieces, int seg,
                  Gate gate) {
  if (!gate_open(S, gate)) {
    if (!gate.begun && blockIdx.x == 0 && threadIdx.x == 0) S->active = 0;
    return;
  }
  extern __shared__ unsigned long long sv[];
  // node columns of the cells the particles are binned to (the key range the
  // scatter just rolled over), plus the column right of them
  const int L = S->krange[0], K = S->krange[1];
  const int2 share = plan_share(pieces);
  for (int q = share.x; q < pieces; q += share.y) {
    int strip, slot, c_lo = L / G.nrows, c_hi = min(K / G.nrows + 1, G.ncols);
    piece_of(G, q, seg, strip, slot, c_lo, c_hi);
    if (L <= K && c_lo <= c_hi) {
      const int n = plan_columns(o.start, G, unit_weight(S, u), strip, unit_buf(sv), u, slot,
                                 kColWeight, c_lo, c_hi,
                                 [&](int cA, int cB) { return make_int4(strip, cA, cB, 0); });
      if ((threadIdx.x & 31) == 0) u.piece_n[q] = n;
    } else if ((threadIdx.x & 31) == 0) {
      u.piece_n[q] = 0;
    }
  }
  order_share<kRepeats>(o, S->np, pieces, sv);
  __syncthreads();  // the shared memory is free again
  order_crowded(o, sv);
  if (!last_block(u.ucount + kOrderDone, gridDim.x)) return;
  if (threadIdx.x == 0) {
    *o.list_n = 0;
    if (!gate.begun) step_begin_one(S, G, P);
  }
}

// kUnroll: chain steps per loop trip.  Two in the single-scenario kernel (4M
// particles: 1 % faster than one).  One in a batch: its units are a few short
// columns, so the four warps' loops keep leaving and entering the instruction
// cache (at two, 1.9 cycles of every issue wait for an instruction; this kernel
// takes 138 us with 96 scenarios at two, 118 at one, 234 at four; in FP32 129, 97
// and 269).
template <class R, int kUnroll>
__device__ __forceinline__ void p2g_unit(
    const ParticlesT<R>& p, const int* __restrict__ perm,
    const int* __restrict__ cstart, const NodesT<R>& nodes,
    double* __restrict__ led_part, const Geom& G, const Phys& P,
    const Scalars* S, int record, P2GSmemT<R>& s, int slot, int4 unit) {
  const int nrows = G.nrows, ncols = G.ncols;
  const int r0 = unit.x * kTR;
  const int cA = unit.y;
  const int cB = unit.z;
  const int rlo = max(r0 - 1, 0);
  const int rhi = min(r0 + kTR - 1, nrows - 1);
  const int ccFirst = max(cA - 1, 0);
  const int ccLast = min(cB - 1, ncols - 1);
  const int nrs = rhi - rlo + 2;  // row starts per column
  const int tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31;
  const int grp = warp;  // quantity group (warp-uniform)
  const int row = lane;
  const int r = r0 + row;
  const bool lane_ok = row < kTR;  // lanes kTR..31 idle
  const bool row_ok = lane_ok && (r <= nrows);
  const double dt = S->dt;
  const ShapeT<R> sh = shape_of<R>(G);
  // exchange slots of each group's quantities: g0 0-2, g1 3-6, g2 7, g3 8
  const int slot0 = grp == 0 ? 0 : grp == 1 ? 3 : grp == 2 ? 7 : 8;
  const int nq = grp == 0 ? 3 : grp == 1 ? 4 : 1;
  const bool last_unit_col = (cB == ncols + 1);  // this unit closes node column ncols

  double lp0 = 0, lp1 = 0, lp2 = 0, ln0 = 0, ln1 = 0, ln2 = 0;
  Chains<R> a;
#pragma unroll
  for (int q = 0; q < kMaxQ; ++q) a.f[q] = a.fc[q] = a.s[q] = a.sc[q] = R(0);

  // prologue: row starts of the first two columns, sorted indices of batch 0
  for (int q = tid; q < 2 * nrs; q += kP2GThreads) {
    const int k = q / nrs, rr = q - k * nrs;
    const int cc = ccFirst + k;
    if (cc <= ccLast) s.rowstart[cc % 3][rr] = cstart[rlo + rr + cc * nrows];
  }
  __syncthreads();
  int pf[kPf];
  Batch cur;
  cur.cc = ccFirst;
  cur.bb = s.rowstart[ccFirst % 3][0];
  cur.be = min(cur.bb + kCap, s.rowstart[ccFirst % 3][nrs - 1]);
  cur.valid = true;
  load_perm(pf, perm, cur);
  int a0 = 0, a1 = 0, b1 = 0;  // my rows' ranges in the current column

  while (true) {
    issue_gather(s, p, pf, cur);
    // while the copies fly: this batch's bookkeeping and the next batch's
    // sorted indices
    const int* RS = s.rowstart[cur.cc % 3];
    const bool first_of_col = (cur.bb == RS[0]);
    const bool last_of_col = (cur.be == RS[nrs - 1]);
    int rs2 = 0;
    const bool has_rs2 = last_of_col && cur.cc + 2 <= ccLast && tid < nrs;
    if (has_rs2) rs2 = cstart[rlo + tid + (cur.cc + 2) * nrows];
    if (first_of_col) {
      // cell r-1: [a0, a1), cell r: [a1, b1) (empty where the cell is absent)
      a0 = a1 = b1 = 0;
      if (row_ok && r >= rlo && r <= rhi + 1) {
        const int k = r - rlo;  // row start of cell r (= end of cell r-1)
        a1 = RS[k];
        a0 = (r - 1 >= rlo) ? RS[k - 1] : a1;
        b1 = (r <= rhi) ? RS[k + 1] : a1;
      }
    }
    const Batch nxt = next_batch(cur, s, nrs, ccLast);
    load_perm(pf, perm, nxt);
    cp_async_wait_all();
    __syncthreads();  // batch `cur` is in shared memory
    const bool own = r >= r0 && r < r0 + kTR && cur.cc >= cA && cur.cc >= G.pc_lo &&
                     cur.cc < G.pc_hi;
    const bool lead = cur.cc < cA;  // started chains only
    const int rc = solo_row(a0, a1, b1, cur.bb, cur.be, r0);  // the same in every warp
    if (rc >= 0) {
      // own as the cell's lower lane sees it (its row lies in the unit)
      const bool own_c = cur.cc >= cA && cur.cc >= G.pc_lo && cur.cc < G.pc_hi;
      solo_batch<R>(a, s, rc, r0, nrows, grp, slot0, nq, lead, own_c, cur.be - cur.bb, sh,
                    lp0, lp1, lp2);
    } else {
      switch (grp) {
        case 0:
          chain_group<R, 0, kUnroll>(a, s, lead, a0, a1, b1, cur.bb, cur.be, sh, own, lp0, lp1, lp2);
          break;
        case 1:
          chain_group<R, 1, kUnroll>(a, s, lead, a0, a1, b1, cur.bb, cur.be, sh, own, lp0, lp1, lp2);
          break;
        case 2:
          chain_group<R, 2, kUnroll>(a, s, lead, a0, a1, b1, cur.bb, cur.be, sh, own, lp0, lp1, lp2);
          break;
        default:
          chain_group<R, 3, kUnroll>(a, s, lead, a0, a1, b1, cur.bb, cur.be, sh, own, lp0, lp1, lp2);
          break;
      }
    }
    if (last_of_col) {
      if (lane_ok)
        for (int q = 0; q < nq; ++q) s.xch[slot0 + q][row] = acc_value(a.f[q], a.fc[q]);
      if (has_rs2) s.rowstart[(cur.cc + 2) % 3][tid] = rs2;
    }
    __syncthreads();  // shared records free; finished sums exchanged
    if (last_of_col) {
      // ---- nodal update of node column cc ------------------------------
      if (warp == kNodalWarp && row_ok && cur.cc >= cA) {
        const R (*X)[kTR] = s.xch;
        nodal_update<R>(X[0][row], X[1][row], X[2][row], X[3][row], X[4][row],
                        X[5][row], X[6][row], X[7][row], X[8][row], r, cur.cc, G, P,
                        dt, nodes, record, ln0, ln1, ln2);
      }
      if (cur.cc == ncols - 1 && last_unit_col) {
        // node column ncols: its chains end with this column
        __syncthreads();  // warp 0 is done reading the exchange
        if (lane_ok)
          for (int q = 0; q < nq; ++q) s.xch[slot0 + q][row] = acc_value(a.s[q], a.sc[q]);
        __syncthreads();
        if (warp == kNodalWarp && row_ok) {
          const R (*X)[kTR] = s.xch;
          nodal_update<R>(X[0][row], X[1][row], X[2][row], X[3][row], X[4][row],
                          X[5][row], X[6][row], X[7][row], X[8][row], r, ncols, G, P,
                          dt, nodes, record, ln0, ln1, ln2);
        }
      }
#pragma unroll
      for (int q = 0; q < kMaxQ; ++q) {
        a.f[q] = a.s[q];
        a.fc[q] = a.sc[q];
        a.s[q] = R(0);
        a.sc[q] = R(0);
      }
    }
    if (!nxt.valid) break;
    cur = nxt;
  }
  // ---- ledger partials: fixed-order block reduction ----------------------
  {
    double v[6] = {lp0, lp1, lp2, ln0, ln1, ln2};
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      double x = v[q];
      for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
      if (lane == 0) s.led[q][warp] = x;
    }
    __syncthreads();
    if (tid < 6) {
      double x = 0.0;
      for (int w = 0; w < kP2GThreads / 32; ++w) x += s.led[tid][w];
      led_part[(size_t)slot * 6 + tid] = x;
    }
    __syncthreads();
  }
}

// kRecord: the nodal output fields are written (compiled out of the plain
// step)
template <bool kRecord>
__global__ void __launch_bounds__(kP2GThreads, kP2GMinBlocks)
    k_p2g(Particles p, const int* __restrict__ perm,
          const int* __restrict__ cstart, Nodes nodes,
          double* __restrict__ led_part, Geom G, Phys P, const Scalars* S, UnitPlan u) {
  constexpr int record = kRecord ? 1 : 0;
  if (!S->active) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  P2GSmem& s = *reinterpret_cast<P2GSmem*>(smem_raw);
  const int nheavy = u.ucount[kUnitsHeavy], nunits = nheavy + u.ucount[kUnitsPlain];
  __shared__ int next_unit;
  while (true) {
    // units are taken from a shared cursor, the heavy ones first: CTAs that
    // drew light units take more (the per-SM load stays even)
    if (threadIdx.x == 0) next_unit = atomicAdd(u.ucount + kUnitCursor, 1);
    __syncthreads();
    const int k = next_unit;
    __syncthreads();
    if (k >= nunits) break;
    const int f = k < nheavy ? u.cap + k : k - nheavy;
    p2g_unit<double, kChainUnroll>(p, perm, cstart, nodes, led_part, G, P, S, record, s,
                                   u.uslot[f], u.ulist[f]);
  }
}

size_t order_smem_bytes() { return 2 * sizeof(unsigned long long) * kBigRun; }

int setup_sort() {
  for (const void* f : {(const void*)k_order_units<false>, (const void*)k_order_units<true>,
                        (const void*)k_b_order_units})
    if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             int(order_smem_bytes())) != cudaSuccess)
      return 0;
  return cudaFuncSetAttribute(k_scan_scatter, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              int(sizeof(int)) * kSmallCells) == cudaSuccess;
}

void launch_order_units(int grid, cudaStream_t st, const CellOrder& o, const UnitPlan& u, Geom G,
                        Phys P, Scalars* S, int pieces, int seg, Gate gate, bool repeats) {
  auto* kernel = repeats ? k_order_units<true> : k_order_units<false>;
  kernel<<<grid, kOrderThreads, order_smem_bytes(), st>>>(o, u, G, P, S, pieces, seg, gate);
}

int setup_p2g() {
  const size_t smem = p2g_smem_bytes();
  for (const void* f : {(const void*)k_p2g<false>, (const void*)k_p2g<true>}) {
    if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) !=
        cudaSuccess)
      return 0;
    cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout,
                         int(cudaSharedmemCarveoutMaxShared));
  }
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_p2g<false>, kP2GThreads, smem);
  return per_sm < 1 ? 1 : per_sm;
}

void launch_p2g(int grid, cudaStream_t st, Particles p, const int* perm, const int* cstart,
                Nodes nodes, double* led_part, Geom G, Phys P, const Scalars* S, int record,
                const UnitPlan& u) {
  if (record)
    k_p2g<true><<<grid, kP2GThreads, p2g_smem_bytes(), st>>>(p, perm, cstart, nodes, led_part,
                                                             G, P, S, u);
  else
    k_p2g<false><<<grid, kP2GThreads, p2g_smem_bytes(), st>>>(p, perm, cstart, nodes, led_part,
                                                              G, P, S, u);
}

// Block reduction, in a fixed order, of the threads' ledger sums into S->ledger,
// and the conservation errors.
__device__ __forceinline__ void ledger_close(const double (&v)[6], Scalars* S) {
  __shared__ double sm[6][32];
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    double x = v[q];
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if ((threadIdx.x & 31) == 0) sm[q][threadIdx.x >> 5] = x;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double t[6];
    for (int q = 0; q < 6; ++q) {
      t[q] = 0.0;
      for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t[q] += sm[q][w];
      S->ledger[q] = t[q];
    }
    // main/optim_par.cpp:416-425
    const double err_mass = fabs(t[0] - t[3]) / t[0];
    const double a = fabs(t[1]), b = fabs(t[2]);
    const double m = (a < b) ? b : a;
    const double norm_mom = (1.0 < m) ? m : 1.0;
    const double ex = fabs(t[1] - t[4]) / norm_mom;
    const double ey = fabs(t[2] - t[5]) / norm_mom;
    S->ledger[6] = err_mass;
    S->ledger[7] = (ex < ey) ? ey : ex;
    S->ledger[8] = S->t;
  }
}

// The ledger of a grid from the partials of its units: piece_n[q] of them for
// piece q, `per` pieces of `cols` columns to a strip, whose slots lie at its first
// column among its strip's seg.  One warp takes a piece, its lanes the units.
// (Not inlined: inside G2P its loops changed what the compiler spills there, 200
// against 214 us at 4M particles.)
__device__ __noinline__ void ledger_reduce(const double* __restrict__ led_part,
                                           const int* __restrict__ piece_n, int pieces, int per,
                                           int cols, int seg, Scalars* S) {
  double v[6] = {0, 0, 0, 0, 0, 0};
  for (int b = threadIdx.x >> 5; b < pieces; b += blockDim.x >> 5) {
    const int strip = per == 1 ? b : b / per;
    const int slot0 = strip * seg + (b - strip * per) * cols;
    const double* part = led_part + (size_t)slot0 * 6;
    const int n = piece_n[b];
    for (int f = threadIdx.x & 31; f < n; f += 32)
#pragma unroll
      for (int q = 0; q < 6; ++q) v[q] += part[(size_t)f * 6 + q];
  }
  ledger_close(v, S);
}

// The same for many pieces of few units: a warp takes 32 pieces at a time, lane by
// lane, sums up their counts, and its lanes take the units of all of them side by
// side.  (In place of ledger_reduce it costs G2P 1 % at 4M particles, in registers.)
__device__ __forceinline__ void ledger_reduce_many(const double* __restrict__ led_part,
                                                   const int* __restrict__ piece_n, int pieces,
                                                   int per, int cols, int seg, Scalars* S) {
  double v[6] = {0, 0, 0, 0, 0, 0};
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int b0 = threadIdx.x >> 5; b0 < pieces; b0 += 32 * nw) {
    const int b = b0 + lane * nw, strip = per == 1 ? b : b / per;
    const int n = b < pieces ? piece_n[b] : 0;
    int upto = n;  // units of this piece and those before it
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += t;
    }
    const int slot = strip * seg + (b - strip * per) * cols - (upto - n);
    const int units = __shfl_sync(0xffffffffu, upto, 31);
#pragma unroll 2
    for (int f0 = 0; f0 < units; f0 += 32) {
      const int f = min(f0 + lane, units - 1);
      int q = 0;  // the unit's piece: as many end at f or before
#pragma unroll
      for (int step = 16; step > 0; step >>= 1)
        if (__shfl_sync(0xffffffffu, upto, q + step - 1) <= f) q += step;
      const int at = __shfl_sync(0xffffffffu, slot, q) + f;
      if (f0 + lane < units) {
        const double2* part = reinterpret_cast<const double2*>(led_part) + 3 * (size_t)at;
        const double2 a = part[0], c = part[1], d = part[2];
        v[0] += a.x;
        v[1] += a.y;
        v[2] += c.x;
        v[3] += c.y;
        v[4] += d.x;
        v[5] += d.y;
      }
    }
  }
  ledger_close(v, S);
}

// log: a ring of kLedgerLog rows {t, err_mass, err_mom}, row (it-1) % kLedgerLog
__device__ __forceinline__ void ledger_log(const Scalars* S, double* __restrict__ log) {
  if (threadIdx.x == 0 && log) {
    double* row = log + 3 * ((S->it - 1) % kLedgerLog);
    row[0] = S->ledger[8];
    row[1] = S->ledger[6];
    row[2] = S->ledger[7];
  }
}

// The ledger as a launch of its own, after G2P (which was given no pieces): see
// ledger_apart.
__global__ void __launch_bounds__(kLedgerThreads)
    k_ledger(const double* __restrict__ led_part, const int* __restrict__ piece_n, int pieces,
             int seg, Geom G, Scalars* S, double* __restrict__ log) {
  if (!S->active) return;
  ledger_reduce_many(led_part, piece_n, pieces, G.pieces, G.plan_cols, seg, S);
  ledger_log(S, log);
}

// ---------------------------------------------------------------------------
// G2P: velocity, advection, velocity gradients at the new position with the
// cell of the step start, height update, Bingham stress, next cell key and
// the CFL max-reductions (main/optim_par.cpp:532-651).
// ---------------------------------------------------------------------------
// The step-start values G2P reads of a particle.
template <class R>
struct G2PIn {
  R x, y, hp, H, Mp, Vp;
  int idx;
};
template <class R>
__device__ __forceinline__ G2PIn<R> g2p_in(const ParticlesT<R>& src, int s) {
  return G2PIn<R>{src.x[s], src.y[s], src.hp[s], src.H[s], src.Mp[s], src.Vp[s], src.idx[s]};
}

// One particle of G2P (the body of k_g2p and of the batched G2P): the
// particle in slot `s` of the step-start buffer `src` -- its values `in` --
// binned to cell `key`, written to slot `j` of `dst` (its position in this
// step's sorted order).  key_off is the scenario's first cell in a batch (its
// cell keys are offset by it); the new key is returned in `nkey`.
template <class R>
__device__ __forceinline__ void g2p_particle(
    const ParticlesT<R>& src, int s, const G2PIn<R>& in, int key_in,
    const ParticlesT<R>& dst, int j,
    const NodesT<R>& nodes, const double* __restrict__ Z, const Geom& G, const Phys& P,
    const ShapeT<R>& sh, double dtd, int record, int want_grad, int key_off,
    unsigned long long& m0, unsigned long long& m1, unsigned long long& m2, int& nkey) {
  const int nrows = G.nrows;
  const R ihx = sh.ihx, mihx = sh.mihx;
  const R ihy = sh.ihy, mihy = sh.mihy;
  const R eps = R(1e-10);
  const R dt = R(dtd);
  const int key = key_in - key_off;
  const int c = column_of(key, G), r = key - c * nrows;
  int nd[4];
  R vxn[4], vyn[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    nd[k] = node_of(k, c, r, nrows);
    const V2<R> v = nodes.vvL[nd[k]];
    vxn[k] = v.x;
    vyn[k] = v.y;
  }
  R x = in.x, y = in.y;
  R xi, eta;
  local_xy_g(x, y, c, r, G, ihx, ihy, xi, eta);
  R vxL = R(0), vyL = R(0);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const R N = shp(xi, eta, k);
    vxL += N * vxn[k];
    vyL += N * vyn[k];
  }
  if (record) {
    // this step's intermediates as the reference's dprops hold them after
    // the step (main/optim_par.cpp:387-459,542): apx/apy, grad Z and the
    // gravity and friction forces of this step's P2G
    R ax = R(0), ay = R(0);
    double dzx = 0.0, dzy = 0.0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const R N = shp(xi, eta, k);
      ax += N * nodes.avx[nd[k]];
      ay += N * nodes.avy[nd[k]];
      const double zn = Z[nd[k]];
      dzx += double(shg_x(eta, k, ihx, mihx)) * zn;
      dzy += double(shg_y(xi, k, ihy, mihy)) * zn;
    }
    dst.apx[j] = ax;
    dst.apy[j] = ay;
    dst.dZxp[j] = R(dzx);
    dst.dZyp[j] = R(dzy);
    const V2<R> qg = src.qg[s], qf = src.qf[s];
    dst.Fpx[j] = qg.x;
    dst.Fpy[j] = qg.y;
    dst.Frx[j] = qf.x;
    dst.Fry[j] = qf.y;
  }
  const R vpx = vxL, vpy = vyL;
  x = x + dt * vpx;
  y = y + dt * vpy;
  if (x < eps) x = eps;
  if (x > R(G.Lx) - eps) x = R(G.Lx) - eps;
  if (y < eps) y = eps;
  if (y > R(G.Ly) - eps) y = R(G.Ly) - eps;
  // g2pd {vvxL, vvyL} at the new position, old cell (main/optim_par.cpp:578)
  local_xy_g(x, y, c, r, G, ihx, ihy, xi, eta);
  R vxdx = R(0), vydx = R(0), vxdy = R(0), vydy = R(0);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const R Nx = shg_x(eta, k, ihx, mihx);
    const R Ny = shg_y(xi, k, ihy, mihy);
    vxdx += Nx * vxn[k];
    vxdy += Ny * vxn[k];
    vydx += Nx * vyn[k];
    vydy += Ny * vyn[k];
  }
  // height from the strain rate (main/optim_par.cpp:595-599)
  const R div = vxdx + vydy;
  R hp = in.hp;
  hp = hp / (R(1) + dt * div);
  hp = hp < R(1e-2) ? R(1e-2) : hp;
  R F11, F12, F22;
  const R H = in.H;
  const R Mp = in.Mp, Vp = in.Vp;
  rheology_stress(P, vpx, vpy, hp, H, vxdx, vydy, vxdy, vydx, F11, F12, F22);
  dst.x[j] = x;
  dst.y[j] = y;
  dst.vpx[j] = vpx;
  dst.vpy[j] = vpy;
  dst.hp[j] = hp;
  dst.F11[j] = F11;
  dst.F12[j] = F12;
  dst.F22[j] = F22;
  dst.Mp[j] = Mp;
  dst.Vp[j] = Vp;
  dst.H[j] = H;
  dst.idx[j] = in.idx;
  const int nr = cell_row(double(y), G), ncl = cell_col(double(x), G);
  nkey = nr + ncl * nrows + key_off;
  dst.key[j] = nkey;
  if (want_grad) {
    dst.vpx_dx[j] = vxdx;
    dst.vpx_dy[j] = vxdy;
    dst.vpy_dx[j] = vydx;
    dst.vpy_dy[j] = vydy;
  }
  // the record of the next P2G: what the reference stores at the end of
  // the step (main/optim_par.cpp:600-626: momentum, Ap, basal friction) and
  // the local coordinates and gravity force in the cell of the next
  // binning (:387,447-454)
  {
    dst.mp[j] = V2<R>{vpx * Mp, vpy * Mp};
    const R Ap = hp > R(1.e-2) ? Vp / hp : R(0);
    R fbx, fby;
    rheology_friction(P, vpx, vpy, hp, fbx, fby);
    dst.qf[j] = V2<R>{Ap * fbx, Ap * fby};
    R qxi, qeta, qgx, qgy;
    next_record(G, P, Z, x, y, hp, H, Vp, qxi, qeta, qgx, qgy);
    dst.xe[j] = V2<R>{qxi, qeta};
    dst.qg[j] = V2<R>{qgx, qgy};
  }
  if (record) {
    // g2p Z -> Zp at the new position, old cell (main/optim_par.cpp:642)
    double zp = 0.0;
#pragma unroll
    for (int k = 0; k < 4; ++k) zp += double(shp(xi, eta, k)) * Z[nd[k]];
    dst.Zp[j] = R(zp);
    dst.hpZ[j] = R(double(hp) + zp);
  }
  // bits of non-negative values: ordered as they are; a value that is not
  // finite is above all others
  m0 = max(m0, (unsigned long long)__double_as_longlong(fabs(double(vpx))));
  m1 = max(m1, (unsigned long long)__double_as_longlong(fabs(double(vpy))));
  m2 = max(m2, (unsigned long long)__double_as_longlong(double(hp)));
}

// Copies the moving fields of slot s of src to slot j of dst (a particle
// that does not step in this pass, or the reordering into reference order).
template <class R>
__device__ __forceinline__ void copy_moving(const ParticlesT<R>& src, int s,
                                            const ParticlesT<R>& dst, int j) {
  dst.x[j] = src.x[s];
  dst.y[j] = src.y[s];
  dst.vpx[j] = src.vpx[s];
  dst.vpy[j] = src.vpy[s];
  dst.hp[j] = src.hp[s];
  dst.F11[j] = src.F11[s];
  dst.F12[j] = src.F12[s];
  dst.F22[j] = src.F22[s];
  dst.Mp[j] = src.Mp[s];
  dst.Vp[j] = src.Vp[s];
  dst.H[j] = src.H[s];
  dst.key[j] = src.key[s];
  dst.idx[j] = src.idx[s];
  dst.slot[j] = src.slot[s];
  dst.mp[j] = src.mp[s];
  dst.qf[j] = src.qf[s];
  dst.xe[j] = src.xe[s];
  dst.qg[j] = src.qg[s];
  if (src.vpx_dx) {
    dst.vpx_dx[j] = src.vpx_dx[s];
    dst.vpx_dy[j] = src.vpx_dy[s];
    dst.vpy_dx[j] = src.vpy_dx[s];
    dst.vpy_dy[j] = src.vpy_dy[s];
  }
}

// Raises kStatusNonFinite in S when any thread of the block saw a diverged
// particle (all threads of the block call it).
__device__ __forceinline__ void flag_non_finite(int bad, Scalars* S) {
  if (__syncthreads_or(bad) && threadIdx.x == 0) atomicOr(&S->status, kStatusNonFinite);
}

// Block min/max of the new keys into knext (the scan range of the next
// sort); all threads of the block call it.
__device__ __forceinline__ void key_range(int kmin, int kmax, int* sred, Scalars* S) {
  kmin = __reduce_min_sync(0xffffffffu, kmin);
  kmax = __reduce_max_sync(0xffffffffu, kmax);
  if ((threadIdx.x & 31) == 0) {
    atomicMin(&sred[0], kmin);
    atomicMax(&sred[1], kmax);
  }
  __syncthreads();
  if (threadIdx.x == 0 && sred[1] >= 0) {
    atomicMin(&S->knext[0], sred[0]);
    atomicMax(&S->knext[1], sred[1]);
  }
}

// The maximum over a warp, half by half with the warp's integer reduction (six
// of them for the three maxima; 64-bit shuffles took about a hundred
// instructions, a tenth of what a particle takes).
__device__ __forceinline__ unsigned long long warp_max(unsigned long long k) {
  const unsigned hi = unsigned(k >> 32);
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? unsigned(k) : 0u);
  return ((unsigned long long)mh << 32) | ml;
}

// A thread's maxima (bits of |vpx|, |vpy|, hp) tell whether one of its particles
// diverged: a velocity or a depth that is not finite is the maximum, a depth is
// at least 1e-2 or no number, and a position is not finite only where the
// velocity is not either (it is clamped to the domain).
__device__ __forceinline__ bool diverged(unsigned long long m0, unsigned long long m1,
                                         unsigned long long m2) {
  return max(m0, max(m1, m2)) >= 0x7ff0000000000000ull;
}
constexpr unsigned long long kKeySign = 0x8000000000000000ull;  // ordered_key of a value >= 0

// Block reduction of the CFL maxima into one scenario's next-step slots.
__device__ __forceinline__ void cfl_block_max(unsigned long long m0,
                                              unsigned long long m1,
                                              unsigned long long m2,
                                              unsigned long long* red,
                                              Scalars* S) {
  m0 = warp_max(m0);
  m1 = warp_max(m1);
  m2 = warp_max(m2);
  if ((threadIdx.x & 31) == 0) {
    atomicMax(&red[0], m0);
    atomicMax(&red[1], m1);
    atomicMax(&red[2], m2);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    atomicMax(&S->red_next[0], red[0] | kKeySign);
    atomicMax(&S->red_next[1], red[1] | kKeySign);
    atomicMax(&S->red_next[2], red[2] | kKeySign);
  }
}

// Bound by latency and issue together (32 warps per SM at 64 registers): what
// takes instructions or registers out of a particle's 900 counts, more loads in
// flight at the price of either do not (the count's atomic sent early and the next
// particle's position read ahead: 5 % slower; three blocks per SM without spills:
// 5 %; five: 3 %).  The maxima kept as bits, which also tell a diverged particle,
// their reduction by halves, 1/h from the constant bank, the cell's column by a
// product and the cell by a conversion: 210 -> 196 us at 4M particles (4.6 TB/s
// on its 900 MB), 22.4 -> 18 at 0.25M.
//
// kRecord / kGrad: the output fields and the velocity gradients are
// written (compiled out of the plain step).  Thread t takes the particle
// at position ng + t of this step's sorted order: slot perm[ng + t] of
// `cur`, written to slot t of `nxt`.  ng = 0 outside slab mode; in slab
// mode the first ng positions are the copies of the neighbour's last column
// (they sort first), which only P2G reads, and a particle whose new cell
// lies outside the slab's columns is listed in `leave` (and not counted:
// it moves to the neighbour).  A pass whose loop condition failed copies
// `cur` to `nxt` unchanged (the host exchanges the buffers after every
// pass).
template <bool kRecord, bool kGrad>
__global__ void __launch_bounds__(kG2PThreads, kG2PMinBlocks)
    k_g2p_t(Particles cur, Particles nxt, const int* __restrict__ perm,
            const int* __restrict__ skey, Nodes nodes, const double* __restrict__ Z, Geom G,
            Phys P, Scalars* S, int* __restrict__ count, int* __restrict__ tile_sum,
            int* __restrict__ leave,
            const double* __restrict__ led_part, const int* __restrict__ piece_n, int pieces,
            int seg, double* __restrict__ log) {
  const int ng = S->nghost;
  const int n = S->np - ng;  // the slab's own particles
  const int blk = blockIdx.x - 1;  // the first block sums the ledger
  const int stride = (gridDim.x - 1) * blockDim.x;
  if (!S->active) {  // (ghosts, imported last, sit in the slots after n)
    if (blk >= 0)
      for (int j = blk * blockDim.x + threadIdx.x; j < n; j += stride)
        copy_moving(cur, j, nxt, j);
    return;
  }
  if (blk < 0) {
    ledger_reduce(led_part, piece_n, pieces, G.pieces, G.plan_cols, seg, S);
    ledger_log(S, log);
    if (threadIdx.x == 0) S->pending = 1;
    return;
  }
  if (blk * int(blockDim.x) >= n) return;  // (the grid is for the capacity)
  __shared__ unsigned long long red[3];
  __shared__ int kred[2];
  if (threadIdx.x < 3) red[threadIdx.x] = 0ull;
  if (threadIdx.x == 0) {
    kred[0] = 0x7fffffff;
    kred[1] = -1;
  }
  __syncthreads();
  const double dt = S->dt;
  const Shape sh = shape_of<double>(G);
  unsigned long long m0 = 0, m1 = 0, m2 = 0;
  int kmin = 0x7fffffff, kmax = -1;
  const int lane = threadIdx.x & 31;
  for (int t0 = blk * blockDim.x + (threadIdx.x & ~31); t0 < n; t0 += stride) {
    const int t = t0 + lane;
    const bool ok = t < n;
    int nkey = -1;
    bool stay = ok;
    if (ok) {
      const int j = ng + t;
      const int s = perm[j];
      g2p_particle(cur, s, g2p_in(cur, s), skey[j], nxt, t, nodes, Z, G, P, sh, dt,
                   kRecord ? 1 : 0, kGrad ? 1 : 0, 0, m0, m1, m2, nkey);
      kmin = min(kmin, nkey);
      kmax = max(kmax, nkey);
      if (leave) {
        const int col = nkey / G.nrows;
        if (col < G.pc_lo || col >= G.pc_hi) {
          stay = false;
          leave[atomicAdd(&S->nleave, 1)] = t;
        }
      }
    }
    count_key(nkey, stay, count, tile_sum, nxt.slot + (ok ? t : 0));
  }
  const bool bad = diverged(m0, m1, m2);
  cfl_block_max(m0, m1, m2, red, S);
  key_range(kmin, kmax, kred, S);
  flag_non_finite(bad, S);
}

void launch_g2p(int grid, cudaStream_t st, Particles cur, Particles nxt, const int* perm,
                const int* skey, Nodes nodes, const double* Z, Geom G, Phys P, Scalars* S,
                int* count, int* tile_sum, int* leave, const double* led_part, const UnitPlan& u,
                int pieces, int seg, double* log, int record, int want_grad, bool apart) {
  auto* kernel = record ? k_g2p_t<true, true>
                        : want_grad ? k_g2p_t<false, true> : k_g2p_t<false, false>;
  kernel<<<grid + 1, kG2PThreads, 0, st>>>(cur, nxt, perm, skey, nodes, Z, G, P, S, count,
                                           tile_sum, leave, led_part, u.piece_n,
                                           apart ? 0 : pieces, seg, log);
  if (apart)
    k_ledger<<<1, kLedgerThreads, 0, st>>>(led_part, u.piece_n, pieces, seg, G, S, log);
}

size_t p2g_smem_bytes() { return sizeof(P2GSmemT<double>); }

__global__ void k_pair_join(const double* __restrict__ a, const double* __restrict__ b,
                            double2* __restrict__ out, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    out[i] = double2{a[i], b[i]};
}

__global__ void k_pair_half(const double2* __restrict__ a, int half, double* __restrict__ out,
                            long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const double2 v = a[i];
    out[i] = half ? v.y : v.x;
  }
}

// ---------------------------------------------------------------------------
// BATCH: the same step over many independent scenarios packed back to back.
// Each scenario keeps its own loop state (Scalars), geometry and physics; the
// sort runs over the cells of all of them at once (keys are offset by each
// scenario's first cell), P2G takes units of every scenario from one list,
// and G2P runs one block per 256 particles of one scenario.  A scenario's
// numbers are the same alone and in a batch: its sums run in the same
// per-node order whatever the unit cuts.
// ---------------------------------------------------------------------------
// The scan tiles of a batch pass: those that meet the batch-wide range
// (every cell after a layout change) or a scenario's keys -- the keys its
// cell starts describe (krange) or the keys its last G2P made (knext).  A
// tile that meets neither holds no particle now or at the last sort, and
// its cells' starts (the particles of the scenarios before them) stand
// while the layout does.  One thread per tile; the scenarios' cells are
// consecutive, so a binary search finds the first that meets the tile.
// One more block, the first, ends every scenario's step before and begins
// this one (the tile blocks read neither).
__global__ void k_b_step_begin(const Scn* __restrict__ scn, Scalars* S, int nscn, Scalars* Sg,
                               unsigned char* __restrict__ tflag, int ntiles) {
  if (blockIdx.x == 0) {
    int any = 0;
    for (int s = threadIdx.x; s < nscn; s += blockDim.x) {
      if (scn[s].live) {
        step_begin_one(&S[s], scn[s].G, scn[s].P);
        any |= S[s].active;
      } else {
        S[s].active = 0;
      }
    }
    any = __syncthreads_or(any);
    if (threadIdx.x == 0) Sg->active = any;
    return;
  }
  const int gL = min(Sg->krange[0], Sg->knext[0]), gH = max(Sg->krange[1], Sg->knext[1]);
  for (int t = (blockIdx.x - 1) * blockDim.x + threadIdx.x; t < ntiles;
       t += (gridDim.x - 1) * blockDim.x) {
    const int c0 = t * kScanTile, c1 = c0 + kScanTile - 1;
    bool f = gL <= gH && gL <= c1 && gH >= c0;
    int lo = 0, hi = nscn;  // the first scenario whose cells end after c0
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (scn[mid].c_off + scn[mid].G.nrows * scn[mid].G.ncols <= c0) lo = mid + 1;
      else hi = mid;
    }
    for (int s = lo; !f && s < nscn && scn[s].c_off <= c1; ++s) {
      const int L = min(S[s].krange[0], S[s].knext[0]);
      const int H = max(S[s].krange[1], S[s].knext[1]);
      f = L <= H && L <= c1 && H >= c0;
    }
    tflag[t] = f ? 1 : 0;
  }
}

// The last pass of a call: every scenario's step ends.
__global__ void k_b_step_end(const Scn* __restrict__ scn, Scalars* S, int nscn) {
  for (int s = threadIdx.x; s < nscn; s += blockDim.x)
    if (scn[s].live) step_end_one(&S[s]);
}

// k_order_units of a batch: the list holds {scenario, strip, cA, cB}; the last
// block to finish rolls the scenarios' key ranges over.
__global__ void __launch_bounds__(kOrderThreads, 1)
    k_b_order_units(CellOrder o, UnitPlan u, const Scn* __restrict__ scn, Scalars* S, int nscn,
                    const int* __restrict__ piece_scn, int pieces, const Scalars* Sg,
                    int col_weight) {
  if (!Sg->active) return;
  extern __shared__ unsigned long long sv[];
  const int2 share = plan_share(pieces);
  for (int b = share.x; b < pieces; b += share.y) {
    const int s = piece_scn[b];
    const Geom G = scn[s].G;
    // node columns of the cells the scenario's particles are binned to (the
    // keys its last G2P made), plus the column right of them; every column
    // after a layout change
    int strip, slot, c_lo = 0, c_hi = G.ncols;
    if (!(Sg->krange[0] <= Sg->krange[1])) {
      const int L = S[s].knext[0], H = S[s].knext[1];
      c_lo = (L - scn[s].c_off) / G.nrows;
      c_hi = L > H ? -1 : min((H - scn[s].c_off) / G.nrows + 1, G.ncols);
    }
    piece_of(G, b - scn[s].piece_off, G.ncols + 1, strip, slot, c_lo, c_hi);
    if (S[s].active && c_lo <= c_hi) {  // (else no particle)
      const int n = plan_columns(o.start + scn[s].c_off, G, unit_weight(Sg, u), strip,
                                 unit_buf(sv), u, scn[s].useg_off + slot, col_weight, c_lo, c_hi,
                                 [&](int cA, int cB) { return make_int4(s, strip, cA, cB); });
      if ((threadIdx.x & 31) == 0) u.piece_n[b] = n;
    } else if ((threadIdx.x & 31) == 0) {
      u.piece_n[b] = 0;
    }
  }
  order_share<false>(o, Sg->np, pieces, sv);
  __syncthreads();  // the shared memory is free again
  order_crowded(o, sv);
  if (!last_block(u.ucount + kOrderDone, gridDim.x)) return;
  if (threadIdx.x == 0) *o.list_n = 0;
  for (int s = threadIdx.x; s < nscn; s += blockDim.x) roll_keys(&S[s]);
}

template <class R>
__global__ void __launch_bounds__(kP2GThreads, kP2GMinBlocks)
    k_b_p2g(ParticlesT<R> p, const int* __restrict__ perm, const int* __restrict__ cstart,
            V2<R>* __restrict__ vvL,
            double* __restrict__ led_part, const Scn* __restrict__ scn, Scalars* S,
            UnitPlan up, const Scalars* Sg) {
  if (!Sg->active) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  P2GSmemT<R>& sm = *reinterpret_cast<P2GSmemT<R>*>(smem_raw);
  const int nheavy = up.ucount[kUnitsHeavy], nunits = nheavy + up.ucount[kUnitsPlain];
  __shared__ int next_unit;
  while (true) {
    if (threadIdx.x == 0) next_unit = atomicAdd(up.ucount + kUnitCursor, 1);
    __syncthreads();
    const int k = next_unit;
    __syncthreads();
    if (k >= nunits) break;
    const int f = k < nheavy ? up.cap + k : k - nheavy;  // heavy units first
    const int4 u = up.ulist[f];
    const Geom G = scn[u.x].G;
    const Phys P = scn[u.x].P;
    const int n_off = scn[u.x].n_off, c_off = scn[u.x].c_off;
    NodesT<R> nd{};
    nd.vvL = vvL + n_off;
    p2g_unit<R, 1>(p, perm, cstart + c_off, nd, led_part, G, P, &S[u.x], 0, sm,
                up.uslot[f], make_int4(u.y, u.z, u.w, 0));
  }
}

// gblk[b] = {scenario, its first particle handled by block b}.  A
// scenario's particles are positions [p_off, p_off + np) of the sorted order
// (its cell keys lie between those of the scenarios before and after it).
// Thread j takes position j: slot perm[j] of `cur`, written to slot j of
// `nxt`; a scenario that does not step in this pass (finished, stopped or
// removed) is copied through in sorted order and counted for the next sort;
// a pass in which no scenario steps copies `cur` to `nxt` unchanged.  The
// first nscn blocks sum one scenario's ledger each.
template <class R>
__global__ void __launch_bounds__(kG2PThreads, kG2PMinBlocks)
    k_b_g2p(ParticlesT<R> cur, ParticlesT<R> nxt, const int* __restrict__ perm,
            const int* __restrict__ skey, const V2<R>* __restrict__ vvL,
            const double* __restrict__ Z,
            const Scn* __restrict__ scn, Scalars* S, const int2* __restrict__ gblk,
            const Scalars* Sg, int* __restrict__ count, int* __restrict__ tile_sum,
            const double* __restrict__ led_part, const int* __restrict__ piece_n, int nscn) {
  if (blockIdx.x < nscn) {
    const int q = blockIdx.x;
    if (!Sg->active) return;
    if (scn[q].live && S[q].active) {
      ledger_reduce(led_part + (size_t)scn[q].useg_off * 6, piece_n + scn[q].piece_off,
                    scn[q].led_pieces, scn[q].G.pieces, scn[q].G.plan_cols, scn[q].G.ncols + 1,
                    &S[q]);
      if (threadIdx.x == 0) S[q].pending = 1;
    }
    return;
  }
  const int2 e = gblk[blockIdx.x - nscn];
  const int s = e.x;
  const int p_off = scn[s].p_off, np = scn[s].np;
  const int li = e.y + threadIdx.x;
  const int j = p_off + li;
  const bool ok = li < np;
  if (!Sg->active) {
    if (ok) copy_moving(cur, j, nxt, j);
    return;
  }
  __shared__ unsigned long long red[3];
  __shared__ int kred[2];
  if (threadIdx.x < 3) red[threadIdx.x] = 0ull;
  if (threadIdx.x == 0) {
    kred[0] = 0x7fffffff;
    kred[1] = -1;
  }
  __syncthreads();
  int nkey = -1;
  if (!S[s].active) {  // block-uniform
    if (ok) {
      copy_moving(cur, perm[j], nxt, j);
      nkey = nxt.key[j];
    }
    count_key(nkey, ok, count, tile_sum, nxt.slot + (ok ? j : 0));
    key_range(ok ? nkey : 0x7fffffff, ok ? nkey : -1, kred, &S[s]);
    return;
  }
  const Geom G = scn[s].G;
  const Phys P = scn[s].P;
  const int n_off = scn[s].n_off, c_off = scn[s].c_off;
  NodesT<R> nd{};
  nd.vvL = const_cast<V2<R>*>(vvL) + n_off;
  // (by division: as values read with the scenario they would stay in registers
  // from here on, 136 bytes of spills in place of 32 and 2 % of an ensemble's pass)
  const ShapeT<R> sh{R(1) / R(G.hx), -R(1) / R(G.hx), R(1) / R(G.hy), -R(1) / R(G.hy)};
  unsigned long long m0 = 0, m1 = 0, m2 = 0;
  if (ok)
    g2p_particle(cur, perm[j], g2p_in(cur, perm[j]), skey[j], nxt, j, nd, Z + n_off, G, P,
                 sh, S[s].dt, 0, 0,
                 c_off, m0, m1, m2, nkey);
  count_key(nkey, ok, count, tile_sum, nxt.slot + (ok ? j : 0));
  const bool bad = diverged(m0, m1, m2);
  cfl_block_max(m0, m1, m2, red, &S[s]);
  key_range(ok ? nkey : 0x7fffffff, ok ? nkey : -1, kred, &S[s]);
  flag_non_finite(bad, &S[s]);
}

// k_ledger of a batch, a block per scenario.
__global__ void __launch_bounds__(kLedgerThreads)
    k_b_ledger(const double* __restrict__ led_part, const int* __restrict__ piece_n,
               const Scn* __restrict__ scn, Scalars* S, const Scalars* Sg) {
  const int q = blockIdx.x;
  if (!Sg->active || !scn[q].live || !S[q].active || scn[q].led_pieces > 0) return;
  ledger_reduce_many(led_part + (size_t)scn[q].useg_off * 6, piece_n + scn[q].piece_off,
                     scn[q].nstrips * scn[q].G.pieces, scn[q].G.pieces, scn[q].G.plan_cols,
                     scn[q].G.ncols + 1, &S[q]);
}

template <class R>
__global__ void k_b_unpack(ParticlesT<R> p, const double* __restrict__ raw, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    R* const dst[8] = {p.x, p.y, p.Mp, p.Ap, p.vpx, p.vpy, p.hp, p.Vp};
    constexpr int at[8] = {0, 1, 2, 3, 4, 5, 6, 9};
#pragma unroll
    for (int k = 0; k < 8; ++k) dst[k][i] = R(raw[(size_t)at[k] * n + i]);
    p.mp[i] = V2<R>{R(raw[(size_t)7 * n + i]), R(raw[(size_t)8 * n + i])};
  }
}

__global__ void k_b_layout(Scalars* Sg, int np, int ncells) {
  Scalars s{};
  s.np = np;
  s.active = 1;
  s.krange[0] = 0x7fffffff;
  s.krange[1] = -1;
  s.knext[0] = 0;
  s.knext[1] = ncells - 1;
  *Sg = s;
}

// Compaction of a batch into the other half of its double buffer:
// mblk[b] = {destination first particle, source first particle, count <= 256,
// cell-key shift}.
template <class R>
__global__ void k_b_move(ParticlesT<R> dst, ParticlesT<R> src, const int4* __restrict__ mblk) {
  const int4 m = mblk[blockIdx.x];
  if ((int)threadIdx.x >= m.z) return;
  const int i = m.y + threadIdx.x, o = m.x + threadIdx.x;
  copy_moving(src, i, dst, o);
  dst.key[o] = src.key[i] + m.w;
}

// nblk[b] = {destination first node, source first node, count <= 256, 0}
__global__ void k_b_move_nodes(double* __restrict__ dst, const double* __restrict__ src,
                               const int4* __restrict__ nblk) {
  const int4 m = nblk[blockIdx.x];
  if ((int)threadIdx.x < m.z) dst[m.x + threadIdx.x] = src[m.y + threadIdx.x];
}

// HV: p2g of the updated depth hp at the updated positions, each particle
// still in the cell it was binned to at the start of the step
// (main/optim_par.cpp:650, after the vars were zeroed at :362-364).  `p` is
// the buffer this step's G2P wrote, in this step's sorted order, so the
// particles of a cell are the slots [cstart[cell], cstart[cell+1]) in
// reference index order.  One thread per node walks its four cells in id
// order -- (r-1,c-1) local 3, (r,c-1) local 2, (r-1,c) local 1, (r,c) local
// 0 -- the quadgrid cell-sweep order.  Output-only: launched when outputs
// are recorded.
__global__ void k_hv(const Particles p, const int* __restrict__ cstart,
                     double* __restrict__ HV, Geom G, const Scalars* S) {
  if (!S->active) return;
  const int nrows = G.nrows, ncols = G.ncols;
  const int nn = (nrows + 1) * (ncols + 1);
  const double ihx = 1.0 / G.hx, ihy = 1.0 / G.hy;
  for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < nn;
       n += gridDim.x * blockDim.x) {
    const int r = n % (nrows + 1), c = n / (nrows + 1);
    double acc = 0.0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      // q: 0 -> cell (r-1,c-1) local 3, 1 -> (r,c-1) local 2,
      //    2 -> (r-1,c) local 1,   3 -> (r,c) local 0
      const int cr = (q & 1) ? r : r - 1;
      const int cc = (q & 2) ? c : c - 1;
      const int inode = 3 - q;
      if (cr < 0 || cr >= nrows || cc < 0 || cc >= ncols) continue;
      const int cell = cr + cc * nrows;
      for (int j = cstart[cell]; j < cstart[cell + 1]; ++j) {
        double xi, eta;
        local_xy_g(p.x[j], p.y[j], cc, cr, G, ihx, ihy, xi, eta);
        acc += shp(xi, eta, inode) * p.hp[j];
      }
    }
    HV[n] = acc;
  }
}

// ---- host launchers: the FP64 path and the FP32 form -----------------------
template <class R>
void launch_init_particles(int grid, int block, cudaStream_t st, ParticlesT<R> p,
                           const double* Z, const double* dZdx, const double* dZdy,
                           Geom G, Phys P, Scalars* S, int np, int key_off) {
  k_init_particles<R><<<grid, block, 0, st>>>(p, Z, dZdx, dZdy, G, P, S, np, key_off);
}

template <class R>
void launch_prep(int grid, int block, cudaStream_t st, ParticlesT<R> p, const double* Z,
                 Geom G, Phys P, const Scalars* S, int derive) {
  k_prep<R><<<grid, block, 0, st>>>(p, Z, G, P, S, derive);
}

template <class R>
void launch_b_p2g(int grid, cudaStream_t st, ParticlesT<R> p, const int* perm,
                  const int* cstart, V2<R>* vvL, double* led_part, const Scn* scn,
                  Scalars* S, const UnitPlan& u, const Scalars* Sg) {
  k_b_p2g<R><<<grid, kP2GThreads, sizeof(P2GSmemT<R>), st>>>(p, perm, cstart, vvL, led_part, scn,
                                                             S, u, Sg);
}

template <class R>
int setup_b_p2g() {
  const int smem = int(sizeof(P2GSmemT<R>));
  if (cudaFuncSetAttribute(k_b_p2g<R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           smem) != cudaSuccess)
    return 0;
  cudaFuncSetAttribute(k_b_p2g<R>, cudaFuncAttributePreferredSharedMemoryCarveout,
                       int(cudaSharedmemCarveoutMaxShared));
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_b_p2g<R>, kP2GThreads,
                                                    smem) != cudaSuccess)
    return 0;
  return per_sm < 1 ? 1 : per_sm;
}

template <class R>
void launch_b_g2p(int nblk, cudaStream_t st, ParticlesT<R> cur, ParticlesT<R> nxt,
                  const int* perm, const int* skey, const V2<R>* vvL, const double* Z,
                  const Scn* scn, Scalars* S, const int2* gblk, Scalars* Sg, int* count,
                  int* tile_sum, const double* led_part, const UnitPlan& u, int nscn) {
  k_b_g2p<R><<<nblk + nscn, kG2PThreads, 0, st>>>(cur, nxt, perm, skey, vvL, Z, scn, S, gblk,
                                                  Sg, count, tile_sum, led_part, u.piece_n, nscn);
}

template <class R>
void launch_b_unpack(int grid, cudaStream_t st, ParticlesT<R> p, const double* raw, int n) {
  k_b_unpack<R><<<grid, 256, 0, st>>>(p, raw, n);
}

template <class R>
void launch_b_move(int grid, cudaStream_t st, ParticlesT<R> dst, ParticlesT<R> src,
                   const int4* mblk) {
  k_b_move<R><<<grid, kG2PThreads, 0, st>>>(dst, src, mblk);
}

#define DAMPM_INSTANTIATE(R)                                                          \
  template void launch_init_particles<R>(int, int, cudaStream_t, ParticlesT<R>,       \
                                         const double*, const double*, const double*, \
                                         Geom, Phys, Scalars*, int, int);             \
  template void launch_prep<R>(int, int, cudaStream_t, ParticlesT<R>, const double*,  \
                               Geom, Phys, const Scalars*, int);                      \
  template void launch_b_p2g<R>(int, cudaStream_t, ParticlesT<R>, const int*,         \
                                const int*, V2<R>*, double*, const Scn*, Scalars*,    \
                                const UnitPlan&, const Scalars*);                     \
  template int setup_b_p2g<R>();                                                      \
  template void launch_b_g2p<R>(int, cudaStream_t, ParticlesT<R>, ParticlesT<R>,      \
                                const int*, const int*, const V2<R>*, const double*,  \
                                const Scn*, Scalars*, const int2*, Scalars*, int*,    \
                                int*, const double*, const UnitPlan&, int);           \
  template void launch_b_unpack<R>(int, cudaStream_t, ParticlesT<R>, const double*, int); \
  template void launch_b_move<R>(int, cudaStream_t, ParticlesT<R>, ParticlesT<R>,     \
                                 const int4*);
DAMPM_INSTANTIATE(double)
DAMPM_INSTANTIATE(float)
#undef DAMPM_INSTANTIATE

}  // namespace dampm
