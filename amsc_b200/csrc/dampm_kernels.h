// dampm_kernels.h -- device buffers and kernel entry points of the step.
#pragma once
#include <algorithm>
#include <cstddef>
#include <utility>

#include "dampm_device.cuh"

namespace dampm {

// P2G tiling: kTR node rows per strip (one lane per row in each of the four
// warps, one per quantity group, finishing and starting chains); units of
// variable column width cut to about np / (kUnitsPerCta * CTAs) particles
// (at least kUnitMinWeight), a column weighing its particles + kColWeight;
// particle records staged in shared memory kCap at a time.
constexpr int kTR = 30;
#ifndef DAMPM_UNITS_PER_CTA
#define DAMPM_UNITS_PER_CTA 2
#endif
#ifndef DAMPM_COL_WEIGHT
#define DAMPM_COL_WEIGHT 192
#endif
constexpr int kUnitsPerCta = DAMPM_UNITS_PER_CTA;
// A batch's columns are short (120 particles in 30 rows at 4 per cell), so the
// leading column that each unit stages again weighs more than an even load, as long
// as the units are not long.  Microseconds a pass at one unit per CTA and at two: 96
// scenarios of 64 to 128 cells a side 85.8 and 96.5 (FP32 77.3 and 88.0), 40 of 200
// to 500 183 and 199, 24 requests 196 and 209, four 512 x 512 flows 166 and 177, one
// of 1536 x 1536 292 and 301.  From a weight of 4096 on the load counts: 512
// scenarios (14600 a CTA) take 1640 at one unit per CTA, 1340 at 8192 a unit, 1330
// at 4096, and 2650, 2060 and 2050 when crowded columns have formed (P2G takes units
// of more than twice the weight first); 16 dense flows (7000 a CTA) 557 either way.
constexpr int kBatchUnitsPerCta = 1;
constexpr int kBatchUnitMaxWeight = 4096;
inline int batch_units(int units_per_cta, int ctas, long long np) {
  return int(std::max((long long)units_per_cta * ctas,
                      (np + kBatchUnitMaxWeight - 1) / kBatchUnitMaxWeight));
}
constexpr int kUnitMinWeight = 1024;
// The least weight of a unit, from the number of (strip, column) pairs of the
// grids and P2G's resident CTAs.  Where the pairs that hold particles (a quarter
// of the grid in most flows, at most all) about fit the CTAs, a unit is one
// column: a step of the 4096-particle dam break (195 pairs) takes 28 us against
// 32, of the slab of 10000 (102 pairs) 29 against 35.  Above that the leading
// column that every unit stages again costs more than the shorter chain gives (a
// 0.58M-particle flow: 3 % slower).
inline int unit_min_weight(long long pairs, int ctas) {
  return pairs <= 4LL * ctas ? 1 : kUnitMinWeight;
}
constexpr int kColWeight = DAMPM_COL_WEIGHT;
constexpr int kOrderThreads = 1024;
// A strip is planned in pieces of kPlanCols columns or a multiple of them, a warp
// each: one warp takes 9 us for 512 columns, 35 for the 2048 of a strip, which a flow
// of few particles waits for, and 4 ms for those of a strip of 200000.  The
// particles are ordered beside it, a million in 9 us: a piece has 512 columns for
// every million, and strips of up to 2048 columns with 4M particles stay whole.
// (Each cut between two pieces adds at most one unit to the 50 or more that the
// columns of a piece make by their weight alone.)
constexpr int kPlanCols = 512;
inline void set_pieces(Geom& G, long long np) {
  G.plan_cols = kPlanCols * int((np >> 20) + 1);
  G.pieces = (G.ncols + G.plan_cols - 1) / G.plan_cols;
}
// Strips of a batch (the size of its planner's tables, whatever its capacity), and
// of a single grid, which keeps to the same limit.
constexpr int kMaxStrips = 8192;
constexpr int kP2GThreads = 128;
#ifndef DAMPM_P2G_CAP
#define DAMPM_P2G_CAP 512
#endif
#ifndef DAMPM_P2G_MIN_BLOCKS
#define DAMPM_P2G_MIN_BLOCKS 4
#endif
#ifndef DAMPM_CHAIN_UNROLL
#define DAMPM_CHAIN_UNROLL 2  // single-scenario P2G: chain steps per loop trip
#endif
constexpr int kChainUnroll = DAMPM_CHAIN_UNROLL;
constexpr int kCap = DAMPM_P2G_CAP;
constexpr int kP2GMinBlocks = DAMPM_P2G_MIN_BLOCKS;
constexpr int kG2PThreads = 256;
#ifndef DAMPM_G2P_MIN_BLOCKS
#define DAMPM_G2P_MIN_BLOCKS 4
#endif
constexpr int kG2PMinBlocks = DAMPM_G2P_MIN_BLOCKS;
constexpr int kScanTile = 4096;
// Tile totals lie apart: the atomics that count a flow's few dozen tiles would
// queue at one or two lines of L2 (the count of 1M uploaded particles: 16 us side by
// side, 10 a sector apart).
constexpr int kTileStride = 8;
constexpr int kScanThreads = 1024;
constexpr int kApplyThreads = 256, kApplyRows = kScanTile / (4 * kApplyThreads);
constexpr int kSmallCells = 4 * kScanTile;  // grids that k_scan_scatter takes

// Two values of R side by side (one 16-byte load in FP64, 8 in FP32).
template <class R>
struct Vec2T;
template <>
struct Vec2T<double> {
  using type = double2;
};
template <>
struct Vec2T<float> {
  using type = float2;
};
template <class R>
using V2 = typename Vec2T<R>::type;

// Particle SoA.  The moving fields are kept in cell-sorted order -- by
// (cell of the last binning, reference index) -- in two buffers: each step's
// G2P reads one through the sort permutation and writes the other in the new
// sorted order, so P2G and G2P stream contiguous runs of a cell column
// instead of gathering across the whole set.  `idx` is each slot's index in
// the reference's particle order (DATA order, then the compacted order
// merge/split produces); data going in and out of the library is in that
// order.  R = double is the FP64 path, R = float the FP32 form (batches).
template <class R>
struct ParticlesT {
  // ---- moving (double-buffered, sorted order) ----
  R *x, *y, *vpx, *vpy, *hp, *F11, *F12, *F22, *Mp, *Vp, *H;
  // key: cell of the next binning; idx: reference index; slot: rank among
  // the particles of its cell from the counting sort's atomics
  int *key, *idx, *slot;
  // the record the next P2G transfers, written by G2P (or by k_prep after an
  // upload, a state upload or a merge/split), as pairs that P2G gathers
  // with one copy each:
  //   mp = (mom_px, mom_py)  momentum v*Mp, and qf = (Ap*Fb_x, Ap*Fb_y) the
  //        friction force, as the reference stores them at the end of a
  //        step (main/optim_par.cpp:456-459,600-626);
  //   xe = (xi, eta)  local coordinates in the cell of the next binning;
  //   qg = gravity force -g*Vp*rho*grad(Z)*(1 - H/hp) there
  //        (main/optim_par.cpp:387,447-454).
  V2<R> *mp, *qf, *xe, *qg;
  // velocity gradients (merge/split input, outputs); null in batches
  R *vpx_dx, *vpx_dy, *vpy_dx, *vpy_dy;
  // ---- reference order (not moved by the step) ----
  int *label, *level;
  R *xp, *yp;
  // Ap and Fb as stored at upload / merge/split: valid while Scalars::fresh
  // is set, when the slots are in reference order (otherwise they are
  // derived from the state)
  R *Ap, *Fbx, *Fby;
  // ---- output-only fields of a recorded step (G2P's sorted order) ----
  R *apx, *apy, *Zp, *hpZ, *dZxp, *dZyp, *Fpx, *Fpy, *Frx, *Fry;
};

// Pointers to the moving fields of p, in a fixed order.
constexpr int kMovingR = 15, kMovingI = 3, kMovingV = 4;
template <class R>
struct MovingRefs {
  R** r[kMovingR];
  int** i[kMovingI];
  V2<R>** v[kMovingV];
};
template <class R>
inline MovingRefs<R> moving_refs(ParticlesT<R>& p) {
  return MovingRefs<R>{{&p.x, &p.y, &p.vpx, &p.vpy, &p.hp, &p.F11, &p.F12, &p.F22, &p.Mp,
                        &p.Vp, &p.H, &p.vpx_dx, &p.vpx_dy, &p.vpy_dx, &p.vpy_dy},
                       {&p.key, &p.idx, &p.slot},
                       {&p.mp, &p.qf, &p.xe, &p.qg}};
}
// exchanges the moving buffers of a and b (the other pointers are shared)
template <class R>
inline void swap_moving(ParticlesT<R>& a, ParticlesT<R>& b) {
  MovingRefs<R> ra = moving_refs(a), rb = moving_refs(b);
  for (int k = 0; k < kMovingR; ++k) std::swap(*ra.r[k], *rb.r[k]);
  for (int k = 0; k < kMovingI; ++k) std::swap(*ra.i[k], *rb.i[k]);
  for (int k = 0; k < kMovingV; ++k) std::swap(*ra.v[k], *rb.v[k]);
}
using Particles = ParticlesT<double>;

// Nodal fields, quadgrid node order.
template <class R>
struct NodesT {
  V2<R>* vvL;  // (vvxL, vvyL): the velocities G2P interpolates, one load per node
  // recorded only on output steps
  R *Mv, *mvx, *mvy, *avx, *avy, *vvx, *vvy, *FPxv, *FPyv, *Fricx,
      *Fricy, *Fintx, *Finty, *HV;
};
using Nodes = NodesT<double>;

__global__ void k_step_begin(Scalars* S, Geom G, Phys P);
__global__ void k_step_end(Scalars* S);
// Host launchers of the kernels that exist in both precisions (the kernel
// templates are instantiated in step_kernels.cu, next to their definitions).
template <class R>
void launch_init_particles(int grid, int block, cudaStream_t st, ParticlesT<R> p,
                           const double* Z, const double* dZdx, const double* dZdy,
                           Geom G, Phys P, Scalars* S, int np, int key_off);
// cell keys of the current positions (and idx = slot when set_idx: slots
// in reference order); the next sort scans every cell
__global__ void k_keys(Particles p, Geom G, Scalars* S, int set_idx);
__global__ void k_reduce_state(Particles p, Scalars* S);
template <class R>
void launch_prep(int grid, int block, cudaStream_t st, ParticlesT<R> p, const double* Z,
                 Geom G, Phys P, const Scalars* S, int derive);
// counting sort: slots and counts (after an upload, a state upload or a
// merge/split; a step's G2P counts the keys it makes), the scan of the
// counts over the key range (ranged != 0; else over all n), the scatter into
// perm, and the order by reference index inside each cell
__global__ void k_count(const int* key, int* count, int* tile_sum, int* slot, const Scalars* S);
__global__ void k_count_n(const int* key, int* count, int* tile_sum, int* slot, int n);
// the tile totals of counts that count_key did not make
__global__ void k_scan_sums(const int* count, int n, int* tile_sum, const Scalars* S);
// tflag (may be null): scan only the flagged tiles (k_b_step_begin); big (its size
// in list_n[0]; may be null: a scan alone): the crowded cells
__global__ void k_scan_apply(int* count, int n, const int* tile_sum, int* start, int* big,
                             int* list_n, const Scalars* S, Gate gate, int ranged,
                             const unsigned char* tflag);
// The binning of the particles as they lie in storage, and at each sorted
// position the storage slot, the reference index and the cell key.
struct Binning {
  const int *key, *slot, *idx;
  int *sslot, *sidx, *skey;
};
// (both scatters empty P2G's unit list, counters ucount)
__global__ void k_scatter(Binning n, const int* start, int* tile_sum, int ntiles, int* ucount,
                          Scalars* S, Gate gate);
// scan and scatter in one, for up to kSmallCells cells (dynamic shared memory:
// ncell ints); leaves the counts to be zeroed by the ordering
__global__ void k_scan_scatter(const int* count, int ncell, int* start, int* big, int* ucount,
                               Binning n, Scalars* S, Gate gate);
// What it takes to order the particles inside the cells.
struct CellOrder {
  Binning n;
  const int *start, *big;
  int *list_n, *perm;
  unsigned long long* pk;  // 2 x cap entries, for the crowded cells
  long long cap;
  int* count;  // counts to be zeroed (n_count of them; 0: they are zero)
  int n_count;
};
// The counters of a pass: the crowded cells (k_order_units, which uses them,
// empties the list), P2G's units (plain, heavy) and its work cursor (set to zero
// by the scatter), the blocks of k_order_units that are done.
constexpr int kUnitsPlain = 1, kUnitsHeavy = 2, kUnitCursor = 3, kUnitCounts = 3, kOrderDone = 4;
// P2G's unit list -- the plain units from 0, the heavy ones (which P2G takes
// first) from cap -- with each unit's ledger slot.
struct UnitPlan {
  int target_units, min_weight, cap;
  int4* ulist;
  int* uslot;
  int* piece_n;  // units of each piece of each strip
  int* ucount;   // the counters
};
// orders the particles inside the cells and, with pieces > 0 (all strips'), makes
// the unit list (seg: unit slots per strip) and ends the step before and begins this
// one unless it has begun.  order_smem_bytes(): its dynamic shared memory;
// setup_sort sets the sort kernels' limits (0 on failure)
// repeats: reference indices may repeat inside a cell
void launch_order_units(int grid, cudaStream_t st, const CellOrder& o, const UnitPlan& u, Geom G,
                        Phys P, Scalars* S, int pieces, int seg, Gate gate, bool repeats);
size_t order_smem_bytes();
int setup_sort();
// blocks of 1024 threads for np particles and (k_order_units) `pieces` to plan,
// four to a block, one per SM at most
inline int order_blocks(long long np, long long pieces) {
  const long long b = std::max((np + kOrderThreads - 1) / kOrderThreads, (pieces + 3) / 4);
  return int(b < 1 ? 1 : b > 148 ? 148 : b);
}
// P2G of the single-scenario step (k_p2g specialised for recorded outputs);
// setup_p2g sets its shared-memory attributes and returns the resident CTAs
// per SM (0 on failure)
void launch_p2g(int grid, cudaStream_t st, Particles p, const int* perm, const int* cstart,
                Nodes nodes, double* led_part, Geom G, Phys P, const Scalars* S, int record,
                const UnitPlan& u);
int setup_p2g();
constexpr int kLedgerLog = 1024;  // rows of the per-step ledger log
constexpr int kLedgerThreads = 1024;
// Whether the ledger is summed by a launch of its own (4 us, and in a batch one for
// all) and not by a block of G2P, whose eight warps take 1.3 us a piece while the
// others take 50 us a million particles: where that block would be the last for
// long.
inline bool ledger_apart(long long pieces, long long np, int least) {
  return pieces > least && 4096 * pieces > np;
}
constexpr int kApartLeast = 64, kBatchApartLeast = 256;
// G2P of the single-scenario step (k_g2p_t specialised for the two flags):
// reads `cur` through perm, writes `nxt` in this step's sorted order, counts
// the next binning's keys and sums the ledger (apart: by a launch of its own); the
// step's end is left pending
void launch_g2p(int grid, cudaStream_t st, Particles cur, Particles nxt, const int* perm,
                const int* skey, Nodes nodes, const double* Z, Geom G, Phys P, Scalars* S,
                int* count, int* tile_sum, int* leave, const double* led_part, const UnitPlan& u,
                int pieces, int seg, double* log, int record, int want_grad, bool apart);

// ---- batches of independent scenarios --------------------------------------
// One scenario of a batch: its geometry, physics and place in the packed
// arrays (particles, nodes and cells of all scenarios, back to back).
struct Scn {
  Geom G;
  Phys P;
  int p_off, np;           // particles [p_off, p_off + np)
  int n_off;               // first node
  int c_off;               // first cell (cell keys are c_off + r + c*nrows)
  int nstrips;
  int piece_off;           // its pieces in the batch's order
  int useg_off;            // first unit-plan slot of its first strip
  int live;                // 0 once removed
  int led_pieces;          // its pieces, or 0 where k_b_ledger sums its ledger
};

__global__ void k_b_order_units(CellOrder o, UnitPlan u, const Scn* scn, Scalars* S, int nscn,
                                const int* piece_scn, int pieces, const Scalars* Sg,
                                int col_weight);
__global__ void k_b_step_begin(const Scn* scn, Scalars* S, int nscn, Scalars* Sg,
                               unsigned char* tflag, int ntiles);
__global__ void k_b_step_end(const Scn* scn, Scalars* S, int nscn);
__global__ void k_b_ledger(const double* led_part, const int* piece_n, const Scn* scn, Scalars* S,
                           const Scalars* Sg);
template <class R>
void launch_b_p2g(int grid, cudaStream_t st, ParticlesT<R> p, const int* perm,
                  const int* cstart, V2<R>* vvL, double* led_part, const Scn* scn,
                  Scalars* S, const UnitPlan& u, const Scalars* Sg);
// sets the batched P2G kernel's shared-memory attributes; returns the
// resident CTAs per SM (0 on failure)
template <class R>
int setup_b_p2g();
template <class R>
void launch_b_g2p(int nblk, cudaStream_t st, ParticlesT<R> cur, ParticlesT<R> nxt,
                  const int* perm, const int* skey, const V2<R>* vvL, const double* Z,
                  const Scn* scn, Scalars* S, const int2* gblk, Scalars* Sg, int* count,
                  int* tile_sum, const double* led_part, const UnitPlan& u, int nscn);
template <class R>
void launch_b_move(int grid, cudaStream_t st, ParticlesT<R> dst, ParticlesT<R> src,
                   const int4* mblk);
// n particles of a new scenario from raw[10][n] (x, y, Mp, Ap, vpx, vpy, hp,
// mom_px, mom_py, Vp), converted to R
template <class R>
void launch_b_unpack(int grid, cudaStream_t st, ParticlesT<R> p, const double* raw, int n);
// the totals of a batch's layout; the next sort scans every cell of it
__global__ void k_b_layout(Scalars* Sg, int np, int ncells);
// pairs from their halves, and one half of them
__global__ void k_pair_join(const double* a, const double* b, double2* out, long long n);
__global__ void k_pair_half(const double2* a, int half, double* out, long long n);
__global__ void k_b_move_nodes(double* dst, const double* src, const int4* nblk);

__global__ void k_hv(const Particles p, const int* cstart, double* HV, Geom G,
                     const Scalars* S);

size_t p2g_smem_bytes();  // FP64 P2G staging (the single-scenario path)

// ---- one scenario over slabs of cell columns (slab_kernels.cu) ---------------
constexpr int kSlabRecord = 20;  // doubles per particle record that travels
__global__ void k_slab_pack(Particles p, const int* slots, int n, double* buf);
__global__ void k_slab_unpack(Particles p, const double* buf, int n, int base);
__global__ void k_slab_select(const int* key, int n, int col, int nrows, int* slots,
                              int* count);
__global__ void k_slab_keys(const int* key, const int* slots, int n, int* out);
__global__ void k_slab_check(const int* key, int n, int col_lo, int col_hi, int nrows,
                             Scalars* S);
__global__ void k_slab_move(Particles p, const int2* moves, int n);
__global__ void k_slab_scalars(Scalars* S, int np, int ghosts_added, int ncells);
__global__ void k_slab_set_red(Scalars* S, unsigned long long a, unsigned long long b,
                               unsigned long long c);

}  // namespace dampm
