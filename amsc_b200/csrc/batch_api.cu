// batch_api.cu -- the extern "C" boundary of batches of independent scenarios
// (include/dampm_cuda.h, dampm_batch_*).
//
// A batch packs many scenarios (each its own grid, terrain, particles,
// rheology and loop: fixed dt for NSTEPS or CFL until T) back to back in one
// set of device arrays and advances all of them with one launch per kernel
// and pass.  Scenarios join at the end of the packed arrays (dampm_batch_add)
// and leave by being marked dead (dampm_batch_remove); dampm_batch_compact
// moves the live ones into the other half of a double buffer so that the
// freed room can be reused.  Merge/split and recorded outputs are not part of
// a batch.
#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/dampm_cuda.h"
#include "dampm_kernels.h"
#include "host_util.h"

using namespace dampm;

namespace {

// A piece of an addition's arrays (1 MB: a larger one costs more to set up
// than it saves)
constexpr size_t kRawDoubles = size_t(1) << 17;

struct HostScn {
  int handle = -1;
  Scn d{};  // the device table entry
  dampm_grid grid{};
  dampm_params params{};
  long long nn = 0, nc = 0;
};

}  // namespace

struct dampm_batch {
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  long long P_cap = 0, N_cap = 0;
  int S_cap = 0, STRIP_cap = 0, B_cap = 0;
  long long USEG_cap = 0;
  // packed totals (live and dead scenarios)
  long long P_tot = 0, N_tot = 0, C_tot = 0, useg_tot = 0;
  int strips_tot = 0, pieces_tot = 0, nblk = 0;
  std::vector<HostScn> scns;  // packed order = device table order
  int next_handle = 0;
  // device
  int precision = DAMPM_FP64;
  // the two halves of the double buffer of the moving particle fields: each
  // pass's G2P reads half `cur` and writes the other, and so does a
  // compaction; the fields that only an upload uses are shared
  ParticlesT<double> p64[2]{};  // FP64
  ParticlesT<float> p32[2]{};   // FP32 form
  double* Z[2] = {nullptr, nullptr};
  int cur = 0;  // half holding the particles; also the terrain's half
  int zcur = 0;
  void* vvL = nullptr;  // pairs (vvxL, vvyL) of the precision's real type
  double* stage = nullptr;  // one field in reference order, for downloads
  unsigned long long* sortbuf = nullptr;  // 2 x capacity: crowded cells' order
  int *count = nullptr, *start = nullptr, *perm = nullptr;
  // of each sorted position: cell, storage slot and reference index before the
  // order inside the cells (the last two in `stage`: a pass uses them, a download
  // comes between passes)
  int *skey = nullptr, *sslot = nullptr, *sidx = nullptr;
  int *tile_sum = nullptr, *cbig = nullptr;
  unsigned char* tflag = nullptr;  // the scan tiles of a pass (k_b_step_begin)
  int4* ulist = nullptr;  // plain units, then heavy ones (USEG_cap each)
  int* uslot = nullptr;   // their ledger slots
  int *piece_n = nullptr, *ucount = nullptr, *piece_scn = nullptr;
  double* led_part = nullptr;
  int2* gblk = nullptr;
  int4 *mblk = nullptr, *nmove = nullptr;
  Scn* scn = nullptr;
  Scalars *S = nullptr, *Sg = nullptr;
  Scalars* Sh = nullptr;  // pinned mirror of S
  void* pinned = nullptr;  // the host memory of Sh, the mirrors and raw_h
  // pinned mirrors of the tables: an addition appends its entries and copies
  // them without waiting (only a compaction, which waits, rewrites them)
  Scn* scn_h = nullptr;
  int* piece_scn_h = nullptr;
  int2* gblk_h = nullptr;
  // staging of an addition's arrays, pinned and on the device, two of each:
  // one is filled while the other travels
  double* raw_h[2] = {nullptr, nullptr};
  double* raw_d[2] = {nullptr, nullptr};
  cudaEvent_t raw_ev[2] = {nullptr, nullptr};
  int raw_turn = 0;
  int p2g_grid = 1;
  long long launches = 0;
  // tuning: P2G units per CTA and the weight of a column in the unit plan
  int units_per_cta = kBatchUnitsPerCta, col_weight = kColWeight;
  // kBatchGraphPasses passes captured in a CUDA graph, replayed while the
  // layout holds; one graph per half the passes start from
  int use_graphs = 1;
  bool graph_dirty[2] = {true, true};
  cudaGraphExec_t graph[2] = {nullptr, nullptr};
  std::vector<void*> allocs;
  std::string err;
};

namespace {

#define BCK(call)                                                         \
  do {                                                                    \
    cudaError_t e_ = (call);                                              \
    if (e_ != cudaSuccess) {                                              \
      b->err = std::string(#call) + ": " + cudaGetErrorString(e_);        \
      return DAMPM_ERR_CUDA;                                              \
    }                                                                     \
  } while (0)

int bfail(dampm_batch* b, int code, const std::string& msg) {
  if (b) b->err = msg;
  return code;
}

template <class T>
int balloc(dampm_batch* b, T** ptr, size_t n) {
  void* q = nullptr;
  if (n == 0) n = 1;
  cudaError_t e = cudaMalloc(&q, n * sizeof(T));
  if (e != cudaSuccess) {
    b->err = std::string("cudaMalloc: ") + cudaGetErrorString(e);
    return DAMPM_ERR_CUDA;
  }
  b->allocs.push_back(q);
  *ptr = static_cast<T*>(q);
  return DAMPM_OK;
}

template <class R>
ParticlesT<R>* halves(dampm_batch* b);
template <>
ParticlesT<double>* halves<double>(dampm_batch* b) { return b->p64; }
template <>
ParticlesT<float>* halves<float>(dampm_batch* b) { return b->p32; }

// the particle arrays of both halves: the moving fields of each half, and
// the fields only an upload uses (Ap, Fb, label, level) shared
template <class R>
int alloc_particles(dampm_batch* b, ParticlesT<R>* h) {
  for (int k = 0; k < 2; ++k) {
    MovingRefs<R> m = moving_refs(h[k]);
    for (int f = 0; f < kMovingR; ++f) {
      if (m.r[f] == &h[k].vpx_dx || m.r[f] == &h[k].vpx_dy || m.r[f] == &h[k].vpy_dx ||
          m.r[f] == &h[k].vpy_dy)
        continue;  // no gradients in a batch (no merge/split)
      int rc = balloc(b, m.r[f], size_t(b->P_cap));
      if (rc) return rc;
    }
    for (int f = 0; f < kMovingI; ++f) {
      int rc = balloc(b, m.i[f], size_t(b->P_cap));
      if (rc) return rc;
    }
    for (int f = 0; f < kMovingV; ++f) {
      int rc = balloc(b, m.v[f], size_t(b->P_cap));
      if (rc) return rc;
    }
  }
  R** f[] = {&h[0].Ap, &h[0].Fbx, &h[0].Fby};
  for (R** q : f) {
    int rc = balloc(b, q, size_t(b->P_cap));
    if (rc) return rc;
  }
  int** fi[] = {&h[0].label, &h[0].level};
  for (int** q : fi) {
    int rc = balloc(b, q, size_t(b->P_cap));
    if (rc) return rc;
  }
  h[1].Ap = h[0].Ap;
  h[1].Fbx = h[0].Fbx;
  h[1].Fby = h[0].Fby;
  h[1].label = h[0].label;
  h[1].level = h[0].level;
  return DAMPM_OK;
}

template <class R>
ParticlesT<R> shifted(const ParticlesT<R>& p, long long off) {
  ParticlesT<R> q = p;
  MovingRefs<R> m = moving_refs(q);
  for (R** d : m.r)
    if (*d) *d += off;
  for (int** d : m.i)
    if (*d) *d += off;
  for (V2<R>** d : m.v)
    if (*d) *d += off;
  R** f[] = {&q.Ap, &q.Fbx, &q.Fby};
  for (R** d : f)
    if (*d) *d += off;
  int** fi[] = {&q.label, &q.level};
  for (int** d : fi)
    if (*d) *d += off;
  return q;
}

int strips_of(const dampm_grid& g) { return (g.Ney + 1 + kTR - 1) / kTR; }
int pieces_of(const Scn& d) { return d.nstrips * d.G.pieces; }

// Appends scenario `pos` to the table mirrors; the entries' ranges in *piece
// and *blk.
void append_tables(dampm_batch* b, size_t pos, int2* piece, int2* blk) {
  const Scn& d = b->scns[pos].d;
  b->scn_h[pos] = d;
  *piece = make_int2(d.piece_off, pieces_of(d));
  for (int k = 0; k < piece->y; ++k) b->piece_scn_h[d.piece_off + k] = int(pos);
  blk->x = b->nblk;
  for (int f = 0; f < d.np; f += kG2PThreads) b->gblk_h[b->nblk++] = make_int2(int(pos), f);
  blk->y = b->nblk - blk->x;
}

// Uploads entries of the tables (scenarios, pieces, G2P blocks) with the
// batch totals, without waiting.
int upload_tables(dampm_batch* b, int2 scn, int2 piece, int2 blk) {
  if (scn.y > 0)
    BCK(cudaMemcpyAsync(b->scn + scn.x, b->scn_h + scn.x, sizeof(Scn) * size_t(scn.y),
                        cudaMemcpyHostToDevice, b->stream));
  if (piece.y > 0)
    BCK(cudaMemcpyAsync(b->piece_scn + piece.x, b->piece_scn_h + piece.x,
                        sizeof(int) * size_t(piece.y), cudaMemcpyHostToDevice, b->stream));
  if (blk.y > 0)
    BCK(cudaMemcpyAsync(b->gblk + blk.x, b->gblk_h + blk.x, sizeof(int2) * size_t(blk.y),
                        cudaMemcpyHostToDevice, b->stream));
  // the next sort scans every cell of the new layout
  k_b_layout<<<1, 1, 0, b->stream>>>(b->Sg, int(b->P_tot),
                                     int(std::max<long long>(b->C_tot, 1)));
  BCK(cudaGetLastError());
  b->graph_dirty[0] = b->graph_dirty[1] = true;  // launch sizes or buffers changed
  return DAMPM_OK;
}

int find(dampm_batch* b, int handle) {
  for (size_t s = 0; s < b->scns.size(); ++s)
    if (b->scns[s].handle == handle) return int(s);
  return -1;
}

int read_scalars(dampm_batch* b) {
  if (b->scns.empty()) return DAMPM_OK;
  BCK(cudaMemcpyAsync(b->Sh, b->S, sizeof(Scalars) * b->scns.size(),
                      cudaMemcpyDeviceToHost, b->stream));
  BCK(cudaStreamSynchronize(b->stream));
  return DAMPM_OK;
}

bool ledgers_apart(const dampm_batch* b) {
  for (const HostScn& h : b->scns)
    if (h.d.led_pieces == 0) return true;
  return false;
}

// One pass of every live scenario: pass_launches() kernel launches.
int pass_launches(const dampm_batch* b) { return ledgers_apart(b) ? 7 : 6; }
int enqueue_pass(dampm_batch* b) {
  cudaStream_t st = b->stream;
  const int nscn = int(b->scns.size());
  const int ncell = int(std::max<long long>(b->C_tot, 1));
  const int ntiles = (ncell + kScanTile - 1) / kScanTile;
  const int nxt = 1 - b->cur;
  const int* key = b->precision == DAMPM_FP32 ? b->p32[b->cur].key : b->p64[b->cur].key;
  const int* slot = b->precision == DAMPM_FP32 ? b->p32[b->cur].slot : b->p64[b->cur].slot;
  const int* idx = b->precision == DAMPM_FP32 ? b->p32[b->cur].idx : b->p64[b->cur].idx;
  const int gp = grid_blocks(b->P_tot, 256);
  // the step's begin, and the scan tiles of the sort: the counting sort of
  // every scenario at once (G2P counted the keys), over the tiles the
  // scenarios' key ranges meet
  k_b_step_begin<<<1 + grid_blocks(ntiles, 256), 256, 0, st>>>(b->scn, b->S, nscn, b->Sg,
                                                                b->tflag, ntiles);
  const Gate gate = kGateBegun;
  k_scan_apply<<<ntiles, kApplyThreads, 0, st>>>(b->count, ncell, b->tile_sum, b->start, b->cbig,
                                                b->ucount, b->Sg, gate, 0, b->tflag);
  const Binning n{key, slot, idx, b->sslot, b->sidx, b->skey};
  k_scatter<<<gp, 256, 0, st>>>(n, b->start, b->tile_sum, ntiles, b->ucount, b->Sg, gate);
  const UnitPlan u{batch_units(b->units_per_cta, b->p2g_grid, b->P_tot),
                   unit_min_weight(b->useg_tot, b->p2g_grid), int(b->USEG_cap), b->ulist,
                   b->uslot, b->piece_n, b->ucount};
  k_b_order_units<<<order_blocks(b->P_tot, b->pieces_tot), kOrderThreads, order_smem_bytes(), st>>>(
      CellOrder{n, b->start, b->cbig, b->ucount, b->perm, b->sortbuf, b->P_cap, b->count, 0},
      u, b->scn, b->S, nscn, b->piece_scn, b->pieces_tot, b->Sg, b->col_weight);
  if (b->precision == DAMPM_FP32)
    launch_b_p2g<float>(b->p2g_grid, st, b->p32[b->cur], b->perm, b->start,
                        static_cast<float2*>(b->vvL),
                        b->led_part, b->scn, b->S, u, b->Sg);
  else
    launch_b_p2g<double>(b->p2g_grid, st, b->p64[b->cur], b->perm, b->start,
                         static_cast<double2*>(b->vvL),
                         b->led_part, b->scn, b->S, u, b->Sg);
  if (b->precision == DAMPM_FP32)
    launch_b_g2p<float>(b->nblk, st, b->p32[b->cur], b->p32[nxt], b->perm, b->skey,
                        static_cast<const float2*>(b->vvL), b->Z[b->zcur], b->scn, b->S,
                        b->gblk, b->Sg, b->count, b->tile_sum, b->led_part, u, nscn);
  else
    launch_b_g2p<double>(b->nblk, st, b->p64[b->cur], b->p64[nxt], b->perm, b->skey,
                         static_cast<const double2*>(b->vvL), b->Z[b->zcur], b->scn, b->S,
                         b->gblk, b->Sg, b->count, b->tile_sum, b->led_part, u, nscn);
  if (ledgers_apart(b))
    k_b_ledger<<<nscn, kLedgerThreads, 0, st>>>(b->led_part, b->piece_n, b->scn, b->S, b->Sg);
  b->cur = nxt;
  b->launches += pass_launches(b);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return bfail(b, DAMPM_ERR_CUDA, cudaGetErrorString(e));
  return DAMPM_OK;
}

// Ends the last pass of a call (a pass ends with the begin of the next one).
int enqueue_end(dampm_batch* b) {
  k_b_step_end<<<1, 1024, 0, b->stream>>>(b->scn, b->S, int(b->scns.size()));
  b->launches += 1;
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return bfail(b, DAMPM_ERR_CUDA, cudaGetErrorString(e));
  return DAMPM_OK;
}

// A piece of an addition's host arrays in flight: `fill` writes it into a
// pinned buffer, which is copied to its device twin (*dev).  Two buffers
// alternate, so the host fills one while the other travels; raw_sent marks
// the end of what reads the device twin.
template <class F>
int stage_raw(dampm_batch* b, size_t n, F fill, double** dev) {
  const int t = b->raw_turn;
  BCK(cudaEventSynchronize(b->raw_ev[t]));
  fill(b->raw_h[t]);
  BCK(cudaMemcpyAsync(b->raw_d[t], b->raw_h[t], sizeof(double) * n, cudaMemcpyHostToDevice,
                      b->stream));
  *dev = b->raw_d[t];
  return DAMPM_OK;
}
int raw_sent(dampm_batch* b) {
  BCK(cudaEventRecord(b->raw_ev[b->raw_turn], b->stream));
  b->raw_turn ^= 1;
  return DAMPM_OK;
}

// Terrain and particles of one scenario into the current half, then the
// initial state of main/optim_par.cpp:239-264 on the device.  The arrays go
// through the staging in pieces and are converted on the device, so the call
// waits for nothing but a free piece (96 scenarios of 12000 particles: 31 ms
// in FP64 and 42 in FP32 with one copy, one wait and a conversion on the host
// per array).
template <class R>
int upload_scenario(dampm_batch* b, const Scn& d, int pos, long long np, long long nn,
                    const double* Z, const double* const* in, double* Zs) {
  ParticlesT<R> p = shifted(halves<R>(b)[b->cur], d.p_off);
  cudaStream_t st = b->stream;
  for (long long o = 0; o < nn; o += (long long)kRawDoubles) {
    const size_t n = size_t(std::min<long long>((long long)kRawDoubles, nn - o));
    double* dev = nullptr;
    int rc = stage_raw(b, n, [&](double* h) { std::memcpy(h, Z + o, sizeof(double) * n); }, &dev);
    if (rc) return rc;
    BCK(cudaMemcpyAsync(Zs + o, dev, sizeof(double) * n, cudaMemcpyDeviceToDevice, st));
    rc = raw_sent(b);
    if (rc) return rc;
  }
  const long long per = (long long)(kRawDoubles / 10);
  for (long long o = 0; o < np; o += per) {
    const size_t n = size_t(std::min(per, np - o));
    double* dev = nullptr;
    int rc = stage_raw(
        b, 10 * n,
        [&](double* h) {
          for (int k = 0; k < 10; ++k) std::memcpy(h + k * n, in[k] + o, sizeof(double) * n);
        },
        &dev);
    if (rc) return rc;
    launch_b_unpack<R>(grid_blocks((long long)n, 256), st, shifted(p, o), dev, int(n));
    b->launches += 1;
    rc = raw_sent(b);
    if (rc) return rc;
  }
  // (the terrain gradients only feed recorded outputs, which a batch does
  // not keep, so Z stands in for them)
  launch_init_particles<R>(grid_blocks(np, 256), 256, st, p, Zs, Zs, Zs, d.G, d.P,
                           b->S + pos, int(np), d.c_off);
  // the new keys join the counts the last pass left for the next sort
  k_count_n<<<grid_blocks(np, 256), 256, 0, st>>>(p.key, b->count, b->tile_sum, p.slot, int(np));
  launch_prep<R>(grid_blocks(np, 256), 256, st, p, Zs, d.G, d.P, b->S + pos, 0);
  b->launches += 3;
  BCK(cudaGetLastError());
  return DAMPM_OK;
}

// out[idx[j]] = a[j] over one scenario's n particles (idx: its reference
// index), converted to double
template <class R>
__global__ void k_b_to_ref(const R* __restrict__ a, const int* __restrict__ idx,
                           double* __restrict__ out, int n) {
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x)
    out[idx[j]] = double(a[j]);
}

template <class R>
__global__ void k_b_pair_to_ref(const V2<R>* __restrict__ a, int half,
                                const int* __restrict__ idx, double* __restrict__ out,
                                int n) {
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    const V2<R> v = a[j];
    out[idx[j]] = double(half ? v.y : v.x);
  }
}

template <class R>
int download_field(dampm_batch* b, const Scn& d, const std::string& f, double* out) {
  const ParticlesT<R> p = shifted(halves<R>(b)[b->cur], d.p_off);
  const R* src = nullptr;
  int pair_half = -1;  // mom_px / mom_py: one half of the momentum pair
  if (f == "x") src = p.x;
  else if (f == "y") src = p.y;
  else if (f == "vpx") src = p.vpx;
  else if (f == "vpy") src = p.vpy;
  else if (f == "hp") src = p.hp;
  else if (f == "F_11") src = p.F11;
  else if (f == "F_12" || f == "F_21") src = p.F12;
  else if (f == "F_22") src = p.F22;
  else if (f == "Mp") src = p.Mp;
  else if (f == "Vp") src = p.Vp;
  else if (f == "H") src = p.H;
  else if (f == "mom_px" || f == "mom_py") pair_half = f == "mom_px" ? 0 : 1;
  if (!src && pair_half < 0)
    return bfail(b, DAMPM_ERR_UNKNOWN_FIELD, "unknown batch field " + f);
  if (d.np == 0) return DAMPM_OK;
  const int gp = grid_blocks(d.np, 256);
  if (pair_half >= 0)
    k_b_pair_to_ref<R><<<gp, 256, 0, b->stream>>>(p.mp, pair_half, p.idx, b->stage, d.np);
  else
    k_b_to_ref<R><<<gp, 256, 0, b->stream>>>(src, p.idx, b->stage, d.np);
  BCK(cudaGetLastError());
  BCK(cudaMemcpyAsync(out, b->stage, sizeof(double) * size_t(d.np), cudaMemcpyDeviceToHost,
                      b->stream));
  BCK(cudaStreamSynchronize(b->stream));
  return DAMPM_OK;
}

}  // namespace

extern "C" {

int dampm_batch_create(long long particle_cap, long long node_cap, int scenario_cap,
                       int precision, void* cuda_stream, dampm_batch** out) {
  if (!out || particle_cap < 1 || node_cap < 4 || scenario_cap < 1 ||
      particle_cap > 0x7fffffffLL || node_cap > 0x7fffffffLL)
    return DAMPM_ERR_ARG;
  if (precision != DAMPM_FP64 && precision != DAMPM_FP32) return DAMPM_ERR_ARG;
  dampm_batch* b = new dampm_batch();
  b->precision = precision;
  const bool f32 = precision == DAMPM_FP32;
  const size_t rsz = f32 ? sizeof(float) : sizeof(double);
  b->P_cap = particle_cap;
  b->N_cap = node_cap;
  b->S_cap = scenario_cap;
  b->STRIP_cap = kMaxStrips;
  // unit-plan slots: a scenario takes ceil((Ney+1)/30) * (Nex+1) of them,
  // at most nn/30 + (Nex+1)
  b->USEG_cap = node_cap / 24 + 2048LL * scenario_cap + 1024;
  b->B_cap = int(particle_cap / kG2PThreads) + scenario_cap + 1;
  if (cuda_stream) {
    b->stream = static_cast<cudaStream_t>(cuda_stream);
  } else {
    if (cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking) != cudaSuccess) {
      delete b;
      return DAMPM_ERR_CUDA;
    }
    b->own_stream = true;
  }
  int rc = f32 ? alloc_particles(b, b->p32) : alloc_particles(b, b->p64);
  const size_t nn = size_t(node_cap), pc = size_t(particle_cap);
  rc = rc ? rc : balloc(b, &b->stage, pc);
  rc = rc ? rc : balloc(b, &b->sortbuf, 2 * pc);
  rc = rc ? rc : balloc(b, &b->Z[0], nn);
  rc = rc ? rc : balloc(b, &b->Z[1], nn);
  rc = rc ? rc : balloc(b, reinterpret_cast<unsigned char**>(&b->vvL), 2 * nn * rsz);
  // cells of all scenarios: fewer than their nodes
  rc = rc ? rc : balloc(b, &b->count, nn + 4);
  rc = rc ? rc : balloc(b, &b->start, nn + 1);
  rc = rc ? rc : balloc(b, &b->tile_sum, (nn / kScanTile + 2) * kTileStride);
  rc = rc ? rc : balloc(b, &b->tflag, nn / kScanTile + 2);
  rc = rc ? rc : balloc(b, &b->perm, pc);
  rc = rc ? rc : balloc(b, &b->skey, pc);
  b->sslot = reinterpret_cast<int*>(b->stage);
  b->sidx = b->sslot + pc;
  rc = rc ? rc : balloc(b, &b->cbig, pc / 256 + 4);
  const size_t us = size_t(b->USEG_cap);
  rc = rc ? rc : balloc(b, &b->ulist, 2 * us);
  rc = rc ? rc : balloc(b, &b->uslot, 2 * us);
  rc = rc ? rc : balloc(b, &b->led_part, us * 6);
  // a strip of n columns has at most n / kPlanCols + 1 pieces
  const size_t pieces = size_t(b->STRIP_cap) + us / kPlanCols;
  rc = rc ? rc : balloc(b, &b->piece_n, pieces);
  rc = rc ? rc : balloc(b, &b->piece_scn, pieces);
  rc = rc ? rc : balloc(b, &b->ucount, 8);
  if (rc == DAMPM_OK && cudaMemsetAsync(b->ucount, 0, sizeof(int) * 8, b->stream) != cudaSuccess)
    rc = bfail(b, DAMPM_ERR_CUDA, "cudaMemsetAsync failed");
  rc = rc ? rc : balloc(b, &b->gblk, size_t(b->B_cap));
  rc = rc ? rc : balloc(b, &b->mblk, size_t(b->B_cap));
  rc = rc ? rc : balloc(b, &b->nmove, nn / kG2PThreads + size_t(scenario_cap) + 1);
  rc = rc ? rc : balloc(b, &b->scn, size_t(scenario_cap));
  rc = rc ? rc : balloc(b, &b->S, size_t(scenario_cap));
  rc = rc ? rc : balloc(b, &b->Sg, 1);
  for (int k = 0; k < 2; ++k) {
    rc = rc ? rc : balloc(b, &b->raw_d[k], kRawDoubles);
    if (rc == DAMPM_OK &&
        cudaEventCreateWithFlags(&b->raw_ev[k], cudaEventDisableTiming) != cudaSuccess)
      rc = bfail(b, DAMPM_ERR_CUDA, "cudaEventCreate failed");
  }
  if (rc == DAMPM_OK) {  // one pinned allocation, cut up
    size_t bytes = 0;
    auto place = [&](size_t n) {
      const size_t at = bytes;
      bytes += (n + 255) / 256 * 256;
      return at;
    };
    const size_t at_S = place(sizeof(Scalars) * size_t(scenario_cap));
    const size_t at_scn = place(sizeof(Scn) * size_t(scenario_cap));
    const size_t at_piece = place(sizeof(int) * pieces);
    const size_t at_blk = place(sizeof(int2) * size_t(b->B_cap));
    const size_t at_raw[2] = {place(sizeof(double) * kRawDoubles),
                              place(sizeof(double) * kRawDoubles)};
    if (cudaMallocHost(&b->pinned, bytes) != cudaSuccess) {
      rc = bfail(b, DAMPM_ERR_CUDA, "cudaMallocHost failed");
    } else {
      char* p = static_cast<char*>(b->pinned);
      b->Sh = reinterpret_cast<Scalars*>(p + at_S);
      b->scn_h = reinterpret_cast<Scn*>(p + at_scn);
      b->piece_scn_h = reinterpret_cast<int*>(p + at_piece);
      b->gblk_h = reinterpret_cast<int2*>(p + at_blk);
      for (int k = 0; k < 2; ++k) b->raw_h[k] = reinterpret_cast<double*>(p + at_raw[k]);
    }
  }
  if (rc == DAMPM_OK) {
    cudaMemsetAsync(b->count, 0, sizeof(int) * (nn + 4), b->stream);
    cudaMemsetAsync(b->tile_sum, 0, sizeof(int) * kTileStride * (nn / kScanTile + 2), b->stream);
    cudaMemsetAsync(b->vvL, 0, 2 * rsz * nn, b->stream);
    cudaMemsetAsync(b->S, 0, sizeof(Scalars) * size_t(scenario_cap), b->stream);
    cudaMemsetAsync(b->Sg, 0, sizeof(Scalars), b->stream);
    const int per_sm = f32 ? setup_b_p2g<float>() : setup_b_p2g<double>();
    if (per_sm == 0) rc = bfail(b, DAMPM_ERR_CUDA, "cannot configure P2G shared memory");
    if (!setup_sort()) rc = bfail(b, DAMPM_ERR_CUDA, "cannot configure the sort's shared memory");
    int nsm = 0, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    b->p2g_grid = std::max(1, nsm * std::max(per_sm, 1));
    if (cudaStreamSynchronize(b->stream) != cudaSuccess) rc = DAMPM_ERR_CUDA;
  }
  if (rc != DAMPM_OK) {
    dampm_batch_destroy(b);
    return rc;
  }
  *out = b;
  return DAMPM_OK;
}

int dampm_batch_destroy(dampm_batch* b) {
  if (!b) return DAMPM_ERR_ARG;
  if (b->stream) cudaStreamSynchronize(b->stream);
  for (cudaGraphExec_t g : b->graph)
    if (g) cudaGraphExecDestroy(g);
  for (void* q : b->allocs) cudaFree(q);
  if (b->pinned) cudaFreeHost(b->pinned);
  for (cudaEvent_t e : b->raw_ev)
    if (e) cudaEventDestroy(e);
  if (b->own_stream) cudaStreamDestroy(b->stream);
  delete b;
  return DAMPM_OK;
}

const char* dampm_batch_last_error(dampm_batch* b) {
  return b ? b->err.c_str() : "null batch";
}

int dampm_batch_add(dampm_batch* b, const dampm_grid* grid, const dampm_params* params,
                    const double* Z, long long np, const double* x, const double* y,
                    const double* Mp, const double* Ap, const double* vpx,
                    const double* vpy, const double* hp, const double* mom_px,
                    const double* mom_py, const double* Vp, int* handle) {
  if (!b || !grid || !params || !Z || !handle || np < 1) return DAMPM_ERR_ARG;
  if (!x || !y || !Mp || !Ap || !vpx || !vpy || !hp || !mom_px || !mom_py || !Vp)
    return DAMPM_ERR_ARG;
  if (grid->Nex < 1 || grid->Ney < 1 || !(grid->hx > 0) || !(grid->hy > 0))
    return bfail(b, DAMPM_ERR_ARG, "bad grid");
  // An addition runs when it is called: captured, its copies would read staging
  // buffers that have moved on by the time the graph is launched.
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  BCK(cudaStreamIsCapturing(b->stream, &cs));
  if (cs != cudaStreamCaptureStatusNone)
    return bfail(b, DAMPM_ERR_CUDA, "a scenario cannot be added while its stream is captured");
  HostScn h;
  h.grid = *grid;
  h.params = *params;
  h.nn = (long long)(grid->Nex + 1) * (grid->Ney + 1);
  h.nc = (long long)grid->Nex * grid->Ney;
  const int nstrips = strips_of(*grid);
  const long long useg = (long long)nstrips * (grid->Nex + 1);
  const int blocks = int((np + kG2PThreads - 1) / kG2PThreads);
  if (int(b->scns.size()) >= b->S_cap || b->P_tot + np > b->P_cap ||
      b->N_tot + h.nn > b->N_cap || b->strips_tot + nstrips > b->STRIP_cap ||
      b->useg_tot + useg > b->USEG_cap || b->nblk + blocks > b->B_cap)
    return bfail(b, DAMPM_ERR_CAPACITY,
                 "batch full: remove finished scenarios and compact, or create a larger batch");
  Scn& d = h.d;
  d.G = make_geom(*grid);
  set_pieces(d.G, np);
  d.P = make_phys(*params);
  d.p_off = int(b->P_tot);
  d.np = int(np);
  d.n_off = int(b->N_tot);
  d.c_off = int(b->C_tot);
  d.nstrips = nstrips;
  d.piece_off = b->pieces_tot;
  d.led_pieces = ledger_apart(pieces_of(d), np, kBatchApartLeast) ? 0 : pieces_of(d);
  d.useg_off = int(b->useg_tot);
  d.live = 1;
  h.handle = b->next_handle++;
  const int pos = int(b->scns.size());
  // particles and terrain into the current half
  cudaStream_t st = b->stream;
  double* Zs = b->Z[b->zcur] + d.n_off;
  Scalars s0{};
  s0.fresh = 1;
  s0.np = int(np);
  // the first plan covers all of the scenario's cells
  s0.krange[0] = 0x7fffffff;
  s0.krange[1] = -1;
  s0.knext[0] = d.c_off;
  s0.knext[1] = d.c_off + int(h.nc) - 1;
  b->Sh[pos] = s0;
  BCK(cudaMemcpyAsync(b->S + pos, b->Sh + pos, sizeof(Scalars), cudaMemcpyHostToDevice,
                      st));
  const double* in[10] = {x, y, Mp, Ap, vpx, vpy, hp, mom_px, mom_py, Vp};
  int urc = b->precision == DAMPM_FP32
                ? upload_scenario<float>(b, d, pos, np, h.nn, Z, in, Zs)
                : upload_scenario<double>(b, d, pos, np, h.nn, Z, in, Zs);
  if (urc) return urc;
  BCK(cudaGetLastError());
  b->scns.push_back(h);
  b->P_tot += np;
  b->N_tot += h.nn;
  b->C_tot += h.nc;
  b->strips_tot += nstrips;
  b->pieces_tot += pieces_of(d);
  b->useg_tot += useg;
  int2 piece, blk;
  append_tables(b, size_t(pos), &piece, &blk);
  int rc = upload_tables(b, make_int2(pos, 1), piece, blk);
  if (rc) return rc;
  *handle = h.handle;
  return DAMPM_OK;
}

int dampm_batch_remove(dampm_batch* b, int handle) {
  if (!b) return DAMPM_ERR_ARG;
  const int s = find(b, handle);
  if (s < 0) return bfail(b, DAMPM_ERR_ARG, "unknown scenario handle");
  b->scns[s].d.live = 0;
  b->scns[s].handle = -1;
  const int live = 0;
  BCK(cudaMemcpyAsync(reinterpret_cast<char*>(b->scn + s) + offsetof(Scn, live), &live,
                      sizeof(int), cudaMemcpyHostToDevice, b->stream));
  BCK(cudaStreamSynchronize(b->stream));
  return DAMPM_OK;
}

int dampm_batch_compact(dampm_batch* b) {
  if (!b) return DAMPM_ERR_ARG;
  bool any_dead = false;
  for (const HostScn& h : b->scns) any_dead |= !h.d.live;
  if (!any_dead) return DAMPM_OK;
  int rc = read_scalars(b);
  if (rc) return rc;
  std::vector<HostScn> keep;
  std::vector<Scalars> S;
  std::vector<int4> mv, nm;
  long long P = 0, N = 0, C = 0, U = 0;
  int strips = 0, pieces = 0;
  for (size_t s = 0; s < b->scns.size(); ++s) {
    HostScn h = b->scns[s];
    if (!h.d.live) continue;
    const Scn old = h.d;
    h.d.p_off = int(P);
    h.d.n_off = int(N);
    h.d.c_off = int(C);
    h.d.piece_off = pieces;
    h.d.useg_off = int(U);
    for (int f = 0; f < old.np; f += kG2PThreads)
      mv.push_back(make_int4(h.d.p_off + f, old.p_off + f,
                             std::min(kG2PThreads, old.np - f), h.d.c_off - old.c_off));
    for (long long f = 0; f < h.nn; f += kG2PThreads)
      nm.push_back(make_int4(int(h.d.n_off + f), int(old.n_off + f),
                             int(std::min<long long>(kG2PThreads, h.nn - f)), 0));
    P += old.np;
    N += h.nn;
    C += h.nc;
    strips += old.nstrips;
    pieces += pieces_of(old);
    U += (long long)old.nstrips * (h.grid.Nex + 1);
    S.push_back(b->Sh[s]);
    // its cells move: the first plan after the move covers all of them
    S.back().krange[0] = 0x7fffffff;
    S.back().krange[1] = -1;
    S.back().knext[0] = h.d.c_off;
    S.back().knext[1] = h.d.c_off + int(h.nc) - 1;
    keep.push_back(h);
  }
  const int nxt = 1 - b->cur, znxt = 1 - b->zcur;
  // the counts of the moved keys, for the next sort (the whole array: cells
  // beyond the new total may hold counts of removed scenarios, which a later
  // scenario's cells would otherwise inherit)
  BCK(cudaMemsetAsync(b->count, 0, sizeof(int) * size_t(b->N_cap + 4), b->stream));
  BCK(cudaMemsetAsync(b->tile_sum, 0, sizeof(int) * kTileStride * size_t(b->N_cap / kScanTile + 2),
                      b->stream));
  if (!mv.empty()) {
    BCK(cudaMemcpyAsync(b->mblk, mv.data(), sizeof(int4) * mv.size(),
                        cudaMemcpyHostToDevice, b->stream));
    if (b->precision == DAMPM_FP32)
      launch_b_move<float>(int(mv.size()), b->stream, b->p32[nxt], b->p32[b->cur], b->mblk);
    else
      launch_b_move<double>(int(mv.size()), b->stream, b->p64[nxt], b->p64[b->cur],
                            b->mblk);
    const int* key = b->precision == DAMPM_FP32 ? b->p32[nxt].key : b->p64[nxt].key;
    int* slot = b->precision == DAMPM_FP32 ? b->p32[nxt].slot : b->p64[nxt].slot;
    k_count_n<<<grid_blocks(P, 256), 256, 0, b->stream>>>(key, b->count, b->tile_sum, slot, int(P));
  }
  if (!nm.empty()) {
    BCK(cudaMemcpyAsync(b->nmove, nm.data(), sizeof(int4) * nm.size(),
                        cudaMemcpyHostToDevice, b->stream));
    k_b_move_nodes<<<int(nm.size()), kG2PThreads, 0, b->stream>>>(b->Z[znxt], b->Z[b->zcur],
                                                                  b->nmove);
  }
  for (size_t s = 0; s < S.size(); ++s) b->Sh[s] = S[s];
  if (!S.empty())
    BCK(cudaMemcpyAsync(b->S, b->Sh, sizeof(Scalars) * S.size(), cudaMemcpyHostToDevice,
                        b->stream));
  BCK(cudaGetLastError());
  b->cur = nxt;
  b->zcur = znxt;
  b->scns = keep;
  b->P_tot = P;
  b->N_tot = N;
  b->C_tot = C;
  b->strips_tot = strips;
  b->pieces_tot = pieces;
  b->useg_tot = U;
  // every table entry anew, once the copies of the old ones have been made
  BCK(cudaStreamSynchronize(b->stream));
  b->nblk = 0;
  int2 piece, blk;
  for (size_t s = 0; s < keep.size(); ++s) append_tables(b, s, &piece, &blk);
  return upload_tables(b, make_int2(0, int(keep.size())), make_int2(0, pieces),
                       make_int2(0, b->nblk));
}

// Passes per graph: even, so that a replay ends on the half it began.
constexpr int kBatchGraphPasses = 16;

// The graph of kBatchGraphPasses passes from half h, captured after any
// change of layout (the launches' sizes and pointers depend only on the
// layout and on the half the passes start from; every other change lives in
// device memory).  Nothing runs.
int ensure_batch_graph(dampm_batch* b, int h) {
  if (!b->graph_dirty[h] && b->graph[h]) return DAMPM_OK;
  if (b->graph[h]) {
    cudaGraphExecDestroy(b->graph[h]);
    b->graph[h] = nullptr;
  }
  const int cur0 = b->cur;
  const long long l0 = b->launches;
  b->cur = h;
  BCK(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
  int rc = DAMPM_OK;
  for (int k = 0; k < kBatchGraphPasses && rc == DAMPM_OK; ++k) rc = enqueue_pass(b);
  if (rc == DAMPM_OK) rc = enqueue_end(b);
  b->launches = l0;
  b->cur = cur0;  // nothing ran
  cudaGraph_t g = nullptr;
  const cudaError_t e = cudaStreamEndCapture(b->stream, &g);
  if (rc) {
    if (g) cudaGraphDestroy(g);
    return rc;
  }
  if (e != cudaSuccess) return bfail(b, DAMPM_ERR_CUDA, cudaGetErrorString(e));
  const cudaError_t ei = cudaGraphInstantiate(&b->graph[h], g, 0);
  cudaGraphDestroy(g);
  if (ei != cudaSuccess) {
    b->graph[h] = nullptr;
    return bfail(b, DAMPM_ERR_CUDA, cudaGetErrorString(ei));
  }
  b->graph_dirty[h] = false;
  return DAMPM_OK;
}

int dampm_batch_step(dampm_batch* b, int nsteps) {
  if (!b || nsteps < 0) return DAMPM_ERR_ARG;
  if (b->scns.empty() || nsteps == 0) return DAMPM_OK;
  // no graph of our own inside the caller's capture
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  const bool graphs = b->use_graphs &&
                      cudaStreamIsCapturing(b->stream, &cs) == cudaSuccess &&
                      cs == cudaStreamCaptureStatusNone;
  int left = nsteps;
  if (graphs && left >= kBatchGraphPasses) {
    const int h = b->cur;
    int rc = ensure_batch_graph(b, h);
    if (rc) return rc;
    for (; left >= kBatchGraphPasses; left -= kBatchGraphPasses) {
      BCK(cudaGraphLaunch(b->graph[h], b->stream));
      b->launches += (long long)pass_launches(b) * kBatchGraphPasses + 1;
    }
  }
  const bool plain = left > 0;
  for (; left > 0; --left) {
    int rc = enqueue_pass(b);
    if (rc) return rc;
  }
  if (plain) {  // (a graph ends its last pass itself)
    int rc = enqueue_end(b);
    if (rc) return rc;
  }
  // the graph the next call starts from, captured now rather than inside it
  if (graphs) return ensure_batch_graph(b, b->cur);
  return DAMPM_OK;
}

int dampm_batch_tune(dampm_batch* b, int units_per_cta, int col_weight, int use_graphs) {
  if (!b || units_per_cta < 0 || col_weight < 0 || use_graphs < -1) return DAMPM_ERR_ARG;
  if (units_per_cta > 0) b->units_per_cta = units_per_cta;
  if (col_weight > 0) b->col_weight = col_weight;
  if (use_graphs >= 0) b->use_graphs = use_graphs;
  b->graph_dirty[0] = b->graph_dirty[1] = true;
  return DAMPM_OK;
}

int dampm_batch_sync(dampm_batch* b) {
  if (!b) return DAMPM_ERR_ARG;
  int rc = read_scalars(b);
  if (rc) return rc;
  for (size_t s = 0; s < b->scns.size(); ++s)
    if (b->scns[s].d.live && b->Sh[s].status)
      return bfail(b, DAMPM_ERR_DEVICE,
                   "a scenario's state diverged (non-finite or negative) and was stopped");
  return DAMPM_OK;
}

int dampm_batch_query(dampm_batch* b, int handle, int* it, double* t, double* dt_last,
                      int* running, long long* np) {
  if (!b) return DAMPM_ERR_ARG;
  const int s = find(b, handle);
  if (s < 0) return bfail(b, DAMPM_ERR_ARG, "unknown scenario handle");
  int rc = read_scalars(b);
  if (rc) return rc;
  const Scalars& S = b->Sh[s];
  const Phys& P = b->scns[s].d.P;
  if (it) *it = S.it;
  if (t) *t = S.t;
  if (dt_last) *dt_last = S.dt;
  // the loop condition of the next pass (main/optim_par.cpp:281)
  if (running) *running = (S.status == 0) && (P.fixed ? (S.it < P.NSTEPS) : (S.t < P.T));
  if (np) *np = b->scns[s].d.np;
  return S.status ? bfail(b, DAMPM_ERR_DEVICE, "device status word set") : DAMPM_OK;
}

int dampm_batch_download(dampm_batch* b, int handle, const char* field, double* out) {
  if (!b || !field || !out) return DAMPM_ERR_ARG;
  const int s = find(b, handle);
  if (s < 0) return bfail(b, DAMPM_ERR_ARG, "unknown scenario handle");
  const std::string f(field);
  return b->precision == DAMPM_FP32 ? download_field<float>(b, b->scns[s].d, f, out)
                                    : download_field<double>(b, b->scns[s].d, f, out);
}

int dampm_batch_ledgers(dampm_batch* b, int handle, double out[9]) {
  if (!b || !out) return DAMPM_ERR_ARG;
  const int s = find(b, handle);
  if (s < 0) return bfail(b, DAMPM_ERR_ARG, "unknown scenario handle");
  int rc = read_scalars(b);
  if (rc) return rc;
  for (int k = 0; k < 9; ++k) out[k] = b->Sh[s].ledger[k];
  return DAMPM_OK;
}

int dampm_batch_states(dampm_batch* b, int cap, int* handles, int* running, int* its,
                       double* ts, int* count) {
  if (!b || !count || cap < 0 || (cap > 0 && (!handles || !running || !its || !ts)))
    return DAMPM_ERR_ARG;
  int rc = read_scalars(b);
  if (rc) return rc;
  int n = 0;
  for (size_t s = 0; s < b->scns.size(); ++s) {
    const HostScn& h = b->scns[s];
    if (!h.d.live) continue;
    if (n >= cap) return bfail(b, DAMPM_ERR_ARG, "state arrays shorter than the live count");
    const Scalars& S = b->Sh[s];
    const Phys& P = h.d.P;
    handles[n] = h.handle;
    // a scenario stopped by its status word reports -1; the others go on
    running[n] = S.status ? -1 : (P.fixed ? (S.it < P.NSTEPS) : (S.t < P.T)) ? 1 : 0;
    its[n] = S.it;
    ts[n] = S.t;
    ++n;
  }
  *count = n;
  return DAMPM_OK;
}

int dampm_batch_usage(dampm_batch* b, long long out[8]) {
  if (!b || !out) return DAMPM_ERR_ARG;
  long long live = 0, dead = 0;
  for (const HostScn& h : b->scns) (h.d.live ? live : dead) += 1;
  out[0] = live;
  out[1] = dead;
  out[2] = b->P_tot;
  out[3] = b->P_cap;
  out[4] = b->N_tot;
  out[5] = b->N_cap;
  out[6] = b->S_cap;
  out[7] = b->launches;
  return DAMPM_OK;
}

}  // extern "C"
