// Tiled sweeps on TMA-streamed planes, host side (tensor maps, work items, tile configuration, launches): the fused
// two-colour kernel (sweep_fused.cuh) and the in-place colour passes (sweep_pass.cuh) share the work items, the
// per-item partials and the finalisation; the tile configuration selects the kernel.
#include <stdlib.h>

#include <algorithm>
#include <cmath>
#include <functional>
#include <map>
#include <mutex>
#include <vector>

#include "fused.h"
#include "sweep_pass.cuh"
#include "sweep_resident.cuh"

namespace mcl {

// 0, 1: fused (7 slots of TY + 4 rows: one CTA per SM either way); 2-4: colour passes (4 slots of TY + 2 rows; 3 has
// 2 CTAs per SM, for flip models; 4 has 32-wide tiles, for lattices whose width is not a multiple of 64).
static const FusedCfg kCfgs[kNumCfgs] = {{14, 256, 1, 0, 64}, {28, 512, 1, 0, 64}, {16, 256, 3, 1, 64},
                                         {16, 256, 2, 1, 64}, {16, 128, 5, 1, 32}};

struct FusedPlan {
  int cfg = 0, tx = 64, ty = 14, seg = 32;
  FusedCfg C{};              // the tile configuration (kCfgs[cfg], or the learned plan's own)
  bool learned = false;      // the learned colour passes' plan: its kernel sets its own shared-memory limit
  FusedPlan *lplan = nullptr;  // that plan, built at the first learned sweep
  int seg_override = 0;  // planes per z segment chosen by the autotuner (0: heuristic)
  int n_items = 0;
  FusedItem *d_items = nullptr;
  CUtensorMap *d_tmaps = nullptr;
  double *d_partials = nullptr;
  int *d_first = nullptr;  // first item of each replica (n_rep + 1)
  unsigned int *d_err = nullptr;
  size_t smem = 0;
  long long timeout_ns = 2000000000ll;
  int skip_first_load = 0;
  bool asked = false;          // a plan was asked for (mcl_set_plan, the autotuner, MCL_FUSED_CFG)
  int res_cluster = 0;         // CTAs per replica of the resident kernel (0: it is not used)
  size_t res_smem = 0;
  int res_calls = 1;           // sweeps a call needs for it
};

// ---- host side ----------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)p;
  }
  return fn;
}

bool fused_supported(const mcl_engine *e) {
  if (e->geo != GEO_BULK && e->geo != GEO_SLAB) return false;
  return get_encode() != nullptr;
}

// Box of `cells` half-row cells (TX / 2 + 8) and `rows` padded rows (fused: TY + 4, colour pass: TY + 2).
static int encode_map(CUtensorMap *map, float *base, const RepDesc &D, int cells, int rows) {
  // 5-D view of the split layout: (half-row cell, x parity, padded row, plane, component)
  cuuint64_t dims[5] = {(cuuint64_t)D.hp, 2, (cuuint64_t)D.py, (cuuint64_t)D.nz, 3};
  cuuint64_t strides[4] = {(cuuint64_t)D.hp * 4, (cuuint64_t)D.px * 4, (cuuint64_t)D.px * D.py * 4, (cuuint64_t)D.comp * 4};
  cuuint32_t box[5] = {(cuuint32_t)cells, 2, (cuuint32_t)rows, 1, 3};
  cuuint32_t es[5] = {1, 1, 1, 1, 1};
  CUresult r = get_encode()(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 5, base + D.off, dims, strides, box, es,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(MCL_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
  return MCL_OK;
}

#define CKF(call)                                        \
  do {                                                   \
    cudaError_t e_ = (call);                             \
    if (e_ != cudaSuccess) return cuda_fail(e_, #call);  \
  } while (0)

// Colour passes: what a plane costs a CTA, in us, by model (Lebwohl-Lasher, GHRL, chiral GHRL, models with flips) and
// configuration (2, 3, 4): `issue` times the CTAs that share an SM, but at least `chain`, the latency of one plane. From
// sweeps of lattices between 64^3 and 256^3 over all configurations and 2-24 planes per segment.
struct PassCost {
  double issue[3], chain[3];
};
static const PassCost kPassCost[4] = {{{0.76, 0.85, 0.43}, {1.05, 1.05, 1.00}},
                                      {{1.08, 1.02, 0.456}, {1.50, 1.46, 1.25}},
                                      {{1.20, 1.25, 0.62}, {1.60, 1.30, 1.05}},
                                      {{1.58, 1.40, 0.80}, {2.90, 2.08, 2.20}}};

static int pass_model(const mcl_engine *e) {
  if (e->model.flip != 0 || e->model.potential == POT_PEAR) return 3;
  if (e->model.potential == POT_GHRL) return e->model.sigma != 0.f ? 2 : 1;
  return 0;
}

static long long tiles_of(const mcl_engine *e, const FusedCfg &C) {
  long long tiles = 0;
  for (const auto &D : e->desc) tiles += (long long)((D.nx + C.tx - 1) / C.tx) * ((D.ny + C.ty - 1) / C.ty);
  return tiles;
}

// Expected time of one colour pass in us: 3.8 us of launch and first planes, then the planes of a segment for every wave
// of CTAs (the last wave counts half when it is not full: CTAs are handed out as they end).
static double pass_time(const mcl_engine *e, int cfg, int seg, int sms) {
  const FusedCfg &C = kCfgs[cfg];
  const PassCost &K = kPassCost[pass_model(e)];
  long long items = 0;
  for (const auto &D : e->desc)
    items += (long long)((D.nx + C.tx - 1) / C.tx) * ((D.ny + C.ty - 1) / C.ty) * ((D.nz + seg - 1) / seg);
  const double slots = (double)C.ctas_per_sm * sms, waves = items / slots;
  const double share = std::min<double>(C.ctas_per_sm, std::ceil((double)items / sms));
  const double plane = std::max(K.chain[cfg - 2], K.issue[cfg - 2] * share);
  return 3.8 + (waves <= 1 ? seg : (seg + 1.2) * std::max(waves, std::ceil(waves) - 0.5)) * plane;
}

// Segment choice for configuration `cfg`. Fused kernel and learned passes: segments sized so that the number of work
// items is close to a multiple of the resident CTAs, and long enough that the extra planes of each stay cheap (fused:
// four loaded, two of them computed; learned pass: two loaded). Colour passes: the shortest expected pass over 2-15
// planes. Per sweep in us, unmeasured / measured, with the work-item rule for both and configuration 2 (3 with flips)
// -> with the shortest pass over configurations too: LL 64^3 29.1 / 33.2 -> 16.8 / 18.9, LL 100^3 37.0 / 41.4 ->
// 31.9 / 35.5, GHRL slab 128^3 54.9 / 63.5 -> 46.5 / 52.8, 256^3 240 / 274 -> 215 / 240, chiral 101 x 75 x 50
// 35.2 / 39.4 -> 22.9 / 26.0, pear slab 64^3 41.3 / 45.5 -> 20.9 / 25.1.
static void choose_segments(const mcl_engine *e, FusedPlan &P, int sms) {
  const FusedCfg &C = P.C;
  P.tx = C.tx;
  P.ty = C.ty;
  long long maxz = 1;
  for (auto &D : e->desc) maxz = std::max<long long>(maxz, D.nz);
  if (C.kind == 1 && !P.learned) {
    P.seg = (int)std::min<long long>(2, maxz);
    for (int seg = 3; seg <= 15 && seg <= maxz; seg++)
      if (pass_time(e, P.cfg, seg, sms) < pass_time(e, P.cfg, P.seg, sms)) P.seg = seg;
  } else {
    const long long tiles = tiles_of(e, C), slots = (long long)C.ctas_per_sm * sms;
    int best = 1;
    double best_score = -1;
    for (int nseg = 1; nseg <= 256; nseg++) {
      const double seg_len = (double)maxz / nseg;
      if (seg_len < 6 && nseg > 1) break;
      const double waves = (double)(tiles * nseg) / slots;
      const double eff = waves / std::ceil(waves);
      const double extra = C.kind ? 2.0 * 0.15 : 4.0 * 0.35;  // extra planes mostly hit L2
      const double score = eff * seg_len / (seg_len + extra);
      if (score > best_score + 1e-9) {
        best_score = score;
        best = nseg;
      }
    }
    P.seg = (int)((maxz + best - 1) / best);
  }
  if (P.seg_override > 0) P.seg = (int)std::min<long long>(P.seg_override, maxz);
}

// The colour passes (faster than the fused kernel on every measured workload) in the configuration with the shortest
// expected pass.
static int choose_cfg(const mcl_engine *e) {
  const char *env = getenv("MCL_FUSED_CFG");
  if (env) return std::max(0, std::min(kNumCfgs - 1, atoi(env)));
  int sms = 148, best = 2;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, e->device);
  double best_time = 1e30;
  for (int cfg = 2; cfg < kNumCfgs; cfg++) {
    FusedPlan P;
    P.cfg = cfg;
    P.C = kCfgs[cfg];
    choose_segments(e, P, sms);
    const double t = pass_time(e, cfg, P.seg, sms);
    if (t < best_time) {
      best_time = t;
      best = cfg;
    }
  }
  return best;
}

static int prepare_kernel(mcl_engine *e, FusedPlan *P);
static void free_plan(FusedPlan *P);
static void resident_choose(const mcl_engine *e, FusedPlan *P);

// The fused plans read one director buffer and write the other; the colour passes and the learned passes update
// one buffer in place. The second buffer (211 MB for a 256^3 lattice) therefore exists only while a fused plan is
// selected: switching to an in-place plan brings the state into buffer 0 and frees buffer 1. The learned plan's
// tensor maps name the buffers, so it is rebuilt at the next learned sweep.
static int set_buffers(mcl_engine *e, FusedPlan *P) {
  const bool two = P->C.kind == 0;
  if (two == (e->d_dir[1] != nullptr)) return MCL_OK;
  CKF(cudaStreamSynchronize(e->stream));
  if (two) {
    CKF(cudaMalloc(&e->d_dir[1], (size_t)e->dir_floats * sizeof(float)));
    CKF(cudaMemsetAsync(e->d_dir[1], 0, (size_t)e->dir_floats * sizeof(float), e->stream));
  } else {
    if (e->cur == 1)
      CKF(cudaMemcpyAsync(e->d_dir[0], e->d_dir[1], (size_t)e->dir_floats * sizeof(float), cudaMemcpyDeviceToDevice,
                          e->stream));
    CKF(cudaStreamSynchronize(e->stream));
    CKF(cudaFree(e->d_dir[1]));
    e->d_dir[1] = nullptr;
    e->cur = 0;
  }
  if (P->lplan) {
    free_plan(P->lplan);
    delete P->lplan;
    P->lplan = nullptr;
  }
  return MCL_OK;
}

static int build_items(mcl_engine *e, FusedPlan *P) {
  if (!P->learned) {
    P->C = kCfgs[P->cfg];
    const int rc = set_buffers(e, P);
    if (rc) return rc;
  }
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, e->device);
  choose_segments(e, *P, sms);
  // maps of buffer 0 and buffer 1 per replica (buffer 0's twice while there is one buffer: the state is in buffer 0)
  std::vector<CUtensorMap> maps(2 * e->n_rep);
  for (int r = 0; r < e->n_rep; r++)
    for (int b = 0; b < 2; b++) {
      int rc = encode_map(&maps[2 * r + b], e->d_dir[e->d_dir[1] ? b : 0], e->desc[r], P->tx / 2 + 8,
                          P->ty + (P->C.kind ? 2 : 4));
      if (rc) return rc;
    }
  cudaFree(P->d_tmaps);
  cudaFree(P->d_items);
  cudaFree(P->d_first);
  cudaFree(P->d_partials);
  CKF(cudaMalloc(&P->d_tmaps, maps.size() * sizeof(CUtensorMap)));
  CKF(copy_in(e->stream, P->d_tmaps, maps.data(), maps.size() * sizeof(CUtensorMap)));
  std::vector<FusedItem> items;
  std::vector<int> first;
  for (int r = 0; r < e->n_rep; r++) {
    first.push_back((int)items.size());
    const RepDesc &D = e->desc[r];
    const int zlo = D.zslab ? 1 : 0, zhi = D.zslab ? D.nz - 1 : D.nz;  // a z-slab's halo planes are not swept
    for (int z0 = zlo; z0 < zhi; z0 += P->seg)
      for (int y0 = 0; y0 < D.ny; y0 += P->ty)
        for (int x0 = 0; x0 < D.nx; x0 += P->tx) items.push_back(FusedItem{r, x0, y0, z0, std::min(zhi, z0 + P->seg)});
  }
  first.push_back((int)items.size());
  P->n_items = (int)items.size();
  CKF(cudaMalloc(&P->d_items, items.size() * sizeof(FusedItem)));
  CKF(copy_in(e->stream, P->d_items, items.data(), items.size() * sizeof(FusedItem)));
  CKF(cudaMalloc(&P->d_first, first.size() * sizeof(int)));
  CKF(copy_in(e->stream, P->d_first, first.data(), first.size() * sizeof(int)));
  CKF(cudaMalloc(&P->d_partials, (size_t)P->n_items * kPartials * sizeof(double)));
  CKF(cudaStreamSynchronize(e->stream));
  const bool pass = P->C.kind == 1;
  const int nsl = pass ? NSLP : NSL;
  const size_t slot_floats = ((size_t)3 * (P->tx + 16) * (P->ty + (pass ? 2 : 4)) + 31) / 32 * 32;
  P->smem = 128 + (size_t)nsl * slot_floats * sizeof(float) + nsl * sizeof(unsigned long long);
  return P->learned ? MCL_OK : prepare_kernel(e, P);
}

int fused_create(mcl_engine *e) {
  FusedPlan *P = new FusedPlan();
  e->fused = P;
  P->cfg = choose_cfg(e);
  P->asked = getenv("MCL_FUSED_CFG") != nullptr;
  CKF(cudaMalloc(&P->d_err, sizeof(unsigned int)));
  CKF(cudaMemsetAsync(P->d_err, 0, sizeof(unsigned int), e->stream));
  const int rc = build_items(e, P);
  if (rc == MCL_OK) resident_choose(e, P);
  return rc;
}

// Selects a plan and rebuilds the work items, tensor maps and buffers for it; if that fails (an allocation), the
// previous plan is rebuilt, so the engine keeps a consistent plan, and the first error is returned.
static int apply_plan(mcl_engine *e, int cfg, int seg) {
  FusedPlan *P = e->fused;
  const int cfg0 = P->cfg, seg0 = P->seg_override;
  P->cfg = cfg;
  P->seg_override = seg;
  const int rc = build_items(e, P);
  if (rc == MCL_OK) return MCL_OK;
  P->cfg = cfg0;
  P->seg_override = seg0;
  build_items(e, P);
  return rc;
}

int fused_set_cfg(mcl_engine *e, int cfg) {
  if (!e->fused) return fail(MCL_ERR_STATE, "this engine does not use the fused tiled sweep");
  if (cfg < 0 || cfg >= kNumCfgs) return fail(MCL_ERR_ARG, "tile configuration %d outside 0..%d", cfg, kNumCfgs - 1);
  CKF(cudaStreamSynchronize(e->stream));
  e->fused->asked = true;
  return apply_plan(e, cfg, e->fused->seg_override);
}

int fused_set_plan(mcl_engine *e, int cfg, int seg) {
  if (!e->fused) return fail(MCL_ERR_STATE, "this engine does not use the fused tiled sweep");
  if (cfg < 0 || cfg >= kNumCfgs) return fail(MCL_ERR_ARG, "tile configuration %d outside 0..%d", cfg, kNumCfgs - 1);
  if (kCfgs[cfg].kind == 0 && e->zslab)
    return fail(MCL_ERR_STATE, "a z-slab engine runs the colour passes (tile configurations 2-%d)", kNumCfgs - 1);
  CKF(cudaStreamSynchronize(e->stream));
  e->fused->asked = true;
  return apply_plan(e, cfg, std::max(0, seg));
}

void fused_plan_candidates(const mcl_engine *e, std::vector<std::pair<int, int>> &out) {
  out.clear();
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, e->device);
  int maxz = 1;
  for (auto &D : e->desc) maxz = std::max(maxz, D.nz);
  for (int cfg = 0; cfg < kNumCfgs; cfg++) {
    FusedPlan P;
    P.cfg = cfg;
    P.C = kCfgs[cfg];
    choose_segments(e, P, sms);
    std::vector<int> segs = {P.seg, P.seg * 2, (P.seg + 1) / 2, maxz};
    // lattices too small to give every SM a work item (C1's 32^3: 10 items) also try short segments in the colour
    // passes, which trade two extra planes per item for more items in flight
    const long long tiles = tiles_of(e, P.C);
    const bool few = P.C.kind == 1 && tiles * ((maxz + P.seg - 1) / P.seg) < sms;
    if (few)
      for (int sg : {2, 3, 4}) segs.push_back(sg);
    std::sort(segs.begin(), segs.end());
    segs.erase(std::unique(segs.begin(), segs.end()), segs.end());
    for (int sg : segs)
      if (sg >= 6 || sg == P.seg || sg == maxz || (few && sg >= 2)) out.push_back({cfg, std::min(sg, maxz)});
  }
  std::sort(out.begin(), out.end());
  out.erase(std::unique(out.begin(), out.end()), out.end());
}

int fused_threads(int cfg) { return kCfgs[std::max(0, std::min(kNumCfgs - 1, cfg))].nt; }

int fused_get_cfg(const mcl_engine *e, int *cfg, int *ty, int *seg, int *items) {
  if (!e->fused) return fail(MCL_ERR_STATE, "this engine does not use the fused tiled sweep");
  if (cfg) *cfg = e->fused->cfg;
  if (ty) *ty = e->fused->ty;
  if (seg) *seg = e->fused->seg;
  if (items) *items = e->fused->n_items;
  return MCL_OK;
}

static void free_plan(FusedPlan *P) {
  cudaFree(P->d_items);
  cudaFree(P->d_tmaps);
  cudaFree(P->d_partials);
  cudaFree(P->d_first);
}

int fused_learned_view(mcl_engine *e, LearnedPassView *v) {
  FusedPlan *P = e->fused;
  if (!P) return fail(MCL_ERR_STATE, "the learned colour passes need the tiled sweep");
  if (!P->lplan) {
    FusedPlan *L = new FusedPlan();
    L->learned = true;
    L->C = FusedCfg{8, 256, 2, 1, 64};  // 64 x 8 tiles: 256 sites of a colour per plane, one tcgen05 batch
    L->cfg = -1;
    const int rc = build_items(e, L);
    if (rc) {
      free_plan(L);
      delete L;
      return rc;
    }
    P->lplan = L;
  }
  v->tmaps = P->lplan->d_tmaps;
  v->items = P->lplan->d_items;
  v->n_items = P->lplan->n_items;
  v->partials = P->lplan->d_partials;
  v->first = P->lplan->d_first;
  return MCL_OK;
}

void fused_destroy(mcl_engine *e) {
  FusedPlan *P = e->fused;
  if (!P) return;
  if (P->lplan) {
    free_plan(P->lplan);
    delete P->lplan;
  }
  cudaFree(P->d_items);
  cudaFree(P->d_tmaps);
  cudaFree(P->d_partials);
  cudaFree(P->d_first);
  cudaFree(P->d_err);
  delete P;
  e->fused = nullptr;
}

// ---- the resident kernel -------------------------------------------------------------------------------------
static ResidentLaunch resident_desc(const mcl_engine *e, int cluster, size_t smem) {
  ResidentLaunch l{};
  l.geo = e->geo;
  l.clusters = e->n_rep;
  l.cluster_size = cluster;
  l.flip = e->model.flip != 0 || e->model.potential == POT_PEAR;
  l.pxy = true;
  for (const auto &D : e->desc) l.pxy = l.pxy && D.periodic[0] && D.periodic[1];
  l.chiral = e->model.potential == POT_GHRL && e->model.sigma != 0.f;
  l.field = e->model.field_on != 0;
  l.smem = smem;
  l.stream = e->stream;
  return l;
}

static cudaError_t resident_dispatch(const mcl_engine *e, const ResidentArgs &a, const ResidentLaunch &l) {
  if (e->model.potential == POT_GHRL) return launch_resident_ghrl(e->model, a, l);
  if (e->model.potential == POT_PEAR) return launch_resident_pear(e->model, a, l);
  return launch_resident_ll(e->model, a, l);
}

// Clusters of C CTAs that run at once on the engine's device: a property of the device, since every resident kernel
// takes a whole SM per CTA (512 threads of 128 registers). The query takes about a millisecond, so its answers are kept.
static int clusters_that_fit(const mcl_engine *e, int C) {
  static std::mutex mu;
  static std::map<std::pair<int, int>, int> known;
  std::lock_guard<std::mutex> lock(mu);
  auto it = known.find({e->device, C});
  if (it != known.end()) return it->second;
  int fit = 0;
  ResidentLaunch l = resident_desc(e, C, kResMaxSmem);
  l.max_clusters = &fit;
  if (resident_dispatch(e, ResidentArgs{}, l) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  known[{e->device, C}] = fit;
  return fit;
}

// CTAs per replica of the resident kernel, or 0 where the colour passes are faster or a replica does not fit.
//
// Measured per sweep on one B200 (us, unmeasured / measured sweeps in long calls; colour passes on their best plan with
// graph replay; the resident kernel as chosen here where it is):
//                     resident, C = 4     C = 8          C = 16         chosen         colour passes
//   LL 16^3           3.6 / 4.5           3.2 / 4.0      3.5 / 4.2      3.6 / 4.4      10.5 / 12.8
//   LL 32^3           12.9 / 14.3         7.8 / 8.5      6.7 / 6.9      6.6 / 6.7      10.8 / 12.7
//   LL 48^3           does not fit        does not fit   12.8 / 13.6    -              12.0 / 14.9
//   GHRL 32^3         16.4 / 17.6         9.5 / 10.1     7.6 / 7.8      7.5 / 7.6      11.3 / 13.3
//   chiral 32^3       20.2 / 21.7         11.5 / 12.2    8.6 / 8.8      8.2 / 8.3      11.6 / 14.0
//   pear 48 x 48 x 24 41 / 45             23.6 / 25.4    18.0 / 19.7    -              16.4 / 20.8
//   LL 32 x 32^3      13.2 / 16.8         23.3 / 27.9    32.4 / 37.2    13.0 / 14.2    24.4 / 27.5
//   LL 64 x 24^3      15.1 / 18.4         25.4 / 30.2    44.2 / 74.9    12.9 / 13.8    38.6 / 41.8
//   LL 128 x 16^3     14.4 / 20.0         28.0 / 40.5    62.6 / 86.9    7.3 / 8.2      28.0 / 31.7
// A colour costs a chain of one task or the issue of the tasks of a full CTA, `round` us per 512, and a cluster barrier
// that grows with C; replicas beyond the clusters that fit the device (33, 15 and 7) wait for a free one.
static void resident_choose(const mcl_engine *e, FusedPlan *P) {
  P->res_cluster = 0;
  static const double kRound[4] = {1.45, 1.9, 2.4, 3.3};  // by pass_model
  const double round = kRound[pass_model(e)];
  int min_nz = 1 << 30, sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, e->device);
  for (const auto &D : e->desc) min_nz = std::min(min_nz, D.nz);
  if (P->C.kind != 1) return;
  // Setting the kernel's limits loads it, which takes milliseconds: not before a replica fits and could be faster.
  bool prepared = false;
  const double pass = 5.0 + 2.0 * pass_time(e, P->cfg, P->seg, sms);  // the finalisation and the gaps between launches
  double best = pass;
  for (int C = 1; C <= kResMaxC && C <= min_nz; C *= 2) {
    size_t smem = 0;
    for (const auto &D : e->desc)
      smem = std::max(smem, kResHead + ((size_t)(D.nz + C - 1) / C + 2) * res_plane(D.nx, D.ny) * sizeof(float));
    if (smem > kResMaxSmem) continue;
    auto alone = [&](const RepDesc &D) {  // one sweep of a replica
      const double tasks = std::ceil((double)D.nz / C) * D.ny * res_pairs(D.nx);
      return 2.0 * (std::max(0.8, round * tasks / kResThreads) + 0.4 + 0.08 * C);
    };
    double cost = 0;
    for (const auto &D : e->desc) cost = std::max(cost, alone(D));
    if (1.1 * cost + 3.0 >= best) continue;  // all replicas at once
    if (!prepared) {
      ResidentLaunch limits = resident_desc(e, 1, 0);
      limits.prepare = true;
      if (resident_dispatch(e, ResidentArgs{}, limits) != cudaSuccess) {
        cudaGetLastError();  // this combination of options has no kernel
        return;
      }
      prepared = true;
    }
    const int fit = clusters_that_fit(e, C);
    if (fit < 1) continue;
    // replicas in order onto the cluster that is free first
    std::vector<double> busy((size_t)std::min(fit, e->n_rep), 0.0);
    std::make_heap(busy.begin(), busy.end(), std::greater<double>());
    cost = 0;
    for (const auto &D : e->desc) {
      std::pop_heap(busy.begin(), busy.end(), std::greater<double>());
      busy.back() += alone(D);
      cost = std::max(cost, busy.back());
      std::push_heap(busy.begin(), busy.end(), std::greater<double>());
    }
    // Fewer clusters than the query says may run at once, so a margin per wave.
    const double gain = pass - cost, waves = std::ceil((double)e->n_rep / fit);
    cost = 1.1 * cost + 3.0 * waves;
    if (cost < best) {
      best = cost;
      P->res_cluster = C;
      P->res_smem = smem;
      // A call also reads and writes the lattice, for every wave of clusters: one sweep of 53 pear slabs of
      // 48 x 48 x 12 per call took 151 us against 97, of 24 LL 32^3 76 against 42, of LL 20^3 33 against 29, while 20
      // sweeps per call took 362 against 566 and 132 against 297.
      P->res_calls = (int)std::ceil((4.0 + 10.0 * waves) / std::max(gain, 0.1));
    }
  }
}

int fused_resident_calls(const mcl_engine *e) {
  const FusedPlan *P = e->fused;
  return P && P->res_cluster && !P->skip_first_load && !e->zslab && e->d_dir[1] == nullptr ? P->res_calls : 0;
}

bool fused_resident(const mcl_engine *e, int n) {
  const int calls = fused_resident_calls(e);
  return calls > 0 && n >= calls && !e->fused->asked;
}

void fused_release_plan(mcl_engine *e) { e->fused->asked = false; }

FusedChoice fused_choice(const mcl_engine *e) { return {e->fused->cfg, e->fused->seg_override, e->fused->asked}; }

int fused_restore(mcl_engine *e, const FusedChoice &c) {
  CKF(cudaStreamSynchronize(e->stream));
  e->fused->asked = c.asked;
  return apply_plan(e, c.cfg, c.seg_override);
}

int fused_resident_sweeps(mcl_engine *e, int n, bool measure) {
  FusedPlan *P = e->fused;
  ResidentArgs a;
  a.reps = e->d_desc;
  a.st = e->d_state;
  a.dir = e->d_dir[e->cur];
  a.sweep_ctr = e->d_sweep;
  a.series = e->d_series;
  a.series_len = e->d_series_len;
  a.done = e->d_done;
  a.n_sweeps = n;
  a.measure = measure ? 1 : 0;
  a.n_rep = e->n_rep;
  a.adapt = (e->adapt && !e->d_mlp) ? 1 : 0;
  CKF(resident_dispatch(e, a, resident_desc(e, P->res_cluster, P->res_smem)));
  e->launches += 1;
  return MCL_OK;
}

static FusedLaunch launch_desc(const mcl_engine *e, const FusedPlan *P) {
  FusedLaunch l;
  l.geo = e->geo;
  l.cfg = P->cfg;
  l.flip = e->model.flip != 0 || e->model.potential == POT_PEAR;
  l.pxy = true;
  for (const auto &D : e->desc) l.pxy = l.pxy && D.periodic[0] && D.periodic[1];
  l.chiral = e->model.potential == POT_GHRL && e->model.sigma != 0.f;
  l.field = e->model.field_on != 0;
  l.n_items = P->n_items;
  l.smem = P->smem;
  l.stream = e->stream;
  return l;
}

static cudaError_t dispatch(const mcl_engine *e, const FusedArgs &a, const FusedLaunch &l) {
  if (kCfgs[l.cfg].kind == 1) {
    if (e->model.potential == POT_GHRL) return launch_pass_ghrl(e->model, a, l);
    if (e->model.potential == POT_PEAR) return launch_pass_pear(e->model, a, l);
    return launch_pass_ll(e->model, a, l);
  }
  if (e->model.potential == POT_GHRL) return launch_fused_ghrl(e->model, a, l);
  if (e->model.potential == POT_PEAR) return launch_fused_pear(e->model, a, l);
  return launch_fused_ll(e->model, a, l);
}

// Sets the dynamic shared-memory limit of the kernel this plan launches (once per plan, so that launches inside a
// stream capture make no attribute calls).
static int prepare_kernel(mcl_engine *e, FusedPlan *P) {
  FusedLaunch l = launch_desc(e, P);
  l.prepare = true;
  FusedArgs a{};
  const cudaError_t err = dispatch(e, a, l);
  if (err != cudaSuccess) return cuda_fail(err, "fused sweep: shared-memory attribute");
  return MCL_OK;
}

int fused_launches_per_sweep(const mcl_engine *e) { return e->fused && kCfgs[e->fused->cfg].kind == 1 ? 3 : 2; }

int fused_sweep(mcl_engine *e, bool measure, cudaEvent_t ev0, cudaEvent_t ev1) {
  FusedPlan *P = e->fused;
  const bool pass = kCfgs[P->cfg].kind == 1;
  FusedArgs a;
  a.tmaps = P->d_tmaps;
  a.out = e->d_dir[pass ? e->cur : e->cur ^ 1];  // colour passes update in place
  a.reps = e->d_desc;
  a.st = e->d_state;
  a.items = P->d_items;
  a.partials = P->d_partials;
  a.sweep_ctr = e->d_sweep;
  a.err = P->d_err;
  a.cur = e->cur;
  a.measure = measure ? 1 : 0;
  a.timeout_ns = P->timeout_ns;
  a.skip_first_load = P->skip_first_load;
  a.colour = 0;
  if (ev0) CKF(cudaEventRecord(ev0, e->stream));
  const FusedLaunch l = launch_desc(e, P);
  if (pass) {  // colour 0 without measurement, then colour 1 with the observables of the whole lattice
    FusedArgs a0 = a;
    a0.measure = 0;
    cudaError_t err = dispatch(e, a0, l);
    if (err != cudaSuccess) return cuda_fail(err, "colour pass launch");
    a.colour = 1;
    err = dispatch(e, a, l);
    if (err != cudaSuccess) return cuda_fail(err, "colour pass launch");
  } else {
    const cudaError_t err = dispatch(e, a, l);
    if (err != cudaSuccess) return cuda_fail(err, "fused sweep launch");
    e->cur ^= 1;
  }
  if (ev1) CKF(cudaEventRecord(ev1, e->stream));
  e->launches += fused_launches_per_sweep(e);
  BlockTable t;
  t.first = P->d_first;
  LaunchCtx c = e->ctx();
  CKF(launch_finalize(c, t, P->d_partials, measure ? 1 : 0, e->d_series, e->d_series_len, e->d_done));
  return MCL_OK;
}

bool fused_is_pass_plan(const mcl_engine *e) { return e->fused && kCfgs[e->fused->cfg].kind == 1; }

int fused_pass(mcl_engine *e, int colour, bool measure) {
  FusedPlan *P = e->fused;
  if (!P || kCfgs[P->cfg].kind != 1) return fail(MCL_ERR_STATE, "single colour passes need a colour-pass plan");
  FusedArgs a;
  a.tmaps = P->d_tmaps;
  a.out = e->d_dir[e->cur];
  a.reps = e->d_desc;
  a.st = e->d_state;
  a.items = P->d_items;
  a.partials = P->d_partials;
  a.sweep_ctr = e->d_sweep;
  a.err = P->d_err;
  a.cur = e->cur;
  a.measure = measure && colour == 1 ? 1 : 0;
  a.timeout_ns = P->timeout_ns;
  a.skip_first_load = P->skip_first_load;
  a.colour = colour;
  const cudaError_t err = dispatch(e, a, launch_desc(e, P));
  if (err != cudaSuccess) return cuda_fail(err, "colour pass launch");
  e->launches += 1;
  return MCL_OK;
}

int fused_item_sums(mcl_engine *e, int measure, double *d_sums) {
  FusedPlan *P = e->fused;
  if (!P) return fail(MCL_ERR_STATE, "this engine does not use the tiled sweep");
  BlockTable t;
  t.first = P->d_first;
  CKF(launch_item_sums(e->ctx(), t, P->d_partials, measure, d_sums));
  e->launches += 1;
  return MCL_OK;
}

int fused_finalize_global(mcl_engine *e, const double *d_sums, int measure) {
  FusedPlan *P = e->fused;
  if (!P) return fail(MCL_ERR_STATE, "this engine does not use the tiled sweep");
  BlockTable t;
  t.first = P->d_first;
  CKF(launch_finalize(e->ctx(), t, P->d_partials, measure, e->d_series, e->d_series_len, e->d_done, d_sums));
  e->launches += 1;
  return MCL_OK;
}

int fused_check_error(mcl_engine *e) {
  if (!e->fused) return MCL_OK;
  unsigned int v = 0;
  CKF(cudaMemcpyAsync(&v, e->fused->d_err, sizeof v, cudaMemcpyDeviceToHost, e->stream));
  CKF(cudaStreamSynchronize(e->stream));
  return fused_report_error(e, v);
}

unsigned int *fused_error_word(mcl_engine *e) { return e->fused ? e->fused->d_err : nullptr; }

int fused_report_error(mcl_engine *e, unsigned int v) {
  if (!v || !e->fused) return MCL_OK;
  CKF(cudaMemsetAsync(e->fused->d_err, 0, sizeof v, e->stream));
  return fail(MCL_ERR_CUDA, "fused sweep: a TMA load did not complete within %.3f s (error word 0x%x)",
              e->fused->timeout_ns * 1e-9, v);
}

void fused_set_test_hooks(mcl_engine *e, long long timeout_ns, int skip_first_load) {
  if (!e->fused) return;
  if (timeout_ns > 0) e->fused->timeout_ns = timeout_ns;
  e->fused->skip_first_load = skip_first_load;
}

}  // namespace mcl
