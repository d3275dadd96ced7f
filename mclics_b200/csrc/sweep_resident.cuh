// Resident sweep: small bulk and slab lattices swept entirely in shared memory, any number of sweeps in one launch.
//
// A 32^3 lattice is 393 KB: the colour passes (sweep_pass.cuh) give it 10-32 work items, and a sweep costs three
// dependent launches whose chains of plane loads leave the chip idle (13-28 us for a measured sweep of 32^3 by plan, of
// which under 1 us is work). Here one thread-block cluster holds a replica: CTA c of C keeps the planes
// [c nz / C, (c + 1) nz / C) and a copy of the two planes next to them, and all sweeps of a call run without leaving
// the kernel. Per colour, a task is the same pair of sites (x, x + 2) with the same draws and the same site_update as
// in the colour passes, so directors, acceptances and amplitudes are the same bits. Its sites of the first or last
// owned plane are also stored into the neighbouring CTA's copy (distributed shared memory); one cluster barrier then
// ends the colour. Replicas do not wait for one another.
//
// Bound by the instruction issue of the C <= 16 SMs a replica occupies (1.45 us per colour for one LL pair per thread)
// and by the latency of one task and one cluster barrier (1.6 us per colour at least). LL 32^3 per sweep of a long call:
// 6.6 us, measured 6.7 (three launches on the best colour-pass plan, replayed from graphs: 10.8, 12.7); 32 such replicas
// 13.0, 14.2 (24.4, 27.5). resident_choose (sweep_fused.cu) has both sides over the sizes. Counters: 332 (measured 384)
// instructions per site update at 40-46 % issue of the 16 SMs it runs on.
//
// Planes in shared memory: [plane][component][y][x parity][cell], cells of a half-row as in HBM (common.cuh) with two
// cells of padding left and right, which hold the periodic x ghosts; periodic y is an address, periodic z the copies.
// There is no wait in this kernel other than the cluster barrier, whose CTAs are scheduled together.
#pragma once
#include <cuda_runtime.h>

#include "common.cuh"
#include "physics.cuh"
#include "site_access.cuh"
#include "sweep_draws.cuh"

namespace mcl {

constexpr int kResThreads = 512, kResWarps = kResThreads / 32, kResMaxC = 16;
// shared memory ahead of the planes: accepted rotations per warp of the cluster, observables per warp, and per CTA
constexpr int kResAcc = kResMaxC * kResWarps * 4, kResRed = kResWarps * kPartials * 8, kResMail = kResMaxC * kPartials * 8;
constexpr int kResMaxSmem = 227 * 1024;
constexpr int kResHead = kResAcc + kResRed + kResMail;
static_assert(kResHead % 16 == 0, "the planes are 16-byte aligned");

// Half-row pitch in shared memory and pairs per half-row of a lattice nx wide.
__host__ __device__ constexpr int res_pairs(int nx) { return ((nx + 1) / 2 + 1) / 2; }
__host__ __device__ constexpr int res_pitch(int nx) { return 2 * res_pairs(nx) + 4; }
// Floats of one plane.
__host__ __device__ constexpr int res_plane(int nx, int ny) { return 3 * ny * 2 * res_pitch(nx); }

struct ResidentArgs {
  const RepDesc *reps;
  RepState *st;
  float *dir;  // directors in HBM, read at the start and written at the end with their ghost copies
  unsigned long long *sweep_ctr;
  ObsRecord *series;
  int *series_len;
  unsigned int *done;
  int n_sweeps, measure, n_rep, adapt;
};

struct ResidentLaunch {
  int geo, clusters, cluster_size;
  bool flip, pxy, chiral, field;
  size_t smem;
  cudaStream_t stream;
  bool prepare = false;         // only set the kernel's limits
  int *max_clusters = nullptr;  // not null: only query how many clusters run at once on the device
};

cudaError_t launch_resident_ll(const ModelDev &m, const ResidentArgs &a, const ResidentLaunch &l);
cudaError_t launch_resident_ghrl(const ModelDev &m, const ResidentArgs &a, const ResidentLaunch &l);
cudaError_t launch_resident_ghrl_chiral(const ModelDev &m, const ResidentArgs &a, const ResidentLaunch &l);
cudaError_t launch_resident_pear(const ModelDev &m, const ResidentArgs &a, const ResidentLaunch &l);

#ifdef __CUDACC__
__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned cluster_ctas() {
  unsigned r;
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  __syncwarp();  // the aligned forms want the warp together
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ unsigned cluster_addr(unsigned smem_addr, unsigned rank) {
  unsigned r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_cluster(unsigned addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ void st_cluster(unsigned addr, float2 v) {
  asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(v.x), "f"(v.y) : "memory");
}
__device__ __forceinline__ void st_cluster(unsigned addr, unsigned v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void st_cluster(unsigned addr, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}

template <int POT, bool SLAB, bool FLIP, bool PXY, bool CHIRAL, bool FIELD>
__global__ void __launch_bounds__(kResThreads, 1) k_sweep_resident(ModelDev m, ResidentArgs a) {
  extern __shared__ __align__(16) unsigned char res_smem[];
  unsigned *s_acc = reinterpret_cast<unsigned *>(res_smem);
  double(*s_red)[kPartials] = reinterpret_cast<double(*)[kPartials]>(res_smem + kResAcc);
  double(*s_mail)[kPartials] = reinterpret_cast<double(*)[kPartials]>(res_smem + kResAcc + kResRed);
  float *planes = reinterpret_cast<float *>(res_smem + kResHead);
  const unsigned smem0 = (unsigned)__cvta_generic_to_shared(res_smem);
  const int rank = (int)cluster_rank(), C = (int)cluster_ctas();
  const int rep = (int)blockIdx.x / C;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const RepDesc R = a.reps[rep];
  const RepState S = a.st[rep];
  const int nx = R.nx, ny = R.ny, nz = R.nz;
  const bool perx = PXY || R.periodic[0], pery = PXY || R.periodic[1], perz = R.periodic[2];
  const int NP = res_pairs(nx), hps = res_pitch(nx), plane = res_plane(nx, ny), PF = ny * 2 * hps;
  auto first_plane = [&](int r) { return (int)((long long)r * nz / C); };
  const int z0 = first_plane(rank), nzl = first_plane(rank + 1) - z0;
  const int rank_dn = rank == 0 ? C - 1 : rank - 1, rank_up = rank == C - 1 ? 0 : rank + 1;
  const int dn_halo = first_plane(rank_dn + 1) - first_plane(rank_dn) + 1;  // its copy of the plane above its own
  const unsigned long long seed = R.seed, sweep0 = *a.sweep_ctr;
  const int row0 = *a.series_len;
  const float T = S.T, invT = 1.f / S.T, elecE = S.elecE;
  float av = S.ang_var;
  const unsigned long long n_valid = (unsigned long long)nx * ny * nz;
  const float *gdir = a.dir + R.off;
  const long long gplane = (long long)R.py * R.px;

  // the owned planes and their neighbours, ghost cells included (cells of an absent plane are read with weight 0)
  const int pairs_in_row = hps / 2, n2 = (nzl + 2) * (plane / 2);
  constexpr int kBatch = 8;  // loads in flight per thread: one at a time, the 15-40 rounds took 10-25 us of every call
  for (int e0 = tid; e0 < n2; e0 += kBatch * kResThreads) {
    float2 v[kBatch];
#pragma unroll
    for (int i = 0; i < kBatch; i++) {
      const int e = e0 + i * kResThreads;
      v[i] = make_float2(0.f, 0.f);
      if (e < n2) {
        const int rowh = e / pairs_in_row, jj = e - rowh * pairs_in_row;  // [plane][component][y][parity], cell pair
        const int lp = rowh / (6 * ny), in = rowh - lp * 6 * ny;
        const int q = in / (2 * ny), yh = in - q * 2 * ny;
        int z = z0 + lp - 1;
        if (perz) z = z < 0 ? z + nz : (z >= nz ? z - nz : z);
        if (z >= 0 && z < nz)
          v[i] = *reinterpret_cast<const float2 *>(gdir + q * R.comp + z * gplane + (long long)((yh >> 1) + GY) * R.px +
                                                   (yh & 1) * R.hp + GH - 2 + 2 * jj);
      }
    }
#pragma unroll
    for (int i = 0; i < kBatch; i++)
      if (e0 + i * kResThreads < n2) reinterpret_cast<float2 *>(planes)[e0 + i * kResThreads] = v[i];
  }
  cluster_sync();

  const unsigned tasks = (unsigned)(nzl * ny * NP);
  // t / d as the high word of t * ceil(2^32 / d): exact for t d < 2^32 (t below 2^20, d below 2^12 here)
  const unsigned mNP = 0xFFFFFFFFu / (unsigned)NP + 1u, mNy = 0xFFFFFFFFu / (unsigned)ny + 1u;
  auto div_by = [](unsigned t, unsigned magic) { return magic ? __umulhi(t, magic) : t; };  // magic 0: d = 1
  const int yhalf = (ny + 1) >> 1;
  const int half = nx >> 1;

  unsigned nacc = 0;
  auto write_record = [&](int s) {  // warp 0 of CTA 0: the observables of sweep s, whose sums have arrived
    double v = 0.0;
    if (lane < kPartials)
      for (int c = 0; c < C; c++) v += s_mail[c][lane];
    ObsRecord *o = a.series + (long long)(row0 + s) * a.n_rep + rep;
    const double nv = (double)n_valid;
    if (lane == 0) o->energy = v / nv;
    else if (lane <= 6) o->q[lane - 1] = v / nv;
    else if (lane < kPartials) o->nsum[lane - 7] = v;
    else if (lane == 10) o->n_valid = nv;
    else if (lane == 11) o->acceptance = (double)nacc / nv;
    else if (lane == 12) o->ang_var = av;
    else if (lane == 13) o->sweep = (double)(sweep0 + (unsigned long long)s);
  };

  for (int s = 0; s < a.n_sweeps; s++) {
    const unsigned long long sweep = sweep0 + (unsigned long long)s;
    unsigned accepted = 0;
    int n_meas = 0;
    float facc[kPartials];
#pragma unroll
    for (int k = 0; k < kPartials; k++) facc[k] = 0.f;
#pragma unroll 1
    for (int colour = 0; colour < 2; colour++) {
      const bool meas = a.measure && colour == 1;
#pragma unroll 1
      for (unsigned t = tid; t < tasks; t += kResThreads) {
        // rows of one parity together, so that a warp's sites mostly have one x parity
        const unsigned row = div_by(t, mNP), p = t - row * NP;
        const unsigned zl = div_by(row, mNy);
        const int yi = (int)(row - zl * ny);
        const int y = yi < yhalf ? 2 * yi : 2 * (yi - yhalf) + 1, z = z0 + (int)zl;
        const int h = (colour + y + z) & 1;
        const int in_plane = y * 2 * hps + 2 + 2 * (int)p;  // parity 0, cell of the pair's first site
        float *pl = planes + (zl + 1) * plane + in_plane;
        float *own = pl + h * hps;
        const float *oc = pl + (h ^ 1) * hps;
        const int xb = 4 * (int)p;
        const bool v0 = xb + h < nx, v1 = xb + h + 2 < nx;
        const bool c0 = xb + (h ^ 1) < nx, c1 = xb + (h ^ 1) + 2 < nx;
        float2 pn[3];
#pragma unroll
        for (int q = 0; q < 3; q++) pn[q] = *reinterpret_cast<const float2 *>(oc + q * PF);
        int sid = -1;
        float sz = 0.f;
        if (SLAB) sid = slab_surface(z, nz, sz);
        const Vec3 sn{0.f, 0.f, sz};
        SiteResultT<float2> res;
        float2 fin[3];
        if (v0) {
          const int ypo = y + 1 < ny ? 2 * hps : (pery ? -(ny - 1) * 2 * hps : 0);
          const int ymo = y > 0 ? -2 * hps : (pery ? (ny - 1) * 2 * hps : 0);
          float2 o[3], yu[3], yd[3], pu[3], pd[3];
          float sx[3];
          const float *ocx = oc + (h ? 2 : -1);
#pragma unroll
          for (int q = 0; q < 3; q++) {
            o[q] = *reinterpret_cast<const float2 *>(own + q * PF);
            yu[q] = *reinterpret_cast<const float2 *>(own + q * PF + ypo);
            yd[q] = *reinterpret_cast<const float2 *>(own + q * PF + ymo);
            pu[q] = *reinterpret_cast<const float2 *>(own + q * PF + plane);
            pd[q] = *reinterpret_cast<const float2 *>(own + q * PF - plane);
            sx[q] = ocx[q * PF];
          }
          const unsigned ctr = (unsigned)(xb + h) + (unsigned)nx * ((unsigned)y + (unsigned)ny * (unsigned)z);
          const LaneDraw<float2> ld = pair_draws<FLIP>(seed, sweep, ctr);
          const V3<float2> n{o[0], o[1], o[2]};
          V3<float2> nbp, nbm;
          nbp.x = h ? make_float2(pn[0].y, sx[0]) : pn[0];
          nbp.y = h ? make_float2(pn[1].y, sx[1]) : pn[1];
          nbp.z = h ? make_float2(pn[2].y, sx[2]) : pn[2];
          nbm.x = h ? pn[0] : make_float2(sx[0], pn[0].x);
          nbm.y = h ? pn[1] : make_float2(sx[1], pn[1].x);
          nbm.z = h ? pn[2] : make_float2(sx[2], pn[2].x);
          const V3<float2> nb[6] = {nbp, nbm, V3<float2>{yu[0], yu[1], yu[2]}, V3<float2>{yd[0], yd[1], yd[2]},
                                    V3<float2>{pu[0], pu[1], pu[2]}, V3<float2>{pd[0], pd[1], pd[2]}};
          float2 w[6];
          if (PXY) {
            w[0] = w[1] = w[2] = w[3] = make_float2(1.f, 1.f);
          } else {
            const int x = xb + h;
            w[0] = make_float2((perx || x + 1 < nx) ? 1.f : 0.f, (perx || x + 3 < nx) ? 1.f : 0.f);
            w[1] = make_float2((perx || x - 1 >= 0) ? 1.f : 0.f, 1.f);
            const float wp = (pery || y + 1 < ny) ? 1.f : 0.f, wm = (pery || y > 0) ? 1.f : 0.f;
            w[2] = make_float2(wp, wp);
            w[3] = make_float2(wm, wm);
          }
          const float wu = (perz || z + 1 < nz) ? 1.f : 0.f, wd = (perz || z > 0) ? 1.f : 0.f;
          w[4] = make_float2(wu, wu);
          w[5] = make_float2(wd, wd);
          constexpr int PRES = PXY ? kPresentXY : 0;
          if (SLAB || FIELD || POT != POT_LL || meas)
            res = site_update<POT, FLIP, PRES, CHIRAL, FIELD, float2, SLAB || FIELD>(m, n, nb, w, sid, sn, elecE, ld, av,
                                                                                      T, invT);
          else  // the difference as the unmeasured colour pass rounds it
            res = site_update<POT, FLIP, PRES, CHIRAL, FIELD, float2, false, true>(m, n, nb, w, sid, sn, elecE, ld, av, T,
                                                                                    invT);
          fin[0] = res.n.x;
          fin[1] = res.n.y;
          fin[2] = res.n.z;
          accepted += (res.rot.x ? 1u : 0u) + (v1 && res.rot.y ? 1u : 0u);
          if (v1) {
#pragma unroll
            for (int q = 0; q < 3; q++) *reinterpret_cast<float2 *>(own + q * PF) = fin[q];
          } else {
#pragma unroll
            for (int q = 0; q < 3; q++) own[q * PF] = fin[q].x;
          }
          if (perx) {  // ghost cells: the half-row's first site again at half index nx / 2, its last at -1
            const int jl = 2 * (int)p;
            if (p == 0) {
#pragma unroll
              for (int q = 0; q < 3; q++) own[q * PF + half] = fin[q].x;
            }
            if (jl == half - 1 || jl + 1 == half - 1) {
#pragma unroll
              for (int q = 0; q < 3; q++) own[q * PF - 1 - jl] = jl == half - 1 ? fin[q].x : fin[q].y;
            }
          }
          // the copies the neighbouring CTAs keep of this CTA's first and last plane
          const int cell = in_plane + h * hps;
          if (zl == 0 && (perz || z > 0)) {
            const unsigned dst = cluster_addr(smem0 + kResHead + 4u * (unsigned)(dn_halo * plane + cell), rank_dn);
#pragma unroll
            for (int q = 0; q < 3; q++) {
              if (v1) st_cluster(dst + 4u * (unsigned)(q * PF), fin[q]);
              else st_cluster(dst + 4u * (unsigned)(q * PF), fin[q].x);
            }
          }
          if ((int)zl == nzl - 1 && (perz || z + 1 < nz)) {
            const unsigned dst = cluster_addr(smem0 + kResHead + 4u * (unsigned)cell, rank_up);
#pragma unroll
            for (int q = 0; q < 3; q++) {
              if (v1) st_cluster(dst + 4u * (unsigned)(q * PF), fin[q]);
              else st_cluster(dst + 4u * (unsigned)(q * PF), fin[q].x);
            }
          }
        }
        if (meas) {  // the updated pair with 2 bond + single, the colour-0 pair of the same cells with its single terms
          float2 eb = make_float2(0.f, 0.f), va[3], vb[3];
#pragma unroll
          for (int q = 0; q < 3; q++) vb[q] = make_float2(0.f, 0.f);
          if (v0) {
            eb = __ffma2_rn(make_float2(2.f, 2.f), res.bond, res.single);
            if (!v1) eb.y = 0.f;
#pragma unroll
            for (int q = 0; q < 3; q++) vb[q] = make_float2(fin[q].x, v1 ? fin[q].y : 0.f);
          }
          if (SLAB || FIELD) {
            const float2 s0 = single_energy<FIELD>(m, V3<float2>{pn[0], pn[1], pn[2]}, sid, sn, elecE);
            eb.x += c0 ? s0.x : 0.f;
            eb.y += c1 ? s0.y : 0.f;
          }
#pragma unroll
          for (int q = 0; q < 3; q++) va[q] = make_float2(c0 ? pn[q].x : 0.f, c1 ? pn[q].y : 0.f);
          n_meas += (int)v0 + (int)v1 + (int)c0 + (int)c1;
          float2 f[kPartials];
          f[0] = eb;
          pair_moments(reinterpret_cast<float2(&)[9]>(f[1]), vb, va);
#pragma unroll
          for (int k = 0; k < kPartials; k++) facc[k] += f[k].x + f[k].y;
        }
      }
      if (colour == 1) {  // this warp's accepted rotations to every CTA, its observables to its own
        const unsigned wacc = __reduce_add_sync(0xffffffffu, accepted);
        if (lane < C) st_cluster(cluster_addr(smem0 + 4u * (unsigned)(rank * kResWarps + warp), lane), wacc);
        if (a.measure) {
          double dsum[kPartials], mine;
#pragma unroll
          for (int k = 0; k < kPartials; k++) dsum[k] = (double)facc[k] * (k >= 1 && k <= 6 ? 1.5 : 1.0);
          dsum[1] -= 0.5 * n_meas;
          dsum[4] -= 0.5 * n_meas;
          dsum[6] -= 0.5 * n_meas;
          const int k = warp_sum10(dsum, mine);
          if (k >= 0) s_red[warp][k] = mine;
        }
      }
      cluster_sync();
      // the sums of sweep s - 1 reached CTA 0 before this barrier (colour 0)
      if (colour == 0 && a.measure && s > 0 && rank == 0 && warp == 0) write_record(s - 1);
    }
    // every thread knows the cluster's count, and adapts the amplitude by the rule and arithmetic of k_finalize (its
    // comparison of the acceptance with 0.5, exact in integers)
    unsigned v = 0;
    for (int i = lane; i < C * kResWarps; i += 32) v += s_acc[i];
    nacc = __reduce_add_sync(0xffffffffu, v);
    if (a.adapt) {
      if (2ull * nacc < n_valid) {
        av = (float)((double)av * 0.99);
        if (av < 0.01) av = 0.01f;
      } else if (2ull * nacc > n_valid) {
        av = (float)((double)av / 0.99);
        if (av > 1.0) av -= 0.5f;
      }
    }
    if (a.measure && warp == 0 && lane < kPartials) {  // this CTA's sums to CTA 0 (read after the next barrier)
      double sum = 0.0;
      for (int w2 = 0; w2 < kResWarps; w2++) sum += s_red[w2][lane];
      st_cluster(cluster_addr(smem0 + kResAcc + kResRed + 8u * (unsigned)(rank * kPartials + lane), 0), sum);
    }
  }
  cluster_sync();
  if (a.measure && rank == 0 && warp == 0) write_record(a.n_sweeps - 1);

  // the owned planes back to HBM with the ghost copies of edge sites
  float *out = a.dir + R.off;
  const int cells = (nx + 1) >> 1;
  const int n1 = nzl * 6 * ny * cells;
  for (int e = tid; e < n1; e += kResThreads) {
    const int rowh = e / cells, j = e - rowh * cells;
    const int lp = rowh / (6 * ny), in = rowh - lp * 6 * ny;
    const int q = in / (2 * ny), yh = in - q * 2 * ny, y = yh >> 1, h = yh & 1;
    if (2 * j + h >= nx) continue;
    const float v = planes[(lp + 1) * plane + in * hps + 2 + j];
    float *g = out + q * R.comp + (z0 + lp) * gplane + (long long)(y + GY) * R.px + h * R.hp + GH;
    for (int iy = 0; iy < 3; iy++) {
      if (iy == 1 && !(pery && y < 2)) continue;
      if (iy == 2 && !(pery && y >= ny - 2)) continue;
      float *rowp = g + (long long)(iy == 0 ? 0 : (iy == 1 ? ny : -ny)) * R.px;
      rowp[j] = v;
      if (perx && j == 0) rowp[half] = v;
      if (perx && j == half - 1) rowp[-1] = v;
    }
  }
  if (rank == 0 && tid == 0) {
    a.st[rep].ang_var = av;
    a.st[rep].pad = (float)((double)nacc / (double)n_valid);
    __threadfence();
    const unsigned prev = atomicAdd(a.done, 1u);
    if (prev == (unsigned)a.n_rep - 1) {  // every replica has read both counters
      *a.done = 0u;
      *a.sweep_ctr = sweep0 + (unsigned long long)a.n_sweeps;
      if (a.measure) *a.series_len = row0 + a.n_sweeps;
      __threadfence();
    }
  }
}

template <int POT, bool SLAB, bool FLIP, bool PXY, bool CHIRAL, bool FIELD>
cudaError_t launch_resident_one(const ModelDev &m, const ResidentArgs &a, const ResidentLaunch &l) {
  auto k = k_sweep_resident<POT, SLAB, FLIP, PXY, CHIRAL, FIELD>;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(l.clusters * l.cluster_size));
  cfg.blockDim = dim3(kResThreads);
  cfg.dynamicSmemBytes = l.smem;
  cfg.stream = l.stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim = {(unsigned)l.cluster_size, 1, 1};
  cfg.attrs = at;
  cfg.numAttrs = 1;
  if (l.prepare) {
    // the same limit for every engine: a launch of another engine may need more than this one's
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kResMaxSmem);
    return e != cudaSuccess ? e : cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  }
  if (l.max_clusters) return cudaOccupancyMaxActiveClusters(l.max_clusters, k, &cfg);
  return cudaLaunchKernelEx(&cfg, k, m, a);
}

template <int POT, bool FLIP, bool CHIRAL, bool FIELD>
cudaError_t launch_resident_gp(const ModelDev &m, const ResidentArgs &a, const ResidentLaunch &l) {
  if (l.geo == GEO_SLAB)
    return l.pxy ? launch_resident_one<POT, true, FLIP, true, CHIRAL, FIELD>(m, a, l)
                 : launch_resident_one<POT, true, FLIP, false, CHIRAL, FIELD>(m, a, l);
  return l.pxy ? launch_resident_one<POT, false, FLIP, true, CHIRAL, FIELD>(m, a, l)
               : launch_resident_one<POT, false, FLIP, false, CHIRAL, FIELD>(m, a, l);
}
#endif

}  // namespace mcl
