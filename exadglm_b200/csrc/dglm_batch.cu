// Batched advection: many independent meshes of uneven size and polynomial
// order advance together, one persistent launch per LSERK stage.
//
// The reference runs one mesh per process (advec_nopad_time.cu:32-108).
// Here a batch owns the concatenated per-element arrays of all its
// instances and a tile list: (instance, first element, count, order) with
// E_N elements per tile, E_N chosen per order so that tiles carry similar
// work (Np (3Np + NFF) multiply-adds per element).  Every CTA of the stage
// kernel walks the tile list with a static stride and runs the device
// function compiled for the tile's order -- one launch covers every order.
// The list is sorted by order, largest first, so each CTA gets a similar mix.
//
// Operators with the symmetry of the reference tetrahedron (every symmetric
// node set's) run on batch_sym_kernel: tiles of 8 elements, a warp per tile,
// the symmetry-adapted advection tile of dglm_stage_sym_adv.cuh.  The tile
// list is sorted by order; each CTA takes one stretch of it, cut by cost, and
// loads an order's operator once per stretch.  Otherwise batch_stage_kernel:
//
// Per tile (advection, one variable): stage u and the tile's metrics and
// face data in shared memory; volume fluxes v u combined with the metrics;
// contraction with [WDr WDs WDt] on the FP64 tensor cores (m8n8k4, the
// operator's A fragments per order, as the single-mesh DMMA path builds
// them); face traces through vmapP and the DGLM flux; contraction with
// -LIFT into the same accumulators; LSERK update with the instance's dt.
//
// Per instance: velocity v (constant, the per-node velocity the reference
// takes reduces to it), tau from the face wave speed |v| (update_tau,
// advec_dglm.cpp), the CFL dt from a per-instance max of |v| Fscale
// (calc_dt), clipped to tmax, and the simulated time.  Steps are captured as
// CUDA graphs.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <utility>
#include <vector>

#include "dglm_common.cuh"
#include "dglm_handle.cuh"
#include "dglm_sym.cuh"

namespace dglm {

struct BatchTile {
  int inst, e0, ne, N;
};

struct BatchInst {
  long node_off;   // first node of the instance in the field arrays
  long elem_off;   // first element in the per-element arrays
  long fp_off;     // first face point in vmapP
  int K, N;
  double vx, vy, vz, tau;
};

struct BatchScalars {
  double t, dt_cfl, dt;           // time, CFL dt, dt of the step in flight
  unsigned long long acc;         // max |v| Fscale over the instance's faces (bits)
  int tstep, active;
};

struct BatchArgs {
  const BatchTile *tiles;
  int ntiles;
  const BatchInst *inst;
  BatchScalars *sc;
  const double *ops[kMaxOrder + 1];   // A fragments per order
  const int *Fmask[kMaxOrder + 1];
  const double *geo;     // [9][gs]
  const double *nrm;     // [3][4 gs]
  const double *fscale;  // [4 gs]
  long gs;
  const int *vmapP;      // instance-local node ids
  const double *u_in;
  double *u_out, *kreg;
  double rka, rkb;
};

constexpr int kBatchThreads = 256;
constexpr int kBatchWarps = kBatchThreads / 32;

template <int N>
struct BT {
  static constexpr int Np = np_of(N), Nfp = nfp_of(N), NFF = 4 * Nfp;
  static constexpr int E = N <= 3 ? 64 : N == 4 ? 32 : 16;
  static constexpr int EP = E + 1;
  static constexpr int MT = (Np + 7) / 8, NT = E / 8;
  static constexpr int KV = 3 * Np, KVP = (KV + 3) / 4 * 4;
  static constexpr int KF = NFF, KFP = (KF + 3) / 4 * 4;
  static constexpr int BROWS = KVP > KFP ? KVP : KFP;
  static constexpr int BLD = E + 4;                 // conflict-free B fragments
  static constexpr int PAIRS = MT * NT, WP = (PAIRS + kBatchWarps - 1) / kBatchWarps;
  static constexpr int VMLD = NFF + 1;
  static constexpr int S_U = Np * EP, S_B = BROWS * BLD, S_GEO = 9 * E, S_FACE = 4 * 4 * E;
  static constexpr size_t SMEM =
      sizeof(double) * (S_U + S_B + S_GEO + S_FACE) + sizeof(int) * ((size_t)E * VMLD + NFF);
  static_assert(S_B >= Np * EP, "epilogue reuses B");
  static constexpr int KSTEPS = KVP / 4 + KFP / 4;   // A fragment k-steps
};

// 8- and 4-byte asynchronous global -> shared copies (all of a tile's staging
// is issued before one wait)
__device__ __forceinline__ void b_cp8(void *dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                   (unsigned)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}
__device__ __forceinline__ void b_cp4(void *dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                   (unsigned)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}
__device__ __forceinline__ void b_cp_wait() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}

template <int N>
__device__ __forceinline__ void batch_tile(const BatchArgs &a, const BatchTile &t,
                                           double *smem) {
  using C = BT<N>;
  constexpr int Np = C::Np, Nfp = C::Nfp, NFF = C::NFF, E = C::E, EP = C::EP, BLD = C::BLD,
                T = kBatchThreads;
  double *sU = smem;                 // [i][EP]
  double *sB = sU + C::S_U;          // [k][BLD]
  double *sGeo = sB + C::S_B;        // [9][E]
  double *sFace = sGeo + C::S_GEO;   // [4][4][E]: nx ny nz fs
  int *sVm = reinterpret_cast<int *>(sFace + C::S_FACE);
  int *sFm = sVm + E * C::VMLD;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const BatchInst I = a.inst[t.inst];
  const int ne = t.ne;
  const long eg0 = I.elem_off + t.e0;                 // global element of the tile
  const long nb = I.node_off + (long)t.e0 * Np;       // first node of the tile
  const double *Afrag = a.ops[N];
  const double dt = a.sc[t.inst].dt;

  // this thread's RK register values for the update, fetched now so their
  // latency overlaps the tile's work
  constexpr int KPT = (E * Np + T - 1) / T;
  double kr[KPT];
#pragma unroll
  for (int q = 0; q < KPT; q++) {
    const int g = tid + q * T;
    kr[q] = g < ne * Np ? a.kreg[nb + g] : 0.0;
  }
  // staging: every copy is issued before one wait; padding is zero-filled
  for (int i = tid; i < NFF; i += T) b_cp4(sFm + i, a.Fmask[N] + i);
  for (int g = tid; g < E * Np; g += T) {
    const int e = g / Np, i = g - e * Np;
    if (g < ne * Np)
      b_cp8(sU + i * EP + e, a.u_in + nb + g);
    else
      sU[i * EP + e] = 0.0;
  }
  for (int g = tid; g < 9 * E; g += T) {
    const int m = g / E, e = g - m * E;
    if (e < ne)
      b_cp8(sGeo + g, a.geo + (long)m * a.gs + eg0 + e);
    else
      sGeo[g] = 0.0;
  }
  for (int g = tid; g < 4 * E; g += T) {
    const int e = g >> 2, f = g & 3;
    const long gf = (eg0 + e) * 4 + f;
    if (e < ne) {
      b_cp8(sFace + (0 * 4 + f) * E + e, a.nrm + gf);
      b_cp8(sFace + (1 * 4 + f) * E + e, a.nrm + 4 * a.gs + gf);
      b_cp8(sFace + (2 * 4 + f) * E + e, a.nrm + 8 * a.gs + gf);
      b_cp8(sFace + (3 * 4 + f) * E + e, a.fscale + gf);
    } else {
      for (int q = 0; q < 4; q++) sFace[(q * 4 + f) * E + e] = 0.0;
    }
  }
  const long fp0 = I.fp_off + (long)t.e0 * NFF;
  for (int g = tid; g < E * NFF; g += T) {
    const int e = g / NFF, fj = g - e * NFF;
    if (g < ne * NFF)
      b_cp4(sVm + e * C::VMLD + fj, a.vmapP + fp0 + g);
    else
      sVm[e * C::VMLD + fj] = 0;
  }
  b_cp_wait();
  __syncthreads();

  // volume fluxes -> B rows [0, 3Np)
  for (int it = tid; it < E * Np; it += T) {
    const int i = it / E, e = it - i * E;
    const double *g = sGeo + e;
    const double uu = sU[i * EP + e];
    const double F = I.vx * uu, G = I.vy * uu, W = I.vz * uu;
    sB[(0 * Np + i) * BLD + e] = g[0] * F + g[E] * G + g[2 * E] * W;
    sB[(1 * Np + i) * BLD + e] = g[3 * E] * F + g[4 * E] * G + g[5 * E] * W;
    sB[(2 * Np + i) * BLD + e] = g[6 * E] * F + g[7 * E] * G + g[8 * E] * W;
  }
  for (int g = tid; g < (C::KVP - C::KV) * BLD; g += T) sB[C::KV * BLD + g] = 0.0;
  __syncthreads();

  double acc[C::WP][2];
#pragma unroll
  for (int j = 0; j < C::WP; j++) acc[j][0] = acc[j][1] = 0.0;
#pragma unroll
  for (int j = 0; j < C::WP; j++) {
    const int p = warp + kBatchWarps * j;
    if (p < C::PAIRS) {
      const int mt = p % C::MT, nt = p / C::MT;
      const double *Ab = Afrag + (long)mt * 32 + lane;
      const double *Bb = sB + (lane & 3) * BLD + nt * 8 + (lane >> 2);
#pragma unroll 4
      for (int ks = 0; ks < C::KVP / 4; ks++)
        dmma_8x8x4(acc[j], __ldg(Ab + (long)ks * C::MT * 32), Bb[ks * 4 * BLD]);
    }
  }
  __syncthreads();

  // face traces and fluxes -> B rows [0, NFF)
  for (int it = tid; it < E * NFF; it += T) {
    const int fj = it / E, e = it - fj * E, f = fj / Nfp;
    if (e >= ne) {
      sB[fj * BLD + e] = 0.0;
      continue;
    }
    const double um = sU[sFm[fj] * EP + e];
    const double ub = 0.5 * (um + a.u_in[I.node_off + sVm[e * C::VMLD + fj]]);
    const double F = I.vx * ub, G = I.vy * ub, W = I.vz * ub;
    const double nd = sFace[(0 * 4 + f) * E + e] * F + sFace[(1 * 4 + f) * E + e] * G +
                      sFace[(2 * 4 + f) * E + e] * W;
    sB[fj * BLD + e] = (nd - I.tau * (ub - um)) * sFace[(3 * 4 + f) * E + e];
  }
  for (int g = tid; g < (C::KFP - C::KF) * BLD; g += T) sB[C::KF * BLD + g] = 0.0;
  __syncthreads();

#pragma unroll
  for (int j = 0; j < C::WP; j++) {
    const int p = warp + kBatchWarps * j;
    if (p < C::PAIRS) {
      const int mt = p % C::MT, nt = p / C::MT;
      const double *Ab = Afrag + ((long)(C::KVP / 4) * C::MT + mt) * 32 + lane;
      const double *Bb = sB + (lane & 3) * BLD + nt * 8 + (lane >> 2);
#pragma unroll 4
      for (int ks = 0; ks < C::KFP / 4; ks++)
        dmma_8x8x4(acc[j], __ldg(Ab + (long)ks * C::MT * 32), Bb[ks * 4 * BLD]);
    }
  }
  __syncthreads();

  // rhs -> sB as [i][EP], then the LSERK update with coalesced stores
  double *sR = sB;
#pragma unroll
  for (int j = 0; j < C::WP; j++) {
    const int p = warp + kBatchWarps * j;
    if (p < C::PAIRS) {
      const int mt = p % C::MT, nt = p / C::MT;
      const int i = mt * 8 + (lane >> 2);
      if (i < Np) {
#pragma unroll
        for (int h = 0; h < 2; h++) sR[i * EP + nt * 8 + (lane & 3) * 2 + h] = acc[j][h];
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < KPT; q++) {
    const int g = tid + q * T;
    if (g >= ne * Np) continue;
    const int e = g / Np, i = g - e * Np;
    const double kn = a.rka * kr[q] + dt * sR[i * EP + e];
    a.kreg[nb + g] = kn;
    a.u_out[nb + g] = sU[i * EP + e] + a.rkb * kn;
  }
}

template <int N>
constexpr size_t bt_smem() {
  return BT<N>::SMEM;
}
constexpr size_t cmax(size_t a, size_t b) { return a > b ? a : b; }
constexpr size_t kBatchSmem =
    cmax(cmax(cmax(bt_smem<2>(), bt_smem<3>()), cmax(bt_smem<4>(), bt_smem<5>())), bt_smem<6>());

__global__ void __launch_bounds__(kBatchThreads, 3) batch_stage_kernel(const BatchArgs a) {
  extern __shared__ __align__(16) double smem[];
  for (int ti = blockIdx.x; ti < a.ntiles; ti += gridDim.x) {
    const BatchTile t = a.tiles[ti];
    switch (t.N) {
      case 2: batch_tile<2>(a, t, smem); break;
      case 3: batch_tile<3>(a, t, smem); break;
      case 4: batch_tile<4>(a, t, smem); break;
      case 5: batch_tile<5>(a, t, smem); break;
      case 6: batch_tile<6>(a, t, smem); break;
      default: break;
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// symmetry-adapted path
// ---------------------------------------------------------------------------

struct BatchSymArgs {
  const BatchTile *tiles;     // sorted by order, largest first
  int begin[8];               // tiles of order N: [begin[N], begin[N - 1])
  const int *cut;             // gridDim.x + 1: the CTAs' stretches of the tile list
  const BatchInst *inst;
  const BatchScalars *sc;
  const double *image[kMaxOrder + 1];   // operator images per order
  const double *rec;          // per element: kSymRec flux weights
  const int *nb[kMaxOrder + 1];         // per tile of an order: neighbour nodes, lane order
  const double *u_in;
  double *u_out, *kreg;
  double rka, rkb;
  int *err;                   // set when a bounded wait expired
  long long wait_cycles;      // bound of the waits for a tile's state
};

// Per element: (grad r_a + sum_b grad r_b) . v (a = 1..3), Fscale n . v / 2 and
// Fscale tau / 2 of the four faces by label, one pad.
constexpr int kSymRec = 12;
constexpr int kSymWarps = 12;
// warps that take tiles of order N (N=6: the state buffers of eight leave L1
// room for the gathers)
template <int N>
constexpr int sym_warps() {
  return N == 6 ? 8 : kSymWarps;
}
template <int N>
using BSC = SymAdvCfg<N, sym_warps<N>()>;
constexpr size_t kBatchSymSmem =
    cmax(cmax(cmax(BSC<2>::SMEM, BSC<3>::SMEM), cmax(BSC<4>::SMEM, BSC<5>::SMEM)),
         BSC<6>::SMEM) + 16 * kSymWarps;
// Cost of a tile of order N (a single mesh's stage over its tiles, in ns), the
// weight by which the stretches are cut.
constexpr double kSymCost[7] = {0, 0, 1.6, 2.7, 4.2, 7.5, 13.9};

// Tiles [lo, hi) of order N by this CTA.  it: buffer uses of the warp so far.
template <int N>
__device__ __forceinline__ bool batch_sym_tiles(const BatchSymArgs &a, int lo, int hi,
                                                double *smem, unsigned long long *full,
                                                int &it) {
  using C = BSC<N>;
  constexpr int NW = sym_warps<N>(), Np = C::Np, P4 = 32 * C::KSF;
  double *sBuf = smem + C::S_A;
  int *tabs = reinterpret_cast<int *>(sBuf + NW * 2 * C::S_U);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const SymAdvOp op = sym_adv_operator<C>(a.image[N], smem, tabs, tid, 32 * kSymWarps);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncthreads();
  pdl_wait();
  bool ok = true;
  if (warp < NW && lo + warp < hi) {
    double *buf = sBuf + warp * 2 * C::S_U;
    auto fetch = [&](int ti, int b) {   // lane 0
      const BatchTile t = a.tiles[ti];
      mbar_arrive_expect_tx(&full[b], 8u * C::S_U);
      bulk_g2s(buf + b * C::S_U, a.u_in + a.inst[t.inst].node_off + (long)t.e0 * Np,
               8u * C::S_U, &full[b]);
    };
    if (lane == 0) fetch(lo + warp, it & 1);
    for (int ti = lo + warp; ti < hi; ti += NW, it++) {
      const int b = it & 1;
      const BatchTile t = a.tiles[ti];
      const BatchInst &I = a.inst[t.inst];
      const long node0 = I.node_off + (long)t.e0 * Np;
      double *u = buf + b * C::S_U;
      FlowConstant fl;
      double s[4];
      {
        // elements past the instance's last: zero weights on a zero state
        const int el = C::elem(lane >> 2);
        double2 q[kSymRec / 2];
#pragma unroll
        for (int i = 0; i < kSymRec / 2; i++)
          q[i] = el < t.ne ? __ldg(reinterpret_cast<const double2 *>(
                                 a.rec + (I.elem_off + t.e0 + el) * kSymRec) + i)
                           : make_double2(0.0, 0.0);
        fl.va[0] = q[0].x, fl.va[1] = q[0].y, fl.va[2] = q[1].x;
        fl.wf[0] = q[1].y, fl.wf[1] = q[2].x, fl.wf[2] = q[2].y, fl.wf[3] = q[3].x;
        s[0] = q[3].y, s[1] = q[4].x, s[2] = q[4].y, s[3] = q[5].x;
      }
      ok = sym_adv_tile<C>(
          op, u, fl,
          reinterpret_cast<const int4 *>(a.nb[N]) + (long)(ti - a.begin[N]) * P4 + lane,
          a.u_in + I.node_off, s, a.kreg + node0, a.sc[t.inst].dt, a.rka, a.rkb, a.rka != 0.0,
          false, lane,
          [&]() {
            return __all_sync(0xffffffffu, mbar_wait(&full[b], (it >> 1) & 1, a.wait_cycles)) != 0;
          },
          [&]() {
            // the next tile's state, once the previous tile's store has read its buffer
            if (lane == 0 && ti + NW < hi) {
              bulk_wait_read();
              fetch(ti + NW, b ^ 1);
            }
          });
      if (!ok) {
        if (lane == 0) *a.err = 1;
        mbar_wait(&full[b], (it >> 1) & 1);   // the tile in flight settles
        break;
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        bulk_s2g(a.u_out + node0, u, 8u * C::S_U);
        bulk_commit();
      }
    }
    if (lane == 0) bulk_wait_all();
  }
  // the shared memory of this stretch is free
  return __syncthreads_and(ok) != 0;
}

__global__ void __launch_bounds__(32 * kSymWarps, 1) batch_sym_kernel(const BatchSymArgs a) {
  extern __shared__ __align__(16) double smem[];
  pdl_launch();
  // the warps' barriers sit behind the largest order's layout
  unsigned long long *full = reinterpret_cast<unsigned long long *>(
      reinterpret_cast<char *>(smem) + kBatchSymSmem - 16 * kSymWarps) + 2 * (threadIdx.x >> 5);
  if ((threadIdx.x & 31) == 0) {
    mbar_init(&full[0], 1);
    mbar_init(&full[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  const int first = a.cut[blockIdx.x], last = a.cut[blockIdx.x + 1];
  if (first == last) pdl_wait();   // no tile: still after the launch before
  int it = 0;
  bool ok = true;
  auto stretch = [&](int N, int &lo, int &hi) {
    lo = max(first, a.begin[N]);
    hi = min(last, a.begin[N - 1]);
    return ok && lo < hi;
  };
  int lo, hi;
  if (stretch(6, lo, hi)) ok = batch_sym_tiles<6>(a, lo, hi, smem, full, it);
  if (stretch(5, lo, hi)) ok = batch_sym_tiles<5>(a, lo, hi, smem, full, it);
  if (stretch(4, lo, hi)) ok = batch_sym_tiles<4>(a, lo, hi, smem, full, it);
  if (stretch(3, lo, hi)) ok = batch_sym_tiles<3>(a, lo, hi, smem, full, it);
  if (stretch(2, lo, hi)) ok = batch_sym_tiles<2>(a, lo, hi, smem, full, it);
}

// Neighbour nodes of the tiles of order N in lane order (instance-local).
template <int N>
__global__ void batch_neighbour_kernel(const double *__restrict__ image,
                                       const BatchTile *__restrict__ tiles, int ntiles,
                                       const BatchInst *__restrict__ inst,
                                       const int *__restrict__ vmapP, int *__restrict__ nb) {
  using C = BSC<N>;
  constexpr int P4 = 32 * C::KSF;
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= (long)ntiles * P4) return;
  const int ti = (int)(i / P4), p = (int)(i % P4), f = p / 32, lane = p % 32;
  const BatchTile t = tiles[ti];
  const int el = C::elem(lane >> 2), j = min(f * 4 + (lane & 3), C::Nfp - 1);
  const int *tab = reinterpret_cast<const int *>(image + C::S_A) + C::T_VOL + j * 4;
  for (int v = 0; v < 4; v++)
    nb[i * 4 + v] = el < t.ne ? vmapP[inst[t.inst].fp_off + (long)(t.e0 + el) * C::NFF + (tab[v] >> 16)]
                              : 0;
}

// Flux weights of every element of every instance (blockIdx.y).
__global__ void batch_record_kernel(const BatchInst *__restrict__ inst,
                                    const int *const *__restrict__ labels,
                                    const double *__restrict__ geo,
                                    const double *__restrict__ nrm,
                                    const double *__restrict__ fscale, long gs,
                                    double *__restrict__ rec) {
  const BatchInst I = inst[blockIdx.y];
  const int *face_of = labels[I.N];
  const double v[3] = {I.vx, I.vy, I.vz};
  for (long k = blockIdx.x * (long)blockDim.x + threadIdx.x; k < I.K;
       k += (long)gridDim.x * blockDim.x) {
    const long e = I.elem_off + k;
    double *r = rec + e * kSymRec;
    for (int d = 0; d < 3; d++) {
      double x = 0.0;
      for (int q = 0; q < 3; q++)
        x += (geo[(3 * d + q) * gs + e] +
              (geo[q * gs + e] + geo[(3 + q) * gs + e] + geo[(6 + q) * gs + e])) * v[q];
      r[d] = x;
    }
    for (int l = 0; l < 4; l++) {
      const long f = 4 * e + face_of[l];
      double vn = 0.0;
      for (int q = 0; q < 3; q++) vn += nrm[4 * q * gs + f] * v[q];
      r[3 + l] = 0.5 * fscale[f] * vn;
      r[7 + l] = 0.5 * fscale[f] * I.tau;
    }
    r[11] = 0.0;
  }
}

// Per-instance max of |v| Fscale over its faces (calc_maxv + calc_dt of the
// reference with a frozen velocity), one block per instance.
__global__ void batch_wavespeed_kernel(const BatchInst *inst, const double *fscale,
                                       BatchScalars *sc) {
  const BatchInst I = inst[blockIdx.x];
  const double mv = sqrt(I.vx * I.vx + I.vy * I.vy + I.vz * I.vz);
  unsigned long long b = 0ull;
  for (long f = threadIdx.x; f < 4L * I.K; f += blockDim.x) {
    const unsigned long long x = dbits(mv * fscale[I.elem_off * 4 + f]);
    b = x > b ? x : b;
  }
  b = warp_max_bits(b);
  __shared__ unsigned long long s[32];
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = b;
  __syncthreads();
  if (threadIdx.x < 32) {
    b = threadIdx.x < blockDim.x / 32 ? s[threadIdx.x] : 0ull;
    b = warp_max_bits(b);
    if (threadIdx.x == 0) sc[blockIdx.x].acc = b;
  }
}

// dt of every instance for the coming step: CFL dt (euler_time.cpp:49-57 /
// advec_time.cpp), clipped so the instance ends at tmax; 0 once it has.
__global__ void batch_step_begin_kernel(int n, const BatchInst *inst, double cfl, double tmax,
                                        BatchScalars *sc) {
  pdl_launch();
  pdl_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double m = __longlong_as_double((long long)sc[i].acc);
  double dt = (cfl / (2 * inst[i].N + 1)) * (1 / m);
  const int active = sc[i].t < tmax;
  if (active && sc[i].t + dt > tmax) dt = tmax - sc[i].t;
  if (!active) dt = 0.0;
  sc[i].dt_cfl = (cfl / (2 * inst[i].N + 1)) * (1 / m);
  sc[i].dt = dt;
  sc[i].active = active;
}

__global__ void batch_step_end_kernel(int n, BatchScalars *sc) {
  pdl_launch();
  pdl_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || !sc[i].active) return;
  sc[i].t += sc[i].dt;
  sc[i].tstep += 1;
}

}  // namespace dglm

using namespace dglm;

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

struct BatchHostInst {
  int N, K;
  double v[3];
  std::vector<double> geo[9], nrm[3], fscale, u0;
  std::vector<int> vmapP;
};

struct dglm_batch {
  dglm_batch_desc d{};
  int dev = 0;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  std::vector<BatchHostInst> host;
  std::vector<double> Ahost[kMaxOrder + 1];   // stacked [WDr WDs WDt -LIFT] per order
  std::vector<int> Fm[kMaxOrder + 1];
  bool finalized = false;
  // device
  std::vector<void *> allocs;
  size_t bytes = 0;
  BatchArgs args{};
  BatchInst *inst = nullptr;
  BatchTile *tiles = nullptr;
  BatchScalars *sc = nullptr;
  double *u[2] = {nullptr, nullptr};
  int cur = 0, ntiles = 0, grid = 0;
  std::vector<BatchInst> hinst;
  bool sym = false;                 // all orders on the symmetry-adapted path
  BatchSymArgs sargs{};
  int *err = nullptr;
  std::atomic<int> expired{-1};     // *err after the last dglm_batch_step (-1: not read yet)
  long long wait_cycles = kWaitCycles;
  cudaGraphExec_t graph[2] = {nullptr, nullptr};
  long launches = 0;
};

namespace {



template <typename T>
dglm_status balloc(dglm_batch *b, T **p, size_t count) {
  void *q = nullptr;
  const size_t n = std::max<size_t>(count * sizeof(T), 16);
  cudaError_t e = cudaMalloc(&q, n);
  if (e != cudaSuccess) {
    *p = nullptr;
    return set_error(DGLM_ERR_NOMEM, std::string("dglm_batch: cudaMalloc failed: ") +
                                         cudaGetErrorString(e));
  }
  b->allocs.push_back(q);
  b->bytes += n;
  *p = static_cast<T *>(q);
  return DGLM_OK;
}

// m8n8k4 A fragments of [WDr WDs WDt | -LIFT] (as the single-mesh DMMA
// layout): [kstep][mtile][lane], row 8*mtile + lane/4, column 4*kstep +
// lane%4 of the volume block, then of the lift block.
template <int N>
std::vector<double> batch_fragments(const std::vector<double> &A) {
  using C = BT<N>;
  const int Np = C::Np, NFF = C::NFF, KA = 3 * Np + NFF, KV = 3 * Np;
  const int kv4 = C::KVP / 4, kf4 = C::KFP / 4;
  std::vector<double> out((size_t)(kv4 + kf4) * C::MT * 32, 0.0);
  for (int ks = 0; ks < kv4 + kf4; ks++)
    for (int mt = 0; mt < C::MT; mt++)
      for (int lane = 0; lane < 32; lane++) {
        const int row = mt * 8 + lane / 4;
        int k;
        bool ok;
        if (ks < kv4) {
          k = ks * 4 + lane % 4;
          ok = k < KV;
        } else {
          const int kk = (ks - kv4) * 4 + lane % 4;
          k = KV + kk;
          ok = kk < NFF;
        }
        if (ok && row < Np) out[((size_t)ks * C::MT + mt) * 32 + lane] = A[(size_t)row * KA + k];
      }
  return out;
}

std::vector<double> fragments_for(int N, const std::vector<double> &A) {
  switch (N) {
    case 2: return batch_fragments<2>(A);
    case 3: return batch_fragments<3>(A);
    case 4: return batch_fragments<4>(A);
    case 5: return batch_fragments<5>(A);
    case 6: return batch_fragments<6>(A);
  }
  return {};
}

int tile_elems(int N) {
  switch (N) {
    case 2: return BT<2>::E;
    case 3: return BT<3>::E;
    case 4: return BT<4>::E;
    case 5: return BT<5>::E;
    case 6: return BT<6>::E;
  }
  return 0;
}

void drop_batch_graphs(dglm_batch *b) {
  for (auto &g : b->graph) {
    if (g) cudaGraphExecDestroy(g);
    g = nullptr;
  }
}

cudaError_t issue_batch_step(dglm_batch *b, int cur, cudaStream_t s) {
  const int n = (int)b->hinst.size();
  const int tb = 128, nb = (n + tb - 1) / tb;
  cudaError_t e = launch_pdl(batch_step_begin_kernel, dim3(nb), dim3(tb), 0, s, n, b->inst,
                             b->d.cfl, b->d.tmax, b->sc);
  for (int st = 0; st < 5 && e == cudaSuccess; st++) {
    const int in = (cur + st) & 1;
    if (b->sym) {
      BatchSymArgs q = b->sargs;
      q.u_in = b->u[in];
      q.u_out = b->u[in ^ 1];
      q.rka = RKA[st];
      q.rkb = RKB[st];
      q.wait_cycles = b->wait_cycles;
      e = launch_pdl(batch_sym_kernel, dim3(b->grid), dim3(32 * kSymWarps), kBatchSymSmem, s, q);
      continue;
    }
    BatchArgs a = b->args;
    a.u_in = b->u[in];
    a.u_out = b->u[in ^ 1];
    a.rka = RKA[st];
    a.rkb = RKB[st];
    batch_stage_kernel<<<b->grid, kBatchThreads, kBatchSmem, s>>>(a);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) {
    e = launch_pdl(batch_step_end_kernel, dim3(nb), dim3(tb), 0, s, n, b->sc);
  }
  return e;
}

template <int N>
std::pair<size_t, int> label_offset() {
  using Z = SymSize<N>;
  return {(size_t)Z::S_A, Z::T_VOL + Z::T_FACE + Z::T_OUT};
}
// where an operator image holds its face labels: (doubles, then ints)
std::pair<size_t, int> sym_label_offset(int N) {
  switch (N) {
    case 2: return label_offset<2>();
    case 3: return label_offset<3>();
    case 4: return label_offset<4>();
    case 5: return label_offset<5>();
    default: return label_offset<6>();
  }
}
// ints of a tile's neighbour list
size_t sym_neighbour_ints(int N) { return (size_t)128 * ((nfp_of(N) + 3) / 4); }

template <int N>
cudaError_t launch_neighbours(dglm_batch *b, int begin, int ntiles, const int *vmapP, int *nb) {
  const long n = (long)ntiles * 32 * BSC<N>::KSF;
  batch_neighbour_kernel<N><<<(unsigned)((n + 255) / 256), 256>>>(
      b->sargs.image[N], b->tiles + begin, ntiles, b->inst, vmapP, nb);
  return cudaGetLastError();
}

// Operator images, flux weights, neighbour lists and the cut of the tile list
// for the symmetry-adapted path.
dglm_status finalize_sym(dglm_batch *b, const std::vector<BatchTile> &tiles,
                         const std::vector<double> *image, const double *geo, const double *nrm,
                         const double *fscale, long gs, const int *vmapP, double *kreg,
                         long elems) {
  BatchSymArgs &q = b->sargs;
  q = BatchSymArgs{};
  int count[kMaxOrder + 1] = {};
  for (const BatchTile &t : tiles) count[t.N]++;
  q.begin[7] = q.begin[6] = 0;
  for (int N = 6; N >= 1; N--) q.begin[N - 1] = q.begin[N] + (N >= 2 ? count[N] : 0);
  int sms = 0;
  cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, b->dev);
  if (e != cudaSuccess) return cuda_check(e, "dglm_batch_finalize");
  b->grid = std::max(1, std::min((int)tiles.size(), sms));
  // stretches of equal cost
  double total = 0;
  for (const BatchTile &t : tiles) total += kSymCost[t.N];
  std::vector<int> cut(b->grid + 1, (int)tiles.size());
  double sum = 0;
  int c = 0;
  for (int i = 0; i < (int)tiles.size() && c < b->grid; i++) {
    while (c < b->grid && sum >= total * c / b->grid) cut[c++] = i;
    sum += kSymCost[tiles[i].N];
  }
  // all arrays of the path in one allocation (each takes some 0.3 ms)
  size_t bytes = 0;
  auto place = [&](size_t n) {
    const size_t at = bytes;
    bytes += (n + 255) / 256 * 256;
    return at;
  };
  const size_t at_rec = place(sizeof(double) * elems * kSymRec),
               at_cut = place(sizeof(int) * cut.size()),
               at_lab = place(sizeof(int *) * (kMaxOrder + 1)), at_err = place(sizeof(int));
  size_t at_img[kMaxOrder + 1] = {}, at_nb[kMaxOrder + 1] = {};
  for (int N = 2; N <= 6; N++) {
    at_img[N] = place(sizeof(double) * image[N].size());
    at_nb[N] = place(sizeof(int) * sym_neighbour_ints(N) * count[N]);
  }
  char *base = nullptr;
  const dglm_status st = balloc(b, &base, bytes);
  if (st != DGLM_OK) return st;
  double *rec = reinterpret_cast<double *>(base + at_rec);
  int *dcut = reinterpret_cast<int *>(base + at_cut);
  const int **labels = reinterpret_cast<const int **>(base + at_lab);
  b->err = reinterpret_cast<int *>(base + at_err);
  const auto H2D = cudaMemcpyHostToDevice;
  e = cudaMemcpy(dcut, cut.data(), sizeof(int) * cut.size(), H2D);
  if (e == cudaSuccess) e = cudaMemset(b->err, 0, sizeof(int));
  std::vector<const int *> hl(kMaxOrder + 1, nullptr);
  for (int N = 2; N <= 6 && e == cudaSuccess; N++) {
    if (image[N].empty()) continue;
    double *img = reinterpret_cast<double *>(base + at_img[N]);
    int *nb = reinterpret_cast<int *>(base + at_nb[N]);
    e = cudaMemcpy(img, image[N].data(), sizeof(double) * image[N].size(), H2D);
    q.image[N] = img;
    q.nb[N] = nb;
    // the face labels sit behind the image's tables
    hl[N] = reinterpret_cast<const int *>(img + sym_label_offset(N).first) +
            sym_label_offset(N).second;
    if (e != cudaSuccess) break;
    switch (N) {
      case 2: e = launch_neighbours<2>(b, q.begin[2], count[2], vmapP, nb); break;
      case 3: e = launch_neighbours<3>(b, q.begin[3], count[3], vmapP, nb); break;
      case 4: e = launch_neighbours<4>(b, q.begin[4], count[4], vmapP, nb); break;
      case 5: e = launch_neighbours<5>(b, q.begin[5], count[5], vmapP, nb); break;
      default: e = launch_neighbours<6>(b, q.begin[6], count[6], vmapP, nb); break;
    }
  }
  if (e == cudaSuccess) e = cudaMemcpy(labels, hl.data(), sizeof(int *) * hl.size(), H2D);
  const int ninst = (int)b->hinst.size();
  for (int i = 0; i < ninst && e == cudaSuccess; i += 65535) {
    const int m = std::min(65535, ninst - i);
    batch_record_kernel<<<dim3(16, m), 128>>>(b->inst + i, labels, geo, nrm, fscale, gs, rec);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(batch_sym_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)kBatchSymSmem);
  if (e == cudaSuccess) e = cudaStreamSynchronize(nullptr);
  if (e != cudaSuccess) return cuda_check(e, "dglm_batch_finalize");
  q.tiles = b->tiles;
  q.cut = dcut;
  q.inst = b->inst;
  q.sc = b->sc;
  q.rec = rec;
  q.kreg = kreg;
  q.err = b->err;
  return DGLM_OK;
}

}  // namespace

extern "C" {

dglm_status dglm_batch_create(const dglm_batch_desc *desc, dglm_batch **out) {
  if (!desc || !out) return set_error(DGLM_ERR_INVALID, "dglm_batch_create: NULL argument");
  *out = nullptr;
  if (desc->physics != DGLM_ADVECTION)
    return set_error(DGLM_ERR_UNSUPPORTED, "dglm_batch_create: batches are advection only");
  if (!(desc->cfl > 0) || !(desc->tau_scale >= 0) || !(desc->tmax > 0))
    return set_error(DGLM_ERR_INVALID, "dglm_batch_create: cfl/tau_scale/tmax out of range");
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0)
    return set_error(DGLM_ERR_CUDA, "dglm_batch_create: no CUDA device");
  if (desc->device >= ndev)
    return set_error(DGLM_ERR_INVALID, "dglm_batch_create: device out of range");
  dglm_batch *b = new dglm_batch();
  b->d = *desc;
  if (desc->device < 0) cudaGetDevice(&b->dev); else b->dev = desc->device;
  DeviceGuard g(b->dev);
  if (cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking) != cudaSuccess) {
    delete b;
    return set_error(DGLM_ERR_CUDA, "dglm_batch_create: stream creation failed");
  }
  b->own_stream = true;
  *out = b;
  return DGLM_OK;
}

dglm_status dglm_batch_add(dglm_batch *b, int N, int K, const dglm_mesh_arrays *m,
                           const double *u0, const double *velocity, int *index) {
  if (!b || !m || !u0 || !velocity)
    return set_error(DGLM_ERR_INVALID, "dglm_batch_add: NULL argument");
  if (b->finalized) return set_error(DGLM_ERR_STATE, "dglm_batch_add: batch already finalized");
  if (N < 2 || N > 6) return set_error(DGLM_ERR_UNSUPPORTED, "dglm_batch_add: orders 2..6");
  if (K <= 0) return set_error(DGLM_ERR_INVALID, "dglm_batch_add: K must be positive");
  const int Np = np_of(N), NFF = 4 * nfp_of(N);
  const double *req[] = {m->WDr, m->WDs, m->WDt, m->LIFT, m->rx, m->ry, m->rz, m->sx,
                         m->sy,  m->sz,  m->tx,  m->ty,   m->tz, m->Fscale, m->nx, m->ny, m->nz};
  for (const double *p : req)
    if (!p) return set_error(DGLM_ERR_INVALID, "dglm_batch_add: a real array is NULL");
  if (!m->vmapP || !m->Fmask) return set_error(DGLM_ERR_INVALID, "dglm_batch_add: index array is NULL");
  if (m->matrix_order != 'c' && m->matrix_order != 'f')
    return set_error(DGLM_ERR_INVALID, "dglm_batch_add: matrix_order must be 'c' or 'f'");
  for (long i = 0; i < (long)K * NFF; i++)
    if (m->vmapP[i] < 0 || m->vmapP[i] >= (long)K * Np)
      return set_error(DGLM_ERR_INVALID, "dglm_batch_add: vmapP entry outside [0, K*Np)");
  for (int i = 0; i < NFF; i++)
    if (m->Fmask[i] < 0 || m->Fmask[i] >= Np)
      return set_error(DGLM_ERR_INVALID, "dglm_batch_add: Fmask entry outside [0, Np)");
  for (long i = 0; i < (long)K * Np; i++)
    if (!std::isfinite(u0[i]))
      return set_error(DGLM_ERR_NONFINITE, "dglm_batch_add: non-finite initial state");
  for (int q = 0; q < 3; q++)
    if (!std::isfinite(velocity[q]))
      return set_error(DGLM_ERR_INVALID, "dglm_batch_add: non-finite velocity");
  // operators: one copy per order, the first instance of that order provides it
  const bool cm = m->matrix_order == 'f';
  const int KA = 3 * Np + NFF;
  std::vector<double> A((size_t)Np * KA);
  auto at = [&](const double *M, long i, long j, long cols) {
    return cm ? M[j * Np + i] : M[i * cols + j];
  };
  for (long i = 0; i < Np; i++) {
    for (long j = 0; j < Np; j++) {
      A[i * KA + j] = at(m->WDr, i, j, Np);
      A[i * KA + Np + j] = at(m->WDs, i, j, Np);
      A[i * KA + 2 * Np + j] = at(m->WDt, i, j, Np);
    }
    for (long j = 0; j < NFF; j++) A[i * KA + 3 * Np + j] = -at(m->LIFT, i, j, NFF);
  }
  std::vector<int> Fm(m->Fmask, m->Fmask + NFF);
  if (b->Ahost[N].empty()) {
    b->Ahost[N] = A;
    b->Fm[N] = Fm;
  } else if (b->Ahost[N] != A || b->Fm[N] != Fm) {
    return set_error(DGLM_ERR_INVALID,
                     "dglm_batch_add: operators differ from an earlier instance of this order");
  }
  BatchHostInst I;
  I.N = N;
  I.K = K;
  for (int q = 0; q < 3; q++) I.v[q] = velocity[q];
  const double *g9[9] = {m->rx, m->ry, m->rz, m->sx, m->sy, m->sz, m->tx, m->ty, m->tz};
  for (int q = 0; q < 9; q++) I.geo[q].assign(g9[q], g9[q] + K);
  I.nrm[0].assign(m->nx, m->nx + 4L * K);
  I.nrm[1].assign(m->ny, m->ny + 4L * K);
  I.nrm[2].assign(m->nz, m->nz + 4L * K);
  I.fscale.assign(m->Fscale, m->Fscale + 4L * K);
  I.vmapP.assign(m->vmapP, m->vmapP + (long)K * NFF);
  I.u0.assign(u0, u0 + (long)K * Np);
  b->host.push_back(std::move(I));
  if (index) *index = (int)b->host.size() - 1;
  return DGLM_OK;
}

// Uploads the instances for the path b->sym names and prepares their steps.
static dglm_status finalize_path(dglm_batch *b, const std::vector<double> *image) {
  const int n = (int)b->host.size();
  long nodes = 0, elems = 0, fps = 0;
  b->hinst.resize(n);
  for (int i = 0; i < n; i++) {
    const BatchHostInst &H = b->host[i];
    const int Np = np_of(H.N), NFF = 4 * nfp_of(H.N);
    BatchInst &I = b->hinst[i];
    I.node_off = nodes;
    I.elem_off = elems;
    I.fp_off = fps;
    I.K = H.K;
    I.N = H.N;
    I.vx = H.v[0];
    I.vy = H.v[1];
    I.vz = H.v[2];
    // update_tau with maxv = |v| on both sides (advec_dglm.cpp)
    const double mv = std::sqrt(I.vx * I.vx + I.vy * I.vy + I.vz * I.vz);
    I.tau = 0.25 * (mv + mv) * b->d.tau_scale;
    // whole tiles of 8 elements (their padding is zero and stays zero)
    nodes += ((long)H.K + 7) / 8 * 8 * Np;
    elems += H.K;
    fps += (long)H.K * NFF;
  }
  const long gs = elems;
  // tiles, largest order first
  std::vector<BatchTile> tiles;
  for (int N = 6; N >= 2; N--)
    for (int i = 0; i < n; i++) {
      if (b->host[i].N != N) continue;
      const int E = b->sym ? 8 : tile_elems(N);
      for (int e0 = 0; e0 < b->host[i].K; e0 += E)
        tiles.push_back(BatchTile{i, e0, std::min(E, b->host[i].K - e0), N});
    }
  b->ntiles = (int)tiles.size();
  // host staging of the concatenated arrays
  std::vector<double> geo((size_t)9 * gs), nrm((size_t)12 * gs), fs((size_t)4 * gs),
      u0((size_t)nodes, 0.0);
  std::vector<int> vm((size_t)fps);
  for (int i = 0; i < n; i++) {
    const BatchHostInst &H = b->host[i];
    const BatchInst &I = b->hinst[i];
    for (int q = 0; q < 9; q++)
      std::copy(H.geo[q].begin(), H.geo[q].end(), geo.begin() + (size_t)q * gs + I.elem_off);
    for (int q = 0; q < 3; q++)
      std::copy(H.nrm[q].begin(), H.nrm[q].end(),
                nrm.begin() + (size_t)q * 4 * gs + 4 * I.elem_off);
    std::copy(H.fscale.begin(), H.fscale.end(), fs.begin() + 4 * I.elem_off);
    std::copy(H.vmapP.begin(), H.vmapP.end(), vm.begin() + I.fp_off);
    std::copy(H.u0.begin(), H.u0.end(), u0.begin() + I.node_off);
  }
  dglm_status st = DGLM_OK;
  auto chk = [&](dglm_status s) {
    if (st == DGLM_OK) st = s;
  };
  double *dgeo = nullptr, *dnrm = nullptr, *dfs = nullptr, *dk = nullptr;
  int *dvm = nullptr;
  chk(balloc(b, &b->inst, (size_t)n));
  chk(balloc(b, &b->sc, (size_t)n));
  chk(balloc(b, &b->tiles, tiles.size()));
  chk(balloc(b, &dgeo, geo.size()));
  chk(balloc(b, &dnrm, nrm.size()));
  chk(balloc(b, &dfs, fs.size()));
  chk(balloc(b, &dvm, vm.size()));
  chk(balloc(b, &b->u[0], (size_t)nodes));
  chk(balloc(b, &b->u[1], (size_t)nodes));
  chk(balloc(b, &dk, (size_t)nodes));
  if (st != DGLM_OK) return st;
  const auto H2D = cudaMemcpyHostToDevice;
  cudaError_t e = cudaMemcpy(b->inst, b->hinst.data(), sizeof(BatchInst) * n, H2D);
  if (e == cudaSuccess) e = cudaMemcpy(b->tiles, tiles.data(), sizeof(BatchTile) * tiles.size(), H2D);
  if (e == cudaSuccess) e = cudaMemcpy(dgeo, geo.data(), sizeof(double) * geo.size(), H2D);
  if (e == cudaSuccess) e = cudaMemcpy(dnrm, nrm.data(), sizeof(double) * nrm.size(), H2D);
  if (e == cudaSuccess) e = cudaMemcpy(dfs, fs.data(), sizeof(double) * fs.size(), H2D);
  if (e == cudaSuccess) e = cudaMemcpy(dvm, vm.data(), sizeof(int) * vm.size(), H2D);
  if (e == cudaSuccess) e = cudaMemcpy(b->u[0], u0.data(), sizeof(double) * nodes, H2D);
  if (e == cudaSuccess) e = cudaMemset(b->u[1], 0, sizeof(double) * nodes);
  if (e == cudaSuccess) e = cudaMemset(dk, 0, sizeof(double) * nodes);
  if (e == cudaSuccess) e = cudaMemset(b->sc, 0, sizeof(BatchScalars) * n);
  BatchArgs &a = b->args;
  a = BatchArgs{};
  for (int N = 2; N <= 6 && e == cudaSuccess; N++) {
    if (b->sym || b->Ahost[N].empty()) continue;
    std::vector<double> fr = fragments_for(N, b->Ahost[N]);
    double *dops = nullptr;
    int *dfm = nullptr;
    if (balloc(b, &dops, fr.size()) != DGLM_OK || balloc(b, &dfm, b->Fm[N].size()) != DGLM_OK)
      return DGLM_ERR_NOMEM;
    e = cudaMemcpy(dops, fr.data(), sizeof(double) * fr.size(), H2D);
    if (e == cudaSuccess)
      e = cudaMemcpy(dfm, b->Fm[N].data(), sizeof(int) * b->Fm[N].size(), H2D);
    a.ops[N] = dops;
    a.Fmask[N] = dfm;
  }
  if (e != cudaSuccess) return cuda_check(e, "dglm_batch_finalize");
  a.tiles = b->tiles;
  a.ntiles = b->ntiles;
  a.inst = b->inst;
  a.sc = b->sc;
  a.geo = dgeo;
  a.nrm = dnrm;
  a.fscale = dfs;
  a.gs = gs;
  a.vmapP = dvm;
  a.kreg = dk;
  if (b->sym) {
    st = finalize_sym(b, tiles, image, dgeo, dnrm, dfs, gs, dvm, dk, elems);
    if (st != DGLM_OK) return st;
  }
  e = cudaFuncSetAttribute(batch_stage_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)kBatchSmem);
  int per_sm = 0, sms = 0;
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, batch_stage_kernel,
                                                      kBatchThreads, kBatchSmem);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, b->dev);
  if (e != cudaSuccess) return cuda_check(e, "dglm_batch_finalize");
  if (!b->sym) b->grid = std::max(1, std::min(b->ntiles, std::max(per_sm, 1) * sms));
  batch_wavespeed_kernel<<<n, 256, 0, b->stream>>>(b->inst, dfs, b->sc);
  e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaStreamSynchronize(b->stream);
  if (e != cudaSuccess) return cuda_check(e, "dglm_batch_finalize");
  return DGLM_OK;
}

dglm_status dglm_batch_finalize(dglm_batch *b) {
  if (!b) return set_error(DGLM_ERR_INVALID, "dglm_batch_finalize: NULL batch");
  if (b->finalized) return set_error(DGLM_ERR_STATE, "dglm_batch_finalize: already finalized");
  if (b->host.empty()) return set_error(DGLM_ERR_STATE, "dglm_batch_finalize: no instances");
  DeviceGuard g(b->dev);
  std::vector<double> image[kMaxOrder + 1];
  b->sym = true;
  for (int N = 2; N <= 6; N++)
    if (!b->Ahost[N].empty())
      b->sym = b->sym && sym_operator_image(N, b->Ahost[N].data(), b->Fm[N].data(), image[N]);
  dglm_status st = finalize_path(b, image);
  if (st == DGLM_ERR_NOMEM && b->sym) {
    // without memory for the symmetry-adapted path's lists and records: the
    // dense kernel takes less
    cudaGetLastError();
    for (void *p : b->allocs) cudaFree(p);
    b->allocs.clear();
    b->bytes = 0;
    b->err = nullptr;
    b->sym = false;
    st = finalize_path(b, image);
  }
  if (st != DGLM_OK) return st;
  b->host.clear();
  b->host.shrink_to_fit();
  b->cur = 0;
  b->finalized = true;
  return DGLM_OK;
}

dglm_status dglm_batch_step(dglm_batch *b, int nsteps) {
  if (!b) return set_error(DGLM_ERR_INVALID, "dglm_batch_step: NULL batch");
  if (!b->finalized) return set_error(DGLM_ERR_STATE, "dglm_batch_step: finalize first");
  if (nsteps < 0) return set_error(DGLM_ERR_INVALID, "dglm_batch_step: negative step count");
  DeviceGuard g(b->dev);
  b->launches = 0;
  b->expired.store(-1);
  for (int i = 0; i < nsteps; i++) {
    const int c = b->cur;
    if (!b->graph[c]) {
      cudaGraph_t graph = nullptr;
      cudaStream_t cs = b->stream;
      bool ok = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal) == cudaSuccess;
      cudaError_t le = ok ? issue_batch_step(b, c, cs) : cudaSuccess;
      ok = (cudaStreamEndCapture(cs, &graph) == cudaSuccess) && ok && le == cudaSuccess;
      if (ok && cudaGraphInstantiate(&b->graph[c], graph, 0) != cudaSuccess) {
        b->graph[c] = nullptr;
        ok = false;
      }
      if (graph) cudaGraphDestroy(graph);
      cudaGetLastError();
      if (!ok) {
        cudaError_t e = issue_batch_step(b, c, b->stream);
        if (e != cudaSuccess) return cuda_check(e, "dglm_batch_step");
        b->launches += 7;
        b->cur ^= 1;
        continue;
      }
    }
    cudaError_t e = cudaGraphLaunch(b->graph[c], b->stream);
    if (e != cudaSuccess) return cuda_check(e, "dglm_batch_step: graph launch");
    b->launches += 7;
    b->cur ^= 1;
  }
  return DGLM_OK;
}

// Waits for the batch's stream and reports an expired wait of the steps taken
// so far.  The flag is read once per dglm_batch_step: a caller that takes every
// instance's state out does not pay for it each time.
static dglm_status batch_sync(dglm_batch *b, const char *what) {
  int err = b->err ? b->expired.load() : 0;
  const bool read = err < 0;
  cudaError_t e = cudaSuccess;
  if (read) e = cudaMemcpyAsync(&err, b->err, sizeof(int), cudaMemcpyDeviceToHost, b->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(b->stream);
  if (e != cudaSuccess) return cuda_check(e, what);
  if (read) b->expired.store(err);
  if (err)
    return set_error(DGLM_ERR_CUDA, std::string(what) + ": a bounded wait in the stage kernel "
                                    "expired; results are invalid");
  return DGLM_OK;
}

dglm_status dglm_batch_sync(dglm_batch *b) {
  if (!b) return set_error(DGLM_ERR_INVALID, "dglm_batch_sync: NULL batch");
  DeviceGuard g(b->dev);
  return batch_sync(b, "dglm_batch_sync");
}

int dglm_batch_count(dglm_batch *b) {
  if (!b) return -1;
  return b->finalized ? (int)b->hinst.size() : (int)b->host.size();
}

dglm_status dglm_batch_get_state(dglm_batch *b, int index, double *u, int on_device) {
  if (!b || !u) return set_error(DGLM_ERR_INVALID, "dglm_batch_get_state: NULL argument");
  if (!b->finalized) return set_error(DGLM_ERR_STATE, "dglm_batch_get_state: finalize first");
  if (index < 0 || index >= (int)b->hinst.size())
    return set_error(DGLM_ERR_INVALID, "dglm_batch_get_state: no such instance");
  DeviceGuard g(b->dev);
  const BatchInst &I = b->hinst[index];
  cudaError_t e = cudaMemcpyAsync(u, b->u[b->cur] + I.node_off,
                                  sizeof(double) * (size_t)I.K * np_of(I.N),
                                  on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost,
                                  b->stream);
  if (e != cudaSuccess) return cuda_check(e, "dglm_batch_get_state");
  return batch_sync(b, "dglm_batch_get_state");
}

dglm_status dglm_batch_get_time(dglm_batch *b, int index, double *t, double *dt, int *tstep) {
  if (!b) return set_error(DGLM_ERR_INVALID, "dglm_batch_get_time: NULL batch");
  if (!b->finalized) return set_error(DGLM_ERR_STATE, "dglm_batch_get_time: finalize first");
  if (index < 0 || index >= (int)b->hinst.size())
    return set_error(DGLM_ERR_INVALID, "dglm_batch_get_time: no such instance");
  DeviceGuard g(b->dev);
  BatchScalars s{};
  const dglm_status st = batch_sync(b, "dglm_batch_get_time");
  if (st != DGLM_OK) return st;
  cudaError_t e = cudaMemcpy(&s, b->sc + index, sizeof(BatchScalars), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return cuda_check(e, "dglm_batch_get_time");
  if (t) *t = s.t;
  if (dt) *dt = s.dt;
  if (tstep) *tstep = s.tstep;
  return DGLM_OK;
}

dglm_status dglm_batch_set_stream(dglm_batch *b, void *stream) {
  if (!b) return set_error(DGLM_ERR_INVALID, "dglm_batch_set_stream: NULL batch");
  DeviceGuard g(b->dev);
  cudaStreamSynchronize(b->stream);
  drop_batch_graphs(b);
  if (b->own_stream) cudaStreamDestroy(b->stream);
  b->own_stream = false;
  b->stream = (cudaStream_t)stream;
  return DGLM_OK;
}

dglm_status dglm_batch_set_wait_limit(dglm_batch *b, long long cycles) {
  if (!b) return set_error(DGLM_ERR_INVALID, "dglm_batch_set_wait_limit: NULL batch");
  if (cycles < 0)
    return set_error(DGLM_ERR_INVALID, "dglm_batch_set_wait_limit: negative bound");
  DeviceGuard g(b->dev);
  cudaStreamSynchronize(b->stream);
  drop_batch_graphs(b);   // the captured steps carry the bound in their arguments
  b->wait_cycles = cycles ? cycles : kWaitCycles;
  return DGLM_OK;
}

long dglm_batch_kernel_launches(dglm_batch *b) { return b ? b->launches : -1; }

size_t dglm_batch_device_bytes(dglm_batch *b) { return b ? b->bytes : 0; }

dglm_status dglm_batch_destroy(dglm_batch *b) {
  if (!b) return DGLM_OK;
  DeviceGuard g(b->dev);
  if (b->stream) cudaStreamSynchronize(b->stream);
  drop_batch_graphs(b);
  for (void *p : b->allocs) cudaFree(p);
  if (b->own_stream && b->stream) cudaStreamDestroy(b->stream);
  delete b;
  return DGLM_OK;
}

}  // extern "C"
