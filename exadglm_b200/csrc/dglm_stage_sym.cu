// Symmetry-adapted FP64 Euler stage: variants and the host side of the
// operators (see dglm_stage_sym.cuh for the decomposition).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "dglm_sym.cuh"

namespace dglm {

namespace {

// chi_c(a) of V4 with vertex i -> i^a: chi_1 = + on {0,1}, chi_2 on {0,2}, chi_3 on {0,3}
__host__ __device__ constexpr int chi(int c, int a) { return c == 0 || a == 0 || a == c ? 1 : -1; }

// The node set of order N under V4 and the kernel's numbering of it.  Nodes
// are in the datain order: the lattice (i_1, i_2, i_3) of barycentric counts,
// i_1 (r) fastest.
template <int N>
struct SymLayout {
  using Z = SymSize<N>;
  int bary[Z::Np][4];
  int perm[4][Z::Np];                  // perm[a][i]: the node that V4 element a maps i to
  int slot_node[8 * Z::MT0][4];        // chi_0's slot -> its orbit's nodes by label (-1: empty)
  int vol_node[Z::KSV * 4], vol_src[Z::KSV * 4][4];   // k position -> node, lane of its image
  bool vol_pad[Z::KSV * 4];

  SymLayout() {
    int n = 0;
    for (int i3 = 0; i3 <= N; i3++)
      for (int i2 = 0; i2 + i3 <= N; i2++)
        for (int i1 = 0; i1 + i2 + i3 <= N; i1++, n++) {
          bary[n][0] = N - i1 - i2 - i3;
          bary[n][1] = i1;
          bary[n][2] = i2;
          bary[n][3] = i3;
        }
    for (int a = 0; a < 4; a++)
      for (int i = 0; i < Z::Np; i++) {
        perm[a][i] = -1;
        for (int j = 0; j < Z::Np; j++) {
          bool same = true;
          for (int q = 0; q < 4; q++) same &= bary[j][q ^ a] == bary[i][q];
          if (same) perm[a][i] = j;
        }
      }
    // orbits by their first node
    std::vector<int> o4, o2[4], o1;
    for (int i = 0; i < Z::Np; i++) {
      int first = i, fixed = 0, by = 0;
      for (int a = 1; a < 4; a++) {
        first = std::min(first, perm[a][i]);
        if (perm[a][i] == i) {
          fixed++;
          by = a;
        }
      }
      if (first != i) continue;
      if (fixed == 0) o4.push_back(i);
      else if (fixed == 1) o2[by].push_back(i);
      else o1.push_back(i);
    }
    for (auto &s : slot_node)
      for (int &x : s) x = -1;
    auto set = [&](int slot, int i) {
      for (int a = 0; a < 4; a++) slot_node[slot][a] = perm[a][i];
    };
    for (int q = 0; q < Z::N4; q++) set(q, o4[q]);
    for (int b = 1; b < 4; b++)
      for (int i = 0; i < Z::N2; i++) set(Z::slot0(b, i), o2[b][i]);
    for (int i = 0; i < Z::N1; i++) set(Z::N4 + 3 * Z::N2 + i, o1[i]);
    // k positions: one orbit of size 4 per k-step, then the orbits of size 2
    // in pairs, then the centroid; padding repeats node 0 with zero columns
    int p = 0;
    auto put = [&](int node, int s1, int s2, int s3, bool pad) {
      vol_node[p] = node;
      vol_src[p][0] = p % 4;
      vol_src[p][1] = s1;
      vol_src[p][2] = s2;
      vol_src[p][3] = s3;
      vol_pad[p] = pad;
      p++;
    };
    for (int i : o4)
      for (int l = 0; l < 4; l++) put(perm[l][i], l ^ 1, l ^ 2, l ^ 3, false);
    for (int b = 1; b < 4; b++)
      for (int i : o2[b]) {
        const int other = perm[b == 1 ? 2 : 1][i];
        for (int h = 0; h < 2; h++) {
          const int l = p % 4;
          put(h ? other : i, b == 1 ? l : l ^ 1, b == 2 ? l : l ^ 1, b == 3 ? l : l ^ 1, false);
        }
      }
    for (int i : o1) put(i, p % 4, p % 4, p % 4, false);
    while (p < Z::KSV * 4) put(0, p % 4, p % 4, p % 4, true);
  }
};

template <int N>
const SymLayout<N> &sym_layout() {
  static const SymLayout<N> l;
  return l;
}

// Largest deviation from the symmetry, of the largest entry, up to which the
// operators' average over V4 stands for them.  The symmetry holds to rounding
// for every node set that is symmetric itself (orders 3..8 of this package: 1e-16
// to 5.7e-15, with the linear algebra library's rounding; a set made elsewhere
// may have some other); operators further off run on the dense kernels as they
// are.
constexpr double kSymTol = 1e-14;

// face label v (0..3: opposite vertex v) -> face and its points' positions;
// aligned: position pos[v][j] of face_of[v] is the image under v of point j
// of face_of[0]
template <int N>
bool face_labels(const int *Fmask, int face_of[4], int pos[4][SymSize<N>::Nfp]) {
  using Z = SymSize<N>;
  const SymLayout<N> &L = sym_layout<N>();
  for (int v = 0; v < 4; v++) face_of[v] = -1;
  for (int f = 0; f < 4; f++)
    for (int v = 0; v < 4; v++) {
      bool on = true;
      for (int j = 0; j < Z::Nfp; j++) on &= L.bary[Fmask[f * Z::Nfp + j]][v] == 0;
      if (on) {
        if (face_of[v] >= 0) return false;
        face_of[v] = f;
      }
    }
  for (int v = 0; v < 4; v++)
    if (face_of[v] < 0) return false;
  for (int v = 0; v < 4; v++)
    for (int j = 0; j < Z::Nfp; j++) {
      const int want = L.perm[v][Fmask[face_of[0] * Z::Nfp + j]];
      pos[v][j] = -1;
      for (int i = 0; i < Z::Nfp; i++)
        if (Fmask[face_of[v] * Z::Nfp + i] == want) {
          if (pos[v][j] >= 0) return false;
          pos[v][j] = i;
        }
      if (pos[v][j] < 0) return false;
    }
  return true;
}

// Operator image of the kernel from A = [WDr WDs WDt -LIFT] (row-major, Np x
// (3Np + NFF)); false when the operators or Fmask lack the symmetry.
template <int N>
bool build_image(const double *A, const int *Fmask, std::vector<double> &img) {
  using Z = SymSize<N>;
  const SymLayout<N> &L = sym_layout<N>();
  constexpr int Np = Z::Np, Nfp = Z::Nfp, KA = 3 * Np + Z::NFF;
  int face_of[4], pos[4][Nfp];
  if (!face_labels<N>(Fmask, face_of, pos)) return false;
  // barycentric derivative operators W_v = WD_v + W_0, W_0 = -(sum WD)/4
  std::vector<double> W((size_t)4 * Np * Np);
  auto w = [&](int v, int i, int j) -> double & { return W[((size_t)v * Np + i) * Np + j]; };
  double wmax = 0, lmax = 0;
  for (int i = 0; i < Np; i++)
    for (int j = 0; j < Np; j++) {
      const double r = A[i * KA + j], s = A[i * KA + Np + j], t = A[i * KA + 2 * Np + j];
      w(0, i, j) = -0.25 * (r + s + t);
      w(1, i, j) = r + w(0, i, j);
      w(2, i, j) = s + w(0, i, j);
      w(3, i, j) = t + w(0, i, j);
      wmax = std::max({wmax, std::fabs(r), std::fabs(s), std::fabs(t)});
    }
  for (int i = 0; i < Np; i++)
    for (int j = 0; j < Z::NFF; j++) lmax = std::max(lmax, std::fabs(A[i * KA + 3 * Np + j]));
  auto lift = [&](int v, int i, int j) {
    return A[i * KA + 3 * Np + face_of[v] * Nfp + pos[v][j]];
  };
  // averages over V4, and the deviation from them
  std::vector<double> Wa((size_t)Np * Np), La((size_t)Np * Nfp);
  for (int i = 0; i < Np; i++) {
    for (int j = 0; j < Np; j++) {
      double sum = 0;
      for (int v = 0; v < 4; v++) sum += w(v, L.perm[v][i], L.perm[v][j]);
      Wa[(size_t)i * Np + j] = 0.25 * sum;
      for (int v = 0; v < 4; v++)
        if (std::fabs(w(v, L.perm[v][i], L.perm[v][j]) - 0.25 * sum) > kSymTol * wmax)
          return false;
    }
    for (int j = 0; j < Nfp; j++) {
      double sum = 0;
      for (int v = 0; v < 4; v++) sum += lift(v, L.perm[v][i], j);
      La[(size_t)i * Nfp + j] = 0.25 * sum;
      for (int v = 0; v < 4; v++)
        if (std::fabs(lift(v, L.perm[v][i], j) - 0.25 * sum) > kSymTol * lmax) return false;
    }
  }
  // rows of the characters: (1/4) sum_a chi(a) [W_0 | -L_0](perm_a(rep), :)
  img.assign((size_t)Z::S_A + (Z::TABS + 1) / 2, 0.0);
  for (int c = 0; c < 4; c++)
    for (int m = 0; m < (c == 0 ? Z::MT0 : Z::MTB); m++)
      for (int row = 0; row < 8; row++) {
        const int slot = 8 * m + row;
        if (Z::krow(c, slot) < 0) continue;
        // the orbit of this row (chi_b's size-2 rows may sit in other slots than chi_0's)
        int o = slot;
        if (c > 0 && slot >= Z::N4) o = Z::slot0(c, slot - Z::slotb(c, 0));
        const int mt = c == 0 ? m : Z::MT0 + (c - 1) * Z::MTB + m;
        for (int ks = 0; ks < Z::KS; ks++)
          for (int l = 0; l < 4; l++) {
            double x = 0;
            if (ks < Z::KSV) {
              const int p = ks * 4 + l;
              if (!L.vol_pad[p])
                for (int a = 0; a < 4; a++)
                  x += chi(c, a) * Wa[(size_t)L.slot_node[o][a] * Np + L.vol_node[p]];
            } else {
              const int j = (ks - Z::KSV) * 4 + l;
              if (j < Nfp)
                for (int a = 0; a < 4; a++)
                  x += chi(c, a) * La[(size_t)L.slot_node[o][a] * Nfp + j];
            }
            img[((size_t)ks * Z::MTT + mt) * 32 + row * 4 + l] = 0.25 * x;
          }
      }
  std::vector<int> tab(Z::TABS, 0);
  for (int p = 0; p < Z::KSV * 4; p++)
    tab[p] = L.vol_node[p] | L.vol_src[p][1] << 16 | L.vol_src[p][2] << 18 |
             L.vol_src[p][3] << 20;
  for (int j = 0; j < Z::KSF * 4; j++)
    for (int v = 0; v < 4; v++) {
      const int jj = pos[v][j < Nfp ? j : 0], fp = face_of[v] * Nfp + jj;
      tab[Z::T_VOL + j * 4 + v] = Fmask[fp] | fp << 16;
    }
  for (int s = 0; s < 8 * Z::MT0; s++)
    for (int a = 0; a < 4; a++)
      tab[Z::T_VOL + Z::T_FACE + s * 4 + a] = std::max(0, L.slot_node[s][a]);
  int *rest = &tab[Z::T_VOL + Z::T_FACE + Z::T_OUT];
  for (int v = 0; v < 4; v++) rest[v] = face_of[v];
  // face point i = (element, face point) of a tile: trace slot << 16 | code position
  for (int e = 0; e < 8; e++)
    for (int v = 0; v < 4; v++)
      for (int j = 0; j < Nfp; j++)
        rest[4 + e * Z::NFF + face_of[v] * Nfp + pos[v][j]] =
            (Z::col(e) * Z::UPS + v * Nfp + j) << 16 | ((Z::col(e) * Z::NBS + j) * 4 + v);
  std::memcpy(&img[Z::S_A], tab.data(), sizeof(int) * tab.size());
  return true;
}

// nodes of chi_0's slots by label, for the register kernel
template <int N>
struct SlotNodes {
  unsigned char n[SymSize<N>::R0][4];
};

// RK register between nodal (variable blocks of vs doubles) and fragment order:
// a thread per (tile, variable, slot, MMA column), the slot's four characters.
// Elements past K are zero in nodal order.
template <int N>
__global__ void register_order_kernel(SlotNodes<N> slots, long threads, int K, int nvar, long vs,
                                      const double *__restrict__ in, double *__restrict__ out,
                                      bool to_sym) {
  using Z = SymSize<N>;
  constexpr int Np = Z::Np, E = 8;
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= threads) return;
  const int e = (int)(i % E), slot = (int)(i / E % Z::R0), v = (int)(i / (E * Z::R0) % nvar);
  const long t = i / ((long)E * Z::R0 * nvar), k = t * E + Z::elem(e);
  const long nod = v * vs + k * Np, frag = (t * nvar + v) * Np * E + e;
  int nd[4], row[4];
#pragma unroll
  for (int c = 0; c < 4; c++) {
    nd[c] = slots.n[slot][c];
    // the row of character c for this slot's orbit (-1: none)
    const int q = slot - Z::slot0(c, 0);
    row[c] = c == 0 || slot < Z::N4 ? Z::krow(c, slot)
             : q >= 0 && q < Z::N2  ? Z::krow(c, Z::slotb(c, q))
                                    : -1;
  }
  if (to_sym) {
#pragma unroll
    for (int c = 0; c < 4; c++) {
      double x = 0;
#pragma unroll
      for (int a = 0; a < 4; a++) x += chi(c, a) * in[nod + nd[a]];
      if (row[c] >= 0) out[frag + (long)row[c] * E] = 0.25 * x;
    }
    return;
  }
  double y[4];
#pragma unroll
  for (int c = 0; c < 4; c++) y[c] = row[c] >= 0 ? in[frag + (long)row[c] * E] : 0.0;
#pragma unroll
  for (int a = 0; a < 4; a++) {   // (a node that repeats in its orbit gets equal values)
    double x = 0;
#pragma unroll
    for (int c = 0; c < 4; c++) x += chi(c, a) * y[c];
    out[nod + nd[a]] = k < K ? x : 0.0;
  }
}

template <int N>
cudaError_t register_order(int K, int nvar, long vs, const double *in, double *out, bool to_sym,
                           cudaStream_t s) {
  SlotNodes<N> slots;
  for (int q = 0; q < SymSize<N>::R0; q++)
    for (int a = 0; a < 4; a++) slots.n[q][a] = (unsigned char)sym_layout<N>().slot_node[q][a];
  const long n = ((long)K + 7) / 8 * nvar * SymSize<N>::R0 * 8;
  register_order_kernel<N><<<(unsigned)((n + 255) / 256), 256, 0, s>>>(slots, n, K, nvar, vs, in,
                                                                      out, to_sym);
  return cudaGetLastError();
}

template <int N, int NS, int NG, int NB>
cudaError_t launch_sym(const StageArgs &a, cudaStream_t s) {
  using C = SymCfg<N, NS, NG, NB>;
  auto k = stage_sym_kernel<N, NS, NG, NB>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)C::SMEM);
  if (e != cudaSuccess) return e;
  // the split of the registers must fit what the block is launched with, or
  // the compute warps would wait for registers for ever
  static const int regs = [&] {
    cudaFuncAttributes fa{};
    return cudaFuncGetAttributes(&fa, k) == cudaSuccess ? fa.numRegs : 0;
  }();
  if (regs * (C::NWC + C::PW) < C::REGC * C::NWC + C::REGP * C::PW)
    return cudaErrorInvalidConfiguration;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (sms <= 0) sms = 148;
  const int ntiles = (a.K + C::E - 1) / C::E;
  return launch_pdl(k, dim3(ntiles < sms ? ntiles : sms), dim3(C::THREADS), C::SMEM, s, a, ntiles);
}

template <int N, int NS, int NG, int NB>
StageVariant make_sym(const StageVariant &fallback) {
  using C = SymCfg<N, NS, NG, NB>;
  StageVariantInfo i{};
  i.mode = MODE_SYM;
  i.E = C::E;
  i.threads = C::THREADS;
  i.smem = C::SMEM;
  i.bimg = 8 * C::S_A + 4 * ((C::TABS + 1) / 2 * 2);
  i.groups = C::NG;
  i.R = C::WPG;
  i.ring = NB;
  i.persistent = 1;
  return StageVariant{i, &launch_sym<N, NS, NG, NB>, fallback.launch};
}

template <int N, int NW>
cudaError_t launch_sym_adv(const StageArgs &a, cudaStream_t s) {
  using C = SymAdvCfg<N, NW>;
  auto k = stage_sym_adv_kernel<N, NW>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)C::SMEM);
  if (e != cudaSuccess) return e;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (sms <= 0) sms = 148;
  const int ntiles = (a.K + C::E - 1) / C::E;
  return launch_pdl(k, dim3(ntiles < sms ? ntiles : sms), dim3(C::THREADS), C::SMEM, s, a, ntiles);
}

template <int N, int NW>
StageVariant make_sym_adv(const StageVariant &fallback) {
  using C = SymAdvCfg<N, NW>;
  StageVariantInfo i{};
  i.mode = MODE_SYM;
  i.E = C::E;
  i.threads = C::THREADS;
  i.smem = C::SMEM;
  i.bimg = 8 * C::S_A + 4 * ((C::Z::TABS + 1) / 2 * 2);
  i.groups = NW;
  i.R = 1;
  i.ring = 2;
  i.persistent = 1;
  return StageVariant{i, &launch_sym_adv<N, NW>, fallback.launch};
}

template <int N>
cudaError_t flow_launch(const double *image, const double *geo, const double *nrm,
                        const double *fscale, const double *vel, const int *vmapP, long vs,
                        long Kp, int K, double *flow) {
  const int ntiles = (K + 7) / 8;
  const long n = (long)ntiles * 32 * (SymSize<N>::KSV + SymSize<N>::KSF);
  sym_flow_kernel<N><<<(unsigned)((n + 255) / 256), 256>>>(image, geo, nrm, fscale, vel, vmapP,
                                                           vs, Kp, K, ntiles, flow);
  return cudaGetLastError();
}

__global__ void element_record_kernel(const double *__restrict__ geo,
                                      const double *__restrict__ nrm,
                                      const double *__restrict__ fscale, long Kp, bool sym,
                                      double *__restrict__ rec) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= Kp * kRecord) return;
  const long k = i / kRecord;
  const int q = (int)(i - k * kRecord);
  double x = 0.0;   // the pad
  if (q < 9) {
    x = geo[q * Kp + k];
    if (sym) x += geo[(q % 3) * Kp + k] + geo[(3 + q % 3) * Kp + k] + geo[(6 + q % 3) * Kp + k];
  } else if (q < 25) {
    const int d = (q - 9) / 4, f = (q - 9) % 4;
    const double fs = fscale[4 * k + f], c = sym ? 0.5 * fs : 1.0;
    x = d < 3 ? c * nrm[d * 4 * Kp + 4 * k + f] : sym ? c : fs;
  }
  rec[i] = x;
}

}  // namespace

cudaError_t launch_element_records(const double *geo, const double *nrm, const double *fscale,
                                   long Kp, bool sym, double *rec) {
  const long n = Kp * kRecord;
  element_record_kernel<<<(unsigned)((n + 255) / 256), 256>>>(geo, nrm, fscale, Kp, sym, rec);
  return cudaGetLastError();
}

StageVariant sym_variant(int physics, int N, const StageVariant &fallback) {
  // Warps per CTA: what the registers allow (N=3 spills 4 bytes), less where the
  // shared memory they take is better left to L1 for the gathers (ms per stage,
  // counted with the gathers before the first k-step: N=6, K=63,888: 8 warps
  // 0.125, 12 warps 0.154; N=3, K=162,000: 24 0.057, 16 0.059, 12 0.063; N=5,
  // K=93,750: 16 0.092, 12 0.097, 20 0.111).  Against the dense kernels: N=2,
  // K=384,000 0.313 -> 0.077, N=3 0.096 -> 0.054, N=4, K=105,456 0.118 -> 0.056,
  // N=5 0.235 -> 0.088 (4.4 TB/s of HBM traffic, 67 % of the copy rate), N=6
  // 0.254 -> 0.111.
  if (physics == DGLM_ADVECTION) switch (N) {
    case 2: return make_sym_adv<2, 16>(fallback);
    case 3: return make_sym_adv<3, 24>(fallback);
    case 4: return make_sym_adv<4, 16>(fallback);
    case 5: return make_sym_adv<5, 16>(fallback);
    default: return make_sym_adv<6, 8>(fallback);
  }
  switch (N) {
    case 3: return make_sym<3, 1, 4, 8>(fallback);
    case 4: return make_sym<4, 1, 4, 6>(fallback);
    case 5: return make_sym<5, 2, 2, 3>(fallback);
    default: return make_sym<6, 2, 2, 2>(fallback);
  }
}

#define SYM_ORDER(N, ...)        \
  switch (N) {                   \
    case 2: { constexpr int n = 2; __VA_ARGS__; break; } \
    case 3: { constexpr int n = 3; __VA_ARGS__; break; } \
    case 4: { constexpr int n = 4; __VA_ARGS__; break; } \
    case 5: { constexpr int n = 5; __VA_ARGS__; break; } \
    case 6: { constexpr int n = 6; __VA_ARGS__; break; } \
    default: break;              \
  }

bool sym_operator_image(int N, const double *A, const int *Fmask, std::vector<double> &img) {
  bool ok = false;
  SYM_ORDER(N, ok = build_image<n>(A, Fmask, img))
  return ok;
}

size_t sym_flow_doubles(int N, int K) {
  size_t per = 0;
  SYM_ORDER(N, per = SymAdvCfg<n, 4>::FLOW)
  return per * (((size_t)K + 7) / 8);
}

cudaError_t launch_sym_flow(int N, const double *image, const double *geo, const double *nrm,
                            const double *fscale, const double *vel, const int *vmapP, long vs,
                            long Kp, int K, double *flow) {
  cudaError_t e = cudaErrorInvalidValue;
  SYM_ORDER(N, e = flow_launch<n>(image, geo, nrm, fscale, vel, vmapP, vs, Kp, K, flow))
  return e;
}

cudaError_t launch_register_order(int N, int K, int nvar, long vs, const double *in, double *out,
                                  bool to_sym, cudaStream_t s) {
  cudaError_t e = cudaErrorInvalidValue;
  SYM_ORDER(N, e = register_order<n>(K, nvar, vs, in, out, to_sym, s))
  return e;
}

}  // namespace dglm
