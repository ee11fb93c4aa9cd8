// FP64 advection stage on the symmetry-adapted operators of
// dglm_stage_sym.cuh (included by dglm_stage_sym.cu).
//
// The fluxes of linear advection are the state times fixed numbers, so the
// mesh upload forms those numbers once, in the order in which the kernel's
// lanes take them (sym_flow_kernel): per tile of 8 elements
//   V  [KSV][3][32]  contravariant velocities (grad r_a + sum_b grad r_b) . v of
//                    the lane's node's image under vertex permutation a;
//   W  [KSF][4][32]  Fscale n . v / 2 of the lane's point of each face;
//   P  [KSF][32][4]  its neighbour node (ints).
// A lane reads u at the three images of its node, so the sums over V4 need no
// shuffle: seven FP64 operations per volume k-step, 24 per face k-step.  V is
// as many bytes as the velocity it replaces, W stands for normals and Fscale.
//
// Each warp takes whole tiles by itself (eight MMA columns, one per element):
// the state arrives and leaves by bulk copies, double-buffered per warp, k
// comes and goes straight from registers in fragment order, the traces are
// plain gathers.  Warps share only the operator, so there is no barrier after
// the start.  Waits are bounded as in the other persistent kernels.
// Bound by the load path and HBM: figures beside the variant table.
#pragma once

template <int N, int NW_>
struct SymAdvCfg : SymSize<N> {
  using Z = SymSize<N>;
  static constexpr int E = 8, NW = NW_, THREADS = 32 * NW;
  static constexpr int S_U = E * Z::Np;
  // doubles of a tile's flow record
  static constexpr int F_V = 96 * Z::KSV, F_W = 128 * Z::KSF, F_P = 64 * Z::KSF;
  static constexpr int FLOW = F_V + F_W + F_P;
  // per volume k position the nodes of its three images, 10 bits each
  static constexpr int TABS = Z::KSV * 4 + Z::T_FACE + Z::T_OUT;
  static constexpr size_t SMEM =
      sizeof(double) * (Z::S_A + (size_t)NW * 2 * S_U + NW * 2) + sizeof(int) * TABS;
  // face k-steps whose traces are on their way during the volume k-steps
  static constexpr int FH = (Z::KSF + 1) / 2;
  static_assert(SMEM <= 232448, "shared memory per CTA exceeds 227 KB");
  static_assert(S_U % 2 == 0, "16-byte aligned copies");
};

template <int N, int NW>
__global__ void __launch_bounds__(32 * NW, 1)
    stage_sym_adv_kernel(const StageArgs a, int ntiles) {
  using C = SymAdvCfg<N, NW>;
  constexpr int Np = C::Np, Nfp = C::Nfp, E = C::E, MTT = C::MTT, MT0 = C::MT0, MTB = C::MTB,
                KSF = C::KSF, KSV = C::KSV, FH = C::FH;
  extern __shared__ __align__(16) double smem[];
  double *sA = smem, *sBuf = sA + C::S_A;
  unsigned long long *bars = reinterpret_cast<unsigned long long *>(sBuf + NW * 2 * C::S_U);
  int *tabs = reinterpret_cast<int *>(bars + NW * 2);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (lane == 0) {
    mbar_init(&bars[2 * warp], 1);
    mbar_init(&bars[2 * warp + 1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  const long stride = (long)gridDim.x * NW, t0 = blockIdx.x + (long)gridDim.x * warp;
  double *buf = sBuf + warp * 2 * C::S_U;
  unsigned long long *full = bars + 2 * warp;
  auto fetch = [&](long t, int b) {   // lane 0
    mbar_arrive_expect_tx(&full[b], 8u * C::S_U);
    bulk_g2s(buf + b * C::S_U, a.u_in + t * C::S_U, 8u * C::S_U, &full[b]);
  };
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  if (lane == 0 && t0 < ntiles) fetch(t0, 0);
  {
    const double2 *src = reinterpret_cast<const double2 *>(a.AT);
    double2 *dst = reinterpret_cast<double2 *>(sA);
    for (int i = tid; i < C::S_A / 2; i += C::THREADS) dst[i] = __ldg(src + i);
    const int *ts = reinterpret_cast<const int *>(a.AT + C::S_A);
    // volume entries with the images' nodes in place of the shuffle lanes
    for (int i = tid; i < KSV * 4; i += C::THREADS) {
      const int q = i & ~3, x = __ldg(ts + i);
      tabs[i] = (__ldg(ts + (q | ((x >> 16) & 3))) & 0x3ff) |
                (__ldg(ts + (q | ((x >> 18) & 3))) & 0x3ff) << 10 |
                (__ldg(ts + (q | ((x >> 20) & 3))) & 0x3ff) << 20;
    }
    for (int i = tid; i < C::T_FACE + C::T_OUT; i += C::THREADS)
      tabs[KSV * 4 + i] = __ldg(ts + C::T_VOL + i);
  }
  __syncthreads();
  const int *tvol = tabs;
  const int4 *tface = reinterpret_cast<const int4 *>(tabs + KSV * 4);
  const int4 *tout = tface + C::T_FACE / 4;
  const int *ft = reinterpret_cast<const int *>(a.AT + C::S_A) + C::T_VOL + C::T_FACE + C::T_OUT;
  const int f0 = __ldg(ft), f1 = __ldg(ft + 1), f2 = __ldg(ft + 2), f3 = __ldg(ft + 3);
  const double dt = a.rhs_only ? 1.0 : a.dt_override >= 0 ? a.dt_override : a.sc->dt;
  const bool use_k = !a.rhs_only && a.rka != 0.0;
  const int l = lane & 3, row = lane >> 2, el = C::elem(lane >> 2);
  auto mt0 = [](int c) { return c == 0 ? 0 : MT0 + (c - 1) * MTB; };
  double acc[MTT][2];
  auto mma = [&](int ks, double h0, double h1, double h2, double h3) {
    const double *A = sA + (long)ks * MTT * 32 + lane;
#pragma unroll
    for (int m = 0; m < MT0; m++) dmma(acc[m], A[m * 32], h0);
#pragma unroll
    for (int m = 0; m < MTB; m++) {
      dmma(acc[mt0(1) + m], A[(mt0(1) + m) * 32], h1);
      dmma(acc[mt0(2) + m], A[(mt0(2) + m) * 32], h2);
      dmma(acc[mt0(3) + m], A[(mt0(3) + m) * 32], h3);
    }
  };
  bool ok = true;
  int it = 0;
  for (long t = t0; t < ntiles; t += stride, it++) {
    const int b = it & 1;
    double *u = buf + b * C::S_U;
    const double *uE = u + el * Np;
    const double *V = a.erec + t * C::FLOW + lane, *W = V + C::F_V;
    const int4 *P = reinterpret_cast<const int4 *>(a.erec + t * C::FLOW + C::F_V + C::F_W) + lane;
    // neighbours, then the first traces: on their way under the volume k-steps
    int4 nb[KSF];
#pragma unroll
    for (int f = 0; f < KSF; f++) nb[f] = __ldg(P + f * 32);
    // Fscale tau / 2 of the element's faces, by label
    double s0, s1, s2, s3;
    {
      const double *fs = a.fscale + (t * E + el) * 4, *ta = a.tau + (t * E + el) * 4;
      s0 = 0.5 * __ldg(fs + f0) * __ldg(ta + f0);
      s1 = 0.5 * __ldg(fs + f1) * __ldg(ta + f1);
      s2 = 0.5 * __ldg(fs + f2) * __ldg(ta + f2);
      s3 = 0.5 * __ldg(fs + f3) * __ldg(ta + f3);
    }
#pragma unroll
    for (int m = 0; m < MTT; m++) acc[m][0] = acc[m][1] = 0.0;
    double up[FH][4];
    auto gather = [&](int f, double (&x)[4]) {
      x[0] = __ldg(a.u_in + nb[f].x);
      x[1] = __ldg(a.u_in + nb[f].y);
      x[2] = __ldg(a.u_in + nb[f].z);
      x[3] = __ldg(a.u_in + nb[f].w);
    };
#pragma unroll
    for (int f = 0; f < FH; f++) gather(f, up[f]);
    ok = __all_sync(0xffffffffu, mbar_wait(&full[b], (it >> 1) & 1, a.wait_cycles));
    if (!ok) break;
#pragma unroll 4
    for (int ks = 0; ks < KSV; ks++) {
      const int n = tvol[ks * 4 + l];
      const double u1 = uE[n & 0x3ff], u2 = uE[(n >> 10) & 0x3ff], u3 = uE[n >> 20];
      const double v1 = __ldg(V + ks * 96), v2 = __ldg(V + ks * 96 + 32),
                   v3 = __ldg(V + ks * 96 + 64);
      const double p3 = u3 * v3, s = fma(u2, v2, p3), d = fma(u2, v2, -p3);
      mma(ks, fma(u1, v1, s), fma(u1, v1, -s), fma(-u1, v1, d), -fma(u1, v1, d));
    }
    // the next tile's state, once the previous tile's store has read its buffer
    if (lane == 0 && t + stride < ntiles) {
      bulk_wait_read();
      fetch(t + stride, b ^ 1);
    }
    double2 kr[MTT];
    auto face = [&](int f, const double (&x)[4]) {
      // (padding positions repeat the last point: finite values, zero columns)
      const int4 q = tface[min(f * 4 + l, Nfp - 1)];
      const double *w = W + f * 128;
      const double w0 = __ldg(w), w1 = __ldg(w + 32), w2 = __ldg(w + 64), w3 = __ldg(w + 96);
      const double p0 = fma(uE[q.x & 0xffff], w0 + s0, x[0] * (w0 - s0));
      const double p1 = fma(uE[q.y & 0xffff], w1 + s1, x[1] * (w1 - s1));
      const double p2 = fma(uE[q.z & 0xffff], w2 + s2, x[2] * (w2 - s2));
      const double p3 = fma(uE[q.w & 0xffff], w3 + s3, x[3] * (w3 - s3));
      const double a0 = p0 + p1, a1 = p0 - p1, c = p2 + p3, d = p2 - p3;
      mma(KSV + f, a0 + c, a0 - c, a1 + d, a1 - d);
    };
    double *kt = a.kreg + t * C::S_U + 2 * l;
#pragma unroll
    for (int f = 0; f < FH; f++) face(f, up[f]);
    // the other traces and the register
#pragma unroll
    for (int f = FH; f < KSF; f++) gather(f, up[f - FH]);
#pragma unroll
    for (int c = 0; c < 4; c++)
#pragma unroll
      for (int m = 0; m < (c == 0 ? MT0 : MTB); m++) {
        const int r = C::krow(c, 8 * m + row);
        kr[mt0(c) + m] = make_double2(0.0, 0.0);
        if (use_k && r >= 0)
          kr[mt0(c) + m] = *reinterpret_cast<const double2 *>(kt + r * E);
      }
#pragma unroll
    for (int f = FH; f < KSF; f++) face(f, up[f - FH]);
    // acc = dt rhs + rka k, the new register; u += rkb * y, y from the four characters
    double un[MT0][2][4];
    int4 nd[MT0];
    double *const ue[2] = {u + C::elem(2 * l) * Np, u + C::elem(2 * l + 1) * Np};
    __syncwarp();   // u has been read for the last fluxes
#pragma unroll
    for (int m = 0; m < MT0; m++) {
      nd[m] = tout[8 * m + row];   // (empty slots name node 0)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        un[m][h][0] = ue[h][nd[m].x], un[m][h][1] = ue[h][nd[m].y];
        un[m][h][2] = ue[h][nd[m].z], un[m][h][3] = ue[h][nd[m].w];
      }
    }
#pragma unroll
    for (int c = 0; c < 4; c++)
#pragma unroll
      for (int m = 0; m < (c == 0 ? MT0 : MTB); m++) {
        const int r = C::krow(c, 8 * m + row), i = mt0(c) + m;
        acc[i][0] = dt * acc[i][0] + a.rka * kr[i].x;
        acc[i][1] = dt * acc[i][1] + a.rka * kr[i].y;
        if (!a.rhs_only && r >= 0)
          *reinterpret_cast<double2 *>(kt + r * E) = make_double2(acc[i][0], acc[i][1]);
      }
    __syncwarp();   // every lane has its old values
#pragma unroll
    for (int m = 0; m < MT0; m++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        double y0 = acc[m][h], y1, y2, y3;
        sym_characters<C>(acc, m, h, row, lane, y1, y2, y3);
        const double s01 = y0 + y1, d01 = y0 - y1, s23 = y2 + y3, d23 = y2 - y3;
        const double *const o = un[m][h];
        if (8 * m + row < C::R0) {
          ue[h][nd[m].x] = a.rhs_only ? s01 + s23 : o[0] + a.rkb * (s01 + s23);
          ue[h][nd[m].y] = a.rhs_only ? s01 - s23 : o[1] + a.rkb * (s01 - s23);
          ue[h][nd[m].z] = a.rhs_only ? d01 + d23 : o[2] + a.rkb * (d01 + d23);
          ue[h][nd[m].w] = a.rhs_only ? d01 - d23 : o[3] + a.rkb * (d01 - d23);
        }
      }
    const int ne = (int)min((long)E, (long)a.K - t * E);
    if (ne < E) {
      __syncwarp();
      for (int i = lane; i < ne * Np; i += 32) a.u_out[t * C::S_U + i] = u[i];
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (lane == 0 && ne == E) {
      bulk_s2g(a.u_out + t * C::S_U, u, 8u * C::S_U);
      bulk_commit();
    }
  }
  if (!ok) {
    atomicOr(&a.sc->flags, 4);
    mbar_wait(&full[it & 1], (it >> 1) & 1);   // the tile in flight settles
  }
  if (lane == 0) bulk_wait_all();
}

// Flow records of the uploaded mesh (see above), one thread per (tile, lane
// position).
template <int N>
__global__ void sym_flow_kernel(const double *__restrict__ image, const double *__restrict__ geo,
                                const double *__restrict__ nrm,
                                const double *__restrict__ fscale,
                                const double *__restrict__ vel, const int *__restrict__ vmapP,
                                long vs, long Kp, int K, int ntiles, double *__restrict__ flow) {
  using C = SymAdvCfg<N, 4>;
  constexpr int Np = C::Np, Nfp = C::Nfp, NFF = C::NFF, P32 = 32 * (C::KSV + C::KSF);
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= (long)ntiles * P32) return;
  const long t = i / P32;
  const int p = (int)(i - t * P32), ks = p / 32, lane = p % 32, l = lane & 3;
  const long k = t * 8 + C::elem(lane >> 2);
  const int *tab = reinterpret_cast<const int *>(image + C::S_A);
  double *F = flow + t * C::FLOW;
  if (ks < C::KSV) {
    const int x = tab[ks * 4 + l];
    for (int d = 0; d < 3; d++) {
      double v = 0.0;
      if (k < K) {
        const int n = tab[ks * 4 + ((x >> (16 + 2 * d)) & 3)] & 0xffff;
        for (int q = 0; q < 3; q++)
          v += (geo[(3 * d + q) * Kp + k] +
                (geo[q * Kp + k] + geo[(3 + q) * Kp + k] + geo[(6 + q) * Kp + k])) *
               vel[q * vs + k * Np + n];
      }
      F[(ks * 3 + d) * 32 + lane] = v;
    }
    return;
  }
  const int f = ks - C::KSV, j = min(f * 4 + l, Nfp - 1);
  int *P = reinterpret_cast<int *>(F + C::F_V + C::F_W) + (f * 32 + lane) * 4;
  for (int v = 0; v < 4; v++) {
    const int q = tab[C::T_VOL + j * 4 + v], node = q & 0xffff, fp = q >> 16, face = fp / Nfp;
    double w = 0.0;
    int nb = 0;
    if (k < K) {
      double vn = 0.0;
      for (int d = 0; d < 3; d++) vn += nrm[d * 4 * Kp + 4 * k + face] * vel[d * vs + k * Np + node];
      w = 0.5 * fscale[4 * k + face] * vn;
      nb = vmapP[k * NFF + fp];
    }
    F[C::F_V + (f * 4 + v) * 32 + lane] = w;
    P[v] = nb;
  }
}
