// FP64 advection stage on the symmetry-adapted operators of
// dglm_stage_sym.cuh (included by dglm_sym.cuh).
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

// Flux weights of a tile, read from its flow record (single meshes), or the
// lane's element's own for a velocity that is constant (batches).
struct FlowRecord {
  const double *V, *W;   // at the lane
  __device__ __forceinline__ double vol(int ks, int d) const {
    return __ldg(V + ks * 96 + 32 * d);
  }
  __device__ __forceinline__ double face(int f, int v) const {
    return __ldg(W + f * 128 + 32 * v);
  }
};
struct FlowConstant {
  double va[3], wf[4];
  __device__ __forceinline__ double vol(int, int d) const { return va[d]; }
  __device__ __forceinline__ double face(int, int v) const { return wf[v]; }
};

// The operator image in shared memory: fragments and tables.
struct SymAdvOp {
  const double *A;
  const int *tvol;       // nodes of the three images, 10 bits each
  const int4 *tface, *tout;
};
// Copies it there (all threads of the block; the caller synchronises).
template <class C>
__device__ __forceinline__ SymAdvOp sym_adv_operator(const double *image, double *sA, int *tabs,
                                                     int tid, int nt) {
  const double2 *src = reinterpret_cast<const double2 *>(image);
  double2 *dst = reinterpret_cast<double2 *>(sA);
  for (int i = tid; i < C::S_A / 2; i += nt) dst[i] = __ldg(src + i);
  const int *ts = reinterpret_cast<const int *>(image + C::S_A);
  // volume entries with the images' nodes in place of the shuffle lanes
  for (int i = tid; i < C::KSV * 4; i += nt) {
    const int q = i & ~3, x = __ldg(ts + i);
    tabs[i] = (__ldg(ts + (q | ((x >> 16) & 3))) & 0x3ff) |
              (__ldg(ts + (q | ((x >> 18) & 3))) & 0x3ff) << 10 |
              (__ldg(ts + (q | ((x >> 20) & 3))) & 0x3ff) << 20;
  }
  for (int i = tid; i < C::T_FACE + C::T_OUT; i += nt)
    tabs[C::KSV * 4 + i] = __ldg(ts + C::T_VOL + i);
  const int4 *tface = reinterpret_cast<const int4 *>(tabs + C::KSV * 4);
  return SymAdvOp{sA, tabs, tface, tface + C::T_FACE / 4};
}

// One tile by one warp, in its state buffer u: returns false when the wait
// for the buffer expired.  P: the tile's neighbour nodes at the lane, counted
// from ubase; s: Fscale tau / 2 of the lane's element's faces by label; kt: the
// tile's register.  wait() waits for the buffer, ahead() runs after the volume
// k-steps.
template <class C, class Flow, class Wait, class Ahead>
__device__ __forceinline__ bool sym_adv_tile(const SymAdvOp &op, double *u, const Flow &fl,
                                             const int4 *P, const double *ubase,
                                             const double (&s)[4], double *kt, double dt,
                                             double rka, double rkb, bool use_k, bool rhs_only,
                                             int lane, Wait wait, Ahead ahead) {
  constexpr int Np = C::Np, Nfp = C::Nfp, E = C::E, MTT = C::MTT, MT0 = C::MT0, MTB = C::MTB,
                KSF = C::KSF, KSV = C::KSV, FH = C::FH;
  const int l = lane & 3, row = lane >> 2;
  const double *uE = u + C::elem(lane >> 2) * Np;
  auto mt0 = [](int c) { return c == 0 ? 0 : MT0 + (c - 1) * MTB; };
  double acc[MTT][2];
  auto mma = [&](int ks, double h0, double h1, double h2, double h3) {
    const double *A = op.A + (long)ks * MTT * 32 + lane;
#pragma unroll
    for (int m = 0; m < MT0; m++) dmma(acc[m], A[m * 32], h0);
#pragma unroll
    for (int m = 0; m < MTB; m++) {
      dmma(acc[mt0(1) + m], A[(mt0(1) + m) * 32], h1);
      dmma(acc[mt0(2) + m], A[(mt0(2) + m) * 32], h2);
      dmma(acc[mt0(3) + m], A[(mt0(3) + m) * 32], h3);
    }
  };
  // neighbours, then the first traces: on their way under the volume k-steps.
  // (The traces are asked for after two k-steps, which cover the latency of
  // their addresses; before the first the warp waits for those: N=5, K=93,750
  // 981 us per two steps against 924, N=6, K=63,888 1,222 against 1,152.)
  int4 nb[KSF];
#pragma unroll
  for (int f = 0; f < KSF; f++) nb[f] = __ldg(P + f * 32);
#pragma unroll
  for (int m = 0; m < MTT; m++) acc[m][0] = acc[m][1] = 0.0;
  double up[FH][4];
  // (the state is written by the launch before: plain loads, see launch_pdl)
  auto gather = [&](int f, double (&x)[4]) {
    x[0] = ubase[nb[f].x];
    x[1] = ubase[nb[f].y];
    x[2] = ubase[nb[f].z];
    x[3] = ubase[nb[f].w];
  };
  if (!wait()) return false;
  auto volume = [&](int ks) {
    const int n = op.tvol[ks * 4 + l];
    const double u1 = uE[n & 0x3ff], u2 = uE[(n >> 10) & 0x3ff], u3 = uE[n >> 20];
    const double v1 = fl.vol(ks, 0), v2 = fl.vol(ks, 1), v3 = fl.vol(ks, 2);
    const double p3 = u3 * v3, sum = fma(u2, v2, p3), d = fma(u2, v2, -p3);
    mma(ks, fma(u1, v1, sum), fma(u1, v1, -sum), fma(-u1, v1, d), -fma(u1, v1, d));
  };
  constexpr int K0 = 2;
  static_assert(K0 <= KSV, "k-steps before the gathers");
#pragma unroll
  for (int ks = 0; ks < K0; ks++) volume(ks);
#pragma unroll
  for (int f = 0; f < FH; f++) gather(f, up[f]);
#pragma unroll 4
  for (int ks = K0; ks < KSV; ks++) volume(ks);
  ahead();
  auto face = [&](int f, const double (&x)[4]) {
    // (padding positions repeat the last point: finite values, zero columns)
    const int4 q = op.tface[min(f * 4 + l, Nfp - 1)];
    const double w0 = fl.face(f, 0), w1 = fl.face(f, 1), w2 = fl.face(f, 2), w3 = fl.face(f, 3);
    const double p0 = fma(uE[q.x & 0xffff], w0 + s[0], x[0] * (w0 - s[0]));
    const double p1 = fma(uE[q.y & 0xffff], w1 + s[1], x[1] * (w1 - s[1]));
    const double p2 = fma(uE[q.z & 0xffff], w2 + s[2], x[2] * (w2 - s[2]));
    const double p3 = fma(uE[q.w & 0xffff], w3 + s[3], x[3] * (w3 - s[3]));
    const double a0 = p0 + p1, a1 = p0 - p1, c = p2 + p3, d = p2 - p3;
    mma(KSV + f, a0 + c, a0 - c, a1 + d, a1 - d);
  };
  kt += 2 * l;
#pragma unroll
  for (int f = 0; f < FH; f++) face(f, up[f]);
  // the other traces and the register
#pragma unroll
  for (int f = FH; f < KSF; f++) gather(f, up[f - FH]);
  double2 kr[MTT];
#pragma unroll
  for (int c = 0; c < 4; c++)
#pragma unroll
    for (int m = 0; m < (c == 0 ? MT0 : MTB); m++) {
      const int r = C::krow(c, 8 * m + row);
      kr[mt0(c) + m] = make_double2(0.0, 0.0);
      if (use_k && r >= 0) kr[mt0(c) + m] = *reinterpret_cast<const double2 *>(kt + r * E);
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
    nd[m] = op.tout[8 * m + row];   // (empty slots name node 0)
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
      acc[i][0] = dt * acc[i][0] + rka * kr[i].x;
      acc[i][1] = dt * acc[i][1] + rka * kr[i].y;
      if (!rhs_only && r >= 0)
        *reinterpret_cast<double2 *>(kt + r * E) = make_double2(acc[i][0], acc[i][1]);
    }
  __syncwarp();   // every lane has its old values
#pragma unroll
  for (int m = 0; m < MT0; m++)
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const double y0 = acc[m][h];
      double y1, y2, y3;
      sym_characters<C>(acc, m, h, row, lane, y1, y2, y3);
      const double s01 = y0 + y1, d01 = y0 - y1, s23 = y2 + y3, d23 = y2 - y3;
      const double *const o = un[m][h];
      if (8 * m + row < C::R0) {
        ue[h][nd[m].x] = rhs_only ? s01 + s23 : o[0] + rkb * (s01 + s23);
        ue[h][nd[m].y] = rhs_only ? s01 - s23 : o[1] + rkb * (s01 - s23);
        ue[h][nd[m].z] = rhs_only ? d01 + d23 : o[2] + rkb * (d01 + d23);
        ue[h][nd[m].w] = rhs_only ? d01 - d23 : o[3] + rkb * (d01 - d23);
      }
    }
  return true;
}

template <int N, int NW>
__global__ void __launch_bounds__(32 * NW, 1)
    stage_sym_adv_kernel(const StageArgs a, int ntiles) {
  using C = SymAdvCfg<N, NW>;
  constexpr int Np = C::Np, E = C::E;
  extern __shared__ __align__(16) double smem[];
  double *sA = smem, *sBuf = sA + C::S_A;
  unsigned long long *bars = reinterpret_cast<unsigned long long *>(sBuf + NW * 2 * C::S_U);
  int *tabs = reinterpret_cast<int *>(bars + NW * 2);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  double *buf = sBuf + warp * 2 * C::S_U;
  unsigned long long *full = bars + 2 * warp;
  if (lane == 0) {
    mbar_init(&full[0], 1);
    mbar_init(&full[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  const long stride = (long)gridDim.x * NW, t0 = blockIdx.x + (long)gridDim.x * warp;
  auto fetch = [&](long t, int b) {   // lane 0
    mbar_arrive_expect_tx(&full[b], 8u * C::S_U);
    bulk_g2s(buf + b * C::S_U, a.u_in + t * C::S_U, 8u * C::S_U, &full[b]);
  };
  pdl_launch();
  const SymAdvOp op = sym_adv_operator<C>(a.AT, sA, tabs, tid, C::THREADS);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncthreads();
  pdl_wait();
  if (lane == 0 && t0 < ntiles) fetch(t0, 0);
  const int *ft = reinterpret_cast<const int *>(a.AT + C::S_A) + C::T_VOL + C::T_FACE + C::T_OUT;
  const int fo[4] = {__ldg(ft), __ldg(ft + 1), __ldg(ft + 2), __ldg(ft + 3)};
  const double dt = a.rhs_only ? 1.0 : a.dt_override >= 0 ? a.dt_override : a.sc->dt;
  const bool use_k = !a.rhs_only && a.rka != 0.0;
  const int el = C::elem(lane >> 2);
  bool ok = true;
  int it = 0;
  for (long t = t0; t < ntiles; t += stride, it++) {
    const int b = it & 1;
    double *u = buf + b * C::S_U;
    const double *F = a.erec + t * C::FLOW;
    double s[4];
#pragma unroll
    for (int v = 0; v < 4; v++)
      s[v] = 0.5 * __ldg(a.fscale + (t * E + el) * 4 + fo[v]) *
             a.tau[(t * E + el) * 4 + fo[v]];
    ok = sym_adv_tile<C>(
        op, u, FlowRecord{F + lane, F + C::F_V + lane},
        reinterpret_cast<const int4 *>(F + C::F_V + C::F_W) + lane, a.u_in, s,
        a.kreg + t * C::S_U, dt, a.rka, a.rkb, use_k, a.rhs_only != 0, lane,
        [&]() {
          return __all_sync(0xffffffffu, mbar_wait(&full[b], (it >> 1) & 1, a.wait_cycles)) != 0;
        },
        [&]() {
          // the next tile's state, once the previous tile's store has read its buffer
          if (lane == 0 && t + stride < ntiles) {
            bulk_wait_read();
            fetch(t + stride, b ^ 1);
          }
        });
    if (!ok) break;
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
