// FP64 Euler stage kernel on symmetry-adapted operators (included by
// dglm_sym.cuh).
//
// The nodes of the reference tetrahedron are symmetric under the four vertex
// permutations V4 = {id, (01)(23), (02)(13), (03)(12)}.  With the barycentric
// derivative operators W_v (v = 0..3, sum zero; WD_a = W_a - W_0) and node
// permutations P_v (vertex i -> vertex i^v), W_v = P_v W_0 P_v, and the lift of
// the face opposite vertex v is P_v L_0 P_v likewise.  The right-hand side of a
// column is then
//   y = sum_v P_v W_0 (P_v g_v) - sum_v P_v L_0 (P_v phi_v)
// for contravariant fluxes g_v (free up to a common term per node; g_0 = 0
// here, so g_a = (grad r_a + sum_b grad r_b) . F, a = 1..3) and face fluxes
// phi_v.  Projecting on the four characters chi of V4,
//   y_chi = (E_chi W_0) h_chi - (E_chi L_0) h^F_chi,
//   h_chi = sum_v chi(v) P_v g_v,  h^F_chi = sum_v chi(v) P_v phi_v,
// and y_chi is fixed by one value per orbit of nodes.  So the contraction has
// about Np/4 rows per character over Np + Nfp columns: Np (Np + Nfp)
// multiply-adds per column instead of Np (3 Np + 4 Nfp) (N=4: 65 m8n8k4 MMAs
// per eight columns instead of 210, tiles' padding included), and the operator
// is as much smaller (N=6: 86 KB, it fits shared memory; 258 KB before).  The
// sums over V4 are additions: the arithmetic stays FP64 throughout.
//
// How it is laid out.  A warp forms its B fragments in registers: lane 4 c + l
// handles MMA column c (an element of the tile) and the l-th node of an orbit
// (one k-step = one orbit); h_chi needs g_a at node l^a, a quad shuffle away,
// and in a face k-step one lane forms its node's four faces' flux values
// itself.  No flux goes through shared memory.
//   group    2 NS compute warps that share a tile of 8 elements: NS pairs, each
//            with its variables; a pair splits the k-steps, exchanges partial
//            sums (in the place of the tile's traces) and finishes half of the
//            variables each.  Groups walk the tiles independently: the only
//            waits are on mbarriers of the tile or the group.
//   movers   bring a tile's state, records and penalty in and its new state
//            out by bulk copies; the update is made in place.
//   gatherers  the traces of neighbours outside the tile (cp.async).
//   k        the RK register is kept in fragment order (tile, variable,
//            operator row, column): compute warps load and store it straight
//            from registers, in full sectors.
// Bound by (N=4, K=196,608): nothing alone.  The FP64 pipe needs 2.4k cycles per
// tile (MMAs 1.4k, flux arithmetic 1.0k: counters of profiles/) and HBM 2.0k; a
// tile takes 4.7k, where the warps wait on shared memory (a third of it the
// update's and the traces' scattered nodes), on the shared FP64 pipe (a warp's
// flux arithmetic gets one slot per MMA of the other's) and on each other.
// 0.399 ms per stage against 0.780 of the dense pipelined kernel; N=3
// (K=105,456) 0.136 against 0.201, N=5 (K=82,944) 0.420 against 0.674, N=6
// (K=82,944, where a thread spills 100 bytes) 0.800 against 1.243.
// Measured and not kept: each warp on its own tile with the traces gathered
// into registers (0.698; the gathers stall the load path), one warp of the pair
// on the volume k-steps and the other on faces and update (0.53), twelve
// compute warps with the variables split in two (0.54; the flux arithmetic is
// repeated).
// Every mbarrier wait is bounded; on expiry a warp sets flag bit 2 of the
// device scalars, waits for its copies and leaves, and the others' waits expire.
#pragma once

// sizes of the symmetry-adapted operators of order N
template <int N>
struct SymSize {
  static constexpr int Np = np_of(N), Nfp = nfp_of(N), NFF = 4 * Nfp;
  static constexpr int FIX = N % 2 ? 0 : N / 2 + 1;        // nodes fixed by an involution
  static constexpr int N1 = N % 4 == 0 ? 1 : 0;            // the centroid
  static constexpr int N2 = (FIX - N1) / 2;                // orbits of size 2 per involution
  static constexpr int N4 = (Np - 6 * N2 - N1) / 4;        // orbits of size 4
  static constexpr int R0 = N4 + 3 * N2 + N1, RB = N4 + N2;   // rows of chi_0, chi_1..3
  static constexpr int MT0 = (R0 + 7) / 8, MTB = (RB + 7) / 8, MTT = MT0 + 3 * MTB;
  // chi_b's rows of the size-2 orbits sit in chi_0's slots of the same orbits
  // where the m-tiles have room, else right after the size-4 rows
  static constexpr bool ALIGNED = N4 + 3 * N2 <= 8 * MTB;
  static constexpr int KSV = (Np + 3) / 4, KSF = (Nfp + 3) / 4, KS = KSV + KSF;
  // operator image: fragments [k-step][m-tile][lane] doubles, then the tables
  // (ints): volume k positions, face k positions, output slots, face labels,
  // and per face point of a tile its trace slot and code position
  static constexpr int S_A = KS * MTT * 32;
  static constexpr int T_VOL = KSV * 4, T_FACE = KSF * 4 * 4, T_OUT = 8 * MT0 * 4;
  static constexpr int T_SLOT = 8 * NFF;
  static constexpr int TABS = T_VOL + T_FACE + T_OUT + 4 + T_SLOT;
  // MMA column -> element of the tile, and back; and the doubles between the
  // tile's first and last four elements in shared memory.  Chosen over all
  // splits of the columns so that the lanes' nodes spread over the banks (mean
  // conflict degree of the volume, face and update accesses; N=3: 2.0, 1.3,
  // 1.5; N=4: 2.6, 2.3, 2.0; N=5: 1.9, 1.8, 1.5, in order and without the gap
  // 2.9, 2.5, 5.0; N=6: 2.2, 2.0, 1.7).
  static constexpr unsigned ORDER = N == 4 ? 0x73516240u : N == 5 ? 0x65217430u : 0x65437210u;
  static constexpr int GAP = N == 5 ? 4 : 0;
  __host__ __device__ static constexpr int elem(int c) { return (ORDER >> 4 * c) & 7; }
  __host__ __device__ static constexpr int col(int e) {
    for (int c = 0; c < 8; c++)
      if (elem(c) == e) return c;
    return 0;
  }
  // neighbour traces [v][column][UPS], position Nfp label + j; UPS = 4 (mod 8), so
  // that four consecutive points of four elements are on distinct bank pairs.
  // Neighbour codes, 4 x 16 bits per (column, face k position), stride NBS.
  static constexpr int UPS = NFF % 8 == 4 ? NFF : NFF + 4, NBS = 4 * KSF + 1;
  // slot of chi_b's row for the i-th size-2 orbit of involution b, and of chi_0's
  __host__ __device__ static constexpr int slot0(int b, int i) { return N4 + (b - 1) * N2 + i; }
  __host__ __device__ static constexpr int slotb(int b, int i) {
    return ALIGNED ? slot0(b, i) : N4 + i;
  }
  // compact index (0..Np-1) of row `slot` of character c in the RK register's
  // layout, -1 for an empty slot
  __host__ __device__ static constexpr int krow(int c, int slot) {
    if (c == 0) return slot < R0 ? slot : -1;
    const int base = R0 + (c - 1) * RB;
    if (slot < N4) return base + slot;
    const int i = slot - slotb(c, 0);
    return i >= 0 && i < N2 ? base + N4 + i : -1;
  }
};

template <int N, int NS_, int NG_, int NB_>
struct SymCfg : SymSize<N> {
  using Z = SymSize<N>;
  static constexpr int E = 8, NV = 5;
  static constexpr int NS = NS_, NG = NG_, NB = NB_;
  static constexpr int WPG = 2 * NS;                       // warps per group
  static constexpr int NWC = NG * WPG, PW = 8;             // compute and loader warps
  static constexpr int THREADS = 32 * (NWC + PW);
  // loader warps: NM movers, and NL x GP gatherers (GP share a tile); each
  // serves its own buffers, so it sees every phase of their barriers and a
  // parity wait is never two off
  static constexpr int NM = NB % 2 == 0 ? 2 : 1, NL = NB == 8 ? 4 : NB, GP = (PW - NM) / NL;
  static_assert(NB % NM == 0 && NB % NL == 0 && GP >= 1, "loader warps");
  // registers per thread: of the launch, and after the split between compute
  // and loader warps (multiples of 8 whose sum is the launch's)
  static constexpr int REG0 = 65536 / THREADS / 8 * 8, REGP = N == 6 ? 32 : N == 5 ? 48 : 40,
                       REGC = (REG0 * (NWC + PW) - REGP * PW) / NWC / 8 * 8;
  // state [v][element][node], one bulk copy per variable (two around the gap).
  // (Bulk copies cost some 80 cycles of the mover each, whatever their size:
  // with a pad after every pair of elements, 20 per tile, the copies alone
  // took longer than the tile's MMAs at N=4.)
  static constexpr int VS = E * Z::Np + Z::GAP, CPV = Z::GAP ? 2 : 1;
  static constexpr int S_U = NV * VS, S_REC = E * kRecord, S_TAU = 4 * E;
  static constexpr int S_TR = NV * E * Z::UPS;
  static constexpr int S_NB = Z::NBS * E;
  static constexpr int S_BUF = S_U + S_REC + S_TAU + S_TR + S_NB;
  static constexpr unsigned TX = 8u * (NV * E * Z::Np + S_REC + S_TAU);
  // element -> offset in the state
  __host__ __device__ static constexpr int eoff(int e) {
    return e * Z::Np + (e >= E / 2 ? Z::GAP : 0);
  }
  static constexpr int NVW = (NV + NS - 1) / NS;   // variables of a warp (the last has fewer)
  static constexpr int NBAR = 4 * NB + 2 * NG;   // full, trace, done, tile numbers; read, dump
  // face points of a tile per lane, per lane of one gatherer, and per batch of
  // index loads
  static constexpr int GPL = E * Z::NFF / 32, GPW = (GPL + GP - 1) / GP, GCH = N == 6 ? 3 : N == 5 ? 5 : 4;
  static constexpr size_t SMEM =
      sizeof(double) * (Z::S_A + (size_t)NB * S_BUF + NBAR) + sizeof(int) * Z::TABS;
  static_assert(NWC % 4 == 0, "whole warpgroups of compute warps");
  static_assert(REGC <= 255 && REGC * NWC + REGP * PW <= REG0 * (NWC + PW), "register split");
  static_assert(VS % 2 == 0 && (E / CPV * Z::Np + Z::GAP) % 2 == 0 && VS < 32768,
                "16-byte aligned copies, 16-bit codes");
  static_assert(SMEM <= 232448, "shared memory per CTA exceeds 227 KB");
  static_assert(NV * Z::MTT * 64 <= S_TR, "partial sums reuse the traces");
};

__device__ __forceinline__ void bulk_s2g(void *dst, const void *src, unsigned bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst),
               "r"(smem_u32(src)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() {
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
__device__ __forceinline__ void bulk_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}
__device__ __forceinline__ void bulk_wait_all() {
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}
// 1/x by Newton's iteration from the hardware's approximation, branch-free: two
// steps take its 2^-23 below the rounding of the last, so the result is within
// an ulp of the rounded quotient where x and 1/x are normal numbers.  Outside,
// unlike the division: 0, subnormal numbers and infinities give NaN, and from
// 2^1022 on the result is 0 (densities below 2.2e-308 or above 4.5e307).  With
// 1.0 / x a step takes 5 % longer at N=3, 3.5 % at N=4, 7 % at N=5; with a range
// check and a second pass with divisions for the tiles that fail it 1 to 3 %.
__device__ __forceinline__ double recip(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  y = fma(y, fma(-x, y, 1.0), y);
  return fma(y, fma(-x, y, 1.0), y);
}
// as dmma_8x8x4, free to be scheduled among the flux arithmetic
__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}
__device__ __forceinline__ void bulk_prefetch_l2(const void *src, unsigned bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
}

// chi_1..chi_3 values of this lane's slot of chi_0's m-tile m, column half h
// (m is a literal after unrolling; the whole warp takes part).
template <class C>
__device__ __forceinline__ void sym_characters(const double (&acc)[C::MTT][2], int m, int h,
                                               int row, int lane, double &y1, double &y2,
                                               double &y3) {
  constexpr int MT0 = C::MT0, MTB = C::MTB;
  const int mb = m < MTB ? m : 0;
  if constexpr (C::ALIGNED || C::N2 == 0) {
    y1 = m < MTB ? acc[MT0 + mb][h] : 0.0;
    y2 = m < MTB ? acc[MT0 + MTB + mb][h] : 0.0;
    y3 = m < MTB ? acc[MT0 + 2 * MTB + mb][h] : 0.0;
  } else {
    // size-2 orbits: chi_1's rows are in chi_0's slots of involution 1; those
    // of chi_2 and chi_3 sit in the same rows of their last tile
    constexpr int ML = MTB - 1, RS = C::N4 - 8 * ML;   // first special row of that tile
    static_assert(C::N4 + C::N2 == 8 * MTB && MT0 == MTB + 1, "layout of the size-2 rows");
    if (m < MTB) {
      const bool sp = m == ML && row >= RS;
      y1 = acc[MT0 + mb][h];
      y2 = sp ? 0.0 : acc[MT0 + MTB + mb][h];
      y3 = sp ? 0.0 : acc[MT0 + 2 * MTB + mb][h];
    } else {
      const int src = (RS + (row < C::N2 ? row : row - C::N2)) * 4 + (lane & 3);
      const double t2 = __shfl_sync(0xffffffffu, acc[MT0 + MTB + ML][h], src & 31);
      const double t3 = __shfl_sync(0xffffffffu, acc[MT0 + 2 * MTB + ML][h], src & 31);
      y1 = 0.0;
      y2 = row < C::N2 ? t2 : 0.0;
      y3 = row >= C::N2 && row < 2 * C::N2 ? t3 : 0.0;
    }
  }
}

// One warp's share of a tile's stage: variables [V0, V0 + NVW).
template <class C, int V0, int NVW>
struct SymWarp {
  static constexpr int Np = C::Np, Nfp = C::Nfp, NFF = C::NFF, E = C::E, MTT = C::MTT,
                       MT0 = C::MT0, MTB = C::MTB;
  double acc[NVW][MTT][2];

  // first m-tile of character c
  __device__ static constexpr int mt0(int c) { return c == 0 ? 0 : MT0 + (c - 1) * MTB; }

  // compact RK-register row of this lane's row of m-tile m of character c (-1: none)
  __device__ static __forceinline__ int krow(int c, int m, int row) {
    return C::krow(c, 8 * m + row);
  }

  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int v = 0; v < NVW; v++)
#pragma unroll
      for (int m = 0; m < MTT; m++) acc[v][m][0] = acc[v][m][1] = 0.0;
  }
  // this lane's rows of the RK register of variable V0 + v
  __device__ __forceinline__ void load_k(const double *k, bool use, int v, int lane,
                                         double2 (&kr)[MTT]) const {
    const int row = lane >> 2, c2 = (lane & 3) * 2;
#pragma unroll
    for (int c = 0; c < 4; c++)
#pragma unroll
      for (int m = 0; m < (c == 0 ? MT0 : MTB); m++) {
        const int r = krow(c, m, row);
        double2 x = make_double2(0.0, 0.0);
        if (use && r >= 0 && v < NVW)
          x = *reinterpret_cast<const double2 *>(k + ((V0 + v) * Np + r) * E + c2);
        kr[mt0(c) + m] = x;
      }
  }
  __device__ __forceinline__ void store_k(double *k, int v, int lane) const {
    const int row = lane >> 2, c2 = (lane & 3) * 2;
#pragma unroll
    for (int c = 0; c < 4; c++)
#pragma unroll
      for (int m = 0; m < (c == 0 ? MT0 : MTB); m++) {
        const int r = krow(c, m, row);
        if (r >= 0)
          *reinterpret_cast<double2 *>(k + ((V0 + v) * Np + r) * E + c2) =
              make_double2(acc[v][mt0(c) + m][0], acc[v][mt0(c) + m][1]);
      }
  }
  // variables the pair's warp kc finishes: the first VH, or the others
  static constexpr int VH = (NVW + 1) / 2;
  __device__ static __forceinline__ bool owns(int kc, int v) { return (kc == 0) == (v < VH); }
  // partial sums of the variables the pair's other warp finishes -> px
  __device__ __forceinline__ void dump(double2 *px, int kc, int lane) const {
#pragma unroll
    for (int v = 0; v < NVW; v++)
      if (!owns(kc, v))
#pragma unroll
      for (int m = 0; m < MTT; m++)
        px[((V0 + v) * MTT + m) * 32 + lane] = make_double2(acc[v][m][0], acc[v][m][1]);
  }
  // acc[v] += A of k-step ks times the fragments h[chi]
  __device__ __forceinline__ void mma(int v, const double (&A)[MTT], double h0, double h1,
                                      double h2, double h3) {
#pragma unroll
    for (int m = 0; m < MT0; m++) dmma(acc[v][m], A[m], h0);
#pragma unroll
    for (int m = 0; m < MTB; m++) {
      dmma(acc[v][mt0(1) + m], A[mt0(1) + m], h1);
      dmma(acc[v][mt0(2) + m], A[mt0(2) + m], h2);
      dmma(acc[v][mt0(3) + m], A[mt0(3) + m], h3);
    }
  }
  __device__ __forceinline__ void load_A(double (&A)[MTT], const double *sA, int ks, int lane) {
#pragma unroll
    for (int m = 0; m < MTT; m++) A[m] = sA[(ks * MTT + m) * 32 + lane];
  }

  // volume k-steps: the state of the lane's node of an orbit, its
  // contravariant fluxes (mr: 9 metrics of the lane's element, gauge g_0 = 0),
  // their sums over V4 and the MMAs
  struct Node {
    double q[5];
    int tab;
  };
  __device__ __forceinline__ void load_node(const double *bE, int tab, Node &n) const {
    const double *u = bE + (tab & 0xffff);
    n.tab = tab;
#pragma unroll
    for (int v = 0; v < 5; v++) n.q[v] = u[v * C::VS];
  }
  __device__ __forceinline__ void fluxes(const Node &n, const double (&mr)[9], double gamma,
                                         double (&g)[3][NVW]) const {
    const double r = n.q[0], m1 = n.q[1], m2 = n.q[2], m3 = n.q[3], en = n.q[4];
    const double ir = recip(r);
    const double vx = m1 * ir, vy = m2 * ir, vz = m3 * ir;
    const double p = (gamma - 1) * (en - 0.5 * (m1 * vx + m2 * vy + m3 * vz));
    const double H = en + p;
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const double ax = mr[3 * d], ay = mr[3 * d + 1], az = mr[3 * d + 2];
      const double V = ax * vx + ay * vy + az * vz;
#pragma unroll
      for (int v = 0; v < NVW; v++)
        g[d][v] = V0 + v == 0   ? r * V
                  : V0 + v == 1 ? m1 * V + p * ax
                  : V0 + v == 2 ? m2 * V + p * ay
                  : V0 + v == 3 ? m3 * V + p * az
                                : H * V;
    }
  }
  __device__ __forceinline__ void volume(const double (&g)[3][NVW], const double *sA, int tab,
                                         int ks, int lane) {
    double A[MTT];
    load_A(A, sA, ks, lane);
    const int quad = lane & ~3, s1 = quad | ((tab >> 16) & 3), s2 = quad | ((tab >> 18) & 3),
              s3 = quad | ((tab >> 20) & 3);
#pragma unroll
    for (int v = 0; v < NVW; v++) {
      const double x1 = __shfl_sync(0xffffffffu, g[0][v], s1);
      const double x2 = __shfl_sync(0xffffffffu, g[1][v], s2);
      const double x3 = __shfl_sync(0xffffffffu, g[2][v], s3);
      const double s = x2 + x3, d = x2 - x3;
      mma(v, A, x1 + s, x1 - s, d - x1, -(x1 + d));
    }
  }

  // flux of one face point: the sum form F(um + up) = 2 F(ub), the halves in
  // the face data (c n and c, c = Fscale / 2).  bE, bF, bT: at the
  // lane's element; code >= 0: the neighbour node is in this tile, at that
  // offset of the state bU; code < 0: its trace was gathered to up
  __device__ __forceinline__ void face_point(const double *bU, const double *bE,
                                             const double *bF, const double *bT,
                                             const double *up, int code, int node, int f,
                                             double gamma, double (&phi)[NVW]) {
    const double *u = bE + node;
    const double *F = bF + 9 + f;
    const double nx = F[0], ny = F[4], nz = F[8], tau = F[12] * bT[f];
    const double *q = code >= 0 ? bU + code : up;
    const int qs = code >= 0 ? C::VS : E * C::UPS;
    double s[5], d[5];
#pragma unroll
    for (int v = 0; v < 5; v++) {
      const double um = u[v * C::VS], uv = q[v * qs];
      s[v] = um + uv;
      d[v] = uv - um;
    }
    // (velocities first, as in the dense kernels: the square of a momentum
    // leaves the range of doubles long before the state does)
    const double ir = recip(s[0]);
    const double mn = nx * s[1] + ny * s[2] + nz * s[3];
    const double vx = s[1] * ir, vy = s[2] * ir, vz = s[3] * ir, vn = mn * ir;
    const double p = (gamma - 1) * (s[4] - 0.5 * (s[1] * vx + s[2] * vy + s[3] * vz));
#pragma unroll
    for (int v = 0; v < NVW; v++) {
      const double fl = V0 + v == 0   ? mn
                        : V0 + v == 1 ? s[1] * vn + p * nx
                        : V0 + v == 2 ? s[2] * vn + p * ny
                        : V0 + v == 3 ? s[3] * vn + p * nz
                                      : (s[4] + p) * vn;
      phi[v] = fl - tau * d[V0 + v];
    }
  }
  // q: node per face label, nb: neighbour codes per label
  __device__ __forceinline__ void face(const double *bU, const double *bE, const double *bF,
                                       const double *bT, const double *up, const double *sA,
                                       int4 q, short4 nb, int4 faces, int ks, double gamma,
                                       int lane) {
    double p0[NVW], p1[NVW], a0[NVW], a1[NVW];
    face_point(bU, bE, bF, bT, up, nb.x, q.x & 0xffff, faces.x, gamma, p0);
    face_point(bU, bE, bF, bT, up + Nfp, nb.y, q.y & 0xffff, faces.y, gamma, p1);
#pragma unroll
    for (int v = 0; v < NVW; v++) {
      a0[v] = p0[v] + p1[v];
      a1[v] = p0[v] - p1[v];
    }
    face_point(bU, bE, bF, bT, up + 2 * Nfp, nb.z, q.z & 0xffff, faces.z, gamma, p0);
    face_point(bU, bE, bF, bT, up + 3 * Nfp, nb.w, q.w & 0xffff, faces.w, gamma, p1);
    double A[MTT];
    load_A(A, sA, ks, lane);
#pragma unroll
    for (int v = 0; v < NVW; v++) {
      const double c = p0[v] + p1[v], d = p0[v] - p1[v];
      mma(v, A, a0[v] + c, a0[v] - c, a1[v] + d, a1[v] - d);
    }
  }

  // acc[v] = dt (acc[v] + the other warp's) + rka k, the new register, and
  // u += rkb * y of variable V0 + v in place (rhs_only: u = y), y from the four
  // characters.  All of a variable's loads are made before its first store, so
  // that their latencies overlap.
  __device__ __forceinline__ void update(double *bU, const double2 *px, const int4 *tout, int v,
                                         double dt, double rka, const double2 (&kr)[MTT],
                                         double rkb, bool rhs, int lane) {
    const int row = lane >> 2, c2 = (lane & 3) * 2;
    double2 x[MTT];
#pragma unroll
    for (int m = 0; m < MTT; m++) x[m] = px[((V0 + v) * MTT + m) * 32 + lane];
    double *const u0 = bU + (V0 + v) * C::VS + C::eoff(C::elem(c2));
    double *const u1 = bU + (V0 + v) * C::VS + C::eoff(C::elem(c2 + 1));
    double un[MT0][2][4];
    int4 nd[MT0];
#pragma unroll
    for (int m = 0; m < MT0; m++) {
      nd[m] = tout[8 * m + row];   // (empty slots name node 0)
      un[m][0][0] = u0[nd[m].x], un[m][0][1] = u0[nd[m].y];
      un[m][0][2] = u0[nd[m].z], un[m][0][3] = u0[nd[m].w];
      un[m][1][0] = u1[nd[m].x], un[m][1][1] = u1[nd[m].y];
      un[m][1][2] = u1[nd[m].z], un[m][1][3] = u1[nd[m].w];
    }
#pragma unroll
    for (int m = 0; m < MTT; m++) {
      acc[v][m][0] = dt * (acc[v][m][0] + x[m].x) + rka * kr[m].x;
      acc[v][m][1] = dt * (acc[v][m][1] + x[m].y) + rka * kr[m].y;
    }
#pragma unroll
    for (int m = 0; m < MT0; m++) {
      const int slot = 8 * m + row;
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const double y0 = acc[v][m][h];
        double y1, y2, y3;
        sym_characters<C>(acc[v], m, h, row, lane, y1, y2, y3);
        const double s01 = y0 + y1, d01 = y0 - y1, s23 = y2 + y3, d23 = y2 - y3;
        double *const u = h ? u1 : u0;
        const double *const o = un[m][h];
        // the four nodes of an orbit of size 2 or 1 repeat: equal values are written
        if (slot < C::R0) {
          u[nd[m].x] = rhs ? s01 + s23 : o[0] + rkb * (s01 + s23);
          u[nd[m].y] = rhs ? s01 - s23 : o[1] + rkb * (s01 - s23);
          u[nd[m].z] = rhs ? d01 + d23 : o[2] + rkb * (d01 + d23);
          u[nd[m].w] = rhs ? d01 - d23 : o[3] + rkb * (d01 - d23);
        }
      }
    }
  }
};

// Buffers and barriers of a CTA: NB tile buffers; per buffer the arrival of the
// bulk copies (full), of the traces (trace) and of the finished update (done),
// and the number of the tile it is being loaded with (seq).  A group may get
// to a buffer before the tile that precedes its own there is through; seq
// tells it when a parity wait means its own tile.  Per group: all its warps
// have read the tile's state and traces (read), the partial sums are in the
// traces' place (dump).
struct SymRing {
  double *buf0;
  unsigned long long *full, *trace, *done, *read, *dump;
  volatile int *seq;
};

// Mover warp mw of NM: the tiles it = mw, mw + NM, ... in order: once the compute warps are done with a buffer's
// tile, sends its new state out and brings in the next tile's state, records
// and penalty by bulk copies.
template <class C>
__device__ __forceinline__ void sym_mover(const StageArgs &a, int ntiles, const SymRing &r,
                                          int mw, int lane) {
  constexpr int Np = C::Np, E = C::E, NV = C::NV, NB = C::NB;
  const bool use_k = !a.rhs_only && a.rka != 0.0;
  const long g = gridDim.x;
  const int total = (int)((ntiles - 1 - blockIdx.x) / g) + 1;   // tiles of this CTA
  // lanes 0..: copy cp of variable cv
  constexpr int CPV = C::CPV, CE = E / CPV;
  const int cv = lane / CPV, cp = lane % CPV;
  const bool copies = lane < CPV * NV;
  bool ok = true;
  int it = mw;
  for (; it < total + NB; it += C::NM) {
    const int b = it % NB;
    const long t = blockIdx.x + it * g;
    double *B = r.buf0 + b * C::S_BUF, *bT = B + C::S_U + C::S_REC;
    double *Bc = B + cv * C::VS + C::eoff(cp * CE);
    if (it >= NB && it - NB < total) {
      ok = __all_sync(0xffffffffu, mbar_wait(&r.done[b], ((it / NB) - 1) & 1, a.wait_cycles));
      if (!ok) break;
      const long to = t - NB * g;
      if (copies && (to + 1) * E <= a.K) {   // a ragged tile was stored by the compute warps
        bulk_s2g(a.u_out + cv * a.vs + (to * E + cp * CE) * Np, Bc, 8u * CE * Np);
        bulk_commit();
        bulk_wait_read();
      }
    }
    if (it < total) {
      __syncwarp();
      if (lane == 0) {
        r.seq[b] = it;
        mbar_arrive_expect_tx(&r.full[b], C::TX);
      }
      __syncwarp();
      // one copy per lane: the state, the records, the penalty, and k into L2
      if (copies)
        bulk_g2s(Bc, a.u_in + cv * a.vs + (t * E + cp * CE) * Np, 8u * CE * Np, &r.full[b]);
      else if (lane == 29)
        bulk_g2s(B + C::S_U, a.erec + t * C::S_REC, 8u * C::S_REC, &r.full[b]);
      else if (lane == 30)
        bulk_g2s(bT, a.tau + t * C::S_TAU, 8u * C::S_TAU, &r.full[b]);
      else if (lane == 31 && use_k)
        bulk_prefetch_l2(a.kreg + t * NV * Np * E, 8u * NV * Np * E);
    }
  }
  if (!ok) {
    // an expired wait: the copies of the tiles in flight settle before the warp leaves
    if (lane == 0) atomicOr(&a.sc->flags, 4);
    mover_in_flight<NB, C::NM>(it, total,
                               [&](int q) { mbar_wait(&r.full[q % NB], (q / NB) & 1); });
  }
  if (copies) bulk_wait_all();
}

// Gather warp gw of NL (part gp of GP): the tiles it = gw, gw + NL, ...
// Neighbours inside the tile are read from its state (their code says where);
// the others' traces are gathered by cp.async once the buffer's previous tile
// is done.  (8-byte cp.asyncs to scattered nodes take the load path some 40
// cycles each; several warps at it hide their latency, and the nodes inside
// the tile, a third on a box of hexahedra cut in six, are not gathered.)
template <class C>
__device__ __forceinline__ void sym_gather(const StageArgs &a, int ntiles, const int *tabs,
                                           const SymRing &r, int gw, int gp, int lane) {
  constexpr int Np = C::Np, NFF = C::NFF, E = C::E, NV = C::NV, NB = C::NB, NL = C::NL;
  const int *tslot = tabs + C::T_VOL + C::T_FACE + C::T_OUT + 4 + lane;
  const long g = gridDim.x;
  bool ok = true;
  for (int it = gw; blockIdx.x + it * g < ntiles; it += NL) {
    const long t = blockIdx.x + it * g;
    const int b = it % NB, base = (int)(t * E * Np);
    const int ne = (int)min((long)E, (long)a.K - t * E);
    if (it >= NB) {
      ok = __all_sync(0xffffffffu, mbar_wait(&r.done[b], ((it / NB) - 1) & 1, a.wait_cycles));
      if (!ok) break;
    }
    double *bUP = r.buf0 + b * C::S_BUF + C::S_U + C::S_REC + C::S_TAU;
    short *bNB = reinterpret_cast<short *>(bUP + C::S_TR);
#pragma unroll 1
    for (int q0 = gp * C::GPW; q0 < (gp + 1) * C::GPW; q0 += C::GCH) {
      int nb[C::GCH], slot[C::GCH];
#pragma unroll
      for (int q = 0; q < C::GCH; q++) {
        const int i = lane + 32 * (q0 + q);
        const bool mine = q0 + q < (gp + 1) * C::GPW && i < E * NFF;
        slot[q] = mine ? tslot[32 * (q0 + q)] : -1;
        nb[q] = mine && i < ne * NFF ? __ldg(a.vmapP + t * E * NFF + i) : -1;
      }
#pragma unroll
      for (int q = 0; q < C::GCH; q++) {
        const unsigned n = (unsigned)(nb[q] - base);
        const int e = n / Np;
        const bool in = n < (unsigned)(ne * Np);
        // (also of elements past K: codes are always in bounds)
        if (slot[q] >= 0)
          bNB[slot[q] & 0xffff] = in ? (short)(C::eoff(e) + n - e * Np) : (short)-1;
        if (!in && nb[q] >= 0)
#pragma unroll
          for (int v = 0; v < NV; v++)
            cp_async8(bUP + v * E * C::UPS + (slot[q] >> 16), a.u_in + v * a.vs + nb[q]);
      }
    }
    cp_async_arrive_noinc(&r.trace[b]);   // the traces; the codes with the next
    mbar_arrive(&r.trace[b]);
  }
  if (!ok && lane == 0) atomicOr(&a.sc->flags, 4);
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// Compute warp: variables V0..V0+NVW of group grp's tiles.  A pair of warps
// shares them: each takes half of the k-steps (kc), then they exchange partial
// sums and each finishes half of the variables.
template <class C, int V0, int NVW>
__device__ __forceinline__ void sym_tiles(const StageArgs &a, int ntiles, const double *sA,
                                          const int *tabs, const SymRing &r, int grp, int kc,
                                          int lane) {
  constexpr int Np = C::Np, E = C::E, NV = C::NV, NB = C::NB, NG = C::NG;
  const int *tvol = tabs;
  const int4 *tface = reinterpret_cast<const int4 *>(tabs + C::T_VOL);
  const int4 *tout = tface + C::T_FACE / 4;
  const int4 faces = *reinterpret_cast<const int4 *>(tabs + C::T_VOL + C::T_FACE + C::T_OUT);
  const double dt = a.rhs_only ? 1.0 : a.dt_override >= 0 ? a.dt_override : a.sc->dt;
  const bool use_k = !a.rhs_only && a.rka != 0.0;
  // the warp with fewer variables to finish takes the odd k-steps
  const int vb = kc ? C::KSV / 2 : 0, ve = kc ? C::KSV : C::KSV / 2;
  const int fb = kc ? C::KSF / 2 : 0, fe = kc ? C::KSF : C::KSF / 2;
  // the buffer's tile is `it` and its copies are there
  auto wait_tile = [&](unsigned long long *bar, int it) {
    bool w = r.seq[it % NB] == it;
    if (!w) {
      const long long t0 = clock64();
      while (!(w = r.seq[it % NB] == it) && clock64() - t0 <= a.wait_cycles) {
      }
    }
    return w && mbar_wait(&bar[it % NB], (it / NB) & 1, a.wait_cycles);
  };
  SymWarp<C, V0, NVW> w;
  bool ok = true;
  int it = grp;
  unsigned ph = 0;   // parity of the group's barriers for this tile
  for (long t = blockIdx.x + (long)grp * gridDim.x; t < ntiles;
       t += (long)NG * gridDim.x, it += NG, ph ^= 1) {
    const int b = it % NB;
    double *bU = r.buf0 + b * C::S_BUF, *bF = bU + C::S_U, *bT = bF + C::S_REC,
           *bUP = bT + C::S_TAU;
    const short4 *bNB = reinterpret_cast<const short4 *>(bUP + C::S_TR);
    double2 *px = reinterpret_cast<double2 *>(bUP);
    const int el = C::elem(lane >> 2);
    const double *bE = bU + C::eoff(el), *g = bF + el * kRecord;
    w.clear();
    ok = wait_tile(r.full, it);
    if (!__all_sync(0xffffffffu, ok)) break;
    {
      double mr[9];
#pragma unroll
      for (int q = 0; q < 9; q++) mr[q] = g[q];
      typename SymWarp<C, V0, NVW>::Node n;
      w.load_node(bE, tvol[vb * 4 + (lane & 3)], n);
#pragma unroll 1
      for (int ks = vb; ks < ve; ks++) {
        double gf[3][NVW];
        const int tab = n.tab;
        w.fluxes(n, mr, a.gamma, gf);
        // the next k-step's state is on its way under this one's MMAs
        w.load_node(bE, tvol[min(ks + 1, ve - 1) * 4 + (lane & 3)], n);
        w.volume(gf, sA, tab, ks, lane);
      }
    }
    ok = wait_tile(r.trace, it);
    if (!__all_sync(0xffffffffu, ok)) break;
#pragma unroll 1
    for (int fs = fb; fs < fe; fs++) {
      // (padding positions repeat the last point: finite values, zero columns)
      const int j = min(fs * 4 + (lane & 3), C::Nfp - 1), c = lane >> 2;
      w.face(bU, bE, g, bT + el * 4, bUP + c * C::UPS + j, sA, tface[j], bNB[c * C::NBS + j],
             faces, C::KSV + fs, a.gamma, lane);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&r.read[grp]);
    ok = mbar_wait(&r.read[grp], ph, a.wait_cycles);
    if (!__all_sync(0xffffffffu, ok)) break;
    w.dump(px, kc, lane);
    __syncwarp();
    if (lane == 0) mbar_arrive(&r.dump[grp]);
    double *kt = a.kreg + t * NV * Np * E;
    constexpr int VH = SymWarp<C, V0, NVW>::VH;
    constexpr int KE = C::MTT > 5 ? 1 : VH;   // variables whose k is on its way
    double2 kr[KE][C::MTT];
#pragma unroll
    for (int i = 0; i < KE; i++) w.load_k(kt, use_k, kc ? VH + i : i, lane, kr[i]);
    ok = mbar_wait(&r.dump[grp], ph, a.wait_cycles);
    if (!__all_sync(0xffffffffu, ok)) break;
#pragma unroll
    for (int i = 0; i < VH; i++) {
#pragma unroll
      for (int v = i; v < NVW; v += VH)
        if (v < i + VH + 1 && w.owns(kc, v)) {
          w.update(bU, px, tout, v, dt, a.rka, kr[i % KE], a.rkb, a.rhs_only != 0, lane);
          if (!a.rhs_only) w.store_k(kt, v, lane);
        }
      if (i + KE < VH) w.load_k(kt, use_k, kc ? VH + i + KE : i + KE, lane, kr[i % KE]);
    }
    const int ne = (int)min((long)E, (long)a.K - t * E);
    if (ne < E) {
      __syncwarp();
      for (int v = V0 + (kc ? VH : 0); v < V0 + (kc ? NVW : VH); v++)
        for (int i = lane; i < ne * Np; i += 32)
          a.u_out[v * a.vs + t * E * Np + i] =
              bU[v * C::VS + i + (i >= E / 2 * Np ? C::GAP : 0)];
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (lane == 0) mbar_arrive(&r.done[b]);
  }
  if (!ok) atomicOr(&a.sc->flags, 4);
}

template <int N, int NS, int NG, int NB>
__global__ void __launch_bounds__(SymCfg<N, NS, NG, NB>::THREADS, 1)
    stage_sym_kernel(const StageArgs a, int ntiles) {
  using C = SymCfg<N, NS, NG, NB>;
  extern __shared__ __align__(16) double smem[];
  double *sA = smem;
  SymRing r;
  r.buf0 = sA + C::S_A;
  r.full = reinterpret_cast<unsigned long long *>(r.buf0 + NB * C::S_BUF);
  r.trace = r.full + NB;
  r.done = r.trace + NB;
  r.read = r.done + NB;
  r.dump = r.read + NG;
  r.seq = reinterpret_cast<volatile int *>(r.dump + NG);
  int *tabs = reinterpret_cast<int *>(r.full + C::NBAR);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  pdl_launch();
  if (tid == 0) {
    for (int i = 0; i < NB; i++) {
      mbar_init(&r.full[i], 1);
      mbar_init(&r.trace[i], 64 * C::GP);   // per lane of its gatherers: codes, gathers
      mbar_init(&r.done[i], C::WPG);
      r.seq[i] = -1;
    }
    for (int i = 0; i < NG; i++) {
      mbar_init(&r.read[i], C::WPG);
      mbar_init(&r.dump[i], C::WPG);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // the operator image: fragments, then the tables
  {
    const double2 *src = reinterpret_cast<const double2 *>(a.AT);
    double2 *dst = reinterpret_cast<double2 *>(sA);
    for (int i = tid; i < C::S_A / 2; i += C::THREADS) dst[i] = __ldg(src + i);
    const int *ts = reinterpret_cast<const int *>(a.AT + C::S_A);
    for (int i = tid; i < C::TABS; i += C::THREADS) tabs[i] = __ldg(ts + i);
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncthreads();
  pdl_wait();
  if (warp >= C::NWC) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(C::REGP));
    const int lw = warp - C::NWC;
    if (lw < C::NM)
      sym_mover<C>(a, ntiles, r, lw, lane);
    else if (lw < C::NM + C::NL * C::GP)
      sym_gather<C>(a, ntiles, tabs, r, (lw - C::NM) % C::NL, (lw - C::NM) / C::NL, lane);
    return;
  }
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(C::REGC));
  const int grp = warp / C::WPG, ns = warp % C::WPG / 2;
  const int kc = warp & 1;
  if constexpr (NS == 1) {
    sym_tiles<C, 0, 5>(a, ntiles, sA, tabs, r, grp, kc, lane);
  } else {
    static_assert(NS == 1 || NS == 2, "variables on one or two pairs");
    if (ns == 0)
      sym_tiles<C, 0, 3>(a, ntiles, sA, tabs, r, grp, kc, lane);
    else
      sym_tiles<C, 3, 2>(a, ntiles, sA, tabs, r, grp, kc, lane);
  }
}
