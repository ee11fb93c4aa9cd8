// Internal: the solver handle and the helpers shared by the translation
// units that operate on it (dglm_solver.cu, dglm_adjoint.cu).
#pragma once

#include <cuda_runtime.h>

#include <string>
#include <vector>

#include "dglm_common.cuh"

struct AdjointTape;

struct dglm_handle {
  dglm_desc d{};
  int nvar = 0, Np = 0, Nfp = 0, NFF = 0;
  int variant = 0;                // selected by the caller
  int run_variant = 0;            // launched: the selected one, or its fallback when the
                                  // uploaded operators lack the symmetry it needs
  dglm::StageVariantInfo vinfo{}; // of run_variant
  bool op_symmetric = false;      // whether the uploaded operators have that symmetry
  std::vector<double> Ahost;      // stacked [WDr WDs WDt -LIFT], Np x (3Np+NFF) row-major
  std::vector<double> sym_image;  // operator image of the symmetry-adapted kernel
  long vs = 0;                    // doubles between variables of a field
  long Kp = 0;                    // K rounded up to a multiple of 64 (tile padding)
  int dev = 0;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  // mesh, operators
  double *AT = nullptr, *geo = nullptr, *fscale = nullptr, *nrm = nullptr;
  double *tau = nullptr, *maxv = nullptr, *vel = nullptr;
  int *vmapP = nullptr, *vmapF = nullptr, *Fmask = nullptr;
  // record of the tensor-memory and symmetry-adapted kernels: [Kp][kRecord] per
  // element (Euler: the 9 metrics, nx, ny, nz and Fscale of the 4 faces, one
  // pad double; one bulk copy per tile) or the flow records (advection).  TF32x3
  // and BF16x3 Euler handles always have it; FP64 handles have it while a
  // symmetry-adapted variant runs and there is memory for it
  double *erec = nullptr;
  size_t erec_bytes = 0;   // of an FP64 handle's
  // compact face maps (dglm_set_compact_face_maps), built from vmapP on first
  // use: per face the neighbour element and a code of its node list
  int *etoe = nullptr, *ftab = nullptr;
  unsigned char *fcode = nullptr;
  int ftab_lists = 0;
  bool compact_built = false, compact = false;
  // state
  double *u[2] = {nullptr, nullptr};
  double *kreg = nullptr;
  int cur = 0;
  dglm::DevScalars *sc = nullptr;
  double dt_fixed = -1.0;         // sc->dt_fixed as last written (-1: not known)
  double *dt_hist = nullptr;
  // one-off right-hand side evaluation
  double *rhs_in = nullptr, *rhs_out = nullptr, *maxv_s = nullptr, *tau_s = nullptr;
  dglm::DevScalars *sc_s = nullptr;
  bool mesh_ready = false, state_ready = false;
  cudaGraphExec_t graph[2] = {nullptr, nullptr};
  long launches = 0;
  size_t bytes = 0;
  std::vector<void *> allocs;
  long long wait_cycles = 0;     // > 0: shortened hand-off wait bound (dglm_set_wait_limit)
  AdjointTape *tape = nullptr;   // discrete adjoint (dglm_adjoint.cu)
  int adj_variant = 0;           // adjoint tile shape
  // dglm_run_ensemble: double-buffered device copies of the members' input
  // and output states, a copy-in and a copy-out stream, and their events
  // (in_ready[2], in_free[2], out_ready[2], out_free[2])
  double *ens_in[2] = {nullptr, nullptr}, *ens_out[2] = {nullptr, nullptr};
  int *ens_flags = nullptr;
  int ens_cap = 0;
  cudaStream_t ens_cin = nullptr, ens_cout = nullptr;
  cudaEvent_t ens_ev[8] = {};
};


namespace dglm {

// Carpenter & Kennedy 5-stage 4th-order 2N-storage coefficients
// (euler_data.cpp:41-60).
constexpr double RKA[5] = {0.0, -567301805773.0 / 1357537059087.0,
                       -2404267990393.0 / 2016746695238.0, -3550918686646.0 / 2091501179385.0,
                       -1275806237668.0 / 842570457699.0};
constexpr double RKB[5] = {1432997174477.0 / 9575080441755.0, 5161836677717.0 / 13612068292357.0,
                       1720146321549.0 / 2090206949498.0, 3134564353537.0 / 4481467310338.0,
                       2277821191437.0 / 14882151754819.0};

struct DeviceGuard {
  int prev = -1;
  explicit DeviceGuard(int dev) {
    cudaGetDevice(&prev);
    if (dev >= 0 && dev != prev) cudaSetDevice(dev);
  }
  ~DeviceGuard() {
    if (prev >= 0) cudaSetDevice(prev);
  }
};

// Gives back the record of an FP64 handle's symmetry-adapted kernel, which then
// runs on its fallback; false when there is none to give back.
bool drop_record(dglm_handle *h);

// cudaMalloc; where memory is short, with that record given back.
inline cudaError_t handle_malloc(dglm_handle *h, void **q, size_t n) {
  cudaError_t e = cudaMalloc(q, n);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    if (drop_record(h)) e = cudaMalloc(q, n);
  }
  return e;
}

template <typename T>
inline dglm_status dalloc(dglm_handle *h, T **p, size_t count) {
  void *q = nullptr;
  const size_t n = count * sizeof(T);
  cudaError_t e = handle_malloc(h, &q, n ? n : 16);
  if (e != cudaSuccess) {
    *p = nullptr;
    return set_error(DGLM_ERR_NOMEM, std::string("cudaMalloc failed: ") + cudaGetErrorString(e));
  }
  h->allocs.push_back(q);
  h->bytes += n;
  *p = static_cast<T *>(q);
  return DGLM_OK;
}

// Several arrays that are all there or not at all.  Those of 1 MiB and more share
// one allocation (each 256-byte aligned), which takes some 0.3 ms whatever its
// size; the driver cuts smaller ones out of memory that it holds (0.01 ms).
struct Arrays {
  struct Item {
    void **p;
    size_t bytes;
  };
  std::vector<Item> items;
  template <typename T>
  void add(T **p, size_t count) {
    items.push_back({reinterpret_cast<void **>(p), (count * sizeof(T) + 255) / 256 * 256});
  }
  dglm_status allocate(dglm_handle *h) {
    constexpr size_t kLarge = 1u << 20;
    const size_t before = h->allocs.size();
    size_t shared = 0, taken = 0;
    for (const Item &i : items) {
      *i.p = nullptr;
      if (i.bytes >= kLarge) shared += i.bytes;
    }
    char *base = nullptr;
    dglm_status st = shared ? dalloc(h, &base, shared) : DGLM_OK;
    if (st == DGLM_OK) taken = shared;
    for (const Item &i : items) {
      if (st != DGLM_OK) break;
      if (i.bytes >= kLarge) {
        *i.p = base;
        base += i.bytes;
        continue;
      }
      char *own = nullptr;
      st = dalloc(h, &own, i.bytes);
      *i.p = own;
      if (st == DGLM_OK) taken += i.bytes;
    }
    if (st == DGLM_OK) return st;
    for (; h->allocs.size() > before; h->allocs.pop_back()) cudaFree(h->allocs.back());
    h->bytes -= taken;
    for (const Item &i : items) *i.p = nullptr;
    return st;
  }
};

StageArgs stage_args(dglm_handle *h, const double *u_in, double *u_out, int s);
void free_tape(dglm_handle *h);
dglm_status run_steps(dglm_handle *h, int nsteps);
dglm_status set_dt_fixed(dglm_handle *h, double dt);
dglm_status issue_step_ptrs(dglm_handle *h, const double *const *in, double *const *out,
                            cudaStream_t s);
dglm_status ensure_rhs_scratch(dglm_handle *h);

}  // namespace dglm
