// FP64 kernels of the explicit multi-fluid Hall-MHD step on sm_100a, run by
// the batched engine (mhd_engine.cuh): every kernel is a persistent
// grid-stride loop over the tile work-list of all active solves.
//
// Each kernel restates one pass of the reference step in the reference's own
// operation order (the library is built without FMA contraction), so the
// FP64 path reproduces the reference bitwise.  Restructurings that keep the
// arithmetic identical:
//   * the contravariant velocity u^a = (K^a . U_plus) / (|J| + 1e-30) of every
//     cell (cell_u_contra, Z4_Mercury/src/physics/MercurySolver_MagExplicit_Ideal.cpp:180-199)
//     is computed once per step into UCON instead of up to 16 times per edge;
//   * the fluid update runs one work item per (cell, species) in FP64, per cell in FP32;
//   * B_cell/Bind_cell and J_edge share one pass over the face fluxes;
//   * the next step's CFL dt is reduced in the same pass that refreshes the
//     primitive variables (both read U and B_cell after their syncs).
#include <mutex>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <type_traits>

#include "mhd_engine.cuh"
#include "mhd_kernels.cuh"

namespace mhd {

namespace {

// Slots of k_pv_uplus's stage, and its resident CTAs per SM.
constexpr int kPvSlots = 30;
constexpr int kPvCtas = 5;
constexpr int cUH = 0, cUN = 5;
constexpr int cBX = kComp.first[MHD_B_XI], cBY = kComp.first[MHD_B_ETA], cBZ = kComp.first[MHD_B_ZETA];
constexpr int cPVH = kComp.first[MHD_PV_H], cPVN = kComp.first[MHD_PV_NA], cUP = kComp.first[MHD_U_PLUS];
constexpr int cBC = kComp.first[MHD_B_CELL], cBIC = kComp.first[MHD_BIND_CELL], cJC = kComp.first[MHD_J_CELL];
constexpr int cJX = kComp.first[MHD_J_XI], cJY = kComp.first[MHD_J_ETA], cJZ = kComp.first[MHD_J_ZETA];
constexpr int cEX = kComp.first[MHD_E_XI], cEY = kComp.first[MHD_E_ETA], cEZ = kComp.first[MHD_E_ZETA];
constexpr int cHX = kComp.first[MHD_EHALL_XI], cHY = kComp.first[MHD_EHALL_ETA], cHZ = kComp.first[MHD_EHALL_ZETA];
constexpr int cEFX = kComp.first[MHD_EFACE_XI], cEFY = kComp.first[MHD_EFACE_ETA], cEFZ = kComp.first[MHD_EFACE_ZETA];
constexpr int cEHC = kComp.first[MHD_EHC], cHB = kComp.first[MHD_HALL_BETA], cUC = kComp.first[MHD_UCON];
constexpr int cDIVB = kComp.first[MHD_DIVB];
constexpr int cETAR = kComp.first[MHD_ETA_RES_XI];  // ETA_RES_ETA, ETA_RES_ZETA follow
constexpr int cRW = kComp.first[MHD_RES_W], cRX = kComp.first[MHD_RES_X], cRR = kComp.first[MHD_RES_R],
              cRP = kComp.first[MHD_RES_P], cRQ = kComp.first[MHD_RES_Q], cRBS = kComp.first[MHD_RES_BSTAR];
constexpr int cFNX = kComp.first[MHD_FNORM_XI], cFNY = kComp.first[MHD_FNORM_ETA], cFNZ = kComp.first[MHD_FNORM_ZETA];
constexpr int cPEN = kComp.first[MHD_PE_NODE], cAMB = kComp.first[MHD_AMBI_COEF], cDPE = kComp.first[MHD_DPE];
constexpr int cUCK = kComp.first[MHD_UCON_COEF];
constexpr int cIHX = kComp.first[MHD_HALL_IH_XI], cIHY = kComp.first[MHD_HALL_IH_ETA], cIHZ = kComp.first[MHD_HALL_IH_ZETA];
constexpr int cFM = kComp.first[MHD_FLUX_METRIC];
constexpr int cFT = kFirstInternal;  // re, c of H+, re, c of Na+
constexpr int cJAC = kComp.first[MHD_JAC], cJDX = kComp.first[MHD_JDXI], cJDY = kComp.first[MHD_JDET],
              cJDZ = kComp.first[MHD_JDZE];
constexpr int cAX = kComp.first[MHD_AREA_XI], cAY = kComp.first[MHD_AREA_ETA], cAZ = kComp.first[MHD_AREA_ZETA];
constexpr int cDLX = kComp.first[MHD_DL_XI], cDLY = kComp.first[MHD_DL_ETA], cDLZ = kComp.first[MHD_DL_ZETA];
constexpr int cDRX = kComp.first[MHD_DR_XI], cDRY = kComp.first[MHD_DR_ETA], cDRZ = kComp.first[MHD_DR_ZETA];
constexpr int cBFX = kComp.first[MHD_HODGE_FACE_XI], cBFY = kComp.first[MHD_HODGE_FACE_ETA],
              cBFZ = kComp.first[MHD_HODGE_FACE_ZETA];
constexpr int cALX = kComp.first[MHD_HODGE_EDGE_XI], cALY = kComp.first[MHD_HODGE_EDGE_ETA],
              cALZ = kComp.first[MHD_HODGE_EDGE_ZETA];
constexpr int cWB = kComp.first[MHD_BCELL_W], cWJ = kComp.first[MHD_JCELL_W];
static_assert(cBFY == cBFX + 1 && cBFZ == cBFX + 2 && cALY == cALX + 1 && cALZ == cALX + 2, "xi, eta, zeta consecutive");
constexpr int cBAX = kComp.first[MHD_BADD_XI], cBAY = kComp.first[MHD_BADD_ETA], cBAZ = kComp.first[MHD_BADD_ZETA];
constexpr int cPHOTO = kComp.first[MHD_PHOTO], cCX = kComp.first[MHD_CELL_X];  // CELL_Y, CELL_Z follow
constexpr int cTPX = kComp.first[MHD_TAPER_XI];  // TAPER_ETA, TAPER_ZETA follow
constexpr int cTPC = kComp.first[MHD_TAPER_CELL];
constexpr int cLEX = kComp.first[MHD_LOCAL_ETA_XI];  // LOCAL_ETA_ETA, LOCAL_ETA_ZETA follow

// std::max / std::min semantics (first argument wins ties, incl. signed zeros).
template <class R>
__device__ __forceinline__ R dmax(R a, R b) { return (a < b) ? b : a; }
template <class R>
__device__ __forceinline__ R dmin(R a, R b) { return (b < a) ? b : a; }

// One block's fields for the current step: U = current buffer, M = metric
// (double) then, at Mr, the other real-valued components (mhd_engine.cuh).
// Element offsets inside a block are 32-bit (mhd_batch_add keeps every
// block's component arrays below 2^31 elements in total).
template <class R>
struct V {
  char *U, *Un, *M, *Mr;  // U, Un: the current and the other buffer
  char *narrow;           // DevBlock::narrow
  uint32_t tb;  // bytes of one real-valued component array
  int total, si, sj;
  int G, n0, n1, n2;
  // real-valued component (U or M)
  __device__ __forceinline__ R *c(int comp) const {
    return (R *)(comp < kNumUComps ? U + (uint64_t)comp * tb : Mr + (uint64_t)rslot(comp) * tb);
  }
  __device__ __forceinline__ R *next(int comp) const { return (R *)(Un + (uint64_t)comp * tb); }  // U, the other buffer
  // metric component (JAC, JD*), double in every precision
  __device__ __forceinline__ double *m(int comp) const {
    return (double *)(M + (uint64_t)(comp - kMetricFirst) * (tb * (8 / (uint32_t)sizeof(R))));
  }
  // Component `comp` at byte offset bo of its array (bo = off() times the
  // element size), through the read-only path: only for what no kernel writes
  // while this one runs, the static fields, and, in kernels that are launched
  // after their predecessor in full (k_fluid), the fields of earlier passes.  The array's address is
  // warp-uniform (build_item) and bo is 32 bits, so no thread holds 64-bit
  // addresses: without that k_fluid spilled 700 bytes at 80 registers.
  __device__ __forceinline__ R fixed1(int comp, uint32_t bo) const {
    return __ldg((const R *)((const char *)c(comp) + bo));
  }
  __device__ __forceinline__ double ldm(int comp, uint32_t bo) const {
    return __ldg((const double *)((const char *)m(comp) + bo));
  }
  __device__ __forceinline__ int off(int i, int j, int k) const { return (i + G) * si + (j + G) * sj + (k + G); }
};
#define AT(cc, i, j, k) (B.c(cc)[B.off((i), (j), (k))])
#define ATM(cc, i, j, k) (B.m(cc)[B.off((i), (j), (k))])

struct Item {
  int s;       // solve
  int blk;     // block of the solve
  int species; // fluid ranges only
  int i, j, k;
  bool in;     // inside the kernel's range
  int hi[3];   // range upper bounds (exclusive)
  int lo[3];   // range lower bounds
};

// Programmatic dependent launch: the kernels of a step are launched while their
// predecessor drains (launch_dependent).  A kernel first looks its first tile
// up in the directory, which nothing writes during a step, then waits until
// every earlier kernel has completed and its writes are visible.  CTAs without
// work may leave before the wait, but never CTA 0: a kernel must not complete
// before its predecessor has.
__device__ __forceinline__ void let_dependents_launch() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void wait_for_predecessors() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// The solve s, its block b and the block's tile t of work item w of range
// KIND (two binary searches over the directory's prefix sums).
template <int KIND>
__device__ __forceinline__ void lookup_item(const Dir &D, int w, int &s, int &b, int &t) {
  const int *sp = D.solve_tile_prefix[KIND];
  int lo = 0, hi = D.nsolves;  // largest s with sp[s] <= w
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (sp[mid] <= w) lo = mid; else hi = mid;
  }
  s = lo;
  const int lw = w - sp[s];
  const int *bp = D.solves[s].tile_prefix[KIND];
  int blo = 0, bhi = D.solves[s].nblocks;
  while (bhi - blo > 1) {
    const int mid = (blo + bhi) >> 1;
    if (bp[mid] <= lw) blo = mid; else bhi = mid;
  }
  b = blo;
  t = lw - bp[blo];
}

// The view of block DB with U buffer `cur` current.
template <class R>
__device__ __forceinline__ void set_view(V<R> &B, const DevBlock &DB, int cur) {
  B.U = (char *)DB.U[cur];
  B.Un = (char *)DB.U[cur ^ 1];
  B.M = DB.M;
  B.total = (int)DB.total;
  B.tb = (uint32_t)B.total * (uint32_t)sizeof(R);
  B.Mr = DB.M + (int64_t)kNumMetric * DB.total * 8;
  B.narrow = DB.narrow;
  B.si = (int)DB.si;
  B.sj = (int)DB.sj;
  B.G = DB.G;
  B.n0 = DB.n[0];
  B.n1 = DB.n[1];
  B.n2 = DB.n[2];
}

// A value that every lane of the (converged) warp holds, in a form the
// compiler knows to be the same for the warp.
__device__ __forceinline__ int uniform(int v) { return __shfl_sync(0xffffffffu, v, 0); }
template <class T>
__device__ __forceinline__ T *uniform(T *p) {
  const unsigned long long v = (unsigned long long)p;
  const unsigned lo = __shfl_sync(0xffffffffu, (unsigned)v, 0), hi = __shfl_sync(0xffffffffu, (unsigned)(v >> 32), 0);
  return (T *)(((unsigned long long)hi << 32) | lo);
}

// Whether solve s is active and which U buffer is current.  In a step (mode 0)
// they only change in its passes that end by them (flip_solve in k_bface,
// retire_solve in k_pv_uplus), whose successors are launched after them in full,
// so they may be read ahead of the wait; the mask of a targeted pass may not.
struct Status {
  int active, cur;
};
__device__ __forceinline__ Status status_of(const Dir &D, int s) {
  const SolveState &st = D.state[s];
  return Status{D.mode ? st.mask != 0 : st.remaining != 0, st.cur};
}

// The work item (s, b, t) of range KIND as this thread sees it, and the
// block's fields of the current step.
template <class R, int KIND>
__device__ __forceinline__ void build_item(const Dir &D, int s, int b, int t, Item &it, V<R> &B) {
  const int tid = threadIdx.x;
  const DevSolve &S = D.solves[s];
  const DevBlock &DB = S.blocks[b];
  RangeBox r = range_of(KIND, DB.n, S.c.nghost);
  it.s = s;
  it.blk = b;
  for (int a = 0; a < 3; ++a) {
    it.hi[a] = r.hi[a];
    it.lo[a] = r.lo[a];
  }
  if constexpr (fluid_variant(KIND) >= 0) {  // a fluid tile: one thread per column of cells along i
    constexpr FluidTile T = fluid_tile(fluid_variant(KIND));
    const int tk = (r.hi[2] - r.lo[2] + T.k - 1) / T.k, tj = (r.hi[1] - r.lo[1] + T.j - 1) / T.j;
    const int q = t >> 1, rest = q / tk;
    it.species = t & 1;
    it.k = r.lo[2] + (q - rest * tk) * T.k + tid % T.k;
    it.j = r.lo[1] + (rest % tj) * T.j + tid / T.k;
    it.i = r.lo[0] + (rest / tj) * T.i;  // the column's first cell
    it.in = it.j < r.hi[1] && it.k < r.hi[2];
  } else {  // a run of kTileThreads consecutive positions of the range box (k fastest)
    const int ek = r.hi[2] - r.lo[2], ej = r.hi[1] - r.lo[1];
    const int L = t * kTileThreads + tid;
    const int rest = L / ek;
    it.k = r.lo[2] + (L - rest * ek);
    it.j = r.lo[1] + rest % ej;
    it.i = r.lo[0] + rest / ej;
    it.in = L < ek * ej * (r.hi[0] - r.lo[0]);
  }
  const int cur = D.state[s].cur;
  set_view(B, DB, cur);
  B.U = uniform(B.U);
  B.Un = uniform(B.Un);
  B.M = uniform(B.M);
  B.Mr = uniform(B.Mr);
  B.tb = uniform((int)B.tb);
  B.total = uniform(B.total);
  B.si = uniform(B.si);
  B.sj = uniform(B.sj);
}

// Work-item loop: for every tile of range `KIND` of every active solve, call
// f(S, B, item).  Tile lookup by thread 0, broadcast through shared
// memory.
template <class R, int KIND, class F>
__device__ __forceinline__ void for_items(const Dir &D, F &&f) {
  __shared__ int sh[3];
  let_dependents_launch();
  const int total = D.solve_tile_prefix[KIND][D.nsolves];
  const int tid = threadIdx.x;
  if ((int)blockIdx.x >= total) {
    if (blockIdx.x == 0) wait_for_predecessors();
    return;
  }
  for (int w = blockIdx.x; w < total; w += gridDim.x) {
    if (tid == 0) lookup_item<KIND>(D, w, sh[0], sh[1], sh[2]);
    __syncthreads();
    const int s = sh[0], b = sh[1], t = sh[2];
    __syncthreads();
    if (w == (int)blockIdx.x) wait_for_predecessors();
    if (!solve_active(D, s)) continue;  // inactive solve (the whole CTA agrees)
    Item it;
    V<R> B;
    build_item<R, KIND>(D, s, b, t, it, B);
    f(D.solves[s], B, it);
  }
}

// ------------------------------------------------------------------ vector items
// The step's stencil passes take 16 bytes of consecutive k positions (4 FP32 or
// 2 FP64 values, aligned: rows are padded to 8 elements) per thread and
// array, element by element with the operations of the scalar form.
template <class R, int M = 16 / (int)sizeof(R)>
struct alignas(M * sizeof(R)) Vec {
  static constexpr int N = M;
  R v[M];
};
template <class R, int M = 16 / (int)sizeof(R), class F>
__device__ __forceinline__ Vec<R, M> vmap(F &&f) {
  Vec<R, M> r;
#pragma unroll
  for (int e = 0; e < M; ++e) r.v[e] = f(e);
  return r;
}
#define MHD_VEC_OP(op)                                                                  \
  template <class R, int M>                                                             \
  __device__ __forceinline__ Vec<R, M> operator op(const Vec<R, M> &a, const Vec<R, M> &b) { \
    return vmap<R, M>([&](int e) { return a.v[e] op b.v[e]; });                         \
  }                                                                                     \
  template <class R, int M>                                                             \
  __device__ __forceinline__ Vec<R, M> operator op(R a, const Vec<R, M> &b) {           \
    return vmap<R, M>([&](int e) { return a op b.v[e]; });                              \
  }                                                                                     \
  template <class R, int M>                                                             \
  __device__ __forceinline__ Vec<R, M> operator op(const Vec<R, M> &a, R b) {           \
    return vmap<R, M>([&](int e) { return a.v[e] op b; });                              \
  }
MHD_VEC_OP(+)
MHD_VEC_OP(-)
MHD_VEC_OP(*)
MHD_VEC_OP(/)
#undef MHD_VEC_OP
template <class R, int M>
__device__ __forceinline__ Vec<R, M> operator-(const Vec<R, M> &a) {
  return vmap<R, M>([&](int e) { return -a.v[e]; });
}
template <class R, int M = 16 / (int)sizeof(R)>
__device__ __forceinline__ Vec<R, M> vset(R x) {
  return vmap<R, M>([&](int) { return x; });
}
template <class R, int M>
__device__ __forceinline__ Vec<R, M> vabs(const Vec<R, M> &a) {
  return vmap<R, M>([&](int e) { return fabs(a.v[e]); });
}
template <class R, int M>
__device__ __forceinline__ Vec<R, M> vsqrt(const Vec<R, M> &a) {
  return vmap<R, M>([&](int e) { return sqrt(a.v[e]); });
}
template <class R, int M>
__device__ __forceinline__ Vec<R, M> vmax(const Vec<R, M> &a, const Vec<R, M> &b) {
  return vmap<R, M>([&](int e) { return dmax(a.v[e], b.v[e]); });
}
// The values one k lower (the lowest from `prev`), one k higher (the highest from `next`).
template <class R, int M>
__device__ __forceinline__ Vec<R, M> vdown(const Vec<R, M> &a, R prev) {
  return vmap<R, M>([&](int e) { return e == 0 ? prev : a.v[e > 0 ? e - 1 : 0]; });
}
template <class R, int M>
__device__ __forceinline__ Vec<R, M> vup(const Vec<R, M> &a, R next) {
  return vmap<R, M>([&](int e) { return e == M - 1 ? next : a.v[e < M - 1 ? e + 1 : e]; });
}

// One thread's part of a vector item: positions k .. k + N - 1 of row (i, j),
// of which [klo, khi) are in the range.
struct VItem {
  int s, blk, w, i, j, k;  // w: the tile's index over all solves
  bool in;
  uint32_t o;  // byte offset of position (i, j, k) in a real-valued component array
  int klo, khi;
  __device__ __forceinline__ bool has(int e) const { return k + e >= klo && k + e < khi; }
};
// The static operands of a pass (weights, metric terms: set by mhd_prepare) stream
// through shared memory: every thread copies its own 16 bytes of each array
// with cp.async and reads them back itself, so no barrier is needed, all of
// them are in flight at once, and the first tile's are issued ahead of the wait
// for the predecessors, which do not write them.
// This thread's address in slot 0 of a stage of `size`-byte groups.
__device__ __forceinline__ uint32_t stage_base(int size) {
  extern __shared__ __align__(16) unsigned char stage_smem[];
  return (uint32_t)__cvta_generic_to_shared(stage_smem) + threadIdx.x * (uint32_t)size;
}
constexpr int stage_bytes(int slots, int size) { return slots * kVecThreads * size; }
__device__ __forceinline__ void staged_arrived() { asm volatile("cp.async.wait_all;" ::: "memory"); }

template <class R, int M = 16 / (int)sizeof(R)>
struct VV : V<R> {
  static constexpr int N = M;
  using Vc = Vec<R, M>;
  using V<R>::c;
  using V<R>::m;
  uint32_t di, dj;  // bytes to the neighbour along i and j (k: sizeof(R))
  // 4, 8 or 16 aligned bytes as one load
  template <class T>
  __device__ __forceinline__ static void load(T *to, const void *p) {
    if constexpr (sizeof(R) * M == 16) *(float4 *)to = __ldg((const float4 *)p);
    else if constexpr (sizeof(R) * M == 8) *(float2 *)to = __ldg((const float2 *)p);
    else *(float *)to = __ldg((const float *)p);
  }
  // A static field (fixed1's conditions).
  __device__ __forceinline__ Vc fixed(int comp, uint32_t o) const {
    Vc r;
    const char *p = (const char *)c(comp) + o;
    if constexpr (M == 1) r.v[0] = __ldg((const R *)p);
    else if constexpr (sizeof(R) == 8) *(double2 *)r.v = __ldg((const double2 *)p);
    else load(r.v, p);
    return r;
  }
  // A field that a pass of the step or of the substep writes.  These passes start
  // while their predecessor may still write it, and the wait
  // (wait_for_predecessors) orders ordinary loads only.  An ordinary load does not
  // pass a store that could be to its address, so k_edge_emf, k_bcell_jedge,
  // k_pv_uplus, k_res_db, k_res_pupd_e, k_res_bupdate and in FP64 k_face_emf load
  // all they need ahead of their first store (k_bcell_jedge on the 96^3 mixed box
  // 0.038 ms instead of 0.041, k_pv_uplus 0.076 instead of 0.081, a step of the
  // 8^3 FP64 box 48 us instead of 50); k_bface and k_res_cg are no faster that
  // way.  With every launch in full and read-only loads instead, a step takes
  // 63 us on the 8^3 FP64 box, 95 (73) on 32^3, 164 (139) on 64^3 mixed.
  __device__ __forceinline__ Vc lv(int comp, uint32_t o) const { return *(const Vc *)((const char *)c(comp) + o); }
  __device__ __forceinline__ R ld(int comp, uint32_t bo) const { return *(const R *)((const char *)c(comp) + bo); }
  // lv of a static field of the implicit substep: an FP64 companion reads the
  // FP32 values it was widened from (half the bytes, the same numbers)
  __device__ __forceinline__ Vc stat(int comp, uint32_t o) const {
    if constexpr (sizeof(R) == 8 && M == 2) {
      if (this->narrow) {
        const float2 f = __ldg((const float2 *)(this->narrow + (uint64_t)rslot(comp) * (this->tb / 2) + o / 2));
        Vc r;
        r.v[0] = (R)f.x;
        r.v[1] = (R)f.y;
        return r;
      }
    }
    return fixed(comp, o);
  }
  __device__ __forceinline__ R stat1(int comp, uint32_t o) const {  // one value of stat
    if constexpr (sizeof(R) == 8 && M == 2)
      if (this->narrow)
        return (R)__ldg((const float *)(this->narrow + (uint64_t)rslot(comp) * (this->tb / 2) + o / 2));
    return this->fixed1(comp, o);
  }
  // the values one k lower / higher than lv(comp, o), of which v holds the shared ones
  __device__ __forceinline__ Vc lower(const Vc &v, int comp, uint32_t o) const {
    return vdown(v, ld(comp, o - (uint32_t)sizeof(R)));
  }
  __device__ __forceinline__ Vc upper(const Vc &v, int comp, uint32_t o) const {
    return vup(v, ld(comp, o + (uint32_t)sizeof(Vc)));
  }
  __device__ __forceinline__ Vc fixed_upper(const Vc &v, int comp, uint32_t o) const {
    return vup(v, this->fixed1(comp, o + (uint32_t)sizeof(Vc)));
  }
  // lv(comp, o) copied to this thread's bytes of slot q of the CTA's stage
  // (cp.async: in flight without holding a register) and, after staged_arrived, read back
  __device__ __forceinline__ void stage(uint32_t base, int q, int comp, uint32_t o) const {
    const uint32_t to = base + (uint32_t)q * (uint32_t)(kVecThreads * sizeof(Vc));
    const char *from = (const char *)c(comp) + o;
    if constexpr (sizeof(Vc) == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(from) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(to), "l"(from), "n"(sizeof(Vc)) : "memory");
  }
  __device__ __forceinline__ Vc staged(int q) const {
    extern __shared__ __align__(16) unsigned char stage_smem[];
    return reinterpret_cast<const Vc *>(stage_smem)[q * kVecThreads + (int)threadIdx.x];
  }
  // metric values (double) at the item's positions
  __device__ __forceinline__ Vc lm(int comp, uint32_t o) const {
    const double *p = (const double *)((const char *)m(comp) + (uint64_t)o * (8 / sizeof(R)));
    Vc r;
    if constexpr (M == 1) {
      r.v[0] = (R)__ldg(p);
    } else {
#pragma unroll
      for (int e = 0; e < M; e += 2) {
        const double2 a = __ldg((const double2 *)p + e / 2);
        r.v[e] = (R)a.x;
        r.v[e + 1] = (R)a.y;
      }
    }
    return r;
  }
  // writes the positions k + e in [lo, hi) where the item is in the range and `cond`
  __device__ __forceinline__ void st(int comp, const VItem &it, const Vc &v, int lo, int hi, bool cond = true) const {
    char *p = (char *)c(comp) + it.o;
    const bool w = it.in && cond, all = w && it.k >= lo && it.k + N <= hi;
    if (all) *(Vc *)p = v;
    if constexpr (M > 1) {
#pragma unroll
      for (int e = 0; e < N; ++e)
        if (w && !all && it.k + e >= lo && it.k + e < hi) ((R *)p)[e] = v.v[e];
    }
  }
};

template <class R, int KIND>
__device__ __forceinline__ void build_vec_item(const Dir &D, int s, int b, int t, VItem &it,
                                               VV<R, group_size(KIND, sizeof(R))> &B) {
  constexpr int N = group_size(KIND, sizeof(R));
  const DevSolve &S = D.solves[s];
  const DevBlock &DB = S.blocks[b];
  RangeBox r = range_of(KIND, DB.n, S.c.nghost);
  if constexpr (KIND == kResK) r.hi[2] = DB.reskhi;
  set_view(B, DB, 0);  // the buffers of cur = 0: use_current after the state can be read
  B.U = uniform(B.U);
  B.Un = uniform(B.Un);
  B.M = uniform(B.M);
  B.Mr = uniform(B.Mr);
  B.narrow = uniform(B.narrow);
  B.tb = uniform((int)B.tb);
  B.di = uniform((int)((uint32_t)B.si * (uint32_t)sizeof(R)));
  B.dj = uniform((int)((uint32_t)B.sj * (uint32_t)sizeof(R)));
  B.G = uniform(B.G);
  B.n0 = uniform(B.n0);
  B.n1 = uniform(B.n1);
  B.n2 = uniform(B.n2);
  const RowGroups g = row_groups(r, B.G, N);
  const int ej = r.hi[1] - r.lo[1];
  const int L = t * kVecThreads + (int)threadIdx.x;
  const int row = L / g.count, ri = row / ej;
  it.s = s;
  it.blk = b;
  it.k = (g.first + (L - row * g.count)) * N - B.G;
  it.j = r.lo[1] + (row - ri * ej);
  it.i = r.lo[0] + ri;
  it.in = it.i < r.hi[0];
  if (!it.in) {  // past the last row: work on the first one and write nothing (no divergence)
    it.i = r.lo[0];
    it.j = r.lo[1];
    it.k = g.first * N - B.G;
  }
  it.klo = r.lo[2];
  it.khi = r.hi[2];
  it.o = (uint32_t)B.off(it.i, it.j, it.k) * (uint32_t)sizeof(R);
}

template <class R>
__device__ __forceinline__ void use_current(V<R> &B, int cur) {
  char *const a = B.U, *const b = B.Un;
  B.U = cur ? b : a;
  B.Un = cur ? a : b;
}

// Work-item loop over the vector ranges: f(S, B, item) for every tile of
// range KIND of every active solve, pre(B, item) before it (staged static
// operands).  Thread 0 looks the next tile up while the
// CTA works on the current one (one barrier per tile).
struct NoStage {
  template <class B>
  __device__ void operator()(const B &, const VItem &) const {}
};
template <class R, int KIND, class F, class P = NoStage>
__device__ __forceinline__ void for_vec_items(const Dir &D, F &&f, P &&pre = P{}) {
  __shared__ int sh[2][3];
  let_dependents_launch();
  const int total = D.solve_tile_prefix[KIND][D.nsolves];
  int w = blockIdx.x, p = 0;
  if (w >= total) {
    if (w == 0) wait_for_predecessors();
    return;
  }
  if (threadIdx.x == 0) lookup_item<KIND>(D, w, sh[0][0], sh[0][1], sh[0][2]);
  __syncthreads();
  for (; w < total; w += gridDim.x, p ^= 1) {
    const int s = uniform(sh[p][0]), b = uniform(sh[p][1]), t = uniform(sh[p][2]);
    if (threadIdx.x == 0 && w + (int)gridDim.x < total)
      lookup_item<KIND>(D, w + gridDim.x, sh[p ^ 1][0], sh[p ^ 1][1], sh[p ^ 1][2]);
    __syncwarp();
    VItem it;
    VV<R, group_size(KIND, sizeof(R))> B;
    build_vec_item<R, KIND>(D, s, b, t, it, B);
    it.w = w;
    pre(B, it);  // loads of what no pass of the step writes
    Status st{};
    if (D.mode == 0) st = status_of(D, s);
    if (w == (int)blockIdx.x) wait_for_predecessors();
    if (D.mode != 0) st = status_of(D, s);
    if (uniform(st.active)) {
      use_current(B, uniform(st.cur));
      f(D.solves[s], B, it);
    } else if constexpr (!std::is_same_v<P, NoStage>) {
      staged_arrived();  // the next tile takes the same slots
    }
    __syncthreads();
  }
}
// Runs f(state) for every solve once all CTAs of this kernel that had tiles of
// range KIND have done them (a ticket): the last of them does it.
template <int KIND, class F>
__device__ __forceinline__ void after_all_tiles(const Dir &D, unsigned int *ticket, F &&f) {
  const int total = D.solve_tile_prefix[KIND][D.nsolves];
  if ((int)blockIdx.x >= total) return;
  __shared__ int last;
  if (threadIdx.x == 0) {  // the CTA's tiles are done (for_vec_items ends in a barrier)
    __threadfence();
    last = atomicAdd(ticket, 1u) == (unsigned)min(total, (int)gridDim.x) - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (int s = threadIdx.x; s < D.nsolves; s += blockDim.x) f(D.state[s]);
  if (threadIdx.x == 0) *ticket = 0;
}
// The same, position by position: f(S, B, pos) (passes that run once per solve).
struct Pos {
  int s, blk, i, j, k;
};
template <class R, int KIND, class F>
__device__ __forceinline__ void for_positions(const Dir &D, F &&f) {
  for_vec_items<R, KIND>(D, [&](const DevSolve &S, const auto &B, const VItem &it) {
#pragma unroll 1
    for (int e = 0; e < group_size(KIND, sizeof(R)); ++e)
      if (it.in && it.has(e)) f(S, B, Pos{it.s, it.blk, it.i, it.j, it.k + e});
  });
}

template <class R>
struct Num {
  R nH, nNa, ne_eff, chiH, chiNa, wH, wNa;
};

// Hall_Num_Limiter (Z4_Mercury/src/physics/MercurySolver_Tools.cpp:111-157)
template <class R>
__device__ __forceinline__ Num<R> num_limiter(const ConstsT<R> &c, R rhoH, R rhoNa) {
  Num<R> d;
  const R rH = dmax(rhoH, R(0.0)), rN = dmax(rhoNa, R(0.0));
  if constexpr (sizeof(R) == 4) {  // one reciprocal per divisor
    d.nH = rH * c.n_of_rho[0];
    d.nNa = rN * c.n_of_rho[1];
  } else {
    d.nH = rH / c.M_H * c.M_ref;
    d.nNa = rN / c.M_Na * c.M_ref;
  }
  const R ne_true = d.nH + d.nNa;
  d.ne_eff = sqrt(ne_true * ne_true + c.ne_hall_floor * c.ne_hall_floor);
  if constexpr (sizeof(R) == 4) {
    const R it = R(1.0) / ne_true, ie = R(1.0) / d.ne_eff;
    d.chiH = d.nH * it;
    d.chiNa = d.nNa * it;
    if (!(ne_true >= R(1.2e-38))) {  // no normal number: its reciprocal may overflow, the quotients are at most 1
      const bool some = ne_true > R(0.0);
      d.chiH = some ? d.nH / ne_true : R(1.0);
      d.chiNa = some ? d.nNa / ne_true : R(0.0);
    }
    d.wH = d.nH * ie;
    d.wNa = d.nNa * ie;
    return d;
  }
  if ((double)ne_true > 1.0e-300) {
    d.chiH = d.nH / ne_true;
    d.chiNa = d.nNa / ne_true;
  } else {
    d.chiH = R(1.0);
    d.chiNa = R(0.0);
  }
  d.wH = d.nH / d.ne_eff;
  d.wNa = d.nNa / d.ne_eff;
  return d;
}

__device__ __forceinline__ void shift1(int axis, int &i, int &j, int &k, int s) {
  if (axis == 0) i += s;
  else if (axis == 1) j += s;
  else k += s;
}

// ------------------------------------------------------------------ ideal EMF
// AssembleOneDirectionEMF_ (Ideal.cpp:433-594) for all three face families on
// [-1, inner_hi + 1) (the one locally evaluated ghost layer, Ideal.cpp:548-555),
// and, with the ambipolar term on, the node electron pressure on [0, n + 1)
// that the edge EMFs of the owned edges read (each node is shared by six
// edges) and the grad p_e source term of the owned cells that the fluid
// update of both species reads.  A cell is the right cell of its three faces:
// its cell-averaged total and induced B and its contravariant velocities are
// evaluated once.
template <class R>
__global__ void __launch_bounds__(kVecThreads, sizeof(R) == 8 ? 2 : 3) k_face_emf(Dir D) {
  for_vec_items<R, kExt>(D, [&](const DevSolve &S, const VV<R> &B, const VItem &it) {
    const int i = it.i, j = it.j;
    const uint32_t o = it.o, di = B.di, dj = B.dj;
    // Behind every load where the registers allow it (FP64; lv): a step of the 32^3
    // FP64 box takes 73 us, 77 with stores in between; in FP32 one fewer CTA fits.
    constexpr bool kLate = sizeof(R) == 8;
    const bool ambi = uniform(consts_of<R>(S).ambipolar) != 0;
    Vec<R> pnode, dpe[3];
    auto put_pe = [&] {
      B.st(cPEN, it, pnode, 0, B.n2 + 1, i >= 0 && j >= 0 && i <= B.n0 && j <= B.n1);
#pragma unroll
      for (int q = 0; q < 3; ++q) B.st(cDPE + q, it, dpe[q], 0, B.n2, i >= 0 && j >= 0 && i < B.n0 && j < B.n1);
    };
    if (ambi) {
      auto pe = [&](uint32_t q) { return B.lv(cPVH + 3, q) + B.lv(cPVN + 3, q); };
      auto pe1 = [&](uint32_t q) { return B.ld(cPVH + 3, q) + B.ld(cPVN + 3, q); };
      constexpr uint32_t es = sizeof(R);
      const Vec<R> p0 = pe(o), pim = pe(o - di), pjm = pe(o - dj), pijm = pe(o - di - dj);
      const Vec<R> pkm = vdown(p0, pe1(o - es));
      // the mean of p_H + p_Na over the 8 cells around the node, summed in the
      // order of AddAmbipolarEdgeEMF_ (MercurySolver_MagExplicit_Ambipo.cpp:3-143)
      Vec<R> sum = R(0.0) + vdown(pijm, pe1(o - di - dj - es));
      sum = sum + pijm;
      sum = sum + vdown(pim, pe1(o - di - es));
      sum = sum + pim;
      sum = sum + vdown(pjm, pe1(o - dj - es));
      sum = sum + pjm;
      sum = sum + pkm;
      sum = sum + p0;
      pnode = R(0.125) * sum;
      {
        // grad p_e term of the ion momentum sources of an owned cell, the
        // same for both species (AddSourceToRHS_Fluid, FluidRHS.cpp:206-527)
        const Vec<R> gi = pe(o + di) - pim, gj = pe(o + dj) - pjm, gk = vup(p0, pe1(o + 16u)) - pkm;
#pragma unroll
        for (int q = 0; q < 3; ++q)
          dpe[q] = R(0.5) * (B.fixed(cAMB + q, o) * gi + B.fixed(cAMB + 3 + q, o) * gj + B.fixed(cAMB + 6 + q, o) * gk);
      }
      if (!kLate) put_pe();
    }
    // induced and total B averaged to the cells (cell_beta_ind, cell_beta_tot)
    auto ind = [&](int a, uint32_t q, uint32_t d) { return R(0.5) * (B.lv(cBX + a, q) + B.lv(cBX + a, q + d)); };
    auto tot = [&](int a, uint32_t q, uint32_t d) {
      return R(0.5) * ((B.lv(cBX + a, q) + B.fixed(cBAX + a, q)) + (B.lv(cBX + a, q + d) + B.fixed(cBAX + a, q + d)));
    };
    auto ind_k = [&](uint32_t q) {  // along k: the cell's upper face is the next position
      const Vec<R> b = B.lv(cBZ, q);
      return R(0.5) * (b + B.upper(b, cBZ, q));
    };
    auto tot_k = [&](uint32_t q) {
      const Vec<R> b = B.lv(cBZ, q) + B.fixed(cBAZ, q);
      return R(0.5) * (b + vup(b, B.ld(cBZ, q + 16u) + B.fixed1(cBAZ, q + 16u)));
    };
    const Vec<R> bt[3] = {tot(0, o, di), tot(1, o, dj), tot_k(o)};
    const Vec<R> bi[3] = {ind(0, o, di), ind(1, o, dj), ind_k(o)};
    const Vec<R> u[3] = {B.lv(cUC, o), B.lv(cUC + 1, o), B.lv(cUC + 2, o)};
    // flux() of AssembleOneDirectionEMF_ (Ideal.cpp:517-536) of component a of B
    // through the face family f, from the left cell's values
    auto flux = [&](int a, int f, const Vec<R> &btL, const Vec<R> &biL, const Vec<R> &ufL, const Vec<R> &ubL,
                    const Vec<R> &bff) {
      const Vec<R> GL = ufL * btL - ubL * bff, GR = u[f] * bt[a] - u[a] * bff;
      const Vec<R> r = vmax(vabs(ufL), vabs(u[f]));
      return R(0.5) * (GL + GR) - R(0.5) * r * (bi[a] - biL);
    };
    const bool ri = i < B.n0 + 1, rj = j < B.n1 + 1;  // in the range of the other families
    const int k1 = B.n2 + 1;
    Vec<R> xe, xz, yx, yz;  // the fluxes: face family, component
    auto put_x = [&] {
      B.st(cEFX, it, vset(R(0.0)), -1, k1, rj);
      B.st(cEFX + 1, it, xz, -1, k1, rj);
      B.st(cEFX + 2, it, -xe, -1, k1, rj);
    };
    auto put_y = [&] {
      B.st(cEFY, it, -yz, -1, k1, ri);
      B.st(cEFY + 1, it, vset(R(0.0)), -1, k1, ri);
      B.st(cEFY + 2, it, yx, -1, k1, ri);
    };
    {
      const Vec<R> bff = B.lv(cBX, o) + B.fixed(cBAX, o);
      const uint32_t q = o - di;
      const Vec<R> ufL = B.lv(cUC, q);
      xe = flux(1, 0, tot(1, q, dj), ind(1, q, dj), ufL, B.lv(cUC + 1, q), bff);
      xz = flux(2, 0, tot_k(q), ind_k(q), ufL, B.lv(cUC + 2, q), bff);
      if (!kLate) put_x();
    }
    {
      const Vec<R> bff = B.lv(cBY, o) + B.fixed(cBAY, o);
      const uint32_t q = o - dj;
      const Vec<R> ufL = B.lv(cUC + 1, q);
      yx = flux(0, 1, tot(0, q, di), ind(0, q, di), ufL, B.lv(cUC, q), bff);
      yz = flux(2, 1, tot_k(q), ind_k(q), ufL, B.lv(cUC + 2, q), bff);
      if (!kLate) put_y();
    }
    {
      const Vec<R> bff = B.lv(cBZ, o) + B.fixed(cBAZ, o);
      const uint32_t q = o - (uint32_t)sizeof(R);  // the cell one k lower: its values from this thread's, and one more
      auto totL = [&](int a, uint32_t d) {
        return vdown(bt[a], R(0.5) * ((B.ld(cBX + a, q) + B.fixed1(cBAX + a, q)) + (B.ld(cBX + a, q + d) + B.fixed1(cBAX + a, q + d))));
      };
      auto indL = [&](int a, uint32_t d) { return vdown(bi[a], R(0.5) * (B.ld(cBX + a, q) + B.ld(cBX + a, q + d))); };
      const Vec<R> ufL = vdown(u[2], B.ld(cUC + 2, q));
      const Vec<R> Gx = flux(0, 2, totL(0, di), indL(0, di), ufL, vdown(u[0], B.ld(cUC, q)), bff);
      const Vec<R> Ge = flux(1, 2, totL(1, dj), indL(1, dj), ufL, vdown(u[1], B.ld(cUC + 1, q)), bff);
      if (kLate) {
        put_x();
        put_y();
        if (ambi) put_pe();
      }
      B.st(cEFZ, it, Ge, -1, k1 + 1, ri && rj);
      B.st(cEFZ + 1, it, -Gx, -1, k1 + 1, ri && rj);
      B.st(cEFZ + 2, it, vset(R(0.0)), -1, k1 + 1, ri && rj);
    }
  });
}

// AddArtificialResistivityToEdgeEMF_ and AddLocalArtificialResistivityToEdgeEMF_
// (Z4_Mercury/src/physics/MercurySolver_MagExplicit_Resis.cpp:6-64, 66-185) on owned edges of
// family `axis`: E += eta_art(|J| / |dr|) J, then E += eta_local J.
template <class R>
__device__ __forceinline__ Vec<R> add_artificial(const VV<R> &B, const ConstsT<R> &c, int axis, uint32_t o, Vec<R> e) {
  const int cj = cJX + axis;
  if (uniform((int)(c.arti_eta_max > R(0.0)))) {
    const int cd = axis == 0 ? cDRX : axis == 1 ? cDRY : cDRZ;
    const Vec<R> J = B.lv(cj, o), dx = B.fixed(cd, o), dy = B.fixed(cd + 1, o), dz = B.fixed(cd + 2, o);
#pragma unroll
    for (int q = 0; q < Vec<R>::N; ++q) {
      const R dr_len = sqrt(dx.v[q] * dx.v[q] + dy.v[q] * dy.v[q] + dz.v[q] * dz.v[q]);
      const R Jmag = fabs(J.v[q]) / dmax(dr_len, R(1.0e-30));
      R eta;
      if (c.arti_J_on <= c.arti_J_start) {
        eta = (Jmag > c.arti_J_start) ? c.arti_eta_max : R(0.0);
      } else {
        R x = (Jmag - c.arti_J_start) / (c.arti_J_on - c.arti_J_start);
        x = dmax(R(0.0), dmin(R(1.0), x));
        const R S = x * x * (R(3.0) - R(2.0) * x);
        eta = c.arti_eta_max * S;
      }
      e.v[q] += eta * J.v[q];
    }
  }
  if (uniform(c.local_arti)) e = e + B.fixed(cLEX + axis, o) * B.lv(cj, o);
  return e;
}

// AssembleEdgeEMF_FromFaceE_Ideal_ (Ideal.cpp:138-372) + AddAmbipolarEdgeEMF_
// (Z4_Mercury/src/physics/MercurySolver_MagExplicit_Ambipo.cpp:3-143), then the Hall EMF
// (BuildHallFaceEMF_Rusanov_diff_ steps 2-4, Hall.cpp:148-400) on the owned
// edges.  An edge inside the block has no alias: its sum E + Ehall
// (MercurySolver_MagneticRHS.cpp:135-147) is written at once, so only the edges
// on the block's faces wait for the alias reduction and k_add_hall.
template <class R>
__global__ void __launch_bounds__(kVecThreads, 3) k_edge_emf(Dir D) {
  for_vec_items<R, kBox>(D, [&](const DevSolve &S, const VV<R> &B, const VItem &it) {
    const ConstsT<R> &c = consts_of<R>(S);
    const uint32_t o = it.o, di = B.di, dj = B.dj;
    const R Cuct = R(0.5);
    Vec<R> E[3];
    const R pc = c.pe_coeff;
    auto lowk = [&](const Vec<R> &v, int comp, uint32_t q) { return B.lower(v, comp, q); };
    // max |u^a| over the four cells at an edge: this row, the row below along
    // d, and, for the edges that are not along k, both one k lower
    auto umax_k = [&](int a, uint32_t d) {
      const Vec<R> x = B.lv(cUC + a, o), y = B.lv(cUC + a, o - d);
      Vec<R> r = vmax(vset(R(0.0)), vabs(x));
      r = vmax(r, vabs(y));
      r = vmax(r, vabs(lowk(x, cUC + a, o)));
      return vmax(r, vabs(lowk(y, cUC + a, o - d)));
    };
    auto umax_ij = [&](int a) {
      Vec<R> r = vmax(vset(R(0.0)), vabs(B.lv(cUC + a, o)));
      r = vmax(r, vabs(B.lv(cUC + a, o - di)));
      r = vmax(r, vabs(B.lv(cUC + a, o - dj)));
      return vmax(r, vabs(B.lv(cUC + a, o - di - dj)));
    };
    // ne_eff of the densities averaged over the four cells
    auto ne_of = [&](const Vec<R> &rH, const Vec<R> &rN) {
      return vmap<R>([&](int e) { return num_limiter(c, R(0.25) * rH.v[e], R(0.25) * rN.v[e]).ne_eff; });
    };
    auto rho_k = [&](int comp, uint32_t d) {  // the row below along d first, k - 1 before k
      const Vec<R> y = B.lv(comp, o - d), x = B.lv(comp, o);
      Vec<R> r = R(0.0) + lowk(y, comp, o - d);
      r = r + y;
      r = r + lowk(x, comp, o);
      return r + x;
    };
    auto rho_ij = [&](int comp) {
      Vec<R> r = R(0.0) + B.lv(comp, o - di - dj);
      r = r + B.lv(comp, o - di);
      r = r + B.lv(comp, o - dj);
      return r + B.lv(comp, o);
    };
    const int ambi = uniform(c.ambipolar);
    const Vec<R> pn = ambi ? B.lv(cPEN, o) : vset(R(0.0));
    {
      const Vec<R> fy = B.lv(cEFY, o), by = B.lv(cBY, o);
      const Vec<R> Ec = R(0.25) * (fy + lowk(fy, cEFY, o) + B.lv(cEFZ, o) + B.lv(cEFZ, o - dj));
      const Vec<R> ae = umax_k(1, dj), az = umax_k(2, dj);
      const Vec<R> d1 = B.lv(cBZ, o) - B.lv(cBZ, o - dj);
      const Vec<R> d2 = by - lowk(by, cBY, o);
      Vec<R> e = Ec + Cuct * (R(0.5) * ae * d1 - R(0.5) * az * d2);
      if (ambi) e = e - pc * (B.lv(cPEN, o + di) - pn) / ne_of(rho_k(cUH, dj), rho_k(cUN, dj));
      E[0] = add_artificial(B, c, 0, o, e);
    }
    {
      const Vec<R> fx = B.lv(cEFX + 1, o), bx = B.lv(cBX, o);
      const Vec<R> Ec = R(0.25) * (fx + lowk(fx, cEFX + 1, o) + B.lv(cEFZ + 1, o) + B.lv(cEFZ + 1, o - di));
      const Vec<R> az = umax_k(2, di), ax = umax_k(0, di);
      const Vec<R> d1 = bx - lowk(bx, cBX, o);
      const Vec<R> d2 = B.lv(cBZ, o) - B.lv(cBZ, o - di);
      Vec<R> e = Ec + Cuct * (R(0.5) * az * d1 - R(0.5) * ax * d2);
      if (ambi) e = e - pc * (B.lv(cPEN, o + dj) - pn) / ne_of(rho_k(cUH, di), rho_k(cUN, di));
      E[1] = add_artificial(B, c, 1, o, e);
    }
    {
      const Vec<R> Ec =
          R(0.25) * (B.lv(cEFX + 2, o) + B.lv(cEFX + 2, o - dj) + B.lv(cEFY + 2, o) + B.lv(cEFY + 2, o - di));
      const Vec<R> ax = umax_ij(0), ae = umax_ij(1);
      const Vec<R> d1 = B.lv(cBY, o) - B.lv(cBY, o - di);
      const Vec<R> d2 = B.lv(cBX, o) - B.lv(cBX, o - dj);
      Vec<R> e = Ec + Cuct * (R(0.5) * ax * d1 - R(0.5) * ae * d2);
      if (ambi) e = e - pc * (B.upper(pn, cPEN, o) - pn) / ne_of(rho_ij(cUH), rho_ij(cUN));
      E[2] = add_artificial(B, c, 2, o, e);
    }
    const R Cwh = R(0.1);
    Vec<R> h[3];  // E_Hall
    // over the four cells at an edge, in the reference's order: lower row and
    // lower k first
    auto mean_k = [&](int comp, uint32_t d) {
      const Vec<R> y = B.lv(comp, o - d), x = B.lv(comp, o);
      return R(0.25) * (B.lower(y, comp, o - d) + y + B.lower(x, comp, o) + x);
    };
    auto max_k = [&](int comp, uint32_t d) {
      const Vec<R> y = B.lv(comp, o - d), x = B.lv(comp, o);
      return vmax(vmax(B.lower(y, comp, o - d), y), vmax(B.lower(x, comp, o), x));
    };
    auto mean_ij = [&](int comp) {
      return R(0.25) * (B.lv(comp, o - di - dj) + B.lv(comp, o - di) + B.lv(comp, o - dj) + B.lv(comp, o));
    };
    auto tail = [&](int ax, const Vec<R> &Ecen, const Vec<R> &be, const Vec<R> &d1, const Vec<R> &d2) {
      const int ci = ax == 0 ? cIHX : ax == 1 ? cIHY : cIHZ;
      const Vec<R> ih1 = B.fixed(ci, o), ih2 = B.fixed(ci + 1, o);
      const Vec<R> mu1 = Cwh * be * ih1 * ih1;
      const Vec<R> mu2 = Cwh * be * ih2 * ih2;
      return B.fixed(cTPX + ax, o) * (Ecen + R(0.5) * mu1 * d1 - R(0.5) * mu2 * d2);
    };
    {
      const Vec<R> Ecen = mean_k(cEHC, dj) * B.fixed(cDRX, o) + mean_k(cEHC + 1, dj) * B.fixed(cDRX + 1, o) +
                          mean_k(cEHC + 2, dj) * B.fixed(cDRX + 2, o);
      const Vec<R> by = B.lv(cBY, o);
      h[0] = tail(0, Ecen, max_k(cHB, dj), B.lv(cBZ, o) - B.lv(cBZ, o - dj), by - B.lower(by, cBY, o));
    }
    {
      const Vec<R> Ecen = mean_k(cEHC, di) * B.fixed(cDRY, o) + mean_k(cEHC + 1, di) * B.fixed(cDRY + 1, o) +
                          mean_k(cEHC + 2, di) * B.fixed(cDRY + 2, o);
      const Vec<R> bx = B.lv(cBX, o);
      h[1] = tail(1, Ecen, max_k(cHB, di), bx - B.lower(bx, cBX, o), B.lv(cBZ, o) - B.lv(cBZ, o - di));
    }
    {
      const Vec<R> Ecen =
          mean_ij(cEHC) * B.fixed(cDRZ, o) + mean_ij(cEHC + 1) * B.fixed(cDRZ + 1, o) + mean_ij(cEHC + 2) * B.fixed(cDRZ + 2, o);
      const Vec<R> be = vmax(vmax(B.lv(cHB, o - di - dj), B.lv(cHB, o - di)), vmax(B.lv(cHB, o - dj), B.lv(cHB, o)));
      h[2] = tail(2, Ecen, be, B.lv(cBY, o) - B.lv(cBY, o - di), B.lv(cBX, o) - B.lv(cBX, o - dj));
    }
    // E_Hall of family ax, and E: with it inside the block, without on its faces
    // (the stores behind every load: lv)
    const bool late = S.hall_late != 0;
    auto put = [&](int ax, int hi, bool owned, bool face, bool kfaces) {
      B.st(cHX + ax, it, h[ax], 0, hi, owned);
      B.st(cEX + ax, it, vmap<R>([&](int e) {
             const bool f = face || (kfaces && (it.k + e == 0 || it.k + e == B.n2));
             return f ? E[ax].v[e] : E[ax].v[e] + h[ax].v[e];
           }), 0, hi, owned);
    };
    put(0, B.n2 + 1, it.i < B.n0, late || it.j == 0 || it.j == B.n1, true);
    put(1, B.n2 + 1, it.j < B.n1, late || it.i == 0 || it.i == B.n0, true);
    put(2, B.n2, true, late || it.i == 0 || it.i == B.n0 || it.j == 0 || it.j == B.n1, false);
  });
}

// E += Ehall (Z4_Mercury/src/physics/MercurySolver_MagneticRHS.cpp:135-147) on the owned
// edges that lie in the block's faces (k_edge_emf has summed the others).
template <class R>
__global__ void __launch_bounds__(kVecThreads) k_add_hall(Dir D) {
  for_vec_items<R, kBox>(D, [&](const DevSolve &S, const VV<R> &B, const VItem &it) {
    const bool late = S.hall_late != 0;  // every edge
    const bool fi = late || it.i == 0 || it.i == B.n0, fj = late || it.j == 0 || it.j == B.n1;
    const bool k0 = it.k <= 0, k1 = it.k <= B.n2 && it.k + Vec<R>::N > B.n2;
    if (!it.in || !(fi || fj || k0 || k1)) return;
    // each thread reads and writes its own positions only
    auto add = [&](int ax, int lo, int hi, bool cond) {
      B.st(cEX + ax, it, B.lv(cEX + ax, it.o) + B.lv(cHX + ax, it.o), lo, hi, cond);
    };
    // family xi: on the eta faces whole rows, else the ends of the row; eta likewise; zeta: whole rows
    if (it.i < B.n0) {
      add(0, 0, B.n2 + 1, fj);
      add(0, 0, 1, !fj && k0);
      add(0, B.n2, B.n2 + 1, !fj && k1);
    }
    if (it.j < B.n1) {
      add(1, 0, B.n2 + 1, fi);
      add(1, 0, 1, !fi && k0);
      add(1, B.n2, B.n2 + 1, !fi && k1);
    }
    if (fi || fj) add(2, 0, B.n2, true);
  });
}

// ------------------------------------------------------------------ fluid update
// A cell's quantities in the Rusanov flux of Scheme_U_
// (Z4_Mercury/src/physics/MercurySolver_FluidRHS.cpp:36-104): rho, u, v, w, p
// and re = p / (g - 1) + rho |u|^2 / 2, c = sqrt(g p / rho), which Scheme_U_
// evaluates per face with the same operations on the same cell values
// (k_pv_uplus stores them per cell).
template <class R>
struct FluidCell {
  R rho, u, v, w, p, re, c;
};
template <class R>
__device__ __forceinline__ FluidCell<R> fluid_cell(const V<R> &B, int s, uint32_t o) {
  const int pv0 = s ? cPVN : cPVH, t0 = cFT + 2 * s;
  FluidCell<R> q;
  q.rho = B.fixed1(s ? cUN : cUH, o);
  q.u = B.fixed1(pv0, o);
  q.v = B.fixed1(pv0 + 1, o);
  q.w = B.fixed1(pv0 + 2, o);
  q.p = B.fixed1(pv0 + 3, o);
  q.re = B.fixed1(t0, o);
  q.c = B.fixed1(t0 + 1, o);
  return q;
}
// A face's JD and |JD|: FP32 reads the real-typed copy (k_face_normals), FP64
// the metric itself (the same values).
template <class R>
struct FluidFace {
  R k1, k2, k3, sk;
};
template <class R, int DIR>
__device__ __forceinline__ FluidFace<R> fluid_face(const V<R> &B, uint32_t o) {
  constexpr int cm = sizeof(R) == 4 ? cFM + 3 * DIR : DIR == 0 ? cJDX : DIR == 1 ? cJDY : cJDZ;
  constexpr int cn = DIR == 0 ? cFNX : DIR == 1 ? cFNY : cFNZ;
  FluidFace<R> f;
  if constexpr (sizeof(R) == 4) {
    f.k1 = B.fixed1(cm, o);
    f.k2 = B.fixed1(cm + 1, o);
    f.k3 = B.fixed1(cm + 2, o);
  } else {
    f.k1 = B.ldm(cm, o);
    f.k2 = B.ldm(cm + 1, o);
    f.k3 = B.ldm(cm + 2, o);
  }
  f.sk = B.fixed1(cn + 3, o);
  return f;
}
template <class R>
__device__ __forceinline__ void rusanov(const FluidCell<R> &L, const FluidCell<R> &Q, const FluidFace<R> &f, R out[5]) {
  const R uvwL = f.k1 * L.u + f.k2 * L.v + f.k3 * L.w, uvwR = f.k1 * Q.u + f.k2 * Q.v + f.k3 * Q.w;
  const R rad = dmax(fabs(uvwL) + L.c * f.sk, fabs(uvwR) + Q.c * f.sk);
  out[0] = R(0.5) * (L.rho * uvwL + Q.rho * uvwR) - R(0.5) * rad * (Q.rho - L.rho);
  out[1] = R(0.5) * ((L.rho * uvwL * L.u + f.k1 * L.p) + (Q.rho * uvwR * Q.u + f.k1 * Q.p)) -
           R(0.5) * rad * (Q.rho * Q.u - L.rho * L.u);
  out[2] = R(0.5) * ((L.rho * uvwL * L.v + f.k2 * L.p) + (Q.rho * uvwR * Q.v + f.k2 * Q.p)) -
           R(0.5) * rad * (Q.rho * Q.v - L.rho * L.v);
  out[3] = R(0.5) * ((L.rho * uvwL * L.w + f.k3 * L.p) + (Q.rho * uvwR * Q.w + f.k3 * Q.p)) -
           R(0.5) * rad * (Q.rho * Q.w - L.rho * L.w);
  out[4] = R(0.5) * (uvwL * (L.re + L.p) + uvwR * (Q.re + Q.p)) - R(0.5) * rad * (Q.re - L.re);
}

// ZeroRHS_ + Scheme_U_ + AddSourceToRHS_Fluid (FluidRHS.cpp:206-527) +
// ApplyUpdate_Euler_ (Z4_Mercury/src/physics/MercurySolver_Advance.cpp:73-147)
// for one tile of owned cells and both ion species; the state goes to the
// other buffer.  A thread takes a column of the tile's cells along i: the
// flux through the face between two of them is computed once and carried
// over, the fluxes of the cell's four other faces are computed by each of
// the two cells that share one, from loads that hit L1 (no shared memory, no
// barrier).  Every cell then takes its six faces' differences direction by
// direction, r[m] -= (F+ - F-) / J, the per-component order of Scheme_U_'s
// divergence.
// Bound by the latency of its loads: 15 to 24 warps per SM at the register
// budget that keeps most of a cell's loads in flight.  On the 96^3 mixed box
// 0.086 ms (0.150 for the shared-memory tile of face fluxes this replaced: 84 M
// warp instructions against 40 M), on 64 x 64 x 128 cells in FP64 0.112 ms
// (0.178); 236 B per cell would take 0.032 and 472 B 0.038.
// Columns are the tile's whole depth along i; when the tiles would not fill the
// grid they are cut into single cells, which trades the carried flux for four
// times the threads (32^3 in FP64: 0.025 ms in columns, 0.017 in cells; 64^3
// mixed, where the tiles fill the grid: 0.040 and 0.041).
template <class R, int VT>
__global__ void __launch_bounds__(fluid_threads(VT), fluid_ctas(VT, sizeof(R))) k_fluid(Dir D) {
  constexpr int KIND = fluid_kind(VT), NS = fluid_species(sizeof(R)), TI = fluid_tile(VT).i;
  __shared__ int sh[3];
  let_dependents_launch();
  const int items = D.solve_tile_prefix[KIND][D.nsolves] / NS;
  const int split = items < (int)gridDim.x ? TI : 1;
  const int li = TI / split;
  if ((int)blockIdx.x >= items * split) {
    if (blockIdx.x == 0) wait_for_predecessors();
    return;
  }
  for (int q = blockIdx.x; q < items * split; q += gridDim.x) {
    const int part = q % split;
    if (threadIdx.x == 0) lookup_item<KIND>(D, q / split * NS, sh[0], sh[1], sh[2]);
    __syncthreads();
    const int is = sh[0], ib = sh[1], t = sh[2];
    __syncthreads();
    Item it;
    V<R> B;
    build_item<R, KIND>(D, is, ib, t, it, B);
    if (q == (int)blockIdx.x) wait_for_predecessors();
    if (!solve_active(D, is)) continue;  // inactive solve (the whole CTA agrees)
    it.i += part;
    const DevSolve &S = D.solves[is];
    const ConstsT<R> &c = consts_of<R>(S);
    const R dt = __longlong_as_double((long long)D.state[it.s].dt_bits);
    // the reference aborts; flip_solve records the status (and a solve with a
    // non-finite cell is not advanced)
    if (!(dt >= R(1e-7)) || !isfinite(dt) || D.state[it.s].nonfinite || !it.in || it.i >= it.hi[0]) continue;
    const int j = it.j, k = it.k;
    const int s0 = NS == 2 ? 0 : it.species;
    {
      const uint32_t di = (uint32_t)B.si * sizeof(R), dj = (uint32_t)B.sj * sizeof(R), dk = sizeof(R);
      uint32_t o = (uint32_t)B.off(it.i, j, k) * sizeof(R);
      FluidCell<R> C[NS], N[NS];
      R Fm[NS][5];
      {
        const FluidFace<R> f = fluid_face<R, 0>(B, o);
#pragma unroll
        for (int q = 0; q < NS; ++q) {
          const int s = s0 + q, u0 = s ? cUN : cUH, pv0 = s ? cPVN : cPVH;
          const FluidCell<R> L = fluid_cell(B, s, o - di);
          C[q] = fluid_cell(B, s, o);
          rusanov(L, C[q], f, Fm[q]);
        }
      }
#pragma unroll 1
      for (int i = it.i; i < min(it.i + li, it.hi[0]); ++i, o += di) {
        const R invJ = B.fixed1(cFM + 9, o);  // R(1) / R(Jac), from k_face_normals
        R r[NS][5];
        {
          const FluidFace<R> f = fluid_face<R, 0>(B, o + di);
#pragma unroll
          for (int q = 0; q < NS; ++q) {
            const int s = s0 + q;
            N[q] = fluid_cell(B, s, o + di);
            R F[5];
            rusanov(C[q], N[q], f, F);
#pragma unroll
            for (int m = 0; m < 5; ++m) {
              r[q][m] = R(0.0) - (F[m] - Fm[q][m]) * invJ;
              Fm[q][m] = F[m];
            }
          }
        }
        auto across = [&](auto dirc, uint32_t d) {  // the faces below and above along j or k
          constexpr int dir = decltype(dirc)::value;
          const FluidFace<R> fl = fluid_face<R, dir>(B, o), fh = fluid_face<R, dir>(B, o + d);
#pragma unroll
          for (int q = 0; q < NS; ++q) {
            const int s = s0 + q;
            R Fl[5], Fh[5];
            rusanov(fluid_cell(B, s, o - d), C[q], fl, Fl);
            rusanov(C[q], fluid_cell(B, s, o + d), fh, Fh);
#pragma unroll
            for (int m = 0; m < 5; ++m) r[q][m] -= (Fh[m] - Fl[m]) * invJ;
          }
        };
        across(std::integral_constant<int, 1>{}, dj);
        across(std::integral_constant<int, 2>{}, dk);
        // sources (FluidRHS.cpp:206-527)
        auto at = [&](int comp) -> R { return B.fixed1(comp, o); };
        const R Tn0 = R(1000.0), sk1 = R(5.0e-5), sk2 = R(1.0e-5);
        const R a4 = c.src_a4, a5 = c.src_a5;
        const R upx = at(cUP), upy = at(cUP + 1), upz = at(cUP + 2);
        const R Bx = at(cBC), By = at(cBC + 1), Bz = at(cBC + 2);
        const R Jx = at(cJC), Jy = at(cJC + 1), Jz = at(cJC + 2);
        const R sjbx = Jy * Bz - Jz * By, sjby = Jz * Bx - Jx * Bz, sjbz = Jx * By - Jy * Bx;
        const Num<R> num = num_limiter(c, at(cUH), at(cUN));
        R dpex = R(0.0), dpey = R(0.0), dpez = R(0.0);
        if (c.ambipolar) {  // grad p_e term, once per cell (k_face_emf)
          dpex = at(cDPE);
          dpey = at(cDPE + 1);
          dpez = at(cDPE + 2);
        }
        const R x = at(cCX), y = at(cCX + 1), z = at(cCX + 2);
        const R rho_cyl = sqrt(y * y + z * z);
        const R vst = (x < R(0.0) && rho_cyl < R(1.0)) ? sk2 : sk1;
#pragma unroll
        for (int q = 0; q < NS; ++q) {
          const int s = s0 + q, u0 = s ? cUN : cUH, pv0 = s ? cPVN : cPVH;
          const R nS = s ? num.nNa : num.nH;
          const R chi = s ? num.wNa : num.wH;
          const R rho = dmax(C[q].rho, R(0.0));
          const R u = C[q].u, v = C[q].v, w = C[q].w;
          const R u2 = u * u + v * v + w * w;
          const R subx = (v - upy) * Bz - (w - upz) * By;
          const R suby = (w - upz) * Bx - (u - upx) * Bz;
          const R subz = (u - upx) * By - (v - upy) * Bx;
          const R subu = subx * u + suby * v + subz * w;
          const R sjbu = sjbx * u + sjby * v + sjbz * w;
          const R dpeu = dpex * u + dpey * v + dpez * w;
          const R Ts0 = at(pv0 + 4) * c.T_ref;
          const R b1 = vst * (Tn0 - Ts0) * c.src_b1[s], b2 = c.src_b2[s] * vst;
          R *rr = r[q];
          rr[1] += c.momentum_induce_coeff * nS * subx + c.momentum_hall_coeff * chi * sjbx;
          rr[2] += c.momentum_induce_coeff * nS * suby + c.momentum_hall_coeff * chi * sjby;
          rr[3] += c.momentum_induce_coeff * nS * subz + c.momentum_hall_coeff * chi * sjbz;
          rr[4] += c.momentum_induce_coeff * nS * subu + c.momentum_hall_coeff * chi * sjbu;
          if (c.ambipolar) {
            rr[1] -= chi * dpex;
            rr[2] -= chi * dpey;
            rr[3] -= chi * dpez;
            rr[4] -= chi * dpeu;
          }
          if (s) {
            const R sss = at(cPHOTO);
            rr[0] += c.src_a1Na * sss;
            rr[4] += c.src_a6 * sss * Tn0;
          }
          rr[1] -= a4 * rho * u * vst;
          rr[2] -= a4 * rho * v * vst;
          rr[3] -= a4 * rho * w * vst;
          rr[4] -= a4 * rho * u2 * vst;
          rr[4] += a5 * nS * b1;
          rr[4] += a4 * rho * u2 * b2;
          auto put = [&](int m, R v) { *(R *)((char *)B.next(u0 + m) + o) = v; };
          put(0, C[q].rho + dt * rr[0]);
#pragma unroll
          for (int m = 1; m < 5; ++m) put(m, at(u0 + m) + dt * rr[m]);
          C[q] = N[q];
        }
      }
    }
  }
}

// After the updates: flip the state buffer, account time/step
// (Z4_Mercury/src/MercurySolver_Driver.cpp:40-45), record a dt failure (the
// reference's exit(-1), Timestep.cpp:129-140) and re-arm the dt reduction.
__device__ __forceinline__ void flip_solve(SolveState &st) {
  if (!st.remaining) return;
  if (st.nonfinite) {  // a NaN/Inf cell: retire the solve, the others go on
    st.status = MHD_ERR_NONFINITE;
    st.remaining = 0;
    return;
  }
  const double dt = __longlong_as_double((long long)st.dt_bits);
  if (!(dt >= 1e-7) || !isfinite(dt)) {
    st.status = MHD_ERR_DT;
    st.remaining = 0;
    return;
  }
  st.cur ^= 1;
  st.dt = dt;
  st.time += dt;
  st.step += 1;
  st.dt_bits = (unsigned long long)__double_as_longlong(1e100);
}
// End of a step: one step fewer to go (after every pass of the step has run).
__device__ __forceinline__ void retire_solve(SolveState &st) {
  if (st.remaining > 0) st.remaining -= 1;
}

// B_face += dt * (-curl E) on the owned faces (CTOperators.cpp:6-56 with multiplier -1),
// and, the fluid update before it being complete, the flip of every solve's state.
template <class R>
__global__ void __launch_bounds__(kVecThreads) k_bface(Dir D) {
  for_vec_items<R, kBox>(D, [&](const DevSolve &S, const VV<R> &B, const VItem &it) {
    const R dt = __longlong_as_double((long long)D.state[it.s].dt_bits);
    if (uniform((int)(!(dt >= R(1e-7)) || !isfinite(dt) || D.state[it.s].nonfinite))) return;  // flip_solve records the status
    const uint32_t o = it.o, di = B.di, dj = B.dj;
    const bool ic = it.i < B.n0, jc = it.j < B.n1;
    const Vec<R> ex = B.lv(cEX, o), ey = B.lv(cEY, o), ez = B.lv(cEZ, o);
    {
      const Vec<R> rb = -R(1.0) * ((ey - B.upper(ey, cEY, o)) + (B.lv(cEZ, o + dj) - ez));
      B.st(cBX, it, B.lv(cBX, o) + dt * rb, 0, B.n2, jc);
    }
    {
      const Vec<R> rb = -R(1.0) * ((B.upper(ex, cEX, o) - ex) + (ez - B.lv(cEZ, o + di)));
      B.st(cBY, it, B.lv(cBY, o) + dt * rb, 0, B.n2, ic);
    }
    {
      const Vec<R> rb = -R(1.0) * ((ex - B.lv(cEX, o + dj)) + (B.lv(cEY, o + di) - ey));
      B.st(cBZ, it, B.lv(cBZ, o) + dt * rb, 0, B.n2 + 1, ic && jc);
    }
  });
  after_all_tiles<kBox>(D, D.tickets, [](SolveState &st) { flip_solve(st); });
}

// ------------------------------------------------------------------ derived fields
// calc_Bcell (Z4_Mercury/src/physics/MercurySolver_MagneticCell.cpp:3-90) on owned cells and
// CurlAdjFaceToEdge + alpha scaling of Calc_J_Edge (CTOperators.cpp:59-110,
// Z4_Mercury/src/physics/MercurySolver_Current.cpp:140-190) on owned edges.
template <class R>
__global__ void __launch_bounds__(kVecThreads, 3) k_bcell_jedge(Dir D) {
  for_vec_items<R, kBox>(D, [&](const DevSolve &S, const VV<R> &B, const VItem &it) {
    const uint32_t o = it.o, di = B.di, dj = B.dj;
    const bool ic = it.i < B.n0, jc = it.j < B.n1;
    const Vec<R> bx = B.lv(cBX, o), by = B.lv(cBY, o), bz = B.lv(cBZ, o);
    // beta B on this position's faces and the lower neighbours'
    const Vec<R> fx = B.fixed(cBFX, o) * bx, fy = B.fixed(cBFY, o) * by, fz = B.fixed(cBFZ, o) * bz;
    auto below = [&](int a, uint32_t d) { return B.fixed(cBFX + a, o - d) * B.lv(cBX + a, o - d); };
    constexpr uint32_t es = sizeof(R);
    Vec<R> J[3];
    {
      const Vec<R> v = ((vdown(fy, B.fixed1(cBFY, o - es) * B.ld(cBY, o - es)) - fy) + (fz - below(2, dj))) * R(1.0);
      J[0] = v * B.fixed(cALX, o);
    }
    {
      const Vec<R> v = ((fx - vdown(fx, B.fixed1(cBFX, o - es) * B.ld(cBX, o - es))) + (below(2, di) - fz)) * R(1.0);
      J[1] = v * B.fixed(cALY, o);
    }
    {
      const Vec<R> v = ((below(0, dj) - fx) + (fy - below(1, di))) * R(1.0);
      J[2] = v * B.fixed(cALZ, o);
    }
    const Vec<R> ax = B.fixed(cBAX, o), ay = B.fixed(cBAY, o), az = B.fixed(cBAZ, o);
    const Vec<R> bxp = B.lv(cBX, o + di), byp = B.lv(cBY, o + dj), bzp = B.upper(bz, cBZ, o);
    Vec<R> t[3] = {vset(R(0.0)), vset(R(0.0)), vset(R(0.0))}, in[3] = {t[0], t[0], t[0]};
    auto add = [&](int q, const Vec<R> &total, const Vec<R> &induced) {  // face q of the cell
#pragma unroll
      for (int x = 0; x < 3; ++x) {
        const Vec<R> w = B.fixed(cWB + 6 * x + q, o);
        t[x] = t[x] + w * total;
        in[x] = in[x] + w * induced;
      }
    };
    add(0, -bx - ax, -bx);
    add(1, bxp + B.fixed(cBAX, o + di), bxp);
    add(2, -by - ay, -by);
    add(3, byp + B.fixed(cBAY, o + dj), byp);
    add(4, -bz - az, -bz);
    add(5, bzp + B.fixed_upper(az, cBAZ, o), bzp);
    // the stores behind every load
#pragma unroll
    for (int x = 0; x < 3; ++x) {
      B.st(cBC + x, it, t[x], 0, B.n2, ic && jc);
      B.st(cBIC + x, it, in[x], 0, B.n2, ic && jc);
    }
    B.st(cJX, it, J[0], 0, B.n2 + 1, ic);
    B.st(cJY, it, J[1], 0, B.n2 + 1, jc);
    B.st(cJZ, it, J[2], 0, B.n2);
  });
}

// calc_Jcell (Current.cpp:203-243), owned cells.
template <class R>
__global__ void __launch_bounds__(kVecThreads, 3) k_jcell(Dir D) {
  for_vec_items<R, kCells>(D, [&](const DevSolve &S, const VV<R> &B, const VItem &it) {
    const uint32_t o = it.o, di = B.di, dj = B.dj;
    Vec<R> j[3] = {vset(R(0.0)), vset(R(0.0)), vset(R(0.0))};
    auto add = [&](int q, const Vec<R> &s) {  // edge q of the cell, the summation order of calc_Jcell
#pragma unroll
      for (int x = 0; x < 3; ++x) j[x] = j[x] + B.fixed(cWJ + 12 * x + q, o) * s;
    };
    const Vec<R> ax = B.lv(cJX, o), bx = B.lv(cJX, o + dj), ay = B.lv(cJY, o), by = B.lv(cJY, o + di);
    const Vec<R> ux = B.upper(ax, cJX, o), vx = B.upper(bx, cJX, o + dj);
    const Vec<R> uy = B.upper(ay, cJY, o), vy = B.upper(by, cJY, o + di);
    const Vec<R> z0 = B.lv(cJZ, o), z1 = B.lv(cJZ, o + di), z2 = B.lv(cJZ, o + dj), z3 = B.lv(cJZ, o + di + dj);
    add(0, ax);
    add(1, bx);
    add(2, ux);
    add(3, vx);
    add(4, ay);
    add(5, by);
    add(6, uy);
    add(7, vy);
    add(8, z0);
    add(9, z1);
    add(10, z2);
    add(11, z3);
#pragma unroll
    for (int x = 0; x < 3; ++x) B.st(cJC + x, it, j[x], 0, B.n2);
  });
}

// Quotients by one divisor b >= 1e-12.  FP32: by its reciprocal.  FP64: the quotient
// that IEEE division rounds to, from the correctly rounded reciprocal y = RN(1/b)
// and one residual, q = RN(a y), RN(q + RN(a - b q) y) (Markstein, "Computation
// of elementary functions on the IBM RISC System/6000 processor", 1990): exact
// while y, the quotient and the residual are normal numbers, so a outside
// [2^-600, 2^930) and any a by a divisor from 2^332 on (or NaN) is divided (a zero
// keeps its sign).  The ranges are tested on the upper words: tests of the
// quotient in FP64 took 6 to 10 % of a step.
template <class R>
struct Divisor {
  static constexpr uint32_t kLow = (1023u - 600u) << 20, kSpan = ((1023u + 930u) << 20) - kLow, kTop = (1023u + 332u) << 20;
  R b, y;
  uint32_t span;  // FP64: the range's width, 0 where everything is divided
  __device__ __forceinline__ Divisor(R d, R recip) : b(d), y(recip), span(0) {
    if constexpr (sizeof(R) == 8) span = (uint32_t)__double2hiint(d) < kTop ? kSpan : 0u;
  }
  __device__ __forceinline__ explicit Divisor(R d) : Divisor(d, reciprocal(d)) {}
  __device__ __forceinline__ static R reciprocal(R d) {
    if constexpr (sizeof(R) == 4) return R(1.0) / d;
    else return __drcp_rn(d);
  }
  __device__ __forceinline__ R operator()(R a) const {
    if constexpr (sizeof(R) == 4) return a * y;
    else {
      const R q = a * y;
      if (((uint32_t)__double2hiint(a) & 0x7fffffffu) - kLow < span) return fma(fma(-b, q, a), y, q);
      return a == R(0.0) ? q : a / b;
    }
  }
};

// CFL time step of a thread's cells and both species (Compute_Timestep,
// Z4_Mercury/src/physics/MercurySolver_Timestep.cpp:8-141): the smallest over
// the cells.  (nx, ny, nz, An) are a face's precomputed a / |a| and |a|
// (k_face_normals: the same operations as the reference evaluates per face);
// vA2 = inver_MA2 * B2 / rho is the same for all faces of a cell and species.
template <class R>
__device__ __forceinline__ R fast_cf(R cs2, R vA2, R vAn2) {
  const R term = cs2 + vA2;
  R disc = term * term - R(4.0) * cs2 * vAn2;
  if (disc < R(0.0)) disc = R(0.0);
  return sqrt(R(0.5) * (term + sqrt(disc)));
}
template <class R, int N>
__device__ __forceinline__ R cells_dt(const VV<R, N> &B, const ConstsT<R> &c, const VItem &it, bool own,
                                      const Vec<R, N> &Bx, const Vec<R, N> &By, const Vec<R, N> &Bz, bool &bad) {
  using Vc = Vec<R, N>;
  const uint32_t o = it.o;
  const Vc Vol = vabs(B.lm(cJAC, o));
  const Vc B2 = Bx * Bx + By * By + Bz * Bz;
  Vc d = vset<R, N>(R(1e100));
#pragma unroll 1
  for (int s = 0; s < 2; ++s) {
    const int u0 = s ? cUN : cUH;
    const Vc rho0 = B.lv(u0, o), m1 = B.lv(u0 + 1, o), m2 = B.lv(u0 + 2, o), m3 = B.lv(u0 + 3, o), E = B.lv(u0 + 4, o);
    Vc ux, uy, uz, cs2, vA2, den = vset<R, N>(R(0.0)), rho, y;
#pragma unroll
    for (int e = 0; e < N; ++e) {
      rho.v[e] = dmax(rho0.v[e], R(1e-2));
      const Divisor<R> by(rho.v[e]);
      y.v[e] = by.y;
      const R u = by(m1.v[e]), v = by(m2.v[e]), w = by(m3.v[e]);
      const R ke = R(0.5) * rho.v[e] * (u * u + v * v + w * w);
      const R pr = (c.gamma - R(1.0)) * (E.v[e] - ke);
      cs2.v[e] = by(c.gamma * pr);
      vA2.v[e] = by(c.inver_MA2 * B2.v[e]);
      ux.v[e] = u;
      uy.v[e] = v;
      uz.v[e] = w;
    }
    // faces xi-, xi+, eta-, eta+, zeta-, zeta+ (the reference's summation order)
    // (the outward normal's sign changes neither |u . n| nor (B . n)^2)
    auto face = [&](const Vc &px, const Vc &py, const Vc &pz, const Vc &An) {
#pragma unroll
      for (int e = 0; e < N; ++e) {
        const R nx = px.v[e], ny = py.v[e], nz = pz.v[e];
        const R un = ux.v[e] * nx + uy.v[e] * ny + uz.v[e] * nz;
        const R Bn = Bx.v[e] * nx + By.v[e] * ny + Bz.v[e] * nz;
        const Divisor<R> by(rho.v[e], y.v[e]);
        const R vAn2 = by(c.inver_MA2 * (Bn * Bn));
        if (!(An.v[e] <= R(0.0))) den.v[e] += (fabs(un) + fast_cf(cs2.v[e], vA2.v[e], vAn2)) * An.v[e];
      }
    };
#pragma unroll 1
    for (int a = 0; a < 2; ++a) {
      face(B.staged(8 * a), B.staged(8 * a + 1), B.staged(8 * a + 2), B.staged(8 * a + 3));
      face(B.staged(8 * a + 4), B.staged(8 * a + 5), B.staged(8 * a + 6), B.staged(8 * a + 7));
    }
    const Vc zx = B.staged(16), zy = B.staged(17), zz = B.staged(18), zA = B.staged(19);
    face(zx, zy, zz, zA);
    face(B.fixed_upper(zx, cFNZ, o), B.fixed_upper(zy, cFNZ + 1, o), B.fixed_upper(zz, cFNZ + 2, o), B.fixed_upper(zA, cFNZ + 3, o));
#pragma unroll
    for (int e = 0; e < N; ++e)
      if (Vol.v[e] > R(0.0) && den.v[e] > R(0.0)) d.v[e] = dmin(d.v[e], c.CFL * Vol.v[e] / den.v[e]);
  }
  R dtl = R(1e100);
#pragma unroll
  for (int e = 0; e < N; ++e) {
    if (!own || it.k + e < 0 || it.k + e >= B.n2) continue;
    // a NaN drops out of the minimum: record it instead
    bad = bad || !isfinite(d.v[e]);
    dtl = dmin(dtl, d.v[e]);
  }
  return dtl;
}

// calc_divB (Z4_Mercury/src/physics/MercurySolver_MagneticCell.cpp:186-193) on the owned cells,
// and max |div B| per solve (atomicMax on the bits of the non-negative double).
template <class R>
__global__ void __launch_bounds__(kVecThreads) k_div_b(Dir D) {
  for_vec_items<R, kCells>(D, [&](const DevSolve &S, const VV<R> &B, const VItem &it) {
    double a = 0.0;
    {
      const uint32_t o = it.o;
      const Vec<R> bz = B.lv(cBZ, o);
      const Vec<R> v = (B.lv(cBX, o + B.di) - B.lv(cBX, o) + B.lv(cBY, o + B.dj) - B.lv(cBY, o) + B.upper(bz, cBZ, o) - bz) /
                       B.lm(cJAC, o);
      B.st(cDIVB, it, v, 0, B.n2);
#pragma unroll
      for (int e = 0; e < Vec<R>::N; ++e) {
        if (!it.in || !it.has(e)) continue;
        double x = fabs((double)v.v[e]);
        if (!(x == x)) x = __longlong_as_double(0x7ff0000000000000LL);  // NaN counts as infinite
        a = fmax(a, x);
      }
    }
    for (int w = 16; w > 0; w >>= 1) a = fmax(a, __shfl_xor_sync(0xffffffffu, a, w));
    if ((threadIdx.x & 31) == 0) atomicMax(&D.state[it.s].divb_bits, (unsigned long long)__double_as_longlong(a));
  });
}

// ------------------------------------------------------------------ implicit resistive substep
// SolveImplicitResistiveDiffusion_ (Z4_Mercury/src/implicit/Mercury_ImplicitResistive.cpp:475-575):
// (I + dt eta alpha C^T beta C) E = eta J(B*) on the owned edges with eta > 0.
// The operator is self-adjoint in the inner product weighted by
// W = 1 / (eta alpha), so CG runs in that inner product; the edge and J fields
// of the explicit step are the operator's scratch (E: E_res, J: dJ), dB has
// arrays of its own (RES_BSTAR), with the E and J sync and alias tables and
// Sync(dB)'s.

// Owned-range test of an edge of family a at (i, j, k).
__device__ __forceinline__ bool edge_owned(int a, int i, int j, int k, int n0, int n1, int n2) {
  return a == 0 ? (i < n0 && j <= n1 && k <= n2) : a == 1 ? (i <= n0 && j < n1 && k <= n2) : (i <= n0 && j <= n1 && k < n2);
}

// E = 1 on every edge of the owned range; the owner phase of Sync(E_res)
// run in mark mode then zeros its destinations, the non-owner aliases, so
// an edge still at 1 is its own unknown.
template <class R>
__global__ void __launch_bounds__(kVecThreads) k_res_seed(Dir D) {
  for_positions<R, kBox>(D, [&](const DevSolve &S, const auto &B, const Pos &it) {
    const int o = B.off(it.i, it.j, it.k);
    for (int a = 0; a < 3; ++a) B.c(cEX + a)[o] = R(1.0);
  });
}

// W = 1 / (eta alpha) on the unknowns (owned, not a non-owner alias, eta > 0,
// alpha > 0: BuildImplicitResistiveEdgeDofMap_, Mercury_ImplicitResistive.cpp:168-226), 0 elsewhere.
template <class R>
__global__ void __launch_bounds__(kVecThreads) k_res_w(Dir D) {
  for_positions<R, kBox>(D, [&](const DevSolve &S, const auto &B, const Pos &it) {
    const int o = B.off(it.i, it.j, it.k);
    for (int a = 0; a < 3; ++a) {
      R w = R(0.0);
      if (edge_owned(a, it.i, it.j, it.k, B.n0, B.n1, B.n2) && B.c(cEX + a)[o] != R(0.0)) {
        const R eta = B.c(cETAR + a)[o], alpha = B.c(cALX + a)[o];
        if (eta > R(0.0) && alpha > R(0.0)) w = R(1.0) / (eta * alpha);
      }
      B.c(cRW + a)[o] = w;
    }
  });
}

// Per block of the masked solve: the largest k of an edge with W > 0 (out
// starts at -1).  The substep's work range kResK ends two layers above it:
// the faces below the unknowns' top layer read E_res one layer up, the
// current on the unknowns reads those faces.
template <class R>
__global__ void __launch_bounds__(kVecThreads) k_res_kmax(Dir D, int *out) {
  for_vec_items<R, kBox>(D, [&](const DevSolve &S, const VV<R> &B, const VItem &it) {
    int k = -1;
    for (int e = 0; e < Vec<R>::N; ++e) {
      if (!it.in || !it.has(e)) continue;
      const int o = B.off(it.i, it.j, it.k + e);
      if (B.c(cRW)[o] > R(0.0) || B.c(cRW + 1)[o] > R(0.0) || B.c(cRW + 2)[o] > R(0.0)) k = it.k + e;
    }
    for (int of = 16; of > 0; of >>= 1) k = max(k, __shfl_xor_sync(0xffffffffu, k, of));
    if ((threadIdx.x & 31) == 0 && k >= 0) atomicMax(out + it.blk, k);
  });
}

// The solution of a CG loop: x with the last direction's step where the loop
// ended ahead of it (k_res_pupd_e updates x for a loop that goes on).
template <class R>
__device__ __forceinline__ R final_x(const ResCG &cg, R x, R p) {
  if (cg.it == 0) return R(0.0);
  if (!cg.pending) return x;
  const R step = R(cg.alpha) * p;
  return cg.it == 1 ? step : x + step;
}
// The direction p of the CG: E_res holds it on the unknowns; a solve whose
// Sync(Eres) may write those keeps it in RES_P as well (use_p).
__device__ __forceinline__ int dir_comp(int use_p) { return use_p ? cRP : cEX; }

// Vector operations of the CG on the unknowns (W > 0); other entries stay 0.
template <class R>
__global__ void __launch_bounds__(kVecThreads) k_res_vec(Dir D, int op, const ResCG *cg, int use_p) {
  for_vec_items<R, kResK>(D, [&](const DevSolve &S, const VV<R> &B, const VItem &it) {
    const uint32_t o = it.o;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const Vec<R> W = B.stat(cRW + a, o);
      auto put = [&](int comp, const Vec<R> &v) {  // v on the unknowns, 0 elsewhere
        B.st(comp + a, it, vmap<R>([&](int e) { return W.v[e] > R(0.0) ? v.v[e] : R(0.0); }), it.klo, it.khi);
      };
      switch (op) {
        case RES_INIT:  // r = b = eta J (PackImplicitJedgeToVec_, :395-418); the CG's start sets p
          put(cRR, R(0.0) + B.stat(cETAR + a, o) * B.lv(cJX + a, o));
          break;
        case RES_E_FROM_P: put(cEX, B.lv(cRP + a, o)); break;  // UnpackVecToImplicitEres_ (:294-312)
        case RES_E_FROM_X: put(cEX, B.lv(cRX + a, o)); break;
        case RES_E_FROM_CG: {  // the solution of the finished CG
          const Vec<R> p = B.lv(dir_comp(use_p) + a, o), x0 = B.lv(cRX + a, o);
          const Vec<R> x = vmap<R>([&](int e) { return final_x(cg[it.s], x0.v[e], p.v[e]); });
          put(cRX, x);
          put(cEX, x);
          break;
        }
        case RES_P_FROM_X: put(cRP, B.lv(cRX + a, o)); break;
        case RES_RESID:  // r = b - q, b kept in the face arrays (FP64 companion of a mixed solve)
          put(cRR, B.lv(cBX + a, o) - B.lv(cRQ + a, o));
          break;
        default: break;
      }
    }
  });
}

// dB = -dt curl E on the owned faces (CurlEdgeToFace with multiplier -dt,
// Z4_Mercury/src/operators/CTOperators.cpp:6-56; MatMultImplicitResistive_, :420-445).
// dB has arrays of its own (RES_BSTAR), so B keeps B* and nothing is saved or restored.
template <class R>
__global__ void __launch_bounds__(kVecThreads) k_res_db(Dir D) {
  for_vec_items<R, kResK>(D, [&](const DevSolve &S, const VV<R> &B, const VItem &it) {
    const R m = R(-D.state[it.s].dt);
    const uint32_t o = it.o, di = B.di, dj = B.dj;
    const bool ic = it.i < B.n0, jc = it.j < B.n1;
    const int hi = min(B.n2, it.khi);
    const Vec<R> ex = B.lv(cEX, o), ey = B.lv(cEY, o), ez = B.lv(cEZ, o);
    const Vec<R> bx = m * ((ey - B.upper(ey, cEY, o)) + (B.lv(cEZ, o + dj) - ez));
    const Vec<R> by = m * ((B.upper(ex, cEX, o) - ex) + (ez - B.lv(cEZ, o + di)));
    const Vec<R> bz = m * ((ex - B.lv(cEX, o + dj)) + (B.lv(cEY, o + di) - ey));
    B.st(cRBS, it, bx, 0, hi, jc);
    B.st(cRBS + 1, it, by, 0, hi, ic);
    B.st(cRBS + 2, it, bz, 0, it.khi, ic && jc);
  });
}

// alpha CurlAdjFaceToEdge(beta B) on this thread's edges (CTOperators.cpp:59-110):
// J of the field in the face arrays from component cb.
template <class R>
__device__ __forceinline__ void edge_current(const VV<R> &B, int cb, uint32_t o, Vec<R> J[3]) {
  const uint32_t di = B.di, dj = B.dj;
  constexpr uint32_t es = sizeof(R);
  auto on = [&](int a, uint32_t q) { return B.stat(cBFX + a, q) * B.lv(cb + a, q); };
  auto before = [&](int a) { return R(B.stat1(cBFX + a, o - es)) * B.ld(cb + a, o - es); };
  const Vec<R> fx = on(0, o), fy = on(1, o), fz = on(2, o);
  J[0] = ((vdown(fy, before(1)) - fy) + (fz - on(2, o - dj))) * R(1.0) * B.stat(cALX, o);
  J[1] = ((fx - vdown(fx, before(0))) + (on(2, o - di) - fz)) * R(1.0) * B.stat(cALY, o);
  J[2] = ((on(0, o - dj) - fx) + (fy - on(1, o - di))) * R(1.0) * B.stat(cALZ, o);
}

// dJ = alpha CurlAdjFaceToEdge(beta dB) on the owned edges (CalcImplicitDeltaJedgeFromDeltaB_,
// Mercury_ImplicitResistive.cpp:314-393; CTOperators.cpp:59-110), or J of B (ResField).
template <class R>
__global__ void __launch_bounds__(kVecThreads) k_res_dj(Dir D, int field) {
  for_vec_items<R, kResK>(D, [&](const DevSolve &S, const VV<R> &B, const VItem &it) {
    Vec<R> J[3];
    edge_current(B, field == RES_OF_B ? cBX : cRBS, it.o, J);
    B.st(cJX, it, J[0], 0, it.khi, it.i < B.n0);
    B.st(cJY, it, J[1], 0, it.khi, it.j < B.n1);
    B.st(cJZ, it, J[2], 0, min(B.n2, it.khi));
  });
}

// dB = 0 on every face of the block outside the owned range: the reference
// clears dB before the curl (clear_triplet, Mercury_ImplicitResistive.cpp:428),
// so Sync(dB) starts from zero ghosts; a Coupled-Solid boundary leaves them
// at zero and the halo copies of a rotated seam can read them.
template <class R>
__global__ void __launch_bounds__(kTileThreads) k_res_clearb(Dir D) {
  for_items<R, kFull>(D, [&](const DevSolve &S, const V<R> &B, const Item &it) {
    if (!it.in) return;
    const int i = it.i, j = it.j, k = it.k;
    const bool ci = i >= 0 && i < B.n0, cj = j >= 0 && j < B.n1, ck = k >= 0 && k < B.n2;
    const int o = B.off(i, j, k);
    if (!(i >= 0 && i <= B.n0 && cj && ck)) B.c(cRBS)[o] = R(0.0);
    if (!(ci && j >= 0 && j <= B.n1 && ck)) B.c(cRBS + 1)[o] = R(0.0);
    if (!(ci && cj && k >= 0 && k <= B.n2)) B.c(cRBS + 2)[o] = R(0.0);
  });
}

// q = A p = E_res - eta dJ on the unknowns (MatMultImplicitResistive_, :446-468).
template <class R>
__global__ void __launch_bounds__(kVecThreads) k_res_q(Dir D) {
  for_vec_items<R, kResK>(D, [&](const DevSolve &S, const VV<R> &B, const VItem &it) {
    const uint32_t o = it.o;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const Vec<R> W = B.stat(cRW + a, o), q = B.lv(cEX + a, o) - B.stat(cETAR + a, o) * B.lv(cJX + a, o);
      B.st(cRQ + a, it, vmap<R>([&](int e) { return W.v[e] > R(0.0) ? q.v[e] : R(0.0); }), it.klo, it.khi);
    }
  });
}

// The CTA's sums of two values, in thread 0 (fixed order).
__device__ __forceinline__ void cta_sum(double &a, double &b) {
  __shared__ double sh[2][kVecThreads / 32];
  for (int w = 16; w > 0; w >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, w);
    b += __shfl_xor_sync(0xffffffffu, b, w);
  }
  __syncthreads();  // sh of the previous sum has been read
  if ((threadIdx.x & 31) == 0) {
    sh[0][threadIdx.x >> 5] = a;
    sh[1][threadIdx.x >> 5] = b;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    a = b = 0.0;
    for (int w = 0; w < kVecThreads / 32; ++w) {
      a += sh[0][w];
      b += sh[1][w];
    }
  }
}

// Dot products of r on the unknowns of the masked solve: (sum W r r, sum r r).  Per-CTA partial sums in a fixed order (deterministic).
template <class R>
__global__ void __launch_bounds__(kVecThreads) k_res_dot(Dir D, double *partial) {
  double acc0 = 0.0, acc1 = 0.0;
  for_vec_items<R, kResK>(D, [&](const DevSolve &S, const VV<R> &B, const VItem &it) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const Vec<R> W = B.stat(cRW + a, it.o), r = B.lv(cRR + a, it.o);
#pragma unroll
      for (int e = 0; e < Vec<R>::N; ++e) {
        if (!it.in || !it.has(e) || !(W.v[e] > R(0.0))) continue;
        const double w = (double)W.v[e], x = (double)r.v[e];
        acc0 += w * x * x;
        acc1 += x * x;
      }
    }
  });
  cta_sum(acc0, acc1);
  if (threadIdx.x == 0) {
    partial[2 * blockIdx.x] = acc0;
    partial[2 * blockIdx.x + 1] = acc1;
  }
}
__global__ void k_res_sum(const double *partial, int n, double *result) {
  double s0 = 0.0, s1 = 0.0;
  for (int q = threadIdx.x; q < n; q += 32) {
    s0 += partial[2 * q];
    s1 += partial[2 * q + 1];
  }
  for (int w = 16; w > 0; w >>= 1) {
    s0 += __shfl_xor_sync(0xffffffffu, s0, w);
    s1 += __shfl_xor_sync(0xffffffffu, s1, w);
  }
  if (threadIdx.x == 0) {
    result[0] = s0;
    result[1] = s1;
  }
}

// The end of a k_res_cg step of solve s, by one thread, from its sums t0, t1:
// the solve's scalars, and whether its loop ends (converged, max_it,
// breakdown): it then leaves the mask, so the following kernels skip it.
__device__ __forceinline__ void res_cg_end(ResCG &cs, int op, double t0, double t1) {
  if (op == CG_INIT) {
    cs.rho = t0;
    cs.r0 = cs.rnorm = sqrt(t1);
    cs.tol = cs.tol_factor * cs.r0;
    cs.it = 0;
    cs.pending = 0;
    cs.converged = cs.rnorm <= cs.tol;
    cs.done = cs.converged || cs.max_it <= 0;
  } else if (op == CG_PQ) {
    if (!(t0 > 0.0)) cs.done = 1;  // breakdown: not positive definite on these unknowns
    else cs.alpha = cs.rho / t0;
  } else {
    cs.it += 1;
    cs.rnorm = sqrt(t1);
    if (cs.rnorm <= cs.tol) cs.converged = cs.done = 1;
    else if (cs.it >= cs.max_it) cs.done = 1;
    cs.pending = cs.done;  // x lacks alpha p: k_res_pupd_e adds it while the loop goes on
    cs.beta = t0 / cs.rho;
    cs.rho = t0;
  }
}

// One step of the CG iteration of every masked solve with its dot products.
// Each tile's sums go to its own slot of tpart (2 doubles); the CTA that
// finishes a solve's last tile (a ticket per solve) adds the solve's slots in a
// fixed order (deterministic, and the same for a solve alone or in a batch)
// and ends the step.  Warps without an unknown skip the vectors.  CG_PQ first
// clears the condition of the loop graph (build_cg_graph), and a solve that goes
// on sets it, so a loop whose stop test did not run ends; the condition is only
// written when launched inside the graph (in_graph; the host-driven loop of
// res_cg_batch reads the states instead).
template <class R, int OP>
__global__ void __launch_bounds__(kVecThreads) k_res_cg(Dir D, double *tpart, ResCG *cg, unsigned int *sarr,
                                                        cudaGraphConditionalHandle handle, int in_graph, int use_p) {
  if (in_graph && OP == CG_PQ && blockIdx.x == 0 && threadIdx.x == 0) cudaGraphSetConditional(handle, 0u);
  for_vec_items<R, kResK>(D, [&](const DevSolve &S, const VV<R> &B, const VItem &it) {
    constexpr int N = Vec<R>::N;
    const uint32_t o = it.o;
    double acc0 = 0.0, acc1 = 0.0;
    Vec<R> W[3];
    bool some = false;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      W[a] = B.stat(cRW + a, o);
#pragma unroll
      for (int e = 0; e < N; ++e) some = some || W[a].v[e] > R(0.0);
    }
    if (OP == CG_INIT || __any_sync(0xffffffffu, some && it.in)) {
      const R alpha = R(cg[it.s].alpha);
      auto mask = [&](int a, const Vec<R> &v) { return vmap<R>([&](int e) { return W[a].v[e] > R(0.0) ? v.v[e] : R(0.0); }); };
      auto counts = [&](int a, int e) { return it.in && it.has(e) && W[a].v[e] > R(0.0); };
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        if (OP == CG_INIT) {  // x = 0 (final_x), p = r (the start), E_res = p
          const Vec<R> r = B.lv(cRR + a, o), p = mask(a, r);
          if (use_p) B.st(cRP + a, it, p, it.klo, it.khi);
          B.st(cEX + a, it, p, it.klo, it.khi);
#pragma unroll
          for (int e = 0; e < N; ++e) {
            if (!counts(a, e)) continue;
            const double w = (double)W[a].v[e], rv = (double)r.v[e];
            acc0 += w * rv * rv;
            acc1 += rv * rv;
          }
        } else if (OP == CG_PQ) {
          const Vec<R> E = B.lv(cEX + a, o), q = mask(a, E - B.stat(cETAR + a, o) * B.lv(cJX + a, o));
          const Vec<R> p = use_p ? B.lv(cRP + a, o) : E;
          B.st(cRQ + a, it, q, it.klo, it.khi);
#pragma unroll
          for (int e = 0; e < N; ++e)
            if (counts(a, e)) acc0 += (double)W[a].v[e] * (double)p.v[e] * (double)q.v[e];
        } else {
          const Vec<R> r = B.lv(cRR + a, o), q = B.lv(cRQ + a, o);
          Vec<R> rn = r;
#pragma unroll
          for (int e = 0; e < N; ++e) {
            if (!(W[a].v[e] > R(0.0))) continue;
            rn.v[e] -= alpha * q.v[e];
            if (!counts(a, e)) continue;
            const double w = (double)W[a].v[e], rv = (double)rn.v[e];
            acc0 += w * rv * rv;
            acc1 += rv * rv;
          }
          B.st(cRR + a, it, rn, it.klo, it.khi);
        }
      }
    }
    __shared__ int last;
    cta_sum(acc0, acc1);
    const int *sp = D.solve_tile_prefix[kResK];
    const int t0 = sp[it.s], nt = sp[it.s + 1] - t0;
    if (threadIdx.x == 0) {
      tpart[2 * (int64_t)it.w] = acc0;
      tpart[2 * (int64_t)it.w + 1] = acc1;
      __threadfence();
      last = atomicAdd(&sarr[it.s], 1u) == (unsigned)nt - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();  // every tile of the solve is in
    double s0 = 0.0, s1 = 0.0;
    for (int q = threadIdx.x; q < nt; q += kVecThreads) {
      const double2 v = __ldcg((const double2 *)tpart + t0 + q);
      s0 += v.x;
      s1 += v.y;
    }
    cta_sum(s0, s1);
    if (threadIdx.x == 0) {
      sarr[it.s] = 0;
      res_cg_end(cg[it.s], OP, s0, s1);
      if (cg[it.s].done) D.state[it.s].mask = 0;
      else if (in_graph && OP != CG_PQ) cudaGraphSetConditional(handle, 1u);
    }
  });
}

// x += alpha p, then p = r + beta p and E_res = p (the next iteration's operator
// input) on the unknowns of every solve still iterating (in the mask): p is read
// once for both.  Warps without an unknown have nothing to update (their E_res
// is 0, or an owner copy that the next operator writes again).
template <class R>
__global__ void __launch_bounds__(kVecThreads) k_res_pupd_e(Dir D, const ResCG *cg, int use_p) {
  for_vec_items<R, kResK>(D, [&](const DevSolve &S, const VV<R> &B, const VItem &it) {
    constexpr int N = Vec<R>::N;
    const uint32_t o = it.o;
    Vec<R> W[3];
    bool some = false;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      W[a] = B.stat(cRW + a, o);
#pragma unroll
      for (int e = 0; e < N; ++e) some = some || W[a].v[e] > R(0.0);
    }
    if (!__any_sync(0xffffffffu, some && it.in)) return;
    const R alpha = R(cg[it.s].alpha), beta = R(cg[it.s].beta);
    const bool first = cg[it.s].it == 1;  // x = 0 until now
    Vec<R> x1[3], e1[3];  // stored behind every load
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const Vec<R> p = B.lv(dir_comp(use_p) + a, o), pn = B.lv(cRR + a, o) + beta * p, step = alpha * p;
      Vec<R> x = step;
      if (!first) x = B.lv(cRX + a, o) + step;
      x1[a] = vmap<R>([&](int e) { return W[a].v[e] > R(0.0) ? x.v[e] : R(0.0); });
      e1[a] = vmap<R>([&](int e) { return W[a].v[e] > R(0.0) ? pn.v[e] : R(0.0); });
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      B.st(cRX + a, it, x1[a], it.klo, it.khi);
      if (use_p) B.st(cRP + a, it, e1[a], it.klo, it.khi);
      B.st(cEX + a, it, e1[a], it.klo, it.khi);
    }
  });
}

// B into dB's arrays and back over the whole box (an explicit Sync(dB), which is
// asked of the face fluxes).
template <class R>
__global__ void __launch_bounds__(kTileThreads) k_res_copyb(Dir D, int op) {
  for_items<R, kFull>(D, [&](const DevSolve &S, const V<R> &B, const Item &it) {
    if (!it.in) return;
    const int o = B.off(it.i, it.j, it.k);
    for (int a = 0; a < 3; ++a) {
      if (op == RES_DB_FROM_B) B.c(cRBS + a)[o] = B.c(cBX + a)[o];
      else B.c(cBX + a)[o] = B.c(cRBS + a)[o];
    }
  });
}

// B += dt (-curl E_res) on the owned faces (ApplyImplicitResistiveUpdate_, :557-575;
// ApplyUpdate_Euler_BfaceOnly_, Z4_Mercury/src/physics/MercurySolver_MagExplicit_Hall.cpp:435-473).
template <class R>
__global__ void __launch_bounds__(kVecThreads) k_res_bupdate(Dir D) {
  for_vec_items<R, kResK>(D, [&](const DevSolve &S, const VV<R> &B, const VItem &it) {
    const R dt = R(D.state[it.s].dt);
    const uint32_t o = it.o, di = B.di, dj = B.dj;
    const bool ic = it.i < B.n0, jc = it.j < B.n1;
    // the faces whose edges E_res covers (k + 1 below the range's bound);
    // above them E_res is 0 and B does not change
    const int hi = it.khi - 1;
    const Vec<R> ex = B.lv(cEX, o), ey = B.lv(cEY, o), ez = B.lv(cEZ, o);
    const Vec<R> bx = B.lv(cBX, o) + dt * (R(-1.0) * ((ey - B.upper(ey, cEY, o)) + (B.lv(cEZ, o + dj) - ez)));
    const Vec<R> by = B.lv(cBY, o) + dt * (R(-1.0) * ((B.upper(ex, cEX, o) - ex) + (ez - B.lv(cEZ, o + di))));
    const Vec<R> bz = B.lv(cBZ, o) + dt * (R(-1.0) * ((ex - B.lv(cEX, o + dj)) + (B.lv(cEY, o + di) - ey)));
    B.st(cBX, it, bx, 0, hi, jc);
    B.st(cBY, it, by, 0, hi, ic);
    B.st(cBZ, it, bz, 0, it.khi, ic && jc);
  });
}

// Per-solve static terms, evaluated once at prepare with the reference's
// expressions: the face normals a / |a| and |a| of the area vectors JD that Compute_Timestep
// (Timestep.cpp:15-16,78-93) and calc_Jac_radius_GCL (FluidRHS.cpp:5-14) apply
// every step (owned faces and one more layer), the ambipolar gradient
// coefficients (owned cells), the contravariant-velocity coefficients (the
// cells k_pv_uplus refreshes), the Hall diffusion ratios (owned edges) and
// the fluid fluxes' face JD and 1 / Jac in the real type.
template <class R>
__global__ void __launch_bounds__(kVecThreads) k_face_normals(Dir D) {
  for_positions<R, kAlloc>(D, [&](const DevSolve &S, const auto &B, const Pos &it) {
    {
      // Coefficients of the contravariant velocities (calc_Uplus,
      // Tools.cpp:159-301) on the cells k_pv_uplus refreshes them on: the
      // face JD of each axis averaged to the cell, and 1 / (|Jac| + 1e-30).
      const int i = it.i, j = it.j, k = it.k;
      const int gm = min(consts_of<R>(S).nghost - 1, kStepGhost);
      if (i >= -gm && i < B.n0 + gm && j >= -gm && j < B.n1 + gm && k >= -gm && k < B.n2 + gm) {
#pragma unroll
        for (int axis = 0; axis < 3; ++axis) {
          int ip = i, jp = j, kp = k;
          shift1(axis, ip, jp, kp, 1);
          const int cm = axis == 0 ? cJDX : axis == 1 ? cJDY : cJDZ;
#pragma unroll
          for (int q = 0; q < 3; ++q)
            AT(cUCK + 3 * axis + q, i, j, k) = R(0.5) * (R(ATM(cm + q, i, j, k)) + R(ATM(cm + q, ip, jp, kp)));
        }
        AT(cUCK + 9, i, j, k) = R(1.0) / (fabs(R(ATM(cJAC, i, j, k))) + R(1.0e-30));
      }
    }
    if (it.i < 0 || it.j < 0 || it.k < 0 || it.i > B.n0 || it.j > B.n1 || it.k > B.n2) return;  // [0, n + 1) below
    {
      // the face JD the fluid fluxes read and the cell's 1 / Jac, converted
      // to the real type once (the values the fluid kernel would form)
      const int i = it.i, j = it.j, k = it.k;
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        AT(cFM + q, i, j, k) = R(ATM(cJDX + q, i, j, k));
        AT(cFM + 3 + q, i, j, k) = R(ATM(cJDY + q, i, j, k));
        AT(cFM + 6 + q, i, j, k) = R(ATM(cJDZ + q, i, j, k));
      }
      AT(cFM + 9, i, j, k) = R(1.0) / R(ATM(cJAC, i, j, k));
    }
    {
      // Hall diffusion ratios of the owned edges (BuildHallFaceEMF_Rusanov_diff_
      // step 3, Hall.cpp:148-400): edge length over the face area averaged
      // to the edge, both floored at 1e-14, per transverse direction.
      const int i = it.i, j = it.j, k = it.k;
      const R eps = R(1e-14);
      if (i < B.n0) {
        const R L = dmax(AT(cDLX, i, j, k), eps);
        const R Abz = R(0.5) * (AT(cAZ, i, j, k) + AT(cAZ, i, j - 1, k));
        const R Abe = R(0.5) * (AT(cAY, i, j, k) + AT(cAY, i, j, k - 1));
        AT(cIHX, i, j, k) = L / dmax(Abz, eps);
        AT(cIHX + 1, i, j, k) = L / dmax(Abe, eps);
      }
      if (j < B.n1) {
        const R L = dmax(AT(cDLY, i, j, k), eps);
        const R Abx = R(0.5) * (AT(cAX, i, j, k) + AT(cAX, i, j, k - 1));
        const R Abz = R(0.5) * (AT(cAZ, i, j, k) + AT(cAZ, i - 1, j, k));
        AT(cIHY, i, j, k) = L / dmax(Abx, eps);
        AT(cIHY + 1, i, j, k) = L / dmax(Abz, eps);
      }
      if (k < B.n2) {
        const R L = dmax(AT(cDLZ, i, j, k), eps);
        const R Abe = R(0.5) * (AT(cAY, i, j, k) + AT(cAY, i - 1, j, k));
        const R Abx = R(0.5) * (AT(cAX, i, j, k) + AT(cAX, i, j - 1, k));
        AT(cIHZ, i, j, k) = L / dmax(Abe, eps);
        AT(cIHZ + 1, i, j, k) = L / dmax(Abx, eps);
      }
    }
    {
      // Ambipolar pressure-gradient coefficients of an owned cell
      // (AddSourceToRHS_Fluid, FluidRHS.cpp:206-527): face JD averaged to the
      // cell and divided by |Jac| (zero where |Jac| is not positive).
      const int i = it.i, j = it.j, k = it.k;
      if (consts_of<R>(S).ambipolar && i < B.n0 && j < B.n1 && k < B.n2) {
        const R Vol = fabs(R(ATM(cJAC, i, j, k)));
        R a[9] = {R(0.0), R(0.0), R(0.0), R(0.0), R(0.0), R(0.0), R(0.0), R(0.0), R(0.0)};
        if (Vol > R(0.0)) {
          a[0] = R(0.5) * (R(ATM(cJDX, i - 1, j, k)) + R(ATM(cJDX, i, j, k))) / Vol;
          a[1] = R(0.5) * (R(ATM(cJDX + 1, i - 1, j, k)) + R(ATM(cJDX + 1, i, j, k))) / Vol;
          a[2] = R(0.5) * (R(ATM(cJDX + 2, i - 1, j, k)) + R(ATM(cJDX + 2, i, j, k))) / Vol;
          a[3] = R(0.5) * (R(ATM(cJDY, i, j - 1, k)) + R(ATM(cJDY, i, j, k))) / Vol;
          a[4] = R(0.5) * (R(ATM(cJDY + 1, i, j - 1, k)) + R(ATM(cJDY + 1, i, j, k))) / Vol;
          a[5] = R(0.5) * (R(ATM(cJDY + 2, i, j - 1, k)) + R(ATM(cJDY + 2, i, j, k))) / Vol;
          a[6] = R(0.5) * (R(ATM(cJDZ, i, j, k - 1)) + R(ATM(cJDZ, i, j, k))) / Vol;
          a[7] = R(0.5) * (R(ATM(cJDZ + 1, i, j, k - 1)) + R(ATM(cJDZ + 1, i, j, k))) / Vol;
          a[8] = R(0.5) * (R(ATM(cJDZ + 2, i, j, k - 1)) + R(ATM(cJDZ + 2, i, j, k))) / Vol;
        }
#pragma unroll
        for (int q = 0; q < 9; ++q) AT(cAMB + q, i, j, k) = a[q];
      }
    }
#pragma unroll 1
    for (int a = 0; a < 3; ++a) {
      const int cm = a == 0 ? cJDX : a == 1 ? cJDY : cJDZ;
      const int cn = a == 0 ? cFNX : a == 1 ? cFNY : cFNZ;
      const int o = B.off(it.i, it.j, it.k);
      const double ax = B.m(cm)[o], ay = B.m(cm + 1)[o], az = B.m(cm + 2)[o];
      const double An = sqrt(ax * ax + ay * ay + az * az);
      B.c(cn)[o] = R(ax / An);
      B.c(cn + 1)[o] = R(ay / An);
      B.c(cn + 2)[o] = R(az / An);
      B.c(cn + 3)[o] = R(An);
    }
  });
}

// A cell's terms of the Rusanov flux (FluidCell) from its density as it stands in
// U, |u|^2 and the pressure.
template <class R>
__device__ __forceinline__ void flux_terms(const ConstsT<R> &c, R rho, R u2, R p, R &re, R &cs) {
  if constexpr (sizeof(R) == 4) re = p * c.inv_g1 + R(0.5) * rho * u2;
  else re = p / (c.gamma - R(1.0)) + R(0.5) * rho * u2;
  cs = sqrt(dmax(R(0.0), c.gamma * p / dmax(rho, R(1e-30))));
}

// The flux terms again after an explicit Sync(U) between steps: it may give ghosts
// on rotated seams other densities than the step's sync left there, and the
// next step's fluxes take these with the primitive variables as they are.
template <class R>
__global__ void __launch_bounds__(kVecThreads) k_flux_terms(Dir D) {
  for_vec_items<R, kAlloc>(D, [&](const DevSolve &S, const auto &B, const VItem &it) {
    constexpr int N = group_size(kAlloc, sizeof(R));
    const ConstsT<R> &c = consts_of<R>(S);
    const uint32_t o = it.o;
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const int pv0 = s ? cPVN : cPVH;
      const auto rho = B.lv(s ? cUN : cUH, o), u = B.lv(pv0, o), v = B.lv(pv0 + 1, o), w = B.lv(pv0 + 2, o), p = B.lv(pv0 + 3, o);
      Vec<R, N> re, cs;
#pragma unroll
      for (int e = 0; e < N; ++e)
        flux_terms(c, rho.v[e], u.v[e] * u.v[e] + v.v[e] * v.v[e] + w.v[e] * w.v[e], p.v[e], re.v[e], cs.v[e]);
      B.st(cFT + 2 * s, it, re, it.klo, it.khi);
      B.st(cFT + 2 * s + 1, it, cs, it.klo, it.khi);
    }
  });
}

// calc_PV + calc_Uplus (Z4_Mercury/src/physics/MercurySolver_Tools.cpp:159-301) on the allocated
// cell range the step keeps, the fluid fluxes' cell terms, the contravariant
// velocities UCON and the next step's Hall cell field there, and the next
// step's CFL dt on owned cells (warp min, one atomicMin per warp on the bit
// pattern of the positive double).  The step's last pass ends it (retire_solve).
// Bound by latency: a cell is a chain of divisions and square roots behind some
// 50 operands.  So 8-byte groups (twice the threads of 16-byte ones), and the 30
// static operands on their way before the wait (kPvCtas x the stage fits an SM):
// a step takes 55 us for a box of 8^3 FP64 cells (62 with 16-byte groups and
// plain loads), 85 (93) for 32^3, 153 (163) for 64^3 mixed.
template <class R>
__global__ void __launch_bounds__(kVecThreads, kPvCtas) k_pv_uplus(Dir D, int end_of_step) {
  for_vec_items<R, kAlloc>(D, [&](const DevSolve &S, const auto &B, const VItem &it) {
    constexpr int N = group_size(kAlloc, sizeof(R));
    using Vc = Vec<R, N>;
    const ConstsT<R> &c = consts_of<R>(S);
    R dtl = R(1e100);
    bool bad = false;
    {
      const uint32_t o = it.o;
      auto put = [&](int comp, const Vc &v) { B.st(comp, it, v, it.klo, it.khi); };
      // every field ahead of the first store
      Vc U[2][5];
#pragma unroll
      for (int s = 0; s < 2; ++s)
#pragma unroll
        for (int m = 0; m < 5; ++m) U[s][m] = B.lv((s ? cUN : cUH) + m, o);
      const Vc Bx = B.lv(cBC, o), By = B.lv(cBC + 1, o), Bz = B.lv(cBC + 2, o);
      const Vc Jx = B.lv(cJC, o), Jy = B.lv(cJC + 1, o), Jz = B.lv(cJC + 2, o);
      Vc rho[2], vel[2][3];
      Vc chk = vset<R, N>(R(0.0));  // sum of the conserved components: non-finite if any of them is
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int pv0 = s ? cPVN : cPVH;
        const R coeff = s ? c.state_coeff_Na : c.state_coeff_H;
        const Vc r0 = U[s][0], m1 = U[s][1], m2 = U[s][2], m3 = U[s][3], E = U[s][4];
        rho[s] = r0;
        chk = chk + (((r0 + m1) + (m2 + m3)) + E);
        Vc pr, T, re, cs;
#pragma unroll
        for (int e = 0; e < N; ++e) {
          const R rh = dmax(r0.v[e], R(1e-12));
          const Divisor<R> by(rh);
          const R u = by(m1.v[e]), v = by(m2.v[e]), w = by(m3.v[e]);
          const R u2 = u * u + v * v + w * w;
          const R ke = R(0.5) * rh * u2;
          R eint = E.v[e] - ke;
          if (eint < R(0.0)) eint = R(0.0);
          const R p = dmax((c.gamma - R(1.0)) * eint, R(1e-12));
          pr.v[e] = p;
          if constexpr (sizeof(R) == 4) T.v[e] = by(p) * c.inv_coeff[s];
          else T.v[e] = p / (rh * coeff);
          flux_terms(c, r0.v[e], u2, p, re.v[e], cs.v[e]);
          vel[s][0].v[e] = u;
          vel[s][1].v[e] = v;
          vel[s][2].v[e] = w;
        }
        put(pv0, vel[s][0]);
        put(pv0 + 1, vel[s][1]);
        put(pv0 + 2, vel[s][2]);
        put(pv0 + 3, pr);
        put(pv0 + 4, T);
        put(cFT + 2 * s, re);
        put(cFT + 2 * s + 1, cs);
      }
      Vc alpha, up[3];
#pragma unroll
      for (int e = 0; e < N; ++e) {
        const R rH = dmax(rho[0].v[e], R(0.0)), rN = dmax(rho[1].v[e], R(0.0));
        const Num<R> d = num_limiter(c, rH, rN);
        alpha.v[e] = c.hall_coef / d.ne_eff;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          const R uH = rH > R(1e-20) ? vel[0][q].v[e] : R(0.0);
          const R uN = rN > R(1e-20) ? vel[1][q].v[e] : R(0.0);
          up[q].v[e] = d.chiH * uH + d.chiNa * uN;
        }
      }
      {
        // the next step's Hall cell field, BuildHallFaceEMF_Rusanov_diff_ step 1
        // (Z4_Mercury/src/physics/MercurySolver_MagExplicit_Hall.cpp:110-146): its inputs (J_cell,
        // B_cell, the densities) are final here (num_limiter clamps the
        // densities at zero itself, so it is the limiter of the raw densities)
        put(cEHC, alpha * (Jy * Bz - Jz * By));
        put(cEHC + 1, alpha * (Jz * Bx - Jx * Bz));
        put(cEHC + 2, alpha * (Jx * By - Jy * Bx));
        put(cHB, vabs(alpha) * vsqrt(Bx * Bx + By * By + Bz * Bz));
      }
#pragma unroll
      for (int q = 0; q < 3; ++q) put(cUP + q, up[q]);
      const int gm = min(c.nghost - 1, kStepGhost);
      const bool near = it.i >= -gm && it.i < B.n0 + gm && it.j >= -gm && it.j < B.n1 + gm;
      {
        // coefficients (cell-averaged JD, 1 / (|Jac| + 1e-30)) from k_face_normals
        staged_arrived();
        const Vc inv_jac = B.staged(29);
#pragma unroll
        for (int axis = 0; axis < 3; ++axis)
          B.st(cUC + axis, it,
               (B.staged(20 + 3 * axis) * up[0] + B.staged(21 + 3 * axis) * up[1] +
                B.staged(22 + 3 * axis) * up[2]) *
                   inv_jac,
               max(it.klo, -gm), min(it.khi, B.n2 + gm), near);
      }
      const bool own = it.in && it.i >= 0 && it.i < B.n0 && it.j >= 0 && it.j < B.n1;
      if (__any_sync(0xffffffffu, own)) {
        dtl = cells_dt<R, N>(B, c, it, own, Bx, By, Bz, bad);
        // the pressure floors can hide a non-finite energy from the dt
#pragma unroll
        for (int e = 0; e < N; ++e) bad = bad || (own && it.k + e >= 0 && it.k + e < B.n2 && !isfinite(chk.v[e]));
      }
    }
    // warp minimum, one atomicMin per warp (min is exact in any order)
    for (int w = 16; w > 0; w >>= 1) dtl = dmin(dtl, __shfl_xor_sync(0xffffffffu, dtl, w));
    if ((threadIdx.x & 31) == 0 && dtl < R(1e100))
      atomicMin(&D.state[it.s].dt_bits, (unsigned long long)__double_as_longlong(dtl));
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicExch(&D.state[it.s].nonfinite, 1);
  }, [&](const auto &B, const VItem &it) {
    const uint32_t w = stage_base(group_size(kAlloc, sizeof(R)) * (int)sizeof(R)), o = it.o;
#pragma unroll
    for (int q = 0; q < 4; ++q) {  // the faces' normals and |a|: xi-, xi+, eta-, eta+, zeta-
      B.stage(w, q, cFNX + q, o);
      B.stage(w, 4 + q, cFNX + q, o + B.di);
      B.stage(w, 8 + q, cFNY + q, o);
      B.stage(w, 12 + q, cFNY + q, o + B.dj);
      B.stage(w, 16 + q, cFNZ + q, o);
    }
#pragma unroll
    for (int q = 0; q < 10; ++q) B.stage(w, 20 + q, cUCK + q, o);
  });
  if (end_of_step) after_all_tiles<kAlloc>(D, D.tickets + 1, [](SolveState &st) { retire_solve(st); });
}

#undef AT
#undef ATM

// ------------------------------------------------------------------ sync, alias, bookkeeping
__device__ __forceinline__ int find_solve(const int *prefix, int nsolves, int e) {
  int lo = 0, hi = nsolves;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (prefix[mid] <= e) lo = mid; else hi = mid;
  }
  return lo;
}
template <class R>
__device__ __forceinline__ R *at_code(const DevSolve &S, int cur, int64_t code) {
  return (R *)(S.arena + (code & kCodeOffMask) + ((code & kCodeUFlag) ? (int64_t)cur * S.ubuf : int64_t(0)));
}
__device__ __forceinline__ const int *op_prefix(const Dir &D, const SyncOp &op) {
  if (op.kind == SYNC_COPY) return D.copy_prefix[op.arg][op.phase];
  return op.arg ? D.aliasJ_prefix : D.aliasE_prefix;
}

// MercuryBoundary::Sync_ stages (Z4_Mercury/src/boundary/Boundary_Sync_.cpp:4-110) and
// ReduceEdgeAliasCandidatesToOwners_ (Z4_Mercury/src/physics/MercurySolver_Current.cpp:3-57)
// for every active solve, up to kMaxSyncOps independent operations per launch.
// Work unit: a group of 8 lanes.  A copy phase gives each group one segment
// (dst <- sign * src on up to kSegElems elements: reps strided runs of len
// consecutive elements); an alias reduction gives each lane one class, whose
// members are summed in stored order from 0.0 and written to the owner as
// owner_sign * sum / count.
template <class R, int N>  // N: the most operations of the launch
__global__ void __launch_bounds__(256) k_sync(Dir D, SyncOps ops) {
  const int lane = threadIdx.x & 7;
  const int stride = (gridDim.x * blockDim.x) >> 3;
  let_dependents_launch();
  // the operations' work units follow one another
  int end[N], total = 0;
#pragma unroll
  for (int p = 0; p < N; ++p) {
    if (N <= 2 || p < ops.n) total += op_prefix(D, ops.op[p])[D.nsolves];
    end[p] = total;
  }
  bool first = true;
  if (((int)(blockIdx.x * blockDim.x) >> 3) >= total) {
    if (blockIdx.x == 0) wait_for_predecessors();
    return;
  }
  for (int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 3; g < total; g += stride) {
    SyncOp op = ops.op[0];
    int e = g;
#pragma unroll
    for (int p = 1; p < N; ++p)
      if (g >= end[p - 1]) {
        op = ops.op[p];
        e = g - end[p - 1];
      }
    const int *pre = op_prefix(D, op);
    const int s = find_solve(pre, D.nsolves, e);
    const DevSolve &S = D.solves[s];
    const int q = e - pre[s];
    const bool copy = op.kind == SYNC_COPY;
    const DevAlias &A = op.arg ? S.aliasJ : S.aliasE;
    // the tables are as static as the directory
    int64_t dcode = 0, scode = 0, rw = 0;
    if (copy) {
      const int64_t *w = S.tab[op.arg][op.phase].seg + kSegWords * (int64_t)q;
      dcode = w[0];
      scode = w[1];
      rw = w[2];
    }
    // a class's first members (most have two or four)
    constexpr int kAhead = 4;
    int m0 = 0, m1 = 0;
    int64_t mcode[kAhead], ocode = 0;
    double msign[kAhead], osign = 0.0;
    const int cls = q * 8 + lane;
    const bool alias = !copy && cls < A.n;
    if (alias) {
      m0 = A.offset[cls];
      m1 = A.offset[cls + 1];
      ocode = A.owner[cls];
      osign = A.osign[cls];
#pragma unroll
      for (int m = 0; m < kAhead; ++m) {
        const bool has = m0 + m < m1;
        mcode[m] = has ? A.member[m0 + m] : ocode;
        msign[m] = has ? A.msign[m0 + m] : 0.0;
      }
    }
    Status st{};
    if (D.mode == 0) st = status_of(D, s);
    if (first) wait_for_predecessors();
    first = false;
    if (D.mode != 0) st = status_of(D, s);
    if (!st.active) continue;
    const int cur = st.cur;
    if (copy) {
      const int len = (int)((dcode >> kSegLenShift) & 31) + 1;
      const int n = len * ((int)(rw & 0xffff) + 1);
      const int64_t stride = rw >> kSegStrideShift;  // bytes between runs
      const bool neg = (dcode >> kSegNegBit) & 1;
      const char *src = (const char *)at_code<R>(S, cur ^ op.prev, scode);
      char *dst = (char *)at_code<R>(S, cur, dcode);
      // element e of the segment: run e / len, offset e % len (e < 64, so
      // e * ceil(2^16 / len) >> 16 is the exact quotient)
      const int inv = (65536 + len - 1) / len;
      R v[kSegElems / 8];
      int64_t off[kSegElems / 8];
#pragma unroll
      for (int u = 0; u < kSegElems / 8; ++u) {
        const int e = lane + 8 * u;
        const int r = (e * inv) >> 16;
        off[u] = r * stride + (int64_t)(e - r * len) * (int64_t)sizeof(R);
        if (e < n) v[u] = *(const R *)(src + off[u]);
      }
#pragma unroll
      for (int u = 0; u < kSegElems / 8; ++u)
        if (lane + 8 * u < n) *(R *)(dst + off[u]) = op.mark ? R(0.0) : (neg ? -v[u] : v[u]);
    } else if (alias) {
      R v[kAhead];
#pragma unroll
      for (int m = 0; m < kAhead; ++m) v[m] = *at_code<R>(S, cur, mcode[m]);
      R sum = R(0.0);
#pragma unroll
      for (int m = 0; m < kAhead; ++m)
        if (m0 + m < m1) sum += R(msign[m]) * v[m];
      for (int m = m0 + kAhead; m < m1; ++m) sum += R(A.msign[m]) * *at_code<R>(S, cur, A.member[m]);
      const R mean = R(osign) * sum / (R)(m1 - m0);
      *at_code<R>(S, cur, ocode) = mean;
      if (op.mark) {
#pragma unroll
        for (int m = 0; m < kAhead; ++m)
          if (m0 + m < m1) *at_code<R>(S, cur, mcode[m]) = msign[m] == osign ? mean : -mean;
        for (int m = m0 + kAhead; m < m1; ++m)
          *at_code<R>(S, cur, A.member[m]) = A.msign[m] == osign ? mean : -mean;
      }
    }
  }
}

#define AT(cc, i, j, k) (B.c(cc)[B.off((i), (j), (k))])
#define ATM(cc, i, j, k) (B.m(cc)[B.off((i), (j), (k))])

// A block's view outside the tile loop (the singular-edge passes).
template <class R>
__device__ __forceinline__ V<R> block_view(const Dir &D, int s, int b) {
  const DevBlock &DB = D.solves[s].blocks[b];
  V<R> B;
  const int cur = D.state[s].cur;
  set_view(B, DB, cur);
  return B;
}

// Physical boundary operations of table `which` (a sync group, or the wall
// EMF) for every active solve (mhd_phys_op; BoundaryCore::ApplyPhysical with
// MercuryBoundary's handlers, Z4_Mercury/src/boundary/Boundary_Build.cpp:5-300).
// The operations of one table write distinct DOFs and read none another
// writes, so they run in any order.
// Up to two tables per launch (t1 < 0: one).  A group of 8 lanes takes a
// constant segment (up to 32 elements) or one other operation (one per lane, eight
// chains of scattered stores in a warp's way: a step of the shell of 8 x 8 x 12
// cells 75 us instead of 68).
template <class R>
__global__ void __launch_bounds__(256) k_phys(Dir D, int t0, int t1) {
  let_dependents_launch();
  const int *pre0 = D.phys_prefix[t0], *pre1 = t1 >= 0 ? D.phys_prefix[t1] : nullptr;
  const int n0 = pre0[D.nsolves], total = n0 + (pre1 ? pre1[D.nsolves] : 0);
  if (((int)(blockIdx.x * blockDim.x) >> 3) >= total) {
    if (blockIdx.x == 0) wait_for_predecessors();
    return;
  }
  const int lane = threadIdx.x & 7;
  const int stride = (gridDim.x * blockDim.x) >> 3;
  bool first = true;
  for (int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 3; g < total; g += stride) {
    const bool second = g >= n0;
    const int *pre = second ? pre1 : pre0;
    const int e = second ? g - n0 : g;
    const int s = find_solve(pre, D.nsolves, e);
    const DevSolve &S = D.solves[s];
    const ConstsT<R> &c = consts_of<R>(S);
    const DevPhys &P = S.phys[second ? t1 : t0];
    const int q = e - pre[s];
    const bool set = q < P.nset;  // destinations <- bc[arg]: nr runs of len elements, step bytes apart
    int64_t w0 = 0, w1 = 0;
    R v = R(0.0);
    if (set) {
      w0 = P.set[2 * q];
      w1 = P.set[2 * q + 1];
      v = c.bc[(int)((w0 >> kPhysArgShift) & 31)];
    }
    Status st{};
    if (D.mode == 0) st = status_of(D, s);
    if (first) wait_for_predecessors();
    first = false;
    if (D.mode != 0) st = status_of(D, s);
    if (!st.active) continue;
    const int cur = st.cur;
    if (set) {
      char *p0 = (char *)at_code<R>(S, cur, w0 & ~(int64_t(31) << kPhysArgShift));
      const int len = (int)(w1 & 255) + 1, nr = (int)((w1 >> 8) & 255) + 1;
      const int64_t step = w1 >> 16;
      for (int u = lane; u < len * nr; u += 8) {
        const int r = u / len;
        *(R *)(p0 + r * step + (int64_t)(u - r * len) * (int64_t)sizeof(R)) = v;
      }
      continue;
    }
    if (lane != 0) continue;
    const DevPhysOp &op = P.op[q - P.nset];
    if (op.kind == MHD_PHYS_WALL) {
      // BC_Solid_Surface_ (Z4_Mercury/src/boundary/Boundary_Condition_Fluid.cpp:37-259), H+:
      // the boundary cell from the cell one deeper (density floor 2.5e-3,
      // no-slip, pressure from the conserved state with its floors), then
      // the ghost cells from the boundary cell's new state
      const R floor = R(2.5e-3), g1 = c.gamma - R(1.0);
      auto wall = [&](const R *U, R *out) {
        const R rho_r = dmax(U[0], floor);
        const R rho = dmax(rho_r, floor);
        const R ke = R(0.5) * (U[1] * U[1] + U[2] * U[2] + U[3] * U[3]) / rho;
        R eint = U[4] - ke;
        if (eint < R(0.0)) eint = R(0.0);
        const R p = dmax(g1 * eint, R(1.0e-12));
        out[0] = rho_r;
        out[1] = out[2] = out[3] = rho_r * R(0.0);
        out[4] = p / g1 + R(0.5) * rho_r * R(0.0);
      };
      R u[5], w1[5], w2[5];
      for (int m = 0; m < 5; ++m) u[m] = *at_code<R>(S, cur, op.src + m * op.cstride);
      wall(u, w1);
      wall(w1, w2);
      for (int m = 0; m < 5; ++m) *at_code<R>(S, cur, op.dst + m * op.cstride) = w1[m];
      for (int g = 0; g < op.nghost; ++g)
        for (int m = 0; m < 5; ++m) *at_code<R>(S, cur, op.ghost[g] + m * op.cstride) = w2[m];
    } else {
      // BC_Farfield_Eedge_set_zerocurl (Z4_Mercury/src/boundary/Boundary_Condition.cpp:573-624):
      // E = E_inf . dr with E_inf = -u_inf x B_imf
      const R *u = c.bc + MHD_BC_UINF, *Bi = c.bc + MHD_BC_BIMF;
      const R E0 = Bi[1] * u[2] - Bi[2] * u[1], E1 = Bi[2] * u[0] - Bi[0] * u[2], E2 = Bi[0] * u[1] - Bi[1] * u[0];
      const R d0 = *at_code<R>(S, cur, op.src), d1 = *at_code<R>(S, cur, op.src + op.cstride),
              d2 = *at_code<R>(S, cur, op.src + 2 * op.cstride);
      *at_code<R>(S, cur, op.dst) = E0 * d0 + E1 * d1 + E2 * d2;
    }
  }
}

// One thread per singular edge of every active solve.
template <class F>
__device__ __forceinline__ void for_singular(const Dir &D, F &&f) {
  let_dependents_launch();
  const int total = D.sing_prefix[D.nsolves];
  wait_for_predecessors();
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < total; e += gridDim.x * blockDim.x) {
    const int s = find_solve(D.sing_prefix, D.nsolves, e);
    if (!solve_active(D, s)) continue;
    f(s, D.solves[s].sing, e - D.sing_prefix[s]);
  }
}

// The geometric data of the singular edges (SingularEdgeRegistry::build,
// src/7_metric/SingularEdgeRegistry.cpp:78-300) from the uploaded geometry,
// in the reference's operation order: the mean primal length and the
// canonical edge vector over the aliases, the |Jac| weights of the incident
// cells, the dual polygon through their centres (sorted by angle about the
// edge) and its area, the inverse Hodge star, which also replaces the edge
// Hodge field of every alias.  Computed in FP64 from the double metric and
// the real-typed edge fields.
template <class R>
__global__ void k_sing_setup(Dir D) {
  for_singular(D, [&](int s, const DevSingular &G, int e) {
    double len = 0.0, dr[3] = {0.0, 0.0, 0.0};
    int nlen = 0;
    for (int a = G.aoff[e]; a < G.aoff[e + 1]; ++a) {
      const int *r = G.alias + 6 * a;
      const V<R> B = block_view<R>(D, s, r[0]);
      const int ax = r[1];
      const double L = (double)AT(cDLX + ax, r[2], r[3], r[4]);
      if (isfinite(L) && L > 0.0) {
        len += L;
        ++nlen;
      }
      for (int q = 0; q < 3; ++q) dr[q] += r[5] * (double)AT((ax == 0 ? cDRX : ax == 1 ? cDRY : cDRZ) + q, r[2], r[3], r[4]);
    }
    double gv = 0.0;
    constexpr int kMaxCells = 16;
    double pts[kMaxCells][3];
    int np = 0;
    for (int q = G.coff[e]; q < G.coff[e + 1]; ++q) {
      const int *r = G.cell + 6 * q;
      const V<R> B = block_view<R>(D, s, r[0]);
      const double v = fabs(ATM(cJAC, r[2], r[3], r[4]));
      if (isfinite(v) && v > 1.e-30) {
        gv += v;
        if (np < kMaxCells) {
          for (int c = 0; c < 3; ++c) pts[np][c] = (double)AT(cCX + c, r[2], r[3], r[4]);
          ++np;
        }
      }
    }
    for (int q = G.coff[e]; q < G.coff[e + 1]; ++q) {
      const int *r = G.cell + 6 * q;
      const V<R> B = block_view<R>(D, s, r[0]);
      const double v = fabs(ATM(cJAC, r[2], r[3], r[4]));
      G.w[q] = (isfinite(v) && v > 1.e-30 && gv > 0.0) ? v / gv : 0.0;
    }
    const double primal = nlen ? len / nlen : 0.0;
    double dual = 0.0;
    if (np >= 3) {
      double cen[3] = {0.0, 0.0, 0.0};
      for (int n = 0; n < np; ++n)
        for (int c = 0; c < 3; ++c) cen[c] += pts[n][c];
      for (int c = 0; c < 3; ++c) cen[c] /= np;
      double t[3] = {dr[0], dr[1], dr[2]};
      const double tn = sqrt(t[0] * t[0] + t[1] * t[1] + t[2] * t[2]);
      if (tn > 0.0)
        for (double &x : t) x /= tn;
      const double ref[3] = {fabs(t[0]) < 0.9 ? 1.0 : 0.0, fabs(t[0]) < 0.9 ? 0.0 : 1.0, 0.0};
      double u[3] = {t[1] * ref[2] - t[2] * ref[1], t[2] * ref[0] - t[0] * ref[2], t[0] * ref[1] - t[1] * ref[0]};
      const double un = sqrt(u[0] * u[0] + u[1] * u[1] + u[2] * u[2]);
      if (un > 0.0)
        for (double &x : u) x /= un;
      const double v[3] = {t[1] * u[2] - t[2] * u[1], t[2] * u[0] - t[0] * u[2], t[0] * u[1] - t[1] * u[0]};
      double ang[kMaxCells];
      for (int n = 0; n < np; ++n) {
        double du = 0.0, dv = 0.0;
        for (int c = 0; c < 3; ++c) {
          du += (pts[n][c] - cen[c]) * u[c];
          dv += (pts[n][c] - cen[c]) * v[c];
        }
        ang[n] = atan2(dv, du);
      }
      int ord[kMaxCells];
      for (int n = 0; n < np; ++n) ord[n] = n;
      for (int n = 1; n < np; ++n)  // insertion sort by angle (the points are few and their angles distinct)
        for (int m = n; m > 0 && ang[ord[m]] < ang[ord[m - 1]]; --m) {
          const int tmp = ord[m];
          ord[m] = ord[m - 1];
          ord[m - 1] = tmp;
        }
      double av[3] = {0.0, 0.0, 0.0};
      for (int n = 0; n < np; ++n) {
        const double *a = pts[ord[n]], *b = pts[ord[(n + 1) % np]];
        av[0] += a[1] * b[2] - a[2] * b[1];
        av[1] += a[2] * b[0] - a[0] * b[2];
        av[2] += a[0] * b[1] - a[1] * b[0];
      }
      dual = 0.5 * sqrt(av[0] * av[0] + av[1] * av[1] + av[2] * av[2]);
    }
    if (!(dual > 0.0)) dual = primal > 0.0 ? gv / primal : 0.0;
    const double ih = dual > 0.0 ? primal / dual : 0.0;
    double *geo = G.geo + 4 * e;
    for (int q = 0; q < 3; ++q) geo[q] = nlen > 0 ? dr[q] / nlen : 0.0;
    geo[3] = ih;
    for (int a = G.aoff[e]; a < G.aoff[e + 1]; ++a) {  // the registry publishes it to every alias
      const int *r = G.alias + 6 * a;
      const V<R> B = block_view<R>(D, s, r[0]);
      AT(cALX + r[1], r[2], r[3], r[4]) = (R)ih;
    }
  });
}

// The EMF and the Hall EMF of the singular edges' owners:
// AssembleSingularEdgeEMF_NonHall_ (Z4_Mercury/src/physics/MercurySolver_MagExplicit_Ideal.cpp:57-130) and
// AssembleSingularEdgeEMF_HallExplicit_ (MercurySolver_MagExplicit_Hall.cpp:32-56): the |Jac|-weighted
// sum over the incident cells of the cell field projected on the canonical
// edge vector, times the owner's orientation.  (The local artificial
// resistivity term of the non-Hall EMF is not included.)
// The cell fields are the last step's, final before this step's first kernel
// starts, so the sums are made ahead of the wait and only the owners are written
// behind it (the alias reduction writes them first): 68 us for a step of the
// shell of 8 x 8 x 12 cells in FP64, 74 with the sums behind the wait.
template <class R>
__global__ void k_sing_emf(Dir D) {
  let_dependents_launch();
  const int total = D.sing_prefix[D.nsolves];
  if ((int)(blockIdx.x * blockDim.x) >= total) {
    if (blockIdx.x == 0) wait_for_predecessors();
    return;
  }
  bool first = true;
  for (int e0 = blockIdx.x * blockDim.x; e0 < total; e0 += gridDim.x * blockDim.x) {
    const int ge = e0 + (int)threadIdx.x, s = find_solve(D.sing_prefix, D.nsolves, min(ge, total - 1));
    const DevSingular &G = D.solves[s].sing;
    const int e = min(ge, total - 1) - D.sing_prefix[s];
    const bool on = ge < total && solve_active(D, s);
    const ConstsT<R> &c = consts_of<R>(D.solves[s]);
    const double *geo = G.geo + 4 * e;
    const R cv[3] = {(R)geo[0], (R)geo[1], (R)geo[2]};
    R sumE = R(0.0), sumH = R(0.0);
    for (int q = G.coff[e]; on && q < G.coff[e + 1]; ++q) {
      const int *r = G.cell + 6 * q;
      const V<R> B = block_view<R>(D, s, r[0]);
      const int i = r[2], j = r[3], k = r[4];
      const R u0 = AT(cUP, i, j, k), u1 = AT(cUP + 1, i, j, k), u2 = AT(cUP + 2, i, j, k);
      const R b0 = AT(cBC, i, j, k), b1 = AT(cBC + 1, i, j, k), b2 = AT(cBC + 2, i, j, k);
      const R ex = -(u1 * b2 - u2 * b1), ey = -(u2 * b0 - u0 * b2), ez = -(u0 * b1 - u1 * b0);
      R emf = ex * cv[0] + ey * cv[1] + ez * cv[2];
      const Num<R> num = num_limiter<R>(c, AT(cUH, i, j, k), AT(cUN, i, j, k));
      if (c.ambipolar) {
        const int ax = r[1];
        const int im = i - (ax == 0), jm = j - (ax == 1), km = k - (ax == 2);
        const int ip = i + (ax == 0), jp = j + (ax == 1), kp = k + (ax == 2);
        const R dp = R(0.5) * ((AT(cPVH + 3, ip, jp, kp) + AT(cPVN + 3, ip, jp, kp)) -
                               (AT(cPVH + 3, im, jm, km) + AT(cPVN + 3, im, jm, km)));
        const R pressure_coef = (c.rho_ref * c.U_ref) / (c.q_e * c.L_ref * c.B_ref * c.n_ref);
        emf -= pressure_coef * R(r[5]) * dp / num.ne_eff;
      }
      const R j0 = AT(cJC, i, j, k), j1 = AT(cJC + 1, i, j, k), j2 = AT(cJC + 2, i, j, k);
      if (c.arti_eta_max > R(0.0)) {
        const R jedge = j0 * cv[0] + j1 * cv[1] + j2 * cv[2];
        const R jmag = sqrt(j0 * j0 + j1 * j1 + j2 * j2);
        R qq = (jmag - c.arti_J_start) / dmax(c.arti_J_on - c.arti_J_start, R(1.e-30));
        qq = dmax(R(0.0), dmin(R(1.0), qq));
        emf += c.arti_eta_max * qq * qq * (R(3.0) - R(2.0) * qq) * jedge;
      }
      const R w = (R)G.w[q];
      sumE += w * emf;
      // Hall: alpha (J x B) at the cell, times the radial taper at its centre
      const R alpha = c.hall_coef / num.ne_eff;
      const R hx = alpha * (j1 * b2 - j2 * b1), hy = alpha * (j2 * b0 - j0 * b2), hz = alpha * (j0 * b1 - j1 * b0);
      sumH += w * (AT(cTPC, i, j, k) * (hx * cv[0] + hy * cv[1] + hz * cv[2]));
    }
    if (first) wait_for_predecessors();
    first = false;
    if (!on) continue;
    const R os = (R)G.osign[e];
    *at_code<R>(D.solves[s], D.state[s].cur, G.owner[3 * e]) = os * sumE;
    *at_code<R>(D.solves[s], D.state[s].cur, G.owner[3 * e + 1]) = os * sumH;
  }
}

// The current of the singular edges' owners (AssembleSingularEdgeCurrent_,
// Z4_Mercury/src/physics/MercurySolver_Current.cpp:59-138): the inverse Hodge star times the sum
// over the incident owner faces of the signed beta B, times the owner's
// orientation.
template <class R>
__global__ void k_sing_j(Dir D, int field) {
  for_singular(D, [&](int s, const DevSingular &G, int e) {
    const R ih = (R)G.geo[4 * e + 3];
    R sum = R(0.0);
    for (int q = G.foff[e]; q < G.foff[e + 1]; ++q) {
      const int *r = G.face + 6 * q;
      if (r[5] == 0) continue;
      const V<R> B = block_view<R>(D, s, r[0]);
      const int ax = r[1];
      R beta = R(0.0);
      if constexpr (sizeof(R) == 8)
        if (B.narrow) beta = (R)((const float *)(B.narrow + (uint64_t)rslot(cBFX + ax) * (B.tb / 2)))[B.off(r[2], r[3], r[4])];
      if (sizeof(R) == 4 || !B.narrow) beta = AT(cBFX + ax, r[2], r[3], r[4]);
      sum += ih * R(r[5]) * beta * AT((field == RES_OF_DB ? cRBS : cBX) + ax, r[2], r[3], r[4]);
    }
    *at_code<R>(D.solves[s], D.state[s].cur, G.owner[3 * e + 2]) = R(G.osign[e]) * sum;
  });
}

#undef AT
#undef ATM

}  // namespace

// ------------------------------------------------------------------ launchers
// Every range kernel is persistent (grid-stride over tiles): its grid is the
// SM count times the CTAs of it that fit on one SM, so all CTAs
// are resident at once and none starts in a late partial wave.  The
// residual-dot kernel keeps a fixed grid: its partial sums are indexed by CTA.
static int g_grid_tiles = 0;
static int g_grid_kernel[SK_COUNT];
static int g_grid_fluid[kNumFluidTiles];  // the fluid kernel's, per tile variant

template <class T>
struct SameAs {
  using type = T;
};
template <class T>
using Same = typename SameAs<T>::type;
// A launch that may begin while its predecessor in the stream drains; the kernel
// waits itself (wait_for_predecessors).  t_full: after it instead, in full.
static thread_local bool t_full = false;
static thread_local int t_smem = 0;  // dynamic shared memory of the next launch
template <class... P>
static void launch_dependent(void (*fn)(P...), int grid, int threads, cudaStream_t st, Same<P>... args) {
  cudaLaunchAttribute a[1];
  a[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  a[0].val.programmaticStreamSerializationAllowed = t_full ? 0 : 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.stream = st;
  cfg.dynamicSmemBytes = (size_t)t_smem;
  cfg.attrs = a;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, fn, args...);
  t_smem = 0;
}

template <class R>
static const void *fluid_fn(int v) {
  switch (v) {
    case 1: return (const void *)k_fluid<R, 1>;
    case 2: return (const void *)k_fluid<R, 2>;
    case 3: return (const void *)k_fluid<R, 3>;
    case 4: return (const void *)k_fluid<R, 4>;
    case 5: return (const void *)k_fluid<R, 5>;
    case 6: return (const void *)k_fluid<R, 6>;
    default: return (const void *)k_fluid<R, 0>;
  }
}
static_assert(kNumFluidTiles == 7, "fluid_fn lists every variant");
template <class R>
static void launch_fluid(int v, const Dir &D, cudaStream_t st) {
  v = (v >= 0 && v < kNumFluidTiles) ? v : 0;
  launch_dependent((void (*)(Dir))fluid_fn<R>(v), g_grid_fluid[v], fluid_threads(v), st, D);
}

template <class R>
static const void *kernel_fn(StepKernel k) {
  switch (k) {
    case SK_FACE_EMF: return (const void *)k_face_emf<R>;
    case SK_EDGE_EMF: return (const void *)k_edge_emf<R>;
    case SK_ADD_HALL: return (const void *)k_add_hall<R>;
    case SK_FLUID: return fluid_fn<R>(0);
    case SK_BFACE: return (const void *)k_bface<R>;
    case SK_BCELL_JEDGE: return (const void *)k_bcell_jedge<R>;
    case SK_JCELL: return (const void *)k_jcell<R>;
    case SK_PV_UPLUS: return (const void *)k_pv_uplus<R>;
    case SK_SYNC: return (const void *)k_sync<R, kMaxSyncOps>;
    case SK_FACE_NORMALS: return (const void *)k_face_normals<R>;
    case SK_FLUX_TERMS: return (const void *)k_flux_terms<R>;
    case SK_DIVB: return (const void *)k_div_b<R>;
    case SK_RES_SEED: return (const void *)k_res_seed<R>;
    case SK_RES_W: return (const void *)k_res_w<R>;
    case SK_RES_VEC: return (const void *)k_res_vec<R>;
    case SK_RES_DB: return (const void *)k_res_db<R>;
    case SK_RES_DJ: return (const void *)k_res_dj<R>;
    case SK_RES_Q: return (const void *)k_res_q<R>;
    case SK_RES_COPYB: return (const void *)k_res_copyb<R>;
    case SK_RES_BUPDATE: return (const void *)k_res_bupdate<R>;
    case SK_RES_CG: return (const void *)k_res_cg<R, CG_RR>;
    case SK_RES_PUPD_E: return (const void *)k_res_pupd_e<R>;
    case SK_PHYS: return (const void *)k_phys<R>;
    case SK_RES_CLEARB: return (const void *)k_res_clearb<R>;
    default: return nullptr;
  }
}

// Threads of a kernel's CTAs.
static int kernel_threads(StepKernel k) {
  switch (k) {
    case SK_FACE_EMF: case SK_EDGE_EMF: case SK_ADD_HALL: case SK_BFACE: case SK_BCELL_JEDGE:
    case SK_JCELL: case SK_PV_UPLUS: case SK_FACE_NORMALS: case SK_DIVB: case SK_RES_SEED: case SK_RES_W:
    case SK_RES_VEC: case SK_RES_DB: case SK_RES_DJ: case SK_RES_Q: case SK_RES_BUPDATE: case SK_RES_CG:
    case SK_RES_PUPD_E: case SK_FLUX_TERMS:
      return kVecThreads;
    default: return kTileThreads;
  }
}

// Dynamic shared memory of a kernel (its stage).
template <class R>
static int kernel_smem(StepKernel k) {
  switch (k) {
    case SK_PV_UPLUS: return stage_bytes(kPvSlots, group_size(kAlloc, sizeof(R)) * (int)sizeof(R));
    default: return 0;
  }
}

static std::once_flag g_grids_once;

template <class R>
static void grids_init() {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  for (int k = 0; k < SK_COUNT; ++k) {
    int per_sm = 8;
    const void *fn = kernel_fn<R>((StepKernel)k);
    const int smem = kernel_smem<R>((StepKernel)k);
    if (smem > 0) cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (fn && (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kernel_threads((StepKernel)k), smem) != cudaSuccess ||
               per_sm < 1)) {
      cudaGetLastError();
      per_sm = 1;
    }
    g_grid_kernel[k] = sms * per_sm;
  }
  for (int v = 0; v < kNumFluidTiles; ++v) {
    int per_sm = 1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fluid_fn<R>(v), fluid_threads(v), 0) != cudaSuccess ||
        per_sm < 1) {
      cudaGetLastError();
      per_sm = 1;
    }
    g_grid_fluid[v] = sms * per_sm;
  }
  g_grid_tiles = sms * 8;
}

template <class R>
static void grids() {
  std::call_once(g_grids_once, grids_init<R>);
}

template <class R>
static void launch_as(StepKernel k, const Dir &D, cudaStream_t st, const SyncOps *ops, int iarg, double darg,
                      ResScratch rs) {
  const int G = g_grid_kernel[k];
  t_smem = kernel_smem<R>(k);
  switch (k) {
    case SK_FACE_EMF: launch_dependent(k_face_emf<R>, G, kVecThreads, st, D); break;
    case SK_EDGE_EMF: launch_dependent(k_edge_emf<R>, G, kVecThreads, st, D); break;
    case SK_ADD_HALL: launch_dependent(k_add_hall<R>, G, kVecThreads, st, D); break;
    case SK_FLUID: launch_fluid<R>(iarg, D, st); break;  // iarg: the tile variant
    case SK_BFACE: launch_dependent(k_bface<R>, G, kVecThreads, st, D); break;
    case SK_BCELL_JEDGE: launch_dependent(k_bcell_jedge<R>, G, kVecThreads, st, D); break;
    case SK_JCELL: launch_dependent(k_jcell<R>, G, kVecThreads, st, D); break;
    case SK_PV_UPLUS: launch_dependent(k_pv_uplus<R>, G, kVecThreads, st, D, iarg); break;
    case SK_SYNC:
      if (ops->n == 1) launch_dependent(k_sync<R, 1>, G, kTileThreads, st, D, *ops);
      else if (ops->n == 2) launch_dependent(k_sync<R, 2>, G, kTileThreads, st, D, *ops);
      else launch_dependent(k_sync<R, kMaxSyncOps>, G, kTileThreads, st, D, *ops);
      break;
    case SK_FACE_NORMALS: k_face_normals<R><<<G, kVecThreads, 0, st>>>(D); break;
    case SK_FLUX_TERMS: launch_dependent(k_flux_terms<R>, G, kVecThreads, st, D); break;
    case SK_DIVB: k_div_b<R><<<G, kVecThreads, 0, st>>>(D); break;
    case SK_RES_SEED: k_res_seed<R><<<G, kVecThreads, 0, st>>>(D); break;
    case SK_RES_W: k_res_w<R><<<G, kVecThreads, 0, st>>>(D); break;
    case SK_RES_VEC: launch_dependent(k_res_vec<R>, G, kVecThreads, st, D, iarg, rs.cg, rs.use_p); break;
    case SK_RES_DB: launch_dependent(k_res_db<R>, G, kVecThreads, st, D); break;
    case SK_RES_DJ: launch_dependent(k_res_dj<R>, G, kVecThreads, st, D, iarg); break;
    case SK_RES_Q: launch_dependent(k_res_q<R>, G, kVecThreads, st, D); break;
    case SK_RES_DOT: k_res_dot<R><<<g_grid_tiles, kVecThreads, 0, st>>>(D, rs.partial); break;
    case SK_RES_SUM: k_res_sum<<<1, 32, 0, st>>>(rs.partial, g_grid_tiles, rs.result); break;
    case SK_RES_COPYB: launch_dependent(k_res_copyb<R>, G, kTileThreads, st, D, iarg); break;
    case SK_RES_BUPDATE: launch_dependent(k_res_bupdate<R>, G, kVecThreads, st, D); break;
    case SK_RES_CG:
      if (iarg == CG_INIT)
        launch_dependent(k_res_cg<R, CG_INIT>, G, kVecThreads, st, D, rs.tpartial, rs.cg, rs.sarrivals, rs.handle,
                         rs.in_graph, rs.use_p);
      else if (iarg == CG_PQ)
        launch_dependent(k_res_cg<R, CG_PQ>, G, kVecThreads, st, D, rs.tpartial, rs.cg, rs.sarrivals, rs.handle,
                         rs.in_graph, rs.use_p);
      else
        launch_dependent(k_res_cg<R, CG_RR>, G, kVecThreads, st, D, rs.tpartial, rs.cg, rs.sarrivals, rs.handle,
                         rs.in_graph, rs.use_p);
      break;
    case SK_RES_PUPD_E: launch_dependent(k_res_pupd_e<R>, G, kVecThreads, st, D, rs.cg, rs.use_p); break;
    case SK_PHYS: launch_dependent(k_phys<R>, G, 256, st, D, iarg & 255, (iarg >> 8) - 1); break;
    // one thread per singular edge (8 radial lines of nr edges per shell)
    case SK_SING_SETUP: k_sing_setup<R><<<g_grid_tiles / 2, 64, 0, st>>>(D); break;
    case SK_SING_EMF: launch_dependent(k_sing_emf<R>, g_grid_tiles / 2, 64, st, D); break;
    case SK_SING_J: launch_dependent(k_sing_j<R>, g_grid_tiles / 2, 64, st, D, iarg); break;
    case SK_RES_CLEARB: launch_dependent(k_res_clearb<R>, G, kTileThreads, st, D); break;
    default: break;
  }
}

// The FP32 instantiations are compiled in their own translation unit (this
// file built with MHD_KERNELS_F32 and FP32 fast-math flags: FMA contraction,
// approximate division and square root); the FP64 one keeps the bit-exact
// flags.
#if MHD_KERNELS_F32
// Vectors of the mixed-precision implicit substep between a solve's FP32
// arena (every masked solve of D) and its FP64 companion (DevSolve::companion:
// the companion's blocks, the same boxes)
// over the substep's range (kResK), where its unknowns are:
// RES_X_SETUP: the companion's r = the solve's r (the FP32 right-hand side
//   eta J(B*)) and its dt = the step's; with cg (direct) r is made here, without
//   (refinement) also the companion's b (in its face arrays) = r and x = 0.
// RES_X_DEMOTE_R: r = (float) companion r (the next correction's right-hand side).
// RES_X_ADD_X: companion x += the correction (the solve's CG cg).
// RES_X_DEMOTE_X: x = (float) companion x: the solution of the companion's CG cg
//   (E_res = x too),
//   or without it the refined x.
template <int OP>
__global__ void __launch_bounds__(kVecThreads) k_res_cross(Dir D, const ResCG *cg, int use_p) {
  for_vec_items<float, kResK>(D, [&](const DevSolve &S, const VV<float> &B, const VItem &it) {
    if (OP == RES_X_SETUP && threadIdx.x == 0 && it.w == D.solve_tile_prefix[kResK][it.s]) {
      S.companion_state->dt = D.state[it.s].dt;  // the step's dt, once per solve
      S.companion_state->dt_bits = D.state[it.s].dt_bits;
    }
    V<double> C;
    set_view(C, S.companion[it.blk], 0);
    // the four positions in the companion's arrays (the same box: twice the byte offset, 32-byte aligned)
    auto at = [&](int comp) { return (double2 *)((char *)C.c(comp) + 2 * (uint64_t)it.o); };
    auto widen = [&](int comp, const Vec<float> &v) {  // positions outside the range keep their values
      double2 *p = at(comp);
      if (!it.in) return;
      if (it.k >= it.klo && it.k + 4 <= it.khi) {
        p[0] = make_double2((double)v.v[0], (double)v.v[1]);
        p[1] = make_double2((double)v.v[2], (double)v.v[3]);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (it.has(e)) ((double *)p)[e] = (double)v.v[e];
      }
    };
    auto narrow = [&](int comp) {
      const double2 *p = at(comp);
      const double2 a = p[0], b = p[1];
      Vec<float> v;
      v.v[0] = (float)a.x;
      v.v[1] = (float)a.y;
      v.v[2] = (float)b.x;
      v.v[3] = (float)b.y;
      return v;
    };
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      if (OP == RES_X_SETUP) {
        Vec<float> r;
        if (cg) {  // RES_INIT
          const Vec<float> W = B.fixed(cRW + a, it.o), b = 0.0f + B.fixed(cETAR + a, it.o) * B.lv(cJX + a, it.o);
          r = vmap<float>([&](int e) { return W.v[e] > 0.0f ? b.v[e] : 0.0f; });
          B.st(cRR + a, it, r, it.klo, it.khi);
        } else {
          r = B.lv(cRR + a, it.o);
        }
        widen(cRR + a, r);
        if (!cg) {  // refinement: b and x
          widen(cBX + a, r);
          widen(cRX + a, vset(0.0f));
        }
      } else if (OP == RES_X_DEMOTE_R) {
        B.st(cRR + a, it, narrow(cRR + a), it.klo, it.khi);
      } else if (OP == RES_X_ADD_X) {
        const Vec<float> x = B.lv(cRX + a, it.o), d = B.lv(dir_comp(use_p) + a, it.o), W = B.fixed(cRW + a, it.o);
        double *p = (double *)at(cRX + a);
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (it.in && it.has(e) && W.v[e] > 0.0f) p[e] += (double)final_x(cg[it.s], x.v[e], d.v[e]);
      } else if (cg) {  // RES_X_DEMOTE_X of a finished CG on the companion (its own slot's state)
        const ResCG &c = cg[S.companion_slot];
        const double *x = (const double *)at(cRX + a), *p = (const double *)at(dir_comp(use_p) + a);
        const Vec<float> W = B.fixed(cRW + a, it.o);
        Vec<float> v;
#pragma unroll
        for (int e = 0; e < 4; ++e) v.v[e] = W.v[e] > 0.0f ? (float)final_x(c, x[e], p[e]) : 0.0f;
        B.st(cRX + a, it, v, it.klo, it.khi);
        B.st(cEX + a, it, v, it.klo, it.khi);  // RES_E_FROM_X
      } else {  // RES_X_DEMOTE_X of a refined solution
        B.st(cRX + a, it, narrow(cRX + a), it.klo, it.khi);
      }
    }
  });
}

void launch_res_cross(const Dir &D, int op, cudaStream_t st, const ResCG *cg, int use_p, bool full) {
  grids<float>();
  t_full = full;
  switch (op) {
    case RES_X_SETUP: launch_dependent(k_res_cross<RES_X_SETUP>, g_grid_tiles, kVecThreads, st, D, cg, use_p); break;
    case RES_X_DEMOTE_R: launch_dependent(k_res_cross<RES_X_DEMOTE_R>, g_grid_tiles, kVecThreads, st, D, cg, use_p); break;
    case RES_X_ADD_X: launch_dependent(k_res_cross<RES_X_ADD_X>, g_grid_tiles, kVecThreads, st, D, cg, use_p); break;
    default: launch_dependent(k_res_cross<RES_X_DEMOTE_X>, g_grid_tiles, kVecThreads, st, D, cg, use_p); break;
  }
}

void launch_step_kernel_f32(StepKernel k, const Dir &D, cudaStream_t st, const SyncOps *ops, int iarg, double darg,
                            ResScratch rs, bool full) {
  grids<float>();
  t_full = full;
  launch_as<float>(k, D, st, ops, iarg, darg, rs);
}

void init_launch_grids_f32() { grids<float>(); }

void launch_res_kmax_f32(const Dir &D, int *out, cudaStream_t st) {
  grids<float>();
  k_res_kmax<float><<<g_grid_tiles, kVecThreads, 0, st>>>(D, out);
}
#else
void launch_res_kmax_f32(const Dir &D, int *out, cudaStream_t st);

void launch_res_kmax(const Dir &D, int precision, int *out, cudaStream_t st) {
  if (precision == kMixed) {
    launch_res_kmax_f32(D, out, st);
  } else {
    grids<double>();
    k_res_kmax<double><<<g_grid_tiles, kVecThreads, 0, st>>>(D, out);
  }
}

__global__ void k_res_begin(Dir D, ResCG *cg, int mixed) {
  for (int s = threadIdx.x; s < D.nsolves; s += blockDim.x) {
    const DevSolve &S = D.solves[s];
    SolveState &st = D.state[s];
    const bool on = S.nblocks > 0 && S.c.resistive && st.remaining > 0 && st.status == 0;
    st.mask = on;
    if (mixed && !(S.nblocks > 0 && S.c.resistive)) continue;
    ResCG h{};
    h.done = !on;
    h.ran = on;
    h.tol_factor = S.res_tol;
    h.max_it = S.res_max_it;
    cg[mixed ? S.companion_slot : s] = h;
    if (mixed) S.companion_state->mask = on;
  }
}
__global__ void k_res_end(Dir D, const ResCG *cg, ResCG *host, int n, int mixed, int last) {
  for (int s = threadIdx.x; s < D.nsolves; s += blockDim.x) {
    const DevSolve &S = D.solves[s];
    SolveState &st = D.state[s];
    if (!(S.nblocks > 0 && S.c.resistive)) continue;
    const ResCG &h = cg[mixed ? S.companion_slot : s];
    st.mask = !last && h.ran;
    if (!last && h.ran && !h.converged) st.status = MHD_ERR_SOLVE;
  }
  if (!last)
    for (int q = threadIdx.x; q < n; q += blockDim.x) host[q] = cg[q];
}

void launch_res_begin(const Dir &D, ResCG *cg, bool mixed, cudaStream_t st) {
  k_res_begin<<<1, 256, 0, st>>>(D, cg, mixed);
}
void launch_res_end(const Dir &D, const ResCG *cg, ResCG *host, int n, bool mixed, bool last, cudaStream_t st) {
  k_res_end<<<1, 256, 0, st>>>(D, cg, host, n, mixed, last);
}

void launch_step_kernel_f32(StepKernel k, const Dir &D, cudaStream_t st, const SyncOps *ops, int iarg, double darg,
                            ResScratch rs, bool full);

void launch_step_kernel(StepKernel k, const Dir &D, cudaStream_t st, const SyncOps *ops, int precision, int iarg,
                        double darg, ResScratch rs, bool full) {
  if (precision == kMixed) {
    launch_step_kernel_f32(k, D, st, ops, iarg, darg, rs, full);
  } else {
    grids<double>();
    t_full = full;
    launch_as<double>(k, D, st, ops, iarg, darg, rs);
  }
}

void init_launch_grids_f32();

void init_launch_grids() {
  grids<double>();
  init_launch_grids_f32();
}

int res_dot_grid() {
  grids<double>();
  return g_grid_tiles;
}

const char *step_kernel_name(StepKernel k) {
  static const char *names[] = {"k_face_emf", "k_edge_emf", "k_add_hall",
                                "k_fluid",    "k_bface",    "k_bcell_jedge", "k_jcell",   "k_pv_uplus",
                                "k_sync",     "k_face_normals", "k_div_b",
                                "k_res_seed", "k_res_w",    "k_res_vec",     "k_res_db",   "k_res_dj",
                                "k_res_q",    "k_res_dot",  "k_res_sum",     "k_res_copyb", "k_res_bupdate",
                                "k_res_cg",   "k_res_pupd_e", "k_phys",      "k_sing_setup", "k_sing_emf",
                                "k_sing_j",   "k_res_clearb", "k_flux_terms"};
  static_assert(sizeof(names) / sizeof(names[0]) == SK_COUNT, "a name per kernel");
  return (k >= 0 && k < SK_COUNT) ? names[k] : "?";
}
#endif  // MHD_KERNELS_F32

}  // namespace mhd
