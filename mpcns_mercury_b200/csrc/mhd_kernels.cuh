// Launch interface of the engine's step kernels (mhd_kernels.cu).
#pragma once
#include <cuda_runtime.h>

#include "mhd_engine.cuh"

namespace mhd {

enum StepKernel {
  SK_FACE_EMF = 0, SK_EDGE_EMF, SK_ADD_HALL, SK_FLUID, SK_BFACE, SK_BCELL_JEDGE,
  SK_JCELL, SK_PV_UPLUS, SK_SYNC, SK_FACE_NORMALS, SK_DIVB,
  // implicit resistive substep
  SK_RES_SEED, SK_RES_W, SK_RES_VEC, SK_RES_DB, SK_RES_DJ, SK_RES_Q, SK_RES_DOT, SK_RES_SUM, SK_RES_COPYB,
  SK_RES_BUPDATE, SK_RES_CG, SK_RES_PUPD_E,
  // grids with physical boundaries and singular edges
  SK_PHYS, SK_SING_SETUP, SK_SING_EMF, SK_SING_J,
  // implicit resistive substep on grids with physical boundaries: zero the ghost faces of dB
  SK_RES_CLEARB,
  SK_FLUX_TERMS, SK_COUNT
};

// One launch of k_sync runs up to kMaxSyncOps independent sync operations: a copy
// phase of a group (halo or owner copies) or an edge alias reduction.
enum SyncKind { SYNC_COPY = 0, SYNC_ALIAS = 1 };
struct SyncOp {
  int kind;   // SyncKind
  int arg;    // SYNC_COPY: group; SYNC_ALIAS: 0 = E, 1 = J
  int phase;  // SYNC_COPY: a CopyPhase (mhd_engine.cuh)
  int prev;   // SYNC_COPY: read U components from the other buffer (1) -- the staged
              // ghosts of Sync(U) inside the step, whose last synced values are there
  int mark;   // SYNC_COPY: write 0 to every destination instead of the copy (marks
              // the phase's destinations, e.g. the non-owner aliases of an owner phase);
              // SYNC_ALIAS: write every member of a class, not only its owner
};
constexpr int kMaxSyncOps = 6;
struct SyncOps {
  SyncOp op[kMaxSyncOps];
  int n;
};

// Operations of SK_RES_VEC / SK_RES_COPYB / SK_RES_DJ (the arg of the launch).
enum ResVecOp { RES_INIT = 0, RES_E_FROM_P, RES_E_FROM_X, RES_E_FROM_CG, RES_P_FROM_X, RES_RESID };
enum ResCopyOp { RES_DB_FROM_B = 0, RES_B_FROM_DB };
enum ResField { RES_OF_B = 0, RES_OF_DB };  // SK_RES_DJ, SK_SING_J: the current of B, or of the operator's dB

// CG state of one solve on the device (one per slot), for the iteration
// loop run as a CUDA graph over every masked solve at once (k_res_cg,
// k_res_pupd_e): the host sets tol_factor and max_it (and
// zeros the rest) before the graph and reads it back after.
struct ResCG {
  double rho, alpha, beta;  // W-weighted r.r, step length, direction update
  double r0, rnorm, tol;    // ||r|| at the start and now, stop when rnorm <= tol = tol_factor * r0
  double tol_factor;
  int it, max_it;           // iterations taken, at most max_it
  int done, converged;      // loop over (converged, max_it reached, or breakdown)
  int pending;              // x lacks the last step alpha p (final_x)
  int ran;                  // the solve took part in the last substep (launch_res_begin)
};
// Steps of k_res_cg: CG_INIT: p = r, E = p, (r.r)_W and r.r, sets rho, r0, tol;
// CG_PQ: q = A p (its last part, E - eta dJ) and (p.q)_W, sets alpha;
// CG_RR: r -= alpha q, (r.r)_W and r.r, the stop test and beta (k_res_pupd_e then
// updates x and p).
// Every tile writes its pair of partial sums; the CTA that finishes a solve's
// last tile adds them in a fixed order and updates the solve's state; a solve
// whose loop is over leaves the mask.
enum ResCgOp { CG_INIT = 0, CG_PQ, CG_RR };

// Scratch of the CG dot products: per-CTA partial sums and the two results
// (k_res_dot, one masked solve); the per-slot CG states, the tile partials of
// the batched loop, its tickets and the graph's loop condition.
struct ResScratch {
  double *partial;  // 2 * grid
  double *result;   // 2
  ResCG *cg = nullptr;
  double *tpartial = nullptr;         // 2 per kResK tile
  unsigned int *sarrivals = nullptr;  // per slot: its tiles summed so far
  unsigned long long handle = 0;  // cudaGraphConditionalHandle of the loop
  int in_graph = 0;               // the CG kernels set the loop condition (launched inside the loop graph)
  int use_p = 0;                  // the direction is kept in RES_P beside E_res
};

// Launch one engine kernel over the directory D (ops: SK_SYNC only) in the
// batch's precision (Precision); iarg / darg: the operation and scalar of the
// implicit resistive kernels (SK_PV_UPLUS: iarg = 1 ends the step).  full: the launch
// waits for its predecessor to complete instead of overlapping its end.
void launch_step_kernel(StepKernel k, const Dir &D, cudaStream_t st, const SyncOps *ops, int precision, int iarg = 0,
                        double darg = 0.0, ResScratch rs = ResScratch{nullptr, nullptr}, bool full = false);
int res_dot_grid();
// Mixed-precision implicit substep: moves its vectors between every masked
// solve of the FP32 directory D and its FP64 companion (DevSolve::companion;
// RES_X_SETUP also hands over the step's dt) (k_res_cross, FP32 translation
// unit).  cg, use_p: the states and the direction of the CG whose solution is taken;
// full: as in launch_step_kernel.
enum ResCrossOp { RES_X_SETUP = 0, RES_X_DEMOTE_R, RES_X_ADD_X, RES_X_DEMOTE_X };
void launch_res_cross(const Dir &D, int op, cudaStream_t st, const ResCG *cg, int use_p, bool full);
// The ends of a substep whose decisions stay on the device.  launch_res_begin
// masks the resistive solves that take this step (and their companions; mixed:
// the CG runs on these) and sets up their CG states.  launch_res_end after the
// CG: masks them again, gives a solve that did not converge MHD_ERR_SOLVE and
// writes the n states to host (pinned); with last, clears the masks.
void launch_res_begin(const Dir &D, ResCG *cg, bool mixed, cudaStream_t st);
void launch_res_end(const Dir &D, const ResCG *cg, ResCG *host, int n, bool mixed, bool last, cudaStream_t st);
// Per block of the masked solve of D: the largest k of an unknown of the
// implicit substep into out[block] (atomic max; out starts at -1).
void launch_res_kmax(const Dir &D, int precision, int *out, cudaStream_t st);
// Queries every kernel's resident CTAs per SM once (call before any stream capture).
void init_launch_grids();
const char *step_kernel_name(StepKernel k);

}  // namespace mhd
