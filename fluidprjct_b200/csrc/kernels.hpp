// kernels.hpp -- host launchers of the PIC/FLIP kernels (implemented in *.cu).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "common.cuh"

namespace fp {

// Scratch of the persistent PCG kernel: a grid barrier and FP64 partials.
struct GridBar {
    unsigned count;
    unsigned limit;  // polls after which a wait gives up (set at launch)
    unsigned long long* gave_up;  // where a wait that gives up notes the device clock, or null
};

// Polls after which a grid-barrier wait of the persistent solvers gives up
// and reports DEV_TIMEOUT (fp_set_wait_limit lowers it for tests).  Each
// launch stores it in its GridBar, where the polling thread reads it.
constexpr unsigned kDefaultWaitPolls = 1u << 27;

struct PcgOut {
    int iters;
    int status;     // DEV_*
    double rr;      // ||r||^2 of the recurrence at exit
    double bb;      // ||b||^2
    double rz;
    double rr0;     // ||b - A x0||^2 of the initial iterate (MG and mixed)
    int outer;      // refinement loops (plain PCG: 1; MG leaves it alone)
    int pad_;
    // device clock (clock_ns) at the start of launch_pressure_setup, and at the
    // solve kernel's start and end (or when a wait of it gave up)
    unsigned long long t_setup, t_begin, t_end;
};

// Device buffers of the pressure system.  Compact arrays are indexed by the
// fluid number n (i-fastest order of FLUID cells); padded dense grids have a
// one-cell zero halo, (W+2)*(H+2)*(D+2) entries.  Vector storage is sized for
// FP64 and reinterpreted as FP32 by the mixed-precision solves.
struct PressureBufs {
    int* nf;              // [1] number of FLUID cells
    int* fidx;            // [nc] padded index of the n-th FLUID cell
    uint8_t* diag;        // [nc] diagonal of the unit operator (compact)
    float* b;             // [nc] right-hand side (compact)
    float* bin;           // [nc] right-hand side of an inner refinement solve
    void* R[2];           // padded dense residual (double-buffered); R[0] also u = M^-1 r
    void* Wv[2];          // padded dense w = A M^-1 r
    void* S[2];           // padded dense s = A p
    void* invd;           // padded dense 1/diag
    void* P;              // [nc] compact search direction
    void* X;              // [nc] compact solution
    double* x64;          // [nc] refinement accumulator (compact)
    double* xd;           // padded dense FP64 iterate
    double* part;         // [6 * max_blocks] per-block partial sums
    GridBar* bar;         // [1]
    PcgOut* out;          // [1]
    int* tile_sums;       // scan scratch
    double* red;          // [2] FP64 reduction results (true residual)
};

// -------- multigrid-preconditioned PCG (kernels_mg.cu) --------
constexpr int MG_MAX_LEVELS = 8;
constexpr int MG_BLOCK_CELLS = 4096;           // levels at most this big are solved by one block ...
constexpr int MG_SMEM_BUDGET = 188 * 1024;     // ... in shared memory, when their copies fit in this
constexpr int MG_OX = 4;                       // cells before a padded row's first one
// One multigrid level: padded dense grids with a SOLID / zero halo; cell
// (i, j, k) at (i + MG_OX) + (j + 1) sy + (k + 1) sz.
struct MgLevel {
    int W, H, D;    // interior cells
    int sy, sz;     // padded strides: W up to a multiple of 4, + MG_OX; sy (H + 2)
    uint8_t* lab;   // labels (BODY folded into SOLID)
    float* x;       // correction (level 0: the preconditioned residual z)
    float* b;       // right-hand side (level 0: the residual r)
    uint8_t* code;  // per solve: FLUID cells 1 + diagonal, every other cell 0
};
// A quad -- four aligned cells of a row, at least one of them FLUID -- in a
// level's list, as an int4: x the first cell's padded index; y the four codes
// (level 0 only) and the bits below; z the padded index, on the next level, of
// the first two cells' parent; w level 0: the first cell's dense index in
// W x H x D, other levels: the padded index, on the finer level, of the first
// cell's first child.
constexpr uint32_t QUAD_CODES = 0x07070707u;
constexpr uint32_t QUAD_ODD = 0x80u;            // j + k is odd: the first cell is black
constexpr uint32_t QUAD_PARENT_ODD = 0x8000u;   // the parent row's J + K is odd
constexpr uint32_t QUAD_Z = 0x800000u;          // the children's second z plane lies in the finer level
constexpr uint32_t QUAD_PAR = QUAD_ODD | QUAD_PARENT_ODD;
// The hierarchy and its buffers.
struct MgBufs {
    int L = 0;
    MgLevel lv[MG_MAX_LEVELS]{};
    int4* q[MG_MAX_LEVELS]{};   // quad lists of the grid-wide levels (level 0: from launch_pressure_setup)
    int* nq = nullptr;          // [MG_MAX_LEVELS] their lengths
    float4* rhs = nullptr;      // right-hand side by level-0 quad
    // FP64 Krylov vectors by quad, 2 * cap pairs each
    double2 *p = nullptr, *s = nullptr, *xs = nullptr, *r = nullptr, *w = nullptr;
    int cap = 0;                // quads of level 0's grid
    double* xd = nullptr;       // level-0 padded grid, zero between solves
};
// Fills lv[].W/H/D/sy/sz of the level hierarchy for a W x H x D grid (down to
// at most 2 cells per axis, or MG_MAX_LEVELS levels); returns L.
int mg_levels_for(int W, int H, int D, MgLevel* lv);
int mg_npad(const MgLevel& L);  // cells of a level's padded grid, up to a multiple of 16
int mg_max_blocks();
// First block-solved level G of the hierarchy and the shared memory its
// copies take (0: the block levels stay in global memory).
int mg_split(const MgLevel* lv, int L, int* smem_bytes);
// Level labels and quad lists of the grid-wide coarse levels from the cell
// labels (per solve; nq[1..] zero before, as launch_pressure_setup leaves
// them); the solver kernel coarsens the shared-memory levels itself.  Returns
// the number of launches.
int launch_mg_setup(const uint8_t* labels, const MgBufs& m, cudaStream_t st);
// MG-preconditioned PCG (FP32 V-cycle, FP64 Krylov vectors and reductions) for
// the system of launch_pressure_setup to ||r||/||rhs|| <= tol; dense pressure
// to pout (its non-FLUID cells must be zero), the true residual's
// ||rhs - A x||^2 and ||rhs||^2 (FP64) to pb.red.
// guess: a dense W x H x D guess (scaled on the device by its energy-optimal
// factor; pout itself may be passed), or null to start from x = 0.  guess_dir:
// it becomes the first search direction (a network's guess); otherwise
// non-finite values in it read as 0.
// nu0: red-black sweep pairs before and after the coarse correction on the
// finest level.
int launch_pcg_mg(Dims g, PressureBufs& pb, const MgBufs& m, double tol, int maxit, const float* guess, int guess_dir,
                  int nu0, float* pout, cudaStream_t st);

// -------- labelling and the particle sort (kernels_sort.cu) --------
// counts must be zero on entry.  Writes key/rank per particle.
void launch_bin(const float4* pos, int64_t np, Dims g, int* counts, int* key, int* rank, cudaStream_t st);
// Labels from the SOLID map, the body mark and counts; exclusive scan of counts
// into start[nc+1]; start[nc] = np; counts left zero.
void launch_label_scan(const uint8_t* base, const uint8_t* body_mark, int* counts, uint8_t* labels, int* start,
                       int* tile_sums, Dims g, cudaStream_t st);
void launch_scatter(const float4* pos, const float4* vel, const int* key, const int* rank, const int* start, int64_t np,
                    float4* pos2, float4* vel2, cudaStream_t st);

// In-place exclusive scan of n ints, the sum to *total; tile_sums has room for
// scan_tiles(n) ints; the start's device clock to *at if it is not null.
// Returns the number of launches.
int launch_scan(int* data, int n, int* total, int* tile_sums, cudaStream_t st, unsigned long long* at = nullptr);
int scan_tiles(int64_t n);

// -------- P2G with the fused normalise / save / gravity epilogue (kernels_p2g.cu) --------
// acc: [nu + nv + nw] (num, den) pairs, zero on entry and left zero (two launches).
void launch_p2g(const float4* pos, const float4* vel, const int* start, Dims g, float dt, float3 gravity,
                float2* acc, float* u, float* v, float* w, float* us, float* vs, float* ws, int fused_forces,
                cudaStream_t st);
void launch_forces(float* u, float* v, float* w, Dims g, float dt, float3 gravity, cudaStream_t st);
void launch_copy(const float* src, float* dst, int64_t n, cudaStream_t st);

// -------- pressure (kernels_pressure.cu) --------
// Compacts FLUID cells, builds rhs (FluidSolver3D.cu:1360-1474) and diagonals,
// zeroes p off the fluid, and readies the solvers' barrier and status (poll
// limit wait_polls).  If rhs_dense is non-null it replaces the computed rhs
// (caller-provided system).  With a multigrid hierarchy (mg->L > 0) it also
// lists level 0's quads with their right-hand sides and zeroes the lengths of
// the other levels' lists.  pb.tile_sums: pressure_tiles(g) ints.
void launch_pressure_setup(const uint8_t* labels, const float* u, const float* v, const float* w, Dims g, float dt,
                           BodyKin body, const float* rhs_dense, float* p, PressureBufs& pb, const MgBufs* mg,
                           unsigned wait_polls, cudaStream_t st);
int pressure_tiles(Dims g);

// -------- plain and mixed-precision PCG (kernels_pcg.cu) --------
// Jacobi PCG with FP64 vectors from x0 = 0 for A x = b (the system of
// launch_pressure_setup) to ||r||/||b|| <= tol.  Dense pressure to pout (its
// non-FLUID cells must be zero), the true residual's ||b - A x||^2 and ||b||^2
// to pb.red, diagnostics to pb.out.  The padded work grids must be zero on
// entry and are zero again on exit, unless a wait gave up.
int launch_pcg(Dims g, PressureBufs& pb, double tol, int maxit, float* pout, cudaStream_t st);
// The same by FP64 iterative refinement around FP32-vector PCG solves, from
// x = 0 or from the compact guess x0 scaled by its energy-optimal factor
// (x0, b) / (x0, A x0).
int launch_pcg_mixed(Dims g, PressureBufs& pb, const float* x0, double tol, int maxit, float* pout, cudaStream_t st);
// Barrier word to zero with its poll limit, status word to DEV_OK: before a
// second persistent solver on the same system (launch_pressure_setup does it
// for the first).
void launch_reset_barrier(GridBar* bar, int* status, unsigned wait_polls, cudaStream_t st);
int pcg_max_blocks();

// -------- projection (kernels_pressure.cu) --------
// guard: the status word of the solve that produced p, or null; the kernel
// does nothing when that solve failed (solve_failed).
void launch_project(float* u, float* v, float* w, const float* p, const uint8_t* labels, Dims g, float dt, BodyKin b,
                    cudaStream_t st, const int* guard = nullptr);

// -------- G2P + advection (kernels_advect.cu) --------
void launch_g2p_advect(float4* pos, float4* vel, int64_t np, const float* u, const float* v, const float* w,
                       const float* us, const float* vs, const float* ws, const uint8_t* labels, Dims g, float alpha,
                       float dt, float cfl, int do_g2p, int do_advect, int rk2, cudaStream_t st,
                       const int* guard = nullptr, const BodyShape* collide = nullptr);
// collide: the body for SDF collision projection (sdf_push_out, eps = dx/4),
// or null for the reference's label search alone.

// -------- rigid body (kernels_body.cu) --------
// mark[c] = 1 where the cell centre is inside the body (SDF <= 0).
void launch_mark_body(uint8_t* mark, Dims g, const BodyShape& b, cudaStream_t st);
// labels[c] = BODY where mark[c] and labels[c] != SOLID (init-time marking).
void launch_apply_mark(uint8_t* labels, const uint8_t* mark, Dims g, cudaStream_t st);
// Fluid force and torque on the body (FP64): out[0..2] force, out[3..5]
// torque about b.com; part holds body_force_partials() doubles.
void launch_body_force(const float* p, const uint8_t* labels, Dims g, const BodyShape& b, double* part, double* out,
                       cudaStream_t st);
int body_force_partials();
// The reference's body forces: out[0..5] = panel drag + lift force and torque
// about cm, out[6..7] = body volume and submerged volume from the SDF voxels.
// part holds body_force_partials() doubles; pos/start are the cell-sorted
// particles.  sdf = null samples the analytic sphere |x - local_com| - radius.
struct RefBuoyancy {
    const float* sdf;
    int sw, sh, sd;
    float cs;
    float3 origin, local_com, com;
    float radius;
    float rot[9];
};
void launch_ref_body_forces(const uint8_t* labels, const float* u, const float* v, const float* w, Dims g, float3 cm,
                            float3 bvel, const RefBuoyancy& b, const float4* pos, const int* start, double* part,
                            double* out, cudaStream_t st);

// -------- particle order helpers --------
// out[pid] = in[slot] for the xyz part of float4 arrays (pid in pos.w bits).
void launch_unsort(const float4* pos, const float4* vel, int64_t np, float* pos_out, float* vel_out, cudaStream_t st);
// rec[6 pid + 0..5] = x y z vx vy vz (frame records in the original order).
void launch_unsort_records(const float4* pos, const float4* vel, int64_t np, float* rec, cudaStream_t st);
// AoS to float4 (w = original index); the lowest index holding a non-finite
// value goes to *bad (set to INT_MAX before the call), if bad is not null.
void launch_pack(const float* pos, const float* vel, int64_t np, float4* pos4, float4* vel4, int* bad,
                 cudaStream_t st);

// -------- generic CSR CG with FP64 vectors (kernels_pressure.cu) --------
// Control block and results of one CSR solve on the device.
struct CsrCtl {
    GridBar bar;
    int status;  // DEV_*
    // 1: the check found malformed offsets, or columns; no solve ran.  Two words: a block may still be
    // reading the first while another already checks columns.
    int bad_off, bad_col;
    int iters;
    double rr, bb;  // ||r||^2 and ||b||^2
};
constexpr int kCsrVectors = 6;  // work vectors of launch_csr_cg
constexpr int kCsrMaxBlocks = 256;
constexpr int kCsrPartials = 4 * kCsrMaxBlocks;  // doubles in part
// Queues the whole solve (two launches): device arrays, work vector i at
// work + i * stride (stride >= n); results in *ctl.  check: validate offsets
// and columns first (x is written only if they pass).  Returns 0 or a
// cudaError_t value.
int launch_csr_cg(int n, const int* off, const int* cols, const double* vals, const double* b, double* x, double* work,
                  int64_t stride, double* part, CsrCtl* ctl, int check, double tol, int maxit, cudaStream_t st,
                  unsigned wait_polls = kDefaultWaitPolls);
// The same from host arrays, complete on return, as an FP_* status; x, *iters
// and *relres are written only with FP_OK.
int csr_cg_solve(int n, const int* offsets, const int* cols, const double* vals, const double* b, double* x, double tol,
                 int maxit, int* iters, double* relres, cudaStream_t st, unsigned wait_polls = kDefaultWaitPolls);

// -------- velocity extrapolation (kernels_extrap.cu) --------
// Values equal to VEL_UNKNOWN on an nx x ny face grid, depth waves; the first
// front reads neighbour markers at row stride front_stride.  mark: nx*ny ints.
// Returns the number of launches.
int launch_extrapolate_unknown(float* v, int nx, int ny, int depth, int front_stride, int* mark, cudaStream_t st);
// Faces of component axis (0 u, 1 v, 2 w) with no FLUID side, depth waves.
// guard: as in launch_project.
int launch_extrapolate_from_fluid(float* v, int axis, const uint8_t* labels, Dims g, int depth, int* mark,
                                  const int* guard, cudaStream_t st);

// -------- scene generation (kernels_scene.cu) --------
void launch_seabed_labels(uint8_t* labels, int W, int H, int D, double dx, double level, double bed_base,
                          double bed_amp, uint64_t seed, double water_xmin, cudaStream_t st);
void launch_levelset_labels(const float* solid, const float* fluid, int64_t n, uint8_t* labels, cudaStream_t st);

// -------- the reference's own 2D step, scheme "ref2d" (kernels_ref2d.cu) --------
// Scratch: start[(W+4)*(H+4)+1] (bins of cells -2..W+1 x -2..H+1), list, key,
// rank [np], keep [np+1], misc[3] (non-finite u and v velocities, capped
// substep loops), tiles (launch_scan over the bins or the keep flags).
struct R2Scratch {
    int *start, *list, *key, *rank, *keep, *misc, *tiles;
    unsigned long long* clock;  // [R2_CLOCKS] device clock at the start of the phases' first kernels
};
enum { R2_AT_LABEL, R2_AT_P2G, R2_AT_PROJECT, R2_AT_PARTICLES, R2_AT_END, R2_CLOCKS };
// Without particles the kernels that note P2G, particles and the end do not run.
void launch_r2_note(R2Scratch& sc, int which, cudaStream_t st);
void launch_r2_label(const uint8_t* base, uint8_t* labels, const float4* pos, int64_t np, Dims g, float dx,
                     R2Scratch& sc, cudaStream_t st);
// mode 0: u, v = P2G; mode 1: u*, v* = P2G and u, v = P2G + gravity.  Returns the number of launches.
int launch_r2_p2g(const float4* pos, const float4* vel, int64_t np, Dims g, float dx, float dt, int mode,
                   R2Scratch& sc, float* u, float* v, float* us, float* vs, cudaStream_t st);
void launch_r2_forces(float* u, float* v, Dims g, float dt, cudaStream_t st);
void launch_r2_project(float* u, float* v, const float* p, const uint8_t* labels, Dims g, float dx, float dt,
                       R2Scratch& sc, cudaStream_t st);
// flags: 1 G2P, 2 advection, 4 clean-up (sets sc.keep)
void launch_r2_particles(float4* pos, float4* vel, int64_t np, const float* u, const float* v, const float* us,
                         const float* vs, const uint8_t* labels, Dims g, float dx, float dt, float alpha, int flags,
                         R2Scratch& sc, cudaStream_t st);
// kept particles of sc.keep, in order, to pos2/vel2 (w = new index); the
// count lands in sc.keep[np].  Returns the number of launches.
int launch_r2_compact(const float4* pos, const float4* vel, int64_t np, R2Scratch& sc, float4* pos2, float4* vel2,
                       cudaStream_t st);

}  // namespace fp
