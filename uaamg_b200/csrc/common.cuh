// Shared device-side definitions of the B200 UAAMG-PCG engine.
//
// Memory layout (the reference's, include/core/mesh_3d.h:38 and mesh.h:35): every
// per-cell array of a level is ghost-padded and column-major with i fastest,
// id = i + j*(nx+2) + k*(nx+2)*(ny+2).  2D levels have no z ghosts: the interior
// is the single plane k = 0.  Ghost entries of vectors and coefficient channels
// stay 0, which is what makes Neumann walls need no special-casing in the
// V-cycle kernels.
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

namespace uaamg {

// Cell code bits (one byte a cell, vec.cuh k_codes): interior fluid cell, colour
// (i + j + k odd); on the finest level bits 0-5 mark the +x,-x,+y,-y,+z,-z
// neighbours that are interior fluid cells.
constexpr uint32_t kActive = 64u, kOdd = 128u;

struct Geom {
    int nx, ny, nz;  // interior cells; nz == 0 for a 2D level
    int sx, sxy;     // strides in cells: sx = nx+2, sxy = (nx+2)(ny+2)
    int n;           // padded cell count
};

// The reference's layout: row pitch nx+2.
inline Geom make_geom(int dim, int nx, int ny, int nz) {
    Geom g;
    g.nx = nx; g.ny = ny; g.nz = dim == 3 ? nz : 0;
    g.sx = nx + 2;
    g.sxy = (nx + 2) * (ny + 2);
    g.n = dim == 3 ? g.sxy * (nz + 2) : g.sxy;
    return g;
}

// The engines' internal layout: the same ghost-padded i-fastest order with the row
// pitch rounded up to a multiple of 16 cells, so every row of every array starts
// on a 16-byte boundary (a tensor-map requirement for TMA, and 128-bit loads).
// Columns nx+2 .. sx-1 are padding and stay 0.
constexpr int kPitchAlign = 16;
inline Geom make_geom_pitched(int dim, int nx, int ny, int nz) {
    Geom g = make_geom(dim, nx, ny, nz);
    g.sx = (nx + 2 + kPitchAlign - 1) / kPitchAlign * kPitchAlign;
    g.sxy = g.sx * (ny + 2);
    g.n = dim == 3 ? g.sxy * (nz + 2) : g.sxy;
    return g;
}

// Run status written by the device-side finalisers (CGState::status).
enum : int {
    CG_RUNNING = 0,
    CG_CONVERGED = 1,
    CG_MAXITER = 2,
    CG_BREAKDOWN = 3,
    CG_NAN = 4,
    CG_DIVERGED = 5,  // covering aggregates only: the solve is repeated on the reference's
};

// Device-resident PCG state.  All scalars are FP64; the loop never copies a
// scalar to the host: alpha/beta/stopping decisions are taken by the last block
// of the kernel that finishes each reduction.
struct CGState {
    double rz_old;     // r.z of the previous iteration
    double pap;        // p.Ap
    double alpha, beta;
    double rr;         // recursive r.r
    double rr_true;    // FP64 true residual b - A x (residual replacement / exit)
    double r0;         // ||r0||
    double tol_abs;    // stop when sqrt(r.r) < tol_abs
    double mean_z;     // fluid mean of z (null-space projection)
    double nfluid;     // fluid cell count
    double sum0, sum1; // right-hand side: sum over the fluid cells, sum after the first
                       // projection; sum0 also of the result's mean projection
    double bnorm;      // ||b|| of the normalised right-hand side
    double breakdown;  // p.Ap below this stops the solve (the reference's 1e-15)
    double rr_best;    // the least rr of the solve's iterations
    double rz0, rz_peak;  // rz_old of its first one, the largest rz_old so far
    int done;          // 1 once the solve stopped; every loop kernel then returns at once
    int status;        // CG_* above
    int iter;          // completed x/r updates
    int cand;          // mixed mode: recursive residual met tol, confirm with the true one
    int max_iter;
    int replace_every; // mixed mode residual-replacement period (0 = off)
    int replacements;  // replacements performed
    int dirichlet;     // 1: no null space (skip mean projections)
    int init;          // 1 while forming p0 = z0 (beta = 0)
    int fold;          // mixed mode: the next x update first folds x_lo into x_hi
    unsigned int counter[8];  // last-block counters, one per reduction site
    int err;           // set by a kernel whose TMA wait gave up
    int epoch;         // number of this solve (its progress words carry it)
    int cover;         // 1: preconditioned on covering aggregates; a residual that grew ends the solve
    unsigned long long* progress;  // pinned host word: where the solve is (publish)
};

// A solve's progress word in pinned host memory: epoch, completed updates, status.  The
// host reads it instead of queueing a copy of the stop flag and an event behind every
// step (two stream operations a step, and a gap before the next step).
__host__ __device__ inline unsigned long long progress_word(int epoch, int iter, int status) {
    return ((unsigned long long)(epoch & 0xffff) << 48) | ((unsigned long long)(unsigned)iter << 3) |
           (unsigned)(status & 7);
}
__device__ __forceinline__ void publish(unsigned long long* to, int epoch, int iter, int status) {
    if (to) *(volatile unsigned long long*)to = progress_word(epoch, iter, status);
}

// Whether the residual of iteration it shows that a solve on covering aggregates runs away
// (squared norms: rr, the least so far best; rz, the preconditioner's norm r.Mr one
// iteration before, its first value rz0 and the largest so far).  A right-hand side that is inconsistent on
// separate parts of the fluid (a chamber with a net source) has no solution; the covering
// aggregates join such parts on coarse levels, and CG then runs away instead of stalling
// at the inconsistency: 1e6 times where it began (or a thousandth of ||b|| when it began
// below that) within 8 to 15 iterations.  A consistent solve also rises first when its
// right-hand side is smooth, since the 2-norm weighs the rough error that the coarse
// levels bring in: 130 times at 2048 x 1024 with scattered solids, 420 at 2000 x 6, 9400
// at 60000 x 8, falling again from the second iteration on.  Its rz does not rise, but in
// channels (from some six times as long as wide), where it falls again within four
// iterations; that of an inconsistent one rises on from the third iteration, which is what
// counts when max_iter ends a solve (last).
// With a small inconsistent share of b the residual falls to it first and rises from there
// (share 1e-4: to 1e-3 in 6 iterations, past 1 in 15).  Once it has been below half of r0,
// 1000 times the best ends the solve, 30 times at max_iter; consistent solves rise 28 times
// over their best at most there (1000 x 5 x 5; other shapes 3, few past 5).  Not below 1e-6
// r0: there a tolerance out of reach lets the rounding of a consistent right-hand side run
// away (two chambers, 1e-15 after 60 iterations and 1e-8 after 200), and the reference's
// hierarchy may not get that far in max_iter iterations at all.
__device__ __forceinline__ bool residual_grew(double rr, double best, double r0, double bnorm, double rz,
                                              double rz0, double rz_peak, int it, bool last) {
    const double f = fmax(r0, 1e-3 * bnorm);
    return rr > 1e12 * f * f ||
           (last && it > 1 && rr > 4.0 * f * f && rz > rz0 && 4.0 * rz > rz_peak) ||
           (4.0 * best < r0 * r0 && rr > 1e-12 * r0 * r0 && rr > (last ? 9e2 : 1e6) * best);
}

// q = a / d and r = a % d for 0 <= a < 2^31, 0 < d, from a reciprocal 1/d computed
// once (rd): the double-precision estimate is off by at most one and one exact
// correction step fixes it.  A fraction of the instructions of an integer division
// by a value known only at run time, which the grid-stride walks would otherwise
// pay per item.
__device__ __forceinline__ int divmod_rcp(int a, int d, double rd, int& r) {
    int q = (int)((double)a * rd);
    r = a - q * d;
    if (r < 0) { --q; r += d; }
    else if (r >= d) { ++q; r -= d; }
    return q;
}

// Programmatic dependent launch: the engine launches its kernels so that each may
// be scheduled while its predecessor on the stream is still finishing.  Every
// kernel therefore first waits until the preceding grid has completed and its
// memory operations are visible (a no-op when it was launched without the
// attribute), and then lets its own successor be launched.
__device__ __forceinline__ void pdl_entry() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
// The kernels of an iteration do what does not depend on their predecessor ahead of
// this wait: index arithmetic, tables, barriers, loads of the hierarchy's constant
// arrays, and of arrays last written two or more kernels earlier (a kernel is launched
// only after its predecessor's own wait, so everything before the predecessor is
// complete and visible).  Every path of every kernel executes the wait, also one that
// has nothing to do: its successor relies on it for the kernels further back.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
// A load that stays where it is written (the compiler may otherwise move it behind the
// test of another one, and pay their latencies in turn).
__device__ __forceinline__ int ld_now(const int* p) {
    int v;
    asm volatile("ld.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ unsigned long long* ld_now(unsigned long long* const* p) {
    unsigned long long* v;
    asm volatile("ld.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ float ld_now(const float* p) {
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ double ld_now(const double* p) {
    double v;
    asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    return v;
}

// Host-visible launch helpers ------------------------------------------------

template <int DIM>
inline dim3 cell_block() { return DIM == 3 ? dim3(32, 4, 2) : dim3(32, 8, 1); }

template <int DIM>
inline dim3 cell_grid(int nx, int ny, int nz) {
    dim3 b = cell_block<DIM>();
    return dim3((nx + b.x - 1) / b.x, (ny + b.y - 1) / b.y,
                DIM == 3 ? (nz + b.z - 1) / b.z : 1);
}

}  // namespace uaamg
