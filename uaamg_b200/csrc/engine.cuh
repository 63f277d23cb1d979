// Host orchestration of one precision mode of the B200 UAAMG-PCG engine
// (EngineT<double> = reference-exact FP64; EngineT<float> = plain FP32 or, with
// mixed = true, FP32 CG with FP64 residual replacement).  Included by exactly one
// translation unit per T, so the kernels it launches live in the same unit.
//
// Reference structure followed:
//   hierarchy   UAAMGPreconditioner3D::buildHierarchy / apply set-up
//               (uaamg_preconditioner_3d.cpp:11-32, 205-214), once per problem
//               here instead of once per apply
//   V-cycle     vCycle (uaamg_preconditioner_3d.cpp:183-196), iterative
//   PCG         PCG3D::solve (pcg_3d.cpp:18-125), every scalar device-resident
//
// Layout: every level array uses the pitched layout (common.cuh,
// make_geom_pitched); the caller's arrays use the reference layout and are
// converted on the way in (rhs, warm-start p, preconditioner input) and out.
#pragma once
#include <algorithm>
#include <cstdlib>
#include <map>
#include <mutex>
#include <new>
#include <tuple>
#include <type_traits>
#include <utility>
#include <vector>

#include "engine.h"
#include "fused.cuh"
#include "kernels.cuh"
#include "quad.cuh"
#include "tail.cuh"
#include "tma.cuh"
#include "vec.cuh"

namespace uaamg {
namespace {

// Tensor maps of one box geometry over a level: b, codes, diagonal, couplings.
struct BoxMaps {
    CUtensorMap b, code, dg, cx, cy, cz;
};

template <class T, class CS>
struct LevelBuf {
    Geom g;
    double hx, hy, hz;
    uint8_t* solid = nullptr;
    T *cx = nullptr, *cy = nullptr, *cz = nullptr, *wd = nullptr, *dg = nullptr;
    CS *hcx = nullptr, *hcy = nullptr, *hcz = nullptr;  // couplings as the marches read them
    T *x = nullptr, *b = nullptr;  // level >= 1 only (level 0 uses the CG's r and z)
    uint8_t* code = nullptr;       // cell codes (vec.cuh k_codes)
    int zc = 2, zu = 2;            // planes per block of the z marches, way down and up
    // FP32 couplings on a level of a mixed engine whose face counts exceed 2048 (3D
    // levels 6 and down, 2D levels 12 and down): FP16 holds integers exactly only up
    // to 2048 and overflows above 65504
    bool c32 = false;
    // plane-box tensor maps of the marches: b, x, codes, couplings, diagonal, and x
    // as the parent box read by the next-finer level's prolongation
    CUtensorMap mb, mx, mcode, mcx, mcy, mcz, mdg, mxq;
    // boxes for the fused marches (fused.cuh) with a 2-cell ring (f) and, for the way down
    // with STAR transfers, a 3-cell ring (fd); this level's x and codes as their parent
    // boxes with STAR
    BoxMaps f, fd;
    CUtensorMap mxs, mps;
    // small 3D levels: whole-tile boxes (fused.cuh k_level_box), likewise; this level's x
    // as their parent box (bxq; STAR: x and codes bxs, bps)
    bool box = false;
    BoxMaps bx, bd;
    CUtensorMap bxq, bxs, bps;
    T* trim = nullptr;  // coarse box levels: per box {d, c_x, c_y, c_z} or d = 0 (k_box_trim)
};

// 3D levels of at most this many cells run the fused steps as whole-tile boxes
// (UAAMG_BOX_MAX_CELLS overrides it, for comparisons)
constexpr double kBoxCells = 64.0 * 64.0 * 64.0;

// Kernel classes for the in-situ per-kernel timing (uaamg_profile_solve).
enum KClass : int {
    K_SWEEP = 0, K_RESTRICT, K_PROLONG, K_COARSEST, K_PMATVEC, K_UPDATE, K_ZDOT, K_FWD, K_RES,
    K_UPE, K_UPO, K_TRUE_RESIDUAL, K_RHS, K_OUTPUT, K_CAST, K_SETUP, K_TAIL, K_REPLACE, K_DOWN,
    K_UP, K_NCLASS
};
static const char* const kclass_names[K_NCLASS] = {
    "rbgs_sweep", "restrict_residual", "prolong_add", "coarsest_solve", "p_matvec_dot",
    "cg_update", "z_dot", "smooth_fwd", "residual_restrict", "prolong_smooth_even",
    "smooth_odd", "true_residual", "rhs_prepare", "output", "cast", "hierarchy_setup",
    "small_levels", "residual_replacement", "level_down", "level_up"};

struct KTag {
    int cls;
    int level;
    double bytes;  // algorithmic (compulsory) bytes of this launch (K_REPLACE: of one
                   // launch that performs the replacement; most launches return at once)
};

// Kernel launch on the engine's stream.  Outside the per-kernel profiler every
// launch on a created stream (the CUDA-graph captures always use one) carries the
// programmatic-stream-serialisation attribute (the kernels begin with pdl_entry,
// common.cuh), so a kernel's launch and block scheduling overlap the end of the one
// before it; launches on the legacy default stream are plain.
#define UAAMG_LAUNCH_SMEM(tag, kern, grid, block, smem, ...)              \
    do {                                                                  \
        const KTag tg_ = (tag);                                           \
        cudaEvent_t e0_ = nullptr, e1_ = nullptr;                         \
        if (prof_on_) prof_begin(tg_, &e0_, &e1_);                        \
        if (pdl_ && !nopdl_next_ && !prof_on_ && st_ != nullptr) {        \
            cudaLaunchConfig_t cf_ = {};                                  \
            cudaLaunchAttribute at_[1];                                   \
            at_[0].id = cudaLaunchAttributeProgrammaticStreamSerialization; \
            at_[0].val.programmaticStreamSerializationAllowed = 1;        \
            cf_.gridDim = dim3(grid);                                     \
            cf_.blockDim = dim3(block);                                   \
            cf_.dynamicSmemBytes = (smem);                                \
            cf_.stream = st_;                                             \
            cf_.attrs = at_;                                              \
            cf_.numAttrs = 1;                                             \
            cudaLaunchKernelEx(&cf_, kern, __VA_ARGS__);                  \
        } else {                                                          \
            kern<<<(grid), (block), (smem), st_>>>(__VA_ARGS__);          \
        }                                                                 \
        if (prof_on_) cudaEventRecord(e1_, st_);                          \
        nopdl_next_ = false;                                              \
        ++launches_;                                                      \
    } while (0)
#define UAAMG_LAUNCH(tag, kern, grid, block, ...) \
    UAAMG_LAUNCH_SMEM(tag, kern, grid, block, 0, __VA_ARGS__)

// CS: storage type of the coarse-level couplings the marches read (T, or __half
// in the mixed form: face counts with a per-axis scale).
template <class T, class CS = T>
class EngineT final : public Engine {
    static constexpr bool kHalf = !std::is_same<CS, T>::value;

public:
    // cover: the hierarchy of a solve (covering aggregates, see build); apply_only: the
    // engine only applies its V-cycle and reports its levels (no CG buffers).
    explicit EngineT(bool mixed, bool cover = false, bool apply_only = false)
        : mixed_(mixed), cover_(cover), apply_only_(apply_only) {
        // UAAMG_NO_PDL=1 launches every kernel without the programmatic-dependent-launch
        // attribute (fully serialised on the stream), for comparisons
        const char* v = std::getenv("UAAMG_NO_PDL");
        pdl_ = !(v && v[0] == '1');
        const char* pv = std::getenv("UAAMG_PMV2D_PER_SM");
        if (pv && pv[0]) pmv2d_env_ = std::max(1, std::atoi(pv));
        const char* bc = std::getenv("UAAMG_BOX_MAX_CELLS");
        if (bc && bc[0]) box_cells_ = std::atof(bc);
        // UAAMG_NO_TRIM=1: coarse boxes always load their diagonals and couplings
        const char* nt = std::getenv("UAAMG_NO_TRIM");
        trim_ = !(nt && nt[0] == '1');
    }
    ~EngineT() override {
        delete fb_;
        release();
        if (cap_) cudaStreamDestroy(cap_);
    }

    // A new problem.  All device buffers of a problem live in one block of memory, kept
    // while the next problem needs about as much: a mask change on the same grid -- moving
    // solids -- allocates nothing, and keeps the captured step too, whose kernels see the
    // same addresses and sizes.
    int set_problem(int dim, int nx, int ny, int nz, double dx, double dy, double dz,
                    const uint8_t* d_solid, int dirichlet) override {
        plain_ = false;
        return set_problem_now(dim, nx, ny, nz, dx, dy, dz, d_solid, dirichlet);
    }
    int set_problem_now(int dim, int nx, int ny, int nz, double dx, double dy, double dz,
                        const uint8_t* d_solid, int dirichlet) {
        delete fb_;
        fb_ = nullptr;
        fb_on_ = false;
        release(true);
        if (dim != 2 && dim != 3) { release(); return E_ARG; }
        if (nx < 2 || ny < 2 || (dim == 3 && nz < 2)) { release(); return E_ARG; }
        dim_ = dim; dirichlet_ = dirichlet;
        dx_ = dx; dy_ = dy; dz_ = dim == 3 ? dz : 1.0;
        int e = dim == 3 ? build<3>(nx, ny, nz, d_solid) : build<2>(nx, ny, nz, d_solid);
        if (e != E_OK) { release(); return e; }
        std::vector<double> sig = graph_signature();
        if (sig != gsig_) {
            drop_graph();
            gsig_ = std::move(sig);
        }
        return E_OK;
    }

    int precond_apply(const double* d_r, double* d_z) override {
        if (lv_.empty()) return E_NOPROB;
        launches_ = 0;
        cudaMemsetAsync(err_, 0, sizeof(int), st_);
        err_known_ = false;
        if (dim_ == 3) precond_impl<3>(d_r, d_z); else precond_impl<2>(d_r, d_z);
        return sync_check();
    }

    int solve_begin(const SolveArgs& a) override {
        if (lv_.empty() || apply_only_) return E_NOPROB;
        launches_ = 0;
        fb_on_ = false;
        return dim_ == 3 ? begin_impl<3>(a) : begin_impl<2>(a);
    }

    int solve_step() override {
        if (fb_on_) return fb_->solve_step();
        if (stopped_) return E_OK;
        return dim_ == 3 ? step_impl<3>() : step_impl<2>();
    }

    // The progress word (common.cuh) says how many updates are done and whether the device
    // has stopped; a step is seen once its second update is.  Now and then the stream is
    // asked too: a failed launch ends in E_CUDA, and steps that ran without advancing the
    // word (a kernel gave up on its loads) count as seen, so that max_iter ends the solve.
    int solve_poll(bool wait, bool* stopped) override {
        if (fb_on_) return fb_->solve_poll(wait, stopped);
        while (!stopped_ && seen_ < nstep_) {
            const unsigned long long w = *(volatile unsigned long long*)flag_host_;
            if ((w >> 48) == (unsigned long long)(epoch_ & 0xffff)) {
                if (w & 7) {
                    stopped_ = true;
                    if ((w & 7) == CG_DIVERGED) return fall_back(stopped);
                    break;
                }
                if ((long long)((w & 0xffffffffffffull) >> 3) >= 2LL * (seen_ + 1)) { ++seen_; continue; }
            }
            if ((++polls_ & 0xffff) == 0) {
                const cudaError_t q = cudaStreamQuery(st_);
                if (q == cudaSuccess && w == *(volatile unsigned long long*)flag_host_) {
                    seen_ = nstep_;
                    break;
                }
                if (q != cudaSuccess && q != cudaErrorNotReady) return E_CUDA;
            }
            if (!wait) break;
        }
        if (!stopped_ && seen_ == nstep_ && it_ >= cur_.max_iter) stopped_ = true;
        *stopped = stopped_;
        return E_OK;
    }

    // Steps queued but not yet seen by solve_poll (at most two are useful).
    int solve_inflight() const override { return fb_on_ ? fb_->solve_inflight() : nstep_ - seen_; }

    int solve_end(SolveResult* res) override {
        int e = solve_end_enqueue();
        return e != E_OK ? e : solve_end_collect(res);
    }

    int solve_end_enqueue() override {
        if (fb_on_) return fb_->solve_end_enqueue();
        return dim_ == 3 ? end_enqueue<3>() : end_enqueue<2>();
    }

    int enqueue_step(cudaStream_t s, int* flag_dst) override {
        if (lv_.empty()) return E_NOPROB;
        const cudaStream_t saved = st_;
        st_ = s;
        if (dim_ == 3) {
            cg_iteration<3>(true);
            cg_iteration<3>(false);
        } else {
            cg_iteration<2>(true);
            cg_iteration<2>(false);
        }
        if (flag_dst) cudaMemcpyAsync(flag_dst, &cg_->done, sizeof(int), cudaMemcpyDeviceToHost, st_);
        st_ = saved;
        return E_OK;
    }

    int steps_done(bool* stopped) override {
        const unsigned long long w = *(volatile unsigned long long*)flag_host_;
        *stopped = true;
        if ((w >> 48) != (unsigned long long)(epoch_ & 0xffff) || (w & 7) != CG_DIVERGED) return E_OK;
        return fall_back(stopped);
    }

    int solve_end_collect(SolveResult* res) override {
        if (fb_on_) {
            const int e = fb_->solve_end_collect(res);
            cuda_error = fb_->cuda_error;
            return e;
        }
        int e = sync_check();
        if (e != E_OK) return e;
        const CGState& c = *cg_host_;
        err_known_ = true;
        res->status = c.status;
        res->iterations = c.iter;
        res->replacements = c.replacements;
        res->rr = c.rr;
        res->rr_true = c.rr_true;
        res->bnorm = c.bnorm;
        res->r0 = c.r0;
        res->tol_abs = c.tol_abs;
        return E_OK;
    }

    // The whole solve: the host keeps two steps queued and polls one behind, so it
    // never idles the GPU waiting for a scalar.
    int solve(const SolveArgs& a, SolveResult* res) override {
        int e = solve_begin(a);
        if (e != E_OK) return e;
        bool stopped = false;
        while (!stopped) {
            if ((e = solve_step()) != E_OK) return e;
            if ((e = solve_poll(solve_inflight() >= 2 || queued_all(), &stopped)) != E_OK) return e;
        }
        return solve_end(res);
    }

    int nlevels() const override { return (int)lv_.size(); }

    void level_dims(int l, int* nx, int* ny, int* nz) const override {
        *nx = lv_[l].g.nx; *ny = lv_[l].g.ny; *nz = lv_[l].g.nz;
    }

    int level_trim(int l, int* boxes, int* trimmed) override {
        if (l < 0 || l >= (int)lv_.size()) return E_ARG;
        const LevelBuf<T, CS>& L = lv_[l];
        *boxes = *trimmed = 0;
        if (!L.box) return E_OK;
        const dim3 bg = box_grid(L.g);
        *boxes = (int)(bg.x * bg.y * bg.z);
        if (!L.trim || !trim_) return E_OK;
        std::vector<T> rec((size_t)4 * *boxes);
        if (cudaMemcpy(rec.data(), L.trim, rec.size() * sizeof(T), cudaMemcpyDeviceToHost) !=
            cudaSuccess)
            return E_CUDA;
        for (int b = 0; b < *boxes; ++b) *trimmed += rec[(size_t)4 * b] != T(0);
        return E_OK;
    }

    // Host copies in the reference layout of level l (row pitch nx_l + 2).
    int copy_level(int l, uint8_t* solid, double* cx, double* cy, double* cz) override {
        if (l < 0 || l >= (int)lv_.size()) return E_ARG;
        const LevelBuf<T, CS>& L = lv_[l];
        const Geom g = L.g;
        const Geom gr = make_geom(dim_, g.nx, g.ny, g.nz);
        if (cudaStreamSynchronize(st_) != cudaSuccess) return E_CUDA;
        const int nzi = dim_ == 3 ? g.nz + 2 : 1;
        auto depitch = [&](auto* dst, const auto* src) {
            for (int k = 0; k < nzi; ++k)
                for (int j = 0; j < g.ny + 2; ++j)
                    for (int i = 0; i < g.nx + 2; ++i)
                        dst[i + j * gr.sx + k * gr.sxy] = src[i + j * g.sx + k * g.sxy];
        };
        if (solid) {
            std::vector<uint8_t> tmp(g.n);
            if (cudaMemcpy(tmp.data(), L.solid, g.n, cudaMemcpyDeviceToHost) != cudaSuccess)
                return E_CUDA;
            depitch(solid, tmp.data());
        }
        std::vector<T> tmp(g.n);
        std::vector<double> tmpd(g.n);
        const T* src[3] = {L.cx, L.cy, L.cz};
        double* dst[3] = {cx, cy, cz};
        for (int q = 0; q < 3; ++q) {
            if (!dst[q]) continue;
            if (!src[q]) { for (int c = 0; c < gr.n; ++c) dst[q][c] = 0.0; continue; }
            if (cudaMemcpy(tmp.data(), src[q], g.n * sizeof(T), cudaMemcpyDeviceToHost) != cudaSuccess)
                return E_CUDA;
            for (int c = 0; c < g.n; ++c) tmpd[c] = (double)tmp[c];
            depitch(dst[q], tmpd.data());
        }
        return E_OK;
    }

    void set_stream(cudaStream_t s) override {
        st_ = s;
        if (fb_) fb_->st_ = s;  // (its next use may be its release)
    }
    size_t device_bytes() const override { return bytes_ + (fb_ ? fb_->device_bytes() : 0); }
    long launches() const override { return launches_ + (fb_on_ ? fb_->launches() : 0); }
    void set_vcycle_sweeps(bool on) override { sweeps_ = on; }
    void set_graphs(bool on) override { graphs_ = on; }
    void set_autotune(bool on) override { autotune_ = on; }
    void set_small_levels(bool on) override { tail_on_ = on; }
    void set_smoothing(int fine, int coarse) override {
        if (fine == nu_fine_ && coarse == nu_coarse_) return;
        drop_graph();
        nu_fine_ = fine;
        nu_coarse_ = coarse;
    }
    void set_fused(bool on) override {
        if (on == fused_) return;
        drop_graph();
        fused_ = on;
    }
    void set_operator(const double* d, const double* ox, const double* oy, int sx,
                      long version) override {
        vver_ = version;
        if (d == vd_ && ox == vox_ && oy == voy_ && sx == vsx_) return;
        // a captured step holds the operator's pointers: capture again
        if (gexec_) {
            cudaStreamSynchronize(st_);
            cudaGraphExecDestroy(gexec_);
            gexec_ = nullptr;
        }
        gkey_ = -1;
        vd_ = d; vox_ = ox; voy_ = oy; vsx_ = sx;
    }

    void set_profiling(bool on) override {
        prof_on_ = on;
        prof_count_ = 0;
    }

    int profile_results(std::vector<KernelTime>& out) override {
        out.clear();
        if (cudaStreamSynchronize(st_) != cudaSuccess) return E_CUDA;
        for (int q = 0; q < prof_count_; ++q) {
            float ms = 0.f;
            if (cudaEventElapsedTime(&ms, prof_ev_[q].first, prof_ev_[q].second) != cudaSuccess)
                return E_CUDA;
            const KTag& t = prof_tag_[q];
            KernelTime* slot = nullptr;
            for (auto& kt : out)
                if (kt.cls == t.cls && kt.level == t.level) { slot = &kt; break; }
            if (!slot) {
                KernelTime kt;
                kt.cls = t.cls;
                kt.name = kclass_names[t.cls];
                kt.level = t.level;
                kt.launches = 0;
                kt.total_ms = 0.0;
                kt.bytes = t.bytes;
                out.push_back(kt);
                slot = &out.back();
            }
            slot->launches += 1;
            slot->total_ms += ms;
        }
        // the residual replacement kernel runs every iteration but works only when a
        // replacement is due: its bytes per launch are those of the replacements
        // performed, spread over all its launches
        for (auto& kt : out)
            if (kt.cls == K_REPLACE && kt.launches > 0)
                kt.bytes = kt.bytes * (double)cg_host_->replacements / (double)kt.launches;
        return E_OK;
    }

    int timed_out() override {
        if (fb_on_) return fb_->timed_out();
        int v = 0;
        if (!err_) return 0;
        if (err_known_) return cg_host_->err;  // a finished solve: copied with its state
        if (cudaMemcpy(&v, err_, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return 0;
        return v;
    }

private:
    bool queued_all() const { return fb_on_ ? fb_->queued_all() : it_ >= cur_.max_iter; }

    // The residual of a solve on covering aggregates grew (common.cuh, residual_grew): the
    // same solve from its beginning on the reference's hierarchy, by an engine of its own
    // (made here, kept while the mask stays); the stages then go to it.  Without room for
    // one, this engine takes the reference's hierarchy until the next mask (its buffers are
    // no larger).  Nothing has been added to the caller's x yet.
    int fall_back(bool* stopped) {
        *stopped = true;
        if (!cur_.ref_solid) return E_OK;
        const Geom g = lv_[0].g;
        const SolveArgs a = cur_;
        int e = E_OK;
        if (!fb_) {
            fb_ = new (std::nothrow) EngineT<T, CS>(mixed_);
            if (fb_) fb_->st_ = st_;
            e = fb_ ? fb_->set_problem(dim_, g.nx, g.ny, g.nz, dx_, dy_, dz_, a.ref_solid, dirichlet_) : E_OOM;
        }
        if (e == E_OK) {
            fb_->st_ = st_;
            fb_->set_vcycle_sweeps(sweeps_);
            fb_->set_small_levels(tail_on_);
            fb_->set_fused(fused_);
            fb_->set_graphs(graphs_);
            fb_->set_operator(vd_, vox_, voy_, vsx_, vver_);
            fb_->set_smoothing(nu_fine_, nu_coarse_);
            fb_->prof_on_ = false;
            e = fb_->solve_begin(a);
            if (e == E_OK) {
                fb_on_ = true;
                *stopped = false;
                return E_OK;
            }
        }
        if (e != E_OOM) {
            cuda_error = fb_->cuda_error;
            delete fb_;  // (its set-up failed: nothing to keep)
            fb_ = nullptr;
            return e;
        }
        const long before = launches_;
        plain_ = true;
        e = set_problem_now(dim_, g.nx, g.ny, g.nz, dx_, dy_, dz_, a.ref_solid, dirichlet_);
        if (e == E_OK) e = solve_begin(a);
        launches_ += before;
        if (e == E_OK) *stopped = false;
        return e;
    }

    EngineT<T, CS>* fb_ = nullptr;
    bool fb_on_ = false;
    bool mixed_;
    bool cover_ = false, apply_only_ = false;
    bool plain_ = false;  // this mask on the reference's hierarchy (fall_back without room)
    bool star_ = false;  // the current hierarchy covers and its transfers reach face neighbours
    int dim_ = 0, dirichlet_ = 0;
    double dx_ = 1, dy_ = 1, dz_ = 1;
    Geom gref_;                      // the caller's (reference) layout of level 0
    std::vector<LevelBuf<T, CS>> lv_;
    T *r_ = nullptr, *z_ = nullptr, *p_ = nullptr, *p2_ = nullptr, *ap_ = nullptr, *xlo_ = nullptr;
    // variable-coefficient operator (set_operator); not owned
    const double *vd_ = nullptr, *vox_ = nullptr, *voy_ = nullptr;
    int vsx_ = 0;
    long vver_ = 0, vconv_ = -1;     // contents version set / converted into vf_
    float* vf_[3] = {nullptr, nullptr, nullptr};  // FP32 forms: s, ox, oy (level layout)
    double *b64_ = nullptr, *xd_ = nullptr, *partials_ = nullptr;
    int* err_ = nullptr;             // cg_'s error word, set by a kernel whose TMA wait gave up
    bool err_known_ = false;         // cg_host_ holds it
    CUtensorMap map_p_, map_p2_;     // plane boxes of the two search-direction buffers
    CUtensorMap map_b64_, map_xd_, map_xlo_;  // plane boxes of b, x_hi (FP64) and x_lo (3D)
    SolveArgs cur_{};                // the solve in progress
    bool use_graph_ = false;
    int it_ = 0;                     // iterations queued
    int nstep_ = 0, seen_ = 0;       // steps queued / steps whose flag was read
    bool stopped_ = false;
    long long reduce_blocks_ = 0;    // partials_ capacity in blocks (4 doubles each)
    CGState* cg_ = nullptr;
    CGState* cg_host_ = nullptr;  // pinned
    unsigned long long* flag_host_ = nullptr;  // pinned: the progress word
    int epoch_ = 0;               // solves begun
    unsigned polls_ = 0;
    cudaStream_t st_ = 0;
    unsigned char* arena_ = nullptr;  // one block for all buffers of a problem
    size_t arena_cap_ = 0, arena_used_ = 0;
    bool arena_dry_ = false;          // alloc only adds up the sizes
    std::vector<void*> extra_;        // buffers made after set_problem (vf_)
    std::vector<double> gsig_;        // what the captured step's arguments depend on
    size_t bytes_ = 0;
    long launches_ = 0;
    int num_sms_ = 148;
    bool sweeps_ = false;  // V-cycle as per-colour sweeps (cross-check) instead of the marches
    bool graphs_ = true;   // replay the PCG step as a CUDA graph
    bool autotune_ = false;  // time the marches' z-chunk lengths at set-up
    bool tail_on_ = true;    // small levels in one one-block kernel (tail.cuh)
    bool fused_ = true;      // two fused marches a level (fused.cuh) instead of four
    double box_cells_ = kBoxCells;
    // blocks per SM of the 2D search direction: as many as are resident at once (one
    // wave: a second, partial wave left SMs idle at its end); UAAMG_PMV2D_PER_SM overrides
    int pmv2d_per_sm_ = 8;
    int pm_zc_ = 2;   // planes per block of the 3D search direction (k_pmatvec)
    int zdot_zc_ = 2;  // FP64, 3D: of the z sums' partition (k_zdot_tiles)
    int rx_zc_ = 16;  // planes per block of the 3D replacement march (k_resid_march)
    int pmv2d_env_ = 0;
    int resid_per_sm_ = 8;  // the FP64 residual walk: resident blocks per SM (one wave)
    bool trim_ = true;       // trimmed coarse boxes (fused.cuh k_box_trim)
    bool pdl_ = true;        // programmatic dependent launch between the kernels
    bool nopdl_next_ = false;  // the next launch is plain (a kernel that usually exits at
                               // once: its blocks should not wait resident for their turn)
    int nu_fine_ = 1, nu_coarse_ = 1;  // pre- and post-smoothing sweeps: finest / coarse levels
    int tail_lt_ = 0;        // first level of the small-level kernel
    int tail_nc_ = 0;        // 1: the hierarchy has a tail (0: it does not fit the kernel)
    T* dense_ = nullptr;      // the tail's cycle as a matrix (n rows, stride ld)
    int* dense_cell_ = nullptr;
    int dense_n_ = 0, dense_ld_ = 0, dense_cells_ = 0;  // rows in use, stride, rows planned
    size_t tail_smem_ = 0;   // its dynamic shared memory (x and b of every tail level)
    cudaStream_t cap_ = nullptr;      // capture stream
    cudaGraphExec_t gexec_ = nullptr; // two PCG iterations
    long long gkey_ = -1;
    const double* ghist_ = nullptr;
    long glaunches_ = 0;              // kernels in one graph replay
    // in-situ per-launch timing (set_profiling)
    bool prof_on_ = false;
    int prof_count_ = 0;
    std::vector<std::pair<cudaEvent_t, cudaEvent_t>> prof_ev_;
    std::vector<KTag> prof_tag_;

    int max_reduce_blocks() const { return 4 * num_sms_; }

    // Blocks of the CG update: one vector a thread on small grids (idle blocks only
    // lengthen the reduction's end); FP64 keeps its partition of r.r.
    unsigned update_blocks(long long nvec) const {
        if (sizeof(T) == 8) return (unsigned)max_reduce_blocks();
        return (unsigned)std::max<long long>(1, std::min<long long>(max_reduce_blocks(), (nvec + 255) / 256));
    }

    void drop_graph() {
        if (gexec_) {
            cudaStreamSynchronize(st_);
            cudaGraphExecDestroy(gexec_);
            gexec_ = nullptr;
        }
        gkey_ = -1;
    }

    // grid of the 2D search-direction kernel (kernels.cuh k_pmatvec_2d): 32 column
    // pairs of two rows a warp, eight warps a block, up to 8 blocks per SM (within
    // the partials' capacity)
    dim3 flat2d_grid(const Geom& g) const {
        const long long items = (long long)((g.ny + 1) / 2) * ((g.nx + 31) / 32);
        long long nb = std::min<long long>((items + 7) / 8, (long long)pmv2d_per_sm_ * num_sms_);
        nb = std::min<long long>(nb, reduce_blocks_);
        return dim3((unsigned)(nb < 1 ? 1 : nb));
    }

    // grid of the FP64 residual column walk (kernels.cuh k_resid_x64): tiles of
    // 32 x 8 columns and kResidZc planes, at most 8 blocks of 256 threads per SM
    static constexpr int kResidZc = 16;
    dim3 resid_grid(const Geom& g) const {
        const long long tiles = (long long)((g.nx + 31) / 32) * ((g.ny + 7) / 8) *
                                (g.nz ? (g.nz + kResidZc - 1) / kResidZc : 1);
        return dim3((unsigned)std::min<long long>(tiles, (long long)resid_per_sm_ * num_sms_));
    }

    // grid of the row-walk kernels (kernels.cuh for_cells): capped at 4 blocks per SM
    dim3 vec_grid(const Geom& g) const {
        const long long items = (long long)g.ny * (g.nz ? g.nz : 1) * ((g.nx + 31) / 32);
        long long nb = (items + 7) / 8;
        if (nb > max_reduce_blocks()) nb = max_reduce_blocks();
        return dim3((unsigned)(nb < 1 ? 1 : nb));
    }

    void prof_begin(const KTag& t, cudaEvent_t* e0, cudaEvent_t* e1) {
        if (prof_count_ == (int)prof_ev_.size()) {
            cudaEvent_t a = nullptr, b = nullptr;
            cudaEventCreate(&a);
            cudaEventCreate(&b);
            prof_ev_.push_back({a, b});
            prof_tag_.push_back(t);
        }
        prof_tag_[prof_count_] = t;
        *e0 = prof_ev_[prof_count_].first;
        *e1 = prof_ev_[prof_count_].second;
        ++prof_count_;
        cudaEventRecord(*e0, st_);
    }

    static double cells(const Geom& g) {
        return (double)g.nx * g.ny * (g.nz ? g.nz : 1);
    }

    // The next count elements of the problem's block (zeroed by arena_ready).
    template <class P>
    int alloc(P*& p, size_t count) {
        const size_t nb = (count * sizeof(P) + 255) / 256 * 256;
        if (!arena_dry_) {
            if (arena_used_ + nb > arena_cap_) return E_OOM;
            p = reinterpret_cast<P*>(arena_ + arena_used_);
        }
        arena_used_ += nb;
        return E_OK;
    }

    // After a dry pass of the alloc calls: a zeroed block of at least that size, the
    // present one unless it is too small or more than a quarter too large.
    int arena_ready() {
        const size_t need = arena_used_;
        arena_dry_ = false;
        arena_used_ = 0;
        if (!arena_ || arena_cap_ < need || arena_cap_ > need + need / 4) {
            if (arena_) cudaFree(arena_);
            arena_ = nullptr;
            arena_cap_ = 0;
            void* q = nullptr;
            if (cudaMalloc(&q, need) != cudaSuccess) {
                cudaGetLastError();
                return E_OOM;
            }
            arena_ = static_cast<unsigned char*>(q);
            arena_cap_ = need;
        }
        bytes_ = arena_cap_;
        return cudaMemsetAsync(arena_, 0, need, st_) == cudaSuccess ? E_OK : E_CUDA;
    }

    // A zeroed buffer of its own, freed with the problem.
    template <class P>
    int alloc_extra(P*& p, size_t count) {
        void* q = nullptr;
        if (cudaMalloc(&q, count * sizeof(P)) != cudaSuccess) {
            cudaGetLastError();
            return E_OOM;
        }
        extra_.push_back(q);
        bytes_ += count * sizeof(P);
        if (cudaMemsetAsync(q, 0, count * sizeof(P), st_) != cudaSuccess) return E_CUDA;
        p = static_cast<P*>(q);
        return E_OK;
    }

    // Every value that a captured step's launches take from the problem, beside what
    // drops the graph by itself (operator, smoothing, V-cycle kernels, history buffer).
    std::vector<double> graph_signature() const {
        const Geom& g = lv_[0].g;
        std::vector<double> v = {(double)dim_, (double)g.nx, (double)g.ny, (double)g.nz, dx_, dy_, dz_,
                                 (double)dirichlet_, (double)(uintptr_t)arena_, (double)arena_used_,
                                 (double)pm_zc_, (double)zdot_zc_, (double)rx_zc_, (double)pmv2d_per_sm_,
                                 (double)resid_per_sm_, (double)tail_lt_, (double)tail_nc_,
                                 (double)dense_n_, (double)star_};
        for (const auto& L : lv_) {
            v.push_back(L.zc);
            v.push_back(L.zu);
        }
        return v;
    }

    // keep: the buffers' block, the captured step and the pinned host words stay
    // (set_problem).
    void release(bool keep = false) {
        if (arena_ || cg_host_) cudaStreamSynchronize(st_);
        for (void* q : extra_) cudaFree(q);
        extra_.clear();
        if (!keep && arena_) {
            cudaFree(arena_);
            arena_ = nullptr;
            arena_cap_ = 0;
        }
        arena_used_ = 0;
        lv_.clear();
        bytes_ = 0;
        r_ = z_ = p_ = p2_ = ap_ = xlo_ = nullptr;
        b64_ = xd_ = partials_ = nullptr;
        vf_[0] = vf_[1] = vf_[2] = nullptr;
        dense_ = nullptr;
        dense_cell_ = nullptr;
        dense_n_ = 0;
        vconv_ = -1;
        err_ = nullptr;
        cg_ = nullptr;
        for (auto& pr : prof_ev_) { cudaEventDestroy(pr.first); cudaEventDestroy(pr.second); }
        prof_ev_.clear();
        prof_tag_.clear();
        prof_count_ = 0;
        if (keep) return;
        if (cg_host_) { cudaFreeHost(cg_host_); cg_host_ = nullptr; }
        if (flag_host_) { cudaFreeHost(flag_host_); flag_host_ = nullptr; }
        if (gexec_) { cudaGraphExecDestroy(gexec_); gexec_ = nullptr; }
        gkey_ = -1;
        gsig_.clear();
        ghist_ = nullptr;
    }

    int sync_check() {
        cudaError_t e = cudaGetLastError();
        const cudaError_t es = cudaStreamSynchronize(st_);
        if (e == cudaSuccess) e = es;
        if (e == cudaSuccess) e = cudaGetLastError();
        if (e != cudaSuccess) cuda_error = e;
        return e == cudaSuccess ? E_OK : E_CUDA;
    }

    // Blocks of a march over level g: 32 x 8 column tiles, z chunks of zc planes.
    template <int DIM>
    static dim3 march_grid(const Geom& g, int zc) {
        return dim3((unsigned)((g.nx + kMX - 1) / kMX), (unsigned)((g.ny + kMY - 1) / kMY),
                    DIM == 3 ? (unsigned)((g.nz + zc - 1) / zc) : 1u);
    }

    // The tensor maps of level l's b (given), codes, diagonal and couplings with the boxes
    // BT (T), BC (codes), BS (CS couplings) and BF (FP32 couplings), bz planes deep.
    template <class B> static constexpr int box_rows(const B*) { return B::H; }
    template <class E, int R> static constexpr int box_rows(const BBox<E, R>*) { return BBox<E, R>::N; }
    template <int DIM, class BT, class BC, class BS, class BF>
    bool box_maps(const LevelBuf<T, CS>& L, const T* b, int l, int bz, BoxMaps* m) const {
        constexpr int H = box_rows((const BT*)nullptr);
        bool ok = encode_level_map<T>(&m->b, b, L.g, DIM, BT::W, H, bz) &&
                  encode_level_map<uint8_t>(&m->code, L.code, L.g, DIM, BC::W, H, bz);
        if (l == 0) return ok;
        ok = ok && encode_level_map<T>(&m->dg, L.dg, L.g, DIM, BT::W, H, bz);
        if (L.c32)
            return ok && encode_level_map<T>(&m->cx, L.cx, L.g, DIM, BF::W, H, bz) &&
                   encode_level_map<T>(&m->cy, L.cy, L.g, DIM, BF::W, H, bz) &&
                   (DIM == 2 || encode_level_map<T>(&m->cz, L.cz, L.g, DIM, BF::W, H, bz));
        return ok && encode_level_map<CS>(&m->cx, L.hcx, L.g, DIM, BS::W, H, bz) &&
               encode_level_map<CS>(&m->cy, L.hcy, L.g, DIM, BS::W, H, bz) &&
               (DIM == 2 || encode_level_map<CS>(&m->cz, L.hcz, L.g, DIM, BS::W, H, bz));
    }

    // Blocks of the whole-tile box kernels over level g: 8^3 tiles.
    static dim3 box_grid(const Geom& g) {
        return dim3((unsigned)((g.nx + kBT - 1) / kBT), (unsigned)((g.ny + kBT - 1) / kBT),
                    (unsigned)((g.nz + kBT - 1) / kBT));
    }

    // Planes per block of a z march over level g with per_sm resident blocks per SM, whose
    // blocks walk extra planes beside their chunk: the even length with the least
    // steps x waves.  A step of an SM's k resident blocks takes k issue-bound units, and
    // four at least (up to four blocks it is bound by its chain of loads, shared-memory
    // round trips and barrier), so long chunks save the extra planes, short ones fill a
    // last wave or a small level.
    // Against chunks halved from 16 until every SM had four blocks: 256^3 mixed, level 1
    // 49 / 40 -> 31 / 28 us a launch down / up, level 0 85 / 91 -> 79 / 83, the solve 8.1 ->
    // 7.55 ms; 96^3 FP64, level 0 way down 28 -> 18 us.
    int pick_zc(const Geom& g, int per_sm, int extra) const {
        const long long tiles = (long long)((g.nx + kMX - 1) / kMX) * ((g.ny + kMY - 1) / kMY);
        int best = 2;
        double best_cost = 1e300;
        for (int zc = 2; zc < g.nz + 2 && zc <= 128; zc += 2) {
            const long long k = (tiles * ((g.nz + zc - 1) / zc) + num_sms_ - 1) / num_sms_;
            const long long full = k / per_sm, rest = k % per_sm;
            const double cost = (zc + extra) * ((double)full * std::max(4, per_sm) +
                                                (rest ? std::max<double>(4.0, (double)rest) : 0.0));
            if (cost < best_cost) { best_cost = cost; best = zc; }
        }
        return best;
    }
    template <class K>
    static int resident(K kern, size_t smem) {
        int per_sm = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreads, smem) != cudaSuccess ||
            per_sm < 1) {
            cudaGetLastError();
            per_sm = 1;
        }
        return per_sm;
    }
    template <int DIM, bool FINE, class CSL, bool STAR>
    void pick_chunks_as(LevelBuf<T, CS>& L) const {
        if constexpr (FINE && STAR) {
            L.zc = pick_zc(L.g, resident(k_level_quad<DIM, CSL, false, false>, QCfg<DIM, CSL, false>::BYTES), 6);
            L.zu = pick_zc(L.g, resident(k_level_quad<DIM, CSL, true, true>, QCfg<DIM, CSL, true>::BYTES), 4);
        } else {
            L.zc = pick_zc(L.g, resident(k_level_fused<DIM, T, FINE, CSL, false, false, STAR>,
                                         FCfg<DIM, T, CSL, FINE, false, STAR>::BYTES), STAR ? 6 : 4);
            L.zu = pick_zc(L.g, resident(k_level_fused<DIM, T, FINE, CSL, true, FINE, STAR>,
                                         FCfg<DIM, T, CSL, FINE, true, STAR>::BYTES), 4);
        }
    }
    // Chunk lengths of level l's fused marches (the four-march kernels take the way down's)
    // and of the search direction.
    template <int DIM, bool STAR>
    void pick_chunks() {
        for (size_t l = 0; l < lv_.size(); ++l) {
            LevelBuf<T, CS>& L = lv_[l];
            if (l == 0) pick_chunks_as<DIM, true, CS, STAR>(L);
            else if (L.c32) pick_chunks_as<DIM, false, T, STAR>(L);
            else pick_chunks_as<DIM, false, CS, STAR>(L);
        }
        // chunks halved from 16 planes until every SM has four blocks
        const Geom& g = lv_[0].g;
        const long long tiles = (long long)((g.nx + kMX - 1) / kMX) * ((g.ny + kMY - 1) / kMY);
        int zc = 16;
        while (zc > 2 && tiles * ((g.nz + zc - 1) / zc) < 4LL * num_sms_) zc /= 2;
        // The finest level with Dirichlet walls runs as four marches, whose blocks need no
        // long chunks to pay for their start: on the fused march's length instead, solves of
        // 224^3 take 16.8 (FP64) and 6.2 ms (mixed), here 13.2 and 5.5; 128^3 4.34 and 1.72,
        // here 3.62 and 1.60; below 96^3 the same.
        if (dirichlet_) lv_[0].zc = zc;
        if constexpr (sizeof(T) == 8) {
            // The FP64 form's dot products are summed per block (search direction, z sums); their
            // partition stays: 256^3 on another one stops after 81 iterations instead of the
            // reference's 82.
            zdot_zc_ = pm_zc_ = zc;
            return;
        }
        pm_zc_ = pick_zc(lv_[0].g, dirichlet_ ? resident(k_pmatvec<DIM, T, true>, PmvCfg<DIM, T>::BYTES)
                                              : resident(k_pmatvec<DIM, T, false>, PmvCfg<DIM, T>::BYTES), 2);
    }

    template <class K>
    static int smem_attr(K kern, size_t bytes) {
        return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) ==
                       cudaSuccess
                   ? E_OK
                   : E_CUDA;
    }

    template <int DIM, bool FINE, class CSL>
    int march_attrs() {
        int e;
        if ((e = smem_attr(k_fwd_smooth<DIM, T, FINE, CSL>, FwdCfg<DIM, T, FINE, CSL>::BYTES)) ||
            (e = smem_attr(k_restrict_res<DIM, T, FINE, CSL>, ResCfg<DIM, T, FINE, CSL>::BYTES)) ||
            (e = smem_attr(k_up_even<DIM, T, FINE, CSL>, UpeCfg<DIM, T, FINE, CSL>::BYTES)) ||
            (e = smem_attr(k_up_odd<DIM, T, FINE, false, CSL>, UpoCfg<DIM, T, FINE, CSL>::BYTES)) ||
            (e = smem_attr(k_up_odd<DIM, T, FINE, true, CSL>, UpoCfg<DIM, T, FINE, CSL>::BYTES)))
            return e;
        return E_OK;
    }

    template <bool FINE, class CSL>
    int box_attrs() {
        int e;
        if ((e = smem_attr(k_level_box<T, FINE, CSL, false, false>, BPlan<T, CSL, FINE, false>::BYTES)) ||
            (e = smem_attr(k_level_box<T, FINE, CSL, true, false>, BPlan<T, CSL, FINE, true>::BYTES)) ||
            (e = smem_attr(k_level_box<T, FINE, CSL, true, true>, BPlan<T, CSL, FINE, true>::BYTES)))
            return e;
        if constexpr (sizeof(T) == 4) {
            if ((e = smem_attr(k_level_box<T, FINE, CSL, false, false, true>,
                               BPlan<T, CSL, FINE, false, true>::BYTES)) ||
                (e = smem_attr(k_level_box<T, FINE, CSL, true, false, true>,
                               BPlan<T, CSL, FINE, true, true>::BYTES)) ||
                (e = smem_attr(k_level_box<T, FINE, CSL, true, true, true>,
                               BPlan<T, CSL, FINE, true, true>::BYTES)))
                return e;
        }
        return E_OK;
    }

    template <int DIM, bool FINE, class CSL>
    int fused_attrs() {
        int e;
        if ((e = smem_attr(k_level_fused<DIM, T, FINE, CSL, false, false>,
                           FCfg<DIM, T, CSL, FINE, false>::BYTES)) ||
            (e = smem_attr(k_level_fused<DIM, T, FINE, CSL, true, false>,
                           FCfg<DIM, T, CSL, FINE, true>::BYTES)) ||
            (e = smem_attr(k_level_fused<DIM, T, FINE, CSL, true, true>,
                           FCfg<DIM, T, CSL, FINE, true>::BYTES)))
            return e;
        if constexpr (sizeof(T) == 4 && FINE) {
            if ((e = smem_attr(k_level_quad<DIM, CSL, false, false>, QCfg<DIM, CSL, false>::BYTES)) ||
                (e = smem_attr(k_level_quad<DIM, CSL, true, false>, QCfg<DIM, CSL, true>::BYTES)) ||
                (e = smem_attr(k_level_quad<DIM, CSL, true, true>, QCfg<DIM, CSL, true>::BYTES)))
                return e;
        } else if constexpr (sizeof(T) == 4) {
            if ((e = smem_attr(k_level_fused<DIM, T, FINE, CSL, false, false, true>,
                               FCfg<DIM, T, CSL, FINE, false, true>::BYTES)) ||
                (e = smem_attr(k_level_fused<DIM, T, FINE, CSL, true, false, true>,
                               FCfg<DIM, T, CSL, FINE, true, true>::BYTES)) ||
                (e = smem_attr(k_level_fused<DIM, T, FINE, CSL, true, true, true>,
                               FCfg<DIM, T, CSL, FINE, true, true>::BYTES)))
                return e;
        }
        return E_OK;
    }

    // The problem's buffers, in order (run twice: sizes, then addresses).
    template <int DIM>
    int buffers() {
        const int nl = (int)lv_.size();
        int e;
        for (int l = 0; l < nl; ++l) {
            LevelBuf<T, CS>& L = lv_[l];
            const size_t n = (size_t)L.g.n;
            if ((e = alloc(L.solid, n))) return e;
            if ((e = alloc(L.code, n))) return e;
            if ((e = alloc(L.cx, n))) return e;
            if ((e = alloc(L.cy, n))) return e;
            if (DIM == 3 && (e = alloc(L.cz, n))) return e;
            if (dirichlet_ && (e = alloc(L.wd, n))) return e;
            if (l > 0) {
                if ((e = alloc(L.x, n))) return e;
                if ((e = alloc(L.b, n))) return e;
                if ((e = alloc(L.dg, n))) return e;
                if (L.box && !star_ && !plain_) {
                    const dim3 bg = box_grid(L.g);
                    if ((e = alloc(L.trim, (size_t)4 * bg.x * bg.y * bg.z))) return e;
                }
                if constexpr (kHalf) {
                    if (!L.c32) {
                        if ((e = alloc(L.hcx, n)) || (e = alloc(L.hcy, n))) return e;
                        if (DIM == 3 && (e = alloc(L.hcz, n))) return e;
                    }
                } else {
                    L.hcx = L.cx; L.hcy = L.cy; L.hcz = L.cz;
                }
            }
        }
        const Geom g0 = lv_[0].g;
        const size_t n0 = (size_t)g0.n;
        if ((e = alloc(r_, n0)) || (e = alloc(z_, n0))) return e;
        if (!apply_only_ &&
            ((e = alloc(p_, n0)) || (e = alloc(p2_, n0)) || (e = alloc(ap_, n0)) ||
             (e = alloc(xlo_, n0)) || (e = alloc(b64_, n0)) || (e = alloc(xd_, n0))))
            return e;
        // reductions: the finest-level marches (one partial per block) and the
        // row-walk kernels (vec_grid)
        {
            const dim3 mg = march_grid<DIM>(g0, 2);  // the most blocks any chunk length gives
            reduce_blocks_ = (long long)mg.x * mg.y * mg.z;
            const dim3 rg = resid_grid(g0);
            reduce_blocks_ = std::max(reduce_blocks_, (long long)rg.x * rg.y * rg.z);
            const dim3 bg = box_grid(g0);  // a small finest level runs as boxes
            if (lv_[0].box) reduce_blocks_ = std::max(reduce_blocks_, (long long)bg.x * bg.y * bg.z);
            if (reduce_blocks_ < max_reduce_blocks()) reduce_blocks_ = max_reduce_blocks();
        }
        if ((e = alloc(partials_, (size_t)reduce_blocks_ * 4))) return e;
        if ((e = alloc(cg_, 1))) return e;
        err_ = reinterpret_cast<int*>(reinterpret_cast<unsigned char*>(cg_) + offsetof(CGState, err));
        if (dense_cells_ > 0) {
            if ((e = alloc(dense_, (size_t)dense_cells_ * dense_ld_))) return e;
            if ((e = alloc(dense_cell_, (size_t)dense_cells_))) return e;
        }
        return E_OK;
    }

    template <int DIM>
    int build(int nx, int ny, int nz, const uint8_t* d_solid) {
        gref_ = make_geom(DIM, nx, ny, nz);
        {
            const Geom gp = make_geom_pitched(DIM, nx, ny, nz);
            if ((long long)gp.sx * (ny + 2) * (DIM == 3 ? nz + 2 : 1) >= (1LL << 31)) return E_ARG;
        }
        // Levels.  The reference's rule (floor sizes, a coarse cell solid when half of its
        // children are) drops fluid cells: the last row of an odd size, and cells whose
        // parent became solid, belong to no aggregate, get no coarse correction, and the
        // coarse couplings towards them act as Dirichlet walls.  CG then needs many
        // iterations for the modes this pins (without solids 8-13).  The FP32 and mixed
        // solves (cover_) aggregate every fluid cell instead: sizes rounded up, a coarse
        // cell fluid when any child is, the same Galerkin sums.  Iterations of mixed solves to
        // 1e-6 with the reference's rule, with this one and constant transfers, and with star
        // transfers (fused.cuh): 96^3 with 8 spheres 47 / 14 / 11, 256^3 with 32 spheres 82 /
        // 15 / 12, 384^2 with one disk 78 / 11 / 9, 2048 x 1024 155 / 19 / 12, 129 x 97 x 65
        // 197 / 45 / 15; an iteration takes about the same time.  The FP64 form and every
        // V-cycle applied by itself keep the reference's rule, and so do problems with
        // Dirichlet walls (their wall channel is defined by it).
        const bool cover = cover_ && !plain_ && !dirichlet_;
        star_ = cover;
        const int up = cover ? 1 : 0;
        double hx = dx_, hy = dy_, hz = dz_;
        while (nx >= 2 && ny >= 2 && (DIM == 2 || nz >= 2)) {
            LevelBuf<T, CS> L;
            L.g = make_geom_pitched(DIM, nx, ny, nz);
            L.hx = hx; L.hy = hy; L.hz = hz;
            lv_.push_back(L);
            if (nx <= 4 || ny <= 4 || (DIM == 3 && nz <= 4)) break;
            nx = (nx + up) / 2; ny = (ny + up) / 2; nz = (nz + up) / 2;
            hx *= 2.0; hy *= 2.0; hz *= 2.0;
        }
        int dev = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&num_sms_, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
            return E_CUDA;
        {
            int per_sm = 0;
            if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_resid_x64<DIM, T>, 256, 0) ==
                    cudaSuccess && per_sm > 0)
                resid_per_sm_ = std::min(per_sm, 8);
            else
                cudaGetLastError();
        }
        if (pmv2d_env_ > 0) {
            pmv2d_per_sm_ = pmv2d_env_;
        } else if (sizeof(T) == 8) {
            pmv2d_per_sm_ = 4;  // the partition of the FP64 form's p.Ap (k_pmatvec_2d)
        } else {
            int per_sm = 0;
            if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_pmatvec_2d<T>, 256, 0) ==
                    cudaSuccess && per_sm > 0)
                pmv2d_per_sm_ = std::min(per_sm, 8);
            else
                cudaGetLastError();
        }
        const int nl = (int)lv_.size();
        int e;
        for (int l = 0; l < nl; ++l) {
            LevelBuf<T, CS>& L = lv_[l];
            // largest face count of a level-l coupling: 4^l (3D), 2^l (2D)
            L.c32 = kHalf && l > 0 && (DIM == 3 ? 2 * l : l) > 11;
            L.box = DIM == 3 && cells(L.g) <= box_cells_;
        }
        if ((e = tail_setup<DIM>()) != E_OK) return e;
        arena_dry_ = true;
        arena_used_ = 0;
        if ((e = buffers<DIM>()) || (e = arena_ready()) || (e = buffers<DIM>())) return e;
        const Geom g0 = lv_[0].g;
        if (!cg_host_ && cudaMallocHost(&cg_host_, sizeof(CGState)) != cudaSuccess) return E_OOM;
        if (!flag_host_ && cudaMallocHost(&flag_host_, sizeof(*flag_host_)) != cudaSuccess) return E_OOM;
        // dynamic shared memory of the marches
        if ((e = march_attrs<DIM, true, CS>()) || (e = march_attrs<DIM, false, CS>()) ||
            (e = smem_attr(k_pmatvec<DIM, T, true>, PmvCfg<DIM, T>::BYTES)) ||
            (e = smem_attr(k_pmatvec<DIM, T, false>, PmvCfg<DIM, T>::BYTES)) ||
            (e = fused_attrs<DIM, true, CS>()) || (e = fused_attrs<DIM, false, CS>()))
            return e;
        if constexpr (kHalf) {  // levels with FP32 couplings
            if ((e = march_attrs<DIM, false, T>()) || (e = fused_attrs<DIM, false, T>())) return e;
        }
        if (DIM == 3) {
            if ((e = smem_attr(k_resid_march<T, true>, RxCfg<T>::BYTES)) ||
                (e = smem_attr(k_resid_march<T, false>, RxCfg<T>::BYTES)) ||
                (e = smem_attr(k_resid_march<T, true, true>, RxCfg<T>::BYTES)) ||
                (e = smem_attr(k_resid_march<T, false, true>, RxCfg<T>::BYTES)))
                return e;
            // planes per block of the replacement march: chunks doubled until the blocks
            // fit in one wave (256^3: 64 planes, 512 blocks; 1.31 against 1.37 ms a solve
            // with 32 planes and 1024 blocks)
            int per_sm = 0;
            if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_resid_march<T, false>, kThreads,
                                                              RxCfg<T>::BYTES) != cudaSuccess ||
                per_sm < 1) {
                cudaGetLastError();
                per_sm = 1;
            }
            const Geom& g = lv_[0].g;
            const long long tiles = (long long)((g.nx + kMX - 1) / kMX) * ((g.ny + kMY - 1) / kMY);
            rx_zc_ = 2;
            while (rx_zc_ < g.nz && tiles * ((g.nz + rx_zc_ - 1) / rx_zc_) > (long long)per_sm * num_sms_)
                rx_zc_ *= 2;
        }
        if constexpr (DIM == 3) {  // (after the kernels' shared-memory attributes)
            if constexpr (sizeof(T) == 4) {
                if (star_) pick_chunks<DIM, true>();
                else pick_chunks<DIM, false>();
            } else {
                pick_chunks<DIM, false>();
            }
        }
        if (DIM == 3) {
            if ((e = box_attrs<true, CS>()) || (e = box_attrs<false, CS>())) return e;
            if constexpr (kHalf) {
                if ((e = box_attrs<false, T>())) return e;
            }
        }
        // plane-box tensor maps
        constexpr int BW = PBox<T>::W, BH = PBox<T>::H;
        for (int l = 0; l < nl; ++l) {
            LevelBuf<T, CS>& L = lv_[l];
            const T* b = l == 0 ? r_ : L.b;
            const T* x = l == 0 ? z_ : L.x;
            bool ok = encode_level_map<T>(&L.mb, b, L.g, DIM, BW, BH, 1) &&
                      encode_level_map<T>(&L.mx, x, L.g, DIM, BW, BH, 1) &&
                      encode_level_map<uint8_t>(&L.mcode, L.code, L.g, DIM, PBox<uint8_t>::W,
                                                PBox<uint8_t>::H, 1);
            constexpr int CW = PBox<CS>::W;
            if (ok && l > 0 && !L.c32)
                ok = encode_level_map<CS>(&L.mcx, L.hcx, L.g, DIM, CW, BH, 1) &&
                     encode_level_map<CS>(&L.mcy, L.hcy, L.g, DIM, CW, BH, 1) &&
                     (DIM == 2 || encode_level_map<CS>(&L.mcz, L.hcz, L.g, DIM, CW, BH, 1));
            if (ok && l > 0 && L.c32)  // FP32 couplings read as T
                ok = encode_level_map<T>(&L.mcx, L.cx, L.g, DIM, BW, BH, 1) &&
                     encode_level_map<T>(&L.mcy, L.cy, L.g, DIM, BW, BH, 1) &&
                     (DIM == 2 || encode_level_map<T>(&L.mcz, L.cz, L.g, DIM, BW, BH, 1));
            if (ok && l > 0)
                ok = encode_level_map<T>(&L.mdg, L.dg, L.g, DIM, BW, BH, 1) &&
                     encode_level_map<T>(&L.mxq, L.x, L.g, DIM, QBox<T>::W, QBox<T>::H, 1);
            if (ok) ok = box_maps<DIM, RBox<T, 2>, RBox<uint8_t, 2>, RBox<CS, 2>, RBox<T, 2>>(L, b, l, 1, &L.f);
            if constexpr (sizeof(T) == 4) {
                if (ok && star_)
                    ok = box_maps<DIM, RBox<T, 3>, RBox<uint8_t, 3>, RBox<CS, 3>, RBox<T, 3>>(L, b, l, 1, &L.fd);
                if (ok && star_ && l > 0) {
                    using B = SBox<T, DIM>;
                    ok = encode_level_map<T>(&L.mxs, L.x, L.g, DIM, B::W, B::H, DIM == 3 ? 2 : 1) &&
                         encode_level_map<uint8_t>(&L.mps, L.code, L.g, DIM, B::CW, B::CH, 1);
                }
            }
            if (ok && DIM == 3) {
                // whole-tile boxes (small levels) and this level's x (STAR: and codes) as the
                // parent box of the next-finer level's box kernels
                if (l > 0) ok = encode_level_map<T>(&L.bxq, L.x, L.g, DIM, BQBox<T>::W, 6, 6);
                if (ok && l > 0 && star_) {
                    using B = BSBox<T>;
                    ok = encode_level_map<T>(&L.bxs, L.x, L.g, DIM, B::W, B::N, B::N) &&
                         encode_level_map<uint8_t>(&L.bps, L.code, L.g, DIM, B::CW, B::CN, B::CN);
                }
                if (ok && L.box)
                    ok = box_maps<DIM, BBox<T, 2>, BBox<uint8_t, 2>, BBox<CS, 2>, BBox<T, 2>>(
                        L, b, l, BBox<T, 2>::N, &L.bx);
                if constexpr (sizeof(T) == 4) {
                    if (ok && L.box && star_)
                        ok = box_maps<DIM, BBox<T, 3>, BBox<uint8_t, 3>, BBox<CS, 3>, BBox<T, 3>>(
                            L, b, l, BBox<T, 3>::N, &L.bd);
                }
            }
            if (!ok) return E_CUDA;
        }
        if (apply_only_) {
        } else if (!encode_level_map<T>(&map_p_, p_, g0, DIM, BW, BH, 1) ||
            !encode_level_map<T>(&map_p2_, p2_, g0, DIM, BW, BH, 1))
            return E_CUDA;
        if (DIM == 3 && !apply_only_ &&
            (!encode_level_map<double>(&map_b64_, b64_, g0, DIM, PBox<double>::W, PBox<double>::H, 1) ||
             !encode_level_map<double>(&map_xd_, xd_, g0, DIM, PBox<double>::W, PBox<double>::H, 1) ||
             !encode_level_map<T>(&map_xlo_, xlo_, g0, DIM, BW, BH, 1)))
            return E_CUDA;

        // hierarchy: masks, couplings, coarse diagonals
        const dim3 blk = cell_block<DIM>();
        UAAMG_LAUNCH((KTag{K_SETUP, 0, 0.0}), k_import_mask<DIM>, vec_grid(g0), dim3(32, 8), g0, gref_,
                     d_solid, lv_[0].solid);
        for (int l = 1; l < nl; ++l)
            UAAMG_LAUNCH((KTag{K_SETUP, l, 0.0}), k_restrict_solid<DIM>,
                         cell_grid<DIM>(lv_[l].g.nx, lv_[l].g.ny, lv_[l].g.nz), blk, lv_[l - 1].g,
                         lv_[l - 1].solid, lv_[l].g, lv_[l].solid, cover ? 1 : 0);
        {
            const LevelBuf<T, CS>& L = lv_[0];
            const T idx2 = (T)(1.0 / (L.hx * L.hx)), idy2 = (T)(1.0 / (L.hy * L.hy));
            const T idz2 = DIM == 3 ? (T)(1.0 / (L.hz * L.hz)) : T(0);
            UAAMG_LAUNCH((KTag{K_SETUP, 0, 0.0}), (k_fine_coeffs<DIM, T>),
                         cell_grid<DIM>(L.g.nx, L.g.ny, L.g.nz), blk, L.g, L.solid, L.cx, L.cy, L.cz,
                         L.wd, idx2, idy2, idz2);
        }
        for (int l = 1; l < nl; ++l) {
            const LevelBuf<T, CS>& F = lv_[l - 1];
            LevelBuf<T, CS>& Cl = lv_[l];
            UAAMG_LAUNCH((KTag{K_SETUP, l, 0.0}), (k_galerkin<DIM, T>),
                         cell_grid<DIM>(Cl.g.nx, Cl.g.ny, Cl.g.nz), blk, F.g, F.cx, F.cy, F.cz, F.wd,
                         Cl.g, Cl.solid, Cl.cx, Cl.cy, Cl.cz, Cl.wd);
        }
        for (int l = 1; l < nl; ++l) {
            LevelBuf<T, CS>& Cl = lv_[l];
            if constexpr (kHalf) {  // FP16 face counts (after every level's Galerkin sums)
              if (!Cl.c32) {
                const Geom& g0 = lv_[0].g;
                const float cs[3] = {(float)(1.0 / (lv_[0].hx * lv_[0].hx)),
                                     (float)(1.0 / (lv_[0].hy * lv_[0].hy)),
                                     (float)(1.0 / (lv_[0].hz * lv_[0].hz))};
                (void)g0;
                T* src[3] = {Cl.cx, Cl.cy, Cl.cz};
                CS* dst[3] = {Cl.hcx, Cl.hcy, Cl.hcz};
                for (int a = 0; a < DIM; ++a)
                    UAAMG_LAUNCH((KTag{K_SETUP, l, 0.0}), k_coupling_half, max_reduce_blocks(), 256,
                                 (long long)Cl.g.n, src[a], dst[a], cs[a]);
              }
            }
            UAAMG_LAUNCH((KTag{K_SETUP, l, 0.0}), (k_diag<DIM, T>), vec_grid(Cl.g), dim3(32, 8), Cl.g,
                         Cl.solid, Cl.cx, Cl.cy, Cl.cz, Cl.wd, Cl.dg);
        }
        for (int l = 0; l < nl; ++l)
            UAAMG_LAUNCH((KTag{K_SETUP, l, 0.0}), (k_codes<DIM, T>), vec_grid(lv_[l].g), dim3(32, 8),
                         lv_[l].g, lv_[l].solid, lv_[l].code, l == 0 ? 1 : 0,
                         star_ && l > 0 ? lv_[l].cx : (const T*)nullptr, lv_[l].cy, lv_[l].cz);
        if constexpr (DIM == 3) {  // trimmed boxes of the coarse box levels
            for (int l = 1; l < nl; ++l) {
                const LevelBuf<T, CS>& Cl = lv_[l];
                // (not for the covering hierarchy: its dozen iterations took the same time with
                // trimming and without, and finding the boxes costs 65 us of set-up)
                if (!Cl.box || !Cl.trim) continue;
                const MLevel<T> m = mlevel(l);
                if (kHalf && !Cl.c32)
                    UAAMG_LAUNCH((KTag{K_SETUP, l, 0.0}), (k_box_trim<T, CS>), box_grid(Cl.g), 256,
                                 Cl.g, Cl.code, Cl.dg, Cl.hcx, Cl.hcy, Cl.hcz, m.csx, m.csy, m.csz,
                                 Cl.trim);
                else
                    UAAMG_LAUNCH((KTag{K_SETUP, l, 0.0}), (k_box_trim<T, T>), box_grid(Cl.g), 256,
                                 Cl.g, Cl.code, Cl.dg, Cl.cx, Cl.cy, Cl.cz, m.csx, m.csy, m.csz,
                                 Cl.trim);
            }
        }
        if ((e = dense_setup<DIM>()) != E_OK) return e;
        if ((e = sync_check()) != E_OK) return e;
        if (DIM == 3 && autotune_) return tune<DIM>();
        return E_OK;
    }

    bool use_tail() const { return tail_on_ && !sweeps_ && tail_nc_ > 0; }

    // The small levels' one-block kernel (tail.cuh): from the first level (>= 1) of at
    // most kTailCells cells down to the coarsest, while their x and b fit its shared
    // memory and the coarsest has at most two cells a thread.
    static size_t tail_cells_padded(const Geom& g) {
        return (size_t)(g.nx + 2) * (g.ny + 2) * (g.nz ? g.nz + 2 : 1);
    }

    template <int DIM>
    int tail_setup() {
        const int nl = (int)lv_.size();
        tail_nc_ = 0;
        tail_lt_ = nl;
        dense_cells_ = 0;
        if (nl < 2) return E_OK;
        const Geom& gc = lv_[nl - 1].g;
        size_t elems = 2 * tail_cells_padded(gc);
        if (cells(gc) > 2.0 * tail_threads<T>() || elems * sizeof(T) > kTailSmemBytes) return E_OK;
        int lt = nl - 1;
        while (lt > 1 && cells(lv_[lt - 1].g) <= (double)kTailCells && nl - (lt - 1) <= kTailMaxLevels &&
               (elems + 2 * tail_cells_padded(lv_[lt - 1].g)) * sizeof(T) <= kTailSmemBytes) {
            --lt;
            elems += 2 * tail_cells_padded(lv_[lt].g);
        }
        // the attribute belongs to the kernel, not to this engine: always the cap
        if (cudaFuncSetAttribute(k_tail<DIM, T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)kTailSmemBytes) != cudaSuccess)
            return E_CUDA;
        tail_lt_ = lt;
        tail_nc_ = 1;
        tail_smem_ = elems * sizeof(T);
        if (sizeof(T) == 4 && cover_ && !plain_ && cells(lv_[lt].g) <= (double)kDenseCells) {
            dense_cells_ = (int)cells(lv_[lt].g);
            dense_ld_ = (dense_cells_ + 3) / 4 * 4;
        }
        return E_OK;
    }

    template <int DIM>
    TailArgs<T> tail_args() const {
        const int nl = (int)lv_.size();
        TailArgs<T> a{};
        a.nlev = nl - tail_lt_;
        int off = 0;
        for (int q = 0; q < a.nlev; ++q) {
            const LevelBuf<T, CS>& L = lv_[tail_lt_ + q];
            TailLevel<T>& t = a.lv[q];
            t.g = L.g;
            t.csx = L.g.nx + 2;
            t.csxy = (L.g.nx + 2) * (L.g.ny + 2);
            t.xs = off;
            t.bs = off + (int)tail_cells_padded(L.g);
            off += 2 * (int)tail_cells_padded(L.g);
            t.code = L.code;
            t.cx = L.cx;
            t.cy = L.cy;
            t.cz = DIM == 3 ? L.cz : nullptr;
            t.dg = L.dg;
            t.x = L.x;
            t.b = L.b;
            t.rnx = 1.0f / (float)L.g.nx;
            t.rny = 1.0f / (float)L.g.ny;
        }
        a.smem_elems = off;
        a.star = star_ ? 1 : 0;
        return a;
    }

    // The tail's cycle as a dense matrix (solves in FP32 and mixed; tail.cuh).  Its
    // buffers have one size whatever the mask, so a mask change allocates nothing.
    template <int DIM>
    int dense_setup() {
        dense_n_ = 0;
        if constexpr (sizeof(T) == 4) {
            if (dense_cells_ == 0) return E_OK;
            const Geom& g = lv_[tail_lt_].g;
            const int n = dense_cells_;
            UAAMG_LAUNCH((KTag{K_SETUP, tail_lt_, 0.0}), k_tail_cells<DIM>, 1, 256, g, dense_cell_);
            // small blocks, five a SM, unless the coarsest level needs more threads (two cells
            // each): the phases are latency-bound
            const int nt = cells(lv_.back().g) <= 512.0 ? 256 : tail_threads<T>();
            UAAMG_LAUNCH_SMEM((KTag{K_SETUP, tail_lt_, 0.0}), (k_tail<DIM, T>), n, nt, tail_smem_,
                              tail_args<DIM>(), (const int*)nullptr, dense_, dense_ld_);
            dense_n_ = n;
        }
        return E_OK;
    }

    // Levels tail_lt_ .. nl-1 of the V-cycle (b of tail_lt_ in, its x out).
    template <int DIM>
    void tail_launch(const int* done) {
        const LevelBuf<T, CS>& L0 = lv_[tail_lt_];
        if constexpr (sizeof(T) == 4) {
            if (dense_n_ > 0) {
                const int n = dense_n_, nb = (n + 7) / 8, n4 = (dense_ld_ + 127) / 128;
                // matrix, cell numbers and b in, x out
                const KTag tag{K_TAIL, tail_lt_, (double)n * dense_ld_ * sizeof(T) + 12.0 * n};
#define UAAMG_DENSE(N4)                                                                     \
    UAAMG_LAUNCH(tag, k_tail_dense<N4>, nb, 256, n, dense_ld_, dense_, dense_cell_, L0.b, L0.x, done)
                if (n4 <= 1) UAAMG_DENSE(1);
                else if (n4 <= 2) UAAMG_DENSE(2);
                else if (n4 <= 4) UAAMG_DENSE(4);
                else UAAMG_DENSE(8);
#undef UAAMG_DENSE
                return;
            }
        }
        double bytes = 2.0 * cells(L0.g) * sizeof(T);  // the first level's b in, x out
        for (size_t l = tail_lt_; l < lv_.size(); ++l)
            // codes, couplings and diagonal read once per pass, four passes
            bytes += 4.0 * cells(lv_[l].g) * ((1.0 + DIM) * sizeof(T) + 1.0);
        UAAMG_LAUNCH_SMEM((KTag{K_TAIL, tail_lt_, bytes}), (k_tail<DIM, T>), 1, tail_threads<T>(),
                          tail_smem_, tail_args<DIM>(), done, (T*)nullptr, 0);
    }

    // Autotuner: for every level with marches, time its V-cycle marches (down and up,
    // on the level's own buffers) for the rule's lengths and for each of 2, 4, ..., 128 and
    // keep the fastest; the choice is cached per GPU, precision, level shape and
    // march kind (tune_lookup / tune_store: for the process, and in the cache file
    // when one is set).  Chunk length changes only the blocks' shape, not a per-cell
    // value; the FP64 dot products are summed per block, so their rounding (and so
    // the last bits of the iterates) may differ.
    template <int DIM>
    int tune() {
        cudaEvent_t a = nullptr, b = nullptr;
        if (cudaEventCreate(&a) != cudaSuccess || cudaEventCreate(&b) != cudaSuccess) return E_CUDA;
        const bool prof = prof_on_;
        prof_on_ = false;
        int e = E_OK;
        for (int l = 0; l + 1 < (int)lv_.size() && e == E_OK; ++l) {
            if (use_tail() && l >= tail_lt_) break;  // the small-level kernel runs those levels
            LevelBuf<T, CS>& L = lv_[l];
            if (L.box && fused_ && level_nu(l) == 1) continue;  // whole-tile boxes: no chunks
            const std::string key = "zc|" + tune_gpu_id() + "|" + (sizeof(T) == 8 ? "f64" : mixed_ ? "mixed" : "f32") +
                                    "|" + std::to_string(L.g.nx) + "x" + std::to_string(L.g.ny) + "x" +
                                    std::to_string(L.g.nz) + "|" + (l == 0 ? "fine" : "coarse") + "|" +
                                    (fused_ && level_nu(l) == 1 ? star_ ? "star" : "fused" : "four") +
                                    (L.c32 ? "|c32" : "");
            {
                std::vector<int> v;
                if (tune_lookup(key, &v) && v.size() == 1 && (v[0] == 0 || (v[0] >= 2 && v[0] <= 128))) {
                    if (v[0]) L.zc = L.zu = v[0];
                    continue;
                }
            }
            const int zc0 = L.zc, zu0 = L.zu;  // the rule's own choice: candidate 0
            int best = 0;
            float best_ms = 1e30f;
            for (int zc = 0; zc <= 128 && e == E_OK; zc = zc ? 2 * zc : 2) {
                if (zc > 2 && zc / 2 >= L.g.nz) break;
                L.zc = zc ? zc : zc0;
                L.zu = zc ? zc : zu0;
                for (int rep = 0; rep < 3; ++rep) {  // rep 0 warms up
                    if (rep == 1) cudaEventRecord(a, st_);
                    if (l == 0) { down_level<DIM, true>(l, nullptr); up_level<DIM, true>(l, nullptr, false); }
                    else { down_level<DIM, false>(l, nullptr); up_level<DIM, false>(l, nullptr, false); }
                }
                cudaEventRecord(b, st_);
                float ms = 0.f;
                if (cudaEventSynchronize(b) != cudaSuccess || cudaEventElapsedTime(&ms, a, b) != cudaSuccess) {
                    e = sync_check();
                    if (e == E_OK) e = E_CUDA;
                    break;
                }
                if (ms < best_ms) { best_ms = ms; best = zc; }
            }
            L.zc = best ? best : zc0;
            L.zu = best ? best : zu0;
            tune_store(key, {best});
        }
        prof_on_ = prof;
        cudaEventDestroy(a);
        cudaEventDestroy(b);
        if (e == E_OK) e = sync_check();
        return e;
    }

    LevelView<T> view(int l, const T* r, T* z) const {
        const LevelBuf<T, CS>& L = lv_[l];
        LevelView<T> v;
        v.g = L.g;
        v.solid = L.solid;
        v.cx = L.cx; v.cy = L.cy; v.cz = L.cz; v.wd = L.wd;
        v.x = l == 0 ? z : L.x;
        v.b = l == 0 ? r : L.b;
        return v;
    }

    template <int DIM>
    void sweep(const LevelView<T>& v, int parity, const int* done, int lvl) {
        UAAMG_LAUNCH((KTag{K_SWEEP, lvl, cells(v.g) * ((2.0 + DIM) * sizeof(T) + 0.5)}), (k_sweep<DIM, T>),
                     cell_grid<DIM>((v.g.nx + 1) / 2, v.g.ny, v.g.nz), cell_block<DIM>(), v, parity,
                     done);
    }

    // z = M^{-1} r with one kernel per colour sweep, restriction and prolongation
    // (uaamg_preconditioner_3d.cpp:183-196 step by step); kept as the cross-check
    // of the fused V-cycle.
    template <int DIM>
    void vcycle_sweeps(const T* r, T* z, const int* done) {
        const int nl = (int)lv_.size();
        const dim3 blk = cell_block<DIM>();
        cudaMemsetAsync(z, 0, (size_t)lv_[0].g.n * sizeof(T), st_);
        for (int l = 0; l + 1 < nl; ++l) {
            const LevelView<T> v = view(l, r, z);
            sweep<DIM>(v, 1, done, l);
            sweep<DIM>(v, 0, done, l);
            const LevelBuf<T, CS>& Cl = lv_[l + 1];
            UAAMG_LAUNCH((KTag{K_RESTRICT, l, cells(v.g) * ((2.0 + DIM) * sizeof(T) + 1.0) + cells(Cl.g) * sizeof(T)}),
                         (k_restrict<DIM, T>), cell_grid<DIM>(Cl.g.nx, Cl.g.ny, Cl.g.nz), blk, v, Cl.g,
                         Cl.solid, Cl.b, done);
            cudaMemsetAsync(Cl.x, 0, (size_t)Cl.g.n * sizeof(T), st_);
        }
        coarsest<DIM>(r, z, done);
        for (int l = nl - 2; l >= 0; --l) {
            const LevelView<T> v = view(l, r, z);
            const LevelBuf<T, CS>& Cl = lv_[l + 1];
            UAAMG_LAUNCH((KTag{K_PROLONG, l, cells(v.g) * (2.0 * sizeof(T) + 1.0) + cells(Cl.g) * (sizeof(T) + 1.0)}),
                         (k_prolong<DIM, T>), cell_grid<DIM>(Cl.g.nx, Cl.g.ny, Cl.g.nz), blk, Cl.g,
                         Cl.solid, Cl.x, v.g, v.solid, v.x, done);
            sweep<DIM>(v, 0, done, l);
            sweep<DIM>(v, 1, done, l);
        }
    }

    // Coarsest level: 10 x (forward + reverse) sweeps from x = 0.
    template <int DIM>
    void coarsest(const T* r, T* z, const int* done) {
        const int nl = (int)lv_.size();
        const LevelBuf<T, CS>& C = lv_[nl - 1];
        T* cxp = nl == 1 ? z : C.x;
        cudaMemsetAsync(cxp, 0, (size_t)C.g.n * sizeof(T), st_);
        LevelView<T> v = view(nl - 1, r, z);
        const int ncell = v.g.nx * v.g.ny * (DIM == 3 ? v.g.nz : 1);
        if (ncell <= 65536) {
            UAAMG_LAUNCH((KTag{K_COARSEST, nl - 1, 40.0 * cells(v.g) * ((2.0 + DIM) * sizeof(T) + 0.5)}),
                         (k_coarsest<DIM, T>), 1, 1024, v, done);
        } else {
            for (int q = 0; q < 10; ++q) {
                sweep<DIM>(v, 1, done, nl - 1); sweep<DIM>(v, 0, done, nl - 1);
                sweep<DIM>(v, 0, done, nl - 1); sweep<DIM>(v, 1, done, nl - 1);
            }
        }
    }

    MLevel<T> mlevel(int l, bool up = false) const {
        const LevelBuf<T, CS>& L = lv_[l];
        MLevel<T> v;
        v.g = L.g;
        v.cg = l + 1 < (int)lv_.size() ? lv_[l + 1].g : L.g;
        v.idx2 = (T)(1.0 / (L.hx * L.hx));
        v.idy2 = (T)(1.0 / (L.hy * L.hy));
        v.idz2 = L.g.nz ? (T)(1.0 / (L.hz * L.hz)) : T(0);
        // FP16 couplings are face counts times the finest level's 1/h^2 per axis
        const bool half = kHalf && !L.c32;
        v.csx = half ? (T)(1.0 / (lv_[0].hx * lv_[0].hx)) : T(1);
        v.csy = half ? (T)(1.0 / (lv_[0].hy * lv_[0].hy)) : T(1);
        v.csz = half ? (T)(1.0 / (lv_[0].hz * lv_[0].hz)) : T(1);
        v.dirichlet = dirichlet_;
        v.zc = up ? L.zu : L.zc;
        v.ccode = l + 1 < (int)lv_.size() ? lv_[l + 1].code : nullptr;
        return v;
    }

    // Tensor maps of a march over level l: value slots b, [x], [cx, cy, (cz), dg]
    // (coefficients on coarse levels), the codes and, for the prolongation, the
    // next-coarser level's x as parent boxes.
    template <int DIM>
    MarchMaps maps(int l, bool hasx, bool parent) const {
        const LevelBuf<T, CS>& L = lv_[l];
        MarchMaps m;
        int q = 0;
        m.v[q++] = L.mb;
        if (hasx) m.v[q++] = L.mx;
        if (l > 0) {  // slot order of MPlan: the T boxes, then the couplings
            m.v[q++] = L.mdg;
            m.v[q++] = L.mcx;
            m.v[q++] = L.mcy;
            if (DIM == 3) m.v[q++] = L.mcz;
        }
        m.code = L.mcode;
        if (parent) m.xc = lv_[l + 1].mxq;
        return m;
    }

    // Tensor maps of a fused march over level l; up: the way up, with the next-coarser
    // level's x (STAR: and codes) as parent boxes.
    FMaps fmaps(int l, bool up) const {
        const LevelBuf<T, CS>& L = lv_[l];
        const BoxMaps& f = star_ && !up ? L.fd : L.f;
        FMaps m{};
        m.b = f.b;
        m.code = f.code;
        if (l > 0) {
            m.dg = f.dg;
            m.cx = f.cx;
            m.cy = f.cy;
            m.cz = f.cz;
        }
        if (up) m.xc = star_ ? lv_[l + 1].mxs : lv_[l + 1].mxq;
        if (up && star_) m.pc = lv_[l + 1].mps;
        return m;
    }

    // Tensor maps of a whole-tile box kernel over level l, likewise.
    BMaps bmaps(int l, bool up) const {
        const LevelBuf<T, CS>& L = lv_[l];
        const BoxMaps& f = star_ && !up ? L.bd : L.bx;
        BMaps m{};
        m.b = f.b;
        m.code = f.code;
        if (l > 0) {
            m.dg = f.dg;
            m.cx = f.cx;
            m.cy = f.cy;
            m.cz = f.cz;
            m.trim = trim_ ? L.trim : nullptr;
        }
        if (up) m.xc = star_ ? lv_[l + 1].bxs : lv_[l + 1].bxq;
        if (up && star_) m.pc = lv_[l + 1].bps;
        return m;
    }

    // The way down through level l: b (and on coarse levels the couplings) in,
    // coarse b out.  CSL: the coupling storage of this level.
    template <int DIM, bool FINE>
    void down_level(int l, const int* done) {
        if constexpr (kHalf && !FINE) {
            if (lv_[l].c32) { down_level_cs<DIM, FINE, T>(l, done); return; }
        }
        down_level_cs<DIM, FINE, CS>(l, done);
    }

    int level_nu(int l) const { return l == 0 ? nu_fine_ : nu_coarse_; }

    // b, code (coarse levels: diagonal, couplings) in; coarse b out; whole-tile boxes on
    // the small 3D levels, else the march
    template <int DIM, bool FINE, class CSL, bool STAR>
    void down_fused(int l, const int* done) {
        const LevelBuf<T, CS>& L = lv_[l];
        const LevelBuf<T, CS>& Cl = lv_[l + 1];
        const double c = cells(L.g), cc = cells(Cl.g), t = sizeof(T);
        const double coef = FINE ? 0.0 : DIM * (double)sizeof(CSL) + t;  // couplings + diagonal
        const KTag tag{K_DOWN, l, c * (t + 1.0 + coef) + cc * t};
        if (DIM == 3 && L.box)
            UAAMG_LAUNCH_SMEM(tag, (k_level_box<T, FINE, CSL, false, false, STAR>), box_grid(L.g),
                              dim3(kThreads), (BPlan<T, CSL, FINE, false, STAR>::BYTES), bmaps(l, false),
                              mlevel(l), Cl.b, done, err_, partials_, cg_);
        else if constexpr (FINE && STAR)
            UAAMG_LAUNCH_SMEM(tag, (k_level_quad<DIM, CSL, false, false>), march_grid<DIM>(L.g, L.zc),
                              dim3(kThreads), (QCfg<DIM, CSL, false>::BYTES), fmaps(l, false), mlevel(l),
                              Cl.b, done, err_, partials_, cg_);
        else
            UAAMG_LAUNCH_SMEM(tag, (k_level_fused<DIM, T, FINE, CSL, false, false, STAR>),
                              march_grid<DIM>(L.g, L.zc), dim3(kThreads),
                              (FCfg<DIM, T, CSL, FINE, false, STAR>::BYTES), fmaps(l, false), mlevel(l),
                              Cl.b, done, err_, partials_, cg_);
    }

    // b, code (coarse levels: diagonal, couplings), coarse x in; x out
    template <int DIM, bool FINE, class CSL, bool ZDOT, bool STAR>
    void up_fused(int l, const int* done) {
        const LevelBuf<T, CS>& L = lv_[l];
        const double c = cells(L.g), cc = cells(lv_[l + 1].g), t = sizeof(T);
        const double coef = FINE ? 0.0 : DIM * (double)sizeof(CSL) + t;  // couplings + diagonal
        const KTag tag{K_UP, l, c * (2.0 * t + 1.0 + coef) + cc * t};
        T* x = l == 0 ? z_ : L.x;
        if (DIM == 3 && L.box)
            UAAMG_LAUNCH_SMEM(tag, (k_level_box<T, FINE, CSL, true, ZDOT, STAR>), box_grid(L.g),
                              dim3(kThreads), (BPlan<T, CSL, FINE, true, STAR>::BYTES), bmaps(l, true),
                              mlevel(l, true), x, done, err_, partials_, cg_);
        else if constexpr (FINE && STAR)
            UAAMG_LAUNCH_SMEM(tag, (k_level_quad<DIM, CSL, true, ZDOT>), march_grid<DIM>(L.g, L.zu),
                              dim3(kThreads), (QCfg<DIM, CSL, true>::BYTES), fmaps(l, true),
                              mlevel(l, true), x, done, err_, partials_, cg_);
        else
            UAAMG_LAUNCH_SMEM(tag, (k_level_fused<DIM, T, FINE, CSL, true, ZDOT, STAR>),
                              march_grid<DIM>(L.g, L.zu), dim3(kThreads),
                              (FCfg<DIM, T, CSL, FINE, true, STAR>::BYTES), fmaps(l, true), mlevel(l, true), x,
                              done, err_, partials_, cg_);
    }

    template <int DIM, bool FINE, class CSL>
    void down_level_cs(int l, const int* done) {
        const int nu = level_nu(l);
        const LevelBuf<T, CS>& L = lv_[l];
        const LevelBuf<T, CS>& Cl = lv_[l + 1];
        const double c = cells(L.g), cc = cells(Cl.g), t = sizeof(T);
        const double coef = FINE ? 0.0 : DIM * (double)sizeof(CSL) + t;  // couplings + diagonal
        const dim3 grid = march_grid<DIM>(L.g, L.zc), blk(kThreads);
        // a finest level with Dirichlet walls takes the four-march path (the fused
        // finest level's branch-free cell table holds no wall terms)
        if (fused_ && nu == 1 && !(FINE && dirichlet_)) {
            if constexpr (sizeof(T) == 4) {
                if (star_) { down_fused<DIM, FINE, CSL, true>(l, done); return; }
            }
            down_fused<DIM, FINE, CSL, false>(l, done);
            return;
        }
        T* x = l == 0 ? z_ : L.x;
        UAAMG_LAUNCH_SMEM((KTag{K_FWD, l, c * (2.0 * t + 1.0 + coef)}), (k_fwd_smooth<DIM, T, FINE, CSL>),
                          grid, blk, (FwdCfg<DIM, T, FINE, CSL>::BYTES), maps<DIM>(l, false, false),
                          mlevel(l), x, done, err_);
        for (int q = 1; q < nu; ++q) {  // further forward sweeps (colour 1, then 0) on the stored x
            const LevelView<T> v = view(l, r_, z_);
            sweep<DIM>(v, 1, done, l);
            sweep<DIM>(v, 0, done, l);
        }
        UAAMG_LAUNCH_SMEM((KTag{K_RES, l, c * (2.0 * t + 1.0 + coef) + cc * t}),
                          (k_restrict_res<DIM, T, FINE, CSL>), grid, blk, (ResCfg<DIM, T, FINE, CSL>::BYTES),
                          maps<DIM>(l, true, false), mlevel(l), Cl.code, Cl.b, done, err_);
    }

    // The way up through level l: coarse x in, x out (level 0 with zdot: also the
    // CG's z sums).
    template <int DIM, bool FINE>
    void up_level(int l, const int* done, bool zdot) {
        if constexpr (kHalf && !FINE) {
            if (lv_[l].c32) { up_level_cs<DIM, FINE, T>(l, done, zdot); return; }
        }
        up_level_cs<DIM, FINE, CS>(l, done, zdot);
    }

    template <int DIM, bool FINE, class CSL>
    void up_level_cs(int l, const int* done, bool zdot) {
        const int nu = level_nu(l);
        const LevelBuf<T, CS>& L = lv_[l];
        const LevelBuf<T, CS>& Cl = lv_[l + 1];
        const double c = cells(L.g), cc = cells(Cl.g), t = sizeof(T);
        const double coef = FINE ? 0.0 : DIM * (double)sizeof(CSL) + t;  // couplings + diagonal
        const dim3 grid = march_grid<DIM>(L.g, L.zc), blk(kThreads);
        T* x = l == 0 ? z_ : L.x;
        if (fused_ && nu == 1 && !(FINE && dirichlet_)) {
            const bool zd = FINE && zdot;
            if constexpr (sizeof(T) == 4) {
                if (star_) {
                    if (zd) up_fused<DIM, FINE, CSL, true, true>(l, done);
                    else up_fused<DIM, FINE, CSL, false, true>(l, done);
                    return;
                }
            }
            if constexpr (DIM == 3 && sizeof(T) == 8) {
                if (zd && !L.box) {
                    up_fused<DIM, FINE, CSL, false, false>(l, done);
                    UAAMG_LAUNCH((KTag{K_ZDOT, 0, c * (2.0 * t + 1.0)}), (k_zdot_tiles<T>),
                                 march_grid<DIM>(L.g, zdot_zc_), dim3(256), L.g, zdot_zc_, L.code, r_, z_,
                                 partials_, cg_);
                    return;
                }
            }
            if (zd) up_fused<DIM, FINE, CSL, true, false>(l, done);
            else up_fused<DIM, FINE, CSL, false, false>(l, done);
            return;
        }
        if (nu > 1) {  // (the marches' first colour starts from x of a single forward sweep)
            const LevelView<T> v = view(l, r_, z_);
            UAAMG_LAUNCH((KTag{K_PROLONG, l, c * (2.0 * t + 1.0) + cc * (t + 1.0)}), (k_prolong<DIM, T>),
                         cell_grid<DIM>(Cl.g.nx, Cl.g.ny, Cl.g.nz), cell_block<DIM>(), Cl.g, Cl.solid, Cl.x,
                         v.g, v.solid, v.x, done);
            for (int q = 0; q < nu; ++q) {  // reverse sweeps: colour 0, then 1
                sweep<DIM>(v, 0, done, l);
                sweep<DIM>(v, 1, done, l);
            }
            if (FINE && zdot)
                UAAMG_LAUNCH((KTag{K_ZDOT, 0, c * (2.0 * t + 1.0)}), (k_zdot<DIM, T>), vec_grid(L.g),
                             dim3(32, 8), L.g, L.solid, r_, z_, partials_, cg_);
            return;
        }
        UAAMG_LAUNCH_SMEM((KTag{K_UPE, l, c * (2.0 * t + 1.0 + coef) + cc * t}),
                          (k_up_even<DIM, T, FINE, CSL>), grid, blk, (UpeCfg<DIM, T, FINE, CSL>::BYTES),
                          maps<DIM>(l, false, true), mlevel(l), x, done, err_);
        MLevel<T> m = mlevel(l);
        dim3 zgrid = grid;
        if (DIM == 3 && sizeof(T) == 8) {  // the z sums' own partition (pick_chunks)
            m.zc = zdot_zc_;
            zgrid = march_grid<DIM>(L.g, zdot_zc_);
        }
        if (zdot)
            UAAMG_LAUNCH_SMEM((KTag{K_UPO, l, c * (2.5 * t + 1.0 + coef)}),
                              (k_up_odd<DIM, T, FINE, true, CSL>), zgrid, blk, (UpoCfg<DIM, T, FINE, CSL>::BYTES),
                              maps<DIM>(l, true, false), m, x, done, err_, partials_, cg_);
        else
            UAAMG_LAUNCH_SMEM((KTag{K_UPO, l, c * (2.5 * t + 1.0 + coef)}),
                              (k_up_odd<DIM, T, FINE, false, CSL>), grid, blk, (UpoCfg<DIM, T, FINE, CSL>::BYTES),
                              maps<DIM>(l, true, false), mlevel(l), x, done, err_, partials_, cg_);
    }

    // z_ = M^{-1} r_ with marches on every level down to the small-level kernel (two
    // fused marches a level, fused.cuh, or four, march.cuh); the finest level's last
    // march also reduces the CG's z sums when zdot is set.
    template <int DIM>
    void vcycle_march(const int* done, bool zdot) {
        const int nl = (int)lv_.size();
        const int lt = use_tail() ? tail_lt_ : nl - 1;  // first level below the marches
        for (int l = 0; l < lt; ++l) {
            if (l == 0) down_level<DIM, true>(l, done);
            else down_level<DIM, false>(l, done);
        }
        if (use_tail()) tail_launch<DIM>(done);
        else coarsest<DIM>(r_, z_, done);
        if (nl == 1 && zdot) {
            const Geom& g = lv_[0].g;
            UAAMG_LAUNCH((KTag{K_ZDOT, 0, cells(g) * (2.0 * sizeof(T) + 1.0)}), (k_zdot<DIM, T>),
                         vec_grid(g), dim3(32, 8), g, lv_[0].solid, r_, z_, partials_, cg_);
        }
        for (int l = lt - 1; l >= 0; --l) {
            if (l == 0) up_level<DIM, true>(l, done, zdot);
            else up_level<DIM, false>(l, done, false);
        }
    }

    // z = M^{-1} r_, then (zdot) the z sums -> mean, r.z, beta.
    template <int DIM>
    void vcycle(T* z, const int* done, bool zdot) {
        if (sweeps_) {
            vcycle_sweeps<DIM>(r_, z, done);
            if (zdot) {
                const Geom& g = lv_[0].g;
                UAAMG_LAUNCH((KTag{K_ZDOT, 0, cells(g) * (2.0 * sizeof(T) + 1.0)}), (k_zdot<DIM, T>),
                             vec_grid(g), dim3(32, 8), g, lv_[0].solid, r_, z, partials_, cg_);
            }
        } else {
            vcycle_march<DIM>(done, zdot);
        }
    }

    template <int DIM>
    void precond_impl(const double* d_r, double* d_z) {
        const Geom& g = lv_[0].g;
        UAAMG_LAUNCH((KTag{K_CAST, 0, cells(g) * (8.0 + sizeof(T))}), (k_import<DIM, T>), vec_grid(g),
                     dim3(32, 8), g, gref_, d_r, r_);
        vcycle<DIM>(z_, nullptr, false);
        UAAMG_LAUNCH((KTag{K_CAST, 0, cells(g) * (8.0 + sizeof(T))}), (k_export<DIM, T>), vec_grid(g),
                     dim3(32, 8), g, gref_, z_, d_z, 0);
    }

    // ---- PCG solve, in four stages so that many engines can interleave (batch and
    // serving): begin (right-hand side, initial residual, graph capture), step (queue two
    // iterations, each begun at its preconditioner application), poll (has the device
    // stopped?), end (solution out, exit diagnostics).

    Stencil stencil() const {
        Stencil st;
        st.idx2 = 1.0 / (dx_ * dx_);
        st.idy2 = 1.0 / (dy_ * dy_);
        st.idz2 = dim_ == 3 ? 1.0 / (dz_ * dz_) : 0.0;
        st.diag = dim_ == 3 ? 2.0 * (st.idx2 + st.idy2 + st.idz2) : 2.0 * (st.idx2 + st.idy2);
        st.dirichlet = dirichlet_;
        const bool var = dim_ == 2 && vd_ && vox_ && voy_;
        st.vsx = var ? vsx_ : 0;
        st.vd = var ? vd_ : nullptr;
        st.vox = var ? vox_ : nullptr;
        st.voy = var ? voy_ : nullptr;
        st.fs = var ? vf_[0] : nullptr;
        st.fx = var ? vf_[1] : nullptr;
        st.fy = var ? vf_[2] : nullptr;
        return st;
    }

    // z = M r (or z = r), then the z sums -> mean, r.z, beta
    template <int DIM>
    void cg_precond() {
        const Geom& g = lv_[0].g;
        if (cur_.precond) {
            vcycle<DIM>(z_, &cg_->done, true);
        } else {
            cudaMemcpyAsync(z_, r_, (size_t)g.n * sizeof(T), cudaMemcpyDeviceToDevice, st_);
            UAAMG_LAUNCH((KTag{K_ZDOT, 0, cells(g) * (2.0 * sizeof(T) + 1.0)}), (k_zdot<DIM, T>),
                         vec_grid(g), dim3(32, 8), g, lv_[0].solid, r_, z_, partials_, cg_);
        }
    }

    // One PCG iteration (pcg_3d.cpp:93-124), begun at its preconditioner application: z =
    // M r, the search direction, the update, the residual replacement when due -- so the
    // captured step holds a solve's first application too.  The search direction
    // alternates between p_ and p2_ (from_p: the current one lives in p_).
    template <int DIM>
    void cg_iteration(bool from_p) {
        cg_precond<DIM>();
        const Geom& g = lv_[0].g;
        const Stencil st = stencil();
        T* pnew = from_p ? p2_ : p_;
        if (DIM == 2) {
            // z, p_old, codes (and the three coefficients) in; p, Ap out
            const double nb = st.vd ? 7.0 * sizeof(T) + 1.0 : 4.0 * sizeof(T) + 1.0;
            UAAMG_LAUNCH((KTag{K_PMATVEC, 0, cells(g) * nb}), k_pmatvec_2d<T>, flat2d_grid(g),
                         dim3(32, 8), g, lv_[0].code, z_, from_p ? p_ : p2_, pnew, ap_, st,
                         partials_, cg_);
        } else {
            MarchMaps pm = maps<DIM>(0, true, false);  // z and the current search direction
            pm.v[0] = lv_[0].mx;
            pm.v[1] = from_p ? map_p_ : map_p2_;
            const KTag tag{K_PMATVEC, 0, cells(g) * (4.0 * sizeof(T) + 1.0)};
            const int zc = pm_zc_;
            if (dirichlet_)
                UAAMG_LAUNCH_SMEM(tag, (k_pmatvec<DIM, T, true>), march_grid<DIM>(g, zc),
                                  dim3(kThreads), (PmvCfg<DIM, T>::BYTES), pm, g, zc, pnew, ap_, st,
                                  partials_, cg_, err_);
            else
                UAAMG_LAUNCH_SMEM(tag, (k_pmatvec<DIM, T, false>), march_grid<DIM>(g, zc),
                                  dim3(kThreads), (PmvCfg<DIM, T>::BYTES), pm, g, zc, pnew, ap_, st,
                                  partials_, cg_, err_);
        }
        const long long nvec = (long long)g.n / Vec16<T>::N;
        // x_lo, r, p, Ap in; x_lo, r out (a fold after a replacement adds x_hi in and out)
        UAAMG_LAUNCH((KTag{K_UPDATE, 0, cells(g) * (6.0 * sizeof(T))}), k_update_flat<T>,
                     update_blocks(nvec), 256, nvec, xlo_, r_, pnew, ap_, mixed_ ? xd_ : nullptr,
                     partials_, cg_, cur_.hist);
        if (mixed_) {
            // residual replacement (when due, one iteration in replace_every; the others
            // return at once): b, x_hi, x_lo, codes in; r out
            nopdl_next_ = cells(g) > 1048576.0;
            const KTag tag{K_REPLACE, 0, cells(g) * (17.0 + 2.0 * sizeof(T))};
            if constexpr (DIM == 3) {
                if (dirichlet_) resid_march<true, false>(tag, nullptr);
                else resid_march<false, false>(tag, nullptr);
            } else {
                UAAMG_LAUNCH(tag, (k_resid_x64<DIM, T>), resid_grid(g), dim3(32, 8), g, lv_[0].code, b64_,
                             xd_, xlo_, r_, st, kResidZc, partials_, cg_, 5, 1, cur_.tol, cur_.tol_mode,
                             gref_, (double*)nullptr);
            }
        }
    }

    // The FP64 residual march: a replacement, or (EXIT) a solve's end, adding x to dst.
    template <bool DIRW, bool EXIT>
    void resid_march(const KTag& tag, double* dst) {
        const Geom& g = lv_[0].g;
        MarchMaps rm;
        rm.v[0] = map_b64_;
        rm.v[1] = map_xd_;
        rm.v[2] = map_xlo_;
        rm.code = lv_[0].mcode;
        UAAMG_LAUNCH_SMEM(tag, (k_resid_march<T, DIRW, EXIT>), march_grid<3>(g, rx_zc_), dim3(kThreads),
                          (RxCfg<T>::BYTES), rm, g, rx_zc_, r_, stencil(), partials_, cg_, 5, cur_.tol,
                          cur_.tol_mode, err_, gref_, dst);
    }

    template <int DIM>
    int begin_impl(const SolveArgs& a) {
        cur_ = a;
        const Geom g = lv_[0].g;
        const uint8_t* s = lv_[0].solid;
        const dim3 vb(32, 8);
        const dim3 vg = vec_grid(g);
        const int n = g.n;
        if (DIM == 2 && sizeof(T) == 4 && vd_ && vox_ && voy_ && vconv_ != vver_) {
            // FP32 copies of the variable-coefficient operator (once per contents)
            if (!vf_[0]) {
                for (int q = 0; q < 3; ++q)
                    if (int e = alloc_extra(vf_[q], (size_t)n)) return e;
                if (gexec_) {  // a captured step holds the copies' (null) pointers
                    cudaStreamSynchronize(st_);
                    cudaGraphExecDestroy(gexec_);
                    gexec_ = nullptr;
                }
                gkey_ = -1;
            }
            UAAMG_LAUNCH((KTag{K_SETUP, 0, cells(g) * 36.0}), k_var_coeffs, vg, vb, g, stencil(),
                         vf_[0], vf_[1], vf_[2]);
            vconv_ = vver_;
        }
        const Stencil st = stencil();

        CGState init = {};
        init.max_iter = a.max_iter;
        init.replace_every = mixed_ ? (a.replace_every > 0 ? a.replace_every : 10) : 0;
        init.breakdown = a.tol_mode == 0 ? 1e-15 : 1e-300;
        init.dirichlet = dirichlet_;
        init.init = 1;
        init.epoch = ++epoch_;
        init.progress = flag_host_;
        init.rr_best = 1e300;
        init.cover = star_ && a.precond ? 1 : 0;  // (plain CG applies no hierarchy)
        *flag_host_ = progress_word(epoch_, 0, 0);
        *cg_host_ = init;
        if (cudaMemcpyAsync(cg_, cg_host_, sizeof(CGState), cudaMemcpyHostToDevice, st_) != cudaSuccess)
            return E_CUDA;
        err_known_ = false;

        // b = -(rhs - mean), re-projected; ||b|| (pcg_3d.cpp:22-36, 80-81); r, x and p
        UAAMG_LAUNCH((KTag{K_RHS, 0, cells(g) * 9.0}), k_rhs_sum<DIM>, vg, vb, g, gref_, s, a.rhs,
                     partials_, cg_, 3, 0, a.hist);
        UAAMG_LAUNCH((KTag{K_RHS, 0, cells(g) * 9.0}), k_rhs_sum<DIM>, vg, vb, g, gref_, s, a.rhs,
                     partials_, cg_, 3, 1, (double*)nullptr);
        UAAMG_LAUNCH((KTag{K_RHS, 0, cells(g) * (25.0 + 3.0 * sizeof(T))}), (k_rhs_write<DIM, T>), vg, vb,
                     g, gref_, s, a.rhs, b64_, a.warm ? (T*)nullptr : r_, xlo_, p_, xd_, partials_, cg_, 4,
                     a.tol, a.tol_mode);
        if (a.warm) {  // b <- b - A x_in: the solve then finds the correction to x_in
            if (a.x_ready) cudaStreamWaitEvent(st_, a.x_ready, 0);
            UAAMG_LAUNCH((KTag{K_RHS, 0, cells(g) * 16.0}), (k_import<DIM, double>), vg, vb, g, gref_, a.x, xd_);
            UAAMG_LAUNCH((KTag{K_TRUE_RESIDUAL, 0, cells(g) * 25.0}), (k_true_residual<DIM, double>), vg, vb,
                         g, s, b64_, xd_, b64_, st, partials_, cg_, 5, 3, a.tol, a.tol_mode);
            UAAMG_LAUNCH((KTag{K_RHS, 0, cells(g) * (9.0 + sizeof(T))}), (k_true_residual<DIM, T>), vg, vb, g, s,
                         b64_, (const double*)nullptr, r_, st, partials_, cg_, 5, 0, a.tol, a.tol_mode);
            cudaMemsetAsync(xd_, 0, (size_t)n * sizeof(double), st_);
        }

        // Two iterations form one step (the search direction is back in p_ after
        // it); outside profiling the step is a CUDA graph captured once per problem
        // and options.
        use_graph_ = graphs_ && !prof_on_;
        if (use_graph_) {
            const long long key = ((long long)a.precond << 2) | (use_tail() ? 2 : 0) | (sweeps_ ? 1 : 0);
            if (!gexec_ || key != gkey_ || a.hist != ghist_) {
                if (gexec_) { cudaGraphExecDestroy(gexec_); gexec_ = nullptr; }
                if (!cap_ && cudaStreamCreateWithFlags(&cap_, cudaStreamNonBlocking) != cudaSuccess)
                    return E_CUDA;
                cudaStream_t saved = st_;
                const long before = launches_;
                st_ = cap_;
                cudaGraph_t graph = nullptr;
                cudaError_t ce = cudaStreamBeginCapture(cap_, cudaStreamCaptureModeThreadLocal);
                if (ce == cudaSuccess) {
                    cg_iteration<DIM>(true);
                    cg_iteration<DIM>(false);
                    ce = cudaStreamEndCapture(cap_, &graph);
                }
                st_ = saved;
                if (ce == cudaSuccess && graph) {
                    ce = cudaGraphInstantiate(&gexec_, graph, 0);
                    if (ce != cudaSuccess) gexec_ = nullptr;
                    cudaGraphDestroy(graph);
                }
                // A capture that another thread broke (a device synchronisation): this solve
                // launches its kernels one by one.
                if (!gexec_) {
                    cudaGetLastError();
                    use_graph_ = false;
                }
                glaunches_ = launches_ - before;
                launches_ = before;
                gkey_ = key;
                ghist_ = a.hist;
            }
        }
        it_ = 0;
        nstep_ = 0;
        seen_ = 0;
        stopped_ = false;
        return E_OK;
    }

    // Queues one step (two iterations) unless max_iter is reached.  Kernels queued after
    // the solve stopped return at once.
    template <int DIM>
    int step_impl() {
        // at most two steps ahead of what has been polled
        if (it_ >= cur_.max_iter || nstep_ - seen_ >= 2) return E_OK;
        if (use_graph_) {
            if (cudaGraphLaunch(gexec_, st_) != cudaSuccess) return E_CUDA;
            launches_ += glaunches_;
        } else {
            cg_iteration<DIM>(true);
            if (it_ + 1 < cur_.max_iter) cg_iteration<DIM>(false);
        }
        it_ += 2;
        ++nstep_;
        return E_OK;
    }

    template <int DIM>
    int end_enqueue() {
        const Geom g = lv_[0].g;
        const dim3 vb(32, 8);
        const dim3 vg = vec_grid(g);
        const Stencil st = stencil();
        const SolveArgs& a = cur_;
        // exit diagnostics, the FP64 true residual of the accumulated solution (x_hi + x_lo in
        // mixed mode, else the working x; x_hi is 0 then), and that solution out
        const double xb = (mixed_ ? 8.0 : 0.0) + sizeof(T);
        if (a.x_ready) cudaStreamWaitEvent(st_, a.x_ready, 0);  // the caller's x, accumulated into
        const KTag tag{K_TRUE_RESIDUAL, 0, cells(g) * (25.0 + xb)};
        if constexpr (DIM == 3) {
            if (dirichlet_) resid_march<true, true>(tag, a.x);
            else resid_march<false, true>(tag, a.x);
        } else {
            UAAMG_LAUNCH(tag, (k_resid_x64<DIM, T>), resid_grid(g), dim3(32, 8), g, lv_[0].code, b64_,
                         mixed_ ? xd_ : (double*)nullptr, xlo_, (T*)nullptr, st, kResidZc, partials_, cg_,
                         5, 2, a.tol, a.tol_mode, gref_, a.x);
        }
        if (a.project_mean && a.ref_solid) {
            const dim3 rg = vec_grid(gref_);
            UAAMG_LAUNCH((KTag{K_OUTPUT, 0, cells(g) * 9.0}), k_sum_count<DIM>, rg, vb, gref_, a.ref_solid,
                         a.x, partials_, cg_, 3);
            UAAMG_LAUNCH((KTag{K_OUTPUT, 0, cells(g) * 17.0}), k_sub_mean<DIM>, rg, vb, gref_, a.ref_solid,
                         a.x, cg_);
        }
        if (cudaMemcpyAsync(cg_host_, cg_, sizeof(CGState), cudaMemcpyDeviceToHost, st_) != cudaSuccess)
            return E_CUDA;
        return E_OK;
    }
};

#undef UAAMG_LAUNCH
#undef UAAMG_LAUNCH_SMEM

}  // namespace
}  // namespace uaamg
