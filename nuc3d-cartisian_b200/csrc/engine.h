// Engine: the host side of the batched solver.  Owns the boxes' device
// memory, the device box table, the per-kernel work-item lists and a CUDA
// graph of one TVD-RK3 step of every active box.  Internal; nuc3d_ctx and
// nuc3d_batch in the C ABI are thin handles over it.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <string>
#include <vector>

#include "nuc3d_b200.h"
#include "rhs_kernels.h"
#include "spectra_kernels.h"

namespace nuc3d {

struct EngineBox {
    nuc3d_box_desc desc{};
    BoxDev dev{};          // host copy of the box's table entry
    int prim_off = 0, prim_n = 0;  // the box's k_prim work items (set by rebuild)
    void *mem = nullptr;   // one stream-ordered allocation holding all fields
    void *force_mem = nullptr;  // spectral forcing scratch (forced boxes only)
    size_t bytes = 0;      // of mem and force_mem
    double cfl = 0.5;
    long long steps = 0;   // host mirror of the device step counter
    bool live = false;     // slot in use
};

class Engine {
public:
    Engine(int precision, cudaStream_t stream);
    ~Engine();

    // Adds a box (allocates its device memory, stream-ordered); returns slot id.
    int add_box(const nuc3d_box_desc &d, int *id);
    int remove_box(int id);
    int set_active(int id, bool on);
    int set_cfl(int id, double cfl);
    // host transfers in the device's copy lanes (see chained_host_copy)
    bool copy_lane = false;
    int set_state(int id, const double *const q[5], cudaMemcpyKind kind, bool sync);
    int get_state(int id, double *const q[5], cudaMemcpyKind kind, bool sync);
    // nsteps TVD-RK3 steps of every active box (graph replay unless profiling)
    int step(int nsteps);
    // dt / residual history of the last `n` steps of box id into host arrays
    int history(int id, int n, double *h_dt, double *h_res);
    int rhs(int id, double *const d_rhs[5], double *h_dt_local);
    // Initial state of box id generated on the device (Taylor-Green or HIT);
    // info (may be null): u_rms, Taylor microscale, Reynolds number.  A HIT
    // request with re_lambda > 0 also sets the box's Reynolds number.
    int init_state(int id, const nuc3d_init_desc &in, double info[3]);
    // Turbulence statistics of box id's current state (NUC3D_STATS values).
    int stats(int id, double out[26]);
    // the nine shell spectra of box id into out[9 * kmax] (host); *kmax_out
    // receives kmax = min(nx, ny, nz)/2.  out may be NULL to query kmax.
    int spectra(int id, double *out, int *kmax_out);
    int sync_and_check(int id_or_all);
    double time(int id);
    long long box_steps(int id) const;
    double reynolds(int id) const {
        return id >= 0 && id < (int)boxes_.size() && boxes_[id].live ? boxes_[id].dev.p.reynolds : 0.0;
    }
    int nboxes() const { return (int)boxes_.size(); }
    int precision() const { return precision_; }
    cudaStream_t stream() const { return stream_; }

    // accounting
    long long launches = 0;
    long long graph_captures = 0;  // step graphs captured (one per membership change)
    bool prof_on = false;
    double prof_ms[NUC3D_PROF_CLASSES] = {};
    long long prof_n[NUC3D_PROF_CLASSES] = {};
    int profile_flush();
    // autotuned sweep variant (tile length and run length, kInvTileCells /
    // kInvRunLen) per [scheme JS/Z/-/W7][dir] (-1: not tuned yet) and the
    // milliseconds per launch of each variant when it was last timed (0: not)
    int inv_variant[kSchemes][3] = {{-1, -1, -1}, {-1, -1, -1}, {-1, -1, -1},
                                    {-1, -1, -1}, {-1, -1, -1}, {-1, -1, -1},
                                    {-1, -1, -1}, {-1, -1, -1}, {-1, -1, -1}};
    double inv_tune_ms[kSchemes][3][kInvVariants] = {};
    // faces per thread and cells per tile of variant v (marched pairs: both are
    // the chunk length)
    int sweep_run(int s, int d, int v) const {
        return marched(s, d, precision_ == NUC3D_MIXED) ? march_cells(d, v) : kInvRunLen[v];
    }
    int sweep_tile(int s, int d, int v) const {
        return marched(s, d, precision_ == NUC3D_MIXED) ? march_cells(d, v) : kInvTileCells[v];
    }
    // autotuned pencil depth of the 2.5-D stencil kernels: index into
    // kPencilDepths (-1: not tuned yet), the measured milliseconds of one
    // viscous-flux + update pass per depth of the last tuning (0: not timed), and
    // the depth found for each power of four of active cells, with and without
    // the short depths and for each power of two of the tiles' mean planes up to
    // 64 (flat boxes cannot tell the depths beyond their own extent apart).  A
    // batch that grows or shrinks into a class it has been in takes its depth.
    int pencil_variant = -1;
    double pencil_tune_ms[kPencils] = {};
    static constexpr int kSizeClasses = 20;  // floor(log4(cells))
    static constexpr int kPlaneClasses = 4;  // 8, 16, 32, 64 planes and more
    signed char pencil_of_class[2][kPlaneClasses][kSizeClasses];

    static long long box_bytes(const nuc3d_box_desc &d);
    static int validate(const nuc3d_box_desc &d, std::string *why);

private:
    // issues this engine's copies of a host<->device state transfer (dir 0:
    // upload, 1: download) after the last such transfer any engine on the
    // device issued in that direction (copy lanes, engine.cu)
    int chained_host_copy(int dir, int id, double *const host[5]);
    int rebuild();
    // launches of one step into stream s (eager on stream_, or on the private
    // capture stream while recording the graph)
    int enqueue_step(cudaStream_t s);
    template <typename B>
    int enqueue_step_t(cudaStream_t s);
    template <typename B>
    int enqueue_rhs_t(int id, double *const d_rhs[5]);
    template <typename B>
    cudaError_t enqueue_forcing(cudaStream_t st);
    // the 2.5-D kernels of both stencil classes at pencil-depth variant v
    template <typename B>
    cudaError_t launch_visc_classes(int v, cudaStream_t st);
    template <typename B>
    cudaError_t launch_update_classes(int v, StageArgs sa, cudaStream_t st);
    void invalidate_graph();
    int autotune();
    static int size_class(long long cells);
    // the pair's variant from now on (marched pairs: at this size)
    void keep_variant(int s, int d, int v);

    // stream-ordered device memory from the pool that the engines of a device
    // share (DevicePool, engine.cu)
    cudaError_t device_alloc(void **p, size_t bytes);
    template <typename T>
    cudaError_t device_alloc(T **p, size_t bytes) {
        return device_alloc(reinterpret_cast<void **>(p), bytes);
    }
    cudaMemPool_t pool_ = nullptr;  // null: none could be made, the default pool serves
    SpectraPlan spectra_plan_;  // of the last box size asked for

    int precision_;
    cudaStream_t stream_;
    std::vector<EngineBox> boxes_;
    bool dirty_ = true;
    bool any_visc_ = false;
    int nactive_ = 0;
    BoxDev *d_boxes_ = nullptr;
    int d_boxes_cap_ = 0;
    WorkItem *d_items_ = nullptr;
    size_t d_items_cap_ = 0;
    // offsets/counts into d_items_
    struct Range {
        size_t off = 0;
        int n = 0;
    };
    Range r_prim_;
    Range r_inv_[kSchemes][3][kInvTileClasses];  // [scheme id][dir][32/64-cell tiles]
    // marched pairs (marched()): the work items of each variant, and the length
    // that its boxes' lines share (items are line groups, one list for all
    // variants) or 0 (lines of several lengths: items are the groups' chunks,
    // so that a long box adds no empty ones to the others).  A variant
    // has a list if it may be the pair's best: the chosen one alone once there is
    // one, else the longest chunks and the next shorter ones while the longer
    // make fewer than kChunkUnits (eight waves of 148 SMs x 4 units, whose tail
    // costs less than the shorter chunks' extra overlap)
    static constexpr long long kChunkUnits = 8 * 148 * 4;
    Range r_march_[kSchemes][3][kInvVariants];
    int march_n_[kSchemes][3] = {};
    // The variant found for each power of four of a marched pair's cells and for
    // lines below 32, below 128 and longer: the best chunk grows with both (see
    // kMarchLen), so what small boxes were tuned to does not stay for large ones.
    // -1: not tuned yet.  variant_slot_: the current batch's entry.
    signed char variant_of_class_[kSchemes][3][3][kSizeClasses];
    signed char *variant_slot_[kSchemes][3] = {};
    bool has_sweep(int s, int d) const {
        for (int v = 0; v < kInvVariants; ++v)
            if (has_list(s, d, v)) return true;
        return false;
    }
    // variant v of the pair can be launched on this batch's boxes
    bool has_list(int s, int d, int v) const {
        return r_inv_[s][d][inv_tile_class(v)].n > 0 || r_march_[s][d][v].n > 0;
    }
    // line groups of the CRWENO5 sweeps that march (thomas_lines_of)
    Range r_thomas_[3];
    bool any_thomas() const { return r_thomas_[1].n > 0 || r_thomas_[2].n > 0; }
    // the line-solve schemes' sweeps along d
    template <typename B>
    cudaError_t launch_lines(int d, int in, int prim_mode, cudaStream_t st);
    // variant v of the directional sweep of scheme s on this batch's boxes
    template <typename B>
    cudaError_t launch_sweep(int s, int d, int v, int in, int prim_mode, cudaStream_t st);
    // 2.5-D stencil tiles per [stencil class (kVisReach)][pencil depth of
    // kPencilDepths]; the short depths' lists only where short_pencils_
    Range r_25d_[kVisClasses][kPencils];
    bool short_pencils_ = false;
    int plane_class_ = 0;
    long long active_cells_ = 0;
    // blocks up to which the short pencils are worth timing: two waves of 148
    // SMs x 2 blocks at depth 16
    static constexpr long long kPencilShortBlocks = 600;
    // Short depths are gone into only if the pass at 8 planes is this much faster
    // than at 16.  Where they tie, the short one loses in the step, whose sweeps run
    // beside the viscous fluxes and share HBM with its deeper halos: two steps of
    // 160 x 100 x 60 FP64 1478 against 1450 us at 16 planes, of 90 x 150 x 70 hccs
    // mixed 3512 against 3478.  Boxes that the short depths are for gain 10 to 50 % of the pass.
    static constexpr double kShortPencilGain = 0.97;
    int pv() const { return pencil_variant < 0 ? 0 : pencil_variant; }
    // Mixed precision stages each line's split fluxes as FP32 offsets from
    // their value at the tile's first cell, so the rounding depends on where
    // tiles start: only the 32-cell tiles run there, which keeps every
    // variant (and a box alone or in any batch) bitwise the same.
    bool mixed_tiles_only32() const { return precision_ == NUC3D_MIXED; }
    // line-solve tiles per [line scheme: 0 crweno5, 1 hccs, 2 hccs77][dir],
    // with the longest line and the rows per lane that size each launch's
    // shared memory
    Range r_cr_[kLineSchemes][3];
    int cr_nmax_[kLineSchemes][3] = {}, cr_ms_[kLineSchemes][3] = {};
    int launches_per_step_ = 0;
    cudaGraph_t graph_ = nullptr;
    cudaGraphExec_t exec_ = nullptr;
    cudaStream_t cap_stream_ = nullptr;  // graphs cannot be captured on the legacy stream
    cudaStream_t fork_stream_ = nullptr;  // the captured step's viscous-flux branch
    cudaEvent_t fork_ev_[2] = {nullptr, nullptr};  // fork after the x sweep, join before the update
    unsigned *h_flags_ = nullptr;      // mapped page-locked mirror of the boxes' flags
    unsigned *h_flags_dev_ = nullptr;  // its device address
    int h_flags_cap_ = 0;
    int device_ = 0;                      // the device current at construction
    cudaEvent_t copy_ev_[2] = {nullptr, nullptr};  // this engine's last upload / download
    double **d_rhs_ptrs_ = nullptr;  // 5 per box, for stage -1
    double *d_stats_ = nullptr;       // statistics scratch
    // profiling events
    std::vector<cudaEvent_t> ev_pool_;
    struct Mark {
        int cls;
        cudaEvent_t a, b;
    };
    std::vector<Mark> pending_;
    size_t ev_next_ = 0;
    friend struct ProfScope;
};

}  // namespace nuc3d
