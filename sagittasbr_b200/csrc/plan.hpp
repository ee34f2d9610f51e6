// plan.hpp -- the opaque handles behind sbr_scene and sbr_plan.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <memory>
#include <mutex>
#include <vector>

#include "common.hpp"
#include "devpool.hpp"

namespace sbr {
// Streams of a per-angle sweep's launches.  Measured on B200 with 1 / 4 / 8 / 16: plates, 73
// angles x 2 frequencies, 6 bounces, FP32 36.2 / 11.1 / 6.8 / 6.2 ms; sphere, 360 angles, 25 /
// 6.0 / 3.1 / 1.7 ms.
constexpr int kSideStreams = 16;
}

struct sbr_scene {
    int device = 0;
    int num_sms = 0;
    cudaStream_t stream = nullptr;
    int64_t ntris = 0;
    double model_scale = 1.0;
    double aabb_lo[3] = {0, 0, 0}, aabb_hi[3] = {0, 0, 0};  // conservative, FP64
    int64_t nverts = 0;
    // device: one block (nodes to d_cancel), the others apart
    void* block = nullptr;
    sbr::GNode4* d_nodes = nullptr;
    int64_t n_gnodes = 0;
    sbr::GNode8* d_nodes8 = nullptr;  // node_width 8: the same leaves under 8-wide nodes
    int64_t n_gnodes8 = 0;
    int64_t n_bin_nodes = 0;
    sbr::GTri* d_tris = nullptr;
    sbr::GTri64* d_tris64 = nullptr;
    int32_t* d_leaf_of = nullptr;    // with d_tris64, in its block: 4 * node + child of each slot's leaf
    int32_t* d_tri_id = nullptr;
    int32_t* d_tie = nullptr;        // exact-tie ranks (coincident faces of opposite winding), or null
    unsigned long long* d_horizon = nullptr;  // per slot: escape elevations by octant (horizon.cu)
    bool horizon_built = false;      // false: all bytes 255, every ray walks
    int64_t horizon_rays = 0;        // launched without them
    cudaEvent_t horizon_done = nullptr;
    std::mutex horizon_mu;
    float* d_xyz = nullptr;          // caller vertices (unscaled) and triangles
    uint32_t* d_idx = nullptr;
    uint32_t* d_err = nullptr;
    int32_t* d_cancel = nullptr;     // device word polled by the kernels
    cudaStream_t cancel_stream = nullptr;
    cudaStream_t side[sbr::kSideStreams] = {};  // per-angle launches (made by the first such plan)
    std::mutex side_mu;
    int depth = 0;
    double build_ms = 0.0;
    double sah_ms = 0.0;
    // refit: 4-wide node indices grouped by depth (offsets per depth), and the
    // per-triangle box scratch of a refit
    std::vector<int32_t> refit_level_off;
    int32_t* d_refit_nodes = nullptr;
    float* d_tri_box = nullptr;
    int64_t device_bytes = 0;

    sbr::SceneView view() const {
        double reach = 0.0;
        for (int a = 0; a < 3; ++a) reach = std::max(reach, std::max(std::fabs(aabb_lo[a]), std::fabs(aabb_hi[a])));
        return sbr::SceneView{d_nodes, d_tris, d_tris64, d_tri_id, d_nodes8, d_tie, d_horizon, d_leaf_of, float(1.001 * reach)};
    }
};

struct sbr_plan {
    sbr_scene* scene = nullptr;
    int mode = SBR_MODE_BATCHED;
    int prec = SBR_PREC_MIXED;
    int pol = SBR_POL_SCALAR;
    int use_graph = 0;
    int ctas_per_sm = 0;
    int blocks_per_item = 0;
    int node_width = 4;                      // tree the mixed scalar sweep walks
    int num_sms = 0;
    cudaStream_t stream = nullptr;
    sbr::SceneView scene_view{};
    bool multi = false;                      // jobs trace different scenes (JobConst::scene)
    std::vector<sbr::SceneView> scene_views; // multi-scene plans: one per scene
    std::vector<std::pair<sbr_scene*, int64_t>> scene_rays;  // rays launched on each scene
    sbr::SceneView* d_scenes = nullptr;

    std::vector<sbr::Segment> segs;
    std::vector<int64_t> seg_base;     // [n_segs + 1] first item of each segment
    std::vector<sbr::JobConst> jobs;
    std::vector<sbr::FreqConst> freqs;
    std::vector<double> quantum;       // per sample and polarisation
    std::vector<sbr::SegPol> segpol;   // per segment (SBR_POL_HHVV)
    int n_pol = 1;
    int64_t n_segs = 0, n_items = 0, n_samples = 0;
    int64_t n_rays_clipped = 0, n_rays_grid = 0;
    int k_max = 1;
    int persistent_grid = 0;
    int launches = 0;

    // device: the tables, accumulators and results in one block; the raster's buffers in
    // another
    int device = 0;
    void* block = nullptr;
    void* raster_block = nullptr;
    sbr::Segment* d_segs = nullptr;
    int64_t* d_seg_base = nullptr;
    sbr::JobConst* d_jobs = nullptr;
    sbr::FreqConst* d_freqs = nullptr;
    double* d_quantum = nullptr;
    sbr::SegPol* d_segpol = nullptr;
    unsigned long long* d_acc = nullptr;
    unsigned long long* d_acc_stats = nullptr;
    double* d_field = nullptr;
    unsigned long long* d_stats = nullptr;
    unsigned long long* d_queue = nullptr;
    uint32_t* d_err = nullptr;         // this plan's error word; the fields and counters follow it
    bool handed_out = false;           // the caller has the results' device addresses
    size_t results_bytes = 0;          // error word (256 bytes), d_field and d_stats: one copy
    size_t stats_at = 0;               // of d_stats from d_err
    const volatile int32_t* d_cancel = nullptr;
    int64_t device_bytes = 0;

    // first-hit rasterisation: segments are processed in chunks whose first-hit
    // buffers fit `d_zbuf`; each chunk = tile binning + tile raster + trace launch
    struct Chunk {
        int64_t seg_begin, seg_end, item_begin, item_end, zcount, tiles;
    };
    bool raster = false;
    std::vector<Chunk> chunks;
    unsigned long long* d_zbuf = nullptr;
    int64_t zbuf_elems = 0;
    int64_t tiles_max = 0;              // tiles of the largest chunk
    uint32_t tile_cap = 0;              // list entries per tile (longer lists walk)
    uint32_t* d_tile_cnt = nullptr;     // [tiles_max]
    int32_t* d_tile_list = nullptr;     // [tiles_max * tile_cap]

    // per-angle plans: the scene's side streams, and the events of their fork and joins
    const cudaStream_t* side = nullptr;
    int n_side = 0;
    bool forked = false;               // between fork and join
    cudaEvent_t fork = nullptr, join[sbr::kSideStreams] = {};

    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    cudaGraphExec_t graph = nullptr;
    bool executed = false;
};

namespace sbr {

// Receives the host tables of a sweep as build_tables produces them; a sink
// returns false when it has no room left.
struct TableSink {
    virtual ~TableSink() = default;
    virtual bool job(const JobConst& j) = 0;
    virtual bool freq(const FreqConst& f) = 0;
    // one (job, angle) segment, the first item of the next segment, and the job's
    // per-frequency accumulator units (one per output sample of this segment)
    virtual bool segment(const Segment& g, int64_t next_item, const double* quantum, int n_freqs) = 0;
};

struct TableTotals {
    int64_t n_segs = 0, n_items = 0, n_samples = 0, n_rays_clipped = 0, n_rays_grid = 0;
    int k_max = 1;
};

// Argument checks shared by every sweep entry point.
sbr_status validate_run(const sbr_scene* s, const sbr_job* jobs, size_t n_jobs, const sbr_run_opts& o);
// Launcher frames, aperture clipping, work items and fixed-point units of a sweep.
// Job j is clipped against the bounds of job_scene[j] (an index into scenes) when
// job_scene is given, else every job uses scenes[0].
sbr_status build_tables(const sbr_scene* const* scenes, const int32_t* job_scene, const sbr_job* jobs,
                        size_t n_jobs, const sbr_run_opts& o, TableSink& sink, TableTotals& tot);

// Blocks per work item of a segment of a batched sweep, before they are cut down.
inline int auto_run(int blocks) { return blocks / 1024 < 1 ? 1 : blocks / 1024 > 8 ? 8 : blocks / 1024; }
// use_horizons for every scene of the plan.
sbr_status plan_horizons(sbr_plan* pl);
// Makes the scene's side streams follow the plan's stream, and the plan's follow them.
sbr_status plan_fork(sbr_plan* pl);
sbr_status plan_join(sbr_plan* pl);
sbr_status plan_launch(sbr_plan* pl, bool records, sbr_ray_record* d_records);

sbr_status fill_records(sbr_ray_record* d, long long n, cudaStream_t st);
// Traces the listed rays (angle index, i, j; checked by the caller) of a one-job plan.
sbr_status trace_list_launch(sbr_plan* pl, const int32_t* d_rays, long long n, sbr_ray_record* d_out);
int max_freqs_per_job();
int max_lane_channels();  // channels up to which every lane sums its own rays' terms
sbr_status ensure_fp64(sbr_scene* s);
// Triangle records, their FP64 twins and boxes (any may be null) from the scene's
// vertices, on its stream.
sbr_status write_triangles(sbr_scene* s, GTri* tris, GTri64* tris64, float* box);
// 4 * node + child of every slot's leaf, on the scene's stream.
sbr_status write_leaf_of(sbr_scene* s, int32_t* leaf_of);
// Tells the scene that `rays` rays are about to be launched on `stream`; computes its
// horizons there first when they pay by now.
sbr_status use_horizons(sbr_scene* s, int64_t rays, cudaStream_t stream);
// Takes them back, in stream order, so that every ray walks (plans that exist see it).
sbr_status clear_horizons(sbr_scene* s);
}  // namespace sbr
