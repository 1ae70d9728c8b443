// dg_host.h -- host-side state of the GB300 rasterizer, shared by the C ABI
// (dg_api.cu) and the render server (dg_server.cu): scene and camera state,
// resident resources, the per-frame host setup of Scene::render and the
// launch of one render job on a job slot.
//
// Host floating point follows the reference's Rust semantics: the files
// including this header are compiled with -ffp-contract=off, so every
// expression rounds each operation to f32 in source order.
#pragma once

#include <cmath>
#include <cstring>
#include <vector>

#include "dg_internal.cuh"

namespace dgh {

// ------------------------------------------------------------ host vectors
struct HV3 {
    float x, y, z;
};
inline HV3 h3(float x, float y, float z) { return HV3{x, y, z}; }
inline HV3 hadd(HV3 a, HV3 b) { return h3(a.x + b.x, a.y + b.y, a.z + b.z); }
inline HV3 hsub(HV3 a, HV3 b) { return h3(a.x - b.x, a.y - b.y, a.z - b.z); }
inline HV3 hmul(HV3 a, float s) { return h3(a.x * s, a.y * s, a.z * s); }
inline HV3 hdiv(HV3 a, float s) { return h3(a.x / s, a.y / s, a.z / s); }
inline float hdot(HV3 a, HV3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }       // linalg.rs:182-184
inline float hnorm(HV3 a) { return std::sqrt(a.x * a.x + a.y * a.y + a.z * a.z); }  // linalg.rs:167-171
inline HV3 hnormalized(HV3 a) { return hdiv(a, hnorm(a)); }                           // linalg.rs:173-175
inline HV3 hcross(HV3 a, HV3 b) {                                                      // linalg.rs:186-200
    return h3((a.y * b.z) - (a.z * b.y), (a.z * b.x) - (a.x * b.z), (a.x * b.y) - (a.y * b.x));
}

struct HM4 {
    float m[4][4];
};

struct Camera {  // scene/mod.rs:282-294
    HV3 position, direction, up;
    float top, bottom, right, left;
    float near_, far_;
    HV3 u, v, w;
};

struct Scene {  // scene/mod.rs:749-757
    uint64_t width = 0, height = 0;
    Camera cam;
    std::vector<int32_t> objects;
    std::vector<HV3> lights;
    int32_t exponent = 2;
    int32_t interpolation = DG_INTERP_AFFINE;  // extension (dg_scene_set_interpolation)
};

dg_status camera_init(Camera& c, HV3 pos, HV3 dir, float ratio, float near_, float far_, float fov_x);
void camera_update_basis(Camera& c);
dg_status camera_op(Scene& s, int32_t op, const float* a);
// gen_transformation_matrix (scene/mod.rs:817-899) and gen_view_planes (:481-593).
dg_status frame_setup(Scene& s, float M[4][4], float planes[6][4]);

// ------------------------------------------------------------- resources
struct TexMap {
    uint32_t* d_words = nullptr;
    uint64_t len = 0;
    uint32_t w = 0, h = 0, comps = 0;
    uint32_t filter = DG_FILTER_NEAREST;  // extension (dg_texmap_set_filter)
};

struct Object {
    bool alive = false;
    float4* d_pos = nullptr;
    float4* d_nrm = nullptr;
    float2* d_uv = nullptr;
    uint4* d_tri_pos = nullptr;
    uint4* d_tri_uv = nullptr;
    uint4* d_tri_nrm = nullptr;
    DgMatDev* d_mats = nullptr;
    uint32_t nv = 0, nn = 0, nuv = 0, ntri_opaque = 0, nmats = 0;
    // Transparent meshes (object.rs:45-53: material alpha < 1), concatenated in
    // mesh order: mesh m holds triangles [tmesh_off[m], tmesh_off[m + 1]) as
    // (position indices, material), (uv indices, m), (normal indices). The
    // painter's sort of every frame reorders each mesh and the order persists
    // (scene/mod.rs:1100-1115): d_tt[tcur] holds the current order, and a
    // render writes the next one into d_tt[1 - tcur].
    uint4* d_tt[2][3] = {};
    int tcur = 0;
    uint32_t nt = 0;
    std::vector<uint32_t> tmesh_off;
    uint32_t* d_tmesh_off = nullptr;
    uint32_t tmesh_max = 0;  // triangles of the largest transparent mesh
};

struct Canvas {
    bool alive = false;
    uint64_t w = 0, h = 0;
    uint32_t* d_colour = nullptr;
    float* d_depth = nullptr;
    uint64_t* d_vis = nullptr;
    uint32_t* d_cells = nullptr;  // DgFrameDev::cells; zeroed at allocation
    uint32_t epoch = 0;           // advanced for every frame rendered into the canvas
    bool depth_init = false;
    float depth_max = 0.0f;
    float off_x = 0.0f, off_y = 0.0f;
    // dg_canvas_read_async: the copy runs on the context's copy stream after
    // ev_rendered; ev_read marks its end. While read_pending, the next operation
    // that looks the canvas up first makes the context stream wait for ev_read.
    cudaEvent_t ev_rendered = nullptr, ev_read = nullptr;
    uint32_t* h_err = nullptr;  // pinned: the error word copied with the frame
    bool read_pending = false;
};

// The buffers one frame renders into.
struct FrameTarget {
    uint32_t* colour;
    float* depth;
    uint64_t* vis;  // all DG_VIS_EMPTY on entry; left so on exit
    uint64_t w, h;
    float clear_depth;
    float off_x, off_y;
    uint32_t* cells;  // DgFrameDev::cells (or null)
    uint32_t epoch;   // differs from the frame's other renders into the same cells
};

// Whether a frame of this many opaque triangles, vertices, lights and pixels gets
// DG_FRAME_LAZY: at least as many triangles as pixels, and a light/halfway table (32
// bytes per vertex and light) beyond the L2. The small triangles then get no rows and
// no records, and the pixels they win are shaded from the mesh. Measured without the
// rows alone: the 3840x2160 frame of 10M micro triangles and 4 lights gained 5% (most
// of its triangles win no pixel); a 256x256 frame of a 300k-triangle mesh and 1 light
// (a 5 MB table) lost 14%, so it keeps both. k_setup_lean has the figures without the
// records.
inline bool dg_frame_lazy(uint64_t tris, uint64_t vertices, uint64_t lights, uint64_t pixels) {
    return tris >= pixels && vertices * lights * 32u >= (128ull << 20);
}

// Words of DgFrameDev::cells for a w x h canvas.
inline uint64_t dg_cell_count(uint64_t w, uint64_t h) { return ((w + 31u) / 32u) * ((h + 31u) / 32u); }

// Scratch, staging and stream of one render job in flight. The context owns
// one; the render server owns one per concurrent batch.
struct JobSlot {
    cudaStream_t stream = nullptr;
    uint16_t* d_vmask = nullptr;  // plane-sign masks of the job's vertices
    size_t vmask_cap = 0;
    float4* d_vrec = nullptr;  // vertex records (screen centre, eye distance, masks)
    size_t vrec_cap = 0;
    float4* d_vshade = nullptr;
    size_t vshade_cap = 0;
    uint8_t* d_vmark = nullptr;  // zeroed at allocation; the queue pass clears what setup sets
    size_t vmark_cap = 0;
    DgQueueRec* d_queue = nullptr;
    DgSmallRec* d_small = nullptr;  // small-triangle list
    size_t small_cap = 0;
    // transparent pass scratch (DgJobDev)
    uint64_t* d_tkey[2] = {};
    uint32_t* d_tval[2] = {};
    size_t tsort_cap = 0;
    DgTriRec* d_ttrec = nullptr;
    uint4* d_tbox = nullptr;
    uint2* d_tmeta = nullptr;
    float* d_talpha = nullptr;
    size_t tout_cap = 0;  // clip outputs the arrays above hold
    uint4* d_titem = nullptr;
    size_t titem_cap = 0;
    uint4* d_fnode = nullptr;
    size_t fnode_cap = 0;
    uint32_t* d_fhead = nullptr;  // zeroed at allocation; the fold clears what the raster sets
    size_t fhead_cap = 0;
    uint32_t* d_hist = nullptr;
    size_t hist_cap = 0;  // entries
    uint2* d_items = nullptr;  // raster work items
    size_t queue_cap = 0;
    size_t items_cap = 0;
    uint32_t* d_surv = nullptr;  // cull survivors
    size_t surv_cap = 0;
    uint32_t* d_rest = nullptr;  // DgJobDev::rest (grown only for lazy jobs)
    size_t rest_cap = 0;
    uint32_t* d_rec_of = nullptr;  // first triangle record of each survivor
    size_t rec_of_cap = 0;
    DgTriRec* d_trec = nullptr;
    size_t trec_cap = 0;
    float4* d_trec_w = nullptr;  // perspective weights per record (grown only for perspective frames)
    size_t trec_w_cap = 0;
    float4* d_ttrec_w = nullptr;  // the same for the transparent records
    size_t ttrec_w_cap = 0;
    uint32_t small_max_px = DG_SMALL_MAX_PX_AUTO;  // dg_tuning knobs
    uint32_t setup_blocks_per_sm = DG_SETUP_BLOCKS_PER_SM;
    uint32_t queue_blocks_per_sm = DG_QUEUE_BLOCKS_PER_SM;
    uint32_t cull_blocks_per_sm = DG_CULL_BLOCKS_PER_SM;
    uint32_t tile_rows = 0;  // 0: chosen per job (build_job)
    uint32_t item_units = DG_ITEM_UNITS;
    uint32_t record_limit = 0;
    // Two sets of job counters (DG_CNT_*, DG_NCOUNTERS words each): jobs alternate,
    // and a job's first kernel zeroes the other set for the job after it. A third
    // one is for jobs that the caller captures into a graph, which zero it themselves.
    static const int kCapturedSet = 2;
    unsigned long long* d_counters = nullptr;
    int cnt_set = 0;   // the next job's set
    int last_set = 0;  // the last job's set
    uint32_t* d_err = nullptr;
    static const int kStage = 4;  // pinned staging ring for job descriptors
    void* h_stage[kStage] = {};
    void* d_stage[kStage] = {};
    size_t stage_cap[kStage] = {};    // bytes of d_stage
    size_t h_stage_cap[kStage] = {};  // bytes of h_stage (inline descriptors need none)
    cudaEvent_t stage_ev[kStage] = {};
    int stage = 0;
    // Set when a job may have left state behind that jobs expect to be zero (counters,
    // fhead, vmark): build_job clears it all before the next job.
    bool dirty = false;
    int32_t fail_before = 0;  // dg_ctx_inject_launch_failure, for the next job
    bool timing = false;
    cudaEvent_t ev[DG_NKERNELS + 1] = {};
    bool ev_valid = false;
    uint64_t last_vtx = 0, last_tri = 0, last_h2d = 0, last_launches = 0;
    uint64_t last_tile_rows = 0, last_small_max_px = 0;  // the last job's resolve tile height, first frame's threshold
    uint64_t scratch_bytes = 0;  // device bytes held by the scratch buffers
};

}  // namespace dgh

namespace dgh {
// Scratch of dg_canvas_draw_triangles_2d (grow-only, on the context stream).
struct OverlaySlot {
    // One batch's upload: the node counter (16 bytes, zero), 96 bytes of vertices
    // and 16 of box per triangle, 8 per work item. Built in a ring of pinned
    // buffers, so a call neither waits for the frame before it nor stages its
    // copies from pageable memory.
    uint8_t* d_in = nullptr;
    size_t in_cap = 0;
    static const int kStage = 4;
    void* h_stage[kStage] = {};
    size_t stage_cap[kStage] = {};
    cudaEvent_t stage_ev[kStage] = {};
    int stage = 0;
    std::vector<uint4> box;
    uint4* d_node = nullptr;
    size_t node_cap = 0;
    uint32_t* d_head = nullptr;  // zeroed at allocation; the fold clears what the raster sets
    size_t head_cap = 0;
    bool dirty = false;        // a batch may have left heads behind: cleared before the next one
    bool fail_launch = false;  // dg_ctx_inject_launch_failure, for the next batch
    uint32_t* d_rgba = nullptr;  // staging of dg_canvas_read_rgba
    size_t rgba_cap = 0;
};
}  // namespace dgh

struct dg_ctx {
    int device = 0;
    int nsm = 152;
    cudaStream_t own_stream = nullptr;
    cudaStream_t copy_stream = nullptr;  // device-to-host copies of dg_canvas_read_async
    std::vector<dgh::TexMap> tex;  // [0] = 1x1 white default map
    DgTexDev* d_tex = nullptr;
    size_t d_tex_cap = 0;
    bool tex_dirty = true;
    std::vector<dgh::Object> objects;
    std::vector<dgh::Scene> scenes;
    std::vector<dgh::Canvas> canvases;
    dgh::JobSlot main;  // the slot of dg_scene_render / dg_render_batch (main.stream = the context stream)
    dgh::OverlaySlot overlay;
};

namespace dgh {

dg_status set_device(dg_ctx* c);
dg_status slot_init(dg_ctx* c, JobSlot& s, cudaStream_t stream);
void slot_free(JobSlot& s);
// Returns the lowest error code the slot's kernels raised since the last call, and clears it.
dg_status slot_take_errors(JobSlot& s);
// Uploads the texture table if textures were added.
dg_status sync_tex_table(dg_ctx* c, cudaStream_t s);
// Device bytes slot s's scratch will hold after launching a job of V vertices,
// T triangles and L lights per vertex, lazy: one of whose frames is dg_frame_lazy
// (same sizing rules as launch_frames).
uint64_t slot_scratch_after(const JobSlot& s, uint64_t V, uint64_t T, uint32_t L, bool lazy);
// Builds and launches one render job over n frames on slot s (asynchronous).
dg_status launch_frames(dg_ctx* c, JobSlot& s, Scene* const* scenes, const FrameTarget* targets, uint32_t n);

// Host part of one render job: the per-frame and per-segment descriptors (the
// bytes uploaded before the kernels run), the job descriptor the kernels take
// by value (its frames/segs pointers are set by enqueue_job) and the grid sizes.
struct JobBuild {
    bool inline_ok = false;  // set by a caller that can pass the descriptors of a small job inline
    std::vector<DgFrameDev> frames;
    std::vector<DgSegDev> segs;
    size_t fbytes = 0, sbytes = 0;
    DgJobDev job{};
    DgLaunchCfg cfg{};
    uint64_t total_vtx = 0, total_tri = 0, launches = 0;
    bool inline_desc = false;  // the descriptors go as k_vertex's (k_front's) parameter
    std::vector<int32_t> transparent_objects;  // objects whose transparent order the job advances
};
// Host frame setup of every frame (camera basis, matrix, view planes) and the
// scratch sizing of slot s (grows its buffers; synchronizes s only when one grows).
dg_status build_job(dg_ctx* c, JobSlot& s, Scene* const* scenes, const FrameTarget* targets, uint32_t n,
                    JobBuild& b);
// Resolves scene and canvas ids into frames (DG_E_INVALID for a bad id,
// DG_E_DEPTH_UNINIT for a canvas without init_depth).
dg_status resolve_frames(dg_ctx* c, const int32_t* scenes, const int32_t* canvases, uint32_t n,
                         std::vector<Scene*>& sc, std::vector<FrameTarget>& tg);
// dg_scene_render / dg_render_batch on the context's own slot and stream.
dg_status render_job(dg_ctx* c, const int32_t* scenes, const int32_t* canvases, uint32_t n);
// Enqueues the counter reset and the kernels of a built job whose descriptors
// are (or will be, in stream order) at d_stage on the device.
dg_status enqueue_job(JobBuild& b, JobSlot& s, void* d_stage, cudaStream_t stream, bool timing);
// After a job is enqueued: the painter's order it wrote becomes each
// transparent object's current order.
void advance_transparent(dg_ctx* c, const JobBuild& b);

}  // namespace dgh
