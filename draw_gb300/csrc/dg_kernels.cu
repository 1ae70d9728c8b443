// dg_kernels.cu -- sm_103a kernels of the GB300 rasterizer.
//
// Pipeline of one render job (one or many frames), all on one stream:
//   k_vertex        per position vertex: eye distance, projected and snapped
//                   screen centre, plane-sign masks (scene/mod.rs:917-926,
//                   :1047-1058, canvas.rs:585-587)
//   k_cull          per input triangle: lateral and near reject from the sign
//                   masks, back-face cull, triangles without area; survivors are
//                   compacted
//   k_setup_lean    (frames of micro triangles) list entries of the small
//                   unclipped survivors, which get no record
//   k_setup_raster  per survivor: near/far clipping, triangle records, bounding
//                   box, edge functions; small triangles go to a list, the others
//                   to the queue (scene/mod.rs:933-1063, canvas.rs:585-681)
//   (k_front        all of these in one kernel, for small jobs)
//   k_queue_raster  light/halfway vectors of the marked vertices, then the small
//                   triangles 32 per warp, then the queued ones by parts of their
//                   boxes, whose covered row spans are finished 32 pixels at a time
//   k_resolve       per 32 x tile_rows tile: a tile that no triangle box reached
//                   (its 32x32 cell lacks the frame's epoch) gets the clear
//                   values without reading its keys; otherwise empty pixels
//                   get the clear colour and depth, covered ones are compacted into the tile's
//                   shade list and their winning fragment is shaded once
//                   (canvas.rs:682-745, 906-930)
//
// Exactness. The reference writes a fragment when its depth is strictly below
// the stored depth (canvas.rs:923) and processes fragments in submission
// order, so the final pixel is the fragment with the smallest
// (depth, submission index) among those with depth < the clear depth. Each
// covered pixel therefore does one 64-bit atomicMin of
// key = (order-preserving depth bits << 32) | (triangle index * 4 + clip output)
// into the canvas's visibility buffer; the result does not depend on thread
// order. Every expression uses __fadd_rn/__fsub_rn/__fmul_rn/__fdiv_rn/
// __fsqrt_rn in the reference's evaluation order (no contraction), Rust's
// saturating float->int casts, and wrapping usize arithmetic for texel offsets.
#include "dg_device.cuh"

#include <nvtx3/nvToolsExt.h>

namespace {

// ================================================================ kernels
// Each pass is a device function over the whole grid (grid-stride or
// block-uniform loops) wrapped by its kernel; the five kernels run as a chain
// with programmatic dependent launch.
// seg(i) and frame(i) give the job's descriptors (from global memory, or from
// the first kernel's parameter for a small job).
#if DG_TIMELINE
// [kernel][first start, first wait passed, last wait passed, last end]
__device__ unsigned long long g_timeline[DG_NKERNELS][4] = {
    {~0ull, ~0ull, 0ull, 0ull}, {~0ull, ~0ull, 0ull, 0ull}, {~0ull, ~0ull, 0ull, 0ull},
    {~0ull, ~0ull, 0ull, 0ull}, {~0ull, ~0ull, 0ull, 0ull}};
__device__ __forceinline__ unsigned long long timeline_now() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// A block's start on construction, its end on destruction (every return path).
struct TimelineBlock {
    int k;
    __device__ explicit TimelineBlock(int kernel) : k(kernel) {
        if (threadIdx.x == 0) atomicMin(&g_timeline[k][0], timeline_now());
    }
    __device__ ~TimelineBlock() {
        if (threadIdx.x == 0) atomicMax(&g_timeline[k][3], timeline_now());
    }
};
__device__ __forceinline__ void timeline_waited(int k) {
    if (threadIdx.x == 0) {
        const unsigned long long t = timeline_now();
        atomicMin(&g_timeline[k][1], t);
        atomicMax(&g_timeline[k][2], t);
    }
}
// k_front does the vertex and cull passes too: each is a point at its first block's
// start, and the kernel itself is the setup pass.
__device__ __forceinline__ void timeline_folded() {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        const unsigned long long t = timeline_now();
        for (int k = 0; k < 2; k++) {
            atomicMin(&g_timeline[k][0], t);
            atomicMax(&g_timeline[k][3], t);
        }
    }
}
#define DG_TL_BLOCK(k) TimelineBlock dg_timeline_block_(k)
#define DG_TL_WAITED(k) timeline_waited(k)
#define DG_TL_FOLDED() timeline_folded()
#else
#define DG_TL_BLOCK(k) ((void)0)
#define DG_TL_WAITED(k) ((void)0)
#define DG_TL_FOLDED() ((void)0)
#endif

// The plane-sign mask of a vertex: bit p: plane p has f > 0; bit 8 + p: f <= 0.
__device__ __forceinline__ uint32_t plane_mask(const DgFrameDev& fr, float4 p4) {
    const V3 p = {p4.x, p4.y, p4.z};
    uint32_t mask = 0;
#pragma unroll
    for (int pl = 0; pl < 6; pl++) {
        const float f = plane_f(fr, pl, p);
        if (f > 0.0f) mask |= 1u << pl;
        if (f <= 0.0f) mask |= 1u << (8 + pl);
    }
    return mask;
}

template <bool MASKS, class SEG, class FRM>
__device__ __forceinline__ void dev_vertex(const DgJobDev& job, uint32_t nsegs, SEG seg, FRM frame) {
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < job.total_vtx; v += stride) {
        uint32_t si = last_le(nsegs, v, [&](uint32_t i) { return seg(i).vtx_begin; });
        const DgSegDev& sg = seg(si);
        const DgFrameDev& fr = frame(sg.frame);
        const float4 p4 = __ldg(sg.pos + (v - sg.vtx_begin));
        const uint32_t mask = plane_mask(fr, p4);
        job.vrec[v] = vertex_screen(fr, p4, mask);
        if (MASKS) job.vmask[v] = (uint16_t)mask;
    }
}

// A job's first kernel: zeroes the counters of the slot's next job (this job's
// were zeroed by the job before it) and, for a small job, writes the descriptors
// of its parameter `in` to job.frames and job.segs.
template <class IN>
__device__ __forceinline__ void begin_job(const DgJobDev& job, const IN& in) {
    if (job.cnt_next && blockIdx.x == 0)
        for (uint32_t i = threadIdx.x; i < DG_NCOUNTERS; i += blockDim.x) job.cnt_next[i] = 0ull;
    if (in.nsegs) {
        constexpr uint32_t fw = sizeof(DgFrameDev) / 8, sw = sizeof(DgSegDev) / 8;
        static_assert(sizeof(DgFrameDev) % 8 == 0 && sizeof(DgSegDev) % 8 == 0, "8-byte words");
        uint2* fd = reinterpret_cast<uint2*>(const_cast<DgFrameDev*>(job.frames));
        uint2* sd = reinterpret_cast<uint2*>(const_cast<DgSegDev*>(job.segs));
        const uint2* fs = reinterpret_cast<const uint2*>(in.frames);
        const uint2* ss = reinterpret_cast<const uint2*>(in.segs);
        const uint32_t nf = in.nframes * fw, stride = gridDim.x * blockDim.x;
        for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nf + in.nsegs * sw; i += stride) {
            if (i < nf)
                fd[i] = fs[i];
            else
                sd[i - nf] = ss[i - nf];
        }
    }
}

template <class IN>
__global__ void __launch_bounds__(256, 8) k_vertex(const __grid_constant__ DgJobDev job,
                                                   const __grid_constant__ IN in) {
    DG_TL_BLOCK(0);
    allow_next_kernel();
    DG_TL_WAITED(0);  // the first kernel of a job waits on nothing (a stream-ordered launch)
    begin_job(job, in);
    if (in.nsegs)
        dev_vertex<true>(job, in.nsegs, [&](uint32_t i) -> const DgSegDev& { return in.segs[i]; },
                   [&](uint32_t i) -> const DgFrameDev& { return in.frames[IN::kFrames == 1u ? 0u : i]; });
    else
        dev_vertex<true>(job, job.nsegs, [&](uint32_t i) -> const DgSegDev& { return job.segs[i]; },
                   [&](uint32_t i) -> const DgFrameDev& { return job.frames[i]; });
}


// Cull pass: one thread per input triangle. A triangle is dropped when one
// lateral plane has all three vertices at f <= 0 (Triangle::clip_against_planes,
// scene/mod.rs:59-66), when all three are at f <= 0 for the near plane (the
// near clip then outputs nothing, :67-87 with ViewPlane::clip :662-690), when it
// faces away from the camera (:1016-1027), or when it is not clipped and provably
// covers no pixel (covers_nothing). All are pure predicates of the triangle, so
// testing them in this order leaves every triangle with a fragment; the plane
// tests read only the vertex records' sign masks. Survivors are
// appended (in any order: the visibility key carries the submission index).
__device__ __forceinline__ bool outside_planes(uint32_t m) { return ((m >> 8) & 0x3Du) != 0u; }
// Triangle::calc_normal and get_center; a triangle is skipped when (cam - centre) . n <= 0.
__device__ __forceinline__ bool faces_camera(const DgFrameDev& fr, V3 a, V3 b, V3 c) {
    const V3 n = vcross(vsub(b, a), vsub(c, b));
    const V3 zero = {0.0f, 0.0f, 0.0f};
    const V3 ctr = vdiv(vadd(vadd(vadd(zero, a), b), c), 3.0f);
    const V3 cam = {fr.cam[0], fr.cam[1], fr.cam[2]};
    return !(vdot(vsub(cam, ctr), n) <= 0.0f);
}

__device__ __forceinline__ void dev_cull(const DgJobDev& job) {
    __shared__ uint32_t s_warp[8];
    __shared__ unsigned long long s_base;
    const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    const uint32_t stride = gridDim.x * blockDim.x;
    // block-uniform loop: survivors are appended with one atomic per block
    for (uint32_t base = blockIdx.x * blockDim.x; base < job.total_tri; base += stride) {
        const uint32_t g = base + threadIdx.x;
        bool keep = false;
        if (g < job.total_tri) {
            const uint32_t si = seg_of_tri(job, g);
            const DgSegDev& sg = job.segs[si];
            const uint4 tp = __ldg(sg.tri_pos + (g - sg.tri_begin));
            const uint16_t* vm = job.vmask + sg.vtx_begin;
            const bool ok = DG_IN_RANGE(tp.x < sg.nv && tp.y < sg.nv && tp.z < sg.nv, job.err);
            const uint32_t m = ok ? (uint32_t)__ldg(vm + tp.x) & (uint32_t)__ldg(vm + tp.y) & (uint32_t)__ldg(vm + tp.z)
                                  : 0xFFFFu;
            if (!outside_planes(m)) {
                const float4 pa = __ldg(sg.pos + tp.x), pb = __ldg(sg.pos + tp.y), pc = __ldg(sg.pos + tp.z);
                const V3 a = {pa.x, pa.y, pa.z}, b = {pb.x, pb.y, pb.z}, c = {pc.x, pc.y, pc.z};
                const DgFrameDev& fr = job.frames[sg.frame];
                keep = faces_camera(fr, a, b, c);
                if (keep && (m & 0x3u) == 0x3u) {  // unclipped: the snapped centres are its own
                    const float4 ra = __ldg(job.vrec + sg.vtx_begin + tp.x), rb = __ldg(job.vrec + sg.vtx_begin + tp.y),
                                 rc = __ldg(job.vrec + sg.vtx_begin + tp.z);
                    keep = !covers_nothing(ra.x, ra.y, rb.x, rb.y, rc.x, rc.y, fr.width, fr.height);
                }
            }
        }
        const unsigned kb = __ballot_sync(FULL, keep);
        if (lane == 0u) s_warp[wid] = (uint32_t)__popc(kb);
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t run = 0;
            for (uint32_t w = 0; w < 8u; w++) {
                const uint32_t c = s_warp[w];
                s_warp[w] = run;
                run += c;
            }
            s_base = run ? atomicAdd(job.cnt + DG_CNT_SURV, (unsigned long long)run) : 0ull;
        }
        __syncthreads();
        if (keep) job.surv[s_base + s_warp[wid] + __popc(kb & ((1u << lane) - 1u))] = g;
        __syncthreads();  // s_warp and s_base are reused by the next iteration
    }
}

__global__ void __launch_bounds__(256) k_cull(const DgJobDev job) {
    DG_TL_BLOCK(1);
    wait_previous_kernel();
    DG_TL_WAITED(1);
    dev_cull(job);
}


// Setup pass over the cull survivors (dense, one per thread): near/far
// clipping, triangle records, bounding boxes and edge functions; tiny
// triangles are rasterized by their warp, the others are queued
// (scene/mod.rs:1029-1063, canvas.rs:585-681).
// Whether a triangle with a box of px pixels goes to the small-triangle list.
__device__ __forceinline__ bool small_listed(const DgFrameDev& fr, const RTri& tr, uint64_t px) {
    return px <= fr.small_max_px && tr.xhi < 65536u && tr.yhi < 65536u && tr.xhi - tr.xlo < 255u &&
           tr.yhi - tr.ylo < 255u && tr.frame < 65536u;
}
__device__ __forceinline__ void store_small(DgSmallRec* s, const RTri& tr) {
    float4* d = reinterpret_cast<float4*>(s);
    d[0] = make_float4(tr.ax, tr.bx, tr.cx, tr.ay);
    d[1] = make_float4(tr.by, tr.cy, tr.da, tr.db);
    reinterpret_cast<uint4*>(s)[2] =
        make_uint4(__float_as_uint(tr.dc), tr.seq, (tr.ylo << 16) | tr.xlo,
                   (tr.frame << 16) | ((tr.yhi - tr.ylo + 1u) << 8) | (tr.xhi - tr.xlo + 1u));
}

// FRONT: the whole front of a small job (k_front): the triangles themselves are
// looped over, and their vertices' masks and screen positions, the plane and the
// back-face tests computed here instead of read from k_vertex's and k_cull's
// results; a triangle's record has its job-wide index.
template <bool FRONT, class SEG, class FRM>
__device__ __forceinline__ void dev_setup(const DgJobDev& job, uint32_t nsegs, SEG seg, FRM frame) {
    __shared__ uint32_t s_records;  // statistics: record requests of the block
    __shared__ uint32_t s_surv;     // statistics: survivors of the block's culling (FRONT)
    __shared__ uint32_t s_nclip;    // clipped survivors the block deferred
    __shared__ uint32_t s_clip_i[DG_CLIP_DEFER], s_clip_g[DG_CLIP_DEFER];  // their survivor slots and indices
    if (threadIdx.x == 0) {
        s_records = 0u;
        s_surv = 0u;
        s_nclip = 0u;
    }
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31u;
    // (in a lazy job, k_setup_lean has taken most survivors and listed the rest)
    const uint32_t* list = job.lazy ? job.rest : job.surv;
    const unsigned long long ns64 = FRONT ? job.total_tri : __ldcg(job.cnt + (job.lazy ? DG_CNT_REST : DG_CNT_SURV));
    const uint32_t nsurv = (uint32_t)(ns64 < job.total_tri ? ns64 : job.total_tri);
    // Pass 0 sets up the survivors, strided over the grid, but defers those that
    // need near/far clipping (up to DG_CLIP_DEFER per block) to pass 1, where the
    // block's warps set them up 32 at a time: the long clip path then runs with
    // all lanes busy instead of holding a warp of mostly unclipped lanes. Both
    // passes are block-uniform (pass 1 starts after a barrier).
    for (int pass = 0; pass < 2; pass++) {
        uint32_t lim = nsurv, start = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u, step = gridDim.x * blockDim.x;
        if (pass == 1) {
            __syncthreads();
            lim = s_nclip < DG_CLIP_DEFER ? s_nclip : DG_CLIP_DEFER;
            start = threadIdx.x & ~31u;
            step = blockDim.x;
        }
        for (uint32_t base = start; base < lim; base += step) {
            bool valid = base + lane < lim;
            uint32_t i = base + lane, g = 0;
            if (pass == 1) {
                i = valid ? s_clip_i[base + lane] : 0u;
                g = valid ? s_clip_g[base + lane] : 0u;
            } else if (valid) {
                g = FRONT ? i : __ldcg(list + i);
            }
            int nout = 0;
            uint32_t si = 0, t = 0, row0 = 0, nrows = 0;
            uint4 tp = make_uint4(0, 0, 0, 0), tuv = tp, tnr = tp;
            float4 r[3];
            bool clipped = false;
            ClipProg P;  // built once per clipped triangle, used by every output
            if (valid) {
                si = last_le(nsegs, g, [&](uint32_t k) { return seg(k).tri_begin; });
                const DgSegDev& sg = seg(si);
                t = g - sg.tri_begin;
                tp = __ldg(sg.tri_pos + t);
                tuv = __ldg(sg.tri_uv + t);  // for the triangle record, loaded alongside the vertex records
                tnr = __ldg(sg.tri_nrm + t);
                if (FRONT) {
                    valid = DG_IN_RANGE(tp.x < sg.nv && tp.y < sg.nv && tp.z < sg.nv, job.err);
                    if (valid) {
                        const DgFrameDev& fr = frame(sg.frame);
                        const float4 pa = __ldg(sg.pos + tp.x), pb = __ldg(sg.pos + tp.y), pc = __ldg(sg.pos + tp.z);
                        const uint32_t ma = plane_mask(fr, pa), mb = plane_mask(fr, pb), mc = plane_mask(fr, pc);
                        // (in pass 1 these hold again: the triangle passed them in pass 0)
                        valid = !outside_planes(ma & mb & mc) &&
                                faces_camera(fr, V3{pa.x, pa.y, pa.z}, V3{pb.x, pb.y, pb.z}, V3{pc.x, pc.y, pc.z});
                        if (valid) {
                            r[0] = vertex_screen(fr, pa, ma);
                            r[1] = vertex_screen(fr, pb, mb);
                            r[2] = vertex_screen(fr, pc, mc);
                            valid = (ma & mb & mc & 0x3u) != 0x3u ||
                                    !covers_nothing(r[0].x, r[0].y, r[1].x, r[1].y, r[2].x, r[2].y, fr.width, fr.height);
                        }
                    }
                } else {
                    triangle_vertices(job, sg, frame(sg.frame), tp, r);
                }
            }
            if (FRONT && pass == 0) {
                const unsigned kept = __ballot_sync(FULL, valid);
                if (kept == 0u) continue;
                if (lane == 0u) atomicAdd(&s_surv, (uint32_t)__popc(kept));
            }
            if (valid) {
                const DgSegDev& sg = seg(si);
                const uint32_t m = __float_as_uint(r[0].w) & __float_as_uint(r[1].w) & __float_as_uint(r[2].w);
                uint32_t dslot = DG_CLIP_DEFER;
                if ((m & 0x3u) == 0x3u) {
                    nout = 1;  // inside near and far: the triangle passes unchanged
                } else if (pass == 0 && (dslot = atomicAdd(&s_nclip, 1u)) < DG_CLIP_DEFER) {
                    s_clip_i[dslot] = i;  // set up in pass 1 (nout stays 0 here)
                    s_clip_g[dslot] = g;
                } else {
                    const DgFrameDev& fr = frame(sg.frame);
                    float4 pa = __ldg(sg.pos + tp.x), pb = __ldg(sg.pos + tp.y), pc = __ldg(sg.pos + tp.z);
                    build_clip(fr, V3{pa.x, pa.y, pa.z}, V3{pb.x, pb.y, pb.z}, V3{pc.x, pc.y, pc.z}, P);
                    nout = P.nout;
                    clipped = true;
                    if (nout > 0 && P.nv > 3) nrows = (uint32_t)(P.nv - 3);  // light rows for the new vertices
                }
                if (nout > 0) {  // its vertices need light/halfway vectors for shading
                    const uint32_t vv[3] = {sg.vtx_begin + tp.x, sg.vtx_begin + tp.y, sg.vtx_begin + tp.z};
                    for (int k = 0; k < 3; k++) job.vmark[vv[k]] = 1u;  // plain stores: every writer writes 1
                }
            }
            // Rows of the light/halfway table for clip vertices, one atomic per warp.
            {
                const unsigned long long r0 = warp_alloc(job.cnt + DG_CNT_VROW, nrows);
                if (nrows != 0u) {
                    if (r0 + nrows <= job.vrow_extra) {
                        row0 = (uint32_t)r0;
                        clip_shade_rows(job, frame(seg(si).frame), P, job.total_vtx + row0);
                    } else {
                        nrows = DG_NONE;  // no room: k_resolve shades these pixels the long way
                    }
                }
            }
            // Triangle records: a triangle with one output uses record i (its survivor
            // slot); the clip outputs of one with more take consecutive records after
            // the first total_tri (one atomic per warp).
            uint32_t rbase = DG_NONE;
            {
                const uint32_t multi = (nout > 1 && nrows != DG_NONE) ? (uint32_t)nout : 0u;
                const unsigned long long rb = (unsigned long long)job.total_tri + warp_alloc(job.cnt + DG_CNT_TRECX, multi);
                if (nout == 1 && nrows != DG_NONE) {
                    if (i < job.trec_cap) rbase = i;
                } else if (multi && rb + (unsigned long long)nout <= job.trec_cap) {
                    rbase = (uint32_t)rb;
                }
            }
            {
                const uint32_t nrec = __reduce_add_sync(FULL, (uint32_t)nout);
                if (lane == 0u && nrec) atomicAdd(&s_records, nrec);  // 32-bit shared atomic, one per warp
            }
            if (valid) job.rec_of[g] = rbase;  // a deferred triangle's entry is rewritten in pass 1

            for (int rr = 0;; rr++) {
                bool has = rr < nout;
                if (__ballot_sync(FULL, has) == 0u) break;
                RTri tr;
                EdgeSet e;
                bool small = false;  // goes to the small-triangle list
                uint32_t nu = 0;     // 32-pixel units of the box to queue (0: not queued)
                bool inplace = false;
                bool boxed = false;  // the triangle has a box (no NaN centre)
                tr.xlo = tr.xhi = tr.ylo = tr.yhi = 0;
                tr.frame = 0;
                if (has) {
                    const DgSegDev& sg = seg(si);
                    const DgFrameDev& fr = frame(sg.frame);
                    tr.frame = sg.frame;
                    tr.seq = ((sg.seq_base + t) << 2) | (uint32_t)rr;
                    if (!clipped) {
                        tr.ax = r[0].x; tr.ay = r[0].y;
                        tr.bx = r[1].x; tr.by = r[1].y;
                        tr.cx = r[2].x; tr.cy = r[2].y;
                        tr.da = r[0].z; tr.db = r[1].z; tr.dc = r[2].z;
                    } else {
                        clip_output_tri(fr, P, rr, r, tr);
                    }
                    bool nan = isnan(tr.ax) || isnan(tr.ay) || isnan(tr.bx) || isnan(tr.by) || isnan(tr.cx) ||
                               isnan(tr.cy);
                    // any NaN centre makes every barycentric NaN: nothing is covered (unclipped
                    // triangles without area were dropped before)
                    if (!nan && !(clipped && covers_nothing(tr.ax, tr.ay, tr.bx, tr.by, tr.cx, tr.cy, fr.width, fr.height))) {
                        bbox_axis(tr.ax, tr.bx, tr.cx, fr.width, tr.xlo, tr.xhi);
                        bbox_axis(tr.ay, tr.by, tr.cy, fr.height, tr.ylo, tr.yhi);
                        boxed = true;
                        make_edges(tr.ax, tr.ay, tr.bx, tr.by, tr.cx, tr.cy, e);
                        const uint64_t px = (uint64_t)(tr.xhi - tr.xlo + 1u) * (uint64_t)(tr.yhi - tr.ylo + 1u);
                        if (rbase != DG_NONE) {
                            float4* wout = (fr.flags & DG_FRAME_PERSPECTIVE) && job.trec_w
                                               ? job.trec_w + rbase + (uint32_t)rr
                                               : nullptr;
                            if (!clipped)
                                write_record(job, job.trec + rbase, sg, tp, tuv, tnr, e, r, fr, wout);
                            else
                                write_clip_record(job, job.trec + rbase + (uint32_t)rr, sg, tp, tuv, tnr, e, tr, P, rr,
                                                  job.total_vtx + row0, fr, wout);
                        }
                        if (rbase == DG_NONE) {
                            inplace = true;
                        } else if (small_listed(fr, tr, px)) {
                            small = true;
                        } else {
                            nu = (uint32_t)((px + DG_UNIT_PX - 1u) / DG_UNIT_PX);
                        }
                    }
                }
                // Every fragment of a triangle lies in its box: mark the box's 32x32 cells in
                // the frame's cell map. A box of more than 16 cells is marked by the whole
                // warp, row by row (a near triangle's box can span the canvas).
                {
                    uint32_t* cells = nullptr;
                    uint32_t ep = 0, cw = 0, ncx = 0, ncy = 0;
                    if (boxed) {
                        const DgFrameDev& fm = frame(tr.frame);
                        cells = fm.cells;
                        ep = fm.epoch;
                        cw = fm.tiles_x;
                        if (cells != nullptr) {
                            ncx = (tr.xhi >> 5) - (tr.xlo >> 5) + 1u;
                            ncy = (tr.yhi >> 5) - (tr.ylo >> 5) + 1u;
                        }
                    }
                    const uint32_t c0 = (tr.ylo >> 5) * cw + (tr.xlo >> 5), ncell = ncx * ncy;
                    if (ncell <= 16u) {
                        for (uint32_t cy = 0; cy < ncy; cy++)
                            for (uint32_t cx = 0; cx < ncx; cx++) cells[c0 + cy * cw + cx] = ep;
                    }
                    unsigned big = __ballot_sync(FULL, ncell > 16u);
                    while (big) {
                        const int L = __ffs(big) - 1;
                        big &= big - 1u;
                        uint32_t* lc = reinterpret_cast<uint32_t*>(
                            __shfl_sync(FULL, (unsigned long long)reinterpret_cast<uintptr_t>(cells), L));
                        const uint32_t ly = __shfl_sync(FULL, ncy, L), lx = __shfl_sync(FULL, ncx, L);
                        const uint32_t l0 = __shfl_sync(FULL, c0, L), lw = __shfl_sync(FULL, cw, L);
                        const uint32_t le = __shfl_sync(FULL, ep, L);
                        for (uint32_t cy = 0; cy < ly; cy++)
                            for (uint32_t cx = lane; cx < lx; cx += 32u) lc[l0 + cy * lw + cx] = le;
                    }
                }
                // Queue the large triangles of this output index with one 64-bit atomic per warp: it hands out
                // the queue records and their work items together; the warp then writes all its
                // items, each lane taking every 32nd.
                // The small-triangle list's atomic (one per warp) is issued first, so that its
                // latency overlaps the queue's.
                const unsigned smask = __ballot_sync(FULL, small);
                unsigned long long sold = 0;
                if (smask && (int)lane == __ffs(smask) - 1)
                    sold = atomicAdd(job.cnt + DG_CNT_SMALL, (unsigned long long)__popc(smask));
                const unsigned qmask = __ballot_sync(FULL, nu != 0u);
                if (qmask) {
                    const uint32_t bw = tr.xhi - tr.xlo + 1u, bh = tr.yhi - tr.ylo + 1u;
                    const uint32_t ni = nu ? dg_item_grid(bw, bh, job.item_log2).n : 0u;
                    uint32_t incl = ni, uincl = nu;
    #pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const uint32_t v = __shfl_up_sync(FULL, incl, o);
                        const uint32_t vu = __shfl_up_sync(FULL, uincl, o);
                        if (lane >= (uint32_t)o) {
                            incl += v;
                            uincl += vu;
                        }
                    }
                    const uint32_t total_items = __shfl_sync(FULL, incl, 31);
                    const uint32_t total_units = __shfl_sync(FULL, uincl, 31);
                    const int leader = __ffs(qmask) - 1;
                    unsigned long long old = 0;
                    if ((int)lane == leader) {
                        old = atomicAdd(job.cnt + DG_CNT_QUEUE,
                                        ((unsigned long long)__popc(qmask) << DG_PACK_SHIFT) | total_items);
                        atomicAdd(job.cnt + DG_CNT_UNITS, (unsigned long long)total_units);
                    }
                    old = __shfl_sync(FULL, old, leader);
                    const uint64_t rec = (old >> DG_PACK_SHIFT) + __popc(qmask & ((1u << lane) - 1u));
                    const uint64_t ibase = (old & ((1ull << DG_PACK_SHIFT) - 1ull)) + (incl - ni);
                    const bool fits = nu != 0u && rec < job.queue_cap && ibase + ni <= job.items_cap;
                    if (fits) {
                        uint4* qd = reinterpret_cast<uint4*>(job.queue + rec);
                        qd[0] = make_uint4(rbase + (uint32_t)rr, tr.seq, tr.frame, tr.xlo);
                        qd[1] = make_uint4(tr.ylo, bw, bh, 0u);
                    } else if (nu != 0u) {
                        inplace = true;  // queue full: this lane rasterizes the box itself
                    }
                    // Items of a lane that did not fit are marked empty (their slots are handed out).
                    // Lanes with at least 32 items: the whole warp writes them, one lane after another.
                    unsigned big = __ballot_sync(FULL, ni >= 32u);
                    while (big) {
                        const int L = __ffs(big) - 1;
                        big &= big - 1u;
                        const uint32_t lni = __shfl_sync(FULL, ni, L);
                        const uint32_t orec = (uint32_t)__shfl_sync(FULL, (unsigned long long)rec, L);
                        const uint64_t oib = __shfl_sync(FULL, (unsigned long long)ibase, L);
                        const bool ofits = __shfl_sync(FULL, fits ? 1u : 0u, L) != 0u;
                        for (uint32_t k = lane; k < lni; k += 32u)
                            if (oib + k < job.items_cap)
                                job.items[oib + k] = ofits ? make_uint2(orec, k) : make_uint2(DG_NONE, 0u);
                    }
                    // The other lanes' items numbered together: item j belongs to the first lane
                    // whose inclusive count exceeds it.
                    const uint32_t ns = ni < 32u ? ni : 0u;
                    uint32_t sincl = ns;
    #pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const uint32_t v = __shfl_up_sync(FULL, sincl, o);
                        if (lane >= (uint32_t)o) sincl += v;
                    }
                    const uint32_t stotal = __shfl_sync(FULL, sincl, 31);
                    const uint32_t sexcl = sincl - ns;
                    for (uint32_t b0 = 0; b0 < stotal; b0 += 32u) {
                        const uint32_t j = b0 + lane;
                        int lo = 0, hi = 31;
    #pragma unroll
                        for (int it = 0; it < 5; it++) {
                            const int mid = (lo + hi) >> 1;
                            if (__shfl_sync(FULL, sincl, mid) > j)
                                hi = mid;
                            else
                                lo = mid + 1;
                        }
                        const uint32_t orec = (uint32_t)__shfl_sync(FULL, (unsigned long long)rec, lo);
                        const uint64_t oib = __shfl_sync(FULL, (unsigned long long)ibase, lo);
                        const uint32_t oex = __shfl_sync(FULL, sexcl, lo);
                        const bool ofits = __shfl_sync(FULL, fits ? 1u : 0u, lo) != 0u;
                        const uint32_t k = j - oex;  // item index within its record
                        if (j < stotal && oib + k < job.items_cap)
                            job.items[oib + k] = ofits ? make_uint2(orec, k) : make_uint2(DG_NONE, 0u);
                    }
                }
                // Small triangles go to the small-triangle list, which the queue pass rasterizes.
                if (smask) {
                    sold = __shfl_sync(FULL, sold, __ffs(smask) - 1);
                    const uint64_t slot = sold + __popc(smask & ((1u << lane) - 1u));
                    if (small) {
                        if (slot < job.small_cap) {
                            store_small(job.small + slot, tr);
                        } else {
                            inplace = true;  // list full
                        }
                    }
                }
                if (inplace) {  // this lane rasterizes the box itself
                    atomicAdd(job.cnt + DG_CNT_INPLACE, 1ull);
                    raster_box(e, tr.da, tr.db, tr.dc, tr.seq, tr.xlo, tr.ylo, tr.xhi - tr.xlo + 1u, tr.yhi - tr.ylo + 1u,
                               frame(tr.frame));
                }
            }
        }
    }
    __syncthreads();
    if (threadIdx.x == 0 && s_records) atomicAdd(job.cnt + DG_CNT_TREC, (unsigned long long)s_records);  // statistics only
    if (FRONT && threadIdx.x == 0 && s_surv) atomicAdd(job.cnt + DG_CNT_SURV, (unsigned long long)s_surv);
}

__global__ void __launch_bounds__(256) k_setup_raster(const __grid_constant__ DgJobDev job) {
    DG_TL_BLOCK(2);
    wait_previous_kernel();
    DG_TL_WAITED(2);
    dev_setup<false>(job, job.nsegs, [&](uint32_t i) -> const DgSegDev& { return job.segs[i]; },
                     [&](uint32_t i) -> const DgFrameDev& { return job.frames[i]; });
}

// Setup of the small unclipped triangles of DG_FRAME_LAZY frames, before
// k_setup_raster: their box and their small-list entry, and nothing else (no
// edges, no record, no vertex marks); the other survivors go to the rest list.
// Most triangles of such a frame win no pixel, so what shading needs is gathered
// for the pixels instead. Bound by the gathers of the vertex records and by the
// entries written; without the clip program and the record it runs at three times
// the occupancy of k_setup_raster.
__global__ void __launch_bounds__(256, 6) k_setup_lean(const __grid_constant__ DgJobDev job) {
    DG_TL_BLOCK(2);  // a part of the setup pass
    wait_previous_kernel();
    DG_TL_WAITED(2);
    __shared__ uint32_t s_records;  // statistics, as in dev_setup
    if (threadIdx.x == 0) s_records = 0u;
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31u;
    const unsigned long long ns64 = __ldcg(job.cnt + DG_CNT_SURV);
    const uint32_t nsurv = (uint32_t)(ns64 < job.total_tri ? ns64 : job.total_tri);
    for (uint32_t base = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u; base < nsurv; base += gridDim.x * blockDim.x) {
        uint32_t g = 0;
        bool lean = false, rest = false, counted = false;
        RTri tr;
        const DgFrameDev* fr = job.frames;
        if (base + lane < nsurv) {
            g = __ldcg(job.surv + base + lane);
            const DgSegDev& sg = job.segs[seg_of_tri(job, g)];
            fr = job.frames + sg.frame;
            const uint32_t t = g - sg.tri_begin;
            float4 r[3];
            triangle_vertices(job, sg, *fr, __ldg(sg.tri_pos + t), r);
            const uint32_t m = __float_as_uint(r[0].w) & __float_as_uint(r[1].w) & __float_as_uint(r[2].w);
            rest = !(fr->flags & DG_FRAME_LAZY) || (m & 0x3u) != 0x3u;
            if (!rest) {
                tr.ax = r[0].x; tr.ay = r[0].y;
                tr.bx = r[1].x; tr.by = r[1].y;
                tr.cx = r[2].x; tr.cy = r[2].y;
                tr.da = r[0].z; tr.db = r[1].z; tr.dc = r[2].z;
                tr.frame = sg.frame;
                tr.seq = (sg.seq_base + t) << 2;
                if (isnan(tr.ax) || isnan(tr.ay) || isnan(tr.bx) || isnan(tr.by) || isnan(tr.cx) || isnan(tr.cy)) {
                    counted = true;  // every barycentric is NaN: nothing is covered
                } else {
                    bbox_axis(tr.ax, tr.bx, tr.cx, fr->width, tr.xlo, tr.xhi);
                    bbox_axis(tr.ay, tr.by, tr.cy, fr->height, tr.ylo, tr.yhi);
                    lean = small_listed(*fr, tr, (uint64_t)(tr.xhi - tr.xlo + 1u) * (tr.yhi - tr.ylo + 1u));
                    rest = !lean;
                }
            }
        }
        const unsigned lmask = __ballot_sync(FULL, lean), rmask = __ballot_sync(FULL, rest);
        unsigned long long lold = 0, rold = 0;
        if (lane == 0u) {
            if (lmask) lold = atomicAdd(job.cnt + DG_CNT_SMALL, (unsigned long long)__popc(lmask));
            if (rmask) rold = atomicAdd(job.cnt + DG_CNT_REST, (unsigned long long)__popc(rmask));
        }
        const unsigned below = (1u << lane) - 1u;
        const uint64_t slot = __shfl_sync(FULL, lold, 0) + __popc(lmask & below);
        uint64_t rpos = __shfl_sync(FULL, rold, 0) + __popc(rmask & below);
        if (lean && slot >= job.small_cap) {  // list full
            lean = false;
            rest = true;
            rpos = atomicAdd(job.cnt + DG_CNT_REST, 1ull);
        }
        if (rest) job.rest[rpos] = g;  // each survivor once: at most total_tri
        if (lean) {
            store_small(job.small + slot, tr);
            job.rec_of[g] = DG_LEAN | (uint32_t)slot;
            if (fr->cells != nullptr)  // the box's 32x32 cells, as in dev_setup
                for (uint32_t cy = tr.ylo >> 5; cy <= tr.yhi >> 5; cy++)
                    for (uint32_t cx = tr.xlo >> 5; cx <= tr.xhi >> 5; cx++)
                        fr->cells[cy * fr->tiles_x + cx] = fr->epoch;
        }
        const uint32_t n = (uint32_t)__popc(__ballot_sync(FULL, lean || counted));
        if (lane == 0u && n) atomicAdd(&s_records, n);
    }
    __syncthreads();
    if (threadIdx.x == 0 && s_records) atomicAdd(job.cnt + DG_CNT_TREC, (unsigned long long)s_records);
}

// The front of a small job as one kernel instead of three: vertex, cull and setup
// passes of a few thousand triangles are a few microseconds of launch and
// dependent loads each. A thread computes its triangle's three vertices itself
// (about three times the vertex arithmetic of k_vertex); the vertex records that
// the transparent pass and record-less pixels read are written at the end.
template <class IN>
__global__ void __launch_bounds__(DG_FRONT_THREADS) k_front(const __grid_constant__ DgJobDev job,
                                                            const __grid_constant__ IN in) {
    DG_TL_FOLDED();
    DG_TL_BLOCK(2);
    allow_next_kernel();
    begin_job(job, in);
    auto seg = [&](uint32_t i) -> const DgSegDev& { return in.segs[i]; };
    auto frame = [&](uint32_t i) -> const DgFrameDev& { return in.frames[IN::kFrames == 1u ? 0u : i]; };
    dev_setup<true>(job, in.nsegs, seg, frame);
    dev_vertex<false>(job, in.nsegs, seg, frame);
    // After k_tsort_first, the kernels behind this one need both complete (no wait otherwise).
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Row of pixel k (row-major) of a box whose width's reciprocal is rw:
// (k + 0.5) / width is at least 0.5 / width from an integer, far more than the
// error of the product (boxes of at most 65025 pixels).
__device__ __forceinline__ uint32_t box_row(uint32_t k, float rw) { return (uint32_t)(((float)k + 0.5f) * rw); }

// An entry of the small-triangle list as the raster reads it.
struct SmallTri {
    EdgeSet e;
    float da, db, dc;
    uint32_t seq, x0, y0, w, h, frame;
};
__device__ __forceinline__ SmallTri load_small(const DgSmallRec* s) {
    const float4* q = reinterpret_cast<const float4*>(s);
    const float4 a = __ldcg(q), b = __ldcg(q + 1);
    const uint4 c = __ldcg(reinterpret_cast<const uint4*>(s) + 2);
    SmallTri t;
    make_edges(a.x, a.w, a.y, b.x, a.z, b.y, t.e);
    t.da = b.z;
    t.db = b.w;
    t.dc = __uint_as_float(c.x);
    t.seq = c.y;
    t.x0 = c.z & 0xFFFFu;
    t.y0 = c.z >> 16;
    t.w = c.w & 0xFFu;
    t.h = (c.w >> 8) & 0xFFu;
    t.frame = c.w >> 16;
    return t;
}

// A warp's 32 small triangles in shared memory: 24 words each, with a stride of
// seven 16-byte words so that lanes on different triangles read different banks.
#define DG_SMALL_STRIDE 7
#define DG_SMALL_WINDOW 512u  // covered pixels listed at a time
// Rasterizes entries first .. first + 31 of the small-triangle list. Each lane
// tests its box's pixels one after another into a mask (edge values in registers,
// one addition per edge and pixel); the covered pixels of all 32 are then listed together
// and finished one per lane, so that the divisions and the keyed minimum run on
// full warps (about a fifth of the box pixels are covered, unevenly). Measured
// for the queue pass on 10M micro triangles and on 32 small frames, by events between
// the kernels: 305 and 53 us; with the pixels of all boxes numbered together and one
// per lane, 393 and 57; before these and covers_nothing, a lane finishing its own
// pixels, triangles ordered by box size, 411 and 70. Of the micro frame's pass alone
// (ncu), 264 us, the edge values evaluated anew at each pixel, clip outputs without
// area listed too (57 us), plain divisions (bary_fast) and a load of the vertex marks
// per 32 (40 us) were 94; it takes 170 now.
__device__ __forceinline__ void raster_small_chunk(const DgJobDev& job, uint32_t first, uint32_t nsmall, float4* st,
                                                   uint16_t* list) {
    const uint32_t lane = threadIdx.x & 31u;
    uint64_t mask = 0;
    bool whole = false;  // beyond 64 pixels, or not finite: the whole warp takes it below
    if (first + lane < nsmall) {
        const SmallTri t = load_small(job.small + first + lane);
        const uint32_t n = t.w * t.h;
        whole = n > 64u || !(t.e.tie & DG_EDGE_FAST);
        float4* d = st + lane * DG_SMALL_STRIDE;
        d[0] = make_float4(t.e.A[0], t.e.A[1], t.e.A[2], t.e.B[0]);
        d[1] = make_float4(t.e.B[1], t.e.B[2], t.e.C[0], t.e.C[1]);
        d[2] = make_float4(t.e.C[2], t.e.D[0], t.e.D[1], t.e.D[2]);
        d[3] = make_float4(__uint_as_float((t.y0 << 16) | t.x0), __uint_as_float(t.w), __fdividef(1.0f, (float)t.w),
                           __uint_as_float(t.frame));
        d[4] = make_float4(t.e.den[0], t.e.den[1], t.e.den[2], __uint_as_float(t.seq));
        d[5] = make_float4(t.da, t.db, t.dc, 0.0f);
        if (!whole) {
            // covered_signs as a sign: the edge values are integer-valued (or infinite),
            // so "> 0, or 0 with the tie bit" is "> -1/2" or "> 1/2".
            const float t0 = (t.e.tie & 1u) ? 0.5f : -0.5f, t1 = (t.e.tie & 2u) ? 0.5f : -0.5f,
                        t2 = (t.e.tie & 4u) ? 0.5f : -0.5f;
            // When no step of an edge value rounds anywhere in the box, moving a pixel
            // adds exactly A and moving a row exactly B: |C|, |D| < 2^23 and |A| x + |B| y
            // < 2^22 keep the sums integers below 2^24, and values below 2^22 in the box
            // take the half exactly.
            const float bx = (float)(t.x0 + t.w), by = (float)(t.y0 + t.h), bw = (float)t.w, bh = (float)t.h;
            const float xf = (float)t.x0, yf = (float)t.y0;
            float f0 = edge_eval(t.e, 0, xf, yf), f1 = edge_eval(t.e, 1, xf, yf), f2 = edge_eval(t.e, 2, xf, yf);
            const float fm[3] = {fabsf(f0), fabsf(f1), fabsf(f2)};
            bool exact = true;
#pragma unroll
            for (int k = 0; k < 3; k++) {
                const float aA = fabsf(t.e.A[k]), aB = fabsf(t.e.B[k]);
                exact = exact && fmaxf(fabsf(t.e.C[k]), fabsf(t.e.D[k])) < 0x1p23f && aA * bx + aB * by < 0x1p22f &&
                        fm[k] + aA * bw + aB * bh < 0x1p22f;
            }
            f0 += t0;
            f1 += t1;
            f2 += t2;
            const float wm = (float)(t.w - 1u);  // from a row's last pixel to the next row's first
            const float w0 = t.e.B[0] - wm * t.e.A[0], w1 = t.e.B[1] - wm * t.e.A[1], w2 = t.e.B[2] - wm * t.e.A[2];
            uint32_t m[2] = {0u, 0u}, c = 0;
#pragma unroll
            for (int half = 0; half < 2; half++) {
                const uint32_t begin = 32u * half, end = n < begin + 32u ? n : begin + 32u;
                uint32_t out = 0;  // outside bits, the first pixel's highest
                for (uint32_t k = begin; k < end; k++) {
                    out = __funnelshift_l(__float_as_uint(f0) | __float_as_uint(f1) | __float_as_uint(f2), out, 1u);
                    const bool wrap = ++c == t.w;
                    c = wrap ? 0u : c;
                    f0 += wrap ? w0 : t.e.A[0];
                    f1 += wrap ? w1 : t.e.A[1];
                    f2 += wrap ? w2 : t.e.A[2];
                }
                if (end > begin) m[half] = __brev(~out) >> (32u - (end - begin));
            }
            if (!exact) {  // the edge values as the reference evaluates them
                float x = xf, y = yf;
                uint64_t mm = 0;
                for (uint32_t k = 0; k < n; k++) {
                    const bool in = (edge_eval(t.e, 0, x, y) > -t0) & (edge_eval(t.e, 1, x, y) > -t1) &
                                    (edge_eval(t.e, 2, x, y) > -t2);
                    mm |= (in ? 1ull : 0ull) << k;
                    x += 1.0f;
                    if (x == bx) {
                        x = xf;
                        y += 1.0f;
                    }
                }
                m[0] = (uint32_t)mm;
                m[1] = (uint32_t)(mm >> 32);
            }
            mask = ((uint64_t)m[1] << 32) | m[0];
        }
    }
    const uint32_t cnt = (uint32_t)__popcll((long long)mask);
    uint32_t incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(FULL, incl, o);
        if (lane >= (uint32_t)o) incl += v;
    }
    const uint32_t total = __shfl_sync(FULL, incl, 31);
    uint32_t pos = incl - cnt;
    for (uint32_t w0 = 0; w0 < total; w0 += DG_SMALL_WINDOW) {
        const uint32_t end = min(total, w0 + DG_SMALL_WINDOW);
        while (mask != 0ull && pos < end) {
            const uint32_t k = (uint32_t)__ffsll((long long)mask) - 1u;
            mask &= mask - 1ull;
            list[pos - w0] = (uint16_t)((lane << 6) | k);
            pos++;
        }
        __syncwarp();
        for (uint32_t j = w0 + lane; j < end; j += 32u) {
            const uint32_t at = list[j - w0];
            const float4* d = st + (at >> 6) * DG_SMALL_STRIDE;
            const float4 a = d[0], b = d[1], c = d[2], box = d[3], den = d[4], dd = d[5];
            EdgeSet e;
            e.A[0] = a.x; e.A[1] = a.y; e.A[2] = a.z; e.B[0] = a.w;
            e.B[1] = b.x; e.B[2] = b.y; e.C[0] = b.z; e.C[1] = b.w;
            e.C[2] = c.x; e.D[0] = c.y; e.D[1] = c.z; e.D[2] = c.w;
            const uint32_t k = at & 63u, xy = __float_as_uint(box.x), dy = box_row(k, box.z);
            const uint32_t x = (xy & 0xFFFFu) + (k - dy * __float_as_uint(box.y)), y = (xy >> 16) + dy;
            const float xf = (float)x, yf = (float)y;
            const DgFrameDev& fr = job.frames[__float_as_uint(box.w)];
            const float al = bary_fast(edge_eval(e, 0, xf, yf), den.x);
            const float be = bary_fast(edge_eval(e, 1, xf, yf), den.y);
            const float ga = bary_fast(edge_eval(e, 2, xf, yf), den.z);
            const float depth = interp(al, be, ga, dd.x, dd.y, dd.z);
            if (depth < fr.clear_depth)
                atomicMin(reinterpret_cast<unsigned long long*>(fr.vis) + (y * fr.width + x),
                          depth_key(depth, __float_as_uint(den.w)));
        }
        __syncwarp();
    }
    unsigned big = __ballot_sync(FULL, whole);
    while (big) {
        const uint32_t L = (uint32_t)__ffs(big) - 1u;
        big &= big - 1u;
        const SmallTri t = load_small(job.small + first + L);
        const float rw = __fdividef(1.0f, (float)t.w);
        for (uint32_t k = lane; k < t.w * t.h; k += 32u) {
            const uint32_t r = box_row(k, rw);
            raster_pixel(t.e, t.da, t.db, t.dc, t.seq, t.x0 + (k - r * t.w), t.y0 + r, job.frames[t.frame]);
        }
        __syncwarp();
    }
}

__device__ __forceinline__ void dev_queue(const DgJobDev& job) {
    __shared__ float4 s_tri[8][32 * DG_SMALL_STRIDE];  // per-warp small triangles
    __shared__ uint16_t s_list[8][DG_SMALL_WINDOW];    // and their covered pixels
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    // Prologue: light/halfway vectors of the vertices the setup pass marked, 32
    // vertices per warp; the marks are cleared for the next job.
    const uint32_t ngroups = (job.total_vtx + 31u) >> 5;
    auto shade_group = [&](uint32_t w) {
        const uint32_t v = (w << 5) + lane;
        if (v < job.total_vtx && __ldcg(job.vmark + v)) {
            shade_vertex(job, v);
            job.vmark[v] = 0u;
        }
    };
    if (ngroups <= 4u * nwarps) {
        for (uint32_t w = warp; w < ngroups; w += nwarps) shade_group(w);
    } else {
        // Many vertices: 512 marks per load first (a load per 32 of 9M vertices was a chain
        // of 19 per warp, 40 us of the queue pass).
        for (uint32_t w = warp; w < (ngroups + 15u) >> 4; w += nwarps) {
            const uint4 m = __ldcg(reinterpret_cast<const uint4*>(job.vmark) + (w << 5) + lane);
            unsigned any = __ballot_sync(FULL, (m.x | m.y | m.z | m.w) != 0u);
            while (any) {  // lanes 2 g and 2 g + 1 hold the marks of group g
                const uint32_t g = ((uint32_t)__ffs(any) - 1u) >> 1;
                any &= ~(3u << (2u * g));
                shade_group((w << 4) + g);
            }
        }
    }
    const unsigned long long cnt = __ldcg(job.cnt + DG_CNT_QUEUE);
    const uint64_t ni64 = cnt & ((1ull << DG_PACK_SHIFT) - 1ull);
    const uint32_t nitems = (uint32_t)(ni64 < job.items_cap ? ni64 : job.items_cap);
    const unsigned long long ns64 = __ldcg(job.cnt + DG_CNT_SMALL);
    const uint32_t nsmall = (uint32_t)(ns64 < job.small_cap ? ns64 : job.small_cap);
    // Small triangles go in chunks of 32 to single warps (raster_small_chunk), ahead
    // of the work items. With fewer than two per warp, a chunk would be the pass's
    // longest chain: they go in pairs, 16 lanes each (measured with a lane per
    // triangle: a 1283x717 frame of 679 small triangles, the pass 20.5 -> 12.3 us;
    // 512x512 with 23,500, 1.6 per warp, 20.5 -> 18.4).
    const bool few_small = nsmall < nwarps * 2u;
    // Work index wi: chunks of small triangles (wi < nchunks), then the work items.
    const uint32_t nchunks = few_small ? (nsmall + 1u) >> 1 : (nsmall + 31u) >> 5;
    for (uint32_t wi = warp; wi < nchunks + nitems; wi += nwarps) {
        if (wi < nchunks && few_small) {
            const uint32_t i = 2u * wi + (lane >> 4);
            if (i < nsmall) {
                const SmallTri t = load_small(job.small + i);
                const float rw = __fdividef(1.0f, (float)t.w);
                for (uint32_t k = lane & 15u; k < t.w * t.h; k += 16u) {
                    const uint32_t r = box_row(k, rw);
                    raster_pixel(t.e, t.da, t.db, t.dc, t.seq, t.x0 + (k - r * t.w), t.y0 + r, job.frames[t.frame]);
                }
            }
            __syncwarp();
            continue;
        }
        if (wi < nchunks) {
            raster_small_chunk(job, wi << 5, nsmall, s_tri[threadIdx.x >> 5], s_list[threadIdx.x >> 5]);
            continue;
        }
        const uint32_t it = wi - nchunks;
        const uint2 item = __ldcg(job.items + it);
        if (item.x >= job.queue_cap) continue;  // an item of a triangle that did not fit the queue
        const uint4* qs = reinterpret_cast<const uint4*>(job.queue + item.x);
        const uint4 q0 = __ldcg(qs), q1 = __ldcg(qs + 1);
        const DgTriRec* R = job.trec + q0.x;
        EdgeSet e;
        load_edges<true>(R, e);
        const float4 dd = __ldg(reinterpret_cast<const float4*>(R) + 4);
        const uint32_t seq = q0.y;
        const DgFrameDev& fr = job.frames[q0.z];
        const float clear_depth = fr.clear_depth;
        unsigned long long* vis = reinterpret_cast<unsigned long long*>(fr.vis);
        const uint32_t width = fr.width;
        const uint32_t xlo = q0.w, ylo = q1.x, w = q1.y, h = q1.z;
        if (!DG_IN_RANGE(w != 0u && xlo + w <= width && ylo + h <= fr.height && q0.x < job.trec_cap, job.err)) continue;
        if (w * h <= 32u) {  // one pixel per lane: cheaper than spans (32 small frames: the pass 77.8 -> 69.6 us)
            if (lane < w * h) {
                const uint32_t r = box_row(lane, __fdividef(1.0f, (float)w));
                raster_pixel(e, dd.x, dd.y, dd.z, seq, xlo + (lane - r * w), ylo + r, fr);
            }
            __syncwarp();
            continue;
        }
        const DgItemGrid grid = dg_item_grid(w, h, job.item_log2);
        const uint32_t iy = grid.nx == 1u ? item.y : item.y / grid.nx, ix = item.y - iy * grid.nx;
        const uint32_t x0 = xlo + ix * grid.cw, xe = min(x0 + grid.cw, xlo + w);  // columns [x0, xe)
        const uint32_t y0 = ylo + iy * grid.rh, ye = min(y0 + grid.rh, ylo + h);  // rows [y0, ye)
        if (!(e.tie & DG_EDGE_SPAN)) {  // huge or not finite edge constants: the reference's test per pixel
            const uint32_t cw = xe - x0, n = cw * (ye - y0);
            for (uint32_t k = lane; k < n; k += 32u) raster_pixel(e, dd.x, dd.y, dd.z, seq, x0 + k % cw, y0 + k / cw, fr);
            __syncwarp();
            continue;
        }
        const float3 yr = make_float3(__frcp_rn(e.den[0]), __frcp_rn(e.den[1]), __frcp_rn(e.den[2]));
        const float3 rA = make_float3(__fdividef(1.0f, e.A[0]), __fdividef(1.0f, e.A[1]), __fdividef(1.0f, e.A[2]));
        for (uint32_t yb = y0; yb < ye; yb += 32u) {
            // One row per lane: its covered span.
            int lo = (int)x0, hi = (int)xe - 1;
            if (yb + lane < ye) {
                const float yf = (float)(yb + lane);
                row_span(e, 0, rA.x, yf, (int)x0, (int)xe - 1, lo, hi);
                row_span(e, 1, rA.y, yf, (int)x0, (int)xe - 1, lo, hi);
                row_span(e, 2, rA.z, yf, (int)x0, (int)xe - 1, lo, hi);
            } else {
                hi = lo - 1;
            }
            const uint32_t cnt = hi >= lo ? (uint32_t)(hi - lo + 1) : 0u;
            uint32_t incl = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t v = __shfl_up_sync(FULL, incl, o);
                if (lane >= (uint32_t)o) incl += v;
            }
            const uint32_t total = __shfl_sync(FULL, incl, 31);
            const uint32_t first = (uint32_t)lo - (incl - cnt);  // column of the row's fragment j: first + j
            // The covered pixels, 32 at a time: fragment j is in the first row whose inclusive count exceeds it.
            for (uint32_t b0 = 0; b0 < total; b0 += 32u) {
                const uint32_t j = b0 + lane;
                int r = 0, re = 31;
#pragma unroll
                for (int it = 0; it < 5; it++) {
                    const int mid = (r + re) >> 1;
                    if (__shfl_sync(FULL, incl, mid) > j)
                        re = mid;
                    else
                        r = mid + 1;
                }
                const uint32_t x = __shfl_sync(FULL, first, r) + j, y = yb + (uint32_t)r;
                if (j < total) {
                    const float xf = (float)x, yf = (float)y;
                    const float al = div_rcp(edge_eval(e, 0, xf, yf), e.den[0], yr.x);
                    const float be = div_rcp(edge_eval(e, 1, xf, yf), e.den[1], yr.y);
                    const float ga = div_rcp(edge_eval(e, 2, xf, yf), e.den[2], yr.z);
                    const float depth = interp(al, be, ga, dd.x, dd.y, dd.z);
                    if (depth < clear_depth) atomicMin(vis + (y * width + x), depth_key(depth, seq));
                }
            }
        }
    }
}

// Tile `tile` of the job: its frame, column and row (of tiles).
__device__ __forceinline__ const DgFrameDev& find_tile(const DgJobDev& job, uint32_t tile, uint32_t& tx, uint32_t& ty) {
    const uint32_t fi = last_le(job.nframes, tile, [&](uint32_t i) { return job.frames[i].tile_begin; });
    const DgFrameDev& fr = job.frames[fi];
    const uint32_t lt = tile - fr.tile_begin;
    ty = lt / fr.tiles_x;
    tx = lt - ty * fr.tiles_x;
    return fr;
}

// The number of cells that a triangle box reached this frame, for k_resolve_split,
// which reads it before its wait: counted before this kernel's launch signal.
__device__ __forceinline__ void count_reached_cells(const DgJobDev& job) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t w = warp; w < (job.total_tiles + 31u) >> 5; w += nwarps) {
        const uint32_t c = (w << 5) + lane;
        bool reached = false;
        if (c < job.total_tiles) {
            uint32_t tx, ty;
            const DgFrameDev& fr = find_tile(job, c, tx, ty);
            reached = fr.cells == nullptr || __ldcg(fr.cells + (c - fr.tile_begin)) == fr.epoch;
        }
        const unsigned rb = __ballot_sync(FULL, reached);
        if (lane == 0u && rb) atomicAdd(job.cnt + DG_CNT_CELLS, (unsigned long long)__popc(rb));
    }
    __threadfence();
}

// The resolve pass may start only after this kernel's blocks have waited for
// the setup pass, so that its early clear of untouched tiles (k_resolve) reads
// a complete cell map: the wait comes before the launch signal here.
__global__ void __launch_bounds__(256, 4) k_queue_raster(const DgJobDev job) {
    DG_TL_BLOCK(3);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    DG_TL_WAITED(3);
    if (job.split_below) {
        count_reached_cells(job);
        // A block's launch signal is the first one that any of its threads gives, so
        // all of them must have counted: without the barrier k_resolve_split's blocks
        // could read different partial counts and disagree on strips.
        __syncthreads();
    }
    allow_next_kernel();
    dev_queue(job);
}

// Pixels of tile `tile` whose winning triangle has no record (the record
// buffers were full) kept their keys in phase 1: they are shaded here from the
// mesh (shade_without_record) and their keys reset. The tile's own CTA calls it
// at the end of k_resolve, each thread on the pixels it read in phase 1. Out of
// line, so that the long path costs the main path no registers (the job is a
// __grid_constant__ parameter: its address needs no copy).
template <uint32_t TH>
__device__ __noinline__ void shade_tile_without_records(const DgJobDev& job, const DgFrameDev& fr, uint32_t tx,
                                                        uint32_t ty, const float* inv255, const DgTexDev* stex) {
    const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    const uint32_t x = tx * DG_TILE_W + lane;
    const uint32_t W = fr.width, H = fr.height;
    uint32_t shaded = 0;
    for (uint32_t j = 0; j < TH / 8u; j++) {
        const uint32_t y = ty * TH + wid + 8u * j;
        if (x >= W || y >= H) continue;
        const uint64_t i = (uint64_t)y * W + x;
        const uint64_t key = __ldcg(reinterpret_cast<const unsigned long long*>(fr.vis) + i);
        if (key == DG_VIS_EMPTY) continue;  // empty, or shaded from its record
        fr.vis[i] = DG_VIS_EMPTY;
        float d = 0.0f;
        int errc;
        uint32_t c = shade_without_record(job, fr, (uint32_t)key, x, y, inv255, stex, d, errc);
        if (errc != DG_OK) {
            c = AZUL_BB;
            atomicOr(job.err, 1u << errc);
        }
        fr.depth[i] = d;
        fr.colour[(uint64_t)(H - 1u - y) * W + x] = c;
        shaded++;
    }
    if (shaded) atomicAdd(job.cnt + DG_CNT_COVERED, (unsigned long long)shaded);
}

// Resolve and shade, fused: one 32 x TH tile per CTA of 256 threads (TH = 8,
// 16 or 32: the tile_rows knob).
//  0. If the tile's 32x32 cell does not hold the frame's epoch, no triangle's
//     box reached it and every key is empty: the clear values, and return.
//  1. Each thread reads the visibility keys of TH/8 pixels (rows r, r+8, ...
//     of its column). An empty pixel gets the clear colour and depth
//     (this is Canvas::clear, canvas.rs:425-433); a covered one has its key
//     reset for the next frame and goes into the tile's shade list in shared
//     memory with its triangle record, in row-major order. A covered pixel
//     whose triangle has no record keeps its key for step 3.
//  2. The CTA shades its list densely: the winning fragment of every covered
//     pixel is shaded once (canvas.rs:682-741) and its colour (row H-1-y) and
//     depth (y*W+x) are written (canvas.rs:923-930).
//  3. If a pixel of the tile had no record, shade_tile_without_records.
// The resolve pass's tables, independent of the previous passes: the 256
// quotients byte / 255 and the first DG_SMEM_TEX texture descriptors.
__device__ __forceinline__ void resolve_prologue(const DgJobDev& job, float* inv255, DgTexDev* stex) {
    inv255[threadIdx.x] = fD((float)threadIdx.x, 255.0f);
    const uint32_t nst = job.ntex < DG_SMEM_TEX ? job.ntex : DG_SMEM_TEX;
    for (uint32_t i = threadIdx.x; i < nst * 3u; i += blockDim.x)
        reinterpret_cast<uint4*>(stex)[i] = __ldg(reinterpret_cast<const uint4*>(job.tex) + i);
}

// Canvas::clear (canvas.rs:425-433) of one 32 x TH tile (tile column tx, row ty):
// 16-byte stores of four pixels where the rows are 16-byte aligned.
template <uint32_t TH>
__device__ __forceinline__ void clear_tile(const DgFrameDev& fr, uint32_t tx, uint32_t ty) {
    const uint32_t W = fr.width, H = fr.height;
    const uint32_t x0 = tx * DG_TILE_W;
    const bool vec = (W & 3u) == 0u && x0 + DG_TILE_W <= W &&
                     ((reinterpret_cast<uintptr_t>(fr.depth) | reinterpret_cast<uintptr_t>(fr.colour)) & 15u) == 0u;
    if (vec) {
        const uint32_t r = threadIdx.x >> 3, c = (threadIdx.x & 7u) * 4u;
        const float cd = fr.clear_depth;
        for (uint32_t yy = r; yy < TH; yy += 32u) {
            const uint32_t y = ty * TH + yy;
            if (y < H) {
                *reinterpret_cast<float4*>(fr.depth + (uint64_t)y * W + x0 + c) = make_float4(cd, cd, cd, cd);
                *reinterpret_cast<uint4*>(fr.colour + (uint64_t)(H - 1u - y) * W + x0 + c) =
                    make_uint4(AZUL_BB, AZUL_BB, AZUL_BB, AZUL_BB);
            }
        }
        return;
    }
    const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    const uint32_t x = x0 + lane;
#pragma unroll
    for (uint32_t j = 0; j < TH / 8u; j++) {
        const uint32_t y = ty * TH + wid + 8u * j;
        if (x < W && y < H) {
            fr.depth[(uint64_t)y * W + x] = fr.clear_depth;
            fr.colour[(uint64_t)(H - 1u - y) * W + x] = AZUL_BB;
        }
    }
}

// One tile of the resolve pass (block-uniform; the tables of resolve_prologue
// must be in place). EXT: the job uses an extension mode (perspective-correct
// interpolation or bilinear fetch); false compiles the reference's shading only.
// LAZY: a frame of the job has DG_FRAME_LAZY (its small triangles have no
// records); the resolve kernels then run at three blocks per SM, since the mesh's
// attributes and the vertices' vectors need registers.
template <uint32_t TH, bool EXT, bool LAZY>
__device__ __forceinline__ void dev_resolve_tile(const DgJobDev& job, const DgFrameDev& fr, const uint32_t tx,
                                                 const uint32_t ty, const float* inv255, const DgTexDev* stex) {
    __shared__ uint16_t s_pix[DG_TILE_W * TH];  // pixel index within the tile
    __shared__ uint32_t s_val[DG_TILE_W * TH];  // triangle record
    __shared__ uint32_t s_row[33];  // shade-list offset of each tile row; [32] = total
    const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    const uint32_t x = tx * DG_TILE_W + lane;
    const uint32_t W = fr.width, H = fr.height;
    constexpr int R = TH / 8;
    if (fr.cells != nullptr && __ldcg(fr.cells + ((ty * TH) >> 5) * fr.tiles_x + tx) != fr.epoch) {
        // No triangle's box reached the tile's 32x32 cell this frame, so all its
        // keys are empty: the clear values, without reading the keys (block-uniform).
        clear_tile<TH>(fr, tx, ty);
        return;
    }
    uint64_t key[R];
#pragma unroll
    for (int j = 0; j < R; j++) {  // all loads first: R keys in flight per thread
        const uint32_t y = ty * TH + wid + 8u * j;
        key[j] = (x < W && y < H) ? __ldcg(reinterpret_cast<const unsigned long long*>(fr.vis) + (y * W + x))
                                  : DG_VIS_EMPTY - 1ull;  // outside the canvas
    }
    const bool one_seg = fr.seg_count == 1u;
    const DgSegDev& sg0 = job.segs[one_seg ? fr.seg_begin : 0u];
    const uint32_t* rec0 = job.rec_of + sg0.tri_begin;
    const uint32_t ntri0 = sg0.ntri;
    uint32_t val[R];
    unsigned hit[R];
    int no_record = 0;
#pragma unroll
    for (int j = 0; j < R; j++) {
        const uint32_t y = ty * TH + wid + 8u * j;
        const uint32_t i = y * W + x;  // below 2^31 (pixels of a job)
        val[j] = DG_NONE;
        if (key[j] == DG_VIS_EMPTY) {
            fr.depth[i] = fr.clear_depth;
            fr.colour[(H - 1u - y) * W + x] = AZUL_BB;
        } else if (key[j] != DG_VIS_EMPTY - 1ull) {
            // the triangle record of the key: segment of the submission index, then rec_of
            const uint32_t tl = (uint32_t)key[j] >> 2;
            if (one_seg) {
                if (tl < ntri0) val[j] = __ldg(rec0 + tl);
            } else {
                const uint32_t si = fr.seg_begin + last_le(fr.seg_count, tl, [&](uint32_t k) {
                                        return job.segs[fr.seg_begin + k].seq_base;
                                    });
                const DgSegDev& sg = job.segs[si];
                const uint32_t t = tl - sg.seq_base;
                if (t < sg.ntri) val[j] = __ldg(job.rec_of + sg.tri_begin + t);
            }
            const uint32_t o = (uint32_t)key[j] & 3u;
            if (LAZY && val[j] != DG_NONE && (val[j] & DG_LEAN)) {
                fr.vis[i] = DG_VIS_EMPTY;  // (its one output)
            } else if (val[j] != DG_NONE && val[j] + o < job.trec_cap) {  // trec_cap <= 2^32 - 16
                val[j] += o;
                fr.vis[i] = DG_VIS_EMPTY;
            } else {
                val[j] = DG_NONE;  // shaded at the end, from the mesh, which resets the key
                no_record = 1;
            }
        }
        hit[j] = __ballot_sync(FULL, val[j] != DG_NONE);
        if (lane == 0) s_row[wid + 8u * j] = __popc(hit[j]);
    }
    const int any_no_record = __syncthreads_or(no_record);
    if (wid == 0) {  // exclusive scan of the TH row counts
        const uint32_t c = lane < TH ? s_row[lane] : 0u;
        uint32_t incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(FULL, incl, o);
            if (lane >= (uint32_t)o) incl += v;
        }
        s_row[lane] = incl - c;
        if (lane == 31u) {
            s_row[32] = incl;
            if (incl) atomicAdd(job.cnt + DG_CNT_COVERED, (unsigned long long)incl);
        }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < R; j++) {
        if ((hit[j] >> lane) & 1u) {
            const uint32_t row = wid + 8u * j;
            const uint32_t slot = s_row[row] + __popc(hit[j] & ((1u << lane) - 1u));
            s_pix[slot] = (uint16_t)(row * DG_TILE_W + lane);
            s_val[slot] = val[j];
        }
    }
    __syncthreads();
    const uint32_t n = s_row[32];
    uint32_t errors = 0;
    for (uint32_t k = threadIdx.x; k < n; k += blockDim.x) {
        const uint32_t pe = s_pix[k];
        const uint32_t px = tx * DG_TILE_W + (pe & 31u), py = ty * TH + (pe >> 5);
        float d = 0.0f;
        int errc;
        const uint32_t rec = s_val[k];
        const DgSmallRec* lean = LAZY && (rec & DG_LEAN) ? job.small + (rec & ~DG_LEAN) : nullptr;
        const float4* wp =
            EXT && (fr.flags & DG_FRAME_PERSPECTIVE) && job.trec_w && !lean ? job.trec_w + rec : nullptr;
        uint32_t c = shade_from_record<EXT, LAZY, true>(job, fr, job.trec + rec, px, py, inv255, stex, d, errc, wp, lean);
        if (errc != DG_OK) {
            c = AZUL_BB;
            errors |= 1u << errc;
        }
        fr.depth[py * W + px] = d;
        fr.colour[(H - 1u - py) * W + px] = c;
    }
    // one error-word update per warp (every pixel of a bad job may fail)
    errors = __reduce_or_sync(FULL, errors);
    if (errors != 0u && lane == 0u) atomicOr(job.err, errors);
    // pixels whose triangle has no record: shaded the long way (block-uniform)
    if (any_no_record) shade_tile_without_records<TH>(job, fr, tx, ty, inv255, stex);
}

// Whether a job's descriptors and cell map may be read before waiting for the
// previous kernel: k_queue_raster signals its dependent kernel only after it
// waited for the setup pass. With a transparent pass or without triangles, the
// kernel before the resolve pass is another.
__device__ __forceinline__ bool resolve_early(const DgJobDev& job) { return job.ntt == 0u && job.total_tri != 0u; }

template <uint32_t TH, bool EXT, bool LAZY>
__global__ void __launch_bounds__(256, LAZY ? 3 : 4) k_resolve(const __grid_constant__ DgJobDev job) {
    DG_TL_BLOCK(4);  // tiles cleared before the wait record no wait
    __shared__ float inv255[256];
    __shared__ DgTexDev stex[DG_SMEM_TEX];
    uint32_t tx, ty;
    if (resolve_early(job)) {
        // A tile that no triangle box reached is cleared before waiting for the
        // raster pass: its keys are all empty.
        const DgFrameDev& fr = find_tile(job, blockIdx.x, tx, ty);
        if (fr.cells != nullptr && __ldcg(fr.cells + ((ty * TH) >> 5) * fr.tiles_x + tx) != fr.epoch) {
            clear_tile<TH>(fr, tx, ty);  // (block-uniform) without the shading tables
            return;
        }
    }
    resolve_prologue(job, inv255, stex);
    wait_previous_kernel();
    DG_TL_WAITED(4);
    const DgFrameDev& fr = find_tile(job, blockIdx.x, tx, ty);
    dev_resolve_tile<TH, EXT, LAZY>(job, fr, tx, ty, inv255, stex);
}

// The resolve pass of a job that has enough 32-row tiles to fill the GPU, but not
// many times over (job.split_below): if fewer cells were reached than that, its
// reached tiles leave most of the GPU idle behind blocks that shade four pixels
// per thread, so each is taken as four strips of 8 rows by four blocks. Block strip * tiles + t
// works on strip `strip` of tile t, or, when enough cells were reached, blocks of
// strip 0 take whole tiles and the others leave before the wait. Measured on a
// 1283x717 field that covers 17% of the frame: 53.4 us whole, 46.8 us by this
// kernel; strips of more cells lose (ten frames of 500 reached cells 83 -> 86 us).
template <bool EXT, bool LAZY>
__global__ void __launch_bounds__(256, LAZY ? 3 : 4) k_resolve_split(const __grid_constant__ DgJobDev job) {
    DG_TL_BLOCK(4);
    __shared__ float inv255[256];
    __shared__ DgTexDev stex[DG_SMEM_TEX];
    const uint32_t strip = blockIdx.x / job.total_tiles;
    uint32_t tx, ty;
    const bool early = resolve_early(job);
    bool strips = true;
    // 0: nothing to do, 1: this block's tile or strip is to be resolved
    auto look = [&](const DgFrameDev& fr) -> bool {
        if (fr.cells != nullptr && __ldcg(fr.cells + ty * fr.tiles_x + tx) != fr.epoch) {
            if (strip == 0u) clear_tile<32>(fr, tx, ty);
            return false;
        }
        strips = __ldcg(job.cnt + DG_CNT_CELLS) < job.split_below;
        return strips ? ty * 32u + strip * 8u < fr.height : strip == 0u;
    };
    if (early && !look(find_tile(job, blockIdx.x - strip * job.total_tiles, tx, ty))) return;
    resolve_prologue(job, inv255, stex);
    wait_previous_kernel();
    DG_TL_WAITED(4);
    const DgFrameDev& fr = find_tile(job, blockIdx.x - strip * job.total_tiles, tx, ty);
    if (!early && !look(fr)) return;
    if (strips)
        dev_resolve_tile<8, EXT, LAZY>(job, fr, tx, ty * 4u + strip, inv255, stex);
    else
        dev_resolve_tile<32, EXT, LAZY>(job, fr, tx, ty, inv255, stex);
}

__global__ void k_fill(uint32_t* colour, float* depth, uint64_t n, uint32_t cv, float dv, int fc, int fd) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        if (fc) colour[i] = cv;
        if (fd) depth[i] = dv;
    }
}

// The RGBA view of a BGRA frame: bytes 0 and 2 of every pixel swapped, the
// fourth byte kept (Application::export_frame_as, app/mod.rs:345-350).
__global__ void k_bgra_to_rgba(const uint32_t* src, uint32_t* dst, uint64_t n) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t s = src[i];
        dst[i] = (s & 0xFF00FF00u) | ((s >> 16) & 0xFFu) | ((s & 0xFFu) << 16);
    }
}

__global__ void k_vis_reset(uint64_t* vis, uint64_t n) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        vis[i] = DG_VIS_EMPTY;
}

}  // namespace

// NVTX ranges name each pass's launch on a profiler's timeline (nvtx3 is
// header-only; without an attached tool a range costs a branch).
struct NvtxRange {
    explicit NvtxRange(const char* name) { nvtxRangePushA(name); }
    ~NvtxRange() { nvtxRangePop(); }
};

bool dg_timeline_copy(unsigned long long* out, cudaStream_t s, cudaError_t* err) {
#if DG_TIMELINE
    unsigned long long init[DG_NKERNELS][4];
    for (int k = 0; k < DG_NKERNELS; k++) {
        init[k][0] = init[k][1] = ~0ull;
        init[k][2] = init[k][3] = 0ull;
    }
    cudaError_t e = cudaStreamSynchronize(s);
    if (e == cudaSuccess) e = cudaMemcpyFromSymbol(out, g_timeline, sizeof(init));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_timeline, init, sizeof(init));
    *err = e;
    return true;
#else
    (void)out;
    (void)s;
    *err = cudaSuccess;
    return false;
#endif
}

cudaError_t dg_launch_job(const DgJobDev& job, const DgLaunchCfg& cfg, cudaStream_t s, cudaEvent_t* ev) {
    NvtxRange job_range("draw_gb300 render job");
    cudaError_t e;
    auto mark = [&](int i) { return ev ? cudaEventRecord(ev[i], s) : cudaSuccess; };
    // dg_ctx_inject_launch_failure: the job ends before launch k
    auto refused = [&](int32_t k) { return cfg.fail_before == k ? cudaErrorMemoryAllocation : cudaSuccess; };
    if ((e = mark(0)) != cudaSuccess) return e;
    DgInlineDesc none;
    none.nsegs = 0;
    // calls f with the descriptors of the job's first kernel
    auto with_inline = [&](auto f) {
        if (cfg.inl_large)
            f(*cfg.inl_large);
        else if (cfg.inl_batch)
            f(*cfg.inl_batch);
        else
            f(cfg.inl ? *cfg.inl : none);
    };
    const bool front =
        cfg.front && (cfg.inl || cfg.inl_batch || cfg.inl_large) && job.total_vtx && job.total_tri;
    const bool sort_first = front && job.ntt && cfg.tplan.tsort_meshes;
    if ((e = refused(1)) != cudaSuccess) return e;
    if (job.total_vtx && !front) {
        NvtxRange r("k_vertex");
        const unsigned vb = cfg.vertex_blocks < 1u ? 1u : cfg.vertex_blocks;
        with_inline([&](const auto& in) { k_vertex<<<grid_for(job.total_vtx, vb), 256, 0, s>>>(job, in); });
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    if ((e = mark(1)) != cudaSuccess || (e = refused(2)) != cudaSuccess) return e;
    if (job.total_tri && !front) {
        NvtxRange r("k_cull");
        const unsigned cb = cfg.cull_blocks < 1u ? 1u : cfg.cull_blocks;
        if ((e = launch_dependent(k_cull, grid_for(job.total_tri, cb), 256, job, s)) != cudaSuccess) return e;
    }
    if ((e = mark(2)) != cudaSuccess || (e = refused(3)) != cudaSuccess) return e;
    if (front) {
        NvtxRange r("k_front");
        const uint32_t blocks = (job.total_tri + DG_FRONT_THREADS - 1u) / DG_FRONT_THREADS;
        with_inline([&](const auto& in) {
            if (sort_first) {
                if ((e = dg_launch_tsort_first(in, cfg.tplan, s)) == cudaSuccess)
                    e = launch_dependent(k_front<std::decay_t<decltype(in)>>, blocks, DG_FRONT_THREADS, job, s, in);
            } else {
                k_front<<<blocks, DG_FRONT_THREADS, 0, s>>>(job, in);
                e = cudaGetLastError();
            }
        });
        if (e != cudaSuccess) return e;
    } else if (job.total_tri) {
        NvtxRange r("k_setup_raster");
        if (job.lazy) {
            const unsigned lb = cfg.lean_blocks < 1u ? 1u : cfg.lean_blocks;
            if ((e = launch_dependent(k_setup_lean, grid_for(job.total_tri, lb), 256, job, s)) != cudaSuccess) return e;
        }
        const unsigned sb = cfg.setup_blocks < 1u ? 1u : cfg.setup_blocks;
        if ((e = launch_dependent(k_setup_raster, grid_for(job.total_tri, sb), 256, job, s)) != cudaSuccess) return e;
    }
    if ((e = mark(3)) != cudaSuccess || (e = refused(4)) != cudaSuccess) return e;
    // transparent pass, part 0: painter's sort and setup (its vertices join the
    // lighting prologue of the queue pass)
    if ((e = dg_launch_transparent(0, job, cfg.tplan, s, sort_first)) != cudaSuccess) return e;
    if ((e = refused(5)) != cudaSuccess) return e;
    if (job.total_tri || job.ntt) {
        NvtxRange r("k_queue_raster");
        // Blocks beyond a job's possible work only cost their launch: at most a warp per
        // triangle, and one per 8 pixels for what its triangles' boxes may be cut into
        // (a 96x64 frame of 200 triangles 24.3 -> 23.0 us).
        const uint64_t qw = (uint64_t)job.total_tri + job.total_px / 8u + job.total_vtx / 32u;
        const unsigned qb = grid_for(qw * 32u, cfg.queue_blocks < 1u ? 1u : cfg.queue_blocks);
        if ((e = launch_dependent(k_queue_raster, qb, 256, job, s)) != cudaSuccess) return e;
    }
    if ((e = mark(4)) != cudaSuccess || (e = refused(6)) != cudaSuccess) return e;
    // part 1: transparent fragments, read against the opaque winners' keys
    if ((e = dg_launch_transparent(1, job, cfg.tplan, s)) != cudaSuccess) return e;
    if ((e = refused(7)) != cudaSuccess) return e;
    if (job.total_tiles) {
        NvtxRange r("k_resolve");
        using KR = void (*)(const DgJobDev);
        // [lazy][ext][tile rows 8, 16, 32]
        static const KR kr_table[2][2][3] = {
            {{k_resolve<8, false, false>, k_resolve<16, false, false>, k_resolve<32, false, false>},
             {k_resolve<8, true, false>, k_resolve<16, true, false>, k_resolve<32, true, false>}},
            {{k_resolve<8, false, true>, k_resolve<16, false, true>, k_resolve<32, false, true>},
             {k_resolve<8, true, true>, k_resolve<16, true, true>, k_resolve<32, true, true>}}};
        static const KR split_table[2][2] = {{k_resolve_split<false, false>, k_resolve_split<true, false>},
                                             {k_resolve_split<false, true>, k_resolve_split<true, true>}};
        const int lz = job.lazy ? 1 : 0, ex = job.ext ? 1 : 0;
        const KR kr = job.split_below ? split_table[lz][ex]
                                      : kr_table[lz][ex][job.tile_rows == 8u ? 0 : job.tile_rows == 16u ? 1 : 2];
        const unsigned grid = job.split_below ? 4u * job.total_tiles : job.total_tiles;
        if ((e = launch_dependent(kr, grid, 256, job, s)) != cudaSuccess) return e;
    }
    if ((e = refused(8)) != cudaSuccess) return e;
    // part 2: the ordered blend over the opaque colours
    if ((e = dg_launch_transparent(2, job, cfg.tplan, s)) != cudaSuccess) return e;
    return mark(5);
}

cudaError_t dg_launch_fill(uint32_t* colour, float* depth, uint64_t n, uint32_t colour_value, float depth_value,
                           int fill_colour, int fill_depth, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    k_fill<<<grid_for(n, 4096u), 256, 0, s>>>(colour, depth, n, colour_value, depth_value, fill_colour, fill_depth);
    return cudaGetLastError();
}

cudaError_t dg_launch_bgra_to_rgba(const uint32_t* src, uint32_t* dst, uint64_t n, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    k_bgra_to_rgba<<<grid_for(n, 4096u), 256, 0, s>>>(src, dst, n);
    return cudaGetLastError();
}

cudaError_t dg_launch_vis_reset(uint64_t* vis, uint64_t n, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    k_vis_reset<<<grid_for(n, 4096u), 256, 0, s>>>(vis, n);
    return cudaGetLastError();
}
