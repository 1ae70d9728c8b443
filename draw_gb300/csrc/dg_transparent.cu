// dg_transparent.cu -- the transparent pass of Scene::render on the GPU
// (scene/mod.rs:1088-1247 with canvas.rs:906-930 and the Pixel arithmetic of
// canvas.rs:136-169), and the 2D overlay triangles of Canvas::draw_triangle
// (canvas.rs:435-575), the other order-dependent blend of the reference.
//
// In the reference, each object draws its opaque meshes with depth writes on,
// then its transparent meshes with depth writes off: every transparent mesh is
// first re-sorted in place by descending distance of its triangle centres from
// the camera (a stable sort; the order persists into the next frame), then its
// triangles are clipped and rasterized, and every fragment whose depth is below
// the depth buffer blends into the colour buffer:
//   colour = bg * (1 - alpha) + colour * alpha
// with each product truncated to u8 and the sum wrapping per channel.
//
// The order-independent formulation used here: let j* be the pixel's winning
// opaque fragment (the last opaque write) and d* its depth. Transparent
// fragments submitted before j* are overwritten by it; those after it (objects
// at or after j*'s object) see the depth buffer at d*. So the final colour is
// the opaque result blended, in submission order, with exactly the transparent
// fragments that come from an object at or after j*'s and whose depth is < d*
// (d* = the clear depth and every object qualifies when no opaque fragment
// covers the pixel). The pass:
//   part 0 (after the opaque setup; the sort beside it in a job with k_front):
//          the painter's sort of each mesh (one block per mesh in shared memory,
//          or keys, a stable LSD radix sort and the permutation for larger ones)
//          into the new persistent order, and the transparent setup (clipping,
//          triangle records, bounding boxes, vertices marked for lighting);
//   part 1 (after the opaque raster, while the visibility keys still hold j*):
//          the work items of the outputs' bounding boxes are rasterized with the
//          exact coverage test, and every qualifying fragment is shaded and
//          linked into its pixel's list;
//   part 2 (after the opaque resolve has written the opaque colours): each
//          pixel's list is put in submission order and blended.
#include "dg_device.cuh"

namespace {

// ------------------------------------------------------------ radix sort
// Stable LSD radix sort of 64-bit keys with 32-bit values, one 8-bit digit per
// pass: per-tile digit histograms, one exclusive scan over (digit, tile), and a
// scatter that ranks keys within each tile in their original order (a warp's
// keys with __match_any_sync, then warp by warp).
struct DgSortArgs {
    const uint64_t* key_in;
    const uint32_t* val_in;
    uint64_t* key_out;
    uint32_t* val_out;
    uint32_t* hist;  // 256 per tile, digit-major
    uint32_t n;
    uint32_t shift;
};
constexpr uint32_t kSortItems = DG_SORT_TILE / 256u;  // keys per thread and tile

__global__ void __launch_bounds__(256) k_sort_hist(const DgSortArgs a) {
    __shared__ uint32_t h[256];
    wait_previous_kernel();
    const uint32_t n = a.n;
    const uint32_t ntiles = (n + DG_SORT_TILE - 1u) / DG_SORT_TILE;
    for (uint32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        h[threadIdx.x] = 0u;
        __syncthreads();
        for (uint32_t i = 0; i < kSortItems; i++) {
            const uint32_t idx = tile * DG_SORT_TILE + i * 256u + threadIdx.x;
            if (idx < n) atomicAdd(&h[(uint32_t)(a.key_in[idx] >> a.shift) & 255u], 1u);
        }
        __syncthreads();
        a.hist[threadIdx.x * ntiles + tile] = h[threadIdx.x];
        __syncthreads();
    }
}

// Exclusive scan of n u32 counts in place (one block of 1024 threads, each a
// contiguous chunk).
__device__ __forceinline__ void block_scan_1024(uint32_t* data, uint32_t n) {
    __shared__ uint32_t part[1024];
    const uint32_t chunk = (n + 1023u) / 1024u;
    const uint32_t b = threadIdx.x * chunk;
    const uint32_t e = b + chunk < n ? b + chunk : n;
    uint32_t sum = 0;
    for (uint32_t i = b; i < e; i++) sum += data[i];
    part[threadIdx.x] = sum;
    __syncthreads();
    for (uint32_t o = 1; o < 1024u; o <<= 1) {
        const uint32_t v = threadIdx.x >= o ? part[threadIdx.x - o] : 0u;
        __syncthreads();
        part[threadIdx.x] += v;
        __syncthreads();
    }
    uint32_t run = part[threadIdx.x] - sum;
    for (uint32_t i = b; i < e; i++) {
        const uint32_t c = data[i];
        data[i] = run;
        run += c;
    }
}

__global__ void __launch_bounds__(1024) k_sort_scan(const DgSortArgs a) {
    wait_previous_kernel();
    const uint32_t n = a.n;
    block_scan_1024(a.hist, 256u * ((n + DG_SORT_TILE - 1u) / DG_SORT_TILE));
}

__global__ void __launch_bounds__(256) k_sort_scatter(const DgSortArgs a) {
    __shared__ uint32_t wc[8][257];  // per-warp digit counts ([256]: keys past the end)
    wait_previous_kernel();
    const uint32_t n = a.n;
    const uint32_t ntiles = (n + DG_SORT_TILE - 1u) / DG_SORT_TILE;
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    for (uint32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        for (uint32_t i = threadIdx.x; i < 8u * 257u; i += 256u) (&wc[0][0])[i] = 0u;
        __syncthreads();
        uint32_t dig[kSortItems], rank[kSortItems];
        const uint32_t base = tile * DG_SORT_TILE + w * (DG_SORT_TILE / 8u);
#pragma unroll
        for (uint32_t i = 0; i < kSortItems; i++) {  // the warp's keys in their order
            const uint32_t idx = base + i * 32u + lane;
            const uint32_t d = idx < n ? (uint32_t)(a.key_in[idx] >> a.shift) & 255u : 256u;
            const unsigned peers = __match_any_sync(0xFFFFFFFFu, d);
            const uint32_t before = wc[w][d];
            __syncwarp();
            if (lane == (uint32_t)(__ffs(peers) - 1)) wc[w][d] = before + (uint32_t)__popc(peers);
            __syncwarp();
            dig[i] = d;
            rank[i] = before + (uint32_t)__popc(peers & ((1u << lane) - 1u));
        }
        __syncthreads();
        {  // offsets of each warp's keys among the tile's keys of the same digit
            uint32_t run = 0;
            for (uint32_t ww = 0; ww < 8u; ww++) {
                const uint32_t c = wc[ww][threadIdx.x];
                wc[ww][threadIdx.x] = run;
                run += c;
            }
        }
        __syncthreads();
#pragma unroll
        for (uint32_t i = 0; i < kSortItems; i++) {
            const uint32_t idx = base + i * 32u + lane;
            if (idx < n) {
                const uint32_t d = dig[i];
                const uint32_t pos = a.hist[d * ntiles + tile] + wc[w][d] + rank[i];
                a.key_out[pos] = a.key_in[idx];
                a.val_out[pos] = a.val_in[idx];
            }
        }
        __syncthreads();
    }
}

// One pass per shift; an even number of passes leaves the result in buffer 0.
cudaError_t radix_sort(uint64_t* const key[2], uint32_t* const val[2], uint32_t* hist, uint32_t n,
                       const uint32_t* shifts, uint32_t npass, unsigned blocks, cudaStream_t s) {
    cudaError_t e = cudaSuccess;
    const unsigned tiles = (n + DG_SORT_TILE - 1u) / DG_SORT_TILE;
    const unsigned grid = tiles < blocks ? (tiles ? tiles : 1u) : blocks;
    for (uint32_t p = 0; p < npass && e == cudaSuccess; p++) {
        DgSortArgs a;
        a.key_in = key[p & 1u];
        a.val_in = val[p & 1u];
        a.key_out = key[(p + 1u) & 1u];
        a.val_out = val[(p + 1u) & 1u];
        a.hist = hist;
        a.n = n;
        a.shift = shifts[p];
        if ((e = launch_dependent(k_sort_hist, grid, 256, a, s)) != cudaSuccess) break;
        if ((e = launch_dependent(k_sort_scan, 1u, 1024, a, s)) != cudaSuccess) break;
        e = launch_dependent(k_sort_scatter, grid, 256, a, s);
    }
    return e;
}

// ----------------------------------------------------------- part 0
__device__ __forceinline__ uint32_t seg_of_ttri(const DgJobDev& job, uint32_t j) {
    return last_le(job.nsegs, j, [&](uint32_t i) { return job.segs[i].t_begin; });
}

// Painter's sort key, scene/mod.rs:1100-1115: the distance of a triangle's
// centre (a + b + c) / 3.0 from the camera, in descending f32::total_cmp order.
__device__ __forceinline__ uint32_t painter_key(const DgSegDev& sg, const DgFrameDev& fr, uint32_t loc) {
    const uint4 tp = __ldg(sg.tsrc[0] + loc);
    const float4 pa = __ldg(sg.pos + tp.x), pb = __ldg(sg.pos + tp.y), pc = __ldg(sg.pos + tp.z);
    const V3 ctr = vdiv(vadd(vadd(V3{pa.x, pa.y, pa.z}, V3{pb.x, pb.y, pb.z}), V3{pc.x, pc.y, pc.z}), 3.0f);
    const float dist = vnorm(vsub(ctr, V3{fr.cam[0], fr.cam[1], fr.cam[2]}));  // Vec3::dist, linalg.rs:177-180
    const uint32_t bits = __float_as_uint(dist);
    const uint32_t ord = (bits & 0x80000000u) ? ~bits : (bits | 0x80000000u);  // total_cmp order
    return ~ord;
}

// The painter's sort of one mesh per block, in shared memory: a bitonic sort of
// (painter_key << 32 | current slot), a total order, so the sort is stable; then
// the permutation into the new persistent order. Bound by the barriers of the
// wide exchange steps; those within 64 keys stay inside a warp. For meshes of at
// most DG_TSORT_MAX triangles it replaces k_tkeys, six or more radix passes of
// three kernels and k_tgather (24 meshes of 800 triangles: 210 us).
template <class SEG, class FRM>
__device__ __forceinline__ void dev_tsort(uint32_t nsegs, SEG seg, FRM frame) {
    extern __shared__ uint64_t s_key[];
    const uint32_t mesh = blockIdx.x;
    const DgSegDev& sg = seg(last_le(nsegs, mesh, [&](uint32_t i) { return seg(i).tmesh_base; }));
    const DgFrameDev& fr = frame(sg.frame);
    const uint32_t first = __ldg(sg.tmesh_off + (mesh - sg.tmesh_base));
    const uint32_t n = __ldg(sg.tmesh_off + (mesh - sg.tmesh_base) + 1u) - first;
    uint32_t n2 = 64u;  // keys sorted: a power of two, at least one warp's
    while (n2 < n) n2 *= 2u;
    for (uint32_t i = threadIdx.x; i < n2; i += blockDim.x)
        s_key[i] = i < n ? ((uint64_t)painter_key(sg, fr, first + i) << 32) | i : ~0ull;
    __syncthreads();
    for (uint32_t size = 2u; size <= n2; size *= 2u)
        for (uint32_t j = size / 2u; j != 0u; j /= 2u) {
            for (uint32_t t = threadIdx.x; t < n2 / 2u; t += blockDim.x) {
                const uint32_t i = 2u * t - (t & (j - 1u));
                const uint64_t a = s_key[i], b = s_key[i + j];
                if ((a > b) == ((i & size) == 0u)) {
                    s_key[i] = b;
                    s_key[i + j] = a;
                }
            }
            // the next step's pairs: within this warp's 64 keys when both distances are at most 32
            if (j > 32u || (j == 1u && size >= 64u))
                __syncthreads();
            else
                __syncwarp();
        }
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
        const uint32_t src = first + (uint32_t)s_key[i];
#pragma unroll
        for (int k = 0; k < 3; k++) sg.tdst[k][first + i] = __ldg(sg.tsrc[k] + src);
    }
}

__global__ void __launch_bounds__(1024) k_tsort(const __grid_constant__ DgJobDev job) {
    wait_previous_kernel();
    dev_tsort(job.nsegs, [&](uint32_t i) -> const DgSegDev& { return job.segs[i]; },
              [&](uint32_t i) -> const DgFrameDev& { return job.frames[i]; });
}
// The same as the first kernel of a job with k_front, on the descriptors that
// travel with the job: neither reads what the other writes, so k_front starts
// under it (and waits for it at its end, so that the kernels after k_front find
// both complete). Measured on a 1280x720 frame with 24 transparent meshes of 812
// triangles: the frame 168.7 -> 160.5 us.
template <class IN>
__global__ void __launch_bounds__(1024) k_tsort_first(const __grid_constant__ IN in) {
    allow_next_kernel();  // the first kernel of a job waits on nothing (a stream-ordered launch)
    dev_tsort(in.nsegs, [&](uint32_t i) -> const DgSegDev& { return in.segs[i]; },
              [&](uint32_t i) -> const DgFrameDev& { return in.frames[IN::kFrames == 1u ? 0u : i]; });
}

// Keys of the radix sort: the painter's key behind the job-wide index of the
// triangle's mesh; the value is the triangle's current slot.
__global__ void __launch_bounds__(256) k_tkeys(const DgJobDev job) {
    wait_previous_kernel();
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < job.ntt; j += stride) {
        const DgSegDev& sg = job.segs[seg_of_ttri(job, j)];
        const DgFrameDev& fr = job.frames[sg.frame];
        const uint32_t loc = j - sg.t_begin;
        const uint32_t mesh = __ldg(sg.tsrc[1] + loc).w;
        job.tkey[0][j] = ((uint64_t)(sg.tmesh_base + mesh) << 32) | painter_key(sg, fr, loc);
        job.tval[0][j] = j;
    }
}

// The new persistent order: slot j receives the triangle the sort put there.
__global__ void __launch_bounds__(256) k_tgather(const DgJobDev job) {
    wait_previous_kernel();
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < job.ntt; j += stride) {
        const DgSegDev& sg = job.segs[seg_of_ttri(job, j)];
        const uint32_t src = job.tval[0][j] - sg.t_begin;  // same mesh, so the same segment
        const uint32_t dst = j - sg.t_begin;
#pragma unroll
        for (int k = 0; k < 3; k++) sg.tdst[k][dst] = __ldg(sg.tsrc[k] + src);
    }
}

// Transparent setup, one sorted triangle per thread: lateral reject and
// near/far clipping (no back-face test in this pass, scene/mod.rs:1117-1227),
// a triangle record and a bounding box per clip output (4 j + o), light rows
// of the clip vertices at total_vtx + vrow_extra + 6 j, and the work items of
// the outputs' boxes.
__global__ void __launch_bounds__(256) k_tsetup(const DgJobDev job) {
    wait_previous_kernel();
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t stride = gridDim.x * blockDim.x;
    // warp-uniform loop: the items are handed out to whole warps
    for (uint32_t base = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u; base < job.ntt; base += stride) {
        const uint32_t j = base + lane;
        const bool valid = j < job.ntt;
        const uint32_t si = seg_of_ttri(job, valid ? j : base);
        const DgSegDev& sg = job.segs[si];
        const DgFrameDev& fr = job.frames[sg.frame];
        uint4 tp = make_uint4(0, 0, 0, 0), tuv = tp, tnr = tp;
        float4 r[3];
        const uint32_t rowbase = job.total_vtx + job.vrow_extra + 6u * j;
        ClipProg P;
        int nout = 0;
        bool clipped = false;
        float alpha = 1.0f;
        if (valid) {
            const uint32_t loc = j - sg.t_begin;
            tp = __ldg(sg.tdst[0] + loc);
            tuv = __ldg(sg.tdst[1] + loc);
            tnr = __ldg(sg.tdst[2] + loc);
            triangle_vertices(job, sg, fr, tp, r);
            const uint32_t m = __float_as_uint(r[0].w) & __float_as_uint(r[1].w) & __float_as_uint(r[2].w);
            if ((m >> 8) & 0x3Cu) {
                nout = 0;  // outside a lateral plane (scene/mod.rs:59-66)
            } else if ((m & 0x3u) == 0x3u) {
                nout = 1;  // inside near and far
            } else {
                float4 pa = __ldg(sg.pos + tp.x), pb = __ldg(sg.pos + tp.y), pc = __ldg(sg.pos + tp.z);
                build_clip(fr, V3{pa.x, pa.y, pa.z}, V3{pb.x, pb.y, pb.z}, V3{pc.x, pc.y, pc.z}, P);
                nout = P.nout;
                clipped = true;
                if (nout > 0 && P.nv > 3) clip_shade_rows(job, fr, P, rowbase);
            }
            if (nout > 0) {  // its vertices need light/halfway vectors for shading
                const uint32_t vv[3] = {sg.vtx_begin + tp.x, sg.vtx_begin + tp.y, sg.vtx_begin + tp.z};
                for (int k = 0; k < 3; k++) job.vmark[vv[k]] = 1u;
            }
            alpha = tp.w < sg.nmats ? __ldg(&sg.mats[tp.w].alpha) : 1.0f;
        }
        const uint32_t tseq = (j - fr.tt_begin) << 2;
        for (int o = 0; o < 4; o++) {
            if (__ballot_sync(FULL, o < nout) == 0u) break;
            const uint32_t ri = 4u * j + (uint32_t)o;
            uint32_t px = 0;  // bounding-box pixels, 0: no output
            if (o < nout) {
                RTri tr;
                if (!clipped) {
                    tr.ax = r[0].x; tr.ay = r[0].y;
                    tr.bx = r[1].x; tr.by = r[1].y;
                    tr.cx = r[2].x; tr.cy = r[2].y;
                    tr.da = r[0].z; tr.db = r[1].z; tr.dc = r[2].z;
                } else {
                    clip_output_tri(fr, P, o, r, tr);
                }
                const bool nan = isnan(tr.ax) || isnan(tr.ay) || isnan(tr.bx) || isnan(tr.by) || isnan(tr.cx) ||
                                 isnan(tr.cy);
                if (!nan) {  // any NaN centre makes every barycentric NaN: nothing is covered
                    EdgeSet e;
                    bbox_axis(tr.ax, tr.bx, tr.cx, fr.width, tr.xlo, tr.xhi);
                    bbox_axis(tr.ay, tr.by, tr.cy, fr.height, tr.ylo, tr.yhi);
                    make_edges(tr.ax, tr.ay, tr.bx, tr.by, tr.cx, tr.cy, e);
                    float4* wout = (fr.flags & DG_FRAME_PERSPECTIVE) && job.ttrec_w ? job.ttrec_w + ri : nullptr;
                    if (!clipped)
                        write_record(job, job.ttrec + ri, sg, tp, tuv, tnr, e, r, fr, wout);
                    else
                        write_clip_record(job, job.ttrec + ri, sg, tp, tuv, tnr, e, tr, P, o, rowbase, fr, wout);
                    px = (tr.xhi - tr.xlo + 1u) * (tr.yhi - tr.ylo + 1u);  // below 2^31: the canvas is smaller
                    job.tbox[ri] = make_uint4(tr.xlo, tr.ylo, tr.xhi - tr.xlo + 1u, sg.frame);
                    job.tmeta[ri] = make_uint2(sg.obj_rank, tseq | (uint32_t)o);
                    job.talpha[ri] = alpha;
                }
            }
            // Work items of DG_TITEM_UNITS units: the first one of each output in the
            // first 4 ntt entries (they always fit), the further ones after them.
            const uint32_t units = (px + DG_UNIT_PX - 1u) / DG_UNIT_PX;
            const uint32_t more = px ? (units - 1u) / DG_TITEM_UNITS : 0u;
            const unsigned long long first = warp_alloc(job.cnt + DG_CNT_TITEM, px ? 1u : 0u);
            const unsigned long long ext = 4ull * job.ntt + warp_alloc(job.cnt + DG_CNT_TITEMX, more);
            const bool fits = ext + more <= job.titem_cap;
            if (px) job.titem[first] = make_uint4(ri, 0u, fits ? min(units, DG_TITEM_UNITS) : units, px);
            const uint32_t own = fits && more < 32u ? more : 0u;
            for (uint32_t k = 0; k < own; k++)
                job.titem[ext + k] = make_uint4(ri, (k + 1u) * DG_TITEM_UNITS, min(units, (k + 2u) * DG_TITEM_UNITS), px);
            unsigned big = __ballot_sync(FULL, more >= 32u);  // large boxes: the whole warp writes
            while (big) {
                const int L = __ffs(big) - 1;
                big &= big - 1u;
                const uint32_t lmore = __shfl_sync(FULL, more, L), lri = __shfl_sync(FULL, ri, L);
                const uint32_t lunits = __shfl_sync(FULL, units, L), lpx = __shfl_sync(FULL, px, L);
                const unsigned long long lext = __shfl_sync(FULL, ext, L);
                const bool lfits = lext + lmore <= job.titem_cap;
                for (uint32_t k = lane; k < lmore; k += 32u)
                    if (lext + k < job.titem_cap)
                        job.titem[lext + k] = lfits ? make_uint4(lri, (k + 1u) * DG_TITEM_UNITS,
                                                                 min(lunits, (k + 2u) * DG_TITEM_UNITS), lpx)
                                                    : make_uint4(0u, 0u, 0u, 0u);
            }
            if (!fits && more < 32u)  // handed-out entries that stay unused are empty
                for (uint32_t k = 0; k < more; k++)
                    if (ext + k < job.titem_cap) job.titem[ext + k] = make_uint4(0u, 0u, 0u, 0u);
        }
    }
}

// ----------------------------------------------------------- part 1
// Fragments as one linked list per pixel. A warp takes nodes from the shared
// array DG_FRAG_CHUNK at a time (one counter update per chunk: an update per 32
// fragments serializes at the L2). Every lane of the warp calls take().
struct FragNodes {
    uint4* node;
    uint32_t cap;
    unsigned long long* slots;  // nodes handed out
    uint32_t base, left;        // the warp's current chunk
    uint32_t total;             // fragments of this warp
    // The node index of this lane's fragment, or DG_NONE (no fragment, or no node left).
    __device__ __forceinline__ uint32_t take(bool emit, uint32_t* err) {
        const uint32_t lane = threadIdx.x & 31u;
        const unsigned em = __ballot_sync(FULL, emit);
        const uint32_t m = (uint32_t)__popc(em), rank = (uint32_t)__popc(em & ((1u << lane) - 1u));
        uint32_t next = DG_NONE;
        if (m > left) {
            unsigned long long b = 0;
            if (lane == 0u) b = atomicAdd(slots, (unsigned long long)DG_FRAG_CHUNK);
            b = __shfl_sync(FULL, b, 0);
            if (b + DG_FRAG_CHUNK <= cap) next = (uint32_t)b;
        }
        uint32_t slot = DG_NONE;
        if (emit) {
            if (rank < left)
                slot = base + rank;
            else if (next != DG_NONE)
                slot = next + (rank - left);
            else
                atomicOr(err, 1u << DG_E_LIMIT);
        }
        total += m;
        if (m <= left) {
            base += m;
            left -= m;
        } else if (next != DG_NONE) {
            base = next + (m - left);
            left = DG_FRAG_CHUNK - (m - left);
        } else {
            left = 0u;
        }
        return slot;
    }
};
// Links a fragment's node in front of its pixel's list.
__device__ __forceinline__ void link_fragment(uint4* node, uint32_t* head, uint32_t slot, uint32_t key, uint32_t colour,
                                              float alpha) {
    const uint32_t prev = atomicExch(head, slot + 1u);
    node[slot] = make_uint4(prev, key, colour, __float_as_uint(alpha));
}

// The depth of a visibility key (the inverse of depth_key's order-preserving map).
__device__ __forceinline__ float key_depth(uint64_t key) {
    const uint32_t hi = (uint32_t)(key >> 32);
    return __uint_as_float((hi & 0x80000000u) ? (hi & 0x7FFFFFFFu) : ~hi);
}

// Rasterizes the transparent outputs' boxes and shades the qualifying
// fragments. Bound by the latency of the shading chain (record, light rows,
// texel), so every 32 shading lanes are kept busy: each warp tests its items'
// box pixels one per lane (division-free), packs the candidates of all its
// items into one buffer, and finishes them 32 at a time: the exact coverage
// test, the depth, the qualifying test against the pixel's opaque winner (its
// key is still in the visibility buffer: depth < d* and the triangle's object
// at or after the winner's), the shading, and the link into the pixel's list.
// Measured on a 1280x720 frame with 19,000 transparent triangles and about 0.9M
// fragments: 80 us (37M warp instructions, most of them the shading); see k_tfold
// for the form it replaced.
template <bool EXT>
__global__ void __launch_bounds__(256, DG_TRASTER_BLOCKS_PER_SM) k_traster(const __grid_constant__ DgJobDev job) {
    __shared__ float inv255[256];
    __shared__ DgTexDev stex[DG_SMEM_TEX];
    __shared__ uint32_t s_xy[8][64], s_rec[8][64];  // per-warp candidates: y << 16 | x, output record
    inv255[threadIdx.x] = fD((float)threadIdx.x, 255.0f);
    const uint32_t nst = job.ntex < DG_SMEM_TEX ? job.ntex : DG_SMEM_TEX;
    for (uint32_t i = threadIdx.x; i < nst * 3u; i += blockDim.x)
        reinterpret_cast<uint4*>(stex)[i] = __ldg(reinterpret_cast<const uint4*>(job.tex) + i);
    wait_previous_kernel();
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t* bxy = s_xy[threadIdx.x >> 5];
    uint32_t* brec = s_rec[threadIdx.x >> 5];
    FragNodes nodes = {job.fnode, job.fnode_cap, job.cnt + DG_CNT_TSLOT, 0u, 0u, 0u};
    uint32_t pending = 0;
    // Finishes the first n (<= 32) buffered candidates, one per lane (converged warp).
    auto finish = [&](uint32_t n) {
        bool emit = false;
        uint32_t rec = 0, x = 0, y = 0, pix = 0, key = 0;
        const DgFrameDev* fr = nullptr;
        if (lane < n) {
            rec = brec[lane];
            x = bxy[lane] & 0xFFFFu;
            y = bxy[lane] >> 16;
            const DgTriRec* R = job.ttrec + rec;
            EdgeSet e;
            load_edges<false>(R, e);
            float al, be, ga;
            if (covered(e, (float)x, (float)y, al, be, ga)) {
                fr = job.frames + __ldcg(&job.tbox[rec].w);
                const float4 dd = __ldg(reinterpret_cast<const float4*>(R) + 4);
                const float depth = interp(al, be, ga, dd.x, dd.y, dd.z);
                const uint32_t local = y * fr->width + x;
                const uint64_t vk = __ldcg(reinterpret_cast<const unsigned long long*>(fr->vis) + local);
                float dstar = fr->clear_depth;
                int objj = -1;
                if (vk != DG_VIS_EMPTY) {
                    dstar = key_depth(vk);
                    const uint32_t tl = (uint32_t)vk >> 2;
                    objj = (int)last_le(fr->seg_count, tl, [&](uint32_t s) { return job.segs[fr->seg_begin + s].seq_base; });
                }
                const uint2 meta = __ldcg(job.tmeta + rec);
                if (depth < dstar && (int)meta.x >= objj) {
                    emit = true;
                    pix = fr->pix_begin + local;
                    key = meta.y;
                }
            }
        }
        const uint32_t slot = nodes.take(emit, job.err);
        if (slot != DG_NONE) {
            float d;
            int errc;
            const float4* wp = EXT && (fr->flags & DG_FRAME_PERSPECTIVE) && job.ttrec_w ? job.ttrec_w + rec : nullptr;
            const uint32_t c = shade_from_record<EXT, false, false>(job, *fr, job.ttrec + rec, x, y, inv255, stex, d, errc, wp, nullptr);
            if (errc != DG_OK) atomicOr(job.err, 1u << errc);
            link_fragment(job.fnode, job.fhead + pix, slot, key, c, __ldcg(job.talpha + rec));
        }
        __syncwarp();
    };
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t n1 = (uint32_t)__ldcg(job.cnt + DG_CNT_TITEM);  // at most 4 ntt
    const unsigned long long nx = __ldcg(job.cnt + DG_CNT_TITEMX);
    const uint32_t room = job.titem_cap - 4u * job.ntt;
    const uint32_t n2 = (uint32_t)(nx < room ? nx : room);
    // One unit per iteration; the last iterations drain the buffer.
    uint4 item = make_uint4(0u, 0u, 0u, 0u), box = item;
    EdgeSet e;
    bool fast = false;
    uint32_t k = 0, yy = 0, xx = 0, q32 = 0, r32 = 0;
    for (uint32_t wi = warp;;) {
        while (item.y >= item.z && wi < n1 + n2) {  // next item (entries left empty are skipped)
            item = __ldcg(job.titem + (wi < n1 ? wi : 4u * job.ntt + (wi - n1)));
            wi += nwarps;
            if (item.y >= item.z) continue;
            box = __ldcg(job.tbox + item.x);
            load_edges<false>(job.ttrec + item.x, e);
            fast = (e.tie & DG_EDGE_FAST) != 0u;
            // this lane's pixel of the box, stepped by DG_UNIT_PX pixels per unit (as in the opaque raster)
            k = item.y * DG_UNIT_PX + lane;
            yy = k / box.z;
            xx = k - yy * box.z;
            q32 = DG_UNIT_PX / box.z;
            r32 = DG_UNIT_PX - q32 * box.z;
        }
        const bool drain = item.y >= item.z;
        if (drain && pending == 0u) break;
        if (!drain) {
            const uint32_t x = box.x + xx, y = box.y + yy;
            bool cand = false;
            if (k < item.w) {
                const float xf = (float)x, yf = (float)y;
                const float n0_ = edge_eval(e, 0, xf, yf), n1_ = edge_eval(e, 1, xf, yf), n2_ = edge_eval(e, 2, xf, yf);
                cand = fast ? covered_signs(e.tie, n0_, n1_, n2_)
                            : !(prereject(n0_, e.den[0]) || prereject(n1_, e.den[1]) || prereject(n2_, e.den[2]));
            }
            const unsigned b = __ballot_sync(FULL, cand);
            if (cand) {
                const uint32_t at = pending + (uint32_t)__popc(b & ((1u << lane) - 1u));
                bxy[at] = (y << 16) | x;
                brec[at] = item.x;
            }
            pending += (uint32_t)__popc(b);
            item.y++;
            k += DG_UNIT_PX;
            xx += r32;
            yy += q32;
            if (xx >= box.z) {
                xx -= box.z;
                yy++;
            }
        }
        if (drain || pending >= 32u) {
            const uint32_t n = pending < 32u ? pending : 32u;
            __syncwarp();
            finish(n);
            if (lane < pending - n) {
                bxy[lane] = bxy[32u + lane];
                brec[lane] = brec[32u + lane];
            }
            __syncwarp();
            pending -= n;
        }
    }
    if (lane == 0u && nodes.total) atomicAdd(job.cnt + DG_CNT_TFRAG, (unsigned long long)nodes.total);
}

// ----------------------------------------------------------- part 2
// Pixel * f32 (canvas.rs:155-169): each channel (c as f32 * f) as u8, padd 0.
__device__ __forceinline__ uint32_t px_mul(uint32_t p, float f) {
    const uint32_t b = as_u8(fM((float)(p & 0xFFu), f));
    const uint32_t g = as_u8(fM((float)((p >> 8) & 0xFFu), f));
    const uint32_t r = as_u8(fM((float)((p >> 16) & 0xFFu), f));
    return b | (g << 8) | (r << 16);
}
// Pixel + Pixel (canvas.rs:136-153): u8 channel sums (wrapping), padd 0.
__device__ __forceinline__ uint32_t px_add(uint32_t p, uint32_t q) {
    return ((p + q) & 0xFFu) | (((p >> 8) + (q >> 8)) & 0xFFu) << 8 | (((p >> 16) + (q >> 16)) & 0xFFu) << 16;
}

// Puts a list of fragment nodes in ascending key order (a stable LSD radix sort
// of the links, 4 bits per pass) and returns its head; for lists too long for
// fold_list's registers. Its walks end because every list does: heads are zero
// before a job (JobSlot::dirty, OverlaySlot::dirty) and a job hands every node out
// once. Counting the nodes against the number of keys in the loop doubled the
// time of long lists (200 full-frame layers at 1920x1080: 22.4 -> 45.3 ms).
__device__ __noinline__ uint32_t sort_list(uint4* node, uint32_t head, uint32_t key_bits) {
    for (uint32_t shift = 0; shift < key_bits; shift += 4u) {
        uint32_t hd[16], tl[16];
        for (int d = 0; d < 16; d++) hd[d] = tl[d] = 0u;
        for (uint32_t m = head; m != 0u;) {
            const uint2 nk = *reinterpret_cast<const uint2*>(node + (m - 1u));  // next, key
            const uint32_t d = (nk.y >> shift) & 15u;
            if (hd[d] != 0u)
                node[tl[d] - 1u].x = m;
            else
                hd[d] = m;
            tl[d] = m;
            m = nk.x;
        }
        uint32_t last = 0;
        head = 0;
        for (int d = 0; d < 16; d++) {
            if (hd[d] == 0u) continue;
            if (last != 0u)
                node[last - 1u].x = hd[d];
            else
                head = hd[d];
            last = tl[d];
        }
        node[last - 1u].x = 0u;
    }
    return head;
}

// Blends a pixel's fragments over bg in ascending key order
// (draw_pixel_coord_with_depth, canvas.rs:906-930, with depth writes off).
// Lists of up to kFoldRegs fragments are ordered in registers.
constexpr int kFoldRegs = 8;
__device__ __forceinline__ uint32_t fold_list(uint4* node, uint32_t head, uint32_t key_bits, uint32_t bg) {
    auto blend = [&](uint32_t m) {
        const uint4 f = node[m - 1u];
        const float a = __uint_as_float(f.w);
        bg = a < 1.0f ? px_add(px_mul(bg, fS(1.0f, a)), px_mul(f.z, a)) : f.z;
    };
    uint32_t key[kFoldRegs], at[kFoldRegs];
    int n = 0;
#pragma unroll
    for (int i = 0; i < kFoldRegs; i++) {
        key[i] = DG_NONE;  // above every key
        at[i] = 0u;
    }
    for (uint32_t m = head; m != 0u && n <= kFoldRegs; n++) {
        const uint2 nk = *reinterpret_cast<const uint2*>(node + (m - 1u));
        uint32_t k = nk.y, s = m;
#pragma unroll
        for (int i = 0; i < kFoldRegs; i++)
            if (k < key[i]) {
                const uint32_t tk = key[i], ts = at[i];
                key[i] = k;
                at[i] = s;
                k = tk;
                s = ts;
            }
        m = nk.x;
    }
    if (n <= kFoldRegs) {
#pragma unroll
        for (int i = 0; i < kFoldRegs; i++)
            if (i < n) blend(at[i]);
    } else {
        for (uint32_t m = sort_list(node, head, key_bits); m != 0u; m = node[m - 1u].x) blend(m);
    }
    return bg;
}

// The ordered blend, one pixel per thread. Its reads are the 4-byte heads of all
// pixels and a short chain of nodes per covered one; the fragments were shaded
// when they were rasterized, where they fill whole warps. The earlier form
// (fragments radix-sorted by pixel and key, then shaded here by the thread that
// held the pixel's first one) took 800 us for parts 1 and 2 on the frame of
// k_traster's comment.
__global__ void __launch_bounds__(256) k_tfold(const __grid_constant__ DgJobDev job, const uint32_t key_bits) {
    wait_previous_kernel();
    const uint32_t stride = gridDim.x * blockDim.x;
    if (blockIdx.x == 0u && threadIdx.x == 0u && __ldcg(job.cnt + DG_CNT_TFRAG) > job.fcap)
        atomicOr(job.err, 1u << DG_E_LIMIT);  // more fragments than a job may have
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < job.total_px; p += stride) {
        const uint32_t head = __ldcg(job.fhead + p);
        if (head == 0u) continue;
        job.fhead[p] = 0u;
        const uint32_t fi = last_le(job.nframes, p, [&](uint32_t k) { return job.frames[k].pix_begin; });
        const DgFrameDev& fr = job.frames[fi];
        const uint32_t local = p - fr.pix_begin;
        const uint32_t y = local / fr.width, x = local - y * fr.width;
        uint32_t* colour = fr.colour + (uint64_t)(fr.height - 1u - y) * fr.width + x;
        *colour = fold_list(job.fnode, head, key_bits, *colour);
    }
}

// ------------------------------------------------------------ 2D overlay
// TextureMap::get_rgba_slice (scene/mod.rs:137-152): (u * width) and
// (v * height) floored, wrapping usize offset, four bytes; false where the
// reference's slice index would panic.
__device__ __forceinline__ bool tex_rgba(const DgTexDev& tx, float u, float v, uint32_t& rgba) {
    const uint64_t ui = as_usize(floorf(fM(u, (float)tx.width)));
    const uint64_t vi = (uint64_t)tx.height - 1ull - as_usize(floorf(fM(v, (float)tx.height)));
    const uint64_t off = (vi * (uint64_t)tx.width + ui) * (uint64_t)tx.comps;
    if (tx.len < 4ull || off > tx.len - 4ull) return false;
    const uint64_t w = off >> 2;
    const uint32_t sh = (uint32_t)(off & 3ull) * 8u;
    const uint32_t lo = __ldg(tx.words + w);
    rgba = sh == 0u ? lo : __funnelshift_r(lo, __ldg(tx.words + w + 1), sh);
    return true;
}

// Edges of overlay triangle t from its snapped centres (pos_map_center,
// canvas.rs:896-904).
__device__ __forceinline__ void overlay_edges(const DgOverlayJob& job, uint32_t t, EdgeSet& e) {
    float cx[3], cy[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const float4 a = __ldg(job.verts + 6ull * t + 2 * k);
        cx[k] = floorf(fA(a.x, 0.5f));
        cy[k] = floorf(fA(a.y, 0.5f));
    }
    make_edges(cx[0], cy[0], cx[1], cy[1], cx[2], cy[2], e);
}

// Canvas::draw_triangle's raster and shading (canvas.rs:435-575): the coverage
// test of the 3D rasterizer (the same edge functions and tie rule) on every
// pixel of every clipped bounding box, and for each covered pixel the vertex
// colours and alphas and the texture coordinates interpolated with the
// barycentrics, the RGBA texel and the colour blend with it. A fragment that
// passes draw_pixel_coord_with_depth's depth test at depth 0 (the overlay never
// writes depth: depth updates are off outside the opaque pass) is linked into
// its pixel's list. As in k_traster, a warp packs the candidates of all its items
// and finishes 32 at a time, since a GUI's triangles are glyph quads of a few
// dozen pixels. Measured with k_o_fold on 1,800 triangles over an 800x600 frame:
// 30 us, against 280 for the form with a fragment radix sort (18 + 230 + 20 us
// with a serial fold).
__global__ void __launch_bounds__(256, DG_OVERLAY_BLOCKS_PER_SM) k_o_raster(const __grid_constant__ DgOverlayJob job) {
    __shared__ uint32_t s_xy[8][64], s_tri[8][64];  // per-warp candidates: y << 16 | x, triangle
    wait_previous_kernel();
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t* bxy = s_xy[threadIdx.x >> 5];
    uint32_t* btri = s_tri[threadIdx.x >> 5];
    FragNodes nodes = {job.node, job.node_cap, job.cnt, 0u, 0u, 0u};
    uint32_t pending = 0;
    auto finish = [&](uint32_t n) {  // as in k_traster
        bool emit = false;
        uint32_t tri = 0, pix = 0, cp = 0;
        float fa = 0.0f;
        if (lane < n) {
            tri = btri[lane];
            const uint32_t x = bxy[lane] & 0xFFFFu, y = bxy[lane] >> 16;
            EdgeSet e;
            overlay_edges(job, tri, e);
            float al, be, ga;
            if (covered(e, (float)x, (float)y, al, be, ga)) {
                const float4* v = job.verts + 6ull * tri;
                const float4 a0 = __ldg(v), b0 = __ldg(v + 2), c0 = __ldg(v + 4);      // x, y, u, v
                const float4 a1 = __ldg(v + 1), b1 = __ldg(v + 3), c1 = __ldg(v + 5);  // r, g, b, alpha
                // Color::Custom([r, g, b]).as_pixel(): b, g, r bytes
                auto pixel = [](float4 c) { return (uint32_t)c.z | ((uint32_t)c.y << 8) | ((uint32_t)c.x << 16); };
                // (alpha * color_a) + (beta * color_b) + (gama * color_c): Pixel products and sums
                const uint32_t cp0 = px_add(px_add(px_mul(pixel(a1), al), px_mul(pixel(b1), be)), px_mul(pixel(c1), ga));
                const float calpha = fA(fA(fM(al, a1.w), fM(be, b1.w)), fM(ga, c1.w));
                const float cu = fA(fA(fM(a0.z, al), fM(b0.z, be)), fM(c0.z, ga));
                const float cv = fA(fA(fM(a0.w, al), fM(b0.w, be)), fM(c0.w, ga));
                uint32_t rgba;
                if (!tex_rgba(job.tex, cu, cv, rgba)) {
                    atomicOr(job.err, 1u << DG_E_TEXTURE_RANGE);
                } else {
                    const float talpha = fD((float)(rgba >> 24), 255.0f);
                    const uint32_t ct = ((rgba >> 16) & 0xFFu) | (((rgba >> 8) & 0xFFu) << 8) | ((rgba & 0xFFu) << 16);
                    cp = px_add(px_mul(cp0, talpha), px_mul(ct, fS(1.0f, talpha)));
                    fa = fM(calpha, talpha);
                    pix = y * job.width + x;
                    emit = 0.0f < __ldg(job.depth + pix);
                }
            }
        }
        const uint32_t slot = nodes.take(emit, job.err);
        if (slot != DG_NONE) link_fragment(job.node, job.head + pix, slot, tri, cp, fa);
        __syncwarp();
    };
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    // One unit per iteration; the last iterations drain the buffer.
    uint32_t tri = 0, u = 0, u_end = 0, xx = 0, yy = 0, k = 0, q32 = 0, r32 = 0;
    uint4 box = make_uint4(0u, 0u, 1u, 0u);
    EdgeSet e;
    for (uint32_t wi = warp;;) {
        if (u >= u_end && wi < job.nitems) {
            const uint2 item = __ldg(job.items + wi);
            wi += nwarps;
            tri = item.x;
            u = item.y;
            box = __ldg(job.box + tri);
            u_end = min(u + dg_overlay_units(box.w), (box.w + DG_UNIT_PX - 1u) / DG_UNIT_PX);
            overlay_edges(job, tri, e);
            k = u * DG_UNIT_PX + lane;
            yy = k / box.z;
            xx = k - yy * box.z;
            q32 = DG_UNIT_PX / box.z;
            r32 = DG_UNIT_PX - q32 * box.z;
        }
        const bool drain = u >= u_end;
        if (drain && pending == 0u) break;
        if (!drain) {
            const uint32_t x = box.x + xx, y = box.y + yy;
            bool cand = false;
            if (k < box.w) {
                const float xf = (float)x, yf = (float)y;
                const float n0 = edge_eval(e, 0, xf, yf), n1 = edge_eval(e, 1, xf, yf), n2 = edge_eval(e, 2, xf, yf);
                cand = (e.tie & DG_EDGE_FAST)
                           ? covered_signs(e.tie, n0, n1, n2)
                           : !(prereject(n0, e.den[0]) || prereject(n1, e.den[1]) || prereject(n2, e.den[2]));
            }
            const unsigned b = __ballot_sync(FULL, cand);
            if (cand) {
                const uint32_t at = pending + (uint32_t)__popc(b & ((1u << lane) - 1u));
                bxy[at] = (y << 16) | x;
                btri[at] = tri;
            }
            pending += (uint32_t)__popc(b);
            u++;
            k += DG_UNIT_PX;
            xx += r32;
            yy += q32;
            if (xx >= box.z) {
                xx -= box.z;
                yy++;
            }
        }
        if (drain || pending >= 32u) {
            const uint32_t n = pending < 32u ? pending : 32u;
            __syncwarp();
            finish(n);
            if (lane < pending - n) {
                bxy[lane] = bxy[32u + lane];
                btri[lane] = btri[32u + lane];
            }
            __syncwarp();
            pending -= n;
        }
    }
}

// Each pixel's fragments blended over the canvas in triangle order.
__global__ void __launch_bounds__(256) k_o_fold(const __grid_constant__ DgOverlayJob job) {
    wait_previous_kernel();
    const uint32_t px = job.width * job.height, stride = gridDim.x * blockDim.x;
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < px; p += stride) {
        const uint32_t head = __ldcg(job.head + p);
        if (head == 0u) continue;
        job.head[p] = 0u;
        const uint32_t y = p / job.width, x = p - y * job.width;
        uint32_t* colour = job.colour + (uint64_t)(job.height - 1u - y) * job.width + x;
        *colour = fold_list(job.node, head, job.key_bits, *colour);
    }
}

}  // namespace

cudaError_t dg_launch_overlay(const DgOverlayJob& job, unsigned blocks, cudaStream_t s, bool fail) {
    if (job.n == 0u) return cudaSuccess;
    const unsigned g = blocks < 1u ? 1u : blocks;
    const cudaError_t e = launch_dependent(k_o_raster, g, 256, job, s);
    if (e != cudaSuccess) return e;
    if (fail) return cudaErrorMemoryAllocation;
    return launch_dependent(k_o_fold, g * 4u, 256, job, s);
}

namespace {
unsigned tsort_threads(const DgTransparentPlan& plan) {
    return plan.tsort_pow2 / 2u < 1024u ? plan.tsort_pow2 / 2u : 1024u;
}
}  // namespace

template <class IN>
cudaError_t dg_launch_tsort_first(const IN& in, const DgTransparentPlan& plan, cudaStream_t s) {
    k_tsort_first<<<plan.tsort_meshes, tsort_threads(plan), plan.tsort_pow2 * sizeof(uint64_t), s>>>(in);
    return cudaGetLastError();
}
template cudaError_t dg_launch_tsort_first(const DgInlineDesc&, const DgTransparentPlan&, cudaStream_t);
template cudaError_t dg_launch_tsort_first(const DgInlineBatch&, const DgTransparentPlan&, cudaStream_t);
template cudaError_t dg_launch_tsort_first(const DgInlineLarge&, const DgTransparentPlan&, cudaStream_t);

cudaError_t dg_launch_transparent(int part, const DgJobDev& job, const DgTransparentPlan& plan, cudaStream_t s,
                                  bool sorted) {
    if (job.ntt == 0u) return cudaSuccess;
    const unsigned g = plan.blocks < 1u ? 1u : plan.blocks;
    cudaError_t e = cudaSuccess;
    if (part == 0) {
        if (sorted) {  // by dg_launch_tsort_first
        } else if (plan.tsort_meshes) {
            if ((e = launch_dependent_smem(k_tsort, plan.tsort_meshes, tsort_threads(plan),
                                           plan.tsort_pow2 * sizeof(uint64_t), job, s)) != cudaSuccess)
                return e;
        } else {
            if ((e = launch_dependent(k_tkeys, grid_for(job.ntt, g), 256, job, s)) != cudaSuccess) return e;
            if ((e = radix_sort(job.tkey, job.tval, job.sort_hist, job.ntt, plan.tsort_shift, plan.n_tsort, g,
                                s)) != cudaSuccess)
                return e;
            if ((e = launch_dependent(k_tgather, grid_for(job.ntt, g), 256, job, s)) != cudaSuccess) return e;
        }
        return launch_dependent(k_tsetup, grid_for(job.ntt, g), 256, job, s);
    }
    if (part == 1)
        return launch_dependent(job.ext ? k_traster<true> : k_traster<false>, plan.raster_blocks, 256, job, s);
    return launch_dependent(k_tfold, g * 2u, 256, job, s, plan.key_bits);
}
