// Dice, shade and rasterize kernels.
//
// Batched path: raster_fused dices groups of sub-patches into shared memory
// (a block per group, the group's control points and matrices staged with
// bulk copies while the previous group is processed), applies the
// reference's per-8x8-block rules (a block with a vertex at eye z == 0 is
// dropped, kernels/reyes.cl:130-162; the block bound over front-facing quads
// and its is_empty test of kernels/reyes.cl:287) and rasterizes every quad
// with the integer edge functions of kernels/reyes.cl:240-265.  Visibility is
// one 64-bit atomicMin of (idepth << 32 | micropolygon id) per covered
// pixel, so the nearest fragment wins exactly and ties go to the smaller id.
// No grid is stored: resolve recomputes the winning quad's colour from its id.
//
// Quads whose pixel bbox is small (<= 1024 fixed-point units) and whose
// coordinates are within +-2^19 are rasterized over their own bbox: there the
// wrapped int32 edge functions equal the exact ones, so no pixel outside the
// bbox can pass and the bbox holds every pixel the reference's tile loop
// would accept.  Any other quad goes to raster_big, which replays the
// reference's per-tile candidate loop (kernels/reyes.cl:333-381) exactly.
//
// Plain path: dice_grid / shade_grid / sample_grid keep the reference's
// per-pass structure (kernels/dice.cl, kernels/reyes.cl shade and sample)
// with position, pixel, depth and colour grids in HBM; pass_resolve takes a
// winning fragment's colour from this pass's colour grid.
#include "mp_bns_loop.cuh"

namespace mp {

namespace {

constexpr int kFastCoord = 1 << 19;
constexpr int kFastExtent = 1024;
constexpr int kWidePixels = 4;   // a warp with a box of more pixels sets edges up once (raster_quad_fast)

// Block bound of kernels/reyes.cl:97-166 for one quad: pmin/pmax start at
// the viewport max/min, is_front_facing on the wrapped integer coordinates.
struct QuadBound {
    int pminx, pminy, pmaxx, pmaxy;
    bool ff;
};
__device__ __forceinline__ QuadBound quad_block_bound(const FrameDev& fr, const int* qx, const int* qy) {
    const int vmaxx = (fr.W << fr.shift) - 1, vmaxy = (fr.H << fr.shift) - 1;
    QuadBound b{vmaxx, vmaxy, 0, 0, true};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        b.pminx = min(b.pminx, qx[k]);
        b.pminy = min(b.pminy, qy[k]);
        b.pmaxx = max(b.pmaxx, qx[k]);
        b.pmaxy = max(b.pmaxy, qy[k]);
    }
    if (fr.backface) {
        int d1x = wsub(qx[1], qx[0]), d1y = wsub(qy[1], qy[0]);
        int d2x = wsub(qx[2], qx[0]), d2y = wsub(qy[2], qy[0]);
        int d3x = wsub(qx[3], qx[0]), d3y = wsub(qy[3], qy[0]);
        b.ff = wsub(wmul(d1x, d3y), wmul(d3x, d1y)) < 0 || wsub(wmul(d3x, d2y), wmul(d2x, d3y)) < 0;
    }
    return b;
}

// Final block bound (clamp, allnormal) -> tile range; returns false when the
// block is skipped by the is_empty(block_bound.xy, block_bound.zx) test.
__device__ __forceinline__ bool block_tiles(const FrameDev& fr, int xmin, int ymin, int xmax, int ymax,
                                            bool allnormal, int* tiles) {
    const int vmaxx = (fr.W << fr.shift) - 1, vmaxy = (fr.H << fr.shift) - 1;
    xmin = max(0, xmin);
    ymin = max(0, ymin);
    xmax = min(vmaxx, xmax);
    ymax = min(vmaxy, ymax);
    if (!allnormal) { xmin = 1; ymin = 1; xmax = -1; ymax = -1; }
    if (xmin >= xmax && ymin >= xmin) return false;
    tiles[0] = xmin >> (fr.shift + 3);
    tiles[1] = ymin >> (fr.shift + 3);
    tiles[2] = xmax >> (fr.shift + 3);
    tiles[3] = ymax >> (fr.shift + 3);
    return true;
}

__device__ __forceinline__ bool quad_is_fast(const int* qx, const int* qy, int& minx, int& miny, int& maxx,
                                             int& maxy) {
    minx = min(min(qx[0], qx[1]), min(qx[2], qx[3]));
    maxx = max(max(qx[0], qx[1]), max(qx[2], qx[3]));
    miny = min(min(qy[0], qy[1]), min(qy[2], qy[3]));
    maxy = max(max(qy[0], qy[1]), max(qy[2], qy[3]));
    if (minx < -kFastCoord || maxx > kFastCoord || miny < -kFastCoord || maxy > kFastCoord) return false;
    return (maxx - minx) <= kFastExtent && (maxy - miny) <= kFastExtent;
}

// Pixels whose sample point lies in the fixed-point bbox, clipped to the
// frame; false when there are none.
__device__ __forceinline__ bool quad_pixels(const FrameDev& fr, int minx, int miny, int maxx, int maxy, int& x0,
                                            int& y0, int& x1, int& y1) {
    const int one = (1 << fr.shift) - 1;
    x0 = max((minx + one) >> fr.shift, 0);
    x1 = min(maxx >> fr.shift, fr.W - 1);
    y0 = max((miny + one) >> fr.shift, 0);
    y1 = min(maxy >> fr.shift, fr.H - 1);
    return x0 <= x1 && y0 <= y1;
}

// One triangle (a, b, c) of a quad at one sample, kernels/reyes.cl:240-265
// with the vertices taken relative to the sample (r = sample - vertex): edge
// a -> b's function (b.y - a.y) (t.x - a.x) + (a.x - b.x) (t.y - a.y) is
// rb.x ra.y - rb.y ra.x, the reference's value exactly (wrapped int32 is a
// ring), and the three functions add up to the barycentric denominator (see
// tri_setup), so a quad that covers one pixel, the usual case, needs no edge
// setup, and no reciprocal unless it covers it.
__device__ __forceinline__ bool edge_inside(int v, int ax, int ay, int bx, int by) {
    // V > C with C = -1 where Dx > 0 or (Dx == 0 and Dy > 0), else 0; Dx = ra.y - rb.y, Dy = rb.x - ra.x
    return v > ((ay > by || (ay == by && bx > ax)) ? -1 : 0);
}
__device__ __forceinline__ float tri_rcp(int va, int vb, int vc) { return frcp((float)wadd(wadd(va, vb), vc)); }
__device__ __forceinline__ float tri_depth(int va, int vb, int vc, float rdn, float da, float db, float dc) {
    // weights: edge b -> c's function for a, c -> a's for b, a -> b's for c (va, vb, vc: edges from a, b, c)
    return ffma(dc, fmul((float)va, rdn), ffma(db, fmul((float)vc, rdn), fmul(da, fmul((float)vb, rdn))));
}
// Writes a covered sample.  The reference writes only depths below the cleared
// 0x7fffffff (kernels/reyes.cl:389).
__device__ __forceinline__ void put_fragment(unsigned long long* key, float depth, unsigned mp_id) {
    const unsigned idp = idepth_of(depth);
    if (idp < 0x7fffffffu) atomicMin(key, ((unsigned long long)idp << 32) | mp_id);
}

// raster_quad_fast for boxes of many pixels: the five edges (0 -> 3 is 3 -> 0
// turned around) set up once and stepped along a row, and one reciprocal a
// triangle.  The same integers and floats at every sample.
__device__ __forceinline__ int raster_quad_wide(const FrameDev& fr, unsigned long long* keys, const int* px,
                                                const int* py, const float* qd, int4 box, unsigned mp_id) {
    const int x0 = box.x, y0 = box.y, x1 = box.z, y1 = box.w, shift = fr.shift;
    const int from[5] = {0, 1, 3, 3, 2}, to[5] = {1, 3, 0, 2, 0};
    int row[5], step[5], down[5];   // each edge's function at the row's first sample, per pixel and per row
    bool low[5];                    // accepts 0
#pragma unroll
    for (int e = 0; e < 5; ++e) {
        const int a = from[e], b = to[e], dx = wsub(py[b], py[a]), dy = wsub(px[a], px[b]);
        row[e] = wadd(wmul(dx, (x0 << shift) - px[a]), wmul(dy, (y0 << shift) - py[a]));
        step[e] = wmul(dx, 1 << shift);
        down[e] = wmul(dy, 1 << shift);
        low[e] = dx > 0 || (dx == 0 && dy > 0);
    }
    const bool low03 = !low[2] && (px[0] != px[3] || py[0] != py[3]);
    const float r1 = tri_rcp(row[0], row[1], row[2]), r2 = tri_rcp(wsub(0, row[2]), row[3], row[4]);
    int frags = 0;
    for (int y = y0; y <= y1; ++y) {
        int v[5];
#pragma unroll
        for (int e = 0; e < 5; ++e) v[e] = row[e];
        for (int x = x0; x <= x1; ++x) {
            const int v03 = wsub(0, v[2]);
            auto in = [](int value, bool zero) { return value > (zero ? -1 : 0); };
            const bool in1 = in(v[0], low[0]) && in(v[1], low[1]) && in(v[2], low[2]);
            const bool in2 = in(v03, low03) && in(v[3], low[3]) && in(v[4], low[4]);
            if (in1 || in2) {
                float depth = 1.0f;
                if (in1) {
                    const float d = tri_depth(v[0], v[1], v[2], r1, qd[0], qd[1], qd[3]);
                    if (d < depth) depth = d;
                }
                if (in2) {
                    const float d = tri_depth(v03, v[3], v[4], r2, qd[0], qd[3], qd[2]);
                    if (d < depth) depth = d;
                }
                put_fragment(keys + key_index(fr, x, y), depth, mp_id);
                ++frags;
            }
#pragma unroll
            for (int e = 0; e < 5; ++e) v[e] = wadd(v[e], step[e]);
        }
#pragma unroll
        for (int e = 0; e < 5; ++e) row[e] = wadd(row[e], down[e]);
    }
    return frags;
}

// Fast path: rasterize one quad over its own pixel bbox (see file header).
// The quad's triangles are (0, 1, 3) and (0, 3, 2).  A warp with a box of more
// than kWidePixels takes `wide` for all of its quads: its time is that of its
// largest box, and both ways one after the other would add up.  Dice+raster of
// the mixed 4,096-patch scene at 1920x1080, split limits 24, 32, 64 and 200
// (quads of some 9, 16, 64 and 625 pixels): 0.215, 0.190, 0.313 and 0.502 ms
// without it, 0.200, 0.154, 0.136 and 0.176 with it (boxes above 3 or 8:
// 0.201 and 0.205 at limit 24, 0.338 and 0.334 at 16; each lane by its own
// box: 0.232 at 24).
template <bool WIDE, typename F>
__device__ __forceinline__ int raster_quad_fast(const FrameDev& fr, unsigned long long* keys, const int* qx,
                                                const int* qy, const float* qd, int minx, int miny, int maxx,
                                                int maxy, unsigned mp_id, F&& wide) {
    int x0, y0, x1, y1;
    if (!quad_pixels(fr, minx, miny, maxx, maxy, x0, y0, x1, y1)) return 0;
    if (WIDE && __any_sync(__activemask(), (x1 - x0 + 1) * (y1 - y0 + 1) > kWidePixels)) return wide(make_int4(x0, y0, x1, y1));
    int frags = 0;
    for (int y = y0; y <= y1; ++y)
        for (int x = x0; x <= x1; ++x) {
            int rx[4], ry[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                rx[k] = (x << fr.shift) - qx[k];
                ry[k] = (y << fr.shift) - qy[k];
            }
            auto edge = [&](int a, int b) { return wsub(wmul(rx[b], ry[a]), wmul(ry[b], rx[a])); };
            auto in = [&](int v, int a, int b) { return edge_inside(v, rx[a], ry[a], rx[b], ry[b]); };
            const int v01 = edge(0, 1), v13 = edge(1, 3), v30 = edge(3, 0), v32 = edge(3, 2), v20 = edge(2, 0);
            const int v03 = wsub(0, v30);
            const bool in1 = in(v01, 0, 1) && in(v13, 1, 3) && in(v30, 3, 0);
            const bool in2 = in(v03, 0, 3) && in(v32, 3, 2) && in(v20, 2, 0);
            if (in1 || in2) {
                float depth = 1.0f;
                if (in1) {
                    const float d = tri_depth(v01, v13, v30, tri_rcp(v01, v13, v30), qd[0], qd[1], qd[3]);
                    if (d < depth) depth = d;
                }
                if (in2) {
                    const float d = tri_depth(v03, v32, v20, tri_rcp(v03, v32, v20), qd[0], qd[3], qd[2]);
                    if (d < depth) depth = d;
                }
                put_fragment(keys + key_index(fr, x, y), depth, mp_id);
                ++frags;
            }
        }
    return frags;
}

__device__ __forceinline__ void push_big(BigQuad* big, long long big_cap, unsigned long long* ctrl, const int* qx,
                                         const int* qy, const float* qd, unsigned mp_id, int view,
                                         const int* tiles) {
    unsigned long long i = atomicAdd(cw(ctrl, kBigCount), 1ull);
    if ((long long)i >= big_cap) {
        atomicAdd(cw(ctrl, kBigOverflow), 1ull);
        atomicCAS(cw(ctrl, kStatus), 0ull, (unsigned long long)kErrOverflow);
        return;
    }
    BigQuad b;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        b.px[k] = qx[k];
        b.py[k] = qy[k];
        b.depth[k] = qd[k];
        b.tile[k] = tiles[k];
    }
    b.mp_id = mp_id;
    b.view = view;
    big[i] = b;
}

// The fused kernel works on groups of NS sub-patches per block: their dice
// vertices are spread over the threads in runs of kRun of one column
// (27 runs a sub-patch at PS = 8), then the quads in strips of 8 of one
// column (8 strips a sub-patch), then one thread per quad that can touch a
// pixel.  The inputs of the next group (sub-patch records, control points,
// matrices) are copied into the other half of a double buffer with bulk
// copies, one per sub-patch, while the current group is diced and rasterized.
//
// Instruction issue and the latency of short chains bound the kernel (no
// pipe is above 40 %, DRAM at 2 %).  Runs of 3 vertices load each control
// point, matrix and column weight once for three independent chains: with one
// vertex per thread the dice issued 209 instructions a vertex.  Strips load
// two vertices a row instead of four a quad and skip the block bound.  Runs
// take 96 registers, so the shapes hold 20 warps per SM; NS is chosen so that
// both the runs and the strips of a group nearly fill whole rounds of its
// threads (14 at 128 threads: 98 % and 88 %).  Dice+raster on the mixed
// 4096-patch scene at 1920x1080: 1.72 ms (one vertex per thread, groups of 11
// in 6 blocks of 128) -> 1.42 ms; groups of 13: 1.47, of 9: 1.57, of 11 in
// 160 threads: 1.61, of 7 in 64: 1.59, of 18 in 256: 1.55, of 12 in 6 blocks
// (80 registers, spills): 1.61.  At 16x16 dicing 5.63 -> 4.56 ms (groups of
// 5; 4: 4.74, 6 in 256 threads: 4.92).  Bulk copies by the lanes of one warp
// instead of a 16-byte copy per thread and point, and the registers freed by
// 32-bit list positions and the light in shared memory (no spills):
// 1.41 -> 1.36 ms, 64 views 5.14 -> 4.90 ms.  One range test for a run's three
// projections (and displacements) instead of a branch each, so that their
// chains run side by side: 1.36 -> 1.34 ms, 4.90 -> 4.82, displaced 512x512
// heightfield at 3840x2160 3.76 -> 3.51.
constexpr int kRun = 3;
template <int NS>
constexpr int fused_threads() {
    return NS == 2 || NS == 7 ? 64 : NS == 18 ? 256 : NS == 21 ? 192 : 128;
}
// resident blocks per SM the kernels are compiled for
template <int NS>
constexpr int fused_blocks() {
    return NS == 2 || NS == 7 ? 10 : NS == 18 || NS == 21 ? 3 : 5;
}

static_assert(offsetof(DrawDev, proj) == offsetof(DrawDev, mv) + 16 * sizeof(float), "mv, proj adjacent");
static_assert(offsetof(DrawDev, mv) % 16 == 0 && sizeof(DrawDev) % 16 == 0, "16-byte copies of mv/proj");

// Inputs of one group.  Sub-patches of one draw follow each other in the
// canonical list, so a group holds few runs of equal draws: the matrices are
// staged once per run, the first kMatrixRuns runs of a group (later ones read
// them from the draw records).
constexpr int kMatrixRuns = 2;
template <int NS>
struct GroupStage {
    float4 cp[NS][20];
    float mvp[kMatrixRuns][32];   // modelview, then projection
    float4 range[NS];
    int2 meta[NS];                // (patch id, draw)
    int tv[NS][2];                // draw type, view
    int run[NS];                  // run of equal draws
};

template <int PS, int NS_>
struct FusedSmem {
    static constexpr int NS = NS_, G = PS + 1, NV = G * G;
    GroupStage<NS> st[2];
    unsigned long long full[2];   // mbarriers: the copies into st[b] have arrived
    V3 light;                     // light_dir(), here because the dice needs every register
    // per group state, double-buffered with st: blocks with a vertex at eye
    // z == 0, and the number of listed quads
    unsigned zero[2][NS];
    unsigned n_live[2];
    unsigned claimed;         // the group after the next one (raster_fused_kernel)
    unsigned short live[NS * PS * PS];   // quads that may touch a pixel
    float tx[NS][G], ty[NS][G];
    float4 vw[NS][G], cw[NS][G];
    float4 edep[NS * NV];     // eye position and NDC depth of each dice vertex
    int2 pxy[NS * NV];        // fixed-point pixel coordinates
};

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

// Starts a copy of `bytes` (a multiple of 16; both addresses 16-byte aligned)
// that completes on the mbarrier.
__device__ __forceinline__ void bulk_copy(void* smem, const void* gmem, unsigned bytes, unsigned long long* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_addr(smem)),
                 "l"(__cvta_generic_to_global(gmem)), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}
// Waits (bounded) for the mbarrier's phase; false when the wait ran out.
__device__ __forceinline__ bool bulk_wait(unsigned long long* bar, unsigned parity) {
    for (int tries = 0; tries < (1 << 20); ++tries) {
        unsigned done;
        asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
                     : "=r"(done)
                     : "r"(smem_addr(bar)), "r"(parity)
                     : "memory");
        if (done) return true;
    }
    return false;
}

// Stores the records of a group's n sub-patches, one per lane of warp 0 (its
// callers), numbers their runs of equal draws, and starts the copies of their
// control points (one per sub-patch) and of the runs' matrices.
template <int NS>
__device__ __forceinline__ void stage_inputs(GroupStage<NS>& st, unsigned long long* full, int n, float4 range, int2 meta,
                                             const DrawDev* __restrict__ draws) {
    static_assert(NS <= 32, "one record per lane of warp 0");
    const int lane = threadIdx.x;
    const int before = __shfl_up_sync(0xffffffffu, meta.y, 1);
    const bool starts = lane > 0 && lane < n && meta.y != before;
    const int run = __popc(__ballot_sync(0xffffffffu, starts) & (lanemask_lt() | (1u << lane)));
    const bool copies_matrices = lane < n && run < kMatrixRuns && (lane == 0 || starts);
    unsigned bytes = 0;
    const DrawDev* d = draws + meta.y;
    if (lane < n) {
        const int type = d->type;
        bytes = type == 0 ? 16 * sizeof(float4) : 20 * sizeof(float4);
        st.range[lane] = range;
        st.meta[lane] = meta;
        st.run[lane] = run;
        st.tv[lane][0] = type;
        st.tv[lane][1] = d->view;
    }
    const unsigned total = __reduce_add_sync(0xffffffffu, bytes + (copies_matrices ? 32 * (unsigned)sizeof(float) : 0u));
    if (lane == 0)
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(full)), "r"(total)
                     : "memory");
    __syncwarp();
    if (lane < n)
        bulk_copy(&st.cp[lane][0], reinterpret_cast<const char*>(d->cp) + (size_t)meta.x * bytes, bytes, full);
    if (copies_matrices) bulk_copy(st.mvp[run], d->mv, 32 * sizeof(float), full);
}

// Prepares the state of a group of n sub-patches whose records are in
// sm.st[b]: the dice parameters and Bernstein weights of each row / column of
// vertices, reset eye-plane flags and listed quad count.  This thread takes the items first, first + threads, ...
template <int PS, int NS>
__device__ __forceinline__ void prepare_group(FusedSmem<PS, NS>& sm, int b, int n, const FrameDev& fr, int first) {
    constexpr int G = PS + 1;
    const GroupStage<NS>& st = sm.st[b];
    for (int i = first; i < n * 2 * G; i += fused_threads<NS>()) {
        const int k = i / (2 * G), c = i % (2 * G);
        const float4 rg = st.range[k];
        if (c < G) {
            const float t = dice_param(rg.x, rg.z, c, fr);
            sm.tx[k][c] = t;
            sm.vw[k][c] = row_weights(t);
        } else {
            const float t = dice_param(rg.y, rg.w, c - G, fr);
            sm.ty[k][c - G] = t;
            sm.cw[k][c - G] = col_weights(t);
        }
    }
    if (first < n) sm.zero[b][first] = 0;
    if (first == 0) sm.n_live[b] = 0;
}

// Initializes the mbarriers and the light; ends with a barrier.
template <int PS, int NS>
__device__ __forceinline__ void init_stages(FusedSmem<PS, NS>& sm) {
    if (threadIdx.x == 0) {
        sm.light = light_dir();
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&sm.full[0])) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&sm.full[1])) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
}

// The record of list entry base + lane, for lane < n.
struct GroupRecord {
    float4 range;
    int2 meta;
};
__device__ __forceinline__ GroupRecord load_record(const SubPatches& sub, int base, int n) {
    GroupRecord g{make_float4(0.f, 0.f, 0.f, 0.f), make_int2(0, 0)};
    if ((int)threadIdx.x < n) {
        g.range = sub.range[base + threadIdx.x];
        g.meta = sub.meta[base + threadIdx.x];
    }
    return g;
}

// Stages the group [base, base + n) into sm.st[b] from scratch and prepares
// it; parity: the phase of its mbarrier.  Ends with a barrier; false when the
// copies did not arrive.
template <int PS, int NS>
__device__ __forceinline__ bool stage_group(FusedSmem<PS, NS>& sm, int b, unsigned parity, int base, int n,
                                            const SubPatches& sub, const DrawDev* __restrict__ draws,
                                            const FrameDev& fr) {
    const GroupRecord g = load_record(sub, base, n);
    if (threadIdx.x < 32) stage_inputs(sm.st[b], &sm.full[b], n, g.range, g.meta, draws);
    __syncthreads();
    prepare_group(sm, b, n, fr, threadIdx.x);
    return __syncthreads_and(bulk_wait(&sm.full[b], parity));
}

// The 8x8 block bound over front-facing quads (kernels/reyes.cl:120-166) of a
// block whose first vertex is pxy[0] (rows G apart), clamped, as its tile
// range (which may hold no tile); x < 0 when is_empty (kernels/reyes.cl:287)
// skips the block.
template <int G>
__device__ __forceinline__ int4 group_block_tiles(const int2* pxy, int W, int H, int shift, int backface) {
    FrameDev fr{};
    fr.W = W;
    fr.H = H;
    fr.shift = shift;
    fr.backface = backface;
    int x0 = (W << shift) - 1, y0 = (H << shift) - 1, x1 = 0, y1 = 0;
#pragma unroll 1
    for (int q = 0; q < 64; ++q) {
        const int2* at = pxy + (q & 7) + (q >> 3) * G;
        const int2 c0 = at[0], c1 = at[1], c2 = at[G], c3 = at[G + 1];
        const int qx[4] = {c0.x, c1.x, c2.x, c3.x}, qy[4] = {c0.y, c1.y, c2.y, c3.y};
        const QuadBound qb = quad_block_bound(fr, qx, qy);
        if (qb.ff) {
            x0 = min(x0, qb.pminx);
            y0 = min(y0, qb.pminy);
            x1 = max(x1, qb.pmaxx);
            y1 = max(y1, qb.pmaxy);
        }
    }
    int t[4];
    if (!block_tiles(fr, x0, y0, x1, y1, true, t)) return make_int4(-1, 0, 0, 0);
    return make_int4(t[0], t[1], t[2], t[3]);
}

// raster_quad_wide for a quad of the group whose first vertex is at pxy[0],
// edep[0] (rows G apart).  Out of line, and the quad read again from shared
// memory: its state, or its operands as arguments, cost the usual case
// registers.
template <int G>
static __device__ __noinline__ int raster_wide_shared(unsigned long long* keys, const int2* pxy, const float4* edep,
                                                      int shift, int kshift, int kgx, int4 box, unsigned mp_id) {
    FrameDev fr{};
    fr.shift = shift;
    fr.kshift = kshift;
    fr.kgx = kgx;
    const int at[4] = {0, 1, G, G + 1};
    int qx[4], qy[4];
    float qd[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        qx[c] = pxy[at[c]].x;
        qy[c] = pxy[at[c]].y;
        qd[c] = edep[at[c]].w;
    }
    return raster_quad_wide(fr, keys, qx, qy, qd, box, mp_id);
}

// Modelview and the perspective matrix's entries 0, 5, 10, 14 from 32 floats
// (modelview, projection; 16-byte aligned).
__device__ __forceinline__ void load_matrices(const float* m, float (&mv)[16], float (&pr)[4]) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float4 v = reinterpret_cast<const float4*>(m)[j];
        mv[4 * j] = v.x;
        mv[4 * j + 1] = v.y;
        mv[4 * j + 2] = v.z;
        mv[4 * j + 3] = v.w;
    }
    pr[0] = m[16];
    pr[1] = m[21];
    pr[2] = m[26];
    pr[3] = m[30];
}

// The vertices of run i (raster_group's numbering) for any positions: every
// NaN of a face point zeroed, the general projection where a position is not
// plain, and the blocks of a vertex on the eye plane noted.
// The dice takes a run here when one of its positions is not finite or lies
// on the eye plane, so its own loop carries none of this: dice+raster, mixed
// 4096 patches 1.23 -> 1.17 ms, at 16x16 dicing 4.04 -> 3.78, 64 views
// 4.40 -> 4.30, displaced 512x512 heightfield at 3840x2160 3.12 -> 3.03 (with
// a flag per sub-patch and a second dice after the barrier the 64 views and
// the heightfield lost 1.4 %).
template <int PS, int NS, bool DISP>
__device__ __noinline__ void dice_run_general(FusedSmem<PS, NS>& sm, int b, int i, const DrawDev* __restrict__ draws,
                                              FrameDev fr) {
    constexpr int G = PS + 1, NR = (G + kRun - 1) / kRun, RPS = G * NR, BPL = PS / 8;
    const GroupStage<NS>& cur = sm.st[b];
    const int k = i / RPS, c = i - k * RPS, nv0 = c / G * kRun, nu = c % G;
#pragma unroll 1
    for (int nv = nv0; nv < min(nv0 + kRun, G); ++nv) {
        const float ty[1] = {sm.ty[k][nv]};
        const float4 cw[1] = {sm.cw[k][nv]};
        DiceColumn<1> d;
        dice_column<1, true>(d, cur.tv[k][0], cur.cp[k], sm.tx[k][nu], ty, sm.vw[k][nu], cw);
        float mv[16], pr[4];
        load_matrices(draws[cur.meta[k].y].mv, mv, pr);
        float4 pos[1] = {mul_m44v4(mv, make_float4(d.xy[0].x, d.xy[0].y, d.zw[0].x, d.zw[0].y))};
        if (DISP) displace_vertices<1>(pos, fr.fdisp);
        int2 px[1];
        float dep[1];
        if (positions_plain<1, !DISP>(pos)) {
            project_vertices_plain<1>(pr, fr, pos, px, dep);
        } else {
            const int4 r = project_vertex_general(make_float4(pr[0], pr[1], pr[2], pr[3]), fr.W, fr.H, fr.shift, pos[0]);
            px[0] = make_int2(r.x, r.y);
            dep[0] = __int_as_float(r.z);
        }
        const int at = k * G * G + nv * G + nu;
        sm.pxy[at] = px[0];
        sm.edep[at] = make_float4(pos[0].x, pos[0].y, pos[0].z, dep[0]);
        if (pos[0].z == 0.0f) {
            // a vertex at eye z == 0 drops every 8x8 block it belongs to (kernels/reyes.cl:130-162)
            unsigned zb = 0;
            for (int bv = max(nv - 1, 0) / 8; bv <= min(nv, PS - 1) / 8; ++bv)
                for (int bu = max(nu - 1, 0) / 8; bu <= min(nu, PS - 1) / 8; ++bu) zb |= 1u << (bu + bv * BPL);
            atomicOr(&sm.zero[b][k], zb);
        }
    }
}

// Dices, shades and rasterizes the n (<= NS) sub-patches at [base, base+n)
// of the emitted list, whose inputs are staged and prepared in buffer b, with
// the whole block; meanwhile stages and prepares the n_next sub-patches at
// next_base in buffer b ^ 1, next_parity the phase of its mbarrier.  Three phases (dice; the list of quads that can
// touch a pixel; raster), each ending with a barrier; after the last one the
// next group's buffer is complete, or the result is false.  tickets, if not
// null, counts claimed groups: one is claimed into sm.claimed.
//
// The 8x8 block bound decides only whether a block is skipped, and the tiles
// of quads too large for the fast raster.  A small front-facing quad with a
// pixel centre in its bbox has that centre inside the clamped bound, and the
// bound is not empty unless every front-facing quad of the block ends at
// x = 0, so only large quads and those with maxx <= 0 look at the bound, each
// on its own (group_block_tiles); an eye-plane vertex still skips the block.
// DISP is the frame's displacement option, compiled in: frames without it
// carry neither its code nor its registers; WIDE (wide_quads) likewise.
template <int PS, int NS, bool DISP, bool WIDE>
__device__ __forceinline__ bool raster_group(FusedSmem<PS, NS>& sm, int b, int base, int n, int next_base, int n_next,
                                             unsigned next_parity, const DrawDev* __restrict__ draws, const FrameDev& fr,
                                             const SubPatches& sub, const Framebuffer& fb,
                                             float* __restrict__ mshade, BigQuad* big, long long big_cap,
                                             unsigned long long* ctrl, unsigned long long* tickets, int& frags) {
    using SM = FusedSmem<PS, NS>;
    constexpr int G = SM::G, NV = SM::NV, NQ = PS * PS, BPL = PS / 8, TH = fused_threads<NS>();
    GroupStage<NS>& cur = sm.st[b];
    GroupStage<NS>& nxt = sm.st[b ^ 1];
    const int tid = threadIdx.x, lane = tid & 31;
    // The next group's records travel in registers until this group's vertices
    // are done (8x8 dicing; staging them at once costs 0.5-1 % there: warp 0
    // waits for them); a 16x16 group has 5 and dices longer, and there
    // staging at once is 0.7 % faster.
    const GroupRecord next = load_record(sub, next_base, n_next);
    if (PS == 16 && n_next > 0 && tid < 32)
        stage_inputs(nxt, &sm.full[b ^ 1], n_next, next.range, next.meta, draws);
    // dice vertices (kernels/dice.cl:37-80): run i of a sub-patch holds the
    // vertices (nu, nv0 .. nv0 + kRun - 1), nu = i % G, nv0 = kRun (i / G)
    constexpr int NR = (G + kRun - 1) / kRun, RPS = G * NR;
    for (int i = tid; i < n * RPS; i += TH) {
        const int k = i / RPS, c = i - k * RPS, nv0 = c / G * kRun, nu = c % G;
        float4 cw[kRun];
        float ty[kRun];
#pragma unroll
        for (int v = 0; v < kRun; ++v) {
            // (a run past the last row repeats it)
            const int nv = G % kRun ? min(nv0 + v, G - 1) : nv0 + v;
            cw[v] = sm.cw[k][nv];
            ty[v] = sm.ty[k][nv];
        }
        DiceColumn<kRun> d;
        dice_column<kRun, false>(d, cur.tv[k][0], cur.cp[k], sm.tx[k][nu], ty, sm.vw[k][nu], cw);
        // the draw's modelview, and the perspective's entries 0, 5, 10, 14
        float mv[16], pr[4];
        const int run = cur.run[k];
        if (run < kMatrixRuns) {
            load_matrices(cur.mvp[run], mv, pr);
        } else {
            load_matrices(draws[cur.meta[k].y].mv, mv, pr);
        }
        float4 pos[kRun];
#pragma unroll
        for (int v = 0; v < kRun; ++v)
            pos[v] = mul_m44v4(mv, make_float4(d.xy[v].x, d.xy[v].y, d.zw[v].x, d.zw[v].y));
        if (DISP) displace_vertices<kRun>(pos, fr.fdisp);
        if (!positions_plain<kRun, !DISP>(pos)) {
            dice_run_general<PS, NS, DISP>(sm, b, i, draws, fr);
            continue;
        }
        int2 px[kRun];
        float dep[kRun];
        project_vertices_plain<kRun>(pr, fr, pos, px, dep);
        const int at = k * NV + nv0 * G + nu;
#pragma unroll
        for (int v = 0; v < kRun; ++v) {
            if (G % kRun && nv0 + v >= G) break;
            sm.pxy[at + v * G] = px[v];
            sm.edep[at + v * G] = make_float4(pos[v].x, pos[v].y, pos[v].z, dep[v]);
        }
    }
    if (PS != 16 && n_next > 0 && tid < 32)
        stage_inputs(nxt, &sm.full[b ^ 1], n_next, next.range, next.meta, draws);
    __syncthreads();
    unsigned claimed = 0;
    if (tickets && tid == 0) claimed = (unsigned)atomicAdd(tickets, 1ull);   // used after the list
    // The list of quads that can touch a pixel: a quad with a large bbox, or a
    // small one with an accepted winding and a pixel centre in its bbox.  A
    // thread walks a strip of 8 quads (column nu, rows 8 h .. 8 h + 7), so
    // each row's two vertices and their bounds serve two quads.  (Pixel
    // centres by rounding the upper bound down, and the strip's bounds every
    // second row: dice+raster, mixed 4096 patches 1.122 -> 1.114 ms, 64 views
    // 4.08 -> 4.05, displaced 512x512 heightfield at 3840x2160 2.93 -> 2.90;
    // the winding of only the quads with a pixel centre: 1.150, 4.27, 2.89.)
    constexpr int SPS = PS * BPL;   // strips of a sub-patch
    for (int i0 = tid & ~31; i0 < n * SPS; i0 += TH) {
        const int i = i0 + lane;
        unsigned live = 0;   // bit r: quad of row 8 h + r
        int first = 0;       // list entry of row 0
        if (i < n * SPS) {
            const int k = i / SPS, c = i % SPS, nu = c % PS, h = c / PS;
            first = k * NQ + nu + 8 * h * PS;
            const int2* at = sm.pxy + k * NV + nu + 8 * h * G;
            const int one = (1 << fr.shift) - 1;
            int2 a = at[0], q = at[1];
            int lx = min(a.x, q.x), hx = max(a.x, q.x), ly = min(a.y, q.y), hy = max(a.y, q.y);
            int slx = lx, shx = hx, sly = ly, shy = hy;   // the strip's bounds
            unsigned inside = 0;                          // quads with a pixel centre in their bbox, frame ignored
            unsigned wind = 0;
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const int2 c2 = at[(r + 1) * G], c3 = at[(r + 1) * G + 1];
                const int nlx = min(c2.x, c3.x), nhx = max(c2.x, c3.x), nly = min(c2.y, c3.y), nhy = max(c2.y, c3.y);
                const int minx = min(lx, nlx), maxx = max(hx, nhx), miny = min(ly, nly), maxy = max(hy, nhy);
                if ((maxx & ~one) >= minx && (maxy & ~one) >= miny) inside |= 1u << r;
                // is_front_facing (kernels/reyes.cl:54-65) on wrapped int32
                const int d1x = wsub(q.x, a.x), d1y = wsub(q.y, a.y);
                const int d2x = wsub(c2.x, a.x), d2y = wsub(c2.y, a.y);
                const int d3x = wsub(c3.x, a.x), d3y = wsub(c3.y, a.y);
                if (wsub(wmul(d1x, d3y), wmul(d3x, d1y)) < 0 || wsub(wmul(d3x, d2y), wmul(d2x, d3y)) < 0) wind |= 1u << r;
                if (r & 1) {   // two rows at once
                    slx = min(slx, minx);
                    shx = max(shx, maxx);
                    sly = min(sly, miny);
                    shy = max(shy, maxy);
                }
                lx = nlx; hx = nhx; ly = nly; hy = nhy;
                a = c2;
                q = c3;
            }
            if (slx >= 0 && sly >= 0 && shx < (fr.W << fr.shift) && shy < (fr.H << fr.shift) &&
                shx - slx <= kFastExtent && shy - sly <= kFastExtent) {
                // the strip is small and inside the frame, so every quad of it is
                live = inside & wind;
            } else {
#pragma unroll 1
                for (int r = 0; r < 8; ++r) {
                    const int2 p0 = at[r * G], p1 = at[r * G + 1], p2 = at[(r + 1) * G], p3 = at[(r + 1) * G + 1];
                    const int qx[4] = {p0.x, p1.x, p2.x, p3.x}, qy[4] = {p0.y, p1.y, p2.y, p3.y};
                    int minx, miny, maxx, maxy, x0, y0, x1, y1;
                    if (!quad_is_fast(qx, qy, minx, miny, maxx, maxy) ||
                        (((wind >> r) & 1u) && quad_pixels(fr, minx, miny, maxx, maxy, x0, y0, x1, y1)))
                        live |= 1u << r;
                }
            }
        }
        // append the strips' quads: one shared add per warp, a prefix over the lanes
        const int cnt = __popc(live);
        const int total = __reduce_add_sync(0xffffffffu, cnt);
        if (total == 0) continue;
        int pre = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, pre, o);
            if (lane >= o) pre += y;
        }
        unsigned at = 0;
        if (lane == 0) at = atomicAdd(&sm.n_live[b], (unsigned)total);
        at = __shfl_sync(0xffffffffu, at, 0) + (unsigned)(pre - cnt);
        for (unsigned m = live; m; m &= m - 1) sm.live[at++] = (unsigned short)(first + (__ffs(m) - 1) * PS);
    }
    __syncthreads();
    // the next group's weights and state, from the highest thread down (the
    // raster below occupies the lowest threads)
    prepare_group(sm, b ^ 1, n_next, fr, TH - 1 - tid);
    if (tickets && tid == 0) sm.claimed = claimed;
    // rasterize the listed quads of live blocks
    const int n_live = (int)sm.n_live[b];
    for (int j = tid; j < n_live; j += TH) {
        const int i = sm.live[j];
        const int k = i / NQ, q = i % NQ;
        const int nu = q % PS, nv = q / PS, blk = (nu >> 3) + (nv >> 3) * BPL;
        if ((sm.zero[b][k] >> blk) & 1) continue;   // an eye-plane vertex skips the block
        const int i0 = k * NV + nu + nv * G;
        const int idx[4] = {i0, i0 + 1, i0 + G, i0 + G + 1};
        int qx[4], qy[4];
        float qd[4];
        float4 e[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int2 q = sm.pxy[idx[c]];
            e[c] = sm.edep[idx[c]];
            qx[c] = q.x;
            qy[c] = q.y;
            qd[c] = e[c].w;
        }
        const unsigned mp_id = (unsigned)(base + k) * NQ + nu + nv * PS;
        const int view = cur.tv[k][1];
        unsigned long long* keys = fb.keys + (long long)view * fb.key_pixels;
        int minx, miny, maxx, maxy, f = 0;
        const bool fast = quad_is_fast(qx, qy, minx, miny, maxx, maxy);
        if (!fast || maxx <= 0) {
            const int4 t = group_block_tiles<G>(sm.pxy + k * NV + (nu & ~7) + (nv & ~7) * G, fr.W, fr.H, fr.shift,
                                                fr.backface);
            if (t.x < 0) continue;
            const int tiles[4] = {t.x, t.y, t.z, t.w};
            if (!fast) {
                // (with no tile to replay, a large quad is only counted)
                if (t.x > t.z) atomicAdd(cw(ctrl, kBigTotal), 1ull);
                else push_big(big, big_cap, ctrl, qx, qy, qd, mp_id, view, tiles);
            }
        }
        if (fast)
            f = raster_quad_fast<WIDE>(fr, keys, qx, qy, qd, minx, miny, maxx, maxy, mp_id, [&](int4 box) {
                return raster_wide_shared<G>(keys, sm.pxy + i0, sm.edep + i0, fr.shift, fr.kshift, fr.kgx, box, mp_id);
            });
        if (f > 0 || !fast) {
            // the diffuse factor of a quad that may own pixels; resolve
            // turns it into the colour of kernels/reyes.cl:191
            mshade[mp_id] = shade_m_l(sm.light, e[0].x, e[0].y, e[0].z, e[1].x, e[1].y, e[1].z, e[2].x, e[2].y, e[2].z,
                                      e[3].x, e[3].y, e[3].z);
        }
        frags += f;
    }
    return __syncthreads_and(n_next == 0 || bulk_wait(&sm.full[b ^ 1], next_parity));
}

template <int PS, int NS, bool DISP, bool WIDE>
__global__ void __launch_bounds__(fused_threads<NS>(), fused_blocks<NS>())
    raster_fused_kernel(const DrawDev* __restrict__ draws, FrameDev frp, SubPatches sub, Framebuffer fb,
                        float* __restrict__ mshade, BigQuad* big, long long big_cap, unsigned long long* ctrl) {
    using SM = FusedSmem<PS, NS>;
    FrameDev fr = frp;
    load_amplitude(fr);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SM& sm = *reinterpret_cast<SM*>(smem_raw);
    stamp_start(ctrl, 3);
    // an earlier stage of the frame failed (the host reports it): the list
    // may be incomplete, so nothing is rasterized.  The whole block decides
    // the same: blocks that already run can set the status meanwhile (the list
    // of large quads overflows), and a block without its first warp would work
    // on records that nobody staged.
    if (__syncthreads_or(*(volatile unsigned long long*)cw(ctrl, kStatus) != 0)) return;
    // (list positions fit 32 bits: micropolygon ids do)
    const int S = (int)min((long long)*(volatile unsigned long long*)cw(ctrl, kOutCount), sub.capacity);
    int frags = 0;
    // The first two groups of a block are its own, the others claimed two
    // ahead (thread 0 counts them between the dice and the raster, when its
    // warp has nothing to wait for): groups differ in their patch type, matrix
    // runs and covered quads, and with a fixed share of them the last block
    // ended some 10 % after the average one.  Dice+raster: mixed 4096 patches
    // 1.34 -> 1.23 ms, at 16x16 dicing 4.45 -> 4.04, 64 views 4.82 -> 4.40,
    // displaced 512x512 heightfield at 3840x2160 3.51 -> 3.12.
    int base = (int)blockIdx.x * NS, next = base + (int)gridDim.x * NS;
    auto count = [&](int at) { return at < S ? min(NS, S - at) : 0; };
    if (base < S) {
        init_stages(sm);
        bool ok = stage_group(sm, 0, 0, base, count(base), sub, draws, fr);
        for (unsigned it = 0; ok && base < S; ++it) {
            ok = raster_group<PS, NS, DISP, WIDE>(sm, it & 1, base, count(base), next, count(next), ((it + 1) >> 1) & 1, draws,
                                            fr, sub, fb, mshade, big, big_cap, ctrl, cw(ctrl, kGroupTicket), frags);
            base = next;
            next = (2 * (int)gridDim.x + (int)sm.claimed) * NS;
        }
        // (a copy that never arrives: the frame reports it, like every wait that runs out)
        if (!ok && threadIdx.x == 0) set_status(ctrl, kErrTimeout);
    }
    frags = __reduce_add_sync(0xffffffffu, (unsigned)frags);
    if ((threadIdx.x & 31) == 0 && frags) atomicAdd(cw(ctrl, kFragments), (unsigned long long)frags);
}

// One launch per frame: blocks [0, n_bns_ctas) first run the bound-and-split
// warp loop (each emitted slot is marked with the frame's epoch); then every
// block claims groups of NS consecutive emitted slots, waits (bounded) until
// they are marked or lie beyond the final count, and rasterizes them.  The
// grid is sized to what is resident at once, and the bound-and-split blocks
// have the lowest indices, so the blocks that wait never wait on a block that
// has not started; a wait that runs out stops consumption and reports
// MP_ERR_TIMEOUT.
// Shared memory of the frame kernel: the raster's, or what its
// bound-and-split blocks hold (draw records, samples and stacks of the warp loop).
constexpr int kFrameStagedDraws = 8;
constexpr size_t kFramePtsOffset = (kFrameStagedDraws * sizeof(DrawDev) + 15) / 16 * 16;
template <int PS, int NS>
constexpr size_t frame_smem() {
    return sizeof(FusedSmem<PS, NS>) > kFramePtsOffset + bns_smem<fused_threads<NS>(), kStackPairsFrame>()
               ? sizeof(FusedSmem<PS, NS>)
               : kFramePtsOffset + bns_smem<fused_threads<NS>(), kStackPairsFrame>();
}

template <int PS, int NS, bool WIDE>
__global__ void __launch_bounds__(fused_threads<NS>(), fused_blocks<NS>())
    frame_kernel(const DrawDev* __restrict__ gdraws, const int* __restrict__ root_prefix, int n_draws, FrameDev frp,
                 Queue q, SubPatches sub, Framebuffer fb, float* __restrict__ mshade, BigQuad* big, long long big_cap,
                 unsigned long long* ctrl, long long spin_limit, int n_bns_ctas) {
    using SM = FusedSmem<PS, NS>;
    FrameDev fr = frp;
    load_amplitude(fr);
    // bound-and-split blocks: draw records, then the warp loop's buffers
    // (frame_smem() sizes the launch for both uses)
    constexpr int kStaged = kFrameStagedDraws;
    constexpr size_t kPtsOffset = kFramePtsOffset;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ long long s_group;
    __shared__ unsigned s_claim;
    stamp_start(ctrl, 3);
    if ((int)blockIdx.x < n_bns_ctas) {
        if (threadIdx.x == 0) s_claim = bns_claim(ctrl);
        // draw constants staged in the (not yet used) raster buffer
        DrawDev* sd = reinterpret_cast<DrawDev*>(smem_raw);
        const bool staged = n_draws <= kStaged;
        if (staged) {
            const int words = n_draws * (int)(sizeof(DrawDev) / 4);
            for (int i = threadIdx.x; i < words; i += blockDim.x)
                reinterpret_cast<int*>(sd)[i] = __ldg(reinterpret_cast<const int*>(gdraws) + i);
        }
        __syncthreads();
        // the CPU criterion only: the host runs the GPU criterion as two launches
        bns_warp_loop<0, kStackPairsFrame>(
            staged ? sd : gdraws, root_prefix, n_draws, fr, q, sub, sub.seq, nullptr, ctrl, spin_limit,
            reinterpret_cast<float*>(smem_raw + kPtsOffset), s_claim, (unsigned)n_bns_ctas);
        // the rings were written by ordinary stores, and bulk copies (another
        // proxy) write the same bytes next: each thread orders its own before them
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
    }
    SM& sm = *reinterpret_cast<SM*>(smem_raw);
    const unsigned epoch = (unsigned)*(volatile unsigned long long*)cw(ctrl, kEpoch);
    int frags = 0;
    init_stages(sm);
    unsigned parity = 0;
    while (true) {
        if (threadIdx.x == 0) s_group = (long long)atomicAdd(cw(ctrl, kGroupTicket), 1ull);
        __syncthreads();
        const long long base = s_group * NS;
        int ready = 0, gave_up = 0;
        if ((int)threadIdx.x < NS) {
            const long long slot = base + threadIdx.x;
            long long idle = 0;
            unsigned ns = 32;
            while (true) {
                if (slot < sub.capacity && ld_acquire_u32(sub.seq + slot) == epoch) {
                    ready = 1;
                    break;
                }
                if (ld_acquire_u64(cw(ctrl, kDone))) {
                    // every emit's count update precedes the done flag
                    const long long fin = (long long)atomicAdd(cw(ctrl, kOutCount), 0ull);
                    if (slot >= fin || slot >= sub.capacity) break;  // beyond the end of the list
                }
                if (++idle > spin_limit) {
                    set_status(ctrl, kErrTimeout);
                    gave_up = 1;
                    break;
                }
                __nanosleep(ns);
                if (ns < 256) ns <<= 1;
            }
        }
        const int n = __syncthreads_count(ready);
        if (n == 0 || __syncthreads_or(gave_up)) break;
        bool ok = stage_group(sm, 0, parity, (int)base, n, sub, gdraws, fr);
        parity ^= 1;
        if (ok && fr.displacement)
            ok = raster_group<PS, NS, true, WIDE>(sm, 0, (int)base, n, 0, 0, 0, gdraws, fr, sub, fb, mshade, big, big_cap, ctrl,
                                            nullptr, frags);
        else if (ok)
            ok = raster_group<PS, NS, false, WIDE>(sm, 0, (int)base, n, 0, 0, 0, gdraws, fr, sub, fb, mshade, big, big_cap, ctrl,
                                             nullptr, frags);
        if (!ok) {
            if (threadIdx.x == 0) set_status(ctrl, kErrTimeout);
            break;
        }
    }
    frags = __reduce_add_sync(0xffffffffu, (unsigned)frags);
    if ((threadIdx.x & 31) == 0 && frags) atomicAdd(cw(ctrl, kFragments), (unsigned long long)frags);
}

// Exact replay of the reference's per-tile candidate loop for one quad
// (kernels/reyes.cl:333-381): the candidate set is the product of the x and y
// candidates of every tile in the block's tile range, each clamped to
// [0, 8 << shift) after subtracting the tile origin.
constexpr int kBigThreads = 256;
constexpr int kBigMaxAxis = 4096;

__global__ void __launch_bounds__(kBigThreads) raster_big_kernel(FrameDev fr, Framebuffer fb,
                                                                 const BigQuad* __restrict__ big,
                                                                 long long big_cap, unsigned long long* ctrl) {
    __shared__ short s_x[kBigMaxAxis], s_y[kBigMaxAxis];
    __shared__ int s_nx, s_ny;
    __shared__ int s_frags;
    stamp_start(ctrl, 4);
    long long n = (long long)*(volatile unsigned long long*)cw(ctrl, kBigCount);
    if (n > big_cap) n = big_cap;
    const int maxl = (8 << fr.shift) - 1;
    for (long long bi = blockIdx.x; bi < n; bi += gridDim.x) {
        const BigQuad b = big[bi];
        if (threadIdx.x == 0) {
            const int vmaxx = (fr.W << fr.shift) - 1, vmaxy = (fr.H << fr.shift) - 1;
            int mingx = vmaxx + 1, mingy = vmaxy + 1, maxgx = -1, maxgy = -1;
            for (int k = 0; k < 4; ++k) {
                mingx = min(mingx, b.px[k]);
                mingy = min(mingy, b.py[k]);
                maxgx = max(maxgx, b.px[k]);
                maxgy = max(maxgy, b.py[k]);
            }
            int nx = 0, ny = 0;
            for (int tx = b.tile[0]; tx <= b.tile[2]; ++tx) {
                int os = (tx * 8) << fr.shift;
                int lo = min(max(wsub(mingx, os), 0), maxl) >> fr.shift;
                int hi = min(max(wsub(maxgx, os), 0), maxl) >> fr.shift;
                for (int x = lo; x <= hi && nx < kBigMaxAxis; ++x) s_x[nx++] = (short)(tx * 8 + x);
            }
            for (int ty = b.tile[1]; ty <= b.tile[3]; ++ty) {
                int os = (ty * 8) << fr.shift;
                int lo = min(max(wsub(mingy, os), 0), maxl) >> fr.shift;
                int hi = min(max(wsub(maxgy, os), 0), maxl) >> fr.shift;
                for (int y = lo; y <= hi && ny < kBigMaxAxis; ++y) s_y[ny++] = (short)(ty * 8 + y);
            }
            s_nx = nx;
            s_ny = ny;
            s_frags = 0;
        }
        __syncthreads();
        Tri t1, t2;
        tri_setup(t1, b.px[0], b.py[0], b.depth[0], b.px[1], b.py[1], b.depth[1], b.px[3], b.py[3], b.depth[3]);
        tri_setup(t2, b.px[0], b.py[0], b.depth[0], b.px[3], b.py[3], b.depth[3], b.px[2], b.py[2], b.depth[2]);
        unsigned long long* keys = fb.keys + (long long)b.view * fb.key_pixels;
        long long total = (long long)s_nx * s_ny;
        int frags = 0;
        for (long long c = threadIdx.x; c < total; c += kBigThreads) {
            int x = s_x[c % s_nx], y = s_y[c / s_nx];
            int tx = wadd(x << fr.shift, 0), ty = y << fr.shift;
            float depth = 1.0f;
            bool in1 = tri_test(t1, tx, ty, depth);
            bool in2 = tri_test(t2, tx, ty, depth);
            if (in1 || in2) {
                const unsigned idp = idepth_of(depth);
                if (idp < 0x7fffffffu)
                    atomicMin(keys + key_index(fr, x, y), ((unsigned long long)idp << 32) | b.mp_id);
                ++frags;
            }
        }
        atomicAdd(&s_frags, frags);
        __syncthreads();
        if (threadIdx.x == 0 && s_frags) atomicAdd(cw(ctrl, kFragments), (unsigned long long)s_frags);
        __syncthreads();
    }
    if (blockIdx.x == 0 && threadIdx.x == 0 && n > 0) atomicAdd(cw(ctrl, kBigTotal), (unsigned long long)n);
}

__global__ void clear_kernel(Framebuffer fb, FrameDev fr, int with_color, unsigned long long* reset_ctrl,
                             long long roots, RootInfo* root_info) {
    // the frame's bound-and-split reset rides along (one thread)
    if (reset_ctrl && blockIdx.x == 0 && threadIdx.x == 0) bns_reset(reset_ctrl, roots);
    if (reset_ctrl) stamp_start(reset_ctrl, 0);
    const long long nk = fb.key_pixels * fb.views, n = fb.pixels * fb.views;
    const float4 cc = make_float4(fr.clear[0], fr.clear[1], fr.clear[2], fr.clear[3]);
    const long long stride = (long long)gridDim.x * blockDim.x;
    if (root_info)
        for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < roots; i += stride)
            reinterpret_cast<uint4*>(root_info)[i] = make_uint4(0u, 0xffffffffu, 0u, 0u);
    // the key buffer is a whole number of 32x32 tiles per view: two keys per 16-byte store
    ulonglong2* k2 = reinterpret_cast<ulonglong2*>(fb.keys);
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < nk / 2; i += stride)
        k2[i] = make_ulonglong2(kClearKey, kClearKey);
    if (with_color)
        for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
            fb.color[i] = cc;
            fb.depth[i] = 0x7fffffff;
        }
}

// Key of output pixel i (all views).
__device__ __forceinline__ unsigned long long key_of(const FrameDev& fr, const Framebuffer& fb, long long i) {
    const long long v = i / fb.pixels;
    int x, y;
    fb_pixel(fr, i - v * fb.pixels, x, y);
    return fb.keys[v * fb.key_pixels + key_index(fr, x, y)];
}

// Colour of each pixel from its winning micropolygon: the diffuse factor the
// fused kernel stored, the draw's colour (kernels/reyes.cl:191), and the
// winning depth (kernels/reyes.cl:389).  Each thread takes kResolvePixels
// pixels a grid apart and issues their key loads, then their gathers, before
// any use, so the dependent loads of several pixels are in flight at once.
// (Views go along the grid's y axis, so pixel indices are 32-bit; with one
// 64-bit index over all views, its divisions made 64 views 107 us, now 96.)
constexpr int kResolvePixels = 4;
template <int PS>
__global__ void resolve_kernel(const DrawDev* __restrict__ draws, FrameDev fr, SubPatches sub, Framebuffer fb,
                               const float* __restrict__ mshade, unsigned long long* ctrl) {
    if (blockIdx.y == 0) stamp_start(ctrl, 5);
    const unsigned n = (unsigned)fb.pixels, stride = gridDim.x * blockDim.x;
    for (int view = blockIdx.y; view < fb.views; view += gridDim.y) {
        const unsigned long long* keys = fb.keys + (long long)view * fb.key_pixels;
        float4* color = fb.color + (long long)view * fb.pixels;
        int* depth = fb.depth + (long long)view * fb.pixels;
        for (unsigned i0 = blockIdx.x * blockDim.x + threadIdx.x; i0 < n; i0 += kResolvePixels * stride) {
            unsigned long long key[kResolvePixels];
#pragma unroll
            for (int u = 0; u < kResolvePixels; ++u) {
                const unsigned i = i0 + u * stride;
                key[u] = kClearKey;
                if (i < n) {
                    const unsigned t = i >> 6, ty = t / (unsigned)fr.gx, tx = t - ty * (unsigned)fr.gx;
                    key[u] = keys[key_index(fr, (int)((tx << 3) + (i & 7)), (int)((ty << 3) + ((i >> 3) & 7)))];
                }
            }
            int draw[kResolvePixels];
            float m[kResolvePixels];
#pragma unroll
            for (int u = 0; u < kResolvePixels; ++u) {
                draw[u] = 0;
                m[u] = 0.0f;
                if (key[u] != kClearKey) {
                    const unsigned id = (unsigned)(key[u] & 0xffffffffu);
                    draw[u] = sub.meta[id / (PS * PS)].y;
                    m[u] = mshade[id];
                }
            }
#pragma unroll
            for (int u = 0; u < kResolvePixels; ++u) {
                const unsigned i = i0 + u * stride;
                if (i >= n) break;
                if (key[u] == kClearKey) {
                    color[i] = make_float4(fr.clear[0], fr.clear[1], fr.clear[2], fr.clear[3]);
                    depth[i] = 0x7fffffff;
                } else {
                    color[i] = shade_color(m[u], draws[draw[u]].color);
                    depth[i] = (int)(key[u] >> 32);
                }
            }
        }
    }
    if (threadIdx.x == 0) atomicMax(cw(ctrl, kStampEnd), global_ns());
}

// ---------------------------------------------------------------------------
// Plain per-pass kernels

template <int PS>
__global__ void dice_grid_kernel(const DrawDev* __restrict__ draws, FrameDev frp, SubPatches sub, long long base,
                                 int count, float4* pos_grid, int2* pxl_grid, float* depth_grid) {
    FrameDev fr = frp;
    load_amplitude(fr);
    constexpr int G = PS + 1, NV = G * G;
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)count * NV) return;
    int s = (int)(i / NV), v = (int)(i % NV);
    int nu = v % G, nv = v / G;
    const float4 r = sub.range[base + s];
    const int2 m = sub.meta[base + s];
    const DrawDev& d = draws[m.y];
    const float4* P = d.cp + (size_t)m.x * (d.type == 0 ? 16 : 20);
    float4 pos = dice_eye(d, fr, P, r, nu, nv);
    int px, py;
    float dep;
    project_vertex(d, fr, pos, px, py, dep);
    // grid index nu + nv*(PS+1) + range*(PS+1)^2 (kernels/dice.cl:21-24)
    pos_grid[i] = pos;
    pxl_grid[i] = make_int2(px, py);
    depth_grid[i] = dep;
}

// One 8x8 thread block per 8x8 quad block (kernels/reyes.cl:84-199).
template <int PS>
__global__ void __launch_bounds__(64) shade_grid_kernel(const DrawDev* __restrict__ draws, FrameDev fr,
                                                        SubPatches sub, long long base, const float4* pos_grid,
                                                        const int2* pxl_grid, int4* block_index,
                                                        float4* color_grid) {
    constexpr int G = PS + 1, BPL = PS / 8, BPP = BPL * BPL;
    __shared__ int s_b[4];
    __shared__ int s_allnormal;
    const int s = blockIdx.x / BPP, blk = blockIdx.x % BPP;
    const int lx = threadIdx.x & 7, ly = threadIdx.x >> 3;
    const int nu = (blk % BPL) * 8 + lx, nv = (blk / BPL) * 8 + ly;
    const int vmaxx = (fr.W << fr.shift) - 1, vmaxy = (fr.H << fr.shift) - 1;
    if (threadIdx.x == 0) {
        s_b[0] = vmaxx; s_b[1] = vmaxy; s_b[2] = 0; s_b[3] = 0;
        s_allnormal = 1;
    }
    __syncthreads();
    float4 pos[4];
    int qx[4], qy[4];
    const long long g0 = (long long)s * G * G;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        long long gi = g0 + (nu + (k & 1)) + (nv + (k >> 1)) * G;
        pos[k] = pos_grid[gi];
        int2 p = pxl_grid[gi];
        qx[k] = p.x;
        qy[k] = p.y;
        if (pos[k].z == 0.0f) s_allnormal = 0;
    }
    QuadBound qb = quad_block_bound(fr, qx, qy);
    if (qb.ff) {
        atomicMin(&s_b[0], qb.pminx);
        atomicMin(&s_b[1], qb.pminy);
        atomicMax(&s_b[2], qb.pmaxx);
        atomicMax(&s_b[3], qb.pmaxy);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int xmin = max(0, s_b[0]), ymin = max(0, s_b[1]), xmax = min(vmaxx, s_b[2]), ymax = min(vmaxy, s_b[3]);
        if (!s_allnormal) { xmin = 1; ymin = 1; xmax = -1; ymax = -1; }
        block_index[(long long)s * BPP + blk] = make_int4(xmin, ymin, xmax, ymax);
    }
    const DrawDev& d = draws[sub.meta[base + s].y];
    color_grid[(long long)s * PS * PS + nu + nv * PS] = shade_quad(pos, d.color);
}

// One thread per quad; the block bound decides the tile range (kernels/reyes.cl:270-398).
template <int PS>
__global__ void sample_grid_kernel(const DrawDev* __restrict__ draws, FrameDev fr, SubPatches sub, long long base,
                                   int count, const int4* block_index, const int2* pxl_grid,
                                   const float* depth_grid, Framebuffer fb, BigQuad* big, long long big_cap,
                                   unsigned long long* ctrl) {
    constexpr int G = PS + 1, BPL = PS / 8, BPP = BPL * BPL;
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    int frags = 0;
    if (i < (long long)count * PS * PS) {
        int s = (int)(i / (PS * PS)), q = (int)(i % (PS * PS));
        int nu = q % PS, nv = q / PS;
        int blk = (nu >> 3) + (nv >> 3) * BPL;
        int4 bb = block_index[(long long)s * BPP + blk];
        if (!(bb.x >= bb.z && bb.y >= bb.x)) {
            int tiles[4] = {bb.x >> (fr.shift + 3), bb.y >> (fr.shift + 3), bb.z >> (fr.shift + 3),
                            bb.w >> (fr.shift + 3)};
            long long g0 = (long long)s * G * G + nu + nv * G;
            const long long idx[4] = {g0, g0 + 1, g0 + G, g0 + G + 1};
            int qx[4], qy[4];
            float qd[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                int2 p = pxl_grid[idx[k]];
                qx[k] = p.x;
                qy[k] = p.y;
                qd[k] = depth_grid[idx[k]];
            }
            const int view = draws[sub.meta[base + s].y].view;
            unsigned long long* keys = fb.keys + (long long)view * fb.key_pixels;
            unsigned mp_id = (unsigned)((base + s) * PS * PS + nu + nv * PS);
            int minx, miny, maxx, maxy;
            if (quad_is_fast(qx, qy, minx, miny, maxx, maxy))
                frags = raster_quad_fast<true>(fr, keys, qx, qy, qd, minx, miny, maxx, maxy, mp_id, [&](int4 box) {
                    return raster_quad_wide(fr, keys, qx, qy, qd, box, mp_id);
                });
            else
                push_big(big, big_cap, ctrl, qx, qy, qd, mp_id, view, tiles);
        }
    }
    frags = __reduce_add_sync(0xffffffffu, (unsigned)frags);
    if ((threadIdx.x & 31) == 0 && frags) atomicAdd(cw(ctrl, kFragments), (unsigned long long)frags);
}

// Pixels won by a micropolygon of this pass take its colour from the colour grid.
__global__ void pass_resolve_kernel(FrameDev fr, Framebuffer fb, unsigned long long id_lo, unsigned long long id_hi,
                                    const float4* color_grid) {
    long long n = fb.pixels * fb.views;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const unsigned long long key = key_of(fr, fb, i);
        const unsigned long long id = key & 0xffffffffull;
        if (key != kClearKey && id >= id_lo && id < id_hi) {
            fb.color[i] = color_grid[id - id_lo];
            fb.depth[i] = (int)(key >> 32);
        }
    }
}

// Display image of one framebuffer layer, as the reference's tex_draw shader
// shows it (shaders/tex_draw.frag): untile, gamma pow(c, 0.454545) on RGB,
// then the unorm8 conversion of an 8-bit window (round(clamp(c, 0, 1) * 255)).
// Rows are written top first; the shader's gl_FragCoord.y counts from the
// bottom, so output row r is framebuffer row H - 1 - r.
__global__ void image_kernel(const float4* __restrict__ color, FrameDev fr, unsigned char* __restrict__ rgb) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)fr.W * fr.H) return;
    const int x = (int)(i % fr.W), r = (int)(i / fr.W);
    const float4 c = color[fb_index(fr, x, fr.H - 1 - r)];
    const float v[3] = {c.x, c.y, c.z};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float g = fminf(fmaxf(powf(v[k], 0.454545f), 0.0f), 1.0f);
        rgb[3 * i + k] = (unsigned char)__float2int_rn(fmul(g, 255.0f));
    }
}

// Control points from xyz triples to (x, y, z, 1).
__global__ void widen_points_kernel(const float* __restrict__ xyz, float4* __restrict__ out, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        out[i] = make_float4(xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2], 1.0f);
}

// 64-bit atomicMin throughput probe: pattern 0 = uniform random slots,
// pattern 1 = each warp updates one 8x8-pixel tile (micropolygon-like locality).
__global__ void atomic_bench_kernel(unsigned long long* buf, long long n_slots, long long n_ops, int pattern) {
    long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    long long stride = (long long)gridDim.x * blockDim.x;
    unsigned long long x = 0x9E3779B97F4A7C15ull * (unsigned long long)(tid + 1);
    for (long long i = tid; i < n_ops; i += stride) {
        x ^= x << 13; x ^= x >> 7; x ^= x << 17;
        long long slot;
        if (pattern == 0) {
            slot = (long long)(x % (unsigned long long)n_slots);
        } else {
            long long tile = (long long)((i >> 5) * 2654435761ull % (unsigned long long)(n_slots >> 6));
            slot = (tile << 6) + (long long)((i & 31) + (x & 31)) % 64;
        }
        atomicMin(buf + slot, x >> 1);
    }
}

template <typename K>
int resident_grid(K kernel, size_t smem, int threads) {
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
    if (per_sm < 1) per_sm = 1;
    return sms * per_sm;
}

// Calls f(kernel instantiation tag) for the (PS, dice_group) pair: the shape
// next to the nominal group whose threads the runs and strips fill.
template <int PS, int NS>
struct Tag {
    static constexpr int ps = PS, ns = NS;
};
template <typename F>
void dispatch_group(int PS, int group, F&& f) {
    if (PS == 16) {
        if (group == 2) f(Tag<16, 2>{});
        else if (group == 3) f(Tag<16, 3>{});
        else if (group == 4) f(Tag<16, 4>{});
        else f(Tag<16, 5>{});
    } else {
        if (group == 8) f(Tag<8, 7>{});
        else if (group == 16) f(Tag<8, 18>{});
        else if (group == 22) f(Tag<8, 21>{});
        else f(Tag<8, 14>{});
    }
}

// Whether a frame's quads are expected to cover many pixels: a sub-patch of PS
// quads a side is split while it is wider than the limit.  The wide raster pays
// from some three pixels a side, and its mere presence costs frames of smaller
// quads 0.4-1.3 % of dice+raster (64 views 4.056 -> 4.073 ms, displaced Gregory
// patches 0.215 -> 0.218); at two pixels a side (limit 16) both take 0.333 ms.
bool wide_quads(const FrameDev& fr) { return fr.limit > 2.0f * (float)fr.PS; }

// Calls f(the fused kernel of the shape T and the frame's options).
template <typename T, typename F>
void with_fused(const FrameDev& fr, F&& f) {
    if (wide_quads(fr)) {
        if (fr.displacement)
            f(raster_fused_kernel<T::ps, T::ns, true, true>);
        else
            f(raster_fused_kernel<T::ps, T::ns, false, true>);
    } else {
        if (fr.displacement)
            f(raster_fused_kernel<T::ps, T::ns, true, false>);
        else
            f(raster_fused_kernel<T::ps, T::ns, false, false>);
    }
}

int grid_for(long long n, int block) {
    long long g = (n + block - 1) / block;
    if (g < 1) g = 1;
    if (g > 1 << 20) g = 1 << 20;
    return (int)g;
}

}  // namespace

// ---------------------------------------------------------------------------
// launchers

void launch_clear(const Framebuffer& fb, const FrameDev& fr, int with_color, cudaStream_t s,
                  unsigned long long* reset_ctrl, long long roots, RootInfo* root_info) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const long long want = with_color ? fb.pixels * fb.views : fb.key_pixels * fb.views / 2;
    clear_kernel<<<(int)std::min<long long>(grid_for(want, 256), (long long)sms * 8), 256, 0, s>>>(
        fb, fr, with_color, reset_ctrl, roots, root_info);
}

int raster_fused_grid(const FrameDev& fr, int group) {
    int g = 0;
    dispatch_group(fr.PS, group, [&](auto t) {
        using T = decltype(t);
        auto fit = [&](auto kernel) {
            g = resident_grid(kernel, sizeof(FusedSmem<T::ps, T::ns>), fused_threads<T::ns>());
        };
        with_fused<T>(fr, fit);
    });
    return g;
}

void launch_raster_fused(const DrawDev* draws, const FrameDev& fr, const SubPatches& sub, const Framebuffer& fb,
                         float* mshade, BigQuad* big, long long big_cap, unsigned long long* ctrl, int grid, int group,
                         cudaStream_t s) {
    dispatch_group(fr.PS, group, [&](auto t) {
        using T = decltype(t);
        auto launch = [&](auto kernel) {
            kernel<<<grid, fused_threads<T::ns>(), sizeof(FusedSmem<T::ps, T::ns>), s>>>(draws, fr, sub, fb, mshade, big,
                                                                                        big_cap, ctrl);
        };
        with_fused<T>(fr, launch);
    });
}

int frame_kernel_grid(const FrameDev& fr, int group) {
    int g = 0;
    dispatch_group(fr.PS, group, [&](auto t) {
        using T = decltype(t);
        auto fit = [&](auto kernel) {
            g = resident_grid(kernel, frame_smem<T::ps, T::ns>(), fused_threads<T::ns>());
        };
        if (wide_quads(fr))
            fit(frame_kernel<T::ps, T::ns, true>);
        else
            fit(frame_kernel<T::ps, T::ns, false>);
    });
    return g;
}

void launch_frame_kernel(const DrawDev* draws, const int* root_prefix, int n_draws, const FrameDev& fr, const Queue& q,
                         const SubPatches& sub, const Framebuffer& fb, float* mshade, BigQuad* big, long long big_cap,
                         unsigned long long* ctrl, long long spin_limit, int grid, int n_bns_ctas, int group,
                         cudaStream_t s) {
    dispatch_group(fr.PS, group, [&](auto t) {
        using T = decltype(t);
        auto launch = [&](auto kernel) {
            kernel<<<grid, fused_threads<T::ns>(), frame_smem<T::ps, T::ns>(), s>>>(
                draws, root_prefix, n_draws, fr, q, sub, fb, mshade, big, big_cap, ctrl, spin_limit, n_bns_ctas);
        };
        if (wide_quads(fr))
            launch(frame_kernel<T::ps, T::ns, true>);
        else
            launch(frame_kernel<T::ps, T::ns, false>);
    });
}

void launch_raster_big(const DrawDev*, const FrameDev& fr, const Framebuffer& fb, const BigQuad* big,
                       long long big_cap, unsigned long long* ctrl, cudaStream_t s) {
    raster_big_kernel<<<256, kBigThreads, 0, s>>>(fr, fb, big, big_cap, ctrl);
}

void launch_resolve(const DrawDev* draws, const FrameDev& fr, const SubPatches& sub, const Framebuffer& fb,
                    const float* mshade, unsigned long long* ctrl, cudaStream_t s) {
    const dim3 g((unsigned)grid_for((fb.pixels + kResolvePixels - 1) / kResolvePixels, 256),
                 (unsigned)std::min(fb.views, 65535));
    if (fr.PS == 16)
        resolve_kernel<16><<<g, 256, 0, s>>>(draws, fr, sub, fb, mshade, ctrl);
    else
        resolve_kernel<8><<<g, 256, 0, s>>>(draws, fr, sub, fb, mshade, ctrl);
}

void launch_dice_grid(const DrawDev* draws, const FrameDev& fr, const SubPatches& sub, long long base, int count,
                      float4* pos, int2* pxl, float* depth, cudaStream_t s) {
    if (count <= 0) return;
    long long n = (long long)count * (fr.PS + 1) * (fr.PS + 1);
    if (fr.PS == 16)
        dice_grid_kernel<16><<<grid_for(n, 128), 128, 0, s>>>(draws, fr, sub, base, count, pos, pxl, depth);
    else
        dice_grid_kernel<8><<<grid_for(n, 128), 128, 0, s>>>(draws, fr, sub, base, count, pos, pxl, depth);
}

void launch_shade_grid(const DrawDev* draws, const FrameDev& fr, const SubPatches& sub, long long base, int count,
                       const float4* pos, const int2* pxl, int4* block_index, float4* color, cudaStream_t s) {
    if (count <= 0) return;
    int bpp = (fr.PS / 8) * (fr.PS / 8);
    if (fr.PS == 16)
        shade_grid_kernel<16><<<count * bpp, 64, 0, s>>>(draws, fr, sub, base, pos, pxl, block_index, color);
    else
        shade_grid_kernel<8><<<count * bpp, 64, 0, s>>>(draws, fr, sub, base, pos, pxl, block_index, color);
}

void launch_sample_grid(const DrawDev* draws, const FrameDev& fr, const SubPatches& sub, long long base, int count,
                        const int4* block_index, const int2* pxl, const float* depth, const Framebuffer& fb,
                        BigQuad* big, long long big_cap, unsigned long long* ctrl, cudaStream_t s) {
    if (count <= 0) return;
    long long n = (long long)count * fr.PS * fr.PS;
    if (fr.PS == 16)
        sample_grid_kernel<16><<<grid_for(n, 128), 128, 0, s>>>(draws, fr, sub, base, count, block_index, pxl, depth,
                                                                fb, big, big_cap, ctrl);
    else
        sample_grid_kernel<8><<<grid_for(n, 128), 128, 0, s>>>(draws, fr, sub, base, count, block_index, pxl, depth,
                                                               fb, big, big_cap, ctrl);
}

void launch_pass_resolve(const FrameDev& fr, const Framebuffer& fb, long long base, int count, const float4* color,
                         cudaStream_t s) {
    if (count <= 0) return;
    unsigned long long lo = (unsigned long long)base * fr.PS * fr.PS;
    unsigned long long hi = lo + (unsigned long long)count * fr.PS * fr.PS;
    pass_resolve_kernel<<<grid_for(fb.pixels * fb.views, 256), 256, 0, s>>>(fr, fb, lo, hi, color);
}

void launch_dice_debug(const DrawDev* draws, const FrameDev& fr, const SubPatches& sub, int count, float4* pos,
                       int2* pxl, float* depth, cudaStream_t s) {
    launch_dice_grid(draws, fr, sub, 0, count, pos, pxl, depth, s);
}

void launch_widen_points(const float* xyz, float4* out, long long n, cudaStream_t s) {
    if (n > 0) widen_points_kernel<<<grid_for(n, 256), 256, 0, s>>>(xyz, out, n);
}

void launch_image(const float4* color, const FrameDev& fr, unsigned char* rgb, cudaStream_t s) {
    const long long n = (long long)fr.W * fr.H;
    image_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(color, fr, rgb);
}

void launch_atomic_bench(unsigned long long* buf, long long n_slots, long long n_ops, int pattern, cudaStream_t s) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    atomic_bench_kernel<<<sms * 8, 256, 0, s>>>(buf, n_slots, n_ops, pattern);
}

}  // namespace mp
