// Adjoint of the image with respect to control points and the displacement
// amplitude, with visibility held fixed (the winning micropolygon of every
// pixel comes from the forward pass's depth|id buffer).
//
// One thread per pixel.  The winning quad's four dice vertices are
// recomputed (Bernstein weights, modelview, displacement of
// kernels/dice.cl:51-67) instead of being stored, the flat colour of
// kernels/reyes.cl:172-191 is differentiated back to the four eye
// positions, through the displacement steps in reverse, through the
// modelview, and onto the 16 (Bezier) or 20 (Gregory) control points with
// their Bernstein / face-blend weights.  A warp puts its lanes' 48 (or 60)
// partial gradients into shared memory and adds them up patch by patch, a
// lane per control-point coordinate, so that each patch of the warp gets one
// set of atomics on consecutive addresses.
//
// What is left is the arithmetic's latency at 16 warps per SM (127 registers).
// Before, lanes whose warp saw several patches added their own 48 values to
// scattered addresses (a sector of L2 each), every vertex loaded the patch's
// points again, and the weights of every control point and vertex sat in a
// local array (158 registers, 12 warps).  backward() calls: 512x512-patch
// heightfield at 3840x2160 1.69 -> 0.65 ms, 777 Gregory patches at 1280x720
// 0.62 -> 0.13 ms, 16x16 heightfield at 512x512 0.155 -> 0.12 ms.
#include "mp_internal.h"

namespace mp {

namespace {

constexpr int kAdjBlock = 128;
constexpr int kAdjStride = 61;   // values of a lane in shared memory, odd against bank conflicts

__device__ __forceinline__ void bern4(float t, float (&b)[4]) {
    const float s = 1.0f - t;
    b[0] = s * s * s;
    b[1] = 3.0f * s * s * t;
    b[2] = 3.0f * s * t * t;
    b[3] = t * t * t;
}

__device__ __forceinline__ V3 axpy(float a, V3 x, V3 y) { return V3{ffma(a, x.x, y.x), ffma(a, x.y, y.y), ffma(a, x.z, y.z)}; }
__device__ __forceinline__ V3 scale(float a, V3 x) { return V3{fmul(a, x.x), fmul(a, x.y), fmul(a, x.z)}; }

// 1 / (a + b) of a face blend, 0 where the blend is 0 / 0 (its weight is 0 there)
__device__ __forceinline__ float face_rcp(float den) { return den == 0.0f ? 0.0f : frcp(den); }

// Gradients of the eye position of one vertex before displacement, from
// those after it (g), and the amplitude's (added to gamp); pos is the
// position before displacement.
__device__ __forceinline__ V3 displace_adjoint(float4 pos, const FrameDev& fr, V3 g, float& gamp) {
    const float K[3] = {10.0f, 14.0f, 22.0f}, B[3] = {0.04f, 0.02f, 0.01f};
    const bool small = displace_is_small(pos, fr.fdisp);
    // two arguments at a time, as in displace_vertices: those of one x, and of one y
    auto sines = [&](float a, float b) { return small ? sin2_small(a, b) : make_float2(mp_sinf(a), mp_sinf(b)); };
    auto cosines = [&](float a, float b) { return small ? cos2_small(a, b) : make_float2(mp_cosf(a), mp_cosf(b)); };
    auto both = [&](float a) {
        return small ? make_float2(sin_small(a), cos_small(a)) : make_float2(mp_sinf(a), mp_cosf(a));
    };
    float2 sy0[3], sx1[3], s6[3], sy1[3];   // sine, cosine
    float x = pos.x, y = pos.y;
    sy0[0] = both(fmul(K[0], y));
#pragma unroll
    for (int st = 0; st < 3; ++st) {
        x = ffma(sy0[st].x, fr.fdisp[st], x);
        const float a = fmul(K[st], x), b = fmul(6.0f, x);
        const float2 s = sines(a, b), c = cosines(a, b);
        sx1[st] = make_float2(s.x, c.x);
        s6[st] = make_float2(s.y, c.y);
        y = ffma(sx1[st].x, fr.fdisp[st], y);
        const float d = fmul(K[st], y);
        if (st < 2) {
            const float e = fmul(K[st < 2 ? st + 1 : 2], y);
            const float2 t = sines(d, e), u = cosines(d, e);
            sy1[st] = make_float2(t.x, u.x);
            sy0[st + 1] = make_float2(t.y, u.y);
        } else {
            sy1[st] = both(d);
        }
    }
#pragma unroll
    for (int st = 2; st >= 0; --st) {
        const float F = fr.fdisp[st];
        gamp += g.z * sy1[st].x * s6[st].x * B[st];
        g.y += g.z * F * K[st] * sy1[st].y * s6[st].x;
        g.x += g.z * F * sy1[st].x * 6.0f * s6[st].y;
        gamp += g.y * sx1[st].x * B[st];
        g.x += g.y * F * K[st] * sx1[st].y;
        gamp += g.x * sy0[st].x * B[st];
        g.y += g.x * F * K[st] * sy0[st].y;
    }
    return g;
}

// The sum of one value of each lane (kAdjStride apart) of a warp that sees one
// patch, in pairs: one after the other the rounding of 32 values is 1.7 times
// as large, and a small value beside a large partial sum is lost.  (Patches
// that share a warp have few lanes each, and each lane's value was an atomic
// before; their sums stay one after the other.  Pairs for those too made
// backward() on the displaced 512x512 heightfield at 3840x2160 4 % slower.)
__device__ __forceinline__ float sum_lanes(const float* v) {
    float block[4];
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        float x[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = v[(8 * b + j) * kAdjStride];
        block[b] = ((x[0] + x[1]) + (x[2] + x[3])) + ((x[4] + x[5]) + (x[6] + x[7]));
    }
    return (block[0] + block[1]) + (block[2] + block[3]);
}

__global__ void __launch_bounds__(kAdjBlock, 4) adjoint_kernel(const DrawDev* __restrict__ draws, FrameDev frp,
                                                               SubPatches sub, Framebuffer fb,
                                                               const float4* __restrict__ grad_color, float* grad_amp,
                                                               int view) {
    __shared__ float s_values[kAdjBlock * kAdjStride];
    FrameDev fr = frp;
    load_amplitude(fr);
    const int PS = fr.PS;
    const int lane = threadIdx.x & 31;
    float* values = s_values + (threadIdx.x & ~31) * kAdjStride;   // of this warp
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    bool active = false;
    int pid = -1, draw = -1, nu = 0, nv = 0;
    float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < fb.pixels) {
        int px, py;
        fb_pixel(fr, i, px, py);
        const unsigned long long key = fb.keys[(long long)view * fb.key_pixels + key_index(fr, px, py)];
        if (key != kClearKey) {
            const unsigned id = (unsigned)(key & 0xffffffffu);
            const unsigned s = id / (unsigned)(PS * PS), q = id % (unsigned)(PS * PS);
            nu = (int)(q % PS);
            nv = (int)(q / PS);
            const int2 m = sub.meta[s];
            r = sub.range[s];
            pid = m.x;
            draw = m.y;
            active = draws[draw].grad_cp != nullptr;
        }
    }
    const unsigned covered = __ballot_sync(0xffffffffu, active);
    if (covered == 0) return;
    const DrawDev& d = draws[active ? draw : 0];
    const int ncp = d.type == 0 ? 16 : 20;
    float gamp = 0.0f;
    if (active) {
        const float4* P = d.cp + (size_t)pid * ncp;
        // the quad's vertices k = a + 2 b: columns a at tu[a], rows b at tv[b]
        const float tu[2] = {dice_param(r.x, r.z, nu, fr), dice_param(r.x, r.z, nu + 1, fr)};
        const float tv[2] = {dice_param(r.y, r.w, nv, fr), dice_param(r.y, r.w, nv + 1, fr)};
        float bx[2][4], by[2][4];
        bern4(tu[0], bx[0]);
        bern4(tu[1], bx[1]);
        bern4(tv[0], by[0]);
        bern4(tv[1], by[1]);
        float4 eye[4];   // before displacement
        V3 pos[4];       // after it
        {
            // the dicer's operations in its order: the quad's sides are small
            // differences of these positions, so their roundings show in the normal
            float2 oxy[4], ozw[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) oxy[k] = ozw[k] = make_float2(0.f, 0.f);
            const float4 rw[2] = {row_weights(tu[0]), row_weights(tu[1])}, cw[2] = {col_weights(tv[0]), col_weights(tv[1])};
            auto elem = [](const float4& v, int j) { return j == 0 ? v.x : j == 1 ? v.y : j == 2 ? v.z : v.w; };
            auto add = [&](int k, int e, int j, float4 c) {
                const float2 w = fmul2(dup2(elem(rw[k & 1], e)), dup2(elem(cw[k >> 1], j)));
                oxy[k] = ffma2(w, make_float2(c.x, c.y), oxy[k]);
                ozw[k] = ffma2(w, make_float2(c.z, c.w), ozw[k]);
            };
            if (d.type == 0) {
#pragma unroll
                for (int e = 0; e < 4; ++e)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float4 c = __ldg(P + 4 * e + j);
#pragma unroll
                        for (int k = 0; k < 4; ++k) add(k, e, j, c);
                    }
            } else {
                // kernels/utility.h:155-206: rows 1 and 2 hold two face points each
                const int row[4][4] = {{0, 4, 9, 1}, {8, -1, -1, 5}, {7, -1, -1, 10}, {3, 11, 6, 2}};
#pragma unroll
                for (int e = 0; e < 4; ++e)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        if (row[e][j] >= 0) {
                            const float4 c = __ldg(P + row[e][j]);
#pragma unroll
                            for (int k = 0; k < 4; ++k) add(k, e, j, c);
                            continue;
                        }
                        const float4 A = __ldg(P + (e == 1 ? (j == 1 ? 12 : 17) : (j == 1 ? 19 : 14)));
                        const float4 B = __ldg(P + (e == 1 ? (j == 1 ? 16 : 13) : (j == 1 ? 15 : 18)));
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const float u = tu[k & 1], v = tv[k >> 1];
                            const float a = j == 1 ? u : fsub(1.0f, u), b = e == 1 ? v : fsub(1.0f, v);
                            const float den = e == 1 ? (j == 1 ? fadd(u, v) : fadd(fsub(1.0f, u), v))
                                                     : (j == 1 ? fsub(fadd(1.0f, u), v) : fsub(fsub(2.0f, u), v));
                            add(k, e, j, blend4(a, A, b, B, den));
                        }
                    }
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                eye[k] = mul_m44v4(d.mv, make_float4(oxy[k].x, oxy[k].y, ozw[k].x, ozw[k].y));
                const float4 p = fr.displacement ? displace(eye[k], fr.fdisp) : eye[k];
                pos[k] = V3{p.x, p.y, p.z};
            }
        }
        // shade forward
        V3 du{0.5f * (((pos[1].x - pos[0].x) + pos[3].x) - pos[2].x),
              0.5f * (((pos[1].y - pos[0].y) + pos[3].y) - pos[2].y),
              0.5f * (((pos[1].z - pos[0].z) + pos[3].z) - pos[2].z)};
        V3 dv{0.5f * (((pos[2].x - pos[0].x) + pos[3].x) - pos[1].x),
              0.5f * (((pos[2].y - pos[0].y) + pos[3].y) - pos[1].y),
              0.5f * (((pos[2].z - pos[0].z) + pos[3].z) - pos[1].z)};
        V3 cr{dv.y * du.z - dv.z * du.y, dv.z * du.x - dv.x * du.z, dv.x * du.y - dv.y * du.x};
        const float len = sqrtf(cr.x * cr.x + cr.y * cr.y + cr.z * cr.z);
        const V3 n{cr.x / len, cr.y / len, cr.z / len};
        const float ln = sqrtf(89.0f);
        const V3 L{4.0f / ln, 3.0f / ln, 8.0f / ln};
        const float nl = n.x * L.x + n.y * L.y + n.z * L.z;
        const float4 gc = grad_color[(long long)view * fb.pixels + i];
        const float gm = gc.x * d.color[0] + gc.y * d.color[1] + gc.z * d.color[2] + gc.w * d.color[3];
        V3 go[4];   // object-space gradient of each vertex
        if (nl > 0.0f && len > 0.0f && isfinite(len)) {
            const V3 gcr{gm * (L.x - n.x * nl) / len, gm * (L.y - n.y * nl) / len, gm * (L.z - n.z * nl) / len};
            const V3 gdv{du.y * gcr.z - du.z * gcr.y, du.z * gcr.x - du.x * gcr.z, du.x * gcr.y - du.y * gcr.x};
            const V3 gdu{gcr.y * dv.z - gcr.z * dv.y, gcr.z * dv.x - gcr.x * dv.z, gcr.x * dv.y - gcr.y * dv.x};
            float sdu[4] = {-0.5f, 0.5f, -0.5f, 0.5f}, sdv[4] = {-0.5f, -0.5f, 0.5f, 0.5f};
            // one vertex per round (the displacement's adjoint is long): the
            // arrays turn by one so that every index is a constant
#pragma unroll 1
            for (int k = 0; k < 4; ++k) {
                V3 g{sdu[0] * gdu.x + sdv[0] * gdv.x, sdu[0] * gdu.y + sdv[0] * gdv.y, sdu[0] * gdu.z + sdv[0] * gdv.z};
                if (fr.displacement) g = displace_adjoint(eye[0], fr, g, gamp);
                const float* mm = d.mv;
                const V3 t{mm[0] * g.x + mm[1] * g.y + mm[2] * g.z, mm[4] * g.x + mm[5] * g.y + mm[6] * g.z,
                           mm[8] * g.x + mm[9] * g.y + mm[10] * g.z};
                const float4 e0 = eye[0];
                const float u0 = sdu[0], v0 = sdv[0];
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    eye[j] = eye[j + 1];
                    sdu[j] = sdu[j + 1];
                    sdv[j] = sdv[j + 1];
                    go[j] = go[j + 1];
                }
                eye[3] = e0;
                sdu[3] = u0;
                sdv[3] = v0;
                go[3] = t;
            }
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) go[k] = V3{0.0f, 0.0f, 0.0f};
        }
        // control-point gradients: sum_k w_j(vertex k) * go(vertex k)
        float* mine = values + lane * kAdjStride;
        auto put = [&](int j, V3 v) {
            mine[3 * j] = v.x;
            mine[3 * j + 1] = v.y;
            mine[3 * j + 2] = v.z;
        };
        const int slot[16] = {0, 4, 9, 1, 8, -1, -1, 5, 7, -1, -1, 10, 3, 11, 6, 2};   // Gregory's corner and edge points
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const V3 h0 = axpy(by[0][j], go[0], scale(by[1][j], go[2])), h1 = axpy(by[0][j], go[1], scale(by[1][j], go[3]));
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const V3 v = axpy(bx[0][e], h0, scale(bx[1][e], h1));
                if (d.type == 0) put(4 * e + j, v);
                else if (slot[4 * e + j] >= 0) put(slot[4 * e + j], v);
            }
        }
        if (d.type != 0) {
            // the face points' pairs: e the row, j the column of the face
#pragma unroll
            for (int f = 0; f < 4; ++f) {
                const int e = 1 + (f >> 1), j = 1 + (f & 1);
                V3 ga{0.f, 0.f, 0.f}, gb{0.f, 0.f, 0.f};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float a = j == 1 ? tu[k & 1] : 1.0f - tu[k & 1], b = e == 1 ? tv[k >> 1] : 1.0f - tv[k >> 1];
                    const float w = bx[k & 1][e] * by[k >> 1][j] * face_rcp(a + b);
                    ga = axpy(w * a, go[k], ga);
                    gb = axpy(w * b, go[k], gb);
                }
                // F0 (12, 16), F1 (17, 13), F3 (19, 15), F2 (14, 18)
                put(f == 0 ? 12 : f == 1 ? 17 : f == 2 ? 19 : 14, ga);
                put(f == 0 ? 16 : f == 1 ? 13 : f == 2 ? 15 : 18, gb);
            }
        }
    }
    // amplitude gradient: one atomic per warp
    if (grad_amp && fr.displacement) {
        float ga = __shfl_xor_sync(0xffffffffu, gamp, 16) + gamp;
        ga += __shfl_xor_sync(0xffffffffu, ga, 8);
        ga += __shfl_xor_sync(0xffffffffu, ga, 4);
        ga += __shfl_xor_sync(0xffffffffu, ga, 2);
        ga += __shfl_xor_sync(0xffffffffu, ga, 1);
        if (lane == 0 && ga != 0.0f) atomicAdd(grad_amp, ga);
    }
    // control-point gradients, patch by patch: lane l adds up coordinates l and l + 32 of the patch's lanes
    const unsigned long long patch = active ? ((unsigned long long)draw << 32) | (unsigned)pid : ~0ull;
    const unsigned peers = __match_any_sync(0xffffffffu, patch);
    float* target = active ? d.grad_cp + (size_t)pid * ncp * 3 : nullptr;
    __syncwarp();
    for (unsigned todo = covered; todo;) {
        const int leader = __ffs(todo) - 1;
        unsigned group = __shfl_sync(0xffffffffu, peers, leader);
        todo &= ~group;
        float* g = reinterpret_cast<float*>(
            __shfl_sync(0xffffffffu, (unsigned long long)reinterpret_cast<size_t>(target), leader));
        const bool high = lane + 32 < 3 * __shfl_sync(0xffffffffu, ncp, leader);
        float s0 = 0.0f, s1 = 0.0f;
        if (group == 0xffffffffu) {
            s0 = sum_lanes(values + lane);
            if (high) s1 = sum_lanes(values + lane + 32);
        } else {
            while (group) {
                const float* v = values + (__ffs(group) - 1) * kAdjStride + lane;
                group &= group - 1;
                s0 += v[0];
                if (high) s1 += v[32];
            }
        }
        if (s0 != 0.0f) atomicAdd(g + lane, s0);
        if (high && s1 != 0.0f) atomicAdd(g + lane + 32, s1);
    }
}

}  // namespace

void launch_adjoint(const DrawDev* draws, const FrameDev& fr, const SubPatches& sub, const Framebuffer& fb,
                    const float4* grad_color, float* grad_amp, int view, cudaStream_t s) {
    long long n = fb.pixels;
    adjoint_kernel<<<(unsigned)((n + kAdjBlock - 1) / kAdjBlock), kAdjBlock, 0, s>>>(draws, fr, sub, fb, grad_color,
                                                                                    grad_amp, view);
}

}  // namespace mp
