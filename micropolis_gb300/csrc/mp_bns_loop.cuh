// The bound-and-split warp loop, shared by the standalone persistent kernel
// (mp_bns.cu) and the frame kernel that overlaps it with rasterization
// (mp_raster.cu).  See mp_bns.cu for the queue protocol.
#pragma once
#include "mp_internal.h"

namespace mp {

__device__ __forceinline__ unsigned long long* cw(unsigned long long* ctrl, int w) { return ctrl + w * kCtrlStride; }

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ unsigned long long ld_relaxed_u64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed_u64(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ void st_release_u32(unsigned* p, unsigned v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_u64(unsigned long long* p, unsigned long long v) {
    asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned lanemask_lt() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// Stage k of a batched frame starts: its kernel's first block notes the time.
// (An event between every two kernels of the frame's graph cost 28 us a
// frame, 19 % of the 8x8 heightfield's; the timer ticks every 32 ns.)
__device__ __forceinline__ void stamp_start(unsigned long long* ctrl, int k) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *cw(ctrl, kStamp + k) = global_ns();
}

// The per-frame reset of the bound-and-split control words: every root
// outstanding, counters cleared, the frame epoch advanced.
__device__ __forceinline__ void bns_reset(unsigned long long* ctrl, long long roots) {
    *cw(ctrl, kQTail) = handover_start((unsigned long long)roots);
    *cw(ctrl, kQHead) = 0;
    *cw(ctrl, kClaims) = 0;
    *cw(ctrl, kRootHead) = 0;
    *cw(ctrl, kSplits) = 0;
    *cw(ctrl, kGiven) = 0;
    *cw(ctrl, kOutCount) = 0;
    *cw(ctrl, kDone) = roots == 0 ? 1 : 0;
    *cw(ctrl, kStatus) = 0;
    *cw(ctrl, kEpoch) = *cw(ctrl, kEpoch) + 1;
    *cw(ctrl, kRoots) = (unsigned long long)roots;
    *cw(ctrl, kBigCount) = 0;
    *cw(ctrl, kFragments) = 0;
    *cw(ctrl, kBigOverflow) = 0;
    *cw(ctrl, kGroupTicket) = 0;
    *cw(ctrl, kMaxDepth) = 0;
    *cw(ctrl, kSortDone) = 0;
    *cw(ctrl, kSortMost) = 0;
    *cw(ctrl, kStampEnd) = 0;
}

// This block's claim, by its first thread: the number of claims before it.
__device__ __forceinline__ unsigned bns_claim(unsigned long long* ctrl) {
    return (unsigned)atomicAdd(cw(ctrl, kClaims), 1ull);
}

__device__ __forceinline__ void set_status(unsigned long long* ctrl, int code) {
    atomicCAS(cw(ctrl, kStatus), 0ull, (unsigned long long)code);
}

// A warp's stack of pairs (the two children of a split) in shared memory: a
// ring of C pairs and, beside it, a column of scratch for each lane's range;
// word w of ring slot i at s[w * stack_stride<C>() + i], of lane l's scratch
// at s[w * stack_stride<C>() + C + l].
//   words 0-26   the parent's nine bound samples (spi() order), CPU criterion
//   words 27-30  the parent's range
//   word 31      patch id | split direction << 31 (1: x halved), GPU criterion
//   word 32      draw | parent's depth << 24
//   word 33      the parent's split path
// Bundles of the global queue hold up to kBundlePairs pairs with the same
// words, word w of pair p at kBundlePairs * w + p, and the number of pairs in
// the last one.  Every word carries the frame's epoch in its upper half, so a
// reader knows each word valid by itself and neither side needs a fence: a
// gpu-scope acquire empties the SM's L1 of the patches its other warps work
// on and made the receiver's next loads wait some 5,000 cycles.  The count of
// unfinished units needs none either (mp_handover.h).
constexpr int kPairWords = 34;
constexpr int kStackPairs = 64;        // ring size of the standalone kernel
constexpr int kStackPairsFrame = 32;   // and of the overlapped kernel, whose blocks also hold the raster's buffers
// an odd stride: lanes on neighbouring words of one column use different banks
template <int C>
constexpr int stack_stride() {
    return C + 33;
}

// Shared memory of the warp loop in a block of `threads`.
template <int THREADS, int C>
constexpr size_t bns_smem() {
    return (THREADS / 32) * kPairWords * stack_stride<C>() * sizeof(float);
}

// Runs one warp's share of a frame's bound-and-split until the done flag is
// raised.  Emitted sub-patches go to `out`; when out_seq is given, each
// emitted slot is also marked with the frame's epoch (release) for consumers
// that run concurrently; when roots is given, each root's record counts its
// sub-patches and bounds their paths (for the canonical sort).  CRIT selects
// the bound criterion (bns_decide).
// `blocks` blocks run the loop; `claim` is this one's number in the order in
// which they started (bns_claim).
//
// Roots are dealt in shares: share s to warp s / blocks of the block with claim
// s % blocks, the rest with atomics.  A warp that has waited a microsecond takes
// the claims of blocks that have not started, so every root that nobody works
// on yet can be taken by any warp that runs, and a warp waits only for warps
// that hold work: the launch ends whatever part of its blocks the device holds
// at once.  (Against shares and tickets dealt by block number without atomics:
// 64 views 0.91 -> 0.83 ms, the displaced 512x512 heightfield at 3840x2160
// 0.443 -> 0.410, 24 objects 0.124 -> 0.126, the 8x8 heightfield 0.045 as before.)
//
// A warp works depth first on a stack of its own: a step takes up to 16
// pairs (32 ranges, one per lane) and, while few pairs are left and roots
// remain, roots on the lanes left over; every range that splits pushes one
// pair.  Nothing is exchanged with other warps meanwhile but the output
// count (one atomic per step).  Warps without work take a ticket of the
// bundle queue and wait for its slot.  A warp with pairs to spare gives the
// oldest (shallowest) ones away, up to kBundlePairs at a time, while tickets
// outnumber bundles, and whenever its ring could overflow.  With the CPU criterion a step has three parts:
//   the two lanes of a pair find its split direction, one the three lengths
//   along x, the other those along y (only ranges that split pay for them);
//   the new samples of all the step's ranges (three of a child, the other six
//   are its parent's, nine of a root) are dealt to the lanes one by one, so
//   a step of ten ranges takes a third of the time of a full one and lanes
//   do not diverge by split direction;
//   each lane bounds its range's nine points.
// With the GPU criterion all nine samples of every range are dealt.
template <int CRIT, int C>
__device__ __forceinline__ void bns_warp_loop(const DrawDev* draws, const int* __restrict__ root_prefix, int n_draws,
                                              const FrameDev& fr, const Queue& q, const SubPatches& out,
                                              unsigned* out_seq, RootInfo* roots, unsigned long long* ctrl,
                                              long long spin_limit, float* smem, unsigned claim, unsigned blocks) {
    static_assert(stack_stride<C>() > C + 32 && kPairWords > 27, "scratch columns and the words beside them");
    static_assert(C >= 32, "a step adds up to 16 pairs, or 32 to an empty ring");
    // Pairs are given to waiting warps when more than kGiveAbove are left, and
    // kKeep stay (a step of 16 ranges: on 1,024 Gregory patches bound-and-split
    // takes 0.145 ms, 0.174 ms when 16 stay); the ring is relieved when the
    // next step's pairs might not fit.
    constexpr int kGiveAbove = 11, kKeep = 8, kFull = C - 16;
    auto wrap = [](int i) { return i >= C ? i - C : i; };
    constexpr bool samples = CRIT == 0;
    constexpr int S = stack_stride<C>();
    const int lane = threadIdx.x & 31;
    float* ring = smem + (threadIdx.x >> 5) * (kPairWords * S);
    const unsigned epoch = (unsigned)*(volatile unsigned long long*)cw(ctrl, kEpoch);
    const unsigned R = (unsigned)*(volatile unsigned long long*)cw(ctrl, kRoots);   // (below 2^31)
    const unsigned warps = blockDim.x >> 5, n_warps = blocks * warps;
    const unsigned share = min(32u, (R + n_warps - 1) / n_warps);
    const unsigned dealt = n_warps * share;                   // roots from here on are taken with atomics
    // the claims that have roots (share s holds some while s * share < R)
    const unsigned busy = share ? min(blocks, (R + share - 1) / share) : 0;
    unsigned sh = claim + blocks * (threadIdx.x >> 5);        // the next share of this warp
    unsigned sh_left = claim < blocks ? 1 : 0;                // its shares left: sh, sh + blocks, ...
    unsigned root = 0, root_end = 0;                          // its next roots: [root, root_end)
    bool roots_left = dealt < R, claims_left = busy > 0;
    unsigned units = 0;                                       // units taken since the last report
    // in the words beside the scratch columns: ranges split since the last
    // report (lane 0), the depth of the deepest sub-patch emitted so far
    unsigned* kept = reinterpret_cast<unsigned*>(ring + C + 32);
    if (lane == 0) kept[0] = kept[S] = 0;
    __syncwarp();
    unsigned slot = 0;                                        // of this warp's ticket
    bool has_ticket = false;
    int bottom = 0, n = 0;    // ring: pairs bottom .. bottom + n - 1 (mod C)
    while (true) {
        if (root >= root_end && n < 8) {
            if (sh_left) {
                root = sh * share;
                root_end = max(root, min(root + share, R));
                sh += blocks;
                --sh_left;
                units += root_end - root;
            } else if (roots_left) {
                unsigned long long t = 0;
                if (lane == 0) t = atomicAdd(cw(ctrl, kRootHead), (unsigned long long)share);
                root = dealt + (unsigned)__shfl_sync(0xffffffffu, t, 0);
                root_end = max(root, min(root + share, R));
                units += root_end - root;
                roots_left = root < root_end;
            }
        }
        if (n == 0 && root >= root_end) {
            // out of work: report, then wait (bounded) for a bundle: first for
            // its pair count, then for its words, each valid once it carries
            // this frame's epoch
            int got = 0;
            unsigned stolen = busy;
            if (lane == 0) {
                if (kept[0]) atomicAdd(cw(ctrl, kSplits), (unsigned long long)kept[0]);
                kept[0] = 0;
                if (units && handover_ended(atomicAdd(cw(ctrl, kQTail), handover_finish(units)), units))
                    st_release_u64(cw(ctrl, kDone), 1ull);
                if (!has_ticket) slot = (unsigned)atomicAdd(cw(ctrl, kQHead), 1ull);
                unsigned idle = 0;
                unsigned sleep_ns = 32;
                while (true) {
                    if ((long long)slot < q.capacity) {
                        const unsigned long long v = ld_relaxed_u64(q.words + (size_t)slot * kBundleWords + kBundleWords - 1);
                        if ((unsigned)(v >> 32) == epoch) {
                            got = (int)(unsigned)v;
                            break;
                        }
                    }
                    if (*(volatile unsigned long long*)cw(ctrl, kDone)) break;
                    if (sleep_ns == 512 && claims_left) {
                        // a microsecond without work: blocks may not have started (claims only grow)
                        if (*(volatile unsigned long long*)cw(ctrl, kClaims) < busy)
                            stolen = (unsigned)atomicAdd(cw(ctrl, kClaims), 1ull);
                        if (stolen < busy) break;
                        claims_left = false;
                    }
                    if (++idle > spin_limit) {
                        set_status(ctrl, kErrTimeout);
                        st_release_u64(cw(ctrl, kDone), 1ull);
                        break;
                    }
                    __nanosleep(sleep_ns);
                    if (sleep_ns < 512) sleep_ns <<= 1;
                }
            }
            units = 0;
            stolen = __shfl_sync(0xffffffffu, stolen, 0);
            has_ticket = stolen < busy;   // (kept for the next wait)
            if (has_ticket) {
                sh = stolen;
                sh_left = warps;
                continue;
            }
            n = __shfl_sync(0xffffffffu, got, 0);
            if (n == 0) break;
            slot = __shfl_sync(0xffffffffu, slot, 0);
            units = 1;
            bottom = 0;
            const unsigned long long* rec = q.words + (size_t)slot * kBundleWords;
            unsigned tries = 0;
            bool valid;
            do {
                valid = true;
                for (int i = lane; i < kPairWords * kBundlePairs; i += 32)
                    if (i % kBundlePairs < n) {
                        const unsigned long long v = ld_relaxed_u64(rec + i);
                        valid = valid && (unsigned)(v >> 32) == epoch;
                        ring[(i / kBundlePairs) * S + (i % kBundlePairs)] = __uint_as_float((unsigned)v);
                    }
                valid = __all_sync(0xffffffffu, valid);
            } while (!valid && ++tries <= spin_limit);
            if (!valid) {
                if (lane == 0) {
                    set_status(ctrl, kErrTimeout);
                    st_release_u64(cw(ctrl, kDone), 1ull);
                }
                break;
            }
            __syncwarp();
        }
        // this step's ranges: pairs from the top of the ring, then roots
        const int pop = min(n, 16);
        const int n_root = (int)min((unsigned)(32 - 2 * pop), root_end - root);
        // tickets taken and bundles given so far, for the hand-over below
        // (loaded here so that the bounds cover the latency, and the bundles
        // from a word of their own: polled in kQTail, which every giver and
        // finisher updates, 64 views took 0.975 ms for 0.911, the 512x512
        // heightfield at 3840x2160 0.478 for 0.443)
        const bool may_give = n + pop + n_root > kGiveAbove;
        unsigned taken = 0, filled = 0;
        if (may_give && lane == 0) {
            taken = (unsigned)*(volatile unsigned long long*)cw(ctrl, kQHead);
            filled = (unsigned)*(volatile unsigned long long*)cw(ctrl, kGiven);
        }
        const int src = wrap(bottom + max(n - 1 - (lane >> 1), 0));
        const bool child = lane < 2 * pop, active = lane < 2 * pop + n_root;
        const int half = lane & 1;
        float4 r = make_float4(0.f, 0.f, 1.f, 1.f);
        int pid = 0, draw = 0, depth = 0;
        unsigned path = 0;
        bool split_x = false;   // of the pair's parent
        int dec = -1;
        float length = 0.0f;
        if (samples && child) length = split_length(ring + src, S, half);
        if (samples) {
            const float other = __shfl_xor_sync(0xffffffffu, length, 1);
            split_x = !(half ? other < length : length < other);   // vlen < hlen halves y
        }
        if (child) {
            const float* it = ring + src;
            const float4 pr = make_float4(it[27 * S], it[28 * S], it[29 * S], it[30 * S]);
            const unsigned w31 = __float_as_uint(it[31 * S]), w32 = __float_as_uint(it[32 * S]);
            if (!samples) split_x = w31 >> 31;
            pid = (int)(w31 & 0x7fffffffu);
            draw = (int)(w32 & 0xffffffu);
            depth = (int)(w32 >> 24) + 1;
            path = __float_as_uint(it[33 * S]);
            float4 c0, c1;
            split_children(pr, split_x ? kSplitX : kSplitY, c0, c1);
            r = half ? c1 : c0;
            // the high half sets bit 31 - parent's depth (paths deeper than 32 keep their first 32 bits)
            if (half && depth <= 32) path |= 0x80000000u >> (depth - 1);
        } else if (active) {
            // root: find the draw whose patch range holds it
            const int rt = (int)root + (lane - 2 * pop);
            int lo = 0, hi = n_draws - 1;
            while (lo < hi) {
                int mid = (lo + hi + 1) >> 1;
                if (__ldg(root_prefix + mid) <= rt) lo = mid; else hi = mid - 1;
            }
            draw = lo;
            pid = rt - __ldg(root_prefix + lo);
        }
        F3 pts[9];   // the range's samples, (iu, iv) at 3 * iv + iu (CPU criterion)
        if (samples) {
            // past the depth where sample parameters stay exact nothing is shared
            const bool share_pts = !__any_sync(0xffffffffu, child && depth > kInheritMaxDepth);
            const int flag = !child || !share_pts ? kInheritNone : split_x ? kInheritX : kInheritY;
            const int n_ct = 2 * pop * (share_pts ? 3 : 9), n_t = n_ct + 9 * n_root;
#pragma unroll 1
            for (int t0 = 0; t0 < n_t; t0 += 32) {
                const int t = t0 + lane;
                int q, k;   // sample k of lane q's range
                if (share_pts && t < n_ct) {
                    q = t / 3;
                    k = t - 3 * q;
                } else {
                    const int u = share_pts ? t - n_ct : t;
                    q = u / 9;
                    k = u - 9 * q;
                    if (share_pts) q += 2 * pop;
                }
                q &= 31;
                const float4 rq = make_float4(__shfl_sync(0xffffffffu, r.x, q), __shfl_sync(0xffffffffu, r.y, q),
                                              __shfl_sync(0xffffffffu, r.z, q), __shfl_sync(0xffffffffu, r.w, q));
                const int pq = __shfl_sync(0xffffffffu, pid, q);
                const int dq = __shfl_sync(0xffffffffu, draw | (flag << 24), q);
                if (t < n_t) {
                    const int fq = dq >> 24;
                    const int iu = fq == kInheritX ? 1 : fq == kInheritY ? k : k % 3;
                    const int iv = fq == kInheritX ? k : fq == kInheritY ? 1 : k / 3;
                    const float sv = fadd(rq.x, fmul(fmul(fsub(rq.z, rq.x), (float)iu), 0.5f));
                    const float su = fadd(rq.y, fmul(fmul(fsub(rq.w, rq.y), (float)iv), 0.5f));
                    const F3 p = bound_sample(draws[dq & 0xffffff], pq, sv, su);
                    float* to = ring + C + q + spi(iu, iv, 0, S);
                    to[0] = p.x;
                    to[S] = p.y;
                    to[2 * S] = p.z;
                }
            }
            __syncwarp();
            if (active) {
#pragma unroll
                for (int iv = 0; iv < 3; ++iv)
#pragma unroll
                    for (int iu = 0; iu < 3; ++iu) {
                        // the child's line 0 / 2 is the parent's line half / half + 1
                        int at = C + lane + spi(iu, iv, 0, S);
                        if (flag == kInheritX && iu != 1) at = src + spi(half + (iu >> 1), iv, 0, S);
                        if (flag == kInheritY && iv != 1) at = src + spi(iu, half + (iv >> 1), 0, S);
                        pts[3 * iv + iu] = F3{ring[at], ring[at + S], ring[at + 2 * S]};
                    }
                dec = bns_decide_points(draws[draw], fr, pts, depth);
            }
        } else {
            // nine samples of five words each, word w of sample k of lane l's
            // range: pairs keep no samples under this criterion, so words past
            // the scratch column's rows go to the unused rows of the ring
            auto word = [&](int l, int k, int w) {
                const int j = 5 * k + w;
                return j < 27 ? j * S + C + l : (j - 27) * S + l;
            };
            const int n_t = 9 * (2 * pop + n_root);
#pragma unroll 1
            for (int t0 = 0; t0 < n_t; t0 += 32) {
                const int t = t0 + lane, q = (t / 9) & 31, k = t % 9;   // sample k of lane q's range
                const float4 rq = make_float4(__shfl_sync(0xffffffffu, r.x, q), __shfl_sync(0xffffffffu, r.y, q),
                                              __shfl_sync(0xffffffffu, r.z, q), __shfl_sync(0xffffffffu, r.w, q));
                const int pq = __shfl_sync(0xffffffffu, pid, q), dq = __shfl_sync(0xffffffffu, draw, q);
                if (t < n_t) {
                    const GpuSample g = gpu_sample(draws[dq], pq, rq, k / 3, k % 3);
                    ring[word(q, k, 0)] = g.x;
                    ring[word(q, k, 1)] = g.y;
                    ring[word(q, k, 2)] = g.z;
                    ring[word(q, k, 3)] = g.s.x;
                    ring[word(q, k, 4)] = g.s.y;
                }
            }
            __syncwarp();
            if (active) {
                dec = kCull;
                if (depth < fr.max_depth - 1) {
                    GpuBound b;
                    b.clear();
#pragma unroll
                    for (int u = 0; u < 3; ++u) {
                        GpuSample c[3];
#pragma unroll
                        for (int v = 0; v < 3; ++v)
                            c[v] = GpuSample{ring[word(lane, 3 * u + v, 0)], ring[word(lane, 3 * u + v, 1)],
                                             ring[word(lane, 3 * u + v, 2)],
                                             make_float2(ring[word(lane, 3 * u + v, 3)], ring[word(lane, 3 * u + v, 4)])};
                        b.add(c, u == 0);
                    }
                    dec = b.decide(draws[draw], fr, r);
                }
            }
        }
        root += n_root;
        // emitted sub-patches: slots from one atomic, whose round trip the pushes below overlap
        const unsigned emask = __ballot_sync(0xffffffffu, dec == kDraw);
        const bool split = dec == kSplitX || dec == kSplitY;
        const unsigned smask = __ballot_sync(0xffffffffu, split);
        const unsigned emit_depth = __reduce_max_sync(0xffffffffu, dec == kDraw ? (unsigned)depth : 0u);
        unsigned obase = 0;
        if (lane == 0 && emask) obase = (unsigned)atomicAdd(cw(ctrl, kOutCount), (unsigned long long)__popc(emask));
        if (emit_depth > kept[S]) {
            // the sort packs the frame's keys into root bits above this many path bits
            __syncwarp();
            if (lane == 0) {
                kept[S] = emit_depth;
                atomicMax(cw(ctrl, kMaxDepth), (unsigned long long)emit_depth);
            }
        }
        if (roots && emask) {
            // one update per warp while its emitted ranges share a root, as
            // they do below the first levels of a tree, else one per root
            const unsigned ri = (unsigned)(__ldg(root_prefix + draw) + pid);
            const unsigned r0 = __shfl_sync(0xffffffffu, ri, __ffs(emask) - 1);
            if (__all_sync(0xffffffffu, dec != kDraw || ri == r0)) {
                const unsigned low = __reduce_min_sync(0xffffffffu, dec == kDraw ? path : 0xffffffffu);
                const unsigned high = __reduce_max_sync(0xffffffffu, dec == kDraw ? path : 0u);
                if (lane == 0) {
                    atomicAdd(&roots[r0].count, (unsigned)__popc(emask));
                    atomicMin(&roots[r0].low, low);
                    atomicMax(&roots[r0].high, high);
                }
            } else if (dec == kDraw) {
                const unsigned peers = __match_any_sync(emask, ri);
                const unsigned low = __reduce_min_sync(peers, path), high = __reduce_max_sync(peers, path);
                if ((peers & lanemask_lt()) == 0) {
                    atomicAdd(&roots[ri].count, (unsigned)__popc(peers));
                    atomicMin(&roots[ri].low, low);
                    atomicMax(&roots[ri].high, high);
                }
            }
        }
        // split ranges: one pair each, once every lane has read the popped pairs
        __syncwarp();
        n -= pop;
        if (split) {
            float* it = ring + wrap(bottom + n + __popc(smask & lanemask_lt()));
            if (samples) {
#pragma unroll
                for (int j = 0; j < 9; ++j) {
                    it[3 * j * S] = pts[j].x;
                    it[(3 * j + 1) * S] = pts[j].y;
                    it[(3 * j + 2) * S] = pts[j].z;
                }
            }
            it[27 * S] = r.x;
            it[28 * S] = r.y;
            it[29 * S] = r.z;
            it[30 * S] = r.w;
            it[31 * S] = __uint_as_float((unsigned)pid | (!samples && dec == kSplitX ? 0x80000000u : 0u));
            it[32 * S] = __uint_as_float((unsigned)draw | ((unsigned)depth << 24));
            it[33 * S] = __uint_as_float(path);
        }
        n += __popc(smask);
        if (lane == 0) kept[0] += (unsigned)__popc(smask);
        obase = __shfl_sync(0xffffffffu, obase, 0);
        if (dec == kDraw) {
            const unsigned o = obase + __popc(emask & lanemask_lt());
            if ((long long)o < out.capacity) {
                out.range[o] = r;
                out.meta[o] = make_int2(pid, draw);
                if (out.path) out.path[o] = path;
                // consumers running in the same launch wait for this flag
                if (out_seq) st_release_u32(out_seq + o, epoch);
            } else {
                set_status(ctrl, kErrOverflow);
            }
        }
        __syncwarp();
        // hand the oldest pairs over: to waiting warps, and what crowds the ring
        int wanting = 0;
        if (may_give && n > kGiveAbove) {
            if ((long long)filled < q.capacity) wanting = (int)taken - (int)filled;
            wanting = __shfl_sync(0xffffffffu, wanting, 0);
        }
        while (n > kFull || (wanting > 0 && n > kGiveAbove)) {
            const int give = min(kBundlePairs, n - kKeep);
            unsigned long long slot = 0;
            if (lane == 0) {
                slot = handover_slot(atomicAdd(cw(ctrl, kQTail), handover_give()));
                atomicAdd(cw(ctrl, kGiven), 1ull);
                if ((long long)slot >= q.capacity) atomicAdd(cw(ctrl, kQTail), handover_finish(1));
            }
            slot = __shfl_sync(0xffffffffu, slot, 0);
            if ((long long)slot < q.capacity) {
                unsigned long long* rec = q.words + slot * kBundleWords;
                const unsigned long long tag = (unsigned long long)epoch << 32;
                for (int i = lane; i < kPairWords * kBundlePairs; i += 32)
                    if (i % kBundlePairs < give)
                        st_relaxed_u64(rec + i, tag | __float_as_uint(ring[(i / kBundlePairs) * S +
                                                                           wrap(bottom + i % kBundlePairs)]));
                if (lane == 0) st_relaxed_u64(rec + kBundleWords - 1, tag | (unsigned)give);
            } else if (n > kFull) {
                set_status(ctrl, kErrOverflow);   // no room: the pairs are lost, the host grows the queue
            } else {
                break;                            // no room, but they can stay here
            }
            bottom = wrap(bottom + give);
            n -= give;
            --wanting;
        }
        __syncwarp();
    }
}

}  // namespace mp
