// Canonical order of a frame's emitted sub-patches.
//
// Bound-and-split emits sub-patches in whatever order its warps finish
// them, and the rasterizer numbers micropolygons by their sub-patch's list
// position (ties in depth go to the smaller number).  So that a frame's
// numbering, its winners at depth ties and everything read back from it are
// the same on every run, the list is put into one canonical order before
// rasterization: ascending (root, split path), where root = the draw's first
// root + patch id (draws in call order, as the reference's Scene::draw
// issues them, src/micropolis/Scene.cpp:179-197) and the split path holds,
// from the root down, 1 for each split whose high half the sub-patch lies in
// (bit 31 - d for the split at depth d).  Within one patch that is the
// depth-first order of its split tree, low half first.  The oracle numbers
// its sub-patches in the same order, so the two break ties identically.
//
// The sort is one launch of a resident grid, in phases separated by grid
// barriers (bounded waits on a counter of the frame's control words).
// Bound-and-split has counted each root's sub-patches and their lowest and
// highest path, so a root's place in the list is known after one prefix sum,
// and its paths are spread over as many buckets as it has sub-patches:
//   roots -- the roots' starts;
//   count -- every sub-patch takes a place in its bucket, the leading bits of
//            its path above the root's lowest (one atomic);
//   scan  -- the buckets' starts (sums of each block's stretch, then prefixes);
//   place -- path and source slot go to the bucket's next place;
//   rank  -- each sub-patch counts the smaller paths of its bucket and its
//            record is written to its final place.
// Each phase is one or two round trips to L2 per sub-patch and a barrier
// (about 4 us on a small frame).  Against the radix passes below, which cost
// some 20 us each: 13,496 sub-patches 51 -> 23 us, the mixed scene's 1.38 M
// 150 -> 61 us, 64 views' 5.66 M 593 -> 206 us, 2.73 M of the 512x512
// heightfield 240 -> 100 us.  Buckets of one size for the whole frame
// (leading bits of root and path) left thousands of a deeply split patch's
// sub-patches in one bucket.  A frame whose fullest
// bucket still holds more than kMaxBucket (a patch split deeply in a small
// part of its visible range) is sorted by radix passes instead, whose cost
// does not depend on the paths.  Their key packs the root above the frame's D
// path bits (D = the deepest emitted sub-patch; below bit 32 - D every path
// is zero, so the order is that of (root << 32 | path)); keys are 32 bits wide
// when the frame's root and path bits fit, else 64:
//   counts -- the digit counts of every pass at once (Adinets & Merrill's
//             one-sweep radix sort; warp matches aggregate a warp's equal
//             digits into one shared add), added to the frame's table;
//   plan   -- every block reads the table: a pass whose digit is the same
//             for every key moves nothing and is skipped;
//   passes -- each moving pass splits the keys into tiles of kSortTile, one
//             per block at a time (rounds of nblk tiles): each tile
//             ranks its digits stably (per-warp counters, warp matches),
//             publishes its digit counts, reorders itself by digit in shared
//             memory while it waits until every tile of its round and the
//             earlier ones has published, adds up the counts of the tiles
//             before it (independent loads, no chain of waits), and writes
//             each digit's run of the tile to consecutive addresses.  The
//             first moving pass forms the keys from the records; the last
//             writes the sub-patch records themselves in canonical order.
// Every wait is bounded (MP_ERR_TIMEOUT, no write after it).
#include "mp_bns_loop.cuh"

namespace mp {

namespace {

// The largest bucket that is ranked by counting: 2,048 paths cost each of them
// 2,048 compares of words in L1, a few microseconds, less than a radix pass.
constexpr unsigned kMaxBucket = 2048;
// Up to this many entries each block adds up the stretches before its own
// (32 loads a thread) instead of waiting for every block's sum.
constexpr unsigned kSumAlone = 16384;
// Up to this many roots each block keeps all their starts in shared memory (16
// loads a thread) instead of waiting for them to be written.
constexpr unsigned kRootsAlone = 8192;
constexpr int kSortBlock = 512;
constexpr int kSortWarps = kSortBlock / 32;
constexpr int kSortItems = 8;
constexpr int kSortTile = kSortBlock * kSortItems;   // keys per tile
constexpr int kDigits = 256;
static_assert(kRootsAlone <= 2 * kSortTile, "the starts take the place of the radix passes' keys");

__device__ __forceinline__ long long sort_count(const unsigned long long* ctrl, const SubPatches& in,
                                                const SortBuffers& sb) {
    long long n = (long long)*(volatile const unsigned long long*)(ctrl + kOutCount * kCtrlStride);
    if (n > in.capacity) n = in.capacity;
    if (n > sb.capacity) n = sb.capacity;
    return n;
}

template <typename K>
__device__ __forceinline__ unsigned digit_of(K key, int pass) {
    return (unsigned)(key >> (8 * pass)) & 0xffu;
}

// The root above D path bits (the path's bits below 32 - D are zero).
__device__ __forceinline__ unsigned long long pack_key(unsigned root, unsigned path, unsigned D) {
    return D == 0 ? (unsigned long long)root : ((unsigned long long)root << D) | (path >> (32u - D));
}

// Lanes of the warp whose 8-bit digit equals this lane's (valid = false
// lanes form a group of their own).
__device__ __forceinline__ unsigned match_digit(unsigned d, bool valid) {
    return __match_any_sync(0xffffffffu, valid ? d : 0x100u);
}

// Bits of the frame's keys: the root bits of its root count above D path bits.
__device__ __forceinline__ int key_bits(const unsigned long long* ctrl, unsigned* D_out) {
    const unsigned long long R = *(volatile const unsigned long long*)(ctrl + kRoots * kCtrlStride);
    unsigned D = (unsigned)*(volatile const unsigned long long*)(ctrl + kMaxDepth * kCtrlStride);
    if (D > 32) D = 32;
    if (D_out) *D_out = D;
    const int root_bits = R > 1 ? 64 - __clzll((long long)(R - 1)) : 0;
    return root_bits + (int)D;
}

// Waits (bounded) until all nblk working blocks have arrived at barrier
// number `k` of the frame (the counter ctrl kSortDone is zeroed by the
// frame's reset); false when the wait ran out (the status is then set).
__device__ __forceinline__ bool grid_barrier(unsigned long long* ctrl, unsigned long long k, int nblk,
                                             long long spin_limit, int* s_flag) {
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long* ctr = ctrl + kSortDone * kCtrlStride;
        __threadfence();
        atomicAdd(ctr, 1ull);
        const unsigned long long need = k * (unsigned long long)nblk;
        long long spins = 0;
        int ok = 1;
        while (ld_acquire_u64(ctr) < need) {
            if (++spins > spin_limit) {
                ok = 0;
                set_status(ctrl, kErrTimeout);
                break;
            }
            __nanosleep(32);
        }
        __threadfence();
        *s_flag = ok;
    }
    __syncthreads();
    return *s_flag != 0;
}

// Shared memory of one pass block (the 64-bit layout; 32-bit keys use the
// front half of `keys`).
struct PassSmem {
    unsigned long long keys[kSortTile];           // the tile in digit order
    unsigned vals[kSortTile];
    unsigned short wcount[kSortWarps][kDigits];   // per warp digit counts, then offsets in the tile's digit run
    unsigned tstart[kDigits];                     // exclusive digit starts within the tile
    unsigned start[kDigits];                      // exclusive digit starts of the pass
    unsigned base[kDigits];                       // global position of the tile's first key of each digit
    unsigned part[kDigits];                       // the earlier tiles of the tile's own group, per digit
    unsigned warp_sum[kSortWarps];
    int fail;
};

// Exclusive prefix over the 256 values that threads 0-255 hold (every
// thread of the block calls it; ends with a barrier).
__device__ __forceinline__ unsigned scan_digits(unsigned v, unsigned* warp_sum) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    unsigned x = v;
    if (tid < kDigits) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) warp_sum[warp] = x;
    }
    __syncthreads();
    unsigned before = 0;
    if (tid < kDigits)
        for (int w = 0; w < warp; ++w) before += warp_sum[w];
    __syncthreads();
    return before + x - v;
}

// One moving pass over keys of type K (see sort_kernel).
//   from_records -- the first moving pass: keys formed from the records
//   last         -- the last moving pass: records written in key order
template <typename K>
__device__ __forceinline__ bool pass_body(PassSmem& sm, const int* __restrict__ root_prefix, const SubPatches& in,
                                          const SubPatches& out, const SortBuffers& sb, unsigned long long* ctrl,
                                          int pass, long long n, unsigned D, int moves_before, bool last,
                                          unsigned h_pass, long long spin_limit, int nblk) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool from_records = moves_before == 0;
    // (selects, not an indexed load: the parameter arrays stay in registers)
    const int src = (moves_before - 1) & 1, dst_buf = moves_before & 1;
    const K* __restrict__ kin = reinterpret_cast<const K*>(src ? sb.keys[1] : sb.keys[0]);
    const unsigned* __restrict__ vin = src ? sb.vals[1] : sb.vals[0];
    K* kout = reinterpret_cast<K*>(dst_buf ? sb.keys[1] : sb.keys[0]);
    unsigned* vout = dst_buf ? sb.vals[1] : sb.vals[0];
    K* skeys = reinterpret_cast<K*>(sm.keys);
    unsigned* groups = sb.group_counts + (long long)pass * sb.groups * kDigits;
    unsigned long long* published = ctrl + (kSortTicket + pass) * kCtrlStride;
    {
        const unsigned st = scan_digits(tid < kDigits ? h_pass : 0u, sm.warp_sum);
        if (tid < kDigits) sm.start[tid] = st;
        if (tid == 0) sm.fail = 0;
    }
    const long long n_tiles = (n + kSortTile - 1) / kSortTile;
    const unsigned lt = (1u << lane) - 1u;
    for (long long tile = blockIdx.x; tile < n_tiles; tile += nblk) {
        const long long t0 = tile * kSortTile;
        const int tn = (int)(n - t0 < kSortTile ? n - t0 : kSortTile);
        for (int i = tid; i < kSortWarps * kDigits; i += kSortBlock) (&sm.wcount[0][0])[i] = 0;
        __syncthreads();
        // warp w ranks the keys [t0 + w * 32 * kSortItems, + 32 * kSortItems):
        // item i of lane l is key i * 32 + l of that run, so the ranks follow key order
        const long long run = t0 + (long long)warp * 32 * kSortItems;
        K k[kSortItems];
        unsigned v[kSortItems];
#pragma unroll
        for (int i = 0; i < kSortItems; ++i) {
            const long long idx = run + i * 32 + lane;
            k[i] = 0;
            v[i] = 0;
            if (idx < n) {
                if (from_records) {
                    const int2 m = __ldcg(in.meta + idx);
                    k[i] = (K)pack_key((unsigned)(__ldg(root_prefix + m.y) + m.x), __ldcg(in.path + idx), D);
                    v[i] = (unsigned)idx;
                } else {
                    k[i] = __ldcg(kin + idx);
                    v[i] = __ldcg(vin + idx);
                }
            }
        }
        unsigned short* wc = sm.wcount[warp];
        unsigned rank[kSortItems];
#pragma unroll
        for (int i = 0; i < kSortItems; ++i) {
            const bool valid = run + i * 32 + lane < n;
            const unsigned d = digit_of(k[i], pass);
            const unsigned peers = match_digit(d, valid);
            const unsigned before = valid ? wc[d] : 0u;
            rank[i] = before + (unsigned)__popc(peers & lt);
            __syncwarp();
            if (valid && (peers & lt) == 0) wc[d] = (unsigned short)(before + (unsigned)__popc(peers));
            __syncwarp();
        }
        __syncthreads();
        // thread d: the warps' offsets within digit d's run of the tile, the
        // tile's count of d (published), and the tile's digit starts
        unsigned tot = 0;
        if (tid < kDigits) {
#pragma unroll
            for (int w = 0; w < kSortWarps; ++w) {
                const unsigned c = sm.wcount[w][tid];
                sm.wcount[w][tid] = (unsigned short)tot;
                tot += c;
            }
            sb.counts[tile * kDigits + tid] = tot;
            if (tot) atomicAdd(groups + (tile / kSortGroup) * kDigits + tid, tot);
            __threadfence();
        }
        const unsigned ts = scan_digits(tot, sm.warp_sum);
        if (tid == 0) {
            // publish (every count above is fenced before the barrier in scan_digits)
            __threadfence();
            atomicAdd(published, 1ull);
        }
        if (tid < kDigits) sm.tstart[tid] = ts;
        __syncthreads();
        // the tile in digit order, in shared memory
#pragma unroll
        for (int i = 0; i < kSortItems; ++i) {
            if (run + i * 32 + lane < n) {
                const unsigned d = digit_of(k[i], pass);
                const unsigned local = sm.tstart[d] + sm.wcount[warp][d] + rank[i];
                skeys[local] = k[i];
                sm.vals[local] = v[i];
            }
        }
        if (tid == 0) {
            // wait until every tile up to the end of this round has published
            const long long round_end = (tile / nblk + 1) * nblk;
            const unsigned long long need = (unsigned long long)(round_end < n_tiles ? round_end : n_tiles);
            long long spins = 0;
            while (ld_acquire_u64(published) < need) {
                if (++spins > spin_limit) {
                    sm.fail = 1;
                    break;
                }
                __nanosleep(64);
            }
            __threadfence();
        }
        __syncthreads();
        if (sm.fail) {
            // a wait ran out: report it and write nothing with a wrong base
            if (tid == 0) set_status(ctrl, kErrTimeout);
            return false;
        }
        {
            // counts of the earlier tiles, digit d: thread d adds the whole
            // groups before this tile's group, thread d + 256 the earlier
            // tiles of its own group
            const int d = tid & (kDigits - 1);
            const long long g = tile / kSortGroup;
            unsigned sum = 0;
            if (tid < kDigits) {
                for (long long j = 0; j < g; j += 16) {
                    unsigned x[16];
#pragma unroll
                    for (int u = 0; u < 16; ++u) x[u] = j + u < g ? __ldcg(groups + (j + u) * kDigits + d) : 0u;
#pragma unroll
                    for (int u = 0; u < 16; ++u) sum += x[u];
                }
            } else {
                for (long long j = g * kSortGroup; j < tile; j += 16) {
                    unsigned x[16];
#pragma unroll
                    for (int u = 0; u < 16; ++u) x[u] = j + u < tile ? __ldcg(sb.counts + (j + u) * kDigits + d) : 0u;
#pragma unroll
                    for (int u = 0; u < 16; ++u) sum += x[u];
                }
                sm.part[d] = sum;
            }
            __syncthreads();
            if (tid < kDigits) sm.base[d] = sm.start[d] + sum + sm.part[d];
            __syncthreads();
        }
        // each digit's run of the tile to consecutive addresses
        if (last) {
            // the records, gathered two at a time with their loads issued together
            constexpr int kBatch = 2;
            for (int j0 = tid; j0 < tn; j0 += kBatch * kSortBlock) {
                float4 rg[kBatch];
                int2 mt[kBatch];
                long long dst[kBatch];
#pragma unroll
                for (int u = 0; u < kBatch; ++u) {
                    const int j = j0 + u * kSortBlock;
                    dst[u] = -1;
                    if (j < tn) {
                        const unsigned d = digit_of(skeys[j], pass);
                        const long long o = (long long)sm.base[d] + (j - (int)sm.tstart[d]);
                        const unsigned sv = sm.vals[j];
                        if (o < n && o < out.capacity && sv < (unsigned)n) {
                            dst[u] = o;
                            rg[u] = __ldcg(in.range + sv);
                            mt[u] = __ldcg(in.meta + sv);
                        }
                    }
                }
#pragma unroll
                for (int u = 0; u < kBatch; ++u)
                    if (dst[u] >= 0) {
                        out.range[dst[u]] = rg[u];
                        out.meta[dst[u]] = mt[u];
                    }
            }
        } else {
            for (int j = tid; j < tn; j += kSortBlock) {
                const K key = skeys[j];
                const unsigned d = digit_of(key, pass);
                const long long dst = (long long)sm.base[d] + (j - (int)sm.tstart[d]);
                if (dst < n) {
                    kout[dst] = key;
                    vout[dst] = sm.vals[j];
                }
            }
        }
        __syncthreads();
    }
    return true;
}

// Sum over the block (every thread calls it and gets the sum; ends with a barrier).
__device__ __forceinline__ unsigned block_sum(unsigned v, unsigned* warp_sum) {
    const int tid = threadIdx.x;
    v = __reduce_add_sync(0xffffffffu, v);
    if ((tid & 31) == 0) warp_sum[tid >> 5] = v;
    __syncthreads();
    unsigned t = 0;
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) t += warp_sum[w];
    __syncthreads();
    return t;
}

// How many of keys[from, to) are below `key`: eight at a time, so that a
// crowded bucket (up to kMaxBucket; the usual one holds a few) costs a few
// cycles a key and not a load's latency each.
__device__ __forceinline__ unsigned count_below(const unsigned* keys, unsigned from, unsigned to, unsigned key) {
    unsigned c = 0, j = from;
    for (; j < to && (j & 3u); ++j) c += keys[j] < key;
    for (; j + 8 <= to; j += 8) {
        const uint4 a = *reinterpret_cast<const uint4*>(keys + j), b = *reinterpret_cast<const uint4*>(keys + j + 4);
        c += (a.x < key) + (a.y < key) + (a.z < key) + (a.w < key) + (b.x < key) + (b.y < key) + (b.z < key) +
             (b.w < key);
    }
    for (; j < to; ++j) c += keys[j] < key;
    return c;
}

// A root's bucket of a path: the root's start and the leading bits of the
// path above its lowest, at most as many buckets as it has sub-patches.
__device__ __forceinline__ unsigned bucket_of(const RootInfo& ri, unsigned path) {
    const int range_bits = 32 - __clz((int)(ri.high - ri.low));
    const int shift = max(0, range_bits - (31 - __clz((int)ri.count)));
    return ri.start + ((path - ri.low) >> shift);
}

__device__ __forceinline__ RootInfo load_root(const RootInfo* r) {
    const uint4 v = __ldcg(reinterpret_cast<const uint4*>(r));
    return RootInfo{v.x, v.y, v.z, v.w};
}

// Exclusive prefix over the block of each thread's v, from `run`; adds the
// block's total to run (every thread calls it; ends with a barrier).
__device__ __forceinline__ unsigned block_prefix(unsigned v, unsigned& run, unsigned* warp_sum) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sum[warp] = x;
    __syncthreads();
    unsigned pre = run, all = 0;
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) {
        if (w < warp) pre += warp_sum[w];
        all += warp_sum[w];
    }
    __syncthreads();
    run += all;
    return pre + x - v;
}

// The sum of all entries before this block's stretch: `entry(i)` reads one,
// lo is the stretch's begin, per its length, own its sum.  Long tables go
// through every block's sum and a barrier; false when that wait ran out.
template <typename F>
__device__ __forceinline__ bool sum_before(F entry, unsigned total, unsigned lo, unsigned own, unsigned* sums,
                                           unsigned long long* ctrl, int nblk, unsigned long long& barrier,
                                           long long spin_limit, unsigned* warp_sum, int* s_flag, unsigned& before) {
    const int tid = threadIdx.x;
    unsigned v = 0;
    if (total <= kSumAlone) {
        for (unsigned i = tid; i < lo; i += kSortBlock) v += entry(i);
    } else {
        own = block_sum(own, warp_sum);
        if (tid == 0) sums[blockIdx.x] = own;
        if (!grid_barrier(ctrl, ++barrier, nblk, spin_limit, s_flag)) return false;
        for (int j = tid; j < (int)blockIdx.x; j += kSortBlock) v += __ldcg(sums + j);
    }
    before = block_sum(v, warp_sum);
    return true;
}

// The bucket sort (file header).  Returns 1 when done, 0 when a bucket is too
// full (nothing is written to `out`), -1 when a wait ran out.
__device__ __forceinline__ int bucket_sort(const int* __restrict__ root_prefix, const SubPatches& in,
                                           const SubPatches& out, const SortBuffers& sb, unsigned long long* ctrl,
                                           long long n, int nblk, unsigned long long& barrier, long long spin_limit,
                                           unsigned* s_start, unsigned* warp_sum, int* s_flag) {
    constexpr int kBatch = 4;   // sub-patches a thread handles at a time, their loads in flight together
    const int tid = threadIdx.x;
    const long long gt = (long long)blockIdx.x * kSortBlock + tid, stride = (long long)nblk * kSortBlock;
    const unsigned R = (unsigned)*(volatile unsigned long long*)cw(ctrl, kRoots);
    RootInfo* roots = sb.roots;
    unsigned* table = sb.table;
    unsigned* place = sb.vals[0];
    unsigned* slot_path = reinterpret_cast<unsigned*>(sb.keys[0]);
    unsigned* slot_src = sb.vals[1];
    // the starts replace the counts, but of a short table other blocks still
    // read the counts when this one writes
    unsigned* starts = n <= kSumAlone ? reinterpret_cast<unsigned*>(sb.keys[1]) : table;
    // the next frame's bound-and-split clears what this one uses of the table
    if (gt == 0) *sb.used = (unsigned)n + 4;
    // roots
    const bool alone = R <= kRootsAlone;
    if (alone) {
        unsigned run = 0;
        for (unsigned t0 = 0; t0 < R; t0 += kSortBlock) {
            const unsigned i = t0 + tid;
            const unsigned pre = block_prefix(i < R ? __ldcg(&roots[i].count) : 0u, run, warp_sum);
            if (i < R) s_start[i] = pre;
        }
        __syncthreads();
    } else {
        const unsigned per = (R + nblk - 1) / nblk, lo = min(per * blockIdx.x, R), hi = min(lo + per, R);
        unsigned own = 0, run = 0;
        if (R > kSumAlone)
            for (unsigned i = lo + tid; i < hi; i += kSortBlock) own += __ldcg(&roots[i].count);
        if (!sum_before([&](unsigned i) { return __ldcg(&roots[i].count); }, R, lo, own, sb.sums, ctrl, nblk, barrier,
                        spin_limit, warp_sum, s_flag, run))
            return -1;
        for (unsigned t0 = lo; t0 < hi; t0 += kSortBlock) {
            const unsigned i = t0 + tid;
            const unsigned pre = block_prefix(i < hi ? __ldcg(&roots[i].count) : 0u, run, warp_sum);
            if (i < hi) roots[i].start = pre;
        }
        if (!grid_barrier(ctrl, ++barrier, nblk, spin_limit, s_flag)) return -1;
    }
    // a record's bucket
    auto bucket = [&](int2 m, unsigned path) {
        const int r = __ldg(root_prefix + m.y) + m.x;
        RootInfo ri = load_root(roots + r);
        if (alone) ri.start = s_start[r];
        return bucket_of(ri, path);
    };
    // count
    for (long long i0 = gt; i0 < n; i0 += kBatch * stride) {
        int2 m[kBatch];
        unsigned p[kBatch], at[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            const long long i = min(i0 + u * stride, n - 1);
            m[u] = __ldcg(in.meta + i);
            p[u] = __ldcg(in.path + i);
        }
#pragma unroll
        for (int u = 0; u < kBatch; ++u) at[u] = bucket(m[u], p[u]);
#pragma unroll
        for (int u = 0; u < kBatch; ++u)
            if (i0 + u * stride < n && at[u] < (unsigned)n) at[u] = atomicAdd(table + at[u], 1u);
#pragma unroll
        for (int u = 0; u < kBatch; ++u)
            if (i0 + u * stride < n) place[i0 + u * stride] = at[u];
    }
    if (!grid_barrier(ctrl, ++barrier, nblk, spin_limit, s_flag)) return -1;
    {
        // scan: this block's stretch of the table, whole uint4s
        const unsigned nb = (unsigned)n, per = ((nb + nblk - 1) / nblk + 3) & ~3u;
        const unsigned lo = min(per * blockIdx.x, nb), hi = min(lo + per, nb);
        unsigned own = 0, most = 0, run = 0;
        for (unsigned i = lo + 4 * tid; i < hi; i += 4 * kSortBlock) {
            const uint4 c = __ldcg(reinterpret_cast<const uint4*>(table + i));
            own += c.x + c.y + c.z + c.w;
            most = max(max(max(most, c.x), max(c.y, c.z)), c.w);
        }
        most = __reduce_max_sync(0xffffffffu, most);
        if ((tid & 31) == 0 && most > kMaxBucket) atomicMax(cw(ctrl, kSortMost), (unsigned long long)most);
        if (!sum_before([&](unsigned i) { return __ldcg(table + i); }, nb, lo, own, sb.sums, ctrl, nblk, barrier,
                        spin_limit, warp_sum, s_flag, run))
            return -1;
        for (unsigned t0 = lo; t0 < hi; t0 += 4 * kSortBlock) {
            const unsigned i = t0 + 4 * tid;
            uint4 c = make_uint4(0, 0, 0, 0);
            if (i < hi) c = __ldcg(reinterpret_cast<const uint4*>(table + i));
            const unsigned pre = block_prefix(c.x + c.y + c.z + c.w, run, warp_sum);
            if (i < hi)
                *reinterpret_cast<uint4*>(starts + i) = make_uint4(pre, pre + c.x, pre + c.x + c.y, pre + c.x + c.y + c.z);
        }
        if (hi == nb && lo < nb && tid == 0) starts[nb] = nb;
    }
    if (!grid_barrier(ctrl, ++barrier, nblk, spin_limit, s_flag)) return -1;
    if (*(volatile unsigned long long*)cw(ctrl, kSortMost)) return 0;
    // place
    for (long long i0 = gt; i0 < n; i0 += kBatch * stride) {
        int2 m[kBatch];
        unsigned p[kBatch], at[kBatch], b[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            const long long i = min(i0 + u * stride, n - 1);
            m[u] = __ldcg(in.meta + i);
            p[u] = __ldcg(in.path + i);
            at[u] = __ldcg(place + i);
        }
#pragma unroll
        for (int u = 0; u < kBatch; ++u) b[u] = bucket(m[u], p[u]);
#pragma unroll
        for (int u = 0; u < kBatch; ++u) at[u] += __ldcg(starts + min(b[u], (unsigned)n));
#pragma unroll
        for (int u = 0; u < kBatch; ++u)
            if (i0 + u * stride < n && at[u] < (unsigned)n) {
                slot_path[at[u]] = p[u];
                slot_src[at[u]] = (unsigned)(i0 + u * stride);
            }
    }
    if (!grid_barrier(ctrl, ++barrier, nblk, spin_limit, s_flag)) return -1;
    // rank
    constexpr int kRank = 2;
    const bool ties = *(volatile unsigned long long*)cw(ctrl, kMaxDepth) >= 32;   // paths beyond 32 splits: by place
    for (long long i0 = gt; i0 < n; i0 += kRank * stride) {
        unsigned src[kRank], p[kRank], b[kRank];
        int2 m[kRank];
        float4 rg[kRank];
#pragma unroll
        for (int u = 0; u < kRank; ++u) src[u] = min(__ldcg(slot_src + min(i0 + u * stride, n - 1)), (unsigned)n - 1);
#pragma unroll
        for (int u = 0; u < kRank; ++u) {
            m[u] = __ldcg(in.meta + src[u]);
            p[u] = __ldcg(in.path + src[u]);
            rg[u] = __ldcg(in.range + src[u]);
        }
#pragma unroll
        for (int u = 0; u < kRank; ++u) b[u] = min(bucket(m[u], p[u]), (unsigned)n - 1);
#pragma unroll
        for (int u = 0; u < kRank; ++u) {
            if (i0 + u * stride >= n) break;
            const unsigned start = __ldcg(starts + b[u]), end = min(__ldcg(starts + b[u] + 1), (unsigned)n);
            unsigned to = start;
            if (end - start > 1) {
                to += count_below(slot_path, start, end, p[u]);
                if (ties)
                    for (unsigned j = start; j < (unsigned)(i0 + u * stride); ++j) to += slot_path[j] == p[u];
            }
            if (to < (unsigned)n && (long long)to < out.capacity) {
                out.range[to] = rg[u];
                out.meta[to] = m[u];
            }
        }
    }
    return 1;
}

// The whole sort in one launch of a resident grid (see the file header).
__global__ void __launch_bounds__(kSortBlock, 2) sort_kernel(const int* __restrict__ root_prefix, SubPatches in,
                                                             SubPatches out, SortBuffers sb, unsigned long long* ctrl,
                                                             int n_passes, long long spin_limit) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    PassSmem& sm = *reinterpret_cast<PassSmem*>(smem_raw);
    __shared__ int s_flag;
    stamp_start(ctrl, 2);
    const int tid = threadIdx.x, lane = tid & 31;
    const long long n = sort_count(ctrl, in, sb);
    unsigned D = 0;
    const int bits = key_bits(ctrl, &D);
    // the working blocks: enough for a sub-patch and a root per thread, at most
    // the grid; the others return at once and every barrier counts the working
    // blocks only
    const long long R = (long long)*(volatile unsigned long long*)cw(ctrl, kRoots);
    const long long want = ((n > R ? n : R) + kSortBlock - 1) / kSortBlock;
    const int nblk = (int)(want < 1 ? 1 : want < gridDim.x ? want : gridDim.x);
    if ((int)blockIdx.x >= nblk || n == 0) return;
    unsigned long long barrier = 0;
    if (bucket_sort(root_prefix, in, out, sb, ctrl, n, nblk, barrier, spin_limit, reinterpret_cast<unsigned*>(sm.keys),
                    sm.warp_sum, &s_flag) != 0)
        return;
    // radix passes: a table and counters of zeros first
    const int active = (bits + 7) / 8 < n_passes ? (bits + 7) / 8 : n_passes;
    unsigned* hist = sb.hist;
    {
        const long long gt = (long long)blockIdx.x * kSortBlock + tid, gstride = (long long)nblk * kSortBlock;
        for (long long i = gt; i < kSortPasses * kDigits; i += gstride) hist[i] = 0;
        for (long long i = gt; i < kSortPasses * sb.groups * kDigits; i += gstride) sb.group_counts[i] = 0;
        if (blockIdx.x == 0 && tid < kSortPasses) ctrl[(kSortTicket + tid) * kCtrlStride] = 0;
        if (!grid_barrier(ctrl, ++barrier, nblk, spin_limit, &s_flag)) return;
        // counts: of this block's stripe of keys into shared memory (the
        // front of the pass buffers), then into the frame's table
        unsigned* s_hist = reinterpret_cast<unsigned*>(smem_raw);
        for (int i = tid; i < kSortPasses * kDigits; i += kSortBlock) s_hist[i] = 0;
        __syncthreads();
        const unsigned lt = (1u << lane) - 1u;
        // whole warps step together so that the warp matches below see every lane
        for (long long base = (long long)blockIdx.x * kSortBlock + (tid & ~31); base < n; base += gstride) {
            const long long i = base + lane;
            const bool valid = i < n;
            unsigned long long key = 0;
            if (valid) {
                const int2 m = __ldcg(in.meta + i);
                key = pack_key((unsigned)(__ldg(root_prefix + m.y) + m.x), __ldcg(in.path + i), D);
            }
            for (int p = 0; p < active; ++p) {
                const unsigned d = digit_of(key, p);
                const unsigned peers = match_digit(d, valid);
                if (valid && (peers & lt) == 0) atomicAdd(&s_hist[p * kDigits + d], (unsigned)__popc(peers));
            }
        }
        __syncthreads();
        for (int i = tid; i < active * kDigits; i += kSortBlock) {
            const unsigned v = s_hist[i];
            if (v) atomicAdd(hist + i, v);
        }
    }
    if (!grid_barrier(ctrl, ++barrier, nblk, spin_limit, &s_flag)) return;
    // plan: a pass moves keys unless one digit holds them all
    int moving = 0;
    unsigned moves_mask = 0;
#pragma unroll 1
    for (int q = 0; q < active; ++q) {
        const unsigned hq = tid < kDigits ? __ldcg(hist + q * kDigits + tid) : 0u;
        if (!__syncthreads_or(tid < kDigits && (long long)hq == n)) {
            moves_mask |= 1u << q;
            ++moving;
        }
    }
    if (moving == 0) {
        // no pass moves anything (n <= 1): the records are already in order
        const long long stride = (long long)nblk * kSortBlock;
        for (long long j = (long long)blockIdx.x * kSortBlock + tid; j < n && j < out.capacity; j += stride) {
            out.range[j] = in.range[j];
            out.meta[j] = in.meta[j];
        }
        return;
    }
    int before = 0;
#pragma unroll 1
    for (int q = 0; q < active; ++q) {
        if (!((moves_mask >> q) & 1u)) continue;
        const unsigned hq = tid < kDigits ? __ldcg(hist + q * kDigits + tid) : 0u;   // thread d: count of digit d
        const bool last = before == moving - 1;
        bool ok;
        if (bits <= 32)
            ok = pass_body<unsigned>(sm, root_prefix, in, out, sb, ctrl, q, n, D, before, last, hq, spin_limit, nblk);
        else
            ok = pass_body<unsigned long long>(sm, root_prefix, in, out, sb, ctrl, q, n, D, before, last, hq,
                                               spin_limit, nblk);
        if (!ok) return;
        // the next pass reads what every block of this one wrote
        if (!last && !grid_barrier(ctrl, ++barrier, nblk, spin_limit, &s_flag)) return;
        ++before;
    }
}

int sm_count() {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

}  // namespace

long long sort_tiles(long long n) { return (n + kSortTile - 1) / kSortTile; }

int canonical_sort_passes(int max_split_depth, long long roots) {
    // leaves lie at depth <= max_split_depth + 1; a path keeps 32 bits
    const int path_bits = max_split_depth + 1 < 32 ? max_split_depth + 1 : 32;
    int root_bits = 0;
    while (root_bits < 32 && ((roots - 1) >> root_bits) > 0) ++root_bits;
    const int bits = path_bits + root_bits;
    return bits <= 8 ? 1 : (bits + 7) / 8;
}

int canonical_sort_grid() {
    // blocks resident at once (the grid barriers and round waits rely on it)
    cudaFuncSetAttribute(sort_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(PassSmem));
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, sort_kernel, kSortBlock, sizeof(PassSmem));
    return sm_count() * (per_sm < 1 ? 1 : per_sm);
}

void launch_canonical_sort(const int* root_prefix, const SubPatches& in, const SubPatches& out, const SortBuffers& sb,
                           unsigned long long* ctrl, long long spin_limit, int n_passes, int resident_grid,
                           cudaStream_t s) {
    const long long want = (sb.capacity + kSortBlock - 1) / kSortBlock;
    const int grid = (int)(want < 1 ? 1 : want < resident_grid ? want : resident_grid);
    sort_kernel<<<grid, kSortBlock, sizeof(PassSmem), s>>>(root_prefix, in, out, sb, ctrl, n_passes, spin_limit);
}

}  // namespace mp
