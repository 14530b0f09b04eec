// Per-substep particle ordering by grid cell, grouped by 4x4x4 grid block.
//
// The reference scatters every particle straight into global memory
// (p2g_apic_stress_given, engine_stress/mpm_utils.py:190-227: 7 float
// atomics per node, 189 per particle).  Here particles are ordered by the
// cell of their stencil base, block-major, so P2G can accumulate a block's
// nodes in shared memory and find each cell's particles as one range.  The
// order is a two-level counting (radix) sort on the cell key
// block * 64 + cell:
//   keys + histograms -- written by G2P for the next substep (block and
//                        cell counts), or by key_kernel after a load moved
//                        particles
//   scan              -- block offsets, the P2G block list and the G2P chunk
//                        list; for each non-empty block, its 64 cell offsets
//                        (after bucket_sums on large grids)
//   scatter           -- order[] via warp-aggregated cell-cursor atomics
// G2P then writes every record to the other state buffer at its sorted
// position, so order[] stays close to the identity from one substep to the
// next and the gathers through it stay coalesced.
#include "mpm_device.cuh"
#include "mpm_launch.h"

namespace mpm {

// keys + histogram straight from x0 + u (used after loads)
__global__ void key_kernel(const MpmScene *__restrict__ scenes, int n_scenes, PState st, Ws ws,
                           int n, int *status) {
    chain_wait();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int key = -1;
    if (i < n) {
        const float4 q0 = ldrec(st, i, 0), q1 = ldrec(st, i, 1), q2 = ldrec(st, i, 2);
        const int uid = __float_as_int(q1.y);
        const MpmScene &S = scenes[scene_of_particle(scenes, n_scenes, uid)];
        bool ok;
        key = particle_key(S, q0.x, q0.y, q0.z, q2.x, q2.y, q2.z, ws.nbk - 1, ok);
        if (!ok) atomicOr(status, MPM_ST_OUT_OF_DOMAIN);
        st.key[i] = key;
    }
    warp_histogram(ws.counts, ws.cell_counts, key);
}

__device__ __forceinline__ int4 add4(int4 a, int4 b) {
    return make_int4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}

// inclusive scan of an int4 over the kScanThreads threads of a CTA; returns
// the thread's inclusive value and leaves the CTA total in total
constexpr int kScanWarps = kScanThreads / 32;
__device__ __forceinline__ int4 cta_scan4(int4 v, int4 *wsum /* [kScanWarps] shared */, int4 &total) {
    int4 x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int4 y;
        y.x = __shfl_up_sync(0xffffffffu, x.x, o);
        y.y = __shfl_up_sync(0xffffffffu, x.y, o);
        y.z = __shfl_up_sync(0xffffffffu, x.z, o);
        y.w = __shfl_up_sync(0xffffffffu, x.w, o);
        if ((threadIdx.x & 31) >= o) x = add4(x, y);
    }
    if ((threadIdx.x & 31) == 31) wsum[threadIdx.x >> 5] = x;
    __syncthreads();
    int4 pre = make_int4(0, 0, 0, 0);
    total = make_int4(0, 0, 0, 0);
    for (int w = 0; w < kScanWarps; ++w) {
        if (w < (int)(threadIdx.x >> 5)) pre = add4(pre, wsum[w]);
        total = add4(total, wsum[w]);
    }
    __syncthreads();
    return add4(pre, x);
}

// per-bucket triple: (particles, G2P chunks, non-empty blocks) -- the
// sentinel bucket (out-of-domain particles) gets copy chunks but no block
__device__ __forceinline__ int4 bucket_triple(const Ws &ws, int b, int cnt) {
    const int ch = (cnt + ws.chunk_size - 1) / ws.chunk_size;
    if (b >= ws.nbk - 1) return make_int4(cnt, ch, 0, 0);
    return make_int4(cnt, ch, cnt > 0 ? 1 : 0, 0);
}

// sum of an int4 over the kScanThreads threads of a CTA (every thread gets it)
__device__ __forceinline__ int4 cta_sum4(int4 v, int4 *wsum /* [kScanWarps] shared */) {
    v.x = __reduce_add_sync(0xffffffffu, v.x);
    v.y = __reduce_add_sync(0xffffffffu, v.y);
    v.z = __reduce_add_sync(0xffffffffu, v.z);
    if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5] = v;
    __syncthreads();
    int4 t = make_int4(0, 0, 0, 0);
    for (int w = 0; w < kScanWarps; ++w) t = add4(t, wsum[w]);
    __syncthreads();
    return t;
}

// Sums of kSumTile buckets each, for grids too large for scan_kernel to add up
// the counts themselves.
constexpr int kSumTile = 512;
__global__ void __launch_bounds__(kScanThreads) bucket_sums_kernel(Ws ws) {
    chain_wait();
    __shared__ int4 wsum[kScanWarps];
    int4 acc = make_int4(0, 0, 0, 0);
#pragma unroll
    for (int k = 0; k < kSumTile / kScanThreads; ++k) {
        const int b = blockIdx.x * kSumTile + k * kScanThreads + (int)threadIdx.x;
        if (b < ws.nbk) acc = add4(acc, bucket_triple(ws, b, ws.counts[b]));
    }
    const int4 t = cta_sum4(acc, wsum);
    if (threadIdx.x == 0) ws.tile_sums[blockIdx.x] = t;
}

// Sums of kSuperTiles tile sums each, for grids of so many buckets that a CTA's sum over
// all earlier tiles counts (it grows with the square of the buckets).  A group's three sums
// go into the unused fourth words of its first three tile sums; nobody needs those of a
// last group that has fewer.
constexpr int kSuperTiles = kScanThreads;
__global__ void __launch_bounds__(kScanThreads) super_sums_kernel(Ws ws, int n_tiles) {
    chain_wait();
    __shared__ int4 wsum[kScanWarps];
    const int i = blockIdx.x * kSuperTiles + (int)threadIdx.x;
    int4 v = i < n_tiles ? ws.tile_sums[i] : make_int4(0, 0, 0, 0);
    const int4 t = cta_sum4(v, wsum);
    if (threadIdx.x < 3 && i < n_tiles) ws.tile_sums[i].w = threadIdx.x == 0 ? t.x : (threadIdx.x == 1 ? t.y : t.z);
}

// Bucket offsets / cursors, the G2P chunk list and the P2G block list.  A CTA
// owns KB buckets and finds what lies before them by itself, so no
// CTA waits for another and no pass over tile sums comes in between: from the
// counts of all earlier buckets (a few independent loads a thread while there are
// at most kDirectBuckets of them), from bucket_sums_kernel's sums, or (past
// kSuperBuckets) from super_sums_kernel's first.  Then its warps take its
// non-empty buckets and write the 64 cell offsets of each with a warp scan (two
// cells per lane), and its chunk-list entries with one lane per chunk.  The last
// CTA publishes the list lengths.
// (A kernel that scanned all tile sums behind an atomic ticket cost 5 to 12 us a
// substep.  Handing the ranges out with atomics, in the order CTAs arrive, is as
// fast here but scatters neighbouring blocks: P2G 3 % slower on 64 scenes.)
constexpr int kDirectBuckets = 8192;  // an 80^3 grid: up to eight 16-byte loads a thread
// KB buckets per CTA: the non-empty blocks of a column lie side by side, so a
// few CTAs hold most of them and need the warps (64 buckets a CTA instead of
// 256: sort of the 1M column 26.8 -> 22.5 us).  Past kWideBuckets there are
// CTAs enough, and each one's sum over the tile sums counts (256 instead of 64:
// 64 scenes, 420k buckets, 74 -> 62 us).
constexpr int kWideBuckets = 1 << 17;
// Past kSuperBuckets that sum is what counts: sort of a 512^3 grid (2.1M buckets) 121 us
// with one level of sums, 119 with two; 800^3 441, 364; 1024^3 1,078, 692; 1280^3 2,809, 1,275.
constexpr int kSuperBuckets = 1 << 20;
template <int SUMS, int KB>  // SUMS: levels of sums to read (0-2)
__global__ void __launch_bounds__(kScanThreads) scan_kernel(const MpmScene *__restrict__ scenes, int n_scenes,
                                                            Ws ws) {
    chain_wait();
    __shared__ int4 wsum[kScanWarps];
    __shared__ int s_off[KB], s_coff[KB], s_boff[KB], s_cnt[KB];
    __shared__ int s_list[KB];
    const int tile = blockIdx.x;
    const int b0 = tile * KB;
    const bool owner = (int)threadIdx.x < KB;  // of bucket b
    const int b = owner ? b0 + (int)threadIdx.x : ws.nbk;
    const int cnt = b < ws.nbk ? ws.counts[b] : 0;
    // what lies before the CTA's buckets (b0 is a multiple of four, and no bucket
    // before it is the sentinel, the last one)
    int4 pre = make_int4(0, 0, 0, 0);
    if (SUMS > 0) {
        const int full = b0 / kSumTile;
        int first = 0;  // tile
        if (SUMS > 1) {
            const int groups = full / kSuperTiles;
            for (int g = threadIdx.x; g < groups; g += kScanThreads) {
                const int4 *s = ws.tile_sums + (int64_t)g * kSuperTiles;
                pre = add4(pre, make_int4(s[0].w, s[1].w, s[2].w, 0));
            }
            first = groups * kSuperTiles;
        }
        for (int t = first + (int)threadIdx.x; t < full; t += kScanThreads) pre = add4(pre, ws.tile_sums[t]);
        for (int h = full * kSumTile + (int)threadIdx.x; h < b0; h += kScanThreads)
            pre = add4(pre, bucket_triple(ws, h, ws.counts[h]));
    } else {
        const int4 *c4 = reinterpret_cast<const int4 *>(ws.counts);
#pragma unroll 8
        for (int i = threadIdx.x; i < b0 / 4; i += kScanThreads) {
            const int4 c = c4[i];
            pre = add4(pre, add4(add4(bucket_triple(ws, 0, c.x), bucket_triple(ws, 0, c.y)),
                                 add4(bucket_triple(ws, 0, c.z), bucket_triple(ws, 0, c.w))));
        }
    }
    pre = cta_sum4(pre, wsum);
    int4 mine = b < ws.nbk ? bucket_triple(ws, b, cnt) : make_int4(0, 0, 0, 0);
    // the out-of-domain bucket always gets its cursor (G2P's copy chunks count its particles again)
    const bool listed = b < ws.nbk && (cnt > 0 || b == ws.nbk - 1);
    mine.w = listed ? 1 : 0;
    int4 total;
    const int4 inc = cta_scan4(mine, wsum, total);
    const int nlist = total.w;
    if (listed) s_list[inc.w - 1] = (int)threadIdx.x;
    if (owner) {
        s_off[threadIdx.x] = pre.x + inc.x - mine.x;
        s_coff[threadIdx.x] = pre.y + inc.y - mine.y;
        s_boff[threadIdx.x] = pre.z + inc.z - mine.z;
        s_cnt[threadIdx.x] = cnt;
    }
    if (threadIdx.x == 0 && tile == (int)gridDim.x - 1) {
        // counts always sum to n when the stages run in order; the clamps keep
        // a mis-sequenced call from walking past the work lists
        *ws.n_chunks = min(pre.y + total.y, ws.max_chunks);
        *ws.n_blocks = min(pre.z + total.z, ws.nbk - 1);
        *ws.n_active_prev = *ws.n_active;
        *ws.n_active = 0;
    }
    const int lane = threadIdx.x & 31;
    const int cs = ws.chunk_size;
    // a warp takes kScanPrefetch of the tile's non-empty buckets at a time and
    // loads all their cell counts before scanning any, so the loads' round
    // trips overlap instead of queueing one after another
    constexpr int kScanPrefetch = 8;
    const int warp = (int)(threadIdx.x >> 5);
    __syncthreads();
    for (int i0 = warp; i0 < nlist; i0 += kScanWarps * kScanPrefetch) {
        int lis[kScanPrefetch];
        int2 ks[kScanPrefetch];
#pragma unroll
        for (int u = 0; u < kScanPrefetch; ++u) {
            const int i = i0 + u * kScanWarps;
            lis[u] = i < nlist ? s_list[i] : -1;
            ks[u] = lis[u] >= 0 ? reinterpret_cast<const int2 *>(
                                      ws.cell_counts + (int64_t)(b0 + lis[u]) * 64)[lane]
                                : make_int2(0, 0);
        }
#pragma unroll
        for (int u = 0; u < kScanPrefetch; ++u) {
            const int li = lis[u];
            if (li < 0) break;  // uniform over the warp
            const int bk = b0 + li;
            const int bo = s_off[li], n_b = s_cnt[li];
            // cell offsets of the block: lane owns cells 2 lane, 2 lane + 1
            const int2 k = ks[u];
            const int sum = k.x + k.y;
            int incl = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            const int st = bo + incl - sum;
            const int2 st2 = make_int2(st, st + k.x);
            reinterpret_cast<int2 *>(ws.cell_start + (int64_t)bk * 64)[lane] = st2;
            reinterpret_cast<int2 *>(ws.cell_cursor + (int64_t)bk * 64)[lane] = st2;
            reinterpret_cast<int2 *>(ws.cell_counts + (int64_t)bk * 64)[lane] = make_int2(0, 0);
            if (n_b > 0) {
                const bool real = bk < ws.nbk - 1;
                const int sc = real ? scene_of_block(scenes, n_scenes, bk) : -1;  // -1: copy chunk
                const int at_b = s_boff[li];
                if (real && lane == 0 && at_b < ws.nbk - 1) ws.blocks[at_b] = make_int4(bk, bo, n_b, sc);
                const int nch = (n_b + cs - 1) / cs;
                for (int c = lane; c < nch; c += 32) {
                    const int at = s_coff[li] + c;
                    if (at < ws.max_chunks) ws.chunks[at] = make_int4(bk, bo + c * cs, min(cs, n_b - c * cs), sc);
                }
            }
        }
    }
}

// order[cell_cursor[key]++] = slot, warp-aggregated.  Each thread takes
// kScatterPer keys (strided by the grid's thread count) so that their
// cursor atomics are in flight together.  Also zeroes the grid accumulator
// of the previous substep's active blocks (kept until now so grid mass and
// momentum stay readable between substeps) and the block counts that the scan
// has read, for G2P to count into.
constexpr int kScatterPer = 4;

__global__ void __launch_bounds__(256) scatter_kernel(PState st, Ws ws, int n) {
    chain_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int stride = gridDim.x * blockDim.x;
    const int lane = threadIdx.x & 31;
    int key[kScatterPer], base[kScatterPer];
    unsigned peers[kScatterPer];
    // the keys' loads first, so their round trip overlaps the clearing below
#pragma unroll
    for (int r = 0; r < kScatterPer; ++r) {
        const int64_t idx = (int64_t)i + (int64_t)r * stride;
        key[r] = idx < n ? __ldcs(st.key + idx) : -1;
    }
    for (int j = i; j < ws.nbk; j += stride) ws.counts[j] = 0;
    const int nclear = *ws.n_active_prev * kBlockNodes;
    for (int j = i; j < nclear; j += stride)
        ws.grid_acc[(int64_t)ws.active_list[j >> 6] * kBlockNodes + (j & 63)] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int r = 0; r < kScatterPer; ++r) {
        peers[r] = __match_any_sync(0xffffffffu, key[r]);
        const int leader = __ffs(peers[r]) - 1;
        base[r] = 0;
        if (key[r] >= 0 && lane == leader) base[r] = atomicAdd(ws.cell_cursor + key[r], __popc(peers[r]));
    }
#pragma unroll
    for (int r = 0; r < kScatterPer; ++r) {
        const int leader = __ffs(peers[r]) - 1;
        const int b = __shfl_sync(0xffffffffu, base[r], leader);
        const int pos = b + __popc(peers[r] & ((1u << lane) - 1u));
        const int64_t idx = (int64_t)i + (int64_t)r * stride;
        if (key[r] >= 0 && pos < n) ws.order[pos] = (int)idx;
    }
}

cudaError_t launch_keys(const Ctx &cx) {
    if (cx.n == 0) return cudaSuccess;
    launch_chained(key_kernel, (cx.n + 255) / 256, 256, 0, cx.stream, cx.scenes, cx.n_scenes, cx.st, cx.ws, cx.n,
                   cx.status);
    return cudaGetLastError();
}

cudaError_t launch_sort(const Ctx &cx) {
    const int nbk = cx.ws.nbk;
    if (nbk <= kDirectBuckets) {
        launch_chained(scan_kernel<0, 64>, (nbk + 63) / 64, kScanThreads, 0, cx.stream, cx.scenes, cx.n_scenes,
                       cx.ws);
    } else {
        const int n_tiles = (nbk + kSumTile - 1) / kSumTile;
        launch_chained(bucket_sums_kernel, n_tiles, kScanThreads, 0, cx.stream, cx.ws);
        if (nbk > kSuperBuckets)
            launch_chained(super_sums_kernel, (n_tiles + kSuperTiles - 1) / kSuperTiles, kScanThreads, 0, cx.stream,
                           cx.ws, n_tiles);
        if (nbk <= kWideBuckets)
            launch_chained(scan_kernel<1, 64>, (nbk + 63) / 64, kScanThreads, 0, cx.stream, cx.scenes,
                           cx.n_scenes, cx.ws);
        else
            launch_chained(nbk > kSuperBuckets ? scan_kernel<2, 256> : scan_kernel<1, 256>, (nbk + 255) / 256,
                           kScanThreads, 0, cx.stream, cx.scenes, cx.n_scenes, cx.ws);
    }
    // kScatterPer keys a thread, but never fewer than two CTAs an SM: the blocks to
    // clear do not shrink with the particles (a few CTAs clearing a sparse scene's
    // 500 blocks: 34.1 us per substep of 4,096 particles on a 72^3 grid, 21.4 so;
    // 32k on 64^3 27.2 -> 25.6, 131k on 72^3 42.4 -> 41.6; four an SM the same)
    const int per = 256 * kScatterPer;
    int sgrid = (cx.n + per - 1) / per;
    if (sgrid < 2 * cx.num_sms) sgrid = 2 * cx.num_sms;
    launch_chained(scatter_kernel, sgrid, 256, 0, cx.stream, cx.st, cx.ws, cx.n);
    return cudaGetLastError();
}


}  // namespace mpm
