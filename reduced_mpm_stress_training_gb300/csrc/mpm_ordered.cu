// Ordered P2G: grid sums that do not depend on the order in which warps run.
//
// The regular P2G (p2g_kernel) is exact up to float32 rounding, but two
// things make its rounding vary from run to run: the sort's scatter places
// the particles of one cell in the order in which warps reach the cell's
// cursor, and the per-block tiles are flushed into the grid with float
// atomics from up to eight warps per node.  A finite-difference check of a
// gradient compares two forward runs whose inputs differ by 1e-3 relative;
// that needs the forward to be a deterministic function of its inputs.
// This mode removes both sources:
//   canonical_cells_kernel -- each cell's range of order[] sorted by particle
//                             uid (the user's index), so every run sums its
//                             particles in the same order
//   p2g_tiles_kernel       -- each non-empty block's 6x6x6 tile written whole
//                             to its own slot instead of atomics
//   gather_partials_kernel -- each node of an active grid block sums the
//                             <= 8 tiles that cover it in a fixed order
//                             (source block offsets (0,0,0), (0,0,1), ...,
//                             (1,1,1)) into grid_acc
// The grid update and G2P that follow are per node / per particle and
// deterministic already.  Results equal the regular P2G's up to float32
// rounding (the same terms, summed in another order).
#include "mpm_device.cuh"
#include "mpm_launch.h"

namespace mpm {

namespace {

constexpr int64_t kAlignBytes = 256;
inline int64_t align_up(int64_t x) { return (x + kAlignBytes - 1) / kAlignBytes * kAlignBytes; }

__device__ __forceinline__ int rec_uid(const PState &st, int slot) {
    return __float_as_int(ldrec(st, slot, 1).y);
}

// one thread per (work-list block, cell): insertion sort of the cell's range
// of order[] by uid.  Cells hold a handful of particles; the sort is
// quadratic in the cell's count.
__global__ void __launch_bounds__(256) canonical_cells_kernel(PState st, Ws ws) {
    chain_wait();
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int bi = (int)(t >> 6), c = (int)(t & 63);
    if (bi >= *ws.n_blocks) return;
    const int4 be = ws.blocks[bi];
    if ((unsigned)be.x >= (unsigned)(ws.nbk - 1)) return;
    const int64_t cell = (int64_t)be.x * 64 + c;
    const int s = ws.cell_start[cell], e = ws.cell_cursor[cell];
    if (s < 0 || e > ws.n || e - s < 2) return;
    int *o = ws.order;
    for (int i = s + 1; i < e; ++i) {
        const int slot = o[i];
        if ((unsigned)slot >= (unsigned)ws.n) return;  // damaged list: leave it
        const int uid = rec_uid(st, slot);
        int j = i - 1;
        while (j >= s) {
            const int sj = o[j];
            if (rec_uid(st, sj) <= uid) break;
            o[j + 1] = sj;
            --j;
        }
        o[j + 1] = slot;
    }
}

// ---------------------------------------------------------------------------
// The ordered P2G's accumulation.  One warp per non-empty grid block, with a
// warp-private 6x6x6 node tile in shared memory.  Particles of one cell share
// their 27 stencil nodes, so a lane takes a run of consecutive particles of
// one cell, sums their contributions in registers (27 nodes x 4 = 108
// accumulators) and adds them to the tile once.  A round gives each lane a run
// of the same length L from a DISTINCT cell, whose stencils hit distinct nodes
// for every node offset, so the tile updates are race-free.  The cells are
// chosen longest-remaining first (every cell with at least t particles left, t
// the smallest threshold that leaves at most 32 such cells, filled up to 32
// with cells that have t - 1 left: Hu's list schedule for chains), and L is the
// fewest particles any chosen cell has left, at most kRunMax, so no lane idles
// inside a round.  Each lane streams its run's 128-byte records into shared
// memory with cp.async one particle ahead.
//
// The unordered P2G (p2g_kernel) splits its sums over more lanes and is faster (on 1M particles
// 72 us where this form took 90).  The ordered mode keeps this order of summation: any
// fixed order gives it equal runs (of one build: the compiler decides which multiplies
// and adds are fused), but particles that yield sit on the yield surface, where the
// gradient jumps, so another rounding of the forward moves a gradient with respect to the
// friction angle by about 1e-4 of itself.
//
// Tile layout: rows of 6 nodes along z padded to 8 slots and rotated by
// 4 (y & 1), so a node's 16-byte bank group is (z + 4 (y & 1)) mod 8: the 8
// lanes of a quarter-warp (one 128-bit shared access phase) holding two
// y-adjacent rows of 4 cells hit 8 distinct bank groups for every offset.
// ---------------------------------------------------------------------------
constexpr int kRunMax = 4;     // most particles of one cell a lane takes per round
constexpr int kP2GQuads = 8;   // record quads P2G reads (q0-q7, 128 B)
constexpr int kRowSlots = 8;
constexpr int kP2GSlots = kTile * kTile * kRowSlots;

__device__ __forceinline__ int p2g_slot(int x, int y, int z) {
    return (x * kTile + y) * kRowSlots + ((z + 4 * (y & 1)) & 7);
}

struct P2GWarpSmem {
    float4 tile[kP2GSlots];
    float4 rec[2][kP2GQuads][32];  // each lane's current and next record
    int4 seg[32];                  // the round's runs: first sorted position, cell
};

struct P2GParticle {
    Weights W;
    int lx, ly, lz;
    float m;
    float a0[3];  // v - C fx dx
    float Cd[9];  // C dx
    float T[9];   // -dt vol inv_dx tau
};

__device__ __forceinline__ bool p2g_load(const MpmScene &S, const float4 (&q)[kP2GQuads], int bx, int by,
                                         int bz, float dt, P2GParticle &P) {
    // record quads 0-7: x0 m | vol .. | u v.x | v.yz C0 C1 | C2-5 | C6-8 tau0 | tau1-4 | tau5-8
    const float4 q0 = q[0], q1 = q[1], q2 = q[2], q3 = q[3], q4 = q[4], q5 = q[5], q6 = q[6], q7 = q[7];
    const float x0[3] = {q0.x, q0.y, q0.z}, u[3] = {q2.x, q2.y, q2.z};
    float gp[3];
    int base[3];
    bool ok = true;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        gp[d] = grid_coord(x0[d], u[d], S.inv_dx);
        ok &= stencil_base(gp[d], S.n_grid, base[d]);
    }
    P.lx = base[0] - 4 * bx;
    P.ly = base[1] - 4 * by;
    P.lz = base[2] - 4 * bz;
    ok &= (unsigned)P.lx < 4u && (unsigned)P.ly < 4u && (unsigned)P.lz < 4u;
    if (!ok) return false;
    make_weights(gp, base, P.W);
    P.m = q0.w;
    const float vol = q1.x;
    const float dx = S.dx;
    const float v[3] = {q2.w, q3.x, q3.y};
    const float Cm[9] = {q3.z, q3.w, q4.x, q4.y, q4.z, q4.w, q5.x, q5.y, q5.z};
    const float tau[9] = {q5.w, q6.x, q6.y, q6.z, q6.w, q7.x, q7.y, q7.z, q7.w};
    const float tscale = -vol * dt * S.inv_dx;
#pragma unroll
    for (int k = 0; k < 9; ++k) P.T[k] = tau[k] * tscale;
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        const float cf = Cm[r * 3 + 0] * P.W.fx[0] + Cm[r * 3 + 1] * P.W.fx[1] + Cm[r * 3 + 2] * P.W.fx[2];
        P.a0[r] = v[r] - cf * dx;
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) P.Cd[k] = Cm[k] * dx;
    return true;
}

// add one particle's 27 node contributions to the lane's accumulators
// (x, y packed in axy, z and mass in azw: Blackwell's two-wide FP32 FMA).
// Per (i,j) the node value factors over k:
//   add_r = wz_k A_r + k wz_k B_r + dwz_k D_r,  mass = pm wz_k
// with pm = wx_i wy_j m, A_r = pm (a0_r + i Cdx_r + j Cdy_r) + T_r0 dwx_i wy_j
// + T_r1 wx_i dwy_j, B_r = pm Cdz_r, D_r = T_r2 wx_i wy_j.
__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }

__device__ __forceinline__ void p2g_accumulate(const P2GParticle &P, float2 (&axy)[27], float2 (&azw)[27]) {
    const float2 a0 = f2(P.a0[0], P.a0[1]);
    const float2 cdx = f2(P.Cd[0], P.Cd[3]), cdy = f2(P.Cd[1], P.Cd[4]), cdz = f2(P.Cd[2], P.Cd[5]);
    const float2 t0 = f2(P.T[0], P.T[3]), t1 = f2(P.T[1], P.T[4]), t2 = f2(P.T[2], P.T[5]);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const float p1 = P.W.dw[0][i] * P.W.w[1][j];
            const float p2 = P.W.w[0][i] * P.W.dw[1][j];
            const float p3 = P.W.w[0][i] * P.W.w[1][j];
            const float pm = p3 * P.m;
            float2 aij = a0;
            if (i > 0) aij = __ffma2_rn(f2((float)i, (float)i), cdx, aij);
            if (j > 0) aij = __ffma2_rn(f2((float)j, (float)j), cdy, aij);
            const float2 A = __ffma2_rn(f2(pm, pm), aij, __ffma2_rn(t0, f2(p1, p1), __fmul2_rn(t1, f2(p2, p2))));
            const float2 B = __fmul2_rn(f2(pm, pm), cdz);
            const float2 D = __fmul2_rn(t2, f2(p3, p3));
            const float az = P.a0[2] + (float)i * P.Cd[6] + (float)j * P.Cd[7];
            const float Az = pm * az + P.T[6] * p1 + P.T[7] * p2;
            const float Bz = pm * P.Cd[8];
            const float Dz = P.T[8] * p3;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const float wz = P.W.w[2][k], dwz = P.W.dw[2][k];
                float2 &xy = axy[(i * 3 + j) * 3 + k];
                float2 &zw = azw[(i * 3 + j) * 3 + k];
                xy = __ffma2_rn(f2(wz, wz), A, xy);
                zw = __ffma2_rn(f2(wz, wz), f2(Az, pm), zw);
                xy = __ffma2_rn(f2(dwz, dwz), D, xy);
                zw.x = fmaf(dwz, Dz, zw.x);
                if (k > 0) {
                    const float kwz = k == 1 ? wz : 2.0f * wz;
                    xy = __ffma2_rn(f2(kwz, kwz), B, xy);
                    zw.x = fmaf(kwz, Bz, zw.x);
                }
            }
        }
    }
}

// add a segment's accumulated nodes into the tile (read-modify-write; the
// lanes of `mask` hold distinct cells)
__device__ __forceinline__ void p2g_flush(const float2 (&axy)[27], const float2 (&azw)[27], int lx, int ly,
                                          int lz, float4 *tile, unsigned mask) {
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                float4 *t = tile + p2g_slot(lx + i, ly + j, lz + k);
                const int n = (i * 3 + j) * 3 + k;
                float4 o = *t;
                o.x += axy[n].x;
                o.y += axy[n].y;
                o.z += azw[n].x;
                o.w += azw[n].y;
                *t = o;
                __syncwarp(mask);
            }
}

__device__ __forceinline__ void p2g_cp_async16(void *smem, const void *gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}

// queue the copy of one record (slot >= 0) into the lane's buffer b
__device__ __forceinline__ void p2g_prefetch(P2GWarpSmem &sm, const PState &st, int slot, int b, int lane, int n) {
    if (slot >= 0 && slot < n) {
#pragma unroll
        for (int q = 0; q < kP2GQuads; ++q) p2g_cp_async16(&sm.rec[b][q][lane], recq(st, slot, q));
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
}

// Choose the next round of a block: up to 32 distinct cells, longest
// remaining first, each giving its next L particles.  Lane `lane` owns cells
// lane and lane + 32 (remaining counts rem0/rem1, next positions pos0/pos1).
// Returns false when the block is done; else the lane's run (first sorted
// position, cell, length len: L or 0) and the round length L.
__device__ __forceinline__ bool p2g_next_round(int &rem0, int &rem1, int &pos0, int &pos1, int lane, unsigned lt,
                                               int4 *seg, int &start, int &cell, int &len, int &L) {
    const unsigned full = 0xffffffffu;
    const int maxrem = __reduce_max_sync(full, max(rem0, rem1));
    if (maxrem == 0) return false;
    // smallest t >= 1 with at most 32 cells holding >= t particles
    int lo = 1, hi = maxrem + 1;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        const int cnt = __popc(__ballot_sync(full, rem0 >= mid)) + __popc(__ballot_sync(full, rem1 >= mid));
        if (cnt <= 32) hi = mid;
        else lo = mid + 1;
    }
    const unsigned h0 = __ballot_sync(full, rem0 >= lo), h1 = __ballot_sync(full, rem1 >= lo);
    const int need = 32 - __popc(h0) - __popc(h1);
    const unsigned f0 = __ballot_sync(full, lo > 1 && rem0 == lo - 1);
    const unsigned f1 = __ballot_sync(full, lo > 1 && rem1 == lo - 1);
    const bool p0 = rem0 >= lo || (((f0 >> lane) & 1u) && __popc(f0 & lt) < need);
    const bool p1 = rem1 >= lo || (((f1 >> lane) & 1u) && __popc(f0) + __popc(f1 & lt) < need);
    const unsigned b0 = __ballot_sync(full, p0), b1 = __ballot_sync(full, p1);
    // every chosen cell gives its next L particles, L = the fewest any of them has left
    const unsigned least =
        __reduce_min_sync(full, min(p0 ? (unsigned)rem0 : 0xffffffffu, p1 ? (unsigned)rem1 : 0xffffffffu));
    L = min((int)least, kRunMax);
    if (p0) {
        seg[__popc(b0 & lt)] = make_int4(pos0, lane, 0, 0);
        pos0 += L;
        rem0 -= L;
    }
    if (p1) {
        seg[__popc(b0) + __popc(b1 & lt)] = make_int4(pos1, lane + 32, 0, 0);
        pos1 += L;
        rem1 -= L;
    }
    const int tot = __popc(b0) + __popc(b1);
    __syncwarp();
    const int4 mine = lane < tot ? seg[lane] : make_int4(0, 0, 0, 0);
    __syncwarp();  // seg[] is rewritten by the next call
    start = mine.x;
    cell = mine.y;
    len = lane < tot ? L : 0;
    return true;
}

// The whole 6x6x6 tile of work-list entry bi goes to partials[bi] and
// blk_index[block] = bi; the gather kernel then sums the <= 8 tiles covering
// each node in a fixed order.
__global__ void __launch_bounds__(32, 2) p2g_tiles_kernel(const MpmScene *__restrict__ scenes, int n_scenes,
                                                          PState st, Ws ws, float dt, int *status,
                                                          float4 *partials, int *blk_index) {
    chain_wait();
    __shared__ P2GWarpSmem sm;
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const int nblk = *ws.n_blocks;
    for (int bi = blockIdx.x; bi < nblk; bi += gridDim.x) {
        const int4 be = ws.blocks[bi];
        if ((unsigned)be.x >= (unsigned)(ws.nbk - 1) || (unsigned)be.w >= (unsigned)n_scenes) {
            // a damaged work list: skip, never index with it
            if (lane == 0) atomicOr(status, MPM_ST_INTERNAL);
            continue;
        }
        // by value: the compiler loads the few fields P2G uses once per block into
        // registers (measured 1 us per launch faster than reading them through a reference)
        const MpmScene S = scenes[be.w];
        int bx, by, bz;
        chunk_block(S, be.x, bx, by, bz);
        for (int i = lane; i < kP2GSlots; i += 32) sm.tile[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        // cell ranges of this block: lane owns cells lane and lane + 32
        const int64_t cb = (int64_t)be.x * 64;
        const int s0 = ws.cell_start[cb + lane], s1 = ws.cell_start[cb + lane + 32];
        const int c0 = max(0, ws.cell_cursor[cb + lane] - s0);
        const int c1 = max(0, ws.cell_cursor[cb + lane + 32] - s1);
        // Rounds are software-pipelined: while round A is summed, round B is
        // chosen and its order[] entries load, and A's last iteration already
        // streams B's first records.
        int rem0 = c0, rem1 = c1, pos0 = s0, pos1 = s1;
        int startA, cellA, lenA, LA;
        bool haveA = p2g_next_round(rem0, rem1, pos0, pos1, lane, lt, sm.seg, startA, cellA, lenA, LA);
        int slA[kRunMax];
#pragma unroll
        for (int t = 0; t < kRunMax; ++t) slA[t] = t < lenA && startA + t < ws.n ? ws.order[startA + t] : -1;
        int buf = 0;
        if (haveA) p2g_prefetch(sm, st, slA[0], 0, lane, ws.n);
        bool bad = false;
        while (haveA) {
            int startB, cellB, lenB, LB;
            const bool haveB = p2g_next_round(rem0, rem1, pos0, pos1, lane, lt, sm.seg, startB, cellB, lenB, LB);
            int slB[kRunMax];
#pragma unroll
            for (int t = 0; t < kRunMax; ++t)
                slB[t] = haveB && t < lenB && startB + t < ws.n ? ws.order[startB + t] : -1;
            const int cx = cellA >> 4, cy = (cellA >> 2) & 3, cz = cellA & 3;
            float2 axy[27], azw[27];
#pragma unroll
            for (int k = 0; k < 27; ++k) {
                axy[k] = make_float2(0.f, 0.f);
                azw[k] = make_float2(0.f, 0.f);
            }
#pragma unroll
            for (int t = 0; t < kRunMax; ++t) {
                if (t < LA) {  // warp-uniform
                    // the next record (this run's, or the next round's first) streams in
                    // while this one is summed
                    int nxt = slB[0];
#pragma unroll
                    for (int u = 0; u + 1 < kRunMax; ++u)
                        if (u == t && t + 1 < LA) nxt = slA[u + 1];
                    p2g_prefetch(sm, st, nxt, buf ^ 1, lane, ws.n);
                    asm volatile("cp.async.wait_group 1;\n" ::: "memory");
                    if (t < lenA && slA[t] < 0) {
                        bad = true;  // position or slot out of range: nothing was staged
                    } else if (t < lenA) {
                        float4 q[kP2GQuads];
#pragma unroll
                        for (int qq = 0; qq < kP2GQuads; ++qq) q[qq] = sm.rec[buf][qq][lane];
                        P2GParticle P;
                        const bool ok =
                            p2g_load(S, q, bx, by, bz, dt, P) && P.lx == cx && P.ly == cy && P.lz == cz;
                        if (ok) p2g_accumulate(P, axy, azw);
                        bad |= !ok;
                    }
                    buf ^= 1;
                }
            }
            const unsigned fm = __ballot_sync(full, lenA > 0);
            if (lenA > 0) p2g_flush(axy, azw, cx, cy, cz, sm.tile, fm);
            __syncwarp();
            haveA = haveB;
            startA = startB;
            cellA = cellB;
            lenA = lenB;
            LA = LB;
#pragma unroll
            for (int t = 0; t < kRunMax; ++t) slA[t] = slB[t];
        }
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        if (bad) atomicOr(status, MPM_ST_INTERNAL);
        const int nb = S.n_blocks_axis;
        // the whole tile to this entry's slot, in node order
        float4 *dst = partials + (int64_t)bi * kTileNodes;
        for (int i = lane; i < kTileNodes; i += 32)
            dst[i] = sm.tile[p2g_slot(i / (kTile * kTile), (i / kTile) % kTile, i % kTile)];
        if (lane == 0) blk_index[be.x] = bi;
        if (lane < 8) {
            const int gx = bx + (lane >> 2), gy = by + ((lane >> 1) & 1), gz = bz + (lane & 1);
            if (gx < nb && gy < nb && gz < nb) {
                const int gb = (int)(S.block_begin + ((int64_t)(gx * nb + gy) * nb + gz));
                if (atomicExch(ws.block_flag + gb, 1) == 0)
                    ws.active_list[atomicAdd(ws.n_active, 1)] = gb;
            }
        }
        __syncwarp();
    }
}

// one thread per node of each active grid block: grid_acc = the sum of the
// tiles of the (up to 8) non-empty blocks whose 6x6x6 tile covers the node,
// in the fixed order of the source block offsets
__global__ void __launch_bounds__(256) gather_partials_kernel(const MpmScene *__restrict__ scenes, int n_scenes,
                                                              Ws ws, const float4 *__restrict__ partials,
                                                              const int *__restrict__ blk_index) {
    chain_wait();
    const int n_active = *ws.n_active;
    const int l = threadIdx.x & 63;
    for (int base = blockIdx.x * 4; base < n_active; base += gridDim.x * 4) {
        const int li = base + (threadIdx.x >> 6);
        if (li >= n_active) continue;
        const int gb = ws.active_list[li];
        const MpmScene &S = scenes[scene_of_block(scenes, n_scenes, gb)];
        const int nb = S.n_blocks_axis;
        int bx, by, bz;
        chunk_block(S, gb, bx, by, bz);
        const int lx = l >> 4, ly = (l >> 2) & 3, lz = l & 3;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int d = 0; d < 8; ++d) {
            const int dx = d >> 2, dy = (d >> 1) & 1, dz = d & 1;
            const int sx = bx - dx, sy = by - dy, sz = bz - dz;
            const int tx = 4 * dx + lx, ty = 4 * dy + ly, tz = 4 * dz + lz;
            if (sx < 0 || sy < 0 || sz < 0 || tx >= kTile || ty >= kTile || tz >= kTile) continue;
            const int64_t sb = S.block_begin + ((int64_t)(sx * nb + sy) * nb + sz);
            const int idx = blk_index[sb];
            if (idx < 0) continue;
            const float4 p = partials[(int64_t)idx * kTileNodes + (tx * kTile + ty) * kTile + tz];
            acc.x += p.x;
            acc.y += p.y;
            acc.z += p.z;
            acc.w += p.w;
        }
        ws.grid_acc[(int64_t)gb * kBlockNodes + l] = acc;
    }
}

}  // namespace

int64_t ordered_scratch_bytes(int64_t total_blocks) {
    return align_up(total_blocks * kTileNodes * 16) + align_up(total_blocks * 4);
}

cudaError_t launch_p2g_ordered(const Ctx &cx, float dt, void *scratch) {
    float4 *partials = static_cast<float4 *>(scratch);
    int *blk_index = reinterpret_cast<int *>(static_cast<char *>(scratch) +
                                             align_up(cx.total_blocks * kTileNodes * 16));
    cudaError_t e = cudaMemsetAsync(blk_index, 0xff, (size_t)cx.total_blocks * sizeof(int), cx.stream);
    if (e != cudaSuccess) return e;
    const int64_t threads = cx.total_blocks * 64;
    if (threads > 0) {
        launch_chained(canonical_cells_kernel, (unsigned)((threads + 255) / 256), 256, 0, cx.stream, cx.st, cx.ws);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    // up to 32 single-warp CTAs per SM, several times the resident ones: the
    // rest start as others finish, which balances blocks of unequal size
    const int64_t tw = cx.total_blocks < (int64_t)cx.num_sms * 32 ? cx.total_blocks : (int64_t)cx.num_sms * 32;
    launch_chained(p2g_tiles_kernel, (unsigned)(tw > 0 ? tw : 1), 32, 0, cx.stream, cx.scenes, cx.n_scenes, cx.st,
                   cx.ws, dt, cx.status, partials, blk_index);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    int64_t want = (cx.total_blocks + 3) / 4;
    int grid = (int)(want < (int64_t)cx.num_sms * 8 ? want : (int64_t)cx.num_sms * 8);
    if (grid < 1) grid = 1;
    launch_chained(gather_partials_kernel, grid, 256, 0, cx.stream, cx.scenes, cx.n_scenes, cx.ws, partials,
                   blk_index);
    return cudaGetLastError();
}

}  // namespace mpm
