// The three transfer stages of the substep.
//
// Grid storage is block-major: the nodes of each 4x4x4 grid block are 64
// consecutive float4 (momentum xyz + mass, or velocity xyz + mass), blocks
// of all scenes concatenated.  The particles whose stencil base cells lie in
// one grid block have all their 3x3x3 stencils in the 6x6x6 node tile
// anchored at that block.
//
//   p2g  -- one CTA per non-empty block, a warp per x-slab: lanes are stencil
//           nodes, per-cell runs of particles summed in registers and added
//           to private slab tiles in shared memory, each non-zero node
//           flushed with ONE float4 atomicAdd to global memory, and the 8
//           grid blocks the tile covers registered in the active-block list.
//   grid -- one thread per node of each active block: momentum/mass +
//           gravity, colliders in registration order; clears the block
//           flag.  (The accumulator is zeroed by the next substep's
//           scatter, so grid mass and momentum stay readable meanwhile.)
//   g2p  -- one CTA per chunk (up to chunk_size sorted particles of one
//           block): stage the tile of grid velocities in shared
//           memory, gather 27 nodes per particle, APIC C, velocity
//           gradient, F update, return map + stress on one SVD, the
//           displacement update and the cell key + histograms of the next
//           substep.  Each updated record is written to the other state
//           buffer at its sorted position, so every substep leaves the
//           particle state physically sorted by cell.
#include "mpm_device.cuh"
#include "mpm_launch.h"

namespace mpm {

// ---------------------------------------------------------------------------
// P2G: p2g_apic_stress_given, engine_stress/mpm_utils.py:190-227
//   grid_v_in += (w m)(v + C dpos) + dt (-vol tau) grad w,  grid_m += w m
//
// One CTA of four warps per non-empty grid block.  The sort delivers the
// block's particles ordered by cell (x slowest), so the particles of the four
// cells-thick x-slabs are four contiguous ranges: warp w takes the slab with
// local x = w, whose stencils cover three node planes.
//
// A warp takes 32 of its particles at a time.  Each lane loads one record and
// reduces it to the 25 numbers the scatter needs, in shared memory.  Then
// three groups of nine lanes take a third of the 32 each: a group's lanes are
// the nine (x, y) node offsets of the stencil, and each lane sums its three
// z nodes (12 accumulators) over the group's consecutive particles until the
// cell changes, when it adds them to the group's own slab tile (plain
// read-modify-writes of distinct nodes, no atomics).  At the block's end the
// CTA sums the tiles that cover each node of the 6x6x6 tile and issues one
// float4 atomicAdd per non-zero node.
// ---------------------------------------------------------------------------
constexpr int kP2GWarps = 4;                  // one per x-slab of the block
constexpr int kP2GQuads = 8;                  // record quads P2G reads (q0-q7, 128 B)
constexpr int kP2GGroups = 3;                 // groups of nine lanes
constexpr int kP2GPay = 7;                    // float4 of a particle's scatter data
constexpr int kSlabPlane = kTile * kTile + 1; // nodes of a plane, padded: the rows of a stencil's
                                              // nine lanes fall on (almost) distinct bank groups
constexpr int kSlabNodes = 3 * kSlabPlane;

struct P2GSmem {
    float4 tile[kP2GWarps][kP2GGroups][kSlabNodes];
    float4 pay[kP2GWarps][kP2GPay][32];
    int used[kP2GWarps];  // the warp's slab holds particles
};

// one particle's scatter data (see p2g_add): the offsets fx and mass; v - C fx dx and
// the cell within the block; C dx; -dt vol inv_dx tau.  False: not inside this block.
__device__ __forceinline__ bool p2g_load(const MpmScene &S, const float4 (&q)[kP2GQuads], int bx, int by,
                                         int bz, float dt, float4 (&o)[kP2GPay]) {
    // record quads 0-7: x0 m | vol .. | u v.x | v.yz C0 C1 | C2-5 | C6-8 tau0 | tau1-4 | tau5-8
    const float4 q0 = q[0], q1 = q[1], q2 = q[2], q3 = q[3], q4 = q[4], q5 = q[5], q6 = q[6], q7 = q[7];
    const float x0[3] = {q0.x, q0.y, q0.z}, u[3] = {q2.x, q2.y, q2.z};
    float fx[3];
    int base[3];
    bool ok = true;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const float gp = grid_coord(x0[d], u[d], S.inv_dx);
        ok &= stencil_base(gp, S.n_grid, base[d]);
        fx[d] = __fsub_rn(gp, (float)base[d]);
    }
    const int lx = base[0] - 4 * bx, ly = base[1] - 4 * by, lz = base[2] - 4 * bz;
    ok &= (unsigned)lx < 4u && (unsigned)ly < 4u && (unsigned)lz < 4u;
    const float dx = S.dx;
    const float v[3] = {q2.w, q3.x, q3.y};
    const float Cm[9] = {q3.z, q3.w, q4.x, q4.y, q4.z, q4.w, q5.x, q5.y, q5.z};
    const float tau[9] = {q5.w, q6.x, q6.y, q6.z, q6.w, q7.x, q7.y, q7.z, q7.w};
    const float ts = -q1.x * dt * S.inv_dx;  // -vol dt / dx
    float a0[3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        const float cf = Cm[r * 3 + 0] * fx[0] + Cm[r * 3 + 1] * fx[1] + Cm[r * 3 + 2] * fx[2];
        a0[r] = v[r] - cf * dx;
    }
    o[0] = make_float4(fx[0], fx[1], fx[2], q0.w);
    o[1] = make_float4(a0[0], a0[1], a0[2], __int_as_float((lx << 4) | (ly << 2) | lz));
    o[2] = make_float4(Cm[0] * dx, Cm[3] * dx, Cm[6] * dx, Cm[8] * dx);
    o[3] = make_float4(Cm[1] * dx, Cm[4] * dx, Cm[7] * dx, tau[8] * ts);
    o[4] = make_float4(Cm[2] * dx, Cm[5] * dx, tau[0] * ts, tau[3] * ts);
    o[5] = make_float4(tau[6] * ts, tau[1] * ts, tau[4] * ts, tau[7] * ts);
    o[6] = make_float4(tau[2] * ts, tau[5] * ts, 0.0f, 0.0f);
    return ok;
}

// a lane's stencil offset (i, j): weight s (f - c)^2 + t and its derivative 2 s (f - c) per axis
struct P2GLane {
    float fi, fj, cx, sx, tx, cy, sy, ty;
};
__device__ __forceinline__ void p2g_axis(int i, float &c, float &s, float &t) {
    c = i == 0 ? 1.5f : (i == 1 ? 1.0f : 0.5f);
    s = i == 1 ? -1.0f : 0.5f;
    t = i == 1 ? 0.75f : 0.0f;
}

// add one particle's contributions to the lane's three z nodes.  Per (i, j) the
// node value factors over k:
//   add_r = wz_k (A_r + k B_r) + dwz_k D_r,  mass = wz_k pm
// with pm = wx_i wy_j m, A_r = pm (a0_r + i Cdx_r + j Cdy_r) + T_r0 dwx_i wy_j
// + T_r1 wx_i dwy_j, B_r = pm Cdz_r, D_r = T_r2 wx_i wy_j.
__device__ __forceinline__ void p2g_add(const P2GLane &L, const float4 (&o)[kP2GPay], float (&acc)[3][4]) {
    const float dxi = o[0].x - L.cx, dyj = o[0].y - L.cy;
    const float ex = L.sx * dxi, ey = L.sy * dyj;
    const float wx = fmaf(ex, dxi, L.tx), wy = fmaf(ey, dyj, L.ty);
    const float za = o[0].z - 1.5f, zb = o[0].z - 1.0f, zc = o[0].z - 0.5f;
    const float w[3] = {0.5f * za * za, fmaf(-zb, zb, 0.75f), 0.5f * zc * zc};
    const float dw[3] = {za, -2.0f * zb, zc};
    const float p1 = 2.0f * ex * wy, p2 = 2.0f * ey * wx, p3 = wx * wy, pm = p3 * o[0].w;
    const float a0[3] = {o[1].x, o[1].y, o[1].z};
    const float cdx[3] = {o[2].x, o[2].y, o[2].z}, cdy[3] = {o[3].x, o[3].y, o[3].z};
    const float cdz[3] = {o[4].x, o[4].y, o[2].w};
    const float t0[3] = {o[4].z, o[4].w, o[5].x}, t1[3] = {o[5].y, o[5].z, o[5].w};
    const float t2[3] = {o[6].x, o[6].y, o[3].w};
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        const float a = fmaf(L.fi, cdx[r], fmaf(L.fj, cdy[r], a0[r]));
        const float A0 = fmaf(pm, a, fmaf(t0[r], p1, t1[r] * p2));
        const float A1 = fmaf(pm, cdz[r], A0), A2 = fmaf(pm, cdz[r], A1);
        const float D = t2[r] * p3;
        acc[0][r] = fmaf(w[0], A0, fmaf(dw[0], D, acc[0][r]));
        acc[1][r] = fmaf(w[1], A1, fmaf(dw[1], D, acc[1][r]));
        acc[2][r] = fmaf(w[2], A2, fmaf(dw[2], D, acc[2][r]));
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) acc[k][3] = fmaf(w[k], pm, acc[k][3]);
}

// add a lane's sums of one cell (its y, z within the slab) to its three nodes of
// the group's tile and clear them.  The group's lanes write distinct nodes here,
// but an earlier flush may have been another lane's: order the group first.
__device__ __forceinline__ void p2g_flush(float4 *mytile, int cell, unsigned gmask, float (&acc)[3][4]) {
    float4 *t = mytile + (cell >> 2) * kTile + (cell & 3);
    __syncwarp(gmask);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        float4 v = t[k];
        v.x += acc[k][0];
        v.y += acc[k][1];
        v.z += acc[k][2];
        v.w += acc[k][3];
        t[k] = v;
        acc[k][0] = acc[k][1] = acc[k][2] = acc[k][3] = 0.0f;
    }
}

// NARROW: a state buffer of 16-byte alignment (see ldpair)
template <bool NARROW>
__global__ void __launch_bounds__(kP2GWarps * 32, 6) p2g_kernel(const MpmScene *__restrict__ scenes,
                                                                int n_scenes, PState st, Ws ws, float dt,
                                                                int *status) {
    chain_wait();
    extern __shared__ __align__(16) unsigned char p2g_smem_raw[];
    P2GSmem &sm = *reinterpret_cast<P2GSmem *>(p2g_smem_raw);
    const int tid = (int)threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int group = lane / 9;                    // 0-2; lanes 27-31 only load
    const int ij = lane - 9 * group;
    const int li = ij / 3, lj = ij - 3 * li;
    P2GLane L;
    L.fi = (float)li;
    L.fj = (float)lj;
    p2g_axis(li, L.cx, L.sx, L.tx);
    p2g_axis(lj, L.cy, L.sy, L.ty);
    const unsigned gmask = 0x1ffu << (9 * (group < kP2GGroups ? group : 0));
    float4 *mytile = sm.tile[warp][group < kP2GGroups ? group : 0] + li * kSlabPlane + lj * kTile;
    const int nblk = *ws.n_blocks;
    for (int bi = blockIdx.x; bi < nblk; bi += gridDim.x) {
        const int4 be = ws.blocks[bi];
        if ((unsigned)be.x >= (unsigned)(ws.nbk - 1) || (unsigned)be.w >= (unsigned)n_scenes) {
            // a damaged work list: skip, never index with it (uniform over the CTA)
            if (tid == 0) atomicOr(status, MPM_ST_INTERNAL);
            continue;
        }
        const MpmScene &S = scenes[be.w];
        int bx, by, bz;
        chunk_block(S, be.x, bx, by, bz);
        // this warp's slab: cells 16 warp .. 16 warp + 15 of the block
        const int64_t cb = (int64_t)be.x * 64 + 16 * warp;
        const int s0 = ws.cell_start[cb], s1 = ws.cell_cursor[cb + 15];
        bool bad = s0 < 0 || s1 > ws.n;
        const int end = bad ? s0 : s1;
        if (lane == 0) sm.used[warp] = end > s0;
        if (end > s0)
            for (int i = lane; i < kP2GGroups * kSlabNodes; i += 32)
                (&sm.tile[warp][0][0])[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        float acc[3][4];
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int r = 0; r < 4; ++r) acc[k][r] = 0.0f;
        int slot = s0 + lane < end ? ws.order[s0 + lane] : -1;
        for (int p0 = s0; p0 < end; p0 += 32) {
            const int cnt = min(32, end - p0);
            __syncwarp();  // the previous batch is consumed (and the tile cleared)
            if (lane < cnt) {
                float4 o[kP2GPay];
                bool ok = (unsigned)slot < (unsigned)ws.n;
                if (ok) {
                    float4 q[kP2GQuads];
#pragma unroll
                    for (int k = 0; k < kP2GQuads; k += 2) ldpair<NARROW>(st, slot, k / 2, q[k], q[k + 1]);
                    ok = p2g_load(S, q, bx, by, bz, dt, o) && (__float_as_int(o[1].w) >> 4) == warp;
                }
                if (!ok) {  // contributes zeros
                    bad = true;
#pragma unroll
                    for (int k = 0; k < kP2GPay; ++k) o[k] = make_float4(0.f, 0.f, 0.f, 0.f);
                }
#pragma unroll
                for (int k = 0; k < kP2GPay; ++k) sm.pay[warp][k][lane] = o[k];
            }
            const int pn = p0 + 32 + lane;
            slot = pn < end ? ws.order[pn] : -1;  // the next batch's, while this one is summed
            __syncwarp();
            const int per = (cnt + kP2GGroups - 1) / kP2GGroups;
            const int first = group * per, last = group < kP2GGroups ? min(cnt, first + per) : 0;
            int cur = -1;  // the cell being summed
            for (int p = first; p < last; ++p) {
                float4 o[kP2GPay];
#pragma unroll
                for (int k = 0; k < kP2GPay; ++k) o[k] = sm.pay[warp][k][p];
                const int cell = __float_as_int(o[1].w) & 15;  // y, z within the slab
                if (cell != cur && cur >= 0) p2g_flush(mytile, cur, gmask, acc);
                cur = cell;
                p2g_add(L, o, acc);
            }
            if (cur >= 0) p2g_flush(mytile, cur, gmask, acc);
        }
        if (bad) atomicOr(status, MPM_ST_INTERNAL);
        __syncthreads();
        // the block's 6x6x6 tile: node plane x is covered by the slabs x - 2 .. x
        const int nb = S.n_blocks_axis;
        for (int i = tid; i < kTileNodes; i += kP2GWarps * 32) {
            const int tx = i / (kTile * kTile), yz = i - tx * (kTile * kTile);
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const int w = tx - d;
                if (w < 0 || w >= kP2GWarps || !sm.used[w]) continue;
#pragma unroll
                for (int g = 0; g < kP2GGroups; ++g) {
                    const float4 v = sm.tile[w][g][d * kSlabPlane + yz];
                    a.x += v.x;
                    a.y += v.y;
                    a.z += v.z;
                    a.w += v.w;
                }
            }
            if (a.x != 0.0f || a.y != 0.0f || a.z != 0.0f || a.w != 0.0f) {
                const int ix = 4 * bx + tx, iy = 4 * by + yz / kTile, iz = 4 * bz + yz % kTile;
                if (ix < S.n_grid && iy < S.n_grid && iz < S.n_grid)
                    atomicAdd(ws.grid_acc + node_addr(S.block_begin, nb, ix, iy, iz), a);
            }
        }
        if (tid < 8) {
            const int gx = bx + (tid >> 2), gy = by + ((tid >> 1) & 1), gz = bz + (tid & 1);
            if (gx < nb && gy < nb && gz < nb) {
                const int gb = (int)(S.block_begin + ((int64_t)(gx * nb + gy) * nb + gz));
                if (atomicExch(ws.block_flag + gb, 1) == 0)
                    ws.active_list[atomicAdd(ws.n_active, 1)] = gb;
            }
        }
        __syncthreads();  // the tiles are read: the next block may clear them
    }
}

// The reference's modify_bc callbacks (:561-565, :594-603, :690-693,
// :716-718): after an active substep's grid update, a moving collider's point
// advances by dt times its velocity (the circling column's velocity from its
// current angle), summed in double and stored in float as the host-side
// update does.  One thread per collider slot.
__global__ void advance_colliders_kernel(MpmScene *__restrict__ scenes, int n_scenes, float time, float dt) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_scenes * MPM_MAX_COLLIDERS) return;
    MpmScene &S = scenes[i / MPM_MAX_COLLIDERS];
    const int k = i % MPM_MAX_COLLIDERS;
    if (k >= S.n_colliders) return;
    MpmCollider &cl = S.colliders[k];
    if (!(time >= cl.start_time && time < cl.end_time)) return;
    float vel[3];
    if (cl.kind == MPM_COLLIDER_VPLANE || cl.kind == MPM_COLLIDER_CUBE || cl.kind == MPM_COLLIDER_SPHERE) {
        vel[0] = cl.velocity[0];
        vel[1] = cl.velocity[1];
        vel[2] = cl.velocity[2];
    } else if (cl.kind == MPM_COLLIDER_CIRCLE) {
        const float th = circle_theta(cl.point);
        vel[0] = -cl.v_scale * sinf(th);
        vel[1] = 0.0f;
        vel[2] = cl.v_scale * cosf(th);
    } else {
        return;
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) cl.point[d] = (float)((double)cl.point[d] + (double)dt * (double)vel[d]);
}

// ---------------------------------------------------------------------------
// Grid update: grid_normalization_and_gravity (engine_stress/mpm_utils.py:229-237)
// then the colliders of engine_stress/mpm_solver_warp.py:429-449 and :505-523.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) grid_kernel(const MpmScene *__restrict__ scenes,
                                                   int n_scenes, Ws ws, float time, float dt) {
    chain_wait();
    const int n_active = *ws.n_active;
    const int l = threadIdx.x & 63;
    for (int base = blockIdx.x * 4; base < n_active; base += gridDim.x * 4) {
        const int li = base + (threadIdx.x >> 6);
        if (li >= n_active) continue;
        const int gb = ws.active_list[li];
        const MpmScene &S = scenes[scene_of_block(scenes, n_scenes, gb)];
        int bx, by, bz;
        chunk_block(S, gb, bx, by, bz);
        const int ix = 4 * bx + (l >> 4), iy = 4 * by + ((l >> 2) & 3), iz = 4 * bz + (l & 3);
        const int64_t a = (int64_t)gb * kBlockNodes + l;
        const float4 acc = ws.grid_acc[a];
        float v[3] = {0.f, 0.f, 0.f};
        if (acc.w > 1e-15f) {
            const float inv = 1.0f / acc.w;
            v[0] = __fadd_rn(__fmul_rn(acc.x, inv), __fmul_rn(dt, S.gravity[0]));
            v[1] = __fadd_rn(__fmul_rn(acc.y, inv), __fmul_rn(dt, S.gravity[1]));
            v[2] = __fadd_rn(__fmul_rn(acc.z, inv), __fmul_rn(dt, S.gravity[2]));
        }
        for (int k = 0; k < S.n_colliders; ++k) apply_collider(S.colliders[k], S, ix, iy, iz, time, dt, v);
        ws.grid_v[a] = make_float4(v[0], v[1], v[2], acc.w);
        if (l == 0) ws.block_flag[gb] = 0;
    }
}

// ---------------------------------------------------------------------------
// G2P: g2p_apic_and_stress (engine_stress/mpm_utils.py:241-306) fused with
// update_x_from_u / update_u_from_x (:4-15) and the next substep's key.
// Reads records from `st` through order[], writes them to `out` at the
// sorted position.  Chunks with scene -1 hold out-of-domain particles,
// which are carried over unchanged.
//
// Software-pipelined over the CTA's chunks: while chunk k is computed, the
// particle records (quads 0,1,2,8,9) and the 6x6x6 grid-velocity tile of
// chunk k+1 stream into the other half of a double buffer in shared memory
// with cp.async, and the order[] indices of chunk k+2 are loaded.  Each lane
// writes its updated record straight to its sorted position, a quad pair per
// 32-byte store (consecutive lanes, consecutive addresses).  Staging the
// records in shared memory for stores of whole 64-byte pieces took 22 KB of
// shared memory per CTA and 96 us per launch on the 1M column; this takes 86
// us, and 80 us at five CTAs per SM.  It is bound by latency at 20 warps per
// SM (57 % of the issue slots, 34 % of DRAM bandwidth).
// ---------------------------------------------------------------------------
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem, int src_bytes) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(src_bytes)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait0() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// three velocity components: x, y as a pair for the two-wide FP32 FMA, z alone
struct V3 {
    float2 xy;
    float z;
};
__device__ __forceinline__ V3 v3zero() { return {make_float2(0.0f, 0.0f), 0.0f}; }
__device__ __forceinline__ V3 v3of(const float4 &g) { return {make_float2(g.x, g.y), g.z}; }
__device__ __forceinline__ V3 v3mul(float a, const V3 &x) { return {__fmul2_rn(make_float2(a, a), x.xy), a * x.z}; }
__device__ __forceinline__ V3 v3fma(float a, const V3 &x, const V3 &acc) {
    return {__ffma2_rn(make_float2(a, a), x.xy, acc.xy), fmaf(a, x.z, acc.z)};
}

constexpr int kG2PQuads = 5;  // record quads G2P reads: 0, 1, 2, 8, 9
__device__ __forceinline__ int g2p_quad(int q) { return q < 3 ? q : q + 5; }

template <int CH>
struct G2PSmem {
    float4 tile[2][kTileNodes];
    float4 rec[2][kG2PQuads][CH];
};

// a chunk's records (lanes of the chunk) into half b of the buffer
template <int CH>
__device__ __forceinline__ void g2p_prefetch_records(const PState &st, const Ws &ws, const int4 &ch, int slot,
                                                     G2PSmem<CH> &sm, int b) {
    if ((int)threadIdx.x < ch.z && ch.y + (int)threadIdx.x < ws.n) {
#pragma unroll
        for (int q = 0; q < kG2PQuads; ++q)
            cp_async16(&sm.rec[b][q][threadIdx.x], recq(st, slot, g2p_quad(q)), 16);
    }
}

// queue the async copies of one chunk into buffer b
template <int CH>
__device__ __forceinline__ void g2p_prefetch(const MpmScene *__restrict__ scenes, const PState &st,
                                             const Ws &ws, const int4 &ch, int slot,
                                             G2PSmem<CH> &sm, int b) {
    if (ch.w < 0) return;  // copy chunk: no compute, nothing to stage
    g2p_prefetch_records<CH>(st, ws, ch, slot, sm, b);
    const MpmScene &S = scenes[ch.w];
    int bx, by, bz;
    chunk_block(S, ch.x, bx, by, bz);
    const int nb = S.n_blocks_axis;
    for (int i = threadIdx.x; i < kTileNodes; i += CH) {
        const int tx = i / 36, ty = (i / 6) % 6, tz = i % 6;
        const int ix = 4 * bx + tx, iy = 4 * by + ty, iz = 4 * bz + tz;
        const bool in = ix < S.n_grid && iy < S.n_grid && iz < S.n_grid;
        const float4 *src = ws.grid_v + (in ? node_addr(S.block_begin, nb, ix, iy, iz) : 0);
        cp_async16(&sm.tile[b][i], src, in ? 16 : 0);  // outside the grid: zero fill
    }
}

// The same copies with less integer work per chunk: the thread's tile nodes are
// decoded once per CTA (x | y << 3 | z << 6 each), the node address comes from
// the block id, and the chunk's block coordinates (x | y << 10 | z << 20; at most
// 1024 blocks an axis) are handed to the chunk's compute.
template <int CH>
constexpr int kG2PTileIters = (kTileNodes + CH - 1) / CH;
template <int CH>
__device__ __forceinline__ void g2p_prefetch_fast(const MpmScene *__restrict__ scenes, const PState &st, const Ws &ws,
                                                  const int4 &ch, int slot, const int (&tn)[kG2PTileIters<CH>],
                                                  G2PSmem<CH> &sm, int b, int &blk) {
    if (ch.w < 0) return;  // copy chunk: no compute, nothing to stage
    g2p_prefetch_records<CH>(st, ws, ch, slot, sm, b);
    const MpmScene &S = scenes[ch.w];
    int bx, by, bz;
    chunk_block(S, ch.x, bx, by, bz);
    blk = bx | (by << 10) | (bz << 20);
    const int nb = S.n_blocks_axis;
    const int mx = S.n_grid - 4 * bx, my = S.n_grid - 4 * by, mz = S.n_grid - 4 * bz;
#pragma unroll
    for (int k = 0; k < kG2PTileIters<CH>; ++k) {
        const int i = (int)threadIdx.x + k * CH;
        if (i >= kTileNodes) break;
        const int tx = tn[k] & 7, ty = (tn[k] >> 3) & 7, tz = tn[k] >> 6;
        const bool in = tx < mx && ty < my && tz < mz;
        const int gb = ch.x + ((tx >> 2) * nb + (ty >> 2)) * nb + (tz >> 2);
        const int l = ((tx & 3) << 4) | ((ty & 3) << 2) | (tz & 3);
        const float4 *src = ws.grid_v + (in ? (int64_t)gb * kBlockNodes + l : 0);
        cp_async16(&sm.tile[b][i], src, in ? 16 : 0);  // outside the grid: zero fill
    }
}

__device__ __forceinline__ int g2p_slot(const Ws &ws, const int4 &ch) {
    const int pos = ch.y + (int)threadIdx.x;
    return ((int)threadIdx.x < ch.z && pos < ws.n) ? ws.order[pos] : 0;
}

// DEFER: leave the return map and stress to a later pass (the surrogate stress
// stage): F_trial is stored as F and the stress words are zeroed.
// NARROW: `out` is a buffer of 16-byte alignment (see ldpair).
// FAST: the form that mpm_p2g2p runs (on buffers that take 32-byte accesses), with five
// 128-thread CTAs per SM (96 registers) instead of four and less integer work.  The mpm_g2p
// stage and the ordered mode run the other form: ptxas fuses multiplies and adds
// differently under another register budget, and the ordered mode keeps its roundings
// (see mpm_ordered.cu).
template <int CH, bool DEFER, bool FAST, bool NARROW>
__global__ void __launch_bounds__(CH, FAST ? 640 / CH : 0) g2p_kernel(const MpmScene *__restrict__ scenes, PState st,
                                                 PState out, Ws ws, float dt, int *status) {
    chain_wait();
    extern __shared__ __align__(16) unsigned char g2p_smem_raw[];
    G2PSmem<CH> &sm = *reinterpret_cast<G2PSmem<CH> *>(g2p_smem_raw);
    const int n_chunks = *ws.n_chunks;
    // The chunk list is walked from its end.  P2G has just streamed the records
    // in ascending block order, so the highest positions are the ones still in
    // L2; and the records written last here (the lowest positions) are the
    // first that the next substep's P2G reads.  Measured 207.2 -> 203.7 us per
    // substep on the 1M column against walking it from the start.
    const int sentinel = (ws.nbk - 1) * 64;  // out-of-domain cell key
    int c = blockIdx.x;
    if (c >= n_chunks) return;
    int4 ch = ws.chunks[n_chunks - 1 - c];
    int slot = g2p_slot(ws, ch);
    [[maybe_unused]] int tn[kG2PTileIters<CH>];
    [[maybe_unused]] int blk = 0, blkn = 0;
    if constexpr (FAST) {
#pragma unroll
        for (int k = 0; k < kG2PTileIters<CH>; ++k) {
            const int i = (int)threadIdx.x + k * CH;
            tn[k] = i / 36 | ((i / 6) % 6) << 3 | (i % 6) << 6;
        }
        g2p_prefetch_fast<CH>(scenes, st, ws, ch, slot, tn, sm, 0, blk);
    } else {
        g2p_prefetch<CH>(scenes, st, ws, ch, slot, sm, 0);
    }
    cp_async_commit();
    int cn = c + gridDim.x;
    int4 chn = make_int4(0, 0, 0, -1);
    int slotn = 0;
    if (cn < n_chunks) {
        chn = ws.chunks[n_chunks - 1 - cn];
        slotn = g2p_slot(ws, chn);
    }
    int buf = 0;
    while (c < n_chunks) {
        // order[] indices two chunks ahead
        const int cnn = cn + gridDim.x;
        int4 chnn = make_int4(0, 0, 0, -1);
        int slotnn = 0;
        if (cnn < n_chunks) {
            chnn = ws.chunks[n_chunks - 1 - cnn];
            slotnn = g2p_slot(ws, chnn);
        }
        // this chunk's records and tile have landed, for every thread; and every
        // warp is done with the other half of the buffer (the previous chunk),
        // so the next chunk's copies may go there now -- the only CTA-wide
        // barrier of the iteration
        cp_async_wait0();
        __syncthreads();
        if constexpr (FAST) {
            if (cn < n_chunks) g2p_prefetch_fast<CH>(scenes, st, ws, chn, slotn, tn, sm, buf ^ 1, blkn);
        } else {
            if (cn < n_chunks) g2p_prefetch<CH>(scenes, st, ws, chn, slotn, sm, buf ^ 1);
        }
        cp_async_commit();

        const int pos = ch.y + (int)threadIdx.x;
        const bool mine = (int)threadIdx.x < ch.z && pos < ws.n;
        int key = -1;
        if (ch.w < 0) {  // out-of-domain particles: carry the records over (uniform per CTA)
            if (mine) {
#pragma unroll
                for (int q = 0; q < kRecQuads; ++q) strec(out, pos, q, ldrec(st, slot, q));
                key = st.key[slot];  // counted again below: the next sort keeps their copy chunk
                out.key[pos] = key;
            }
        } else if (mine) {
            const MpmScene &S = scenes[ch.w];
            int bx, by, bz;
            if constexpr (FAST) {
                bx = blk & 1023;
                by = (blk >> 10) & 1023;
                bz = blk >> 20;
            } else {
                chunk_block(S, ch.x, bx, by, bz);
            }
            const float4 *tile = sm.tile[buf];
            const float4 q0 = sm.rec[buf][0][threadIdx.x], q1 = sm.rec[buf][1][threadIdx.x],
                         q2 = sm.rec[buf][2][threadIdx.x], q8 = sm.rec[buf][3][threadIdx.x],
                         q9 = sm.rec[buf][4][threadIdx.x];
            const float x0[3] = {q0.x, q0.y, q0.z};
            const float xo[3] = {__fadd_rn(q0.x, q2.x), __fadd_rn(q0.y, q2.y), __fadd_rn(q0.z, q2.z)};
            const float Fp[9] = {q8.x, q8.y, q8.z, q8.w, q9.x, q9.y, q9.z, q9.w, q1.w};
            float gp[3];
            int base[3];
            bool ok = true;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                gp[d] = __fmul_rn(xo[d], S.inv_dx);
                ok &= stencil_base(gp[d], S.n_grid, base[d]);
            }
            const int lx = base[0] - 4 * bx, ly = base[1] - 4 * by, lz = base[2] - 4 * bz;
            ok &= (unsigned)lx < 4u && (unsigned)ly < 4u && (unsigned)lz < 4u;
            if (!ok) {
                atomicOr(status, MPM_ST_INTERNAL);
                key = sentinel;
#pragma unroll
                for (int q = 0; q < kRecQuads; ++q) strec(out, pos, q, ldrec(st, slot, q));
                out.key[pos] = key;
            } else {
                Weights W;
                make_weights(gp, base, W);
                const float inv_dx = S.inv_dx;
                // Separable gather (same sums as :261-273, regrouped by axis):
                //   nv  = sum_ijk wx_i wy_j wz_k g
                //   nF  = sum g (x) (dwx wy wz, wx dwy wz, wx wy dwz)   (times inv_dx)
                //   M_c = sum (w g) * (ijk)_c,  C = 4 inv_dx (M - nv (x) fx)
                // z first (S, D, K per (i,j)), then y, then x.  Velocity
                // components x, y ride together in Blackwell's two-wide FP32
                // FMA (a V3 is (xy pair, z)); nF and M are kept by column.
                V3 nvp = v3zero(), nF0 = v3zero(), nF1 = v3zero(), nF2 = v3zero();
                V3 M0 = v3zero(), M1 = v3zero(), M2 = v3zero();
                const float wz0 = W.w[2][0], wz1 = W.w[2][1], wz2 = W.w[2][2];
                const float dz0 = W.dw[2][0], dz1 = W.dw[2][1], dz2 = W.dw[2][2];
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    V3 Ti = v3zero(), Ui = v3zero(), Ri = v3zero(), Ji = v3zero(), Ki = v3zero();
#pragma unroll
                    for (int j = 0; j < 3; ++j) {
                        const float4 *row = tile + ((lx + i) * kTile + (ly + j)) * kTile + lz;
                        const V3 g0 = v3of(row[0]), g1 = v3of(row[1]), g2 = v3of(row[2]);
                        const V3 Sz = v3fma(wz2, g2, v3fma(wz1, g1, v3mul(wz0, g0)));
                        const V3 Dz = v3fma(dz2, g2, v3fma(dz1, g1, v3mul(dz0, g0)));
                        const V3 Kz = v3fma(2.0f * wz2, g2, v3mul(wz1, g1));
                        const float wy = W.w[1][j], dwy = W.dw[1][j];
                        Ti = v3fma(wy, Sz, Ti);
                        Ui = v3fma(dwy, Sz, Ui);
                        Ri = v3fma(wy, Dz, Ri);
                        Ki = v3fma(wy, Kz, Ki);
                        if (j > 0) Ji = v3fma((float)j * wy, Sz, Ji);
                    }
                    const float wx = W.w[0][i], dwx = W.dw[0][i];
                    nvp = v3fma(wx, Ti, nvp);
                    nF0 = v3fma(dwx, Ti, nF0);
                    nF1 = v3fma(wx, Ui, nF1);
                    nF2 = v3fma(wx, Ri, nF2);
                    if (i > 0) M0 = v3fma((float)i * wx, Ti, M0);
                    M1 = v3fma(wx, Ji, M1);
                    M2 = v3fma(wx, Ki, M2);
                }
                const float nv[3] = {nvp.xy.x, nvp.xy.y, nvp.z};
                float nF[9] = {nF0.xy.x, nF1.xy.x, nF2.xy.x, nF0.xy.y, nF1.xy.y, nF2.xy.y, nF0.z, nF1.z, nF2.z};
                const float M[9] = {M0.xy.x, M1.xy.x, M2.xy.x, M0.xy.y, M1.xy.y, M2.xy.y, M0.z, M1.z, M2.z};
                float nC[9];
                const float c4 = 4.0f * inv_dx;
#pragma unroll
                for (int r = 0; r < 3; ++r)
#pragma unroll
                    for (int q = 0; q < 3; ++q) nC[r * 3 + q] = c4 * (M[r * 3 + q] - nv[r] * W.fx[q]);
#pragma unroll
                for (int k = 0; k < 9; ++k) nF[k] *= inv_dx;
                // x += dt v (:277), u = x - x0 (:12-15)
                float un[3];
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    const float xn = __fadd_rn(xo[d], __fmul_rn(dt, nv[d]));
                    un[d] = __fsub_rn(xn, x0[d]);
                }
                // F_trial = (I + dt grad v) F (:281)
                float A[9], Ft[9];
#pragma unroll
                for (int k = 0; k < 9; ++k) A[k] = ((k % 4 == 0) ? 1.0f : 0.0f) + nF[k] * dt;
#pragma unroll
                for (int r = 0; r < 3; ++r)
#pragma unroll
                    for (int q = 0; q < 3; ++q)
                        Ft[r * 3 + q] = A[r * 3 + 0] * Fp[0 * 3 + q] + A[r * 3 + 1] * Fp[1 * 3 + q] +
                                        A[r * 3 + 2] * Fp[2 * 3 + q];
                float yld = (S.material == MPM_METAL) ? q1.z : 0.0f;
                float Fo[9], tau[9];
                if (DEFER) {
#pragma unroll
                    for (int k = 0; k < 9; ++k) {
                        Fo[k] = Ft[k];
                        tau[k] = 0.0f;
                    }
                } else {
                    return_map_stress(S, Ft, yld, Fo, tau);
                }
                // stores: the whole record at its sorted position
                float chk = 0.0f;
#pragma unroll
                for (int k = 0; k < 9; ++k) chk += fabsf(Fo[k]) + fabsf(tau[k]);
                if (!(S.material == MPM_METAL && S.hardening == 1)) yld = q1.z;
                stpair<NARROW>(out, pos, 0, q0, make_float4(q1.x, q1.y, yld, Fo[8]));
                stpair<NARROW>(out, pos, 1, make_float4(un[0], un[1], un[2], nv[0]),
                       make_float4(nv[1], nv[2], nC[0], nC[1]));
                stpair<NARROW>(out, pos, 2, make_float4(nC[2], nC[3], nC[4], nC[5]),
                       make_float4(nC[6], nC[7], nC[8], tau[0]));
                stpair<NARROW>(out, pos, 3, make_float4(tau[1], tau[2], tau[3], tau[4]),
                       make_float4(tau[5], tau[6], tau[7], tau[8]));
                stpair<NARROW>(out, pos, 4, make_float4(Fo[0], Fo[1], Fo[2], Fo[3]),
                       make_float4(Fo[4], Fo[5], Fo[6], Fo[7]));
                int flags = 0;
                const float vmax = S.dx / dt;
                if (fabsf(nv[0]) > vmax || fabsf(nv[1]) > vmax || fabsf(nv[2]) > vmax) flags |= MPM_ST_CFL;
                if (!isfinite(chk)) flags |= MPM_ST_NONFINITE;
                bool kok;
                key = particle_key(S, x0[0], x0[1], x0[2], un[0], un[1], un[2], ws.nbk - 1, kok);
                if (!kok) flags |= MPM_ST_OUT_OF_DOMAIN;
                if (flags) atomicOr(status, flags);
                out.key[pos] = key;
            }
        }
        if constexpr (FAST) {
            sorted_histogram(ws.counts, ws.cell_counts, key, ch.x);
            blk = blkn;
        } else {
            warp_histogram(ws.counts, ws.cell_counts, key);
        }
        c = cn; ch = chn; slot = slotn;
        cn = cnn; chn = chnn; slotn = slotnn;
        buf ^= 1;
    }
    cp_async_wait0();
}

static int persistent_grid(const Ctx &cx, int per_sm) {
    int g = cx.num_sms * per_sm;
    return g < cx.ws.max_chunks ? g : (cx.ws.max_chunks > 0 ? cx.ws.max_chunks : 1);
}

// One wave of persistent CTAs: as many as fit on the GPU at once (the
// occupancy of this instance, looked up once per device).  A second wave
// would start only as the first one exits, so the first wave's chunks would
// spread over the whole list instead of sweeping it as one band, and the L2
// reuse with P2G (the chunk list walked from its end) would fall: 200.2 ->
// 198.8 us per substep on the 1M column against twice the resident count.
template <int CH, bool DEFER, bool FAST, bool NARROW>
static cudaError_t g2p_t(const Ctx &cx, float dt) {
    // more than the 48 KB of static shared memory: opt in once per instance and device
    static int resident[64] = {0};
    const int bytes = (int)sizeof(G2PSmem<CH>);
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    const auto kernel = g2p_kernel<CH, DEFER, FAST, NARROW>;
    if (resident[dev] == 0) {
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (e != cudaSuccess) return e;
        int nb = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel, CH, bytes);
        if (e != cudaSuccess) return e;
        resident[dev] = nb > 0 ? nb : 1;
    }
    const int grid = persistent_grid(cx, resident[dev]);
    launch_chained(kernel, grid, CH, bytes, cx.stream, cx.scenes, cx.st, cx.st2, cx.ws, dt, cx.status);
    return cudaGetLastError();
}

cudaError_t launch_p2g(const Ctx &cx, float dt) {
    const int bytes = (int)sizeof(P2GSmem);
    static_assert(sizeof(P2GSmem) <= 48 * 1024, "static shared-memory limit");
    // up to 24 CTAs per SM, several times the resident ones: the rest start as
    // others finish, which balances blocks of unequal size; CTAs loop over
    // blocks when there are more blocks than CTAs
    int grid = (int)(cx.total_blocks < (int64_t)cx.num_sms * 24 ? cx.total_blocks : (int64_t)cx.num_sms * 24);
    if (grid < 1) grid = 1;
    launch_chained(cx.st.wide ? p2g_kernel<false> : p2g_kernel<true>, grid, kP2GWarps * 32, bytes, cx.stream, cx.scenes,
                   cx.n_scenes, cx.st, cx.ws, dt, cx.status);
    return cudaGetLastError();
}

cudaError_t launch_grid(const Ctx &cx, float time, float dt) {
    int64_t want = (cx.total_blocks + 3) / 4;
    int grid = (int)(want < (int64_t)cx.num_sms * 8 ? want : (int64_t)cx.num_sms * 8);
    if (grid < 1) grid = 1;
    launch_chained(grid_kernel, grid, 256, 0, cx.stream, cx.scenes, cx.n_scenes, cx.ws, time, dt);
    return cudaGetLastError();
}

cudaError_t launch_advance_colliders(MpmScene *scenes, int n_scenes, float time, float dt, cudaStream_t stream) {
    const int slots = n_scenes * MPM_MAX_COLLIDERS;
    if (slots <= 0) return cudaSuccess;
    advance_colliders_kernel<<<(slots + 127) / 128, 128, 0, stream>>>(scenes, n_scenes, time, dt);
    return cudaGetLastError();
}

template <bool DEFER, bool FAST, bool NARROW>
static cudaError_t g2p_sized(const Ctx &cx, float dt) {
    switch (cx.ws.chunk_size) {
        case 32: return g2p_t<32, DEFER, FAST, NARROW>(cx, dt);
        case 64: return g2p_t<64, DEFER, FAST, NARROW>(cx, dt);
        case 128: return g2p_t<128, DEFER, FAST, NARROW>(cx, dt);
        case 256: return g2p_t<256, DEFER, FAST, NARROW>(cx, dt);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_g2p(const Ctx &cx, float dt, G2PForm form) {
    if (!cx.st2.wide)  // one form for each result
        return form == G2PForm::kDeferStress ? g2p_sized<true, false, true>(cx, dt)
                                             : g2p_sized<false, false, true>(cx, dt);
    switch (form) {
        case G2PForm::kFast: return g2p_sized<false, true, false>(cx, dt);
        case G2PForm::kDeferStress: return g2p_sized<true, true, false>(cx, dt);
        default: return g2p_sized<false, false, false>(cx, dt);
    }
}

}  // namespace mpm
