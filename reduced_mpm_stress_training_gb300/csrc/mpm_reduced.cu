// Reduced sampled-quadrature substep: MPM_Simulator_WARP.p2g2p_reduced
// (engine_stress/mpm_solver_warp.py:214-227), experiment_for_C (:207-209)
// and the sample-point gather g2p_sample (engine_stress/mpm_utils.py:415-471).
//
// The product of this path is the reference's dense (n, n, n) grid itself,
// so it keeps that layout (C-order, vec3 AoS) for grid_m / grid_v_in /
// grid_v_out and the two int32 mark arrays.  Momentum and mass are
// accumulated with one 16-byte vector atomic per node into a float4 scratch
// grid (the reference issues seven scalar atomics per node), and a single
// sweep then normalizes, applies gravity and every collider, and writes the
// three reference-layout grids.  Particles are read from the cell-sorted
// state records; the user-order side arrays (F_disp, density) and the
// sample list are indexed through the particle's uid.
#include "mpm_launch.h"

namespace mpm {

namespace {

__device__ __forceinline__ int64_t dense_index(int n, int ix, int iy, int iz) {
    return ((int64_t)ix * n + iy) * n + iz;
}

// grid position of a particle record: x = x_initial + u, gp = x * inv_dx
__device__ __forceinline__ void record_gp(const PState &st, int slot, float inv_dx, float gp[3]) {
    const float4 q0 = ldrec(st, slot, 0), q2 = ldrec(st, slot, 2);
    gp[0] = grid_coord(q0.x, q2.x, inv_dx);
    gp[1] = grid_coord(q0.y, q2.y, inv_dx);
    gp[2] = grid_coord(q0.z, q2.z, inv_dx);
}

// kirchoff_stress_FCR (mpm_utils.py:29-34): 2 mu (F - R) F^T + lam J (J - 1) I, R = U V^T
__device__ __forceinline__ void stress_fcr(const float F[9], const Svd &d, float J, float mu, float lam,
                                           float tau[9]) {
    const float one[3] = {1.f, 1.f, 1.f};
    float R[9], D[9];
    udwt(d.U, one, d.V, R);
    const float tm = 2.0f * mu;
#pragma unroll
    for (int i = 0; i < 9; ++i) D[i] = tm * (F[i] - R[i]);
    const float dia = lam * J * (J - 1.0f);
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c)
            tau[r * 3 + c] = D[r * 3 + 0] * F[c * 3 + 0] + D[r * 3 + 1] * F[c * 3 + 1] + D[r * 3 + 2] * F[c * 3 + 2] +
                             (r == c ? dia : 0.0f);
}

// kirchoff_stress_drucker_prager (mpm_utils.py:45-52): U diag(c) V^T F^T with
// c_i = (2 mu ln s_i + lam sum ln s) / s_i, logarithms unclamped
__device__ __forceinline__ void stress_dp(const float F[9], const Svd &d, float mu, float lam, float tau[9]) {
    const float l0 = logf(d.s[0]), l1 = logf(d.s[1]), l2 = logf(d.s[2]);
    const float ls = l0 + l1 + l2;
    const float tm = 2.0f * mu;
    const float c[3] = {tm * l0 * (1.0f / d.s[0]) + lam * ls * (1.0f / d.s[0]),
                        tm * l1 * (1.0f / d.s[1]) + lam * ls * (1.0f / d.s[1]),
                        tm * l2 * (1.0f / d.s[2]) + lam * ls * (1.0f / d.s[2])};
    float T[9];
    udwt(d.U, c, d.V, T);
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int k = 0; k < 3; ++k)
            tau[r * 3 + k] = T[r * 3 + 0] * F[k * 3 + 0] + T[r * 3 + 1] * F[k * 3 + 1] + T[r * 3 + 2] * F[k * 3 + 2];
}

// the reduced kernels serve single-scene plans whose dense grid matches the scene
__device__ __forceinline__ bool grid_matches(const MpmScene &S, const MpmReducedGrid &g, int *status) {
    if (S.n_grid == g.n_grid) return true;
    if (threadIdx.x == 0) atomicOr(status, MPM_ST_BAD_INPUT);
    return false;
}

}  // namespace

// update_neighboring_cells (mpm_utils.py:318-335, offsets -2..2, HI = 2) and
// update_neighboring_cells_for_grid_v (:338-351, offsets -2..4, HI = 4): one
// warp per sample point, its lanes over the (HI + 3)^3 offsets; cells
// outside the grid are not marked, as there.
template <int HI>
__global__ void __launch_bounds__(256) mark_kernel(const MpmScene *__restrict__ scenes, PState st,
                                                   const int *__restrict__ slot_of_uid, MpmReducedGrid g,
                                                   int32_t *__restrict__ mask, int n, int *status) {
    chain_wait();
    const MpmScene &S = scenes[0];
    if (!grid_matches(S, g, status)) return;
    const int64_t s = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (s >= g.n_samples) return;
    const int p = g.sample_index[s];
    if (p < 0 || p >= n) {
        if (lane == 0) atomicOr(status, MPM_ST_BAD_INPUT);
        return;
    }
    const int N = g.n_grid;
    float gp[3];
    record_gp(st, slot_of_uid[p], S.inv_dx, gp);
    int b[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const float t = __fsub_rn(gp[d], 0.5f);
        // beyond 8 cells outside the grid no offset lands inside; NaN marks nothing
        if (!(t > -8.0f && t < (float)(N + 8))) {
            if (lane == 0 && !(t == t)) atomicOr(status, MPM_ST_OUT_OF_DOMAIN);
            return;
        }
        b[d] = (int)t;  // wp.int truncates toward zero
    }
    constexpr int W = HI + 3;
    for (int o = lane; o < W * W * W; o += 32) {
        const int ix = b[0] + o / (W * W) - 2, iy = b[1] + (o / W) % W - 2, iz = b[2] + o % W - 2;
        if (ix >= 0 && ix < N && iy >= 0 && iy < N && iz >= 0 && iz < N) mask[dense_index(N, ix, iy, iz)] = 1;
    }
}

// The Drucker-Prager Kirchhoff stress of F without an SVD: tau = 2 mu E +
// lam tr(E) I with E = log(F F^T) / 2, in Newton form on the closed-form
// eigenvalues of B = F F^T - I (as sand_return_map_spectral, which also says
// why it is the more accurate form near F = I).  False (SVD path) for inverted
// elements and where the strain makes the SVD the more accurate one.
__device__ __forceinline__ bool stress_dp_spectral(const float F[9], float mu, float lam, float tau[9]) {
    const float J = F[0] * (F[4] * F[8] - F[5] * F[7]) - F[1] * (F[3] * F[8] - F[5] * F[6]) +
                    F[2] * (F[3] * F[7] - F[4] * F[6]);
    if (!(J > 0.0f)) return false;
    float B[6], ev[3];
    left_strain(F, B);
    sym_eig3(B, ev);
    if (!spectral_as_accurate(ev)) return false;
    const float e0 = 0.5f * log1pf(ev[0]), e1 = 0.5f * log1pf(ev[1]), e2 = 0.5f * log1pf(ev[2]);
    const float q0 = 1.0f + ev[0], q1 = 1.0f + ev[1], q2 = 1.0f + ev[2];
    Newton3 N;
    newton3_setup(B, ev, N);
    float T[6];
    newton3_eval(N, e0, e2, 0.5f * log_ratio_div(q0, q1), 0.5f * log_ratio_div(q1, q2), T);
    const float dia = lam * (e0 + e1 + e2), tm = 2.0f * mu;
#pragma unroll
    for (int k = 0; k < 6; ++k) T[k] = tm * T[k] + ((k == 0 || k == 3 || k == 5) ? dia : 0.0f);
    sym_full(T, tau);
    return true;
}

// p2g_sample_all (mpm_utils.py:353-402).  A particle whose base cell is marked
// sets F = F_disp + I, takes the stress of that F (FCR for jelly and metal,
// Drucker-Prager for sand; :368-378) and scatters, per node,
// w m v + dt (-(m / density) stress grad w) and w m.
//
// A warp takes 32 consecutive records.  Each lane prepares its particle (stress
// and the 17 numbers the scatter needs, in shared memory); then, as in the
// substep's P2G, three groups of nine lanes take a third of them each: lane
// (i, j) sums its three z nodes in registers over consecutive particles of one
// base cell and issues one 16-byte atomic per node when the cell changes.  The
// records are in the cell order of the last substep and the particles have
// moved since, so the warp first brings particles of one cell together, for fewer
// runs of 27 atomics.  Measured on 1M marked particles displaced by an eighth of a
// cell: 82 us; with an SVD per stress and segmented shuffles over the runs as they
// lie, 126 us.  64 M warp instructions at 66 % of the issue slots, DRAM 21 %: issue,
// and the latency of the record, F_disp and density loads.
constexpr int kRedWarps = 4;
constexpr int kRedPay = 5;  // float4 of a particle's scatter data
template <bool NARROW>
__global__ void __launch_bounds__(kRedWarps * 32) reduced_p2g_kernel(const MpmScene *__restrict__ scenes, PState st,
                                                                     MpmReducedGrid g, int n, float dt,
                                                                     int *status) {
    chain_wait();
    __shared__ float4 pay[kRedWarps][kRedPay][32];
    const MpmScene &S = scenes[0];
    if (!grid_matches(S, g, status)) return;  // the same for every thread
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int warp = (int)(threadIdx.x >> 5), lane = (int)(threadIdx.x & 31u);
    const int N = g.n_grid;
    const float inv_dx = S.inv_dx;
    float4 q0, q1, q2, q3;
    float fx[3] = {1.0f, 1.0f, 1.0f};
    int base[3] = {0, 0, 0};
    bool act = false;
    if (i < n) {
        ldpair<NARROW>(st, i, 0, q0, q1);
        ldpair<NARROW>(st, i, 1, q2, q3);
        const float gp[3] = {grid_coord(q0.x, q2.x, inv_dx), grid_coord(q0.y, q2.y, inv_dx),
                             grid_coord(q0.z, q2.z, inv_dx)};
        bool cell_in = true, stencil_in = true;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const float t = __fsub_rn(gp[d], 0.5f);
            cell_in = cell_in && t > -1.0f && t < (float)N;
            stencil_in = stencil_in && t > -1.0f && t < (float)(N - 2);
            base[d] = (t > -1.0f && t < (float)N) ? (int)t : 0;
            fx[d] = __fsub_rn(gp[d], (float)base[d]);
        }
        if (!cell_in) {  // the reference reads the mark array out of bounds here
            atomicOr(status, MPM_ST_OUT_OF_DOMAIN);
        } else if (g.neighboring_cells[dense_index(N, base[0], base[1], base[2])] > 0) {
            if (stencil_in) act = true;
            else atomicOr(status, MPM_ST_OUT_OF_DOMAIN);  // marked, but the stencil would leave the grid
        }
    }
    if (__ballot_sync(0xffffffffu, act) == 0u) return;  // the whole warp leaves together
    // the particle's place among the warp's, grouped by cell in the order of the
    // cells' first lanes (-1: not marked)
    const int key = act ? ((base[0] << 20) | (base[1] << 10) | base[2]) : -1;
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    const int leader = __ffs(peers) - 1;
    int at = __popc(peers & ((1u << lane) - 1u));
    for (unsigned heads = __ballot_sync(0xffffffffu, leader == lane); heads; heads &= heads - 1u) {
        const int h = __ffs(heads) - 1;
        const int size = __popc(__shfl_sync(0xffffffffu, peers, h));
        at += h < leader ? size : 0;
    }
    if (act) {
        const int uid = __float_as_int(q1.y);
        const float *fd = g.f_disp + (int64_t)uid * 9;
        float F[9], tau[9], Fo[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) F[k] = __fadd_rn(fd[k], (k % 4 == 0) ? 1.0f : 0.0f);  // F_disp + I (:364)
        stpair<NARROW>(st, i, 0, q0, make_float4(q1.x, q1.y, q1.z, F[8]));
        stpair<NARROW>(st, i, 4, make_float4(F[0], F[1], F[2], F[3]), make_float4(F[4], F[5], F[6], F[7]));
        const bool sand = S.material == MPM_SAND;
        if (!(sand ? stress_dp_spectral(F, S.mu, S.lam, tau) : jelly_stress_spectral<true>(S, F, Fo, tau))) {
            Svd d;
            svd3(F, d);
            if (sand) stress_dp(F, d, S.mu, S.lam, tau);
            else stress_fcr(F, d, d.s[0] * d.s[1] * d.s[2], S.mu, S.lam, tau);
        }
        const float m = q0.w;
        const float ts = -__fdiv_rn(m, g.density[uid]) * dt * inv_dx;  // -(m / density) dt / dx, :395
        pay[warp][0][at] = make_float4(fx[0], fx[1], fx[2], m);
        pay[warp][1][at] = make_float4(q2.w, q3.x, q3.y, __int_as_float(key));
        pay[warp][2][at] = make_float4(tau[0] * ts, tau[1] * ts, tau[2] * ts, tau[3] * ts);
        pay[warp][3][at] = make_float4(tau[4] * ts, tau[5] * ts, tau[6] * ts, tau[7] * ts);
        pay[warp][4][at] = make_float4(tau[8] * ts, 0.0f, 0.0f, 0.0f);
    } else {
        pay[warp][1][at] = make_float4(0.0f, 0.0f, 0.0f, __int_as_float(-1));  // no cell: skipped
    }
    __syncwarp();
    const int group = lane / 9, ij = lane - 9 * group;
    if (group >= 3) return;  // lanes 27-31 only prepare (no warp-wide operation follows)
    const int li = ij / 3, lj = ij - 3 * li;
    // weight along x: sx (f - cx)^2 + tx, its derivative 2 sx (f - cx); y likewise
    const float cx = li == 0 ? 1.5f : (li == 1 ? 1.0f : 0.5f), sx = li == 1 ? -1.0f : 0.5f,
                tx = li == 1 ? 0.75f : 0.0f;
    const float cy = lj == 0 ? 1.5f : (lj == 1 ? 1.0f : 0.5f), sy = lj == 1 ? -1.0f : 0.5f,
                ty = lj == 1 ? 0.75f : 0.0f;
    float4 *grid = static_cast<float4 *>(g.grid_acc);
    float acc[3][4];
#pragma unroll
    for (int k = 0; k < 3; ++k) acc[k][0] = acc[k][1] = acc[k][2] = acc[k][3] = 0.0f;
    int cur = -1;
    const int last = min(32, 11 * group + 11);
    for (int p = 11 * group; p <= last; ++p) {
        const float4 o1 = p < last ? pay[warp][1][p] : make_float4(0.0f, 0.0f, 0.0f, __int_as_float(-1));
        const int key = __float_as_int(o1.w);
        if (key != cur && cur >= 0) {
            float4 *t = grid + dense_index(N, (cur >> 20) + li, ((cur >> 10) & 1023) + lj, cur & 1023);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                atomicAdd(t + k, make_float4(acc[k][0], acc[k][1], acc[k][2], acc[k][3]));
                acc[k][0] = acc[k][1] = acc[k][2] = acc[k][3] = 0.0f;
            }
        }
        cur = key;
        if (key < 0) continue;
        const float4 o0 = pay[warp][0][p], o2 = pay[warp][2][p], o3 = pay[warp][3][p];
        const float t22 = pay[warp][4][p].x;
        const float dxi = o0.x - cx, dyj = o0.y - cy;
        const float ex = sx * dxi, ey = sy * dyj;
        const float wx = fmaf(ex, dxi, tx), wy = fmaf(ey, dyj, ty);
        const float za = o0.z - 1.5f, zb = o0.z - 1.0f, zc = o0.z - 0.5f;
        const float w[3] = {0.5f * za * za, fmaf(-zb, zb, 0.75f), 0.5f * zc * zc};
        const float dw[3] = {za, -2.0f * zb, zc};
        const float p1 = 2.0f * ex * wy, p2 = 2.0f * ey * wx, p3 = wx * wy, pm = p3 * o0.w;
        const float v[3] = {o1.x, o1.y, o1.z};
        const float t0[3] = {o2.x, o2.w, o3.z}, t1[3] = {o2.y, o3.x, o3.w}, t2[3] = {o2.z, o3.y, t22};
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            const float a = fmaf(pm, v[r], fmaf(t0[r], p1, t1[r] * p2)), d = t2[r] * p3;
#pragma unroll
            for (int k = 0; k < 3; ++k) acc[k][r] = fmaf(w[k], a, fmaf(dw[k], d, acc[k][r]));
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) acc[k][3] = fmaf(w[k], pm, acc[k][3]);
    }
}

// grid_normalization_and_gravity_sample_all (mpm_utils.py:405-413) fused with
// the collider sweeps (mpm_solver_warp.py:220-224): every node of the dense
// grid writes grid_m, grid_v_in and grid_v_out.  v_out = v_in / m + dt g on
// marked nodes with m > 1e-10 (a true division, as there), else 0; then each
// collider in registration order, over every node.
__global__ void __launch_bounds__(256) reduced_grid_kernel(const MpmScene *__restrict__ scenes, MpmReducedGrid g,
                                                           float time, float dt, int *status) {
    chain_wait();
    const MpmScene &S = scenes[0];
    if (!grid_matches(S, g, status)) return;
    const int N = g.n_grid;
    const int64_t nn = (int64_t)N * N * N;
    const float4 *acc = static_cast<const float4 *>(g.grid_acc);
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < nn; q += (int64_t)gridDim.x * blockDim.x) {
        const float4 a = acc[q];
        g.grid_m[q] = a.w;
        g.grid_v_in[3 * q + 0] = a.x;
        g.grid_v_in[3 * q + 1] = a.y;
        g.grid_v_in[3 * q + 2] = a.z;
        float v[3] = {0.0f, 0.0f, 0.0f};
        if (g.neighboring_cells[q] > 0 && a.w > 1e-10f) {
            v[0] = __fadd_rn(__fdiv_rn(a.x, a.w), __fmul_rn(dt, S.gravity[0]));
            v[1] = __fadd_rn(__fdiv_rn(a.y, a.w), __fmul_rn(dt, S.gravity[1]));
            v[2] = __fadd_rn(__fdiv_rn(a.z, a.w), __fmul_rn(dt, S.gravity[2]));
        }
        const int ix = (int)(q / ((int64_t)N * N)), iy = (int)((q / N) % N), iz = (int)(q % N);
        for (int k = 0; k < S.n_colliders; ++k) apply_collider(S.colliders[k], S, ix, iy, iz, time, dt, v);
        g.grid_v_out[3 * q + 0] = v[0];
        g.grid_v_out[3 * q + 1] = v[1];
        g.grid_v_out[3 * q + 2] = v[2];
    }
}

// g2p_sample (mpm_utils.py:415-471): one thread per sample point.  Reads the
// dense grid_v_out; writes the particle's u, v, F and F_disp (C and stress
// are left as they are).  The von Mises return map takes yield_stress of the
// sample's list position s (the reference passes its loop index, :464).
// Words are stored one by one: another sample's thread may update the yield
// word of this record.
__global__ void __launch_bounds__(128) g2p_sample_kernel(const MpmScene *__restrict__ scenes, PState st,
                                                         const int *__restrict__ slot_of_uid, MpmReducedGrid g,
                                                         int n, float dt, int *status) {
    chain_wait();
    const MpmScene &S = scenes[0];
    if (!grid_matches(S, g, status)) return;
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= g.n_samples) return;
    const int p = g.sample_index[s];
    const bool metal = S.material == MPM_METAL;
    if (p < 0 || p >= n || (metal && s >= n)) {
        atomicOr(status, MPM_ST_BAD_INPUT);
        return;
    }
    const int N = g.n_grid;
    const int slot = slot_of_uid[p];
    const float4 q0 = ldrec(st, slot, 0), q2 = ldrec(st, slot, 2);
    float gp[3];
    gp[0] = grid_coord(q0.x, q2.x, S.inv_dx);
    gp[1] = grid_coord(q0.y, q2.y, S.inv_dx);
    gp[2] = grid_coord(q0.z, q2.z, S.inv_dx);
    int base[3];
    bool ok = true;
#pragma unroll
    for (int d = 0; d < 3; ++d) ok = stencil_base(gp[d], N, base[d]) && ok;
    if (!ok) {
        atomicOr(status, MPM_ST_OUT_OF_DOMAIN);
        return;
    }
    Weights W;
    make_weights(gp, base, W);
    const float inv_dx = S.inv_dx;
    float nv[3] = {0.f, 0.f, 0.f}, nF[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) nF[k] = 0.f;
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const float weight = W.w[0][a] * W.w[1][b] * W.w[2][c];
                const float dg[3] = {W.dw[0][a] * W.w[1][b] * W.w[2][c] * inv_dx,
                                     W.w[0][a] * W.dw[1][b] * W.w[2][c] * inv_dx,
                                     W.w[0][a] * W.w[1][b] * W.dw[2][c] * inv_dx};
                const float *gv = g.grid_v_out + 3 * dense_index(N, base[0] + a, base[1] + b, base[2] + c);
                const float v0 = gv[0], v1 = gv[1], v2 = gv[2];
                nv[0] += v0 * weight;
                nv[1] += v1 * weight;
                nv[2] += v2 * weight;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    nF[0 + k] += v0 * dg[k];
                    nF[3 + k] += v1 * dg[k];
                    nF[6 + k] += v2 * dg[k];
                }
            }
    // x = x_initial + u (update_x_from_u at the start of p2g2p_reduced), x += dt v (:458)
    float u[3];
    const float x0[3] = {q0.x, q0.y, q0.z}, uo[3] = {q2.x, q2.y, q2.z};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const float x = __fadd_rn(__fadd_rn(x0[d], uo[d]), __fmul_rn(dt, nv[d]));
        u[d] = __fsub_rn(x, x0[d]);  // :469
    }
    const float4 q8 = ldrec(st, slot, 8), q9 = ldrec(st, slot, 9);
    const float Fo_[9] = {q8.x, q8.y, q8.z, q8.w, q9.x, q9.y, q9.z, q9.w, recword(st, slot, rec::F8)};
    float A[9], Ft[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) A[k] = ((k % 4 == 0) ? 1.0f : 0.0f) + dt * nF[k];
    mat_mul(A, Fo_, Ft);
    float yld = 0.0f;
    const int yslot = metal ? slot_of_uid[s] : 0;
    if (metal) yld = recword(st, yslot, rec::YLD);
    float Fn[9], tau[9];
    if (S.material == MPM_JELLY) {
#pragma unroll
        for (int k = 0; k < 9; ++k) Fn[k] = Ft[k];
    } else {
        return_map_stress(S, Ft, yld, Fn, tau);
    }
    if (metal && S.hardening == 1) recword(st, yslot, rec::YLD) = yld;
    bool finite = true;
#pragma unroll
    for (int k = 0; k < 9; ++k) finite = finite && isfinite(Fn[k]);
    if (!finite) atomicOr(status, MPM_ST_NONFINITE);
    recword(st, slot, rec::U + 0) = u[0];
    recword(st, slot, rec::U + 1) = u[1];
    recword(st, slot, rec::U + 2) = u[2];
    recword(st, slot, rec::V + 0) = nv[0];
    recword(st, slot, rec::V + 1) = nv[1];
    recword(st, slot, rec::V + 2) = nv[2];
#pragma unroll
    for (int k = 0; k < 8; ++k) recword(st, slot, rec::F0 + k) = Fn[k];
    recword(st, slot, rec::F8) = Fn[8];
    float *fd = g.f_disp + (int64_t)p * 9;
#pragma unroll
    for (int k = 0; k < 9; ++k) fd[k] = Fn[k] - ((k % 4 == 0) ? 1.0f : 0.0f);  // :471
}

// zero_grid (both mark arrays and the accumulator) and slot_of_uid, in one launch
__global__ void __launch_bounds__(256) reduced_clear_kernel(PState st, int n, int *__restrict__ slot_of_uid,
                                                            MpmReducedGrid g, int64_t nn) {
    chain_wait();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
    float4 *acc = static_cast<float4 *>(g.grid_acc);
    for (int64_t q = i; q < nn; q += stride) acc[q] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (int64_t q = i; q < nn; q += stride) g.neighboring_cells[q] = 0;
    for (int64_t q = i; q < nn; q += stride) g.neighboring_cells_grid_v[q] = 0;
    for (int64_t p = i; p < n; p += stride) slot_of_uid[__float_as_int(ldrec(st, (int)p, 1).y)] = (int)p;
}

cudaError_t launch_p2g2p_reduced(const Ctx &cx, const MpmReducedGrid &g, float time, float dt) {
    const int64_t nn = (int64_t)g.n_grid * g.n_grid * g.n_grid;
    launch_chained(reduced_clear_kernel, cx.num_sms * 8, 256, 0, cx.stream, cx.st, cx.n, cx.ws.slot_of_uid, g, nn);
    if (cx.n > 0) {
        if (g.n_samples > 0)
            launch_chained(mark_kernel<2>, (unsigned)((g.n_samples + 7) / 8), 256, 0, cx.stream, cx.scenes, cx.st,
                           cx.ws.slot_of_uid, g, g.neighboring_cells, cx.n, cx.status);
        launch_chained(cx.st.wide ? reduced_p2g_kernel<false> : reduced_p2g_kernel<true>,
                       (cx.n + kRedWarps * 32 - 1) / (kRedWarps * 32), kRedWarps * 32, 0, cx.stream, cx.scenes,
                       cx.st, g, cx.n, dt, cx.status);
    }
    const int64_t want = (nn + 255) / 256;
    const int blocks = (int)(want < (int64_t)cx.num_sms * 16 ? want : (int64_t)cx.num_sms * 16);
    launch_chained(reduced_grid_kernel, blocks > 0 ? blocks : 1, 256, 0, cx.stream, cx.scenes, g, time, dt, cx.status);
    return cudaGetLastError();
}

cudaError_t launch_mark_grid_v(const Ctx &cx, const MpmReducedGrid &g) {
    if (cx.n == 0 || g.n_samples == 0) return cudaSuccess;
    cudaError_t e = launch_slot_of_uid(cx);
    if (e != cudaSuccess) return e;
    launch_chained(mark_kernel<4>, (unsigned)((g.n_samples + 7) / 8), 256, 0, cx.stream, cx.scenes, cx.st,
                   cx.ws.slot_of_uid, g, g.neighboring_cells_grid_v, cx.n, cx.status);
    return cudaGetLastError();
}

cudaError_t launch_g2p_sample(const Ctx &cx, const MpmReducedGrid &g, float dt) {
    if (cx.n == 0 || g.n_samples == 0) return cudaSuccess;
    cudaError_t e = launch_slot_of_uid(cx);
    if (e != cudaSuccess) return e;
    launch_chained(g2p_sample_kernel, (unsigned)((g.n_samples + 127) / 128), 128, 0, cx.stream, cx.scenes, cx.st,
                   cx.ws.slot_of_uid, g, cx.n, dt, cx.status);
    return cudaGetLastError();
}

}  // namespace mpm
