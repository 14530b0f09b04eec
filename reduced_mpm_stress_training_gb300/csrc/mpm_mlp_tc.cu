// Stress-surrogate network forward on the 5th-generation tensor cores
// (tcgen05.mma, accumulators in tensor memory).  Same network, parameter blob
// and bf16 rounding points as mlp_forward_kernel (mpm_mlp.cu):
//   Z_l = H_{l-1} W_l^T + b_l (fp32 accumulate), H_l = bf16(silu(Z_l)).
//
// One persistent CTA per SM runs kPipes tile pipelines of 256 threads over one
// copy of the weights.  A pipeline takes a 128-row tile through the layers: one
// thread issues a layer's MMAs (M = 128 rows, N = 128 or 16, K = 16 each) into
// the pipeline's 128 tensor-memory columns and commits them to its mbarrier;
// then two threads per row read the row's accumulators with tcgen05.ld, apply
// SiLU and write the bf16 activations back as the next layer's A operand.  The
// other pipelines' epilogues run meanwhile.  Operands live in shared memory
// in the canonical K-major layout without swizzle: 8-row x 16-byte core
// matrices, K-adjacent core matrices 128 B apart (leading byte offset), 8-row
// groups 256 B apart (stride byte offset), one 16-wide K slab per MMA.
//
// W1-W3 and their biases are staged halved (exact: a power of two), so the
// accumulator is z / 2 = g and silu(z) = z (1 + tanh(z / 2)) / 2 = g (1 + tanh(g)):
// per pair of elements a packed add for the bias, two MUFU, a packed add and a
// packed multiply, with the very roundings of z sigmoid(z).  The next tile's
// inputs are loaded a tile ahead.
//
// What bounds it: a pipeline's chain of MMAs, commit, barrier and epilogue (with
// the activation left out, 1M rows still take 120 us; reading both MMA operands
// from shared memory costs 64 of a K step's cycles).  Measured on 1M rows, 200
// us -> 182 us: before, two CTAs per SM with their own weights, scalar epilogues
// (8.8 instructions per activation) and the inputs' latency exposed.
// Every mbarrier wait is bounded: on timeout the pipeline raises an error
// flag, stops issuing work, and the CTA frees its tensor memory and returns.
#include "mpm_mlp_tc.cuh"
#include "mpm_launch.h"

namespace mpm {
namespace mlptc {

constexpr int kPipes = 3;
constexpr int kFwThreads = kPipes * kThreads;
constexpr uint32_t kFwCols = 512;  // 128 per pipeline, rounded up to a power of two

struct TcIO {
    const float *x;        // [n][12]
    float *y;              // [n][6] or null
    const float *target;   // [n][6] or null
    __nv_bfloat16 *z;      // [3][n][128] or null
    __nv_bfloat16 *dy;     // [n][16] or null
    float *loss;           // or null
    float grad_scale;
    int64_t n;
    bool x16, dy16;        // x, dy are 16-byte aligned
};

struct FwSmem {
    alignas(128) unsigned char w1[kWSlab];            // W1 / 2: one slab
    alignas(128) unsigned char w2[8 * kWSlab];
    alignas(128) unsigned char w3[8 * kWSlab];
    alignas(128) unsigned char w4[8 * kW4Slab];
    alignas(128) unsigned char x[kPipes][kSlab];      // input tile: one slab
    alignas(128) unsigned char h[kPipes][8 * kSlab];  // activations: eight slabs
    alignas(16) float bias[3 * H];                    // b1 / 2, b2 / 2, b3 / 2
    float b4[N4];
    float loss[kFwThreads / 32];
    alignas(8) unsigned long long mbar[kPipes];
    uint32_t tmem_base;
    int fail[kPipes];
};

__device__ __forceinline__ uint32_t halve_bf16x2(uint32_t u) {
    const float2 f = unpack_bf16(u);
    return pack_bf16(0.5f * f.x, 0.5f * f.y);
}
__device__ __forceinline__ uint4 halved(uint4 v) {
    return make_uint4(halve_bf16x2(v.x), halve_bf16x2(v.y), halve_bf16x2(v.z), halve_bf16x2(v.w));
}

__device__ __forceinline__ void stage_forward(FwSmem &s, const __nv_bfloat16 *w, const float *b) {
    const uint4 *g = reinterpret_cast<const uint4 *>(w);
    for (int i = threadIdx.x; i < H * (K1 / 8); i += kFwThreads) {  // W1 [128][16]
        const int n = i / (K1 / 8), k8 = i % (K1 / 8);
        *reinterpret_cast<uint4 *>(s.w1 + chunk_off(n, k8, kWSlab)) = halved(g[W1_OFF / 8 + i]);
    }
    for (int i = threadIdx.x; i < H * (H / 8); i += kFwThreads) {   // W2, W3 [128][128]
        const int n = i / (H / 8), k8 = i % (H / 8);
        *reinterpret_cast<uint4 *>(s.w2 + chunk_off(n, k8, kWSlab)) = halved(g[W2_OFF / 8 + i]);
        *reinterpret_cast<uint4 *>(s.w3 + chunk_off(n, k8, kWSlab)) = halved(g[W3_OFF / 8 + i]);
    }
    for (int i = threadIdx.x; i < N4 * (H / 8); i += kFwThreads) {  // W4 [16][128]
        const int n = i / (H / 8), k8 = i % (H / 8);
        *reinterpret_cast<uint4 *>(s.w4 + chunk_off(n, k8, kW4Slab)) = g[W4_OFF / 8 + i];
    }
    for (int i = threadIdx.x; i < 3 * H; i += kFwThreads) s.bias[i] = 0.5f * b[B1_OFF + i];
    for (int i = threadIdx.x; i < N4; i += kFwThreads) s.b4[i] = b[B4_OFF + i];
}

// barrier over the 256 threads of a pipeline (ids 1 .. kPipes; immediates, so that the
// kernel reserves no more barriers than it uses).  bar.sync is warp-wide (.aligned), as
// tcgen05.ld is: the kernel brings a warp's lanes together where they may have parted (the
// rows past n, the poll loop) and not before each of these (1M rows 183 us, 187 so).
__device__ __forceinline__ void pipe_barrier(int pipe) {
    static_assert(kPipes == 3 && kThreads == 256, "barrier ids and counts");
    if (pipe == 0) asm volatile("bar.sync 1, 256;\n" ::: "memory");
    else if (pipe == 1) asm volatile("bar.sync 2, 256;\n" ::: "memory");
    else asm volatile("bar.sync 3, 256;\n" ::: "memory");
}

// bias + SiLU of 32 accumulator columns of this thread's row (acc and bias halved);
// writes the bf16 activations (columns c0 .. c0 + 31) into the A slabs and, if
// given, Z to zrow
__device__ __forceinline__ void activate_chunk(unsigned char *h, const float acc[32], const float *bias, int row,
                                               int c0, __nv_bfloat16 *zrow) {
    const float2 one = make_float2(1.0f, 1.0f);
#pragma unroll
    for (int q = 0; q < 4; ++q) {  // 4 chunks of 8 columns = 16 bytes
        uint32_t hv[4], zv[4] = {0u, 0u, 0u, 0u};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int c = q * 8 + 2 * e;
            const float2 g = __fadd2_rn(make_float2(acc[c], acc[c + 1]),
                                        *reinterpret_cast<const float2 *>(bias + c0 + c));
            const float2 v = __fmul2_rn(g, __fadd2_rn(make_float2(tanh_approx(g.x), tanh_approx(g.y)), one));
            hv[e] = pack_bf16(v.x, v.y);
            if (zrow) {
                const float2 z = __fadd2_rn(g, g);
                zv[e] = pack_bf16(z.x, z.y);
            }
        }
        *reinterpret_cast<uint4 *>(h + chunk_off(row, (c0 >> 3) + q, kSlab)) = make_uint4(hv[0], hv[1], hv[2], hv[3]);
        if (zrow) *reinterpret_cast<uint4 *>(zrow + c0 + q * 8) = make_uint4(zv[0], zv[1], zv[2], zv[3]);
    }
}

__device__ __forceinline__ void load_x(const TcIO &io, int64_t row, float (&v)[IN]) {
    if (io.x16) {
        const float4 *p = reinterpret_cast<const float4 *>(io.x + row * IN);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float4 f = p[k];
            v[4 * k] = f.x;
            v[4 * k + 1] = f.y;
            v[4 * k + 2] = f.z;
            v[4 * k + 3] = f.w;
        }
    } else {
#pragma unroll
        for (int k = 0; k < IN; ++k) v[k] = io.x[row * IN + k];
    }
}

__global__ void __launch_bounds__(kFwThreads, 1) mlp_forward_tc_kernel(const __nv_bfloat16 *__restrict__ w,
                                                                       const float *__restrict__ b, TcIO io,
                                                                       int *__restrict__ err) {
    chain_wait();
    extern __shared__ __align__(128) unsigned char tc_smem_raw[];
    FwSmem &s = *reinterpret_cast<FwSmem *>(tc_smem_raw);
    const int pipe = (int)threadIdx.x / kThreads, tid = (int)threadIdx.x % kThreads, warp = tid >> 5;
    const int row = tid & (kRows - 1), half = tid >> 7;
    const bool lead = half == 0;  // the thread that owns the row's inputs and outputs
    stage_forward(s, w, b);
    if (threadIdx.x < kPipes) {
        s.fail[threadIdx.x] = 0;
        const uint32_t a = (uint32_t)__cvta_generic_to_shared(&s.mbar[threadIdx.x]);
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(a) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (threadIdx.x < 32) {
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&s.tmem_base);
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(dst), "r"(kFwCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    fence_async_smem();
    tc_before_sync();
    __syncthreads();
    tc_after_sync();
    const uint32_t tbase = s.tmem_base + (uint32_t)(pipe * H);
    const uint32_t tlane = tbase + ((uint32_t)((warp & 3) * 32) << 16);
    unsigned char *sx = s.x[pipe], *sh = s.h[pipe];
    unsigned long long *mbar = &s.mbar[pipe];
    volatile int *fail = &s.fail[pipe];
    uint32_t phase = 0;
    bool ok = true;
    float lsum = 0.0f;
    const int64_t tiles = (io.n + kRows - 1) / kRows, step = (int64_t)gridDim.x * kPipes;
    int64_t tile = blockIdx.x + (int64_t)gridDim.x * pipe;
    float xv[IN];
#pragma unroll
    for (int k = 0; k < IN; ++k) xv[k] = 0.0f;
    if (lead && tile * kRows + row < io.n) load_x(io, tile * kRows + row, xv);
    for (; tile < tiles; tile += step) {
        const int64_t grow = tile * kRows + row;
        const bool valid = grow < io.n;
        if (lead) {
            *reinterpret_cast<uint4 *>(sx + chunk_off(row, 0, kSlab)) =
                make_uint4(pack_bf16(xv[0], xv[1]), pack_bf16(xv[2], xv[3]), pack_bf16(xv[4], xv[5]),
                           pack_bf16(xv[6], xv[7]));
            *reinterpret_cast<uint4 *>(sx + chunk_off(row, 1, kSlab)) =
                make_uint4(pack_bf16(xv[8], xv[9]), pack_bf16(xv[10], xv[11]), 0u, 0u);
            // the next tile's inputs arrive while this one is evaluated
            const int64_t next = grow + step * kRows;
#pragma unroll
            for (int k = 0; k < IN; ++k) xv[k] = 0.0f;
            if (next < io.n) load_x(io, next, xv);
        }
        __syncwarp();
#pragma unroll 1
        for (int layer = 0; layer < 4; ++layer) {
            fence_async_smem();
            tc_before_sync();
            pipe_barrier(pipe);
            tc_after_sync();
            if (*fail) {  // a wait of this pipeline ran out (uniform after the barrier)
                ok = false;
                break;
            }
            if (tid == 0) {
                if (layer == 0) {
                    mma_bf16(tbase, smem_desc(sx), smem_desc(s.w1), idesc_bf16(kRows, H), false);
                } else {
                    const unsigned char *wl = layer == 1 ? s.w2 : layer == 2 ? s.w3 : s.w4;
                    const int wslab = layer == 3 ? kW4Slab : kWSlab;
                    const uint32_t id = idesc_bf16(kRows, layer == 3 ? N4 : H);
#pragma unroll
                    for (int ks = 0; ks < 8; ++ks)
                        mma_bf16(tbase, smem_desc(sh + ks * kSlab), smem_desc(wl + ks * wslab), id, ks > 0);
                }
                mma_commit(mbar);
            }
            if (!mbar_wait(mbar, phase)) *fail = 1;
            __syncwarp();
            phase ^= 1u;
            tc_after_sync();
            if (layer == 3) break;
            // the layer's MMAs are done reading sh: overwrite it with the next activations
            __nv_bfloat16 *zrow = io.z && valid ? io.z + (int64_t)layer * io.n * H + grow * H : nullptr;
#pragma unroll 1
            for (int c0 = half * (H / 2); c0 < (half + 1) * (H / 2); c0 += 32) {
                float acc[32];
                tmem_ld32<true>(tlane + (uint32_t)c0, acc);
                activate_chunk(sh, acc, s.bias + layer * H, row, c0, zrow);
                if (io.z) __syncwarp();  // rows past n store no Z
            }
        }
        if (!ok) break;
        float acc[32];
        tmem_ld32<true>(tlane, acc);
#pragma unroll
        for (int c = 0; c < OUT; ++c) acc[c] += s.b4[c];
        if (lead && valid) {
            float d[8];
#pragma unroll
            for (int c = 0; c < 8; ++c) d[c] = 0.0f;
#pragma unroll
            for (int c = 0; c < OUT; ++c) {
                if (io.y) io.y[grow * OUT + c] = acc[c];
                if (io.target) {
                    const float r = acc[c] - io.target[grow * OUT + c];
                    lsum += r * r;
                    d[c] = io.grad_scale * r;
                }
            }
            if (io.dy) {
                if (io.dy16) {
                    uint4 *p = reinterpret_cast<uint4 *>(io.dy + grow * N4);
                    p[0] = make_uint4(pack_bf16(d[0], d[1]), pack_bf16(d[2], d[3]), pack_bf16(d[4], d[5]), 0u);
                    p[1] = make_uint4(0u, 0u, 0u, 0u);
                } else {
#pragma unroll
                    for (int c = 0; c < N4; ++c) io.dy[grow * N4 + c] = __float2bfloat16_rn(c < OUT ? d[c] : 0.0f);
                }
            }
        }
    }
    if (io.loss) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
        if ((threadIdx.x & 31) == 0) s.loss[threadIdx.x >> 5] = lsum;
    }
    // a wait that ran out in the pipeline's last layer shows here; then the MMAs may still be
    // in flight, so they get a bounded grace period before the tensor memory is released
    tc_before_sync();
    __syncthreads();
    tc_after_sync();
    if (tid == 0 && *fail) {
        atomicOr(err, 1);
        mbar_wait(mbar, phase ^ 1u);
    }
    if (io.loss && threadIdx.x == 0) {  // one atomic per CTA: few roundings of the running sum
        float sum = 0.0f;
        for (int k = 0; k < kFwThreads / 32; ++k) sum += s.loss[k];
        atomicAdd(io.loss, sum);
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        __syncwarp();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(s.tmem_base), "r"(kFwCols)
                     : "memory");
    }
}

}  // namespace mlptc

int64_t mlp_tc_smem_bytes() {
    static_assert(sizeof(mlptc::FwSmem) <= 227 * 1024, "shared memory of one CTA");
    return (int64_t)sizeof(mlptc::FwSmem);
}

cudaError_t launch_mlp_forward_tc(const void *params, const float *x, float *y, const float *target, void *zsave,
                                  void *dy, float *loss, float grad_scale, int64_t n, int *err, int num_sms,
                                  cudaStream_t stream) {
    using namespace mlptc;
    if (n <= 0) return cudaSuccess;
    static bool attr_set[64] = {false};
    const int bytes = (int)mlp_tc_smem_bytes();
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64 || !attr_set[dev]) {
        e = cudaFuncSetAttribute(mlp_forward_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) attr_set[dev] = true;
    }
    const __nv_bfloat16 *w = static_cast<const __nv_bfloat16 *>(params);
    const float *b = reinterpret_cast<const float *>(static_cast<const char *>(params) + (int64_t)mlp::W_COUNT * 2);
    TcIO io{x, y, target, static_cast<__nv_bfloat16 *>(zsave), static_cast<__nv_bfloat16 *>(dy), loss, grad_scale, n,
            (reinterpret_cast<uintptr_t>(x) & 15) == 0, (reinterpret_cast<uintptr_t>(dy) & 15) == 0};
    const int64_t tiles = (n + kRows - 1) / kRows;
    // small batches spread over the SMs before they fill a CTA's pipelines
    const int grid = (int)(tiles < (int64_t)num_sms ? tiles : (int64_t)num_sms);
    launch_chained(mlp_forward_tc_kernel, grid, kFwThreads, bytes, stream, w, b, io, err);
    return cudaGetLastError();
}

}  // namespace mpm
