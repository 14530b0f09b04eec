// Stress-surrogate network backward on the 5th-generation tensor cores
// (tcgen05.mma, accumulators in tensor memory).  Same gradients, parameter
// blob and bf16 rounding points as the mma.sync kernels of mpm_mlp.cu:
//   dZ_4 = dY (bf16, from the forward)
//   dH_{l-1} = dZ_l W_l            (fp32 accumulate)
//   dZ_{l-1} = bf16(dH_{l-1} * silu'(Z_{l-1}))
//   dW_l += dZ_l^T H_{l-1},  db_l += sum_rows dZ_l,  H_{l-1} = bf16(silu(Z_{l-1})) (H_0 = bf16(x))
//
// One persistent CTA per SM (512 threads, the whole 512-column tensor memory)
// walks 128-row tiles.  The weight gradients stay in tensor memory across all
// of the CTA's tiles:
//   columns   0-127  dH (the data gradient of the current layer, per tile)
//   columns 128-255  dW2 [out = lane][in = column]
//   columns 256-383  dW3
//   columns 384-399  dW1 [out][in 0-11], column 12 = db1
//   columns 400-415  dW4^T [in = lane][out 0-15]
//   columns 416-431, 432-447  column 12: db3, db2
// so no weight-gradient sum goes through global memory until the end, when
// each CTA adds its accumulators into grad once.  The bias sums come out of
// the tensor cores too: x carries a column of ones, and dZ_l^T times it is db_l.
//
// Every operand has one copy in shared memory, as 8-row x 16-byte core
// matrices with uniform strides: 128 B between column-adjacent ones, 128 B x
// (columns / 8) between row-adjacent ones.  The data gradient reads dZ with
// rows as M and columns as K, the weight gradient reads the same bytes with
// columns as M and rows as K (an MN-major operand), and the weights, stored
// [out][in], are MN-major operands of the data gradient as they are; nothing
// is transposed by hand.  Activations are evaluated in place: Z_l arrives by
// cp.async in the buffer where each thread then writes the H_l of the columns
// it read.  A phase waits for its data gradient only (committed first); the
// weight gradients run behind the next epilogue, and the next commit covers
// them, which is when their operands' buffers may be overwritten.
//
// What it replaces wrote every dZ and H a second time, transposed, element by
// element, and summed biases serially.  Bound now by the epilogues' latency
// (four phases a tile, 2 MUFU per element; issue slots 26 %, tensor pipe 9 % busy,
// waits for tensor memory and at the barriers).  Measured on 65,536 rows: 93 us ->
// 54 us.  Every mbarrier wait is bounded: on timeout the kernel raises the error
// flag, stops issuing work, frees its tensor memory after a bounded grace
// wait and returns.
#include "mpm_mlp_tc.cuh"
#include "mpm_launch.h"

namespace mpm {
namespace mlpbw {

using namespace mpm::mlp;
using namespace mpm::mlptc;

constexpr int kBwThreads = 512;     // four threads per row, 32 columns each
constexpr uint32_t kBwCols = 512;
constexpr uint32_t C_DH = 0, C_W2 = 128, C_W3 = 256, C_W1 = 384, C_W4 = 400, C_B3 = 416, C_B2 = 432;
constexpr int kOne = 12;            // the ones column of xo

constexpr int kWide = (kRows / 8) * (H / 8) * 128;    // a [128][128] operand: 32 KB
constexpr int kNarrow = (kRows / 8) * (N4 / 8) * 128; // [128][16] and [16][128]: 4 KB

struct BwSmem {
    alignas(128) unsigned char w2[kWide];     // W2 [out][in]
    alignas(128) unsigned char w3[kWide];
    alignas(128) unsigned char w4[kNarrow];   // W4 [out 16][in]
    alignas(128) unsigned char h[2][kWide];   // Z_l, then H_l [rows][in]
    alignas(128) unsigned char dz[2][kWide];  // dZ_l [rows][out]
    alignas(128) unsigned char dz4[kNarrow];  // dY [rows][out 16]
    alignas(128) unsigned char xo[kNarrow];   // [rows][x 0-11 | 1 | 0 0 0]
    alignas(8) unsigned long long mbar;
    uint32_t tmem_base;
    int fail;
};

// byte offset of the 16-byte chunk (row, columns 8 c8 .. 8 c8 + 7) of an operand with
// CC = columns / 8 chunks a row
template <int CC>
__device__ __forceinline__ uint32_t core_off(int row, int c8) {
    return (uint32_t)(((row >> 3) * CC + c8) * 128 + (row & 7) * 16);
}

// shared-memory descriptor without swizzle: lbo / sbo = the strides (bytes)
// between core matrices along K / along M or N
__device__ __forceinline__ uint64_t desc(const void *p, uint32_t k_stride, uint32_t mn_stride) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    uint64_t d = 0;
    d |= (uint64_t)((a >> 4) & 0x3FFF);
    d |= (uint64_t)((k_stride >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)((mn_stride >> 4) & 0x3FFF) << 32;
    d |= (uint64_t)1 << 46;
    return d;
}
// K step ks (16 wide) of an operand whose columns are K (rows are M)
template <int CC>
__device__ __forceinline__ uint64_t desc_rows(const unsigned char *p, int ks) {
    return desc(p + ks * 256, 128, CC * 128);
}
// K step ks of an operand whose rows are K (columns are M or N): MN-major
template <int CC>
__device__ __forceinline__ uint64_t desc_cols(const unsigned char *p, int ks) {
    return desc(p + ks * 2 * CC * 128, CC * 128, 128);
}
constexpr uint32_t kAMn = 1u << 15, kBMn = 1u << 16;  // instruction descriptor: operand is MN-major

// [n_rows][128] weights, row-major in the blob -> core matrices
__device__ __forceinline__ void stage_w(unsigned char *dst, const __nv_bfloat16 *w, int n_rows) {
    const uint4 *g = reinterpret_cast<const uint4 *>(w);
    for (int i = threadIdx.x; i < n_rows * (H / 8); i += kBwThreads)
        *reinterpret_cast<uint4 *>(dst + core_off<H / 8>(i / (H / 8), i % (H / 8))) = g[i];
}

// queue the copy of a tile of pre-activations (rows past n read as zero); a warp
// takes 8 rows x 64 bytes at a time (whole half lines, conflict-free banks)
__device__ __forceinline__ void load_z(unsigned char *dst, const __nv_bfloat16 *z, int64_t row0, int64_t n) {
    const int warp = (int)(threadIdx.x >> 5), lane = (int)(threadIdx.x & 31u);
#pragma unroll
    for (int k = 0; k < 64 / (kBwThreads / 32); ++k) {
        const int idx = warp + k * (kBwThreads / 32);
        const int row = (idx >> 2) * 8 + (lane & 7), c8 = (idx & 3) * 4 + (lane >> 3);
        const bool in = row0 + row < n;
        const void *src = z + (in ? (row0 + row) * H + c8 * 8 : 0);
        const uint32_t a = (uint32_t)__cvta_generic_to_shared(dst + core_off<H / 8>(row, c8));
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(a), "l"(src), "r"(in ? 16 : 0)
                     : "memory");
    }
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int LEFT>
__device__ __forceinline__ void cp_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(LEFT) : "memory");
}

// this thread's 32 columns of a Z tile into registers, H = bf16(silu(Z)) in their place
__device__ __forceinline__ void activate(unsigned char *h, int row, int c0, uint32_t (&z)[16]) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        uint4 *at = reinterpret_cast<uint4 *>(h + core_off<H / 8>(row, (c0 >> 3) + q));
        const uint4 v = *at;
        z[4 * q] = v.x;
        z[4 * q + 1] = v.y;
        z[4 * q + 2] = v.z;
        z[4 * q + 3] = v.w;
        uint32_t o[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float2 f = unpack_bf16(z[4 * q + e]);
            o[e] = pack_bf16(silu(f.x), silu(f.y));
        }
        *at = make_uint4(o[0], o[1], o[2], o[3]);
    }
}

// dZ = bf16(dH silu'(Z)) of this thread's 32 columns
__device__ __forceinline__ void data_gradient(unsigned char *dz, uint32_t tdh, int row, int c0,
                                              const uint32_t (&z)[16]) {
    float acc[32];
    tmem_ld32(tdh + (uint32_t)c0, acc);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        uint32_t o[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float2 f = unpack_bf16(z[4 * q + e]);
            o[e] = pack_bf16(acc[8 * q + 2 * e] * silu_grad(f.x), acc[8 * q + 2 * e + 1] * silu_grad(f.y));
        }
        *reinterpret_cast<uint4 *>(dz + core_off<H / 8>(row, (c0 >> 3) + q)) = make_uint4(o[0], o[1], o[2], o[3]);
    }
}

// everything written to shared memory and read from tensor memory so far is
// ordered before the MMAs that thread 0 issues next
__device__ __forceinline__ void bw_sync() {
    fence_async_smem();
    tc_before_sync();
    __syncthreads();
    tc_after_sync();
}

__global__ void __launch_bounds__(kBwThreads, 1) mlp_backward_tc_kernel(const __nv_bfloat16 *__restrict__ w,
                                                                     const float *__restrict__ x,
                                                                     const __nv_bfloat16 *__restrict__ zsave,
                                                                     const __nv_bfloat16 *__restrict__ dy,
                                                                     float *__restrict__ grad, int64_t n,
                                                                     int *__restrict__ err) {
    chain_wait();
    extern __shared__ __align__(128) unsigned char bw_smem_raw[];
    BwSmem &s = *reinterpret_cast<BwSmem *>(bw_smem_raw);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int row = tid & (kRows - 1), quarter = tid >> 7, c0 = quarter * 32;
    const __nv_bfloat16 *z1g = zsave, *z2g = zsave + n * H, *z3g = zsave + 2 * n * H;
    const int64_t tiles = (n + kRows - 1) / kRows;
    int a = 0;  // buffer of H3 and H1 of this tile; the other one holds H2
    load_z(s.h[0], z3g, (int64_t)blockIdx.x * kRows, n);
    cp_commit();
    stage_w(s.w2, w + W2_OFF, H);
    stage_w(s.w3, w + W3_OFF, H);
    stage_w(s.w4, w + W4_OFF, N4);
    if (tid == 0) {
        s.fail = 0;
        const uint32_t m = (uint32_t)__cvta_generic_to_shared(&s.mbar);
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(m) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 0) {
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&s.tmem_base);
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(dst),
                     "r"(kBwCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    bw_sync();
    const uint32_t tbase = s.tmem_base;
    const uint32_t tlane = tbase + ((uint32_t)((warp & 3) * 32) << 16);  // this warp's TMEM lane quarter
    uint32_t phase = 0;
    bool first = true;
    float db4[N4];
#pragma unroll
    for (int c = 0; c < N4; ++c) db4[c] = 0.0f;
    const uint32_t id_dh = idesc_bf16(kRows, H) | kBMn, id_w = idesc_bf16(kRows, H) | kAMn | kBMn,
                   id_w16 = idesc_bf16(kRows, N4) | kAMn | kBMn;
    // wait for the last commit; a timeout is seen by every thread after its next barrier
    auto wait_mma = [&]() {
        if (!mbar_wait(&s.mbar, phase)) *reinterpret_cast<volatile int *>(&s.fail) = 1;
        phase ^= 1u;
        tc_after_sync();
    };
    auto failed = [&]() { return *reinterpret_cast<volatile int *>(&s.fail) != 0; };
    bool stopped = false;     // a wait ran out (uniform: read behind a barrier)
    uint32_t zl[16], zp[16];  // Z of this phase's data gradient, Z of its activations
    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int64_t row0 = tile * kRows, grow = row0 + row;
        const bool valid = grow < n;
        // ---- layer 4: dZ4 = dY, H3 ----
        uint4 d0 = make_uint4(0u, 0u, 0u, 0u), d1 = d0;
        if (valid && quarter == 0) {
            d0 = reinterpret_cast<const uint4 *>(dy + grow * N4)[0];
            d1 = reinterpret_cast<const uint4 *>(dy + grow * N4)[1];
        }
        float xv[IN];
        if (quarter == 1) {
#pragma unroll
            for (int k = 0; k < IN; ++k) xv[k] = valid ? x[grow * IN + k] : 0.0f;
        }
        if (!first) wait_mma();  // the previous tile's last MMAs: xo, dz and both h buffers are free
        load_z(s.h[a ^ 1], z2g, row0, n);
        cp_commit();
        cp_wait<1>();     // Z3
        __syncthreads();  // every thread's part of it
        if ((stopped = failed())) break;
        activate(s.h[a], row, c0, zl);
        if (quarter == 0) {
            *reinterpret_cast<uint4 *>(s.dz4 + core_off<2>(row, 0)) = d0;
            *reinterpret_cast<uint4 *>(s.dz4 + core_off<2>(row, 1)) = d1;
            const uint32_t u[8] = {d0.x, d0.y, d0.z, d0.w, d1.x, d1.y, d1.z, d1.w};
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const float2 f = unpack_bf16(u[c]);
                db4[2 * c] += f.x;
                db4[2 * c + 1] += f.y;
            }
        } else if (quarter == 1) {
            *reinterpret_cast<uint4 *>(s.xo + core_off<2>(row, 0)) =
                make_uint4(pack_bf16(xv[0], xv[1]), pack_bf16(xv[2], xv[3]), pack_bf16(xv[4], xv[5]),
                           pack_bf16(xv[6], xv[7]));
            *reinterpret_cast<uint4 *>(s.xo + core_off<2>(row, 1)) =
                make_uint4(pack_bf16(xv[8], xv[9]), pack_bf16(xv[10], xv[11]), pack_bf16(1.0f, 0.0f), 0u);
        }
        bw_sync();
        if (tid == 0) {
            // dH3 = dZ4 W4 (K = 16), then dW4^T += H3^T dZ4
            mma_bf16(tbase + C_DH, desc_rows<2>(s.dz4, 0), desc_cols<H / 8>(s.w4, 0), id_dh, false);
            mma_commit(&s.mbar);
#pragma unroll 1
            for (int ks = 0; ks < 8; ++ks)
                mma_bf16(tbase + C_W4, desc_cols<H / 8>(s.h[a], ks), desc_cols<2>(s.dz4, ks), id_w16,
                         !first || ks > 0);
        }
        // ---- layer 3: dZ3 = dH3 silu'(Z3), H2 ----
        wait_mma();
        cp_wait<0>();  // Z2
        data_gradient(s.dz[0], tlane + C_DH, row, c0, zl);
        __syncthreads();
        if ((stopped = failed())) break;
        activate(s.h[a ^ 1], row, c0, zp);
        bw_sync();
        if (tid == 0) {
#pragma unroll 1
            for (int ks = 0; ks < 8; ++ks)
                mma_bf16(tbase + C_DH, desc_rows<H / 8>(s.dz[0], ks), desc_cols<H / 8>(s.w3, ks), id_dh, ks > 0);
            mma_commit(&s.mbar);
#pragma unroll 1
            for (int ks = 0; ks < 8; ++ks) {
                mma_bf16(tbase + C_W3, desc_cols<H / 8>(s.dz[0], ks), desc_cols<H / 8>(s.h[a ^ 1], ks), id_w,
                         !first || ks > 0);
                mma_bf16(tbase + C_B3, desc_cols<H / 8>(s.dz[0], ks), desc_cols<2>(s.xo, ks), id_w16,
                         !first || ks > 0);
            }
        }
        // ---- layer 2: dZ2 = dH2 silu'(Z2), H1 ----
        wait_mma();  // ... and dW4's MMAs before it: H3's buffer is free
        load_z(s.h[a], z1g, row0, n);
        cp_commit();
        data_gradient(s.dz[1], tlane + C_DH, row, c0, zp);
        cp_wait<0>();
        __syncthreads();
        if ((stopped = failed())) break;
        activate(s.h[a], row, c0, zl);
        bw_sync();
        if (tid == 0) {
#pragma unroll 1
            for (int ks = 0; ks < 8; ++ks)
                mma_bf16(tbase + C_DH, desc_rows<H / 8>(s.dz[1], ks), desc_cols<H / 8>(s.w2, ks), id_dh, ks > 0);
            mma_commit(&s.mbar);
#pragma unroll 1
            for (int ks = 0; ks < 8; ++ks) {
                mma_bf16(tbase + C_W2, desc_cols<H / 8>(s.dz[1], ks), desc_cols<H / 8>(s.h[a], ks), id_w,
                         !first || ks > 0);
                mma_bf16(tbase + C_B2, desc_cols<H / 8>(s.dz[1], ks), desc_cols<2>(s.xo, ks), id_w16,
                         !first || ks > 0);
            }
        }
        // ---- layer 1: dZ1 = dH1 silu'(Z1); dW1 and db1 ----
        wait_mma();  // ... and dW3's MMAs: dz[0] and H2's buffer are free
        if (tile + gridDim.x < tiles) load_z(s.h[a ^ 1], z3g, (tile + gridDim.x) * kRows, n);
        cp_commit();
        data_gradient(s.dz[0], tlane + C_DH, row, c0, zl);
        bw_sync();
        if ((stopped = failed())) break;
        if (tid == 0) {
#pragma unroll 1
            for (int ks = 0; ks < 8; ++ks)
                mma_bf16(tbase + C_W1, desc_cols<H / 8>(s.dz[0], ks), desc_cols<2>(s.xo, ks), id_w16,
                         !first || ks > 0);
            mma_commit(&s.mbar);
        }
        first = false;
        a ^= 1;
    }
    cp_wait<0>();
    if (!stopped && !first) wait_mma();  // the last tile's weight gradients
    tc_before_sync();
    __syncthreads();
    tc_after_sync();
    const bool ok = !failed();
    if (ok && !first) {
        // the CTA's weight gradients and bias sums into grad (once per CTA)
#pragma unroll 1
        for (int m = 0; m < 2; ++m) {
            float *g = grad + (m == 0 ? W2_OFF : W3_OFF) + row * H + c0;
            float acc[32];
            tmem_ld32(tlane + (m == 0 ? C_W2 : C_W3) + (uint32_t)c0, acc);
#pragma unroll
            for (int q = 0; q < 8; ++q)
                atomicAdd(reinterpret_cast<float4 *>(g) + q,
                          make_float4(acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]));
        }
        float *gb = grad + W_COUNT;
        if (quarter < 2) {
            float acc[32];  // quarter 0: columns 384-415 (dW1 row | dW4^T row); 1: 416-447 (db3 | db2)
            tmem_ld32(tlane + (quarter == 0 ? C_W1 : C_B3), acc);
            if (quarter == 0) {
#pragma unroll
                for (int q = 0; q < IN / 4; ++q)
                    atomicAdd(reinterpret_cast<float4 *>(grad + W1_OFF + row * K1) + q,
                              make_float4(acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]));
                atomicAdd(gb + B1_OFF + row, acc[kOne]);
#pragma unroll
                for (int o = 0; o < N4; ++o) atomicAdd(grad + W4_OFF + o * H + row, acc[16 + o]);
            } else {
                atomicAdd(gb + B3_OFF + row, acc[kOne]);
                atomicAdd(gb + B2_OFF + row, acc[16 + kOne]);
            }
        }
        if (quarter == 0) {
#pragma unroll
            for (int c = 0; c < N4; ++c) {
                float v = db4[c];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                if (lane == 0) atomicAdd(gb + B4_OFF + c, v);
            }
        }
    }
    if (!ok && tid == 0) {
        atomicOr(err, 1);
        // before the tensor memory is released, a bounded grace wait for the MMAs in flight:
        // for the commit whose wait ran out, and for those issued since
        mma_commit(&s.mbar);
        mbar_wait(&s.mbar, phase ^ 1u);
        mbar_wait(&s.mbar, phase);
    }
    tc_before_sync();
    __syncthreads();
    tc_after_sync();
    if (warp == 0) {
        __syncwarp();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tbase), "r"(kBwCols)
                     : "memory");
    }
}

}  // namespace mlpbw

// all of an SM's shared memory: a second CTA could not have tensor memory anyway
int64_t mlp_bw_tc_smem_bytes() {
    static_assert(sizeof(mlpbw::BwSmem) <= 227 * 1024, "shared memory of one CTA");
    return 227 * 1024;
}

cudaError_t launch_mlp_backward_tc(const void *params, const float *x, const void *zsave, const void *dy,
                                   float *grad, int64_t n, int *err, int num_sms, cudaStream_t stream) {
    using namespace mlpbw;
    if (n <= 0) return cudaSuccess;
    static bool attr_set[64] = {false};
    const int bytes = (int)mlp_bw_tc_smem_bytes();
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64 || !attr_set[dev]) {
        e = cudaFuncSetAttribute(mlp_backward_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) attr_set[dev] = true;
    }
    const __nv_bfloat16 *w = static_cast<const __nv_bfloat16 *>(params);
    const int64_t tiles = (n + kRows - 1) / kRows;
    // one CTA per SM (each holds all 512 tensor-memory columns)
    const int grid = (int)(tiles < (int64_t)num_sms ? tiles : (int64_t)num_sms);
    launch_chained(mlp_backward_tc_kernel, grid, kBwThreads, bytes, stream, w, x,
                   static_cast<const __nv_bfloat16 *>(zsave), static_cast<const __nv_bfloat16 *>(dy), grad, n, err);
    return cudaGetLastError();
}

}  // namespace mpm
