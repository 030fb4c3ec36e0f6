// Weight gradient of a 3x3 convolution (stride 1, zero padding 1) of NHWC BF16 tensors on the
// tcgen05 tensor cores:
//   dW[co, tap, ci] = sum_p dz[p, co] x[p + off(tap), ci]
// as D[co, (dx, dy, ci)] = A^T B with the pixels p as the contraction: A = dz and B = x shifted
// by the tap, both as they lie in memory (channels contiguous), which the tensor core reads as
// M- and N-major operands; nothing is transposed or copied.
//
// A CTA takes 32 (or 16) input channels and every output channel, and walks the pixel tiles
// t = blockIdx.x, + gridDim.x, ... of 16 x 8 pixels.  Per tile, TMA brings dz (one box of 128
// pixels per 32 channels) and three boxes of x of 18 x 8 pixels, one per dx, zero-filled outside
// the image.  8 pixels of an image row are one swizzle atom, so 16 pixels of the contraction are
// two atoms, and the three dy are the same box started 0, 1 or 2 atoms further: one MMA of
// N = 3 * 32 covers them (the operand's N blocks lie one atom apart, as its K blocks do).  The
// 9 * 32 columns of all taps stay in tensor memory over the CTA's tiles, and each CTA writes
// one partial sum, added over the CTAs by k_sum_parts in a fixed order.
//   warp 4: TMA producer; warp 5: MMA issuer (24 instructions of 128 x 96 x 16 a tile);
//   warps 0-3: the bias gradient from the dz tiles in shared memory (first channel block only),
//   then the epilogue.
// Fewer than 128 output channels leave rows of D unused: the instruction reads what lies behind
// the dz boxes for them (other boxes, and kWgBehind bytes kept after the last stage), and they are
// not written.
// Bound: the MMAs, 24 x about 90 cycles a tile and channel block (the narrow N and the unused
// rows cost up to 4x the useful products at 32 channels).  Four images of 256 x 256, all ten
// layers: CUDA-core sums over 32 x 32 blocks 8.40 ms, 0.29 ms so.
#pragma once
#include "unet_conv.cuh"

namespace lica {
namespace unet {

constexpr int kWgThreads = 192;
constexpr int kWgMaxStages = 6;
constexpr int kWgDzBox = kTileM * 64;   // bytes of a dz box: 128 pixels x 32 channels
constexpr int kWgBehind = 4 * kWgDzBox; // room behind the last stage for the unused rows' reads

struct WgradParams {
    int h, w, tiles;      // image size, pixel tiles of the launch
    int cout, ctot;
    int cblk;             // input channels of a block: 32 or 16
    int c0;               // channels of the first input
    int nstages, stage;   // ring stages and bytes of one
    float* part;          // [gridDim.x][cout][9][ctot]
    float* bpart;         // [gridDim.x][cout]
    int* err;
};

// M- or N-major swizzled operand of rows (one pixel's channels) of 64 or 32 bytes: row blocks of
// that many bytes lie mn bytes apart along M or N, groups of 8 pixels k bytes apart.
__device__ __forceinline__ uint64_t mn_desc(uint32_t addr, uint32_t row_bytes, uint32_t mn, uint32_t k) {
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)(mn >> 4) << 16;
    d |= (uint64_t)(k >> 4) << 32;
    d |= 1ull << 46;
    d |= (row_bytes == 64 ? 4ull : 6ull) << 61;
    return d;
}

__global__ void __launch_bounds__(kWgThreads, 1)
    k_wgrad3x3(const __grid_constant__ CUtensorMap tm_dz, const __grid_constant__ CUtensorMap tm_x0,
               const __grid_constant__ CUtensorMap tm_x1, const WgradParams P) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    __shared__ uint64_t full[kWgMaxStages], empty[kWgMaxStages], done;
    __shared__ uint32_t tmem_slot;
    __shared__ float sbias[4][128];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int NS = P.nstages, nco = P.cout / 32;
    const bool bias = blockIdx.y == 0;
    if (threadIdx.x == 0) {
        for (int s = 0; s < NS; ++s) {
            tc::mbar_init(&full[s], 1);
            tc::mbar_init(&empty[s], bias ? 5 : 1);   // the MMAs, and the four warps that sum dz
        }
        tc::mbar_init(&done, 1);
        tc::fence_barrier_init();
    }
    after_previous();  // before the tensor memory is taken
    if (warp == 0) tc::tmem_alloc(&tmem_slot, 512);
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = tmem_slot;
    const int ci0 = (int)blockIdx.y * P.cblk;
    const int row = 2 * P.cblk;                        // bytes of a pixel of x
    const int dz_bytes = nco * kWgDzBox, xbox = kHaloRows * row;
    const int ncol = 3 * P.cblk;                       // columns of one dx

    if (warp == 4) {
        int s = 0;
        uint32_t ph = 0;
        const void* tmx = ci0 < P.c0 ? (const void*)&tm_x0 : (const void*)&tm_x1;
        const int cx = ci0 < P.c0 ? ci0 : ci0 - P.c0;
        int g = 0;
        for (int t = blockIdx.x; t < P.tiles; t += gridDim.x, ++g) {
            if (g >= NS && !tc::mbar_wait_warp(&empty[s], ph ^ 1u, lane)) {
                if (lane == 0) atomicExch(P.err, 1);
                break;
            }
            const int tiles_x = P.w / kTileW, tiles_y = P.h / kTileH;
            const int x0 = (t % tiles_x) * kTileW, y0 = (t / tiles_x) % tiles_y * kTileH, img = t / (tiles_x * tiles_y);
            if (tc::elect_one()) {
                unsigned char* st = base + s * P.stage;
                tc::mbar_expect_tx(&full[s], (uint32_t)(dz_bytes + 3 * xbox));
                for (int b = 0; b < nco; ++b) tc::tma_load_4d(st + b * kWgDzBox, &tm_dz, &full[s], 32 * b, x0, y0, img);
                for (int dx = 0; dx < 3; ++dx)
                    tc::tma_load_4d(st + dz_bytes + dx * xbox, tmx, &full[s], cx, x0 + dx - 1, y0 - 1, img);
            }
            __syncwarp();
            if (++s == NS) {
                s = 0;
                ph ^= 1u;
            }
        }
    } else if (warp == 5) {
        // both operands M-/N-major: bits 15 and 16
        const uint32_t idesc = tc::idesc_bf16_f32(128, (uint32_t)ncol) | (1u << 15) | (1u << 16);
        const uint32_t atom = 8u * (uint32_t)row;
        int s = 0;
        uint32_t ph = 0;
        for (int t = blockIdx.x; t < P.tiles; t += gridDim.x) {
            if (!tc::mbar_wait_warp(&full[s], ph, lane)) {
                if (lane == 0) atomicExch(P.err, 1);
                break;
            }
            const uint32_t st = tc::smem_u32(base + s * P.stage);
            const uint64_t a0 = mn_desc(st, 64, (uint32_t)kWgDzBox, 512);
            const uint64_t b0 = mn_desc(st + (uint32_t)dz_bytes, (uint32_t)row, atom, atom);
            if (tc::elect_one()) {
#pragma unroll 1
                for (int k = 0; k < kTileM / 16; ++k)
#pragma unroll
                    for (int dx = 0; dx < 3; ++dx)
                        tc::mma_bf16(tmem + (uint32_t)(dx * ncol), a0 + (uint32_t)(k * 1024 / 16),
                                     b0 + (uint32_t)(dx * xbox) / 16u + (uint32_t)k * (2u * atom / 16u), idesc,
                                     t != (int)blockIdx.x || k != 0);
                tc::mma_commit(&empty[s]);
            }
            __syncwarp();
            if (++s == NS) {
                s = 0;
                ph ^= 1u;
            }
        }
        if (tc::elect_one()) tc::mma_commit(&done);
        __syncwarp();
    } else {
        if (bias) {
            // thread = 8 channels (one 16-byte chunk of 4) of every 32-channel box, pixels p, p + 32, ...
            float acc[4][8];
#pragma unroll
            for (int b = 0; b < 4; ++b)
#pragma unroll
                for (int q = 0; q < 8; ++q) acc[b][q] = 0.f;
            const int chunk = threadIdx.x & 3, p0 = threadIdx.x >> 2;
            int s = 0;
            uint32_t ph = 0;
            for (int t = blockIdx.x; t < P.tiles; t += gridDim.x) {
                if (!tc::mbar_wait_warp(&full[s], ph, lane)) {
                    if (lane == 0) atomicExch(P.err, 1);
                    break;
                }
                const unsigned char* st = base + s * P.stage;
#pragma unroll
                for (int b = 0; b < 4; ++b)
                    if (b < nco)
                        for (int p = p0; p < kTileM; p += 32) {
                            // the 64-byte swizzle: address bits 4-5 exclusive-or bits 7-8
                            const uint4 v = *reinterpret_cast<const uint4*>(st + b * kWgDzBox + p * 64 +
                                                                            ((chunk ^ ((p >> 1) & 3)) << 4));
                            const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                            for (int q = 0; q < 4; ++q) {
                                acc[b][2 * q] += __uint_as_float(u[q] << 16);
                                acc[b][2 * q + 1] += __uint_as_float(u[q] & 0xffff0000u);
                            }
                        }
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(&empty[s]);
                if (++s == NS) {
                    s = 0;
                    ph ^= 1u;
                }
            }
            // over the 8 pixels groups of a warp (lanes of one chunk are 4 apart), then the warps
#pragma unroll
            for (int b = 0; b < 4; ++b)
                if (b < nco)
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        float v = acc[b][q];
                        for (int o = 16; o >= 4; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                        if (lane < 4) sbias[warp][32 * b + 8 * chunk + q] = v;
                    }
            asm volatile("bar.sync 1, 128;" ::: "memory");
            if ((int)threadIdx.x < P.cout)
                P.bpart[(size_t)blockIdx.x * P.cout + threadIdx.x] =
                    (sbias[0][threadIdx.x] + sbias[1][threadIdx.x]) + (sbias[2][threadIdx.x] + sbias[3][threadIdx.x]);
        }
        if (!tc::mbar_wait_warp(&done, 0, lane)) {
            if (lane == 0) atomicExch(P.err, 1);
        } else if (32 * warp < P.cout) {
            tc::tc_fence_after();
            const int co = 32 * warp + lane;
            float* dst = P.part + ((size_t)blockIdx.x * P.cout + co) * 9 * P.ctot + ci0;
            const uint32_t taddr = tmem + ((uint32_t)(32 * warp) << 16);
            for (int dx = 0; dx < 3; ++dx)
                for (int dy = 0; dy < 3; ++dy) {
                    float* d = dst + (3 * dy + dx) * P.ctot;
                    for (int c = 0; c < P.cblk; c += 16) {
                        float v[16];
                        tc::tmem_ld16(taddr + (uint32_t)(dx * ncol + dy * P.cblk + c), v);
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            *reinterpret_cast<float4*>(d + c + 4 * q) =
                                make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
                    }
                }
        }
        tc::tc_fence_before();
    }
    __syncwarp();
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc::tc_fence_after();
        tc::tmem_dealloc(tmem, 512);
    }
}

}  // namespace unet
}  // namespace lica
