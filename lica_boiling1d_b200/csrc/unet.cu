// Learned initial guess of the pressure solve: the convolution primitive of the U-Net on
// the tcgen05 tensor cores and its host plumbing (TMA tensor maps, launch shapes).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <vector>

#include "common.cuh"
#include "unet_conv.cuh"
#include "unet_wgrad.cuh"

extern "C" void lica_count_launches(int64_t n);

using namespace lica;
using namespace lica::unet;

namespace {

// Shared-memory limits of the tensor-core kernels, set once for each device (they are the device's),
// and the SMs of the current one.
constexpr int kMaxDevices = 64;
constexpr int kConvSmemMax = 227 * 1024, kWgSmemMax = 220 * 1024;
cudaError_t device_setup(int& sms) {
    struct Device {
        std::once_flag once;
        cudaError_t err = cudaSuccess;
        int sms = 1;
    };
    static Device devices[kMaxDevices];
    int dev = 0;
    const cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev >= kMaxDevices) return cudaErrorInvalidDevice;
    Device& d = devices[dev];
    std::call_once(d.once, [&d, dev] {
        d.err = cudaFuncSetAttribute(k_conv3x3_tcp, cudaFuncAttributeMaxDynamicSharedMemorySize, kConvSmemMax);
        if (d.err == cudaSuccess)
            d.err = cudaFuncSetAttribute(k_wgrad3x3, cudaFuncAttributeMaxDynamicSharedMemorySize, kWgSmemMax);
        if (d.err == cudaSuccess) d.err = cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev);
    });
    sms = d.sms;
    return d.err;
}

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    });
    return fn;
}

CUtensorMapSwizzle swizzle_for(int row_bytes) {
    return row_bytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B
                            : (row_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
}

// NHWC BF16 activations (c channels): box = cblk channels x tw x th pixels of one image.
int act_map(CUtensorMap* m, const void* p, int c, int w, int h, int n, int cblk, int tw, int th) {
    auto fn = encode_fn();
    if (!fn) {
        lica_set_last_error("cuTensorMapEncodeTiled", "driver entry point unavailable", __FILE__, __LINE__);
        return LICA_ERR_CUDA;
    }
    cuuint64_t dims[4] = {(cuuint64_t)c, (cuuint64_t)w, (cuuint64_t)h, (cuuint64_t)n};
    cuuint64_t strides[3] = {(cuuint64_t)c * 2, (cuuint64_t)c * w * 2, (cuuint64_t)c * w * h * 2};
    cuuint32_t box[4] = {(cuuint32_t)cblk, (cuuint32_t)tw, (cuuint32_t)th, 1};
    cuuint32_t es[4] = {1, 1, 1, 1};
    CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(p), dims, strides, box, es,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle_for(cblk * 2), CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        lica_set_last_error("cuTensorMapEncodeTiled", "activation map rejected", __FILE__, __LINE__);
        return LICA_BAD_ARG;
    }
    return LICA_OK;
}

// Weight matrix cout x ktot (BF16, K contiguous): box = cblk columns x cout rows.
int weight_map(CUtensorMap* m, const void* p, int ktot, int cout, int cblk) {
    auto fn = encode_fn();
    if (!fn) {
        lica_set_last_error("cuTensorMapEncodeTiled", "driver entry point unavailable", __FILE__, __LINE__);
        return LICA_ERR_CUDA;
    }
    cuuint64_t dims[2] = {(cuuint64_t)ktot, (cuuint64_t)cout};
    cuuint64_t strides[1] = {(cuuint64_t)ktot * 2};
    cuuint32_t box[2] = {(cuuint32_t)cblk, (cuuint32_t)cout};
    cuuint32_t es[2] = {1, 1};
    CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(p), dims, strides, box, es,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle_for(cblk * 2), CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        lica_set_last_error("cuTensorMapEncodeTiled", "weight map rejected", __FILE__, __LINE__);
        return LICA_BAD_ARG;
    }
    return LICA_OK;
}

int channel_block(int c) { return (c % 64 == 0) ? 64 : ((c % 32 == 0) ? 32 : 16); }

int tmem_columns(int cout) {
    int c = 32;
    while (c < cout) c *= 2;
    return c;
}

bool aligned16(const void* p) { return ((uintptr_t)p & 15u) == 0; }

}  // namespace

namespace lica {
namespace unet {

// Fused consumers of a convolution's BF16 output (see ConvParams).
struct ConvFuse {
    __nv_bfloat16* pool = nullptr;
    const float* head_w = nullptr;
    float* head_out = nullptr;
    double* head_x0 = nullptr;
    const double* head_rho = nullptr;
    const double* head_sigma = nullptr;
    double hsq = 0.0;
};

// out[:, :, :, out_c0 : out_c0 + cout] = conv3x3([x0, x1]) (+ bias, ReLU), NHWC BF16.
int conv3x3(const __nv_bfloat16* x0, int c0, const __nv_bfloat16* x1, int c1, const __nv_bfloat16* w,
            const float* bias, int n, int h, int wd, int cout, int relu, __nv_bfloat16* out, float* out32, int out_c,
            int out_c0, int* err, cudaStream_t s, const ConvFuse* fuse = nullptr) {
    if (n < 1 || h < 1 || wd < 1 || c0 <= 0 || c0 % 16 || c1 < 0 || c1 % 16 || (c1 > 0 && !x1) || cout < 16 ||
        cout > 256 || cout % 16 || out_c0 < 0 || out_c0 % 8 || out_c % 8 || out_c0 + cout > out_c) {
        lica_set_last_error("lica_unet_conv3x3", "unsupported channel counts", __FILE__, __LINE__);
        return LICA_BAD_ARG;
    }
    if (!aligned16(x0) || (x1 && !aligned16(x1)) || !aligned16(w) || (out && !aligned16(out)) ||
        (out32 && !aligned16(out32))) {
        lica_set_last_error("lica_unet_conv3x3", "arrays must be 16-byte aligned", __FILE__, __LINE__);
        return LICA_BAD_ARG;
    }
    const int tw = kTileW, th = kTileH;
    if (wd % tw || h % th) {
        lica_set_last_error("lica_unet_conv3x3", "image width must be a multiple of 8 and height of 16", __FILE__,
                            __LINE__);
        return LICA_BAD_ARG;
    }
    int num_sms = 0;
    LICA_CUDA_TRY(device_setup(num_sms));
    ConvParams P{};
    P.n = n; P.h = h; P.w = wd; P.tw = tw; P.th = th;
    P.nsrc = c1 > 0 ? 2 : 1;
    P.cin[0] = c0; P.cin[1] = c1;
    P.cblk[0] = channel_block(c0); P.cblk[1] = c1 > 0 ? channel_block(c1) : 16;
    P.ctot = c0 + c1;
    P.cout = cout;
    P.tmem_cols = tmem_columns(cout);
    P.out_c = out_c; P.out_c0 = out_c0;
    P.relu = relu;
    P.bias = bias;
    P.out = out;
    P.out32 = out32;
    P.err = err;
    if (fuse) {
        if ((fuse->pool || fuse->head_w) && (cout > 64 || out_c0 != 0 || out_c != cout)) {
            lica_set_last_error("lica_unet_conv3x3", "fused pool/head need cout <= 64 and a dense output", __FILE__,
                                __LINE__);
            return LICA_BAD_ARG;
        }
        if (fuse->head_w && (cout != 32 || !fuse->head_out || (fuse->head_x0 && (!fuse->head_rho || !fuse->head_sigma)))) {
            lica_set_last_error("lica_unet_conv3x3", "fused head needs 32 channels and its outputs", __FILE__,
                                __LINE__);
            return LICA_BAD_ARG;
        }
        P.pool = fuse->pool;
        P.head_w = fuse->head_w;
        P.head_out = fuse->head_out;
        P.head_x0 = fuse->head_x0;
        P.head_rho = fuse->head_rho;
        P.head_sigma = fuse->head_sigma;
        P.hsq = fuse->hsq;
    }
    const int cbmax = std::max(P.cblk[0], P.nsrc > 1 ? P.cblk[1] : 0);
    const auto round_kb = [](int b) { return ((b + 1023) / 1024) * 1024; };
    // Resident weights: the whole cout x (9 ctot) matrix (one box per tap, input and
    // channel block) stays in shared memory for all tiles of the CTA when it fits beside
    // the ring and every box starts on its swizzle atom; the ring then carries only the
    // activation boxes.
    const int wres = 18 * cout * P.ctot;
    const int avail = kConvSmemMax - 1024 - kBarBytes - kBiasBytes;
    const auto boxes_aligned = [&](bool wide) {
        for (int tap = 0; tap < 9; ++tap)
            for (int src = 0; src < P.nsrc; ++src)
                for (int c = src ? c0 : 0; c < (src ? P.ctot : c0); c += P.cblk[src]) {
                    const int at = wide ? 3 * (tap / 3) * P.ctot + 3 * c + (tap % 3) * P.cblk[src] : tap * P.ctot + c;
                    if ((2 * cout * at) % (16 * P.cblk[src])) return false;
                }
        return true;
    };
    // wide mode (N = 3 cout): resident weights beside at least two window stages.  Chosen
    // for 32 output channels from at least 64 input channels, where one N = 96 MMA
    // replaces three N = 32 ones and the tile's 9 ctot / 16 of them dominate; for fewer
    // input channels or 64 outputs the 14-column tiles and the shifted-sum epilogue cost
    // more than they save.
    const int stage_w = round_kb(kWideRows * cbmax * 2);
    P.stage_a = round_kb(kHaloRows * cbmax * 2);
    if (cout == 32 && P.ctot >= 64 && wd >= kWideBoxW && h >= kWideBoxH && avail - wres >= 2 * stage_w && boxes_aligned(true)) {
        P.wide = 1;
        P.tw = kWideTileW;
        P.th = kWideTileH;
        P.tmem_cols = tmem_columns(3 * cout);
        P.wres = wres;
        P.stage_a = stage_w;
        P.stage_b = 0;
        P.kdx = 3;
        P.nstages = std::min<int>(kStages, (avail - wres) / stage_w);
    } else if (avail - wres >= 3 * P.stage_a && boxes_aligned(false)) {
        P.wres = wres;
        P.stage_b = 0;
        // all three dx boxes per stage when at least two such stages fit
        const int stage3 = round_kb(3 * kHaloRows * cbmax * 2);
        if ((avail - wres) / stage3 >= 2) {
            P.kdx = 3;
            P.stage_a = stage3;
        } else {
            P.kdx = 1;
        }
        P.nstages = std::min<int>(kStages, (avail - wres) / P.stage_a);
    } else {
        P.wres = 0;
        P.kdx = 1;
        P.stage_b = round_kb(3 * cout * cbmax * 2);
        P.nstages = std::min<int>(kStages, avail / (P.stage_a + P.stage_b));
    }
    const int box_w = P.wide ? kWideBoxW : tw, box_h = P.wide ? kWideBoxH : th + 2;
    CUtensorMap mx0, mx1, mw0, mw1;
    int st;
    if ((st = act_map(&mx0, x0, c0, wd, h, n, P.cblk[0], box_w, box_h))) return st;
    if ((st = weight_map(&mw0, w, 9 * P.ctot, cout, P.cblk[0]))) return st;
    if (P.nsrc > 1) {
        if ((st = act_map(&mx1, x1, c1, wd, h, n, P.cblk[1], box_w, box_h))) return st;
        if ((st = weight_map(&mw1, w, 9 * P.ctot, cout, P.cblk[1]))) return st;
    } else {
        mx1 = mx0;
        mw1 = mw0;
    }
    const int tiles = n * (h / P.th) * ((wd + P.tw - 1) / P.tw);
    P.tiles = tiles;
    if (P.nstages < 1) return LICA_BAD_ARG;
    const size_t smem = conv_p_smem_bytes(P.stage_a, P.stage_b, P.nstages, P.wres);
    // CTAs per SM: shared memory and tensor memory (two accumulators of tmem_cols each)
    int per_sm = 0;
    LICA_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_conv3x3_tcp, kConvThreads, smem));
    per_sm = std::max(1, std::min(per_sm, 512 / (2 * P.tmem_cols)));
    const int grid = std::min(tiles, per_sm * num_sms);
    LICA_CUDA_TRY(launch_next(k_conv3x3_tcp, grid, kConvThreads, smem, s, mx0, mx1, mw0, mw1, P));
    lica_count_launches(1);
    return LICA_OK;
}

}  // namespace unet
}  // namespace lica

extern "C" {

int lica_unet_conv3x3_device(const void* x0, int32_t c0, const void* x1, int32_t c1, const void* w, const float* bias,
                             int32_t n, int32_t h, int32_t wd, int32_t cout, int32_t relu, void* out, float* out32,
                             int32_t out_c, int32_t out_c0, int32_t* err, void* stream) {
    if (!x0 || !w || !err || (!out && !out32)) return LICA_BAD_ARG;
    return lica::unet::conv3x3((const __nv_bfloat16*)x0, c0, (const __nv_bfloat16*)x1, c1,
                               (const __nv_bfloat16*)w, bias, n, h, wd, cout, relu, (__nv_bfloat16*)out, out32, out_c,
                               out_c0, err, (cudaStream_t)stream, nullptr);
}

}  // extern "C"

// ====================================================================================
// The U-Net of the learned initial guess.
//
// Input (per image, h x w): channel 0 = log10(rho) / 3, channel 1 = f / sigma with
// sigma = sqrt(mean f^2); channels 2..15 zero (the tensor-core K step is 16 channels).
// Levels 0, 1, 2 at h x w, h/2 x w/2, h/4 x w/4 with 32, 64, 128 channels:
//   L0 x16 -> e1a   L1 e1a -> e1b            pool -> p1
//   L2 p1 -> e2a    L3 e2a -> e2b            pool -> p2
//   L4 p2 -> e3a    L5 e3a -> e3b            up   -> u2
//   L6 [u2, e2b] -> d2a   L7 d2a -> d2b      up   -> u1
//   L8 [u1, e1b] -> d1a   L9 d1a -> d1b
//   head: out = wh . d1b + bh (1x1), guess x0 = out * sigma * h^2 * rho
// 3x3 convolutions with bias and ReLU, 2x2 average pooling, nearest upsampling.
// Training loss: the guess's relative residual squared, ||f - A x0||^2 / ||f||^2, with A
// the pressure operator of the multigrid solver (averaged over the images).
// ====================================================================================
namespace {

struct LayerDef {
    int cin0, cin1, cout, level;
};
constexpr int kLayers = 10;
constexpr LayerDef kNet[kLayers] = {{16, 0, 32, 0},  {32, 0, 32, 0},   {32, 0, 64, 1},  {64, 0, 64, 1},
                                    {64, 0, 128, 2}, {128, 0, 128, 2}, {128, 64, 64, 1}, {64, 0, 64, 1},
                                    {64, 32, 32, 0}, {32, 0, 32, 0}};
constexpr int kHead = 32;
constexpr int kIn = 16;
constexpr int kNT = 256;

using bf16 = __nv_bfloat16;

// ---------------------------------------------------------------- elementwise kernels
// sigma[n] = sqrt(mean f^2) of each image: kRmsParts blocks per image write partial
// sums, one block per image adds them (fixed order).
constexpr int kRmsParts = 512;
__global__ void k_rms_part(const double* __restrict__ f, double* __restrict__ part, int npix) {
    __shared__ double red[32];
    const double* fi = f + (size_t)blockIdx.y * npix;
    double s = 0.0;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < npix; k += gridDim.x * blockDim.x) s += fi[k] * fi[k];
    s = block_sum(s, red);
    if (threadIdx.x == 0) part[blockIdx.y * kRmsParts + blockIdx.x] = s;
}
__global__ void k_rms_final(const double* part, double* __restrict__ sigma, int npix) {
    after_previous();
    __shared__ double red[32];
    double s = 0.0;
    for (int k = threadIdx.x; k < kRmsParts; k += blockDim.x) s += part[blockIdx.x * kRmsParts + k];
    s = block_sum(s, red);
    if (threadIdx.x == 0) {
        const double m = s / npix;
        sigma[blockIdx.x] = m > 0.0 ? sqrt(m) : 1.0;
    }
}

__global__ void k_input(const double* rho, const double* f, const double* sigma,
                        bf16* __restrict__ x, int npix, int nimg) {
    after_previous();
    const size_t total = (size_t)npix * nimg;
    for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < total; p += (size_t)gridDim.x * blockDim.x) {
        const int img = (int)(p / npix);
        __align__(16) bf16 v[kIn];
        v[0] = __float2bfloat16_rn((float)(log10(rho[p]) / 3.0));
        v[1] = __float2bfloat16_rn((float)(f[p] / sigma[img]));
#pragma unroll
        for (int c = 2; c < kIn; ++c) v[c] = __float2bfloat16_rn(0.f);
        uint4* d = reinterpret_cast<uint4*>(x + p * kIn);
        d[0] = reinterpret_cast<const uint4*>(v)[0];
        d[1] = reinterpret_cast<const uint4*>(v)[1];
    }
}

// nearest upsampling x2 (H x W the output size): each thread copies one 8-channel group
// of an input pixel to its 2 x 2 output pixels.
__global__ void k_up(const bf16* in, bf16* __restrict__ out, int nimg, int H, int W, int c) {
    after_previous();
    const int c8 = c / 8, Hi = H / 2, Wi = W / 2;
    const size_t total = (size_t)nimg * Hi * Wi * c8;
    for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < total; q += (size_t)gridDim.x * blockDim.x) {
        const int ch = (int)(q % c8) * 8;
        const size_t r = q / c8;  // input pixel
        const int X = (int)(r % Wi);
        const size_t r2 = r / Wi;
        const int Y = (int)(r2 % Hi);
        const int img = (int)(r2 / Hi);
        const uint4 v = *reinterpret_cast<const uint4*>(in + r * c + ch);
        bf16* o = out + (((size_t)img * H + 2 * Y) * W + 2 * X) * c + ch;
        *reinterpret_cast<uint4*>(o) = v;
        *reinterpret_cast<uint4*>(o + c) = v;
        *reinterpret_cast<uint4*>(o + (size_t)W * c) = v;
        *reinterpret_cast<uint4*>(o + (size_t)W * c + c) = v;
    }
}

__device__ __forceinline__ float bf_lo(uint32_t u) { return __uint_as_float(u << 16); }
__device__ __forceinline__ float bf_hi(uint32_t u) { return __uint_as_float(u & 0xffff0000u); }
__device__ __forceinline__ uint32_t bf_pack(float lo, float hi) {
    const __nv_bfloat162 b = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&b);
}
// the gradients v of eight channels where the layer's output y is positive, in BF16
__device__ __forceinline__ uint4 relu_mask8(const float* v, const uint4 y) {
    const uint32_t u[4] = {y.x, y.y, y.z, y.w};
    uint32_t r[4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
        r[q] = bf_pack(bf_lo(u[q]) > 0.f ? v[2 * q] : 0.f, bf_hi(u[q]) > 0.f ? v[2 * q + 1] : 0.f);
    return make_uint4(r[0], r[1], r[2], r[3]);
}

// The head's backward pass, one sweep over d1b (d) and gout: per-block partial sums of its
// gradients, part[b][c] = sum gout * d1b[:, c] (c < 32), part[b][32] = sum gout, over the pixels of
// block b (fixed order), and dz = gout * wh through the last layer's ReLU.
__global__ void k_head_bwd(const float* gout, const float* wh, const bf16* d,
                           bf16* __restrict__ dz, float* __restrict__ part, size_t total) {
    after_previous();
    __shared__ float red[kNT / 32][kHead + 1];
    __shared__ float w[kHead];
    if (threadIdx.x < kHead) w[threadIdx.x] = wh[threadIdx.x];
    __syncthreads();
    float acc[kHead + 1];
#pragma unroll
    for (int c = 0; c <= kHead; ++c) acc[c] = 0.f;
    for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < total; p += (size_t)gridDim.x * blockDim.x) {
        const float g = gout[p];
        const uint4* src = reinterpret_cast<const uint4*>(d + p * kHead);
        uint4* dst = reinterpret_cast<uint4*>(dz + p * kHead);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint4 y = src[q];
            const uint32_t u[4] = {y.x, y.y, y.z, y.w};
            float v[8];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                acc[8 * q + 2 * i] += g * bf_lo(u[i]);
                acc[8 * q + 2 * i + 1] += g * bf_hi(u[i]);
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = g * w[8 * q + i];
            dst[q] = relu_mask8(v, y);
        }
        acc[kHead] += g;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int c = 0; c <= kHead; ++c) {
        float v = acc[c];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) red[warp][c] = v;
    }
    __syncthreads();
    if (threadIdx.x <= kHead) {
        float v = 0.f;
        for (int w_ = 0; w_ < kNT / 32; ++w_) v += red[w_][threadIdx.x];
        part[(size_t)blockIdx.x * (kHead + 1) + threadIdx.x] = v;
    }
}

// dz = g through the layer's ReLU (y > 0), eight channels a thread; g = the channel slice
// [g_c0, g_c0 + c) of a tensor with g_cs channels, plus (optionally) 0.25 * gp at the parent cell
// of a half-size tensor (pool backward).  H and W are the image's, c a multiple of 8.
__global__ void k_relu_bwd(const bf16* g, int g_cs, int g_c0, const bf16* gp,
                           const bf16* y, bf16* __restrict__ dz, int nimg, int H, int W, int c) {
    after_previous();
    const int c8 = c / 8;
    const size_t total = (size_t)nimg * H * W * c8;
    for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < total; q += (size_t)gridDim.x * blockDim.x) {
        const int ch = (int)(q % c8) * 8;
        const size_t pix = q / c8;
        const uint4 gv = *reinterpret_cast<const uint4*>(g + pix * g_cs + g_c0 + ch);
        const uint32_t u[4] = {gv.x, gv.y, gv.z, gv.w};
        float v[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            v[2 * i] = bf_lo(u[i]);
            v[2 * i + 1] = bf_hi(u[i]);
        }
        if (gp) {
            const int x = (int)(pix % W);
            const size_t r = pix / W;
            const int yy = (int)(r % H);
            const int img = (int)(r / H);
            const uint4 pv = *reinterpret_cast<const uint4*>(
                gp + (((size_t)img * (H / 2) + yy / 2) * (W / 2) + x / 2) * c + ch);
            const uint32_t w[4] = {pv.x, pv.y, pv.z, pv.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                v[2 * i] += 0.25f * bf_lo(w[i]);
                v[2 * i + 1] += 0.25f * bf_hi(w[i]);
            }
        }
        *reinterpret_cast<uint4*>(dz + pix * c + ch) =
            relu_mask8(v, *reinterpret_cast<const uint4*>(y + pix * c + ch));
    }
}

// Upsampling backward and the layer's ReLU: dz[n, Y, X, c] = the sum of the 4 children of g
// (channel slice [g_c0, g_c0 + c) of a tensor with g_cs channels), rounded to BF16, where y > 0.
__global__ void k_up_relu_bwd(const bf16* g, int g_cs, int g_c0, const bf16* y,
                              bf16* __restrict__ dz, int nimg, int Ho, int Wo, int c) {
    after_previous();
    const int c8 = c / 8, W = 2 * Wo;
    const size_t total = (size_t)nimg * Ho * Wo * c8;
    for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < total; q += (size_t)gridDim.x * blockDim.x) {
        const int ch = (int)(q % c8) * 8;
        const size_t pix = q / c8;
        const int X = (int)(pix % Wo);
        const size_t r = pix / Wo;
        const int Y = (int)(r % Ho);
        const int img = (int)(r / Ho);
        const bf16* b = g + (((size_t)img * 2 * Ho + 2 * Y) * W + 2 * X) * g_cs + g_c0 + ch;
        const uint4 c00 = *reinterpret_cast<const uint4*>(b), c01 = *reinterpret_cast<const uint4*>(b + g_cs),
                    c10 = *reinterpret_cast<const uint4*>(b + (size_t)W * g_cs),
                    c11 = *reinterpret_cast<const uint4*>(b + (size_t)W * g_cs + g_cs);
        const uint32_t p[4] = {c00.x, c00.y, c00.z, c00.w}, s[4] = {c01.x, c01.y, c01.z, c01.w},
                       t[4] = {c10.x, c10.y, c10.z, c10.w}, u[4] = {c11.x, c11.y, c11.z, c11.w};
        float v[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            v[2 * i] = (bf_lo(p[i]) + bf_lo(s[i])) + (bf_lo(t[i]) + bf_lo(u[i]));
            v[2 * i + 1] = (bf_hi(p[i]) + bf_hi(s[i])) + (bf_hi(t[i]) + bf_hi(u[i]));
        }
        *reinterpret_cast<uint4*>(dz + pix * c + ch) =
            relu_mask8(v, *reinterpret_cast<const uint4*>(y + pix * c + ch));
    }
}

// grad[k] = sum over chunks of part[chunk][k], for k < n, and the same of a second set (bpart, nb
// values to bgrad, may be empty): 8 threads per value take every 8th chunk, then add up in a
// fixed order.  Block: 32 values x 8 threads.
__global__ void __launch_bounds__(256) k_sum_parts(const float* part, int nchunk, size_t n,
                                                   float* __restrict__ grad, const float* bpart, size_t nb,
                                                   float* __restrict__ bgrad) {
    after_previous();
    __shared__ float red[8][33];
    const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
    const size_t blocks = (n + 31) / 32;
    const bool second = blockIdx.x >= blocks;
    const float* src = second ? bpart : part;
    const size_t len = second ? nb : n, k = (blockIdx.x - (second ? blocks : 0)) * 32 + x;
    float s = 0.f;
    if (k < len) {
#pragma unroll 4
        for (int c = y; c < nchunk; c += 8) s += src[(size_t)c * len + k];
    }
    red[y][x] = s;
    __syncthreads();
    if (y == 0 && k < len) {
        const float v = ((red[0][x] + red[1][x]) + (red[2][x] + red[3][x])) +
                        ((red[4][x] + red[5][x]) + (red[6][x] + red[7][x]));
        (second ? bgrad : grad)[k] = v;
    }
}
int sum_parts(const float* part, int nchunk, size_t n, float* grad, const float* bpart, size_t nb, float* bgrad,
              cudaStream_t s) {
    LICA_CUDA_TRY(launch_next(k_sum_parts, (unsigned)((n + 31) / 32 + (nb + 31) / 32), 256, 0, s, part, nchunk, n, grad, bpart,
                              nb, bgrad));
    lica_count_launches(1);
    return LICA_OK;
}

// Adam (FP32 master weights).
__global__ void k_adam(float* __restrict__ w, const float* g, float* __restrict__ m,
                       float* __restrict__ v, size_t n, float lr, float b1, float b2, float eps, float c1, float c2) {
    after_previous();
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) {
        const float gk = g[k];
        const float mk = b1 * m[k] + (1.f - b1) * gk;
        const float vk = b2 * v[k] + (1.f - b2) * gk * gk;
        m[k] = mk;
        v[k] = vk;
        w[k] -= lr * (mk / c1) / (sqrtf(vk / c2) + eps);
    }
}

// BF16 copies of a layer's weights: wb[co][tap][ci] = w, and the transposed, tap-flipped
// copy wf[ci][8 - tap][co] that turns the input-gradient into a forward convolution.
__global__ void k_pack(const float* __restrict__ w, bf16* __restrict__ wb, bf16* __restrict__ wf, int cout, int ctot) {
    const size_t n = (size_t)cout * 9 * ctot;
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) {
        const int ci = (int)(k % ctot);
        const size_t r = k / ctot;
        const int tap = (int)(r % 9);
        const int co = (int)(r / 9);
        const bf16 b = __float2bfloat16_rn(w[k]);
        wb[k] = b;
        wf[((size_t)ci * 9 + (8 - tap)) * cout + co] = b;
    }
}

// FP64 pressure operator of the solver: out = s - d*u (x periodic, bottom Neumann, top
// p = 0 on the face), the oracle's apply, for nimg images.
__global__ void k_apply_op(const double* u, const double* bx, const double* by,
                           double* __restrict__ out, int nimg, int ny, int nx, double cx, double cy) {
    after_previous();
    const size_t npix = (size_t)nx * ny, total = npix * nimg;
    for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < total; q += (size_t)gridDim.x * blockDim.x) {
        const size_t img = q / npix, k = q - img * npix;
        const int j = (int)(k / nx), i = (int)(k - (size_t)j * nx);
        const double* U = u + img * npix;
        const double* BX = bx + img * npix;
        const double* BY = by + img * (npix + nx);
        const int ip = (i + 1 == nx) ? 0 : i + 1, im = (i == 0) ? nx - 1 : i - 1;
        const double aw = cx * BX[k];
        const double ae = cx * BX[(size_t)j * nx + ip];
        const double as = (j > 0) ? cy * BY[k] : 0.0;
        const double an = (j < ny - 1) ? cy * BY[k + nx] : (2.0 * cy) * BY[k + nx];
        const double us = (j > 0) ? U[k - nx] : 0.0;
        const double un = (j < ny - 1) ? U[k + nx] : 0.0;
        double s = aw * U[(size_t)j * nx + im];
        s += ae * U[(size_t)j * nx + ip];
        s += as * us;
        s += an * un;
        double d = aw;
        d += ae;
        d += as;
        d += an;
        out[q] = s - d * U[k];
    }
}

// r = f - A x0 (in place over ax), and per-image ||r||^2 (one block per image).
// r = f - (A x0) in place and ||r||^2 per image: kRmsParts blocks per image write partial
// sums (k_part_sum adds them in a fixed order).
__global__ void k_residual(const double* __restrict__ f, double* __restrict__ r, double* __restrict__ part,
                           int npix) {
    __shared__ double red[32];
    const size_t off = (size_t)blockIdx.y * npix;
    double s = 0.0;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < npix; k += gridDim.x * blockDim.x) {
        const double v = f[off + k] - r[off + k];
        r[off + k] = v;
        s += v * v;
    }
    s = block_sum(s, red);
    if (threadIdx.x == 0) part[blockIdx.y * kRmsParts + blockIdx.x] = s;
}

// out[image] = the sum of its kRmsParts partial sums, in index order (one block per image).
__global__ void k_part_sum(const double* __restrict__ part, double* __restrict__ out) {
    __shared__ double red[32];
    double s = 0.0;
    for (int k = threadIdx.x; k < kRmsParts; k += blockDim.x) s += part[blockIdx.x * kRmsParts + k];
    s = block_sum(s, red);
    if (threadIdx.x == 0) out[blockIdx.x] = s;
}

// dL/dout = -2 (A r) sigma h^2 rho / (nimg ||f||^2), ||f||^2 = sigma^2 npix.
__global__ void k_gout(const double* ar, const double* sigma, const double* rho,
                       double hsq, float* __restrict__ gout, int npix, int nimg) {
    after_previous();
    const size_t total = (size_t)npix * nimg;
    for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < total; p += (size_t)gridDim.x * blockDim.x) {
        const double sg = sigma[p / npix];
        gout[p] = (float)(-2.0 * ar[p] * hsq * rho[p] / (sg * nimg * (double)npix));
    }
}

// A-norm loss with the solver's solution p*: e = x0 - p* (into x0's buffer), per image
// num = -e.(A e) (ae holds A e), den = -p*.f = p*.(-A p*), as kRmsParts partial sums per
// image (k_part_sum adds them).
__global__ void k_energy(const double* __restrict__ ae, const double* __restrict__ e, const double* __restrict__ ps,
                         const double* __restrict__ f, double* __restrict__ part_num, double* __restrict__ part_den,
                         int npix) {
    __shared__ double red[32];
    const size_t off = (size_t)blockIdx.y * npix;
    double a = 0.0, b = 0.0;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < npix; k += gridDim.x * blockDim.x) {
        a -= e[off + k] * ae[off + k];
        b -= ps[off + k] * f[off + k];
    }
    a = block_sum(a, red);
    b = block_sum(b, red);
    if (threadIdx.x == 0) {
        part_num[blockIdx.y * kRmsParts + blockIdx.x] = a;
        part_den[blockIdx.y * kRmsParts + blockIdx.x] = b;
    }
}

// dL/dout of L = mean_images num/den: -2 (A e) sigma h^2 rho / (nimg den).
__global__ void k_gout_energy(const double* ae, const double* den,
                              const double* sigma, const double* rho, double hsq,
                              float* __restrict__ gout, int npix, int nimg) {
    after_previous();
    const size_t total = (size_t)npix * nimg;
    for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < total; p += (size_t)gridDim.x * blockDim.x) {
        const size_t img = p / npix;
        gout[p] = (float)(-2.0 * ae[p] * sigma[img] * hsq * rho[p] / (nimg * den[img]));
    }
}

__global__ void k_sub(double* __restrict__ a, const double* b, size_t n) {
    after_previous();
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x)
        a[k] -= b[k];
}

// gout from a given dL/dx0 (the gradient check): gout = gx0 * sigma * h^2 * rho
__global__ void k_gout_from_gx(const double* gx, const double* sigma,
                               const double* rho, double hsq, float* __restrict__ gout, int npix,
                               int nimg) {
    after_previous();
    const size_t total = (size_t)npix * nimg;
    for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < total; p += (size_t)gridDim.x * blockDim.x)
        gout[p] = (float)(gx[p] * sigma[p / npix] * hsq * rho[p]);
}

int grid_for(size_t n) { return (int)std::min<size_t>(4 * 148 * 8, (n + kNT - 1) / kNT); }

// Deterministic normal deviates for the initial weights (splitmix64 + Box-Muller).
struct InitRng {
    uint64_t s;
    uint64_t next() {
        uint64_t z = (s += 0x9E3779B97F4A7C15ull);
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        return z ^ (z >> 31);
    }
    double uniform() { return ((next() >> 11) + 0.5) * (1.0 / 9007199254740992.0); }
    double normal() {
        const double u1 = uniform(), u2 = uniform();
        return sqrt(-2.0 * log(u1)) * cos(6.283185307179586 * u2);
    }
};

}  // namespace

// ---------------------------------------------------------------- host runtime
struct lica_unet {
    int n = 0, h = 0, w = 0;
    size_t nparams = 0;
    size_t woff[kLayers], boff[kLayers], hoff = 0;  // offsets into the FP32 parameter vector
    float* param = nullptr;                         // master weights (device)
    float* grad = nullptr;
    float* adam_m = nullptr;
    float* adam_v = nullptr;
    int adam_t = 0;
    bf16* wb[kLayers] = {};
    bf16* wf[kLayers] = {};
    // activations (NHWC BF16): x16, per layer output, pooled and upsampled tensors
    bf16* x16 = nullptr;
    bf16* y[kLayers] = {};
    bf16 *p1 = nullptr, *p2 = nullptr, *u2 = nullptr, *u1 = nullptr;
    float* out32 = nullptr;
    double* sigma = nullptr;
    double* rms_part = nullptr;
    double* x0 = nullptr;   // guess (training)
    double* ax = nullptr;   // A x0, then r, then A r
    double* rr = nullptr;   // per-image ||r||^2 (or the A-norm loss's numerator)
    double* den = nullptr;  // per-image A-norm of p*
    double* part2 = nullptr;  // the A-norm loss's second set of partial sums (kRmsParts per image)
    // training buffers
    bool train_ready = false;
    float* gout = nullptr;
    bf16* gin = nullptr;     // input gradient of a layer with one input
    bf16* gcat0 = nullptr;   // input gradients of the decoder layers, [upsampled | skip]: L8's (96 channels,
    bf16* gcat1 = nullptr;   // level 0) and L6's (192, level 1), kept for the encoder's layers
    bf16* dz = nullptr;      // a layer's output gradient through its ReLU
    float* part = nullptr;
    float* bpart = nullptr;
    size_t part_elems = 0;
    float* hpart = nullptr;
    int* err = nullptr;
};

namespace {

size_t level_pixels(const lica_unet* u, int level) { return (size_t)u->n * (u->h >> level) * (u->w >> level); }

template <typename T>
int dev_alloc(T** p, size_t count) {
    cudaError_t e = cudaMalloc((void**)p, sizeof(T) * std::max<size_t>(count, 1));
    if (e != cudaSuccess) {
        lica_set_last_error("cudaMalloc", cudaGetErrorString(e), __FILE__, __LINE__);
        return LICA_ERR_NOMEM;
    }
    return LICA_OK;
}

int pack_all(lica_unet* u, cudaStream_t s) {
    for (int l = 0; l < kLayers; ++l) {
        const LayerDef& L = kNet[l];
        const size_t n = (size_t)L.cout * 9 * (L.cin0 + L.cin1);
        k_pack<<<grid_for(n), kNT, 0, s>>>(u->param + u->woff[l], u->wb[l], u->wf[l], L.cout, L.cin0 + L.cin1);
        LICA_CUDA_TRY(cudaGetLastError());
    }
    lica_count_launches(kLayers);
    return LICA_OK;
}

int conv_layer(lica_unet* u, int l, const bf16* x0, const bf16* x1, bf16* out, cudaStream_t s,
               const ConvFuse* fuse = nullptr) {
    const LayerDef& L = kNet[l];
    return conv3x3(x0, L.cin0, x1, L.cin1, u->wb[l], u->param + u->boff[l], u->n, u->h >> L.level, u->w >> L.level,
                   L.cout, 1, out, nullptr, L.cout, 0, u->err, s, fuse);
}

template <typename K, typename... A>
int launch(size_t n, cudaStream_t s, K kernel, A... args) {
    LICA_CUDA_TRY(launch_next(kernel, grid_for(n), kNT, 0, s, args...));
    lica_count_launches(1);
    return LICA_OK;
}

// Forward pass: input tensor from (rho, f), every activation kept (the last one, d1b, only
// with keep_last: the head is fused into its convolution), the head output and the guess
// x0 (if given).  The 2x2 poolings are fused into the convolutions that produce e1b and e2b.
int forward(lica_unet* u, const double* rho, const double* f, double hsq, double* x0, cudaStream_t s,
            bool keep_last = true) {
    const int npix = u->h * u->w;
    int st;
    k_rms_part<<<dim3(kRmsParts, u->n), kNT, 0, s>>>(f, u->rms_part, npix);
    LICA_CUDA_TRY(cudaGetLastError());
    LICA_CUDA_TRY(launch_next(k_rms_final, u->n, kNT, 0, s, u->rms_part, u->sigma, npix));
    lica_count_launches(2);
    if ((st = launch(level_pixels(u, 0), s, k_input, rho, f, (const double*)u->sigma, u->x16, npix, u->n))) return st;
    const int h = u->h, w = u->w, n = u->n;
    ConvFuse pool1, pool2, head;
    pool1.pool = u->p1;
    pool2.pool = u->p2;
    head.head_w = u->param + u->hoff;
    head.head_out = u->out32;
    head.head_x0 = x0;
    head.head_rho = rho;
    head.head_sigma = u->sigma;
    head.hsq = hsq;
    if ((st = conv_layer(u, 0, u->x16, nullptr, u->y[0], s))) return st;
    if ((st = conv_layer(u, 1, u->y[0], nullptr, u->y[1], s, &pool1))) return st;
    if ((st = conv_layer(u, 2, u->p1, nullptr, u->y[2], s))) return st;
    if ((st = conv_layer(u, 3, u->y[2], nullptr, u->y[3], s, &pool2))) return st;
    if ((st = conv_layer(u, 4, u->p2, nullptr, u->y[4], s))) return st;
    if ((st = conv_layer(u, 5, u->y[4], nullptr, u->y[5], s))) return st;
    if ((st = launch(level_pixels(u, 2) * 16, s, k_up, (const bf16*)u->y[5], u->u2, n, h / 2, w / 2, 128))) return st;
    if ((st = conv_layer(u, 6, u->u2, u->y[3], u->y[6], s))) return st;
    if ((st = conv_layer(u, 7, u->y[6], nullptr, u->y[7], s))) return st;
    if ((st = launch(level_pixels(u, 1) * 8, s, k_up, (const bf16*)u->y[7], u->u1, n, h, w, 64))) return st;
    if ((st = conv_layer(u, 8, u->u1, u->y[1], u->y[8], s))) return st;
    return conv_layer(u, 9, u->y[8], nullptr, keep_last ? u->y[9] : nullptr, s, &head);
}

// CTAs along the pixels for a layer's weight gradient: one per SM over the blocks of input
// channels, at most one per pixel tile.
int wgrad_chunks(const lica_unet* u, int l, int sms) {
    const LayerDef& L = kNet[l];
    const int blocks = (L.cin0 + L.cin1) / (L.cin0 % 32 ? 16 : 32);
    const int tiles = (int)(level_pixels(u, L.level) / kTileM);
    return std::max(1, std::min(tiles, sms / blocks));
}

int alloc_training(lica_unet* u) {
    if (u->train_ready) return LICA_OK;
    const size_t p0 = level_pixels(u, 0), p1 = level_pixels(u, 1), p2 = level_pixels(u, 2);
    int st;
    if ((st = dev_alloc(&u->grad, u->nparams))) return st;
    if ((st = dev_alloc(&u->adam_m, u->nparams))) return st;
    if ((st = dev_alloc(&u->adam_v, u->nparams))) return st;
    LICA_CUDA_TRY(cudaMemset(u->adam_m, 0, sizeof(float) * u->nparams));
    LICA_CUDA_TRY(cudaMemset(u->adam_v, 0, sizeof(float) * u->nparams));
    const size_t one = std::max({p0 * 32, p1 * 64, p2 * 128});   // a layer's own channels at its level
    if ((st = dev_alloc(&u->gout, p0))) return st;
    if ((st = dev_alloc(&u->gin, one))) return st;
    if ((st = dev_alloc(&u->dz, one))) return st;
    if ((st = dev_alloc(&u->gcat0, p0 * 96))) return st;
    if ((st = dev_alloc(&u->gcat1, p1 * 192))) return st;
    // weight-gradient partials: the largest layer's chunks x weights
    size_t pe = 0, be = 0;
    int sms = 0;
    LICA_CUDA_TRY(device_setup(sms));
    for (int l = 0; l < kLayers; ++l) {
        const LayerDef& L = kNet[l];
        const size_t chunks = (size_t)wgrad_chunks(u, l, sms);
        pe = std::max(pe, chunks * L.cout * 9 * (L.cin0 + L.cin1));
        be = std::max(be, chunks * L.cout);
    }
    u->part_elems = pe;
    if ((st = dev_alloc(&u->part, pe))) return st;
    if ((st = dev_alloc(&u->bpart, be))) return st;
    if ((st = dev_alloc(&u->hpart, (size_t)grid_for(p0) * (kHead + 1)))) return st;
    u->train_ready = true;
    return LICA_OK;
}

// Weight and bias gradients of layer l from dz (its masked output gradient).
int layer_wgrad(lica_unet* u, int l, const bf16* x0, const bf16* x1, cudaStream_t s) {
    const LayerDef& L = kNet[l];
    const int H = u->h >> L.level, W = u->w >> L.level, ctot = L.cin0 + L.cin1;
    WgradParams P{};
    P.h = H;
    P.w = W;
    P.tiles = (int)(level_pixels(u, L.level) / kTileM);
    P.cout = L.cout;
    P.ctot = ctot;
    P.cblk = L.cin0 % 32 ? 16 : 32;
    P.c0 = L.cin0;
    P.stage = (L.cout / 32) * kWgDzBox + (3 * kHaloRows * 2 * P.cblk + 1023) / 1024 * 1024;
    P.nstages = std::min(kWgMaxStages, (kWgSmemMax - 1024 - kWgBehind) / P.stage);
    P.part = u->part;
    P.bpart = u->bpart;
    P.err = u->err;
    CUtensorMap mdz, m0, m1;
    int st;
    if ((st = act_map(&mdz, u->dz, L.cout, W, H, u->n, 32, kTileW, kTileH))) return st;
    if ((st = act_map(&m0, x0, L.cin0, W, H, u->n, P.cblk, kTileW, kTileH + 2))) return st;
    m1 = m0;
    if (L.cin1 && (st = act_map(&m1, x1, L.cin1, W, H, u->n, P.cblk, kTileW, kTileH + 2))) return st;
    int sms = 0;
    LICA_CUDA_TRY(device_setup(sms));
    const int chunks = wgrad_chunks(u, l, sms);
    LICA_CUDA_TRY(launch_next(k_wgrad3x3, dim3(chunks, ctot / P.cblk), kWgThreads, 1024 + P.nstages * P.stage + kWgBehind, s,
                              mdz, m0, m1, P));
    lica_count_launches(1);
    return sum_parts(u->part, chunks, (size_t)L.cout * 9 * ctot, u->grad + u->woff[l], u->bpart, (size_t)L.cout,
                     u->grad + u->boff[l], s);
}

// Input gradient of layer l: out = conv3x3(dz, wf) (channels [x0 | x1]).
int layer_igrad(lica_unet* u, int l, bf16* out, cudaStream_t s) {
    const LayerDef& L = kNet[l];
    const int ctot = L.cin0 + L.cin1;
    return conv3x3(u->dz, L.cout, nullptr, 0, u->wf[l], nullptr, u->n, u->h >> L.level, u->w >> L.level, ctot, 0,
                   out, nullptr, ctot, 0, u->err, s);
}

// dz = g (channel slice of a tensor) [+ pool backward of gp] masked by the layer's ReLU.
int relu_bwd(lica_unet* u, int l, const bf16* g, int g_cs, int g_c0, const bf16* gp, cudaStream_t s) {
    const LayerDef& L = kNet[l];
    const int H = u->h >> L.level, W = u->w >> L.level;
    return launch(level_pixels(u, L.level) * (L.cout / 8), s, k_relu_bwd, g, g_cs, g_c0, gp, (const bf16*)u->y[l], u->dz,
                  u->n, H, W, L.cout);
}

// dz = the upsampling's backward of a slice of g masked by the ReLU of layer l (before it).
int up_relu_bwd(lica_unet* u, int l, const bf16* g, int g_cs, cudaStream_t s) {
    const LayerDef& L = kNet[l];
    const int H = u->h >> L.level, W = u->w >> L.level;
    return launch(level_pixels(u, L.level) * (L.cout / 8), s, k_up_relu_bwd, g, g_cs, 0, (const bf16*)u->y[l], u->dz,
                  u->n, H, W, L.cout);
}

// Backward pass from gout (dL/d out32): every parameter gradient into u->grad.  Every pass over
// the activations between the convolutions reads and writes 16 bytes a thread, applies the next
// ReLU on the way, and takes the decoder's two input gradients where their convolutions left them
// (gcat1, gcat0): as separate passes of one value a thread with copies of the skip slices, they
// took 0.37 ms of four 256 x 256 images' 1.19, 0.08 so.
int backward(lica_unet* u, cudaStream_t s) {
    const size_t p0 = level_pixels(u, 0);
    int st;
    // head and the ReLU of L9
    const int hb = grid_for(p0);
    LICA_CUDA_TRY(launch_next(k_head_bwd, hb, kNT, 0, s, u->gout, u->param + u->hoff, u->y[9], u->dz, u->hpart, p0));
    lica_count_launches(1);
    if ((st = sum_parts(u->hpart, hb, (size_t)(kHead + 1), u->grad + u->hoff, nullptr, 0, nullptr, s))) return st;
    // L9 (input d1a)
    if ((st = layer_wgrad(u, 9, u->y[8], nullptr, s))) return st;
    if ((st = layer_igrad(u, 9, u->gin, s))) return st;  // d(d1a), 32 ch
    // L8 (inputs [u1 (64), e1b (32)])
    if ((st = relu_bwd(u, 8, u->gin, 32, 0, nullptr, s))) return st;
    if ((st = layer_wgrad(u, 8, u->u1, u->y[1], s))) return st;
    if ((st = layer_igrad(u, 8, u->gcat0, s))) return st;  // [d(u1) 64 | d(e1b) 32]
    // L7 (input d2a)
    if ((st = up_relu_bwd(u, 7, u->gcat0, 96, s))) return st;
    if ((st = layer_wgrad(u, 7, u->y[6], nullptr, s))) return st;
    if ((st = layer_igrad(u, 7, u->gin, s))) return st;  // d(d2a)
    // L6 (inputs [u2 (128), e2b (64)])
    if ((st = relu_bwd(u, 6, u->gin, 64, 0, nullptr, s))) return st;
    if ((st = layer_wgrad(u, 6, u->u2, u->y[3], s))) return st;
    if ((st = layer_igrad(u, 6, u->gcat1, s))) return st;  // [d(u2) 128 | d(e2b) 64]
    // L5 (input e3a)
    if ((st = up_relu_bwd(u, 5, u->gcat1, 192, s))) return st;
    if ((st = layer_wgrad(u, 5, u->y[4], nullptr, s))) return st;
    if ((st = layer_igrad(u, 5, u->gin, s))) return st;  // d(e3a)
    // L4 (input p2)
    if ((st = relu_bwd(u, 4, u->gin, 128, 0, nullptr, s))) return st;
    if ((st = layer_wgrad(u, 4, u->p2, nullptr, s))) return st;
    if ((st = layer_igrad(u, 4, u->gin, s))) return st;  // d(p2), 64 ch at level 2
    // L3 (input e2a): d(e2b) = decoder part + pool backward of d(p2)
    if ((st = relu_bwd(u, 3, u->gcat1, 192, 128, u->gin, s))) return st;
    if ((st = layer_wgrad(u, 3, u->y[2], nullptr, s))) return st;
    if ((st = layer_igrad(u, 3, u->gin, s))) return st;  // d(e2a)
    // L2 (input p1)
    if ((st = relu_bwd(u, 2, u->gin, 64, 0, nullptr, s))) return st;
    if ((st = layer_wgrad(u, 2, u->p1, nullptr, s))) return st;
    if ((st = layer_igrad(u, 2, u->gin, s))) return st;  // d(p1), 32 ch at level 1
    // L1 (input e1a): d(e1b) = decoder part + pool backward of d(p1)
    if ((st = relu_bwd(u, 1, u->gcat0, 96, 64, u->gin, s))) return st;
    if ((st = layer_wgrad(u, 1, u->y[0], nullptr, s))) return st;
    if ((st = layer_igrad(u, 1, u->gin, s))) return st;  // d(e1a)
    // L0 (input x16): weights only
    if ((st = relu_bwd(u, 0, u->gin, 32, 0, nullptr, s))) return st;
    return layer_wgrad(u, 0, u->x16, nullptr, s);
}

int check_err(lica_unet* u, cudaStream_t s) {
    int e = 0;
    LICA_CUDA_TRY(cudaMemcpyAsync(&e, u->err, sizeof(int), cudaMemcpyDeviceToHost, s));
    LICA_CUDA_TRY(cudaStreamSynchronize(s));
    if (e) {
        lica_set_last_error("lica_unet", "a bounded wait in a tensor-core convolution ran out", __FILE__, __LINE__);
        return LICA_ERR_CUDA;
    }
    return LICA_OK;
}

}  // namespace

extern "C" {

int lica_unet_create(lica_unet** out, int32_t n, int32_t h, int32_t w, uint64_t seed) {
    if (!out || n < 1 || h < 64 || w < 64 || h % 64 || w % 64) {
        lica_set_last_error("lica_unet_create", "images must be at least 64 x 64, multiples of 64", __FILE__,
                            __LINE__);
        return LICA_BAD_ARG;
    }
    *out = nullptr;
    lica_unet* u = new lica_unet();
    u->n = n; u->h = h; u->w = w;
    size_t off = 0;
    for (int l = 0; l < kLayers; ++l) {
        const LayerDef& L = kNet[l];
        u->woff[l] = off;
        off += (size_t)L.cout * 9 * (L.cin0 + L.cin1);
        u->boff[l] = off;
        off += L.cout;
    }
    u->hoff = off;
    off += kHead + 1;
    u->nparams = off;
    // He initialisation (deterministic): N(0, 2 / fan_in); input channels 2..15 carry
    // nothing and start at zero; biases zero; head N(0, 1 / 32)
    std::vector<float> host(off, 0.f);
    InitRng rng{seed};
    for (int l = 0; l < kLayers; ++l) {
        const LayerDef& L = kNet[l];
        const int ctot = L.cin0 + L.cin1;
        const int fan = 9 * (l == 0 ? 2 : ctot);
        const double sd = sqrt(2.0 / fan);
        for (int co = 0; co < L.cout; ++co)
            for (int tap = 0; tap < 9; ++tap)
                for (int ci = 0; ci < ctot; ++ci) {
                    const double v = rng.normal() * sd;
                    if (l > 0 || ci < 2) host[u->woff[l] + ((size_t)co * 9 + tap) * ctot + ci] = (float)v;
                }
    }
    for (int c = 0; c < kHead; ++c) host[u->hoff + c] = (float)(rng.normal() * sqrt(1.0 / kHead));
    auto fail = [&](int code) { lica_unet_destroy(u); return code; };
    int st;
    if ((st = dev_alloc(&u->param, off))) return fail(st);
    if (cudaMemcpy(u->param, host.data(), sizeof(float) * off, cudaMemcpyHostToDevice) != cudaSuccess)
        return fail(LICA_ERR_CUDA);
    for (int l = 0; l < kLayers; ++l) {
        const LayerDef& L = kNet[l];
        const size_t nw = (size_t)L.cout * 9 * (L.cin0 + L.cin1);
        if ((st = dev_alloc(&u->wb[l], nw)) || (st = dev_alloc(&u->wf[l], nw))) return fail(st);
        if ((st = dev_alloc(&u->y[l], level_pixels(u, L.level) * L.cout))) return fail(st);
    }
    const size_t p0 = level_pixels(u, 0), p1 = level_pixels(u, 1), p2 = level_pixels(u, 2);
    if ((st = dev_alloc(&u->x16, p0 * kIn)) || (st = dev_alloc(&u->p1, p1 * 32)) || (st = dev_alloc(&u->p2, p2 * 64)) ||
        (st = dev_alloc(&u->u2, p1 * 128)) || (st = dev_alloc(&u->u1, p0 * 64)) || (st = dev_alloc(&u->out32, p0)) ||
        (st = dev_alloc(&u->sigma, n)) || (st = dev_alloc(&u->rms_part, (size_t)n * kRmsParts)) ||
        (st = dev_alloc(&u->rr, n)) || (st = dev_alloc(&u->err, 1)))
        return fail(st);
    if (cudaMemset(u->err, 0, sizeof(int)) != cudaSuccess) return fail(LICA_ERR_CUDA);
    if ((st = pack_all(u, 0))) return fail(st);
    if (cudaDeviceSynchronize() != cudaSuccess) return fail(LICA_ERR_CUDA);
    *out = u;
    return LICA_OK;
}

int lica_unet_destroy(lica_unet* u) {
    if (!u) return LICA_OK;
    void* ptrs[] = {u->param, u->grad, u->adam_m, u->adam_v, u->x16, u->p1, u->p2, u->u2, u->u1, u->out32,
                    u->sigma, u->rms_part, u->x0, u->ax, u->rr, u->den, u->part2, u->gout, u->gin, u->gcat0,
                    u->gcat1, u->dz, u->part, u->bpart, u->hpart, u->err};
    for (void* p : ptrs) cudaFree(p);
    for (int l = 0; l < kLayers; ++l) {
        cudaFree(u->wb[l]);
        cudaFree(u->wf[l]);
        cudaFree(u->y[l]);
    }
    delete u;
    return LICA_OK;
}

int64_t lica_unet_param_count(const lica_unet* u) { return u ? (int64_t)u->nparams : -1; }

int lica_unet_get_params(lica_unet* u, float* host, int64_t count) {
    if (!u || !host || count != (int64_t)u->nparams) return LICA_BAD_ARG;
    LICA_CUDA_TRY(cudaMemcpy(host, u->param, sizeof(float) * u->nparams, cudaMemcpyDeviceToHost));
    return LICA_OK;
}

int lica_unet_set_params(lica_unet* u, const float* host, int64_t count) {
    if (!u || !host || count != (int64_t)u->nparams) return LICA_BAD_ARG;
    LICA_CUDA_TRY(cudaMemcpy(u->param, host, sizeof(float) * u->nparams, cudaMemcpyHostToDevice));
    int st = pack_all(u, 0);
    if (st) return st;
    LICA_CUDA_TRY(cudaDeviceSynchronize());
    u->adam_t = 0;
    if (u->train_ready) {
        LICA_CUDA_TRY(cudaMemset(u->adam_m, 0, sizeof(float) * u->nparams));
        LICA_CUDA_TRY(cudaMemset(u->adam_v, 0, sizeof(float) * u->nparams));
    }
    return LICA_OK;
}

int lica_unet_guess_device(lica_unet* u, const double* rho, const double* f, double hsq, double* x0, void* stream) {
    if (!u || !rho || !f || !x0 || !(hsq > 0)) return LICA_BAD_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    int st = forward(u, rho, f, hsq, x0, s, false);
    if (st) return st;
    return check_err(u, s);
}

int lica_unet_guess_checked_device(lica_unet* u, const double* rho, const double* f, const double* bx,
                                   const double* by, double hx, double hy, double* x0, double* rel0, void* stream) {
    if (!u || !rho || !f || !bx || !by || !x0 || !rel0 || !(hx > 0) || !(hy > 0)) return LICA_BAD_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    int st;
    const size_t p0 = level_pixels(u, 0);
    if (!u->ax) {
        if ((st = dev_alloc(&u->ax, p0))) return st;
    }
    if ((st = forward(u, rho, f, hx * hy, x0, s, false))) return st;
    if ((st = launch(p0, s, k_apply_op, (const double*)x0, bx, by, u->ax, u->n, u->h, u->w, 1.0 / (hx * hx),
                     1.0 / (hy * hy))))
        return st;
    const int npix = u->h * u->w;
    k_residual<<<dim3(kRmsParts, u->n), kNT, 0, s>>>(f, u->ax, u->rms_part, npix);
    k_part_sum<<<u->n, kNT, 0, s>>>(u->rms_part, u->rr);
    LICA_CUDA_TRY(cudaGetLastError());
    lica_count_launches(2);
    std::vector<double> rr(u->n), sg(u->n);
    LICA_CUDA_TRY(cudaMemcpyAsync(rr.data(), u->rr, sizeof(double) * u->n, cudaMemcpyDeviceToHost, s));
    LICA_CUDA_TRY(cudaMemcpyAsync(sg.data(), u->sigma, sizeof(double) * u->n, cudaMemcpyDeviceToHost, s));
    if ((st = check_err(u, s))) return st;
    for (int i = 0; i < u->n; ++i) {
        rel0[i] = sqrt(rr[i] / (sg[i] * sg[i] * npix));
        if (!(rel0[i] < 1.0))  // no better than zero (or not finite): start from zero
            LICA_CUDA_TRY(cudaMemsetAsync(x0 + (size_t)i * npix, 0, sizeof(double) * npix, s));
    }
    return LICA_OK;
}

int lica_unet_grad_device(lica_unet* u, const double* rho, const double* f, double hsq, const double* gx0,
                          float* grad_host, int64_t count, void* stream) {
    if (!u || !rho || !f || !gx0 || !grad_host || count != (int64_t)u->nparams || !(hsq > 0)) return LICA_BAD_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    int st;
    if ((st = alloc_training(u))) return st;
    if ((st = forward(u, rho, f, hsq, nullptr, s))) return st;
    if ((st = launch(level_pixels(u, 0), s, k_gout_from_gx, gx0, (const double*)u->sigma, rho, hsq, u->gout,
                     u->h * u->w, u->n)))
        return st;
    if ((st = backward(u, s))) return st;
    if ((st = check_err(u, s))) return st;
    LICA_CUDA_TRY(cudaMemcpy(grad_host, u->grad, sizeof(float) * u->nparams, cudaMemcpyDeviceToHost));
    return LICA_OK;
}

int lica_unet_train_step_device(lica_unet* u, const double* rho, const double* f, const double* bx, const double* by,
                                const double* p_star, double hx, double hy, float lr, double* loss, void* stream) {
    if (!u || !rho || !f || !bx || !by || !loss || !(hx > 0) || !(hy > 0) || !(lr > 0)) return LICA_BAD_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    int st;
    if ((st = alloc_training(u))) return st;
    const size_t p0 = level_pixels(u, 0);
    if ((!u->x0 && (st = dev_alloc(&u->x0, p0))) || (!u->ax && (st = dev_alloc(&u->ax, p0))) ||
        (!u->den && (st = dev_alloc(&u->den, u->n))) ||
        (!u->part2 && (st = dev_alloc(&u->part2, (size_t)u->n * kRmsParts))))
        return st;
    const double hsq = hx * hy;
    const int npix = u->h * u->w;
    if ((st = forward(u, rho, f, hsq, u->x0, s))) return st;
    const double cx = 1.0 / (hx * hx), cy = 1.0 / (hy * hy);
    if (p_star) {
        // e = x0 - p*, A e, loss = -e.(A e) / (-p*.f) per image, dL/dout
        if ((st = launch(p0, s, k_sub, u->x0, p_star, p0))) return st;
        if ((st = launch(p0, s, k_apply_op, (const double*)u->x0, bx, by, u->ax, u->n, u->h, u->w, cx, cy))) return st;
        k_energy<<<dim3(kRmsParts, u->n), kNT, 0, s>>>(u->ax, u->x0, p_star, f, u->rms_part, u->part2, npix);
        k_part_sum<<<u->n, kNT, 0, s>>>(u->rms_part, u->rr);
        k_part_sum<<<u->n, kNT, 0, s>>>(u->part2, u->den);
        LICA_CUDA_TRY(cudaGetLastError());
        lica_count_launches(3);
        if ((st = launch(p0, s, k_gout_energy, (const double*)u->ax, (const double*)u->den, (const double*)u->sigma,
                         rho, hsq, u->gout, npix, u->n)))
            return st;
    } else {
        // r = f - A x0, ||r||^2; then A r into x0's buffer, and dL/dout
        if ((st = launch(p0, s, k_apply_op, (const double*)u->x0, bx, by, u->ax, u->n, u->h, u->w, cx, cy))) return st;
        k_residual<<<dim3(kRmsParts, u->n), kNT, 0, s>>>(f, u->ax, u->rms_part, npix);
        k_part_sum<<<u->n, kNT, 0, s>>>(u->rms_part, u->rr);
        LICA_CUDA_TRY(cudaGetLastError());
        lica_count_launches(2);
        if ((st = launch(p0, s, k_apply_op, (const double*)u->ax, bx, by, u->x0, u->n, u->h, u->w, cx, cy))) return st;
        if ((st = launch(p0, s, k_gout, (const double*)u->x0, (const double*)u->sigma, rho, hsq, u->gout, npix, u->n)))
            return st;
    }
    if ((st = backward(u, s))) return st;
    u->adam_t += 1;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f - powf(b1, (float)u->adam_t), c2 = 1.f - powf(b2, (float)u->adam_t);
    if ((st = launch(u->nparams, s, k_adam, u->param, (const float*)u->grad, u->adam_m, u->adam_v, u->nparams, lr, b1,
                     b2, 1e-8f, c1, c2)))
        return st;
    if ((st = pack_all(u, s))) return st;
    // loss = mean over images of ||r||^2 / ||f||^2, or of the relative A-norm error squared
    std::vector<double> rr(u->n), sg(u->n), dn(u->n);
    LICA_CUDA_TRY(cudaMemcpyAsync(rr.data(), u->rr, sizeof(double) * u->n, cudaMemcpyDeviceToHost, s));
    LICA_CUDA_TRY(cudaMemcpyAsync(sg.data(), u->sigma, sizeof(double) * u->n, cudaMemcpyDeviceToHost, s));
    LICA_CUDA_TRY(cudaMemcpyAsync(dn.data(), u->den, sizeof(double) * u->n, cudaMemcpyDeviceToHost, s));
    if ((st = check_err(u, s))) return st;
    double L = 0.0;
    for (int i = 0; i < u->n; ++i) L += p_star ? rr[i] / dn[i] : rr[i] / (sg[i] * sg[i] * npix);
    *loss = L / u->n;
    return LICA_OK;
}

}  // extern "C"
