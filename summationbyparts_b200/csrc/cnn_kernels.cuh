// Kernels of the learned correction network: a 5-layer 3x3 convolutional network on the 64 x 64
// coarse grid (4 -> 32 -> 32 -> 32 -> 32 -> 4 channels, GELU between layers).  Activations are
// BF16, accumulation is FP32 on the tcgen05 tensor cores with TMEM accumulators (convolutions
// forward and backward-data, and the weight gradients); pre-activations, outputs, gradients and
// parameters are FP32.
//
// Layout.  Activations and output gradients are chunk-major, [image][channel / 8][pixel][channel % 8]:
// the 16 bytes of 8 channels of consecutive pixels are contiguous.  In shared memory that is the
// tensor core's no-swizzle layout for both kinds of product -- rows of 16 bytes, 8 consecutive rows
// a core matrix: K-major with pixels as M (convolutions) and MN-major with pixels as K (weight
// gradients) -- and a tap's shift by whole pixels is an offset of the operand's start address, so no
// operand is rearranged by a thread.  A warp's epilogue stores are 512 contiguous bytes.
// Pre-activations are [image][channel / 4][pixel][channel % 4] for the same reason.
//
// Channel counts are padded to what one MMA step consumes: the 4-channel input is stored with
// 16 channels (zeros above 4), the 4-channel output with 8, and the gradient of the output with
// 16.  Padded weights, biases and their gradients are zero and stay zero.
#pragma once

#include <cuda_bf16.h>
#include <cstdint>

#include "bulk_copy.cuh"
#include "dependent_launch.cuh"

namespace sbp {
namespace cnn {

constexpr int kImg = 64;           // image side: the coarse grid
constexpr int kPix = kImg * kImg;  // pixels per image
constexpr int kBand = 4;           // image rows of one band of the convolution kernel
constexpr int kConvGroups = 3;     // groups of four epilogue warps of the convolution kernel
constexpr int kConvThreads = 64 + 128 * kConvGroups;  // a copy warp, a product warp, the epilogue warps
constexpr int kWgradThreads = 128; // 4 warps: one accumulator row of a 128-row tile per thread
constexpr int kWgradRows = 4;      // image rows per CTA in the weight-gradient kernel

enum Epilogue { EPI_GELU = 0, EPI_LINEAR = 1, EPI_DGELU = 2, EPI_APPLY = 3 };

// erf(z) by the rational approximation of Abramowitz and Stegun, Handbook of Mathematical
// Functions, formula 7.1.26: erf(z) = 1 - t (a1 + t (a2 + t (a3 + t (a4 + t a5)))) exp(-z^2),
// t = 1 / (1 + p z) for z >= 0, odd in z; |error| <= 1.5e-7 in exact arithmetic, 5.4e-7 in this
// f32 evaluation (checked against a double-precision erf on [-6, 6]).  g returns exp(-z^2),
// which the GELU derivative shares.  The activations are rounded to bf16 (3.9e-3 relative).
__device__ __forceinline__ float erf_as(float z, float& g) {
    const float az = fabsf(z);
    const float t = __fdividef(1.0f, fmaf(0.3275911f, az, 1.0f));
    g = __expf(-az * az);
    const float poly =
        t * fmaf(t, fmaf(t, fmaf(t, fmaf(t, 1.061405429f, -1.453152027f), 1.421413741f), -0.284496736f), 0.254829592f);
    return copysignf(fmaf(-poly, g, 1.0f), z);
}

// GELU with the Gaussian CDF, x * Phi(x), and its derivative Phi(x) + x * phi(x), with
// Phi(x) = (1 + erf(x / sqrt 2)) / 2 and phi(x) = exp(-x^2 / 2) / sqrt(2 pi).
__device__ __forceinline__ float gelu(float x) {
    float g;
    return 0.5f * x * (1.0f + erf_as(x * 0.70710678118654752f, g));
}
__device__ __forceinline__ float gelu_grad(float x) {
    float g;
    const float e = erf_as(x * 0.70710678118654752f, g);
    return fmaf(0.5f, 1.0f + e, x * 0.39894228040143268f * g);
}

__device__ __forceinline__ unsigned pack_bf16(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const unsigned*>(&v);
}

// ---- tcgen05 (5th-generation tensor core) helpers, sm_100a --------------------------------

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor of a bf16 operand in the canonical layout without swizzling: core
// matrices of 8 rows x 16 bytes (128 contiguous bytes, row after row).  K-major: a row holds 8 values
// along K, core matrices are `lbo` bytes apart along K and `sbo` bytes apart along M (or N).
// MN-major: a row holds 8 values along M (or N), core matrices are `lbo` bytes apart along K and
// `sbo` bytes apart along M (or N).  Fields: start address / 16 (bits 0-13), lbo / 16 (16-29),
// sbo / 16 (32-45), descriptor version 1 (46-47), base offset 0, layout type 0 = no swizzle (61-63).
__device__ __forceinline__ uint64_t umma_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | ((uint64_t)1 << 46);
}

// Instruction descriptor of tcgen05.mma kind::f16 with bf16 A and B and an f32 accumulator, M x N:
// D format (bits 4-5) = f32, A and B formats (7-9, 10-12) = bf16, A and B MN-major (15, 16; both or
// neither here), N / 8 (17-22), M / 16 (24-28).
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int M, int N, bool mn_major) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (mn_major ? 3u << 15 : 0u) | ((uint32_t)(N >> 3) << 17) |
           ((uint32_t)(M >> 4) << 24);
}

// D (tmem) = A * B (+ D when accumulate != 0), issued by one thread.
__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
}

// Arrive on the mbarrier once every tcgen05.mma issued so far by this thread has completed.
__device__ __forceinline__ void umma_commit(uint64_t* mbar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(mbar))
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* mbar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(mbar)) : "memory");
}

// The kernels are dependent launches (launch_after).  Before its dependency_wait a kernel sets up
// barriers, TMEM and zero padding and reads the weights, which the optimiser's kernel two or more
// launches before wrote.

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 32 consecutive f32 TMEM columns of this thread's lane (32x32b shape: warp w reads lanes
// 32 w .. 32 w + 31, so the lane field of taddr must be 32 w).
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float v[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,"
        "%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float v[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// Bit of the network's status word set when a kernel gave up waiting for its copies or its tensor-core
// work (the waits are bounded, so a fault cannot hang the stream).  Such a kernel leaves outputs
// unwritten: the optimiser changes nothing while the bit is set, and the host reports it at its next
// synchronisation.  Before it returns it waits once more for what it has in flight, which ends
// in the CTA's shared memory and TMEM.
constexpr unsigned kStatusMmaTimeout = 1u;
struct StatusWord {
    unsigned* dev;
    unsigned* host;  // the same in mapped host memory: the host reads it without a copy
    __device__ void gave_up() const {
        atomicOr(dev, kStatusMmaTimeout);
        atomicOr_system(host, kStatusMmaTimeout);
    }
};
constexpr int kMmaWaitLimit = 1 << 22;  // mbarrier polls before giving up

// bulk_wait for a whole warp: the lanes agree, so that they stay together for what is warp-wide.  give_up:
// without a poll (the limit itself as an argument costs the apply pass of 512 states 4 of 728 us).
__device__ __forceinline__ bool warp_wait(uint64_t* mbar, uint32_t parity, bool give_up = false) {
    return __all_sync(0xffffffffu, !give_up && bulk_wait(mbar, parity, kMmaWaitLimit));
}

// Shared-memory layout of the tcgen05 convolution (dynamic): the weights, then kConvStages band stages.
// A band of kBand rows with one halo row on each side is one sequence of positions per channel chunk:
// each image row is preceded by a zero position, which pads it on the left and the row before it on
// the right, so pixel (r, c) of the band is position 1 + (r + 1) kPitch + c and the operand of tap
// (dy, dx) is the output's sequence shifted by dy kPitch + dx.  Output position f = r kPitch + c; c = 64
// is computed and dropped.
constexpr int kConvStages = 2;
constexpr int kConvAccs = 8;  // accumulator tiles in flight between the products and the epilogue
template <int CIN, int COUT>
struct ConvTcLayout {
    static constexpr int NP = COUT < 16 ? 16 : COUT;         // N of the MMA (multiple of 16 for M = 128)
    static constexpr int HR = kBand + 2;                     // rows with the halo
    static constexpr int PITCH = kImg + 1;
    static constexpr int TILES = (kBand * PITCH + 127) / 128;  // M = 128 accumulator tiles (3)
    static constexpr int TMEM_COLS = kConvAccs * NP;         // 256 or 128 (a power of two)
    static constexpr int POS = TILES * 128 + 2 * PITCH + 2;  // positions the operands can reach
    static constexpr int CH = CIN / 8;                       // 16-byte channel chunks per pixel
    static constexpr int PLANE = POS * 16;                   // bytes of one chunk's positions
    static constexpr int STAGE = CH * PLANE;
    static constexpr int B_TAP = NP * CIN * 2;               // weights of one tap: [chunk][NP][8]
    static constexpr int X_OFF = 9 * B_TAP;
    static constexpr int BAR_OFF = X_OFF + kConvStages * STAGE;
    // mbarriers: weights; per stage full, empty; per accumulator tile full, empty
    static constexpr int BYTES = BAR_OFF + 8 * (1 + 2 * kConvStages + 2 * kConvAccs) + 8;
    static_assert(BAR_OFF % 8 == 0 && (TMEM_COLS & (TMEM_COLS - 1)) == 0 && HR * PITCH + 1 <= POS, "layout");
};

// Weights of a convolution as one contiguous block in the order of shared memory:
// [tap][input chunk][NP outputs][8 input channels].
__host__ __device__ constexpr int conv_weight_index(int n, int tap, int k, int cin, int np) {
    return ((tap * (cin / 8) + k / 8) * np + n) * 8 + k % 8;
}

struct ConvArgs {
    const __nv_bfloat16* x;    // input activations (or output gradients)
    const __nv_bfloat16* w;    // weights, conv_weight_index order
    const float* bias;         // forward
    const float* zprev;        // EPI_DGELU: pre-activations of the layer below
    float* zout;               // EPI_GELU: pre-activations (null: not kept); EPI_LINEAR, EPI_APPLY: y
    __nv_bfloat16* yout;       // EPI_GELU, EPI_DGELU
    const void* coarse;        // EPI_APPLY: states to correct (f64 or f32) and the corrected states
    int coarse_f64;
    int64_t img_stride;
    float4 oscale;
    double* out;
    int bands;                 // bands of all images
    bool give_up;              // at every wait (for tests)
    StatusWord status;
};

// 3x3 convolution with zero padding as an implicit GEMM on the tcgen05 tensor cores:
// out[p][n] = sum over taps t and input channels k of x[p + off(t)][k] * w[n][t][k],
// off(t) = (t / 3 - 1, t % 3 - 1).  Two persistent CTAs per SM keep the layer's weights (one bulk copy)
// and take bands of kBand image rows in turn; a CTA's warps work on different bands at once:
//   warp 0     bulk copies of a band's rows into a free stage (1 KB per row and chunk)
//   warp 1     zeroes a row outside the image, then one thread issues the 9 x CIN / 16 MMAs (K = 16
//              each) of each of the band's 3 accumulator tiles into a free accumulator
//   warps 2-13 take the finished tiles, four warps each of a band's three, warp w lanes 32 (w % 4) .. --
//              one position per thread, all channels -- and run the epilogue; of the 384 positions 256
//              are pixels, all but 3 of them in the first two tiles:
//   EPI_GELU   z = acc + bias -> zout (f32, if kept), gelu(z) -> yout (bf16)   (hidden layers)
//   EPI_LINEAR acc + bias -> zout (f32, [pixel][8])                            (output layer)
//   EPI_APPLY  as EPI_LINEAR, and coarse + y * out_scale -> out (f64 planes)
//   EPI_DGELU  acc * gelu'(zprev) -> yout (bf16)                       (gradient of a hidden layer)
// What bounds it on 64 images: the start and the drain of the launch (about 8 us of the 20), then the
// epilogue's issue slots and the tensor pipe (an M = 128, N = 32 product takes 64 cycles, 13 us of a
// 32 -> 32 layer), then memory (34 MB a layer, 67 MB with pre-activations).  Measured, apply pass of 512
// states / training step on 64: one CTA per band with copies, products and epilogue in sequence, 4
// an SM 938 / 422 us; this form 743 / 374 before and 736 / 364 after its launches became dependent ones
// (apply 741 with the votes and last waits of kStatusMmaTimeout); one CTA an SM with 8-row bands 945 / 402; three an SM with
// one stage 755 / 394; three copies of a band, one per column offset, with no accumulator row spent
// on padding 829 / 378 (three times the L2 traffic).
template <int CIN, int COUT, int EPI>
__global__ void __launch_bounds__(kConvThreads, 2) conv3x3_tc_kernel(const ConvArgs A) {
    using L = ConvTcLayout<CIN, COUT>;
    static_assert(CIN % 16 == 0 && COUT % 8 == 0 && L::NP <= 32, "channel padding");
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t* wbar = reinterpret_cast<uint64_t*>(smem + L::BAR_OFF);
    uint64_t *full = wbar + 1, *empty = full + kConvStages, *afull = empty + kConvStages, *aempty = afull + kConvAccs;
    uint32_t* tslot = reinterpret_cast<uint32_t*>(aempty + kConvAccs);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)),
                     "r"(L::TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 32) {
        bulk_mbar_init(wbar, 1);
        for (int i = 0; i < kConvStages; ++i) {
            bulk_mbar_init(full + i, 1);
            bulk_mbar_init(empty + i, 1);
        }
        for (int i = 0; i < kConvAccs; ++i) {
            bulk_mbar_init(afull + i, 1);
            bulk_mbar_init(aempty + i, 4);
        }
    }
    // the zero positions between the rows, which no copy touches
    for (int i = tid; i < kConvStages * L::CH * (L::HR + 1); i += kConvThreads)
        *reinterpret_cast<uint4*>(smem + L::X_OFF + (i / (L::HR + 1)) * L::PLANE + (i % (L::HR + 1)) * L::PITCH * 16) =
            make_uint4(0u, 0u, 0u, 0u);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;
    constexpr int kBands = kImg / kBand;  // bands of an image
    bool ok = true;
    if (warp == 0) {
        if (lane == 0) {
            bulk_expect(wbar, 9 * L::B_TAP);
            bulk_g2s(smem, A.w, 9 * L::B_TAP, wbar);
        }
        dependency_wait();
        int i = 0;
        for (int band = blockIdx.x; band < A.bands; band += gridDim.x, ++i) {
            const int st = i % kConvStages, img = band / kBands, r0 = band % kBands * kBand;
            if (i >= kConvStages) ok = warp_wait(empty + st, (i / kConvStages - 1) & 1, A.give_up);
            if (!ok) break;
            const int hlo = r0 == 0 ? 1 : 0, rows = (r0 + kBand == kImg ? L::HR - 1 : L::HR) - hlo;
            if (lane == 0) bulk_expect(full + st, (uint32_t)(L::CH * rows * kImg * 16));
            __syncwarp();
            for (int k = lane; k < rows * L::CH; k += 32) {
                const int kc = k % L::CH, hr = hlo + k / L::CH;
                bulk_g2s(smem + L::X_OFF + st * L::STAGE + kc * L::PLANE + (1 + hr * L::PITCH) * 16,
                         A.x + (((int64_t)img * L::CH + kc) * kPix + (r0 + hr - 1) * kImg) * 8, kImg * 16, full + st);
            }
        }
        // the copies of the weights and of the last bands have arrived, whatever the other warps did
        ok = warp_wait(wbar, 0) && ok;
        for (int b = i < kConvStages ? 0 : i - kConvStages; b < i; ++b)
            ok = warp_wait(full + b % kConvStages, (b / kConvStages) & 1) && ok;
    } else if (warp == 1) {
        constexpr uint32_t idesc = umma_idesc_bf16(128, L::NP, false);
        const uint32_t wbase = smem_u32(smem);
        dependency_wait();
        ok = warp_wait(wbar, 0, A.give_up);
        int i = 0, j = 0;  // bands and accumulator tiles so far
        for (int band = blockIdx.x; band < A.bands && ok; band += gridDim.x, ++i) {
            const int st = i % kConvStages, r0 = band % kBands * kBand;
            unsigned char* stage = smem + L::X_OFF + st * L::STAGE;
            ok = warp_wait(full + st, (i / kConvStages) & 1, A.give_up);
            if (!ok) break;
            if (r0 == 0 || r0 + kBand == kImg) {
                const int r = r0 == 0 ? 0 : L::HR - 1;
                for (int k = lane; k < L::CH * kImg; k += 32)
                    reinterpret_cast<uint4*>(stage + (k / kImg) * L::PLANE)[1 + r * L::PITCH + k % kImg] =
                        make_uint4(0u, 0u, 0u, 0u);
                // what the lanes wrote becomes visible to the tensor core's proxy
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            }
            __syncwarp();
            const uint32_t base = smem_u32(stage);
            for (int h = 0; h < L::TILES; ++h, ++j) {
                const int acc = j % kConvAccs;
                if (j >= kConvAccs) ok = warp_wait(aempty + acc, (j / kConvAccs - 1) & 1, A.give_up);
                if (!ok) break;
                tc_fence_after();
                if (lane == 0) {
#pragma unroll
                    for (int t = 0; t < 9; ++t) {
                        const uint32_t a = base + (h * 128 + (t / 3) * L::PITCH + t % 3) * 16;
                        const uint32_t b = wbase + t * L::B_TAP;
#pragma unroll
                        for (int kk = 0; kk < CIN / 16; ++kk)
                            umma_bf16(tmem + acc * L::NP, umma_desc(a + 2 * kk * L::PLANE, L::PLANE, 128),
                                      umma_desc(b + 2 * kk * L::NP * 16, L::NP * 16, 128), idesc, t > 0 || kk > 0);
                    }
                    if (h == L::TILES - 1) umma_commit(empty + st);
                    umma_commit(afull + acc);
                }
                __syncwarp();
            }
        }
        // the products issued so far are done
        if (j > 0) ok = warp_wait(afull + (j - 1) % kConvAccs, ((j - 1) / kConvAccs) & 1) && ok;
    } else {
        dependency_wait();
        for (int t = (warp - 2) >> 2;; t += kConvGroups) {  // tile t of the CTA: tile t % TILES of its band t / TILES
            const int band = blockIdx.x + t / L::TILES * gridDim.x, h = t % L::TILES;
            if (band >= A.bands) break;
            const int acc = t % kConvAccs, img = band / kBands;
            const int f = h * 128 + (warp & 3) * 32 + lane, r = f / L::PITCH, c = f % L::PITCH;  // position
            const bool real = c < kImg && r < kBand;
            const int pix = real ? ((band % kBands) * kBand + r) * kImg + c : 0;
            float4 zp[EPI == EPI_DGELU ? COUT / 4 : 1];
            if constexpr (EPI == EPI_DGELU) {
                const float4* src = reinterpret_cast<const float4*>(A.zprev) + (int64_t)img * (COUT / 4) * kPix + pix;
#pragma unroll
                for (int q = 0; q < COUT / 4; ++q) zp[q] = real ? __ldg(src + q * kPix) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
            __syncwarp();
            ok = warp_wait(afull + acc, (t / kConvAccs) & 1, A.give_up);
            if (!ok) break;
            tc_fence_after();
            float v[32];
            const uint32_t taddr = tmem + ((uint32_t)((warp & 3) * 32) << 16) + acc * L::NP;
            if constexpr (L::NP == 32) tmem_ld32(taddr, v);
            else tmem_ld16(taddr, v);
            // the accumulator is free once its 4 warps have read it
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(aempty + acc);
            if (!real) continue;
            if constexpr (EPI == EPI_GELU) {
                float4* z = A.zout ? reinterpret_cast<float4*>(A.zout) + (int64_t)img * (COUT / 4) * kPix + pix : nullptr;
                uint4* y = reinterpret_cast<uint4*>(A.yout) + (int64_t)img * (COUT / 8) * kPix + pix;
#pragma unroll
                for (int q = 0; q < COUT / 8; ++q) {
                    float zz[8];
#pragma unroll
                    for (int k = 0; k < 8; ++k) zz[k] = v[8 * q + k] + __ldg(A.bias + 8 * q + k);
                    if (z) {
                        z[(2 * q) * kPix] = make_float4(zz[0], zz[1], zz[2], zz[3]);
                        z[(2 * q + 1) * kPix] = make_float4(zz[4], zz[5], zz[6], zz[7]);
                    }
                    y[q * kPix] = make_uint4(pack_bf16(gelu(zz[0]), gelu(zz[1])), pack_bf16(gelu(zz[2]), gelu(zz[3])),
                                             pack_bf16(gelu(zz[4]), gelu(zz[5])), pack_bf16(gelu(zz[6]), gelu(zz[7])));
                }
            } else if constexpr (EPI == EPI_LINEAR || EPI == EPI_APPLY) {
                static_assert(EPI == EPI_GELU || EPI == EPI_DGELU || COUT == 8, "output layer");
#pragma unroll
                for (int k = 0; k < 8; ++k) v[k] += __ldg(A.bias + k);
                float4* y = reinterpret_cast<float4*>(A.zout) + ((int64_t)img * kPix + pix) * 2;
                y[0] = make_float4(v[0], v[1], v[2], v[3]);
                y[1] = make_float4(v[4], v[5], v[6], v[7]);
                if constexpr (EPI == EPI_APPLY) {
                    const float sc[4] = {A.oscale.x, A.oscale.y, A.oscale.z, A.oscale.w};
                    double* o = A.out + (int64_t)img * 4 * kPix + pix;
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int64_t at = img * A.img_stride + k * kPix + pix;
                        const double cv = A.coarse_f64 ? static_cast<const double*>(A.coarse)[at]
                                                       : double(static_cast<const float*>(A.coarse)[at]);
                        o[k * kPix] = cv + double(v[k]) * double(sc[k]);
                    }
                }
            } else {
                uint4* y = reinterpret_cast<uint4*>(A.yout) + (int64_t)img * (COUT / 8) * kPix + pix;
#pragma unroll
                for (int q = 0; q < COUT / 8; ++q) {
                    const float4 z0 = zp[2 * q], z1 = zp[2 * q + 1];
                    const float* g = v + 8 * q;
                    y[q * kPix] =
                        make_uint4(pack_bf16(g[0] * gelu_grad(z0.x), g[1] * gelu_grad(z0.y)),
                                   pack_bf16(g[2] * gelu_grad(z0.z), g[3] * gelu_grad(z0.w)),
                                   pack_bf16(g[4] * gelu_grad(z1.x), g[5] * gelu_grad(z1.y)),
                                   pack_bf16(g[6] * gelu_grad(z1.z), g[7] * gelu_grad(z1.w)));
                }
            }
        }
    }
    if (!ok && lane == 0) A.status.gave_up();
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(L::TMEM_COLS) : "memory");
    }
}

// Shared-memory layout of the tcgen05 weight-gradient kernel.  A: planes of 16-byte pixel rows, one
// per group of 8 accumulator rows: plane dx CIN / 8 + kc holds chunk kc of the band's x rows shifted
// so that position (hr, c) is pixel (hr, c + dx - 1), then one plane of ones (channel 0), whose
// accumulator row is the bias gradient.  An MMA takes 16 planes; those after the ones plane belong to
// rows that are dropped, and may be any memory: they overlap B.
template <int CIN, int M>
struct WgradTcLayout {
    static constexpr int CH = CIN / 8;
    static constexpr int HR = kWgradRows + 2;                // x rows with the halo
    static constexpr int PLANE = HR * kImg * 16;
    static constexpr int ONES = 3 * CH;                      // the ones plane
    static constexpr int B_OFF = (ONES + 1) * PLANE;         // dz: [row][chunk][64][8]
    static constexpr int BLINE = kImg * 16;                  // a chunk of one dz row
    static constexpr int BROW = (M / 8) * BLINE;
    static constexpr int END = B_OFF + kWgradRows * BROW;
    static constexpr int BAR_OFF = END > 16 * PLANE ? END : 16 * PLANE;
    static constexpr int BYTES = BAR_OFF + 24;
    static constexpr int TMEM_COLS = 3 * M <= 64 ? 64 : 128;
};

// Weight and bias gradients of one layer on the tcgen05 tensor cores, as partial sums per CTA
// (kWgradRows image rows each) that wgrad_reduce_kernel adds up in a fixed order:
// dw[m][t][k] = sum over pixels p of dz[p][m] * x[p + off(t)][k], db[m] = sum over p of dz[p][m].
// For each x row the GEMM D[(dx, k)][(dy, m)] = sum over pixels p of A[(dx, k)][p] * B[(dy, m)][p]
// has the 3 CIN (column offset, channel) pairs as its rows (M = 128 with the ones row and dropped
// rows), the up to three dz rows that meet this x row, by dy, and their channels as N and the pixels as K;
// both operands are MN-major, as the chunk-major rows lie in memory, so the bulk copies put them in
// place and one thread issues all MMAs (K = 16) into one accumulator of 3 M columns.  The column offsets are
// three copies of the x rows (an MMA's row groups lie one stride apart); dz lies row by row, chunk by
// chunk, so that the chunks of adjacent rows are one stride apart too.
//   An MN-major MMA takes about 137 cycles here whatever its N up to 96: the fetch of its 128 A rows.  So
// the three row offsets share one A row: 26 MMAs a CTA, 48 with a product per offset (N = M); a training
// step of 64 images 365 -> 355 us.  What is left is the CTA's own chain: one x copy instead of three takes
// 2 us of a layer's 22, all MMAs left out 6.
// M = channels of dz as stored (16 or 32), MSTORE = rows of the layer's weight tensor (<= M).
template <int CIN, int M, int MSTORE>
__global__ void __launch_bounds__(kWgradThreads) wgrad_tc_kernel(const __nv_bfloat16* __restrict__ x,
                                                                const __nv_bfloat16* __restrict__ dz,
                                                                float* __restrict__ part_w,
                                                                float* __restrict__ part_b, bool give_up,
                                                                const StatusWord status) {
    using L = WgradTcLayout<CIN, M>;
    static_assert(CIN % 16 == 0 && M % 16 == 0 && MSTORE <= M && L::ONES < 16, "channel padding");
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + L::BAR_OFF);  // operands, products
    uint32_t* tslot = reinterpret_cast<uint32_t*>(bar + 2);
    constexpr int chunks_per_img = kImg / kWgradRows;
    const int img = blockIdx.x / chunks_per_img;
    const int rbase = (blockIdx.x % chunks_per_img) * kWgradRows;
    const int tid = threadIdx.x, warp = tid >> 5;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)),
                     "r"(L::TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 32) {
        bulk_mbar_init(bar, 1);
        bulk_mbar_init(bar + 1, 1);
    }
    // the ones plane
    for (int i = tid; i < L::HR * kImg; i += kWgradThreads)
        *reinterpret_cast<uint4*>(smem + L::ONES * L::PLANE + i * 16) = make_uint4(0x3F80u, 0u, 0u, 0u);  // bf16 1.0
    const int hlo = rbase == 0 ? 1 : 0, hhi = rbase + kWgradRows == kImg ? L::HR - 1 : L::HR;
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;
    dependency_wait();
    // The copies: dz a chunk at a time, and the rows of x a chunk at a time for each dx, shifted by
    // one position to the right (dx = 0, without the last pixel) or left (dx = 2, without the first)
    if (tid == 32) bulk_expect(bar, (uint32_t)((hhi - hlo) * L::CH * 3 * kImg * 16 - 2 * L::CH * 16 + kWgradRows * L::BROW));
    if (warp == 1) {
        const int lane = tid & 31;
        __syncwarp();
        for (int i = lane; i < kWgradRows * (M / 8); i += 32) {
            const int lr = i / (M / 8), kc = i % (M / 8);
            bulk_g2s(smem + L::B_OFF + i * L::BLINE, dz + (((int64_t)img * (M / 8) + kc) * kPix + (rbase + lr) * kImg) * 8,
                     L::BLINE, bar);
        }
        for (int i = lane; i < 3 * L::CH; i += 32) {
            const int dx = i / L::CH, kc = i % L::CH;
            const __nv_bfloat16* src = x + (((int64_t)img * L::CH + kc) * kPix + (rbase + hlo - 1) * kImg + (dx == 2)) * 8;
            bulk_g2s(smem + i * L::PLANE + (hlo * kImg + (dx == 0)) * 16, src, ((hhi - hlo) * kImg - (dx != 1)) * 16, bar);
        }
    }
    const bool arrived = !give_up && bulk_wait(bar, 0, kMmaWaitLimit);
    // the column that a shifted copy took from the row beside it is zero padding, and so are the
    // rows outside the image
    for (int i = tid; i < L::HR * L::CH * 2; i += kWgradThreads) {
        const int side = i & 1, kc = (i >> 1) % L::CH, hr = (i >> 1) / L::CH;
        *reinterpret_cast<uint4*>(smem + (2 * side * L::CH + kc) * L::PLANE + (hr * kImg + side * (kImg - 1)) * 16) =
            make_uint4(0u, 0u, 0u, 0u);
    }
    if (hlo == 1 || hhi == L::HR - 1)
        for (int i = tid; i < 3 * L::CH * kImg; i += kWgradThreads) {
            uint4* pl = reinterpret_cast<uint4*>(smem + (i / kImg) * L::PLANE) + i % kImg;
            if (hlo == 1) pl[0] = make_uint4(0u, 0u, 0u, 0u);
            if (hhi == L::HR - 1) pl[(L::HR - 1) * kImg] = make_uint4(0u, 0u, 0u, 0u);
        }
    // what the threads wrote becomes visible to the tensor core's proxy
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    const bool loaded = __syncthreads_and(arrived);
    if (tid == 0 && loaded) {
        const uint32_t base = smem_u32(smem);
        // x row hr with the dz rows r, r + 1, .. (n of them) and pixels 16 s ..: row r is dy = hr - r
        auto product = [&](int hr, int s, int r, int n, uint32_t accumulate) {
            umma_bf16(tmem + (2 - hr + r) * M, umma_desc(base + (hr * kImg + 16 * s) * 16, 128, L::PLANE),
                      umma_desc(base + L::B_OFF + r * L::BROW + 16 * s * 16, 128, L::BLINE),
                      umma_idesc_bf16(128, n * M, true), accumulate);
        };
#pragma unroll
        for (int hr = 0; hr < L::HR; ++hr)
#pragma unroll
            for (int s = 0; s < kImg / 16; ++s) {
                const int lo = hr < 2 ? 0 : hr - 2, hi = hr < kWgradRows ? hr : kWgradRows - 1;
                if (s == 0 && hr < 3) {  // dz row 0 starts the sums of dy = hr
                    product(hr, s, 0, 1, 0u);
                    if (hr > 0) product(hr, s, 1, hr, 1u);
                } else {
                    product(hr, s, lo, hi - lo + 1, 1u);
                }
            }
        umma_commit(bar + 1);
    }
    __syncwarp();
    const bool done = loaded && warp_wait(bar + 1, 0);
    tc_fence_after();
    if (done) {
        float* pw = part_w + (int64_t)blockIdx.x * (MSTORE * 9 * CIN);
#pragma unroll 1
        for (int dy = 0; dy < 3; ++dy) {
            const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16) + (2 - dy) * M;
            float v[32];
            if constexpr (M == 32) tmem_ld32(taddr, v);
            else tmem_ld16(taddr, v);
            if (tid < 3 * CIN) {  // accumulator row tid: column offset tid / CIN, channel tid % CIN
                const int t = 3 * dy + tid / CIN, k = tid % CIN;
#pragma unroll
                for (int m = 0; m < MSTORE; ++m) pw[(m * 9 + t) * CIN + k] = v[m];
            } else if (tid == 3 * CIN && dy == 0) {
#pragma unroll
                for (int m = 0; m < MSTORE; ++m) part_b[(int64_t)blockIdx.x * MSTORE + m] = v[m];
            }
        }
    } else {
        if ((tid & 31) == 0) status.gave_up();
        bulk_wait(loaded ? bar + 1 : bar, 0, kMmaWaitLimit);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(L::TMEM_COLS)
                     : "memory");
    }
}

// Sum of the per-CTA partials in a fixed order: grad[e] for the weights (nw elements) then the
// biases (nb elements).  A CTA of 32 x kReduceSplit threads covers 32 elements: thread (lane, g)
// sums the partials g, g + kReduceSplit, ... of element lane in that order (coalesced across
// lanes), and lane's kReduceSplit sums are then added in order of g.
constexpr int kReduceSplit = 32;
__global__ void __launch_bounds__(32 * kReduceSplit) wgrad_reduce_kernel(const float* __restrict__ part_w,
                                                                       const float* __restrict__ part_b, int nparts,
                                                                       int nw, int nb, float* __restrict__ gw,
                                                                       float* __restrict__ gb) {
    __shared__ float sums[kReduceSplit][32];
    dependency_wait();
    const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
    const int e = blockIdx.x * 32 + lane;
    const bool is_w = e < nw;
    const int j = is_w ? e : e - nw;
    const float* src = is_w ? part_w : part_b;
    const int stride = is_w ? nw : nb;
    float s = 0.0f;
    if (e < nw + nb) {
#pragma unroll 4
        for (int c = g; c < nparts; c += kReduceSplit) s += src[(int64_t)c * stride + j];
    }
    sums[g][lane] = s;
    __syncthreads();
    if (g == 0 && e < nw + nb) {
        float t = sums[0][lane];
#pragma unroll
        for (int k = 1; k < kReduceSplit; ++k) t += sums[k][lane];
        (is_w ? gw : gb)[j] = t;
    }
}

}  // namespace cnn
}  // namespace sbp
