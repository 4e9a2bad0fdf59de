// mlp_tc.cu -- the embedding network on the tensor cores: inference and the
// GEMMs of training.  The network is 136 -> 256 -> 128 -> 64 (GELU).
//
// Forward (k_mlp_fwd_tc): the three layers fused in one persistent kernel, a
// CTA per 128-row tile at a time.  Each layer is one run of tcgen05.mma
// (kind::f16, BF16 x BF16 -> FP32 in TMEM, M = 128, N = 256 / 128 / 64, K in
// steps of 16) issued by one thread: the tile's activations are the A operand
// and the layer's weights the B operand, both K-major in shared memory in the
// 128-byte-swizzled layout (8 rows x 128 bytes per 1 KB atom, the 16-byte
// granule g of row r stored at g ^ (r mod 8)).  The weights are laid out in
// that image once per call (k_mlp_wimage) and copied into shared memory with
// one bulk copy per layer; the input rows are centred, scaled and rounded to
// BF16 by the CTA's threads as they are staged.  Four threads share a TMEM
// lane (a row of the tile): a layer's epilogue reads their parts of the row's
// accumulator (tcgen05.ld), adds the bias, applies GELU, rounds to BF16 and
// writes the row into the next layer's A operand; the last layer's row goes to
// global memory in FP32.  For training the forward pass also keeps the
// pre-activations (FP32) and the BF16 layer inputs, feature-major (the latter
// are the operands of the weight gradients).
//
// Backward (k_mlp_bwd_tc): per 128-row tile, dH2 = dZ3 W3 and dH1 = dZ2 W2 as
// the same fused two-layer scheme (B operands: the transposed weight images),
// each epilogue multiplying by GELU' of the saved pre-activation, adding dZ's
// FP32 column sums into the bias gradients and writing it in transposed BF16.  Weight gradients
// (k_mlp_dw_tc): dW = dZ^T H with K = the batch's rows, split over CTAs, the
// A and B tiles brought by TMA from the transposed arrays, partial sums added
// into the FP32 gradient.  Numerics: BF16 GEMM operands, FP32 accumulation.  All
// waits are bounded.
#include <cuda_bf16.h>

#include <algorithm>

#include "mlp.cuh"

namespace {

constexpr int kRows = 128;                 // rows per tile = TMEM lanes
constexpr int kThreads = 128;              // weight gradients: one thread per TMEM lane
// The layer chains run kSplit threads per row: the epilogues (GELU, BF16,
// the kept arrays) are what bounds a tile, and one CTA of 128 threads left
// three quarters of an SM's warps unused.
constexpr int kSplit = 4;
constexpr int kChainThreads = kRows * kSplit;
constexpr uint32_t kChunkA = kRows * 128;  // one 64-element K chunk of a 128-row operand
// K chunks (64 elements) of each layer's input; 136 is padded to 192
constexpr int kKc1 = 3, kKc2 = MLP_H1 / 64, kKc3 = MLP_H2 / 64;
// weight images: N rows x KC chunks x 128 bytes
constexpr uint32_t kW1Bytes = MLP_H1 * kKc1 * 128;   // 96 KB
constexpr uint32_t kW2Bytes = MLP_H2 * kKc2 * 128;   // 64 KB
constexpr uint32_t kW3Bytes = MLP_OUT * kKc3 * 128;  // 16 KB
constexpr uint32_t kActBytes = kRows * kKc2 * 128;   // 64 KB (the widest input, H1)
constexpr uint32_t kSmem = kActBytes + kW1Bytes + 1024;
// backward images: W3^T (128 rows, K = 64) and W2^T (256 rows, K = 128)
constexpr uint32_t kW3tBytes = MLP_H2 * 1 * 128;      // 16 KB
constexpr uint32_t kW2tBytes = MLP_H1 * 2 * 128;      // 64 KB
constexpr uint32_t kImgBytes = kW1Bytes + kW2Bytes + kW3Bytes + kW3tBytes + kW2tBytes;
// the backward kernel's operands take 96 KB; 120 KB keeps it at one CTA per
// SM, so that its 512 TMEM columns are never contended
constexpr uint32_t kSmemBwd = 120 * 1024;
constexpr uint32_t kTmemCols = 512;                  // layer outputs at columns 0, 256, 384
constexpr uint32_t kLayoutSW128 = 2;

// byte offset of element (r, k) in a K-major SW128 operand of `rows` rows
__host__ __device__ __forceinline__ uint32_t swz(uint32_t rows, uint32_t r, uint32_t k) {
    return (k >> 6) * rows * 128 + r * 128 + ((((k & 63) >> 3) ^ (r & 7)) << 4) + (k & 7) * 2;
}

__device__ __forceinline__ uint64_t desc_sw128(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;  // 8-row atoms 1 KB apart
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)kLayoutSW128 << 61;
    return d;
}

// BF16 x BF16 -> FP32, M = 128, N = n, A and B K-major
__host__ __device__ constexpr uint32_t idesc(uint32_t n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((n >> 3) << 17) | ((128u >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t id,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(id), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 32 consecutive FP32 columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
        "tcgen05.wait::ld.sync.aligned;\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
#pragma unroll
    for (int k = 0; k < 32; ++k) v[k] = __uint_as_float(r[k]);
}

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.f + erff(z * 0.70710678118654752f)); }

__device__ __forceinline__ float gelu_grad(float z) {
    const float cdf = 0.5f * (1.f + erff(z * 0.70710678118654752f));
    const float pdf = 0.39894228040143268f * expf(-0.5f * z * z);
    return cdf + z * pdf;
}

__device__ __forceinline__ __nv_bfloat16 bf(float v) { return __float2bfloat16_rn(v); }

__device__ __forceinline__ uint32_t pack2(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// The weight images, one after another: W1, W2, W3 (element (n, k) =
// BF16(W[n][k]), 0 in the K padding), then W3^T and W2^T (element (n, k) =
// BF16(W[k][n])), the B operands of the backward pass.
__global__ void k_mlp_wimage(const float* __restrict__ P, unsigned char* __restrict__ img) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;  // one element
    const uint32_t n1 = MLP_H1 * kKc1 * 64, n2 = MLP_H2 * kKc2 * 64, n3 = MLP_OUT * kKc3 * 64;
    const uint32_t n4 = MLP_H2 * 64, n5 = MLP_H1 * 128;
    uint32_t rows, kin, kc, e;
    bool tr = false;
    const float* W;
    unsigned char* base;
    if (i < n1) {
        e = i, rows = MLP_H1, kin = MLP_IN, kc = kKc1, W = P + MLP_W1, base = img;
    } else if (i < n1 + n2) {
        e = i - n1, rows = MLP_H2, kin = MLP_H1, kc = kKc2, W = P + MLP_W2, base = img + kW1Bytes;
    } else if (i < n1 + n2 + n3) {
        e = i - n1 - n2, rows = MLP_OUT, kin = MLP_H2, kc = kKc3, W = P + MLP_W3, base = img + kW1Bytes + kW2Bytes;
    } else if (i < n1 + n2 + n3 + n4) {  // W3^T: rows = h2 units, K = output units
        e = i - n1 - n2 - n3, rows = MLP_H2, kin = MLP_OUT, kc = 1, W = P + MLP_W3, tr = true;
        base = img + kW1Bytes + kW2Bytes + kW3Bytes;
    } else if (i < n1 + n2 + n3 + n4 + n5) {  // W2^T: rows = h1 units, K = h2 units
        e = i - n1 - n2 - n3 - n4, rows = MLP_H1, kin = MLP_H2, kc = 2, W = P + MLP_W2, tr = true;
        base = img + kW1Bytes + kW2Bytes + kW3Bytes + kW3tBytes;
    } else {
        return;
    }
    const uint32_t r = e / (kc * 64), k = e % (kc * 64);
    float w = 0.f;
    if (k < kin) w = tr ? W[k * rows + r] : W[r * kin + k];
    *reinterpret_cast<__nv_bfloat16*>(base + swz(rows, r, k)) = __float2bfloat16_rn(w);
}

struct __align__(8) MlpCtl {
    uint64_t w_full, mma_done;
    uint32_t tmem_base;
};

// The per-CTA machinery of a fused layer chain: kSplit threads per TMEM lane
// (tile row), an A operand (act) written by the threads and a B operand (wsm)
// bulk-copied from a weight image.
struct Chain {
    MlpCtl* ctl;
    unsigned char* act;
    unsigned char* wsm;
    uint32_t tmem, sa, sw, ph_w, ph_m;
    int* flag;

    __device__ void init(MlpCtl* c, unsigned char* smem, uint32_t act_bytes, uint32_t tmem_cols, int* f) {
        ctl = c;
        act = smem;
        wsm = smem + act_bytes;
        flag = f;
        ph_w = ph_m = 0;
        if (threadIdx.x == 0) {
            mbar_init(&ctl->w_full, 1);
            mbar_init(&ctl->mma_done, 1);
            mbar_fence_init();
        }
        if (threadIdx.x < 32) {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                             smem_u32(&ctl->tmem_base)),
                         "r"(tmem_cols)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
        fence_before();
        __syncthreads();
        fence_after();
        tmem = ctl->tmem_base;
        sa = smem_u32(act);
        sw = smem_u32(wsm);
    }
    __device__ void finish(uint32_t tmem_cols) {
        fence_before();
        __syncthreads();
        fence_after();
        if (threadIdx.x < 32)
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols)
                         : "memory");
    }
    // thread 0: the layer's weights into shared memory, then its MMAs (A: kc
    // K chunks of the 128-row act operand, B: rows_b rows); every thread
    // then waits for them.  Block-uniform result: a timeout anywhere ends
    // every thread's loop at the same point.
    __device__ bool layer(uint32_t wbytes, const unsigned char* src, int kc, uint32_t ncols, uint32_t col,
                          uint32_t rows_b) {
        const uint32_t t = threadIdx.x;
        if (t == 0) {
            mbar_arrive_tx(&ctl->w_full, wbytes);
            bulk_g2s(wsm, src, wbytes, &ctl->w_full);
        }
        fence_proxy_async_smem();  // this thread's operand stores, before the MMAs read them
        fence_before();
        __syncthreads();
        fence_after();
        bool issued = true;
        if (t == 0) {
            issued = mbar_wait(&ctl->w_full, ph_w, flag);
            if (issued) {
                fence_after();
                for (int s = 0; s < 4 * kc; ++s) {
                    const uint32_t c = s >> 2, off = (s & 3) * 32;  // 16 K elements = 32 bytes of a row
                    mma_bf16(tmem + col, desc_sw128(sa + c * kChunkA + off), desc_sw128(sw + c * rows_b * 128 + off),
                             idesc(ncols), s > 0 ? 1u : 0u);
                }
                mma_commit(&ctl->mma_done);
            }
        }
        ph_w ^= 1;
        // no commit means no completion: skip the wait rather than time out
        if (__syncthreads_or(!issued)) return false;
        const bool ok = mbar_wait(&ctl->mma_done, ph_m, flag);
        ph_m ^= 1;
        fence_after();
        return !__syncthreads_or(!ok);
    }
};

// Outputs the training pass keeps (null in inference), all feature-major so
// that a warp's 32 rows are one run (ld = the padded row count): FP32
// pre-activations [256][ld] and [128][ld]; BF16 layer inputs [192][ld],
// [256][ld] and [128][ld].
struct FwdKeep {
    float* z1;
    float* z2;
    __nv_bfloat16* xT;
    __nv_bfloat16* h1T;
    __nv_bfloat16* h2T;
    uint64_t ld;
};

// A hidden layer's epilogue for this thread's part of row r (global row g,
// kept when g < n): its share of the columns [col0, col0 + 32 * NQ) of the
// accumulator, + bias, GELU, BF16 into the next A operand; the training pass
// also keeps z^T and h^T.
template <int NQ>
__device__ __forceinline__ void epi_hidden(uint32_t tmem_row, uint32_t col0, const float* __restrict__ bias,
                                           unsigned char* act, uint32_t r, uint32_t part, float* zkeep,
                                           __nv_bfloat16* hT, uint64_t ld, uint64_t g, bool keep) {
    static_assert(NQ % kSplit == 0, "whole groups of 32 columns per thread");
#pragma unroll 1
    for (int q = part * (NQ / kSplit); q < (int)(part + 1) * (NQ / kSplit); ++q) {
        float v[32];
        tmem_ld32(tmem_row + col0 + 32 * q, v);
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] += __ldg(bias + 32 * q + j);
        if (zkeep && keep) {
#pragma unroll
            for (int j = 0; j < 32; ++j) zkeep[(uint64_t)(32 * q + j) * ld + g] = v[j];
        }
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = gelu(v[j]);
        if (hT) {
#pragma unroll
            for (int j = 0; j < 32; ++j) hT[(uint64_t)(32 * q + j) * ld + g] = bf(keep ? v[j] : 0.f);
        }
#pragma unroll
        for (int c8 = 0; c8 < 4; ++c8) {  // 16-byte granules of 8 columns
            uint4 u;
            u.x = pack2(v[8 * c8 + 0], v[8 * c8 + 1]);
            u.y = pack2(v[8 * c8 + 2], v[8 * c8 + 3]);
            u.z = pack2(v[8 * c8 + 4], v[8 * c8 + 5]);
            u.w = pack2(v[8 * c8 + 6], v[8 * c8 + 7]);
            *reinterpret_cast<uint4*>(act + swz(kRows, r, (uint32_t)(32 * q + 8 * c8))) = u;
        }
    }
}

// Forward pass over n rows (row i is tnf row idx[i], or i without idx): the
// embedding into z (FP32 [n][64]); with keep, the training outputs too.
__global__ void __launch_bounds__(kChainThreads, 1) k_mlp_fwd_tc(const float* __restrict__ tnf,
                                                             const uint32_t* __restrict__ idx, uint64_t n,
                                                             const float* __restrict__ P,
                                                             const unsigned char* __restrict__ wimg,
                                                             float* __restrict__ z, FwdKeep keep, int* flag) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ MlpCtl ctl;
    __shared__ float mu[MLP_IN];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t t = threadIdx.x, warp = t >> 5;
    const uint32_t row = t % kRows, part = t / kRows;  // warps w, w + 4, ... share a TMEM lane quarter
    for (uint32_t k = t; k < MLP_IN; k += kChainThreads) mu[k] = P[MLP_MU + k];
    Chain ch;
    ch.init(&ctl, smem, kActBytes, kTmemCols, flag);
    const uint32_t tmem_row = ch.tmem + (((warp & 3) * 32) << 16);
    const float scale = P[MLP_SCALE];
    const uint64_t tiles = (n + kRows - 1) / kRows;
    const bool train = keep.xT != nullptr;

    for (uint64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const uint64_t r0 = tile * kRows;
        // stage the tile's rows: centred, scaled, BF16, K padded to 192
        // (granule g: row g % 128, K columns 8 * (g / 128) .. + 7)
#pragma unroll 2
        for (uint32_t gi = t; gi < kRows * kKc1 * 8; gi += kChainThreads) {
            const uint32_t r = gi % kRows, k = (gi / kRows) * 8;
            float e[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            if (r0 + r < n && k < MLP_IN) {
                const uint64_t src_row = idx ? idx[r0 + r] : r0 + r;
                const float4* src = reinterpret_cast<const float4*>(tnf + src_row * MLP_IN + k);
                const float4 a = __ldg(src), b = __ldg(src + 1);
                e[0] = (a.x - mu[k + 0]) * scale;
                e[1] = (a.y - mu[k + 1]) * scale;
                e[2] = (a.z - mu[k + 2]) * scale;
                e[3] = (a.w - mu[k + 3]) * scale;
                e[4] = (b.x - mu[k + 4]) * scale;
                e[5] = (b.y - mu[k + 5]) * scale;
                e[6] = (b.z - mu[k + 6]) * scale;
                e[7] = (b.w - mu[k + 7]) * scale;
            }
            uint4 u;
            u.x = pack2(e[0], e[1]);
            u.y = pack2(e[2], e[3]);
            u.z = pack2(e[4], e[5]);
            u.w = pack2(e[6], e[7]);
            *reinterpret_cast<uint4*>(ch.act + swz(kRows, r, k)) = u;
            if (train)
#pragma unroll
                for (int j = 0; j < 8; ++j) keep.xT[(uint64_t)(k + j) * keep.ld + r0 + r] = bf(e[j]);
        }
        const uint64_t g = r0 + row;
        const bool valid = g < n;
        if (!ch.layer(kW1Bytes, wimg, kKc1, MLP_H1, 0, MLP_H1)) break;
        epi_hidden<MLP_H1 / 32>(tmem_row, 0, P + MLP_B1, ch.act, row, part, keep.z1, keep.h1T, keep.ld, g,
                                     valid);
        if (!ch.layer(kW2Bytes, wimg + kW1Bytes, kKc2, MLP_H2, 256, MLP_H2)) break;
        epi_hidden<MLP_H2 / 32>(tmem_row, 256, P + MLP_B2, ch.act, row, part, keep.z2, keep.h2T, keep.ld, g,
                                     valid);
        if (!ch.layer(kW3Bytes, wimg + kW1Bytes + kW2Bytes, kKc3, MLP_OUT, 384, MLP_OUT)) break;
        // the embedding: + b3, FP32 to global
        if (part < MLP_OUT / 32) {
            const int q = part;
            float v[32];
            tmem_ld32(tmem_row + 384 + 32 * q, v);
            if (valid) {
                float4* dst = reinterpret_cast<float4*>(z + g * MLP_OUT + 32 * q);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int c = 32 * q + 4 * j;
                    dst[j] = make_float4(v[4 * j] + __ldg(P + MLP_B3 + c), v[4 * j + 1] + __ldg(P + MLP_B3 + c + 1),
                                         v[4 * j + 2] + __ldg(P + MLP_B3 + c + 2),
                                         v[4 * j + 3] + __ldg(P + MLP_B3 + c + 3));
                }
            }
        }
        fence_before();
        __syncthreads();  // the next tile overwrites the A operand and the accumulators
        fence_after();
    }
    ch.finish(kTmemCols);
}

// Adds the 32 columns of v over the warp's 32 rows into g[0..31]: a
// reduce-scatter (31 shuffles), after which lane j holds column j.
__device__ __forceinline__ void add_columns(float (&v)[32], float* __restrict__ g) {
    const uint32_t lane = lane_id();
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < o; ++i) {
            const float keep = up ? v[i + o] : v[i], send = up ? v[i] : v[i + o];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    atomicAdd(g + lane, v[0]);
}

// A backward layer's epilogue for this thread's part of row r: its share of
// the columns [col0, col0 + 32 * NQ) of dH, times GELU' of the saved
// pre-activation zs (feature-major FP32) -> dZ: its column sums in FP32 into
// the bias gradient db, BF16 transposed into dT (weight gradients), and BF16
// into the next A operand when act is non-null.  Rows at or past n give zeros.
template <int NQ>
__device__ __forceinline__ void epi_back(uint32_t tmem_row, uint32_t col0, const float* zs, float* db,
                                         __nv_bfloat16* dT, uint64_t ld, unsigned char* act, uint32_t r,
                                         uint32_t part, uint64_t g, bool valid) {
#pragma unroll 1
    for (int q = part * (NQ / kSplit); q < (int)(part + 1) * (NQ / kSplit); ++q) {
        float v[32];
        tmem_ld32(tmem_row + col0 + 32 * q, v);
        if (valid) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] *= gelu_grad(zs[(uint64_t)(32 * q + j) * ld + g]);
        } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = 0.f;
        }
#pragma unroll
        for (int j = 0; j < 32; ++j) dT[(uint64_t)(32 * q + j) * ld + g] = bf(v[j]);
        if (act) {
#pragma unroll
            for (int c8 = 0; c8 < 4; ++c8) {
                uint4 u;
                u.x = pack2(v[8 * c8 + 0], v[8 * c8 + 1]);
                u.y = pack2(v[8 * c8 + 2], v[8 * c8 + 3]);
                u.z = pack2(v[8 * c8 + 4], v[8 * c8 + 5]);
                u.w = pack2(v[8 * c8 + 6], v[8 * c8 + 7]);
                *reinterpret_cast<uint4*>(act + swz(kRows, r, (uint32_t)(32 * q + 8 * c8))) = u;
            }
        }
        add_columns(v, db + 32 * q);
    }
}

// Backward of the two upper layers over ld rows (n of them real): from
// dZ3 (FP32 [ld][64]) to dZ2 and dZ1 (BF16 transposed, dZ3^T too) and the
// three bias gradients (FP32 column sums added into grad).
//
// 16,384 rows (one tile per SM), forward and backward: 39.6 and 37.4 us with
// 128 threads a tile, row-major FP32 arrays (every store of a warp on 32
// lines) and a separate pass for the bias gradients (11 us); 25.6 and 22.8 us
// so.
__global__ void __launch_bounds__(kChainThreads, 1) k_mlp_bwd_tc(const float* __restrict__ d3, uint64_t n, uint64_t ld,
                                                                 const float* __restrict__ z1,
                                                                 const float* __restrict__ z2,
                                                                 const unsigned char* __restrict__ wimg,
                                                                 float* __restrict__ grad,
                                                                 __nv_bfloat16* __restrict__ d3T,
                                                                 __nv_bfloat16* __restrict__ d2T,
                                                                 __nv_bfloat16* __restrict__ d1T, int* flag) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ MlpCtl ctl;
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const uint32_t row = t % kRows, part = t / kRows;
    Chain ch;
    ch.init(&ctl, smem, kRows * 2 * 128, kTmemCols, flag);  // A: up to 128 K (dZ2)
    const uint32_t tmem_row = ch.tmem + (((warp & 3) * 32) << 16);
    const unsigned char* w3t = wimg + kW1Bytes + kW2Bytes + kW3Bytes;
    const unsigned char* w2t = w3t + kW3tBytes;
    const uint64_t tiles = (ld + kRows - 1) / kRows;
    for (uint64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const uint64_t r0 = tile * kRows;
        // stage dZ3 as BF16 (K = 64), and dZ3^T; a warp's 32 rows share a
        // granule of eight columns, whose sums go into the bias gradient
#pragma unroll 2
        for (uint32_t gi = t; gi < kRows * 8; gi += kChainThreads) {
            const uint32_t r = gi % kRows, k = (gi / kRows) * 8;
            float e[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            if (r0 + r < n) {
                const float4* src = reinterpret_cast<const float4*>(d3 + (r0 + r) * MLP_OUT + k);
                const float4 a = src[0], b = src[1];
                e[0] = a.x, e[1] = a.y, e[2] = a.z, e[3] = a.w, e[4] = b.x, e[5] = b.y, e[6] = b.z, e[7] = b.w;
            }
            uint4 u;
            u.x = pack2(e[0], e[1]);
            u.y = pack2(e[2], e[3]);
            u.z = pack2(e[4], e[5]);
            u.w = pack2(e[6], e[7]);
            *reinterpret_cast<uint4*>(ch.act + swz(kRows, r, k)) = u;
#pragma unroll
            for (int j = 0; j < 8; ++j) d3T[(uint64_t)(k + j) * ld + r0 + r] = bf(e[j]);
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) {  // lane l then holds column l % 8 of its quarter-warp's rows
                const bool up = (lane & o) != 0;
#pragma unroll
                for (int i = 0; i < o; ++i) {
                    const float keep = up ? e[i + o] : e[i], send = up ? e[i] : e[i + o];
                    e[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                }
            }
            e[0] += __shfl_xor_sync(0xffffffffu, e[0], 8);
            e[0] += __shfl_xor_sync(0xffffffffu, e[0], 16);
            if (lane < 8) atomicAdd(grad + MLP_B3 + k + lane, e[0]);
        }
        const uint64_t g = r0 + row;
        const bool valid = g < n;
        // dH2 = dZ3 W3 (N = 128, K = 64)
        if (!ch.layer(kW3tBytes, w3t, 1, MLP_H2, 0, MLP_H2)) break;
        epi_back<MLP_H2 / 32>(tmem_row, 0, z2, grad + MLP_B2, d2T, ld, ch.act, row, part, g, valid);
        // dH1 = dZ2 W2 (N = 256, K = 128)
        if (!ch.layer(kW2tBytes, w2t, 2, MLP_H1, 256, MLP_H1)) break;
        epi_back<MLP_H1 / 32>(tmem_row, 256, z1, grad + MLP_B1, d1T, ld, nullptr, row, part, g, valid);
        fence_before();
        __syncthreads();
        fence_after();
    }
    ch.finish(kTmemCols);
}

// Weight gradients dW[m][c] += sum_k A[m][k] B[c][k], A = dZ^T ([M][ld]
// BF16), B = H^T ([nb][ld] BF16): the three layers in one launch.  A CTA
// takes one 128-row block of one dW (blockIdx.x: dW3, dW2, the two halves of
// dW1) over a span of K chunks (64 rows of the batch each, blockIdx.y).
//
// The work is small (2.5 GFLOP and 32 MB from L2 at 16,384 rows), so what
// bounds a CTA is the latency of its chunks: they come by TMA into a
// four-stage ring (one thread issues the copies, another the MMAs), all of a
// short span in flight at once, and the spans are as many as keep one CTA on
// every SM.  Partial sums go into the FP32 gradient four columns at a time
// (red.v4).  16,384 rows: 317 us for the three launches whose threads
// staged 512-row spans synchronously, 15.4 us so.
constexpr int kDwStages = 4;
constexpr uint32_t kDwStageBytes = kChunkA + 256 * 128;
constexpr uint32_t kSmemDw = kDwStages * kDwStageBytes + 1024;

struct DwMaps {
    CUtensorMap a[3], b[3];
};
struct DwJob {
    uint32_t M, nn, nout;  // rows of dW, accumulator columns (a multiple of 16), columns of dW
    float* out;
};
struct DwArgs {
    DwJob job[3];
    uint32_t chunks, span;  // K chunks in all and per CTA
    int* flag;
};
struct __align__(8) DwCtl {
    uint64_t full[kDwStages], empty[kDwStages], done;
    uint32_t tmem_base;
};

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            smem_u32(dst)),
        "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void red_add4(float* p, float a, float b, float c, float d) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

__global__ void __launch_bounds__(kThreads, 1) k_mlp_dw_tc(const __grid_constant__ DwMaps maps, DwArgs p) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ DwCtl ctl;
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t t = threadIdx.x, warp = t >> 5;
    if (t == 0) {
        for (int s = 0; s < kDwStages; ++s) {
            mbar_init(&ctl.full[s], 1);
            mbar_init(&ctl.empty[s], 1);
        }
        mbar_init(&ctl.done, 1);
        mbar_fence_init();
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctl.tmem_base)),
                     "r"(256u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = ctl.tmem_base;
    const uint32_t which = blockIdx.x < 2 ? blockIdx.x : 2, m0 = blockIdx.x == 3 ? kRows : 0;
    const DwJob job = p.job[which];
    const uint32_t c0 = blockIdx.y * p.span, c1 = min(p.chunks, c0 + p.span);
    if (t == 0) {
        const uint32_t bytes = kChunkA + job.nn * 128;
        for (uint32_t c = c0; c < c1; ++c) {
            const uint32_t s = (c - c0) % kDwStages, round = (c - c0) / kDwStages;
            if (!mbar_wait(&ctl.empty[s], (round & 1) ^ 1, p.flag)) break;
            unsigned char* st = smem + s * kDwStageBytes;
            mbar_arrive_tx(&ctl.full[s], bytes);
            tma_load_2d(st, &maps.a[which], (int)(c * 64), (int)m0, &ctl.full[s]);
            tma_load_2d(st + kChunkA, &maps.b[which], (int)(c * 64), 0, &ctl.full[s]);
        }
    } else if (t == 32) {
        const uint32_t base = smem_u32(smem), id = idesc(job.nn);
        for (uint32_t c = c0; c < c1; ++c) {
            const uint32_t s = (c - c0) % kDwStages, round = (c - c0) / kDwStages;
            if (!mbar_wait(&ctl.full[s], round & 1, p.flag)) break;
            fence_after();
            const uint32_t sa = base + s * kDwStageBytes, sb = sa + kChunkA;
            for (int k = 0; k < 4; ++k)
                mma_bf16(tmem, desc_sw128(sa + k * 32), desc_sw128(sb + k * 32), id, (c > c0 || k > 0) ? 1u : 0u);
            mma_commit(&ctl.empty[s]);
            if (c + 1 == c1) mma_commit(&ctl.done);
        }
    }
    __syncwarp();
    // every thread waits for the last MMA, also to keep the ring alive
    const bool ok = c0 < c1 && mbar_wait(&ctl.done, 0, p.flag);
    fence_after();
    if (__syncthreads_and(ok)) {
        const uint32_t tmem_row = tmem + ((warp * 32) << 16);
        const uint32_t m = m0 + t;
        float* row = job.out + (uint64_t)m * job.nout;
#pragma unroll 1
        for (uint32_t q = 0; q * 32 < job.nout; ++q) {
            float v[32];
            tmem_ld32(tmem_row + 32 * q, v);
            if (m < job.M)
#pragma unroll
                for (int j = 0; j < 32; j += 4)
                    if (32 * q + j < job.nout) red_add4(row + 32 * q + j, v[j], v[j + 1], v[j + 2], v[j + 3]);
        }
    }
    fence_before();
    __syncthreads();
    fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256u) : "memory");
}

int weight_images(mdet_ctx* ctx, const float* P, unsigned char** img) {
    *img = (unsigned char*)ctx_scratch(ctx, "mlptc.wimg", kImgBytes);
    if (!*img) return MDET_ERR_NOMEM;
    const uint32_t nel = kImgBytes / 2;
    k_mlp_wimage<<<(nel + 255) / 256, 256, 0, ctx->stream>>>(P, *img);
    MDET_LAUNCHED(ctx, "k_mlp_wimage");
    return MDET_OK;
}

int set_attrs(mdet_ctx* ctx) {
    static bool attr[64] = {false};
    if (!attr[ctx->device & 63]) {
        MDET_CUDA(ctx, cudaFuncSetAttribute(k_mlp_fwd_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem));
        MDET_CUDA(ctx, cudaFuncSetAttribute(k_mlp_bwd_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBwd));
        MDET_CUDA(ctx, cudaFuncSetAttribute(k_mlp_dw_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemDw));
        attr[ctx->device & 63] = true;
    }
    return MDET_OK;
}

int fwd_launch(mdet_ctx* ctx, const float* P, const unsigned char* img, const float* tnf, const uint32_t* idx,
               uint64_t n, float* z, const FwdKeep& keep) {
    const uint64_t tiles = (n + kRows - 1) / kRows;
    const unsigned grid = (unsigned)std::min<uint64_t>(tiles, (uint64_t)ctx->num_sms);
    ctx_timer_begin(ctx, "k_mlp_fwd_tc");
    k_mlp_fwd_tc<<<grid, kChainThreads, kSmem, ctx->stream>>>(tnf, idx, n, P, img, z, keep, ctx->d_flag);
    MDET_LAUNCHED(ctx, "k_mlp_fwd_tc");
    ctx_timer_end(ctx, "k_mlp_fwd_tc");
    return MDET_OK;
}

}  // namespace

// Embeddings of n rows on the tensor cores (rows idx[i] of tnf when idx is
// non-null): z (n x 64).
int mlp_embed_tc(mdet_ctx* ctx, const float* P, const float* tnf, uint64_t n, float* z, const uint32_t* idx) {
    if (n == 0) return MDET_OK;
    MDET_TRY(set_attrs(ctx));
    unsigned char* img = nullptr;
    MDET_TRY(weight_images(ctx, P, &img));
    return fwd_launch(ctx, P, img, tnf, idx, n, z, FwdKeep{nullptr, nullptr, nullptr, nullptr, nullptr, 0});
}

int mlp_tc_alloc(mdet_ctx* ctx, const char* tag, uint64_t rows, MlpTcActs* a) {
    const uint64_t ld = (rows + kRows - 1) / kRows * kRows;
    std::string t(tag);
    auto f = [&](const char* nm, uint64_t cols) { return (float*)ctx_scratch(ctx, (t + nm).c_str(), ld * cols * 4); };
    auto h = [&](const char* nm, uint64_t feats) {
        return (__nv_bfloat16*)ctx_scratch(ctx, (t + nm).c_str(), ld * feats * 2);
    };
    a->ld = ld;
    a->z1 = f(".z1", MLP_H1);
    a->z2 = f(".z2", MLP_H2);
    a->z3 = f(".z3", MLP_OUT);
    a->d3 = f(".d3", MLP_OUT);
    a->xT = h(".xT", 64 * kKc1);
    a->h1T = h(".h1T", MLP_H1);
    a->h2T = h(".h2T", MLP_H2);
    a->d3T = h(".d3T", MLP_OUT);
    a->d2T = h(".d2T", MLP_H2);
    a->d1T = h(".d1T", MLP_H1);
    return (a->z1 && a->z2 && a->z3 && a->d3 && a->xT && a->h1T && a->h2T && a->d3T && a->d2T &&
            a->d1T)
               ? MDET_OK
               : MDET_ERR_NOMEM;
}

int mlp_forward_tc(mdet_ctx* ctx, const float* P, const float* tnf, const uint32_t* idx, uint64_t rows,
                   const MlpTcActs& a) {
    if (rows == 0) return MDET_OK;
    MDET_TRY(set_attrs(ctx));
    unsigned char* img = nullptr;
    MDET_TRY(weight_images(ctx, P, &img));
    return fwd_launch(ctx, P, img, tnf, idx, rows, a.z3, FwdKeep{a.z1, a.z2, a.xT, a.h1T, a.h2T, a.ld});
}

int mlp_backward_tc(mdet_ctx* ctx, const float* P, const MlpTcActs& a, uint64_t np, const float* labels, float m_pos,
                    float m_neg, float* grad, double* loss_sum) {
    cudaStream_t s = ctx->stream;
    const uint64_t rows = 2 * np, ld = a.ld;
    if (np == 0) return MDET_OK;
    MDET_TRY(set_attrs(ctx));
    const unsigned char* img = (const unsigned char*)ctx_scratch(ctx, "mlptc.wimg", kImgBytes);  // from the forward
    MDET_CUDA(ctx, cudaMemsetAsync(grad, 0, MLP_NTRAIN * 4, s));
    if (ld > rows)  // the loss writes the real rows
        MDET_CUDA(ctx, cudaMemsetAsync(a.d3 + rows * MLP_OUT, 0, (ld - rows) * MLP_OUT * 4, s));
    MDET_TRY(mlp_pair_loss(ctx, a.z3, np, labels, m_pos, m_neg, a.d3, loss_sum));
    const uint64_t tiles = ld / kRows;
    const unsigned grid = (unsigned)std::min<uint64_t>(tiles, (uint64_t)ctx->num_sms);
    k_mlp_bwd_tc<<<grid, kChainThreads, kSmemBwd, s>>>(a.d3, rows, ld, a.z1, a.z2, img, grad, a.d3T, a.d2T, a.d1T,
                                                       ctx->d_flag);
    MDET_LAUNCHED(ctx, "k_mlp_bwd_tc");
    // weight gradients: the K chunks in as many spans as give every SM one CTA
    struct Src {
        const __nv_bfloat16* A;
        const __nv_bfloat16* B;
        uint32_t nb;
    } src[3] = {{a.d3T, a.h2T, MLP_H2}, {a.d2T, a.h1T, MLP_H1}, {a.d1T, a.xT, 64 * kKc1}};
    DwArgs p;
    p.job[0] = {MLP_OUT, MLP_H2, MLP_H2, grad + MLP_W3};
    p.job[1] = {MLP_H2, MLP_H1, MLP_H1, grad + MLP_W2};
    p.job[2] = {MLP_H1, 144, MLP_IN, grad + MLP_W1};  // 136 columns, padded to 144
    DwMaps maps;
    for (int k = 0; k < 3; ++k) {
        MDET_TRY(tensor_map_2d(ctx, &maps.a[k], src[k].A, ld, p.job[k].M, 64, kRows, CU_TENSOR_MAP_SWIZZLE_128B, 2));
        MDET_TRY(tensor_map_2d(ctx, &maps.b[k], src[k].B, ld, src[k].nb, 64, p.job[k].nn, CU_TENSOR_MAP_SWIZZLE_128B,
                               2));
    }
    constexpr uint32_t kBlocks = 4;  // 128-row blocks of the three gradients
    p.chunks = (uint32_t)(ld / 64);
    p.span = std::max<uint32_t>(1, (p.chunks * kBlocks + ctx->num_sms - 1) / ctx->num_sms);
    p.flag = ctx->d_flag;
    k_mlp_dw_tc<<<dim3(kBlocks, (p.chunks + p.span - 1) / p.span), kThreads, kSmemDw, s>>>(maps, p);
    MDET_LAUNCHED(ctx, "k_mlp_dw_tc");
    return MDET_OK;
}
