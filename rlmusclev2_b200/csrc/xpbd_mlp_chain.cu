// The cage network's layers in one launch (64 -> 4 x 256 GELU -> 3, BF16
// operands, FP32 accumulation): a CTA takes 64 samples through every layer.
//
// As five GEMM launches the network was bound by everything around the tensor
// cores: at 9,425 samples each 256-wide layer took 17 us for 0.5 us of MMAs
// (operands in 16-byte-wide TMA boxes, activations out to memory and back,
// launch and ramp per layer), 76 us in all against 20 in this form (a pass
// through CageMLP.forward, launches back to back).  Here the activations stay in
// shared memory as the next layer's A operand, in the 128-byte-swizzled
// K-major layout (one TMA box or one 4-byte store pattern, no bank
// conflicts), and the weights arrive through TMA one layer ahead, while the
// epilogue of the layer before runs.  What bounds it now is that epilogue:
// two special-function operations and about twenty others per activation.
//
// 64 samples per CTA (148 CTAs at 9,472 samples, one per SM) and 128-row MMAs:
// the MMA's other 64 rows are never written or read, they only cost tensor
// cycles that are not the limit.  The samples sit in rows 0-15 of each TMEM
// lane quarter, so the 16x256b loads give every lane of all 16 warps work
// (with 128 samples per CTA only 74 SMs run, each with twice the epilogue).
//
// The accumulation order over k (64-wide blocks, 16 per MMA, ascending) and
// the epilogue arithmetic are those of xpbd_gemm_bf16, so the results are bit
// for bit those of the five launches.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "xpbd_common.cuh"
#include "xpbd_mma.cuh"

using namespace xpbd;

namespace {

constexpr int kRows = 64;                     // samples per CTA
constexpr int kChainThreads = 512;
constexpr int kHid = 256;                     // hidden width
constexpr uint32_t kABlock = 128 * 128;       // bytes of one 64-wide k block of A (128 rows)
constexpr uint32_t kWBlock = kHid * 128;      // bytes of one 64-wide k block of a 256-row weight
constexpr size_t kChainSmem = 4 * kABlock + 4 * kWBlock + 1024;  // + alignment slack

struct ChainMaps {
    CUtensorMap x;     // [rows][64], boxes of 64 x 16 rows
    CUtensorMap w[5];  // per layer, boxes of 64 x all output rows
};

// Shared-memory descriptor of a K-major tile with 128-byte swizzle: 8-row
// groups 1024 B apart, version 1, layout type 2 (the leading offset is unused).
__device__ __forceinline__ uint64_t desc_sw128(uint32_t addr) {
    return uint64_t((addr >> 4) & 0x3FFFu) | (uint64_t(1) << 16) | (uint64_t(1024 >> 4) << 32) | (uint64_t(1) << 46) |
           (uint64_t(2) << 61);
}

// D += A B^T over one 64-wide k block: four MMAs of k 16 (32 bytes apart).
__device__ __forceinline__ void mma_block(uint32_t tmem, uint32_t a, uint32_t b, uint32_t idesc, bool first) {
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
        const uint32_t acc = (first && ks == 0) ? 0u : 1u;
        asm volatile(
            "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
            " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
            "l"(desc_sw128(a + 32u * ks)), "l"(desc_sw128(b + 32u * ks)), "r"(idesc), "r"(acc));
    }
}

// 16 lanes x 32 columns of TMEM into a warp: register 4 i + 0, 1 hold row
// lane / 4, columns 8 i + 2 (lane % 4) + 0, 1; registers 4 i + 2, 3 row lane / 4 + 8.
__device__ __forceinline__ void tmem_ld_16x32(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// Byte offset of (row, k) in the A operand: k block, row, 16-byte chunk
// swizzled by the row.
__device__ __forceinline__ uint32_t a_off(int row, int k) {
    return uint32_t(k >> 6) * kABlock + uint32_t(row) * 128u + ((uint32_t((k & 63) >> 3) ^ uint32_t(row & 7)) << 4) +
           uint32_t(k & 7) * 2u;
}

// A layer's activations, transposed, to global memory: out[col][ld] for the
// CTA's 64 samples.  A lane reads 8 columns of two neighbouring samples (16
// swizzled bytes each) and stores pairs: one full 128-byte line per column.
__device__ __forceinline__ void store_transposed(const unsigned char* sa, uint16_t* out, int ld, int m0) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int j = 2 * lane, row = (j >> 4) * 32 + (j & 15);
    for (int u = warp; u < kHid / 8; u += kChainThreads / 32) {
        const int c0 = 8 * u;
        const uint4 a = *reinterpret_cast<const uint4*>(sa + a_off(row, c0));
        const uint4 b = *reinterpret_cast<const uint4*>(sa + a_off(row + 1, c0));
        const uint32_t wa[4] = {a.x, a.y, a.z, a.w}, wb[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int e = 0; e < 8; ++e)
            *reinterpret_cast<uint32_t*>(out + size_t(c0 + e) * ld + m0 + j) =
                __byte_perm(wa[e >> 1], wb[e >> 1], e & 1 ? 0x7632 : 0x5410);
    }
}

// INFER: outputs only.  TRAIN: also the hidden layers' pre-activations and
// transposed activations.  BACK: the deltas of the hidden layers from the
// loss gradient at the outputs, dZ_{l-1} = (dZ_l W_l) gelu'(Z_{l-1}): the same
// chain with the transposed weights (last layer first), four layers long; the
// first A operand is the loss gradient itself, formed here from y and target.
enum { INFER, TRAIN, BACK };

template <int MODE>
__global__ void __launch_bounds__(kChainThreads, 1)
    k_mlp_chain(const __grid_constant__ XpbdMlp P, const __grid_constant__ ChainMaps M) {
    constexpr int kLayers = MODE == BACK ? 4 : 5;
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t s_x, s_w[4], s_acc;
    __shared__ uint32_t s_tmem;
    __shared__ int s_ok;
    __shared__ __align__(16) float s_bias[MODE == BACK ? 4 : 4 * kHid + 16];
    __shared__ float s_loss;
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;  // swizzle atoms are 1024 bytes
    unsigned char* sa = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t aw = base, ww = base + 4 * kABlock;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = int(blockIdx.x) * kRows;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&s_tmem)),
                     "r"(256));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
    }
    if (threadIdx.x == 32) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&s_x)));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&s_acc)));
        for (int i = 0; i < 4; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&s_w[i])));
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        s_ok = 1;
        s_loss = 0.f;
    }
    if constexpr (MODE != BACK) {
        for (int i = threadIdx.x; i < 4 * kHid + 16; i += kChainThreads)
            s_bias[i] = i < 4 * kHid ? P.b[i >> 8][i & 255] : (i - 4 * kHid < 3 ? P.b[4][i - 4 * kHid] : 0.f);
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = s_tmem;
    // weights of layer l into the ring: 64-wide k block kb in slot kb
    auto load_weights = [&](int l) {
        const int nkb = l == 0 ? 1 : 4;
        const uint32_t bytes = l == 4 ? 16u * 128u : kWBlock;
        for (int kb = 0; kb < nkb; ++kb) {
            mbar_expect_tx(smem_u32(&s_w[kb]), bytes);
            tma_load_2d(ww + uint32_t(kb) * kWBlock, &M.w[l], kb * 64, 0, smem_u32(&s_w[kb]));
        }
    };
    if (threadIdx.x == 0) {
        if constexpr (MODE != BACK) {
            mbar_expect_tx(smem_u32(&s_x), kRows * 128);
            for (int q = 0; q < 4; ++q) tma_load_2d(aw + uint32_t(q) * 32u * 128u, &M.x, 0, m0 + 16 * q, smem_u32(&s_x));
        }
        load_weights(0);
    }
    if constexpr (MODE == BACK) {
        // 2 (y - t) / (3 m) of the valid samples in columns 0..2, zero elsewhere;
        // eight threads per sample, one 16-byte chunk each
        const int j = threadIdx.x >> 3, chunk = threadIdx.x & 7, r = m0 + j;
        uint4 d = make_uint4(0u, 0u, 0u, 0u);
        float e2 = 0.f;
        if (chunk == 0) {
            float g[3] = {0.f, 0.f, 0.f};
            if (r < P.m) {
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const float e = P.y[size_t(r) * 16 + c] - P.target[size_t(r) * 3 + c];
                    g[c] = 2.f * e / float(P.m * 3);
                    e2 += e * e;
                }
            }
            d.x = pack_bf16(g[0], g[1]);
            d.y = pack_bf16(g[2], 0.f);
            P.dyt[r] = uint16_t(d.x & 0xffffu);
            P.dyt[size_t(P.m_pad) + r] = uint16_t(d.x >> 16);
            P.dyt[size_t(2 * P.m_pad) + r] = uint16_t(d.y & 0xffffu);
        }
        *reinterpret_cast<uint4*>(sa + a_off((j >> 4) * 32 + (j & 15), 8 * chunk)) = d;
        for (int k = 16; k > 0; k >>= 1) e2 += __shfl_xor_sync(0xffffffffu, e2, k);
        if (lane == 0) atomicAdd(&s_loss, e2);
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        __syncthreads();
        if (threadIdx.x == 0) atomicAdd(P.loss, s_loss);
    }
    int loaded = 0;  // last layer whose weights were asked for (thread 0)
    bool ok = true;
    for (int l = 0; l < kLayers; ++l) {
        const int nkb = l == 0 ? 1 : 4;
        const int n = l == 4 ? 16 : kHid;
        if (threadIdx.x == 32) {
            bool up = MODE == BACK || l > 0 || mbar_wait(smem_u32(&s_x), 0);
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            for (int kb = 0; kb < nkb && up; ++kb) {
                // slot 0 is used by every layer, the others from layer 1 on
                up = mbar_wait(smem_u32(&s_w[kb]), uint32_t((kb == 0 ? l : l - 1) & 1));
                if (up) mma_block(tmem, aw + uint32_t(kb) * kABlock, ww + uint32_t(kb) * kWBlock, instr_desc(n), kb == 0);
            }
            // committed in any case: what was issued completes before the CTA leaves
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                             smem_u32(&s_acc))
                         : "memory");
            if (!up) s_ok = 0;
        }
        __syncwarp();
        if (!mbar_wait(smem_u32(&s_acc), uint32_t(l & 1))) s_ok = 0;
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        if (threadIdx.x == 0 && l + 1 < kLayers) {  // the MMAs have read every slot: the next layer's weights may land
            loaded = l + 1;
            load_weights(l + 1);
        }
        __syncwarp();
        const int q = warp & 3, cg = warp >> 2;
        const int r0 = lane >> 2, cp = 2 * (lane & 3);
        if (l < 4) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int c0 = cg * 64 + h * 32;
                float v[16];
                tmem_ld_16x32(tmem + (uint32_t(q * 32) << 16) + uint32_t(c0), v);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int c = c0 + 8 * i + cp;
#pragma unroll
                    for (int s = 0; s < 2; ++s) {
                        const int r = r0 + 8 * s;
                        const size_t g = size_t(m0 + 16 * q + r) * kHid + c;
                        float y0 = v[4 * i + 2 * s], y1 = v[4 * i + 2 * s + 1];
                        if constexpr (MODE == BACK) {
                            const float2 z = *reinterpret_cast<const float2*>(P.z[3 - l] + g);
                            y0 *= gelu_grad_f(z.x);
                            y1 *= gelu_grad_f(z.y);
                        } else {
                            const float2 bb = *reinterpret_cast<const float2*>(s_bias + l * kHid + c);
                            y0 += bb.x;
                            y1 += bb.y;
                            if (MODE == TRAIN) *reinterpret_cast<float2*>(P.z[l] + g) = make_float2(y0, y1);
                            y0 = gelu_f(y0);
                            y1 = gelu_f(y1);
                        }
                        *reinterpret_cast<uint32_t*>(sa + a_off(q * 32 + r, c)) = pack_bf16(y0, y1);
                    }
                }
            }
        } else if (MODE != BACK && cg == 0) {
            float v[16];
            tmem_ld_16x32(tmem + (uint32_t(q * 32) << 16), v);
#pragma unroll
            for (int s = 0; s < 2; ++s)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int c = cp + e;
                    if (c < 3)
                        P.y[size_t(m0 + 16 * q + r0 + 8 * s) * 16 + c] = v[2 * s + e] + s_bias[4 * kHid + c];
                }
        }
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
        __syncthreads();
        ok = s_ok != 0;
        if (!ok) break;
        if (MODE != INFER && l < 4) {
            store_transposed(sa, MODE == BACK ? P.dzt[3 - l] : P.ht[l], P.m_pad, m0);
            __syncthreads();  // read before the next epilogue overwrites it
        }
    }
    if (!ok && threadIdx.x == 0) {
        if (P.status) atomicOr(P.status, XPBD_STATUS_MMA_TIMEOUT);
        // bounded waits for the copies in flight before the shared memory is given up
        if (MODE != BACK) mbar_wait(smem_u32(&s_x), 0);
        for (int kb = 0; kb < (loaded == 0 ? 1 : 4); ++kb)
            mbar_wait(smem_u32(&s_w[kb]), uint32_t((kb == 0 ? loaded : loaded - 1) & 1));
    }
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(256));
    }
}

// Weight and bias gradients of all five layers, dW = dZ^T H over the samples
// and db = sum of dZ, in one launch.  A tile of a 256 x 256 gradient has the
// whole batch as its k (9,472): as GEMM launches of 2 to 8 CTAs they took
// 131 us each, bound by the 16-byte-wide boxes that one CTA's operands came in.
// Here 60 CTAs, one per 128 x 32 tile of any layer, stream swizzled 64-wide k
// blocks eight deep, 50 us for all five.  The k blocks are accumulated in one
// ascending chain in tensor memory as xpbd_gemm_bf16 does, so the sums are bit
// for bit the same, and that chain of 592 dependent MMAs (about 160 cycles
// each) is what bounds it: halving each CTA's operand bytes (112 CTAs of 64
// rows) changed nothing.  A split over k is faster (25 us) and ten times
// closer to the 64-bit sums, but then differs from the chain by 2.5e-4 of the
// gradient's norm.  The other CTAs, on the SMs the tiles leave free, sum the
// rows of dZ^T and dY^T.
constexpr int kGradStages = 8;
constexpr int kGradThreads = 256;
constexpr int kGradM = 128, kGradN = 32;
constexpr int kGradTiles = 3 * 16 + 4 + 8;
constexpr uint32_t kGradStage = (kGradM + kGradN) * 128;  // A and B rows of one k block
constexpr size_t kGradSmem = kGradStages * kGradStage + 1024;
constexpr int kSumRows = 4 * kHid + 3;                 // rows of dZ^T and dY^T, one warp each
constexpr int kSumCtas = (kSumRows + kGradThreads / 32 - 1) / (kGradThreads / 32);

struct GradMaps {
    CUtensorMap a[5];  // dZ^T of layers 0..3 and dY^T: [rows][m_pad], boxes 64 x 128
    CUtensorMap b[5];  // X^T and H^T of layers 0..3, boxes 64 x 32
};

// db of one row, in xpbd_colsum_bf16's order (lane i adds elements i, i + 32,
// ... of the m samples, then the lanes); 16 loads in flight hide their latency.
__device__ __forceinline__ void row_sum(const XpbdMlp& P, int row) {
    const int lane = threadIdx.x & 31;
    if (row >= kSumRows) return;
    const int l = row >> 8, r = row & 255;  // l = 4: dY^T
    const uint16_t* src = (l == 4 ? P.dyt : P.dzt[l]) + size_t(r) * P.m_pad;
    float s = 0.f;
    int i = lane;
    for (; i + 15 * 32 < P.m; i += 16 * 32) {
        uint16_t v[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) v[k] = src[i + 32 * k];
#pragma unroll
        for (int k = 0; k < 16; ++k) s += __uint_as_float(uint32_t(v[k]) << 16);
    }
    for (; i < P.m; i += 32) s += __uint_as_float(uint32_t(src[i]) << 16);
    for (int k = 16; k > 0; k >>= 1) s += __shfl_xor_sync(0xffffffffu, s, k);
    if (lane == 0) P.gb[l][r] = s;
}

__global__ void __launch_bounds__(kGradThreads, 1)
    k_mlp_wgrad(const __grid_constant__ XpbdMlp P, const __grid_constant__ GradMaps M) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t s_full[kGradStages], s_free[kGradStages], s_acc;
    __shared__ uint32_t s_tmem;
    __shared__ int s_ok;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile = int(blockIdx.x);
    if (tile >= kGradTiles) {
        row_sum(P, (tile - kGradTiles) * (kGradThreads / 32) + warp);
        return;
    }
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    // tiles 0..47: the 256 x 256 layers, 16 each; 48..51: layer 0 (256 x 64); 52..59: the output layer (3 x 256)
    int l, mi, ni;
    if (tile < 48) {
        l = 1 + tile / 16;
        mi = (tile >> 3) & 1;
        ni = tile & 7;
    } else {
        l = tile < 52 ? 0 : 4;
        mi = tile < 52 ? (tile >> 1) & 1 : 0;
        ni = tile < 52 ? tile & 1 : tile - 52;
    }
    const int rows = l == 4 ? 3 : kHid, ldw = l == 0 ? 64 : kHid, nkb = P.m_pad / 64;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&s_tmem)),
                     "r"(kGradN));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
    }
    if (threadIdx.x == 32) {
        for (int i = 0; i < kGradStages; ++i) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&s_full[i])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&s_free[i])));
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&s_acc)));
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        s_ok = 1;
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = s_tmem;
    if (threadIdx.x == 0) {  // copies
        int kb = 0;
        for (; kb < nkb; ++kb) {
            const int st = kb % kGradStages;
            if (kb >= kGradStages && !mbar_wait(smem_u32(&s_free[st]), uint32_t(((kb / kGradStages) - 1) & 1))) {
                s_ok = 0;
                break;
            }
            const uint32_t bar = smem_u32(&s_full[st]), sa = base + uint32_t(st) * kGradStage;
            mbar_expect_tx(bar, kGradStage);
            tma_load_2d(sa, &M.a[l], kb * 64, mi * kGradM, bar);
            tma_load_2d(sa + kGradM * 128, &M.b[l], kb * 64, ni * kGradN, bar);
        }
        // every copy has landed before the CTA gives up its shared memory
        for (int k = max(0, kb - kGradStages); k < kb; ++k)
            if (!mbar_wait(smem_u32(&s_full[k % kGradStages]), uint32_t((k / kGradStages) & 1))) s_ok = 0;
    } else if (threadIdx.x == 32) {  // MMAs
        for (int kb = 0; kb < nkb; ++kb) {
            const int st = kb % kGradStages;
            if (!mbar_wait(smem_u32(&s_full[st]), uint32_t((kb / kGradStages) & 1))) {
                s_ok = 0;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const uint32_t sa = base + uint32_t(st) * kGradStage;
            mma_block(tmem, sa, sa + kGradM * 128, instr_desc(kGradN), kb == 0);
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                             smem_u32(&s_free[st]))
                         : "memory");
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                         smem_u32(&s_acc))
                     : "memory");
        if (!mbar_wait(smem_u32(&s_acc), 0)) s_ok = 0;
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    if (s_ok) {
        const int q = warp & 3, row = mi * kGradM + q * 32 + lane, c0 = 16 * (warp >> 2);
        float v[16];
        tmem_ld16(tmem + (uint32_t(q * 32) << 16) + uint32_t(c0), v);
        if (row < rows) {
            float4* d = reinterpret_cast<float4*>(P.gw[l] + size_t(row) * ldw + ni * kGradN + c0);
#pragma unroll
            for (int i = 0; i < 4; ++i) d[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
        }
    } else if (threadIdx.x == 0 && P.status) {
        atomicOr(P.status, XPBD_STATUS_MMA_TIMEOUT);
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(kGradN));
    }
}

// Tensor map of a K-major BF16 operand [rows][ld]: boxes of 64 k-elements (128
// bytes, swizzled) x box_rows rows, zero fill outside.
bool encode_sw128(CUtensorMap* map, const uint16_t* ptr, int rows, int k, int ld, int box_rows) {
    PFN_cuTensorMapEncodeTiled_v12000 fn = encode_tiled();
    if (!fn) return false;
    const cuuint64_t dims[2] = {cuuint64_t(k), cuuint64_t(rows)};
    const cuuint64_t strides[1] = {cuuint64_t(ld) * 2u};
    const cuuint32_t box[2] = {64u, cuuint32_t(box_rows)};
    const cuuint32_t es[2] = {1u, 1u};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<uint16_t*>(ptr), dims, strides, box, es,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int check_mlp(const XpbdMlp* p, const char* who) {
    if (!p) return fail(XPBD_ERR_ARG, who);
    if (p->m_pad <= 0 || p->m_pad % kRows || p->m < 0 || p->m > p->m_pad)
        return fail(XPBD_ERR_ARG, "XpbdMlp: 0 <= m <= m_pad, m_pad a positive multiple of 64");
    return XPBD_OK;
}

}  // namespace

extern "C" int xpbd_mlp_forward(const XpbdMlp* p, int32_t train, xpbd_stream_t stream) {
    int rc;
    if ((rc = check_mlp(p, "xpbd_mlp_forward: null argument"))) return rc;
    if (!p->x || !p->y) return fail(XPBD_ERR_ARG, "xpbd_mlp_forward: x and y required");
    if (!aligned16(p->x)) return fail(XPBD_ERR_ALIGN, "xpbd_mlp_forward: x must be 16-byte aligned");
    for (int l = 0; l < 5; ++l) {
        if (!p->w[l] || !p->b[l]) return fail(XPBD_ERR_ARG, "xpbd_mlp_forward: weights and biases required");
        if (!aligned16(p->w[l])) return fail(XPBD_ERR_ALIGN, "xpbd_mlp_forward: weights must be 16-byte aligned");
    }
    for (int l = 0; l < 4 && train; ++l) {
        if (!p->z[l] || !p->ht[l]) return fail(XPBD_ERR_ARG, "xpbd_mlp_forward: training needs z and ht");
        if (!aligned16(p->z[l]) || !aligned16(p->ht[l]))
            return fail(XPBD_ERR_ALIGN, "xpbd_mlp_forward: z and ht must be 16-byte aligned");
    }
    // before the maps: in a thread's first call it makes the device's context
    // current, without which the driver encodes none
    auto kern = train ? k_mlp_chain<TRAIN> : k_mlp_chain<INFER>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kChainSmem)) != cudaSuccess)
        return cuda_check("xpbd_mlp_forward: smem attribute");
    ChainMaps maps;
    bool enc = encode_sw128(&maps.x, p->x, p->m_pad, 64, 64, 16);
    for (int l = 0; l < 5 && enc; ++l)
        enc = encode_sw128(&maps.w[l], p->w[l], l == 4 ? 16 : kHid, l == 0 ? 64 : kHid, l == 0 ? 64 : kHid,
                           l == 4 ? 16 : kHid);
    if (!enc) return fail(XPBD_ERR_CUDA, "xpbd_mlp_forward: tensor maps");
    kern<<<p->m_pad / kRows, kChainThreads, kChainSmem, (cudaStream_t)stream>>>(*p, maps);
    return cuda_check("xpbd_mlp_forward");
}

extern "C" int xpbd_mlp_backward(const XpbdMlp* p, xpbd_stream_t stream) {
    int rc;
    if ((rc = check_mlp(p, "xpbd_mlp_backward: null argument"))) return rc;
    if (p->m < 1 || !p->y || !p->xt || !p->target || !p->dyt || !p->loss)
        return fail(XPBD_ERR_ARG, "xpbd_mlp_backward: m >= 1, y, xt, target, dyt and loss required");
    if (!aligned16(p->xt) || !aligned16(p->dyt)) return fail(XPBD_ERR_ALIGN, "xpbd_mlp_backward: 16-byte alignment");
    for (int l = 0; l < 5; ++l) {
        if (!p->gw[l] || !p->gb[l] || (l > 0 && !p->wt[l]) || (l < 4 && (!p->z[l] || !p->ht[l] || !p->dzt[l])))
            return fail(XPBD_ERR_ARG, "xpbd_mlp_backward: wt, z, ht, dzt, gw and gb required");
        if (!aligned16(p->gw[l]) || !aligned16(p->wt[l]) ||
            (l < 4 && (!aligned16(p->z[l]) || !aligned16(p->ht[l]) || !aligned16(p->dzt[l]))))
            return fail(XPBD_ERR_ALIGN, "xpbd_mlp_backward: 16-byte alignment");
    }
    // first, as in xpbd_mlp_forward
    if (cudaFuncSetAttribute(k_mlp_chain<BACK>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kChainSmem)) !=
            cudaSuccess ||
        cudaFuncSetAttribute(k_mlp_wgrad, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kGradSmem)) != cudaSuccess)
        return cuda_check("xpbd_mlp_backward: smem attribute");
    ChainMaps cm = {};
    bool enc = true;
    for (int l = 0; l < 4 && enc; ++l) {  // wt[4] (k 64), wt[3], wt[2], wt[1]
        const int k = l == 0 ? 64 : kHid;
        enc = encode_sw128(&cm.w[l], p->wt[4 - l], kHid, k, k, kHid);
    }
    GradMaps gm;
    const int M = p->m_pad;
    for (int l = 0; l < 5 && enc; ++l) {
        enc = encode_sw128(&gm.a[l], l == 4 ? p->dyt : p->dzt[l], l == 4 ? 3 : kHid, M, M, kGradM);
        enc = enc && encode_sw128(&gm.b[l], l == 0 ? p->xt : p->ht[l - 1], l == 0 ? 64 : kHid, M, M, kGradN);
    }
    if (!enc) return fail(XPBD_ERR_CUDA, "xpbd_mlp_backward: tensor maps");
    k_mlp_chain<BACK><<<M / kRows, kChainThreads, kChainSmem, (cudaStream_t)stream>>>(*p, cm);
    k_mlp_wgrad<<<kGradTiles + kSumCtas, kGradThreads, kGradSmem, (cudaStream_t)stream>>>(*p, gm);
    return cuda_check("xpbd_mlp_backward");
}
