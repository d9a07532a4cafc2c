// mlp.cu — the learned warm start's network (no counterpart in the
// reference): 48 -> 256 -> 256 -> 256 -> 12, GELU, BF16 weights and
// activations, FP32 accumulation.
//
// Inference (every step of warm_start 3): one CTA of 16 warps runs 128 bodies
// through all four layers.  Layer weights are stored once in the UMMA
// canonical K-major layout (8x8 core matrices, no swizzle) and copied into
// shared memory with one bulk asynchronous copy per layer; the activations
// stay in shared memory in the same layout.  One elected thread issues
// tcgen05.mma (kind::f16, M = 128, N = 256 or 16, K = 16 per instruction)
// with the FP32 accumulator in tensor memory; the four warps read their 32
// accumulator lanes back with tcgen05.ld, add the bias, apply GELU and write
// the next layer's BF16 operand.  Every wait is bounded and reports through
// an error flag; tensor memory is freed on every path.
//
// Training: FP32 master weights, Adam; every GEMM of the forward and backward
// pass (Z = H W^T, dW = dZ^T H, dH = dZ W) on the tensor cores (tcgen05,
// BF16 operands, FP32 accumulation in tensor memory), the forward with
// BF16-rounded weights and activations like inference, MSE loss, backward
// with straight-through rounding.
#include "engine.cuh"
#include <mutex>
#include <cuda_bf16.h>

namespace {

constexpr int MI = ABD_MLP_IN, MH = ABD_MLP_HIDDEN, MO = ABD_MLP_OUT;
constexpr int K1 = 64;            // input width padded to a multiple of 16
constexpr int NO = 16;            // output width padded to the MMA's N step
// parameter blob offsets (FP32, W[out][in] row-major then bias)
constexpr int OW1 = 0, OB1 = OW1 + MH * MI, OW2 = OB1 + MH, OB2 = OW2 + MH * MH, OW3 = OB2 + MH, OB3 = OW3 + MH * MH,
              OW4 = OB3 + MH, OB4 = OW4 + MO * MH, NPARAM = OB4 + MO;
static_assert(NPARAM == ABD_MLP_NPARAM, "parameter count");
// packed BF16 weights (canonical layout), byte offsets
constexpr int PW1 = 0, PW2 = PW1 + MH * K1 * 2, PW3 = PW2 + MH * MH * 2, PW4 = PW3 + MH * MH * 2, PTOT = PW4 + NO * MH * 2;
// shared memory of the inference kernel
constexpr int S_A = 0, S_W = S_A + 128 * MH * 2, S_BAR = S_W + MH * MH * 2, S_TM = S_BAR + 16, S_TOT = S_TM + 16;
constexpr int NTHR = 512;
constexpr long WAIT_LIMIT = 1L << 22;

// element index of (r, k) in a K-major canonical tile with K columns
HD int canon(int r, int k, int K) { return (r >> 3) * (K * 8) + (k >> 3) * 64 + (r & 7) * 8 + (k & 7); }

DV float gelu(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }
DV float gelu_grad(float x) {
    return 0.5f * (1.0f + erff(x * 0.70710678118654752f)) + x * 0.39894228040143268f * expf(-0.5f * x * x);
}

DV uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// UMMA shared-memory descriptor: no swizzle, K-major; lbo = byte distance of
// the two 8-column halves of a K = 16 slice, sbo = byte distance of 8-row groups
DV uint64_t sdesc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = (uint64_t)((addr & 0x3FFFF) >> 4);
    d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
    d |= (uint64_t)1 << 46;                       // descriptor version of sm_100
    return d;                                     // base offset 0, no swizzle
}
// instruction descriptor: BF16 x BF16 -> FP32, both K-major, M = 128
HD uint32_t idesc(int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}

DV void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(bar), "r"(count) : "memory");
}
DV bool mbar_wait(uint32_t bar, uint32_t parity) {
    for (long i = 0; i < WAIT_LIMIT; i++) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\t"
                     "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (ok) return true;
    }
    return false;
}
// one bulk copy of `bytes` (multiple of 16) from global into shared memory,
// completing on `bar`
DV void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"(bytes) : "memory");
    for (uint32_t off = 0; off < bytes; off += 32768) {
        uint32_t n = bytes - off < 32768 ? bytes - off : 32768;
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                     :: "r"(dst + off), "l"((const char*)src + off), "r"(n), "r"(bar) : "memory");
    }
}
DV void mma_bf16(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t id, uint32_t acc) {
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "setp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
                 :: "r"(tmem_d), "l"(da), "l"(db), "r"(id), "r"(acc), "r"(0), "r"(0), "r"(0), "r"(0) : "memory");
}
DV void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(bar) : "memory");
}
DV void tmem_ld32(uint32_t taddr, float* v) {
    uint32_t r[32];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                 "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]);
}
DV void tmem_ld16(uint32_t taddr, float* v) {
    uint32_t r[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                 "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

// Y[n][12] = net((X - mean) / std) * ystd + ymean, 128 rows per CTA.  One CTA
// fits an SM (operands and weights take 200 KB), and the epilogues (GELU of
// 128 x 256 values per layer) bound it, so 16 warps share them: 50,021 rows
// take 84 us, with four warps 105.
__global__ void __launch_bounds__(NTHR, 1) k_mlp_infer(int n, const float* __restrict__ X, const float* __restrict__ norm,
                                                      const uint8_t* __restrict__ wpack, const float* __restrict__ bias,
                                                      float* __restrict__ Y, int* err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __nv_bfloat16* sA = reinterpret_cast<__nv_bfloat16*>(smem + S_A);
    const uint32_t aA = smem_u32(smem + S_A), aW = smem_u32(smem + S_W);
    const uint32_t bar_w = smem_u32(smem + S_BAR), bar_m = bar_w + 8;
    uint32_t* tm_holder = reinterpret_cast<uint32_t*>(smem + S_TM);
    __shared__ int status;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int row0 = blockIdx.x * 128;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"(smem_u32(tm_holder)), "r"(256) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        status = 0;
        mbar_init(bar_w, 1);
        mbar_init(bar_m, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tm_holder;
    if (tid == 0) bulk_load(aW, wpack + PW1, MH * K1 * 2, bar_w);

    // layer-1 operand: normalised inputs of this CTA's rows, BF16, K = 64
    {
        const int r = tid & 127, gr = row0 + r;
        for (int k0 = (tid >> 7) * 8; k0 < K1; k0 += NTHR / 128 * 8) {
            __align__(16) __nv_bfloat16 v[8];
#pragma unroll
            for (int j = 0; j < 8; j++) {
                int k = k0 + j;
                float x = 0.0f;
                if (gr < n && k < MI) x = (X[(long)gr * MI + k] - norm[k]) / norm[MI + k];
                v[j] = __float2bfloat16_rn(x);
            }
            *reinterpret_cast<uint4*>(sA + canon(r, k0, K1)) = *reinterpret_cast<const uint4*>(v);
        }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();

    const int Ks[4] = {K1, MH, MH, MH};
    const int Ns[4] = {MH, MH, MH, NO};
    const int Poff[4] = {PW1, PW2, PW3, PW4};
    const int Boff[4] = {0, MH, 2 * MH, 3 * MH};
    for (int l = 0; l < 4; l++) {
        const int K = Ks[l], N = Ns[l];
        if (tid == 0) {
            bool ok = mbar_wait(bar_w, l & 1);
            if (ok) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t id = idesc(N), sbo = (uint32_t)K * 16;
                for (int kk = 0; kk < K / 16; kk++)
                    mma_bf16(tmem, sdesc(aA + kk * 256, 128, sbo), sdesc(aW + kk * 256, 128, sbo), id, kk > 0);
                mma_commit(bar_m);
                ok = mbar_wait(bar_m, l & 1);
            }
            if (!ok) { status = 1; atomicExch(err, 1); }
            else if (l < 3) {
                // the MMAs of this layer are done with the weights: fetch the next layer's
                int bytes = (l + 1 < 3) ? MH * MH * 2 : NO * MH * 2;
                bulk_load(aW, wpack + Poff[l + 1], bytes, bar_w);
            }
        }
        __syncthreads();
        if (status) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // a warp reads the tensor-memory rows of its place among four; the four
        // groups of four warps take a quarter of the columns each
        const int r = (warp & 3) * 32 + lane, gr = row0 + r, part = warp >> 2;
        const uint32_t trow = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        if (l < 3) {
            const int cols = N / (NTHR / 128);
            for (int c0 = part * cols; c0 < (part + 1) * cols; c0 += 32) {
                float v[32];
                tmem_ld32(trow + c0, v);
#pragma unroll
                for (int j0 = 0; j0 < 32; j0 += 8) {
                    __align__(16) __nv_bfloat16 h[8];
#pragma unroll
                    for (int j = 0; j < 8; j++) h[j] = __float2bfloat16_rn(gelu(v[j0 + j] + bias[Boff[l] + c0 + j0 + j]));
                    *reinterpret_cast<uint4*>(sA + canon(r, c0 + j0, MH)) = *reinterpret_cast<const uint4*>(h);
                }
            }
        } else if (part == 0) {
            float v[16];
            tmem_ld16(trow, v);
            if (gr < n) {
                const float* ym = norm + 2 * MI;
                const float* ys = norm + 2 * MI + MO;
#pragma unroll
                for (int j = 0; j < MO; j++) Y[(long)gr * MO + j] = (v[j] + bias[Boff[3] + j]) * ys[j] + ym[j];
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
    }
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(256) : "memory");
    }
}

// FP32 parameter blob -> BF16 canonical tiles + FP32 biases (output padded to 16)
__global__ void k_mlp_pack(const float* __restrict__ P, __nv_bfloat16* pack, float* bias) {
    GS_LOOP(i, (long)MH * K1 + 2L * MH * MH + (long)NO * MH) {
        long j = i;
        if (j < (long)MH * K1) {
            int r = (int)(j / K1), k = (int)(j % K1);
            pack[PW1 / 2 + canon(r, k, K1)] = __float2bfloat16_rn(k < MI ? P[OW1 + r * MI + k] : 0.0f);
            continue;
        }
        j -= (long)MH * K1;
        if (j < 2L * MH * MH) {
            int layer = (int)(j / (MH * MH)), e = (int)(j % (MH * MH));
            int r = e / MH, k = e % MH;
            int src = layer == 0 ? OW2 : OW3, dst = layer == 0 ? PW2 : PW3;
            pack[dst / 2 + canon(r, k, MH)] = __float2bfloat16_rn(P[src + r * MH + k]);
            continue;
        }
        j -= 2L * MH * MH;
        int r = (int)(j / MH), k = (int)(j % MH);
        pack[PW4 / 2 + canon(r, k, MH)] = __float2bfloat16_rn(r < MO ? P[OW4 + r * MH + k] : 0.0f);
    }
    GS_LOOP(i, 4 * MH) {
        int l = (int)(i / MH), c = (int)(i % MH);
        float b = 0.0f;
        if (l == 0) b = P[OB1 + c];
        else if (l == 1) b = P[OB2 + c];
        else if (l == 2) b = P[OB3 + c];
        else b = c < MO ? P[OB4 + c] : 0.0f;
        bias[i] = b;
    }
}

// ------------------------------------------------------------------ training kernels
// One mini-batch is eight launches: three hidden layers forward, the output
// layer with the loss and the gradient of the last hidden layer, two hidden
// layers backward, all weight and bias gradients, Adam.  Every product
//   Z = H W^T,  dH = dZ W,  dW = dZ^T H
// runs on the tensor cores (tcgen05, BF16 operands, FP32 accumulation in
// tensor memory).  Each epilogue leaves its result in the layouts that the
// next products read: BF16 row-major for the products over features, and
// BF16 transposed ([column][row], rows padded with zeros to the 128-row
// tile) for the products over rows, so every operand is K-contiguous and is
// staged with 16-byte cp.async straight into the UMMA canonical layout.  The
// mini-batch of 512 rows moves about 5 MB through L2 and is bound by launch
// and pipeline latency, not by bytes or by the tensor cores; the figures at
// tr_forward_backward are measured.  Waits are bounded and report through
// *err; tensor memory is freed on every path.
constexpr int TR_THR = 256;
// BF16 copies of the weights: W[out][in] (W1 padded to 64 inputs, W4 to 16
// outputs) and W^T[in][out] of layers 2..4, element offsets
constexpr int BW1 = 0, BW2 = BW1 + MH * K1, BW3 = BW2 + MH * MH, BW4 = BW3 + MH * MH, BT2 = BW4 + NO * MH,
              BT3 = BT2 + MH * MH, BT4 = BT3 + MH * MH, BTOT = BT4 + MH * NO;

// parameter i of the blob, rounded, into its places of the BF16 copies
DV void tr_pack_one(long i, float p, __nv_bfloat16* W) {
    const __nv_bfloat16 q = __float2bfloat16_rn(p);
    if (i < OB1) { const int r = (int)i / MI, k = (int)i % MI; W[BW1 + r * K1 + k] = q; }
    else if (i >= OW2 && i < OB2) { const int j = (int)i - OW2, r = j / MH, k = j % MH; W[BW2 + j] = q; W[BT2 + k * MH + r] = q; }
    else if (i >= OW3 && i < OB3) { const int j = (int)i - OW3, r = j / MH, k = j % MH; W[BW3 + j] = q; W[BT3 + k * MH + r] = q; }
    else if (i >= OW4 && i < OB4) { const int j = (int)i - OW4, r = j / MH, k = j % MH; W[BW4 + j] = q; W[BT4 + k * NO + r] = q; }
}
__global__ void k_tr_pack(const float* __restrict__ P, __nv_bfloat16* W) { GS_LOOP(i, NPARAM) tr_pack_one(i, P[i], W); }

DV void cp16_zfill(uint32_t dst, const void* src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
// rows r0 .. r0 + ROWS of a K-contiguous BF16 matrix (row pitch ld, rows past
// nrows and columns past the tile are zero) into a canonical K-major tile.
// Eight lanes take eight rows of one 8-column group: 128 contiguous bytes of
// shared memory, and four lane groups cover 64 bytes of each row.
template <int ROWS, int K>
DV void tr_stage(uint32_t dst, const __nv_bfloat16* __restrict__ src, long ld, int r0, int nrows) {
    constexpr int KG = K / 8;
    static_assert(KG % 4 == 0 || KG == 2, "column groups");
    constexpr int GW = KG == 2 ? 2 : 4;
    for (int e = threadIdx.x; e < ROWS * KG; e += TR_THR) {
        const int rl = e & 7, kl = (e >> 3) % GW, rest = (e >> 3) / GW;
        const int kg = (rest % (KG / GW)) * GW + kl, r = (rest / (KG / GW)) * 8 + rl;
        const bool ok = r0 + r < nrows;
        cp16_zfill(dst + (uint32_t)((r >> 3) * (K * 16) + kg * 128 + (r & 7) * 16),
                   src + (ok ? (long)(r0 + r) * ld + kg * 8 : 0), ok);
    }
}
DV void tr_stage_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> DV void tr_stage_wait() { asm volatile("cp.async.wait_group %0;" :: "n"(N) : "memory"); }
DV void tmem_alloc(uint32_t holder, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(holder), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
DV void tmem_free(uint32_t tmem, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(cols) : "memory");
}
DV void tc_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
DV void tc_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
DV void proxy_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
DV void mma_tile(uint32_t tmem, uint32_t aA, uint32_t aB, int K, int N, bool fresh) {
    const uint32_t id = idesc(N), sbo = (uint32_t)K * 16;
    for (int kk = 0; kk < K / 16; kk++)
        mma_bf16(tmem, sdesc(aA + kk * 256, 128, sbo), sdesc(aB + kk * 256, 128, sbo), id, (fresh && kk == 0) ? 0u : 1u);
}

// One 128-row x 64-column tile of a hidden layer, forward or backward.
// FWD: z = A W^T + bias; G = gelu'(z), H = bf16(gelu(z)) and H^T.
// else: d = (A W) * G of the layer below; D (FP32), H = bf16(d), H^T.
// K = 64: the input layer, whose operand is gathered from the FP32 data set
// (rows idx[], or all rows in order) and rounded; block column 0 also writes
// its transpose XT.
template <int K, bool FWD>
__global__ void __launch_bounds__(TR_THR) k_tr_layer(int b, int pitch, const __nv_bfloat16* __restrict__ A,
        const float* __restrict__ X, const int* __restrict__ idx, __nv_bfloat16* __restrict__ XT,
        const __nv_bfloat16* __restrict__ W, const float* __restrict__ bias, float* __restrict__ G, float* __restrict__ D,
        __nv_bfloat16* __restrict__ H, __nv_bfloat16* __restrict__ HT, int* err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t bar_s;
    __shared__ uint32_t tm_s;
    __shared__ int status;
    const uint32_t aA = smem_u32(smem), aB = aA + 128 * K * 2, bar = smem_u32(&bar_s);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.y * 128, n0 = blockIdx.x * 64;
    tr_stage<64, K>(aB, W, K, n0, MH);
    if constexpr (K == MH) {
        tr_stage<128, K>(aA, A, MH, m0, b);
    } else {
        for (int e = tid; e < 128 * (K / 8); e += TR_THR) {
            const int r = (e & 7) + 8 * (e >> 6), kg = (e >> 3) & 7, row = m0 + r;
            __align__(16) __nv_bfloat16 v[8];
            float f[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            if (row < b && kg < MI / 8) {
                const float4* p = reinterpret_cast<const float4*>(X + (long)(idx ? idx[row] : row) * MI + kg * 8);
                const float4 u = p[0], w = p[1];
                f[0] = u.x; f[1] = u.y; f[2] = u.z; f[3] = u.w; f[4] = w.x; f[5] = w.y; f[6] = w.z; f[7] = w.w;
            }
#pragma unroll
            for (int j = 0; j < 8; j++) v[j] = __float2bfloat16_rn(f[j]);
            *reinterpret_cast<uint4*>(smem + (r >> 3) * (K * 16) + kg * 128 + (r & 7) * 16) = *reinterpret_cast<const uint4*>(v);
            if (blockIdx.x == 0) {
#pragma unroll
                for (int j = 0; j < 8; j++) XT[(long)(kg * 8 + j) * pitch + row] = v[j];
            }
        }
    }
    tr_stage_commit();
    if (warp == 0) tmem_alloc(smem_u32(&tm_s), 64);
    if (tid == 0) {
        status = 0;
        mbar_init(bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    tr_stage_wait<0>();
    proxy_fence();
    tc_before();
    __syncthreads();
    tc_after();
    const uint32_t tmem = tm_s;
    if (tid == 0) {
        mma_tile(tmem, aA, aB, K, 64, true);
        mma_commit(bar);
        if (!mbar_wait(bar, 0)) { status = 1; atomicExch(err, 1); }
    }
    __syncthreads();
    tc_after();
    if (!status) {
        const int row = m0 + (warp & 3) * 32 + lane, c0 = n0 + (warp >> 2) * 32;
        float v[32];
        tmem_ld32(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (warp >> 2) * 32, v);
        const bool in = row < b;
        const long at = (long)row * MH + c0;
        __align__(16) __nv_bfloat16 h[32];
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
            if (FWD) {
                float g[4];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const float z = v[j + q] + bias[c0 + j + q];
                    h[j + q] = __float2bfloat16_rn(gelu(z));
                    g[q] = gelu_grad(z);
                }
                if (in) *reinterpret_cast<float4*>(G + at + j) = make_float4(g[0], g[1], g[2], g[3]);
            } else {
                float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
                if (in) g = *reinterpret_cast<const float4*>(G + at + j);
                const float4 d = make_float4(v[j] * g.x, v[j + 1] * g.y, v[j + 2] * g.z, v[j + 3] * g.w);
                if (in) *reinterpret_cast<float4*>(D + at + j) = d;
                h[j] = __float2bfloat16_rn(d.x); h[j + 1] = __float2bfloat16_rn(d.y);
                h[j + 2] = __float2bfloat16_rn(d.z); h[j + 3] = __float2bfloat16_rn(d.w);
            }
        }
        if (in) {
#pragma unroll
            for (int j = 0; j < 32; j += 8) *reinterpret_cast<uint4*>(H + at + j) = *reinterpret_cast<const uint4*>(h + j);
        }
        const __nv_bfloat16 zero = __float2bfloat16_rn(0.f);
#pragma unroll
        for (int j = 0; j < 32; j++) HT[(long)(c0 + j) * pitch + row] = in ? h[j] : zero;
    }
    tc_before();
    __syncthreads();
    if (warp == 0) { tc_after(); tmem_free(tmem, 64); }
}

// Output layer of 128 rows, the loss and 64 columns of the last hidden
// layer's gradient: Y = H W4^T + b4, dY = 2 (Y - T) / (12 b),
// d = (dY W4) * G.  Every block column forms Y (one 16-column product);
// column 0 writes dY, dY^T and the loss.
__global__ void __launch_bounds__(TR_THR) k_tr_out(int b, int pitch, const __nv_bfloat16* __restrict__ H3,
        const float* __restrict__ T, const int* __restrict__ idx, const __nv_bfloat16* __restrict__ W,
        const float* __restrict__ bias, const float* __restrict__ G, float* __restrict__ dY, __nv_bfloat16* __restrict__ dYT,
        float* __restrict__ D, __nv_bfloat16* __restrict__ H, __nv_bfloat16* __restrict__ HT, float* __restrict__ loss,
        int* err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t bar_s;
    __shared__ uint32_t tm_s;
    __shared__ int status;
    const uint32_t aA = smem_u32(smem), aW = aA + 128 * MH * 2, aT = aW + NO * MH * 2, aD = aT + 64 * NO * 2,
                   bar = smem_u32(&bar_s);
    uint8_t* sD = smem + (128 * MH + NO * MH + 64 * NO) * 2;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.y * 128, n0 = blockIdx.x * 64;
    tr_stage<NO, MH>(aW, W + BW4, MH, 0, NO);
    tr_stage<64, NO>(aT, W + BT4, NO, n0, MH);
    tr_stage<128, MH>(aA, H3, MH, m0, b);
    tr_stage_commit();
    if (warp == 0) tmem_alloc(smem_u32(&tm_s), 128);
    if (tid == 0) {
        status = 0;
        mbar_init(bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    tr_stage_wait<0>();
    proxy_fence();
    tc_before();
    __syncthreads();
    tc_after();
    const uint32_t tmem = tm_s;
    if (tid == 0) {
        mma_tile(tmem, aA, aW, MH, NO, true);
        mma_commit(bar);
        if (!mbar_wait(bar, 0)) { status = 1; atomicExch(err, 1); }
    }
    __syncthreads();
    tc_after();
    const int row = m0 + (warp & 3) * 32 + lane;
    const bool in = row < b;
    if (!status && warp < 4) {
        float v[16], l = 0.0f;
        tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16), v);
        const float s = 1.0f / ((float)b * MO);
        const float* t = T + (long)(in ? (idx ? idx[row] : row) : 0) * MO;
        __align__(16) __nv_bfloat16 q[16];
#pragma unroll
        for (int j = 0; j < 16; j++) {
            float d = 0.0f;
            if (in && j < MO) {
                const float e = (v[j] + bias[j]) - t[j];
                d = 2.0f * e * s;
                l += e * e * s;
                if (blockIdx.x == 0) dY[(long)row * MO + j] = d;
            }
            q[j] = __float2bfloat16_rn(d);
            if (blockIdx.x == 0) dYT[(long)j * pitch + row] = q[j];
        }
        const int r = warp * 32 + lane;
        *reinterpret_cast<uint4*>(sD + (r >> 3) * (NO * 16) + (r & 7) * 16) = *reinterpret_cast<const uint4*>(q);
        *reinterpret_cast<uint4*>(sD + (r >> 3) * (NO * 16) + 128 + (r & 7) * 16) = *reinterpret_cast<const uint4*>(q + 8);
        if (blockIdx.x == 0) {
            for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
            if (lane == 0) atomicAdd(loss, l);
        }
    }
    proxy_fence();
    tc_before();
    __syncthreads();
    tc_after();
    if (!status && tid == 0) {
        mma_tile(tmem + 32, aD, aT, NO, 64, true);
        mma_commit(bar);
        if (!mbar_wait(bar, 1)) { status = 1; atomicExch(err, 1); }
    }
    __syncthreads();
    tc_after();
    if (!status) {
        const int c0 = n0 + (warp >> 2) * 32;
        float v[32];
        tmem_ld32(tmem + ((uint32_t)((warp & 3) * 32) << 16) + 32 + (warp >> 2) * 32, v);
        const long at = (long)row * MH + c0;
        __align__(16) __nv_bfloat16 h[32];
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
            float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
            if (in) g = *reinterpret_cast<const float4*>(G + at + j);
            const float4 d = make_float4(v[j] * g.x, v[j + 1] * g.y, v[j + 2] * g.z, v[j + 3] * g.w);
            if (in) *reinterpret_cast<float4*>(D + at + j) = d;
            h[j] = __float2bfloat16_rn(d.x); h[j + 1] = __float2bfloat16_rn(d.y);
            h[j + 2] = __float2bfloat16_rn(d.z); h[j + 3] = __float2bfloat16_rn(d.w);
        }
        if (in) {
#pragma unroll
            for (int j = 0; j < 32; j += 8) *reinterpret_cast<uint4*>(H + at + j) = *reinterpret_cast<const uint4*>(h + j);
        }
        const __nv_bfloat16 zero = __float2bfloat16_rn(0.f);
#pragma unroll
        for (int j = 0; j < 32; j++) HT[(long)(c0 + j) * pitch + row] = in ? h[j] : zero;
    }
    tc_before();
    __syncthreads();
    if (warp == 0) { tc_after(); tmem_free(tmem, 128); }
}

// All weight gradients dW = dZ^T H and bias gradients of one mini-batch in one
// launch.  Blocks 0..43: one 128 x 32 tile of a layer's dW each, the rows of
// the mini-batch streamed through a three-stage ring of 128-row chunks in
// row order (44 tiles of that size keep four times more SMs busy than the
// 128 x 64 tiles of one layer at a time).  Blocks 44..47: column sums of one
// layer's dZ, one thread per column adding the rows in order, 64 loads in
// flight.
constexpr int DW_TILES = 16 + 16 + 4 + 8, DW_KC = 128, DW_ST = 3, DW_N = 32;
constexpr int DW_SA = 128 * DW_KC * 2, DW_SB = DW_N * DW_KC * 2;
struct TrGrads {
    const __nv_bfloat16* XT; const __nv_bfloat16* HT[3]; const __nv_bfloat16* DT[4];   // DT[l]: dZ of layer l, transposed
    const float* D[4];
    float* G;
};
__global__ void __launch_bounds__(TR_THR) k_tr_grads(int b, int pitch, TrGrads T, int* err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    const int gW[4] = {OW1, OW2, OW3, OW4}, gB[4] = {OB1, OB2, OB3, OB4};
    const int in[4] = {MI, MH, MH, MH}, out[4] = {MH, MH, MH, MO};
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int t = blockIdx.x;
    if (t >= DW_TILES) {
        const int l = t - DW_TILES, cols = out[l];
        if (tid < cols) {
            const float* d = T.D[l] + tid;
            float s = 0.0f;
            int r = 0;
            for (; r + 64 <= b; r += 64) {
                float v[64];
#pragma unroll
                for (int j = 0; j < 64; j++) v[j] = d[(long)(r + j) * cols];
#pragma unroll
                for (int j = 0; j < 64; j++) s += v[j];
            }
            for (; r < b; r++) s += d[(long)r * cols];
            T.G[gB[l] + tid] = s;
        }
        return;
    }
    int l, tm, tn;
    if (t < 16) { l = 2; tm = t >> 3; tn = t & 7; }
    else if (t < 32) { l = 1; tm = (t - 16) >> 3; tn = (t - 16) & 7; }
    else if (t < 40) { l = 3; tm = 0; tn = t - 32; }
    else { l = 0; tm = (t - 40) >> 1; tn = (t - 40) & 1; }
    __shared__ __align__(8) uint64_t bar_s[DW_ST];
    __shared__ uint32_t tm_s;
    __shared__ int status;
    const __nv_bfloat16* A = T.DT[l];
    const __nv_bfloat16* B = l == 0 ? T.XT : T.HT[l - 1];
    const uint32_t s0 = smem_u32(smem);
    const int nch = pitch / DW_KC, m0 = tm * 128, n0 = tn * DW_N;
    auto stage = [&](int c) {
        if (c < nch) {
            const uint32_t at = s0 + (c % DW_ST) * (DW_SA + DW_SB);
            tr_stage<128, DW_KC>(at, A + c * DW_KC, pitch, m0, out[l]);
            tr_stage<DW_N, DW_KC>(at + DW_SA, B + c * DW_KC, pitch, n0, in[l]);
        }
        tr_stage_commit();
    };
    stage(0);
    stage(1);
    if (warp == 0) tmem_alloc(smem_u32(&tm_s), 32);
    if (tid == 0) {
        status = 0;
        for (int i = 0; i < DW_ST; i++) mbar_init(smem_u32(bar_s + i), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    tc_before();
    __syncthreads();
    tc_after();
    const uint32_t tmem = tm_s;
    for (int c = 0; c < nch; c++) {
        // chunk c + 2 goes where chunk c - 1 was: its products must have been read
        if (c > 0 && !mbar_wait(smem_u32(bar_s + (c - 1) % DW_ST), ((c - 1) / DW_ST) & 1)) { status = 1; atomicExch(err, 1); }
        stage(c + 2);
        tr_stage_wait<2>();
        proxy_fence();
        __syncthreads();
        if (status) break;
        if (tid == 0) {
            const uint32_t at = s0 + (c % DW_ST) * (DW_SA + DW_SB);
            mma_tile(tmem, at, at + DW_SA, DW_KC, DW_N, c == 0);
            mma_commit(smem_u32(bar_s + c % DW_ST));
        }
    }
    if (!status && !mbar_wait(smem_u32(bar_s + (nch - 1) % DW_ST), ((nch - 1) / DW_ST) & 1)) { status = 1; atomicExch(err, 1); }
    tr_stage_wait<0>();
    __syncthreads();
    tc_after();
    if (!status) {
        const int m = m0 + (warp & 3) * 32 + lane, c0 = (warp >> 2) * 16;
        float v[16];
        tmem_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + c0, v);
        if (m < out[l]) {
#pragma unroll
            for (int j = 0; j < 16; j++)
                if (n0 + c0 + j < in[l]) T.G[gW[l] + (long)m * in[l] + n0 + c0 + j] = v[j];
        }
    }
    tc_before();
    __syncthreads();
    if (warp == 0) { tc_after(); tmem_free(tmem, 32); }
}
// Adam step and the rounded copies of the new weights
__global__ void k_adam(long n, float* P, const float* __restrict__ G, float* m, float* v, float lr, float b1t, float b2t,
                       __nv_bfloat16* W) {
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    GS_LOOP(i, n) {
        float g = G[i];
        float mi = b1 * m[i] + (1.0f - b1) * g, vi = b2 * v[i] + (1.0f - b2) * g * g;
        m[i] = mi; v[i] = vi;
        float p = P[i];
        p -= lr * (mi / (1.0f - b1t)) / (sqrtf(vi / (1.0f - b2t)) + eps);
        P[i] = p;
        tr_pack_one(i, p, W);
    }
}

} // namespace

// ------------------------------------------------------------------ inference state per handle
struct MlpDev {
    uint8_t* pack = nullptr;   // PTOT bytes
    float* bias = nullptr;     // 4 * 256
    float* norm = nullptr;     // ABD_MLP_NNORM
    float* y = nullptr; int ycap = 0;
    float* feat = nullptr;
    int* err = nullptr;
    float* io = nullptr; int iocap = 0;      // rows in and out of abd_mlp_forward
    std::mutex io_mu;                        // one call at a time uses them
};
// rows that abd_mlp_forward takes at once, and so the most it keeps room for
// (15 MB); more rows than that hide the copies' fixed costs anyway
constexpr int MLP_SLAB = 65536;

void eng_mlp_free(Engine* E) {
    MlpDev* M = reinterpret_cast<MlpDev*>(E->mlp);
    if (!M) return;
    void* ps[] = {M->pack, M->bias, M->norm, M->y, M->feat, M->err, M->io};
    for (void* p : ps) if (p) cudaFree(p);
    delete M;
    E->mlp = nullptr;
}

static int mlp_infer(Engine* E, const float* X, int n, float* Y) {
    MlpDev* M = reinterpret_cast<MlpDev*>(E->mlp);
    static bool attr_set[64] = {false};
    int dev = E->device;
    if (dev < 64 && !attr_set[dev]) {
        CUDA_TRY(cudaFuncSetAttribute(k_mlp_infer, cudaFuncAttributeMaxDynamicSharedMemorySize, S_TOT));
        attr_set[dev] = true;
    }
    if (n <= 0) return ABD_OK;
    k_mlp_infer<<<(n + 127) / 128, NTHR, S_TOT, E->stream>>>(n, X, M->norm, M->pack, M->bias, Y, M->err);
    E->launches++;
    return ABD_OK;
}
// learned increment: ws = inertial increment + dt * (body frame -> world) y
__global__ void k_ws_learned(int nb, const double* __restrict__ st, const float* __restrict__ y,
                             const double* __restrict__ mass, double dt, double g0, double g1, double g2, double* ws) {
    GS_LOOP(b, nb) {
        double* w = ws + 12 * b;
        if (!(mass[b] > 0.0)) { for (int i = 0; i < 12; i++) w[i] = 0.0; continue; }
        const double* now = st + ST_STRIDE * b + ST_NOW;
        const double* q = now + ST_Q;
        // inverse of q by the adjugate
        double c00 = q[4] * q[8] - q[5] * q[7], c01 = q[5] * q[6] - q[3] * q[8], c02 = q[3] * q[7] - q[4] * q[6];
        double det = q[0] * c00 + q[1] * c01 + q[2] * c02;
        double id = det != 0.0 ? 1.0 / det : 0.0;
        double qi[9] = {c00 * id, (q[2] * q[7] - q[1] * q[8]) * id, (q[1] * q[5] - q[2] * q[4]) * id,
                        c01 * id, (q[0] * q[8] - q[2] * q[6]) * id, (q[2] * q[3] - q[0] * q[5]) * id,
                        c02 * id, (q[1] * q[6] - q[0] * q[7]) * id, (q[0] * q[4] - q[1] * q[3]) * id};
        const float* r = y + 12 * b;
        double gv[3] = {g0, g1, g2};
        for (int i = 0; i < 3; i++) {
            double s = 0;
            for (int k = 0; k < 3; k++) s += qi[3 * i + k] * r[k];
            w[i] = dt * now[ST_V + i] + dt * dt * gv[i] + dt * s;
        }
        // dq = (q^-1 M)^T: row i of dq, column j = (q^-1 M)[j][i]
        for (int i = 0; i < 3; i++)
            for (int j = 0; j < 3; j++) {
                double s = 0;
                for (int k = 0; k < 3; k++) s += qi[3 * j + k] * r[3 + 3 * k + i];
                w[3 + 3 * i + j] = dt * now[ST_QD + 3 * i + j] + dt * s;
            }
    }
}

int eng_features(Engine* E, float* feat_dev);

// warm start of the next step from the network (warm_start 3)
int eng_learned_ws(Engine* E) {
    MlpDev* M = reinterpret_cast<MlpDev*>(E->mlp);
    if (!M) return E->fail(ABD_ERR_INVALID_ARG, "warm_start 3 needs abd_set_mlp first");
    int rc;
    if ((rc = eng_features(E, M->feat))) return rc;
    if ((rc = mlp_infer(E, M->feat, E->nb, M->y))) return rc;
    const AbdParams& P = E->P;
    k_ws_learned<<<grid_for(E->nb), 256, 0, E->stream>>>(E->nb, E->st, M->y, E->mass, P.dt, P.gravity[0], P.gravity[1],
                                                         P.gravity[2], E->ws);
    E->launches++;
    return ABD_OK;
}

extern "C" int abd_set_mlp(AbdHandle* h, const float* params, const float* norm) {
    Engine* E = reinterpret_cast<Engine*>(h);
    if (!E) return ABD_ERR_INVALID_ARG;
    if (!params || !norm) return E->fail(ABD_ERR_INVALID_ARG, "abd_set_mlp: null");
    if (cudaSetDevice(E->device) != cudaSuccess) return E->fail(ABD_ERR_CUDA, "cudaSetDevice");
    if (!E->mlp) {
        MlpDev* M = new MlpDev();
        E->mlp = M;
        if (cudaMalloc(&M->pack, PTOT) != cudaSuccess || cudaMalloc(&M->bias, sizeof(float) * 4 * MH) != cudaSuccess ||
            cudaMalloc(&M->norm, sizeof(float) * ABD_MLP_NNORM) != cudaSuccess ||
            cudaMalloc(&M->y, sizeof(float) * MO * (size_t)E->nb) != cudaSuccess ||
            cudaMalloc(&M->feat, sizeof(float) * MI * (size_t)E->nb) != cudaSuccess ||
            cudaMalloc(&M->err, sizeof(int)) != cudaSuccess) {
            eng_mlp_free(E);
            return E->fail(ABD_ERR_CUDA, "cudaMalloc mlp");
        }
    }
    MlpDev* M = reinterpret_cast<MlpDev*>(E->mlp);
    float* P = nullptr;
    if (cudaMalloc(&P, sizeof(float) * NPARAM) != cudaSuccess) return E->fail(ABD_ERR_CUDA, "cudaMalloc params");
    cudaError_t e = cudaMemcpyAsync(P, params, sizeof(float) * NPARAM, cudaMemcpyHostToDevice, E->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(M->err, 0, sizeof(int), E->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(M->norm, norm, sizeof(float) * ABD_MLP_NNORM, cudaMemcpyHostToDevice, E->stream);
    if (e == cudaSuccess) {
        k_mlp_pack<<<grid_for((long)MH * MH), 256, 0, E->stream>>>(P, reinterpret_cast<__nv_bfloat16*>(M->pack), M->bias);
        e = eng_stream_sync(E);
    }
    cudaFree(P);
    if (e != cudaSuccess) return E->fail(ABD_ERR_CUDA, std::string("abd_set_mlp: ") + cudaGetErrorString(e));
    return ABD_OK;
}

extern "C" int abd_mlp_forward(AbdHandle* h, const float* x, int32_t n, float* y) {
    Engine* E = reinterpret_cast<Engine*>(h);
    if (!E) return ABD_ERR_INVALID_ARG;
    if (!E->mlp) return E->fail(ABD_ERR_INVALID_ARG, "abd_mlp_forward: no network set");
    if (n < 0 || (n > 0 && (!x || !y))) return E->fail(ABD_ERR_INVALID_ARG, "abd_mlp_forward: bad arguments");
    if (n == 0) return ABD_OK;
    if (cudaSetDevice(E->device) != cudaSuccess) return E->fail(ABD_ERR_CUDA, "cudaSetDevice");
    MlpDev* M = reinterpret_cast<MlpDev*>(E->mlp);
    std::lock_guard<std::mutex> lock(M->io_mu);
    // two buffers kept for the next call: allocating and freeing them on each
    // call took 1,280 of 2,290 us for 50,021 rows
    const int rows = n < MLP_SLAB ? n : MLP_SLAB;
    if (rows > M->iocap) {
        if (M->io) { CUDA_TRY(eng_stream_sync(E)); cudaFree(M->io); }
        M->io = nullptr; M->iocap = 0;
        if (cudaMalloc(&M->io, sizeof(float) * (MI + MO) * (size_t)rows) != cudaSuccess) {
            M->io = nullptr;
            return E->fail(ABD_ERR_CUDA, "cudaMalloc mlp io");
        }
        M->iocap = rows;
    }
    float *dx = M->io, *dy = M->io + (size_t)MI * M->iocap;
    int flag = 0;
    CUDA_TRY(cudaMemsetAsync(M->err, 0, sizeof(int), E->stream));
    for (int r = 0; r < n; r += rows) {
        const int k = n - r < rows ? n - r : rows;
        if (cudaMemcpyAsync(dx, x + (size_t)MI * r, sizeof(float) * MI * (size_t)k, cudaMemcpyHostToDevice, E->stream) != cudaSuccess)
            return E->fail(ABD_ERR_CUDA, "abd_mlp_forward: copy in");
        int rc = mlp_infer(E, dx, k, dy);
        if (rc) return rc;
        if (cudaMemcpyAsync(y + (size_t)MO * r, dy, sizeof(float) * MO * (size_t)k, cudaMemcpyDeviceToHost, E->stream) != cudaSuccess)
            return E->fail(ABD_ERR_CUDA, "abd_mlp_forward: copy out");
    }
    cudaError_t e = cudaMemcpyAsync(&flag, M->err, sizeof(int), cudaMemcpyDeviceToHost, E->stream);
    if (e == cudaSuccess) e = eng_stream_sync(E);
    if (e != cudaSuccess) return E->fail(ABD_ERR_CUDA, "abd_mlp_forward: copy out");
    if (flag) return E->fail(ABD_ERR_CUDA, "mlp inference: a wait ran out");
    return ABD_OK;
}

// ------------------------------------------------------------------ trainer
struct AbdTrainer {
    int device = 0;
    cudaStream_t s = nullptr;
    float *P = nullptr, *G = nullptr, *m = nullptr, *v = nullptr;
    __nv_bfloat16* W = nullptr;        // BF16 copies of the weights (BTOT)
    long t = 0;
    float *X = nullptr, *T = nullptr; int n = 0;
    // mini-batch workspace for bcap rows, kept between calls
    int bcap = 0;
    uint8_t* ws = nullptr;
    int* idx = nullptr; int icap = 0;  // row order of an epoch
    float* loss = nullptr; int lcap = 0;   // losses of an epoch's mini-batches
    int* dflag = nullptr;              // set by a tensor-core product whose wait gave up
    std::string err;
};

// the workspace of b rows: activations and gradients of the three hidden
// layers (BF16 row-major and transposed, FP32 gradients, gelu') and of the output
struct TrWork {
    int pitch;
    __nv_bfloat16 *XT, *H[3], *HT[3], *DB[3], *DT[3], *dYT;
    float *G[3], *D[3], *dY, *Xg, *Tg;
};
static size_t tr_layout(uint8_t* base, int b, TrWork* w) {
    TrWork l;
    size_t at = 0;
    auto take = [&](size_t bytes) { uint8_t* p = base + at; at += (bytes + 255) / 256 * 256; return p; };
    l.pitch = (b + 127) / 128 * 128;
    const size_t row = (size_t)b * MH, col = (size_t)l.pitch * MH;
    l.XT = (__nv_bfloat16*)take(2 * (size_t)K1 * l.pitch);
    for (int i = 0; i < 3; i++) {
        l.H[i] = (__nv_bfloat16*)take(2 * row); l.HT[i] = (__nv_bfloat16*)take(2 * col);
        l.DB[i] = (__nv_bfloat16*)take(2 * row); l.DT[i] = (__nv_bfloat16*)take(2 * col);
        l.G[i] = (float*)take(4 * row); l.D[i] = (float*)take(4 * row);
    }
    l.dYT = (__nv_bfloat16*)take(2 * (size_t)NO * l.pitch);
    l.dY = (float*)take(4 * (size_t)MO * b);
    l.Xg = (float*)take(4 * (size_t)MI * b); l.Tg = (float*)take(4 * (size_t)MO * b);
    if (w) *w = l;
    return at;
}
static bool tr_reserve(AbdTrainer* T, int b) {
    if (b <= T->bcap) return true;
    if (T->ws) { cudaStreamSynchronize(T->s); cudaFree(T->ws); }
    T->ws = nullptr; T->bcap = 0;
    if (cudaMalloc(&T->ws, tr_layout(nullptr, b, nullptr)) != cudaSuccess) { T->ws = nullptr; return false; }
    T->bcap = b;
    return true;
}
constexpr int TR_S64 = (128 + 64) * K1 * 2, TR_S256 = (128 + 64) * MH * 2,
              TR_SOUT = (128 * MH + NO * MH + 64 * NO + 128 * NO) * 2, TR_SDW = DW_ST * (DW_SA + DW_SB);
static cudaError_t tr_attributes() {
    cudaError_t e;
    if ((e = cudaFuncSetAttribute(k_tr_layer<MH, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, TR_S256))) return e;
    if ((e = cudaFuncSetAttribute(k_tr_layer<MH, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, TR_S256))) return e;
    if ((e = cudaFuncSetAttribute(k_tr_out, cudaFuncAttributeMaxDynamicSharedMemorySize, TR_SOUT))) return e;
    return cudaFuncSetAttribute(k_tr_grads, cudaFuncAttributeMaxDynamicSharedMemorySize, TR_SDW);
}

// loss (added to *loss) and gradient (into T->G) of b rows of X / Tg, in the
// order idx (null: all in order).  A pass over 10,007 rows in mini-batches of
// 512 takes 2.01 ms (8 launches of about 9.5 us per mini-batch with Adam)
// against 12.08 ms with one product per launch on FP32 operands staged
// element by element, separate activation kernels and one-block column sums;
// gradients and weights are the same bits.
static void tr_forward_backward(AbdTrainer* T, int b, const float* X, const float* Tg, const int* idx, float* loss) {
    cudaStream_t s = T->s;
    TrWork w;
    tr_layout(T->ws, b, &w);
    const dim3 g(MH / 64, (b + 127) / 128);
    const float* P = T->P;
    k_tr_layer<K1, true><<<g, TR_THR, TR_S64, s>>>(b, w.pitch, nullptr, X, idx, w.XT, T->W + BW1, P + OB1, w.G[0], nullptr,
                                                   w.H[0], w.HT[0], T->dflag);
    k_tr_layer<MH, true><<<g, TR_THR, TR_S256, s>>>(b, w.pitch, w.H[0], nullptr, nullptr, nullptr, T->W + BW2, P + OB2, w.G[1],
                                                    nullptr, w.H[1], w.HT[1], T->dflag);
    k_tr_layer<MH, true><<<g, TR_THR, TR_S256, s>>>(b, w.pitch, w.H[1], nullptr, nullptr, nullptr, T->W + BW3, P + OB3, w.G[2],
                                                    nullptr, w.H[2], w.HT[2], T->dflag);
    k_tr_out<<<g, TR_THR, TR_SOUT, s>>>(b, w.pitch, w.H[2], Tg, idx, T->W, P + OB4, w.G[2], w.dY, w.dYT, w.D[2], w.DB[2],
                                        w.DT[2], loss, T->dflag);
    k_tr_layer<MH, false><<<g, TR_THR, TR_S256, s>>>(b, w.pitch, w.DB[2], nullptr, nullptr, nullptr, T->W + BT3, nullptr, w.G[1],
                                                     w.D[1], w.DB[1], w.DT[1], T->dflag);
    k_tr_layer<MH, false><<<g, TR_THR, TR_S256, s>>>(b, w.pitch, w.DB[1], nullptr, nullptr, nullptr, T->W + BT2, nullptr, w.G[0],
                                                     w.D[0], w.DB[0], w.DT[0], T->dflag);
    TrGrads q;
    q.XT = w.XT;
    for (int i = 0; i < 3; i++) { q.HT[i] = w.HT[i]; q.DT[i] = w.DT[i]; q.D[i] = w.D[i]; }
    q.DT[3] = w.dYT; q.D[3] = w.dY; q.G = T->G;
    k_tr_grads<<<DW_TILES + 4, TR_THR, TR_SDW, s>>>(b, w.pitch, q, T->dflag);
}

#define TR_TRY(x) do { cudaError_t _e = (x); if (_e != cudaSuccess) { T->err = std::string(#x) + ": " + cudaGetErrorString(_e); return ABD_ERR_CUDA; } } while (0)

extern "C" int abd_trainer_create(int32_t device, const float* params, AbdTrainer** out) {
    if (!params || !out) return ABD_ERR_INVALID_ARG;
    AbdTrainer* T = new AbdTrainer();
    T->device = device;
    *out = nullptr;
    if (cudaSetDevice(device) != cudaSuccess || cudaStreamCreateWithFlags(&T->s, cudaStreamNonBlocking) != cudaSuccess) {
        delete T;
        return ABD_ERR_NO_DEVICE;
    }
    size_t nb = sizeof(float) * NPARAM;
    if (cudaMalloc(&T->P, nb) != cudaSuccess || cudaMalloc(&T->W, 2 * BTOT) != cudaSuccess || cudaMalloc(&T->G, nb) != cudaSuccess ||
        cudaMalloc(&T->m, nb) != cudaSuccess || cudaMalloc(&T->v, nb) != cudaSuccess ||
        cudaMalloc(&T->dflag, sizeof(int)) != cudaSuccess) {
        *out = T;
        T->err = "cudaMalloc trainer";
        return ABD_ERR_CUDA;
    }
    *out = T;
    TR_TRY(cudaMemcpyAsync(T->P, params, nb, cudaMemcpyHostToDevice, T->s));
    TR_TRY(cudaMemsetAsync(T->m, 0, nb, T->s));
    TR_TRY(cudaMemsetAsync(T->v, 0, nb, T->s));
    TR_TRY(cudaMemsetAsync(T->dflag, 0, sizeof(int), T->s));
    TR_TRY(cudaMemsetAsync(T->W, 0, 2 * BTOT, T->s));      // the padding stays zero
    TR_TRY(tr_attributes());
    k_tr_pack<<<grid_for(NPARAM), 256, 0, T->s>>>(T->P, T->W);
    TR_TRY(cudaStreamSynchronize(T->s));
    return ABD_OK;
}

extern "C" int abd_trainer_destroy(AbdTrainer* T) {
    if (!T) return ABD_ERR_INVALID_ARG;
    cudaSetDevice(T->device);
    void* ps[] = {T->P, T->W, T->G, T->m, T->v, T->X, T->T, T->loss, T->idx, T->ws, T->dflag};
    for (void* p : ps) if (p) cudaFree(p);
    if (T->s) cudaStreamDestroy(T->s);
    delete T;
    return ABD_OK;
}

extern "C" const char* abd_trainer_last_error(AbdTrainer* T) { return T ? T->err.c_str() : "null trainer"; }

extern "C" int abd_trainer_set_data(AbdTrainer* T, const float* x, const float* y, int32_t n) {
    if (!T || n <= 0 || !x || !y) return ABD_ERR_INVALID_ARG;
    if (cudaSetDevice(T->device) != cudaSuccess) return ABD_ERR_CUDA;
    if (T->X) cudaFree(T->X);
    if (T->T) cudaFree(T->T);
    T->X = T->T = nullptr;
    TR_TRY(cudaMalloc(&T->X, sizeof(float) * MI * (size_t)n));
    TR_TRY(cudaMalloc(&T->T, sizeof(float) * MO * (size_t)n));
    TR_TRY(cudaMemcpyAsync(T->X, x, sizeof(float) * MI * (size_t)n, cudaMemcpyHostToDevice, T->s));
    TR_TRY(cudaMemcpyAsync(T->T, y, sizeof(float) * MO * (size_t)n, cudaMemcpyHostToDevice, T->s));
    TR_TRY(cudaStreamSynchronize(T->s));
    T->n = n;
    return ABD_OK;
}

// One pass over `order` (n row indices into the data set) in mini-batches of
// `batch` rows, one Adam step per mini-batch; *mean_loss gets the mean of
// the mini-batch losses.
extern "C" int abd_trainer_epoch(AbdTrainer* T, const int32_t* order, int32_t n, int32_t batch, float lr, float* mean_loss) {
    if (!T || !order || n <= 0 || batch <= 0 || !T->X) return ABD_ERR_INVALID_ARG;
    for (int i = 0; i < n; i++) if (order[i] < 0 || order[i] >= T->n) { T->err = "abd_trainer_epoch: index out of range"; return ABD_ERR_INVALID_ARG; }
    if (cudaSetDevice(T->device) != cudaSuccess) return ABD_ERR_CUDA;
    batch = std::min(batch, n);
    if (!tr_reserve(T, batch)) { T->err = "cudaMalloc batch"; return ABD_ERR_CUDA; }
    const int nbat = (n + batch - 1) / batch;
    if (n > T->icap) {
        if (T->idx) cudaFree(T->idx);
        T->idx = nullptr; T->icap = 0;
        TR_TRY(cudaMalloc(&T->idx, sizeof(int) * (size_t)n));
        T->icap = n;
    }
    if (nbat > T->lcap) {
        if (T->loss) cudaFree(T->loss);
        T->loss = nullptr; T->lcap = 0;
        TR_TRY(cudaMalloc(&T->loss, sizeof(float) * (size_t)nbat));
        T->lcap = nbat;
    }
    TR_TRY(cudaMemcpyAsync(T->idx, order, sizeof(int) * (size_t)n, cudaMemcpyHostToDevice, T->s));
    TR_TRY(cudaMemsetAsync(T->loss, 0, sizeof(float) * (size_t)nbat, T->s));
    for (int k = 0; k < nbat; k++) {
        int b = std::min(batch, n - k * batch);
        tr_forward_backward(T, b, T->X, T->T, T->idx + (long)k * batch, T->loss + k);
        T->t++;
        float b1t = powf(0.9f, (float)T->t), b2t = powf(0.999f, (float)T->t);
        k_adam<<<grid_for(NPARAM), 256, 0, T->s>>>(NPARAM, T->P, T->G, T->m, T->v, lr, b1t, b2t, T->W);
    }
    std::vector<float> hl(nbat);
    TR_TRY(cudaGetLastError());
    TR_TRY(cudaMemcpyAsync(hl.data(), T->loss, sizeof(float) * nbat, cudaMemcpyDeviceToHost, T->s));
    int flag = 0;
    TR_TRY(cudaMemcpyAsync(&flag, T->dflag, sizeof(int), cudaMemcpyDeviceToHost, T->s));
    TR_TRY(cudaStreamSynchronize(T->s));
    if (flag) { T->err = "tensor-core GEMM: an mbarrier wait gave up"; return ABD_ERR_CUDA; }
    double s = 0;
    for (float v : hl) s += v;
    if (mean_loss) *mean_loss = (float)(s / nbat);
    return ABD_OK;
}

// Loss and gradient of the current parameters on the given rows (no update).
extern "C" int abd_trainer_grad(AbdTrainer* T, const float* x, const float* y, int32_t n, float* grad, float* loss) {
    if (!T || !x || !y || n <= 0 || !grad) return ABD_ERR_INVALID_ARG;
    if (cudaSetDevice(T->device) != cudaSuccess) return ABD_ERR_CUDA;
    if (!tr_reserve(T, n)) { T->err = "cudaMalloc batch"; return ABD_ERR_CUDA; }
    if (!T->loss) { TR_TRY(cudaMalloc(&T->loss, sizeof(float))); T->lcap = 1; }
    TrWork w;
    tr_layout(T->ws, n, &w);
    TR_TRY(cudaMemcpyAsync(w.Xg, x, sizeof(float) * MI * (size_t)n, cudaMemcpyHostToDevice, T->s));
    TR_TRY(cudaMemcpyAsync(w.Tg, y, sizeof(float) * MO * (size_t)n, cudaMemcpyHostToDevice, T->s));
    TR_TRY(cudaMemsetAsync(T->loss, 0, sizeof(float), T->s));
    tr_forward_backward(T, n, w.Xg, w.Tg, nullptr, T->loss);
    TR_TRY(cudaGetLastError());
    TR_TRY(cudaMemcpyAsync(grad, T->G, sizeof(float) * NPARAM, cudaMemcpyDeviceToHost, T->s));
    float l = 0;
    int flag = 0;
    TR_TRY(cudaMemcpyAsync(&l, T->loss, sizeof(float), cudaMemcpyDeviceToHost, T->s));
    TR_TRY(cudaMemcpyAsync(&flag, T->dflag, sizeof(int), cudaMemcpyDeviceToHost, T->s));
    TR_TRY(cudaStreamSynchronize(T->s));
    if (flag) { T->err = "tensor-core GEMM: an mbarrier wait gave up"; return ABD_ERR_CUDA; }
    if (loss) *loss = l;
    return ABD_OK;
}

extern "C" int abd_trainer_params(AbdTrainer* T, float* params) {
    if (!T || !params) return ABD_ERR_INVALID_ARG;
    if (cudaSetDevice(T->device) != cudaSuccess) return ABD_ERR_CUDA;
    TR_TRY(cudaMemcpyAsync(params, T->P, sizeof(float) * NPARAM, cudaMemcpyDeviceToHost, T->s));
    TR_TRY(cudaStreamSynchronize(T->s));
    return ABD_OK;
}
