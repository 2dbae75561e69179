// Fused self-attention forward of the transformer clients (bfloat16, head dimension 64, any sequence length):
//
//   ctx[b, q, h*64 + :] = softmax( Q[b,h,q,:] . K[b,h,:,:]^T * scale  (+ causal mask) ) . V[b,h,:,:]
//
// read straight from the fused projection output qkv [B, S, 3, H, 64] and written as [B, S, H*64] — no probability tensor
// and no re-laid-out Q / K / V copies in HBM.  It stands in for the two cublasSgemmStridedBatched calls around a softmax
// kernel that the reference replays for an attention layer (reference src/scheduler/utils_sched.cpp:502-513).
//
// One work item = 128 query rows of one (batch, head); a persistent grid walks the items, 64 keys a step by the online softmax
// (Milakov and Gimelshein, 2018): sums and output are relative to a running reference maximum, here one that moves only when a
// row's maximum has outgrown it by 2^8.  Bound: the exponentials (16 per clock and SM; the two products of a step take a third of that time), so what
// counts is that twelve softmax warps per SM always have scores to work on: scores and output of one item take 128
// tensor-memory columns and 66 KB of shared memory, and three items share an SM.
// 8 x 384 x 12 heads: 33.1 us with all scores of a query tile in tensor memory (one item per SM, two passes over them), 15.0 now;
// 16 x 512 x 16 heads, causal, in three launches: 43 us.
// Every wait is bounded; on expiry the kernel sets the status word, frees tensor memory and returns.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#include "elastic.h"
#include "sm100_primitives.cuh"

namespace ob200 {

constexpr int AT_D = 64;            // head dimension
constexpr int AT_QROWS = 128;       // query rows per work item
constexpr int AT_KEYS = 64;         // keys per step
constexpr int AT_THREADS = 192;     // warps 0-3: softmax / epilogue (one thread per query row), warp 4: TMA, warp 5: MMA issue
constexpr int AT_Q_BYTES = AT_QROWS * 128, AT_KV_BYTES = AT_KEYS * 128, AT_P_BYTES = AT_QROWS * 128;
constexpr int AT_RING = 2;          // K tiles and V tiles in flight
constexpr int AT_SMEM = AT_Q_BYTES + 2 * AT_RING * AT_KV_BYTES + AT_P_BYTES + 1024 + 256;   // + alignment, barriers
constexpr int AT_CTAS_PER_SM = 3;   // 66 KB of shared memory, 128 tensor-memory columns and at most 112 registers per thread each
constexpr float AT_RESCALE = 8.f;   // the reference maximum moves when a row's maximum outgrows it by 2^8

struct AttnParams {
    void* ctx;             // [B, S, H*64] bfloat16
    int* status;
    int B, S, H;
    int causal;
    float factor;          // what the scores are multiplied by ahead of the mask: 1, or -1 / 0 for a negative / zero scale
    float scale_log2;      // |scale| * log2(e); 1 for a zero scale, so that a masked score stays -infinity
    int q_tiles;           // ceil(S / 128)
    int first, last;       // work items [first, last) of this launch
    alignas(64) unsigned char tmap[128];   // qkv as [B][S][3H][64], boxes of 64 rows
};

struct AttnCtl {
    uint64_t q_full, q_empty;
    uint64_t k_full[AT_RING], k_empty[AT_RING], v_full[AT_RING], v_empty[AT_RING];
    uint64_t s_full, s_free, p_full, o_full;
    uint32_t tmem_base;
    int abort_flag;
};

__device__ __forceinline__ float exp2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ void attn_give_up(AttnCtl* ctl, int* status, int code) {
    if (!*(volatile int*)&ctl->abort_flag) {
        ctl->abort_flag = 1;
        if (status) atomicExch(status, code);
    }
}

// Work item -> (query tile, head, batch, key steps).  The longest items of a causal problem come first, so that the last
// wave is made of short ones.
struct AttnItem {
    int qt, h, b, steps;
    __device__ __forceinline__ AttnItem(const AttnParams& p, int item) {
        const int bh_count = p.B * p.H;
        qt = p.q_tiles - 1 - item / bh_count;
        const int bh = item % bh_count;
        h = bh % p.H;
        b = bh / p.H;
        int keys = p.S;
        if (p.causal && (qt + 1) * AT_QROWS < keys) keys = (qt + 1) * AT_QROWS;   // keys past the tile's last query row never count
        steps = (keys + AT_KEYS - 1) / AT_KEYS;
    }
};

__global__ void __launch_bounds__(AT_THREADS, AT_CTAS_PER_SM) attention_fwd_kernel(const __grid_constant__ AttnParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* q_s = smem;
    uint8_t* k_s = q_s + AT_Q_BYTES;
    uint8_t* v_s = k_s + AT_RING * AT_KV_BYTES;
    uint8_t* p_s = v_s + AT_RING * AT_KV_BYTES;
    AttnCtl* ctl = reinterpret_cast<AttnCtl*>(p_s + AT_P_BYTES);
    const int tid = threadIdx.x, warp = uniform_warp_index(), lane = tid & 31;

    if (tid == 0) {
        mbar_init(&ctl->q_full, 1);
        mbar_init(&ctl->q_empty, 1);
        for (int i = 0; i < AT_RING; i++) {
            mbar_init(&ctl->k_full[i], 1);
            mbar_init(&ctl->k_empty[i], 1);
            mbar_init(&ctl->v_full[i], 1);
            mbar_init(&ctl->v_empty[i], 1);
        }
        mbar_init(&ctl->s_full, 1);
        mbar_init(&ctl->s_free, 4);    // one elected lane per softmax warp
        mbar_init(&ctl->p_full, 4);
        mbar_init(&ctl->o_full, 1);
        ctl->abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 5) {
        if (lane == 0) prefetch_tensormap(p.tmap);
        tmem_alloc(&ctl->tmem_base, 2 * AT_KEYS);   // 64 columns of scores, 64 of output
        tmem_relinquish();
        tc_fence_before_sync();
    }
    __syncthreads();
    tc_fence_after_sync();
    pdl_wait();
    if (tid == 0) pdl_launch_dependents();
    const uint32_t t_s = ctl->tmem_base, t_o = t_s + AT_KEYS;
    volatile int* abort_flag = &ctl->abort_flag;
    const int items = p.last;

    if (warp == 4) {
        // ------------------------------------------------------------ TMA (the warp as one, see elect_one)
        uint32_t n = 0, local = 0;   // key steps, items
        bool dead = false;
        for (int item = p.first + blockIdx.x; item < items && !dead; item += gridDim.x, local++) {
            const AttnItem it(p, item);
            dead = !mbar_wait_warp(&ctl->q_empty, (local & 1u) ^ 1u, abort_flag);
            if (dead) break;
            if (elect_one()) {
                mbar_arrive_expect_tx(&ctl->q_full, AT_Q_BYTES);
#pragma unroll
                for (int g = 0; g < 2; g++)
                    tma_load_tile_4d(smem_u32(q_s + g * 64 * 128), p.tmap, &ctl->q_full, 0, it.h, it.qt * AT_QROWS + g * 64, it.b);
            }
            __syncwarp();
            for (int t = 0; t < it.steps; t++, n++) {
                const uint32_t s = n % AT_RING, ph = (n / AT_RING) & 1u;
                dead = !mbar_wait_warp(&ctl->k_empty[s], ph ^ 1u, abort_flag);
                if (dead) break;
                if (elect_one()) {
                    mbar_arrive_expect_tx(&ctl->k_full[s], AT_KV_BYTES);
                    tma_load_tile_4d(smem_u32(k_s + s * AT_KV_BYTES), p.tmap, &ctl->k_full[s], 0, p.H + it.h, t * AT_KEYS, it.b);
                }
                __syncwarp();
                dead = !mbar_wait_warp(&ctl->v_empty[s], ph ^ 1u, abort_flag);
                if (dead) break;
                if (elect_one()) {
                    mbar_arrive_expect_tx(&ctl->v_full[s], AT_KV_BYTES);
                    tma_load_tile_4d(smem_u32(v_s + s * AT_KV_BYTES), p.tmap, &ctl->v_full[s], 0, 2 * p.H + it.h, t * AT_KEYS, it.b);
                }
                __syncwarp();
            }
        }
        if (dead) attn_give_up(ctl, p.status, OB200_ERR_WAIT_EMPTY);
    } else if (warp == 5) {
        // ------------------------------------------------------------ MMA issue (the warp as one)
        // S(n) = Q . K(n)^T is issued as soon as the softmax warps have the scores of step n-1 in registers, before P(n-1) is
        // ready, so it runs under their exponentials; O += P(n) . V(n) follows when P(n) is in shared memory.
        const uint32_t idesc_s = umma_idesc(1, AT_QROWS, AT_KEYS), idesc_o = umma_idesc(1, AT_QROWS, AT_D) | UMMA_IDESC_B_MN;
        const uint64_t qd = umma_desc_sw128(smem_u32(q_s)), pd = umma_desc_sw128(smem_u32(p_s));
        // V lies as [key][64]: MN-major, atoms of 8 keys x 128 bytes, 1024 bytes apart along the reduction
        const uint64_t v_bits = ((uint64_t)(8192 >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
        uint32_t n = 0, local = 0;
        bool dead = false;
        auto scores = [&](uint32_t i, bool last) {
            const uint32_t s = i % AT_RING;
            if (!mbar_wait_warp(&ctl->k_full[s], (i / AT_RING) & 1u, abort_flag)) return false;
            if (i > 0 && !mbar_wait_warp(&ctl->s_free, (i - 1) & 1u, abort_flag)) return false;
            tc_fence_after_sync();
            if (elect_one()) {
                const uint64_t kd = umma_desc_sw128(smem_u32(k_s + s * AT_KV_BYTES));
#pragma unroll
                for (int ks = 0; ks < AT_D / 16; ks++) umma_f16(t_s, qd + (uint64_t)ks * 2, kd + (uint64_t)ks * 2, idesc_s, ks > 0 ? 1u : 0u);
                umma_commit(&ctl->k_empty[s]);
                if (last) umma_commit(&ctl->q_empty);   // every product with this Q tile is issued
                umma_commit(&ctl->s_full);
            }
            __syncwarp();
            return true;
        };
        for (int item = p.first + blockIdx.x; item < items && !dead; item += gridDim.x, local++) {
            const AttnItem it(p, item);
            dead = !mbar_wait_warp(&ctl->q_full, local & 1u, abort_flag) || !scores(n, it.steps == 1);
            for (int t = 0; t < it.steps && !dead; t++, n++) {
                if (t + 1 < it.steps && !scores(n + 1, t + 2 == it.steps)) { dead = true; break; }
                const uint32_t s = n % AT_RING;
                if (!mbar_wait_warp(&ctl->v_full[s], (n / AT_RING) & 1u, abort_flag) || !mbar_wait_warp(&ctl->p_full, n & 1u, abort_flag)) { dead = true; break; }
                tc_fence_after_sync();
                if (elect_one()) {
                    const uint64_t vd = umma_desc_mn(v_bits, smem_u32(v_s + s * AT_KV_BYTES));
#pragma unroll
                    for (int ks = 0; ks < AT_KEYS / 16; ks++)
                        umma_f16(t_o, pd + (uint64_t)ks * 2, vd + (uint64_t)ks * (2048 >> 4), idesc_o, ks > 0 ? 1u : (t > 0 ? 1u : 0u));
                    umma_commit(&ctl->v_empty[s]);
                    umma_commit(&ctl->o_full);
                }
                __syncwarp();
            }
        }
        // The CTA's shared and tensor memory go only when no copy and no product is under way to them.  Given up at step n of item
        // local - 1, K copies may be out up to step n + 2, V copies and score products up to n + 1, Q up to the next item.
        const long long t0 = clock64();
        if (dead) {
            attn_give_up(ctl, p.status, OB200_ERR_WAIT_FULL);
            for (uint32_t i = n; i < n + 3; i++) mbar_wait_landed(&ctl->k_full[i % AT_RING], (i / AT_RING) & 1u, t0);
            for (uint32_t i = n; i < n + 2; i++) mbar_wait_landed(&ctl->v_full[i % AT_RING], (i / AT_RING) & 1u, t0);
            for (uint32_t i = n; i < n + 2; i++) mbar_wait_landed(&ctl->s_full, i & 1u, t0);
            for (uint32_t i = local - 1; i != local + 1; i++) mbar_wait_landed(&ctl->q_full, i & 1u, t0);
        }
        if (n > 0) mbar_wait_landed(&ctl->o_full, (n - 1) & 1u, t0);
        __syncwarp();
    } else {
        // ------------------------------------------------------------ softmax: thread r owns query row q0 + r (tensor-memory lane r)
        const int r = warp * 32 + lane;
        const uint32_t lanes = (uint32_t)(warp * 32) << 16;
        uint32_t n = 0;
        bool ok = true;
        for (int item = p.first + blockIdx.x; item < items && ok; item += gridDim.x) {
            const AttnItem it(p, item);
            const int qpos = it.qt * AT_QROWS + r;
            const int key_end = p.causal && qpos + 1 < p.S ? qpos + 1 : p.S;   // keys [0, key_end) count
            float m_ref = 0.f, sum = 0.f;   // reference maximum (scaled, base 2) and the sum of 2^(score - m_ref)
            for (int t = 0; t < it.steps; t++, n++) {
                ok = __all_sync(0xffffffffu, mbar_wait(&ctl->s_full, n & 1u, abort_flag));
                if (!ok) break;
                tc_fence_after_sync();
                float x[AT_KEYS];
                {
                    uint32_t lo[32], hi[32];
                    tmem_ld_32x32(t_s + lanes, lo);
                    tmem_ld_32x32(t_s + lanes + 32, hi);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 32; j++) { x[j] = __uint_as_float(lo[j]); x[32 + j] = __uint_as_float(hi[j]); }
                }
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&ctl->s_free);
                if (p.factor != 1.f) {
#pragma unroll
                    for (int j = 0; j < AT_KEYS; j++) x[j] *= p.factor;
                }
                const int left = key_end - t * AT_KEYS;
                if (left < AT_KEYS) {
#pragma unroll
                    for (int j = 0; j < AT_KEYS; j++)
                        if (j >= left) x[j] = -INFINITY;
                }
                float mx[4] = {x[0], x[1], x[2], x[3]};
#pragma unroll
                for (int j = 4; j < AT_KEYS; j++) mx[j & 3] = fmaxf(mx[j & 3], x[j]);
                const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * p.scale_log2;
                // The sums and the output stay relative to m_ref, which follows the row's maximum only when that has grown by
                // 2^AT_RESCALE: float32 has the range, and the output in tensor memory is hardly ever read back.
                bool waited = false;
                if (t == 0) {
                    m_ref = fmaxf(top, -FLT_MAX);   // finite where all scores so far are -infinity: they weigh nothing, unless no other follows
                } else if (__any_sync(0xffffffffu, top > m_ref + AT_RESCALE)) {
                    const bool grow = top > m_ref + AT_RESCALE;
                    const float f = grow ? exp2_approx(m_ref - top) : 1.f;
                    if (grow) m_ref = top;
                    sum *= f;
                    ok = __all_sync(0xffffffffu, mbar_wait(&ctl->o_full, (n - 1) & 1u, abort_flag));
                    if (!ok) break;
                    waited = true;
                    tc_fence_after_sync();
#pragma unroll 1
                    for (int c = 0; c < AT_D; c += 16) {
                        uint32_t o[16];
                        tmem_ld_32x16(t_o + lanes + c, o);
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 16; j++) o[j] = __float_as_uint(__uint_as_float(o[j]) * f);
                        tmem_st_32x16(t_o + lanes + c, o);
                    }
                    tmem_st_wait();
                }
                uint32_t pk[AT_KEYS / 2];
                float part[2] = {0.f, 0.f};
#pragma unroll
                for (int j = 0; j < AT_KEYS; j += 2) {
                    const __nv_bfloat162 h2 = __floats2bfloat162_rn(exp2_approx(fmaf(x[j], p.scale_log2, -m_ref)),
                                                                    exp2_approx(fmaf(x[j + 1], p.scale_log2, -m_ref)));
                    // the row sum is taken over the rounded values the tensor core will multiply
                    part[0] += __low2float(h2);
                    part[1] += __high2float(h2);
                    pk[j / 2] = *reinterpret_cast<const uint32_t*>(&h2);
                }
                sum += part[0] + part[1];
                if (n > 0 && !waited) {   // O += P(n-1) . V(n-1) has read the shared-memory tile
                    ok = __all_sync(0xffffffffu, mbar_wait(&ctl->o_full, (n - 1) & 1u, abort_flag));
                    if (!ok) break;
                }
#pragma unroll
                for (int ch = 0; ch < AT_KEYS / 8; ch++)
                    *reinterpret_cast<uint4*>(p_s + sw128_offset((uint32_t)r, (uint32_t)ch)) =
                        make_uint4(pk[4 * ch], pk[4 * ch + 1], pk[4 * ch + 2], pk[4 * ch + 3]);
                fence_proxy_async_smem();   // the tensor core reads P through the async proxy
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&ctl->p_full);
            }
            if (!ok) break;
            ok = __all_sync(0xffffffffu, mbar_wait(&ctl->o_full, (n - 1) & 1u, abort_flag));
            if (!ok) break;
            tc_fence_after_sync();
            const float inv = 1.0f / sum;
            __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(p.ctx) + ((long long)it.b * p.S + qpos) * (p.H * AT_D) + it.h * AT_D;
#pragma unroll
            for (int half = 0; half < 2; half++) {
                uint32_t v[32];
                tmem_ld_32x32(t_o + lanes + half * 32, v);
                tmem_ld_wait();
                if (qpos < p.S) {
#pragma unroll
                    for (int ch = 0; ch < 4; ch++) {
                        uint4 o4;
                        uint32_t* w = &o4.x;
#pragma unroll
                        for (int e = 0; e < 4; e++) {
                            const __nv_bfloat162 h2 = __floats2bfloat162_rn(__uint_as_float(v[ch * 8 + e * 2]) * inv,
                                                                            __uint_as_float(v[ch * 8 + e * 2 + 1]) * inv);
                            w[e] = *reinterpret_cast<const uint32_t*>(&h2);
                        }
                        *reinterpret_cast<uint4*>(out + half * 32 + ch * 8) = o4;
                    }
                }
            }
            tc_fence_before_sync();   // the next item's first product overwrites O only behind its p_full
        }
        if (!ok) attn_give_up(ctl, p.status, OB200_ERR_WAIT_TMEM_FULL);
    }
    __syncthreads();
    if (warp == 5) {
        __syncwarp();
        tc_fence_after_sync();
        tmem_dealloc(t_s, 2 * AT_KEYS);
    }
}

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                   const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn attn_encode_fn() {
    static const EncodeTiledFn fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess)
            f = nullptr;
        return reinterpret_cast<EncodeTiledFn>(f);
    }();
    return fn;
}

}  // namespace ob200

extern "C" int* ob200_status_word_for_current_device(void);

// See include/orion_kernels.h.  Returns -1 for unsupported sizes, -2 for misaligned pointers, -4 when the TMA descriptor cannot
// be built.
extern "C" int ob200_attention_long_bf16(const void* qkv, void* ctx, int B, int S, int H, int head_dim, float scale, int causal, int part,
                                         int parts, int num_ctas, void* stream) {
    using namespace ob200;
    if (B <= 0 || S <= 0) return 0;
    if (head_dim != AT_D || H <= 0 || num_ctas <= 0 || parts < 1 || part < 0 || part >= parts) return -1;
    if (((uintptr_t)qkv | (uintptr_t)ctx) % 16) return -2;
    EncodeTiledFn enc = attn_encode_fn();
    if (!enc) return -4;
    AttnParams p;
    memset(&p, 0, sizeof p);
    p.ctx = ctx;
    p.status = ob200_status_word_for_current_device();
    p.B = B; p.S = S; p.H = H;
    p.causal = causal ? 1 : 0;
    p.factor = scale < 0.f ? -1.f : scale == 0.f ? 0.f : 1.f;
    p.scale_log2 = scale == 0.f ? 1.f : (scale < 0.f ? -scale : scale) * 1.4426950408889634f;
    p.q_tiles = (S + AT_QROWS - 1) / AT_QROWS;
    const long long all = (long long)B * H * p.q_tiles;
    if (all > 0x3fffffffLL) return -1;
    p.first = (int)(all * part / parts);
    p.last = (int)(all * (part + 1) / parts);
    const int items = p.last - p.first;
    if (items == 0) return 0;
    cuuint64_t dims[4] = {(cuuint64_t)AT_D, (cuuint64_t)(3 * H), (cuuint64_t)S, (cuuint64_t)B};
    cuuint64_t strides[3] = {(cuuint64_t)AT_D * 2, (cuuint64_t)3 * H * AT_D * 2, (cuuint64_t)S * 3 * H * AT_D * 2};
    cuuint32_t box[4] = {AT_D, 1, AT_KEYS, 1};
    cuuint32_t steps[4] = {1, 1, 1, 1};
    if (enc(reinterpret_cast<CUtensorMap*>(p.tmap), CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(qkv), dims, strides, box, steps,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return -4;
    static bool attr_set[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 64 && !attr_set[dev]) {
        cudaError_t e = cudaFuncSetAttribute(attention_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, AT_SMEM);
        if (e != cudaSuccess) return (int)e;
        attr_set[dev] = true;
    }
    OB200_ELASTIC(attention_fwd_kernel, AT_CTAS_PER_SM);
    annotate_launch(1, 4.0 * B * H * (double)S * S * AT_D / parts, 2.0 * B * S * H * AT_D * 4.0 / parts);
    const long long most = (long long)num_ctas * AT_CTAS_PER_SM;
    // Programmatic dependent launch: barriers and tensor memory are set up under the tail of the kernel before it; global memory
    // is read and written only behind griddepcontrol.wait.
    static const bool pdl = [] {   // ORION_PDL=0: plain stream order between consecutive kernels
        const char* e = getenv("ORION_PDL");
        return !(e && e[0] == '0');
    }();
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof cfg);
    cfg.gridDim = dim3((unsigned)(items < most ? items : most));
    cfg.blockDim = dim3(AT_THREADS);
    cfg.dynamicSmemBytes = AT_SMEM;
    cfg.stream = (cudaStream_t)stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    return (int)cudaLaunchKernelEx(&cfg, attention_fwd_kernel, p);
}

// The entry point of the inference clients: sequences up to 384 keys.
extern "C" int ob200_attention_fwd_bf16(const void* qkv, void* ctx, int B, int S, int H, int head_dim, float scale, int causal,
                                        int num_ctas, void* stream) {
    if (B > 0 && S > 384) return -1;
    return ob200_attention_long_bf16(qkv, ctx, B, S, H, head_dim, scale, causal, 0, 1, num_ctas, stream);
}
